"""What a build has to hold to for the kernels that load from tensor memory: no spilled registers, and the number of registers a thread that
k_gemm_tc shares out anew among its warps (a launch with fewer would wait for more without end).  The launchers refuse other builds; here the compiler is asked."""
import os
import re
import subprocess

import pytest

from densecore_b200 import build as B


def test_a_build_with_other_registers_is_refused(tmp_path):
    """The rule that the launchers apply, as the host compiler sees it: a launch hands out registers in eights."""
    src = tmp_path / "rule.cpp"
    src.write_text('#include <stdio.h>\n#include "dc_registers.h"\n'
                   "int main() { for (int r = 1; r <= 256; ++r) printf(\"%d%d\\n\", dc_registers_match(r, 72), dc_registers_match(r, 0)); }\n")
    subprocess.check_call(["g++", "-I", B.CSRC, str(src), "-o", str(tmp_path / "rule")])
    out = subprocess.check_output([str(tmp_path / "rule")], text=True).split()
    assert [r + 1 for r, s in enumerate(out) if s[0] == "1"] == list(range(65, 73)) and all(s[1] == "1" for s in out)


KERNELS = {"gemm_tc": ["k_gemm_tc"], "linear_tc": ["k_linear_tc", "k_linear_tc_wide"], "mix_gqa": ["k_gqa_prompt_tc"]}


@pytest.mark.parametrize("source", list(KERNELS))
def test_no_spills_and_the_registers_asked_for(tmp_path, source):
    path = os.path.join(B.CSRC, source + ".cu")
    wanted = re.search(r"TC_LAUNCH_REGS = (\d+)", open(path).read())
    cmd = [B.nvcc(), "-Xptxas", "-v", *B.NVCC_FLAGS, "-I", os.path.join(B.ROOT, "include"), "-c", path, "-o", str(tmp_path / "o.o")]
    out = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True, check=True).stdout
    seen = set()
    for name, body in re.findall(r"Compiling entry function '(\w+)'(.*?)(?=Compiling entry|\Z)", out, re.S):
        kernel = next((k for k in KERNELS[source] if re.search(rf"\d{k}(?!_)", name)), None)
        if not kernel:
            continue
        seen.add(kernel)
        assert "0 bytes stack frame, 0 bytes spill stores, 0 bytes spill loads" in body, (name, body)
        if wanted:
            assert (int(re.search(r"Used (\d+) registers", body)[1]) + 7) // 8 * 8 == int(wanted[1])
    assert seen == set(KERNELS[source])
