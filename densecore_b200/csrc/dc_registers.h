// Whether a kernel starts with the registers a thread that it shares out anew among its warps (setmaxnreg draws on those alone).
#pragma once

// numRegs as cudaFuncGetAttributes gives it; a launch rounds it up to whole eights.  wanted 0: any number.
inline bool dc_registers_match(int num_regs, int wanted) { return wanted == 0 || (num_regs + 7) / 8 * 8 == wanted; }
