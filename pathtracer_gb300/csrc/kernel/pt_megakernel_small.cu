// pt_megakernel_small.cu — pt_megakernel_analytic.cu for small frames: with a
// block an SM the time is the longest path's chain of steps, which calls
// lengthen, and the warps are too few to wait for one another's instructions.
#define PT_MK_SMALL
#define ptk_launch_megakernel_analytic ptk_launch_megakernel_small
#include "pt_megakernel_analytic.cu"
