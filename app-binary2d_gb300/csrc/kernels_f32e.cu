// kernels_f32e.cu — the FP32 stage kernel of the Euler system.
#define B2D_NF 4
#define B2D_LAUNCH launch_stage_f32_euler
#define B2D_RESIDENT resident_f32_euler
#include "kernels_f32w.inc"
