// kernels_f32.cu — the FP32 stage kernel of the isothermal system, over FP64
// state or compensated FP32 state.
#define B2D_NF 3
#define B2D_LAUNCH launch_stage_f32_iso
#define B2D_RESIDENT resident_f32_iso
#include "kernels_f32w.inc"
