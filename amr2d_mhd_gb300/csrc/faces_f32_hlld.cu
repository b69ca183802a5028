// Face-flux kernels of the split stage: f32 arithmetic, HLLD Riemann solver.
#include "stage_inst.cuh"

AMR_FACES_DEFINE(f32, hlld, amr::FLX_HLLD, float)
