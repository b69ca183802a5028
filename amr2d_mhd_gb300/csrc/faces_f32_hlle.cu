// Face-flux kernels of the split stage: f32 arithmetic, HLLE Riemann solver.
#include "stage_inst.cuh"

AMR_FACES_DEFINE(f32, hlle, amr::FLX_HLLE, float)
