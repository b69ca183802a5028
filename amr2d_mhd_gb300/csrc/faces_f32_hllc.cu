// Face-flux kernels of the split stage: f32 arithmetic, HLLC Riemann solver.
#include "stage_inst.cuh"

AMR_FACES_DEFINE(f32, hllc, amr::FLX_HLLC, float)
