// Face-flux kernels of the split stage: f32 arithmetic, RUSA Riemann solver.
#include "stage_inst.cuh"

AMR_FACES_DEFINE(f32, rusa, amr::FLX_RUSA, float)
