// Face-flux kernels of the split stage: f64 arithmetic, RUSA Riemann solver.
#include "stage_inst.cuh"

AMR_FACES_DEFINE(f64, rusa, amr::FLX_RUSA, double)
