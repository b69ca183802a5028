// Face-flux kernels of the split stage: f64 arithmetic, HLLD Riemann solver.
#include "stage_inst.cuh"

AMR_FACES_DEFINE(f64, hlld, amr::FLX_HLLD, double)
