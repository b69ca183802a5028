// Face-flux kernels of the split stage: f64 arithmetic, HLLC Riemann solver.
#include "stage_inst.cuh"

AMR_FACES_DEFINE(f64, hllc, amr::FLX_HLLC, double)
