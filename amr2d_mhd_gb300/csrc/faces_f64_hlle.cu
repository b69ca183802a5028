// Face-flux kernels of the split stage: f64 arithmetic, HLLE Riemann solver.
#include "stage_inst.cuh"

AMR_FACES_DEFINE(f64, hlle, amr::FLX_HLLE, double)
