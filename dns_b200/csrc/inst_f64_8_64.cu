#include "ops.cuh"

// the kernels of these sizes (instances.cuh): taking setup's address compiles
// every kernel it prepares
extern cudaError_t (*const dnsb_inst_f64_8_64[])();
cudaError_t (*const dnsb_inst_f64_8_64[])() = {&Ops<double, 8>::setup, &Ops<double, 16>::setup, &Ops<double, 32>::setup, &Ops<double, 64>::setup};
