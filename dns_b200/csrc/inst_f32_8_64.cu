#include "ops.cuh"

// the kernels of these sizes (instances.cuh): taking setup's address compiles
// every kernel it prepares
extern cudaError_t (*const dnsb_inst_f32_8_64[])();
cudaError_t (*const dnsb_inst_f32_8_64[])() = {&Ops<float, 8>::setup, &Ops<float, 16>::setup, &Ops<float, 32>::setup, &Ops<float, 64>::setup};
