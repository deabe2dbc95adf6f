#include "ops.cuh"

// the kernels of these sizes (instances.cuh): taking setup's address compiles
// every kernel it prepares
extern cudaError_t (*const dnsb_inst_f32_512[])();
cudaError_t (*const dnsb_inst_f32_512[])() = {&Ops<float, 512>::setup};
