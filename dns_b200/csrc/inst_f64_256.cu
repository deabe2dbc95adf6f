#include "ops.cuh"

// the kernels of these sizes (instances.cuh): taking setup's address compiles
// every kernel it prepares
extern cudaError_t (*const dnsb_inst_f64_256[])();
cudaError_t (*const dnsb_inst_f64_256[])() = {&Ops<double, 256>::setup};
