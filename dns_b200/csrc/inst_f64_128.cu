#include "ops.cuh"

// the kernels of these sizes (instances.cuh): taking setup's address compiles
// every kernel it prepares
extern cudaError_t (*const dnsb_inst_f64_128[])();
cudaError_t (*const dnsb_inst_f64_128[])() = {&Ops<double, 128>::setup};
