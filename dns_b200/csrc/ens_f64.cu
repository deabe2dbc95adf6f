#include "ens_kernel.cuh"

namespace dnsb {

cudaError_t p_barrier_selftest(PSync *sy, cudaStream_t st, unsigned long long wait_ns) {
  k_barrier_selftest<<<2, 32, 0, st>>>(sy, wait_ns);
  return cudaGetLastError();
}

template cudaError_t p_prepare<double>(size_t, int *);
template cudaError_t p_launch<double>(int, size_t, cudaStream_t, const PPlan<double> *, PSync *,
                                     unsigned long long);

}  // namespace dnsb
