#include "ens_kernel.cuh"

namespace dnsb {

template cudaError_t p_prepare<float>(size_t, int *);
template cudaError_t p_launch<float>(int, size_t, cudaStream_t, const PPlan<float> *, PSync *,
                                     unsigned long long);

}  // namespace dnsb
