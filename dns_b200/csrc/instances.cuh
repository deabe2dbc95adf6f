// instances.cuh -- the kernels that the inst_*.cu translation units hold: a
// translation unit that includes this launches them without compiling them.
#pragma once
#include "kernels.cuh"

namespace dnsb {

#define DNSB_COL_M(R, N, A, F, M)                                                        \
  extern template __global__ void k_colpass_minb<R, N, A, F, M>(                         \
      const cx<R> *__restrict__, cx<R> *__restrict__, const cx<R> *__restrict__, Geo, ColJobs);
#define DNSB_COL(R, N, A, F)                                                             \
  extern template __global__ void k_colpass<R, N, A, F>(                                 \
      const cx<R> *__restrict__, cx<R> *__restrict__, const cx<R> *__restrict__, Geo, ColJobs); \
  DNSB_COL_MINB(DNSB_COL_M, R, N, A, F)
#define DNSB_X(R, N, S, T) \
  extern template __global__ void k_xstage<R, N, S, T>(XArgs<R>, const cx<R> *__restrict__, Geo);
#define DNSB_SIZE(R, N)                                                                  \
  DNSB_COL(R, N, 0, false) DNSB_COL(R, N, 0, true) DNSB_COL(R, N, 1, false)              \
  DNSB_COL(R, N, 1, true)                                                                \
  DNSB_X(R, N, -1, true) DNSB_X(R, N, 0, true) DNSB_X(R, N, 1, true) DNSB_X(R, N, 2, true) \
  DNSB_X(R, N, 3, true) DNSB_X(R, N, 3, false)                                           \
  extern template __global__ void k_zr2c<R, N>(const R *__restrict__, cx<R> *__restrict__, \
                                               const cx<R> *__restrict__, Geo);          \
  extern template __global__ void k_zc2r<R, N>(const cx<R> *__restrict__, double *__restrict__, \
                                               const cx<R> *__restrict__, Geo, double);
#define DNSB_YZ(R, N, K, KEEP)                                                           \
  extern template __global__ void k_yz<R, N, K, KEEP>(cx<R> *__restrict__, R *__restrict__, \
                                                      const cx<R> *__restrict__, Geo, R, \
                                                      R *__restrict__);
#define DNSB_PLANE(R, N)                                                                 \
  DNSB_YZ(R, N, 0, false) DNSB_YZ(R, N, 1, false) DNSB_YZ(R, N, 2, false)
#define DNSB_PLANE_KEEP(R, N) DNSB_YZ(R, N, 0, true) DNSB_YZ(R, N, 1, true)
#define DNSB_Z(R, N, K)                                                                  \
  extern template __global__ void k_zstage<R, N, K>(cx<R> *__restrict__, R *__restrict__, \
                                                    const cx<R> *__restrict__, Geo, R);
#define DNSB_ZK(R, N, K)                                                                 \
  extern template __global__ void k_zstage_keep<R, N, K>(cx<R> *__restrict__, R *__restrict__, \
                                                         const cx<R> *__restrict__, Geo, R, \
                                                         R *__restrict__);
#define DNSB_LINES(R, N)                                                                 \
  DNSB_Z(R, N, 0) DNSB_Z(R, N, 1) DNSB_Z(R, N, 2) DNSB_ZK(R, N, 0) DNSB_ZK(R, N, 1)
#define DNSB_PRECISION(R)                                                                \
  DNSB_PLANE(R, 8) DNSB_PLANE(R, 16) DNSB_PLANE(R, 32) DNSB_PLANE(R, 64)                 \
  DNSB_PLANE_KEEP(R, 8) DNSB_PLANE_KEEP(R, 16) DNSB_PLANE_KEEP(R, 32)                    \
  DNSB_LINES(R, 64) DNSB_LINES(R, 128) DNSB_LINES(R, 256) DNSB_LINES(R, 512)             \
  DNSB_SIZE(R, 8) DNSB_SIZE(R, 16) DNSB_SIZE(R, 32) DNSB_SIZE(R, 64)                     \
  DNSB_SIZE(R, 128) DNSB_SIZE(R, 256) DNSB_SIZE(R, 512)

DNSB_PRECISION(double)
DNSB_PRECISION(float)

}  // namespace dnsb
