// The plane kernel (k_yz) on the host, for test_plane_kernel_order.py.
#include "emulate.h"
#include "kernels.cuh"

namespace dnsb {
__attribute__((aligned(16))) unsigned char smem_raw[1 << 18];
}

namespace {

using namespace dnsb;

template <class R, int N, int KIND>
struct Call {
  cx<R> *work;
  R *stale;
  const cx<R> *tw;
  Geo g;
  static void body(void *p) {
    Call &c = *(Call *)p;
    k_yz<R, N, KIND, false>(c.work, c.stale, c.tw, c.g, (R)(1.0 / ((double)N * N * N)), nullptr);
  }
};

template <class R, int N, int KIND>
int run(void *work, void *stale, const void *tw, int nfp, int kcut, int plane, int descending) {
  Geo g{};
  g.n = N;
  g.nf = N / 2 + 1;
  g.nfp = nfp;
  g.kcut = kcut;
  g.slot = (long long)N * N * nfp;
  g.nreal = (long long)N * N * N;
  Call<R, N, KIND> c{(cx<R> *)work, (R *)stale, (const cx<R> *)tw, g};
  return emu::run_block(YZ<R, N>::THREADS, descending, {(unsigned)plane, 0, 0},
                        Call<R, N, KIND>::body, &c);
}

template <class R, int N>
int run_kind(int kind, void *work, void *stale, const void *tw, int nfp, int kcut, int plane,
             int descending) {
  return kind == 0   ? run<R, N, 0>(work, stale, tw, nfp, kcut, plane, descending)
         : kind == 1 ? run<R, N, 1>(work, stale, tw, nfp, kcut, plane, descending)
                     : run<R, N, 2>(work, stale, tw, nfp, kcut, plane, descending);
}
template <class R>
int run_n(int n, int kind, void *work, void *stale, const void *tw, int nfp, int kcut, int plane,
          int descending) {
  switch (n) {
    case 8: return run_kind<R, 8>(kind, work, stale, tw, nfp, kcut, plane, descending);
    case 16: return run_kind<R, 16>(kind, work, stale, tw, nfp, kcut, plane, descending);
    case 32: return run_kind<R, 32>(kind, work, stale, tw, nfp, kcut, plane, descending);
    case 64: return run_kind<R, 64>(kind, work, stale, tw, nfp, kcut, plane, descending);
  }
  return -1;
}

}  // namespace

// 1: the block has run to its end
extern "C" int plane_run(int fp64, int n, int kind, void *work, void *stale, const void *tw, int nfp,
                         int kcut, int plane, int descending) {
  return fp64 ? run_n<double>(n, kind, work, stale, tw, nfp, kcut, plane, descending)
              : run_n<float>(n, kind, work, stale, tw, nfp, kcut, plane, descending);
}
