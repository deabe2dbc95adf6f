// adjoint.cuh -- pointwise kernels of the discrete adjoint of the RK4 step.
// Templates on the storage complex type C (double2 for the FP64 adjoint,
// float2 for the mixed one); the arithmetic is FP64 in registers, rounded
// once on store.  The forward stage of main.c:344-413 is, per RK stage s with input
// U_s (half spectrum) and, at s == 0, the stale real velocity:
//   u   = s > 0 ? a c2r(U_s) : stale          a = 1/n^3
//   w   = a c2r(D U_s)                        D U = i k x U  (curl)
//   N   = u x w
//   dU  = Pi(m dt r2c(N)) - nu dt kk U_s       Pi(X) = X - k (k.X)/kk
// Its transpose under the real inner product of the stored entries uses
//   c2r^T(y) = w_z * r2c(y),  r2c^T(Y) = c2r(Y / w_z),
//   w_z = 1 on the kz = 0 and kz = n/2 planes, 2 elsewhere,
// (c2r with FFTW's semantics is sum_k w_z Re(X e^{ik.x})); D and Pi are
// self-adjoint; (u x w)^T: lambda_u = w x lambda_N, lambda_w = lambda_N x u.
#pragma once
#include "kernels.cuh"

namespace dnsb {

// the loop over the valid half-spectrum points of one slot set
#define DNSB_FOR_POINTS(g)                                                              \
  for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x,                 \
                 npts_ = (long long)(g).n * (g).n * (g).nf;                             \
       q < npts_; q += (long long)gridDim.x * blockDim.x)

struct PointK {
  long long o;     // offset in a slot
  double kx, ky, kz, kk;
  int col;
  bool in;         // inside the 2/3 mask
  double wz;       // 1 on kz = 0, n/2; 2 elsewhere
};

__device__ __forceinline__ PointK point_k(const Geo &g, long long q) {
  PointK p;
  const long long row = q / g.nf;
  const int col = (int)(q - row * g.nf);
  const int i = (int)(row / g.n), j = (int)(row - (long long)i * g.n);
  p.o = row * g.nfp + col;
  const int ikx = kwave(i, g.n), iky = kwave(j, g.n);
  p.kx = ikx;
  p.ky = iky;
  p.kz = col;
  p.kk = p.kx * p.kx + p.ky * p.ky + p.kz * p.kz;
  p.col = col;
  p.in = (ikx < 0 ? -ikx : ikx) <= g.kcut && (iky < 0 ? -iky : iky) <= g.kcut && col <= g.kcut;
  p.wz = (col == 0 || col == g.n / 2) ? 1.0 : 2.0;
  return p;
}

// i k x U at one point (main.c:359-361, with kx[n/2] = -n/2)
__device__ __forceinline__ void curl_at(const PointK &p, cd u, cd v, cd w, cd &ox, cd &oy, cd &oz) {
  // i * (a) = (-a.y, a.x)
  const cd ax = make_double2(p.ky * w.x - p.kz * v.x, p.ky * w.y - p.kz * v.y);
  const cd ay = make_double2(p.kz * u.x - p.kx * w.x, p.kz * u.y - p.kx * w.y);
  const cd az = make_double2(p.kx * v.x - p.ky * u.x, p.kx * v.y - p.ky * u.y);
  ox = make_double2(-ax.y, ax.x);
  oy = make_double2(-ay.y, ay.x);
  oz = make_double2(-az.y, az.x);
}

// Input U_s of RK stage s at a point: the state (s == 0), the packed stage
// input inside the 2/3 rule, the state times lin_coef outside it.
template <class C>
struct StageIn {
  const C *u0, *rk;
  int s;
  double nudt;
  __device__ __forceinline__ C at(const Geo &g, const PointK &p, int f) const {
    using R = sc<C>;
    if (s > 0 && p.in) {
      const int ix = (int)p.kx < 0 ? (int)p.kx + g.mk : (int)p.kx;
      const int iy = (int)p.ky < 0 ? (int)p.ky + g.mk : (int)p.ky;
      return rk[(3 * (s - 1) + f) * g.slotc + ((long long)ix * g.mk + iy) * g.mp + p.col];
    }
    const C z = u0[f * g.slot + p.o];
    if (s == 0) return z;
    const R c = (R)(nudt * p.kk);
    const R m = s == 1 ? lin_coef<0>(c) : s == 2 ? lin_coef<1>(c) : lin_coef<2>(c);
    return cmk<C>(fma_rn(m, z.x, z.x), fma_rn(m, z.y, z.y));
  }
};

// out = (m dt Pi(ldU)) / w_z : the adjoint of N_hat, divided by the c2r
// weights so that a plain c2r of `out` is r2c^T of m dt Pi(ldU)
template <class C>
__global__ void k_adj_lamN(const C *__restrict__ ldU, C *__restrict__ out, Geo g, double dt) {
  DNSB_FOR_POINTS(g) {
    const PointK p = point_k(g, q);
    cd x = to_d(ldU[p.o]), y = to_d(ldU[g.slot + p.o]), z = to_d(ldU[2 * g.slot + p.o]);
    if (p.kk > 0) {
      const double sr = (x.x * p.kx + y.x * p.ky + z.x * p.kz) / p.kk;
      const double si = (x.y * p.kx + y.y * p.ky + z.y * p.kz) / p.kk;
      x = make_double2(x.x - sr * p.kx, x.y - si * p.kx);
      y = make_double2(y.x - sr * p.ky, y.y - si * p.ky);
      z = make_double2(z.x - sr * p.kz, z.y - si * p.kz);
    }
    const double s = (p.in ? dt : 0.0) / p.wz;
    out[p.o] = from_d<C>(cscale(x, s));
    out[g.slot + p.o] = from_d<C>(cscale(y, s));
    out[2 * g.slot + p.o] = from_d<C>(cscale(z, s));
  }
}

// The z part of a transposed stage, per z line: lambda_N (slots 0-2 of work,
// zero past kcut) to real space, with the stage's real velocity u and
// vorticity om
//   lambda_u = om x lambda_N (+ lst),  lambda_om = lambda_N x u
// in FP64, rounded once to the storage type, and their forward transforms:
// lambda_om to slots 0-2, lambda_u to slots 3-5, or with LAST (stage 0, whose
// velocity is the stale one) lambda_u itself, real, to lst_out.  Two real
// transforms run as one complex one, as in the z pass.  One kernel in place
// of a c2r, a pointwise and two r2c passes: 15 slots of traffic a stage, not
// 33.
template <class R, int N>
struct ZA {
  using P = Plan<N>;
  static constexpr int E = P::E, T = N / E, M = N / 2;
  static constexpr int THREADS = (N * N * T) < 128 ? (N * N * T) : 128;
  static constexpr int LINES = THREADS / T;
  static constexpr int PADSH = E >= 16 ? 4 : 3;
  static constexpr int XB = N + (N >> PADSH);
  static constexpr int TWN = StageTw<P>::SIZE / 2 * 2 + 2;
  static constexpr size_t SMEM = (size_t)(TWN + LINES * XB) * sizeof(cx<R>) + (size_t)LINES * 3 * N * sizeof(R);
  static constexpr int MINB = sizeof(R) == 8 ? 2 : 4;
};
template <class R, int N, bool LAST>
__global__ void __launch_bounds__(ZA<R, N>::THREADS, ZA<R, N>::MINB)
    k_zadj(cx<R> *work, const R *__restrict__ u, const R *__restrict__ om,
           const double *__restrict__ lst, double *__restrict__ lst_out,
           const cx<R> *__restrict__ twg, Geo g) {
  using C = cx<R>;
  using Z = ZA<R, N>;
  constexpr int E = Z::E, T = Z::T, M = Z::M;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C *tw = (C *)smem_raw;
  build_stage_tw<N, typename Z::P>(tw, twg, N, threadIdx.x, blockDim.x);
  __syncthreads();
  const int lid = threadIdx.x / T, t = threadIdx.x % T;
  C *xb = tw + Z::TWN + lid * Z::XB;
  R *sl = (R *)(tw + Z::TWN + Z::LINES * Z::XB) + lid * 3 * N + t;  // own points: sl[f * N + T * e]
  const long long line = (long long)blockIdx.x * Z::LINES + lid;  // N * N is a multiple of LINES
  C *row = work + line * g.nfp;
  const long long r0 = line * N + t;
  const LineSync<(T > 32)> sync{};
  const PadShift<Z::PADSH> idx{};
  C y[E];
  auto ext = [&](const C *a, const C *b) {  // the pair's Hermitian extension
#pragma unroll
    for (int e = 0; e < E; e++) {
      const int k = t + T * e;
      const bool direct = k <= M;
      const int q = direct ? k : N - k;
      C va = q <= g.kcut ? a[q] : czero<C>();
      C vb = b && q <= g.kcut ? b[q] : czero<C>();
      if (q == 0 || q == M) {
        va.y = 0;
        vb.y = 0;
      }
      if (!direct) {
        va.y = -va.y;
        vb.y = -vb.y;
      }
      y[e] = cmk<C>(va.x - vb.y, va.y + vb.x);
    }
  };
  ext(row, row + g.slot);
  line_fft<N, typename Z::P, false>(y, t, tw, xb, idx, sync);
#pragma unroll
  for (int e = 0; e < E; e++) {
    sl[T * e] = y[e].x;
    sl[N + T * e] = y[e].y;
  }
  ext(row + 2 * g.slot, nullptr);
  line_fft<N, typename Z::P, false>(y, t, tw, xb, idx, sync);
#pragma unroll
  for (int e = 0; e < E; e++) sl[2 * N + T * e] = y[e].x;

  // component f of the cross product of two fields at own point e: from lambda_N
  // and the velocity (OM) or from the vorticity and lambda_N
  auto l_ = [&](int f, int e) -> double { return sl[f * N + T * e]; };
  auto lom = [&](int f, int e) -> R {
    const int a = (f + 1) % 3, b = (f + 2) % 3;
    const double ua = u[a * g.nreal + r0 + T * e], ub = u[b * g.nreal + r0 + T * e];
    return (R)(l_(a, e) * ub - l_(b, e) * ua);
  };
  auto lu = [&](int f, int e) -> R {
    const int a = (f + 1) % 3, b = (f + 2) % 3;
    const double wa = om[a * g.nreal + r0 + T * e], wb = om[b * g.nreal + r0 + T * e];
    double v = wa * l_(b, e) - wb * l_(a, e);
    if (lst) v += lst[f * g.nreal + r0 + T * e];
    return (R)v;
  };
  // forward transform of the pair in y into two slots (the second may be none)
  auto out = [&](int sa, int sb) {
    line_fft<N, typename Z::P, true>(y, t, tw, xb, idx, sync);
    C *oa = row + sa * g.slot, *ob = row + sb * g.slot;
    if (sb < 0) {
#pragma unroll
      for (int e = 0; e <= E / 2; e++)
        if (t + T * e <= M) oa[t + T * e] = y[e];
      return;
    }
#pragma unroll
    for (int e = 0; e < E; e++) xb[idx(t + T * e)] = y[e];
    sync();
#pragma unroll
    for (int e = 0; e <= E / 2; e++) {
      const int k = t + T * e;
      if (k <= M) {
        const C z = y[e], p = xb[idx((N - k) & (N - 1))];
        oa[k] = cmk<C>(R(0.5) * (z.x + p.x), R(0.5) * (z.y - p.y));
        ob[k] = cmk<C>(R(0.5) * (z.y + p.y), -R(0.5) * (z.x - p.x));  // -i (Z - conj P) / 2
      }
    }
    sync();
  };
#pragma unroll
  for (int e = 0; e < E; e++) y[e] = cmk<C>(lom(0, e), lom(1, e));
  out(0, 1);
  if constexpr (LAST) {
#pragma unroll
    for (int e = 0; e < E; e++) {
      y[e] = cmk<C>(lom(2, e), R(0));
#pragma unroll
      for (int f = 0; f < 3; f++) lst_out[f * g.nreal + r0 + T * e] = (double)lu(f, e);
    }
    out(2, -1);
  } else {
#pragma unroll
    for (int e = 0; e < E; e++) y[e] = cmk<C>(lom(2, e), lu(0, e));
    out(2, 3);
#pragma unroll
    for (int e = 0; e < E; e++) y[e] = cmk<C>(lu(1, e), lu(2, e));
    out(4, 5);
  }
}

// lUs = a w_z (curl(Rw) + Ru) - nu dt kk ldU       (Ru may be null: stage 0),
// the adjoint of the stage input U_s = U0 + b dU_{s-1}, consumed at once:
//   lhat_out = lhat_in + lUs                (lambda of U0, accumulated)
//   ldU      = bn lUs + an lacc             (lambda of dU_{s-1}; not at stage 0)
// with ldU overwritten in place; and the nu-gradient terms <ldU, -dt kk Us>,
// double-double block partials
template <int BS, class C>
__global__ void __launch_bounds__(BS)
    k_adj_collect(const C *__restrict__ Rw, const C *__restrict__ Ru, C *ldU,
                  StageIn<C> Us, const C *lhat_in, C *lhat_out,
                  const C *__restrict__ lacc, Geo g, double a, double nu, double dt, double bn,
                  double an, bool next, double4 *__restrict__ partial) {
  DD gn{0.0, 0.0}, unused{0.0, 0.0};
  DNSB_FOR_POINTS(g) {
    const PointK p = point_k(g, q);
    cd cxyz[3];
    curl_at(p, to_d(Rw[p.o]), to_d(Rw[g.slot + p.o]), to_d(Rw[2 * g.slot + p.o]), cxyz[0],
            cxyz[1], cxyz[2]);
    const double s = a * p.wz, c = nu * dt * p.kk;
    double dotp = 0.0;
#pragma unroll
    for (int f = 0; f < 3; f++) {
      const long long o = f * g.slot + p.o;
      cd cf = cxyz[f];
      if (Ru) cf = cadd(cf, to_d(Ru[o]));
      const cd l = to_d(ldU[o]), u = to_d(Us.at(g, p, f));
      dotp += l.x * u.x;
      dotp += l.y * u.y;
      const cd lus = make_double2(s * cf.x - c * l.x, s * cf.y - c * l.y);
      lhat_out[o] = from_d<C>(cadd(to_d(lhat_in[o]), lus));
      if (next) ldU[o] = from_d<C>(cadd(cscale(lus, bn), cscale(to_d(lacc[o]), an)));
    }
    gn = dd_add_d(gn, -dt * p.kk * dotp);
  }
  dd_block_reduce<BS>(gn, unused, partial + blockIdx.x);
}

// acc (device double-double, .x .y) += sum of np block partials (.x .y)
template <int BS>
__global__ void __launch_bounds__(BS) k_dd_accumulate(const double4 *__restrict__ partial, int np,
                                                      double4 *__restrict__ acc) {
  DD e{0.0, 0.0}, unused{0.0, 0.0};
  for (int q = threadIdx.x; q < np; q += BS) e = dd_add(e, DD{partial[q].x, partial[q].y});
  __shared__ double4 tot;
  dd_block_reduce<BS>(e, unused, &tot);
  __syncthreads();
  if (threadIdx.x == 0) {
    const DD s = dd_add(DD{acc->x, acc->y}, DD{tot.x, tot.y});
    acc->x = s.hi;
    acc->y = s.lo;
  }
}

// out = a x + b y on 3 slots (y may be null)
template <class C>
__global__ void k_lincomb3(const C *__restrict__ x, const C *__restrict__ y, C *__restrict__ out,
                           Geo g, double a, double b) {
  DNSB_FOR_POINTS(g) {
    const long long row = q / g.nf;
    const long long o = row * g.nfp + (q - row * g.nf);
#pragma unroll
    for (int f = 0; f < 3; f++) {
      const cd xv = to_d(x[f * g.slot + o]);
      cd r = cscale(xv, a);
      if (y) r = cadd(r, cscale(to_d(y[f * g.slot + o]), b));
      out[f * g.slot + o] = from_d<C>(r);
    }
  }
}

// out = x / w_z on 3 slots (r2c^T = c2r of this)
template <class C>
__global__ void k_div_wz3(const C *__restrict__ x, C *__restrict__ out, Geo g) {
  DNSB_FOR_POINTS(g) {
    const PointK p = point_k(g, q);
#pragma unroll
    for (int f = 0; f < 3; f++)
      out[f * g.slot + p.o] = from_d<C>(cscale(to_d(x[f * g.slot + p.o]), 1.0 / p.wz));
  }
}

// y += x on n real values
__global__ void k_add_real(const double *__restrict__ x, double *__restrict__ y, long long n) {
  for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < n;
       q += (long long)gridDim.x * blockDim.x)
    y[q] += x[q];
}

}  // namespace dnsb
