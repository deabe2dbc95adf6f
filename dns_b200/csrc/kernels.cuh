// kernels.cuh -- the sm_100a kernels of one RK4 stage of the pseudo-spectral
// Navier-Stokes step (slitvinov/dns main.c:343-414), plus the initial
// forward transform (main.c:249-251), the dump transforms (main.c:270-279)
// and the energy/enstrophy reduction (main.c:257-266).
//
// Every kernel is a template on the storage scalar R: double for the FP64
// path, float for the mixed path (FP32 fields, FFTs and pointwise arithmetic;
// FP64 reductions, and the viscous coefficient nu dt |k|^2 is formed in FP64
// and rounded once).
//
// HBM layout (one "slot" = one complex field on the half spectrum):
//   spectral slot  [i = kx index][j = ky index][k = kz index], k fastest,
//                  row pitch nfp = nf rounded up to the column tile width W
//                  (nf = n/2 + 1; W * sizeof(complex) = 128 bytes), so every
//                  tile row starts on a 128-byte boundary; the padding
//                  columns are never written by a pass and their values never
//                  used (the FP32 kernels' 16-byte copies of pairs of columns
//                  read the first of them).
//   real slot      [x][y][z], z fastest (the .raw layout of main.c:180-185).
// The same slot shape holds partially transformed data: after the x pass the
// first index is x instead of kx, after the y pass the second is y.
//
// One RK stage = four kernels (two where YZ runs B, C and D in one: n <= 32,
// and three or more runs of n = 64):
//   B   y backward  5 slots -> u,v,w, omega_z = dv/dx - du/dy, dw/dx, dw/dy
//   C   z pass      per z line: vorticity from the 6 slots, u and omega to
//                   real space, N = u x omega, N back to z spectral (stored
//                   for kz <= kcut); real space touches HBM only for the
//                   stale velocity
//   D   y forward   3 slots, in place, tiles with kz <= kcut, |ky| <= kcut kept
//   X   x update    per x line of all three fields: x forward of N, 2/3 mask,
//                   projection, viscous term and RK4 update, and the x
//                   backward transforms of the next stage's input: u,v,w and
//                   d/dx of v,w
// The first stage of a dns_step call is preceded by X's backward half alone
// (from the stored state), its last step's last X ends with the update.
// The vorticity is assembled from spectral derivatives taken on the axis a
// pass owns (x in X, y in B, z in C), so B and D work on one field per tile
// and need no cross-field staging.  N only enters the update through the 2/3
// rule (main.c:381-386), so C, D and X move only those modes of it.
#pragma once
#include "fft_core.cuh"

namespace dnsb {

// work slots of the stage (after pass B, SOMZ holds omega_z = dv/dx - du/dy;
// after the x pass it holds dv/dx).  The z pass writes N = u x omega over the
// slots SNX, SNY, SNZ (those of u, v and dw/dy), each once the line's input
// in it has been read, and D and X take N from there.
enum { SU = 0, SV = 1, SDWDY = 2, SOMZ = 3, SDWDX = 4, SW = 5, NWORK = 6 };
enum { SNX = 0, SNY = 1, SNZ = 2 };

// Loads that leave no line in L1: where shared memory leaves little of it, the
// lines reserved for loads in flight bound how many there are.
template <class C>
__device__ __forceinline__ C ldcg(const C *p) {
  return __ldcg(p);
}
// 16-byte asynchronous copy from global to shared memory, past L1
__device__ __forceinline__ void copy16(void *dst, const void *src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}

struct Geo {
  int n, nf, nfp;
  int kcut;              // 2/3 rule: a wavenumber is kept iff |k| <= kcut
  // RK stage inputs are stored inside the 2/3 rule only, packed as
  // [stage][field][mk: kx][mk: ky][mp: kz] with mk = 2 kcut + 1 rows (index
  // k for k >= 0, mk + k for k < 0) of pitch mp
  int mk, mp;
  long long slotc;       // mk * mk * mp: complex elements per packed field
  long long slot;        // complex elements per spectral slot (n*n*nfp)
  long long nreal;       // n^3
  long long run_spec;    // complex elements between two runs' slot sets
  long long run_real;    // real elements between two runs' stale velocities
};

// A column pass processes tiles of W adjacent kz columns x the full line
// along x or y.  block.z = job + njobs * run: each job maps an input slot to
// an output slot and optionally the derivative i*k*f (k along the pass axis)
// to a der slot, in every run of the batch; with an add slot the derivative
// output is add - i*k*f instead (the same tile of another slot).  A masked
// pass (the y forward pass of N, whose result only enters the update inside
// the 2/3 rule, main.c:381-386) is launched on the column tiles that hold
// kz <= kcut only and stores only |ky| <= kcut.
struct ColJobs {  // der_slot and add_slot: y only
  int in_slot[8];
  int out_slot[8];   // -1: no plain output
  int der_slot[8];   // -1: no derivative output
  int add_slot[8];   // -1: none
  int njobs;
  int masked;
};

// column tile width: 128-byte tile rows (wider rows for the x passes, whose
// rows lie a kx plane apart, measured slower: fewer, heavier blocks), capped
// so that a block stays within 1024 threads
template <class R, int AXIS, int N>
struct ColW {
  static constexpr int WB = 128 / (int)sizeof(cx<R>);
  static constexpr int WT = 1024 / (N / Plan<N>::E);
  static constexpr int W = WB < WT ? WB : WT;
};
// row pitch granularity (128 bytes): every tile width divides it
template <class R>
struct PitchW {
  static constexpr int W = 128 / (int)sizeof(cx<R>);
};

template <int W>
struct ColIdx {
  int p;
  __device__ __forceinline__ int operator()(int pos) const { return pos * W + p; }
};
struct BlockSync {
  __device__ __forceinline__ void operator()() const { __syncthreads(); }
};
// barrier of a sub-block of `count` threads (a multiple of 32) with its own
// hardware barrier id (1..15): several work items share one block of the
// persistent ensemble kernel
struct NamedSync {
  int id, count;
  __device__ __forceinline__ void operator()() const {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(count) : "memory");
  }
};
// coordinates of one work item: the launch's blockIdx / threadIdx in the
// standalone kernels, a virtual block of the persistent ensemble kernel
struct Blk {
  int x, y, z;  // block index
  int tid;      // thread index within the item
  int nt;       // threads of the item
};
__device__ __forceinline__ Blk launch_blk() {
  return Blk{(int)blockIdx.x, (int)blockIdx.y, (int)blockIdx.z, (int)threadIdx.x, (int)blockDim.x};
}
struct WarpSync {
  __device__ __forceinline__ void operator()() const { __syncwarp(); }
};
// per-line exchange buffer with one pad element per 2^SH to spread banks
template <int SH>
struct PadShift {
  __device__ __forceinline__ int operator()(int pos) const { return pos + (pos >> SH); }
};
// exchange barrier of one line: the block's barrier when a line spans
// several warps, else the warp's
template <bool BLOCK, class BSync = BlockSync>
struct LineSync {
  BSync bsync{};
  __device__ __forceinline__ void operator()() const {
    if (BLOCK) bsync(); else __syncwarp();
  }
};

// ---------------------------------------------------------------------------
// Column pass along x (AXIS 0) or y (AXIS 1), forward or backward.
// grid: (nfp / W, n, njobs * nruns); block: (N / E) * W threads
// (W = ColW<R, AXIS, N>::W).
// ---------------------------------------------------------------------------
template <class R, int N, int AXIS, bool FWD, class Sync>
__device__ __forceinline__ void colpass_body(const cx<R> *__restrict__ in, cx<R> *__restrict__ out,
                                             const cx<R> *__restrict__ twg, const Geo &g,
                                             const ColJobs &jobs, const Blk b, Sync sync,
                                             unsigned char *smem) {
  using C = cx<R>;
  constexpr int W = ColW<R, AXIS, N>::W;
  constexpr int E = Plan<N>::E, T = N / E;
  C *st = (C *)smem;  // stage twiddles (<= N entries)
  C *xb = st + N;
  build_stage_tw<N, Plan<N>>(st, twg, N, b.tid, b.nt);
  sync();
  const int p = b.tid % W, t = b.tid / W;
  const int col = b.x * W + p;
  const bool ok = col < g.nf;
  const int fixed = b.y;  // j for the x pass, i for the y pass
  const int job = b.z % jobs.njobs;
  const long long rb = (long long)(b.z / jobs.njobs) * g.run_spec;
  in += rb;
  out += rb;
  long long base, rs;
  if (AXIS == 0) {
    base = (long long)fixed * g.nfp + col;
    rs = (long long)N * g.nfp;
  } else {
    base = (long long)fixed * N * g.nfp + col;
    rs = g.nfp;
  }
  const C *src = in + (long long)jobs.in_slot[job] * g.slot + base;
  // derivatives are taken along y only (the x pass of a step forms its own)
  const int oslot = jobs.out_slot[job], dslot = AXIS == 1 ? jobs.der_slot[job] : -1,
            aslot = jobs.add_slot[job];
  C v[E];
  // the input is read twice (the second read is an L2 hit) rather than kept
  // in a second register array: first for the derivative i k f, then for the
  // plain transform, which may overwrite the input in place
#pragma unroll
  for (int pass = 0; pass < 2; pass++) {
    const int dst_slot = pass == 0 ? dslot : oslot;
    if (dst_slot < 0) continue;
#pragma unroll
    for (int e = 0; e < E; e++) v[e] = ok ? src[(t + T * e) * rs] : czero<C>();
    if (pass == 0 && aslot < 0) {
#pragma unroll
      for (int e = 0; e < E; e++) {
        const R k = (R)kwave(t + T * e, N);
        v[e] = cmk<C>(mul_rn(-k, v[e].y), mul_rn(k, v[e].x));  // i k f
      }
    } else if (pass == 0) {
      const C *add = in + (long long)aslot * g.slot + base;
#pragma unroll
      for (int e = 0; e < E; e++) {
        const R k = (R)kwave(t + T * e, N);
        const C a = ok ? add[(t + T * e) * rs] : czero<C>();
        v[e] = cmk<C>(fma_rn(k, v[e].y, a.x), fma_rn(-k, v[e].x, a.y));  // add - i k f
      }
    }
    line_fft<N, Plan<N>, FWD>(v, t, st, xb, ColIdx<W>{p}, sync);
    if (ok) {
      C *dst = out + (long long)dst_slot * g.slot + base;
#pragma unroll
      for (int e = 0; e < E; e++) {
        const int k = kwave(t + T * e, N);
        if (!jobs.masked || (k < 0 ? -k : k) <= g.kcut) dst[(t + T * e) * rs] = v[e];
      }
    }
  }
}

template <class R, int N, int AXIS, bool FWD>
__global__ void __launch_bounds__((N / Plan<N>::E) * ColW<R, AXIS, N>::W)
    k_colpass(const cx<R> *__restrict__ in, cx<R> *__restrict__ out,
              const cx<R> *__restrict__ twg, Geo g, ColJobs jobs) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  colpass_body<R, N, AXIS, FWD>(in, out, twg, g, jobs, launch_blk(), BlockSync{}, smem_raw);
}

// The same pass with its registers held so that MINB blocks fit per SM (a
// register schedule the autotuner may pick).
template <class R, int N, int AXIS, bool FWD, int MINB>
__global__ void __launch_bounds__((N / Plan<N>::E) * ColW<R, AXIS, N>::W, MINB)
    k_colpass_minb(const cx<R> *__restrict__ in, cx<R> *__restrict__ out,
                   const cx<R> *__restrict__ twg, Geo g, ColJobs jobs) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  colpass_body<R, N, AXIS, FWD>(in, out, twg, g, jobs, launch_blk(), BlockSync{}, smem_raw);
}

// Register-schedule candidates of a column-pass tile of THREADS threads
// with complex values of CB bytes: a minimum of m[i] resident blocks per SM
// (0: the compiler's register choice; otherwise register caps of about 170,
// 128, 102, 85, 64; FP64 tiles stop at 80: at 64 they spill a kilobyte per
// thread).
// DNSB_COL_MINB lists every m > 0, for the declarations of instances.cuh: a
// candidate missing from it would be compiled again in each unit that uses it.
#define DNSB_COL_MINB(X, ...)                                                        \
  X(__VA_ARGS__, 1) X(__VA_ARGS__, 2) X(__VA_ARGS__, 3) X(__VA_ARGS__, 4) X(__VA_ARGS__, 5) \
  X(__VA_ARGS__, 6) X(__VA_ARGS__, 8) X(__VA_ARGS__, 10) X(__VA_ARGS__, 12)
constexpr bool col_minb_listed(int m) {
#define DNSB_COL_IS(M, V) || M == V
  return false DNSB_COL_MINB(DNSB_COL_IS, m);
#undef DNSB_COL_IS
}
template <int THREADS, int CB>
struct ColCands {
  static constexpr int n = 1;
  static constexpr int m[1] = {0};
};
template <>
struct ColCands<64, 16> {
  static constexpr int n = 5;
  static constexpr int m[5] = {0, 6, 8, 10, 12};
};
template <>
struct ColCands<128, 16> {
  static constexpr int n = 5;
  static constexpr int m[5] = {0, 3, 4, 5, 6};
};
template <>
struct ColCands<256, 16> {
  static constexpr int n = 3;
  static constexpr int m[3] = {0, 2, 3};
};
template <>
struct ColCands<128, 8> {
  static constexpr int n = 6;
  static constexpr int m[6] = {0, 3, 4, 5, 6, 8};
};
template <>
struct ColCands<256, 8> {
  static constexpr int n = 4;
  static constexpr int m[4] = {0, 2, 3, 4};
};
template <>
struct ColCands<512, 8> {
  static constexpr int n = 3;
  static constexpr int m[3] = {0, 1, 2};
};

// ---------------------------------------------------------------------------
// Real transforms of single z lines (initial r2c, dump c2r) through a
// half-length complex FFT: TZ = M / E threads per line (M = N/2).
// ---------------------------------------------------------------------------
template <int N>
struct ZCfg {
  static constexpr int M = N / 2;
  static constexpr int E = ZPlan<M>::E;
  static constexpr int TZ = M / E;
  static constexpr int THREADS = (N * N * TZ) < 256 ? (N * N * TZ) : 256;
  static constexpr int LINES = THREADS / TZ;   // lines per block
  static constexpr int XB = M + M / 8;         // padded exchange buffer per line
};

// Partner exchange for the real-transform pre/post-processing: the value at
// position M - k for every k = t + TZ*e held by this thread.  For t > 0 it
// sits in lane (TZ - t) of the same line, register E-1-e; for t == 0 it is
// this thread's register E-e, or `m_val` (position M) for e == 0.
template <int E, int TZ, class C>
__device__ __forceinline__ void partners(const C (&v)[E], C (&pp)[E], int t, int lane0, C m_val) {
  const int src = lane0 + ((TZ - t) & (TZ - 1));
#pragma unroll
  for (int e = 0; e < E; e++) {
    C s;
    s.x = __shfl_sync(0xffffffffu, v[E - 1 - e].x, src);
    s.y = __shfl_sync(0xffffffffu, v[E - 1 - e].y, src);
    if (t == 0) s = (e == 0) ? m_val : v[(E - e) % E];
    pp[e] = s;
  }
}

// c2r of one z line: in: X[k] at k = t + TZ*e, X[M] in xm (lane t == 0);
// out: z[m] = (x[2m], x[2m+1]) at m = t + TZ*e, unnormalised like FFTW.
// The imaginary parts of X[0] and X[M] are ignored (FFTW c2r semantics).
template <int N, class C>
__device__ __forceinline__ void c2r_line(C (&v)[ZCfg<N>::E], C xm, int t, int lane0, const C *tw,
                                         const C *st, C *xb) {
  using Z = ZCfg<N>;
  constexpr int E = Z::E, TZ = Z::TZ;
  if (t == 0) {
    v[0].y = 0;
    xm.y = 0;
  }
  C pp[E];
  partners<E, TZ>(v, pp, t, lane0, xm);
#pragma unroll
  for (int e = 0; e < E; e++) {
    const int k = t + TZ * e;
    const C a = cmk<C>(v[e].x + pp[e].x, v[e].y - pp[e].y);  // X + conj P
    const C b = cmk<C>(v[e].x - pp[e].x, v[e].y + pp[e].y);  // X - conj P
    const C c = cmulc(b, tw[k]);                             // W^{-k} b
    v[e] = cmk<C>(a.x - c.y, a.y + c.x);                     // a + i c
  }
  line_fft<Z::M, ZPlan<Z::M>, false>(v, t, st, xb, PadShift<3>{}, WarpSync{});
}

// r2c of one z line: in: z[m] = (x[2m], x[2m+1]) at m = t + TZ*e;
// out: X[k] at k = t + TZ*e, and X[M] returned in xm (valid in lane t == 0).
template <int N, class C>
__device__ __forceinline__ void r2c_line(C (&v)[ZCfg<N>::E], C &xm, int t, int lane0, const C *tw,
                                         const C *st, C *xb) {
  using Z = ZCfg<N>;
  using S = sc<C>;
  constexpr int E = Z::E, TZ = Z::TZ;
  line_fft<Z::M, ZPlan<Z::M>, true>(v, t, st, xb, PadShift<3>{}, WarpSync{});
  C pp[E];
  partners<E, TZ>(v, pp, t, lane0, v[0]);
  xm = cmk<C>(v[0].x - v[0].y, S(0));
#pragma unroll
  for (int e = 0; e < E; e++) {
    const int k = t + TZ * e;
    const C ev = cmk<C>(S(0.5) * (v[e].x + pp[e].x), S(0.5) * (v[e].y - pp[e].y));
    const C dv = cmk<C>(S(0.5) * (v[e].x - pp[e].x), S(0.5) * (v[e].y + pp[e].y));
    const C q = cmul(tw[k], dv);
    v[e] = cmk<C>(ev.x + q.y, ev.y - q.x);  // ev - i q
  }
}

// z r2c of real slots (initial transform, main.c:249-251): real slot f ->
// work slot f.  grid: (N*N / LINES, nfields)
template <class R, int N>
__global__ void __launch_bounds__(ZCfg<N>::THREADS)
    k_zr2c(const R *__restrict__ real, cx<R> *__restrict__ work, const cx<R> *__restrict__ twg,
           Geo g) {
  using C = cx<R>;
  using Z = ZCfg<N>;
  constexpr int E = Z::E, TZ = Z::TZ;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C *tw = (C *)smem_raw;  // full table exp(-2 pi i k / N): pre/post twiddles
  C *st = tw + N;         // stage twiddles of ZPlan<N/2>
  for (int k = threadIdx.x; k < N; k += blockDim.x) tw[k] = twg[k];
  build_stage_tw<N / 2, ZPlan<N / 2>>(st, twg, N, threadIdx.x, blockDim.x);
  __syncthreads();
  const int lid = threadIdx.x / TZ, t = threadIdx.x % TZ;
  const int lane0 = (threadIdx.x & 31) - t;
  C *xb = tw + 2 * N + lid * Z::XB;
  const long long line = (long long)blockIdx.x * Z::LINES + lid;
  const bool ok = line < (long long)N * N;
  const R *s = real + blockIdx.y * g.nreal + line * N;
  C v[E], xm;
#pragma unroll
  for (int e = 0; e < E; e++) {
    const int m = t + TZ * e;
    v[e] = ok ? cmk<C>(s[2 * m], s[2 * m + 1]) : czero<C>();
  }
  r2c_line<N>(v, xm, t, lane0, tw, st, xb);
  if (ok) {
    C *d = work + blockIdx.y * g.slot + line * g.nfp;
#pragma unroll
    for (int e = 0; e < E; e++) d[t + TZ * e] = v[e];
    if (t == 0) d[Z::M] = xm;
  }
}

// z c2r of work slots into float64 real slots scaled by `scale` (dump,
// main.c:274-277; fields handed to the host are always float64)
template <class R, int N>
__global__ void __launch_bounds__(ZCfg<N>::THREADS)
    k_zc2r(const cx<R> *__restrict__ work, double *__restrict__ real,
           const cx<R> *__restrict__ twg, Geo g, double scale) {
  using C = cx<R>;
  using Z = ZCfg<N>;
  constexpr int E = Z::E, TZ = Z::TZ;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C *tw = (C *)smem_raw;
  C *st = tw + N;
  for (int k = threadIdx.x; k < N; k += blockDim.x) tw[k] = twg[k];
  build_stage_tw<N / 2, ZPlan<N / 2>>(st, twg, N, threadIdx.x, blockDim.x);
  __syncthreads();
  const int lid = threadIdx.x / TZ, t = threadIdx.x % TZ;
  const int lane0 = (threadIdx.x & 31) - t;
  C *xb = tw + 2 * N + lid * Z::XB;
  const long long line = (long long)blockIdx.x * Z::LINES + lid;
  const bool ok = line < (long long)N * N;
  const C *src = work + blockIdx.y * g.slot + line * g.nfp;
  C v[E];
#pragma unroll
  for (int e = 0; e < E; e++) v[e] = ok ? src[t + TZ * e] : czero<C>();
  C xm = (ok && t == 0) ? src[Z::M] : czero<C>();
  c2r_line<N>(v, xm, t, lane0, tw, st, xb);
  if (ok) {
    double *d = real + blockIdx.y * g.nreal + line * N;
#pragma unroll
    for (int e = 0; e < E; e++) {
      const int m = t + TZ * e;
      *(double2 *)(d + 2 * m) = make_double2((double)v[e].x * scale, (double)v[e].y * scale);
    }
  }
}

// ---------------------------------------------------------------------------
// Pass C: per z line, build omega, c2r u and omega, N = u x omega, r2c N.
//
// Each real transform pair runs as ONE complex N-point FFT ("two for one"):
//   c2r: Y[k] = A_ext[k] + i B_ext[k] with the Hermitian extension
//        X_ext[k] = X[k] (k <= N/2), conj(X[N-k]) (k > N/2) and the
//        imaginary parts of X[0], X[N/2] dropped (FFTW c2r semantics, the
//        z axis being the last, real one); Re y = a, Im y = b.
//   r2c: Y = a + i b; X_a[k] = (Z[k] + conj Z[N-k]) / 2,
//        X_b[k] = -i (Z[k] - conj Z[N-k]) / 2.
// T = N/E threads per line hold E points each.  The pairs (u, omega_y), (v,
// omega_x), (w, omega_z) read each input slot once; what of them waits for the
// products is in registers or, in FP64 with 16 values per thread, in shared
// memory (ZC; each thread only reads back its own points).  The first stage
// transforms the vorticity alone, (omega_x, omega_y) and (omega_z, 0).
// KIND 0: first stage, velocity from the stale real slots (main.c:344 skips
//         the back transform at rk == 0); KIND 1: middle stage;
// KIND 2: last stage, also stores the real velocity as the next stale one.
// ---------------------------------------------------------------------------
// The z pass runs the column plans: up to 16 values per thread, one exchange
// fewer per FFT than 8 values at n = 128, 256.
template <class R, int N, int KIND>
struct ZC {
  using P = Plan<N>;
  static constexpr int E = P::E;
  static constexpr int T = N / E;                 // threads per line
  static constexpr int M = N / 2;
  // The pairs run in the order (u, omega_y), (v, omega_x), (w, omega_z), so
  // that N_z is complete after the second and goes through its forward FFT
  // and out before the third; N_x and N_y are then formed in place in the FFT
  // registers.  At most two fields beyond the FFT's own values are live: FP64
  // with 16 values per thread (S2) keeps (u, omega_y) in shared memory and
  // (v, omega_x) in registers (128-thread blocks of 8 lines, 2 per SM, which
  // build the stage twiddles once for 8 lines: 1-10 % faster than 64-thread
  // blocks at 4 per SM; capping the registers for more blocks measured
  // slower); with 8 values, and in FP32, both pairs are in registers (128 of
  // them; FP32 512^3 in 256-thread blocks at 2 per SM, 10 % faster there than
  // 128-thread blocks at 4, 1 % slower at 256^3).  The first stage reads the
  // stale velocity where it needs it.
  static constexpr bool S2 = sizeof(R) == 8 && E >= 16;
  static constexpr bool F32 = sizeof(R) == 4;
  static constexpr int WANT = (F32 && N > 256) ? 256 : 128;
  static constexpr int THREADS = (N * N * T) < WANT ? (N * N * T) : WANT;
  static constexpr int LINES = THREADS / T;
  static constexpr int MINB = S2 ? 2 : (F32 && N > 256) ? 2 : 4;  // blocks per SM
  static constexpr int PADSH = (E >= 16) ? 4 : 3;
  static constexpr int XB = N + (N >> PADSH);     // padded exchange buffer (complex)
  // stage twiddle entries held (even, so the exchange buffers stay 16-byte
  // aligned)
  static constexpr int TWN = (StageTw<P>::SIZE + 1) / 2 * 2 > 2 ? (StageTw<P>::SIZE + 1) / 2 * 2 : 2;
  // staged scalars per line: S2 none (first stage) or (u, omega_y)
  static constexpr int STASH = S2 && KIND != 0 ? 2 * N : 0;
  static constexpr size_t SMEM =
      (size_t)(TWN + LINES * XB) * sizeof(cx<R>) + (size_t)LINES * STASH * sizeof(R);
};

// Hermitian-extended pair  Y[k] = A_ext[k] + i B_ext[k]  at k = t + T*e.
// Loads are issued in chunks of CH positions (an empty asm with a memory
// clobber keeps the compiler from hoisting all of them), which bounds the
// registers held by loads in flight.
template <class R, int N, int KIND, int CH = 4, class C, class FA, class FB>
__device__ __forceinline__ void ext_pair(C (&y)[ZC<R, N, KIND>::E], int t, FA fa, FB fb) {
  using Z = ZC<R, N, KIND>;
#pragma unroll
  for (int e0 = 0; e0 < Z::E; e0 += CH) {
#pragma unroll
    for (int e = e0; e < e0 + CH && e < Z::E; e++) {
      const int k = t + Z::T * e;
      const bool direct = k <= Z::M;
      const int s = direct ? k : N - k;
      C a = fa(s), b = fb(s);
      if (s == 0 || s == Z::M) {
        a.y = 0;
        b.y = 0;
      }
      if (!direct) {
        a.y = -a.y;
        b.y = -b.y;
      }
      y[e] = cmk<C>(a.x - b.y, a.y + b.x);
    }
    asm volatile("" ::: "memory");
  }
}

// Same, with one functor giving both spectra at a position, so that a field
// feeding both halves (u for u and omega_y) is loaded once.
template <class R, int N, int KIND, int CH = 4, class C, class FAB>
__device__ __forceinline__ void ext_gen(C (&y)[ZC<R, N, KIND>::E], int t, FAB fab) {
  using Z = ZC<R, N, KIND>;
#pragma unroll
  for (int e0 = 0; e0 < Z::E; e0 += CH) {
#pragma unroll
    for (int e = e0; e < e0 + CH && e < Z::E; e++) {
      const int k = t + Z::T * e;
      const bool direct = k <= Z::M;
      const int s = direct ? k : N - k;
      C a, b;
      fab(s, a, b);
      if (s == 0 || s == Z::M) {
        a.y = 0;
        b.y = 0;
      }
      if (!direct) {
        a.y = -a.y;
        b.y = -b.y;
      }
      y[e] = cmk<C>(a.x - b.y, a.y + b.x);
    }
    asm volatile("" ::: "memory");
  }
}

// The forward transforms of the z pass for one line (main.c:378-380); only
// kz <= kcut is stored (N enters the update through the 2/3 rule only).
// `row` = the line's row of work slot 0.
// (N_x, N_y) held in y as one complex line: FFT, unpack, store into SNX,
// SNY (ends with a barrier: the exchange buffer is free again)
template <class R, int N, int KIND, class Idx, class Sync>
__device__ __forceinline__ void zfwd_xy(cx<R> (&y)[ZC<R, N, KIND>::E], int t, const cx<R> *tw,
                                        cx<R> *xb, Idx idx, Sync sync, cx<R> *row, const Geo &g,
                                        bool ok) {
  using C = cx<R>;
  using Z = ZC<R, N, KIND>;
  constexpr int E = Z::E, T = Z::T, M = Z::M;
  const int KZ = g.kcut < M ? g.kcut : M;
  line_fft<N, typename Z::P, true>(y, t, tw, xb, idx, sync);
#pragma unroll
  for (int e = 0; e < E; e++) xb[idx(t + T * e)] = y[e];
  sync();
  C *oU = row + SNX * g.slot, *oV = row + SNY * g.slot;
#pragma unroll
  for (int e = 0; e <= E / 2; e++) {
    const int k = t + T * e;
    if (k <= KZ) {
      const C z = y[e], p = xb[idx((N - k) & (N - 1))];
      const C a = cmk<C>(R(0.5) * (z.x + p.x), R(0.5) * (z.y - p.y));  // (Z + conj P) / 2
      const C d = cmk<C>(R(0.5) * (z.x - p.x), R(0.5) * (z.y + p.y));  // (Z - conj P) / 2
      if (ok) {
        oU[k] = a;
        oV[k] = cmk<C>(d.y, -d.x);  // -i d
      }
    }
  }
  sync();
}
// N_z held in y as (N_z, 0): FFT, store into SNZ
template <class R, int N, int KIND, class Idx, class Sync>
__device__ __forceinline__ void zfwd_z(cx<R> (&y)[ZC<R, N, KIND>::E], int t, const cx<R> *tw,
                                       cx<R> *xb, Idx idx, Sync sync, cx<R> *row, const Geo &g,
                                       bool ok) {
  using C = cx<R>;
  using Z = ZC<R, N, KIND>;
  constexpr int E = Z::E, T = Z::T, M = Z::M;
  const int KZ = g.kcut < M ? g.kcut : M;
  line_fft<N, typename Z::P, true>(y, t, tw, xb, idx, sync);
  C *oW = row + SNZ * g.slot;
#pragma unroll
  for (int e = 0; e <= E / 2; e++) {
    const int k = t + T * e;
    if (k <= KZ && ok) oW[k] = y[e];
  }
}
// One block of the z pass: Z::LINES lines starting at line b.x * LINES of
// run b.y (block-wide barriers through `bsync`, which lines of more than 32
// threads also use between FFT stages).  KEEP: also store the real velocity
// and vorticity the pass forms in keep[f][n^3], f = u, v, w, omega_x, omega_y, omega_z of the run (the
// first stage: the vorticity only), for the discrete adjoint.
template <class R, int N, int KIND, bool KEEP = false, class BSync>
__device__ __forceinline__ void zstage_body(cx<R> *__restrict__ work, R *__restrict__ stale,
                                            const cx<R> *__restrict__ twg, const Geo &g, R invn3,
                                            const Blk b, BSync bsync, unsigned char *smem,
                                            R *__restrict__ keep = nullptr) {
  using C = cx<R>;
  using Z = ZC<R, N, KIND>;
  constexpr int E = Z::E, T = Z::T;
  C *tw = (C *)smem;  // stage twiddles of the z plan (Z::TWN entries)
  build_stage_tw<N, typename Z::P>(tw, twg, N, b.tid, b.nt);
  bsync();
  const int lid = b.tid / T, t = b.tid % T;
  C *xb = tw + Z::TWN + lid * Z::XB;
  R *st = (R *)(tw + Z::TWN + Z::LINES * Z::XB) + lid * Z::STASH;
  // own points of staged field f: st[(f * E + e) * T + t]
  auto SU_ = [&](int f, int e) -> R & { return st[(f * E + e) * T + t]; };
  const long long line = (long long)b.x * Z::LINES + lid;
  const bool ok = line < (long long)N * N;
  work += (long long)b.y * g.run_spec;  // run of the batch
  stale += (long long)b.y * g.run_real;
  if constexpr (KEEP) keep += (long long)b.y * 6 * g.nreal;
  const long long off = line * g.nfp;
  const C *pU = work + SU * g.slot + off, *pV = work + SV * g.slot + off;
  const C *pW = work + SW * g.slot + off, *pOMZ = work + SOMZ * g.slot + off;
  const C *pDWDX = work + SDWDX * g.slot + off;
  const C *pDWDY = work + SDWDY * g.slot + off;
  auto ld = [&](const C *p, int s) -> C { return ok ? p[s] : czero<C>(); };
  auto f_ox = [&](int s) -> C {  // omega_x = dw/dy - i kz v
    const C a = ld(pDWDY, s), v = ld(pV, s);
    return cmk<C>(fma_rn((R)s, v.y, a.x), fma_rn(-(R)s, v.x, a.y));
  };
  auto f_oy = [&](int s) -> C {  // omega_y = i kz u - dw/dx
    const C u = ld(pU, s), b = ld(pDWDX, s);
    return cmk<C>(fma_rn(-(R)s, u.y, -b.x), fma_rn((R)s, u.x, -b.y));
  };
  auto f_oz = [&](int s) -> C {  // omega_z = dv/dx - du/dy
    return ld(pOMZ, s);
  };
  auto f_zero = [&](int) -> C { return czero<C>(); };
  // L2 prefetch of a row of `bytes` starting on a 128-byte line: the next
  // pair's inputs are on their way from DRAM while this pair's FFT runs
  // (the waits on those loads were the pass's largest stall)
  auto pf = [&](const void *row, int bytes) {
    if (!ok) return;
    for (int l = t; l * 128 < bytes; l += T)
      asm volatile("prefetch.global.L2 [%0];" ::"l"((const char *)row + l * 128));
  };
  constexpr int ROWB = (N / 2 + 1) * (int)sizeof(C), REALB = N * (int)sizeof(R);
  const LineSync<(T > 32), BSync> sync{bsync};
  const PadShift<Z::PADSH> idx{};
  const long long roff = line * N;
  auto kp = [&](int f, int e, R v) {
    if constexpr (KEEP) {
      if (ok) keep[f * g.nreal + roff + t + T * e] = v;
    }
  };

  C y[E];
  if constexpr (KIND == 0) {
    // first stage: (omega_x, omega_y) with the stale real velocity read
    // where it is needed (L1/L2 hits the second time); N_z is complete
    // after this pair and leaves before (omega_z, 0)
    auto sv = [&](int f, int e) -> R { return ok ? stale[f * g.nreal + roff + t + T * e] : R(0); };
    R nx[E], ny[E];
    ext_pair<R, N, KIND>(y, t, f_ox, f_oy);
    pf(pOMZ, ROWB);
    pf(stale + roff, REALB);
    pf(stale + g.nreal + roff, REALB);
    pf(stale + 2 * g.nreal + roff, REALB);
    line_fft<N, typename Z::P, false>(y, t, tw, xb, idx, sync);
#pragma unroll
    for (int e = 0; e < E; e++) {
      const R ox = y[e].x * invn3, oy = y[e].y * invn3;
      const R u = sv(0, e), v = sv(1, e), w = sv(2, e);
      nx[e] = mul_rn(-w, oy);
      ny[e] = mul_rn(w, ox);
      y[e] = cmk<C>(fma_rn(-v, ox, mul_rn(u, oy)), R(0));  // N_z
      kp(3, e, ox);
      kp(4, e, oy);
    }
    zfwd_z<R, N, KIND>(y, t, tw, xb, idx, sync, work + off, g, ok);
    ext_pair<R, N, KIND>(y, t, f_oz, f_zero);
    line_fft<N, typename Z::P, false>(y, t, tw, xb, idx, sync);
#pragma unroll
    for (int e = 0; e < E; e++) {
      const R oz = y[e].x * invn3;
      y[e] = cmk<C>(fma_rn(sv(1, e), oz, nx[e]), fma_rn(-sv(0, e), oz, ny[e]));  // (N_x, N_y)
      kp(5, e, oz);
    }
    zfwd_xy<R, N, KIND>(y, t, tw, xb, idx, sync, work + off, g, ok);
  } else {
    // middle and last stages: (u, omega_y), (v, omega_x): N_z = u oy - v ox
    // leaves; (w, omega_z): N_x = v oz - w oy, N_y = w ox - u oz formed in
    // place and leave.  The last stage stores the velocity as the next
    // stale one as it comes.
    R su[Z::S2 ? 1 : E], soy[Z::S2 ? 1 : E];  // (u, omega_y) in registers
    ext_gen<R, N, KIND>(y, t, [&](int s, C &a, C &b) {
      const C uu = ld(pU, s), d = ld(pDWDX, s);
      a = uu;
      b = cmk<C>(fma_rn(-(R)s, uu.y, -d.x), fma_rn((R)s, uu.x, -d.y));  // i kz u - dw/dx
    });
    pf(pV, ROWB);
    pf(pDWDY, ROWB);
    line_fft<N, typename Z::P, false>(y, t, tw, xb, idx, sync);
#pragma unroll
    for (int e = 0; e < E; e++) {
      const R u = y[e].x * invn3, oy = y[e].y * invn3;
      if constexpr (Z::S2) {
        SU_(0, e) = u;
        SU_(1, e) = oy;
      } else {
        su[e] = u;
        soy[e] = oy;
      }
      if (KIND == 2 && ok) stale[roff + t + T * e] = u;
      kp(0, e, u);
      kp(4, e, oy);
    }
    auto U_ = [&](int e) -> R { if constexpr (Z::S2) return SU_(0, e); else return su[e]; };
    auto OY_ = [&](int e) -> R { if constexpr (Z::S2) return SU_(1, e); else return soy[e]; };
    ext_gen<R, N, KIND>(y, t, [&](int s, C &a, C &b) {
      const C vv = ld(pV, s), d = ld(pDWDY, s);
      a = vv;
      b = cmk<C>(fma_rn((R)s, vv.y, d.x), fma_rn(-(R)s, vv.x, d.y));  // dw/dy - i kz v
    });
    pf(pW, ROWB);
    pf(pOMZ, ROWB);
    line_fft<N, typename Z::P, false>(y, t, tw, xb, idx, sync);
    R sv_[E], sox[E];
#pragma unroll
    for (int e = 0; e < E; e++) {
      const R v = y[e].x * invn3, ox = y[e].y * invn3;
      sv_[e] = v;
      sox[e] = ox;
      y[e] = cmk<C>(fma_rn(-v, ox, mul_rn(U_(e), OY_(e))), R(0));  // N_z
      if (KIND == 2 && ok) stale[g.nreal + roff + t + T * e] = v;
      kp(1, e, v);
      kp(3, e, ox);
    }
    zfwd_z<R, N, KIND>(y, t, tw, xb, idx, sync, work + off, g, ok);
    ext_gen<R, N, KIND>(y, t, [&](int s, C &a, C &b) {
      a = ld(pW, s);
      b = ld(pOMZ, s);
    });
    line_fft<N, typename Z::P, false>(y, t, tw, xb, idx, sync);
#pragma unroll
    for (int e = 0; e < E; e++) {
      const R w = y[e].x * invn3, oz = y[e].y * invn3;
      const R nx = mul_rn(-w, OY_(e)), ny = mul_rn(-U_(e), oz);
      y[e] = cmk<C>(fma_rn(sv_[e], oz, nx), fma_rn(w, sox[e], ny));  // (N_x, N_y)
      if (KIND == 2 && ok) stale[2 * g.nreal + roff + t + T * e] = w;
      kp(2, e, w);
      kp(5, e, oz);
    }
    zfwd_xy<R, N, KIND>(y, t, tw, xb, idx, sync, work + off, g, ok);
  }
}

template <class R, int N, int KIND>
__global__ void __launch_bounds__(ZC<R, N, KIND>::THREADS, ZC<R, N, KIND>::MINB)
    k_zstage(cx<R> *__restrict__ work, R *__restrict__ stale, const cx<R> *__restrict__ twg, Geo g,
             R invn3) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  zstage_body<R, N, KIND>(work, stale, twg, g, invn3, launch_blk(), BlockSync{}, smem_raw);
}

// The z pass that also keeps the real velocity and vorticity (KEEP above),
// for the forward recomputation of the discrete adjoint.
template <class R, int N, int KIND>
__global__ void __launch_bounds__(ZC<R, N, KIND>::THREADS, ZC<R, N, KIND>::MINB)
    k_zstage_keep(cx<R> *__restrict__ work, R *__restrict__ stale, const cx<R> *__restrict__ twg,
                  Geo g, R invn3, R *__restrict__ keep) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  zstage_body<R, N, KIND, true>(work, stale, twg, g, invn3, launch_blk(), BlockSync{}, smem_raw,
                                keep);
}

// ---------------------------------------------------------------------------
// YZ: for n <= 64 a whole x plane (six fields, ky or y by kz) fits the shared
// memory of one SM (FP64 n = 64: 217 KB), so the y backward pass, the z pass
// and the y forward pass of a plane (B, C and D above) run as one kernel:
// 6.3 slots of traffic a stage instead of 22.3, and two launches fewer.
//
// The plane is held as three pairs of fields, (u, dw/dx), (v, dw/dy) and
// (w, omega_z), a row of a pair being RP complex values: the first field's
// kz = 0..n/2 from 0, the second's from HP on.  A row of a pair is exactly the
// exchange buffer of that pair's z transforms (the pair of fields that the
// two-for-one FFT takes), and a column of a field that of its y transforms,
// so no transform needs other shared memory.  Every transform runs inside
// one warp; the block meets twice, between the axes.  The arithmetic is that
// of colpass_body and zstage_body, bit for bit.
//
// Step of n = 16 FP64 0.117 -> 0.047 ms, n = 32 0.086 -> 0.058; 32 runs of
// 64^3 in FP32 1.67 -> 1.06 ms (the x pass alone had brought 1.40).  At n = 64 it is
// bound by the shared-memory pipe of the SMs that have a plane: some 2.4 MB a
// plane in FP64.
// ---------------------------------------------------------------------------
template <class R, int N>
struct YZ {
  using P = Plan<N>;
  static constexpr int E = P::E, T = N / E, NF = N / 2 + 1, M = N / 2;
  static constexpr int PW = 32 / T;  // columns of a warp in the y passes
  static constexpr int PADSH = E >= 16 ? 4 : 3;
  // half a row, even so that pairs of FP32 columns stay 16-byte aligned
  static constexpr int HP = ((N + (N >> PADSH)) / 2 > NF ? (N + (N >> PADSH)) / 2 : NF + 1) / 2 * 2;
  static constexpr int RP = 2 * HP;
  static constexpr int TWN = StageTw<P>::SIZE / 2 * 2 + 2;
  static constexpr size_t SMEM = (size_t)(TWN + 3 * N * RP) * sizeof(cx<R>);
  static constexpr int THREADS = N == 64 ? (sizeof(R) == 8 ? 512 : 256) : N == 32 ? 256 : 128;
  static constexpr int MINB = N == 64 ? (sizeof(R) == 8 ? 1 : 2) : 1;
  static constexpr int LINES = THREADS / T < N ? THREADS / T : N;  // z lines at a time
  static_assert(T == 1 || LINES * T % 32 == 0, "a warp's lanes have all a line or need no barrier");
  // n = 64: rows are a multiple of 128 bytes (FP64; 64 in FP32) apart, so the
  // four columns of a warp's lanes change places from row to row
  __device__ static __forceinline__ int sw(int row) {
    if (N != 64) return 0;
    return ((sizeof(R) == 8 ? row ^ (row >> 3) : (row >> 1) ^ (row >> 3)) & 1) << 2;
  }
};
template <class R, int N>
struct YZCol {  // position (row) of one column
  int o;
  __device__ __forceinline__ int operator()(int pos) const {
    return pos * YZ<R, N>::RP + (o ^ YZ<R, N>::sw(pos));
  }
};
template <class R, int N>
struct YZRow {  // position in a pair's row
  int s;
  __device__ __forceinline__ int operator()(int pos) const {
    return (pos + (pos >> YZ<R, N>::PADSH)) ^ s;
  }
};

// extension of a pair of spectra to N positions, as in ext_gen
template <class R, int N, class FAB>
__device__ __forceinline__ void yz_ext(cx<R> (&y)[YZ<R, N>::E], int t, FAB fab) {
  using C = cx<R>;
  constexpr int M = N / 2;
#pragma unroll
  for (int e = 0; e < YZ<R, N>::E; e++) {
    const int k = t + YZ<R, N>::T * e;
    const bool direct = k <= M;
    const int s = direct ? k : N - k;
    C a, b;
    fab(s, a, b);
    if (s == 0 || s == M) {
      a.y = 0;
      b.y = 0;
    }
    if (!direct) {
      a.y = -a.y;
      b.y = -b.y;
    }
    y[e] = cmk<C>(a.x - b.y, a.y + b.x);
  }
}

// grid: (n planes, nruns); KIND and KEEP as in the z pass (KEEP: one run, so
// n <= 32, where one run takes this kernel)
template <class R, int N, int KIND, bool KEEP>
__global__ void __launch_bounds__(YZ<R, N>::THREADS, YZ<R, N>::MINB)
    k_yz(cx<R> *__restrict__ work, R *__restrict__ stale, const cx<R> *__restrict__ twg, Geo g,
         R invn3, R *__restrict__ keep) {
  using C = cx<R>;
  using Y = YZ<R, N>;
  using P = typename Y::P;
  constexpr int E = Y::E, T = Y::T, RP = Y::RP, HP = Y::HP, NF = Y::NF, M = Y::M, PW = Y::PW;
  constexpr int WARPS = Y::THREADS / 32;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C *tw = (C *)smem_raw;
  C *pl = tw + Y::TWN;
  build_stage_tw<N, P>(tw, twg, N, threadIdx.x, blockDim.x);
  __syncthreads();
  const int plane = blockIdx.x;
  work += (long long)blockIdx.y * g.run_spec + (long long)plane * N * g.nfp;
  stale += (long long)blockIdx.y * g.run_real + (long long)plane * N * N;
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;

  {  // u, v, w, dv/dx and dw/dx to their places, all on their way at once
    constexpr int V = 16 / (int)sizeof(C), CP = (NF + V - 1) / V;  // columns a copy, copies a row
    for (int q = threadIdx.x; q < N * CP; q += Y::THREADS) {
      const int row = q / CP, col = (q - row * CP) * V, o = row * g.nfp + col;
      C *d = pl + row * RP;
      const int a = col ^ Y::sw(row), b = (HP + col) ^ Y::sw(row);
      copy16(d + a, work + SU * g.slot + o);
      copy16(d + b, work + SDWDX * g.slot + o);
      copy16(d + N * RP + a, work + SV * g.slot + o);
      copy16(d + 2 * N * RP + a, work + SW * g.slot + o);
      copy16(d + 2 * N * RP + b, work + SOMZ * g.slot + o);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  }
  __syncthreads();

  {  // y backward (B), in place
    const int t = lane / PW, p = lane % PW;
    constexpr int TILES = (NF + PW - 1) / PW;
    for (int task = warp; task < 4 * TILES; task += WARPS) {
      const int job = task / TILES;
      // columns past the last repeat it (the same values to the same places)
      const int c0 = (task % TILES) * PW + p, col = c0 < NF ? c0 : NF - 1;
      const YZCol<R, N> lo{col}, hi{HP + col};
      auto get = [&](C (&v)[E], const C *f, const YZCol<R, N> &idx) {
#pragma unroll
        for (int e = 0; e < E; e++) v[e] = f[idx(t + T * e)];
      };
      auto fft = [&](C (&v)[E], C *f, const YZCol<R, N> &idx) {
        __syncwarp();  // the column has been read, also by the lanes that repeat it
        line_fft<N, P, false>(v, t, tw, f, idx, WarpSync{});
#pragma unroll
        for (int e = 0; e < E; e++) f[idx(t + T * e)] = v[e];
      };
      C *f0 = pl, *f1 = pl + N * RP, *f2 = pl + 2 * N * RP;
      C v[E];
      if (job == 0) {  // omega_z = dv/dx - i ky u, and u
        C u[E];
        get(u, f0, lo);
        get(v, f2, hi);
#pragma unroll
        for (int e = 0; e < E; e++) {
          const R k = (R)kwave(t + T * e, N);
          v[e] = cmk<C>(fma_rn(k, u[e].y, v[e].x), fma_rn(-k, u[e].x, v[e].y));
        }
        fft(v, f2, hi);
        fft(u, f0, lo);
      } else if (job == 1) {  // dw/dy = i ky w, and w (not needed in the first stage)
        C w[E];
        get(w, f2, lo);
#pragma unroll
        for (int e = 0; e < E; e++) {
          const R k = (R)kwave(t + T * e, N);
          v[e] = cmk<C>(mul_rn(-k, w[e].y), mul_rn(k, w[e].x));
        }
        fft(v, f1, hi);
        if (KIND != 0) fft(w, f2, lo);
      } else if (job == 2) {
        get(v, f1, lo);
        fft(v, f1, lo);
      } else {
        get(v, f0, hi);
        fft(v, f0, hi);
      }
    }
  }
  __syncthreads();

  const int KZ = g.kcut < M ? g.kcut : M;
  for (int l0 = 0; l0 < N; l0 += Y::LINES) {  // z lines (C)
    const int lid = threadIdx.x / T, t = threadIdx.x % T;
    if (lid >= Y::LINES) break;  // whole warps, or T == 1
    const int line = l0 + lid;
    const YZRow<R, N> idx{Y::sw(line)};
    C *r0 = pl + line * RP, *r1 = r0 + N * RP, *r2 = r1 + N * RP;
    R *st = stale + line * N;
    auto kp = [&](int f, int e, R v) {
      if constexpr (KEEP)
        keep[f * g.nreal + ((long long)plane * N + line) * N + t + T * e] = v;
    };
    auto at = [&](const C *r, int o) -> C { return r[o ^ idx.s]; };
    auto fft_inv = [&](C (&y)[E], C *r) {
      if (T > 1) __syncwarp();  // the row has been read
      line_fft<N, P, false>(y, t, tw, r, idx, WarpSync{});
    };
    auto fft_fwd = [&](C (&y)[E], C *r) {
      if (T > 1) __syncwarp();
      line_fft<N, P, true>(y, t, tw, r, idx, WarpSync{});
    };
    auto f_ox = [&](int s) -> C {  // omega_x = dw/dy - i kz v
      const C a = at(r1, HP + s), v = at(r1, s);
      return cmk<C>(fma_rn((R)s, v.y, a.x), fma_rn(-(R)s, v.x, a.y));
    };
    auto f_oy = [&](int s) -> C {  // omega_y = i kz u - dw/dx
      const C u = at(r0, s), d = at(r0, HP + s);
      return cmk<C>(fma_rn(-(R)s, u.y, -d.x), fma_rn((R)s, u.x, -d.y));
    };
    auto out_z = [&](const C (&y)[E]) {  // N_z to the first half of pair 0
#pragma unroll
      for (int e = 0; e <= E / 2; e++) {
        const int k = t + T * e;
        if (k <= KZ) r0[k ^ idx.s] = y[e];
      }
    };
    C y[E];
    if constexpr (KIND == 0) {
      R nx[E], ny[E];
      auto sv = [&](int f, int e) -> R { return st[f * g.nreal + t + T * e]; };
      yz_ext<R, N>(y, t, [&](int s, C &a, C &b) {
        a = f_ox(s);
        b = f_oy(s);
      });
      fft_inv(y, r0);
#pragma unroll
      for (int e = 0; e < E; e++) {
        const R ox = y[e].x * invn3, oy = y[e].y * invn3;
        const R u = sv(0, e), v = sv(1, e), w = sv(2, e);
        nx[e] = mul_rn(-w, oy);
        ny[e] = mul_rn(w, ox);
        y[e] = cmk<C>(fma_rn(-v, ox, mul_rn(u, oy)), R(0));  // N_z
        kp(3, e, ox);
        kp(4, e, oy);
      }
      fft_fwd(y, r0);
      out_z(y);
      yz_ext<R, N>(y, t, [&](int s, C &a, C &b) {
        a = at(r2, HP + s);
        b = czero<C>();
      });
      fft_inv(y, r2);
#pragma unroll
      for (int e = 0; e < E; e++) {
        const R oz = y[e].x * invn3;
        y[e] = cmk<C>(fma_rn(sv(1, e), oz, nx[e]), fma_rn(-sv(0, e), oz, ny[e]));
        kp(5, e, oz);
      }
    } else {
      R su[E], soy[E], sv[E], sox[E];
      yz_ext<R, N>(y, t, [&](int s, C &a, C &b) {
        a = at(r0, s);
        b = f_oy(s);
      });
      fft_inv(y, r0);
#pragma unroll
      for (int e = 0; e < E; e++) {
        su[e] = y[e].x * invn3;
        soy[e] = y[e].y * invn3;
        if (KIND == 2) st[t + T * e] = su[e];
        kp(0, e, su[e]);
        kp(4, e, soy[e]);
      }
      yz_ext<R, N>(y, t, [&](int s, C &a, C &b) {
        a = at(r1, s);
        b = f_ox(s);
      });
      fft_inv(y, r1);
#pragma unroll
      for (int e = 0; e < E; e++) {
        const R v = y[e].x * invn3, ox = y[e].y * invn3;
        sv[e] = v;
        sox[e] = ox;
        y[e] = cmk<C>(fma_rn(-v, ox, mul_rn(su[e], soy[e])), R(0));
        if (KIND == 2) st[g.nreal + t + T * e] = v;
        kp(1, e, v);
        kp(3, e, ox);
      }
      fft_fwd(y, r1);
      out_z(y);
      yz_ext<R, N>(y, t, [&](int s, C &a, C &b) {
        a = at(r2, s);
        b = at(r2, HP + s);
      });
      fft_inv(y, r2);
#pragma unroll
      for (int e = 0; e < E; e++) {
        const R w = y[e].x * invn3, oz = y[e].y * invn3;
        y[e] = cmk<C>(fma_rn(sv[e], oz, mul_rn(-w, soy[e])),
                      fma_rn(w, sox[e], mul_rn(-su[e], oz)));
        if (KIND == 2) st[2 * g.nreal + t + T * e] = w;
        kp(2, e, w);
        kp(5, e, oz);
      }
    }
    fft_fwd(y, r2);
#pragma unroll
    for (int e = 0; e < E; e++) r2[idx(t + T * e)] = y[e];
    if (T > 1) __syncwarp();
#pragma unroll
    for (int e = 0; e <= E / 2; e++) {  // N_x, N_y to pair 1
      const int k = t + T * e;
      if (k <= KZ) {
        const C z = y[e], q = r2[idx((N - k) & (N - 1))];
        const C a = cmk<C>(R(0.5) * (z.x + q.x), R(0.5) * (z.y - q.y));
        const C d = cmk<C>(R(0.5) * (z.x - q.x), R(0.5) * (z.y + q.y));
        r1[k ^ idx.s] = a;
        r1[(HP + k) ^ idx.s] = cmk<C>(d.y, -d.x);  // -i d
      }
    }
  }
  __syncthreads();

  {  // y forward (D), inside the 2/3 rule
    const int t = lane / PW, p = lane % PW;
    const int tiles = KZ / PW + 1;
    for (int task = warp; task < 3 * tiles; task += WARPS) {
      const int job = task / tiles;  // N_x, N_y, N_z
      const int c0 = (task % tiles) * PW + p, col = c0 <= KZ ? c0 : KZ;
      C *f = pl + (job == 2 ? 0 : N * RP);
      const YZCol<R, N> idx{(job == 1 ? HP : 0) + col};
      C v[E];
#pragma unroll
      for (int e = 0; e < E; e++) v[e] = f[idx(t + T * e)];
      __syncwarp();
      line_fft<N, P, true>(v, t, tw, f, idx, WarpSync{});
      C *dst = work + (job == 0 ? SNX : job == 1 ? SNY : SNZ) * g.slot + col;
#pragma unroll
      for (int e = 0; e < E; e++) {
        const int k = kwave(t + T * e, N);
        if ((k < 0 ? -k : k) <= g.kcut) dst[(t + T * e) * g.nfp] = v[e];
      }
    }
  }
}

// ---------------------------------------------------------------------------
// X: one block holds the x lines of the three fields over W adjacent kz
// columns at one ky (N / E * W threads) and takes RK stage ST from N to the
// next stage's x-transformed fields:
//   x forward of N (main.c:378-380), inside the 2/3 rule only,
//   dU  = N * dt,  P = kk > 0 ? (dU kx + dV ky + dW kz) / kk : 0
//   dU -= P kx + nu dt kk U_s            (same for V, W; main.c:381-413)
//   ST 0:  U_1 = U_0 + dU / 2     ST 1: U_2 = U_0 + dU / 2
//   ST 2:  U_3 = U_0 + dU
//   ST 3:  U_0' = U_3 + ((U_1 - U_0) + 2 (U_2 - U_0) - 2 (U_3 - U_0)) / 3 + dU / 6
//          (the RK4 sum of main.c:15 written with the stage inputs, which
//          are kept, in place of an accumulator; the bracket is a sum of
//          increments, so it is the roundings at |U| of the stored U_1, U_2
//          and U_3, weighted by 1/3, 2/3 and 1/3, and the last addition's that
//          enter, where an accumulator rounds at |U| four times)
//   x backward of the result: u, v, w and i kx v, i kx w  (TAIL; ST < 0: of
//   the stored state alone)
// Outside the 2/3 rule N is masked to zero, so the stage inputs there are the
// state times a polynomial in c = nu dt kk and are formed from the state where
// they are needed (lin_coef): only the state itself is stored there, by ST 3.
//
// The fields go through the block one after another, each thread owning the
// same points of all three, so that the projection needs no exchange; the
// transformed N of two fields (then the results that wait for their
// transform) are held in shared memory, each thread reading back its own.
//
// One launch reads N (4/9 of 3 slots), the state (3 slots) and the packed
// stage inputs, and writes 5 slots and one packed triple: 11.1 slots in a
// middle stage, where the three kernels it replaces (the x forward pass, the
// update and the next x backward pass) moved 26.1.  Middle stage, one B200,
// before (sum of the three) and now: FP64 n = 128 0.098 -> 0.056 ms, n = 256
// 0.62 -> 0.36 (4.2 TB/s), n = 512 5.24 -> 3.56; FP32 0.070 -> 0.033, 0.345 ->
// 0.194 (3.9 TB/s), 2.76 -> 1.86.  It is bound by the shared-memory pipe (the
// exchanges and the waiting fields) and by the loads in flight.
// ---------------------------------------------------------------------------
template <class R>
struct XArgs {
  cx<R> *u0;    // state (3 slots); ST 3 writes the new state here
  cx<R> *rk;    // packed stage inputs U_1, U_2, U_3 inside the 2/3 rule
  cx<R> *work;  // work slots
  cx<R> *ph;    // pressure slot or nullptr
  const double *coef;  // coef[2 r] = nu, coef[2 r + 1] = dt of run r (device
                       // memory, so a captured graph picks up new values)
};

// Plans of the X pass: 8 values per thread, one exchange more than the
// column plans at n = 128 and 256, for 12 warps of FP64 (168 registers) and
// 24 of FP32 (80) beside the buffers (16 values per thread, n = 256 FP64 at 6
// or 8 warps: middle stage 0.38 ms against 0.36; FP32 0.209 against 0.194).
template <int L>
struct XPlan : Plan<L> {};
template <> struct XPlan<16>  { static constexpr int E = 8, NS = 2, R0 = 8, R1 = 2, R2 = 1, R3 = 1; };
template <> struct XPlan<128> { static constexpr int E = 8, NS = 3, R0 = 8, R1 = 8, R2 = 2, R3 = 1; };
template <> struct XPlan<256> { static constexpr int E = 8, NS = 3, R0 = 8, R1 = 8, R2 = 4, R3 = 1; };
template <> struct XPlan<512> { static constexpr int E = 8, NS = 3, R0 = 8, R1 = 8, R2 = 8, R3 = 1; };

// Tile of the X pass.  Its three buffers (3 N W values) and L1 share the SM's
// 256 KB, and what is left to L1 bounds the loads in flight: more resident
// blocks than these measured slower (FP64 n = 256: 3 blocks of 64-byte rows
// 0.36 ms, 4 blocks 0.42, 2 of 128-byte rows 0.39; FP32 n = 256: 3 blocks of
// 64-byte rows 0.194, 4 blocks 0.25, 2 of 128-byte rows 0.23).  At n = 512 one
// block of 128-byte rows beats two of 64-byte rows (FP64 3.56 against 3.90
// ms, FP32 1.86 against 2.03).
template <class R, int N>
struct XC {
  using P = XPlan<N>;
  static constexpr int W = sizeof(R) == 8 ? (N == 256 ? 4 : 8) : (N == 512 ? 16 : 8);
  static constexpr int E = P::E, T = N / E;
  static constexpr int THREADS = T * W;
  // twiddle entries (even, so the buffers stay 16-byte aligned)
  static constexpr int TWN = (StageTw<P>::SIZE + 2) / 2 * 2;
  // rows shorter than 128 bytes: one row of pad per R0 positions, which the
  // first exchange writes R0 apart
  static constexpr int SH = W * sizeof(cx<R>) >= 128 ? 30 : P::R0 == 16 ? 4 : 3;
  static constexpr int XB = (N + (N >> SH)) * W;  // exchange buffer
  static constexpr size_t SMEM = (size_t)(TWN + XB + 2 * N * W) * sizeof(cx<R>);
  static constexpr int WANT = (sizeof(R) == 8 ? 384 : 768) / THREADS;
  static constexpr int MINB = N <= 32 || WANT < 1 ? 1 : WANT;  // blocks per SM
};
template <int W, int SH>
struct XIdx {
  int p;
  __device__ __forceinline__ int operator()(int pos) const { return (pos + (pos >> SH)) * W + p; }
};

// Outside the 2/3 rule dU = -c U_s with c = nu dt kk: the stage input that
// stage ST forms (ST 3: the new state) is U_0 + m U_0 with this m.
template <int ST, class R>
__device__ __forceinline__ R lin_coef(R c) {
  const R h = R(0.5) * c;
  const R m1 = -h;
  if (ST == 0) return m1;
  const R m2 = mul_rn(-h, R(1) + m1);
  if (ST == 1) return m2;
  const R m3 = mul_rn(-c, R(1) + m2);
  if (ST == 2) return m3;
  return fma_rn(m1 + R(2) * m2 + m3, R(1.0 / 3.0), mul_rn(mul_rn(-c, R(1) + m3), R(1.0 / 6.0)));
}

template <class R, int N, int ST, bool TAIL, class Sync>
__device__ __forceinline__ void xstage_body(const XArgs<R> &a, const cx<R> *__restrict__ twg,
                                            const Geo &g, const Blk b, Sync sync,
                                            unsigned char *smem) {
  using C = cx<R>;
  using X = XC<R, N>;
  using P = typename X::P;
  constexpr int W = X::W, E = X::E, T = X::T, TH = X::THREADS;
  static_assert(ST >= 0 || TAIL, "the plain backward pass has a tail");
  C *st = (C *)smem;
  C *xb = st + X::TWN;
  const int p = b.tid % W, t = b.tid / W;
  // own points of the two fields that wait: s0[e * TH], s1[e * TH]
  C *s0 = xb + X::XB + b.tid, *s1 = s0 + E * TH;
  const int j = b.y, col = b.x * W + p;
  const bool ok = col < g.nf;
  const int iky = kwave(j, N);
  const bool yin = (iky < 0 ? -iky : iky) <= g.kcut;             // same for the block
  const bool hasn = ST >= 0 && yin && (int)(b.x * W) <= g.kcut;  // same for the block
  const bool zin = yin && col <= g.kcut;
  const long long rb = (long long)b.z * g.run_spec;
  const unsigned rs = (unsigned)N * g.nfp;
  const unsigned base = (unsigned)j * g.nfp + col + t * rs;  // of point e = 0
  C *u0 = a.u0 + rb + base;
  C *wk = a.work + rb + base;
  const XIdx<W, X::SH> idx{p};
  // offset of own point e in a slot, relative to `base`
  auto at = [&](int e) -> long long { return (long long)((unsigned)(T * e) * rs); };
  const double nu = ST < 0 ? 0.0 : a.coef[2 * b.z], dt = ST < 0 ? 0.0 : a.coef[2 * b.z + 1];
  const double nudt = nu * dt;
  const int kyz = iky * iky + col * col;
  auto kin = [&](int ik) { return (ik < 0 ? -ik : ik) <= g.kcut; };
  C v[E];

  // The first inputs: one field to registers, the other two on their way to
  // their places in shared memory meanwhile (N, or the state where there is
  // no N).  FP32 copies pairs of columns, the even thread those of s0 and the
  // odd thread those of s1; a pair's second column may lie past the valid
  // ones (in the row's padding, or past kcut) and is not used then.
  const bool first_ok = hasn ? zin : ok;
  const C *f0 = hasn ? wk + SNX * g.slot : u0;
  const C *f1 = hasn ? wk + SNY * g.slot : u0 + g.slot;
  const C *f2 = hasn ? wk + SNZ * g.slot : u0 + 2 * g.slot;
  if constexpr (sizeof(C) == 16) {
    if (first_ok) {
#pragma unroll
      for (int e = 0; e < E; e++) {
        copy16(s0 + e * TH, f1 + at(e));
        copy16(s1 + e * TH, f2 + at(e));
      }
    }
  } else {
    static_assert(W % 2 == 0, "pairs of columns");
    const int odd = p & 1;
    if (odd ? (hasn ? col - 1 <= g.kcut : col - 1 < g.nf) : first_ok) {
      C *d = (odd ? s1 : s0) - odd;
      const C *s = (odd ? f2 : f1) - odd;
#pragma unroll
      for (int e = 0; e < E; e++) copy16(d + e * TH, s + at(e));
    }
  }
#pragma unroll
  for (int e = 0; e < E; e++) v[e] = first_ok ? ldcg(f0 + at(e)) : czero<C>();
  auto copies_done = [&]() {
    asm volatile("cp.async.wait_all;" ::: "memory");
    if (sizeof(C) != 16) __syncwarp();
  };
  auto landed = [&](const C *s, int e) { return first_ok ? s[e * TH] : czero<C>(); };
  build_stage_tw<N, P>(st, twg, N, b.tid, b.nt);
  sync();

  if (!hasn) {
    copies_done();
    if constexpr (ST >= 0) {
#pragma unroll
      for (int e = 0; e < E; e++) {
        const int ik = kwave(t + T * e, N);
        const R m = lin_coef<ST>((R)(nudt * (double)(ik * ik + kyz)));
        const C z1 = landed(s0, e), z2 = landed(s1, e);
        v[e] = cmk<C>(fma_rn(m, v[e].x, v[e].x), fma_rn(m, v[e].y, v[e].y));
        const C r1 = cmk<C>(fma_rn(m, z1.x, z1.x), fma_rn(m, z1.y, z1.y));
        const C r2 = cmk<C>(fma_rn(m, z2.x, z2.x), fma_rn(m, z2.y, z2.y));
        s0[e * TH] = r1;
        s1[e * TH] = r2;
        if (ST == 3 && ok) {
          u0[at(e)] = v[e];
          u0[at(e) + g.slot] = r1;
          u0[at(e) + 2 * g.slot] = r2;
        }
      }
    }
  } else if constexpr (ST >= 0) {
    // packed stage inputs, this thread's column of field 0 of stage 1
    const unsigned crs = (unsigned)g.mk * g.mp;
    C *rk = a.rk + rb + (unsigned)(iky < 0 ? iky + g.mk : iky) * g.mp + col;
    auto crow = [&](int ik) -> long long {
      return (long long)((unsigned)(ik < 0 ? ik + g.mk : ik) * crs);
    };
    // State and stage inputs of a point: DEPTH points are on their way at a
    // time (as far as the compiler knows a store may alias a later load).
    // n <= 32, where latency is all, spends some 170 registers on them; else
    // stage 3's four triples leave none for a second point.
    constexpr int PER = 3 * (ST == 0 ? 1 : ST < 3 ? 2 : 4) * (int)sizeof(C) / 4;
    constexpr int DEPTH = N <= 32 ? (170 / PER < E ? 170 / PER : E) : ST < 3 ? 2 : 1;
    struct In {
      C z[3], us[3], r1[3], r2[3];
    };
    auto load = [&](In &q, int e) {
      const int ik = kwave(t + T * e, N);
      const bool in = zin && kin(ik);
#pragma unroll
      for (int f = 0; f < 3; f++) {
        q.z[f] = ok ? ldcg(u0 + at(e) + f * g.slot) : czero<C>();
        if constexpr (ST > 0)
          q.us[f] = in ? ldcg(rk + crow(ik) + (3 * (ST - 1) + f) * g.slotc) : czero<C>();
        if constexpr (ST == 3) {
          q.r1[f] = in ? ldcg(rk + crow(ik) + f * g.slotc) : czero<C>();
          q.r2[f] = in ? ldcg(rk + crow(ik) + (3 + f) * g.slotc) : czero<C>();
        }
      }
    };
    In in[DEPTH];
    auto load_first = [&]() {
#pragma unroll
      for (int e = 0; e + 1 < DEPTH; e++) load(in[e], e);
    };
    if (N <= 32) load_first();
    line_fft<N, P, true>(v, t, st, xb, idx, sync);
    copies_done();
#pragma unroll
    for (int e = 0; e < E; e++) {  // N_x takes N_y's place
      const C y = landed(s0, e);
      s0[e * TH] = v[e];
      v[e] = y;
    }
    line_fft<N, P, true>(v, t, st, xb, idx, sync);
#pragma unroll
    for (int e = 0; e < E; e++) {
      const C y = landed(s1, e);
      s1[e * TH] = v[e];
      v[e] = y;
    }
    if (N > 32) load_first();
    line_fft<N, P, true>(v, t, st, xb, idx, sync);
    const R dtr = (R)dt, ky = (R)iky, kz = (R)col;
    auto update = [&](const In &q, int e) {
      const int ik = kwave(t + T * e, N);
      const int ikk = ik * ik + kyz;
      const R c = (R)(nudt * (double)ikk);  // formed in FP64, rounded once
      C r[3];
      if (zin && kin(ik)) {
        const R kk = (R)ikk, k[3] = {(R)ik, ky, kz};
        C n[3] = {s0[e * TH], s1[e * TH], v[e]};
#pragma unroll
        for (int f = 0; f < 3; f++) n[f] = cmk<C>(mul_rn(n[f].x, dtr), mul_rn(n[f].y, dtr));
        auto dot = [&](R x, R y, R z) -> R {
          return fma_rn(z, k[2], fma_rn(y, k[1], mul_rn(x, k[0])));
        };
        C pr = czero<C>();
        if (ikk > 0) {
          pr.x = div_rn(dot(n[0].x, n[1].x, n[2].x), kk);
          pr.y = div_rn(dot(n[0].y, n[1].y, n[2].y), kk);
        }
#pragma unroll
        for (int f = 0; f < 3; f++) {
          const C us = ST == 0 ? q.z[f] : q.us[f];
          const C dd = cmk<C>(n[f].x - fma_rn(pr.x, k[f], mul_rn(c, us.x)),
                              n[f].y - fma_rn(pr.y, k[f], mul_rn(c, us.y)));
          if constexpr (ST < 3) {
            constexpr R bs = ST < 2 ? R(0.5) : R(1);
            r[f] = cmk<C>(fma_rn(bs, dd.x, q.z[f].x), fma_rn(bs, dd.y, q.z[f].y));
            rk[crow(ik) + (3 * ST + f) * g.slotc] = r[f];
          } else {
            auto sum = [](R q0, R q1, R q2, R q3, R du) -> R {
              const R inc = (q1 - q0) + R(2) * (q2 - q0) - R(2) * (q3 - q0);
              return fma_rn(inc, R(1.0 / 3.0), fma_rn(du, R(1.0 / 6.0), q3));
            };
            r[f] = cmk<C>(sum(q.z[f].x, q.r1[f].x, q.r2[f].x, us.x, dd.x),
                          sum(q.z[f].y, q.r1[f].y, q.r2[f].y, us.y, dd.y));
          }
        }
        if (ST == 3 && a.ph) a.ph[rb + base + at(e)] = pr;
      } else {
        const R m = lin_coef<ST>(c);
#pragma unroll
        for (int f = 0; f < 3; f++)
          r[f] = cmk<C>(fma_rn(m, q.z[f].x, q.z[f].x), fma_rn(m, q.z[f].y, q.z[f].y));
      }
      if (ST == 3 && ok) {
#pragma unroll
        for (int f = 0; f < 3; f++) u0[at(e) + f * g.slot] = r[f];
      }
      v[e] = r[0];
      s0[e * TH] = r[1];
      s1[e * TH] = r[2];
    };
#pragma unroll
    for (int e = 0; e < E; e++) {
      if (e + DEPTH <= E) load(in[(e + DEPTH - 1) % DEPTH], e + DEPTH - 1);
      update(in[e % DEPTH], e);
    }
  }
  if constexpr (!TAIL) return;

  // x backward of u, and of i kx f and f for f = v, w
  auto back = [&](int slot) {  // transform v into a work slot
    line_fft<N, P, false>(v, t, st, xb, idx, sync);
    if (ok) {
      C *dst = wk + slot * g.slot;
#pragma unroll
      for (int e = 0; e < E; e++) dst[at(e)] = v[e];
    }
  };
  back(SU);
#pragma unroll
  for (int f = 1; f < 3; f++) {
    const C *s = f == 1 ? s0 : s1;
#pragma unroll
    for (int e = 0; e < E; e++) {
      const R k = (R)kwave(t + T * e, N);
      const C z = s[e * TH];
      v[e] = cmk<C>(mul_rn(-k, z.y), mul_rn(k, z.x));  // i kx f
    }
    back(f == 1 ? SOMZ : SDWDX);
#pragma unroll
    for (int e = 0; e < E; e++) v[e] = s[e * TH];
    back(f == 1 ? SV : SW);
  }
}

// grid: (ceil(nf / W), n, nruns); block: XC::THREADS
template <class R, int N, int ST, bool TAIL>
__global__ void __launch_bounds__(XC<R, N>::THREADS, XC<R, N>::MINB)
    k_xstage(XArgs<R> a, const cx<R> *__restrict__ twg, Geo g) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  xstage_body<R, N, ST, TAIL>(a, twg, g, launch_blk(), BlockSync{}, smem_raw);
}

// ---------------------------------------------------------------------------
// Energy / enstrophy (main.c:257-266): sums over the half spectrum of
//   e = |U|^2 + |V|^2 + |W|^2   and   kk * e,
// each term rounded like the reference's double expression (no FMA), summed
// in double-double (error-free TwoSum), block partials then one final block.
// FP32 storage is widened to FP64 first.
// ---------------------------------------------------------------------------
struct DD {
  double hi, lo;
};
__device__ __forceinline__ DD dd_add_d(DD a, double b) {
  const double s = __dadd_rn(a.hi, b);
  const double bb = __dsub_rn(s, a.hi);
  const double err = __dadd_rn(__dsub_rn(a.hi, __dsub_rn(s, bb)), __dsub_rn(b, bb));
  return DD{s, __dadd_rn(a.lo, err)};
}
__device__ __forceinline__ DD dd_add(DD a, DD b) {
  const double s = __dadd_rn(a.hi, b.hi);
  const double bb = __dsub_rn(s, a.hi);
  double err = __dadd_rn(__dsub_rn(a.hi, __dsub_rn(s, bb)), __dsub_rn(b.hi, bb));
  err = __dadd_rn(err, __dadd_rn(a.lo, b.lo));
  const double hi = __dadd_rn(s, err);
  const double lo = __dsub_rn(err, __dsub_rn(hi, s));
  return DD{hi, lo};
}
__device__ __forceinline__ DD dd_shfl_down(DD a, int d) {
  return DD{__shfl_down_sync(0xffffffffu, a.hi, d), __shfl_down_sync(0xffffffffu, a.lo, d)};
}
__device__ __forceinline__ double cabs2_rn(double2 z) {
  return __dadd_rn(__dmul_rn(z.x, z.x), __dmul_rn(z.y, z.y));
}

template <int BS>
__device__ __forceinline__ void dd_block_reduce(DD &e, DD &o, double4 *out) {
  __shared__ DD se[BS / 32], so[BS / 32];
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) {
    e = dd_add(e, dd_shfl_down(e, d));
    o = dd_add(o, dd_shfl_down(o, d));
  }
  const int w = threadIdx.x / 32, l = threadIdx.x % 32;
  if (l == 0) {
    se[w] = e;
    so[w] = o;
  }
  __syncthreads();
  if (w == 0) {
    e = l < BS / 32 ? se[l] : DD{0.0, 0.0};
    o = l < BS / 32 ? so[l] : DD{0.0, 0.0};
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
      e = dd_add(e, dd_shfl_down(e, d));
      o = dd_add(o, dd_shfl_down(o, d));
    }
    if (l == 0) *out = make_double4(e.hi, e.lo, o.hi, o.lo);
  }
}

// grid: (blocks per run, nruns); partials [run][gridDim.x]
template <int BS, class C>
__global__ void __launch_bounds__(BS)
    k_diag(const C *__restrict__ u, Geo g, double4 *__restrict__ partial) {
  u += (long long)blockIdx.y * g.run_spec;
  partial += (long long)blockIdx.y * gridDim.x;
  DD e{0.0, 0.0}, o{0.0, 0.0};
  const int n = g.n;
  const long long npts = (long long)n * n * g.nf;
  for (long long q = (long long)blockIdx.x * BS + threadIdx.x; q < npts;
       q += (long long)gridDim.x * BS) {
    const long long row = q / g.nf;
    const int k = (int)(q - row * g.nf);
    const int i = (int)(row / n), j = (int)(row % n);
    const long long l = row * g.nfp + k;
    const double s = __dadd_rn(__dadd_rn(cabs2_rn(to_d(u[l])), cabs2_rn(to_d(u[g.slot + l]))),
                               cabs2_rn(to_d(u[2 * g.slot + l])));
    const double kx = kwave(i, n), ky = kwave(j, n), kz = k;
    const double kk = __dadd_rn(__dadd_rn(__dmul_rn(kx, kx), __dmul_rn(ky, ky)), __dmul_rn(kz, kz));
    e = dd_add_d(e, s);
    o = dd_add_d(o, __dmul_rn(kk, s));
  }
  dd_block_reduce<BS>(e, o, partial + blockIdx.x);
}

// grid: (nruns); out[run]
template <int BS>
__global__ void __launch_bounds__(BS) k_diag_final(const double4 *__restrict__ partial, int np,
                                                   double4 *__restrict__ out) {
  partial += (long long)blockIdx.x * np;
  out += blockIdx.x;
  DD e{0.0, 0.0}, o{0.0, 0.0};
  for (int q = threadIdx.x; q < np; q += BS) {
    const double4 v = partial[q];
    e = dd_add(e, DD{v.x, v.y});
    o = dd_add(o, DD{v.z, v.w});
  }
  dd_block_reduce<BS>(e, o, out);
}

// ---------------------------------------------------------------------------
// Precision conversions for the FP32 path (host data is always float64).
// ---------------------------------------------------------------------------
template <class A, class B>
__global__ void k_real_convert(const A *__restrict__ in, B *__restrict__ out, long long n) {
  for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < n;
       q += (long long)gridDim.x * blockDim.x)
    out[q] = (B)in[q];
}
// spectral: nfields padded slots (type C, pitch nfp) <-> unpadded double2
// [nfields][n][n][nf]; TO_PADDED selects the direction
template <class C, bool TO_PADDED>
__global__ void k_spec_convert(C *__restrict__ padded, double2 *__restrict__ dense, Geo g,
                               int nfields) {
  const long long per = (long long)g.n * g.n * g.nf;
  const long long total = per * nfields;
  for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < total;
       q += (long long)gridDim.x * blockDim.x) {
    const long long f = q / per, r = q - f * per;
    const long long row = r / g.nf;
    const long long l = f * g.slot + row * g.nfp + (r - row * g.nf);
    if (TO_PADDED)
      padded[l] = from_d<C>(dense[q]);
    else
      dense[q] = to_d(padded[l]);
  }
}

}  // namespace dnsb
