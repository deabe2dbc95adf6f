// ops.cuh -- a group of runs (one arena, one grid size and precision) and the
// kernel launches of its passes, per precision and grid size.  The kernels
// themselves are instantiated in the inst_*.cu translation units (one per
// precision and range of sizes, so that they compile side by side).
#pragma once
#include "dns_b200.h"
#include "persistent.cuh"

#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <map>
#include <mutex>
#include <string>

namespace {

enum { SLOT_SA = 0, SLOT_RK = 3, SLOT_WORK = 7, SLOT_P = 14, NSLOTS = 15 };
// passes of an RK stage, as dns_time_kernels reports them: A x-inverse, B
// y-inverse, C z fused, D y-forward, E1 x-forward, E2 pointwise update
enum { PASSES_PER_STAGE = 6 };
// the launches that run them: B, C and D (or YZ, the three in one: plane()), and
// X, which is a stage's E1 and E2 and the next stage's A in one kernel
enum { K_B = 0, K_C = 1, K_D = 2, K_X = 3, K_YZ = 4 };

}  // namespace

// A group: nruns runs of one grid size and precision in one arena, stepped
// by the same (batched) kernel launches.  A dns_ctx is a group of one run;
// a dns_ens holds one group per distinct grid size.
struct Group {
  long n = 0;
  int precision = 0;
  unsigned flags = 0;
  int nruns = 1;
  size_t csize = 16;      // bytes of one complex element
  size_t rsize = 8;       // bytes of one real element
  dnsb::Geo g{};
  char *arena = nullptr;
  size_t arena_bytes = 0;
  void *S = nullptr;      // spectral slots [nruns][NSLOTS][slot]
  void *stale = nullptr;  // stale real velocity [nruns][3][n^3]
  void *tw = nullptr;     // twiddles exp(-2 pi i k / n)
  double4 *diag_part = nullptr;  // [nruns][diag_blocks]
  double4 *diag_out = nullptr;   // [nruns]
  double *coef = nullptr;        // [nruns][2]: nu, dt
  int diag_blocks = 0;
  double *realbuf = nullptr;     // [4][n^3] float64, allocated on first field read
  // column-pass register schedules [axis][forward] picked by the autotuner
  // for this group's launches, and the run count they were timed on
  int pick[2][2] = {{0, 0}, {0, 0}};
  int tune_runs = 1;

  char *slot_ptr(int run, int s) const {
    return (char *)S + ((size_t)run * g.run_spec + (size_t)s * g.slot) * csize;
  }
  // float64 staging for host transfers of the FP32 path: the run's work
  // slots (7 * n^2 * nfp * 8 bytes >= 3 n^3 * 8 and >= 3 n^2 nf * 16)
  double *staging(int run) const { return (double *)slot_ptr(run, SLOT_WORK); }
  // the same arena seen as a batch of one run
  Group one(int run) const {
    Group v = *this;
    v.nruns = 1;
    v.S = slot_ptr(run, 0);
    v.stale = (char *)stale + (size_t)run * g.run_real * rsize;
    v.diag_part = diag_part + (size_t)run * diag_blocks;
    v.diag_out = diag_out + run;
    v.coef = coef + 2 * run;
    return v;
  }
};

namespace {

using namespace dnsb;

ColJobs jobs_empty(int njobs) {
  ColJobs j;
  for (int q = 0; q < 8; q++)
    j.in_slot[q] = 0, j.out_slot[q] = -1, j.der_slot[q] = -1, j.add_slot[q] = -1;
  j.njobs = njobs;
  j.masked = 0;
  return j;
}
ColJobs jobs_pass_b(bool first) {
  ColJobs j = jobs_empty(4);
  const int w = SLOT_WORK;
  // u, and omega_z = dv/dx - i ky u over the dv/dx slot (same tile, same block)
  j.in_slot[0] = w + SU; j.out_slot[0] = w + SU; j.der_slot[0] = w + SOMZ; j.add_slot[0] = w + SOMZ;
  j.in_slot[1] = w + SV; j.out_slot[1] = w + SV;
  // the first stage reads the stale real velocity, so W itself is not needed
  j.in_slot[2] = w + SW; j.out_slot[2] = first ? -1 : w + SW; j.der_slot[2] = w + SDWDY;
  j.in_slot[3] = w + SDWDX; j.out_slot[3] = w + SDWDX;
  return j;
}
ColJobs jobs_map(const int *in, const int *out, int cnt) {
  ColJobs j = jobs_empty(cnt);
  for (int q = 0; q < cnt; q++) j.in_slot[q] = in[q], j.out_slot[q] = out[q];
  return j;
}

template <class R, int N>
struct Ops {
  using Real = R;
  using C = cx<R>;
  static constexpr int Nval = N;
  static constexpr int E = Plan<N>::E;
  template <int AXIS>
  static constexpr int CW = ColW<R, AXIS, N>::W;
  template <int AXIS>
  static constexpr int CT = (N / E) * CW<AXIS>;
  template <int AXIS>
  static constexpr size_t COL_SMEM = (size_t)(N + N * CW<AXIS>) * sizeof(C);
  static constexpr size_t Z_SMEM = (size_t)(2 * N + ZCfg<N>::LINES * ZCfg<N>::XB) * sizeof(C);
  template <int KIND>
  static constexpr size_t ZS_SMEM = ZC<R, N, KIND>::SMEM;
  using X = XC<R, N>;
  static constexpr size_t XS_SMEM = X::SMEM;
  // A plane fits one SM's shared memory: B, C and D may run as one kernel.  At
  // n = 64 one or two runs have fewer planes than the GPU has SMs, and the
  // three kernels are faster (a step of one run: FP64 0.109 ms against 0.113,
  // FP32 0.090 against 0.092; three runs 0.186 ms before, 0.133 with it).
  static constexpr bool HAS_YZ = N <= 64;
  static bool plane(const Group &G) { return HAS_YZ && (N <= 32 || G.nruns >= 3); }
  // the kernels of a stage, in order
  static int kernels(const Group &G) { return plane(G) ? 2 : 4; }
  static int kernel(const Group &G, int q) { return plane(G) ? (q == 0 ? K_YZ : K_X) : q; }

  // Column-pass register schedules.  Candidate I of a pass is the same
  // kernel compiled with a minimum of ColCands::m[I] resident blocks per SM
  // (0: the compiler's own register choice); the candidates differ only in
  // register allocation, so every one computes bit-identical results.  The
  // autotuner (tune()) times them once per process, size and batch shape
  // (the run count it times on) and keeps the fastest; sizes below 64 have
  // the compiler's choice only.
  using ColFn = void (*)(const C *, C *, const C *, Geo, ColJobs);
  template <int AXIS>
  using Cands = ColCands<(N >= 64 ? (N / Plan<N>::E) * ColW<R, AXIS, N>::W : 0), (int)sizeof(C)>;
  template <int AXIS, bool FWD, int I>
  static ColFn col_cand() {
    constexpr int m = Cands<AXIS>::m[I];
    static_assert(m == 0 || col_minb_listed(m), "a candidate that DNSB_COL_MINB does not list");
    if constexpr (m == 0)
      return k_colpass<R, N, AXIS, FWD>;
    else
      return k_colpass_minb<R, N, AXIS, FWD, m>;
  }
  template <int AXIS, bool FWD, int I = 0>
  static ColFn col_cand_at(int i) {
    if constexpr (I + 1 < Cands<AXIS>::n) {
      if (i != I) return col_cand_at<AXIS, FWD, I + 1>(i);
    }
    return col_cand<AXIS, FWD, I>();
  }
  // chosen candidate of [AXIS][FWD] and the measured time per launch (ms)
  // of every candidate, per tuning run count
  struct TuneRec {
    int pick[2][2];
    float ms[2][2][16];
  };
  static inline std::map<int, TuneRec> tune_cache;
  static inline std::mutex tune_mu;  // guards tune_cache
  template <int AXIS, bool FWD>
  static ColFn colkern(const Group &G) {
    return col_cand_at<AXIS, FWD>(G.pick[AXIS][FWD]);
  }
  // runs a batch is tuned on: all of them up to the volume of two 256^3
  // runs, which fills the GPU like any larger batch
  static int tune_runs(int nruns) {
    long long cap = 2LL * 256 * 256 * 256 / ((long long)N * N * N);
    if (cap < 1) cap = 1;
    return (int)(nruns < cap ? nruns : cap);
  }

  template <class K>
  static cudaError_t allow(K kern, size_t smem) {
    if (smem <= 48 * 1024) return cudaSuccess;  // what every kernel may have
    return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  }
  template <int AXIS, bool FWD>
  static cudaError_t allow_cands() {
    cudaError_t e = cudaSuccess;
    for (int i = 0; i < Cands<AXIS>::n && e == cudaSuccess; i++)
      e = allow(col_cand_at<AXIS, FWD>(i), COL_SMEM<AXIS>);
    return e;
  }
  // also instantiates every kernel of this size (inst_*.cu)
  static cudaError_t setup() {
    cudaError_t e;
    if ((e = allow_cands<0, false>())) return e;
    if ((e = allow_cands<0, true>())) return e;
    if ((e = allow_cands<1, false>())) return e;
    if ((e = allow_cands<1, true>())) return e;
    if constexpr (HAS_YZ) {
      constexpr size_t sm = YZ<R, N>::SMEM;
      if ((e = allow(k_yz<R, N, 0, false>, sm))) return e;
      if ((e = allow(k_yz<R, N, 1, false>, sm))) return e;
      if ((e = allow(k_yz<R, N, 2, false>, sm))) return e;
      if constexpr (N <= 32) {
        if ((e = allow(k_yz<R, N, 0, true>, sm))) return e;
        if ((e = allow(k_yz<R, N, 1, true>, sm))) return e;
      }
    }
    if constexpr (N > 32) {
      if ((e = allow(k_zstage<R, N, 0>, ZS_SMEM<0>))) return e;
      if ((e = allow(k_zstage<R, N, 1>, ZS_SMEM<1>))) return e;
      if ((e = allow(k_zstage<R, N, 2>, ZS_SMEM<2>))) return e;
      if ((e = allow(k_zstage_keep<R, N, 0>, ZS_SMEM<0>))) return e;
      if ((e = allow(k_zstage_keep<R, N, 1>, ZS_SMEM<1>))) return e;
    }
    if ((e = allow(k_xstage<R, N, -1, true>, XS_SMEM))) return e;
    if ((e = allow(k_xstage<R, N, 0, true>, XS_SMEM))) return e;
    if ((e = allow(k_xstage<R, N, 1, true>, XS_SMEM))) return e;
    if ((e = allow(k_xstage<R, N, 2, true>, XS_SMEM))) return e;
    if ((e = allow(k_xstage<R, N, 3, true>, XS_SMEM))) return e;
    if ((e = allow(k_xstage<R, N, 3, false>, XS_SMEM))) return e;
    if ((e = allow(k_zr2c<R, N>, Z_SMEM))) return e;
    if ((e = allow(k_zc2r<R, N>, Z_SMEM))) return e;
    return cudaSuccess;
  }

  // ---- autotuner of the column-pass register schedules ----
  template <int AXIS, bool FWD>
  static cudaError_t time_cands(Group &Gt, cudaStream_t st, const ColJobs &jobs, cudaEvent_t e0,
                                cudaEvent_t e1, int force, int force_m, TuneRec &rec) {
    constexpr int n = Cands<AXIS>::n;
    int &pick = Gt.pick[AXIS][FWD];
    if (force_m >= 0) {  // a given register schedule: its candidate, else the compiler's
      pick = 0;
      for (int i = 0; i < n; i++)
        if (Cands<AXIS>::m[i] == force_m) pick = i;
      rec.pick[AXIS][FWD] = pick;
      return cudaSuccess;
    }
    int best = 0;
    for (int i = 0; i < n; i++) {
      pick = i;
      colpass_io<AXIS, FWD>(Gt, st, (C *)Gt.S, (C *)Gt.S, jobs, Gt.nruns);  // warm-up
      cudaError_t e = cudaEventRecord(e0, st);
      for (int r = 0; r < 3 && e == cudaSuccess; r++) {
        colpass_io<AXIS, FWD>(Gt, st, (C *)Gt.S, (C *)Gt.S, jobs, Gt.nruns);
        e = cudaGetLastError();
      }
      if (e == cudaSuccess) e = cudaEventRecord(e1, st);
      if (e == cudaSuccess) e = cudaEventSynchronize(e1);
      float ms = 0.f;
      if (e == cudaSuccess) e = cudaEventElapsedTime(&ms, e0, e1);
      if (e != cudaSuccess) return e;
      rec.ms[AXIS][FWD][i] = ms / 3.f;
      if (rec.ms[AXIS][FWD][i] < rec.ms[AXIS][FWD][best]) best = i;
    }
    pick = force >= 0 ? (force < n ? force : n - 1) : best;
    rec.pick[AXIS][FWD] = pick;
    return cudaSuccess;
  }
  // Time every register schedule of the four column passes (y: the job
  // tables of an RK stage, x: three fields, as the initial transform and the
  // field reads run them; batched over the group's first tune_runs(nruns)
  // runs, on their work slots, whose contents do not matter to an FFT's
  // timing) and keep the fastest of each; once per process, size and tuning
  // run count.  The group launches with the picks (G.pick).  DNS_B200_TUNE=0 keeps the compiler's schedule,
  // DNS_B200_TUNE=f<k> forces candidate k (the last where there are fewer),
  // DNS_B200_TUNE=m<a>,<b>,<c>,<d> the schedules of min blocks/SM a, b, c, d
  // for the x inverse, x forward, y inverse and y forward passes (as
  // dns_get_schedule reports them; a value that is not a candidate means
  // the compiler's).
  static cudaError_t tune(Group &G, cudaStream_t st, bool *ran) {
    std::lock_guard<std::mutex> lock(tune_mu);
    *ran = false;
    G.tune_runs = tune_runs(G.nruns);
    auto it = tune_cache.find(G.tune_runs);
    if (it != tune_cache.end()) {
      memcpy(G.pick, it->second.pick, sizeof G.pick);
      return cudaSuccess;
    }
    TuneRec rec{};
    const char *env = getenv("DNS_B200_TUNE");
    if (env && strcmp(env, "0") == 0) {
      tune_cache[G.tune_runs] = rec;
      memset(G.pick, 0, sizeof G.pick);
      return cudaSuccess;
    }
    const int force = (env && env[0] == 'f') ? atoi(env + 1) : -1;
    int fm[4] = {-1, -1, -1, -1};  // x inverse, x forward, y inverse, y forward
    if (env && env[0] == 'm') {
      const char *c = env + 1;
      for (int i = 0; i < 4 && *c; i++) {
        fm[i] = atoi(c);
        while (*c && *c != ',') c++;
        if (*c == ',') c++;
      }
    }
    Group Gt = G;  // the first tune_runs runs
    Gt.nruns = G.tune_runs;
    const int io[3] = {SLOT_WORK + SNX, SLOT_WORK + SNY, SLOT_WORK + SNZ};
    const ColJobs jx = jobs_map(io, io, 3);
    ColJobs jm = jx;
    jm.masked = 1;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    cudaError_t e = cudaEventCreate(&e0);
    if (e == cudaSuccess) e = cudaEventCreate(&e1);
    if (e == cudaSuccess)
      e = time_cands<0, false>(Gt, st, jx, e0, e1, force, fm[0], rec);
    if (e == cudaSuccess)
      e = time_cands<1, false>(Gt, st, jobs_pass_b(false), e0, e1, force, fm[2], rec);
    if (e == cudaSuccess) e = time_cands<1, true>(Gt, st, jm, e0, e1, force, fm[3], rec);
    if (e == cudaSuccess) e = time_cands<0, true>(Gt, st, jx, e0, e1, force, fm[1], rec);
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
    if (e == cudaSuccess) tune_cache[G.tune_runs] = rec;
    memcpy(G.pick, rec.pick, sizeof G.pick);
    *ran = true;
    return e;
  }
  // text description of the schedules chosen for G
  static std::string schedule(const Group &G) {
    std::string out;
    TuneRec rec{};
    memcpy(rec.pick, G.pick, sizeof rec.pick);
    {
      std::lock_guard<std::mutex> lock(tune_mu);
      auto it = tune_cache.find(G.tune_runs);
      if (it != tune_cache.end()) rec = it->second;
    }
    if (G.tune_runs > 1) out = "timed on " + std::to_string(G.tune_runs) + " runs: ";
    const char *name[2][2] = {{"x inverse", "x forward"}, {"y inverse", "y forward"}};
    char buf[160];
    for (int a = 0; a < 2; a++)
      for (int f = 0; f < 2; f++) {
        const int n = a == 0 ? Cands<0>::n : Cands<1>::n;
        const int *m = a == 0 ? Cands<0>::m : Cands<1>::m;
        const int k = rec.pick[a][f];
        snprintf(buf, sizeof buf, "%scolumn pass %s: min blocks/SM %d of {",
                 (a == 0 && f == 0) ? "" : "; ", name[a][f], m[k]);
        out += buf;
        for (int i = 0; i < n; i++) {
          snprintf(buf, sizeof buf, "%s%d: %.4f ms", i ? ", " : "", m[i], (double)rec.ms[a][f][i]);
          out += buf;
        }
        out += "}";
      }
    return out;
  }

  // the z pass of RK stage s, or all of B, C and D (plane); with `keep`
  // (one run; stage 3 in the middle stages' form) also keeping the real
  // velocity and vorticity in keep[6][n^3]
  template <int KIND>
  static void zpass(const Group &G, cudaStream_t st, R *keep) {
    C *work = slot(G, SLOT_WORK);
    R *stale = (R *)G.stale;
    const R invn3 = (R)(1.0 / (double)G.g.nreal);
    if constexpr (HAS_YZ) if (plane(G)) {
      const dim3 grid(N, G.nruns);
      if constexpr (KIND < 2 && N <= 32) {
        if (keep) {
          k_yz<R, N, KIND, true><<<grid, YZ<R, N>::THREADS, YZ<R, N>::SMEM, st>>>(
              work, stale, tw(G), G.g, invn3, keep);
          return;
        }
      }
      k_yz<R, N, KIND, false><<<grid, YZ<R, N>::THREADS, YZ<R, N>::SMEM, st>>>(
          work, stale, tw(G), G.g, invn3, nullptr);
      return;
    }
    if constexpr (N > 32) {
      constexpr int th = ZC<R, N, KIND>::THREADS;
      if constexpr (KIND < 2) {
        if (keep) {
          k_zstage_keep<R, N, KIND><<<zsgrid<KIND>(G.nruns), th, ZS_SMEM<KIND>, st>>>(
              work, stale, tw(G), G.g, invn3, keep);
          return;
        }
      }
      k_zstage<R, N, KIND><<<zsgrid<KIND>(G.nruns), th, ZS_SMEM<KIND>, st>>>(work, stale, tw(G),
                                                                             G.g, invn3);
    }
  }

  static C *slot(const Group &G, int s) { return (C *)G.S + (long long)s * G.g.slot; }
  static const C *tw(const Group &G) { return (const C *)G.tw; }

  template <int AXIS, bool FWD>
  static void colpass_io(const Group &G, cudaStream_t st, const C *in, C *out, const ColJobs &jobs,
                         int nruns) {
    // a masked pass covers the tiles holding kz <= kcut
    const int tiles = jobs.masked ? G.g.kcut / CW<AXIS> + 1 : G.g.nfp / CW<AXIS>;
    dim3 grid(tiles, N, jobs.njobs * nruns);
    colkern<AXIS, FWD>(G)<<<grid, CT<AXIS>, COL_SMEM<AXIS>, st>>>(in, out, tw(G), G.g, jobs);
  }
  template <int AXIS, bool FWD>
  static void colpass(const Group &G, cudaStream_t st, const ColJobs &jobs) {
    colpass_io<AXIS, FWD>(G, st, (C *)G.S, (C *)G.S, jobs, G.nruns);
  }

  static dim3 zgrid(int nfields) { return dim3((N * N) / ZCfg<N>::LINES, nfields); }
  template <int KIND>
  static dim3 zsgrid(int nruns) {
    return dim3((N * N + ZC<R, N, KIND>::LINES - 1) / ZC<R, N, KIND>::LINES, nruns);
  }

  static XArgs<R> xargs(const Group &G, int s) {
    return XArgs<R>{slot(G, SLOT_SA), slot(G, SLOT_RK), slot(G, SLOT_WORK),
                    (s == 3 && (G.flags & DNS_FLAG_PRESSURE)) ? slot(G, SLOT_P) : nullptr, G.coef};
  }
  static dim3 xgrid(const Group &G) { return dim3((G.g.nf + X::W - 1) / X::W, N, G.nruns); }

  // Kernel `k` (K_B..K_X) of RK stage `s` for all runs of G, or with s < 0
  // the x transform of the state a step starts from: what it runs, its job
  // table or arguments, and its work items (the launch grid, threads and
  // shared memory of one block).  The persistent ensemble kernel's plan is made
  // from it, and the standalone launches of B and D (stage_kernel).
  static PPhase<R> describe(const Group &G, int s, int k) {
    const Geo &g = G.g;
    PPhase<R> P{};
    P.gz = 1;
    if (k == K_B || k == K_D) {
      P.kind = PK_COL;
      P.fwd = k == K_D;
      if (k == K_B) {
        P.jobs = jobs_pass_b(s == 0);
      } else {
        // y forward, in place on the three N slots; only the modes inside
        // the 2/3 rule are computed and stored
        const int io[3] = {SLOT_WORK + SNX, SLOT_WORK + SNY, SLOT_WORK + SNZ};
        P.jobs = jobs_map(io, io, 3);
        P.jobs.masked = 1;
      }
      // a masked pass covers the tiles holding kz <= kcut
      constexpr int cw = CW<1>;
      P.gx = P.jobs.masked ? g.kcut / cw + 1 : g.nfp / cw;
      P.gy = N;
      P.gz = P.jobs.njobs * G.nruns;
      P.tpi = CT<1>;
      P.smem = (int)COL_SMEM<1>;
    } else if (k == K_C) {
      P.kind = PK_Z;
      P.sub = s == 0 ? 0 : s < 3 ? 1 : 2;
      const int lines = P.sub == 0 ? ZC<R, N, 0>::LINES : P.sub == 1 ? ZC<R, N, 1>::LINES
                                                                      : ZC<R, N, 2>::LINES;
      P.gx = (N * N + lines - 1) / lines;
      P.gy = G.nruns;
      P.tpi = ZC<R, N, 0>::THREADS;
      P.smem = (int)(P.sub == 0 ? ZS_SMEM<0> : P.sub == 1 ? ZS_SMEM<1> : ZS_SMEM<2>);
    } else {
      P.kind = PK_X;
      P.sub = s;
      P.xa = xargs(G, s);
      const dim3 grid = xgrid(G);
      P.gx = grid.x;
      P.gy = grid.y;
      P.gz = grid.z;
      P.tpi = X::THREADS;
      P.smem = (int)XS_SMEM;
    }
    return P;
  }

  template <int ST, bool TAIL>
  static void xpass(const Group &G, cudaStream_t st) {
    k_xstage<R, N, ST, TAIL>
        <<<xgrid(G), X::THREADS, XS_SMEM, st>>>(xargs(G, ST), tw(G), G.g);
  }

  // kernel `k` of RK stage `s`, all runs of G; `tail`: the last stage's x
  // pass also transforms the new state for the next step; `keep`: of zpass
  static void stage_kernel(const Group &G, cudaStream_t st, int s, int k, bool tail,
                           R *keep = nullptr) {
    if (k == K_X) {
      if (s < 0)
        xpass<-1, true>(G, st);
      else if (s == 0)
        xpass<0, true>(G, st);
      else if (s == 1)
        xpass<1, true>(G, st);
      else if (s == 2)
        xpass<2, true>(G, st);
      else if (tail)
        xpass<3, true>(G, st);
      else
        xpass<3, false>(G, st);
    } else if (k == K_C || k == K_YZ) {
      if (s == 0)
        zpass<0>(G, st, keep);
      else if (s < 3 || keep)
        zpass<1>(G, st, keep);
      else
        zpass<2>(G, st, nullptr);
    } else {
      const PPhase<R> P = describe(G, s, k);
      ColFn f = P.fwd ? colkern<1, true>(G) : colkern<1, false>(G);
      f<<<dim3(P.gx, P.gy, P.gz), P.tpi, P.smem, st>>>((C *)G.S, (C *)G.S, tw(G), G.g, P.jobs);
    }
  }

  // this group's part of the persistent ensemble kernel's plan
  static void plan_group(const Group &G, PGroup<R> &pg) {
    pg.n = N;
    pg.g = G.g;
    pg.S = (C *)G.S;
    pg.work = slot(G, SLOT_WORK);
    pg.stale = (R *)G.stale;
    pg.tw = tw(G);
    pg.invn3 = (R)(1.0 / (double)G.g.nreal);
    pg.ph[0] = describe(G, -1, K_X);
    for (int s = 0; s < 4; s++)
      for (int k = K_B; k <= K_X; k++) pg.ph[1 + 4 * s + k] = describe(G, s, k);
  }

  // the x transform of the state, which a step starts from
  static void first(const Group &G, cudaStream_t st) { stage_kernel(G, st, -1, K_X, true); }
  static void step(const Group &G, cudaStream_t st, bool tail) {
    for (int s = 0; s < 4; s++)
      for (int q = 0; q < kernels(G); q++) stage_kernel(G, st, s, kernel(G, q), tail);
  }

  // forward transform of the three stale real slots into SA (one run)
  static void forward(const Group &G, cudaStream_t st) {
    k_zr2c<R, N><<<zgrid(3), ZCfg<N>::THREADS, Z_SMEM, st>>>((const R *)G.stale,
                                                              slot(G, SLOT_WORK), tw(G), G.g);
    const int w3[3] = {SLOT_WORK + 0, SLOT_WORK + 1, SLOT_WORK + 2};
    const int sa[3] = {SLOT_SA + 0, SLOT_SA + 1, SLOT_SA + 2};
    colpass<1, true>(G, st, jobs_map(w3, w3, 3));
    colpass<0, true>(G, st, jobs_map(w3, sa, 3));
  }

  // c2r(X) / n^3 of SA (and P) into realbuf [4][n^3] float64 (one run)
  static void backward(const Group &G, cudaStream_t st, int nfields) {
    const int in[4] = {SLOT_SA + 0, SLOT_SA + 1, SLOT_SA + 2, SLOT_P};
    const int w4[4] = {SLOT_WORK + 0, SLOT_WORK + 1, SLOT_WORK + 2, SLOT_WORK + 3};
    colpass<0, false>(G, st, jobs_map(in, w4, nfields));
    colpass<1, false>(G, st, jobs_map(w4, w4, nfields));
    k_zc2r<R, N><<<zgrid(nfields), ZCfg<N>::THREADS, Z_SMEM, st>>>(
        slot(G, SLOT_WORK), G.realbuf, tw(G), G.g, 1.0 / (double)G.g.nreal);
  }

  // c2r of K spectral fields (in + in_slots[f] * slot) into out[f * nreal],
  // scaled (one run; uses the work slots)
  static void c2r_fields(const Group &G, cudaStream_t st, const C *in, const int *in_slots, int K,
                         double *out, double scale) {
    C *wk = slot(G, SLOT_WORK);
    ColJobs j1 = jobs_empty(K), j2 = jobs_empty(K);
    for (int f = 0; f < K; f++) {
      j1.in_slot[f] = in_slots[f];
      j1.out_slot[f] = f;
      j2.in_slot[f] = f;
      j2.out_slot[f] = f;
    }
    colpass_io<0, false>(G, st, in, wk, j1, 1);
    colpass_io<1, false>(G, st, wk, wk, j2, 1);
    k_zc2r<R, N><<<zgrid(K), ZCfg<N>::THREADS, Z_SMEM, st>>>(wk, out, tw(G), G.g, scale);
  }

  // energy / enstrophy sums of every run into diag_out[run]
  static void diag(const Group &G, cudaStream_t st) {
    k_diag<256, C><<<dim3(G.diag_blocks, G.nruns), 256, 0, st>>>(slot(G, SLOT_SA), G.g, G.diag_part);
    k_diag_final<256><<<G.nruns, 256, 0, st>>>(G.diag_part, G.diag_blocks, G.diag_out);
  }
};

}  // namespace
