// k_dss.cuh -- direct-stiffness gather-scatter (GGFX::doOp) kernels.
//
// One thread per equivalence class (a lattice point on box grids, a node
// of a singleton class or a shared class on CSR grids): it gathers the
// class members in ascending local id, folds them exactly as the
// reference's reduction functors do (comm/ggfx.hpp:36-76: std::accumulate
// from 0 for Sum and Smooth, std::max/std::min folds from lowest()/max()),
// and scatters the result to every member.  The fold order is fixed, so
// FP64 results are bit-identical to the reference's and independent of the
// launch shape.
#pragma once
#include <cfloat>

#include "gf_common.cuh"
#include "k_vec.cuh"

namespace gfk {

template <typename T> struct Lim;
template <> struct Lim<double> {
  static __device__ __forceinline__ double lowest() { return -DBL_MAX; }
  static __device__ __forceinline__ double highest() { return DBL_MAX; }
};
template <> struct Lim<float> {
  static __device__ __forceinline__ float lowest() { return -FLT_MAX; }
  static __device__ __forceinline__ float highest() { return FLT_MAX; }
};

// The box-lattice walk of a problem whose gather-scatter can take the box
// kernels below: a GGridBox problem (classes = lattice points) with no
// periodic direction of a single element (members then come in the
// (z, y, x) nesting in ascending local id).
inline bool dss_box_walk(const gf_problem *prob, BoxWalk &w) {
  if (!prob->has_box) return false;
  w = BoxWalk::make(prob->box);
  return w.sorted;
}

// Blocks of the run kernels (one run per thread): tiles of x by the next
// direction (y in 3-d, the layers in 2-d), so that the rows of an element that
// share cache lines belong to one block.  Tiles of 32 lanes in x, or narrower
// where that would idle more than an eighth of them; 64 threads where there would
// otherwise be SMs without a block.
struct RunGrid {
  unsigned blocks;
  dim3 block;
  int nx, ny;      // tiles along x, rows of tiles per layer
  FastDiv fx, fy;  // by nx, ny
};
template <int P>
inline RunGrid run_grid(const gf_problem *prob, const RunWalk<P> &w) {
  const int th = w.n < prob->ctx->sm_count * 512 ? 64 : 256;
  if (w.one) {  // lattice order
    RunGrid g{};
    g.block = dim3(128);
    g.blocks = (unsigned)((w.npts + 127) / 128);
    return g;
  }
  int tx = 32;
  while (tx > 8 && (int64_t)((w.M0 + tx - 1) / tx * tx) * 7 > (int64_t)w.M0 * 8) tx /= 2;
  const int ty = th / tx, layers = w.neL + (w.perL ? 0 : 1);
  const int rows = w.dim > 2 ? w.M1 : layers;
  RunGrid g;
  g.block = dim3(tx, ty);
  g.nx = (w.M0 + tx - 1) / tx;
  g.ny = (rows + ty - 1) / ty;
  g.fx = FastDiv::make(g.nx);
  g.fy = FastDiv::make(g.ny);
  g.blocks = (unsigned)g.nx * (unsigned)g.ny * (unsigned)(w.dim > 2 ? layers : 1);
  return g;
}
// whether this thread has a run, and the run
template <int P>
__device__ __forceinline__ bool run_of_thread(const RunWalk<P> &w, const RunGrid &g, LatRun &k) {
  const int row = g.fx.div((int)blockIdx.x), bx = (int)blockIdx.x - row * g.nx;
  int q = 0, by = row;
  if (w.dim > 2) {
    q = g.fy.div(row);
    by = row - q * g.ny;
  }
  const int g0 = bx * (int)blockDim.x + (int)threadIdx.x;
  const int r = by * (int)blockDim.y + (int)threadIdx.y;
  if (g0 >= w.M0 || r >= (w.dim > 2 ? w.M1 : w.neL + (w.perL ? 0 : 1))) return false;
  k = w.dim > 2 ? w.run(g0, r, q) : w.run(g0, 0, r);
  return true;
}

// 1/(copies of a point): 1, 1/2, 1/4 or 1/8, so that multiplying by it rounds
// exactly as the division by the count does
template <typename T>
__device__ __forceinline__ T run_inv_count(const LatRun &k, int r) {
  return (k.nx > 1 ? T(0.5) : T(1)) * (k.ny > 1 ? T(0.5) : T(1)) *
         (r == 0 && k.nz > 1 ? T(0.5) : T(1));
}

// one step of the GGFX fold, and its start from the first copy
template <typename T, int OP>
__device__ __forceinline__ T dss_first(T v) {
  if (OP == GF_DSS_MAX) return (Lim<T>::lowest() < v) ? v : Lim<T>::lowest();
  if (OP == GF_DSS_MIN) return (v < Lim<T>::highest()) ? v : Lim<T>::highest();
  return __fadd_rn_t(T(0), v);
}
template <typename T, int OP>
__device__ __forceinline__ T dss_next(T acc, T v) {
  if (OP == GF_DSS_MAX) return (acc < v) ? v : acc;
  if (OP == GF_DSS_MIN) return (v < acc) ? v : acc;
  return __fadd_rn_t(acc, v);
}

// The folds of a run of lattice points (ascending local id per point); every
// first copy is read before any fold.
template <typename T, int OP, int P>
__device__ __forceinline__ void dss_run(const T *u, const RunWalk<P> &w,
                                        const LatRun &k, T (&acc)[P]) {
  w.first(k, [&](int r, int m) { acc[r] = u[m]; });
#pragma unroll
  for (int r = 0; r < P; r++) acc[r] = dss_first<T, OP>(acc[r]);
  w.rest(k, [&](int r, int m) { acc[r] = dss_next<T, OP>(acc[r], u[m]); });
  if (OP == GF_DSS_SMOOTH) {
#pragma unroll
    for (int r = 0; r < P; r++) acc[r] *= run_inv_count<T>(k, r);
  }
}

// Whether a gather walks its lattice by points (k_dss_point) or in runs (k_dss_box).
// Runs save index arithmetic but are p times fewer threads.  They lose where too few
// are left to cover the latency: lattices of fewer than POINT_NODES points (476 x 476
// points, p = 7, FP64: 4.9 us, in runs 5.7) and in 3-d, where a run's copies lie
// further apart, of fewer than RUNS_3D runs (FP64 and FP32 alike: 71^3 points, p = 7,
// 51 k runs: 6.2 us by points, 8.3 in runs; 73^3, p = 9, 43 k: 6.5 and 8.3; 78^3,
// p = 11, 43 k: 6.3 and 8.2; even at 78^3, p = 7, 68 k, and 82^3, p = 9, 61 k; runs
// ahead at 66^3, p = 5, 57 k, FP32, 8.2 and 6.2), and at p = 1, where a run is a point
// (80^3: FP64 25.5 us by points, 26.7 in runs, FP32 18.5 and 22.3; 549^2: 8.4 and 10.3).
constexpr int RUNS_3D = 56000;
inline bool dss_by_points(const gf_problem *prob, const BoxWalk &w) {
  const int p = prob->n - 1;
  return p == 1 || w.nL < POINT_NODES || (prob->dim == 3 && w.nL < RUNS_3D * p);
}

// Box-lattice form of k_dss_split (GGridBox problems, whose classes are the
// lattice points; no periodic direction with a single element): one thread
// per run of P lattice points (RunWalk), the members computed from the
// coordinates in ascending local id, so no index arrays are read.  Same folds,
// same order: bit-identical to the CSR form.  A block folds all of its points
// before it writes any: a store drops its line from the L1, where the block's
// other rows would still find their values.
template <typename T, int OP, int P>
__global__ void __launch_bounds__(256) k_dss_box(T *u, const RunWalk<P> w, const RunGrid g) {
  LatRun k;
  T acc[P] = {};
  const bool on = run_of_thread(w, g, k);
  if (on) dss_run<T, OP, P>(u, w, k, acc);
  __syncthreads();
  if (!on) return;
  auto put = [&](int r, int m) { u[m] = acc[r]; };
  w.first(k, put);
  w.rest(k, put);
}

// The same, one thread per point.
template <typename T, int OP>
__global__ void __launch_bounds__(256) k_dss_point(T *__restrict__ u, BoxWalk w) {
  const int stride = gridDim.x * blockDim.x;
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < w.nL;
       c = (c < w.nL - stride) ? c + stride : w.nL) {
    const BoxCopies k = w.copies(c);
    T acc = OP == GF_DSS_MAX ? Lim<T>::lowest() : (OP == GF_DSS_MIN ? Lim<T>::highest() : T(0));
    k.each([&](int m) { acc = dss_next<T, OP>(acc, u[m]); });
    if (OP == GF_DSS_SMOOTH) acc = acc / (T)k.count();
    k.each([&](int m) { u[m] = acc; });
  }
}

// The classes of a CSR problem split by size: a class with one member (an
// interior node, most of them on icosahedral and deformed grids) is folded
// by the thread of that node, in node order (coalesced, no index arrays;
// imult = 1 marks it), and a class with several members by one thread from
// the shared-class list (sh_ptr / sh_members, members in ascending local
// id).  Items: the n nodes, then the nsh shared classes.  Each class is
// folded exactly as the full CSR walk folds it.
struct SplitCls {
  int64_t n;              // element-local nodes
  const float *imult;     // 1/multiplicity per node
  const int32_t *shp;     // nsh + 1
  const int32_t *shm;
  int64_t nsh;
};

inline SplitCls split_of(const gf_problem *p) {
  return SplitCls{p->nlocal, p->imult_f, p->sh_ptr, p->sh_members, p->nshared};
}

// f(get, cnt): get(k) is the k-th member (ascending local id) of item it's
// class, cnt the member count; nothing for a node of a shared class.
template <class F>
__device__ __forceinline__ void split_item(const SplitCls &s, int64_t it, F f) {
  if (it < s.n) {
    if (s.imult[it] != 1.0f) return;
    f([&](int) { return it; }, 1);
  } else {
    const int64_t c = it - s.n;
    const int32_t b = s.shp[c], e = s.shp[c + 1];
    f([&](int k) { return (int64_t)s.shm[b + k]; }, e - b);
  }
}

template <typename T, int OP>
__global__ void __launch_bounds__(256) k_dss_split(T *__restrict__ u, SplitCls s) {
  for (int64_t it = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; it < s.n + s.nsh;
       it += (int64_t)gridDim.x * blockDim.x)
    split_item(s, it, [&](auto get, int cnt) {
      T acc;
      if (OP == GF_DSS_SUM || OP == GF_DSS_SMOOTH) {
        acc = T(0);
        for (int k = 0; k < cnt; k++) acc = __fadd_rn_t(acc, u[get(k)]);
        if (OP == GF_DSS_SMOOTH) acc = acc / (T)cnt;
      } else if (OP == GF_DSS_MAX) {
        acc = Lim<T>::lowest();
        for (int k = 0; k < cnt; k++) {
          const T v = u[get(k)];
          acc = (acc < v) ? v : acc;
        }
      } else {
        acc = Lim<T>::highest();
        for (int k = 0; k < cnt; k++) {
          const T v = u[get(k)];
          acc = (v < acc) ? v : acc;
        }
      }
      for (int k = 0; k < cnt; k++) u[get(k)] = acc;
    });
}

// ---- gather-scatter fused with the RK stage updates (api_rk.cu) ----
// The stage arithmetic of GExRKStepper, with explicit round-to-nearest
// operations so that it rounds the same wherever it runs:
//   step_euler + saxpby (gexrk_stepper.ipp:809-819, 533-780):
//     v = dt x + 1 uin;  v = a v + b y (if y);  v = a2 v + b2 y2 (if y2)
//   step_b accumulation (252-341): uout += (K * ch)
// (y[i] and y2[i] are read before the arithmetic, so that a caller's loads
// of several points are all in flight together; measured on the FP64
// stage-update pass at 64^3 p = 5: 1.68 -> 1.57 ms)
template <typename T>
__device__ __forceinline__ T rk_euler_vals(T x, T dt, T uin, T a, bool has_y, T yv, T b, T a2,
                                           bool has_y2, T y2v, T b2) {
  T v = add_rn(mul_rn(dt, x), mul_rn(T(1), uin));
  if (has_y) v = add_rn(mul_rn(a, v), mul_rn(b, yv));
  if (has_y2) v = add_rn(mul_rn(a2, v), mul_rn(b2, y2v));
  return v;
}
template <typename T>
__device__ __forceinline__ T rk_euler_point(T x, T dt, T uin, T a, const T *y, T b, T a2,
                                            const T *y2, T b2, int64_t i) {
  return rk_euler_vals(x, dt, uin, a, y != nullptr, y ? y[i] : T(0), b, a2, y2 != nullptr,
                       y2 ? y2[i] : T(0), b2);
}
template <typename T>
__device__ __forceinline__ T rk_accum_point(T uout, T K, T ch) {
  return add_rn(uout, mul_rn(K, ch));
}
// step_b stage input (252-341): y = uin + ((0 + b0 K0) + b1 K1 + ...), the
// isum accumulation over the nk earlier slopes
template <typename T>
__device__ __forceinline__ T rk_stage_point(T uin, int nk, const T *__restrict__ K0,
                                            const T *__restrict__ K1, const T *__restrict__ K2,
                                            T b0, T b1, T b2, int64_t i) {
  T s = T(0);
  if (nk > 0) s = T(1) * s + b0 * K0[i];
  if (nk > 1) s = T(1) * s + b1 * K1[i];
  if (nk > 2) s = T(1) * s + b2 * K2[i];
  T v = uin;
  v += s;
  return v;
}

// y = uin + (0 + b K), rounded as rk_stage_point rounds a sum of one slope
template <typename T>
__device__ __forceinline__ T rk_input_point(T uin, T b, T K) {
  return add_rn(uin, __fadd_rn_t(T(0), mul_rn(b, K)));
}

// One pass per stage over the gather-scatter classes (members in ascending
// local id, Smooth folds):
//   RK_EULER  (SSP substep)       out <- fold(rk_euler_point(x, ...))
//   RK_MID    (step_b stage m)    K = fold(x);  acc_m = rk_accum_point(accin_m, K, ch);
//                                 out_m = uin_m + b K, the next stage's input
//   RK_MIDS   (the last but one)  the same with out folded: the last stage's
//                                 input is smoothed (gexrk_stepper.ipp:252-341)
//   RK_LAST   (last stage)        K = fold(x);  out <- fold(rk_accum_point(accin, K, ch))
//   RK_SMOOTH                     out <- fold(x)
// Each reads x, uin and accin once and writes what the next kernel reads, so a
// step_b stage is this pass and the right-hand side, with no separate stage
// sum, slope write-back, state copy or second Smooth pass.  The reverse sweep
// of step_b (api_adjoint.cu) has passes of the same form:
//   ADJ_START       s = fold(x);  acc = aux = s;  out = ch s
//   ADJ_STAGE       s = fold(x);  acc_m += x_m;   out_m = ch aux_m + b s
//   ADJ_STAGE_LAST  s = fold(x);  acc_m += s;     out_m = ch aux_m + b s
enum {
  RK_EULER = 0,
  RK_MID = 1,
  RK_MIDS = 2,
  RK_LAST = 3,
  RK_SMOOTH = 4,
  ADJ_START = 5,
  ADJ_STAGE = 6,
  ADJ_STAGE_LAST = 7
};

template <typename T>
struct RKPass {
  const T *x[3], *uin[3], *y[3], *y2[3], *accin[3];
  T *out[3], *acc[3], *aux[3];
  T dt, a, b, a2, b2, ch;
};

// which modes read uin and accin, and what they fold after K
template <int MODE>
struct RKMode {
  static constexpr bool ADJ = MODE >= ADJ_START;
  static constexpr bool MID = MODE == RK_MID || MODE == RK_MIDS;
  static constexpr bool UIN = MODE == RK_EULER || MID, ACC = MID || MODE == RK_LAST;
  // the members share one result: out <- the fold s
  static constexpr bool SAME = MODE == RK_EULER || MODE == RK_LAST || MODE == RK_SMOOTH;
};

// what the pass folds at member m, v = x[m] and u = uin[m] read already
template <typename T, int MODE>
__device__ __forceinline__ T rk_value(const RKPass<T> &p, int j, T v, T u, int64_t m) {
  if constexpr (MODE == RK_EULER)
    return rk_euler_point(v, p.dt, u, p.a, p.y[j], p.b, p.a2, p.y2[j], p.b2, m);
  return v;
}

// the writes of one member of the modes whose members differ: s the folded K,
// o the folded input (RK_MIDS), x, u and c the member's x, uin and accin
template <typename T, int MODE>
__device__ __forceinline__ void rk_write(const RKPass<T> &p, int j, T s, T o, T x, T u, T c,
                                         int64_t m) {
  if constexpr (RKMode<MODE>::MID) {
    p.acc[j][m] = rk_accum_point(c, s, p.ch);
    p.out[j][m] = MODE == RK_MIDS ? o : rk_input_point(u, p.b, s);
  } else if constexpr (MODE == ADJ_START) {
    p.acc[j][m] = s;
    p.aux[j][m] = s;
    p.out[j][m] = p.ch * s;
  } else {
    const T a = p.acc[j][m], l = p.aux[j][m];
    p.acc[j][m] = a + (MODE == ADJ_STAGE ? x : s);
    p.out[j][m] = fma(p.b, s, p.ch * l);
  }
}

// the members of one class in ascending local id: first(), rest(f) the others,
// each(f) all; mean(s) = s / count
template <class GET>
struct SplitMembers {
  const GET &get;
  int cnt;
  __device__ __forceinline__ int64_t first() const { return get(0); }
  template <class F> __device__ __forceinline__ void rest(F f) const {
    for (int i = 1; i < cnt; i++) f(get(i));
  }
  template <class F> __device__ __forceinline__ void each(F f) const {
    for (int i = 0; i < cnt; i++) f(get(i));
  }
  template <typename T> __device__ __forceinline__ T mean(T s) const { return s / (T)cnt; }
};

// Component j of one class.  The first member's values (the only ones of most
// classes) are read before any arithmetic, and every read before the first
// write, so a class costs one memory round trip.
template <typename T, int MODE, class MEM>
__device__ __forceinline__ void rk_class(const RKPass<T> &p, int j, const MEM &mem) {
  using M = RKMode<MODE>;
  const int64_t m0 = mem.first();
  const T *x = p.x[j], *uin = p.uin[j], *accin = p.accin[j];
  const T x0 = x[m0], u0 = M::UIN ? uin[m0] : T(0), c0 = M::ACC ? accin[m0] : T(0);
  T s = __fadd_rn_t(T(0), rk_value<T, MODE>(p, j, x0, u0, m0)), o = T(0);
  mem.rest([&](int64_t m) {
    s = __fadd_rn_t(s, rk_value<T, MODE>(p, j, x[m], M::UIN ? uin[m] : T(0), m));
  });
  s = mem.mean(s);
  if constexpr (MODE == RK_LAST) {
    o = __fadd_rn_t(T(0), rk_accum_point(c0, s, p.ch));
    mem.rest([&](int64_t m) { o = __fadd_rn_t(o, rk_accum_point(accin[m], s, p.ch)); });
    s = mem.mean(o);
  }
  if constexpr (MODE == RK_MIDS) {
    o = __fadd_rn_t(T(0), rk_input_point(u0, p.b, s));
    mem.rest([&](int64_t m) { o = __fadd_rn_t(o, rk_input_point(uin[m], p.b, s)); });
    o = mem.mean(o);
  }
  if constexpr (M::SAME) {
    T *out = p.out[j];
    mem.each([&](int64_t m) { out[m] = s; });
  } else {
    mem.rest([&](int64_t m) {
      rk_write<T, MODE>(p, j, s, o, x[m], M::UIN ? uin[m] : T(0), M::ACC ? accin[m] : T(0), m);
    });
    rk_write<T, MODE>(p, j, s, o, x0, u0, c0, m0);
  }
}

// Box problems: one run of P lattice points per thread, the state components
// one after the other (the copies are found once).
template <typename T, int MODE, int P>
__device__ __forceinline__ void rk_run(const RKPass<T> &p, int nc, const RunWalk<P> &w,
                                       const LatRun &k) {
  using M = RKMode<MODE>;
#pragma unroll 1
  for (int j = 0; j < nc; j++) {
    const T *x = p.x[j], *uin = p.uin[j], *accin = p.accin[j];
    T *out = p.out[j];
    T s[P] = {}, x0[P] = {}, u0[P] = {}, c0[P] = {};
    w.first(k, [&](int r, int m) {
      x0[r] = x[m];
      if (M::UIN) u0[r] = uin[m];
      if (M::ACC) c0[r] = accin[m];
    });
    w.first(k, [&](int r, int m) {
      s[r] = __fadd_rn_t(T(0), rk_value<T, MODE>(p, j, x0[r], u0[r], m));
    });
    w.rest(k, [&](int r, int m) {
      s[r] = __fadd_rn_t(s[r], rk_value<T, MODE>(p, j, x[m], M::UIN ? uin[m] : T(0), m));
    });
#pragma unroll
    for (int r = 0; r < P; r++) s[r] *= run_inv_count<T>(k, r);
    T o[P] = {};
    if constexpr (MODE == RK_LAST) {
#pragma unroll
      for (int r = 0; r < P; r++) o[r] = __fadd_rn_t(T(0), rk_accum_point(c0[r], s[r], p.ch));
      w.rest(k, [&](int r, int m) {
        o[r] = __fadd_rn_t(o[r], rk_accum_point(accin[m], s[r], p.ch));
      });
#pragma unroll
      for (int r = 0; r < P; r++) s[r] = o[r] * run_inv_count<T>(k, r);
    }
    if constexpr (MODE == RK_MIDS) {
#pragma unroll
      for (int r = 0; r < P; r++) o[r] = __fadd_rn_t(T(0), rk_input_point(u0[r], p.b, s[r]));
      w.rest(k, [&](int r, int m) {
        o[r] = __fadd_rn_t(o[r], rk_input_point(uin[m], p.b, s[r]));
      });
#pragma unroll
      for (int r = 0; r < P; r++) o[r] *= run_inv_count<T>(k, r);
    }
    if constexpr (M::SAME) {
      auto put = [&](int r, int m) { out[m] = s[r]; };
      w.first(k, put);
      w.rest(k, put);
    } else {
      w.first(k, [&](int r, int m) {
        rk_write<T, MODE>(p, j, s[r], o[r], x0[r], u0[r], c0[r], m);
      });
      w.rest(k, [&](int r, int m) {
        rk_write<T, MODE>(p, j, s[r], o[r], x[m], M::UIN ? uin[m] : T(0), M::ACC ? accin[m] : T(0),
                          m);
      });
    }
  }
}

template <typename T, int MODE, int P>
__global__ void __launch_bounds__(256)
    k_rk_box(const __grid_constant__ RKPass<T> p, int nc, const RunWalk<P> w, const RunGrid g) {
  LatRun k;
  if (w.one) {
    const int t = (int)(blockIdx.x * blockDim.x + threadIdx.x);
    if (t < w.npts) rk_run<T, MODE, P>(p, nc, w, w.point(t));
  } else if (run_of_thread(w, g, k)) {
    rk_run<T, MODE, P>(p, nc, w, k);
  }
}

// Other problems, one component: the nodes of singleton classes, four per thread
// with all of their reads in flight together (one at a time the pass was
// bound by the latency of its three reads: 9.5 us at 0.75 M FP32 nodes).  The
// shared classes, whose reads are a chain of three, have the first nbs blocks
// to themselves, so that the two latencies overlap.
template <typename T, int MODE>
__global__ void __launch_bounds__(256)
    k_rk_split(const __grid_constant__ RKPass<T> p, int j, SplitCls s, unsigned nbs) {
  using M = RKMode<MODE>;
  constexpr int U = 4;
  if (blockIdx.x < nbs) {
    for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < s.nsh;
         c += (int64_t)nbs * blockDim.x) {
      const int32_t b = s.shp[c], e = s.shp[c + 1];
      auto get = [&](int k) { return (int64_t)s.shm[b + k]; };
      rk_class<T, MODE>(p, j, SplitMembers<decltype(get)>{get, e - b});
    }
    return;
  }
  const int64_t t0 = (int64_t)(blockIdx.x - nbs) * blockDim.x + threadIdx.x;
  const int64_t stride = (int64_t)(gridDim.x - nbs) * blockDim.x;
  const T *x = p.x[j], *uin = p.uin[j], *accin = p.accin[j];
  for (int64_t b = t0; b < s.n; b += U * stride) {
    T v[U] = {}, u[U] = {}, c[U] = {};
    bool on[U];
#pragma unroll
    for (int i = 0; i < U; i++) on[i] = b + i * stride < s.n && s.imult[b + i * stride] == 1.0f;
#pragma unroll
    for (int i = 0; i < U; i++) {
      const int64_t m = b + i * stride;
      if (!on[i]) continue;
      v[i] = x[m];
      if (M::UIN) u[i] = uin[m];
      if (M::ACC) c[i] = accin[m];
    }
#pragma unroll
    for (int i = 0; i < U; i++) {
      const int64_t m = b + i * stride;
      if (!on[i]) continue;
      // folds of one member: 0 + v
      const T k = __fadd_rn_t(T(0), rk_value<T, MODE>(p, j, v[i], u[i], m));
      if constexpr (MODE == RK_LAST) {
        p.out[j][m] = __fadd_rn_t(T(0), rk_accum_point(c[i], k, p.ch));
      } else if constexpr (M::SAME) {
        p.out[j][m] = k;
      } else {
        const T o = MODE == RK_MIDS ? __fadd_rn_t(T(0), rk_input_point(u[i], p.b, k)) : T(0);
        rk_write<T, MODE>(p, j, k, o, v[i], u[i], c[i], m);
      }
    }
  }
}

}  // namespace gfk
