// k_cg_cluster.cuh -- one Jacobi-PCG solve (GCG::solve_impl's DFM iteration,
// solvers/gcg.ipp:239-382) of a 2-d affine box inside ONE thread-block
// cluster, from the initial residual to the stop test, in one launch.
//
// A 2-d solve of up to a few hundred thousand lattice points is bound by what
// separates its phases, not by its work: four dependent kernels per iteration
// (element apply, assembly and <w, q>, update, direction) cost 25 us at 26 k
// points on a B200, and a grid-wide barrier in a persistent kernel costs 3.3 us.
// The iteration runs on up to 16 SMs with three hardware cluster barriers:
//   1. q = mask A w on the lattice, <w, q>           | cluster sum -> alpha
//   2. x += alpha w, r -= alpha q, <r, z>, norm(r)   | cluster sum -> beta, stop
//   3. w = z + beta w                                | cluster barrier
// The apply works on the lattice directly, point by point: an x-line of
// element e contributes p Jac X0^2 W_ly (K1 w)_lx and a y-line likewise
// (K1 = D^T diag(W) D, k_helm_k1.cuh), summed over the one or two elements per
// direction that hold the point, so there is no element-local vector and no
// assembly pass.  A CTA owns whole lattice rows and holds w there, with the P
// rows on either side that its y-lines reach, in shared memory; a thread always
// owns the same points, with their x, r, q and Jacobi weight in registers when
// it has at most four.  Only the rows near a CTA's boundaries travel, through
// global memory between two barriers.  (With w, and everything else, read from
// global memory an iteration cost 10 us at 26 k points: every barrier
// invalidates the L1.)
//
// Sums are folded in a fixed order and every CTA forms the same scalars from the
// same partials: results are deterministic.
#pragma once
#include <cstdint>
#include <utility>

#include "gf_common.cuh"
#include "lattice.cuh"

namespace gfk {

constexpr int CL_THREADS = 512;
constexpr int CL_MAX = 16;  // CTAs per cluster (non-portable size; 8 elsewhere, cl_cluster_size)

__device__ __forceinline__ unsigned cl_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ unsigned cl_size() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}
// all threads of all CTAs; orders shared and global memory of the cluster
__device__ __forceinline__ void cl_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::
                   : "memory");
}
// v into the double at address p of this CTA's shared memory, in CTA `rank`
__device__ __forceinline__ void cl_store(double *p, unsigned rank, double v) {
  uint32_t a = (uint32_t)__cvta_generic_to_shared(p), b;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(b) : "r"(a), "r"(rank));
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(b), "d"(v) : "memory");
}

// Shared memory of one CTA: the partials of every warp of the cluster (two
// slots, used in turn, so that a slot is rewritten only after another cluster
// barrier), K1 with rows of odd length, W.
constexpr int CL_WARPS = CL_THREADS / 32;
struct ClShared {
  double part[2][2][CL_MAX * CL_WARPS];
  double K1[GF_MAXN * (GF_MAXN + 1)];
  double W[GF_MAXN];
  double geom[3];  // uniform geometry: Jac X0^2, Jac X1^2, Jac
};

// Cluster-wide totals of a (sum) and b (sum, or max), in every thread: every
// warp pushes its partials to all CTAs, the cluster barrier makes them visible
// (with the global writes before it), and every warp folds the same values in
// the same order.  No CTA-level barrier and no read of another CTA's memory.
__device__ __forceinline__ void cl_total(ClShared &sh, int slot, bool bmax, double &a, double &b) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, n = (int)cl_size();
  auto fold = [&](double &u, double &v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      u += __shfl_xor_sync(0xffffffffu, u, o);
      const double t = __shfl_xor_sync(0xffffffffu, v, o);
      v = bmax ? fmax(v, t) : v + t;
    }
  };
  fold(a, b);
  if (lane < n) {
    const int i = (int)cl_rank() * CL_WARPS + wid;
    cl_store(&sh.part[slot][0][i], lane, a);
    cl_store(&sh.part[slot][1][i], lane, b);
  }
  cl_sync();
  a = b = 0.0;
  for (int i = lane; i < n * CL_WARPS; i += 32) {
    a += sh.part[slot][0][i];
    const double t = sh.part[slot][1][i];
    b = bmax ? fmax(b, t) : b + t;
  }
  fold(a, b);
}

// One 2-d box problem with affine elements, its vectors on the lattice.
struct ClProblem {
  int ne0, ne1, per0, per1, M0, M1;
  FastDiv f0;            // by M0
  const double *egeom;   // dXidX0, dXidX1, Jac per element
  const uint8_t *mask;   // 1 keep, 0 Dirichlet; null: none
  const uint8_t *mult;   // element copies per point (EUC norm)
  const double *massL;   // assembled mass (L2, L1 norms)
  const double *dinv64;  // Jacobi inverse in FP64 or FP32; both null: none
  const float *dinv32;
  const double *b;       // assembled right-hand side
  double *x, *r, *w, *q;
  double p, qm;          // operator p L + qm M
  int normtype;
  double ntot, ivol;     // EUC: element-local nodes; L2, L1: 1/volume
  int uniform;           // every element has the geometry of the first
};

// shared memory for w: a CTA's rows, P more on either side, and a column that
// repeats the first (periodic x-lines)
__host__ __device__ inline size_t cl_slab_bytes(int M0, int M1, int P, int ctas) {
  return sizeof(double) * (size_t)(M0 + 1) * ((M1 + ctas - 1) / ctas + 2 * P);
}
constexpr size_t CL_SLAB_MAX = 208 * 1024;
// A CTA's work in one iteration, in points: its own and, at a third of their cost, the
// 2 P halo rows that it reads back.
inline double cl_work(int M0, int M1, int P, int ctas) {
  return M0 * ((M1 + ctas - 1) / ctas + 0.35 * 2 * P);
}
// Boxes whose single solve takes the cluster: where it beats the whole chip with a
// launch per pass.  Beside the lattice points there is a limit on a CTA's work, which
// a box wide in x reaches early, above all where its halo outweighs its rows (unless
// its points stay in registers, cl_solve_any: 400 x 2, p = 5: 27.9, 30.7).  Solves in
// ms, cluster against separate kernels (whose iterations come in batches, so that their
// time moves by a tenth from box to box): squares, 79 k points, p = 3: 0.80, 1.11,
// p = 5: 1.86, 2.01, p = 7: 3.13, 2.87; 75 k, p = 8: 3.71, 3.45; 68 k, p = 7: 2.57, 2.96,
// p = 10: 4.96, 4.79; 59 k, p = 9: 3.44, 3.79; 64 k, p = 11: 4.68, 5.37.  Wide: 400 x 8
// elements, p = 4 (53 k points): 22.4, 16.6; 700 x 20, p = 2 (57 k): 6.02, 5.35;
// 160 x 16, p = 5 (65 k): 7.25, 5.50; 60 x 12, p = 8 (47 k): 6.95, 6.74; 150 x 30, p = 4
// (73 k): 2.25, 2.54; 40 x 12, p = 8 (31 k): 4.53, 5.81; 300 x 9, p = 3 (25 k): 3.65, 6.55.
inline bool cl_fits(int M0, int M1, int P, int ctas) {
  const int64_t rows = (M1 + ctas - 1) / ctas, nL = (int64_t)M0 * M1;
  const double most = (rows >= 2 * P ? 6500.0 : 6050.0) * CL_MAX / ctas;
  return nL <= (P <= 6 ? 80000 : 68000) &&
         (M0 * rows <= 4 * CL_THREADS || cl_work(M0, M1, P, ctas) <= most) &&
         cl_slab_bytes(M0, M1, P, ctas) <= CL_SLAB_MAX;
}

inline ClProblem cl_problem(const BoxLattice &L) {
  ClProblem c{};
  c.ne0 = L.ne[0];
  c.ne1 = L.ne[1];
  c.per0 = L.per[0];
  c.per1 = L.per[1];
  c.M0 = (int)L.M[0];
  c.M1 = (int)L.M[1];
  c.f0 = FastDiv::make(c.M0);
  return c;
}

// (element, local index) pairs of lattice coordinate g along one direction
template <int P>
__device__ __forceinline__ int cl_cands(int g, int ne, int per, int (&e)[2], int (&l)[2]) {
  const int q = g / P, r = g - q * P;
  e[0] = q;
  l[0] = r;
  e[1] = 0;
  l[1] = 0;
  if (r != 0) return 1;
  const int left = q > 0 ? q - 1 : ne - 1;
  if (!per) {
    if (q == 0) return 1;
    e[0] = left;
    l[0] = P;
    e[1] = q;
    return q < ne ? 2 : 1;
  }
  e[1] = left;
  l[1] = P;
  return 2;
}

// (A v) at lattice point (g0, g1), A = p L + qm M assembled on the lattice; v
// points at the point's value, rows at stride b.M0 + 1
template <int N>
__device__ __forceinline__ double cl_apply(const ClProblem &b, const ClShared &sh,
                                           const double *v, int g0, int g1) {
  constexpr int P = N - 1, S = N | 1;
  const int ld = b.M0 + 1;
  int ex[2], lx[2], ey[2], ly[2];
  const int nx = cl_cands<P>(g0, b.ne0, b.per0, ex, lx);
  const int ny = cl_cands<P>(g1, b.ne1, b.per1, ey, ly);
  double cx[2] = {0.0, 0.0}, cy[2] = {0.0, 0.0}, cm = 0.0;
  if (b.uniform) {
    const double wx = sh.W[lx[0]] + (nx > 1 ? sh.W[lx[1]] : 0.0);
    const double wy = sh.W[ly[0]] + (ny > 1 ? sh.W[ly[1]] : 0.0);
    cx[0] = cx[1] = sh.geom[0] * wy;
    cy[0] = cy[1] = sh.geom[1] * wx;
    cm = sh.geom[2] * (wx * wy);
  } else {
#pragma unroll
    for (int j = 0; j < 2; j++) {
      if (j >= ny) break;
      const double wy = sh.W[ly[j]];
#pragma unroll
      for (int i = 0; i < 2; i++) {
        if (i >= nx) break;
        const double *ge = b.egeom + 3 * (ex[i] + b.ne0 * ey[j]);
        const double X0 = ge[0], X1 = ge[1], J = ge[2], wx = sh.W[lx[i]];
        cx[i] += J * wy * (X0 * X0);
        cy[j] += J * wx * (X1 * X1);
        cm += J * wx * wy;
      }
    }
  }
  double s = 0.0;
#pragma unroll
  for (int i = 0; i < 2; i++) {
    if (i >= nx) break;
    const double *K = sh.K1 + lx[i] * S, *a = v + (ex[i] * P - g0);
    double t = K[0] * a[0];
#pragma unroll
    for (int m = 1; m < N; m++) t = fma(K[m], a[m], t);
    s = fma(cx[i], t, s);
  }
#pragma unroll
  for (int j = 0; j < 2; j++) {
    if (j >= ny) break;
    const double *K = sh.K1 + ly[j] * S, *a = v - ly[j] * ld;
    double t = K[0] * a[0];
#pragma unroll
    for (int m = 1; m < N; m++) t = fma(K[m], a[m * ld], t);
    s = fma(cy[j], t, s);
  }
  return fma(b.qm * cm, *v, b.p * s);
}

__device__ __forceinline__ void cl_norm_add(const ClProblem &b, double &acc, double r, int c) {
  if (b.normtype == GF_NORM_INF) acc = fmax(acc, fabs(r));
  else if (b.normtype == GF_NORM_EUC) acc += (double)b.mult[c] * (r * r);
  else if (b.normtype == GF_NORM_L2) acc += b.massL[c] * (r * r);
  else acc += b.massL[c] * fabs(r);
}
__device__ __forceinline__ double cl_norm(const ClProblem &b, double v) {
  if (b.normtype == GF_NORM_INF) return v;
  if (b.normtype == GF_NORM_EUC) return sqrt(v / b.ntot);
  if (b.normtype == GF_NORM_L2) return sqrt(v * b.ivol);
  return v * b.ivol;
}
__device__ __forceinline__ double cl_dinv(const ClProblem &b, int c) {
  return b.dinv64 ? b.dinv64[c] : (b.dinv32 ? (double)b.dinv32[c] : 1.0);
}

struct ClState {
  double rho, rnorm, res;  // res: norm of the initial residual
  int iters;
  bool bad;  // a non-finite scalar
};

// K1, W and the geometry of a problem into shared memory (all threads; ends
// with a cluster barrier)
__device__ __forceinline__ void cl_load_basis(ClShared &sh, int N, const double *K1, const double *W,
                                              const ClProblem &b) {
  const int S = N | 1;
  for (int i = threadIdx.x; i < N * N; i += blockDim.x) sh.K1[(i / N) * S + i % N] = K1[i];
  for (int i = threadIdx.x; i < N; i += blockDim.x) sh.W[i] = W[i];
  if (threadIdx.x == 0) {
    const double X0 = b.egeom[0], X1 = b.egeom[1], J = b.egeom[2];
    sh.geom[0] = J * (X0 * X0);
    sh.geom[1] = J * (X1 * X1);
    sh.geom[2] = J;
  }
  cl_sync();  // also: every CTA has started before another stores into it
}

// The solve.  start(st) is called once, by every thread with the same values,
// after the initial residual (st.rho, st.res): it returns whether to iterate
// and sets rtol and maxit; the iteration ends at norm(r) <= rtol, maxit
// iterations or a non-finite scalar (st.bad).  hist (null: none) receives the
// norms.  slab: cl_slab_bytes of shared memory.  PT points per thread in
// registers, or PT = 0: any number, in the problem's vectors.
template <int N, int PT, class START>
__device__ void cl_solve(const ClProblem &b, ClShared &sh, double *slab, ClState &st, START start,
                         double *hist) {
  constexpr int P = N - 1, NP = PT > 0 ? PT : 1;
  const int M0 = b.M0, ld = M0 + 1, tid = (int)threadIdx.x;
  const int per = (b.M1 + (int)cl_size() - 1) / (int)cl_size();
  const int lo = min(b.M1, (int)cl_rank() * per), rows = min(per, b.M1 - lo);
  const int nown = rows * M0, c0 = lo * M0;
  const bool first = cl_rank() == 0 && tid == 0, inf = b.normtype == GF_NORM_INF;
  double *own = slab + P * ld;  // row lo
  // slab rows [s0, s1) from the lattice vector v (rows that exist)
  auto fetch = [&](const double *v, int s0, int s1) {
    for (int i = tid; i < (s1 - s0) * ld; i += CL_THREADS) {
      const int s = s0 + i / ld, x = i - (s - s0) * ld;
      int g = lo - P + s;
      if (b.per1) g = g < 0 ? g + b.M1 * ((-g + b.M1 - 1) / b.M1) : g % b.M1;
      if (g >= 0 && g < b.M1) slab[s * ld + x] = __ldcg(v + g * M0 + (x == M0 ? 0 : x));
    }
  };
  // f(i, k): own point i of the CTA, slot k of the registers
  auto points = [&](auto f) {
    if constexpr (PT > 0) {
#pragma unroll
      for (int k = 0; k < PT; k++)
        if (tid + k * CL_THREADS < nown) f(tid + k * CL_THREADS, k);
    } else {
#pragma unroll 4
      for (int i = tid; i < nown; i += CL_THREADS) f(i, 0);
    }
  };
  auto at = [&](int i, int &g0, int &r) {  // offset of own point i in the slab's own rows
    r = b.f0.div(i);
    g0 = i - r * M0;
    return r * ld + g0;
  };
  auto put = [&](int i, double w) {  // the direction at own point i
    int g0, row;
    const int s = at(i, g0, row);
    own[s] = w;
    if (g0 == 0) own[s + M0] = w;
    b.w[c0 + i] = w;
  };
  double xr[NP], rr[NP], qr[NP], dr[NP];
  (void)xr, (void)qr;
  fetch(b.x, 0, rows + 2 * P);
  __syncthreads();
  double rho = 0.0, rn = 0.0;
  points([&](int i, int k) {
    int g0, row;
    const int s = at(i, g0, row), c = c0 + i;
    const double r =
        !b.mask || b.mask[c] ? b.b[c] - cl_apply<N>(b, sh, own + s, g0, lo + row) : 0.0;
    const double d = cl_dinv(b, c);
    if (PT > 0) {
      xr[k] = own[s];
      rr[k] = r;
      dr[k] = d;
    } else {
      b.r[c] = r;
    }
    rho += r * (d * r);
    cl_norm_add(b, rn, r, c);
  });
  __syncthreads();  // the slab turns from x to w
  points([&](int i, int k) {
    put(i, PT > 0 ? dr[k] * rr[k] : cl_dinv(b, c0 + i) * b.r[c0 + i]);
  });
  cl_total(sh, 1, inf, rho, rn);
  st.rho = rho;
  st.res = st.rnorm = cl_norm(b, rn);
  st.iters = 0;
  st.bad = !isfinite(rho) || !isfinite(st.res);
  double rtol = 0.0;
  int maxit = 0;
  bool run = start(st, rtol, maxit) && maxit > 0;
  while (run) {
    fetch(b.w, 0, P);
    fetch(b.w, rows + P, rows + 2 * P);
    __syncthreads();
    double wq = 0.0, unused = 0.0;
    points([&](int i, int k) {
      int g0, row;
      const int s = at(i, g0, row), c = c0 + i;
      const double q =
          !b.mask || b.mask[c] ? cl_apply<N>(b, sh, own + s, g0, lo + row) : 0.0;
      if (PT > 0) qr[k] = q;
      else b.q[c] = q;
      wq += own[s] * q;
    });
    cl_total(sh, 0, false, wq, unused);
    const double alpha = st.rho / wq;
    if (!isfinite(alpha)) {
      st.bad = true;
      break;
    }
    rho = rn = 0.0;
    points([&](int i, int k) {
      int g0, row;
      const int s = at(i, g0, row), c = c0 + i;
      double r, d;
      if (PT > 0) {
        xr[k] = fma(alpha, own[s], xr[k]);
        r = rr[k] = fma(-alpha, qr[k], rr[k]);
        d = dr[k];
      } else {
        b.x[c] = fma(alpha, own[s], b.x[c]);
        r = fma(-alpha, b.q[c], b.r[c]);
        b.r[c] = r;
        d = cl_dinv(b, c);
      }
      rho += r * (d * r);
      cl_norm_add(b, rn, r, c);
    });
    cl_total(sh, 1, inf, rho, rn);
    const double beta = rho / st.rho;
    st.rho = rho;
    st.rnorm = cl_norm(b, rn);
    if (hist && first) hist[st.iters] = st.rnorm;
    st.iters++;
    st.bad = !isfinite(beta) || !isfinite(st.rnorm);
    if (st.bad || st.rnorm <= rtol || st.iters >= maxit) break;
    points([&](int i, int k) {
      int g0, row;
      const int s = at(i, g0, row);
      const double z = PT > 0 ? dr[k] * rr[k] : cl_dinv(b, c0 + i) * b.r[c0 + i];
      put(i, fma(beta, own[s], z));
    });
    cl_sync();
  }
  if constexpr (PT > 0) points([&](int i, int k) { b.x[c0 + i] = xr[k]; });
}

// cl_solve with the points in registers where they fit
template <int N, class START>
__device__ __forceinline__ void cl_solve_any(const ClProblem &b, ClShared &sh, double *slab,
                                             ClState &st, START start, double *hist) {
  const int per = (b.M1 + (int)cl_size() - 1) / (int)cl_size();
  if (per * b.M0 <= 4 * CL_THREADS) cl_solve<N, 4>(b, sh, slab, st, start, hist);
  else cl_solve<N, 0>(b, sh, slab, st, start, hist);
}

// CTAs per cluster that this kernel can be launched with, given the most dynamic
// shared memory that it is ever launched with: 16, the portable 8, or 0 (a device
// or a partition of one whose GPCs have too few SMs for that memory: the caller
// then takes the separate kernels).
template <typename K>
inline int cl_cluster_size(K kern, int threads, size_t smem) {
  static KernelRecord<int> sizes;  // of the kernels of this type
  int device = 0;
  cudaGetDevice(&device);
  return cluster_size_for(sizes, device, (const void *)kern, [&](int size) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(size);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = size;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int n = 0;
    const bool ok =
        set_smem(kern, smem) &&
        cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, size > 8) ==
            cudaSuccess &&
        cudaOccupancyMaxActiveClusters(&n, kern, &cfg) == cudaSuccess && n > 0;
    if (!ok) cudaGetLastError();
    return ok;
  });
}

template <typename... Exp, typename... Act>
inline cudaError_t cl_launch(void (*kern)(Exp...), int clusters, int size, int threads,
                             size_t smem, cudaStream_t st, Act &&...args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(clusters * size));
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)size;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, std::forward<Act>(args)...);
}

}  // namespace gfk
