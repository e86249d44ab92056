// rk_cluster.cuh -- the RK steps of a small 2-d box inside one thread-block
// cluster, all steps of an advance in one launch.
//
// A step of a small grid is a chain of short dependent kernels (a right-hand
// side and a class pass per stage, 3-4 us each where their work is a fraction of
// one), so it is bound by the launches.  One cluster of up to 16 SMs runs the
// same two bodies (dudt2d_group, k_dudt.cuh; rk_run, k_dss.cuh) with its
// hardware barrier between them.  Same arithmetic node by node as the separate
// kernels: bit-identical.
#pragma once
#include "k_cg_cluster.cuh"
#include "k_dss.cuh"
#include "k_dudt.cuh"

namespace gfk {

constexpr int RKC_THREADS = 256;
// Grids that take the cluster: above them the 148 SMs of the separate kernels win.
// One component is bound by the right-hand side's share of an SM (nodes), more of them
// also by the class passes (nodes times components).  The crossover moves with the
// order (whether a CTA's elements fit one group), the scheme, and by a tenth with the
// host, whose launches the separate kernels wait for (some 5 us each); over 812 grids of
// p = 1 to 11 these limits leave 0.7 % of time on average against the better side, at
// most a fifth.  Eight steps in us, cluster against separate kernels (FP64): advection
// p = 4, RK4, 12.1 k nodes 310, 339, 16.9 k 326, 344, 20.3 k 362, 345; p = 7, 14.4 k
// 304, 352, 17.4 k 397, 354, 19.6 k 416, 359; Burgers (two components) RK4, p = 5,
// 9.2 k nodes 369, 394, 13.7 k 471, 423, p = 3, 8.8 k 385, 334, p = 7, 17.4 k 606, 406;
// SSP33, p = 3, 12.1 k 253, 263, p = 5, 13.7 k 331, 311, p = 9, 14.4 k 305, 362, p = 7,
// 17.4 k 389, 312; 40 k values, p = 2, SSP33: 480, 214.
constexpr int64_t RKC_NODES = 18000, RKC_VALUES = 28000, RKC_VALUES_SSP = 30000;
inline bool rk_cluster_fits(int64_t n, int nstate, bool ssp) {
  return n <= RKC_NODES && n * nstate <= (ssp ? RKC_VALUES_SSP : RKC_VALUES);
}

// one stage: the right-hand side of in -> out, then the class pass
template <typename T>
struct RKPhase {
  const T *in[3];
  T *out[3];
  RKPass<T> pass;
  int mode;
};
template <typename T>
struct RKProgram {
  RKPhase<T> ph[4];
  int nph, nc, nsteps, epb;
  const T *c[2], *imass;
  Geom<T> g;
  int64_t ne;
  T nu;
};

template <typename T, int N, int EQN>
__global__ void __launch_bounds__(RKC_THREADS)
    k_rk_cluster(const __grid_constant__ Basis<T, N> B, const __grid_constant__ RKProgram<T> pr,
                 const RunWalk<N - 1> w) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ T sW[N];
  T *sm = reinterpret_cast<T *>(smem_raw);
  if (threadIdx.x < N) sW[threadIdx.x] = B.W[threadIdx.x];
  const int rank = (int)cl_rank(), size = (int)cl_size();
  const int t0 = rank * RKC_THREADS + (int)threadIdx.x, dt = size * RKC_THREADS;
  for (int s = 0; s < pr.nsteps; s++)
    for (int i = 0; i < pr.nph; i++) {
      const RKPhase<T> &h = pr.ph[i];
      for (int64_t e0 = (int64_t)rank * pr.epb; e0 < pr.ne; e0 += (int64_t)size * pr.epb) {
        const int nel = pr.ne - e0 < pr.epb ? (int)(pr.ne - e0) : pr.epb;
        for (int j = 0; j < (EQN == GF_EQN_HEAT ? pr.nc : 1); j++) {
          dudt2d_group<T, N, EQN, MODE_DUDT>(B, pr.g, e0, nel, pr.nu, h.in[j],
                                             EQN == GF_EQN_ADVECT ? pr.c[0] : h.in[1], pr.c[1],
                                             pr.imass, h.out[j], h.out[1], sm, sW);
          __syncthreads();  // before the next group reuses shared memory
        }
      }
      cl_sync();
      for (int t = t0; t < w.n; t += dt) {
        const LatRun k = w.run(t);
        if (h.mode == RK_EULER) rk_run<T, RK_EULER, N - 1>(h.pass, pr.nc, w, k);
        else if (h.mode == RK_MID) rk_run<T, RK_MID, N - 1>(h.pass, pr.nc, w, k);
        else if (h.mode == RK_MIDS) rk_run<T, RK_MIDS, N - 1>(h.pass, pr.nc, w, k);
        else rk_run<T, RK_LAST, N - 1>(h.pass, pr.nc, w, k);
      }
      cl_sync();
    }
}

template <typename T>
struct RKClusterLaunch {
  template <int N>
  struct F {
    static int run(gf_problem *prob, int eqn, RKProgram<T> &pr, cudaStream_t st) {
      if (eqn == GF_EQN_ADVECT) return go<GF_EQN_ADVECT>(prob, pr, st);
      if (eqn == GF_EQN_BURGERS) return go<GF_EQN_BURGERS>(prob, pr, st);
      return go<GF_EQN_HEAT>(prob, pr, st);
    }
    template <int EQN>
    static int go(gf_problem *prob, RKProgram<T> &pr, cudaStream_t st) {
      gf_context *ctx = prob->ctx;
      auto kern = k_rk_cluster<T, N, EQN>;
      // elements per group: all CTAs busy, at most 2 N threads per element
      constexpr int most = RKC_THREADS / (2 * N);
      const int size = cl_cluster_size(kern, RKC_THREADS, sizeof(T) * dudt2_words<N, EQN>() * most);
      if (!size) return GF_ERR_UNSUPPORTED;
      pr.epb = (int)std::min<int64_t>(most, (prob->ne + size - 1) / size);
      const size_t smem = sizeof(T) * dudt2_words<N, EQN>() * pr.epb;
      const Basis<T, N> B = make_basis<T, N>(prob);
      const RunWalk<N - 1> w = RunWalk<N - 1>::make(prob->box);
      prob->launches++;
      GF_CUDA(ctx, cl_launch(kern, 1, size, RKC_THREADS, smem, st, B, pr, w));
      return GF_OK;
    }
  };
};

}  // namespace gfk

// GF_ERR_UNSUPPORTED, with nothing launched, on a device that holds no such cluster
template <typename T>
int launch_rk_cluster(gf_problem *prob, int eqn, gfk::RKProgram<T> &pr, cudaStream_t st);
