// rk_pass.cuh -- launch of the stage passes of k_dss.cuh and k_dss_elem.cuh.
#pragma once
#include <algorithm>

#include "k_dss_elem.cuh"

// One pass (RK_* or ADJ_*) on nc state components; GF_OK or an error code.
template <typename T>
int rk_pass(gf_problem *prob, int mode, int nc, const gfk::RKPass<T> &p, cudaStream_t st);

namespace gfk {

template <typename T, int MODE>
struct RKBoxLaunch {
  template <int N>
  struct F {
    static int run(gf_problem *prob, cudaStream_t st, int nc, const RKPass<T> &p) {
      const RunWalk<N - 1> w = RunWalk<N - 1>::make(prob->box);
      const RunGrid g = run_grid(prob, w);
      prob->launches++;
      k_rk_box<T, MODE, N - 1><<<g.blocks, g.block, 0, st>>>(p, nc, w, g);
      return GF_OK;
    }
  };
};

// Whether the element pass (k_dss_elem.cuh) takes a pass.  It writes coalesced
// but gathers each copy (N + 2)^3 / N^3 times, so it pays where a pass touches
// several arrays per copy: RK_MID and the reverse stages (40^3 elements, N = 6,
// three FP32 components: 236 us against 513 for the lattice walk; 12^3, N = 7,
// FP64: 19 against 47), RK_MIDS from N = 5 on (387 against 531; two gathers).
// RK_LAST (two gathers, one write), RK_SMOOTH and RK_EULER stay with the walk (74
// against 118, 155 against 180).  It reads arrays that other blocks' elements
// hold, so it must not write one of them.
template <typename T, int MODE>
inline bool elem_pass_ok(const gf_problem *prob, int nc, const RKPass<T> &p) {
  constexpr int least = el_min_n<MODE>();
  if constexpr (least > GF_MAXN) {
    return false;
  } else {
    if (prob->dim != 3 || prob->n < least) return false;
    for (int i = 0; i < nc; i++)
      for (int j = 0; j < nc; j++) {
        const T *in[2] = {p.x[i], MODE == RK_MIDS ? p.uin[i] : nullptr};
        for (const T *a : in)
          if (a && (a == p.out[j] || a == p.acc[j] || a == p.aux[j])) return false;
      }
    return true;
  }
}

template <typename T, int MODE>
inline int rk_pass_mode(gf_problem *prob, int nc, const RKPass<T> &p, cudaStream_t st) {
  BoxWalk w;
  if (dss_box_walk(prob, w)) {
    if (elem_pass_ok<T, MODE>(prob, nc, p))
      return dispatch_n<RKElemLaunch<T, MODE>::template F>(prob->n, prob, st, nc, p);
    return dispatch_n<RKBoxLaunch<T, MODE>::template F>(prob->n, prob, st, nc, p);
  }
  const SplitCls sc = split_of(prob);
  const int most = prob->ctx->sm_count * 8;
  const unsigned nbs = sc.nsh ? grid_for(sc.nsh, 256, most) : 0;
  const unsigned nbn = grid_for((sc.n + 3) / 4, 256, most);  // four nodes per thread
  prob->launches += nc;
  for (int j = 0; j < nc; j++) k_rk_split<T, MODE><<<nbs + nbn, 256, 0, st>>>(p, j, sc, nbs);
  return GF_OK;
}

}  // namespace gfk
