// api_rk.cu -- explicit Runge-Kutta steps of GExRKStepper
// (pdes/gexrk_stepper.ipp) on the GBurgers right-hand side, with the DSS
// Smooth calls exactly where the reference places them:
//   Butcher step_b (1)  (gexrk_stepper.ipp:252-341), tableau of
//                       GButcherRK::computeCoeffs (gbutcherrk.ipp:69-125)
//   SSP22 / SSP33 / SSP34 (gexrk_stepper.ipp:533-780), step_euler (809-819)
// and GBurgers::step_impl (gburgers.ipp:275-333).
//
// Per stage: the fused element kernel of the RHS (k_dudt*) and one class pass
// (rk_pass.cuh) that smooths its result and forms the next stage's input and the
// running sum; the step reads its input state and writes the result, in place
// where they are the same.
#include <algorithm>
#include <cstring>
#include <vector>

#include "gf_common.cuh"
#include "k_dss.cuh"
#include "k_vec.cuh"
#include "ops_launch.cuh"
#include "rk_cluster.cuh"
#include "rk_common.cuh"
#include "rk_pass.cuh"

using namespace gfk;

namespace gfrk {

// slot of the problem's host scalar block holding the RK non-finite flag
constexpr int RK_FLAG_SLOT = 62;

void butcher(int order, double *alpha, double beta[4][4], double *c) {
  std::memset(beta, 0, sizeof(double) * 16);
  for (int i = 0; i < 4; i++) alpha[i] = c[i] = 0.0;
  if (order == 1) {
    c[0] = 1.0;
  } else if (order == 2) {
    c[0] = 0.5;
    alpha[1] = 1.0;
    c[1] = 0.5;
    beta[1][0] = 1.0;
  } else if (order == 3) {
    c[0] = 0.25;
    alpha[1] = 1.0 / 3.0;
    c[1] = 0.0;
    alpha[2] = 2.0 / 3.0;
    c[2] = 0.75;
    beta[1][0] = 1.0 / 3.0;
    beta[2][1] = 2.0 / 3.0;
  } else {
    c[0] = 1.0 / 6.0;
    alpha[1] = 0.5;
    c[1] = 1.0 / 3.0;
    alpha[2] = 0.5;
    c[2] = 1.0 / 3.0;
    alpha[3] = 1.0;
    c[3] = 1.0 / 6.0;
    beta[1][0] = 0.5;
    beta[2][1] = 0.5;
    beta[3][2] = 1.0;
  }
}

// y = uin + ((0 + b0 K0) + b1 K1 + ...)   (isum accumulation of step_b)
template <typename T>
__global__ void k_stage_sum(int64_t n, const T *__restrict__ uin, int nk, const T *__restrict__ K0,
                            const T *__restrict__ K1, const T *__restrict__ K2, T b0, T b1, T b2,
                            T *__restrict__ y) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    y[i] = rk_stage_point(uin[i], nk, K0, K1, K2, b0, b1, b2, i);
}

// flag[0] = 1 when any of the nstate fields holds a non-finite value
// (GBurgers::step_impl asserts isfinite on the evolved state after every
// step, gburgers.ipp:325-331).  Only a bad value writes the flag.  16-byte
// loads where the field is aligned to them, several in flight per thread
// (scalar: 59 us for three FP32 fields of 13.8 M values, 25 at HBM rate).
template <typename T>
__global__ void __launch_bounds__(256)
    k_nonfinite(int64_t n, int nstate, const T *u0, const T *u1, const T *u2, double *flag) {
  constexpr int V = 16 / sizeof(T);
  struct alignas(16) Vec {
    T v[V];
  };
  const T *const u[3] = {u0, u1, u2};
  const int64_t t0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  bool bad = false;
#pragma unroll
  for (int f = 0; f < 3; f++) {
    if (f >= nstate) break;
    const int64_t nv = reinterpret_cast<uintptr_t>(u[f]) % 16 == 0 ? n / V : 0;
#pragma unroll 4
    for (int64_t i = t0; i < nv; i += stride) {
      const Vec q = reinterpret_cast<const Vec *>(u[f])[i];
#pragma unroll
      for (int k = 0; k < V; k++) bad |= !isfinite(q.v[k]);
    }
    for (int64_t i = nv * V + t0; i < n; i += stride) bad |= !isfinite(u[f][i]);
  }
  if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) flag[0] = 1.0;
}

template <typename T>
struct AdvLaunch {
  template <int N>
  struct F {
    static int run(gf_problem *prob, const T *u, const T *b0, const T *b1, T *out,
                   cudaStream_t st) {
      const Basis<T, N> B = make_basis<T, N>(prob);
      prob->launches++;
      constexpr int EPB = epb2l<N>();
      k_adv_def<T, N, EPB, LoadE<T>>
          <<<(unsigned)((prob->ne + EPB - 1) / EPB), 2 * N * EPB, 0, st>>>(B, prob->ne, LoadE<T>{u},
                                                                          b0, b1, out);
      return GF_OK;
    }
  };
};

template <typename T>
struct AdvCoefLaunch {
  template <int N>
  struct F {
    static int run(gf_problem *prob, const T *const *c, T *b0, T *b1, cudaStream_t st) {
      const Basis<T, N> B = make_basis<T, N>(prob);
      prob->launches++;
      k_adv_coef<T, N><<<grid_for(prob->nlocal, 256, prob->ctx->sm_count * 8), 256, 0, st>>>(
          B, def_of<T>(prob), c[0], c[1], c[2], imass_of<T>(prob), b0, b1);
      return GF_OK;
    }
  };
};

template <typename T>
int adv_coef_launch(gf_problem *prob, const T *const *c, T *b0, T *b1, cudaStream_t st) {
  return dispatch_n<AdvCoefLaunch<T>::template F>(prob->n, prob, c, b0, b1, st);
}
template int adv_coef_launch<double>(gf_problem *, const double *const *, double *, double *,
                                     cudaStream_t);
template int adv_coef_launch<float>(gf_problem *, const float *const *, float *, float *,
                                    cudaStream_t);

template <typename T>
bool Stepper<T>::adv_ok() const {
  if (eqn != GF_EQN_ADVECT || nu != T(0) || prob->geom < GF_GEOM_DEFORMED || prob->dim != 2)
    return false;
  for (int k = 0; k < gf_nvel(prob); k++)
    if (!c[k]) return false;
  return true;
}

template <typename T>
bool Stepper<T>::prepare_adv() {
  advb[0] = advb[1] = nullptr;
  if (!adv_ok() || !advbuf[0] || !advbuf[1]) return false;
  const T *cc[3] = {c[0], c[1], gf_nvel(prob) > 2 ? c[2] : nullptr};
  if (adv_coef_launch<T>(prob, cc, advbuf[0], advbuf[1], st)) return false;
  advb[0] = advbuf[0];
  advb[1] = advbuf[1];
  return true;
}

template <typename T>
int Stepper<T>::rhs(T *const *u, T *const *K) {
  const T *f[4] = {nullptr, nullptr, nullptr, nullptr};
  T *o[3] = {nullptr, nullptr, nullptr};
  if (eqn == GF_EQN_ADVECT && advb[0])
    return dispatch_n<AdvLaunch<T>::template F>(prob->n, prob, (const T *)u[0],
                                                (const T *)advb[0], (const T *)advb[1], K[0], st);
  if (eqn == GF_EQN_ADVECT) {
    f[0] = u[0];
    for (int k = 0; k < gf_nvel(prob); k++) f[1 + k] = c[k];
    o[0] = K[0];
    return launch_dudt<T>(prob, eqn, 0, nu, f, o, st);
  }
  if (eqn == GF_EQN_HEAT) {
    for (int k = 0; k < nstate; k++) {
      const T *fk[4] = {u[k], nullptr, nullptr, nullptr};
      T *ok[3] = {K[k], nullptr, nullptr};
      int rc = launch_dudt<T>(prob, eqn, 0, nu, fk, ok, st);
      if (rc) return rc;
    }
    return GF_OK;
  }
  for (int k = 0; k < gf_nvel(prob); k++) {
    f[k] = u[k];
    o[k] = K[k];
  }
  return launch_dudt<T>(prob, eqn, 0, nu, f, o, st);
}

template <typename T>
bool Stepper<T>::rhs_euler_smooth(T *const *u, T *const *x, T dt, T *const *uin, T a,
                                  T *const *y, T b, T a2, T *const *y2, T b2, int *rc) {
  // FP32 only: measured on B200 (64^3 p=5 SSP-RK3 Burgers), the fused
  // epilogue takes an FP32 stage from 1.96 to 1.75 ms but an FP64 one from
  // 3.28 to 3.59 ms (the FP64 RHS kernel, at 104-109 registers and 3 blocks
  // per SM, absorbs the extra loads badly)
  if (sizeof(T) != 4 || prob->dim != 3 || prob->geom >= GF_GEOM_DEFORMED) return false;
  auto epi_for = [&](int k0, int nk) {
    RKEpi<T> e{};
    for (int j = 0; j < nk; j++) {
      e.uin[j] = uin[k0 + j];
      e.y[j] = y ? y[k0 + j] : nullptr;
      e.y2[j] = y2 ? y2[k0 + j] : nullptr;
    }
    e.dt = dt;
    e.a = a;
    e.b = b;
    e.a2 = a2;
    e.b2 = b2;
    e.uin_is_u = 1;
    for (int j = 0; j < nk; j++)
      if (uin[k0 + j] != u[k0 + j]) e.uin_is_u = 0;
    return e;
  };
  const T *f[4] = {nullptr, nullptr, nullptr, nullptr};
  T *o[3] = {nullptr, nullptr, nullptr};
  if (eqn == GF_EQN_HEAT) {
    for (int k = 0; k < nstate; k++) {
      const T *fk[4] = {u[k], nullptr, nullptr, nullptr};
      T *ok[3] = {utmp[k], nullptr, nullptr};
      const RKEpi<T> e = epi_for(k, 1);
      if ((*rc = launch_dudt<T>(prob, eqn, MODE_EULER, nu, fk, ok, st, &e))) return true;
    }
  } else {
    if (eqn == GF_EQN_ADVECT) {
      f[0] = u[0];
      for (int k = 0; k < gf_nvel(prob); k++) f[1 + k] = c[k];
      o[0] = utmp[0];
    } else {
      for (int k = 0; k < gf_nvel(prob); k++) {
        f[k] = u[k];
        o[k] = utmp[k];
      }
    }
    const RKEpi<T> e = epi_for(0, nstate);
    if ((*rc = launch_dudt<T>(prob, eqn, MODE_EULER, nu, f, o, st, &e))) return true;
  }
  *rc = smooth_to(utmp, x);
  return true;
}

// v <- Smooth(v) in place
template <typename T>
int Stepper<T>::smooth_n(T *const *v) {
  return smooth_to(v, v);
}

template <typename T>
int Stepper<T>::smooth_to(T *const *v, T *const *out) {
  RKPass<T> p{};
  for (int k = 0; k < nstate; k++) {
    p.x[k] = v[k];
    p.out[k] = out[k];
  }
  return rk_pass<T>(prob, RK_SMOOTH, nstate, p, st);
}

template <typename T>
int Stepper<T>::euler_smooth_n(T *const *x, T *const *out, T dt, T *const *uin, T a, T *const *y,
                               T b, T a2, T *const *y2, T b2) {
  RKPass<T> p{};
  for (int k = 0; k < nstate; k++) {
    p.x[k] = x[k];
    p.out[k] = out[k];
    p.uin[k] = uin[k];
    p.y[k] = y ? y[k] : nullptr;
    p.y2[k] = y2 ? y2[k] : nullptr;
  }
  p.dt = dt;
  p.a = a;
  p.b = b;
  p.a2 = a2;
  p.b2 = b2;
  return rk_pass<T>(prob, RK_EULER, nstate, p, st);
}

template <typename T>
int Stepper<T>::stage_pass(int mode, T *const *x, T *const *accin, T ch, T *const *accout,
                           T *const *uin, T b, T *const *out) {
  RKPass<T> p{};
  for (int k = 0; k < nstate; k++) {
    p.x[k] = x[k];
    p.accin[k] = accin[k];
    p.acc[k] = accout ? accout[k] : nullptr;
    p.uin[k] = uin ? uin[k] : nullptr;
    p.out[k] = out[k];
  }
  p.ch = ch;
  p.b = b;
  return rk_pass<T>(prob, mode, nstate, p, st);
}

template <typename T>
bool Stepper<T>::constrains() const {
  return prob->geom == GF_GEOM_EMBEDDED && nstate >= 3 && prob->xyz_d;
}

template <typename T>
void Stepper<T>::constrain(T *const *u) {
  if (!constrains()) return;
  const T *x = sizeof(T) == 8 ? (const T *)prob->xyz_d : (const T *)prob->xyz_f;
  const unsigned g = grid_for(n, 256, prob->ctx->sm_count * 8);
  prob->launches++;
  k_constrain2sphere<T><<<g, 256, 0, st>>>(n, u[0], u[1], u[2], x, x + n, x + 2 * n);
}

template <typename T>
bool Stepper<T>::alloc() {
  const size_t bytes = sizeof(T) * n;
  int slot = 30 + (sizeof(T) == 8 ? 0 : 20);
  // step_b keeps one slope (its accumulated state in uacc); the SSP schemes
  // the results of all substeps but the last
  const int nK = scheme <= 4 ? 1 : stages() - 1;
  for (int k = 0; k < nstate; k++, slot += 5) {
    if (scheme <= 4 && !(uacc[k] = (T *)gf_work(prob, slot, bytes))) return false;
    if (!(utmp[k] = (T *)gf_work(prob, slot + 1, bytes))) return false;
    for (int j = 0; j < nK; j++)
      if (!(K[j][k] = (T *)gf_work(prob, slot + 2 + j, bytes))) return false;
  }
  if (adv_ok()) {
    const int s2 = sizeof(T) == 8 ? 70 : 72;
    advbuf[0] = (T *)gf_work(prob, s2, bytes);
    advbuf[1] = (T *)gf_work(prob, s2 + 1, bytes);
    if (!advbuf[0] || !advbuf[1]) return false;
  }
  return true;
}

// One step uin -> uout (which may be uin).
template <typename T>
int Stepper<T>::step(T *const *uin, T *const *uout, T dt, T *const *tape) {
  int rc;
  auto copy = [&](T *const *dst, T *const *src) {  // a caller's tape may hold uin already
    for (int k = 0; k < nstate; k++)
      if (dst[k] != src[k])
        cudaMemcpyAsync(dst[k], src[k], sizeof(T) * n, cudaMemcpyDeviceToDevice, st);
  };
  if (scheme >= 1 && scheme <= 4) {
    double alpha[4], beta[4][4], cc[4];
    butcher(scheme, alpha, beta, cc);
    const int ns = scheme;
    const T h = dt;
    // stage inputs go to the tape when one is given; stage 0's is uin itself
    auto stage_in = [&](int m) { return tape ? tape + 3 * m : (T *const *)utmp; };
    T *const *um = uin, *const *acc = uin;
    if (ns == 1 || tape || constrains()) {
      um = stage_in(0);
      if (ns == 1 && um[0] == uin[0]) copy(acc = utmp, uin);  // smoothed in place below
      copy(um, uin);
      if (ns == 1 && (rc = smooth_n(um))) return rc;
      constrain(um);
    }
    for (int m = 0; m < ns - 1; m++) {
      if ((rc = rhs(um, K[0]))) return rc;
      // the tableaux here have one term per stage: beta[m+1][m]
      um = stage_in(m + 1);
      rc = stage_pass(m == ns - 2 ? RK_MIDS : RK_MID, K[0], acc, (T)cc[m] * h, uacc, uin,
                      (T)beta[m + 1][m] * h, um);
      if (rc) return rc;
      acc = uacc;
      constrain(um);
      constrain(uacc);
    }
    if ((rc = rhs(um, K[0]))) return rc;
    rc = stage_pass(RK_LAST, K[0], acc, (T)cc[ns - 1] * h, nullptr, nullptr, T(0), uout);
    if (rc) return rc;
    constrain(uout);
    return GF_OK;
  }
  // SSP stage inputs are uin and the substep results left in K[0..ns-2]
  if (tape) {
    if ((rc = step_ssp(uin, uout, dt))) return rc;
    copy(tape, uin);
    for (int m = 1; m < stages(); m++) copy(tape + 3 * m, K[m - 1]);
    return GF_OK;
  }
  return step_ssp(uin, uout, dt);
}

// One SSP substep: x = Smooth(update(dudt(u))), as the RHS call followed by
// euler_smooth_n, or in two passes (the RHS kernel writing the update,
// then the Smooth) where the RHS kernel has the fused epilogue.  x may be y
// or y2 (a step in place): both forms read a node's or class's y before they
// write it.
template <typename T>
static int ssp_substep(Stepper<T> &S, T *const *u, T *const *x, T dt, T *const *uin, T a,
                       T *const *y, T b, T a2, T *const *y2, T b2) {
  int rc = GF_OK;
  if (S.rhs_euler_smooth(u, x, dt, uin, a, y, b, a2, y2, b2, &rc)) return rc;
  if ((rc = S.rhs(u, S.utmp))) return rc;
  return S.euler_smooth_n(S.utmp, x, dt, uin, a, y, b, a2, y2, b2);
}

// Substep m of the SSP schemes (gexrk_stepper.ipp:533-780): from stage input
// s_m to s_{m+1} = Smooth(a (dt dudt(s_m) + s_m) + b s_y + b2 s_y2), s_0 the
// step's input (y or y2 -1: no such term).
template <typename T>
struct SSPSubstep {
  T a, b, b2;
  int y, y2;
};
template <typename T>
static SSPSubstep<T> ssp_coeffs(int scheme, int m) {
  const T h = T(0.5);
  if (scheme == GF_SSP22 && m == 1) return {h, h, T(0), 0, -1};
  if (scheme == GF_SSP33 && m == 1) return {T(0.25), T(0.75), T(0), 0, -1};
  if (scheme == GF_SSP33 && m == 2) return {T(2.0 / 3.0), T(1.0 / 3.0), T(0), 0, -1};
  if (scheme == GF_SSP34) {
    if (m == 2) return {T(1.0 / 6.0), T(1.0 / 6.0), T(2.0 / 3.0), 2, 0};
    return {h, h, T(0), m, -1};
  }
  return {T(1), T(0), T(0), -1, -1};
}

template <typename T>
int Stepper<T>::step_ssp(T *const *uin, T *const *uout, T dt) {
  const int ns = stages();
  auto state = [&](int i) -> T *const * { return i == 0 ? uin : K[i - 1]; };
  for (int m = 0; m < ns; m++) {
    const SSPSubstep<T> q = ssp_coeffs<T>(scheme, m);
    int rc = ssp_substep<T>(*this, state(m), m + 1 < ns ? (T *const *)K[m] : uout, dt, state(m), q.a,
                            q.y >= 0 ? state(q.y) : nullptr, q.b, T(1),
                            q.y2 >= 0 ? state(q.y2) : nullptr, q.b2);
    if (rc) return rc;
  }
  return GF_OK;
}

// Small 2-d boxes with a diagonal metric take all steps in one cluster
// (rk_cluster.cuh); step_b of order 1 smooths its input first and does not.
template <typename T>
bool Stepper<T>::cluster_ok() const {
  BoxWalk w;
  return prob->dim == 2 && prob->geom <= GF_GEOM_REGULAR && scheme != GF_RK1 &&
         rk_cluster_fits(n, nstate, scheme > 4) && dss_box_walk(prob, w);
}

template <typename T>
int Stepper<T>::cluster_steps(T *const *u, T dt, int nsteps) {
  RKProgram<T> pr{};
  pr.nsteps = nsteps;
  pr.nc = nstate;
  pr.c[0] = c[0];
  pr.c[1] = c[1];
  pr.imass = imass_of<T>(prob);
  pr.g = geom_of<T>(prob);
  pr.ne = prob->ne;
  pr.nu = nu;
  pr.nph = stages();
  auto set = [&](auto &dst, T *const *src) {
    for (int k = 0; k < nstate; k++) dst[k] = src[k];
  };
  if (scheme <= 4) {  // step()'s stages, in place
    double alpha[4], beta[4][4], cc[4];
    butcher(scheme, alpha, beta, cc);
    for (int m = 0; m < scheme; m++) {
      RKPhase<T> &h = pr.ph[m];
      set(h.in, m ? (T *const *)utmp : u);
      set(h.out, K[0]);
      set(h.pass.x, K[0]);
      set(h.pass.accin, m ? (T *const *)uacc : u);
      h.pass.ch = (T)cc[m] * dt;
      if (m == scheme - 1) {
        h.mode = RK_LAST;
        set(h.pass.out, u);
        continue;
      }
      h.mode = m == scheme - 2 ? RK_MIDS : RK_MID;
      set(h.pass.acc, uacc);
      set(h.pass.uin, u);
      set(h.pass.out, utmp);
      h.pass.b = (T)beta[m + 1][m] * dt;
    }
  } else {
    for (int m = 0; m < pr.nph; m++) {
      RKPhase<T> &h = pr.ph[m];
      const SSPSubstep<T> q = ssp_coeffs<T>(scheme, m);
      auto state = [&](int i) { return i == 0 ? u : (T *const *)K[i - 1]; };  // stage inputs
      set(h.in, state(m));
      set(h.out, utmp);
      h.mode = RK_EULER;
      set(h.pass.x, utmp);
      set(h.pass.uin, state(m));
      if (q.y >= 0) set(h.pass.y, state(q.y));
      if (q.y2 >= 0) set(h.pass.y2, state(q.y2));
      set(h.pass.out, m + 1 < pr.nph ? (T *const *)K[m] : u);
      h.pass.dt = dt;
      h.pass.a = q.a;
      h.pass.b = q.b;
      h.pass.a2 = T(1);
      h.pass.b2 = q.b2;
    }
  }
  return launch_rk_cluster<T>(prob, eqn, pr, st);
}

template struct Stepper<double>;
template struct Stepper<float>;

int check_traits(gf_problem *prob, const gf_rk_traits *tr, const void *const *u, const void *const *c) {
  gf_context *ctx = prob->ctx;
  GF_REQUIRE(ctx, tr && u, "traits and u are required");
  GF_REQUIRE(ctx, tr->eqn == GF_EQN_ADVECT || tr->eqn == GF_EQN_BURGERS || tr->eqn == GF_EQN_HEAT,
             "unknown equation %d", tr->eqn);
  const int s = tr->scheme;
  GF_REQUIRE(ctx, (s >= 1 && s <= 4) || s == GF_SSP22 || s == GF_SSP33 || s == GF_SSP34,
             "unknown RK scheme %d", s);
  if (tr->eqn == GF_EQN_BURGERS)
    GF_REQUIRE(ctx, tr->nstate == gf_nvel(prob),
               "Burgers evolves one component per physical coordinate");
  else if (tr->eqn == GF_EQN_ADVECT)
    GF_REQUIRE(ctx, tr->nstate == 1 && c, "pure advection: one component and dim velocities");
  else
    GF_REQUIRE(ctx, tr->nstate >= 1 && tr->nstate <= 3, "heat: 1..3 components");
  for (int k = 0; k < tr->nstate; k++) GF_REQUIRE(ctx, u[k], "state component %d missing", k);
  if (tr->eqn == GF_EQN_ADVECT)
    for (int k = 0; k < gf_nvel(prob); k++) GF_REQUIRE(ctx, c[k], "velocity component %d missing", k);
  return GF_OK;
}

template <typename T>
int advance(gf_problem *prob, const gf_rk_traits *tr, void *const *u, const void *const *c,
            double dt, int nsteps) {
  gf_context *ctx = prob->ctx;
  Stepper<T> S(prob, tr, c);
  if (!S.alloc()) return gf_fail(ctx, GF_ERR_NOMEM, "RK work allocation failed");
  S.prepare_adv();  // advection with a prescribed velocity and nu = 0
  T *uu[3] = {nullptr, nullptr, nullptr};
  for (int k = 0; k < tr->nstate; k++) uu[k] = (T *)u[k];
  int rc = GF_ERR_UNSUPPORTED;
  if (nsteps > 0 && S.cluster_ok()) {
    rc = S.cluster_steps(uu, (T)dt, nsteps);
    if (rc && rc != GF_ERR_UNSUPPORTED) return gf_fail(ctx, rc, "RK steps failed");
  }
  if (rc == GF_ERR_UNSUPPORTED)
    for (int s = 0; s < nsteps; s++)
      if ((rc = S.step(uu, uu, (T)dt))) return gf_fail(ctx, rc, "RK step failed");
  GF_CHECK_LAUNCH(ctx);
  // The reference asserts a finite state after every step; a NaN or Inf
  // stays in the state once made, so one check of the result after the
  // last step finds the same failures.  It reads the state once and waits
  // for the stream; inside a stream capture (a recorded step graph) it is
  // skipped, since the capture cannot wait.
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  GF_CUDA(ctx, cudaStreamIsCapturing(S.st, &cs));
  if (nsteps > 0 && cs == cudaStreamCaptureStatusNone) {
    // the flag is in the problem's pinned host block: no memset, no copy back
    volatile double *flag = prob->scal_h + RK_FLAG_SLOT;
    *flag = 0.0;
    prob->launches++;
    k_nonfinite<T><<<grid_for(S.n, 256, ctx->sm_count * 8), 256, 0, S.st>>>(
        S.n, tr->nstate, uu[0], uu[tr->nstate > 1 ? 1 : 0], uu[tr->nstate > 2 ? 2 : 0],
        prob->scal_h + RK_FLAG_SLOT);
    GF_CHECK_LAUNCH(ctx);
    GF_CUDA(ctx, cudaStreamSynchronize(S.st));
    if (*flag != 0.0)
      return gf_fail(ctx, GF_ERR_NONFINITE, "solution not finite after %d RK steps", nsteps);
  }
  return GF_OK;
}

}  // namespace gfrk

using namespace gfrk;

extern "C" int gf_rk_advance(gf_problem_t prob, int dtype, const gf_rk_traits *tr, void *const *u,
                             const void *const *c, double t0, double dt, int nsteps) {
  if (!prob) return GF_ERR_ARG;
  (void)t0;
  int rc = check_traits(prob, tr, (const void *const *)u, c);
  if (rc) return rc;
  GF_REQUIRE(prob->ctx, nsteps >= 0, "nsteps must be >= 0");
  if (dtype == GF_F64) return advance<double>(prob, tr, u, c, dt, nsteps);
  if (dtype == GF_F32) return advance<float>(prob, tr, u, c, dt, nsteps);
  return gf_fail(prob->ctx, GF_ERR_ARG, "unknown dtype %d", dtype);
}

// y = uin + ((0 + b0 K0) + b1 K1 + ...) on the problem's nlocal nodes: the
// stage input of step_b, as the stepper forms it (k_stage_sum); used by the
// partitioned stepper (geoflow_b200/dist.py).
extern "C" int gf_rk_stage_sum(gf_problem_t prob, int dtype, const void *uin, int nk,
                               const void *K0, const void *K1, const void *K2, double b0,
                               double b1, double b2, void *y) {
  if (!prob) return GF_ERR_ARG;
  gf_context *ctx = prob->ctx;
  GF_REQUIRE(ctx, uin && y && nk >= 0 && nk <= 3, "stage sum needs uin, y and 0..3 terms");
  GF_REQUIRE(ctx, (nk < 1 || K0) && (nk < 2 || K1) && (nk < 3 || K2), "missing stage vector");
  const int64_t n = prob->nlocal;
  const unsigned g = grid_for(n, 256, ctx->sm_count * 8);
  prob->launches++;
  if (dtype == GF_F64)
    k_stage_sum<double><<<g, 256, 0, ctx->stream>>>(n, (const double *)uin, nk,
                                                    (const double *)K0, (const double *)K1,
                                                    (const double *)K2, b0, b1, b2, (double *)y);
  else if (dtype == GF_F32)
    k_stage_sum<float><<<g, 256, 0, ctx->stream>>>(n, (const float *)uin, nk, (const float *)K0,
                                                   (const float *)K1, (const float *)K2,
                                                   (float)b0, (float)b1, (float)b2, (float *)y);
  else
    return gf_fail(ctx, GF_ERR_ARG, "unknown dtype %d", dtype);
  GF_CHECK_LAUNCH(ctx);
  return GF_OK;
}

extern "C" int gf_rk_advance_host(gf_problem_t prob, int dtype, const gf_rk_traits *tr,
                                  void *const *u, const void *const *c, double t0, double dt,
                                  int nsteps) {
  if (!prob) return GF_ERR_ARG;
  gf_context *ctx = prob->ctx;
  int rc = check_traits(prob, tr, (const void *const *)u, c);
  if (rc) return rc;
  const size_t bytes = (dtype == GF_F64 ? 8 : 4) * (size_t)prob->nlocal;
  void *du[3] = {nullptr, nullptr, nullptr};
  const void *dc[3] = {nullptr, nullptr, nullptr};
  for (int k = 0; k < tr->nstate; k++) {
    du[k] = gf_work(prob, 90 + k, bytes);
    if (!du[k]) return gf_fail(ctx, GF_ERR_NOMEM, "staging allocation failed");
    GF_CUDA(ctx, cudaMemcpyAsync(du[k], u[k], bytes, cudaMemcpyHostToDevice, ctx->stream));
  }
  if (tr->eqn == GF_EQN_ADVECT) {
    for (int k = 0; k < gf_nvel(prob); k++) {
      void *d = gf_work(prob, 93 + k, bytes);
      if (!d) return gf_fail(ctx, GF_ERR_NOMEM, "staging allocation failed");
      GF_CUDA(ctx, cudaMemcpyAsync(d, c[k], bytes, cudaMemcpyHostToDevice, ctx->stream));
      dc[k] = d;
    }
  }
  rc = gf_rk_advance(prob, dtype, tr, du, dc, t0, dt, nsteps);
  if (rc) return rc;
  for (int k = 0; k < tr->nstate; k++)
    GF_CUDA(ctx, cudaMemcpyAsync(u[k], du[k], bytes, cudaMemcpyDeviceToHost, ctx->stream));
  GF_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  return GF_OK;
}
