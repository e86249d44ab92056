// rk_common.cuh -- the device-side RK stepper object shared by the
// forward stepper (api_rk.cu) and its adjoint (api_adjoint.cu).
#pragma once
#include "gf_common.cuh"

namespace gfrk {

void butcher(int order, double *alpha, double beta[4][4], double *c);
// the coefficient planes of the advection fast path (k_def.cuh
// adv_coef_point) of a 2-d deformed or embedded problem, velocity c[nxy]
template <typename T>
int adv_coef_launch(gf_problem *prob, const T *const *c, T *b0, T *b1, cudaStream_t st);
int check_traits(gf_problem *prob, const gf_rk_traits *tr, const void *const *u,
                 const void *const *c);

template <typename T>
struct Stepper {
  gf_problem *prob;
  cudaStream_t st;
  int64_t n;
  int eqn, nstate, scheme;
  T nu;
  const T *c[3] = {nullptr, nullptr, nullptr};
  T *uacc[3] = {nullptr, nullptr, nullptr};
  T *utmp[3] = {nullptr, nullptr, nullptr};
  T *K[3][3] = {{nullptr}};
  // advection fast path (prescribed velocity, nu = 0, 2-d deformed or
  // embedded): coefficient planes b_0, b_1 of adv_element, or null
  T *advb[2] = {nullptr, nullptr};
  T *advbuf[2] = {nullptr, nullptr};  // their storage (alloc), unused until prepare_adv
  bool adv_ok() const;

  Stepper(gf_problem *p, const gf_rk_traits *tr, const void *const *cv)
      : prob(p), st(p->ctx->stream), n(p->nlocal), eqn(tr->eqn), nstate(tr->nstate),
        scheme(tr->scheme), nu((T)tr->nu) {
    if (cv)
      for (int k = 0; k < gf_nvel(p); k++) c[k] = (const T *)cv[k];
  }
  bool alloc();
  // forms the fast path's coefficients when the problem and equation allow
  // it (k_def.cuh adv_coef_point); returns false when they do not
  bool prepare_adv();
  int rhs(T *const *u, T *const *Kout);
  // x = the SSP substep update of dudt(u) before its Smooth (the RHS
  // kernel's MODE_EULER epilogue; 3-d non-deformed problems), then Smooth;
  // false when the problem takes the separate RHS and update passes
  bool rhs_euler_smooth(T *const *u, T *const *x, T dt, T *const *uin, T a, T *const *y, T b,
                        T a2, T *const *y2, T b2, int *rc);
  // GMTK::constrain2sphere on the state where step_b calls it, on embedded
  // surfaces with node coordinates and a state of >= 3 components
  bool constrains() const;
  void constrain(T *const *u);
  // Smooth on every state component, in place or into out
  int smooth_n(T *const *v);
  int smooth_to(T *const *v, T *const *out);
  // out = Smooth(the SSP substep update of x = dudt) (y and y2 may be null)
  int euler_smooth_n(T *const *x, T *const *out, T dt, T *const *uin, T a, T *const *y, T b,
                     T a2, T *const *y2, T b2);
  // the class pass after a step_b stage (k_dss.cuh RK_MID, RK_MIDS, RK_LAST):
  // K = Smooth(x), accout = accin + ch K, out = uin + b K or the step's result
  int stage_pass(int mode, T *const *x, T *const *accin, T ch, T *const *accout, T *const *uin,
                 T b, T *const *out);
  // One step uin -> uout.  With a tape (pointers tape[3*m + k], m = 0 ..
  // stages-1), stage m's input state (the argument of its RHS call) is left
  // in tape[3*m + k] for the adjoint sweep.
  int step(T *const *uin, T *const *uout, T dt, T *const *tape = nullptr);
  int step_ssp(T *const *uin, T *const *uout, T dt);
  // nsteps steps in place in one launch, where cluster_ok()
  bool cluster_ok() const;
  int cluster_steps(T *const *u, T dt, int nsteps);
  int stages() const { return scheme <= 4 ? scheme : (scheme == GF_SSP22 ? 2 : (scheme == GF_SSP33 ? 3 : 4)); }
};

}  // namespace gfrk
