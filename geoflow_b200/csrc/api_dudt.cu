// api_dudt.cu -- launchers of the advection and Burgers right-hand sides
// (GBurgers::dudt_impl, pdes/gburgers.ipp:203-257; GAdvect::apply,
// sem/gadvect.ipp:58-100), shared by the operator entry points and the RK
// stepper.
#include "gf_common.cuh"
#include "k_dudt.cuh"
#include "ops_launch.cuh"

using namespace gfk;

// Deformed / embedded elements: one k_def launch per evolved component,
// the reference gradient shared by advection and diffusion.  f as for
// launch_dudt: ADVECT {p, c0, c1, c2}, BURGERS {u0, u1, u2}, HEAT {u}.
template <typename T>
static int launch_def_dudt(gf_problem *prob, int eqn, int mode, T nu, const T *const *f,
                           T *const *o, cudaStream_t st) {
  const int nv = prob->nxy;
  if (eqn == GF_EQN_ADVECT) {
    const T *c[3] = {f[1], f[2], f[3]};
    return dispatch_n<DefLaunch<T, LoadE<T>>::template F>(
        prob->n, prob, mode == MODE_ADVECT ? (int)DEF_ADVECT : (int)DEF_DUDT, nu,
        LoadE<T>{f[0]}, nv, (const T *const *)c, 0, o[0], st);
  }
  if (eqn == GF_EQN_HEAT)
    return dispatch_n<DefLaunch<T, LoadE<T>>::template F>(
        prob->n, prob, (int)DEF_DUDT, nu, LoadE<T>{f[0]}, 0, (const T *const *)nullptr, 0, o[0],
        st);
  for (int k = 0; k < nv; k++) {  // Burgers: the velocity is the state
    int rc = dispatch_n<DefLaunch<T, LoadE<T>>::template F>(
        prob->n, prob, (int)DEF_DUDT, nu, LoadE<T>{f[k]}, nv, f, 0, o[k], st);
    if (rc) return rc;
  }
  return GF_OK;
}

template <typename T>
int launch_dudt(gf_problem *prob, int eqn, int mode, T nu, const T *const *f, T *const *o,
                cudaStream_t st, const gfk::RKEpi<T> *epi) {
  if (prob->geom >= GF_GEOM_DEFORMED) {
    if (mode == MODE_EULER) return GF_ERR_UNSUPPORTED;
    return launch_def_dudt<T>(prob, eqn, mode, nu, f, o, st);
  }
  const RKEpi<T> none{};
  return dispatch_n<DudtLaunch<T>::template F>(prob->n, prob, eqn, mode, nu, f, o, st,
                                               epi ? *epi : none);
}
template int launch_dudt<double>(gf_problem *, int, int, double, const double *const *,
                                 double *const *, cudaStream_t, const gfk::RKEpi<double> *);
template int launch_dudt<float>(gf_problem *, int, int, float, const float *const *,
                                float *const *, cudaStream_t, const gfk::RKEpi<float> *);
