// api_rk_cluster32.cu -- the FP32 instances of the one-cluster RK steps.
#include <algorithm>

#include "rk_cluster.cuh"

template <typename T>
int launch_rk_cluster(gf_problem *prob, int eqn, gfk::RKProgram<T> &pr, cudaStream_t st) {
  return dispatch_n<gfk::RKClusterLaunch<T>::template F>(prob->n, prob, eqn, pr, st);
}
template int launch_rk_cluster<float>(gf_problem *, int, gfk::RKProgram<float> &, cudaStream_t);
