// api_rk_pass32.cu -- the FP32 stage passes.
#include "rk_pass.cuh"

template <>
int rk_pass<float>(gf_problem *prob, int mode, int nc, const gfk::RKPass<float> &p,
                   cudaStream_t st) {
  switch (mode) {
    case gfk::RK_EULER: return gfk::rk_pass_mode<float, gfk::RK_EULER>(prob, nc, p, st);
    case gfk::RK_MID: return gfk::rk_pass_mode<float, gfk::RK_MID>(prob, nc, p, st);
    case gfk::RK_MIDS: return gfk::rk_pass_mode<float, gfk::RK_MIDS>(prob, nc, p, st);
    case gfk::RK_LAST: return gfk::rk_pass_mode<float, gfk::RK_LAST>(prob, nc, p, st);
    default: return gfk::rk_pass_mode<float, gfk::RK_SMOOTH>(prob, nc, p, st);
  }
}
