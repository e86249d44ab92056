// api_rk_pass32.cu -- the FP32 stage passes.
#include "rk_pass.cuh"

template <>
void rk_pass<float>(gf_problem *prob, int mode, int nc, const gfk::RKPass<float> &p,
                 cudaStream_t st) {
  switch (mode) {
    case gfk::RK_EULER: gfk::rk_pass_mode<float, gfk::RK_EULER>(prob, nc, p, st); break;
    case gfk::RK_MID: gfk::rk_pass_mode<float, gfk::RK_MID>(prob, nc, p, st); break;
    case gfk::RK_MIDS: gfk::rk_pass_mode<float, gfk::RK_MIDS>(prob, nc, p, st); break;
    case gfk::RK_LAST: gfk::rk_pass_mode<float, gfk::RK_LAST>(prob, nc, p, st); break;
    default: gfk::rk_pass_mode<float, gfk::RK_SMOOTH>(prob, nc, p, st); break;
  }
}
