// api_rk_pass64.cu -- the FP64 stage passes and the reverse sweep (FP64 only).
#include "rk_pass.cuh"

template <>
int rk_pass<double>(gf_problem *prob, int mode, int nc, const gfk::RKPass<double> &p,
                    cudaStream_t st) {
  switch (mode) {
    case gfk::RK_EULER: return gfk::rk_pass_mode<double, gfk::RK_EULER>(prob, nc, p, st);
    case gfk::RK_MID: return gfk::rk_pass_mode<double, gfk::RK_MID>(prob, nc, p, st);
    case gfk::RK_MIDS: return gfk::rk_pass_mode<double, gfk::RK_MIDS>(prob, nc, p, st);
    case gfk::RK_LAST: return gfk::rk_pass_mode<double, gfk::RK_LAST>(prob, nc, p, st);
    case gfk::ADJ_START: return gfk::rk_pass_mode<double, gfk::ADJ_START>(prob, nc, p, st);
    case gfk::ADJ_STAGE: return gfk::rk_pass_mode<double, gfk::ADJ_STAGE>(prob, nc, p, st);
    case gfk::ADJ_STAGE_LAST: return gfk::rk_pass_mode<double, gfk::ADJ_STAGE_LAST>(prob, nc, p, st);
    default: return gfk::rk_pass_mode<double, gfk::RK_SMOOTH>(prob, nc, p, st);
  }
}
