// api_rk_pass64.cu -- the FP64 stage passes and the reverse sweep (FP64 only).
#include "rk_pass.cuh"

template <>
void rk_pass<double>(gf_problem *prob, int mode, int nc, const gfk::RKPass<double> &p,
                 cudaStream_t st) {
  switch (mode) {
    case gfk::RK_EULER: gfk::rk_pass_mode<double, gfk::RK_EULER>(prob, nc, p, st); break;
    case gfk::RK_MID: gfk::rk_pass_mode<double, gfk::RK_MID>(prob, nc, p, st); break;
    case gfk::RK_MIDS: gfk::rk_pass_mode<double, gfk::RK_MIDS>(prob, nc, p, st); break;
    case gfk::RK_LAST: gfk::rk_pass_mode<double, gfk::RK_LAST>(prob, nc, p, st); break;
    case gfk::ADJ_START: gfk::rk_pass_mode<double, gfk::ADJ_START>(prob, nc, p, st); break;
    case gfk::ADJ_STAGE: gfk::rk_pass_mode<double, gfk::ADJ_STAGE>(prob, nc, p, st); break;
    case gfk::ADJ_STAGE_LAST: gfk::rk_pass_mode<double, gfk::ADJ_STAGE_LAST>(prob, nc, p, st); break;
    default: gfk::rk_pass_mode<double, gfk::RK_SMOOTH>(prob, nc, p, st); break;
  }
}
