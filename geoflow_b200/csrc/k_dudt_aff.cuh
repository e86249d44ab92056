// k_dudt_aff.cuh -- the right-hand side of GBurgers::dudt_impl
// (pdes/gburgers.ipp:203-257) on affine 3-d elements; k_dudt.cuh has the same
// operator for per-node geometry, and states its terms.
//
// With dXi/dX and Jac constant in the element, the diffusion term of a line is
// the 1-d matrix K1 = D^T diag(W) D times a constant (k_helm_k1.cuh), so one
// read of a line yields both D u (advection) and K1 u (diffusion):
//   x-line of component c:  r_i = nu J X0^2 W_j W_k (K1 a)_i
//                                 + J X0 W_j W_k W_i c0_i (D a)_i
// and likewise along y and z; dudt_c = -Minv (r_x + r_y + r_z).  Both matrices
// run in even-odd form on the same sums and differences of the line (D is
// centro-antisymmetric: D(N-1-i, N-1-m) = -D(i, m)), which halves their
// multiply-adds; in FP32 each pair runs on the packed FP32x2 FMA.
//
// Bound: with D then D^T per direction the kernel moved 13 shared-memory words
// per node and component (93 % of the L1/shared pipe in FP32) through four
// barriers; here it is 7 words and one or two barriers.  In FP32 the velocity
// lines and the inverse mass stay in registers across the components; in FP64
// they are read where they are used (at N = 7, 168 registers and two blocks
// per SM otherwise).
#pragma once
#include <utility>

#include "k_dudt.cuh"
#include "k_helm_k1.cuh"

namespace gfk {

// Even-odd form of a centro-antisymmetric matrix (D or its transpose):
// {(A(i,m) + A(i,N-1-m)) / 2, (A(i,m) - A(i,N-1-m)) / 2}, i, m < N / 2.
template <typename T, int N>
struct AntiBasis {
  static constexpr int H = N / 2;
  typename Pair2<T>::type AP[H * H];
  T col[H], row[H];  // odd N: A(i, MID) and A(MID, m)
};
template <typename T, int N>
inline AntiBasis<T, N> make_antibasis(const gf_problem *p, bool transpose) {
  constexpr int H = N / 2, MID = (N - 1) / 2;
  AntiBasis<T, N> b{};
  // the antisymmetric part of D (which is D up to rounding)
  auto d = [&](int l, int m) {
    if (transpose) std::swap(l, m);
    return 0.5 * (p->D[l + m * N] - p->D[(N - 1 - l) + (N - 1 - m) * N]);
  };
  for (int i = 0; i < H; i++)
    for (int m = 0; m < H; m++) {
      b.AP[i * H + m].x = (T)(0.5 * (d(i, m) + d(i, N - 1 - m)));
      b.AP[i * H + m].y = (T)(0.5 * (d(i, m) - d(i, N - 1 - m)));
    }
  if (N % 2)
    for (int i = 0; i < H; i++) {
      b.col[i] = (T)d(i, MID);
      b.row[i] = (T)d(MID, i);
    }
  return b;
}

// out(l, i, (A a_l)_i) for L lines at once, from their even-odd forms and middle
// values (lines_K1 says why at once)
template <typename T, int N, int L, class OUT>
__device__ __forceinline__ void lines_anti(const AntiBasis<T, N> &B,
                                           const typename Pair2<T>::type (&eo)[L][N / 2],
                                           const T (&mid)[L], OUT out) {
  constexpr int H = N / 2, MID = (N - 1) / 2;
#pragma unroll
  for (int i = 0; i < H; i++) {
    typename Pair2<T>::type s[L];
#pragma unroll
    for (int m = 0; m < H; m++) {
      const typename Pair2<T>::type k = B.AP[i * H + m];
#pragma unroll
      for (int l = 0; l < L; l++) s[l] = m == 0 ? pmul(k, eo[l][0]) : pfma(k, eo[l][m], s[l]);
    }
#pragma unroll
    for (int l = 0; l < L; l++) {
      if (N % 2) s[l].x = fma(B.col[i], mid[l], s[l].x);
      out(l, i, s[l].y + s[l].x);
      out(l, N - 1 - i, s[l].y - s[l].x);
    }
  }
  if (N % 2) {
#pragma unroll
    for (int l = 0; l < L; l++) {
      T s = T(0);
#pragma unroll
      for (int m = 0; m < H; m++) s = fma(B.row[m], eo[l][m].y, s);
      out(l, MID, s);
    }
  }
}

template <typename T, int N>
struct DKBasis {
  AntiBasis<T, N> D;
  K1Basis<T, N> K;
};
template <typename T, int N>
inline DKBasis<T, N> make_dkbasis(const gf_problem *p) {
  return DKBasis<T, N>{make_antibasis<T, N>(p, false), make_k1basis<T, N>(p)};
}

// out(l, i, cd[l] (K1 a_l)_i + w(l, i) (D a_l)_i) for L lines at once (the
// first term alone when !ADV)
template <typename T, int N, bool ADV, int L, class WV, class OUT>
__device__ __forceinline__ void lines_rhs(const DKBasis<T, N> &B,
                                          const typename Pair2<T>::type (&eo)[L][N / 2],
                                          const T (&mid)[L], const T (&cd)[L], WV w, OUT out) {
  using P2 = typename Pair2<T>::type;
  constexpr int H = N / 2, MID = (N - 1) / 2;
#pragma unroll
  for (int i = 0; i < H; i++) {
    P2 k[L], d[L];
#pragma unroll
    for (int m = 0; m < H; m++) {
      const P2 km = B.K.KP[i * H + m];
#pragma unroll
      for (int l = 0; l < L; l++) k[l] = m == 0 ? pmul(km, eo[l][0]) : pfma(km, eo[l][m], k[l]);
      if (ADV) {
        const P2 dm = B.D.AP[i * H + m];
#pragma unroll
        for (int l = 0; l < L; l++) d[l] = m == 0 ? pmul(dm, eo[l][0]) : pfma(dm, eo[l][m], d[l]);
      }
    }
#pragma unroll
    for (int l = 0; l < L; l++) {
      if (N % 2) k[l].x = fma(B.K.Kcol[i], mid[l], k[l].x);
      const T s = k[l].x * cd[l];
      T r0 = fma(k[l].y, cd[l], s), r1 = fma(-k[l].y, cd[l], s);
      if (ADV) {
        if (N % 2) d[l].x = fma(B.D.col[i], mid[l], d[l].x);
        r0 = fma(w(l, i), d[l].y + d[l].x, r0);
        r1 = fma(w(l, N - 1 - i), d[l].y - d[l].x, r1);
      }
      out(l, i, r0);
      out(l, N - 1 - i, r1);
    }
  }
  if (N % 2) {
#pragma unroll
    for (int l = 0; l < L; l++) {
      T s = B.K.Kmm * mid[l], d = T(0);
#pragma unroll
      for (int m = 0; m < H; m++) s = fma(B.K.Krow[m], eo[l][m].x, s);
      s *= cd[l];
      if (ADV) {
#pragma unroll
        for (int m = 0; m < H; m++) d = fma(B.D.row[m], eo[l][m].y, d);
        s = fma(w(l, MID), d, s);
      }
      out(l, MID, s);
    }
  }
}

// Volumes of the element in shared memory: the evolved components, the x- and
// y-velocity where they are fields of their own, and the x- and y-terms (in
// FP32 twice, so that a component's terms are written while the last one's
// are read: one barrier per component instead of two).
template <typename T, int EQN>
constexpr int aff_vols() {
  return (EQN == GF_EQN_BURGERS ? 3 : (EQN == GF_EQN_ADVECT ? 3 : 1)) +
         2 * (sizeof(T) == 4 && EQN == GF_EQN_BURGERS ? 2 : 1);
}
// Elements per block: about 160 threads in FP32, about 128 in FP64, whose
// threads need twice the registers.
template <typename T, int N> constexpr int epb_aff() {
  return ((sizeof(T) == 4 ? 160 : 128) / (N * N)) < 1 ? 1 : (sizeof(T) == 4 ? 160 : 128) / (N * N);
}

// MODE_DUDT or MODE_EULER (k_dudt.cuh); fields as k_dudt3d.
template <typename T, int N, int EPB, int EQN, int MODE>
__global__ void __launch_bounds__(N *N *EPB)
    k_dudt3a(const __grid_constant__ DKBasis<T, N> B, const T *__restrict__ egeom, int64_t ne, T nu,
             const T *__restrict__ f0, const T *__restrict__ f1, const T *__restrict__ f2,
             const T *__restrict__ f3, const T *__restrict__ imass, T *__restrict__ o0,
             T *__restrict__ o1, T *__restrict__ o2, const RKEpi<T> epi) {
  constexpr bool ADV = EQN != GF_EQN_HEAT;
  constexpr int NC = EQN == GF_EQN_BURGERS ? 3 : 1;
  constexpr int NS = EQN == GF_EQN_HEAT ? 1 : 3;  // staged fields
  constexpr int NB = (aff_vols<T, EQN>() - NS) / 2;
  constexpr int P = Pad<N>::P, PLANE = N * P, VOL = N * PLANE, NN = N * N, NNN = N * N * N;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T *s = reinterpret_cast<T *>(smem_raw) + threadIdx.y * (aff_vols<T, EQN>() * VOL);
  const int t = threadIdx.x, a0 = t % N, a1 = t / N;
  const int64_t e = (int64_t)blockIdx.x * EPB + threadIdx.y;
  const bool active = e < ne;
  const int64_t base = e * NNN;
  const T *fin[3] = {f0, f1, f2};

  // this thread's z-column (i = a0, j = a1): the staged fields, the z-velocity
  // (Burgers: component 2) and the inverse mass
  constexpr bool KEEP = sizeof(T) == 4;
  T im[KEEP ? N : 1], vz[KEEP ? N : 1], vx[KEEP ? N : 1], vy[KEEP ? N : 1];
#pragma unroll
  for (int f = 0; f < NS; f++) {
#pragma unroll
    for (int k = 0; k < N; k++) {
      const T v = active ? fin[f][base + k * NN + t] : T(0);
      s[f * VOL + k * PLANE + a1 * P + a0] = v;
      if (KEEP && EQN == GF_EQN_BURGERS && f == 2) vz[KEEP ? k : 0] = v;
    }
  }
  if (KEEP) {
#pragma unroll
    for (int k = 0; k < N; k++) {
      if (EQN == GF_EQN_ADVECT) vz[KEEP ? k : 0] = active ? f3[base + k * NN + t] : T(0);
      im[KEEP ? k : 0] = active ? imass[base + k * NN + t] : T(0);
    }
  }
  T X[3] = {T(0), T(0), T(0)}, J = T(0);
  if (active) {
    const T *ge = egeom + e * 4;
    X[0] = ge[0];
    X[1] = ge[1];
    X[2] = ge[2];
    J = ge[3];
  }
  // the x-line is (j = a0, k = a1), the y-line (i = a0, k = a1)
  const T w2 = J * (B.K.W[a0] * B.K.W[a1]);
  const T cax = w2 * X[0], cay = w2 * X[1], caz = w2 * X[2];
  const T cdx = nu * (cax * X[0]), cdy = nu * (cay * X[1]), cdz = nu * (caz * X[2]);
  const int xl = a1 * PLANE + a0 * P, yl = a1 * PLANE + a0, zl = a1 * P + a0;
  __syncthreads();
  constexpr int fx = EQN == GF_EQN_BURGERS ? 0 : 1, fy = EQN == GF_EQN_BURGERS ? 1 : 2;
  if (KEEP && ADV) {
#pragma unroll
    for (int m = 0; m < N; m++) {
      vx[KEEP ? m : 0] = s[fx * VOL + xl + m];
      vy[KEEP ? m : 0] = s[fy * VOL + yl + m * P];
    }
  }
  auto velx = [&](int m) -> T { return KEEP ? vx[KEEP ? m : 0] : s[fx * VOL + xl + m]; };
  auto vely = [&](int m) -> T { return KEEP ? vy[KEEP ? m : 0] : s[fy * VOL + yl + m * P]; };
  auto velz = [&](int m) -> T {
    if (KEEP) return vz[KEEP ? m : 0];
    if (EQN == GF_EQN_BURGERS) return s[2 * VOL + zl + m * PLANE];
    return active ? f3[base + m * NN + t] : T(0);
  };
#pragma unroll
  for (int c = 0; c < NC; c++) {
    const T *su = s + c * VOL;
    T *sx = s + (NS + 2 * (c % NB)) * VOL, *sy = sx + VOL;
    // line l (0 x, 1 y, 2 z) of component c at local index m
    T r[N], col[N];
    auto line = [&](int l, int m) -> T {
      if (KEEP && EQN == GF_EQN_BURGERS && l == c) return l == 0 ? velx(m) : (l == 1 ? vely(m) : velz(m));
      return su[l == 0 ? xl + m : (l == 1 ? yl + m * P : zl + m * PLANE)];
    };
    auto weight = [&](int l, int i) -> T {
      const T ca = l == 0 ? cax : (l == 1 ? cay : caz);
      return ca * B.K.W[i] * (l == 0 ? velx(i) : (l == 1 ? vely(i) : velz(i)));
    };
    auto put = [&](int l, int i, T v) {
      if (l == 0) sx[xl + i] = v;
      else if (l == 1) sy[yl + i * P] = v;
      else r[i] = v;
    };
    // the update's other terms, read before the barrier: behind it their latency
    // is exposed once per node (259 us against 105 without the update, 64000
    // elements at N = 6)
    T yv[MODE == MODE_EULER ? N : 1], y2v[MODE == MODE_EULER ? N : 1];
    const T *const yc = c == 0 ? epi.y[0] : (c == 1 ? epi.y[1] : epi.y[2]);
    const T *const y2c = c == 0 ? epi.y2[0] : (c == 1 ? epi.y2[1] : epi.y2[2]);
    auto prefetch = [&] {
      if constexpr (MODE != MODE_EULER) return;
#pragma unroll
      for (int k = 0; k < N; k++) yv[MODE == MODE_EULER ? k : 0] = yc && active ? yc[base + k * NN + t] : T(0);
#pragma unroll
      for (int k = 0; k < N; k++) y2v[MODE == MODE_EULER ? k : 0] = y2c && active ? y2c[base + k * NN + t] : T(0);
    };
    const T cd[3] = {cdx, cdy, cdz};
    // L lines share one read of a matrix entry: all three in FP64 from N = 7 on
    // (66 us against 80 at N = 8), where an entry is a load from the parameter
    // bank and the registers allow it; one elsewhere (FP32 at N = 6: 138 us
    // against 150 for three)
    constexpr int L = sizeof(T) == 8 && N >= 7 ? 3 : 1;
#pragma unroll
    for (int l0 = 0; l0 < 3; l0 += L) {
      if (l0 + L == 3) prefetch();
      typename Pair2<T>::type eo[L][N / 2];
      T mid[L], cl[L];
#pragma unroll
      for (int l = 0; l < L; l++) {
        T a[N];
#pragma unroll
        for (int m = 0; m < N; m++) a[m] = line(l0 + l, m);
        if (l0 + l == 2) {
#pragma unroll
          for (int m = 0; m < N; m++) col[m] = a[m];
        }
        line_eo<T, N>(a, eo[l]);
        mid[l] = a[(N - 1) / 2];
        cl[l] = cd[l0 + l];
      }
      lines_rhs<T, N, ADV, L>(
          B, eo, mid, cl, [&](int l, int i) { return weight(l0 + l, i); },
          [&](int l, int i, T v) { put(l0 + l, i, v); });
    }
    __syncthreads();
    if (active) {
      T *const oc = c == 0 ? o0 : (c == 1 ? o1 : o2);
#pragma unroll
      for (int k = 0; k < N; k++) {
        const int64_t node = base + k * NN + t;
        const T K = -(KEEP ? im[KEEP ? k : 0] : imass[node]) * ((sx[zl + k * PLANE] + sy[zl + k * PLANE]) + r[k]);
        if constexpr (MODE == MODE_EULER) {
          const T *ui = c == 0 ? epi.uin[0] : (c == 1 ? epi.uin[1] : epi.uin[2]);
          const T uv = epi.uin_is_u ? col[k] : ui[node];
          oc[node] = rk_euler_vals(K, epi.dt, uv, epi.a, yc != nullptr, yv[k], epi.b, epi.a2,
                                   y2c != nullptr, y2v[k], epi.b2);
        } else {
          oc[node] = K;
        }
      }
    }
    if (NB == 1 && c + 1 < NC) __syncthreads();
  }
}

}  // namespace gfk
