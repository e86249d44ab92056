// k_tensor.cuh -- element-local sum-factorised kernels (sm_100a).
//
// One element's n^3 (n^2 in 2-d) block is staged in shared memory.  Each
// thread owns one 1-d line of the element in turn: an x-line, a y-line and
// a z-line, so that every 1-d contraction y = D a (or D^T a) runs on a line
// held in registers, with D read from the kernel parameter block (uniform
// across the warp, so it feeds the FMAs straight from the constant bank).
// Each node therefore costs one shared-memory load per direction instead of
// n.  Rows are padded to an odd length so that x-line reads by consecutive
// threads fall in distinct banks.
//
// These kernels implement GHelmholtz::reg_prod (sem/ghelmholtz.ipp:309-378):
// gdu_k = Mass (G_kk (D_k u)), uo = sum_k D_k^T gdu_k, times p, plus q M u.
#pragma once
#include "gf_common.cuh"
#include "k_maps.cuh"

namespace gfk {

template <int N> struct Pad { static constexpr int P = (N % 2) ? N : N + 1; };

// d[i] = sum_m D(i,m) a[m]
template <typename T, int N>
__device__ __forceinline__ void line_D(const T *__restrict__ D, const T (&a)[N], T (&d)[N]) {
#pragma unroll
  for (int i = 0; i < N; i++) {
    T s = D[i] * a[0];
#pragma unroll
    for (int m = 1; m < N; m++) s = fma(D[i + m * N], a[m], s);
    d[i] = s;
  }
}

// d[i] = sum_m D(m,i) a[m]
template <typename T, int N>
__device__ __forceinline__ void line_DT(const T *__restrict__ D, const T (&a)[N], T (&d)[N]) {
#pragma unroll
  for (int i = 0; i < N; i++) {
    T s = D[i * N] * a[0];
#pragma unroll
    for (int m = 1; m < N; m++) s = fma(D[m + i * N], a[m], s);
    d[i] = s;
  }
}

// L lines at once, one read of a matrix entry for all of them: out(l, i,
// sum_m A(i, m) a[l][m]), A = D, or D^T with TR; same sums in the same order as
// line_D and line_DT.  In FP64 an entry is a load from the parameter bank, 6 N^2
// of them per thread with a line at a time: the full-metric apply at N = 8 took
// 70 us that way and 43 with three lines.
template <typename T, int N, int L, bool TR, class OUT>
__device__ __forceinline__ void lines_D(const T *__restrict__ D, const T (&a)[L][N], OUT out) {
#pragma unroll
  for (int i = 0; i < N; i++) {
    T s[L];
#pragma unroll
    for (int m = 0; m < N; m++) {
      const T c = TR ? D[m + i * N] : D[i + m * N];
#pragma unroll
      for (int l = 0; l < L; l++) s[l] = m == 0 ? c * a[l][0] : fma(c, a[l][m], s[l]);
    }
#pragma unroll
    for (int l = 0; l < L; l++) out(l, i, s[l]);
  }
}

template <int N> constexpr int epb3() {
  return N <= 2 ? 32 : ((160 / (N * N)) < 1 ? 1 : (160 / (N * N)));
}
template <int N> constexpr int epb2() {
  return (256 / (N * N)) < 1 ? 1 : (256 / (N * N));
}

// Per-node geometric factors of element e at local node a.
template <typename T, int DIM>
struct NodeGeom {
  T X[DIM];  // dXidX_k
  T J;       // Jacobian
};

template <typename T, int DIM>
__device__ __forceinline__ void elem_geom(const Geom<T> &g, int64_t e, NodeGeom<T, DIM> &out) {
  if (g.egeom) {
    const T *ge = g.egeom + e * (DIM + 1);
#pragma unroll
    for (int k = 0; k < DIM; k++) out.X[k] = ge[k];
    out.J = ge[DIM];
  }
}

template <typename T, int DIM>
__device__ __forceinline__ void node_geom(const Geom<T> &g, int64_t node, NodeGeom<T, DIM> &out) {
  if (!g.egeom) {
#pragma unroll
    for (int k = 0; k < DIM; k++) out.X[k] = g.ngeom[k * g.nlocal + node];
    out.J = g.ngeom[DIM * g.nlocal + node];
  }
}

// ---------------------------------------------------------------------
// Helmholtz apply with a diagonal metric: uo = p sum_k Dk^T M Gk Dk u + q M u,
// per-node geometry (REGULAR) or per-node p on affine elements.
// ---------------------------------------------------------------------
// LD is the input loader (k_maps.cuh): the element-local vector itself, or
// a unique-node vector gathered through the box lattice or node_class.
// T is the arithmetic type; the input is stored as LD::value_type and the
// output as TO (FP32 storage with FP64 arithmetic keeps the apply's
// rounding at the storage level, which the mixed-precision CG relies on).
//
// With a diagonal metric D^T (M G p) D acts along one line, so a line is read
// once, contracted twice in registers and written once.  The weights M G p are
// formed by the owner of the node's z-column, which reads the geometry and
// coefficient planes once and coalesced, and go through shared memory to the
// x- and y-lines (a line's result then overwrites its weights).  Reading the
// planes where each direction needs them cost three passes over them, two of
// them strided: 70 us at 17x22x19 elements, p = 6, FP64 with per-node p and q,
// against a floor of 23 us for the planes themselves.
// FP64 holds a line and its contraction in registers and waits on memory and on
// the line's chain, so small blocks that leave room for many others come first:
// about 96 threads (N = 4, 5, 6: 33, 43, 54 us against 35, 55, 60 with 160 to
// 192), one element from N = 7, and the register cap below.  Per-node p and q,
// 2.4 M nodes (N = 7: cap 64, 72, 80, none: 58, 54, 51, 57 us) and 1.7 M (N = 8:
// 80, 96, 128, none: 58, 50, 43, 49; a cap that spills loses more than the extra
// warps give; N = 9: 80, 128, none: 74, 59, 104).
//
// Two choices by order, each where it measured faster (1.5 M nodes, us; per-node
// geometry with per-node p and q, with scalar ones, affine with per-node ones):
// * helm3_regz: the z-column's weights and mass term, which no other thread reads,
//   stay in registers instead of shared memory (three volumes instead of five)
//   while they fit there: FP64 N = 2: 18.1 14.4 14.4 against 20.5 18.2 16.4, N = 4:
//   18.6 12.7 12.4 against 22.6 16.2 15.4, N = 6: 24.5 16.1 14.9 against 28.7 18.5
//   18.5; from N = 7 it spills (35.2 22.3 22.4 against 30.4 18.5 20.5).  FP32 N = 8:
//   10.3 10.3 10.3 against 14.4 12.4 13.1; from N = 9 it loses (14.4 12.4 14.4 against
//   12.4 11.9 12.3).
// * helm3_joint: the three lines of a thread share one read of a matrix entry
//   (lines_D).  FP64 from N = 10, where a line at a time spills under the cap (344
//   bytes at N = 10) and without it leaves two blocks per SM: N = 10: 43 25 27
//   against 56 39 35 a line at a time and 69 32 39 without a cap; N = 11: 35 21 21
//   against 44 27 27 and 56 28 31; N = 12: 45 27 27 against 41 25 27 and 90 43 49,
//   but 10.3 against 12.4 on 17 elements.
template <typename T, int N> constexpr int epb_diag() {
  return sizeof(T) == 4 ? epb3<N>() : (N <= 2 ? 24 : (96 / (N * N) < 1 ? 1 : 96 / (N * N)));
}
template <typename T, int N, int EPB> constexpr int helm3_blocks() {
  constexpr int warps = (N * N * EPB + 31) / 32, regs = N <= 6 ? 56 : (N == 7 ? 80 : 128);
  return sizeof(T) == 4 ? 0 : 65536 / (warps * 32 * regs);
}
template <typename T, int N> constexpr bool helm3_regz() {
  return N <= (sizeof(T) == 4 ? 8 : 6);
}
template <typename T, int N> constexpr bool helm3_joint() { return sizeof(T) == 8 && N >= 10; }
template <typename T, int N> constexpr int helm3_vols() { return helm3_regz<T, N>() ? 3 : 5; }
template <typename T, int N, int EPB, class LD, typename TO = T>
__global__ void __launch_bounds__(N *N *EPB, helm3_blocks<T, N, EPB>())
    k_helm3d(const __grid_constant__ Basis<T, N> B, const Geom<T> g, int64_t ne, T p,
             const T *__restrict__ pvec, T q, const T *__restrict__ qvec, int use_mass,
             const LD ld, TO *__restrict__ uo, const double *__restrict__ stop) {
  if (stop && stop[0] != 0.0) return;
  constexpr int P = Pad<N>::P, PLANE = N * P, VOL = N * PLANE, NN = N * N, NNN = N * N * N;
  constexpr bool REGZ = helm3_regz<T, N>(), JOINT = helm3_joint<T, N>();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T *su = reinterpret_cast<T *>(smem_raw) + threadIdx.y * helm3_vols<T, N>() * VOL;
  T *sx = su + VOL, *sy = su + 2 * VOL, *sz = su + 3 * VOL, *so = su + 4 * VOL;  // !REGZ: sz, so
  const int t = threadIdx.x, a0 = t % N, a1 = t / N;
  const int64_t e = (int64_t)blockIdx.x * EPB + threadIdx.y;
  const bool active = e < ne;
  const int64_t base = e * NNN;
  const int xl = a1 * PLANE + a0 * P, yl = a1 * PLANE + a0, zl = a1 * P + a0;

  // this thread's z-column (i = a0, j = a1): u, the weights, the mass term
  T rz[REGZ ? N : 1], ro[REGZ ? N : 1];
  auto put = [&](int k, T u, T wx, T wy, T wz, T o) {
    const int s = zl + k * PLANE;
    su[s] = u;
    sx[s] = wx;
    sy[s] = wy;
    if constexpr (REGZ) {
      rz[k] = wz;
      ro[k] = o;
    } else {
      sz[s] = wz;
      so[s] = o;
    }
  };
  if (active) {
    NodeGeom<T, 3> eg;
    eg.X[0] = eg.X[1] = eg.X[2] = eg.J = T(0);
    elem_geom<T, 3>(g, e, eg);
    typename LD::value_type lv[N];
    ld.template zline<N>(e, a0, a1, lv);
    const T w2 = B.W[a0] * B.W[a1];
#pragma unroll
    for (int k = 0; k < N; k++) {
      const int64_t node = base + k * NN + t;
      NodeGeom<T, 3> ng = eg;
      node_geom<T, 3>(g, node, ng);
      const T u = (T)lv[k], mass = B.W[k] * w2 * ng.J;
      const T mp = pvec ? mass * pvec[node] : mass * p;
      put(k, u, mp * (ng.X[0] * ng.X[0]), mp * (ng.X[1] * ng.X[1]), mp * (ng.X[2] * ng.X[2]),
          use_mass ? mass * (qvec ? qvec[node] : q) * u : T(0));
    }
  } else {
#pragma unroll
    for (int k = 0; k < N; k++) put(k, T(0), T(0), T(0), T(0), T(0));
  }
  __syncthreads();
  auto wz = [&](int k) -> T {
    if constexpr (REGZ) return rz[k];
    else return sz[zl + k * PLANE];
  };
  T oz[N];  // the z-line's D^T (w (D u)); the others' overwrite their weights
  if constexpr (JOINT) {
    T a[3][N], d[3][N];
#pragma unroll
    for (int m = 0; m < N; m++) {
      a[0][m] = su[xl + m];
      a[1][m] = su[yl + m * P];
      a[2][m] = su[zl + m * PLANE];
    }
    lines_D<T, N, 3, false>(B.D, a, [&](int l, int i, T v) {
      d[l][i] = v * (l == 0 ? sx[xl + i] : (l == 1 ? sy[yl + i * P] : wz(i)));
    });
    lines_D<T, N, 3, true>(B.D, d, [&](int l, int i, T v) {
      if (l == 0) sx[xl + i] = v;
      else if (l == 1) sy[yl + i * P] = v;
      else oz[i] = v;
    });
  } else {
    // one line: a = D^T (w (D a))
    T a[1][N], d[1][N];
    auto line = [&](int s0, int st, auto w) {
#pragma unroll
      for (int m = 0; m < N; m++) a[0][m] = su[s0 + m * st];
      lines_D<T, N, 1, false>(B.D, a, [&](int, int i, T v) { d[0][i] = v * w(i); });
      lines_D<T, N, 1, true>(B.D, d, [&](int, int i, T v) { a[0][i] = v; });
    };
    line(xl, 1, [&](int i) { return sx[xl + i]; });
#pragma unroll
    for (int m = 0; m < N; m++) sx[xl + m] = a[0][m];
    line(yl, P, [&](int i) { return sy[yl + i * P]; });
#pragma unroll
    for (int m = 0; m < N; m++) sy[yl + m * P] = a[0][m];
    line(zl, PLANE, wz);
#pragma unroll
    for (int m = 0; m < N; m++) oz[m] = a[0][m];
  }
  __syncthreads();
  if (active) {
#pragma unroll
    for (int k = 0; k < N; k++) {
      const int s = zl + k * PLANE;
      const T o = [&] {
        if constexpr (REGZ) return ro[k];
        else return so[s];
      }();
      uo[base + k * NN + t] = (TO)(((sx[s] + sy[s]) + oz[k]) + o);
    }
  }
}

// 2-d: 2 N threads per element, one x-line (threads < N) or y-line each; the
// block's nodes are loaded and stored by all of its threads, coalesced.  (One
// thread per node reads D at a run-time row from the parameter bank, which
// serves one address per cycle: 2 N N-way replays per node.)
template <int N> constexpr int epb2l() {
  return (256 / (2 * N)) < 1 ? 1 : 256 / (2 * N);
}
template <typename T, int N, int EPB, class LD>
__global__ void __launch_bounds__(2 * N *EPB)
    k_helm2d(const __grid_constant__ Basis<T, N> B, const Geom<T> g, int64_t ne, T p,
             const T *__restrict__ pvec, T q, const T *__restrict__ qvec, int use_mass,
             const LD ld, T *__restrict__ uo, const double *__restrict__ stop) {
  if (stop && stop[0] != 0.0) return;
  constexpr int P = Pad<N>::P, AREA = N * P, NN = N * N, NT = 2 * N * EPB;
  constexpr int IT = (EPB * NN + NT - 1) / NT;
  __shared__ T su[EPB * AREA], sx[EPB * AREA], sy[EPB * AREA], sW[N];
  const int64_t e0 = (int64_t)blockIdx.x * EPB;
  const int nel = ne - e0 < EPB ? (int)(ne - e0) : EPB;
  const int t = threadIdx.x;
  if (t < N) sW[t] = B.W[t];
  __syncthreads();
#pragma unroll
  for (int it = 0; it < IT; it++) {
    const int i = t + it * NT;
    if (i >= nel * NN) continue;
    const int el = i / NN, a = i - el * NN, y = a / N, x = a - y * N;
    const int64_t e = e0 + el, node = e * NN + a;
    const int s = el * AREA + y * P + x;
    NodeGeom<T, 2> ng;
    elem_geom<T, 2>(g, e, ng);
    node_geom<T, 2>(g, node, ng);
    const T mass = sW[y] * sW[x] * ng.J;
    const T mp = pvec ? mass * pvec[node] : mass * p;
    su[s] = (T)ld.template point2<N>(e, x, y);
    sx[s] = mp * (ng.X[0] * ng.X[0]);
    sy[s] = mp * (ng.X[1] * ng.X[1]);
  }
  __syncthreads();
  {
    const int el = t / (2 * N), l = t - el * 2 * N;
    if (el < nel) {
      const bool xdir = l < N;
      const int s0 = el * AREA + (xdir ? l * P : l - N), st = xdir ? 1 : P;
      T *w = xdir ? sx : sy;
      T a[N], d[N];
#pragma unroll
      for (int m = 0; m < N; m++) a[m] = su[s0 + m * st];
      line_D<T, N>(B.D, a, d);
#pragma unroll
      for (int m = 0; m < N; m++) d[m] *= w[s0 + m * st];
      line_DT<T, N>(B.D, d, a);
#pragma unroll
      for (int m = 0; m < N; m++) w[s0 + m * st] = a[m];
    }
  }
  __syncthreads();
#pragma unroll
  for (int it = 0; it < IT; it++) {
    const int i = t + it * NT;
    if (i >= nel * NN) continue;
    const int el = i / NN, a = i - el * NN, y = a / N, x = a - y * N;
    const int64_t e = e0 + el, node = e * NN + a;
    const int s = el * AREA + y * P + x;
    T o = sx[s] + sy[s];
    if (use_mass) {
      NodeGeom<T, 2> ng;
      elem_geom<T, 2>(g, e, ng);
      node_geom<T, 2>(g, node, ng);
      o = fma(sW[y] * sW[x] * ng.J * (qvec ? qvec[node] : q), su[s], o);
    }
    uo[node] = o;
  }
}

// The same, one thread per node: N = 2, where a line has two nodes and an element as
// many nodes as lines, so that the line form only adds a trip through shared memory
// (5 M nodes: FP64 40.3 us against 49.3 by lines, FP32 28.8 against 33.0; 1.5 M: 12.4
// against 16.4 and 10.5 against 12.4).  From N = 3 on the lines are as fast or faster.
template <typename T, int N, int EPB, class LD>
__global__ void __launch_bounds__(N *N *EPB)
    k_helm2d_node(const __grid_constant__ Basis<T, N> B, const Geom<T> g, int64_t ne, T p,
             const T *__restrict__ pvec, T q, const T *__restrict__ qvec, int use_mass,
             const LD ld, T *__restrict__ uo, const double *__restrict__ stop) {
  if (stop && stop[0] != 0.0) return;
  constexpr int P = Pad<N>::P, AREA = N * P, NN = N * N;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T *s = reinterpret_cast<T *>(smem_raw) + threadIdx.y * 3 * AREA;
  T *su = s, *sgx = s + AREA, *sgy = s + 2 * AREA;
  const int t = threadIdx.x;
  const int64_t e = (int64_t)blockIdx.x * EPB + threadIdx.y;
  const bool active = e < ne;
  const int i = t % N, j = t / N;
  const int64_t node = e * NN + t;
  NodeGeom<T, 2> ng;
  ng.X[0] = ng.X[1] = ng.J = T(0);
  T uv = T(0), pv = T(1);
  if (active) {
    elem_geom<T, 2>(g, e, ng);
    node_geom<T, 2>(g, node, ng);
    uv = ld.template point2<N>(e, i, j);
    if (pvec) pv = pvec[node];
  }
  su[j * P + i] = uv;
  __syncthreads();
  T dx = B.D[i] * su[j * P];
  T dy = B.D[j] * su[i];
#pragma unroll
  for (int m = 1; m < N; m++) {
    dx = fma(B.D[i + m * N], su[j * P + m], dx);
    dy = fma(B.D[j + m * N], su[m * P + i], dy);
  }
  const T mass = B.W[j] * B.W[i] * ng.J;
  T gx = dx * (ng.X[0] * ng.X[0]);
  T gy = dy * (ng.X[1] * ng.X[1]);
  if (pvec) {
    gx *= pv;
    gy *= pv;
  }
  sgx[j * P + i] = mass * gx;
  sgy[j * P + i] = mass * gy;
  __syncthreads();
  T ox = B.D[i * N] * sgx[j * P];
  T oy = B.D[j * N] * sgy[i];
#pragma unroll
  for (int m = 1; m < N; m++) {
    ox = fma(B.D[m + i * N], sgx[j * P + m], ox);
    oy = fma(B.D[m + j * N], sgy[m * P + i], oy);
  }
  if (active) {
    T o = ox + oy;
    if (!pvec) o *= p;
    if (use_mass) {
      T mu = mass * uv;
      mu *= qvec ? qvec[node] : q;
      o += mu;
    }
    uo[node] = o;
  }
}

// ---------------------------------------------------------------------
// Single-direction reference derivative (GGrid::compute_grefderiv) and
// its physical form (GGrid::deriv): one thread per node.
// dotrans selects D^T; phys multiplies by dXidX_idir.
// ---------------------------------------------------------------------
template <typename T, int N, int DIM, int EPB>
__global__ void __launch_bounds__(N *N *(DIM == 3 ? 1 : EPB))
    k_grefderiv(const __grid_constant__ Basis<T, N> B, const Geom<T> g, int64_t ne,
                const T *__restrict__ u, int idir, int dotrans, int phys, int accum,
                T *__restrict__ du) {
  // 3-d: blockDim = (N*N) threads per element-plane loop; 2-d: (N*N, EPB)
  constexpr int NN = N * N, NE = (DIM == 3) ? NN * N : NN;
  constexpr int BPE = (DIM == 3) ? 1 : EPB;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T *su = reinterpret_cast<T *>(smem_raw) + threadIdx.y * NE;
  const int64_t e = (int64_t)blockIdx.x * BPE + threadIdx.y;
  const bool active = e < ne;
  const int64_t base = e * NE;
  for (int a = threadIdx.x; a < NE; a += NN) su[a] = active ? u[base + a] : T(0);
  __syncthreads();
  if (!active) return;
  NodeGeom<T, DIM> eg;
#pragma unroll
  for (int k = 0; k < DIM; k++) eg.X[k] = T(0);
  eg.J = T(0);
  elem_geom<T, DIM>(g, e, eg);
  for (int a = threadIdx.x; a < NE; a += NN) {
    int i = a % N, j = (a / N) % N, k = (DIM == 3) ? a / NN : 0;
    int c = idir == 1 ? i : (idir == 2 ? j : k);
    int stride = idir == 1 ? 1 : (idir == 2 ? N : NN);
    int b0 = a - c * stride;
    T s = T(0);
#pragma unroll
    for (int m = 0; m < N; m++) {
      T Dv = dotrans ? B.D[m + c * N] : B.D[c + m * N];
      s = (m == 0) ? Dv * su[b0] : fma(Dv, su[b0 + m * stride], s);
    }
    if (phys) {
      NodeGeom<T, DIM> ng = eg;
      node_geom<T, DIM>(g, base + a, ng);
      s *= ng.X[idir - 1];
    }
    du[base + a] = accum ? du[base + a] + s : s;
  }
}

}  // namespace gfk
