// k_dss_elem.cuh -- the stage passes of k_dss.cuh element by element, for 3-d
// boxes whose pass does not write an array it gathers.
//
// The lattice walks (k_dss.cuh) touch the E-vector in rows of N values, each in
// another element: about six cache-tag accesses per load and store at N = 6, at
// which rate the pass runs at a quarter of HBM bandwidth whatever the type (FP32
// and FP64 take the same time).  Here a block stages an element with one layer
// of its neighbours' copies around it (N + 2 values per direction: own, and the
// copies that the six faces, twelve edges and eight corners share), folds every
// own node from shared memory and writes only its own nodes, in memory order.
// Copies are gathered (N + 2)^3 / N^3 times instead of once, from cache; each
// class is folded once per copy, in the same order, so every copy gets the same
// bits, those of the lattice walk.
//
// A persistent block keeps what depends on the cell alone (its place in the
// neighbour element, its neighbour) in registers; per element it forms 27
// neighbour offsets and a word of face flags.
#pragma once
#include "k_dss.cuh"

namespace gfk {

constexpr int EL_THREADS = 256;

template <typename T, int N>
struct ElemTile {
  static constexpr int S = N + 2, EXT = S * S * S, NN = N * N, NNN = NN * N;
  static constexpr int EPB = (512 / NNN) < 1 ? 1 : (512 / NNN);
  static constexpr int CELLS = EPB * EXT, NODES = EPB * NNN;
  static constexpr int CPT = (CELLS + EL_THREADS - 1) / EL_THREADS;
  static constexpr int NPT = (NODES + EL_THREADS - 1) / EL_THREADS;
};

struct ElemBox {
  int ne[3], per[3], nel;
  FastDiv f0, f1;
  static ElemBox make(const BoxLattice &L) {
    ElemBox b;
    b.nel = 1;
    for (int d = 0; d < 3; d++) {
      b.ne[d] = L.ne[d];
      b.per[d] = L.per[d];
      b.nel *= L.ne[d];
    }
    b.f0 = FastDiv::make(b.ne[0]);
    b.f1 = FastDiv::make(b.ne[1]);
    return b;
  }
};

// Along one direction, a node of face f (1 low, 2 high, 0 none): the offsets of
// its copies in fold order (ascending element; a wrapped neighbour comes after
// at the low face of the first element, before at the high face of the last).
// flags: bit 0/1 a neighbour at the low/high face, bit 2/3 it is a wrapped one.
__device__ __forceinline__ int elem_copies(int f, int flags, int st, int &s0, int &s1) {
  s0 = s1 = 0;
  if (f == 0 || !(flags & f)) return 1;
  const int other = f == 1 ? -st : st;
  const bool first = (f == 1) != ((flags & (f << 2)) != 0);
  s0 = first ? other : 0;
  s1 = first ? 0 : other;
  return 2;
}

// NC components from the pass's component 0
template <typename T, int MODE, int N, int NC>
__global__ void __launch_bounds__(EL_THREADS)
    k_rk_elem(const __grid_constant__ RKPass<T> p, const ElemBox box) {
  using E = ElemTile<T, N>;
  using M = RKMode<MODE>;
  constexpr int S = E::S, P = N - 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T *sm = reinterpret_cast<T *>(smem_raw);  // NC * CELLS
  __shared__ int nb[E::EPB * 27], fl[E::EPB];

  // this thread's cells: slot in nb, and offset in that element; its nodes: the
  // cell of the node and its faces
  int cnb[E::CPT], cloc[E::CPT], ncell[E::NPT], nface[E::NPT];
#pragma unroll
  for (int i = 0; i < E::CPT; i++) {
    const int c = (int)threadIdx.x + i * EL_THREADS;
    const int el = c / E::EXT, a = c - el * E::EXT;
    const int z = a / (S * S), y = (a / S) % S, x = a % S;
    // -1, 0 or 1 along each direction, and the local index there
    const int dx = x == 0 ? 0 : (x == S - 1 ? 2 : 1), lx = x == 0 ? P : (x == S - 1 ? 0 : x - 1);
    const int dy = y == 0 ? 0 : (y == S - 1 ? 2 : 1), ly = y == 0 ? P : (y == S - 1 ? 0 : y - 1);
    const int dz = z == 0 ? 0 : (z == S - 1 ? 2 : 1), lz = z == 0 ? P : (z == S - 1 ? 0 : z - 1);
    cnb[i] = c < E::CELLS ? el * 27 + dx + 3 * (dy + 3 * dz) : -1;
    cloc[i] = lx + N * (ly + N * lz);
  }
#pragma unroll
  for (int i = 0; i < E::NPT; i++) {
    const int n = (int)threadIdx.x + i * EL_THREADS;
    const int el = n / E::NNN, a = n - el * E::NNN;
    const int z = a / E::NN, y = (a / N) % N, x = a % N;
    auto face = [](int l) { return l == 0 ? 1 : (l == P ? 2 : 0); };
    ncell[i] = n < E::NODES ? el * E::EXT + ((z + 1) * S + y + 1) * S + x + 1 : -1;
    nface[i] = face(x) | face(y) << 2 | face(z) << 4 | el << 6;
  }

  auto fold = [&](int i, const T *src, auto value) {  // over node i's copies in src
    const int f = nface[i], flags = fl[f >> 6];
    int x0, x1, y0, y1, z0, z1;
    const int nx = elem_copies(f & 3, flags, 1, x0, x1);
    const int ny = elem_copies((f >> 2) & 3, flags >> 4, S, y0, y1);
    const int nz = elem_copies((f >> 4) & 3, flags >> 8, S * S, z0, z1);
    T s = T(0);
#pragma unroll
    for (int az = 0; az < 2; az++) {
      if (az >= nz) break;
#pragma unroll
      for (int ay = 0; ay < 2; ay++) {
        if (ay >= ny) break;
        const T *row = src + ncell[i] + (az ? z1 : z0) + (ay ? y1 : y0);
        s = __fadd_rn_t(s, value(row[x0]));
        if (nx > 1) s = __fadd_rn_t(s, value(row[x1]));
      }
    }
    return s * ((nx > 1 ? T(0.5) : T(1)) * (ny > 1 ? T(0.5) : T(1)) * (nz > 1 ? T(0.5) : T(1)));
  };

  for (int e0 = blockIdx.x * E::EPB; e0 < box.nel; e0 += gridDim.x * E::EPB) {
    for (int i = threadIdx.x; i < E::EPB * 27; i += EL_THREADS) {
      const int el = i / 27, d = i - el * 27, e = e0 + el;
      const int row = box.f0.div(e), ex = e - row * box.ne[0];
      const int ez = box.f1.div(row), ey = row - ez * box.ne[1];
      const int ec[3] = {ex, ey, ez}, dd[3] = {d % 3 - 1, (d / 3) % 3 - 1, d / 9 - 1};
      int at[3], flags = 0;
      bool ok = e < box.nel;
#pragma unroll
      for (int k = 0; k < 3; k++) {
        at[k] = ec[k] + dd[k];
        const bool lo = ec[k] == 0, hi = ec[k] == box.ne[k] - 1;
        if (at[k] < 0 || at[k] >= box.ne[k]) {
          ok = ok && box.per[k];
          at[k] = at[k] < 0 ? box.ne[k] - 1 : 0;
        }
        flags |= ((!lo || box.per[k] ? 1 : 0) | (!hi || box.per[k] ? 2 : 0) | (lo ? 4 : 0) |
                  (hi ? 8 : 0)) << (4 * k);
      }
      nb[i] = ok ? (at[0] + box.ne[0] * (at[1] + box.ne[1] * at[2])) * E::NNN : -1;
      if (d == 13) fl[el] = flags;
    }
    __syncthreads();
    // gather: the cells of every component
    auto fill = [&](auto load) {
      int off[E::CPT];
#pragma unroll
      for (int i = 0; i < E::CPT; i++) {
        const int b = cnb[i] >= 0 ? nb[cnb[i]] : -1;
        off[i] = b >= 0 ? b + cloc[i] : -1;
      }
#pragma unroll
      for (int j = 0; j < NC; j++) {
        T v[E::CPT];
#pragma unroll
        for (int i = 0; i < E::CPT; i++) v[i] = off[i] >= 0 ? load(j, off[i]) : T(0);
#pragma unroll
        for (int i = 0; i < E::CPT; i++)
          if (cnb[i] >= 0) sm[j * E::CELLS + (int)threadIdx.x + i * EL_THREADS] = v[i];
      }
    };
    fill([&](int j, int m) { return p.x[j][m]; });
    // own values of the other arrays, in flight while the gather completes
    T u0[E::NPT][NC], c0[E::NPT][NC], s[E::NPT][NC];
    const int64_t base = (int64_t)e0 * E::NNN + threadIdx.x;
    bool on[E::NPT];
#pragma unroll
    for (int i = 0; i < E::NPT; i++) {
      on[i] = ncell[i] >= 0 && e0 + (nface[i] >> 6) < box.nel;
#pragma unroll
      for (int j = 0; j < NC; j++) {
        const int64_t m = base + i * EL_THREADS;
        u0[i][j] = M::MID && MODE != RK_MIDS && on[i] ? p.uin[j][m] : T(0);
        c0[i][j] = M::MID && on[i] ? p.accin[j][m] : T(0);
      }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < E::NPT; i++) {
      if (!on[i]) continue;
#pragma unroll
      for (int j = 0; j < NC; j++) {
        const int64_t m = base + i * EL_THREADS;
        s[i][j] = fold(i, sm + j * E::CELLS, [](T v) { return v; });
        if constexpr (MODE != RK_MIDS)
          rk_write<T, MODE>(p, j, s[i][j], T(0), sm[j * E::CELLS + ncell[i]], u0[i][j], c0[i][j], m);
      }
    }
    __syncthreads();
    if constexpr (MODE == RK_MIDS) {  // the second fold, of the stage input
      fill([&](int j, int m) { return p.uin[j][m]; });
      __syncthreads();
#pragma unroll
      for (int i = 0; i < E::NPT; i++) {
        if (!on[i]) continue;
#pragma unroll
        for (int j = 0; j < NC; j++) {
          const T k = s[i][j];
          const T o = fold(i, sm + j * E::CELLS, [&](T v) { return rk_input_point(v, p.b, k); });
          rk_write<T, MODE>(p, j, k, o, T(0), T(0), c0[i][j], base + i * EL_THREADS);
        }
      }
      __syncthreads();
    }
  }
}

// The smallest N whose passes of this mode it takes (elem_pass_ok, rk_pass.cuh).
template <int MODE>
constexpr int el_min_n() {
  return MODE == RK_MID || RKMode<MODE>::ADJ ? 3 : (MODE == RK_MIDS ? 5 : GF_MAXN + 1);
}

template <typename T, int MODE>
struct RKElemLaunch {
  template <int N>
  struct F {
    static int run(gf_problem *prob, cudaStream_t st, int nc, const RKPass<T> &p) {
      if constexpr (N < el_min_n<MODE>()) {
        return GF_ERR_UNSUPPORTED;
      } else if (nc == 3) {
        return go<N, 3>(prob, st, p);
      } else {
        for (int j = 0; j < nc; j++) {  // one component at a time
          RKPass<T> q = p;
          q.x[0] = p.x[j];
          q.uin[0] = p.uin[j];
          q.y[0] = p.y[j];
          q.y2[0] = p.y2[j];
          q.accin[0] = p.accin[j];
          q.out[0] = p.out[j];
          q.acc[0] = p.acc[j];
          q.aux[0] = p.aux[j];
          int rc = go<N, 1>(prob, st, q);
          if (rc) return rc;
        }
        return GF_OK;
      }
    }
    template <int N2, int NC>
    static int go(gf_problem *prob, cudaStream_t st, const RKPass<T> &p) {
      using E = ElemTile<T, N2>;
      constexpr size_t smem = sizeof(T) * NC * E::CELLS;
      auto kern = k_rk_elem<T, MODE, N2, NC>;
      if (!set_smem(kern, smem)) return GF_ERR_CUDA;
      // blocks per SM (of the first device; the same kernel on any sm_100a)
      static const int resident = [&] {
        int nb = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kern, EL_THREADS, smem);
        return std::max(nb, 1);
      }();
      const int64_t groups = (prob->ne + E::EPB - 1) / E::EPB;
      prob->launches++;
      kern<<<(unsigned)std::min<int64_t>(groups, (int64_t)resident * prob->ctx->sm_count),
             EL_THREADS, smem, st>>>(p, ElemBox::make(prob->box));
      return GF_OK;
    }
  };
};

}  // namespace gfk
