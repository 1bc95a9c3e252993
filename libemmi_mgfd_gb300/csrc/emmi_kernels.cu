// Multigrid kernels for the finite-integration curl-curl system on sm_103a.
//
// residual      r = f - A u, fused FP64 norm             (src/gmg.c:1316-1410)
// line sweep    zebra (4-colour) line block relaxation,  (src/gmg.c:340-1298)
//               one thread per line, streaming complex-symmetric LDL^T
// point sweep   8-colour node-patch (6x6) block relaxation (src/gmg.c:116-336)
// restrict      f_c = P^T r_f as a gather                (src/gmg.c:1510-1573)
// prolong       u_f += P u_c                              (src/gmg.c:1463-1505)
// coarsen       coarse-cell sums / repeat                 (src/gmg.c:1803-1858)
//
// The smoothers update in correction form: each block solves A_bb d = r_b
// with r_b the current residual of its rows and adds d.  In exact arithmetic
// this equals the reference's zero-then-solve form (src/gmg.c:395-405) and it
// keeps the relative precision of complex64 updates as the solve converges.
// Blocks of one colour neither overlap nor read each other's unknowns: a line
// along d through (ta,tb) reads transverse neighbours at ta+-1 / tb+-1 only
// (checked by tests/test_coloring.py), so a colour is one parallel launch.
#include "emmi_line.cuh"
#include "emmi_node.cuh"

#include <cstdio>
#include <type_traits>

namespace emmi {

long line_count(const int n[3], int d, int color) {
  const int a = (d == 0) ? 1 : 0, b = (d == 2) ? 1 : 2;
  const int pa = color & 1, pb = (color >> 1) & 1;
  const int fa = pa ? 1 : 2, fb = pb ? 1 : 2;
  const long la = (n[a] - 1 >= fa) ? (n[a] - 1 - fa) / 2 + 1 : 0;
  const long lb = (n[b] - 1 >= fb) ? (n[b] - 1 - fb) / 2 + 1 : 0;
  return la * lb;
}

long line_scratch_elems(const int n[3], int d, int nrhs) {
  long mx = 0;
  for (int c = 0; c < 4; c++) mx = line_count(n, d, c) > mx ? line_count(n, d, c) : mx;
  return (long)(5 * n[d] - 4) * 6 * mx * nrhs;
}

// ------------------------------------------------------------ reductions
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}
// a thread's partial sum of squares in working precision: complex64
// residuals square and add across the warp in fp32 and widen once per warp
// (conversions to FP64 and FP64 arithmetic are low-rate on this GPU); the
// block and the grid sum in FP64
template <typename T>
__device__ __forceinline__ double warp_partial(T v) {
  if constexpr (sizeof(T) == 4) return (double)warp_sum(v);
  else return warp_sum((double)v);
}

__device__ __forceinline__ void block_add(double v, double* dst) {
  __shared__ double red[32];
  v = warp_sum(v);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (lane == 0) red[w] = v;
  __syncthreads();
  if (w == 0) {
    const int nw = (blockDim.x + 31) >> 5;
    v = lane < nw ? red[lane] : 0.0;
    v = warp_sum(v);
    if (lane == 0 && v != 0.0) atomicAdd(dst, v);
  }
}

// block_add for a thread's partial of type T (see warp_partial)
template <typename T>
__device__ __forceinline__ void block_add_t(T v, double* dst) {
  __shared__ double red[32];
  double w = warp_partial<T>(v);
  const int lane = threadIdx.x & 31, wi = threadIdx.x >> 5;
  if (lane == 0) red[wi] = w;
  __syncthreads();
  if (wi == 0) {
    const int nw = (blockDim.x + 31) >> 5;
    w = lane < nw ? red[lane] : 0.0;
    w = warp_sum(w);
    if (lane == 0 && w != 0.0) atomicAdd(dst, w);
  }
}

// ------------------------------------------------------------ residual
template <int C>
__device__ __forceinline__ bool is_unknown(const int n[3], const int P[3]) {
  constexpr int p = Cyc<C>::p, q = Cyc<C>::q;
  return P[C] < n[C] && P[p] >= 1 && P[p] < n[p] && P[q] >= 1 && P[q] < n[q];
}

template <typename T, typename TO, int C>
__device__ __forceinline__ T residual_comp(const LevelView<T>& L, const C_t<T>* u,
                                                const C_t<T>* f, const T* cells, const Geo<T>& G,
                                                T wmu, const int P[3], long s, const long ss[3],
                                                C_t<TO>* rout) {
  const int o = C * (int)L.S + (int)s;  // 32-bit offset within the RHS's field
  C_t<T> r = f ? f[o] : mk<T>(0, 0);     // f null: r = -A u
  if (is_unknown<C>(L.n, P)) {
    EdgeCoef<T> e;
    const C_t<T> au = apply_row<T, C, 0>(L, u, cells, G, wmu, P, s, ss, e);
    r = csub<T>(r, au);
  }
  if (rout) rout[o] = mk<TO>((TO)r.x, (TO)r.y);
  return r.x * r.x + r.y * r.y;
}

// a thread per (component, slot), the component = blockIdx.z: one edge
// equation per thread keeps more independent loads in flight than three
template <typename T, typename TO>
__global__ void __launch_bounds__(256) k_residual(LevelView<T> L, C_t<TO>* __restrict__ rout,
                                                  double* __restrict__ norm2) {
  dep_wait();
  dep_next();
  const int rhs = blockIdx.y;
  if (L.active && !L.active[rhs]) return;
  const long s = blockIdx.x * (long)blockDim.x + threadIdx.x;
  T acc = 0;
  if (s < L.S) {
    const int n0 = L.n[0] + 1, n1 = L.n[1] + 1;
    int P[3];
    slot_nodes(s, L, P);
    const long ss[3] = {1, (long)n0, (long)n0 * n1};
    const C_t<T>* u = L.u + (long)rhs * 3 * L.S;
    const C_t<T>* f = L.f ? L.f + (long)rhs * 3 * L.S : nullptr;
    const T* cells = L.cells + (long)op_of(L, rhs) * 4 * L.ncell;
    const Geo<T> G{L.geo + (long)op_of(L, rhs) * L.gstride, L.gmax1};
    const T wmu = L.wmu[rhs];
    C_t<TO>* ro = rout ? rout + (long)rhs * 3 * L.S : nullptr;
    switch (blockIdx.z) {
      case 0: acc = residual_comp<T, TO, 0>(L, u, f, cells, G, wmu, P, s, ss, ro); break;
      case 1: acc = residual_comp<T, TO, 1>(L, u, f, cells, G, wmu, P, s, ss, ro); break;
      default: acc = residual_comp<T, TO, 2>(L, u, f, cells, G, wmu, P, s, ss, ro); break;
    }
  }
  if (norm2) block_add_t<T>(acc, norm2 + rhs);
}

// the complex64 residual with the coefficients from the spacings: a thread per
// slot and its three edges, each value they share loaded once (node_residual).
// Level 0 of 4 RHS at 128^3: 232 us, 3.0 TB/s, where an edge a thread took 318
// (and the tensor-copy one 316); bound by load latency at 24 warps an SM.
// Columns of eight planes with the shared values in registers take as long
// (239 us: fewer loads, 16 warps).
__global__ void __launch_bounds__(256) k_residual_nodes(LevelView<float> L,
                                                        float2* __restrict__ rout,
                                                        double* __restrict__ norm2) {
  dep_wait();
  dep_next();
  const int rhs = blockIdx.y;
  if (L.active && !L.active[rhs]) return;
  const long s = blockIdx.x * (long)blockDim.x + threadIdx.x;
  float acc = 0.f;
  if (s < L.S) {
    int P[3];
    slot_nodes(s, L, P);
    const int op = op_of(L, rhs);
    const Geo<float> G{L.geo + (long)op * L.gstride, L.gmax1};
    float2 r[3], d[3];
    bool unk[3];
    node_residual(L, L.u + (long)rhs * 3 * L.S, L.f ? L.f + (long)rhs * 3 * L.S : nullptr,
                  L.cells + (long)op * 4 * L.ncell, G, L.wmu[rhs], P, (int)s, r, d, unk);
#pragma unroll
    for (int c = 0; c < 3; c++) {
      if (rout) rout[((long)rhs * 3 + c) * L.S + s] = r[c];
      acc += r[c].x * r[c].x + r[c].y * r[c].y;
    }
  }
  if (norm2) block_add_t<float>(acc, norm2 + rhs);
}

template <typename T, typename TO>
void launch_residual(const LevelView<T>& L, C_t<TO>* rout, double* norm2, cudaStream_t st) {
  // with a norm the kernel follows a memset, not another kernel of the cycle
  auto go = [&](auto k, unsigned nz) {
    const dim3 grid((unsigned)((L.S + 255) / 256), L.nrhs, nz);
    if (norm2) k<<<grid, 256, 0, st>>>(L, rout, norm2);
    else launch_dep(k, grid, 256, 0, st, L, rout, norm2);
  };
  if constexpr (sizeof(T) == 4 && sizeof(TO) == 4) {
    if (L.imu_vol) return go(k_residual_nodes, 1);
  }
  go(k_residual<T, TO>, 3);
}

// ------------------------------------------------------------ stored FP64 coefficients
// The FP64 refinement residual of the mixed solver recomputes, per edge, 8
// coupling values with 8 divisions at GB300's FP64 rate.  They depend on the
// operator only (the imaginary diagonal on omega too, as -omega*mu0 * sbar),
// so they are stored once per operator: planes [op][10][3][S] of kpp, kpm,
// kqp, kqm (c[0..3]), xp, xm, yp, ym (c[4], c[7], c[8], c[11]), the real
// diagonal and sbar, taken from edge_coef itself.  The residual then applies
// them in edge_coef/apply_row's order: the same result, bit for bit.
constexpr int kCoef = 10;

template <int C>
__device__ __forceinline__ void store_coef(const LevelView<double>& L, const double* cells,
                                           const Geo<double>& G, const int P[3], long s,
                                           double* __restrict__ out) {
  EdgeCoef<double> e;
  // omega*mu0 = -1 gives dim = -(-1)*sbar = sbar exactly
  edge_coef<double, C>(L.n, P, cells + (long)C * L.ncell, cells + 3 * L.ncell, G, -1.0, e);
  const long n3s = 3 * L.S, o = (long)C * L.S + s;
  const double v[kCoef] = {e.c[0], e.c[1], e.c[2], e.c[3], e.c[4], e.c[7], e.c[8], e.c[11],
                           e.dre, e.dim};
#pragma unroll
  for (int k = 0; k < kCoef; k++) out[k * n3s + o] = v[k];
}

// blockIdx.y = operator
__global__ void __launch_bounds__(256) k_coef64(LevelView<double> L, double* __restrict__ coef) {
  const int op = blockIdx.y;
  const long s = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (s >= L.S) return;
  int P[3];
  slot_nodes(s, L, P);
  const double* cells = L.cells + (long)op * 4 * L.ncell;
  const Geo<double> G{L.geo + (long)op * L.gstride, L.gmax1};
  double* out = coef + (long)op * kCoef * 3 * L.S;
  if (is_unknown<0>(L.n, P)) store_coef<0>(L, cells, G, P, s, out);
  if (is_unknown<1>(L.n, P)) store_coef<1>(L, cells, G, P, s, out);
  if (is_unknown<2>(L.n, P)) store_coef<2>(L, cells, G, P, s, out);
}

template <typename TO, int C>
__device__ __forceinline__ double residual_comp_coef(const LevelView<double>& L,
                                                     const double2* u, const double2* f,
                                                     const double* __restrict__ cf, double wmu,
                                                     const int P[3], long s, const long ss[3],
                                                     C_t<TO>* rout) {
  double2 r = f ? f[(long)C * L.S + s] : make_double2(0.0, 0.0);
  if (is_unknown<C>(L.n, P)) {
    const long n3s = 3 * L.S, o = (long)C * L.S + s;
    double k8[kCoef];
#pragma unroll
    for (int k = 0; k < kCoef; k++) k8[k] = ldro(cf + k * n3s + o);
    const double c[12] = {k8[0], k8[1], k8[2], k8[3], k8[4], -k8[4], -k8[5], k8[5],
                          k8[6], -k8[6], -k8[7], k8[7]};
    const double dre = k8[8], dim = -wmu * k8[9];
    const double2 uc = ldro(u + o);
    double ar = dre * uc.x - dim * uc.y;
    double ai = dre * uc.y + dim * uc.x;
#pragma unroll
    for (int k = 0; k < 12; k++) {
      const double2 v = ldro(u + s + nbr_slot_delta<C>(k, ss, L.S));
      ar += c[k] * v.x;
      ai += c[k] * v.y;
    }
    r = csub<double>(r, mk<double>(ar, ai));
  }
  if (rout) rout[(long)C * L.S + s] = mk<TO>((TO)r.x, (TO)r.y);
  return r.x * r.x + r.y * r.y;
}

template <typename TO>
__global__ void __launch_bounds__(256) k_residual_coef(LevelView<double> L,
                                                       const double* __restrict__ coef,
                                                       C_t<TO>* __restrict__ rout,
                                                       double* __restrict__ norm2) {
  const int rhs = blockIdx.y;
  if (L.active && !L.active[rhs]) return;
  const long s = blockIdx.x * (long)blockDim.x + threadIdx.x;
  double acc = 0.0;
  if (s < L.S) {
    const int n0 = L.n[0] + 1, n1 = L.n[1] + 1;
    int P[3];
    slot_nodes(s, L, P);
    const long ss[3] = {1, (long)n0, (long)n0 * n1};
    const double2* u = L.u + (long)rhs * 3 * L.S;
    const double2* f = L.f ? L.f + (long)rhs * 3 * L.S : nullptr;
    const double* cf = coef + (long)op_of(L, rhs) * kCoef * 3 * L.S;
    const double wmu = L.wmu[rhs];
    C_t<TO>* ro = rout ? rout + (long)rhs * 3 * L.S : nullptr;
    acc += residual_comp_coef<TO, 0>(L, u, f, cf, wmu, P, s, ss, ro);
    acc += residual_comp_coef<TO, 1>(L, u, f, cf, wmu, P, s, ss, ro);
    acc += residual_comp_coef<TO, 2>(L, u, f, cf, wmu, P, s, ss, ro);
  }
  if (norm2) block_add(acc, norm2 + rhs);
}

long coef64_elems(const int n[3]) {
  return (long)kCoef * 3 * (n[0] + 1) * (n[1] + 1) * (n[2] + 1);
}

void launch_coef64(const LevelView<double>& L, double* coef, cudaStream_t st) {
  dim3 grid((unsigned)((L.S + 255) / 256), L.nrhs);
  k_coef64<<<grid, 256, 0, st>>>(L, coef);
}

template <typename TO>
void launch_residual_coef(const LevelView<double>& L, const double* coef, C_t<TO>* rout,
                          double* norm2, cudaStream_t st) {
  dim3 grid((unsigned)((L.S + 255) / 256), L.nrhs);
  k_residual_coef<TO><<<grid, 256, 0, st>>>(L, coef, rout, norm2);
}
template void launch_residual_coef<float>(const LevelView<double>&, const double*, C_t<float>*,
                                          double*, cudaStream_t);
template void launch_residual_coef<double>(const LevelView<double>&, const double*,
                                           C_t<double>*, double*, cudaStream_t);

template <typename T>
__global__ void __launch_bounds__(256) k_norm(const C_t<T>* __restrict__ v, long n, const int* active,
                                              double* norm2) {
  const int rhs = blockIdx.y;
  if (active && !active[rhs]) return;
  double acc = 0;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    const C_t<T> z = v[(long)rhs * n + i];
    acc += (double)z.x * z.x + (double)z.y * z.y;
  }
  block_add(acc, norm2 + rhs);
}

template <typename T>
void launch_norm(const C_t<T>* v, long n3s, int nrhs, const int* active, double* norm2,
                 cudaStream_t st) {
  long blocks = (n3s + 255) / 256;
  if (blocks > 1216) blocks = 1216;
  dim3 grid((unsigned)blocks, nrhs);
  k_norm<T><<<grid, 256, 0, st>>>(v, n3s, active, norm2);
}

// ------------------------------------------------------------ line sweep
// One colour of line relaxation along D is three launches:
//   assemble  thread per (line, node): for the rows of the node, the lower
//             band entries (offsets -5..-1, real), the complex diagonal and
//             the current residual, into a record buffer [row][line][12];
//             threads run along the contiguous memory direction so every
//             stencil load is coalesced
//   solve     thread per line: streaming complex-symmetric LDL^T over its
//             records (factors written in place), then back substitution;
//             records of one row are contiguous across lines (coalesced)
//   apply     thread per (line, node): u += correction, coalesced like
//             assemble
// Record of one row, T-typed: [0..4] band, [5,6] diagonal, [7,8] residual;
// after the forward pass [0..9] = l_1..l_5 (complex), [10,11] = z; after the
// backward pass [10,11] = the correction x.
// Records are stored as 16-byte planes, [row][plane][line]: plane q of a row
// holds record values [q*L, q*L+L) with L = 16/sizeof(T) (3 planes for float,
// 6 for double), so one warp-wide 16-byte access of consecutive lines reads
// or writes 512 contiguous bytes.
// the record of row type TT of node s: band entries, diagonal, residual
template <typename T, int D, int TT, int C>
__device__ __forceinline__ void assemble_row(const LevelView<T>& L, const C_t<T>* u,
                                             const C_t<T>* f, const T* cells, const Geo<T>& G,
                                             T wmu, int ta, int tb, int s, int row,
                                             const long ss[3], typename Vec16<T>::V* rp,
                                             long ps) {
  constexpr int A = (D == 0) ? 1 : 0, B = (D == 2) ? 1 : 2;
  int P[3];
  P[D] = (TT == 0) ? s - 1 : s;
  P[A] = ta - (TT == 1 ? 1 : 0);
  P[B] = tb - (TT == 3 ? 1 : 0);
  const int sl = P[0] + (L.n[0] + 1) * (P[1] + (L.n[1] + 1) * P[2]);  // 32-bit slot
  EdgeCoef<T> e;
  const C_t<T> au = apply_row<T, C, 2, true>(L, u, cells, G, wmu, P, sl, ss, e);
  const C_t<T> r = csub<T>(f[C * (int)L.S + sl], au);
  T band[5] = {0, 0, 0, 0, 0};
#define LINE_ENTRY(K)                                                         \
  {                                                                           \
    constexpr int off = line_off(D, TT, K);                                   \
    if constexpr (off < 0) {                                                  \
      if (row + off >= 0) band[5 + off] = e.c[K];                             \
    }                                                                         \
  }
  LINE_ENTRY(0) LINE_ENTRY(1) LINE_ENTRY(2) LINE_ENTRY(3) LINE_ENTRY(4) LINE_ENTRY(5)
  LINE_ENTRY(6) LINE_ENTRY(7) LINE_ENTRY(8) LINE_ENTRY(9) LINE_ENTRY(10) LINE_ENTRY(11)
#undef LINE_ENTRY
  T rec[kRec];
#pragma unroll
  for (int i = 0; i < 5; i++) rec[i] = band[i];
  rec[5] = e.dre;
  rec[6] = e.dim;
  rec[7] = r.x;
  rec[8] = r.y;
  rec[9] = rec[10] = rec[11] = 0;
  rec_put<T>(rp, ps, rec);
}

// neighbouring lines are neighbouring slots
template <typename T, int D>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 3 : 2) k_line_assemble(LevelView<T> L,
                                                                              int pa, int pb,
                                                                              T* __restrict__ buf) {
  constexpr int A = (D == 0) ? 1 : 0, B = (D == 2) ? 1 : 2;
  const int rhs = blockIdx.y;
  if (L.active && !L.active[rhs]) return;
  const LineGeom g = line_geom<D>(L.n, pa, pb);
  long l;
  int s;
  if (!line_item<D>(g, blockIdx.x * (long)blockDim.x + threadIdx.x, l, s)) return;
  const unsigned lq = (unsigned)l / (unsigned)g.la;
  const int ta = g.fa + 2 * (int)((unsigned)l - lq * (unsigned)g.la), tb = g.fb + 2 * (int)lq;
  const int n0 = L.n[0] + 1, n1 = L.n[1] + 1;
  const long ss[3] = {1, (long)n0, (long)n0 * n1};
  const C_t<T>* u = L.u + (long)rhs * 3 * L.S;
  const C_t<T>* f = L.f + (long)rhs * 3 * L.S;
  const T* cells = L.cells + (long)op_of(L, rhs) * 4 * L.ncell;
  const Geo<T> G{L.geo + (long)op_of(L, rhs) * L.gstride, L.gmax1};
  const T wmu = L.wmu[rhs];
  using V = typename Vec16<T>::V;
  V* base = reinterpret_cast<V*>(buf) + (long)rhs * g.m * kPlanes<T> * g.nl;
  const long ps = g.nl;
  const int r0 = 5 * (s - 1);
  auto rec = [&](int row) { return base + (long)row * kPlanes<T> * g.nl + l; };
  assemble_row<T, D, 0, D>(L, u, f, cells, G, wmu, ta, tb, s, r0, ss, rec(r0), ps);
  if (s < g.nd) {
    assemble_row<T, D, 1, A>(L, u, f, cells, G, wmu, ta, tb, s, r0 + 1, ss, rec(r0 + 1), ps);
    assemble_row<T, D, 2, A>(L, u, f, cells, G, wmu, ta, tb, s, r0 + 2, ss, rec(r0 + 2), ps);
    assemble_row<T, D, 3, B>(L, u, f, cells, G, wmu, ta, tb, s, r0 + 3, ss, rec(r0 + 3), ps);
    assemble_row<T, D, 4, B>(L, u, f, cells, G, wmu, ta, tb, s, r0 + 4, ss, rec(r0 + 4), ps);
  }
}

// one thread per (row type, line, node), row type slowest: x lines, where a
// thread owning all five rows of a node holds too many registers for the
// latency of its scattered record stores (a warp shares one row type)
template <typename T, int D>
__global__ void __launch_bounds__(256) k_line_assemble_rows(LevelView<T> L, int pa, int pb,
                                                            T* __restrict__ buf) {
  constexpr int A = (D == 0) ? 1 : 0, B = (D == 2) ? 1 : 2;
  const int rhs = blockIdx.y;
  if (L.active && !L.active[rhs]) return;
  const LineGeom g = line_geom<D>(L.n, pa, pb);
  const long items = g.nl * g.nd;
  const long id = blockIdx.x * (long)blockDim.x + threadIdx.x;
  const int rt = (int)((unsigned)id / (unsigned)items);
  if (rt >= 5) return;
  long l;
  int s;
  if (!line_item<D>(g, id - rt * items, l, s)) return;
  if (rt > 0 && s == g.nd) return;  // the last node carries only its E_D row
  const unsigned lq = (unsigned)l / (unsigned)g.la;
  const int ta = g.fa + 2 * (int)((unsigned)l - lq * (unsigned)g.la), tb = g.fb + 2 * (int)lq;
  const int n0 = L.n[0] + 1, n1 = L.n[1] + 1;
  const long ss[3] = {1, (long)n0, (long)n0 * n1};
  const C_t<T>* u = L.u + (long)rhs * 3 * L.S;
  const C_t<T>* f = L.f + (long)rhs * 3 * L.S;
  const T* cells = L.cells + (long)op_of(L, rhs) * 4 * L.ncell;
  const Geo<T> G{L.geo + (long)op_of(L, rhs) * L.gstride, L.gmax1};
  const T wmu = L.wmu[rhs];
  using V = typename Vec16<T>::V;
  V* base = reinterpret_cast<V*>(buf) + (long)rhs * g.m * kPlanes<T> * g.nl;
  const long ps = g.nl;
  const int row = 5 * (s - 1) + rt;
  V* rp = base + (long)row * kPlanes<T> * g.nl + l;
  switch (rt) {
    case 0: assemble_row<T, D, 0, D>(L, u, f, cells, G, wmu, ta, tb, s, row, ss, rp, ps); break;
    case 1: assemble_row<T, D, 1, A>(L, u, f, cells, G, wmu, ta, tb, s, row, ss, rp, ps); break;
    case 2: assemble_row<T, D, 2, A>(L, u, f, cells, G, wmu, ta, tb, s, row, ss, rp, ps); break;
    case 3: assemble_row<T, D, 3, B>(L, u, f, cells, G, wmu, ta, tb, s, row, ss, rp, ps); break;
    default: assemble_row<T, D, 4, B>(L, u, f, cells, G, wmu, ta, tb, s, row, ss, rp, ps); break;
  }
}

// Each thread streams its line's records through a private ring of kRing
// rows in shared memory ([slot][plane][thread], conflict-free 16-byte
// accesses), filled by cp.async kRing-1 rows ahead of the elimination: the
// row-to-row dependency of the factorization no longer waits on a memory
// round trip.
template <typename T>
__global__ void __launch_bounds__(kSolveThreads) k_line_solve(const int* __restrict__ active,
                                                              long nl, int m,
                                                              T* __restrict__ buf) {
  using V = typename Vec16<T>::V;
  constexpr int NP = kPlanes<T>;
  __shared__ V ring[kRing][NP][kSolveThreads];
  const int rhs = blockIdx.y;
  if (active && !active[rhs]) return;
  const int tid = threadIdx.x;
  const long l = blockIdx.x * (long)blockDim.x + tid;
  if (l >= nl) return;
  V* base = reinterpret_cast<V*>(buf) + (long)rhs * m * NP * nl + l;
  const long rs = NP * nl;  // distance between rows
  auto issue = [&](int row) {
    const V* src = base + (long)row * rs;
    const int slot = row % kRing;
#pragma unroll
    for (int q = 0; q < NP; q++) cp_async16(&ring[slot][q][tid], src + q * nl);
  };
  auto take = [&](int row, T (&v)[kRec]) {
    const int slot = row % kRing;
#pragma unroll
    for (int q = 0; q < NP; q++) unpack16(ring[slot][q][tid], v + q * kLanes<T>);
  };
  C_t<T> W[21], y[6];
#pragma unroll
  for (int i = 0; i < 21; i++) W[i] = mk<T>(0, 0);
#pragma unroll
  for (int i = 0; i < 5; i++) {
    W[WI(i, i)] = mk<T>(1, 0);  // dummy leading rows
    y[i] = mk<T>(0, 0);
  }
  for (int p = 0; p < kRing - 1; p++) {
    if (p < m) issue(p);
    cp_async_commit();
  }
  // forward: arriving row r eliminates pivot r-5
  for (int row = 0; row < m + 5; row++) {
    if (row < m) {
      if (row + kRing - 1 < m) issue(row + kRing - 1);
      cp_async_commit();
      cp_async_wait<kRing - 1>();
      T nxt[kRec];
      take(row, nxt);
#pragma unroll
      for (int j = 0; j < 5; j++) W[WI(5, j)] = mk<T>(nxt[j], 0);
      W[WI(5, 5)] = mk<T>(nxt[5], nxt[6]);
      y[5] = mk<T>(nxt[7], nxt[8]);
    } else {
#pragma unroll
      for (int j = 0; j < 5; j++) W[WI(5, j)] = mk<T>(0, 0);
      W[WI(5, 5)] = mk<T>(1, 0);
      y[5] = mk<T>(0, 0);
    }
    const C_t<T> id = crcp<T>(W[0]);
    C_t<T> lq[6];
#pragma unroll
    for (int i = 1; i < 6; i++) lq[i] = cmul<T>(W[WI(i, 0)], id);
#pragma unroll
    for (int i = 1; i < 6; i++) {
#pragma unroll
      for (int j = 1; j <= i; j++) W[WI(i, j)] = cfms<T>(W[WI(i, j)], lq[i], W[WI(j, 0)]);
      y[i] = cfms<T>(y[i], lq[i], y[0]);
    }
    const int piv = row - 5;
    if (piv >= 0) {
      const C_t<T> z = cmul<T>(y[0], id);
      T o[kRec];
#pragma unroll
      for (int i = 1; i < 6; i++) {
        o[2 * (i - 1)] = lq[i].x;
        o[2 * (i - 1) + 1] = lq[i].y;
      }
      o[10] = z.x;
      o[11] = z.y;
      rec_put<T>(base + (long)piv * rs, nl, o);
    }
#pragma unroll
    for (int i = 0; i < 5; i++) {
#pragma unroll
      for (int j = 0; j <= i; j++) W[WI(i, j)] = W[WI(i + 1, j + 1)];
      y[i] = y[i + 1];
    }
  }
  cp_async_wait<0>();
  __threadfence_block();  // the factors just stored are read back below
  // backward: x_k = z_k - sum_i l_{k+i,k} x_{k+i}
  C_t<T> xw[5];
#pragma unroll
  for (int i = 0; i < 5; i++) xw[i] = mk<T>(0, 0);
  for (int p = 0; p < kRing - 1; p++) {
    if (m - 1 - p >= 0) issue(m - 1 - p);
    cp_async_commit();
  }
  for (int row = m - 1; row >= 0; row--) {
    if (row - (kRing - 1) >= 0) issue(row - (kRing - 1));
    cp_async_commit();
    cp_async_wait<kRing - 1>();
    T v[kRec];
    take(row, v);
    C_t<T> x = mk<T>(v[10], v[11]);
#pragma unroll
    for (int i = 0; i < 5; i++) x = cfms<T>(x, mk<T>(v[2 * i], v[2 * i + 1]), xw[i]);
#pragma unroll
    for (int i = 4; i > 0; i--) xw[i] = xw[i - 1];
    xw[0] = x;
    T last[kLanes<T>];
#pragma unroll
    for (int i = 0; i < kLanes<T>; i++) last[i] = v[kRec - kLanes<T> + i];
    last[kLanes<T> - 2] = x.x;
    last[kLanes<T> - 1] = x.y;
    base[(long)row * rs + (NP - 1) * nl] = pack16(last);
  }
  cp_async_wait<0>();
}

template <typename T, int D>
__global__ void __launch_bounds__(256) k_line_apply(LevelView<T> L, int pa, int pb,
                                                    const T* buf) {
  const int rhs = blockIdx.y;
  if (L.active && !L.active[rhs]) return;
  const LineGeom g = line_geom<D>(L.n, pa, pb);
  long l;
  int s;
  if (!line_item<D>(g, blockIdx.x * (long)blockDim.x + threadIdx.x, l, s)) return;
  const unsigned lq = (unsigned)l / (unsigned)g.la;
  const int ta = g.fa + 2 * (int)((unsigned)l - lq * (unsigned)g.la), tb = g.fb + 2 * (int)lq;
  using V = typename Vec16<T>::V;
  C_t<T>* u = L.u + (long)rhs * 3 * L.S;
  const V* base = reinterpret_cast<const V*>(buf) + (long)rhs * g.m * kPlanes<T> * g.nl + l;
  const int r0 = 5 * (s - 1);
  // every load before the first store
  auto x = [&](int row) { return rec_get_x<T>(base + (long)row * kPlanes<T> * g.nl, g.nl); };
  const long sl[5] = {line_slot<D, 0>(L.n, L.S, ta, tb, s), line_slot<D, 1>(L.n, L.S, ta, tb, s),
                      line_slot<D, 2>(L.n, L.S, ta, tb, s), line_slot<D, 3>(L.n, L.S, ta, tb, s),
                      line_slot<D, 4>(L.n, L.S, ta, tb, s)};
  const int nr = s < g.nd ? 5 : 1;
  C_t<T> v[5];
#pragma unroll
  for (int t = 0; t < 5; t++)
    if (t < nr) v[t] = cadd<T>(u[sl[t]], x(r0 + t));
#pragma unroll
  for (int t = 0; t < 5; t++)
    if (t < nr) u[sl[t]] = v[t];
}

template <typename T, int D>
static void line_sweep_d(const LevelView<T>& L, int color, T* buf, cudaStream_t st) {
  const int pa = color & 1, pb = (color >> 1) & 1;
  const long nl = line_count(L.n, D, color);
  if (nl == 0) return;
  const long items = nl * L.n[D];
  const int m = 5 * L.n[D] - 4;
  dim3 g1((unsigned)((items + 255) / 256), L.nrhs);
  // launched the ordinary way: blocks of the solve that start beside the
  // assembly's last ones find its shared-memory carveout, too small for more
  // than a few of them an SM (complex128, four shots at 128^3, three cycles:
  // 1.06 s with dependent launches, 0.79 s so)
  if (D == 0) {
    dim3 g5((unsigned)((5 * items + 255) / 256), L.nrhs);
    k_line_assemble_rows<T, D><<<g5, 256, 0, st>>>(L, pa, pb, buf);
  } else {
    k_line_assemble<T, D><<<g1, 256, 0, st>>>(L, pa, pb, buf);
  }
  dim3 g2((unsigned)((nl + kSolveThreads - 1) / kSolveThreads), L.nrhs);
  k_line_solve<T><<<g2, kSolveThreads, 0, st>>>(L.active, nl, m, buf);
  k_line_apply<T, D><<<g1, 256, 0, st>>>(L, pa, pb, buf);
}
// the line solve keeps a cp.async ring in shared memory: ask for the
// largest shared-memory carveout so 12 blocks fit on an SM
void init_line_kernels() {
  static DeviceOnce once;
  once_on_device(once, [] {
    cudaFuncSetAttribute(k_line_solve<float>, cudaFuncAttributePreferredSharedMemoryCarveout,
                         cudaSharedmemCarveoutMaxShared);
    cudaFuncSetAttribute(k_line_solve<double>, cudaFuncAttributePreferredSharedMemoryCarveout,
                         cudaSharedmemCarveoutMaxShared);
    init_stored_line_kernels();
  });
}


// scratch: m * lines * kRec values of T (see line_scratch_elems)
template <typename T>
void launch_line_sweep(const LevelView<T>& L, int d, int color, C_t<T>* scratch, cudaStream_t st) {
  T* buf = reinterpret_cast<T*>(scratch);
  if (d == 0) line_sweep_d<T, 0>(L, color, buf, st);
  else if (d == 1) line_sweep_d<T, 1>(L, color, buf, st);
  else line_sweep_d<T, 2>(L, color, buf, st);
}

// ------------------------------------------------------------ transfers
template <typename T>
struct Xfer {
  int nf[3], nc[3], sc[3];
};

// the transfer weights of a level (LevelView::xw), once per set-up: the
// arithmetic the transfers used to repeat in every thread
template <typename T>
__global__ void __launch_bounds__(256) k_xfer_weights(LevelView<T> F, LevelView<T> Cc, int sc0,
                                                      int sc1, int sc2, int nop, T* __restrict__ out) {
  const int g1 = F.gmax1;
  const long id = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (id >= (long)nop * 3 * g1) return;
  const int o = (int)(id / (3 * g1));
  const int e = (int)((id / g1) % 3);
  const int f = (int)(id % g1);
  const int sc = e == 0 ? sc0 : e == 1 ? sc1 : sc2;
  const int c = sc == 2 ? f / 2 : f;
  T w = 0;
  if (f <= F.n[e] && c < Cc.n[e]) {
    const T* xf = F.geo + (long)o * F.gstride + (long)e * g1;
    const T* xc = Cc.geo + (long)o * Cc.gstride + (long)e * g1;
    w = (xf[f] - xc[c]) / (xc[c + 1] - xc[c]);
  }
  out[id] = w;
}

template <typename T>
void launch_xfer_weights(const LevelView<T>& F, const LevelView<T>& Cc, const int sc[3], int nop,
                         T* out, cudaStream_t st) {
  const long n = (long)nop * 3 * F.gmax1;
  k_xfer_weights<T><<<(unsigned)((n + 255) / 256), 256, 0, st>>>(F, Cc, sc[0], sc[1], sc[2], nop, out);
}
template void launch_xfer_weights<float>(const LevelView<float>&, const LevelView<float>&,
                                         const int*, int, float*, cudaStream_t);
template void launch_xfer_weights<double>(const LevelView<double>&, const LevelView<double>&,
                                          const int*, int, double*, cudaStream_t);

// The fine nodes along axis e restricted to coarse node Ce, in the order of
// src/gmg.c:1510-1573: those whose coarse interval starts at Ce (weight
// 1 - wr), then those whose interval ends at Ce (weight wr).  Fine nodes that
// are coarse nodes have wr exactly 0 (the coordinates are sub-sampled), so a
// coarsened axis (SC = 2) takes 2 Ce, 2 Ce + 1 and 2 Ce - 1 and the other one
// Ce alone; a slot is used when its node is an interior fine node.
template <int SC, typename T>
__device__ __forceinline__ void xfer_slots(int Ce, int nfe, int nce, const T* __restrict__ wr,
                                           int (&idx)[3], T (&w)[3], bool (&ok)[3]) {
  const int F = SC * Ce;
  idx[0] = F;
  idx[1] = F + 1;
  idx[2] = F - 1;
  ok[0] = Ce < nce && F >= 1 && F < nfe;
  ok[1] = SC == 2 && Ce < nce && F + 1 >= 1 && F + 1 < nfe;
  ok[2] = SC == 2 && Ce >= 1 && F - 1 >= 1 && F - 1 < nfe;
  w[0] = ok[0] ? T(1) - ldro(wr + F) : T(0);
  w[1] = ok[1] ? T(1) - ldro(wr + F + 1) : T(0);
  w[2] = ok[2] ? ldro(wr + F - 1) : T(0);
}

template <typename T, int C, int SC0, int SC1, int SC2>
__device__ __forceinline__ C_t<T> restrict_comp(const LevelView<T>& F, const LevelView<T>& Cc,
                                                const int Cn[3], const C_t<T>* rf,
                                                const T* __restrict__ xw) {
  constexpr int p = Cyc<C>::p, q = Cyc<C>::q;
  constexpr int t1 = p < q ? p : q, t2 = p < q ? q : p;
  constexpr int sc[3] = {SC0, SC1, SC2};
  constexpr int n1 = sc[t1] == 2 ? 3 : 1, n2 = sc[t2] == 2 ? 3 : 1;
  int i1[3], i2[3];
  T w1[3], w2[3];
  bool o1[3], o2[3];
  xfer_slots<sc[t1]>(Cn[t1], F.n[t1], Cc.n[t1], xw + t1 * F.gmax1, i1, w1, o1);
  xfer_slots<sc[t2]>(Cn[t2], F.n[t2], Cc.n[t2], xw + t2 * F.gmax1, i2, w2, o2);
  const int fs[3] = {1, F.n[0] + 1, (F.n[0] + 1) * (F.n[1] + 1)};
  // every load before the first use, none behind a branch
  C_t<T> v[sc[C]][n1][n2];
#pragma unroll
  for (int t = 0; t < sc[C]; t++) {
    const int fc = sc[C] * Cn[C] + t;
    const C_t<T>* base = rf + (C * (int)F.S + fc * fs[C]);
#pragma unroll
    for (int a = 0; a < n1; a++)
#pragma unroll
      for (int b = 0; b < n2; b++)
        v[t][a][b] = fc < F.n[C] && o1[a] && o2[b] ? base[i1[a] * fs[t1] + i2[b] * fs[t2]]
                                                   : mk<T>(0, 0);
  }
  T ar = 0, ai = 0;
#pragma unroll
  for (int t = 0; t < sc[C]; t++)
#pragma unroll
    for (int a = 0; a < n1; a++)
#pragma unroll
      for (int b = 0; b < n2; b++) {
        const T w = w1[a] * w2[b];
        ar += w * v[t][a][b].x;
        ai += w * v[t][a][b].y;
      }
  return mk<T>(ar, ai);
}

// one component per thread (blockIdx.z); SC: the axes' factors, known to the
// compiler, so that a thread's up to 18 loads are in flight together (level 0
// of 25 RHS at 128^3: 653 -> 350 us, 5.5 TB/s; the loads used to wait behind a
// branch each)
template <typename T, int SC0, int SC1, int SC2>
__global__ void __launch_bounds__(256) k_restrict(LevelView<T> F, LevelView<T> Cc) {
  dep_wait();
  dep_next();
  const int rhs = blockIdx.y;
  if (Cc.active && !Cc.active[rhs]) return;
  const long s = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (s >= Cc.S) return;
  int Cn[3];
  slot_nodes(s, Cc, Cn);
  const C_t<T>* rf = F.r + (long)rhs * 3 * F.S;
  const int c = blockIdx.z;
  C_t<T>* fc = Cc.f + ((long)rhs * 3 + c) * Cc.S;
  C_t<T>* uc = Cc.u + ((long)rhs * 3 + c) * Cc.S;
  const T* xw = F.xw + (long)op_of(F, rhs) * 3 * F.gmax1;
  C_t<T> v;
  switch (c) {
    case 0: v = restrict_comp<T, 0, SC0, SC1, SC2>(F, Cc, Cn, rf, xw); break;
    case 1: v = restrict_comp<T, 1, SC0, SC1, SC2>(F, Cc, Cn, rf, xw); break;
    default: v = restrict_comp<T, 2, SC0, SC1, SC2>(F, Cc, Cn, rf, xw); break;
  }
  fc[s] = v;
  uc[s] = mk<T>(0, 0);
}

template <typename T>
void launch_restrict(const LevelView<T>& F, const LevelView<T>& Cc, const int sc[3], cudaStream_t st) {
  dim3 grid((unsigned)((Cc.S + 255) / 256), Cc.nrhs, 3);
  auto go = [&](auto k) { launch_dep(k, grid, 256, 0, st, F, Cc); };
  switch ((sc[0] == 2) + 2 * (sc[1] == 2) + 4 * (sc[2] == 2)) {
    case 0: go(k_restrict<T, 1, 1, 1>); break;
    case 1: go(k_restrict<T, 2, 1, 1>); break;
    case 2: go(k_restrict<T, 1, 2, 1>); break;
    case 3: go(k_restrict<T, 2, 2, 1>); break;
    case 4: go(k_restrict<T, 1, 1, 2>); break;
    case 5: go(k_restrict<T, 2, 1, 2>); break;
    case 6: go(k_restrict<T, 1, 2, 2>); break;
    default: go(k_restrict<T, 2, 2, 2>); break;
  }
}

template <typename T, int C>
__device__ __forceinline__ void prolong_comp(const LevelView<T>& F, const LevelView<T>& Cc,
                                             const int sc[3], const int P[3], C_t<T>* uf,
                                             const C_t<T>* __restrict__ uc,
                                             const T* __restrict__ xw, long s) {
  constexpr int p = Cyc<C>::p, q = Cyc<C>::q;
  constexpr int t1 = p < q ? p : q, t2 = p < q ? q : p;
  if (!(P[C] < F.n[C] && P[t1] >= 1 && P[t1] < F.n[t1] && P[t2] >= 1 && P[t2] < F.n[t2])) return;
  int Cn[3];
#pragma unroll
  for (int e = 0; e < 3; e++) Cn[e] = sc[e] == 2 ? P[e] / 2 : P[e];
  const T wr1 = ldro(xw + t1 * F.gmax1 + P[t1]);
  const T wr2 = ldro(xw + t2 * F.gmax1 + P[t2]);
  const T wl1 = T(1) - wr1, wl2 = T(1) - wr2;
  // 32-bit offsets: the four coarse neighbours differ by the strides of t1, t2
  const int cs[3] = {1, Cc.n[0] + 1, (Cc.n[0] + 1) * (Cc.n[1] + 1)};
  const int q00 = C * (int)Cc.S + slot_id32(Cc.n, Cn[0], Cn[1], Cn[2]);
  const C_t<T> u00 = uc[q00];
  const C_t<T> u01 = uc[q00 + cs[t2]];
  const C_t<T> u10 = uc[q00 + cs[t1]];
  const C_t<T> u11 = uc[q00 + cs[t1] + cs[t2]];
  C_t<T> v = uf[C * (int)F.S + (int)s];
  v.x += wl1 * (wl2 * u00.x + wr2 * u01.x) + wr1 * (wl2 * u10.x + wr2 * u11.x);
  v.y += wl1 * (wl2 * u00.y + wr2 * u01.y) + wr1 * (wl2 * u10.y + wr2 * u11.y);
  uf[C * (int)F.S + (int)s] = v;
}

template <typename T>
__global__ void __launch_bounds__(256) k_prolong(LevelView<T> F, LevelView<T> Cc, int sc0, int sc1,
                                                 int sc2) {
  dep_wait();
  dep_next();
  const int rhs = blockIdx.y;
  if (F.active && !F.active[rhs]) return;
  const long s = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (s >= F.S) return;
  const int sc[3] = {sc0, sc1, sc2};
  int P[3];
  slot_nodes(s, F, P);
  C_t<T>* uf = F.u + (long)rhs * 3 * F.S;
  const C_t<T>* uc = Cc.u + (long)rhs * 3 * Cc.S;
  const T* xw = F.xw + (long)op_of(F, rhs) * 3 * F.gmax1;
  switch (blockIdx.z) {  // one component per thread
    case 0: prolong_comp<T, 0>(F, Cc, sc, P, uf, uc, xw, s); break;
    case 1: prolong_comp<T, 1>(F, Cc, sc, P, uf, uc, xw, s); break;
    default: prolong_comp<T, 2>(F, Cc, sc, P, uf, uc, xw, s); break;
  }
}

// complex64: a thread per slot and its three components, whose fifteen loads
// are in flight together (level 0 of 25 RHS at 128^3: 765 -> 530 us, 5.5 TB/s,
// against a component a thread)
__global__ void __launch_bounds__(256) k_prolong_nodes(LevelView<float> F, LevelView<float> Cc,
                                                       int sc0, int sc1, int sc2) {
  dep_wait();
  dep_next();
  const int rhs = blockIdx.y;
  if (F.active && !F.active[rhs]) return;
  const long s = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (s >= F.S) return;
  int P[3];
  slot_nodes(s, F, P);
  const bool in0 = P[0] >= 1 && P[0] < F.n[0], in1 = P[1] >= 1 && P[1] < F.n[1],
             in2 = P[2] >= 1 && P[2] < F.n[2];
  const bool unk[3] = {P[0] < F.n[0] && in1 && in2, P[1] < F.n[1] && in2 && in0,
                       P[2] < F.n[2] && in0 && in1};
  float2* uf = F.u + (long)rhs * 3 * F.S + s;
  const int cs[3] = {1, Cc.n[0] + 1, (Cc.n[0] + 1) * (Cc.n[1] + 1)};
  const float2* uc = Cc.u + (long)rhs * 3 * Cc.S +
                     slot_id32(Cc.n, sc0 == 2 ? P[0] / 2 : P[0], sc1 == 2 ? P[1] / 2 : P[1],
                               sc2 == 2 ? P[2] / 2 : P[2]);
  const float* xw = F.xw + (long)op_of(F, rhs) * 3 * F.gmax1;
  float wr[3];
#pragma unroll
  for (int e = 0; e < 3; e++) wr[e] = ldro(xw + e * F.gmax1 + P[e]);
  const float2 zero = make_float2(0.f, 0.f);
  float2 u0[3], u00[3], u01[3], u10[3], u11[3];
#pragma unroll
  for (int c = 0; c < 3; c++) {
    const int t1 = c == 0 ? 1 : 0, t2 = c == 2 ? 1 : 2;
    const float2* q = uc + (long)c * Cc.S;
    u0[c] = unk[c] ? uf[(long)c * F.S] : zero;
    u00[c] = unk[c] ? q[0] : zero;
    u01[c] = unk[c] ? q[cs[t2]] : zero;
    u10[c] = unk[c] ? q[cs[t1]] : zero;
    u11[c] = unk[c] ? q[cs[t1] + cs[t2]] : zero;
  }
#pragma unroll
  for (int c = 0; c < 3; c++) {
    if (!unk[c]) continue;
    const int t1 = c == 0 ? 1 : 0, t2 = c == 2 ? 1 : 2;
    const float wr1 = wr[t1], wr2 = wr[t2], wl1 = 1.f - wr1, wl2 = 1.f - wr2;
    float2 v = u0[c];
    v.x += wl1 * (wl2 * u00[c].x + wr2 * u01[c].x) + wr1 * (wl2 * u10[c].x + wr2 * u11[c].x);
    v.y += wl1 * (wl2 * u00[c].y + wr2 * u01[c].y) + wr1 * (wl2 * u10[c].y + wr2 * u11[c].y);
    uf[(long)c * F.S] = v;
  }
}

template <typename T>
void launch_prolong(const LevelView<T>& F, const LevelView<T>& Cc, const int sc[3], cudaStream_t st) {
  if constexpr (sizeof(T) == 4) {
    launch_dep(k_prolong_nodes, dim3((unsigned)((F.S + 255) / 256), F.nrhs), dim3(256), 0, st, F, Cc,
               sc[0], sc[1], sc[2]);
  } else {
    dim3 grid((unsigned)((F.S + 255) / 256), F.nrhs, 3);
    launch_dep(k_prolong<T>, grid, 256, 0, st, F, Cc, sc[0], sc[1], sc[2]);
  }
}

// ------------------------------------------------------------ coarsening
template <typename T>
__global__ void __launch_bounds__(256) k_coarsen(const T* __restrict__ fine, int nf0, int nf1, int nf2,
                                                 T* __restrict__ coarse, int sc0, int sc1, int sc2) {
  const int nc0 = nf0 / sc0, nc1 = nf1 / sc1, nc2 = nf2 / sc2;
  const long ncc = (long)nc0 * nc1 * nc2, nfc = (long)nf0 * nf1 * nf2;
  const long id = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (id >= ncc) return;
  const long arr = blockIdx.y;  // rhs*4 + which
  // 32-bit decode (a level has fewer than 2^31 cells)
  const unsigned t = (unsigned)id / (unsigned)nc0;
  const int i = (int)((unsigned)id - t * (unsigned)nc0);
  const int j = (int)(t % (unsigned)nc1), k = (int)(t / (unsigned)nc1);
  const int i0 = sc0 == 2 ? 2 * i : i, i1 = sc0 == 2 ? 2 * i + 1 : i;
  const int j0 = sc1 == 2 ? 2 * j : j, j1 = sc1 == 2 ? 2 * j + 1 : j;
  const int k0 = sc2 == 2 ? 2 * k : k, k1 = sc2 == 2 ? 2 * k + 1 : k;
  const T* F = fine + arr * nfc;
#define CF(a, b, c) F[(a) + (long)nf0 * ((b) + (long)nf1 * (c))]
  const T v = CF(i0, j0, k0) + CF(i1, j0, k0) + CF(i0, j1, k0) + CF(i1, j1, k0) + CF(i0, j0, k1) +
              CF(i1, j0, k1) + CF(i0, j1, k1) + CF(i1, j1, k1);
#undef CF
  const int repeat = 8 / (sc0 * sc1 * sc2);
  coarse[arr * ncc + id] = v / (T)repeat;
}

template <typename T>
void launch_coarsen_cells(const T* fine, const int nf[3], T* coarse, const int sc[3], int nrhs,
                          cudaStream_t st) {
  const long ncc = (long)(nf[0] / sc[0]) * (nf[1] / sc[1]) * (nf[2] / sc[2]);
  dim3 grid((unsigned)((ncc + 255) / 256), 4 * nrhs);
  k_coarsen<T><<<grid, 256, 0, st>>>(fine, nf[0], nf[1], nf[2], coarse, sc[0], sc[1], sc[2]);
}

template <typename T>
__global__ void k_zero(C_t<T>* p, long n) {
  dep_wait();
  dep_next();
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
    p[i] = mk<T>(0, 0);
}

template <typename T>
void launch_zero(C_t<T>* p, long n, cudaStream_t st) {
  long blocks = (n + 255) / 256;
  if (blocks > 4864) blocks = 4864;
  if (blocks < 1) blocks = 1;
  launch_dep(k_zero<T>, (unsigned)blocks, 256, 0, st, p, n);
}

// ------------------------------------------------------------ instantiations
#define EMMI_INST(T)                                                                               \
  template void launch_norm<T>(const C_t<T>*, long, int, const int*, double*, cudaStream_t);        \
  template void launch_line_sweep<T>(const LevelView<T>&, int, int, C_t<T>*, cudaStream_t);         \
  template void launch_restrict<T>(const LevelView<T>&, const LevelView<T>&, const int*,            \
                                   cudaStream_t);                                                   \
  template void launch_prolong<T>(const LevelView<T>&, const LevelView<T>&, const int*,             \
                                  cudaStream_t);                                                    \
  template void launch_coarsen_cells<T>(const T*, const int*, T*, const int*, int, cudaStream_t);   \
  template void launch_zero<T>(C_t<T>*, long, cudaStream_t);
EMMI_INST(float)
EMMI_INST(double)
template void launch_residual<float, float>(const LevelView<float>&, C_t<float>*, double*, cudaStream_t);
template void launch_residual<double, double>(const LevelView<double>&, C_t<double>*, double*, cudaStream_t);
template void launch_residual<double, float>(const LevelView<double>&, C_t<float>*, double*, cudaStream_t);

}  // namespace emmi
