// Line relaxation with stored factors, and the one-launch line sweep.
//
// A line's band matrix depends on the operator only, never on the iterate.
// The solvers therefore keep the LDL^T factors of every line and sweep with
// the residual of every row and a substitution.
//
// complex128 (records as k_line_solve writes them in place, planes
// [row][plane][line]: L(p+i, p) for i = 1..5 and 1/d_p): one thread
// substitutes along a line, the same arithmetic in the same order as
// k_line_solve, so the same result.
//
// complex64 eliminates a line from both ends.  With nd nodes along the line
// (nd even: a line is relaxed only along a direction the next level
// coarsens) its 5 nd - 4 rows are G = (nd - 2) / 2 groups of five from the
// top (E_d(j) and the four transverse edges of node j + 1), six middle rows
// (E_d(G), node G + 1, E_d(G + 1)) and G groups from the bottom, the mirror
// image of the top ones.  Both ends eliminate their groups towards the middle
// at the same time, the middle six rows take both Schur complements, and both
// ends substitute back outwards: the serial chain is half as long and twice
// as many threads share a line, with the same multipliers per row (five) and
// no fill.  Storage is by position: top rows and middle in row order, the
// bottom rows in the order of their elimination (last row first).
#include <cuda_fp16.h>

#include <algorithm>
#include <type_traits>

#include "emmi_line.cuh"
#include "emmi_node.cuh"

namespace emmi {

// ---------------------------------------------------------------- two-ended storage
// A level's lines of one colour in tiles of 1 << shift neighbouring lines:
// element (row, line) of a row buffer lies at
// ((line >> shift) * m + pos(row)) << shift | (line & (1 << shift) - 1).
struct LineTile {
  int shift;  // log2 of the lines per tile
  int mid;    // position of the first middle row, 5 G
  int m;      // rows of a line
  __host__ __device__ __forceinline__ int pos(int row) const {
    return row < mid + 6 ? row : mid + 6 + (m - 1 - row);
  }
};
inline LineTile line_tile(int nd, int tile) {
  LineTile t;
  t.shift = tile == 8 ? 3 : 5;
  t.mid = 5 * ((nd - 2) / 2);
  t.m = 5 * nd - 4;
  return t;
}
// where row `row` of line l goes in a right-hand side's row buffer, and the
// values of that buffer: two-ended tiles for complex64, [row][line] for
// complex128
template <typename T>
__device__ __forceinline__ long rb_index(const LineTile& t, long nl, long l, int row) {
  if constexpr (sizeof(T) == 4)
    return ((((l >> t.shift) * t.m + t.pos(row)) << t.shift) | (l & ((1 << t.shift) - 1)));
  else
    return (long)row * nl + l;
}
template <typename T>
__host__ __device__ __forceinline__ long rb_elems(const LineTile& t, long nl) {
  if constexpr (sizeof(T) == 4)
    return (((nl + (1 << t.shift) - 1) >> t.shift) * t.m) << t.shift;
  else
    return nl * t.m;
}

template <typename T, int D, int TT, int C, bool RO>
__device__ __forceinline__ C_t<T> row_residual(const LevelView<T>& L, const C_t<T>* u,
                                               const C_t<T>* f, const T* cells,
                                               const Geo<T>& G, T wmu, int ta, int tb, int s,
                                               const long ss[3]) {
  constexpr int A = (D == 0) ? 1 : 0, B = (D == 2) ? 1 : 2;
  int P[3];
  P[D] = (TT == 0) ? s - 1 : s;
  P[A] = ta - (TT == 1 ? 1 : 0);
  P[B] = tb - (TT == 3 ? 1 : 0);
  const int sl = P[0] + (L.n[0] + 1) * (P[1] + (L.n[1] + 1) * P[2]);  // 32-bit slot
  EdgeCoef<T> e;
  const C_t<T> au = apply_row<T, C, 0, RO>(L, u, cells, G, wmu, P, sl, ss, e);
  return csub<T>(f[C * (int)L.S + sl], au);
}

// the same from stored coefficients (coef64_elems per operator: planes
// [10][3][S], see emmi_kernels.cu), applied in edge_coef / apply_row's order:
// 30 FP64 instructions a row where recomputing the coefficients takes eight
// divisions of 13 besides (one RHS at 16^3 32 -> 18 us a launch, four at
// 64 x 56 x 48 60 -> 23)
template <int D, int TT, int C>
__device__ __forceinline__ double2 row_residual_coef(const LevelView<double>& L, const double2* u,
                                                     const double2* f,
                                                     const double* __restrict__ cf, double wmu,
                                                     int ta, int tb, int s, const long ss[3]) {
  constexpr int A = (D == 0) ? 1 : 0, B = (D == 2) ? 1 : 2;
  int P[3];
  P[D] = (TT == 0) ? s - 1 : s;
  P[A] = ta - (TT == 1 ? 1 : 0);
  P[B] = tb - (TT == 3 ? 1 : 0);
  const int S = (int)L.S;
  const int sl = P[0] + (L.n[0] + 1) * (P[1] + (L.n[1] + 1) * P[2]), o = C * S + sl;
  const long n3s = 3 * L.S;
  double k[10];
#pragma unroll
  for (int c = 0; c < 10; c++) k[c] = ldro(cf + c * n3s + o);
  const double c12[12] = {k[0], k[1], k[2], k[3], k[4], -k[4], -k[5], k[5],
                          k[6], -k[6], -k[7], k[7]};
  const double dre = k[8], dim = -wmu * k[9];
  const int s3[3] = {1, (int)ss[1], (int)ss[2]};
  const double2 uc = u[o];
  // the diagonal's product contracted as apply_row's is
  double ar = rfma(dre, uc.x, -rmul(dim, uc.y));
  double ai = rfma(dre, uc.y, rmul(dim, uc.x));
#pragma unroll
  for (int c = 0; c < 12; c++) {
    const double2 v = u[sl + nbr_delta32<C>(c, s3, S)];
    ar = rfma(c12[c], v.x, ar);
    ai = rfma(c12[c], v.y, ai);
  }
  const double2 r = f[o];
  return mk<double>(rsub(r.x, ar), rsub(r.y, ai));
}

// rb = residual of every row of one colour; y and z lines:
// a thread per (line, node) and its five rows; x lines: a thread per
// (row type, line, node), row type slowest
template <typename T, int D, bool CF, bool RO>
__global__ void __launch_bounds__(256) k_line_rhs(LevelView<T> L, int pa, int pb, LineDiv dv,
                                                  LineTile tl, C_t<T>* __restrict__ rb,
                                                  const double* __restrict__ coef) {
  if constexpr (!RO) {
    dep_wait();
    dep_next();
  }
  constexpr int A = (D == 0) ? 1 : 0, B = (D == 2) ? 1 : 2;
  const int rhs = blockIdx.y;
  if (L.active && !L.active[rhs]) return;
  const LineGeom g = line_geom<D>(L.n, pa, pb);
  unsigned id = blockIdx.x * blockDim.x + threadIdx.x;
  int rt = 0;
  if (D == 0) {
    rt = (int)fdiv(id, dv.rows);
    if (rt >= 5) return;
    id -= (unsigned)rt * dv.items;
  }
  long l;
  int s;
  if (!line_item_fd<D>(g, dv, id, l, s)) return;
  if (D == 0 && rt > 0 && s == g.nd) return;
  const unsigned lq = fdiv((unsigned)l, dv.la);
  const int ta = g.fa + 2 * (int)((unsigned)l - lq * (unsigned)g.la), tb = g.fb + 2 * (int)lq;
  const int n0 = L.n[0] + 1, n1 = L.n[1] + 1;
  const long ss[3] = {1, (long)n0, (long)n0 * n1};
  const C_t<T>* u = L.u + (long)rhs * 3 * L.S;
  const C_t<T>* f = L.f + (long)rhs * 3 * L.S;
  const T* cells = L.cells + (long)op_of(L, rhs) * 4 * L.ncell;
  const Geo<T> G{L.geo + (long)op_of(L, rhs) * L.gstride, L.gmax1};
  const T wmu = L.wmu[rhs];
  C_t<T>* out = rb + (long)rhs * rb_elems<T>(tl, g.nl);
  const int r0 = 5 * (s - 1);
  const double* cf = CF ? coef + (long)op_of(L, rhs) * 30 * L.S : nullptr;
  auto row = [&](auto tt, auto comp) {
    constexpr int TT = decltype(tt)::value, C = decltype(comp)::value;
    if constexpr (CF) return row_residual_coef<D, TT, C>(L, u, f, cf, wmu, ta, tb, s, ss);
    else return row_residual<T, D, TT, C, RO>(L, u, f, cells, G, wmu, ta, tb, s, ss);
  };
  auto put = [&](int row, C_t<T> v) { out[rb_index<T>(tl, g.nl, l, row)] = v; };
  if (D == 0) {
    switch (rt) {
      case 0: put(r0, row(std::integral_constant<int, 0>(), std::integral_constant<int, D>())); break;
      case 1: put(r0 + 1, row(std::integral_constant<int, 1>(), std::integral_constant<int, A>())); break;
      case 2: put(r0 + 2, row(std::integral_constant<int, 2>(), std::integral_constant<int, A>())); break;
      case 3: put(r0 + 3, row(std::integral_constant<int, 3>(), std::integral_constant<int, B>())); break;
      default: put(r0 + 4, row(std::integral_constant<int, 4>(), std::integral_constant<int, B>())); break;
    }
  } else {
    put(r0, row(std::integral_constant<int, 0>(), std::integral_constant<int, D>()));
    if (s < g.nd) {
      put(r0 + 1, row(std::integral_constant<int, 1>(), std::integral_constant<int, A>()));
      put(r0 + 2, row(std::integral_constant<int, 2>(), std::integral_constant<int, A>()));
      put(r0 + 3, row(std::integral_constant<int, 3>(), std::integral_constant<int, B>()));
      put(r0 + 4, row(std::integral_constant<int, 4>(), std::integral_constant<int, B>()));
    }
  }
}

// ---------------------------------------------------------------- row residuals by node
// The complex64 residuals of a colour's rows with the coefficients from the
// spacings (imu_vol): a thread takes a line's node s -- E_D of the edge below
// it and the node's four transverse edges -- and loads each of the 30 edge
// values, 20 conductivities and six spacings the five equations share once
// (row by row they are 65, 20 and 25), all of them before the first use.
// With hat sizes h = (d- + d+) / 2, the equation of an edge along C of size
// d_C between the directions X and Y reads (edge_coef with cell weight =
// volume)
//   sum over (X, Y): d_C h_Y [(E - E(+X)) / d_X+ + (E - E(-X)) / d_X-]
//                    + h_Y [E_X(+C) - E_X - E_X(+C, -X) + E_X(-X)]
//   - i wmu sbar E.
// y and z lines: a warp takes 32 lines at a node, a block NW nodes.  x lines:
// a warp takes 32 nodes of a line (neighbours in memory), a block NW lines,
// whose rows are staged in shared memory and stored line by line of a tile.
// Bound by DRAM: level 0 of 4 right-hand sides at 128^3, a colour of y lines,
// reads and writes 503 MB (u, f and sigma once) in 90 us, 5.6 TB/s; row by row
// the same bytes took 131 us, waiting for loads.  A sweep of 25 right-hand
// sides with it: x 7.57 -> 5.95, y 6.37 -> 5.39, z 5.90 -> 5.47 ms.
template <int D>
__device__ __forceinline__ void node_rows(const LevelView<float>& L, int rhs, int ta, int tb,
                                          int s, float2 (&r)[5]) {
  constexpr int A = (D == 0) ? 1 : 0, B = (D == 2) ? 1 : 2;
  const int op = op_of(L, rhs);
  const int ss[3] = {1, L.n[0] + 1, (L.n[0] + 1) * (L.n[1] + 1)};
  const int cs[3] = {1, L.n[0], L.n[0] * L.n[1]};
  const int sd = ss[D], sa = ss[A], sb = ss[B], cd = cs[D], ca = cs[A], cb = cs[B];
  const int S = (int)L.S;
  const int o = s * sd + ta * sa + tb * sb;  // the node's slot
  const float2* u = L.u + (long)rhs * 3 * S;
  const float2* f = L.f + (long)rhs * 3 * S;
  const float2 *ud = u + (D * S + o), *ua = u + (A * S + o), *ub = u + (B * S + o);
  const float2 *fd = f + (D * S + o), *fa = f + (A * S + o), *fb = f + (B * S + o);
  const float* cells = L.cells + (long)op * 4 * L.ncell;
  const int nc = (int)L.ncell, co = s * cd + ta * ca + tb * cb;
  const float *gd = cells + ((long)D * nc + co), *ga = cells + ((long)A * nc + co),
              *gb = cells + ((long)B * nc + co);
  const Geo<float> G{L.geo + (long)op * L.gstride, L.gmax1};
  const float wmu = L.wmu[rhs];
  const bool node = s < L.n[D];  // the last node carries its E_D row only
  // edges along D below (0) and above (1) the node, at the five transverse
  // positions; transverse edges - and + of the node
  const float2 d0 = ud[-sd], d0am = ud[-sd - sa], d0ap = ud[-sd + sa],
               d0bm = ud[-sd - sb], d0bp = ud[-sd + sb];
  const float2 am = ua[-sa], ap = ua[0], bm = ub[-sb], bp = ub[0];
  const float2 am_dm = ua[-sa - sd], ap_dm = ua[-sd], bm_dm = ub[-sb - sd],
               bp_dm = ub[-sd];
  const float sg0 = ldro(gd - cd - ca - cb), sg1 = ldro(gd - cd - ca), sg2 = ldro(gd - cd - cb),
              sg3 = ldro(gd - cd);
  const float2 f0 = fd[-sd];
  const float D0 = ldro(G.ds(D) + s - 1);
  const float A0 = ldro(G.ds(A) + ta - 1), A1 = ldro(G.ds(A) + ta);
  const float B0 = ldro(G.ds(B) + tb - 1), B1 = ldro(G.ds(B) + tb);
  const float2 zero = make_float2(0.f, 0.f);
  float2 d1 = zero, d1am = zero, d1ap = zero, d1bm = zero, d1bp = zero;
  float2 am_dp = zero, ap_dp = zero, bm_dp = zero, bp_dp = zero;
  float2 am_bm = zero, am_bp = zero, ap_bm = zero, ap_bp = zero;
  float2 bm_am = zero, bm_ap = zero, bp_am = zero, bp_ap = zero;
  float2 f1 = zero, f2 = zero, f3 = zero, f4 = zero;
  float sa0 = 0.f, sa1 = 0.f, sb0 = 0.f, sb1 = 0.f, D1 = 1.f;
  if (node) {
    d1 = ud[0];
    d1am = ud[-sa];
    d1ap = ud[sa];
    d1bm = ud[-sb];
    d1bp = ud[sb];
    am_dp = ua[-sa + sd];
    ap_dp = ua[sd];
    bm_dp = ub[-sb + sd];
    bp_dp = ub[sd];
    am_bm = ua[-sa - sb];
    am_bp = ua[-sa + sb];
    ap_bm = ua[-sb];
    ap_bp = ua[sb];
    bm_am = ub[-sb - sa];
    bm_ap = ub[-sb + sa];
    bp_am = ub[-sa];
    bp_ap = ub[sa];
    f1 = fa[-sa];
    f2 = fa[0];
    f3 = fb[-sb];
    f4 = fb[0];
    // conductivities around the four transverse edges
    sa0 = ((ldro(ga - ca - cd - cb) + ldro(ga - ca - cd)) + ldro(ga - ca - cb)) + ldro(ga - ca);
    sa1 = ((ldro(ga - cd - cb) + ldro(ga - cd)) + ldro(ga - cb)) + ldro(ga);
    sb0 = ((ldro(gb - cb - cd - ca) + ldro(gb - cb - cd)) + ldro(gb - cb - ca)) + ldro(gb - cb);
    sb1 = ((ldro(gb - cd - ca) + ldro(gb - cd)) + ldro(gb - ca)) + ldro(gb);
    D1 = ldro(G.ds(D) + s);
  }
  const float rD0 = qdiv(1.f, D0), rD1 = qdiv(1.f, D1), rA0 = qdiv(1.f, A0),
              rA1 = qdiv(1.f, A1), rB0 = qdiv(1.f, B0), rB1 = qdiv(1.f, B1);
  const float hd = 0.5f * (D0 + D1), ha = 0.5f * (A0 + A1), hb = 0.5f * (B0 + B1);
  const float qw = 0.25f * wmu;
  {
    float2 c = edge_pair(zero, d0, d0ap, d0am, D0 * hb, rA1, rA0, hb, ap, ap_dm, am, am_dm);
    c = edge_pair(c, d0, d0bp, d0bm, D0 * ha, rB1, rB0, ha, bp, bp_dm, bm, bm_dm);
    r[0] = edge_done(f0, c, d0, qw * (((sg0 + sg1) + sg2) + sg3));
  }
  if (node) {
    float2 c = edge_pair(zero, am, am_dp, am_dm, A0 * hb, rD1, rD0, hb, d1, d1am, d0, d0am);
    c = edge_pair(c, am, am_bp, am_bm, A0 * hd, rB1, rB0, hd, bp, bp_am, bm, bm_am);
    r[1] = edge_done(f1, c, am, qw * sa0);
    c = edge_pair(zero, ap, ap_dp, ap_dm, A1 * hb, rD1, rD0, hb, d1ap, d1, d0ap, d0);
    c = edge_pair(c, ap, ap_bp, ap_bm, A1 * hd, rB1, rB0, hd, bp_ap, bp, bm_ap, bm);
    r[2] = edge_done(f2, c, ap, qw * sa1);
    c = edge_pair(zero, bm, bm_dp, bm_dm, B0 * ha, rD1, rD0, ha, d1, d1bm, d0, d0bm);
    c = edge_pair(c, bm, bm_ap, bm_am, B0 * hd, rA1, rA0, hd, ap, ap_bm, am, am_bm);
    r[3] = edge_done(f3, c, bm, qw * sb0);
    c = edge_pair(zero, bp, bp_dp, bp_dm, B1 * ha, rD1, rD0, ha, d1bp, d1, d0bp, d0);
    c = edge_pair(c, bp, bp_ap, bp_am, B1 * hd, rA1, rA0, hd, ap_bp, ap, am_bp, am);
    r[4] = edge_done(f4, c, bp, qw * sb1);
  }
}

template <int D, int NW>
__global__ void __launch_bounds__(32 * NW, 16 / NW) k_line_rows(LevelView<float> L, int pa, int pb,
                                                       LineDiv dv, LineTile tl, int nodes,
                                                       int lines, float2* __restrict__ rb) {
  dep_wait();
  dep_next();
  const int rhs = blockIdx.y;
  if (L.active && !L.active[rhs]) return;
  const LineGeom g = line_geom<D>(L.n, pa, pb);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  // blocks along the nodes (y lines) or the lines (z and x) first: planes of z
  // are swept one after the other
  const int bn = D == 1 ? blockIdx.x % nodes : blockIdx.x / lines;
  const int bl = D == 1 ? blockIdx.x / nodes : blockIdx.x % lines;
  const int s = D == 0 ? 1 + bn * 32 + lane : 1 + bn * NW + w;
  const int l = D == 0 ? bl * NW + w : bl * 32 + lane;
  const bool live = l < (int)g.nl && s <= g.nd;
  if (D != 0 && !live) return;
  float2 r[5];
#pragma unroll
  for (int t = 0; t < 5; t++) r[t] = make_float2(0.f, 0.f);
  if (live) {
    const unsigned lq = fdiv((unsigned)l, dv.la);
    const int ta = g.fa + 2 * (l - (int)lq * g.la), tb = g.fb + 2 * (int)lq;
    node_rows<D>(L, rhs, ta, tb, s, r);
  }
  const int shift = tl.shift, mask = (1 << shift) - 1;
  float2* out = rb + (long)rhs * rb_elems<float>(tl, g.nl);
  const int r0 = 5 * (s - 1);
  if constexpr (D != 0) {
    float2* q = out + ((long)(l >> shift) * tl.m << shift) + (l & mask);
#pragma unroll
    for (int t = 0; t < 5; t++)
      if (r0 + t < tl.m) q[(long)tl.pos(r0 + t) << shift] = r[t];
  } else {
    constexpr int kPitch = 5 * 32 + 1;
    __shared__ float2 st[NW * kPitch];
#pragma unroll
    for (int t = 0; t < 5; t++) st[w * kPitch + 5 * lane + t] = r[t];
    __syncthreads();
    for (int e = threadIdx.x; e < 160 * NW; e += 32 * NW) {
      const int row = 160 * bn + e / NW, ll = bl * NW + e % NW;
      if (row < tl.m && ll < (int)g.nl)
        out[(((long)(ll >> shift) * tl.m + tl.pos(row)) << shift) | (ll & mask)] =
            st[(e % NW) * kPitch + e / NW];
    }
  }
}

// band entries (lower, real) and diagonal of row type TT of node s: the
// band part of assemble_row's record; MIR: the entries to the rows after it
// (band[5 - i] to row + i; the operator is bitwise symmetric), what the row
// brings to an elimination from the line's other end
template <typename T, int D, int TT, int C, bool MIR = false>
__device__ __forceinline__ void band_row(const LevelView<T>& L, const T* cells, const Geo<T>& G,
                                         T wmu, int ta, int tb, int s, int row, T (&band)[5],
                                         C_t<T>& diag) {
  constexpr int A = (D == 0) ? 1 : 0, B = (D == 2) ? 1 : 2;
  int P[3];
  P[D] = (TT == 0) ? s - 1 : s;
  P[A] = ta - (TT == 1 ? 1 : 0);
  P[B] = tb - (TT == 3 ? 1 : 0);
  EdgeCoef<T> e;
  edge_coef<T, C>(L.n, P, cells + (long)C * L.ncell, cells + 3 * L.ncell, G, wmu, e, L.imu_vol);
#pragma unroll
  for (int j = 0; j < 5; j++) band[j] = 0;
#define LINE_ENTRY(K)                                                         \
  {                                                                           \
    constexpr int off = line_off(D, TT, K);                                   \
    if constexpr (!MIR && off < 0) {                                          \
      if (row + off >= 0) band[5 + off] = e.c[K];                             \
    }                                                                         \
    if constexpr (MIR && off > 0 && off < 127) {                              \
      if (row + off < 5 * L.n[D] - 4) band[5 - off] = e.c[K];                 \
    }                                                                         \
  }
  LINE_ENTRY(0) LINE_ENTRY(1) LINE_ENTRY(2) LINE_ENTRY(3) LINE_ENTRY(4) LINE_ENTRY(5)
  LINE_ENTRY(6) LINE_ENTRY(7) LINE_ENTRY(8) LINE_ENTRY(9) LINE_ENTRY(10) LINE_ENTRY(11)
#undef LINE_ENTRY
  diag = mk<T>(e.dre, e.dim);
}

// ---------------------------------------------------------------- two-ended factors
// A group of five rows in a tile of TW lines, as global and shared memory hold
// it: [row][TW] multipliers (fp16: L1..L4 in 16 bytes, then a plane of L5 in
// 4; fp32: planes of 16, 16 and 8 bytes), then [row][TW] 1/d in fp32.  The
// middle group has six rows.  Multiplier i of a row couples it to the i-th
// row eliminated after it.
__device__ __forceinline__ uint32_t h2u(__half2 h) { return *reinterpret_cast<uint32_t*>(&h); }
__device__ __forceinline__ float2 u2f2(uint32_t u) {
  return __half22float2(*reinterpret_cast<__half2*>(&u));
}
template <int FMT> constexpr int kFacL = FMT == kFacF16 ? 20 : 40;  // bytes of a row's multipliers
template <int FMT> constexpr int kFacRow = kFacL<FMT> + 8;          // and its 1/d

// multipliers of row t of the group at base (lane of TW lines)
template <int FMT>
__device__ __forceinline__ void fac_get(const unsigned char* base, int TW, int t, int lane,
                                        float2 (&v)[5]) {
  const unsigned char* r = base + t * kFacL<FMT> * TW;
  if constexpr (FMT == kFacF16) {
    const uint4 a = *reinterpret_cast<const uint4*>(r + lane * 16);
    const uint32_t b = *reinterpret_cast<const uint32_t*>(r + 16 * TW + lane * 4);
    v[0] = u2f2(a.x);
    v[1] = u2f2(a.y);
    v[2] = u2f2(a.z);
    v[3] = u2f2(a.w);
    v[4] = u2f2(b);
  } else {
    const float4 a = *reinterpret_cast<const float4*>(r + lane * 16);
    const float4 b = *reinterpret_cast<const float4*>(r + 16 * TW + lane * 16);
    v[0] = make_float2(a.x, a.y);
    v[1] = make_float2(a.z, a.w);
    v[2] = make_float2(b.x, b.y);
    v[3] = make_float2(b.z, b.w);
    v[4] = *reinterpret_cast<const float2*>(r + 32 * TW + lane * 8);
  }
}
template <int FMT>
__device__ __forceinline__ void fac_put(unsigned char* base, int TW, int rows, int t, int lane,
                                        const float2 (&l)[6], float2 id, bool& over) {
  unsigned char* r = base + t * kFacL<FMT> * TW;
  if constexpr (FMT == kFacF16) {
    __half2 h[5];
#pragma unroll
    for (int i = 1; i < 6; i++) {
      over |= !(fabsf(l[i].x) <= 65504.f && fabsf(l[i].y) <= 65504.f);
      h[i - 1] = __floats2half2_rn(l[i].x, l[i].y);
    }
    *reinterpret_cast<uint4*>(r + lane * 16) = make_uint4(h2u(h[0]), h2u(h[1]), h2u(h[2]), h2u(h[3]));
    *reinterpret_cast<uint32_t*>(r + 16 * TW + lane * 4) = h2u(h[4]);
  } else {
    *reinterpret_cast<float4*>(r + lane * 16) = make_float4(l[1].x, l[1].y, l[2].x, l[2].y);
    *reinterpret_cast<float4*>(r + 16 * TW + lane * 16) = make_float4(l[3].x, l[3].y, l[4].x, l[4].y);
    *reinterpret_cast<float2*>(r + 32 * TW + lane * 8) = l[5];
  }
  *reinterpret_cast<float2*>(base + rows * kFacL<FMT> * TW + (t * TW + lane) * 8) = id;
}

// one step of a streaming LDL^T over a 6 x 6 window (k_line_solve's order):
// eliminates W[0] against the rows that follow, returns 1/d, the multipliers
// in l[1..5], and moves the window on
__device__ __forceinline__ float2 window_step(float2 (&W)[21], float2 (&l)[6]) {
  const float2 id = crcp<float>(W[0]);
#pragma unroll
  for (int i = 1; i < 6; i++) l[i] = cmul<float>(W[WI(i, 0)], id);
#pragma unroll
  for (int i = 1; i < 6; i++) {
#pragma unroll
    for (int j = 1; j <= i; j++) W[WI(i, j)] = cfms<float>(W[WI(i, j)], l[i], W[WI(j, 0)]);
  }
#pragma unroll
  for (int i = 0; i < 5; i++) {
#pragma unroll
    for (int j = 0; j <= i; j++) W[WI(i, j)] = W[WI(i + 1, j + 1)];
  }
  return id;
}

// The elimination of one end's G groups and the arrival of the five middle
// rows next to it, shared by the factor kernel and the one-launch sweep.
// row(tt, s, k, w, r): entries w (five to the rows before it, the diagonal)
// and residual r of row type tt of node s; k is the row's place in its group,
// or k - 6 for the middle rows, of which the mirrored end keeps only the
// entries to its own rows.  piv(j, k): the pivot of group j, row k, is in
// W[0], the row that arrived in W[WI(5, .)], its residual in y5.  A node's
// five rows are assembled together, so that it waits on memory once.
// Leaves the middle rows' window (A's entries and this end's Schur complement
// for the top, the complement alone for the mirrored end).
template <bool MIR, typename RowF, typename PivF>
__device__ __forceinline__ void eliminate_end(int G, int nd, float2 (&W)[21], float2& y5,
                                              RowF&& row, PivF&& piv) {
  using I0 = std::integral_constant<int, 0>;
  using I1 = std::integral_constant<int, MIR ? 4 : 1>;
  using I2 = std::integral_constant<int, MIR ? 3 : 2>;
  using I3 = std::integral_constant<int, MIR ? 2 : 3>;
  using I4 = std::integral_constant<int, MIR ? 1 : 4>;
  float2 rw[5][6], rr[5];
  for (int j = 0; j <= G; j++) {  // j = G: the middle rows
    const int s = MIR ? nd - 1 - j : j + 1;
    const int q = j < G ? 0 : -6;
    row(I0{}, MIR ? s + 1 : s, q + 0, rw[0], rr[0]);
    row(I1{}, s, q + 1, rw[1], rr[1]);
    row(I2{}, s, q + 2, rw[2], rr[2]);
    row(I3{}, s, q + 3, rw[3], rr[3]);
    row(I4{}, s, q + 4, rw[4], rr[4]);
#pragma unroll
    for (int k = 0; k < 5; k++) {
#pragma unroll
      for (int i = 0; i < 6; i++) W[WI(5, i)] = rw[k][i];
      if (MIR && q < 0) {  // middle row k of the mirrored end
#pragma unroll
        for (int i = 0; i < 6; i++)
          if (i >= 5 - k) W[WI(5, i)] = make_float2(0.f, 0.f);
      }
      y5 = MIR && q < 0 ? make_float2(0.f, 0.f) : rr[k];
      piv(j - 1, k);
    }
  }
}

// where the factors of a direction's four colours lie, and of a group in them
struct FacBlocks {
  long off[4], gstride[4];
};

// Factors of every line of a direction's four colours, for group blockIdx.y of
// operators and frequencies.  A thread per end of a line, each assembling its
// rows in registers (band_row) and eliminating them; the mirrored end hands its
// Schur complement of the middle rows to the other through shared memory.
// What bounds it is the latency of the cells' loads and of the elimination, 16
// warps an SM: the colours read the same cells, so that the four of a block of
// 64 lines are neighbouring blocks (set-up's line factors of 25 operators at
// 128^3 29.8 ms with one colour after the other, 19.6 so; 75 groups 61.5 and
// 54.4).  A line's rows are a chain of some 40 dependent operations each and a
// colour has few lines (1024 at 64^3), so that the chain is the launch's time:
// all of 64^3's one colour a launch 4.5 ms, in one launch a direction 1.0.
// SERIAL: a thread eliminates both ends of its line, the mirrored one first,
// for launches whose lines fill the device several times over (serial_factors);
// the same operations, so the same factors.
// An fp16 L value outside its range (or not finite) sets *ovf.
constexpr int kFacLines = 64;  // lines of a block
template <int D, int FMT, bool SERIAL>
__global__ void __launch_bounds__(SERIAL ? kFacLines : 2 * kFacLines)
    k_line_factor_ends(LevelView<float> L, LineTile tl, FacBlocks fb, float* __restrict__ fac,
                       int* __restrict__ ovf) {
  constexpr int A = (D == 0) ? 1 : 0, B = (D == 2) ? 1 : 2;
  __shared__ float2 schur[15][kFacLines];
  const int grp = blockIdx.y, color = blockIdx.x & 3;
  const LineGeom g = line_geom<D>(L.n, color & 1, color >> 1);
  const int lane = threadIdx.x & (kFacLines - 1);
  const bool bottom = SERIAL || threadIdx.x >= kFacLines, top = SERIAL || threadIdx.x < kFacLines;
  const long first = (long)(blockIdx.x >> 2) * kFacLines, l0 = first + lane;
  if (first >= g.nl) return;  // a colour with fewer lines
  const bool live = l0 < g.nl;
  const long l = live ? l0 : g.nl - 1;
  const unsigned lq = (unsigned)l / (unsigned)g.la;
  const int ta = g.fa + 2 * (int)((unsigned)l - lq * (unsigned)g.la), tb = g.fb + 2 * (int)lq;
  const float* cells = L.cells + (long)op_of(L, grp) * 4 * L.ncell;
  const Geo<float> Gm{L.geo + (long)op_of(L, grp) * L.gstride, L.gmax1};
  const float wmu = L.wmu[grp];
  const int nd = g.nd, G = tl.mid / 5, TW = 1 << tl.shift, ln = (int)(l & (TW - 1));
  unsigned char* out = reinterpret_cast<unsigned char*>(fac + fb.off[color] + (long)grp * fb.gstride[color]) +
                       (l >> tl.shift) * g.m * kFacRow<FMT> * TW;
  bool over = false;
  float2 W[21], lq5[6];
  auto run = [&](auto mir) {
    constexpr bool MIR = decltype(mir)::value;
    float2 y5;
#pragma unroll
    for (int i = 0; i < 21; i++) W[i] = make_float2(0.f, 0.f);
#pragma unroll
    for (int i = 0; i < 5; i++) W[WI(i, i)] = make_float2(1.f, 0.f);  // dummy leading rows
    eliminate_end<MIR>(
        G, nd, W, y5,
        [&](auto tt, int s, int k, float2 (&w)[6], float2& r) {
          constexpr int TT = decltype(tt)::value;
          constexpr int C = (TT == 0) ? D : (TT <= 2 ? A : B);
          float band[5];
          band_row<float, D, TT, C, MIR>(L, cells, Gm, wmu, ta, tb, s, 5 * (s - 1) + TT, band,
                                         w[5]);
#pragma unroll
          for (int j = 0; j < 5; j++) w[j] = make_float2(band[j], 0.f);
          r = make_float2(0.f, 0.f);
        },
        [&](int j, int k) {
          const float2 id = window_step(W, lq5);
          if (j >= 0 && live)
            fac_put<FMT>(out + ((MIR ? tl.mid + 6 : 0) + 5 * j) * kFacRow<FMT> * TW, TW, 5, k, ln,
                         lq5, id, over);
        });
  };
  if (bottom) {
    run(std::true_type());
#pragma unroll
    for (int i = 0; i < 15; i++) schur[i][lane] = W[i];
  }
  if (top) run(std::false_type());
  if constexpr (!SERIAL) __syncthreads();
  if (top) {
    // the middle rows: window 0..4 of this end, row 5 = E_d(G + 1) with its
    // own entries, and the mirrored end's complement of rows 5 - i
    float band[5];
    float2 dg;
    band_row<float, D, 0, D>(L, cells, Gm, wmu, ta, tb, G + 2, 5 * (G + 1), band, dg);
#pragma unroll
    for (int j = 0; j < 5; j++) W[WI(5, j)] = make_float2(band[j], 0.f);
    W[WI(5, 5)] = dg;
#pragma unroll
    for (int i = 0; i < 5; i++)
#pragma unroll
      for (int j = 0; j <= i; j++)
        W[WI(5 - j, 5 - i)] = cadd<float>(W[WI(5 - j, 5 - i)], schur[WI(i, j)][lane]);
    for (int k = 0; k < 6; k++) {
      const float2 id = window_step(W, lq5);
      if (live)
        fac_put<FMT>(out + tl.mid * kFacRow<FMT> * TW, TW, 6, k, ln, lq5, id, over);
      // identity rows follow the last middle row
#pragma unroll
      for (int j = 0; j < 5; j++) W[WI(5, j)] = make_float2(0.f, 0.f);
      W[WI(5, 5)] = make_float2(1.f, 0.f);
    }
  }
  if (over && live) atomicOr(ovf, 1);
}

// ---------------------------------------------------------------- two-ended substitution
// a - b c and a c with the products chained into the sum: two dependent
// multiply-adds a part on the chain from row to row
__device__ __forceinline__ float2 cchain(float2 a, float2 b, float2 c) {
  return make_float2(fmaf(-b.x, c.x, fmaf(b.y, c.y, a.x)), fmaf(-b.x, c.y, fmaf(-b.y, c.x, a.y)));
}

// Substitution of a colour's lines with two-ended factors of group grp[rhs]:
// a tile of TW lines takes 2 TW threads, one for each end of a line (TW = 32:
// a warp an end, one or two tiles a block; TW = 8: both ends in half a warp).
// Each end's groups -- factors and the rows' residuals, contiguous in memory
// -- stream through a ring of NG groups in shared memory, filled by cp.async
// NG groups ahead (NG = 0: a slot for every group, six ahead).  z replaces the
// residual in its slot.  The back substitution starts with the groups the
// forward pass left in the ring, the newest first, and fetches the older ones
// again (z written over their residuals for those): with NG >= G nothing is
// read twice.  D = 1, 2: u += x at each row's slot, the old u fetched into the
// place of 1/d; D = 0 (NG = 0 or NG >= G): u += x along the x lines after the
// back substitution, from shared memory; D = -1: x goes to rb for
// k_line_apply_rb.  Every lane's arithmetic is the same for every shape.
//
// What bounds it: for few lines the chain of 5 G rows an end, about 25 ns a
// row (one shot at 64^3, level 0: 108 us a launch for the one-ended
// substitution with six rows in flight, 13 us so); for many the DRAM (25
// shots at 128^3: y and z sweeps 7.47 and 7.11 -> 6.37 and 5.90 ms, the row
// residuals among them).  Loads are cooperative and of 16 bytes, 2.25 a row
// and lane instead of 4; a ring deeper than the latency needs only saves
// re-reads (16 groups, one block an SM: 7.2 ms).
//
// ROWS (TW = 8): the block's 256 threads form the rows' residuals themselves
// (node_rows), straight into the slots -- lines of a colour do not read each
// other's unknowns, so a colour is one launch -- and 16 of them substitute:
// one shot at 16^3 17.3 -> 14.7 ms, at 64^3 37.2 -> 31.4.
constexpr int kXThreads = 256;  // of a block of x lines, or of one that forms its rows
template <int FMT, int TW, int NG, int D, bool ROWS = false>
__global__ void __launch_bounds__(D == 0 || ROWS ? kXThreads : TW == 32 ? 128 : 32)
    k_line_ends(const int* __restrict__ active, const int* __restrict__ grp, long nl, LineTile tl,
                long gstride, const float* __restrict__ fac, float2* __restrict__ rb,
                LevelView<float> L, int pa, int pb, LineDiv dv, int slots, unsigned tile_bytes) {
  constexpr int PD = NG ? NG : 6;
  constexpr int kRow = kFacRow<FMT>;
  constexpr unsigned kFacB = 5 * kRow * TW, kSlot = kFacB + 40 * TW;
  extern __shared__ __align__(16) unsigned char sm[];
  const int rhs = blockIdx.y;
  if (active && !active[rhs]) {
    dep_wait();
    return;
  }
  const int tid = threadIdx.x;
  const int lane = tid & (TW - 1), end = (tid / TW) & 1, tic = D == 0 || ROWS ? 0 : tid / (2 * TW);
  const int tiles = (int)((nl + TW - 1) / TW);
  const int tile = blockIdx.x * (D == 0 || ROWS ? 1 : blockDim.x / (2 * TW)) + tic;
  if (tile >= tiles) {
    dep_wait();
    return;
  }
  const long l = (long)tile * TW + lane;
  const bool live = l < nl;
  const int m = tl.m, G = tl.mid / 5;
  unsigned char* tsm = sm + tic * tile_bytes;
  unsigned char* ring = tsm + (size_t)end * slots * kSlot;
  unsigned char* midf = tsm + (size_t)2 * slots * kSlot;      // the middle group's factors
  float2* midr = reinterpret_cast<float2*>(midf + 6 * kRow * TW);  // its residuals, then x
  float2* exch = midr + 6 * TW;                                // [end][5][TW]
  const unsigned char* fb = reinterpret_cast<const unsigned char*>(fac + (long)grp[rhs] * gstride) +
                            (long)tile * m * kRow * TW;
  float2* rt = rb + ((long)rhs * tiles + tile) * m * TW;  // this tile's rows by position
  const int p0 = end ? tl.mid + 6 : 0;
  auto tile_sync = [&]() {
    if constexpr (TW == 32) asm volatile("bar.sync %0, 64;\n" ::"r"(1 + tic) : "memory");
    else __syncwarp(0xffffu);
  };
  // the lanes that share a ring: an end's warp, or the tile's half warp
  auto ring_sync = [&]() { __syncwarp(TW == 8 ? 0xffffu : 0xffffffffu); };
  auto slot = [&](int g) -> unsigned char* {
    return ring + (size_t)(NG ? g % NG : g) * kSlot;
  };
  auto copy = [&](unsigned char* dst, const void* src, int bytes) {
    const unsigned char* s8 = static_cast<const unsigned char*>(src);
    for (int c = lane; c < bytes / 16; c += TW) cp_async16(dst + 16 * c, s8 + 16 * c);
  };
  auto issue_fac = [&](int g) { copy(slot(g), fb + (long)(p0 + 5 * g) * kRow * TW, kFacB); };
  auto issue_rows = [&](int g) {
    copy(slot(g) + kFacB, rt + (long)(p0 + 5 * g) * TW, 40 * TW);
  };
  auto issue = [&](int g) {
    issue_fac(g);
    if constexpr (!ROWS) issue_rows(g);
  };
  // slots of u: row t of group g at off[t] + g * step
  float2* u = nullptr;
  int off[5], moff[6], step = 0;
  if constexpr (D >= 1) {
    const LineGeom g = line_geom<D>(L.n, pa, pb);
    const long lc = live ? l : nl - 1;
    const unsigned lq = fdiv((unsigned)lc, dv.la);
    const int ta = g.fa + 2 * (int)((unsigned)lc - lq * (unsigned)g.la);
    const int tb = g.fb + 2 * (int)lq;
    u = L.u + (long)rhs * 3 * L.S;
    const int sd = D == 1 ? L.n[0] + 1 : (L.n[0] + 1) * (L.n[1] + 1);
    const int b0 = (int)line_slot<D, 0>(L.n, L.S, ta, tb, 1);
    const int b1 = (int)line_slot<D, 1>(L.n, L.S, ta, tb, 1);
    const int b2 = (int)line_slot<D, 2>(L.n, L.S, ta, tb, 1);
    const int b3 = (int)line_slot<D, 3>(L.n, L.S, ta, tb, 1);
    const int b4 = (int)line_slot<D, 4>(L.n, L.S, ta, tb, 1);
    const int e = (g.nd - 2) * sd;  // to node nd - 1
    off[0] = end ? b0 + e + sd : b0;  // E_d(nd - 1) or E_d(0)
    off[1] = end ? b4 + e : b1;
    off[2] = end ? b3 + e : b2;
    off[3] = end ? b2 + e : b3;
    off[4] = end ? b1 + e : b4;
    step = end ? -sd : sd;
    moff[0] = b0 + G * sd;
    moff[1] = b1 + G * sd;
    moff[2] = b2 + G * sd;
    moff[3] = b3 + G * sd;
    moff[4] = b4 + G * sd;
    moff[5] = b0 + (G + 1) * sd;
  }
  auto issue_u = [&](int g) {  // into the place of 1/d
    if constexpr (D >= 1) {
      if (live) {
        unsigned char* d = slot(g) + 5 * kFacL<FMT> * TW;
#pragma unroll
        for (int t = 0; t < 5; t++) cp_async8(d + (t * TW + lane) * 8, u + (off[t] + g * step));
      }
    }
  };

  // the factors of the first groups and of the middle rows, which no kernel of
  // a cycle writes, before the wait for the residuals
  const bool worker = tid < 2 * TW || (D != 0 && !ROWS);
  const int at = end * TW + lane;
  if (worker) {
#pragma unroll
    for (int p = 0; p < PD; p++)
      if (p < G) issue_fac(p);
    const unsigned char* mf = fb + (long)tl.mid * kRow * TW;
    for (int c = at; c < 6 * kRow * TW / 16; c += 2 * TW) cp_async16(midf + 16 * c, mf + 16 * c);
  }
  dep_wait();
  dep_next();
  if constexpr (ROWS) {
    // y and z lines: neighbouring threads take neighbouring lines, x lines:
    // neighbouring nodes
    const LineGeom g = line_geom<D>(L.n, pa, pb);
    const int li = D == 0 ? tid >> 5 : tid & 7, s0 = 1 + (D == 0 ? tid & 31 : tid >> 3);
    const long ll = (long)tile * TW + li;
    if (ll < nl) {
      const unsigned lq = fdiv((unsigned)ll, dv.la);
      const int ta = g.fa + 2 * (int)((unsigned)ll - lq * (unsigned)g.la);
      const int tb = g.fb + 2 * (int)lq;
      for (int s = s0; s <= g.nd; s += 32) {
        float2 r[5];
        node_rows<D>(L, rhs, ta, tb, s, r);
#pragma unroll
        for (int t = 0; t < 5; t++) {
          const int row = 5 * (s - 1) + t;
          if (row >= m) continue;
          float2* q;
          if (row < tl.mid) {
            q = reinterpret_cast<float2*>(tsm + (size_t)(s - 1) * kSlot + kFacB) + t * TW;
          } else if (row < tl.mid + 6) {
            q = midr + (row - tl.mid) * TW;
          } else {
            const int k = m - 1 - row, j = k / 5;
            q = reinterpret_cast<float2*>(tsm + (size_t)(slots + j) * kSlot + kFacB) +
                (k - 5 * j) * TW;
          }
          q[li] = r[t];
        }
      }
    }
    __syncthreads();
  }
  auto work = [&]() {
  // forward; the middle rows' u (three an end) is asked for first
  float2 um[3];
  if constexpr (D >= 1) {
#pragma unroll
    for (int i = 0; i < 3; i++)
      um[i] = live ? u[end ? moff[3 + i] : moff[i]] : make_float2(0.f, 0.f);
  }
  if constexpr (!ROWS) {
    const unsigned char* mr = reinterpret_cast<const unsigned char*>(rt + (long)tl.mid * TW);
    for (int c = at; c < 3 * TW; c += 2 * TW)
      cp_async16(reinterpret_cast<unsigned char*>(midr) + 16 * c, mr + 16 * c);
  }
#pragma unroll
  for (int p = 0; p < PD; p++) {
    if (!ROWS && p < G) issue_rows(p);
    cp_async_commit();
  }
  float2 w[5];
#pragma unroll
  for (int i = 0; i < 5; i++) w[i] = make_float2(0.f, 0.f);
  for (int g = 0; g < G; g++) {
    cp_async_wait<PD - 1>();
    ring_sync();
    unsigned char* d = slot(g);
    float2* r = reinterpret_cast<float2*>(d + kFacB) + lane;
    const float2* idp = reinterpret_cast<const float2*>(d + 5 * kFacL<FMT> * TW) + lane;
    const bool spill = NG && g + NG < G;
#pragma unroll
    for (int t = 0; t < 5; t++) {
      float2 v[5];
      fac_get<FMT>(d, TW, t, lane, v);
      const float2 y = cadd<float>(r[t * TW], w[0]);
#pragma unroll
      for (int i = 0; i < 4; i++) w[i] = cchain(w[i + 1], v[i], y);
      w[4] = cchain(make_float2(0.f, 0.f), v[4], y);
      const float2 z = cmul<float>(y, idp[t * TW]);
      r[t * TW] = z;
      if (spill) rt[(long)(p0 + 5 * g + t) * TW + lane] = z;
    }
    ring_sync();
    if (NG) {
      if (g + NG < G) issue(g + NG);
      else issue_u(g);
    } else {
      if (g + PD < G) issue(g + PD);
      issue_u(g);
    }
    cp_async_commit();
  }
#pragma unroll
  for (int i = 0; i < 5; i++) exch[(end * 5 + i) * TW + lane] = w[i];
  cp_async_wait<0>();
  __threadfence_block();  // z spilled by this end's lanes is fetched by others
  tile_sync();
  // the middle six rows, by both ends (the same operations)
  float2 xm[6];
  {
#pragma unroll
    for (int i = 0; i < 6; i++) {
      xm[i] = midr[i * TW + lane];
      if (i < 5) xm[i] = cadd<float>(xm[i], exch[i * TW + lane]);
      if (i > 0) xm[i] = cadd<float>(xm[i], exch[(5 + 5 - i) * TW + lane]);
    }
    float2 v[5];
#pragma unroll
    for (int p = 0; p < 5; p++) {
      fac_get<FMT>(midf, TW, p, lane, v);
#pragma unroll
      for (int i = 1; i < 6; i++)
        if (p + i < 6) xm[p + i] = cchain(xm[p + i], v[i - 1], xm[p]);
    }
    const float2* idp = reinterpret_cast<const float2*>(midf + 6 * kFacL<FMT> * TW) + lane;
#pragma unroll
    for (int p = 5; p >= 0; p--) {
      xm[p] = cmul<float>(xm[p], idp[p * TW]);
      fac_get<FMT>(midf, TW, p, lane, v);
#pragma unroll
      for (int i = 5; i >= 1; i--)
        if (p + i < 6) xm[p] = cchain(xm[p], v[i - 1], xm[p + i]);
    }
  }
  float2 xw[5];
#pragma unroll
  for (int i = 0; i < 5; i++) xw[i] = end ? xm[5 - i] : xm[i];
  if constexpr (D >= 1) {
    if (live) {
#pragma unroll
      for (int i = 0; i < 3; i++)
        u[end ? moff[3 + i] : moff[i]] = cadd<float>(um[i], end ? xm[3 + i] : xm[i]);
    }
  } else if constexpr (D == 0) {
    tile_sync();  // both ends have read the middle residuals
#pragma unroll
    for (int i = 0; i < 6; i++)
      if ((i >= 3) == (end == 1)) midr[i * TW + lane] = xm[i];
  } else {
#pragma unroll
    for (int i = 0; i < 6; i++)
      if ((i >= 3) == (end == 1)) rt[(long)(tl.mid + i) * TW + lane] = xm[i];
  }
  // backward: x = z - sum_i L_i x_{i rows towards the middle}
  for (int g = G - 1; g >= 0; g--) {
    if (NG) {
      cp_async_wait<NG ? NG - 1 : 0>();
      ring_sync();
    }
    unsigned char* d = slot(g);
    float2* r = reinterpret_cast<float2*>(d + kFacB) + lane;
    const float2* uo = reinterpret_cast<const float2*>(d + 5 * kFacL<FMT> * TW) + lane;
#pragma unroll
    for (int t = 4; t >= 0; t--) {
      float2 v[5];
      fac_get<FMT>(d, TW, t, lane, v);
      float2 x = r[t * TW];
#pragma unroll
      for (int i = 4; i >= 0; i--) x = cchain(x, v[i], xw[i]);
#pragma unroll
      for (int i = 4; i > 0; i--) xw[i] = xw[i - 1];
      xw[0] = x;
      if constexpr (D >= 1) {
        if (live) u[off[t] + g * step] = cadd<float>(uo[t * TW], x);
      } else if constexpr (D == 0) {
        r[t * TW] = x;
      } else {
        rt[(long)(p0 + 5 * g + t) * TW + lane] = x;
      }
    }
    if (NG) {
      ring_sync();
      if (g - NG >= 0) {  // the group that lay here before: multipliers, z and u
        copy(d, fb + (long)(p0 + 5 * (g - NG)) * kRow * TW, 5 * kFacL<FMT> * TW);
        copy(d + kFacB, rt + (long)(p0 + 5 * (g - NG)) * TW, 40 * TW);
        issue_u(g - NG);
      }
      cp_async_commit();
    }
  }
  };
  if (worker) work();
  if constexpr (D == 0) {
    // u += x along the lines by the whole block, neighbouring nodes by
    // neighbouring threads (the serial part above occupies 2 TW of them)
    __syncthreads();
    const LineGeom g = line_geom<0>(L.n, pa, pb);
    float2* uu = L.u + (long)rhs * 3 * L.S;
    const unsigned total = 5u * TW * (unsigned)g.nd;
    constexpr int kB = 5;  // slots a thread loads before it stores them
    for (unsigned e0 = tid; e0 < total; e0 += kB * blockDim.x) {
      float2 v[kB], x[kB];
      int sl[kB];
#pragma unroll
      for (int b = 0; b < kB; b++) {
        const unsigned e = e0 + b * blockDim.x;
        sl[b] = -1;
        if (e >= total) continue;
        const unsigned q = fdiv(e, dv.item);
        const int s = (int)(e - q * (unsigned)g.nd), rt5 = (int)(q / TW), li = (int)(q % TW);
        const long ll = (long)tile * TW + li;
        if (ll >= nl || (rt5 > 0 && s == g.nd - 1)) continue;
        const unsigned lq = fdiv((unsigned)ll, dv.la);
        const int ta = g.fa + 2 * (int)((unsigned)ll - lq * (unsigned)g.la);
        const int tb = g.fb + 2 * (int)lq;
        const int base = rt5 == 0   ? (int)line_slot<0, 0>(L.n, L.S, ta, tb, 1)
                         : rt5 == 1 ? (int)line_slot<0, 1>(L.n, L.S, ta, tb, 1)
                         : rt5 == 2 ? (int)line_slot<0, 2>(L.n, L.S, ta, tb, 1)
                         : rt5 == 3 ? (int)line_slot<0, 3>(L.n, L.S, ta, tb, 1)
                                    : (int)line_slot<0, 4>(L.n, L.S, ta, tb, 1);
        sl[b] = base + s;
        v[b] = uu[sl[b]];
        const int row = 5 * s + rt5;
        const float2* xs;
        if (row < tl.mid) {
          xs = reinterpret_cast<const float2*>(sm + (size_t)s * kSlot + kFacB) + rt5 * TW;
        } else if (row < tl.mid + 6) {
          xs = midr + (row - tl.mid) * TW;
        } else {
          const int k = tl.m - 1 - row, j = k / 5;
          xs = reinterpret_cast<const float2*>(sm + (size_t)(slots + j) * kSlot + kFacB) +
               (k - 5 * j) * TW;
        }
        x[b] = xs[li];
      }
#pragma unroll
      for (int b = 0; b < kB; b++)
        if (sl[b] >= 0) uu[sl[b]] = cadd<float>(v[b], x[b]);
    }
  }
}

// shared memory of a tile with `slots` groups an end
template <int FMT>
inline unsigned ends_smem(int tw, int slots) {
  return (unsigned)(tw * (2 * slots * 5 * (kFacRow<FMT> + 8) + 6 * (kFacRow<FMT> + 8) + 80));
}
constexpr int kSmBytes = 224 << 10;  // of an SM's shared memory, 1 KB of it per block the system's
constexpr int kSMs = 152;

// Lines per tile of a level's lines along d, nrhs of them a launch: 8 where
// the blocks of 8 lines, every group in shared memory, are all resident at
// once -- the launch is then one wave of short serial chains on as many SMs
// as there are, with everything read once -- else 32 (more lines in flight per
// SM, full warps).  One 64^3 operator, z sweep (8 launches): 123 us with
// tiles of 8; 25 of them: 819 us with tiles of 32, two waves of 8.
int line_tile_width(const int n[3], int d, int nrhs, int fmt) {
  const long nl = line_count(n, d, 3);
  const int G = (n[d] - 2) / 2;
  const unsigned b =
      (fmt == kFacF16 ? ends_smem<kFacF16>(8, G) : ends_smem<kFacF32>(8, G)) + 1024;
  if (b > (unsigned)kSmBytes) return 32;
  const long per_sm = std::min<long>(kSmBytes / b, 32);
  return (nl + 7) / 8 * nrhs <= kSMs * per_sm ? 8 : 32;
}

// complex128 factors of every line of one colour, for group blockIdx.y of the
// chunk, straight from the operator: a thread assembles a node's band rows in
// registers (band_row) and runs the forward elimination of k_line_solve on
// them -- no band records through memory -- writing the record layout, 12
// values per row, L(p+i, p) for i = 1..5 and 1/d_p, to fac + grp * gstride.
// y and z lines: neighbouring lines are neighbouring slots, so a warp's cell
// loads coalesce; x lines read theirs along each thread's line (uncoalesced,
// still faster than assembling records).
template <typename T, int D>
__global__ void __launch_bounds__(kSolveThreads) k_line_factor_direct(LevelView<T> L, int pa,
                                                                      int pb, long gstride,
                                                                      T* __restrict__ fac) {
  constexpr int A = (D == 0) ? 1 : 0, B = (D == 2) ? 1 : 2;
  using V = typename Vec16<T>::V;
  constexpr int NP = kPlanes<T>;
  const int grp = blockIdx.y;
  const LineGeom g = line_geom<D>(L.n, pa, pb);
  const long l = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (l >= g.nl) return;
  const unsigned lq = (unsigned)l / (unsigned)g.la;
  const int ta = g.fa + 2 * (int)((unsigned)l - lq * (unsigned)g.la), tb = g.fb + 2 * (int)lq;
  const T* cells = L.cells + (long)op_of(L, grp) * 4 * L.ncell;
  const Geo<T> G{L.geo + (long)op_of(L, grp) * L.gstride, L.gmax1};
  const T wmu = L.wmu[grp];
  const int m = g.m, nd = g.nd;
  const long nl = g.nl;
  V* fout = reinterpret_cast<V*>(fac + (long)grp * gstride) + l;
  const long rs = NP * nl;
  C_t<T> W[21];
#pragma unroll
  for (int i = 0; i < 21; i++) W[i] = mk<T>(0, 0);
#pragma unroll
  for (int i = 0; i < 5; i++) W[WI(i, i)] = mk<T>(1, 0);
  // the arriving row sits in W[WI(5, .)]: eliminate pivot row - 5 and
  // store its factors
  auto step = [&](int row) {
    const C_t<T> id = crcp<T>(W[0]);
    C_t<T> lqv[6];
#pragma unroll
    for (int i = 1; i < 6; i++) lqv[i] = cmul<T>(W[WI(i, 0)], id);
#pragma unroll
    for (int i = 1; i < 6; i++) {
#pragma unroll
      for (int j = 1; j <= i; j++) W[WI(i, j)] = cfms<T>(W[WI(i, j)], lqv[i], W[WI(j, 0)]);
    }
    const int piv = row - 5;
    if (piv >= 0) {
      T o[kRec];
#pragma unroll
      for (int i = 1; i < 6; i++) {
        o[2 * (i - 1)] = lqv[i].x;
        o[2 * (i - 1) + 1] = lqv[i].y;
      }
      o[10] = id.x;
      o[11] = id.y;
      rec_put<T>(fout + (long)piv * rs, nl, o);
    }
#pragma unroll
    for (int i = 0; i < 5; i++) {
#pragma unroll
      for (int j = 0; j <= i; j++) W[WI(i, j)] = W[WI(i + 1, j + 1)];
    }
  };
  T bd[5][5];
  C_t<T> dg[5];
  auto assemble = [&](auto tt, int s) {
    constexpr int TT = decltype(tt)::value;
    constexpr int C = (TT == 0) ? D : (TT <= 2 ? A : B);
    band_row<T, D, TT, C>(L, cells, G, wmu, ta, tb, s, 5 * (s - 1) + TT, bd[TT], dg[TT]);
  };
  auto arrive = [&](auto tt, int s) {
    constexpr int TT = decltype(tt)::value;
#pragma unroll
    for (int j = 0; j < 5; j++) W[WI(5, j)] = mk<T>(bd[TT][j], 0);
    W[WI(5, 5)] = dg[TT];
    step(5 * (s - 1) + TT);
  };
  // rows in record order: node s brings row 5(s-1) and, below the last
  // node, its four transverse rows; a node's loads are issued together
  for (int s = 1; s <= nd; s++) {
    assemble(std::integral_constant<int, 0>(), s);
    if (s < nd) {
      assemble(std::integral_constant<int, 1>(), s);
      assemble(std::integral_constant<int, 2>(), s);
      assemble(std::integral_constant<int, 3>(), s);
      assemble(std::integral_constant<int, 4>(), s);
    }
    arrive(std::integral_constant<int, 0>(), s);
    if (s < nd) {
      arrive(std::integral_constant<int, 1>(), s);
      arrive(std::integral_constant<int, 2>(), s);
      arrive(std::integral_constant<int, 3>(), s);
      arrive(std::integral_constant<int, 4>(), s);
    }
  }
  // five unit rows flush the last pivots (rows m..m+4)
  for (int row = m; row < m + 5; row++) {
#pragma unroll
    for (int j = 0; j < 5; j++) W[WI(5, j)] = mk<T>(0, 0);
    W[WI(5, 5)] = mk<T>(1, 0);
    step(row);
  }
}


// Substitution with stored factors (group grp[rhs]): rb holds the rows'
// residuals in, z between the passes, the correction x out.
template <typename T>
__global__ void __launch_bounds__(kSolveThreads) k_line_subst(const int* __restrict__ active,
                                                              const int* __restrict__ grp,
                                                              long nl, int m,
                                                              const T* __restrict__ fac,
                                                              C_t<T>* __restrict__ rb) {
  dep_wait();
  dep_next();
  using V = typename Vec16<T>::V;
  constexpr int NP = kPlanes<T>;
  __shared__ V ring[kRing][NP][kSolveThreads];
  __shared__ C_t<T> rring[kRing][kSolveThreads];
  const int rhs = blockIdx.y;
  if (active && !active[rhs]) return;
  const int tid = threadIdx.x;
  const long l = blockIdx.x * (long)blockDim.x + tid;
  if (l >= nl) return;
  const long rs = NP * nl;
  const V* fb = reinterpret_cast<const V*>(fac) + (long)grp[rhs] * m * rs + l;
  C_t<T>* rr = rb + (long)rhs * m * nl + l;
  auto issue_f = [&](int row) {
    const V* src = fb + (long)row * rs;
    const int slot = row % kRing;
#pragma unroll
    for (int q = 0; q < NP; q++) cp_async16(&ring[slot][q][tid], src + q * nl);
  };
  auto take_f = [&](int row, T (&v)[kRec]) {
    const int slot = row % kRing;
#pragma unroll
    for (int q = 0; q < NP; q++) unpack16(ring[slot][q][tid], v + q * kLanes<T>);
  };
  // forward: at step `row` the residual of row `row` arrives and pivot
  // row-5 is eliminated with its stored factors (k_line_solve's order)
  C_t<T> y[6];
#pragma unroll
  for (int i = 0; i < 6; i++) y[i] = mk<T>(0, 0);
  for (int p = 0; p < kRing - 1; p++) {
    if (p < m) cp_async_c<T>(&rring[p % kRing][tid], rr + (long)p * nl);
    if (p - 5 >= 0 && p - 5 < m) issue_f(p - 5);
    cp_async_commit();
  }
  for (int row = 0; row < m + 5; row++) {
    {
      const int q = row + kRing - 1;
      if (q < m) cp_async_c<T>(&rring[q % kRing][tid], rr + (long)q * nl);
      if (q - 5 >= 0 && q - 5 < m) issue_f(q - 5);
      cp_async_commit();
    }
    cp_async_wait<kRing - 1>();
    y[5] = row < m ? rring[row % kRing][tid] : mk<T>(0, 0);
    const int piv = row - 5;
    if (piv >= 0) {
      T v[kRec];
      take_f(piv, v);
#pragma unroll
      for (int i = 1; i < 6; i++) y[i] = cfms<T>(y[i], mk<T>(v[2 * (i - 1)], v[2 * (i - 1) + 1]), y[0]);
      rr[(long)piv * nl] = cmul<T>(y[0], mk<T>(v[10], v[11]));  // z
    }
#pragma unroll
    for (int i = 0; i < 5; i++) y[i] = y[i + 1];
  }
  cp_async_wait<0>();
  __threadfence_block();  // z just stored is read back below
  // backward: x_k = z_k - sum_i L(k+i, k) x_{k+i}
  C_t<T> xw[5];
#pragma unroll
  for (int i = 0; i < 5; i++) xw[i] = mk<T>(0, 0);
  for (int p = 0; p < kRing - 1; p++) {
    const int q = m - 1 - p;
    if (q >= 0) {
      issue_f(q);
      cp_async_c<T>(&rring[q % kRing][tid], rr + (long)q * nl);
    }
    cp_async_commit();
  }
  for (int row = m - 1; row >= 0; row--) {
    {
      const int q = row - (kRing - 1);
      if (q >= 0) {
        issue_f(q);
        cp_async_c<T>(&rring[q % kRing][tid], rr + (long)q * nl);
      }
      cp_async_commit();
    }
    cp_async_wait<kRing - 1>();
    T v[kRec];
    take_f(row, v);
    C_t<T> x = rring[row % kRing][tid];
#pragma unroll
    for (int i = 0; i < 5; i++) x = cfms<T>(x, mk<T>(v[2 * i], v[2 * i + 1]), xw[i]);
#pragma unroll
    for (int i = 4; i > 0; i--) xw[i] = xw[i - 1];
    xw[0] = x;
    rr[(long)row * nl] = x;
  }
  cp_async_wait<0>();
}


// The same substitution with 12 lanes a line, two lines a warp, for few lines:
// an FP64 instruction takes an SM quarter about 60 clocks however many of a
// warp's lanes are active and however independent the instructions are, so
// what a line's chain costs is the number of instructions, not of operations.
// Lane 2 j + part of a line holds the real or imaginary part of the rows with
// row % 6 == j.  Forward, a pivot's value is shuffled to the lanes of the five
// rows that follow, which take their product with the multiplier off it, while
// the pivot's lane forms z with the same instructions: three an FP64 row in
// place of 34.  Backward, the five products are formed in the lanes of the
// known x and subtracted in the pivot's, newest first: seven in place of 30.
// k_line_subst's operations in its order, the same result bit for bit.
// Mean over a cycle's launches: one RHS at 16^3 71 -> 27 us, four at
// 64 x 56 x 48 170 -> 87.
__global__ void __launch_bounds__(128) k_line_subst_lanes(const int* __restrict__ active,
                                                          const int* __restrict__ grp, long nl,
                                                          int m, const double* __restrict__ fac,
                                                          double2* rb) {
  dep_wait();
  dep_next();
  const int rhs = blockIdx.y;
  if (active && !active[rhs]) return;
  const int lane = threadIdx.x & 31;
  const long w = blockIdx.x * 4L + (threadIdx.x >> 5);
  if (2 * w >= nl) return;  // a warp at a time
  const int sub = lane < 12 ? 0 : lane < 24 ? 1 : 2, base = sub * 12;
  const bool live = sub < 2 && 2 * w + sub < nl;
  const long l = live ? 2 * w + sub : 2 * w;
  const int j = ((lane - base) >> 1) % 6, part = (lane - base) & 1;
  const int src = sub < 2 ? base : 0;  // idle lanes shuffle from the first line
  const long rs = 6 * nl;
  const double2* fb = reinterpret_cast<const double2*>(fac) + (long)grp[rhs] * m * rs + l;
  double* rr = reinterpret_cast<double*>(rb + (long)rhs * m * nl + l) + part;
  auto role = [&](int u) { return j >= u ? j - u : j - u + 6; };  // (j - u) mod 6
  auto factor = [&](int row, int i) -> double2 {                  // L_i, 1/d for i = 0
    return row < m ? ldro(fb + row * rs + (i == 0 ? 5 : i - 1) * nl) : make_double2(0.0, 0.0);
  };
  auto res = [&](int row) { return row < m ? rr[2 * (long)row * nl] : 0.0; };
  double2 cur[6], nxt[6];
  double rn, y = res(j);
#pragma unroll
  for (int u = 0; u < 6; u++) cur[u] = factor(u, role(u));
  for (int p0 = 0; p0 < m; p0 += 6) {
    // the next six rows: multipliers, and the residual this lane takes next
    rn = res(p0 + 6 + j);
#pragma unroll
    for (int u = 0; u < 6; u++) nxt[u] = factor(p0 + 6 + u, role(u));
#pragma unroll
    for (int u = 0; u < 6; u++) {
      const double yx = __shfl_sync(0xffffffffu, y, src + 2 * u);
      const double yy = __shfl_sync(0xffffffffu, y, src + 2 * u + 1);
      const bool piv = j == u;
      const double2 v = cur[u];
      // as cfms(., L, y) and, for z, cmul(y, 1/d) round: real L.x y.x with
      // -(L.y y.y) rounded first, imaginary L.y y.x on L.x y.y (z: y.y d.x on
      // y.x d.y)
      const bool sw = part && !piv;
      const double a = sw ? v.y : v.x, b = part && piv ? yy : yx;
      const double c = sw ? v.x : v.y, d = part ? (piv ? yx : yy) : -yy;
      const double t = rfma(a, b, rmul(c, d));
      const int row = p0 + u;
      if (piv) {
        if (live && row < m) rr[2 * (long)row * nl] = t;  // z
        y = rn;
      } else {
        y = rsub(y, t);
      }
    }
#pragma unroll
    for (int u = 0; u < 6; u++) cur[u] = nxt[u];
  }
  __syncwarp();
  // backward: x_k = z_k - sum_i L(k+i, k) x_{k+i}
  double x = 0.0;
  const int c0 = (m - 1) / 6 * 6;
  auto back = [&](int row, int u) -> double2 {  // multipliers, z in the pivot's lane
    if (row >= m) return make_double2(0.0, 0.0);
    return role(u) == 0 ? make_double2(rr[2 * (long)row * nl], 0.0)
                        : ldro(fb + row * rs + (role(u) - 1) * nl);
  };
#pragma unroll
  for (int u = 0; u < 6; u++) cur[u] = back(c0 + u, u);
  for (int p0 = c0; p0 >= 0; p0 -= 6) {
    if (p0 >= 6) {
#pragma unroll
      for (int u = 0; u < 6; u++) nxt[u] = back(p0 - 6 + u, u);
    }
#pragma unroll
    for (int u = 5; u >= 0; u--) {
      const double xo = __shfl_xor_sync(0xffffffffu, x, 1);
      const double2 v = cur[u];
      const double t = part ? rfma(v.y, xo, rmul(v.x, x)) : rfma(v.x, x, -rmul(v.y, xo));
      double s = v.x;  // z in the pivot's lane
#pragma unroll
      for (int q = 1; q < 6; q++)
        s = rsub(s, __shfl_sync(0xffffffffu, t, src + 2 * ((u + q) % 6) + part));
      const int row = p0 + u;
      if (j == u && row < m) {
        x = s;
        if (live) rr[2 * (long)row * nl] = x;
      }
    }
#pragma unroll
    for (int u = 0; u < 6; u++) cur[u] = nxt[u];
  }
}

// u += x from rb
template <typename T, int D>
__global__ void __launch_bounds__(256) k_line_apply_rb(LevelView<T> L, int pa, int pb, LineDiv dv,
                                                       LineTile tl, const C_t<T>* rb) {
  dep_wait();
  dep_next();
  const int rhs = blockIdx.y;
  if (L.active && !L.active[rhs]) return;
  const LineGeom g = line_geom<D>(L.n, pa, pb);
  long l;
  int s;
  if (!line_item_fd<D>(g, dv, blockIdx.x * blockDim.x + threadIdx.x, l, s)) return;
  const unsigned lq = fdiv((unsigned)l, dv.la);
  const int ta = g.fa + 2 * (int)((unsigned)l - lq * (unsigned)g.la), tb = g.fb + 2 * (int)lq;
  C_t<T>* u = L.u + (long)rhs * 3 * L.S;
  const C_t<T>* x = rb + (long)rhs * rb_elems<T>(tl, g.nl);
  const int r0 = 5 * (s - 1);
  // every load before the first store
  const long sl[5] = {line_slot<D, 0>(L.n, L.S, ta, tb, s), line_slot<D, 1>(L.n, L.S, ta, tb, s),
                      line_slot<D, 2>(L.n, L.S, ta, tb, s), line_slot<D, 3>(L.n, L.S, ta, tb, s),
                      line_slot<D, 4>(L.n, L.S, ta, tb, s)};
  const int nr = s < g.nd ? 5 : 1;
  C_t<T> v[5];
#pragma unroll
  for (int t = 0; t < 5; t++)
    if (t < nr) v[t] = cadd<T>(u[sl[t]], x[rb_index<T>(tl, g.nl, l, r0 + t)]);
#pragma unroll
  for (int t = 0; t < 5; t++)
    if (t < nr) u[sl[t]] = v[t];
}
// ---------------------------------------------------------------- launches
// block shapes of the two-ended substitution with 32-line tiles: lines per
// block and groups of the ring; variant 0 is the default
constexpr int kSubstShape[kSubstVariants][2] = {{64, 6}, {32, 5}, {32, 8}, {32, 4}, {64, 4}};

int subst_variant_threads(int v) { return kSubstShape[v][0]; }
int subst_variant_ring(int v) { return kSubstShape[v][1]; }

struct EndsArgs {
  const LevelView<float>* L;
  const int* grp;
  long nl;
  LineTile tl;
  long gstride;
  const float* fac;
  float2* rb;
  int pa, pb;
  LineDiv dv;
};

template <int FMT, int TW, int NG, int D, bool ROWS = false>
static void ends_launch(const EndsArgs& a, int tpc, cudaStream_t st) {
  const int G = a.tl.mid / 5, slots = NG && NG < G ? NG : G;
  const unsigned tb = ends_smem<FMT>(TW, slots);
  static DeviceOnce once;
  once_on_device(once, [] {
    cudaFuncSetAttribute(k_line_ends<FMT, TW, NG, D, ROWS>,
                         cudaFuncAttributeMaxDynamicSharedMemorySize, 227 << 10);
  });
  const long tiles = (a.nl + TW - 1) / TW;
  if (D == 0 || ROWS) tpc = 1;
  dim3 g((unsigned)((tiles + tpc - 1) / tpc), a.L->nrhs);
  launch_dep(k_line_ends<FMT, TW, NG, D, ROWS>, g, D == 0 || ROWS ? kXThreads : 2 * TW * tpc,
             tpc * tb, st, a.L->active, a.grp, a.nl, a.tl, a.gstride, a.fac, a.rb, *a.L, a.pa, a.pb,
             a.dv, slots, tb);
}

// the ring of a launch: NG of the shape, one NG for the fp32 format
template <int FMT>
static int ends_ring(SweepShape sh) {
  return FMT == kFacF16 ? kSubstShape[sh.subst >= 0 && sh.subst < kSubstVariants ? sh.subst : 0][1] : 4;
}
// every group of a line along d in its ring (x lines then update u themselves)
static bool ends_resident(const int n[3], int d, int tile, int fmt, SweepShape sh) {
  const int G = (n[d] - 2) / 2;
  return tile < 32 || G <= (fmt == kFacF16 ? ends_ring<kFacF16>(sh) : ends_ring<kFacF32>(sh));
}

// whether a colour's blocks form their rows themselves: a block an SM holds the
// whole colour (six RHS at 80 x 56 x 72 43.1 ms a solve; 44.6 with up to two
// blocks an SM, 51.4 with four: 256 threads then wait for 16)
static bool ends_rows(long nl, int nrhs, int tile, int imu_vol) {
  return tile == 8 && imu_vol && (nl + 7) / 8 * nrhs <= kSMs;
}

template <int FMT, int D>
static void ends_dispatch(const EndsArgs& a, SweepShape sh, bool rows, cudaStream_t st) {
  const int tw = 1 << a.tl.shift;
  if (tw == 8) {
    if constexpr (D >= 0) {
      if (rows) ends_launch<FMT, 8, 0, D, true>(a, 1, st);
      else ends_launch<FMT, 8, 0, D>(a, 1, st);
    }
    return;
  }
  if constexpr (FMT == kFacF32) {
    ends_launch<FMT, 32, 4, D>(a, 1, st);
  } else {
    const int lines = kSubstShape[sh.subst >= 0 && sh.subst < kSubstVariants ? sh.subst : 0][0];
    switch (ends_ring<FMT>(sh)) {
      case 4: ends_launch<FMT, 32, 4, D>(a, lines / 32, st); break;
      case 5: ends_launch<FMT, 32, 5, D>(a, 1, st); break;
      case 8: ends_launch<FMT, 32, 8, D>(a, 1, st); break;
      default: ends_launch<FMT, 32, 6, D>(a, lines / 32, st); break;
    }
  }
}

// u += x from rb, where the substitution leaves x there
template <typename T, int D>
static void apply_rb(const LevelView<T>& L, int pa, int pb, const LineDiv& dv, const LineTile& tl,
                     const C_t<T>* rb, cudaStream_t st) {
  dim3 g1((dv.items + 255) / 256, L.nrhs);
  launch_dep(k_line_apply_rb<T, D>, g1, 256, 0, st, L, pa, pb, dv, tl, rb);
}

constexpr long kLaneLines = 7680;

template <int D, int NW>
static void line_rows(const LevelView<float>& L, int pa, int pb, long nl, const LineDiv& dv,
                      const LineTile& tl, float2* rb, cudaStream_t st) {
  const int nodes = (L.n[D] + (D == 0 ? 31 : NW - 1)) / (D == 0 ? 32 : NW);
  const int lines = (int)((nl + (D == 0 ? NW - 1 : 31)) / (D == 0 ? NW : 32));
  dim3 g((unsigned)(nodes * lines), L.nrhs);
  launch_dep(k_line_rows<D, NW>, g, 32 * NW, 0, st, L, pa, pb, dv, tl, nodes, lines, rb);
}

template <typename T, int D>
static void line_sweep_fac_d(const LevelView<T>& L, int color, const T* fac, const int* grp,
                             C_t<T>* rb, int fmt, int tile, SweepShape sh, const double* coef,
                             cudaStream_t st) {
  const int pa = color & 1, pb = (color >> 1) & 1;
  const long nl = line_count(L.n, D, color);
  if (nl == 0) return;
  const long items = nl * L.n[D];
  const int m = 5 * L.n[D] - 4;
  const int rt = sh.rhs_threads == 128 ? 128 : 256;
  dim3 gr((unsigned)(((D == 0 ? 5 : 1) * items + rt - 1) / rt), L.nrhs);
  const LineDiv dv = line_div<D>(L.n, pa, pb);
  const LineTile tl = line_tile(L.n[D], tile);
  const bool in_one = std::is_same<T, float>::value && ends_rows(nl, L.nrhs, tile, L.imu_vol);
  bool rows = in_one;
  if constexpr (std::is_same<T, float>::value) {
    if (L.imu_vol && !in_one) {
      rt == 128 ? line_rows<D, 4>(L, pa, pb, nl, dv, tl, rb, st)
                : line_rows<D, 8>(L, pa, pb, nl, dv, tl, rb, st);
      rows = true;
    }
  }
  if (!rows) {
    if constexpr (std::is_same<T, double>::value) {
      if (coef) {
        launch_dep(k_line_rhs<T, D, true, false>, gr, rt, 0, st, L, pa, pb, dv, tl, rb, coef);
        rows = true;
      }
    }
    // a grid too large to be launched dependent reads u by read-only loads
    if (!rows && depends(gr))
      launch_dep(k_line_rhs<T, D, false, false>, gr, rt, 0, st, L, pa, pb, dv, tl, rb, nullptr);
    else if (!rows)
      k_line_rhs<T, D, false, true><<<gr, rt, 0, st>>>(L, pa, pb, dv, tl, rb, nullptr);
  }
  if constexpr (std::is_same<T, float>::value) {
    const EndsArgs a{&L, grp, nl, tl, line_factor_elems(L.n, D, color, fmt, tile), fac, rb, pa, pb,
                     dv};
    const bool res = ends_resident(L.n, D, tile, fmt, sh);
    constexpr int DS = D == 0 ? -1 : D;  // x lines with a ring too short for them
    if (fmt == kFacF16) {
      if (res) ends_dispatch<kFacF16, D>(a, sh, in_one, st);
      else ends_dispatch<kFacF16, DS>(a, sh, false, st);
    } else {
      if (res) ends_dispatch<kFacF32, D>(a, sh, in_one, st);
      else ends_dispatch<kFacF32, DS>(a, sh, false, st);
    }
    if constexpr (D == 0)
      if (!res) apply_rb<T, D>(L, pa, pb, dv, tl, rb, st);
  } else {
    // 12 lanes a line while that is shorter: two lines a warp and 10 FP64
    // instructions a row against 32 lines and 64, on 4 x 152 SM quarters --
    // 60 clocks x 10 x lines / 1216 a row against 60 x 64
    if (nl * L.nrhs <= kLaneLines) {
      launch_dep(k_line_subst_lanes, dim3((unsigned)((nl + 7) / 8), L.nrhs), dim3(128), 0, st,
                 L.active, grp, nl, m, fac, rb);
    } else {
      dim3 g2((unsigned)((nl + kSolveThreads - 1) / kSolveThreads), L.nrhs);
      // not beside the kernel before, whose carveout leaves room for few of
      // its blocks (four shots at 128^3, three cycles: 321 -> 222 ms)
      k_line_subst<T><<<g2, kSolveThreads, 0, st>>>(L.active, grp, nl, m, fac, rb);
    }
    apply_rb<T, D>(L, pa, pb, dv, tl, rb, st);
  }
}

// a line a thread where that alone is four waves of 512 threads an SM (75
// groups at 128^3: 52.1 ms, 54.4 with a thread an end; 25: 18.8 and 19.6), an
// end a thread below (20 at 96^3: 7.3 and 7.1 ms; one at 64^3: 1.44 and 1.02)
static bool serial_factors(long lines, int groups) {
  return 4 * lines * groups >= 4L * kSMs * 512;
}

template <typename T, int D>
static void line_factor_d(const LevelView<T>& L, T* fac, const long off[4], int fmt, int tile,
                          int* ovf, cudaStream_t st) {
  FacBlocks fb;
  long most = 0;
  for (int c = 0; c < 4; c++) {
    fb.off[c] = off[c];
    fb.gstride[c] = line_factor_elems(L.n, D, c, fmt, tile);
    most = std::max(most, line_count(L.n, D, c));
  }
  if (most == 0) return;
  if constexpr (std::is_same<T, float>::value) {
    const LineTile tl = line_tile(L.n[D], tile);
    const dim3 g(4 * (unsigned)((most + kFacLines - 1) / kFacLines), L.nrhs);
    auto go = [&](auto k, int threads) { k<<<g, threads, 0, st>>>(L, tl, fb, fac, ovf); };
    const bool serial = serial_factors(most, L.nrhs);
    if (fmt == kFacF16 && serial) go(k_line_factor_ends<D, kFacF16, true>, kFacLines);
    else if (fmt == kFacF16) go(k_line_factor_ends<D, kFacF16, false>, 2 * kFacLines);
    else if (serial) go(k_line_factor_ends<D, kFacF32, true>, kFacLines);
    else go(k_line_factor_ends<D, kFacF32, false>, 2 * kFacLines);
  } else {
    for (int c = 0; c < 4; c++) {
      const long nl = line_count(L.n, D, c);
      if (nl == 0) continue;
      dim3 g((unsigned)((nl + kSolveThreads - 1) / kSolveThreads), L.nrhs);
      k_line_factor_direct<T, D><<<g, kSolveThreads, 0, st>>>(L, c & 1, c >> 1, fb.gstride[c],
                                                              fac + fb.off[c]);
    }
  }
}

void init_stored_line_kernels() {
  cudaFuncSetAttribute(k_line_subst<double>, cudaFuncAttributePreferredSharedMemoryCarveout,
                       cudaSharedmemCarveoutMaxShared);
}

long line_factor_elems(const int n[3], int d, int color, int fmt, int tile) {
  const int m = 5 * n[d] - 4;
  const long nl = line_count(n, d, color);
  if (!tile) return (long)m * nl * kRec;  // complex128 records
  const long lines = (nl + tile - 1) / tile * tile;
  return lines * m * (fmt == kFacF16 ? kFacRow<kFacF16> : kFacRow<kFacF32>) / 4;
}

long line_rb_elems(const int n[3], int d, int color, int tile) {
  const int m = 5 * n[d] - 4;
  const long nl = line_count(n, d, color);
  return tile ? (nl + tile - 1) / tile * tile * m : nl * m;
}

int line_fac_launches(const int n[3], int d, int color, int nrhs, int tile, int fmt, int imu_vol,
                      SweepShape sh) {
  const long nl = line_count(n, d, color);
  if (nl == 0) return 0;
  if (tile && ends_rows(nl, nrhs, tile, imu_vol)) return 1;
  return tile && (d != 0 || ends_resident(n, d, tile, fmt, sh)) ? 2 : 3;
}

template <typename T>
void launch_line_factor(const LevelView<T>& L, int d, T* fac, const long off[4], int fmt, int tile,
                        int* ovf, cudaStream_t st) {
  if (d == 0) line_factor_d<T, 0>(L, fac, off, fmt, tile, ovf, st);
  else if (d == 1) line_factor_d<T, 1>(L, fac, off, fmt, tile, ovf, st);
  else line_factor_d<T, 2>(L, fac, off, fmt, tile, ovf, st);
}

template <typename T>
void launch_line_sweep_fac(const LevelView<T>& L, int d, int color, const T* fac, const int* grp,
                           C_t<T>* rb, int fmt, int tile, cudaStream_t st, SweepShape sh,
                           const double* coef) {
  if (d == 0) line_sweep_fac_d<T, 0>(L, color, fac, grp, rb, fmt, tile, sh, coef, st);
  else if (d == 1) line_sweep_fac_d<T, 1>(L, color, fac, grp, rb, fmt, tile, sh, coef, st);
  else line_sweep_fac_d<T, 2>(L, color, fac, grp, rb, fmt, tile, sh, coef, st);
}
template void launch_line_factor<float>(const LevelView<float>&, int, float*, const long*, int, int,
                                        int*, cudaStream_t);
template void launch_line_factor<double>(const LevelView<double>&, int, double*, const long*, int,
                                         int, int*, cudaStream_t);
template void launch_line_sweep_fac<float>(const LevelView<float>&, int, int, const float*,
                                           const int*, C_t<float>*, int, int, cudaStream_t,
                                           SweepShape, const double*);
template void launch_line_sweep_fac<double>(const LevelView<double>&, int, int, const double*,
                                            const int*, C_t<double>*, int, int, cudaStream_t,
                                            SweepShape, const double*);

// ---------------------------------------------------------------- fused line relaxation
// One launch per colour and direction.  complex128 (k_line_fused): a thread
// owns one line and walks it twice; complex64 (k_line_fused_ends): two threads,
// one from either end, the multipliers as LineL keeps them.
//   forward   node by node it assembles each row -- band entries and the
//             residual of the current iterate, the row arithmetic of
//             assemble_row -- and feeds it to the streaming LDL^T of
//             k_line_solve: the arriving row eliminates pivot row-5, whose
//             z = D^-1 L^-1 r and L(p+i, p), i = 1..5, are set aside;
//   backward  x_p = z_p - sum_i L(p+i, p) x_{p+i}, u += x at the row's slot.
// z_p waits in the level's residual buffer at row p's own slot: no other line
// of the colour reads or writes it, and that buffer is dead while the level
// smooths (the cycle recomputes the residual after smoothing).  L waits in
// the line scratch, [row][line] planes per RHS:
//   kLExact  the working precision's values (in complex128 k_line_solve's
//            arithmetic, bit for bit the same operations in the same order);
//   kLHalf   (complex64) rounded to fp16 and used rounded by both
//            substitutions while the elimination keeps the unrounded value:
//            each line solve is then exact for a matrix within fp16 rounding
//            of the line's -- the arithmetic of the stored-factor format
//            kFacF16.  An L value outside the fp16 range sets *ovf.
// Against the three-kernel sweep this writes no band records and reads no
// stored factors: per row the neighbourhood of the residual, L (20 or 40
// bytes) and z (8 bytes) out and back, and u read-modify-write.
template <typename T, int LF> struct LineL;
template <> struct LineL<float, kLExact> {
  static constexpr long kBytes = 40;  // per row
  float4* p0;
  float4* p1;
  float2* p2;
  __device__ __forceinline__ LineL(void* base, int m, long nl) {
    p0 = reinterpret_cast<float4*>(base);
    p1 = p0 + (long)m * nl;
    p2 = reinterpret_cast<float2*>(p1 + (long)m * nl);
  }
  __device__ __forceinline__ bool put(long o, const float2 (&l)[6]) {
    p0[o] = make_float4(l[1].x, l[1].y, l[2].x, l[2].y);
    p1[o] = make_float4(l[3].x, l[3].y, l[4].x, l[4].y);
    p2[o] = l[5];
    return false;
  }
  __device__ __forceinline__ void round(float2 (&) [6]) const {}
  __device__ __forceinline__ bool bad(const float2 (&)[6]) const { return false; }
  __device__ __forceinline__ void get(long o, float2 (&l)[5]) const {
    const float4 a = p0[o], b = p1[o];
    l[0] = make_float2(a.x, a.y);
    l[1] = make_float2(a.z, a.w);
    l[2] = make_float2(b.x, b.y);
    l[3] = make_float2(b.z, b.w);
    l[4] = p2[o];
  }
};
template <> struct LineL<double, kLExact> {
  static constexpr long kBytes = 80;
  double2* p;
  long ps;
  __device__ __forceinline__ LineL(void* base, int m, long nl) {
    p = reinterpret_cast<double2*>(base);
    ps = (long)m * nl;
  }
  __device__ __forceinline__ bool put(long o, const double2 (&l)[6]) {
#pragma unroll
    for (int i = 0; i < 5; i++) p[i * ps + o] = l[i + 1];
    return false;
  }
  __device__ __forceinline__ void round(double2 (&) [6]) const {}
  __device__ __forceinline__ void get(long o, double2 (&l)[5]) const {
#pragma unroll
    for (int i = 0; i < 5; i++) l[i] = p[i * ps + o];
  }
};
template <> struct LineL<float, kLHalf> {
  static constexpr long kBytes = 20;
  uint4* la;
  uint32_t* lb;
  __device__ __forceinline__ LineL(void* base, int m, long nl) {
    la = reinterpret_cast<uint4*>(base);
    lb = reinterpret_cast<uint32_t*>(la + (long)m * nl);
  }
  __device__ __forceinline__ bool bad(const float2 (&l)[6]) const {
    bool over = false;
#pragma unroll
    for (int i = 1; i < 6; i++) over |= !(fabsf(l[i].x) <= 65504.f && fabsf(l[i].y) <= 65504.f);
    return over;
  }
  // l[1..5] rounded to fp16 in place (the values both substitutions use);
  // true when one left the fp16 range
  __device__ __forceinline__ void round(float2 (&l)[6]) const {
#pragma unroll
    for (int i = 1; i < 6; i++) l[i] = __half22float2(__floats2half2_rn(l[i].x, l[i].y));
  }
  __device__ __forceinline__ bool put(long o, const float2 (&l)[6]) {
    __half2 h[5];
    bool over = false;
#pragma unroll
    for (int i = 0; i < 5; i++) {
      h[i] = __floats2half2_rn(l[i + 1].x, l[i + 1].y);
      over |= !(fabsf(l[i + 1].x) <= 65504.f && fabsf(l[i + 1].y) <= 65504.f);
    }
    la[o] = make_uint4(h2u(h[0]), h2u(h[1]), h2u(h[2]), h2u(h[3]));
    lb[o] = h2u(h[4]);
    return over;
  }
  __device__ __forceinline__ void get(long o, float2 (&l)[5]) const {
    const uint4 a = la[o];
    l[0] = u2f2(a.x);
    l[1] = u2f2(a.y);
    l[2] = u2f2(a.z);
    l[3] = u2f2(a.w);
    l[4] = u2f2(lb[o]);
  }
};

long line_l_bytes(const int n[3], int d, int color, int lf, int tsize) {
  const long m = 5 * n[d] - 4, nl = line_count(n, d, color);
  const long b = lf == kLHalf ? 20 : (tsize == 8 ? 80 : 40);
  return (m * nl * b + 255) / 256 * 256;
}

// band entries (real; MIR: to the rows after it, band_row), diagonal and
// residual of row type TT of node s
template <typename T, int D, int TT, int C, bool MIR = false, bool RO = false>
__device__ __forceinline__ void fused_row(const LevelView<T>& L, const C_t<T>* u, const C_t<T>* f,
                                          const T* cells, const Geo<T>& G, T wmu, int ta, int tb,
                                          int s, int row, const long ss[3], C_t<T> (&wrow)[6],
                                          C_t<T>& r) {
  constexpr int A = (D == 0) ? 1 : 0, B = (D == 2) ? 1 : 2;
  int P[3];
  P[D] = (TT == 0) ? s - 1 : s;
  P[A] = ta - (TT == 1 ? 1 : 0);
  P[B] = tb - (TT == 3 ? 1 : 0);
  const int sl = P[0] + (L.n[0] + 1) * (P[1] + (L.n[1] + 1) * P[2]);  // 32-bit slot
  EdgeCoef<T> e;
  const C_t<T> au = apply_row<T, C, 2, RO>(L, u, cells, G, wmu, P, sl, ss, e);
  r = csub<T>(f[C * (int)L.S + sl], au);
  T band[5] = {0, 0, 0, 0, 0};
#define LINE_ENTRY(K)                                                         \
  {                                                                           \
    constexpr int off = line_off(D, TT, K);                                   \
    if constexpr (!MIR && off < 0) {                                          \
      if (row + off >= 0) band[5 + off] = e.c[K];                             \
    }                                                                         \
    if constexpr (MIR && off > 0 && off < 127) {                              \
      if (row + off < 5 * L.n[D] - 4) band[5 - off] = e.c[K];                 \
    }                                                                         \
  }
  LINE_ENTRY(0) LINE_ENTRY(1) LINE_ENTRY(2) LINE_ENTRY(3) LINE_ENTRY(4) LINE_ENTRY(5)
  LINE_ENTRY(6) LINE_ENTRY(7) LINE_ENTRY(8) LINE_ENTRY(9) LINE_ENTRY(10) LINE_ENTRY(11)
#undef LINE_ENTRY
#pragma unroll
  for (int j = 0; j < 5; j++) wrow[j] = mk<T>(band[j], 0);
  wrow[5] = mk<T>(e.dre, e.dim);
}

// one elimination step of the streaming LDL^T (k_line_solve's order): the
// new row sits in W[WI(5, .)], y[5]; pivot W[0] is eliminated.  Returns
// z = y_0 / d_0 and the multipliers l[1..5] (rounded by LS::round for kLHalf,
// the unrounded ones updating the window)
template <typename T, typename LS>
__device__ __forceinline__ C_t<T> fused_eliminate(C_t<T> (&W)[21], C_t<T> (&y)[6],
                                                  C_t<T> (&lr)[6], const LS& ls) {
  const C_t<T> id = crcp<T>(W[0]);
  C_t<T> lq[6];
#pragma unroll
  for (int i = 1; i < 6; i++) lq[i] = cmul<T>(W[WI(i, 0)], id);
#pragma unroll
  for (int i = 1; i < 6; i++) lr[i] = lq[i];
  ls.round(lr);
#pragma unroll
  for (int i = 1; i < 6; i++) {
#pragma unroll
    for (int j = 1; j <= i; j++) W[WI(i, j)] = cfms<T>(W[WI(i, j)], lq[i], W[WI(j, 0)]);
    y[i] = cfms<T>(y[i], lr[i], y[0]);
  }
  const C_t<T> z = cmul<T>(y[0], id);
#pragma unroll
  for (int i = 0; i < 5; i++) {
#pragma unroll
    for (int j = 0; j <= i; j++) W[WI(i, j)] = W[WI(i + 1, j + 1)];
    y[i] = y[i + 1];
  }
  return z;
}

// complex128.  Launched the ordinary way, so that its loads of u may be
// read-only ones, which move past its stores (four cycles of four shots at
// 128^3: 1836 ms, with dependent launches and ordinary loads 2106).
template <typename T, int D, int LF, int NT>
__global__ void __launch_bounds__(NT) k_line_fused(LevelView<T> L, int pa, int pb, LineDiv dv,
                                                   void* __restrict__ lbuf, long lstride,
                                                   int* __restrict__ ovf) {
  constexpr int A = (D == 0) ? 1 : 0, B = (D == 2) ? 1 : 2;
  using LS = LineL<T, LF>;
  const int rhs = blockIdx.y;
  if (L.active && !L.active[rhs]) return;
  const LineGeom g = line_geom<D>(L.n, pa, pb);
  const long l = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (l >= g.nl) return;
  const unsigned lq = fdiv((unsigned)l, dv.la);
  const int ta = g.fa + 2 * (int)((unsigned)l - lq * (unsigned)g.la), tb = g.fb + 2 * (int)lq;
  const int n0 = L.n[0] + 1, n1 = L.n[1] + 1;
  const long ss[3] = {1, (long)n0, (long)n0 * n1};
  C_t<T>* __restrict__ u = L.u + (long)rhs * 3 * L.S;
  const C_t<T>* __restrict__ f = L.f + (long)rhs * 3 * L.S;
  C_t<T>* __restrict__ zr = L.r + (long)rhs * 3 * L.S;
  const T* __restrict__ cells = L.cells + (long)op_of(L, rhs) * 4 * L.ncell;
  const Geo<T> G{L.geo + (long)op_of(L, rhs) * L.gstride, L.gmax1};
  const T wmu = L.wmu[rhs];
  LS ls(static_cast<char*>(lbuf) + (long)rhs * lstride, g.m, g.nl);
  const int nd = g.nd;
  bool over = false;

  C_t<T> W[21], y[6], lr[6];
#pragma unroll
  for (int i = 0; i < 21; i++) W[i] = mk<T>(0, 0);
#pragma unroll
  for (int i = 0; i < 5; i++) {
    W[WI(i, i)] = mk<T>(1, 0);  // dummy leading rows
    y[i] = mk<T>(0, 0);
  }
  // Rows are assembled a node at a time -- the five rows' loads issued
  // together, ahead of the node's five elimination steps -- so a node waits
  // on memory once rather than once per row.  The arriving row (s, TT)
  // eliminates pivot (s-1, TT): same row type, one node back; with s = 1 the
  // pivots are the dummy leading rows.
  C_t<T> rw[5][6], rr[5];
  auto assemble = [&](auto tt, int s) {
    constexpr int TT = decltype(tt)::value;
    constexpr int C = (TT == 0) ? D : (TT <= 2 ? A : B);
    fused_row<T, D, TT, C, false, true>(L, u, f, cells, G, wmu, ta, tb, s, 5 * (s - 1) + TT, ss,
                                        rw[TT], rr[TT]);
  };
  auto arrive = [&](auto tt, int s) {
    constexpr int TT = decltype(tt)::value;
#pragma unroll
    for (int j = 0; j < 6; j++) W[WI(5, j)] = rw[TT][j];
    y[5] = rr[TT];
    const C_t<T> z = fused_eliminate<T>(W, y, lr, ls);
    if (s >= 2) {
      const int p = 5 * (s - 2) + TT;
      zr[line_slot<D, TT>(L.n, L.S, ta, tb, s - 1)] = z;
      over |= ls.put((long)p * g.nl + l, lr);
    }
  };
  // trailing steps: identity rows flush pivots (s, TT) of the last rows
  auto flush = [&](auto tt, int s) {
    constexpr int TT = decltype(tt)::value;
#pragma unroll
    for (int j = 0; j < 5; j++) W[WI(5, j)] = mk<T>(0, 0);
    W[WI(5, 5)] = mk<T>(1, 0);
    y[5] = mk<T>(0, 0);
    const C_t<T> z = fused_eliminate<T>(W, y, lr, ls);
    const int p = 5 * (s - 1) + TT;
    zr[line_slot<D, TT>(L.n, L.S, ta, tb, s)] = z;
    over |= ls.put((long)p * g.nl + l, lr);
  };
  using I0 = std::integral_constant<int, 0>;
  using I1 = std::integral_constant<int, 1>;
  using I2 = std::integral_constant<int, 2>;
  using I3 = std::integral_constant<int, 3>;
  using I4 = std::integral_constant<int, 4>;
  for (int s = 1; s < nd; s++) {
    assemble(I0{}, s);
    assemble(I1{}, s);
    assemble(I2{}, s);
    assemble(I3{}, s);
    assemble(I4{}, s);
    arrive(I0{}, s);
    arrive(I1{}, s);
    arrive(I2{}, s);
    arrive(I3{}, s);
    arrive(I4{}, s);
  }
  assemble(I0{}, nd);
  arrive(I0{}, nd);
  flush(I1{}, nd - 1);
  flush(I2{}, nd - 1);
  flush(I3{}, nd - 1);
  flush(I4{}, nd - 1);
  flush(I0{}, nd);
  if (over && ovf) atomicOr(ovf, 1);

  // backward: rows m-1 .. 0, i.e. (nd, 0), then (s, 4..0) for s = nd-1 .. 1
  C_t<T> xw[5];
#pragma unroll
  for (int i = 0; i < 5; i++) xw[i] = mk<T>(0, 0);
  // backward a node at a time as well: its rows' multipliers, z and u are
  // loaded together before the five substitution steps
  C_t<T> bl[5][5], bz[5], bu[5];
  long bs[5];
  auto load = [&](auto tt, int s) {
    constexpr int TT = decltype(tt)::value;
    bs[TT] = line_slot<D, TT>(L.n, L.S, ta, tb, s);
    ls.get((long)(5 * (s - 1) + TT) * g.nl + l, bl[TT]);
    bz[TT] = zr[bs[TT]];
    bu[TT] = u[bs[TT]];
  };
  auto back = [&](auto tt) {
    constexpr int TT = decltype(tt)::value;
    C_t<T> x = bz[TT];
#pragma unroll
    for (int i = 0; i < 5; i++) x = cfms<T>(x, bl[TT][i], xw[i]);
#pragma unroll
    for (int i = 4; i > 0; i--) xw[i] = xw[i - 1];
    xw[0] = x;
    u[bs[TT]] = cadd<T>(bu[TT], x);
  };
  load(I0{}, nd);
  back(I0{});
  for (int s = nd - 1; s >= 1; s--) {
    load(I4{}, s);
    load(I3{}, s);
    load(I2{}, s);
    load(I1{}, s);
    load(I0{}, s);
    back(I4{});
    back(I3{});
    back(I2{});
    back(I1{});
    back(I0{});
  }
}

// complex64: the same sweep with the lines eliminated from both ends, as the
// stored factors are (the multipliers equal theirs): a block is a warp per end
// of 32 lines.  The mirrored end hands its Schur complement of the middle rows
// over in shared memory and takes its side of the middle solution back.
// A block takes ncol colours one after the other, two bits each in `order`: one
// a launch, or all four of a level whose colours each fit one block (then
// gridDim.x = 1).
template <int D, int LF>
__global__ void __launch_bounds__(64) k_line_fused_ends(LevelView<float> L, unsigned order,
                                                        int ncol, int G, void* __restrict__ lbuf,
                                                        long lstride, int* __restrict__ ovf) {
  dep_wait();
  dep_next();
  constexpr int A = (D == 0) ? 1 : 0, B = (D == 2) ? 1 : 2;
  using LS = LineL<float, LF>;
  __shared__ float2 ex[20][32];
  __shared__ float2 xmid[6][32];
  const int rhs = blockIdx.y;
  if (L.active && !L.active[rhs]) return;
  for (int cc = 0; cc < ncol; cc++) {
    if (cc > 0) __syncthreads();  // u of the colours before
    const int pa = (int)(order >> (2 * cc)) & 1, pb = (int)(order >> (2 * cc + 1)) & 1;
    const LineGeom g = line_geom<D>(L.n, pa, pb);
    if (g.nl == 0) continue;
    const int lane = threadIdx.x & 31;
    const long l0 = blockIdx.x * 32L + lane;
    const bool live = l0 < g.nl;
    const long l = live ? l0 : g.nl - 1;
    const unsigned lq = (unsigned)l / (unsigned)g.la;
    const int ta = g.fa + 2 * (int)((unsigned)l - lq * (unsigned)g.la), tb = g.fb + 2 * (int)lq;
    const int n0 = L.n[0] + 1, n1 = L.n[1] + 1;
    const long ss[3] = {1, (long)n0, (long)n0 * n1};
    float2* u = L.u + (long)rhs * 3 * L.S;
    const float2* f = L.f + (long)rhs * 3 * L.S;
    float2* zr = L.r + (long)rhs * 3 * L.S;
    const float* __restrict__ cells = L.cells + (long)op_of(L, rhs) * 4 * L.ncell;
    const Geo<float> Gm{L.geo + (long)op_of(L, rhs) * L.gstride, L.gmax1};
    const float wmu = L.wmu[rhs];
    LS ls(static_cast<char*>(lbuf) + (long)rhs * lstride, g.m, g.nl);
    const int nd = g.nd;
    bool over = false;
    // row k of group j of an end: its slot, and its row number
    auto slot_of = [&](bool mir, int j, int k) -> long {
      const int s = mir ? nd - 1 - j : j + 1;
      const int t = k == 0 ? 0 : mir ? 5 - k : k;
      switch (t) {
        case 0: return line_slot<D, 0>(L.n, L.S, ta, tb, mir ? s + 1 : s);
        case 1: return line_slot<D, 1>(L.n, L.S, ta, tb, s);
        case 2: return line_slot<D, 2>(L.n, L.S, ta, tb, s);
        case 3: return line_slot<D, 3>(L.n, L.S, ta, tb, s);
        default: return line_slot<D, 4>(L.n, L.S, ta, tb, s);
      }
    };
    auto row_of = [&](bool mir, int j, int k) { return mir ? g.m - 1 - (5 * j + k) : 5 * j + k; };
    float2 W[21], y[6], lr[6];
#pragma unroll
    for (int i = 0; i < 21; i++) W[i] = make_float2(0.f, 0.f);
#pragma unroll
    for (int i = 0; i < 5; i++) {
      W[WI(i, i)] = make_float2(1.f, 0.f);  // dummy leading rows
      y[i] = make_float2(0.f, 0.f);
    }
    auto forward = [&](auto mir) {
      constexpr bool MIR = decltype(mir)::value;
      eliminate_end<MIR>(
          G, nd, W, y[5],
          [&](auto tt, int s, int k, float2 (&w)[6], float2& r) {
            constexpr int TT = decltype(tt)::value;
            constexpr int C = (TT == 0) ? D : (TT <= 2 ? A : B);
            fused_row<float, D, TT, C, MIR>(L, u, f, cells, Gm, wmu, ta, tb, s, 5 * (s - 1) + TT, ss,
                                            w, r);
          },
          [&](int j, int k) {
            const float2 z = fused_eliminate<float>(W, y, lr, ls);
            if (j >= 0 && live) {
              zr[slot_of(MIR, j, k)] = z;
              over |= ls.put((long)row_of(MIR, j, k) * g.nl + l, lr);
            }
          });
    };
    const bool bottom = threadIdx.x >= 32;
    if (bottom) {
      forward(std::true_type());
#pragma unroll
      for (int i = 0; i < 15; i++) ex[i][lane] = W[i];
#pragma unroll
      for (int i = 0; i < 5; i++) ex[15 + i][lane] = y[i];
    } else {
      forward(std::false_type());
    }
    __syncthreads();
    if (!bottom) {
      float2 wr[6], r5;
      fused_row<float, D, 0, D>(L, u, f, cells, Gm, wmu, ta, tb, G + 2, 5 * (G + 1), ss, wr, r5);
#pragma unroll
      for (int i = 0; i < 6; i++) W[WI(5, i)] = wr[i];
      y[5] = r5;
#pragma unroll
      for (int i = 0; i < 5; i++) {
        y[5 - i] = cadd<float>(y[5 - i], ex[15 + i][lane]);
#pragma unroll
        for (int j = 0; j <= i; j++)
          W[WI(5 - j, 5 - i)] = cadd<float>(W[WI(5 - j, 5 - i)], ex[WI(i, j)][lane]);
      }
      float2 ml[6][5], xm[6];
#pragma unroll
      for (int p = 0; p < 6; p++) {
        xm[p] = fused_eliminate<float>(W, y, lr, ls);
        over |= ls.bad(lr);
#pragma unroll
        for (int i = 0; i < 5; i++) ml[p][i] = lr[i + 1];
#pragma unroll
        for (int i = 0; i < 5; i++) W[WI(5, i)] = make_float2(0.f, 0.f);
        W[WI(5, 5)] = make_float2(1.f, 0.f);
        y[5] = make_float2(0.f, 0.f);
      }
#pragma unroll
      for (int p = 5; p >= 0; p--) {
#pragma unroll
        for (int i = 5; i >= 1; i--)
          if (p + i < 6) xm[p] = cfms<float>(xm[p], ml[p][i - 1], xm[p + i]);
        xmid[p][lane] = xm[p];
      }
      if (live) {
#pragma unroll
        for (int p = 0; p < 6; p++) {
          const long sl = p < 5 ? slot_of(false, G, p) : line_slot<D, 0>(L.n, L.S, ta, tb, G + 2);
          u[sl] = cadd<float>(u[sl], xm[p]);
        }
      }
    }
    __syncthreads();
    if (over && live && ovf) atomicOr(ovf, 1);
    float2 xw[5];
#pragma unroll
    for (int i = 0; i < 5; i++) xw[i] = xmid[bottom ? 5 - i : i][lane];
    // backward a node at a time: its rows' multipliers, z and u are loaded
    // together before the five substitution steps
    for (int j = live ? G - 1 : -1; j >= 0; j--) {
      float2 bl[5][5], bz[5], bu[5];
      long bs[5];
#pragma unroll
      for (int k = 4; k >= 0; k--) {
        bs[k] = slot_of(bottom, j, k);
        ls.get((long)row_of(bottom, j, k) * g.nl + l, bl[k]);
        bz[k] = zr[bs[k]];
        bu[k] = u[bs[k]];
      }
#pragma unroll
      for (int k = 4; k >= 0; k--) {
        float2 x = bz[k];
#pragma unroll
        for (int i = 4; i >= 0; i--) x = cfms<float>(x, bl[k][i], xw[i]);
#pragma unroll
        for (int i = 4; i > 0; i--) xw[i] = xw[i - 1];
        xw[0] = x;
        u[bs[k]] = cadd<float>(bu[k], x);
      }
    }
  }
}

// a level whose colours of lines along d each fit one block of the one-launch
// sweep takes all four in one launch
bool line_fused_block(const int n[3], int d) { return line_count(n, d, 3) <= 32; }

// complex64: ncol colours of `order` (k_line_fused_ends)
template <int D>
static void line_fused_ends(const LevelView<float>& L, unsigned order, int ncol, void* lbuf, int lf,
                            int* ovf, cudaStream_t st) {
  long nl = 0, lstride = 0;
  for (int c = 0; c < ncol; c++) {
    const int col = (int)(order >> (2 * c)) & 3;
    nl = std::max(nl, line_count(L.n, D, col));
    lstride = std::max(lstride, line_l_bytes(L.n, D, col, lf, 4));
  }
  if (nl == 0) return;
  const dim3 g((unsigned)((nl + 31) / 32), L.nrhs);
  const int G = (L.n[D] - 2) / 2;
  if (lf == kLHalf)
    launch_dep(k_line_fused_ends<D, kLHalf>, g, 64, 0, st, L, order, ncol, G, lbuf, lstride, ovf);
  else
    launch_dep(k_line_fused_ends<D, kLExact>, g, 64, 0, st, L, order, ncol, G, lbuf, lstride, ovf);
}

void launch_line_fused_block(const LevelView<float>& L, int d, bool rev, void* lbuf, int lf,
                             int* ovf, cudaStream_t st) {
  const unsigned order = rev ? 0x1b : 0xe4;  // 3 2 1 0 or 0 1 2 3
  if (d == 0) line_fused_ends<0>(L, order, 4, lbuf, lf, ovf, st);
  else if (d == 1) line_fused_ends<1>(L, order, 4, lbuf, lf, ovf, st);
  else line_fused_ends<2>(L, order, 4, lbuf, lf, ovf, st);
}

template <typename T, int D>
static void line_fused_d(const LevelView<T>& L, int color, void* lbuf, int lf, int* ovf,
                         cudaStream_t st) {
  if constexpr (std::is_same<T, float>::value) {
    line_fused_ends<D>(L, (unsigned)color, 1, lbuf, lf, ovf, st);
  } else {
    const int pa = color & 1, pb = (color >> 1) & 1;
    const long nl = line_count(L.n, D, color);
    if (nl == 0) return;
    const dim3 g((unsigned)((nl + kSolveThreads - 1) / kSolveThreads), L.nrhs);
    k_line_fused<T, D, kLExact, kSolveThreads><<<g, kSolveThreads, 0, st>>>(
        L, pa, pb, line_div<D>(L.n, pa, pb), lbuf, line_l_bytes(L.n, D, color, lf, 8), ovf);
  }
}

template <typename T>
void launch_line_fused(const LevelView<T>& L, int d, int color, void* lbuf, int lf, int* ovf,
                       cudaStream_t st) {
  if (d == 0) line_fused_d<T, 0>(L, color, lbuf, lf, ovf, st);
  else if (d == 1) line_fused_d<T, 1>(L, color, lbuf, lf, ovf, st);
  else line_fused_d<T, 2>(L, color, lbuf, lf, ovf, st);
}
template void launch_line_fused<float>(const LevelView<float>&, int, int, void*, int, int*,
                                       cudaStream_t);
template void launch_line_fused<double>(const LevelView<double>&, int, int, void*, int, int*,
                                        cudaStream_t);

}  // namespace emmi
