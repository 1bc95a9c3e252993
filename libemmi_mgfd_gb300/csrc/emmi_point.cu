// Node-patch relaxation (src/gmg.c:116-336): the coarsest level's smoother, and
// every level's without semi-coarsening.  8 colours of patches of the six
// edges at a node, each patch solved with the current residual of its rows.
#include <algorithm>

#include "emmi_line.cuh"

namespace emmi {

// ------------------------------------------------------------ point sweep
// row (C, side): side 0 = E_C(N - e_C), side 1 = E_C(N); patch index 2C+side.
// its entries of the patch matrix (lower triangle)
template <typename T, int C, int SIDE>
__device__ __forceinline__ void patch_entries(const EdgeCoef<T>& e, C_t<T> (&M)[21]) {
  constexpr int p = Cyc<C>::p, q = Cyc<C>::q;
  constexpr int ri = 2 * C + SIDE;
  M[WI(ri, ri)] = mk<T>(e.dre, e.dim);
  // in-patch neighbours: side 0 -> k=4 (p,1), 6 (p,0), 8 (q,1), 10 (q,0);
  //                      side 1 -> k=5, 7, 9, 11
  constexpr int kp1 = SIDE ? 5 : 4, kp0 = SIDE ? 7 : 6, kq1 = SIDE ? 9 : 8, kq0 = SIDE ? 11 : 10;
  constexpr int ip1 = 2 * p + 1, ip0 = 2 * p, iq1 = 2 * q + 1, iq0 = 2 * q;
  if constexpr (ip1 < ri) M[WI(ri, ip1)] = mk<T>(e.c[kp1], 0);
  if constexpr (ip0 < ri) M[WI(ri, ip0)] = mk<T>(e.c[kp0], 0);
  if constexpr (iq1 < ri) M[WI(ri, iq1)] = mk<T>(e.c[kq1], 0);
  if constexpr (iq0 < ri) M[WI(ri, iq0)] = mk<T>(e.c[kq0], 0);
}

// the row of the current residual
template <typename T, int C, int SIDE>
__device__ __forceinline__ void patch_row(const LevelView<T>& L, const C_t<T>* u, const C_t<T>* f,
                                          const T* cells, const Geo<T>& G, T wmu, const int N[3],
                                          const long ss[3], C_t<T> (&M)[21], C_t<T> (&y)[6]) {
  constexpr int ri = 2 * C + SIDE;
  int P[3] = {N[0], N[1], N[2]};
  P[C] -= 1 - SIDE;
  const long sl = slot_id(L.n, P[0], P[1], P[2]);
  EdgeCoef<T> e;
  const C_t<T> au = apply_row<T, C>(L, u, cells, G, wmu, P, sl, ss, e);
  y[ri] = csub<T>(f[(long)C * L.S + sl], au);
  patch_entries<T, C, SIDE>(e, M);
}

template <typename T>
__global__ void __launch_bounds__(128) k_point_sweep(LevelView<T> L, int color) {
  dep_wait();
  dep_next();
  const int rhs = blockIdx.y;
  if (L.active && !L.active[rhs]) return;
  int cnt[3], first[3];
#pragma unroll
  for (int e = 0; e < 3; e++) {
    const int par = (color >> e) & 1;
    first[e] = par ? 1 : 2;
    cnt[e] = (L.n[e] - 1 >= first[e]) ? (L.n[e] - 1 - first[e]) / 2 + 1 : 0;
  }
  const long tot = (long)cnt[0] * cnt[1] * cnt[2];
  const long id = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (id >= tot) return;
  const int N[3] = {first[0] + 2 * (int)(id % cnt[0]), first[1] + 2 * (int)((id / cnt[0]) % cnt[1]),
                    first[2] + 2 * (int)(id / ((long)cnt[0] * cnt[1]))};
  const int n0 = L.n[0] + 1, n1 = L.n[1] + 1;
  const long ss[3] = {1, (long)n0, (long)n0 * n1};
  C_t<T>* u = L.u + (long)rhs * 3 * L.S;
  const C_t<T>* f = L.f + (long)rhs * 3 * L.S;
  const T* cells = L.cells + (long)op_of(L, rhs) * 4 * L.ncell;
  const Geo<T> G{L.geo + (long)op_of(L, rhs) * L.gstride, L.gmax1};
  const T wmu = L.wmu[rhs];
  C_t<T> M[21], y[6];
#pragma unroll
  for (int i = 0; i < 21; i++) M[i] = mk<T>(0, 0);
  patch_row<T, 0, 0>(L, u, f, cells, G, wmu, N, ss, M, y);
  patch_row<T, 0, 1>(L, u, f, cells, G, wmu, N, ss, M, y);
  patch_row<T, 1, 0>(L, u, f, cells, G, wmu, N, ss, M, y);
  patch_row<T, 1, 1>(L, u, f, cells, G, wmu, N, ss, M, y);
  patch_row<T, 2, 0>(L, u, f, cells, G, wmu, N, ss, M, y);
  patch_row<T, 2, 1>(L, u, f, cells, G, wmu, N, ss, M, y);
  // dense complex-symmetric LDL^T on the lower triangle
  C_t<T> Lm[21], z[6];
#pragma unroll
  for (int k = 0; k < 6; k++) {
    const C_t<T> id = crcp<T>(M[WI(k, k)]);
#pragma unroll
    for (int i = k + 1; i < 6; i++) {
      const C_t<T> l = cmul<T>(M[WI(i, k)], id);
#pragma unroll
      for (int j = k + 1; j <= i; j++) M[WI(i, j)] = cfms<T>(M[WI(i, j)], l, M[WI(j, k)]);
      y[i] = cfms<T>(y[i], l, y[k]);
      Lm[WI(i, k)] = l;
    }
    z[k] = cmul<T>(y[k], id);
  }
#pragma unroll
  for (int k = 5; k >= 0; k--) {
#pragma unroll
    for (int i = k + 1; i < 6; i++) z[k] = cfms<T>(z[k], Lm[WI(i, k)], z[i]);
  }
#pragma unroll
  for (int ri = 0; ri < 6; ri++) {
    const int c = ri / 2;
    int P[3] = {N[0], N[1], N[2]};
    P[c] -= 1 - (ri & 1);
    const long sl = (long)c * L.S + slot_id(L.n, P[0], P[1], P[2]);
    u[sl] = cadd<T>(u[sl], z[ri]);
  }
}

template <typename T>
void launch_point_sweep(const LevelView<T>& L, int color, cudaStream_t st) {
  long cnt = 1;
  for (int e = 0; e < 3; e++) {
    const int par = (color >> e) & 1, first = par ? 1 : 2;
    cnt *= (L.n[e] - 1 >= first) ? (L.n[e] - 1 - first) / 2 + 1 : 0;
  }
  if (cnt == 0) return;
  dim3 grid((unsigned)((cnt + 127) / 128), L.nrhs);
  launch_dep(k_point_sweep<T>, grid, 128, 0, st, L, color);
}

// ---------------------------------------------------------------- coarsest level
// The coarsest level's node-patch sweeps in one launch: a block per right-hand
// side holds u and f in shared memory and goes through the colours of all its
// sweeps, one barrier a colour.  What a patch needs of the operator is stored
// at set-up: the ten coefficients of every edge (planes [op][10][3][S]:
// c0..c3, c4, c7, c8, c11, the real diagonal and sbar) and the LDL^T factors
// of every patch (planes [group][21][patch] in lower-triangle order, 1/d on
// the diagonal).  Six lanes take a patch, one row each: the residual of the
// row, forward substitution with the other rows' values by shuffle, back
// substitution with the products formed in their lanes and subtracted in
// k_point_sweep's order.  The operations and their order are k_point_sweep's:
// the same result, bit for bit.
//
// Level of a block: one whose u and f fit its shared memory and whose largest
// colour is one round of its 16 warps (80 patches; 224 of them took 48.4 ms a
// solve of six RHS at 80 x 56 x 72 where launches by colour, k_point_lanes,
// take 44.6); larger levels take a launch a colour.
//
// What this saves.  complex64: 16 launches a visit and a visit for every level
// of an F-cycle (64 of a 16^3 cycle's 270 launches); one visit of that level
// 16 x 10.2 -> 14.9 us.  complex128: an FP64 instruction of a warp takes an SM
// quarter about 60 clocks whatever its lanes do, so one thread a patch took
// 70 us a launch; one visit 16 x 70 -> 31 us.
constexpr int kPtCoef = 10;

// cfms and cmul as the compiler contracts them in k_point_sweep
template <typename T> __device__ __forceinline__ C_t<T> pt_cfms(C_t<T> a, C_t<T> b, C_t<T> c) {
  const C_t<T> t = cprod_sub<T>(b, c);
  return mk<T>(rsub(a.x, t.x), rsub(a.y, t.y));
}
template <typename T> __device__ __forceinline__ C_t<T> pt_cmul(C_t<T> a, C_t<T> b) {
  return mk<T>(rfma(a.x, b.x, -rmul(a.y, b.y)), rfma(a.x, b.y, rmul(a.y, b.x)));
}

template <typename T, int C>
__device__ __forceinline__ void pt_store_coef(const LevelView<T>& L, const T* cells,
                                              const Geo<T>& G, const int P[3], long s, T* out) {
  EdgeCoef<T> e;
  // omega*mu0 = -1 gives dim = sbar exactly
  edge_coef<T, C>(L.n, P, cells + (long)C * L.ncell, cells + 3 * L.ncell, G, T(-1), e, L.imu_vol);
  const long n3s = 3 * L.S, o = (long)C * L.S + s;
  const T v[kPtCoef] = {e.c[0], e.c[1], e.c[2], e.c[3], e.c[4],
                        e.c[7], e.c[8], e.c[11], e.dre, e.dim};
#pragma unroll
  for (int k = 0; k < kPtCoef; k++) out[k * n3s + o] = v[k];
}

// blockIdx.y = operator
template <typename T>
__global__ void __launch_bounds__(128) k_point_coef(LevelView<T> L, T* __restrict__ coef) {
  const int op = blockIdx.y;
  const long s = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (s >= L.S) return;
  int P[3];
  slot_nodes(s, L, P);
  const T* cells = L.cells + (long)op * 4 * L.ncell;
  const Geo<T> G{L.geo + (long)op * L.gstride, L.gmax1};
  T* out = coef + (long)op * kPtCoef * 3 * L.S;
  const bool i0 = P[0] >= 1 && P[0] < L.n[0], i1 = P[1] >= 1 && P[1] < L.n[1],
             i2 = P[2] >= 1 && P[2] < L.n[2];
  if (P[0] < L.n[0] && i1 && i2) pt_store_coef<T, 0>(L, cells, G, P, s, out);
  if (P[1] < L.n[1] && i2 && i0) pt_store_coef<T, 1>(L, cells, G, P, s, out);
  if (P[2] < L.n[2] && i0 && i1) pt_store_coef<T, 2>(L, cells, G, P, s, out);
}

// a patch's interior node <-> its number
__host__ __device__ inline long pt_patches(const int n[3]) {
  return (long)(n[0] - 1) * (n[1] - 1) * (n[2] - 1);
}

template <typename T, int C, int SIDE>
__device__ __forceinline__ void pt_matrix_row(const LevelView<T>& L, const T* cells,
                                              const Geo<T>& G, T wmu, const int N[3],
                                              C_t<T> (&M)[21]) {
  int P[3] = {N[0], N[1], N[2]};
  P[C] -= 1 - SIDE;
  EdgeCoef<T> e;
  // omega*mu0 = -1 gives dim = sbar exactly; the mass term's product stays out
  // of the elimination's multiply-adds, as it does in k_point_sweep
  edge_coef<T, C>(L.n, P, cells + (long)C * L.ncell, cells + 3 * L.ncell, G, T(-1), e, L.imu_vol);
  e.dim = rmul(-wmu, e.dim);
  patch_entries<T, C, SIDE>(e, M);
}

// factors of every patch for group blockIdx.y (its operator L.op, L.wmu)
template <typename T>
__global__ void __launch_bounds__(64) k_point_factor(LevelView<T> L, C_t<T>* __restrict__ pf) {
  const int grp = blockIdx.y;
  const long np = pt_patches(L.n);
  const long id = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (id >= np) return;
  const int a = L.n[0] - 1, b = L.n[1] - 1;
  const int N[3] = {1 + (int)(id % a), 1 + (int)((id / a) % b), 1 + (int)(id / ((long)a * b))};
  const T* cells = L.cells + (long)op_of(L, grp) * 4 * L.ncell;
  const Geo<T> G{L.geo + (long)op_of(L, grp) * L.gstride, L.gmax1};
  const T wmu = L.wmu[grp];
  C_t<T> M[21];
#pragma unroll
  for (int i = 0; i < 21; i++) M[i] = mk<T>(0, 0);
  pt_matrix_row<T, 0, 0>(L, cells, G, wmu, N, M);
  pt_matrix_row<T, 0, 1>(L, cells, G, wmu, N, M);
  pt_matrix_row<T, 1, 0>(L, cells, G, wmu, N, M);
  pt_matrix_row<T, 1, 1>(L, cells, G, wmu, N, M);
  pt_matrix_row<T, 2, 0>(L, cells, G, wmu, N, M);
  pt_matrix_row<T, 2, 1>(L, cells, G, wmu, N, M);
  C_t<T>* out = pf + (long)grp * 21 * np + id;
#pragma unroll
  for (int k = 0; k < 6; k++) {
    const C_t<T> idg = crcp<T>(M[WI(k, k)]);
#pragma unroll
    for (int i = k + 1; i < 6; i++) {
      const C_t<T> l = cmul<T>(M[WI(i, k)], idg);
#pragma unroll
      for (int j = k + 1; j <= i; j++) M[WI(i, j)] = cfms<T>(M[WI(i, j)], l, M[WI(j, k)]);
      out[WI(i, k) * np] = l;
    }
    out[WI(k, k) * np] = idg;
  }
}

template <typename T>
__device__ __forceinline__ C_t<T> shfl_c(C_t<T> v, int src) {
  return mk<T>(__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src));
}

// the patches of a colour, warps first, first + step, .. of five patches each
template <typename T>
__device__ __forceinline__ void patch_lanes(const LevelView<T>& L, int color, C_t<T>* u,
                                            const C_t<T>* f, const T* __restrict__ cf,
                                            const C_t<T>* __restrict__ fac, T wmu, int first,
                                            int step) {
  const int S = (int)L.S, n3s = 3 * S;
  const int lane = threadIdx.x & 31;
  const int base = lane / 6 * 6, ri = lane - base, C = ri >> 1;
  const int s1 = L.n[0] + 1, s2 = s1 * (L.n[1] + 1);
  // strides and components along (C, p, q), the row's edge relative to its node
  const int sC = C == 0 ? 1 : C == 1 ? s1 : s2;
  const int sp = C == 0 ? s1 : C == 1 ? s2 : 1, sq = C == 0 ? s2 : C == 1 ? 1 : s1;
  const int cp = (C == 2 ? 0 : C + 1) * S, cq = (C == 0 ? 2 : C - 1) * S;
  const int edge = C * S - ((ri & 1) ? 0 : sC);
  const int f0 = color & 1 ? 1 : 2, f1 = color & 2 ? 1 : 2, f2 = color & 4 ? 1 : 2;
  const int c0 = L.n[0] - 1 >= f0 ? (L.n[0] - 1 - f0) / 2 + 1 : 0;
  const int c1 = L.n[1] - 1 >= f1 ? (L.n[1] - 1 - f1) / 2 + 1 : 0;
  const int c2 = L.n[2] - 1 >= f2 ? (L.n[2] - 1 - f2) / 2 + 1 : 0;
  const int cnt = c0 * c1 * c2;
  const long np = pt_patches(L.n);
  for (int w0 = first * 5; w0 < cnt; w0 += step * 5) {
    const int pt = w0 + lane / 6;
    const bool live = lane < 30 && pt < cnt;
    const int q = live ? pt : w0;
    const int i = f0 + 2 * (q % c0), j = f1 + 2 * ((q / c0) % c1), k = f2 + 2 * (q / (c0 * c1));
    const int sl = edge + i + s1 * j + s2 * k;  // this row's edge
    const long pid = (i - 1) + (long)(L.n[0] - 1) * ((j - 1) + (long)(L.n[1] - 1) * (k - 1));
    C_t<T> Lr[6];
#pragma unroll
    for (int c = 0; c < 6; c++)
      Lr[c] = c <= ri ? fac[(ri * (ri + 1) / 2 + c) * np + pid] : mk<T>(0, 0);
    T kk[kPtCoef];
#pragma unroll
    for (int c = 0; c < kPtCoef; c++) kk[c] = ldro(cf + (long)c * n3s + sl);
    const T c12[12] = {kk[0], kk[1], kk[2], kk[3], kk[4], -kk[4], -kk[5], kk[5],
                       kk[6], -kk[6], -kk[7], kk[7]};
    const int node = sl - C * S;  // slot of the edge within a component
    const int at[12] = {sl + sp, sl - sp, sl + sq, sl - sq,
                        cp + node + sC, cp + node, cp + node + sC - sp, cp + node - sp,
                        cq + node + sC, cq + node, cq + node + sC - sq, cq + node - sq};
    const T dre = kk[8], dim = -wmu * kk[9];
    const C_t<T> uc = u[sl];
    T ar = rfma(dre, uc.x, -rmul(dim, uc.y));
    T ai = rfma(dre, uc.y, rmul(dim, uc.x));
#pragma unroll
    for (int c = 0; c < 12; c++) {
      const C_t<T> v = u[at[c]];
      ar = rfma(c12[c], v.x, ar);
      ai = rfma(c12[c], v.y, ai);
    }
    C_t<T> y = csub<T>(f[sl], mk<T>(ar, ai));
#pragma unroll
    for (int c = 0; c < 5; c++) {  // forward: column c
      const C_t<T> yc = shfl_c<T>(y, base + c);
      if (ri > c) y = pt_cfms<T>(y, Lr[c], yc);
    }
    C_t<T> idg = Lr[0];
#pragma unroll
    for (int c = 1; c < 6; c++)
      if (ri == c) idg = Lr[c];
    C_t<T> z = pt_cmul<T>(y, idg);
#pragma unroll
    for (int c = 4; c >= 0; c--) {  // backward: row c from the rows after it
      const C_t<T> t = cprod_sub<T>(Lr[c], z);
#pragma unroll
      for (int i2 = c + 1; i2 < 6; i2++) {
        const C_t<T> ti = shfl_c<T>(t, base + i2);
        if (ri == c) z = csub<T>(z, ti);
      }
    }
    if (live) u[sl] = cadd<T>(uc, z);
  }
}

// nrep sweeps; bit r of rev: sweep r takes the colours backwards; zero: u
// starts from 0 instead of L.u
template <typename T>
__global__ void __launch_bounds__(512) k_point_coarse(LevelView<T> L, const T* __restrict__ coef,
                                                      const C_t<T>* __restrict__ pf,
                                                      const int* __restrict__ grp, int nrep,
                                                      unsigned rev, int zero) {
  dep_wait();
  dep_next();
  extern __shared__ __align__(16) unsigned char pt_sm[];
  const int rhs = blockIdx.x;
  if (L.active && !L.active[rhs]) return;
  const int n3s = 3 * (int)L.S;
  C_t<T>* u = reinterpret_cast<C_t<T>*>(pt_sm);
  C_t<T>* f = u + n3s;
  C_t<T>* gu = L.u + (long)rhs * n3s;
  const C_t<T>* gf = L.f + (long)rhs * n3s;
  for (int i = threadIdx.x; i < n3s; i += blockDim.x) {
    u[i] = zero ? mk<T>(0, 0) : gu[i];
    f[i] = gf[i];
  }
  const T* cf = coef + (long)op_of(L, rhs) * kPtCoef * n3s;
  const C_t<T>* fac = pf + (long)grp[rhs] * 21 * pt_patches(L.n);
  const T wmu = L.wmu[rhs];
  for (int rep = 0; rep < nrep; rep++)
    for (int cc = 0; cc < 8; cc++) {
      __syncthreads();  // u of the colours before
      patch_lanes<T>(L, (rev >> rep) & 1 ? 7 - cc : cc, u, f, cf, fac, wmu, threadIdx.x >> 5,
                     blockDim.x >> 5);
    }
  __syncthreads();
  for (int i = threadIdx.x; i < n3s; i += blockDim.x) gu[i] = u[i];
}

// one colour over the grid, where the level is too large for a block
template <typename T>
__global__ void __launch_bounds__(128) k_point_lanes(LevelView<T> L, int color,
                                                     const T* __restrict__ coef,
                                                     const C_t<T>* __restrict__ pf,
                                                     const int* __restrict__ grp) {
  dep_wait();
  dep_next();
  const int rhs = blockIdx.y;
  if (L.active && !L.active[rhs]) return;
  const long n3s = 3 * L.S;
  patch_lanes<T>(L, color, L.u + rhs * n3s, L.f + rhs * n3s,
                 coef + (long)op_of(L, rhs) * kPtCoef * n3s,
                 pf + (long)grp[rhs] * 21 * pt_patches(L.n), L.wmu[rhs],
                 blockIdx.x * 4 + (threadIdx.x >> 5), gridDim.x * 4);
}

// patches of the largest colour
static long point_colour(const int n[3]) {
  long most = 1;
  for (int e = 0; e < 3; e++) most *= n[e] / 2;
  return most;
}
bool point_in_block(const int n[3], int csize) {
  return point_coarse_smem(n, csize) <= (size_t)kPointSmem && point_colour(n) <= 80;
}
size_t point_coarse_smem(const int n[3], int csize) {
  return (size_t)6 * (n[0] + 1) * (n[1] + 1) * (n[2] + 1) * csize;
}
long point_coef_elems(const int n[3]) {
  return (long)kPtCoef * 3 * (n[0] + 1) * (n[1] + 1) * (n[2] + 1);
}
long point_factor_elems(const int n[3]) { return 21 * pt_patches(n); }

template <typename T>
void launch_point_setup(const LevelView<T>& ops, T* coef, const LevelView<T>& groups, C_t<T>* pf,
                        cudaStream_t st) {
  k_point_coef<T><<<dim3((unsigned)((ops.S + 127) / 128), ops.nrhs), 128, 0, st>>>(ops, coef);
  const long np = pt_patches(groups.n);
  k_point_factor<T><<<dim3((unsigned)((np + 63) / 64), groups.nrhs), 64, 0, st>>>(groups, pf);
}

template <typename T>
void launch_point_coarse(const LevelView<T>& L, const T* coef, const C_t<T>* pf, const int* grp,
                         int nrep, unsigned rev, bool zero, cudaStream_t st) {
  static DeviceOnce once;
  once_on_device(once, [] {
    cudaFuncSetAttribute(k_point_coarse<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         kPointSmem);
  });
  // five patches a warp, up to 16 warps
  const int warps = (int)std::min<long>(16, (point_colour(L.n) + 4) / 5);
  launch_dep(k_point_coarse<T>, dim3(L.nrhs), dim3(32 * warps),
             point_coarse_smem(L.n, (int)sizeof(C_t<T>)), st, L, coef, pf, grp, nrep, rev,
             zero ? 1 : 0);
}

template <typename T>
void launch_point_lanes(const LevelView<T>& L, int color, const T* coef, const C_t<T>* pf,
                        const int* grp, cudaStream_t st) {
  long cnt = 1;
  for (int e = 0; e < 3; e++) {
    const int first = (color >> e) & 1 ? 1 : 2;
    cnt *= (L.n[e] - 1 >= first) ? (L.n[e] - 1 - first) / 2 + 1 : 0;
  }
  if (cnt == 0) return;
  launch_dep(k_point_lanes<T>, dim3((unsigned)((cnt + 19) / 20), L.nrhs), dim3(128), 0, st, L,
             color, coef, pf, grp);
}

#define EMMI_POINT(T)                                                                            \
  template void launch_point_sweep<T>(const LevelView<T>&, int, cudaStream_t);                   \
  template void launch_point_setup<T>(const LevelView<T>&, T*, const LevelView<T>&, C_t<T>*,     \
                                      cudaStream_t);                                             \
  template void launch_point_coarse<T>(const LevelView<T>&, const T*, const C_t<T>*, const int*, \
                                       int, unsigned, bool, cudaStream_t);                       \
  template void launch_point_lanes<T>(const LevelView<T>&, int, const T*, const C_t<T>*,         \
                                      const int*, cudaStream_t);
EMMI_POINT(float)
EMMI_POINT(double)

}  // namespace emmi
