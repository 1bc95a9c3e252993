// Line geometry, thread decode and records shared by the line relaxation's
// two translation units: emmi_kernels.cu (factoring sweeps) and emmi_lines.cu
// (stored factors, one-launch sweep).
#pragma once
#include "emmi_kernels.cuh"

namespace emmi {

// ------------------------------------------------------------ line tables
// Position of an edge on the line along d through transverse nodes (ta,tb)
// (a<b the other directions), in the reference's row order
// (src/gmg.c:413-603): node s=1..n_d-1 holds E_d(s-1), E_a(ta-1), E_a(ta),
// E_b(tb-1), E_b(tb); the last row is E_d(n_d-1).  -1 when not on the line.
__host__ __device__ constexpr int line_pos(int d, int a, int b, int ta, int tb, int nd, int comp,
                                          int p0, int p1, int p2) {
  const int P[3] = {p0, p1, p2};
  if (comp == d) return (P[a] == ta && P[b] == tb && P[d] >= 0 && P[d] < nd) ? 5 * P[d] : -1;
  if (P[d] < 1 || P[d] >= nd) return -1;
  if (comp == a)
    return (P[b] == tb && (P[a] == ta - 1 || P[a] == ta)) ? 5 * (P[d] - 1) + 1 + (P[a] - ta + 1)
                                                           : -1;
  return (P[a] == ta && (P[b] == tb - 1 || P[b] == tb)) ? 5 * (P[d] - 1) + 3 + (P[b] - tb + 1)
                                                         : -1;
}

// band offset of neighbour k of the row of type t on a line along d (127 if
// the neighbour is not on the line); evaluated on an interior row.
__host__ __device__ constexpr int line_off(int d, int t, int k) {
  const int a = (d == 0) ? 1 : 0, b = (d == 2) ? 1 : 2;
  const int s = 8, ta = 8, tb = 8, nd = 64;
  const int comp = (t == 0) ? d : (t <= 2 ? a : b);
  int P[3] = {0, 0, 0};
  P[d] = (t == 0) ? s - 1 : s;
  P[a] = ta - (t == 1 ? 1 : 0);
  P[b] = tb - (t == 3 ? 1 : 0);
  const int row = 5 * (s - 1) + t;
  const NbrOff o = nbr_off(comp, k);
  const int p = (comp + 1) % 3, q = (comp + 2) % 3;
  int Q[3] = {P[0], P[1], P[2]};
  Q[comp] += o.dc;
  Q[p] += o.dp;
  Q[q] += o.dq;
  const int pos = line_pos(d, a, b, ta, tb, nd, o.comp, Q[0], Q[1], Q[2]);
  return pos < 0 ? 127 : pos - row;
}

// lower-triangle index of an elimination window
#define WI(i, j) ((i) * ((i) + 1) / 2 + (j))
constexpr int kRec = 12;

__device__ __forceinline__ float4 pack16(const float* v) { return make_float4(v[0], v[1], v[2], v[3]); }
__device__ __forceinline__ double2 pack16(const double* v) { return make_double2(v[0], v[1]); }
__device__ __forceinline__ void unpack16(const float4& w, float* v) {
  v[0] = w.x; v[1] = w.y; v[2] = w.z; v[3] = w.w;
}
__device__ __forceinline__ void unpack16(const double2& w, double* v) { v[0] = w.x; v[1] = w.y; }

template <typename T> struct Vec16 { using V = float4; };
template <> struct Vec16<double> { using V = double2; };
template <typename T> constexpr int kLanes = 16 / (int)sizeof(T);
template <typename T> constexpr int kPlanes = kRec / kLanes<T>;

// p: plane 0 of one (row, line); ps: distance between planes (= lines)
template <typename T>
__device__ __forceinline__ void rec_put(typename Vec16<T>::V* p, long ps, const T (&v)[kRec]) {
#pragma unroll
  for (int q = 0; q < kPlanes<T>; q++) p[q * ps] = pack16(v + q * kLanes<T>);
}
// values [10,11] (z or x) live in the last plane for both types
template <typename T>
__device__ __forceinline__ C_t<T> rec_get_x(const typename Vec16<T>::V* p, long ps) {
  T v[kLanes<T>];
  unpack16(p[(kPlanes<T> - 1) * ps], v);
  return mk<T>(v[kLanes<T> - 2], v[kLanes<T> - 1]);
}
struct LineGeom {
  int la, lb, fa, fb;  // lines per transverse direction and first index
  long nl;             // lines of the colour
  int nd, m;           // nodes along the line, rows
};

template <int D>
__host__ __device__ __forceinline__ LineGeom line_geom(const int n[3], int pa, int pb) {
  constexpr int A = (D == 0) ? 1 : 0, B = (D == 2) ? 1 : 2;
  LineGeom g;
  g.fa = pa ? 1 : 2;
  g.fb = pb ? 1 : 2;
  g.la = (n[A] - 1 >= g.fa) ? (n[A] - 1 - g.fa) / 2 + 1 : 0;
  g.lb = (n[B] - 1 >= g.fb) ? (n[B] - 1 - g.fb) / 2 + 1 : 0;
  g.nl = (long)g.la * g.lb;
  g.nd = n[D];
  g.m = 5 * n[D] - 4;
  return g;
}

// work item -> (line, node s); threads along memory-contiguous direction
template <int D>
__device__ __forceinline__ bool line_item(const LineGeom& g, long id, long& l, int& s) {
  if (id >= g.nl * g.nd) return false;
  if (D == 0) {  // rows of an x-line are contiguous in memory
    const unsigned u = (unsigned)id, nd = (unsigned)g.nd;
    l = u / nd;
    s = 1 + (int)(u - (unsigned)l * nd);
  } else {  // neighbouring lines (consecutive i) are contiguous
    const unsigned u = (unsigned)id, nl = (unsigned)g.nl;
    const unsigned q = u / nl;
    l = u - q * nl;
    s = 1 + (int)q;
  }
  return true;
}

// the divisors of a colour's thread decode (one launch): rows x items
// (x-line residual), the item-per-line divisor of line_item and the lines
// per transverse direction
struct LineDiv {
  unsigned items;
  FastDiv rows, item, la;
};
template <int D>
LineDiv line_div(const int n[3], int pa, int pb) {
  const LineGeom g = line_geom<D>(n, pa, pb);
  LineDiv v;
  v.items = (unsigned)(g.nl * g.nd);
  v.rows = make_fastdiv(v.items > 0 ? v.items : 1);
  v.item = make_fastdiv((unsigned)(D == 0 ? g.nd : (g.nl > 0 ? g.nl : 1)));
  v.la = make_fastdiv((unsigned)(g.la > 0 ? g.la : 1));
  return v;
}
// line_item with the launch's divisor
template <int D>
__device__ __forceinline__ bool line_item_fd(const LineGeom& g, const LineDiv& v, unsigned id,
                                             long& l, int& s) {
  if (id >= v.items) return false;
  const unsigned q = fdiv(id, v.item);
  if (D == 0) {  // rows of an x-line are contiguous in memory
    l = q;
    s = 1 + (int)(id - q * (unsigned)g.nd);
  } else {  // neighbouring lines (consecutive i) are contiguous
    l = id - q * (unsigned)g.nl;
    s = 1 + (int)q;
  }
  return true;
}

template <int D, int TT>
__device__ __forceinline__ long line_slot(const int n[3], long S, int ta, int tb, int s) {
  constexpr int A = (D == 0) ? 1 : 0, B = (D == 2) ? 1 : 2;
  constexpr int C = (TT == 0) ? D : (TT <= 2 ? A : B);
  int P[3];
  P[D] = (TT == 0) ? s - 1 : s;
  P[A] = ta - (TT == 1 ? 1 : 0);
  P[B] = tb - (TT == 3 ? 1 : 0);
  return (long)C * S + slot_id(n, P[0], P[1], P[2]);
}

// rows of a thread's private cp.async ring in the one-ended solves, and their
// threads per block
constexpr int kRing = 6;
constexpr int kSolveThreads = 64;

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() {
  asm volatile("cp.async.commit_group;\n" ::: "memory");
}
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}
__device__ __forceinline__ void cp_async8(void* smem, const void* gmem) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(sa), "l"(gmem) : "memory");
}
template <typename T>
__device__ __forceinline__ void cp_async_c(C_t<T>* smem, const C_t<T>* gmem) {
  if constexpr (sizeof(C_t<T>) == 8) cp_async8(smem, gmem);
  else cp_async16(smem, gmem);
}

}  // namespace emmi
