// The complex64 edge equations of a grid node with the coefficients from the
// mesh spacings (LevelView::imu_vol: every cell's inverse permeability is its
// volume), for the kernels that take several edges a thread.
#pragma once
#include <type_traits>

#include "emmi_kernels.cuh"

namespace emmi {

// One direction pair (X, Y) of the equation of an edge value e along C, added
// to acc: with k = d_C h_Y and h = h_Y (h the mean of the two spacings at the
// edge), edge_coef's coefficients with cell weight = volume give
//   k [(e - e(+X)) / d_X+ + (e - e(-X)) / d_X-]
//   + h [E_X(+C) - E_X - E_X(+C, -X) + E_X(-X)]
// rp, rm: 1 / d_X+, 1 / d_X-; x1, x0, x1m, x0m: the four E_X in that order.
__device__ __forceinline__ float2 edge_pair(float2 acc, float2 e, float2 ep, float2 em, float k,
                                            float rp, float rm, float h, float2 x1, float2 x0,
                                            float2 x1m, float2 x0m) {
  const float kp = k * rp, km = k * rm;
  acc.x += (kp * (e.x - ep.x) + km * (e.x - em.x)) + h * ((x1.x - x0.x) - (x1m.x - x0m.x));
  acc.y += (kp * (e.y - ep.y) + km * (e.y - em.y)) + h * ((x1.y - x0.y) - (x1m.y - x0m.y));
  return acc;
}
// f - A e of an edge: acc its curl-curl part, m = omega mu0 sbar (the mass
// term is -i m e)
__device__ __forceinline__ float2 edge_done(float2 f, float2 acc, float2 e, float m) {
  return make_float2(f.x - acc.x - m * e.y, f.y - acc.y + m * e.x);
}

// The equations of the three edges that start at node P (slot s of its
// right-hand side): r[C] = f - A u where the edge is unknown (unk[C]), f
// elsewhere; d[C] = the diagonal of an unknown edge.  The 24 edge values the
// three share, 12 conductivities and six spacings are loaded once each, all
// before the first use (edge by edge they are 39, 12 and 15).  u, f: the
// right-hand side's fields; f may be null (0).
__device__ __forceinline__ void node_residual(const LevelView<float>& L, const float2* u,
                                              const float2* f, const float* cells,
                                              const Geo<float>& G, float wmu, const int (&P)[3],
                                              int s, float2 (&r)[3], float2 (&d)[3],
                                              bool (&unk)[3]) {
  const int n0 = L.n[0], n1 = L.n[1], n2 = L.n[2];
  const int ss[3] = {1, n0 + 1, (n0 + 1) * (n1 + 1)};
  const int S = (int)L.S, nc = (int)L.ncell;
  const bool in0 = P[0] >= 1 && P[0] < n0, in1 = P[1] >= 1 && P[1] < n1,
             in2 = P[2] >= 1 && P[2] < n2;
  unk[0] = P[0] < n0 && in1 && in2;
  unk[1] = P[1] < n1 && in2 && in0;
  unk[2] = P[2] < n2 && in0 && in1;
  const float2 zero = make_float2(0.f, 0.f);
  // in an interior row of nodes every one of the values lies in the field, at
  // the ends of the row too (the neighbouring rows' memory), and what an edge
  // that is not unknown would add is dropped: no load waits for a predicate
  // per component C (with p, q the next two directions): its own value, the
  // neighbours +-p and +-q of its equation, and the values -C, (-C, +p) and
  // (-C, +q) that the equations of the p and q edges take from it
  float2 e0[3], pp[3], pm[3], qp[3], qm[3], cm[3], cmp[3], cmq[3];
  float sg[3], dm[3], dp[3];
  const int cs[3] = {1, n0, n0 * n1};
  const int co = P[0] + n0 * (P[1] + n1 * P[2]);
  auto load = [&](auto every) {
    constexpr bool all = decltype(every)::value;
#pragma unroll
    for (int c = 0; c < 3; c++) {
      const int p = (c + 1) % 3, q = (c + 2) % 3;
      const float2* uc = u + ((long)c * S + s);
      const bool uC = unk[c], up = unk[p], uq = unk[q];
      e0[c] = (all || uC || up || uq) ? uc[0] : zero;
      pp[c] = (all || uC || up) ? uc[ss[p]] : zero;
      qp[c] = (all || uC || uq) ? uc[ss[q]] : zero;
      pm[c] = (all || uC) ? uc[-ss[p]] : zero;
      qm[c] = (all || uC) ? uc[-ss[q]] : zero;
      cm[c] = (all || up || uq) ? uc[-ss[c]] : zero;
      cmp[c] = (all || up) ? uc[ss[p] - ss[c]] : zero;
      cmq[c] = (all || uq) ? uc[ss[q] - ss[c]] : zero;
      const float* g = cells + ((long)c * nc + co);
      sg[c] = (all || uC)
                  ? ((ldro(g - cs[p] - cs[q]) + ldro(g - cs[p])) + ldro(g - cs[q])) + ldro(g)
                  : 0.f;
    }
  };
  if (in1 && in2) load(std::true_type());
  else load(std::false_type());
#pragma unroll
  for (int c = 0; c < 3; c++) {
    r[c] = f ? f[(long)c * S + s] : zero;
    dp[c] = ldro(G.ds(c) + P[c]);
    dm[c] = ldro(G.ds(c) + max(P[c] - 1, 0));
  }
  float h[3], rp[3], rm[3];
#pragma unroll
  for (int c = 0; c < 3; c++) {
    h[c] = 0.5f * (dp[c] + dm[c]);
    rp[c] = qdiv(1.f, dp[c]);
    rm[c] = qdiv(1.f, dm[c]);
  }
#pragma unroll
  for (int c = 0; c < 3; c++) {
    const int p = (c + 1) % 3, q = (c + 2) % 3;
    const float m = 0.25f * wmu * sg[c];
    const float kp = dp[c] * h[q], kq = dp[c] * h[p];
    // E_p at +C is p's +q neighbour when C = q of p: (p + 2) % 3 == c
    float2 acc = edge_pair(zero, e0[c], pp[c], pm[c], kp, rp[p], rm[p], h[q], qp[p], e0[p], cmq[p],
                           cm[p]);
    acc = edge_pair(acc, e0[c], qp[c], qm[c], kq, rp[q], rm[q], h[p], pp[q], e0[q], cmp[q], cm[q]);
    if (unk[c]) r[c] = edge_done(r[c], acc, e0[c], m);
    d[c] = make_float2((kp * rp[p] + kp * rm[p]) + (kq * rp[q] + kq * rm[q]), -m);
  }
}

}  // namespace emmi
