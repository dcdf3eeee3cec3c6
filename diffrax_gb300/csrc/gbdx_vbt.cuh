// gbdx_vbt.cuh -- device virtual Brownian tree (BrownianIncrement, and
// SpaceTimeLevyArea in vbt_levy_pair).
//
// W(t) on [vbt_t0, vbt_t0 + T] by binary bridge descent from a counter-based
// generator, as VirtualBrownianTree._evaluate_leaf (diffrax/_brownian/
// tree.py:366-448, 607-621) with the midpoint rule of _brownian_arch
// (:752-768).  Jax's threefry key splitting is replaced by Philox4x32-10
// counters (trajectory, tree node, draw kind, dimension quad): every node has
// its own independent normals, as in the reference.  The FP64 oracle uses the
// same integer stream.
#pragma once

#include <stdint.h>

#include "gbdx_common.cuh"
#include "gbdx_f2.cuh"

namespace gbdx {

__device__ __forceinline__ void philox4x32_10(uint32_t (&c)[4], uint32_t k0, uint32_t k1) {
#pragma unroll
  for (int r = 0; r < 10; r++) {
    const uint32_t lo0 = 0xD2511F53u * c[0], hi0 = __umulhi(0xD2511F53u, c[0]);
    const uint32_t lo1 = 0xCD9E8D57u * c[2], hi1 = __umulhi(0xCD9E8D57u, c[2]);
    const uint32_t n0 = hi1 ^ c[1] ^ k0, n2 = hi0 ^ c[3] ^ k1;
    c[0] = n0;
    c[1] = lo1;
    c[2] = n2;
    c[3] = lo0;
    k0 += 0x9E3779B9u;
    k1 += 0xBB67AE85u;
  }
}

enum { kVbtRoot = 0, kVbtMid = 1, kVbtLeaf = 2, kVbtRootH = 3, kVbtMidH = 4, kVbtLeafH = 5 };

// Two Box--Muller pairs from 24-bit uniforms: u = ((ua >> 8) + 1/2) 2^-24 and v
// alike give (sqrt(-2 log u) cos 2 pi v, sqrt(-2 log u) sin 2 pi v) in z[0], z[1];
// ub, vb in z[2], z[3].  A draw costs as much as the rest of the descent, so the
// functions are spelled out on the packed FP32x2 pipe: log as e ln 2 + log1p(f), u
// = (1 + f) 2^e with 1 + f in [sqrt 1/2, sqrt 2) and a minimax fit (6e-9 relative);
// cos and sin of pi/2 r, r the distance of 4 v from its quadrant (fits 1e-8, 4e-8
// relative, most of the latter the FP32 rounding of pi/2; v needs no other reduction).
// A third of the issue slots of logf, sqrtf and sincospif.  Error against FP64: rms
// 4.8e-8 (theirs 4.4e-8), at most 6.9e-7 (5.9e-7); sums over a tree's levels round by as
// much, and solves come out as far from 64 bits as with the library's functions (the
// Ornstein--Uhlenbeck paths 2.1e-7, the neural SDE's 3.9e-7).  A sine with pi/2 in two
// parts and a rounded root (rms 4.5e-8) cost those solves 7 and 3 %.
__device__ __forceinline__ void box_muller2(uint32_t ua, uint32_t va, uint32_t ub, uint32_t vb,
                                            float (&z)[4]) {
  // (k + 1/2) 2^-24 = (2 k + 1) 2^-25, one rounding
  const F2 u = f2_mul(f2_pack(float((ua >> 7) | 1u), float((ub >> 7) | 1u)),
                      f2_set(0x1p-25f));
  const F2 q = f2_mul(f2_pack(float((va >> 7) | 1u), float((vb >> 7) | 1u)),
                      f2_set(0x1p-23f));  // 4 v
  float u0, u1;
  f2_unpack(u, u0, u1);
  const int i0 = __float_as_int(u0), i1 = __float_as_int(u1);
  const int e0 = (i0 - 0x3f3504f3) >> 23, e1 = (i1 - 0x3f3504f3) >> 23;
  const F2 f = f2_add(f2_pack(__int_as_float(i0 - (e0 << 23)), __int_as_float(i1 - (e1 << 23))),
                      f2_set(-1.f));
  // the exponents as floats (1.5 2^23 + e is exact)
  const F2 e = f2_add(f2_pack(__int_as_float(0x4b400000 + e0), __int_as_float(0x4b400000 + e1)),
                      f2_set(-12582912.f));
  F2 p = f2_set(-0.07634474337100983f);
  p = f2_fma(p, f, f2_set(0.12761567533016205f));
  p = f2_fma(p, f, f2_set(-0.13160187005996704f));
  p = f2_fma(p, f, f2_set(0.14201758801937103f));
  p = f2_fma(p, f, f2_set(-0.16623356938362122f));
  p = f2_fma(p, f, f2_set(0.20001226663589478f));
  p = f2_fma(p, f, f2_set(-0.2500081956386566f));
  p = f2_fma(p, f, f2_set(0.3333333134651184f));
  p = f2_fma(p, f, f2_set(-0.5f));
  const F2 lg = f2_fma(e, f2_set(0.6931471824645996f), f2_fma(f2_mul(f, f), p, f));
  float l0, l1, r0, r1;
  f2_unpack(f2_mul(lg, f2_set(-2.f)), l0, l1);
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r0) : "f"(l0));
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r1) : "f"(l1));
  // quadrant and distance
  const F2 big = f2_add(q, f2_set(12582912.f));
  float b0, b1;
  f2_unpack(big, b0, b1);
  const int n0 = __float_as_int(b0), n1 = __float_as_int(b1);
  const F2 r = f2_fma(f2_add(big, f2_set(-12582912.f)), f2_set(-1.f), q), w = f2_mul(r, r);
  F2 s = f2_set(-0.004601656924933195f);
  s = f2_fma(s, w, f2_set(0.07968003302812576f));
  s = f2_fma(s, w, f2_set(-0.6459634304046631f));
  s = f2_mul(f2_fma(s, w, f2_set(1.5707963705062866f)), r);
  F2 c = f2_set(0.0009040216682478786f);
  c = f2_fma(c, w, f2_set(-0.02086028829216957f));
  c = f2_fma(c, w, f2_set(0.25366923213005066f));
  c = f2_fma(c, w, f2_set(-1.2337005138397217f));
  c = f2_fma(c, w, f2_set(1.f));
  float s0, s1, c0, c1;
  f2_unpack(f2_mul(s, f2_pack(r0, r1)), s0, s1);
  f2_unpack(f2_mul(c, f2_pack(r0, r1)), c0, c1);
  // cos: c, -s, -c, s; sin: s, c, -s, -c for quadrants 0..3
  auto turn = [](float x, int n) {
    return __int_as_float(__float_as_int(x) ^ ((n & 2) << 30));
  };
  z[0] = turn(n0 & 1 ? s0 : c0, n0 + 1);
  z[1] = turn(n0 & 1 ? c0 : s0, n0);
  z[2] = turn(n1 & 1 ? s1 : c1, n1 + 1);
  z[3] = turn(n1 & 1 ? c1 : s1, n1);
}

__device__ __forceinline__ void vbt_philox(uint64_t seed, uint32_t traj, uint32_t node,
                                           uint32_t kind, int quad, uint32_t (&c)[4]) {
  c[0] = traj;
  c[1] = node;
  c[2] = (kind << 24) | uint32_t(quad);
  c[3] = 0x5EEDu;
  philox4x32_10(c, uint32_t(seed), uint32_t(seed >> 32));
}

// Normals of dimensions (col, col + 1), col even, for one tree node.
__device__ __forceinline__ float2 vbt_normal_pair(uint64_t seed, uint32_t traj, uint32_t node,
                                                  uint32_t kind, int col) {
  uint32_t c[4];
  vbt_philox(seed, traj, node, kind, col >> 2, c);
  const bool p = col & 2;  // which Box-Muller pair of the quad
  float z[4];
  box_muller2(p ? c[2] : c[0], p ? c[3] : c[1], 0u, 0u, z);
  return make_float2(z[0], z[1]);
}

// Normals of NQ dimensions for two nodes: NQ = 4, a quad's; NQ = 2, those of pair
// `sel` of the quad.  The two nodes' draws are independent, so they overlap.
template <int NQ>
__device__ __forceinline__ void vbt_normals2(uint64_t seed, uint32_t traj, uint32_t node0,
                                             uint32_t kind0, uint32_t node1, uint32_t kind1,
                                             int quad, int sel, float (&z0)[NQ],
                                             float (&z1)[NQ]) {
  uint32_t a[4], b[4];
  vbt_philox(seed, traj, node0, kind0, quad, a);
  vbt_philox(seed, traj, node1, kind1, quad, b);
  if constexpr (NQ == 4) {
    box_muller2(a[0], a[1], a[2], a[3], z0);
    box_muller2(b[0], b[1], b[2], b[3], z1);
  } else {
    float z[4];
    box_muller2(sel ? a[2] : a[0], sel ? a[3] : a[1], sel ? b[2] : b[0], sel ? b[3] : b[1], z);
    z0[0] = z[0];
    z0[1] = z[1];
    z1[0] = z[2];
    z1[1] = z[3];
  }
}

// The bridge state of one descent path for NQ dimensions: W at the start of each
// level's dyadic interval and the increment across it.  Consecutive evaluations of
// a solve lie close together, so their paths share the upper levels; an evaluation
// re-descends only below the deepest level whose interval also contains the new
// time.
constexpr int kVbtCacheLevels = 24;
template <int NQ>
struct VbtCache {
  float ws[kVbtCacheLevels + 1][NQ], wsu[kVbtCacheLevels + 1][NQ];
  uint32_t node;   // heap index of the cached path's leaf interval
  long long traj;  // trajectory of the cached path (-1: none)
};
using VbtQuadCache = VbtCache<4>;

// sqrt(T) W_unit(r) for NQ dimensions of trajectory `traj` at time t, by the descent
// of tree.py:406-409, 607-621, 752-768: at every level the path takes the half that
// holds r (the left one at its midpoint), down to 2^-level <= tol.  The path is known
// from r alone, so the levels' normals are drawn two at a time (the leaf's with the
// last) and the short bridge recursion follows.  C (may be null): the cached path.
// Trees of at most kVbtWordLevels levels, whose path a 32-bit node holds.
// Bound: issue slots, ~96 a warp and Philox block and ~112 a pair of Box--Muller
// pairs.  The Ornstein--Uhlenbeck solve of 16384 paths and 100 steps (under one warp
// a scheduler, so the overlapped draws count most) went from 0.82 to 0.49 ms, the
// neural SDE of 32768 from 3.75 to 3.64 ms, its gradient at 9001 from 9.0 to 8.5 ms.
template <int NQ>
__device__ __forceinline__ void vbt_w(const SolveParams &P, int64_t traj, double t, int quad,
                                      int sel, VbtCache<NQ> *C, float (&w)[NQ]) {
  const float r = float((t - P.vbt_t0) * P.vbt_inv_len);
  const uint32_t tj = uint32_t(traj);
  const int L = P.vbt_levels;
  // r lies in (i 2^-L, (i + 1) 2^-L]; scaling by 2^L is exact, and from 2^24 on the
  // scaled r is an integer, the interval's end.  node: the leaf interval's; su: its
  // length, f: r's place in it over its length.
  const float x = r * __int_as_float((127 + L) << 23), su = __int_as_float((127 - L) << 23);
  const int i = max(0, min(int(ceilf(x)) - 1, (1 << L) - 1));
  const uint32_t node = (1u << L) + uint32_t(i);
  const float f = fmaxf(x < 16777216.f ? x - float(i) : 1.f, 0.f);
  float ws[NQ], wsu[NQ];
  int d = 0;
  const bool cached = C && L <= kVbtCacheLevels;
  if (cached && C->traj == (long long)traj) {
    const uint32_t x = node ^ C->node;
    d = x == 0 ? L : L - 1 - (31 - __clz(x));  // levels shared with the cached path
#pragma unroll
    for (int q = 0; q < NQ; q++) {
      ws[q] = C->ws[d][q];
      wsu[q] = C->wsu[d][q];
    }
  } else {
    float unused[NQ];
    vbt_normals2<NQ>(P.seed, tj, 0u, kVbtRoot, 0u, kVbtRoot, quad, sel, wsu, unused);
#pragma unroll
    for (int q = 0; q < NQ; q++) ws[q] = 0.f;
    if (cached) {
      C->traj = (long long)traj;
#pragma unroll
      for (int q = 0; q < NQ; q++) {
        C->ws[0][q] = 0.f;
        C->wsu[0][q] = wsu[q];
      }
    }
  }
  // one level: the halves of the interval of level l, and the one with r
  auto descend = [&](int l, const float (&z)[NQ]) {
    // sqrt(2^-l) / 2
    const float a = __int_as_float((126 - ((l + 1) >> 1)) << 23) * (l & 1 ? 1.41421354f : 1.f);
    const bool right = (node >> (L - l - 1)) & 1u;
#pragma unroll
    for (int q = 0; q < NQ; q++) {
      const float m = 0.5f * wsu[q];
      const float wst = m + a * z[q], wtu = m - a * z[q];
      if (right) ws[q] += wst;
      wsu[q] = right ? wtu : wst;
    }
    if (cached) {
#pragma unroll
      for (int q = 0; q < NQ; q++) {
        C->ws[l + 1][q] = ws[q];
        C->wsu[l + 1][q] = wsu[q];
      }
    }
  };
  float z0[NQ], z1[NQ];
  int l = d;
#pragma unroll 1
  for (; l < L; l += 2) {
    const bool leaf = l + 1 == L;
    vbt_normals2<NQ>(P.seed, tj, node >> (L - l), kVbtMid, node >> (L - l - 1),
                     leaf ? kVbtLeaf : kVbtMid, quad, sel, z0, z1);
    descend(l, z0);
    if (!leaf) descend(l + 1, z1);
  }
  if (l == L) vbt_normals2<NQ>(P.seed, tj, node, kVbtLeaf, node, kVbtLeaf, quad, sel, z1, z0);
  if (cached) C->node = node;
  float bb;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(bb) : "f"(f * fmaxf(1.f - f, 0.f) * su));
  const float sq = P.vbt_sqrt_len;
#pragma unroll
  for (int q = 0; q < NQ; q++) w[q] = sq * (ws[q] + f * wsu[q] + bb * z1[q]);
}

// The same for dimensions (col, col + 1) of a deeper tree, level by level: each takes the
// turn that r scaled to it says, and the node's number is kept modulo 2^32, as the draws
// take it.
static __device__ __noinline__ float2 vbt_w_deep(const SolveParams &P, int64_t traj, double t,
                                                 int col) {
  const uint32_t tj = uint32_t(traj);
  const float2 z0 = vbt_normal_pair(P.seed, tj, 0u, kVbtRoot, col);
  float ws0 = 0.f, ws1 = 0.f, wsu0 = z0.x, wsu1 = z0.y;
  uint32_t node = 1;
  // r 2^l, exact
  float x = fminf(fmaxf(float((t - P.vbt_t0) * P.vbt_inv_len), 0.f), 1.f);
#pragma unroll 1
  for (int l = 0; l < P.vbt_deep; l++) {
    const float2 z = vbt_normal_pair(P.seed, tj, node, kVbtMid, col);
    const float a = __int_as_float((126 - ((l + 1) >> 1)) << 23) * (l & 1 ? 1.41421354f : 1.f);
    // the half that holds r: its index among the level's is the largest integer below
    // the scaled r, odd once that is a multiple of 2
    x += x;
    const bool right = x >= 16777216.f || (max(int(ceilf(x)) - 1, 0) & 1);
    const float st0 = 0.5f * wsu0 + a * z.x, st1 = 0.5f * wsu1 + a * z.y;
    if (right) {
      ws0 += st0;
      ws1 += st1;
    }
    wsu0 = right ? 0.5f * wsu0 - a * z.x : st0;
    wsu1 = right ? 0.5f * wsu1 - a * z.y : st1;
    node = 2 * node + (right ? 1u : 0u);
  }
  const float2 z = vbt_normal_pair(P.seed, tj, node, kVbtLeaf, col);
  const float f = x < 16777216.f ? x - fmaxf(ceilf(x) - 1.f, 0.f) : 1.f;
  const float su = P.vbt_deep < 127 ? __int_as_float((127 - P.vbt_deep) << 23) : 0.f;
  const float bb = sqrtf(f * (1.f - f) * su), sq = P.vbt_sqrt_len;
  return make_float2(sq * (ws0 + f * wsu0 + bb * z.x), sq * (ws1 + f * wsu1 + bb * z.y));
}

// Dimensions (col, col + 1).
static __device__ __noinline__ float2 vbt_w_pair(const SolveParams &P, int64_t traj, double t,
                                                 int col) {
  if (P.vbt_deep) return vbt_w_deep(P, traj, t, col);
  float w[2];
  vbt_w<2>(P, traj, t, col >> 2, col & 2, nullptr, w);
  return make_float2(w[0], w[1]);
}

// A quad of dimensions 4 quad .. 4 quad + 3, from the cached path.
static __device__ __noinline__ float4 vbt_w_quad(const SolveParams &P, int64_t traj, double t,
                                                 int quad, VbtQuadCache &C) {
  float w[4];
  vbt_w<4>(P, traj, t, quad, 0, &C, w);
  return make_float4(w[0], w[1], w[2], w[3]);
}

// The same of a tree of either depth class; the launch chooses the kernel by vbt_deep.
// (A choice in the kernel cost 4000 neural SDE trajectories 3 %, 955 to 988 us.)
template <bool DEEP>
__device__ __forceinline__ float4 vbt_w_quad(const SolveParams &P, int64_t traj, double t,
                                             int quad, VbtQuadCache &C) {
  if constexpr (DEEP) {
    const float2 a = vbt_w_deep(P, traj, t, 4 * quad), b = vbt_w_deep(P, traj, t, 4 * quad + 2);
    return make_float4(a.x, a.y, b.x, b.y);
  } else {
    return vbt_w_quad(P, traj, t, quad, C);
  }
}

// The tree with space-time Levy area: W_unit(r) and bar H_unit(r) = r H_{0,r}
// at unit time r for dimensions (col, col + 1), col even, unscaled (the caller
// combines two points by Chen's relation and scales by sqrt(T)).  The descent
// carries W and bar H of each dyadic interval: root W_1 ~ N(0, 1), bar H_1 ~
// N(0, 1/12) (tree.py:389-394); midpoint rule tree.py:727-750; final bridge
// tree.py:562-603.  The kVbt*H draws feed bar H, the others W, as in the
// FP64 oracle.
static __device__ __noinline__ void vbt_levy_pair(const SolveParams &P, int64_t traj, float r, int col,
                                                  float2 &w_r, float2 &bhh_r) {
  const float tol = float(P.vbt_tol_unit);
  const uint32_t tj = uint32_t(traj);
  const float2 z0 = vbt_normal_pair(P.seed, tj, 0u, kVbtRoot, col);
  const float2 n0 = vbt_normal_pair(P.seed, tj, 0u, kVbtRootH, col);
  float ws[2] = {0.f, 0.f}, wsu[2] = {z0.x, z0.y};
  float hs[2] = {0.f, 0.f};
  const float inv_sqrt12 = 0.28867513459481287f;
  float hsu[2] = {n0.x * inv_sqrt12, n0.y * inv_sqrt12};
  float s = 0.f, su = 1.f;
  uint32_t node = 1;
  while (su > tol) {  // while 2^-level > tol (tree.py:406-409)
    const float st = 0.5f * su, t_mid = s + st;
    const float2 z1 = vbt_normal_pair(P.seed, tj, node, kVbtMid, col);
    const float2 z2 = vbt_normal_pair(P.seed, tj, node, kVbtMidH, col);
    const float zs = 0.25f * sqrtf(su), ns = sqrtf(su * (1.0f / 12.0f));
    const float c3 = 1.5f / su, q = 0.25f * su;
    const bool right = r > t_mid;
    const float zz1[2] = {z1.x, z1.y}, zz2[2] = {z2.x, z2.y};
#pragma unroll
    for (int i = 0; i < 2; i++) {
      const float z = zz1[i] * zs, n = zz2[i] * ns;
      const float wt1 = 0.5f * wsu[i], wt2 = c3 * hsu[i] + z;
      const float ht1 = 0.125f * hsu[i] - q * z, ht2 = q * n;
      if (right) {
        const float w_t = ws[i] + (wt1 + wt2);
        hs[i] = hs[i] + (ht1 + ht2) + 0.5f * (t_mid * ws[i] - s * w_t);
        ws[i] = w_t;
        wsu[i] = wt1 - wt2;
        hsu[i] = ht1 - ht2;
      } else {
        wsu[i] = wt1 + wt2;
        hsu[i] = ht1 + ht2;
      }
    }
    if (right) s = t_mid;
    node = 2 * node + (right ? 1u : 0u);
    su = st;
  }
  const float sr = fmaxf(r - s, 0.f), ru = fmaxf(su - sr, 0.f);
  const float2 x1 = vbt_normal_pair(P.seed, tj, node, kVbtLeaf, col);
  const float2 x2 = vbt_normal_pair(P.seed, tj, node, kVbtLeafH, col);
  const float sr3 = sr * sr * sr, ru3 = ru * ru * ru, su3 = su * su * su;
  const float dd = sqrtf(sr3 + ru3);
  const float sr_ru_half = sqrtf(sr * ru);
  const float d_prime = 1.0f / (2.0f * su * dd);
  const float a = d_prime * sr3 * sr_ru_half, b = d_prime * ru3 * sr_ru_half;
  const float c = sqrtf(3.0f * sr3 * ru3) / (6.0f * dd);
  const float fw = sr / su, fh = 6.0f * sr * ru / su3, fx = 2.0f * (a + b) / su, fb = sr3 / su3;
  const float xx1[2] = {x1.x, x1.y}, xx2[2] = {x2.x, x2.y};
  float wo[2], ho[2];
#pragma unroll
  for (int i = 0; i < 2; i++) {
    const float w_sr = fw * wsu[i] + fh * hsu[i] + fx * xx1[i];
    wo[i] = ws[i] + w_sr;
    const float bhh_sr = fb * hsu[i] - a * xx1[i] + c * xx2[i];
    ho[i] = hs[i] + bhh_sr + 0.5f * (r * ws[i] - s * wo[i]);
  }
  w_r = make_float2(wo[0], wo[1]);
  bhh_r = make_float2(ho[0], ho[1]);
}

}  // namespace gbdx
