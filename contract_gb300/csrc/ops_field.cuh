// Field ops for field_ring_kernel (engine_warp.cuh): diquark and sequential sources,
// one propagator-shaped result per site from two fields.
//
// Every result block is a phase times a signed sum of colour wedges x_k ^ y_k of
// blocks of the two fields (four wedges, or one with the block Q), since W is a Gamma
// matrix here and N' = W N a signed permutation of N's blocks: thread (r, c) of a
// site's 16 makes block (r, c).  Roles as in ops.cuh; with s1, s2, sw the classes of
// Gamma_ij, Gamma_kl and W (a Gamma's permutation is r -> r ^ s):
//   Diquark (m, l)   conj sum_i c1(i) P_i[i][l ^ s2] ^ P_j[i ^ s1][m], times c2(l) g5 g5
//                    (include/diquark.cuh:33-57)
//   TriA   (i, k)    sum_m w(m) B[i ^ s1][m] ^ N[m ^ sw][l], l = k ^ s2
//   TriB   (j, m)    sum_l c2(l) A[j ^ s1][l ^ s2] ^ N[m ^ sw][l]
//   TriN   (n, l)    sum_i c1(i) A[i][l ^ s2] ^ B[i ^ s1][n ^ sw]
//   LoopA  (i, k)    B[i ^ s1][k ^ s2] ^ Q
//   LoopB  (j, l)    A[j ^ s1][l ^ s2] ^ Q
//   LoopN  (n, m)    W[m][n] sum_{i,l} c1(i) c2(l) A[i][l ^ s2] ^ B[i ^ s1][l]
// (include/baryon_sequential.cuh:36-163).  The summed index runs over the negative
// terms first, so that the signs cost one negation of the sum.
//
// Complex64 is HBM bound, two fields in and one out.  Complex128 takes its sums of wedges
// on the integer pipe where a site allows it (fixed.cuh), else, and for one wedge a block,
// in FP64.
#pragma once

#include "ops_site.cuh"

namespace cgb {

enum class Wedges { Diquark, TriA, TriB, TriN, LoopA, LoopB, LoopN };

// Fills p.b.fu (classes, order of the summed index) from the gamma rows and W (host).
template <class R> inline void fill_wedges(OpParams<R> &p, Wedges kind)
{
  BaryonSpin<R> &b = p.b;
  const uint8_t *ph = kind == Wedges::TriA ? b.proj[0].ph : kind == Wedges::TriB ? b.ph2[0] : b.ph1[0];
  FusedSpin &f = b.fu;
  f = {};
  int n = 0;
  for (int neg = 1; neg >= 0; --neg) {
    for (int i = 0; i < 4; ++i)
      if ((ph[i] >> 1) == neg) f.rows |= (uint32_t)i << (2 * n++);
    if (neg) f.rows |= (uint32_t)n << 8;
  }
  f.s = b.perm1[0] | (uint32_t)b.perm2[0] << 2 | (uint32_t)b.proj[0].perm[0] << 4;
  f.out = ph[0] & 1u;  // the summed Gamma's common power of i
}

template <class R, class S, int CW, int NST, int MINB, Wedges KIND>
struct WedgeFieldOp : RingOp<R, S, CW, 16, NST, MINB> {
  static constexpr bool LOOP = KIND == Wedges::LoopA || KIND == Wedges::LoopB;  // one wedge with Q
  static constexpr int NIN = 2, OUT_ELEMS = 144, EXTRA_BYTES = LOOP ? cbytes<S>(9) : 0;

  // Terms k0 to k1 of block (r, c): the two blocks of term t.
  __device__ __forceinline__ static void term(const FusedSpin &f, int r, int c, int t, int &x, int &y)
  {
    const int s1 = f.s & 3, s2 = (f.s >> 2) & 3, sw = (f.s >> 4) & 3;
    if constexpr (KIND == Wedges::TriA) {
      x = (r ^ s1) * 4 + t;
      y = (t ^ sw) * 4 + (c ^ s2);
    } else if constexpr (KIND == Wedges::TriB) {
      x = (r ^ s1) * 4 + (t ^ s2);
      y = (c ^ sw) * 4 + t;
    } else {
      x = t * 4 + (c ^ s2);
      y = (t ^ s1) * 4 + (KIND == Wedges::TriN ? r ^ sw : r);
    }
  }
  // The phase of block (r, c), without what the order of the terms has taken.
  __device__ __forceinline__ static uint32_t phase(const BaryonSpin<R> &b, int r, int c)
  {
    const FusedSpin f = b.fu;
    const int i = r ^ (f.s & 3), l = c ^ ((f.s >> 2) & 3);
    const uint8_t *w = b.proj[0].ph;
    if constexpr (KIND == Wedges::Diquark) return f.out + b.ph2[0][c];
    else if constexpr (KIND == Wedges::TriA) return f.out + b.ph1[0][r] + b.ph2[0][l];
    else if constexpr (KIND == Wedges::TriB) return f.out + b.ph1[0][i] + w[c];
    else if constexpr (KIND == Wedges::TriN) return f.out + b.ph2[0][c] + w[r ^ ((f.s >> 4) & 3)];
    else if constexpr (KIND == Wedges::LoopA) return b.ph1[0][r] + b.ph2[0][l];
    else return b.ph1[0][i] + b.ph2[0][c];
  }

  // Four wedges a block.
  __device__ __forceinline__ static void sums(const BaryonSpin<R> &b, S *X, S *Y, int sub, bool live, cx<R> (&d)[9])
  {
    const FusedSpin f = b.fu;
    const int r = sub >> 2, c = sub & 3, turn = (f.rows >> 8) & 7;
    if constexpr (sizeof(R) == 8) {
      FixedScales fs;
      if (fields_to_fixed(X, Y, sub, live, fs, [&](uint32_t x, uint32_t y) {
            uint32_t cover = 0;
#pragma unroll
            for (int t = 0; t < 4; ++t) {
              int xb, yb;
              term(f, r, c, t, xb, yb);
              cover |= wedge_cover(block_word(x, xb), block_word(y, yb));
            }
            return cover;
          })) {
        fixed_wedge_sum(0, 4, fs, [&](int k, const int4 *&x, const int4 *&y) {
          int xb, yb;
          term(f, r, c, two_bits(f.rows, 2 * k), xb, yb);
          x = reinterpret_cast<const int4 *>(X) + xb * 9;
          y = reinterpret_cast<const int4 *>(Y) + yb * 9;
          return k < turn;
        }, d);
        return;
      }
    }
#pragma unroll
    for (int e = 0; e < 9; ++e) d[e] = czero<R>();
#pragma unroll 2
    for (int k = 0; k < 4; ++k) {
      if (k == turn) {  // the same for every thread: the terms so far are the negative ones
#pragma unroll
        for (int e = 0; e < 9; ++e) d[e] = {-d[e].x, -d[e].y};
      }
      int xb, yb;
      term(f, r, c, two_bits(f.rows, 2 * k), xb, yb);
      cx<R> x[9], y[9];
      load9(x, X + xb * 9);
      load9(y, Y + yb * 9);
      wedge_acc(d, x, y);
    }
    if (turn == 4) {
#pragma unroll
      for (int e = 0; e < 9; ++e) d[e] = {-d[e].x, -d[e].y};
    }
  }

  // One wedge a block, with Q (in q) of the field N.  FP64 in complex128: the four products
  // of an entry are too few for one of them to be near its scale as a rule.
  __device__ __forceinline__ static void with_q(const BaryonSpin<R> &b, S *X, const S *N, S *q, int sub, cx<R> (&d)[9])
  {
    const FusedSpin f = b.fu;
    const int xb = sub ^ (f.s & 3) << 2 ^ ((f.s >> 2) & 3);  // block (r ^ s1, c ^ s2)
    build_q<R, S, 16, 1>(b, N, q, sub);
    __syncwarp();
    cx<R> x[9], y[9];
#pragma unroll
    for (int e = 0; e < 9; ++e) d[e] = czero<R>();
    load9(x, X + xb * 9);
    load9(y, q);
    wedge_acc(d, x, y);
  }

  // LoopN: the site's 16 wedges summed, entry e left with thread e (0 to 8).
  __device__ __forceinline__ static cx<R> closed(const BaryonSpin<R> &b, S *A, S *B, int sub, bool live)
  {
    const int i = sub >> 2, l = sub & 3, xb = i * 4 + b.perm2[l], yb = b.perm1[i] * 4 + l;
    const uint32_t ph = (b.ph1[0][i] + b.ph2[0][l]) & 3u;
    if constexpr (sizeof(R) == 8) {
      FixedScales fs;
      if (fields_to_fixed(A, B, sub, live, fs, [&](uint32_t x, uint32_t y) {
            return site_cover(wedge_cover(block_word(x, xb), block_word(y, yb)));
          })) {
        const uint32_t common = (b.ph1[0][0] & 1u) + (b.ph2[0][0] & 1u);
        const longlong2 d = fixed_wedge_scatter(reinterpret_cast<const int4 *>(A) + xb * 9,
                                                reinterpret_cast<const int4 *>(B) + yb * 9, ((ph - common) & 2u) != 0, sub);
        return mul_phase(fixed_entry(d, min(sub, 8), fs), common);
      }
    }
    cx<R> x[9], y[9], d[9];
#pragma unroll
    for (int e = 0; e < 9; ++e) d[e] = czero<R>();
    load9(x, A + xb * 9);
    load9(y, B + yb * 9);
    phase9(x, ph);
    wedge_acc(d, x, y);
    R re[9], im[9];
#pragma unroll
    for (int e = 0; e < 9; ++e) {
      re[e] = d[e].x;
      im[e] = d[e].y;
    }
    R u, v;
    group_sum_scatter9(re, im, sub, u, v);
    return {u, v};
  }

  // The result takes the place of the first field's blocks.
  __device__ static void site(const OpParams<R> &p, S *const *in, S *scratch, int sub, bool live)
  {
    const BaryonSpin<R> &b = p.b;
    const int r = sub >> 2, c = sub & 3;
    S *out = in[0];
    if constexpr (KIND == Wedges::LoopN) {
      const cx<R> v = closed(b, in[0], in[1], sub, live);
      __syncwarp();  // the fields have been read
#pragma unroll
      for (int e = 0; e < 9; ++e) st(out + sub * 9 + e, czero<R>());
      __syncwarp();
      const ProjOperand<R> &w = b.proj[0];
      if (sub < 9) {
#pragma unroll
        for (int m = 0; m < 4; ++m) st(out + (w.perm[m] * 4 + m) * 9 + sub, mul_phase(v, w.ph[m]));
      }
    } else {
      cx<R> d[9];
      if constexpr (LOOP) with_q(b, in[0], in[1], scratch, sub, d);
      else sums(b, in[0], in[1], sub, live, d);
      phase9(d, phase(b, r, c) & 3u);
      if constexpr (KIND == Wedges::Diquark) {
        const uint32_t sgn = ((r >> 1) ^ (c >> 1)) & 1u;  // g5[m] g5[l]
#pragma unroll
        for (int e = 0; e < 9; ++e) d[e] = {flip_sign(d[e].x, sgn), flip_sign(d[e].y, sgn ^ 1u)};
      }
      __syncwarp();  // the fields have been read
#pragma unroll
      for (int e = 0; e < 9; ++e) st(out + sub * 9 + e, d[e]);
    }
  }
};

} // namespace cgb
