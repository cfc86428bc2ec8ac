// All six baryon contraction types in one pass, through the open diquark.
//
// Every type is linear in the 16 colour blocks
//   G[s][n] = sum_i c1(i) P_i[i][s] ^ P_j[perm1 i][n]
// (the diquark of the two quarks with both source spins open; ^ is the colour
// wedge of common.cuh).  With Gamma_kl as c2(l), partner perm2 l, and
// N'[m][l] = sum_n W[m][n] N[n][l]:
//   loop      IK_JL_NM: sum_l   c2(l) G[perm2 l][l] . Q,   Q = sum_m N'[m][m]
//   pass 1    IK_JM_NL: sum_m,l c2(l) G[perm2 l][m] . N'[m][l]
//   pass 2    IM_JK_NL: sum_m,l c2(l) G[m][perm2 l] . N'[m][l]
// Pass 2 swaps the roles of P_i and P_j: its wedge of spins (i, perm2 l, m) is
// P_j[i][perm2 l] ^ P_i[perm1 i][m], the wedge of G at row perm1 i, and the
// transposed Gamma_ij there is c1 at that row, so no second set of blocks is
// needed.  The Gamma_kl^T partners IL_JK_NM, IL_JM_NK and IM_JL_NK are a sign
// away (every Gamma(n) is symmetric or antisymmetric).
//
// Per site that is 64 wedges (2304 complex FMA) and, with the projectors'
// NG <= 2 gamma-basis terms, 2 x 16 x NG dots (9 each): 2 935 complex FMA for
// (1 +- g4)/2, where dotting every wedge E[i][s][n] by itself takes 5 078.
//
// One field for P_i and P_j: with H[s][n] the sum over the two rows i < perm1 i
// only, G[s][n] = H[s][n] + e H[n][s], e = +-1 the symmetry of Gamma_ij, so 32
// wedges do; pass 2 is e times pass 1, and pass 1 over G is pass 1 plus e times
// pass 2 over H.
//
// Thread mapping: thread sub of a site owns column s = sub / (TPS / 4) and the
// 16 / TPS consecutive columns n from n0 = (sub % (TPS / 4)) * (16 / TPS).
// Every Gamma's permutation is r -> r ^ class, so the partners are XORs of
// the classes in FusedSpin and no table is read per site.
#pragma once

#include "engine_warp.cuh"
#include "fixed.cuh"
#include "ops.cuh"

namespace cgb {

// Every Gamma(n): symmetric or antisymmetric, an XOR permutation, and entries
// that differ by signs only.
CGB_HD constexpr bool gammas_are_signed_xor()
{
  constexpr GammaTables g = build_gamma_tables();
  for (int n = 0; n < 16; ++n) {
    const int d = (g.ph_t[n][0] - g.ph[n][0]) & 3;
    if (d & 1) return false;
    for (int r = 0; r < 4; ++r)
      if (((g.ph_t[n][r] - g.ph[n][r]) & 3) != d || g.perm[n][r] != (r ^ g.perm[n][0]) ||
          ((g.ph[n][r] ^ g.ph[n][0]) & 1))
        return false;
  }
  return true;
}
static_assert(gammas_are_signed_xor(), "a Gamma lacks the structure the all-types pass is built on");

// Fills p.b.fu from the gamma rows and the gamma-basis terms (host).  With
// `half`, the rows are the two with i < perm1 i (one field for P_i and P_j).
template <class R> inline void fill_fused_spin(OpParams<R> &p, bool half)
{
  const BaryonSpin<R> &b = p.b;
  FusedSpin &f = p.b.fu;
  f = {};
  const uint32_t par1 = b.ph1[0][0] & 1, par2 = b.ph2[0][0] & 1;
  int n = 0;
  for (int neg = 1; neg >= 0; --neg) {
    for (int i = 0; i < 4; ++i)
      if ((b.ph1[0][i] >> 1) == neg && (!half || i < b.perm1[i])) f.rows |= (uint32_t)i << (2 * n++);
    if (neg) f.rows |= (uint32_t)n << 8;
  }
  f.s = b.perm1[0] | (uint32_t)b.perm2[0] << 2;
  for (int r = 0; r < 4; ++r) f.neg |= (uint32_t)(b.ph2[0][r] >> 1) << r;
  f.out = ((par1 + par2) & 3) | (uint32_t)((b.ph2[1][0] - b.ph2[0][0]) & 3) << 2 |
          (uint32_t)((b.ph1[1][0] - b.ph1[0][0]) & 3) << 4;
  for (int k = 0; k < 2 && k < b.cl.ng; ++k) {
    f.s |= (uint32_t)b.cl.perm[k][0] << (4 + 2 * k);
    for (int m = 0; m < 4; ++m) f.neg |= (uint32_t)(b.cl.ph[k][m] >> 1) << (4 + 4 * k + m);
    f.out |= (uint32_t)((par1 + par2 + (b.cl.ph[k][0] & 1)) & 3) << (8 + 2 * k);
  }
}

__device__ __forceinline__ uint32_t two_bits(uint32_t w, int at) { return (w >> at) & 3u; }
// v with the sign bit `at` of `w` applied
template <class R> __device__ __forceinline__ cx<R> signed_by(cx<R> v, uint32_t w, int at)
{
  const uint32_t s = (w >> at) & 1u;
  return {flip_sign(v.x, s), flip_sign(v.y, s)};
}

// The colour block at spin pair `blk` of a site, and two consecutive ones from
// an even pair (16-byte aligned in complex64: vector loads).
template <int NN, class R, class S> __device__ __forceinline__ void load_blocks(cx<R> (&out)[NN][9], const S *site, int blk)
{
  if constexpr (NN == 2) {
    load9p<false>(out[0], site + blk * 9);
    load9p<true>(out[1], site + blk * 9 + 9);
  } else {
    load9(out[0], site + blk * 9);
  }
}

// G[s][n0 .. n0 + NN) over NROW rows (without Gamma_ij's common power of i).
template <int NROW, int NN, class R, class S>
__device__ __forceinline__ void open_diquark(const FusedSpin &f, const S *A, const S *B, int s, int n0, cx<R> (&g)[NN][9])
{
#pragma unroll
  for (int t = 0; t < NN; ++t)
#pragma unroll
    for (int k = 0; k < 9; ++k) g[t][k] = czero<R>();
  const int s1 = f.s & 3, turn = (f.rows >> 8) & 7;
#pragma unroll 2
  for (int k = 0; k < NROW; ++k) {
    const int i = two_bits(f.rows, 2 * k);
    if (k == turn) {  // the same for every thread of the grid: the rows so far are the negative ones
#pragma unroll
      for (int t = 0; t < NN; ++t)
#pragma unroll
        for (int e = 0; e < 9; ++e) g[t][e] = {-g[t][e].x, -g[t][e].y};
    }
    cx<R> a[9], b[NN][9];
    load9(a, A + (i * 4 + s) * 9);
    load_blocks<NN, R, S>(b, B, (i ^ s1) * 4 + n0);
#pragma unroll
    for (int t = 0; t < NN; ++t) wedge_acc(g[t], a, b[t]);
  }
  if (turn == NROW) {
#pragma unroll
    for (int t = 0; t < NN; ++t)
#pragma unroll
      for (int e = 0; e < 9; ++e) g[t][e] = {-g[t][e].x, -g[t][e].y};
  }
}

// The same in fixed point (fixed.cuh), from blocks that were converted.
template <int NROW, int NN>
__device__ __forceinline__ void open_diquark_fixed(const FusedSpin &f, const int4 *A, const int4 *B, int s, int n0,
                                                   const FixedScales &fs, cx<double> (&g)[NN][9])
{
  const int s1 = f.s & 3, turn = (f.rows >> 8) & 7;
#pragma unroll
  for (int t = 0; t < NN; ++t)
    fixed_wedge_sum(0, NROW, fs, [&](int k, const int4 *&x, const int4 *&y) {
      const int i = two_bits(f.rows, 2 * k);
      x = A + (i * 4 + s) * 9;
      y = B + ((i ^ s1) * 4 + n0 + t) * 9;
      return k < turn;
    }, g[t]);
}

// What open_diquark_fixed's sum for thread (s, n0) covers.  One field: G[s][n] is H[s][n]
// with H[n][s], the other thread's.
template <int NROW>
__device__ __forceinline__ uint32_t open_diquark_cover(const FusedSpin &f, uint32_t x, uint32_t y, int s, int n0)
{
  uint32_t c = 0;
#pragma unroll
  for (int k = 0; k < NROW; ++k) {
    const int i = two_bits(f.rows, 2 * k);
    c |= wedge_cover(block_word(x, i * 4 + s), block_word(y, (i ^ (f.s & 3)) * 4 + n0));
  }
  return NROW == 4 ? c : c | block_word(c, n0 * 4 + s);
}

// Converts the site's blocks of two fields, one of each per thread, in place, if every
// site of the warp suits the integer form.  cover(x, y): what the thread's sum of wedges
// covers, from its own blocks' words.
template <class Cover>
__device__ __forceinline__ bool fields_to_fixed(double2 *A, double2 *B, int sub, bool live, FixedScales &fs, Cover cover)
{
  const double2 *blk[2] = {A + sub * 9, B + sub * 9};
  uint32_t near[2];
  const bool scaled = fixed_scales<16, 1>(blk, fs, near);
  const bool ok = wedges_covered(cover(cover_word(near[0]), cover_word(near[1]))) && scaled;
  if (!__all_sync(0xffffffffu, ok || !live)) return false;
  block_to_fixed(reinterpret_cast<int4 *>(A + sub * 9), blk[0], fs, 0);
  if (A != B) block_to_fixed(reinterpret_cast<int4 *>(B + sub * 9), blk[1], fs, 1);
  __syncwarp();
  return true;
}

// Converts the blocks of P_n in place likewise, if the thread's blocks g of G, which
// may come from the FP64 form, suit it as well.  covered(near): whether all of the
// thread's dots are, from its own block's near bits.
template <int NN, class Covered>
__device__ __forceinline__ bool dots_to_fixed(double2 *N, const cx<double> (&g)[NN][9], int sub, bool live,
                                              FixedDotBlock (&gb)[NN], Covered covered)
{
  FixedScales fs;
  const double2 *blk[1] = {N + sub * 9};
  uint32_t near[1];
  bool ok = fixed_scales<16, 1>(blk, fs, near);
  uint32_t any = 0;  // dots with a block of zeros are exact
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    const int4 v = reinterpret_cast<const int4 *>(blk[0])[k];
    any |= (uint32_t)(v.x | v.z) | ((uint32_t)(v.y | v.w) & 0x7fffffffu);
  }
#pragma unroll
  for (int t = 0; t < NN; ++t) ok = gb[t].fits(g[t], fs) && ok;
  ok = covered(any ? near[0] : 0x1ffu) && ok;
  if (!__all_sync(0xffffffffu, ok || !live)) return false;
  block_to_fixed(reinterpret_cast<int4 *>(N + sub * 9), blk[0], fs, 0);
#pragma unroll
  for (int t = 0; t < NN; ++t) gb[t].set(g[t], fs);
  __syncwarp();
  return true;
}

// A block of G held for several dots.  Complex64: g and its (im, re) swap as
// FP32 pairs, so that each product pair is one packed FMA on the other block
// as loaded: P = sum g (.) y, Q = sum swap(g) (.) y, g . y = (P.x - P.y, Q.x + Q.y).
template <class R> struct DotBlock {
  cx<R> g[9];
  __device__ __forceinline__ void set(const cx<R> (&v)[9])
  {
#pragma unroll
    for (int k = 0; k < 9; ++k) g[k] = v[k];
  }
  template <class S> __device__ __forceinline__ cx<R> dot(const S *blk) const
  {
    cx<R> y[9];
    load9(y, blk);
    return dot9(g, y);
  }
};
template <> struct DotBlock<float> {
  float2 g[9], w[9];
  __device__ __forceinline__ void set(const cx<float> (&v)[9])
  {
#pragma unroll
    for (int k = 0; k < 9; ++k) {
      g[k] = make_float2(v[k].x, v[k].y);
      w[k] = make_float2(v[k].y, v[k].x);
    }
  }
  __device__ __forceinline__ cx<float> dot(const float2 *blk) const
  {
    float2 P = make_float2(0.f, 0.f), Q = P;
#pragma unroll
    for (int k = 0; k < 9; ++k) {
      const float2 y = blk[k];
      P = __ffma2_rn(g[k], y, P);
      Q = __ffma2_rn(w[k], y, Q);
    }
    return {P.x - P.y, Q.x + Q.y};
  }
};

// How the open spin slot is applied, by SRC:
//   1, 2    the projectors in the gamma basis, SRC = b.cl.ng terms: values per
//           term, which combine() turns into the projectors' outputs
//   -1, -2  one projector of rank -SRC, W = sum_r x_r y_r^T (RankForm): blocks
//           Y_r[l] = sum_n y_r[n] N[n][l], N'[m][l] = sum_r x_r[m] Y_r[l]
//   0       N'_w = W_w N materialised per site (any projector)
// The pass leaves NVAL values per site, summed over its threads: the loop,
// pass 1 and (two fields) pass 2 value of every term or projector.
template <class R_, class S_, int CW_, int TPS_, int SRC, int NW, bool SAME = false, int MINB = 1>
struct BaryonFusedOp {
  using R = R_;
  using S = S_;
  using Params = OpParams<R>;
  static constexpr int CW = CW_, TPS = TPS_, MIN_CTAS = MINB;
  static_assert(SRC >= 0 || NW == 1, "the factored form takes one projector");
  static constexpr int NK = SRC > 0 ? SRC : NW;    // values per group
  static constexpr int ND = SRC < 0 ? -SRC : NK;  // dots per pass and column n
  static constexpr int NIN = SAME ? 2 : 3, NOUT = 6 * NW, NVAL = (SAME ? 2 : 3) * NK;
  // scratch: the diagonal blocks of G, then N' and Q, or Y
  static constexpr int NBLK = SRC > 0 ? 0 : (SRC < 0 ? -4 * SRC : 16 * NW);
  static constexpr int EXTRA_BYTES = cbytes<S>(36 + 9 * NBLK + (SRC == 0 ? 9 * NW : 0)) + 16;  // +16: bank stagger
  // Threads of one site read blocks 4 i + (0..3): with 1184-byte slots the next
  // site's blocks start 32 bytes on, in banks the first site's do not use.
  static constexpr int SLOT_PAD = 32;

  static constexpr int TPC = TPS / 4, NN = 4 / TPC;  // threads per column s, columns n per thread
  using State = cx<R>[NN][9];  // the thread's blocks of G

  // P_i and P_j: the thread's blocks of G, and the loop's blocks G[perm2 l][l]
  // to scratch.
  __device__ static void first(const OpParams<R> &p, S *const *in, S *scratch, int sub, bool live, State &g)
  {
    const FusedSpin f = p.b.fu;
    const int s = sub / TPC, n0 = (sub % TPC) * NN, l = s ^ ((f.s >> 2) & 3);
    S *A = in[0], *B = SAME ? in[0] : in[1];
    if constexpr (sizeof(R) == 8) {
      FixedScales fs;
      static_assert(TPS == 16, "one block of G per thread");
      if (fields_to_fixed(A, B, sub, live, fs, [&](uint32_t x, uint32_t y) {
            return open_diquark_cover<SAME ? 2 : 4>(f, x, y, s, n0);
          }))
        open_diquark_fixed<SAME ? 2 : 4, NN>(f, reinterpret_cast<const int4 *>(A), reinterpret_cast<const int4 *>(B), s, n0, fs, g);
      else
        open_diquark<SAME ? 2 : 4, NN, R, S>(f, A, B, s, n0, g);
    } else {
      open_diquark<SAME ? 2 : 4, NN, R, S>(f, A, B, s, n0, g);
    }
#pragma unroll
    for (int t = 0; t < NN; ++t)
      if (l == n0 + t) {
#pragma unroll
        for (int k = 0; k < 9; ++k) st(scratch + l * 9 + k, g[t][k]);
      }
  }

  // P_n: the values of the site (called after a __syncwarp).
  __device__ static void second(const OpParams<R> &p, S *N, S *scratch, int sub, bool live, const State &g,
                                cx<R> (&vals)[NVAL])
  {
    const BaryonSpin<R> &b = p.b;
    const FusedSpin f = b.fu;
    const int s = sub / TPC, n0 = (sub % TPC) * NN, s2 = (f.s >> 2) & 3, l = s ^ s2;
    S *diag = scratch, *blk = scratch + 36, *q = blk + 9 * NBLK;
    if constexpr (SRC == 0) {
      build_nprime<R, S, TPS, NW>(b, N, blk, sub, b.cl.ng <= kNprimeCliffTerms);
      build_q<R, S, TPS, NW>(b, N, q, sub);
      __syncwarp();
    }
    if constexpr (SRC < 0) {
      build_rank_y<R, S, TPS>(b.rk, N, blk, sub);
      __syncwarp();
    }
    // loop: one colour entry per thread
    cx<R> lp[NK];
#pragma unroll
    for (int k = 0; k < NK; ++k) lp[k] = czero<R>();
    for (int e = sub; e < 9; e += TPS) {
      cx<R> r = czero<R>();
#pragma unroll
      for (int c = 0; c < 4; ++c) r = cadd(r, signed_by(ld<R>(diag + c * 9 + e), f.neg, c));
#pragma unroll
      for (int k = 0; k < NK; ++k) {
        cx<R> qk = czero<R>();
        if constexpr (SRC > 0) {
          const int sk = two_bits(f.s, 4 + 2 * k);
#pragma unroll
          for (int m = 0; m < 4; ++m)
            qk = cadd(qk, signed_by(ld<R>(N + ((m ^ sk) * 4 + m) * 9 + e), f.neg, 4 + 4 * k + m));
        } else if constexpr (SRC < 0) {
#pragma unroll
          for (int d = 0; d < ND; ++d)
#pragma unroll
            for (int m = 0; m < 4; ++m)
              cfma(qk, cx<R> {b.rk.x[d][m][0], b.rk.x[d][m][1]}, ld<R>(blk + (d * 4 + m) * 9 + e));
        } else {
          qk = ld<R>(q + k * 9 + e);
        }
        cfma(lp[k], r, qk);
      }
    }
    // passes 1 and 2
    cx<R> v1[NK], v2[NK];
#pragma unroll
    for (int k = 0; k < NK; ++k) v1[k] = v2[k] = czero<R>();
    auto dots = [&](const auto (&gb)[NN]) {
#pragma unroll
      for (int d = 0; d < ND; ++d) {
        const int k = SRC < 0 ? 0 : d, sk = SRC > 0 ? two_bits(f.s, 4 + 2 * d) : 0;
#pragma unroll
        for (int t = 0; t < NN; ++t) {
          const int n = n0 + t, ln = n ^ s2;
          const S *e1, *e2;  // the blocks of N' (or of the term, or Y) for passes 1 and 2
          if constexpr (SRC > 0) {
            e1 = N + ((n ^ sk) * 4 + l) * 9;
            e2 = N + ((s ^ sk) * 4 + ln) * 9;
          } else if constexpr (SRC < 0) {
            e1 = blk + (d * 4 + l) * 9;
            e2 = blk + (d * 4 + ln) * 9;
          } else {
            e1 = blk + (16 * d + n * 4 + l) * 9;
            e2 = blk + (16 * d + s * 4 + ln) * 9;
          }
          const cx<R> d1 = gb[t].dot(e1), d2 = signed_by(gb[t].dot(e2), f.neg, ln);
          if constexpr (SRC < 0) {
            cfma(v1[0], cx<R> {b.rk.x[d][n][0], b.rk.x[d][n][1]}, d1);
            cfma(v2[0], cx<R> {b.rk.x[d][s][0], b.rk.x[d][s][1]}, d2);
          } else {
            v1[k] = cadd(v1[k], SRC > 0 ? signed_by(d1, f.neg, 4 + 4 * d + n) : d1);
            v2[k] = cadd(v2[k], d2);
          }
        }
      }
    };
    auto plain = [&]() {
      DotBlock<R> gb[NN];
#pragma unroll
      for (int t = 0; t < NN; ++t) gb[t].set(g[t]);
      dots(gb);
    };
    if constexpr (sizeof(R) == 8 && SRC > 0) {
      __syncwarp();  // the loop above has read P_n
      FixedDotBlock gb[NN];
      const auto covered = [&](uint32_t near) {
        bool ok = true;
#pragma unroll
        for (int d = 0; d < ND; ++d) {
          const int sk = two_bits(f.s, 4 + 2 * d);
#pragma unroll
          for (int t = 0; t < NN; ++t) {
            const int n = n0 + t;
            ok = (gb[t].near & block_word(near, (n ^ sk) * 4 + l)) != 0 && ok;
            ok = (gb[t].near & block_word(near, (s ^ sk) * 4 + (n ^ s2))) != 0 && ok;
          }
        }
        return ok;
      };
      if (dots_to_fixed(N, g, sub, live, gb, covered)) dots(gb);
      else plain();
    } else {
      plain();
    }
#pragma unroll
    for (int k = 0; k < NK; ++k) {
      v1[k] = signed_by(v1[k], f.neg, l);
      if constexpr (SRC > 0) v2[k] = signed_by(v2[k], f.neg, 4 + 4 * k + s);
    }
    if constexpr (SAME) {
      const uint32_t e = f.out >> 5;  // Gamma_ij antisymmetric
      // G[perm2 l][l] = H[perm2 l][l] + e H[l][perm2 l]; the second term at l is
      // the first at perm2 l, with the sign of Gamma_kl's symmetry
      const uint32_t el = e ^ (f.out >> 3);
#pragma unroll
      for (int k = 0; k < NK; ++k) {
        vals[k] = cadd(lp[k], signed_by(lp[k], el, 0));
        vals[NK + k] = cadd(v1[k], signed_by(v2[k], e, 0));
      }
    } else {
#pragma unroll
      for (int k = 0; k < NK; ++k) {
        vals[k] = lp[k];
        vals[NK + k] = v1[k];
        vals[2 * NK + k] = v2[k];
      }
    }
  }

  // Output o = type * NW + w from the values of a site or a chunk, value r held
  // by lane base + r * stride (every lane of the warp calls).  V: cx<R> or double2.
  template <class V> __device__ static V combine(const OpParams<R> &p, int o, V v, int base, int stride)
  {
    using F = decltype(V::x);
    const int type = o / NW, w = o - type * NW;
    const int kind = type == 0 || type == 2 ? 0 : (type == 1 || type == 3 || SAME ? 1 : 2);
    uint32_t ph = type == 2 || type == 3 || type == 5 ? two_bits(p.b.fu.out, 2) : 0u;  // the Gamma_kl^T partner
    if (SAME && type >= 4) ph += two_bits(p.b.fu.out, 4);
    cx<F> r {F(0), F(0)};
#pragma unroll
    for (int k = 0; k < (SRC > 0 ? SRC : 1); ++k) {
      const int src = base + (kind * NK + (SRC > 0 ? k : w)) * stride;
      const cx<F> x {__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src)};
      if constexpr (SRC > 0)
        cfma(r, cx<F> {F(p.b.cl.coef[w][k][0]), F(p.b.cl.coef[w][k][1])}, mul_phase(x, two_bits(p.b.fu.out, 8 + 2 * k)));
      else
        r = mul_phase(x, two_bits(p.b.fu.out, 0));
    }
    r = mul_phase(r, ph & 3u);
    return V {r.x, r.y};
  }
};

} // namespace cgb
