// Per-site contraction routines and the kernel "ops" that plug them into the
// tile engines (engine.cuh).
//
// Notation (one lattice site): a propagator P[s0][s1][c0][c1] is 16 colour
// blocks of 9 complex numbers; block (s0, s1) starts at (4*s0 + s1)*9.
// Gamma coefficients are phase codes (powers of i) and permutations:
//   c1(i) on spin row i with partner j = perm1[i]   (from Gamma_ij)
//   c2(l) on spin column l with partner k = perm2[l] (from Gamma_kl)
//
// Baryon two-point, canonical forms (F = eps.eps trilinear form, X ^ Y the
// colour wedge of common.cuh, W the 4x4 Gamma_mn/projector operand):
//   loop     C = sum_{i,l} c1(i) c2(l) F(A[i][perm2 l], B[perm1 i][l], Q),
//            Q = sum_{m,n} W[m][n] N[n][m]
//   triangle C = sum_{i,l} c1(i) c2(l) A[i][perm2 l] . sum_m (B[perm1 i][m] ^ N'[m][l]),
//            N'[m][l] = sum_n W[m][n] N[n][l]
// The six contract_enum.h types map onto these (CLQCD/contract
// include/baryon.cuh:43-83, baryon_general.cuh:45-93):
//   IK_JL_NM loop (A=P_i, B=P_j, c1 = Gamma_ij,   c2 = Gamma_kl^T)
//   IL_JK_NM loop (A=P_i, B=P_j, c1 = Gamma_ij,   c2 = Gamma_kl)
//   IK_JM_NL tri  (A=P_i, B=P_j, c1 = Gamma_ij,   c2 = Gamma_kl^T)
//   IL_JM_NK tri  (A=P_i, B=P_j, c1 = Gamma_ij,   c2 = Gamma_kl)
//   IM_JK_NL tri  (A=P_j, B=P_i, c1 = Gamma_ij^T, c2 = Gamma_kl^T)
//   IM_JL_NK tri  (A=P_j, B=P_i, c1 = Gamma_ij^T, c2 = Gamma_kl)
// Types that differ only in c2 share every wedge, which the fused kernel
// exploits: IK_JL/IL_JK, IK_JM/IL_JM and IM_JK/IM_JL each cost one evaluation.
//
// Thread mapping: TPS threads per site; thread `sub` owns spin row
// i = sub / (TPS/4) and LPT = 16/TPS consecutive columns l.
#pragma once

#include "engine.cuh"
#include "gamma.hpp"

namespace cgb {

// Projector operand W[m][n] (the Gamma_mn slot).  When W is a phased
// permutation (always true for a Gamma matrix) the kernels use perm/ph and
// do no multiplications with it.
template <class R> struct ProjOperand {
  R w[16][2];
  uint8_t perm[4];
  uint8_t ph[4];
  int is_perm;
  uint8_t nzk[16];  // indices m*4 + n of W's nonzero entries, in order
  int nnz;
  uint32_t nzmask;  // bit m*4 + n set where W[m][n] != 0
  uint32_t real, imag;  // the same where W[m][n] is real, where it is imaginary (and not 0)
};

// Up to two projectors written in the gamma basis, W_w = sum_k coef[w][k] Gamma(g_k):
// N'_w[m][l] = sum_k coef[w][k] i^ph[k][m] N[perm[k][m]][l], so the triangle
// form needs one spin-permuted pass over N per basis term and no N' buffer.
template <class R> struct CliffordSet {
  int ng;
  uint8_t perm[16][4];
  uint8_t ph[16][4];
  uint8_t has_phase[16];
  R coef[2][16][2];
  R qc[2][16][4][2];  // coef[w][k] * i^ph[k][m]: the coefficient of N[perm[k][m]][m] in Q_w
};

// A projector of rank r <= 2 as W = sum_r x_r y_r^T (W[m][n] = sum_r x_r[m] y_r[n]).
// Each vector is a list of nnz (index, coefficient) entries, padded with zero
// coefficients: [side 0: x_r over rows m, side 1: y_r over columns n][r][k].
template <class R> struct RankForm {
  int r;  // 0: the projector is not of this form
  int nnz;
  uint8_t idx[2][2][4];
  R c[2][2][4][2];
  // unit: every coefficient is scale_v i^ph and scale_x * scale_y is one value
  // `scale` for every r (true for (1 +- g4)/2 and the polarised projectors):
  // the complex128 builds then add phased blocks and the triangle values take
  // `scale` (rank_unit_form).  complex64 keeps the coefficients.
  int unit;
  uint8_t ph[2][2][4];
  R scale;
  R x[2][4][2];  // x_r[m], every entry (the all-types pass)
};

// The all-types pass's spin tables in packed words (fill_fused_spin in
// ops_fused.cuh): one 16-byte load per site.  Every Gamma(n) is real or
// imaginary throughout, so its entries are one common power of i, applied to
// the outputs, times the signs kept here.
struct alignas(16) FusedSpin {
  uint32_t s;     // permutation classes: Gamma_ij at bit 0, Gamma_kl at 2, term k at 4 + 2 k
  uint32_t rows;  // rows of Gamma_ij, negative ones first, at 2 k; number of negative rows at 8
  uint32_t neg;   // sign bits: c2(l) at bit l, term k at row m at bit 4 + 4 k + m
  uint32_t out;   // phase of the outputs at 0 (at 8 + 2 k with term k's), of the Gamma_kl^T partners against them
                  // at 2, of the IM_* group against the IK_JM/IL_JM one (one field) at 4 (the last two 0 or 2)
};

template <class R> struct BaryonSpin {
  uint8_t perm1[4], perm2[4];
  uint8_t ph1[2][4];  // [0]: c1 for A = P_i groups, [1]: c1 for the swapped (IM_*) group
  uint8_t ph2[2][4];  // c2 variants (one per output of a loop/tri evaluation)
  ProjOperand<R> proj[2];
  CliffordSet<R> cl;
  RankForm<R> rk;  // proj[0] factored, for the triangle form
  FusedSpin fu;
};

template <class R> struct MesonSpin {
  uint8_t perm1[4], perm2[4];
  uint8_t ph1[4], ph2[4];
};

template <class R> struct OpParams {
  const void *in[3];
  void *out[16];
  TileGeom geom;
  DeviceStatus *status;
  BaryonSpin<R> b;
  MesonSpin<R> m;
  int latt[4];  // Lx, Ly, Lz, Lt where an op needs site coordinates
};

template <int TPS> struct Lanes {
  static constexpr int TPI = TPS / 4;  // threads per spin row
  static constexpr int LPT = 4 / TPI;  // spin columns per thread
  static_assert(TPS == 4 || TPS == 8 || TPS == 16, "TPS must be 4, 8 or 16");
};

// Q_w[ad] = sum_{m,n} W[m][n] N[n][m][ad], one entry per thread, into smem q[w*9 + ad].
template <class R, class S, int TPS, int NW>
__device__ __forceinline__ void build_q(const BaryonSpin<R> &b, const S *N, S *q, int sub)
{
  for (int e = sub; e < 9 * NW; e += TPS) {
    const int w = e / 9, ad = e % 9;
    const ProjOperand<R> &pw = b.proj[w];
    cx<R> s = czero<R>();
    if (pw.is_perm) {
#pragma unroll
      for (int m = 0; m < 4; ++m) s = cadd(s, mul_phase(ld<R>(N + (pw.perm[m] * 4 + m) * 9 + ad), pw.ph[m]));
    } else if constexpr (sizeof(R) == 8) {
      // complex128: W's nonzero entries from the host's list.  Testing each
      // entry here takes FP64 compares on the FP64 pipe, half busy in the loop
      // form; for the same reason a real or imaginary entry takes two FMAs, not
      // four ((1 + g4)/2: 0.99 ms at 24^3 x 32, one gamma matrix 0.91).
#pragma unroll 1
      for (int t = 0; t < pw.nnz; ++t) {
        const int k = pw.nzk[t];  // W[m][n], m = k / 4, n = k % 4, times N[n][m]
        const cx<R> n = ld<R>(N + ((k & 3) * 4 + (k >> 2)) * 9 + ad);
        if ((pw.real >> k) & 1u) s = {fma(pw.w[k][0], n.x, s.x), fma(pw.w[k][0], n.y, s.y)};
        else if ((pw.imag >> k) & 1u) s = {fma(-pw.w[k][1], n.y, s.x), fma(pw.w[k][1], n.x, s.y)};
        else cfma(s, cx<R> {pw.w[k][0], pw.w[k][1]}, n);
      }
    } else {
      // complex64: unrolled over W with the host's nonzero mask (a list loop
      // measured 2 % slower on this HBM-bound form).
#pragma unroll
      for (int m = 0; m < 4; ++m)
#pragma unroll
        for (int n = 0; n < 4; ++n)
          if ((pw.nzmask >> (m * 4 + n)) & 1u)
            cfma(s, cx<R> {pw.w[m * 4 + n][0], pw.w[m * 4 + n][1]}, ld<R>(N + (n * 4 + m) * 9 + ad));
    }
    st(q + e, s);
  }
}

// Largest gamma-basis term count for which build_nprime takes the basis form:
// ng terms cost ng x 9 complex FMA per N' block, the row form four x 9.
constexpr int kNprimeCliffTerms = 4;

// N'_w[m][l] = sum_n W[m][n] N[n][l] into the w-th scratch slot.  With
// `cliff` (b.cl filled for these projectors, few terms) each block is built
// from the gamma basis instead, N'_w[m][l] = sum_k qc[w][k][m] N[perm[k][m]][l]:
// cl.ng iterations that every lane takes, where the row form skips W's zero
// entries per lane and so runs all four n for a warp whose lanes hold
// different rows m.
template <class R, class S, int TPS, int NW>
__device__ __forceinline__ void build_nprime(const BaryonSpin<R> &b, const S *N, S *np, int sub, bool cliff = false)
{
  for (int e = sub; e < 16 * NW; e += TPS) {
    const int w = e / 16, blk = e % 16, m = blk / 4, l = blk % 4;
    const ProjOperand<R> &pw = b.proj[w];
    S *dst = np + (size_t)w * 144 + blk * 9;
    if (cliff) {
      const CliffordSet<R> &cl = b.cl;
      cx<R> o[9];
#pragma unroll
      for (int k = 0; k < 9; ++k) o[k] = czero<R>();
#pragma unroll 1
      for (int k = 0; k < cl.ng; ++k) {
        const S *src = N + (cl.perm[k][m] * 4 + l) * 9;
        const cx<R> c {cl.qc[w][k][m][0], cl.qc[w][k][m][1]};
#pragma unroll
        for (int q = 0; q < 9; ++q) cfma(o[q], c, ld<R>(src + q));
      }
#pragma unroll
      for (int k = 0; k < 9; ++k) st(dst + k, o[k]);
    } else if (pw.is_perm) {
      const S *src = N + (pw.perm[m] * 4 + l) * 9;
#pragma unroll
      for (int k = 0; k < 9; ++k) st(dst + k, mul_phase(ld<R>(src + k), pw.ph[m]));
    } else {
      cx<R> o[9];
#pragma unroll
      for (int k = 0; k < 9; ++k) o[k] = czero<R>();
#pragma unroll
      for (int n = 0; n < 4; ++n) {
        if (!((pw.nzmask >> (m * 4 + n)) & 1u)) continue;
        const cx<R> wv {pw.w[m * 4 + n][0], pw.w[m * 4 + n][1]};
#pragma unroll
        for (int k = 0; k < 9; ++k) cfma(o[k], wv, ld<R>(N + (n * 4 + l) * 9 + k));
      }
#pragma unroll
      for (int k = 0; k < 9; ++k) st(dst + k, o[k]);
    }
  }
}

// Loop form: this thread's share of C (LPT (i, l) pairs).
template <class R, class S, int TPS>
__device__ __forceinline__ cx<R> loop_site(const BaryonSpin<R> &b, const S *A, const S *B, const S *q, int sub)
{
  using Ln = Lanes<TPS>;
  const int i = sub / Ln::TPI, l0 = (sub % Ln::TPI) * Ln::LPT;
  const int j = b.perm1[i];
  cx<R> d[9], qw[9];
#pragma unroll
  for (int k = 0; k < 9; ++k) d[k] = czero<R>();
#pragma unroll
  for (int lo = 0; lo < Ln::LPT; ++lo) {
    const int l = l0 + lo;
    cx<R> x[9], y[9];
    load9(x, A + (i * 4 + b.perm2[l]) * 9);
    load9(y, B + (j * 4 + l) * 9);
    // several pairs meet before Q: their phases relative to the first one's
    if (lo > 0) phase9(x, (b.ph2[0][l] - b.ph2[0][l0]) & 3u);
    wedge_acc(d, x, y);
  }
  load9(qw, q);
  return mul_phase(dot9(d, qw), (b.ph1[0][i] + b.ph2[0][l0]) & 3u);
}

// Triangle form over N' (16 blocks), one (i, l) pair per thread.
template <class R, class S>
__device__ __forceinline__ cx<R> triangle_site(const BaryonSpin<R> &b, const S *A, const S *B, const S *np, int sub)
{
  const int i = sub >> 2, l = sub & 3, j = b.perm1[i];
  cx<R> d[9];
#pragma unroll
  for (int k = 0; k < 9; ++k) d[k] = czero<R>();
  // Not unrolled: keeps one B block and one N' block live (register pressure).
#pragma unroll 1
  for (int m = 0; m < 4; ++m) {
    cx<R> bm[9], nn[9];
    load9(bm, B + (j * 4 + m) * 9);
    load9(nn, np + (m * 4 + l) * 9);
    wedge_acc(d, bm, nn);
  }
  cx<R> a[9];
  load9(a, A + (i * 4 + b.perm2[l]) * 9);
  return mul_phase(dot9(a, d), (b.ph1[0][i] + b.ph2[0][l]) & 3u);
}

// Triangle form with W one gamma matrix times a number (always so for
// baryon_two_point): N'[m][l] = coef i^ph[m] N[perm m][l], no N' buffer.
// LPT columns l per thread.
template <class R, class S, int TPS>
__device__ __forceinline__ cx<R> triangle_gamma_site(const BaryonSpin<R> &b, const S *A, const S *B, const S *N, int sub)
{
  using Ln = Lanes<TPS>;
  const CliffordSet<R> &cl = b.cl;
  const int i = sub / Ln::TPI, l0 = (sub % Ln::TPI) * Ln::LPT;
  const int j = b.perm1[i];
  const bool phased = cl.has_phase[0];
  cx<R> acc = czero<R>();
#pragma unroll
  for (int lo = 0; lo < Ln::LPT; ++lo) {
    const int l = l0 + lo;
    cx<R> d[9];
#pragma unroll
    for (int e = 0; e < 9; ++e) d[e] = czero<R>();
#pragma unroll 1
    for (int m = 0; m < 4; ++m) {
      cx<R> bm[9], nn[9];
      load9(bm, B + (j * 4 + m) * 9);
      load9(nn, N + (cl.perm[0][m] * 4 + l) * 9);
      if (phased) phase9(nn, cl.ph[0][m]);
      wedge_acc(d, bm, nn);
    }
    cx<R> a[9];
    load9(a, A + (i * 4 + b.perm2[l]) * 9);
    acc = cadd(acc, mul_phase(dot9(a, d), b.ph2[0][l]));
  }
  return cmul(cx<R> {cl.coef[0][0][0], cl.coef[0][0][1]}, mul_phase(acc, b.ph1[0][i]));
}

// Triangle form with a projector of rank r <= 2 (RankForm).  By bilinearity
// of the wedge, sum_m B[j][m] ^ N'[m][l] = sum_r X_r[j] ^ Y_r[l] with
//   X_r[j] = sum_m x_r[m] B[j][m],  Y_r[l] = sum_n y_r[n] N[n][l],
// and by the symmetry of the triple product
//   C = sum_{r,l} c2(l) Y_r[l] . sum_i c1(i) A[i][perm2 l] ^ X_r[perm1 i]:
// 4 r x 4 wedges and 4 r dots a site (1224 complex FMA for r = 2), where the N'
// form takes 64 wedges and 16 dots.
//
// Whether the factors are applied as unit-modulus phases: complex128 only (an
// FP64 add each instead of four FMA); the complex64 build, on packed FP32 FMAs,
// measured 2-4 % slower so.
template <class R> __device__ __forceinline__ bool rank_unit_form(const RankForm<R> &rk)
{
  return sizeof(R) == 8 && rk.unit;
}

// N colour entries of one combined block from entry `first` on (past the ninth: the ninth
// again): side 0, X_r from a row of B (blocks 9 apart); side 1, Y_r from a column of P_n
// (blocks 36 apart).  Part of a block: two terms' loads are in flight.
template <int N, class R, class S>
__device__ __forceinline__ void rank_entries(const RankForm<R> &rk, bool unit, int side, int r, const S *base, int stride,
                                             int first, cx<R> (&o)[N])
{
  int at[N];
#pragma unroll
  for (int t = 0; t < N; ++t) at[t] = N == 9 ? t : min(first + t, 8);
  if (unit) {
    const S *src = base + rk.idx[side][r][0] * stride;
#pragma unroll
    for (int t = 0; t < N; ++t) o[t] = mul_phase(ld<R>(src + at[t]), rk.ph[side][r][0]);
#pragma unroll 1
    for (int k = 1; k < rk.nnz; ++k) {
      src = base + rk.idx[side][r][k] * stride;
      const uint32_t ph = rk.ph[side][r][k];
#pragma unroll
      for (int t = 0; t < N; ++t) o[t] = cadd(o[t], mul_phase(ld<R>(src + at[t]), ph));
    }
    return;
  }
#pragma unroll
  for (int t = 0; t < N; ++t) o[t] = czero<R>();
#pragma unroll (N < 9 ? 2 : 1)
  for (int k = 0; k < rk.nnz; ++k) {
    const S *src = base + rk.idx[side][r][k] * stride;
    const cx<R> c {rk.c[side][r][k][0], rk.c[side][r][k][1]};
#pragma unroll
    for (int t = 0; t < N; ++t) cfma(o[t], c, ld<R>(src + at[t]));
  }
}
template <class R, class S>
__device__ __forceinline__ void rank_block(const RankForm<R> &rk, bool unit, int side, int r, const S *base, int stride,
                                           cx<R> (&o)[9])
{
  rank_entries<9>(rk, unit, side, r, base, stride, 0, o);
}

// Y_r[q] = sum_n y_r[n] N[n][q] at block r*4 + q of y.
template <class R, class S, int TPS>
__device__ __forceinline__ void build_rank_y(const RankForm<R> &rk, const S *N, S *y, int sub)
{
  for (int e = sub; e < 4 * rk.r; e += TPS) {
    cx<R> o[9];
    rank_block(rk, false, 1, e / 4, N + (e % 4) * 9, 36, o);
#pragma unroll
    for (int k = 0; k < 9; ++k) st(y + e * 9 + k, o[k]);
  }
}

// Gamma classes: the permutation of every Gamma(n) is r -> r ^ s for its class s,
// and within a class the (g5 Gamma(a))^T row phases factor as
//   ph(a, r) = beta_s(r) + alpha_a + 2 popcount(h_a & r)  (mod 4)
// with h_a running over 0..3 (Walsh functions): a sum over spin rows for the four
// members of a class is one phase per row and a four-point Walsh-Hadamard
// transform.
struct ClassWalsh {
  uint32_t beta;     // 2 bits per (s, r), index 4 s + r
  uint64_t member;   // 4 bits per (s, h), index 4 s + h
  uint32_t alpha;    // 2 bits per (s, h)
  bool ok;
};
CGB_HD constexpr ClassWalsh class_walsh()
{
  constexpr GammaTables G = build_gamma_tables();
  ClassWalsh w {0u, 0ull, 0u, true};
  for (int s = 0; s < 4; ++s) {
    int base = -1, seen = 0;
    for (int a = 0; a < 16; ++a) {
      if (G.perm[a][0] != s) continue;
      for (int r = 0; r < 4; ++r)
        if (G.perm[a][r] != (r ^ s)) w.ok = false;
      if (base < 0) {
        base = a;
        for (int r = 0; r < 4; ++r) w.beta |= (uint32_t)G.ph_g5g_t[a][r] << (2 * (4 * s + r));
      }
      int d[4] = {0, 0, 0, 0};
      for (int r = 0; r < 4; ++r) d[r] = (G.ph_g5g_t[a][r] - G.ph_g5g_t[base][r] + 4) & 3;
      const int alpha = d[0];
      const int h0 = ((d[1] - alpha + 4) & 3) >> 1, h1 = ((d[2] - alpha + 4) & 3) >> 1;
      for (int r = 0; r < 4; ++r) {
        const int pc = ((r & 1) & h0) + (((r >> 1) & 1) & h1);
        if (d[r] != ((alpha + 2 * pc) & 3)) w.ok = false;
      }
      const int h = h0 | (h1 << 1);
      if (seen & (1 << h)) w.ok = false;
      seen |= 1 << h;
      w.member |= (uint64_t)a << (4 * (4 * s + h));
      w.alpha |= (uint32_t)alpha << (2 * (4 * s + h));
    }
    if (seen != 15) w.ok = false;
  }
  return w;
}
static_assert(class_walsh().ok, "gamma classes must have the Walsh phase structure");
// The phases of a class's rows differ by signs only (every Gamma is real or imaginary).
CGB_HD constexpr bool class_phases_common(const ClassWalsh &w)
{
  for (int k = 0; k < 16; ++k)
    if ((((w.beta >> (2 * k)) ^ (w.beta >> (8 * (k / 4)))) & 1u) != 0) return false;
  return true;
}

// Lexicographic index ((t Lz + z) Ly + y) Lx + x of an even/odd-ordered site; -1
// without a lattice (the engines then skip the site and report it).
template <class R> __device__ __forceinline__ long long lexicographic(const OpParams<R> &p, long long site)
{
  const long long lx = p.latt[0], ly = p.latt[1], lz = p.latt[2], lt = p.latt[3];
  if (lx < 2 || ly < 1 || lz < 1 || lt < 1) return -1;
  const long long half = lx / 2;
  long long r = site / half;
  const long long xh = site - r * half;
  const long long y = r % ly;
  r /= ly;
  const long long z = r % lz;
  r /= lz;
  const long long t = r % lt, par = r / lt;
  const long long x = 2 * xh + ((par + t + z + y) & 1);
  return ((t * lz + z) * ly + y) * lx + x;
}

// ------------------------------------------------------------------ ops --
// Common compile-time configuration of an op: CW consumer warps (plus one
// producer warp), TPS threads per site, NST ring stages.
template <class R_, class S_, int CW_, int TPS_, int NST_> struct OpBase {
  using R = R_;
  using S = S_;
  using Params = OpParams<R_>;
  static constexpr int CW = CW_, TPS = TPS_, NST = NST_;
  static constexpr int SITES = CW_ * (32 / TPS_);
  static constexpr int THREADS = 32 * (CW_ + 1);
  static_assert(32 % TPS_ == 0, "a site's threads must sit in one warp");
};

// Bytes of n complex values of storage type S, rounded up to 16.
template <class S> constexpr int cbytes(int n) { return (int)((n * sizeof(S) + 15) / 16 * 16); }

// x . conj(y) over a colour block.  Complex64: packed FP32x2 FMAs on two
// accumulators, A = sum x.re y and B = sum x.im y (y as a pair, x broadcast),
// then (A.x + B.y, B.x - A.y): no operand needs reordering.
template <class R> __device__ __forceinline__ cx<R> conj_dot9(const cx<R> x[9], const cx<R> y[9])
{
  cx<R> t = czero<R>();
#pragma unroll
  for (int e = 0; e < 9; ++e) cfma_conj(t, x[e], y[e]);
  return t;
}
template <> __device__ __forceinline__ cx<float> conj_dot9<float>(const cx<float> x[9], const cx<float> y[9])
{
  float2 A = make_float2(0.f, 0.f), B = A;
#pragma unroll
  for (int e = 0; e < 9; ++e) {
    const float2 yv = make_float2(y[e].x, y[e].y);
    A = __ffma2_rn(yv, bcast2(x[e].x), A);
    B = __ffma2_rn(yv, bcast2(x[e].y), B);
  }
  return {A.x + B.y, B.x - A.y};
}

// All 16 x 16 meson gamma pairs per site, C[a][b] = meson_two_point(Gamma_a, Gamma_b)
// (include/meson.cuh:33-50 for every pair), written as a 256-entry block per
// site in lexicographic site order ((t*Lz + z)*Ly + y)*Lx + x for the
// momentum projection.  Every Gamma permutes spin rows by XOR with a class
// s = perm(0) in {0,1,2,3}.  Thread (s, i) of a site computes the 16 colour
// dots T[k][l] = P_i[i][k] . conj(P_j[i^s][l]) -- the 256 dots of the site
// exactly once -- then
//   V[b] = sum_l c_b(l) T[l ^ s_b][l]                    (all 16 Gamma_b)
//   C[a][b] += c_a(i) V[b]   for the four Gamma_a of class s,
// summed over the four threads i by a halving shuffle exchange.
// The permutation of every Gamma(n) is r -> r ^ s for its class s, and
// within a class the (g5 Gamma(a))^T row phases factor as
//   ph(a, r) = beta_s(r) + alpha_a + 2 popcount(h_a & r)  (mod 4)
// with h_a running over 0..3 (Walsh functions).  Hence the sum over spin
// rows r of the four members of a class is one phase i^beta per row and a
// four-point Walsh-Hadamard transform across the rows' threads, followed by
// i^alpha per member.  ClassWalsh holds, per (class s, Walsh index h), the
// member a and alpha, and beta per (s, r); built and checked at compile time.
// T[k][l] = sum_e x_k[e] conj(y_l[e]) for the four colour blocks x_k = xr[9k..]
// and y_l = yr[9l..] of one spin row each, with packed FP32x2 FMAs (two lanes
// of one instruction: (re, im) += (a.x, a.y) b.x and (a.y, -a.x) b.y), which
// halves the issue slots of the products.  Colour index outermost, so only
// one colour of each block is live; per element the FMA order is that of
// cfma_conj, so the sums are the same to the bit.
// NK consecutive colour blocks of the spin row (xr[9k..] for k < NK): the
// half-row form serves a site split over two threads.  NL < 4 takes the
// first NL blocks of yr.
template <int NK, int NL = 4>
__device__ __forceinline__ void conj_products_f32x2(cx<float> (&T)[NK][NL], const float2 *xr, const float2 *yr)
{
  float2 acc[NK][NL];
#pragma unroll
  for (int k = 0; k < NK; ++k)
#pragma unroll
    for (int l = 0; l < NL; ++l) acc[k][l] = make_float2(0.f, 0.f);
#pragma unroll 3  // fully unrolled, the loads of later colours run ahead and spill at 128 registers
  for (int e = 0; e < 9; ++e) {
    float2 a[NK], ar[NK], b[NL];
#pragma unroll
    for (int k = 0; k < NK; ++k) {
      a[k] = xr[k * 9 + e];
      ar[k] = make_float2(a[k].y, -a[k].x);
    }
#pragma unroll
    for (int l = 0; l < NL; ++l) b[l] = yr[l * 9 + e];
#pragma unroll
    for (int l = 0; l < NL; ++l) {
      const float2 bx = make_float2(b[l].x, b[l].x), by = make_float2(b[l].y, b[l].y);
#pragma unroll
      for (int k = 0; k < NK; ++k) {
        acc[k][l] = __ffma2_rn(a[k], bx, acc[k][l]);
        acc[k][l] = __ffma2_rn(ar[k], by, acc[k][l]);
      }
    }
  }
#pragma unroll
  for (int k = 0; k < NK; ++k)
#pragma unroll
    for (int l = 0; l < NL; ++l) T[k][l] = {acc[k][l].x, acc[k][l].y};
}


// SPLIT selects the layout [t][pair half][site][128 pairs] (pairs 0-127 and
// 128-255 of a timeslice in separate planes) that the tensor-core projection
// streams as contiguous 8-site tiles; otherwise [t][site][256 pairs].
// PRODUCTS: store the 256 spin-colour products
//   T[i][j][k][l] = sum_c S1[i][k][c] conj(S2[j][l][c])
// instead of the Gamma pairs, product (i, j = i ^ s, k, l) at index
// (4 k + l) * 16 + 4 s + i.  Each pair is a signed sum of 16 products, the same
// at every site, so a linear consumer (the momentum projection) forms the pairs
// once from its sums (map_pairs in kernels_momentum.cu).
template <class R, class S, int CW, int NST, bool SPLIT = false, bool PRODUCTS = false>
struct MesonAllGammaOp : OpBase<R, S, CW, 16, NST> {
  static constexpr int NIN = 2, OUT_ELEMS = 256;
  static_assert(sizeof(R) == 4, "complex128: MesonPairs (ops_site.cuh)");
  __device__ static long long sites_per_slice(const OpParams<R> &p)
  {
    return (long long)p.latt[0] * p.latt[1] * p.latt[2];
  }
  // Destination of site `d` (lexicographic index, 0 <= d < volume): the start
  // of its 256 pairs, or with SPLIT of its first 128 (the second 128 follow
  // one timeslice plane later).
  __device__ static S *out_ptr(const OpParams<R> &p, long long d, S *base)
  {
    if constexpr (SPLIT) {
      const long long v3 = sites_per_slice(p), t = d / v3;
      return base + (d + t * v3) * 128;
    } else {
      return base + d * OUT_ELEMS;
    }
  }

  __device__ static long long out_index(const OpParams<R> &p, long long site) { return lexicographic(p, site); }

  __device__ static void site(const OpParams<R> &ps_, const S *const *in, int sub, S *out)
  {
    constexpr GammaTables G = build_gamma_tables();
    constexpr ClassWalsh CW8 = class_walsh();
    const int s = sub >> 2, i = sub & 3, j = i ^ s;
    cx<R> T[4][4];
    conj_products_f32x2(T, in[0] + i * 36, in[1] + j * 36);
    if constexpr (PRODUCTS) {
      if (!out) return;
#pragma unroll
      for (int k = 0; k < 4; ++k)
#pragma unroll
        for (int l = 0; l < 4; ++l) {
          const int g = (k * 4 + l) * 16 + sub;
          S *dst;
          if constexpr (SPLIT) dst = out + (g >> 7) * sites_per_slice(ps_) * 128 + (g & 127);
          else dst = out + g;
          *dst = S {T[k][l].x, T[k][l].y};
        }
      return;
    }
    // V[b] = i^beta_s(i) sum_l (g5 Gamma(b))^T-phase(l) T[perm_b(l)][l]
    const uint32_t beta = (CW8.beta >> (2 * (4 * s + i))) & 3u;
    cx<R> V[16];
#pragma unroll
    for (int b = 0; b < 16; ++b) {
      cx<R> v = czero<R>();
#pragma unroll
      for (int l = 0; l < 4; ++l) v = cadd(v, mul_phase(T[G.perm[b][l]][l], G.ph_g5g_t[b][l]));
      V[b] = mul_phase(v, beta);
    }
    // Walsh-Hadamard over the row bits of i (lanes ^1, ^2), reduce-scattering b:
    // this thread ends with X[h][kk] for b = 8 i0 + 4 i1 + kk.
    const uint32_t i0 = i & 1, i1 = (i >> 1) & 1;
    cx<R> Y0[8], Y1[8];  // Walsh bit h0 = 0, 1 for b in [8 i0, 8 i0 + 8)
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const cx<R> own = i0 ? V[8 + k] : V[k], send = i0 ? V[k] : V[8 + k];
      const cx<R> recv = shfl_xor(send, 1);
      Y0[k] = cadd(own, recv);
      const cx<R> d = {own.x - recv.x, own.y - recv.y};
      Y1[k] = {flip_sign(d.x, i0), flip_sign(d.y, i0)};
    }
    cx<R> X[4][4];
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
#pragma unroll
      for (int h0 = 0; h0 < 2; ++h0) {
        const cx<R> *Y = h0 ? Y1 : Y0;
        const cx<R> own = i1 ? Y[4 + kk] : Y[kk], send = i1 ? Y[kk] : Y[4 + kk];
        const cx<R> recv = shfl_xor(send, 2);
        X[h0][kk] = cadd(own, recv);
        const cx<R> d = {own.x - recv.x, own.y - recv.y};
        X[2 + h0][kk] = {flip_sign(d.x, i1), flip_sign(d.y, i1)};
      }
    }
    const int b0 = 8 * i0 + 4 * i1;
    if (!out) return;  // a site past the end of the tile (the shuffles above still ran)
#pragma unroll
    for (int h = 0; h < 4; ++h) {
      const int idx = 4 * s + h;
      const int a = (int)((CW8.member >> (4 * idx)) & 15u);
      const uint32_t alpha = (CW8.alpha >> (2 * idx)) & 3u;
      S *dst;  // 32-byte aligned
      if constexpr (SPLIT) dst = out + (a >> 3) * sites_per_slice(ps_) * 128 + (a & 7) * 16 + b0;
      else dst = out + a * 16 + b0;
      st2(dst, mul_phase(X[h][0], alpha), mul_phase(X[h][1], alpha));
      st2(dst + 2, mul_phase(X[h][2], alpha), mul_phase(X[h][3], alpha));
    }
  }
};

} // namespace cgb
