// Per-call ops for ring_kernel (engine_warp.cuh): one baryon contraction
// type, one meson Gamma pair, or all 16 partners of one meson Gamma.
//
// Complex128 baryon wedges and the all-partner meson dots run in fixed point on the
// integer pipe where the site's values allow it (fixed.cuh), in FP64 otherwise;
// complex64 runs on packed FP32 FMAs.
#pragma once

#include "ops_fused.cuh"

namespace cgb {

template <class R_, class S_, int CW_, int TPS_, int NST_, int MINB> struct RingOp {
  using R = R_;
  using S = S_;
  using Params = OpParams<R_>;
  static constexpr int CW = CW_, TPS = TPS_, NST = NST_, MIN_CTAS = MINB;
  static constexpr int NOUT = 1, EXTRA_BYTES = 0;
  static constexpr bool CHANGES_INPUT = false;
  static constexpr int DIRECT = 0;  // fields after NIN that are not staged: site() reads them from memory
};

// Loop form (IK_JL_NM, IL_JK_NM).
template <class R, class S, int CW, int TPS, int NST, int MINB>
struct BaryonLoopOp : RingOp<R, S, CW, TPS, NST, MINB> {
  static constexpr int NIN = 3, EXTRA_BYTES = cbytes<S>(9);
  static constexpr bool CHANGES_INPUT = sizeof(R) == 8;
  __device__ static cx<R> site(const OpParams<R> &p, S *const *in, S *scratch, int sub, bool live)
  {
    const BaryonSpin<R> &b = p.b;
    build_q<R, S, TPS, 1>(b, in[2], scratch, sub);
    __syncwarp();
    if constexpr (sizeof(R) == 8) {
      static_assert(TPS == 16, "one (i, l) pair per thread");
      FixedScales fs;
      const int i = sub >> 2, l = sub & 3, xb = i * 4 + b.perm2[l], yb = b.perm1[i] * 4 + l;
      if (fields_to_fixed(in[0], in[1], sub, live, fs, [&](uint32_t x, uint32_t y) {
            return site_cover(wedge_cover(block_word(x, xb), block_word(y, yb)));
          })) {
        // all wedges of the site have one scale: they meet as integers, entry e of
        // the sum with thread e, which multiplies it by Q's
        const int4 *x = reinterpret_cast<const int4 *>(in[0]) + xb * 9;
        const int4 *y = reinterpret_cast<const int4 *>(in[1]) + yb * 9;
        // Gamma entries: one common power of i, and signs
        const uint32_t common = (b.ph1[0][0] & 1u) + (b.ph2[0][0] & 1u);
        const bool minus = ((b.ph1[0][i] ^ b.ph2[0][l]) & 2u) != 0;
        const longlong2 d = fixed_wedge_scatter(x, y, minus, sub);
        cx<double> v = czero<double>();
        if (sub < 9) {
          const cx<double> z = fixed_entry(d, sub, fs);
          cfma(v, z, ld<double>(scratch + sub));
        }
        return mul_phase(v, common);
      }
    }
    return loop_site<R, S, TPS>(b, in[0], in[1], scratch, sub);
  }
};

// Triangle form (the other four types), N' = W N materialised (any projector).
template <class R, class S, int CW, int NST, int MINB>
struct BaryonTriOp : RingOp<R, S, CW, 16, NST, MINB> {
  static constexpr int NIN = 3, EXTRA_BYTES = cbytes<S>(144) + 16;  // +16: bank stagger
  static constexpr bool CHANGES_INPUT = sizeof(R) == 8;
  __device__ static cx<R> site(const OpParams<R> &p, S *const *in, S *scratch, int sub, bool live)
  {
    const BaryonSpin<R> &b = p.b;
    build_nprime<R, S, 16, 1>(b, in[2], scratch, sub, b.cl.ng <= kNprimeCliffTerms);
    __syncwarp();
    if constexpr (sizeof(R) == 8) {
      FixedScales fs;
      const int i = sub >> 2, l = sub & 3, j = b.perm1[i];
      if (fields_to_fixed(in[1], scratch, sub, live, fs, [&](uint32_t x, uint32_t y) {
            uint32_t c = 0;
#pragma unroll
            for (int m = 0; m < 4; ++m) c |= wedge_cover(block_word(x, j * 4 + m), block_word(y, m * 4 + l));
            return c;
          })) {
        const int4 *B = reinterpret_cast<const int4 *>(in[1]), *np = reinterpret_cast<const int4 *>(scratch);
        cx<double> d[9], a[9];
        fixed_wedge_sum(0, 4, fs, [&](int m, const int4 *&x, const int4 *&y) {
          x = B + (j * 4 + m) * 9;
          y = np + (m * 4 + l) * 9;
          return false;
        }, d);
        load9(a, in[0] + (i * 4 + b.perm2[l]) * 9);
        return mul_phase(dot9(a, d), (b.ph1[0][i] + b.ph2[0][l]) & 3u);
      }
    }
    return triangle_site<R, S>(b, in[0], in[1], scratch, sub);
  }
};

// Triangle form, W a multiple of one gamma matrix.
template <class R, class S, int CW, int TPS, int NST, int MINB>
struct BaryonTriGammaOp : RingOp<R, S, CW, TPS, NST, MINB> {
  static constexpr int NIN = 3;
  static constexpr bool CHANGES_INPUT = sizeof(R) == 8;
  __device__ static cx<R> site(const OpParams<R> &p, S *const *in, S *, int sub, bool live)
  {
    const BaryonSpin<R> &b = p.b;
    if constexpr (sizeof(R) == 8) {
      static_assert(TPS == 16, "one (i, l) pair per thread");
      const CliffordSet<R> &cl = b.cl;
      FixedScales fs;
      const int i = sub >> 2, l = sub & 3, j = b.perm1[i];
      if (fields_to_fixed(in[1], in[2], sub, live, fs, [&](uint32_t x, uint32_t y) {
            uint32_t c = 0;
#pragma unroll
            for (int m = 0; m < 4; ++m)
              c |= wedge_cover(block_word(x, j * 4 + m), block_word(y, cl.perm[0][m] * 4 + l));
            return c;
          })) {
        const int4 *B = reinterpret_cast<const int4 *>(in[1]), *N = reinterpret_cast<const int4 *>(in[2]);
        cx<double> d[9], a[9];
        // the gamma matrix's entries differ by signs
        fixed_wedge_sum(0, 4, fs, [&](int m, const int4 *&x, const int4 *&y) {
          x = B + (j * 4 + m) * 9;
          y = N + (cl.perm[0][m] * 4 + l) * 9;
          return ((cl.ph[0][m] ^ cl.ph[0][0]) & 2u) != 0;
        }, d);
        load9(a, in[0] + (i * 4 + b.perm2[l]) * 9);
        const cx<R> v = mul_phase(dot9(a, d), (b.ph1[0][i] + b.ph2[0][l] + cl.ph[0][0]) & 3u);
        return cmul(cx<R> {cl.coef[0][0][0], cl.coef[0][0][1]}, v);
      }
    }
    return triangle_gamma_site<R, S, TPS>(b, in[0], in[1], in[2], sub);
  }
};

// Triangle form, W of rank 1 or 2: eight threads a site.  Thread (r, l) with two
// factors, thread (half of the rows, l) with one: the wedges A[i][perm2 l] ^
// X_r[perm1 i] over its rows i, then one dot with Y_r[l].  Complex64 writes X over
// P_j's blocks (X_r[j] at block 4 r + j).  Complex128 reads P_j and P_n, every block of
// which is used about once, from memory: with one field and X of a site in shared
// memory 12 warps of 4 sites share an SM, 1.45 ms at 24^3 x 32 with two factors, 1.02
// with one of two terms a vector, 1.69 with one of four.  Before the two had kernels of
// their own it was 1.49 with two; without the L2 prefetch of the fields read from memory
// 1.52; with P_j staged too, 8 warps, 1.73.
template <class R, class S, int CW, int NST, int MINB, bool TWO>
struct BaryonTriRankOp : RingOp<R, S, CW, 8, NST, MINB> {
  static constexpr bool CHANGES_INPUT = true;
  static constexpr int DIRECT = sizeof(R) == 8 ? 2 : 0, NIN = 3 - DIRECT;
  static constexpr int EXTRA_BYTES = DIRECT ? cbytes<S>(72) + 16 : 0;  // X; +16: bank stagger
  __device__ static cx<R> site(const OpParams<R> &p, S *const *in, S *, int sub, bool live)
  {
    return contract(p, in[0], in[1], in[2], in[1], sub, live);
  }
  __device__ static cx<R> site(const OpParams<R> &p, S *const *in, const S *const *more, S *scratch, int sub, bool live)
  {
    return contract(p, in[0], more[0], more[1], scratch, sub, live);
  }
  __device__ static cx<R> contract(const OpParams<R> &p, S *A, const S *B, const S *N, S *X, int sub, bool live)
  {
    const BaryonSpin<R> &b = p.b;
    const RankForm<R> &rk = b.rk;
    const FusedSpin f = b.fu;
    const bool unit = rank_unit_form(rk);
    // One factor, from memory: threads sub and sub + 4 form five entries of X[sub] and Y[sub]
    // each (the ninth twice in effect), half the loads and FP64 adds.
    constexpr int NE = 5;
    const int e0 = (sub >> 2) * NE;
    {
      const S *row = B + (sub & 3) * 36;
      if constexpr (DIRECT && !TWO) {  // two threads share a block
        cx<R> o[NE];
        rank_entries<NE>(rk, unit, 0, 0, row, 9, e0, o);
#pragma unroll
        for (int k = 0; k < NE; ++k)
          if (e0 + k < 9) st(X + (sub & 3) * 9 + e0 + k, o[k]);
      } else {
        cx<R> o[9];
        rank_block(rk, unit, 0, TWO ? sub >> 2 : 0, row, 9, o);
        __syncwarp();  // B, whose place X may take, has been read
        if (TWO || sub < 4) {
#pragma unroll
          for (int k = 0; k < 9; ++k) st(X + sub * 9 + k, o[k]);
        }
      }
    }
    __syncwarp();
    const int l = sub & 3, r = TWO ? sub >> 2 : 0, k0 = TWO ? 0 : (sub >> 2) * 2, k1 = TWO ? 4 : k0 + 2;
    const int s = l ^ ((f.s >> 2) & 3), s1 = f.s & 3, turn = (f.rows >> 8) & 7;
    cx<R> d[9];
    bool done = false;
    if constexpr (sizeof(R) == 8) {
      FixedScales fs;
      S *own = X + (TWO ? sub : sub & 3) * 9;
      const double2 *blk[3] = {A + sub * 9, A + (sub + 8) * 9, own};
      uint32_t near[3];
      bool ok = fixed_scales<8, 2>(blk, fs, near);
      const uint32_t w0 = cover_word(near[0]), w1 = cover_word(near[1]), wx = cover_word(near[2]);
      uint32_t c = 0;
#pragma unroll 2
      for (int k = k0; k < k1; ++k) {
        const int i = two_bits(f.rows, 2 * k), xb = i * 4 + s;
        const uint32_t lo = __shfl_sync(0xffffffffu, w0, xb & 7, 8), hi = __shfl_sync(0xffffffffu, w1, xb & 7, 8);
        c |= wedge_cover(xb & 8 ? hi : lo, __shfl_sync(0xffffffffu, wx, r * 4 + (i ^ s1), 8));
      }
      if constexpr (!TWO) c |= __shfl_xor_sync(0xffffffffu, c, 4);  // the two halves of the rows meet in the dot with Y
      ok = wedges_covered(c) && ok;
      done = __all_sync(0xffffffffu, ok || !live);
      if (done) {
        block_to_fixed(reinterpret_cast<int4 *>(A + sub * 9), blk[0], fs, 0);
        block_to_fixed(reinterpret_cast<int4 *>(A + (sub + 8) * 9), blk[1], fs, 0);
        if (TWO || sub < 4) block_to_fixed(reinterpret_cast<int4 *>(own), own, fs, 1);
        __syncwarp();
        const int4 *Af = reinterpret_cast<const int4 *>(A), *Xf = reinterpret_cast<const int4 *>(X);
        fixed_wedge_sum(k0, k1, fs, [&](int k, const int4 *&x, const int4 *&y) {
          const int i = two_bits(f.rows, 2 * k);
          x = Af + (i * 4 + s) * 9;
          y = Xf + (r * 4 + (i ^ s1)) * 9;
          return k < turn;
        }, d);
      }
    }
    if (!done) {
#pragma unroll
      for (int k = 0; k < 9; ++k) d[k] = czero<R>();
      bool minus = false;
#pragma unroll 1
      for (int k = k0; k < k1; ++k) {
        if ((k < turn) != minus) {
          minus = !minus;
#pragma unroll
          for (int e = 0; e < 9; ++e) d[e] = {-d[e].x, -d[e].y};
        }
        const int i = two_bits(f.rows, 2 * k);
        cx<R> x[9], y[9];
        load9(x, A + (i * 4 + s) * 9);
        load9(y, X + (r * 4 + (i ^ s1)) * 9);
        wedge_acc(d, x, y);
      }
      if (minus) {
#pragma unroll
        for (int e = 0; e < 9; ++e) d[e] = {-d[e].x, -d[e].y};
      }
    }
    cx<R> y[9];
    if constexpr (DIRECT && !TWO) {
      cx<R> o[NE];
      rank_entries<NE>(rk, unit, 1, 0, N + l * 9, 36, e0, o);
#pragma unroll
      for (int k = 0; k < NE; ++k) {
        const cx<R> p = shfl_xor(o[k], 4);
        y[k] = sub & 4 ? p : o[k];
        if (NE + k < 9) y[NE + k < 9 ? NE + k : 0] = sub & 4 ? o[k] : p;
      }
    } else {
      rank_block(rk, unit, 1, r, N + l * 9, 36, y);
    }
    const cx<R> v = mul_phase(signed_by(dot9(d, y), f.neg, l), f.out & 3u);
    const R sc = unit ? rk.scale : R(1);
    return {v.x * sc, v.y * sc};
  }
};

// Meson two-point: C = sum_{i,l} c1(i) c2(l) sum_ad A[i][perm2 l][ad] conj(B[perm1 i][l][ad])
// with c from (g5 Gamma)^T (include/meson.cuh:33-50).
template <class R, class S, int CW, int TPS, int NST, int MINB>
struct MesonOp : RingOp<R, S, CW, TPS, NST, MINB> {
  static constexpr int NIN = 2;
  __device__ static cx<R> site(const OpParams<R> &p, S *const *in, S *, int sub, bool)
  {
    using Ln = Lanes<TPS>;
    const MesonSpin<R> &m = p.m;
    const int i = sub / Ln::TPI, l0 = (sub % Ln::TPI) * Ln::LPT;
    const int j = m.perm1[i];
    cx<R> acc = czero<R>();
#pragma unroll
    for (int lo = 0; lo < Ln::LPT; ++lo) {
      const int l = l0 + lo;
      const S *x = in[0] + (i * 4 + m.perm2[l]) * 9;
      const S *y = in[1] + (j * 4 + l) * 9;
      cx<R> t = czero<R>();
#pragma unroll
      for (int k = 0; k < 9; ++k) cfma_conj(t, ld<R>(x + k), ld<R>(y + k));
      acc = cadd(acc, mul_phase(t, m.ph2[l]));
    }
    return mul_phase(acc, m.ph1[i]);
  }
};

// meson_all_{source,sink}_two_point: one Gamma fixed, all 16 of the other slot.
//   source (Gamma_ij fixed): Z[k][l] = sum_i c1(i) A[i][k] . conj(B[perm1 i][l])
//   sink (Gamma_kl fixed):   Z[i][j] = sum_l c2(l) A[i][perm2 l] . conj(B[j][l])
//   out_g = sum_r c_g(r) Z[r ^ s][r] (source) or Z[r][r ^ s] (sink), s the class of Gamma_g
// Thread (a, b) of a site's 16 forms the four dots over the row r for the summed
// index a and b = k (or j); two halving steps over a leave Z's entry of row r = a
// and other index b with it, and the four threads of one class s = a ^ b meet in a
// Walsh-Hadamard transform of two steps, after which each holds one output: 10 FP
// adds a thread where summing all 16 outputs took 96.
template <class R, class S, int CW, int NST, int MINB, bool SOURCE>
struct MesonAllOp : RingOp<R, S, CW, 16, NST, MINB> {
  static constexpr int NIN = 2, NOUT = 16;
  static constexpr bool CHANGES_INPUT = sizeof(R) == 8;
  __device__ static int output(const OpParams<R> &, int sub)
  {
    constexpr ClassWalsh W = class_walsh();
    const int a = sub >> 2, s = a ^ (sub & 3);
    return (int)((W.member >> (4 * (4 * s + a))) & 15u);
  }
  __device__ static cx<R> site(const OpParams<R> &p, S *const *in, S *, int sub, bool live)
  {
    constexpr ClassWalsh W = class_walsh();
    const int a = sub >> 2, b = sub & 3, s = a ^ b;
    // the fixed block and the four of the other field, `step` blocks apart
    const int own = SOURCE ? a * 4 + b : b * 4 + a;
    const int first = SOURCE ? p.m.perm1[a] * 4 : p.m.perm2[a], step = SOURCE ? 1 : 4;
    cx<R> T[4];
    bool done = false;
    if constexpr (sizeof(R) == 8) {
      FixedScales fs;
      const double2 *blk[2] = {in[0] + sub * 9, in[1] + sub * 9};
      const bool ok = fixed_pair_scales(blk[0], blk[1], live, fs);
      done = __all_sync(0xffffffffu, ok || !live);
      if (done) {
        block_to_fixed(reinterpret_cast<int4 *>(in[0] + sub * 9), blk[0], fs, 0);
        block_to_fixed(reinterpret_cast<int4 *>(in[1] + sub * 9), blk[1], fs, 1);
        __syncwarp();
        const int up = fs.E[0] + fs.E[1] - 2 * 1023 - 54;
        const int4 *x = reinterpret_cast<const int4 *>(in[SOURCE ? 0 : 1]) + own * 9;
        const int4 *y = reinterpret_cast<const int4 *>(in[SOURCE ? 1 : 0]) + first * 9;
        int4 xv[9];
#pragma unroll
        for (int k = 0; k < 9; ++k) xv[k] = x[k];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const cx<double> t = fixed_conj_dot(xv, y + r * step * 9, up);
          T[r] = SOURCE ? t : conj(t);
        }
      }
    }
    if (!done) {
      cx<R> x[9], y[9];
      load9(x, in[SOURCE ? 0 : 1] + own * 9);
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        load9(y, in[SOURCE ? 1 : 0] + (first + r * step) * 9);
        T[r] = SOURCE ? conj_dot9<R>(x, y) : conj_dot9<R>(y, x);
      }
    }
    const uint32_t ph = SOURCE ? p.m.ph1[a] : p.m.ph2[a];
#pragma unroll
    for (int r = 0; r < 4; ++r) T[r] = mul_phase(T[r], ph);
    const bool hi = a & 2, odd = a & 1;
    cx<R> h[2];
#pragma unroll
    for (int r = 0; r < 2; ++r) h[r] = cadd(hi ? T[2 + r] : T[r], shfl_xor(hi ? T[r] : T[2 + r], 8));
    cx<R> u = cadd(odd ? h[1] : h[0], shfl_xor(odd ? h[0] : h[1], 4));  // Z of row r = a
    u = mul_phase(u, (W.beta >> (2 * (4 * s + a))) & 3u);
    cx<R> o = shfl_xor(u, 5);  // (a ^ 1, b ^ 1)
    u = odd ? cx<R> {o.x - u.x, o.y - u.y} : cadd(u, o);
    o = shfl_xor(u, 10);
    u = hi ? cx<R> {o.x - u.x, o.y - u.y} : cadd(u, o);
    return mul_phase(u, (W.alpha >> (2 * (4 * s + a))) & 3u);
  }
};

// All 256 meson Gamma pairs of a site in complex128: what the momentum projection sums.
//   pair(a, b) = sum_{i,l} c_a(i) c_b(l) A[i][l ^ u] . conj(B[i ^ s][l])
// for the Gammas a of class s and b of class u.  Thread (s, u) of a site's 16 forms
// the class's 16 products and turns them into its 16 pairs by Walsh-Hadamard steps
// over l and i in registers; no thread needs another's products.  It stores pair
// (ha, hb) of its classes at (4 ha + hb) 16 + 4 s + u, so that the site's 16 threads
// store 256 bytes at a time (pair_of_class gives the Gammas).
//
// Products and sums are integers where the site allows it (fixed.cuh): a product of
// blocks stays below 2^60.2 units, four of them below 2^62.2; they are rounded to
// quarter units before the four rows meet.
//
// Alone 0.77 ms at 18 x 15 x 20 x 28, bound by the integer pipes.  The projection of 125
// momenta is off by 2.5e-16 of its norm against extended precision at 18 x 15 x 20 x 2 (3.2e-16 in FP64;
// test_extended_precision_gpu.py).
struct MesonPairs {
  // o[ha][hb] += the Walsh-Hadamard sums w over l of row i's four products.  In FP64 row 0
  // begins the sums instead of being added to zero, and so does the first pair of a row: 64
  // adds of 224 less on the pipe that bounds it (integers: a branch costs more).
  template <class V> __device__ __forceinline__ static void add_row(V (&o)[4][4], const V (&w)[4], int i)
  {
    if constexpr (std::is_floating_point<V>::value) {
      if (i == 0) {  // uniform
#pragma unroll
        for (int ha = 0; ha < 4; ++ha)
#pragma unroll
          for (int h = 0; h < 4; ++h) o[ha][h] = w[h];
        return;
      }
    }
#pragma unroll
    for (int ha = 0; ha < 4; ++ha) {
      const bool minus = __popc(ha & i) & 1;  // uniform
#pragma unroll
      for (int h = 0; h < 4; ++h) o[ha][h] = minus ? o[ha][h] - w[h] : o[ha][h] + w[h];
    }
  }
  // w += the sums over l = 2 hi and 2 hi + 1 of products t
  template <class V> __device__ __forceinline__ static void add_pair(V (&w)[4], const V (&t)[2], int hi)
  {
    const V a = t[0] + t[1], b = t[0] - t[1];
    if (std::is_floating_point<V>::value && hi == 0) {
      w[0] = w[2] = a;
      w[1] = w[3] = b;
      return;
    }
    w[0] += a;
    w[1] += b;
    w[2] += hi ? -a : a;
    w[3] += hi ? -b : b;
  }
  template <class V> __device__ __forceinline__ static void quarter(V (&w)[4])
  {
    if constexpr (std::is_integral<V>::value) {
#pragma unroll
      for (int h = 0; h < 4; ++h) w[h] = (w[h] + 2) >> 2;
    }
  }
  template <class V> __device__ __forceinline__ static V signed_if(V v, bool minus) { return minus ? -v : v; }

  template <class V, class Dot>
  __device__ __forceinline__ static void pairs(int s, int u, V (&re)[4][4], V (&im)[4][4], Dot dot)
  {
    constexpr ClassWalsh W = class_walsh();
    static_assert(class_phases_common(W), "a class's phases differ by signs");
#pragma unroll
    for (int ha = 0; ha < 4; ++ha)
#pragma unroll
      for (int h = 0; h < 4; ++h) re[ha][h] = im[ha][h] = V(0);
#pragma unroll 1
    for (int i = 0; i < 4; ++i) {
      V x[4], y[4];
#pragma unroll
      for (int h = 0; h < 4; ++h) x[h] = y[h] = V(0);
      const uint32_t bs = (W.beta >> (2 * (4 * s + i))) ^ (W.beta >> (8 * s));
#pragma unroll
      for (int hi = 0; hi < 2; ++hi) {  // the products of l = 2 hi, 2 hi + 1
        V tx[2], ty[2];
#pragma unroll
        for (int lo = 0; lo < 2; ++lo) {
          const int l = 2 * hi + lo;
          dot((i * 4 + (l ^ u)) * 9, ((i ^ s) * 4 + l) * 9, tx[lo], ty[lo]);
          const bool minus = ((bs ^ (W.beta >> (2 * (4 * u + l))) ^ (W.beta >> (8 * u))) & 2u) != 0;
          tx[lo] = signed_if(tx[lo], minus);
          ty[lo] = signed_if(ty[lo], minus);
        }
        add_pair(x, tx, hi);
        add_pair(y, ty, hi);
      }
      quarter(x);
      quarter(y);
      add_row(re, x, i);
      add_row(im, y, i);
    }
  }

  template <class V, class Make>
  __device__ __forceinline__ static void store(int s, int u, const V (&re)[4][4], const V (&im)[4][4], double2 *dst,
                                               Make make)
  {
    constexpr ClassWalsh W = class_walsh();
    const uint32_t common = (W.beta >> (8 * s)) + (W.beta >> (8 * u));
#pragma unroll
    for (int ha = 0; ha < 4; ++ha)
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        const uint32_t ph = (common + (W.alpha >> (2 * (4 * s + ha))) + (W.alpha >> (2 * (4 * u + h)))) & 3u;
        const cx<double> v = mul_phase(cx<double> {make(re[ha][h]), make(im[ha][h])}, ph);
        dst[(4 * ha + h) * 16 + 4 * s + u] = make_double2(v.x, v.y);
      }
  }

  // in: the site's fields, which are changed; ready(): called when they have been read,
  // before the pairs go to dst.
  template <class Ready>
  __device__ static void site(double2 *const (&in)[2], int sub, bool live, double2 *dst, Ready ready)
  {
    const int s = sub >> 2, u = sub & 3;
    FixedScales fs;
    const bool ok = fixed_pair_scales(in[0] + sub * 9, in[1] + sub * 9, live, fs);
    if (__all_sync(0xffffffffu, ok || !live)) {
#pragma unroll 1
      for (int q = 0; q < 2; ++q)
        block_to_fixed(reinterpret_cast<int4 *>((q ? in[1] : in[0]) + sub * 9), (q ? in[1] : in[0]) + sub * 9, fs, q);
      __syncwarp();
      const int4 *A = reinterpret_cast<const int4 *>(in[0]), *B = reinterpret_cast<const int4 *>(in[1]);
      long long re[4][4], im[4][4];
      pairs(s, u, re, im, [&](int a, int b, long long &x, long long &y) {
        FixedSum sx, sy;
        fixed_conj_sums(sx, sy, A + a, B + b);
        x = sx.units();
        y = sy.units();
      });
      const int up = fs.E[0] + fs.E[1] - 2 * 1023 - 52;
      ready();
      store(s, u, re, im, dst, [&](long long v) { return fixed_value(v, up); });
    } else {
      double re[4][4], im[4][4];
      pairs(s, u, re, im, [&](int a, int b, double &x, double &y) {
        cx<double> t = czero<double>();
#pragma unroll
        for (int k = 0; k < 9; ++k) cfma_conj(t, ld<double>(in[0] + a + k), ld<double>(in[1] + b + k));
        x = t.x;
        y = t.y;
      });
      ready();
      store(s, u, re, im, dst, [](double v) { return v; });
    }
  }
};

// The Gamma pair 16 a + b stored at `at` by MesonPairs.
__device__ __forceinline__ int pair_of_class(int at)
{
  constexpr ClassWalsh W = class_walsh();
  const int s = (at >> 2) & 3, u = at & 3, ha = at >> 6, hb = (at >> 4) & 3;
  return (int)((W.member >> (4 * (4 * s + ha))) & 15u) * 16 + (int)((W.member >> (4 * (4 * u + hb))) & 15u);
}

} // namespace cgb
