// Colour wedges of complex128 blocks on the integer pipe.
//
// The FP64 pipe issues one warp instruction in 64 cycles per scheduler (2 lanes an
// SM and cycle), IMAD.WIDE (32 x 32 + 64 -> 64 bits) one in about 4.2.  So a wedge,
// 36 complex products, is summed in 64-bit integers: every value v of a site's
// field is the fixed-point number (h 2^28 + l) 2^(E - 55), |h| <= 2^28,
// |l| <= 2^27, E the exponent of the field's largest value at that site, and a
// real product is three IMAD.WIDE (h h' into one sum, h l' + l h' into another)
// where it was one DFMA: 13 cycles instead of 64.  The sums of up to 32 products
// stay below 2^62 and are exact; they join, are rounded and become a double once
// per result.
//
// Scales.  An entry [a][d] of a colour block has the scale 2^(E + r_a + c_d): E the
// exponent of the field's largest value at the site, r and c of the colour rows
// and columns, common to both fields (every term of a wedge's entry then has one
// scale).  Colour rows or columns of very different size so keep their bits.
//
// Accuracy.  A value is off by at most 2^-55 of its scale (cut off; exact down to an
// eighth of it), and the dropped l l' and the last rounding leave a wedge sum off by
// about half a unit of 2^-54 of the two scales.  A small result therefore loses bits
// that FP64 would keep, unless it is made of values near their scales.  So the integer
// form is taken only where every sum has at least one product of two values that are
// no more than kFixedNear powers of two below their scales (wedge_cover, fixed_pair_scales,
// FixedDotBlock::near): then its error, entry by entry and against the sum of the sizes
// of its products, is no larger than what FP64 leaves.  In exact arithmetic on the host,
// rms over the sites accepted, sums of four wedges (of two): Gaussian blocks 1.9e-17
// (2.8e-17) against 6.0e-17 in FP64; blocks near a multiple of the unit matrix, the rest
// 0.35, 0.25 and 0.18 as large, 3.6e-17, 4.6e-17 and 5.5e-17 (5.5e-17, 6.4e-17 and
// 6.9e-17) against 7.5e-17, 8.0e-17 and 8.3e-17 (7.1e-17, 7.4e-17 and 7.7e-17); with
// 0.09 no site is accepted.  With 2 for kFixedNear 4 to 5 % of Gaussian sites have a sum
// of two wedges that is refused, with 3 none of 3000.
// Also every value must be finite and all exponents leave room for the
// products; otherwise the warp takes the FP64 form for its sites.  In the norm, against
// extended precision (test_extended_precision_gpu.py): all types 1.5e-16, one call a type
// 1.8e-16, all partners of a meson Gamma 1.2e-16, in FP64 2.2e-16, 2.3e-16 and 1.8e-16.
#pragma once

#include "common.cuh"

namespace cgb {

constexpr int kFixedMinExp = 723, kFixedMaxExp = 1323;  // biased: 2^-300 to 2^300
constexpr int kFixedNear = 3;     // powers of two between a value that covers a sum and its scale
constexpr int kFixedColour = 60;  // and between colour rows or columns at most
// Powers of two that fixed_value may apply: a sum is 1 to 2^62 units.
constexpr int kFixedMinUp = -1022, kFixedMaxUp = 960;
// A wedge's: two fields' scales, two colour rows and two columns (one row and one column have
// the field's scale).
static_assert(2 * kFixedMinExp - 2 * 1023 - 54 - 4 * kFixedColour >= kFixedMinUp &&
              2 * kFixedMaxExp - 2 * 1023 - 54 <= kFixedMaxUp, "a wedge could leave the exponents of a double");
constexpr int kFixedMinDot = 200;  // least biased exponent of a dot block's largest value

// The largest of a site's TPS threads' values.
template <int TPS> __device__ __forceinline__ int group_max(int v)
{
#pragma unroll
  for (int o = TPS / 2; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// The same for two values of 16 bits at a time.
template <int TPS> __device__ __forceinline__ void group_max(int &lo, int &hi)
{
  unsigned int v = ((unsigned int)lo & 0xffffu) | (unsigned int)hi << 16;
#pragma unroll
  for (int o = TPS / 2; o > 0; o >>= 1) v = __vmaxs2(v, __shfl_xor_sync(0xffffffffu, v, o));
  lo = (short)v;
  hi = (int)v >> 16;
}

// The scales of one site: entry [a][d] of field f at 2^(E[f] + r[a] + c[d] - 1023).
struct FixedScales {
  int E[2], r[3], c[3];
};

// Scales of the fields whose blocks this thread reads, over the site's TPS
// threads; false if they do not suit the integer form.
// blk: NA of the first field, then of the second (none: one field).
// near: the entries of each block near their scale, a bit each.
template <int TPS, int NA, int N>
__device__ __forceinline__ bool fixed_scales(const double2 *const (&blk)[N], FixedScales &f, uint32_t (&near)[N])
{
  f.E[0] = f.E[1] = 0;
  // High words without the sign: biased exponent from bit 20 on.  Differences of them
  // wrap only where the values are refused anyway.
  unsigned int e[N][9];
#pragma unroll
  for (int n = 0; n < N; ++n) {
    unsigned int most = 0;
#pragma unroll
    for (int k = 0; k < 9; ++k) {
      const double2 v = blk[n][k];
      e[n][k] = max((unsigned int)__double2hiint(v.x) & 0x7fffffffu, (unsigned int)__double2hiint(v.y) & 0x7fffffffu);
      most = max(most, e[n][k]);
    }
    f.E[n < NA ? 0 : 1] = max(f.E[n < NA ? 0 : 1], (int)(most >> 20));
  }
  group_max<TPS>(f.E[0], f.E[1]);
  if (NA == N) f.E[1] = f.E[0];
  const bool ok = min(f.E[0], f.E[1]) >= kFixedMinExp && max(f.E[0], f.E[1]) <= kFixedMaxExp;
  // Rows, then columns in the scales of the rows.  Zeros (0) lie more than kFixedColour
  // below every scale.
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    f.r[a] = -kFixedColour;
#pragma unroll
    for (int n = 0; n < N; ++n)
      f.r[a] = max(f.r[a], (int)(max(max(e[n][3 * a], e[n][3 * a + 1]), e[n][3 * a + 2]) >> 20) - f.E[n < NA ? 0 : 1]);
  }
  group_max<TPS>(f.r[0], f.r[1]);
  f.r[2] = group_max<TPS>(f.r[2]);
#pragma unroll
  for (int n = 0; n < N; ++n)
#pragma unroll
    for (int k = 0; k < 9; ++k) e[n][k] -= (unsigned int)f.r[k / 3] << 20;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    f.c[d] = -kFixedColour;
#pragma unroll
    for (int n = 0; n < N; ++n)
      f.c[d] = max(f.c[d], (int)(max(max(e[n][d], e[n][3 + d]), e[n][6 + d]) >> 20) - f.E[n < NA ? 0 : 1]);
  }
  group_max<TPS>(f.c[0], f.c[1]);
  f.c[2] = group_max<TPS>(f.c[2]);
#pragma unroll
  for (int n = 0; n < N; ++n) {
    unsigned int far = 0;  // the sign of what an entry lies above the limit, entry by entry
#pragma unroll
    for (int k = 8; k >= 0; --k)
      far = __funnelshift_l(e[n][k] - ((unsigned int)(f.E[n < NA ? 0 : 1] + f.c[k % 3] - kFixedNear) << 20), far, 1);
    near[n] = ~far & 0x1ffu;
  }
  return ok;
}

// What of block w's nine colour entries is near its scale, by the thread of the site's
// 16 that holds the block.
__device__ __forceinline__ uint32_t block_word(uint32_t w, int block) { return __shfl_sync(0xffffffffu, w, block, 16); }

// A block's near bits for wedge_cover: the columns rotated by one in the lower half and
// by two in the upper one, rows 0 to 2 and again 0 and 1.
__device__ __forceinline__ uint32_t cover_word(uint32_t near)
{
  const uint32_t c1 = ((near >> 1) & 0333u) | ((near & 0111u) << 2), c2 = ((near >> 2) & 0111u) | ((near & 0333u) << 1);
  return ((c1 | c1 << 9) & 0x7fffu) | ((c2 | c2 << 9) & 0x7fffu) << 16;
}
// Which entries [a][d] of x ^ y have a product of two near values, x[a + r][d + c] and
// y[a + 2 r][d + 2 c], r, c = 1 or 2: bit 3 a + d of either half (c = 1 and c = 2).
__device__ __forceinline__ uint32_t wedge_cover(uint32_t x, uint32_t y)
{
  const uint32_t z = __byte_perm(y, 0, 0x1032);
  return ((x >> 3) & (z >> 6)) | ((x >> 6) & (z >> 3));
}
// The covers of a site's 16 threads, or-ed (both sites of the warp at once).
__device__ __forceinline__ uint32_t site_cover(uint32_t c)
{
  const uint32_t at = threadIdx.x & 16u;
  return __reduce_or_sync(0xffffffffu, ((c | c >> 16) & 0x1ffu) << at) >> at;
}
// Whether the covers of a sum's wedges, or-ed, leave no entry out.
__device__ __forceinline__ bool wedges_covered(uint32_t c) { return ((c | c >> 16) & 0x1ffu) == 0x1ffu; }

// Scales for dots of the blocks of two fields, one of each per thread of a site's 16: one
// scale per field, colours being summed over.  False if they do not suit the integer form.
// A class of meson pairs sums 16 products of blocks, every block of either field once, so
// two near values meet at a colour entry if more than 16 of the site's 32 blocks are near
// there; usually the first entry shows it.
__device__ __forceinline__ bool fixed_pair_scales(const double2 *x, const double2 *y, bool live, FixedScales &f)
{
  int e[2][9];  // high words without the sign
#pragma unroll
  for (int n = 0; n < 2; ++n) {
    int most = 0;
#pragma unroll
    for (int k = 0; k < 9; ++k) {
      const double2 v = n ? y[k] : x[k];
      e[n][k] = max(__double2hiint(v.x) & 0x7fffffff, __double2hiint(v.y) & 0x7fffffff);
      most = max(most, e[n][k]);
    }
    f.E[n] = group_max<16>(most >> 20);
  }
#pragma unroll
  for (int a = 0; a < 3; ++a) f.r[a] = f.c[a] = 0;
  const bool fits = min(f.E[0], f.E[1]) >= kFixedMinExp && max(f.E[0], f.E[1]) <= kFixedMaxExp;
  const uint32_t site = 0xffffu << (threadIdx.x & 16u);
  bool covered = false;
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    if (__all_sync(0xffffffffu, covered || !fits || !live)) break;
    const uint32_t a = __ballot_sync(0xffffffffu, e[0][k] >= (f.E[0] - kFixedNear) << 20);
    const uint32_t b = __ballot_sync(0xffffffffu, e[1][k] >= (f.E[1] - kFixedNear) << 20);
    covered = covered || __popc(a & site) + __popc(b & site) > 16;
  }
  return fits && covered;
}

// v as h 2^28 + l in units of 2^(E - 55).  The 53-bit significand, 3 bits up, goes
// down by E minus v's exponent (the PTX shift gives 0 from 64 on): exact down to 2^-3
// of the scale, cut off below; 15 instructions (28 with a rounded shift and clamps).
__device__ __forceinline__ int2 to_fixed(double v, int E)
{
  const long long bits = __double_as_longlong(v);
  const int hi = (int)(bits >> 32);
  const uint32_t d = (uint32_t)(E - ((hi >> 20) & 0x7ff));  // negative only where the result is not used
  const unsigned long long t =
    ((unsigned long long)(((uint32_t)hi & 0xfffffu) | 0x100000u) << 35) | ((unsigned long long)(uint32_t)bits << 3);
  unsigned long long u;
  asm("shr.u64 %0, %1, %2;" : "=l"(u) : "l"(t), "r"(d));
  const int h = (int)((u + (1ull << 27)) >> 28), l = (int)((uint32_t)u - ((uint32_t)h << 28));
  return hi < 0 ? make_int2(-h, -l) : make_int2(h, l);
}

// A colour block of field `field` to fixed point: (h, l) of re, then of im; dst may be blk.
__device__ __forceinline__ void block_to_fixed(int4 *dst, const double2 *blk, const FixedScales &f, int field)
{
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    const double2 v = blk[k];
    const int E = f.E[field] + f.r[k / 3] + f.c[k % 3];
    const int2 a = to_fixed(v.x, E), b = to_fixed(v.y, E);
    dst[k] = make_int4(a.x, a.y, b.x, b.y);
  }
}

// v 2^up.
__device__ __forceinline__ double fixed_value(long long v, int up)
{
  const double d = __ll2double_rn(v);
  return v == 0 ? 0.0 : __hiloint2double(__double2hiint(d) + (up << 20), __double2loint(d));
}

// Running sums of fixed-point products: high words' products, and the cross ones
// (2^-28 of a unit of the first).
struct FixedSum {
  long long hh, x;
  __device__ __forceinline__ void mac(int ah, int al, int bh, int bl)
  {
    hh += (long long)ah * bh;
    x += (long long)ah * bl;
    x += (long long)al * bh;
  }
  // In units of 2^(scale + scale - 54).
  __device__ __forceinline__ long long units() const { return hh + ((x + (1ll << 27)) >> 28); }
  // In units of 2^(scale + scale - 53).
  __device__ __forceinline__ long long half_units() const { return (hh + ((x + (1ll << 27)) >> 28) + 1) >> 1; }
  // In units of 2^(scale + scale - 54); `up` is that power of two.
  __device__ __forceinline__ double value(int up) const
  {
    return fixed_value(units(), up);
  }
};

// Row a of a sum of wedges x ^ y of converted blocks (see wedge_acc): three
// results at a time, so that their sums take 24 registers and not 72.
struct FixedWedgeRow {
  FixedSum re[3], im[3];
  __device__ __forceinline__ void clear()
  {
#pragma unroll
    for (int e = 0; e < 3; ++e) re[e] = im[e] = FixedSum {0, 0};
  }
  __device__ __forceinline__ void negate()
  {
#pragma unroll
    for (int e = 0; e < 3; ++e) {
      re[e] = FixedSum {-re[e].hh, -re[e].x};
      im[e] = FixedSum {-im[e].hh, -im[e].x};
    }
  }
  __device__ __forceinline__ void add(int a, const int4 *xp, const int4 *yp)
  {
    const int a1 = (a + 1) % 3, a2 = (a + 2) % 3;
    // half 0: x row a1 with y row a2, half 1: x row a2 with y row a1
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      int4 x[3], y[3];
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        x[k] = xp[3 * (half ? a2 : a1) + k];
        y[k] = yp[3 * (half ? a1 : a2) + k];
      }
#pragma unroll
      for (int e = 0; e < 3; ++e) {
        const int e1 = (e + 1) % 3, e2 = (e + 2) % 3;
        // + x[e1] y[e2] - x[e2] y[e1] in half 0, the signs exchanged in half 1
        term(e, x[e1], y[e2], half != 0);
        term(e, x[e2], y[e1], half == 0);
      }
    }
  }
  __device__ __forceinline__ void term(int e, int4 u, int4 v, bool minus)
  {
    const int4 n = make_int4(-u.x, -u.y, -u.z, -u.w);
    const int4 p = minus ? n : u, q = minus ? u : n;
    re[e].mac(p.x, p.y, v.x, v.y);
    re[e].mac(q.z, q.w, v.z, v.w);
    im[e].mac(p.x, p.y, v.z, v.w);
    im[e].mac(p.z, p.w, v.x, v.y);
  }
  // The sums as doubles: entry [a][e] multiplies the two other rows and columns.
  __device__ __forceinline__ void get(int a, cx<double> *out, const FixedScales &f) const
  {
    const int up = f.E[0] + f.E[1] - 2 * 1023 - 54 + f.r[(a + 1) % 3] + f.r[(a + 2) % 3];
#pragma unroll
    for (int e = 0; e < 3; ++e) {
      const int at = up + f.c[(e + 1) % 3] + f.c[(e + 2) % 3];
      out[e] = {re[e].value(at), im[e].value(at)};
    }
  }
};

// d = sum over k in [k0, k1) of (+-) x_k ^ y_k: pair(k, x, y) gives the converted
// blocks and returns whether the term is subtracted (the same for every thread).
template <class Pair>
__device__ __forceinline__ void fixed_wedge_sum(int k0, int k1, const FixedScales &f, Pair pair, cx<double> (&d)[9])
{
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    FixedWedgeRow w;
    w.clear();
    bool minus = false;  // w holds the negative of the sum so far
#pragma unroll 1
    for (int k = k0; k < k1; ++k) {
      const int4 *x, *y;
      if (pair(k, x, y) != minus) {
        w.negate();
        minus = !minus;
      }
      w.add(a, x, y);
    }
    if (minus) w.negate();
    w.get(a, d + 3 * a, f);
  }
}

// Sums of nine pairs of numbers over a site's 16 threads, entry e with thread e
// (threads 9-15 receive nothing): recursive halving of 16 slots, seven of them empty.
template <class V>
__device__ __forceinline__ void group_sum_scatter9(const V (&re)[9], const V (&im)[9], int sub, V &x, V &y)
{
  V a[8], b[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) {  // slots k and 8 + k: only slot 8 of the upper half is used
    const bool up = (sub & 8) != 0;
    const V sa = up ? re[k] : (k == 0 ? re[8] : V(0)), sb = up ? im[k] : (k == 0 ? im[8] : V(0));
    a[k] = (up ? (k == 0 ? re[8] : V(0)) : re[k]) + __shfl_xor_sync(0xffffffffu, sa, 8);
    b[k] = (up ? (k == 0 ? im[8] : V(0)) : im[k]) + __shfl_xor_sync(0xffffffffu, sb, 8);
  }
#pragma unroll
  for (int h = 4; h > 0; h >>= 1) {
    const bool up = (sub & h) != 0;
#pragma unroll
    for (int k = 0; k < h; ++k) {
      const V sa = up ? a[k] : a[h + k], sb = up ? b[k] : b[h + k];
      a[k] = (up ? a[h + k] : a[k]) + __shfl_xor_sync(0xffffffffu, sa, h);
      b[k] = (up ? b[h + k] : b[k]) + __shfl_xor_sync(0xffffffffu, sb, h);
    }
  }
  x = a[0];
  y = b[0];
}

// The wedges x ^ y of a site's 16 threads (one scale), negated where `minus`, summed:
// entry e with thread e, in half units (16 sums of up to 2^59 leave a bit to spare).
__device__ __forceinline__ longlong2 fixed_wedge_scatter(const int4 *x, const int4 *y, bool minus, int sub)
{
  long long re[9], im[9];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    FixedWedgeRow w;
    w.clear();
    w.add(a, x, y);
#pragma unroll
    for (int e = 0; e < 3; ++e) {
      const long long u = w.re[e].half_units(), v = w.im[e].half_units();
      re[3 * a + e] = minus ? -u : u;
      im[3 * a + e] = minus ? -v : v;
    }
  }
  longlong2 d;
  group_sum_scatter9(re, im, sub, d.x, d.y);
  return d;
}

// Entry e of a wedge sum held in half units as a double.
__device__ __forceinline__ cx<double> fixed_entry(longlong2 v, int e, const FixedScales &f)
{
  const int a = e / 3, c = e - 3 * a;
  int rows = 0, cols = 0;  // the two other rows and columns
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    if (k != a) rows += f.r[k];
    if (k != c) cols += f.c[k];
  }
  const int up = f.E[0] + f.E[1] - 2 * 1023 - 53 + rows + cols;
  return {fixed_value(v.x, up), fixed_value(v.y, up)};
}

// re + i im = x . conj(y) over two converted blocks (held in registers or memory).
template <class X> __device__ __forceinline__ void fixed_conj_sums(FixedSum &re, FixedSum &im, const X &x, const int4 *y)
{
  FixedSum minus {0, 0};
  re = im = FixedSum {0, 0};
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    const int4 u = x[k], v = y[k];
    re.mac(u.x, u.y, v.x, v.y);
    re.mac(u.z, u.w, v.z, v.w);
    im.mac(u.z, u.w, v.x, v.y);
    minus.mac(u.x, u.y, v.z, v.w);
  }
  im.hh -= minus.hh;
  im.x -= minus.x;
}
// The same as doubles, blocks of one scale each; up = 2^ of their scales - 54.
__device__ __forceinline__ cx<double> fixed_conj_dot(const int4 (&x)[9], const int4 *y, int up)
{
  FixedSum re, im;
  fixed_conj_sums(re, im, x, y);
  return {re.value(up), im.value(up)};
}

// A block of doubles held for several dots with converted blocks of one field: its
// entries' scales are the inverse of that field's colour scales, so that all nine
// products have one.
struct FixedDotBlock {
  int4 g[9];
  int E, up;
  uint32_t near;  // the entries near the scale; all of a block of zeros, whose dots are exact
  // The block's scale beside that of the field; false if the block does not suit the
  // integer form: a value is not finite, all are so small that denormal ones count, or
  // a dot could leave the exponents of a double (fixed_value tests nothing).  Its values
  // come from either form of the wedges, so they may be anything.
  __device__ __forceinline__ bool fits(const cx<double> (&v)[9], const FixedScales &f)
  {
    int most = 0;
    uint32_t any = 0;
    E = -8192;
#pragma unroll
    for (int k = 0; k < 9; ++k) {
      const int hx = __double2hiint(v[k].x) & 0x7fffffff, hy = __double2hiint(v[k].y) & 0x7fffffff, x = max(hx, hy) >> 20;
      any |= (uint32_t)(hx | hy) | (uint32_t)__double2loint(v[k].x) | (uint32_t)__double2loint(v[k].y);
      most = max(most, x);
      E = max(E, x ? x + f.r[k / 3] + f.c[k % 3] : -8192);
    }
    near = any ? 0u : 0x1ffu;
#pragma unroll
    for (int k = 0; k < 9; ++k) {
      const int x = max(__double2hiint(v[k].x) & 0x7fffffff, __double2hiint(v[k].y) & 0x7fffffff) >> 20;
      near |= (uint32_t)(x + f.r[k / 3] + f.c[k % 3] >= E - kFixedNear) << k;
    }
    up = E + f.E[0] - 2 * 1023 - 54;
    return any == 0 || (most < 2047 && most >= kFixedMinDot && up >= kFixedMinUp && up <= kFixedMaxUp);
  }
  __device__ __forceinline__ void set(const cx<double> (&v)[9], const FixedScales &f)
  {
#pragma unroll
    for (int k = 0; k < 9; ++k) {
      const int2 a = to_fixed(v[k].x, E - f.r[k / 3] - f.c[k % 3]), b = to_fixed(v[k].y, E - f.r[k / 3] - f.c[k % 3]);
      g[k] = make_int4(a.x, a.y, b.x, b.y);
    }
  }
  __device__ __forceinline__ cx<double> dot(const double2 *blk) const
  {
    const int4 *y = reinterpret_cast<const int4 *>(blk);
    FixedSum re {0, 0}, im {0, 0}, minus {0, 0};
#pragma unroll
    for (int k = 0; k < 9; ++k) {
      const int4 u = g[k], v = y[k];
      re.mac(u.x, u.y, v.x, v.y);
      minus.mac(u.z, u.w, v.z, v.w);
      im.mac(u.x, u.y, v.z, v.w);
      im.mac(u.z, u.w, v.x, v.y);
    }
    re.hh -= minus.hh;
    re.x -= minus.x;
    return {re.value(up), im.value(up)};
  }
};

} // namespace cgb
