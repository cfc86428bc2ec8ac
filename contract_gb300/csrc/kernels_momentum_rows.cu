// Fused all-gamma meson momentum projection, mixed form, one or many items:
// the spin-colour products of every site and the X and Y transforms of the
// separable projection in one kernel, the products never leaving registers.
//
// One persistent CTA of W warps per SM walks the (t, z) planes of every item,
// unit blockIdx.x, + gridDim.x, ..., and its planes' rows y one after another, W
// rows (a batch) at a time, one row a warp:
//
//   X  the warp goes along its row site by site.  A lane forms 8 of a site's 256
//      products T[i][j][k][l] = sum_c S1[i][k][c] conj(S2[j][l][c]) and adds
//      them, times the row's X phases, to its sums C = sum cos v, S = sum sin v
//      of every X group; at the end of the row G(+k) = C + i S, G(-k) = C - i S go
//      to shared memory.
//   Y  a thread per (product, nx) adds the batch's rows to H[q] += exp(i ky y) G(nx)
//      for every (nx, ny) pair q of that nx; H lives in the plane buffer (L2)
//      between the batches of a plane.
//
// momentum_finalize and batch_finalize_combined apply the Z transform.
//
// What bounds it: shared memory and FP32 together.  A site takes 9216 FMA for the
// products and 256 (2 + 8) for the X sums of nx in {-2..2}, about 97 cycles of an
// SM; the lane's 2 x 4 tile reads 6 values per 8 products and colour, of which
// lanes 2 m and 2 m + 1 share the four of S2 (one cycle instead of two where pairs
// of lanes read one address): 72 cycles a site, beside 18 for the copies.  Taken
// apart at 32^3 x 32 with 125 momenta, 211 cycles a site: products 138, X sums 21,
// Y 25, the batch's barrier 4, waiting for copies 23.  Handing every site's 256
// products to separate transform warps through shared memory (the form this one
// replaced: 8 site and 8 transform warps, or 16 and 8) cost a store, a load and a
// hand-off per product.  Before and after, with the finalisation, at 32^3 x 64:
//   momenta            125 two fields   27 two    27 one    125 one   zero alone
//   hand-off           1.784 ms         1.637     1.495     1.699     1.596
//   this kernel        1.598 ms         1.178     0.852     1.159     0.931
// A 4 x 4 tile of 16 lanes a site reads less shared memory but takes 255 registers
// (two warps a scheduler) and was slower: 0.94 ms against 0.76 at 32^3 x 32.
//
// One field for both propagators (SAME): T[j][i][l][k] = conj(T[i][j][k][l]), so
// 136 products do.  A half-warp forms them, at most 9 a lane, lanes 0-15 on the
// row's parity-0 sites and 16-31 on the parity-1 ones; the halves join at the
// row's end, where the transposed products' G(+-k) are conj(G(-+k)).
//
// Every mbarrier wait is bounded in wall time; a wait that runs out reports
// kDevErrWaitTimeout, raises the CTA's abort flag and returns.
#include <algorithm>

#include "engine.cuh"
#include "momentum.hpp"

namespace cgb {

namespace {

constexpr uint32_t kSiteBytes = 1152;  // complex64 propagator site
constexpr int kRowMax = 12;            // rows (warps) per CTA at most
// shared memory: barriers (full[W][stages], rows ready, rows consumed; abort flag at 504), then
constexpr size_t kRowTab = 512;                                                // phase tables
constexpr size_t kRowPh = kRowTab + sizeof(float2) * kMomBatchMaxExt * kMomMaxL;  // [q][row] Y phases (c, c, s, s)
constexpr size_t kRowQ = kRowPh + sizeof(float4) * kMomQChunk * kRowMax;          // pairs by slot
constexpr size_t kRowG = kRowQ + 256;                                           // G[W][slot][256]
constexpr int kRowMaxStages = 4;
static_assert((kRowMax * kRowMaxStages + 2) * 8 <= 504, "barriers overlap the abort flag");

__device__ __forceinline__ int item_of_unit(const MomBatchParams &p, int unit)
{
  int lo = 0, hi = p.n_items - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (p.items[mid].unit_begin <= unit) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// A row of the CTA's planes.
struct RowCursor {
  int unit, item, y;
  __device__ __forceinline__ void start(const MomBatchParams &p)
  {
    unit = blockIdx.x;
    y = 0;
    item = unit < p.total_units ? item_of_unit(p, unit) : 0;
  }
  __device__ __forceinline__ bool valid(const MomBatchParams &p) const { return unit < p.total_units; }
  __device__ __forceinline__ void advance(const MomBatchParams &p, int n)
  {
    y += n;
    while (unit < p.total_units && y >= p.items[item].latt[1]) {
      y -= p.items[item].latt[1];
      unit += gridDim.x;
      if (unit < p.total_units) item = item_of_unit(p, unit);
    }
  }
};

// A product T = sum_c x conj(y) as two packed sums: P = sum x (.) y and Q = sum
// swap(x) (.) y, T = (P.x + P.y, Q.x - Q.y).  Only x needs its halves exchanged.
struct PackedSum {
  float2 P, Q;
  __device__ __forceinline__ void add(float2 x, float2 xs, float2 y)
  {
    P = __ffma2_rn(x, y, P);
    Q = __ffma2_rn(xs, y, Q);
  }
  __device__ __forceinline__ float2 value() const { return make_float2(P.x + P.y, Q.x - Q.y); }
};
__device__ __forceinline__ float2 swapped(float2 v) { return make_float2(v.y, v.x); }

// The products of a lane: NP of them, formed from the site slots of S1 and S2,
// and where they go among a row's 256.
// UNROLL: colours in flight.
template <bool SAME, int UNROLL> struct LaneProducts;

// Lane 8 j + 2 i + h: rows (i, 2 h) and (i, 2 h + 1) against spin j.
template <int UNROLL> struct LaneProducts<false, UNROLL> {
  static constexpr int NP = 8, SITES = 1;  // sites a warp works on at a time
  int i, j, h;
  __device__ __forceinline__ void init(int lane)
  {
    h = lane & 1;
    i = (lane >> 1) & 3;
    j = lane >> 3;
  }
  __device__ __forceinline__ void form(const float2 *a, const float2 *b, float2 (&T)[NP]) const
  {
    const float2 *xr = a + (i * 4 + 2 * h) * 9, *yr = b + j * 36;
    PackedSum t[NP] = {};
#pragma unroll UNROLL
    for (int e = 0; e < 9; ++e) {
      float2 y[4];
#pragma unroll
      for (int l = 0; l < 4; ++l) y[l] = yr[l * 9 + e];
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const float2 x = xr[k * 9 + e], xs = swapped(x);
#pragma unroll
        for (int l = 0; l < 4; ++l) t[4 * k + l].add(x, xs, y[l]);
      }
    }
#pragma unroll
    for (int m = 0; m < NP; ++m) T[m] = t[m].value();
  }
  __device__ __forceinline__ int slot(int m) const  // product m: k = 2 h + m / 4, l = m % 4
  {
    return (8 * h + m) * 16 + 4 * (i ^ j) + i;
  }
};

// Lanes 0-11 of a half take two rows k0, k0 + 1 of an off-diagonal block
// T[X][Y], X < Y (lanes 2 m and 2 m + 1 the two halves of one block), and one of
// the entries (2, 2), (2, 3), (3, 3) of a diagonal block; lanes 12-15 rows 0 and
// 1 of the diagonal blocks, whose entry (1, 0) repeats (0, 1).
template <int UNROLL> struct LaneProducts<true, UNROLL> {
  static constexpr int NP = 9, SITES = 2;
  int X, Y, k0, E, ea, eb;
  __device__ __forceinline__ void init(int lane)
  {
    const int sub = lane & 15;
    if (sub < 12) {
      const int m = sub >> 1;
      X = m < 3 ? 0 : (m < 5 ? 1 : 2);
      Y = m < 3 ? m + 1 : (m < 5 ? m - 1 : 3);
      k0 = 2 * (sub & 1);
      E = sub / 3;
      ea = sub % 3 == 2 ? 3 : 2;
      eb = sub % 3 == 0 ? 2 : 3;
    } else {
      X = Y = sub - 12;
      k0 = 0;
      E = ea = eb = 0;  // unused
    }
  }
  __device__ __forceinline__ void form(const float2 *a, const float2 *, float2 (&T)[NP]) const
  {
    const float2 *xr = a + (X * 4 + k0) * 9, *yr = a + Y * 36, *ar = a + (E * 4 + ea) * 9, *br = a + (E * 4 + eb) * 9;
    PackedSum t[NP] = {};
#pragma unroll UNROLL
    for (int e = 0; e < 9; ++e) {
      float2 y[4];
#pragma unroll
      for (int l = 0; l < 4; ++l) y[l] = yr[l * 9 + e];
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const float2 x = xr[k * 9 + e], xs = swapped(x);
#pragma unroll
        for (int l = 0; l < 4; ++l) t[4 * k + l].add(x, xs, y[l]);
      }
      const float2 u = ar[e];
      t[8].add(u, swapped(u), br[e]);
    }
#pragma unroll
    for (int m = 0; m < NP; ++m) T[m] = t[m].value();
  }
  // Slots of product m and of its conjugate transpose; -1: not stored.
  __device__ __forceinline__ void slots(int m, int &own, int &conj) const
  {
    const int k = m < 8 ? k0 + (m >> 2) : ea, l = m < 8 ? (m & 3) : eb;
    const int i = m < 8 ? X : E, j = m < 8 ? Y : E, s = i ^ j;
    own = (4 * k + l) * 16 + 4 * s + i;
    conj = (4 * l + k) * 16 + 4 * s + j;
    const bool diag = i == j;
    if (diag && k == l) conj = -1;
    if (m < 8 && diag && l < k) own = conj = -1;
    if (m == 8 && X == Y) own = conj = -1;  // lanes 12-15 form no ninth product
  }
};

// Z: whether X group 0 is nx = 0 (a plain sum); NS: the other X groups; W: warps;
// UNROLL: colours of a product in flight.
template <int Z, int NS, bool SAME, int W, int UNROLL>
__global__ void __launch_bounds__(32 * W, 1)
  momentum_rows_kernel(const __grid_constant__ MomBatchParams p, const int nst)
{
  using LP = LaneProducts<SAME, UNROLL>;
  constexpr int NP = LP::NP, PX = Z + 2 * NS;  // PX rows of 256: nx = 0, then +-k of each group
  constexpr int NIN = SAME ? 1 : 2;
  constexpr uint32_t kStage = LP::SITES * NIN * kSiteBytes;
  extern __shared__ __align__(128) unsigned char smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint64_t *bars = reinterpret_cast<uint64_t *>(smem);
  uint64_t *full = bars + warp * nst, *ready = bars + W * nst, *consumed = ready + 1;
  volatile int *abort_flag = reinterpret_cast<volatile int *>(smem + 504);
  float2 *tab = reinterpret_cast<float2 *>(smem + kRowTab);
  float4 *ph = reinterpret_cast<float4 *>(smem + kRowPh);
  const uint8_t *qlist = reinterpret_cast<const PairOrder *>(smem + kRowQ)->list;
  const uint8_t *qstart = reinterpret_cast<const PairOrder *>(smem + kRowQ)->start;
  float2 *G = reinterpret_cast<float2 *>(smem + kRowG);  // [warp][PX][256]
  unsigned char *ring = reinterpret_cast<unsigned char *>(G + (size_t)W * PX * 256) + (size_t)warp * nst * kStage;

  if (lane == 0) {
    for (int s = 0; s < nst; ++s) mbar_init(&full[s], 1);
    if (warp == 0) {
      mbar_init(ready, W);
      mbar_init(consumed, W);
      *abort_flag = 0;
    }
    fence_barrier_init();
  }
  __syncwarp();

  const int hw = SAME ? lane >> 4 : 0;  // SAME: the half-warp's parity
  LP lp;
  lp.init(lane);

  // copies: this warp's rows are w, w + W, ... of the CTA's; a stage holds one
  // site of a row (parities in turn; lane q copies field q), or with SAME one of
  // each parity (lane par).  The row's addresses are worked out once.
  RowCursor fc;
  fc.start(p);
  fc.advance(p, warp);
  int fleft = 0, fstage = 0;       // copies left in the row
  const char *src0 = nullptr, *src1 = nullptr;  // the lane's next site, and the one after the next
  auto fetch = [&]() {  // the next copies into the next stage
    if (fleft == 0) {
      const MomBatchItem &it = p.items[fc.item];
      const int ly = it.latt[1], lz = it.latt[2], lt = it.latt[3], half = it.latt[0] >> 1;
      const int local = fc.unit - it.unit_begin, t = local / lz, z = local - t * lz;
      const long long row = (((long long)t * lz + z) * ly + fc.y) * half, other = (long long)lt * lz * ly * half;
      fleft = SAME ? half : 2 * half;
      src0 = it.in[SAME ? 0 : lane & 1] + (row + (SAME && (lane & 1) ? other : 0)) * kSiteBytes;
      src1 = SAME ? src0 + kSiteBytes : src0 + other * kSiteBytes;
    }
    if (lane == 0) mbar_arrive_expect_tx(&full[fstage], kStage);
    __syncwarp();
    if (lane < 2)
      bulk_g2s(ring + fstage * kStage + (uint32_t)lane * kSiteBytes, src0, kSiteBytes, &full[fstage]);
    const char *after = SAME ? src1 + kSiteBytes : src0 + kSiteBytes;
    src0 = src1;
    src1 = after;
    if (++fstage == nst) fstage = 0;
    if (--fleft == 0) fc.advance(p, W);
  };
  int in_flight = 0;
  for (; in_flight < nst && fc.valid(p); ++in_flight) fetch();
  // while they come: the tables that all warps read
  for (int e = threadIdx.x; e < p.n_ext * kMomMaxL; e += 32 * W) tab[e] = p.tab[e / kMomMaxL][e % kMomMaxL];
  for (int e = threadIdx.x; e < kMomQChunk * kRowMax; e += 32 * W) ph[e] = make_float4(0.f, 0.f, 0.f, 0.f);
  if (threadIdx.x < sizeof(p.pairs) / 4)
    reinterpret_cast<uint32_t *>(smem + kRowQ)[threadIdx.x] = reinterpret_cast<const uint32_t *>(&p.pairs)[threadIdx.x];
  __syncthreads();

  int cstage = 0;
  uint32_t cphase = 0;
  // Gives up: every copy this warp issued and has not waited for lands (or its
  // wait runs out) before the warp leaves.
  auto give_up = [&]() {
    if (lane == 0) {
      *abort_flag = 1;
      report(p.status, kDevErrWaitTimeout, (unsigned int)fc.unit);
      for (int s = cstage, n = 0, ps = cphase; n < in_flight; ++n) {
        mbar_wait_bounded(&full[s], ps, kWaitLimitNs / 8);
        if (++s == nst) {
          s = 0;
          ps ^= 1u;
        }
      }
    }
  };
  auto wait_all = [&](uint64_t *bar, uint32_t parity) -> bool {
    if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
    const bool ok = mbar_wait_bounded(bar, parity, kWaitLimitNs);
    return __all_sync(0xffffffffu, ok) && !*abort_flag;
  };

  RowCursor base;
  base.start(p);
  for (uint32_t batch = 0; base.valid(p); ++batch) {
    RowCursor my = base;
    my.advance(p, warp);
    if (my.valid(p)) {
      const MomBatchItem &it = p.items[my.item];
      const int lx = it.latt[0], lz = it.latt[2], local = my.unit - it.unit_begin;
      const int t = local / lz, z = local - t * lz, y = my.y;
      const float2 *tx = tab + it.tx * kMomMaxL;
      const int odd = (t + z + y) & 1;  // parity-0 sites have x = 2 xh + odd, parity-1 ones 2 xh + 1 - odd
      int pair[NS > 0 ? NS : 1], kx[NS > 0 ? NS : 1];  // k 2 xh mod Lx and k mod Lx of each group
#pragma unroll
      for (int s = 0; s < NS; ++s) {
        pair[s] = 0;
        kx[s] = p.gx_k[Z + s] % lx;
      }
      float2 c0[NP], cc[NS > 0 ? NS : 1][NP], cs[NS > 0 ? NS : 1][NP];
#pragma unroll
      for (int m = 0; m < NP; ++m) {
        c0[m] = make_float2(0.f, 0.f);
#pragma unroll
        for (int s = 0; s < NS; ++s) cc[s][m] = cs[s][m] = make_float2(0.f, 0.f);
      }
      const int iters = SAME ? lx >> 1 : lx;
#pragma unroll 1
      for (int n = 0; n < iters; ++n) {
        if (!wait_all(&full[cstage], cphase)) {
          give_up();
          return;
        }
        const float2 *a = reinterpret_cast<const float2 *>(ring + cstage * kStage + hw * kSiteBytes);
        float2 T[NP];
        lp.form(a, a + kSiteBytes / 8, T);
        if (++cstage == nst) {
          cstage = 0;
          cphase ^= 1u;
        }
        --in_flight;
        __syncwarp();  // every lane has read the stage that the next copies fill
        if (fc.valid(p)) {
          fetch();
          ++in_flight;
        }
        if (Z) {
#pragma unroll
          for (int m = 0; m < NP; ++m) c0[m] = __fadd2_rn(c0[m], T[m]);
        }
#pragma unroll
        for (int s = 0; s < NS; ++s) {
          const int up = ((SAME ? hw : n & 1) ^ odd) ? kx[s] : 0;
          const int at = pair[s] + up < lx ? pair[s] + up : pair[s] + up - lx;
          const float2 e = tx[at];
          const float2 c2 = make_float2(e.x, e.x), s2 = make_float2(e.y, e.y);
#pragma unroll
          for (int m = 0; m < NP; ++m) {
            cc[s][m] = __ffma2_rn(T[m], c2, cc[s][m]);
            cs[s][m] = __ffma2_rn(T[m], s2, cs[s][m]);
          }
          if (SAME || (n & 1)) {
            pair[s] += 2 * kx[s];
            if (pair[s] >= lx) pair[s] -= lx;
            if (pair[s] >= lx) pair[s] -= lx;
          }
        }
      }
      // the previous batch's rows have been used
      if (batch > 0 && !wait_all(consumed, (batch - 1) & 1u)) {
        give_up();
        return;
      }
      float2 *row = G + (size_t)warp * PX * 256;
      if constexpr (SAME) {
        // The halves of the warp join: the lower one takes products 0 .. NH - 1
        // of each lane, the upper one the rest.
        constexpr int NH = (NP + 1) / 2;
        auto join = [&](const float2 (&v)[NP], int m) {
          const float2 lo = v[m], hi = NH + m < NP ? v[NH + m < NP ? NH + m : 0] : make_float2(0.f, 0.f);
          const float2 send = hw ? lo : hi, keep = hw ? hi : lo;
          return make_float2(keep.x + __shfl_xor_sync(0xffffffffu, send.x, 16),
                             keep.y + __shfl_xor_sync(0xffffffffu, send.y, 16));
        };
        auto put = [&](int sl, int m, float2 plus, float2 minus, bool both) {
          const int mm = m + (hw ? NH : 0);
          if (mm >= NP) return;
          int own, cj;
          lp.slots(mm, own, cj);
          if (own >= 0) {
            row[sl * 256 + own] = plus;
            if (both) row[(sl + 1) * 256 + own] = minus;
          }
          if (cj >= 0) {  // conj(T): G'(+k) = conj(G(-k))
            row[sl * 256 + cj] = make_float2(minus.x, -minus.y);
            if (both) row[(sl + 1) * 256 + cj] = make_float2(plus.x, -plus.y);
          }
        };
#pragma unroll
        for (int m = 0; m < NH; ++m) {
          if (Z) {
            const float2 v = join(c0, m);
            put(0, m, v, v, false);
          }
#pragma unroll
          for (int s = 0; s < NS; ++s) {
            const float2 c = join(cc[s], m), sn = join(cs[s], m);
            put(Z + 2 * s, m, make_float2(c.x - sn.y, c.y + sn.x), make_float2(c.x + sn.y, c.y - sn.x), true);
          }
        }
      } else {
#pragma unroll
        for (int m = 0; m < NP; ++m) {
          const int own = lp.slot(m);
          if (Z) row[own] = c0[m];
#pragma unroll
          for (int s = 0; s < NS; ++s) {
            const float2 c = cc[s][m], sn = cs[s][m];
            row[(Z + 2 * s) * 256 + own] = make_float2(c.x - sn.y, c.y + sn.x);
            row[(Z + 2 * s + 1) * 256 + own] = make_float2(c.x + sn.y, c.y - sn.x);
          }
        }
      }
      if (lane < p.nq) {
        const int ly = it.latt[1];
        const float2 e = tab[it.ty * kMomMaxL + ((p.q_ny[lane] * y) % ly + ly) % ly];
        ph[lane * kRowMax + warp] = make_float4(e.x, e.x, e.y, e.y);
      }
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(ready);
    // Y: this batch's rows, plane by plane; a thread's (nx slot, product) pairs
    // are the same in every batch, so a plane's H goes through memory by itself.
    // The sums of a plane that goes on are on their way while the rows get ready.
    constexpr int ROUNDS = (PX * 256 + 32 * W - 1) / (32 * W), QB = 5;
    float2 held[ROUNDS][QB];
    {
      const MomBatchItem &it = p.items[base.item];
      const float2 *planes = it.planes + (size_t)(base.unit - it.unit_begin) * p.nq * 256;
#pragma unroll
      for (int rd = 0; rd < ROUNDS; ++rd) {
        const int u = threadIdx.x + rd * 32 * W, sl = min(u >> 8, PX), q0 = qstart[sl], q1 = sl < PX ? qstart[sl + 1] : q0;
#pragma unroll
        for (int c = 0; c < QB; ++c)
          held[rd][c] = base.y > 0 && q0 + c < q1 ? planes[(size_t)qlist[q0 + c] * 256 + (u & 255)]
                                                  : make_float2(0.f, 0.f);
      }
    }
    if (!wait_all(ready, batch & 1u)) {
      give_up();
      return;
    }
    RowCursor rc = base;
    for (int r = 0; r < W && rc.valid(p);) {
      const MomBatchItem &it = p.items[rc.item];
      const int n = min(W - r, it.latt[1] - rc.y);
      const bool begins = rc.y == 0;
      float2 *planes = it.planes + (size_t)(rc.unit - it.unit_begin) * p.nq * 256;
#pragma unroll
      for (int rd = 0; rd < ROUNDS; ++rd) {
        const int u = threadIdx.x + rd * 32 * W;
        if (u >= PX * 256) break;
        const int sl = u >> 8, g = u & 255, q0 = qstart[sl], q1 = qstart[sl + 1];
        float2 v[W], iv[W];  // the rows' values and i times them
#pragma unroll
        for (int k = 0; k < W; ++k) {
          v[k] = k >= r && k < r + n ? G[((size_t)k * PX + sl) * 256 + g] : make_float2(0.f, 0.f);
          iv[k] = make_float2(-v[k].y, v[k].x);
        }
        auto step = [&](float2 h, int q) {
          const float4 *e = ph + q * kRowMax;
#pragma unroll
          for (int k = 0; k < W; ++k) {
            const float4 w = e[k];
            h = __ffma2_rn(v[k], make_float2(w.x, w.y), h);
            h = __ffma2_rn(iv[k], make_float2(w.z, w.w), h);
          }
          planes[(size_t)q * 256 + g] = h;
        };
#pragma unroll
        for (int c = 0; c < QB; ++c)
          if (q0 + c < q1) step(begins ? make_float2(0.f, 0.f) : held[rd][c], qlist[q0 + c]);
        for (int c = q0 + QB; c < q1; ++c)
          step(begins ? make_float2(0.f, 0.f) : planes[(size_t)qlist[c] * 256 + g], qlist[c]);
      }
      r += n;
      rc.advance(p, n);
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(consumed);
    base.advance(p, W);
  }
}

template <int Z, int NS, bool SAME> cudaError_t launch_rows(const Job &job, const MomBatchParams &p)
{
  // Twelve warps have 168 registers; the one-field form of five slots holds 90
  // sums a lane and spills there (0.649 ms at 32^3 x 32, 0.541 with eight warps).
  // Two fields and up to three slots, and one field and one slot, leave room to unroll the
  // products' colour loop (0.543 -> 0.474 ms, 0.627 -> 0.595 and 0.369 -> 0.359; two fields
  // and five slots 0.758 -> 0.830).
  constexpr int W = SAME && NS >= 2 ? 8 : 12, UNROLL = NS == 0 || (!SAME && NS == 1) ? 9 : 3;
  constexpr size_t kMax = 232448;
  constexpr size_t stage = (size_t)W * 2 * kSiteBytes, fixed = kRowG + sizeof(float2) * 256 * W * (Z + 2 * NS);
  constexpr int stages = std::min<int>(kRowMaxStages, (kMax - fixed) / stage);
  static_assert(stages >= 2, "fewer than two stages fit");
  constexpr size_t smem = fixed + stages * stage;
  static int attr_set[64] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev >= 64 || !attr_set[dev]) {
    e = cudaFuncSetAttribute(momentum_rows_kernel<Z, NS, SAME, W, UNROLL>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)smem);
    if (e != cudaSuccess) return e;
    if (dev < 64) attr_set[dev] = 1;
  }
  const int grid = std::min(p.total_units, job.num_sms);
  momentum_rows_kernel<Z, NS, SAME, W, UNROLL><<<grid, 32 * W, smem, job.stream>>>(p, stages);
  return cudaGetLastError();
}

template <bool SAME> cudaError_t launch_rows_groups(const Job &job, const MomBatchParams &p)
{
  const bool zero = p.gx_k[0] == 0;
  switch (p.ngx * 2 + (zero ? 1 : 0)) {
  case 3: return launch_rows<1, 0, SAME>(job, p);
  case 5: return launch_rows<1, 1, SAME>(job, p);
  case 7: return launch_rows<1, 2, SAME>(job, p);
  case 2: return launch_rows<0, 1, SAME>(job, p);
  case 4: return launch_rows<0, 2, SAME>(job, p);
  case 6: return launch_rows<0, 3, SAME>(job, p);
  default: return cudaErrorInvalidValue;
  }
}

} // namespace

void order_pairs(MomBatchParams &p)
{
  const int zero = p.gx_k[0] == 0 ? 1 : 0, slots = zero + 2 * (p.ngx - zero);
  auto px = [&](int slot) {  // the nx of a slot; -1: none (a group without its partner)
    if (slot < zero) return std::max(p.gx_plus[0], p.gx_minus[0]);
    const int group = zero + (slot - zero) / 2;
    return (slot - zero) & 1 ? p.gx_minus[group] : p.gx_plus[group];
  };
  int n = 0;
  for (int slot = 0; slot < slots; ++slot) {
    p.pairs.start[slot] = (uint8_t)n;
    for (int q = 0; q < p.nq; ++q)
      if (p.q_ix[q] == px(slot)) p.pairs.list[n++] = (uint8_t)q;
  }
  p.pairs.start[slots] = (uint8_t)n;
}

cudaError_t launch_momentum_rows(const Job &job, const MomBatchParams &p, bool same_field)
{
  if (p.total_units <= 0) return cudaSuccess;
  if (p.ngx < 1 || p.ngx > 3 || p.nq < 1 || p.nq > kMomQChunk) return cudaErrorInvalidValue;
  return same_field ? launch_rows_groups<true>(job, p) : launch_rows_groups<false>(job, p);
}

} // namespace cgb
