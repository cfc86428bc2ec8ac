// Tile pipelines in which every warp streams its own tiles: warp_kernel for the all-types
// baryon pass, ring_kernel for the per-call contractions, field_ring_kernel for diquark
// and sequential sources.  First the all-types pass.
//
// A tile is SPW = 32 / TPS consecutive sites of one reduction segment (a
// half-timeslice, or the whole volume for per-site outputs); chunks of tiles
// are dealt to warps, round-robin (ChunkWalk) or from a device queue
// (QueueWalk, batch.cuh).  A warp owns one shared-memory slot per site and
// input, filled with cp.async.bulk by its own lanes, and two mbarriers.  Ops
// work in two steps (Op::first on the inputs before the last one, Op::second on
// the last), so a slot is refilled as soon as its step is done: P_i and P_j of
// the next tile arrive while this one's dots run, P_n during the next tile's
// wedges.  One slot instead of a two-stage ring takes half the shared memory a
// site, and no warp waits for another.  At 24^3 x 64 in complex64 the pass took
// 0.740 ms on the shared ring of engine.cuh with its producer warp (12 consumer
// warps an SM of 2 sites: shared memory full, issue slots 59 % used, dependent
// instructions the first stall), 0.666 ms here with 20 such warps and 0.590 ms
// with 12 warps of 4 sites, which hold two blocks a thread (HBM: 0.457 ms).
//
// Every wait is bounded in wall time; a warp that times out reports it, waits
// (bounded) for its copies still in flight and returns.
//
// An op yields NVAL values per site and combine() makes its NOUT outputs of
// them: per site, or per chunk after a compensated sum over the chunk's sites
// (partial[chunk][NOUT], reduced per timeslice by finalize_kernel).
#pragma once

#include "engine.cuh"

namespace cgb {

template <class Op> struct WarpSmem {
  using L = OpLayout<Op>;
  static constexpr int SPW = 32 / Op::TPS;
  static constexpr size_t IN = 16;  // the warp's two mbarriers come first
  static constexpr size_t EXTRA = IN + (size_t)Op::NIN * SPW * L::SLOT;
  static constexpr size_t WARP = EXTRA + (size_t)SPW * Op::EXTRA_BYTES;
  static constexpr size_t BYTES = Op::CW * WARP;
  static_assert(WARP % 16 == 0 && Op::EXTRA_BYTES % 16 == 0, "slots must stay 16-byte aligned");
};

// A warp's walk over its tiles of one lattice: chunks w, w + (warps of the grid), ...
// With one CTA an SM, which has many warps then, consecutive chunks go to consecutive CTAs:
// fewer chunks than warps, or the last round's, spread over all SMs.  All types in
// complex64, 12 warps, 4^3 x 8, 8^3 x 16 and 24^3 x 64: 12.0, 19.9 and 597 us with the chunks
// side by side in a CTA, 7.8, 16.2 and 580 so.  Several small CTAs an SM spread by themselves
// and read memory in longer runs side by side: four warps 604 against 614, sequential
// sources at 32^3 x 48 920 against 947.
template <class Op> struct ChunkWalk {
  static constexpr int SITES = 32 / Op::TPS;
  static constexpr bool SPREAD = Op::MIN_CTAS == 1;
  using Params = typename Op::Params;
  TileIter<SITES> it;
  int stride;

  static int ctas_for(int chunks) { return SPREAD ? chunks : (chunks + Op::CW - 1) / Op::CW; }
  __device__ __forceinline__ void start(const Params &p)
  {
    stride = gridDim.x * Op::CW;
    const int warp = threadIdx.x >> 5;
    it.set_chunk(p.geom, SPREAD ? blockIdx.x + gridDim.x * warp : blockIdx.x * Op::CW + warp);
  }
  __device__ __forceinline__ bool valid(const Params &p) const { return it.valid(p.geom); }
  __device__ __forceinline__ void next(const Params &p) { it.next(p.geom, stride); }
  __device__ __forceinline__ bool last_in_chunk() const { return it.last_in_chunk(); }
  __device__ __forceinline__ long long first() const { return it.first; }
  __device__ __forceinline__ int sites() const { return it.sites(); }
  __device__ __forceinline__ int where() const { return it.chunk; }
  __device__ __forceinline__ bool withheld(const Params &p) const { return it.k == 0 && it.chunk == p.geom.withhold_chunk; }
  __device__ __forceinline__ const char *in(const Params &p, int q) const { return static_cast<const char *>(p.in[q]); }
  __device__ __forceinline__ double2 *partial(const Params &p) const
  {
    return static_cast<double2 *>(p.out[0]) + (size_t)it.chunk * Op::NOUT;
  }
};
template <class Op> __device__ __forceinline__ const typename Op::Params &op_params(const typename Op::Params &p)
{
  return p;
}

template <class Op, class Walk>
__global__ void __launch_bounds__(32 * Op::CW, Op::MIN_CTAS) warp_kernel(const __grid_constant__ typename Walk::Params p)
{
  using S = typename Op::S;
  using R = typename Op::R;
  using L = OpLayout<Op>;
  constexpr int NIN = Op::NIN, TPS = Op::TPS, SPW = 32 / TPS, NVAL = Op::NVAL, NOUT = Op::NOUT;
  constexpr int SH = values_shift<TPS, NVAL>();  // value r of a site: thread r << SH

  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ __align__(16) typename Op::Params ps;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  unsigned char *mine = smem + warp * WarpSmem<Op>::WARP;
  uint64_t *bars = reinterpret_cast<uint64_t *>(mine);  // [0]: all inputs but the last, [1]: the last
  if (lane == 0) {
    mbar_init(&bars[0], 1);
    mbar_init(&bars[1], 1);
    fence_barrier_init();
  }
  copy_params(ps, op_params<Op>(p));
  __syncthreads();

  const int local = lane / TPS, sub = lane % TPS;
  S *in[NIN];  // an op may change its inputs in place
#pragma unroll
  for (int q = 0; q < NIN; ++q)
    in[q] = reinterpret_cast<S *>(mine + WarpSmem<Op>::IN + ((size_t)q * SPW + local) * L::SLOT);
  S *scratch = reinterpret_cast<S *>(mine + WarpSmem<Op>::EXTRA + (size_t)local * Op::EXTRA_BYTES);

  // Issue the copies of a tile's inputs [q0, q1) on barrier b.
  auto fetch = [&](const Walk &w, int q0, int q1, int b) {
    if (w.withheld(p)) return;  // test hook: this tile never arrives
    const int n = w.sites();
    if (lane == 0) mbar_arrive_expect_tx(&bars[b], (uint32_t)(n * (q1 - q0)) * L::SITE_BYTES);
    __syncwarp();
    if (lane < SPW * (q1 - q0)) {
      const int q = q0 + lane / SPW, s = lane % SPW;
      if (s < n)
        bulk_g2s(mine + WarpSmem<Op>::IN + ((size_t)q * SPW + s) * L::SLOT, w.in(p, q) + (w.first() + s) * L::SITE_BYTES,
                 L::SITE_BYTES, &bars[b]);
    }
  };
  Walk cur;
  cur.start(p);
  if (cur.valid(p)) {
    fetch(cur, 0, NIN - 1, 0);
    fetch(cur, NIN - 1, NIN, 1);
  }
  const unsigned long long wait_ns = ps.geom.wait_ns;
  // Both barriers complete once per tile.  A warp that gave up waits for what
  // may still be in flight: this tile's copies on either barrier, and with
  // `next_too` the next tile's on the first.
  auto give_up = [&](uint32_t parity, bool next_too) {
    report(p.status, kDevErrWaitTimeout, (unsigned int)cur.where());
    if (lane == 0) {
      mbar_wait_bounded(&bars[0], next_too ? parity ^ 1u : parity, wait_ns / 8);
      mbar_wait_bounded(&bars[1], parity, wait_ns / 8);
    }
  };
  ChunkSum<R> chunk_acc;
  for (uint32_t u = 0; cur.valid(p); ++u) {
    if (!__all_sync(0xffffffffu, mbar_wait_bounded(&bars[0], u & 1u, wait_ns))) {
      give_up(u & 1u, false);
      return;
    }
    typename Op::State state;
    Op::first(ps, in, scratch, sub, local < cur.sites(), state);
    Walk nx = cur;
    nx.next(p);
    fence_proxy_async_smem();
    __syncwarp();
    if (nx.valid(p)) fetch(nx, 0, NIN - 1, 0);
    if (!__all_sync(0xffffffffu, mbar_wait_bounded(&bars[1], u & 1u, wait_ns))) {
      give_up(u & 1u, nx.valid(p));
      return;
    }
    cx<R> vals[NVAL];
    Op::second(ps, in[NIN - 1], scratch, sub, local < cur.sites(), state, vals);
    fence_proxy_async_smem();
    __syncwarp();
    if (nx.valid(p)) fetch(nx, NIN - 1, NIN, 1);
    const cx<R> v = group_reduce_values<TPS, NVAL>(vals, sub);
    const bool ok = local < cur.sites();
    if (ps.geom.per_site) {
#pragma unroll
      for (int o0 = 0; o0 < NOUT; o0 += TPS) {
        const int o = o0 + sub;
        const cx<R> z = Op::combine(ps, o < NOUT ? o : 0, v, lane - sub, 1 << SH);
        if (o < NOUT && ok)
          static_cast<double2 *>(ps.out[o])[cur.first() + local] = make_double2(double(z.x), double(z.y));
      }
    } else {
      // each lane sums the value it holds of its own site; the warp's sites
      // meet in FP64 at the end of the chunk
      chunk_acc.add(ok ? v : czero<R>());
      if (cur.last_in_chunk()) {
        double2 c = chunk_acc.value();
#pragma unroll
        for (int o = 16; o >= TPS; o >>= 1) {
          c.x += __shfl_xor_sync(0xffffffffu, c.x, o);
          c.y += __shfl_xor_sync(0xffffffffu, c.y, o);
        }
        const double2 z = Op::combine(ps, lane < NOUT ? lane : 0, c, 0, 1 << SH);
        if (lane < NOUT) cur.partial(p)[lane] = z;
        chunk_acc.reset();
      }
    }
    cur = nx;
  }
}

// ---------------------------------------------------------------- rings --
// The same for ops of one step: a warp has an NST-stage ring of whole tiles, and
// Op::site() yields the site's value -- the sum over its threads is one output
// (NOUT == 1), or with NOUT > 1 thread sub holds output Op::output(p, sub) complete.
template <class Op> struct RingSmem {
  using L = OpLayout<Op>;
  static constexpr int SPW = 32 / Op::TPS;
  static constexpr size_t IN = (Op::NST * 8 + 15) / 16 * 16;  // after the warp's mbarriers
  static constexpr size_t STAGE = (size_t)Op::NIN * SPW * L::SLOT;
  static constexpr size_t EXTRA = IN + Op::NST * STAGE;
  static constexpr size_t WARP = EXTRA + (size_t)SPW * Op::EXTRA_BYTES;
  static constexpr size_t BYTES = Op::CW * WARP;
  static_assert(Op::EXTRA_BYTES % 16 == 0, "slots must stay 16-byte aligned");
};

template <class Op, class Walk>
__global__ void __launch_bounds__(32 * Op::CW, Op::MIN_CTAS) ring_kernel(const __grid_constant__ typename Walk::Params p)
{
  using S = typename Op::S;
  using R = typename Op::R;
  using L = OpLayout<Op>;
  using M = RingSmem<Op>;
  constexpr int NIN = Op::NIN, TPS = Op::TPS, SPW = 32 / TPS, NOUT = Op::NOUT, NST = Op::NST;

  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ __align__(16) typename Op::Params ps;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  unsigned char *mine = smem + warp * M::WARP;
  uint64_t *full = reinterpret_cast<uint64_t *>(mine);
  if (lane == 0) {
    for (int s = 0; s < NST; ++s) mbar_init(&full[s], 1);
    fence_barrier_init();
  }
  copy_params(ps, op_params<Op>(p));
  __syncthreads();
  grid_dependents_may_launch();

  const int local = lane / TPS, sub = lane % TPS;
  S *scratch = reinterpret_cast<S *>(mine + M::EXTRA + (size_t)local * Op::EXTRA_BYTES);
  auto fetch = [&](const Walk &w, int stage) {
    if (w.withheld(p)) return;  // test hook: this tile never arrives
    const int n = w.sites();
    if (lane == 0) mbar_arrive_expect_tx(&full[stage], (uint32_t)(n * NIN) * L::SITE_BYTES);
    __syncwarp();
    if (lane < SPW * NIN) {
      const int q = lane / SPW, s = lane % SPW;
      if (s < n)
        bulk_g2s(mine + M::IN + stage * M::STAGE + ((size_t)q * SPW + s) * L::SLOT,
                 w.in(p, q) + (w.first() + s) * L::SITE_BYTES, L::SITE_BYTES, &full[stage]);
    }
    if constexpr (Op::DIRECT > 0) {  // what the op will read from memory is in L2 by then
      if (lane < Op::DIRECT) bulk_prefetch_l2(w.in(p, NIN + lane) + w.first() * L::SITE_BYTES, (uint32_t)n * L::SITE_BYTES);
    }
  };
  static_assert(SPW * NIN <= 32, "one copy per lane");
  Walk cur, ahead;
  cur.start(p);
  ahead = cur;
  int issued = 0;
  for (; issued < NST && ahead.valid(p); ++issued, ahead.next(p)) fetch(ahead, issued);
  const unsigned long long wait_ns = ps.geom.wait_ns;
  ChunkSum<R> chunk_acc;
  ChunkPart<R> chunk_part;
  for (int u = 0; cur.valid(p); ++u) {
    const int stage = u % NST;
    if (!__all_sync(0xffffffffu, mbar_wait_bounded(&full[stage], (u / NST) & 1, wait_ns))) {
      report(p.status, kDevErrWaitTimeout, (unsigned int)cur.where());
      if (lane == 0)  // the copies that may still be in flight
        for (int v = u; v < issued; ++v) mbar_wait_bounded(&full[v % NST], (v / NST) & 1, wait_ns / 8);
      return;
    }
    S *in[NIN];
#pragma unroll
    for (int q = 0; q < NIN; ++q)
      in[q] = reinterpret_cast<S *>(mine + M::IN + stage * M::STAGE + ((size_t)q * SPW + local) * L::SLOT);
    const bool ok = local < cur.sites();
    cx<R> v;
    if constexpr (Op::DIRECT > 0) {  // fields NIN and on are read from memory by the op
      const long long at = (cur.first() + (ok ? local : 0)) * L::SITE_BYTES;
      const S *more[Op::DIRECT];
#pragma unroll
      for (int q = 0; q < Op::DIRECT; ++q) more[q] = reinterpret_cast<const S *>(cur.in(p, NIN + q) + at);
      v = Op::site(ps, in, more, scratch, sub, ok);
    } else {
      v = Op::site(ps, in, scratch, sub, ok);
    }
    if constexpr (Op::CHANGES_INPUT) fence_proxy_async_smem();
    __syncwarp();  // every lane is done with the stage
    if (ahead.valid(p)) {
      fetch(ahead, stage);
      ++issued;
      ahead.next(p);
    }
    if constexpr (NOUT == 1) {
      // even threads are left with the site's real part, odd ones with the imaginary:
      // half the adds of two full sums, which the FP64 pipe feels
      const bool odd = lane & 1;
      R part = (odd ? v.y : v.x) + __shfl_xor_sync(0xffffffffu, odd ? v.x : v.y, 1);
#pragma unroll
      for (int o = TPS / 2; o > 1; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
      if (ps.geom.per_site) {
        if (ok && sub < 2) static_cast<double *>(ps.out[0])[2 * (cur.first() + local) + sub] = double(part);
      } else {
        chunk_part.add(ok ? part : R(0));
        if (cur.last_in_chunk()) {
          double c = chunk_part.value();
#pragma unroll
          for (int o = 16; o >= TPS; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
          if (lane < 2) reinterpret_cast<double *>(cur.partial(p))[lane] = c;
          chunk_part = {};
        }
      }
    } else {
      static_assert(NOUT == TPS, "one output per thread of a site");
      if (ps.geom.per_site) {
        if (ok)
          static_cast<double2 *>(ps.out[Op::output(ps, sub)])[cur.first() + local] = make_double2(double(v.x), double(v.y));
      } else {
        chunk_acc.add(ok ? v : czero<R>());
        if (cur.last_in_chunk()) {
          double2 c = chunk_acc.value();
#pragma unroll
          for (int o = 16; o >= TPS; o >>= 1) {
            c.x += __shfl_xor_sync(0xffffffffu, c.x, o);
            c.y += __shfl_xor_sync(0xffffffffu, c.y, o);
          }
          if (lane < NOUT) cur.partial(p)[Op::output(ps, lane)] = c;
          chunk_acc.reset();
        }
      }
    }
    cur.next(p);
  }
}

// ---------------------------------------------------------------- fields --
// The same for ops with a propagator-shaped result per site: Op::site() leaves it in
// the first input's slot, from where lane 0 stores it (cp.async.bulk).  A stage is
// filled again one tile later than it was used, when its stores have been read:
// NST - 1 tiles are in flight and no warp waits for its own stores.
template <class Op, class Walk>
__global__ void __launch_bounds__(32 * Op::CW, Op::MIN_CTAS)
  field_ring_kernel(const __grid_constant__ typename Walk::Params p)
{
  using S = typename Op::S;
  using L = OpLayout<Op>;
  using M = RingSmem<Op>;
  constexpr int NIN = Op::NIN, TPS = Op::TPS, SPW = 32 / TPS, NST = Op::NST;
  static_assert(NST >= 2, "a stage rests for one tile");
  constexpr uint32_t OUT = Op::OUT_ELEMS * sizeof(S);
  static_assert(OUT <= L::SITE_BYTES, "the result takes the place of an input");

  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ __align__(16) typename Op::Params ps;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  unsigned char *mine = smem + warp * M::WARP;
  uint64_t *full = reinterpret_cast<uint64_t *>(mine);
  if (lane == 0) {
    for (int s = 0; s < NST; ++s) mbar_init(&full[s], 1);
    fence_barrier_init();
  }
  copy_params(ps, op_params<Op>(p));
  __syncthreads();

  const int local = lane / TPS, sub = lane % TPS;
  S *scratch = reinterpret_cast<S *>(mine + M::EXTRA + (size_t)local * Op::EXTRA_BYTES);
  auto fetch = [&](const Walk &w, int stage) {
    if (w.withheld(p)) return;  // test hook: this tile never arrives
    const int n = w.sites();
    if (lane == 0) mbar_arrive_expect_tx(&full[stage], (uint32_t)(n * NIN) * L::SITE_BYTES);
    __syncwarp();
    if (lane < SPW * NIN) {
      const int q = lane / SPW, s = lane % SPW;
      if (s < n)
        bulk_g2s(mine + M::IN + stage * M::STAGE + ((size_t)q * SPW + s) * L::SLOT,
                 w.in(p, q) + (w.first() + s) * L::SITE_BYTES, L::SITE_BYTES, &full[stage]);
    }
  };
  static_assert(SPW * NIN <= 32, "one copy per lane");
  Walk cur, ahead;
  cur.start(p);
  ahead = cur;
  int issued = 0;
  for (; issued < NST - 1 && ahead.valid(p); ++issued, ahead.next(p)) fetch(ahead, issued);
  const unsigned long long wait_ns = ps.geom.wait_ns;
  for (int u = 0; cur.valid(p); ++u) {
    const int stage = u % NST;
    if (!__all_sync(0xffffffffu, mbar_wait_bounded(&full[stage], (u / NST) & 1, wait_ns))) {
      report(p.status, kDevErrWaitTimeout, (unsigned int)cur.where());
      if (lane == 0) {  // the copies that may still be in flight
        for (int v = u; v < issued; ++v) mbar_wait_bounded(&full[v % NST], (v / NST) & 1, wait_ns / 8);
        bulk_wait<0>();
      }
      return;
    }
    unsigned char *sb = mine + M::IN + stage * M::STAGE;
    S *in[NIN];
#pragma unroll
    for (int q = 0; q < NIN; ++q) in[q] = reinterpret_cast<S *>(sb + ((size_t)q * SPW + local) * L::SLOT);
    const int n = cur.sites();
    Op::site(ps, in, scratch, sub, local < n);
    fence_proxy_async_smem();
    __syncwarp();
    if (lane == 0) {
      for (int s = 0; s < n; ++s)
        bulk_s2g(static_cast<char *>(p.out[0]) + (cur.first() + s) * OUT, sb + (size_t)s * L::SLOT, OUT);
      bulk_commit();
      bulk_wait_read<1>();  // the previous tile's stores have left its stage
    }
    __syncwarp();
    if (ahead.valid(p)) {
      fetch(ahead, issued % NST);
      ++issued;
      ahead.next(p);
    }
    cur.next(p);
  }
  if (lane == 0) bulk_wait<0>();
}

} // namespace cgb
