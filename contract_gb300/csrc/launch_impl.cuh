// Launch helpers shared by the kernel translation units.
#pragma once

#include <algorithm>
#include <climits>
#include <mutex>

#include "engine_warp.cuh"
#include "launch.hpp"

namespace cgb {

// Tile geometry for an op with `sites` sites per tile, its chunks dealt round-robin to
// `warps` persistent warps (or CTAs).  About `chunks_per_warp` chunks each keep the tail
// of the round-robin (warps that draw one chunk more than others) near
// 1/chunks_per_warp of a warp's work; chunks never span segments and hold at most 64
// tiles.  `level`: where that makes chunks of four tiles or fewer, of these lengths and
// longer ones the one that takes least time if all warps run alike and the end of a chunk
// costs half a tile.
inline TileGeom make_geom(const Job &job, int sites, long long warps, int chunks_per_warp, bool level = false)
{
  TileGeom g {};
  g.volume = job.volume;
  if (job.per_site) {
    g.seg_len = job.volume;
    g.num_segs = 1;
    g.per_site = 1;
  } else {
    g.seg_len = job.half_slice;
    g.num_segs = 2 * job.lt;
    g.per_site = 0;
  }
  g.tiles_per_seg = (int)((g.seg_len + sites - 1) / sites);
  const long long tiles = (long long)g.tiles_per_seg * g.num_segs;
  warps = std::max(1LL, warps);
  const int most = std::min(64, g.tiles_per_seg);
  g.chunk_tiles = (int)std::max(1LL, std::min<long long>(tiles / (warps * chunks_per_warp), most));
  if (level && g.chunk_tiles <= 4) {
    long long best = LLONG_MAX;
    for (int n = g.chunk_tiles; n <= most; ++n) {
      const long long chunks = (long long)((g.tiles_per_seg + n - 1) / n) * g.num_segs;
      const long long cost = (chunks + warps - 1) / warps * (2 * n + 1);
      if (cost < best) {
        best = cost;
        g.chunk_tiles = n;
      }
    }
  }
  g.chunks_per_seg = (g.tiles_per_seg + g.chunk_tiles - 1) / g.chunk_tiles;
  g.total_chunks = g.chunks_per_seg * g.num_segs;
  g.wait_ns = job.wait_ns ? job.wait_ns : kWaitLimitNs;
  g.withhold_chunk = job.withhold_chunk;
  return g;
}

// Chunks per warp of the kernels of engine_warp.cuh (per CTA of field_kernel).  Sums in
// complex64 then level the rounds: with one tile a chunk, as middle sizes had, the ends of
// the chunks and the partials that they leave took a fifth of the time.  us before and
// after, 12^3 x 24, 16 x 15 x 16 x 32 and 20^3 x 36: all types 47.7, 113.8, 210.6 and
// 40.0, 93.5, 192.6; all partners of a Gamma 32.7, 55.4 and 23.6, 49.2 (the last alike);
// one meson at the last two 53.5, 116.1 and 48.2, 103.9.  Longer chunks gain nothing
// (loop at 28^3 x 56: 595, 621 with level rounds of 25 tiles).  Per-site results end a chunk
// for nothing, and in complex128 fewer warps at work cost more than the ends: both keep
// the plain rule (all types at 8^3 x 16 in complex128 79 us, 95 with level rounds).
constexpr int kChunksPerWarp = 12;

template <class K> struct KernelAttr {
  int bps[64] = {};  // resident CTAs per SM, per device ordinal (0 = not yet queried)
};

template <class Op, class K> cudaError_t prepare(K kernel, size_t smem, int &bps_out, int threads = Op::THREADS)
{
  static KernelAttr<K> cache;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 64 && cache.bps[dev] > 0) {
    bps_out = cache.bps[dev];
    return cudaSuccess;
  }
  e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  int bps = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, kernel, threads, smem);
  if (e != cudaSuccess) return e;
  if (bps < 1) return cudaErrorInvalidConfiguration;
  if (dev < 64) cache.bps[dev] = bps;
  bps_out = bps;
  return cudaSuccess;
}

// Launches a kernel that begins with grid_dependency_wait(): its grid comes up while
// the kernel before it on the stream drains.  The finalisation of per-timeslice sums
// this way: 22.7 -> 21.0 us for a call of all types at 8^3 x 16, 299.4 -> 297.3 for one
// type at 22 x 17 x 25 x 54.
template <class... Params, class... Args>
cudaError_t launch_overlapped(void (*kernel)(Params...), dim3 grid, int threads, size_t smem, cudaStream_t stream,
                              const Args &...args)
{
  cudaLaunchAttribute overlap {};
  overlap.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  overlap.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = &overlap;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}

struct OutPtrs {
  double2 *p[16];
};

constexpr int kFinThreads = 64;  // finalize_kernel's block: the partials of one (output, timeslice)
// Reduces the chunk partials left by the kernel launched before it on the job's stream.
cudaError_t launch_finalize_chunks(const Job &job, const double2 *partial, const OutPtrs &out, int nout,
                                   int chunks_per_seg);

// Launches a kernel of engine_warp.cuh over the job's chunks, dealt to the grid's
// warps, and reduces the chunk partials if the job sums timeslices.
template <class Op, class K> cudaError_t launch_chunks(const Job &job, OpParams<typename Op::R> p, K kernel, size_t smem)
{
  int bps = 0;
  cudaError_t e = prepare<Op>(kernel, smem, bps, 32 * Op::CW);
  if (e != cudaSuccess) return e;
  const int ctas = job.num_sms * bps;
  p.geom = make_geom(job, ChunkWalk<Op>::SITES, (long long)ctas * Op::CW, kChunksPerWarp,
                     sizeof(typename Op::R) == 4 && !job.per_site);
  p.status = job.status;
  static_assert(Op::NOUT <= 16, "at most 16 outputs per site");
  OutPtrs user_out {};
  for (int o = 0; o < Op::NOUT; ++o) user_out.p[o] = static_cast<double2 *>(p.out[o]);
  double2 *partial = nullptr;
  if (!job.per_site) {
    if (!job.ws) return cudaErrorInvalidValue;
    partial = static_cast<double2 *>(job.ws->get((size_t)p.geom.total_chunks * Op::NOUT * sizeof(double2)));
    if (!partial) return cudaErrorMemoryAllocation;
    p.out[0] = partial;
  }
  const int grid = std::min(ChunkWalk<Op>::ctas_for(p.geom.total_chunks), ctas);
  kernel<<<grid, 32 * Op::CW, smem, job.stream>>>(p);
  e = cudaGetLastError();
  if (e != cudaSuccess || job.per_site) return e;
  return launch_finalize_chunks(job, partial, user_out, Op::NOUT, p.geom.chunks_per_seg);
}

// One launch of a per-call scalar op's ring kernel, then, for per-timeslice sums,
// the finalisation of its chunk partials.
template <class Op> cudaError_t run_ring(const Job &job, OpParams<typename Op::R> p)
{
  if (job.volume == 0) return cudaSuccess;
  using Walk = ChunkWalk<Op>;
  constexpr size_t smem = RingSmem<Op>::BYTES;
  static_assert(smem <= 232448, "op does not fit in shared memory");
  return launch_chunks<Op>(job, p, ring_kernel<Op, Walk>, smem);
}

// One launch of an op of the field ring kernel.
template <class Op> cudaError_t run_field_ring(const Job &job, const OpParams<typename Op::R> &p)
{
  if (job.volume == 0) return cudaSuccess;
  Job j = job;
  j.per_site = true;
  constexpr size_t smem = RingSmem<Op>::BYTES;
  static_assert(smem <= 232448, "op does not fit in shared memory");
  return launch_chunks<Op>(j, p, field_ring_kernel<Op, ChunkWalk<Op>>, smem);
}

template <class Op> cudaError_t run_field(const Job &job, OpParams<typename Op::R> p)
{
  if (job.volume == 0) return cudaSuccess;
  Job j = job;
  j.per_site = true;
  constexpr size_t smem = engine_smem_bytes<Op>();
  static_assert(smem <= 232448, "op does not fit in shared memory");
  int bps = 0;
  cudaError_t e = prepare<Op>(field_kernel<Op>, smem, bps);
  if (e != cudaSuccess) return e;
  const long long ctas = (long long)job.num_sms * bps;
  p.geom = make_geom(j, Op::SITES, ctas, kChunksPerWarp);
  p.status = job.status;
  const int grid = (int)std::min<long long>(p.geom.total_chunks, ctas);
  field_kernel<Op><<<grid, Op::THREADS, smem, job.stream>>>(p);
  return cudaGetLastError();
}

} // namespace cgb
