// Persistent batched launch over a device work queue.
//
// A batch is up to kMaxBatch work items -- one per (source position,
// propagator triple, lattice) -- that share one op and its spin tables.  The
// items travel as a kernel parameter (so a CUDA graph captures them by
// value).  Each item's chunks are laid end to end in one global chunk space,
// and the queue is a counter in device memory over that space (zeroed by the
// host before every launch): each warp of warp_kernel (engine_warp.cuh) takes
// the next chunk with an atomic add when it has issued the last tile of its
// own, so warps that finish early take more chunks and items of very different
// sizes balance without a static schedule.  The warp looks up the chunk's item
// (binary search on chunk_begin) for its geometry, inputs and partial sums.
//
// Every item is validated on the device before use (extents, chunk ranges,
// 16-byte alignment); a chunk of a bad item is skipped and reported through
// the status word as kDevErrBadWork.
#pragma once

#include "engine_warp.cuh"
#include "ops.cuh"

namespace cgb {

constexpr int kMaxBatch = 128;

struct BatchItem {
  const void *in[3];
  double2 *partial;  // [chunks][NOUT] of this item
  TileGeom geom;     // per_site == 0: segments are half-timeslices
  int chunk_begin;   // first global chunk of this item
  int lt;            // timeslices (for the finalisation)
  double2 *out;      // [NOUT][lt] complex128 result
};

template <class R> struct BatchParams {
  OpParams<R> op;  // spin tables; op.in/op.out unused
  DeviceStatus *status;
  unsigned int *queue;  // next global chunk (zero at launch)
  int n_items;
  int total_chunks;
  BatchItem items[kMaxBatch];
};

// Structural checks of one descriptor.
template <int SITES, int NIN> __device__ __forceinline__ bool item_ok(const BatchItem &it)
{
  const TileGeom &g = it.geom;
  if (g.seg_len <= 0 || g.num_segs <= 0 || g.chunk_tiles <= 0 || g.chunks_per_seg <= 0) return false;
  if ((long long)g.tiles_per_seg * SITES < g.seg_len || (long long)(g.tiles_per_seg - 1) * SITES >= g.seg_len) return false;
  if (g.total_chunks != g.chunks_per_seg * g.num_segs) return false;
  if ((long long)g.seg_len * g.num_segs != g.volume) return false;
  for (int q = 0; q < NIN; ++q)
    if (!it.in[q] || (reinterpret_cast<uintptr_t>(it.in[q]) & 15)) return false;
  return it.partial != nullptr;
}

template <class P> __device__ __forceinline__ int find_item(const P &p, int chunk)
{
  int lo = 0, hi = p.n_items - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (p.items[mid].chunk_begin <= chunk) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// A warp's walk over the tiles of the chunks it takes from the queue.
template <class Op> struct QueueWalk {
  static constexpr int SITES = 32 / Op::TPS;
  using Params = BatchParams<typename Op::R>;
  int chunk, item, local, k, ntiles;
  long long at, end;  // first site of the tile, end of its segment

  __device__ __forceinline__ void take(const Params &p)
  {
    for (;;) {
      unsigned int c = 0;
      if ((threadIdx.x & 31) == 0) c = atomicAdd(p.queue, 1u);
      c = __shfl_sync(0xffffffffu, c, 0);
      chunk = (int)min(c, (unsigned int)p.total_chunks);
      if (chunk >= p.total_chunks) return;
      item = find_item(p, chunk);
      const BatchItem &it = p.items[item];
      const TileGeom &g = it.geom;
      local = chunk - it.chunk_begin;
      if (local >= 0 && local < g.total_chunks && item_ok<SITES, Op::NIN>(it)) {
        const int seg = local / g.chunks_per_seg, cc = local - seg * g.chunks_per_seg;
        k = 0;
        ntiles = min(g.chunk_tiles, g.tiles_per_seg - cc * g.chunk_tiles);
        at = (long long)seg * g.seg_len + (long long)cc * g.chunk_tiles * SITES;
        end = (long long)(seg + 1) * g.seg_len;
        if (ntiles > 0) return;
      }
      if ((threadIdx.x & 31) == 0) report(p.status, kDevErrBadWork, c);  // a rejected item: its chunks are skipped
    }
  }
  __device__ __forceinline__ void start(const Params &p) { take(p); }
  __device__ __forceinline__ bool valid(const Params &p) const { return chunk < p.total_chunks; }
  __device__ __forceinline__ void next(const Params &p)
  {
    at += SITES;
    if (++k == ntiles) take(p);
  }
  __device__ __forceinline__ bool last_in_chunk() const { return k == ntiles - 1; }
  __device__ __forceinline__ long long first() const { return at; }
  __device__ __forceinline__ int sites() const { return (int)min((long long)SITES, end - at); }
  __device__ __forceinline__ int where() const { return chunk; }
  __device__ __forceinline__ bool withheld(const Params &) const { return false; }
  __device__ __forceinline__ const char *in(const Params &p, int q) const
  {
    return static_cast<const char *>(p.items[item].in[q]);
  }
  __device__ __forceinline__ double2 *partial(const Params &p) const
  {
    return p.items[item].partial + (size_t)local * Op::NOUT;
  }
};
template <class Op> __device__ __forceinline__ const typename Op::Params &op_params(const BatchParams<typename Op::R> &p)
{
  return p.op;
}

// out_i[o][t] = sum over parity and the item's chunk partials, FP64, fixed order.  Grid: (items, ceil(nout * max_lt / 128)).
template <class R>
__global__ void batch_finalize_kernel(const __grid_constant__ BatchParams<R> p, int nout)
{
  const int i = blockIdx.x;
  const BatchItem &it = p.items[i];
  const int idx = blockIdx.y * blockDim.x + threadIdx.x;
  if (idx >= nout * it.lt || it.geom.chunks_per_seg <= 0) return;
  const int o = idx / it.lt, t = idx % it.lt;
  const int per_seg = it.geom.chunks_per_seg;
  double sx = 0.0, sy = 0.0;
  for (int par = 0; par < 2; ++par) {
    const double2 *row = it.partial + ((size_t)(par * it.lt + t) * per_seg) * nout + o;
    for (int c = 0; c < per_seg; ++c) {
      const double2 v = row[(size_t)c * nout];
      sx += v.x;
      sy += v.y;
    }
  }
  it.out[(size_t)o * it.lt + t] = make_double2(sx, sy);
}

} // namespace cgb
