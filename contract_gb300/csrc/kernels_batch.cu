// Batched all-types baryon contractions: many sources / lattices per launch.
#include <mutex>
#include <tuple>
#include <vector>

#include "batch.cuh"
#include "ops_fused.cuh"
#include "launch_impl.cuh"
#include "batch.hpp"
#include "momentum.hpp"

namespace cgb {

// One persistent launch over the n items, then (fin == nullptr) the
// finalisation launch, or (fin != nullptr) the finalisation left to the
// caller's combined launch: fin receives each item's partials and outputs.
template <class Op>
static cudaError_t run_batch(const Job &job, const OpParams<typename Op::R> &op, const BatchSpec *specs, int n,
                             BaryonFinParams *fin)
{
  using R = typename Op::R;
  if (n <= 0) return cudaSuccess;
  if (n > kMaxBatch) return cudaErrorInvalidValue;
  static BatchParams<R> bp;  // large (~10 KB): built on the host, passed by value
  static std::mutex mu;
  std::lock_guard<std::mutex> lk(mu);
  bp = {};
  bp.op = op;
  bp.op.geom.wait_ns = job.wait_ns ? job.wait_ns : kWaitLimitNs;
  bp.status = job.status;
  bp.n_items = n;
  using Walk = QueueWalk<Op>;
  constexpr size_t smem = WarpSmem<Op>::BYTES;
  static_assert(smem <= 232448, "op does not fit in shared memory");
  int bps = 0;
  cudaError_t e = prepare<Op>(warp_kernel<Op, Walk>, smem, bps, 32 * Op::CW);
  if (e != cudaSuccess) return e;
  const int warps = job.num_sms * bps * Op::CW;
  size_t partial_total = 0;
  int chunks = 0;
  long long max_lt = 0;
  for (int i = 0; i < n; ++i) {
    Job ji = job;
    ji.volume = (long long)specs[i].latt[0] * specs[i].latt[1] * specs[i].latt[2] * specs[i].latt[3];
    ji.per_site = false;
    ji.lt = specs[i].latt[3];
    ji.half_slice = (long long)specs[i].latt[0] * specs[i].latt[1] * specs[i].latt[2] / 2;
    BatchItem &it = bp.items[i];
    for (int q = 0; q < 3; ++q) it.in[q] = specs[i].in[q];
    it.geom = make_geom(ji, Walk::SITES, warps, 3);  // the device queue balances the warps
    it.chunk_begin = chunks;
    it.lt = ji.lt;
    it.out = specs[i].out;
    chunks += it.geom.total_chunks;
    partial_total += (size_t)it.geom.total_chunks * Op::NOUT;
    max_lt = std::max<long long>(max_lt, ji.lt);
  }
  bp.total_chunks = chunks;
  // the partial sums, then the queue's counter
  const size_t partial_bytes = (partial_total * sizeof(double2) + 255) / 256 * 256;
  char *ws = static_cast<char *>(job.ws->get(partial_bytes + 256));
  if (!ws) return cudaErrorMemoryAllocation;
  double2 *partial = reinterpret_cast<double2 *>(ws);
  bp.queue = reinterpret_cast<unsigned int *>(ws + partial_bytes);
  size_t off = 0;
  for (int i = 0; i < n; ++i) {
    bp.items[i].partial = partial + off;
    off += (size_t)bp.items[i].geom.total_chunks * Op::NOUT;
  }
  const int grid = std::min((chunks + Op::CW - 1) / Op::CW, job.num_sms * bps);
  e = cudaMemsetAsync(bp.queue, 0, sizeof(unsigned int), job.stream);
  if (e != cudaSuccess) return e;
  warp_kernel<Op, Walk><<<grid, 32 * Op::CW, smem, job.stream>>>(bp);
  e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  if (fin) {
    fin->n_items = n;
    fin->nout = Op::NOUT;
    int blocks = 0;
    for (int i = 0; i < n; ++i) {
      BaryonFinItem &f = fin->items[i];
      f.partial = bp.items[i].partial;
      f.out = bp.items[i].out;
      f.lt = bp.items[i].lt;
      f.per_seg = bp.items[i].geom.chunks_per_seg;
      f.blk_begin = blocks;
      blocks += (Op::NOUT * f.lt + 255) / 256;
    }
    fin->total_blocks = blocks;
    return cudaSuccess;
  }
  const dim3 fg(n, (unsigned)((Op::NOUT * max_lt + 127) / 128));
  batch_finalize_kernel<R><<<fg, 128, 0, job.stream>>>(bp, Op::NOUT);
  return cudaGetLastError();
}

// Tile shapes of the batched launch (the autotuner's choice per batch: one
// shape serves every item of a launch).
template <int NG, int NW, bool SAME>
using BatchShapes = std::tuple<BaryonFusedOp<float, float2, 4, 8, NG, NW, SAME, 2>,
                               BaryonFusedOp<float, float2, 12, 8, NG, NW, SAME, 1>,
                               BaryonFusedOp<float, float2, 4, 16, NG, NW, SAME, 5>>;
static const char *const kBatchShapeNames[] = {"w4.tps8.occ2", "w12.tps8.occ1", "w4.tps16.occ5"};
static const char *const kBatchSameShapeNames[] = {"same.w4.tps8.occ2", "same.w12.tps8.occ1", "same.w4.tps16.occ5"};

template <class Tuple>
static cudaError_t run_shape(int v, const Job &job, const OpParams<float> &q, const BatchSpec *specs, int n,
                             BaryonFinParams *fin)
{
  switch (v) {
  case 1: return run_batch<std::tuple_element_t<1, Tuple>>(job, q, specs, n, fin);
  case 2: return run_batch<std::tuple_element_t<2, Tuple>>(job, q, specs, n, fin);
  default: return run_batch<std::tuple_element_t<0, Tuple>>(job, q, specs, n, fin);
  }
}

int batch_variants(bool same_field, const char *const **names)
{
  if (names) *names = same_field ? kBatchSameShapeNames : kBatchShapeNames;
  return 3;
}

bool batch_same_field(const OpParams<double> &p, const BatchSpec *specs, int n)
{
  bool same = n > 0;  // every item's P_i and P_j one field: the one-pass form
  for (int i = 0; i < n; ++i) same = same && specs[i].in[0] == specs[i].in[1];
  return same && p.b.perm1[0] != 0;
}

bool batch_rank_form(int nw, const OpParams<double> &p) { return nw == 1 && p.b.cl.ng > 1 && p.b.rk.r > 0; }

cudaError_t launch_baryon_fused_batch(const Job &job, int nw, const OpParams<double> &p, const BatchSpec *specs, int n,
                                      BaryonFinParams *fin)
{
  const int ng = p.b.cl.ng, v = job.variant;
  const bool rank = batch_rank_form(nw, p);
  if (!rank && ng > nw) return cudaErrorInvalidValue;
  OpParams<double> d = p;
  if (job.prec == Prec::C128) {
    fill_fused_spin(d, false);
    if (ng == 2) return nw == 1 ? run_batch<BaryonFusedOp<double, double2, 4, 16, 2, 1, false, 3>>(job, d, specs, n, fin)
                                : run_batch<BaryonFusedOp<double, double2, 4, 16, 2, 2, false, 3>>(job, d, specs, n, fin);
    if (ng > 2) return p.b.rk.r == 1 ? run_batch<BaryonFusedOp<double, double2, 4, 16, -1, 1, false, 3>>(job, d, specs, n, fin)
                                     : run_batch<BaryonFusedOp<double, double2, 4, 16, -2, 1, false, 3>>(job, d, specs, n, fin);
    return nw == 1 ? run_batch<BaryonFusedOp<double, double2, 4, 16, 1, 1, false, 3>>(job, d, specs, n, fin)
                   : run_batch<BaryonFusedOp<double, double2, 4, 16, 1, 2, false, 3>>(job, d, specs, n, fin);
  }
  OpParams<float> q = convert_params<float>(p);
  if (ng <= 2 && batch_same_field(p, specs, n)) {
    fill_fused_spin(q, true);
    std::vector<BatchSpec> one(specs, specs + n);  // inputs: the field once, then P_n
    for (BatchSpec &b : one) b.in[1] = b.in[2];
    if (ng == 2) return nw == 1 ? run_batch<BaryonFusedOp<float, float2, 4, 8, 2, 1, true, 2>>(job, q, one.data(), n, fin)
                                : run_shape<BatchShapes<2, 2, true>>(v, job, q, one.data(), n, fin);
    return nw == 1 ? run_shape<BatchShapes<1, 1, true>>(v, job, q, one.data(), n, fin)
                   : run_batch<BaryonFusedOp<float, float2, 4, 8, 1, 2, true, 2>>(job, q, one.data(), n, fin);
  }
  fill_fused_spin(q, false);
  if (ng == 2) return nw == 1 ? run_batch<BaryonFusedOp<float, float2, 4, 8, 2, 1, false, 2>>(job, q, specs, n, fin)
                              : run_shape<BatchShapes<2, 2, false>>(v, job, q, specs, n, fin);
  if (ng > 2) return p.b.rk.r == 1 ? run_batch<BaryonFusedOp<float, float2, 4, 8, -1, 1, false, 2>>(job, q, specs, n, fin)
                                   : run_batch<BaryonFusedOp<float, float2, 4, 8, -2, 1, false, 2>>(job, q, specs, n, fin);
  return nw == 1 ? run_shape<BatchShapes<1, 1, false>>(v, job, q, specs, n, fin)
                 : run_batch<BaryonFusedOp<float, float2, 4, 8, 1, 2, false, 2>>(job, q, specs, n, fin);
}

} // namespace cgb
