// All six baryon contraction types (x up to two projectors) in one pass.
// Op template arguments: <R, S, warps, threads per site, open slot, projectors, one field, CTAs per SM>.
#include "launch_variants.cuh"
#include "ops_fused.cuh"

namespace cgb {

template <class Op> static cudaError_t run_warps(const Job &job, const OpParams<typename Op::R> &p)
{
  if (job.volume == 0) return cudaSuccess;
  constexpr size_t smem = WarpSmem<Op>::BYTES;
  static_assert(smem <= 232448, "op does not fit in shared memory");
  return launch_chunks<Op>(job, p, warp_kernel<Op, ChunkWalk<Op>>, smem);
}

template <class R, class S, int CW, int TPS, int SRC, int NW, bool SAME, int MINB>
static cudaError_t fused(const Job &job, OpParams<R> q)
{
  fill_fused_spin(q, SAME);
  if (SAME) q.in[1] = q.in[2];  // inputs: the field once, then P_n
  return run_warps<BaryonFusedOp<R, S, CW, TPS, SRC, NW, SAME, MINB>>(job, q);
}

// complex64 tile shapes: 16 threads a site (one block of G each) or 8 (two blocks of G each, which share the
// loads of one P_i block and take half the reduction).  At 24^3 x 64 with two projectors, two fields / one field:
// in this order 0.588 / 0.426 ms, 0.613 / 0.421, 0.622 / 0.429, 0.624 / 0.430, 0.636 / 0.437 and 0.675 / 0.473.
template <int SRC, int NW, bool SAME> static VariantSet<float, 7> shapes_m(int def)
{
  return {{fused<float, float2, 12, 8, SRC, NW, SAME, 1>, fused<float, float2, 4, 8, SRC, NW, SAME, 2>,
           fused<float, float2, 4, 8, SRC, NW, SAME, 3>, fused<float, float2, 2, 8, SRC, NW, SAME, 6>,
           fused<float, float2, 6, 8, SRC, NW, SAME, 2>, fused<float, float2, 4, 16, SRC, NW, SAME, 5>,
           fused<float, float2, 4, 16, SRC, NW, SAME, 4>},
          {"w12.tps8.occ1", "w4.tps8.occ2", "w4.tps8.occ3", "w2.tps8.occ6", "w6.tps8.occ2", "w4.tps16.occ5",
           "w4.tps16.occ4"},
          def};
}
static const VariantSet<float, 7> kFused1M = shapes_m<1, 1, false>(0), kFused2M = shapes_m<2, 2, false>(0),
                                  kSame1M = shapes_m<1, 1, true>(1), kSame2M = shapes_m<2, 2, true>(1);

// complex128 (integer pipe, fixed.cuh): 16^3 x 48 with two projectors, ms in this order, 1.59, 1.80 and 1.64
// (in FP64 only 4.24; the shared-wedge FP64 kernel before it 7.28).
template <int SRC, int NW> static VariantSet<double, 3> shapes_p()
{
  return {{fused<double, double2, 4, 16, SRC, NW, false, 3>, fused<double, double2, 4, 16, SRC, NW, false, 2>,
           fused<double, double2, 2, 16, SRC, NW, false, 7>},
          {"w4.tps16.occ3", "w4.tps16.occ2", "w2.tps16.occ7"},
          0};
}
static const VariantSet<double, 3> kFused1P = shapes_p<1, 1>(), kFused2P = shapes_p<2, 2>();

// The shapes without variants: one projector of two gamma-basis terms, two projectors of one common term, a
// projector of rank 1 or 2, and any projectors (N' per site).
template <class R, class S, int CW, int SRC, int NW>
static cudaError_t fused_one(const Job &job, const OpParams<R> &q)
{
  return fused<R, S, CW, sizeof(R) == 4 ? 8 : 16, SRC, NW, false, sizeof(R) == 4 ? 2 : 3>(job, q);
}

cudaError_t launch_baryon_fused(const Job &job, int nw, const OpParams<double> &p)
{
  const int ng = p.b.cl.ng;  // 0 for projectors that vanish: one term with coefficient 0
  // P_i and P_j one field: half the wedges, where Gamma_ij's permutation has no fixed point
  const bool same = fused_same_ij(p) && p.b.perm1[0] != 0;
  if (job.prec == Prec::C128) {
    if (ng <= 2) {
      if (same) {
        if (ng == 2) return nw == 1 ? fused<double, double2, 4, 16, 2, 1, true, 3>(job, p)
                                    : fused<double, double2, 4, 16, 2, 2, true, 3>(job, p);
        return nw == 1 ? fused<double, double2, 4, 16, 1, 1, true, 3>(job, p)
                       : fused<double, double2, 4, 16, 1, 2, true, 3>(job, p);
      }
      if (ng == 2) return nw == 1 ? fused_one<double, double2, 4, 2, 1>(job, p) : kFused2P.launch(job, p);
      return nw == 1 ? kFused1P.launch(job, p) : fused_one<double, double2, 4, 1, 2>(job, p);
    }
    if (nw == 1 && p.b.rk.r > 0)
      return p.b.rk.r == 1 ? fused_one<double, double2, 4, -1, 1>(job, p) : fused_one<double, double2, 4, -2, 1>(job, p);
    return nw == 1 ? fused_one<double, double2, 4, 0, 1>(job, p) : fused_one<double, double2, 4, 0, 2>(job, p);
  }
  const OpParams<float> q = convert_params<float>(p);
  if (ng <= 2) {
    if (same) {
      if (ng == 2) return nw == 1 ? fused<float, float2, 4, 8, 2, 1, true, 2>(job, q) : kSame2M.launch(job, q);
      return nw == 1 ? kSame1M.launch(job, q) : fused<float, float2, 4, 8, 1, 2, true, 2>(job, q);
    }
    if (ng == 2) return nw == 1 ? fused<float, float2, 4, 8, 2, 1, false, 2>(job, q) : kFused2M.launch(job, q);
    return nw == 1 ? kFused1M.launch(job, q) : fused<float, float2, 4, 8, 1, 2, false, 2>(job, q);
  }
  if (nw == 1 && q.b.rk.r > 0)
    return q.b.rk.r == 1 ? fused_one<float, float2, 4, -1, 1>(job, q) : fused_one<float, float2, 4, -2, 1>(job, q);
  return nw == 1 ? fused_one<float, float2, 4, 0, 1>(job, q) : fused_one<float, float2, 4, 0, 2>(job, q);
}

// aux = nw + 4 * (P_i and P_j one field)
int fused_variants(Prec prec, int aux, const char *const **names)
{
  const int nw = aux & 3;
  if (prec == Prec::C128) return (aux & 4) ? 1 : (nw == 1 ? kFused1P : kFused2P).describe(names);
  if (aux & 4) return (nw == 1 ? kSame1M : kSame2M).describe(names);
  return (nw == 1 ? kFused1M : kFused2M).describe(names);
}

} // namespace cgb
