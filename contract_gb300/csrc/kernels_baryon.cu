// Baryon two-point kernels, one contraction type per launch.
// Op template arguments: <R, S, warps, (threads per site,) ring stages, CTAs per SM>.
#include "launch_variants.cuh"
#include "ops_site.cuh"

namespace cgb {

// One or two factors: kernels of their own, each with the registers that its sums need.
template <class R, class S, int CW, int NST, int MINB> static cudaError_t run_rank(const Job &job, OpParams<R> p)
{
  fill_fused_spin(p, false);
  return p.b.rk.r == 2 ? run_ring<BaryonTriRankOp<R, S, CW, NST, MINB, true>>(job, p)
                       : run_ring<BaryonTriRankOp<R, S, CW, NST, MINB, false>>(job, p);
}

// complex128 on the integer pipe (fixed.cuh): bound by IMAD.WIDE issue and the
// conversions, so warps in flight count and a second ring stage, which costs warps,
// does not pay.  24^3 x 32 per site, three different fields, ms (the FP64 kernels
// that these replaced in brackets): loop 0.91 [2.86 with a projector of two terms],
// one gamma matrix 2.33, dense projector 3.43, rank 2 1.45 [4.65], a polarised projector
// (rank 1) 1.02, four terms a vector 1.69.  On fields that the integer form refuses, at
// 24^3 x 16 (replaced kernels in brackets; accepted in parentheses): loop 1.26 [1.46]
// (0.54), gamma 3.70 [3.78] (1.19), dense 4.46 to 4.70 [4.65] (1.78), rank 2 2.15 [2.35]
// (0.78), rank 1 1.25 to 1.65 [1.52 to 2.09] (0.55 to 0.88).
static const VariantSet<double, 4> kLoopP = {
  {run_ring<BaryonLoopOp<double, double2, 4, 16, 1, 3>>, run_ring<BaryonLoopOp<double, double2, 4, 16, 1, 2>>,
   run_ring<BaryonLoopOp<double, double2, 2, 16, 1, 6>>, run_ring<BaryonLoopOp<double, double2, 13, 16, 1, 1>>},
  {"w4.st1.occ3", "w4.st1.occ2", "w2.st1.occ6", "w13.st1.occ1"},
  0};
// Dense: 12 warps, three a scheduler, which matters where the fields refuse the integer form and the FP64 pipe bounds
// all warps alike: 24^3 x 16 1.81 ms, refused 4.68; ten warps 1.85 and 4.87 (in five CTAs) or 1.96 and 4.73 (in one).
static const VariantSet<double, 4> kTriP = {
  {run_ring<BaryonTriOp<double, double2, 12, 1, 1>>, run_ring<BaryonTriOp<double, double2, 2, 1, 5>>,
   run_ring<BaryonTriOp<double, double2, 4, 1, 2>>, run_ring<BaryonTriOp<double, double2, 10, 1, 1>>},
  {"w12.st1.occ1", "w2.st1.occ5", "w4.st1.occ2", "w10.st1.occ1"},
  0};
static const VariantSet<double, 4> kTriRankP = {
  {run_rank<double, double2, 4, 1, 3>, run_rank<double, double2, 12, 1, 1>,
   run_rank<double, double2, 4, 1, 2>, run_rank<double, double2, 10, 1, 1>},
  {"w4.st1.occ3", "w12.st1.occ1", "w4.st1.occ2", "w10.st1.occ1"},
  0};
static const VariantSet<double, 4> kTriGammaP = {
  {run_ring<BaryonTriGammaOp<double, double2, 4, 16, 1, 3>>, run_ring<BaryonTriGammaOp<double, double2, 4, 16, 1, 2>>,
   run_ring<BaryonTriGammaOp<double, double2, 2, 16, 1, 6>>, run_ring<BaryonTriGammaOp<double, double2, 4, 16, 2, 1>>},
  {"w4.st1.occ3", "w4.st1.occ2", "w2.st1.occ6", "w4.st2.occ1"},
  0};

// complex64: HBM bound; sites in flight against warps.  24^3 x 64 per timeslice, ms
// (one producer warp and a CTA-wide ring before, in brackets): loop 0.436 [0.440],
// one gamma matrix 0.500 [0.565], dense 0.563 [0.655], rank 2 0.445 [0.492],
// rank 1 0.432; the three fields take 0.457 ms at the copy rate's 6.68 TB/s.
static const VariantSet<float, 4> kLoopM = {
  {run_ring<BaryonLoopOp<float, float2, 4, 8, 1, 3>>, run_ring<BaryonLoopOp<float, float2, 4, 16, 1, 6>>,
   run_ring<BaryonLoopOp<float, float2, 3, 8, 2, 2>>, run_ring<BaryonLoopOp<float, float2, 4, 16, 2, 3>>},
  {"w4.tps8.st1.occ3", "w4.tps16.st1.occ6", "w3.tps8.st2.occ2", "w4.tps16.st2.occ3"},
  0};
static const VariantSet<float, 4> kTriM = {
  {run_ring<BaryonTriOp<float, float2, 4, 1, 5>>, run_ring<BaryonTriOp<float, float2, 4, 2, 3>>,
   run_ring<BaryonTriOp<float, float2, 3, 2, 4>>, run_ring<BaryonTriOp<float, float2, 4, 1, 4>>},
  {"w4.st1.occ5", "w4.st2.occ3", "w3.st2.occ4", "w4.st1.occ4"},
  0};
static const VariantSet<float, 4> kTriRankM = {
  {run_rank<float, float2, 4, 1, 3>, run_rank<float, float2, 3, 1, 5>,
   run_rank<float, float2, 5, 1, 3>, run_rank<float, float2, 8, 1, 2>},
  {"w4.st1.occ3", "w3.st1.occ5", "w5.st1.occ3", "w8.st1.occ2"},
  0};
static const VariantSet<float, 4> kTriGammaM = {
  {run_ring<BaryonTriGammaOp<float, float2, 4, 16, 1, 5>>, run_ring<BaryonTriGammaOp<float, float2, 4, 16, 2, 3>>,
   run_ring<BaryonTriGammaOp<float, float2, 4, 16, 1, 6>>, run_ring<BaryonTriGammaOp<float, float2, 4, 8, 1, 3>>},
  {"w4.tps16.st1.occ5", "w4.tps16.st2.occ3", "w4.tps16.st1.occ6", "w4.tps8.st1.occ3"},
  0};

cudaError_t launch_baryon(const Job &job, bool loop, const OpParams<double> &p)
{
  // A projector that is one gamma matrix (baryon_two_point) needs no N' buffer;
  // one of rank <= 2 takes the factored form.
  const bool gamma = p.b.cl.ng == 1, rank = !gamma && p.b.rk.r > 0;
  if (job.prec == Prec::C128) {
    if (loop) return kLoopP.launch(job, p);
    if (rank) return kTriRankP.launch(job, p);
    return gamma ? kTriGammaP.launch(job, p) : kTriP.launch(job, p);
  }
  const OpParams<float> q = convert_params<float>(p);
  if (loop) return kLoopM.launch(job, q);
  if (rank) return kTriRankM.launch(job, q);
  return gamma ? kTriGammaM.launch(job, q) : kTriM.launch(job, q);
}

// form: 0 loop, 1 triangle with one gamma, 2 triangle with N' materialised,
// 3 triangle with a projector of rank <= 2.
int baryon_variants(Prec prec, int form, const char *const **names)
{
  if (prec == Prec::C128) {
    if (form == 0) return kLoopP.describe(names);
    if (form == 3) return kTriRankP.describe(names);
    return form == 1 ? kTriGammaP.describe(names) : kTriP.describe(names);
  }
  if (form == 0) return kLoopM.describe(names);
  if (form == 3) return kTriRankM.describe(names);
  return form == 1 ? kTriGammaM.describe(names) : kTriM.describe(names);
}

} // namespace cgb
