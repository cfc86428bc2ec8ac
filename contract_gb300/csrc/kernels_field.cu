// Field-valued kernels: diquark and sequential sources.
// Op template arguments: <R, S, warps, ring stages, CTAs per SM, wedges>.
#include "launch_variants.cuh"
#include "ops_field.cuh"

namespace cgb {

template <class R, class S, int CW, int NST, int MINB, Wedges KIND>
static cudaError_t wedges(const Job &job, OpParams<R> p)
{
  fill_wedges(p, KIND);
  return run_field_ring<WedgeFieldOp<R, S, CW, NST, MINB, KIND>>(job, p);
}

// complex64: HBM bound; tiles in flight against warps.  32^3 x 48, ms in this order:
// diquark 0.911, 0.950, 0.918, 1.07, four-wedge sequential sources 0.90 to 0.92,
// 0.93 to 0.94, 0.90 to 0.92, 1.05, loop ones 0.83 to 0.84, 0.87 to 0.90, 0.83 to 0.85,
// 0.87 to 0.90 (a CTA-wide ring with a producer warp: 1.00, 1.24, 0.86); the three
// fields take 0.814 at the copy rate.
template <Wedges KIND> static VariantSet<float, 4> shapes_m()
{
  return {{wedges<float, float2, 4, 2, 5, KIND>, wedges<float, float2, 4, 3, 4, KIND>, wedges<float, float2, 4, 2, 6, KIND>,
           wedges<float, float2, 4, 4, 3, KIND>},
          {"w4.st2.occ5", "w4.st3.occ4", "w4.st2.occ6", "w4.st4.occ3"},
          0};
}
// complex128: integer pipe.  24^4, ms in this order: four wedges a block 1.83 to 1.88,
// 1.90 to 1.93, 1.88 to 1.90 (5.2 to 5.7 in FP64 on a CTA-wide ring; where the fields refuse the
// integer form 5.3), the closed loop 0.75, 0.86, 0.82 (2.29).  One wedge a block runs in
// FP64 (WedgeFieldOp::with_q): 1.71, 1.44, 1.44.
template <Wedges KIND> static VariantSet<double, 3> shapes_p()
{
  return {{wedges<double, double2, 4, 3, 2, KIND>, wedges<double, double2, 4, 2, 3, KIND>,
           wedges<double, double2, 4, 2, 2, KIND>},
          {"w4.st3.occ2", "w4.st2.occ3", "w4.st2.occ2"},
          KIND == Wedges::LoopA || KIND == Wedges::LoopB ? 1 : 0};
}

static const VariantSet<float, 4> kDiquarkM = shapes_m<Wedges::Diquark>();
static const VariantSet<double, 3> kDiquarkP = shapes_p<Wedges::Diquark>();
// [loop][role]
static const VariantSet<float, 4> kSequentialM[2][3] = {
  {shapes_m<Wedges::TriA>(), shapes_m<Wedges::TriB>(), shapes_m<Wedges::TriN>()},
  {shapes_m<Wedges::LoopA>(), shapes_m<Wedges::LoopB>(), shapes_m<Wedges::LoopN>()}};
static const VariantSet<double, 3> kSequentialP[2][3] = {
  {shapes_p<Wedges::TriA>(), shapes_p<Wedges::TriB>(), shapes_p<Wedges::TriN>()},
  {shapes_p<Wedges::LoopA>(), shapes_p<Wedges::LoopB>(), shapes_p<Wedges::LoopN>()}};

cudaError_t launch_diquark(const Job &job, const OpParams<double> &p)
{
  if (job.prec == Prec::C128) return kDiquarkP.launch(job, p);
  return kDiquarkM.launch(job, convert_params<float>(p));
}

cudaError_t launch_sequential(const Job &job, bool loop, int role, const OpParams<double> &p)
{
  if (job.prec == Prec::C128) return kSequentialP[loop][role].launch(job, p);
  return kSequentialM[loop][role].launch(job, convert_params<float>(p));
}

int field_variants(Prec prec, bool sequential, const char *const **names)
{
  if (prec == Prec::C128) return (sequential ? kSequentialP[0][0] : kDiquarkP).describe(names);
  return (sequential ? kSequentialM[0][0] : kDiquarkM).describe(names);
}

} // namespace cgb
