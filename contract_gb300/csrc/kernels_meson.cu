// Meson kernels: one Gamma pair per site, and the all-source / all-sink forms.
// Op template arguments: <R, S, warps, (threads per site,) ring stages, CTAs per SM>.
#include "launch_variants.cuh"
#include "ops_site.cuh"

namespace cgb {

// One Gamma pair.  complex128: FP64 pipe and HBM within a third of each other;
// 0.51 ms at 24^3 x 32 per site, 0.305 of it the two fields at the copy rate.
static const VariantSet<double, 4> kMesonP = {
  {run_ring<MesonOp<double, double2, 4, 8, 1, 3>>, run_ring<MesonOp<double, double2, 2, 8, 2, 3>>,
   run_ring<MesonOp<double, double2, 4, 16, 1, 5>>, run_ring<MesonOp<double, double2, 4, 16, 2, 2>>},
  {"w4.tps8.st1.occ3", "w2.tps8.st2.occ3", "w4.tps16.st1.occ5", "w4.tps16.st2.occ2"},
  0};
// complex64: HBM bound; sites in flight against warps.
static const VariantSet<float, 4> kMesonM = {
  {run_ring<MesonOp<float, float2, 4, 8, 1, 5>>, run_ring<MesonOp<float, float2, 4, 8, 2, 2>>,
   run_ring<MesonOp<float, float2, 4, 8, 4, 1>>, run_ring<MesonOp<float, float2, 4, 16, 2, 5>>},
  {"w4.tps8.st1.occ5", "w4.tps8.st2.occ2", "w4.tps8.st4.occ1", "w4.tps16.st2.occ5"},
  0};

cudaError_t launch_meson(const Job &job, const OpParams<double> &p)
{
  if (job.prec == Prec::C128) return kMesonP.launch(job, p);
  return kMesonM.launch(job, convert_params<float>(p));
}

// All partners of one Gamma.  complex128: 0.69 ms at 24^3 x 32 per site, a seventh of
// the FP64 form's time (2304 FP64 FMAs and 1536 adds a site, on two warps an SM);
// here the products run on the integer pipe.
// complex64 at 24^3 x 64 per timeslice: 0.311 (source) and 0.323 ms (sink) against
// 0.336, with 0.305 for the two fields at the copy rate: stages before warps.
template <bool SOURCE> static VariantSet<double, 3> all_p()
{
  return {{run_ring<MesonAllOp<double, double2, 4, 1, 4, SOURCE>>, run_ring<MesonAllOp<double, double2, 4, 2, 2, SOURCE>>,
           run_ring<MesonAllOp<double, double2, 4, 1, 3, SOURCE>>},
          {"w4.st1.occ4", "w4.st2.occ2", "w4.st1.occ3"},
          0};
}
template <bool SOURCE> static VariantSet<float, 4> all_m()
{
  return {{run_ring<MesonAllOp<float, float2, 4, 2, 5, SOURCE>>, run_ring<MesonAllOp<float, float2, 4, 3, 3, SOURCE>>,
           run_ring<MesonAllOp<float, float2, 4, 1, 8, SOURCE>>, run_ring<MesonAllOp<float, float2, 4, 4, 2, SOURCE>>},
          {"w4.st2.occ5", "w4.st3.occ3", "w4.st1.occ8", "w4.st4.occ2"},
          SOURCE ? 3 : 1};
}
static const VariantSet<double, 3> kMesonAllSrcP = all_p<true>(), kMesonAllSnkP = all_p<false>();
static const VariantSet<float, 4> kMesonAllSrcM = all_m<true>(), kMesonAllSnkM = all_m<false>();

cudaError_t launch_meson_all(const Job &job, bool source, const OpParams<double> &p)
{
  if (job.prec == Prec::C128) return source ? kMesonAllSrcP.launch(job, p) : kMesonAllSnkP.launch(job, p);
  const OpParams<float> q = convert_params<float>(p);
  return source ? kMesonAllSrcM.launch(job, q) : kMesonAllSnkM.launch(job, q);
}

int meson_all_variants(Prec prec, bool source, const char *const **names)
{
  if (prec == Prec::C128) return source ? kMesonAllSrcP.describe(names) : kMesonAllSnkP.describe(names);
  return source ? kMesonAllSrcM.describe(names) : kMesonAllSnkM.describe(names);
}

int meson_variants(Prec prec, const char *const **names)
{
  if (prec == Prec::C128) return kMesonP.describe(names);
  return kMesonM.describe(names);
}

} // namespace cgb
