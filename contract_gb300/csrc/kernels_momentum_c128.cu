// Complex128 meson momentum projection: Gamma pairs and X transform in one launch,
// then the Y transform per (t, z) plane and the Z transform per (nx, ny) and t.
//
// The pairs of a site run on the integer pipe (MesonPairs, ops_site.cuh), the
// transforms on the FP64 pipe; as two launches they took 0.77 and 0.83 ms at
// 18 x 15 x 20 x 28 with 125 momenta, each with the other's pipe idle.  Here a CTA
// has NI warps for the pairs and NF for the X sums: a pair warp takes sites x and
// Lx - x of a row (0 and Lx / 2 together), leaves their 2 x 256 pairs in its slot of
// shared memory and goes on to its next sites while the X warps, a thread per 4 or 8
// pairs, add the slots up in the order of x.  Only the X sums of a row leave the chip.
// 1.23 ms (both pipes about 60 % busy) where pairs, X and Y transform in two launches
// took 1.68 and the FP64 form 4.60; 24^3 x 16: one momentum 1.15 (1.60), 27 momenta 1.30
// (2.06), 125 momenta 1.68 (2.49), and 27 momenta where the fields refuse the integer form
// 5.52 (5.67 in the FP64 form).  Twelve pair warps make as many pairs as 16 did with
// an SM of their own.
#include "launch_variants.cuh"
#include "momentum.hpp"
#include "ops_site.cuh"

namespace cgb {

constexpr int kC128Warps = 16;
constexpr uint32_t kC128Site = 144 * 16, kC128In = kC128Site + 16, kC128Slot = 2 * 256 * 16;

struct RowsC128 {
  const char *in[2];
  double2 *g;  // [Lt][Lz][Ly][npx][256] X sums, pairs in the order of MesonPairs
  DeviceStatus *status;
  unsigned long long wait_ns;
  int withhold_row;  // test hook: this row's first sites never arrive; -1 in normal use
};

// Shared memory: in[NI], full[NI], empty[NI] mbarriers, abort flag at 504; phases; NI
// times two sites of two fields; NI slots.
template <int NG> constexpr size_t rows_c128_phases() { return (size_t)NG * (kMomMaxL / 2 + 1) * 16; }
template <int NG, int NI> constexpr size_t rows_c128_smem()
{
  return 512 + rows_c128_phases<NG>() + (size_t)NI * (4 * kC128In + kC128Slot);
}

template <int NG, int NF>
__global__ void __launch_bounds__(32 * kC128Warps, 1) rows_c128_kernel(const RowsC128 a, const __grid_constant__ MomPlan plan)
{
  constexpr int NI = kC128Warps - NF, NC = 256 / (32 * NF);  // pair warps; columns of an X thread
  extern __shared__ __align__(128) unsigned char smem[];
  uint64_t *in_bar = reinterpret_cast<uint64_t *>(smem), *full = in_bar + NI, *empty = full + NI;
  volatile int *abort_flag = reinterpret_cast<volatile int *>(smem + 504);
  double2 *phx = reinterpret_cast<double2 *>(smem + 512);  // [NG][Lx / 2 + 1] cos, sin of 2 pi k x / Lx
  unsigned char *inputs = smem + 512 + rows_c128_phases<NG>();
  unsigned char *slots = inputs + (size_t)NI * 4 * kC128In;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int lx = plan.latt[0], ly = plan.latt[1], lz = plan.latt[2], lt = plan.latt[3], half = lx / 2;
  if (threadIdx.x == 0) {
    for (int w = 0; w < NI; ++w) {
      mbar_init(&in_bar[w], 1);
      mbar_init(&full[w], 1);
      mbar_init(&empty[w], NF);
    }
    *abort_flag = 0;
    fence_barrier_init();
  }
  for (int e = threadIdx.x; e < NG * (half + 1); e += blockDim.x) {
    const int gi = e / (half + 1), x = e % (half + 1), k = (plan.gx_k[gi] * x) % lx;
    phx[e] = make_double2(plan.cosx[k], plan.sinx[k]);
  }
  __syncthreads();
  // This CTA's rows blockIdx, blockIdx + grid, ..., Lx / 2 pairs of sites each.
  const int rows = lt * lz * ly, mine = (int)blockIdx.x < rows ? (rows - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
  const long long tiles = (long long)mine * half;
  auto wait = [&](uint64_t *bar, uint32_t parity) -> bool {
    const bool ok = mbar_wait_bounded(bar, parity, a.wait_ns);
    if (__all_sync(0xffffffffu, ok) && !*abort_flag) return true;
    if (lane == 0) {
      *abort_flag = 1;
      report(a.status, kDevErrWaitTimeout, blockIdx.x);
    }
    return false;
  };

  if (warp < NI) {
    unsigned char *in = inputs + (size_t)warp * 4 * kC128In;
    const int local = lane >> 4, sub = lane & 15;
    double2 *field[2] = {reinterpret_cast<double2 *>(in + (0 * 2 + local) * kC128In),
                         reinterpret_cast<double2 *>(in + (1 * 2 + local) * kC128In)};
    double2 *dst = reinterpret_cast<double2 *>(slots + (size_t)warp * kC128Slot) + local * 256;
    auto fetch = [&](long long T) {
      const int k = (int)(T / half), j = (int)(T - (long long)k * half);
      int row = (int)blockIdx.x + k * (int)gridDim.x;
      if (row == a.withhold_row && j == 0) return;
      if (lane == 0) mbar_arrive_expect_tx(&in_bar[warp], 4 * kC128Site);
      __syncwarp();
      if (lane < 4) {
        const int q = lane >> 1, s = lane & 1, x = j ? (s ? lx - j : j) : (s ? half : 0);
        const int y = row % ly;
        row /= ly;
        const int z = row % lz, t = row / lz, par = (x + y + z + t) & 1;
        const long long site = ((((long long)par * lt + t) * lz + z) * ly + y) * half + (x >> 1);
        bulk_g2s(in + lane * kC128In, a.in[q] + site * kC128Site, kC128Site, &in_bar[warp]);
      }
    };
    if (warp < tiles) fetch(warp);
    uint32_t n = 0;
    for (long long T = warp; T < tiles; T += NI, ++n) {
      if (!wait(&in_bar[warp], n & 1)) {
        if (lane == 0) mbar_wait_bounded(&in_bar[warp], n & 1, a.wait_ns / 8);  // the copies that may still be in flight
        return;
      }
      bool ok = true;
      MesonPairs::site(field, sub, true, dst, [&] {
        // the fields have been read: the next ones may come, then the slot must be free
        fence_proxy_async_smem();
        __syncwarp();
        if (T + NI < tiles) fetch(T + NI);
        if (n > 0) ok = wait(&empty[warp], (n - 1) & 1);
      });
      if (!ok) {  // the pairs went to a slot that nobody reads any more
        if (lane == 0 && T + NI < tiles) mbar_wait_bounded(&in_bar[warp], (n + 1) & 1, a.wait_ns / 8);
        return;
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&full[warp]);
    }
    return;
  }

  const int f = (warp - NI) * 32 + lane;
  const bool zero = plan.gx_k[0] == 0;  // the k = 0 group, if there is one, is the first
  cx<double> gc[NG][NC], gs[NG][NC];
  int w = 0;
  uint32_t n = 0;
  for (int k = 0; k < mine; ++k) {
#pragma unroll
    for (int gi = 0; gi < NG; ++gi)
#pragma unroll
      for (int c = 0; c < NC; ++c) gc[gi][c] = gs[gi][c] = czero<double>();
    for (int j = 0; j < half; ++j) {
      if (!wait(&full[w], n & 1)) return;
      const double2 *slot = reinterpret_cast<const double2 *>(slots + (size_t)w * kC128Slot) + f;
      cx<double> v[NC], u[NC];
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        v[c] = ld<double>(slot + c * 32 * NF);
        u[c] = ld<double>(slot + 256 + c * 32 * NF);
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty[w]);
      if (++w == NI) {
        w = 0;
        ++n;
      }
      // sites 0 and Lx / 2 have no partner: cos v + cos u, the sine of the first is 0
      const int x = j ? j : half;
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        const cx<double> s = cadd(v[c], u[c]), d = j ? cx<double> {v[c].x - u[c].x, v[c].y - u[c].y} : u[c];
#pragma unroll
        for (int gi = 0; gi < NG; ++gi) {
          if (gi == 0 && zero) {
            gc[0][c] = cadd(gc[0][c], s);
            continue;
          }
          const double2 ph = phx[gi * (half + 1) + x];
          const cx<double> e = j ? s : u[c];
          if (!j) gc[gi][c] = cadd(gc[gi][c], v[c]);
          gc[gi][c] = {fma(ph.x, e.x, gc[gi][c].x), fma(ph.x, e.y, gc[gi][c].y)};
          gs[gi][c] = {fma(ph.y, d.x, gs[gi][c].x), fma(ph.y, d.y, gs[gi][c].y)};
        }
      }
    }
    double2 *out = a.g + ((size_t)blockIdx.x + (size_t)k * gridDim.x) * plan.npx * 256 + f;
#pragma unroll
    for (int gi = 0; gi < NG; ++gi) {  // G(+k) = C + iS, G(-k) = C - iS
      const int plus = plan.gx_plus[gi], minus = plan.gx_minus[gi];
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        const cx<double> p = gc[gi][c], s = gs[gi][c];
        if (plus >= 0) out[plus * 256 + c * 32 * NF] = make_double2(p.x - s.y, p.y + s.x);
        if (minus >= 0) out[minus * 256 + c * 32 * NF] = make_double2(p.x + s.y, p.y - s.x);
      }
    }
  }
}

// Y transform of a (t, z) plane's X sums, YC groups of (nx, +-ny); one thread per
// pair.  Rows y and Ly - y have the same cosine and opposite sines: their sum and
// difference, through the thread's own column of shared memory, serve every ny.  FP64
// pipe 83 % busy, 0.2 ms at the size above.
template <int YC>
__global__ void __launch_bounds__(256) y_c128_kernel(const double2 *__restrict__ g, double2 *__restrict__ planes,
                                                     const __grid_constant__ MomPlan plan)
{
  const int z = blockIdx.x, t = blockIdx.y, y0 = blockIdx.z * YC;
  const int ly = plan.latt[1], lz = plan.latt[2], npx = plan.npx, ny = min(YC, plan.nyg - y0);
  __shared__ double2 phy[YC][kMomMaxL / 2 + 1];
  __shared__ int ygx[YC], odd[YC];  // odd: the group has a sine sum
  extern __shared__ __align__(16) double2 cols[];  // [2][npx][256]
  double2 *gp = cols + threadIdx.x, *gm = gp + npx * 256;
  if (threadIdx.x < YC) {
    const bool in = (int)threadIdx.x < ny;
    ygx[threadIdx.x] = in ? plan.yg_ix[y0 + threadIdx.x] : 0;
    odd[threadIdx.x] = in && plan.yg_k[y0 + threadIdx.x] != 0;
  }
  for (int e = threadIdx.x; e < YC * (ly / 2 + 1); e += blockDim.x) {
    const int q = e / (ly / 2 + 1), y = e % (ly / 2 + 1), k = q < ny ? (plan.yg_k[y0 + q] * y) % ly : 0;
    phy[q][y] = q < ny ? make_double2(plan.cosy[k], plan.siny[k]) : make_double2(0.0, 0.0);
  }
  __syncthreads();
  grid_dependency_wait();
  cx<double> hc[YC], hs[YC];
#pragma unroll
  for (int q = 0; q < YC; ++q) hc[q] = hs[q] = czero<double>();
  const double2 *plane = g + (size_t)(t * lz + z) * ly * npx * 256 + threadIdx.x;
  for (int y = 0; y <= ly / 2; ++y) {
    const bool alone = y == 0 || 2 * y == ly;
    const double2 *r0 = plane + (size_t)y * npx * 256, *r1 = plane + (size_t)(alone ? y : ly - y) * npx * 256;
#pragma unroll 4
    for (int ix = 0; ix < npx; ++ix) {
      const double2 v = r0[ix * 256], u = r1[ix * 256];
      gp[ix * 256] = alone ? v : make_double2(v.x + u.x, v.y + u.y);
      gm[ix * 256] = alone ? v : make_double2(v.x - u.x, v.y - u.y);
    }
#pragma unroll
    for (int q = 0; q < YC; ++q) {
      const double2 p = gp[ygx[q] * 256], ph = phy[q][y];
      hc[q] = {fma(ph.x, p.x, hc[q].x), fma(ph.x, p.y, hc[q].y)};
      if (odd[q]) {  // the same for every thread
        const double2 d = gm[ygx[q] * 256];
        hs[q] = {fma(ph.y, d.x, hs[q].x), fma(ph.y, d.y, hs[q].y)};
      }
    }
  }
  double2 *out = planes + (size_t)(t * lz + z) * plan.nq * 256 + threadIdx.x;
#pragma unroll
  for (int q = 0; q < YC; ++q) {
    if (q >= ny) break;
    const int qp = plan.yg_plus[y0 + q], qm = plan.yg_minus[y0 + q];
    if (qp >= 0) out[(size_t)qp * 256] = make_double2(hc[q].x - hs[q].y, hc[q].y + hs[q].x);
    if (qm >= 0) out[(size_t)qm * 256] = make_double2(hc[q].x + hs[q].y, hc[q].y - hs[q].x);
  }
}

// out[p][t][pair] = sum_z exp(2 pi i nz z / Lz) planes[t][z][q(p)]: a CTA per ((nx, ny)
// pair q, t), CNT Z groups of it at a time, z and Lz - z together.
template <int CNT>
__global__ void __launch_bounds__(256) z_c128_kernel(const double2 *__restrict__ planes, double2 *__restrict__ out,
                                                     const __grid_constant__ MomPlan plan)
{
  const int q = blockIdx.x, t = blockIdx.y, lz = plan.latt[2], lt = plan.latt[3];
  __shared__ double2 phz[kMomMaxL];
  for (int k = threadIdx.x; k < lz; k += blockDim.x) phz[k] = make_double2(plan.cosz[k], plan.sinz[k]);
  __syncthreads();
  grid_dependency_wait();
  const int at = pair_of_class(threadIdx.x), g0 = plan.q_g0[q], g1 = plan.q_g0[q + 1];
  const double2 *col = planes + ((size_t)t * lz * plan.nq + q) * 256 + threadIdx.x;
  const size_t step = (size_t)plan.nq * 256;
  for (int base = g0; base < g1; base += CNT) {
    cx<double> c[CNT], s[CNT];
    int kz[CNT], k1[CNT];  // k z mod Lz, k
#pragma unroll
    for (int k = 0; k < CNT; ++k) {
      c[k] = s[k] = czero<double>();
      kz[k] = 0;
      k1[k] = base + k < g1 ? plan.gz_k[base + k] : 0;
    }
    constexpr int ZB = 4;  // pairs of loads in flight per thread
    for (int z0 = 0; z0 <= lz / 2; z0 += ZB) {
      cx<double> v[ZB], u[ZB];
#pragma unroll
      for (int b = 0; b < ZB; ++b) {
        const int z = z0 + b;
        v[b] = z <= lz / 2 ? ld<double>(col + z * step) : czero<double>();
        u[b] = z > 0 && 2 * z < lz ? ld<double>(col + (lz - z) * step) : czero<double>();
      }
#pragma unroll
      for (int b = 0; b < ZB; ++b) {
        if (z0 + b > lz / 2) break;
        const cx<double> e = cadd(v[b], u[b]), d = {v[b].x - u[b].x, v[b].y - u[b].y};
#pragma unroll
        for (int k = 0; k < CNT; ++k) {
          if (base + k >= g1) break;
          if (k1[k] == 0) {
            c[k] = cadd(c[k], e);
            continue;
          }
          const double2 ph = phz[kz[k]];
          c[k] = {fma(ph.x, e.x, c[k].x), fma(ph.x, e.y, c[k].y)};
          s[k] = {fma(ph.y, d.x, s[k].x), fma(ph.y, d.y, s[k].y)};
          if ((kz[k] += k1[k]) >= lz) kz[k] -= lz;
        }
      }
    }
#pragma unroll
    for (int k = 0; k < CNT; ++k) {
      if (base + k >= g1) break;
      const int pp = plan.gz_plus[base + k], pm = plan.gz_minus[base + k];
      if (pp >= 0) out[((size_t)pp * lt + t) * 256 + at] = make_double2(c[k].x - s[k].y, c[k].y + s[k].x);
      if (pm >= 0) out[((size_t)pm * lt + t) * 256 + at] = make_double2(c[k].x + s[k].y, c[k].y - s[k].x);
    }
  }
}

template <int NG, int NF> static cudaError_t launch_rows(const Job &job, const RowsC128 &a, const MomPlan &plan)
{
  constexpr size_t smem = rows_c128_smem<NG, kC128Warps - NF>();
  static_assert(smem <= 232448, "the rings do not fit in shared memory");
  const cudaError_t e =
    cudaFuncSetAttribute(rows_c128_kernel<NG, NF>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  const int rows = plan.latt[1] * plan.latt[2] * plan.latt[3];
  rows_c128_kernel<NG, NF><<<std::min(rows, job.num_sms), 32 * kC128Warps, smem, job.stream>>>(a, plan);
  return cudaGetLastError();
}
template <int YC> static cudaError_t launch_y(const Job &job, const double2 *g, double2 *planes, const MomPlan &plan)
{
  const size_t smem = (size_t)2 * plan.npx * 256 * sizeof(double2);
  if (smem > 32768) {
    const cudaError_t e = cudaFuncSetAttribute(y_c128_kernel<YC>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               2 * kMomMaxPx * 256 * (int)sizeof(double2));
    if (e != cudaSuccess) return e;
  }
  const dim3 grid(plan.latt[2], plan.latt[3], (plan.nyg + YC - 1) / YC);
  return launch_overlapped(y_c128_kernel<YC>, grid, 256, smem, job.stream, g, planes, plan);
}

// The plan with one X sum for all nx that agree modulo Lx: at most Lx a row, so that
// the row sums never take more room than the pairs of every site would.
static void merge_nx(MomPlan &plan)
{
  const int lx = plan.latt[0];
  int sum[kMomMaxPx], n = 0;
  for (int ip = 0; ip < plan.npx; ++ip) {
    int j = 0;
    while (j < n && (plan.px[ip] - plan.px[j]) % lx != 0) ++j;
    if (j == n) plan.px[n++] = plan.px[ip];
    sum[ip] = j;
  }
  if (n == plan.npx) return;
  plan.npx = n;
  for (int g = 0; g < plan.nyg; ++g) plan.yg_ix[g] = sum[plan.yg_ix[g]];
  int groups = 0;  // the groups keep their order, k = 0 first; those of repeated nx go
  for (int g = 0; g < plan.ngx; ++g) {
    int seen = 0;
    while (seen < groups && plan.gx_k[seen] != plan.gx_k[g]) ++seen;
    const int plus = plan.gx_plus[g] < 0 ? -1 : sum[plan.gx_plus[g]];
    const int minus = plan.gx_minus[g] < 0 ? -1 : sum[plan.gx_minus[g]];
    if (seen == groups) {
      plan.gx_k[groups] = plan.gx_k[g];
      plan.gx_plus[groups] = plan.gx_minus[groups] = -1;
      ++groups;
    }
    if (plus >= 0) plan.gx_plus[seen] = plus;
    if (minus >= 0) plan.gx_minus[seen] = minus;
  }
  plan.ngx = groups;
}

size_t momentum_c128_row_bytes(MomPlan plan)
{
  merge_nx(plan);
  return (size_t)plan.latt[1] * plan.latt[2] * plan.latt[3] * plan.npx * 256 * sizeof(double2);
}

cudaError_t launch_momentum_c128(const Job &job, const void *in_i, const void *in_j, double2 *row_sums, double2 *planes,
                                 double2 *out, MomPlan plan)
{
  merge_nx(plan);
  RowsC128 a {};
  a.in[0] = static_cast<const char *>(in_i);
  a.in[1] = static_cast<const char *>(in_j);
  a.g = row_sums;
  a.status = job.status;
  a.wait_ns = job.wait_ns ? job.wait_ns : kWaitLimitNs;
  a.withhold_row = job.withhold_chunk;
  cudaError_t e;
  // More X groups: a thread per pair, for its registers, and fewer pair warps.
  switch (plan.ngx) {
  case 1: e = launch_rows<1, 4>(job, a, plan); break;
  case 2: e = launch_rows<2, 4>(job, a, plan); break;
  case 3: e = launch_rows<3, 4>(job, a, plan); break;
  case 4: e = launch_rows<4, 8>(job, a, plan); break;
  case 5: e = launch_rows<5, 8>(job, a, plan); break;
  case 6: e = launch_rows<6, 8>(job, a, plan); break;
  case 7: e = launch_rows<7, 8>(job, a, plan); break;
  case 8: e = launch_rows<8, 8>(job, a, plan); break;
  default: return cudaErrorInvalidValue;
  }
  if (e != cudaSuccess) return e;
  // few enough accumulators for the list, or chunks of 15
  if (plan.nyg <= 2) e = launch_y<2>(job, row_sums, planes, plan);
  else if (plan.nyg <= 6) e = launch_y<6>(job, row_sums, planes, plan);
  else e = launch_y<kMomYChunk>(job, row_sums, planes, plan);
  if (e != cudaSuccess) return e;
  int most = 1;  // Z groups of the pair with the most
  for (int q = 0; q < plan.nq; ++q) most = std::max(most, plan.q_g0[q + 1] - plan.q_g0[q]);
  const dim3 grid(plan.nq, plan.latt[3]);
  auto *const z = most <= 1 ? z_c128_kernel<1> : most <= 2 ? z_c128_kernel<2> : most <= 3 ? z_c128_kernel<3> : z_c128_kernel<6>;
  return launch_overlapped(z, grid, 256, 0, job.stream, planes, out, plan);
}

} // namespace cgb
