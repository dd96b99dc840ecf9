// r-space sum of the FP64 path: forces, energies and virial of every site
// (cook/ljqqnp.c, cook/ljqqpol.c).
//
// The GPU's FP64 pipe is narrow (a warp's instruction holds an SM's for 16
// cycles, however few lanes take part), so a pair's 40-odd FP64 instructions
// are to run in full warps.  A warp takes one home site; its lanes test the
// sites of the stencil's cells, 32 at a time, in FP32 (nearest image, the
// cutoff widened by the rounding) and queue those inside, apart for pairs
// with a Lennard-Jones term, pairs of charges alone and pairs of one molecule
// (exact exclusion terms): 32 of a queue are then one full warp of one kind of
// work, each lane a neighbour, with the exact cutoff test in FP64.  The lanes'
// sums are added in a fixed order at the end.  Every pair is met from both
// ends: meeting it once would halve the arithmetic but scatter the reaction in
// FP64.  (A lane per home site of a cell left most lanes idle and ran each
// candidate's FP64 branch for a few of them: 1173 us on 864 waters, with energies
// and virial 1855; this 153 and 306, with 4 warps per CTA 173 and 307.  Bound by
// the FP64 pipe.)
#include "mg_internal.h"
#include "mg_device.cuh"
#include "mg_pair64.cuh"

namespace mg {

// The force arithmetic rounds explicitly (`_rn`): the measuring instantiation
// also uses the force for the virial, and a product fused in one instantiation
// and not in the other would move the sites of a measured step differently.
__device__ __forceinline__ double p64_r2(double dx, double dy, double dz) {
  return __fma_rn(dx, dx, __fma_rn(dy, dy, __dmul_rn(dz, dz)));
}
// force over separation of a pair of charges; energy to en[0]
template <bool MEASURE, bool EXCL>
__device__ __forceinline__ double p64_charge(const PairArgs& a, const double* __restrict__ ert,
                                             double r2, double qq, double* en) {
  double f, e;
  if (EXCL) {
    e = excl_term<double>(r2, a.alpha, &f);
  } else {
    const double* p = ert + 6 * min((int)(r2 * a.sgrid), a.ntab - 1);
    f = __dadd_rn(__ddiv_rn(p[4], __dadd_rn(p[5], r2)), p[3]);
    e = p[1] / (p[2] + r2) + p[0];
  }
  if (MEASURE) en[0] += e * qq;
  return __dmul_rn(f, qq);
}
template <bool MEASURE>
__device__ __forceinline__ void p64_add(double f, double dx, double dy, double dz, double& fx,
                                        double& fy, double& fz, double* en) {
  fx = __fma_rn(f, dx, fx);
  fy = __fma_rn(f, dy, fy);
  fz = __fma_rn(f, dz, fz);
  if (MEASURE) {
    const double fdx = f * dx, fdy = f * dy, fdz = f * dz;
    en[3] += dx * fdx;
    en[4] += dy * fdy;
    en[5] += dz * fdz;
    en[6] += dz * fdy;
    en[7] += dx * fdz;
    en[8] += dy * fdx;
  }
}

template <bool MEASURE, bool POLAR>
__global__ void __launch_bounds__(P64_THREADS)
    pair64_kernel(const __grid_constant__ PairArgs a, const double4* __restrict__ pd,
                  const float4* __restrict__ pf, const PairD* __restrict__ ptab_g,
                  const double* __restrict__ ert, float cqf) {
  extern __shared__ __align__(16) unsigned char p64_smem[];
  __shared__ P64Queue queue[P64_WARPS];
  __shared__ double ered[P64_WARPS][9];
  const int nk = a.nkind, nk2 = nk * nk;
  PairD* ptab = reinterpret_cast<PairD*>(p64_smem);
  unsigned char* flag = reinterpret_cast<unsigned char*>(ptab + nk2);
  for (int t = threadIdx.x; t < nk2; t += P64_THREADS) {
    const PairD P = ptab_g[t];
    ptab[t] = P;
    flag[t] = (unsigned char)((P.E24 != 0 || P.E4 != 0 || P.A != 0 || P.A4 != 0 ? 1 : 0) |
                              (P.qq != 0 || P.qpc != 0 || P.qcp != 0 || P.qpp != 0 ? 2 : 0));
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ti = blockIdx.x * P64_WARPS + warp;
  double en[NEN];
#pragma unroll
  for (int k = 0; k < NEN; k++) en[k] = 0;
  if (ti < a.ns) {
    const double4 me = pd[ti];
    const double4 md = POLAR ? a.pdd[ti] : make_double4(0, 0, 0, 0);
    const int kind_i = (int)(__double_as_longlong(me.w) & 255);
    const PairD* prow = ptab + kind_i * nk;
    const bool tight = p64_tight(a);
    double fx = 0, fy = 0, fz = 0, gx = 0, gy = 0, gz = 0;
    auto work = [&](auto cls, const int2 e, bool on) {
      constexpr int CLS = decltype(cls)::value;
      if (!on) return;
      const double4 q = pd[e.x];
      const double dx = p64_image(me.x - q.x, e.y, a.Lx, tight),
                   dy = p64_image(me.y - q.y, e.y >> 2, a.Ly, tight),
                   dz = p64_image(me.z - q.z, e.y >> 4, a.Lz, tight);
      const double rr = p64_r2(dx, dy, dz);
      if (!(rr < a.cutoff_sq)) return;
      const PairD& P = prow[e.y >> 8];
      constexpr bool excl = CLS == P64_EXCL;
      double ft = 0;   // the force of the pair, centres, over its separation
      if (CLS == P64_LJ && rr < P.C2q) {
        double f, U;
        if (rr < P.C1q) {
          const double x = __ddiv_rn(P.Sq, rr), y = __dmul_rn(__dmul_rn(x, x), x),
                       z = __dmul_rn(y, y);
          f = __dmul_rn(__dmul_rn(P.E24, __fma_rn(2, z, -y)), x);
          U = P.E4 * (z - y);
        } else {
          const double x = __dadd_rn(rr, -P.C2q);
          f = __dmul_rn(P.A4, x);
          U = x * x * P.A;
        }
        ft = f;
        if (MEASURE) {
          en[1] += U;
          en[2] += rr * f;
        }
      }
      if (P.qq != 0) ft = __dadd_rn(ft, p64_charge<MEASURE, excl>(a, ert, rr, P.qq, en));
      p64_add<MEASURE>(ft, dx, dy, dz, fx, fy, fz, en);
      if (POLAR) {
        const double4 qd = a.pdd[e.x];
        const double ux = dx + md.x, uy = dy + md.y, uz = dz + md.z;
        if (P.qpc != 0)
          p64_add<MEASURE>(p64_charge<MEASURE, excl>(a, ert, p64_r2(ux, uy, uz), P.qpc, en), ux, uy,
                           uz, gx, gy, gz, en);
        const double vx = dx - qd.x, vy = dy - qd.y, vz = dz - qd.z;
        if (P.qcp != 0)
          p64_add<MEASURE>(p64_charge<MEASURE, excl>(a, ert, p64_r2(vx, vy, vz), P.qcp, en), vx, vy,
                           vz, fx, fy, fz, en);
        const double wx = ux - qd.x, wy = uy - qd.y, wz = uz - qd.z;
        if (P.qpp != 0)
          p64_add<MEASURE>(p64_charge<MEASURE, excl>(a, ert, p64_r2(wx, wy, wz), P.qpp, en), wx, wy,
                           wz, gx, gy, gz, en);
      }
    };
    p64_walk(a, pf, ti, flag + kind_i * nk, queue[warp], cqf, work);
    fx = p64_sum(fx);
    fy = p64_sum(fy);
    fz = p64_sum(fz);
    if (POLAR) {
      gx = p64_sum(gx);
      gy = p64_sum(gy);
      gz = p64_sum(gz);
    }
    if (lane == 0) {
      double* f = a.f + 3 * (long)a.order[ti];
      f[0] = fx;
      f[1] = fy;
      f[2] = fz;
      if (POLAR) {
        f += 3 * (long)a.ns;
        f[0] = gx;
        f[1] = gy;
        f[2] = gz;
      }
    }
  }
  if (MEASURE) {
#pragma unroll
    for (int k = 0; k < 9; k++) {
      const double v = p64_sum(en[k]);
      if (lane == 0) ered[warp][k] = v;
    }
    __syncthreads();
    if (threadIdx.x < NEN) {
      double v = 0;
      if (threadIdx.x < 9)
        for (int w = 0; w < P64_WARPS; w++) v += ered[w][threadIdx.x];
      a.epart[(long)blockIdx.x * NEN + threadIdx.x] = 0.5 * v;
    }
  }
}

int pair64_blocks(int ns) { return (ns + P64_WARPS - 1) / P64_WARPS; }

cudaError_t k_pair_fp64(const Launch& L, const PairArgs& a, const double4* pd, const float4* pf,
                        const PairD* ptab, const double* ertab, bool measure, bool polar) {
  const int grid = pair64_blocks(a.ns);
  const size_t sm = (size_t)a.nkind * a.nkind * (sizeof(PairD) + 1);
  const float cqf = p64_cutoff(a);
  if (polar) {
    if (measure) pair64_kernel<true, true><<<grid, P64_THREADS, sm, L.s>>>(a, pd, pf, ptab, ertab, cqf);
    else pair64_kernel<false, true><<<grid, P64_THREADS, sm, L.s>>>(a, pd, pf, ptab, ertab, cqf);
  } else {
    if (measure) pair64_kernel<true, false><<<grid, P64_THREADS, sm, L.s>>>(a, pd, pf, ptab, ertab, cqf);
    else pair64_kernel<false, false><<<grid, P64_THREADS, sm, L.s>>>(a, pd, pf, ptab, ertab, cqf);
  }
  ++*L.counter;
  return cudaGetLastError();
}

}  // namespace mg
