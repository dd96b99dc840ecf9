// sm_103a kernels of the cook force path.
//
//   cell list      k_cell_list: a counting sort of the sites by cell (count,
//                  scan, scatter, per-cell rank) with the fixed-point site
//                  records of the FP32 path; k_gather_* for the FP64 path
//   r-space sum    k_pair_mixed: the half-shell kernel (every pair once, a warp
//                  on 8 home sites, lanes on the neighbours), the all-pairs
//                  kernel of small boxes, the cell and the group kernel;
//                  k_excl_mixed: the Ewald terms of pairs within a molecule.
//                  The FP64 path: mg_pair64.cu
//   k-space        the phase rows and S(k) sums of the direct FP32 engines
//                  (passes: mg_kspace.cu, mg_kspace_tc.cu; transforms:
//                  mg_nufft.cu; FP64: mg_kspace64.cu)
//   integrator     k_shake: leap-frog + SHAKE sweeps, one thread per molecule
//
// Mixed precision: positions enter the pair kernel as 32-bit fixed-point
// fractions of the box, so the nearest-image difference is an exact integer
// subtraction; pair arithmetic is FP32; per-site sums are carried in FP32
// within a neighbour-cell batch and folded into compensated FP32 sums; all
// global reductions are FP64 in a fixed order.
#include "mg_internal.h"
#include "mg_device.cuh"

namespace mg {

#define LAUNCHED(L) (++*(L).counter)

static inline int cdiv(long a, long b) { return (int)((a + b - 1) / b); }

// ------------------------------------------------------------- cell list --



// ------------------------------------------------------ the cell list --
//
// cook threads the sites of every cell into a linked list
// (cook/linklist.c:38-269).  Here the cells are runs of one array: the sites
// sorted by cell and within a cell by z, then site index (a fixed order, so
// the order and every sum over it are the same run to run), cell c holding
// order[start[c] .. start[c+1]).  A counting sort in four kernels:
//   cell_count    key of every site, sites per cell (atomic increments)
//   cell_scan     one CTA: start = exclusive scan of the counts, cursor =
//                 start, the counts zeroed again for the next list
//   cell_scatter  every site into a free slot of its cell (atomic cursor)
//   cell_order    a warp per cell ranks its sites by z (then site index)
//                 and writes order[] and the sorted keys (the slots of
//                 cell_scatter depend on the timing of the atomics; the ranks
//                 do not)

// the fixed-point record of every site (site order) and its cell, from the
// fixed-point coordinates (so that the cell and the coordinates the pair
// kernels use agree to the last bit); a non-finite coordinate sets bit 1 of
// *status and the site is binned into cell 0 so that every later index
// stays in range
MG_BODY void cell_count_kernel_body(int ns, const double* __restrict__ r, const double* iL,
                                   int ncx, int ncy, int ncz, const int* __restrict__ kind,
                                   const int* __restrict__ mol, int4* __restrict__ pfix,
                                   int* __restrict__ key, int* __restrict__ count,
                                   int* __restrict__ status, const int bx_) {
  const int i = bx_ * blockDim.x + threadIdx.x;
  if (i >= ns) return;
  const double x = r[3 * i], y = r[3 * i + 1], z = r[3 * i + 2];
  int k = 0;
  const int4 q = make_int4(fixed32(x, iL[0]), fixed32(y, iL[1]), fixed32(z, iL[2]),
                           (mol[i] << 8) | kind[i]);
  if (isfinite(x) && isfinite(y) && isfinite(z)) {
    k = (fixed_cell(q.x, ncx) * ncy + fixed_cell(q.y, ncy)) * ncz + fixed_cell(q.z, ncz);
  } else {
    atomicOr(status, 2);
  }
  pfix[i] = q;
  key[i] = k;
  atomicAdd(count + k, 1);
}

struct Inv3 {
  double v[3];
};

__global__ void cell_count_kernel(int ns, const double* __restrict__ r, const __grid_constant__ Inv3 iL, int ncx,
                                  int ncy, int ncz, const int* __restrict__ kind,
                                  const int* __restrict__ mol, int4* __restrict__ pfix,
                                  int* __restrict__ key, int* __restrict__ count,
                                  int* __restrict__ status) {
  after_previous();
  cell_count_kernel_body(ns, r, iL.v, ncx, ncy, ncz, kind, mol, pfix, key, count, status,
                         blockIdx.x);
}

// exclusive scan of count[0..ncell) into start[0..ncell] and cursor[], in
// tiles of 4 x 1024 counts (int4 loads; count is padded with zeros to a
// multiple of 4 entries); the counts are cleared for the next list.  With
// gstart the same scan of the group counts ceil(count / GROUP_SITES) (the
// work items of the group pair kernel) goes to gstart[0..ncell]; gstart[ncell + 1],
// the half-shell kernel's mark (PairArgs::over), is cleared.
constexpr int SCAN_THREADS = 1024;
__device__ __forceinline__ int2 add2(int2 a, int2 b) { return make_int2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ int2 shfl_up2(int2 v, int o) {
  return make_int2(__shfl_up_sync(0xffffffffu, v.x, o), __shfl_up_sync(0xffffffffu, v.y, o));
}
__device__ __forceinline__ int ngroups(int n) { return (n + GROUP_SITES - 1) / GROUP_SITES; }

MG_BODY void cell_scan_kernel_body(int ncell,
    int* __restrict__ count,
    int* __restrict__ start,
    int* __restrict__ cursor,
    int* __restrict__ gstart,
    const int bx_,
    const int by_) {
  __shared__ int2 wsum[SCAN_THREADS / 32];
  __shared__ int2 carry_s;
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  if (t == 0) carry_s = make_int2(0, 0);
  __syncthreads();
  const int n4 = (ncell + 3) / 4;
  for (int base = 0; base < n4; base += SCAN_THREADS) {
    const int q = base + t;
    int4 v = make_int4(0, 0, 0, 0);
    if (q < n4) {
      v = reinterpret_cast<int4*>(count)[q];
      reinterpret_cast<int4*>(count)[q] = make_int4(0, 0, 0, 0);
    }
    // (sites, groups) of the four cells
    const int2 tot = make_int2(v.x + v.y + v.z + v.w,
                               ngroups(v.x) + ngroups(v.y) + ngroups(v.z) + ngroups(v.w));
    int2 incl = tot;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int2 y = shfl_up2(incl, o);
      if (lane >= o) incl = add2(incl, y);
    }
    if (lane == 31) wsum[w] = incl;
    const int2 carry = carry_s;
    __syncthreads();
    if (w == 0) {
      int2 x = wsum[lane];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int2 y = shfl_up2(x, o);
        if (lane >= o) x = add2(x, y);
      }
      wsum[lane] = x;   // inclusive sums of the warps
    }
    __syncthreads();
    const int2 wprev = w ? wsum[w - 1] : make_int2(0, 0);
    const int ex = carry.x + wprev.x + incl.x - tot.x;
    const int gx = carry.y + wprev.y + incl.y - tot.y;
    if (q < n4) {
      const int e[4] = {ex, ex + v.x, ex + v.x + v.y, ex + v.x + v.y + v.z};
      const int g[4] = {gx, gx + ngroups(v.x), gx + ngroups(v.x) + ngroups(v.y),
                        gx + ngroups(v.x) + ngroups(v.y) + ngroups(v.z)};
#pragma unroll
      for (int k = 0; k < 4; k++)
        if (4 * q + k < ncell) {
          start[4 * q + k] = e[k];
          cursor[4 * q + k] = e[k];
          if (gstart) gstart[4 * q + k] = g[k];
        }
    }
    __syncthreads();
    if (t == SCAN_THREADS - 1) carry_s = add2(carry, wsum[31]);
    __syncthreads();
  }
  if (t == 0) {
    start[ncell] = carry_s.x;
    if (gstart) {
      gstart[ncell] = carry_s.y;
      gstart[ncell + 1] = 0;
    }
  }
}

__global__ void __launch_bounds__(SCAN_THREADS)
cell_scan_kernel(int ncell, int* __restrict__ count, int* __restrict__ start, int* __restrict__ cursor, int* __restrict__ gstart) {
  after_previous();
  cell_scan_kernel_body(ncell, count, start, cursor, gstart, blockIdx.x, 0);
}

__global__ void cell_scatter_kernel(int ns, const int* __restrict__ key, int* __restrict__ cursor,
                                    int* __restrict__ slot_site) {
  after_previous();
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= ns) return;
  slot_site[atomicAdd(cursor + key[i], 1)] = i;
}

constexpr int ORDER_THREADS = 256;
MG_BODY void cell_order_kernel_body(int ncell,
    const int* __restrict__ start,
    const int* __restrict__ slot_site,
    const int4* __restrict__ pfix,
    int* __restrict__ order,
    int* __restrict__ key_s,
    int4* __restrict__ pj,
    const int* __restrict__ gstart,
    int* __restrict__ gcell,
    const int bx_,
    const int by_) {
  const int c = bx_ * (ORDER_THREADS / 32) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (c >= ncell) return;
  const int s0 = start[c], n = start[c + 1] - s0;
  // the cell of each of its groups (work items of the group pair kernel)
  if (gcell)
    for (int g = gstart[c] + lane; g < gstart[c + 1]; g += 32) gcell[g] = c;
  // the sites of a cell in increasing z (ties by site index): runs of
  // consecutive sites are then thin slabs, which the group kernel's
  // bounding boxes prune well
  if (n <= 32) {
    // one site per lane, ranks by shuffles
    const int mine = lane < n ? slot_site[s0 + lane] : 0x7fffffff;
    const unsigned mz = lane < n ? (unsigned)pfix[mine].z : 0xffffffffu;
    int rank = 0;
    for (int j = 0; j < n; j++) {
      const int os = __shfl_sync(0xffffffffu, mine, j);
      const unsigned oz = __shfl_sync(0xffffffffu, mz, j);
      rank += oz < mz || (oz == mz && os < mine);
    }
    if (lane < n) {
      order[s0 + rank] = mine;
      key_s[s0 + rank] = c;
      if (pj) pj[s0 + rank] = pfix[mine];
    }
  } else {
    for (int e = lane; e < n; e += 32) {
      const int mine = slot_site[s0 + e];
      const unsigned mz = (unsigned)pfix[mine].z;
      int rank = 0;
      for (int j = 0; j < n; j++) {
        const int os = slot_site[s0 + j];
        const unsigned oz = (unsigned)pfix[os].z;
        rank += oz < mz || (oz == mz && os < mine);
      }
      order[s0 + rank] = mine;
      key_s[s0 + rank] = c;
      if (pj) pj[s0 + rank] = pfix[mine];
    }
  }
}

__global__ void __launch_bounds__(ORDER_THREADS)
cell_order_kernel(int ncell, const int* __restrict__ start, const int* __restrict__ slot_site, const int4* __restrict__ pfix, int* __restrict__ order, int* __restrict__ key_s, int4* __restrict__ pj, const int* __restrict__ gstart, int* __restrict__ gcell) {
  after_previous();
  cell_order_kernel_body(ncell, start, slot_site, pfix, order, key_s, pj, gstart, gcell, blockIdx.x, 0);
}

// the list of a box held in one cell: the sites in their own order (the pair
// kernel takes all pairs, so no order helps it), one launch
__global__ void cell_one_kernel(int ns, const double* __restrict__ r, const __grid_constant__ Inv3 iL,
                                const int* __restrict__ kind, const int* __restrict__ mol,
                                int* __restrict__ status, int* __restrict__ order,
                                int* __restrict__ key_s, int* __restrict__ start,
                                int* __restrict__ gstart, int4* __restrict__ pj,
                                int* __restrict__ gcell) {
  after_previous();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0) {
    start[0] = gstart[0] = 0;
    start[1] = ns;
    gstart[1] = ngroups(ns);
  }
  if (i >= ns) return;
  const double x = r[3 * i], y = r[3 * i + 1], z = r[3 * i + 2];
  if (!(isfinite(x) && isfinite(y) && isfinite(z))) atomicOr(status, 2);
  order[i] = i;
  key_s[i] = 0;
  if (gcell && i % GROUP_SITES == 0) gcell[i / GROUP_SITES] = 0;
  if (pj)
    pj[i] = make_int4(fixed32(x, iL.v[0]), fixed32(y, iL.v[1]), fixed32(z, iL.v[2]),
                      (mol[i] << 8) | kind[i]);
}

cudaError_t k_cell_list(const Launch& L, int ns, const double* r, int* status, const double iL[3],
                        int ncx, int ncy, int ncz, const int* kind, const int* mol, int4* pfix,
                        int* key, int* count, int* cursor, int* slot_site, int* order,
                        int* key_s, int* start, int* gstart, int4* pj, int* gcell) {
  const int ncell = ncx * ncy * ncz;
  const Inv3 il{{iL[0], iL[1], iL[2]}};
  if (ncell == 1) {
    cell_one_kernel<<<cdiv(ns, 128), 128, 0, L.s>>>(ns, r, il, kind, mol, status, order, key_s,
                                                    start, gstart, pj, gcell);
    LAUNCHED(L);
    return cudaGetLastError();
  }
  cell_count_kernel<<<cdiv(ns, 256), 256, 0, L.s>>>(ns, r, il, ncx, ncy, ncz, kind, mol, pfix, key,
                                                    count, status);
  LAUNCHED(L);
  launch_after(L, cell_scan_kernel, 1, SCAN_THREADS, 0, ncell, count, start, cursor, gstart);
  LAUNCHED(L);
  launch_after(L, cell_scatter_kernel, cdiv(ns, 256), 256, 0, ns, key, cursor, slot_site);
  LAUNCHED(L);
  launch_after(L, cell_order_kernel, cdiv(ncell, ORDER_THREADS / 32), ORDER_THREADS, 0, ncell,
               start, slot_site, pfix, order, key_s, pj, gstart, gcell);
  LAUNCHED(L);
  return cudaGetLastError();
}

__global__ void gather_mixed_kernel(int ns, const double* __restrict__ r,
                                    const int* __restrict__ order, const int* __restrict__ kind,
                                    const int* __restrict__ mol, double iLx, double iLy,
                                    double iLz, int4* __restrict__ pj) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= ns) return;
  int i = order[t];
  pj[t] = make_int4(fixed32(r[3 * i], iLx), fixed32(r[3 * i + 1], iLy),
                    fixed32(r[3 * i + 2], iLz), (mol[i] << 8) | kind[i]);
}

cudaError_t k_gather_mixed(const Launch& L, int ns, const double* r, const int* order,
                           const int* kind, const int* mol, const double iL[3], int4* pj) {
  gather_mixed_kernel<<<cdiv(ns, 256), 256, 0, L.s>>>(ns, r, order, kind, mol, iL[0], iL[1],
                                                      iL[2], pj);
  LAUNCHED(L);
  return cudaGetLastError();
}

__global__ void gather_fp64_kernel(int ns, const double* __restrict__ r,
                                   const int* __restrict__ order, const int* __restrict__ kind,
                                   const int* __restrict__ mol, double Lx, double Ly, double Lz,
                                   double4* __restrict__ pd, float4* __restrict__ pf) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= ns) return;
  int i = order[t];
  double x = r[3 * i], y = r[3 * i + 1], z = r[3 * i + 2];
  x -= Lx * floor(x / Lx);
  y -= Ly * floor(y / Ly);
  z -= Lz * floor(z / Lz);
  const int w = (mol[i] << 8) | kind[i];
  pd[t] = make_double4(x, y, z, __longlong_as_double((long long)w));
  if (pf) pf[t] = make_float4((float)x, (float)y, (float)z, __int_as_float(w));
}

cudaError_t k_gather_fp64(const Launch& L, int ns, const double* r, const int* order,
                          const int* kind, const int* mol, double Lx, double Ly, double Lz,
                          double4* pd, float4* pf) {
  gather_fp64_kernel<<<cdiv(ns, 256), 256, 0, L.s>>>(ns, r, order, kind, mol, Lx, Ly, Lz, pd, pf);
  LAUNCHED(L);
  return cudaGetLastError();
}

// ---------------------------------------------------------- pair kernels --

constexpr int NWARP = PAIR_THREADS / 32;
constexpr int FOLD = 8;   // stencil cells per FP32 force batch before the FP64 fold

// One CTA per home cell; its 4 warps split the neighbour-cell stencil, each
// staging 32 neighbour sites at a time in shared memory; lane = home site.
// Full shell: forces only on the home site.  POLAR adds the Drude terms of
// cook/ljqqpol.c (centre-Drude, Drude-centre, Drude-Drude, each at its own
// separation); Drude forces go to the second half of f.
//
// Every grid has at least 2 cdiv + 1 cells per edge (boxes of one cell run
// pair_all_kernel): a staged site is converted once, as the float offset of
// its nearest image from the centre of the home cell (exact 32-bit
// fixed-point difference, then one rounding); a pair then costs three
// subtractions and no int-to-float conversion (conversions are slow on this
// GPU).  Every stencil cell lies within half a box of the home-cell centre,
// so the image taken is the nearest one for every pair inside the cutoff.
// NW warps per CTA (the autotuner picks 4, 8 or 16: more warps per home
// cell finish a cell sooner, which shortens the tail of the grid); STAB: the
// force spline in
// shared memory (dynamic, ntab float4) instead of read through L1.
// Intramolecular pairs are skipped: their Ewald exclusion terms come from
// excl_mixed_kernel, once per pair.  Forces are summed in FP32 per batch of
// FOLD stencil cells and folded into an FP32 sum with a compensation term
// (Knuth's TwoSum): no FP64 instruction in the loop (the FP64 pipe of this
// GPU is narrow and also serves the float/double conversions).
template <bool MEASURE, bool POLAR, int NW, bool STAB>
MG_BODY void pair_mixed_kernel_body(const PairArgs& a,
    const int4* __restrict__ pj,
    const PairF* __restrict__ ptab_g,
    const float4* __restrict__ erd_g,
    const float4* __restrict__ eru,
    float sx,
    float sy,
    float sz,
    float cq,
    float sgrid,
    float alpha,
    const int bx_,
    const int by_) {
  constexpr int NT = NW * 32;
  // dynamic shared memory: the nk x nk FP32 pair table, then (STAB) the
  // force spline
  extern __shared__ float4 dyn_smem[];
  __shared__ int4 sj[NW][32];
  __shared__ float4 sjd[POLAR ? NW : 1][32];
  __shared__ double red[NW][32][POLAR ? 6 : 3];
  __shared__ double ered[NT];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nk = a.nkind, ntab = a.ntab;
  PairFS* ptab = reinterpret_cast<PairFS*>(dyn_smem);
  float4* s_erd = dyn_smem + 3 * nk * nk;
  for (int t = threadIdx.x; t < 3 * nk * nk; t += NT)
    dyn_smem[t] = reinterpret_cast<const float4*>(ptab_g + t / 3)[t % 3];
  if (STAB)
    for (int t = threadIdx.x; t < ntab; t += NT) s_erd[t] = erd_g[t];
  const float4* erd = STAB ? s_erd : erd_g;
  __syncthreads();

  const int c = bx_;
  const int cz = c % a.ncz, cy = (c / a.ncz) % a.ncy, cx = c / (a.ncy * a.ncz);
  const int i0 = a.cell_start[c], ni = a.cell_start[c + 1] - i0;
  // fixed-point centre of the home cell
  const unsigned refx = (unsigned)((((unsigned long long)(2 * cx + 1)) << 31) / a.ncx),
                 refy = (unsigned)((((unsigned long long)(2 * cy + 1)) << 31) / a.ncy),
                 refz = (unsigned)((((unsigned long long)(2 * cz + 1)) << 31) / a.ncz);
  // per-lane energy sums: FP32 per neighbour cell, folded into compensated
  // FP32 sums (the FP64 pipe of this GPU is narrow); FP64 from the CTA sum on
  CSum es[9];

  for (int ib = 0; ib < ni; ib += 32) {
    const bool vi = ib + lane < ni;
    const int ti = i0 + ib + lane;
    const int4 me = vi ? pj[ti] : make_int4(0, 0, 0, 0);
    const float4 md = (POLAR && vi) ? a.pdj[ti] : make_float4(0.f, 0.f, 0.f, 0.f);
    const int kind_i = me.w & 255, mol_i = me.w >> 8;
    const float xi = (float)(int)((unsigned)me.x - refx) * sx,
                yi = (float)(int)((unsigned)me.y - refy) * sy,
                zi = (float)(int)((unsigned)me.z - refz) * sz;
    CSum fx, fy, fz, gx, gy, gz;
    float ax = 0, ay = 0, az = 0, bx = 0, by = 0, bz = 0;
    float e_el = 0, e_lj = 0, e_vir = 0;
    PvF pv;
    pv.zero();
    int nb = 0;
    for (int s = warp; s < a.nstencil; s += NW) {
      const int4 o = a.stencil[s];
      int x2 = cx + o.x, y2 = cy + o.y, z2 = cz + o.z;
      x2 += (x2 < 0) ? a.ncx : (x2 >= a.ncx ? -a.ncx : 0);
      y2 += (y2 < 0) ? a.ncy : (y2 >= a.ncy ? -a.ncy : 0);
      z2 += (z2 < 0) ? a.ncz : (z2 >= a.ncz ? -a.ncz : 0);
      const int c2 = (x2 * a.ncy + y2) * a.ncz + z2;
      const int j0 = a.cell_start[c2], nj = a.cell_start[c2 + 1] - j0;
      for (int jb = 0; jb < nj; jb += 32) {
        if (jb + lane < nj) {
          int4 q = pj[j0 + jb + lane];
          // offset of the neighbour's nearest image from the home-cell centre
          const float4 f = make_float4((float)(int)((unsigned)q.x - refx) * sx,
                                       (float)(int)((unsigned)q.y - refy) * sy,
                                       (float)(int)((unsigned)q.z - refz) * sz,
                                       __int_as_float(q.w));
          q = make_int4(__float_as_int(f.x), __float_as_int(f.y), __float_as_int(f.z), q.w);
          sj[warp][lane] = q;
          if (POLAR) sjd[warp][lane] = a.pdj[j0 + jb + lane];
        }
        __syncwarp();
        const int cnt = min(32, nj - jb);
        for (int jj = 0; jj < cnt; jj++) {
          const int4 q = sj[warp][jj];
          const float dx = xi - __int_as_float(q.x), dy = yi - __int_as_float(q.y),
                      dz = zi - __int_as_float(q.z);
          const float rr = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
          // the site itself and its own molecule (exclusions) are skipped
          if (!vi || rr >= cq || (q.w >> 8) == mol_i) continue;
          const PairFS P = ptab[kind_i * nk + (q.w & 255)];
          float4 qd = make_float4(0.f, 0.f, 0.f, 0.f);
          if (POLAR) qd = sjd[warp][jj];
          float f = 0;
          if (rr < P.C2q) {
            float U;
            if (rr < P.C1q) {
              const float x = __fdividef(P.Sq, rr), y = x * x * x;
              f = P.E24 * (fmaf(2.f, y, -P.lam) * y) * x;
              U = P.E4 * ((y - P.lam) * y);
            } else {
              const float x = rr - P.C2q;
              f = P.A4 * x;
              U = P.A * x * x;
            }
            if (MEASURE) {
              e_lj += U;
              e_vir += rr * f;
            }
          }
          if (P.qq != 0.f) f += spline_any<MEASURE, !STAB>(erd, eru, rr, sgrid, ntab, P.qq, e_el);
          ax = fmaf(f, dx, ax);
          ay = fmaf(f, dy, ay);
          az = fmaf(f, dz, az);
          if (MEASURE) pv.add(dx, dy, dz, f);
          if (POLAR) {
            if (P.qpc != 0.f) {  // Drude(i) - centre(j)
              const float ex = dx + md.x, ey = dy + md.y, ez = dz + md.z;
              const float fp = spline_any<MEASURE, !STAB>(erd, eru, fmaf(ex, ex, fmaf(ey, ey, ez * ez)),
                                                    sgrid, ntab, P.qpc, e_el);
              bx = fmaf(fp, ex, bx);
              by = fmaf(fp, ey, by);
              bz = fmaf(fp, ez, bz);
              if (MEASURE) pv.add(ex, ey, ez, fp);
            }
            if (P.qcp != 0.f) {  // centre(i) - Drude(j)
              const float ex = dx - qd.x, ey = dy - qd.y, ez = dz - qd.z;
              const float fp = spline_any<MEASURE, !STAB>(erd, eru, fmaf(ex, ex, fmaf(ey, ey, ez * ez)),
                                                    sgrid, ntab, P.qcp, e_el);
              ax = fmaf(fp, ex, ax);
              ay = fmaf(fp, ey, ay);
              az = fmaf(fp, ez, az);
              if (MEASURE) pv.add(ex, ey, ez, fp);
            }
            if (P.qpp != 0.f) {  // Drude(i) - Drude(j)
              const float ex = dx + md.x - qd.x, ey = dy + md.y - qd.y, ez = dz + md.z - qd.z;
              const float fp = spline_any<MEASURE, !STAB>(erd, eru, fmaf(ex, ex, fmaf(ey, ey, ez * ez)),
                                                    sgrid, ntab, P.qpp, e_el);
              bx = fmaf(fp, ex, bx);
              by = fmaf(fp, ey, by);
              bz = fmaf(fp, ez, bz);
              if (MEASURE) pv.add(ex, ey, ez, fp);
            }
          }
        }
        __syncwarp();
      }
      // energies fold into the compensated sums after every neighbour cell,
      // forces every FOLD cells
      if (MEASURE) {
        es[0].add(e_el); es[1].add(e_lj); es[2].add(e_vir);
        es[3].add(pv.p0); es[4].add(pv.p1); es[5].add(pv.p2);
        es[6].add(pv.p3); es[7].add(pv.p4); es[8].add(pv.p5);
        e_el = e_lj = e_vir = 0;
        pv.zero();
      }
      if (++nb == FOLD) {
        nb = 0;
        fx.add(ax); fy.add(ay); fz.add(az);
        ax = ay = az = 0;
        if (POLAR) {
          gx.add(bx); gy.add(by); gz.add(bz);
          bx = by = bz = 0;
        }
      }
    }
    fx.add(ax); fy.add(ay); fz.add(az);
    red[warp][lane][0] = fx.value();
    red[warp][lane][1] = fy.value();
    red[warp][lane][2] = fz.value();
    if (POLAR) {
      gx.add(bx); gy.add(by); gz.add(bz);
      red[warp][lane][POLAR ? 3 : 0] = gx.value();
      red[warp][lane][POLAR ? 4 : 0] = gy.value();
      red[warp][lane][POLAR ? 5 : 0] = gz.value();
    }
    __syncthreads();
    if (warp == 0 && vi) {
      double g[6] = {0, 0, 0, 0, 0, 0};
#pragma unroll
      for (int w = 0; w < NW; w++)
#pragma unroll
        for (int k = 0; k < (POLAR ? 6 : 3); k++) g[k] += red[w][lane][k];
      const int site = a.order[ti];
      a.f[3 * site] = g[0];
      a.f[3 * site + 1] = g[1];
      a.f[3 * site + 2] = g[2];
      if (POLAR) {
        a.f[3 * (long)a.ns + 3 * site] = g[3];
        a.f[3 * (long)a.ns + 3 * site + 1] = g[4];
        a.f[3 * (long)a.ns + 3 * site + 2] = g[5];
      }
    }
    __syncthreads();
  }
  if (MEASURE) {
    // each unordered pair was visited from both ends
    for (int k = 0; k < 9; k++) {
      ered[threadIdx.x] = 0.5 * es[k].value();
      __syncthreads();
      for (int w = NT / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w) ered[threadIdx.x] += ered[threadIdx.x + w];
        __syncthreads();
      }
      if (threadIdx.x == 0) a.epart[bx_ * NEN + k] = ered[0];
      __syncthreads();
    }
  }
}

template <bool MEASURE, bool POLAR, int NW, bool STAB>
__global__ void __launch_bounds__(NW * 32)
    pair_mixed_kernel(const __grid_constant__ PairArgs a, const int4* __restrict__ pj, const PairF* __restrict__ ptab_g, const float4* __restrict__ erd_g, const float4* __restrict__ eru, float sx, float sy, float sz, float cq, float sgrid, float alpha) {
  pair_mixed_kernel_body<MEASURE, POLAR, NW, STAB>(a, pj, ptab_g, erd_g, eru, sx, sy, sz, cq, sgrid, alpha, blockIdx.x, 0);
}

// ------------------------------------------------- group pair kernel --
//
// The same pair terms as pair_mixed_kernel with the work cut by pruning.
// One warp per group of up to GROUP_SITES = 8 sites of a home cell (the
// group's sites are consecutive in the cell's site order); lane = (i = lane
// & 7, s = lane >> 3).  The neighbour sites come from the stencil's z-runs
// (cells consecutive along z are consecutive in the sorted array, so a run
// is one or, across the periodic edge, two contiguous ranges) in batches of
// 32: every neighbour is tested once against the cutoff sphere around the
// group's bounding box, the kept ones are compacted into shared memory
// (warp ballot, fixed order) and taken four at a time, one per s, each
// against the lane's own site i.  The test keeps every pair within the
// cutoff (the box distance is a lower bound of every pair distance, with the
// same FP32 operations), so the pair set is the cell kernel's.  The pair
// terms are predicated rather than branched (the lanes of a warp hold
// different kinds of pairs, and a branch per kind would run every path one
// after the other).  Forces: FP32 per z-run, folded into compensated sums;
// at the end the four s-lanes of a site are summed in a fixed order.  No
// atomics: results are reproducible.
template <bool MEASURE, bool POLAR, int NW>
__global__ void __launch_bounds__(NW * 32)
    pair_group_mixed_kernel(PairArgs a, const int4* __restrict__ pj,
                            const PairF* __restrict__ ptab_g, const float4* __restrict__ erd,
                            const float4* __restrict__ eru, float sx, float sy, float sz, float cq,
                            float sgrid) {
  constexpr int NT = NW * 32;
  extern __shared__ float4 dyn_smem[];   // the nk x nk FP32 pair table
  __shared__ float4 sj[NW][32];
  __shared__ float4 sjd[POLAR ? NW : 1][32];
  __shared__ double ered[NT];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int il = lane & 7, sl = lane >> 3;
  const int nk = a.nkind, ntab = a.ntab;
  PairFS* ptab = reinterpret_cast<PairFS*>(dyn_smem);
  for (int t = threadIdx.x; t < 3 * nk * nk; t += NT)
    dyn_smem[t] = reinterpret_cast<const float4*>(ptab_g + t / 3)[t % 3];
  __syncthreads();
  const int ncell = a.ncx * a.ncy * a.ncz;
  const int nitems = a.gstart[ncell];
  CSum es[9];

  for (int item = blockIdx.x * NW + warp; item < nitems; item += gridDim.x * NW) {
    const int c = a.gcell[item];
    const int cz = c % a.ncz, cy = (c / a.ncz) % a.ncy, cx = c / (a.ncy * a.ncz);
    const int i0 = a.cell_start[c] + GROUP_SITES * (item - a.gstart[c]);
    const int ni = min(GROUP_SITES, a.cell_start[c + 1] - i0);
    const unsigned refx = (unsigned)((((unsigned long long)(2 * cx + 1)) << 31) / a.ncx),
                   refy = (unsigned)((((unsigned long long)(2 * cy + 1)) << 31) / a.ncy),
                   refz = (unsigned)((((unsigned long long)(2 * cz + 1)) << 31) / a.ncz);
    const bool vi = il < ni;
    const int ti = i0 + il;
    const int4 me = vi ? pj[ti] : make_int4(0, 0, 0, 0);
    const float4 md = (POLAR && vi) ? a.pdj[ti] : make_float4(0.f, 0.f, 0.f, 0.f);
    const int kind_i = me.w & 255, mol_i = me.w >> 8;
    const float xi = (float)(int)((unsigned)me.x - refx) * sx,
                yi = (float)(int)((unsigned)me.y - refy) * sy,
                zi = (float)(int)((unsigned)me.z - refz) * sz;
    // bounding box of the group's sites (the same in all four s-copies)
    float blx = vi ? xi : 3e38f, bly = vi ? yi : 3e38f, blz = vi ? zi : 3e38f;
    float bhx = vi ? xi : -3e38f, bhy = vi ? yi : -3e38f, bhz = vi ? zi : -3e38f;
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) {
      blx = fminf(blx, __shfl_xor_sync(0xffffffffu, blx, o));
      bly = fminf(bly, __shfl_xor_sync(0xffffffffu, bly, o));
      blz = fminf(blz, __shfl_xor_sync(0xffffffffu, blz, o));
      bhx = fmaxf(bhx, __shfl_xor_sync(0xffffffffu, bhx, o));
      bhy = fmaxf(bhy, __shfl_xor_sync(0xffffffffu, bhy, o));
      bhz = fmaxf(bhz, __shfl_xor_sync(0xffffffffu, bhz, o));
    }
    CSum fx, fy, fz, gx, gy, gz;
    for (int sp = 0; sp < a.nspans; sp++) {
      const int4 o = a.spans[sp];
      int x2 = cx + o.x, y2 = cy + o.y;
      x2 += (x2 < 0) ? a.ncx : (x2 >= a.ncx ? -a.ncx : 0);
      y2 += (y2 < 0) ? a.ncy : (y2 >= a.ncy ? -a.ncy : 0);
      const int col = (x2 * a.ncy + y2) * a.ncz;
      int za = cz + o.z, zb = cz + o.w;
      if (zb < 0) { za += a.ncz; zb += a.ncz; }
      if (za >= a.ncz) { za -= a.ncz; zb -= a.ncz; }
      // the z-run (at most ncz cells) as one or two contiguous ranges
      int ra0, ra1, rb0 = 0, rb1 = -1;
      if (za < 0) { ra0 = za + a.ncz; ra1 = a.ncz - 1; rb0 = 0; rb1 = zb; }
      else if (zb >= a.ncz) { ra0 = za; ra1 = a.ncz - 1; rb0 = 0; rb1 = zb - a.ncz; }
      else { ra0 = za; ra1 = zb; }
      float ax = 0, ay = 0, az = 0, bx = 0, by = 0, bz = 0;
      float e_el = 0, e_lj = 0, e_vir = 0;
      PvF pv;
      pv.zero();
      for (int part = 0; part < 2; part++) {
        const int z0 = part ? rb0 : ra0, z1 = part ? rb1 : ra1;
        if (z1 < z0) continue;
        const int j0 = a.cell_start[col + z0], j1 = a.cell_start[col + z1 + 1];
        for (int jb = j0; jb < j1; jb += 32) {
          const int j = jb + lane;
          bool keep = false;
          float4 f4 = make_float4(0.f, 0.f, 0.f, 0.f);
          if (j < j1) {
            const int4 q = pj[j];
            f4 = make_float4((float)(int)((unsigned)q.x - refx) * sx,
                             (float)(int)((unsigned)q.y - refy) * sy,
                             (float)(int)((unsigned)q.z - refz) * sz, __int_as_float(q.w));
            const float ddx = fmaxf(fmaxf(blx - f4.x, f4.x - bhx), 0.f),
                        ddy = fmaxf(fmaxf(bly - f4.y, f4.y - bhy), 0.f),
                        ddz = fmaxf(fmaxf(blz - f4.z, f4.z - bhz), 0.f);
            keep = fmaf(ddx, ddx, fmaf(ddy, ddy, ddz * ddz)) < cq;
          }
          const unsigned M = __ballot_sync(0xffffffffu, keep);
          if (keep) {
            const int slot = __popc(M & ((1u << lane) - 1u));
            sj[warp][slot] = f4;
            if (POLAR) sjd[warp][slot] = a.pdj[j];
          }
          __syncwarp();
          const int n = __popc(M);
          for (int t = sl; t < n; t += 4) {
            const float4 q = sj[warp][t];
            const float dx = xi - q.x, dy = yi - q.y, dz = zi - q.z;
            const float rr = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
            const int qw = __float_as_int(q.w);
            const bool ok = vi && rr < cq && (qw >> 8) != mol_i;
            const PairFS P = ptab[kind_i * nk + (qw & 255)];
            const float x = __fdividef(P.Sq, rr), y = x * x * x, xt = rr - P.C2q;
            const bool core = rr < P.C1q, tail = rr < P.C2q;
            const float flj = core ? P.E24 * (fmaf(2.f, y, -P.lam) * y) * x : (tail ? P.A4 * xt : 0.f);
            float e_el_p = 0.f;
            float f = flj + spline_any<MEASURE, true>(erd, eru, rr, sgrid, ntab, P.qq, e_el_p);
            f = ok ? f : 0.f;
            ax = fmaf(f, dx, ax);
            ay = fmaf(f, dy, ay);
            az = fmaf(f, dz, az);
            if (MEASURE && ok) {
              e_lj += core ? P.E4 * ((y - P.lam) * y) : (tail ? P.A * xt * xt : 0.f);
              e_vir += rr * flj;
              e_el += e_el_p;
              pv.add(dx, dy, dz, f);
            }
            if (POLAR) {
              // Drude(i) - centre(j), centre(i) - Drude(j), Drude(i) -
              // Drude(j): zero charge products give zero terms
              const float4 qd = sjd[warp][t];
              float e_p = 0.f;
              const float ex = dx + md.x, ey = dy + md.y, ez = dz + md.z;
              float fp = spline_any<MEASURE, true>(
                  erd, eru, fmaf(ex, ex, fmaf(ey, ey, ez * ez)), sgrid, ntab, P.qpc, e_p);
              fp = ok ? fp : 0.f;
              bx = fmaf(fp, ex, bx);
              by = fmaf(fp, ey, by);
              bz = fmaf(fp, ez, bz);
              const float cx2 = dx - qd.x, cy2 = dy - qd.y, cz2 = dz - qd.z;
              float fc = spline_any<MEASURE, true>(
                  erd, eru, fmaf(cx2, cx2, fmaf(cy2, cy2, cz2 * cz2)), sgrid, ntab, P.qcp, e_p);
              fc = ok ? fc : 0.f;
              ax = fmaf(fc, cx2, ax);
              ay = fmaf(fc, cy2, ay);
              az = fmaf(fc, cz2, az);
              const float px = ex - qd.x, py = ey - qd.y, pz = ez - qd.z;
              float fd = spline_any<MEASURE, true>(
                  erd, eru, fmaf(px, px, fmaf(py, py, pz * pz)), sgrid, ntab, P.qpp, e_p);
              fd = ok ? fd : 0.f;
              bx = fmaf(fd, px, bx);
              by = fmaf(fd, py, by);
              bz = fmaf(fd, pz, bz);
              if (MEASURE && ok) {
                pv.add(ex, ey, ez, fp);
                pv.add(cx2, cy2, cz2, fc);
                pv.add(px, py, pz, fd);
                e_el += e_p;
              }
            }
          }
          __syncwarp();
        }
      }
      // the z-run's FP32 sums into the compensated sums
      fx.add(ax); fy.add(ay); fz.add(az);
      if (POLAR) { gx.add(bx); gy.add(by); gz.add(bz); }
      if (MEASURE) {
        es[0].add(e_el); es[1].add(e_lj); es[2].add(e_vir);
        es[3].add(pv.p0); es[4].add(pv.p1); es[5].add(pv.p2);
        es[6].add(pv.p3); es[7].add(pv.p4); es[8].add(pv.p5);
      }
    }
    // the four s-lanes of a site, summed in a fixed order (xor 8, then 16:
    // every lane holds (s0 + s1) + (s2 + s3))
    double g[6] = {fx.value(), fy.value(), fz.value(), 0, 0, 0};
    if (POLAR) {
      g[3] = gx.value();
      g[4] = gy.value();
      g[5] = gz.value();
    }
#pragma unroll
    for (int k = 0; k < (POLAR ? 6 : 3); k++) {
      g[k] += __shfl_xor_sync(0xffffffffu, g[k], 8);
      g[k] += __shfl_xor_sync(0xffffffffu, g[k], 16);
    }
    if (sl == 0 && vi) {
      const int site = a.order[ti];
      a.f[3 * site] = g[0];
      a.f[3 * site + 1] = g[1];
      a.f[3 * site + 2] = g[2];
      if (POLAR) {
        a.f[3 * (long)a.ns + 3 * site] = g[3];
        a.f[3 * (long)a.ns + 3 * site + 1] = g[4];
        a.f[3 * (long)a.ns + 3 * site + 2] = g[5];
      }
    }
  }
  if (MEASURE) {
    // each unordered pair was visited from both ends; one row per CTA
    for (int k = 0; k < 9; k++) {
      ered[threadIdx.x] = 0.5 * es[k].value();
      __syncthreads();
      for (int w = NT / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w) ered[threadIdx.x] += ered[threadIdx.x + w];
        __syncthreads();
      }
      if (threadIdx.x == 0) a.epart[blockIdx.x * NEN + k] = ered[0];
      __syncthreads();
    }
  }
}

// ---------------------------------------- fixed-point force sums --
//
// The half-shell kernel below adds forces as 64-bit fixed-point numbers
// (FIX_SCALE units per K/A, sorted order) by integer atomics: integer addition
// does not depend on the order, so the forces come out the same bit for bit
// on every run.  finish_forces_kernel turns the sums into the FP64 forces
// (site order) and clears them for the next evaluation.
//
// A sum holds 2^31 K/A, less than two oxygens 1 A apart repel each other by, and
// a conversion makes a number of a NaN.  Every term is therefore compared with
// PairArgs::flim before its conversion (written so that a NaN fails); where one
// fails, its site is marked and finish_forces_kernel forms that site's force pair
// by pair instead (direct_forces).
constexpr double FIX_SCALE = 4294967296.0;  // 2^32: steps of 2.3e-10 K/A, |F| < 2^31 K/A


__device__ __forceinline__ float rcp_approx(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// The erfc splines t0 + t1 / (t2 + r^2) of the FP32 pair kernels.  t1 and t2 are
// rounded; the constant makes up for what that, the sum and the approximate
// reciprocal leave on the average over the interval (32 points).  Rounded alone, the
// three gave every pair of an interval the same error: 1.3 K of the virial of 864
// waters, whose charge terms add up to 2e-5 of their size.
__global__ void round_spline_kernel(int n, const double* __restrict__ ert, double step,
                                    float4* __restrict__ erd, float4* __restrict__ eru) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= 2 * n) return;
  const int iv = i >> 1;
  const double* t = ert + 6 * (long)iv + 3 * (i & 1);
  const float B = (float)t[1], C = (float)t[2];
  double off = 0;
  for (int k = 0; k < 32; k++) {
    const float x = (float)((iv + (k + 0.5) / 32) * step);
    off += t[1] / (t[2] + x) - (double)B * rcp_approx(__fadd_rn(C, x));
  }
  (i & 1 ? erd : eru)[iv] = make_float4((float)(t[0] + off / 32), B, C, 0.f);
}

cudaError_t k_round_spline(const Launch& L, int n, const double* ert, double sgrid, float4* erd,
                           float4* eru) {
  round_spline_kernel<<<cdiv(2 * n, 128), 128, 0, L.s>>>(n, ert, 1 / sgrid, erd, eru);
  LAUNCHED(L);
  return cudaGetLastError();
}

// a compile-time truth value (which terms a quad of home sites takes)
template <bool B>
struct BoolC {
  static constexpr bool value = B;
};

// a store that the compiler need not take for a change of the kernel's other
// integers (a batch's arguments, in memory, would be read again after it)
__device__ __forceinline__ void mark(int* flag) {
  asm volatile("st.global.u32 [%0], 1;" ::"l"(flag));
}

// the half-shell kernel's pair force factor f (force on i = f (r_i - r_j))
// with every rounding explicit; flj: the LJ part, y: (Sq / r^2)^3 for its
// energy.  The same terms as
// spline_any and the group kernel: smoothed LJ (core below C1q, quadratic
// tail up to C2q) and the hyperbolic erfc spline d.x + d.y / (d.z + r^2)
__device__ __forceinline__ float pair_force_rn(const PairFS& P, float rr,
                                               const float4* __restrict__ erd, float sgrid,
                                               int ntab, float& flj, float& y) {
  const float x = __fmul_rn(P.Sq, rcp_approx(rr));
  y = __fmul_rn(__fmul_rn(x, x), x);
  flj = rr < P.C1q ? __fmul_rn(__fmul_rn(P.E24, __fmul_rn(__fmaf_rn(2.f, y, -P.lam), y)), x)
                   : (rr < P.C2q ? __fmul_rn(P.A4, __fadd_rn(rr, -P.C2q)) : 0.f);
  const int ix = min(__float_as_int(__fmaf_rz(rr, sgrid, 12582912.f)) - 0x4B400000, ntab - 1);
  const float4 d = __ldg(erd + ix);
  return __fmaf_rn(__fmaf_rn(d.y, rcp_approx(__fadd_rn(d.z, rr)), d.x), P.qq, flj);
}

// the Drude terms of a pair in the half-shell kernel, every rounding
// explicit: (charge product) x (d.x + d.y / (d.z + r^2)) at the separation
// (ex, ey, ez); e: its energy when measuring
template <bool MEASURE>
__device__ __forceinline__ float drude_force_rn(const float4* __restrict__ erd,
                                                const float4* __restrict__ eru, float ex,
                                                float ey, float ez, float sgrid, int ntab,
                                                float q, float& e) {
  const float r2 = __fmaf_rn(ex, ex, __fmaf_rn(ey, ey, __fmul_rn(ez, ez)));
  const int ix = min(__float_as_int(__fmaf_rz(r2, sgrid, 12582912.f)) - 0x4B400000, ntab - 1);
  const float4 d = __ldg(erd + ix);
  if (MEASURE) {
    const float4 u = __ldg(eru + ix);
    e += fmaf(u.y, rcp_approx(u.z + r2), u.x) * q;
  }
  return __fmul_rn(__fmaf_rn(d.y, rcp_approx(__fadd_rn(d.z, r2)), d.x), q);
}

// ------------------------------------------------- all-pairs kernel --
//
// Small boxes (one cell holds every site, or the cutoff sphere covers a good
// part of the box): a CTA per 8 consecutive sorted sites, its 16 warps taking
// batches of 32 of all sites in turn, staged in shared memory; lane = (site,
// one of four neighbours at a time).  Every pair is evaluated from both ends, its nearest image from the
// exact fixed-point difference.  With the cells of such a box a few dozen
// warps wait for short runs of sites one after the other; here every SM has
// work and the only waste is the pairs beyond the cutoff, whose terms are
// skipped when no lane needs them.  Measured at 1500 sites: 11 us, the cell
// kernel 85 and the half-shell kernel 17; at 648 sites held in one cell, where
// one warp of the cell kernel did all the work, a measured evaluation went
// from 3.2 ms to about 20 us.  Where a cell holds more than three or four sites
// the half-shell kernel is the faster one.  Forces: FP32 per batch, folded into
// compensated sums, the warps' sums added in order in FP64; every rounding of
// the force arithmetic is explicit (measured and plain forces are the same).
constexpr int ALL_WARPS = 16, ALL_SITES = 8;

template <bool MEASURE, bool POLAR>
MG_BODY void pair_all_kernel_body(const PairArgs& a, const int4* __restrict__ pj,
                                  const PairF* __restrict__ ptab_g,
                                  const float4* __restrict__ erd, const float4* __restrict__ eru,
                                  float sx, float sy, float sz, float cq, float sgrid,
                                  const int bx_) {
  constexpr int NW = ALL_WARPS, NT = NW * 32, NC = POLAR ? 6 : 3;
  extern __shared__ float4 dyn_smem[];   // the nk x nk FP32 pair table
  __shared__ int4 sj[NW][32];
  __shared__ float4 sjd[POLAR ? NW : 1][32];
  __shared__ double red[NW][NC][ALL_SITES];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nk = a.nkind, ntab = a.ntab;
  PairFS* ptab = reinterpret_cast<PairFS*>(dyn_smem);
  for (int t = threadIdx.x; t < 3 * nk * nk; t += NT)
    dyn_smem[t] = reinterpret_cast<const float4*>(ptab_g + t / 3)[t % 3];
  const int ti = bx_ * ALL_SITES + (lane & 7), sl = lane >> 3;
  const bool vi = ti < a.ns;
  const int4 me = vi ? pj[ti] : make_int4(0, 0, 0, 0);
  const float4 md = (POLAR && vi) ? a.pdj[ti] : make_float4(0.f, 0.f, 0.f, 0.f);
  const PairFS* prow = ptab + (me.w & 255) * nk;
  const float lim = vi ? cq : 0.f;
  CSum fx, fy, fz, gx, gy, gz;
  CSum es[9];
  __syncthreads();
  for (int jb = warp * 32; jb < a.ns; jb += NT) {
    const int j = jb + lane;
    __syncwarp();
    // slots past the last site hold a site of kind 0 (their pairs are masked,
    // but their kind still indexes the pair table)
    sj[warp][lane] = j < a.ns ? pj[j] : make_int4(0, 0, 0, 0);
    if (POLAR) sjd[warp][lane] = j < a.ns ? a.pdj[j] : make_float4(0.f, 0.f, 0.f, 0.f);
    __syncwarp();
    const int cnt = min(32, a.ns - jb);
    float ax = 0, ay = 0, az = 0, bx = 0, by = 0, bz = 0;
    float e_el = 0, e_lj = 0, e_vir = 0;
    PvF pv;
    pv.zero();
#pragma unroll 4
    for (int j0 = 0; j0 < cnt; j0 += 4) {
      const int jj = j0 + sl;
      const int4 q = sj[warp][jj];
      const float dx = __fmul_rn((float)(int)((unsigned)me.x - (unsigned)q.x), sx),
                  dy = __fmul_rn((float)(int)((unsigned)me.y - (unsigned)q.y), sy),
                  dz = __fmul_rn((float)(int)((unsigned)me.z - (unsigned)q.z), sz);
      const float rr = __fmaf_rn(dx, dx, __fmaf_rn(dy, dy, __fmul_rn(dz, dz)));
      // the site itself and its own molecule (exclusions) are skipped
      const bool ok = jj < cnt && rr < lim && ((q.w ^ me.w) >> 8) != 0;
      if (!__any_sync(0xffffffffu, ok)) continue;
      const PairFS P = prow[q.w & 255];
      float flj, y;
      float f = pair_force_rn(P, ok ? rr : 1.f, erd, sgrid, ntab, flj, y);
      f = ok ? f : 0.f;
      ax = __fmaf_rn(f, dx, ax);
      ay = __fmaf_rn(f, dy, ay);
      az = __fmaf_rn(f, dz, az);
      float e_p = 0.f;
      if (POLAR) {
        // shell(i) - centre(j), centre(i) - shell(j), shell(i) - shell(j)
        const float4 qd = sjd[warp][jj];
        const float ex = __fadd_rn(dx, md.x), ey = __fadd_rn(dy, md.y), ez = __fadd_rn(dz, md.z);
        const float cx = __fadd_rn(dx, -qd.x), cy = __fadd_rn(dy, -qd.y),
                    cz = __fadd_rn(dz, -qd.z);
        const float ux = __fadd_rn(ex, -qd.x), uy = __fadd_rn(ey, -qd.y),
                    uz = __fadd_rn(ez, -qd.z);
        float fp = drude_force_rn<MEASURE>(erd, eru, ex, ey, ez, sgrid, ntab, P.qpc, e_p);
        float fc = drude_force_rn<MEASURE>(erd, eru, cx, cy, cz, sgrid, ntab, P.qcp, e_p);
        float fd = drude_force_rn<MEASURE>(erd, eru, ux, uy, uz, sgrid, ntab, P.qpp, e_p);
        fp = ok ? fp : 0.f;
        fc = ok ? fc : 0.f;
        fd = ok ? fd : 0.f;
        ax = __fmaf_rn(fc, cx, ax);
        ay = __fmaf_rn(fc, cy, ay);
        az = __fmaf_rn(fc, cz, az);
        bx = __fmaf_rn(fp, ex, __fmaf_rn(fd, ux, bx));
        by = __fmaf_rn(fp, ey, __fmaf_rn(fd, uy, by));
        bz = __fmaf_rn(fp, ez, __fmaf_rn(fd, uz, bz));
        if (MEASURE && ok) {
          pv.add(ex, ey, ez, fp);
          pv.add(cx, cy, cz, fc);
          pv.add(ux, uy, uz, fd);
        }
      }
      if (MEASURE && ok) {
        // energies and virial: no effect on the forces
        const float xt = rr - P.C2q;
        e_lj += rr < P.C1q ? P.E4 * ((y - P.lam) * y) : (rr < P.C2q ? P.A * xt * xt : 0.f);
        e_vir += rr * flj;
        float e_el_p = 0.f;
        spline_any<true, true>(erd, eru, rr, sgrid, ntab, P.qq, e_el_p);
        e_el += e_el_p + e_p;
        pv.add(dx, dy, dz, f);
      }
    }
    fx.add(ax); fy.add(ay); fz.add(az);
    if (POLAR) { gx.add(bx); gy.add(by); gz.add(bz); }
    if (MEASURE) {
      es[0].add(e_el); es[1].add(e_lj); es[2].add(e_vir);
      es[3].add(pv.p0); es[4].add(pv.p1); es[5].add(pv.p2);
      es[6].add(pv.p3); es[7].add(pv.p4); es[8].add(pv.p5);
    }
  }
  double g[6] = {fx.value(), fy.value(), fz.value(), gx.value(), gy.value(), gz.value()};
#pragma unroll
  for (int k = 0; k < NC; k++) {
    g[k] += __shfl_xor_sync(0xffffffffu, g[k], 8);
    g[k] += __shfl_xor_sync(0xffffffffu, g[k], 16);
    if (sl == 0) red[warp][k][lane] = g[k];
  }
  __syncthreads();
  if (warp == 0 && vi)
    for (int k = sl; k < NC; k += 4) {
      double t = 0;
#pragma unroll
      for (int w = 0; w < NW; w++) t += red[w][k][lane & 7];
      a.f[(k >= 3 ? 3 * (long)a.ns : 0) + 3 * (long)a.order[ti] + k % 3] = t;
    }
  if (MEASURE) {
    // each unordered pair was visited from both ends; the lanes' sums by
    // butterfly, compensated in FP32 (the FP64 pipe is narrow), then the
    // warps in order in FP64
    double e[9];
#pragma unroll
    for (int k = 0; k < 9; k++) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const float s = __shfl_xor_sync(0xffffffffu, es[k].s, o),
                    c = __shfl_xor_sync(0xffffffffu, es[k].c, o);
        es[k].add(s);
        es[k].c += c;
      }
      e[k] = 0.5 * es[k].value();
    }
    __syncthreads();
    double* er = &red[0][0][0];   // at least 9 NW values
    static_assert(NC * ALL_SITES >= 9, "energy sums fit the force sums");
    if (lane == 0)
#pragma unroll
      for (int k = 0; k < 9; k++) er[k * NW + warp] = e[k];
    __syncthreads();
    if (threadIdx.x < 9) {
      double t = 0;
      for (int w = 0; w < NW; w++) t += er[threadIdx.x * NW + w];
      a.epart[bx_ * NEN + threadIdx.x] = t;
    }
  }
}

template <bool MEASURE, bool POLAR>
__global__ void __launch_bounds__(ALL_WARPS * 32, POLAR ? 1 : 2)
    pair_all_kernel(const __grid_constant__ PairArgs a, const int4* __restrict__ pj,
                    const PairF* __restrict__ ptab_g, const float4* __restrict__ erd,
                    const float4* __restrict__ eru, float sx, float sy, float sz, float cq,
                    float sgrid) {
  after_previous();
  pair_all_kernel_body<MEASURE, POLAR>(a, pj, ptab_g, erd, eru, sx, sy, sz, cq, sgrid, blockIdx.x);
}

// ------------------------------ group kernel, half shell, lanes on the
// neighbours --
//
// Every pair once, over a half-shell stencil (the columns with dx > 0, or
// dx = 0 and dy > 0, whole; the column (0, 0) from the home cell up, pairs
// inside the home cell taken from their site with the lower sorted index).
// Work item: a group of up to GROUP_SITES = 8 consecutive sorted sites of a
// home cell; `split` warps share one, each taking every split-th batch of its
// candidates (one warp a group fills the GPU from about 40000 sites on;
// smaller boxes have too few groups).
//
// The candidates are the sites of the half-shell's z-runs: one run per lane
// (its bounds found side by side; one after the other they cost a chain of
// dependent loads each), read in batches of 32, each loaded before the one
// before it is used.  Those outside the cutoff sphere around
// the group's bounding box are dropped, the others compacted into a ring of 64
// per warp; whenever 32 are queued, each lane takes one and runs it against
// the group's home sites, which every lane reads from shared memory
// (broadcast).  The neighbour's force stays in the lane's registers and goes
// into the 64-bit fixed-point sums with three atomics after the home sites;
// the home sites' forces stay in registers and are reduce-scattered over the
// warp once per group.
//
// The home sites come with those that have a Lennard-Jones term or a shell
// first, in quads: a quad without any of them takes the Coulomb term alone
// (half of the quads in water; about 31 instead of 46 instructions a pair).
// The two quads stand in one block, so that the compiler interleaves their
// eight independent chains: a branch per quad measured 0.305 ms on 32768
// waters, a branch per site as slow.
// With Drude shells (POLAR) a heavy quad takes the four charge terms of a
// pair, a light one the two of the home centre.
//
// Every rounding of the force arithmetic is explicit, so the measuring and
// the plain instantiation move the sites identically; the integer sums make
// the forces bit-reproducible.
//
// The virial of a measured evaluation needs no term per pair: the sum of
// (r_i - r_j) x f_ij over pairs is that of r_i x F_i over the ends, positions
// from the cell centre, so each candidate and each home site adds six products
// to compensated sums.
//
// Bound by issue (63 %) and the gathers of the erfc table through L1.  Measured:
// 0.255 ms on 32768 waters (lane per home site 0.363, without the quads and
// the side-by-side runs 0.267), 45 us on 12544 sites (61), 25 us on 864 waters
// (61; cell kernel 110), 0.59 ms with 32768 shells (lane per home site 0.67),
// 0.65 ms on a batch of 256 ionic boxes (cell kernel 0.94).

// the z-ranges of half-shell span sp around cell (cx, cy, cz): column index
// col; run [ra0, ra1] and, where the run wraps through the box, [rb0, rb1]
__device__ __forceinline__ void half_span_runs(const PairArgs& a, int sp, int cx, int cy,
                                               int cz, int& col, int& ra0, int& ra1, int& rb0,
                                               int& rb1) {
  const int4 o = a.hspans[sp];
  int x2 = cx + o.x, y2 = cy + o.y;
  x2 += (x2 < 0) ? a.ncx : (x2 >= a.ncx ? -a.ncx : 0);
  y2 += (y2 < 0) ? a.ncy : (y2 >= a.ncy ? -a.ncy : 0);
  col = (x2 * a.ncy + y2) * a.ncz;
  int za = cz + o.z, zb = cz + o.w;
  if (zb < 0) { za += a.ncz; zb += a.ncz; }
  if (za >= a.ncz) { za -= a.ncz; zb -= a.ncz; }
  rb0 = 0;
  rb1 = -1;
  if (za < 0) { ra0 = za + a.ncz; ra1 = a.ncz - 1; rb1 = zb; }
  else if (zb >= a.ncz) { ra0 = za; ra1 = a.ncz - 1; rb1 = zb - a.ncz; }
  else { ra0 = za; ra1 = zb; }
}

constexpr int HT_RING = 64;   // compacted candidates per warp (a power of two >= 63)

// the sums v[0..23] of a warp's lanes (v[24..31] zero), in a fixed order: lane
// k ends with the sum of v[k] in v[0]
__device__ __forceinline__ void reduce_scatter(float (&v)[32], int lane) {
#pragma unroll
  for (int w = 16; w >= 1; w >>= 1) {
    const bool up = (lane & w) != 0;
#pragma unroll
    for (int k = 0; k < w; k++) {
      const float keepv = up ? v[w + k] : v[k], sendv = up ? v[k] : v[w + k];
      v[k] = __fadd_rn(keepv, __shfl_xor_sync(0xffffffffu, sendv, w));
    }
  }
}

template <bool MEASURE, bool POLAR, int NW>
__device__ __forceinline__ void pair_half_kernel_body(const PairArgs& a, const int4* __restrict__ pj,
                                   const PairF* __restrict__ ptab_g,
                                   const float4* __restrict__ erd,
                                   const float4* __restrict__ eru, float sx, float sy, float sz,
                                   float cq, float sgrid, const int bx_) {
  constexpr int NT = NW * 32, GS = GROUP_SITES;
  extern __shared__ float4 dyn_smem[];   // the nk x nk FP32 pair table
  __shared__ float4 sq[NW][HT_RING];     // candidate positions (w: kind | mol << 8)
  __shared__ int sqt[NW][HT_RING];       // candidate sorted index
  __shared__ float4 sqd[POLAR ? NW : 1][HT_RING];   // candidate shells
  __shared__ float4 sh[NW][GS];          // the group's home sites, heavy ones first
  __shared__ float4 shd[POLAR ? NW : 1][GS];
  __shared__ int so[NW][GS];             // their places in the group
  __shared__ int spm[NW][GS + 1];        // [k]: the home sites of places below k
  __shared__ int2 runs[NW][64];          // first site and end of the candidate runs
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int il = lane & 7;
  const int nk = a.nkind, ntab = a.ntab;
  PairFS* ptab = reinterpret_cast<PairFS*>(dyn_smem);
  for (int t = threadIdx.x; t < 3 * nk * nk; t += NT)
    dyn_smem[t] = reinterpret_cast<const float4*>(ptab_g + t / 3)[t % 3];
  __syncthreads();
  const int ncell = a.ncx * a.ncy * a.ncz;
  const int split = a.split, w = bx_ * NW + warp, item = w / split, part = w - item * split;
  CSum es[9];

  if (item < a.gstart[ncell]) {
    const int c = a.gcell[item];
    const int cz = c % a.ncz, cy = (c / a.ncz) % a.ncy, cx = c / (a.ncy * a.ncz);
    const int hs = a.cell_start[c], he = a.cell_start[c + 1];
    const int i0 = hs + GS * (item - a.gstart[c]);
    const int ni = min(GS, he - i0);
    if (ngroups(he - hs) > a.maxgroups) mark(a.over);
    const unsigned refx = (unsigned)((((unsigned long long)(2 * cx + 1)) << 31) / a.ncx),
                   refy = (unsigned)((((unsigned long long)(2 * cy + 1)) << 31) / a.ncy),
                   refz = (unsigned)((((unsigned long long)(2 * cz + 1)) << 31) / a.ncz);
    // the home sites (every 8-lane group holds all of them) and their box
    const bool vi = il < ni;
    const int4 me = vi ? pj[i0 + il] : make_int4(0, 0, 0, 0);
    const float xi = __fmul_rn((float)(int)((unsigned)me.x - refx), sx),
                yi = __fmul_rn((float)(int)((unsigned)me.y - refy), sy),
                zi = __fmul_rn((float)(int)((unsigned)me.z - refz), sz);
    float blx = vi ? xi : 3e38f, bly = vi ? yi : 3e38f, blz = vi ? zi : 3e38f;
    float bhx = vi ? xi : -3e38f, bhy = vi ? yi : -3e38f, bhz = vi ? zi : -3e38f;
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) {
      blx = fminf(blx, __shfl_xor_sync(0xffffffffu, blx, o));
      bly = fminf(bly, __shfl_xor_sync(0xffffffffu, bly, o));
      blz = fminf(blz, __shfl_xor_sync(0xffffffffu, blz, o));
      bhx = fmaxf(bhx, __shfl_xor_sync(0xffffffffu, bhx, o));
      bhy = fmaxf(bhy, __shfl_xor_sync(0xffffffffu, bhy, o));
      bhz = fmaxf(bhz, __shfl_xor_sync(0xffffffffu, bhz, o));
    }
    // slots: the heavy sites, the light ones, then the unused (their pairs
    // are masked; a site of kind 0 at the cell centre keeps them finite)
    const bool heavy = vi && ((a.heavy >> (me.w & 255)) & 1);
    const unsigned below = (1u << il) - 1u;
    const unsigned hm = __ballot_sync(0xffffffffu, heavy) & 255u,
                   lm = __ballot_sync(0xffffffffu, vi && !heavy) & 255u;
    const int nh = __popc(hm);
    const int slot = heavy ? __popc(hm & below)
                           : (vi ? nh + __popc(lm & below) : il);
    if (lane < GS) {
      sh[warp][slot] = make_float4(xi, yi, zi, __int_as_float(me.w));
      if (POLAR) shd[warp][slot] = vi ? a.pdj[i0 + il] : make_float4(0.f, 0.f, 0.f, 0.f);
      so[warp][slot] = il;
    }
    int pm = 0;
#pragma unroll
    for (int k = 0; k < GS; k++) {
      const int o = __shfl_sync(0xffffffffu, slot, k);
      if (k < lane && k < ni) pm |= 1 << o;
    }
    if (lane <= GS) spm[warp][lane] = pm;
    __syncwarp();
    const int all = (1 << ni) - 1;
    float hx[GS], hy[GS], hz[GS];
    float gx[POLAR ? GS : 1], gy[POLAR ? GS : 1], gz[POLAR ? GS : 1];
#pragma unroll
    for (int i = 0; i < GS; i++) {
      hx[i] = hy[i] = hz[i] = 0.f;
      if (POLAR) gx[POLAR ? i : 0] = gy[POLAR ? i : 0] = gz[POLAR ? i : 0] = 0.f;
    }

    // cnt queued candidates from ring slot h0: lane -> one candidate
    // against the home sites
    auto run = [&](int h0, int cnt) {
      const bool vt = lane < cnt;
      const int e = vt ? (h0 + lane) & (HT_RING - 1) : h0;   // a valid slot for idle lanes
      const float4 q = sq[warp][e];
      const int tj = sqt[warp][e];
      const float4 qd = POLAR ? sqd[POLAR ? warp : 0][e] : make_float4(0.f, 0.f, 0.f, 0.f);
      const int qw = __float_as_int(q.w);
      const PairFS* pcol = ptab + (qw & 255);
      // the home sites this candidate pairs with: none for an idle lane, the
      // group's, and of a candidate in the home cell only those before it
      const bool inh = (unsigned)(tj - hs) < (unsigned)(he - hs);
      const int mask = !vt ? 0 : (inh ? spm[warp][min(ni, max(tj - i0, 0))] : all);
      float px = 0.f, py = 0.f, pz = 0.f;            // on the candidate
      float ux = 0.f, uy = 0.f, uz = 0.f;            // on its shell
      float e_el = 0.f, e_lj = 0.f, e_vir = 0.f;
      auto pair = [&](const int i, auto full) {
        constexpr bool HEAVY = decltype(full)::value;
        const float4 h = sh[warp][i];
        const float dx = __fadd_rn(h.x, -q.x), dy = __fadd_rn(h.y, -q.y),
                    dz = __fadd_rn(h.z, -q.z);
        const float rr = __fmaf_rn(dx, dx, __fmaf_rn(dy, dy, __fmul_rn(dz, dz)));
        const int hw = __float_as_int(h.w);
        const bool ok = (mask >> i & 1) && rr < cq && ((hw ^ qw) >> 8) != 0;
        const PairFS* pp = pcol + (hw & 255) * nk;
        float f, flj = 0.f, y = 0.f, e_p = 0.f;
        PairFS P;
        if (HEAVY) {
          P = *pp;
          f = pair_force_rn(P, rr, erd, sgrid, ntab, flj, y);
        } else {
          P.qq = pp->qq;
          // no LJ at this home site
          const int ix =
              min(__float_as_int(__fmaf_rz(rr, sgrid, 12582912.f)) - 0x4B400000, ntab - 1);
          const float4 d = __ldg(erd + ix);
          f = __fmul_rn(__fmaf_rn(d.y, rcp_approx(__fadd_rn(d.z, rr)), d.x), P.qq);
        }
        f = ok ? f : 0.f;
        hx[i] = __fmaf_rn(f, dx, hx[i]);
        hy[i] = __fmaf_rn(f, dy, hy[i]);
        hz[i] = __fmaf_rn(f, dz, hz[i]);
        px = __fmaf_rn(f, dx, px);
        py = __fmaf_rn(f, dy, py);
        pz = __fmaf_rn(f, dz, pz);
        if (POLAR) {
          const int ip = POLAR ? i : 0;
          // centre(i) - shell(j)
          const float cx2 = __fadd_rn(dx, -qd.x), cy2 = __fadd_rn(dy, -qd.y),
                      cz2 = __fadd_rn(dz, -qd.z);
          float fc = drude_force_rn<MEASURE>(erd, eru, cx2, cy2, cz2, sgrid, ntab, pp->qcp, e_p);
          fc = ok ? fc : 0.f;
          hx[i] = __fmaf_rn(fc, cx2, hx[i]);
          hy[i] = __fmaf_rn(fc, cy2, hy[i]);
          hz[i] = __fmaf_rn(fc, cz2, hz[i]);
          ux = __fmaf_rn(fc, cx2, ux);
          uy = __fmaf_rn(fc, cy2, uy);
          uz = __fmaf_rn(fc, cz2, uz);
          if (HEAVY) {
            // shell(i) - centre(j), shell(i) - shell(j)
            const float4 md = shd[POLAR ? warp : 0][i];
            const float ex = __fadd_rn(dx, md.x), ey = __fadd_rn(dy, md.y),
                        ez = __fadd_rn(dz, md.z);
            float fp = drude_force_rn<MEASURE>(erd, eru, ex, ey, ez, sgrid, ntab, pp->qpc, e_p);
            const float sx2 = __fadd_rn(ex, -qd.x), sy2 = __fadd_rn(ey, -qd.y),
                        sz2 = __fadd_rn(ez, -qd.z);
            float fd = drude_force_rn<MEASURE>(erd, eru, sx2, sy2, sz2, sgrid, ntab, pp->qpp, e_p);
            fp = ok ? fp : 0.f;
            fd = ok ? fd : 0.f;
            gx[ip] = __fmaf_rn(fp, ex, __fmaf_rn(fd, sx2, gx[ip]));
            gy[ip] = __fmaf_rn(fp, ey, __fmaf_rn(fd, sy2, gy[ip]));
            gz[ip] = __fmaf_rn(fp, ez, __fmaf_rn(fd, sz2, gz[ip]));
            px = __fmaf_rn(fp, ex, px);
            py = __fmaf_rn(fp, ey, py);
            pz = __fmaf_rn(fp, ez, pz);
            ux = __fmaf_rn(fd, sx2, ux);
            uy = __fmaf_rn(fd, sy2, uy);
            uz = __fmaf_rn(fd, sz2, uz);
          }
        }
        if (MEASURE) {
          // energies: no effect on the forces; masked, not branched around, as
          // the forces are
          if (HEAVY) {
            const float xt = rr - P.C2q;
            const float u = rr < P.C1q ? P.E4 * ((y - P.lam) * y) : (rr < P.C2q ? P.A * xt * xt : 0.f);
            e_lj += ok ? u : 0.f;
            e_vir += ok ? rr * flj : 0.f;
          }
          const float4 eu = __ldg(eru + min(__float_as_int(__fmaf_rz(rr, sgrid, 12582912.f)) -
                                                0x4B400000, ntab - 1));
          e_el += ok ? fmaf(fmaf(eu.y, rcp_approx(eu.z + rr), eu.x), P.qq, e_p) : 0.f;
        }
      };
      // the two quads in one block, their eight chains interleaved
      auto quad = [&](const int k, auto full) {
#pragma unroll
        for (int i = 0; i < 4; i++) pair(k + i, full);
      };
      if (nh > 4) { quad(0, BoolC<true>()); quad(4, BoolC<true>()); }
      else if (nh > 0 && ni > 4) { quad(0, BoolC<true>()); quad(4, BoolC<false>()); }
      else if (nh > 0) quad(0, BoolC<true>());
      else if (ni > 4) { quad(0, BoolC<false>()); quad(4, BoolC<false>()); }
      else quad(0, BoolC<false>());
      if (vt) {
        // a term beyond the sums' range, or not a number
        float big = fabsf(px) + fabsf(py) + fabsf(pz);
        if (POLAR) big += fabsf(ux) + fabsf(uy) + fabsf(uz);
        if (!(big < a.flim)) mark(a.bad + tj);
        unsigned long long* fj = reinterpret_cast<unsigned long long*>(a.facc) + 3 * (long)tj;
        atomicAdd(fj, (unsigned long long)__float2ll_rn(__fmul_rn(px, -(float)FIX_SCALE)));
        atomicAdd(fj + 1, (unsigned long long)__float2ll_rn(__fmul_rn(py, -(float)FIX_SCALE)));
        atomicAdd(fj + 2, (unsigned long long)__float2ll_rn(__fmul_rn(pz, -(float)FIX_SCALE)));
        if (POLAR && ((a.shells >> (qw & 255)) & 1)) {
          fj += 3 * (long)a.ns;
          atomicAdd(fj, (unsigned long long)__float2ll_rn(__fmul_rn(ux, -(float)FIX_SCALE)));
          atomicAdd(fj + 1, (unsigned long long)__float2ll_rn(__fmul_rn(uy, -(float)FIX_SCALE)));
          atomicAdd(fj + 2, (unsigned long long)__float2ll_rn(__fmul_rn(uz, -(float)FIX_SCALE)));
        }
      }
      if (MEASURE) {
        es[0].add(e_el); es[1].add(e_lj); es[2].add(e_vir);
        // the candidate's end of the virial sum of r x F
        float w[6] = {q.x * px, q.y * py, q.z * pz, q.z * py, q.x * pz, q.y * px};
        if (POLAR) {
          const float tx = q.x + qd.x, ty = q.y + qd.y, tz = q.z + qd.z;
          w[0] = fmaf(tx, ux, w[0]);
          w[1] = fmaf(ty, uy, w[1]);
          w[2] = fmaf(tz, uz, w[2]);
          w[3] = fmaf(tz, uy, w[3]);
          w[4] = fmaf(tx, uz, w[4]);
          w[5] = fmaf(ty, ux, w[5]);
        }
#pragma unroll
        for (int k = 0; k < 6; k++) es[3 + k].add(-w[k]);
      }
      __syncwarp();   // the slots read here may be refilled next
    };

    int qh = 0, qn = 0;   // ring head and count (warp-uniform)
    for (int sb = 0; sb < a.nhspans; sb += 32) {
      // the runs of spans sb .. sb + 31, the wrapped parts after the others
      int ja = 0, la = 0, jw = 0, lw = 0;
      if (sb + lane < a.nhspans) {
        int col, ra0, ra1, rb0, rb1;
        half_span_runs(a, sb + lane, cx, cy, cz, col, ra0, ra1, rb0, rb1);
        // home-cell sites before the group pair with it from their own group
        ja = max(a.cell_start[col + ra0], col + ra0 == c ? i0 : 0);
        la = a.cell_start[col + ra1 + 1] - ja;
        if (rb1 >= rb0) {
          jw = max(a.cell_start[col + rb0], col + rb0 == c ? i0 : 0);
          lw = a.cell_start[col + rb1 + 1] - jw;
        }
      }
      auto sum = [&](int v) {   // inclusive prefix over the lanes
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int u = __shfl_up_sync(0xffffffffu, v, o);
          if (lane >= o) v += u;
        }
        return v;
      };
      const int pa = sum(la), ta = __shfl_sync(0xffffffffu, pa, 31);
      const int pw = sum(lw), total = ta + __shfl_sync(0xffffffffu, pw, 31);
      // this warp's share [k0, k1) of the candidates: each run cut to it
      const int share = (total + split - 1) / split, k0 = share * part, k1 = k0 + share;
      auto cut = [&](int& first, int len, int before) {
        const int lo = min(max(k0 - before, 0), len), hi = min(max(k1 - before, 0), len);
        first += lo;
        return hi - lo;
      };
      la = cut(ja, la, pa - la);
      lw = cut(jw, lw, ta + pw - lw);
      const unsigned ma = __ballot_sync(0xffffffffu, la > 0),
                     mw = __ballot_sync(0xffffffffu, lw > 0), lt = (1u << lane) - 1u;
      const int na = __popc(ma), nr = na + __popc(mw);
      __syncwarp();
      if (la > 0) runs[warp][__popc(ma & lt)] = make_int2(ja, ja + la);
      if (lw > 0) runs[warp][na + __popc(mw & lt)] = make_int2(jw, jw + lw);
      __syncwarp();
      if (nr == 0) continue;
      // batches of 32 of each run, loaded one batch ahead
      int r = 0;
      int2 u = runs[warp][0];
      int jn = u.x + lane;
      bool in = jn < u.y;
      int4 pn = in ? pj[jn] : make_int4(0, 0, 0, 0);
      for (bool more = true; more;) {
        const int j = in ? jn : -1;
        const int4 p = pn;
        u.x += 32;
        if (u.x >= u.y) {
          r++;
          more = r < nr;
          if (more) u = runs[warp][r];
        }
        jn = u.x + lane;
        in = more && jn < u.y;
        if (in) pn = pj[jn];
        const float4 f4 = make_float4(__fmul_rn((float)(int)((unsigned)p.x - refx), sx),
                                      __fmul_rn((float)(int)((unsigned)p.y - refy), sy),
                                      __fmul_rn((float)(int)((unsigned)p.z - refz), sz),
                                      __int_as_float(p.w));
        const float ddx = fmaxf(fmaxf(blx - f4.x, f4.x - bhx), 0.f),
                    ddy = fmaxf(fmaxf(bly - f4.y, f4.y - bhy), 0.f),
                    ddz = fmaxf(fmaxf(blz - f4.z, f4.z - bhz), 0.f);
        const bool keep = j >= 0 && fmaf(ddx, ddx, fmaf(ddy, ddy, ddz * ddz)) < cq;
        const unsigned M = __ballot_sync(0xffffffffu, keep);
        if (keep) {
          // qn < 32 here, so the new slots never reach the queued ones
          const int e = (qh + qn + __popc(M & ((1u << lane) - 1u))) & (HT_RING - 1);
          sq[warp][e] = f4;
          sqt[warp][e] = j;
          if (POLAR) sqd[POLAR ? warp : 0][e] = a.pdj[j];
        }
        qn += __popc(M);
        __syncwarp();
        if (qn >= 32) {
          run(qh, 32);
          qh = (qh + 32) & (HT_RING - 1);
          qn -= 32;
        }
      }
    }
    if (qn > 0) run(qh, qn);

    if (MEASURE) {
      // the home sites' end of the virial sum
#pragma unroll
      for (int i = 0; i < GS; i++) {
        const float4 h = sh[warp][i];
        float w[6] = {h.x * hx[i], h.y * hy[i], h.z * hz[i], h.z * hy[i], h.x * hz[i], h.y * hx[i]};
        if (POLAR) {
          const int ip = POLAR ? i : 0;
          const float4 d = shd[POLAR ? warp : 0][i];
          const float tx = h.x + d.x, ty = h.y + d.y, tz = h.z + d.z;
          w[0] = fmaf(tx, gx[ip], w[0]);
          w[1] = fmaf(ty, gy[ip], w[1]);
          w[2] = fmaf(tz, gz[ip], w[2]);
          w[3] = fmaf(tz, gy[ip], w[3]);
          w[4] = fmaf(tx, gz[ip], w[4]);
          w[5] = fmaf(ty, gx[ip], w[5]);
        }
#pragma unroll
        for (int k = 0; k < 6; k++) es[3 + k].add(w[k]);
      }
    }

    // the home sites' sums: lane 3 i + d ends with component d of slot i
    unsigned long long* facc = reinterpret_cast<unsigned long long*>(a.facc);
    const int slot_i = min(lane / 3, GS - 1), d = lane % 3;
    const long at = 3 * (long)(i0 + so[warp][slot_i]) + d;
    float v[32];
#pragma unroll
    for (int k = 3 * GS; k < 32; k++) v[k] = 0.f;
#pragma unroll
    for (int i = 0; i < GS; i++) {
      v[3 * i] = hx[i];
      v[3 * i + 1] = hy[i];
      v[3 * i + 2] = hz[i];
    }
    reduce_scatter(v, lane);
    if (!(fabsf(v[0]) < a.flim)) mark(a.bad + at / 3);   // lanes from 3 ni on: zero
    if (lane < 3 * ni)
      atomicAdd(facc + at, (unsigned long long)__float2ll_rn(__fmul_rn(v[0], (float)FIX_SCALE)));
    if (POLAR && nh > 0) {
#pragma unroll
      for (int k = 3 * GS; k < 32; k++) v[k] = 0.f;
#pragma unroll
      for (int i = 0; i < GS; i++) {
        const int ip = POLAR ? i : 0;
        v[3 * i] = gx[ip];
        v[3 * i + 1] = gy[ip];
        v[3 * i + 2] = gz[ip];
      }
      reduce_scatter(v, lane);
      if (!(fabsf(v[0]) < a.flim)) mark(a.bad + at / 3);
      if (lane < 3 * nh)
        atomicAdd(facc + 3 * (long)a.ns + at,
                  (unsigned long long)__float2ll_rn(__fmul_rn(v[0], (float)FIX_SCALE)));
    }
  }
  if (MEASURE) {
    // every unordered pair once; one row per CTA.  The lanes' sums stay
    // compensated FP32 (lane 9 t + k adds sum k of the lanes of third t): an
    // FP64 butterfly of nine sums kept the narrow FP64 pipe busy for 21 us on
    // 864 waters; the warps' sums are added in FP64, in order
    __shared__ float2 em[NW][32][9];
    __shared__ double er[NW][27];
#pragma unroll
    for (int k = 0; k < 9; k++) em[warp][lane][k] = make_float2(es[k].s, es[k].c);
    __syncwarp();
    if (lane < 27) {
      const int t = lane / 9, k = lane - 9 * t;
      CSum e;
      for (int l = 11 * t; l < min(32, 11 * t + 11); l++) {
        const float2 v = em[warp][l][k];
        e.add(v.x);
        e.c += v.y;
      }
      er[warp][lane] = e.value();
    }
    __syncthreads();
    if (threadIdx.x < 9) {
      double e = 0;
#pragma unroll
      for (int q = 0; q < NW; q++)
#pragma unroll
        for (int t = 0; t < 3; t++) e += er[q][9 * t + threadIdx.x];
      a.epart[bx_ * NEN + threadIdx.x] = e;
    }
  }
}

template <bool MEASURE, bool POLAR, int NW>
__global__ void __launch_bounds__(NW * 32, MEASURE ? (POLAR ? 2 : 3) : (POLAR ? 4 : 5))
    pair_half_mixed_kernel(const __grid_constant__ PairArgs a, const int4* __restrict__ pj,
                           const PairF* __restrict__ ptab_g, const float4* __restrict__ erd,
                           const float4* __restrict__ eru, float sx, float sy, float sz, float cq,
                           float sgrid) {
  after_previous();
  pair_half_kernel_body<MEASURE, POLAR, NW>(a, pj, ptab_g, erd, eru, sx, sy, sz, cq, sgrid,
                                            blockIdx.x);
}

// The force on sorted site t from all its pairs by a warp, FP32 pair terms (those
// of the half-shell kernel) added in FP64: marked sites, overlapping ones of a
// random start or a hot fluid.  Some 5 us a site.
template <bool POLAR>
__device__ __noinline__ void direct_forces(const PairArgs& a, int t, const int4* __restrict__ pj,
                                           const PairF* __restrict__ ptab,
                                           const float4* __restrict__ erd, float sx, float sy,
                                           float sz, float cq, float sgrid) {
  constexpr int NC = POLAR ? 6 : 3;
  const int ntab = a.ntab, c = a.key_s[t], lane = threadIdx.x & 31;
  const int cz = c % a.ncz, cy = (c / a.ncz) % a.ncy, cx = c / (a.ncy * a.ncz);
  const int4 me = pj[t];
  const float4 md = POLAR ? a.pdj[t] : make_float4(0.f, 0.f, 0.f, 0.f);
  double F[NC];
#pragma unroll
  for (int k = 0; k < NC; k++) F[k] = 0;
  auto add = [&](int k, float f, float x, float y, float z) {
    F[k] += (double)f * x;
    F[k + 1] += (double)f * y;
    F[k + 2] += (double)f * z;
  };
  for (int s = 0; s < a.nstencil; s++) {
    const int4 o = a.stencil[s];
    int x = cx + o.x, y = cy + o.y, z = cz + o.z;
    x += x < 0 ? a.ncx : (x >= a.ncx ? -a.ncx : 0);
    y += y < 0 ? a.ncy : (y >= a.ncy ? -a.ncy : 0);
    z += z < 0 ? a.ncz : (z >= a.ncz ? -a.ncz : 0);
    const int c2 = (x * a.ncy + y) * a.ncz + z;
    for (int j = a.cell_start[c2] + lane; j < a.cell_start[c2 + 1]; j += 32) {
      const int4 q = pj[j];
      const float dx = __fmul_rn((float)(int)((unsigned)me.x - (unsigned)q.x), sx),
                  dy = __fmul_rn((float)(int)((unsigned)me.y - (unsigned)q.y), sy),
                  dz = __fmul_rn((float)(int)((unsigned)me.z - (unsigned)q.z), sz);
      const float rr = __fmaf_rn(dx, dx, __fmaf_rn(dy, dy, __fmul_rn(dz, dz)));
      if (!(rr < cq) || ((q.w ^ me.w) >> 8) == 0) continue;
      const PairFS& P =
          *reinterpret_cast<const PairFS*>(ptab + (me.w & 255) * a.nkind + (q.w & 255));
      float flj, lj6;
      add(0, pair_force_rn(P, rr, erd, sgrid, ntab, flj, lj6), dx, dy, dz);
      if constexpr (POLAR) {
        const float4 qd = a.pdj[j];
        float e = 0.f;
        const float ex = __fadd_rn(dx, md.x), ey = __fadd_rn(dy, md.y), ez = __fadd_rn(dz, md.z);
        add(3, drude_force_rn<false>(erd, nullptr, ex, ey, ez, sgrid, ntab, P.qpc, e), ex, ey, ez);
        const float vx = __fadd_rn(dx, -qd.x), vy = __fadd_rn(dy, -qd.y), vz = __fadd_rn(dz, -qd.z);
        add(0, drude_force_rn<false>(erd, nullptr, vx, vy, vz, sgrid, ntab, P.qcp, e), vx, vy, vz);
        const float ux = __fadd_rn(ex, -qd.x), uy = __fadd_rn(ey, -qd.y), uz = __fadd_rn(ez, -qd.z);
        add(3, drude_force_rn<false>(erd, nullptr, ux, uy, uz, sgrid, ntab, P.qpp, e), ux, uy, uz);
      }
    }
  }
#pragma unroll
  for (int k = 0; k < NC; k++) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) F[k] += __shfl_xor_sync(0xffffffffu, F[k], o);
    if (lane == 0) a.f[(k < 3 ? 0 : 3 * (long)a.ns) + 3 * (long)a.order[t] + k % 3] = F[k];
  }
}

// the fixed-point sums (sorted order) into the FP64 forces (site order),
// with shells the second half of each; the sums are cleared for the next
// evaluation, and the marks.  Whole warps.
template <bool POLAR>
__device__ __forceinline__ void finish_forces(const PairArgs& a, const int4* __restrict__ pj,
                                              const PairF* __restrict__ ptab,
                                              const float4* __restrict__ erd, float sx, float sy,
                                              float sz, float cq, float sgrid) {
  constexpr int NH = POLAR ? 2 : 1;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  bool redo = false;
  if (t < a.ns) {
    // every load before the first store
    const int site = a.order[t], bad = a.bad[t], over = *a.over;
    long long v[NH][3];
#pragma unroll
    for (int h = 0; h < NH; h++)
#pragma unroll
      for (int k = 0; k < 3; k++) v[h][k] = a.facc[3 * ((long)a.ns * h + t) + k];
#pragma unroll
    for (int h = 0; h < NH; h++)
#pragma unroll
      for (int k = 0; k < 3; k++) {
        a.f[3 * ((long)a.ns * h + site) + k] = (double)v[h][k] * (1.0 / FIX_SCALE);
        a.facc[3 * ((long)a.ns * h + t) + k] = 0;
      }
    redo = (bad | over) != 0;
    if (bad) a.bad[t] = 0;
  }
  unsigned m = __ballot_sync(0xffffffffu, redo);
  __syncwarp();
  for (; m; m &= m - 1)
    direct_forces<POLAR>(a, t - (int)(threadIdx.x & 31) + __ffs(m) - 1, pj, ptab, erd, sx, sy, sz,
                         cq, sgrid);
}

template <bool POLAR>
__global__ void __launch_bounds__(256)
    finish_forces_kernel(const __grid_constant__ PairArgs a, const int4* __restrict__ pj,
                         const PairF* __restrict__ ptab, const float4* __restrict__ erd, float sx,
                         float sy, float sz, float cq, float sgrid) {
  after_previous();
  finish_forces<POLAR>(a, pj, ptab, erd, sx, sy, sz, cq, sgrid);
}

cudaError_t k_pair_mixed(const Launch& L, const PairArgs& a, const int4* pj, const PairF* ptab,
                         const float4* erd, const float4* eru, bool measure, bool polar) {
  int ncell = a.ncx * a.ncy * a.ncz;
  float sx = (float)(a.Lx / 4294967296.0), sy = (float)(a.Ly / 4294967296.0),
        sz = (float)(a.Lz / 4294967296.0);
  const float cq = (float)a.cutoff_sq, sg = (float)a.sgrid, al = (float)a.alpha;
  if (a.small) {
    const size_t sm = sizeof(PairFS) * (size_t)a.nkind * a.nkind;
    cudaError_t se = cudaSuccess;
    // with the static part (22 KB with shells) this may pass 48 KB
#define PAIR_ALL(M, P)                                                                          \
  do {                                                                                          \
    if (sm > 24 * 1024)                                                                         \
      se = cudaFuncSetAttribute(pair_all_kernel<M, P>,                                          \
                                cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);          \
    if (se == cudaSuccess)                                                                      \
      launch_after(L, pair_all_kernel<M, P>, pair_all_blocks(a.ns), ALL_WARPS * 32, sm, a, pj,  \
                   ptab, erd, eru, sx, sy, sz, cq, sg);                                         \
  } while (0)
    if (polar) { if (measure) PAIR_ALL(true, true); else PAIR_ALL(false, true); }
    else { if (measure) PAIR_ALL(true, false); else PAIR_ALL(false, false); }
#undef PAIR_ALL
    if (se != cudaSuccess) return se;
    LAUNCHED(L);
    return cudaGetLastError();
  }
  if (a.group && a.newton) {
    const size_t gsm = sizeof(PairFS) * (size_t)a.nkind * a.nkind;
    cudaError_t ge = cudaSuccess;
    // with the static part (up to 23 KB) this may pass 48 KB
#define PAIR_HALF(M, P)                                                                         \
  do {                                                                                          \
    if (gsm > 24 * 1024)                                                                        \
      ge = cudaFuncSetAttribute(pair_half_mixed_kernel<M, P, GROUP_WARPS>,                     \
                                cudaFuncAttributeMaxDynamicSharedMemorySize, (int)gsm);         \
    if (ge == cudaSuccess)                                                                      \
      pair_half_mixed_kernel<M, P, GROUP_WARPS>                                                 \
          <<<a.ngrid * a.split, GROUP_WARPS * 32, gsm, L.s>>>(a, pj, ptab, erd, eru, sx, sy, sz, \
                                                              cq, sg);                          \
  } while (0)
    if (polar) { if (measure) PAIR_HALF(true, true); else PAIR_HALF(false, true); }
    else { if (measure) PAIR_HALF(true, false); else PAIR_HALF(false, false); }
#undef PAIR_HALF
    if (ge != cudaSuccess) return ge;
    LAUNCHED(L);
    // with shells plainly: set up beside the last pair CTAs, 59 registers a thread,
    // it cost 32768 Drude waters 19 us a step; without shells set up early (864
    // waters 138 -> 132 us an evaluation)
    if (polar) {
      finish_forces_kernel<true>
          <<<cdiv(a.ns, 256), 256, 0, L.s>>>(a, pj, ptab, erd, sx, sy, sz, cq, sg);
    } else {
      launch_after(L, finish_forces_kernel<false>, cdiv(a.ns, 256), 256, 0, a, pj, ptab, erd, sx,
                   sy, sz, cq, sg);
    }
    LAUNCHED(L);
    return cudaGetLastError();
  }
  if (a.group) {
    const size_t gsm = sizeof(PairFS) * (size_t)a.nkind * a.nkind;
    cudaError_t ge = cudaSuccess;
#define PAIR_GROUP(M, P)                                                                        \
  do {                                                                                          \
    if (gsm > 48 * 1024)                                                                        \
      ge = cudaFuncSetAttribute(pair_group_mixed_kernel<M, P, GROUP_WARPS>,                    \
                                cudaFuncAttributeMaxDynamicSharedMemorySize, (int)gsm);         \
    if (ge == cudaSuccess)                                                                      \
      pair_group_mixed_kernel<M, P, GROUP_WARPS><<<a.ngrid, GROUP_WARPS * 32, gsm, L.s>>>(     \
          a, pj, ptab, erd, eru, sx, sy, sz, cq, sg);                                           \
  } while (0)
    if (polar) { if (measure) PAIR_GROUP(true, true); else PAIR_GROUP(false, true); }
    else { if (measure) PAIR_GROUP(true, false); else PAIR_GROUP(false, false); }
#undef PAIR_GROUP
    if (ge != cudaSuccess) return ge;
    LAUNCHED(L);
    return cudaGetLastError();
  }
  // the measuring kernel (energies, virial) always runs with 4 warps and the
  // spline through L1: with more registers per thread it keeps more CTAs
  // resident that way (1.0 ms on 32768 waters; 16 warps + shared-memory
  // spline, the fastest force-only choice there, 1.8 ms)
  const int nw = measure ? 4 : (a.pair_warps == 16 ? 16 : (a.pair_warps == 8 ? 8 : 4));
  const bool stab = a.spline_smem && !measure;
  const size_t dsm = sizeof(PairFS) * (size_t)a.nkind * a.nkind +
                     (stab ? sizeof(float4) * (size_t)a.ntab : 0);
  cudaError_t e = cudaSuccess;
#define PAIR_MIXED(M, P, W, S)                                                                  \
  do {                                                                                          \
    if (dsm > 48 * 1024)                                                                        \
      e = cudaFuncSetAttribute(pair_mixed_kernel<M, P, W, S>,                                   \
                               cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dsm);          \
    if (e == cudaSuccess)                                                                       \
      pair_mixed_kernel<M, P, W, S><<<ncell, W * 32, dsm, L.s>>>(a, pj, ptab, erd, eru, sx, sy, \
                                                                 sz, cq, sg, al);               \
  } while (0)
#define PAIR_MIXED_W(M, P)                              \
  do {                                                  \
    if (nw == 16) {                                     \
      if (stab) PAIR_MIXED(M, P, 16, true);             \
      else PAIR_MIXED(M, P, 16, false);                 \
    } else if (nw == 8) {                               \
      if (stab) PAIR_MIXED(M, P, 8, true);              \
      else PAIR_MIXED(M, P, 8, false);                  \
    } else {                                            \
      if (stab) PAIR_MIXED(M, P, 4, true);              \
      else PAIR_MIXED(M, P, 4, false);                  \
    }                                                   \
  } while (0)
  if (polar) { if (measure) PAIR_MIXED_W(true, true); else PAIR_MIXED_W(false, true); }
  else { if (measure) PAIR_MIXED_W(true, false); else PAIR_MIXED_W(false, false); }
#undef PAIR_MIXED_W
#undef PAIR_MIXED
  if (e != cudaSuccess) return e;
  LAUNCHED(L);
  return cudaGetLastError();
}

// ------------------------------------------------ Ewald exclusion terms --

// -erf(alpha r)/r of the intramolecular pairs (cook/ljqqnp.c:131-141, its
// Drude forms cook/ljqqpol.c) for the mixed cell path: each pair once, from
// the FP64 positions (nearest image), the term in FP32 but for its last steps
// (excl_mixed), forces and energy summed in FP64.  Pairs beyond the cutoff are
// skipped, as the cell traversal never meets them.
// The force arithmetic rounds explicitly (`_rn`): the measuring
// instantiation also uses the products for the virial, and a product the
// compiler fuses into the force sum in one instantiation and not in the
// other would move the sites of a measured step differently.
__device__ __forceinline__ double excl_r2(double dx, double dy, double dz) {
  return __fma_rn(dx, dx, __fma_rn(dy, dy, __dmul_rn(dz, dz)));
}

template <bool MEASURE>
__device__ __forceinline__ void excl_pair(double dx, double dy, double dz, double qq, double alpha,
                                          double* fi, double* fj, double* en) {
  double fe;
  const double e = excl_mixed(excl_r2(dx, dy, dz), alpha, &fe);
  const double fq = __dmul_rn(fe, qq);
  const double Fx = __dmul_rn(fq, dx), Fy = __dmul_rn(fq, dy), Fz = __dmul_rn(fq, dz);
  fi[0] = __dadd_rn(fi[0], Fx);
  fi[1] = __dadd_rn(fi[1], Fy);
  fi[2] = __dadd_rn(fi[2], Fz);
  fj[0] = __dadd_rn(fj[0], -Fx);
  fj[1] = __dadd_rn(fj[1], -Fy);
  fj[2] = __dadd_rn(fj[2], -Fz);
  if (MEASURE) {
    en[0] += e * qq;
    en[1] += Fx * dx;
    en[2] += Fy * dy;
    en[3] += Fz * dz;
    en[4] += Fz * dy;
    en[5] += Fx * dz;
    en[6] += Fy * dx;
  }
}

__device__ __forceinline__ double near_img(double d, double L, double iL) {
  return d - L * rint(d * iL);
}

// A warp per CTA (a molecule's pairs are one chain of loads and FP64 products,
// so the molecules spread over the SMs); rigid three-site molecules keep their
// sites in registers.  864 waters 9.0 -> 7.4 us, measured 15 -> 10.5 us (6.2 and 8.5
// with the terms as FP32 differences, good to 3e-6 where the series are to 1e-7).
template <bool MEASURE, bool POLAR>
MG_BODY void excl_mixed_kernel_body(const ExclArgs& a,
    const int bx_,
    const int by_) {
  static_assert(EXCL_THREADS == 32, "one warp per CTA");
  const int n = bx_ * EXCL_THREADS + threadIdx.x;
  double en[7] = {0, 0, 0, 0, 0, 0, 0};
  if (n < a.nmol) {
    const int b = POLAR ? -1 : a.base3[n];
    if (b >= 0) {
      // the three pairs (0,1), (0,2), (1,2) of sites b, b+1, b+2: positions and
      // forces read once, the same additions in the same order
      double x[3][3], F[3][3];
      const double* r = a.r + 3 * (long)b;
      double* f = a.f + 3 * (long)b;
#pragma unroll
      for (int s = 0; s < 3; s++)
#pragma unroll
        for (int d = 0; d < 3; d++) {
          x[s][d] = r[3 * s + d];
          F[s][d] = f[3 * s + d];
        }
      const int p0 = a.xfirst[n];
#pragma unroll
      for (int p = 0; p < 3; p++) {
        const int i = p == 2 ? 1 : 0, j = p == 0 ? 1 : 2;
        const double q = a.xq[p0 + p].x;
        const double dx = near_img(x[i][0] - x[j][0], a.Lx, a.iLx),
                     dy = near_img(x[i][1] - x[j][1], a.Ly, a.iLy),
                     dz = near_img(x[i][2] - x[j][2], a.Lz, a.iLz);
        if (excl_r2(dx, dy, dz) < a.cutoff_sq)
          excl_pair<MEASURE>(dx, dy, dz, q, a.alpha, F[i], F[j], en);
      }
#pragma unroll
      for (int s = 0; s < 3; s++)
#pragma unroll
        for (int d = 0; d < 3; d++) f[3 * s + d] = F[s][d];
    } else {
    const long ns3 = 3 * (long)a.ns;
    for (int p = a.xfirst[n]; p < a.xfirst[n + 1]; p++) {
      const int2 ij = a.xpair[p];
      const double4 q = a.xq[p];
      const double* ri = a.r + 3 * (long)ij.x;
      const double* rj = a.r + 3 * (long)ij.y;
      const double dx = near_img(ri[0] - rj[0], a.Lx, a.iLx),
                   dy = near_img(ri[1] - rj[1], a.Ly, a.iLy),
                   dz = near_img(ri[2] - rj[2], a.Lz, a.iLz);
      if (!(excl_r2(dx, dy, dz) < a.cutoff_sq)) continue;
      double* fi = a.f + 3 * (long)ij.x;
      double* fj = a.f + 3 * (long)ij.y;
      if (q.x != 0) excl_pair<MEASURE>(dx, dy, dz, q.x, a.alpha, fi, fj, en);
      if (POLAR) {
        const double* mi = ri + ns3;
        const double* mj = rj + ns3;
        double* gi = fi + ns3;
        double* gj = fj + ns3;
        if (q.y != 0)  // Drude(i) - centre(j)
          excl_pair<MEASURE>(dx + mi[0], dy + mi[1], dz + mi[2], q.y, a.alpha, gi, fj, en);
        if (q.z != 0)  // centre(i) - Drude(j)
          excl_pair<MEASURE>(dx - mj[0], dy - mj[1], dz - mj[2], q.z, a.alpha, fi, gj, en);
        if (q.w != 0)  // Drude(i) - Drude(j)
          excl_pair<MEASURE>(dx + mi[0] - mj[0], dy + mi[1] - mj[1], dz + mi[2] - mj[2], q.w,
                             a.alpha, gi, gj, en);
      }
    }
  }
  }
  if (MEASURE) {
    // row layout of the pair kernels: el, lj, vir, Pvir[6], spare
#pragma unroll
    for (int m = 0; m < 7; m++)
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) en[m] += __shfl_xor_sync(0xffffffffu, en[m], o);
    if (threadIdx.x == 0) {
      double* e = a.epart + (long)bx_ * NEN;
      e[0] = en[0];
      e[1] = e[2] = e[9] = 0;
#pragma unroll
      for (int m = 1; m < 7; m++) e[m + 2] = en[m];
    }
  }
}

template <bool MEASURE, bool POLAR>
__global__ void __launch_bounds__(EXCL_THREADS) excl_mixed_kernel(const __grid_constant__ ExclArgs a) {
  after_previous();
  excl_mixed_kernel_body<MEASURE, POLAR>(a, blockIdx.x, 0);
}

cudaError_t k_excl_mixed(const Launch& L, const ExclArgs& a, bool measure, bool polar) {
  if (a.nmol <= 0) return cudaSuccess;
  const int nb = cdiv(a.nmol, EXCL_THREADS);
  if (measure) {
    if (polar) launch_after(L, excl_mixed_kernel<true, true>, nb, EXCL_THREADS, 0, a);
    else launch_after(L, excl_mixed_kernel<true, false>, nb, EXCL_THREADS, 0, a);
  } else {
    if (polar) launch_after(L, excl_mixed_kernel<false, true>, nb, EXCL_THREADS, 0, a);
    else launch_after(L, excl_mixed_kernel<false, false>, nb, EXCL_THREADS, 0, a);
  }
  LAUNCHED(L);
  return cudaGetLastError();
}

__global__ void gather_drude_kernel(int ns, const double* __restrict__ r,
                                    const int* __restrict__ order, float4* __restrict__ pdj,
                                    double4* __restrict__ pdd) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= ns) return;
  const int i = order[t];
  const double* d = r + 3 * (long)ns + 3 * i;
  if (pdj) pdj[t] = make_float4((float)d[0], (float)d[1], (float)d[2], 0.f);
  if (pdd) pdd[t] = make_double4(d[0], d[1], d[2], 0.0);
}

cudaError_t k_gather_drude(const Launch& L, int ns, const double* r, const int* order,
                           float4* pdj, double4* pdd) {
  gather_drude_kernel<<<cdiv(ns, 256), 256, 0, L.s>>>(ns, r, order, pdj, pdd);
  LAUNCHED(L);
  return cudaGetLastError();
}

// --------------------------------------------------------------- k-space --

// Row of charge j: [q e^{2 pi i kx sx}, kx=0..Kx | e^{2 pi i ky sy}, ky=-Ky..Ky |
//                   e^{2 pi i kz sz}, kz=-Kz..Kz]
// f += fk (the k-space forces of the concurrent chain)
__global__ void add_forces_kernel(size_t n, const double* __restrict__ fk, double* __restrict__ f) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) f[i] += fk[i];
}

cudaError_t k_add_forces(const Launch& L, size_t n, const double* fk, double* f) {
  add_forces_kernel<<<(unsigned)((n + 255) / 256), 256, 0, L.s>>>(n, fk, f);
  LAUNCHED(L);
  return cudaGetLastError();
}

// fixed-point coordinates of every charge (Drude charges at r + rpol)
MG_BODY void charge_fixed_kernel_body(const KArgs& a,
    const double* __restrict__ r,
    uint4* __restrict__ qf,
    const int bx_,
    const int by_) {
  const int j = bx_ * blockDim.x + threadIdx.x;
  if (j >= a.nq) return;
  const int site = a.qsite[j];
  double x = r[3 * site], y = r[3 * site + 1], z = r[3 * site + 2];
  if (a.qdrude && a.qdrude[j]) {
    x += r[3 * (long)a.ns + 3 * site];
    y += r[3 * (long)a.ns + 3 * site + 1];
    z += r[3 * (long)a.ns + 3 * site + 2];
  }
  qf[j] = make_uint4((unsigned)fixed32(x, a.iLx), (unsigned)fixed32(y, a.iLy),
                     (unsigned)fixed32(z, a.iLz), 0u);
}

__global__ void charge_fixed_kernel(const __grid_constant__ KArgs a, const double* __restrict__ r, uint4* __restrict__ qf) {
  charge_fixed_kernel_body(a, r, qf, blockIdx.x, 0);
}

MG_BODY void phase_tables_mixed_kernel_body(const KArgs& a,
    const uint4* __restrict__ qf,
    float2* __restrict__ tab,
    const int bx_,
    const int by_) {
  long t = (long)bx_ * blockDim.x + threadIdx.x;
  if (t >= (long)a.nq * a.row) return;
  int j = (int)(t / a.row), e = (int)(t % a.row);
  int d, n;
  if (e <= a.Kx) { d = 0; n = e; }
  else if (e <= a.Kx + 2 * a.Ky + 1) { d = 1; n = e - (a.Kx + 1) - a.Ky; }
  else { d = 2; n = e - (a.Kx + 2 * a.Ky + 2); }   // Z(0..Kz) only
  const uint4 S4 = qf[j];
  const unsigned S = d == 0 ? S4.x : (d == 1 ? S4.y : S4.z);
  // exact integer phase n*s mod 1 in units of 2^-32
  int ph = (int)(S * (unsigned int)n);
  float tt = (float)ph * 2.3283064365386963e-10f;   // in [-0.5, 0.5)
  float sn, cs;
  sincospif(2.f * tt, &sn, &cs);
  if (d == 0) {
    float q = (float)a.qval[j];
    cs *= q;
    sn *= q;
  }
  tab[t] = make_float2(cs, sn);
}

__global__ void phase_tables_mixed_kernel(const __grid_constant__ KArgs a, const uint4* __restrict__ qf, float2* __restrict__ tab) {
  phase_tables_mixed_kernel_body(a, qf, tab, blockIdx.x, 0);
}

__global__ void phase_tables_fp64_kernel(KArgs a, const double* __restrict__ r,
                                         double2* __restrict__ tab) {
  long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long)a.nq * a.row) return;
  int j = (int)(t / a.row), e = (int)(t % a.row);
  int site = a.qsite[j];
  int d, n;
  if (e <= a.Kx) { d = 0; n = e; }
  else if (e <= a.Kx + 2 * a.Ky + 1) { d = 1; n = e - (a.Kx + 1) - a.Ky; }
  else { d = 2; n = e - (a.Kx + 2 * a.Ky + 2) - a.Kz; }
  double Lb = d == 0 ? a.Lx : (d == 1 ? a.Ly : a.Lz);
  double xd = r[3 * site + d];
  if (a.qdrude && a.qdrude[j]) xd += r[3 * (long)a.ns + 3 * site + d];
  double s = xd / Lb;
  double ph = n * s;
  ph -= rint(ph);
  double sn, cs;
  sincospi(2.0 * ph, &sn, &cs);
  if (d == 0) {
    cs *= a.qval[j];
    sn *= a.qval[j];
  }
  tab[t] = make_double2(cs, sn);
}

cudaError_t k_phase_tables_mixed(const Launch& L, const KArgs& a, const double* r, float2* tab,
                                 uint4* qf) {
  charge_fixed_kernel<<<cdiv(a.nq, 256), 256, 0, L.s>>>(a, r, qf);
  LAUNCHED(L);
  long n = (long)a.nq * a.row;
  phase_tables_mixed_kernel<<<(int)((n + 255) / 256), 256, 0, L.s>>>(a, qf, tab);
  LAUNCHED(L);
  return cudaGetLastError();
}
cudaError_t k_phase_tables_fp64(const Launch& L, const KArgs& a, const double* r, double2* tab) {
  long n = (long)a.nq * a.row;
  phase_tables_fp64_kernel<<<(int)((n + 255) / 256), 256, 0, L.s>>>(a, r, tab);
  LAUNCHED(L);
  return cudaGetLastError();
}

// S(k) = sum over chunks (FP64, fixed order); energy and virial per k
// (sim/ewpass2m.c: E1 = |S|^2 ekk, ptf = 1/kk + (pi/alpha)^2) reduced per block
MG_BODY void sk_reduce_kernel_body(const KArgs& a,
    const float2* __restrict__ part,
    bool measure,
    double pi2_over_a2,
    const int bx_,
    const int by_) {
  __shared__ double red[256][7];
  const int k = bx_ * 256 + threadIdx.x;
  double e[7] = {0, 0, 0, 0, 0, 0, 0};
  if (k < a.nk) {
    double sr = 0, si = 0;
    for (int c = 0; c < a.nchunk; c++) {
      const float2 v = part[(long)c * a.nk + k];
      sr += v.x;
      si += v.y;
    }
    a.S[2 * k] = sr;
    a.S[2 * k + 1] = si;
    const double ek = a.ekk[k];
    if (a.Wf) a.Wf[k] = make_float2((float)(ek * sr), (float)(-ek * si));
    if (measure) {
      const int4 kv = a.kvec[k];
      const double kx = kv.x / a.Lx, ky = kv.y / a.Ly, kz = kv.z / a.Lz;
      const double kk = kx * kx + ky * ky + kz * kz;
      const double E1 = (sr * sr + si * si) * a.ekk[k];
      const double ptf = 1 / kk + pi2_over_a2;
      e[0] = E1;
      e[1] = E1 * ptf * kx * kx;
      e[2] = E1 * ptf * ky * ky;
      e[3] = E1 * ptf * kz * kz;
      e[4] = E1 * ptf * ky * kz;
      e[5] = E1 * ptf * kx * kz;
      e[6] = E1 * ptf * kx * ky;
    }
  }
  if (!measure) return;
  for (int m = 0; m < 7; m++) red[threadIdx.x][m] = e[m];
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if (threadIdx.x < w)
      for (int m = 0; m < 7; m++) red[threadIdx.x][m] += red[threadIdx.x + w][m];
    __syncthreads();
  }
  if (threadIdx.x == 0)
    for (int m = 0; m < 7; m++) a.ek_part[bx_ * 7 + m] = red[0][m];
}

__global__ void sk_reduce_kernel(const __grid_constant__ KArgs a, const float2* __restrict__ part, bool measure, double pi2_over_a2) {
  sk_reduce_kernel_body(a, part, measure, pi2_over_a2, blockIdx.x, 0);
}

cudaError_t k_sk_reduce_mixed(const Launch& L, const KArgs& a, const float2* part, bool measure) {
  const double pa = 9.869604401089358 / (a.alpha * a.alpha);
  sk_reduce_kernel<<<cdiv(a.nk, 256), 256, 0, L.s>>>(a, part, measure, pa);
  LAUNCHED(L);
  return cudaGetLastError();
}
// out[k] = sum over rows of part[row*width+k], in a fixed order (one CTA): the
// warps share the columns, several warps a column where there are fewer
// columns than warps; lanes take rows in turn; the two tables of a phase in one
// launch.  (One column after the other with a CTA-wide tree each, a launch per
// table: 13 us a launch on 864 waters; this 6.8 us for both.)
constexpr int RED_THREADS = 512;
MG_BODY void reduce_rows_kernel_body(const double* __restrict__ part,
    int nrows,
    int width,
    double* __restrict__ out,
    const int bx_,
    const int by_) {
  constexpr int NW = RED_THREADS / 32;
  __shared__ double red[NW];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int k0 = 0; k0 < width; k0 += NW) {
    const int nc = min(NW, width - k0), ns = NW / nc;   // columns, warps a column
    const int c = warp % nc, sh = warp / nc;
    double v = 0;
    if (sh < ns) {
      const int step = 32 * ns;
#pragma unroll 8
      for (int r = 32 * sh + lane; r < nrows; r += step) v += part[(long)r * width + k0 + c];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) red[warp] = v;
    __syncthreads();
    if (threadIdx.x < nc) {
      double t = 0;
      for (int q = 0; q < ns; q++) t += red[q * nc + threadIdx.x];
      out[k0 + threadIdx.x] = t;
    }
    __syncthreads();
  }
}

// up to two tables in a launch, one CTA each
struct RedTab {
  const double* part;
  int nrows, width;
  double* out;
};
__global__ void __launch_bounds__(RED_THREADS) reduce_rows_kernel(const __grid_constant__ RedTab a,
                                                                  const __grid_constant__ RedTab b) {
  after_previous();
  if (blockIdx.x == 0) reduce_rows_kernel_body(a.part, a.nrows, a.width, a.out, 0, 0);
  else reduce_rows_kernel_body(b.part, b.nrows, b.width, b.out, 0, 0);
}

cudaError_t k_reduce_sum(const Launch& L, const double* part, int nrows, int width, double* out) {
  const RedTab a{part, nrows, width, out};
  launch_after(L, reduce_rows_kernel, 1, RED_THREADS, 0, a, a);
  LAUNCHED(L);
  return cudaGetLastError();
}
cudaError_t k_reduce_two(const Launch& L, const double* pa, int ra, int wa, double* oa,
                         const double* pb, int rb, int wb, double* ob) {
  launch_after(L, reduce_rows_kernel, 2, RED_THREADS, 0, RedTab{pa, ra, wa, oa},
               RedTab{pb, rb, wb, ob});
  LAUNCHED(L);
  return cudaGetLastError();
}

// -------------------------------------------------------------- SHAKE --

// sim/constrd.c:767-839 + sim/verlet.c:101-104 + sim/shakev3.c (SHAKE=1,
// VERLET=3; Nose-Hoover's friction term of sim/verlet.c:22-37 when the
// thermostat state is given), one thread per molecule, FP64.  The new
// positions are then wrapped as cook's normalize(-1) does after the step
// (sim/norm.c:415-444): the molecule's lowest coordinate over its massive
// sites decides a shift of +L (below r0), -L (at or above r0 + L) or none.
constexpr int SH_THREADS = SHAKE_THREADS;
int shake_blocks(int nmol) { return cdiv(nmol, SHAKE_THREADS); }

__device__ __forceinline__ double wrap_shift(double lo, double r0, double L) {
  return lo < r0 ? L : (lo >= r0 + L ? -L : 0.0);
}

// three-site, three-constraint molecules (rigid water) with the positions in
// registers: the same sweeps in the same order as the general path below
// (which works on the global array p), 15 FP64 operations per constraint
// and sweep: the per-constraint factors m^-1 omega/(m_i^-1 + m_j^-1)/d^2 and
// the tolerance eps d^2 are formed once per call (FP64 divisions and
// multiplications are slow on this GPU's narrow FP64 pipe).
__device__ __forceinline__ double3 sh_get(int k, const double3& a, const double3& b,
                                          const double3& c) {
  return k == 0 ? a : (k == 1 ? b : c);
}
__device__ __forceinline__ void sh_add(int k, double3& a, double3& b, double3& c, double s,
                                       double x, double y, double z) {
  if (k == 0) { a.x += s * x; a.y += s * y; a.z += s * z; }
  else if (k == 1) { b.x += s * x; b.y += s * y; b.z += s * z; }
  else { c.x += s * x; c.y += s * y; c.z += s * z; }
}

// Nose-Hoover with Verlet + SHAKE (cook's T_NOSE): the time-reversible
// velocity predictor of length k (sim/trvpscale.c:31-57; J. Chem. Theory
// Comput. 7, 3596 (2011)), b_0 = (2k+1)/(k+1), b_{j+1} = -b_j (k-j)/(k+j+2),
// predicts h v(t) = sum_j b_j r1(t - j h) for every degree of freedom and
// Vfactor = h dlogs/dt from the history of logs; the step then adds
// -Vfactor vpred to h^2 f/m (sim/verlet.c:22-37).  k grows by one per step
// up to the predictor length.
struct NoseStep {
  double b[MG_NOSE_MAXPRED + 1];
  double vf;
  int k, knew;
};

__device__ __forceinline__ NoseStep nose_begin(const ShakeArgs& a) {
  NoseStep q;
  q.k = (int)a.nh[NH_K];
  q.knew = min(a.nh_pred, q.k + 1);
  q.b[0] = (double)(2 * q.k + 1) / (q.k + 1);
  for (int j = 0; j < q.k; j++) q.b[j + 1] = -q.b[j] * (double)(q.k - j) / (q.k + j + 2);
  q.vf = 0;
  q.vf += q.b[0] * a.nh[NH_LOGSV];
  for (int j = 1; j <= q.k; j++) q.vf += q.b[j] * a.nh[NH_HIST + j - 1];
  return q;
}

// the friction displacement of degree of freedom t (r1 = its r1(t)); the
// history moves one slot back and takes r1
__device__ __forceinline__ double nose_dof(const ShakeArgs& a, const NoseStep& q, long long t,
                                           double r1) {
  double v = 0;
  v += q.b[0] * r1;
  for (int j = 1; j <= q.k; j++) v += q.b[j] * a.vhist[(j - 1) * a.nstride + t];
  for (int j = q.knew - 1; j >= 1; j--) a.vhist[j * a.nstride + t] = a.vhist[(j - 1) * a.nstride + t];
  if (q.knew > 0) a.vhist[t] = r1;
  return -q.vf * v;
}

// the measured quantities of a SHAKE step (MEAS): cook's En.virc and
// PTvirc (sim/virc.c, summed over the sweeps before the division by h^2 of
// sim/constrd.c:1038-1040) and the VERLET=3 kinetic tensor sum
// m (V1 V1 + V2 V2) of sim/shakev3.c:20-32 (before hscale), per molecule
struct ShakeMeas {
  double virc, pt[6], pk[6];
};
__device__ __forceinline__ void meas_zero(ShakeMeas& m) {
  m.virc = 0;
#pragma unroll
  for (int k = 0; k < 6; k++) m.pt[k] = m.pk[k] = 0;
}
// constraint virial of one constraint: virc += sq, PTvirc += (sq/bondq) rij rij
// (xx yy zz yz zx xy); sq = the sweep sum of (bondq - |pij|^2) omega/(mi+mj)
__device__ __forceinline__ void meas_cons(ShakeMeas& m, double sq, double sqb, double x, double y,
                                          double z) {
  m.virc += sq;
  m.pt[0] += sqb * (x * x);
  m.pt[1] += sqb * (y * y);
  m.pt[2] += sqb * (z * z);
  m.pt[3] += sqb * (y * z);
  m.pt[4] += sqb * (z * x);
  m.pt[5] += sqb * (x * y);
}
__device__ __forceinline__ void meas_kin(ShakeMeas& m, double mi, double v1x, double v1y,
                                         double v1z, double v2x, double v2y, double v2z) {
  m.pk[0] += (v1x * v1x + v2x * v2x) * mi;
  m.pk[1] += (v1y * v1y + v2y * v2y) * mi;
  m.pk[2] += (v1z * v1z + v2z * v2z) * mi;
  m.pk[3] += (v1y * v1z + v2y * v2z) * mi;
  m.pk[4] += (v1z * v1x + v2z * v2x) * mi;
  m.pk[5] += (v1x * v1y + v2x * v2y) * mi;
}

// ---- float-float SHAKE sweeps (mixed path, three-site molecules) ----
//
// The sweeps of the three-site path in float-float arithmetic: every site's
// position relative to the molecule's first site as hi + lo floats (about
// 48 bits), the bond vector and its squared length to about 1e-14 A^2, the
// deviation d then rounded to float (it only scales the displacements and
// meets the tolerance test).  The FP64 sweeps run on GB300's narrow FP64
// pipe; these run on the FP32 pipe.  Every rounding is explicit (`_rn`), so
// the measuring and the plain instantiation sweep identically.

__device__ __forceinline__ void ff_two_sum(float a, float b, float& s, float& e) {
  s = __fadd_rn(a, b);
  const float bb = __fadd_rn(s, -a);
  e = __fadd_rn(__fadd_rn(a, -__fadd_rn(s, -bb)), __fadd_rn(b, -bb));
}
__device__ __forceinline__ float ff_sel(int k, const float (&v)[3]) {
  return k == 0 ? v[0] : (k == 1 ? v[1] : v[2]);
}
// (h, l) of site k += v: the hi sum's rounding error goes into lo exactly
__device__ __forceinline__ void ff_add(int k, float (&h)[3], float (&l)[3], float v) {
#pragma unroll
  for (int s = 0; s < 3; s++)
    if (s == k) {
      float t, e;
      ff_two_sum(h[s], v, t, e);
      h[s] = t;
      l[s] = __fadd_rn(l[s], e);
    }
}
// component of p_i - p_j: (hi, lo), not renormalised
__device__ __forceinline__ void ff_diff(int i, int j, const float (&h)[3], const float (&l)[3],
                                        float& dh, float& dl) {
  float e;
  ff_two_sum(ff_sel(i, h), -ff_sel(j, h), dh, e);
  dl = __fadd_rn(e, __fadd_rn(ff_sel(i, l), -ff_sel(j, l)));
}

// the SHAKE sweeps of cook (sim/constrd.c:821-839) on the three sites P
// (updated in place); returns true if the tolerance was not met in maxit
// sweeps; dsum: the deviations summed per constraint (measured steps)
template <bool MEAS>
__device__ __forceinline__ bool shake3_ff(double3 (&P)[3], const int (&ci)[3], const int (&cj)[3],
                                          const float4* __restrict__ ftab,
                                          const double (&rx)[3], const double (&ry)[3],
                                          const double (&rz)[3], int maxit,
                                          double (&dsum)[3]) {
  const double3 o = P[0];
  float hx[3], hy[3], hz[3], lx[3], ly[3], lz[3];
  hx[0] = hy[0] = hz[0] = lx[0] = ly[0] = lz[0] = 0.f;
#pragma unroll
  for (int s = 1; s < 3; s++) {
    const double ux = P[s].x - o.x, uy = P[s].y - o.y, uz = P[s].z - o.z;
    hx[s] = __double2float_rn(ux);
    hy[s] = __double2float_rn(uy);
    hz[s] = __double2float_rn(uz);
    lx[s] = __double2float_rn(ux - (double)hx[s]);
    ly[s] = __double2float_rn(uy - (double)hy[s]);
    lz[s] = __double2float_rn(uz - (double)hz[s]);
  }
  float bqh[3], bql[3], tf[3], wi[3], wj[3], qx[3], qy[3], qz[3];
#pragma unroll
  for (int q = 0; q < 3; q++) {
    const float4 u = __ldg(ftab + 2 * q), v = __ldg(ftab + 2 * q + 1);
    bqh[q] = u.x;
    bql[q] = u.y;
    tf[q] = u.z;
    wi[q] = u.w;
    wj[q] = v.x;
    qx[q] = __double2float_rn(rx[q]);
    qy[q] = __double2float_rn(ry[q]);
    qz[q] = __double2float_rn(rz[q]);
  }
  int it = 0;
  bool over;
  do {
    it++;
    over = false;
#pragma unroll
    for (int q = 0; q < 3; q++) {
      const int i = ci[q], j = cj[q];
      float xh, xl, yh, yl, zh, zl;
      ff_diff(i, j, hx, lx, xh, xl);
      ff_diff(i, j, hy, ly, yh, yl);
      ff_diff(i, j, hz, lz, zh, zl);
      // squares: hi^2 exactly as p + e, plus 2 hi lo
      const float px = __fmul_rn(xh, xh), py = __fmul_rn(yh, yh), pz = __fmul_rn(zh, zh);
      const float ex = __fmaf_rn(__fmul_rn(2.f, xh), xl, __fmaf_rn(xh, xh, -px)),
                  ey = __fmaf_rn(__fmul_rn(2.f, yh), yl, __fmaf_rn(yh, yh, -py)),
                  ez = __fmaf_rn(__fmul_rn(2.f, zh), zl, __fmaf_rn(zh, zh, -pz));
      float s1, e1, s2, e2;
      ff_two_sum(px, py, s1, e1);
      ff_two_sum(s1, pz, s2, e2);
      const float E = __fadd_rn(__fadd_rn(__fadd_rn(e1, e2), __fadd_rn(ex, ey)), ez);
      // d = bq - |p_i - p_j|^2
      float t, te;
      ff_two_sum(bqh[q], -s2, t, te);
      const float d = __fadd_rn(t, __fadd_rn(te, __fadd_rn(bql[q], -E)));
      over |= fabsf(d) > tf[q];
      if constexpr (MEAS) dsum[q] += (double)d;
      const float gi = __fmul_rn(d, wi[q]), gj = __fmul_rn(d, wj[q]);
      ff_add(i, hx, lx, __fmul_rn(gi, qx[q]));
      ff_add(i, hy, ly, __fmul_rn(gi, qy[q]));
      ff_add(i, hz, lz, __fmul_rn(gi, qz[q]));
      ff_add(j, hx, lx, __fmul_rn(gj, qx[q]));
      ff_add(j, hy, ly, __fmul_rn(gj, qy[q]));
      ff_add(j, hz, lz, __fmul_rn(gj, qz[q]));
    }
  } while (over && it < maxit);
#pragma unroll
  for (int s = 0; s < 3; s++)
    P[s] = make_double3(o.x + ((double)hx[s] + (double)lx[s]), o.y + ((double)hy[s] + (double)ly[s]),
                        o.z + ((double)hz[s] + (double)lz[s]));
  return over;
}

// the sweeps on the three sites P at the displacements' directions r_ij of the
// old positions R, constraint order (ci, cj); true if they did not converge
template <bool MEAS, bool DF>
__device__ __forceinline__ bool shake3(const ShakeArgs& a, const bool df, int c0,
                                       const int (&ci)[3], const int (&cj)[3],
                                       const double3 (&R)[3], double3 (&P)[3], ShakeMeas& ms) {
  double rx[3], ry[3], rz[3];
  double dsum[3] = {0, 0, 0};
#pragma unroll
  for (int q = 0; q < 3; q++) {
    const double3 ri = sh_get(ci[q], R[0], R[1], R[2]), rj = sh_get(cj[q], R[0], R[1], R[2]);
    rx[q] = ri.x - rj.x;
    ry[q] = ri.y - rj.y;
    rz[q] = ri.z - rj.z;
  }
  const double* t = a.ctab + 6 * (long)c0;
  bool over = false;
  if (DF && df) {
    over = shake3_ff<MEAS>(P, ci, cj, a.ftab + 2 * (long)c0, rx, ry, rz, a.maxit, dsum);
  } else {
    double bq[3], tol[3], awi[3], awj[3];
#pragma unroll
    for (int q = 0; q < 3; q++) {
      bq[q] = t[6 * q];
      tol[q] = t[6 * q + 1];
      awi[q] = t[6 * q + 2];
      awj[q] = t[6 * q + 3];
    }
    int it = 0;
    do {
      it++;
      over = false;
#pragma unroll
      for (int q = 0; q < 3; q++) {
        const double3 pi = sh_get(ci[q], P[0], P[1], P[2]), pj = sh_get(cj[q], P[0], P[1], P[2]);
        const double px = pi.x - pj.x, py = pi.y - pj.y, pz = pi.z - pj.z;
        const double d = bq[q] - (px * px + py * py + pz * pz);
        over |= fabs(d) > tol[q];
        if constexpr (MEAS) dsum[q] += d;
        sh_add(ci[q], P[0], P[1], P[2], d * awi[q], rx[q], ry[q], rz[q]);
        sh_add(cj[q], P[0], P[1], P[2], d * awj[q], rx[q], ry[q], rz[q]);
      }
    } while (over && it < a.maxit);
  }
  if constexpr (MEAS) {
#pragma unroll
    for (int q = 0; q < 3; q++)
      meas_cons(ms, dsum[q] * t[6 * q + 4], dsum[q] * t[6 * q + 5], rx[q], ry[q], rz[q]);
  }
  return over;
}

// A warp per CTA: a molecule's set-up and sweeps are one chain, so what counts
// is how many SMs share the work (and their narrow FP64 pipes).  Molecules with
// three constraints over their first three sites (rigid water; TIP4P with its
// massless site behind) keep the sites in registers; where the constraints are
// (0,1), (0,2), (1,2) the indices are compile-time constants and a sweep needs
// no selection.  The per-constraint factors come from a table (formed per call
// they cost six FP64 divisions a molecule).  Measured, float-float sweeps: 864
// waters 43 -> 13.7 us, 32768 waters 55 -> 21 us.
template <bool NOSE, bool MEAS, bool DF>
MG_BODY void shake_kernel_body(const ShakeArgs& a,
    const int bx_,
    const int by_) {
  static_assert(SHAKE_THREADS == 32, "one warp per CTA");
  const int n = bx_ * SHAKE_THREADS + threadIdx.x;
  double kin = 0;
  ShakeMeas ms;
  if constexpr (MEAS) meas_zero(ms);
  [[maybe_unused]] NoseStep nose;
  if constexpr (NOSE) nose = nose_begin(a);
  if (n < a.nmol) {
    const int i0 = a.mol_first[n], i1 = a.mol_first[n + 1];
    const int c0 = a.mol_cfirst[n], c1 = a.mol_cfirst[n + 1];
    // 1: the constraints are (0,1), (0,2), (1,2); 2: others over the first
    // three sites; 0: anything else
    const int kind = a.kind3[n];
    if (kind) {
      double3 P[3], R[3], V[3];
#pragma unroll
      for (int s = 0; s < 3; s++) {
        const int i = i0 + s;
        R[s] = make_double3(a.r[3 * i], a.r[3 * i + 1], a.r[3 * i + 2]);
        V[s] = make_double3(a.r1[3 * i], a.r1[3 * i + 1], a.r1[3 * i + 2]);
        const double hm = a.hh * a.imass[i];
        if constexpr (NOSE) {
          const double dx = nose_dof(a, nose, 3 * i, V[s].x);
          const double dy = nose_dof(a, nose, 3 * i + 1, V[s].y);
          const double dz = nose_dof(a, nose, 3 * i + 2, V[s].z);
          P[s] = make_double3(a.f[3 * i] * hm + dx + R[s].x + V[s].x,
                              a.f[3 * i + 1] * hm + dy + R[s].y + V[s].y,
                              a.f[3 * i + 2] * hm + dz + R[s].z + V[s].z);
        } else {
          P[s] = make_double3(a.f[3 * i] * hm + R[s].x + V[s].x,
                              a.f[3 * i + 1] * hm + R[s].y + V[s].y,
                              a.f[3 * i + 2] * hm + R[s].z + V[s].z);
        }
      }
      // float-float sweeps for molecules of exactly three sites
      const bool df = i1 - i0 == 3;
      bool over;
      if (kind == 1) {
        const int ci[3] = {0, 0, 1}, cj[3] = {1, 2, 2};
        over = shake3<MEAS, DF>(a, df, c0, ci, cj, R, P, ms);
      } else {
        int ci[3], cj[3];
#pragma unroll
        for (int q = 0; q < 3; q++) {
          const int2 ij = a.cons[c0 + q];
          ci[q] = ij.x - i0;
          cj[q] = ij.y - i0;
        }
        over = shake3<MEAS, DF>(a, df, c0, ci, cj, R, P, ms);
      }
      if (over) atomicOr(a.status, 1);
      double sx = 0, sy = 0, sz = 0;
      if (a.normalize) {
        double lx = 9e9, ly = 9e9, lz = 9e9;
#pragma unroll
        for (int s = 0; s < 3; s++)
          if (a.mass[i0 + s] != 0) {
            lx = fmin(lx, P[s].x);
            ly = fmin(ly, P[s].y);
            lz = fmin(lz, P[s].z);
          }
        sx = wrap_shift(lx, a.r0, a.Lb[0]);
        sy = wrap_shift(ly, a.r0, a.Lb[1]);
        sz = wrap_shift(lz, a.r0, a.Lb[2]);
      }
#pragma unroll
      for (int s = 0; s < 3; s++) {
        const int i = i0 + s;
        const double v1x = V[s].x, v1y = V[s].y, v1z = V[s].z;
        const double v2x = P[s].x - R[s].x, v2y = P[s].y - R[s].y, v2z = P[s].z - R[s].z;
        double v1s = 0, v2s = 0;
        v1s += v1x * v1x;
        v2s += v2x * v2x;
        v1s += v1y * v1y;
        v2s += v2y * v2y;
        v1s += v1z * v1z;
        v2s += v2z * v2z;
        kin += (v1s + v2s) * a.mass[i];
        if constexpr (MEAS) meas_kin(ms, a.mass[i], v1x, v1y, v1z, v2x, v2y, v2z);
        a.r1[3 * i] = v2x;
        a.r1[3 * i + 1] = v2y;
        a.r1[3 * i + 2] = v2z;
        a.r[3 * i] = P[s].x + sx;
        a.r[3 * i + 1] = P[s].y + sy;
        a.r[3 * i + 2] = P[s].z + sz;
      }
      // massless sites behind the three: moved along, placed by their parents
      for (int i = i0 + 3; i < i1; i++)
        for (int k = 0; k < 3; k++) {
          const double r = a.r[3 * i + k], v = a.r1[3 * i + k];
          double p = a.f[3 * i + k] * (a.hh * a.imass[i]);
          if constexpr (NOSE) p = p + nose_dof(a, nose, 3 * i + k, v);
          p = p + r + v;
          a.r1[3 * i + k] = p - r;
          a.r[3 * i + k] = p + (k == 0 ? sx : (k == 1 ? sy : sz));
        }
    } else {
    double* p = a.p;
    for (int i = i0; i < i1; i++)
      for (int k = 0; k < 3; k++)
        if constexpr (NOSE)
          p[3 * i + k] = a.f[3 * i + k] * (a.hh * a.imass[i]) +
                         nose_dof(a, nose, 3 * i + k, a.r1[3 * i + k]) + a.r[3 * i + k] +
                         a.r1[3 * i + k];
        else
          p[3 * i + k] = a.f[3 * i + k] * (a.hh * a.imass[i]) + a.r[3 * i + k] + a.r1[3 * i + k];
    if (c1 > c0) {
      int it = 0;
      double maxsq;
      do {
        it++;
        maxsq = 0;
        for (int al = c0; al < c1; al++) {
          const int2 ij = a.cons[al];
          const double bq = a.bondq[al];
          const double mi = a.imass[ij.x], mj = a.imass[ij.y];
          const double ibq = 1.0 / bq, wq = a.omega / (mi + mj) * ibq;
          double px = p[3 * ij.x] - p[3 * ij.y], py = p[3 * ij.x + 1] - p[3 * ij.y + 1],
                 pz = p[3 * ij.x + 2] - p[3 * ij.y + 2];
          const double d = bq - (px * px + py * py + pz * pz);
          maxsq = fmax(maxsq, fabs(d) * ibq);
          const double sq = d * wq;
          if constexpr (MEAS)
            meas_cons(ms, d * (a.omega / (mi + mj)), sq, a.r[3 * ij.x] - a.r[3 * ij.y],
                      a.r[3 * ij.x + 1] - a.r[3 * ij.y + 1], a.r[3 * ij.x + 2] - a.r[3 * ij.y + 2]);
          const double rx = (a.r[3 * ij.x] - a.r[3 * ij.y]) * sq,
                       ry = (a.r[3 * ij.x + 1] - a.r[3 * ij.y + 1]) * sq,
                       rz = (a.r[3 * ij.x + 2] - a.r[3 * ij.y + 2]) * sq;
          p[3 * ij.x] += mi * rx;
          p[3 * ij.x + 1] += mi * ry;
          p[3 * ij.x + 2] += mi * rz;
          p[3 * ij.y] -= mj * rx;
          p[3 * ij.y + 1] -= mj * ry;
          p[3 * ij.y + 2] -= mj * rz;
        }
      } while (maxsq > a.eps && it < a.maxit);
      if (maxsq > a.eps) atomicOr(a.status, 1);
    }
    double sh[3] = {0, 0, 0};
    if (a.normalize)
      for (int k = 0; k < 3; k++) {
        double lo = 9e9;
        for (int i = i0; i < i1; i++)
          if (a.mass[i] != 0) lo = fmin(lo, p[3 * i + k]);
        sh[k] = wrap_shift(lo, a.r0, a.Lb[k]);
      }
    for (int i = i0; i < i1; i++) {
      double v1s = 0, v2s = 0, v1[3], v2[3];
      for (int k = 0; k < 3; k++) {
        v1[k] = a.r1[3 * i + k];
        v2[k] = p[3 * i + k] - a.r[3 * i + k];
        v1s += v1[k] * v1[k];
        v2s += v2[k] * v2[k];
        a.r1[3 * i + k] = v2[k];
        a.r[3 * i + k] = p[3 * i + k] + sh[k];
      }
      kin += (v1s + v2s) * a.mass[i];
      if constexpr (MEAS) meas_kin(ms, a.mass[i], v1[0], v1[1], v1[2], v2[0], v2[1], v2[2]);
    }
    }
  }
  // the CTA's sums: a shuffle tree, in a fixed order
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) kin += __shfl_down_sync(0xffffffffu, kin, o);
  if (threadIdx.x == 0) a.kin_part[bx_] = kin;
  if constexpr (MEAS) {
    double v[13];
    v[0] = ms.virc;
#pragma unroll
    for (int k = 0; k < 6; k++) {
      v[1 + k] = ms.pt[k];
      v[7 + k] = ms.pk[k];
    }
#pragma unroll
    for (int k = 0; k < 13; k++) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_down_sync(0xffffffffu, v[k], o);
      if (threadIdx.x == 0) a.meas_part[(long)bx_ * 13 + k] = v[k];
    }
  }
}

template <bool NOSE, bool MEAS, bool DF>
__global__ void __launch_bounds__(SH_THREADS) shake_kernel(const __grid_constant__ ShakeArgs a) {
  after_previous();
  shake_kernel_body<NOSE, MEAS, DF>(a, blockIdx.x, 0);
}

cudaError_t k_shake(const Launch& L, const ShakeArgs& a) {
  const int nb = cdiv(a.nmol, SH_THREADS);
#define SHAKE_LAUNCH(DF)                                                  \
  do {                                                                    \
    if (a.vhist) {                                                        \
      if (a.meas_part)                                                    \
        launch_after(L, shake_kernel<true, true, DF>, nb, SH_THREADS, 0, a); \
      else                                                                \
        launch_after(L, shake_kernel<true, false, DF>, nb, SH_THREADS, 0, a); \
    } else {                                                              \
      if (a.meas_part)                                                    \
        launch_after(L, shake_kernel<false, true, DF>, nb, SH_THREADS, 0, a); \
      else                                                                \
        launch_after(L, shake_kernel<false, false, DF>, nb, SH_THREADS, 0, a); \
    }                                                                     \
  } while (0)
  if (a.ffsweep) SHAKE_LAUNCH(true);
  else SHAKE_LAUNCH(false);
#undef SHAKE_LAUNCH
  LAUNCHED(L);
  return cudaGetLastError();
}

// ---------------------------------------------------------- FP32 probe --

// 8 independent FMA chains per thread: the FP32 issue rate of the device
__global__ void fma_probe_kernel(int iters, float* __restrict__ out) {
  float x[8];
  const float a = 0.999999f, b = 1e-7f;
#pragma unroll
  for (int k = 0; k < 8; k++) x[k] = (float)(threadIdx.x + k);
  for (int i = 0; i < iters; i++) {
#pragma unroll
    for (int k = 0; k < 8; k++) x[k] = fmaf(x[k], a, b);
  }
  float s = 0;
#pragma unroll
  for (int k = 0; k < 8; k++) s += x[k];
  out[blockIdx.x * blockDim.x + threadIdx.x] = s;
}

cudaError_t k_fma_probe(cudaStream_t s, int blocks, int threads, int iters, float* out) {
  fma_probe_kernel<<<blocks, threads, 0, s>>>(iters, out);
  return cudaGetLastError();
}

}  // namespace mg

namespace mg {

// ------------------------------------------------------------ batches --
//
// The kernels of one MD step over every box of a batch, one launch each:
// blockIdx.y is the box, blockIdx.x the CTA of that box's own grid (the
// same CTAs, threads and arguments as the box's single launch, so every box
// gets its single-launch results bit for bit); CTAs beyond a box's grid
// return at once.

int cell_site_blocks(int ns) { return cdiv(ns, 256); }
int cell_order_blocks(int ncell) { return cdiv(ncell, ORDER_THREADS / 32); }
int pair_all_blocks(int ns) { return cdiv(ns, ALL_SITES); }

__global__ void batch_cell_count_kernel(const BoxStep* __restrict__ B) {
  const BoxStep& e = B[blockIdx.y];
  cell_count_kernel_body(e.ns, e.r, e.iL, e.ncx, e.ncy, e.ncz, e.kind, e.mol, e.pfix, e.key,
                         e.count, e.status, blockIdx.x);
}

__global__ void __launch_bounds__(SCAN_THREADS) batch_cell_scan_kernel(const BoxStep* __restrict__ B) {
  const BoxStep& e = B[blockIdx.y];
  cell_scan_kernel_body(e.ncx * e.ncy * e.ncz, e.count, e.start, e.cursor, e.gstart, 0, 0);
}

__global__ void batch_cell_scatter_kernel(const BoxStep* __restrict__ B) {
  const BoxStep& e = B[blockIdx.y];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= e.ns) return;
  e.slot_site[atomicAdd(e.cursor + e.key[i], 1)] = i;
}

__global__ void __launch_bounds__(ORDER_THREADS) batch_cell_order_kernel(const BoxStep* __restrict__ B) {
  const BoxStep& e = B[blockIdx.y];
  if ((int)blockIdx.x >= e.g_order) return;
  cell_order_kernel_body(e.ncx * e.ncy * e.ncz, e.start, e.slot_site, e.pfix, e.order, e.key_s,
                         e.pj, e.gstart, e.gcell, blockIdx.x, 0);
}

template <bool MEASURE>
__global__ void __launch_bounds__(GROUP_WARPS * 32, MEASURE ? 4 : 6)
    batch_pair_half_kernel(const BoxStep* __restrict__ B) {
  const BoxStep& e = B[blockIdx.y];
  if ((int)blockIdx.x >= e.g_half) return;
  pair_half_kernel_body<MEASURE, false, GROUP_WARPS>(e.pa, e.pj, e.ptab, e.erd, e.eru, e.sx, e.sy,
                                                     e.sz, e.cq, e.sg, blockIdx.x);
}

__global__ void batch_finish_kernel(const BoxStep* __restrict__ B) {
  const BoxStep& e = B[blockIdx.y];
  if (e.g_half > 0)
    finish_forces<false>(e.pa, e.pj, e.ptab, e.erd, e.sx, e.sy, e.sz, e.cq, e.sg);
}

template <bool MEASURE>
__global__ void __launch_bounds__(ALL_WARPS * 32, 2) batch_pair_all_kernel(const BoxStep* __restrict__ B) {
  const BoxStep& e = B[blockIdx.y];
  if ((int)blockIdx.x >= e.g_all) return;
  pair_all_kernel_body<MEASURE, false>(e.pa, e.pj, e.ptab, e.erd, e.eru, e.sx, e.sy, e.sz, e.cq,
                                       e.sg, blockIdx.x);
}

template <bool MEASURE>
__global__ void __launch_bounds__(EXCL_THREADS) batch_excl_kernel(const BoxStep* __restrict__ B) {
  const BoxStep& e = B[blockIdx.y];
  if ((int)blockIdx.x >= e.g_excl) return;
  excl_mixed_kernel_body<MEASURE, false>(e.xa, blockIdx.x, 0);
}

__global__ void batch_charge_fixed_kernel(const BoxStep* __restrict__ B) {
  const BoxStep& e = B[blockIdx.y];
  if ((int)blockIdx.x >= e.g_charge) return;
  charge_fixed_kernel_body(e.ka, e.r, e.qf, blockIdx.x, 0);
}

__global__ void batch_phase_kernel(const BoxStep* __restrict__ B) {
  const BoxStep& e = B[blockIdx.y];
  if ((int)blockIdx.x >= e.g_phase) return;
  phase_tables_mixed_kernel_body(e.ka, e.qf, e.tab, blockIdx.x, 0);
}

__global__ void batch_sk_reduce_kernel(const BoxStep* __restrict__ B, bool measure) {
  const BoxStep& e = B[blockIdx.y];
  if ((int)blockIdx.x >= e.g_skr) return;
  const double pa = 9.869604401089358 / (e.ka.alpha * e.ka.alpha);
  sk_reduce_kernel_body(e.ka, e.part, measure, pa, blockIdx.x, 0);
}

template <bool MEAS>
__global__ void __launch_bounds__(SH_THREADS) batch_shake_kernel(const BoxStep* __restrict__ B) {
  const BoxStep& e = B[blockIdx.y];
  if ((int)blockIdx.x >= e.g_shake) return;
  if (e.sa.ffsweep) shake_kernel_body<false, MEAS, true>(e.sa, blockIdx.x, 0);
  else shake_kernel_body<false, MEAS, false>(e.sa, blockIdx.x, 0);
}

// sums k0..k1-1 of every box (one CTA each)
__global__ void __launch_bounds__(RED_THREADS) batch_reduce_kernel(const BoxStep* __restrict__ B, int k0, int k1) {
  const BoxStep& e = B[blockIdx.y];
  for (int k = k0; k < k1; k++)
    reduce_rows_kernel_body(e.rpart[k], e.rrows[k], e.rwidth[k], e.rout[k], 0, 0);
}

__global__ void gather_status_kernel(const int* const* __restrict__ p, int n,
                                     int* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = *p[i];
}

cudaError_t k_gather_status(cudaStream_t s, const int* const* p, int n, int* out) {
  gather_status_kernel<<<cdiv(n, 256), 256, 0, s>>>(p, n, out);
  return cudaGetLastError();
}

cudaError_t k_batch_cells(const Launch& L, const BoxStep* d, int nbox, const BatchGrid& g) {
  batch_cell_count_kernel<<<dim3(g.site, nbox), 256, 0, L.s>>>(d);
  batch_cell_scan_kernel<<<dim3(1, nbox), SCAN_THREADS, 0, L.s>>>(d);
  batch_cell_scatter_kernel<<<dim3(g.site, nbox), 256, 0, L.s>>>(d);
  batch_cell_order_kernel<<<dim3(g.order, nbox), ORDER_THREADS, 0, L.s>>>(d);
  *L.counter += 4;
  return cudaGetLastError();
}

cudaError_t k_batch_pairs(const Launch& L, const BoxStep* d, int nbox, const BatchGrid& g,
                          bool measure) {
  cudaError_t e = cudaSuccess;
  // the boxes of the half-shell kernel, those of the all-pairs kernel, the
  // exclusions
#define BATCH_PAIRS(M)                                                                          \
  do {                                                                                          \
    if (g.half > 0 && g.pair_smem > 24 * 1024)                                                  \
      e = cudaFuncSetAttribute(batch_pair_half_kernel<M>,                                       \
                               cudaFuncAttributeMaxDynamicSharedMemorySize, (int)g.pair_smem);  \
    if (e == cudaSuccess && g.all > 0 && g.pair_smem > 24 * 1024)                               \
      e = cudaFuncSetAttribute(batch_pair_all_kernel<M>,                                        \
                               cudaFuncAttributeMaxDynamicSharedMemorySize, (int)g.pair_smem);  \
    if (e != cudaSuccess) return e;                                                             \
    if (g.half > 0) {                                                                           \
      batch_pair_half_kernel<M><<<dim3(g.half, nbox), GROUP_WARPS * 32, g.pair_smem, L.s>>>(d); \
      batch_finish_kernel<<<dim3(g.site, nbox), 256, 0, L.s>>>(d);                              \
    }                                                                                           \
    if (g.all > 0)                                                                              \
      batch_pair_all_kernel<M><<<dim3(g.all, nbox), ALL_WARPS * 32, g.pair_smem, L.s>>>(d);     \
    if (g.excl > 0) batch_excl_kernel<M><<<dim3(g.excl, nbox), EXCL_THREADS, 0, L.s>>>(d);      \
  } while (0)
  if (measure) BATCH_PAIRS(true);
  else BATCH_PAIRS(false);
#undef BATCH_PAIRS
  *L.counter += (g.half > 0 ? 2 : 0) + (g.all > 0 ? 1 : 0) + (g.excl > 0 ? 1 : 0);
  // the FP32-core phase rows (none when every box is on the tensor cores)
  if (g.charge > 0) {
    batch_charge_fixed_kernel<<<dim3(g.charge, nbox), 256, 0, L.s>>>(d);
    ++*L.counter;
  }
  if (g.phase > 0) {
    batch_phase_kernel<<<dim3(g.phase, nbox), 256, 0, L.s>>>(d);
    ++*L.counter;
  }
  return cudaGetLastError();
}

cudaError_t k_batch_sk_reduce(const Launch& L, const BoxStep* d, int nbox, const BatchGrid& g,
                              bool measure) {
  batch_sk_reduce_kernel<<<dim3(g.skr, nbox), 256, 0, L.s>>>(d, measure);
  LAUNCHED(L);
  return cudaGetLastError();
}

cudaError_t k_batch_step(const Launch& L, const BoxStep* d, int nbox, const BatchGrid& g,
                         bool measure) {
  if (measure) {
    // the energies of the force evaluation (rows 0, 1), the step, its sums (2, 3)
    batch_reduce_kernel<<<dim3(1, nbox), RED_THREADS, 0, L.s>>>(d, 0, 2);
    batch_shake_kernel<true><<<dim3(g.shake, nbox), SH_THREADS, 0, L.s>>>(d);
    batch_reduce_kernel<<<dim3(1, nbox), RED_THREADS, 0, L.s>>>(d, 2, 4);
    *L.counter += 3;
  } else {
    batch_shake_kernel<false><<<dim3(g.shake, nbox), SH_THREADS, 0, L.s>>>(d);
    LAUNCHED(L);
  }
  return cudaGetLastError();
}

}  // namespace mg
