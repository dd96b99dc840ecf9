// Widom test-particle insertions on the device (cook/widom.c:175-288 Einsert,
// sim/simmeas.c:1821-1958 Widom).
//
// One warp per insertion: the ghost's sites are placed from a counter-based
// stream (insertion k, word c: the SplitMix64 output function of
// seed + (8k+c+1)*gamma, Steele, Lea and Flood, OOPSLA 2014), each site's
// energy against the box is summed over the cell stencil of its home cell
// in the cell list of the last force evaluation (cook uses the last cell
// list the same way), and lane 0 adds exp(-U/T) (skipped when -U/T <= -700,
// sim/simmeas.c:1934) to the warp's sum.  Lanes take stencil cells (or, for
// grids of few cells, the sites of one cell).  Sums per CTA in FP64, in a
// fixed order, so the result does not depend on scheduling.  blockIdx.y
// selects the box: one launch serves a whole batch of boxes, each with its
// own cell list, pair table and ghost.
//
// Many insertions a cell (mixed precision) are sorted by place instead, 32
// neighbouring ghost sites to a warp (widom_sorted_kernel below).
#include <algorithm>

#include "mg_internal.h"

namespace mg {

constexpr int WD_THREADS = 128;
constexpr int WD_WARPS = WD_THREADS / 32;

__device__ __forceinline__ unsigned long long wd_word(unsigned long long seed, long long k, int c) {
  unsigned long long z = seed + (unsigned long long)(8 * k + c + 1) * 0x9E3779B97F4A7C15ULL;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
  return z ^ (z >> 31);
}

// uniform random rotation of Shoemake (Graphics Gems III, 1992) from words
// 3..5 of insertion k; identity for a one-site ghost
__device__ void wd_rotation(unsigned long long seed, long long k, int nps, double R[9]) {
  if (nps < 2) {
    R[0] = R[4] = R[8] = 1;
    R[1] = R[2] = R[3] = R[5] = R[6] = R[7] = 0;
    return;
  }
  const double s53 = 1.0 / 9007199254740992.0;
  const double u1 = (double)(wd_word(seed, k, 3) >> 11) * s53;
  const double u2 = (double)(wd_word(seed, k, 4) >> 11) * s53;
  const double u3 = (double)(wd_word(seed, k, 5) >> 11) * s53;
  const double a = sqrt(1 - u1), b = sqrt(u1);
  double s2, c2, s3, c3;
  sincospi(2 * u2, &s2, &c2);
  sincospi(2 * u3, &s3, &c3);
  const double x = a * s2, y = a * c2, z = b * s3, w = b * c3;
  R[0] = 1 - 2 * (y * y + z * z); R[1] = 2 * (x * y - z * w);     R[2] = 2 * (x * z + y * w);
  R[3] = 2 * (x * y + z * w);     R[4] = 1 - 2 * (x * x + z * z); R[5] = 2 * (y * z - x * w);
  R[6] = 2 * (x * z - y * w);     R[7] = 2 * (y * z + x * w);     R[8] = 1 - 2 * (x * x + y * y);
}

__device__ __forceinline__ int wd_wrap(int c, int n) { return c < 0 ? c + n : (c >= n ? c - n : c); }

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// the end of the kernel: per-warp Boltzmann sums into one FP64 value per CTA
__device__ __forceinline__ void wd_block_sum(double wacc, double* part) {
  __shared__ double ws[WD_WARPS];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) ws[warp] = wacc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0;
    for (int w = 0; w < WD_WARPS; w++) s += ws[w];
    part[blockIdx.x] = s;
  }
}

// mixed path: fixed-point ghost sites, FP32 pair energies, FP64 sums per cell
__global__ void __launch_bounds__(WD_THREADS) widom_mixed_kernel(const WidomBox* __restrict__ boxes) {
  __shared__ PairF tab[MAX_WPROBE * MAX_KINDS];
  const WidomBox& B = boxes[blockIdx.y];
  const WidomArgs a = B.a;
  const int4* __restrict__ pj = B.pj;
  const float4* __restrict__ eru = B.eru;
  for (int t = threadIdx.x; t < a.nps * a.nkind; t += WD_THREADS) tab[t] = B.tabf[t];
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const long long nw = (long long)gridDim.x * WD_WARPS;
  const float sx = (float)(a.Lx * 2.3283064365386963e-10), sy = (float)(a.Ly * 2.3283064365386963e-10),
              sz = (float)(a.Lz * 2.3283064365386963e-10);
  const float cq = (float)a.cutoff_sq, sgrid = (float)a.sgrid;
  double wacc = 0;
  for (long long k = blockIdx.x * (long long)WD_WARPS + (threadIdx.x >> 5); k < a.n; k += nw) {
    double R[9];
    wd_rotation(a.seed, k, a.nps, R);
    const unsigned px = (unsigned)(wd_word(a.seed, k, 0) >> 32),
                   py = (unsigned)(wd_word(a.seed, k, 1) >> 32),
                   pz = (unsigned)(wd_word(a.seed, k, 2) >> 32);
    double U = 0;
    for (int s = 0; s < a.nps; s++) {
      const double g0 = a.geom[3 * s], g1 = a.geom[3 * s + 1], g2 = a.geom[3 * s + 2];
      // site = point + R g, as 32-bit fractions of the box (wrap-around)
      const unsigned ux = px + (unsigned)(int)llrint((R[0] * g0 + R[1] * g1 + R[2] * g2) / a.Lx * 4294967296.0);
      const unsigned uy = py + (unsigned)(int)llrint((R[3] * g0 + R[4] * g1 + R[5] * g2) / a.Ly * 4294967296.0);
      const unsigned uz = pz + (unsigned)(int)llrint((R[6] * g0 + R[7] * g1 + R[8] * g2) / a.Lz * 4294967296.0);
      const int cx = (int)(((unsigned long long)ux * a.ncx) >> 32),
                cy = (int)(((unsigned long long)uy * a.ncy) >> 32),
                cz = (int)(((unsigned long long)uz * a.ncz) >> 32);
      const PairF* T = tab + s * a.nkind;
      const int s0 = a.lanes_sites ? 0 : lane, ds = a.lanes_sites ? 1 : 32;
      for (int st = s0; st < a.nstencil; st += ds) {
        const int4 o = a.stencil[st];
        const int c2 = (wd_wrap(cx + o.x, a.ncx) * a.ncy + wd_wrap(cy + o.y, a.ncy)) * a.ncz +
                       wd_wrap(cz + o.z, a.ncz);
        const int j0 = a.cell_start[c2], j1 = a.cell_start[c2 + 1];
        float u = 0;
        for (int j = j0 + (a.lanes_sites ? lane : 0); j < j1; j += a.lanes_sites ? 32 : 1) {
          const int4 q = pj[j];
          const float dx = (float)(int)(ux - (unsigned)q.x) * sx;
          const float dy = (float)(int)(uy - (unsigned)q.y) * sy;
          const float dz = (float)(int)(uz - (unsigned)q.z) * sz;
          const float rr = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
          if (rr >= cq) continue;
          const PairF P = T[q.w & 255];
          if (rr < P.C2q) {
            if (rr < P.C1q) {
              const float x = P.Sq / rr, y = x * x * x;
              u += P.E4 * fmaf(y, y, -y);
            } else {
              const float x = rr - P.C2q;
              u += P.A * x * x;
            }
          }
          if (P.qq != 0.f) {
            const float4 e = __ldg(eru + min((int)(rr * sgrid), a.ntab - 1));
            u += (__fdividef(e.y, e.z + rr) + e.x) * P.qq;
          }
        }
        U += u;
      }
    }
    U = warp_sum(U);
    if (lane == 0) {
      if (a.U) a.U[k] = U;
      const double e = -U / a.T;
      if (e > -700) wacc += exp(e);
    }
  }
  wd_block_sum(wacc, a.part);
}

// ---- mixed path, sorted by place ------------------------------------------
//
// A warp per insertion repeats the ghost's FP64 set-up (three divisions, the
// Boltzmann factor) in all lanes and fills its lanes with the few sites of
// single cells: 5.9 ns an insertion into ionic boxes of 500 to 4000 sites
// (28.3 ms for 48 boxes of 100000); this 0.4 ns (1.9 ms, of which the sorted
// kernel, bound by its instruction issue at 88 %, takes 1.56).
// Here the set-up is done once, a thread per insertion, and the ghost sites
// are counting-sorted into bins (the cells, cut so that a bin gets about
// WS_FILL sites), each bin's segment padded to whole warps.  A warp
// then takes 32 ghost sites of one bin, one a lane; its lanes test the sites
// of the stencil's cells against the bin's box, 32 at a time, and every lane
// takes every survivor from shared memory.  A ghost site's terms are added in
// cell-list order to an unevaluated sum of two floats (about 48 bits), so that
// U depends neither on the sort nor on the bins.

constexpr int WS_FILL = 48;     // ghost sites per bin: beyond this the bins are cut finer
constexpr int WS_SPAN = 1024;   // insertions per CTA of the finishing kernel
constexpr int WS_BUF = 64;      // survivors buffered per warp

__device__ __forceinline__ unsigned ws_bin(unsigned u, int n) {
  return (unsigned)(((unsigned long long)u * n) >> 32);
}

// sites of the insertions n0..n0+cn-1: fixed-point position and rank within
// their bin.  A one-site ghost is not turned: its offset, three divisions, is
// formed once per CTA.
__global__ void __launch_bounds__(WD_THREADS)
    widom_place_kernel(const WidomBox* __restrict__ boxes, long long n0, int cn) {
  __shared__ unsigned off[3];
  const WidomBox& B = boxes[blockIdx.y];
  const WidomArgs& a = B.a;
  const int nps = a.nps;
  if (nps == 1 && threadIdx.x < 3) {
    const double Lk = threadIdx.x == 0 ? a.Lx : (threadIdx.x == 1 ? a.Ly : a.Lz);
    off[threadIdx.x] = (unsigned)(int)llrint(a.geom[threadIdx.x] / Lk * 4294967296.0);
  }
  __syncthreads();
  const int t = blockIdx.x * WD_THREADS + threadIdx.x;
  if (t >= cn) return;
  const long long k = n0 + t;
  const int nbx = B.nbx, nby = B.nby, nbz = B.nbz;
  const unsigned px = (unsigned)(wd_word(a.seed, k, 0) >> 32),
                 py = (unsigned)(wd_word(a.seed, k, 1) >> 32),
                 pz = (unsigned)(wd_word(a.seed, k, 2) >> 32);
  double R[9];
  if (nps > 1) wd_rotation(a.seed, k, nps, R);
  for (int s = 0; s < nps; s++) {
    unsigned ux = px, uy = py, uz = pz;
    if (nps > 1) {
      const double g0 = a.geom[3 * s], g1 = a.geom[3 * s + 1], g2 = a.geom[3 * s + 2];
      ux += (unsigned)(int)llrint((R[0] * g0 + R[1] * g1 + R[2] * g2) / a.Lx * 4294967296.0);
      uy += (unsigned)(int)llrint((R[3] * g0 + R[4] * g1 + R[5] * g2) / a.Ly * 4294967296.0);
      uz += (unsigned)(int)llrint((R[6] * g0 + R[7] * g1 + R[8] * g2) / a.Lz * 4294967296.0);
    } else {
      ux += off[0];
      uy += off[1];
      uz += off[2];
    }
    const int bin = (ws_bin(ux, nbx) * nby + ws_bin(uy, nby)) * nbz + ws_bin(uz, nbz);
    B.pos[t * nps + s] = make_int4((int)ux, (int)uy, (int)uz, atomicAdd(B.cnt + bin, 1));
  }
}

// first slot of every bin, segments padded to whole warps (one CTA a box)
__global__ void __launch_bounds__(1024) widom_scan_kernel(const WidomBox* __restrict__ boxes) {
  __shared__ int ws[32];
  const WidomBox& B = boxes[blockIdx.y];
  const int nbin = B.nbx * B.nby * B.nbz;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int carry = 0;
  for (int b0 = 0; b0 < nbin; b0 += 1024) {
    const int b = b0 + threadIdx.x;
    const int c = b < nbin ? (B.cnt[b] + 31) & ~31 : 0;
    int v = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, v, o);
      if (lane >= o) v += u;
    }
    if (lane == 31) ws[warp] = v;
    __syncthreads();
    if (warp == 0) {
      int w = ws[lane];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, w, o);
        if (lane >= o) w += u;
      }
      ws[lane] = w;
    }
    __syncthreads();
    if (b < nbin) B.start[b] = carry + v - c + (warp ? ws[warp - 1] : 0);
    carry += ws[31];
    __syncthreads();
  }
  if (threadIdx.x == 0) B.start[nbin] = carry;
}

__global__ void __launch_bounds__(WD_THREADS)
    widom_slot_kernel(const WidomBox* __restrict__ boxes, int cn) {
  const WidomBox& B = boxes[blockIdx.y];
  const int e = blockIdx.x * WD_THREADS + threadIdx.x;
  if (e >= cn * B.a.nps) return;
  const int4 p = B.pos[e];
  const int bin = (ws_bin(p.x, B.nbx) * B.nby + ws_bin(p.y, B.nby)) * B.nbz + ws_bin(p.z, B.nbz);
  B.slot[B.start[bin] + p.w] = e;
}

__global__ void __launch_bounds__(WD_THREADS)
    widom_sorted_kernel(const WidomBox* __restrict__ boxes) {
  __shared__ PairFS tab[MAX_WPROBE * MAX_KINDS];
  __shared__ int4 buf[WD_WARPS][WS_BUF];
  const WidomBox& B = boxes[blockIdx.y];
  const WidomArgs& a = B.a;
  const int ncx = a.ncx, ncy = a.ncy, ncz = a.ncz, nbx = B.nbx, nby = B.nby, nbz = B.nbz;
  const int nslot = B.start[nbx * nby * nbz];
  if ((int)blockIdx.x * WD_THREADS >= nslot) return;
  const int nkind = a.nkind, nps = a.nps, nstencil = a.nstencil;
  for (int t = threadIdx.x; t < nps * nkind; t += WD_THREADS)
    tab[t] = *reinterpret_cast<const PairFS*>(B.tabf + t);
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int slot = blockIdx.x * WD_THREADS + threadIdx.x;
  if (slot - lane >= nslot) return;   // whole warps: segments are whole warps
  const int4* __restrict__ pj = B.pj;
  const float4* __restrict__ eru = B.eru;
  const int4* __restrict__ stencil = a.stencil;
  const int* __restrict__ cell_start = a.cell_start;
  const int e = B.slot[slot];
  // the first slot of a segment's warp is always taken; lanes past the
  // segment's end repeat it
  const int e0 = __shfl_sync(0xffffffffu, e, 0);
  const int4 p = B.pos[e < 0 ? e0 : e];
  const int4 p0 = make_int4(__shfl_sync(0xffffffffu, p.x, 0), __shfl_sync(0xffffffffu, p.y, 0),
                            __shfl_sync(0xffffffffu, p.z, 0), 0);
  const int bx = ws_bin(p0.x, nbx), by = ws_bin(p0.y, nby), bz = ws_bin(p0.z, nbz);
  // a cell is a whole number of bins
  const int cx = bx / (nbx / ncx), cy = by / (nby / ncy), cz = bz / (nbz / ncz);
  const unsigned mx = (unsigned)((unsigned long long)(2 * bx + 1) * 2147483648ULL / (unsigned)nbx),
                 my = (unsigned)((unsigned long long)(2 * by + 1) * 2147483648ULL / (unsigned)nby),
                 mz = (unsigned)((unsigned long long)(2 * bz + 1) * 2147483648ULL / (unsigned)nbz);
  const float sx = (float)(a.Lx * 2.3283064365386963e-10), sy = (float)(a.Ly * 2.3283064365386963e-10),
              sz = (float)(a.Lz * 2.3283064365386963e-10);
  const float hx = 0.5f * (float)a.Lx / nbx, hy = 0.5f * (float)a.Ly / nby,
              hz = 0.5f * (float)a.Lz / nbz;
  // the bin test may keep too many, never too few: rounding is far below 1e-4
  const float cq = (float)a.cutoff_sq, cqb = 1.0001f * cq, sgrid = (float)a.sgrid;
  const PairFS* T = tab + (e < 0 ? 0 : e % nps) * nkind;
  const int ntab1 = a.ntab - 1;
  const unsigned below = (1u << lane) - 1u;
  float uh = 0, ul = 0;

  auto term = [&](const int4 q) {
    const float dx = (float)(int)((unsigned)p.x - (unsigned)q.x) * sx;
    const float dy = (float)(int)((unsigned)p.y - (unsigned)q.y) * sy;
    const float dz = (float)(int)((unsigned)p.z - (unsigned)q.z) * sz;
    const float rr = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
    if (rr < cq) {
      const PairFS& P = T[q.w & 255];
      float u = 0;
      if (rr < P.C2q) {
        if (rr < P.C1q) {
          const float x = P.Sq / rr, y = x * x * x;
          u = P.E4 * fmaf(y, y, -y);
        } else {
          const float x = rr - P.C2q;
          u = P.A * x * x;
        }
      }
      if (P.qq != 0.f) {
        const float4 s = __ldg(eru + min((int)(rr * sgrid), ntab1));
        u += (__fdividef(s.y, s.z + rr) + s.x) * P.qq;
      }
      // uh + ul += u (Knuth's two-sum)
      const float t = __fadd_rn(uh, u), b = __fsub_rn(t, uh);
      ul = __fadd_rn(ul, __fadd_rn(__fsub_rn(uh, __fsub_rn(t, b)), __fsub_rn(u, b)));
      uh = t;
    }
  };

  int head = 0, fill = 0;
  for (int st0 = 0; st0 < nstencil; st0 += 32) {
    // 32 cells of the stencil: their sites as one list, 32 of it at a time
    int j0 = 0, cnt = 0;
    if (st0 + lane < nstencil) {
      const int4 o = stencil[st0 + lane];
      const int c2 = (wd_wrap(cx + o.x, ncx) * ncy + wd_wrap(cy + o.y, ncy)) * ncz +
                     wd_wrap(cz + o.z, ncz);
      j0 = cell_start[c2];
      cnt = cell_start[c2 + 1] - j0;
    }
    int incl = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += u;
    }
    const int total = __shfl_sync(0xffffffffu, incl, 31);
    j0 -= incl - cnt;   // site t of the list is j0 + t in its cell
    for (int base = 0; base < total; base += 32) {
      const int t = base + lane;
      int c = 0;   // the cell of t: the number of cells that end at or before it
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const int u = __shfl_sync(0xffffffffu, incl, c + o - 1);
        if (u <= t) c += o;
      }
      const int jc = __shfl_sync(0xffffffffu, j0, min(c, 31));
      bool keep = false;
      int4 q = make_int4(0, 0, 0, 0);
      if (t < total) {
        q = pj[jc + t];
        const float ex = fmaxf(fabsf((float)(int)((unsigned)q.x - mx) * sx) - hx, 0.f),
                    ey = fmaxf(fabsf((float)(int)((unsigned)q.y - my) * sy) - hy, 0.f),
                    ez = fmaxf(fabsf((float)(int)((unsigned)q.z - mz) * sz) - hz, 0.f);
        keep = fmaf(ex, ex, fmaf(ey, ey, ez * ez)) < cqb;
      }
      const unsigned vote = __ballot_sync(0xffffffffu, keep);
      if (keep) buf[warp][(head + fill + __popc(vote & below)) & (WS_BUF - 1)] = q;
      fill += __popc(vote);
      __syncwarp();
      if (fill >= 32) {
#pragma unroll 4
        for (int i = 0; i < 32; i++) term(buf[warp][head + i]);
        head = (head + 32) & (WS_BUF - 1);
        fill -= 32;
        __syncwarp();
      }
    }
  }
  for (int i = 0; i < fill; i++) term(buf[warp][(head + i) & (WS_BUF - 1)]);
  // an overflowed sum stays what it is
  if (e >= 0) B.ue[e] = isinf(uh) ? (double)uh : (double)uh + (double)ul;
}

// U and the Boltzmann factor of every insertion, summed per CTA; a further
// chunk adds to the sums of the ones before
__global__ void __launch_bounds__(WD_THREADS)
    widom_finish_kernel(const WidomBox* __restrict__ boxes, long long n0, int cn) {
  const WidomBox& B = boxes[blockIdx.y];
  const WidomArgs& a = B.a;
  const double beta = -1 / a.T;
  double acc = 0;
  for (int t = blockIdx.x * WS_SPAN + threadIdx.x; t < min(cn, ((int)blockIdx.x + 1) * WS_SPAN);
       t += WD_THREADS) {
    double U = 0;
    for (int s = 0; s < a.nps; s++) U += B.ue[t * a.nps + s];
    if (a.U) a.U[n0 + t] = U;
    const double e = U * beta;
    if (e > -700) acc += exp(e);
  }
  acc = warp_sum(acc);
  __shared__ double ws[WD_WARPS];
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = n0 ? a.part[blockIdx.x] : 0;
    for (int w = 0; w < WD_WARPS; w++) s += ws[w];
    a.part[blockIdx.x] = s;
  }
}

// FP64 path: the same in double, nearest image by rint
__global__ void __launch_bounds__(WD_THREADS) widom_fp64_kernel(const WidomBox* __restrict__ boxes) {
  __shared__ PairD tab[MAX_WPROBE * MAX_KINDS];
  const WidomBox& B = boxes[blockIdx.y];
  const WidomArgs a = B.a;
  const double4* __restrict__ pd = B.pd;
  const double* __restrict__ ert = B.ert;
  for (int t = threadIdx.x; t < a.nps * a.nkind; t += WD_THREADS) tab[t] = B.tabd[t];
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const long long nw = (long long)gridDim.x * WD_WARPS;
  const double s32 = 2.3283064365386963e-10;
  double wacc = 0;
  for (long long k = blockIdx.x * (long long)WD_WARPS + (threadIdx.x >> 5); k < a.n; k += nw) {
    double R[9];
    wd_rotation(a.seed, k, a.nps, R);
    const double px = (double)(unsigned)(wd_word(a.seed, k, 0) >> 32) * s32 * a.Lx,
                 py = (double)(unsigned)(wd_word(a.seed, k, 1) >> 32) * s32 * a.Ly,
                 pz = (double)(unsigned)(wd_word(a.seed, k, 2) >> 32) * s32 * a.Lz;
    double U = 0;
    for (int s = 0; s < a.nps; s++) {
      const double g0 = a.geom[3 * s], g1 = a.geom[3 * s + 1], g2 = a.geom[3 * s + 2];
      const double x = px + (R[0] * g0 + R[1] * g1 + R[2] * g2);
      const double y = py + (R[3] * g0 + R[4] * g1 + R[5] * g2);
      const double z = pz + (R[6] * g0 + R[7] * g1 + R[8] * g2);
      const double fx = x / a.Lx - floor(x / a.Lx), fy = y / a.Ly - floor(y / a.Ly),
                   fz = z / a.Lz - floor(z / a.Lz);
      const int cx = min((int)(fx * a.ncx), a.ncx - 1), cy = min((int)(fy * a.ncy), a.ncy - 1),
                cz = min((int)(fz * a.ncz), a.ncz - 1);
      const PairD* T = tab + s * a.nkind;
      const int s0 = a.lanes_sites ? 0 : lane, ds = a.lanes_sites ? 1 : 32;
      for (int st = s0; st < a.nstencil; st += ds) {
        const int4 o = a.stencil[st];
        const int c2 = (wd_wrap(cx + o.x, a.ncx) * a.ncy + wd_wrap(cy + o.y, a.ncy)) * a.ncz +
                       wd_wrap(cz + o.z, a.ncz);
        const int j0 = a.cell_start[c2], j1 = a.cell_start[c2 + 1];
        for (int j = j0 + (a.lanes_sites ? lane : 0); j < j1; j += a.lanes_sites ? 32 : 1) {
          const double4 q = pd[j];
          double dx = x - q.x, dy = y - q.y, dz = z - q.z;
          dx -= a.Lx * rint(dx / a.Lx);
          dy -= a.Ly * rint(dy / a.Ly);
          dz -= a.Lz * rint(dz / a.Lz);
          const double rr = dx * dx + dy * dy + dz * dz;
          if (rr >= a.cutoff_sq) continue;
          const PairD P = T[(int)(__double_as_longlong(q.w) & 255)];
          if (rr < P.C2q) {
            if (rr < P.C1q) {
              const double xx = P.Sq / rr, yy = xx * xx * xx;
              U += P.E4 * (yy * yy - yy);
            } else {
              const double xx = rr - P.C2q;
              U += P.A * xx * xx;
            }
          }
          if (P.qq != 0) {
            const double* e = ert + 6 * min((int)(rr * a.sgrid), a.ntab - 1);
            U += (e[1] / (e[2] + rr) + e[0]) * P.qq;
          }
        }
      }
    }
    U = warp_sum(U);
    if (lane == 0) {
      if (a.U) a.U[k] = U;
      const double e = -U / a.T;
      if (e > -700) wacc += exp(e);
    }
  }
  wd_block_sum(wacc, a.part);
}

// ------------------------------------------------- identity change --
//
// cook/widom.c:16-170 (Eidchange), sim/simmeas.c:1961-2003 (XWidom): a warp
// per listed molecule; each of its sites against every site of the other
// molecules within the cutoff, with the virtual minus the real constants
// (smoothed LJ, erfc spline times the charge change); lane 0 adds
// exp(-dU/T) (skipped for -dU/T <= -700).

__device__ __forceinline__ float xw_lj(const PairF& P, float rr) {
  if (rr >= P.C2q) return 0.f;
  if (rr < P.C1q) {
    const float x = P.Sq / rr, y = x * x * x;
    return P.E4 * fmaf(y, y, -y);
  }
  const float x = rr - P.C2q;
  return P.A * x * x;
}
__device__ __forceinline__ double xw_lj(const PairD& P, double rr) {
  if (rr >= P.C2q) return 0.0;
  if (rr < P.C1q) {
    const double x = P.Sq / rr, y = x * x * x;
    return P.E4 * (y * y - y);
  }
  const double x = rr - P.C2q;
  return P.A * x * x;
}

__device__ __forceinline__ int xw_cell(double x, double L, int n) {
  const double s = x / L - floor(x / L);
  const int c = (int)(s * n);
  return c < 0 ? 0 : (c >= n ? n - 1 : c);
}

template <bool FP64>
__global__ void __launch_bounds__(WD_THREADS) xwidom_kernel(XWidomArgs a) {
  __shared__ PairF tf[FP64 ? 1 : 2 * MAX_WPROBE * MAX_KINDS];
  __shared__ PairD td[FP64 ? 2 * MAX_WPROBE * MAX_KINDS : 1];
  for (int t = threadIdx.x; t < 2 * MAX_WPROBE * MAX_KINDS; t += WD_THREADS) {
    if (FP64) td[t] = a.tabd[t];
    else tf[t] = a.tabf[t];
  }
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int nw = gridDim.x * WD_WARPS;
  const float sx = (float)(a.Lx * 2.3283064365386963e-10), sy = (float)(a.Ly * 2.3283064365386963e-10),
              sz = (float)(a.Lz * 2.3283064365386963e-10);
  const float cqf = (float)a.cutoff_sq, sgf = (float)a.sgrid;
  double wacc = 0;
  for (int l = blockIdx.x * WD_WARPS + (threadIdx.x >> 5); l < a.nlist; l += nw) {
    const int n = a.list[l], i0 = a.mol_first[n];
    double U = 0;
    for (int s = 0; s < a.nps; s++) {
      const double* ri = a.r + 3 * (long)(i0 + s);
      const double x = ri[0], y = ri[1], z = ri[2];
      const int cx = xw_cell(x, a.Lx, a.ncx), cy = xw_cell(y, a.Ly, a.ncy),
                cz = xw_cell(z, a.Lz, a.ncz);
      // the site as the cell list stores it: 32-bit box fraction (mixed) or
      // the position wrapped into the box (FP64)
      const unsigned ux = (unsigned)llrint((x / a.Lx - floor(x / a.Lx)) * 4294967296.0),
                     uy = (unsigned)llrint((y / a.Ly - floor(y / a.Ly)) * 4294967296.0),
                     uz = (unsigned)llrint((z / a.Lz - floor(z / a.Lz)) * 4294967296.0);
      const double wx = x - a.Lx * floor(x / a.Lx), wy = y - a.Ly * floor(y / a.Ly),
                   wz = z - a.Lz * floor(z / a.Lz);
      const int s0 = a.lanes_sites ? 0 : lane, ds = a.lanes_sites ? 1 : 32;
      for (int st = s0; st < a.nstencil; st += ds) {
        const int4 o = a.stencil[st];
        const int c2 = (wd_wrap(cx + o.x, a.ncx) * a.ncy + wd_wrap(cy + o.y, a.ncy)) * a.ncz +
                       wd_wrap(cz + o.z, a.ncz);
        const int j0 = a.cell_start[c2], j1 = a.cell_start[c2 + 1];
        double u = 0;
        for (int j = j0 + (a.lanes_sites ? lane : 0); j < j1; j += a.lanes_sites ? 32 : 1) {
          if (FP64) {
            const double4 q = a.pd[j];
            const long long w = __double_as_longlong(q.w);
            if ((int)(w >> 8) == n) continue;
            double dx = wx - q.x, dy = wy - q.y, dz = wz - q.z;
            dx -= a.Lx * rint(dx / a.Lx);
            dy -= a.Ly * rint(dy / a.Ly);
            dz -= a.Lz * rint(dz / a.Lz);
            const double rr = dx * dx + dy * dy + dz * dz;
            if (rr >= a.cutoff_sq) continue;
            const PairD& PR = td[s * MAX_KINDS + (int)(w & 255)];
            const PairD& PV = td[(MAX_WPROBE + s) * MAX_KINDS + (int)(w & 255)];
            u += xw_lj(PV, rr) - xw_lj(PR, rr);
            const double dq = PV.qq - PR.qq;
            if (dq != 0) {
              const double* e = a.ert + 6 * min((int)(rr * a.sgrid), a.ntab - 1);
              u += (e[1] / (e[2] + rr) + e[0]) * dq;
            }
          } else {
            const int4 q = a.pj[j];
            if ((q.w >> 8) == n) continue;
            const float dx = (float)(int)(ux - (unsigned)q.x) * sx;
            const float dy = (float)(int)(uy - (unsigned)q.y) * sy;
            const float dz = (float)(int)(uz - (unsigned)q.z) * sz;
            const float rr = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
            if (rr >= cqf) continue;
            const PairF& PR = tf[s * MAX_KINDS + (q.w & 255)];
            const PairF& PV = tf[(MAX_WPROBE + s) * MAX_KINDS + (q.w & 255)];
            float du = xw_lj(PV, rr) - xw_lj(PR, rr);
            const float dq = PV.qq - PR.qq;
            if (dq != 0.f) {
              const float4 e = __ldg(a.eru + min((int)(rr * sgf), a.ntab - 1));
              du += (__fdividef(e.y, e.z + rr) + e.x) * dq;
            }
            u += du;
          }
        }
        U += u;
      }
    }
    U = warp_sum(U);
    if (lane == 0) {
      if (a.U) a.U[l] = U;
      const double e = -U / a.T;
      if (e > -700) wacc += exp(e);
    }
  }
  wd_block_sum(wacc, a.part);
}

cudaError_t k_xwidom(const Launch& L, const XWidomArgs& a, bool fp64) {
  const int nb = widom_blocks(a.nlist);
  if (fp64) xwidom_kernel<true><<<nb, WD_THREADS, 0, L.s>>>(a);
  else xwidom_kernel<false><<<nb, WD_THREADS, 0, L.s>>>(a);
  ++*L.counter;
  return cudaGetLastError();
}

int widom_blocks(long long n) {
  long long b = (n + WD_WARPS - 1) / WD_WARPS;
  return (int)(b < PARTITION_SMS * 8 ? (b > 0 ? b : 1) : PARTITION_SMS * 8);
}

// Sorted from WS_MIN ghost sites a cell on, so that a warp's fixed work (its
// stencil, the bin tests) is shared by enough lanes, and from WS_SITES ghost
// sites in all: a warp's walk through its stencil and the five launches take
// 100 to 200 us at any number, which a warp per insertion (8 ns a site) reaches
// at about that many.  Measured, one box of 3000 ions: 4000 insertions 100 us
// unsorted, 214 sorted; 16000 205 and 225; 64000 644 and 179; 256000 2174 and
// 309.
constexpr int WS_MIN = 4;
constexpr long long WS_SITES = 24576;
// ghost sites sorted at a time over all boxes of a launch (28 bytes each)
constexpr long long WS_CHUNK = 1LL << 23;

// bins of a box for nent ghost sites: the cells, cut along the longest edge
// while that leaves WS_FILL sites a bin.  Finer bins keep fewer sites that
// only the bin's box, not the ghost site, reaches, but pad more slots.
// Measured, 100000 insertions into each of 48 boxes of 500 to 4000 ions, cut
// alike along the edges: 2.45 ms at 96 sites, 1.59 ms at 48.
int3 widom_bins(const WidomArgs& a, double nent) {
  int m[3] = {1, 1, 1};
  const int nc[3] = {a.ncx, a.ncy, a.ncz};
  const double L[3] = {a.Lx, a.Ly, a.Lz};
  for (;;) {
    int k = 0;
    for (int d = 1; d < 3; d++)
      if (L[d] / (nc[d] * m[d]) > L[k] / (nc[k] * m[k])) k = d;
    m[k]++;
    if ((double)nc[0] * m[0] * nc[1] * m[1] * nc[2] * m[2] * WS_FILL > nent) {
      m[k]--;
      return make_int3(nc[0] * m[0], nc[1] * m[1], nc[2] * m[2]);
    }
  }
}

WidomPlan widom_plan(const WidomBox* boxes, int nbox, long long n, bool fp64) {
  WidomPlan P;
  long long ncell = 0;
  int nps = 1;
  for (int i = 0; i < nbox; i++) {
    const WidomArgs& a = boxes[i].a;
    ncell = std::max(ncell, (long long)a.ncx * a.ncy * a.ncz);
    nps = std::max(nps, a.nps);
  }
  P.nblk = widom_blocks(n);
  if (fp64) return P;
  // insertions a chunk (parts of them are summed by at most as many CTAs as
  // the part array has room for), boxes a launch
  P.cn = (int)std::min(n, std::min(WS_CHUNK / nps, (long long)WS_SPAN * PARTITION_SMS * 8));
  if ((double)P.cn * nps < (double)WS_MIN * ncell || (long long)nbox * P.cn * nps < WS_SITES ||
      ncell > (1 << 20))
    return P;
  const int most = (int)std::max(1LL, std::min((long long)nbox, WS_CHUNK / ((long long)P.cn * nps)));
  const int groups = (nbox + most - 1) / most;
  P.boxes = (nbox + groups - 1) / groups;
  for (int i = 0; i < nbox; i++) {
    const int3 b = widom_bins(boxes[i].a, (double)P.cn * boxes[i].a.nps);
    P.nbin = std::max(P.nbin, (size_t)b.x * b.y * b.z);
  }
  P.nblk = (P.cn + WS_SPAN - 1) / WS_SPAN;
  P.nent = (size_t)P.cn * nps;
  P.nslot = (P.nent + 31 * P.nbin + WD_THREADS - 1) / WD_THREADS * WD_THREADS;
  P.sorted = true;
  return P;
}

size_t WidomPlan::bytes() const {
  return boxes * (nent * (sizeof(int4) + sizeof(double)) + (nslot + 2 * nbin + 4) * sizeof(int)) + 64;
}

// the boxes' parts of the workspace
void widom_layout(const WidomPlan& P, WidomBox* boxes, int nbox, void* work) {
  const size_t nb = P.boxes;
  int4* pos = (int4*)work;
  double* ue = (double*)(pos + nb * P.nent);
  int* slot = (int*)(ue + nb * P.nent);
  int* cnt = slot + nb * P.nslot;
  int* start = cnt + nb * P.nbin;
  for (int i = 0; i < nbox; i++) {
    const size_t g = i % nb;
    const int3 b = widom_bins(boxes[i].a, (double)P.cn * boxes[i].a.nps);
    boxes[i].nbx = b.x;
    boxes[i].nby = b.y;
    boxes[i].nbz = b.z;
    boxes[i].pos = pos + g * P.nent;
    boxes[i].ue = ue + g * P.nent;
    boxes[i].slot = slot + g * P.nslot;
    boxes[i].cnt = cnt + g * P.nbin;
    boxes[i].start = start + g * (P.nbin + 1);
  }
}

cudaError_t k_widom(const Launch& L, const WidomBox* boxes, int nbox, long long n, bool fp64,
                    const WidomPlan& P, void* work) {
  if (P.sorted) {
    int* slot = (int*)((double*)((int4*)work + P.boxes * P.nent) + P.boxes * P.nent);
    for (int g = 0; g < nbox; g += P.boxes) {
      const int ng = std::min(P.boxes, nbox - g);
      for (long long n0 = 0; n0 < n; n0 += P.cn) {
        const int cn = (int)std::min((long long)P.cn, n - n0);
        // slots empty (-1), counts zero
        cudaError_t e = cudaMemsetAsync(slot, 0xff, P.boxes * P.nslot * sizeof(int), L.s);
        if (e == cudaSuccess)
          e = cudaMemsetAsync(slot + P.boxes * P.nslot, 0, P.boxes * P.nbin * sizeof(int), L.s);
        if (e != cudaSuccess) return e;
        const unsigned np = (cn + WD_THREADS - 1) / WD_THREADS,
                       ne = (unsigned)((P.nent + WD_THREADS - 1) / WD_THREADS);
        widom_place_kernel<<<dim3(np, ng), WD_THREADS, 0, L.s>>>(boxes + g, n0, cn);
        widom_scan_kernel<<<dim3(1, ng), 1024, 0, L.s>>>(boxes + g);
        widom_slot_kernel<<<dim3(ne, ng), WD_THREADS, 0, L.s>>>(boxes + g, cn);
        widom_sorted_kernel<<<dim3((unsigned)(P.nslot / WD_THREADS), ng), WD_THREADS, 0, L.s>>>(boxes + g);
        widom_finish_kernel<<<dim3(P.nblk, ng), WD_THREADS, 0, L.s>>>(boxes + g, n0, cn);
        *L.counter += 5;
      }
    }
    return cudaGetLastError();
  }
  const dim3 grid(widom_blocks(n), nbox);
  if (fp64)
    widom_fp64_kernel<<<grid, WD_THREADS, 0, L.s>>>(boxes);
  else
    widom_mixed_kernel<<<grid, WD_THREADS, 0, L.s>>>(boxes);
  ++*L.counter;
  return cudaGetLastError();
}

}  // namespace mg
