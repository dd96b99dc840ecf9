// The walk of the FP64 pair kernels: a warp per home site, its neighbours
// found in FP32 and handed on 32 at a time, sorted by the work they need.
#pragma once
#include <algorithm>
#include <cmath>
#include <type_traits>

#include "mg_internal.h"

namespace mg {

constexpr int P64_WARPS = 2;
constexpr int P64_THREADS = 32 * P64_WARPS;
// a Lennard-Jones term (and charges), charges alone, one molecule
constexpr int P64_LJ = 0, P64_Q = 1, P64_EXCL = 2;

// per class a ring of {sorted site, image of x | y << 2 | z << 4 | kind << 8}
// (image: 1 + the number of box edges to take from the separation)
struct P64Queue {
  int2 e[3][64];
};

// tight: the cutoff comes so close to half an edge that a separation inside it
// may be of either image to FP32; the image is then taken in FP64
__device__ __forceinline__ bool p64_tight(const PairArgs& a) {
  const double Lm = fmin(a.Lx, fmin(a.Ly, a.Lz));
  return a.cutoff_sq > 0.25 * 0.9999 * Lm * Lm;
}
__device__ __forceinline__ double p64_image(double d, int code, double L, bool tight) {
  if (tight) return d - L * rint(d / L);
  const int s = code & 3;
  return s == 1 ? d : (s == 2 ? d - L : d + L);
}

__device__ __forceinline__ double p64_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// nearest image of a separation of two wrapped coordinates; code: 0, 1, 2
__device__ __forceinline__ float p64_near(float d, float L, float iL, int* code) {
  const float s = rintf(d * iL);
  *code = 1 + (int)s;
  return fmaf(-s, L, d);
}

// flag [kind]: 1 a Lennard-Jones term with the home site's kind, 2 charges;
// work(class, entry, on) is called by whole warps, `on` where the lane has an
// entry
template <class W>
__device__ __forceinline__ void p64_walk(const PairArgs& a, const float4* __restrict__ pf, int ti,
                                         const unsigned char* flag, P64Queue& Q, float cqf,
                                         const W& work) {
  const int lane = threadIdx.x & 31;
  const unsigned below = (1u << lane) - 1u;
  const float4 me = pf[ti];
  const int mol_i = __float_as_int(me.w) >> 8;
  const float Lx = (float)a.Lx, Ly = (float)a.Ly, Lz = (float)a.Lz;
  const float iLx = 1.f / Lx, iLy = 1.f / Ly, iLz = 1.f / Lz;
  const int ncx = a.ncx, ncy = a.ncy, ncz = a.ncz, nstencil = a.nstencil;
  const int c = a.allpairs ? 0 : a.key_s[ti];
  const int cz = c % ncz, cy = (c / ncz) % ncy, cx = c / (ncy * ncz);
  int head[3] = {0, 0, 0}, fill[3] = {0, 0, 0};

  auto drain = [&](auto cls) {
    constexpr int C = decltype(cls)::value;
    __syncwarp();
    if (fill[C] >= 32) {
      work(cls, Q.e[C][head[C] + lane], true);
      head[C] ^= 32;
      fill[C] -= 32;
      __syncwarp();
    }
  };
  auto push = [&](auto cls, bool on, int2 e) {
    constexpr int C = decltype(cls)::value;
    const unsigned vote = __ballot_sync(0xffffffffu, on);
    if (on) Q.e[C][(head[C] + fill[C] + __popc(vote & below)) & 63] = e;
    fill[C] += __popc(vote);
    drain(cls);
  };
  std::integral_constant<int, P64_LJ> lj;
  std::integral_constant<int, P64_Q> qq;
  std::integral_constant<int, P64_EXCL> ex;

  for (int st0 = 0; st0 < nstencil; st0 += 32) {
    // 32 cells of the stencil: their sites as one list, 32 of it at a time
    int j0 = 0, cnt = 0;
    if (st0 + lane < nstencil) {
      const int4 o = a.stencil[st0 + lane];
      int x = cx + o.x, y = cy + o.y, z = cz + o.z;
      x += x < 0 ? ncx : (x >= ncx ? -ncx : 0);
      y += y < 0 ? ncy : (y >= ncy ? -ncy : 0);
      z += z < 0 ? ncz : (z >= ncz ? -ncz : 0);
      const int c2 = (x * ncy + y) * ncz + z;
      j0 = a.cell_start[c2];
      cnt = a.cell_start[c2 + 1] - j0;
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
      int k = 0;   // the cell of t: the number of cells that end at or before it
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const int u = __shfl_sync(0xffffffffu, incl, k + o - 1);
        if (u <= t) k += o;
      }
      const int j = __shfl_sync(0xffffffffu, j0, k) + t;
      int cls = -1;
      int2 e = make_int2(0, 0);
      if (t < total && j != ti) {
        const float4 q = pf[j];
        int ix, iy, iz;
        const float dx = p64_near(me.x - q.x, Lx, iLx, &ix), dy = p64_near(me.y - q.y, Ly, iLy, &iy),
                    dz = p64_near(me.z - q.z, Lz, iLz, &iz);
        if (fmaf(dx, dx, fmaf(dy, dy, dz * dz)) < cqf) {
          const int w = __float_as_int(q.w), f = flag[w & 255];
          if ((w >> 8) == mol_i) cls = f & 2 ? P64_EXCL : -1;
          else cls = f & 1 ? P64_LJ : (f & 2 ? P64_Q : -1);
          e = make_int2(j, ix | iy << 2 | iz << 4 | (w & 255) << 8);
        }
      }
      push(lj, cls == P64_LJ, e);
      push(qq, cls == P64_Q, e);
      if (__any_sync(0xffffffffu, cls == P64_EXCL)) push(ex, cls == P64_EXCL, e);
    }
  }
  // what is left of the queues
  if (fill[P64_LJ]) work(lj, Q.e[P64_LJ][(head[P64_LJ] + lane) & 63], lane < fill[P64_LJ]);
  if (fill[P64_Q]) work(qq, Q.e[P64_Q][(head[P64_Q] + lane) & 63], lane < fill[P64_Q]);
  if (fill[P64_EXCL])
    work(ex, Q.e[P64_EXCL][(head[P64_EXCL] + lane) & 63], lane < fill[P64_EXCL]);
}

// the cutoff of the FP32 test: coordinates up to L are rounded to 2^-24 L
inline float p64_cutoff(const PairArgs& a) {
  const double Lm = std::max(a.Lx, std::max(a.Ly, a.Lz));
  const double rc = std::sqrt(a.cutoff_sq) + 1e-6 * Lm;
  return (float)(rc * rc * (1 + 1e-5));
}

}  // namespace mg
