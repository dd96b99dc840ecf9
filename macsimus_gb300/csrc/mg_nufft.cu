// Ewald k-space sums of the FP32 path as non-uniform Fourier transforms.
//
// The direct passes form S(k) and the forces with a product per (k-vector,
// charge): 16700 x 98304 of them on 32768 waters, in each pass.  The same two
// sums over the same k set factor into a spreading of the charges on a grid,
// a discrete Fourier transform of the grid onto the k set, and the two steps
// back (type 1 and type 2 non-uniform transforms; Dutt and Rokhlin, SIAM J.
// Sci. Comput. 14, 1368 (1993)), with the "exponential of semicircle" window
//   phi(t) = exp(beta (sqrt(1 - (2t/w)^2) - 1)), |t| < w/2, w = 8 grid steps
// of Barnett, Magland and af Klinteberg (SIAM J. Sci. Comput. 41, C479
// (2019)), whose transform is divided out exactly at every k (host
// quadrature).  The grid has at least 1.86 points per resolved mode.
//
// Measured on 32768 waters: 0.13 ms (spread 57 us, x 6, planes 16, x 6, interp
// 45) against 0.52 ms for the direct tensor-core passes; the MD step
// 0.87 -> 0.43 ms; 256 ionic boxes 3.3 -> 2.7 ms.  Error against 64 bits,
// k-space force relative RMS, mean over 46 boxes of 650 to 98000 sites: 7.2e-7 (the
// direct tensor-core passes 11.5e-7; 9.8e-7 with 1.75 points a mode, the weights
// not cut off and the potential taken whole in the interpolation).
// Every sum runs in a fixed order (a grid point gathers its charges
// in the sorted order of the cell list; no floating-point atomics), so the
// results are reproducible bit for bit, alone or in a batch.
//
// Five launches, every one over all boxes of a batch (blockIdx.z = box):
//   spread  charges (cell-sorted) -> real grid G[x][y][z]
//   dft_x   G -> A[kx][y][z], kx = 0..Kx (G real: the half kx >= 0)
//   plane   per kx (four CTAs): y -> ky, z -> kz, S(k) times ekk / (window transform)^2,
//           and back to A[kx][y][z], the plane's modes in shared memory
//   idft_x  A -> the potential grid (real) in G
//   interp  potential grid -> forces of the charges (gradient of the window)
// The transforms are dense sums against small tables (at most some 50 points
// onto some 20 modes a line) folded by parity: inputs at a and M - a are
// added and subtracted once, and one pair of cosine and sine sums gives the
// outputs at +k and -k, a quarter of the plain products.
#include <cooperative_groups.h>

#include <cmath>
#include <vector>

#include "mg_internal.h"
#include "mg_device.cuh"
#include "mg_nufft.h"

namespace mg {

#define LAUNCHED(L) (++*(L).counter)
static inline int cdiv(long a, long b) { return (int)((a + b - 1) / b); }

namespace {

constexpr int W = NF_W;

__device__ __forceinline__ float nf_sqrt(float x) {
  float r;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float nf_rcp(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float nf_ex2(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// the window at z = 2 t / w; nb = -beta log2(e).  The exponent is taken as
// -beta z^2 / (1 + s), s = sqrt(1 - z^2): beta (s - 1) would carry the
// rounding of s times beta (1e-6 of the weight near its centre).  Zero beyond the
// window (reached by points of a tile that a charge does not touch): the same
// arithmetic with |1 - z^2| would leave up to 1e-7 there, which of two boxes of
// some 75000 sites made 2.3e-6 of the k-space force, 1.3e-6 and 1.5e-6 without.
__device__ __forceinline__ float nf_window(float z, float nb, float& s) {
  const float z2 = __fmul_rn(z, z);
  s = nf_sqrt(fabsf(__fmaf_rn(-z, z, 1.f)));
  const float w = nf_ex2(__fmul_rn(__fmul_rn(nb, z2), nf_rcp(__fadd_rn(1.f, s))));
  return z2 < 1.f ? w : 0.f;
}

// pairs of floats: acc += a * w, a * w
__device__ __forceinline__ void nf_fma2(unsigned long long& acc, unsigned long long a,
                                        unsigned long long w) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(w));
}
__device__ __forceinline__ unsigned long long nf_mul2(unsigned long long a, unsigned long long w) {
  unsigned long long r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(w));
  return r;
}
__device__ __forceinline__ void nf_copy16(void* smem, const void* g) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(
                   (unsigned)__cvta_generic_to_shared(smem)),
               "l"(g)
               : "memory");
}
__device__ __forceinline__ void nf_copy8(void* smem, const void* g) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(
                   (unsigned)__cvta_generic_to_shared(smem)),
               "l"(g)
               : "memory");
}
__device__ __forceinline__ void nf_copy_wait() {
  asm volatile("cp.async.commit_group;\n cp.async.wait_group 0;" ::: "memory");
}

// grid cell and offset in it of a fixed-point coordinate (exact product)
__device__ __forceinline__ int nf_cell(int fx, int M, float& frac) {
  const unsigned long long p = (unsigned long long)(unsigned)fx * (unsigned)M;
  frac = __fmul_rn((float)(unsigned)p, 2.3283064365386963e-10f);
  return (int)(p >> 32);
}

// a Drude shell's fixed-point coordinate: the site's plus the displacement
__device__ __forceinline__ int nf_shift(int fx, float d, float scale) {
  return (int)((unsigned)fx + (unsigned)__float2int_rn(__fmul_rn(d, scale)));
}

}  // namespace

// the charges near a box of the grid: the columns (cx, cy) of the cells that
// hold them 32 at a time, one per lane with its run of sites along z (two
// parts where it wraps), read as one list of candidates whatever the runs'
// lengths
struct NfRuns {
  int c0[3], cn[3], ncol;

  // cells of the grid steps [o - lo, o + hi) in every direction; Drude shells
  // are looked up by their site, up to `marg` grid steps away (and by scanning
  // the whole box when a displacement is larger than that)
  __device__ __forceinline__ void set(const NfBox& b, int ox, int oy, int oz, int lo, int hi) {
    const bool all = b.nsub > 1 && *b.far != 0;
    const int o[3] = {ox, oy, oz};
#pragma unroll
    for (int d = 0; d < 3; d++) {
      const int M = b.M[d], n = b.nc[d], len = lo + hi + 2 * b.marg[d];
      if (all || len >= M) {
        c0[d] = 0;
        cn[d] = n;
      } else {
        // grid step m lies in cell floor(m n / M), taken a little wide (the
        // candidates are tested exactly)
        int l = o[d] - lo - b.marg[d];
        l += l < 0 ? M : 0;
        const int a = max((int)(l * b.cpg[d] - 1e-3f), 0);
        const int e = (int)((l + len) * b.cpg[d] + 1e-3f);
        c0[d] = a;
        cn[d] = min(n, e - a + 1);
      }
    }
    ncol = cn[0] * cn[1];
  }

  // the runs of columns cb .. cb + 31 into runs[] (first candidate, site,
  // length, wrapped part); returns the number of candidates
  __device__ __forceinline__ int columns(const NfBox& b, int cb, int lane, int4* runs) const {
    int ja = 0, la = 0, jw = 0, lw = 0;
    if (cb + lane < ncol) {
      int cx = c0[0] + (cb + lane) / cn[1], cy = c0[1] + (cb + lane) % cn[1];
      cx -= cx >= b.nc[0] ? b.nc[0] : 0;
      cy -= cy >= b.nc[1] ? b.nc[1] : 0;
      const int* cs = b.cell_start + (cx * b.nc[1] + cy) * b.nc[2];
      const int e = c0[2] + cn[2];
      ja = cs[c0[2]];
      la = cs[min(e, b.nc[2])] - ja;
      if (e > b.nc[2]) {
        jw = cs[0];
        lw = cs[e - b.nc[2]] - jw;
      }
    }
    int pre = la + lw;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, pre, o);
      if (lane >= o) pre += v;
    }
    const int total = __shfl_sync(0xffffffffu, pre, 31);
    pre -= la + lw;
    __syncwarp();
    runs[lane] = make_int4(pre, ja, la, jw);
    __syncwarp();
    return total;
  }

  // candidate k: the last run that starts at or before it (never an empty
  // one: the next run starts at the same place)
  static __device__ __forceinline__ int site(const int4* runs, int k) {
    int r = 0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
      if (runs[r + o].x <= k) r += o;
    const int4 u = runs[r];
    const int d = k - u.x;
    return d < u.z ? u.y + d : u.w + d - u.z;
  }
};

// charge `sub` of sorted site j with record p: its charge, and its fixed-point
// position in r
__device__ __forceinline__ float nf_charge(const NfBox& b, int j, const int4& p, int sub, int4& r) {
  r = p;
  if (j < 0) return 0.f;
  const float q = sub ? b.qp[p.w & 255] : b.q[p.w & 255];
  if (sub && q != 0.f) {
    const float4 d = b.pdj[j];
    r.x = nf_shift(p.x, d.x, b.fix[0]);
    r.y = nf_shift(p.y, d.y, b.fix[1]);
    r.z = nf_shift(p.z, d.z, b.fix[2]);
  }
  return q;
}

// ------------------------------------------------------------- spreading --
//
// A tile of 8 x 8 x 8 grid points; lane = (pair of x, y), 2 x 8 points in
// registers.  The charges whose window reaches the tile are compacted 32 at a
// time into shared memory as their 1-D weights at the tile's points (lane =
// charge, 24 windows), and every lane adds q wx wy wz to its points, two at
// a time (f32x2): no atomics, a fixed order.  Dense boxes: eight warps share a
// tile, each taking every eighth batch of candidates, their sums added in
// order; sparse ones (a few charges a tile): one warp a tile.
// (Weights of x and y are kept twice, so that a pair product needs no moves.)
constexpr int TILE = NF_TILE, SP_WARPS = 8, TP = TILE * TILE * TILE;
constexpr int SP_ST = 5 * 32 * TILE;

__global__ void __launch_bounds__(SP_WARPS * 32) nf_spread_kernel(const NfBox* __restrict__ boxes) {
  after_previous();
  const NfBox& b = boxes[blockIdx.z];
  const int ntz = (b.M[2] + TILE - 1) / TILE, nty = (b.M[1] + TILE - 1) / TILE,
            ntx = (b.M[0] + TILE - 1) / TILE;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool dense = b.dense != 0;
  const int tile = dense ? blockIdx.x : blockIdx.x * SP_WARPS + warp;
  // 1-D weights of 32 charges per warp; at the end the warps' tile sums
  extern __shared__ float4 zs[];
  float (*st)[SP_ST] = reinterpret_cast<float (*)[SP_ST]>(zs);   // [SP_WARPS]
  __shared__ int4 que[SP_WARPS][64];
  __shared__ int4 runs[SP_WARPS][32];
  if (tile >= ntx * nty * ntz) return;
  const int x0 = tile / (nty * ntz) * TILE, y0 = tile / ntz % nty * TILE, z0 = tile % ntz * TILE;
  const unsigned Mx = b.M[0], My = b.M[1], Mz = b.M[2];
  // the tile's window box in fixed point: origin o - w/2, extent
  const unsigned lox = (unsigned)((x0 - W / 2) * b.step[0] >> 32),
                 loy = (unsigned)((y0 - W / 2) * b.step[1] >> 32),
                 loz = (unsigned)((z0 - W / 2) * b.step[2] >> 32);
  const unsigned exx = b.ext[0], exy = b.ext[1], exz = b.ext[2];
  const float nbx = b.nb[0], nby = b.nb[1], nbz = b.nb[2];
  float2* wx = reinterpret_cast<float2*>(st[warp]);   // [32][8] q * window, twice
  float2* wy = wx + 32 * TILE;                        // [32][8], twice
  float* wz = st[warp] + 4 * 32 * TILE;               // [32][8]
  const int lx = lane >> 3, ly = lane & 7;
  unsigned long long g[2][TILE / 2];
#pragma unroll
  for (int k = 0; k < TILE / 2; k++) g[0][k] = g[1][k] = 0ull;

  int qh = 0, qn = 0;
  auto flush = [&](int cnt) {
    const int4 r = que[warp][(qh + lane) & 63];
    // steps from the window box's origin: 0 .. 15, and the rest
    auto place = [](unsigned rel, unsigned M, float& base) {
      const unsigned long long p = (unsigned long long)rel * M;
      base = __fmul_rn((float)(unsigned)p, 2.3283064365386963e-10f);
      return (float)((int)(p >> 32) - W / 2);
    };
    float fx, fy, fz, s;
    const float dx = place((unsigned)r.x - lox, Mx, fx), dy = place((unsigned)r.y - loy, My, fy),
                dz = place((unsigned)r.z - loz, Mz, fz);
    const float q = __int_as_float(r.w);
    auto window = [&](float d, float f, float nb, int k) {
      return nf_window(__fmul_rn(__fadd_rn(__fadd_rn(d, -(float)k), f), 2.f / W), nb, s);
    };
    __syncwarp();
#pragma unroll
    for (int h = 0; h < TILE; h += 2) {
      const float u = __fmul_rn(q, window(dx, fx, nbx, h)),
                  v = __fmul_rn(q, window(dx, fx, nbx, h + 1));
      *reinterpret_cast<float4*>(wx + lane * TILE + h) = make_float4(u, u, v, v);
    }
#pragma unroll
    for (int h = 0; h < TILE; h += 2) {
      const float u = window(dy, fy, nby, h), v = window(dy, fy, nby, h + 1);
      *reinterpret_cast<float4*>(wy + lane * TILE + h) = make_float4(u, u, v, v);
    }
#pragma unroll
    for (int h = 0; h < TILE; h += 4)
      *reinterpret_cast<float4*>(wz + lane * TILE + h) =
          make_float4(window(dz, fz, nbz, h), window(dz, fz, nbz, h + 1),
                      window(dz, fz, nbz, h + 2), window(dz, fz, nbz, h + 3));
    __syncwarp();
#pragma unroll 2
    for (int c = 0; c < cnt; c++) {
      const ulonglong2 vx = *reinterpret_cast<const ulonglong2*>(wx + c * TILE + 2 * lx);
      const unsigned long long vy = *reinterpret_cast<const unsigned long long*>(wy + c * TILE + ly);
      const unsigned long long a0 = nf_mul2(vx.x, vy), a1 = nf_mul2(vx.y, vy);
      const ulonglong2 u = *reinterpret_cast<const ulonglong2*>(wz + c * TILE),
                       v = *reinterpret_cast<const ulonglong2*>(wz + c * TILE + 4);
      nf_fma2(g[0][0], a0, u.x);
      nf_fma2(g[0][1], a0, u.y);
      nf_fma2(g[0][2], a0, v.x);
      nf_fma2(g[0][3], a0, v.y);
      nf_fma2(g[1][0], a1, u.x);
      nf_fma2(g[1][1], a1, u.y);
      nf_fma2(g[1][2], a1, v.x);
      nf_fma2(g[1][3], a1, v.y);
    }
    __syncwarp();
  };

  NfRuns R;
  R.set(b, x0, y0, z0, W / 2, TILE + W / 2);
  const int step = dense ? 32 * SP_WARPS : 32, first = dense ? 32 * warp : 0;
  for (int cb = 0; cb < R.ncol; cb += 32) {
    const int total = R.columns(b, cb, lane, runs[warp]);
    // a batch is loaded before the one before it is used
    int jn = first + lane < total ? NfRuns::site(runs[warp], first + lane) : -1;
    int4 pn = jn >= 0 ? b.pj[jn] : make_int4(0, 0, 0, 0);
    for (int kb = first; kb < total; kb += step) {
      const int j = jn, kn = kb + step + lane;
      const int4 p = pn;
      jn = kn < total ? NfRuns::site(runs[warp], kn) : -1;
      pn = jn >= 0 ? b.pj[jn] : make_int4(0, 0, 0, 0);
      for (int sub = 0; sub < b.nsub; sub++) {
        int4 r;
        const float q = nf_charge(b, j, p, sub, r);
        const bool keep = q != 0.f && (unsigned)r.x - lox <= exx && (unsigned)r.y - loy <= exy &&
                          (unsigned)r.z - loz <= exz;
        const unsigned m = __ballot_sync(0xffffffffu, keep);
        if (keep)
          que[warp][(qh + qn + __popc(m & ((1u << lane) - 1u))) & 63] =
              make_int4(r.x, r.y, r.z, __float_as_int(q));
        qn += __popc(m);
        __syncwarp();
        if (qn >= 32) {
          flush(32);
          qh = (qh + 32) & 63;
          qn -= 32;
        }
      }
    }
  }
  if (qn > 0) flush(qn);
  if (!dense) {
    const int y = y0 + ly;
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int x = x0 + 2 * lx + h;
      if (x >= (int)Mx || y >= (int)My) continue;
      float* o = b.G + ((long)x * My + y) * Mz + z0;
      // Mz is a multiple of 4
      *reinterpret_cast<ulonglong2*>(o) = make_ulonglong2(g[h][0], g[h][1]);
      if (z0 + 4 < (int)Mz) *reinterpret_cast<ulonglong2*>(o + 4) = make_ulonglong2(g[h][2], g[h][3]);
    }
    return;
  }
  // the warps' sums of the tile, points ((x 8) + y) 8 + z, added in order
  __syncwarp();
#pragma unroll
  for (int h = 0; h < 2; h++) {
    float* o = st[warp] + ((2 * lx + h) * TILE + ly) * TILE;
    *reinterpret_cast<ulonglong2*>(o) = make_ulonglong2(g[h][0], g[h][1]);
    *reinterpret_cast<ulonglong2*>(o + 4) = make_ulonglong2(g[h][2], g[h][3]);
  }
  __syncthreads();
  const int i = threadIdx.x * 2, z = z0 + i % TILE, y = y0 + i / TILE % TILE,
            x = x0 + i / (TILE * TILE);
  static_assert(SP_WARPS * 32 * 2 == TP, "two points per thread");
  if (x < (int)Mx && y < (int)My && z < (int)Mz) {
    float2 v = *reinterpret_cast<const float2*>(st[0] + i);
#pragma unroll
    for (int w = 1; w < SP_WARPS; w++) {
      const float2 u = *reinterpret_cast<const float2*>(st[w] + i);
      v.x = __fadd_rn(v.x, u.x);
      v.y = __fadd_rn(v.y, u.y);
    }
    *reinterpret_cast<float2*>(b.G + ((long)x * My + y) * Mz + z) = v;
  }
}

// ------------------------------------------------------------ transforms --
//
// Tables: fwd [chunk][a = 0..M/2][KC] and inv [chunk][k = 0..K][KC], entries
// (cos, sin) of 2 pi a k / M, KC outputs of a thread per chunk; the columns
// of a stage are contiguous, so every grid access is coalesced.

// Each CTA of the stages over x takes 32 columns (y, z) whole into shared
// memory (one round trip to L2; a loop of loads per thread waited for one
// round trip per few steps, 20 us on 32768 waters), a warp per chunk of
// outputs.
constexpr int DF_COLS = 32, DF_THREADS = 256, PL_THREADS = 128, PL_KC = NF_KC;
constexpr int NF_CSB = 2, NF_TB = 256;   // CTAs a plane and their threads in a batch

// G[x][c] -> A[kx][c], c = (y, z)
__global__ void __launch_bounds__(DF_THREADS) nf_dft_x_kernel(const NfBox* __restrict__ boxes) {
  after_previous();
  const NfBox& b = boxes[blockIdx.z];
  const int ncol = b.M[1] * b.M[2], c0 = blockIdx.x * DF_COLS, M = b.M[0], H = M / 2, K = b.K[0];
  if (c0 >= ncol) return;
  extern __shared__ float4 zs[];
  float* in = reinterpret_cast<float*>(zs);      // [M][32]
  float4* tw = zs + M * (DF_COLS / 4);           // [chunk][H + 1][NF_KC / 2]
  const int nch = K / NF_KC + 1, ntw = nch * (H + 1) * (NF_KC / 2);
  for (int i = threadIdx.x; i < M * (DF_COLS / 4); i += DF_THREADS) {
    const int c = c0 + i % (DF_COLS / 4) * 4;    // ncol is a multiple of 16
    if (c < ncol) nf_copy16(in + 4 * i, b.G + (long)(i / (DF_COLS / 4)) * ncol + c);
  }
  for (int i = threadIdx.x; i < ntw; i += DF_THREADS)
    nf_copy16(tw + i, reinterpret_cast<const float4*>(b.fwd[0]) + i);
  nf_copy_wait();
  __syncthreads();
  const int lane = threadIdx.x & 31, c = c0 + lane;
  if (c >= ncol) return;
  for (int ch = threadIdx.x >> 5; ch < nch; ch += DF_THREADS / 32) {
    const float* g = in + lane;
    const float4* t = tw + ch * (H + 1) * (NF_KC / 2);
    float re[NF_KC], im[NF_KC];
    const float g0 = g[0], gh = g[H * DF_COLS];
#pragma unroll
    for (int k = 0; k < NF_KC; k++) {
      re[k] = (k & 1) ? __fadd_rn(g0, -gh) : __fadd_rn(g0, gh);   // NF_KC is even
      im[k] = 0.f;
    }
#pragma unroll 4
    for (int x = 1; x < H; x++) {
      const float a = g[x * DF_COLS], d = g[(M - x) * DF_COLS];
      const float e = __fadd_rn(a, d), o = __fadd_rn(a, -d);
#pragma unroll
      for (int k = 0; k < NF_KC; k += 2) {
        const float4 w = t[x * (NF_KC / 2) + k / 2];
        re[k] = __fmaf_rn(e, w.x, re[k]);
        im[k] = __fmaf_rn(o, w.y, im[k]);
        re[k + 1] = __fmaf_rn(e, w.z, re[k + 1]);
        im[k + 1] = __fmaf_rn(o, w.w, im[k + 1]);
      }
    }
#pragma unroll
    for (int k = 0; k < NF_KC; k++)
      if (ch * NF_KC + k <= K) b.A[(long)(ch * NF_KC + k) * ncol + c] = make_float2(re[k], im[k]);
  }
}

// One plane kx per cluster of four CTAs, from A[kx][y][z] and back to it: the
// transform over y, the transform over z, S(k) and the potential modes, and
// the two transforms back.  The CTAs split the plane by z for the sums over y
// and by ky for those over z, and hand the halves over through each other's
// shared memory.  Measured, the energy and virial sums of the plane.
// (One CTA per plane: 26 us on 32768 waters, 21 SMs at work; three launches
// with the plane in memory between them: 51 us.)
// CS CTAs of T threads a plane: four of 128 for one box, whose planes are too few
// for the GPU; two of 256 for the plain steps of a batch that fills it, which
// copy the tables half as often and sum more items each (256 ionic boxes 625 ->
// 533 us; one of 512 535 us; tables through L1 instead 714; 564 with 1.86 points a
// mode).  Every sum of the
// modes and of the grid is a thread's own, so the split does not change them; it
// would change the order of the energy sums, and a measured step keeps four.
template <int CS, int T>
__global__ void __cluster_dims__(CS, 1, 1) __launch_bounds__(T)
    nf_plane_kernel(const NfBox* __restrict__ boxes, const bool measure) {
  after_previous();
  const NfBox& b = boxes[blockIdx.z];
  const int kx = blockIdx.x / CS;
  if (kx > b.K[0]) return;   // the whole cluster
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = cluster.block_rank();
  const int My = b.M[1], Mz = b.M[2], Hy = My / 2, Hz = Mz / 2, Ky = b.K[1], Kz = b.K[2],
            NY = 2 * Ky + 1, ld = Mz + 1;   // odd row length: no bank conflicts along ky
  const int nzq = Mz / CS, zq = rank * nzq;          // this CTA's columns z
  const int nrow = (NY + CS - 1) / CS, r0 = rank * nrow,
            nr = max(0, min(nrow, NY - r0));            // and rows ky
  extern __shared__ float4 zs[];
  // the four tables: y forwards, z forwards, z backwards, y backwards
  const int nky = Ky / PL_KC + 1, nkz = Kz / 2 + 1, nz = Hz / 2 + 1, ny = Hy / PL_KC + 1;
  const int n0 = nky * (Hy + 1) * (PL_KC / 2), n1 = nkz * (Hz + 1), n2 = nz * (Kz + 1),
            n3 = ny * (Ky + 1) * (PL_KC / 2);
  const float4 *tab0 = zs, *tab1 = tab0 + n0, *tab2 = tab1 + n1, *tab3 = tab2 + n2;
  float4* pm = zs + n0 + n1 + n2 + n3;                       // [Kz + 1][nrow]
  float2* rows = reinterpret_cast<float2*>(pm + (Kz + 1) * nrow);  // [nrow][ld]
  float2* cols = rows + nrow * ld + (nrow * ld & 1);         // [max(My, NY)][nzq]
  __shared__ double red[7][T / 32];
  float2* A = b.A + (long)kx * My * Mz;
  {
    // this CTA's columns (nzq may be odd: 8-byte copies), then the tables
    for (int i = threadIdx.x; i < My * nzq; i += T) {
      const int y = i / nzq;
      nf_copy8(cols + i, A + y * Mz + zq + i - y * nzq);
    }
    const float4* src[4] = {
        reinterpret_cast<const float4*>(b.fwd[1]), reinterpret_cast<const float4*>(b.fwd[2]),
        reinterpret_cast<const float4*>(b.inv[2]), reinterpret_cast<const float4*>(b.inv[1])};
    const int n[4] = {n0, n1, n2, n3};
    float4* dst = zs;
#pragma unroll
    for (int k = 0; k < 4; k++) {
      for (int i = threadIdx.x; i < n[k]; i += T) nf_copy16(dst + i, src[k] + i);
      dst += n[k];
    }
    nf_copy_wait();
  }
  cluster.sync();   // every CTA runs and has its data
  // y -> ky: item = (chunk of PL_KC ky, z); row ky to the CTA that holds it
  for (int it = threadIdx.x; it < nky * nzq; it += T) {
    const int ch = it / nzq, z = it - ch * nzq, k0 = ch * PL_KC;
    const float2* a = cols + z;
    const float4* t = tab0 + ch * (Hy + 1) * (PL_KC / 2);
    float cr[PL_KC], ci[PL_KC], dr[PL_KC], di[PL_KC];
    const float2 a0 = a[0], ah = a[Hy * nzq];
#pragma unroll
    for (int k = 0; k < PL_KC; k++) {
      const float s = (k & 1) ? -1.f : 1.f;   // k0 is even
      cr[k] = __fmaf_rn(s, ah.x, a0.x);
      ci[k] = __fmaf_rn(s, ah.y, a0.y);
      dr[k] = di[k] = 0.f;
    }
#pragma unroll 4
    for (int y = 1; y < Hy; y++) {
      const float2 p = a[y * nzq], m = a[(My - y) * nzq];
      const float er = __fadd_rn(p.x, m.x), ei = __fadd_rn(p.y, m.y), orr = __fadd_rn(p.x, -m.x),
                  oi = __fadd_rn(p.y, -m.y);
#pragma unroll
      for (int k = 0; k < PL_KC; k += 2) {
        const float4 w = t[y * (PL_KC / 2) + k / 2];
        cr[k] = __fmaf_rn(er, w.x, cr[k]);
        ci[k] = __fmaf_rn(ei, w.x, ci[k]);
        dr[k] = __fmaf_rn(orr, w.y, dr[k]);
        di[k] = __fmaf_rn(oi, w.y, di[k]);
        cr[k + 1] = __fmaf_rn(er, w.z, cr[k + 1]);
        ci[k + 1] = __fmaf_rn(ei, w.z, ci[k + 1]);
        dr[k + 1] = __fmaf_rn(orr, w.w, dr[k + 1]);
        di[k + 1] = __fmaf_rn(oi, w.w, di[k + 1]);
      }
    }
    auto put = [&](int r, float x, float y) {
      const int o = r / nrow;
      cluster.map_shared_rank(rows, o)[(r - o * nrow) * ld + zq + z] = make_float2(x, y);
    };
#pragma unroll
    for (int k = 0; k < PL_KC; k++) {
      const int ky = k0 + k;
      if (ky > Ky) break;
      // sum a e^{+i ky y} = C + i D, at -ky C - i D
      put(Ky + ky, __fadd_rn(cr[k], -di[k]), __fadd_rn(ci[k], dr[k]));
      if (ky) put(Ky - ky, __fadd_rn(cr[k], di[k]), __fadd_rn(ci[k], -dr[k]));
    }
  }
  cluster.sync();
  // z -> kz and the potential modes: item = (pair of kz, ky)
  double e[7] = {0, 0, 0, 0, 0, 0, 0};
  const int P = (b.K[0] + 1) * NY;
  for (int it = threadIdx.x; it < nkz * nr; it += T) {
    const int kp = it / nr, r = it - kp * nr, k0 = 2 * kp;
    const float4* t = tab1 + kp * (Hz + 1);
    const float2* in = rows + r * ld;
    float cr[2], ci[2], dr[2], di[2];
    const float2 a0 = in[0], ah = in[Hz];
    cr[0] = __fadd_rn(a0.x, ah.x);
    ci[0] = __fadd_rn(a0.y, ah.y);
    cr[1] = __fadd_rn(a0.x, -ah.x);
    ci[1] = __fadd_rn(a0.y, -ah.y);
    dr[0] = dr[1] = di[0] = di[1] = 0.f;
#pragma unroll 4
    for (int z = 1; z < Hz; z++) {
      const float2 p = in[z], m = in[Mz - z];
      const float4 w = t[z];
      const float er = __fadd_rn(p.x, m.x), ei = __fadd_rn(p.y, m.y), orr = __fadd_rn(p.x, -m.x),
                  oi = __fadd_rn(p.y, -m.y);
      cr[0] = __fmaf_rn(er, w.x, cr[0]);
      ci[0] = __fmaf_rn(ei, w.x, ci[0]);
      dr[0] = __fmaf_rn(orr, w.y, dr[0]);
      di[0] = __fmaf_rn(oi, w.y, di[0]);
      cr[1] = __fmaf_rn(er, w.z, cr[1]);
      ci[1] = __fmaf_rn(ei, w.z, ci[1]);
      dr[1] = __fmaf_rn(orr, w.w, dr[1]);
      di[1] = __fmaf_rn(oi, w.w, di[1]);
    }
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int kz = k0 + h;
      if (kz > Kz) break;
      // S(+kz) = C + i D, S(-kz) = C - i D
      const float pr = __fadd_rn(cr[h], -di[h]), pi = __fadd_rn(ci[h], dr[h]),
                  mr = __fadd_rn(cr[h], di[h]), mi = __fadd_rn(ci[h], -dr[h]);
      const int p = kx * NY + r0 + r;
      const float wp = b.wk[(long)(Kz + kz) * P + p], wm = kz ? b.wk[(long)(Kz - kz) * P + p] : 0.f;
      // potential modes: w conj(S)
      const float hpr = __fmul_rn(wp, pr), hpi = -__fmul_rn(wp, pi), hmr = __fmul_rn(wm, mr),
                  hmi = -__fmul_rn(wm, mi);
      pm[kz * nrow + r] = make_float4(__fadd_rn(hpr, hmr), __fadd_rn(hpi, hmi),
                                      __fadd_rn(hpr, -hmr), __fadd_rn(hpi, -hmi));
      if (measure) {
        const double x = kx * b.iL[0], y = (r0 + r - Ky) * b.iL[1], z = kz * b.iL[2];
        const double kk = x * x + y * y + z * z;
        const double ep = 6.283185307179586 * wp * ((double)pr * pr + (double)pi * pi),
                     em = 6.283185307179586 * wm * ((double)mr * mr + (double)mi * mi);
        if (kk > 0) {
          const double f = 1 / kk + b.pi2_over_a2, s = (ep + em) * f, df = (ep - em) * f;
          e[0] += ep + em;
          e[1] += s * x * x;
          e[2] += s * y * y;
          e[3] += s * z * z;
          e[4] += df * y * z;
          e[5] += df * x * z;
          e[6] += s * x * y;
        }
      }
    }
  }
  __syncthreads();
  // kz -> z: item = (pair of z, ky); column z to the CTA that holds it
  for (int it = threadIdx.x; it < nz * nr; it += T) {
    const int zp = it / nr, r = it - zp * nr, z0 = 2 * zp;
    const float4* t = tab2 + zp * (Kz + 1);
    const float4 v0 = pm[r];
    float er[2] = {v0.x, v0.x}, ei[2] = {v0.y, v0.y}, orr[2] = {0.f, 0.f}, oi[2] = {0.f, 0.f};
#pragma unroll 4
    for (int k = 1; k <= Kz; k++) {
      const float4 v = pm[k * nrow + r], w = t[k];
      er[0] = __fmaf_rn(v.x, w.x, er[0]);
      ei[0] = __fmaf_rn(v.y, w.x, ei[0]);
      orr[0] = __fmaf_rn(v.z, w.y, orr[0]);
      oi[0] = __fmaf_rn(v.w, w.y, oi[0]);
      er[1] = __fmaf_rn(v.x, w.z, er[1]);
      ei[1] = __fmaf_rn(v.y, w.z, ei[1]);
      orr[1] = __fmaf_rn(v.z, w.w, orr[1]);
      oi[1] = __fmaf_rn(v.w, w.w, oi[1]);
    }
    auto put = [&](int z, float x, float y) {
      const int o = z / nzq;
      cluster.map_shared_rank(cols, o)[(r0 + r) * nzq + z - o * nzq] = make_float2(x, y);
    };
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int z = z0 + h;
      if (z > Hz) break;
      // sum H e^{+i kz z} = E + i O, at M - z E - i O
      put(z, __fadd_rn(er[h], -oi[h]), __fadd_rn(ei[h], orr[h]));
      if (z > 0 && z < Hz) put(Mz - z, __fadd_rn(er[h], oi[h]), __fadd_rn(ei[h], -orr[h]));
    }
  }
  cluster.sync();
  // ky -> y: item = (chunk of PL_KC y, z)
  for (int it = threadIdx.x; it < ny * nzq; it += T) {
    const int ch = it / nzq, z = it - ch * nzq, y0 = ch * PL_KC;
    const float4* t = tab3 + ch * (Ky + 1) * (PL_KC / 2);
    const float2* in = cols + Ky * nzq + z;
    float er[PL_KC], ei[PL_KC], orr[PL_KC], oi[PL_KC];
    const float2 h0 = in[0];
#pragma unroll
    for (int k = 0; k < PL_KC; k++) {
      er[k] = h0.x;
      ei[k] = h0.y;
      orr[k] = oi[k] = 0.f;
    }
#pragma unroll 4
    for (int ky = 1; ky <= Ky; ky++) {
      const float2 u = in[ky * nzq], v = in[-ky * nzq];
      const float pr = __fadd_rn(u.x, v.x), pi = __fadd_rn(u.y, v.y), mr = __fadd_rn(u.x, -v.x),
                  mi = __fadd_rn(u.y, -v.y);
#pragma unroll
      for (int k = 0; k < PL_KC; k += 2) {
        const float4 w = t[ky * (PL_KC / 2) + k / 2];
        er[k] = __fmaf_rn(pr, w.x, er[k]);
        ei[k] = __fmaf_rn(pi, w.x, ei[k]);
        orr[k] = __fmaf_rn(mr, w.y, orr[k]);
        oi[k] = __fmaf_rn(mi, w.y, oi[k]);
        er[k + 1] = __fmaf_rn(pr, w.z, er[k + 1]);
        ei[k + 1] = __fmaf_rn(pi, w.z, ei[k + 1]);
        orr[k + 1] = __fmaf_rn(mr, w.w, orr[k + 1]);
        oi[k + 1] = __fmaf_rn(mi, w.w, oi[k + 1]);
      }
    }
    float2* o = A + zq + z;
#pragma unroll
    for (int k = 0; k < PL_KC; k++) {
      const int y = y0 + k;
      if (y > Hy) break;
      o[y * Mz] = make_float2(__fadd_rn(er[k], -oi[k]), __fadd_rn(ei[k], orr[k]));
      if (y > 0 && y < Hy)
        o[(My - y) * Mz] = make_float2(__fadd_rn(er[k], oi[k]), __fadd_rn(ei[k], -orr[k]));
    }
  }
  if (measure) {
    // fixed order: lanes by butterfly, then the warps in turn
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int m = 0; m < 7; m++) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) e[m] += __shfl_xor_sync(0xffffffffu, e[m], o);
      if (lane == 0) red[m][w] = e[m];
    }
    __syncthreads();
    if (threadIdx.x < 7) {
      double s = 0;
      for (int i = 0; i < T / 32; i++) s += red[threadIdx.x][i];
      b.ek_part[blockIdx.x * 7 + threadIdx.x] = s;
    }
  }
}

// A[kx][c] -> G[x][c]: the real part (the half kx >= 0 carries both signs)
// (half the threads where a batch fills the GPU: 256 ionic boxes 225 -> 189 us,
// 864 waters 3.2 -> 3.5, on grids of 1.75 points a mode; 223 and 4.5 at 1.86)
__global__ void __launch_bounds__(DF_THREADS) nf_idft_x_kernel(const NfBox* __restrict__ boxes) {
  after_previous();
  const NfBox& b = boxes[blockIdx.z];
  const int ncol = b.M[1] * b.M[2], c0 = blockIdx.x * DF_COLS, M = b.M[0], H = M / 2, K = b.K[0];
  if (c0 >= ncol) return;
  extern __shared__ float4 zs[];
  float2* in = reinterpret_cast<float2*>(zs);    // [K + 1][32]
  float4* tw = zs + (K + 1) * (DF_COLS / 2);     // [chunk][K + 1][NF_KC / 2]
  const int nch = H / NF_KC + 1, ntw = nch * (K + 1) * (NF_KC / 2);
  for (int i = threadIdx.x; i < (K + 1) * (DF_COLS / 2); i += (int)blockDim.x) {
    const int c = c0 + i % (DF_COLS / 2) * 2;
    if (c < ncol) nf_copy16(in + 2 * i, b.A + (long)(i / (DF_COLS / 2)) * ncol + c);
  }
  for (int i = threadIdx.x; i < ntw; i += (int)blockDim.x)
    nf_copy16(tw + i, reinterpret_cast<const float4*>(b.inv[0]) + i);
  nf_copy_wait();
  __syncthreads();
  const int lane = threadIdx.x & 31, c = c0 + lane;
  if (c >= ncol) return;
  for (int ch = threadIdx.x >> 5; ch < nch; ch += (int)blockDim.x / 32) {
    const float2* a = in + lane;
    const float4* t = tw + ch * (K + 1) * (NF_KC / 2);
    float e[NF_KC], o[NF_KC];
    const float a0 = a[0].x;
#pragma unroll
    for (int k = 0; k < NF_KC; k++) {
      e[k] = a0;
      o[k] = 0.f;
    }
#pragma unroll 4
    for (int kx = 1; kx <= K; kx++) {
      const float2 v = a[kx * DF_COLS];
#pragma unroll
      for (int k = 0; k < NF_KC; k += 2) {
        const float4 w = t[kx * (NF_KC / 2) + k / 2];
        e[k] = __fmaf_rn(v.x, w.x, e[k]);
        o[k] = __fmaf_rn(v.y, w.y, o[k]);
        e[k + 1] = __fmaf_rn(v.x, w.z, e[k + 1]);
        o[k + 1] = __fmaf_rn(v.y, w.w, o[k + 1]);
      }
    }
#pragma unroll
    for (int k = 0; k < NF_KC; k++) {
      const int x = ch * NF_KC + k;
      if (x > H) break;
      b.G[(long)x * ncol + c] = __fadd_rn(e[k], -o[k]);
      if (x > 0 && x < H) b.G[(long)(M - x) * ncol + c] = __fadd_rn(e[k], o[k]);
    }
  }
}

// --------------------------------------------------------- interpolation --
//
// Four charges at a time, eight lanes each: lane = z step of the window.  A
// load takes the 8 consecutive grid values of one (x, y) row for each of the
// four charges; the sums over y run per x with the 1-D weights and
// derivatives (each lane computes one of the 8 and passes it on by
// shuffles): two FMAs per load.
//
// The potential of the charge's own grid cell is subtracted from every value.  A
// constant has no gradient, but the window's derivatives add up to zero only to
// their rounding and the window's error, both of which it would multiply: the
// potential is mostly long waves, hundreds of times its change over the window.
// Of a brine's k-space force (12544 sites) the error fell from 1.2e-6 to 0.9e-6.
struct NfWeights {
  float w[3], g[3];   // window and derivative of this lane's step, x y z

  __device__ __forceinline__ void set(const NfBox& b, int l8, float fx, float fy, float fz) {
    const float f[3] = {fx, fy, fz};
    // this lane's window step: offset l8 - 3 of [-3, 4]
    const float o = (float)(l8 - (W / 2 - 1));
#pragma unroll
    for (int d = 0; d < 3; d++) {
      const float t = __fadd_rn(f[d], -o);
      float s;
      w[d] = nf_window(__fmul_rn(t, 2.f / W), b.nb[d], s);
      // d phi / dt = -beta (2/w)^2 t phi / s; s bounded below (the window
      // ends at phi = e^-beta with a vertical tangent)
      g[d] = __fmul_rn(__fmul_rn(b.db[d], t), __fmul_rn(w[d], nf_rcp(fmaxf(s, 0.02f))));
    }
  }
};

// The force of a charge onto its site: lane l8 = 0, 1, 2 of its eight holds
// component l8 (no other lane touches it in the launch).  The old value is
// read when the charge is taken up, long before the sum is known: read at the
// end, every four charges waited for one round trip to memory.
struct NfForce {
  double* at;
  double old;

  __device__ __forceinline__ void begin(const NfBox& b, double* f, int site, int sub, int l8,
                                        bool on) {
    at = on && l8 < 3 ? f + (sub ? 3 * (long)b.ns : 0) + 3 * (long)site + l8 : nullptr;
    old = at ? *at : 0.0;
  }

  // F = -q grad of the potential, grid steps -> A
  __device__ __forceinline__ void end(const NfBox& b, float q, int l8, float Fx, float Fy,
                                      float Fz) {
#pragma unroll
    for (int d = 4; d > 0; d >>= 1) {
      Fx = __fadd_rn(Fx, __shfl_xor_sync(0xffffffffu, Fx, d));
      Fy = __fadd_rn(Fy, __shfl_xor_sync(0xffffffffu, Fy, d));
      Fz = __fadd_rn(Fz, __shfl_xor_sync(0xffffffffu, Fz, d));
    }
    const float v = l8 == 0 ? Fx : (l8 == 1 ? Fy : Fz);
    if (at) *at = old + (double)__fmul_rn(v, __fmul_rn(q, -b.fac[l8]));
  }
};

// Dense boxes: a CTA per tile of 8 x 8 x 8 grid steps takes the tile's
// potential with its halo (15 x 15 x 16 points) into shared memory; the
// charges whose grid cell lies in the tile come from the cell list as in the
// spreading, and every row of a window is a shared-memory load at a fixed
// offset from the charge's first.  Bound by the shared-memory wavefronts (64
// loads of four unaligned 32-byte rows each per four charges): 45 us on 32768
// waters, 10 us on 864, with the charge's own potential taken out; before that 35
// and 8.8, where reading the rows from memory (below) took 36 and 12.  Two CTAs an
// SM: left to itself the compiler takes 80 registers and spills, 1 us more on 12544
// sites.
constexpr int IT_LD = 2 * TILE, IT_PL = IT_LD * IT_LD;

__global__ void __launch_bounds__(SP_WARPS * 32, 2)
    nf_interp_tile_kernel(const NfBox* __restrict__ boxes, double* __restrict__ f_or_null) {
  after_previous();
  const NfBox& b = boxes[blockIdx.z];
  const int ntz = (b.M[2] + TILE - 1) / TILE, nty = (b.M[1] + TILE - 1) / TILE,
            ntx = (b.M[0] + TILE - 1) / TILE, tile = blockIdx.x;
  if (!b.dense || tile >= ntx * nty * ntz) return;
  __shared__ __align__(16) float ph[15 * IT_PL];   // [x][y][z] from (x0 - 3, y0 - 3, z0 - 4)
  __shared__ int4 que[SP_WARPS][64];               // fixed-point position, charge
  __shared__ int qix[SP_WARPS][64];                // site, sub in bit 30
  __shared__ int4 runs[SP_WARPS][32];
  const int x0 = tile / (nty * ntz) * TILE, y0 = tile / ntz % nty * TILE, z0 = tile % ntz * TILE;
  const int Mx = b.M[0], My = b.M[1], Mz = b.M[2];
  for (int i = threadIdx.x; i < 15 * 15 * 4; i += SP_WARPS * 32) {
    const int k = i % 4, y = i / 4 % 15, x = i / 60;
    int gx = x0 + x - 3, gy = y0 + y - 3, gz = z0 + 4 * k - 4;
    gx += gx < 0 ? Mx : (gx >= Mx ? -Mx : 0);
    gy += gy < 0 ? My : (gy >= My ? -My : 0);
    gz += gz < 0 ? Mz : (gz >= Mz ? -Mz : 0);
    nf_copy16(ph + x * IT_PL + y * IT_LD + 4 * k, b.G + ((long)gx * My + gy) * Mz + gz);
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
  double* f = f_or_null ? f_or_null : b.f;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, l8 = lane & 7, grp = lane >> 3;

  int qh = 0, qn = 0;
  auto flush = [&](int cnt) {
    for (int i = 0; i < cnt; i += 4) {
      const bool on = i + grp < cnt;
      const int e = (qh + (on ? i + grp : i)) & 63;
      const int4 r = que[warp][e];
      const int ix = qix[warp][e];
      NfForce out;
      out.begin(b, f, ix & 0x3fffffff, ix >> 30, l8, on);
      float fx, fy, fz;
      const int jx = nf_cell(r.x, Mx, fx) - x0, jy = nf_cell(r.y, My, fy) - y0,
                jz = nf_cell(r.z, Mz, fz) - z0;
      NfWeights k;
      k.set(b, l8, fx, fy, fz);
      const float* row = ph + jx * IT_PL + jy * IT_LD + jz + 1 + l8;
      const float home = ph[(jx + W / 2 - 1) * IT_PL + (jy + W / 2 - 1) * IT_LD + jz + W / 2];
      float wy[W], gy[W];
#pragma unroll
      for (int c = 0; c < W; c++) {
        wy[c] = __shfl_sync(0xffffffffu, k.w[1], c, 8);
        gy[c] = __shfl_sync(0xffffffffu, k.g[1], c, 8);
      }
      float P = 0.f, Px = 0.f, Py = 0.f;
#pragma unroll
      for (int a = 0; a < W; a++) {
        const float vx = __shfl_sync(0xffffffffu, k.w[0], a, 8),
                    hx = __shfl_sync(0xffffffffu, k.g[0], a, 8);
        float u = 0.f, v = 0.f;
#pragma unroll
        for (int c = 0; c < W; c++) {
          const float g = __fadd_rn(row[a * IT_PL + c * IT_LD], -home);
          u = __fmaf_rn(wy[c], g, u);
          v = __fmaf_rn(gy[c], g, v);
        }
        P = __fmaf_rn(vx, u, P);
        Px = __fmaf_rn(hx, u, Px);
        Py = __fmaf_rn(vx, v, Py);
      }
      out.end(b, __int_as_float(r.w), l8, __fmul_rn(Px, k.w[2]), __fmul_rn(Py, k.w[2]),
              __fmul_rn(P, k.g[2]));
    }
  };

  NfRuns R;
  R.set(b, x0, y0, z0, 0, TILE);
  const int step = 32 * SP_WARPS, first = 32 * warp;
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  for (int cb = 0; cb < R.ncol; cb += 32) {
    const int total = R.columns(b, cb, lane, runs[warp]);
    int jn = first + lane < total ? NfRuns::site(runs[warp], first + lane) : -1;
    int4 pn = jn >= 0 ? b.pj[jn] : make_int4(0, 0, 0, 0);
    for (int kb = first; kb < total; kb += step) {
      const int j = jn, kn = kb + step + lane;
      const int4 p = pn;
      jn = kn < total ? NfRuns::site(runs[warp], kn) : -1;
      pn = jn >= 0 ? b.pj[jn] : make_int4(0, 0, 0, 0);
      for (int sub = 0; sub < b.nsub; sub++) {
        int4 r;
        const float q = nf_charge(b, j, p, sub, r);
        // the charges whose grid cell lies in the tile: every charge is in one
        const int jx = (int)__umulhi((unsigned)r.x, Mx) - x0,
                  jy = (int)__umulhi((unsigned)r.y, My) - y0,
                  jz = (int)__umulhi((unsigned)r.z, Mz) - z0;
        const bool keep = q != 0.f && (unsigned)jx < TILE && (unsigned)jy < TILE &&
                          (unsigned)jz < TILE;
        const unsigned m = __ballot_sync(0xffffffffu, keep);
        if (keep) {
          const int e = (qh + qn + __popc(m & ((1u << lane) - 1u))) & 63;
          que[warp][e] = make_int4(r.x, r.y, r.z, __float_as_int(q));
          qix[warp][e] = b.order[j] | sub << 30;
        }
        qn += __popc(m);
        __syncwarp();
        if (qn >= 32) {
          flush(32);
          qh = (qh + 32) & 63;
          qn -= 32;
        }
      }
    }
  }
  if (qn > 0) flush(qn);
}

// Sparse boxes (a few charges a tile): a warp per 16 sorted sites, the rows
// from memory.  The warps wait for these loads, so eight CTAs an SM, at 64
// registers and a few spills: 256 ionic boxes 330 -> 216 us (at 80 registers
// five; ten CTAs spill more, 387).
constexpr int IP_WARPS = 4, IP_SITES = 16;

__global__ void __launch_bounds__(IP_WARPS * 32, 8)
    nf_interp_kernel(const NfBox* __restrict__ boxes, double* __restrict__ f_or_null) {
  after_previous();
  const NfBox& b = boxes[blockIdx.z];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int t0 = (blockIdx.x * IP_WARPS + warp) * IP_SITES;
  if (b.dense || t0 >= b.ns) return;
  __shared__ int sidx[IP_WARPS][IP_SITES];
  double* f = f_or_null ? f_or_null : b.f;
  const float* __restrict__ G = b.G;
  const int t = t0 + lane;
  const bool in = lane < IP_SITES && t < b.ns;
  const int4 p = in ? b.pj[t] : make_int4(0, 0, 0, 0);
  const int site = in ? b.order[t] : 0;
  const int Mx = b.M[0], My = b.M[1], Mz = b.M[2];
  const int l8 = lane & 7, grp = lane >> 3;
  for (int sub = 0; sub < b.nsub; sub++) {
    int4 r;
    const float q = nf_charge(b, in ? t : -1, p, sub, r);
    float frx, fry, frz;
    const int ix = nf_cell(r.x, Mx, frx), iy = nf_cell(r.y, My, fry), iz = nf_cell(r.z, Mz, frz);
    const unsigned m = __ballot_sync(0xffffffffu, q != 0.f);
    const int n = __popc(m);
    __syncwarp();
    if (q != 0.f) sidx[warp][__popc(m & ((1u << lane) - 1u))] = lane;
    __syncwarp();
    for (int i = 0; i < n; i += 4) {
      const bool on = i + grp < n;
      const int src = sidx[warp][on ? i + grp : i];
      const int jx = __shfl_sync(0xffffffffu, ix, src), jy = __shfl_sync(0xffffffffu, iy, src),
                jz = __shfl_sync(0xffffffffu, iz, src);
      const float fx = __shfl_sync(0xffffffffu, frx, src), fy = __shfl_sync(0xffffffffu, fry, src),
                  fz = __shfl_sync(0xffffffffu, frz, src);
      const float qq = __shfl_sync(0xffffffffu, q, src);
      NfForce out;
      out.begin(b, f, __shfl_sync(0xffffffffu, site, src), sub, l8, on);
      NfWeights k;
      k.set(b, l8, fx, fy, fz);
      int ax = jx + l8 - (W / 2 - 1), ay = jy + l8 - (W / 2 - 1), az = jz + l8 - (W / 2 - 1);
      ax += ax < 0 ? Mx : (ax >= Mx ? -Mx : 0);
      ay += ay < 0 ? My : (ay >= My ? -My : 0);
      az += az < 0 ? Mz : (az >= Mz ? -Mz : 0);
      const float home = __ldg(G + ((long)jx * My + jy) * Mz + jz);
      ax *= My * Mz;
      ay *= Mz;
      float wy[W], gy[W];
      int yo[W];
#pragma unroll
      for (int c = 0; c < W; c++) {
        wy[c] = __shfl_sync(0xffffffffu, k.w[1], c, 8);
        gy[c] = __shfl_sync(0xffffffffu, k.g[1], c, 8);
        yo[c] = __shfl_sync(0xffffffffu, ay, c, 8) + az;
      }
      float P = 0.f, Px = 0.f, Py = 0.f;
#pragma unroll
      for (int a = 0; a < W; a++) {
        const float* row = G + __shfl_sync(0xffffffffu, ax, a, 8);
        const float vx = __shfl_sync(0xffffffffu, k.w[0], a, 8),
                    hx = __shfl_sync(0xffffffffu, k.g[0], a, 8);
        float u = 0.f, v = 0.f;
#pragma unroll
        for (int c = 0; c < W; c++) {
          const float g = __fadd_rn(__ldg(row + yo[c]), -home);
          u = __fmaf_rn(wy[c], g, u);
          v = __fmaf_rn(gy[c], g, v);
        }
        P = __fmaf_rn(vx, u, P);
        Px = __fmaf_rn(hx, u, Px);
        Py = __fmaf_rn(vx, v, Py);
      }
      out.end(b, qq, l8, __fmul_rn(Px, k.w[2]), __fmul_rn(Py, k.w[2]), __fmul_rn(P, k.g[2]));
    }
  }
}

// whether a Drude displacement exceeds the margin of the spreading's lookup
__global__ void nf_far_kernel(int ns, const float4* __restrict__ pdj, float lim,
                              int* __restrict__ far) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= ns) return;
  const float4 d = pdj[t];
  // written so that a NaN counts as far
  if (!(fabsf(d.x) <= lim && fabsf(d.y) <= lim && fabsf(d.z) <= lim)) *far = 1;
}

// -------------------------------------------------------------- host side --

// the grid of K modes on an edge: the next multiple of 4 of `points` per mode,
// (2 K + 1) modes, at least a tile and a window (16)
static int nf_points(int K, double points) {
  const int m = ((int)std::ceil(points * (2 * K + 1)) + 3) / 4 * 4;
  return m < 16 ? 16 : m;
}

double nf_beta(int M, int K) {
  // pi w (1 - 1/(2 sigma)) is the band limit of the window for a grid of
  // sigma points per mode; 8 % above it the forces, which differentiate the
  // window, are the most accurate
  const double sigma = (double)M / (2 * K + 1);
  return 1.08 * 3.14159265358979324 * W * (1 - 1 / (2 * sigma));
}

// the window's transform at the modes 0..K of an M-point edge by the
// midpoint rule in th, t = (w/2) sin th (the integrand and its slope are
// below e^-beta at the ends: 200 points leave an error below 1e-13)
static std::vector<double> nf_hat(double beta, int M, int K) {
  const double pi = 3.14159265358979324;
  const int n = 200;
  std::vector<double> g(n), x(n), h(K + 1, 0.0);
  for (int i = 0; i < n; i++) {
    const double th = pi * ((i + 0.5) / n - 0.5);
    g[i] = std::exp(beta * (std::cos(th) - 1)) * std::cos(th) * pi / n * 0.5 * W;
    x[i] = 2 * pi * 0.5 * W * std::sin(th) / M;
  }
  for (int k = 0; k <= K; k++)
    for (int i = 0; i < n; i++) h[k] += g[i] * std::cos(k * x[i]);
  return h;
}

void nf_tables(const int K[3], const int M[3], const std::vector<int4>& kvec,
               const std::vector<double>& ekk, std::vector<float2> fwd[3],
               std::vector<float2> inv[3], std::vector<float>* wk) {
  const double pi = 3.14159265358979324;
  std::vector<double> dec[3];
  for (int d = 0; d < 3; d++) {
    for (double h : nf_hat(nf_beta(M[d], K[d]), M[d], K[d])) dec[d].push_back(1 / (h * h));
    const int KC = d == 2 ? 2 : (d == 1 ? PL_KC : NF_KC), H = M[d] / 2;
    std::vector<float2> cs(M[d]);
    for (int i = 0; i < M[d]; i++)
      cs[i] = make_float2((float)std::cos(2 * pi * i / M[d]), (float)std::sin(2 * pi * i / M[d]));
    auto entry = [&](int a, int k) { return cs[(long)a * k % M[d]]; };
    for (int k0 = 0; k0 <= K[d]; k0 += KC)
      for (int a = 0; a <= H; a++)
        for (int k = 0; k < KC; k++) {
          float2 e = entry(a, k0 + k);
          // a = 0 and M/2 have no partner: their odd part is zero
          if (a == 0 || a == H) e.y = 0.f;
          fwd[d].push_back(e);
        }
    for (int a0 = 0; a0 <= H; a0 += KC)
      for (int k = 0; k <= K[d]; k++)
        for (int a = 0; a < KC; a++) inv[d].push_back(entry(a0 + a, k));
  }
  const int NY = 2 * K[1] + 1, P = (K[0] + 1) * NY;
  wk->assign((size_t)P * (2 * K[2] + 1), 0.f);
  for (size_t i = 0; i < kvec.size(); i++) {
    const int4 v = kvec[i];
    const int p = v.x * NY + v.y + K[1];
    (*wk)[(size_t)(v.z + K[2]) * P + p] =
        (float)(ekk[i] * dec[0][std::abs(v.x)] * dec[1][std::abs(v.y)] * dec[2][std::abs(v.z)] /
                (2 * pi));
  }
}

// shared memory of the plane kernel: potential modes, tables, the plane
static size_t nf_plane_smem(const int K[3], const int M[3], int cs) {
  const int NY = 2 * K[1] + 1, Hy = M[1] / 2, Hz = M[2] / 2;
  const size_t tab = (size_t)(K[1] / PL_KC + 1) * (Hy + 1) * (PL_KC / 2) +
                     (size_t)(K[2] / 2 + 1) * (Hz + 1) + (size_t)(Hz / 2 + 1) * (K[2] + 1) +
                     (size_t)(Hy / PL_KC + 1) * (K[1] + 1) * (PL_KC / 2);
  const int nrow = (NY + cs - 1) / cs;
  return 16 * ((size_t)(K[2] + 1) * nrow + tab) + 8 * ((size_t)(M[2] + 1) * nrow + 1) +
         8 * (size_t)(M[1] > NY ? M[1] : NY) * (M[2] / cs);
}
static size_t nf_x_smem(int K, int M) {
  return 4 * (size_t)DF_COLS * M + 16 * (size_t)(K / NF_KC + 1) * (M / 2 + 1) * (NF_KC / 2);
}
static size_t nf_ix_smem(int K, int M) {
  return 8 * (size_t)DF_COLS * (K + 1) + 16 * (size_t)(M / 2 / NF_KC + 1) * (K + 1) * (NF_KC / 2);
}

// a CTA's 227 KB less the kernels' static part
constexpr int NF_MAX_SMEM = 225 * 1024;

// The grids M of the modes K; false where the transforms do not fit a CTA.  The
// window's error at the highest modes falls with the points per mode and the
// transforms grow with their cube.  At 1.86 the k-space force is closer to the
// 64-bit sums than the direct tensor-core passes take it, in every one of 46 boxes
// of 650 to 98000 sites (water, brine, Drude water, TIP4P; |n| 6 to 20); at 1.75 it
// was 1.4 and 2.6 times as far for brines with |n| <= 12 and 20.  1.75 only for the
// largest sets, which fit no more points (|n| 44 and 45).
bool nf_grids(const int K[3], int M[3]) {
  for (double points : {1.86, 1.75}) {
    for (int d = 0; d < 3; d++) M[d] = nf_points(K[d], points);
    if (nf_plane_smem(K, M, NF_CS) <= NF_MAX_SMEM && nf_x_smem(K[0], M[0]) <= NF_MAX_SMEM &&
        nf_ix_smem(K[0], M[0]) <= NF_MAX_SMEM)
      return true;
  }
  return false;
}

static int nf_tiles(const NfBox& b) {
  return cdiv(b.M[0], TILE) * cdiv(b.M[1], TILE) * cdiv(b.M[2], TILE);
}

// a box with at least 12 charges a tile on average shares a tile among eight
// warps (spreading) and keeps it in shared memory (interpolation): 32768
// waters hold 133, 216 waters 15, the ionic boxes of a batch about 4
int nf_dense(int nq, const int M[3]) {
  return (double)nq * TP >= 12.0 * M[0] * M[1] * M[2] ? 1 : 0;
}

void nf_launch(const NfBox& b, NfGrid* g) {
  auto up = [](int& a, int v) { a = a > v ? a : v; };
  up(g->spread, b.dense ? nf_tiles(b) : cdiv(nf_tiles(b), SP_WARPS));
  up(g->x, cdiv((long)b.M[1] * b.M[2], DF_COLS));
  up(g->plane, NF_CS * (b.K[0] + 1));
  if (b.dense) up(g->interp_tile, nf_tiles(b));
  else up(g->interp, cdiv(b.ns, IP_WARPS * IP_SITES));
  up(g->sx, (int)nf_x_smem(b.K[0], b.M[0]));
  up(g->six, (int)nf_ix_smem(b.K[0], b.M[0]));
  up(g->splane, (int)nf_plane_smem(b.K, b.M, NF_CS));
  up(g->splane_few, (int)nf_plane_smem(b.K, b.M, NF_CSB));
}

// the same limit whatever the box: a captured launch of a larger box must not
// find the limit a smaller one set
static cudaError_t nf_smem(const void* kernel, int bytes) {
  return bytes <= 47 * 1024
             ? cudaSuccess
             : cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    NF_MAX_SMEM);
}

cudaError_t k_nf_far(const Launch& L, int ns, const float4* pdj, float lim, int* far) {
  cudaError_t e = cudaMemsetAsync(far, 0, sizeof(int), L.s);
  if (e != cudaSuccess) return e;
  nf_far_kernel<<<cdiv(ns, 256), 256, 0, L.s>>>(ns, pdj, lim, far);
  LAUNCHED(L);
  return cudaGetLastError();
}

cudaError_t k_nf_forward(const Launch& L, const NfBox* d, int nbox, const NfGrid& g) {
  const int st = SP_WARPS * SP_ST * (int)sizeof(float);
  cudaError_t e = cudaFuncSetAttribute(nf_spread_kernel,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, st);
  if (e != cudaSuccess) return e;
  nf_spread_kernel<<<dim3(g.spread, 1, nbox), SP_WARPS * 32, st, L.s>>>(d);
  LAUNCHED(L);
  e = nf_smem((const void*)nf_dft_x_kernel, g.sx);
  if (e != cudaSuccess) return e;
  launch_after(L, nf_dft_x_kernel, dim3(g.x, 1, nbox), DF_THREADS, g.sx, d);
  LAUNCHED(L);
  return cudaGetLastError();
}

// more CTAs than two waves of eight an SM: throughput counts, not the latency of
// one
static bool nf_many(long ctas) { return ctas > 16L * PARTITION_SMS; }

cudaError_t k_nf_modes(const Launch& L, const NfBox* d, int nbox, const NfGrid& g, bool measure) {
  const bool many = !measure && nf_many((long)g.plane * nbox) && g.splane_few <= NF_MAX_SMEM;
  cudaError_t e = many ? nf_smem((const void*)nf_plane_kernel<NF_CSB, NF_TB>, g.splane_few)
                       : nf_smem((const void*)nf_plane_kernel<NF_CS, PL_THREADS>, g.splane);
  if (e != cudaSuccess) return e;
  if (many)
    launch_after(L, nf_plane_kernel<NF_CSB, NF_TB>, dim3(g.plane / NF_CS * NF_CSB, 1, nbox), NF_TB,
                 g.splane_few, d, measure);
  else
    launch_after(L, nf_plane_kernel<NF_CS, PL_THREADS>, dim3(g.plane, 1, nbox), PL_THREADS, g.splane,
                 d, measure);
  LAUNCHED(L);
  return cudaGetLastError();
}

cudaError_t k_nf_back(const Launch& L, const NfBox* d, int nbox, const NfGrid& g) {
  cudaError_t e = nf_smem((const void*)nf_idft_x_kernel, g.six);
  if (e != cudaSuccess) return e;
  launch_after(L, nf_idft_x_kernel, dim3(g.x, 1, nbox),
               nf_many((long)g.x * nbox) ? DF_THREADS / 2 : DF_THREADS, g.six, d);
  LAUNCHED(L);
  return cudaGetLastError();
}

cudaError_t k_nf_interp(const Launch& L, const NfBox* d, int nbox, const NfGrid& g, double* f) {
  if (g.interp_tile > 0) {
    nf_interp_tile_kernel<<<dim3(g.interp_tile, 1, nbox), SP_WARPS * 32, 0, L.s>>>(d, f);
    LAUNCHED(L);
  }
  if (g.interp > 0) {
    nf_interp_kernel<<<dim3(g.interp, 1, nbox), IP_WARPS * 32, 0, L.s>>>(d, f);
    LAUNCHED(L);
  }
  return cudaGetLastError();
}

}  // namespace mg
