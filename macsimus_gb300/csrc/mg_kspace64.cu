// Ewald k-space sums of the FP64 path and of the adjoint, as direct sums
// (sim/ewpass2m.c, sim/ewpass2.c, sim/ewaldf.c).
//
// Every k of the set is one of a row (kx, ky) of consecutive kz.  With
// A_j(row) = q_j X_j(kx) Y_j(ky) = (ax, ay) and Z_j(kz) = (c, s), Z(-kz) =
// conj Z(kz), both signs of kz come from four real sums over the charges,
//   P = (sum ax c, sum ax s),  Q = (sum ay s, sum ay c),
//   S(row, kz) = (P.x - Q.x, P.y + Q.y),  S(row, -kz) = (P.x + Q.x, Q.y - P.y),
// and, with W = ekk conj(S), P = W+ + W-, M = W+ - W- of the two signs,
//   H  = sum (P.x c - M.y s, M.x s + P.y c),  Hz = sum kz (M.x c - P.y s, P.x s + M.y c),
//   F_j = sum over rows of (kx Im(A H) / Lx, ky Im(A H) / Ly, Im(A Hz) / Lz).
// What bounds all of it is the FP64 pipe (a warp's instruction holds an SM's
// for 16 cycles), so an item (row, |kz|) is stored and multiplied only where
// the set has it: no tiles, no padding.  Tasks of up to K64_RUN items of one
// row, sorted by length, are a lane each in pass 1; rows, sorted by length,
// are dealt to lanes in pass 2.  (Tiles of 64 rows by 16 kz with a complex
// product per kz took 695 us on 864 waters and |n| <= 8, on 15 CTAs, and
// pass 2 285 us; these 29 + 10 and 46.)
#include <algorithm>

#include "mg_internal.h"

namespace mg {

constexpr int K64_WARPS = 8;
constexpr int K64_THREADS = 32 * K64_WARPS;

__device__ __forceinline__ double2 k64_mul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

// Pass 1: the lanes of a CTA take 32 tasks, its warps the charges of its chunk
// in turn; part [chunk][item][4] gets (P.x, P.y, Q.x, Q.y).  ADJ: the same
// sums of w A and g_z A, w = g_x kx/Lx + g_y ky/Ly: part [chunk][item][8].
template <bool ADJ>
__global__ void __launch_bounds__(K64_THREADS)
    sk64_kernel(const __grid_constant__ KArgs a, const __grid_constant__ K64 k,
                const double2* __restrict__ tab, const double* __restrict__ g, int nch) {
  constexpr int NV = ADJ ? 8 : 4;
  __shared__ double red[K64_WARPS][NV][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int task = blockIdx.x * 32 + lane;
  const KTask64 t = k.tasks[min(task, k.ntask - 1)];
  const int nmax = k.tasks[blockIdx.x * 32].n;   // sorted: the longest of the 32
  const int oy = a.Kx + 1 + a.Ky, oz = a.Kx + 2 * a.Ky + 2 + a.Kz;
  const int j0 = (int)((long)a.nq * blockIdx.y / nch), j1 = (int)((long)a.nq * (blockIdx.y + 1) / nch);
  const double kx = t.kx / a.Lx, ky = t.ky / a.Ly;
  double acc[K64_RUN][NV];
#pragma unroll
  for (int m = 0; m < K64_RUN; m++)
#pragma unroll
    for (int v = 0; v < NV; v++) acc[m][v] = 0;
  for (int j = j0 + warp; j < j1; j += K64_WARPS) {
    const double2* __restrict__ R = tab + (long)j * a.row;
    const double2 A = k64_mul(R[t.kx], R[oy + t.ky]);
    double2 u = A, w = A;
    if constexpr (ADJ) {
      const double* gj = g + 3 * (long)a.qsite[j];
      const double wj = gj[0] * kx + gj[1] * ky, gz = gj[2];
      u = make_double2(wj * A.x, wj * A.y);
      w = make_double2(gz * A.x, gz * A.y);
    }
#pragma unroll
    for (int m = 0; m < K64_RUN; m++)
      if (m < nmax) {
        const double2 z = R[oz + min(t.z0 + m, a.Kz)];
        acc[m][0] = fma(u.x, z.x, acc[m][0]);
        acc[m][1] = fma(u.x, z.y, acc[m][1]);
        acc[m][2] = fma(u.y, z.y, acc[m][2]);
        acc[m][3] = fma(u.y, z.x, acc[m][3]);
        if constexpr (ADJ) {
          acc[m][4] = fma(w.x, z.x, acc[m][4]);
          acc[m][5] = fma(w.x, z.y, acc[m][5]);
          acc[m][6] = fma(w.y, z.y, acc[m][6]);
          acc[m][7] = fma(w.y, z.x, acc[m][7]);
        }
      }
  }
  // over the warps, in warp order
#pragma unroll
  for (int m = 0; m < K64_RUN; m++)
    if (m < nmax) {
#pragma unroll
      for (int v = 0; v < NV; v++) red[warp][v][lane] = acc[m][v];
      __syncthreads();
      const int v = warp;
      if (v < NV && task < k.ntask && m < t.n) {
        double s = 0;
#pragma unroll
        for (int q = 0; q < K64_WARPS; q++) s += red[q][v][lane];
        k.part[((long)blockIdx.y * k.nitem + t.item0 + m) * NV + v] = s;
      }
      __syncthreads();
    }
}

// items per CTA of the reductions, and the warps that share the chunks of each
// (one warp alone keeps its quarter of the FP64 pipe busy for 18 us)
constexpr int K64_RED = 32, K64_RW = 8;

// the chunks' sums of item i, NV values, in warp 0 (every warp calls)
template <int NV>
__device__ __forceinline__ void k64_gather(const K64& k, int nch, int i, double (&s)[NV]) {
  __shared__ double red[K64_RW][NV][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
  for (int v = 0; v < NV; v++) s[v] = 0;
  if (i < k.nitem)
#pragma unroll 2
    for (int c = warp; c < nch; c += K64_RW) {
      const double2* p = reinterpret_cast<const double2*>(k.part + ((long)c * k.nitem + i) * NV);
#pragma unroll
      for (int v = 0; v < NV / 2; v++) {
        const double2 u = p[v];
        s[2 * v] += u.x;
        s[2 * v + 1] += u.y;
      }
    }
#pragma unroll
  for (int v = 0; v < NV; v++) red[warp][v][lane] = s[v];
  __syncthreads();
  if (warp == 0)
#pragma unroll
    for (int v = 0; v < NV; v++)
      for (int w = 1; w < K64_RW; w++) s[v] += red[w][v][lane];
}

__device__ __forceinline__ double4 k64_pm(double ep, double em, double2 sp, double2 sm) {
  // W = ekk conj(S): sums and differences of both signs of kz
  const double2 wp = make_double2(ep * sp.x, -ep * sp.y), wm = make_double2(em * sm.x, -em * sm.y);
  return make_double4(wp.x + wm.x, wp.y + wm.y, wp.x - wm.x, wp.y - wm.y);
}

// S(k) from the chunks' sums (fixed order), {P, M} of every item for pass 2;
// energy and virial (E1 = |S|^2 ekk, ptf = 1/kk + (pi/alpha)^2) per CTA
__global__ void __launch_bounds__(32 * K64_RW)
    sk64_reduce_kernel(const __grid_constant__ KArgs a, const __grid_constant__ K64 k, int nch,
                       bool measure, double pi2_over_a2) {
  const int i = blockIdx.x * K64_RED + (threadIdx.x & 31);
  double e[7] = {0, 0, 0, 0, 0, 0, 0};
  double s[4];
  k64_gather(k, nch, i, s);
  if (threadIdx.x >= 32) return;
  if (i < k.nitem) {
    const KItem64 it = k.items[i];
    const double2 S[2] = {make_double2(s[0] - s[2], s[1] + s[3]),
                          make_double2(s[0] + s[2], s[3] - s[1])};
    const int kn[2] = {it.kp, it.km};
    double ek[2] = {0, 0};
#pragma unroll
    for (int q = 0; q < 2; q++)
      if (kn[q] >= 0) {
        ek[q] = a.ekk[kn[q]];
        a.S[2 * (long)kn[q]] = S[q].x;
        a.S[2 * (long)kn[q] + 1] = S[q].y;
        if (measure) {
          const KRow64 r = k.rows[it.row];
          const double kx = r.kx / a.Lx, ky = r.ky / a.Ly, kz = (q ? -it.z : it.z) / a.Lz;
          const double kk = kx * kx + ky * ky + kz * kz;
          const double E1 = (S[q].x * S[q].x + S[q].y * S[q].y) * ek[q];
          const double ptf = 1 / kk + pi2_over_a2;
          e[0] += E1;
          e[1] += E1 * ptf * kx * kx;
          e[2] += E1 * ptf * ky * ky;
          e[3] += E1 * ptf * kz * kz;
          e[4] += E1 * ptf * ky * kz;
          e[5] += E1 * ptf * kx * kz;
          e[6] += E1 * ptf * kx * ky;
        }
      }
    k.pm[i] = k64_pm(ek[0], ek[1], S[0], S[1]);
  }
  if (!measure) return;
#pragma unroll
  for (int m = 0; m < 7; m++) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) e[m] += __shfl_xor_sync(0xffffffffu, e[m], o);
    if (threadIdx.x == 0) a.ek_part[blockIdx.x * 7 + m] = e[m];
  }
}

// T(k) = sum_j q_j (g_j.k/L) Phi_j(k): {P, M} of ekk conj(T) of every item
__global__ void __launch_bounds__(32 * K64_RW)
    tk64_reduce_kernel(const __grid_constant__ KArgs a, const __grid_constant__ K64 k, int nch) {
  const int i = blockIdx.x * K64_RED + (threadIdx.x & 31);
  double s[8];
  k64_gather(k, nch, i, s);
  if (threadIdx.x >= 32 || i >= k.nitem) return;
  const KItem64 it = k.items[i];
  const double kz = it.z / a.Lz;
  const double2 tp = make_double2((s[0] - s[2]) + kz * (s[4] - s[6]), (s[1] + s[3]) + kz * (s[5] + s[7]));
  const double2 tm = make_double2((s[0] + s[2]) - kz * (s[4] + s[6]), (s[3] - s[1]) - kz * (s[7] - s[5]));
  k.pt[i] = k64_pm(it.kp >= 0 ? a.ekk[it.kp] : 0, it.km >= 0 ? a.ekk[it.km] : 0, tp, tm);
}

// Pass 2: C charges per CTA, a lane per charge and one of 32/C rows, the rows
// dealt over the warps; Z and kz Z of the charges in shared memory.  ADJ: the
// charge gradients instead of the forces: psi = Re(A H), F^k and, with the
// {P, M} of T, Im(conj(A) T) from one more H.
template <bool ADJ>
__global__ void __launch_bounds__(K64_THREADS)
    kf64_kernel(const __grid_constant__ KArgs a, const __grid_constant__ K64 k,
                const double2* __restrict__ tab, int C, const double* __restrict__ g,
                double* __restrict__ dEq, double* __restrict__ dLq) {
  constexpr int NV = ADJ ? 5 : 3;
  extern __shared__ __align__(16) unsigned char k64_smem[];
  const int nz = a.Kz + 1;
  double2* Zs = reinterpret_cast<double2*>(k64_smem);       // [nz][C]
  double2* Zk = Zs + (size_t)nz * C;                          // [nz][C]
  double* red = reinterpret_cast<double*>(Zk + (size_t)nz * C);   // [warps][NV][32]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int jb = blockIdx.x * C, c = lane & (C - 1), h = lane / C, G = 32 / C;
  const int oy = a.Kx + 1 + a.Ky, oz = a.Kx + 2 * a.Ky + 2 + a.Kz;
  for (int t = threadIdx.x; t < nz * C; t += K64_THREADS) {
    const int z = t / C, j = jb + t % C;
    const double2 v = j < a.nq ? tab[(long)j * a.row + oz + z] : make_double2(0, 0);
    Zs[t] = v;
    Zk[t] = make_double2(z * v.x, z * v.y);
  }
  __syncthreads();
  const double2* __restrict__ R = tab + (long)min(jb + c, a.nq - 1) * a.row;
  const double4* __restrict__ pm = k.pm;
  const double4* __restrict__ pt = k.pt;
  double F[NV];
#pragma unroll
  for (int v = 0; v < NV; v++) F[v] = 0;
  for (int r0 = warp * G; r0 < k.nrow; r0 += K64_WARPS * G) {
    const int zmax = k.rows[r0].ext;   // sorted: the longest of the G
    const KRow64 row = k.rows[min(r0 + h, k.nrow - 1)];
    const int ext = r0 + h < k.nrow ? row.ext : -1;
    double hx = 0, hy = 0, gx = 0, gy = 0, vx = 0, vy = 0;
#pragma unroll 4
    for (int z = 0; z <= zmax; z++) {
      const double4 w = z <= ext ? pm[row.item0 + z] : make_double4(0, 0, 0, 0);
      const double2 e = Zs[z * C + c], f = Zk[z * C + c];
      hx = fma(w.x, e.x, hx);
      hx = fma(-w.w, e.y, hx);
      hy = fma(w.z, e.y, hy);
      hy = fma(w.y, e.x, hy);
      gx = fma(w.z, f.x, gx);
      gx = fma(-w.y, f.y, gx);
      gy = fma(w.x, f.y, gy);
      gy = fma(w.w, f.x, gy);
      if (ADJ && pt) {
        const double4 t = z <= ext ? pt[row.item0 + z] : make_double4(0, 0, 0, 0);
        vx = fma(t.x, e.x, vx);
        vx = fma(-t.w, e.y, vx);
        vy = fma(t.z, e.y, vy);
        vy = fma(t.y, e.x, vy);
      }
    }
    const double2 A = k64_mul(R[row.ikx], R[oy + row.iky]);
    const double im = A.x * hy + A.y * hx;
    F[0] += row.kx * im;
    F[1] += row.ky * im;
    F[2] += A.x * gy + A.y * gx;
    if constexpr (ADJ) {
      F[3] += A.x * hx - A.y * hy;
      F[4] -= A.x * vy + A.y * vx;
    }
  }
#pragma unroll
  for (int v = 0; v < NV; v++) red[(warp * NV + v) * 32 + lane] = F[v];
  __syncthreads();
  const int j = jb + threadIdx.x;
  if (threadIdx.x >= C || j >= a.nq) return;
  double s[NV];
#pragma unroll
  for (int v = 0; v < NV; v++) {
    s[v] = 0;
    for (int w = 0; w < K64_WARPS; w++)
      for (int q = 0; q < G; q++) s[v] += red[(w * NV + v) * 32 + q * C + threadIdx.x];
  }
  const int site = a.qsite[j];
  if constexpr (ADJ) {
    const double q = a.qval[j], iq = 1.0 / q;
    dEq[site] += s[3] * iq / (2 * 3.14159265358979323846) - 2 * a.alpha / 1.772453850905516 * q;
    if (g)
      dLq[site] += (g[3 * site] * s[0] / a.Lx + g[3 * site + 1] * s[1] / a.Ly +
                    g[3 * site + 2] * s[2] / a.Lz + s[4]) * iq;
  } else {
    double* f = a.f + 3 * (long)site + (a.qdrude && a.qdrude[j] ? 3 * (long)a.ns : 0);
    f[0] += s[0] / a.Lx;
    f[1] += s[1] / a.Ly;
    f[2] += s[2] / a.Lz;
  }
}

// charge chunks of pass 1: as many as keep the CTAs in one wave (two fit on an
// SM, one with the adjoint's sums), at least a charge per warp.  (12544
// charges, 12 x 26 CTAs in two waves 398 us, 12 x 25 in one 286; the adjoint's
// sums 820 us in 26 chunks, 615 in 12.)
int k64_chunks(int ntask, int nq, bool adj) {
  const int nblk = (ntask + 31) / 32;
  return std::max(1, std::min({(adj ? 1 : 2) * PARTITION_SMS / nblk, nq / K64_WARPS, 64}));
}
int k64_red_blocks(int nitem) { return (nitem + K64_RED - 1) / K64_RED; }

cudaError_t k_sk64(const Launch& L, const KArgs& a, const K64& k, const double2* tab, bool measure) {
  const int nch = k64_chunks(k.ntask, a.nq, false);
  sk64_kernel<false><<<dim3((k.ntask + 31) / 32, nch), K64_THREADS, 0, L.s>>>(a, k, tab, nullptr, nch);
  sk64_reduce_kernel<<<k64_red_blocks(k.nitem), 32 * K64_RW, 0, L.s>>>(
      a, k, nch, measure, 9.869604401089358 / (a.alpha * a.alpha));
  *L.counter += 2;
  return cudaGetLastError();
}

template <bool ADJ>
static cudaError_t launch_kf64(const Launch& L, const KArgs& a, const K64& k, const double2* tab,
                               const double* g, double* dEq, double* dLq) {
  // charges per CTA: 32 while that leaves two CTAs per SM, down to 8; fewer
  // where their Z rows would not fit
  int C = 32;
  while (C > 8 && a.nq < 2 * PARTITION_SMS * C) C /= 2;
  auto smem = [&](int c) {
    return 2 * (size_t)(a.Kz + 1) * c * sizeof(double2) +
           sizeof(double) * K64_WARPS * 32 * (ADJ ? 5 : 3);
  };
  while (C > 1 && smem(C) > 200 * 1024) C /= 2;
  if (smem(C) > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(kf64_kernel<ADJ>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)smem(C));
    if (e != cudaSuccess) return e;
  }
  kf64_kernel<ADJ><<<(a.nq + C - 1) / C, K64_THREADS, smem(C), L.s>>>(a, k, tab, C, g, dEq, dLq);
  ++*L.counter;
  return cudaGetLastError();
}

cudaError_t k_kf64(const Launch& L, const KArgs& a, const K64& k, const double2* tab) {
  return launch_kf64<false>(L, a, k, tab, nullptr, nullptr, nullptr);
}

cudaError_t k_adjoint64(const Launch& L, const KArgs& a, K64 k, const double2* tab, const double* g,
                        double* dEq, double* dLq) {
  if (g) {
    const int nch = k64_chunks(k.ntask, a.nq, true);
    sk64_kernel<true><<<dim3((k.ntask + 31) / 32, nch), K64_THREADS, 0, L.s>>>(a, k, tab, g, nch);
    tk64_reduce_kernel<<<k64_red_blocks(k.nitem), 32 * K64_RW, 0, L.s>>>(a, k, nch);
    *L.counter += 2;
  } else {
    k.pt = nullptr;
  }
  return launch_kf64<true>(L, a, k, tab, g, dEq, dLq);
}

}  // namespace mg
