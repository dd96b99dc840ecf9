// Adjoint of the force path (FP64): gradients of the energy E, the scalar
// virial W = sum r.f (LJ) + E_el and of a loss of the forces (through its
// weights g_i = dLoss/dF_i) with respect to the LJ (epsilon, sigma) of every
// pair of site kinds and to every site charge.  Pair terms are recomputed,
// nothing of the forward pass is stored but S(k) and the cell list.
//
//   LJ, below C1:  u = E4 (y^2 - y), y = (sigma/r)^6, f = 6 E4 (2y^2 - y)/r^2
//                  du/dsigma = E4 (12 y^2 - 6 y)/sigma,
//                  df/dsigma = 36 E4 y (4y - 1)/(sigma r^2)
//   smooth part:   u = A (r^2 - C2^2)^2, f = A4 (r^2 - C2^2), with
//                  dA/dsigma, dA4/dsigma from the host
//   both:          du/deps = u/eps, df/deps = f/eps  (u is linear in eps)
//   charges:       dE/dq_i = psi_i (r-space + k-space + self),
//                  dLoss/dq_i = sum_j (g_i - g_j).r_ij e_ij q_j + g_i.F^k_i/q_i
//                               + sum_k ekk Im(conj(Phi_i(k)) T(k)),
//                  T(k) = sum_j q_j (g_j.k/L) Phi_j(k)
// (the k-space parts: mg_kspace64.cu)
#include "mg_internal.h"
#include "mg_device.cuh"
#include "mg_pair64.cuh"

namespace mg {

// gradient weights in cell order: (g_x, g_y, g_z, q) of every sorted site
__global__ void adj_gather_kernel(int ns, const int* __restrict__ order,
                                  const double* __restrict__ g, const double* __restrict__ q,
                                  double4* __restrict__ gs) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= ns) return;
  const int i = order[t];
  gs[t] = g ? make_double4(g[3 * i], g[3 * i + 1], g[3 * i + 2], q[i])
            : make_double4(0, 0, 0, q[i]);
}

// The walk of the FP64 force kernel (mg_pair64.cuh): a warp per home site, its
// neighbours in full warps.  The kind of the home site is the warp's, a
// neighbour's kind the lane's: 6 sums per neighbour kind and lane stay in
// shared memory (u, du/dsigma, r^2 f, r^2 df/dsigma, g.r f, g.r df/dsigma) and
// are added over the lanes at the end.  row [site][6 nkind + 1]: these sums,
// and q_i times the r-space potential; per site: dE/dq and dL/dq of the
// r-space sum.  The energies come out of the same sums, so no force kernel
// runs for them.  (A lane per home site of a cell, shared-memory atomics per
// pair and seven divisions: 4.7 ms on 12544 sites, and 0.7 ms for the energies;
// this 0.64 ms.)
__global__ void __launch_bounds__(P64_THREADS)
    adj_pair_kernel(const __grid_constant__ PairArgs a, const double4* __restrict__ pd,
                    const float4* __restrict__ pf, const double4* __restrict__ gs,
                    const AdjPair* __restrict__ tab_g, const double* __restrict__ ert,
                    double* __restrict__ row, double* __restrict__ dEq, double* __restrict__ dLq,
                    float cqf) {
  extern __shared__ __align__(16) unsigned char adj_smem[];
  __shared__ P64Queue queue[P64_WARPS];
  const int nk = a.nkind, nk2 = nk * nk, nc = 6 * nk;
  double* accs = reinterpret_cast<double*>(adj_smem);                  // [warps][6 nk][32]
  AdjPair* tab = reinterpret_cast<AdjPair*>(accs + (size_t)P64_WARPS * nc * 32);
  unsigned char* flag = reinterpret_cast<unsigned char*>(tab + nk2);
  for (int t = threadIdx.x; t < nk2; t += P64_THREADS) {
    const AdjPair P = tab_g[t];
    tab[t] = P;
    flag[t] = (unsigned char)(2 | (P.E4 != 0 ? 1 : 0));
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ti = blockIdx.x * P64_WARPS + warp;
  if (ti >= a.ns) return;
  double* acc = accs + (size_t)warp * nc * 32;
  for (int t = lane; t < nc * 32; t += 32) acc[t] = 0;
  const double4 me = pd[ti], gi = gs[ti];
  const int kind_i = (int)(__double_as_longlong(me.w) & 255);
  const AdjPair* prow = tab + kind_i * nk;
  const bool tight = p64_tight(a);
  double eq = 0, lq = 0;
  auto work = [&](auto cls, const int2 e, bool on) {
    constexpr int CLS = decltype(cls)::value;
    if (!on) return;
    const double4 q = pd[e.x];
    const double dx = p64_image(me.x - q.x, e.y, a.Lx, tight),
                 dy = p64_image(me.y - q.y, e.y >> 2, a.Ly, tight),
                 dz = p64_image(me.z - q.z, e.y >> 4, a.Lz, tight);
    const double rr = dx * dx + dy * dy + dz * dz;
    if (!(rr < a.cutoff_sq)) return;
    const double4 gj = gs[e.x];
    const double gd = (gi.x - gj.x) * dx + (gi.y - gj.y) * dy + (gi.z - gj.z) * dz;
    const int kj = e.y >> 8;
    if (CLS == P64_LJ) {
      const AdjPair& P = prow[kj];
      if (rr < P.C2q) {
        double u, f, du, df;
        if (rr < P.C1q) {
          const double ir = 1 / rr, x = P.Sq * ir, y = x * x * x;
          const double b = P.E4 * y * P.isig;
          u = P.E4 * y * (y - 1);
          f = 6 * P.E4 * y * (2 * y - 1) * ir;
          du = 6 * b * (2 * y - 1);
          df = 36 * b * (4 * y - 1) * ir;
        } else {
          const double x = rr - P.C2q;
          u = P.A * x * x;
          f = P.A4 * x;
          du = P.dA * x * x;
          df = P.dA4 * x;
        }
        double* A = acc + (size_t)(6 * kj) * 32 + lane;
        A[0] += u;
        A[32] += du;
        A[64] += rr * f;
        A[96] += rr * df;
        A[128] += gd * f;
        A[160] += gd * df;
      }
    }
    double phi = 0, er = 0;
    if (CLS == P64_EXCL) {
      phi = excl_term<double>(rr, a.alpha, &er);
    } else if (gj.w != 0) {
      const double* p = ert + 6 * min((int)(rr * a.sgrid), a.ntab - 1);
      phi = p[1] / (p[2] + rr) + p[0];
      er = p[4] / (p[5] + rr) + p[3];
    }
    eq += gj.w * phi;
    lq += gd * er * gj.w;
  };
  p64_walk(a, pf, ti, flag + kind_i * nk, queue[warp], cqf, work);
  eq = p64_sum(eq);
  lq = p64_sum(lq);
  __syncwarp();
  const int site = a.order[ti];
  double* out = row + (size_t)ti * (nc + 1);
  // a lane adds one column, starting at its own so that the lanes meet
  // different banks
  for (int c = lane; c < nc; c += 32) {
    double s = 0;
    for (int l = 0; l < 32; l++) s += acc[(size_t)c * 32 + ((l + lane) & 31)];
    out[c] = s;
  }
  if (lane == 0) {
    out[nc] = gi.w * eq;
    dEq[site] = eq;
    dLq[site] = lq;
  }
}

// part [CTA][6 nkind^2 + 1]: the rows of the CTA's share of the sites, by the
// kind of the site; a thread owns one column of a row
__global__ void __launch_bounds__(128)
    adj_rows_kernel(int ns, int nk, const double4* __restrict__ pd, const double* __restrict__ row,
                    double* __restrict__ part) {
  extern __shared__ __align__(16) unsigned char adj_smem[];
  double* acc = reinterpret_cast<double*>(adj_smem);   // [nk][6 nk + 1]
  const int nc = 6 * nk + 1;
  for (int t = threadIdx.x; t < nk * nc; t += 128) acc[t] = 0;
  __syncthreads();
  const int t0 = (int)((long)ns * blockIdx.x / gridDim.x),
            t1 = (int)((long)ns * (blockIdx.x + 1) / gridDim.x);
  if ((int)threadIdx.x < nc)
#pragma unroll 4
    for (int t = t0; t < t1; t++)
      acc[(int)(__double_as_longlong(pd[t].w) & 255) * nc + threadIdx.x] +=
          row[(size_t)t * nc + threadIdx.x];
  __syncthreads();
  double* out = part + (size_t)blockIdx.x * (6 * nk * nk + 1);
  for (int t = threadIdx.x; t < 6 * nk * nk; t += 128) out[t] = acc[t / (6 * nk) * nc + t % (6 * nk)];
  if (threadIdx.x == 0) {
    double e = 0;
    for (int k = 0; k < nk; k++) e += acc[k * nc + 6 * nk];
    out[6 * nk * nk] = e;
  }
}

static inline int cdiv_a(long a, long b) { return (int)((a + b - 1) / b); }

int adj_parts(int ns) { return std::min(2 * PARTITION_SMS, std::max(1, ns / 8)); }

cudaError_t k_adjoint(const Launch& L, const PairArgs& pa, const double4* pd, const float4* pf,
                      const AdjPair* tab, const double* ert, const double* g, const double* q,
                      double4* gs, double* row, double* part, double* sums, double* dEq,
                      double* dLq) {
  const int nk = pa.nkind, np = adj_parts(pa.ns);
  static_assert(6 * MAX_KINDS + 1 <= 128, "adj_rows_kernel: a thread per column");
  adj_gather_kernel<<<cdiv_a(pa.ns, 256), 256, 0, L.s>>>(pa.ns, pa.order, g, q, gs);
  const size_t sm = sizeof(double) * P64_WARPS * 6 * nk * 32 + (sizeof(AdjPair) + 1) * (size_t)nk * nk;
  if (sm > 32 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(adj_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)sm);
    if (e != cudaSuccess) return e;
  }
  adj_pair_kernel<<<cdiv_a(pa.ns, P64_WARPS), P64_THREADS, sm, L.s>>>(pa, pd, pf, gs, tab, ert, row,
                                                                     dEq, dLq, p64_cutoff(pa));
  adj_rows_kernel<<<np, 128, sizeof(double) * nk * (6 * nk + 1), L.s>>>(pa.ns, nk, pd, row, part);
  *L.counter += 3;
  return k_reduce_sum(L, part, np, 6 * nk * nk + 1, sums);
}

}  // namespace mg
