// Ewald k-space sums as non-uniform transforms (mg_nufft.cu): the arguments
// of one box and the launches of a list of boxes.
#pragma once

#include <vector>

#include "mg_internal.h"

namespace mg {

constexpr int NF_W = 8;       // window width, grid steps
constexpr int NF_TILE = 8;    // edge of a tile of grid points
constexpr int NF_CS = 4;      // CTAs of a plane (M is a multiple of it)
constexpr int NF_KC = 4;      // outputs per thread of the transforms over x and y
constexpr float NF_MARGIN = 0.5f;  // A: Drude displacement covered by the cell lookup

struct NfBox {
  int ns, nsub;            // sites; charges per site (2 with Drude shells)
  int dense;               // nf_dense
  int M[3], K[3];          // grid points and largest modes
  int nc[3];               // cells of the cell list
  int marg[3];             // extra grid steps of the cell lookup (Drude shells)
  const int4* pj;          // sorted fixed-point sites
  const float4* pdj;       // sorted Drude displacements
  const int* order;
  const int* cell_start;
  const int* far;          // set when a displacement exceeds NF_MARGIN
  float q[MAX_KINDS], qp[MAX_KINDS];   // charge and Drude charge of every kind
  float nb[3], db[3];      // -beta log2(e); -beta (2/w)^2
  float fac[3], fix[3];    // grid steps per A; fixed-point units per A
  float cpg[3];            // cells per grid step
  unsigned long long step[3];  // 2^64 / M: a grid step in fixed point, 32 more bits
  unsigned ext[3];         // a tile's window box (TILE + w - 1 steps) in fixed point
  double iL[3], pi2_over_a2;
  float* G;                // [Mx][My][Mz] charge grid, then potential grid
  float2* A;               // [Kx+1][My][Mz]
  const float2* fwd[3];
  const float2* inv[3];
  const float* wk;         // [2Kz+1][Kx+1][2Ky+1] ekk / (2 pi window^2), zero off the k set
  double* ek_part;         // [(Kx+1) * NF_CS * 7] energy and virial sums
  double* f;               // forces the batched launch adds to
};

// the largest grids and shared memory over the boxes of a launch
struct NfGrid {
  int spread, x, plane, interp, interp_tile;
  int sx, six, splane, splane_few;
};

bool nf_grids(const int K[3], int M[3]);
double nf_beta(int M, int K);
int nf_dense(int nq, const int M[3]);
void nf_tables(const int K[3], const int M[3], const std::vector<int4>& kvec,
               const std::vector<double>& ekk, std::vector<float2> fwd[3],
               std::vector<float2> inv[3], std::vector<float>* wk);
// raises the grids of g to those box b needs
void nf_launch(const NfBox& b, NfGrid* g);

cudaError_t k_nf_far(const Launch& L, int ns, const float4* pdj, float lim, int* far);
// charges -> grid -> modes over x; the planes (S(k), energies); back to the
// potential grid; forces added to f (or each box's own)
cudaError_t k_nf_forward(const Launch& L, const NfBox* d, int nbox, const NfGrid& g);
cudaError_t k_nf_modes(const Launch& L, const NfBox* d, int nbox, const NfGrid& g, bool measure);
cudaError_t k_nf_back(const Launch& L, const NfBox* d, int nbox, const NfGrid& g);
cudaError_t k_nf_interp(const Launch& L, const NfBox* d, int nbox, const NfGrid& g, double* f);

}  // namespace mg
