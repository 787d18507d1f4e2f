// kernels_split.cuh - one-thread-per-cell H and E passes for any grid shape.
//
// These passes cover every case the reference covers (1D, 2D in any plane,
// 3D; collapsed axes drop their curl terms); 3D grids normally take the
// vector passes of kernels_vec3d.cuh. The per-component arithmetic lives in
// cell_update.cuh. Update order per component
// (src/photonfdtd/simulation.py:1252-1309):
//   curl = dA - dB (or dA, or -dB when one axis is collapsed)
//   F   += K * curl                          (bulk)
//   psiA = bA*psiA + cA*dA ; F += (+K)*psiA   (only where cA != 0)
//   psiB = bB*psiB + cB*dB ; F += (-K)*psiB   (only where cB != 0)
// with d = (a_hi - a_lo) / dl and K = ce (E) or -ch (H).
#pragma once

#include "cell3d.cuh"
#include "kernels_vec3d.cuh"

namespace pfb {

// Load f[id + off] only when the neighbour exists (cond), else 0.
template <typename T>
__device__ __forceinline__ T ld_if(const T* f, long long id, long long off, bool cond) {
  return cond ? f[id + off] : T(0);
}

// H pass: H^{n+1/2} = H^{n-1/2} - ch (curl E^n + psi).
template <typename T>
__global__ void __launch_bounds__(256) k_h_split(const __grid_constant__ StepArgs<T> a) {
  pdl_enter();
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  const int i = blockIdx.z;
  if (k >= a.nz || j >= a.ny) return;
  const long long sy = a.pz, sx = (long long)a.ny * a.pz;
  const long long id = i * sx + j * sy + k;
  const T ex = a.Ein[0][id], ey = a.Ein[1][id], ez = a.Ein[2][id];
  const bool hx = i + 1 < a.nx, hy = j + 1 < a.ny, hz = k + 1 < a.nz;
  a.Hout[0][id] = upd_hx<T>(a, i, j, k, a.Hin[0][id], ld_if(a.Ein[2], id, sy, hy), ez,
                            ld_if(a.Ein[1], id, 1, hz), ey, true);
  a.Hout[1][id] = upd_hy<T>(a, i, j, k, a.Hin[1][id], ld_if(a.Ein[0], id, 1, hz), ex,
                            ld_if(a.Ein[2], id, sx, hx), ez, true);
  a.Hout[2][id] = upd_hz<T>(a, i, j, k, a.Hin[2][id], ld_if(a.Ein[1], id, sx, hx), ey,
                            ld_if(a.Ein[0], id, sy, hy), ex, true);
}

// E pass: E^{n+1} = E^n + ce (curl H^{n+1/2} + psi), then ADE.
template <typename T, int CE, bool ADE>
__global__ void __launch_bounds__(256) k_e_split(const __grid_constant__ StepArgs<T> a) {
  pdl_enter();
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  const int i = blockIdx.z;
  if (k >= a.nz || j >= a.ny) return;
  const MediumT<T>* media = a.media;
  const long long sy = a.pz, sx = (long long)a.ny * a.pz;
  const long long id = i * sx + j * sy + k;
  // Loads are issued in dependency order: the per-cell word and the cell's
  // fields first, then what the word selects (coefficient, ADE record).
  T K[3];
  uint32_t t, w;
  cell_word<T, CE, ADE>(a, id, K, t);
  const T hx = a.Hin[0][id], hy = a.Hin[1][id], hz = a.Hin[2][id];
  const T en[3] = {a.Ein[0][id], a.Ein[1][id], a.Ein[2][id]};
  cell_decode<T, CE, ADE>(a, media, t, K, w);
  AdeRec<T> rec;
  if (ADE && w) ade_load<T>(a, media, w, rec);
  const bool lx = i > 0, ly = j > 0, lz = k > 0;
  T e[3];
  e[0] = upd_ex<T>(a, i, j, k, en[0], K[0], hz, ld_if(a.Hin[2], id, -sy, ly), hy,
                   ld_if(a.Hin[1], id, -1, lz));
  e[1] = upd_ey<T>(a, i, j, k, en[1], K[1], hx, ld_if(a.Hin[0], id, -1, lz), hz,
                   ld_if(a.Hin[2], id, -sx, lx));
  e[2] = upd_ez<T>(a, i, j, k, en[2], K[2], hy, ld_if(a.Hin[1], id, -sx, lx), hx,
                   ld_if(a.Hin[0], id, -sy, ly));
  if (ADE && w) ade_update<T>(a, media, rec, a.lvl, en, e);
  a.Eout[0][id] = e[0];
  a.Eout[1][id] = e[1];
  a.Eout[2][id] = e[2];
}

// The E pass of a 3D grid with dispersive cells, one cell per thread, on the
// layout of the vector passes (which run the H half). For scenes whose
// polarisation records seldom form aligned runs (see ade_by_cell in engine.cu):
// here every record is loaded ahead of the curl whatever lies beside it.
template <typename T, int CE>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 5 : 4)
    k_e_cell(const __grid_constant__ StepArgs<T> a) {
  pdl_enter();
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  const int i = blockIdx.z;
  const bool live = k < a.nz && j < a.ny;
  const bool box = warp_bulk<1>(live, i, j, k, a.eb0, a.eb1);
  if (!live) return;
  const long long sy = a.pz, sx = (long long)a.ny * a.pz;
  const long long id = i * sx + j * sy + k;
  T K[3];
  uint32_t t, w;
  cell_word<T, CE, true>(a, id, K, t);
  const T hx = a.Hin[0][id], hy = a.Hin[1][id], hz = a.Hin[2][id];
  const T en[3] = {a.Ein[0][id], a.Ein[1][id], a.Ein[2][id]};
  const bool lx = i > 0, ly = j > 0, lz = k > 0;
  // Ex: +dHz/dy - dHy/dz; Ey: +dHx/dz - dHz/dx; Ez: +dHy/dx - dHx/dy
  const T h[6] = {ld_if(a.Hin[2], id, -sy, ly), ld_if(a.Hin[1], id, -1, lz),
                  ld_if(a.Hin[0], id, -1, lz),  ld_if(a.Hin[2], id, -sx, lx),
                  ld_if(a.Hin[1], id, -sx, lx), ld_if(a.Hin[0], id, -sy, ly)};
  cell_decode<T, CE, true>(a, a.media, t, K, w);
  AdeRec<T> rec;
  if (w) ade_load<T>(a, a.media, w, rec);
  const T n[6] = {sub_rn(hz, h[0]), sub_rn(hy, h[1]), sub_rn(hx, h[2]),
                  sub_rn(hz, h[3]), sub_rn(hy, h[4]), sub_rn(hx, h[5])};
  T e[3];
  if (box) {
    const int ax[6] = {1, 2, 2, 0, 0, 1};
    T d[6];
    divide6<T>(a, n, ax, d);
#pragma unroll
    for (int c = 0; c < 3; ++c) e[c] = bulk(en[c], K[c], d[2 * c], d[2 * c + 1]);
  } else {
    e3<T>(a, i, j, k, en, K, n, e);
  }
  if (w) ade_update<T>(a, a.media, rec, a.lvl, en, e);
#pragma unroll
  for (int c = 0; c < 3; ++c) a.Eout[c][id] = e[c];
}

}  // namespace pfb
