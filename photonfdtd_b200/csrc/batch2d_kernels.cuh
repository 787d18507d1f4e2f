// batch2d_kernels.cuh - kernels of the batched 2D TE engine (batch2d.cu).
//
// Layout: each instance's rows are padded to a pitch of a multiple of 32
// cells and start 32-aligned, so a warp's row access is one aligned line.
// Work list: tiles of 32 columns (y) x 8R rows (x) drawn from every
// instance; a block of 32 x 8 threads takes one tile, each thread R
// consecutive rows of one column. Every thread issues all its loads before
// its first store (the row it shares with the next row is loaded once), so a
// block keeps 8R cells per column in flight. A tile record carries everything
// needed to address its cells; the instance record is read only for CPML
// psi, design-window and output-line cells.
//
// The step index n of a kernel is *base + t: base is set once per chunk of
// steps, t is baked into the launch, so a captured chunk replays for any
// segment without per-step counter kernels.
#pragma once

#include "common.cuh"

namespace pfb {
namespace b2d {

constexpr int kWarps = 8;     // warps per block
// Minimum resident blocks per SM the fused forward and reverse steps are
// compiled for.
#ifndef PFB_MINB_STEP
#define PFB_MINB_STEP 4
#endif
#ifndef PFB_MINB_ASTEP
#define PFB_MINB_ASTEP 4
#endif
// Minimum resident 256-thread blocks per SM of the vector steps (float).
#ifndef PFB_MINB_TILE
#define PFB_MINB_TILE 4
#endif
#ifndef PFB_MINB_ATILE
#define PFB_MINB_ATILE 4
#endif
#ifndef PFB_MINB_EDGE
#define PFB_MINB_EDGE 2
#endif
#ifndef PFB_MINB_AEDGE
#define PFB_MINB_AEDGE 3
#endif
constexpr int kDftRing = 32;  // line samples kept before a DFT flush

struct Inst {
  int nx, ny;
  int pitch;                             // row stride: ny rounded up to 32
  long long off;                         // first cell in the pooled field arrays (32-aligned)
  int ox, oy;                            // first entry in the pooled x / y coefficients
  long long p_hzx, p_hzy, p_exy, p_eyx;  // first element of each psi array
  int nphx, nphy, npex, npey;            // psi extents along their axes (y: whole groups of 4)
  int di0, dj0, dn;                      // design window
  long long goff;                        // first design cell (dn * dn per instance)
  int line_i;                            // x index of the output line
  long long loff;                        // first line cell (ny per instance)
};

struct __align__(16) TileRec {
  long long base;      // pooled index of the tile origin (i0, j0)
  int nx, ny, pitch;   // instance extents, row stride
  int i0, j0;          // tile origin in the instance
  int ox, oy;          // pooled coefficient index of row i0 / column j0
  int k;               // instance
  int wdi, wdj, wdn;   // design window relative to the tile origin, its size
  int flags;           // kTile* below
  long long p_hzx, p_hzy, p_exy, p_eyx;  // the instance's psi arrays
  int nphy, npey;
  int nx_end;          // edge tiles: rows from here on belong to another tile
  int pad;
};
// A tile of the vector steps whose cells and the row above and column left of
// them lie in the interior (every difference exists) and hold no CPML state.
constexpr int kTileBulk = 1;
constexpr int kTileWindow = 2;  // some cells of the design window
constexpr int kTilePost = 4;    // the output line or a row with sources

// Columns per thread of the vector steps (16 bytes), and threads per tile row:
// bulk tiles are 32 columns wide, edge tiles 16 (the CPML layers at the ends
// of a row are about that wide) and twice as high.
template <typename T>
constexpr int kTileV = 16 / (int)sizeof(T);
template <typename T>
__host__ __device__ constexpr int tile_x(bool edge) {
  return (edge ? 16 : 32) / kTileV<T>;
}

template <typename T>
struct BArgs {
  const Inst* inst;
  const TileRec* tiles;
  int ntiles;
  int nedge;  // the first nedge tiles are not kTileBulk
  T *Ex, *Ey, *Hz;
  const T* ce;
  const T *bex, *cex, *bhx, *chx, *bey, *cey, *bhy, *chy;
  const int *mex, *mhx, *mey, *mhy;
  const int *gey, *ghy;  // per 4 pooled columns: psi group (4 entries), or -1
  T *pHzx, *pHzy, *pExy, *pEyx;
  T dx, dy, rdx, rdy, ch;
  T idx, idy;  // 1/dx, 1/dy rounded once (adjoint kernels only)
  bool fdx, fdy;
  bool fast;   // fdx, fdy, and ch scaled down by QScale is exact
  const long long* base;  // first step of the running chunk
  T* ring;                // design-window curls, slot = n mod ring_len
  long long n_design;
  int ring_len;
  // The fused step's double-buffered state: step n reads level n & 1 and
  // writes level (n & 1) ^ 1 (level 0 is Ex / Ey / Hz / pHzx / pHzy above).
  T *Ex2[2], *Ey2[2], *Hz2[2], *pHzx2[2], *pHzy2[2];
};

// ---- forward ---------------------------------------------------------------
// Hz^{n+1/2} = Hz - ch (dEy/dx - dEx/dy) - ch psi_x + ch psi_y where both
// forward differences exist (i < nx-1, j < ny-1); the reference's operation
// order (simulation.py:1284-1309).
template <typename T, int R>
__global__ void __launch_bounds__(32 * kWarps) kb_h(const __grid_constant__ BArgs<T> a) {
  for (int t = blockIdx.x; t < a.ntiles; t += gridDim.x) {
    const TileRec tr = a.tiles[t];
    const int r0 = threadIdx.y * R;
    const int i = tr.i0 + r0, j = tr.j0 + threadIdx.x;
    if (j >= tr.ny - 1 || i >= tr.nx - 1) continue;
    const long long id0 = tr.base + (long long)r0 * tr.pitch + threadIdx.x;
    T ey[R + 1], ex0[R], ex1[R], hz[R];
    int mx[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const bool ok = i + r < tr.nx - 1;  // an H row
      const long long id = id0 + (long long)r * tr.pitch;
      ey[r] = i + r < tr.nx ? a.Ey[id] : T(0);  // also the row after the last H row
      ex0[r] = ok ? a.Ex[id] : T(0);
      ex1[r] = ok ? a.Ex[id + 1] : T(0);
      hz[r] = ok ? a.Hz[id] : T(0);
      mx[r] = ok ? a.mhx[tr.ox + r0 + r] : -1;
    }
    ey[R] = (i + R < tr.nx) ? a.Ey[id0 + (long long)R * tr.pitch] : T(0);
    const int my = a.mhy[tr.oy + threadIdx.x];
    const T mch = -a.ch;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if (i + r >= tr.nx - 1) break;
      const T dA = qdiv(sub_rn(ey[r + 1], ey[r]), a.dx, a.rdx, a.fdx);
      const T dB = qdiv(sub_rn(ex1[r], ex0[r]), a.dy, a.rdy, a.fdy);
      T h = add_rn(hz[r], mul_rn(sub_rn(dA, dB), mch));
      if (mx[r] >= 0 || my >= 0) {
        const Inst& I = a.inst[tr.k];
        if (mx[r] >= 0) {
          const long long q = I.p_hzx + (long long)mx[r] * tr.pitch + j;
          const int c = tr.ox + r0 + r;
          const T psi = add_rn(mul_rn(a.bhx[c], a.pHzx[q]), mul_rn(a.chx[c], dA));
          a.pHzx[q] = psi;
          h = add_rn(h, mul_rn(mch, psi));
        }
        if (my >= 0) {
          const long long q = I.p_hzy + (long long)(i + r) * I.nphy + my;
          const int c = tr.oy + threadIdx.x;
          const T psi = add_rn(mul_rn(a.bhy[c], a.pHzy[q]), mul_rn(a.chy[c], dB));
          a.pHzy[q] = psi;
          h = add_rn(h, mul_rn(a.ch, psi));
        }
      }
      a.Hz[id0 + (long long)r * tr.pitch] = h;
    }
  }
}

// Ex^{n+1} = Ex + K dHz/dy + K psi_y (j >= 1); Ey^{n+1} = Ey - K dHz/dx -
// K psi_x (i >= 1). Design cells also store the curls that multiplied K:
// ring[n mod ring_len][cell] = (cEx, cEy), n = *base + step_t.
template <typename T, int R>
__global__ void __launch_bounds__(32 * kWarps) kb_e(const __grid_constant__ BArgs<T> a,
                                                   int step_t) {
  for (int t = blockIdx.x; t < a.ntiles; t += gridDim.x) {
    const TileRec tr = a.tiles[t];
    const int r0 = threadIdx.y * R;
    const int i = tr.i0 + r0, j = tr.j0 + threadIdx.x;
    if (j >= tr.ny || i >= tr.nx) continue;
    const long long id0 = tr.base + (long long)r0 * tr.pitch + threadIdx.x;
    T hz[R + 1], hzl[R], ex[R], ey[R], K[R];
    int mx[R];
    hz[0] = i >= 1 ? a.Hz[id0 - tr.pitch] : T(0);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const bool ok = i + r < tr.nx;
      const long long id = id0 + (long long)r * tr.pitch;
      hz[r + 1] = ok ? a.Hz[id] : T(0);
      hzl[r] = (ok && j >= 1) ? a.Hz[id - 1] : T(0);
      ex[r] = ok ? a.Ex[id] : T(0);
      ey[r] = ok ? a.Ey[id] : T(0);
      K[r] = ok ? a.ce[id] : T(0);
      mx[r] = ok ? a.mex[tr.ox + r0 + r] : -1;
    }
    const int my = a.mey[tr.oy + threadIdx.x];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if (i + r >= tr.nx) break;
      const long long id = id0 + (long long)r * tr.pitch;
      T cx = T(0), cy = T(0);
      if (j >= 1) {
        const T dA = qdiv(sub_rn(hz[r + 1], hzl[r]), a.dy, a.rdy, a.fdy);
        T e = add_rn(ex[r], mul_rn(dA, K[r]));
        cx = dA;
        if (my >= 0) {
          const Inst& I = a.inst[tr.k];
          const long long q = I.p_exy + (long long)(i + r) * I.npey + my;
          const int c = tr.oy + threadIdx.x;
          const T psi = add_rn(mul_rn(a.bey[c], a.pExy[q]), mul_rn(a.cey[c], dA));
          a.pExy[q] = psi;
          e = add_rn(e, mul_rn(K[r], psi));
          cx = add_rn(dA, psi);
        }
        a.Ex[id] = e;
      }
      if (i + r >= 1) {
        const T dB = qdiv(sub_rn(hz[r + 1], hz[r]), a.dx, a.rdx, a.fdx);
        T e = add_rn(ey[r], mul_rn(-dB, K[r]));
        cy = -dB;
        if (mx[r] >= 0) {
          const Inst& I = a.inst[tr.k];
          const long long q = I.p_eyx + (long long)mx[r] * tr.pitch + j;
          const int c = tr.ox + r0 + r;
          const T psi = add_rn(mul_rn(a.bex[c], a.pEyx[q]), mul_rn(a.cex[c], dB));
          a.pEyx[q] = psi;
          e = add_rn(e, mul_rn(-K[r], psi));
          cy = sub_rn(cy, psi);
        }
        a.Ey[id] = e;
      }
      const int di = r0 + r - tr.wdi, dj = (int)threadIdx.x - tr.wdj;
      if (di >= 0 && di < tr.wdn && dj >= 0 && dj < tr.wdn) {
        const Inst& I = a.inst[tr.k];
        const long long slot = (*a.base + step_t) % a.ring_len;
        T* rr = a.ring + (slot * a.n_design + I.goff + (long long)di * tr.wdn + dj) * 2;
        rr[0] = cx;
        rr[1] = cy;
      }
    }
  }
}

// ---- fused forward step ------------------------------------------------------
// One launch per step on double-buffered fields: a tile first updates Hz of
// its own cells and, recomputed from the previous level, of the one-cell halo
// its E update needs (the row above, the column to the left), keeping them in
// shared memory; then it updates Ex and Ey of its own cells from there.
// Everything is read from level n & 1 and written to level (n & 1) ^ 1 (the
// E psi, which no other tile reads, in place), so tiles never race and the
// fields cross HBM once per step: Ex, Ey, Hz and ce read, Ex, Ey, Hz written.
// The arithmetic of every cell is kb_h's and kb_e's, operation for operation,
// so the results equal the split passes' bit for bit. Used when no source
// drives Hz (an H source would have to reach the halo recomputation).

// Hz^{n+1/2} of cell (i, j) from its own old value and its E neighbours, as
// kb_h computes it. crow / ccol: pooled x / y coefficient index of the cell;
// psi_out == nullptr recomputes a halo cell without storing its psi.
template <typename T>
__device__ __forceinline__ T hz_value(const BArgs<T>& a, const Inst& I, int i, int j, int ny,
                                      int crow, int ccol, int mx, int my, T hz, T eyp, T ey,
                                      T exp_, T ex, const T* pzx, T* pzxo, const T* pzy,
                                      T* pzyo) {
  const T mch = -a.ch;
  T dA, dB;
  qdiv2(sub_rn(eyp, ey), a.dx, a.rdx, a.fdx, sub_rn(exp_, ex), a.dy, a.rdy, a.fdy, dA, dB);
  T h = add_rn(hz, mul_rn(sub_rn(dA, dB), mch));
  if (mx >= 0) {
    const long long q = I.p_hzx + (long long)mx * I.pitch + j;
    const T psi = add_rn(mul_rn(a.bhx[crow], pzx[q]), mul_rn(a.chx[crow], dA));
    if (pzxo) pzxo[q] = psi;
    h = add_rn(h, mul_rn(mch, psi));
  }
  if (my >= 0) {
    const long long q = I.p_hzy + (long long)i * I.nphy + my;
    const T psi = add_rn(mul_rn(a.bhy[ccol], pzy[q]), mul_rn(a.chy[ccol], dB));
    if (pzyo) pzyo[q] = psi;
    h = add_rn(h, mul_rn(a.ch, psi));
  }
  return h;
}

// Every global load of a tile is issued before its barrier: the own cells'
// E and H values, coefficients and CPML maps (the E update reuses the Ex / Ey
// values the H update loaded), the halo row's inputs (warp 0) and the halo
// column's (warp 1, one row per lane), so a block waits out one memory
// latency per tile.
template <typename T, int R>
__global__ void __launch_bounds__(32 * kWarps, PFB_MINB_STEP) kb_step(
    const __grid_constant__ BArgs<T> a, int step_t) {
  constexpr int TR = kWarps * R;
  static_assert(TR <= 32, "the halo column is one warp's work");
  __shared__ T sH[TR + 1][33];  // [1 + row][1 + column]; row / column 0 = halo
  const long long n = *a.base + step_t;
  const int L = (int)(n & 1);
  const T* Ex = a.Ex2[L];
  const T* Ey = a.Ey2[L];
  const T* Hz = a.Hz2[L];
  T* Exo = a.Ex2[L ^ 1];
  T* Eyo = a.Ey2[L ^ 1];
  T* Hzo = a.Hz2[L ^ 1];
  const T* pzx = a.pHzx2[L];
  const T* pzy = a.pHzy2[L];
  T* pzxo = a.pHzx2[L ^ 1];
  T* pzyo = a.pHzy2[L ^ 1];
  const int lane = threadIdx.x;
  const int r0 = threadIdx.y * R;
  for (int t = blockIdx.x; t < a.ntiles; t += gridDim.x) {
    const TileRec tr = a.tiles[t];
    const Inst& I = a.inst[tr.k];
    const int i = tr.i0 + r0, j = tr.j0 + lane;
    const bool jv = j < tr.ny;
    const long long id0 = tr.base + (long long)r0 * tr.pitch + lane;
    // ---- loads: own cells
    T ey[R + 1], ex0[R], ex1[R], hz[R], K[R];
    int mxh[R], mxe[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const bool ok = jv && i + r < tr.nx;
      const long long id = id0 + (long long)r * tr.pitch;
      ey[r] = ok ? Ey[id] : T(0);
      ex0[r] = ok ? Ex[id] : T(0);
      ex1[r] = (ok && j + 1 < tr.ny) ? Ex[id + 1] : T(0);
      hz[r] = ok ? Hz[id] : T(0);
      K[r] = ok ? a.ce[id] : T(0);
      mxh[r] = ok ? a.mhx[tr.ox + r0 + r] : -1;
      mxe[r] = ok ? a.mex[tr.ox + r0 + r] : -1;
    }
    ey[R] = (jv && i + R < tr.nx) ? Ey[id0 + (long long)R * tr.pitch] : T(0);
    const int myh = jv ? a.mhy[tr.oy + lane] : -1;
    const int mye = jv ? a.mey[tr.oy + lane] : -1;
    // ---- loads: the halo cell this thread recomputes, if any (warp 0: row
    // i0 - 1 at column j; warp 1: column j0 - 1 at tile row `lane`)
    int hrole = 0;  // 1 halo row, 2 halo column
    int hi = 0, hj = 0, hcrow = 0, hccol = 0, hmx = -1, hmy = -1;
    T hz_h = T(0), hey1 = T(0), hey0 = T(0), hex1 = T(0), hex0 = T(0);
    if (threadIdx.y == 0 && tr.i0 >= 1 && jv) {
      hrole = 1;
      hi = tr.i0 - 1;
      hj = j;
      hcrow = tr.ox - 1;
      hccol = tr.oy + lane;
    } else if (threadIdx.y == 1 && lane < TR && tr.j0 >= 1 && tr.i0 + lane < tr.nx) {
      hrole = 2;
      hi = tr.i0 + lane;
      hj = tr.j0 - 1;
      hcrow = tr.ox + lane;
      hccol = tr.oy - 1;
    }
    const bool hupd = hrole && hi < tr.nx - 1 && hj < tr.ny - 1;
    if (hrole) {
      const long long id = tr.base + (long long)(hi - tr.i0) * tr.pitch + (hj - tr.j0);
      hz_h = Hz[id];
      if (hupd) {
        hey1 = Ey[id + tr.pitch];
        hey0 = Ey[id];
        hex1 = Ex[id + 1];
        hex0 = Ex[id];
        hmx = a.mhx[hcrow];
        hmy = a.mhy[hccol];
      }
    }
    // ---- Hz of the tile's own cells
#pragma unroll
    for (int r = 0; r < R; ++r) {
      T h = hz[r];
      if (jv && i + r < tr.nx - 1 && j < tr.ny - 1)
        h = hz_value<T>(a, I, i + r, j, tr.ny, tr.ox + r0 + r, tr.oy + lane, mxh[r], myh, hz[r],
                        ey[r + 1], ey[r], ex1[r], ex0[r], pzx, pzxo, pzy, pzyo);
      if (jv && i + r < tr.nx) Hzo[id0 + (long long)r * tr.pitch] = h;
      sH[r0 + r + 1][lane + 1] = h;
    }
    // ---- the halo cell, recomputed from level L (its psi is not stored)
    {
      T h = hz_h;
      if (hupd)
        h = hz_value<T>(a, I, hi, hj, tr.ny, hcrow, hccol, hmx, hmy, hz_h, hey1, hey0, hex1,
                        hex0, pzx, nullptr, pzy, nullptr);
      if (threadIdx.y == 0) sH[0][lane + 1] = hrole == 1 ? h : T(0);
      if (threadIdx.y == 1 && lane < TR) sH[lane + 1][0] = hrole == 2 ? h : T(0);
    }
    __syncthreads();
    // ---- Ex, Ey of the tile's own cells (kb_e's arithmetic, Hz from shared memory)
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if (!(jv && i + r < tr.nx)) break;
      const long long id = id0 + (long long)r * tr.pitch;
      const T hc = sH[r0 + r + 1][lane + 1];
      T cx = T(0), cy = T(0);
      T e = ex0[r];
      if (j >= 1) {
        const T dA = qdiv(sub_rn(hc, sH[r0 + r + 1][lane]), a.dy, a.rdy, a.fdy);
        e = add_rn(ex0[r], mul_rn(dA, K[r]));
        cx = dA;
        if (mye >= 0) {
          const long long q = I.p_exy + (long long)(i + r) * I.npey + mye;
          const int c = tr.oy + lane;
          const T psi = add_rn(mul_rn(a.bey[c], a.pExy[q]), mul_rn(a.cey[c], dA));
          a.pExy[q] = psi;
          e = add_rn(e, mul_rn(K[r], psi));
          cx = add_rn(dA, psi);
        }
      }
      Exo[id] = e;
      e = ey[r];
      if (i + r >= 1) {
        const T dB = qdiv(sub_rn(hc, sH[r0 + r][lane + 1]), a.dx, a.rdx, a.fdx);
        e = add_rn(ey[r], mul_rn(-dB, K[r]));
        cy = -dB;
        if (mxe[r] >= 0) {
          const long long q = I.p_eyx + (long long)mxe[r] * tr.pitch + j;
          const int c = tr.ox + r0 + r;
          const T psi = add_rn(mul_rn(a.bex[c], a.pEyx[q]), mul_rn(a.cex[c], dB));
          a.pEyx[q] = psi;
          e = add_rn(e, mul_rn(-K[r], psi));
          cy = sub_rn(cy, psi);
        }
      }
      Eyo[id] = e;
      const int di = r0 + r - tr.wdi, dj = lane - tr.wdj;
      if (di >= 0 && di < tr.wdn && dj >= 0 && dj < tr.wdn) {
        const long long slot = n % a.ring_len;
        T* rr = a.ring + (slot * a.n_design + I.goff + (long long)di * tr.wdn + dj) * 2;
        rr[0] = cx;
        rr[1] = cy;
      }
    }
    __syncthreads();  // sH is rewritten by the next tile
  }
}

// ---- vector forward step -------------------------------------------------------
// What the vector step does after its E update: the E sources and the
// output-line samples (kb_post's work; a separate launch per step cost 3 us).
// srow[x row]: -1, or where the row's source groups per column start in scol
// (Ex for ny columns, then Ey); dring: null in replays.
template <typename T>
struct StepPost {
  const int* srow;
  const int* scol;
  const int* start;
  const int* wave_row;
  const double* amp;
  const double* wave;
  long long n_steps;
  T* dring;
  long long nline;
};

__device__ __forceinline__ void tld(const float* p, float (&o)[4]) {
  const float4 v = *reinterpret_cast<const float4*>(p);
  o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w;
}
__device__ __forceinline__ void tld(const double* p, double (&o)[2]) {
  const double2 v = *reinterpret_cast<const double2*>(p);
  o[0] = v.x; o[1] = v.y;
}
// The vector at p when ok, else zeros.
template <typename T>
__device__ __forceinline__ void tld_if(const T* p, bool ok, T (&o)[kTileV<T>]) {
  if (ok) {
    tld(p, o);
  } else {
#pragma unroll
    for (int v = 0; v < kTileV<T>; ++v) o[v] = T(0);
  }
}
// Stores the vector's first n columns (n >= 1).
__device__ __forceinline__ void tst(float* p, const float (&o)[4], int n) {
  if (n >= 4) {
    *reinterpret_cast<float4*>(p) = make_float4(o[0], o[1], o[2], o[3]);
  } else {
    p[0] = o[0];
    if (n > 1) p[1] = o[1];
    if (n > 2) p[2] = o[2];
  }
}
__device__ __forceinline__ void tst(double* p, const double (&o)[2], int n) {
  if (n >= 2) *reinterpret_cast<double2*>(p) = make_double2(o[0], o[1]);
  else p[0] = o[0];
}

// CPML of a thread's columns (y axis) and row (x axis) of one field family.
// The y layers' psi rows hold whole groups of four columns, the x layers' rows
// have the fields' pitch, so psi and column coefficients are vectors like the
// fields; a column has CPML state exactly where its coefficient c is not 0.
// An edge thread loads everything in two rounds before its first use (fields
// and indices, then coefficients and psi): loaded where they are used, between
// the psi stores, they made one serial chain of memory latencies.
template <typename T, int NV>
struct ColPml {
  T b[NV], c[NV];
};
template <typename T>
__device__ __forceinline__ void load_cols(const T* b, const T* c, int at, bool ok,
                                          ColPml<T, kTileV<T>>& p) {
  tld_if<T>(b + at, ok, p.b);
  tld_if<T>(c + at, ok, p.c);
}
template <typename T>
struct RowPml {
  int m;
  T b, c;
};
template <typename T>
__device__ __forceinline__ RowPml<T> load_row(const int* map, const T* b, const T* c, int at,
                                              bool ok) {
  RowPml<T> p;
  p.m = ok ? __ldg(map + at) : -1;
  p.b = ok ? __ldg(b + at) : T(0);
  p.c = ok ? __ldg(c + at) : T(0);
  return p;
}

// Hz^{n+1/2} of NV interior columns without CPML state.
template <typename T, int NV>
__device__ __forceinline__ void h_cols(const BArgs<T>& a, const T (&ey)[NV], const T (&eyn)[NV],
                                       const T (&ex)[NV], T exr, const T (&hz)[NV], T (&h)[NV]) {
  const T up = QScale<T>::up;
  const T mch = -a.ch, mchs = mul_rn(mch, QScale<T>::down);
  T nA[NV], nB[NV];
  QCheck<T, true, true> range;
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    nA[v] = fma_rn(eyn[v], up, -mul_rn(ey[v], up));
    nB[v] = fma_rn(v + 1 < NV ? ex[v + 1 < NV ? v + 1 : 0] : exr, up, -mul_rn(ex[v], up));
    range.take(nA[v]);
    range.take(nB[v]);
  }
  bool fast = range.ok();
  if (range.kAgain && !fast) {
    fast = true;
#pragma unroll
    for (int v = 0; v < NV; ++v) fast = fast && range.sure(nA[v]) && range.sure(nB[v]);
  }
  if (a.fast && fast) {
#pragma unroll
    for (int v = 0; v < NV; ++v)
      h[v] = add_rn(hz[v], mul_rn(sub_rn(qscaled(nA[v], a.dx, a.rdx), qscaled(nB[v], a.dy, a.rdy)),
                                  mchs));
    return;
  }
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    const T dA = div_cold(sub_rn(eyn[v], ey[v]), a.dx);
    const T dB = div_cold(sub_rn(v + 1 < NV ? ex[v + 1 < NV ? v + 1 : 0] : exr, ex[v]), a.dy);
    h[v] = add_rn(hz[v], mul_rn(sub_rn(dA, dB), mch));
  }
}
// The same anywhere: kb_h's tests, and psi (vx, vy: before and after).
template <typename T, int NV>
__device__ __forceinline__ void h_cols_pml(const BArgs<T>& a, int j, int ny, bool row,
                                           const RowPml<T>& rp, const ColPml<T, NV>& cp,
                                           const T (&ey)[NV], const T (&eyn)[NV],
                                           const T (&ex)[NV], T exr, const T (&hz)[NV],
                                           T (&vx)[NV], T (&vy)[NV], T (&h)[NV]) {
  const T mch = -a.ch;
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    h[v] = hz[v];
    if (!row || j + v >= ny - 1) continue;
    const T nA = sub_rn(eyn[v], ey[v]);
    const T nB = sub_rn(v + 1 < NV ? ex[v + 1 < NV ? v + 1 : 0] : exr, ex[v]);
    T dA, dB;
    if (a.fast && qdiv_ok<T>(nA, nB)) {
      dA = qdiv_fast(nA, a.dx, a.rdx);
      dB = qdiv_fast(nB, a.dy, a.rdy);
    } else {
      dA = div_cold(nA, a.dx);
      dB = div_cold(nB, a.dy);
    }
    h[v] = add_rn(hz[v], mul_rn(sub_rn(dA, dB), mch));
    if (rp.m >= 0) {
      vx[v] = add_rn(mul_rn(rp.b, vx[v]), mul_rn(rp.c, dA));
      h[v] = add_rn(h[v], mul_rn(mch, vx[v]));
    }
    if (cp.c[v] != T(0)) {
      vy[v] = add_rn(mul_rn(cp.b[v], vy[v]), mul_rn(cp.c[v], dB));
      h[v] = add_rn(h[v], mul_rn(a.ch, vy[v]));
    }
  }
}

// The step of one thread's V columns of row r. Everything it needs is loaded
// at once; Hz of the row above and of the column to the left are recomputed
// (the left one by the first thread of a tile row, the others take their
// neighbour's by shuffle). EDGE: tiles with grid edges or CPML state.
template <typename T, bool EDGE>
__device__ __forceinline__ void tile_step(const BArgs<T>& a, const StepPost<T>& post,
                                          const TileRec& tr, long long n, int step_t) {
  constexpr int V = kTileV<T>, X = tile_x<T>(EDGE);
  const int L = (int)(n & 1);
  const int r = tr.i0 + threadIdx.y, j = tr.j0 + threadIdx.x * V;
  const bool live = !EDGE || (r < tr.nx_end && j < tr.ny);
  const int nv = EDGE ? (live ? min(V, tr.ny - j) : 0) : V;
  const int pitch = tr.pitch;
  const long long id = tr.base + (long long)threadIdx.y * pitch + threadIdx.x * V;
  const T* Ex = a.Ex2[L] + id;
  const T* Ey = a.Ey2[L] + id;
  const T* Hz = a.Hz2[L] + id;
  const bool top = !EDGE || (live && r >= 1);              // the row above exists
  const bool low = !EDGE || (live && r + 1 < tr.nx);       // the row below
  const bool right = !EDGE || (live && j + V < tr.ny);
  const bool left = threadIdx.x == 0 && (!EDGE || (live && j >= 1));
  T ey0[V], ey1[V], ey2[V], ex0[V], ex1[V], hz0[V], hz1[V], K[V];
  tld_if<T>(Ey - pitch, top, ey0);
  tld_if<T>(Ey, live, ey1);
  tld_if<T>(Ey + pitch, low, ey2);
  tld_if<T>(Ex - pitch, top, ex0);
  tld_if<T>(Ex, live, ex1);
  tld_if<T>(Hz - pitch, top, hz0);
  tld_if<T>(Hz, live, hz1);
  tld_if<T>(a.ce + id, live, K);
  const T exr0 = top && right ? Ex[V - pitch] : T(0), exr1 = right ? Ex[V] : T(0);
  T eyl[1] = {T(0)}, eyln[1] = {T(0)}, exl[1] = {T(0)}, hzl[1] = {T(0)};
  if (left) {
    eyl[0] = Ey[-1];
    if (low) eyln[0] = Ey[pitch - 1];
    exl[0] = Ex[-1];
    hzl[0] = Hz[-1];
  }
  T hp[V], h[V], hl[1] = {T(0)};
  ColPml<T, V> ce;
  RowPml<T> re;
  T wx[V], wy[V];  // E psi
  long long qex = 0, qey = 0;
  bool ecol = false;
  if constexpr (EDGE) {
    const int cy = tr.oy + (j - tr.j0), cx = tr.ox + (r - tr.i0);
    const int gh = live ? __ldg(a.ghy + (cy >> 2)) : -1, ge = live ? __ldg(a.gey + (cy >> 2)) : -1;
    const int gl = left ? __ldg(a.ghy + ((cy - 1) >> 2)) : -1;
    const RowPml<T> r1 = load_row<T>(a.mhx, a.bhx, a.chx, cx, live);
    const RowPml<T> r0 = load_row<T>(a.mhx, a.bhx, a.chx, cx - 1, top);
    re = load_row<T>(a.mex, a.bex, a.cex, cx, live);
    const long long qhx = tr.p_hzx + (long long)r1.m * pitch + j;
    const long long qhy = tr.p_hzy + (long long)r * tr.nphy + 4 * gh + (cy & 3);
    qex = tr.p_eyx + (long long)re.m * pitch + j;
    qey = tr.p_exy + (long long)r * tr.npey + 4 * ge + (cy & 3);
    ecol = ge >= 0;
    ColPml<T, V> cp;
    ColPml<T, 1> cl = {{T(0)}, {T(0)}};
    load_cols<T>(a.bhy, a.chy, cy, gh >= 0, cp);
    load_cols<T>(a.bey, a.cey, cy, ge >= 0, ce);
    T x1[V], y1[V], x0[V], y0[V], xl[1] = {T(0)}, yl[1] = {T(0)};
    tld_if<T>(a.pHzx2[L] + qhx, r1.m >= 0, x1);
    tld_if<T>(a.pHzy2[L] + qhy, gh >= 0, y1);
    tld_if<T>(a.pHzx2[L] + tr.p_hzx + (long long)r0.m * pitch + j, r0.m >= 0, x0);
    tld_if<T>(a.pHzy2[L] + qhy - tr.nphy, top && gh >= 0, y0);
    tld_if<T>(a.pEyx + qex, re.m >= 0, wx);
    tld_if<T>(a.pExy + qey, ge >= 0, wy);
    if (left && r1.m >= 0) xl[0] = a.pHzx2[L][qhx - 1];
    if (gl >= 0) {
      cl.b[0] = a.bhy[cy - 1];
      cl.c[0] = a.chy[cy - 1];
      yl[0] = a.pHzy2[L][tr.p_hzy + (long long)r * tr.nphy + 4 * gl + ((cy - 1) & 3)];
    }
    h_cols_pml<T, V>(a, j, tr.ny, top && r - 1 < tr.nx - 1, r0, cp, ey0, ey1, ex0, exr0, hz0, x0, y0,
                     hp);
    h_cols_pml<T, V>(a, j, tr.ny, live && r < tr.nx - 1, r1, cp, ey1, ey2, ex1, exr1, hz1, x1, y1,
                     h);
    h_cols_pml<T, 1>(a, j - 1, tr.ny, left && r < tr.nx - 1, r1, cl, eyl, eyln, exl, ex1[0], hzl, xl,
                     yl, hl);
    if (r1.m >= 0) tst(a.pHzx2[L ^ 1] + qhx, x1, V);
    if (gh >= 0) tst(a.pHzy2[L ^ 1] + qhy, y1, V);
  } else {
    h_cols<T, V>(a, ey0, ey1, ex0, exr0, hz0, hp);
    h_cols<T, V>(a, ey1, ey2, ex1, exr1, hz1, h);
    if (left) h_cols<T, 1>(a, eyl, eyln, exl, ex1[0], hzl, hl);
  }
  const T hs = __shfl_up_sync(0xffffffffu, h[V - 1], 1, X);
  const T hl0 = threadIdx.x == 0 ? hl[0] : hs;
  if (EDGE && !live) return;
  tst(a.Hz2[L ^ 1] + id, h, nv);
  // ---- Ex, Ey: kb_e's arithmetic (both quotients formed; each is used only
  // where its difference exists)
  const T up = QScale<T>::up, down = QScale<T>::down;
  T e[V], f[V], cx[V], cy[V], nA[V], nB[V];
  QCheck<T, true, true> range;
#pragma unroll
  for (int v = 0; v < V; ++v) {
    const T s = mul_rn(h[v], up);
    nA[v] = fma_rn(-(v > 0 ? h[v > 0 ? v - 1 : 0] : hl0), up, s);
    nB[v] = fma_rn(-hp[v], up, s);
    range.take(nA[v]);
    range.take(nB[v]);
  }
  bool fast = range.ok();
  if (range.kAgain && !fast) {
    fast = true;
#pragma unroll
    for (int v = 0; v < V; ++v) fast = fast && range.sure(nA[v]) && range.sure(nB[v]);
  }
  fast = fast && a.fast;
#pragma unroll
  for (int v = 0; v < V; ++v) {
    T dA, dB;
    if (fast) {
      dA = mul_rn(qscaled(nA[v], a.dy, a.rdy), down);
      dB = mul_rn(qscaled(nB[v], a.dx, a.rdx), down);
    } else {
      dA = div_cold(sub_rn(h[v], v > 0 ? h[v > 0 ? v - 1 : 0] : hl0), a.dy);
      dB = div_cold(sub_rn(h[v], hp[v]), a.dx);
    }
    e[v] = ex1[v];
    f[v] = ey1[v];
    cx[v] = cy[v] = T(0);
    if (!EDGE || j + v >= 1) {
      e[v] = add_rn(ex1[v], mul_rn(dA, K[v]));
      cx[v] = dA;
    }
    if (!EDGE || r >= 1) {
      f[v] = add_rn(ey1[v], mul_rn(-dB, K[v]));
      cy[v] = -dB;
    }
    if constexpr (EDGE) {
      if (ce.c[v] != T(0) && j + v >= 1) {
        wy[v] = add_rn(mul_rn(ce.b[v], wy[v]), mul_rn(ce.c[v], dA));
        e[v] = add_rn(e[v], mul_rn(K[v], wy[v]));
        cx[v] = add_rn(dA, wy[v]);
      }
      if (re.m >= 0 && r >= 1 && v < nv) {
        wx[v] = add_rn(mul_rn(re.b, wx[v]), mul_rn(re.c, dB));
        f[v] = add_rn(f[v], mul_rn(-K[v], wx[v]));
        cy[v] = sub_rn(cy[v], wx[v]);
      }
    }
  }
  if constexpr (EDGE) {
    if (ecol) tst(a.pExy + qey, wy, V);
    if (re.m >= 0) tst(a.pEyx + qex, wx, V);
  }
  if (tr.flags & kTileWindow) {
    const int di = (int)threadIdx.y - tr.wdi;
    if (di >= 0 && di < tr.wdn) {
      T* ring = a.ring + ((n % a.ring_len) * a.n_design + a.inst[tr.k].goff + (long long)di * tr.wdn) * 2;
#pragma unroll
      for (int v = 0; v < V; ++v) {
        const int dj = (int)threadIdx.x * V + v - tr.wdj;
        if (dj < 0 || dj >= tr.wdn) continue;
        ring[2 * dj] = cx[v];
        ring[2 * dj + 1] = cy[v];
      }
    }
  }
  if (tr.flags & kTilePost) {
    const int srow = post.srow ? post.srow[tr.ox + threadIdx.y] : -1;
    if (srow >= 0) {
#pragma unroll
      for (int v = 0; v < V; ++v) {
        if (v >= nv) continue;
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const int g = post.scol[srow + c * tr.ny + j + v];
          if (g < 0) continue;
          T x = c == 0 ? e[v] : f[v];
          for (int q = post.start[g]; q < post.start[g + 1]; ++q)
            x = add_double<T>(x, __dmul_rn(post.amp[q],
                                           post.wave[(long long)post.wave_row[q] * post.n_steps + n]));
          if (c == 0) e[v] = x;
          else f[v] = x;
        }
      }
    }
    const Inst& I = a.inst[tr.k];
    if (r == I.line_i && post.dring) {
      T* ring = post.dring + (long long)(step_t % kDftRing) * post.nline + I.loff + j;
#pragma unroll
      for (int v = 0; v < V; ++v)
        if (v < nv) ring[v] = f[v];
    }
  }
  tst(a.Ex2[L ^ 1] + id, e, nv);
  tst(a.Ey2[L ^ 1] + id, f, nv);
}

// One thread per 16-byte vector of a tile row, one tile per block; level n & 1
// is read and level (n & 1) ^ 1 written, as in kb_step, with kb_h's and kb_e's
// arithmetic, so the same bits. Edge and bulk tiles run as two kernels side
// by side: the edge code needs twice the registers, and mixed in one kernel
// the two kept missing the instruction cache (a third of all stalls).
//
// A step is bound by how many loads are in flight. Marching down the rows
// (one warp per 31-column strip, the form before this one) kept one row of
// 16 bytes per lane in flight, 25 KB per SM, and reached 2.9 TB/s; two columns
// per lane cut its instructions but also its warps and was slower (457 us).
// Here every thread issues eight vectors at once and has no loop; the Hz it
// recomputes costs 13 operations per cell. us per step, marching -> this: 256
// instances (36.1M cells) forward 376 -> 307, reverse 428 -> 381, 8 instances
// (1.5M cells) 37 -> 14 and 31 -> 14. The bulk tiles alone (about four fifths)
// took 180 us of 321 (before the range test became a chain of compares); scalar
// CPML code in 32-column edge tiles cost 70 more.
template <typename T, bool EDGE>
__global__ void __launch_bounds__(32 * tile_x<T>(false), sizeof(T) == 4 ? (EDGE ? PFB_MINB_EDGE : PFB_MINB_TILE) : 1) kb_tile(const __grid_constant__ BArgs<T> a,
                                                             const __grid_constant__ StepPost<T> post,
                                                             int step_t) {
  const TileRec tr = a.tiles[EDGE ? blockIdx.x : a.nedge + blockIdx.x];
  tile_step<T, EDGE>(a, post, tr, *a.base + step_t, step_t);
}

// Field pointers kb_post writes through: level 0 for the in-place split
// passes; for the fused step (flip = 1) the level step n has just written.
template <typename T>
struct BFields {
  T* Ex[2];
  T* Ey[2];
  T* Hz[2];
  int flip;
};

struct BSources {
  const long long* cell;  // pooled cell of each group
  const int* comp;        // 0 Ex, 1 Ey, 2 Hz
  const int* start;       // group q owns entries start[q] .. start[q+1]-1
  const int* wave_row;
  const double* amp;
  const double* wave;     // (rows, n_steps) waveform values at the family's times
  long long n_steps;
  int n_groups;
};

// Soft sources of one family (field += amp * waveform, in list order per
// cell, each term added in double and rounded once, as numpy's in-place add
// of a float64 scalar does) and, with `dring`, the step's Ey samples of the
// output lines into the DFT ring. Threads [0, n_groups) inject, the next
// nline threads sample: one launch is correct only when no group of this
// family sits on a line cell, which the host checks.
template <typename T>
__global__ void kb_post(BSources s, BFields<T> f, int family_h, const long long* base,
                        int step_t, const long long* lcell, long long nline, T* dring) {
  const long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long n = *base + step_t;
  const int lv = f.flip ? (int)((n & 1) ^ 1) : 0;
  T* Ex = f.Ex[lv];
  T* Ey = f.Ey[lv];
  T* Hz = f.Hz[lv];
  if (g < s.n_groups) {
    const int c = s.comp[g];
    if ((c == 2) != (family_h != 0)) return;
    T* F = c == 0 ? Ex : (c == 1 ? Ey : Hz);
    T v = F[s.cell[g]];
    for (int q = s.start[g]; q < s.start[g + 1]; ++q)
      v = add_double<T>(v, __dmul_rn(s.amp[q], s.wave[(long long)s.wave_row[q] * s.n_steps + n]));
    F[s.cell[g]] = v;
    return;
  }
  const long long c = g - s.n_groups;
  if (dring && c < nline) dring[(long long)(step_t % kDftRing) * nline + c] = Ey[lcell[c]];
}

// Folds n_pend ring samples (chunk steps t_first ..) into the line DFT in
// step order, acc += (exp(i w (n+1) dt) * Ey) * dt with the reference's two
// roundings per part (simulation.py:1116-1133). One thread per (cell, freq).
template <typename T>
__global__ void kb_dft_flush(const T* dring, long long nline, double* acc, const double* phase,
                             int n_freq, double dt, const long long* base, int t_first,
                             int n_pend) {
  const long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= nline * n_freq) return;
  const long long c = g / n_freq;
  const int f = (int)(g % n_freq);
  double re = acc[2 * g], im = acc[2 * g + 1];
  const long long n0 = *base;
  for (int q = 0; q < n_pend; ++q) {
    const int tt = t_first + q;
    const double v = (double)dring[(long long)(tt % kDftRing) * nline + c];
    const double* p = phase + ((n0 + tt) * n_freq + f) * 2;
    re = __dadd_rn(re, __dmul_rn(__dmul_rn(p[0], v), dt));
    im = __dadd_rn(im, __dmul_rn(__dmul_rn(p[1], v), dt));
  }
  acc[2 * g] = re;
  acc[2 * g + 1] = im;
}

__global__ void kb_set(long long* v, long long x) { *v = x; }

// Writes packed design-window coefficients into the pooled ce array.
template <typename T>
__global__ void kb_scatter_design(const Inst* inst, int n_inst, const T* src, T* ce) {
  const int k = blockIdx.y;
  if (k >= n_inst) return;
  const Inst& I = inst[k];
  const int n = I.dn * I.dn;
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x) {
    const int di = q / I.dn, dj = q % I.dn;
    ce[I.off + (long long)(I.di0 + di) * I.pitch + I.dj0 + dj] = src[I.goff + q];
  }
}

// ---- adjoint ---------------------------------------------------------------
template <typename T>
struct AArgs {
  T *aEx, *aEy, *aHz, *aHzx, *aHzy, *aExy, *aEyx;  // adjoint state
  T *gA, *gB, *hA, *hB;                             // adjoints of the per-cell differences
  double* grad;                                     // dL/dK per design cell
  const double* cot;                                // DFT cotangent, (line cells, n_freq)
  const double* phase;                              // exp(i w (n+1) dt), (n_steps, n_freq)
  int n_freq;
  double dt;
  // The fused reverse step's double-buffered state (level 0 = the arrays
  // above): the E transpose of step m writes gA / gB into level m & 1; the H
  // transpose of step n reads aHz and its psi adjoints from level (n + 1) & 1
  // and writes them into level n & 1.
  T *aHz2[2], *aHzx2[2], *aHzy2[2], *gA2[2], *gB2[2];
};

// The adjoint arithmetic is written with explicitly rounded operations, so
// its result does not depend on the tile shape (no compiler contraction).

// Transpose of the H update: gathers the E-update terms into aHz
// (gA from j and j+1, gB from i and i+1), then the H psi adjoints and
// hA = adjoint of dEy/dx, hB = adjoint of dEx/dy.
template <typename T, int R>
__global__ void __launch_bounds__(32 * kWarps) kb_adj_h(const __grid_constant__ BArgs<T> a,
                                                       const __grid_constant__ AArgs<T> d) {
  for (int t = blockIdx.x; t < a.ntiles; t += gridDim.x) {
    const TileRec tr = a.tiles[t];
    const int r0 = threadIdx.y * R;
    const int i = tr.i0 + r0, j = tr.j0 + threadIdx.x;
    if (j >= tr.ny || i >= tr.nx) continue;
    const long long id0 = tr.base + (long long)r0 * tr.pitch + threadIdx.x;
    const bool jn = j + 1 < tr.ny;
    T ah[R], ga0[R], ga1[R], gb[R + 1];
    int mx[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const bool ok = i + r < tr.nx;
      const long long id = id0 + (long long)r * tr.pitch;
      ah[r] = ok ? d.aHz[id] : T(0);
      ga0[r] = ok ? d.gA[id] : T(0);
      ga1[r] = (ok && jn) ? d.gA[id + 1] : T(0);
      gb[r] = ok ? d.gB[id] : T(0);
      mx[r] = ok ? a.mhx[tr.ox + r0 + r] : -1;
    }
    gb[R] = (i + R < tr.nx) ? d.gB[id0 + (long long)R * tr.pitch] : T(0);
    const int my = a.mhy[tr.oy + threadIdx.x];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if (i + r >= tr.nx) break;
      const long long id = id0 + (long long)r * tr.pitch;
      const T h = fma_rn(sub_rn(gb[r], gb[r + 1]), a.idx, fma_rn(sub_rn(ga0[r], ga1[r]), a.idy, ah[r]));
      T ha = T(0), hb = T(0);
      if (i + r < tr.nx - 1 && j < tr.ny - 1) {
        ha = mul_rn(-a.ch, h);
        hb = mul_rn(a.ch, h);
        if (mx[r] >= 0 || my >= 0) {
          const Inst& I = a.inst[tr.k];
          if (mx[r] >= 0) {
            const long long q = I.p_hzx + (long long)mx[r] * tr.pitch + j;
            const int c = tr.ox + r0 + r;
            const T ap = fma_rn(-a.ch, h, d.aHzx[q]);
            ha = fma_rn(a.chx[c], ap, ha);
            d.aHzx[q] = mul_rn(a.bhx[c], ap);
          }
          if (my >= 0) {
            const long long q = I.p_hzy + (long long)(i + r) * I.nphy + my;
            const int c = tr.oy + threadIdx.x;
            const T ap = fma_rn(a.ch, h, d.aHzy[q]);
            hb = fma_rn(a.chy[c], ap, hb);
            d.aHzy[q] = mul_rn(a.bhy[c], ap);
          }
        }
      }
      d.aHz[id] = h;
      d.hA[id] = ha;
      d.hB[id] = hb;
    }
  }
}

// Cell-local part of the reverse pass. With E2, first finishes step n+1's E
// adjoints from the H update's differences (hA from rows i-1 and i, hB from
// columns j-1 and j). With E, then runs the transpose of step n's E update
// (n = *base + step_t): the adjoint source on the output line,
// dt * sum_f Re(conj(G_f) phase_f^n); the K gradient of design cells; the E
// psi adjoints; gA / gB, the adjoints of dHz/dy in Ex and dHz/dx in Ey.
template <typename T, int R, bool E2, bool E>
__global__ void __launch_bounds__(32 * kWarps) kb_adj_cell(const __grid_constant__ BArgs<T> a,
                                                          const __grid_constant__ AArgs<T> d,
                                                          int step_t) {
  for (int t = blockIdx.x; t < a.ntiles; t += gridDim.x) {
    const TileRec tr = a.tiles[t];
    const int r0 = threadIdx.y * R;
    const int i = tr.i0 + r0, j = tr.j0 + threadIdx.x;
    if (j >= tr.ny || i >= tr.nx) continue;
    const long long id0 = tr.base + (long long)r0 * tr.pitch + threadIdx.x;
    T lx[R], ly[R], ha[R + 1], hb0[R], hb1[R], K[R];
    int mx[R];
    if (E2) ha[0] = i >= 1 ? d.hA[id0 - tr.pitch] : T(0);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const bool ok = i + r < tr.nx;
      const long long id = id0 + (long long)r * tr.pitch;
      lx[r] = ok ? d.aEx[id] : T(0);
      ly[r] = ok ? d.aEy[id] : T(0);
      if (E2) {
        ha[r + 1] = ok ? d.hA[id] : T(0);
        hb0[r] = ok ? d.hB[id] : T(0);
        hb1[r] = (ok && j >= 1) ? d.hB[id - 1] : T(0);
      }
      if (E) {
        K[r] = ok ? a.ce[id] : T(0);
        mx[r] = ok ? a.mex[tr.ox + r0 + r] : -1;
      }
    }
    const int my = E ? a.mey[tr.oy + threadIdx.x] : -1;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if (i + r >= tr.nx) break;
      const long long id = id0 + (long long)r * tr.pitch;
      T x = lx[r], y = ly[r];
      if (E2) {
        y = fma_rn(sub_rn(ha[r], ha[r + 1]), a.idx, y);
        x = fma_rn(sub_rn(hb1[r], hb0[r]), a.idy, x);
      }
      if (E) {
        const long long n = *a.base + step_t;
        const Inst& I = a.inst[tr.k];
        if (i + r == I.line_i) {
          const double* ph = d.phase + n * d.n_freq * 2;
          const double* g = d.cot + (I.loff + j) * d.n_freq * 2;
          double s = 0.0;
          for (int f = 0; f < d.n_freq; ++f)
            s = __dadd_rn(s, __dadd_rn(__dmul_rn(g[2 * f], ph[2 * f]),
                                       __dmul_rn(g[2 * f + 1], ph[2 * f + 1])));
          y = (T)__dadd_rn((double)y, __dmul_rn(d.dt, s));
        }
        const int di = r0 + r - tr.wdi, dj = (int)threadIdx.x - tr.wdj;
        if (di >= 0 && di < tr.wdn && dj >= 0 && dj < tr.wdn) {
          const long long dc = I.goff + (long long)di * tr.wdn + dj;
          const T* rr = a.ring + ((n % a.ring_len) * a.n_design + dc) * 2;
          d.grad[dc] = __dadd_rn(d.grad[dc], __dadd_rn(__dmul_rn((double)x, (double)rr[0]),
                                                       __dmul_rn((double)y, (double)rr[1])));
        }
        T ga = T(0), gb = T(0);
        if (j >= 1) {
          ga = mul_rn(K[r], x);
          if (my >= 0) {
            const long long q = I.p_exy + (long long)(i + r) * I.npey + my;
            const int c = tr.oy + threadIdx.x;
            const T ap = fma_rn(K[r], x, d.aExy[q]);
            ga = fma_rn(a.cey[c], ap, ga);
            d.aExy[q] = mul_rn(a.bey[c], ap);
          }
        }
        if (i + r >= 1) {
          gb = mul_rn(-K[r], y);
          if (mx[r] >= 0) {
            const long long q = I.p_eyx + (long long)mx[r] * tr.pitch + j;
            const int c = tr.ox + r0 + r;
            const T ap = fma_rn(-K[r], y, d.aEyx[q]);
            gb = fma_rn(a.cex[c], ap, gb);
            d.aEyx[q] = mul_rn(a.bex[c], ap);
          }
        }
        d.gA[id] = ga;
        d.gB[id] = gb;
      }
      d.aEx[id] = x;
      d.aEy[id] = y;
    }
  }
}

// ---- fused reverse step -------------------------------------------------------
// One launch per reverse step n, on double-buffered adjoint state: the H
// transpose of step n (HT: gather gA / gB into aHz, H psi adjoints, hA / hB),
// the gather of hA / hB into step n's E adjoints, then the E transpose of step
// n - 1 (ET: line source, design gradient, E psi adjoints, new gA / gB). hA
// and hB never leave shared memory: a tile recomputes them on its one-cell
// halo (the row above, the column to the left) from the previous level.
// Without HT the launch is the E transpose of step n alone (a chunk's first
// launch); without ET it ends after the gather (its last). Every cell's
// arithmetic is kb_adj_h's and kb_adj_cell's, operation for operation.

// aHz after the H transpose of one cell and its hA / hB (psi adjoints stored
// only when the output pointers are given).
template <typename T>
__device__ __forceinline__ void adj_h_value(const BArgs<T>& a, const Inst& I, int i, int j,
                                            int nx, int ny, int crow, int ccol, int mx, int my,
                                            T ah, T ga0, T ga1, T gb0, T gb1, const T* pzx,
                                            T* pzxo, const T* pzy, T* pzyo, T& h, T& ha,
                                            T& hb) {
  h = fma_rn(sub_rn(gb0, gb1), a.idx, fma_rn(sub_rn(ga0, ga1), a.idy, ah));
  ha = T(0);
  hb = T(0);
  if (i < nx - 1 && j < ny - 1) {
    ha = mul_rn(-a.ch, h);
    hb = mul_rn(a.ch, h);
    if (mx >= 0) {
      const long long q = I.p_hzx + (long long)mx * I.pitch + j;
      const T ap = fma_rn(-a.ch, h, pzx[q]);
      ha = fma_rn(a.chx[crow], ap, ha);
      if (pzxo) pzxo[q] = mul_rn(a.bhx[crow], ap);
    }
    if (my >= 0) {
      const long long q = I.p_hzy + (long long)i * I.nphy + my;
      const T ap = fma_rn(a.ch, h, pzy[q]);
      hb = fma_rn(a.chy[ccol], ap, hb);
      if (pzyo) pzyo[q] = mul_rn(a.bhy[ccol], ap);
    }
  }
}

template <typename T, int R, bool HT, bool ET>
__global__ void __launch_bounds__(32 * kWarps, PFB_MINB_ASTEP) kb_adj_step(
    const __grid_constant__ BArgs<T> a, const __grid_constant__ AArgs<T> d, int step_t) {
  constexpr int TR = kWarps * R;
  static_assert(TR <= 32, "the halo column is one warp's work");
  __shared__ T sA[TR + 1][33];  // hA: [1 + row][1 + column]; row 0 = halo row
  __shared__ T sB[TR + 1][33];  // hB: column 0 = halo column
  const long long n = *a.base + step_t;
  const long long m = HT ? n - 1 : n;  // the step of the E transpose
  const int lg = (int)(n & 1);         // gA / gB level the H transpose reads
  const int lh = (int)((n + 1) & 1);   // aHz / H psi adjoint level it reads
  const T* gA = d.gA2[lg];
  const T* gB = d.gB2[lg];
  T* gAo = d.gA2[(int)(m & 1)];
  T* gBo = d.gB2[(int)(m & 1)];
  const T* aHz = d.aHz2[lh];
  T* aHzo = d.aHz2[lh ^ 1];
  const T* pzx = d.aHzx2[lh];
  const T* pzy = d.aHzy2[lh];
  T* pzxo = d.aHzx2[lh ^ 1];
  T* pzyo = d.aHzy2[lh ^ 1];
  const int lane = threadIdx.x;
  const int r0 = threadIdx.y * R;
  for (int t = blockIdx.x; t < a.ntiles; t += gridDim.x) {
    const TileRec tr = a.tiles[t];
    const Inst& I = a.inst[tr.k];
    const int i = tr.i0 + r0, j = tr.j0 + lane;
    const bool jv = j < tr.ny;
    const long long id0 = tr.base + (long long)r0 * tr.pitch + lane;
    // ---- loads, all before the barrier: the E adjoints and coefficients of
    // the own cells, then (HT) their H-transpose inputs and the halo's
    T lx[R], ly[R], K[R];
    int mxe[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const bool ok = jv && i + r < tr.nx;
      const long long id = id0 + (long long)r * tr.pitch;
      lx[r] = ok ? d.aEx[id] : T(0);
      ly[r] = ok ? d.aEy[id] : T(0);
      if (ET) {
        K[r] = ok ? a.ce[id] : T(0);
        mxe[r] = ok ? a.mex[tr.ox + r0 + r] : -1;
      }
    }
    const int mye = (ET && jv) ? a.mey[tr.oy + lane] : -1;
    if (HT) {
      T ah[R], ga0[R], ga1[R], gb[R + 1];
      int mxh[R];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const bool ok = jv && i + r < tr.nx;
        const long long id = id0 + (long long)r * tr.pitch;
        ah[r] = ok ? aHz[id] : T(0);
        ga0[r] = ok ? gA[id] : T(0);
        ga1[r] = (ok && j + 1 < tr.ny) ? gA[id + 1] : T(0);
        gb[r] = ok ? gB[id] : T(0);
        mxh[r] = ok ? a.mhx[tr.ox + r0 + r] : -1;
      }
      gb[R] = (jv && i + R < tr.nx) ? gB[id0 + (long long)R * tr.pitch] : T(0);
      const int myh = jv ? a.mhy[tr.oy + lane] : -1;
      // the halo cell of this thread, if any: warp 0 row i0 - 1 (its hA),
      // warp 1 column j0 - 1 at tile row `lane` (its hB)
      int hrole = 0, hi = 0, hj = 0, hcrow = 0, hccol = 0;
      if (threadIdx.y == 0 && tr.i0 >= 1 && jv) {
        hrole = 1;
        hi = tr.i0 - 1;
        hj = j;
        hcrow = tr.ox - 1;
        hccol = tr.oy + lane;
      } else if (threadIdx.y == 1 && lane < TR && tr.j0 >= 1 && tr.i0 + lane < tr.nx) {
        hrole = 2;
        hi = tr.i0 + lane;
        hj = tr.j0 - 1;
        hcrow = tr.ox + lane;
        hccol = tr.oy - 1;
      }
      T hah = T(0), hga0 = T(0), hga1 = T(0), hgb0 = T(0), hgb1 = T(0);
      int hmx = -1, hmy = -1;
      if (hrole) {
        const long long id = tr.base + (long long)(hi - tr.i0) * tr.pitch + (hj - tr.j0);
        hah = aHz[id];
        hga0 = gA[id];
        hga1 = hj + 1 < tr.ny ? gA[id + 1] : T(0);
        hgb0 = gB[id];
        hgb1 = hi + 1 < tr.nx ? gB[id + tr.pitch] : T(0);
        hmx = a.mhx[hcrow];
        hmy = a.mhy[hccol];
      }
      // ---- H transpose of the own cells
#pragma unroll
      for (int r = 0; r < R; ++r) {
        T h = T(0), ha = T(0), hb = T(0);
        if (jv && i + r < tr.nx) {
          adj_h_value<T>(a, I, i + r, j, tr.nx, tr.ny, tr.ox + r0 + r, tr.oy + lane, mxh[r], myh,
                         ah[r], ga0[r], ga1[r], gb[r], gb[r + 1], pzx, pzxo, pzy, pzyo, h, ha,
                         hb);
          aHzo[id0 + (long long)r * tr.pitch] = h;
        }
        sA[r0 + r + 1][lane + 1] = ha;
        sB[r0 + r + 1][lane + 1] = hb;
      }
      // ---- the halo cell, recomputed from the read level (psi not stored)
      {
        T h = T(0), ha = T(0), hb = T(0);
        if (hrole)
          adj_h_value<T>(a, I, hi, hj, tr.nx, tr.ny, hcrow, hccol, hmx, hmy, hah, hga0, hga1,
                         hgb0, hgb1, pzx, nullptr, pzy, nullptr, h, ha, hb);
        if (threadIdx.y == 0) sA[0][lane + 1] = hrole == 1 ? ha : T(0);
        if (threadIdx.y == 1 && lane < TR) sB[lane + 1][0] = hrole == 2 ? hb : T(0);
      }
      __syncthreads();
    }
    // ---- E adjoints: finish step n's (HT), then the E transpose of step m (ET)
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if (!(jv && i + r < tr.nx)) break;
      const long long id = id0 + (long long)r * tr.pitch;
      T x = lx[r], y = ly[r];
      if (HT) {
        y = fma_rn(sub_rn(sA[r0 + r][lane + 1], sA[r0 + r + 1][lane + 1]), a.idx, y);
        x = fma_rn(sub_rn(sB[r0 + r + 1][lane], sB[r0 + r + 1][lane + 1]), a.idy, x);
      }
      if (ET) {
        if (i + r == I.line_i) {
          const double* ph = d.phase + m * d.n_freq * 2;
          const double* g = d.cot + (I.loff + j) * d.n_freq * 2;
          double sum = 0.0;
          for (int f = 0; f < d.n_freq; ++f)
            sum = __dadd_rn(sum, __dadd_rn(__dmul_rn(g[2 * f], ph[2 * f]),
                                           __dmul_rn(g[2 * f + 1], ph[2 * f + 1])));
          y = (T)__dadd_rn((double)y, __dmul_rn(d.dt, sum));
        }
        const int di = r0 + r - tr.wdi, dj = lane - tr.wdj;
        if (di >= 0 && di < tr.wdn && dj >= 0 && dj < tr.wdn) {
          const long long dc = I.goff + (long long)di * tr.wdn + dj;
          const T* rr = a.ring + ((m % a.ring_len) * a.n_design + dc) * 2;
          d.grad[dc] = __dadd_rn(d.grad[dc], __dadd_rn(__dmul_rn((double)x, (double)rr[0]),
                                                       __dmul_rn((double)y, (double)rr[1])));
        }
        T ga = T(0), gbv = T(0);
        if (j >= 1) {
          ga = mul_rn(K[r], x);
          if (mye >= 0) {
            const long long q = I.p_exy + (long long)(i + r) * I.npey + mye;
            const int c = tr.oy + lane;
            const T ap = fma_rn(K[r], x, d.aExy[q]);
            ga = fma_rn(a.cey[c], ap, ga);
            d.aExy[q] = mul_rn(a.bey[c], ap);
          }
        }
        if (i + r >= 1) {
          gbv = mul_rn(-K[r], y);
          if (mxe[r] >= 0) {
            const long long q = I.p_eyx + (long long)mxe[r] * tr.pitch + j;
            const int c = tr.ox + r0 + r;
            const T ap = fma_rn(-K[r], y, d.aEyx[q]);
            gbv = fma_rn(a.cex[c], ap, gbv);
            d.aEyx[q] = mul_rn(a.bex[c], ap);
          }
        }
        gAo[id] = ga;
        gBo[id] = gbv;
      }
      d.aEx[id] = x;
      d.aEy[id] = y;
    }
    if (HT) __syncthreads();  // sA / sB are rewritten by the next tile
  }
}

// ---- vector reverse step -------------------------------------------------------
// H transpose of NV columns (adj_h_value's arithmetic). EDGE: row / col say
// whether the forward update exists, vx / vy are the psi adjoints before and
// after.
template <typename T, int NV, bool EDGE>
__device__ __forceinline__ void adj_h_cols(const BArgs<T>& a, int j, int ny, bool row,
                                           const RowPml<T>& rp, const ColPml<T, NV>& cp,
                                           const T (&ah)[NV], const T (&ga)[NV], T gar,
                                           const T (&gb)[NV], const T (&gbn)[NV], T (&vx)[NV],
                                           T (&vy)[NV], T (&h)[NV], T (&ha)[NV], T (&hb)[NV]) {
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    const T gr = v + 1 < NV ? ga[v + 1 < NV ? v + 1 : 0] : gar;
    h[v] = fma_rn(sub_rn(gb[v], gbn[v]), a.idx, fma_rn(sub_rn(ga[v], gr), a.idy, ah[v]));
    ha[v] = hb[v] = T(0);
    if (EDGE && (!row || j + v >= ny - 1)) continue;
    ha[v] = mul_rn(-a.ch, h[v]);
    hb[v] = mul_rn(a.ch, h[v]);
    if constexpr (EDGE) {
      if (rp.m >= 0) {
        const T ap = fma_rn(-a.ch, h[v], vx[v]);
        ha[v] = fma_rn(rp.c, ap, ha[v]);
        vx[v] = mul_rn(rp.b, ap);
      }
      if (cp.c[v] != T(0)) {
        const T ap = fma_rn(a.ch, h[v], vy[v]);
        hb[v] = fma_rn(cp.c[v], ap, hb[v]);
        vy[v] = mul_rn(cp.b[v], ap);
      }
    }
  }
}

// The reverse step of one thread's V columns of row r: the H transpose of
// step n (its own cells, the row above for hA, the column to the left for
// hB), then step n's E adjoints and the E transpose of step m = n - 1 (or of
// step n alone when HT is false), as kb_adj_step.
template <typename T, bool HT, bool ET, bool EDGE>
__device__ __forceinline__ void adj_tile_step(const BArgs<T>& a, const AArgs<T>& d,
                                              const TileRec& tr, long long n) {
  constexpr int V = kTileV<T>, X = tile_x<T>(EDGE);
  const long long m = HT ? n - 1 : n;  // the step of the E transpose
  const int lg = (int)(n & 1), lh = (int)((n + 1) & 1), lm = (int)(m & 1);
  const int r = tr.i0 + threadIdx.y, j = tr.j0 + threadIdx.x * V;
  const bool live = !EDGE || (r < tr.nx_end && j < tr.ny);
  const int nv = EDGE ? (live ? min(V, tr.ny - j) : 0) : V;
  const int pitch = tr.pitch;
  const long long id = tr.base + (long long)threadIdx.y * pitch + threadIdx.x * V;
  T x[V], y[V], K[V];
  tld_if<T>(d.aEx + id, live, x);
  tld_if<T>(d.aEy + id, live, y);
  if (ET) tld_if<T>(a.ce + id, live, K);
  ColPml<T, V> ce;
  RowPml<T> re;
  T wx[V], wy[V];  // E psi adjoints
  long long qex = 0, qey = 0;
  bool ecol = false;
  const int cy = tr.oy + (j - tr.j0), cx = tr.ox + (r - tr.i0);
  if constexpr (EDGE && ET) {
    const int ge = live ? __ldg(a.gey + (cy >> 2)) : -1;
    re = load_row<T>(a.mex, a.bex, a.cex, cx, live);
    ecol = ge >= 0;
    qex = tr.p_eyx + (long long)re.m * pitch + j;
    qey = tr.p_exy + (long long)r * tr.npey + 4 * ge + (cy & 3);
    load_cols<T>(a.bey, a.cey, cy, ecol, ce);
    tld_if<T>(d.aEyx + qex, re.m >= 0, wx);
    tld_if<T>(d.aExy + qey, ecol, wy);
  }
  if (HT) {
    const T* gA = d.gA2[lg] + id;
    const T* gB = d.gB2[lg] + id;
    const T* aH = d.aHz2[lh] + id;
    const bool top = !EDGE || (live && r >= 1);
    const bool low = !EDGE || (live && r + 1 < tr.nx);
    const bool right = !EDGE || (live && j + V < tr.ny);
    const bool left = threadIdx.x == 0 && (!EDGE || (live && j >= 1));
    T ah0[V], ah1[V], ga0[V], ga1[V], gb0[V], gb1[V], gb2[V];
    tld_if<T>(aH - pitch, top, ah0);
    tld_if<T>(aH, live, ah1);
    tld_if<T>(gA - pitch, top, ga0);
    tld_if<T>(gA, live, ga1);
    tld_if<T>(gB - pitch, top, gb0);
    tld_if<T>(gB, live, gb1);
    tld_if<T>(gB + pitch, low, gb2);
    const T gar0 = top && right ? gA[V - pitch] : T(0), gar1 = right ? gA[V] : T(0);
    T ahl[1] = {T(0)}, gal[1] = {T(0)}, gbl[1] = {T(0)}, gbln[1] = {T(0)};
    if (left) {
      ahl[0] = aH[-1];
      gal[0] = gA[-1];
      gbl[0] = gB[-1];
      if (low) gbln[0] = gB[pitch - 1];
    }
    T h[V], ha[V], hb[V], hap[V], t0[V], t1[V], hl[1], hal[1], hbl[1] = {T(0)};
    ColPml<T, V> cp;
    ColPml<T, 1> cl = {{T(0)}, {T(0)}};
    RowPml<T> r0, r1;
    T x1[V], y1[V], x0[V], y0[V], xl[1] = {T(0)}, yl[1] = {T(0)};
    long long qhx = 0, qhy = 0;
    int gh = -1;
    if constexpr (EDGE) {
      gh = live ? __ldg(a.ghy + (cy >> 2)) : -1;
      const int gl = left ? __ldg(a.ghy + ((cy - 1) >> 2)) : -1;
      r1 = load_row<T>(a.mhx, a.bhx, a.chx, cx, live);
      r0 = load_row<T>(a.mhx, a.bhx, a.chx, cx - 1, top);
      qhx = tr.p_hzx + (long long)r1.m * pitch + j;
      qhy = tr.p_hzy + (long long)r * tr.nphy + 4 * gh + (cy & 3);
      load_cols<T>(a.bhy, a.chy, cy, gh >= 0, cp);
      tld_if<T>(d.aHzx2[lh] + qhx, r1.m >= 0, x1);
      tld_if<T>(d.aHzy2[lh] + qhy, gh >= 0, y1);
      tld_if<T>(d.aHzx2[lh] + tr.p_hzx + (long long)r0.m * pitch + j, r0.m >= 0, x0);
      tld_if<T>(d.aHzy2[lh] + qhy - tr.nphy, top && gh >= 0, y0);
      if (left && r1.m >= 0) xl[0] = d.aHzx2[lh][qhx - 1];
      if (gl >= 0) {
        cl.b[0] = a.bhy[cy - 1];
        cl.c[0] = a.chy[cy - 1];
        yl[0] = d.aHzy2[lh][tr.p_hzy + (long long)r * tr.nphy + 4 * gl + ((cy - 1) & 3)];
      }
    }
    adj_h_cols<T, V, EDGE>(a, j, tr.ny, top && r - 1 < tr.nx - 1, r0, cp, ah0, ga0, gar0, gb0, gb1,
                           x0, y0, t0, hap, t1);
    adj_h_cols<T, V, EDGE>(a, j, tr.ny, live && r < tr.nx - 1, r1, cp, ah1, ga1, gar1, gb1, gb2, x1,
                           y1, h, ha, hb);
    if (left)
      adj_h_cols<T, 1, EDGE>(a, j - 1, tr.ny, r < tr.nx - 1, r1, cl, ahl, gal, ga1[0], gbl, gbln,
                             xl, yl, hl, hal, hbl);
    if constexpr (EDGE) {
      if (r1.m >= 0) tst(d.aHzx2[lh ^ 1] + qhx, x1, V);
      if (gh >= 0) tst(d.aHzy2[lh ^ 1] + qhy, y1, V);
    }
    const T hs = __shfl_up_sync(0xffffffffu, hb[V - 1], 1, X);
    const T hb0 = threadIdx.x == 0 ? hbl[0] : hs;
    if (EDGE && !live) return;
    tst(d.aHz2[lh ^ 1] + id, h, nv);
#pragma unroll
    for (int v = 0; v < V; ++v) {
      y[v] = fma_rn(sub_rn(hap[v], ha[v]), a.idx, y[v]);
      x[v] = fma_rn(sub_rn(v > 0 ? hb[v > 0 ? v - 1 : 0] : hb0, hb[v]), a.idy, x[v]);
    }
  } else if (EDGE && !live) {
    return;
  }
  if (ET) {
    if (tr.flags & kTilePost) {
      const Inst& I = a.inst[tr.k];
      if (r == I.line_i) {
        const double* ph = d.phase + m * d.n_freq * 2;
#pragma unroll
        for (int v = 0; v < V; ++v) {
          if (v >= nv) continue;
          const double* g = d.cot + (I.loff + j + v) * d.n_freq * 2;
          double sum = 0.0;
          for (int f = 0; f < d.n_freq; ++f)
            sum = __dadd_rn(sum, __dadd_rn(__dmul_rn(g[2 * f], ph[2 * f]),
                                           __dmul_rn(g[2 * f + 1], ph[2 * f + 1])));
          y[v] = (T)__dadd_rn((double)y[v], __dmul_rn(d.dt, sum));
        }
      }
    }
    if (tr.flags & kTileWindow) {
      const int di = (int)threadIdx.y - tr.wdi;
      if (di >= 0 && di < tr.wdn) {
        const long long row = a.inst[tr.k].goff + (long long)di * tr.wdn;
        const T* ring = a.ring + ((m % a.ring_len) * a.n_design + row) * 2;
#pragma unroll
        for (int v = 0; v < V; ++v) {
          const int dj = (int)threadIdx.x * V + v - tr.wdj;
          if (dj < 0 || dj >= tr.wdn) continue;
          d.grad[row + dj] =
              __dadd_rn(d.grad[row + dj], __dadd_rn(__dmul_rn((double)x[v], (double)ring[2 * dj]),
                                                    __dmul_rn((double)y[v], (double)ring[2 * dj + 1])));
        }
      }
    }
    T gav[V], gbv[V];
#pragma unroll
    for (int v = 0; v < V; ++v) {
      gav[v] = !EDGE || j + v >= 1 ? mul_rn(K[v], x[v]) : T(0);
      gbv[v] = !EDGE || r >= 1 ? mul_rn(-K[v], y[v]) : T(0);
      if constexpr (EDGE && ET) {
        if (ce.c[v] != T(0) && j + v >= 1) {
          const T ap = fma_rn(K[v], x[v], wy[v]);
          gav[v] = fma_rn(ce.c[v], ap, gav[v]);
          wy[v] = mul_rn(ce.b[v], ap);
        }
        if (re.m >= 0 && r >= 1 && v < nv) {
          const T ap = fma_rn(-K[v], y[v], wx[v]);
          gbv[v] = fma_rn(re.c, ap, gbv[v]);
          wx[v] = mul_rn(re.b, ap);
        }
      }
    }
    if constexpr (EDGE && ET) {
      if (ecol) tst(d.aExy + qey, wy, V);
      if (re.m >= 0) tst(d.aEyx + qex, wx, V);
    }
    tst(d.gA2[lm] + id, gav, nv);
    tst(d.gB2[lm] + id, gbv, nv);
  }
  tst(d.aEx + id, x, nv);
  tst(d.aEy + id, y, nv);
}

// kb_adj_step's work in the shape of kb_tile; same levels and arithmetic, so
// the same bits.
template <typename T, bool HT, bool ET, bool EDGE>
__global__ void __launch_bounds__(32 * tile_x<T>(false), sizeof(T) == 4 ? (EDGE ? PFB_MINB_AEDGE : PFB_MINB_ATILE) : 1) kb_adj_tile(
    const __grid_constant__ BArgs<T> a, const __grid_constant__ AArgs<T> d, int step_t) {
  const TileRec tr = a.tiles[EDGE ? blockIdx.x : a.nedge + blockIdx.x];
  adj_tile_step<T, HT, ET, EDGE>(a, d, tr, *a.base + step_t);
}

}  // namespace b2d
}  // namespace pfb
