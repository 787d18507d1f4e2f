// kernels_vec3d.cuh - H and E passes of 3D grids, one 16-byte vector of z cells per thread.
//
// The per-component arithmetic and its order are the scalar passes'
// (cell_update.cuh; src/photonfdtd/simulation.py:1252-1309), so the bits are
// too. What bounds a step here is memory latency and issue slots, not FLOPs:
// with one cell per thread the passes ran 222 (H) and 414 (E with ADE)
// instructions per cell at 4.2 TB/s, most of them addresses, bounds and CPML
// tests that V cells of one row share. Rows are padded to 32 bytes, short
// ones to 16 (StepArgs::pz), so every row's vectors are aligned. At 256^3 without CPML
// the H pass now runs 88 instructions per cell at 5.5 TB/s of DRAM traffic
// (84% of a plain copy), the E pass with ADE 181 at 5.05 TB/s. us per step with
// the scalar passes and now: 384^3 with ADE (media aligned to vectors; others
// take k_e_cell for the E half, see ade_by_cell) 1453, 1269; 301x287x263 with
// three coefficients 480, 390; 160x152x144 double 146, 134.
//
// A warp covers a patch of rows (blockDim.x vectors along z); when every cell
// of it lies in the bulk box (both differences, no CPML state) the warp takes
// the straight-line path, else curl_general.
#pragma once

#include "cell_update.cuh"

// Minimum resident 128-thread blocks per SM the passes are compiled for:
// float H, float E, float E with ADE or three coefficients, double H, double
// E, double E with ADE or three coefficients. Step kernels in us at 5/5/4,
// 4/4/4 and 5/4/3: 256^3 plain 287, 311, 301; 384^3 with ADE 1278, 1309, 1370;
// 301x287x263 with three coefficients (at 5, 4, 4 blocks) 441, 424, 409.
// Double at 5/5, 6/5, 6/4 and 5/4 (H/E): 144^3 plain 106.8, 109.0, 112.4,
// 109.9; 160x160x147 with ADE 237, 243, 217, 211.
#ifndef PFB_MINB_HV
#define PFB_MINB_HV 5
#endif
#ifndef PFB_MINB_EV
#define PFB_MINB_EV 5
#endif
#ifndef PFB_MINB_EVA
#define PFB_MINB_EVA 4
#endif
#ifndef PFB_MINB_HV64
#define PFB_MINB_HV64 5
#endif
#ifndef PFB_MINB_EV64
#define PFB_MINB_EV64 5
#endif
#ifndef PFB_MINB_EVA64
#define PFB_MINB_EVA64 4
#endif

namespace pfb {

constexpr int kVecThreads = 128;

template <typename T>
constexpr int kVec = 16 / (int)sizeof(T);

__device__ __forceinline__ void vld(const float* p, float (&o)[4]) {
  const float4 v = *reinterpret_cast<const float4*>(p);
  o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w;
}
__device__ __forceinline__ void vld(const double* p, double (&o)[2]) {
  const double2 v = *reinterpret_cast<const double2*>(p);
  o[0] = v.x; o[1] = v.y;
}
__device__ __forceinline__ void vst(float* p, const float* o) {
  *reinterpret_cast<float4*>(p) = make_float4(o[0], o[1], o[2], o[3]);
}
__device__ __forceinline__ void vst(double* p, const double* o) {
  *reinterpret_cast<double2*>(p) = make_double2(o[0], o[1]);
}
__device__ __forceinline__ void wld(const uint32_t* p, uint32_t (&o)[4]) {
  const uint4 v = *reinterpret_cast<const uint4*>(p);
  o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w;
}
__device__ __forceinline__ void wld(const uint32_t* p, uint32_t (&o)[2]) {
  const uint2 v = *reinterpret_cast<const uint2*>(p);
  o[0] = v.x; o[1] = v.y;
}
// The vector at p when ok, else zeros.
template <typename T>
__device__ __forceinline__ void vld_if(const T* p, bool ok, T (&o)[kVec<T>]) {
  if (ok) {
    vld(p, o);
  } else {
#pragma unroll
    for (int q = 0; q < kVec<T>; ++q) o[q] = T(0);
  }
}

// Difference term t of a curl: components of the source field and axes in
// the order x A, x B, y A, y B, z A, z B (A enters with +, B with -).
__device__ __forceinline__ constexpr int term_comp(int t) {
  return t == 0 || t == 3 ? 2 : (t == 1 || t == 4 ? 1 : 0);
}
__device__ __forceinline__ constexpr int term_axis(int t) {
  return t == 0 || t == 5 ? 1 : (t == 1 || t == 2 ? 2 : 0);
}

// *bad = 1 when the reciprocal division by d (r = RN(1/d)) misses the IEEE
// quotient of some float significand.
static __global__ void k_recip_exact(float d, float r, int* bad) {
  for (unsigned m = blockIdx.x * blockDim.x + threadIdx.x; m < 1u << 23;
       m += gridDim.x * blockDim.x) {
    const float a = __uint_as_float(0x3f800000u | m);
    if (qscaled(a, d, r) != __fdiv_rn(a, d)) *bad = 1;
  }
}

// Whether a vector's differences n(term, cell) may take the reciprocal path;
// range: over all of them. WIDE: a float grid with divisors outside [2^-30,
// 2^-23] m, whose limits are its own (above 119 nm small numerators give
// subnormal quotients, so there is a lower one too). It has its own kernels:
// limits read at run time and a skipped loop cost the others 1%. The
// scalar passes divide such grids by IEEE division; 24 of these bound a
// vector's step. us at 200 nm, IEEE in line by the scalar passes, out of line by
// the vector passes, and so: 192^3 float 179, 184, 123, with ADE 221, 239, 175;
// 144^3 double 120, 168, 109.
template <bool WIDE, typename T, bool SCALED, typename N>
__device__ __forceinline__ bool in_range(const StepArgs<T>& a, const QCheck<T, SCALED>& range,
                                         const N& n) {
  constexpr int V = kVec<T>;
  if constexpr (sizeof(T) == 4) {
    bool fast = a.fdvec && range.ok();
    if (WIDE && fast && a.qlow) {
      unsigned low = ~0u;
#pragma unroll
      for (int t = 0; t < 6; ++t)
#pragma unroll
        for (int q = 0; q < V; ++q) low = min(low, range.lowkey(n(t, q)));
      fast = low >= a.qlow;
    }
    return fast;
  } else {
    if (!a.fdvec) return false;
    bool fast = range.ok();
    if (!fast) {
      fast = true;
#pragma unroll
      for (int t = 0; t < 6; ++t)
#pragma unroll
        for (int q = 0; q < V; ++q) fast = fast && range.sure(n(t, q));
    }
    return fast;
  }
}

// out[c] = f[c] + K[c] (d_A - d_B) for V bulk cells. SGN 1: forward
// differences d = (nb - own) / dl (H), -1: backward d = (own - nb) / dl (E).
// Own values are prescaled once; a prescaled difference is then one FMA, and
// the curl is scaled back once per component (QScale in common.cuh): 6.5
// operations per term instead of 11. One range check covers the V cells.
template <typename T, int SGN, int NC, bool WIDE>
__device__ __forceinline__ void curl_bulk(const StepArgs<T>& a, const T (&f)[3][kVec<T>],
                                          const T (&K)[NC][kVec<T>], const T (&own)[3][kVec<T>],
                                          const T (&nb)[6][kVec<T>], T (&out)[3][kVec<T>]) {
  constexpr int V = kVec<T>;
  const T dl[3] = {a.dx, a.dy, a.dz};
  const T rl[3] = {a.rdx, a.rdy, a.rdz};
  const T up = QScale<T>::up;
  QCheck<T, true> range(WIDE ? a.qtop : T(0x1p90));
  auto diff = [&](int t, int q) {
    const T os = mul_rn(own[term_comp(t)][q], up);
    return SGN > 0 ? fma_rn(nb[t][q], up, -os) : fma_rn(-nb[t][q], up, os);
  };
#pragma unroll
  for (int q = 0; q < V; ++q) {
    T n[6];
#pragma unroll
    for (int t = 0; t < 6; ++t) {
      n[t] = diff(t, q);
      range.take(n[t]);
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const T dA = qscaled(n[2 * c], dl[term_axis(2 * c)], rl[term_axis(2 * c)]);
      const T dB = qscaled(n[2 * c + 1], dl[term_axis(2 * c + 1)], rl[term_axis(2 * c + 1)]);
      out[c][q] = add_rn(f[c][q], mul_rn(mul_rn(sub_rn(dA, dB), QScale<T>::down), K[c % NC][q]));
    }
  }
  if (!in_range<WIDE>(a, range, diff)) {
#pragma unroll
    for (int q = 0; q < V; ++q) {
      T d[6];
#pragma unroll
      for (int t = 0; t < 6; ++t) {
        const T o = own[term_comp(t)][q];
        d[t] = div_cold(SGN > 0 ? sub_rn(nb[t][q], o) : sub_rn(o, nb[t][q]), dl[term_axis(t)]);
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) out[c][q] = bulk(f[c][q], K[c % NC][q], d[2 * c], d[2 * c + 1]);
    }
  }
}

// CPML tables of one field family as curl_general reads them.
template <typename T>
struct Cpml {
  const int* map[2];  // x, y
  const int* gz;      // per vector of a row: its group of V z-layer entries, or -1
  const int* np;
  const T* b[3];
  const T* c[3];
  const T* in[6];
  T* out[6];
};

// One CPML term of one cell: psi' = b psi + c d, and its share of the update.
template <typename T>
__device__ __forceinline__ T cpml_term(T f, T k, T d, T b, T c, T& psi) {
  psi = add_rn(mul_rn(b, psi), mul_rn(c, d));
  return add_rn(f, mul_rn(k, psi));
}

// The curl update of V cells anywhere in a 3D grid: components outside the
// reference's loop extents keep their value (and row padding stays zero),
// psi state is touched only in the layers. psi rows of the x and y layers have
// the fields' pitch, those of the z layers whole groups of V entries, so all
// of it is loaded as vectors, and all before the first use: cell by cell,
// each psi load waited behind the stores of the cell before it (256^3 with a
// 12-cell layer on every face: the layers cost 70 us of 314, now 41 of 287; 29
// of these are their bytes).
template <typename T, int SGN, int NC, bool WIDE>
__device__ __forceinline__ void curl_general(const StepArgs<T>& a, const Cpml<T>& p, int i, int j,
                                             int k, const T (&f)[3][kVec<T>],
                                             const T (&K)[NC][kVec<T>],
                                             const T (&own)[3][kVec<T>],
                                             const T (&nb)[6][kVec<T>], T (&out)[3][kVec<T>]) {
  constexpr int V = kVec<T>;
  const bool okx = SGN > 0 ? i < a.nx - 1 : i >= 1;
  const bool oky = SGN > 0 ? j < a.ny - 1 : j >= 1;
  const int mx = p.map[0][i], my = p.map[1][j], gz = p.gz[k / V];
  const T by = p.b[1][j], cy = p.c[1][j], bx = p.b[0][i], cx = p.c[0][i];
  const long long qy = ((long long)i * p.np[1] + my) * a.pz + k;
  const long long qx = ((long long)mx * a.ny + j) * a.pz + k;
  const long long qz = ((long long)i * a.ny + j) * p.np[2] + (long long)gz * V;
  T y0[V], y5[V], x3[V], x4[V], z1[V], z2[V], bz[V], cz[V];
  vld_if(p.in[0] + qy, my >= 0, y0);
  vld_if(p.in[5] + qy, my >= 0, y5);
  vld_if(p.in[3] + qx, mx >= 0, x3);
  vld_if(p.in[4] + qx, mx >= 0, x4);
  vld_if(p.in[1] + qz, gz >= 0, z1);
  vld_if(p.in[2] + qz, gz >= 0, z2);
  vld_if(p.b[2] + k, gz >= 0, bz);
  vld_if(p.c[2] + k, gz >= 0, cz);
  const T dl[3] = {a.dx, a.dy, a.dz};
  const T rl[3] = {a.rdx, a.rdy, a.rdz};
  T d[6][V];
  QCheck<T, false> range(WIDE ? a.qtop : T(0x1p90));
#pragma unroll
  for (int q = 0; q < V; ++q)
#pragma unroll
    for (int t = 0; t < 6; ++t) {
      const T o = own[term_comp(t)][q];
      d[t][q] = SGN > 0 ? sub_rn(nb[t][q], o) : sub_rn(o, nb[t][q]);
      range.take(d[t][q]);
    }
  if (in_range<WIDE>(a, range, [&](int t, int q) { return d[t][q]; })) {
#pragma unroll
    for (int q = 0; q < V; ++q)
#pragma unroll
      for (int t = 0; t < 6; ++t) d[t][q] = qdiv_fast(d[t][q], dl[term_axis(t)], rl[term_axis(t)]);
  } else {
#pragma unroll
    for (int q = 0; q < V; ++q)
#pragma unroll
      for (int t = 0; t < 6; ++t) d[t][q] = div_cold(d[t][q], dl[term_axis(t)]);
  }
#pragma unroll
  for (int q = 0; q < V; ++q) {
    const int kk = k + q;
    const bool okz = SGN > 0 ? kk < a.nz - 1 : (kk >= 1 && kk < a.nz);
    const bool inz = cz[q] != T(0);
    const T k0 = K[0][q], k1 = K[1 % NC][q], k2 = K[2 % NC][q];
    T r0 = f[0][q], r1 = f[1][q], r2 = f[2][q];
    if (oky && okz) {
      r0 = bulk(r0, k0, d[0][q], d[1][q]);
      if (my >= 0) r0 = cpml_term(r0, k0, d[0][q], by, cy, y0[q]);
      if (inz) r0 = cpml_term(r0, -k0, d[1][q], bz[q], cz[q], z1[q]);
    }
    if (okz && okx) {
      r1 = bulk(r1, k1, d[2][q], d[3][q]);
      if (inz) r1 = cpml_term(r1, k1, d[2][q], bz[q], cz[q], z2[q]);
      if (mx >= 0) r1 = cpml_term(r1, -k1, d[3][q], bx, cx, x3[q]);
    }
    if (okx && oky) {
      r2 = bulk(r2, k2, d[4][q], d[5][q]);
      if (mx >= 0) r2 = cpml_term(r2, k2, d[4][q], bx, cx, x4[q]);
      if (my >= 0) r2 = cpml_term(r2, -k2, d[5][q], by, cy, y5[q]);
    }
    out[0][q] = r0;
    out[1][q] = r1;
    out[2][q] = r2;
  }
  if (my >= 0) {
    vst(p.out[0] + qy, y0);
    vst(p.out[5] + qy, y5);
  }
  if (mx >= 0) {
    vst(p.out[3] + qx, x3);
    vst(p.out[4] + qx, x4);
  }
  if (gz >= 0) {
    vst(p.out[1] + qz, z1);
    vst(p.out[2] + qz, z2);
  }
}

// Whether every cell of the warp's patch lies in the bulk box [b0, b1).
template <int V>
__device__ __forceinline__ bool warp_bulk(bool live, int i, int j, int k, const int* b0,
                                          const int* b1) {
  const bool in = live && i >= b0[0] && i < b1[0] && j >= b0[1] && j < b1[1] && k >= b0[2] &&
                  k + V <= b1[2];
  return __all_sync(0xffffffffu, in);
}

// H pass: H^{n+1/2} = H^{n-1/2} - ch (curl E^n + psi), planes i0 + blockIdx.z.
template <typename T, bool WIDE>
__global__ void __launch_bounds__(kVecThreads, sizeof(T) == 4 ? PFB_MINB_HV : PFB_MINB_HV64)
    k_h_vec(const __grid_constant__ StepArgs<T> a, int i0) {
  pdl_enter();
  constexpr int V = kVec<T>;
  const int k = (blockIdx.x * blockDim.x + threadIdx.x) * V;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  const int i = i0 + blockIdx.z;
  const bool live = k < a.nz && j < a.ny;
  const bool box = warp_bulk<V>(live, i, j, k, a.hb0, a.hb1);
  if (!live) return;
  const long long sx = (long long)a.ny * a.pz;
  const long long id = i * sx + (unsigned)(j * a.pz + k);
  T own[3][V], nb[6][V], f[3][V], out[3][V];
  const bool hx = i + 1 < a.nx, hy = j + 1 < a.ny, hz = k + V < a.nz;
  vld(a.Ein[0] + id, own[0]);
  vld(a.Ein[1] + id, own[1]);
  vld(a.Ein[2] + id, own[2]);
  const T e1 = hz ? a.Ein[1][id + V] : T(0), e0 = hz ? a.Ein[0][id + V] : T(0);
  vld_if(a.Ein[2] + id + a.pz, hy, nb[0]);
  vld_if(a.Ein[0] + id + a.pz, hy, nb[5]);
  vld_if(a.Ein[2] + id + sx, hx, nb[3]);
  vld_if(a.Ein[1] + id + sx, hx, nb[4]);
#pragma unroll
  for (int c = 0; c < 3; ++c) vld(a.Hin[c] + id, f[c]);
#pragma unroll
  for (int q = 0; q < V; ++q) {
    nb[1][q] = q + 1 < V ? own[1][q + 1 < V ? q + 1 : 0] : e1;
    nb[2][q] = q + 1 < V ? own[0][q + 1 < V ? q + 1 : 0] : e0;
  }
  T K[1][V];
#pragma unroll
  for (int q = 0; q < V; ++q) K[0][q] = -a.ch;
  if (box) {
    curl_bulk<T, 1, 1, WIDE>(a, f, K, own, nb, out);
  } else {
    Cpml<T> p;
#pragma unroll
    for (int x = 0; x < 3; ++x) {
      if (x < 2) p.map[x] = a.maph[x];
      p.b[x] = a.bh[x];
      p.c[x] = a.cph[x];
    }
    p.np = a.nph;
    p.gz = a.gzh;
#pragma unroll
    for (int t = 0; t < 6; ++t) {
      p.in[t] = a.psiHin[t];
      p.out[t] = a.psiHout[t];
    }
    curl_general<T, 1, 1, WIDE>(a, p, i, j, k, f, K, own, nb, out);
  }
#pragma unroll
  for (int c = 0; c < 3; ++c) vst(a.Hout[c] + id, out[c]);
}

// ---- dispersive cells (simulation.py:645-669), V at a time -------------------
// V cells of one medium with consecutive ranks own 3 V NP consecutive reals
// per level ([cell][pole][component]): NP chunks of three vectors, of V / NP
// cells each. The first chunk of both levels is loaded ahead (c0: P^n, p0:
// P^{n-1}). The operations of each cell are ade_np's.
template <typename T, int NP>
__device__ __forceinline__ void ade_vec(const MediumT<T>& M, const T* Rc, T* Rp,
                                        const T (&en)[3][kVec<T>], T (&e)[3][kVec<T>],
                                        T (&c0)[3][kVec<T>], T (&p0)[3][kVec<T>]) {
  constexpr int V = kVec<T>;
#pragma unroll
  for (int ch = 0; ch < NP; ++ch) {
    if (ch > 0) {
#pragma unroll
      for (int u = 0; u < 3; ++u) {
        vld(Rc + (ch * 3 + u) * V, c0[u]);
        vld(Rp + (ch * 3 + u) * V, p0[u]);
      }
    }
#pragma unroll
    for (int s = 0; s < V / NP; ++s) {
      const int q = ch * (V / NP) + s;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        T delta = T(0);
#pragma unroll
        for (int p = 0; p < NP; ++p) {
          const int x = (s * NP + p) * 3 + c;
          const T pc = c0[x / V][x % V];
          const T pn = add_rn(add_rn(mul_rn(M.a[p], pc), mul_rn(M.b[p], p0[x / V][x % V])),
                              mul_rn(M.c[p], en[c][q]));
          p0[x / V][x % V] = pn;
          const T inc = sub_rn(pn, pc);
          delta = p == 0 ? inc : add_rn(delta, inc);
        }
        e[c][q] = sub_rn(e[c][q], mul_rn(M.inv, delta));
      }
    }
#pragma unroll
    for (int u = 0; u < 3; ++u) vst(Rp + (ch * 3 + u) * V, p0[u]);
  }
}

// Whether a vector of words takes k_e_vec's vector path for its records; their
// pole count and place (reals from the level's start).
template <typename T>
__device__ __forceinline__ bool ade_run(const MediumT<T>* media, const uint32_t (&t)[kVec<T>],
                                        int& np, long long& rec) {
  bool run = (t[0] & kDispersiveBit) && (t[kVec<T> - 1] >> kMediumShift) == (t[0] >> kMediumShift);
#pragma unroll
  for (int q = 1; q < kVec<T>; ++q) run = run && t[q] == t[0] + (uint32_t)q;
  if (!run) return false;
  const MediumT<T>& M = media[(t[0] >> kMediumShift) & 15u];
  np = M.npole;
  rec = M.poff + (long long)(t[0] & kLocMask) * (3 * np);
  return (np == 1 || np == 2) && rec % kVec<T> == 0;
}

// Warps of k_e_vec's grid, and those with aligned runs of one pole, of two, with
// other one-pole records, with other records of more poles.
template <typename T>
__global__ void __launch_bounds__(kVecThreads) k_ade_runs(const uint32_t* word,
                                                          const MediumT<T>* media, int ny, int nz,
                                                          int pz, unsigned long long* count) {
  constexpr int V = kVec<T>;
  const int k = (blockIdx.x * blockDim.x + threadIdx.x) * V;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  __shared__ unsigned n[5];
  const int tid = threadIdx.y * blockDim.x + threadIdx.x;
  if (tid < 5) n[tid] = 0u;
  __syncthreads();
  bool has[5] = {k < nz && j < ny, false, false, false, false};
  if (has[0]) {
    uint32_t t[V];
    wld(word + ((long long)blockIdx.z * ny + j) * pz + k, t);
    int np = 0;
    long long rec = 0;
    if (ade_run<T>(media, t, np, rec)) {
      has[1] = np == 1;
      has[2] = np == 2;
    } else {
#pragma unroll
      for (int q = 0; q < V; ++q)
        if (t[q] & kDispersiveBit) {
          const int p = media[(t[q] >> kMediumShift) & 15u].npole;
          has[3] = has[3] || p == 1;
          has[4] = has[4] || p > 1;
        }
    }
  }
#pragma unroll
  for (int q = 0; q < 5; ++q)
    if (__ballot_sync(0xffffffffu, has[q]) && (tid & 31) == 0) atomicAdd(&n[q], 1u);
  __syncthreads();
  if (tid < 5 && n[tid]) atomicAdd(&count[tid], (unsigned long long)n[tid]);
}

// One dispersive cell, any pole count, state read and written in place.
template <typename T>
__device__ __forceinline__ void ade_cell(const StepArgs<T>& a, uint32_t w, T en0, T en1, T en2,
                                         T& e0, T& e1, T& e2) {
  const MediumT<T>& M = a.media[(w >> kMediumShift) & 15u];
  const int np = M.npole;
  if (np == 0) return;
  const T* Rc = a.P + M.poff + (long long)(w & kLocMask) * (3 * np) + a.lvl * a.plev;
  T* Rp = a.P + M.poff + (long long)(w & kLocMask) * (3 * np) + (a.lvl ^ 1) * a.plev;
  T d0 = T(0), d1 = T(0), d2 = T(0);
  for (int p = 0; p < np; ++p) {
    const T A = M.a[p], B = M.b[p], C = M.c[p];
    const T c0 = Rc[3 * p], c1 = Rc[3 * p + 1], c2 = Rc[3 * p + 2];
    const T n0 = add_rn(add_rn(mul_rn(A, c0), mul_rn(B, Rp[3 * p])), mul_rn(C, en0));
    const T n1 = add_rn(add_rn(mul_rn(A, c1), mul_rn(B, Rp[3 * p + 1])), mul_rn(C, en1));
    const T n2 = add_rn(add_rn(mul_rn(A, c2), mul_rn(B, Rp[3 * p + 2])), mul_rn(C, en2));
    Rp[3 * p] = n0;
    Rp[3 * p + 1] = n1;
    Rp[3 * p + 2] = n2;
    const T i0 = sub_rn(n0, c0), i1 = sub_rn(n1, c1), i2 = sub_rn(n2, c2);
    d0 = p == 0 ? i0 : add_rn(d0, i0);
    d1 = p == 0 ? i1 : add_rn(d1, i1);
    d2 = p == 0 ? i2 : add_rn(d2, i2);
  }
  e0 = sub_rn(e0, mul_rn(M.inv, d0));
  e1 = sub_rn(e1, mul_rn(M.inv, d1));
  e2 = sub_rn(e2, mul_rn(M.inv, d2));
}

// E pass: E^{n+1} = E^n + ce (curl H^{n+1/2} + psi), then ADE. Loads are
// issued in dependency order: the words, every field vector, then what the
// words select (coefficients, ADE records of a run).
template <typename T, int CE, bool ADE>
constexpr int kMinBlocksE = ADE || CE == kCeCell3 ? (sizeof(T) == 4 ? PFB_MINB_EVA : PFB_MINB_EVA64)
                                                  : (sizeof(T) == 4 ? PFB_MINB_EV : PFB_MINB_EV64);
template <typename T, int CE, bool ADE, bool WIDE>
__global__ void __launch_bounds__(kVecThreads, kMinBlocksE<T, CE, ADE>)
    k_e_vec(const __grid_constant__ StepArgs<T> a, int i0) {
  pdl_enter();
  constexpr int V = kVec<T>;
  constexpr int NC = CE == kCeCell3 ? 3 : 1;
  const int k = (blockIdx.x * blockDim.x + threadIdx.x) * V;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  const int i = i0 + blockIdx.z;
  const bool live = k < a.nz && j < a.ny;
  const bool box = warp_bulk<V>(live, i, j, k, a.eb0, a.eb1);
  if (!live) return;
  const long long sx = (long long)a.ny * a.pz;
  const long long id = i * sx + (unsigned)(j * a.pz + k);
  uint32_t t[V];
  T K[NC][V];
  if (CE == kCeTable) wld(a.word + id, t);
  else if (ADE) wld(a.adeword + id, t);
  if (CE != kCeTable) {
#pragma unroll
    for (int c = 0; c < NC; ++c) vld(a.ce[c] + id, K[c]);
  }
  T own[3][V], nb[6][V], en[3][V], e[3][V];
  const bool lx = i > 0, ly = j > 0, lz = k > 0;
#pragma unroll
  for (int c = 0; c < 3; ++c) vld(a.Hin[c] + id, own[c]);
  const T h1 = lz ? a.Hin[1][id - 1] : T(0), h0 = lz ? a.Hin[0][id - 1] : T(0);
  vld_if(a.Hin[2] + id - a.pz, ly, nb[0]);
  vld_if(a.Hin[0] + id - a.pz, ly, nb[5]);
  vld_if(a.Hin[2] + id - sx, lx, nb[3]);
  vld_if(a.Hin[1] + id - sx, lx, nb[4]);
#pragma unroll
  for (int c = 0; c < 3; ++c) vld(a.Ein[c] + id, en[c]);
  // a run: V plain cells of one table entry, or V cells of one dispersive
  // medium with consecutive ranks
  bool vec = false;
  T c0[3][V], p0[3][V];
  const T* Rc = nullptr;
  T* Rp = nullptr;
  int np = 0;
  if (CE == kCeTable || ADE) {
    const bool disp = ADE && (t[0] & kDispersiveBit);
    bool run = (t[V - 1] >> kMediumShift) == (t[0] >> kMediumShift);
#pragma unroll
    for (int q = 1; q < V; ++q) run = run && t[q] == t[0] + (disp ? (uint32_t)q : 0u);
    if (ADE && disp && run) {
      const MediumT<T>& M = a.media[(t[0] >> kMediumShift) & 15u];
      np = M.npole;
      const long long rec = M.poff + (long long)(t[0] & kLocMask) * (3 * np);
      vec = (np == 1 || np == 2) && rec % V == 0;
      if (vec) {
        Rc = a.P + rec + a.lvl * a.plev;
        Rp = a.P + rec + (a.lvl ^ 1) * a.plev;
#pragma unroll
        for (int u = 0; u < 3; ++u) {
          vld(Rc + u * V, c0[u]);
          vld(Rp + u * V, p0[u]);
        }
      }
    }
    if (CE == kCeTable) {
      if (run) {
        const T K0 = disp ? a.media[(t[0] >> kMediumShift) & 15u].ce : a.table[t[0]];
#pragma unroll
        for (int q = 0; q < V; ++q) K[0][q] = K0;
      } else {
#pragma unroll
        for (int q = 0; q < V; ++q)
          K[0][q] = ADE && (t[q] & kDispersiveBit) ? a.media[(t[q] >> kMediumShift) & 15u].ce
                                                   : a.table[t[q]];
      }
    }
  }
#pragma unroll
  for (int q = 0; q < V; ++q) {
    nb[1][q] = q > 0 ? own[1][q > 0 ? q - 1 : 0] : h1;
    nb[2][q] = q > 0 ? own[0][q > 0 ? q - 1 : 0] : h0;
  }
  if (box) {
    curl_bulk<T, -1, NC, WIDE>(a, en, K, own, nb, e);
  } else {
    Cpml<T> p;
#pragma unroll
    for (int x = 0; x < 3; ++x) {
      if (x < 2) p.map[x] = a.mape[x];
      p.b[x] = a.be[x];
      p.c[x] = a.cpe[x];
    }
    p.np = a.npe;
    p.gz = a.gze;
#pragma unroll
    for (int s = 0; s < 6; ++s) {
      p.in[s] = a.psiEin[s];
      p.out[s] = a.psiE[s];
    }
    curl_general<T, -1, NC, WIDE>(a, p, i, j, k, en, K, own, nb, e);
  }
  if (ADE) {
    if (vec) {
      const MediumT<T>& M = a.media[(t[0] >> kMediumShift) & 15u];
      if (np == 1) ade_vec<T, 1>(M, Rc, Rp, en, e, c0, p0);
      else ade_vec<T, 2>(M, Rc, Rp, en, e, c0, p0);
    } else {
#pragma unroll
      for (int q = 0; q < V; ++q)
        if (t[q] & kDispersiveBit)
          ade_cell<T>(a, t[q], en[0][q], en[1][q], en[2][q], e[0][q], e[1][q], e[2][q]);
    }
  }
#pragma unroll
  for (int c = 0; c < 3; ++c) vst(a.Eout[c] + id, e[c]);
}

}  // namespace pfb
