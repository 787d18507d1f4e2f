// kernels_adj_vec.cuh - the reverse step of 3D grids, one 16-byte vector of z cells per thread.
//
// The operations of kernels_adj.cuh in the same order on the layout of the
// vector passes (kernels_vec3d.cuh). One cell per thread, the E half read
// each component's operands behind the stores of the one before it (three
// chains of two memory latencies) and divided by the IEEE routine. Here a
// thread loads everything it needs for its cells first, as vectors (about 200
// registers: two blocks of 128 threads still keep 140 KB in flight per SM). us
// at 97 x 89 x 101, about 60% of the cells in layers, cold caches: E half 43 ->
// 28, H half 24 -> 18.
#pragma once

#include "kernels_adj.cuh"
#include "kernels_vec3d.cuh"

namespace pfb {

// The gather of component c's two quotient adjoints: term and axis.
__device__ __forceinline__ constexpr int gather_term(int c, int u) {
  return u == 0 ? (c == 0 ? 2 : (c == 1 ? 1 : 0)) : (c == 0 ? 5 : (c == 1 ? 4 : 3));
}

// psi-like state of the six terms of one family: where the cell's vector lies
// (x and y layers on the fields' pitch, z layers in groups of V).
template <typename T>
struct LayerAt {
  int mx, my, gz;
  long long q[3];  // element of the vector per axis
  T b[2], c[2];    // x, y
  T bz[kVec<T>], cz[kVec<T>];
};
template <typename T>
__device__ __forceinline__ void layer_at(const int* const map[3], const int* gz, const int* np,
                                         const T* const b[3], const T* const c[3], int i, int j,
                                         int k, int ny, int pz, LayerAt<T>& l) {
  l.mx = map[0][i];
  l.my = map[1][j];
  l.gz = gz[k / kVec<T>];
  l.b[0] = b[0][i];
  l.c[0] = c[0][i];
  l.b[1] = b[1][j];
  l.c[1] = c[1][j];
  l.q[0] = ((long long)l.mx * ny + j) * pz + k;
  l.q[1] = ((long long)i * np[1] + l.my) * pz + k;
  l.q[2] = ((long long)i * ny + j) * np[2] + (long long)l.gz * kVec<T>;
  vld_if(b[2] + k, l.gz >= 0, l.bz);
  vld_if(c[2] + k, l.gz >= 0, l.cz);
}
template <typename T>
__device__ __forceinline__ bool in_layer(const LayerAt<T>& l, int axis) {
  return axis == 0 ? l.mx >= 0 : (axis == 1 ? l.my >= 0 : l.gz >= 0);
}
template <typename T>
__device__ __forceinline__ void layer_coef(const LayerAt<T>& l, int axis, int q, bool& in, T& b,
                                           T& c) {
  b = axis == 2 ? l.bz[q] : l.b[axis];
  c = axis == 2 ? l.cz[q] : l.c[axis];
  in = axis == 2 ? c != T(0) : in_layer(l, axis);
}

// One component's transpose (curl_transpose): quotient adjoints and psi
// adjoints of terms 2c and 2c + 1.
template <typename T>
__device__ __forceinline__ void transpose_cell(const LayerAt<T>& l, int c, int q, T x, T K, T& qa,
                                               T& qb, T& la, T& lb) {
  bool in;
  T b, cc;
  qa = mul_rn(K, x);
  qb = mul_rn(-K, x);
  layer_coef(l, term_axis(2 * c), q, in, b, cc);
  if (in) {
    const T ap = fma_rn(K, x, la);
    qa = fma_rn(cc, ap, qa);
    la = mul_rn(b, ap);
  }
  layer_coef(l, term_axis(2 * c + 1), q, in, b, cc);
  if (in) {
    const T ap = fma_rn(-K, x, lb);
    qb = fma_rn(cc, ap, qb);
    lb = mul_rn(b, ap);
  }
}

template <typename T, int CE>
__global__ void __launch_bounds__(kVecThreads, 2) k_adj_e_vec(const __grid_constant__ StepArgs<T> a,
                                                             const __grid_constant__ AdjState<T> s) {
  pdl_enter();
  constexpr int V = kVec<T>, NC = CE == kCeCell3 ? 3 : 1;
  const int k = (blockIdx.x * blockDim.x + threadIdx.x) * V;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  const int i = blockIdx.z;
  if (k >= a.nz || j >= a.ny) return;
  const long long sx = (long long)a.ny * a.pz;
  const long long id = i * sx + (unsigned)(j * a.pz + k);
  const bool lx = i > 0, ly = j > 0, lz = k > 0;
  T K[NC][V], x[3][V], g[6][V], lo[6][V], own[3][V], nb[6][V], pr[6][V], lp[6][V];
  double gr[NC][V];
  LayerAt<T> l;
  layer_at<T>(a.mape, a.gze, a.npe, a.be, a.cpe, i, j, k, a.ny, a.pz, l);
  if (CE == kCeTable) {
    uint32_t t[V];
    wld(a.word + id, t);
#pragma unroll
    for (int q = 0; q < V; ++q) K[0][q] = a.table[t[q] & ~kDispersiveBit];
  } else {
#pragma unroll
    for (int c = 0; c < NC; ++c) vld(a.ce[c] + id, K[c]);
  }
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    vld(s.lamE[c] + id, x[c]);
    vld(s.Hrec[c] + id, own[c]);
  }
#pragma unroll
  for (int t = 0; t < 6; ++t) {
    const int ax = term_axis(t);
    vld(s.gH[t] + id, g[t]);
    if (ax == 2) {
      const T h = lz ? s.gH[t][id - 1] : T(0);
      const T w = lz ? s.Hrec[term_comp(t)][id - 1] : T(0);
#pragma unroll
      for (int q = 0; q < V; ++q) {
        lo[t][q] = q > 0 ? g[t][q > 0 ? q - 1 : 0] : h;
        nb[t][q] = q > 0 ? own[term_comp(t)][q > 0 ? q - 1 : 0] : w;
      }
    } else {
      const long long d = ax == 1 ? (long long)a.pz : sx;
      const bool ok = ax == 1 ? ly : lx;
      vld_if(s.gH[t] + id - d, ok, lo[t]);
      vld_if(s.Hrec[term_comp(t)] + id - d, ok, nb[t]);
    }
    vld_if(s.psiErec[t] + l.q[ax], in_layer(l, ax), pr[t]);
    vld_if(s.lpE[t] + l.q[ax], in_layer(l, ax), lp[t]);
  }
#pragma unroll
  for (int c = 0; c < NC; ++c)
#pragma unroll
    for (int q = 0; q < V; q += 2) {
      const double2 v = *reinterpret_cast<const double2*>(s.grad + c * s.gstride + id + q);
      gr[c][q] = v.x;
      gr[c][q + 1] = v.y;
    }
  // the quotients of the recorded H
  const T dl[3] = {a.dx, a.dy, a.dz};
  const T rl[3] = {a.rdx, a.rdy, a.rdz};
  QCheck<T, false> range(a.qtop);
#pragma unroll
  for (int t = 0; t < 6; ++t)
#pragma unroll
    for (int q = 0; q < V; ++q) {
      nb[t][q] = sub_rn(own[term_comp(t)][q], nb[t][q]);
      range.take(nb[t][q]);
    }
  if (in_range<true>(a, range, [&](int t, int q) { return nb[t][q]; })) {
#pragma unroll
    for (int t = 0; t < 6; ++t)
#pragma unroll
      for (int q = 0; q < V; ++q) nb[t][q] = qdiv_fast(nb[t][q], dl[term_axis(t)], rl[term_axis(t)]);
  } else {
#pragma unroll
    for (int t = 0; t < 6; ++t)
#pragma unroll
      for (int q = 0; q < V; ++q) nb[t][q] = div_cold(nb[t][q], dl[term_axis(t)]);
  }
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const int tA = 2 * c, tB = 2 * c + 1, xA = term_axis(tA), xB = term_axis(tB);
    T qa[V], qb[V];
#pragma unroll
    for (int q = 0; q < V; ++q) {
      const int kk = k + q;
      const bool ok[3] = {lx, ly, kk >= 1 && kk < a.nz};
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int t = gather_term(c, u);
        x[c][q] = fma_rn(sub_rn(lo[t][q], g[t][q]), s.idl[term_axis(t)], x[c][q]);
      }
      if (kk >= a.nz) x[c][q] = T(0);  // row padding
      qa[q] = qb[q] = T(0);
      if (!(ok[xA] && ok[xB])) continue;
      T w = sub_rn(nb[tA][q], nb[tB][q]), b, cc;
      bool in;
      layer_coef(l, xA, q, in, b, cc);
      if (in) w = add_rn(w, pr[tA][q]);
      layer_coef(l, xB, q, in, b, cc);
      if (in) w = sub_rn(w, pr[tB][q]);
      const double gc = __dmul_rn((double)x[c][q], (double)w);
      if (gc != 0.0) gr[c % NC][q] = __dadd_rn(gr[c % NC][q], gc);
      transpose_cell<T>(l, c, q, x[c][q], K[c % NC][q], qa[q], qb[q], lp[tA][q], lp[tB][q]);
    }
    vst(s.gE[tA] + id, qa);
    vst(s.gE[tB] + id, qb);
    vst(s.lamE[c] + id, x[c]);
    if (in_layer(l, xA)) vst(s.lpE[tA] + l.q[xA], lp[tA]);
    if (in_layer(l, xB)) vst(s.lpE[tB] + l.q[xB], lp[tB]);
  }
#pragma unroll
  for (int c = 0; c < NC; ++c)
#pragma unroll
    for (int q = 0; q < V; q += 2)
      *reinterpret_cast<double2*>(s.grad + c * s.gstride + id + q) =
          make_double2(gr[c][q], gr[c][q + 1]);
}

template <typename T>
__global__ void __launch_bounds__(kVecThreads, 3) k_adj_h_vec(const __grid_constant__ StepArgs<T> a,
                                                             const __grid_constant__ AdjState<T> s) {
  pdl_enter();
  constexpr int V = kVec<T>;
  const int k = (blockIdx.x * blockDim.x + threadIdx.x) * V;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  const int i = blockIdx.z;
  if (k >= a.nz || j >= a.ny) return;
  const long long sx = (long long)a.ny * a.pz;
  const long long id = i * sx + (unsigned)(j * a.pz + k);
  const bool hx = i + 1 < a.nx, hy = j + 1 < a.ny, hz = k + V < a.nz;
  T y[3][V], g[6][V], hi[6][V], lp[6][V];
  LayerAt<T> l;
  layer_at<T>(a.maph, a.gzh, a.nph, a.bh, a.cph, i, j, k, a.ny, a.pz, l);
#pragma unroll
  for (int c = 0; c < 3; ++c) vld(s.lamH[c] + id, y[c]);
#pragma unroll
  for (int t = 0; t < 6; ++t) {
    const int ax = term_axis(t);
    vld(s.gE[t] + id, g[t]);
    if (ax == 2) {
      const T h = hz ? s.gE[t][id + V] : T(0);
#pragma unroll
      for (int q = 0; q < V; ++q)
        hi[t][q] = k + q + 1 < a.nz ? (q + 1 < V ? g[t][q + 1 < V ? q + 1 : 0] : h) : T(0);
    } else {
      const long long d = ax == 1 ? (long long)a.pz : sx;
      vld_if(s.gE[t] + id + d, ax == 1 ? hy : hx, hi[t]);
    }
    vld_if(s.lpH[t] + l.q[ax], in_layer(l, ax), lp[t]);
  }
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const int tA = 2 * c, tB = 2 * c + 1, xA = term_axis(tA), xB = term_axis(tB);
    T qa[V], qb[V];
#pragma unroll
    for (int q = 0; q < V; ++q) {
      const bool ok[3] = {hx, hy, k + q < a.nz - 1};
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int t = gather_term(c, u);
        y[c][q] = fma_rn(sub_rn(g[t][q], hi[t][q]), s.idl[term_axis(t)], y[c][q]);
      }
      qa[q] = qb[q] = T(0);
      if (ok[xA] && ok[xB])
        transpose_cell<T>(l, c, q, y[c][q], -a.ch, qa[q], qb[q], lp[tA][q], lp[tB][q]);
    }
    vst(s.gH[tA] + id, qa);
    vst(s.gH[tB] + id, qb);
    vst(s.lamH[c] + id, y[c]);
    if (in_layer(l, xA)) vst(s.lpH[tA] + l.q[xA], lp[tA]);
    if (in_layer(l, xB)) vst(s.lpH[tB] + l.q[xB], lp[tB]);
  }
}

}  // namespace pfb
