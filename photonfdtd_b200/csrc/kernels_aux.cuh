// kernels_aux.cuh - soft-source injection and the DFT / flux monitor kernels.
#pragma once

#include "common.cuh"

namespace pfb {

// ---------------------------------------------------------------------------
// Soft sources (simulation.py:1367-1390). Sources sharing a (component, cell)
// form one group; a group's sources are applied in the reference's list order,
// each as a double add rounded to the field type, so coincident dipoles round
// exactly as the reference's successive `F[i,j,k] += val` do.
// ---------------------------------------------------------------------------
template <typename T>
__global__ void k_inject(SourceGroups s, T* f0, T* f1, T* f2, long long step) {
  pdl_enter();
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= s.n_groups) return;
  T* F = s.comp[g] == 0 ? f0 : (s.comp[g] == 1 ? f1 : f2);
  const long long c = s.cell[g];
  T v = F[c];
  for (int q = s.start[g]; q < s.start[g + 1]; ++q)
    v = add_double<T>(v, __dmul_rn(s.amp[q], s.wave[(long long)s.wave_row[q] * s.n_steps + step]));
  F[c] = v;
}

// ---------------------------------------------------------------------------
// DFT monitor (simulation.py:1116-1133). Each sampled step writes the region's
// values into a ring of pending samples; a flush folds the pending samples,
// oldest first, into the complex128 accumulators:
//   acc += (phase * f) * dt   per frequency, per cell
// with the same two roundings per real and imaginary part as numpy's
// complex128 * float32 -> complex128 product followed by * dt. Summation order
// over steps is the reference's, so the accumulators match bit for bit.
// ---------------------------------------------------------------------------
// The six field components of one time level, by component code.
template <typename T>
struct Fields6 {
  const T* f[6];
};

// Samples cell `cell` of a region into its ring slot.
template <typename T>
__device__ __forceinline__ void dft_sample_cell(const DftRegion& r, T* ring, int slot,
                                                const Fields6<T>& fields, long long cell, int ny,
                                                int pz) {
  const long long ck = cell % r.count[2];
  const long long rest = cell / r.count[2];
  const long long cj = rest % r.count[1];
  const long long ci = rest / r.count[1];
  const long long id = ((long long)(r.start[0] + ci * r.stride[0]) * ny +
                        (r.start[1] + cj * r.stride[1])) * pz +
                       (r.start[2] + ck * r.stride[2]);
  for (int q = 0; q < r.ncomp; ++q)
    ring[((long long)slot * r.ncomp + q) * r.ncell + cell] = fields.f[r.comps[q]][id];
}

template <typename T>
__global__ void k_dft_sample(DftRegion r, T* ring, int slot, Fields6<T> fields, int ny,
                             int pz) {
  pdl_enter();
  const long long cell = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (cell < r.ncell) dft_sample_cell<T>(r, ring, slot, fields, cell, ny, pz);
}

template <typename T>
__global__ void k_dft_flush(DftRegion r, const T* ring, int n_pending, double* acc,
                            const double* ph_e, const double* ph_h, long long q0, int n_freq,
                            double dt) {
  pdl_enter();
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= r.ncell * r.ncomp) return;
  const long long cell = t % r.ncell;
  const int qc = (int)(t / r.ncell);
  const double* ph = r.comps[qc] < 3 ? ph_e : ph_h;
  constexpr int F = 8;
  for (int f0 = 0; f0 < n_freq; f0 += F) {
    double re[F], im[F];
    const int nf = min(F, n_freq - f0);
#pragma unroll
    for (int f = 0; f < F; ++f) {
      if (f < nf) {
        const long long o = (((long long)qc * n_freq + f0 + f) * r.ncell + cell) * 2;
        re[f] = acc[o];
        im[f] = acc[o + 1];
      }
    }
    for (int q = 0; q < n_pending; ++q) {
      const double s = (double)ring[((long long)q * r.ncomp + qc) * r.ncell + cell];
      const double* row = ph + ((q0 + q) * n_freq + f0) * 2;
#pragma unroll
      for (int f = 0; f < F; ++f) {
        if (f < nf) {
          re[f] = __dadd_rn(re[f], __dmul_rn(__dmul_rn(row[2 * f], s), dt));
          im[f] = __dadd_rn(im[f], __dmul_rn(__dmul_rn(row[2 * f + 1], s), dt));
        }
      }
    }
#pragma unroll
    for (int f = 0; f < F; ++f) {
      if (f < nf) {
        const long long o = (((long long)qc * n_freq + f0 + f) * r.ncell + cell) * 2;
        acc[o] = re[f];
        acc[o + 1] = im[f];
      }
    }
  }
}

// ---------------------------------------------------------------------------
// Flux monitor (simulation.py:1440-1459). Per step, S = E_t1*H_t2 - E_t2*H_t1
// in the field type at every cell of the plane (the same three roundings as
// the reference), summed in double per block; block partials go to a ring.
// The flush reduces each step's partials in a fixed order and accumulates
// flux += double(T(sum) * T(dA)) * dt, as the reference's float32 run does.
// ---------------------------------------------------------------------------
struct FluxPlane {
  int axis, idx;
  int n0, n1;  // plane extents (the two other axes, in order)
  int nblk;
};

// Sum over 256 consecutive threads (the block, or a 256-thread part of it
// with its own sh), the same tree whoever calls it.
template <typename T>
__device__ __forceinline__ double block_sum256(double v, double* sh) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  const int t = threadIdx.x & 255, lane = t & 31, wid = t >> 5;
  if (lane == 0) sh[wid] = v;
  __syncthreads();
  v = (t < 8) ? sh[t] : 0.0;
  if (wid == 0)
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}

// S = E_t1 H_t2 - E_t2 H_t1 at plane cell t (0 past the plane's end).
template <typename T>
__device__ __forceinline__ double flux_cell_value(const FluxPlane& p, long long t,
                                                  const Fields6<T>& fields, int ny, int pz) {
  if (t >= (long long)p.n0 * p.n1) return 0.0;
  const int u = (int)(t / p.n1), w = (int)(t % p.n1);
  long long id;
  int e1, h2, e2, h1;
  if (p.axis == 0) {  // S = Ey*Hz - Ez*Hy
    id = ((long long)p.idx * ny + u) * pz + w;
    e1 = 1; h2 = 5; e2 = 2; h1 = 4;
  } else if (p.axis == 1) {  // S = Ez*Hx - Ex*Hz
    id = ((long long)u * ny + p.idx) * pz + w;
    e1 = 2; h2 = 3; e2 = 0; h1 = 5;
  } else {  // S = Ex*Hy - Ey*Hx
    id = ((long long)u * ny + w) * pz + p.idx;
    e1 = 0; h2 = 4; e2 = 1; h1 = 3;
  }
  return (double)sub_rn(mul_rn(fields.f[e1][id], fields.f[h2][id]),
                        mul_rn(fields.f[e2][id], fields.f[h1][id]));
}

// Flux planes sampled by one launch (up to kFluxBatch): blockIdx.y picks
// the plane; block x of a plane sums S = E_t1 H_t2 - E_t2 H_t1 (rounded in
// the field type, simulation.py:1440-1459) over the plane's cells
// [256 x, 256 x + 256) in row-major (n0, n1) order with block_sum256, and
// stores the partial in the plane's ring slot; k_flux_flush folds the
// partials in block order. Blocks past a plane's own count return before
// any barrier, as a whole.
constexpr int kFluxBatch = 8;
struct FluxBatch {
  FluxPlane p[kFluxBatch];
  double* partial[kFluxBatch];
  int slot[kFluxBatch];
};

template <typename T>
__global__ void __launch_bounds__(256) k_flux_sample_batch(FluxBatch b, Fields6<T> fields, int ny,
                                                           int pz) {
  pdl_enter();
  __shared__ double sh[8];
  const FluxPlane& p = b.p[blockIdx.y];
  if ((int)blockIdx.x >= p.nblk) return;  // uniform over the block
  double v = flux_cell_value<T>(p, (long long)blockIdx.x * 256 + threadIdx.x, fields, ny, pz);
  v = block_sum256<T>(v, sh);
  if (threadIdx.x == 0) b.partial[blockIdx.y][(long long)b.slot[blockIdx.y] * p.nblk + blockIdx.x] = v;
}

// The pending samples of every flux plane of one launch (blockIdx.x picks the
// plane): four 256-thread groups sum the block partials of four samples at a
// time, then one thread folds the sums in step order. One group, one plane
// per launch, took about 0.8 us per sample in a serial chain of barriers.
constexpr int kFluxRing = 32;
struct FluxFold {
  const double* partial[kFluxBatch];
  int nblk[kFluxBatch], pending[kFluxBatch];
  double* acc[kFluxBatch];
  double dA[kFluxBatch], dt[kFluxBatch];
};
template <typename T>
__global__ void __launch_bounds__(1024) k_flux_flush(FluxFold f) {
  pdl_enter();
  __shared__ double sh[4][8];
  __shared__ double sum[kFluxRing];
  const int m = blockIdx.x, grp = threadIdx.x >> 8, t = threadIdx.x & 255;
  const int n = f.pending[m], nblk = f.nblk[m];
  for (int q0 = 0; q0 < n; q0 += 4) {
    const int q = q0 + grp;
    double v = 0.0;
    if (q < n)
      for (int b = t; b < nblk; b += 256) v += f.partial[m][(long long)q * nblk + b];
    v = block_sum256<T>(v, sh[grp]);
    if (q < n && t == 0) sum[q] = v;
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    double total = *f.acc[m];
    for (int q = 0; q < n; ++q) {
      const T sa = mul_rn(to_real(sum[q], T()), (T)f.dA[m]);
      total = __dadd_rn(total, __dmul_rn((double)sa, f.dt[m]));
    }
    *f.acc[m] = total;
  }
}

// Strided sub-block of one field into a compact C-order buffer (the
// FieldMonitor snapshot: every stride-th cell per axis, or one z plane).
template <typename T>
__global__ void k_gather_region(const T* f, int ny, int pz, int3 start, int3 stride,
                                int3 count, T* out) {
  const long long n = (long long)count.x * count.y * count.z;
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n;
       t += (long long)gridDim.x * blockDim.x) {
    const long long ck = t % count.z, rest = t / count.z;
    const long long cj = rest % count.y, ci = rest / count.y;
    out[t] = f[((long long)(start.x + ci * stride.x) * ny + (start.y + cj * stride.y)) * pz +
               (start.z + ck * stride.z)];
  }
}

// Rows of a padded array <-> a compact array: w entries of every p, the first
// ones or (pos) those at given places. Several arrays in one launch
// (blockIdx.y). Bound by memory: each lane moves four entries a warp apart, all
// loads before the stores, the row by a multiplication. A checkpoint of 160 x
// 160 x 147 float32 took 300 us with cudaMemcpy2DAsync per array, 88 so; 1100 x
// 1100 x 4 871, 66.
struct RowCopy {
  void* padded;
  void* compact;
  const int* pos;
  unsigned total;      // entries of the compact array, below 2^31
  unsigned w, p;
  unsigned m;          // n / w == (n m) >> sh for n < 2^31
  int sh;
};
constexpr int kRowCopies = 18;
struct RowCopies {
  RowCopy r[kRowCopies];
};
template <typename U>
__global__ void __launch_bounds__(256) k_copy_rows(const __grid_constant__ RowCopies c, bool get) {
  const RowCopy& r = c.r[blockIdx.y];
  U* pad = (U*)r.padded;
  U* dense = (U*)r.compact;
  const unsigned first = (blockIdx.x * 8 + (threadIdx.x >> 5)) * 128 + (threadIdx.x & 31);
  for (unsigned t = first; t < r.total; t += gridDim.x * 1024) {
    size_t at[4];
    U v[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const unsigned n = t + 32 * q;
      const unsigned row = (unsigned)(((uint64_t)n * r.m) >> r.sh), col = n - row * r.w;
      const bool ok = n < r.total;
      at[q] = (size_t)row * r.p + (r.pos && ok ? (unsigned)r.pos[col] : col);
      if (ok) v[q] = get ? pad[at[q]] : dense[n];
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const unsigned n = t + 32 * q;
      if (n >= r.total) continue;
      if (get) dense[n] = v[q];
      else pad[at[q]] = v[q];
    }
  }
}

// Non-finite scan over a field: sets *flag when any value is inf or nan.
template <typename T>
__global__ void k_nonfinite(const T* f, long long n, int* flag) {
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n;
       t += (long long)gridDim.x * blockDim.x)
    if (!isfinite(f[t])) {
      *flag = 1;
      return;
    }
}

}  // namespace pfb
