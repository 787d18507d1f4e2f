// kernels_resident.cuh - many time steps of a small grid in one launch.
//
// A grid of up to some 10^5 cells has one to five microseconds of work per
// pass, less than a kernel's launch and drain, and a step takes three to six
// launches (104 x 104 float64: 16 us per step, 331 x 217 dispersive with
// spectra: 26 us). This kernel keeps its blocks on the chip for a run of
// steps and separates the passes by barriers. Three forms:
//   kResCell1  one cell per thread, one cluster of up to 16 blocks (hardware
//              barrier)
//   kResGrid1  one cell per thread, a cooperative grid (a counter in L2)
//   kResGridN  several cells per thread, a cooperative grid
// With one cell per thread everything a cell owns - fields, CPML state and
// coefficients, its place in the monitors - stays in registers for the whole
// launch; a pass then costs a barrier, one round of neighbour loads and the
// arithmetic. All loads of a cell are issued before its first use: written
// component by component, each pass waited out nine L2 latencies.
//
// Every cell's operations are the scalar passes' in the same order, and
// monitors are sampled into the same ring slots, so the results equal the
// separate launches' bit for bit. Per step: H pass [H sources] | E pass
// [E sources, samples] | with a barrier at each bar. A flux plane's cells are
// kept as values per step and summed when the ring is flushed.
#pragma once

#include "kernels_aux.cuh"
#include "kernels_split.cuh"
#include "kernels_vec3d.cuh"

namespace pfb {

enum ResMode { kResCell1 = 0, kResGrid1 = 1, kResGridN = 2 };
// Threads per block and blocks per SM of each form. The one-cell forms need
// about 100 registers: at 64 (two blocks per SM, or 1024 threads) they spill,
// 331 x 217 float32 7.3 us per step against 5.1.
template <typename T>
__host__ __device__ constexpr int res_threads(int mode) {
  return mode == kResCell1 && sizeof(T) == 4 ? 768 : 512;
}
template <typename T>
__host__ __device__ constexpr int res_blocks(int mode) {
  return mode == kResGridN && sizeof(T) == 4 ? 2 : 1;
}
constexpr int kResDft = 4;        // DFT monitors one launch samples
constexpr int kResOwned = 32;     // source groups injected by their cells' threads
constexpr int kResSpin = 1 << 22; // polls before a grid barrier gives up (seconds)
constexpr int kResSpinTest = 1 << 12;  // with the test hook (milliseconds)

template <typename T>
struct ResidentArgs {
  StepArgs<T> a;            // in place: Ein == Eout, Hin == Hout
  SourceGroups src[2];      // E, H family; cell = padded index
  long long step0;
  int n;                    // steps of this launch
  int n_dft, n_flux;
  DftRegion dft[kResDft];
  T* dft_ring[kResDft];
  int dft_slot[kResDft];    // ring slot of the launch's first sample
  int dft_interval[kResDft];
  FluxPlane flux[kFluxBatch];
  T* flux_val[kFluxBatch];  // [slot][plane cell]
  int flux_slot[kFluxBatch];
  unsigned* bar;            // grid barrier: arrivals (zero at launch)
  // polls before a barrier gives up, arrivals counted as missing before the first
  // one. The test hook gives few polls and arrivals that never come; as data they
  // cost nothing (a test of the hook in the barrier cost 1 to 2% of a step).
  int spin;
  unsigned phase0;
  int* err;                 // set when a barrier gave up
};

// Barrier over the launch; false when the grid barrier gave up.
template <int MODE>
__device__ __forceinline__ bool res_barrier(unsigned* bar, unsigned& phase, int* err, int limit) {
  if (MODE == kResCell1) {
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
    return true;
  }
  __syncthreads();
  phase += gridDim.x;
  int bad = 0;
  if (threadIdx.x == 0) {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
    unsigned v;
    int spin = 0;
    do {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(bar) : "memory");
    } while (v < phase && ++spin < limit);
    if (v < phase) {
      *(volatile int*)err = 1;
      bad = 1;
    }
  }
  return !__syncthreads_or(bad);
}

// The sources of group g at this step.
template <typename T>
__device__ __forceinline__ void inject_group(const SourceGroups& s, int g, T* const F[3],
                                             long long step) {
  T* f = F[s.comp[g]];
  const long long c = s.cell[g];
  T v = f[c];
  for (int q = s.start[g]; q < s.start[g + 1]; ++q)
    v = add_double<T>(v, __dmul_rn(s.amp[q], s.wave[(long long)s.wave_row[q] * s.n_steps + step]));
  f[c] = v;
}

// What one field family's update of a cell takes from its position: the
// compact CPML index (-1: none) and coefficients per axis.
template <typename T>
struct CellPml {
  int m[3];
  T b[3], c[3];
};
template <typename T>
__device__ __forceinline__ void load_pml(const int* const map[3], const T* const b[3],
                                         const T* const c[3], const int pos[3], CellPml<T>& p) {
#pragma unroll
  for (int x = 0; x < 3; ++x) {
    p.m[x] = map[x][pos[x]];
    p.b[x] = b[x][pos[x]];
    p.c[x] = c[x][pos[x]];
  }
}
// Element of psi term t at the cell (its axis has m >= 0).
__device__ __forceinline__ long long psi_elem(int t, const int m[3], const int* np,
                                              const int pos[3], int ny, int pz) {
  const int x = term_axis(t);
  if (x == 0) return ((long long)m[0] * ny + pos[1]) * pz + pos[2];
  if (x == 1) return ((long long)pos[0] * np[1] + m[1]) * pz + pos[2];
  return ((long long)pos[0] * ny + pos[1]) * np[2] + m[2];
}
template <typename T, typename P>
__device__ __forceinline__ void load_psi(P* const in[6], const int m[3], const int* np,
                                         const int pos[3], int ny, int pz, T v[6]) {
#pragma unroll
  for (int t = 0; t < 6; ++t)
    v[t] = m[term_axis(t)] >= 0 ? in[t][psi_elem(t, m, np, pos, ny, pz)] : T(0);
}
template <typename T>
__device__ __forceinline__ void store_psi(T* const out[6], const int m[3], const int* np,
                                          const int pos[3], int ny, int pz, const T v[6]) {
#pragma unroll
  for (int t = 0; t < 6; ++t)
    if (m[term_axis(t)] >= 0) out[t][psi_elem(t, m, np, pos, ny, pz)] = v[t];
}
// The neighbours term by term (0 where the reference's loop has none).
template <typename T, int SGN>
__device__ __forceinline__ void load_neighbours(const T* const F[3], long long id,
                                                const long long st[3], const int pos[3],
                                                const int n[3], T nb[6]) {
#pragma unroll
  for (int t = 0; t < 6; ++t) {
    const int x = term_axis(t);
    const bool ok = SGN > 0 ? pos[x] + 1 < n[x] : pos[x] >= 1;
    nb[t] = ok ? F[term_comp(t)][id + (SGN > 0 ? st[x] : -st[x])] : T(0);
  }
}
// The three curl updates of a cell on a grid of any dimension (upd_hx ..
// upd_ez of cell_update.cuh with every operand already loaded).
template <typename T, int SGN>
__device__ __forceinline__ void curl_cell(const StepArgs<T>& a, const CellPml<T>& p,
                                          const int pos[3], const int n[3], const T K[3],
                                          const T own[3], const T nb[6], T f[3], T psi[6]) {
  const T dl[3] = {a.dx, a.dy, a.dz};
  const T rl[3] = {a.rdx, a.rdy, a.rdz};
  const bool fl[3] = {a.fdx, a.fdy, a.fdz};
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const int tA = 2 * c, tB = 2 * c + 1, xA = term_axis(tA), xB = term_axis(tB);
    const bool rA = n[xA] > 1, rB = n[xB] > 1;
    const bool okA = SGN > 0 ? pos[xA] < n[xA] - 1 : pos[xA] >= 1;
    const bool okB = SGN > 0 ? pos[xB] < n[xB] - 1 : pos[xB] >= 1;
    if (!((!rA || okA) && (!rB || okB) && (rA || rB))) continue;
    T dA = T(0), dB = T(0);
    if (rA) {
      const T o = own[term_comp(tA)];
      dA = qdiv(SGN > 0 ? sub_rn(nb[tA], o) : sub_rn(o, nb[tA]), dl[xA], rl[xA], fl[xA]);
    }
    if (rB) {
      const T o = own[term_comp(tB)];
      dB = qdiv(SGN > 0 ? sub_rn(nb[tB], o) : sub_rn(o, nb[tB]), dl[xB], rl[xB], fl[xB]);
    }
    const T curl = rA ? (rB ? sub_rn(dA, dB) : dA) : -dB;
    f[c] = add_rn(f[c], mul_rn(curl, K[c]));
    if (rA && p.m[xA] >= 0) f[c] = cpml_term(f[c], K[c], dA, p.b[xA], p.c[xA], psi[tA]);
    if (rB && p.m[xB] >= 0) f[c] = cpml_term(f[c], -K[c], dB, p.b[xB], p.c[xB], psi[tB]);
  }
}

template <typename T, int CE, bool ADE, int MODE>
__global__ void __launch_bounds__(res_threads<T>(MODE), res_blocks<T>(MODE))
    k_resident(const __grid_constant__ ResidentArgs<T> g) {
  constexpr int THR = res_threads<T>(MODE);
  constexpr bool ONE = MODE != kResGridN;
  const StepArgs<T>& a = g.a;
  const unsigned nthr = gridDim.x * THR;
  const unsigned me = blockIdx.x * THR + threadIdx.x;
  const unsigned ny = a.ny, nz = a.nz, N = (unsigned)a.nx * ny * nz;
  const int n[3] = {a.nx, a.ny, a.nz};
  const long long st[3] = {(long long)a.ny * a.pz, a.pz, 1};
  const T Kh[3] = {-a.ch, -a.ch, -a.ch};
  unsigned phase = g.phase0;
  // source groups on this thread's cells (few groups), else a barrier and
  // one thread per group
  unsigned mine[2] = {0u, 0u};
  const bool shared_h = g.src[1].n_groups > kResOwned, shared_e = g.src[0].n_groups > kResOwned;
#pragma unroll
  for (int f = 0; f < 2; ++f) {
    if (g.src[f].n_groups > kResOwned) continue;
    for (int q = 0; q < g.src[f].n_groups; ++q) {
      const unsigned c = (unsigned)g.src[f].cell[q];
      const unsigned flat = c / (unsigned)a.pz * nz + c % (unsigned)a.pz;
      if (flat % nthr == me) mine[f] |= 1u << q;
    }
  }
  auto place = [&](unsigned c, int pos[3]) {
    const unsigned row = nz == 1 ? c : c / nz;
    const unsigned i = row / ny;
    pos[0] = (int)i;
    pos[1] = (int)(row - i * ny);
    pos[2] = nz == 1 ? 0 : (int)(c - row * nz);
    return pos[0] * st[0] + pos[1] * st[1] + pos[2];
  };
  // ---- one cell per thread: its state for the whole launch
  int pos[3] = {0, 0, 0};
  long long id = 0;
  const bool live = ONE && me < N;
  CellPml<T> ph, pe;
  T e[3], h[3], psih[6], psie[6], K[3];
  uint32_t w = 0u;
  int at_dft[kResDft], at_flux[kFluxBatch];
  if (live) {
    id = place(me, pos);
    load_pml<T>(a.maph, a.bh, a.cph, pos, ph);
    load_pml<T>(a.mape, a.be, a.cpe, pos, pe);
    cell_coeffs<T, CE, ADE>(a, a.media, id, K, w);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      e[c] = a.Ein[c][id];
      h[c] = a.Hin[c][id];
    }
    load_psi<T>(a.psiHin, ph.m, a.nph, pos, a.ny, a.pz, psih);
    load_psi<T>(a.psiE, pe.m, a.npe, pos, a.ny, a.pz, psie);
    // place in the monitors, -1: not recorded
#pragma unroll
    for (int m = 0; m < kResDft; ++m) {
      at_dft[m] = -1;
      if (m >= g.n_dft) continue;
      const DftRegion& r = g.dft[m];
      int q[3];
      bool in = true;
#pragma unroll
      for (int x = 0; x < 3; ++x) {
        const int d = pos[x] - r.start[x];
        q[x] = d / r.stride[x];
        in = in && d >= 0 && d % r.stride[x] == 0 && q[x] < r.count[x];
      }
      if (in) at_dft[m] = (q[0] * r.count[1] + q[1]) * r.count[2] + q[2];
    }
#pragma unroll
    for (int m = 0; m < kFluxBatch; ++m) {
      at_flux[m] = -1;
      if (m >= g.n_flux || pos[g.flux[m].axis] != g.flux[m].idx) continue;
      const int u = g.flux[m].axis == 0 ? pos[1] : pos[0];
      const int v = g.flux[m].axis == 2 ? pos[1] : pos[2];
      at_flux[m] = u * g.flux[m].n1 + v;
    }
  }
  int taken[kResDft];
#pragma unroll
  for (int m = 0; m < kResDft; ++m) taken[m] = 0;

  for (int s = 0; s < g.n; ++s) {
    const long long step = g.step0 + s;
    const int lvl = (int)(step & 1);
    // ---- H pass
    if (ONE) {
      if (live) {
        T nb[6];
        load_neighbours<T, 1>(a.Ein, id, st, pos, n, nb);
        curl_cell<T, 1>(a, ph, pos, n, Kh, e, nb, h, psih);
#pragma unroll
        for (int c = 0; c < 3; ++c) a.Hout[c][id] = h[c];
      }
    } else {
      for (unsigned c = me; c < N; c += nthr) {
        int q[3];
        const long long o = place(c, q);
        CellPml<T> p;
        T own[3], f[3], nb[6], psi[6];
        load_pml<T>(a.maph, a.bh, a.cph, q, p);
#pragma unroll
        for (int x = 0; x < 3; ++x) {
          own[x] = a.Ein[x][o];
          f[x] = a.Hin[x][o];
        }
        load_neighbours<T, 1>(a.Ein, o, st, q, n, nb);
        load_psi<T>(a.psiHin, p.m, a.nph, q, a.ny, a.pz, psi);
        curl_cell<T, 1>(a, p, q, n, Kh, own, nb, f, psi);
#pragma unroll
        for (int x = 0; x < 3; ++x) a.Hout[x][o] = f[x];
        store_psi<T>(a.psiHout, p.m, a.nph, q, a.ny, a.pz, psi);
      }
    }
    if (shared_h) {
      if (!res_barrier<MODE>(g.bar, phase, g.err, g.spin)) return;
      for (int q = (int)me; q < g.src[1].n_groups; q += (int)nthr)
        inject_group<T>(g.src[1], q, a.Hout, step);
    } else {
      for (unsigned left = mine[1]; left; left &= left - 1u)
        inject_group<T>(g.src[1], __ffs(left) - 1, a.Hout, step);
    }
    AdeRec<T> rec;
    if (ADE && ONE && live && w) ade_load<T>(a, a.media, w, rec);  // its own: no barrier needed
    if (!res_barrier<MODE>(g.bar, phase, g.err, g.spin)) return;
    // ---- E pass
    if (ONE) {
      if (live) {
        T nb[6];
        load_neighbours<T, -1>(a.Hout, id, st, pos, n, nb);
        if (mine[1] || shared_h) {
#pragma unroll
          for (int c = 0; c < 3; ++c) h[c] = a.Hout[c][id];
        }
        const T en[3] = {e[0], e[1], e[2]};
        curl_cell<T, -1>(a, pe, pos, n, K, h, nb, e, psie);
        if (ADE && w) ade_update<T>(a, a.media, rec, lvl, en, e);
#pragma unroll
        for (int c = 0; c < 3; ++c) a.Eout[c][id] = e[c];
      }
    } else {
      for (unsigned c = me; c < N; c += nthr) {
        int q[3];
        const long long o = place(c, q);
        CellPml<T> p;
        T own[3], f[3], nb[6], psi[6], Kc[3];
        uint32_t t, wc;
        cell_word<T, CE, ADE>(a, o, Kc, t);
        load_pml<T>(a.mape, a.be, a.cpe, q, p);
#pragma unroll
        for (int x = 0; x < 3; ++x) {
          own[x] = a.Hout[x][o];
          f[x] = a.Ein[x][o];
        }
        load_neighbours<T, -1>(a.Hout, o, st, q, n, nb);
        cell_decode<T, CE, ADE>(a, a.media, t, Kc, wc);
        if (ADE && wc) ade_load<T>(a, a.media, wc, rec);
        load_psi<T>(a.psiE, p.m, a.npe, q, a.ny, a.pz, psi);
        const T en[3] = {f[0], f[1], f[2]};
        curl_cell<T, -1>(a, p, q, n, Kc, own, nb, f, psi);
        if (ADE && wc) ade_update<T>(a, a.media, rec, lvl, en, f);
#pragma unroll
        for (int x = 0; x < 3; ++x) a.Eout[x][o] = f[x];
        store_psi<T>(a.psiE, p.m, a.npe, q, a.ny, a.pz, psi);
      }
    }
    if (shared_e) {
      if (!res_barrier<MODE>(g.bar, phase, g.err, g.spin)) return;
      for (int q = (int)me; q < g.src[0].n_groups; q += (int)nthr)
        inject_group<T>(g.src[0], q, a.Eout, step);
      if (ONE && !res_barrier<MODE>(g.bar, phase, g.err, g.spin)) return;
    } else {
      for (unsigned left = mine[0]; left; left &= left - 1u)
        inject_group<T>(g.src[0], __ffs(left) - 1, a.Eout, step);
    }
    if (ONE) {
      // ---- samples of the thread's cell
      if (live) {
        if (mine[0] || shared_e) {
#pragma unroll
          for (int c = 0; c < 3; ++c) e[c] = a.Eout[c][id];
        }
#pragma unroll
        for (int m = 0; m < kResDft; ++m) {
          if (m >= g.n_dft || step % g.dft_interval[m]) continue;
          if (at_dft[m] >= 0) {
            const DftRegion& r = g.dft[m];
            T* ring = g.dft_ring[m] + (long long)(g.dft_slot[m] + taken[m]) * r.ncomp * r.ncell;
            for (int q = 0; q < r.ncomp; ++q) {
              const int c = r.comps[q];
              const T v = c == 0 ? e[0] : c == 1 ? e[1] : c == 2 ? e[2] : c == 3 ? h[0]
                                                                  : c == 4 ? h[1] : h[2];
              ring[q * r.ncell + at_dft[m]] = v;
            }
          }
          ++taken[m];
        }
#pragma unroll
        for (int m = 0; m < kFluxBatch; ++m) {
          if (m >= g.n_flux || at_flux[m] < 0) continue;
          const FluxPlane& p = g.flux[m];
          const T v0 = sub_rn(mul_rn(e[1], h[2]), mul_rn(e[2], h[1]));
          const T v1 = sub_rn(mul_rn(e[2], h[0]), mul_rn(e[0], h[2]));
          const T v2 = sub_rn(mul_rn(e[0], h[1]), mul_rn(e[1], h[0]));
          g.flux_val[m][(long long)(g.flux_slot[m] + s) * p.n0 * p.n1 + at_flux[m]] =
              p.axis == 0 ? v0 : (p.axis == 1 ? v1 : v2);
        }
      }
      if (!shared_e && !res_barrier<MODE>(g.bar, phase, g.err, g.spin)) return;
    } else {
      if (!res_barrier<MODE>(g.bar, phase, g.err, g.spin)) return;
      bool due = g.n_flux > 0;
      Fields6<T> F;
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        F.f[q] = a.Eout[q];
        F.f[3 + q] = a.Hout[q];
      }
#pragma unroll
      for (int m = 0; m < kResDft; ++m) {
        if (m >= g.n_dft || step % g.dft_interval[m]) continue;
        due = true;
        for (long long cell = me; cell < g.dft[m].ncell; cell += nthr)
          dft_sample_cell<T>(g.dft[m], g.dft_ring[m], g.dft_slot[m] + taken[m], F, cell, a.ny,
                             a.pz);
        ++taken[m];
      }
      for (int m = 0; m < g.n_flux; ++m) {
        const FluxPlane& p = g.flux[m];
        const long long np = (long long)p.n0 * p.n1;
        for (long long t = me; t < np; t += nthr)
          g.flux_val[m][(g.flux_slot[m] + s) * np + t] =
              flux_cell_value<T>(p, t, F, a.ny, a.pz);
      }
      if (due && !res_barrier<MODE>(g.bar, phase, g.err, g.spin)) return;
    }
  }
  if (live) {
    store_psi<T>(a.psiHout, ph.m, a.nph, pos, a.ny, a.pz, psih);
    store_psi<T>(a.psiE, pe.m, a.npe, pos, a.ny, a.pz, psie);
  }
}

// Block partials of kept flux values (blockIdx: 256-cell group, ring slot,
// plane), the sums k_flux_sample_batch writes per step.
template <typename T>
struct FluxKept {
  const T* val[kFluxBatch];
  double* partial[kFluxBatch];
  int cells[kFluxBatch], nblk[kFluxBatch], pending[kFluxBatch];
};
template <typename T>
__global__ void __launch_bounds__(256) k_flux_groups(FluxKept<T> f) {
  pdl_enter();
  __shared__ double sh[8];
  const int m = blockIdx.z;
  if ((int)blockIdx.x >= f.nblk[m] || (int)blockIdx.y >= f.pending[m]) return;  // whole block
  const int t = blockIdx.x * 256 + threadIdx.x;
  double v = t < f.cells[m] ? (double)f.val[m][(long long)blockIdx.y * f.cells[m] + t] : 0.0;
  v = block_sum256<T>(v, sh);
  if (threadIdx.x == 0) f.partial[m][(long long)blockIdx.y * f.nblk[m] + blockIdx.x] = v;
}

}  // namespace pfb
