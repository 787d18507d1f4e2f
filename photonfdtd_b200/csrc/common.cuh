// common.cuh - shared types and exactly-rounded arithmetic for the engine.
//
// Every field update in this engine reproduces the reference NumPy path's
// rounding sequence (src/photonfdtd/simulation.py:1138-1309): each add,
// subtract, multiply and divide is one IEEE round-to-nearest operation, and
// none is contracted into an FMA. The *_rn intrinsics below guarantee that
// regardless of -fmad, so a float32 run matches the reference float32 run
// bit for bit wherever the reference's own operation order is used.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace pfb {

__device__ __forceinline__ float add_rn(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double add_rn(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float sub_rn(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ double sub_rn(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float fma_rn(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fma_rn(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float div_rn(float a, float b) { return __fdiv_rn(a, b); }
__device__ __forceinline__ double div_rn(double a, double b) { return __ddiv_rn(a, b); }

// Correctly rounded a / d given r = RN(1/d), by Markstein's correction (P.
// Markstein, IBM J. Res. Dev. 34(1), 1990): q0 = RN(a r), rem = a - q0 d
// (exact in one FMA), q = RN(q0 + rem r). Everything runs on numerators
// prescaled by a power of two (exact), so that rem cannot underflow for any
// a down to the smallest subnormal, and the quotient is scaled back at the
// end; rem is formed as q0 d - a, which keeps the sign of a zero quotient.
//  float: prescale 2^64. Enabled for a divisor d only after checking all 2^23
//    significands of a against IEEE division. For d in [2^-30, 2^-23], |a| <
//    2^26 keeps every intermediate below 2^121, and a quotient is 0 or at least
//    2^-126, so scaling it back is exact; the 3D vector passes take other d with
//    limits of their own (StepArgs::qtop, qlow).
//  double: prescale 2^200, and one more correction: q0 can be two units off,
//    q1 = RN(q0 - rem r) is one of the two neighbours of a / d, and from such
//    a q1 Markstein's theorem makes the second correction the rounded
//    quotient for every d whose significand is not all ones and r = RN(1/d)
//    (the host checks that, and d in [2^-60, 1]). a is 0 or 2^-1022 <=
//    |a| < 2^700, so that a quotient is normal and scaling it back exact.
// Four FP32 (six FP64) operations per quotient and one to scale it back;
// sums and differences of scaled quotients are the scaled sums and
// differences, so a curl scales back once instead of per term.
template <typename T>
struct QScale;
template <>
struct QScale<float> {
  static constexpr float up = 0x1p64f, down = 0x1p-64f;
};
template <>
struct QScale<double> {
  static constexpr double up = 0x1p200, down = 0x1p-200;
};
// Quotient of a prescaled numerator, still scaled.
__device__ __forceinline__ float qscaled(float as, float d, float r) {
  const float q0 = __fmul_rn(as, r);
  return __fmaf_rn(-__fmaf_rn(q0, d, -as), r, q0);
}
__device__ __forceinline__ double qscaled(double as, double d, double r) {
  const double q0 = __dmul_rn(as, r);
  const double q1 = __fma_rn(-__fma_rn(q0, d, -as), r, q0);
  return __fma_rn(-__fma_rn(q1, d, -as), r, q1);
}
template <typename T>
__device__ __forceinline__ T qdiv_fast(T a, T d, T r) {
  return mul_rn(qscaled(mul_rn(a, QScale<T>::up), d, r), QScale<T>::down);
}
// Whether numerators may take the reciprocal path, tested over all of a cell's
// (or vector's) at once. SCALED: they are prescaled.
//  float: |a| < 2^26. A NaN must fail when prescaled: prescaling takes a finite
//    field of 2^64 or more to infinity, and beside an infinite neighbour the
//    prescaled difference is NaN where the difference is infinite.
//  double: 2^-1022 <= |a| < 2^700, by the exponent (infinities and NaN have the
//    largest): one shift-and-add and one compare per numerator. 0 fails that
//    too, so what fails is asked again one by one (sure; kAgain).
// These limits hold for divisors in [2^-30, 2^-23] (double: [2^-60, 1]); the
// constructor takes another upper limit, lowkey() serves a lower one (float).
// CHAIN (float): a chain of compares instead of a maximum and one compare. The
// batch's tile step is faster so (64 instances 59.0 against 62.8 us), the 3D
// passes with ADE, whose registers spill, without (192^3 170 against 173 us).
template <typename T, bool SCALED, bool CHAIN = false>
struct QCheck;
template <bool SCALED, bool CHAIN>
struct QCheck<float, SCALED, CHAIN> {
  static constexpr bool kAgain = false;
  float top;
  float m = 0.f;
  bool in = true;
  // top: prescaled
  __device__ __forceinline__ explicit QCheck(float t = 0x1p90f)
      : top(SCALED ? t : mul_rn(t, QScale<float>::down)) {}
  __device__ __forceinline__ void take(float n) {
    if (CHAIN) in = in & (fabsf(n) < top);
    else if (SCALED) asm("max.NaN.f32 %0, %1, %2;" : "=f"(m) : "f"(m), "f"(fabsf(n)));
    else m = fmaxf(m, fabsf(n));
  }
  __device__ __forceinline__ bool ok() const { return CHAIN ? in : m < top; }
  __device__ static __forceinline__ bool sure(float) { return false; }
  // Orders prescaled magnitudes; 0 comes last.
  __device__ static __forceinline__ unsigned lowkey(float n) {
    return 2u * __float_as_uint(SCALED ? n : mul_rn(n, QScale<float>::up)) - 1u;
  }
};
template <bool SCALED, bool CHAIN>
struct QCheck<double, SCALED, CHAIN> {
  static constexpr bool kAgain = true;
  // high words of 2^-1022 and 2^700, or of these times 2^200
  static constexpr unsigned lo = SCALED ? (1023u - 822u) << 20 : 1u << 20;
  static constexpr unsigned hi = (1023u + (SCALED ? 900u : 700u)) << 20;
  bool in = true;
  __device__ __forceinline__ explicit QCheck(double = 0.0) {}
  __device__ static __forceinline__ bool normal(double n) {
    return 2u * (unsigned)__double2hiint(n) - 2u * lo < 2u * (hi - lo);
  }
  __device__ __forceinline__ void take(double n) { in = in & normal(n); }
  __device__ __forceinline__ bool ok() const { return in; }
  __device__ static __forceinline__ bool sure(double n) { return n == 0.0 || normal(n); }
};
// The same for single numerators that are not prescaled.
template <typename T, typename... N>
__device__ __forceinline__ bool qdiv_ok(N... n) {
  QCheck<T, false, true> c;
  (c.take(n), ...);
  return c.ok() || (c.kAgain && (c.sure(n) && ...));
}
// IEEE division, out of line: the rare numerators beyond the reciprocal
// path's range would otherwise put a division routine at every quotient.
static __device__ __noinline__ float div_cold(float a, float d) { return __fdiv_rn(a, d); }
static __device__ __noinline__ double div_cold(double a, double d) { return __ddiv_rn(a, d); }
template <typename T>
__device__ __forceinline__ T qdiv(T a, T d, T r, bool fast) {
  if (fast && qdiv_ok<T>(a)) return qdiv_fast(a, d, r);
  return div_rn(a, d);
}
// Two exact quotients sharing one range check and one branch: both by the
// reciprocal path when it applies to both, else each by qdiv.
template <typename T>
__device__ __forceinline__ void qdiv2(T a0, T d0, T r0, bool f0, T a1, T d1, T r1, bool f1,
                                      T& q0, T& q1) {
  if (f0 && f1 && qdiv_ok<T>(a0, a1)) {
    q0 = qdiv_fast(a0, d0, r0);
    q1 = qdiv_fast(a1, d1, r1);
  } else {
    q0 = qdiv(a0, d0, r0, f0);
    q1 = qdiv(a1, d1, r1, f1);
  }
}

// Round a double to the field type (round to nearest even).
__device__ __forceinline__ float to_real(double v, float) { return __double2float_rn(v); }
__device__ __forceinline__ double to_real(double v, double) { return v; }

// F += v with v a double: the reference adds a float64 source value to a
// float32 cell in double precision and rounds once on store
// (simulation.py:1371-1372, numpy float32 + float64 -> float64).
template <typename T>
__device__ __forceinline__ T add_double(T f, double v) {
  return to_real(__dadd_rn((double)f, v), T());
}

// First statement of a kernel that launch_pdl launches: lets the next kernel
// of the stream be scheduled as soon as every block of this one has started
// (its blocks then wait here in what the last wave leaves free), and waits
// until everything before this kernel is complete and visible. Without the
// attribute both are no-ops.
__device__ __forceinline__ void pdl_enter() {
  asm volatile("griddepcontrol.launch_dependents;");
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

constexpr int kMaxPoles = 8;
constexpr int kMaxMedia = 16;
constexpr uint32_t kDispersiveBit = 0x80000000u;

// One dispersive medium as the E kernel sees it (simulation.py:572-636).
// Its polarisation state is two arrays, one per time level: level L's record
// of a cell is at P + L * plev + poff + loc * 3 * npole, laid out
// [pole][component]. A step reads both levels and rewrites one, so the
// rewritten records of consecutive cells are contiguous and a warp's stores
// fill whole sectors (each medium's block starts 8-real aligned). A
// dispersive cell's word is kDispersiveBit | medium << kMediumShift | loc.
template <typename T>
struct MediumT {
  long long poff, count;
  int npole;
  T inv;   // 1 / (eps0 * eps_inf), rounded to T as the reference's weak scalar
  T ce;    // dt / (eps_inf * eps0) in table mode
  T a[kMaxPoles], b[kMaxPoles], c[kMaxPoles];
};
constexpr int kMediumShift = 27;
constexpr uint32_t kLocMask = (1u << kMediumShift) - 1u;

// Soft sources of one family (simulation.py:1367-1390). Sources sharing a
// (component, cell) form one group, applied in the reference's list order.
struct SourceGroups {
  const long long* cell;   // flat cell index per group
  const int* comp;         // 0..2 within the family (x, y, z)
  const int* start;        // group g owns sources [start[g], start[g+1])
  const int* wave_row;     // per source
  const double* amp;       // per source
  const double* wave;      // [row][n_steps]
  long long n_steps;
  int n_groups;
};

// A DFT monitor's region: start / stride / count per axis, the components.
struct DftRegion {
  int start[3], stride[3], count[3];
  long long ncell;
  int ncomp;
  int comps[6];
};

// Arguments of one H + E step (split or fused kernels).
template <typename T>
struct StepArgs {
  int nx, ny, nz;
  int pz;  // reals from one row to the next: nz padded to 32 bytes, or 16 (1 when nz = 1)
  T dx, dy, dz;  // derivative divisors (1 on a collapsed axis)
  T rdx, rdy, rdz;      // RN(1/d) per axis
  bool fdx, fdy, fdz;   // reciprocal division verified exact for that axis
  bool fdall;           // and for all three
  // the same for the vector passes, which take divisors in [2^-60, 1]. Prescaled
  // limits of the numerators (float): below qtop, and with a QCheck::lowkey of
  // qlow or more (0: no lower limit)
  bool fdvec;
  T qtop;
  unsigned qlow;
  T ch;          // dt / mu0 rounded to T; the H coefficient is -ch
  const T* Ein[3];
  const T* Hin[3];
  T* Eout[3];
  T* Hout[3];
  // E coefficients: ce[c] per cell (CELL1 repeats one array), or word/table
  const T* ce[3];
  const uint32_t* word;
  const T* table;
  const uint32_t* adeword;  // CELL1 + ADE: 0 = plain, else 1 + compact index
  // CPML: coefficients on the E and H staggers per axis, compact maps
  const T* be[3];
  const T* cpe[3];
  const T* bh[3];
  const T* cph[3];
  const int* mape[3];
  const int* maph[3];
  const int* gze;  // vector passes: z-layer group of each vector of a row, or -1
  const int* gzh;
  int npe[3], nph[3];
  // Bulk boxes: cells [b0, b1) per axis where the H (hb) or E (eb) update has
  // both difference terms and no CPML state; they take the straight-line path.
  int hb0[3], hb1[3], eb0[3], eb1[3];
  // psi: E terms Ex_y, Ex_z, Ey_z, Ey_x, Ez_x, Ez_y; H terms Hx_y, Hx_z,
  // Hy_z, Hy_x, Hz_x, Hz_y (rustbackend.py:200-207 order)
  T* psiE[6];
  const T* psiEin[6];  // vector E pass: psi before the step (psiE, or the last record's)
  const T* psiHin[6];
  T* psiHout[6];
  // ADE
  const MediumT<T>* media;
  int n_media;
  T* P;
  long long plev;  // reals per polarisation level
  int lvl;         // polarisation level holding P^n (n & 1)
  int wait_test;   // test hook of the TMA-staged step (pf_set_wait_test)
};

enum CeMode { kCeCell1 = 0, kCeCell3 = 1, kCeTable = 2 };

// Host: whether the reciprocal division of qdiv is exact for divisor d (float:
// exhaustive check over all significands; double: the theorem's conditions;
// defined in engine.cu).
bool host_recip_division_exact(float d);
bool host_recip_division_exact(double d);

}  // namespace pfb
