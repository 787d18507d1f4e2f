// engine.cu - the C ABI of libpfb200.so (declared in include/pfb200.h).
//
// Device state of one engine (all in HBM for the whole run):
//   fields   6 components, C-order (nx, ny, nz) with rows padded to 32 or 16 bytes
//            (pz reals, the padding zero). The split and vector passes update
//            in place (level 0); the fused kernels recompute H on tile halos,
//            so they read level `cur` and write level `cur ^ 1`
//   ce       one or three per-cell arrays, or a uint32 word per cell + table
//   CPML     b/c per axis and stagger, compact maps (-1 = no psi), psi
//            compacted along its derivative axis
//   ADE      compact polarisation state [level][pole][comp][cells] per medium
//   monitors sample rings + complex128 accumulators (DFT), block partials +
//            float64 accumulators (flux)
#include <algorithm>
#include <atomic>
#include <type_traits>
#include <cstdarg>
#include <cstdio>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/pfb200.h"
#include "common.cuh"
#include "devmem.cuh"
#include "kernels_adj.cuh"
#include "kernels_adj_vec.cuh"
#include "kernels_aux.cuh"
#include "kernels_fused.cuh"
#include "kernels_resident.cuh"
#include "kernels_split.cuh"
#include "kernels_tma.cuh"
#include "kernels_vec3d.cuh"

using namespace pfb;

namespace {

constexpr int kRingMax = 32;
static_assert(kRingMax <= kFluxRing, "k_flux_flush keeps one sum per pending sample");
constexpr size_t kRingBytesCap = 256u << 20;
thread_local std::string g_create_error;

struct DftMon {
  DftRegion r;
  int n_freq = 0, interval = 1;
  double dt = 0;
  std::vector<double> h_ph_e, h_ph_h;
  long long n_samples = 0;   // samples in the whole run
  long long q_done = 0;      // samples folded into acc
  int pending = 0;           // samples waiting in the ring
  int ring_cap = 1;
  void* ring = nullptr;
  double* acc = nullptr;
  double* ph_e = nullptr;
  double* ph_h = nullptr;
};

struct FluxMon {
  FluxPlane p;
  double dA = 0, dt = 0;
  int pending = 0;
  int ring_cap = kRingMax;
  double* partial = nullptr;
  double* acc = nullptr;
  void* val = nullptr;  // resident launches: the plane's values per pending sample
  // adjoint: dJ/dflux and the replay's E plane records (2 * n0 * n1 reals
  // per recorded step, rec_cap steps)
  double cot = 0.0;
  void* rec = nullptr;
  long long rec_cap = 0;
};

struct SrcFamily {
  std::vector<long long> cell;
  std::vector<int> comp, start, wave_row;
  std::vector<double> amp;
  SourceGroups dev{};
};

}  // namespace

struct pf_engine {
  int nx = 0, ny = 0, nz = 0, rb = 4;
  double dl[3] = {1, 1, 1};
  double ch = 0;
  long long n_steps = 0;
  long long ncell = 0;
  int pz = 1;            // row pitch of fields, coefficients, words and psi rows
  long long ncellp = 0;  // nx * ny * pz
  bool vec = false;      // 3D with aligned rows: the vector passes
  int kernel = PF_KERNEL_AUTO;
  bool finalized = false;
  long long step = 0;
  int cur = 0;
  std::string err;
  cudaStream_t stream = nullptr;
  int device = 0;
  size_t dev_bytes = 0;
  std::vector<void*> allocs;

  // staged tables
  int ce_mode = -1;
  std::vector<char> h_ce[3];
  // PF_CE_TABLE: the word goes to the device in pf_set_ce; word_need[m] is
  // 1 + the largest record index its dispersive words give medium m (0: none)
  long long word_need[kMaxMedia] = {};
  std::vector<double> h_table;
  std::vector<char> h_cpml[3][4];  // b_e, c_e, b_h, c_h
  int n_media = 0;
  std::vector<long long> m_count;
  std::vector<int> m_npole;
  std::vector<double> m_coef, m_inv, m_ce;
  std::vector<uint32_t> h_adeword;
  SrcFamily src[2];  // 0 = E family, 1 = H family
  int n_wave = 0;
  std::vector<double> h_wave;
  std::vector<DftMon> dfts;
  std::vector<FluxMon> fluxes;

  // device
  void* E[2][3] = {};
  void* H[2][3] = {};
  void* ce[3] = {};
  uint32_t* word = nullptr;
  void* table = nullptr;
  uint32_t* adeword = nullptr;
  void* cp[3][4] = {};
  int* map_e[3] = {};
  int* map_h[3] = {};
  int npe[3] = {}, nph[3] = {};
  int* gze = nullptr;     // vector passes: z-layer group per vector of a row
  int* gzh = nullptr;
  int ncz_e = 0, ncz_h = 0;  // z cells with CPML state, and their places in a psi row
  int* zpos_e = nullptr;
  int* zpos_h = nullptr;
  int hb0[3] = {}, hb1[3] = {}, eb0[3] = {}, eb1[3] = {};
  void* psiE[6] = {};
  void* psiH[2][6] = {};
  long long npsiE[6] = {}, npsiH[6] = {};  // reals per psi array (padded rows)
  long long rpsiE[6] = {}, rpsiH[6] = {};  // its rows of nz reals (0: contiguous)
  void* P = nullptr;
  long long plev = 0;  // reals per polarisation level
  void* media = nullptr;
  double* wave = nullptr;
  int* flag = nullptr;
  unsigned* res_bar = nullptr;  // resident launches: grid barrier, error (mapped host memory)
  ErrWord res_err;
  bool res_asked = false;       // resident launches fit this context
  bool res_off = false;         // they do not
  bool flux_kept = false;  // the pending flux samples are kept values, not partials
  int sms = 0;
  void* region = nullptr;     // pf_read_region staging buffer (grown on demand)
  size_t region_bytes = 0;
  bool fused = false;
  double rdl[3] = {1, 1, 1};     // RN(1/d) in the real type, per axis
  bool fdiv[3] = {false, false, false};  // reciprocal division verified
  bool vdiv = false;             // the same for the vector passes, all axes
  bool vwide = false;            // with limits other than the scalar passes' window gives
  float qtop = 0;                // which are these (StepArgs)
  uint32_t qlow = 0;
  bool ade_cells = false;        // E pass of a dispersive scene: one cell per thread
  bool tma = false;      // fused path stages planes with TMA
  TmaMaps maps;
  int* tma_err = nullptr;
  int wait_test = 0;     // pf_set_wait_test: 1 a bounded wait runs out, 2 no resident launches
  long long check_every = 0;  // pf_set_check_every: non-finite scan period
  int fused_ty = 8;      // fused tile height (8 or 16), env PFB200_FUSED_TY
  int fused_chunks = 0;  // x chunks per column (0 = auto), env PFB200_XCHUNKS

  // adjoint (pf_adj_*): adjoint fields, quotient and psi adjoints, the
  // gradient, and the ring of per-step forward records a replay writes
  bool adj = false;
  bool recording = false;
  long long rec_step0 = 0, ring_steps = 0, adj_next = 0;
  void* lamE[3] = {};
  void* lamH[3] = {};
  void* gE[6] = {};
  void* gH[6] = {};
  void* lpE[6] = {};
  void* lpH[6] = {};
  double* grad = nullptr;
  char* rec = nullptr;
  size_t rec_slot = 0;          // bytes per recorded step: H (3 fields) + psi_E
  std::vector<double*> dft_cot;  // per DFT monitor: dJ/d acc on the device, or null
  struct RegionSource {
    long long step;
    int comp;
    DftRegion r;
    double* vals;
  };
  std::vector<RegionSource> rsrc;  // FieldMonitor-frame sources of the loss

  // launch accounting (pf_read_profile)
  long long launches[4] = {};
  double prof_ms[4] = {};
  bool profiling = false;
  std::vector<cudaEvent_t> ev_pool;
  std::vector<std::pair<int, int>> ev_pending;  // (kind, first event)
  size_t ev_used = 0;
};

namespace {

int fail(pf_engine* e, int code, const char* fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof buf, fmt, ap);
  va_end(ap);
  if (e)
    e->err = buf;
  else
    g_create_error = buf;
  return code;
}

#define PF_CUDA(e, call)                                                                   \
  do {                                                                                     \
    cudaError_t rc_ = (call);                                                              \
    if (rc_ != cudaSuccess)                                                                \
      return fail((e), rc_ == cudaErrorMemoryAllocation ? PF_ERR_OOM : PF_ERR_CUDA,        \
                  "CUDA error: %s (%s) at %s:%d", cudaGetErrorString(rc_), #call, __FILE__, \
                  __LINE__);                                                               \
  } while (0)

int dalloc(pf_engine* e, void** p, size_t bytes) {
  if (bytes == 0) bytes = 16;
  cudaError_t rc = pool_alloc(p, bytes, e->device, e->stream);
  if (rc != cudaSuccess)
    return fail(e, PF_ERR_OOM, "CUDA error: allocation of %zu bytes failed: %s", bytes,
                cudaGetErrorString(rc));
  e->allocs.push_back(*p);
  e->dev_bytes += bytes;
  rc = cudaMemsetAsync(*p, 0, bytes, e->stream);
  if (rc != cudaSuccess) return fail(e, PF_ERR_CUDA, "CUDA error: %s", cudaGetErrorString(rc));
  return PF_OK;
}

int upload(pf_engine* e, void** p, const void* src, size_t bytes) {
  int rc = dalloc(e, p, bytes);
  if (rc) return rc;
  if (bytes) PF_CUDA(e, cudaMemcpyAsync(*p, src, bytes, cudaMemcpyHostToDevice, e->stream));
  return PF_OK;
}

// The compact staging buffer, grown on demand (pf_read_region and copies
// between compact host arrays and padded rows).
int stage(pf_engine* e, size_t bytes) {
  if (bytes <= e->region_bytes) return PF_OK;
  if (e->region) {
    pool_free(e->region, e->stream);
    e->dev_bytes -= e->region_bytes;
    e->region = nullptr;
    e->region_bytes = 0;
  }
  const cudaError_t rc = pool_alloc(&e->region, bytes, e->device, e->stream);
  if (rc != cudaSuccess)
    return fail(e, PF_ERR_OOM, "CUDA error: allocation of %zu bytes failed", bytes);
  e->region_bytes = bytes;
  e->dev_bytes += bytes;
  return PF_OK;
}

RowCopy row_copy(void* padded, void* compact, size_t rows, int w, int p, const int* pos) {
  // m exceeds 2^(31 + s) / w by at most 1 with 2^s >= w, so the product's
  // error stays below 1 / w of the shift for every n < 2^31
  int s = 0;
  while ((1LL << s) < w) ++s;
  return RowCopy{padded, compact, pos, (unsigned)(rows * w), (unsigned)w, (unsigned)p,
                 (unsigned)((1ull << (31 + s)) / (unsigned)w + 1), 31 + s};
}
void launch_copy_rows(pf_engine* e, const RowCopies& c, int n, size_t elem, bool get) {
  unsigned most = 1;
  for (int q = 0; q < n; ++q) most = std::max(most, c.r[q].total);
  const dim3 g(std::min<unsigned>((most + 1023) / 1024, 148 * 8), n);
  if (elem == 4) k_copy_rows<uint32_t><<<g, 256, 0, e->stream>>>(c, get);
  else k_copy_rows<uint64_t><<<g, 256, 0, e->stream>>>(c, get);
}

// Copies between a compact array (kind says where it lies) and `rows` rows of w
// elements, p apart, through the staging buffer, kStage bytes at a time: the
// buffer is free for the next piece in stream order.
constexpr size_t kStage = 256u << 20;
int copy_staged(pf_engine* e, void* padded, void* compact, size_t rows, int w, int p,
                const int* pos, size_t elem, cudaMemcpyKind kind, bool to_padded) {
  const size_t row = (size_t)w * elem;
  const size_t most = std::max<size_t>(1, kStage / row);  // rows of one piece
  int rc = stage(e, std::min(most, rows) * row);
  if (rc) return rc;
  for (size_t r = 0; r < rows; r += most) {
    const size_t n = std::min(most, rows - r);
    char* at = (char*)compact + r * row;
    if (to_padded) PF_CUDA(e, cudaMemcpyAsync(e->region, at, n * row, kind, e->stream));
    RowCopies c = {};
    c.r[0] = row_copy((char*)padded + r * p * elem, e->region, n, w, p, pos);
    launch_copy_rows(e, c, 1, elem, !to_padded);
    PF_CUDA(e, cudaGetLastError());
    if (!to_padded) PF_CUDA(e, cudaMemcpyAsync(at, e->region, n * row, kind, e->stream));
  }
  return PF_OK;
}

// Copies `rows` rows of nz elements between a host array and a device array with
// the engine's row pitch.
int copy_rows(pf_engine* e, void* padded, void* compact, size_t rows, size_t elem, bool to_padded) {
  const cudaMemcpyKind kind = to_padded ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToHost;
  const size_t bytes = rows * e->nz * elem;
  if (bytes == 0) return PF_OK;
  if (e->nz != e->pz)
    return copy_staged(e, padded, compact, rows, e->nz, e->pz, nullptr, elem, kind, to_padded);
  PF_CUDA(e, cudaMemcpyAsync(to_padded ? padded : compact, to_padded ? compact : padded, bytes,
                             kind, e->stream));
  return PF_OK;
}

// A cell array of the grid from the host, into new padded device memory.
int upload_cells(pf_engine* e, void** p, const void* src, size_t elem) {
  int rc = dalloc(e, p, (size_t)e->ncellp * elem);
  if (rc) return rc;
  return copy_rows(e, *p, const_cast<void*>(src), (size_t)e->nx * e->ny, elem,
                   true);
}

// Whether qdiv's reciprocal division (q0 = a*r, rem = fma(-q0, d, a),
// q = fma(rem, r, q0), r = RN(1/d)) equals IEEE a / d for every float
// significand a in [1, 2). Sign and binade of a do not change the outcome
// while nothing over- or underflows; the device's 2^64 prescaling and the
// range checks keep every input of the fast path in that regime. The answer per
// divisor is kept for the process, so engines on the same grid spacing check
// it once. scan(d): the check itself.
template <typename Scan>
bool recip_division_known(float d, Scan scan) {
  static std::mutex mu;
  static std::map<uint32_t, bool> known;
  uint32_t key;
  memcpy(&key, &d, 4);
  {
    std::lock_guard<std::mutex> lk(mu);
    auto it = known.find(key);
    if (it != known.end()) return it->second;
  }
  const bool ok = scan(d);
  std::lock_guard<std::mutex> lk(mu);
  known[key] = ok;
  return ok;
}
// On the host: about 8.4M fmaf evaluations (~50 ms).
bool recip_division_scan(float d) {
  const float r = 1.0f / d;
  for (uint32_t m = 0; m < (1u << 23); ++m) {
    const uint32_t bits = 0x3f800000u | m;
    float a;
    memcpy(&a, &bits, 4);
    volatile float q0 = a * r;
    const float rem = std::fmaf(-q0, d, a);
    const float q = std::fmaf(rem, r, q0);
    volatile float ref = a / d;
    if (q != ref) return false;
  }
  return true;
}
bool recip_division_exact(float d) {
  return d >= 0x1p-30f && d <= 0x1p-23f && recip_division_known(d, recip_division_scan);
}

// The double reciprocal division of qdiv (two corrections): r = 1 / d is
// correctly rounded here, so Markstein's theorem needs only a divisor whose
// significand is not all ones, and a range where nothing over- or underflows.
bool recip_division_provable(double d) {
  uint64_t bits;
  memcpy(&bits, &d, 8);
  const uint64_t frac = (1ull << 52) - 1;
  return (bits & frac) != frac;
}
bool recip_division_exact(double d) {
  return d >= 0x1p-30 && d <= 0x1p-23 && recip_division_provable(d);
}

// What the vector passes need of the grid's divisors: every one in [2^-60, 1]
// and exact. Divisors outside the scalar passes' window (2^-30 .. 2^-23) are
// checked on the device, some 30 us, since such grids had nothing to check.
int vector_division(pf_engine* e) {
  e->vdiv = false;
  if (!e->vec || e->fused || getenv("PFB200_IEEE_DIV")) return PF_OK;
  const double dmin = std::min({e->dl[0], e->dl[1], e->dl[2]});
  const double dmax = std::max({e->dl[0], e->dl[1], e->dl[2]});
  if (!(dmin >= 0x1p-60 && dmax <= 1.0)) return PF_OK;
  int rc = PF_OK;
  auto scan = [&](float d) {
    int bad = 1;
    cudaMemsetAsync(e->flag, 0, sizeof(int), e->stream);
    k_recip_exact<<<592, 256, 0, e->stream>>>(d, 1.0f / d, e->flag);
    cudaMemcpyAsync(&bad, e->flag, sizeof(int), cudaMemcpyDeviceToHost, e->stream);
    if (cudaStreamSynchronize(e->stream) != cudaSuccess) {
      rc = PF_ERR_CUDA;
      return false;
    }
    return bad == 0;
  };
  bool ok = true;
  for (int ax = 0; ax < 3 && ok; ++ax)
    ok = e->rb == 8 ? recip_division_provable(e->dl[ax])
                    : recip_division_exact((float)e->dl[ax]) ||
                          recip_division_known((float)e->dl[ax], scan);
  if (rc) return fail(e, rc, "CUDA error: checking the grid spacing's reciprocal failed");
  e->vdiv = ok;
  // prescaled numerators: quotients from 2^-62 (normal once scaled back; below
  // 2^-23 every numerator gives one) to 2^121
  int lo, hi;
  std::frexp((float)dmin, &lo);  // dmin >= 2^(lo - 1)
  std::frexp((float)dmax, &hi);  // dmax < 2^hi
  e->qtop = std::min(0x1p90f, std::ldexp(1.0f, 121 + lo - 1));
  e->qlow = 0;
  if (dmax > 0x1p-23) {
    const float low = std::ldexp(1.0f, -62 + hi);
    memcpy(&e->qlow, &low, 4);
    e->qlow = 2 * e->qlow - 1;
  }
  e->vwide = e->qlow || e->qtop != 0x1p90f;
  return PF_OK;
}

// Bracket one launch of `kind` (0 step, 1 sources, 2 sampling, 3 flush).
struct LaunchScope {
  pf_engine* e;
  int kind;
  LaunchScope(pf_engine* eng, int k) : e(eng), kind(k) {
    e->launches[kind]++;
    if (!e->profiling) return;
    while (e->ev_pool.size() < e->ev_used + 2) {
      cudaEvent_t ev;
      cudaEventCreate(&ev);
      e->ev_pool.push_back(ev);
    }
    cudaEventRecord(e->ev_pool[e->ev_used], e->stream);
  }
  ~LaunchScope() {
    if (!e->profiling) return;
    cudaEventRecord(e->ev_pool[e->ev_used + 1], e->stream);
    e->ev_pending.push_back({kind, (int)e->ev_used});
    e->ev_used += 2;
  }
};

// Fold recorded event pairs into prof_ms (the stream must be idle).
void collect_profile(pf_engine* e) {
  for (auto& pr : e->ev_pending) {
    float ms = 0.f;
    if (cudaEventElapsedTime(&ms, e->ev_pool[pr.second], e->ev_pool[pr.second + 1]) == cudaSuccess)
      e->prof_ms[pr.first] += ms;
  }
  e->ev_pending.clear();
  e->ev_used = 0;
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                  const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = (EncodeTiledFn)p;
  }
  return fn;
}

// Tiled map over a C-order (nx, ny, nz) array, box (bw along z) x (bh along y)
// x 1 plane. Zero fill outside the array.
bool make_map(CUtensorMap* m, void* ptr, CUtensorMapDataType dt, int elem, int nx, int ny, int nz,
              int pz, int bw, int bh) {
  EncodeTiledFn enc = encode_fn();
  if (!enc) return false;
  const cuuint64_t dims[3] = {(cuuint64_t)nz, (cuuint64_t)ny, (cuuint64_t)nx};
  const cuuint64_t strides[2] = {(cuuint64_t)pz * elem, (cuuint64_t)ny * pz * elem};
  const cuuint32_t box[3] = {(cuuint32_t)bw, (cuuint32_t)bh, 1};
  const cuuint32_t es[3] = {1, 1, 1};
  return enc(m, dt, 3, ptr, dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
             CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Tensor maps of the TMA fused path (tile height 8); false if any fails.
template <typename T>
bool build_maps(pf_engine* e) {
  const CUtensorMapDataType dt =
      sizeof(T) == 4 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_FLOAT64;
  const int S = sizeof(T), TY = 8;
  memset(&e->maps, 0, sizeof e->maps);
  bool ok = true;
  for (int l = 0; l < 2; ++l)
    for (int c = 0; c < 3; ++c) {
      ok = ok && make_map(&e->maps.e[l][c], e->E[l][c], dt, S, e->nx, e->ny, e->nz, e->pz, kBoxW,
                         TY + 2);
      ok = ok && make_map(&e->maps.h[l][c], e->H[l][c], dt, S, e->nx, e->ny, e->nz, e->pz, kBoxW,
                         TY + 1);
    }
  void* wptr = e->ce_mode == PF_CE_TABLE ? (void*)e->word : (void*)e->adeword;
  if (wptr)
    ok = ok && make_map(&e->maps.word, wptr, CU_TENSOR_MAP_DATA_TYPE_UINT32, 4, e->nx, e->ny,
                        e->nz, e->pz, 32, TY);
  if (e->ce_mode != PF_CE_TABLE)
    for (int c = 0; c < 3; ++c)
      ok = ok && make_map(&e->maps.ce[c], e->ce[c], dt, S, e->nx, e->ny, e->nz, e->pz, 32, TY);
  return ok;
}

template <typename T>
int finalize_typed(pf_engine* e) {
  const size_t S = sizeof(T);
  const long long n = e->ncellp;
  const int dims[3] = {e->nx, e->ny, e->nz};
  int rc;
  const int levels = e->fused ? 2 : 1;
  for (int lvl = 0; lvl < levels; ++lvl)
    for (int c = 0; c < 3; ++c) {
      if ((rc = dalloc(e, &e->E[lvl][c], n * S))) return rc;
      if ((rc = dalloc(e, &e->H[lvl][c], n * S))) return rc;
    }
  // E coefficients
  if (e->ce_mode == PF_CE_CELL1) {
    if ((rc = upload_cells(e, &e->ce[0], e->h_ce[0].data(), S))) return rc;
    e->ce[1] = e->ce[2] = e->ce[0];
  } else if (e->ce_mode == PF_CE_CELL3) {
    for (int c = 0; c < 3; ++c)
      if ((rc = upload_cells(e, &e->ce[c], e->h_ce[c].data(), S))) return rc;
  } else {
    std::vector<T> tab(e->h_table.size());
    for (size_t q = 0; q < tab.size(); ++q) tab[q] = (T)e->h_table[q];
    if ((rc = upload(e, &e->table, tab.data(), tab.size() * S))) return rc;
  }
  // CPML: coefficients, compact maps, psi
  for (int ax = 0; ax < 3; ++ax) {
    const int na = dims[ax];
    std::vector<T> arr[4];
    for (int q = 0; q < 4; ++q) {
      arr[q].assign(ax == 2 ? e->pz : na, T(0));  // z: vectors past the row's end read zeros
      if (!e->h_cpml[ax][q].empty()) memcpy(arr[q].data(), e->h_cpml[ax][q].data(), na * S);
      if ((rc = upload(e, &e->cp[ax][q], arr[q].data(), arr[q].size() * S))) return rc;
    }
    std::vector<int> me(na, -1), mh(na, -1);
    int ce_n = 0, ch_n = 0;
    if (e->vec && ax == 2) {
      // the vector passes keep the z layers' psi in whole groups of V entries
      const int V = 16 / (int)S;
      auto groups = [&](const std::vector<T>& c, std::vector<int>& map, std::vector<int>& pos,
                        int** gdev, int** pdev) {
        std::vector<int> g;
        int n = 0;
        for (int t = 0; t < na; t += V) {
          bool any = false;
          for (int u = t; u < std::min(na, t + V); ++u)
            if (c[u] != T(0)) {
              any = true;
              map[u] = n + (u - t);
              pos.push_back(map[u]);
            }
          g.push_back(any ? n / V : -1);
          if (any) n += V;
        }
        int r = upload(e, (void**)gdev, g.data(), g.size() * 4);
        if (!r) r = upload(e, (void**)pdev, pos.data(), pos.size() * 4);
        if (!r && cudaStreamSynchronize(e->stream) != cudaSuccess) r = PF_ERR_CUDA;
        return r ? -1 : n;
      };
      std::vector<int> pe, ph;
      ce_n = groups(arr[1], me, pe, &e->gze, &e->zpos_e);
      ch_n = groups(arr[3], mh, ph, &e->gzh, &e->zpos_h);
      if (ce_n < 0 || ch_n < 0) return fail(e, PF_ERR_CUDA, "uploading the z-layer groups failed");
      e->ncz_e = (int)pe.size();
      e->ncz_h = (int)ph.size();
    } else {
      for (int t = 0; t < na; ++t) {
        if (arr[1][t] != T(0)) me[t] = ce_n++;
        if (arr[3][t] != T(0)) mh[t] = ch_n++;
      }
      if (ax == 2) {
        e->ncz_e = ce_n;
        e->ncz_h = ch_n;
      }
    }
    e->npe[ax] = ce_n;
    e->nph[ax] = ch_n;
    // Longest run of cells with no psi and both neighbours present: H needs
    // t <= na-2 (forward difference), E needs t >= 1 (backward difference).
    auto longest = [&](const std::vector<int>& map, int lo, int hi, int& b0, int& b1) {
      b0 = b1 = 0;
      int s0 = -1;
      for (int t = lo; t <= hi; ++t) {
        const bool ok = t < hi && map[t] < 0;
        if (ok && s0 < 0) s0 = t;
        if (!ok && s0 >= 0) {
          if (t - s0 > b1 - b0) { b0 = s0; b1 = t; }
          s0 = -1;
        }
      }
    };
    if (na > 1) {
      longest(mh, 0, na - 1, e->hb0[ax], e->hb1[ax]);
      longest(me, 1, na, e->eb0[ax], e->eb1[ax]);
    }
    if ((rc = upload(e, (void**)&e->map_e[ax], me.data(), na * 4))) return rc;
    if ((rc = upload(e, (void**)&e->map_h[ax], mh.data(), na * 4))) return rc;
  }
  const long long nx = e->nx, ny = e->ny, pz = e->pz;
  // psi extents: the term's derivative axis replaced by its PML cell count;
  // the x and y layers keep rows along z with the fields' pitch
  const long long rE[6] = {nx * e->npe[1], 0, 0, e->npe[0] * ny, e->npe[0] * ny, nx * e->npe[1]};
  const long long rH[6] = {nx * e->nph[1], 0, 0, e->nph[0] * ny, e->nph[0] * ny, nx * e->nph[1]};
  long long eE[6], eH[6];
  for (int q = 0; q < 6; ++q) {
    const bool z = q == 1 || q == 2;
    e->rpsiE[q] = rE[q];
    e->rpsiH[q] = rH[q];
    eE[q] = z ? nx * ny * e->npe[2] : rE[q] * pz;
    eH[q] = z ? nx * ny * e->nph[2] : rH[q] * pz;
  }
  for (int q = 0; q < 6; ++q) {
    e->npsiE[q] = eE[q];
    e->npsiH[q] = eH[q];
    if ((rc = dalloc(e, &e->psiE[q], eE[q] * S))) return rc;
    for (int lvl = 0; lvl < levels; ++lvl)
      if ((rc = dalloc(e, &e->psiH[lvl][q], eH[q] * S))) return rc;
  }
  // ADE: two levels of per-medium cell records [pole][component]; each
  // medium's block starts 8-real aligned (vector loads, whole-sector stores)
  if (e->n_media > 0) {
    std::vector<MediumT<T>> md(e->n_media);
    long long off = 0;
    size_t ci = 0;
    for (int m = 0; m < e->n_media; ++m) {
      MediumT<T>& M = md[m];
      memset(&M, 0, sizeof M);
      off = (off + 7) & ~7LL;
      M.poff = off;
      M.count = e->m_count[m];
      M.npole = e->m_npole[m];
      M.inv = (T)e->m_inv[m];
      M.ce = e->m_ce.empty() ? T(0) : (T)e->m_ce[m];
      for (int p = 0; p < M.npole; ++p) {
        M.a[p] = (T)e->m_coef[ci++];
        M.b[p] = (T)e->m_coef[ci++];
        M.c[p] = (T)e->m_coef[ci++];
      }
      off += 3LL * M.npole * M.count;
    }
    e->plev = (off + 7) & ~7LL;
    if ((rc = dalloc(e, &e->P, 2 * e->plev * S))) return rc;
    if ((rc = upload(e, &e->media, md.data(), md.size() * sizeof(MediumT<T>)))) return rc;
    if (e->ce_mode == PF_CE_CELL1)
      if ((rc = upload_cells(e, (void**)&e->adeword, e->h_adeword.data(), 4))) return rc;
    if (e->ce_mode == PF_CE_TABLE && e->m_ce.size() != (size_t)e->n_media)
      return fail(e, PF_ERR_INVALID, "table mode needs each medium's coefficient");
  }
  // sources
  if (e->n_wave > 0)
    if ((rc = upload(e, (void**)&e->wave, e->h_wave.data(), e->h_wave.size() * 8))) return rc;
  for (int f = 0; f < 2; ++f) {
    SrcFamily& s = e->src[f];
    SourceGroups& d = s.dev;
    d.n_groups = (int)s.cell.size();
    d.n_steps = e->n_steps;
    d.wave = e->wave;
    if (d.n_groups == 0) continue;
    std::vector<long long> cell(s.cell);
    for (long long& c : cell) c = c / e->nz * e->pz + c % e->nz;
    if ((rc = upload(e, (void**)&d.cell, cell.data(), cell.size() * 8))) return rc;
    if ((rc = upload(e, (void**)&d.comp, s.comp.data(), s.comp.size() * 4))) return rc;
    if ((rc = upload(e, (void**)&d.start, s.start.data(), s.start.size() * 4))) return rc;
    if ((rc = upload(e, (void**)&d.wave_row, s.wave_row.data(), s.wave_row.size() * 4))) return rc;
    if ((rc = upload(e, (void**)&d.amp, s.amp.data(), s.amp.size() * 8))) return rc;
  }
  // monitors
  for (DftMon& m : e->dfts) {
    const size_t per = (size_t)m.r.ncomp * m.r.ncell * S;
    m.ring_cap = (int)std::max<size_t>(1, std::min<size_t>(kRingMax, kRingBytesCap / std::max<size_t>(per, 1)));
    if ((rc = dalloc(e, &m.ring, per * m.ring_cap))) return rc;
    if ((rc = dalloc(e, (void**)&m.acc, (size_t)m.r.ncomp * m.n_freq * m.r.ncell * 16))) return rc;
    if ((rc = upload(e, (void**)&m.ph_e, m.h_ph_e.data(), m.h_ph_e.size() * 8))) return rc;
    if ((rc = upload(e, (void**)&m.ph_h, m.h_ph_h.data(), m.h_ph_h.size() * 8))) return rc;
  }
  for (FluxMon& f : e->fluxes) {
    if ((rc = dalloc(e, (void**)&f.partial, (size_t)f.ring_cap * f.p.nblk * 8))) return rc;
    if ((rc = dalloc(e, (void**)&f.acc, 8))) return rc;
  }
  if ((rc = dalloc(e, (void**)&e->flag, sizeof(int)))) return rc;
  if ((rc = dalloc(e, (void**)&e->tma_err, sizeof(int)))) return rc;
  // TMA staging needs 16-byte row strides (nz * sizeof(T) % 16 == 0)
  if (e->fused && !getenv("PFB200_NO_TMA") && ((long long)e->nz * S) % 16 == 0 &&
      !(e->n_media > 0 && e->ce_mode == PF_CE_CELL3))
    e->tma = build_maps<T>(e);
  PF_CUDA(e, cudaStreamSynchronize(e->stream));
  return PF_OK;
}

template <typename T>
StepArgs<T> step_args(pf_engine* e) {
  StepArgs<T> a;
  memset(&a, 0, sizeof a);
  a.nx = e->nx;
  a.ny = e->ny;
  a.nz = e->nz;
  a.pz = e->pz;
  a.dx = (T)e->dl[0];
  a.dy = (T)e->dl[1];
  a.dz = (T)e->dl[2];
  a.rdx = (T)e->rdl[0];
  a.rdy = (T)e->rdl[1];
  a.rdz = (T)e->rdl[2];
  a.fdx = e->fdiv[0];
  a.fdy = e->fdiv[1];
  a.fdz = e->fdiv[2];
  a.fdall = a.fdx && a.fdy && a.fdz;
  a.fdvec = e->vdiv;
  a.qtop = (T)e->qtop;
  a.qlow = e->qlow;
  a.ch = (T)e->ch;
  for (int ax = 0; ax < 3; ++ax) {
    a.hb0[ax] = e->hb0[ax];
    a.hb1[ax] = e->hb1[ax];
    a.eb0[ax] = e->eb0[ax];
    a.eb1[ax] = e->eb1[ax];
  }
  const int c0 = e->cur, c1 = e->fused ? e->cur ^ 1 : e->cur;
  for (int c = 0; c < 3; ++c) {
    a.Ein[c] = (const T*)e->E[c0][c];
    a.Hin[c] = (const T*)e->H[c0][c];
    a.Eout[c] = (T*)e->E[c1][c];
    a.Hout[c] = (T*)e->H[c1][c];
    a.ce[c] = (const T*)e->ce[c];
  }
  a.word = e->word;
  a.table = (const T*)e->table;
  a.adeword = e->adeword;
  for (int ax = 0; ax < 3; ++ax) {
    a.be[ax] = (const T*)e->cp[ax][0];
    a.cpe[ax] = (const T*)e->cp[ax][1];
    a.bh[ax] = (const T*)e->cp[ax][2];
    a.cph[ax] = (const T*)e->cp[ax][3];
    a.mape[ax] = e->map_e[ax];
    a.maph[ax] = e->map_h[ax];
    a.gze = e->gze;
    a.gzh = e->gzh;
    a.npe[ax] = e->npe[ax];
    a.nph[ax] = e->nph[ax];
  }
  for (int q = 0; q < 6; ++q) {
    a.psiE[q] = (T*)e->psiE[q];
    a.psiEin[q] = (const T*)e->psiE[q];
    a.psiHin[q] = (const T*)e->psiH[c0][q];
    a.psiHout[q] = (T*)e->psiH[c1][q];
  }
  a.media = (const MediumT<T>*)e->media;
  a.n_media = e->n_media;
  a.P = (T*)e->P;
  a.plev = e->plev;
  a.lvl = (int)(e->step & 1);
  a.wait_test = e->wait_test == 1;
  return a;
}

// Scans the six current fields for inf / nan (synchronous). H: where the H of
// a recorded step lies instead of the engine's own arrays.
int scan_finite(pf_engine* e, void* const H[3] = nullptr) {
  int* flag = e->flag;
  PF_CUDA(e, cudaMemsetAsync(flag, 0, sizeof(int), e->stream));
  for (int c = 0; c < 6; ++c) {
    const void* f = c < 3 ? e->E[e->cur][c] : (H ? H : e->H[e->cur])[c - 3];
    if (e->rb == 4)
      k_nonfinite<float><<<592, 256, 0, e->stream>>>((const float*)f, e->ncellp, flag);
    else
      k_nonfinite<double><<<592, 256, 0, e->stream>>>((const double*)f, e->ncellp, flag);
  }
  int h = 0;
  PF_CUDA(e, cudaMemcpyAsync(&h, flag, sizeof(int), cudaMemcpyDeviceToHost, e->stream));
  PF_CUDA(e, cudaStreamSynchronize(e->stream));
  return h ? fail(e, PF_ERR_NONFINITE, "non-finite field value at step %lld", e->step) : PF_OK;
}

// Launches a kernel that begins with pdl_enter behind the stream's last one,
// overlapping its launch with that one's tail: a step is three to six kernels
// of some microseconds, and each boundary cost two of them (per step: 128^3
// with monitors 81 -> 70 us, 160x152x144 double 152 -> 144, 256^3 298 -> 288).
template <typename... P, typename... A>
void launch_pdl(cudaStream_t st, dim3 grid, dim3 block, void (*kernel)(P...), A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.stream = st;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

// Vectors along z per block of the vector passes: 8 (128 bytes of a row) or,
// where that wastes more of the last block, 4; fewer on short rows. 256^3
// plain: 287 us at 8, 288 at 16, 330 at 32 (a warp that touches a layer at
// the end of a row takes 128 cells along); 301x287x263 406 at 8, 449 at 16.
int vec_lanes(int nzv) {
  if (nzv <= 2) return nzv;
  if (nzv <= 4) return 4;
  return (nzv + 7) / 8 * 8 > (nzv + 3) / 4 * 4 ? 4 : 8;
}

// Whether a dispersive 3D scene's E pass runs one cell per thread. The vector
// pass reads polarisation records as vectors where V cells of one medium have
// consecutive ranks from an aligned one on; other records it takes cell by
// cell, each cell's loads behind the stores of the one before, and a warp runs
// every kind that one of its lanes has. So the shares of warps with aligned
// runs of one pole (a1) and two (a2), other one-pole records (i1) and others of
// more poles (i2) decide, with weights fitted to the difference of the two
// forms' times over 36 scenes in float and 12 in double (blocks of 1 to 40 cells
// on rows of every remainder, boxes, spheres). us per step, vectors / cells:
// float aligned 8-cell blocks in 192^3 170 / 192, the same on 160 x 160 x 147 132 /
// 116, 246 x 257 x 269 570 / 474, 12-cell blocks on 160 x 160 x 163 130 / 135,
// one-pole sphere in 192^3 157 / 171, two-pole 190 / 182, single cells in 160^3
// 171 / 121; double 144^3 aligned blocks 160 / 150, one-pole sphere 128 / 136. Where the
// rule takes the slower form it loses 4% at most.
template <typename T>
int ade_by_cell(pf_engine* e) {
  e->ade_cells = false;
  if (!e->vec || e->fused || e->n_media == 0) return PF_OK;
  const uint32_t* word = e->ce_mode == PF_CE_TABLE ? e->word : e->adeword;
  unsigned long long* dev = nullptr;
  int rc = dalloc(e, (void**)&dev, 5 * sizeof *dev);
  if (rc) return rc;
  const int nzv = (e->nz + kVec<T> - 1) / kVec<T>;
  const dim3 b(vec_lanes(nzv), kVecThreads / vec_lanes(nzv));
  k_ade_runs<T><<<dim3((nzv + b.x - 1) / b.x, (e->ny + b.y - 1) / b.y, e->nx), b, 0, e->stream>>>(
      word, (const MediumT<T>*)e->media, e->ny, e->nz, e->pz, dev);
  PF_CUDA(e, cudaGetLastError());
  unsigned long long n[5];  // warps, a1, a2, i1, i2
  PF_CUDA(e, cudaMemcpyAsync(n, dev, sizeof n, cudaMemcpyDeviceToHost, e->stream));
  PF_CUDA(e, cudaStreamSynchronize(e->stream));
  const double a1 = (double)n[1], a2 = (double)n[2], i1 = (double)n[3], i2 = (double)n[4];
  e->ade_cells = sizeof(T) == 4 ? 2.25 * (a1 + a2) + 4.25 * i1 + 11.5 * i2 > 5.0 * (double)n[0]
                                : 1.4 * a1 + 21.0 * a2 + 8.0 * i1 + 12.0 * i2 > 5.6 * (double)n[0];
  return PF_OK;
}

// H and E passes over planes [i0, i1).
template <typename T>
void launch_h(pf_engine* e, const StepArgs<T>& a, int i0, int i1) {
  if (e->vec) {
    const int nzv = (e->nz + kVec<T> - 1) / kVec<T>;
    const dim3 b(vec_lanes(nzv), kVecThreads / vec_lanes(nzv));
    launch_pdl(e->stream, dim3((nzv + b.x - 1) / b.x, (e->ny + b.y - 1) / b.y, i1 - i0), b,
               sizeof(T) == 4 && e->vwide ? k_h_vec<T, sizeof(T) == 4> : k_h_vec<T, false>, a, i0);
    return;
  }
  const dim3 b = e->nz > 1 ? dim3(32, 8) : dim3(1, 256);
  launch_pdl(e->stream, dim3((e->nz + b.x - 1) / b.x, (e->ny + b.y - 1) / b.y, e->nx), b,
             k_h_split<T>, a);
}

template <typename T, int CE, bool ADE>
void launch_e_mode(pf_engine* e, const StepArgs<T>& a, int i0, int i1) {
  if constexpr (ADE) {
    if (e->ade_cells) {
      launch_pdl(e->stream, dim3((e->nz + 31) / 32, (e->ny + 7) / 8, e->nx), dim3(32, 8),
                 k_e_cell<T, CE>, a);
      return;
    }
  }
  if (e->vec) {
    const int nzv = (e->nz + kVec<T> - 1) / kVec<T>;
    const dim3 b(vec_lanes(nzv), kVecThreads / vec_lanes(nzv));
    launch_pdl(e->stream, dim3((nzv + b.x - 1) / b.x, (e->ny + b.y - 1) / b.y, i1 - i0), b,
               sizeof(T) == 4 && e->vwide ? k_e_vec<T, CE, ADE, sizeof(T) == 4>
                                        : k_e_vec<T, CE, ADE, false>, a, i0);
    return;
  }
  const dim3 b = e->nz > 1 ? dim3(32, 8) : dim3(1, 256);
  launch_pdl(e->stream, dim3((e->nz + b.x - 1) / b.x, (e->ny + b.y - 1) / b.y, e->nx), b,
             k_e_split<T, CE, ADE>, a);
}

template <typename T>
void launch_e(pf_engine* e, const StepArgs<T>& a, int i0, int i1) {
  const bool ade = e->n_media > 0;
  switch (e->ce_mode) {
    case PF_CE_CELL1:
      if (ade) launch_e_mode<T, kCeCell1, true>(e, a, i0, i1);
      else launch_e_mode<T, kCeCell1, false>(e, a, i0, i1);
      break;
    case PF_CE_CELL3:
      launch_e_mode<T, kCeCell3, false>(e, a, i0, i1);
      break;
    default:
      if (ade) launch_e_mode<T, kCeTable, true>(e, a, i0, i1);
      else launch_e_mode<T, kCeTable, false>(e, a, i0, i1);
  }
}

template <typename T>
Fields6<T> level_fields(pf_engine* e, int lvl) {
  Fields6<T> f;
  for (int c = 0; c < 3; ++c) {
    f.f[c] = (const T*)e->E[lvl][c];
    f.f[3 + c] = (const T*)e->H[lvl][c];
  }
  return f;
}

template <typename T>
int flush_monitors(pf_engine* e) {
  for (DftMon& m : e->dfts) {
    if (m.pending == 0) continue;
    const long long nt = m.r.ncell * m.r.ncomp;
    const int B = 128;
    LaunchScope ls(e, 3);
    launch_pdl(e->stream, (unsigned)((nt + B - 1) / B), B, k_dft_flush<T>,
        m.r, (const T*)m.ring, m.pending, m.acc, m.ph_e, m.ph_h, m.q_done, m.n_freq, m.dt);
    m.q_done += m.pending;
    m.pending = 0;
  }
  for (size_t q0 = 0; q0 < e->fluxes.size(); q0 += kFluxBatch) {
    FluxFold ff;
    memset(&ff, 0, sizeof ff);
    FluxKept<T> fk;
    memset(&fk, 0, sizeof fk);
    int n = 0, maxblk = 1, maxpend = 1;
    for (size_t q = q0; q < std::min(e->fluxes.size(), q0 + (size_t)kFluxBatch); ++q) {
      FluxMon& f = e->fluxes[q];
      if (f.pending == 0) continue;
      ff.partial[n] = f.partial;
      ff.nblk[n] = f.p.nblk;
      ff.pending[n] = f.pending;
      ff.acc[n] = f.acc;
      ff.dA[n] = f.dA;
      ff.dt[n] = f.dt;
      fk.val[n] = (const T*)f.val;
      fk.partial[n] = f.partial;
      fk.cells[n] = f.p.n0 * f.p.n1;
      fk.nblk[n] = f.p.nblk;
      fk.pending[n++] = f.pending;
      maxblk = std::max(maxblk, f.p.nblk);
      maxpend = std::max(maxpend, f.pending);
      f.pending = 0;
    }
    if (n == 0) continue;
    if (e->flux_kept) {
      LaunchScope ls(e, 3);
      launch_pdl(e->stream, dim3(maxblk, maxpend, n), 256, k_flux_groups<T>, fk);
    }
    LaunchScope ls(e, 3);
    launch_pdl(e->stream, n, 1024, k_flux_flush<T>, ff);
  }
  e->flux_kept = false;
  PF_CUDA(e, cudaGetLastError());
  return PF_OK;
}

// Monitors of step s read the level just written (E at t_e, H at t_h).
template <typename T>
int sample_monitors(pf_engine* e, long long s, int lvl) {
  if (e->dfts.empty() && e->fluxes.empty()) return PF_OK;
  const Fields6<T> f = level_fields<T>(e, lvl);
  for (DftMon& m : e->dfts) {
    if (s % m.interval) continue;
    if (m.pending == m.ring_cap) {
      int rc = flush_monitors<T>(e);
      if (rc) return rc;
    }
    const int B = 256;
    LaunchScope ls(e, 2);
    launch_pdl(e->stream, (unsigned)((m.r.ncell + B - 1) / B), B, k_dft_sample<T>,
        m.r, (T*)m.ring, m.pending, f, e->ny, e->pz);
    m.pending++;
  }
  // every flux plane samples every step: up to kFluxBatch planes per launch
  for (size_t q0 = 0; q0 < e->fluxes.size(); q0 += kFluxBatch) {
    const size_t q1 = std::min(e->fluxes.size(), q0 + (size_t)kFluxBatch);
    for (size_t q = q0; q < q1; ++q)
      if (e->fluxes[q].pending == e->fluxes[q].ring_cap) {
        int rc = flush_monitors<T>(e);
        if (rc) return rc;
        break;
      }
    FluxBatch fb;
    memset(&fb, 0, sizeof fb);
    int maxblk = 1;
    for (size_t q = q0; q < q1; ++q) {
      FluxMon& fl = e->fluxes[q];
      fb.p[q - q0] = fl.p;
      fb.partial[q - q0] = fl.partial;
      fb.slot[q - q0] = fl.pending;
      maxblk = std::max(maxblk, fl.p.nblk);
    }
    LaunchScope ls(e, 2);
    launch_pdl(e->stream, dim3(maxblk, (unsigned)(q1 - q0)), 256, k_flux_sample_batch<T>, fb, f,
               e->ny, e->pz);
    for (size_t q = q0; q < q1; ++q) e->fluxes[q].pending++;
  }
  return PF_OK;
}

template <typename T>
int inject(pf_engine* e, int fam, T* const F[3], long long s) {
  SourceGroups& d = e->src[fam].dev;
  if (d.n_groups == 0) return PF_OK;
  LaunchScope ls(e, 1);
  launch_pdl(e->stream, (d.n_groups + 127) / 128, 128, k_inject<T>, d, F[0], F[1], F[2], s);
  return PF_OK;
}

// A replay with the vector passes writes its record in place of the state: the
// H pass reads H from the last step's slot and writes this step's, the E pass
// psi_E likewise (the copies into the slot took as long as the H pass).
// Points the step's arguments at slots t - 1 (the engine's own state for t =
// 0) and t.
template <typename T>
void record_into(pf_engine* e, long long t, StepArgs<T>& a, T* Hout[3]) {
  char* at = e->rec + (size_t)t * e->rec_slot;
  const char* last = at - e->rec_slot;
  const size_t S = sizeof(T), n = (size_t)e->ncellp * S;
  size_t off = 0;
  for (int c = 0; c < 3; ++c, off += n) {
    if (t > 0) a.Hin[c] = (const T*)(last + off);
    a.Hout[c] = Hout[c] = (T*)(at + off);
  }
  for (int q = 0; q < 6; ++q) {
    if (t > 0) a.psiEin[q] = (const T*)(last + off);
    a.psiE[q] = (T*)(at + off);
    off += (size_t)e->npsiE[q] * S;
  }
}
// The engine's own state from the last slot of a replay.
int record_out(pf_engine* e, long long t) {
  const char* at = e->rec + (size_t)t * e->rec_slot;
  const size_t n = (size_t)e->ncellp * e->rb;
  for (int c = 0; c < 3; ++c, at += n)
    PF_CUDA(e, cudaMemcpyAsync(e->H[e->cur][c], at, n, cudaMemcpyDeviceToDevice, e->stream));
  for (int q = 0; q < 6; ++q) {
    const size_t b = (size_t)e->npsiE[q] * e->rb;
    if (b) PF_CUDA(e, cudaMemcpyAsync(e->psiE[q], at, b, cudaMemcpyDeviceToDevice, e->stream));
    at += b;
  }
  return PF_OK;
}

// An adjoint replay keeps, per step, H^{n+1/2} and psi_E after the step:
// what the reverse step needs to recompute the gradient's g = curl + psi.
template <typename T>
int record_step(pf_engine* e, long long t) {
  char* base = e->rec + (size_t)t * e->rec_slot;
  const bool direct = e->vec && !e->fused;  // record_into wrote them
  const size_t S = sizeof(T), n = (size_t)e->ncellp * S;
  size_t off = 0;
  for (int c = 0; c < 3 && !direct; ++c, off += n)
    PF_CUDA(e, cudaMemcpyAsync(base + off, e->H[e->cur][c], n, cudaMemcpyDeviceToDevice,
                               e->stream));
  for (int q = 0; q < 6 && !direct; ++q) {
    const size_t b = (size_t)e->npsiE[q] * S;
    if (b) PF_CUDA(e, cudaMemcpyAsync(base + off, e->psiE[q], b, cudaMemcpyDeviceToDevice, e->stream));
    off += b;
  }
  for (FluxMon& f : e->fluxes) {  // E planes of the flux monitors a loss depends on
    if (f.cot == 0.0) continue;
    if (t >= f.rec_cap) return fail(e, PF_ERR_STATE, "flux record slot out of range");
    const long long np = (long long)f.p.n0 * f.p.n1;
    launch_pdl(e->stream, (unsigned)((np + 255) / 256), 256, k_flux_plane_record<T>,
        f.p, (const T*)e->E[e->cur][0], (const T*)e->E[e->cur][1], (const T*)e->E[e->cur][2],
        (T*)f.rec + (size_t)t * 2 * np, e->ny, e->pz);
  }
  PF_CUDA(e, cudaGetLastError());
  return PF_OK;
}

// ---- small grids: runs of steps in one launch (kernels_resident.cuh) ----------
// Cells up to which resident launches beat separate ones (us per step,
// resident / separate): 2D float32 1000^2 33 / 41, 2000^2 127 / 133, float64
// 1500^2 116 / 122, 2000^2 202 / 200; 3D float32 72^3 18 / 28, 88^3 27 / 31,
// 96^3 33 / 33, float64 88^3 32 / 40, 96^3 43 / 41.
constexpr long long kResN2 = 3000000, kResN3 = 700000;

// Engines of this process inside pf_advance now. A cooperative grid takes the
// whole chip, so engines stepped concurrently (24 scenes of 40^3 to 96^3:
// 0.46 s with separate launches, 1.44 s with grids waiting for one another)
// launch their passes separately; one alone takes at most kResChunk steps per
// launch, so that another's arrival is noticed. One cluster never excludes
// other work. The route changes no result.
std::atomic<int> g_advancing{0};
struct Advancing {
  Advancing() { g_advancing.fetch_add(1); }
  ~Advancing() { g_advancing.fetch_sub(1); }
};
constexpr long long kResChunk = 512;

// Not a status of the ABI (those are 0 and below): this engine cannot have resident launches (a context
// with fewer SMs than the grid or cluster needs, or no memory for what they
// take besides). Nothing was launched or counted; its steps go on as separate
// launches.
constexpr int kResRefused = 1;

template <typename T, int CE, bool ADE, int MODE>
int launch_resident_as(pf_engine* e, const ResidentArgs<T>& g) {
  const auto fn = k_resident<T, CE, ADE, MODE>;
  const int thr = res_threads<T>(MODE);
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[1];
  cfg.blockDim = dim3(thr);
  cfg.stream = e->stream;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  const int want = (int)((e->ncell + thr - 1) / thr);
  if (MODE == kResCell1) {
    PF_CUDA(e, cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    int c = 1;  // a power of two up to 16
    while (c < 16 && c < want) c *= 2;
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = c;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(c);
  } else {
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cfg.gridDim = dim3(std::min(want, e->sms * res_blocks<T>(MODE)));
  }
  if (!e->res_asked) {  // once per engine: the launches of a run differ in nothing that counts
    int fit = 0;
    cudaError_t rc;
    if (MODE == kResCell1) {
      rc = cudaOccupancyMaxActiveClusters(&fit, fn, &cfg);
    } else {
      rc = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, fn, thr, 0);
      fit = fit * e->sms >= (int)cfg.gridDim.x;
    }
    if (rc != cudaSuccess || fit < 1 || e->wait_test == 2) {
      cudaGetLastError();
      return kResRefused;
    }
    e->res_asked = true;
  }
  if (MODE != kResCell1) PF_CUDA(e, cudaMemsetAsync(g.bar, 0, sizeof(unsigned), e->stream));
  const cudaError_t rc = cudaLaunchKernelEx(&cfg, fn, g);
  if (rc == cudaErrorCooperativeLaunchTooLarge || rc == cudaErrorInvalidClusterSize ||
      rc == cudaErrorLaunchOutOfResources || rc == cudaErrorNotSupported) {
    cudaGetLastError();
    return kResRefused;
  }
  PF_CUDA(e, rc);
  e->launches[0]++;
  return PF_OK;
}

template <typename T>
int resident_mode(const pf_engine* e) {
  if (e->ncell <= 16LL * res_threads<T>(kResCell1)) return kResCell1;
  if (e->ncell <= (long long)e->sms * res_blocks<T>(kResGrid1) * res_threads<T>(kResGrid1))
    return kResGrid1;
  return kResGridN;
}

template <typename T, int CE, bool ADE>
int launch_resident_mode(pf_engine* e, const ResidentArgs<T>& g) {
  switch (resident_mode<T>(e)) {
    case kResCell1: return launch_resident_as<T, CE, ADE, kResCell1>(e, g);
    case kResGrid1: return launch_resident_as<T, CE, ADE, kResGrid1>(e, g);
    default: return launch_resident_as<T, CE, ADE, kResGridN>(e, g);
  }
}

// Whether this engine is small enough for resident launches, and whether it
// takes them now.
template <typename T>
bool resident_small(const pf_engine* e) {
  const bool d3 = e->nx > 1 && e->ny > 1 && e->nz > 1;
  return !e->fused && e->ncell <= (d3 ? kResN3 : kResN2) && e->dfts.size() <= (size_t)kResDft &&
         e->fluxes.size() <= (size_t)kFluxBatch;
}
template <typename T>
bool resident_ok(const pf_engine* e) {
  return resident_small<T>(e) && !e->recording && !e->profiling && !e->res_off &&
         (g_advancing.load() == 1 || resident_mode<T>(e) == kResCell1);
}

// Up to n steps in one launch: as many as the sample rings have room for.
// Returns the steps taken in *took; the caller flushes full rings first.
template <typename T>
int launch_resident(pf_engine* e, long long n, long long* took) {
  const long long s = e->step;
  auto due = [&](const DftMon& m) { return (s + m.interval - 1) / m.interval * m.interval; };
  for (const DftMon& m : e->dfts)
    n = std::min(n, due(m) + (long long)(m.ring_cap - m.pending) * m.interval - s);
  for (const FluxMon& f : e->fluxes) n = std::min<long long>(n, f.ring_cap - f.pending);
  ResidentArgs<T> g;
  memset(&g, 0, sizeof g);
  g.a = step_args<T>(e);
  g.src[0] = e->src[0].dev;
  g.src[1] = e->src[1].dev;
  g.step0 = s;
  g.n = (int)n;
  for (DftMon& m : e->dfts) {
    const int q = g.n_dft++;
    g.dft[q] = m.r;
    g.dft_ring[q] = (T*)m.ring;
    g.dft_slot[q] = m.pending;
    g.dft_interval[q] = m.interval;
  }
  for (FluxMon& f : e->fluxes) {
    const int q = g.n_flux++;
    if (!f.val && dalloc(e, &f.val, (size_t)f.ring_cap * f.p.n0 * f.p.n1 * sizeof(T)))
      return kResRefused;
    g.flux[q] = f.p;
    g.flux_val[q] = (T*)f.val;
    g.flux_slot[q] = f.pending;
  }
  if (!e->res_bar && dalloc(e, (void**)&e->res_bar, sizeof(unsigned))) return kResRefused;
  if (!e->res_err.p) e->res_err = err_word(e->device, e->stream);
  if (!e->res_err.p) return kResRefused;
  g.bar = e->res_bar;
  g.spin = e->wait_test == 1 ? kResSpinTest : kResSpin;
  g.phase0 = e->wait_test == 1 ? 1u << 30 : 0u;
  PF_CUDA(e, cudaHostGetDevicePointer((void**)&g.err, e->res_err.p, 0));
  const bool ade = e->n_media > 0;
  int rc;
  switch (e->ce_mode) {
    case PF_CE_CELL1:
      rc = ade ? launch_resident_mode<T, kCeCell1, true>(e, g)
               : launch_resident_mode<T, kCeCell1, false>(e, g);
      break;
    case PF_CE_CELL3:
      rc = launch_resident_mode<T, kCeCell3, false>(e, g);
      break;
    default:
      rc = ade ? launch_resident_mode<T, kCeTable, true>(e, g)
               : launch_resident_mode<T, kCeTable, false>(e, g);
  }
  if (rc) return rc;
  for (DftMon& m : e->dfts)
    if (due(m) < s + n) m.pending += (int)((s + n - 1 - due(m)) / m.interval + 1);
  for (FluxMon& f : e->fluxes) f.pending += (int)n;
  e->flux_kept = !e->fluxes.empty();
  *took = n;
  e->step += n;
  return PF_OK;
}

// Resident launches for up to n steps (at most kResChunk); *took: steps taken,
// fewer if a launch was refused.
template <typename T>
int advance_resident(pf_engine* e, long long n, long long* took) {
  *took = 0;
  n = std::min(n, kResChunk);
  while (*took < n) {
    bool full = false;
    for (const DftMon& m : e->dfts) full = full || m.pending == m.ring_cap;
    for (const FluxMon& f : e->fluxes) full = full || f.pending == f.ring_cap;
    int rc;
    if (full && (rc = flush_monitors<T>(e))) return rc;
    long long k = n - *took;
    if (e->check_every > 0) k = std::min(k, e->check_every - e->step % e->check_every);
    rc = launch_resident<T>(e, k, &k);
    if (rc == kResRefused) {
      e->res_off = true;
      return PF_OK;
    }
    if (rc) return rc;
    *took += k;
    if (e->check_every > 0 && e->step % e->check_every == 0) {
      PF_CUDA(e, cudaGetLastError());
      if ((rc = scan_finite(e))) return rc;
    }
  }
  return PF_OK;
}

// One launch per pass.
template <typename T>
int advance_separate(pf_engine* e, long long n_sub) {
  for (long long t = 0; t < n_sub; ++t) {
    const long long s = e->step;
    // the split passes update in place: a cell's pass reads only its own old
    // value and the other family's fields
    const int nxt = e->fused ? e->cur ^ 1 : e->cur;
    StepArgs<T> a = step_args<T>(e);
    void* H[3] = {a.Hout[0], a.Hout[1], a.Hout[2]};
    if (e->fused) {
      int rc;
      {
        LaunchScope ls(e, 0);
        if (e->tma)
          rc = launch_tma<T>(e->stream, a, e->maps, e->cur, e->ce_mode, e->n_media > 0,
                             e->fused_chunks, e->tma_err);
        else
          rc = launch_fused<T>(e->stream, a, e->ce_mode, e->n_media > 0, e->fused_ty,
                               e->fused_chunks);
      }
      if (rc) return fail(e, PF_ERR_UNSUPPORTED, "fused kernel does not cover this case");
      // sources of the fused path are injected after its single pass: an H
      // source must reach the E update, so the fused path is only chosen
      // when there are no H-family sources.
      T* Eout[3] = {a.Eout[0], a.Eout[1], a.Eout[2]};
      inject<T>(e, 0, Eout, s);
    } else {
      T* Hout[3] = {a.Hout[0], a.Hout[1], a.Hout[2]};
      if (e->recording) {
        const long long slot = s - e->rec_step0;
        if (slot < 0 || slot >= e->ring_steps)
          return fail(e, PF_ERR_STATE, "record slot out of range");
        if (e->vec) record_into<T>(e, slot, a, Hout);
        for (int c = 0; c < 3; ++c) H[c] = Hout[c];
      }
      {
        LaunchScope ls(e, 0);
        launch_h<T>(e, a, 0, e->nx);
      }
      inject<T>(e, 1, Hout, s);
      a.Hin[0] = a.Hout[0];
      a.Hin[1] = a.Hout[1];
      a.Hin[2] = a.Hout[2];
      {
        LaunchScope ls(e, 0);
        launch_e<T>(e, a, 0, e->nx);
      }
      T* Eout[3] = {a.Eout[0], a.Eout[1], a.Eout[2]};
      inject<T>(e, 0, Eout, s);
    }
    int rc = e->recording ? PF_OK : sample_monitors<T>(e, s, nxt);
    if (rc) return rc;
    e->cur = nxt;
    e->step++;
    if (e->recording && (rc = record_step<T>(e, s - e->rec_step0))) return rc;
    if (e->check_every > 0 && e->step % e->check_every == 0) {
      PF_CUDA(e, cudaGetLastError());
      if ((rc = scan_finite(e, H))) {
        collect_profile(e);
        return rc;
      }
    }
  }
  return PF_OK;
}

template <typename T>
int advance_typed(pf_engine* e, long long n_sub) {
  Advancing guard;
  long long left = n_sub;
  while (left > 0) {
    const bool res = resident_ok<T>(e);
    // pending flux samples are either kept values or partials, not both
    for (const FluxMon& f : e->fluxes)
      if (f.pending && e->flux_kept != res && !e->recording) {
        int rc = flush_monitors<T>(e);
        if (rc) return rc;
        break;
      }
    long long took = 0;
    int rc;
    if (res) {
      rc = advance_resident<T>(e, left, &took);
      // queued launches must not hide another engine's arrival
      if (!rc && left > took) PF_CUDA(e, cudaStreamSynchronize(e->stream));
    } else {
      took = resident_small<T>(e) ? std::min<long long>(left, kResChunk) : left;
      rc = advance_separate<T>(e, took);
    }
    if (rc) return rc;
    left -= took;
  }
  PF_CUDA(e, cudaGetLastError());
  PF_CUDA(e, cudaStreamSynchronize(e->stream));
  collect_profile(e);
  if (e->tma) {
    int h = 0;
    PF_CUDA(e, cudaMemcpy(&h, e->tma_err, sizeof(int), cudaMemcpyDeviceToHost));
    if (h == 2) return fail(e, PF_ERR_CUDA, "TMA staging buffer misaligned; results are invalid");
    if (h) return fail(e, PF_ERR_TIMEOUT, "a TMA stage wait timed out; results are invalid");
  }
  if (e->res_err.p && *(volatile int*)e->res_err.p)
    return fail(e, PF_ERR_TIMEOUT, "a grid barrier timed out; results are invalid");
  return PF_OK;
}

bool valid_comp(int c) { return c >= 0 && c < 6; }

}  // namespace

namespace pfb {
namespace {
struct DeviceKeep {
  unsigned long long ctx = 0;  // id of the context that the rest belongs to
  cudaMemPool_t pool = nullptr;
  std::vector<int*> err_free;
};
std::mutex g_keep_mu;
std::map<int, DeviceKeep> g_keep;  // per device

// Id of a live stream's context, 0 if the driver does not tell.
unsigned long long context_id(cudaStream_t st) {
  typedef CUresult (*StreamCtxFn)(CUstream, CUcontext*);
  typedef CUresult (*CtxIdFn)(CUcontext, unsigned long long*);
  static const auto entry = [](const char* name) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    // by version: later forms of cuStreamGetCtx take another argument
    const bool ok = cudaGetDriverEntryPointByVersion(name, &p, 12000, cudaEnableDefault, &q) ==
                        cudaSuccess && q == cudaDriverEntryPointSuccess;
    return ok ? p : nullptr;
  };
  static const auto stream_ctx = (StreamCtxFn)entry("cuStreamGetCtx");
  static const auto ctx_id = (CtxIdFn)entry("cuCtxGetId");
  CUcontext c = nullptr;
  unsigned long long id = 0;
  if (!stream_ctx || !ctx_id || stream_ctx((CUstream)st, &c) != CUDA_SUCCESS ||
      ctx_id(c, &id) != CUDA_SUCCESS)
    return 0;
  return id;
}

// What is kept for the context (g_keep_mu held); that of an earlier context
// of the device is dropped.
DeviceKeep* keep_of(int dev, unsigned long long ctx) {
  if (!ctx) return nullptr;
  DeviceKeep& k = g_keep[dev];
  if (k.ctx != ctx) {
    k = DeviceKeep{};
    k.ctx = ctx;
  }
  return &k;
}

cudaMemPool_t device_pool(int dev, cudaStream_t st) {
  std::lock_guard<std::mutex> lk(g_keep_mu);
  DeviceKeep* k = keep_of(dev, context_id(st));
  if (!k || k->pool) return k ? k->pool : nullptr;
  cudaMemPoolProps props = {};
  props.allocType = cudaMemAllocationTypePinned;
  props.location.type = cudaMemLocationTypeDevice;
  props.location.id = dev;
  cudaMemPool_t pool = nullptr;
  if (cudaMemPoolCreate(&pool, &props) != cudaSuccess) {
    cudaGetLastError();
    return nullptr;
  }
  unsigned long long keep = kPoolKeep;
  cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
  k->pool = pool;
  return pool;
}
}  // namespace

ErrWord err_word(int dev, cudaStream_t st) {
  std::lock_guard<std::mutex> lk(g_keep_mu);
  DeviceKeep* k = keep_of(dev, context_id(st));
  if (!k) return {};
  if (k->err_free.empty()) {
    int* page = nullptr;
    if (cudaHostAlloc((void**)&page, 4096, cudaHostAllocMapped | cudaHostAllocPortable) !=
        cudaSuccess) {
      cudaGetLastError();
      return {};
    }
    for (int q = 0; q < 1024; ++q) k->err_free.push_back(page + q);
  }
  ErrWord w{k->err_free.back(), k->ctx};
  k->err_free.pop_back();
  *w.p = 0;
  return w;
}

void err_word_release(int dev, const ErrWord& w) {
  std::lock_guard<std::mutex> lk(g_keep_mu);
  const auto it = g_keep.find(dev);
  if (w.p && it != g_keep.end() && it->second.ctx == w.ctx) it->second.err_free.push_back(w.p);
}

void pool_trim() {
  int dev = 0;
  std::lock_guard<std::mutex> lk(g_keep_mu);
  if (g_keep.empty() || cudaGetDevice(&dev) != cudaSuccess) return;
  const auto it = g_keep.find(dev);
  // the null stream's context is the current one
  if (it != g_keep.end() && it->second.pool && it->second.ctx == context_id(nullptr))
    cudaMemPoolTrimTo(it->second.pool, 0);
}

cudaError_t malloc_trim(void** p, size_t bytes) {
  cudaError_t rc = cudaMalloc(p, bytes);
  if (rc != cudaErrorMemoryAllocation) return rc;
  cudaGetLastError();
  pool_trim();
  return cudaMalloc(p, bytes);
}

cudaError_t pool_alloc(void** p, size_t bytes, int dev, cudaStream_t st) {
  *p = nullptr;
  cudaMemPool_t pool = device_pool(dev, st);
  cudaError_t rc = pool ? cudaMallocFromPoolAsync(p, bytes, pool, st) : cudaErrorMemoryAllocation;
  if (rc == cudaErrorMemoryAllocation && pool) {
    cudaGetLastError();
    // freed blocks that the pool still holds may be what is missing
    cudaStreamSynchronize(st);
    cudaMemPoolTrimTo(pool, 0);
    rc = cudaMallocFromPoolAsync(p, bytes, pool, st);
  }
  if (rc != cudaSuccess) {
    cudaGetLastError();
    *p = nullptr;
  }
  return rc;
}

void pool_free(void* p, cudaStream_t st) {
  if (p) cudaFreeAsync(p, st);
}

bool host_recip_division_exact(float d) { return recip_division_exact(d); }
bool host_recip_division_exact(double d) { return recip_division_exact(d); }
}  // namespace pfb

// ===========================================================================
// C ABI
// ===========================================================================
extern "C" {

const char* pf_version(void) { return "pfb200 0.1.0 sm_100a"; }

const char* pf_last_error(const pf_engine* e) {
  return e ? e->err.c_str() : g_create_error.c_str();
}

int pf_create(int nx, int ny, int nz, int real_bytes, double dx, double dy, double dz, double ch,
              int64_t n_steps, pf_engine** out) {
  if (!out) return fail(nullptr, PF_ERR_INVALID, "out is NULL");
  *out = nullptr;
  if (nx < 1 || ny < 1 || nz < 1)
    return fail(nullptr, PF_ERR_INVALID, "grid shape must be positive, got %d x %d x %d", nx, ny, nz);
  if (real_bytes != 4 && real_bytes != 8)
    return fail(nullptr, PF_ERR_INVALID, "real_bytes must be 4 or 8, got %d", real_bytes);
  if (n_steps < 0) return fail(nullptr, PF_ERR_INVALID, "n_steps must be >= 0");
  if ((long long)nx * ny * nz > 0x7fffffffLL)
    return fail(nullptr, PF_ERR_UNSUPPORTED, "more than 2^31-1 cells");
  if (!(dx > 0 && dy > 0 && dz > 0)) return fail(nullptr, PF_ERR_INVALID, "spacings must be > 0");
  pf_engine* e = new pf_engine();
  e->nx = nx;
  e->ny = ny;
  e->nz = nz;
  e->rb = real_bytes;
  e->dl[0] = dx;
  e->dl[1] = dy;
  e->dl[2] = dz;
  e->ch = ch;
  e->n_steps = n_steps;
  e->ncell = (long long)nx * ny * nz;
  // rows padded to 32 bytes, those under 128 bytes to 16 (a row of four floats
  // would take twice its memory; 1100 x 1100 x 4 124 -> 89 us per step, 800 x 800
  // x 9 184 -> 172, 600 x 600 x 17 190 -> 186), unless that takes a grid past 2^31
  // cells
  const int unit = (nz * real_bytes < 128 ? 16 : 32) / real_bytes;
  e->pz = nz > 1 ? (nz + unit - 1) / unit * unit : 1;
  if ((long long)nx * ny * e->pz > 0x7fffffffLL) e->pz = nz;
  e->ncellp = (long long)nx * ny * e->pz;
  e->vec = nx > 1 && ny > 1 && nz > 1 && e->pz % (16 / real_bytes) == 0;
  cudaError_t rc = cudaGetDevice(&e->device);
  if (rc == cudaSuccess)
    rc = cudaDeviceGetAttribute(&e->sms, cudaDevAttrMultiProcessorCount, e->device);
  if (rc == cudaSuccess) rc = cudaStreamCreateWithFlags(&e->stream, cudaStreamNonBlocking);
  if (rc != cudaSuccess) {
    fail(nullptr, PF_ERR_CUDA, "CUDA error: %s", cudaGetErrorString(rc));
    delete e;
    return PF_ERR_CUDA;
  }
  *out = e;
  return PF_OK;
}

int pf_set_ce(pf_engine* e, int mode, const void* ce0, const void* ce1, const void* ce2,
              const uint32_t* word, int n_table, const double* table) {
  if (!e) return PF_ERR_INVALID;
  if (e->finalized) return fail(e, PF_ERR_STATE, "pf_set_ce after pf_finalize");
  const size_t bytes = (size_t)e->ncell * e->rb;
  for (int c = 0; c < 3; ++c) e->h_ce[c].clear();
  e->h_table.clear();
  if (mode == PF_CE_CELL1) {
    if (!ce0) return fail(e, PF_ERR_INVALID, "PF_CE_CELL1 needs ce0");
    e->h_ce[0].assign((const char*)ce0, (const char*)ce0 + bytes);
  } else if (mode == PF_CE_CELL3) {
    if (!ce0 || !ce1 || !ce2) return fail(e, PF_ERR_INVALID, "PF_CE_CELL3 needs three arrays");
    const void* src[3] = {ce0, ce1, ce2};
    for (int c = 0; c < 3; ++c) e->h_ce[c].assign((const char*)src[c], (const char*)src[c] + bytes);
  } else if (mode == PF_CE_TABLE) {
    if (!word || n_table < 1 || !table) return fail(e, PF_ERR_INVALID, "PF_CE_TABLE needs word and table");
    // one pass: plain words index the table; per medium, the largest record
    // index its dispersive words name (checked against its cell count at
    // pf_finalize). The word then goes to the device straight from the
    // caller's buffer, with no host copy.
    long long need[kMaxMedia] = {};
    for (long long q = 0; q < e->ncell; ++q) {
      const uint32_t w = word[q];
      if (w & kDispersiveBit) {
        const int m = (int)((w >> kMediumShift) & 15u);
        need[m] = std::max(need[m], (long long)(w & kLocMask) + 1);
      } else if (w >= (uint32_t)n_table) {
        return fail(e, PF_ERR_INVALID, "ce word %u at cell %lld exceeds table size %d", w, q, n_table);
      }
    }
    PF_CUDA(e, cudaSetDevice(e->device));
    int rc;
    if (!e->word && (rc = dalloc(e, (void**)&e->word, (size_t)e->ncellp * 4))) return rc;
    if ((rc = copy_rows(e, e->word, const_cast<uint32_t*>(word), (size_t)e->nx * e->ny, 4, true)))
      return rc;
    PF_CUDA(e, cudaStreamSynchronize(e->stream));
    memcpy(e->word_need, need, sizeof need);
    e->h_table.assign(table, table + n_table);
  } else {
    return fail(e, PF_ERR_INVALID, "unknown ce mode %d", mode);
  }
  e->ce_mode = mode;
  return PF_OK;
}

int pf_set_cpml(pf_engine* e, int axis, const void* b_e, const void* c_e, const void* b_h,
                const void* c_h) {
  if (!e) return PF_ERR_INVALID;
  if (e->finalized) return fail(e, PF_ERR_STATE, "pf_set_cpml after pf_finalize");
  if (axis < 0 || axis > 2) return fail(e, PF_ERR_INVALID, "axis must be 0..2");
  const int dims[3] = {e->nx, e->ny, e->nz};
  const size_t bytes = (size_t)dims[axis] * e->rb;
  const void* src[4] = {b_e, c_e, b_h, c_h};
  for (int q = 0; q < 4; ++q) {
    e->h_cpml[axis][q].clear();
    if (src[q]) e->h_cpml[axis][q].assign((const char*)src[q], (const char*)src[q] + bytes);
  }
  return PF_OK;
}

int pf_set_ade(pf_engine* e, int n_media, const int64_t* count, const int32_t* npole,
               const double* coef, const double* inv_eps, const double* ce_m,
               const uint32_t* cell_word) {
  if (!e) return PF_ERR_INVALID;
  if (e->finalized) return fail(e, PF_ERR_STATE, "pf_set_ade after pf_finalize");
  if (n_media < 0 || n_media > kMaxMedia)
    return fail(e, PF_ERR_UNSUPPORTED, "at most %d dispersive media, got %d", kMaxMedia, n_media);
  e->n_media = n_media;
  e->m_count.assign(count, count + n_media);
  e->m_npole.assign(npole, npole + n_media);
  long long ncoef = 0;
  for (int m = 0; m < n_media; ++m) {
    if (npole[m] < 0 || npole[m] > kMaxPoles)
      return fail(e, PF_ERR_UNSUPPORTED, "at most %d poles per medium, got %d", kMaxPoles, npole[m]);
    if (count[m] < 0 || count[m] > (long long)kLocMask + 1)
      return fail(e, PF_ERR_UNSUPPORTED, "at most 2^%d cells per dispersive medium", kMediumShift);
    ncoef += 3LL * npole[m];
  }
  e->m_coef.assign(coef, coef + ncoef);
  e->m_inv.assign(inv_eps, inv_eps + n_media);
  e->m_ce.clear();
  if (ce_m) e->m_ce.assign(ce_m, ce_m + n_media);
  e->h_adeword.clear();
  if (cell_word) {
    for (long long q = 0; q < e->ncell; ++q) {
      const uint32_t w = cell_word[q];
      if (w && (!(w & kDispersiveBit) || (int)((w >> kMediumShift) & 15u) >= n_media ||
                (long long)(w & kLocMask) >= count[(w >> kMediumShift) & 15u]))
        return fail(e, PF_ERR_INVALID, "bad dispersive word 0x%08x at cell %lld", w, q);
    }
    e->h_adeword.assign(cell_word, cell_word + e->ncell);
  }
  return PF_OK;
}

int pf_rank_dispersive_words(uint32_t* word, int64_t n, int n_media, int64_t* counts,
                             int clear_plain) {
  if (!word || !counts || n < 0) return fail(nullptr, PF_ERR_INVALID, "NULL word or counts");
  if (n_media < 0 || n_media > kMaxMedia)
    return fail(nullptr, PF_ERR_UNSUPPORTED, "at most %d dispersive media, got %d", kMaxMedia,
                n_media);
  long long cnt[kMaxMedia] = {0};
  for (long long q = 0; q < n; ++q) {
    const uint32_t w = word[q];
    if (!(w & kDispersiveBit)) {
      if (clear_plain) word[q] = 0u;
      continue;
    }
    const int m = (int)((w >> kMediumShift) & 15u);
    if (m >= n_media || (w & kLocMask))
      return fail(nullptr, PF_ERR_INVALID, "bad dispersive word 0x%08x at cell %lld", w, q);
    if (cnt[m] > (long long)kLocMask)
      return fail(nullptr, PF_ERR_UNSUPPORTED, "more than 2^%d cells in one dispersive medium",
                  kMediumShift);
    word[q] = w | (uint32_t)cnt[m]++;
  }
  for (int m = 0; m < n_media; ++m) counts[m] = cnt[m];
  return PF_OK;
}

int pf_set_sources(pf_engine* e, int n_src, const int32_t* comp, const int64_t* cell,
                   const int32_t* wave_row, const double* amp, int n_wave, const double* wave) {
  if (!e) return PF_ERR_INVALID;
  if (e->finalized) return fail(e, PF_ERR_STATE, "pf_set_sources after pf_finalize");
  for (int f = 0; f < 2; ++f) e->src[f] = SrcFamily();
  e->n_wave = n_wave;
  e->h_wave.assign(wave, wave + (size_t)n_wave * e->n_steps);
  // group by (component, cell), keeping list order inside each group
  for (int f = 0; f < 2; ++f) {
    SrcFamily& s = e->src[f];
    std::vector<std::pair<long long, int>> key;  // (comp*ncell + cell, source)
    for (int q = 0; q < n_src; ++q) {
      if (!valid_comp(comp[q])) return fail(e, PF_ERR_INVALID, "source %d: bad component %d", q, comp[q]);
      if (cell[q] < 0 || cell[q] >= e->ncell) return fail(e, PF_ERR_INVALID, "source %d: cell out of range", q);
      if (wave_row[q] < 0 || wave_row[q] >= n_wave) return fail(e, PF_ERR_INVALID, "source %d: bad waveform row", q);
      if ((comp[q] >= 3) != (f == 1)) continue;
      key.push_back({(long long)(comp[q] % 3) * e->ncell + cell[q], q});
    }
    std::stable_sort(key.begin(), key.end(),
                     [](const std::pair<long long, int>& x, const std::pair<long long, int>& y) {
                       return x.first < y.first;
                     });
    for (size_t q = 0; q < key.size(); ++q) {
      if (q == 0 || key[q].first != key[q - 1].first) {
        s.cell.push_back(key[q].first % e->ncell);
        s.comp.push_back((int)(key[q].first / e->ncell));
        s.start.push_back((int)s.wave_row.size());
      }
      s.wave_row.push_back(wave_row[key[q].second]);
      s.amp.push_back(amp[key[q].second]);
    }
    s.start.push_back((int)s.wave_row.size());
  }
  return PF_OK;
}

int pf_add_dft(pf_engine* e, const int32_t start[3], const int32_t stop[3], const int32_t stride[3],
               int comp_mask, int n_freq, int interval, const double* phase_e,
               const double* phase_h, double dt, int* mon) {
  if (!e) return PF_ERR_INVALID;
  if (e->finalized) return fail(e, PF_ERR_STATE, "pf_add_dft after pf_finalize");
  if (n_freq < 1 || interval < 1 || !(comp_mask & 63) || !phase_e || !phase_h)
    return fail(e, PF_ERR_INVALID, "bad DFT monitor arguments");
  const int dims[3] = {e->nx, e->ny, e->nz};
  DftMon m;
  m.r.ncell = 1;
  for (int a = 0; a < 3; ++a) {
    if (start[a] < 0 || stop[a] > dims[a] || stop[a] <= start[a] || stride[a] < 1)
      return fail(e, PF_ERR_INVALID, "bad DFT region on axis %d", a);
    m.r.start[a] = start[a];
    m.r.stride[a] = stride[a];
    m.r.count[a] = (stop[a] - start[a] + stride[a] - 1) / stride[a];
    m.r.ncell *= m.r.count[a];
  }
  m.r.ncomp = 0;
  for (int c = 0; c < 6; ++c)
    if (comp_mask & (1 << c)) m.r.comps[m.r.ncomp++] = c;
  m.n_freq = n_freq;
  m.interval = interval;
  m.dt = dt;
  m.n_samples = e->n_steps > 0 ? (e->n_steps + interval - 1) / interval : 0;
  m.h_ph_e.assign(phase_e, phase_e + m.n_samples * n_freq * 2);
  m.h_ph_h.assign(phase_h, phase_h + m.n_samples * n_freq * 2);
  e->dfts.push_back(std::move(m));
  if (mon) *mon = (int)e->dfts.size() - 1;
  return PF_OK;
}

int pf_add_flux(pf_engine* e, int axis, int idx, double dA, double dt, int* mon) {
  if (!e) return PF_ERR_INVALID;
  if (e->finalized) return fail(e, PF_ERR_STATE, "pf_add_flux after pf_finalize");
  const int dims[3] = {e->nx, e->ny, e->nz};
  if (axis < 0 || axis > 2 || idx < 0 || idx >= dims[axis])
    return fail(e, PF_ERR_INVALID, "bad flux plane (axis %d, index %d)", axis, idx);
  FluxMon f;
  f.p.axis = axis;
  f.p.idx = idx;
  f.p.n0 = axis == 0 ? e->ny : e->nx;
  f.p.n1 = axis == 2 ? e->ny : e->nz;
  f.p.nblk = (int)(((long long)f.p.n0 * f.p.n1 + 255) / 256);
  f.dA = dA;
  f.dt = dt;
  e->fluxes.push_back(f);
  if (mon) *mon = (int)e->fluxes.size() - 1;
  return PF_OK;
}

int pf_set_kernel(pf_engine* e, int kernel) {
  if (!e) return PF_ERR_INVALID;
  if (e->finalized) return fail(e, PF_ERR_STATE, "pf_set_kernel after pf_finalize");
  if (kernel < PF_KERNEL_AUTO || kernel > PF_KERNEL_FUSED)
    return fail(e, PF_ERR_INVALID, "unknown kernel %d", kernel);
  e->kernel = kernel;
  return PF_OK;
}

int pf_finalize(pf_engine* e) {
  if (!e) return PF_ERR_INVALID;
  if (e->finalized) return fail(e, PF_ERR_STATE, "pf_finalize called twice");
  if (e->ce_mode < 0) return fail(e, PF_ERR_INVALID, "pf_set_ce was not called");
  if (e->n_media > 0 && e->ce_mode == PF_CE_CELL3)
    return fail(e, PF_ERR_UNSUPPORTED, "dispersive media with a three-component coefficient");
  if (e->n_media > 0 && e->ce_mode == PF_CE_CELL1 && e->h_adeword.size() != (size_t)e->ncell)
    return fail(e, PF_ERR_INVALID, "PF_CE_CELL1 with dispersive media needs cell_word");
  if (e->ce_mode == PF_CE_TABLE)
    for (int m = 0; m < kMaxMedia; ++m)
      if (e->word_need[m] > 0 && (m >= e->n_media || e->word_need[m] > e->m_count[m]))
        return fail(e, PF_ERR_INVALID,
                    "bad dispersive word: medium %d record %lld, but the medium has %lld cells", m,
                    e->word_need[m] - 1, m < e->n_media ? e->m_count[m] : 0LL);
  const bool has_h_src = !e->src[1].cell.empty();
  const bool fusable = fused_supported(e->nx, e->ny, e->nz) && !has_h_src;
  if (e->kernel == PF_KERNEL_FUSED && !fusable)
    return fail(e, PF_ERR_UNSUPPORTED, "the fused kernel needs a 3D grid without H-family sources");
  // AUTO takes the split passes: on B200 they currently outrun the fused
  // kernel (measured: config-3 384^3 2.05 vs 2.54 ms/step), whose plane loop
  // is latency-bound. PF_KERNEL_FUSED selects it explicitly.
  e->fused = e->kernel == PF_KERNEL_FUSED;
  (void)fusable;
  if (e->fused) {
    if (const char* v = getenv("PFB200_FUSED_TY")) e->fused_ty = atoi(v) == 16 ? 16 : 8;
    const long long tiles = (long long)((e->nz + 31) / 32) * ((e->ny + e->fused_ty - 1) / e->fused_ty);
    // about one resident wave of blocks (148 SMs x 1024 threads), at least
    // 8 planes per chunk
    int nch = (int)std::max<long long>(1, (148LL * 1024 / (32 * e->fused_ty) + tiles / 2) / tiles);
    nch = std::max(nch, (e->nx + 11) / 12);  // short chunks hide the plane-loop latency
    nch = std::min(nch, std::max(1, e->nx / 8));
    if (const char* v = getenv("PFB200_XCHUNKS")) nch = std::max(1, atoi(v));
    e->fused_chunks = nch;
  }
  {
    const int dims[3] = {e->nx, e->ny, e->nz};
    for (int ax = 0; ax < 3; ++ax) {
      const double d = e->rb == 4 ? (double)(float)e->dl[ax] : e->dl[ax];
      e->rdl[ax] = e->rb == 4 ? (double)(1.0f / (float)d) : 1.0 / d;
      if (dims[ax] > 1 && !getenv("PFB200_IEEE_DIV"))
        e->fdiv[ax] = e->rb == 4 ? recip_division_exact((float)d) : recip_division_exact(d);
    }
  }
  int rc = e->rb == 4 ? finalize_typed<float>(e) : finalize_typed<double>(e);
  if (!rc) rc = vector_division(e);
  if (!rc) rc = e->rb == 4 ? ade_by_cell<float>(e) : ade_by_cell<double>(e);
  if (rc) return rc;
  // host staging no longer needed
  for (int c = 0; c < 3; ++c) std::vector<char>().swap(e->h_ce[c]);
  std::vector<uint32_t>().swap(e->h_adeword);
  e->finalized = true;
  return PF_OK;
}

int pf_advance(pf_engine* e, int64_t step0, int64_t n_sub) {
  if (!e) return PF_ERR_INVALID;
  if (!e->finalized) return fail(e, PF_ERR_STATE, "pf_advance before pf_finalize");
  if (step0 != e->step)
    return fail(e, PF_ERR_INVALID, "pf_advance(step0=%lld) but the engine is at step %lld",
                (long long)step0, e->step);
  if (n_sub < 0 || e->step + n_sub > e->n_steps)
    return fail(e, PF_ERR_INVALID, "advance past n_steps (%lld)", e->n_steps);
  PF_CUDA(e, cudaSetDevice(e->device));
  return e->rb == 4 ? advance_typed<float>(e, n_sub) : advance_typed<double>(e, n_sub);
}

int pf_read_field(pf_engine* e, int comp, void* dst) {
  if (!e || !dst) return PF_ERR_INVALID;
  if (!e->finalized) return fail(e, PF_ERR_STATE, "pf_read_field before pf_finalize");
  if (!valid_comp(comp)) return fail(e, PF_ERR_INVALID, "bad component %d", comp);
  PF_CUDA(e, cudaSetDevice(e->device));
  void* src = comp < 3 ? e->E[e->cur][comp] : e->H[e->cur][comp - 3];
  int rc = copy_rows(e, src, dst, (size_t)e->nx * e->ny, e->rb, false);
  if (rc) return rc;
  PF_CUDA(e, cudaStreamSynchronize(e->stream));
  return PF_OK;
}

int pf_read_dft(pf_engine* e, int mon, int comp, double* dst) {
  if (!e || !dst) return PF_ERR_INVALID;
  if (!e->finalized) return fail(e, PF_ERR_STATE, "pf_read_dft before pf_finalize");
  if (mon < 0 || mon >= (int)e->dfts.size()) return fail(e, PF_ERR_INVALID, "bad DFT monitor %d", mon);
  DftMon& m = e->dfts[mon];
  int qc = -1;
  for (int q = 0; q < m.r.ncomp; ++q)
    if (m.r.comps[q] == comp) qc = q;
  if (qc < 0) return fail(e, PF_ERR_INVALID, "component %d not recorded by DFT monitor %d", comp, mon);
  int rc = e->rb == 4 ? flush_monitors<float>(e) : flush_monitors<double>(e);
  if (rc) return rc;
  const size_t per = (size_t)m.n_freq * m.r.ncell * 16;
  PF_CUDA(e, cudaMemcpyAsync(dst, (const char*)m.acc + per * qc, per, cudaMemcpyDeviceToHost, e->stream));
  PF_CUDA(e, cudaStreamSynchronize(e->stream));
  return PF_OK;
}

int pf_read_flux(pf_engine* e, int mon, double* dst) {
  if (!e || !dst) return PF_ERR_INVALID;
  if (!e->finalized) return fail(e, PF_ERR_STATE, "pf_read_flux before pf_finalize");
  if (mon < 0 || mon >= (int)e->fluxes.size()) return fail(e, PF_ERR_INVALID, "bad flux monitor %d", mon);
  int rc = e->rb == 4 ? flush_monitors<float>(e) : flush_monitors<double>(e);
  if (rc) return rc;
  PF_CUDA(e, cudaMemcpyAsync(dst, e->fluxes[mon].acc, 8, cudaMemcpyDeviceToHost, e->stream));
  PF_CUDA(e, cudaStreamSynchronize(e->stream));
  return PF_OK;
}

int pf_read_region(pf_engine* e, int comp, const int32_t start[3], const int32_t stop[3],
                   const int32_t stride[3], void* dst) {
  if (!e || !dst || !start || !stop || !stride) return PF_ERR_INVALID;
  if (!e->finalized) return fail(e, PF_ERR_STATE, "pf_read_region before pf_finalize");
  if (!valid_comp(comp)) return fail(e, PF_ERR_INVALID, "bad component %d", comp);
  const int dims[3] = {e->nx, e->ny, e->nz};
  int cnt[3];
  for (int a = 0; a < 3; ++a) {
    if (stride[a] < 1 || start[a] < 0 || stop[a] > dims[a] || start[a] >= stop[a])
      return fail(e, PF_ERR_INVALID, "bad region on axis %d", a);
    cnt[a] = (stop[a] - start[a] + stride[a] - 1) / stride[a];
  }
  const long long n = (long long)cnt[0] * cnt[1] * cnt[2];
  const size_t bytes = (size_t)n * e->rb;
  PF_CUDA(e, cudaSetDevice(e->device));
  const void* src = comp < 3 ? e->E[e->cur][comp] : e->H[e->cur][comp - 3];
  int rc;
  if (n == e->ncell) {  // the whole field: no gather
    if ((rc = copy_rows(e, const_cast<void*>(src), dst, (size_t)e->nx * e->ny, e->rb, false)))
      return rc;
    PF_CUDA(e, cudaStreamSynchronize(e->stream));
    return PF_OK;
  }
  if ((rc = stage(e, bytes))) return rc;
  const int3 st = make_int3(start[0], start[1], start[2]);
  const int3 sd = make_int3(stride[0], stride[1], stride[2]);
  const int3 ct = make_int3(cnt[0], cnt[1], cnt[2]);
  const unsigned g = (unsigned)std::min<long long>((n + 255) / 256, 148LL * 16);
  if (e->rb == 4)
    k_gather_region<float><<<g, 256, 0, e->stream>>>((const float*)src, e->ny, e->pz, st, sd, ct,
                                                     (float*)e->region);
  else
    k_gather_region<double><<<g, 256, 0, e->stream>>>((const double*)src, e->ny, e->pz, st, sd,
                                                      ct, (double*)e->region);
  PF_CUDA(e, cudaGetLastError());
  PF_CUDA(e, cudaMemcpyAsync(dst, e->region, bytes, cudaMemcpyDeviceToHost, e->stream));
  PF_CUDA(e, cudaStreamSynchronize(e->stream));
  return PF_OK;
}

int pf_write_field(pf_engine* e, int comp, const void* src) {
  if (!e || !src) return PF_ERR_INVALID;
  if (!e->finalized) return fail(e, PF_ERR_STATE, "pf_write_field before pf_finalize");
  if (!valid_comp(comp)) return fail(e, PF_ERR_INVALID, "bad component %d", comp);
  PF_CUDA(e, cudaSetDevice(e->device));
  void* dst = comp < 3 ? e->E[e->cur][comp] : e->H[e->cur][comp - 3];
  int rc = copy_rows(e, dst, const_cast<void*>(src), (size_t)e->nx * e->ny, e->rb, true);
  if (rc) return rc;
  PF_CUDA(e, cudaStreamSynchronize(e->stream));
  return PF_OK;
}

namespace {
// The stepping state as a list of pieces in the order of the state blob: the
// six current field components, the six E psi arrays, the six current H psi
// arrays, then the polarisation level holding P^n followed by the one holding
// P^(n-1) for `step` n. The blob is compact: pieces with rows along z (rows
// > 0) lose their padding.
struct StatePiece {
  char* p;
  size_t rows, bytes;  // bytes in the blob
  const int* zpos = nullptr;  // z layers kept in groups: places of the nc entries of a psi row
  int np = 0, nc = 0;
};
std::vector<StatePiece> state_pieces(pf_engine* e, long long step) {
  std::vector<StatePiece> v;
  const size_t S = e->rb, rows = (size_t)e->nx * e->ny, w = (size_t)e->nz * S;
  auto psi = [&](void* p, int q, long long r, long long n, const int* zpos, int np, int nc) {
    if ((q == 1 || q == 2) && np != nc)
      v.push_back({(char*)p, 0, rows * nc * S, zpos, np, nc});
    else
      v.push_back({(char*)p, (size_t)r, r ? (size_t)r * w : (size_t)n * S});
  };
  for (int c = 0; c < 3; ++c) v.push_back({(char*)e->E[e->cur][c], rows, rows * w});
  for (int c = 0; c < 3; ++c) v.push_back({(char*)e->H[e->cur][c], rows, rows * w});
  for (int q = 0; q < 6; ++q) psi(e->psiE[q], q, e->rpsiE[q], e->npsiE[q], e->zpos_e, e->npe[2], e->ncz_e);
  for (int q = 0; q < 6; ++q) psi(e->psiH[e->cur][q], q, e->rpsiH[q], e->npsiH[q], e->zpos_h, e->nph[2], e->ncz_h);
  if (e->n_media > 0) {
    const size_t lev = (size_t)e->plev * S;
    const int ln = (int)(step & 1);
    v.push_back({(char*)e->P + ln * lev, 0, lev});
    v.push_back({(char*)e->P + (ln ^ 1) * lev, 0, lev});
  }
  return v;
}

int copy_state(pf_engine* e, long long step, void* buf, int64_t bytes, int on_device, bool get) {
  if (!e || !buf) return PF_ERR_INVALID;
  if (!e->finalized) return fail(e, PF_ERR_STATE, "state access before pf_finalize");
  const auto pieces = state_pieces(e, step);
  size_t total = 0;
  for (const auto& p : pieces) total += p.bytes;
  if ((int64_t)total != bytes)
    return fail(e, PF_ERR_INVALID, "state buffer holds %lld bytes, the state is %zu",
                (long long)bytes, total);
  PF_CUDA(e, cudaSetDevice(e->device));
  const cudaMemcpyKind kind = on_device ? cudaMemcpyDeviceToDevice
                                        : (get ? cudaMemcpyDeviceToHost : cudaMemcpyHostToDevice);
  // device blobs aligned to their type are read and written as they lie, all
  // arrays in one launch; others go through the staging buffer
  const bool direct = on_device && (uintptr_t)buf % e->rb == 0;
  size_t off = 0;
  RowCopies c = {};
  int n = 0;
  for (const auto& p : pieces) {
    char* b = (char*)buf + off;
    off += p.bytes;
    if (p.bytes == 0) continue;
    const bool same = p.rows ? e->nz == e->pz : !p.zpos;  // the same bytes in both
    if (same) {
      PF_CUDA(e, cudaMemcpyAsync(get ? b : p.p, get ? p.p : b, p.bytes, kind, e->stream));
      continue;
    }
    const size_t rows = p.rows ? p.rows : (size_t)e->nx * e->ny;
    const int w = p.rows ? e->nz : p.nc, pitch = p.rows ? e->pz : p.np;
    if (direct) {
      c.r[n++] = row_copy(p.p, b, rows, w, pitch, p.zpos);
    } else {
      int rc = copy_staged(e, p.p, b, rows, w, pitch, p.zpos, e->rb, kind, !get);
      if (rc) return rc;
    }
  }
  if (n) launch_copy_rows(e, c, n, e->rb, get);
  PF_CUDA(e, cudaGetLastError());
  PF_CUDA(e, cudaStreamSynchronize(e->stream));
  return PF_OK;
}
// The engine is at `step` with no sample pending: the monitors' phase rows follow
// the step, not the count of samples taken so far.
void set_step(pf_engine* e, long long step) {
  e->step = step;
  for (DftMon& m : e->dfts) m.q_done = (step + m.interval - 1) / m.interval;
}
}  // namespace

int pf_state_bytes(const pf_engine* e, int64_t* bytes) {
  if (!e || !bytes) return PF_ERR_INVALID;
  if (!e->finalized) return PF_ERR_STATE;
  size_t total = 0;
  for (const auto& p : state_pieces(const_cast<pf_engine*>(e), e->step)) total += p.bytes;
  *bytes = (int64_t)total;
  return PF_OK;
}

int pf_get_state(pf_engine* e, void* dst, int64_t bytes, int dst_on_device) {
  if (!e) return PF_ERR_INVALID;
  return copy_state(e, e->step, dst, bytes, dst_on_device, true);
}

int pf_set_state(pf_engine* e, int64_t step, const void* src, int64_t bytes, int src_on_device) {
  if (!e) return PF_ERR_INVALID;
  if (!e->finalized) return fail(e, PF_ERR_STATE, "pf_set_state before pf_finalize");
  if (step < 0 || step > e->n_steps)
    return fail(e, PF_ERR_INVALID, "step %lld outside [0, n_steps]", (long long)step);
  // samples already taken belong to the old timeline: fold them first
  int rc = e->rb == 4 ? flush_monitors<float>(e) : flush_monitors<double>(e);
  if (rc) return rc;
  rc = copy_state(e, step, const_cast<void*>(src), bytes, src_on_device, false);
  if (rc) return rc;
  set_step(e, step);
  return PF_OK;
}

int pf_step(const pf_engine* e, int64_t* step) {
  if (!e || !step) return PF_ERR_INVALID;
  *step = e->step;
  return PF_OK;
}

int pf_check_finite(pf_engine* e) {
  if (!e) return PF_ERR_INVALID;
  if (!e->finalized) return fail(e, PF_ERR_STATE, "pf_check_finite before pf_finalize");
  PF_CUDA(e, cudaSetDevice(e->device));
  return scan_finite(e);
}

int pf_set_check_every(pf_engine* e, int64_t k) {
  if (!e) return PF_ERR_INVALID;
  if (k < 0) return fail(e, PF_ERR_INVALID, "check period must be >= 0");
  e->check_every = k;
  return PF_OK;
}

int pf_set_wait_test(pf_engine* e, int on) {
  if (!e) return PF_ERR_INVALID;
  e->wait_test = on == 2 ? 2 : (on ? 1 : 0);
  e->res_asked = e->res_off = false;
  return PF_OK;
}

int pf_stream(const pf_engine* e, void** stream) {
  if (!e || !stream) return PF_ERR_INVALID;
  *stream = (void*)e->stream;
  return PF_OK;
}

int pf_set_profiling(pf_engine* e, int on) {
  if (!e) return PF_ERR_INVALID;
  e->profiling = on != 0;
  return PF_OK;
}

int pf_read_profile(pf_engine* e, int64_t launches[4], double ms[4], int reset) {
  if (!e) return PF_ERR_INVALID;
  PF_CUDA(e, cudaStreamSynchronize(e->stream));
  collect_profile(e);
  for (int k = 0; k < 4; ++k) {
    if (launches) launches[k] = e->launches[k];
    if (ms) ms[k] = e->prof_ms[k];
    if (reset) {
      e->launches[k] = 0;
      e->prof_ms[k] = 0.0;
    }
  }
  return PF_OK;
}

int pf_info(const pf_engine* e, char* buf, int len) {
  if (!e || !buf || len < 1) return PF_ERR_INVALID;
  snprintf(buf, (size_t)len,
           "kernel=%s fused_ty=%d x_chunks=%d qdiv=%d%d%d ce_mode=%d media=%d real_bytes=%d "
           "tma=%d e_pass=%s "
           "shape=%dx%dx%d dft=%zu flux=%zu",
           e->fused ? "fused" : "split", e->fused_ty, e->fused_chunks, (int)e->fdiv[0],
           (int)e->fdiv[1], (int)e->fdiv[2], e->ce_mode, e->n_media, e->rb, (int)e->tma,
           !e->vec || e->ade_cells ? "cell" : "vector", e->nx,
           e->ny, e->nz,
           e->dfts.size(), e->fluxes.size());
  return PF_OK;
}

int pf_device_bytes(const pf_engine* e, int64_t* bytes) {
  if (!e || !bytes) return PF_ERR_INVALID;
  *bytes = (int64_t)e->dev_bytes;
  return PF_OK;
}

int pf_release_memory(void) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaSetDevice(dev) != cudaSuccess)
    return fail(nullptr, PF_ERR_CUDA, "no CUDA device");
  pool_trim();
  return PF_OK;
}

void pf_destroy(pf_engine* e) {
  if (!e) return;
  for (void* p : e->allocs) pool_free(p, e->stream);
  if (e->region) pool_free(e->region, e->stream);
  if (e->stream) cudaStreamSynchronize(e->stream);
  err_word_release(e->device, e->res_err);
  for (cudaEvent_t ev : e->ev_pool) cudaEventDestroy(ev);
  if (e->stream) cudaStreamDestroy(e->stream);
  delete e;
}

}  // extern "C"

// ---------------------------------------------------------------------------
// Adjoint of the stepping (value_and_grad_eps, jaxbackend.py:666-722): the
// caller checkpoints the forward run with pf_get_state, hands the loss's
// sensitivities to its outputs to pf_adj_set_dft_cotangent /
// pf_adj_add_field_source, then calls pf_adj_segment on the checkpointed
// segments from the last to the first. Each call restores the segment's
// state, replays it recording H^{n+1/2} and psi_E per step (no monitor
// sampling), and runs its reverse steps (kernels_adj.cuh), accumulating
// dJ/dK per cell.
// ---------------------------------------------------------------------------
namespace {

template <typename T>
AdjState<T> adj_state(pf_engine* e, long long slot) {
  AdjState<T> s;
  memset(&s, 0, sizeof s);
  const char* base = e->rec + (size_t)slot * e->rec_slot;
  const size_t S = sizeof(T), n = (size_t)e->ncellp * S;
  size_t off = 0;
  for (int c = 0; c < 3; ++c, off += n) s.Hrec[c] = (const T*)(base + off);
  for (int q = 0; q < 6; ++q) {
    s.psiErec[q] = (const T*)(base + off);
    off += (size_t)e->npsiE[q] * S;
  }
  for (int c = 0; c < 3; ++c) {
    s.lamE[c] = (T*)e->lamE[c];
    s.lamH[c] = (T*)e->lamH[c];
  }
  for (int q = 0; q < 6; ++q) {
    s.gE[q] = (T*)e->gE[q];
    s.gH[q] = (T*)e->gH[q];
    s.lpE[q] = (T*)e->lpE[q];
    s.lpH[q] = (T*)e->lpH[q];
  }
  s.grad = e->grad;
  // per-component coefficients are differentiated per component; one
  // coefficient per cell needs only the sum (16 instead of 48 bytes of
  // gradient traffic per cell and reverse step)
  s.gstride = e->ce_mode == PF_CE_CELL3 ? e->ncellp : 0;
  for (int a = 0; a < 3; ++a) s.idl[a] = (T)(1.0 / e->dl[a]);
  return s;
}

// The loss's sources on the fields sampled at step m, family fam (0: E^{m+1},
// 1: H^{m+1/2}).
template <typename T>
int adj_sources(pf_engine* e, long long m, int fam, const AdjState<T>& st, long long slot) {
  const int B = 256;
  T* l[3];
  for (int c = 0; c < 3; ++c) l[c] = (T*)(fam == 0 ? e->lamE[c] : e->lamH[c]);
  for (size_t k = 0; k < e->dfts.size(); ++k) {
    const DftMon& dm = e->dfts[k];
    if (!e->dft_cot[k] || m % dm.interval) continue;
    bool any = false;  // a component of this family
    for (int q = 0; q < dm.r.ncomp; ++q) any = any || (dm.r.comps[q] >= 3) == (fam == 1);
    if (!any) continue;
    const long long q = m / dm.interval;
    const double* ph = (fam == 0 ? dm.ph_e : dm.ph_h) + q * dm.n_freq * 2;
    const long long nt = dm.r.ncell * dm.r.ncomp;
    launch_pdl(e->stream, (unsigned)((nt + B - 1) / B), B, k_adj_dft_src<T>,
        dm.r, e->dft_cot[k], ph, dm.n_freq, dm.dt, fam, l[0], l[1], l[2], e->ny, e->pz);
  }
  for (const FluxMon& f : e->fluxes) {
    if (f.cot == 0.0) continue;
    const long long np = (long long)f.p.n0 * f.p.n1;
    launch_pdl(e->stream, (unsigned)((np + B - 1) / B), B, k_adj_flux_src<T>,
        f.p, f.cot * f.dA * f.dt, fam, st.Hrec[0], st.Hrec[1], st.Hrec[2],
        (const T*)f.rec + (size_t)slot * 2 * np, l[0], l[1], l[2], e->ny, e->pz);
  }
  for (const auto& rs : e->rsrc) {
    if (rs.step != m || (rs.comp >= 3) != (fam == 1)) continue;
    launch_pdl(e->stream, (unsigned)((rs.r.ncell + B - 1) / B), B, k_adj_region_src<T>,
        rs.r, rs.vals, l[rs.comp % 3], e->ny, e->pz);
  }
  PF_CUDA(e, cudaGetLastError());
  return PF_OK;
}

template <typename T>
int adj_segment_typed(pf_engine* e, long long step0, long long n) {
  e->recording = true;
  e->rec_step0 = step0;
  int rc = advance_typed<T>(e, n);
  e->recording = false;
  // the engine's own H and psi_E, also where the periodic scan stopped it
  if ((!rc || rc == PF_ERR_NONFINITE) && e->vec && !e->fused && e->step > step0) {
    const int rc2 = record_out(e, e->step - 1 - step0);
    if (!rc) rc = rc2;
  }
  if (rc) return rc;
  const int nz = e->nz, ny = e->ny, nx = e->nx;
  const int nzv = (nz + kVec<T> - 1) / kVec<T>;
  const dim3 blk = e->vec ? dim3(vec_lanes(nzv), kVecThreads / vec_lanes(nzv))
                          : (nz > 1 ? dim3(32, 8) : dim3(1, 256));
  const dim3 grd(((e->vec ? nzv : nz) + blk.x - 1) / blk.x, (ny + blk.y - 1) / blk.y, nx);
  const StepArgs<T> a = step_args<T>(e);
  for (long long m = step0 + n - 1; m >= step0; --m) {
    const AdjState<T> s = adj_state<T>(e, m - step0);
    if ((rc = adj_sources<T>(e, m, 0, s, m - step0))) return rc;
    if (e->vec && e->ce_mode == PF_CE_CELL1)
      launch_pdl(e->stream, grd, blk, k_adj_e_vec<T, kCeCell1>, a, s);
    else if (e->vec && e->ce_mode == PF_CE_CELL3)
      launch_pdl(e->stream, grd, blk, k_adj_e_vec<T, kCeCell3>, a, s);
    else if (e->vec)
      launch_pdl(e->stream, grd, blk, k_adj_e_vec<T, kCeTable>, a, s);
    else if (e->ce_mode == PF_CE_CELL1)
      launch_pdl(e->stream, grd, blk, k_adj_e<T, kCeCell1>, a, s);
    else if (e->ce_mode == PF_CE_CELL3)
      launch_pdl(e->stream, grd, blk, k_adj_e<T, kCeCell3>, a, s);
    else
      launch_pdl(e->stream, grd, blk, k_adj_e<T, kCeTable>, a, s);
    if ((rc = adj_sources<T>(e, m, 1, s, m - step0))) return rc;
    if (e->vec) launch_pdl(e->stream, grd, blk, k_adj_h_vec<T>, a, s);
    else launch_pdl(e->stream, grd, blk, k_adj_h<T>, a, s);
  }
  PF_CUDA(e, cudaGetLastError());
  PF_CUDA(e, cudaStreamSynchronize(e->stream));
  e->adj_next = step0;
  return PF_OK;
}

int adj_zero(pf_engine* e) {
  const size_t S = e->rb, n = (size_t)e->ncellp * S;
  for (int c = 0; c < 3; ++c) {
    PF_CUDA(e, cudaMemsetAsync(e->lamE[c], 0, n, e->stream));
    PF_CUDA(e, cudaMemsetAsync(e->lamH[c], 0, n, e->stream));
  }
  for (int q = 0; q < 6; ++q) {
    PF_CUDA(e, cudaMemsetAsync(e->gE[q], 0, n, e->stream));
    PF_CUDA(e, cudaMemsetAsync(e->gH[q], 0, n, e->stream));
    if (e->npsiE[q]) PF_CUDA(e, cudaMemsetAsync(e->lpE[q], 0, e->npsiE[q] * S, e->stream));
    if (e->npsiH[q]) PF_CUDA(e, cudaMemsetAsync(e->lpH[q], 0, e->npsiH[q] * S, e->stream));
  }
  PF_CUDA(e, cudaMemsetAsync(e->grad, 0, (size_t)e->ncellp * 24, e->stream));
  PF_CUDA(e, cudaStreamSynchronize(e->stream));
  e->adj_next = e->n_steps;
  return PF_OK;
}

bool make_region(pf_engine* e, const int32_t start[3], const int32_t stop[3],
                 const int32_t stride[3], DftRegion& r) {
  const int dims[3] = {e->nx, e->ny, e->nz};
  r.ncell = 1;
  r.ncomp = 1;
  for (int a = 0; a < 3; ++a) {
    if (start[a] < 0 || stop[a] > dims[a] || stop[a] <= start[a] || stride[a] < 1) return false;
    r.start[a] = start[a];
    r.stride[a] = stride[a];
    r.count[a] = (stop[a] - start[a] + stride[a] - 1) / stride[a];
    r.ncell *= r.count[a];
  }
  return true;
}

}  // namespace

extern "C" {

int pf_adj_init(pf_engine* e, int64_t ring_steps) {
  if (!e) return PF_ERR_INVALID;
  if (!e->finalized) return fail(e, PF_ERR_STATE, "pf_adj_init before pf_finalize");
  if (e->n_media > 0)
    return fail(e, PF_ERR_UNSUPPORTED, "the adjoint does not cover dispersive (ADE) media");
  if (ring_steps < 1 || ring_steps > e->n_steps)
    return fail(e, PF_ERR_INVALID, "ring_steps %lld outside [1, n_steps]", (long long)ring_steps);
  PF_CUDA(e, cudaSetDevice(e->device));
  int rc;
  const size_t S = e->rb, n = (size_t)e->ncellp * S;
  if (!e->adj) {
    for (int c = 0; c < 3; ++c) {
      if ((rc = dalloc(e, &e->lamE[c], n))) return rc;
      if ((rc = dalloc(e, &e->lamH[c], n))) return rc;
    }
    for (int q = 0; q < 6; ++q) {
      if ((rc = dalloc(e, &e->gE[q], n))) return rc;
      if ((rc = dalloc(e, &e->gH[q], n))) return rc;
      if ((rc = dalloc(e, &e->lpE[q], e->npsiE[q] * S))) return rc;
      if ((rc = dalloc(e, &e->lpH[q], e->npsiH[q] * S))) return rc;
    }
    if ((rc = dalloc(e, (void**)&e->grad, (size_t)e->ncellp * 24))) return rc;
    e->dft_cot.assign(e->dfts.size(), nullptr);
    e->adj = true;
  }
  if (ring_steps > e->ring_steps) {
    size_t slot = 3 * n;
    for (int q = 0; q < 6; ++q) slot += e->npsiE[q] * S;
    e->rec_slot = (slot + 255) & ~(size_t)255;
    // the old ring stays allocated (freed with the engine)
    if ((rc = dalloc(e, (void**)&e->rec, e->rec_slot * (size_t)ring_steps))) return rc;
    e->ring_steps = ring_steps;
  }
  return adj_zero(e);
}

int pf_adj_set_dft_cotangent(pf_engine* e, int mon, const double* cot) {
  if (!e || !cot) return PF_ERR_INVALID;
  if (!e->adj) return fail(e, PF_ERR_STATE, "pf_adj_set_dft_cotangent before pf_adj_init");
  if (mon < 0 || mon >= (int)e->dfts.size()) return fail(e, PF_ERR_INVALID, "bad DFT monitor");
  const DftMon& dm = e->dfts[mon];
  const size_t bytes = (size_t)dm.r.ncomp * dm.n_freq * dm.r.ncell * 16;
  int rc;
  if (!e->dft_cot[mon] && (rc = dalloc(e, (void**)&e->dft_cot[mon], bytes))) return rc;
  PF_CUDA(e, cudaMemcpyAsync(e->dft_cot[mon], cot, bytes, cudaMemcpyHostToDevice, e->stream));
  PF_CUDA(e, cudaStreamSynchronize(e->stream));
  return PF_OK;
}

int pf_adj_set_flux_cotangent(pf_engine* e, int mon, double cot) {
  if (!e) return PF_ERR_INVALID;
  if (!e->adj) return fail(e, PF_ERR_STATE, "pf_adj_set_flux_cotangent before pf_adj_init");
  if (mon < 0 || mon >= (int)e->fluxes.size()) return fail(e, PF_ERR_INVALID, "bad flux monitor");
  if (!std::isfinite(cot)) return fail(e, PF_ERR_INVALID, "flux cotangent must be finite");
  FluxMon& f = e->fluxes[mon];
  if (cot != 0.0 && f.rec_cap < e->ring_steps) {
    int rc;
    const size_t bytes = (size_t)e->ring_steps * 2 * f.p.n0 * f.p.n1 * e->rb;
    if ((rc = dalloc(e, &f.rec, bytes))) return rc;
    f.rec_cap = e->ring_steps;
  }
  f.cot = cot;
  return PF_OK;
}

int pf_adj_add_field_source(pf_engine* e, int64_t step, int comp, const int32_t start[3],
                            const int32_t stop[3], const int32_t stride[3], const double* vals) {
  if (!e || !vals || !start || !stop || !stride) return PF_ERR_INVALID;
  if (!e->adj) return fail(e, PF_ERR_STATE, "pf_adj_add_field_source before pf_adj_init");
  if (!valid_comp(comp) || step < 0 || step >= e->n_steps)
    return fail(e, PF_ERR_INVALID, "bad component or step");
  pf_engine::RegionSource rs;
  rs.step = step;
  rs.comp = comp;
  if (!make_region(e, start, stop, stride, rs.r)) return fail(e, PF_ERR_INVALID, "bad region");
  int rc;
  if ((rc = dalloc(e, (void**)&rs.vals, (size_t)rs.r.ncell * 8))) return rc;
  PF_CUDA(e, cudaMemcpyAsync(rs.vals, vals, (size_t)rs.r.ncell * 8, cudaMemcpyHostToDevice,
                             e->stream));
  PF_CUDA(e, cudaStreamSynchronize(e->stream));
  e->rsrc.push_back(rs);
  return PF_OK;
}

int pf_adj_segment(pf_engine* e, int64_t step0, int64_t n, const void* state, int64_t bytes,
                   int state_on_device) {
  if (!e || !state) return PF_ERR_INVALID;
  if (!e->adj) return fail(e, PF_ERR_STATE, "pf_adj_segment before pf_adj_init");
  if (n < 1 || n > e->ring_steps || step0 < 0 || step0 + n != e->adj_next)
    return fail(e, PF_ERR_STATE,
                "segment [%lld, %lld) must end where the reverse pass stands (%lld) and hold at "
                "most %lld steps",
                (long long)step0, (long long)(step0 + n), e->adj_next, e->ring_steps);
  int rc = e->rb == 4 ? flush_monitors<float>(e) : flush_monitors<double>(e);
  if (rc) return rc;
  if ((rc = copy_state(e, step0, const_cast<void*>(state), bytes, state_on_device, false)))
    return rc;
  e->step = step0;
  rc = e->rb == 4 ? adj_segment_typed<float>(e, step0, n) : adj_segment_typed<double>(e, step0, n);
  set_step(e, e->step);  // a replay samples nothing
  return rc;
}

int pf_adj_read_grad_components(pf_engine* e, double* dst) {
  if (!e || !dst) return PF_ERR_INVALID;
  if (!e->adj) return fail(e, PF_ERR_STATE, "gradient read before pf_adj_init");
  if (e->ce_mode != PF_CE_CELL3)
    return fail(e, PF_ERR_STATE,
                "per-component gradient kept only for per-component coefficients "
                "(PF_CE_CELL3); use pf_adj_read_grad");
  PF_CUDA(e, cudaSetDevice(e->device));
  int rc = copy_rows(e, e->grad, dst, (size_t)e->nx * e->ny * 3, 8, false);
  if (rc) return rc;
  PF_CUDA(e, cudaStreamSynchronize(e->stream));
  return PF_OK;
}

int pf_adj_read_grad(pf_engine* e, double* dst) {
  if (!e || !dst) return PF_ERR_INVALID;
  if (!e->adj) return fail(e, PF_ERR_STATE, "gradient read before pf_adj_init");
  const size_t n = (size_t)e->ncell;
  if (e->ce_mode != PF_CE_CELL3) {  // accumulated summed over the components
    PF_CUDA(e, cudaSetDevice(e->device));
    int rc = copy_rows(e, e->grad, dst, (size_t)e->nx * e->ny, 8, false);
    if (rc) return rc;
    PF_CUDA(e, cudaStreamSynchronize(e->stream));
    return PF_OK;
  }
  std::vector<double> g(n * 3);
  int rc = pf_adj_read_grad_components(e, g.data());
  if (rc) return rc;
  for (size_t i = 0; i < n; ++i) dst[i] = (g[i] + g[n + i]) + g[2 * n + i];
  return PF_OK;
}

}  // extern "C"
