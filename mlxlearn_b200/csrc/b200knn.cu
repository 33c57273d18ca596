// C ABI of libb200knn.so: index lifetime and the kNN entry points.
//
// Call flow of one kNN batch (all on one stream):
//   prep_queries  -> per-query screen bound E (and the -2*bf16(q) operand)
//   screen        -> tcgen05 bf16 (screen_tc.cu) or fp32 CUDA-core (screen_simt.cu)
//   certify       -> float64 re-rank + exact near-tie resolution (certify.cu)
//   exact         -> exhaustive exact scan of the rare rows certify could not
//                    finish (list overflow), no-op otherwise
// Scratch buffers come from the stream-ordered allocator (cudaMallocAsync).
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cstdarg>
#include <cmath>
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <utility>
#include <vector>

#include "common.cuh"
#include "internal.cuh"
#include "sinks.cuh"

struct b2k_index {
  b2k::Index ix;
};

namespace b2k {

// ------------------------------------------------------------------ errors
static thread_local std::string g_last_error;

static int fail(int code, const char* fmt, ...) __attribute__((format(printf, 2, 3)));
static int fail(int code, const char* fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof(buf), fmt, ap);
  va_end(ap);
  g_last_error = buf;
  return code;
}

#define B2K_CUDA(call)                                                                      \
  do {                                                                                      \
    cudaError_t e_ = (call);                                                                \
    if (e_ != cudaSuccess)                                                                  \
      return fail(e_ == cudaErrorMemoryAllocation ? B2K_ENOMEM : B2K_ECUDA, "%s: %s (%s:%d)", \
                  #call, cudaGetErrorString(e_), __FILE__, __LINE__);                       \
  } while (0)

// Host-side fault injection for failure-path tests (B2K_FAULT=alloc|alloc:N|launch|timeout).
static int fault_mode() {
  const char* f = getenv("B2K_FAULT");
  if (!f || !*f) return 0;
  if (!strcmp(f, "alloc")) return 1;
  if (!strcmp(f, "launch")) return 2;
  if (!strcmp(f, "timeout")) return 3;
  return 0;
}

// Whether this device allocation is to fail: every one under B2K_FAULT=alloc,
// the N-th since the variable was set under alloc:N (counted while it is set).
static bool inject_alloc_failure() {
  static std::atomic<long> seen{0};
  const char* f = getenv("B2K_FAULT");
  if (!f || strncmp(f, "alloc", 5)) {
    seen.store(0, std::memory_order_relaxed);
    return false;
  }
  if (!f[5]) return true;
  return f[5] == ':' && seen.fetch_add(1) + 1 == atol(f + 6);
}

uint32_t device_spin_limit() {
  const char* e = getenv("B2K_SPIN_LIMIT");
  if (e && *e) {
    const unsigned long v = strtoul(e, nullptr, 10);
    if (v > 0 && v <= kSpinLimit) return (uint32_t)v;
  }
  return kSpinLimit;
}

int num_sms(int device) {
  static int cached[64] = {0};
  if (device < 0 || device >= 64) return 148;
  if (!cached[device]) {
    int v = 0;
    if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, device) != cudaSuccess || v <= 0)
      v = 148;
    cached[device] = v;
  }
  return cached[device];
}

cudaError_t allow_smem_impl(const void* kernel, size_t bytes) {
  int device = 0;
  cudaError_t e = cudaGetDevice(&device);
  if (e != cudaSuccess) return e;
  static std::mutex mu;
  static std::map<std::pair<const void*, int>, size_t> limits;  // one entry per kernel and device
  std::lock_guard<std::mutex> lock(mu);
  size_t& limit = limits[{kernel, device}];
  if (limit >= bytes) return cudaSuccess;
  e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e == cudaSuccess) limit = bytes;
  return e;
}

// --------------------------------------------------------------- TMA maps
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                  const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  static bool tried = false;
  if (!tried) {
    tried = true;
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  }
  return fn;
}

static bool tensor_map_2d(CUtensorMap* map, CUtensorMapDataType type, uint64_t elem_bytes,
                          const void* base, uint64_t inner, uint64_t outer, uint32_t box_inner,
                          uint32_t box_outer, int swizzle_bytes) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return false;
  cuuint64_t dims[2] = {inner, outer};
  cuuint64_t strides[1] = {inner * elem_bytes};
  cuuint32_t box[2] = {box_inner, box_outer};
  cuuint32_t estr[2] = {1, 1};
  const CUtensorMapSwizzle sw = swizzle_bytes == 32   ? CU_TENSOR_MAP_SWIZZLE_32B
                                : swizzle_bytes == 64 ? CU_TENSOR_MAP_SWIZZLE_64B
                                                      : CU_TENSOR_MAP_SWIZZLE_128B;
  CUresult r = fn(map, type, 2, const_cast<void*>(base), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, sw, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}

bool tensor_map_2d_bf16(CUtensorMap* map, const void* base, uint64_t inner, uint64_t outer,
                        uint32_t box_inner, uint32_t box_outer, int swizzle_bytes) {
  return tensor_map_2d(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, base, inner, outer, box_inner,
                       box_outer, swizzle_bytes);
}

bool tensor_map_2d_f32(CUtensorMap* map, const void* base, uint64_t inner, uint64_t outer,
                       uint32_t box_inner, uint32_t box_outer, int swizzle_bytes) {
  return tensor_map_2d(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, base, inner, outer, box_inner,
                       box_outer, swizzle_bytes);
}

// ------------------------------------------------------------------ helpers
static int check_device(int device) {
  int count = 0;
  if (cudaGetDeviceCount(&count) != cudaSuccess || count <= 0)
    return fail(B2K_EUNSUPPORTED, "no CUDA device is available");
  if (device < 0 || device >= count) return fail(B2K_EINVAL, "invalid device %d", device);
  // (cudaGetDeviceProperties takes 2.6 ms: more than most of an index's build)
  int major = 0, minor = 0;
  if (cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, device) != cudaSuccess ||
      cudaDeviceGetAttribute(&minor, cudaDevAttrComputeCapabilityMinor, device) != cudaSuccess)
    return fail(B2K_ECUDA, "cudaDeviceGetAttribute failed");
  if (major != 10)
    return fail(B2K_EUNSUPPORTED, "libb200knn needs an sm_100 (B200) device, found sm_%d%d",
                major, minor);
  return B2K_OK;
}

template <typename T>
static int dalloc(T** p, size_t count, cudaStream_t st) {
  if (inject_alloc_failure())
    return fail(B2K_ENOMEM, "injected allocation failure (B2K_FAULT=alloc)");
  *p = nullptr;
  if (count == 0) count = 1;
  cudaError_t e = cudaMallocAsync(reinterpret_cast<void**>(p), count * sizeof(T), st);
  if (e != cudaSuccess) {
    cudaGetLastError();  // (the next launch's check would report it again)
    return fail(e == cudaErrorMemoryAllocation ? B2K_ENOMEM : B2K_ECUDA,
                "device allocation of %zu bytes failed: %s", count * sizeof(T),
                cudaGetErrorString(e));
  }
  return B2K_OK;
}

// A buffer of the index (freed with it).  Buffers of up to kPoolAlloc bytes come
// from the stream-ordered pool: a cudaMalloc or cudaFree costs 40 to 60 us, and
// an index of a training step lives for one call (17 buffers, 1.8 ms of the 6.5
// ms of 32,768 x 64 rows against themselves).  Larger ones are given back to the
// device when freed, so what the pool keeps stays small.  The index's creators
// synchronise its stream before any other stream sees a buffer.
constexpr size_t kPoolAlloc = (size_t)32 << 20;
template <typename T>
static int ialloc(Index& ix, T** p, size_t count) {
  if (inject_alloc_failure())
    return fail(B2K_ENOMEM, "injected allocation failure (B2K_FAULT=alloc)");
  const size_t bytes = std::max<size_t>(count, 1) * sizeof(T);
  const bool pooled = bytes <= kPoolAlloc;
  void* v = nullptr;
  const cudaError_t e = pooled ? cudaMallocAsync(&v, bytes, ix.stream) : cudaMalloc(&v, bytes);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail(e == cudaErrorMemoryAllocation ? B2K_ENOMEM : B2K_ECUDA,
                "device allocation of %zu bytes failed: %s", bytes, cudaGetErrorString(e));
  }
  ix.owned.emplace_back(v, pooled);
  *p = static_cast<T*>(v);
  return B2K_OK;
}

static int64_t round_up(int64_t v, int64_t m) { return (v + m - 1) / m * m; }

static bool overlaps(const void* a, size_t an, const void* b, size_t bn);

// Whether kNN outputs overlap the queries or each other (internal.cuh).
bool buffers_overlap(const float* dQ, int64_t m, int d, int k, const double* dist,
                     const int64_t* idx) {
  const size_t q = (size_t)m * d * sizeof(float), o = (size_t)m * k * 8;
  return overlaps(idx, o, dQ, q) || overlaps(dist, o, dQ, q) || overlaps(idx, o, dist, o);
}

static bool overlaps(const void* a, size_t an, const void* b, size_t bn) {
  if (!a || !b || !an || !bn) return false;
  auto x = reinterpret_cast<uintptr_t>(a), y = reinterpret_cast<uintptr_t>(b);
  return x < y + bn && y < x + an;
}

// Free a list of stream-ordered allocations (ignores nulls).
struct StreamFree {
  cudaStream_t st;
  std::vector<void*> ptrs;
  ~StreamFree() {
    for (void* p : ptrs)
      if (p) cudaFreeAsync(p, st);
  }
  template <typename T>
  T* keep(T* p) {
    ptrs.push_back(p);
    return p;
  }
};

// The scratch of one call as one stream-ordered allocation: buffers are reserved
// first (256-byte aligned), then placed.  Seventeen cudaMallocAsync and as many
// frees, four memsets and three reads back were 70 of the 155 us of a 2,000
// query call.
class Workspace {
 public:
  template <typename T>
  void reserve(T** p, size_t count) {
    slots_.push_back({reinterpret_cast<void**>(p), bytes_});
    bytes_ += (std::max<size_t>(count, 1) * sizeof(T) + 255) / 256 * 256;
  }
  size_t bytes() const { return bytes_; }
  int place(cudaStream_t st, StreamFree& fr) {
    unsigned char* base = nullptr;
    const int rc = dalloc(&base, bytes_, st);
    if (rc) return rc;
    fr.keep(base);
    for (auto& s : slots_) *s.first = base + s.second;
    return B2K_OK;
  }

 private:
  std::vector<std::pair<void**, size_t>> slots_;
  size_t bytes_ = 0;
};

// Error word, counts and flags of a kNN call, zeroed together and read back
// together.
struct CallState {
  int status[8];                     // [0] error, [2] uncertified rows, [4] range, [5] nonfinite,
                                     // [6] [7] claimed units of the screens
  unsigned long long counters[8];
};

static int finish_index(Index& ix, cudaStream_t st) {
  B2K_CUDA(cudaMemsetAsync(ix.stats_dev, 0, kStatsLen * sizeof(float), st));
  launch_prep_index(&ix, st);
  B2K_CUDA(cudaGetLastError());
  // narrow rows: the sample that chooses their screen (NarrowProfile)
  const bool narrow = ix.d >= kTcMinD && ix.d < kTcAlwaysD && ix.n >= kTcMinN;
  struct Sample {
    double norms[kProfileSamples];
    int hist[kProfileSamples * kProfileBins];
  };
  StreamFree fr{st, {}};
  std::vector<Sample> sample(narrow ? 1 : 0);
  const int rows = profile_rows(ix.n);
  if (narrow) {
    Sample* dev = nullptr;
    if (const int rc = dalloc(&dev, 1, st)) return rc;
    fr.keep(dev);
    B2K_CUDA(cudaMemsetAsync(dev, 0, sizeof(Sample), st));
    launch_narrow_profile(&ix, rows, dev->hist, dev->norms, st);
    B2K_CUDA(cudaGetLastError());
    B2K_CUDA(cudaMemcpyAsync(sample.data(), dev, sizeof(Sample), cudaMemcpyDeviceToHost, st));
  }
  float stats[kStatsLen];
  B2K_CUDA(cudaMemcpyAsync(stats, ix.stats_dev, sizeof(stats), cudaMemcpyDeviceToHost, st));
  B2K_CUDA(cudaStreamSynchronize(st));
  ix.xn_max = stats[0];
  ix.nx_max = stats[1];
  ix.ex32_max = stats[5];
  int bad;
  memcpy(&bad, &stats[2], 4);
  ix.range_ok = bad == 0;
  // (below 2^-80 the bins would leave the float range: such rows take the fp32 screen)
  if (narrow && ix.range_ok && ix.nx_max > 0x1p-80f) {
    NarrowProfile& p = ix.profile;
    std::nth_element(sample[0].norms, sample[0].norms + kProfileSamples / 2,
                     sample[0].norms + kProfileSamples);
    p.rms = (float)std::sqrt(sample[0].norms[kProfileSamples / 2]);
    p.base = profile_base(ix.nx_max);
    p.cum.assign((size_t)kProfileSamples * (kProfileBins + 1), 0);
    for (int s = 0; s < kProfileSamples; ++s) {
      int* cum = p.cum.data() + (size_t)s * (kProfileBins + 1);
      for (int b = 0; b < kProfileBins; ++b)
        cum[b + 1] = cum[b] + sample[0].hist[s * kProfileBins + b];
    }
    p.rows = rows;
  }
  return B2K_OK;
}

// ------------------------------------------- which screen narrow rows take
// Lower edge of bin b of a profile (the first bin reaches down to zero).
static double profile_edge(const NarrowProfile& p, int b) {
  if (b <= 0) return 0.0;
  const uint32_t bits = (uint32_t)(b + p.base) << 21;
  float v;
  memcpy(&v, &bits, sizeof(v));
  return v;
}

// Rows of sample s within squared distance t (interpolated in t's bin).
static double profile_within(const NarrowProfile& p, int s, double t) {
  const int* cum = p.cum.data() + (size_t)s * (kProfileBins + 1);
  const float tf = (float)t;
  uint32_t bits;
  memcpy(&bits, &tf, sizeof(bits));
  const int b = std::max((int)(bits >> 21) - p.base, 0);
  if (b >= kProfileBins) return cum[kProfileBins];
  const double lo = profile_edge(p, b), hi = profile_edge(p, b + 1);
  return cum[b] + (cum[b + 1] - cum[b]) * std::min(1.0, (t - lo) / (hi - lo));
}

// Squared distance within which sample s has `rows` rows.
static double profile_radius2(const NarrowProfile& p, int s, double rows) {
  const int* cum = p.cum.data() + (size_t)s * (kProfileBins + 1);
  const int b = (int)(std::lower_bound(cum + 1, cum + kProfileBins, rows) - cum) - 1;
  const double lo = profile_edge(p, b), hi = profile_edge(p, b + 1);
  const int in = cum[b + 1] - cum[b];
  return in > 0 ? lo + (hi - lo) * std::min(1.0, std::max(0.0, (rows - cum[b]) / in)) : hi;
}

// The certified error of the tensor-core screen for a query at the samples'
// median distance from the centre (prep.cu derives it).
static double profile_error(const Index& ix) {
  const double g = (double)(operand_dp(ix.d) + kTcAug + 16) * 0x1p-20;
  return 1.02 * g * (2.0 * ix.profile.rms * ix.xn_max + ix.nx_max);
}

// Whether AUTO sends m queries to the tensor cores.  Under 16 features by the
// band the sample predicts: rows within 2E of the k-th distance.
// * Large calls: while a quarter of the samples at most hold more than the 1,024
//   that certify takes.  (Tensor cores / fp32 screen by that share, 200,003 rows,
//   50,021 queries: 0.31 10.9 / 17.4 ms at k = 5, 19.3 / 18.5 at k = 15; 0.61
//   15.1 / 16.9 at k = 5 and 51 / 31.5 at k = 50; 0.77 22.5 / 17.5; 0.95 60 / 17.)
// * Small calls (the fp32 screen takes under 0.5 ms) pay every listed row with
//   latency and a second pass whole: 10,000 x 8, 2,000 queries, k = 5: 20 band
//   rows 0.138 / 0.145 ms, 88 0.157 / 0.141, 502 0.265 / 0.146; k = 50: 106
//   0.187 / 0.369.  20,000 x 5, 100 queries, k = 5: 110 0.137 / 0.098.
// The predicted share agrees with the measured one to a few percent over normal,
// uniform, heavy-tailed and clustered rows and one far row or column.
static bool knn_on_tensor_cores(Index& ix, int64_t m, int k) {
  if (ix.d < kTcMinD || ix.n < kTcMinN) return false;
  if (ix.d >= kTcAlwaysD) return true;
  const NarrowProfile& p = ix.profile;
  if (!p.rows) return false;
  const bool small = m * ix.n < ((int64_t)1 << 28);
  std::atomic<signed char>& known = ix.profile.knn[small ? 0 : 1][k];
  if (const signed char said = known.load(std::memory_order_relaxed)) return said > 0;
  const double limit = small ? 2.0 * k + 32.0 : 1024.0;
  const double scale = (double)ix.n / p.rows;
  const double kth = std::max(1.0, k / scale), band = 2.0 * profile_error(ix);
  int wide = 0;
  for (int s = 0; s < kProfileSamples; ++s) {
    const double t = profile_radius2(p, s, kth);
    if ((profile_within(p, s, t + band) - kth) * scale + k > limit) ++wide;
  }
  const bool fits = wide * 4 <= kProfileSamples;
  known.store(fits ? 1 : -1, std::memory_order_relaxed);
  return fits;
}

// Whether the radius search sends a block of m queries to the tensor cores: as
// above, by the rows in (R2, R2 + 2E] a query.  Every one is a candidate (12 bytes
// of scratch and an exact test), so they are kept below 1,024, or below the
// answer's own size: 200,003 x 8, 20,000 queries, 90 neighbours: 421 candidates 1.4
// / 13.1 ms, 2,082 2.0, 38,007 6.9 ms and 9 GB, where the fp32 screen has 93.
// Small calls (pairs with the queries padded to a tile) are launches and host
// reads, of which the list form has more than the fp32 screen's counted form:
// 10,000 x 8, 500 queries: 232 / 167 us; 20,000 x 13, 500: 284 / 207; 50,000 x 8,
// 500 (2.5e7 pairs): 273 / 247; 10,000 x 8, 4,000 (4e7): 229 / 310; 100,000 x 13,
// 500: 328 / 359; 200,000 x 8, 1 (2.6e7): 263 / 367.
static bool radius_on_tensor_cores(const Index& ix, int64_t m, double R2) {
  if (ix.d < kTcMinD || ix.n < kTcMinN) return false;
  if (ix.d >= kTcAlwaysD) return true;
  const NarrowProfile& p = ix.profile;
  if (!p.rows || std::max<int64_t>(m, kTcBM) * ix.n < ((int64_t)3 << 23)) return false;
  const double band = 2.0 * profile_error(ix);
  double inside = 0, wide = 0;
  for (int s = 0; s < kProfileSamples; ++s) {
    inside += profile_within(p, s, R2);
    wide += profile_within(p, s, R2 + band);
  }
  const double scale = (double)ix.n / p.rows / kProfileSamples;
  return (wide - inside) * scale <= std::max(1024.0, inside * scale);
}

// Pivots for query grouping and row grouping (the caller holds ix.mu).  Set
// together and last: ix.pivots tells that all of them are built, so a failed
// allocation or launch leaves the index without pivots and a later call starts
// over.
static int make_pivots(Index& ix) {
  if (ix.pivots) return B2K_OK;
  int rc;
  const int P = pivot_count(ix.n), dpa = pivot_dims_padded(ix.d);
  float *pivots = nullptr, *norms = nullptr;
  uint16_t* rows = nullptr;
  if ((rc = ialloc(ix, &pivots, (size_t)P * ix.d))) return rc;
  if ((rc = ialloc(ix, &norms, (size_t)P))) return rc;
  if ((rc = ialloc(ix, &rows, (size_t)pivot_rows_padded(P) * dpa))) return rc;
  launch_pivots(&ix, P, dpa, pivots, norms, rows, ix.stream);
  B2K_CUDA(cudaGetLastError());
  B2K_CUDA(cudaStreamSynchronize(ix.stream));
  ix.n_pivots = P;
  ix.pivot_dpa = dpa;
  ix.pivot_norms = norms;
  ix.pivots_h = rows;
  ix.pivots = pivots;
  return B2K_OK;
}

// Indexes of at least this many rows get grouped operand rows (unless
// B2K_GROUP_ROWS=0; tests run both ways).
constexpr int64_t kGroupMinRows = 8192;
static bool group_rows_enabled(const Index& ix) {
  const char* e = getenv("B2K_GROUP_ROWS");
  return ix.n >= kGroupMinRows && !(e && e[0] == '0');
}

// Operand row order grouped by nearest pivot (the caller holds ix.mu): a
// stable counting sort on the device, so rows keep their training order within
// a group and the layout is the same on every build.
static int make_row_groups(Index& ix) {
  cudaStream_t st = ix.stream;
  int rc = make_pivots(ix);
  if (rc) return rc;
  const int P = ix.n_pivots;
  StreamFree fr{st, {}};
  int *key = nullptr, *hist = nullptr, *tiles = nullptr;
  if ((rc = dalloc(&key, (size_t)ix.n, st))) return rc;
  fr.keep(key);
  if ((rc = dalloc(&hist, (size_t)P, st))) return rc;
  fr.keep(hist);
  if ((rc = dalloc(&tiles, row_group_scratch(ix.n, P), st))) return rc;
  fr.keep(tiles);
  int *perm = nullptr, *inv = nullptr, *start = nullptr;
  if ((rc = ialloc(ix, &perm, (size_t)ix.n))) return rc;
  if ((rc = ialloc(ix, &inv, (size_t)ix.n))) return rc;
  if ((rc = ialloc(ix, &start, (size_t)P + 1))) return rc;
  unsigned long long* best64 = nullptr;
  if (const size_t words = assign_scratch(&ix, ix.n)) {
    if ((rc = dalloc(&best64, words, st))) return rc;
    fr.keep(best64);
  }
  launch_assign_rows(&ix, ix.X, ix.n, key, hist, best64, st);
  launch_row_groups(key, ix.n, P, hist, tiles, start, perm, inv, st);
  B2K_CUDA(cudaGetLastError());
  // (set together: a failed build leaves the index ungrouped)
  ix.xperm = perm;
  ix.xinv = inv;
  ix.group_start = start;
  return B2K_OK;
}

// Row grouping shared by the tensor-core operands (the caller holds ix.mu):
// decided once, with the first operand built.
static int ensure_row_groups(Index& ix) {
  if (ix.xperm || ix.bf16_ready || ix.tf32_ready || !group_rows_enabled(ix)) return B2K_OK;
  return make_row_groups(ix);
}

static OperandStats bf16_stats(const float* stats) {
  OperandStats s;
  s.xh = stats[3];
  s.ex = stats[4];
  for (int i = 0; i < 3; ++i) s.part[i] = stats[8 + i];
  return s;
}

static int ensure_bf16(Index& ix) {
  std::lock_guard<std::mutex> lock(ix.mu);
  if (ix.bf16_ready) return B2K_OK;
  cudaStream_t st = ix.stream;
  ix.dp = (int32_t)operand_dp(ix.d);
  ix.n_pad_tc = round_up(ix.n, kTcBN);
  int rc;
  if ((rc = ensure_row_groups(ix))) return rc;
  if ((rc = ialloc(ix, &ix.Xh, (size_t)ix.n_pad_tc * ix.dp))) return rc;
  launch_prep_index_bf16(&ix, ix.Xh, st, ix.xperm);
  B2K_CUDA(cudaGetLastError());
  float stats[kStatsLen];
  B2K_CUDA(cudaMemcpyAsync(stats, ix.stats_dev, sizeof(stats), cudaMemcpyDeviceToHost, st));
  B2K_CUDA(cudaStreamSynchronize(st));
  ix.hs = bf16_stats(stats);
  if (!tensor_map_2d_bf16(&ix.tmap_b, ix.Xh, (uint64_t)ix.dp, (uint64_t)ix.n_pad_tc, kTcBK, kTcBN))
    return fail(B2K_ECUDA, "cuTensorMapEncodeTiled failed for the reference rows");
  // norm columns of the reference rows and the matching query-side ones
  if ((rc = ialloc(ix, &ix.Xaug, (size_t)ix.n_pad_tc * kTcAug))) return rc;
  if ((rc = ialloc(ix, &ix.aug_ones, (size_t)kTcBM * kTcAug))) return rc;
  launch_prep_aug(&ix, ix.Xaug, ix.aug_ones, st, ix.xperm);
  B2K_CUDA(cudaGetLastError());
  B2K_CUDA(cudaStreamSynchronize(st));
  if (!tensor_map_2d_bf16(&ix.tmap_baug, ix.Xaug, kTcAug, (uint64_t)ix.n_pad_tc, kTcAug, kTcBN,
                          32) ||
      !tensor_map_2d_bf16(&ix.tmap_aaug, ix.aug_ones, kTcAug, kTcBM, kTcAug, kTcBM, 32))
    return fail(B2K_ECUDA, "cuTensorMapEncodeTiled failed for the norm columns");
  ix.bf16_ready = true;
  return B2K_OK;
}

// tf32 operand of the kind::tf32 screen, in the same row order as the bf16 one.
static int ensure_tf32(Index& ix) {
  std::lock_guard<std::mutex> lock(ix.mu);
  if (ix.tf32_ready) return B2K_OK;
  cudaStream_t st = ix.stream;
  ix.dpt = (int32_t)round_up(ix.d, kTcBKf);
  ix.n_pad_tc = round_up(ix.n, kTcBN);
  int rc;
  if ((rc = ensure_row_groups(ix))) return rc;
  if ((rc = ialloc(ix, &ix.Xt, (size_t)ix.n_pad_tc * ix.dpt))) return rc;
  launch_prep_index_tf32(&ix, ix.Xt, st, ix.xperm);
  B2K_CUDA(cudaGetLastError());
  if ((rc = ialloc(ix, &ix.Xtaug, (size_t)ix.n_pad_tc * kTcAugF))) return rc;
  if ((rc = ialloc(ix, &ix.taug_ones, (size_t)kTcBM * kTcAugF))) return rc;
  launch_prep_aug_tf32(&ix, ix.Xtaug, ix.taug_ones, st, ix.xperm);
  B2K_CUDA(cudaGetLastError());
  float stats[kStatsLen];
  B2K_CUDA(cudaMemcpyAsync(stats, ix.stats_dev, sizeof(stats), cudaMemcpyDeviceToHost, st));
  B2K_CUDA(cudaStreamSynchronize(st));
  ix.xt_max = stats[6];
  ix.ext_max = stats[7];
  if (!tensor_map_2d_f32(&ix.tmap_bt, ix.Xt, (uint64_t)ix.dpt, (uint64_t)ix.n_pad_tc, kTcBKf,
                         kTcBN) ||
      !tensor_map_2d_f32(&ix.tmap_btaug, ix.Xtaug, kTcAugF, (uint64_t)ix.n_pad_tc, kTcAugF, kTcBN,
                         32) ||
      !tensor_map_2d_f32(&ix.tmap_ataug, ix.taug_ones, kTcAugF, kTcBM, kTcAugF, kTcBM, 32))
    return fail(B2K_ECUDA, "cuTensorMapEncodeTiled failed for the tf32 operand");
  ix.tf32_ready = true;
  return B2K_OK;
}

// Whether every one of `count` values is an integer in [0, 255]: one check
// kernel and a 4-byte read (the flag is freed on every path).
static int all_u8(const float* v, int64_t count, cudaStream_t st, bool* yes) {
  *yes = false;
  int* flag = nullptr;
  int rc = dalloc(&flag, 1, st);
  if (rc) return rc;
  int h = 1;
  cudaError_t e = cudaMemsetAsync(flag, 0, sizeof(int), st);
  if (e == cudaSuccess) {
    launch_u8_check(v, count, flag, st);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpyAsync(&h, flag, sizeof(int), cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  cudaFreeAsync(flag, st);
  if (e != cudaSuccess) return fail(B2K_ECUDA, "u8 check: %s", cudaGetErrorString(e));
  *yes = h == 0;
  return B2K_OK;
}

// The exact u8 screen's operand, when every training coordinate is an
// integer in [0, 255] (checked once); *ok tells whether the index qualifies.
static int ensure_u8(Index& ix, bool* ok) {
  std::lock_guard<std::mutex> lock(ix.mu);
  *ok = false;
  if (ix.d > kU8MaxD) return B2K_OK;
  cudaStream_t st = ix.stream;
  int rc;
  if (ix.u8_state == 0) {
    bool yes = false;
    if ((rc = all_u8(ix.X, ix.n * (int64_t)ix.d, st, &yes))) return rc;
    ix.u8_state = yes ? 1 : -1;
  }
  if (ix.u8_state < 0) return B2K_OK;
  if (!ix.u8_ready) {
    // a failed build leaves nothing allocated, so a later call starts over
    struct Partial {
      Index& ix;
      bool done = false;
      ~Partial() {
        if (done) return;
        cudaFree(ix.Xu);
        cudaFree(ix.nxu);
        ix.Xu = nullptr;
        ix.nxu = nullptr;
      }
    } partial{ix};
    ix.dpu = (int32_t)round_up(ix.d, kTcBKu);
    ix.n_pad_tc = round_up(ix.n, kTcBN);
    B2K_CUDA(cudaMalloc(&ix.Xu, (size_t)ix.n_pad_tc * ix.dpu));
    B2K_CUDA(cudaMalloc(&ix.nxu, (size_t)ix.n_pad_tc * sizeof(int)));
    // padding rows: v = INT_MAX, never admitted
    launch_prep_u8(ix.X, ix.n, ix.d, ix.n_pad_tc, ix.dpu, ix.Xu, ix.nxu, nullptr, INT_MAX, st);
    B2K_CUDA(cudaGetLastError());
    B2K_CUDA(cudaStreamSynchronize(st));
    if (!tensor_map_2d(&ix.tmap_bu, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, ix.Xu, (uint64_t)ix.dpu,
                       (uint64_t)ix.n_pad_tc, kTcBKu, kTcBN, 128))
      return fail(B2K_ECUDA, "cuTensorMapEncodeTiled failed for the u8 operand");
    partial.done = true;
    ix.u8_ready = true;
  }
  *ok = true;
  return B2K_OK;
}

static int choose_splits(int64_t m_tiles, int64_t n_tiles, int64_t slots);

// Exact kNN of integer queries on a u8 index (exact_u8.cu): prep, the
// kind::i8 screen, the merge of the lists.  dQ's rows are integers in [0, 255].
static int run_u8(Index& ix, const float* dQ, int64_t m, int k, int exclude_self,
                  int64_t q_offset, double* d_dist, int64_t* d_idx, int squared, int* status,
                  cudaStream_t st, StreamFree& fr, int* splits_out) {
  int rc;
  const int64_t m_pad = round_up(m, kTcBM);
  const int64_t n_tiles = ix.n_pad_tc / kTcBN;
  const int S = choose_splits(m_pad / kTcBM, n_tiles, num_sms(ix.device));
  const int S_lists = S * tc_u8_column_groups(k);
  *splits_out = S;
  uint8_t* Qu = nullptr;
  int64_t* nq = nullptr;
  uint32_t* shared_kth = nullptr;
  if ((rc = dalloc(&Qu, (size_t)m_pad * ix.dpu, st))) return rc;
  fr.keep(Qu);
  if ((rc = dalloc(&nq, (size_t)m_pad, st))) return rc;
  fr.keep(nq);
  if ((rc = dalloc(&shared_kth, (size_t)m_pad, st))) return rc;
  fr.keep(shared_kth);
  B2K_CUDA(cudaMemsetAsync(shared_kth, 0xff, (size_t)m_pad * sizeof(uint32_t), st));
  launch_prep_u8(dQ, m, ix.d, m_pad, ix.dpu, Qu, nullptr, nq, 0, st);
  ScreenOut so{};
  so.cap = k;
  so.m_pad = (int)m_pad;
  if ((rc = dalloc(&so.lists, (size_t)S_lists * m_pad * k, st))) return rc;
  fr.keep(so.lists);
  SinkArgs sa{};
  sa.out = so;
  sa.k = k;
  sa.shared_kth = shared_kth;
  CUtensorMap tmap_a;
  if (!tensor_map_2d(&tmap_a, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, Qu, (uint64_t)ix.dpu,
                     (uint64_t)m_pad, kTcBKu, kTcBM, 128))
    return fail(B2K_ECUDA, "cuTensorMapEncodeTiled failed for the u8 query rows");
  // status[6] (zeroed by the caller) counts the claimed work units
  const int lr = launch_screen_tc_u8(&ix, &tmap_a, m, m_pad, exclude_self, q_offset, S, sa,
                                     status, st, status + 6);
  if (lr) return fail(B2K_ECUDA, "u8 tcgen05 screen launch failed: %s",
                      cudaGetErrorString((cudaError_t)lr));
  launch_u8_merge(so.lists, S_lists, m, m_pad, k, nq, squared, d_dist, d_idx, status, st);
  B2K_CUDA(cudaGetLastError());
  return B2K_OK;
}

static int ensure_pivots(Index& ix) {
  std::lock_guard<std::mutex> lock(ix.mu);
  return make_pivots(ix);
}

// Query grouping is on unless B2K_REORDER=0 (tests run both ways).
static bool reorder_enabled() {
  const char* e = getenv("B2K_REORDER");
  return !(e && e[0] == '0');
}

// Seeding pass over each query tile's home window (grouped rows): on unless
// B2K_SEED=0 (tests run both ways).
// Reference tiles per query tile of the seeding pass's home window
// (B2K_SEED_TILES overrides).  16 was the fastest of 8, 16 and 32 on 100k
// queries of the 1M x 128 mixture, k = 10: 8 tiles admit 4% more list
// entries in the main pass, 32 spend 0.22 ms more seeding than they save.
static int seed_tiles() {
  const char* e = getenv("B2K_SEED_TILES");
  const int t = e ? atoi(e) : 16;
  return t < 1 ? 1 : (t > 256 ? 256 : t);
}
static bool seed_enabled() {
  const char* e = getenv("B2K_SEED");
  return !(e && e[0] == '0');
}

// Reference splits: fill the GPU with (query tile, split) work units while
// keeping the number of candidate lists per query small.  Up to 64 splits, so
// a batch of one or two query tiles (a small call, or the second pass over a
// few uncertified rows) still spreads over most of the SMs.
constexpr int kMaxSplits = 64;
static int choose_splits(int64_t m_tiles, int64_t n_tiles, int64_t slots) {
  if (m_tiles <= 0 || n_tiles <= 0) return 1;
  int best = 1;
  double best_cost = 1e300;
  for (int S = 1; S <= kMaxSplits && S <= n_tiles; ++S) {
    const double units = (double)m_tiles * S;
    const double waves = std::ceil(units / (double)slots);
    // time ~ waves * (n_tiles / S); small penalty per extra split (more list traffic)
    const double cost = waves * std::ceil((double)n_tiles / S) * (1.0 + 0.01 * (S - 1));
    if (cost < best_cost - 1e-9) {
      best_cost = cost;
      best = S;
    }
  }
  return best;
}

static int run_exact(Index& ix, const float* dQ, int64_t m, int k, int exclude_self,
                     int64_t q_offset, double* d_dist, int64_t* d_idx, const int* rows,
                     const int* row_count, unsigned long long* counters, int* status,
                     cudaStream_t st, StreamFree& fr, bool use_scratch,
                     const int* perm = nullptr, int squared = 0) {
  ExactArgs ea{};
  ea.perm = perm;
  ea.squared = squared;
  ea.X = ix.X;
  ea.Q = dQ;
  ea.n = ix.n;
  ea.m = m;
  ea.d = ix.d;
  ea.k = k;
  ea.exclude_self = exclude_self;
  ea.q_offset = q_offset;
  ea.rows = rows;
  ea.row_count = row_count;
  ea.dist = d_dist;
  ea.idx = d_idx;
  ea.counters = counters;
  ea.status = status;
  const int sms = num_sms(ix.device);
  ea.grid = (int)std::min<int64_t>(rows ? sms : m, (int64_t)2 * sms);
  if (ea.grid <= 0) return B2K_OK;
  ea.scratch = nullptr;
  if (use_scratch) {
    int rc = dalloc(&ea.scratch, (size_t)ea.grid * ix.n, st);
    if (rc) return rc;
    fr.keep(ea.scratch);
  }
  launch_exact(ea, st);
  B2K_CUDA(cudaGetLastError());
  return B2K_OK;
}

// ext_perm (optional): the rows of dQ are already in screen order, and row i
// answers query ext_perm[i] (its output row and self index); used for the
// second pass over rows a bf16 pass could not certify.
static int knn_device_impl(Index& ix, const float* dQ, int64_t m, int k, int exclude_self,
                           int64_t q_offset, int mode, double* d_dist, int64_t* d_idx,
                           cudaStream_t st, b2k_stats* stats, const int* ext_perm = nullptr) {
  const int fm = fault_mode();
  if (fm == 2) return fail(B2K_ECUDA, "injected kernel launch failure (B2K_FAULT=launch)");
  const int squared = (mode & B2K_MODE_SQUARED) ? 1 : 0;
  const int sq_flag = squared ? B2K_MODE_SQUARED : 0;
  mode &= ~B2K_MODE_SQUARED;
  int rc;
  bool u8 = false;
  // Integer pixels: the exact u8 screen, when the index and every query
  // coordinate are integers in [0, 255] (AUTO in the bf16 screen's size range,
  // or asked for); otherwise the certified screens.
  if (m > 0 && k <= kU8MaxK && ix.range_ok &&
      (mode == B2K_MODE_U8 || (mode == B2K_MODE_AUTO && ix.d >= 16 && ix.n >= 2048))) {
    bool ok = false;
    if ((rc = ensure_u8(ix, &ok))) return rc;
    if (ok) {
      cudaSetDevice(ix.device);
      if ((rc = all_u8(dQ, m * (int64_t)ix.d, st, &ok))) return rc;
    }
    u8 = ok;
  }
  if (mode == B2K_MODE_U8) mode = B2K_MODE_AUTO;  // not integer pixels: the certified screens
  if (u8) mode = B2K_MODE_U8;
  if (mode == B2K_MODE_AUTO)
    mode = (!ix.range_ok || k > kMaxK)    ? B2K_MODE_EXACT
           : knn_on_tensor_cores(ix, m, k) ? B2K_MODE_BF16
                                           : B2K_MODE_FP32;
  if (mode != B2K_MODE_EXACT && !u8 && (!ix.range_ok || k > kMaxK)) mode = B2K_MODE_EXACT;
  if (stats) {
    memset(stats, 0, sizeof(*stats));
    stats->mode_used = mode;
  }
  if (m == 0) return B2K_OK;
  cudaSetDevice(ix.device);
  StreamFree fr{st, {}};
  // call start, screen start, screen end, call end, seeding pass end
  cudaEvent_t ev[5] = {nullptr, nullptr, nullptr, nullptr, nullptr};
  bool seeded = false;
  if (stats)
    for (auto& e : ev) cudaEventCreate(&e);
  if (stats) cudaEventRecord(ev[0], st);

  int S = 1;
  int64_t second_pass_rows = 0, second_exact_rows = 0;
  CallState* state = nullptr;
  CallState h;
  if (mode == B2K_MODE_EXACT || mode == B2K_MODE_U8) {
    if ((rc = dalloc(&state, 1, st))) return rc;
    fr.keep(state);
    B2K_CUDA(cudaMemsetAsync(state, 0, sizeof(CallState), st));
    // NaN / inf queries: flagged on the device, reported with the final state
    // (the search itself stays bounded on such inputs)
    launch_nonfinite_check(dQ, m * (int64_t)ix.d, state->status + 5, st);
    if (mode == B2K_MODE_EXACT) {
      rc = run_exact(ix, dQ, m, k, exclude_self, q_offset, d_dist, d_idx, nullptr, nullptr,
                     state->counters, state->status, st, fr, true, ext_perm, squared);
      if (rc) return rc;
    } else {
      if (stats) cudaEventRecord(ev[1], st);
      rc = run_u8(ix, dQ, m, k, exclude_self, q_offset, d_dist, d_idx, squared, state->status, st,
                  fr, &S);
      if (rc) return rc;
      if (stats) cudaEventRecord(ev[2], st);
    }
    if (stats) cudaEventRecord(ev[3], st);
    B2K_CUDA(cudaMemcpyAsync(&h, state, sizeof(h), cudaMemcpyDeviceToHost, st));
    B2K_CUDA(cudaStreamSynchronize(st));
  } else {
    if (mode == B2K_MODE_BF16 && (rc = ensure_bf16(ix))) return rc;
    if (mode == B2K_MODE_TF32 && (rc = ensure_tf32(ix))) return rc;
    const bool tf32 = mode == B2K_MODE_TF32;
    const bool tc = mode == B2K_MODE_BF16 || tf32;
    const int64_t bm = tc ? kTcBM : kSimtBM;
    const int64_t m_pad = round_up(m, bm);
    const int64_t n_tiles = tc ? ix.n_pad_tc / kTcBN : (ix.n + kSimtBN - 1) / kSimtBN;
    const int sms = num_sms(ix.device);
    S = choose_splits(m_pad / bm, n_tiles, tc ? sms : 2 * sms);
    const bool lazy = tc && tc_lazy_sink(k);  // its screen leaves V_k to the lists
    // lists per query: one per (split, column group of the screen)
    const int S_lists = S * (tc ? tc_column_groups() : simt_column_groups(kSinkKnn));
    // Group nearby queries (reorder.cu); results go back to the original rows.
    const bool grouped = !ext_perm && m >= 2048 && reorder_enabled();
    if (grouped && (rc = ensure_pivots(ix))) return rc;
    const int64_t m_tiles = m_pad / kTcBM;
    const int kSeedTiles = seed_tiles();
    // A query tile's home window is one unit of 16 tiles, so below a unit an SM
    // the pass is one long wave, and the main screen of a small call is as short.
    // Register trackers (call with the pass / without): 8,192 x 64, 6,000 queries,
    // k = 5: 231 / 198 us; 120,000 x 15, 6,000: 426 / 393; 30,000 x 64, 20,000: 535
    // / 525 and 50,000: 974 / 1,040; 120,000 x 64, 20,000: 966 / 1,057; 500,000 x 15,
    // 20,000, k = 15: 3,576 / 3,726.  A lazy tracker needs some threshold always
    // (as its pass keeps k values a row: with eight epilogue warps, B2K_TC_EW=8, its
    // two column groups hold 32, and larger k take the spread pass below.)
    const int seed_k = lazy ? 16 : k, seed_groups = tc ? tc_column_groups() : 0;
    const bool seed = tc && grouped && ix.group_start && n_tiles >= 2 * kSeedTiles &&
                      seed_enabled() &&
                      (lazy ? seed_groups * seed_k >= k
                            : m_tiles >= sms && m_tiles * n_tiles >= 256 * (int64_t)sms);
    // Lazy lists without grouped queries (m < 2048 or few rows) are seeded from
    // windows spread over the rows: an eighth of the tiles, 4 to 64 (128 where the
    // units would otherwise leave SMs idle), in as many windows as keep two units
    // an SM, at least 8.  Unseeded, a split's list sees fewer columns than it holds
    // and keeps them all, and the certify pass walks every row of the index
    // (100,000 x 20, 100 queries, k = 50: 100,000 entries a row and 1.87 ms, seeded
    // 465 and 0.15; 500,000 x 3, k = 17: 1.31 -> 0.56; 5,000 x 8, 5,000 queries,
    // k = 50: 0.86 -> 0.23).
    const bool spread = lazy && !seed && n_tiles >= 8 && seed_enabled();
    const int spread_most = (int)std::min<int64_t>(128, std::max<int64_t>(64, sms / (m_pad / bm)));
    const int spread_tiles =
        (int)std::min<int64_t>(spread_most, std::max<int64_t>(4, n_tiles / 8));
    const int spread_S = (int)std::min<int64_t>(
        spread_tiles, std::max<int64_t>(8, 2 * sms / (m_pad / bm)));
    const int spread_window = (spread_tiles + spread_S - 1) / spread_S;

    Workspace ws;
    int *hist = nullptr, *key = nullptr, *pm = nullptr, *home = nullptr, *seed_counts = nullptr;
    float *Qp = nullptr, *seed_kth = nullptr;
    unsigned long long* best64 = nullptr;
    uint32_t* shared_kth = nullptr;
    int* fb_list = nullptr;
    QueryPrep qp{};
    ScreenOut so{};
    // zeroed: the call's state and the pivot histogram of the query order
    ws.reserve(&state, 1);
    if (grouped) ws.reserve(&hist, (size_t)ix.n_pivots);
    const size_t zeroed = ws.bytes();
    if (grouped) {
      ws.reserve(&key, (size_t)m);  // nearest pivot of each query
      ws.reserve(&pm, (size_t)m);
      ws.reserve(&Qp, (size_t)m * ix.d);
      if (const size_t words = assign_scratch(&ix, m)) ws.reserve(&best64, words);
    }
    ws.reserve(&shared_kth, (size_t)m_pad);
    ws.reserve(&qp.E, (size_t)m_pad);
    ws.reserve(&qp.nq, (size_t)m_pad);  // ||y_q||^2 for certify's two-stage refinement
    if (tc && !tf32) ws.reserve(&qp.Ah, (size_t)m_pad * ix.dp);
    if (tf32) ws.reserve(&qp.At, (size_t)m_pad * ix.dpt);
    // the register trackers' lists hold 4 x kListCap entries per (split, query)
    // whatever the column groups (the lazy tracker's select is sized for kListCap)
    so.cap = (tc && !lazy) ? kListCap * 4 / tc_column_groups() : kListCap;
    so.m_pad = (int)m_pad;
    ws.reserve(&so.lists, (size_t)S_lists * m_pad * so.cap);
    ws.reserve(&so.counts, (size_t)S_lists * m_pad);
    if (!lazy) ws.reserve(&so.kth, (size_t)S_lists * m_pad * k);
    if (seed) ws.reserve(&home, (size_t)m_tiles);
    if (seed || spread) {
      const size_t seed_lists = (size_t)(spread ? spread_S : 1) * seed_groups;
      ws.reserve(&seed_counts, seed_lists * m_pad);
      ws.reserve(&seed_kth, seed_lists * m_pad * seed_k);
    }
    ws.reserve(&fb_list, (size_t)m);
    if ((rc = ws.place(st, fr))) return rc;
    int* status = state->status;
    unsigned long long* counters = state->counters;
    B2K_CUDA(cudaMemsetAsync(state, 0, zeroed, st));

    const int* perm = ext_perm;
    const float* Qs = dQ;
    if (grouped) {
      launch_query_order(&ix, dQ, m, key, hist, best64, pm, Qp, st);
      B2K_CUDA(cudaGetLastError());
      perm = pm;
      Qs = Qp;
    }
    qp.flags = status + 4;
    qp.nonfinite = status + 5;  // NaN / inf queries, reported with the final state
    qp.shared_kth = shared_kth;
    launch_prep_queries(&ix, Qs, m, m_pad, mode, qp, st);
    B2K_CUDA(cudaGetLastError());
    SinkArgs sa{};
    sa.out = so;
    sa.k = k;
    sa.shared_kth = shared_kth;
    if (stats) cudaEventRecord(ev[1], st);
    if (tc) {
      CUtensorMap tmap_a;
      const bool map_ok =
          tf32 ? tensor_map_2d_f32(&tmap_a, qp.At, (uint64_t)ix.dpt, (uint64_t)m_pad, kTcBKf,
                                   kTcBM)
               : tensor_map_2d_bf16(&tmap_a, qp.Ah, (uint64_t)ix.dp, (uint64_t)m_pad, kTcBK,
                                    kTcBM);
      if (!map_ok) return fail(B2K_ECUDA, "cuTensorMapEncodeTiled failed for the query rows");
      // Seeding: with grouped rows, a query's neighbours sit in the few
      // reference tiles of its pivot's group, which the main screen may
      // reach late; until then its lists would admit the band around the
      // nearest other clusters.  A first pass over each query tile's home
      // window publishes k-th screen values (its sink keeps no list:
      // capacity 0) to the per-query words the main screen's lists start
      // from.  A published value is the k-th smallest of real screen values
      // of the query, so it is >= the final V_k and the certificate holds.
      //
      // For k > 16 the pass runs the register tracker at its widest, 16 values
      // in each of four column groups, and launch_seed_kth takes the k-th
      // smallest of those 64: the k-th smallest of some of the query's values
      // is no smaller than that of all.  60,013 x 100 rows against themselves,
      // k = 50: list entries 88M -> 37M, screen 5.71 -> 2.38 ms (1.79 with
      // sixteen epilogue warps).  Filling the lazy tracker's own lists in the
      // pass instead cost 2.3 ms, the pass itself 0.45.
      if (seed || spread) {
        if (seed)
          launch_home_tiles(perm, key, m, ix.group_start, (int)n_tiles, kSeedTiles, home,
                            (int)m_tiles, st);
        SinkArgs sb = sa;
        sb.out.cap = 0;  // the trackers only: no list entry is written
        sb.out.counts = seed_counts;
        sb.out.kth = seed_kth;
        sb.k = seed_k;
        if (lazy) sb.shared_kth = nullptr;  // a group's 16th value is not the query's k-th
        // status[7] (zeroed above) counts this pass's claimed units
        int lr = launch_screen_tc(&ix, &tmap_a, m, m_pad, exclude_self, q_offset,
                                  spread ? spread_S : 1, qp.E, kSinkKnn, sb, status, st, perm,
                                  status + 7, tf32, home, spread ? spread_window : kSeedTiles);
        if (lr) return fail(B2K_ECUDA, "tcgen05 seeding screen launch failed: %s",
                            cudaGetErrorString((cudaError_t)lr));
        if (spread)
          launch_seed_kth_spread(seed_kth, spread_S * seed_groups, m, m_pad, k, shared_kth, st);
        else if (lazy)
          launch_seed_kth(seed_kth, seed_groups, seed_k, m, m_pad, k, shared_kth, st);
        if (stats) cudaEventRecord(ev[4], st);
        seeded = true;
      }
      // status[6] (zeroed above) counts the claimed work units
      int lr = launch_screen_tc(&ix, &tmap_a, m, m_pad, exclude_self, q_offset, S, qp.E,
                                kSinkKnn, sa, status, st, perm, status + 6, tf32);
      if (lr) return fail(B2K_ECUDA, "tcgen05 screen launch failed: %s",
                          cudaGetErrorString((cudaError_t)lr));
    } else {
      launch_screen_simt(&ix, Qs, m, m_pad, exclude_self, q_offset, S, qp.E, kSinkKnn, sa, st,
                         perm);
      B2K_CUDA(cudaGetLastError());
    }
    if (stats) cudaEventRecord(ev[2], st);
    CertifyArgs ca{};
    ca.X = ix.X;
    ca.Q = Qs;
    ca.n = ix.n;
    ca.m = m;
    ca.d = ix.d;
    ca.k = k;
    ca.S = S_lists;
    ca.scr = so;
    ca.E = qp.E;
    ca.dist = d_dist;
    ca.idx = d_idx;
    ca.fallback_list = fb_list;
    ca.fallback_count = status + 2;
    ca.counters = counters;
    ca.perm = perm;
    ca.squared = squared;
    ca.cols = tc ? ix.xperm : nullptr;  // lists of the grouped bf16 operand
    ca.status = status;
    ca.nq = qp.nq;
    ca.refined = counters + 4;
    ca.shared_kth = shared_kth;
    launch_certify(ca, st);
    B2K_CUDA(cudaGetLastError());
    // Rows the screen could not certify (a list past capacity, too many
    // candidates or survivors).  After a bf16 pass they get a second pass with
    // the fp32 screen, whose bound is ~50x tighter; otherwise (and for rows the
    // fp32 pass cannot certify) the exhaustive exact scan.
    if (!tc) {
      rc = run_exact(ix, Qs, m, k, exclude_self, q_offset, d_dist, d_idx, fb_list, status + 2,
                     counters, status, st, fr, false, perm, squared);
      if (rc) return rc;
    }
    if (stats) cudaEventRecord(ev[3], st);
    B2K_CUDA(cudaMemcpyAsync(&h, state, sizeof(h), cudaMemcpyDeviceToHost, st));
    B2K_CUDA(cudaStreamSynchronize(st));
    const int nfb = h.status[2];
    if (tc && nfb > 0 && h.status[0] == DEV_OK && !h.status[5] && !(h.status[4] & 1)) {
      float* Qfb = nullptr;
      int* pfb = nullptr;
      if ((rc = dalloc(&Qfb, (size_t)nfb * ix.d, st))) return rc;
      fr.keep(Qfb);
      if ((rc = dalloc(&pfb, (size_t)nfb, st))) return rc;
      fr.keep(pfb);
      launch_gather_fallback(Qs, ix.d, fb_list, perm, nfb, Qfb, pfb, st);
      B2K_CUDA(cudaGetLastError());
      b2k_stats sub{};
      rc = knn_device_impl(ix, Qfb, nfb, k, exclude_self, q_offset, B2K_MODE_FP32 | sq_flag,
                           d_dist, d_idx, st, &sub, pfb);
      if (rc) return rc;
      second_pass_rows = nfb;
      second_exact_rows = sub.fallback_rows;
      if (stats) {
        cudaEventRecord(ev[3], st);
        cudaEventSynchronize(ev[3]);
      }
    }
  }
  const int* hstatus = h.status;
  const unsigned long long* hcnt = h.counters;
  const int err = fm == 3 ? (int)DEV_TIMEOUT_FULL : hstatus[0];
  if (hstatus[5]) return fail(B2K_ENONFINITE, "training and query coordinates must be finite");
  if (err == DEV_TOO_MANY_TIES)
    return fail(B2K_EUNSUPPORTED,
                "more than %d training rows tie (within float64 error) with a query's k-th "
                "neighbour",
                kExactCap);
  if (err != DEV_OK) return fail(B2K_ETIMEOUT, "a bounded device wait gave up (code %d)", err);
  if (hstatus[4] & 1) {
    // Some query coordinate is outside the screens' safe range: redo exactly.
    return knn_device_impl(ix, dQ, m, k, exclude_self, q_offset, B2K_MODE_EXACT | sq_flag,
                           d_dist, d_idx, st, stats, ext_perm);
  }
  if (stats) {
    stats->splits = S;
    stats->candidates = (int64_t)hcnt[0];
    stats->list_entries = (int64_t)hcnt[1];
    stats->exact_compares = (int64_t)hcnt[2];
    stats->fallback_rows = (int64_t)hcnt[3] + second_exact_rows;
    stats->second_pass_rows = second_pass_rows;
    stats->refined = (int64_t)hcnt[4];
    float ms = 0;
    if (mode != B2K_MODE_EXACT && cudaEventElapsedTime(&ms, ev[1], ev[2]) == cudaSuccess)
      stats->screen_ms = ms;
    if (cudaEventElapsedTime(&ms, ev[0], ev[3]) == cudaSuccess) stats->total_ms = ms;
    if (seeded && cudaEventElapsedTime(&ms, ev[1], ev[4]) == cudaSuccess) stats->seed_ms = ms;
    for (auto& e : ev) cudaEventDestroy(e);
  }
  return B2K_OK;
}

// Queries of a call that one block answers.  The lazy tracker's four lists a split,
// and those of rows under 16 features, take twice what the eight-warp form and the
// fp32 screen take (16 KB against 8 a query and split), so these calls keep their
// lists within 8 GB (B2K_KNN_LIST_MB) and answer larger batches block by block:
// from about 160,000 queries at three splits, where a block fills the GPU many
// times over.  Lists half as long would take the earlier memory too, but rows
// whose certified band is wide then compact at every chunk: 1M x 128, k = 50,
// 20,000 queries 12 -> 151 ms, 100,000: 33 -> 951.
static int64_t knn_block_rows(const Index& ix, int64_t m, int k, int mode) {
  const int base = mode & ~B2K_MODE_SQUARED;
  if (base == B2K_MODE_FP32 || base == B2K_MODE_EXACT || k > kMaxK ||
      !(tc_lazy_sink(k) || ix.d < kTcAlwaysD) || tc_column_groups() != 4)
    return m;
  const char* mb = getenv("B2K_KNN_LIST_MB");
  const int64_t budget = std::max<int64_t>(1, mb ? atoll(mb) : 8192) << 20;
  if (round_up(m, kTcBM) * kMaxSplits * 4 * kListCap * (int64_t)sizeof(int2) <= budget) return m;
  const int64_t n_tiles = round_up(ix.n, kTcBN) / kTcBN;
  for (int64_t blocks = 1;; blocks *= 2) {
    const int64_t rows = round_up((m + blocks - 1) / blocks, kTcBM);
    const int S = choose_splits(rows / kTcBM, n_tiles, num_sms(ix.device));
    if (rows <= kTcBM || rows * S * 4 * kListCap * (int64_t)sizeof(int2) <= budget)
      return blocks == 1 ? m : rows;
  }
}

// The search of a public entry point: in blocks (knn_block_rows), and in smaller
// ones where the device has no memory left for a block's scratch.  Answers do not
// depend on the blocking.
constexpr int64_t kLeastBlock = 8192;  // queries below which ENOMEM is returned
static int knn_device(Index& ix, const float* dQ, int64_t m, int k, int exclude_self,
                      int64_t q_offset, int mode, double* d_dist, int64_t* d_idx,
                      cudaStream_t st, b2k_stats* stats) {
  int64_t rows = knn_block_rows(ix, m, k, mode);
  b2k_stats all{};
  for (int64_t r0 = 0; r0 < m || m == 0;) {
    const int64_t len = std::min(rows, m - r0);
    b2k_stats one{};
    const int rc = knn_device_impl(ix, dQ + r0 * ix.d, len, k, exclude_self, q_offset + r0, mode,
                                   d_dist ? d_dist + r0 * k : nullptr, d_idx + r0 * k, st,
                                   stats ? &one : nullptr);
    if (rc == B2K_ENOMEM && len > kLeastBlock) {
      rows = round_up((len + 1) / 2, kTcBM);
      continue;
    }
    if (rc) return rc;
    if (stats) {
      all.mode_used = one.mode_used;
      all.splits = one.splits;
      all.candidates += one.candidates;
      all.list_entries += one.list_entries;
      all.fallback_rows += one.fallback_rows;
      all.second_pass_rows += one.second_pass_rows;
      all.exact_compares += one.exact_compares;
      all.screen_ms += one.screen_ms;
      all.total_ms += one.total_ms;
      all.refined += one.refined;
      all.seed_ms += one.seed_ms;
      *stats = all;
    }
    r0 += len;
    if (m == 0) break;
  }
  return B2K_OK;
}

static int validate_knn(const Index& ix, int64_t m, int32_t k, int32_t exclude_self,
                        int64_t q_offset, int32_t mode) {
  if (m < 0) return fail(B2K_EINVAL, "negative query count");
  if (k <= 0) return fail(B2K_EINVAL, "Expected n_neighbors > 0. Got %d", k);
  const int64_t limit = ix.n - (exclude_self ? 1 : 0);
  if (k > limit) return fail(B2K_EINVAL, "n_neighbors must be <= %lld, got %d.", (long long)limit, k);
  if (m >= (int64_t)1 << 31) return fail(B2K_EINVAL, "query count must fit int32");
  if (exclude_self && (q_offset < 0 || q_offset + m > ix.n))
    return fail(B2K_EINVAL,
                "exclude_self requires the query matrix to be the training matrix: got %lld "
                "query rows at offset %lld and %lld training rows.",
                (long long)m, (long long)q_offset, (long long)ix.n);
  const int32_t base = mode & ~B2K_MODE_SQUARED;
  if (base < B2K_MODE_AUTO || base > B2K_MODE_U8) return fail(B2K_EINVAL, "unknown mode %d", mode);
  return B2K_OK;
}

// Shared with the other host translation units (internal.cuh).
int report_error(int code, const char* msg) { return fail(code, "%s", msg); }
int check_knn_args(const Index& ix, int64_t m, int32_t k, int32_t exclude_self,
                   int64_t q_offset) {
  return validate_knn(ix, m, k, exclude_self, q_offset, B2K_MODE_AUTO);
}
Index* index_of(b2k_index* h) { return h ? &h->ix : nullptr; }
int knn_device_run(Index& ix, const float* dQ, int64_t m, int k, int exclude_self,
                   int64_t q_offset, int mode, double* d_dist, int64_t* d_idx, cudaStream_t st) {
  return knn_device(ix, dQ, m, k, exclude_self, q_offset, mode, d_dist, d_idx, st, nullptr);
}
int injected_fault() { return fault_mode(); }
int index_prepare_bf16_stats(Index& ix, uint16_t* Xh, uint16_t* Xaug, uint16_t* ones,
                             cudaStream_t st, OperandStats* out) {
  std::lock_guard<std::mutex> lock(ix.mu);
  launch_prep_index_bf16(&ix, Xh, st);
  B2K_CUDA(cudaGetLastError());
  launch_prep_aug(&ix, Xaug, ones, st);
  B2K_CUDA(cudaGetLastError());
  float stats[kStatsLen];
  B2K_CUDA(cudaMemcpyAsync(stats, ix.stats_dev, sizeof(stats), cudaMemcpyDeviceToHost, st));
  B2K_CUDA(cudaStreamSynchronize(st));
  *out = bf16_stats(stats);
  return B2K_OK;
}

// Whether count device floats are all finite (one pass on the device).
static int device_finite(const float* dv, size_t count, cudaStream_t st, bool* ok) {
  int* flag = nullptr;
  int rc = dalloc(&flag, 1, st);
  if (rc) return rc;
  int h = 0;
  cudaMemsetAsync(flag, 0, sizeof(int), st);
  launch_nonfinite_check(dv, (int64_t)count, flag, st);
  cudaMemcpyAsync(&h, flag, sizeof(int), cudaMemcpyDeviceToHost, st);
  cudaFreeAsync(flag, st);
  B2K_CUDA(cudaStreamSynchronize(st));
  *ok = h == 0;
  return B2K_OK;
}


}  // namespace b2k

using namespace b2k;

// ===================================================================== C ABI
extern "C" {

int b2k_version(void) { return 100; }

const char* b2k_last_error(void) { return g_last_error.c_str(); }

static int create_common(int device, int64_t n, int32_t d, b2k_index** out) {
  if (!out) return fail(B2K_EINVAL, "out must not be NULL");
  *out = nullptr;
  if (n <= 0 || d <= 0) return fail(B2K_EINVAL, "X must be a nonempty two-dimensional matrix");
  if (n >= ((int64_t)1 << 31)) return fail(B2K_EINVAL, "training row count must fit int32 indices");
  if (fault_mode() == 1) return fail(B2K_ENOMEM, "injected allocation failure (B2K_FAULT=alloc)");
  return check_device(device);
}

// Keep the stream-ordered pool's memory mapped between calls (the default
// release threshold of 0 unmaps it at every synchronisation, so each query
// batch would re-map its scratch).
static void keep_pool(int device) {
  static bool done[64] = {false};
  if (device < 0 || device >= 64 || done[device]) return;
  cudaMemPool_t pool;
  if (cudaDeviceGetDefaultMemPool(&pool, device) == cudaSuccess) {
    uint64_t threshold = UINT64_MAX;
    cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &threshold);
  }
  done[device] = true;
}

static int build_from_device(b2k_index* h, const float* src, cudaMemcpyKind kind,
                             cudaStream_t user_st) {
  Index& ix = h->ix;
  B2K_CUDA(cudaSetDevice(ix.device));
  keep_pool(ix.device);
  staging_acquire(ix.device);
  ix.staging = true;
  B2K_CUDA(cudaStreamCreateWithFlags(&ix.stream, cudaStreamNonBlocking));
  const size_t bytes = (size_t)ix.n * ix.d * sizeof(float);
  int rc;
  if ((rc = ialloc(ix, &ix.X, (size_t)ix.n * ix.d))) return rc;
  if ((rc = ialloc(ix, &ix.nx32, (size_t)ix.n))) return rc;
  if ((rc = ialloc(ix, &ix.center, (size_t)ix.d))) return rc;
  if ((rc = ialloc(ix, &ix.colsum, (size_t)ix.d))) return rc;
  if ((rc = ialloc(ix, &ix.nx64, (size_t)ix.n))) return rc;
  if ((rc = ialloc(ix, &ix.stats_dev, kStatsLen))) return rc;
  if (kind == cudaMemcpyDeviceToDevice) {
    // after the caller's work on its stream (NULL: the legacy default stream),
    // which the index's own stream does not wait for by itself
    cudaEvent_t ready;
    B2K_CUDA(cudaEventCreateWithFlags(&ready, cudaEventDisableTiming));
    cudaError_t e = cudaEventRecord(ready, user_st);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(ix.stream, ready, 0);
    cudaEventDestroy(ready);
    B2K_CUDA(e);
  }
  if (kind == cudaMemcpyHostToDevice)
    B2K_CUDA(upload_host(ix.X, src, bytes, ix.stream));
  else
    B2K_CUDA(cudaMemcpyAsync(ix.X, src, bytes, kind, ix.stream));
  return finish_index(ix, ix.stream);
}

int b2k_index_create(const float* X, int64_t n, int32_t d, int32_t device, b2k_index** out) {
  int rc = create_common(device, n, d, out);
  if (rc) return rc;
  if (!X) return fail(B2K_EINVAL, "X must not be NULL");
  auto* h = new b2k_index();
  h->ix.device = device;
  h->ix.n = n;
  h->ix.d = d;
  rc = build_from_device(h, X, cudaMemcpyHostToDevice, nullptr);
  bool ok = true;
  if (!rc) rc = device_finite(h->ix.X, (size_t)n * d, h->ix.stream, &ok);
  if (!rc && !ok) rc = fail(B2K_ENONFINITE, "training coordinates must be finite");
  if (rc) {
    b2k_index_destroy(h);
    return rc;
  }
  *out = h;
  return B2K_OK;
}

int b2k_index_create_device(const float* dX, int64_t n, int32_t d, void* stream,
                            b2k_index** out) {
  int device = 0;
  cudaPointerAttributes attr;
  if (dX && cudaPointerGetAttributes(&attr, dX) == cudaSuccess && attr.type == cudaMemoryTypeDevice)
    device = attr.device;
  int rc = create_common(device, n, d, out);
  if (rc) return rc;
  if (!dX) return fail(B2K_EINVAL, "X must not be NULL");
  auto* h = new b2k_index();
  h->ix.device = device;
  h->ix.n = n;
  h->ix.d = d;
  rc = build_from_device(h, dX, cudaMemcpyDeviceToDevice, (cudaStream_t)stream);
  bool ok = true;
  if (!rc) rc = device_finite(h->ix.X, (size_t)n * d, h->ix.stream, &ok);
  if (!rc && !ok) rc = fail(B2K_ENONFINITE, "training coordinates must be finite");
  if (rc) {
    b2k_index_destroy(h);
    return rc;
  }
  *out = h;
  return B2K_OK;
}

int b2k_index_destroy(b2k_index* h) {
  if (!h) return B2K_OK;
  Index& ix = h->ix;
  cudaSetDevice(ix.device);
  if (ix.stream) cudaStreamSynchronize(ix.stream);
  // work on other streams may still read the index: as cudaFree would, wait
  cudaDeviceSynchronize();
  for (auto& b : ix.owned) {
    if (b.second)
      cudaFreeAsync(b.first, ix.stream);
    else
      cudaFree(b.first);
  }
  cudaFree(ix.Xu);
  cudaFree(ix.nxu);
  if (ix.stream) cudaStreamDestroy(ix.stream);
  if (ix.staging) staging_release(ix.device);
  delete h;
  return B2K_OK;
}

int b2k_index_shape(const b2k_index* h, int64_t* n, int32_t* d) {
  if (!h) return fail(B2K_EINVAL, "index must not be NULL");
  if (n) *n = h->ix.n;
  if (d) *d = h->ix.d;
  return B2K_OK;
}

int b2k_index_download(const b2k_index* h, float* X) {
  if (!h || !X) return fail(B2K_EINVAL, "index and X must not be NULL");
  cudaSetDevice(h->ix.device);
  B2K_CUDA(cudaMemcpy(X, h->ix.X, (size_t)h->ix.n * h->ix.d * sizeof(float),
                      cudaMemcpyDeviceToHost));
  return B2K_OK;
}

const float* b2k_index_device_data(const b2k_index* h) { return h ? h->ix.X : nullptr; }

int b2k_knn_device(b2k_index* h, const float* dQ, int64_t m, int32_t k, int32_t exclude_self,
                   int64_t q_offset, int32_t mode, double* d_dist, int64_t* d_idx, void* stream,
                   b2k_stats* stats) {
  if (!h) return fail(B2K_EINVAL, "index must not be NULL");
  Index& ix = h->ix;
  int rc = validate_knn(ix, m, k, exclude_self, q_offset, mode);
  if (rc) return rc;
  if (m > 0 && (!dQ || !d_idx)) return fail(B2K_EINVAL, "queries and indices must not be NULL");
  if (overlaps(d_idx, (size_t)m * k * 8, dQ, (size_t)m * ix.d * 4) ||
      overlaps(d_dist, (size_t)m * k * 8, dQ, (size_t)m * ix.d * 4) ||
      overlaps(d_idx, (size_t)m * k * 8, d_dist, (size_t)m * k * 8))
    return fail(B2K_EINVAL, "output buffers must not overlap inputs or each other");
  return knn_device(ix, dQ, m, k, exclude_self, q_offset, mode, d_dist, d_idx,
                    (cudaStream_t)stream, stats);
}

int b2k_knn(b2k_index* h, const float* Q, int64_t m, int32_t k, int32_t exclude_self,
            int64_t q_offset, int32_t mode, double* dist, int64_t* idx, b2k_stats* stats) {
  if (!h) return fail(B2K_EINVAL, "index must not be NULL");
  Index& ix = h->ix;
  int rc = validate_knn(ix, m, k, exclude_self, q_offset, mode);
  if (rc) return rc;
  if (m == 0) {
    if (stats) memset(stats, 0, sizeof(*stats));
    return B2K_OK;
  }
  if (!Q || !idx) return fail(B2K_EINVAL, "queries and indices must not be NULL");
  cudaSetDevice(ix.device);
  cudaStream_t st = ix.stream;
  float* dQ = nullptr;
  double* dd = nullptr;
  int64_t* di = nullptr;
  StreamFree fr{st, {}};
  if ((rc = dalloc(&dQ, (size_t)m * ix.d, st))) return rc;
  fr.keep(dQ);
  if ((rc = dalloc(&di, (size_t)m * k, st))) return rc;
  fr.keep(di);
  if (dist) {
    if ((rc = dalloc(&dd, (size_t)m * k, st))) return rc;
    fr.keep(dd);
  }
  B2K_CUDA(upload_host(dQ, Q, (size_t)m * ix.d * sizeof(float), st));
  // finiteness is checked on the device inside the search (one pass over HBM)
  rc = knn_device(ix, dQ, m, k, exclude_self, q_offset, mode, dd, di, st, stats);
  if (rc) return rc;
  B2K_CUDA(cudaMemcpyAsync(idx, di, (size_t)m * k * sizeof(int64_t), cudaMemcpyDeviceToHost, st));
  if (dist)
    B2K_CUDA(cudaMemcpyAsync(dist, dd, (size_t)m * k * sizeof(double), cudaMemcpyDeviceToHost, st));
  B2K_CUDA(cudaStreamSynchronize(st));
  return B2K_OK;
}

}  // extern "C"

// =================================================================== radius
struct b2k_radius_result {
  int device = 0;
  int64_t m = 0, nnz = 0;
  int64_t* indptr = nullptr;   // device [m+1]
  int64_t* indices = nullptr;  // device [nnz]
  double* dist = nullptr;      // device [nnz] or null
  int64_t exact_tests = 0;
  int64_t candidates = 0;
};

namespace b2k {

// Entries per list of the single-pass radius screen: B2K_RADIUS_CAP when set
// (0 = the counted two-pass form), else what a 2 GB budget for the block's
// lists allows (B2K_RADIUS_LIST_MB), a multiple of 32 in [64, 1024], or 0 when
// that budget holds fewer than 64 per list.  With 512 MB a few dense rows of
// 100,003 x 24 (30,011 queries) and 200,000 x 32 (50,000) overflowed, and their
// counted sub-call cost 0.25 of 2.57 ms and 0.2 of 4.55; `lean`, a call that found
// no memory, is held to that budget.
static int radius_list_cap(int S_lists, int64_t m_pad, bool lean) {
  if (const char* e = getenv("B2K_RADIUS_CAP")) {
    const long c = atol(e);
    return c <= 0 ? 0 : (int)std::min<long>(c, 1 << 20);
  }
  const char* mb = getenv("B2K_RADIUS_LIST_MB");
  int64_t budget = (int64_t)(mb ? atoll(mb) : 2048) << 20;
  if (lean) budget = std::min<int64_t>(budget, (int64_t)512 << 20);
  int64_t c = budget / ((int64_t)S_lists * m_pad * (int64_t)sizeof(int)) / 32 * 32;
  return c < 64 ? 0 : (int)std::min<int64_t>(c, 1024);
}

// One block of queries: screen, classify, compact, sort.  The tcgen05 screen
// runs once into fixed-capacity lists; rows that overflow a list are answered
// by a counted sub-call (count pass, then fill at scanned offsets) on those
// rows alone, the form the CUDA-core screen always uses (`counted`).
// qrows: the block row of each query for self-exclusion (sub-calls), or null.
// lean: shorter lists, and narrow rows on the fp32 screen, whose candidates are few.
// Stores device CSR pieces in `res` (which then owns them).
static int radius_block(Index& ix, const float* dQ, int64_t m, double R2, int exclude_self,
                        int64_t q_offset, bool need_distance, bool sort_results, bool admit_all,
                        cudaStream_t st, b2k_radius_result* res, const int* qrows = nullptr,
                        bool counted = false, bool sort_rows = true, bool lean = false) {
  StreamFree fr{st, {}};
  int rc;
  const int mode = !admit_all && !(lean && ix.d < kTcAlwaysD) && radius_on_tensor_cores(ix, m, R2)
                       ? B2K_MODE_BF16
                       : B2K_MODE_FP32;
  if (mode == B2K_MODE_BF16 && (rc = ensure_bf16(ix))) return rc;
  const bool tc = mode == B2K_MODE_BF16;
  const int64_t bm = tc ? kTcBM : kSimtBM;
  const int64_t m_pad = round_up(m, bm);
  const int64_t n_tiles = tc ? ix.n_pad_tc / kTcBN : (ix.n + kSimtBN - 1) / kSimtBN;
  const int sms = num_sms(ix.device);
  const int S = choose_splits(m_pad / bm, n_tiles, tc ? sms : 2 * sms);
  // candidate lists per row: one per (split, column group of the screen)
  const int S_lists = S * (tc ? tc_radius_groups() : simt_column_groups(kSinkRadiusCount));
  const int cap = (tc && !counted) ? radius_list_cap(S_lists, m_pad, lean) : 0;

  // the block's state, zeroed and read back as one; counters: [0] exact tests,
  // [2] overflowed rows, [3] candidates, [4] members
  CallState* state = nullptr;
  QueryPrep qp{};
  float* thr = nullptr;
  SinkArgs sa{};
  int64_t *roff = nullptr, *scan_scratch = nullptr;
  int* ovf = nullptr;  // single pass: overflowed rows [m] + their count
  Workspace ws;
  ws.reserve(&state, 1);
  ws.reserve(&qp.E, (size_t)m_pad);
  ws.reserve(&qp.nq, (size_t)m_pad);
  if (tc) ws.reserve(&qp.Ah, (size_t)m_pad * ix.dp);
  ws.reserve(&thr, (size_t)m_pad);
  ws.reserve(&sa.rcount, (size_t)S_lists * m_pad);
  ws.reserve(&roff, (size_t)S_lists * m_pad + 1);
  if (cap) {
    ws.reserve(&sa.rcols, (size_t)S_lists * m_pad * cap);
    ws.reserve(&ovf, (size_t)m + 1);
  }
  ws.reserve(&scan_scratch, (size_t)scan_scratch_len(m));  // count offsets, then indptr
  if ((rc = ws.place(st, fr))) return rc;
  int* status = state->status;
  unsigned long long* counters = state->counters;
  B2K_CUDA(cudaMemsetAsync(state, 0, sizeof(CallState), st));
  qp.flags = status + 4;
  qp.nonfinite = status + 5;
  launch_prep_queries(&ix, dQ, m, m_pad, mode, qp, st);
  launch_radius_threshold(qp.nq, qp.E, m, m_pad, admit_all ? INFINITY : R2, thr, st);
  B2K_CUDA(cudaGetLastError());

  sa.thr = thr;
  sa.m_pad = (int)m_pad;
  sa.rcap = cap;
  sa.roff = roff;
  if (cap) B2K_CUDA(cudaMemsetAsync(ovf + m, 0, sizeof(int), st));
  CUtensorMap tmap_a;
  if (tc && !tensor_map_2d_bf16(&tmap_a, qp.Ah, (uint64_t)ix.dp, (uint64_t)m_pad, kTcBK, kTcBM))
    return fail(B2K_ECUDA, "cuTensorMapEncodeTiled failed for the query rows");
  auto screen = [&](int kind) -> int {
    if (tc) {
      // status[6], [7] (zeroed above) count the claimed units of the two screens
      int lr = launch_screen_tc(&ix, &tmap_a, m, m_pad, exclude_self, q_offset, S, qp.E, kind,
                                sa, status, st, qrows,
                                status + (kind == kSinkRadiusFill ? 7 : 6));
      if (lr) return fail(B2K_ECUDA, "tcgen05 screen launch failed: %s",
                          cudaGetErrorString((cudaError_t)lr));
      return B2K_OK;
    }
    launch_screen_simt(&ix, dQ, m, m_pad, exclude_self, q_offset, S, qp.E, kind, sa, st, qrows);
    B2K_CUDA(cudaGetLastError());
    return B2K_OK;
  };
  if ((rc = screen(cap ? kSinkRadiusList : kSinkRadiusCount))) return rc;
  if (cap) launch_radius_overflow(sa.rcount, S_lists, m, m_pad, cap, ovf, st);
  launch_scan_split_counts(sa.rcount, S_lists, m, m_pad, roff, roff + (size_t)S_lists * m_pad,
                           scan_scratch, st);
  CallState h;
  const int* hstatus = h.status;
  B2K_CUDA(cudaMemcpyAsync(counters + 3, roff + (size_t)S_lists * m_pad, sizeof(int64_t),
                           cudaMemcpyDeviceToDevice, st));
  if (cap)
    B2K_CUDA(cudaMemcpyAsync(counters + 2, ovf + m, sizeof(int), cudaMemcpyDeviceToDevice, st));
  B2K_CUDA(cudaMemcpyAsync(&h, state, sizeof(h), cudaMemcpyDeviceToHost, st));
  B2K_CUDA(cudaStreamSynchronize(st));
  const int64_t ncand = (int64_t)h.counters[3];
  const int n_ovf = (int)h.counters[2];
  if (hstatus[5]) return fail(B2K_ENONFINITE, "training and query coordinates must be finite");
  if (hstatus[0] != DEV_OK)
    return fail(B2K_ETIMEOUT, "a bounded device wait gave up (code %d)", hstatus[0]);
  if ((hstatus[4] & 1) && !admit_all)
    return radius_block(ix, dQ, m, R2, exclude_self, q_offset, need_distance, sort_results, true,
                        st, res, qrows, counted, sort_rows, lean);
  // the candidates in one array at their scanned offsets, as training rows
  // (grouped operand rows are mapped); rows are re-sorted by index after the
  // compaction when their lists are out of index order (grouped rows, or
  // several lists per row, whose columns interleave)
  const bool grouped = tc && ix.xperm;
  int* cand = nullptr;
  if ((rc = dalloc(&cand, (size_t)ncand, st))) return rc;
  fr.keep(cand);
  if (cap) {
    launch_radius_pack(sa.rcols, cap, sa.rcount, S_lists, m, m_pad, roff,
                       grouped ? ix.xperm : nullptr, cand, ncand, status, st);
  } else {
    sa.rcols = cand;
    if ((rc = screen(kSinkRadiusFill))) return rc;
    if (grouped)
      launch_radius_pack(cand, 0, sa.rcount, S_lists, m, m_pad, roff, ix.xperm, cand, ncand,
                         status, st);
  }
  const bool unordered = grouped || S_lists > S;
  const bool keep_dist = need_distance || sort_results;

  RadiusPlanArgs ra{};
  ra.X = ix.X;
  ra.Q = dQ;
  ra.d = ix.d;
  ra.m = m;
  ra.m_pad = m_pad;
  ra.S = S_lists;
  ra.roff = roff;
  ra.rcount = sa.rcount;
  ra.cols = cand;
  // long rows (an overflow sub-call's) take a CTA each in classify and compact
  ra.wide = ncand >= (int64_t)kWideRowCandidates * m;
  ra.R2 = R2;
  ra.exact_tests = counters;
  ra.status = status;
  if ((rc = dalloc(&ra.cdist, (size_t)ncand, st))) return rc;
  fr.keep(ra.cdist);
  if ((rc = dalloc(&ra.mcount, (size_t)m, st))) return rc;
  fr.keep(ra.mcount);
  launch_classify(ra, st);

  // rows that overflowed their lists: the counted form over those rows alone
  // (their own block; self-exclusion through their block rows)
  b2k_radius_result* sub = nullptr;
  struct SubFree {
    b2k_radius_result*& r;
    ~SubFree() {
      if (r) b2k_radius_result_release(r);
    }
  } sub_free{sub};
  if (n_ovf > 0) {
    float* Qo = nullptr;
    int* orow = nullptr;
    if ((rc = dalloc(&Qo, (size_t)n_ovf * ix.d, st))) return rc;
    fr.keep(Qo);
    if ((rc = dalloc(&orow, (size_t)n_ovf, st))) return rc;
    fr.keep(orow);
    // sub-call row i answers block row ovf[i] (any order: the scatter places it)
    launch_gather_fallback(dQ, ix.d, ovf, qrows, n_ovf, Qo, orow, st);
    B2K_CUDA(cudaGetLastError());
    sub = new b2k_radius_result();
    sub->device = ix.device;
    if ((rc = radius_block(ix, Qo, n_ovf, R2, exclude_self, q_offset, keep_dist, false, admit_all,
                           st, sub, orow, true, false, lean)))
      return rc;
    launch_radius_sub_counts(ovf, n_ovf, sub->indptr, ra.mcount, st);
  }

  StreamFree out{st, {}};  // the result's arrays, until `res` owns them
  int64_t* indptr = nullptr;
  if ((rc = dalloc(&indptr, (size_t)m + 1, st))) return rc;
  out.keep(indptr);
  launch_scan_rows(ra.mcount, m, indptr, scan_scratch, st);
  B2K_CUDA(cudaGetLastError());
  B2K_CUDA(cudaMemcpyAsync(counters + 4, indptr + m, sizeof(int64_t), cudaMemcpyDeviceToDevice,
                           st));
  B2K_CUDA(cudaMemcpyAsync(&h, state, sizeof(h), cudaMemcpyDeviceToHost, st));
  B2K_CUDA(cudaStreamSynchronize(st));
  const int64_t nnz = (int64_t)h.counters[4];
  if (hstatus[0] != DEV_OK)  // the fill pass gave up (classify skipped its rows)
    return fail(B2K_ETIMEOUT, "a bounded device wait gave up (code %d)", hstatus[0]);
  int64_t* indices = nullptr;
  double* dist = nullptr;
  if ((rc = dalloc(&indices, (size_t)nnz, st))) return rc;
  out.keep(indices);
  if (keep_dist) {
    if ((rc = dalloc(&dist, (size_t)nnz, st))) return rc;
    out.keep(dist);
  }
  launch_compact(ra, indptr, indices, dist, st);
  if (sub)
    launch_radius_sub_scatter(ovf, n_ovf, sub->indptr, sub->indices, sub->dist, indptr, indices,
                              dist, st);
  B2K_CUDA(cudaGetLastError());
  if (sort_rows && (sort_results || unordered) && nnz > 1) {
    // (distance, index) order when asked for, else ascending training index
    // (grouped operand rows list candidates out of index order)
    const bool by_dist = sort_results;
    // row lists for the longer rows: [m] rows + count, twice
    int* lists = nullptr;
    if ((rc = dalloc(&lists, 2 * (size_t)m + 2, st))) return rc;
    fr.keep(lists);
    int* mid = lists;
    int* big = lists + m + 1;
    B2K_CUDA(cudaMemsetAsync(mid + m, 0, sizeof(int), st));
    B2K_CUDA(cudaMemsetAsync(big + m, 0, sizeof(int), st));
    launch_sort_rows(indptr, m, indices, dist, mid, mid + m, big, big + m,
                     (int)std::min<int64_t>(m, 4 * sms), st, by_dist);
    int nbig = 0;
    B2K_CUDA(cudaMemcpyAsync(&nbig, big + m, sizeof(int), cudaMemcpyDeviceToHost, st));
    B2K_CUDA(cudaStreamSynchronize(st));
    if (nbig > 0) {
      // scratch sized for the longest row (<= n), one slot per CTA
      int64_t P = 2;
      while (P < ix.n) P <<= 1;
      const int grid = std::min(nbig, 16);
      double* td = nullptr;
      int64_t* ti = nullptr;
      if ((rc = dalloc(&td, (size_t)grid * P, st))) return rc;
      fr.keep(td);
      if ((rc = dalloc(&ti, (size_t)grid * P, st))) return rc;
      fr.keep(ti);
      launch_sort_big_rows(indptr, big, nbig, indices, dist, td, ti, P, grid, st, by_dist);
      B2K_CUDA(cudaGetLastError());
    }
  }
  B2K_CUDA(cudaStreamSynchronize(st));
  out.ptrs.clear();
  if (!need_distance && dist) {
    cudaFree(dist);
    dist = nullptr;
  }
  res->m = m;
  res->nnz = nnz;
  res->indptr = indptr;
  res->indices = indices;
  res->dist = dist;
  res->exact_tests = (int64_t)h.counters[0] + (sub ? sub->exact_tests : 0);
  res->candidates = ncand + (sub ? sub->candidates : 0);
  return B2K_OK;
}

}  // namespace b2k

extern "C" {

int b2k_radius(b2k_index* h, const float* Q, int64_t m, double radius, int32_t exclude_self,
               int64_t q_offset, int32_t need_distance, int32_t sort_results,
               b2k_radius_result** out) {
  if (!h || !out) return fail(B2K_EINVAL, "index and out must not be NULL");
  *out = nullptr;
  Index& ix = h->ix;
  if (std::isnan(radius)) return fail(B2K_EINVAL, "radius must not be NaN");
  if (radius < 0) return fail(B2K_EINVAL, "radius must be non-negative, got %g", radius);
  if (m < 0 || m >= ((int64_t)1 << 31)) return fail(B2K_EINVAL, "invalid query count");
  if (exclude_self && (q_offset < 0 || q_offset + m > ix.n))
    return fail(B2K_EINVAL,
                "exclude_self requires the query matrix to be the training matrix: got %lld "
                "query rows at offset %lld and %lld training rows.",
                (long long)m, (long long)q_offset, (long long)ix.n);
  if (m > 0 && !Q) return fail(B2K_EINVAL, "queries must not be NULL");
  if (fault_mode() == 2) return fail(B2K_ECUDA, "injected kernel launch failure (B2K_FAULT=launch)");
  const double R2 = radius * radius;
  cudaSetDevice(ix.device);
  cudaStream_t st = ix.stream;
  auto* res = new b2k_radius_result();
  res->device = ix.device;
  if (m == 0) {
    res->m = 0;
    if (cudaMalloc(&res->indptr, sizeof(int64_t)) != cudaSuccess ||
        cudaMemset(res->indptr, 0, sizeof(int64_t)) != cudaSuccess) {
      b2k_radius_result_release(res);
      return fail(B2K_ENOMEM, "allocation failed");
    }
    *out = res;
    return B2K_OK;
  }
  float* dQ = nullptr;
  int rc = dalloc(&dQ, (size_t)m * ix.d, st);
  if (rc) {
    delete res;
    return rc;
  }
  if (const cudaError_t e = upload_host(dQ, Q, (size_t)m * ix.d * sizeof(float), st)) {
    cudaFreeAsync(dQ, st);
    delete res;
    return fail(B2K_ECUDA, "upload of the queries: %s", cudaGetErrorString(e));
  }
  // (NaN / inf queries are found by the block's query preparation)
  const bool ordered = sort_results != B2K_RADIUS_ANY_ORDER;
  for (const bool lean : {false, true}) {
    rc = radius_block(ix, dQ, m, R2, exclude_self, q_offset, need_distance != 0,
                      ordered && sort_results != 0, !ix.range_ok, st, res, nullptr, false, ordered,
                      lean);
    if (rc != B2K_ENOMEM) break;
  }
  cudaFreeAsync(dQ, st);
  cudaStreamSynchronize(st);
  if (rc) {
    b2k_radius_result_release(res);
    return rc;
  }
  *out = res;
  return B2K_OK;
}

int b2k_radius_result_nnz(const b2k_radius_result* res, int64_t* nnz) {
  if (!res || !nnz) return fail(B2K_EINVAL, "result and nnz must not be NULL");
  *nnz = res->nnz;
  return B2K_OK;
}

int b2k_radius_result_fetch(const b2k_radius_result* res, int64_t* indptr, int64_t* indices,
                            double* dist) {
  if (!res || !indptr) return fail(B2K_EINVAL, "result and indptr must not be NULL");
  if (res->nnz && !indices) return fail(B2K_EINVAL, "indices must not be NULL");
  if (dist && res->nnz && !res->dist)
    return fail(B2K_EINVAL, "distances were not requested for this result");
  cudaSetDevice(res->device);
  B2K_CUDA(cudaMemcpy(indptr, res->indptr, (size_t)(res->m + 1) * sizeof(int64_t),
                      cudaMemcpyDeviceToHost));
  if (res->nnz) {
    B2K_CUDA(cudaMemcpy(indices, res->indices, (size_t)res->nnz * sizeof(int64_t),
                        cudaMemcpyDeviceToHost));
    if (dist)
      B2K_CUDA(cudaMemcpy(dist, res->dist, (size_t)res->nnz * sizeof(double),
                          cudaMemcpyDeviceToHost));
  }
  return B2K_OK;
}

int b2k_knn_backward(const float* dQ, int64_t m, const float* dX, int64_t n, int32_t d,
                     int32_t k, const int64_t* d_idx, const float* d_grad, const float* d_dist,
                     int32_t squared, float* d_grad_q, float* d_grad_x, void* stream) {
  if (m < 0 || n <= 0 || d <= 0 || k <= 0) return fail(B2K_EINVAL, "invalid backward shapes");
  if (m > 0 && (!dQ || !dX || !d_idx || !d_grad))
    return fail(B2K_EINVAL, "backward inputs must not be NULL");
  if (!squared && !d_dist)
    return fail(B2K_EINVAL, "the euclidean backward needs the forward distances");
  if (fault_mode() == 2) return fail(B2K_ECUDA, "injected kernel launch failure (B2K_FAULT=launch)");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  int* ws = nullptr;
  int rc = 0;
  if (d_grad_x) {
    if ((rc = dalloc(&ws, knn_backward_workspace_ints(m, n, k), st))) return rc;
  }
  const int e = knn_backward(dQ, m, dX, n, d, k, d_idx, d_grad, squared ? nullptr : d_dist,
                             squared, d_grad_q, d_grad_x, ws, st);
  if (ws) cudaFreeAsync(ws, st);
  if (e) return fail(B2K_ECUDA, "backward launch failed: %s", cudaGetErrorString((cudaError_t)e));
  return B2K_OK;
}

int b2k_class_votes(const int64_t* d_idx, const double* d_dist, int64_t m, int32_t k,
                    const int32_t* d_codes, int32_t n_classes, int32_t weighted,
                    double* d_votes, int64_t* d_pred, void* stream) {
  if (m < 0 || k <= 0 || n_classes <= 0) return fail(B2K_EINVAL, "invalid vote shapes");
  if (m > 0 && (!d_idx || !d_codes || !d_votes)) return fail(B2K_EINVAL, "NULL vote buffer");
  if (weighted && !d_dist) return fail(B2K_EINVAL, "distance weights need distances");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  int* status = nullptr;
  int rc = dalloc(&status, 1, st);
  if (rc) return rc;
  B2K_CUDA(cudaMemsetAsync(status, 0, sizeof(int), st));
  launch_votes(d_idx, d_dist, m, k, d_codes, n_classes, weighted, d_votes, d_pred, status, st);
  int h = 0;
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaMemcpyAsync(&h, status, sizeof(int), cudaMemcpyDeviceToHost, st);
  cudaFreeAsync(status, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return fail(B2K_ECUDA, "votes failed: %s", cudaGetErrorString(e));
  if (h) return fail(B2K_EINVAL, "All neighbors of some sample are getting zero weights.");
  return B2K_OK;
}

// -------------------------------------------------------------- row shards
// Relative bound on |canonical distance - exact distance|: the canonical
// squared value is within g = (d+2)u/(1-(d+2)u) of the exact one (u = 2^-53),
// its square root adds half of that plus one rounding; 2g + 4u is generous.
static double shard_eps(int d) {
  const double u = 0x1p-53;
  const double g = (d + 2) * u / (1.0 - (d + 2) * u);
  return 2 * g + 4 * u;
}

static int check_shard_shapes(int32_t n_shards, int64_t m, int32_t k_in, int32_t k) {
  if (n_shards < 1 || n_shards > kMaxShards)
    return fail(B2K_EINVAL, "shard count must be in [1, %d], got %d", kMaxShards, n_shards);
  if (m < 0) return fail(B2K_EINVAL, "query count must be non-negative");
  if (k < 1 || k > kMaxShardK || k_in < k || k_in > kMaxShardK + 1)
    return fail(B2K_EINVAL,
                "shard merge needs 1 <= k <= %d and k <= k_in <= k + 1, got k=%d k_in=%d",
                kMaxShardK, k, k_in);
  return B2K_OK;
}

int b2k_shard_merge(const double* d_dist, const int64_t* d_idx, int32_t n_shards, int64_t m,
                    int32_t k_in, int32_t k, int32_t d, int64_t self_offset, double* d_out_dist,
                    int64_t* d_out_idx, int32_t* d_flags, void* stream) {
  int rc = check_shard_shapes(n_shards, m, k_in, k);
  if (rc) return rc;
  if (d < 1) return fail(B2K_EINVAL, "feature count must be positive");
  if (m == 0) return B2K_OK;
  if (!d_dist || !d_idx || !d_out_dist || !d_out_idx || !d_flags)
    return fail(B2K_EINVAL, "device pointers must not be NULL");
  launch_shard_merge(d_dist, d_idx, n_shards, m, k_in, k, self_offset, shard_eps(d), d_out_dist,
                     d_out_idx, d_flags, static_cast<cudaStream_t>(stream));
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess)
    return fail(B2K_ECUDA, "shard merge launch failed: %s", cudaGetErrorString(e));
  return B2K_OK;
}

int b2k_shard_keys(b2k_index* h, int64_t row_lo, const float* dQ, const int64_t* d_idx,
                   int32_t n_shards, int64_t m, int32_t k_in, const int64_t* d_flagged,
                   int64_t n_flagged, uint64_t* d_keys, void* stream) {
  if (!h) return fail(B2K_EINVAL, "index must not be NULL");
  int rc = check_shard_shapes(n_shards, m, k_in, k_in > 1 ? k_in - 1 : 1);
  if (rc) return rc;
  if (row_lo < 0) return fail(B2K_EINVAL, "row offset must be non-negative");
  if (n_flagged < 0 || n_flagged > m) return fail(B2K_EINVAL, "invalid flagged query count");
  if (n_flagged == 0) return B2K_OK;
  if (!dQ || !d_idx || !d_flagged || !d_keys)
    return fail(B2K_EINVAL, "device pointers must not be NULL");
  Index& ix = h->ix;
  B2K_CUDA(cudaSetDevice(ix.device));
  launch_shard_keys(nullptr, d_idx, n_shards, m, k_in, dQ, ix.X, ix.n, ix.d, row_lo, d_flagged,
                    n_flagged, d_keys, static_cast<cudaStream_t>(stream));
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess)
    return fail(B2K_ECUDA, "shard keys launch failed: %s", cudaGetErrorString(e));
  return B2K_OK;
}

int b2k_shard_resolve(const double* d_dist, const int64_t* d_idx, int32_t n_shards, int64_t m,
                      int32_t k_in, int32_t k, int64_t self_offset, const int64_t* d_flagged,
                      int64_t n_flagged, const uint64_t* d_keys, double* d_out_dist,
                      int64_t* d_out_idx, void* stream) {
  int rc = check_shard_shapes(n_shards, m, k_in, k);
  if (rc) return rc;
  if (n_flagged < 0 || n_flagged > m) return fail(B2K_EINVAL, "invalid flagged query count");
  if (n_flagged == 0) return B2K_OK;
  if (!d_dist || !d_idx || !d_flagged || !d_keys || !d_out_dist || !d_out_idx)
    return fail(B2K_EINVAL, "device pointers must not be NULL");
  launch_shard_resolve(d_dist, d_idx, n_shards, m, k_in, k, self_offset, d_flagged, n_flagged,
                       d_keys, d_out_dist, d_out_idx, static_cast<cudaStream_t>(stream));
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess)
    return fail(B2K_ECUDA, "shard resolve launch failed: %s", cudaGetErrorString(e));
  return B2K_OK;
}

int b2k_radius_result_class_votes(const b2k_radius_result* res, const int32_t* d_codes,
                                  int32_t n_classes, int32_t weighted, double* d_votes,
                                  int64_t* d_counts, void* stream) {
  if (!res) return fail(B2K_EINVAL, "result must not be NULL");
  if (n_classes <= 0) return fail(B2K_EINVAL, "n_classes must be positive");
  if (res->m > 0 && (!d_codes || !d_votes || !d_counts))
    return fail(B2K_EINVAL, "device pointers must not be NULL");
  if (weighted && res->m > 0 && res->nnz > 0 && !res->dist)
    return fail(B2K_EINVAL, "distance weights need a result with distances");
  if (res->m == 0) return B2K_OK;
  B2K_CUDA(cudaSetDevice(res->device));
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  launch_radius_votes(res->indptr, res->indices, res->dist, res->m, d_codes, n_classes,
                      weighted, d_votes, d_counts, st);
  B2K_CUDA(cudaGetLastError());
  B2K_CUDA(cudaStreamSynchronize(st));
  return B2K_OK;
}

int b2k_radius_result_class_predict(const b2k_radius_result* res, const int32_t* d_codes,
                                    int32_t n_classes, int64_t* d_pred, int64_t* d_counts,
                                    void* stream) {
  if (!res) return fail(B2K_EINVAL, "result must not be NULL");
  if (n_classes <= 0) return fail(B2K_EINVAL, "n_classes must be positive");
  if (res->m > 0 && (!d_codes || !d_pred || !d_counts))
    return fail(B2K_EINVAL, "device pointers must not be NULL");
  if (res->m == 0) return B2K_OK;
  B2K_CUDA(cudaSetDevice(res->device));
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  launch_radius_votes(res->indptr, res->indices, res->dist, res->m, d_codes, n_classes,
                      /*weighted=*/0, /*votes=*/nullptr, d_counts, st, d_pred);
  B2K_CUDA(cudaGetLastError());
  B2K_CUDA(cudaStreamSynchronize(st));
  return B2K_OK;
}

int b2k_radius_result_means(const b2k_radius_result* res, const double* d_targets,
                            int32_t weighted, double* d_means, int64_t* d_counts,
                            void* stream) {
  if (!res) return fail(B2K_EINVAL, "result must not be NULL");
  if (res->m > 0 && (!d_targets || !d_means || !d_counts))
    return fail(B2K_EINVAL, "device pointers must not be NULL");
  if (weighted && res->m > 0 && res->nnz > 0 && !res->dist)
    return fail(B2K_EINVAL, "distance weights need a result with distances");
  if (res->m == 0) return B2K_OK;
  B2K_CUDA(cudaSetDevice(res->device));
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  launch_radius_means(res->indptr, res->indices, res->dist, res->m, d_targets, weighted,
                      d_means, d_counts, st);
  B2K_CUDA(cudaGetLastError());
  B2K_CUDA(cudaStreamSynchronize(st));
  return B2K_OK;
}

int b2k_radius_result_release(b2k_radius_result* res) {
  if (!res) return B2K_OK;
  cudaSetDevice(res->device);
  cudaFree(res->indptr);
  cudaFree(res->indices);
  cudaFree(res->dist);
  delete res;
  return B2K_OK;
}

}  // extern "C"
