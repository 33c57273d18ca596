// Query ordering (and index row grouping) for the screens.
//
// A screen tile holds 128 query rows and each epilogue warp 32 of them; the
// warp leaves its fast path whenever ANY of its rows admits a column.  With
// queries in arbitrary order the rows of a warp come from unrelated parts of
// the space and the admissions of the different rows hit different column
// chunks, so nearly every chunk takes the slow path.  Grouping queries that
// are close to each other makes their admissions coincide.
//
// Method: P pivots (every (n/P)-th training row), each query goes to its
// nearest pivot (bf16 Gram form on the tensor cores: the assignment only
// affects speed, a near tie may go either way), then a
// counting sort by pivot gives the permutation `perm` (sorted position ->
// original query row) and the permuted query matrix.  Results are written
// back to the original rows by the certify / exact kernels, so the answer
// does not depend on the order.
//
// The same assignment groups the rows of the index's bf16 operand by pivot
// (b200knn.cu): a tile of grouped queries then finds its candidates in a few
// consecutive reference tiles, and the other tiles' chunks skip admission.
#include <cuda_bf16.h>

#include <algorithm>

#include "common.cuh"
#include "internal.cuh"
#include "tracker.cuh"

namespace b2k {

namespace {

constexpr int kAssignThreads = 128;  // 4 warps x 32 queries
constexpr int kMmaP = 64;            // pivots per shared-memory tile
constexpr int kMmaK = 64;            // features per shared-memory chunk
constexpr int kMmaLd = kMmaK + 8;    // padded row: conflict-free fragment loads

__global__ void pivot_rows_kernel(const float* __restrict__ X, int64_t n, int d, int P,
                                  const float* __restrict__ center, float* __restrict__ piv,
                                  float* __restrict__ pnorm) {
  const int p = blockIdx.x;
  if (p >= P) return;
  const int64_t row = (int64_t)p * (n / P);
  double s = 0.0;
  for (int i = threadIdx.x; i < d; i += 32) {
    const float y = X[row * d + i] - center[i];
    piv[(size_t)p * d + i] = y;
    s += (double)y * (double)y;
  }
  for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (threadIdx.x == 0) pnorm[p] = (float)s;
}

// The bf16 copy of the pivots, [P_pad, dpa] (multiples of 64), zero padded.
__global__ void pivots_bf16_kernel(const float* __restrict__ piv, int P, int d, int P_pad, int dpa,
                                   uint16_t* __restrict__ out) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (int64_t)P_pad * dpa) return;
  const int p = (int)(i / dpa), f = (int)(i % dpa);
  const float v = (p < P && f < d) ? piv[(size_t)p * d + f] : 0.0f;
  out[i] = __bfloat16_as_ushort(__float2bfloat16_rn(v));
}

// D (16 x 8, fp32) += A (16 x 16, bf16, row major) * B (16 x 8, bf16, column major)
__device__ __forceinline__ void mma_16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0,
                                          uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, "
      "{%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// 128 queries per block: argmin_p ||p||^2 - 2 <y_q, p> with bf16 operands and
// fp32 accumulation.  Warp w takes queries [32w, 32w + 32) (two 16-row
// fragments) against each 64-pivot tile (eight 8-column fragments), the
// features streamed through shared memory 64 at a time.  In a fragment of D,
// lane (g = lane / 4, t = lane % 4) holds rows g and g + 8, columns 2t and
// 2t + 1; it sees its pivots in ascending order and the quad's reduction
// prefers the smaller pivot on equal values, so keys are deterministic.
// Block (x, y) takes the pivot tiles [y tiles, (y + 1) tiles): with all of them
// (one y) it writes keys and histogram; with several y the blocks combine (value,
// pivot) by a 64-bit minimum in `best64` and assign_finish_kernel reads it.  A
// batch of 10,000 queries is 79 blocks: at 784 features they took 608 us one
// pivot tile after the other, half the SMs idle; split, and with 16-byte loads,
// 149 us (100,000 x 128: 250 -> 212 us by the loads alone).
// VEC: rows of a multiple of four features at 16-byte boundaries.
template <bool VEC>
__global__ void __launch_bounds__(kAssignThreads)
    assign_kernel(const float* __restrict__ Q, int64_t m, int d, const float* __restrict__ center,
                  const uint16_t* __restrict__ piv_h, int dpa, const float* __restrict__ pnorm,
                  int P, int tiles, int* __restrict__ key, int* __restrict__ hist,
                  unsigned long long* __restrict__ best64) {
  __shared__ __align__(16) uint16_t sq[kAssignThreads][kMmaLd];
  __shared__ __align__(16) uint16_t sp[kMmaP][kMmaLd];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int64_t q0 = (int64_t)blockIdx.x * kAssignThreads;
  const int p_lo = blockIdx.y * tiles * kMmaP;
  const int p_hi = min((P + kMmaP - 1) / kMmaP * kMmaP, p_lo + tiles * kMmaP);
  float best[4];  // rows 32w + 16 (i / 2) + g + 8 (i % 2)
  int best_p[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    best[i] = INFINITY;
    best_p[i] = p_lo;
  }
  for (int p0 = p_lo; p0 < p_hi; p0 += kMmaP) {
    float acc[2][8][4];
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
      for (int b = 0; b < 8; ++b)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[a][b][c] = 0.0f;
    for (int k0 = 0; k0 < dpa; k0 += kMmaK) {
      __syncthreads();
      // coalesced: consecutive threads read consecutive features of one query
      if constexpr (VEC) {
        for (int i = threadIdx.x; i < kAssignThreads * (kMmaK / 4); i += kAssignThreads) {
          const int r = i / (kMmaK / 4), k = i % (kMmaK / 4) * 4;
          const int64_t qr = q0 + r;
          const int f = k0 + k;
          float4 y = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
          if (qr < m && f < d) {
            const float4 v = *reinterpret_cast<const float4*>(Q + qr * d + f);
            y = make_float4(v.x - center[f], v.y - center[f + 1], v.z - center[f + 2],
                            v.w - center[f + 3]);
          }
          const __nv_bfloat162 lo = __floats2bfloat162_rn(y.x, y.y);
          const __nv_bfloat162 hi = __floats2bfloat162_rn(y.z, y.w);
          uint2 packed;
          packed.x = *reinterpret_cast<const uint32_t*>(&lo);
          packed.y = *reinterpret_cast<const uint32_t*>(&hi);
          *reinterpret_cast<uint2*>(&sq[r][k]) = packed;
        }
      } else
      for (int i = threadIdx.x; i < kAssignThreads * kMmaK; i += kAssignThreads) {
        const int r = i / kMmaK, k = i % kMmaK;
        const int64_t qr = q0 + r;
        const int f = k0 + k;
        const float y = (qr < m && f < d) ? Q[qr * d + f] - center[f] : 0.0f;
        sq[r][k] = __bfloat16_as_ushort(__float2bfloat16_rn(y));
      }
      for (int i = threadIdx.x; i < kMmaP * (kMmaK / 8); i += kAssignThreads) {
        const int r = i / (kMmaK / 8), c8 = i % (kMmaK / 8);
        *reinterpret_cast<uint4*>(&sp[r][c8 * 8]) =
            *reinterpret_cast<const uint4*>(piv_h + (size_t)(p0 + r) * dpa + k0 + c8 * 8);
      }
      __syncthreads();
#pragma unroll
      for (int kk = 0; kk < kMmaK; kk += 16) {
        uint32_t a[2][4];
#pragma unroll
        for (int mt = 0; mt < 2; ++mt) {
          const int r = 32 * w + 16 * mt + g;
          a[mt][0] = *reinterpret_cast<const uint32_t*>(&sq[r][kk + 2 * t]);
          a[mt][1] = *reinterpret_cast<const uint32_t*>(&sq[r + 8][kk + 2 * t]);
          a[mt][2] = *reinterpret_cast<const uint32_t*>(&sq[r][kk + 2 * t + 8]);
          a[mt][3] = *reinterpret_cast<const uint32_t*>(&sq[r + 8][kk + 2 * t + 8]);
        }
#pragma unroll
        for (int nt = 0; nt < 8; ++nt) {
          const uint32_t b0 = *reinterpret_cast<const uint32_t*>(&sp[8 * nt + g][kk + 2 * t]);
          const uint32_t b1 = *reinterpret_cast<const uint32_t*>(&sp[8 * nt + g][kk + 2 * t + 8]);
          mma_16816(acc[0][nt], a[0], b0, b1);
          mma_16816(acc[1][nt], a[1], b0, b1);
        }
      }
    }
#pragma unroll
    for (int nt = 0; nt < 8; ++nt)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int pj = p0 + 8 * nt + 2 * t + (e & 1);
        if (pj < P) {
          const float pn = pnorm[pj];
#pragma unroll
          for (int mt = 0; mt < 2; ++mt) {
            const int i = 2 * mt + (e >> 1);
            const float v = fmaf(-2.0f, acc[mt][nt][e], pn);
            if (v < best[i]) {
              best[i] = v;
              best_p[i] = pj;
            }
          }
        }
      }
  }
  // the quad's four lanes hold different pivots of the same rows
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int o = 1; o < 4; o <<= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, best[i], o);
      const int op = __shfl_xor_sync(0xffffffffu, best_p[i], o);
      if (ov < best[i] || (ov == best[i] && op < best_p[i])) {
        best[i] = ov;
        best_p[i] = op;
      }
    }
  if (t == 0) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int64_t q = q0 + 32 * w + 16 * (i >> 1) + g + 8 * (i & 1);
      if (q < m) {
        if (best64) {
          atomicMin(best64 + q, (unsigned long long)float_key(best[i]) << 32 | (uint32_t)best_p[i]);
        } else {
          key[q] = best_p[i];
          atomicAdd(hist + best_p[i], 1);
        }
      }
    }
  }
}

__global__ void assign_finish_kernel(const unsigned long long* __restrict__ best64, int64_t m,
                                     int* __restrict__ key, int* __restrict__ hist) {
  const int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= m) return;
  const int p = (int)(uint32_t)best64[q];
  key[q] = p;
  atomicAdd(hist + p, 1);
}

// Exclusive scan in place, P <= 512 (one block; a single thread took 9 to 15 us).
__global__ void __launch_bounds__(512) bin_scan_kernel(int* __restrict__ hist, int P) {
  __shared__ int warp_sum[16];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int v = (int)threadIdx.x < P ? hist[threadIdx.x] : 0;
  int incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int x = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += x;
  }
  if (lane == 31) warp_sum[w] = incl;
  __syncthreads();
  int base = 0;
  for (int i = 0; i < w; ++i) base += warp_sum[i];
  if ((int)threadIdx.x < P) hist[threadIdx.x] = base + incl - v;
}

__global__ void scatter_kernel(const int* __restrict__ key, int64_t m, int* __restrict__ cursor,
                               int* __restrict__ perm) {
  const int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= m) return;
  perm[atomicAdd(cursor + key[q], 1)] = (int)q;
}

__global__ void gather_rows_kernel(const float* __restrict__ Q, const int* __restrict__ perm,
                                   int64_t m, int d, float* __restrict__ Qp) {
  const int64_t row = (int64_t)blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32;
  if (row >= m) return;
  const float* src = Q + (size_t)perm[row] * d;
  float* dst = Qp + (size_t)row * d;
  for (int i = threadIdx.x & 31; i < d; i += 32) dst[i] = src[i];
}

// Rows the certify pass could not finish, for a second pass: their query
// rows (in the pass's row order) and their output rows.
__global__ void gather_fallback_kernel(const float* __restrict__ Qs, int d,
                                       const int* __restrict__ rows,
                                       const int* __restrict__ perm, int count,
                                       float* __restrict__ Qout, int* __restrict__ pout) {
  const int64_t i = (int64_t)blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32;
  if (i >= count) return;
  const int r = rows[i];
  const float* src = Qs + (size_t)r * d;
  float* dst = Qout + (size_t)i * d;
  for (int c = threadIdx.x & 31; c < d; c += 32) dst[c] = src[c];
  if ((threadIdx.x & 31) == 0) pout[i] = perm ? perm[r] : r;
}

__global__ void home_tiles_kernel(const int* __restrict__ perm, const int* __restrict__ key,
                                  int64_t m, const int* __restrict__ group_start, int n_tiles,
                                  int window, int* __restrict__ home, int m_tiles) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= m_tiles) return;
  const int64_t mid = min((int64_t)t * kTcBM + kTcBM / 2, m - 1);
  const int row = group_start[key[perm[mid]]];
  // one tile of margin before the group; the window stays inside the index
  int j0 = row / kTcBN - 1;
  j0 = min(j0, n_tiles - window);
  home[t] = max(j0, 0);
}

// Stable counting sort of the index's rows by pivot.  A tile is a run of rows
// one warp walks 32 at a time: lanes of one key find each other by match_any,
// so a row's place is its tile's base for the key plus the earlier rows of the
// key in the tile.  At 10^6 rows the host form it replaces (keys down, two
// passes, the permutations up) took 8 ms of an index's first query.
constexpr int kGroupWarps = 4;
constexpr int kGroupMaxP = 512;

__host__ __device__ inline int64_t group_tile_rows(int64_t n) {
  const int64_t r = (n + 2047) / 2048;  // at most 2,048 tiles
  return r < 512 ? 512 : (r + 31) / 32 * 32;
}

// counts[p][t] = rows of key p in tile t
__global__ void __launch_bounds__(kGroupWarps * 32)
    group_count_kernel(const int* __restrict__ key, int64_t n, int P, int64_t rows, int T,
                       int* __restrict__ counts) {
  __shared__ int sm[kGroupWarps][kGroupMaxP];
  const int lane = threadIdx.x & 31;
  int* cnt = sm[threadIdx.x >> 5];
  const int64_t t = (int64_t)blockIdx.x * kGroupWarps + (threadIdx.x >> 5);
  if (t >= T) return;
  for (int p = lane; p < P; p += 32) cnt[p] = 0;
  const int64_t r1 = min(n, (t + 1) * rows);
  for (int64_t r0 = t * rows; r0 < r1; r0 += 32) {
    __syncwarp();
    const int64_t r = r0 + lane;
    const int k = r < r1 ? key[r] : -1;
    const unsigned same = __match_any_sync(0xffffffffu, k);
    if (k >= 0 && lane == __ffs(same) - 1) cnt[k] += __popc(same);
  }
  __syncwarp();
  for (int p = lane; p < P; p += 32) counts[(size_t)p * T + t] = cnt[p];
}

// group_start = exclusive scan of the P <= 512 totals
__global__ void __launch_bounds__(kGroupMaxP)
    group_start_kernel(const int* __restrict__ hist, int P, int* __restrict__ group_start) {
  __shared__ int warp_sum[kGroupMaxP / 32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int v = (int)threadIdx.x < P ? hist[threadIdx.x] : 0;
  int incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int x = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += x;
  }
  if (lane == 31) warp_sum[w] = incl;
  __syncthreads();
  int base = 0;
  for (int i = 0; i < w; ++i) base += warp_sum[i];
  if ((int)threadIdx.x < P) group_start[threadIdx.x] = base + incl - v;
  if ((int)threadIdx.x == P - 1) group_start[P] = base + incl;
}

// One warp per key: counts[p][t] becomes the first position of tile t's rows
__global__ void group_scan_kernel(int* __restrict__ counts, int P, int T,
                                  const int* __restrict__ group_start) {
  const int p = blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32;
  const int lane = threadIdx.x & 31;
  if (p >= P) return;
  int carry = group_start[p];
  for (int t0 = 0; t0 < T; t0 += 32) {
    const int t = t0 + lane;
    const int v = t < T ? counts[(size_t)p * T + t] : 0;
    int incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int x = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += x;
    }
    if (t < T) counts[(size_t)p * T + t] = carry + incl - v;
    carry += __shfl_sync(0xffffffffu, incl, 31);
  }
}

__global__ void __launch_bounds__(kGroupWarps * 32)
    group_scatter_kernel(const int* __restrict__ key, int64_t n, int P, int64_t rows, int T,
                         const int* __restrict__ first, int* __restrict__ perm,
                         int* __restrict__ inv) {
  __shared__ int sm[kGroupWarps][kGroupMaxP];
  const int lane = threadIdx.x & 31;
  int* next = sm[threadIdx.x >> 5];
  const int64_t t = (int64_t)blockIdx.x * kGroupWarps + (threadIdx.x >> 5);
  if (t >= T) return;
  for (int p = lane; p < P; p += 32) next[p] = first[(size_t)p * T + t];
  const int64_t r1 = min(n, (t + 1) * rows);
  for (int64_t r0 = t * rows; r0 < r1; r0 += 32) {
    __syncwarp();
    const int64_t r = r0 + lane;
    const int k = r < r1 ? key[r] : -1;
    const unsigned same = __match_any_sync(0xffffffffu, k);
    const int pos = k >= 0 ? next[k] + __popc(same & ((1u << lane) - 1)) : 0;
    __syncwarp();
    if (k >= 0) {
      perm[pos] = (int)r;
      inv[r] = pos;
      if (lane == __ffs(same) - 1) next[k] += __popc(same);
    }
  }
}

// One thread per query: the k-th smallest of its G ascending lists of kl values
// (a k-way merge by list heads) as its shared k-th key; a query with fewer than
// k finite values keeps its key.
__device__ __forceinline__ void seed_kth_row(const float* __restrict__ kth, int G, int kl,
                                             int64_t r, int64_t m_pad, int k,
                                             uint32_t* __restrict__ shared_kth) {
  constexpr int kMaxG = 4;
  float head[kMaxG];
  int pos[kMaxG];
#pragma unroll
  for (int g = 0; g < kMaxG; ++g) {
    pos[g] = 0;
    head[g] = g < G ? kth[((size_t)g * m_pad + r) * kl] : INFINITY;
  }
  float v = INFINITY;
  for (int t = 0; t < k; ++t) {
    int b = 0;
#pragma unroll
    for (int g = 1; g < kMaxG; ++g)
      if (head[g] < head[b]) b = g;
#pragma unroll
    for (int g = 0; g < kMaxG; ++g)
      if (g == b) {
        v = head[g];
        ++pos[g];
        head[g] = pos[g] < kl ? kth[((size_t)g * m_pad + r) * kl + pos[g]] : INFINITY;
      }
  }
  if (v < INFINITY) shared_kth[r] = float_key(v);
}

__global__ void seed_kth_kernel(const float* __restrict__ kth, int G, int kl, int64_t m,
                                int64_t m_pad, int k, uint32_t* __restrict__ shared_kth) {
  const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (r < m) seed_kth_row(kth, G, kl, r, m_pad, k, shared_kth);
}

// A warp per query: each lane merges its lists (lane, lane + 32, ...) into the 16
// smallest, then the k-th smallest of those by k warp minima.  What a lane drops
// can only make the result larger, which a threshold may be.  Bound by latency:
// a few loads and k reductions; a thread per query walking the heads of 32 or
// more lists would take k times as many dependent steps.
__global__ void seed_kth_spread_kernel(const float* __restrict__ kth, int G, int64_t m,
                                       int64_t m_pad, int k, uint32_t* __restrict__ shared_kth) {
  const int lane = threadIdx.x & 31;
  const int64_t r = (int64_t)blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32;
  if (r >= m) return;
  constexpr int kL = 16;
  const uint32_t none = float_key(INFINITY);
  uint32_t key[kL];
#pragma unroll
  for (int j = 0; j < kL; ++j) key[j] = none;
  for (int g = lane; g < G; g += 32) {
    const float4* src = reinterpret_cast<const float4*>(kth + ((size_t)g * m_pad + r) * kL);
    // both ascend: the 16 smaller of (key[j], list[15 - j]) are the smallest 16,
    // a bitonic sequence
#pragma unroll
    for (int j = 0; j < kL; j += 4) {
      const float4 v = src[j / 4];
      key[kL - 1 - j] = min(key[kL - 1 - j], float_key(v.x));
      key[kL - 2 - j] = min(key[kL - 2 - j], float_key(v.y));
      key[kL - 3 - j] = min(key[kL - 3 - j], float_key(v.z));
      key[kL - 4 - j] = min(key[kL - 4 - j], float_key(v.w));
    }
#pragma unroll
    for (int h = kL / 2; h > 0; h >>= 1)
#pragma unroll
      for (int j = 0; j < kL; ++j)
        if (!(j & h)) {
          const uint32_t a = key[j], b = key[j + h];
          key[j] = min(a, b);
          key[j + h] = max(a, b);
        }
  }
  __syncwarp();
  uint32_t best = none;
  for (int t = 0; t < k; ++t) {
    best = __reduce_min_sync(0xffffffffu, key[0]);
    const unsigned who = __ballot_sync(0xffffffffu, key[0] == best);
    if (lane == __ffs(who) - 1) {
#pragma unroll
      for (int j = 0; j + 1 < kL; ++j) key[j] = key[j + 1];
      key[kL - 1] = none;
    }
  }
  if (lane == 0 && best < none) shared_kth[r] = best;
}

__global__ void seed_kth_batch_kernel(const SeedProblem* __restrict__ tab,
                                      const int64_t* __restrict__ row_start, int P,
                                      int64_t total) {
  const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= total) return;
  const int p = problem_of(row_start, P, g);
  const SeedProblem s = tab[p];
  const int64_t r = g - row_start[p];
  if (r < s.m) seed_kth_row(s.kth, 4, s.kl, r, s.m_pad, s.k, s.shared_kth);
}

}  // namespace

size_t row_group_scratch(int64_t n, int P) {
  const int64_t rows = group_tile_rows(n);
  return (size_t)((n + rows - 1) / rows) * P;
}

void launch_row_groups(const int* key, int64_t n, int P, const int* hist, int* tiles,
                       int* group_start, int* perm, int* inv, cudaStream_t st) {
  const int64_t rows = group_tile_rows(n);
  const int T = (int)((n + rows - 1) / rows);
  const unsigned grid = (unsigned)((T + kGroupWarps - 1) / kGroupWarps);
  group_count_kernel<<<grid, kGroupWarps * 32, 0, st>>>(key, n, P, rows, T, tiles);
  group_start_kernel<<<1, kGroupMaxP, 0, st>>>(hist, P, group_start);
  group_scan_kernel<<<(unsigned)((P + 3) / 4), 128, 0, st>>>(tiles, P, T, group_start);
  group_scatter_kernel<<<grid, kGroupWarps * 32, 0, st>>>(key, n, P, rows, T, tiles, perm, inv);
}

void launch_seed_kth(const float* kth, int groups, int kl, int64_t m, int64_t m_pad, int k,
                     uint32_t* shared_kth, cudaStream_t st) {
  if (m <= 0) return;
  seed_kth_kernel<<<(unsigned)((m + 127) / 128), 128, 0, st>>>(kth, groups, kl, m, m_pad, k,
                                                               shared_kth);
}

void launch_seed_kth_spread(const float* kth, int lists, int64_t m, int64_t m_pad, int k,
                            uint32_t* shared_kth, cudaStream_t st) {
  if (m <= 0) return;
  seed_kth_spread_kernel<<<(unsigned)((m + 3) / 4), 128, 0, st>>>(kth, lists, m, m_pad, k,
                                                                  shared_kth);
}

void launch_seed_kth_batch(const SeedProblem* tab, const int64_t* row_start, int P,
                           int64_t total_rows, cudaStream_t st) {
  if (total_rows <= 0) return;
  seed_kth_batch_kernel<<<(unsigned)((total_rows + 127) / 128), 128, 0, st>>>(tab, row_start, P,
                                                                              total_rows);
}

void launch_home_tiles(const int* perm, const int* key, int64_t m, const int* group_start,
                       int n_tiles, int window, int* home, int m_tiles, cudaStream_t st) {
  if (m_tiles <= 0 || m <= 0) return;
  home_tiles_kernel<<<(unsigned)((m_tiles + 127) / 128), 128, 0, st>>>(
      perm, key, m, group_start, n_tiles, window, home, m_tiles);
}

void launch_gather_fallback(const float* Qs, int d, const int* rows, const int* perm, int count,
                            float* Qout, int* pout, cudaStream_t st) {
  if (count <= 0) return;
  gather_fallback_kernel<<<(unsigned)((count + 7) / 8), 256, 0, st>>>(Qs, d, rows, perm, count,
                                                                      Qout, pout);
}

int pivot_count(int64_t n) {
  int P = 512;
  while (P > 1 && (int64_t)P * 64 > n) P >>= 1;
  return P;
}

int pivot_rows_padded(int P) { return (P + kMmaP - 1) / kMmaP * kMmaP; }
int pivot_dims_padded(int d) { return (d + kMmaK - 1) / kMmaK * kMmaK; }

void launch_pivots(const Index* ix, int P, int dpa, float* pivots, float* norms,
                   uint16_t* pivots_h, cudaStream_t st) {
  pivot_rows_kernel<<<P, 32, 0, st>>>(ix->X, ix->n, ix->d, P, ix->center, pivots, norms);
  const int64_t total = (int64_t)pivot_rows_padded(P) * dpa;
  pivots_bf16_kernel<<<(unsigned)((total + 255) / 256), 256, 0, st>>>(
      pivots, P, ix->d, pivot_rows_padded(P), dpa, pivots_h);
}

// Pivot tiles a block takes: all while the query blocks fill the GPU, else as
// few as give about four blocks an SM.
static int assign_tiles(int64_t m, int P, int sms) {
  const int64_t q_blocks = (m + kAssignThreads - 1) / kAssignThreads;
  const int all = (P + kMmaP - 1) / kMmaP;
  const int64_t ways = std::min<int64_t>(all, (4 * sms + q_blocks - 1) / q_blocks);
  return q_blocks >= 2 * sms ? all : (int)((all + ways - 1) / ways);
}

size_t assign_scratch(const Index* ix, int64_t m) {
  const int all = (ix->n_pivots + kMmaP - 1) / kMmaP;
  return assign_tiles(m, ix->n_pivots, num_sms(ix->device)) < all ? (size_t)m : 0;
}

static void launch_assign(const Index* ix, const float* Q, int64_t m, int* key, int* hist,
                          unsigned long long* best64, cudaStream_t st) {
  const int P = ix->n_pivots, all = (P + kMmaP - 1) / kMmaP;
  const int tiles = best64 ? assign_tiles(m, P, num_sms(ix->device)) : all;
  if (best64) cudaMemsetAsync(best64, 0xff, (size_t)m * sizeof(*best64), st);
  const dim3 grid((unsigned)((m + kAssignThreads - 1) / kAssignThreads),
                  (unsigned)((all + tiles - 1) / tiles));
  const bool vec = (ix->d & 3) == 0 && (reinterpret_cast<uintptr_t>(Q) & 15) == 0;
  auto kern = vec ? assign_kernel<true> : assign_kernel<false>;
  kern<<<grid, kAssignThreads, 0, st>>>(Q, m, ix->d, ix->center, ix->pivots_h, ix->pivot_dpa,
                                        ix->pivot_norms, P, tiles, key, hist, best64);
  if (best64)
    assign_finish_kernel<<<(unsigned)((m + 255) / 256), 256, 0, st>>>(best64, m, key, hist);
}

void launch_assign_rows(const Index* ix, const float* X, int64_t n, int* key, int* hist,
                        unsigned long long* best64, cudaStream_t st) {
  cudaMemsetAsync(hist, 0, (size_t)ix->n_pivots * sizeof(int), st);
  launch_assign(ix, X, n, key, hist, best64, st);
}

void launch_query_order(const Index* ix, const float* Q, int64_t m, int* key, int* hist,
                        unsigned long long* best64, int* perm, float* Qp, cudaStream_t st) {
  launch_assign(ix, Q, m, key, hist, best64, st);
  bin_scan_kernel<<<1, 512, 0, st>>>(hist, ix->n_pivots);
  scatter_kernel<<<(unsigned)((m + 255) / 256), 256, 0, st>>>(key, m, hist, perm);
  gather_rows_kernel<<<(unsigned)((m + 7) / 8), 256, 0, st>>>(Q, perm, m, ix->d, Qp);
}

}  // namespace b2k
