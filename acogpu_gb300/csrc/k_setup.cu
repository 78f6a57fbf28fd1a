// k_setup.cu -- one-time kernels of Colony::initialize (reference:
// src/Colony.cu:185-311, src/Setup.cpp:54-70): EUC_2D distances, the
// heuristic, nn-lists, the greedy tour for tau0, and state reset.
#include <cuda_runtime.h>

#include <algorithm>

#include "aco_kernels.h"

namespace aco {

// ---------------------------------------------------------------- distances
// Utils::round_distance (src/Utils.cu:212-218): float differences, double
// root, +0.5, truncation.  Differences that are whole numbers up to 2^22 (whole
// coordinates, as in the instance files) need no double: s = dx^2 + dy^2 < 2^46
// is exact, and the result is the k with k^2 - k < s <= k^2 + k.  (sqrt(s) is at
// least 2^-26 from every k + 1/2 then, far more than the roundings of the double
// root and sum.)  k is the float root's, at most one off, and two comparisons of
// whole numbers settle it.  Other differences take the double path, whose
// units are few here: n = 4096 466 us by it, 68 by whole numbers.
__device__ __forceinline__ int32_t round_distance(float dx, float dy) {
  const int ix = __float2int_rz(dx), iy = __float2int_rz(dy);
  if (fabsf(dx) <= 0x1p22f && fabsf(dy) <= 0x1p22f && __int2float_rn(ix) == dx &&
      __int2float_rn(iy) == dy) {
    const int64_t s = (int64_t)ix * ix + (int64_t)iy * iy;
    const int k = __float2int_rn(__fsqrt_rn(__ll2float_rn(s)));
    const int64_t p = (int64_t)k * (k + 1);
    return s > p ? k + 1 : k > 0 && s <= p - 2 * (int64_t)k ? k - 1 : k;
  }
  const double a = (double)dx, b = (double)dy;
  const double r = __dadd_rn(__dsqrt_rn(__dadd_rn(__dmul_rn(a, a), __dmul_rn(b, b))), 0.5);
  return __double2int_rz(r);
}

__global__ void k_distances_from_coords(const float *__restrict__ x, const float *__restrict__ y,
                                        int n, int ld, int32_t *__restrict__ dist) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  const int i = blockIdx.y;
  if (j >= ld) return;
  int32_t d = ACO_MAX_DISTANCE;
  if (j < n && i != j) d = round_distance(__fsub_rn(x[i], x[j]), __fsub_rn(y[i], y[j]));
  dist[(size_t)i * ld + j] = d;
}

cudaError_t launch_distances_from_coords(const float *x, const float *y, int n, int ld,
                                         int32_t *dist, cudaStream_t s) {
  dim3 grid((ld + 127) / 128, n);
  k_distances_from_coords<<<grid, 128, 0, s>>>(x, y, n, ld, dist);
  return cudaGetLastError();
}

__global__ void k_fill_padding_int(int32_t *mat, int n, int ld, int32_t value) {
  const int pad = ld - n;
  const int64_t total = (int64_t)n * pad;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = t / pad, j = n + t % pad;
    mat[i * ld + j] = value;
  }
}

cudaError_t launch_fill_padding_int(int32_t *mat, int n, int ld, int32_t value, cudaStream_t s) {
  if (ld == n) return cudaSuccess;
  k_fill_padding_int<<<304, 256, 0, s>>>(mat, n, ld, value);
  return cudaGetLastError();
}

// (A city's own distance may be any sentinel.)
__global__ void k_negative_distance(const int32_t *__restrict__ dist, int64_t total, int ld,
                                    int32_t *out) {
  int32_t signs = 0;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x)
    if (t % (ld + 1) != 0) signs |= dist[t];
  if (signs < 0) atomicOr(out, 1);
}

cudaError_t launch_negative_distance(const int32_t *dist, int n, int ld, int32_t *out,
                                     cudaStream_t s) {
  k_negative_distance<<<608, 256, 0, s>>>(dist, (int64_t)n * ld, ld, out);
  return cudaGetLastError();
}

__global__ void k_max_distance(const int32_t *__restrict__ dist, int n, int ld, int32_t *out) {
  int32_t best = 0;
  const int64_t total = (int64_t)n * n;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = t / n, j = t % n;
    if (i != j) best = max(best, dist[i * ld + j]);
  }
  for (int o = 16; o; o >>= 1) best = max(best, __shfl_xor_sync(kFull, best, o));
  if ((threadIdx.x & 31) == 0) atomicMax(out, best);
}

cudaError_t launch_max_distance(const int32_t *dist, int n, int ld, int32_t *out, cudaStream_t s) {
  k_max_distance<<<304, 256, 0, s>>>(dist, n, ld, out);
  return cudaGetLastError();
}

// ---------------------------------------------------------------- heuristic
// x^b for integer b >= 1 in double-float arithmetic (exact products by FMA),
// then rounded once: the correctly rounded power except within ~b*2^-46 of a
// rounding midpoint.
__device__ __forceinline__ float pow_int_cr(float x, int b) {
  if (b == 0) return 1.0f;
  if (isinf(x) || x == 0.0f) return isinf(x) ? x : 0.0f;
  float hi = x, lo = 0.0f;
  for (int i = 1; i < b; i++) {
    const float p = __fmul_rn(hi, x);
    float e = __fmaf_rn(hi, x, -p);
    e = __fmaf_rn(lo, x, e);
    const float s = __fadd_rn(p, e);
    lo = __fsub_rn(e, __fsub_rn(s, p));
    hi = s;
  }
  return hi;
}

// HURESTIC(d, beta) (inc/Colony.h:17-21) evaluated on the GPU.
__global__ void k_heuristic_device(const int32_t *__restrict__ dist, int n, int ld, float beta,
                                   float *__restrict__ eta) {
  const int64_t total = (int64_t)n * ld;
  const bool int_beta = beta == floorf(beta) && beta >= 0.0f && beta <= 64.0f;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int j = (int)(t % ld);
    const int32_t d = dist[t];
    float e = 0.0f;
    if (j < n && d != ACO_MAX_DISTANCE) {
      const float x = __frcp_rn(__int2float_rn(d));
      e = int_beta ? pow_int_cr(x, (int)beta) : powf(x, beta);
    }
    eta[t] = e;
  }
}

cudaError_t launch_heuristic_device(const int32_t *dist, int n, int ld, float beta, float *eta,
                                    cudaStream_t s) {
  k_heuristic_device<<<608, 256, 0, s>>>(dist, n, ld, beta, eta);
  return cudaGetLastError();
}

// Expansion of a per-distance table (table[d] = eta of distance d).
__global__ void k_heuristic_table(const int32_t *__restrict__ dist, int n, int ld,
                                  const float *__restrict__ table, int32_t table_len,
                                  float *__restrict__ eta, ColonyState *st) {
  const int64_t total = (int64_t)n * ld;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int j = (int)(t % ld);
    const int32_t d = dist[t];
    float e = 0.0f;
    if (j < n && d != ACO_MAX_DISTANCE) {
      if (d >= 0 && d < table_len) {
        e = table[d];
      } else {
        atomicOr(&st->error, kErrCheck);
      }
    }
    eta[t] = e;
  }
}

cudaError_t launch_heuristic_table(const int32_t *dist, int n, int ld, const float *table,
                                   int32_t table_len, float *eta, ColonyState *st,
                                   cudaStream_t s) {
  k_heuristic_table<<<608, 256, 0, s>>>(dist, n, ld, table, table_len, eta, st);
  return cudaGetLastError();
}

// ---------------------------------------------------------------- nn lists
// Stable nn order: each CTA sorts one row of 64-bit keys (distance << 32 |
// city) with a bitonic network in shared memory.  The row is staged into
// shared memory by a TMA bulk copy.  Equal distances keep city order, which
// is the rank-by-counting order of the reference GPU kernel
// (inc/Colony.cuh:101-123).
//
// Thread t of a stage with partner distance j takes the pair (i, i + j), i =
// t with a zero bit inserted at j: for j <= 32 a warp's pairs lie in 64
// consecutive keys of its own, so those stages (six of every merge) need a
// warp barrier only.  One thread a pair up to 2048 keys, 1024 threads above.
// With 1024 threads whatever the row and a block barrier a stage the 512
// instances of a batch (50 to 2000 cities) took 65 us each and n = 4096 1120 us;
// now 46 and 919.
constexpr int kSortMaxThreads = 1024;
constexpr int kMaxSortRow = 16384;
constexpr int kSortPerThread = kMaxSortRow / kSortMaxThreads;

__global__ void __launch_bounds__(kSortMaxThreads)
    k_nn_sort_stable(const int32_t *__restrict__ dist, int n, int ld, int K, int ldk,
                     int32_t *__restrict__ nn, int32_t *__restrict__ nn2, int t2, int P,
                     ColonyState *st) {
  extern __shared__ __align__(128) unsigned char smem[];
  uint64_t *keys = reinterpret_cast<uint64_t *>(smem);
  uint64_t *bar = reinterpret_cast<uint64_t *>(smem + (size_t)P * 8);
  int *flag = reinterpret_cast<int *>(bar + 1);
  const int row = blockIdx.x, tid = threadIdx.x, T = blockDim.x;
  int32_t *drow = reinterpret_cast<int32_t *>(keys);
  if (tid == 0) {
    mbar_init(bar, 1);
    fence_barrier_init();
  }
  __syncthreads();
  if (tid == 0) {
    const uint32_t bytes = (uint32_t)ld * 4u;
    mbar_arrive_expect_tx(bar, bytes);
    tma_load_1d(drow, dist + (size_t)row * ld, bytes, bar);
    *flag = mbar_wait_bounded(bar, 0, st) ? 1 : 0;
  }
  __syncthreads();
  if (!*flag) return;
  uint64_t v[kSortPerThread];  // the launch has P <= kSortPerThread * T
#pragma unroll
  for (int q = 0; q < kSortPerThread; q++) {
    const int i = tid + q * T;
    v[q] = ~0ull;
    if (i < n) v[q] = ((uint64_t)(uint32_t)drow[i] << 32) | (uint32_t)i;
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < kSortPerThread; q++) {
    const int i = tid + q * T;
    if (i < P) keys[i] = v[q];
  }
  __syncthreads();
  for (int k = 2; k <= P; k <<= 1) {
    for (int j = k >> 1; j > 0; j >>= 1) {
      for (int t = tid; t < P / 2; t += T) {
        const int i = ((t & ~(j - 1)) << 1) | (t & (j - 1));
        const uint64_t a = keys[i], b = keys[i + j];
        if ((a > b) == ((i & k) == 0)) {
          keys[i] = b;
          keys[i + j] = a;
        }
      }
      // The next stage's pairs are the warp's own unless it pairs farther
      // apart: the next merge's first stage has j = k.
      if (j > 32 || (j == 1 && k > 32))
        __syncthreads();
      else
        __syncwarp();
    }
  }
  __syncthreads();
  for (int q = tid; q < ldk; q += T)
    nn[(size_t)row * ldk + q] = q < K ? (int32_t)(uint32_t)(keys[q] & 0xffffffffu) : -1;
  if (nn2)  // the fallback's second tier: neighbours K .. K + t2 - 1
    for (int q = tid; q < kTier2; q += T)
      nn2[(size_t)row * kTier2 + q] =
          q < t2 ? (int32_t)(uint32_t)(keys[K + q] & 0xffffffffu) : -1;
}

// The same lists when only the first `need` entries of a row's order are
// wanted (the candidates and the second tier): one warp a row, no block barrier.
// It looks for a distance bound that between `need` and 32 R entries do not
// exceed (bisection from the row's largest distance; a few passes over the row
// in shared memory, as the count may fall anywhere in that range), copies those
// entries out in city order, and sorts them as 64-bit keys in registers, R a
// lane.  If no bound gives such a count -- more than 32 R - need equal distances
// at the bound -- the entries below it are kept and the first of the equal ones
// in city order, which is the order of their keys.  Rows of at most 32 R
// entries are sorted whole.
// Bound by instructions and shared memory, a few thousand cycles a row.  The
// lists of n = 4096 (k + tier = 160) took 919 us by the whole sort, now 45; those
// of 512 instances of 50 to 2000 cities (k = 20) 46 us each, now 8.
constexpr int kSelectWarps = 4;
constexpr int kMaxSelectRow = 8192;  // 4 x (32 KB + 2 KB)

template <int R>
__global__ void __launch_bounds__(kSelectWarps * 32)
    k_nn_select_stable(const int32_t *__restrict__ dist, int n, int ld, int K, int ldk,
                       int32_t *__restrict__ nn, int32_t *__restrict__ nn2, int t2,
                       ColonyState *st) {
  constexpr int CAP = 32 * R;
  extern __shared__ __align__(128) unsigned char smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int row = blockIdx.x * kSelectWarps + warp;
  if (row >= n) return;
  const int chunks = (n + 127) >> 7;  // of 128 entries, four a lane
  unsigned char *mine = smem + (size_t)warp * ((size_t)chunks * 512 + CAP * 8 + 128);
  uint32_t *d = reinterpret_cast<uint32_t *>(mine);
  uint64_t *keys = reinterpret_cast<uint64_t *>(mine + (size_t)chunks * 512);
  uint64_t *bar = keys + CAP;
  int ok = 0;
  if (lane == 0) {
    mbar_init(bar, 1);
    fence_barrier_init();
    const uint32_t bytes = (uint32_t)ld * 4u;
    mbar_arrive_expect_tx(bar, bytes);
    tma_load_1d(d, dist + (size_t)row * ld, bytes, bar);
    ok = mbar_wait_bounded(bar, 0, st) ? 1 : 0;
  }
  if (!__shfl_sync(kFull, ok, 0)) return;
  for (int q = n + lane; q < chunks * 128; q += 32) d[q] = ~0u;
  __syncwarp();
  const uint4 *d4 = reinterpret_cast<const uint4 *>(d);
  const int pads = chunks * 128 - n, need = K + (nn2 ? t2 : 0);
  const unsigned below = (1u << lane) - 1u;

  // Entries up to `bound` are kept; with `ties`, only so many of those equal to it.
  uint32_t bound = ~0u;
  int ties = 0;
  if (n > CAP) {
    auto count = [&](uint32_t t) {
      unsigned c = 0;
      for (int i = 0; i < chunks; i++) {
        const uint4 v = d4[32 * i + lane];
        c += (v.x <= t ? 1u : 0u) + (v.y <= t ? 1u : 0u) + (v.z <= t ? 1u : 0u) +
             (v.w <= t ? 1u : 0u);
      }
      return (int)__reduce_add_sync(kFull, c) - (t == ~0u ? pads : 0);
    };
    uint32_t lo = 0u, hi = 0u;  // the smallest bound with `need` entries is in [lo, hi]
    for (int i = 0; i < chunks; i++) {
      const uint4 v = d4[32 * i + lane];
      const uint32_t e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int t = 0; t < 4; t++) {
        const int city = 128 * i + 4 * lane + t;
        if (city < n && city != row) hi = max(hi, e[t]);  // its own distance may be a sentinel
      }
    }
    hi = __reduce_max_sync(kFull, hi);
    int c_hi = count(hi), c_lo = 0;  // entries up to hi, and below lo
    if (c_hi < need) {  // every entry wanted, the row's own among them
      hi = ~0u;
      c_hi = n;
    }
    while (c_hi > CAP && lo < hi) {
      const uint32_t mid = lo + ((hi - lo) >> 1);
      const int c = count(mid);
      if (c >= need) {
        hi = mid;
        c_hi = c;
      } else {
        lo = mid + 1u;
        c_lo = c;
      }
    }
    bound = hi;
    if (c_hi > CAP) ties = CAP - c_lo;  // lo == hi: the equal ones do not all fit
  }
  int kept = 0, seen = 0;
  for (int i = 0; i < chunks; i++) {
    const uint4 v = d4[32 * i + lane];
    const uint32_t e[4] = {v.x, v.y, v.z, v.w};
    const int city = 128 * i + 4 * lane;
    bool f[4];
#pragma unroll
    for (int t = 0; t < 4; t++) f[t] = city + t < n && e[t] <= bound;
    if (ties > 0) {
      int r = seen;
#pragma unroll
      for (int t = 0; t < 4; t++) {
        const unsigned b = __ballot_sync(kFull, f[t] && e[t] == bound);
        r += __popc(b & below);
        seen += __popc(b);
      }
#pragma unroll
      for (int t = 0; t < 4; t++) {
        const bool tie = f[t] && e[t] == bound;
        if (tie && r >= ties) f[t] = false;
        r += tie ? 1 : 0;
      }
    }
    int pos = kept;
#pragma unroll
    for (int t = 0; t < 4; t++) {
      const unsigned b = __ballot_sync(kFull, f[t]);
      pos += __popc(b & below);
      kept += __popc(b);
    }
#pragma unroll
    for (int t = 0; t < 4; t++)
      if (f[t] && pos < CAP) keys[pos++] = ((uint64_t)e[t] << 32) | (uint32_t)(city + t);
  }
  for (int q = kept + lane; q < CAP; q += 32) keys[q] = ~0ull;
  __syncwarp();
  uint64_t x[R];  // the order in which they enter does not matter
#pragma unroll
  for (int r = 0; r < R; r++) x[r] = keys[32 * r + lane];
  __syncwarp();
  // Bitonic: lane l, register r holds index l R + r.
#pragma unroll
  for (int k = 2; k <= CAP; k <<= 1) {
#pragma unroll
    for (int j = k >> 1; j > 0; j >>= 1) {
      if (j >= R) {
        const bool low = (lane & (j / R)) == 0, up = (lane * R & k) == 0;
#pragma unroll
        for (int r = 0; r < R; r++) {
          const uint64_t y = __shfl_xor_sync(kFull, x[r], j / R);
          x[r] = ((x[r] < y) == (low == up)) ? x[r] : y;
        }
      } else {
#pragma unroll
        for (int r = 0; r < R; r++) {
          if (r & j) continue;
          const bool up = ((lane * R + r) & k) == 0;
          const uint64_t a = x[r], b = x[r | j];
          const bool swap = (a > b) == up;
          x[r] = swap ? b : a;
          x[r | j] = swap ? a : b;
        }
      }
    }
  }
#pragma unroll
  for (int r = 0; r < R; r++) keys[lane * R + r] = x[r];
  __syncwarp();
  for (int q = lane; q < ldk; q += 32)
    nn[(size_t)row * ldk + q] = q < K ? (int32_t)(uint32_t)keys[q] : -1;
  if (nn2)
    for (int q = lane; q < kTier2; q += 32)
      nn2[(size_t)row * kTier2 + q] = q < t2 ? (int32_t)(uint32_t)keys[K + q] : -1;
}

template <int R>
static cudaError_t launch_select(const int32_t *dist, int n, int ld, int K, int ldk, int32_t *nn,
                                 ColonyState *st, cudaStream_t s, int32_t *nn2, int t2) {
  const size_t smem = (size_t)kSelectWarps * ((size_t)((n + 127) / 128) * 512 + 32 * R * 8 + 128);
  if (smem > 48 * 1024) {
    const cudaError_t e = open_smem((const void *)k_nn_select_stable<R>, smem, device_max_smem());
    if (e != cudaSuccess) return e;
  }
  k_nn_select_stable<R><<<(n + kSelectWarps - 1) / kSelectWarps, kSelectWarps * 32, smem, s>>>(
      dist, n, ld, K, ldk, nn, nn2, t2, st);
  return cudaGetLastError();
}

cudaError_t launch_nn_sort_stable(const int32_t *dist, int n, int ld, int K, int ldk, int32_t *nn,
                                  ColonyState *st, cudaStream_t s, int32_t *nn2, int t2) {
  if (nn2 && (t2 < 0 || t2 > kTier2 || K + t2 > n - 1)) return cudaErrorInvalidValue;
  if (n > kMaxSortRow) return cudaErrorInvalidValue;
  // Selection where the wanted entries leave the bisection room below the keys
  // that a warp sorts, and four rows fit in shared memory.
  const int need = K + (nn2 ? t2 : 0);
  if (n <= kMaxSelectRow) {
    if (n <= 128 || need <= 64)
      return launch_select<4>(dist, n, ld, K, ldk, nn, st, s, nn2, t2);
    if (n <= 256 || need <= 192)
      return launch_select<8>(dist, n, ld, K, ldk, nn, st, s, nn2, t2);
  }
  int P = 1;
  while (P < n) P <<= 1;
  if (P < 64) P = 64;  // one warp's keys, and the row's pitch fits (ld <= 2 P)
  const int threads = P / 2 < kSortMaxThreads ? P / 2 : kSortMaxThreads;
  const size_t smem = (size_t)P * 8 + 16;
  if (smem > 48 * 1024) {
    const cudaError_t e = open_smem((const void *)k_nn_sort_stable, smem, device_max_smem());
    if (e != cudaSuccess) return e;
  }
  k_nn_sort_stable<<<n, threads, smem, s>>>(dist, n, ld, K, ldk, nn, nn2, t2, P, st);
  return cudaGetLastError();
}

// Reference CPU order: the permutation Utils::sort2 (src/Utils.cu:136-159)
// produces, ties included.  One thread per row runs the same quicksort
// (middle pivot, pivot kept in the left part) with an explicit stack; the
// smaller part is processed first, so the stack depth stays below 2*log2(n).
// The subranges are disjoint, so the order in which they are processed does
// not change the result.
constexpr int kQsortStack = 96;

__global__ void k_nn_ref_qsort(const int32_t *__restrict__ dist, int n, int ld,
                               int32_t *__restrict__ scratch, int32_t *__restrict__ nn, int ldk,
                               ColonyState *st) {
  const int row = blockIdx.x * blockDim.x + threadIdx.x;
  if (row >= n) return;
  int32_t *v = scratch + (size_t)row * ld;
  int32_t *v2 = nn + (size_t)row * ldk;
  for (int i = 0; i < n; i++) {
    v[i] = dist[(size_t)row * ld + i];
    v2[i] = i;
  }
  int stack[kQsortStack];
  int sp = 0, left = 0, right = n - 1;
  for (;;) {
    if (left < right) {
      const int mid = (left + right) / 2;
      int t = v[left]; v[left] = v[mid]; v[mid] = t;
      t = v2[left]; v2[left] = v2[mid]; v2[mid] = t;
      int last = left;
      const int pivot = v[left];
      for (int k = left + 1; k <= right; k++) {
        const int vk = v[k];
        if (vk < pivot) {
          ++last;
          t = v[last]; v[last] = vk; v[k] = t;
          t = v2[last]; v2[last] = v2[k]; v2[k] = t;
        }
      }
      t = v[left]; v[left] = v[last]; v[last] = t;
      t = v2[left]; v2[left] = v2[last]; v2[last] = t;
      // parts [left, last] and [last+1, right]
      int al = left, ar = last, bl = last + 1, br = right;
      if (ar - al > br - bl) {
        int tl = al, tr = ar;
        al = bl; ar = br; bl = tl; br = tr;
      }
      // (al, ar) is the smaller part: continue with it, push the larger.
      if (sp + 2 > kQsortStack) {
        atomicOr(&st->error, kErrCheck);
        return;
      }
      stack[sp++] = bl;
      stack[sp++] = br;
      left = al;
      right = ar;
    } else {
      if (sp == 0) break;
      right = stack[--sp];
      left = stack[--sp];
    }
  }
}

cudaError_t launch_nn_ref_qsort(const int32_t *dist, int n, int ld, int32_t *scratch, int32_t *nn,
                                int ldk, ColonyState *st, cudaStream_t s) {
  k_nn_ref_qsort<<<(n + 63) / 64, 64, 0, s>>>(dist, n, ld, scratch, nn, ldk, st);
  return cudaGetLastError();
}

// The same quicksort with the row in shared memory, for rows that the warp
// version below has no room for (n above about 11 600): one warp per row, the
// warp copies the row's distances in (coalesced) and its sorted ids out,
// lane 0 runs the sort (the partition is sequential by definition: its swaps
// fix the order of ties).  Distances and ids sit interleaved, one 8-byte
// pair per entry, so a swap is one 8-byte load and store each way.  A
// shared-memory access costs about a tenth of the scattered L2 accesses of
// the global version (one thread per row, rows ld apart).
__global__ void k_nn_ref_qsort_smem(const int32_t *__restrict__ dist, int n, int ld,
                                    int32_t *__restrict__ nn, int ldk, ColonyState *st) {
  extern __shared__ __align__(16) int2 qs_rows[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int row = blockIdx.x * (blockDim.x >> 5) + warp;
  if (row >= n) return;  // warp-uniform
  int2 *v = qs_rows + (size_t)warp * n;
  for (int i = lane; i < n; i += 32) v[i] = make_int2(dist[(size_t)row * ld + i], i);
  __syncwarp();
  if (lane == 0) {
    int stack[kQsortStack];
    int sp = 0, left = 0, right = n - 1;
    bool ok = true;
    for (;;) {
      if (left < right) {
        const int mid = (left + right) / 2;
        int2 t = v[left];
        v[left] = v[mid];
        v[mid] = t;
        int last = left;
        const int pivot = v[left].x;
        for (int k = left + 1; k <= right; k++) {
          const int2 vk = v[k];
          if (vk.x < pivot) {
            ++last;
            v[k] = v[last];
            v[last] = vk;
          }
        }
        t = v[left];
        v[left] = v[last];
        v[last] = t;
        int al = left, ar = last, bl = last + 1, br = right;
        if (ar - al > br - bl) {
          const int tl = al, tr = ar;
          al = bl;
          ar = br;
          bl = tl;
          br = tr;
        }
        if (sp + 2 > kQsortStack) {
          ok = false;
          break;
        }
        stack[sp++] = bl;
        stack[sp++] = br;
        left = al;
        right = ar;
      } else {
        if (sp == 0) break;
        right = stack[--sp];
        left = stack[--sp];
      }
    }
    if (!ok) atomicOr(&st->error, kErrCheck);
  }
  __syncwarp();
  for (int i = lane; i < n; i += 32) nn[(size_t)row * ldk + i] = v[i].y;
}

int nn_ref_qsort_smem_rows(int n, int max_smem) {
  const int per_row = n * 8;
  int rows = per_row > 0 ? (max_smem - 1024) / per_row : 0;
  return rows > 8 ? 8 : rows;
}

// The same permutation with the partitions in parallel, one warp a row.
//
// The partition (pivot in front, then every smaller entry swapped to the end
// of the smaller ones) moves the j-th smaller entry, from position p_j, to
// position j, and the entry it finds at j -- one that is not smaller -- to
// p_j.  So an entry at position x that is not smaller ends where x -> p_x,
// repeated while x <= L (the number of smaller entries), leaves off: the
// chain grows strictly, and has about log2(L / x) links when half the entries
// are smaller.  A warp finds the p_j with ballots and scatters the segment
// through a second buffer.  Segments of at most 32 entries (about n / 20 of
// them) are left to single lanes, which run the sequential sort on them.
//
// A warp holds one row: entries and their copy (int2 each), p (int16), the
// list of small segments (two int16 each): 20 bytes a city.  Against lane 0
// sorting the row alone: n = 783 544 -> 166 us, n = 2392 (four rows an SM) 3.67
// -> 1.86 ms, eight colonies of n = 1000 at once 1160 -> 381 us each.
constexpr int kQsortSmall = 32;

__host__ __device__ constexpr size_t nn_ref_warp_row_bytes(int n) {
  return ((size_t)n * 20 + 15 + 64) / 16 * 16;
}

__global__ void k_nn_ref_qsort_warp(const int32_t *__restrict__ dist, int n, int ld,
                                    int32_t *__restrict__ nn, int ldk, ColonyState *st) {
  extern __shared__ __align__(16) unsigned char qw_rows[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int row = blockIdx.x * (blockDim.x >> 5) + warp;
  if (row >= n) return;  // warp-uniform
  int2 *v = reinterpret_cast<int2 *>(qw_rows + (size_t)warp * nn_ref_warp_row_bytes(n));
  int2 *tmp = v + n;
  uint32_t *small = reinterpret_cast<uint32_t *>(tmp + n);  // at most n / 2 of two or more
  uint16_t *p = reinterpret_cast<uint16_t *>(small + (n / 2 + 1));
  for (int i = lane; i < n; i += 32) v[i] = make_int2(dist[(size_t)row * ld + i], i);
  __syncwarp();
  const unsigned lt = (1u << lane) - 1u;
  int stack[kQsortStack];
  int sp = 0, left = 0, right = n - 1, nsmall = 0;
  bool ok = true;
  for (;;) {
    if (right - left + 1 > kQsortSmall) {
      if (lane == 0) {
        const int mid = (left + right) / 2;
        const int2 t = v[left];
        v[left] = v[mid];
        v[mid] = t;
      }
      __syncwarp();
      const int2 pivot = v[left];
      int L = 0;
      for (int base = left + 1; base <= right; base += 32) {
        const int k = base + lane;
        const bool less = k <= right && v[k].x < pivot.x;
        const unsigned b = __ballot_sync(kFull, less);
        if (less) p[left + L + __popc(b & lt) + 1] = (uint16_t)k;
        L += __popc(b);
      }
      __syncwarp();
      int before = 0;
      for (int base = left + 1; base <= right; base += 32) {
        const int k = base + lane;
        const bool in = k <= right;
        const int2 e = in ? v[k] : make_int2(0, 0);
        const bool less = in && e.x < pivot.x;
        const unsigned b = __ballot_sync(kFull, less);
        if (in) {
          int x = k;
          if (less) {
            x = left + before + __popc(b & lt) + 1;
            if (x == left + L) x = left;  // the last swap, with the pivot
          } else {
            while (x <= left + L) x = p[x];
          }
          tmp[x] = e;
        }
        before += __popc(b);
      }
      if (lane == 0) tmp[left + L] = pivot;
      __syncwarp();
      for (int k = left + lane; k <= right; k += 32) v[k] = tmp[k];
      __syncwarp();
      int al = left, ar = left + L, bl = left + L + 1, br = right;
      if (ar - al > br - bl) {
        const int tl = al, tr = ar;
        al = bl;
        ar = br;
        bl = tl;
        br = tr;
      }
      if (sp + 2 > kQsortStack) {  // the smaller part first: never
        ok = false;
        break;
      }
      stack[sp++] = bl;
      stack[sp++] = br;
      left = al;
      right = ar;
    } else {
      if (right > left) {
        if (lane == 0) small[nsmall] = (uint32_t)left | ((uint32_t)right << 16);
        nsmall++;
      }
      if (sp == 0) break;
      right = stack[--sp];
      left = stack[--sp];
    }
  }
  __syncwarp();
  for (int q = lane; q < nsmall; q += 32) {
    left = (int)(small[q] & 0xffffu);
    right = (int)(small[q] >> 16);
    sp = 0;
    for (;;) {
      if (left < right) {
        const int mid = (left + right) / 2;
        int2 t = v[left];
        v[left] = v[mid];
        v[mid] = t;
        int last = left;
        const int pivot = v[left].x;
        for (int k = left + 1; k <= right; k++) {
          const int2 vk = v[k];
          if (vk.x < pivot) {
            ++last;
            v[k] = v[last];
            v[last] = vk;
          }
        }
        t = v[left];
        v[left] = v[last];
        v[last] = t;
        int al = left, ar = last, bl = last + 1, br = right;
        if (ar - al > br - bl) {
          const int tl = al, tr = ar;
          al = bl;
          ar = br;
          bl = tl;
          br = tr;
        }
        stack[sp++] = bl;  // at most five levels of 32 entries
        stack[sp++] = br;
        left = al;
        right = ar;
      } else {
        if (sp == 0) break;
        right = stack[--sp];
        left = stack[--sp];
      }
    }
  }
  if (!ok && lane == 0) atomicOr(&st->error, kErrCheck);
  __syncwarp();
  for (int i = lane; i < n; i += 32) nn[(size_t)row * ldk + i] = v[i].y;
}

// Rows a CTA holds within max_smem bytes (at most 8; 0: none fits).
static int nn_ref_warp_rows(int n, int max_smem) {
  if (n > 65535) return 0;
  const int rows = (int)((max_smem - 1024) / nn_ref_warp_row_bytes(n));
  return rows > 8 ? 8 : rows;
}

cudaError_t launch_nn_ref_qsort_smem(const int32_t *dist, int n, int ld, int32_t *nn, int ldk,
                                     ColonyState *st, int max_smem, int sms, cudaStream_t s) {
  if (const int wr = nn_ref_warp_rows(n, max_smem)) {
    // Whole rows a CTA, and CTAs for every SM before rows share one.
    const int rows = std::max(1, std::min(wr, n / std::max(1, sms)));
    const size_t smem = (size_t)rows * nn_ref_warp_row_bytes(n);
    const cudaError_t e = open_smem((const void *)k_nn_ref_qsort_warp, smem, max_smem);
    if (e != cudaSuccess) return e;
    k_nn_ref_qsort_warp<<<(n + rows - 1) / rows, rows * 32, smem, s>>>(dist, n, ld, nn, ldk, st);
    return cudaGetLastError();
  }
  const int rows = nn_ref_qsort_smem_rows(n, max_smem);
  if (rows < 1) return cudaErrorInvalidValue;
  const size_t smem = (size_t)rows * n * 8;
  const cudaError_t e = open_smem((const void *)k_nn_ref_qsort_smem, smem, max_smem);
  if (e != cudaSuccess) return e;
  k_nn_ref_qsort_smem<<<(n + rows - 1) / rows, rows * 32, smem, s>>>(dist, n, ld, nn, ldk, st);
  return cudaGetLastError();
}

__global__ void k_gather_nn_f32(const float *__restrict__ src, int n, int ld,
                                const int32_t *__restrict__ nn, int K, int ldk,
                                float *__restrict__ dst) {
  const int64_t total = (int64_t)n * ldk;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t j = t / ldk;
    const int r = (int)(t % ldk);
    dst[t] = r < K ? src[j * ld + nn[t]] : 0.0f;
  }
}

cudaError_t launch_gather_nn_f32(const float *src, int n, int ld, const int32_t *nn, int K, int ldk,
                                 float *dst, cudaStream_t s) {
  k_gather_nn_f32<<<608, 256, 0, s>>>(src, n, ld, nn, K, ldk, dst);
  return cudaGetLastError();
}

// Whether the candidate heuristic is anything but the plain heuristic in
// candidate order (bit for bit): full rows are summed from the plain choice
// matrix only while the two agree.  Run after a checkpoint rewrote eta_nn; the
// prior's own kernel compares while it writes (as a launch of its own after it
// this took 4 to 8 us of an application's 70 to 300).
__global__ void k_prior_set(ColonyDev c) {
  const int64_t total = (int64_t)c.n * c.K;
  bool differs = false;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t j = t / c.K;
    const int r = (int)(t % c.K);
    const float plain = c.eta[j * c.ld + c.nn[j * c.ldk + r]];
    differs |= __float_as_uint(c.eta_nn[j * c.ldk + r]) != __float_as_uint(plain);
  }
  if (__any_sync(kFull, differs) && (threadIdx.x & 31) == 0) c.st->prior_set = 1;
}

cudaError_t launch_prior_set(const ColonyDev &c, cudaStream_t s) {
  cudaError_t e = cudaMemsetAsync(&c.st->prior_set, 0, sizeof(int32_t), s);
  if (e != cudaSuccess) return e;
  k_prior_set<<<608, 256, 0, s>>>(c);
  return cudaGetLastError();
}

// int16 copy of the candidate rows (same pitch; entries past the K
// candidates of a row are -1).  The staged kernel keeps the k <= 32 table in
// shared memory; the long-row kernel reads rows from L2.
__global__ void k_nn_to_i16(const int32_t *__restrict__ nn, int n, int K, int ldk,
                            int16_t *__restrict__ nn16) {
  const int64_t total = (int64_t)n * ldk;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x)
    nn16[t] = (int)(t % ldk) < K ? (int16_t)nn[t] : (int16_t)-1;
}

cudaError_t launch_nn_to_i16(const int32_t *nn, int n, int K, int ldk, int16_t *nn16,
                             cudaStream_t s) {
  k_nn_to_i16<<<304, 256, 0, s>>>(nn, n, K, ldk, nn16);
  return cudaGetLastError();
}

// ---------------------------------------------------------------- tau0
// tau0 from the greedy tour's length C_nn (Dorigo's rules).
__device__ __forceinline__ void greedy_finish(const ColonyDev &c, int64_t len) {
  const float cnn = __ll2float_rn(len);
  float t0;
  if (c.variant == ACO_RANK_BASED) {
    const float num = __fmul_rn(__fmul_rn(0.5f, (float)c.rank_w), (float)(c.rank_w - 1));
    t0 = __fdiv_rn(num, __fmul_rn(c.rho, cnn));
  } else {
    t0 = __fdiv_rn((float)c.m, cnn);
  }
  c.st->tau0 = t0;
  c.st->greedy_length = len;
}

// Greedy nearest-neighbour tour from city 0 (lowest index on ties) on stable
// candidate lists, which hold each row's cities in the order of (distance,
// city): the next city is the first unvisited one of the list.  Warp 0 walks
// the lists, one candidate a lane (the first 32): an id load, a lookup in the
// tabu bits and one warp minimum a step.  The first SK entries of every list are
// copied to shared memory (STAGED: as many as fit, a multiple of eight, or the
// whole list), the others are read from L2 when those are visited, then the
// fallback's second tier where the colony has one.  When no unvisited city is
// left there either the whole CTA takes the minimum over the row.  The tour
// stays in shared memory; its length is summed at the end, an edge a thread.
// One CTA runs alone (16 in a batch's setup), so the step's latency is all
// there is: n = 1000, k = 30 787 -> 113 us, n = 4096, k = 32 5.43 -> 0.82 ms (1.39
// with the lists from L2 and no tier) against the whole-row scan of every step
// below.
constexpr int kGreedyNnThreads = 256;
constexpr size_t kGreedyStageBytes = 200 * 1024;  // with 2 bytes a city more: below 227 KB

// Entries of a list that are staged: 0 if not even eight fit.
__host__ inline int greedy_staged(int n, int ldk) {
  if ((size_t)n * ldk * 2 <= kGreedyStageBytes) return ldk;
  return (int)(kGreedyStageBytes / ((size_t)n * 2)) / 8 * 8;  // below ldk
}

struct GreedyLayout {
  size_t tour_off, tabu_off, bytes;
};
__host__ __device__ inline GreedyLayout greedy_layout(int n, int sk) {
  GreedyLayout L;
  L.tour_off = ((size_t)n * sk * 2 + 15) / 16 * 16;
  L.tabu_off = L.tour_off + ((size_t)n * 2 + 15) / 16 * 16;
  L.bytes = L.tabu_off + (size_t)((n + 31) / 32) * 4;
  return L;
}

template <bool STAGED>
__global__ void __launch_bounds__(kGreedyNnThreads) k_greedy_tau0_nn(ColonyDev c, int sk) {
  extern __shared__ __align__(16) unsigned char smem_greedy[];
  __shared__ unsigned red_d[kGreedyNnThreads / 32], red_j[kGreedyNnThreads / 32];
  __shared__ unsigned long long red_len[kGreedyNnThreads / 32];
  __shared__ int s_cur, s_pos;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n = c.n, words = (n + 31) >> 5;
  const GreedyLayout L = greedy_layout(n, STAGED ? sk : 0);
  int16_t *sids = reinterpret_cast<int16_t *>(smem_greedy);
  int16_t *tour = reinterpret_cast<int16_t *>(smem_greedy + L.tour_off);
  uint32_t *tabu = reinterpret_cast<uint32_t *>(smem_greedy + L.tabu_off);
  if (STAGED) {  // four entries a thread: ldk and sk are multiples of four
    const int q = sk >> 2;
    for (int t = tid; t < n * q; t += kGreedyNnThreads)
      reinterpret_cast<uint2 *>(sids)[t] =
          __ldg(reinterpret_cast<const uint2 *>(c.nn16 + (size_t)(t / q) * c.ldk) + t % q);
  }
  for (int w = tid; w < words; w += kGreedyNnThreads) tabu[w] = w == 0 ? 1u : 0u;
  if (tid == 0) {
    tour[0] = 0;
    s_cur = 0;
    s_pos = 1;
  }
  __syncthreads();
  const bool cand = lane < c.K && lane < c.ldk;
  const bool near = cand && STAGED && lane < sk, far = cand && !near;
  for (int rounds = 0; rounds < n; rounds++) {  // one row scan a round: at most n - 1
    if (warp == 0) {
      int cur = s_cur, s = s_pos;
      while (s < n) {
        auto open = [&](int id) { return id >= 0 && !((tabu[id >> 5] >> (id & 31)) & 1u); };
        unsigned m = ~0u;
        if (STAGED) {
          const int id = near ? (int)sids[cur * sk + lane] : -1;
          m = __reduce_min_sync(kFull, open(id) ? ((unsigned)lane << 16) | (unsigned)id : ~0u);
        }
        if (m == ~0u) {
          if (!STAGED || sk < c.K) {
            const int id = far ? (int)c.nn16[(size_t)cur * c.ldk + lane] : -1;
            m = __reduce_min_sync(kFull, open(id) ? ((unsigned)lane << 16) | (unsigned)id : ~0u);
          }
          if (m == ~0u && c.t2 > 0 && c.K <= 32) {  // the next t2 of the order, -1 past them
            const int4 v =
                __ldg(reinterpret_cast<const int4 *>(c.nn2 + (size_t)cur * kTier2) + lane);
            unsigned k = open(v.w) ? (unsigned)v.w : ~0u;
            if (open(v.z)) k = (unsigned)v.z;
            if (open(v.y)) k = (unsigned)v.y;
            if (open(v.x)) k = (unsigned)v.x;
            m = __reduce_min_sync(kFull, k != ~0u ? ((unsigned)lane << 16) | k : ~0u);
          }
          if (m == ~0u) break;
        }
        cur = (int)(m & 0xffffu);
        if (lane == 0) {
          tabu[cur >> 5] |= 1u << (cur & 31);
          tour[s] = (int16_t)cur;
        }
        __syncwarp();
        s++;
      }
      if (lane == 0) {
        s_cur = cur;
        s_pos = s;
      }
    }
    __syncthreads();
    const int cur = s_cur, s = s_pos;
    if (s >= n) break;
    // The row's unvisited minimum of (distance, city).
    const int32_t *row = c.dist + (size_t)cur * c.ld;
    unsigned bd = ~0u, bj = ~0u;
    for (int j = tid; j < n; j += kGreedyNnThreads) {
      if ((tabu[j >> 5] >> (j & 31)) & 1u) continue;
      const unsigned d = (unsigned)__ldcg(row + j);
      if (d < bd) {  // j increases: the lowest index of a tie stays
        bd = d;
        bj = (unsigned)j;
      }
    }
    const unsigned wd = __reduce_min_sync(kFull, bd);
    const unsigned wj = __reduce_min_sync(kFull, bd == wd ? bj : ~0u);
    if (lane == 0) {
      red_d[warp] = wd;
      red_j[warp] = wj;
    }
    __syncthreads();
    if (warp == 0) {
      const bool in = lane < kGreedyNnThreads / 32;
      const unsigned d = in ? red_d[lane] : ~0u, j = in ? red_j[lane] : ~0u;
      const unsigned md = __reduce_min_sync(kFull, d);
      const unsigned mj = __reduce_min_sync(kFull, d == md ? j : ~0u);
      if (lane == 0) {
        int next = (int)mj;
        if (mj >= (unsigned)n) {  // cannot happen with n >= 2; recorded
          atomicOr(&c.st->error, kErrCheck);
          next = 0;
        }
        tabu[next >> 5] |= 1u << (next & 31);
        tour[s] = (int16_t)next;
        s_cur = next;
        s_pos = s + 1;
      }
    }
    __syncthreads();
  }
  int64_t len = 0;
  for (int i = tid; i < n; i += kGreedyNnThreads)
    len += c.dist[(size_t)tour[i] * c.ld + tour[i + 1 == n ? 0 : i + 1]];
  for (int o = 16; o; o >>= 1) len += __shfl_xor_sync(kFull, len, o);
  if (lane == 0) red_len[warp] = (unsigned long long)len;
  __syncthreads();
  if (tid == 0) {
    for (int w = 1; w < kGreedyNnThreads / 32; w++) len += (int64_t)red_len[w];
    greedy_finish(c, len);
  }
}

// The same tour whatever the candidate lists (none in int16, another tie
// order, or one city a row).  The reference's greedyDistance is a stub returning 0
// (src/Colony.cu:1053-1055) and its tau0 is the constant 1e-6
// (src/AntSystem.cu:200-203), which this kernel also sets.  One CTA of
// kGreedyThreads: each step reads the current row once (coalesced, n /
// kGreedyThreads cities per thread) and takes the block-wide minimum of
// (distance << 32 | city) over unvisited cities, so a step costs one L2 round
// trip and two barriers.
constexpr int kGreedyThreads = 1024;

__global__ void __launch_bounds__(kGreedyThreads)
    k_greedy_tau0(ColonyDev c, int tau0_mode, float tau0_value) {
  extern __shared__ uint32_t tabu[];
  __shared__ unsigned long long red[kGreedyThreads / 32];
  __shared__ int s_next;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int words = (c.n + 31) >> 5;
  if (tau0_mode != ACO_TAU0_DORIGO) {
    if (tid == 0) {
      c.st->tau0 = tau0_mode == ACO_TAU0_REFERENCE ? (float)0.000001 : tau0_value;
      c.st->greedy_length = 0;
    }
    return;
  }
  for (int w = tid; w < words; w += kGreedyThreads) tabu[w] = w == 0 ? 1u : 0u;
  __syncthreads();
  int cur = 0;
  int64_t len = 0;  // kept by thread 0
  for (int s = 1; s < c.n; s++) {
    const int32_t *row = c.dist + (size_t)cur * c.ld;
    unsigned long long best = ~0ull;
    for (int j = tid; j < c.n; j += kGreedyThreads) {
      if ((tabu[j >> 5] >> (j & 31)) & 1u) continue;
      const unsigned long long key =
          ((unsigned long long)(uint32_t)__ldcg(row + j) << 32) | (uint32_t)j;
      best = key < best ? key : best;
    }
    for (int o = 16; o; o >>= 1) {
      const unsigned long long other = __shfl_xor_sync(kFull, best, o);
      best = other < best ? other : best;
    }
    if (lane == 0) red[warp] = best;
    __syncthreads();
    if (warp == 0) {
      best = red[lane];
      for (int o = 16; o; o >>= 1) {
        const unsigned long long other = __shfl_xor_sync(kFull, best, o);
        best = other < best ? other : best;
      }
      if (lane == 0) {
        const int bj = (int)(uint32_t)best;
        if (best == ~0ull || bj >= c.n) {  // cannot happen with n >= 2; recorded
          atomicOr(&c.st->error, kErrCheck);
          s_next = 0;
        } else {
          tabu[bj >> 5] |= 1u << (bj & 31);
          len += (int64_t)(best >> 32);
          s_next = bj;
        }
      }
    }
    __syncthreads();
    cur = s_next;
  }
  if (tid == 0) greedy_finish(c, len + c.dist[(size_t)cur * c.ld + 0]);
}

cudaError_t launch_greedy_tau0(const ColonyDev &c, int tau0_mode, float tau0_value,
                               bool stable_lists, cudaStream_t s) {
  // One candidate a row and no tier: the list is used up at most steps, and then
  // this kernel's 256 threads scan the row slower than that one's 1024 (n = 4000
  // 5.23 ms by lists, 5.31 by rows; 8000 25.0 and 23.9; 16000 138 and 81).  With
  // two candidates the lists win at all sizes (16000 74 and 81).
  const bool lists = c.K > 1 || c.t2 > 0 || c.n <= 4096;
  if (tau0_mode == ACO_TAU0_DORIGO && stable_lists && lists && c.nn16 && c.n < 32768) {
    const int sk = greedy_staged(c.n, c.ldk);
    const size_t smem = greedy_layout(c.n, sk).bytes;
    void (*fn)(ColonyDev, int) = sk > 0 ? k_greedy_tau0_nn<true> : k_greedy_tau0_nn<false>;
    if (smem > 48 * 1024) {
      const cudaError_t e = open_smem((const void *)fn, smem, device_max_smem(), 256);
      if (e != cudaSuccess) return e;
    }
    fn<<<1, kGreedyNnThreads, smem, s>>>(c, sk);
    return cudaGetLastError();
  }
  const size_t smem = (size_t)((c.n + 31) / 32) * 4;
  k_greedy_tau0<<<1, kGreedyThreads, smem, s>>>(c, tau0_mode, tau0_value);
  return cudaGetLastError();
}

// Colony::initPheromone + initAntAges + initTourLengths and the best-so-far
// reset (src/Colony.cu:216-228, 315-351, 38-39).
__global__ void k_init_colony(ColonyDev c) {
  const float t0 = c.st->tau0;
  const int64_t total = (int64_t)c.n * c.ld;
  const int64_t gtid = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t t = gtid; t < total; t += stride) c.tau[t] = t0;
  for (int64_t k = gtid; k < c.m; k += stride) {
    c.age[k] = 0;
    c.perf[k] = 0;
    c.valid[k] = 1;
    c.len[k] = 0;
    c.newlen[k] = 0;
  }
  if (gtid == 0) {
    c.st->iter_best = (int64_t)ACO_MAX_DISTANCE - 1;
    c.st->glob_best = ACO_MAX_DISTANCE;
    c.st->iter_best_ant = -1;
    c.st->iteration = 0;
    c.st->num_valid = c.m;
    c.st->isconverged = 0;
    c.st->globalperformance = 0;
    c.st->dep_count = 0;
    c.st->fallbacks = 0;
    c.st->tours_built = 0;
  }
}

cudaError_t launch_init_colony(const ColonyDev &c, cudaStream_t s) {
  k_init_colony<<<608, 256, 0, s>>>(c);
  return cudaGetLastError();
}

}  // namespace aco
