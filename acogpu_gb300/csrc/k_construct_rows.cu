// k_construct_rows.cu -- tour construction over long candidate rows (k > 32,
// the reference's full-row roulette included), one warp per ant.
//
// Replaces the reference CPU step calculateProbabilityOfSelection +
// selectCities / chooseBestNext (src/Colony.cu:795-864) and the GPU kernels
// dev_compute_probabilities / dev_reduce_probabilities_s / dev_move_ants
// (inc/Colony.cuh:193-229,290-347; src/Colony.cu:643-685).  The reference
// walks all n entries of the current city's nn row for every ant and step:
// it adds the weight of every unvisited entry, in row order, into sum_prob,
// then walks the same entries again until the running sum exceeds
// u * sum_prob.  Visited entries carry weight 0.
//
// Those two walks are sequential float sums; forming them is a dependent add
// per unvisited city.  The pick does not need them to the last bit, only on
// which side of u * sum_prob the running sum lies before and after the picked
// entry, and the distance of a sequential float sum of non-negative numbers
// from the true sum is bounded: after c additions of non-zero terms it is at
// most c 2^-24 (relative; second-order terms covered below).  A step
// therefore
//  1. sums the row in whatever order is fast (S', error bound d_S 2^-24),
//  2. forms approximate prefixes over the row in row order, 128 entries at a
//     time, up to the chunk where they pass u S' (error bound d_P 2^-24),
//  3. takes the crossing entry i if prefix(i) > u S' (1 + E) and
//     prefix(i - 1) <= u S' (1 - E), with E = 1.02 (c + i + d_S + d_P + 8)
//     2^-24: then the reference's own sums cross at i too, whatever its
//     roundings were (the reference's prefix is at least prefix(i)
//     (1 - (i + d_P) 2^-24), its threshold at most u S' (1 + (c + d_S + 2)
//     2^-24), and the other way round for i - 1; sequential sums never
//     decrease, so the crossing is unique).  The 1.02 covers the products of
//     errors (E < 2.1e-3 at c = 8192) and the 8 the roundings of u S' and of
//     the bounds; 2^-147 is added for thresholds in the subnormal range, where
//     products round by up to 2^-150 and sums not at all;
//  4. otherwise -- u S' within the bound of a prefix, or a sum that is not
//     finite -- forms the reference's running sums themselves (rows_exact).
//     u falls into such a window in 0.1 to 3 % of the steps at n = 1000 (the
//     most with fresh pheromone on uniform instances, fewer later, when most
//     weights are smaller than the window), at n = 2392 in 13 % in the first
//     iteration and 4 % in the second.  The
//     walk in 256-entry chunks with a scan in each took 2392 cities from 4.4
//     ms an iteration (128-entry chunks) to 4.0.
//
// Full rows without a learned prior are summed in city order, straight from
// the choice matrix: city 128 j + 4 l + t belongs to lane l, whose open
// (unvisited) cities are the bits 4 j + t of one word, so masking needs no
// lookup and no city ids.  Other rows (k < n, the candidate heuristic carrying
// a prior, at most one chunk) are summed in row order.  Only the prefixes need
// ids, and usually one chunk of 128: the weights fall off with the distance
// (97 % of the steps at n = 1000).  hi and lo, u S' (1 +- E) +- 2^-147, are
// compared with all prefixes; one warp minimum over (lane, city) keys finds
// the first past lo, with no city in it if it is not past hi.
//
// What bounds it: one ant's step is a chain of an L2 round trip (365 cycles,
// 740 for the ten 512-byte loads at n = 1000: beyond about 24 lines of a warp
// the next wait for the first) and some ten shuffles; a batch keeps 32
// independent warps an SM in flight, two thirds of its issue slots taken.  No
// warp waits for another.  The former kernel compacted every row into shared
// memory for a warp of the CTA that ran the sequential sums of all its ants in
// lockstep.  Construction per iteration, before and now: n = m = 100 214 and
// 57 us, n = m = 1000 3019 and 784, n = 2392, m = 512 14.98 and 4.00 ms, n =
// 1501, k = 64, m = 500 about 3.9 ms and 0.88, the batch of 8 x n = 1000 17.8
// and 3.6 ms.
#include "k_construct_steps.cuh"

namespace aco {

// ---- the visited mask -------------------------------------------------------

// The open-city words of an ant, in shared memory.  Word 32 r + l, bit 4 j + t stands for city
// 1024 r + 128 j + 4 l + t; a set bit is an unvisited city of the instance.
// One word a lane for n <= 1024 (R1), else kRowsMaskWords so that any 13-bit
// id (the -1 padding of a row included) indexes inside it.
constexpr int kRowsMaskWords = kRowsMaxCities / 32;

template <bool R1>
__device__ __forceinline__ bool rows_open(const uint32_t *mask, unsigned id) {
  const unsigned word = R1 ? (id >> 2) & 31u : ((id >> 5) & 0xe0u) | ((id >> 2) & 31u);
  return (mask[word] >> (((id >> 5) & 0x1cu) | (id & 3u))) & 1u;
}

// Marks `city` visited; its word belongs to lane (city / 4) % 32, which also
// holds it in `own` when R1.
template <bool R1>
__device__ __forceinline__ void rows_mark(uint32_t *mask, uint32_t &own, int city, int lane) {
  if (lane == ((city >> 2) & 31)) {
    const uint32_t bit = 1u << (((city >> 5) & 0x1c) | (city & 3));
    if (R1) {
      own &= ~bit;
      mask[lane] = own;
    } else {
      mask[((city >> 10) << 5) | lane] &= ~bit;
    }
  }
  __syncwarp();
}

// ---- row reads ----------------------------------------------------------------

// Chunk `ch` of the row of `cur` in row order: entries 128 ch + 4 lane .. + 3,
// weights of visited entries (and of the row's padding) zero.  `id` keeps the
// packed int16 ids.
struct RowsChunk {
  float x[4];
  uint2 id;
};

// Padding entries (positions K .. ldk - 1) have choice 0 in the table, and
// positions past the row load zeros, so their weight is 0 whatever their id;
// a blended weight is formed inside the row only (p0: the lane's position).
template <bool R1, bool BLEND>
__device__ __forceinline__ RowsChunk rows_mask(const ColonyDev &c, const uint32_t *mask,
                                               const float4 &w, const float4 &e, const uint2 &id,
                                               int p0, const AntCtx &a) {
  RowsChunk r;
  r.id = id;
  const float wi[4] = {w.x, w.y, w.z, w.w};
  const unsigned ids[4] = {id.x & 0xffffu, id.x >> 16, id.y & 0xffffu, id.y >> 16};
#pragma unroll
  for (int t = 0; t < 4; t++) {
    float v = wi[t];
    if (BLEND) {
      const float ee = t == 0 ? e.x : t == 1 ? e.y : t == 2 ? e.z : e.w;
      v = p0 + t < c.K ? blend_fitness(wi[t], ee, a.meanc, a.ratio, c.use_alpha, c.alpha) : 0.0f;
    }
    r.x[t] = rows_open<R1>(mask, ids[t]) ? v : 0.0f;
  }
  return r;
}

// Packed pairs of floats: two additions or FMAs an instruction, each rounded
// on its own.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ float sum2(f32x2 a) {
  float x, y;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a));
  return x + y;
}

// 0/1 masks of the four cities of a nibble of the open-city word, in shared
// memory (empty where predicates do the masking).
template <bool LUT>
struct RowsLut {
  float4 m[16];
};
template <>
struct RowsLut<false> {};

__device__ __forceinline__ void rows_lut_init(RowsLut<true> &lut) {
  for (int i = threadIdx.x; i < 16; i += blockDim.x)
    lut.m[i] = make_float4((i & 1) ? 1.f : 0.f, (i & 2) ? 1.f : 0.f, (i & 4) ? 1.f : 0.f,
                           (i & 8) ? 1.f : 0.f);
  __syncthreads();
}

// A lane's masked running sums.  LUT (a single colony, bound by one ant's
// latency): the mask as four floats from the table, two packed FMAs a chunk
// -- a predicate would cost a compare, and 13 cycles until its use, for each
// city: n = m = 1000 844 us an iteration against 1287.  A masked infinity
// turns into a NaN, and a sum that is not finite goes to the exact path.
// Otherwise (batches, whose many warps would queue for shared memory)
// predicated adds, the tests on constant bits of one register: 8 x n = 1000
// 3.6 ms against 4.0.
template <bool LUT>
struct RowsSum;

template <>
struct RowsSum<true> {
  f32x2 s[4] = {0ull, 0ull, 0ull, 0ull};
  // Chunks j0 .. j0 + N - 1 (0 .. 7) of the round that `open` stands for.
  template <int N>
  __device__ __forceinline__ void add(const ulonglong2 (&q)[N], uint32_t open, int j0,
                                      const RowsLut<true> &lut) {
#pragma unroll
    for (int j = 0; j < N; j++) {
      const unsigned at = (j0 + j == 0 ? open << 4 : open >> (4 * (j0 + j) - 4)) & 0xf0u;
      const ulonglong2 m = *reinterpret_cast<const ulonglong2 *>(
          reinterpret_cast<const char *>(lut.m) + at);
      s[2 * (j & 1)] = fma2(q[j].x, m.x, s[2 * (j & 1)]);
      s[2 * (j & 1) + 1] = fma2(q[j].y, m.y, s[2 * (j & 1) + 1]);
    }
  }
  __device__ __forceinline__ float total() const {
    return sum2(add2(add2(s[0], s[1]), add2(s[2], s[3])));
  }
};

template <>
struct RowsSum<false> {
  float s[4] = {0.f, 0.f, 0.f, 0.f};
  template <int N>
  __device__ __forceinline__ void add(const ulonglong2 (&q)[N], uint32_t open, int j0,
                                      const RowsLut<false> &) {
#pragma unroll
    for (int j = 0; j < N; j++) {
      float x, y, z, w;
      asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(q[j].x));
      asm("mov.b64 {%0, %1}, %2;" : "=f"(z), "=f"(w) : "l"(q[j].y));
      const int b = 4 * (j0 + j);
      if (open & (1u << b)) s[0] = __fadd_rn(s[0], x);
      if (open & (2u << b)) s[1] = __fadd_rn(s[1], y);
      if (open & (4u << b)) s[2] = __fadd_rn(s[2], z);
      if (open & (8u << b)) s[3] = __fadd_rn(s[3], w);
    }
  }
  __device__ __forceinline__ float total() const { return (s[0] + s[1]) + (s[2] + s[3]); }
};

// The fields of a colony that every step reads, held in registers (a batch's
// descriptors are in shared memory).
struct RowsView {
  const float *choice, *choice_nn;
  const int16_t *nn16;
  int n, K, ld, ldk;
};

// The choice values of chunks t0 .. t0 + N - 1 of a row (pointer at this
// lane's city of chunk 0; the pitch of a colony whose rows are summed in city
// order is a multiple of 128, so a chunk that holds a city is read whole).
template <int N>
__device__ __forceinline__ void rows_fetch(const float *row, int t0, int n, ulonglong2 (&q)[N]) {
#pragma unroll
  for (int j = 0; j < N; j++) {
    q[j] = make_ulonglong2(0ull, 0ull);
    if ((t0 + j) * 128 < n)  // the same for every lane
      q[j] = __ldcg(reinterpret_cast<const ulonglong2 *>(row + (t0 + j) * 128));
  }
}

// STG: the view's candidate rows are in shared memory.
template <bool BLEND, bool STG>
__device__ __forceinline__ void rows_load(const ColonyDev &c, const RowsView &v, int cur, int ch,
                                          float4 &w, float4 &e, uint2 &id, int lane) {
  const int p0 = ch * 128 + lane * 4;
  const size_t off = (size_t)cur * v.ldk + p0;
  const bool in = p0 < v.K;  // ldk % 4 == 0: the four entries are in the row
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  const uint2 *ip = reinterpret_cast<const uint2 *>(v.nn16 + off);
  const float4 *wp = reinterpret_cast<const float4 *>((BLEND ? c.tau_nn : v.choice_nn) + off);
  if constexpr (STG) {
    id = in ? *ip : make_uint2(0u, 0u);
    w = in ? (BLEND ? __ldcg(wp) : *wp) : zero;
  } else {
    id = in ? __ldg(ip) : make_uint2(0u, 0u);
    w = in ? __ldcg(wp) : zero;
  }
  if (BLEND) e = in ? __ldg(reinterpret_cast<const float4 *>(c.eta_nn + off)) : zero;
}

__device__ __forceinline__ RowsView rows_view(const ColonyDev &c) {
  return RowsView{c.choice, c.choice_nn, c.nn16, c.n, c.K, c.ld, c.ldk};
}

// This lane's part of the sum over the open cities of `cur`'s row, in city
// order (d_S: 4 additions a round, then the tree).  Above one round the loads
// of the next 512 cities are issued before this 512's additions.
template <bool R1, bool BLEND, bool LUT>
__device__ __forceinline__ float rows_city_sum(const ColonyDev &c, const RowsView &v, int cur,
                                               const uint32_t *mask, uint32_t own,
                                               const RowsLut<LUT> &lut, const AntCtx &a,
                                               int lane) {
  const size_t row = (size_t)cur * v.ld + lane * 4;
  if constexpr (BLEND) {  // few ants blend: one chunk at a time, predicated
    float s[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 1
    for (int t = 0; t * 128 < c.n; t++) {
      const uint32_t b = (R1 ? own : mask[32 * (t >> 3) + lane]) >> (4 * (t & 7));
      if (!(b & 0xfu)) continue;
      const float4 x = __ldcg(reinterpret_cast<const float4 *>(c.tau + row + t * 128));
      const float4 e = __ldg(reinterpret_cast<const float4 *>(c.eta + row + t * 128));
      const float v[4] = {blend_fitness(x.x, e.x, a.meanc, a.ratio, c.use_alpha, c.alpha),
                          blend_fitness(x.y, e.y, a.meanc, a.ratio, c.use_alpha, c.alpha),
                          blend_fitness(x.z, e.z, a.meanc, a.ratio, c.use_alpha, c.alpha),
                          blend_fitness(x.w, e.w, a.meanc, a.ratio, c.use_alpha, c.alpha)};
#pragma unroll
      for (int q = 0; q < 4; q++)
        if ((b >> q) & 1u) s[q] = __fadd_rn(s[q], v[q]);
    }
    return (s[0] + s[1]) + (s[2] + s[3]);
  } else {
    const float *p = v.choice + row;
    RowsSum<LUT> sum;
    if constexpr (R1) {
      ulonglong2 q[8];
      rows_fetch<8>(p, 0, v.n, q);
      sum.template add<8>(q, own, 0, lut);
    } else {
      ulonglong2 q0[4], q1[4];
      rows_fetch<4>(p, 0, v.n, q0);
#pragma unroll 1
      for (int r = 0; r * 1024 < v.n; r++) {
        const uint32_t open = mask[32 * r + lane];
        rows_fetch<4>(p, 8 * r + 4, v.n, q1);
        sum.template add<4>(q0, open, 0, lut);
        rows_fetch<4>(p, 8 * r + 8, v.n, q0);
        sum.template add<4>(q1, open, 4, lut);
      }
    }
    return sum.total();
  }
}

// ---- the rare paths -------------------------------------------------------------

// One chunk of 256 entries for the exact path, eight a lane in row order.
template <bool R1, bool BLEND>
__device__ __forceinline__ void rows_load8(const ColonyDev &c, const RowsView &v, int cur, int ch,
                                           float4 (&w)[2], float4 (&e)[2], uint4 &id, int lane) {
  const int p0 = ch * 256 + lane * 8;
  const size_t off = (size_t)cur * v.ldk + p0;
  const bool in = p0 < v.K;  // ldk % 8 == 0: the eight entries are in the row
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  const float4 *wp = reinterpret_cast<const float4 *>((BLEND ? c.tau_nn : v.choice_nn) + off);
  id = in ? __ldg(reinterpret_cast<const uint4 *>(v.nn16 + off)) : make_uint4(0u, 0u, 0u, 0u);
  w[0] = in ? __ldcg(wp) : zero;
  w[1] = in ? __ldcg(wp + 1) : zero;
  if (BLEND) {
    const float4 *ep = reinterpret_cast<const float4 *>(c.eta_nn + off);
    e[0] = in ? __ldg(ep) : zero;
    e[1] = in ? __ldg(ep + 1) : zero;
  }
}

template <bool R1, bool BLEND>
__device__ __forceinline__ void rows_mask8(const ColonyDev &c, const uint32_t *mask,
                                           const float4 (&w)[2], const float4 (&e)[2],
                                           const uint4 &id, int p0, const AntCtx &a,
                                           float (&x)[8]) {
#pragma unroll
  for (int h = 0; h < 2; h++) {
    const RowsChunk r = rows_mask<R1, BLEND>(
        c, mask, w[h], e[h], h ? make_uint2(id.z, id.w) : make_uint2(id.x, id.y), p0 + 4 * h, a);
#pragma unroll
    for (int t = 0; t < 4; t++) x[4 * h + t] = r.x[t];
  }
}

// The reference's running sums over one such chunk (visited entries 0), from
// entry `start` on: from the sum `s` before it to the sum after the chunk; THR:
// only up to the first entry whose running sum exceeds `thr`, in `pos` (-1 if
// there is none).
//
// While the sum stays in one binade, with ulp 2^(e-23), adding w rounds to
// s + RN(w / ulp) ulp unless w / ulp lies halfway between two integers (then
// the parity of s decides).  The rounded terms are multiples of the ulp, so
// their sums below 2^(e+1) are exact in any order, and a scan gives every
// running sum.  RN(w / ulp) ulp is (w + M) - M with M = 1.5 2^e, for
// w < 2^(e-1).  The entries where that does not hold are added one at a
// time: those that would leave the binade (the scan shows the first), large
// ones, halfway cases; so is every non-zero entry from 2^127 on.  Below 2^-125
// every term is a multiple of 2^-149 and adds exactly.  A sum that is not finite
// stays so, but for a NaN among the entries.  Each trip ends the chunk or adds
// one entry, so there are at most 257; most chunks take one, which looks at the
// chunk's total only.
template <bool THR>
__device__ __forceinline__ float rows_walk(const float (&x)[8], int start, float s, float thr,
                                           int lane, int &pos) {
  pos = -1;
  float v[8];
#pragma unroll
  for (int q = 0; q < 8; q++) v[q] = 8 * lane + q >= start ? x[q] : 0.0f;
#pragma unroll 1
  for (int trip = 0; trip < 258; trip++) {
    if (__float_as_uint(s) >= 0x7f800000u) {
      bool nan = false;
#pragma unroll
      for (int q = 0; q < 8; q++) nan |= v[q] != v[q];
      return __any_sync(kFull, nan) ? __uint_as_float(0x7fffffffu) : s;
    }
    const uint32_t eb = __float_as_uint(s) & 0x7f800000u;
    const bool tiny = s < 0x1p-125f;
    // One entry at a time: every non-zero entry counts as large.
    const bool one = s >= 0x1p127f;
    const float M = one || tiny ? 0.0f : __uint_as_float(eb | 0x00400000u);
    const float half_base = one ? 0.0f : tiny ? 0x1p-126f : 0.5f * __uint_as_float(eb);
    const float half_ulp = one || tiny ? -1.0f : 0x1p-23f * half_base;
    const float lim = tiny ? 0x1p-125f : __uint_as_float(eb + 0x00800000u);
    float t[8];
    unsigned ev = 0u;
#pragma unroll
    for (int q = 0; q < 8; q++) {
      t[q] = __fsub_rn(__fadd_rn(v[q], M), M);
      if (!(v[q] < half_base || v[q] == 0.0f) || fabsf(__fsub_rn(v[q], t[q])) == half_ulp)
        ev |= 1u << q;
    }
#pragma unroll
    for (int q = 1; q < 8; q++) t[q] += t[q - 1];  // now this lane's running terms
    float incl = t[7];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) incl = scan_level<32>(incl, o);
    const float end = s + __shfl_sync(kFull, incl, 31);
    const bool any = __any_sync(kFull, ev != 0u);
    if (!any && (one || end < lim) && !(THR && end > thr)) return end;
    // The first special entry, the first that leaves the binade, the first
    // past thr.  Terms from a special entry on are not used: they may be
    // wrong or not finite, and so may what the scan made of them, in later
    // lanes and later entries only.
    float ex = __shfl_up_sync(kFull, incl, 1);
    if (lane == 0) ex = 0.0f;
    unsigned over = 0u;
#pragma unroll
    for (int q = 0; q < 8; q++) {
      const float r = s + (ex + t[q]);
      if (!one && r >= lim) ev |= 1u << q;
      if (THR && r > thr) over |= 1u << q;
    }
    const int ie = (int)__reduce_min_sync(kFull, ev ? 8 * lane + __ffs(ev) - 1 : 256);
    if (THR) {
      const int io = (int)__reduce_min_sync(kFull, over ? 8 * lane + __ffs(over) - 1 : 256);
      if (io < ie) {
        pos = io;
        return s;
      }
    }
    if (ie >= 256) return end;
    const int l = ie >> 3, q = ie & 7;
    float before = ex, w = v[0];
#pragma unroll
    for (int i = 1; i < 8; i++)
      if (q == i) {
        before = ex + t[i - 1];
        w = v[i];
      }
    s = __fadd_rn(s + __shfl_sync(kFull, before, l), __shfl_sync(kFull, w, l));
    if (THR && s > thr) {
      pos = ie;
      return s;
    }
    if (ie == 255) return s;
#pragma unroll
    for (int i = 0; i < 8; i++)
      if (8 * lane + i <= ie) v[i] = 0.0f;
  }
  return s;  // not reached: every trip consumes an entry
}

// The first 64 entries of a row, lanes 0 .. 7, added one after another (most
// of a row's binade changes and halfway cases are there): all lanes run the
// same chain on broadcast values.
template <bool THR>
__device__ __forceinline__ float rows_head(const float (&x)[8], float thr, int &pos) {
  float s = 0.0f;
  pos = -1;
#pragma unroll
  for (int l = 0; l < 8; l++) {
#pragma unroll
    for (int q = 0; q < 8; q++) {
      s = __fadd_rn(s, __shfl_sync(kFull, x[q], l));
      if (THR && s > thr && pos < 0) pos = 8 * l + q;
    }
  }
  return s;
}

// The reference's walk (header): the sum over the row with the running sum at
// every chunk's end kept one a lane, then the chunk of the crossing again.
// Returns the picked city or -1 (no pick: S <= 0, or no running sum above
// u * S).  A NaN threshold (u times an infinite sum cannot give one, a NaN
// weight can) picks the first unvisited entry, as the reference's
// !(sum <= rnd) does.
template <bool R1, bool BLEND>
__device__ __noinline__ int rows_exact(const ColonyDev &c, int cur, const uint32_t *mask, float u,
                                       AntCtx a, int lane) {
  const RowsView v = rows_view(c);
  const int nch = (c.K + 255) >> 8;  // at most 32
  float s = 0.0f, end = 0.0f, x[8];
  float4 w[2], e[2];
  uint4 id;
  int pos;
  rows_load8<R1, BLEND>(c, v, cur, 0, w, e, id, lane);
#pragma unroll 1
  for (int ch = 0; ch < nch; ch++) {
    rows_mask8<R1, BLEND>(c, mask, w, e, id, ch * 256 + lane * 8, a, x);
    rows_load8<R1, BLEND>(c, v, cur, ch + 1, w, e, id, lane);  // zeros past the row
    if (ch == 0) s = rows_head<false>(x, 0.0f, pos);
    s = rows_walk<false>(x, ch == 0 ? 64 : 0, s, 0.0f, lane, pos);
    if (lane == ch) end = s;
  }
  if (s <= 0.0f) return -1;  // chooseBestNext (src/Colony.cu:776-778)
  const float rnd = __fmul_rn(u, s);
  if (rnd != rnd) {
    for (int p0 = 0; p0 < c.K; p0 += 32) {
      const int p = p0 + lane;
      const unsigned city = p < c.K ? (unsigned)(uint16_t)c.nn16[(size_t)cur * c.ldk + p] : 0u;
      const unsigned m = __ballot_sync(kFull, p < c.K && rows_open<R1>(mask, city));
      if (m) return (int)__shfl_sync(kFull, city, __ffs(m) - 1);
    }
    return -1;
  }
  const unsigned h = __ballot_sync(kFull, lane < nch && end > rnd);
  if (!h) return -1;
  const int ch = __ffs(h) - 1;
  rows_load8<R1, BLEND>(c, v, cur, ch, w, e, id, lane);
  rows_mask8<R1, BLEND>(c, mask, w, e, id, ch * 256 + lane * 8, a, x);
  if (ch == 0) {
    s = rows_head<true>(x, rnd, pos);
    if (pos < 0) rows_walk<true>(x, 64, s, rnd, lane, pos);
  } else {
    rows_walk<true>(x, 0, __shfl_sync(kFull, end, ch - 1), rnd, lane, pos);
  }
  if (pos < 0) return -1;
  const unsigned ids = (pos & 4) ? ((pos & 2) ? id.w : id.z) : ((pos & 2) ? id.y : id.x);
  return (int)__shfl_sync(kFull, (pos & 1) ? ids >> 16 : ids & 0xffffu, pos >> 3);
}

// The fallback (fallback_city's rules on this file's mask): the last
// unvisited entry of the row (select_local_best, inc/Colony.cuh:33-43), or
// the unvisited city with the largest choice value, lowest index on ties.
// -1 if there is none.
template <bool R1>
__device__ __noinline__ int rows_fallback(const ColonyDev &c, int cur, const uint32_t *mask,
                                          AntCtx a, int lane) {
  if (c.fallback == ACO_FALLBACK_REFERENCE) {
    const int16_t *ids = c.nn16 + (size_t)cur * c.ldk;
    for (int ch = (c.K - 1) >> 5; ch >= 0; ch--) {
      const int p = ch * 32 + lane;
      const unsigned id = p < c.K ? (unsigned)(uint16_t)ids[p] : 0u;
      const unsigned m = __ballot_sync(kFull, p < c.K && rows_open<R1>(mask, id));
      if (m) return (int)__shfl_sync(kFull, id, 31 - __clz(m));
    }
    return -1;
  }
  float bw = -1.0f;
  int bj = -1;
  const size_t row = (size_t)cur * c.ld;
  for (int r = 0; r * 1024 < c.n; r++) {
    const uint32_t open = mask[32 * r + lane];
#pragma unroll 2
    for (int j = 0; j < 8; j++) {
      const uint32_t b = (open >> (4 * j)) & 0xfu;
      if (!b) continue;
      const int c0 = r * 1024 + j * 128 + lane * 4;
      float v[4];
      if (!a.blend) {
        const float4 q = __ldcg(reinterpret_cast<const float4 *>(c.choice + row + c0));
        v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
      } else {
        const float4 t = __ldcg(reinterpret_cast<const float4 *>(c.tau + row + c0));
        const float4 e = __ldg(reinterpret_cast<const float4 *>(c.eta + row + c0));
        v[0] = blend_fitness(t.x, e.x, a.meanc, a.ratio, c.use_alpha, c.alpha);
        v[1] = blend_fitness(t.y, e.y, a.meanc, a.ratio, c.use_alpha, c.alpha);
        v[2] = blend_fitness(t.z, e.z, a.meanc, a.ratio, c.use_alpha, c.alpha);
        v[3] = blend_fitness(t.w, e.w, a.meanc, a.ratio, c.use_alpha, c.alpha);
      }
#pragma unroll
      for (int t = 0; t < 4; t++)
        if (((b >> t) & 1u) && v[t] > bw) {
          bw = v[t];
          bj = c0 + t;
        }
    }
  }
  for (int o = 16; o; o >>= 1) {
    const float ow = __shfl_xor_sync(kFull, bw, o);
    const int oj = __shfl_xor_sync(kFull, bj, o);
    if (oj >= 0 && (bj < 0 || ow > bw || (ow == bw && oj < bj))) {
      bw = ow;
      bj = oj;
    }
  }
  return bj;
}

// ---- one step -------------------------------------------------------------------

constexpr int kRowsAmbiguous = -2;

// One chunk's prefixes: p[t] = base + the sum of the chunk's entries up to
// this lane's entry t (at most 10 additions each).  A scan within groups of
// eight lanes, then the groups' totals in every lane; `total` is base plus the
// whole chunk.
__device__ __forceinline__ void rows_prefix(const float (&x)[4], float base, int lane,
                                            float (&p)[4], float &total) {
  const float c1 = x[0] + x[1], c2 = c1 + x[2], c3 = c2 + x[3];
  float g = scan_level<8>(c3, 1);
  g = scan_level<8>(g, 2);
  g = scan_level<8>(g, 4);
  const float T0 = __shfl_sync(kFull, g, 7), T1 = __shfl_sync(kFull, g, 15),
              T2 = __shfl_sync(kFull, g, 23), T3 = __shfl_sync(kFull, g, 31);
  float e = __shfl_up_sync(kFull, g, 1, 8);  // the group's entries before this lane
  if ((lane & 7) == 0) e = 0.0f;
  float before = base;
  if (lane >= 8) before += T0;
  if (lane >= 16) before += T1;
  if (lane >= 24) before += T2;
  e += before;
  p[0] = e + x[0];
  p[1] = e + c1;
  p[2] = e + c2;
  p[3] = e + c3;
  total = base + ((T0 + T1) + (T2 + T3));
}

// The sum of a value over the warp, in every lane (five additions).
__device__ __forceinline__ float rows_warp_sum(float x) {
  x += __shfl_xor_sync(kFull, x, 1);
  x += __shfl_xor_sync(kFull, x, 2);
  x += __shfl_xor_sync(kFull, x, 4);
  const float a = __shfl_sync(kFull, x, 0), b = __shfl_sync(kFull, x, 8),
              c = __shfl_sync(kFull, x, 16), d = __shfl_sync(kFull, x, 24);
  return (a + b) + (c + d);
}

// The first entry of the chunk whose prefix is past lo: its city, or 0xffff if
// the prefix is not past hi (inside the window); ~0u if there is none.
__device__ __forceinline__ unsigned rows_first(const float (&p)[4], uint2 id, float lo, float hi,
                                               int lane) {
  unsigned city = p[3] > hi ? id.y >> 16 : 0xffffu;
  if (p[2] > lo) city = p[2] > hi ? id.y & 0xffffu : 0xffffu;
  if (p[1] > lo) city = p[1] > hi ? id.x >> 16 : 0xffffu;
  if (p[0] > lo) city = p[0] > hi ? id.x & 0xffffu : 0xffffu;
  return __reduce_min_sync(kFull, p[3] > lo ? ((unsigned)lane << 16) | city : ~0u);
}

// The guarded pick of the header at city `cur` with `cnt` open cities or
// candidates left: the city, -1 (the weights are all zero: no pick), or
// kRowsAmbiguous.  `own` is this lane's mask word when R1.  Chunk 0 is
// loaded with the sum's rows and scanned before they are waited for, so the
// common step (the crossing in chunk 0: 97 % of the steps at n = 1000) waits
// for one L2 round trip, the sum and one warp minimum.
template <bool R1, bool BLEND, bool LUT, bool STG>
__device__ __forceinline__ int rows_pick(const ColonyDev &c, const RowsView &v, int cur,
                                         const uint32_t *mask, uint32_t own,
                                         const RowsLut<LUT> &lut, bool natural, int cnt, float u,
                                         const AntCtx &a, int lane) {
  const int nch = (v.K + 127) >> 7;
  float4 w, e;
  uint2 id;
  rows_load<BLEND, STG>(c, v, cur, 0, w, e, id, lane);
  // The entries of the sum, d_S + d_P and 8 (a row of 64 chunks adds at most
  // 64 to either): the window's terms but for the entries up to the crossing.
  const int terms = cnt + 28 + nch;
  float p[4], total, S;
  RowsChunk k;
  if (!STG && natural) {
    const float part = rows_city_sum<R1, BLEND, LUT>(c, v, cur, mask, own, lut, a, lane);
    k = rows_mask<R1, BLEND>(c, mask, w, e, id, lane * 4, a);
    rows_prefix(k.x, 0.0f, lane, p, total);
    S = rows_warp_sum(part);
  } else {
    k = rows_mask<R1, BLEND>(c, mask, w, e, id, lane * 4, a);
    rows_prefix(k.x, 0.0f, lane, p, total);
    S = total;
    if (nch > 1) {
      float part = 0.0f;
#pragma unroll 1
      for (int ch = 1; ch < nch; ch++) {
        rows_load<BLEND, STG>(c, v, cur, ch, w, e, id, lane);
        const RowsChunk q = rows_mask<R1, BLEND>(c, mask, w, e, id, ch * 128 + lane * 4, a);
        part += (q.x[0] + q.x[1]) + (q.x[2] + q.x[3]);
      }
      S += rows_warp_sum(part);
    }
  }
  // The first entry of chunk ch past u S' (1 - E) (rows_first).
  auto first_past = [&](const float (&q)[4], const uint2 &ids, int ch) {
    const float E = (float)(terms + min(cnt, 128 * (ch + 1)) + ch) * 6.08e-8f;  // 1.02 * 2^-24
    const float hi = __fmaf_rn(u * (1.0f + E), S, 0x1p-147f);
    const float lo = __fmaf_rn(u * (1.0f - E), S, -0x1p-147f);
    return rows_first(q, ids, lo, hi, lane);
  };
  unsigned first = first_past(p, k.id, 0);
  if ((int)(first & 0xffffu) < v.n && S <= 3e38f) return (int)(first & 0xffffu);
  if (S == 0.0f) return -1;
  // In the window, a sum that is not finite, or u S' close to S'.
  if (first != ~0u || !(S <= 3e38f)) return kRowsAmbiguous;
  if constexpr (LUT && !BLEND && !STG) {
    // Later chunks four at a time, one L2 round trip for all of them and their
    // scans side by side (the first entry found is in the first chunk that has
    // one; chunks past the row are zeros).  First iterations of n = 2392, m =
    // 512: 5.58 ms of construction with one chunk at a time, 5.23 so.
    constexpr int GR = 4;
#pragma unroll 1
    for (int g = 1; g < nch; g += GR) {
      float4 wg[GR];
      uint2 idg[GR];
#pragma unroll
      for (int q = 0; q < GR; q++) rows_load<BLEND, STG>(c, v, cur, g + q, wg[q], e, idg[q], lane);
      unsigned f[GR];
#pragma unroll
      for (int q = 0; q < GR; q++) {
        k = rows_mask<R1, BLEND>(c, mask, wg[q], e, idg[q], (g + q) * 128 + lane * 4, a);
        rows_prefix(k.x, total, lane, p, total);
        f[q] = first_past(p, k.id, g + q);
      }
#pragma unroll
      for (int q = GR - 1; q >= 0; q--)
        if (f[q] != ~0u) first = f[q];
      if (first != ~0u)
        return (int)(first & 0xffffu) < v.n ? (int)(first & 0xffffu) : kRowsAmbiguous;
    }
    return kRowsAmbiguous;
  } else {
#pragma unroll 1
    for (int ch = 1; ch < nch; ch++) {
      rows_load<BLEND, STG>(c, v, cur, ch, w, e, id, lane);
      k = rows_mask<R1, BLEND>(c, mask, w, e, id, ch * 128 + lane * 4, a);
      rows_prefix(k.x, total, lane, p, total);
      first = first_past(p, k.id, ch);
      if ((int)(first & 0xffffu) < v.n) return (int)(first & 0xffffu);
      if (first != ~0u) return kRowsAmbiguous;
    }
    return kRowsAmbiguous;
  }
}

// The tour of one valid ant.
template <bool R1, bool BLEND, bool LUT, bool STG>
__device__ __forceinline__ void rows_tour(const ColonyDev &c, const RowsView &v, int k,
                                          uint32_t *mask, const RowsLut<LUT> &lut, AntCtx a,
                                          int lane) {
  const int n = c.n;
  int32_t *trow = c.tours + (size_t)k * c.ld;
  const bool natural = rows_city_order(n, c.K) && c.st->prior_set == 0;
  uint32_t own = 0u;
  for (int r = 0; r < (R1 ? 1 : kRowsMaskWords / 32); r++) {
    uint32_t open = 0u;
    for (int j = 0; j < 8; j++) {
      const int left = n - (r * 1024 + j * 128 + lane * 4);
      open |= (left >= 4 ? 0xfu : left > 0 ? (1u << left) - 1u : 0u) << (4 * j);
    }
    mask[32 * r + lane] = open;
    if (R1) own = open;
  }
  // initTour placement (src/Colony.cu:518-520)
  const uint32_t akey = aco_ant_key(c.seed, c.st->iteration, (uint32_t)k);
  int start = __float2int_rz(__fmul_rn(aco_uniform_key(akey, 0u), __int2float_rn(n)));
  bool ok = true;
  if (start >= n) {  // impossible for u < 1; recorded, clamped
    ok = false;
    start = n - 1;
  }
  __syncwarp();
  rows_mark<R1>(mask, own, start, lane);
  int cur = start;
  int64_t fallbacks = 0;
  for (int xb = 0; xb < n; xb += 32) {
    // The uniforms of 32 steps, one a lane, and their tour positions.
    const float ublk = aco_uniform_key(akey, (uint32_t)(xb + lane));
    int tpos = (xb == 0 && lane == 0) ? start : 0;
    const int xe = min(n, xb + 32);
#pragma unroll 1
    for (int x = xb == 0 ? 1 : xb; x < xe; x++) {
      const float u = __shfl_sync(kFull, ublk, x & 31);
      if (BLEND) a.meanc = c.mean[cur];
      int next = rows_pick<R1, BLEND, LUT, STG>(c, v, cur, mask, own, lut, natural, min(v.K, n - x), u, a,
                                           lane);
      if (next < 0) {
        if (next == kRowsAmbiguous) next = rows_exact<R1, BLEND>(c, cur, mask, u, a, lane);
        if (next < 0) {
          next = rows_fallback<R1>(c, cur, mask, a, lane);
          fallbacks++;
        }
      }
      if ((unsigned)next >= (unsigned)n) {  // no unvisited city: cannot happen
        ok = false;
        next = cur;
      }
      rows_mark<R1>(mask, own, next, lane);
      tpos = lane == (x & 31) ? next : tpos;
      cur = next;
    }
    if (xb + lane < xe) trow[xb + lane] = tpos;
  }
  __syncwarp();
  // Integer tour length (order-free) and the transposed successor and
  // predecessor lists of the row-owned deposit, one edge per lane.
  const bool all_deposit = !c.epilogue_lists;
  int64_t len = 0;
#pragma unroll 8
  for (int i = lane; i < n; i += 32) {
    const int a0 = trow[i];
    const int b0 = trow[i + 1 == n ? 0 : i + 1];
    if ((unsigned)a0 < (unsigned)n && (unsigned)b0 < (unsigned)n) {
      len += c.dist[(size_t)a0 * c.ld + b0];
      if (all_deposit) {
        c.succT[(size_t)a0 * c.ldm + k] = b0;
        c.predT[(size_t)b0 * c.ldm + k] = a0;
      }
    } else {
      ok = false;
    }
  }
  for (int o = 16; o; o >>= 1) len += __shfl_xor_sync(kFull, len, o);
  if (!__all_sync(kFull, ok) && lane == 0) atomicOr(&c.st->error, kErrCheck);
  if (lane == 0) {
    c.newlen[k] = len;
    if (fallbacks)
      atomicAdd(reinterpret_cast<unsigned long long *>(&c.st->fallbacks),
                (unsigned long long)fallbacks);
  }
}

// One ant: position `pos` of the aging plan's list (k_aging_plan updated the
// ages; blend ants first, then the other valid ones, then the invalid ones),
// or ant `pos` without aging.  An invalid ant keeps a cleared tour
// (src/Colony.cu:507-510).
template <bool R1, bool AGING, bool LUT, bool STG>
__device__ __forceinline__ void rows_ant(const ColonyDev &c, const RowsView &v, int pos,
                                         uint32_t *mask, const RowsLut<LUT> &lut, int lane) {
  AntCtx a;
  a.blend = false;
  a.ratio = 0.0f;
  a.meanc = 0.0f;
  int k = pos;
  if (AGING) {
    k = c.plan[2 + pos];
    if (pos >= c.plan[0] + c.plan[1]) {
      int32_t *trow = c.tours + (size_t)k * c.ld;
      for (int i = lane; i < c.n; i += 32) trow[i] = 0;
      return;
    }
    const int age = c.age[k];
    a.blend = age < c.min_ret && c.st->isconverged;
    if (a.blend) a.ratio = __fdiv_rn(__int2float_rn(age), __int2float_rn(c.min_ret));
  }
  if (AGING && a.blend)
    rows_tour<R1, true, LUT, STG>(c, v, k, mask, lut, a, lane);
  else
    rows_tour<R1, false, LUT, STG>(c, v, k, mask, lut, a, lane);
}

__host__ __device__ constexpr int rows_words(bool r1) { return r1 ? 32 : kRowsMaskWords; }

// ---- kernels ----------------------------------------------------------------------

// Single colony: warp w of CTA b takes positions w * grid + b, + grid * warps,
// ... so that an aging colony's idle positions (the last ones) spread over
// the CTAs.
template <bool R1, bool AGING>
__global__ void __launch_bounds__(kRowsMaxAnts * 32, 1) k_construct_rows(const __grid_constant__ ColonyDev c) {
  __shared__ uint32_t masks[kRowsMaxAnts][rows_words(R1)];
  __shared__ RowsLut<true> lut;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  rows_lut_init(lut);
  const RowsView v = rows_view(c);
  for (int pos = warp * gridDim.x + blockIdx.x; pos < c.m; pos += gridDim.x * warps)
    rows_ant<R1, AGING, true, false>(c, v, pos, masks[warp], lut, lane);
}

// Single colony whose candidate rows fit in shared memory (full rows up to 190
// cities, n * k up to 36 000): every CTA copies choice values and ids by TMA,
// and a step waits for shared memory instead of L2 and sums in row order.
// Layout: [choice n * ldk f32][ids n * ldk int16][mbarrier].
template <bool AGING>
__global__ void __launch_bounds__(kRowsMaxAnts * 32, 1)
    k_construct_rows_staged(const __grid_constant__ ColonyDev c) {
  extern __shared__ __align__(128) unsigned char smem_rs[];
  __shared__ uint32_t masks[kRowsMaxAnts][rows_words(true)];
  __shared__ RowsLut<true> lut;  // for rows in city order only, which are never staged
  __shared__ int flag;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const uint32_t w_bytes = (uint32_t)c.n * c.ldk * 4u, id_bytes = (uint32_t)c.n * c.ldk * 2u;
  uint64_t *bar = reinterpret_cast<uint64_t *>(smem_rs + w_bytes + id_bytes);
  if (threadIdx.x == 0) {
    mbar_init(bar, 1);
    fence_barrier_init();
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    mbar_arrive_expect_tx(bar, w_bytes + id_bytes);
    constexpr uint32_t kPiece = 32768;
    const char *g = reinterpret_cast<const char *>(c.choice_nn);
    for (uint32_t o = 0; o < w_bytes; o += kPiece)
      tma_load_1d(smem_rs + o, g + o, min(kPiece, w_bytes - o), bar);
    g = reinterpret_cast<const char *>(c.nn16);
    for (uint32_t o = 0; o < id_bytes; o += kPiece)
      tma_load_1d(smem_rs + w_bytes + o, g + o, min(kPiece, id_bytes - o), bar);
    flag = mbar_wait_bounded(bar, 0, c.st) ? 1 : 0;
  }
  __syncthreads();
  if (!flag) return;
  RowsView v = rows_view(c);
  v.choice_nn = reinterpret_cast<const float *>(smem_rs);
  v.nn16 = reinterpret_cast<const int16_t *>(smem_rs + w_bytes);
  for (int pos = warp * gridDim.x + blockIdx.x; pos < c.m; pos += gridDim.x * warps)
    rows_ant<true, AGING, true, true>(c, v, pos, masks[warp], lut, lane);
}

size_t construct_rows_staged_bytes(int n, int ldk) { return (size_t)n * ldk * 6 + 16; }

cudaError_t configure_construct_rows_staged(size_t smem) {
  cudaError_t e = cudaFuncSetAttribute(k_construct_rows_staged<false>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_construct_rows_staged<true>,
                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  return e;
}

cudaError_t launch_construct_rows(const ColonyDev &c, int grid, int ants, bool staged,
                                  cudaStream_t s) {
  if (c.aging) {
    cudaError_t e = launch_aging_plan(c, s);
    if (e != cudaSuccess) return e;
  }
  const int threads = ants * 32;
  if (staged) {
    const size_t smem = construct_rows_staged_bytes(c.n, c.ldk);
    if (c.aging)
      k_construct_rows_staged<true><<<grid, threads, smem, s>>>(c);
    else
      k_construct_rows_staged<false><<<grid, threads, smem, s>>>(c);
  } else if (c.n <= 1024) {
    if (c.aging)
      k_construct_rows<true, true><<<grid, threads, 0, s>>>(c);
    else
      k_construct_rows<true, false><<<grid, threads, 0, s>>>(c);
  } else if (c.aging) {
    k_construct_rows<false, true><<<grid, threads, 0, s>>>(c);
  } else {
    k_construct_rows<false, false><<<grid, threads, 0, s>>>(c);
  }
  return cudaGetLastError();
}

// Batches: every warp takes (instance, position) items from the work queue
// (largest instances first) until it is empty, with its own copy of the
// instance's descriptor; no warp waits for another.
// 64 registers: 32 warps an SM.  They do not hold everything: the aging form,
// with both variants of the tour, spills 264 bytes of stores and 500 of loads,
// the other 116 and 164.  More registers and fewer warps were slower all the
// same: a pass of 5 iterations of 8 x n = 1000 took 23.4 ms, 23.8 at 80
// registers, 26.2 at 72 (28 warps), and 24.5 at 56 and 23.6 at 48, which spill
// more.
template <bool R1, bool AGING>
__global__ void __maxnreg__(64)
    k_batch_construct_rows(const ColonyDev *__restrict__ descs, const int4 *__restrict__ items,
                           int num_items, int *queue_head) {
  __shared__ uint32_t masks[kRowsMaxAnts][rows_words(R1)];
  __shared__ ColonyDev s_desc[kRowsMaxAnts];
  const RowsLut<false> lut;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int have = -1;
  for (;;) {
    int it = 0;
    if (lane == 0) it = atomicAdd(queue_head, 1);
    it = __shfl_sync(kFull, it, 0);
    if (it >= num_items) break;
    const int4 w = items[it];
    if (w.x != have) {  // words of the descriptor, one a lane
      static_assert(sizeof(ColonyDev) % 4 == 0, "copied by words");
      const uint32_t *src = reinterpret_cast<const uint32_t *>(descs + w.x);
      uint32_t *dst = reinterpret_cast<uint32_t *>(&s_desc[warp]);
      __syncwarp();
      for (int i = lane; i < (int)(sizeof(ColonyDev) / 4); i += 32) dst[i] = src[i];
      __syncwarp();
      have = w.x;
    }
    const RowsView v = rows_view(s_desc[warp]);
    for (int q = 0; q < w.z; q++)
      rows_ant<R1, AGING, false, false>(s_desc[warp], v, w.y + q, masks[warp], lut, lane);
  }
}

int batch_rows_blocks_per_sm(int ants, int max_n, bool aging) {
  const void *fn = max_n <= 1024 ? (aging ? (const void *)k_batch_construct_rows<true, true>
                                          : (const void *)k_batch_construct_rows<true, false>)
                                 : (aging ? (const void *)k_batch_construct_rows<false, true>
                                          : (const void *)k_batch_construct_rows<false, false>);
  int blocks = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, fn, ants * 32, 0) != cudaSuccess)
    return 1;
  return blocks > 0 ? blocks : 1;
}

cudaError_t launch_batch_construct_rows(const ColonyDev *descs, const int4 *items, int num_items,
                                        int *queue_head, int grid, int ants, int max_n, bool aging,
                                        cudaStream_t s) {
#define ACO_BATCH_ROWS(R1, AG) \
  k_batch_construct_rows<R1, AG><<<grid, ants * 32, 0, s>>>(descs, items, num_items, queue_head)
  if (max_n <= 1024) {
    if (aging)
      ACO_BATCH_ROWS(true, true);
    else
      ACO_BATCH_ROWS(true, false);
  } else {
    if (aging)
      ACO_BATCH_ROWS(false, true);
    else
      ACO_BATCH_ROWS(false, false);
  }
#undef ACO_BATCH_ROWS
  return cudaGetLastError();
}

}  // namespace aco
