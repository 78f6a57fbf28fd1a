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
//     the bounds; a 1e-44 is added for thresholds in the subnormal range;
//  4. otherwise -- u S' within the bound of a prefix, or a sum that is not
//     finite -- forms the reference's running sums themselves (rows_exact).
//     u falls into such a window in 0.1 to 3 % of the steps at n = 1000 (the
//     most with fresh pheromone on uniform instances, fewer later, when most
//     weights are smaller than the window) and in 5 to 8 % at n = 2392.
//
// Full rows without a learned prior are summed in city order, straight from
// the choice matrix: city 128 j + 4 l + t belongs to lane l, whose open
// (unvisited) cities are the bits 4 j + t of one register, so masking a
// weight is one predicated add with no lookup and no city ids, and a lane's
// four cities are not loaded once all are visited.  Other rows (k < n, the
// candidate heuristic carrying a prior, at most one chunk) are summed in row
// order.  Only the prefixes need ids, and usually one chunk of 128: the
// weights fall off with the distance (97 % of the steps at n = 1000).
//
// What bounds it: one ant's step is a chain of an L2 round trip and some
// fifteen shuffles; a batch keeps 32 independent warps an SM in flight and
// is bound by issue (about 320 instructions a step).  No warp waits for
// another.  The former kernel compacted every row into shared memory for a
// warp of the CTA that ran the sequential sums of all its ants in lockstep:
// a pass of 5 iterations of 8 x n = 1000 (m = 1000, setup included) took 95.7
// ms with it and 24.6 with this one, 10 iterations at n = 1501, k = 64 42.4
// and 12.6 ms, 2 iterations at n = 2392, m = 512 35.3 and 22.6 ms.
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

template <bool BLEND>
__device__ __forceinline__ void rows_load(const ColonyDev &c, int cur, int ch, float4 &w,
                                          float4 &e, uint2 &id, int lane) {
  const int p0 = ch * 128 + lane * 4;
  const size_t off = (size_t)cur * c.ldk + p0;
  const bool in = p0 < c.K;  // ldk % 4 == 0: the four entries are in the row
  id = in ? __ldg(reinterpret_cast<const uint2 *>(c.nn16 + off)) : make_uint2(0u, 0u);
  w = in ? __ldcg(reinterpret_cast<const float4 *>((BLEND ? c.tau_nn : c.choice_nn) + off))
         : make_float4(0.f, 0.f, 0.f, 0.f);
  if (BLEND)
    e = in ? __ldg(reinterpret_cast<const float4 *>(c.eta_nn + off))
           : make_float4(0.f, 0.f, 0.f, 0.f);
}

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

// The open cities of one round (1024 cities) of the choice row at offset
// `row` (a blending ant: their blended weights): chunks h .. h + JB - 1 of
// 128 cities, all loads first.  A set bit of `open` lies inside the instance,
// so a load that is made stays inside the row's pitch.
template <bool BLEND, int JB>
__device__ __forceinline__ void rows_round_load(const ColonyDev &c, size_t row, uint32_t open,
                                                int h, const AntCtx &a, float4 (&q)[JB]) {
#pragma unroll
  for (int j = 0; j < JB; j++) {
    const size_t off = row + (h + j) * 128;
    const bool need = (open >> (4 * (h + j))) & 0xfu;
    q[j] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (!BLEND) {
      if (need) q[j] = __ldcg(reinterpret_cast<const float4 *>(c.choice + off));
    } else if (need) {
      const float4 t = __ldcg(reinterpret_cast<const float4 *>(c.tau + off));
      const float4 e = __ldg(reinterpret_cast<const float4 *>(c.eta + off));
      q[j].x = blend_fitness(t.x, e.x, a.meanc, a.ratio, c.use_alpha, c.alpha);
      q[j].y = blend_fitness(t.y, e.y, a.meanc, a.ratio, c.use_alpha, c.alpha);
      q[j].z = blend_fitness(t.z, e.z, a.meanc, a.ratio, c.use_alpha, c.alpha);
      q[j].w = blend_fitness(t.w, e.w, a.meanc, a.ratio, c.use_alpha, c.alpha);
    }
  }
}

// Adds them to four running sums, one per float4 component (predicated adds).
template <int JB>
__device__ __forceinline__ void rows_round_add(const float4 (&q)[JB], uint32_t open, int h,
                                               float (&s)[4]) {
#pragma unroll
  for (int j = 0; j < JB; j++) {
    const uint32_t b = open >> (4 * (h + j));
    if (b & 1u) s[0] = __fadd_rn(s[0], q[j].x);
    if (b & 2u) s[1] = __fadd_rn(s[1], q[j].y);
    if (b & 4u) s[2] = __fadd_rn(s[2], q[j].z);
    if (b & 8u) s[3] = __fadd_rn(s[3], q[j].w);
  }
}

// This lane's part of the sum over the open cities of `cur`'s row, in city
// order (d_S: 8 adds a round, then the tree).  PIPE (several rounds, few
// warps an SM): the next round's loads are issued before this round's adds.
template <bool R1, bool BLEND, bool PIPE>
__device__ __forceinline__ float rows_city_sum(const ColonyDev &c, int cur, const uint32_t *mask,
                                               uint32_t own, const AntCtx &a, int lane) {
  float s[4] = {0.f, 0.f, 0.f, 0.f};
  const size_t row = (size_t)cur * c.ld + lane * 4;
  if constexpr (BLEND) {  // few ants blend: two chunks at a time, fewer registers
#pragma unroll 1
    for (int r = 0; r * 1024 < c.n; r++) {
      const uint32_t open = R1 ? own : mask[32 * r + lane];
#pragma unroll 1
      for (int h = 0; h < 8; h += 2) {
        float4 q[2];
        const uint32_t o2 = open >> (4 * h);
        rows_round_load<true, 2>(c, row + (size_t)r * 1024 + h * 128, o2, 0, a, q);
        rows_round_add<2>(q, o2, 0, s);
      }
    }
  } else if constexpr (R1) {
    float4 q[8];
    rows_round_load<false, 8>(c, row, own, 0, a, q);
    rows_round_add<8>(q, own, 0, s);
  } else if constexpr (!PIPE) {
#pragma unroll 1
    for (int r = 0; r * 1024 < c.n; r++) {
      float4 q[8];
      const uint32_t open = mask[32 * r + lane];
      rows_round_load<false, 8>(c, row + (size_t)r * 1024, open, 0, a, q);
      rows_round_add<8>(q, open, 0, s);
    }
  } else {
    const int R = (c.n + 1023) >> 10;
    float4 q0[8], q1[8];
    uint32_t o0 = mask[lane], o1 = 0u;
    rows_round_load<false, 8>(c, row, o0, 0, a, q0);
#pragma unroll 1
    for (int r = 0; r < R; r += 2) {
      o1 = r + 1 < R ? mask[32 * (r + 1) + lane] : 0u;
      rows_round_load<false, 8>(c, row + (size_t)(r + 1) * 1024, o1, 0, a, q1);
      rows_round_add<8>(q0, o0, 0, s);
      o0 = r + 2 < R ? mask[32 * (r + 2) + lane] : 0u;
      rows_round_load<false, 8>(c, row + (size_t)(r + 2) * 1024, o0, 0, a, q0);
      rows_round_add<8>(q1, o1, 0, s);
    }
  }
  return (s[0] + s[1]) + (s[2] + s[3]);
}

// ---- the rare paths -------------------------------------------------------------

// The reference's running sums over one chunk of 128 entries (four a lane, in
// order; visited ones 0): from the sum `s` before it to the sum after it, and
// in `pos` the first entry whose running sum exceeds `thr`, or -1.
//
// While the sum stays in one binade, with ulp 2^(e-23), adding w rounds to
// s + RN(w / ulp) ulp unless w / ulp lies halfway between two integers (then
// the parity of s decides).  The rounded terms are multiples of the ulp, so
// their sums below 2^(e+1) are exact in any order, and a scan gives every
// running sum.  RN(w / ulp) ulp is (w + M) - M with M = 1.5 2^e, for
// w < 2^(e-1).  The entries where that does not hold are added one at a
// time: those that would leave the binade (the scan shows the first), large
// ones, halfway cases; so is every non-zero entry while s is 0, outside
// 2^-90 .. 2^100 or not finite.  Each trip ends the chunk or adds one such
// entry, so there are at most 129.  A row has few of them: about log2(S / the
// first weight) binade changes, and a halfway case needs a weight within a
// few bits of the sum.
__device__ __forceinline__ float rows_walk(const float (&x)[4], float s, float thr, int lane,
                                           int &pos) {
  pos = -1;
  int start = 0;
  for (;;) {
    const uint32_t eb = __float_as_uint(s) & 0x7f800000u;
    const bool one = !(s >= 0x1p-90f && s <= 0x1p100f);
    const float M = __uint_as_float(eb | 0x00400000u);
    const float lim = __uint_as_float(eb + 0x00800000u);
    const float half_base = 0.5f * __uint_as_float(eb);
    const float half_ulp = __uint_as_float(one ? 0u : eb - (24u << 23));
    float v[4], t[4];
    unsigned ev = 0u;
#pragma unroll
    for (int q = 0; q < 4; q++) {
      v[q] = 4 * lane + q >= start ? x[q] : 0.0f;
      t[q] = one ? 0.0f : __fsub_rn(__fadd_rn(v[q], M), M);
      const bool special = one ? v[q] != 0.0f
                               : !(v[q] < half_base) || fabsf(__fsub_rn(v[q], t[q])) == half_ulp;
      if (special) {
        ev |= 1u << q;
        t[q] = 0.0f;  // only entries before the first special one are used
      }
    }
    const float t1 = t[0] + t[1], t2 = t1 + t[2], t3 = t2 + t[3];
    float incl = t3;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float y = __shfl_up_sync(kFull, incl, o);
      if (lane >= o) incl += y;
    }
    float ex = __shfl_up_sync(kFull, incl, 1);
    if (lane == 0) ex = 0.0f;
    // Running sums after each entry (before the first special one).
    const float r[4] = {s + (ex + t[0]), s + (ex + t1), s + (ex + t2), s + (ex + t3)};
    unsigned over = 0u;
#pragma unroll
    for (int q = 0; q < 4; q++) {
      if (!one && r[q] >= lim) ev |= 1u << q;
      if (r[q] > thr) over |= 1u << q;
    }
    const unsigned mev = __ballot_sync(kFull, ev != 0u), mov = __ballot_sync(kFull, over != 0u);
    int ie = 128, io = 128;  // first special entry, first entry past thr
    if (mev) ie = 4 * (__ffs(mev) - 1) + __ffs(__shfl_sync(kFull, ev, __ffs(mev) - 1)) - 1;
    if (mov) io = 4 * (__ffs(mov) - 1) + __ffs(__shfl_sync(kFull, over, __ffs(mov) - 1)) - 1;
    if (io < ie) {
      pos = io;
      return s;
    }
    if (ie >= 128) return s + __shfl_sync(kFull, incl, 31);
    const int l = ie >> 2, q = ie & 3;
    const float before = s + (q == 0 ? ex : ex + (q == 1 ? t[0] : q == 2 ? t1 : t2));
    const float w = q == 0 ? v[0] : q == 1 ? v[1] : q == 2 ? v[2] : v[3];
    s = __fadd_rn(__shfl_sync(kFull, before, l), __shfl_sync(kFull, w, l));
    if (s > thr) {
      pos = ie;
      return s;
    }
    start = ie + 1;
    if (start >= 128) return s;
  }
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
  const int nch = (c.K + 127) >> 7;  // at most 64
  float s = 0.0f, end0 = 0.0f, end1 = 0.0f;
  float4 w, e;
  uint2 id;
  int pos;
  rows_load<BLEND>(c, cur, 0, w, e, id, lane);
#pragma unroll 1
  for (int ch = 0; ch < nch; ch++) {
    const RowsChunk r = rows_mask<R1, BLEND>(c, mask, w, e, id, ch * 128 + lane * 4, a);
    rows_load<BLEND>(c, cur, ch + 1, w, e, id, lane);  // zeros past the row
    s = rows_walk(r.x, s, INFINITY, lane, pos);
    if (lane == (ch & 31)) (ch < 32 ? end0 : end1) = s;
  }
  if (s <= 0.0f) return -1;  // chooseBestNext (src/Colony.cu:776-778)
  const float rnd = __fmul_rn(u, s);
  if (rnd != rnd) {
    for (int ch = 0; ch < nch; ch++) {
      rows_load<BLEND>(c, cur, ch, w, e, id, lane);
      const unsigned ids[4] = {id.x & 0xffffu, id.x >> 16, id.y & 0xffffu, id.y >> 16};
      int first = -1;
#pragma unroll
      for (int t = 3; t >= 0; t--)
        if (ch * 128 + lane * 4 + t < c.K && rows_open<R1>(mask, ids[t])) first = (int)ids[t];
      const unsigned m = __ballot_sync(kFull, first >= 0);
      if (m) return __shfl_sync(kFull, first, __ffs(m) - 1);
    }
    return -1;
  }
  const unsigned h0 = __ballot_sync(kFull, lane < nch && end0 > rnd);
  const unsigned h1 = __ballot_sync(kFull, lane + 32 < nch && end1 > rnd);
  if (!h0 && !h1) return -1;
  const int ch = h0 ? __ffs(h0) - 1 : 31 + __ffs(h1);
  s = 0.0f;
  if (ch > 0) s = __shfl_sync(kFull, ch - 1 < 32 ? end0 : end1, (ch - 1) & 31);
  rows_load<BLEND>(c, cur, ch, w, e, id, lane);
  const RowsChunk r = rows_mask<R1, BLEND>(c, mask, w, e, id, ch * 128 + lane * 4, a);
  rows_walk(r.x, s, rnd, lane, pos);
  if (pos < 0) return -1;
  const unsigned v = (pos & 2) ? id.y : id.x;
  return (int)__shfl_sync(kFull, (pos & 1) ? v >> 16 : v & 0xffffu, pos >> 2);
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

// Inclusive scan over the warp.
__device__ __forceinline__ float rows_scan(float x, int lane) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const float y = __shfl_up_sync(kFull, x, o);
    if (lane >= o) x += y;
  }
  return x;
}

// The guarded pick of the header at city `cur` with `cnt` open cities or
// candidates left: the city, -1 (the weights are all zero: no pick), or
// kRowsAmbiguous.  `own` is this lane's mask word when R1.  Chunk 0 is
// loaded with the sum's rows and scanned while the sum is reduced, so the
// common step (the crossing in chunk 0: 97 % of the steps at n = 1000) waits
// for one L2 round trip and one chain of shuffles.
template <bool R1, bool BLEND, bool PIPE>
__device__ __forceinline__ int rows_pick(const ColonyDev &c, int cur, const uint32_t *mask,
                                         uint32_t own, bool natural, int cnt, float u,
                                         const AntCtx &a, int lane) {
  const int nch = (c.K + 127) >> 7;
  float4 w, e;
  uint2 id;
  rows_load<BLEND>(c, cur, 0, w, e, id, lane);
  // d_S + d_P + 8 and the entries of both sums: the error terms but for the
  // chunk of the crossing.
  int terms = cnt + 28 + nch;
  RowsChunk k;
  float xs, S, incl;
  if (natural) {
    S = rows_city_sum<R1, BLEND, PIPE>(c, cur, mask, own, a, lane);
    terms += (c.n + 1023) >> 10 << 3;
    k = rows_mask<R1, BLEND>(c, mask, w, e, id, lane * 4, a);
    xs = (k.x[0] + k.x[1]) + (k.x[2] + k.x[3]);
    incl = xs;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float y = __shfl_up_sync(kFull, incl, o);
      S += __shfl_xor_sync(kFull, S, o);
      if (lane >= o) incl += y;
    }
  } else {
    k = rows_mask<R1, BLEND>(c, mask, w, e, id, lane * 4, a);
    xs = (k.x[0] + k.x[1]) + (k.x[2] + k.x[3]);
    incl = rows_scan(xs, lane);
    S = 0.0f;
#pragma unroll 1
    for (int ch = 1; ch < nch; ch++) {
      rows_load<BLEND>(c, cur, ch, w, e, id, lane);
      const RowsChunk q = rows_mask<R1, BLEND>(c, mask, w, e, id, ch * 128 + lane * 4, a);
      S += (q.x[0] + q.x[1]) + (q.x[2] + q.x[3]);
    }
    if (nch > 1) {
#pragma unroll
      for (int o = 16; o; o >>= 1) S += __shfl_xor_sync(kFull, S, o);
    }
    S += __shfl_sync(kFull, incl, 31);
  }
  const float rnd = u * S;
  float base = 0.0f;
#pragma unroll 1
  for (int ch = 0;;) {
    float pe = __shfl_up_sync(kFull, incl, 1);  // prefix before this lane's entries
    if (lane == 0) pe = base;
    const float c1 = k.x[0] + k.x[1], c2 = c1 + k.x[2], c3 = c2 + k.x[3];
    const float p0 = pe + k.x[0], p1 = pe + c1, p2 = pe + c2, p3 = pe + c3;
    const float E = (float)(terms + min(cnt, 128 * (ch + 1))) * 6.08e-8f;  // 1.02 * 2^-24
    const unsigned hit = __ballot_sync(kFull, p3 > rnd);
    if (!(S > 0.0f && S < 1e38f)) return S == 0.0f ? -1 : kRowsAmbiguous;
    if (hit) {
      const float hi = __fadd_ru(__fmaf_ru(rnd, E, rnd), 1e-44f);
      const float lo = __fadd_rd(__fmaf_rd(rnd, -E, rnd), -1e-44f);
      float above = p0, below = pe;
      unsigned city = k.id.x & 0xffffu;
      if (!(p0 > rnd)) { above = p1; below = p0; city = k.id.x >> 16; }
      if (!(p1 > rnd)) { above = p2; below = p1; city = k.id.y & 0xffffu; }
      if (!(p2 > rnd)) { above = p3; below = p2; city = k.id.y >> 16; }
      const int mine = above > hi && below <= lo ? (int)city : kRowsAmbiguous;
      return __shfl_sync(kFull, mine, __ffs(hit) - 1);
    }
    if (++ch >= nch) return kRowsAmbiguous;  // u S' close to S'
    base = __shfl_sync(kFull, incl, 31);
    rows_load<BLEND>(c, cur, ch, w, e, id, lane);
    k = rows_mask<R1, BLEND>(c, mask, w, e, id, ch * 128 + lane * 4, a);
    xs = (k.x[0] + k.x[1]) + (k.x[2] + k.x[3]);
    incl = rows_scan(xs, lane) + base;
  }
}

// The tour of one valid ant.
template <bool R1, bool BLEND, bool PIPE>
__device__ __forceinline__ void rows_tour(const ColonyDev &c, int k, uint32_t *mask, AntCtx a,
                                          int lane) {
  const int n = c.n;
  int32_t *trow = c.tours + (size_t)k * c.ld;
  const bool natural = c.K == n && n > 128 && *c.prior_set == 0;
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
      int next = rows_pick<R1, BLEND, PIPE>(c, cur, mask, own, natural, min(c.K, n - x), u, a, lane);
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
  int64_t len = 0;
#pragma unroll 8
  for (int i = lane; i < n; i += 32) {
    const int a0 = trow[i];
    const int b0 = trow[i + 1 == n ? 0 : i + 1];
    if ((unsigned)a0 < (unsigned)n && (unsigned)b0 < (unsigned)n) {
      len += c.dist[(size_t)a0 * c.ld + b0];
      c.succT[(size_t)a0 * c.ldm + k] = b0;
      c.predT[(size_t)b0 * c.ldm + k] = a0;
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
template <bool R1, bool AGING, bool PIPE>
__device__ __forceinline__ void rows_ant(const ColonyDev &c, int pos, uint32_t *mask, int lane) {
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
    rows_tour<R1, true, PIPE>(c, k, mask, a, lane);
  else
    rows_tour<R1, false, PIPE>(c, k, mask, a, lane);
}

__host__ __device__ constexpr int rows_words(bool r1) { return r1 ? 32 : kRowsMaskWords; }

// ---- kernels ----------------------------------------------------------------------

// Single colony: warp w of CTA b takes positions w * grid + b, + grid * warps,
// ... so that an aging colony's idle positions (the last ones) spread over
// the CTAs.
template <bool R1, bool AGING>
__global__ void __launch_bounds__(kRowsMaxAnts * 32) k_construct_rows(const __grid_constant__ ColonyDev c) {
  __shared__ uint32_t masks[kRowsMaxAnts][rows_words(R1)];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  for (int pos = warp * gridDim.x + blockIdx.x; pos < c.m; pos += gridDim.x * warps)
    rows_ant<R1, AGING, !R1>(c, pos, masks[warp], lane);
}

cudaError_t launch_construct_rows(const ColonyDev &c, int grid, int ants, cudaStream_t s) {
  if (c.aging) {
    cudaError_t e = launch_aging_plan(c, s);
    if (e != cudaSuccess) return e;
    if (c.n <= 1024)
      k_construct_rows<true, true><<<grid, ants * 32, 0, s>>>(c);
    else
      k_construct_rows<false, true><<<grid, ants * 32, 0, s>>>(c);
  } else if (c.n <= 1024) {
    k_construct_rows<true, false><<<grid, ants * 32, 0, s>>>(c);
  } else {
    k_construct_rows<false, false><<<grid, ants * 32, 0, s>>>(c);
  }
  return cudaGetLastError();
}

// Batches: every warp takes (instance, position) items from the work queue
// (largest instances first) until it is empty, with its own copy of the
// instance's descriptor; no warp waits for another.
// Three CTAs of 11 warps an SM (56 registers): the pass named in the header
// took 32.2 ms at 84 to 108 registers, 26.1 at 80 and 24.6 at 56.
template <bool R1, bool AGING>
__global__ void __launch_bounds__(kRowsMaxAnts * 32, 3)
    k_batch_construct_rows(const ColonyDev *__restrict__ descs, const int4 *__restrict__ items,
                           int num_items, int *queue_head) {
  __shared__ uint32_t masks[kRowsMaxAnts][rows_words(R1)];
  __shared__ ColonyDev s_desc[kRowsMaxAnts];
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
    for (int q = 0; q < w.z; q++)
      rows_ant<R1, AGING, false>(s_desc[warp], w.y + q, masks[warp], lane);
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
