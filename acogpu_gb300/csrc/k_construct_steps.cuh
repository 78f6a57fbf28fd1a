// k_construct_steps.cuh -- roulette-wheel tour construction, one warp per
// ant: the device code shared by the construction kernels (k_construct.cu:
// general, staged and direct; k_construct_cluster.cu; k_construct_batch.cu).
//
// Replaces Colony::initTour + constructPath (src/Colony.cu:469-527,
// 689-864) and the reference GPU kernels dev_place_ants /
// dev_compute_probabilities / dev_reduce_probabilities_s / dev_move_ants
// (inc/Colony.cuh:136-162,193-229,290-347; src/Colony.cu:643-685), which the
// reference launches 3(n-1) times per iteration with a device sync after
// each.  Here one launch builds every tour.  Two step loops:
//
//  * construct_ant (any k, full rows included): the tabu list is a bitmask
//    in shared memory; the non-zero weights of each 32-candidate chunk are
//    compacted by ballot and folded in lane order, so every partial sum is
//    the reference's sequential float sum (sum_prob += prob_ptr[i],
//    src/Colony.cu:814; partial_sum += ..., :840); rows longer than 32 keep
//    the prefix at each chunk end and redo only the chunk of the crossing;
//  * staged_steps (k <= 32; the staged, cluster, direct and batch kernels):
//    lane r holding candidate r of the current row, the pick settled by
//    bounded sums (see staged_steps), the rows read through a policy
//    (TableRows: shared or global memory; ClusterRows: distributed shared
//    memory of a thread-block cluster).
//
// In both, the crossing `first i with partial_sum > u * sum` is a ballot;
// when the roulette cannot pick (sum <= 0, or no crossing) the fallback is
// the last unvisited city of the full nn row (select_local_best,
// inc/Colony.cuh:33-43) or the unvisited city with the largest choice value
// (through the second tier where the colony keeps one, see fallback_tier2).
// Ant aging (updateAntAges, src/Colony.cu:353-364; compute_fittness,
// inc/Colony.cuh:14-31) is fused in; the integer tour length (the reference
// adds it per move, inc/Colony.cuh:337-340) is summed by the whole warp after
// the tour is built, so no step waits on a distance load; the
// successor/predecessor of every city is written transposed for the
// row-owned deposit.
#pragma once
#include <cuda_runtime.h>

#include "aco_kernels.h"

namespace aco {

__device__ __forceinline__ bool visited(const uint32_t *tabu, int city) {
  return (tabu[city >> 5] >> (city & 31)) & 1u;
}

// Ordered fold of one chunk of 32 candidates.  The reference adds every
// weight of the row in order, zeros included (src/Colony.cu:801-816); adding
// +0 leaves a non-negative float sum unchanged, so only the non-zero weights
// need to be added, still in lane order.  They are compacted through a
// 32-float shared buffer (ballot + popc rank), then folded with broadcast
// reads; `mine` receives the prefix that ends at this lane's weight (only
// meaningful for lanes with a non-zero weight).
__device__ __forceinline__ float fold_nonzero(float s, float w, int lane, float *wbuf,
                                              float &mine) {
  const unsigned nz = __ballot_sync(kFull, w != 0.0f);
  const int cnt = __popc(nz);
  const int rank = __popc(nz & ((1u << lane) - 1u));
  if (w != 0.0f) wbuf[rank] = w;
  __syncwarp();
  mine = s;
  int i = 0;
#pragma unroll 1
  for (; i + 4 <= cnt; i += 4) {
    const float a0 = wbuf[i], a1 = wbuf[i + 1], a2 = wbuf[i + 2], a3 = wbuf[i + 3];
    s = __fadd_rn(s, a0);
    mine = (rank == i) ? s : mine;
    s = __fadd_rn(s, a1);
    mine = (rank == i + 1) ? s : mine;
    s = __fadd_rn(s, a2);
    mine = (rank == i + 2) ? s : mine;
    s = __fadd_rn(s, a3);
    mine = (rank == i + 3) ? s : mine;
  }
  for (; i < cnt; i++) {
    s = __fadd_rn(s, wbuf[i]);
    mine = (rank == i) ? s : mine;
  }
  __syncwarp();
  return s;
}

// compute_fittness with the aging blend (inc/Colony.cuh:21-30), every
// operation rounded once.
__device__ __forceinline__ float blend_fitness(float tau, float eta, float meanc, float ratio,
                                               int use_alpha, float alpha) {
  float p = __fadd_rn(__fmul_rn(__fsub_rn(tau, meanc), ratio), meanc);
  if (use_alpha) p = powf(p, alpha);
  return __fmul_rn(p, eta);
}

struct AntCtx {
  bool blend;
  float ratio, meanc;
};

// Candidate r of the row of `cur`: id (or -1) and its weight (0 if visited).
template <bool STAGED>
__device__ __forceinline__ void candidate(const ColonyDev &c, int cur, int r,
                                          const uint32_t *tabu, const int16_t *sids,
                                          const float *scw, const AntCtx &a, int &id, float &w) {
  id = -1;
  w = 0.0f;
  if (r >= c.K) return;
  if (!a.blend) {
    float cw;
    if (STAGED) {
      id = sids[cur * 32 + r];
      cw = scw[cur * 32 + r];
    } else {
      const size_t off = (size_t)cur * c.ldk + r;
      id = __ldg(c.nn + off);
      cw = c.choice_nn[off];
    }
    if (!visited(tabu, id)) w = cw;
  } else {
    const size_t off = (size_t)cur * c.ldk + r;
    id = STAGED ? (int)sids[cur * 32 + r] : __ldg(c.nn + off);
    const float t = c.tau_nn[off];
    const float e = __ldg(c.eta_nn + off);
    if (!visited(tabu, id)) w = blend_fitness(t, e, a.meanc, a.ratio, c.use_alpha, c.alpha);
  }
}

// Fallback choice at city `cur` (warp-uniform result, -1 if none).
static __device__ int fallback_city(const ColonyDev &c, int cur, const uint32_t *tabu,
                                    const AntCtx &a, int lane) {
  if (c.fallback == ACO_FALLBACK_REFERENCE) {
    // select_local_best: last unvisited city of the full nn row.
    const int32_t *ids = c.nn + (size_t)cur * c.ldk;
    for (int ch = ((c.K + 31) >> 5) - 1; ch >= 0; ch--) {
      const int r = ch * 32 + lane;
      const int id = r < c.K ? __ldg(ids + r) : -1;
      const unsigned m = __ballot_sync(kFull, id >= 0 && !visited(tabu, id));
      if (m) return __shfl_sync(kFull, id, 31 - __clz(m));
    }
    return -1;
  }
  // Largest choice value among unvisited cities, lowest index on ties.  Each
  // lane scans groups of 4 consecutive cities with float4 loads (rows are
  // 128-byte aligned); the loads of a lane are independent of each other.
  float bw = -1.0f;
  int bj = -1;
  const float *crow = c.choice + (size_t)cur * c.ld;
  const float *trow = c.tau + (size_t)cur * c.ld;
  const float *erow = c.eta + (size_t)cur * c.ld;
#pragma unroll 2
  for (int j4 = lane * 4; j4 < c.n; j4 += 128) {
    const uint32_t bits = (tabu[j4 >> 5] >> (j4 & 31)) & 0xfu;
    if (bits == 0xfu) continue;
    float v[4];
    if (!a.blend) {
      const float4 q = *reinterpret_cast<const float4 *>(crow + j4);
      v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
    } else {
      const float4 t = *reinterpret_cast<const float4 *>(trow + j4);
      const float4 e = *reinterpret_cast<const float4 *>(erow + j4);
      v[0] = blend_fitness(t.x, e.x, a.meanc, a.ratio, c.use_alpha, c.alpha);
      v[1] = blend_fitness(t.y, e.y, a.meanc, a.ratio, c.use_alpha, c.alpha);
      v[2] = blend_fitness(t.z, e.z, a.meanc, a.ratio, c.use_alpha, c.alpha);
      v[3] = blend_fitness(t.w, e.w, a.meanc, a.ratio, c.use_alpha, c.alpha);
    }
#pragma unroll
    for (int q = 0; q < 4; q++) {
      if (!((bits >> q) & 1u) && j4 + q < c.n && v[q] > bw) {
        bw = v[q];
        bj = j4 + q;
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

// SIGNED: weights may be negative.
template <bool MULTI, bool AGING, bool STAGED, bool SIGNED = false>
__device__ void construct_ant(const ColonyDev &c, int k, uint32_t iter, uint32_t *tabu,
                              float *cend, float *wbuf, const int16_t *sids, const float *scw,
                              const float *smean, int nchunks, int lane) {
  const int n = c.n;
  const int words = (n + 31) >> 5;
  int32_t *trow = c.tours + (size_t)k * c.ld;

  AntCtx a;
  a.blend = false;
  a.ratio = 0.0f;
  a.meanc = 0.0f;
  if (AGING) {
    int age = 0;
    if (lane == 0) {
      age = c.age[k] + 1;
      c.age[k] = age;
    }
    age = __shfl_sync(kFull, age, 0);
    if (!c.valid[k]) {  // invalid ants keep a cleared tour (src/Colony.cu:507-510)
      for (int i = lane; i < n; i += 32) trow[i] = 0;
      return;
    }
    a.blend = age < c.min_ret && c.st->isconverged;
    if (a.blend) a.ratio = __fdiv_rn(__int2float_rn(age), __int2float_rn(c.min_ret));
  }
  for (int w = lane; w < words; w += 32) tabu[w] = 0;
  __syncwarp();

  // initTour placement (src/Colony.cu:518-520)
  const uint32_t akey = aco_ant_key(c.seed, iter, (uint32_t)k);
  const float u0 = aco_uniform_key(akey, 0u);
  int start = __float2int_rz(__fmul_rn(u0, __int2float_rn(n)));
  if (start >= n) {  // impossible for u0 < 1; recorded, clamped
    if (lane == 0) atomicOr(&c.st->error, kErrCheck);
    start = n - 1;
  }
  if (lane == 0) {
    tabu[start >> 5] |= 1u << (start & 31);
    trow[0] = start;
  }
  __syncwarp();

  int cur = start;
  int64_t fallbacks = 0;
  for (int x = 1; x < n; x++) {
    const float u = aco_uniform_key(akey, (uint32_t)x);
    if (AGING && a.blend) a.meanc = STAGED ? smean[cur] : c.mean[cur];
    int next = -1;
    if (!MULTI) {
      int id;
      float w;
      candidate<STAGED>(c, cur, lane, tabu, sids, scw, a, id, w);
      float p;
      const float S = fold_nonzero(0.0f, w, lane, wbuf, p);
      if (!(S <= 0.0f)) {
        const float rnd = __fmul_rn(u, S);
        const unsigned hit = __ballot_sync(kFull, w != 0.0f && !(p <= rnd));
        if (hit) next = __shfl_sync(kFull, id, __ffs(hit) - 1);
      }
    } else {
      float s = 0.0f;
      for (int ch = 0; ch < nchunks; ch++) {
        int id;
        float w;
        candidate<false>(c, cur, ch * 32 + lane, tabu, sids, scw, a, id, w);
        if (__ballot_sync(kFull, w != 0.0f)) {
          float p;
          s = fold_nonzero(s, w, lane, wbuf, p);
        }
        if (lane == 0) cend[ch] = s;
      }
      __syncwarp();
      const float S = s;
      if (!(S <= 0.0f)) {
        const float rnd = __fmul_rn(u, S);
        int found = -1;
        for (int base = 0; base < nchunks && !SIGNED; base += 32) {
          const int q = base + lane;
          const unsigned m = __ballot_sync(kFull, q < nchunks && !(cend[q] <= rnd));
          if (m) {
            found = base + __ffs(m) - 1;
            break;
          }
        }
        // Sums of negative weights too may pass rnd inside a chunk and end below
        // it: every chunk is walked again, up to the first that has the crossing.
        for (int ch = 0; ch < nchunks && SIGNED && next < 0; ch++) {
          int id;
          float w;
          candidate<false>(c, cur, ch * 32 + lane, tabu, sids, scw, a, id, w);
          float p;
          fold_nonzero(ch > 0 ? cend[ch - 1] : 0.0f, w, lane, wbuf, p);
          const unsigned hit = __ballot_sync(kFull, w != 0.0f && !(p <= rnd));
          if (hit) next = __shfl_sync(kFull, id, __ffs(hit) - 1);
        }
        if (found >= 0) {
          const float s0 = found > 0 ? cend[found - 1] : 0.0f;
          const int r = found * 32 + lane;
          int id;
          float w;
          candidate<false>(c, cur, r, tabu, sids, scw, a, id, w);
          float p;
          fold_nonzero(s0, w, lane, wbuf, p);
          const unsigned hit = __ballot_sync(kFull, w != 0.0f && !(p <= rnd));
          if (hit) next = __shfl_sync(kFull, id, __ffs(hit) - 1);
        }
      }
      __syncwarp();
    }
    if (next < 0) {
      next = fallback_city(c, cur, tabu, a, lane);
      fallbacks++;
      if (next < 0 || next >= n) {  // no unvisited city: cannot happen
        if (lane == 0) atomicOr(&c.st->error, kErrCheck);
        break;
      }
    }
    if (lane == 0) {
      tabu[next >> 5] |= 1u << (next & 31);
      trow[x] = next;
      c.succT[(size_t)cur * c.ldm + k] = next;
      c.predT[(size_t)next * c.ldm + k] = cur;
    }
    __syncwarp();
    cur = next;
  }
  if (lane == 0) {
    c.succT[(size_t)cur * c.ldm + k] = start;
    c.predT[(size_t)start * c.ldm + k] = cur;
  }
  __syncwarp();
  // Integer tour length, summed by the whole warp (order-free).
  int64_t len = 0;
  for (int i = lane; i < n; i += 32) {
    const int a0 = trow[i];
    const int b0 = trow[i + 1 == n ? 0 : i + 1];
    if ((unsigned)a0 < (unsigned)n && (unsigned)b0 < (unsigned)n)
      len += c.dist[(size_t)a0 * c.ld + b0];
    else
      atomicOr(&c.st->error, kErrCheck);
  }
  for (int o = 16; o; o >>= 1) len += __shfl_xor_sync(kFull, len, o);
  if (lane == 0) {
    c.newlen[k] = len;
    if (fallbacks)
      atomicAdd(reinterpret_cast<unsigned long long *>(&c.st->fallbacks),
                (unsigned long long)fallbacks);
  }
}

// ---------------------------------------------------------------------------
// Staged construction step, specialised for the short critical path of one
// ant: candidate rows in shared memory, the tabu bitmask in registers (lane
// l owns the 32-city words l, l+32, ...; a lookup is one __shfl_sync and the
// owner lane sets the bit).
// TW words per lane cover 1024*TW cities: word w of the tabu list is held
// by lane w % 32 as its register w / 32.  A city past the list (a padding id)
// reads as unvisited.
template <int TW>
__device__ __forceinline__ uint32_t reg_word(const uint32_t (&tw)[TW], int city) {
  const int word = city >> 5;
  uint32_t v = __shfl_sync(kFull, tw[0], word & 31);
#pragma unroll
  for (int t = 1; t < TW; t++) {
    const uint32_t x = __shfl_sync(kFull, tw[t], word & 31);
    v = (word >> 5) == t ? x : v;
  }
  if (TW > 1 && (word >> 5) >= TW) v = 0u;
  return v;
}

// Every register is updated (with the bit or with 0), so the compiler never
// turns the update into a store at a computed index.
template <int TW>
__device__ __forceinline__ void reg_mark(uint32_t (&tw)[TW], int city, int lane) {
  const int word = city >> 5;
  const uint32_t bit = lane == (word & 31) ? 1u << (city & 31) : 0u;
  if constexpr (TW == 1) {  // every city is below 1024
    tw[0] |= bit;
  } else {
#pragma unroll
    for (int t = 0; t < TW; t++) tw[t] |= (word >> 5) == t ? bit : 0u;
  }
}

// Register t of the tabu words, t uniform across the warp (a select chain,
// so the array never needs a dynamic index).
template <int TW>
__device__ __forceinline__ uint32_t tw_pick(const uint32_t (&tw)[TW], int t) {
  uint32_t v = tw[0];
#pragma unroll
  for (int i = 1; i < TW; i++) v = t == i ? tw[i] : v;
  return v;
}

// The tabu list of the step loop: in registers for up to 2048 cities, else as
// TW * 32 words of shared memory (TW shuffles and selects a lookup cost more
// there than one load).
template <int TW>
struct StepTabu {
  static constexpr bool kShared = TW > 2;
  uint32_t tw[kShared ? 1 : TW];
  uint32_t *words;
  __device__ __forceinline__ void clear(int lane) {
    if constexpr (kShared) {
#pragma unroll
      for (int t = 0; t < TW; t++) words[t * 32 + lane] = 0u;
      __syncwarp();
    } else {
#pragma unroll
      for (int t = 0; t < TW; t++) tw[t] = 0u;
    }
  }
  // Every lane takes part; an id past the list (the -1 of a row's padding)
  // gives either answer, its weight is 0.
  __device__ __forceinline__ bool visited(int id) const {
    uint32_t v;
    if constexpr (kShared) v = words[(id >> 5) & (TW * 32 - 1)];
    else v = reg_word(tw, id & 0xffff);
    return (v >> (id & 31)) & 1u;
  }
  __device__ __forceinline__ void mark(int city, int lane) {
    if constexpr (kShared) {
      if (lane == 0) words[city >> 5] |= 1u << (city & 31);
      __syncwarp();
    } else {
      reg_mark(tw, city, lane);
    }
  }
  // The words as registers (the fallback's layout).
  __device__ __forceinline__ void words_of(uint32_t (&out)[TW], int lane) const {
#pragma unroll
    for (int t = 0; t < TW; t++) {
      if constexpr (kShared) out[t] = words[t * 32 + lane];
      else out[t] = tw[t];
    }
  }
};

// x plus the values of the lanes before it, up to lane - 2 o + 1, in its
// segment of W lanes: one level of an inclusive scan.
template <int W>
__device__ __forceinline__ float scan_level(float x, int o) {
  asm("{\n\t.reg .f32 y;\n\t.reg .pred p;\n\t"
      "shfl.sync.up.b32 y|p, %0, %1, %2, 0xffffffff;\n\t"
      "@p add.f32 %0, %0, y;\n\t}"
      : "+f"(x)
      : "r"(o), "n"((32 - W) << 8));
  return x;
}

// The best-choice fallback over the whole row: the unvisited city with the
// largest choice value (a blending ant: its blended weight), lowest index on
// ties, -1 if there is none.  Weights are non-negative, so their bits order
// like they do, and a visited city's are masked to 0: a lane keeps the
// largest of its cities chunk by chunk (128 cities, four a lane, the chunk's
// four values kept with it), one warp maximum gives the value and one warp
// minimum the lowest city that has it.  AHEAD (not in the batch kernel, whose
// many warps cover the loads and whose registers the buffers would cost: 37.2
// ms of construction for 512 instances with it, 27 without): a group of chunks
// is loaded ahead of the one being compared, four (n <= 2048; the whole row at
// n = 1000 takes two groups), eight (n = 4096: construction 1436 us with four,
// 1374 with eight) or, AHEAD = 2, sixteen (n = 8000, k = 20, rank-based 4562 us an
// iteration with eight, 4151 with sixteen); of a blending ant, whose chunks take
// twice the registers, four, and above 2048 cities with AHEAD = 2 only.  If the
// largest value is 0 the lowest unvisited city is the answer, from the tabu words
// alone, and a row with a NaN is scanned again without it (fallback_rest).
template <int TW>
struct TwPack {
  uint32_t w[TW];
};

// One lane's four weights at cities j4 .. j4 + 3 (j4 < n: inside the row's
// pitch; padding has eta 0, so weight 0).
__device__ __forceinline__ uint4 fallback_load(const ColonyDev &c, size_t row, int j4,
                                               const AntCtx &a) {
  uint4 q = make_uint4(0u, 0u, 0u, 0u);
  if (j4 >= c.n) return q;
  if (!a.blend) return __ldcg(reinterpret_cast<const uint4 *>(c.choice + row + j4));
  const float4 t = __ldcg(reinterpret_cast<const float4 *>(c.tau + row + j4));
  const float4 e = __ldg(reinterpret_cast<const float4 *>(c.eta + row + j4));
  q.x = __float_as_uint(blend_fitness(t.x, e.x, a.meanc, a.ratio, c.use_alpha, c.alpha));
  q.y = __float_as_uint(blend_fitness(t.y, e.y, a.meanc, a.ratio, c.use_alpha, c.alpha));
  q.z = __float_as_uint(blend_fitness(t.z, e.z, a.meanc, a.ratio, c.use_alpha, c.alpha));
  q.w = __float_as_uint(blend_fitness(t.w, e.w, a.meanc, a.ratio, c.use_alpha, c.alpha));
  return q;
}

// The tabu word that holds cities j4 .. j4 + 3 (j4 a multiple of four, lane
// l's at 128 t + 4 l), shifted so that they are its low bits.
template <int TW>
__device__ __forceinline__ uint32_t fallback_bits(const TwPack<TW> &p, int t, int lane) {
  const uint32_t v = __shfl_sync(kFull, tw_pick(p.w, t >> 3), (t * 4 + (lane >> 3)) & 31);
  return v >> ((lane * 4) & 31);
}

template <int TW>
__device__ __noinline__ int fallback_rest(const ColonyDev &c, int cur, TwPack<TW> p, AntCtx a,
                                          int lane, bool zero) {
  if (zero) {
    unsigned first = ~0u;
#pragma unroll
    for (int t = TW - 1; t >= 0; t--)
      if (~p.w[t]) first = (unsigned)(32 * (lane + 32 * t) + __ffs(~p.w[t]) - 1);
    first = __reduce_min_sync(kFull, first);
    return first < (unsigned)c.n ? (int)first : -1;
  }
  float bw = -1.0f;
  int bj = -1;
  const size_t row = (size_t)cur * c.ld;
#pragma unroll 1
  for (int t = 0; t * 128 < c.n; t++) {
    const int j4 = t * 128 + lane * 4;
    const uint32_t b = fallback_bits(p, t, lane);
    const uint4 q = fallback_load(c, row, j4, a);
    const float v[4] = {__uint_as_float(q.x), __uint_as_float(q.y), __uint_as_float(q.z),
                        __uint_as_float(q.w)};
#pragma unroll
    for (int r = 0; r < 4; r++)
      if (!((b >> r) & 1u) && j4 + r < c.n && v[r] > bw) {
        bw = v[r];
        bj = j4 + r;
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

// The raw loads of GR chunks from chunk t0 on: choice values, or for a
// blending ant (BL) tau and eta, blended when they are used -- every load of
// a group is issued before any is waited for.
template <bool BL, int GR>
__device__ __forceinline__ void fallback_group(const ColonyDev &c, size_t row, int t0, int lane,
                                               uint4 (&q)[GR], uint4 (&e)[GR]) {
#pragma unroll
  for (int t = 0; t < GR; t++) {
    const int j4 = (t0 + t) * 128 + lane * 4;
    const bool in = j4 < c.n;
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    q[t] = in ? __ldcg(reinterpret_cast<const uint4 *>((BL ? c.tau : c.choice) + row + j4)) : zero;
    if (BL) e[t] = in ? __ldg(reinterpret_cast<const uint4 *>(c.eta + row + j4)) : zero;
  }
}

__device__ __forceinline__ uint32_t blend_bits(const ColonyDev &c, uint32_t t, uint32_t e,
                                               const AntCtx &a) {
  return __float_as_uint(blend_fitness(__uint_as_float(t), __uint_as_float(e), a.meanc, a.ratio,
                                       c.use_alpha, c.alpha));
}

template <int TW, bool BL, int AHEAD>
__device__ __forceinline__ int fallback_scan(const ColonyDev &c, int cur, const TwPack<TW> &p,
                                             const AntCtx &a, int lane) {
  constexpr int GR = TW > 2 && !BL && AHEAD ? 8 * AHEAD : 4;  // chunks a group
  const size_t row = (size_t)cur * c.ld;
  unsigned best = 0u;
  int bt = 0;
  uint4 bq = make_uint4(0u, 0u, 0u, 0u), q[GR], e[GR], nq[GR], ne[GR];
  if (AHEAD) fallback_group<BL, GR>(c, row, 0, lane, q, e);
#pragma unroll 1
  for (int t0 = 0; t0 * 128 < c.n; t0 += GR) {
    if (AHEAD)
      fallback_group<BL, GR>(c, row, t0 + GR, lane, nq, ne);
    else
      fallback_group<BL, GR>(c, row, t0, lane, q, e);
    unsigned m[GR];
#pragma unroll
    for (int t = 0; t < GR; t++) {
      const uint32_t b = fallback_bits(p, t0 + t, lane);
      uint4 &v = q[t];
      if (BL) {
        v.x = blend_bits(c, v.x, e[t].x, a);
        v.y = blend_bits(c, v.y, e[t].y, a);
        v.z = blend_bits(c, v.z, e[t].z, a);
        v.w = blend_bits(c, v.w, e[t].w, a);
      }
      v.x &= ~(uint32_t)((int32_t)(b << 31) >> 31);
      v.y &= ~(uint32_t)((int32_t)(b << 30) >> 31);
      v.z &= ~(uint32_t)((int32_t)(b << 29) >> 31);
      v.w &= ~(uint32_t)((int32_t)(b << 28) >> 31);
      m[t] = max(max(v.x, v.y), max(v.z, v.w));
    }
#pragma unroll
    for (int t = 0; t < GR; t++)
      if (m[t] > best) {
        best = m[t];
        bt = t0 + t;
        bq = q[t];
      }
    if (AHEAD) {
#pragma unroll
      for (int t = 0; t < GR; t++) {
        q[t] = nq[t];
        e[t] = ne[t];
      }
    }
  }
  const unsigned m = __reduce_max_sync(kFull, best);
  if (m == 0u || m > 0x7f800000u) return fallback_rest<TW>(c, cur, p, a, lane, m == 0u);
  const int r = bq.x == m ? 0 : bq.y == m ? 1 : bq.z == m ? 2 : 3;
  return (int)__reduce_min_sync(kFull, best == m ? (unsigned)(bt * 128 + lane * 4 + r) : ~0u);
}

// The fallback's second tier: the largest plain choice value among the
// unvisited cities of the row's k candidates (this lane's) and of its tier
// (the next t2 nearest neighbours, up to four a lane), lowest index on ties.
// Every other city of the row has a choice value of at most mout[cur] (the
// row pass's maximum outside them; NaNs, which the fallback never picks,
// left out), so when the tier's best is larger it is the full scan's answer;
// otherwise -1 sends the step to the full scan.  One L2 round trip instead
// of a pass over the row.  The candidates count too because the fallback also
// runs when u*S rounds up to S with unvisited candidates left; their value
// is read from the choice matrix, as the full scan does, not from the
// candidate table (which may carry a learned prior).
template <int TW>
__device__ __forceinline__ int fallback_tier2(const ColonyDev &c, int cur,
                                              const TwPack<TW> &p, int id, bool vis, int lane) {
  constexpr int Q = kTier2 / 32;
  const size_t base = (size_t)cur * kTier2;
  const bool own = lane < c.K && (unsigned)id < (unsigned)c.n && !vis;
  const float v1 = own ? __ldcg(c.choice + (size_t)cur * c.ld + id) : -1.0f;
  int id2[Q];
  float v2[Q];
#pragma unroll
  for (int q = 0; q < Q; q++) {
    const int e = lane + 32 * q;
    const bool in = e < c.t2;
    id2[q] = in ? __ldg(c.nn2 + base + e) : -1;
    v2[q] = in ? __ldcg(c.t2v + base + e) : -1.0f;
  }
  const float mo = __ldcg(c.mout + cur);
  float bw = -1.0f;
  int bj = -1;
  if (own && v1 > bw) {
    bw = v1;
    bj = id;
  }
#pragma unroll
  for (int q = 0; q < Q; q++) {
    const int city = (unsigned)id2[q] < (unsigned)c.n ? id2[q] : -1;
    const int at = city < 0 ? 0 : city;
    const bool seen = (reg_word(p.w, at) >> (at & 31)) & 1u;  // every lane takes part
    if (city >= 0 && !seen && (v2[q] > bw || (v2[q] == bw && city < bj))) {
      bw = v2[q];
      bj = city;
    }
  }
  // Values are at least 0 where a city was found, so their bits order like
  // they do; a NaN is never kept above.
  const unsigned bits = bj >= 0 ? __float_as_uint(bw) + 1u : 0u;
  const unsigned m = __reduce_max_sync(kFull, bits);
  const unsigned j = __reduce_min_sync(kFull, m != 0u && bits == m ? (unsigned)bj : ~0u);
  return m != 0u && __uint_as_float(m - 1u) > mo ? (int)j : -1;
}

// The whole best-choice fallback, as a called function (the tabu words by
// value, so they stay in registers): its code stays out of the step loop.
template <int TW, int AHEAD>
__device__ __noinline__ int fallback_best(const ColonyDev &c, int cur, TwPack<TW> p, AntCtx a,
                                          int lane, int id, bool vis, bool tier_ok) {
  int next = -1;
  if (tier_ok && c.t2 > 0) next = fallback_tier2<TW>(c, cur, p, id, vis, lane);
  if (next < 0)
    next = a.blend
               ? fallback_scan<TW, true, TW <= 2 || AHEAD == 2 ? AHEAD : 0>(c, cur, p, a, lane)
               : fallback_scan<TW, false, AHEAD>(c, cur, p, a, lane);
  return next;
}

// Where the step loop reads the candidate rows (pitch SP): a whole table in
// shared or global memory, or -- in a thread-block cluster -- the slice of
// the CTA that owns the row (rows r*1024 .. r*1024+1023 in cluster rank r,
// at the same shared-memory offsets in every CTA), through DSMEM.
template <int SP>
struct TableRows {
  const int16_t *ids;
  const float *w;
  const float *mean;
  __device__ __forceinline__ int id(int cur, int lr) const { return ids[cur * SP + lr]; }
  __device__ __forceinline__ float weight(int cur, int lr) const { return w[cur * SP + lr]; }
  __device__ __forceinline__ float row_mean(int cur) const { return mean[cur]; }
};

constexpr int kClusterRows = 1024;  // rows in each CTA's slice

template <int SP>
struct ClusterRows {
  uint32_t ids, w, mean;  // shared::cta addresses of the slice arrays
  __device__ __forceinline__ static uint32_t owner_addr(uint32_t local, int cur) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(cur >> 10));
    return r;
  }
  __device__ __forceinline__ int id(int cur, int lr) const {
    short v;
    asm("ld.shared::cluster.s16 %0, [%1];"
        : "=h"(v)
        : "r"(owner_addr(ids + (uint32_t)((cur & (kClusterRows - 1)) * SP + lr) * 2u, cur)));
    return v;
  }
  __device__ __forceinline__ float weight(int cur, int lr) const {
    float v;
    asm("ld.shared::cluster.f32 %0, [%1];"
        : "=f"(v)
        : "r"(owner_addr(w + (uint32_t)((cur & (kClusterRows - 1)) * SP + lr) * 4u, cur)));
    return v;
  }
  __device__ __forceinline__ float row_mean(int cur) const {
    float v;
    asm("ld.shared::cluster.f32 %0, [%1];"
        : "=f"(v)
        : "r"(owner_addr(mean + (uint32_t)(cur & (kClusterRows - 1)) * 4u, cur)));
    return v;
  }
};

constexpr int kNoPick = -(1 << 30);

// The reference's own walk over one row (staged_steps, below): the id of the
// first candidate past the threshold, or kNoPick.  A called function: within the
// loop it kept the row's weights alive over the fallback (n = m = 1000 with aging,
// clustered, k = 20: 305 us an iteration, 292 so).
template <int SP>
__device__ __noinline__ int exact_pick(float w, int id, float u, int lane) {
  float ra = 0.0f, rs = 0.0f;
#pragma unroll 4
  for (int e = 0; e < SP; e++) {
    const float we = __shfl_sync(kFull, w, e);
    ra = __fmaf_rn(we, e <= lane ? 1.0f : 0.0f, ra);
    rs = __fadd_rn(rs, we);
  }
  const float rnd = __fmul_rn(u, rs);
  const unsigned hit = __ballot_sync(kFull, ra > rnd || rnd != rnd);
  return hit ? __shfl_sync(kFull, id, __ffs(hit) - 1) : kNoPick;
}

// The step loop of one ant; BLEND (the aging fitness blend, fixed for the
// ant's whole tour) is a template parameter so the loop carries no per-step
// test of it.  Rows are padded to the pitch with id -1 and weight 0, so every
// lane inside it loads unconditionally.
//
// The reference adds the row's weights in order, visited ones as 0, into S and
// picks the first candidate whose running sum exceeds fl(u * S)
// (src/Colony.cu:801-846).  Sequential float sums of at most 32 non-negative
// terms lie within 31 * 2^-24 (relative) of the true sums, so sums formed in
// any other order settle the pick unless the threshold is that close to a
// running sum.  One step, with no data-dependent branch on the common path:
//  * lane r holds candidate r: its id and its weight, zeroed when the city is
//    visited;
//  * a scan within groups of eight lanes (three shuffles), then the groups'
//    totals in every lane (independent shuffles): the prefix at each lane and
//    S', within 6 * 2^-24 of the true sums.  Seven independent shuffles in
//    the place of the three were slower (their selects: 321 us an iteration's
//    construction at n = m = 1000 against 268), as were the weights through
//    shared memory and packed FMA chains a lane (310);
//  * hi, lo = u S' (1 +- E) +- 2^-147, E = 1.02 * 94 * 2^-24 covering both
//    errors of both sums and the roundings of the bounds (the 2^-147 where
//    they are not relative any more: products below 2^-126).  If the first prefix past lo is also
//    past hi, the reference's sums pass its threshold at that candidate: a
//    warp minimum of (lane, city) keys finds it and hands over the city;
//  * otherwise -- a prefix in the window (about 1e-4 of the steps), a sum that
//    is or may become infinite or NaN, no candidate left -- the reference's
//    own sums decide: its prefix
//    at lane l as acc = fma(w_e, incl_e, acc) in order (w*1 + acc rounds like
//    its float add, w*0 + acc = acc), the pick a ballot + ffs.  An infinite
//    weight (two cities at distance 0) turns a masked product into a NaN in
//    the lanes before it, where the reference has a finite prefix, so the
//    test is written acc > rnd || rnd is NaN: the same as !(s <= rnd) for
//    every prefix the reference forms, false for the masks' NaNs.  With S =
//    +inf this gives the reference's walk: past the row into the fallback for
//    rnd = +inf, candidate 0 for rnd = NaN.  No crossing (S = 0, or u*S
//    rounding up to S) takes the fallback, as the reference does.
// The next row is loaded before the rare cases resolve.  The uniforms of 32
// consecutive steps are computed one per lane and broadcast; the tour
// positions of the current 32-step block stay in one register per lane and
// are stored together.
template <int TW, bool BLEND, int G, class ROWS, bool TIER, int AHEAD>
__device__ __forceinline__ void staged_steps(const ColonyDev &c, int k, uint32_t akey, int start,
                                             StepTabu<TW> &tabu, const ROWS &rows, AntCtx a,
                                             int lane, int64_t &fallbacks) {
  constexpr int SP = 4 * G;           // row pitch of the staged table
  constexpr int NG = (SP + 7) / 8;    // groups of eight lanes that hold candidates
  constexpr float E = 94 * 6.08e-8f;  // 1.02 * 94 * 2^-24
  const int n = c.n;
  int32_t *trow = c.tours + (size_t)k * c.ld;
  // Lanes past the pitch hold no candidate: they read the last entry and
  // carry weight 0, so they are never the first past the threshold.
  const bool in_row = lane < SP;
  const int lr = in_row ? lane : SP - 1;
  const bool g1 = lane >= 8, g2 = lane >= 16, g3 = lane >= 24;
  const unsigned lane_key = (unsigned)lane << 16;
  int cur = start;
  int id = rows.id(cur, lr);
  float wraw = BLEND ? 0.0f : rows.weight(cur, lr);
  bool ok = true;
  for (int xb = 0; xb < n && ok; xb += 32) {
    const float ublk = aco_uniform_key(akey, (uint32_t)(xb + lane));
    int tpos = (xb == 0 && lane == 0) ? start : 0;  // tour position xb + lane
    const int xe = min(n, xb + 32);
#pragma unroll 1
    for (int x = xb == 0 ? 1 : xb; x < xe; x++) {
      const float u = __shfl_sync(kFull, ublk, x & 31);
      const float uhi = u * (1.0f + E), ulo = u * (1.0f - E);
      float w = wraw;
      if (BLEND) {
        a.meanc = rows.row_mean(cur);  // every lane: the fallback scan uses it too
        const size_t off = (size_t)cur * c.ldk + lane;
        w = lane < c.K ? blend_fitness(c.tau_nn[off], __ldg(c.eta_nn + off), a.meanc, a.ratio,
                                       c.use_alpha, c.alpha)
                       : 0.0f;
      }
      // Padding entries (id -1) carry weight 0, so their tabu lookup result
      // is irrelevant; every lane must take part in it.
      const bool vis = tabu.visited(id);
      if (vis || !in_row) w = 0.0f;
      float p = scan_level<8>(w, 1);
      p = scan_level<8>(p, 2);
      p = scan_level<8>(p, 4);
      const float T0 = __shfl_sync(kFull, p, 7), T1 = __shfl_sync(kFull, p, 15);
      float T2 = 0.0f, T3 = 0.0f;
      if (NG > 2) T2 = __shfl_sync(kFull, p, 23);
      if (NG > 3) T3 = __shfl_sync(kFull, p, 31);
      float S = T0 + T1;
      if (NG > 3) S += T2 + T3;
      else if (NG > 2) S += T2;
      if (g1) p += T0;
      if (g2) p += T1;
      if (NG > 3 && g3) p += T2;
      const float hi = __fmaf_rn(uhi, S, 0x1p-147f), lo = __fmaf_rn(ulo, S, -0x1p-147f);
      // The first lane past lo; its city, or 0xffff (as when there is no such
      // lane) if it is inside the window.
      const unsigned city = p > hi ? (unsigned)(id & 0xffff) : 0xffffu;
      const unsigned key = p > lo ? lane_key | city : ~0u;
      int next = (int)(__reduce_min_sync(kFull, key) & 0xffffu);
      // The next row, loaded before the rare cases resolve (an in-range
      // stand-in keeps the loads inside the table) and reloaded after them.
      const int nx = min(next, n - 1);
      int id_next = rows.id(nx, lr);
      float w_next = BLEND ? 0.0f : rows.weight(nx, lr);
      if (next >= n || !(S <= 3e38f)) {
        // With an infinite weight the threshold is infinite too (u > 0) and no
        // prefix is past it.
        const float inf = __int_as_float(0x7f800000);
        next = S != 0.0f && !(S == inf && __any_sync(kFull, w == inf))
                   ? exact_pick<SP>(w, id, u, lane)
                   : kNoPick;
        if (next != kNoPick) {
          if ((unsigned)next >= (unsigned)n) ok = false;  // recorded, not used
        } else {
          fallbacks++;
          if (c.fallback == ACO_FALLBACK_BEST) {
            if (!BLEND && a.blend) a.meanc = rows.row_mean(cur);  // pre-blended table
            TwPack<TW> pk;
            tabu.words_of(pk.w, lane);
            next = fallback_best<TW, AHEAD>(c, cur, pk, a, lane, id, vis, TIER && !BLEND && !a.blend);
          } else {  // select_local_best on a full row of at most 32 cities (k == n)
            const unsigned um = __ballot_sync(kFull, lane < c.K && id >= 0 && !vis);
            next = um ? __shfl_sync(kFull, id, 31 - __clz(um)) : -1;
          }
          if (next < 0 || next >= n) ok = false;  // no unvisited city, or a bad id
        }
        if (!ok) {
          if (lane == 0) atomicOr(&c.st->error, kErrCheck);
          break;
        }
        id_next = rows.id(next, lr);
        w_next = BLEND ? 0.0f : rows.weight(next, lr);
      }
      tabu.mark(next, lane);
      tpos = lane == (x & 31) ? next : tpos;
      cur = next;
      id = id_next;
      wraw = w_next;
    }
    if (xb + lane < xe) trow[xb + lane] = tpos;
  }
}

// The tour of one valid ant once its blend context is known: placement,
// the step loop (BLEND: the aging fitness blend of every candidate per step;
// otherwise the weights come blended, or plain, from the table), then the
// integer length and the transposed successor/predecessor lists.
template <int TW, int G, bool BLEND, class ROWS, bool TIER = true, int AHEAD = 1>
__device__ void staged_ant_body(const ColonyDev &c, int k, uint32_t iter, uint32_t *words,
                                const ROWS &rows, AntCtx a, int lane) {
  const int n = c.n;
  int32_t *trow = c.tours + (size_t)k * c.ld;
  StepTabu<TW> tabu;
  tabu.words = words;
  tabu.clear(lane);

  // initTour placement (src/Colony.cu:518-520)
  const uint32_t akey = aco_ant_key(c.seed, iter, (uint32_t)k);
  int start = __float2int_rz(__fmul_rn(aco_uniform_key(akey, 0u), __int2float_rn(n)));
  if (start >= n) {  // impossible for u < 1; recorded, clamped
    if (lane == 0) atomicOr(&c.st->error, kErrCheck);
    start = n - 1;
  }
  tabu.mark(start, lane);

  int64_t fallbacks = 0;
  staged_steps<TW, BLEND, G, ROWS, TIER, AHEAD>(c, k, akey, start, tabu, rows, a, lane, fallbacks);
  __syncwarp();
  // Tour length (order-free integer sum) and the transposed successor /
  // predecessor of every city for the row-owned deposit, one edge per lane;
  // unrolled so a lane's distance reads (scattered, from HBM when the L2 is
  // cold) are in flight together.
  // (Both words, though the second would do: the compiler's step loop above is
  // then 4 % faster, n = m = 1000, k = 32 281 us an iteration against 272.)
  const bool all_deposit = !(c.variant == ACO_RANK_BASED && c.epilogue_lists);
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
      atomicOr(&c.st->error, kErrCheck);
    }
  }
  for (int o = 16; o; o >>= 1) len += __shfl_xor_sync(kFull, len, o);
  if (lane == 0) {
    c.newlen[k] = len;
    if (fallbacks)
      atomicAdd(reinterpret_cast<unsigned long long *>(&c.st->fallbacks),
                (unsigned long long)fallbacks);
  }
}

// One ant with its aging step: updateAntAges (src/Colony.cu:353-364), the
// cleared tour of an invalid ant (src/Colony.cu:507-510) and the blend
// decision of compute_fittness (inc/Colony.cuh:21-30).
template <bool AGING, int TW, int G, class ROWS, bool TIER = true, int AHEAD = 1>
__device__ void construct_ant_staged(const ColonyDev &c, int k, uint32_t iter, uint32_t *words,
                                     const ROWS &rows, int lane) {
  AntCtx a;
  a.blend = false;
  a.ratio = 0.0f;
  a.meanc = 0.0f;
  if (AGING) {
    int age = 0;
    if (lane == 0) {
      age = c.age[k] + 1;
      c.age[k] = age;
    }
    age = __shfl_sync(kFull, age, 0);
    if (!c.valid[k]) {
      int32_t *trow = c.tours + (size_t)k * c.ld;
      for (int i = lane; i < c.n; i += 32) trow[i] = 0;
      return;
    }
    a.blend = age < c.min_ret && c.st->isconverged;
    if (a.blend) a.ratio = __fdiv_rn(__int2float_rn(age), __int2float_rn(c.min_ret));
  }
  if (AGING && a.blend)
    staged_ant_body<TW, G, true, ROWS, TIER, AHEAD>(c, k, iter, words, rows, a, lane);
  else
    staged_ant_body<TW, G, false, ROWS, TIER, AHEAD>(c, k, iter, words, rows, a, lane);
}

}  // namespace aco
