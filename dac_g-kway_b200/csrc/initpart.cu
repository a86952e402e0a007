// Device initial partition of the coarsest graph: recursive bisection by
// greedy graph growing (GGGP, Karypis & Kumar's multilevel partitioning
// scheme), replacing the reference's host METIS call
// (gkway/metis_partition.hpp:46-47).
//
// Each recursion depth is one launch (three when some sub-problem may be too
// large for one CTA's shared memory).  A sub-problem is the set of vertices
// whose part range is [p0, p1); it is bisected into [p0, pm) and [pm, p1),
// pm = p0 + (p1 - p0) / 2, with the left side's target weight
// TL = W(S) * (pm - p0) / (p1 - p0).  Its members are indexed in id order, and
// up to eight trials bisect it, each from its own seed vertex:
//   growth      repeatedly add the unassigned vertex with the best key
//               (frontier first, then cut gain 2*conn - deg_S, then the
//               smaller member index) while the region weight is below TL;
//               a vertex that would overshoot TL by more than the region is
//               short of it is not added and growth stops;
//   refinement  move the vertex with the largest positive cut gain to the
//               other side while the receiving side stays within
//               target * (1 + eps/2); at most s/4 + 32 moves.
// The trial with the smallest cut (then smallest |W(R) - TL|, then lowest
// trial index) wins.  Seeds: trial t of sub-problem p0 starts at member
// index mix(seed, p0, t) mod s.  Deterministic for a given seed.
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <climits>
#include <cstring>
#include <type_traits>
#include <vector>

#include "gkw_internal.cuh"

namespace gkw {

static constexpr u32 kFull32 = 0xffffffffu;
constexpr int kInitTrials = 8;

__device__ __forceinline__ u32 mix32(u64 x) {
  x ^= x >> 33;
  x *= 0xff51afd7ed558ccdull;
  x ^= x >> 33;
  x *= 0xc4ceb9fe1a85ec53ull;
  x ^= x >> 33;
  return (u32)x;
}

// Warp maximum of a 64-bit key in two 32-bit reductions (redux.sync): the
// largest high half, then the largest low half among the lanes holding it --
// two dependent steps instead of five shuffle rounds on a growth step's chain.
__device__ __forceinline__ u64 warp_max_u64(u64 x) {
  const u32 hi = (u32)(x >> 32), lo = (u32)x;
  const u32 mh = __reduce_max_sync(kFull32, hi);
  const u32 ml = __reduce_max_sync(kFull32, hi == mh ? lo : 0u);
  return ((u64)mh << 32) | ml;
}

__device__ __forceinline__ i64 warp_sum_i64(i64 x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(kFull32, x, o);
  return x;
}

// growth key: frontier bit, gain (order-preserving bias), smaller index wins
__device__ __forceinline__ u64 grow_key(bool frontier, i32 g, i32 idx) {
  return (1ull << 63) | ((u64)(frontier ? 1 : 0) << 62) | ((u64)((u32)g ^ 0x80000000u) << 30) |
         (u64)(0x3fffffffu - (u32)idx);
}

// refinement key: gain, smaller index wins; top bit marks a valid entry
__device__ __forceinline__ u64 move_key2(i32 g, i32 idx) {
  return (1ull << 63) | ((u64)((u32)g ^ 0x80000000u) << 30) | (u64)(0x3fffffffu - (u32)idx);
}

__device__ __forceinline__ i32 key_idx(u64 key) { return (i32)(0x3fffffffu - (u32)(key & 0x3fffffffu)); }

typedef uint8_t u8;
typedef uint16_t u16;

// One bisection: the sides' parts [p0, pm) and [pm, p1), the left target and
// the weight limits of the refinement.
struct SplitParams {
  i64 WS, TL, capL, capR;
  i32 p0, pm, p1;
};

// Everything the kernels of one call share.  Members of all sub-problems lie
// in M as one permutation of the vertices, sub-problem p0 at
// [off[p0], off[p0] + cnt[p0]) in id order; pos[v] is v's place in it.
struct GggpArgs {
  i32 n, k, trials;
  const i32* __restrict__ xadj;
  const i32* __restrict__ adjncy;
  const i32* __restrict__ adjwgt;
  const i32* __restrict__ vwgt;
  const i32* mcur;    // M at this depth
  i32* mnext;         // M of the next depth
  i32* pos;
  i32* part;          // first part of each vertex's sub-problem (the result at the end)
  i32* cnt;
  i32* off;
  const int2* subs;   // batched: the depth's sub-problems (p0, p1); null: found from the block index
  i32 depth;
  u64 seed;
  double eps;
  const i32* part_base;   // batched: first part of each part's graph
  // large sub-problems: list, per-part marks and the filtered rows
  i32* bigcount;      // per depth
  int2* biglist;
  i32* bigmark;       // [k] depth + 1 when listed at this depth
  u64* bighash;       // [k] signed edge hash: 0 for symmetric rows
  i32* bigwide;       // [k] nonzero: weights need the wide path
  i32* bigdone;       // [maxbig] trials finished
  int4* g_hdr;        // [n] by place: row start, row length, vertex weight, weight to other members
  int2* g_edge;       // [m] rows at the members' own CSR positions: (member index, weight)
  u8* g_R;            // [trials * n] sides of every trial
  i64* tcut;
  i64* tdev;
  u32* g_V;           // [trials * v_stride] growth state that does not fit in shared memory
  size_t v_stride;
  // wide path (see WideState)
  i32* w_state;
  u64* w_keys;
  u64* w_b1;
  u64* w_b2;
  size_t b1_stride, b2_stride;
  size_t smem;        // dynamic shared memory of the launch
  unsigned long long* prof;   // slowest trial's growth and refinement cycles (diagnostic)
};

__host__ __device__ __forceinline__ i32 gggp_nb1(i32 s) { return (s + 31) >> 5; }
__host__ __device__ __forceinline__ i32 gggp_nb2(i32 s) { return (s + 1023) >> 10; }

// Refinement moves of one trial: s/4 + 32, at most 256 (each move scans the
// whole sub-problem).
__host__ __device__ __forceinline__ i32 gggp_max_moves(i32 s) { return s / 4 + 32 < 256 ? s / 4 + 32 : 256; }

__device__ __forceinline__ i64 block_sum_i64(i64 x, i64* s_red) {
  x = warp_sum_i64(x);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) s_red[threadIdx.x >> 5] = x;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  return warp_sum_i64(lane < (int)(blockDim.x >> 5) ? s_red[lane] : 0);
}

// Two sums behind one pair of barriers (s_red: two words a warp).
__device__ __forceinline__ void block_sum2_i64(i64& x, i64& y, i64* s_red) {
  x = warp_sum_i64(x);
  y = warp_sum_i64(y);
  const int lane = threadIdx.x & 31, nw = (int)(blockDim.x >> 5);
  __syncthreads();
  if (lane == 0) {
    s_red[threadIdx.x >> 5] = x;
    s_red[nw + (threadIdx.x >> 5)] = y;
  }
  __syncthreads();
  x = warp_sum_i64(lane < nw ? s_red[lane] : 0);
  y = warp_sum_i64(lane < nw ? s_red[nw + lane] : 0);
}

// ---------------------------------------------------------------------------
// Wide path: 64-bit growth keys, connection weights and sides in separate
// arrays of global memory.  It serves the sub-problems whose weights do not
// fit the packed state below (a member's weight to the others of 2^28 or
// more, a coarse weight that wrapped negative) or whose rows are not
// symmetric; 32-bit wrap-around there is the oracle's.
// Growth keys of one trial: K[i] = grow_key of unassigned member i (0 once
// assigned), B1[b] = max of K over members [32b, 32b + 32), B2[c] = max of B1
// over blocks [32c, 32c + 32).  A key only rises while its member is
// unassigned (conn only grows), so updates are atomic maxima; assigning a
// member recomputes its two blocks.
// ---------------------------------------------------------------------------
struct WideTopo {
  const int4* hdr;    // row start, row length, vertex weight, weight to other members
  const int2* edge;   // (member index, weight)
};
struct WideState {
  i32* C;      // connection weight to the region R
  i32* R;      // in R
  u64* K;
  u64* B1;
  u64* B2;
};

// Growth over the block maxima of the growth keys (WideState).  Returns W(R).
__device__ __noinline__ i64 grow_wide(const WideTopo& T, const WideState& S, i32 s, i32 pick, i64 TL) {
  const int lane = threadIdx.x & 31;
  i32* C = S.C;
  i32* R = S.R;
  u64* K = S.K;
  u64* B1 = S.B1;
  u64* B2 = S.B2;
  const i32 nb1 = gggp_nb1(s), nb2 = gggp_nb2(s);
  for (i32 i = lane; i < s; i += 32) K[i] = grow_key(false, -T.hdr[i].w, i);
  __syncwarp();
  for (i32 b = lane; b < nb1; b += 32) {
    u64 m = 0;
    for (i32 i = b << 5; i < s && i < (b + 1) << 5; ++i) m = m > K[i] ? m : K[i];
    B1[b] = m;
  }
  __syncwarp();
  for (i32 c = lane; c < nb2; c += 32) {
    u64 m = 0;
    for (i32 b = c << 5; b < nb1 && b < (c + 1) << 5; ++b) m = m > B1[b] ? m : B1[b];
    B2[c] = m;
  }
  __syncwarp();
  i64 wR = 0;
  for (i32 step = 0; step < s; ++step) {
    if (step > 0) {
      u64 best = 0;
      for (i32 c = lane; c < nb2; c += 32) {
        const u64 x = __ldcg(reinterpret_cast<const unsigned long long*>(&B2[c]));
        best = best > x ? best : x;
      }
      best = warp_max_u64(best);
      if (best == 0) break;
      pick = key_idx(best);
    }
    // the picked member's weight and row, loaded together
    const int4 hd = T.hdr[pick];
    const i64 vw = (u32)hd.z;
    const i32 rb = hd.x, rn = hd.y;
    if (step > 0 && wR + vw > TL && (wR + vw - TL) > (TL - wR)) break;
    if (lane == 0) {
      R[pick] = 1;
      K[pick] = 0;
    }
    wR += vw;
    __syncwarp();
    // neighbours, four per lane per pass: the row loads, then the state loads
    // and connection updates of all four are issued together.  R[u] and
    // degS[u] do not change in this step (u != pick).
    constexpr i32 kU = 4;
    for (i32 j0 = lane; j0 < rn; j0 += 32 * kU) {
      i32 u[kU], w[kU], ru[kU], du[kU], c[kU];
#pragma unroll
      for (i32 q = 0; q < kU; ++q) {
        const i32 j = j0 + 32 * q;
        const int2 ed = j < rn ? T.edge[rb + j] : make_int2(-1, 0);
        u[q] = ed.x;
        w[q] = ed.y;
      }
#pragma unroll
      for (i32 q = 0; q < kU; ++q) {
        if (u[q] >= 0) {
          ru[q] = __ldcg(&R[u[q]]);
          du[q] = T.hdr[u[q]].w;
          c[q] = atomicAdd(&C[u[q]], w[q]) + w[q];
        }
      }
#pragma unroll
      for (i32 q = 0; q < kU; ++q) {
        if (u[q] >= 0 && !ru[q]) {
          const unsigned long long key = grow_key(c[q] > 0, 2 * c[q] - du[q], u[q]);
          atomicMax(reinterpret_cast<unsigned long long*>(&K[u[q]]), key);
          atomicMax(reinterpret_cast<unsigned long long*>(&B1[u[q] >> 5]), key);
          atomicMax(reinterpret_cast<unsigned long long*>(&B2[u[q] >> 10]), key);
        }
      }
    }
    __syncwarp();
    // the picked member leaves its blocks
    {
      const i32 b = pick >> 5, i = (b << 5) + lane;
      const u64 m = warp_max_u64(i < s ? __ldcg(reinterpret_cast<const unsigned long long*>(&K[i])) : 0ull);
      if (lane == 0) B1[b] = m;
      __syncwarp();
      const i32 c = pick >> 10, bb = (c << 5) + lane;
      const u64 m2 = warp_max_u64(bb < nb1 ? __ldcg(reinterpret_cast<const unsigned long long*>(&B1[bb])) : 0ull);
      if (lane == 0) B2[c] = m2;
      __syncwarp();
    }
    if (wR >= TL) break;
  }
  return wR;
}

// One trial by one warp (growth then positive-gain refinement); see the file
// comment for the rules.  Returns the trial's cut and |W(R) - TL|.
__device__ __noinline__ void trial_wide(const WideTopo& T, const WideState& S, i32 s, i32 pick, const SplitParams& P,
                                        i64& cut_out, i64& dev_out) {
  const int lane = threadIdx.x & 31;
  i32* C = S.C;
  i32* R = S.R;
  for (i32 i = lane; i < s; i += 32) {
    R[i] = 0;
    C[i] = 0;
  }
  __syncwarp();
  i64 wR = grow_wide(T, S, s, pick, P.TL);
  // ---- refinement: positive-gain moves within the side caps ----
  const i32 max_moves = gggp_max_moves(s);
  for (i32 mv = 0; mv < max_moves; ++mv) {
    u64 best = 0;
    // four members per lane per pass, their loads issued together
    constexpr i32 kU = 4;
    for (i32 i0 = lane; i0 < s; i0 += 32 * kU) {
      i32 r[kU], c[kU], d[kU], w[kU];
#pragma unroll
      for (i32 u = 0; u < kU; ++u) {
        const i32 i = i0 + 32 * u;
        const bool in = i < s;
        r[u] = in ? __ldcg(&R[i]) : 0;
        c[u] = in ? __ldcg(&C[i]) : 0;
        const int4 hd = in ? T.hdr[i] : make_int4(0, 0, 0, 0);
        d[u] = hd.w;
        w[u] = hd.z;
      }
#pragma unroll
      for (i32 u = 0; u < kU; ++u) {
        const i32 g = r[u] ? (d[u] - 2 * c[u]) : (2 * c[u] - d[u]);
        const i64 vw = (u32)w[u];
        const bool ok = r[u] ? ((P.WS - wR) + vw <= P.capR) : (wR + vw <= P.capL);
        if (g > 0 && ok) {   // out-of-range lanes have g = 0
          const u64 key = move_key2(g, i0 + 32 * u);
          best = best > key ? best : key;
        }
      }
    }
    best = warp_max_u64(best);
    if (best == 0) break;
    const i32 i = key_idx(best);
    const i32 r = __ldcg(&R[i]);
    __syncwarp();
    if (lane == 0) R[i] = r ^ 1;
    const int4 hd = T.hdr[i];
    wR += r ? -(i64)(u32)hd.z : (i64)(u32)hd.z;
    const i32 sign = r ? -1 : 1;
    for (i32 j = lane; j < hd.y; j += 32) {
      const int2 ed = T.edge[hd.x + j];
      atomicAdd(&C[ed.x], sign * ed.y);
    }
    __syncwarp();
  }
  i64 cut = 0;
  for (i32 i = lane; i < s; i += 32)
    if (__ldcg(&R[i])) cut += T.hdr[i].w - __ldcg(&C[i]);
  cut = warp_sum_i64(cut);
  cut_out = cut;
  dev_out = wR > P.TL ? wR - P.TL : P.TL - wR;
}

// The wide state of trial t of the sub-problem p0 at place o: [C | R] of n
// each per trial; key blocks at o / 32 + p0 and o / 1024 + p0 (disjoint
// across the sub-problems, which lie in part order).
__device__ __forceinline__ WideState wide_state(const GggpArgs& a, i32 t, i32 p0, i32 o) {
  WideState S;
  i32* q = a.w_state + (size_t)t * 2 * a.n;
  S.C = q + o;
  S.R = q + a.n + o;
  S.K = a.w_keys + (size_t)t * a.n + o;
  S.B1 = a.w_b1 + (size_t)t * a.b1_stride + (o >> 5) + p0;
  S.B2 = a.w_b2 + (size_t)t * a.b2_stride + (o >> 10) + p0;
  return S;
}

// ---------------------------------------------------------------------------
// Packed path.  A trial's whole state is one 32-bit word per member:
//   bit 31  not in the region     bit 30  on the frontier
//   then    gain + bias, gain = 2 * conn - deg
//   then    mask - slot, in the low ib bits
// Adding an edge of weight w to the region adds 2w << ib to the word on either
// side, so the word carries the growth key, the region flag and the refinement
// gain at once.  ib is the slots' width when the gains fit the bits left
// (|gain| < bias = 2^(29 - ib)): a maximum then names its member.  Otherwise
// ib = 0 (gains below 2^28) and the member is found by a ballot over its
// block, ties going to the first lane, that is the smaller index.  B1 holds
// the maximum of every 32 words and, above 4096 members, B2 the maximum of
// every 32 of B1; all maxima are native 32-bit shared-memory operations.
//
// Bound: the serial chain of a step -- block maximum, the member's header,
// its row, the words of its neighbours.  Members without edges to the others
// ("inert") never change a key and are all added when the frontier is empty,
// before any other member (their gain 0 exceeds every negative one), in index
// order: one weight scan takes their whole run instead of one step each.  A
// circuit graph's coarsest level has 29,174 of them among 33,910 vertices:
// with the run, the rows below and the packed words its initial partition at
// k = 256 takes 16 ms instead of 230.
// ---------------------------------------------------------------------------
constexpr u32 kOut = 0x80000000u;
constexpr u32 kFront = 0x40000000u;
constexpr u32 kGainBits = 0x3fffffffu;
constexpr i64 kPackedDeg = (i64)1 << 28;   // weights to other members below this

struct Packing {
  i32 ib;
  u32 mask, bias;
  __device__ __forceinline__ u32 initial(i32 deg, i32 slot) const {
    return kOut | ((bias - (u32)deg) << ib) | (mask - ((u32)slot & mask));
  }
  __device__ __forceinline__ i32 gain(u32 x) const { return (i32)((x & kGainBits) >> ib) - (i32)bias; }
  __device__ __forceinline__ i32 slot(u32 x) const { return (i32)(mask - (x & mask)); }
};
__device__ __forceinline__ Packing packing_for(i32 slots, i32 maxdeg) {
  Packing k;
  k.ib = slots > 1 ? 32 - __clz(slots - 1) : 1;
  if (k.ib > 28 || maxdeg >= (1 << (29 - k.ib))) k.ib = 0;
  k.mask = (1u << k.ib) - 1u;
  k.bias = 1u << (29 - k.ib);
  return k;
}
__device__ __forceinline__ bool in_region(u32 x) { return (x & kOut) == 0; }
__device__ __forceinline__ u32 word_enter(u32 x) { return x & kGainBits; }
__device__ __forceinline__ u32 word_leave(u32 x) { return x | kOut; }
// gain of moving the member to the other side
__device__ __forceinline__ i32 move_gain(const Packing& K, u32 x) { return in_region(x) ? -K.gain(x) : K.gain(x); }

// words of the state's arrays for s members: V padded to 32, B1 to the
// layout of its level (one word per lane up to 1024 members, four up to
// 4096, else rows of 32 under B2), B2 to 64
__host__ __device__ __forceinline__ i32 pad_to(i32 x, i32 a) { return (x + a - 1) / a * a; }
__host__ __device__ __forceinline__ i32 packed_b1_words(i32 s) {
  return s <= 1024 ? 32 : s <= 4096 ? 128 : pad_to(gggp_nb1(s), 32);
}
__host__ __device__ __forceinline__ i32 packed_b2_words(i32 s) { return s <= 4096 ? 0 : pad_to(gggp_nb2(s), 64); }
__host__ __device__ __forceinline__ i32 packed_state_words(i32 s) {
  return pad_to(s, 32) + packed_b1_words(s) + packed_b2_words(s);
}

template <bool kGlobal>
__device__ __forceinline__ u32 ldw(const u32* p) { return kGlobal ? __ldcg(p) : *p; }

// Predicated atomics (a branch around each would cost more of a step's chain
// than the operation): shared-memory words by their 32-bit address, or global.
template <bool kGlobal>
__device__ __forceinline__ u32 add_if(bool on, u32* p, u32 v) {
  u32 old;
  if (kGlobal)
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %3, 0;\n\tmov.u32 %0, 0;\n\t@q atom.global.add.u32 %0, [%1], %2;\n\t}"
                 : "=r"(old) : "l"(p), "r"(v), "r"((u32)on) : "memory");
  else
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %3, 0;\n\tmov.u32 %0, 0;\n\t@q atom.shared.add.u32 %0, [%1], %2;\n\t}"
                 : "=r"(old) : "r"((u32)__cvta_generic_to_shared(p)), "r"(v), "r"((u32)on) : "memory");
  return old;
}
template <bool kGlobal>
__device__ __forceinline__ void max_if(bool on, u32* p, u32 v) {
  if (kGlobal)
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\t@q red.global.max.u32 [%0], %1;\n\t}"
                 :: "l"(p), "r"(v), "r"((u32)on) : "memory");
  else
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\t@q red.shared.max.u32 [%0], %1;\n\t}"
                 :: "r"((u32)__cvta_generic_to_shared(p)), "r"(v), "r"((u32)on) : "memory");
}

// One neighbour (member index, weight; weight 0: none) of the member that just
// entered the region; returns its word (0 if it is in the region).  A row may
// list it twice: the add and the maxima commute.  (Reading B1 first, to skip
// the maxima that change nothing, made the growth over rows of about 1100
// entries 15% slower.)
template <int LV, bool kGlobal>
__device__ __forceinline__ u32 touch_neighbour(u32* V, u32* B1, u32* B2, int2 ed, i32 ib) {
  const bool on = ed.y != 0;
  const u32 add = (2u * (u32)ed.y) << ib;
  const u32 nv = (add_if<kGlobal>(on, V + ed.x, add) + add) | kFront;
  const bool out = on && (nv & kOut);
  max_if<kGlobal>(out, V + ed.x, nv);
  max_if<kGlobal>(out, B1 + (ed.x >> 5), nv);
  if (LV == 2) max_if<kGlobal>(out, B2 + (ed.x >> 10), nv);
  return out ? nv : 0u;
}

// The growth of one trial by one warp (lane-converged).  `pick` is the seed's
// slot, or -1 when the seed is inert (its weight is then seed_w).  hdr(i) is
// the header of slot i; fetch(row start, row length) this lane's entry of the
// row's first 32; expand(row start, row length, entry, best) touches the row's
// neighbours (warp-converged) and raises `best` to this lane's largest touched
// word, or returns true when other warps touched some; inert_w(i) the weight
// of member i if it is inert and not the seed, else -1, for the members in
// index order.  *inert_end: members below it that are inert are in the
// region.  Returns W(R).
//
// The next member is the maximum over the blocks' maxima before the last
// step's touches (`top`, loaded and corrected for the member that left while
// the row was fetched) and the touched words in registers (`best`), so the
// chain of a step is one warp maximum, the header, the row and the atomic add
// -- not the maxima's way through shared memory as well.  A million-vertex
// mesh at k = 64 (413 members, 206 steps at depth 0) takes 680 cycles a step
// against 1450 for a scan of the frontier with 64-bit keys; its whole initial
// partition 0.27 ms against 0.48.
template <int LV, bool kGlobal, class Hdr, class Fetch, class Expand, class InertW>
__device__ __forceinline__ i64 grow_packed(const Packing K, u32* V, u32* B1, u32* B2, i32 nb2p, i32 s,
                                           bool inert_left, i32 pick, i64 seed_w, i64 TL, i32* inert_end, Hdr hdr,
                                           Fetch fetch, Expand expand, InertW inert_w) {
  const int lane = threadIdx.x & 31;
  i64 wR = 0;
  *inert_end = 0;
  bool seeded = pick >= 0;
  if (!seeded) {
    wR = seed_w;
    if (wR >= TL) return wR;
  }
  // this lane's largest block maximum, with the one of block b (LV 2: block
  // of blocks) replaced by sub
  auto load_top = [&](i32 b, u32 sub) -> u32 {
    if (LV == 0) {
      const u32 x = ldw<kGlobal>(B1 + lane);
      return lane == b ? sub : x;
    }
    if (LV == 1) {
      uint4 q = *reinterpret_cast<const uint4*>(B1 + 4 * lane);
      if (4 * lane == b) q.x = sub;
      if (4 * lane + 1 == b) q.y = sub;
      if (4 * lane + 2 == b) q.z = sub;
      if (4 * lane + 3 == b) q.w = sub;
      const u32 x = q.x > q.y ? q.x : q.y, z = q.z > q.w ? q.z : q.w;
      return x > z ? x : z;
    }
    u32 x = 0;
    for (i32 q = 2 * lane; q < nb2p; q += 64) {
      u32 x0 = ldw<kGlobal>(B2 + q), x1 = ldw<kGlobal>(B2 + q + 1);
      if (q == b) x0 = sub;
      if (q + 1 == b) x1 = sub;
      x = x0 > x ? x0 : x;
      x = x1 > x ? x1 : x;
    }
    return x;
  };
  u32 top = load_top(-1, 0u), best = 0;
  for (;;) {
    u32 mh;
    if (!seeded) {
      mh = __reduce_max_sync(kFull32, top > best ? top : best);
      if (!(mh & kFront) && inert_left) {
        // empty frontier: the inert members next, in index order, up to the
        // first that reaches TL (taken unless it overshoots by more than the
        // region is short)
        inert_left = false;
        for (i32 z0 = 0; z0 < s; z0 += 32) {
          const i32 z = z0 + lane;
          const i64 w = z < s ? inert_w(z) : -1;
          i64 inc = w > 0 ? w : 0;
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const i64 t = __shfl_up_sync(kFull32, inc, o);
            if (lane >= o) inc += t;
          }
          const u32 cross = __ballot_sync(kFull32, w >= 0 && wR + inc >= TL);
          if (cross) {
            const int j = __ffs(cross) - 1;
            const i64 wj = __shfl_sync(kFull32, w, j);
            const i64 before = wR + __shfl_sync(kFull32, inc, j) - wj;
            const bool take = !(before + wj > TL && (before + wj - TL) > (TL - before));
            *inert_end = z0 + j + (take ? 1 : 0);
            return take ? before + wj : before;
          }
          wR += __shfl_sync(kFull32, inc, 31);
        }
        *inert_end = s;
        continue;
      }
      if (!(mh & kOut)) break;   // every member is in the region
      if (K.ib) {
        pick = K.slot(mh);
      } else {   // the first member with this word, by ballots over the (complete) maxima in memory
        i32 b = 0;
        if (LV == 0) {
          b = __ffs(__ballot_sync(kFull32, ldw<kGlobal>(B1 + lane) == mh)) - 1;
        } else if (LV == 1) {
          const uint4 q = *reinterpret_cast<const uint4*>(B1 + 4 * lane);
          const i32 lb = q.x == mh ? 0 : q.y == mh ? 1 : q.z == mh ? 2 : q.w == mh ? 3 : 128;
          b = (i32)__reduce_min_sync(kFull32, (u32)(4 * lane + lb));
        } else {
          u32 lb = 0xffffffffu;
          for (i32 q = 2 * lane; q < nb2p; q += 64) {
            const u32 x0 = ldw<kGlobal>(B2 + q), x1 = ldw<kGlobal>(B2 + q + 1);
            if (x1 == mh && lb == 0xffffffffu) lb = (u32)q + 1;
            if (x0 == mh && (lb == 0xffffffffu || lb == (u32)q + 1)) lb = (u32)q;
          }
          b = (i32)__reduce_min_sync(kFull32, lb);
          b = (b << 5) + __ffs(__ballot_sync(kFull32, ldw<kGlobal>(B1 + (b << 5) + lane) == mh)) - 1;
        }
        pick = (b << 5) + __ffs(__ballot_sync(kFull32, ldw<kGlobal>(V + (b << 5) + lane) == mh)) - 1;
      }
    } else {
      mh = ldw<kGlobal>(V + pick);
    }
    const int4 h = hdr(pick);
    const u32 y = ldw<kGlobal>(V + (pick & ~31) + lane);
    const u32 xrow = LV == 2 ? ldw<kGlobal>(B1 + ((pick >> 10) << 5) + lane) : 0u;
    const int2 ed = fetch(h.x, h.y);   // (issued before the weight test: the row is on the chain)
    const i64 w = (u32)h.z;
    if (!seeded && wR + w > TL && (wR + w - TL) > (TL - wR)) break;
    seeded = false;
    // the member leaves its blocks' maxima and enters the region
    const u32 nbm = __reduce_max_sync(kFull32, lane == (pick & 31) ? 0u : y);
    if (LV == 2) {
      const u32 m2 = __reduce_max_sync(kFull32, lane == ((pick >> 5) & 31) ? nbm : xrow);
      top = load_top(pick >> 10, m2);
      if (lane == 0) B2[pick >> 10] = m2;
    } else {
      top = load_top(pick >> 5, nbm);
    }
    if (lane == 0) {
      V[pick] = word_enter(mh);
      B1[pick >> 5] = nbm;
    }
    __syncwarp();
    wR += w;
    best = 0;
    const bool others = expand(h.x, h.y, ed, best);
    __syncwarp();
    if (wR >= TL) break;
    if (others) top = load_top(-1, 0u);
  }
  return wR;
}

// The sum of the counts of the warps before this one, and of all nw <= 32
// (whole warps; two warp reductions instead of a loop of dependent adds).
__device__ __forceinline__ i32 warps_before(const i32* s_count, int nw, i32& total) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const i32 x = lane < nw ? s_count[lane] : 0;
  total = __reduce_add_sync(kFull32, x);
  return __reduce_add_sync(kFull32, lane < wid ? x : 0);
}

// Stable bisection of one sub-problem by the whole CTA: the members with
// side(i) go to [p0, pm), the others to [pm, p1), both in id order.
template <class Side>
__device__ void split_members(const GggpArgs& a, const SplitParams& P, i32 s, i32 o, i32* s_scan, Side side) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  i32 nL = 0;
  for (i32 i0 = 0; i0 < s; i0 += blockDim.x) {   // block-uniform trip count
    const i32 i = i0 + threadIdx.x;
    nL += __syncthreads_count(i < s && side(i));
  }
  i32 doneL = 0;
  for (i32 i0 = 0; i0 < s; i0 += blockDim.x) {
    const i32 i = i0 + threadIdx.x;
    const bool in = i < s;
    const bool left = in && side(i);
    const u32 bal = __ballot_sync(kFull32, left);
    if (lane == 0) s_scan[wid] = __popc(bal);
    __syncthreads();
    i32 tot;
    const i32 before = warps_before(s_scan, nw, tot);
    if (in) {
      const i32 rankL = doneL + before + __popc(bal & ((1u << lane) - 1));
      const i32 at = left ? o + rankL : o + nL + (i - rankL);
      const i32 v = a.mcur[o + i];
      a.mnext[at] = v;
      a.pos[v] = at;
      a.part[v] = left ? P.p0 : P.pm;
    }
    doneL += tot;
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    a.cnt[P.p0] = nL;
    a.cnt[P.pm] = s - nL;
    a.off[P.pm] = o + nL;
  }
}

__device__ __forceinline__ SplitParams split_params(const GggpArgs& a, i32 p0, i32 p1, i64 WS) {
  SplitParams P;
  P.p0 = p0;
  P.p1 = p1;
  P.pm = p0 + (p1 - p0) / 2;
  P.WS = WS;
  P.TL = WS * (P.pm - p0) / (p1 - p0);
  P.capL = (i64)((double)P.TL * (1.0 + a.eps * 0.5));
  P.capR = (i64)((double)(WS - P.TL) * (1.0 + a.eps * 0.5));
  return P;
}

// seed member of trial t (batched: the part is named by its own graph's id)
__device__ __forceinline__ i32 seed_member(const GggpArgs& a, i32 p0, i32 t, i32 s) {
  const i32 p0_local = a.part_base ? p0 - a.part_base[p0] : p0;
  return (i32)(mix32(a.seed * 0x9e3779b97f4a7c15ull + (u64)p0_local * 1315423911ull + (u64)t) % (u32)s);
}

// Signed hash of a directed entry (i, j, w): entries (i, j, w) and (j, i, w)
// cancel, so the rows of a sub-problem are symmetric iff the sum is 0 (up to
// a 64-bit collision).
__device__ __forceinline__ u64 entry_hash(i32 i, i32 j, i32 w) {
  const u32 lo = i < j ? i : j, hi = i < j ? j : i;
  u64 x = ((u64)hi << 32 | lo) * 0x9e3779b97f4a7c15ull + (u32)w;
  x ^= x >> 29;
  x *= 0xbf58476d1ce4e5b9ull;
  x ^= x >> 32;
  return i < j ? x : 0ull - x;
}

// ---------------------------------------------------------------------------
// One CTA per sub-problem, one warp per trial, everything in shared memory:
//   hdr   int4[s]   by slot: row start, row length, vertex weight, weight to
//                   the other members; active members first, then the inert
//   edge  int2[L]   (slot, weight), rows at the scan of the full row lengths
//   perm  u16[s]    member -> slot
//   state           per trial: words V, B1 (packed path); first the rows'
//                   counts by member while the rows are built
// A sub-problem that does not fit goes to the large list.
// Growth is 700 cycles a pick; beside it a depth costs about 15k cycles of
// short passes with a barrier each.  Their sums over the warps' counts by two
// warp reductions took 2048 vertices, k = 8 (three depths) from 382 to 374 us
// in all, a million-vertex mesh's six from 239 to 229 us.
// ---------------------------------------------------------------------------
constexpr int kSmallThreads = 512;
constexpr i32 kSmallMax = 4096;            // members
constexpr size_t kGggpSmem = 220 * 1024;   // dynamic shared memory, one CTA per SM
constexpr size_t kGggpSmemHalf = 108 * 1024;   // two CTAs per SM

__host__ __device__ __forceinline__ size_t small_bytes(i64 s, i64 L, i32 trials) {
  const size_t state = (size_t)4 * packed_state_words((i32)s) * trials;
  const size_t temp = (size_t)16 * s;
  return (((size_t)16 * s + (size_t)8 * L + (size_t)2 * s + 15) & ~(size_t)15) + (state > temp ? state : temp);
}

__global__ void __launch_bounds__(kSmallThreads) k_gggp_small(GggpArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ i32 s_scan[kSmallThreads / 32];
  __shared__ i64 s_red[2 * (kSmallThreads / 32)];
  __shared__ i64 s_cut[kInitTrials], s_dev[kInitTrials];
  __shared__ i32 s_inert[kInitTrials];
  __shared__ i32 s_bad, s_carry, s_maxd;
  i32 p0, p1;
  if (a.subs) {
    const int2 q = a.subs[blockIdx.x];
    p0 = q.x;
    p1 = q.y;
  } else {   // the bits of the block index lead from [0, k) to the sub-problem
    p0 = 0;
    p1 = a.k;
    for (i32 b = a.depth - 1; b >= 0; --b) {
      if (p1 - p0 < 2) return;
      const i32 pm = p0 + (p1 - p0) / 2;
      if ((blockIdx.x >> b) & 1) p0 = pm;
      else p1 = pm;
    }
  }
  if (p1 - p0 < 2) return;
  const i32 s = a.cnt[p0];
  if (s == 0) return;   // both sides stay empty
  const i32 o = a.off[p0];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const i32* M = a.mcur + o;
  // ---- does it fit? ----
  i64 lsum = 0, wsum = 0;
  for (i32 i = threadIdx.x; i < s; i += blockDim.x) {
    const i32 v = M[i];
    lsum += a.xadj[v + 1] - a.xadj[v];
    wsum += (u32)a.vwgt[v];
  }
  block_sum2_i64(lsum, wsum, s_red);
  const i64 L = lsum, WS = wsum;
  if (s > kSmallMax || small_bytes(s, L, a.trials) > a.smem) {
    if (threadIdx.x == 0) {
      a.biglist[atomicAdd(a.bigcount + a.depth, 1)] = make_int2(p0, p1);
      a.bigmark[p0] = a.depth + 1;
    }
    return;
  }
  const SplitParams P = split_params(a, p0, p1, WS);
  int4* hdr = reinterpret_cast<int4*>(smem_raw);
  int2* edge = reinterpret_cast<int2*>(hdr + s);
  u16* perm = reinterpret_cast<u16*>(edge + L);
  unsigned char* st_raw =
      smem_raw + (((size_t)16 * s + (size_t)8 * L + (size_t)2 * s + 15) & ~(size_t)15);
  int4* tmp = reinterpret_cast<int4*>(st_raw);   // by member: row start in edge, kept entries, CSR start, weight sum
  if (threadIdx.x == 0) {
    s_bad = 0;
    s_maxd = 0;
    s_carry = 0;
  }
  __syncthreads();
  for (i32 i0 = 0; i0 < s; i0 += blockDim.x) {   // row starts: scan of the row lengths
    const i32 i = i0 + threadIdx.x;
    i32 b = 0, len = 0;
    if (i < s) {
      const i32 v = M[i];
      b = a.xadj[v];
      len = a.xadj[v + 1] - b;
    }
    i32 inc = len;
#pragma unroll
    for (int q = 1; q < 32; q <<= 1) {
      const i32 y = __shfl_up_sync(kFull32, inc, q);
      if (lane >= q) inc += y;
    }
    if (lane == 31) s_scan[wid] = inc;
    __syncthreads();
    i32 tot;
    const i32 before = s_carry + warps_before(s_scan, kSmallThreads / 32, tot);
    if (i < s) tmp[i] = make_int4(before + inc - len, len, b, 0);
    __syncthreads();
    if (threadIdx.x == 0) s_carry += tot;
  }
  __syncthreads();
  // ---- rows: the entries inside the sub-problem, kept in row order ----
  u64 hash = 0;
  i64 maxd = 0;
  bool bad = false;
  auto build_rows = [&](auto lanes_c) {
    constexpr int G = decltype(lanes_c)::value;
    const int sub = lane & (G - 1), grp = lane / G;
    const u32 gmask = (G == 32 ? kFull32 : ((1u << G) - 1u)) << (grp * G);
    const i32 per = (i32)blockDim.x / G;
    const i32 g0 = wid * (32 / G);
    for (i32 r0 = g0; r0 < s; r0 += per) {   // warp-uniform trip count
      const i32 i = r0 + grp;
      const bool act = i < s;
      const int4 t = act ? tmp[i] : make_int4(0, 0, 0, 0);
      i32 c = 0;
      i64 d = 0;
      for (i32 e0 = 0; __any_sync(kFull32, e0 < t.y); e0 += G) {
        const i32 e = e0 + sub;
        bool keep = false;
        i32 lu = 0, w = 0;
        if (e < t.y) {
          const i32 u = a.adjncy[t.z + e];
          w = a.adjwgt[t.z + e];
          lu = a.pos[u] - o;
          keep = (u32)lu < (u32)s;
        }
        const u32 bal = __ballot_sync(kFull32, keep) & gmask;
        if (keep) {
          edge[t.x + c + __popc(bal & ((1u << lane) - 1))] = make_int2(lu, w);
          d += w;
          bad |= w < 0;
          hash += entry_hash(i, lu, w);
        }
        c += __popc(bal);
      }
#pragma unroll
      for (int q = G / 2; q > 0; q >>= 1) d += __shfl_xor_sync(kFull32, d, q);
      bad |= d >= kPackedDeg;
      maxd = d > maxd ? d : maxd;
      if (act && sub == 0) tmp[i] = make_int4(t.x, c, t.z, (i32)d);
    }
  };
  if (L <= (i64)12 * s) build_rows(std::integral_constant<int, 8>());
  else build_rows(std::integral_constant<int, 32>());
  if (bad) s_bad = 1;
  else atomicMax(&s_maxd, (i32)__reduce_max_sync(__activemask(), (u32)maxd));
  const bool asym = block_sum_i64((i64)hash, s_red) != 0;   // (its barriers publish the rows and s_bad)
  const bool wide = asym || s_bad;                          // block-uniform
  // ---- slots: active members first ----
  i32 na = 0;
  for (i32 i0 = 0; i0 < s; i0 += blockDim.x) {
    const i32 i = i0 + threadIdx.x;
    na += __syncthreads_count(i < s && (wide || tmp[i].w != 0));
  }
  i32 doneA = 0;
  for (i32 i0 = 0; i0 < s; i0 += blockDim.x) {
    const i32 i = i0 + threadIdx.x;
    const bool in = i < s;
    const int4 t = in ? tmp[i] : make_int4(0, 0, 0, 0);
    const bool active = in && (wide || t.w != 0);
    const u32 bal = __ballot_sync(kFull32, active);
    if (lane == 0) s_scan[wid] = __popc(bal);
    __syncthreads();
    i32 tot;
    const i32 before = doneA + warps_before(s_scan, kSmallThreads / 32, tot);
    if (in) {
      const i32 ra = before + __popc(bal & ((1u << lane) - 1));
      const i32 slot = active ? ra : na + (i - ra);
      perm[i] = (u16)slot;
      hdr[slot] = make_int4(t.x, t.y, a.vwgt[M[i]], t.w);
    }
    doneA += tot;
    __syncthreads();
  }
  if (!wide && na < s) {   // edges name slots (with every member active they are the members)
    for (i32 i = threadIdx.x; i < na; i += blockDim.x) {
      const int4 h = hdr[i];
      for (i32 e = 0; e < h.y; ++e) edge[h.x + e].x = perm[edge[h.x + e].x];
    }
    __syncthreads();
  }
  // ---- trials ----
  u32* state = reinterpret_cast<u32*>(st_raw);
  const Packing K = packing_for(na, s_maxd);
  const i32 stw = packed_state_words(s);
  const i32 t = wid;
  if (t < a.trials) {
    const i32 sm = seed_member(a, p0, t, s);
    if (wide) {
      WideTopo T;
      T.hdr = hdr;
      T.edge = edge;
      i64 cut, dev;
      trial_wide(T, wide_state(a, t, p0, o), s, sm, P, cut, dev);
      if (lane == 0) {
        s_cut[t] = cut;
        s_dev[t] = dev;
        s_inert[t] = 0;
      }
    } else {
      u32* V = state + (size_t)t * stw;
      u32* B1 = V + pad_to(s, 32);
      const i32 nb1 = gggp_nb1(na);
      for (i32 b = 0; b < packed_b1_words(s); b += 32) B1[b + lane] = 0;
      __syncwarp();
      for (i32 b = 0; b < nb1; ++b) {
        const i32 i = (b << 5) + lane;
        const u32 x = i < na ? K.initial(hdr[i].w, i) : 0u;
        V[i] = x;
        const u32 m = __reduce_max_sync(kFull32, x);
        if (lane == 0) B1[b] = m;
      }
      __syncwarp();
      const long long c0 = clock64();
      auto hdr_of = [&](i32 i) { return hdr[i]; };
      auto fetch = [&](i32 rb, i32 rn) { return lane < rn ? edge[rb + lane] : make_int2(0, 0); };
      auto inert_w = [&](i32 i) -> i64 {
        const i32 sl = perm[i];
        return sl >= na && i != sm ? (i64)(u32)hdr[sl].z : (i64)-1;
      };
      const i32 sslot = perm[sm];
      i32 iend = 0;
      i64 wR;
      if (s <= 1024) {
        auto expand = [&](i32 rb, i32 rn, int2 ed, u32& best) {
          best = touch_neighbour<0, false>(V, B1, nullptr, ed, K.ib);
          for (i32 j0 = 32; j0 < rn; j0 += 32) {   // warp-uniform trip count
            const u32 x = touch_neighbour<0, false>(V, B1, nullptr, fetch(rb + j0, rn - j0), K.ib);
            best = x > best ? x : best;
          }
          return false;
        };
        wR = grow_packed<0, false>(K, V, B1, (u32*)nullptr, 0, s, na < s, sslot < na ? sslot : -1,
                                   (i64)(u32)hdr[sslot].z, P.TL, &iend, hdr_of, fetch, expand, inert_w);
      } else {
        auto expand = [&](i32 rb, i32 rn, int2 ed, u32& best) {
          best = touch_neighbour<1, false>(V, B1, nullptr, ed, K.ib);
          for (i32 j0 = 32; j0 < rn; j0 += 32) {   // warp-uniform trip count
            const u32 x = touch_neighbour<1, false>(V, B1, nullptr, fetch(rb + j0, rn - j0), K.ib);
            best = x > best ? x : best;
          }
          return false;
        };
        wR = grow_packed<1, false>(K, V, B1, (u32*)nullptr, 0, s, na < s, sslot < na ? sslot : -1,
                                   (i64)(u32)hdr[sslot].z, P.TL, &iend, hdr_of, fetch, expand, inert_w);
      }
      const long long c1 = clock64();
      // refinement: positive-gain moves within the side caps (inert members
      // have no gain)
      const i32 max_moves = gggp_max_moves(s);
      for (i32 mv = 0; mv < max_moves; ++mv) {
        i32 bg = 0;
        i32 bi = INT_MAX;
        for (i32 i = lane; i < na; i += 32) {
          const u32 x = V[i];
          const i32 g = move_gain(K, x);
          if (g > bg) {
            const i64 w = (u32)hdr[i].z;
            if (in_region(x) ? ((P.WS - wR) + w <= P.capR) : (wR + w <= P.capL)) {
              bg = g;
              bi = i;
            }
          }
        }
        const u32 mg = __reduce_max_sync(kFull32, (u32)bg);
        if (mg == 0) break;
        const i32 i = (i32)__reduce_min_sync(kFull32, (u32)bg == mg ? (u32)bi : 0x7fffffffu);
        const u32 x = V[i];
        const bool r = in_region(x);
        const int4 h = hdr[i];
        __syncwarp();
        if (lane == 0) V[i] = r ? word_leave(x) : word_enter(x);
        wR += r ? -(i64)(u32)h.z : (i64)(u32)h.z;
        for (i32 j = lane; j < h.y; j += 32) {
          const int2 ed = edge[h.x + j];
          if (ed.y) atomicAdd(&V[ed.x], (r ? 0u - 2u * (u32)ed.y : 2u * (u32)ed.y) << K.ib);
        }
        __syncwarp();
      }
      i64 cut = 0;
      for (i32 i = lane; i < na; i += 32) {
        const u32 x = V[i];
        if (in_region(x)) cut += ((i64)hdr[i].w - K.gain(x)) / 2;   // deg - conn
      }
      cut = warp_sum_i64(cut);
      if (lane == 0) {
        s_cut[t] = cut;
        s_dev[t] = wR > P.TL ? wR - P.TL : P.TL - wR;
        s_inert[t] = iend;
        if (a.prof) {
          atomicMax(a.prof, (unsigned long long)(c1 - c0));
          atomicMax(a.prof + 1, (unsigned long long)(clock64() - c1));
        }
      }
    }
  }
  __syncthreads();
  // ---- the best trial (smallest cut, then |W(R) - TL|, then index) splits ----
  i32 b = 0;
  for (i32 q = 1; q < a.trials; ++q)
    if (s_cut[q] < s_cut[b] || (s_cut[q] == s_cut[b] && s_dev[q] < s_dev[b])) b = q;
  if (wide) {
    const i32* R = wide_state(a, b, p0, o).R;
    split_members(a, P, s, o, s_scan, [&](i32 i) { return __ldcg(&R[i]) != 0; });
  } else {
    const u32* V = state + (size_t)b * stw;
    const i32 sm = seed_member(a, p0, b, s), iend = s_inert[b];
    split_members(a, P, s, o, s_scan, [&](i32 i) {
      const i32 sl = perm[i];
      return sl < na ? in_region(V[sl]) : (i < iend || i == sm);
    });
  }
}

// ---------------------------------------------------------------------------
// Large sub-problems.  k_gggp_rows filters their members' rows into global
// arrays with one warp per row over the whole grid (a dense 34k-vertex
// coarsest graph has 5.4M entries: one CTA took 20 ms for them), then every
// trial is a CTA of its own, and the last of a sub-problem's trials to finish
// splits it.  A trial keeps as much in shared memory as fits:
//   tier 0  words, B1, B2, headers, rows and the member -> slot map
//   tier 1  the same without the rows (read from L2)
//   tier 2  words, B1 and B2 by member; headers and rows from L2
//   tier 3  everything in global memory (more than ~50k members)
// Growth picks are one warp's; rows of more than kHelpRow entries and the
// refinement scans use the whole CTA.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_gggp_rows(GggpArgs a) {
  if (a.bigcount[a.depth] == 0) return;
  const int lane = threadIdx.x & 31;
  const i64 nw = ((i64)gridDim.x * blockDim.x) >> 5;
  for (i64 q = ((i64)blockIdx.x * blockDim.x + threadIdx.x) >> 5; q < a.n; q += nw) {
    const i32 v = a.mcur[q];
    const i32 p0 = a.part[v];
    if (a.bigmark[p0] != a.depth + 1) continue;   // warp-uniform
    const i32 o = a.off[p0], s = a.cnt[p0];
    const i32 b = a.xadj[v], e1 = a.xadj[v + 1];
    const i32 me = (i32)(q - o);
    i32 c = 0;
    i64 d = 0;
    u64 hash = 0;
    bool bad = false;
    constexpr i32 kU = 4;   // entries per lane whose loads are issued together
    i64 at = (i64)b + lane;
    for (i32 left = e1 - b; left > 0; left -= 32 * kU, at += 32 * kU) {   // (warp-uniform)
      i32 u[kU], w[kU], lu[kU];
#pragma unroll
      for (i32 x = 0; x < kU; ++x) {
        u[x] = left - lane > 32 * x ? a.adjncy[at + 32 * x] : -1;
        w[x] = left - lane > 32 * x ? a.adjwgt[at + 32 * x] : 0;
      }
#pragma unroll
      for (i32 x = 0; x < kU; ++x) lu[x] = u[x] >= 0 ? a.pos[u[x]] - o : -1;
#pragma unroll
      for (i32 x = 0; x < kU; ++x) {
        const bool keep = (u32)lu[x] < (u32)s;
        const u32 bal = __ballot_sync(kFull32, keep);
        if (keep) {
          a.g_edge[(i64)b + c + __popc(bal & ((1u << lane) - 1))] = make_int2(lu[x], w[x]);
          d += w[x];
          bad |= w[x] < 0;
          hash += entry_hash(me, lu[x], w[x]);
        }
        c += __popc(bal);
      }
    }
    d = warp_sum_i64(d);
    hash = (u64)warp_sum_i64((i64)hash);
    bad = __any_sync(kFull32, bad) || d >= kPackedDeg;
    if (lane == 0) {
      a.g_hdr[q] = make_int4(b, c, a.vwgt[v], (i32)d);
      if (hash) atomicAdd(reinterpret_cast<unsigned long long*>(a.bighash + p0), (unsigned long long)hash);
      if (bad) a.bigwide[p0] = 1;
    }
  }
}

constexpr int kBigThreads = 512;
constexpr size_t kGggpBigSmem = 224 * 1024;
constexpr i32 kHelpRow = 256;   // rows longer than this are read by the whole CTA

__device__ __forceinline__ void bar_all() { asm volatile("bar.sync 1, 512;" ::: "memory"); }
static_assert(kBigThreads == 512, "bar_all counts every thread of the CTA");

// One trial on the packed state; see grow_packed for the accessors.  `na`
// words, active members first (tiers 0 and 1) or every member (2 and 3).
template <int LV, bool kGlobal, bool kRowsGlobal, class Hdr, class Edge, class InertW>
__device__ void big_trial(const SplitParams& P, const Packing K, u32* V, u32* B1, u32* B2, i32 nb2p, i32 na, i32 s, bool inert,
                          i32 sslot, i64 seed_w, i32* s_cmd, i64* s_wR, i32* s_iend, u32* s_max, i64* s_red,
                          Hdr hdr, Edge edge, InertW inert_w, i64* cut_out, i64* dev_out,
                          unsigned long long* prof) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  // neighbours j, j + nthr, ... of a row; four loads issued together
  auto pass = [&](i32 rb, i32 rn, i32 first, i32 nthr, u32& best) {
    constexpr i32 kU = kRowsGlobal ? 4 : 1;
    for (i32 j0 = first; j0 < rn; j0 += nthr * kU) {
      int2 ed[kU];
#pragma unroll
      for (i32 x = 0; x < kU; ++x) ed[x] = j0 + x * nthr < rn ? edge(rb + j0 + x * nthr) : make_int2(0, 0);
#pragma unroll
      for (i32 x = 0; x < kU; ++x) {
        const u32 y = touch_neighbour<LV, kGlobal>(V, B1, B2, ed[x], K.ib);
        best = y > best ? y : best;
      }
    }
  };
  auto fetch = [&](i32 rb, i32 rn) { return lane < rn && rn <= kHelpRow ? edge(rb + lane) : make_int2(0, 0); };
  const long long c0 = clock64();
  if (wid == 0) {
    auto expand = [&](i32 rb, i32 rn, int2 ed, u32& best) {
      if (rn <= kHelpRow) {
        best = touch_neighbour<LV, kGlobal>(V, B1, B2, ed, K.ib);
        if (rn > 32) pass(rb + 32, rn - 32, lane, 32, best);
        return false;
      }
      if (lane == 0) {
        s_cmd[0] = rb;
        s_cmd[1] = rn;
      }
      bar_all();
      pass(rb, rn, (i32)threadIdx.x, kBigThreads, best);
      bar_all();
      return true;
    };
    i32 iend = 0;
    const i64 wR = grow_packed<LV, kGlobal>(K, V, B1, B2, nb2p, s, inert, sslot, seed_w, P.TL, &iend, hdr, fetch,
                                               expand, inert_w);
    if (lane == 0) {
      s_cmd[1] = -1;
      *s_wR = wR;
      *s_iend = iend;
    }
    bar_all();
  } else {
    for (;;) {   // ends with warp 0's growth, which ends after at most one step per member
      bar_all();
      const i32 rb = s_cmd[0], rn = s_cmd[1];
      if (rn < 0) break;
      u32 best = 0;
      pass(rb, rn, (i32)threadIdx.x, kBigThreads, best);
      bar_all();
    }
  }
  __syncthreads();
  const long long c1 = clock64();
  i64 wR = *s_wR;
  // refinement: positive-gain moves within the side caps; the CTA's largest
  // gain, then the smallest slot that has it
  const i32 max_moves = gggp_max_moves(s);
  for (i32 mv = 0; mv < max_moves; ++mv) {
    i32 bg = 0;
    u32 bi = 0x7fffffffu;
    for (i32 i = threadIdx.x; i < na; i += kBigThreads) {
      const u32 x = ldw<kGlobal>(V + i);
      if (kGlobal || LV == 2) {   // by member: inert words are 0 and never move
        if (x == 0) continue;
      }
      const i32 g = move_gain(K, x);
      if (g > bg) {
        const i64 w = (u32)hdr(i).z;
        if (in_region(x) ? ((P.WS - wR) + w <= P.capR) : (wR + w <= P.capL)) {
          bg = g;
          bi = (u32)i;
        }
      }
    }
    const u32 mg = __reduce_max_sync(kFull32, (u32)bg);
    const u32 mi = __reduce_min_sync(kFull32, (u32)bg == mg ? bi : 0x7fffffffu);
    __syncthreads();
    if (lane == 0) {
      s_max[wid] = mg;
      s_max[32 + wid] = mi;
    }
    __syncthreads();
    u32 g = 0, gi = 0x7fffffffu;
    for (int w = 0; w < kBigThreads / 32; ++w) {
      const u32 x = s_max[w], y = s_max[32 + w];
      if (x > g || (x == g && y < gi)) {
        g = x;
        gi = y;
      }
    }
    if (g == 0) break;   // block-uniform
    const i32 i = (i32)gi;
    const u32 x = ldw<kGlobal>(V + i);
    const bool r = in_region(x);
    const int4 h = hdr(i);
    wR += r ? -(i64)(u32)h.z : (i64)(u32)h.z;
    __syncthreads();   // every thread has read the word
    if (threadIdx.x == 0) V[i] = r ? word_leave(x) : word_enter(x);
    for (i32 j = threadIdx.x; j < h.y; j += kBigThreads) {
      const int2 ed = edge(h.x + j);
      if (ed.y) atomicAdd(&V[ed.x], (r ? 0u - 2u * (u32)ed.y : 2u * (u32)ed.y) << K.ib);
    }
    __syncthreads();
  }
  i64 cut = 0;
  for (i32 i = threadIdx.x; i < na; i += kBigThreads) {
    const u32 x = ldw<kGlobal>(V + i);
    if (x && in_region(x)) cut += ((i64)hdr(i).w - K.gain(x)) / 2;   // deg - conn
  }
  *cut_out = block_sum_i64(cut, s_red);
  *dev_out = wR > P.TL ? wR - P.TL : P.TL - wR;
  if (prof && threadIdx.x == 0) {
    atomicMax(prof, (unsigned long long)(c1 - c0));
    atomicMax(prof + 1, (unsigned long long)(clock64() - c1));
  }
}

__global__ void __launch_bounds__(kBigThreads, 1) k_gggp_big(GggpArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ i64 s_red[kBigThreads / 32];
  __shared__ u32 s_max[64];
  __shared__ i32 s_scan[kBigThreads / 32];
  __shared__ i32 s_cmd[2];
  __shared__ i64 s_wR;
  __shared__ i32 s_iend, s_last;
  const i32 j = blockIdx.x / a.trials, t = blockIdx.x % a.trials;
  if (j >= a.bigcount[a.depth]) return;
  const int2 sub = a.biglist[j];
  const i32 p0 = sub.x;
  const i32 s = a.cnt[p0], o = a.off[p0];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int4* ghdr = a.g_hdr + o;
  const bool wide = a.bighash[p0] != 0 || a.bigwide[p0] != 0;
  i64 wsum = 0, esum = 0;
  i32 act = 0, maxd = 0;
  if (threadIdx.x == 0) s_cmd[0] = 0;
  __syncthreads();
  for (i32 i = threadIdx.x; i < s; i += blockDim.x) {
    const int4 h = ghdr[i];
    wsum += (u32)h.z;
    maxd = h.w > maxd ? h.w : maxd;
    if (h.w != 0) {
      ++act;
      esum += h.y;
    }
  }
  if (maxd) atomicMax(&s_cmd[0], maxd);
  const i64 WS = block_sum_i64(wsum, s_red);
  maxd = s_cmd[0];   // (behind the sum's barriers; set again only after the next ones)
  const i64 ES = block_sum_i64(esum, s_red);
  const i32 na = (i32)block_sum_i64(act, s_red);
  const SplitParams P = split_params(a, p0, sub.y, WS);
  const i32 sm = seed_member(a, p0, t, s);
  u8* R = a.g_R + (size_t)t * a.n + o;
  i64 cut = 0, dev = 0;
  if (wide) {   // block-uniform
    __shared__ i64 s_res[2];
    if (wid == 0) {
      WideTopo T;
      T.hdr = ghdr;
      T.edge = a.g_edge;
      i64 c, d;
      trial_wide(T, wide_state(a, t, p0, o), s, sm, P, c, d);
      if (lane == 0) {
        s_res[0] = c;
        s_res[1] = d;
      }
    }
    __syncthreads();
    cut = s_res[0];
    dev = s_res[1];
    const i32* RW = wide_state(a, t, p0, o).R;
    for (i32 i = threadIdx.x; i < s; i += blockDim.x) R[i] = (u8)(__ldcg(&RW[i]) != 0);
  } else {
    // ---- tier ----
    const size_t state = (size_t)4 * (packed_state_words(na) + 96);   // B1 of at least 128 words
    const size_t mapb = ((size_t)2 * s + 15) & ~(size_t)15;
    const size_t head = state + (size_t)16 * na + mapb;
    const bool mapped = s <= 65535 && head <= a.smem;            // tiers 0 and 1
    const bool rows_in = mapped && head + (size_t)8 * ES <= a.smem;
    const size_t by_member = (size_t)4 * (pad_to(s, 32) + pad_to(gggp_nb1(s), 32) + pad_to(gggp_nb2(s), 64));
    u32 *V, *B1, *B2;
    const i32 ns = mapped ? na : s;   // words
    const Packing K = packing_for(ns, maxd);
    i32 nb1p, nb2p;
    if (mapped) {
      nb1p = packed_b1_words(ns);
      nb2p = packed_b2_words(ns);
      if (ns <= 1024) nb1p = 128;   // level 1's layout for small sets too
    } else {
      nb1p = pad_to(gggp_nb1(ns), 32);
      nb2p = pad_to(gggp_nb2(ns), 64);
    }
    const bool in_smem = mapped || by_member <= a.smem;
    V = in_smem ? reinterpret_cast<u32*>(smem_raw) : a.g_V + (size_t)t * a.v_stride + 2 * (size_t)o;
    B1 = V + pad_to(ns, 32);
    B2 = B1 + nb1p;
    // tiers 0 and 1: headers by slot, the map, and the rows by slot
    int4* hdr = reinterpret_cast<int4*>(smem_raw + (((size_t)4 * (pad_to(ns, 32) + nb1p + nb2p) + 15) & ~(size_t)15));
    u16* perm = reinterpret_cast<u16*>(hdr + ns);
    int2* edge = reinterpret_cast<int2*>(reinterpret_cast<unsigned char*>(perm) + mapb);
    if (mapped) {
      i32 done = 0, ebase = 0;
      for (i32 i0 = 0; i0 < s; i0 += blockDim.x) {   // block-uniform trip count
        const i32 i = i0 + threadIdx.x;
        const int4 h = i < s ? ghdr[i] : make_int4(0, 0, 0, 0);
        const bool on = i < s && h.w != 0;
        const u32 bal = __ballot_sync(kFull32, on);
        i32 inc = on ? h.y : 0;
#pragma unroll
        for (int q = 1; q < 32; q <<= 1) {
          const i32 y = __shfl_up_sync(kFull32, inc, q);
          if (lane >= q) inc += y;
        }
        if (lane == 31) {
          s_scan[wid] = __popc(bal);
          s_max[wid] = (u32)inc;
        }
        __syncthreads();
        i32 before = done, tot = 0, eb = ebase, et = 0;
        for (int w = 0; w < kBigThreads / 32; ++w) {
          const i32 x = s_scan[w], y = (i32)s_max[w];
          before += w < wid ? x : 0;
          tot += x;
          eb += w < wid ? y : 0;
          et += y;
        }
        if (i < s) {
          const i32 slot = before + __popc(bal & ((1u << lane) - 1));
          perm[i] = on ? (u16)slot : (u16)0xffff;
          if (on) hdr[slot] = make_int4(rows_in ? eb + inc - h.y : h.x, h.y, h.z, h.w);
        }
        done += tot;
        ebase += et;
        __syncthreads();
      }
      if (rows_in) {
        for (i32 i = wid; i < s; i += kBigThreads / 32) {   // one warp per row
          const i32 sl = perm[i];
          if (sl == 0xffff) continue;
          const int4 h = ghdr[i];
          const i32 eb = hdr[sl].x;
          for (i32 e = lane; e < h.y; e += 32) {
            const int2 x = a.g_edge[(i64)h.x + e];
            edge[eb + e] = make_int2(x.y ? (i32)perm[x.x] : 0, x.y);
          }
        }
      }
    }
    // words and block maxima (conn = 0)
    for (i32 q = threadIdx.x; q < nb1p + nb2p; q += kBigThreads) B1[q] = 0;
    __syncthreads();
    for (i32 b = wid; b < gggp_nb1(ns); b += kBigThreads / 32) {
      const i32 i = (b << 5) + lane;
      u32 x = 0;
      if (i < ns) {
        const i32 d = mapped ? hdr[i].w : ghdr[i].w;
        x = mapped || d != 0 ? K.initial(d, i) : 0u;
      }
      V[i] = x;
      const u32 m = __reduce_max_sync(kFull32, x);
      if (lane == 0) {
        B1[b] = m;
        if (nb2p) atomicMax(&B2[b >> 5], m);
      }
    }
    __syncthreads();
    auto inert_of = [&](i32 i) { return mapped ? perm[i] == 0xffff : ghdr[i].w == 0; };
    auto inert_w = [&](i32 i) -> i64 { return i != sm && inert_of(i) ? (i64)(u32)ghdr[i].z : (i64)-1; };
    const bool inert = na < s;
    const i32 sslot = inert_of(sm) ? -1 : mapped ? (i32)perm[sm] : sm;
    const i64 seed_w = (u32)ghdr[sm].z;
    auto hdr_s = [&](i32 i) { return hdr[i]; };
    auto hdr_g = [&](i32 i) { return ghdr[i]; };
    auto edge_s = [&](i32 e) { return edge[e]; };
    auto edge_m = [&](i32 e) {
      int2 x = a.g_edge[e];
      x.x = x.y ? (i32)perm[x.x] : 0;
      return x;
    };
    auto edge_g = [&](i32 e) { return a.g_edge[e]; };
    u32* sV = reinterpret_cast<u32*>(smem_raw);   // the shared-memory tiers' words, by their own address space
    u32* sB1 = sV + pad_to(ns, 32);
    u32* sB2 = sB1 + nb1p;
    if (rows_in && ns <= 4096)
      big_trial<1, false, false>(P, K, sV, sB1, sB2, nb2p, ns, s, inert, sslot, seed_w, s_cmd, &s_wR, &s_iend, s_max,
                                 s_red, hdr_s, edge_s, inert_w, &cut, &dev, a.prof);
    else if (mapped && ns <= 4096)
      big_trial<1, false, true>(P, K, sV, sB1, sB2, nb2p, ns, s, inert, sslot, seed_w, s_cmd, &s_wR, &s_iend, s_max,
                                s_red, hdr_s, edge_m, inert_w, &cut, &dev, a.prof);
    else if (rows_in)
      big_trial<2, false, false>(P, K, sV, sB1, sB2, nb2p, ns, s, inert, sslot, seed_w, s_cmd, &s_wR, &s_iend, s_max,
                                 s_red, hdr_s, edge_s, inert_w, &cut, &dev, a.prof);
    else if (mapped)
      big_trial<2, false, true>(P, K, sV, sB1, sB2, nb2p, ns, s, inert, sslot, seed_w, s_cmd, &s_wR, &s_iend, s_max,
                                s_red, hdr_s, edge_m, inert_w, &cut, &dev, a.prof);
    else if (in_smem)
      big_trial<2, false, true>(P, K, sV, sB1, sB2, nb2p, ns, s, inert, sslot, seed_w, s_cmd, &s_wR, &s_iend, s_max,
                                s_red, hdr_g, edge_g, inert_w, &cut, &dev, a.prof);
    else
      big_trial<2, true, true>(P, K, V, B1, B2, nb2p, ns, s, inert, sslot, seed_w, s_cmd, &s_wR, &s_iend, s_max, s_red,
                               hdr_g, edge_g, inert_w, &cut, &dev, a.prof);
    const i32 iend = s_iend;
    for (i32 i = threadIdx.x; i < s; i += kBigThreads) {
      bool r;
      if (inert_of(i)) r = i < iend || i == sm;
      else {
        const u32 x = in_smem ? sV[mapped ? (i32)perm[i] : i] : __ldcg(&V[i]);
        r = in_region(x);
      }
      R[i] = r ? 1 : 0;
    }
  }
  // ---- the sub-problem's last trial picks the best one and splits ----
  if (threadIdx.x == 0) {
    a.tcut[(size_t)j * kInitTrials + t] = cut;
    a.tdev[(size_t)j * kInitTrials + t] = dev;
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    s_last = atomicAdd(&a.bigdone[j], 1) == a.trials - 1;
    __threadfence();
  }
  __syncthreads();
  if (!s_last) return;
  i32 b = 0;
  const long long* tc = reinterpret_cast<const long long*>(a.tcut + (size_t)j * kInitTrials);
  const long long* td = reinterpret_cast<const long long*>(a.tdev + (size_t)j * kInitTrials);
  for (i32 q = 1; q < a.trials; ++q) {
    const i64 cq = __ldcg(tc + q), cb = __ldcg(tc + b);
    if (cq < cb || (cq == cb && __ldcg(td + q) < __ldcg(td + b))) b = q;
  }
  const u8* Rb = a.g_R + (size_t)b * a.n + o;
  split_members(a, P, s, o, s_scan, [&](i32 i) { return __ldcg(Rb + i) != 0; });
  if (threadIdx.x == 0) a.bigdone[j] = 0;   // ready for the next depth
}

// M = pos = identity, every vertex in its graph's first part, the root
// sub-problems' places, and the counters of all depths.  `other`: M's second
// buffer.  A depth writes only the places of the members it splits, and
// k_gggp_rows reads every place: a graph of one part (batched) is never split,
// so its places must name its own vertices in both buffers from the start.
__global__ void k_gggp_init(GggpArgs a, i32* other, i32 depths, i32 maxbig, const i32* __restrict__ gid,
                            const i32* __restrict__ gpbase, const i32* __restrict__ part_v0,
                            const i32* __restrict__ part_v1) {
  const i64 v = (i64)blockIdx.x * blockDim.x + threadIdx.x;
  if (v < a.n) {
    a.mnext[v] = (i32)v;
    if (maxbig > 0) other[v] = (i32)v;
    a.pos[v] = (i32)v;
    a.part[v] = gid ? gpbase[gid[v]] : 0;
  }
  if (v < a.k) {
    const bool root = a.part_base ? a.part_base[v] == (i32)v : v == 0;
    a.off[v] = root && part_v0 ? part_v0[v] : 0;
    a.cnt[v] = !root ? 0 : part_v0 ? part_v1[v] - part_v0[v] : a.n;
    if (maxbig > 0) {
      a.bigmark[v] = 0;
      a.bighash[v] = 0;
      a.bigwide[v] = 0;
    }
  }
  if (maxbig > 0) {
    if (v < depths) a.bigcount[v] = 0;
    if (v < maxbig) a.bigdone[v] = 0;
  }
}

static void device_init_partition_body(Handle& h, const DevGraph& g, i32 k, double eps, u64 seed, i32 trials,
                                       i32* d_part, const GggpBatch* batch);

// The launch sequence (one to three launches per recursion depth, sized by n
// and k) runs through the handle's graph cache, except when traced or batched.
void device_init_partition(Handle& h, const DevGraph& g, i32 k, double eps, u64 seed, i32 trials,
                           i32* d_part, const GggpBatch* batch) {
  GKW_REQUIRE(trials >= 1 && trials <= kInitTrials, GKW_E_INVALID, "init trials must be in [1, 8]");
  if (g.n == 0) return;
  GKW_CUDA(cudaFuncSetAttribute(k_gggp_small, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGggpSmem));
  GKW_CUDA(cudaFuncSetAttribute(k_gggp_big, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGggpBigSmem));
  const bool trace = getenv("GKW_TRACE") && *getenv("GKW_TRACE") == '1';
  auto body = [&] { device_init_partition_body(h, g, k, eps, seed, trials, d_part, batch); };
  if (trace || batch) {
    body();
    return;
  }
  struct K {
    i64 n, m, k, trials;
    double eps;
    u64 seed;
    const void* p[5];
    const void* sbase;
    size_t stop;
    i32 narrow, sms;
  } key;
  memset(&key, 0, sizeof(key));
  key.n = g.n;
  key.m = g.m;
  key.k = k;
  key.trials = trials;
  key.eps = eps;
  key.seed = seed;
  key.p[0] = g.xadj;
  key.p[1] = g.adjncy;
  key.p[2] = g.adjwgt;
  key.p[3] = g.vwgt;
  key.p[4] = d_part;
  const auto fp = h.scratch.fingerprint();
  key.sbase = fp.first;
  key.stop = fp.second;
  key.narrow = h.narrow;
  key.sms = h.sm_count;
  graph_run(h, std::string("gggp", 4) + std::string(reinterpret_cast<const char*>(&key), sizeof(key)), body);
}

static void device_init_partition_body(Handle& h, const DevGraph& g, i32 k, double eps, u64 seed, i32 trials,
                                       i32* d_part, const GggpBatch* batch) {
  const i32 n = g.n;
  Pool::Mark mk = h.scratch.mark();
  i32 depth = 0;
  if (batch) depth = batch->depth;
  else
    while ((1 << depth) < k) ++depth;
  auto subs_at = [&](i32 d) -> i64 {
    return batch ? (i64)batch->sub_ptr[d + 1] - batch->sub_ptr[d] : (i64)1 << d;
  };
  // two CTAs per SM once a depth has more sub-problems than SMs
  auto smem_at = [&](i32 d) { return subs_at(d) > h.sm_count ? kGggpSmemHalf : kGggpSmem; };
  size_t smem_min = kGggpSmem;
  for (i32 d = 0; d < depth; ++d) smem_min = std::min(smem_min, smem_at(d));
  // Sub-problems that one CTA may not hold: each has more than kSmallMax
  // members or needs more than the launch's shared memory, of which
  // (18 + 4 * trials) bytes a member, 8 an entry and 512 a trial for B1
  // (see small_bytes; padding under 128 bytes a trial).
  const double per_member = std::max(34.0, 18.0 + 4.0 * trials);
  const i32 maxbig = (i32)std::min<double>(
      n, std::max((double)n / (kSmallMax + 1),
                  (per_member * n + 8.0 * (double)g.m) / ((double)smem_min - 640.0 * trials - 64.0)) +
             (double)n / (kSmallMax + 1));
  GggpArgs a;
  memset(&a, 0, sizeof(a));
  a.n = n;
  a.k = k;
  a.trials = trials;
  a.xadj = g.xadj;
  a.adjncy = g.adjncy;
  a.adjwgt = g.adjwgt;
  a.vwgt = g.vwgt;
  i32* ml[2] = {h.scratch.alloc_n<i32>(n), h.scratch.alloc_n<i32>(n)};
  a.pos = h.scratch.alloc_n<i32>(n);
  a.part = d_part;
  a.cnt = h.scratch.alloc_n<i32>(k);
  a.off = h.scratch.alloc_n<i32>(k);
  a.seed = seed;
  a.eps = eps;
  a.part_base = batch ? batch->part_base : nullptr;
  a.w_state = h.scratch.alloc_n<i32>((size_t)kInitTrials * 2 * n);
  a.w_keys = h.scratch.alloc_n<u64>((size_t)kInitTrials * n);
  a.b1_stride = (size_t)n / 32 + (size_t)k + 2;
  a.b2_stride = (size_t)n / 1024 + (size_t)k + 2;
  a.w_b1 = h.scratch.alloc_n<u64>((size_t)kInitTrials * a.b1_stride);
  a.w_b2 = h.scratch.alloc_n<u64>((size_t)kInitTrials * a.b2_stride);
  if (maxbig > 0) {
    a.bigcount = h.scratch.alloc_n<i32>(std::max(depth, 1));
    a.biglist = h.scratch.alloc_n<int2>(maxbig);
    a.bigmark = h.scratch.alloc_n<i32>(k);
    a.bighash = h.scratch.alloc_n<u64>(k);
    a.bigwide = h.scratch.alloc_n<i32>(k);
    a.bigdone = h.scratch.alloc_n<i32>(maxbig);
    a.g_hdr = h.scratch.alloc_n<int4>(n);
    a.g_edge = h.scratch.alloc_n<int2>(std::max<i64>(g.m, 1));
    a.g_R = h.scratch.alloc_n<u8>((size_t)kInitTrials * n);
    a.tcut = h.scratch.alloc_n<i64>((size_t)maxbig * kInitTrials);
    a.tdev = h.scratch.alloc_n<i64>((size_t)maxbig * kInitTrials);
    // words of a sub-problem at place o: from 2 * o (s members take s + s/32 +
    // s/1024 words and under 160 of padding, less than 2 * s for the s of 50k
    // and more that come here)
    a.v_stride = 2 * (size_t)n;
    if ((size_t)4 * (pad_to(n, 32) + pad_to(gggp_nb1(n), 32) + pad_to(gggp_nb2(n), 64)) > kGggpBigSmem)
      a.g_V = h.scratch.alloc_n<u32>((size_t)kInitTrials * a.v_stride);
  }
  a.mnext = ml[0];
  launch(k_gggp_init, ceil_div((u64)std::max({n, k, maxbig, depth}), 256), 256, 0, h.stream, a, ml[1], depth, maxbig,
         batch ? batch->gid : (const i32*)nullptr, batch ? batch->gpbase : (const i32*)nullptr,
         batch ? batch->part_v0 : (const i32*)nullptr, batch ? batch->part_v1 : (const i32*)nullptr);
  GKW_CHECK_LAUNCH();
  const bool trace = getenv("GKW_TRACE") && *getenv("GKW_TRACE") == '1';
  std::vector<cudaEvent_t> ev;
  unsigned long long* prof = nullptr;   // per depth: slowest trial's growth / refinement cycles
  if (trace) {
    prof = reinterpret_cast<unsigned long long*>(h.scratch.alloc_n<u64>(2 * (size_t)std::max(depth, 1)));
    GKW_CUDA(cudaMemsetAsync(prof, 0, sizeof(u64) * 2 * std::max(depth, 1), h.stream));
    ev.resize(depth + 1);
    for (auto& e : ev) GKW_CUDA(cudaEventCreate(&e));
    GKW_CUDA(cudaEventRecord(ev[0], h.stream));
  }
  for (i32 d = 0; d < depth; ++d) {
    a.depth = d;
    a.mcur = ml[d & 1];
    a.mnext = ml[(d & 1) ^ 1];
    a.subs = batch ? batch->subs + batch->sub_ptr[d] : nullptr;
    a.prof = prof ? prof + 2 * d : nullptr;
    a.smem = smem_at(d);
    const i64 ns = subs_at(d);
    if (ns > 0) {
      launch(k_gggp_small, (u32)ns, kSmallThreads, a.smem, h.stream, a);
      if (maxbig > 0) {
        a.smem = kGggpBigSmem;
        launch(k_gggp_rows, std::min<u32>(ceil_div((u64)n, 8), (u32)h.sm_count * 8), 256, 0, h.stream, a);
        launch(k_gggp_big, (u32)std::min<i64>(maxbig, ns) * trials, kBigThreads, kGggpBigSmem, h.stream, a);
      }
      GKW_CHECK_LAUNCH();
    }
    if (trace) GKW_CUDA(cudaEventRecord(ev[d + 1], h.stream));
  }
  if (trace) {
    GKW_CUDA(cudaEventSynchronize(ev[depth]));
    std::vector<unsigned long long> hp(2 * (size_t)std::max(depth, 1));
    if (depth) {
      GKW_CUDA(cudaMemcpyAsync(hp.data(), prof, sizeof(u64) * 2 * depth, cudaMemcpyDeviceToHost, h.stream));
      GKW_CUDA(cudaStreamSynchronize(h.stream));
    }
    fprintf(stderr, "[gkw trace] init n=%d k=%d:", n, k);
    for (i32 d = 0; d < depth; ++d) {
      float ms = 0;
      cudaEventElapsedTime(&ms, ev[d], ev[d + 1]);
      fprintf(stderr, " d%d %.1fus (growth %.2f, refinement %.2f Mcycles)", d, ms * 1e3, hp[2 * d] / 1e6,
              hp[2 * d + 1] / 1e6);
    }
    fprintf(stderr, "\n");
    for (auto& e : ev) cudaEventDestroy(e);
  }
  h.scratch.release(mk);   // stream order keeps the scratch alive for the queued work
}

}  // namespace gkw
