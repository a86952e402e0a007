// Coarsening: heavy-edge candidates, union-find grouping, coarse ids, and
// contraction into the coarse CSR.  Semantics follow the reference's
// gkway/coarsen.hpp; the kernels are organised for B200 (sub-warp rows,
// shared-memory hashing, no host round trip per union-find iteration).
#include <algorithm>
#include <climits>
#include <cstddef>
#include <type_traits>

#include "device_util.cuh"

namespace gkw {

static constexpr u32 kFull = 0xffffffffu;

// ===========================================================================
// Heavy-edge candidate (coarsen.hpp:39-78).  G lanes per vertex; each lane
// keeps the best entry of its stride of the row under the key
// (weight desc, neighbour degree asc, position asc), zero weights excluded;
// the G partial results are reduced by shuffles.  This is the serial rule of
// the reference: the first position with minimum degree among the maximum
// weight entries, or the vertex itself when no entry has positive weight.
// ===========================================================================
// Rows longer than kMatchLong are left to k_match_long (one CTA per row), so
// a hub row never holds its group's lanes for thousands of dependent loads.
constexpr i32 kMatchLong = 512;

// the candidate rule's order: weight desc, neighbour degree asc, position asc
__device__ __forceinline__ bool match_better(u32 w, u32 d, i32 pos, u32 bw, u32 bd, i32 bpos) {
  return w > bw || (w == bw && (d < bd || (d == bd && pos < bpos)));
}

// Where the union-find starts (see below), written beside the candidate.
constexpr u32 kUfUnknown = 0xffffffffu;
struct UfStart {
  i32* parent = nullptr;
  u32* dist = nullptr;
  __device__ __forceinline__ void set(i32 v, i32 c) const {
    if (parent) {
      parent[v] = c > v ? c : v;
      dist[v] = kUfUnknown;
    }
  }
};

template <int G>
__global__ void __launch_bounds__(256) k_match(i32 n, const i32* __restrict__ xadj,
                                               const i32* __restrict__ adjncy,
                                               const i32* __restrict__ adjwgt, i32* __restrict__ cand,
                                               i32* __restrict__ longlist, i32* __restrict__ longcnt,
                                               UfStart uf) {
  const i64 t = (i64)blockIdx.x * blockDim.x + threadIdx.x;
  const i32 v = (i32)(t / G);
  const int sub = threadIdx.x & (G - 1);
  u32 bw = 0, bd = kFull;
  i32 bpos = INT_MAX, bu = -1;
  bool skip = false;
  if (v < n) {
    const i32 beg = __ldg(xadj + v), end = __ldg(xadj + v + 1);
    skip = longlist != nullptr && end - beg > kMatchLong;   // uniform within the group
    if (skip) {
      if (sub == 0) longlist[atomicAdd(longcnt, 1)] = v;
    } else {
      const i32 *rw = adjwgt + beg, *ra = adjncy + beg;
      const i32 len = end - beg;
      for (i32 e = sub; e < len; e += G) {   // places from the row's start
        const u32 w = (u32)__ldg(rw + e);
        if (w == 0 || w < bw) continue;
        const i32 u = __ldg(ra + e);
        const u32 d = (u32)(__ldg(xadj + u + 1) - __ldg(xadj + u));
        if (w > bw || d < bd) { bw = w; bd = d; bpos = e; bu = u; }
      }
    }
  }
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1) {
    const u32 ow = __shfl_xor_sync(kFull, bw, o, G);
    const u32 od = __shfl_xor_sync(kFull, bd, o, G);
    const i32 op = __shfl_xor_sync(kFull, bpos, o, G);
    const i32 ou = __shfl_xor_sync(kFull, bu, o, G);
    if (match_better(ow, od, op, bw, bd, bpos)) { bw = ow; bd = od; bpos = op; bu = ou; }
  }
  if (v < n && sub == 0 && !skip) {
    const i32 c = bw > 0 ? bu : v;
    cand[v] = c;
    uf.set(v, c);
  }
}

// One CTA per long row (listed by k_match): the threads stride the row --
// its 16-byte-aligned body four entries per load when both arrays are
// 16-byte aligned -- and the per-thread bests are reduced by the same rule.
constexpr int kMatchLongThreads = 256;
__global__ void __launch_bounds__(kMatchLongThreads) k_match_long(const i32* __restrict__ xadj,
                                                                  const i32* __restrict__ adjncy,
                                                                  const i32* __restrict__ adjwgt,
                                                                  i32* __restrict__ cand,
                                                                  const i32* __restrict__ longlist,
                                                                  const i32* __restrict__ longcnt, UfStart uf) {
  __shared__ u32 s_w[kMatchLongThreads / 32], s_d[kMatchLongThreads / 32];
  __shared__ i32 s_p[kMatchLongThreads / 32], s_u[kMatchLongThreads / 32];
  const i32 nlong = *longcnt;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const bool vec = ((reinterpret_cast<uintptr_t>(adjncy) | reinterpret_cast<uintptr_t>(adjwgt)) & 15) == 0;
  for (i32 r = blockIdx.x; r < nlong; r += gridDim.x) {
    const i32 v = longlist[r];
    const i32 beg = xadj[v], end = xadj[v + 1];
    u32 bw = 0, bd = kFull;
    i32 bpos = INT_MAX, bu = -1;
    auto visit = [&](u32 w, i32 u, i32 e) {
      if (w == 0 || w < bw) return;
      const u32 d = (u32)(__ldg(xadj + u + 1) - __ldg(xadj + u));
      if (match_better(w, d, e, bw, bd, bpos)) { bw = w; bd = d; bpos = e; bu = u; }
    };
    i32 body = beg, tail = end;
    if (vec) {
      body = (beg + 3) & ~3;
      tail = body + ((end - body) & ~3);
      if (tail < body) tail = body;
      for (i32 e = beg + threadIdx.x; e < body && e < end; e += blockDim.x) visit((u32)adjwgt[e], adjncy[e], e);
      for (i32 c = body / 4 + threadIdx.x; c < tail / 4; c += blockDim.x) {
        const int4 w4 = __ldg(reinterpret_cast<const int4*>(adjwgt) + c);
        const int4 u4 = __ldg(reinterpret_cast<const int4*>(adjncy) + c);
        visit((u32)w4.x, u4.x, 4 * c);
        visit((u32)w4.y, u4.y, 4 * c + 1);
        visit((u32)w4.z, u4.z, 4 * c + 2);
        visit((u32)w4.w, u4.w, 4 * c + 3);
      }
      for (u32 e = (u32)(tail > body ? tail : body) + threadIdx.x; e < (u32)end; e += blockDim.x)
        visit((u32)adjwgt[e], adjncy[e], (i32)e);
    } else {
      for (u32 e = (u32)beg + threadIdx.x; e < (u32)end; e += blockDim.x) visit((u32)adjwgt[e], adjncy[e], (i32)e);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const u32 ow = __shfl_xor_sync(kFull, bw, o);
      const u32 od = __shfl_xor_sync(kFull, bd, o);
      const i32 op = __shfl_xor_sync(kFull, bpos, o);
      const i32 ou = __shfl_xor_sync(kFull, bu, o);
      if (match_better(ow, od, op, bw, bd, bpos)) { bw = ow; bd = od; bpos = op; bu = ou; }
    }
    if (lane == 0) {
      s_w[wid] = bw;
      s_d[wid] = bd;
      s_p[wid] = bpos;
      s_u[wid] = bu;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int w = 1; w < (int)(blockDim.x >> 5); ++w)
        if (match_better(s_w[w], s_d[w], s_p[w], bw, bd, bpos)) { bw = s_w[w]; bd = s_d[w]; bpos = s_p[w]; bu = s_u[w]; }
      const i32 c = bw > 0 ? bu : v;
      cand[v] = c;
      uf.set(v, c);
    }
    __syncthreads();
  }
}

// Lanes per vertex by mean degree; defaults 2, 8, 16, 32.  Up to 6.5 entries a
// row two lanes do: a 12M road graph's match 397 us with four, now 278, a
// million-vertex mesh's 53, now 49.
i32 match_bucket(const DevGraph& g) {
  const double avg = g.n ? (double)g.m / g.n : 0.0;
  return avg <= 6.5 ? 0 : avg <= 14 ? 1 : avg <= 28 ? 2 : 3;
}

static void launch_match(Handle& h, const DevGraph& g, i32* cand, i32 G, i32* longlist, i32* longcnt,
                         UfStart uf = {}) {
  const int threads = 256;
  auto go = [&](auto kern) {
    const i64 tot = (i64)g.n * G;
    launch(kern, (u32)((tot + threads - 1) / threads), threads, 0, h.stream, g.n, g.xadj, g.adjncy, g.adjwgt,
           cand, longlist, longcnt, uf);
  };
  if (G == 2) go(k_match<2>);
  else if (G == 4) go(k_match<4>);
  else if (G == 8) go(k_match<8>);
  else if (G == 16) go(k_match<16>);
  else go(k_match<32>);
}

void time_match_variants(Handle& h, const DevGraph& g, i32* cand) {
  if (g.n == 0) return;
  const i32 b = match_bucket(g);
  cudaEvent_t e0, e1;
  GKW_CUDA(cudaEventCreate(&e0));
  GKW_CUDA(cudaEventCreate(&e1));
  Pool::Mark mk = h.scratch.mark();
  i32* longlist = h.scratch.alloc_n<i32>(g.n);
  i32* longcnt = h.scratch.alloc_n<i32>(1);
  const i32 lanes[kMatchLaneChoices] = {2, 4, 8, 16, 32};
  for (i32 q = 0; q < kMatchLaneChoices; ++q) {
    float best = 1e30f;
    for (int rep = 0; rep < 3; ++rep) {
      GKW_CUDA(cudaMemsetAsync(longcnt, 0, sizeof(i32), h.stream));
      GKW_CUDA(cudaEventRecord(e0, h.stream));
      launch_match(h, g, cand, lanes[q], longlist, longcnt);
      GKW_CUDA(cudaEventRecord(e1, h.stream));
      GKW_CUDA(cudaEventSynchronize(e1));
      float ms = 0;
      GKW_CUDA(cudaEventElapsedTime(&ms, e0, e1));
      best = std::min(best, ms);
    }
    h.tune_match_ms[b][q] += best;
  }
  h.scratch.release(mk);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
}

static void run_match_uf(Handle& h, const DevGraph& g, i32* cand, i64 maxdeg, UfStart uf) {
  if (g.n == 0) return;
  const bool split = maxdeg < 0 || maxdeg > kMatchLong;
  Pool::Mark mk = h.scratch.mark();
  i32* longlist = split ? h.scratch.alloc_n<i32>(g.n) : nullptr;
  i32* longcnt = split ? h.scratch.alloc_n<i32>(1) : nullptr;
  if (split) GKW_CUDA(cudaMemsetAsync(longcnt, 0, sizeof(i32), h.stream));
  launch_match(h, g, cand, h.tuning.match_lanes[match_bucket(g)], longlist, longcnt, uf);
  if (split)
    launch(k_match_long, (u32)h.sm_count * 2, kMatchLongThreads, 0, h.stream, g.xadj, g.adjncy, g.adjwgt, cand,
           (const i32*)longlist, (const i32*)longcnt, uf);
  GKW_CHECK_LAUNCH();
  h.scratch.release(mk);
}

void run_match(Handle& h, const DevGraph& g, i32* cand, i64 maxdeg) { run_match_uf(h, g, cand, maxdeg, UfStart{}); }

// ===========================================================================
// Union-find label propagation (coarsen.hpp:80-118, loop :461-469).  Under the
// Jacobi schedule a vertex ends with the largest id of its component of
// candidate edges and the round that brought it, which is its hop distance
// from that vertex; the loop ends with the first quiet round, one after the
// largest distance.  No rounds are run here:
//   hook      every vertex starts at the larger end of its edge; the edges to
//             smaller ends join their roots, the smaller root under the larger
//             (lock-free, compare-and-swap)
//   mark      a component has one cycle of candidates (a mutual pair, or a
//             longer one), so its root walks its candidates once round that
//             cycle and marks the distances of the vertices it meets: the
//             steps taken, and on the cycle the shorter way round
//   walk      every other vertex finds its root, and follows its candidates to
//             the first marked vertex: all its ways to the root lead there, so
//             its distance is the steps plus that mark
// All are chains of dependent loads per vertex that need no barrier between
// them, at full occupancy.  Raising labels round by round took a grid barrier
// and n atomics each (12M-vertex road graph, all levels: 2.66 ms, now 0.92; a
// million-vertex mesh 0.29 ms, now 0.20; the 27-point grid with its 57 rounds
// 0.54 ms, now 0.30).
// ===========================================================================
constexpr int kUfSmallThreads = 1024;
constexpr i32 kUfSmall = 16384;   // levels up to this run on one CTA, in shared memory

// Words that other threads of the launch write: from shared memory, or L2.
template <bool kShared, class T>
__device__ __forceinline__ T uf_ld(const T* p) { return kShared ? *(const volatile T*)p : __ldcg(p); }

template <bool kShared>
__device__ __forceinline__ i32 uf_find(i32* parent, i32 x) {   // parents only rise: ends at the root
  i32 p = uf_ld<kShared>(parent + x);
  while (p != x) {
    const i32 g = uf_ld<kShared>(parent + p);
    if (g != p) *(volatile i32*)(parent + x) = g;   // path halving; any ancestor is a valid parent
    x = p;
    p = g;
  }
  return x;
}

template <bool kShared>
__device__ __forceinline__ void uf_unite(i32* parent, i32 x, i32 y) {
  for (;;) {   // a failed swap means a root rose: ends
    x = uf_find<kShared>(parent, x);
    y = uf_find<kShared>(parent, y);
    if (x == y) return;
    const i32 lo = x < y ? x : y, hi = x < y ? y : x;
    const i32 old = atomicCAS(&parent[lo], lo, hi);
    if (old == lo) return;
    x = hi;
    y = old;
  }
}

// Root r marks the vertices on its walk (only this thread marks its component
// in this phase; the walk closes after at most the component's vertices).
template <bool kShared>
__device__ __forceinline__ void uf_mark_root(const i32* cand, u32* dist, i32 r) {
  i32 x = r;
  u32 i = 0;
  u32 k;   // distance of the vertex where the walk closes
  for (;;) {
    *(volatile u32*)(dist + x) = i;
    const i32 c = cand[x];
    k = uf_ld<kShared>(dist + c);
    if (k != kUfUnknown) {
      x = c;
      break;
    }
    x = c;
    ++i;
  }
  const u32 L = i + 1 - k;   // cycle length
  if (L <= 2) return;
  for (u32 j = 1; j < L; ++j) {
    x = cand[x];
    *(volatile u32*)(dist + x) = k + (j < L - j ? j : L - j);
  }
}

// Distance of v (see walk above); a vertex that another thread has finished
// by now ends the walk as well.
template <bool kShared>
__device__ __forceinline__ u32 uf_walk(const i32* cand, const u32* dist, i32 v) {
  u32 steps = 0;
  i32 x = v;
  for (;;) {
    const i32 c = cand[x];   // (issued beside the mark)
    const u32 d = uf_ld<kShared>(dist + x);
    if (d != kUfUnknown) return steps + d;
    x = c;
    ++steps;
  }
}

__device__ __forceinline__ void uf_max_rounds(u32 d, i32* rounds_out) {   // every thread of the CTA
  const u32 m = __reduce_max_sync(kFull, d);
  if ((threadIdx.x & 31) == 0 && (i32)m + 1 > *(volatile i32*)rounds_out) atomicMax(rounds_out, (i32)m + 1);
}

// One CTA, everything in shared memory (a 2048-vertex level 25 us, now 10).
__global__ void __launch_bounds__(kUfSmallThreads) k_uf_small(i32 n, const i32* __restrict__ cand_in,
                                                              u64* __restrict__ keys, i32* rounds_out) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  i32* parent = reinterpret_cast<i32*>(smem_raw);      // [n]
  u32* dist = reinterpret_cast<u32*>(parent + n);      // [n]
  i32* cand = reinterpret_cast<i32*>(dist + n);        // [n]
  __shared__ i32 s_rounds;
  const i32 T = (i32)blockDim.x;
  for (i32 v = threadIdx.x; v < n; v += T) {
    const i32 c = cand_in[v];
    cand[v] = c;
    parent[v] = c > v ? c : v;
    dist[v] = kUfUnknown;
  }
  if (threadIdx.x == 0) s_rounds = 0;
  __syncthreads();
  for (i32 v = n - 1 - (i32)threadIdx.x; v >= 0; v -= T)   // (largest first: see k_uf_hook)
    if (cand[v] < v) uf_unite<true>(parent, v, cand[v]);
  __syncthreads();
  for (i32 v = threadIdx.x; v < n; v += T)
    if (parent[v] == v) uf_mark_root<true>(cand, dist, v);
  __syncthreads();
  u32 m = 0;
  for (i32 v = threadIdx.x; v < n; v += T) {
    const u32 d = uf_walk<true>(cand, dist, v);
    *(volatile u32*)(dist + v) = d;
    m = d > m ? d : m;
    keys[v] = ((u64)(u32)uf_find<true>(parent, v) << 32) | d;
  }
  uf_max_rounds(m, &s_rounds);
  __syncthreads();
  if (threadIdx.x == 0) *rounds_out = s_rounds;
}

__global__ void k_uf_init(i32 n, const i32* __restrict__ cand, UfStart uf) {
  const i64 v = (i64)blockIdx.x * blockDim.x + threadIdx.x;
  if (v < n) uf.set((i32)v, cand[v]);
}

// Largest vertices first: a hub of small id then has its largest leaf as root
// at once, and every other leaf hangs itself under that, each on its own word;
// from the smallest up, every leaf raised the root that all of them share.
__global__ void k_uf_hook(i32 n, const i32* __restrict__ cand, i32* parent, i32* rounds_out) {
  const i64 v = (i64)n - 1 - ((i64)blockIdx.x * blockDim.x + threadIdx.x);
  if (v == 0) *rounds_out = 0;   // raised by the walk
  if (v < 0) return;
  const i32 c = cand[v];
  if (c < (i32)v) uf_unite<false>(parent, (i32)v, c);
}

__global__ void k_uf_mark(i32 n, const i32* __restrict__ cand, const i32* __restrict__ parent, u32* dist) {
  const i64 v = (i64)blockIdx.x * blockDim.x + threadIdx.x;
  if (v < n && parent[v] == (i32)v) uf_mark_root<false>(cand, dist, (i32)v);
}

// gsize (may be null): the members of each root are counted too, and each
// keeps the count it met as its slot.
__global__ void k_uf_walk(i32 n, const i32* __restrict__ cand, i32* parent, u32* dist, u64* __restrict__ keys,
                          i32* rounds_out, i32* __restrict__ gsize, i32* __restrict__ slot) {
  const i64 v = (i64)blockIdx.x * blockDim.x + threadIdx.x;
  u32 d = 0;
  if (v < n) {
    const i32 r = uf_find<false>(parent, (i32)v);
    d = uf_walk<false>(cand, dist, (i32)v);
    *(volatile u32*)(dist + v) = d;
    keys[v] = ((u64)(u32)r << 32) | d;
    if (gsize) slot[v] = atomicAdd(&gsize[r], 1);
  }
  uf_max_rounds(d, rounds_out);
}

// Writes the final keys to keys_out and the reference's round-launch count
// to *d_rounds (device).  No host synchronisation.
void run_union_find(Handle& h, i32 n, const i32* cand, u64* keys_out, i32* d_rounds) {
  if (n == 0) {
    const i32 one = 1;
    GKW_CUDA(cudaMemcpyAsync(d_rounds, &one, sizeof(i32), cudaMemcpyHostToDevice, h.stream));
    return;
  }
  if (n <= kUfSmall) {
    if (!h.capturing)
      GKW_CUDA(cudaFuncSetAttribute(k_uf_small, cudaFuncAttributeMaxDynamicSharedMemorySize, kUfSmall * 12));
    launch(k_uf_small, 1, kUfSmallThreads, (size_t)n * 12, h.stream, n, cand, keys_out, d_rounds);
    GKW_CHECK_LAUNCH();
    return;
  }
  Pool::Mark mk = h.scratch.mark();
  const u32 nb = ceil_div(n, 256);
  i32* parent = h.scratch.alloc_n<i32>(n);
  u32* dist = h.scratch.alloc_n<u32>(n);
  UfStart uf;
  uf.parent = parent;
  uf.dist = dist;
  launch(k_uf_init, nb, 256, 0, h.stream, n, cand, uf);
  launch(k_uf_hook, nb, 256, 0, h.stream, n, cand, parent, d_rounds);
  launch(k_uf_mark, nb, 256, 0, h.stream, n, cand, (const i32*)parent, dist);
  launch(k_uf_walk, nb, 256, 0, h.stream, n, cand, parent, dist, keys_out, d_rounds, (i32*)nullptr,
         (i32*)nullptr);
  GKW_CHECK_LAUNCH();
  h.scratch.release(mk);
}

// ===========================================================================
// Coarse ids (coarsen.hpp:351-421, 120-155, 474-481).  Sorted order is
// (root, dist, id); each root's run is cut into chunks of group_cap.  A
// group of size s gets ceil(s/cap) consecutive coarse ids starting at the
// exclusive scan of chunk counts over roots in id order.  Groups larger than
// the cap need the rank of each member in (dist, id) order: a warp sorts
// groups of <= 32 members in registers, a CTA sorts groups up to
// kGroupSmem members in shared memory, and bigger groups are sorted by a
// global bitonic network.
// ===========================================================================
constexpr i32 kGroupSmem = 4096;

__global__ void k_group_count(i32 n, const u64* __restrict__ keys, i32* __restrict__ gsize, i32* __restrict__ slot) {
  const i64 v = (i64)blockIdx.x * blockDim.x + threadIdx.x;
  if (v < n) slot[v] = atomicAdd(&gsize[(u32)(keys[v] >> 32)], 1);
}

// The contraction's sums and member lists, taken as each coarse id is known
// (null memtab: not wanted).  A vertex brings its place in the coarse vertex's
// list, so one 64-bit atomic without a result, weight << 32 | row length, is
// all the members share (lengths add up to at most m < 2^31: no carry).
struct Accum {
  const i32 *xadj = nullptr, *vwgt = nullptr;
  u64* sums = nullptr;
  i32 *mcnt = nullptr, *memtab = nullptr;
  // place < cap of `members` in coarse vertex c
  __device__ __forceinline__ void add(i32 v, i32 c, i32 cap, i32 place, i32 members) const {
    const u32 len = (u32)(xadj[v + 1] - xadj[v]);
    atomicAdd(reinterpret_cast<unsigned long long*>(sums + c), (unsigned long long)(u32)vwgt[v] << 32 | len);
    memtab[(i64)c * cap + place] = v;
    if (place == 0) mcnt[c] = members;
  }
  // member `rank` of a group of s whose first coarse id is base
  __device__ __forceinline__ i32 add_ranked(i32 v, i32 base, i32 rank, i32 s, i32 cap) const {
    const i32 q = rank / cap, c = base + q;
    if (memtab) add(v, c, cap, rank - q * cap, min(cap, s - q * cap));
    return c;
  }
};

// Giants' list in the middle of the one list array: groups of more than cap
// members are at most n / 2, from the front those of up to 32, from the back
// those sorted by a CTA (at most n / 33).
__device__ __forceinline__ i32 giant_list_at(i32 n) { return n / 2 + 1; }

// counts[]: [0] groups of 7..32 members (warp sort), [1] groups above kGroupSmem
// (global sort), [2] n_c, [3] members of big groups, [4] groups of
// 33..kGroupSmem members (CTA sort)
// grec: (size, first coarse id) by root, one gather a vertex
__global__ void k_group_scatter(i32 n, const u64* __restrict__ keys, const int2* __restrict__ grec,
                                const i32* __restrict__ goff,
                                const i32* __restrict__ slot, i32 cap, i32* __restrict__ cmap,
                                i32* __restrict__ members, i32* __restrict__ list, i32* __restrict__ counts,
                                Accum acc, ArenaHdr* arena, CoopState* coop) {
  const i64 v = (i64)blockIdx.x * blockDim.x + threadIdx.x;
  if (v == 0 && arena) {   // for the row kernels
    arena->used = 0;
    arena->need = 0;
    arena->overflow = 0;
    coop->max_cvw = 0;
    coop->maxdeg = 0;
  }
  if (v >= n) return;
  const i32 r = (i32)(u32)(keys[v] >> 32);
  const int2 rec = grec[r];
  const i32 s = rec.x;
  if (s <= cap) {
    const i32 c = rec.y;
    cmap[v] = c;
    if (acc.memtab) acc.add((i32)v, c, cap, slot[v], s);
  } else {
    members[goff[r] + slot[v]] = (i32)v;
    if (r == (i32)v) {
      if (s <= 32) list[atomicAdd(&counts[0], 1)] = r;
      else if (s <= kGroupSmem) list[n - 1 - atomicAdd(&counts[4], 1)] = r;
      else list[giant_list_at(n) + atomicAdd(&counts[1], 1)] = r;
    }
  }
}

__device__ __forceinline__ u64 umin64(u64 a, u64 b) { return a < b ? a : b; }
__device__ __forceinline__ u64 umax64(u64 a, u64 b) { return a < b ? b : a; }

// one warp per big group with <= 32 members (CTAs [0, nblocks) of the launch)
__device__ void group_sort_warps(const i32* __restrict__ biglist, const i32* __restrict__ counts,
                                 const u64* __restrict__ keys, const int2* __restrict__ grec,
                                 const i32* __restrict__ goff,
                                 const i32* __restrict__ members, i32 cap, i32* __restrict__ cmap, u32 nblocks,
                                 const Accum& acc) {
  const i32 nbig = counts[0];
  const int lane = threadIdx.x & 31;
  const i64 warp0 = ((i64)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const i64 nwarps = ((i64)nblocks * blockDim.x) >> 5;
  for (i64 w = warp0; w < nbig; w += nwarps) {
    const i32 r = biglist[w];
    const i32 s = grec[r].x;
    if (s > 32) continue;   // warp-uniform
    u64 key = ~0ull;
    if (lane < s) {
      const i32 m = members[goff[r] + lane];
      key = ((keys[m] & 0xffffffffull) << 32) | (u32)m;   // (dist, id)
    }
#pragma unroll
    for (int kk = 2; kk <= 32; kk <<= 1) {
#pragma unroll
      for (int j = kk >> 1; j > 0; j >>= 1) {
        const u64 o = __shfl_xor_sync(kFull, key, j);
        const bool up = (lane & kk) == 0;
        const bool lower = (lane & j) == 0;
        key = (lower == up) ? umin64(key, o) : umax64(key, o);
      }
    }
    if (lane < s) cmap[(u32)key] = acc.add_ranked((i32)(u32)key, grec[r].y, lane, s, cap);
  }
}

// Ascending bitonic sort of a[0..P) (P a power of two) by one CTA.
__device__ void cta_bitonic_u64(u64* a, i32 P) {
  for (i32 kk = 2; kk <= P; kk <<= 1) {
    for (i32 j = kk >> 1; j > 0; j >>= 1) {
      for (i32 i = threadIdx.x; i < P; i += blockDim.x) {
        const i32 l = i ^ j;
        if (l > i) {
          const u64 x = a[i], y = a[l];
          const bool up = (i & kk) == 0;
          if (up ? (x > y) : (x < y)) { a[i] = y; a[l] = x; }
        }
      }
      __syncthreads();
    }
  }
}

// one CTA per big group with 33..kGroupSmem members (CTA `cta` of `nctas`);
// listed from the end of the list backwards
__device__ void group_sort_ctas(const i32* __restrict__ list_last, const i32* __restrict__ counts,
                                const u64* __restrict__ keys, const int2* __restrict__ grec,
                                const i32* __restrict__ goff,
                                const i32* __restrict__ members, i32 cap, i32* __restrict__ cmap, u32 cta,
                                u32 nctas, const Accum& acc) {
  __shared__ u64 sk[kGroupSmem];
  const i32 nbig = counts[4];
  for (i32 b = (i32)cta; b < nbig; b += (i32)nctas) {
    const i32 r = list_last[-b];
    const i32 s = grec[r].x;
    i32 P = 64;
    while (P < s) P <<= 1;
    for (i32 i = threadIdx.x; i < P; i += blockDim.x) {
      u64 key = ~0ull;
      if (i < s) {
        const i32 m = members[goff[r] + i];
        key = ((keys[m] & 0xffffffffull) << 32) | (u32)m;
      }
      sk[i] = key;
    }
    __syncthreads();
    cta_bitonic_u64(sk, P);
    for (i32 i = threadIdx.x; i < s; i += blockDim.x)
      cmap[(u32)sk[i]] = acc.add_ranked((i32)(u32)sk[i], grec[r].y, i, s, cap);
    __syncthreads();
  }
}

// The group orders of one level in one launch: CTAs [0, nwarp_blocks) sort
// the groups of up to 32 members by warps, the CTAs after them the groups of
// up to kGroupSmem members, one CTA each.
__global__ void k_group_sort(const i32* __restrict__ list, i32 n, const i32* __restrict__ counts,
                             const u64* __restrict__ keys, const int2* __restrict__ grec,
                             const i32* __restrict__ goff,
                             const i32* __restrict__ members, i32 cap, i32* __restrict__ cmap, u32 nwarp_blocks,
                             Accum acc) {
  if (blockIdx.x < nwarp_blocks)
    group_sort_warps(list, counts, keys, grec, goff, members, cap, cmap, nwarp_blocks, acc);
  else
    group_sort_ctas(list + n - 1, counts, keys, grec, goff, members, cap, cmap, blockIdx.x - nwarp_blocks,
                    gridDim.x - nwarp_blocks, acc);
}

// Giant groups (more than kGroupSmem members, rare): every CTA of one
// cooperative launch sorts each giant group in turn with a bitonic network in
// global scratch, grid barriers between the stages.
__global__ void __launch_bounds__(512) k_giant_sort(const i32* __restrict__ giantlist, const i32* __restrict__ counts,
                                                    const u64* __restrict__ keys, const int2* __restrict__ grec,
                                                    const i32* __restrict__ goff,
                                                    const i32* __restrict__ members, i32 cap, i32* __restrict__ cmap,
                                                    u64* a, GridBarrier* bar, i32* err, Accum acc) {
  __shared__ i32 s_flag;
  const i32 ng = counts[1];
  if (ng == 0) return;   // uniform: no barrier is entered
  const i64 stride = (i64)gridDim.x * blockDim.x;
  const i64 t0 = (i64)blockIdx.x * blockDim.x + threadIdx.x;
  for (i32 gi = 0; gi < ng; ++gi) {
    const i32 r = giantlist[gi];
    const i32 s = grec[r].x;
    i64 P = 1;
    while (P < s) P <<= 1;
    const i32* mem = members + goff[r];
    for (i64 i = t0; i < P; i += stride) {
      u64 key = ~0ull;
      if (i < s) {
        const i32 m = mem[i];
        key = ((keys[m] & 0xffffffffull) << 32) | (u32)m;
      }
      a[i] = key;
    }
    if (!grid_barrier(bar, err, &s_flag)) return;
    for (i64 kk = 2; kk <= P; kk <<= 1) {
      for (i64 j = kk >> 1; j > 0; j >>= 1) {
        for (i64 i = t0; i < P; i += stride) {
          const i64 l = i ^ j;
          if (l > i) {
            const u64 x = ldcg(a + i), y = ldcg(a + l);
            const bool up = (i & kk) == 0;
            if (up ? (x > y) : (x < y)) { a[i] = y; a[l] = x; }
          }
        }
        if (!grid_barrier(bar, err, &s_flag)) return;
      }
    }
    const i32 base = grec[r].y;
    for (i64 i = t0; i < s; i += stride) {
      const i32 m = (i32)(u32)ldcg(a + i);
      cmap[m] = acc.add_ranked(m, base, (i32)i, s, cap);
    }
    if (!grid_barrier(bar, err, &s_flag)) return;
  }
}

// Group sizes and counters (cleared together) and the rest of the tables.
struct GroupTables {
  i32 *gsize, *counts;
  size_t cleared;   // words from gsize
  i32* slot;        // the caller's: its place among its root's members, by vertex
  int2* grec;
  i32 *goff, *members, *list;
};

static GroupTables group_tables(Handle& h, i32 n) {
  GroupTables t;
  const size_t nz = ((size_t)n + 63) & ~(size_t)63;
  t.cleared = nz + 8;
  t.gsize = h.scratch.alloc_n<i32>(t.cleared);
  t.counts = t.gsize + nz;
  t.grec = h.scratch.alloc_n<int2>(n);
  t.goff = h.scratch.alloc_n<i32>(n);
  t.members = h.scratch.alloc_n<i32>(n);
  t.list = h.scratch.alloc_n<i32>((size_t)n + 1);
  return t;
}

// cmap for every vertex and *d_nc = n_c (device) from the group sizes, with
// the contraction's sums and member lists if acc has them.  gscratch: 2n
// words of 64 bits.
static void run_groups(Handle& h, i32 n, const u64* keys, i32 cap, const GroupTables& t, u64* gscratch, i32* cmap,
                       i32* d_nc, const Accum& acc) {
  scan_group_chunks(h, t.gsize, t.grec, t.goff, t.counts + 3, n, cap, d_nc);
  launch(k_group_scatter, ceil_div(n, 256), 256, 0, h.stream, n, keys, t.grec, t.goff, t.slot, cap, cmap,
         t.members, t.list, t.counts, acc, acc.memtab ? h.arena : (ArenaHdr*)nullptr, h.coop);
  const u32 ng = std::max<u32>(1, std::min<u32>(ceil_div(n, 8 * 32), (u32)h.sm_count * 16));
  launch(k_group_sort, ng + (u32)h.sm_count * 2, 256, 0, h.stream, t.list, n, t.counts, keys, t.grec, t.goff,
         t.members, cap, cmap, ng, acc);
  GKW_CHECK_LAUNCH();
  if (n <= kGroupSmem) return;
  const i32* gl = t.list + (n / 2 + 1);   // giant_list_at
  const i32* cn = t.counts;
  const int2* gs = t.grec;
  const i32* go = t.goff;
  const i32* mb = t.members;
  i32 capv = cap;
  GridBarrier* barp = &h.coop->bar;
  i32* errp = &h.coop->err;
  Accum ac = acc;
  void* args[] = {&gl, &cn, (void*)&keys, &gs, &go, &mb, &capv, &cmap, &gscratch, &barp, &errp, &ac};
  const i32 grid = coop_grid(h, (const void*)k_giant_sort, h.sm_count, 512, 0);
  launch_coop(h, (const void*)k_giant_sort, grid, 512, 0, args);
}

// The group map alone.  No host synchronisation.
void run_group_map(Handle& h, i32 n, const u64* keys, i32 cap, i32* cmap, i32* d_nc) {
  GKW_REQUIRE(cap >= 1, GKW_E_INVALID, "group_cap must be >= 1");
  if (n == 0) {
    GKW_CUDA(cudaMemsetAsync(d_nc, 0, sizeof(i32), h.stream));
    return;
  }
  Pool::Mark mk = h.scratch.mark();
  GroupTables t = group_tables(h, n);
  t.slot = h.scratch.alloc_n<i32>(n);
  u64* gscratch = h.scratch.alloc_n<u64>(2 * (size_t)n);
  GKW_CUDA(cudaMemsetAsync(t.gsize, 0, sizeof(i32) * t.cleared, h.stream));
  launch(k_group_count, ceil_div(n, 256), 256, 0, h.stream, n, keys, t.gsize, t.slot);
  run_groups(h, n, keys, cap, t, gscratch, cmap, d_nc, Accum{});
  h.scratch.release(mk);
}

// ===========================================================================
// Small levels: from the candidates to the contraction's member lists in one
// launch of one CTA with every table in shared memory -- union-find, group
// sizes, coarse ids, group orders, member lists, row-length bounds and their
// scan, the arrays and counters that the row kernels expect cleared.  The
// separate kernels take thirteen launches and nine clears for this, and on a
// level of a few thousand vertices each is mostly its launch: the phases here
// are a chain of shared-memory latencies with a barrier between them.
// Two levels of a 2048-vertex mesh with k = 8: 186 us with the separate
// launches, now 134 with the rows and the host's read; a 100k mesh's small
// levels together 45 us less, a 30k circuit's 55.
// Per vertex 16 bytes: A parent, then group size | member block << 16, then
// row length; D distance, then coarse base | members placed << 16, then
// members; C candidate, then root << 16 | distance, then kPlaced | coarse id;
// K member keys distance << 16 | id of the groups above the cap, then weight.
// ===========================================================================
constexpr int kSmallThreads = 1024;
constexpr i32 kSmallLevel = 14336;             // 16 bytes each: 224 KB
constexpr i32 kSmallWarpSort = 1024;           // larger groups are sorted by the whole CTA
constexpr u32 kPlaced = 0xffff0000u;
static_assert(kSmallLevel * 16 <= 227 * 1024 - 1024 && kSmallLevel < (1 << 15), "two 16-bit fields a word");

// Ascending sort of a[0..s) in shared memory by lanes [lane0, lane0 + L) of
// the group that `barrier` waits for.  Every comparison puts the smaller key
// first, so positions from s to the next power of two act as largest keys
// that never move and need no storage.
template <class Barrier>
__device__ __forceinline__ void sort_in_place(u32* a, i32 s, i32 t, i32 L, Barrier barrier) {
  i32 P = 2;
  while (P < s) P <<= 1;
  for (i32 kk = 2; kk <= P; kk <<= 1) {
    for (i32 j = kk >> 1; j > 0; j >>= 1) {
      const bool mirror = 2 * j == kk;   // the first step of a merge pairs i with its mirror in the block
      for (i32 q = t; q < P / 2; q += L) {
        const i32 i = 2 * (q & ~(j - 1)) | (q & (j - 1));
        const i32 l = mirror ? (i ^ (kk - 1)) : (i | j);
        if (l < s) {
          const u32 x = a[i], y = a[l];
          if (x > y) {
            a[i] = y;
            a[l] = x;
          }
        }
      }
      barrier();
    }
  }
}

// Exclusive scan of x[0..n) (0 <= i < n) by the CTA: each warp a contiguous
// segment, `value(i)` a word, `store(i, exclusive, value)`; returns the total.
// s_warp has one word per warp.  Starts and ends with a barrier.
template <class Value, class Store>
__device__ __forceinline__ u32 scan_segments(i32 n, u32* s_warp, Value value, Store store) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const i32 seg = (((n + warps - 1) / warps) + 31) & ~31;
  const i32 b = warp * seg < n ? warp * seg : n, e = b + seg < n ? b + seg : n;
  __syncthreads();
  u32 sum = 0;
  for (i32 i = b + lane; i < e; i += 32) sum += value(i);
  sum = __reduce_add_sync(kFull, sum);
  if (lane == 0) s_warp[warp] = sum;
  __syncthreads();
  u32 w = lane < warps ? s_warp[lane] : 0;
  const u32 total = __reduce_add_sync(kFull, w);
  u32 run = __reduce_add_sync(kFull, lane < warp ? w : 0);
  for (i32 i0 = b; i0 < e; i0 += 32) {
    const i32 i = i0 + lane;
    const u32 x = i < e ? value(i) : 0;
    u32 inc = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const u32 y = __shfl_up_sync(kFull, inc, o);
      if (lane >= o) inc += y;
    }
    if (i < e) store(i, run + inc - x, x);
    run += __shfl_sync(kFull, inc, 31);
  }
  __syncthreads();
  return total;
}

struct SmallLevel {
  i32 n, cap;
  const i32* cand;
  const i32 *xadj, *vwgt;
  i32 *cmap, *cvwgt, *rowlen, *ub, *mcnt, *memtab, *cnt, *misc;
  ArenaHdr* arena;
  i32 *nc, *uf_rounds, *max_cvw, *maxdeg;
};

__global__ void __launch_bounds__(kSmallThreads) k_group_small(SmallLevel a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ u32 s_warp[kSmallThreads / 32];
  __shared__ i32 s_rounds;
  const i32 n = a.n, cap = a.cap, T = (i32)blockDim.x, t = (i32)threadIdx.x;
  const int lane = threadIdx.x & 31;
  u32* A = reinterpret_cast<u32*>(smem_raw);
  u32* D = A + n;
  u32* C = D + n;
  u32* K = C + n;
  i32* parent = reinterpret_cast<i32*>(A);
  i32* cand = reinterpret_cast<i32*>(C);
  for (i32 v = t; v < n; v += T) {
    const i32 c = a.cand[v];
    cand[v] = c;
    parent[v] = c > v ? c : v;
    D[v] = kUfUnknown;
  }
  if (t == 0) s_rounds = 0;
  if (t < 8) a.misc[t] = 0;
  if (t == 0) {
    a.arena->used = 0;
    a.arena->need = 0;
    a.arena->overflow = 0;
    *a.max_cvw = 0;
    *a.maxdeg = 0;
  }
  __syncthreads();
  for (i32 v = n - 1 - t; v >= 0; v -= T)   // (largest first: see k_uf_hook)
    if (cand[v] < v) uf_unite<true>(parent, v, cand[v]);
  __syncthreads();
  for (i32 v = t; v < n; v += T)
    if (parent[v] == v) uf_mark_root<true>(cand, D, v);
  __syncthreads();
  u32 far = 0;
  for (i32 v = t; v < n; v += T) {
    const u32 d = uf_walk<true>(cand, D, v);
    *(volatile u32*)(D + v) = d;
    far = d > far ? d : far;
  }
  uf_max_rounds(far, &s_rounds);
  __syncthreads();
  for (i32 v = t; v < n; v += T) C[v] = ((u32)uf_find<true>(parent, v) << 16) | D[v];
  __syncthreads();
  for (i32 v = t; v < n; v += T) A[v] = 0;
  __syncthreads();
  for (i32 v = t; v < n; v += T) atomicAdd(&A[C[v] >> 16], 1u);
  // coarse ids in root order, and the member blocks of the groups above the cap
  const u32 sums = scan_segments(
      n, s_warp,
      [&](i32 v) {
        const u32 s = A[v] & 0xffffu;
        return (s + (u32)cap - 1) / (u32)cap | (s > (u32)cap ? s << 16 : 0u);
      },
      [&](i32 v, u32 before, u32) {
        D[v] = before & 0xffffu;
        A[v] |= before & 0xffff0000u;
      });
  const i32 nc = (i32)(sums & 0xffffu);
  for (i32 v = t; v < n; v += T) {
    const u32 key = C[v], r = key >> 16, sz = A[r];
    if ((sz & 0xffffu) <= (u32)cap) {
      C[v] = kPlaced | (D[r] & 0xffffu);
    } else {
      const u32 slot = atomicAdd(&D[r], 1u << 16) >> 16;
      K[(sz >> 16) + slot] = (key << 16) | (u32)v;
    }
  }
  __syncthreads();
  if (sums >> 16) {   // groups above the cap: members in (distance, id) order
    bool large = false;
    for (i32 v0 = t - lane; v0 < n; v0 += T) {
      const i32 v = v0 + lane;
      const u32 s = v < n && C[v] >> 16 == (u32)v ? A[v] & 0xffffu : 0;
      large |= s > (u32)kSmallWarpSort;
      u32 todo = __ballot_sync(kFull, s > 0 && s <= (u32)kSmallWarpSort);   // (placed vertices are no roots)
      while (todo) {
        const int q = __ffs(todo) - 1;
        todo &= todo - 1;
        const u32 w = A[v0 + q], base = D[v0 + q] & 0xffffu;
        const i32 m = (i32)(w & 0xffffu);
        u32* k = K + (w >> 16);
        __syncwarp();
        if (m <= 32) {
          u32 key = lane < m ? k[lane] : ~0u;
#pragma unroll
          for (int kk = 2; kk <= 32; kk <<= 1) {
#pragma unroll
            for (int j = kk >> 1; j > 0; j >>= 1) {
              const u32 o = __shfl_xor_sync(kFull, key, j);
              const bool low = ((lane & kk) == 0) == ((lane & j) == 0);
              key = low ? min(key, o) : max(key, o);
            }
          }
          if (lane < m) C[key & 0xffffu] = kPlaced | (base + (u32)(lane / cap));
        } else {
          sort_in_place(k, m, lane, 32, [] { __syncwarp(); });
          for (i32 i = lane; i < m; i += 32) C[k[i] & 0xffffu] = kPlaced | (base + (u32)(i / cap));
        }
        __syncwarp();
      }
    }
    const bool any = __syncthreads_or(large);
    for (i32 v0 = 0; any && v0 < n; v0 += T) {   // at most n / kSmallWarpSort groups
      const i32 v = v0 + t;
      const bool big = v < n && C[v] >> 16 == (u32)v;
      while (true) {
        const i32 mine = big && C[v] >> 16 == (u32)v ? v : -1;
        if (t == 0) s_warp[0] = 0;
        __syncthreads();
        if (mine >= 0) atomicMax(&s_warp[0], (u32)mine + 1u);
        __syncthreads();
        const i32 r = (i32)s_warp[0] - 1;
        __syncthreads();
        if (r < 0) break;
        const u32 w = A[r], base = D[r] & 0xffffu;
        const i32 m = (i32)(w & 0xffffu);
        u32* k = K + (w >> 16);
        sort_in_place(k, m, t, T, [] { __syncthreads(); });
        for (i32 i = t; i < m; i += T) C[k[i] & 0xffffu] = kPlaced | (base + (u32)(i / cap));
        __syncthreads();
      }
    }
  }
  // member lists, row-length bounds and weights of the coarse vertices
  for (i32 c = t; c < nc; c += T) A[c] = D[c] = K[c] = 0;
  __syncthreads();
#pragma unroll 4
  for (i32 v = t; v < n; v += T) {
    const u32 c = C[v] & 0xffffu;
    const i32 len = __ldg(a.xadj + v + 1) - __ldg(a.xadj + v);
    const u32 w = (u32)__ldg(a.vwgt + v);
    a.cmap[v] = (i32)c;
    atomicAdd(&A[c], (u32)len);
    atomicAdd(&K[c], w);
    a.memtab[(i64)c * cap + (i32)atomicAdd(&D[c], 1u)] = v;
  }
  scan_segments(
      nc, s_warp, [&](i32 c) { return A[c]; },
      [&](i32 c, u32 before, u32 len) {
        a.rowlen[c] = (i32)len;
        a.ub[c] = (i32)before;
        a.mcnt[c] = (i32)D[c];
        a.cvwgt[c] = (i32)K[c];
      });
  for (i32 c = t; c <= n; c += T) a.cnt[c] = 0;   // rows from n_c on are empty
  if (t == 0) {
    *a.nc = nc;
    *a.uf_rounds = s_rounds;
  }
}

// ===========================================================================
// Contraction (coarsen.hpp:157-349).  Members of each coarse vertex are
// listed (at most group_cap of them); then one warp per coarse vertex hashes
// the mapped neighbour ids of all its members into shared memory, summing
// weights, drops the self id, sorts the distinct ids and writes the row to a
// staging area at an upper-bound offset; a scan of the row lengths gives the
// coarse xadj and a copy compacts the rows.  Rows longer than the warp's
// table go to a CTA with a larger shared table, and rows longer than that to
// a CTA with a table in global scratch.
// ===========================================================================
__global__ void k_coarse_accum(i32 n, const i32* __restrict__ xadj, const i32* __restrict__ vwgt,
                               const i32* __restrict__ cmap, i32 cap, i32* __restrict__ cvwgt,
                               i32* __restrict__ rowlen, i32* __restrict__ mcnt, i32* __restrict__ memtab,
                               ArenaHdr* arena, CoopState* coop) {
  const i64 v = (i64)blockIdx.x * blockDim.x + threadIdx.x;
  if (v == 0) {
    if (arena) {
      arena->used = 0;
      arena->need = 0;
      arena->overflow = 0;
    }
    coop->max_cvw = 0;
    coop->maxdeg = 0;
  }
  if (v >= n) return;
  const i32 c = cmap[v];
  atomicAdd((u32*)&cvwgt[c], (u32)vwgt[v]);
  atomicAdd(&rowlen[c], xadj[v + 1] - xadj[v]);
  const i32 slot = atomicAdd(&mcnt[c], 1);
  memtab[(i64)c * cap + slot] = (i32)v;
}

__device__ __forceinline__ u32 hash_u32(u32 x) {
  x ^= x >> 16;
  x *= 0x7feb352du;
  x ^= x >> 15;
  x *= 0x846ca68bu;
  x ^= x >> 16;
  return x;
}

static constexpr u32 kEmpty = 0xffffffffu;

// Slots of a table for a row of L entries: a power of two of at least twice
// that, 2^31 at most.  (A row of more than 2^30 entries has far fewer distinct
// ids, one per coarse vertex; doubling on for it would pass 2^32 to zero and
// never end.)
__host__ __device__ u32 table_slots(u32 L) {
  u32 s = 64;
  while (s < 0x80000000u && s < 2 * (u64)L) s <<= 1;
  return s;
}

// Insert (key, w) into an open-addressing table of size hsz (power of two).
// The table always has free slots (hsz >= 2 * entries), so the probe ends;
// the probe count is still bounded by hsz.
__device__ __forceinline__ void table_add(u32* keys, u32* vals, u32 hsz, u32 key, u32 w) {
  u32 s = hash_u32(key) & (hsz - 1);
  for (u32 probe = 0; probe < hsz; ++probe) {
    const u32 prev = atomicCAS(&keys[s], kEmpty, key);
    if (prev == kEmpty || prev == key) {
      atomicAdd(&vals[s], w);
      return;
    }
    s = (s + 1) & (hsz - 1);
  }
}

template <int WCAP>
struct WarpTable {
  u32 keys[2 * WCAP];
  u32 vals[2 * WCAP];
  u64 out[WCAP];
};

// Warp-level ascending bitonic sort of a[0..P) in shared memory, P power of 2 >= 32.
__device__ void warp_bitonic_u64(u64* a, i32 P, int lane) {
  for (i32 kk = 2; kk <= P; kk <<= 1) {
    for (i32 j = kk >> 1; j > 0; j >>= 1) {
      for (i32 i = lane; i < P; i += 32) {
        const i32 l = i ^ j;
        if (l > i) {
          const u64 x = a[i], y = a[l];
          const bool up = (i & kk) == 0;
          if (up ? (x > y) : (x < y)) { a[i] = y; a[l] = x; }
        }
      }
      __syncwarp();
    }
  }
}

// Merge of one coarse row whose kept entries lie one per lane in a group of G
// lanes: `key` the coarse id (kEmpty: none), w the weight.  The group sorts
// (id, lane) -- 32 bits while ids stay below 2^(32 - log2 G), else 64 -- sums
// each run of equal ids (mod 2^32) and writes the distinct ids in order at o;
// returns their number.  Whole warps call it together.
template <int G, class K>
__device__ __forceinline__ i32 merge_lanes(u32 key, u32 w, i32 o, i32* __restrict__ sadj, i32* __restrict__ swgt) {
  constexpr int kBits = G == 32 ? 5 : G == 16 ? 4 : 3;
  const int lane = threadIdx.x & 31, sub = lane & (G - 1), g0 = lane & ~(G - 1);
  K x = key == kEmpty ? ~(K)0 : ((K)key << kBits) | (K)sub;
#pragma unroll
  for (int kk = 2; kk <= G; kk <<= 1) {
#pragma unroll
    for (int jj = kk >> 1; jj > 0; jj >>= 1) {
      const K y = __shfl_xor_sync(kFull, x, jj, G);
      const bool keep_min = ((sub & kk) == 0) == ((sub & jj) == 0);
      x = keep_min ? (x < y ? x : y) : (x < y ? y : x);
    }
  }
  const bool on = x != ~(K)0;
  const u32 id = on ? (u32)(x >> kBits) : kEmpty;
  const u32 ww = __shfl_sync(kFull, w, (int)(x & (K)(G - 1)), G);
  const u32 prev = __shfl_up_sync(kFull, id, 1, G), next = __shfl_down_sync(kFull, id, 1, G);
  const bool head = sub == 0 || prev != id;
  const bool last = on && (sub == G - 1 || next != id);
  u32 S = on ? ww : 0u;   // inclusive prefix sum (mod 2^32)
#pragma unroll
  for (int d = 1; d < G; d <<= 1) {
    const u32 y = __shfl_up_sync(kFull, S, d, G);
    if (sub >= d) S += y;
  }
  const u32 gmask = G == 32 ? kFull : ((1u << G) - 1u);
  const u32 heads = (__ballot_sync(kFull, head) >> g0) & gmask;
  const u32 lasts = (__ballot_sync(kFull, last) >> g0) & gmask;
  const int start = 31 - __clz(heads & (0xffffffffu >> (31 - sub)));   // first lane of this lane's run
  const u32 before = __shfl_sync(kFull, S, start > 0 ? start - 1 : 0, G);
  if (last) {
    const i32 at = o + __popc(lasts & ((1u << sub) - 1u));
    sadj[at] = (i32)id;
    swgt[at] = (i32)(S - (start > 0 ? before : 0u));
  }
  return __popc(lasts);
}

// Rows of short levels (a road graph's coarse rows have about 7 entries): 16
// lanes per coarse vertex, two rows a warp.  Rows that do not fit are listed
// for k_contract_warp.
constexpr int kContractG = 16;
template <class K>
__global__ void __launch_bounds__(256) k_contract_short(
    const i32* __restrict__ ncp, const i32* __restrict__ xadj, const i32* __restrict__ adjncy,
    const i32* __restrict__ adjwgt, const i32* __restrict__ cmap, const i32* __restrict__ memtab,
    const i32* __restrict__ mcnt, i32 cap, const i32* __restrict__ rowlen, const i32* __restrict__ ub,
    i32* __restrict__ sadj, i32* __restrict__ swgt, i32* __restrict__ cnt, i32* __restrict__ mid,
    i32* __restrict__ nmid) {
  constexpr int G = kContractG;
  const int lane = threadIdx.x & 31, sub = lane & (G - 1);
  const i32 nc = *ncp;
  const i64 ng = ((i64)gridDim.x * blockDim.x) / G;
  for (i64 c0 = ((i64)blockIdx.x * blockDim.x + (threadIdx.x & ~31)) / G; c0 < nc; c0 += ng) {   // warp-uniform
    const i64 c = c0 + lane / G;
    const bool on = c < nc;
    const i32 L = on ? rowlen[c] : 0, nm = on ? mcnt[c] : 0, o = on ? ub[c] : 0;
    const bool fits = L <= G && nm <= G;
    i32 mbeg = 0, mlen = 0;
    if (fits && sub < nm) {
      const i32 mv = memtab[c * cap + sub];
      mbeg = xadj[mv];
      mlen = xadj[mv + 1] - mbeg;
    }
    i32 incl = mlen;
#pragma unroll
    for (int d = 1; d < G; d <<= 1) {
      const i32 y = __shfl_up_sync(kFull, incl, d, G);
      if (sub >= d) incl += y;
    }
    const i32 shift = mbeg - (incl - mlen);
    i32 jm = 0;   // members whose rows end at or before this lane's entry
    const i32 nmx = (i32)__reduce_max_sync(kFull, (u32)(fits ? nm : 0));
    for (i32 j = 0; j < nmx; ++j) jm += sub >= __shfl_sync(kFull, incl, j, G) && j < nm;
    const i32 pos = __shfl_sync(kFull, shift, jm & (G - 1), G) + sub;
    u32 key = kEmpty, w = 0;
    if (fits && sub < L) {
      key = (u32)cmap[adjncy[pos]];
      w = (u32)adjwgt[pos];
      if (key == (u32)c) key = kEmpty;
    }
    const i32 u = merge_lanes<G, K>(key, w, o, sadj, swgt);
    if (on && sub == 0) {
      if (fits) cnt[c] = u;
      else mid[atomicAdd(nmid, 1)] = (i32)c;
    }
  }
}

// One warp per coarse row: all of them, or those of a list.
template <int WCAP, int WARPS, class K>
__global__ void __launch_bounds__(WARPS * 32) k_contract_warp(
    const i32* __restrict__ ncp, const i32* __restrict__ list, const i32* __restrict__ xadj,
    const i32* __restrict__ adjncy, const i32* __restrict__ adjwgt,
    const i32* __restrict__ cmap, const i32* __restrict__ memtab, const i32* __restrict__ mcnt, i32 cap,
    const i32* __restrict__ rowlen, const i32* __restrict__ ub, i32* __restrict__ sadj,
    i32* __restrict__ swgt, i32* __restrict__ cnt, i32* __restrict__ heavy, i32* __restrict__ nheavy) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  WarpTable<WCAP>* tabs = reinterpret_cast<WarpTable<WCAP>*>(smem_raw);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  WarpTable<WCAP>& T = tabs[wid];
  const i32 nrows = *ncp;   // coarse vertices, or entries of the list
  const i64 nw = (i64)gridDim.x * WARPS;
  // The next coarse vertex's header (row length, member count, this lane's
  // member) is loaded while the current one is contracted: two of the five
  // dependent loads of a coarse row leave the chain.
  i64 q = (i64)blockIdx.x * WARPS + wid;
  i32 nL = 0, nnm = 0, nmv = 0, nxc = 0;
  auto header = [&](i64 qq) {
    if (qq < nrows) {
      nxc = list ? list[qq] : (i32)qq;
      nL = rowlen[nxc];
      nnm = mcnt[nxc];
      nmv = lane < cap ? memtab[nxc * (i64)cap + lane] : 0;
    }
  };
  header(q);
  for (; q < nrows; q += nw) {
    const i32 c = nxc, L = nL, nm = nnm, mv = nmv;
    header(q + nw);
    if (L > WCAP || nm > 32) {
      if (lane == 0) heavy[atomicAdd(nheavy, 1)] = c;
      continue;
    }
    // lane j < nm: member j's row; inclusive prefix of the row lengths
    i32 mbeg = 0, mlen = 0;
    if (lane < nm) {
      mbeg = xadj[mv];
      mlen = xadj[mv + 1] - mbeg;
    }
    const i32 o = ub[c];   // needed only at the writes
    i32 incl = mlen;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const i32 y = __shfl_up_sync(kFull, incl, d);
      if (lane >= d) incl += y;
    }
    const i32 shift = mbeg - (incl - mlen);
    // entry i of the concatenated rows -> its CSR position
    auto entry_pos = [&](i32 i) {
      i32 jm = 0;
      for (i32 j = 0; j < nm; ++j) jm += i >= __shfl_sync(kFull, incl, j);
      return __shfl_sync(kFull, shift, jm & 31) + i;
    };
    // Rows whose entries other than self loops fit one per lane merge in
    // registers: every row of up to 32 entries, and rows of up to 64 entries
    // with at most 32 left after the self loops (the members' edges to one
    // another) are dropped -- most coarse rows of a mesh.
    u32 key = kEmpty, w = 0;
    bool in_regs = false;
    if (L <= 32) {
      const i32 pos = entry_pos(lane);
      if (lane < L) {
        key = (u32)cmap[adjncy[pos]];
        w = (u32)adjwgt[pos];
        if (key == (u32)c) key = kEmpty;
      }
      in_regs = true;
    } else if (L <= 64) {
      const i32 p0 = entry_pos(lane), p1 = entry_pos(lane + 32);
      u32 k0 = (u32)cmap[adjncy[p0]], w0 = (u32)adjwgt[p0], k1 = kEmpty, w1 = 0;
      if (lane + 32 < L) {
        k1 = (u32)cmap[adjncy[p1]];
        w1 = (u32)adjwgt[p1];
      }
      if (k0 == (u32)c) k0 = kEmpty;
      if (k1 == (u32)c) k1 = kEmpty;
      const u32 m0 = __ballot_sync(kFull, k0 != kEmpty), m1 = __ballot_sync(kFull, k1 != kEmpty);
      const i32 n0 = __popc(m0), tot = n0 + __popc(m1);
      if (tot <= 32) {   // warp-uniform: compact the kept entries to one per lane
        const u32 lt = (1u << lane) - 1u;
        if (k0 != kEmpty) T.out[__popc(m0 & lt)] = ((u64)k0 << 32) | w0;
        if (k1 != kEmpty) T.out[n0 + __popc(m1 & lt)] = ((u64)k1 << 32) | w1;
        __syncwarp();
        const u64 kv = lane < tot ? T.out[lane] : ~0ull;
        __syncwarp();
        key = (u32)(kv >> 32);
        w = (u32)kv;
        in_regs = true;
      }
    }
    if (in_regs) {
      const i32 u = merge_lanes<32, K>(key, w, o, sadj, swgt);
      if (lane == 0) cnt[c] = u;
      continue;
    }
    u32 hsz = 64;
    while (hsz < 2u * (u32)L) hsz <<= 1;
    for (u32 i = lane; i < hsz; i += 32) { T.keys[i] = kEmpty; T.vals[i] = 0; }
    __syncwarp();
    for (i32 b = 0; b < L; b += 32) {
      const i32 i = b + lane;
      const i32 pos = entry_pos(i);
      if (i < L) {
        const u32 key = (u32)cmap[adjncy[pos]];
        if (key != (u32)c) table_add(T.keys, T.vals, hsz, key, (u32)adjwgt[pos]);
      }
    }
    __syncwarp();
    // compact occupied slots
    i32 U = 0;
    for (u32 base = 0; base < hsz; base += 32) {
      const u32 sl = base + lane;
      const bool occ = T.keys[sl] != kEmpty;
      const u32 bal = __ballot_sync(kFull, occ);
      if (occ) {
        const i32 at = U + __popc(bal & ((1u << lane) - 1));
        T.out[at] = ((u64)T.keys[sl] << 32) | T.vals[sl];
      }
      U += __popc(bal);
    }
    __syncwarp();
    if (U <= 32) {
      u64 key = lane < U ? T.out[lane] : ~0ull;
#pragma unroll
      for (int kk = 2; kk <= 32; kk <<= 1) {
#pragma unroll
        for (int jj = kk >> 1; jj > 0; jj >>= 1) {
          const u64 ot = __shfl_xor_sync(kFull, key, jj);
          const bool up = (lane & kk) == 0;
          const bool lower = (lane & jj) == 0;
          key = (lower == up) ? umin64(key, ot) : umax64(key, ot);
        }
      }
      if (lane < U) {
        sadj[o + lane] = (i32)(u32)(key >> 32);
        swgt[o + lane] = (i32)(u32)key;
      }
    } else {
      i32 P = 64;
      while (P < U) P <<= 1;
      for (i32 i = U + lane; i < P; i += 32) T.out[i] = ~0ull;
      __syncwarp();
      warp_bitonic_u64(T.out, P, lane);
      for (i32 i = lane; i < U; i += 32) {
        const u64 kv = T.out[i];
        sadj[o + i] = (i32)(u32)(kv >> 32);
        swgt[o + i] = (i32)(u32)kv;
      }
    }
    if (lane == 0) cnt[c] = U;
    __syncwarp();
  }
}

// Heavy rows (longer than the warp tables) by direct accumulation: one CTA per
// row, a weight per coarse id in shared memory (kDenseIds ids at a time, a
// window of the id range) and a bit per id that was met, whose order is the
// row's -- no hashing, no sort.  On levels of more than kDenseIds coarse
// vertices the row's own range of ids is found first, and the windows cover
// that: a union of many graphs has millions of ids, its rows one graph's few
// thousand.  Rows that would take more than kDenseWindows windows
// (kDenseNear, if the shared table of k_contract_cta holds them) are left to
// that kernel, whose hashing and sorting cost about as much as that many
// windows (heavy rows of all levels of a 4M-vertex circuit graph 6.8 ms by
// hashing alone, now 1.8).
constexpr i32 kDenseThreads = 1024;
constexpr i32 kDenseIds = 53248;
constexpr i32 kDenseWindows = 32;
constexpr i32 kDenseNear = 4;
constexpr size_t kDenseSmem = (size_t)kDenseIds * 4 + kDenseIds / 8;
constexpr i32 kCtaCap = 4096;   // k_contract_cta: longest row of its shared table

// rest, nrest: the rows left to k_contract_cta
__global__ void __launch_bounds__(kDenseThreads, 1) k_contract_dense(
    const i32* __restrict__ ncp, const i32* __restrict__ heavy, const i32* __restrict__ nheavy,
    const i32* __restrict__ xadj, const i32* __restrict__ adjncy, const i32* __restrict__ adjwgt,
    const i32* __restrict__ cmap, const i32* __restrict__ memtab, const i32* __restrict__ mcnt, i32 cap,
    const i32* __restrict__ rowlen, const i32* __restrict__ ub, i32* __restrict__ sadj, i32* __restrict__ swgt,
    i32* __restrict__ cnt, i32* __restrict__ rest, i32* __restrict__ nrest) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  u32* acc = reinterpret_cast<u32*>(smem_raw);         // [kDenseIds]
  u32* bits = acc + kDenseIds;                         // [kDenseIds / 32]
  __shared__ i32 s_warp[kDenseThreads / 32];
  __shared__ i32 s_lo, s_hi;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const i32 nc = *ncp, nh = *nheavy;
  if (nh == 0) return;
  for (i32 x = threadIdx.x; x < kDenseIds + kDenseIds / 32; x += kDenseThreads) acc[x] = 0;   // bits follow acc
  __syncthreads();
  for (i32 b = blockIdx.x; b < nh; b += gridDim.x) {
    const i32 c = heavy[b];
    const i32 nm = mcnt[c], o = ub[c];
    auto entries = [&](auto visit) {         // visit(coarse id, weight) by every thread's entries, none of them c
      for (i32 j0 = 0; j0 < nm; j0 += 4) {   // four member rows together
        u32 beg[4], end[4];
#pragma unroll
        for (i32 q = 0; q < 4; ++q) {
          const i32 v = j0 + q < nm ? memtab[c * (i64)cap + j0 + q] : -1;
          beg[q] = v >= 0 ? (u32)xadj[v] + threadIdx.x : 0;
          end[q] = v >= 0 ? (u32)xadj[v + 1] : 0;
        }
        bool more = true;
        while (more) {
          i32 u[4], w[4];
#pragma unroll
          for (i32 q = 0; q < 4; ++q) {
            u[q] = beg[q] < end[q] ? adjncy[beg[q]] : -1;
            w[q] = beg[q] < end[q] ? adjwgt[beg[q]] : 0;
          }
#pragma unroll
          for (i32 q = 0; q < 4; ++q) u[q] = u[q] >= 0 ? cmap[u[q]] : -1;
          more = false;
#pragma unroll
          for (i32 q = 0; q < 4; ++q) {
            if (u[q] >= 0 && u[q] != c) visit(u[q], (u32)w[q]);
            if (beg[q] < end[q]) beg[q] += kDenseThreads;   // (a short row's place stays while a longer one goes on)
            more |= beg[q] < end[q];
          }
        }
      }
    };
    i32 lo = 0, hi = nc - 1;
    if (nc > kDenseIds) {   // block-uniform
      if (threadIdx.x == 0) {
        s_lo = INT_MAX;
        s_hi = -1;
      }
      __syncthreads();
      lo = INT_MAX;
      hi = -1;
      entries([&](i32 u, u32) {
        lo = u < lo ? u : lo;
        hi = u > hi ? u : hi;
      });
      lo = __reduce_min_sync(kFull, lo);
      hi = __reduce_max_sync(kFull, hi);
      if (lane == 0) {
        atomicMin(&s_lo, lo);
        atomicMax(&s_hi, hi);
      }
      __syncthreads();
      lo = s_lo;
      hi = s_hi;
      __syncthreads();
      if (hi >= 0 && (hi - lo) / kDenseIds >= (rowlen[c] > kCtaCap ? kDenseWindows : kDenseNear)) {   // block-uniform
        if (threadIdx.x == 0) rest[atomicAdd(nrest, 1)] = c;
        continue;
      }
    }
    i32 U = 0;
    for (i64 w1 = lo; w1 <= hi; w1 += kDenseIds) {
      const i32 w0 = (i32)w1;
      const u32 wn = (u32)(hi - w0 < kDenseIds - 1 ? hi - w0 + 1 : kDenseIds);
      entries([&](i32 u, u32 w) {
        const u32 id = (u32)(u - w0);
        if (id < wn) {
          atomicAdd(&acc[id], w);
          atomicOr(&bits[id >> 5], 1u << (id & 31));
        }
      });
      __syncthreads();
      // the met ids in order: kDenseIds / 32 / kDenseThreads words a thread
      constexpr i32 kW = (kDenseIds / 32 + kDenseThreads - 1) / kDenseThreads;
      const i32 x0 = (i32)threadIdx.x * kW;
      u32 word[kW];
      i32 n = 0;
#pragma unroll
      for (i32 q = 0; q < kW; ++q) {
        word[q] = x0 + q < kDenseIds / 32 ? bits[x0 + q] : 0u;
        n += __popc(word[q]);
      }
      i32 inc = n;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const i32 y = __shfl_up_sync(kFull, inc, d);
        if (lane >= d) inc += y;
      }
      if (lane == 31) s_warp[wid] = inc;
      __syncthreads();
      i32 before = 0, tot = 0;
      for (i32 w = 0; w < kDenseThreads / 32; ++w) {
        const i32 y = s_warp[w];
        before += w < wid ? y : 0;
        tot += y;
      }
      i32 at = o + U + before + inc - n;
#pragma unroll
      for (i32 q = 0; q < kW; ++q) {
        if (word[q]) bits[x0 + q] = 0;
        for (u32 m = word[q]; m; m &= m - 1) {
          const i32 id = ((x0 + q) << 5) + __ffs(m) - 1;
          sadj[at] = w0 + id;
          swgt[at] = (i32)acc[id];
          acc[id] = 0;
          ++at;
        }
      }
      U += tot;
      __syncthreads();   // acc and bits are clear; s_warp is free
    }
    if (threadIdx.x == 0) cnt[c] = U;
  }
}

// One CTA per heavy coarse row.  Table in dynamic shared memory when the row
// fits (L <= cta_cap); longer rows take their table from the handle's arena
// (bump allocation: keys and values of hsz words each, then hsz/2 sorted
// outputs as u64).  A row that does not fit in the arena records the words it
// needs and sets the overflow flag; the host grows the arena and runs the
// contraction again.  Both kinds of row run in one launch.
__global__ void __launch_bounds__(512) k_contract_cta(
    const i32* __restrict__ heavy, const i32* __restrict__ nheavy, i32 cta_cap,
    const i32* __restrict__ xadj, const i32* __restrict__ adjncy, const i32* __restrict__ adjwgt,
    const i32* __restrict__ cmap, const i32* __restrict__ memtab, const i32* __restrict__ mcnt, i32 cap,
    const i32* __restrict__ rowlen, const i32* __restrict__ ub, i32* __restrict__ sadj,
    i32* __restrict__ swgt, i32* __restrict__ cnt, ArenaHdr* arena, u32* arena_words, u64 arena_cap) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ i32 s_count;
  __shared__ u64 s_off;
  const i32 nh = *nheavy;
  for (i32 b = blockIdx.x; b < nh; b += gridDim.x) {
    const i32 c = heavy[b];
    const i32 L = rowlen[c];
    const bool global_table = L > cta_cap;   // block-uniform
    const u32 hsz = table_slots((u32)L);
    u32 *keys, *vals;
    u64* out;
    if (global_table) {
      const u64 words = 3ull * hsz;   // keys + vals + hsz/2 u64 outputs
      if (threadIdx.x == 0) {
        const u64 off = atomicAdd((unsigned long long*)&arena->used, (unsigned long long)words);
        if (off + words > arena_cap) {
          atomicAdd((unsigned long long*)&arena->need, (unsigned long long)words);
          atomicExch(&arena->overflow, 1);
          s_off = ~0ull;
        } else {
          s_off = off;
        }
      }
      __syncthreads();
      const u64 off = s_off;
      __syncthreads();   // every thread has read s_off before thread 0 can set it for the next row
      if (off == ~0ull) continue;   // block-uniform; redone after the arena grows
      keys = arena_words + off;
      vals = keys + hsz;
      out = reinterpret_cast<u64*>(vals + hsz);
    } else {
      keys = reinterpret_cast<u32*>(smem_raw);
      vals = keys + 2 * cta_cap;
      out = reinterpret_cast<u64*>(vals + 2 * cta_cap);
    }
    for (u32 i = threadIdx.x; i < hsz; i += blockDim.x) { keys[i] = kEmpty; vals[i] = 0; }
    if (threadIdx.x == 0) s_count = 0;
    __syncthreads();
    const i32 nm = mcnt[c];
    for (i32 j = 0; j < nm; ++j) {
      const i32 v = memtab[c * (i64)cap + j];
      const i32 beg = xadj[v], end = xadj[v + 1];
      for (u32 e = (u32)beg + threadIdx.x; e < (u32)end; e += blockDim.x) {
        const u32 key = (u32)cmap[adjncy[e]];
        if (key != (u32)c) table_add(keys, vals, hsz, key, (u32)adjwgt[e]);
      }
    }
    __syncthreads();
    for (u32 sl = threadIdx.x; sl < hsz; sl += blockDim.x) {
      if (keys[sl] != kEmpty) {
        const i32 pos = atomicAdd(&s_count, 1);
        out[pos] = ((u64)keys[sl] << 32) | vals[sl];
      }
    }
    __syncthreads();
    const i32 U = s_count;
    i32 P = 64;
    while (P < U) P <<= 1;
    for (i32 i = U + threadIdx.x; i < P; i += blockDim.x) out[i] = ~0ull;
    __syncthreads();
    cta_bitonic_u64(out, P);
    const i32 o = ub[c];
    for (i32 i = threadIdx.x; i < U; i += blockDim.x) {
      const u64 kv = out[i];
      sadj[o + i] = (i32)(u32)(kv >> 32);
      swgt[o + i] = (i32)(u32)kv;
    }
    if (threadIdx.x == 0) cnt[c] = U;
    __syncthreads();
  }
}

// One warp per R consecutive coarse rows (R <= 32): the lanes scan the rows'
// lengths and copy the R rows' entries as one flat range, each lane finding
// its entry's row by a binary search over the lanes' prefix sums.  R is small
// on levels of long rows: a dense level has few rows, and 32 of 1000 entries
// kept one warp for 32k (all levels of a 4M-vertex circuit graph: 4.4 ms, now
// 0.9).  On levels of up to 100k vertices R = 8 (or 4) gives more warps a
// shorter chain (2048 vertices: 7.6 us, now 5.3; on a million R = 8 is 2.6x
// slower than 32; the line: coarsening of a 90k mesh 324 us with 32 and 314
// with 8, of a 130k one the same, of a 200k one 403 and 413).
// Also the level's longest coarse row and heaviest coarse vertex (both
// *maxdeg and *max_cvw start at zero).
__global__ void k_copy_rows(const i32* __restrict__ ncp, i32 R, const i32* __restrict__ ub,
                            const i32* __restrict__ cnt,
                            const i32* __restrict__ cx, const i32* __restrict__ sadj,
                            const i32* __restrict__ swgt, i32* __restrict__ cadj, i32* __restrict__ cwgt,
                            i32* __restrict__ maxdeg, const i32* __restrict__ cvw, i32* __restrict__ max_cvw) {
  const i32 nc = *ncp;
  const int lane = threadIdx.x & 31;
  const i64 warp = ((i64)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const i64 nwarps = ((i64)gridDim.x * blockDim.x) >> 5;
  i32 mx = 0, mw = 0;
  for (i64 c0 = warp * R; c0 < nc; c0 += nwarps * R) {
    const i64 c = c0 + lane;
    i32 src = 0, dst = 0, len = 0;
    if (lane < R && c < nc) {
      src = ub[c];
      dst = cx[c];
      len = cnt[c];
      mw = cvw[c] > mw ? cvw[c] : mw;
    }
    mx = len > mx ? len : mx;
    i32 inc = len;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const i32 y = __shfl_up_sync(kFull, inc, o);
      if (lane >= o) inc += y;
    }
    const i32 total = __shfl_sync(kFull, inc, 31);
    const i32 exc = inc - len;
    if (R == 1) {   // one row: a straight copy, four entries a lane together
      const i32 rs = __shfl_sync(kFull, src, 0), rd = __shfl_sync(kFull, dst, 0);
      constexpr i32 kU = 4;
      for (i32 e0 = lane; e0 < total; e0 += 32 * kU) {
        i32 x[kU], y[kU];
#pragma unroll
        for (i32 q = 0; q < kU; ++q)
          if (e0 + 32 * q < total) {
            x[q] = sadj[rs + e0 + 32 * q];
            y[q] = swgt[rs + e0 + 32 * q];
          }
#pragma unroll
        for (i32 q = 0; q < kU; ++q)
          if (e0 + 32 * q < total) {
            cadj[rd + e0 + 32 * q] = x[q];
            cwgt[rd + e0 + 32 * q] = y[q];
          }
      }
      continue;
    }
    for (i32 base = 0; base < total; base += 32) {   // warp-uniform: every lane takes every shuffle
      const i32 idx = base + lane;
      // the row r with exc_r <= idx < inc_r: the first lane whose inclusive sum exceeds idx
      i32 r = 0;
#pragma unroll
      for (int step = 16; step > 0; step >>= 1) {
        const i32 probe = __shfl_sync(kFull, inc, r + step - 1);
        if (probe <= idx) r += step;
      }
      r = r < 31 ? r : 31;
      const i32 rs = __shfl_sync(kFull, src, r), rd = __shfl_sync(kFull, dst, r), re = __shfl_sync(kFull, exc, r);
      if (idx < total) {
        cadj[rd + (idx - re)] = sadj[rs + (idx - re)];
        cwgt[rd + (idx - re)] = swgt[rs + (idx - re)];
      }
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const i32 y = __shfl_xor_sync(kFull, mx, o);
    mx = mx > y ? mx : y;
    const i32 z = __shfl_xor_sync(kFull, mw, o);
    mw = mw > z ? mw : z;
  }
  if (lane == 0 && mx > 0) atomicMax(maxdeg, mx);
  if (lane == 0 && mw > 0) atomicMax(max_cvw, mw);
}

void ensure_arena(Handle& h, u64 words) {
  if (h.arena && h.arena_words >= words) return;
  GKW_REQUIRE(!h.capturing, GKW_E_INTERNAL, "arena grown during a graph capture");
  graph_cache_clear(h);   // graphs hold the old arena's address
  GKW_CUDA(cudaStreamSynchronize(h.stream));
  if (h.arena) GKW_CUDA(cudaFree(h.arena));
  h.arena = nullptr;
  h.arena_words = 0;
  GKW_CUDA(cudaMalloc(&h.arena, sizeof(ArenaHdr) + sizeof(u32) * words));
  // on the handle's stream: that stream does not wait for the legacy stream
  GKW_CUDA(cudaMemsetAsync(h.arena, 0, sizeof(ArenaHdr), h.stream));
  h.arena_words = words;
}

// The tables that the row kernels share.
struct ContractTables {
  i32 *rowlen, *ub, *mcnt, *memtab, *cnt, *heavy, *mid;
  i32* misc;   // [0] heavy rows, [1] ub total, [2..4] rows listed by the short, the 512 and the dense kernel
  i32 *sadj, *swgt;
  size_t nz;
};

// what the row kernels need besides the members and the lengths
static void row_tables(Handle& h, ContractTables& t, i64 m, i32 nc_ub) {
  const i64 nu = (i64)nc_ub + 1;
  t.ub = h.scratch.alloc_n<i32>(nu);
  t.heavy = h.scratch.alloc_n<i32>(nu);
  t.mid = h.scratch.alloc_n<i32>(nu);
  t.sadj = h.scratch.alloc_n<i32>(std::max<i64>(m, 1));
  t.swgt = h.scratch.alloc_n<i32>(std::max<i64>(m, 1));
}

static ContractTables contract_tables(Handle& h, i64 m, i32 nc_ub, i32 cap) {
  const i64 nu = (i64)nc_ub + 1;
  ContractTables t;
  t.nz = ((size_t)nu + 63) & ~(size_t)63;
  t.rowlen = h.scratch.alloc_n<i32>(3 * t.nz + 8);   // cleared together: rowlen, mcnt, cnt, misc
  t.mcnt = t.rowlen + t.nz;
  t.cnt = t.mcnt + t.nz;
  t.misc = t.cnt + t.nz;
  t.memtab = h.scratch.alloc_n<i32>((i64)nc_ub * cap + 1);
  row_tables(h, t, m, nc_ub);
  return t;
}

static void contract_rows(Handle& h, const DevGraph& g, const ContractTables& t, const i32* cmap, const i32* d_nc,
                          i32 nc_ub, i32 cap, i32* cxadj, i32* cadjncy, i32* cadjwgt, const i32* cvwgt, i32* d_mc);

void run_contract(Handle& h, const DevGraph& g, const i32* cmap, const i32* d_nc, i32 nc_ub, i32 cap, i32* cxadj,
                  i32* cadjncy, i32* cadjwgt, i32* cvwgt, i32* d_mc) {
  Pool::Mark mk = h.scratch.mark();
  const i32 n = g.n;
  const i64 nu = (i64)nc_ub + 1;
  const u32 nb = ceil_div(std::max(n, 1), 256);
  const ContractTables t = contract_tables(h, g.m, nc_ub, cap);
  ensure_arena(h, u64(4) << 20);   // 16 MB of long-row tables to start with
  GKW_CUDA(cudaMemsetAsync(cvwgt, 0, sizeof(i32) * std::max(nc_ub, 1), h.stream));
  GKW_CUDA(cudaMemsetAsync(t.rowlen, 0, sizeof(i32) * (3 * t.nz + 8), h.stream));
  if (n > 0)
    launch(k_coarse_accum, nb, 256, 0, h.stream, n, g.xadj, g.vwgt, cmap, cap, cvwgt, t.rowlen, t.mcnt, t.memtab,
           h.arena, h.coop);
  else   // (two words)
    GKW_CUDA(cudaMemsetAsync(&h.coop->max_cvw, 0, 2 * sizeof(i32), h.stream));
  GKW_CHECK_LAUNCH();
  exclusive_scan_i32(h, t.rowlen, t.ub, nu, t.misc + 1, d_nc);
  contract_rows(h, g, t, cmap, d_nc, nc_ub, cap, cxadj, cadjncy, cadjwgt, cvwgt, d_mc);
  h.scratch.release(mk);
}

// A level of at most kSmallLevel vertices from its candidates on.
static void run_small_level(Handle& h, const DevGraph& g, const i32* cand, i32 cap, const CoarsenOut& out) {
  Pool::Mark mk = h.scratch.mark();
  const ContractTables t = contract_tables(h, g.m, g.n, cap);
  SmallLevel a;
  a.n = g.n;
  a.cap = cap;
  a.cand = cand;
  a.xadj = g.xadj;
  a.vwgt = g.vwgt;
  a.cmap = out.cmap;
  a.cvwgt = out.cvwgt;
  a.rowlen = t.rowlen;
  a.ub = t.ub;
  a.mcnt = t.mcnt;
  a.memtab = t.memtab;
  a.cnt = t.cnt;
  a.misc = t.misc;
  a.arena = h.arena;
  a.nc = &h.coop->nc;
  a.uf_rounds = &h.coop->uf_rounds;
  a.max_cvw = &h.coop->max_cvw;
  a.maxdeg = &h.coop->maxdeg;
  if (!h.capturing)
    GKW_CUDA(cudaFuncSetAttribute(k_group_small, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmallLevel * 16));
  launch(k_group_small, 1, kSmallThreads, (size_t)g.n * 16, h.stream, a);
  GKW_CHECK_LAUNCH();
  contract_rows(h, g, t, out.cmap, &h.coop->nc, g.n, cap, out.cxadj, out.cadjncy, out.cadjwgt, out.cvwgt,
                &h.coop->mc);
  h.scratch.release(mk);
}

// A larger level: the passes between match and rows fused where one knows
// what the next needs.  The match writes the union-find's start; the walk
// counts the groups, and the count a vertex meets is its place in the member
// lists; the scan of the coarse ids takes the sizes as they are and packs them
// with the ids; each vertex adds itself to its coarse vertex when it learns
// its id, with one atomic in place of three; the scans end at n_c.  Five
// launches fewer a level, and on large levels two passes over the vertices
// (coarsening of a million-vertex mesh 870 -> 800 us, a 100k mesh 316 -> 295).
// A 12M-vertex road graph, whose scattered words exceed L2, gains 1%.
static void run_large_level(Handle& h, const DevGraph& g, i32 cap, const CoarsenOut& out) {
  GKW_REQUIRE(cap >= 1, GKW_E_INVALID, "group_cap must be >= 1");
  const i32 n = g.n;
  const u32 nb = ceil_div(n, 256);
  Pool::Mark mk = h.scratch.mark();
  ContractTables t;
  const size_t nz = ((size_t)n + 1 + 63) & ~(size_t)63;
  u64* sums = h.scratch.alloc_n<u64>(nz + 4);   // and misc, cleared together
  t.misc = reinterpret_cast<i32*>(sums + nz);
  t.mcnt = h.scratch.alloc_n<i32>((i64)n + 1);
  t.memtab = h.scratch.alloc_n<i32>((i64)n * cap + 1);
  const Pool::Mark groups = h.scratch.mark();
  u64* block = h.scratch.alloc_n<u64>(2 * (size_t)n);   // union-find and slots, then the giant groups' sort
  UfStart uf;
  uf.parent = reinterpret_cast<i32*>(block);
  uf.dist = reinterpret_cast<u32*>(uf.parent + n);
  i32* cand = uf.parent + 2 * (size_t)n;
  u64* keys = h.scratch.alloc_n<u64>(n);
  GroupTables gt = group_tables(h, n);
  gt.slot = cand + n;
  GKW_CUDA(cudaMemsetAsync(sums, 0, sizeof(u64) * (nz + 4), h.stream));
  GKW_CUDA(cudaMemsetAsync(gt.gsize, 0, sizeof(i32) * gt.cleared, h.stream));
  run_match_uf(h, g, cand, g.maxdeg, uf);
  launch(k_uf_hook, nb, 256, 0, h.stream, n, (const i32*)cand, uf.parent, &h.coop->uf_rounds);
  launch(k_uf_mark, nb, 256, 0, h.stream, n, (const i32*)cand, (const i32*)uf.parent, uf.dist);
  launch(k_uf_walk, nb, 256, 0, h.stream, n, (const i32*)cand, uf.parent, uf.dist, keys, &h.coop->uf_rounds,
         gt.gsize, gt.slot);
  GKW_CHECK_LAUNCH();
  Accum acc;
  acc.xadj = g.xadj;
  acc.vwgt = g.vwgt;
  acc.sums = sums;
  acc.mcnt = t.mcnt;
  acc.memtab = t.memtab;
  run_groups(h, n, keys, cap, gt, block, out.cmap, &h.coop->nc, acc);
  h.scratch.release(groups);   // the row tables take their place
  t.rowlen = h.scratch.alloc_n<i32>((i64)n + 1);
  t.cnt = h.scratch.alloc_n<i32>((i64)n + 1);
  row_tables(h, t, g.m, n);
  scan_coarse_sums(h, sums, t.ub, t.rowlen, out.cvwgt, t.cnt, (i64)n + 1, t.misc + 1, &h.coop->nc);
  contract_rows(h, g, t, out.cmap, &h.coop->nc, n, cap, out.cxadj, out.cadjncy, out.cadjwgt, out.cvwgt, &h.coop->mc);
  h.scratch.release(mk);
}

// The coarse rows from the prepared tables.
static void contract_rows(Handle& h, const DevGraph& g, const ContractTables& t, const i32* cmap, const i32* d_nc,
                          i32 nc_ub, i32 cap, i32* cxadj, i32* cadjncy, i32* cadjwgt, const i32* cvwgt, i32* d_mc) {
  const i32 n = g.n;
  const i64 nu = (i64)nc_ub + 1;
  i32 *const rowlen = t.rowlen, *const ub = t.ub, *const mcnt = t.mcnt, *const memtab = t.memtab, *const cnt = t.cnt;
  i32 *const heavy = t.heavy, *const mid = t.mid, *const misc = t.misc, *const sadj = t.sadj, *const swgt = t.swgt;
  // Expected coarse row: a group's members (about five; at most cap) times the
  // mean degree.  Short rows take 16 lanes each (12M-vertex road graph, 7
  // entries a row: 3.2 ms with a warp each, now 1.4 over all levels); else one
  // warp per row with a table of 128 entries, 256 or 512.  A 27-point grid's
  // rows have up to 156: with 128 nearly all went to one CTA each, 6.5 ms, now
  // 0.73; above 400 expected the 512 table keeps more rows out of the heavy
  // list, below it 256 lets four CTAs share an SM (2.9 -> 0.8 ms on the
  // circuit graph's third level).
  const double avg = n ? (double)g.m / n : 0.0;
  const double expL = avg * std::min(cap, 6);
  const u32 gridw = std::max<u32>(1, std::min<u32>(ceil_div(std::max(nc_ub, 1), 8), (u32)h.sm_count * 32));
  u32* words = reinterpret_cast<u32*>(h.arena + 1);
  const bool wide_ids = n >= (1 << 27);   // (id, lane) keys of 64 bits
  const i32* rows = d_nc;
  const i32* list = nullptr;
  const bool shorts = expL <= 20 && cap <= kContractG;
  if (shorts) {
    auto go = [&](auto kern) {
      launch(kern, std::max<u32>(1, std::min<u32>(ceil_div(std::max(nc_ub, 1), 16), (u32)h.sm_count * 32)), 256, 0,
             h.stream, d_nc, g.xadj, g.adjncy, g.adjwgt, cmap, memtab, mcnt, cap, rowlen, ub, sadj, swgt, cnt, mid,
             misc + 2);
    };
    if (wide_ids) go(k_contract_short<u64>);
    else go(k_contract_short<u32>);
    rows = misc + 2;
    list = mid;
  }
  auto warps = [&](auto w, auto k, i32* over, i32* nover) {   // rows beyond W entries go to `over`
    constexpr int W = decltype(w)::value, WARPS = 8;
    typedef decltype(k) K;
    const size_t sm = sizeof(WarpTable<W>) * WARPS;
    auto kern = k_contract_warp<W, WARPS, K>;
    if (!h.capturing)
      GKW_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
    launch(kern, gridw, WARPS * 32, sm, h.stream, rows, list, g.xadj, g.adjncy, g.adjwgt, cmap, memtab, mcnt, cap,
           rowlen, ub, sadj, swgt, cnt, over, nover);
  };
  if (wide_ids) warps(std::integral_constant<int, 128>(), u64(), heavy, misc);
  else if (expL <= 100) warps(std::integral_constant<int, 128>(), u32(), heavy, misc);   // (W below)
  else if (expL <= 400) warps(std::integral_constant<int, 256>(), u32(), heavy, misc);
  else warps(std::integral_constant<int, 512>(), u32(), heavy, misc);
  GKW_CHECK_LAUNCH();
  // Where a row can outgrow the smaller tables, the rows that did go through
  // the 512 one: a level whose mean hides rows of a few hundred entries (a
  // union of 256 circuits and meshes: 120k of them) left those to one CTA each
  // (5.3 ms on its first level, now 0.84).  A warp takes longer over one row
  // than a CTA, so the pass pays where rows of a few hundred entries are many,
  // which the host does not know.  By n, coarsening in ms without the pass and
  // with it: 60k vertices, circuit 0.71 / 0.98, mesh with 1% of hubs of 100
  // 0.60 / 0.77; 200k, 1.18 / 1.26 and 1.10 / 0.98; 800k, 3.22 / 3.36 and
  // 2.98 / 2.18: below 100k it loses on both, above it a little on the one and
  // much less than it gains on the other.
  constexpr i32 kMid512 = 100000;
  i32 *over = heavy, *nover = misc, *free_list = mid;
  i32 W = wide_ids || expL <= 100 ? 128 : expL <= 400 ? 256 : 512;
  auto can_outgrow = [&] { return g.maxdeg < 0 || g.maxdeg * (i64)cap > W || cap > 32; };
  if (W < 512 && !wide_ids && n > kMid512 && can_outgrow()) {
    rows = misc;
    list = heavy;
    warps(std::integral_constant<int, 512>(), u32(), mid, misc + 3);
    GKW_CHECK_LAUNCH();
    W = 512;
    over = mid;
    nover = misc + 3;
    free_list = heavy;
  }
  // heavy rows: only where a row can outgrow the warp tables.  A shared-memory
  // table up to kCtaCap entries, the arena beyond (2*kCtaCap table slots, a
  // power of two, + kCtaCap sorted outputs: 96 KB)
  if (can_outgrow()) {
    const size_t csm = (size_t)kCtaCap * 2 * 4 * 2 + (size_t)kCtaCap * 8;
    if (!h.capturing) {
      GKW_CUDA(cudaFuncSetAttribute(k_contract_dense, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDenseSmem));
      GKW_CUDA(cudaFuncSetAttribute(k_contract_cta, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)csm));
    }
    launch(k_contract_dense, (u32)h.sm_count, kDenseThreads, kDenseSmem, h.stream, d_nc, over, nover, g.xadj,
           g.adjncy, g.adjwgt, cmap, memtab, mcnt, cap, rowlen, ub, sadj, swgt, cnt, free_list, misc + 4);
    if (nc_ub > kDenseIds)
      launch(k_contract_cta, (u32)h.sm_count * 2, 512, csm, h.stream, (const i32*)free_list, (const i32*)(misc + 4), kCtaCap, g.xadj, g.adjncy,
             g.adjwgt, cmap, memtab, mcnt, cap, rowlen, ub, sadj, swgt, cnt, h.arena, words, h.arena_words);
    GKW_CHECK_LAUNCH();
  }
  exclusive_scan_i32(h, cnt, cxadj, nu, d_mc, d_nc);   // cxadj[n_c] = m_c
  const i32 R = expL > 200 ? 1 : nc_ub > 100000 ? 32 : expL <= 48 ? 8 : 4;
  if (nc_ub > 0)
    launch(k_copy_rows, std::min<u32>(ceil_div((u64)nc_ub, 8 * (u64)R), (u32)h.sm_count * 32), 256, 0, h.stream, d_nc, R, ub, cnt, cxadj, sadj, swgt, cadjncy,
           cadjwgt, &h.coop->maxdeg, cvwgt, &h.coop->max_cvw);
  GKW_CHECK_LAUNCH();
}

// The level's scalars and error words straight into the handle's pinned words.
struct CoopReport {
  CoopState coop;
  ArenaHdr arena;
  i32 scan_err;
};
static_assert(sizeof(CoopReport) <= kPinnedWords * sizeof(i64), "pinned words too few");

__global__ void k_coop_report(const CoopState* coop, const ArenaHdr* arena, const ScanState* scan, CoopReport* out) {
  out->coop = *coop;
  if (arena) out->arena = *arena;
  out->scan_err = scan ? scan->err : 0;
}

static void report_coop(Handle& h) {
  launch(k_coop_report, 1, 1, 0, h.stream, (const CoopState*)h.coop, (const ArenaHdr*)h.arena,
         (const ScanState*)h.scan, reinterpret_cast<CoopReport*>(h.h_pinned));
  GKW_CHECK_LAUNCH();
}

// reported: the stream's last launch was report_coop
CoopState read_coop(Handle& h, bool reported) {
  if (!reported) report_coop(h);
  GKW_CUDA(cudaStreamSynchronize(h.stream));
  const CoopReport* r = reinterpret_cast<const CoopReport*>(h.h_pinned);
  const CoopState* hc = &r->coop;
  const ArenaHdr* ha = &r->arena;
  const i32* hs = &r->scan_err;
  CoopState c = *hc;
  c.arena_overflow = h.arena ? ha->overflow : 0;
  c.arena_need = h.arena ? (i64)ha->need : 0;
  c.scan_err = h.scan ? *hs : 0;
  if (c.err || c.scan_err) {   // report once, leave the handle usable
    GKW_CUDA(cudaMemsetAsync(h.coop, 0, sizeof(CoopState), h.stream));
    if (h.scan) GKW_CUDA(cudaMemsetAsync(&h.scan->err, 0, sizeof(i32), h.stream));
    GKW_CUDA(cudaStreamSynchronize(h.stream));
  }
  if (c.err == 1) throw Error{GKW_E_INTERNAL, "cooperative kernel: grid barrier timed out"};
  if (c.err == 2) throw Error{GKW_E_INTERNAL, "union-find did not converge"};
  if (c.scan_err) throw Error{GKW_E_INTERNAL, "scan: look-back wait timed out"};
  return c;
}

// ===========================================================================
// Fused coarsening step: one persistent launch per level runs every phase of
// the step above -- heavy-edge candidates, union-find rounds, group sizes and
// coarse ids, group orders, member lists, contraction, coarse xadj and row
// compaction -- with grid barriers between the phases instead of a dozen
// launches and more.  The phase bodies apply the same rules to
// the same keys as the per-phase kernels, so the level is identical; the
// scans are grid-wide (each CTA scans a contiguous range after a barrier
// publishes the CTA sums).  Data written by other CTAs in the launch is read
// with ld.global.cg.  Dynamic shared memory (96 KB) is shared by the phases:
// the warps' contraction tables, the CTA group sorts and the CTA table of
// heavy coarse rows.
// ===========================================================================
constexpr int kFusedThreads = 512;
constexpr int kFusedWarps = kFusedThreads / 32;
constexpr i32 kFusedWcap = 128;      // warp table entries (as k_contract_warp<128, 8>)
constexpr i32 kFusedCtaCap = 4096;   // heavy rows up to this length use the shared table
constexpr size_t kFusedSmem = (size_t)kFusedCtaCap * 2 * 4 * 2 + (size_t)kFusedCtaCap * 8;   // 96 KB
static_assert(kFusedSmem >= sizeof(WarpTable<kFusedWcap>) * kFusedWarps, "warp tables fit");
static_assert(kFusedSmem >= sizeof(u64) * kGroupSmem, "CTA group sort fits");

// misc counters of the fused step (zeroed by the host before the launch)
enum { kFzLong = 0, kFzWarpG = 1, kFzGiant = 2, kFzCtaG = 3, kFzHeavy = 4, kFzBig = 5, kFzUb = 6, kFzWords = 8 };

struct FusedArgs {
  i32 n;
  i64 m;
  const i32* xadj;
  const i32* adjncy;
  const i32* adjwgt;
  const i32* vwgt;
  i32 lanes;     // match lanes per vertex (2, 4, 8, 16, 32)
  i32 split;     // rows above kMatchLong may exist
  i32 cap;       // group cap
  i32 max_rounds;
  // outputs (coarse level at upper bounds)
  i32* cmap;
  i32* cxadj;
  i32* cadjncy;
  i32* cadjwgt;
  i32* cvwgt;
  // scratch
  i32* cand;
  u64* k0;
  u64* k1;
  i32* chg;        // [3]
  i32* longlist;   // [n]
  i32* gsize;      // [n]
  i32* cbase;      // [n] first coarse id of each root
  i32* goff;       // [n] member offset of each big group
  i32* gcur;       // [n]
  i32* members;    // [n]
  i32* wlist;      // [n] groups sorted by a warp
  i32* clist;      // [n] groups sorted by a CTA
  i32* glist;      // [n] giant groups
  u64* gscratch;   // [2n] giant sort network
  i32* rowlen;     // [n + 1]
  i32* ub;         // [n + 1]
  i32* mcnt;       // [n + 1]
  i32* memtab;     // [n * cap + 1]
  i32* cnt;        // [n + 1]
  i32* heavy;      // [n + 1]
  i32* sadj;       // [m]
  i32* swgt;       // [m]
  i32* partial;    // [2 * grid] CTA sums of the grid scans
  i32* misc;       // [kFzWords]
  // per-level scalars and barrier (CoopState)
  GridBarrier* bar;
  i32* err;
  i32* nc_out;
  i32* mc_out;
  i32* uf_rounds_out;
  i32* maxdeg_out;
  i32* max_cvw_out;
  ArenaHdr* arena;
  u32* arena_words;
  u64 arena_cap;
};

template <int G>
__device__ void fz_match(const FusedArgs& a) {
  const i64 tot = (i64)a.n * G;
  const i64 stride = (i64)gridDim.x * blockDim.x;
  for (i64 base = (i64)blockIdx.x * blockDim.x; base < tot; base += stride) {   // block-uniform trip count
    const i64 t = base + threadIdx.x;
    const i32 v = (i32)(t / G);
    const int sub = threadIdx.x & (G - 1);
    u32 bw = 0, bd = kFull;
    i32 bpos = INT_MAX, bu = -1;
    bool skip = false;
    if (v < a.n) {
      const i32 beg = __ldg(a.xadj + v), end = __ldg(a.xadj + v + 1);
      skip = a.split && end - beg > kMatchLong;   // uniform within the group
      if (skip) {
        if (sub == 0) a.longlist[atomicAdd(a.misc + kFzLong, 1)] = v;
      } else {
        for (u32 e = (u32)beg + sub; e < (u32)end; e += G) {
          const u32 w = (u32)__ldg(a.adjwgt + e);
          if (w == 0 || w < bw) continue;
          const i32 u = __ldg(a.adjncy + e);
          const u32 d = (u32)(__ldg(a.xadj + u + 1) - __ldg(a.xadj + u));
          if (w > bw || d < bd) { bw = w; bd = d; bpos = (i32)e; bu = u; }
        }
      }
    }
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) {
      const u32 ow = __shfl_xor_sync(kFull, bw, o, G);
      const u32 od = __shfl_xor_sync(kFull, bd, o, G);
      const i32 op = __shfl_xor_sync(kFull, bpos, o, G);
      const i32 ou = __shfl_xor_sync(kFull, bu, o, G);
      if (match_better(ow, od, op, bw, bd, bpos)) { bw = ow; bd = od; bpos = op; bu = ou; }
    }
    if (v < a.n && sub == 0 && !skip) a.cand[v] = bw > 0 ? bu : v;
  }
}

// Long rows listed by fz_match: one CTA per row, as k_match_long (the rule's
// order is total, so the thread count does not change the pick).
__device__ void fz_match_long(const FusedArgs& a) {
  __shared__ u32 s_w[kFusedWarps], s_d[kFusedWarps];
  __shared__ i32 s_p[kFusedWarps], s_u[kFusedWarps];
  const i32 nlong = ldcg(a.misc + kFzLong);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const bool vec = ((reinterpret_cast<uintptr_t>(a.adjncy) | reinterpret_cast<uintptr_t>(a.adjwgt)) & 15) == 0;
  for (i32 r = blockIdx.x; r < nlong; r += gridDim.x) {
    const i32 v = ldcg(a.longlist + r);
    const i32 beg = a.xadj[v], end = a.xadj[v + 1];
    u32 bw = 0, bd = kFull;
    i32 bpos = INT_MAX, bu = -1;
    auto visit = [&](u32 w, i32 u, i32 e) {
      if (w == 0 || w < bw) return;
      const u32 d = (u32)(__ldg(a.xadj + u + 1) - __ldg(a.xadj + u));
      if (match_better(w, d, e, bw, bd, bpos)) { bw = w; bd = d; bpos = e; bu = u; }
    };
    if (vec) {
      i32 body = (beg + 3) & ~3;
      i32 tail = body + ((end - body) & ~3);
      if (tail < body) tail = body;
      for (i32 e = beg + threadIdx.x; e < body && e < end; e += blockDim.x) visit((u32)a.adjwgt[e], a.adjncy[e], e);
      for (i32 c = body / 4 + threadIdx.x; c < tail / 4; c += blockDim.x) {
        const int4 w4 = __ldg(reinterpret_cast<const int4*>(a.adjwgt) + c);
        const int4 u4 = __ldg(reinterpret_cast<const int4*>(a.adjncy) + c);
        visit((u32)w4.x, u4.x, 4 * c);
        visit((u32)w4.y, u4.y, 4 * c + 1);
        visit((u32)w4.z, u4.z, 4 * c + 2);
        visit((u32)w4.w, u4.w, 4 * c + 3);
      }
      for (u32 e = (u32)(tail > body ? tail : body) + threadIdx.x; e < (u32)end; e += blockDim.x)
        visit((u32)a.adjwgt[e], a.adjncy[e], (i32)e);
    } else {
      for (u32 e = (u32)beg + threadIdx.x; e < (u32)end; e += blockDim.x) visit((u32)a.adjwgt[e], a.adjncy[e], (i32)e);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const u32 ow = __shfl_xor_sync(kFull, bw, o);
      const u32 od = __shfl_xor_sync(kFull, bd, o);
      const i32 op = __shfl_xor_sync(kFull, bpos, o);
      const i32 ou = __shfl_xor_sync(kFull, bu, o);
      if (match_better(ow, od, op, bw, bd, bpos)) { bw = ow; bd = od; bpos = op; bu = ou; }
    }
    if (lane == 0) {
      s_w[wid] = bw;
      s_d[wid] = bd;
      s_p[wid] = bpos;
      s_u[wid] = bu;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int w = 1; w < kFusedWarps; ++w)
        if (match_better(s_w[w], s_d[w], s_p[w], bw, bd, bpos)) { bw = s_w[w]; bd = s_d[w]; bpos = s_p[w]; bu = s_u[w]; }
      a.cand[v] = bw > 0 ? bu : v;
    }
    __syncthreads();
  }
}

// Block-wide exclusive scan of two i32 per thread; the block totals in tx, ty.
__device__ __forceinline__ void fz_block_exscan2(i32& x, i32& y, i32* s_warp, i32& tx, i32& ty) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  i32 ix = x, iy = y;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const i32 px = __shfl_up_sync(kFull, ix, o), py = __shfl_up_sync(kFull, iy, o);
    if (lane >= o) { ix += px; iy += py; }
  }
  if (lane == 31) { s_warp[wid] = ix; s_warp[32 + wid] = iy; }
  __syncthreads();
  if (wid == 0) {
    const i32 wx = lane < kFusedWarps ? s_warp[lane] : 0, wy = lane < kFusedWarps ? s_warp[32 + lane] : 0;
    i32 sx = wx, sy = wy;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const i32 px = __shfl_up_sync(kFull, sx, o), py = __shfl_up_sync(kFull, sy, o);
      if (lane >= o) { sx += px; sy += py; }
    }
    if (lane < kFusedWarps) { s_warp[lane] = sx - wx; s_warp[32 + lane] = sy - wy; }
    if (lane == kFusedWarps - 1) { s_warp[64] = sx; s_warp[65] = sy; }
  }
  __syncthreads();
  x = ix - x + s_warp[wid];
  y = iy - y + s_warp[32 + wid];
  tx = s_warp[64];
  ty = s_warp[65];
  __syncthreads();
}

// Grid-wide exclusive scan of two sequences of N items inside the launch.
// CTA b owns the contiguous range [b*span, (b+1)*span): pass 1 sums it, a
// grid barrier publishes the CTA sums, pass 2 scans the range starting from
// the sum of the lower CTAs.  item(i) -> (x, y); out(i, ex, ey) stores.  The
// last CTA stores the totals through tot(tx, ty).  Integer sums: the result
// equals a sequential exclusive scan.  Returns false if the barrier failed.
template <class Item, class Out, class Tot>
__device__ bool fz_grid_scan2(const FusedArgs& a, i64 N, Item item, Out out, Tot tot, i32* s_flag) {
  __shared__ i32 s_warp[66];
  __shared__ i32 s_pre[2];
  const i64 span = (N + gridDim.x - 1) / gridDim.x;
  const i64 lo = (i64)blockIdx.x * span, hi = lo + span < N ? lo + span : N;
  i32 sx = 0, sy = 0;
  for (i64 i = lo + threadIdx.x; i < hi; i += blockDim.x) {
    i32 x, y;
    item(i, x, y);
    sx += x;
    sy += y;
  }
  i32 tx, ty;
  fz_block_exscan2(sx, sy, s_warp, tx, ty);
  if (threadIdx.x == 0) {
    a.partial[2 * blockIdx.x] = tx;
    a.partial[2 * blockIdx.x + 1] = ty;
  }
  if (!grid_barrier(a.bar, a.err, s_flag)) return false;
  if (threadIdx.x < 32) {
    i32 px = 0, py = 0;
    for (i32 b = threadIdx.x; b < (i32)blockIdx.x; b += 32) {
      px += ldcg(a.partial + 2 * b);
      py += ldcg(a.partial + 2 * b + 1);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      px += __shfl_xor_sync(kFull, px, o);
      py += __shfl_xor_sync(kFull, py, o);
    }
    if (threadIdx.x == 0) { s_pre[0] = px; s_pre[1] = py; }
  }
  __syncthreads();
  i32 cx = s_pre[0], cy = s_pre[1];
  for (i64 b0 = lo; b0 < hi; b0 += blockDim.x) {   // block-uniform trip count
    const i64 i = b0 + threadIdx.x;
    i32 x = 0, y = 0;
    if (i < hi) item(i, x, y);
    i32 ex = x, ey = y, bx, by;
    fz_block_exscan2(ex, ey, s_warp, bx, by);
    if (i < hi) out(i, cx + ex, cy + ey);
    cx += bx;
    cy += by;
  }
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) tot(cx, cy);
  return true;
}

__global__ void __launch_bounds__(kFusedThreads, 2) k_coarsen_fused(FusedArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ i32 s_flag, s_any, s_count;
  __shared__ u64 s_off;
  const i32 n = a.n;
  const i64 stride = (i64)gridDim.x * blockDim.x;
  const i64 t0 = (i64)blockIdx.x * blockDim.x + threadIdx.x;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;

  // ---- clear and initialise (the per-phase path's memsets) ----
  for (i64 v = t0; v <= n; v += stride) {
    if (v < n) {
      const u64 key = (u64)(u32)v << 32;
      a.k0[v] = key;
      a.k1[v] = key;
      a.gsize[v] = 0;
      a.gcur[v] = 0;
      a.cvwgt[v] = 0;
    }
    a.rowlen[v] = 0;
    a.mcnt[v] = 0;
    a.cnt[v] = 0;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    a.chg[0] = 0;
    a.chg[1] = 0;
    a.chg[2] = 0;
    a.arena->used = 0;
    a.arena->need = 0;
    a.arena->overflow = 0;
    *a.maxdeg_out = 0;
    *a.max_cvw_out = 0;
  }
  // ---- heavy-edge candidates (coarsen.hpp:39-78) ----
  switch (a.lanes) {
    case 2: fz_match<2>(a); break;
    case 4: fz_match<4>(a); break;
    case 8: fz_match<8>(a); break;
    case 16: fz_match<16>(a); break;
    default: fz_match<32>(a); break;
  }
  if (!grid_barrier(a.bar, a.err, &s_flag)) return;
  if (a.split) {
    fz_match_long(a);
    if (!grid_barrier(a.bar, a.err, &s_flag)) return;
  }

  // ---- union-find rounds (coarsen.hpp:80-118, 461-469) as label raising per round ----
  {
    i32 rounds = -1;
    for (i32 it = 1;; ++it) {
      if (it > a.max_rounds) {   // uniform across CTAs
        if (blockIdx.x == 0 && threadIdx.x == 0) atomicExch(a.err, 2);
        return;
      }
      const u64* src = (it & 1) ? a.k0 : a.k1;   // round it reads buffer (it-1)&1, raises it&1
      u64* dst = (it & 1) ? a.k1 : a.k0;
      if (threadIdx.x == 0) s_any = 0;
      __syncthreads();
      bool diff = false;
      for (i64 v = t0; v < n; v += stride) {
        const i32 c = ldcg(a.cand + v);
        const u64 kv = ldcg(src + v);
        const u64 kc = ldcg(src + c);
        const u32 x = (u32)(kv >> 32), y = (u32)(kc >> 32);
        atomicMax((unsigned long long*)&dst[v], (unsigned long long)kv);
        if (x > y) {
          atomicMax((unsigned long long*)&dst[c], (unsigned long long)(((u64)x << 32) | (u32)it));
          diff = true;
        } else if (x < y) {
          atomicMax((unsigned long long*)&dst[v], (unsigned long long)(((u64)y << 32) | (u32)it));
          diff = true;
        }
      }
      if (diff) s_any = 1;
      __syncthreads();
      if (threadIdx.x == 0 && s_any) atomicOr(&a.chg[it % 3], 1);
      if (blockIdx.x == 0 && threadIdx.x == 0) a.chg[(it + 1) % 3] = 0;
      if (!grid_barrier(a.bar, a.err, &s_flag)) return;
      if (ldcg(&a.chg[it % 3]) == 0) {
        rounds = it;
        break;
      }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) *a.uf_rounds_out = rounds;
  }
  const u64* keys = a.k0;   // both buffers hold the fixed point

  // ---- group sizes (coarsen.hpp:351-359) ----
  for (i64 v = t0; v < n; v += stride) atomicAdd(&a.gsize[(u32)(ldcg(keys + v) >> 32)], 1);
  if (!grid_barrier(a.bar, a.err, &s_flag)) return;
  // ---- coarse ids: ceil(size/cap) per root, scanned; member offsets of big groups ----
  {
    const i32 cap = a.cap;
    auto item = [&](i64 i, i32& x, i32& y) {
      const i32 s = ldcg(a.gsize + i);
      x = (s + cap - 1) / cap;
      y = s > cap ? s : 0;
    };
    auto out = [&](i64 i, i32 ex, i32 ey) {
      a.cbase[i] = ex;
      a.goff[i] = ey;
    };
    auto tot = [&](i32 tx, i32 ty) {
      *a.nc_out = tx;
      a.misc[kFzBig] = ty;
    };
    if (!fz_grid_scan2(a, n, item, out, tot, &s_flag)) return;
  }
  if (!grid_barrier(a.bar, a.err, &s_flag)) return;
  // ---- scatter: cmap of small groups, member lists of big ones (coarsen.hpp:361-421) ----
  for (i64 v = t0; v < n; v += stride) {
    const i32 r = (i32)(u32)(ldcg(keys + v) >> 32);
    const i32 s = ldcg(a.gsize + r);
    if (s <= a.cap) {
      a.cmap[v] = ldcg(a.cbase + r);
    } else {
      const i32 slot = atomicAdd(&a.gcur[r], 1);
      a.members[ldcg(a.goff + r) + slot] = (i32)v;
      if (r == (i32)v) {
        if (s <= 32) a.wlist[atomicAdd(a.misc + kFzWarpG, 1)] = r;
        else if (s <= kGroupSmem) a.clist[atomicAdd(a.misc + kFzCtaG, 1)] = r;
        else a.glist[atomicAdd(a.misc + kFzGiant, 1)] = r;
      }
    }
  }
  if (!grid_barrier(a.bar, a.err, &s_flag)) return;
  // ---- big groups ordered by (dist, id): warps, CTAs, and rare giant groups ----
  {
    const i32 nwg = ldcg(a.misc + kFzWarpG);
    const i64 warp0 = t0 >> 5, nwarps = stride >> 5;
    for (i64 w = warp0; w < nwg; w += nwarps) {
      const i32 r = ldcg(a.wlist + w);
      const i32 s = ldcg(a.gsize + r);
      u64 key = ~0ull;
      if (lane < s) {
        const i32 mb = ldcg(a.members + ldcg(a.goff + r) + lane);
        key = ((ldcg(keys + mb) & 0xffffffffull) << 32) | (u32)mb;   // (dist, id)
      }
#pragma unroll
      for (int kk = 2; kk <= 32; kk <<= 1) {
#pragma unroll
        for (int j = kk >> 1; j > 0; j >>= 1) {
          const u64 o = __shfl_xor_sync(kFull, key, j);
          const bool up = (lane & kk) == 0;
          const bool lower = (lane & j) == 0;
          key = (lower == up) ? umin64(key, o) : umax64(key, o);
        }
      }
      if (lane < s) a.cmap[(u32)key] = ldcg(a.cbase + r) + lane / a.cap;
    }
    const i32 ncg = ldcg(a.misc + kFzCtaG);
    u64* sk = reinterpret_cast<u64*>(smem_raw);
    for (i32 b = blockIdx.x; b < ncg; b += gridDim.x) {
      const i32 r = ldcg(a.clist + b);
      const i32 s = ldcg(a.gsize + r);
      i32 P = 64;
      while (P < s) P <<= 1;
      for (i32 i = threadIdx.x; i < P; i += blockDim.x) {
        u64 key = ~0ull;
        if (i < s) {
          const i32 mb = ldcg(a.members + ldcg(a.goff + r) + i);
          key = ((ldcg(keys + mb) & 0xffffffffull) << 32) | (u32)mb;
        }
        sk[i] = key;
      }
      __syncthreads();
      cta_bitonic_u64(sk, P);
      const i32 cb = ldcg(a.cbase + r);
      for (i32 i = threadIdx.x; i < s; i += blockDim.x) a.cmap[(u32)sk[i]] = cb + i / a.cap;
      __syncthreads();
    }
    const i32 ng = ldcg(a.misc + kFzGiant);   // the same on every CTA
    for (i32 gi = 0; gi < ng; ++gi) {
      const i32 r = ldcg(a.glist + gi);
      const i32 s = ldcg(a.gsize + r);
      i64 P = 1;
      while (P < s) P <<= 1;
      const i32 mo = ldcg(a.goff + r);
      u64* g = a.gscratch;
      for (i64 i = t0; i < P; i += stride) {
        u64 key = ~0ull;
        if (i < s) {
          const i32 mb = ldcg(a.members + mo + i);
          key = ((ldcg(keys + mb) & 0xffffffffull) << 32) | (u32)mb;
        }
        g[i] = key;
      }
      if (!grid_barrier(a.bar, a.err, &s_flag)) return;
      for (i64 kk = 2; kk <= P; kk <<= 1) {
        for (i64 j = kk >> 1; j > 0; j >>= 1) {
          for (i64 i = t0; i < P; i += stride) {
            const i64 l = i ^ j;
            if (l > i) {
              const u64 x = ldcg(g + i), y = ldcg(g + l);
              const bool up = (i & kk) == 0;
              if (up ? (x > y) : (x < y)) { g[i] = y; g[l] = x; }
            }
          }
          if (!grid_barrier(a.bar, a.err, &s_flag)) return;
        }
      }
      const i32 cb = ldcg(a.cbase + r);
      for (i64 i = t0; i < s; i += stride) a.cmap[(u32)ldcg(g + i)] = cb + (i32)(i / a.cap);
      if (!grid_barrier(a.bar, a.err, &s_flag)) return;
    }
  }
  if (!grid_barrier(a.bar, a.err, &s_flag)) return;

  // ---- contraction (coarsen.hpp:157-349) ----
  const i32 cap = a.cap;
  for (i64 v = t0; v < n; v += stride) {   // coarse weights, row lengths, member lists
    const i32 c = ldcg(a.cmap + v);
    atomicAdd((u32*)&a.cvwgt[c], (u32)a.vwgt[v]);
    atomicAdd(&a.rowlen[c], a.xadj[v + 1] - a.xadj[v]);
    const i32 slot = atomicAdd(&a.mcnt[c], 1);
    a.memtab[(i64)c * cap + slot] = (i32)v;
  }
  if (!grid_barrier(a.bar, a.err, &s_flag)) return;
  {   // upper-bound row offsets: exclusive scan of the row lengths (n + 1 entries)
    auto item = [&](i64 i, i32& x, i32& y) {
      x = ldcg(a.rowlen + i);
      y = 0;
    };
    auto out = [&](i64 i, i32 ex, i32) { a.ub[i] = ex; };
    auto tot = [&](i32 tx, i32) { a.misc[kFzUb] = tx; };
    if (!fz_grid_scan2(a, (i64)n + 1, item, out, tot, &s_flag)) return;
  }
  if (!grid_barrier(a.bar, a.err, &s_flag)) return;
  const i32 nc = ldcg(a.nc_out);
  {   // one warp per coarse vertex, as k_contract_warp<128, 8>
    WarpTable<kFusedWcap>& T = reinterpret_cast<WarpTable<kFusedWcap>*>(smem_raw)[wid];
    const i64 nw = (i64)gridDim.x * kFusedWarps;
    for (i64 c = (i64)blockIdx.x * kFusedWarps + wid; c < nc; c += nw) {
      const i32 L = ldcg(a.rowlen + c);
      const i32 nm = ldcg(a.mcnt + c);
      if (L > kFusedWcap || nm > 32) {
        if (lane == 0) a.heavy[atomicAdd(a.misc + kFzHeavy, 1)] = (i32)c;
        continue;
      }
      i32 mbeg = 0, mlen = 0;
      if (lane < nm) {
        const i32 v = ldcg(a.memtab + c * (i64)cap + lane);
        mbeg = a.xadj[v];
        mlen = a.xadj[v + 1] - mbeg;
      }
      i32 moff = mlen;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const i32 y = __shfl_up_sync(kFull, moff, o);
        if (lane >= o) moff += y;
      }
      moff -= mlen;
      auto entry_pos = [&](i32 i) {
        i32 pos = -1;
        for (i32 jm = 0; jm < nm; ++jm) {
          const i32 oj = __shfl_sync(kFull, moff, jm);
          const i32 lj = __shfl_sync(kFull, mlen, jm);
          const i32 bj = __shfl_sync(kFull, mbeg, jm);
          if (i >= oj && i < oj + lj) pos = bj + (i - oj);
        }
        return pos;
      };
      const i32 o = ldcg(a.ub + c);
      if (L <= 32) {
        u64 kv = ~0ull;
        const i32 pos = entry_pos(lane);
        if (lane < L) {
          const u32 key = (u32)ldcg(a.cmap + a.adjncy[pos]);
          if (key != (u32)c) kv = ((u64)key << 32) | (u32)a.adjwgt[pos];
        }
#pragma unroll
        for (int kk = 2; kk <= 32; kk <<= 1) {
#pragma unroll
          for (int jj = kk >> 1; jj > 0; jj >>= 1) {
            const u64 ot = __shfl_xor_sync(kFull, kv, jj);
            const bool up = (lane & kk) == 0;
            const bool lower = (lane & jj) == 0;
            kv = (lower == up) ? umin64(kv, ot) : umax64(kv, ot);
          }
        }
        const u32 key = (u32)(kv >> 32);
        const u32 w = (u32)kv;
        const u32 kprev = __shfl_up_sync(kFull, key, 1);
        const u32 knext = __shfl_down_sync(kFull, key, 1);
        const bool head = lane == 0 || kprev != key;
        const bool last = lane == 31 || knext != key;
        u32 S = w;
        i32 start = head ? lane : 0;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
          const u32 y = __shfl_up_sync(kFull, S, d);
          const i32 z = __shfl_up_sync(kFull, start, d);
          if (lane >= d) {
            S += y;
            start = start > z ? start : z;
          }
        }
        const u32 before = __shfl_sync(kFull, S, start > 0 ? start - 1 : 0);
        const u32 total = S - (start > 0 ? before : 0u);
        const bool valid = last && key != 0xffffffffu;
        const u32 bal = __ballot_sync(kFull, valid);
        if (valid) {
          const i32 at = o + __popc(bal & ((1u << lane) - 1));
          a.sadj[at] = (i32)key;
          a.swgt[at] = (i32)total;
        }
        if (lane == 0) a.cnt[c] = __popc(bal);
        continue;
      }
      u32 hsz = 64;
      while (hsz < 2u * (u32)L) hsz <<= 1;
      for (u32 i = lane; i < hsz; i += 32) { T.keys[i] = kEmpty; T.vals[i] = 0; }
      __syncwarp();
      for (i32 b = 0; b < L; b += 32) {
        const i32 i = b + lane;
        const i32 pos = entry_pos(i);
        if (i < L) {
          const u32 key = (u32)ldcg(a.cmap + a.adjncy[pos]);
          if (key != (u32)c) table_add(T.keys, T.vals, hsz, key, (u32)a.adjwgt[pos]);
        }
      }
      __syncwarp();
      i32 U = 0;
      for (u32 base = 0; base < hsz; base += 32) {
        const u32 sl = base + lane;
        const bool occ = T.keys[sl] != kEmpty;
        const u32 bal = __ballot_sync(kFull, occ);
        if (occ) {
          const i32 at = U + __popc(bal & ((1u << lane) - 1));
          T.out[at] = ((u64)T.keys[sl] << 32) | T.vals[sl];
        }
        U += __popc(bal);
      }
      __syncwarp();
      if (U <= 32) {
        u64 key = lane < U ? T.out[lane] : ~0ull;
#pragma unroll
        for (int kk = 2; kk <= 32; kk <<= 1) {
#pragma unroll
          for (int jj = kk >> 1; jj > 0; jj >>= 1) {
            const u64 ot = __shfl_xor_sync(kFull, key, jj);
            const bool up = (lane & kk) == 0;
            const bool lower = (lane & jj) == 0;
            key = (lower == up) ? umin64(key, ot) : umax64(key, ot);
          }
        }
        if (lane < U) {
          a.sadj[o + lane] = (i32)(u32)(key >> 32);
          a.swgt[o + lane] = (i32)(u32)key;
        }
      } else {
        i32 P = 64;
        while (P < U) P <<= 1;
        for (i32 i = U + lane; i < P; i += 32) T.out[i] = ~0ull;
        __syncwarp();
        warp_bitonic_u64(T.out, P, lane);
        for (i32 i = lane; i < U; i += 32) {
          const u64 kv = T.out[i];
          a.sadj[o + i] = (i32)(u32)(kv >> 32);
          a.swgt[o + i] = (i32)(u32)kv;
        }
      }
      if (lane == 0) a.cnt[c] = U;
      __syncwarp();
    }
  }
  if (!grid_barrier(a.bar, a.err, &s_flag)) return;
  {   // heavy coarse rows, one CTA each: the shared table, or the arena beyond kFusedCtaCap
    const i32 nh = ldcg(a.misc + kFzHeavy);
    for (i32 b = blockIdx.x; b < nh; b += gridDim.x) {
      const i32 c = ldcg(a.heavy + b);
      const i32 L = ldcg(a.rowlen + c);
      const bool global_table = L > kFusedCtaCap;
      const u32 hsz = table_slots((u32)L);
      u32 *tk, *tv;
      u64* out;
      if (global_table) {
        const u64 words = 3ull * hsz;   // keys + vals + hsz/2 u64 outputs
        if (threadIdx.x == 0) {
          const u64 off = atomicAdd((unsigned long long*)&a.arena->used, (unsigned long long)words);
          if (off + words > a.arena_cap) {
            atomicAdd((unsigned long long*)&a.arena->need, (unsigned long long)words);
            atomicExch(&a.arena->overflow, 1);
            s_off = ~0ull;
          } else {
            s_off = off;
          }
        }
        __syncthreads();
        const u64 off = s_off;
        __syncthreads();   // every thread has read s_off before thread 0 can set it for the next row
        if (off == ~0ull) continue;   // block-uniform; the level is redone after the arena grows
        tk = a.arena_words + off;
        tv = tk + hsz;
        out = reinterpret_cast<u64*>(tv + hsz);
      } else {
        tk = reinterpret_cast<u32*>(smem_raw);
        tv = tk + 2 * kFusedCtaCap;
        out = reinterpret_cast<u64*>(tv + 2 * kFusedCtaCap);
      }
      for (u32 i = threadIdx.x; i < hsz; i += blockDim.x) { tk[i] = kEmpty; tv[i] = 0; }
      if (threadIdx.x == 0) s_count = 0;
      __syncthreads();
      const i32 nm = ldcg(a.mcnt + c);
      for (i32 j = 0; j < nm; ++j) {
        const i32 v = ldcg(a.memtab + c * (i64)cap + j);
        const i32 beg = a.xadj[v], end = a.xadj[v + 1];
        for (u32 e = (u32)beg + threadIdx.x; e < (u32)end; e += blockDim.x) {
          const u32 key = (u32)ldcg(a.cmap + a.adjncy[e]);
          if (key != (u32)c) table_add(tk, tv, hsz, key, (u32)a.adjwgt[e]);
        }
      }
      __syncthreads();
      for (u32 sl = threadIdx.x; sl < hsz; sl += blockDim.x) {
        if (tk[sl] != kEmpty) {
          const i32 pos = atomicAdd(&s_count, 1);
          out[pos] = ((u64)tk[sl] << 32) | tv[sl];
        }
      }
      __syncthreads();
      const i32 U = s_count;
      i32 P = 64;
      while (P < U) P <<= 1;
      for (i32 i = U + threadIdx.x; i < P; i += blockDim.x) out[i] = ~0ull;
      __syncthreads();
      cta_bitonic_u64(out, P);
      const i32 o = ldcg(a.ub + c);
      for (i32 i = threadIdx.x; i < U; i += blockDim.x) {
        const u64 kv = out[i];
        a.sadj[o + i] = (i32)(u32)(kv >> 32);
        a.swgt[o + i] = (i32)(u32)kv;
      }
      if (threadIdx.x == 0) a.cnt[c] = U;
      __syncthreads();
    }
  }
  if (!grid_barrier(a.bar, a.err, &s_flag)) return;
  {   // coarse xadj: exclusive scan of the row counts (rows beyond n_c are empty)
    auto item = [&](i64 i, i32& x, i32& y) {
      x = ldcg(a.cnt + i);
      y = 0;
    };
    auto out = [&](i64 i, i32 ex, i32) { a.cxadj[i] = ex; };
    auto tot = [&](i32 tx, i32) { *a.mc_out = tx; };
    if (!fz_grid_scan2(a, (i64)n + 1, item, out, tot, &s_flag)) return;
  }
  if (!grid_barrier(a.bar, a.err, &s_flag)) return;
  {   // compact the rows (one warp per 32 rows, as k_copy_rows); longest row, heaviest vertex
    const i64 warp = t0 >> 5, nwarps = stride >> 5;
    i32 mx = 0, mw = 0;
    for (i64 c0 = warp * 32; c0 < nc; c0 += nwarps * 32) {
      const i64 c = c0 + lane;
      i32 src = 0, dst = 0, len = 0;
      if (c < nc) {
        src = ldcg(a.ub + c);
        dst = ldcg(a.cxadj + c);
        len = ldcg(a.cnt + c);
        const i32 w = ldcg(a.cvwgt + c);
        mw = w > mw ? w : mw;
      }
      mx = len > mx ? len : mx;
      i32 inc = len;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const i32 y = __shfl_up_sync(kFull, inc, o);
        if (lane >= o) inc += y;
      }
      const i32 total = __shfl_sync(kFull, inc, 31);
      const i32 exc = inc - len;
      for (i32 base = 0; base < total; base += 32) {
        const i32 idx = base + lane;
        i32 r = 0;
#pragma unroll
        for (int step = 16; step > 0; step >>= 1) {
          const i32 probe = __shfl_sync(kFull, inc, r + step - 1);
          if (probe <= idx) r += step;
        }
        r = r < 31 ? r : 31;
        const i32 rs = __shfl_sync(kFull, src, r), rd = __shfl_sync(kFull, dst, r), re = __shfl_sync(kFull, exc, r);
        if (idx < total) {
          a.cadjncy[rd + (idx - re)] = ldcg(a.sadj + rs + (idx - re));
          a.cadjwgt[rd + (idx - re)] = ldcg(a.swgt + rs + (idx - re));
        }
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const i32 y = __shfl_xor_sync(kFull, mx, o);
      mx = mx > y ? mx : y;
      const i32 z = __shfl_xor_sync(kFull, mw, o);
      mw = mw > z ? mw : z;
    }
    if (lane == 0 && mx > 0) atomicMax(a.maxdeg_out, mx);
    if (lane == 0 && mw > 0) atomicMax(a.max_cvw_out, mw);
  }
}

static int fused_blocks_per_sm() {
  static int bps = -1;   // the same on every device of the process (one B200 model)
  if (bps < 0) {
    int b = 0;
    if (cudaFuncSetAttribute(k_coarsen_fused, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFusedSmem) !=
            cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_coarsen_fused, kFusedThreads, kFusedSmem) !=
            cudaSuccess) {
      cudaGetLastError();
      b = 0;
    }
    bps = b;
  }
  return bps;
}

// Whether a level runs as one fused launch: levels of at most the handle's
// fused_max_n vertices whose rows are short on average (long coarse rows are
// the per-phase path's wide warp tables), never while the tuner times the
// match variants.
static bool use_fused(Handle& h, const DevGraph& g) {
  return !h.tune_collect && g.n > 0 && (i64)g.n <= (i64)h.tuning.coarsen_fused_max_n &&
         (double)g.m <= 48.0 * (double)g.n && fused_blocks_per_sm() >= 1;
}

static void run_coarsen_fused(Handle& h, const DevGraph& g, i32 cap, CoarsenOut& out) {
  if (!h.capturing)   // per device (the occupancy probe set it on the first device only)
    GKW_CUDA(cudaFuncSetAttribute(k_coarsen_fused, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFusedSmem));
  Pool::Mark mk = h.scratch.mark();
  const i32 n = g.n;
  const i64 nu = (i64)n + 1;
  const i32 bps = fused_blocks_per_sm();
  const i32 vpc = std::max(64, h.tuning.coarsen_verts_per_cta);
  i32 grid = (i32)std::min<i64>((i64)h.sm_count * bps, std::max<i64>(1, ((i64)n + vpc - 1) / vpc));
  grid = coop_grid(h, (const void*)k_coarsen_fused, grid, kFusedThreads, kFusedSmem);
  FusedArgs a;
  a.n = n;
  a.m = g.m;
  a.xadj = g.xadj;
  a.adjncy = g.adjncy;
  a.adjwgt = g.adjwgt;
  a.vwgt = g.vwgt;
  a.lanes = h.tuning.match_lanes[match_bucket(g)];
  a.split = g.maxdeg < 0 || g.maxdeg > kMatchLong;
  a.cap = cap;
  a.max_rounds = n + 2;
  a.cmap = out.cmap;
  a.cxadj = out.cxadj;
  a.cadjncy = out.cadjncy;
  a.cadjwgt = out.cadjwgt;
  a.cvwgt = out.cvwgt;
  a.cand = h.scratch.alloc_n<i32>(n);
  a.k0 = h.scratch.alloc_n<u64>(n);
  a.k1 = h.scratch.alloc_n<u64>(n);
  a.chg = h.scratch.alloc_n<i32>(4);
  a.longlist = h.scratch.alloc_n<i32>(n);
  a.gsize = h.scratch.alloc_n<i32>(n);
  a.cbase = h.scratch.alloc_n<i32>(n);
  a.goff = h.scratch.alloc_n<i32>(n);
  a.gcur = h.scratch.alloc_n<i32>(n);
  a.members = h.scratch.alloc_n<i32>(n);
  a.wlist = h.scratch.alloc_n<i32>(n);
  a.clist = h.scratch.alloc_n<i32>(n);
  a.glist = h.scratch.alloc_n<i32>(n);
  a.gscratch = h.scratch.alloc_n<u64>(2 * (size_t)n);
  a.rowlen = h.scratch.alloc_n<i32>(nu);
  a.ub = h.scratch.alloc_n<i32>(nu);
  a.mcnt = h.scratch.alloc_n<i32>(nu);
  a.memtab = h.scratch.alloc_n<i32>((i64)n * cap + 1);
  a.cnt = h.scratch.alloc_n<i32>(nu);
  a.heavy = h.scratch.alloc_n<i32>(nu);
  a.sadj = h.scratch.alloc_n<i32>(std::max<i64>(g.m, 1));
  a.swgt = h.scratch.alloc_n<i32>(std::max<i64>(g.m, 1));
  a.partial = h.scratch.alloc_n<i32>(2 * (size_t)grid);
  a.misc = h.scratch.alloc_n<i32>(kFzWords);
  a.bar = &h.coop->bar;
  a.err = &h.coop->err;
  a.nc_out = &h.coop->nc;
  a.mc_out = &h.coop->mc;
  a.uf_rounds_out = &h.coop->uf_rounds;
  a.maxdeg_out = &h.coop->maxdeg;
  a.max_cvw_out = &h.coop->max_cvw;
  a.arena = h.arena;
  a.arena_words = reinterpret_cast<u32*>(h.arena + 1);
  a.arena_cap = h.arena_words;
  GKW_CUDA(cudaMemsetAsync(a.misc, 0, sizeof(i32) * kFzWords, h.stream));
  void* args[] = {&a};
  launch_coop(h, (const void*)k_coarsen_fused, grid, kFusedThreads, kFusedSmem, args);
  h.scratch.release(mk);
}

// The key of one level's launch sequence in the handle's graph cache:
// everything the launches depend on.
static std::string level_key(const Handle& h, const DevGraph& g, i32 cap, const CoarsenOut& out) {
  struct K {
    i64 n, m, maxdeg, cap;
    const void* in[4];
    const void* outp[5];
    const void* sbase;
    size_t stop;
    gkw_tuning tuning;
    i32 narrow, sms;
    const void* arena;
    u64 arena_words;
    const void* scan;
  } k;
  memset(&k, 0, sizeof(k));
  k.n = g.n;
  k.m = g.m;
  k.maxdeg = g.maxdeg;
  k.cap = cap;
  k.in[0] = g.xadj;
  k.in[1] = g.adjncy;
  k.in[2] = g.adjwgt;
  k.in[3] = g.vwgt;
  k.outp[0] = out.cmap;
  k.outp[1] = out.cxadj;
  k.outp[2] = out.cvwgt;
  k.outp[3] = out.cadjncy;
  k.outp[4] = out.cadjwgt;
  const auto fp = h.scratch.fingerprint();
  k.sbase = fp.first;
  k.stop = fp.second;
  k.tuning = h.tuning;
  k.narrow = h.narrow;
  k.sms = h.sm_count;
  k.arena = h.arena;
  k.arena_words = h.arena_words;
  k.scan = h.scan;
  return std::string("level", 5) + std::string(reinterpret_cast<const char*>(&k), sizeof(k));
}

// One coarsening step.  Its launch sequence (six kernels on a small level,
// about fifteen and two clears on a large one, all sized by the level's n and
// m) runs through the handle's graph
// cache: repeated partitions of the same graph replay it as one CUDA graph.
// One host sync per level reads the coarse sizes.
void coarsen_level(Handle& h, const DevGraph& g, i32 cap, CoarsenOut& out) {
  // coarse arrays at upper bounds (n_c <= n, m_c <= m)
  out.cmap = h.hier.alloc_n<i32>(std::max(g.n, 1));
  out.cxadj = h.hier.alloc_n<i32>((i64)g.n + 1);
  out.cvwgt = h.hier.alloc_n<i32>(std::max(g.n, 1));
  out.cadjncy = h.hier.alloc_n<i32>(std::max<i64>(g.m, 1));
  out.cadjwgt = h.hier.alloc_n<i32>(std::max<i64>(g.m, 1));
  ensure_arena(h, u64(4) << 20);   // never inside a capture
  const bool tune = h.tune_collect;
  auto body = [&] {
    Pool::Mark mk = h.scratch.mark();
    if (g.n <= kSmallLevel || tune) {
      i32* cand = h.scratch.alloc_n<i32>(std::max(g.n, 1));
      if (tune) time_match_variants(h, g, cand);
      if (g.n <= kSmallLevel) {
        run_match(h, g, cand, g.maxdeg);
        run_small_level(h, g, cand, cap, out);
      }
      h.scratch.release(mk);
    }
    if (g.n > kSmallLevel) run_large_level(h, g, cap, out);
  };
  bool reported = false;
  if (use_fused(h, g)) {
    // one launch: no graph needed (a launch is as cheap as a graph of one)
    run_coarsen_fused(h, g, cap, out);
  } else if (tune) {
    body();   // the tuner's timings synchronise: never captured
  } else {
    graph_run(h, level_key(h, g, cap, out), [&] {
      body();
      report_coop(h);
    });
    reported = true;
  }
  CoopState c = read_coop(h, reported);
  if (c.arena_overflow) {   // very long coarse rows: grow the arena and redo the step
    ensure_arena(h, (u64)((double)(h.arena_words + (u64)c.arena_need) * 1.25) + 1024);
    run_contract(h, g, out.cmap, &h.coop->nc, g.n, cap, out.cxadj, out.cadjncy, out.cadjwgt, out.cvwgt,
                 &h.coop->mc);
    c = read_coop(h);
    GKW_REQUIRE(!c.arena_overflow, GKW_E_INTERNAL, "long-row arena overflow after growth");
  }
  out.nc = c.nc;
  out.mc = c.mc;
  out.uf_rounds = c.uf_rounds;
  out.max_cvw = c.max_cvw;
  out.maxdeg = c.maxdeg;
}

}  // namespace gkw
