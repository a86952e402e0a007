// Errors, the device pool, handles and the device-wide exclusive scan.
#include <algorithm>
#include <atomic>
#include <cstdio>
#include <cstring>
#include <exception>
#include <map>
#include <mutex>
#include <thread>

#include "gkw_internal.cuh"

namespace gkw {

static thread_local std::string g_last_error;
static std::atomic<uint64_t> g_launches{0};

void count_launch() { g_launches.fetch_add(1, std::memory_order_relaxed); }
void count_launches(uint64_t n) { g_launches.fetch_add(n, std::memory_order_relaxed); }
void uncount_launches(uint64_t n) { g_launches.fetch_sub(n, std::memory_order_relaxed); }
uint64_t launch_total() { return g_launches.load(std::memory_order_relaxed); }

void set_error(const std::string& msg) { g_last_error = msg; }
const char* last_error_cstr() { return g_last_error.c_str(); }

}  // namespace gkw

// error hook for the host-only file helpers (graph_io.cpp)
extern "C" void gkw_io_set_error(const std::string& msg) { gkw::set_error(msg); }

namespace gkw {

// ---------------------------------------------------------------------------
// Pool
// ---------------------------------------------------------------------------
Pool::~Pool() {
  for (auto& c : chunks_) cudaFree(c.base);
}

static size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

void* Pool::alloc(size_t bytes) {
  bytes = align_up(bytes == 0 ? 1 : bytes, 256);
  while (cur_ < chunks_.size()) {
    Chunk& c = chunks_[cur_];
    if (c.top + bytes <= c.cap) {
      void* p = c.base + c.top;
      c.top += bytes;
      note_use();
      return p;
    }
    if (cur_ + 1 < chunks_.size()) {
      ++cur_;
      chunks_[cur_].top = 0;
      continue;
    }
    break;
  }
  // need a new chunk (appended after the current one)
  size_t cap = std::max(bytes, min_chunk_);
  if (!chunks_.empty()) cap = std::max(cap, chunks_.back().cap);   // geometric-ish growth
  char* base = nullptr;
  cudaError_t e = cudaMalloc(&base, cap);
  if (e != cudaSuccess) {
    cudaGetLastError();
    throw Error{GKW_E_NOMEM, "device allocation of " + std::to_string(cap) + " bytes failed: " +
                                 cudaGetErrorString(e)};
  }
  chunks_.push_back({base, cap, bytes});
  cur_ = chunks_.size() - 1;
  note_use();
  return base;
}

void Pool::note_use() {
  size_t used = chunks_[cur_].top;
  for (size_t i = 0; i < cur_; ++i) used += chunks_[i].cap;
  peak_ = std::max(peak_, used);
}

void Pool::trim() {
  for (auto& c : chunks_) GKW_REQUIRE(c.top == 0, GKW_E_INTERNAL, "trim of a pool in use");
  for (auto& c : chunks_) cudaFree(c.base);
  chunks_.clear();
  cur_ = 0;
}

void Pool::release(Mark m) {
  if (chunks_.empty()) return;
  cur_ = m.chunk;
  chunks_[cur_].top = m.top;
  for (size_t i = cur_ + 1; i < chunks_.size(); ++i) chunks_[i].top = 0;
}

size_t Pool::capacity() const {
  size_t s = 0;
  for (auto& c : chunks_) s += c.cap;
  return s;
}

void Pool::reserve(size_t bytes) {
  if (!chunks_.empty() && chunks_[0].cap >= bytes) return;
  bool all_free = true;
  for (auto& c : chunks_) all_free &= (c.top == 0);
  if (!all_free) return;
  for (auto& c : chunks_) cudaFree(c.base);
  chunks_.clear();
  cur_ = 0;
  char* base = nullptr;
  cudaError_t e = cudaMalloc(&base, bytes);
  if (e != cudaSuccess) {
    cudaGetLastError();
    throw Error{GKW_E_NOMEM, "device allocation of " + std::to_string(bytes) + " bytes failed: " +
                                 cudaGetErrorString(e)};
  }
  chunks_.push_back({base, bytes, 0});
}

// ---------------------------------------------------------------------------
// Device-wide exclusive scan (reduce, scan the tile sums, scan down).
// ---------------------------------------------------------------------------
constexpr int kScanThreads = 256;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanThreads * kScanItems;

// Exclusive block scan of one value per thread; returns the block total.
__device__ __forceinline__ i32 block_exclusive_scan(i32 x, i32* s_warp, i32& total) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  i32 inc = x;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    i32 y = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += y;
  }
  if (lane == 31) s_warp[wid] = inc;
  __syncthreads();
  if (wid == 0) {
    const int nw = blockDim.x >> 5;
    i32 w = lane < nw ? s_warp[lane] : 0;
    i32 wi = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      i32 y = __shfl_up_sync(0xffffffffu, wi, o);
      if (lane >= o) wi += y;
    }
    if (lane < nw) s_warp[lane] = wi - w;   // exclusive warp offsets
    if (lane == nw - 1) s_warp[32] = wi;     // block total
  }
  __syncthreads();
  i32 r = inc - x + s_warp[wid];
  total = s_warp[32];
  __syncthreads();   // s_warp reusable by the caller afterwards
  return r;
}

// Single-pass scan with decoupled look-back.  Tile t publishes its aggregate
// (status 1) and then its inclusive prefix (status 2) in a status word
// (epoch << 34 | status << 32 | value); a word of an older epoch reads as
// "not published".  Tiles take tickets in launch order, so a tile only waits
// on tiles that already hold an SM.  The ticket counter, the epoch and a
// finished-tile counter live on the device: the last tile to finish resets
// the counters and advances the epoch for the next scan, so a scan needs no
// per-call argument from the host (it can be replayed from a CUDA graph).  A
// wait longer than kScanSpinCycles sets the error word and the tile
// continues (the result is then reported as an error, never a hang).
constexpr long long kScanSpinCycles = 2000000000ll;
constexpr u32 kScanEpochMask = (1u << 29) - 1;

__device__ __forceinline__ u64 ld_relaxed_gpu_u64(const unsigned long long* p) {
  u64 v;
  asm volatile("ld.relaxed.gpu.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}

// What a scan's threads load: eight consecutive values each, as 16-byte words
// where the array allows it.
//   kScanChunks  the input holds group sizes and the values scanned are the
//     coarse ids each group takes, ceil(size / cap); a group above the cap also
//     takes its block of the member list here, from a counter with one atomic
//     per warp (the blocks' order does not matter, since every group is
//     ordered within its own block); (size, first id) pairs go out
//   kScanSums    the input holds 64-bit words, weight << 32 | row length: the
//     lengths are scanned, and both halves are written out as arrays; `last`
//     is cleared at the scan's last element
enum { kScanPlain, kScanChunks, kScanSums };
struct ScanExtra {
  i32 cap = 1;
  i32* goff = nullptr;       // chunks: block of a group above the cap
  i32* mcounter = nullptr;
  i32 *weight = nullptr, *length = nullptr, *last = nullptr;   // sums
};

template <int kMode>
__device__ __forceinline__ i32 scan_load(const i32* in, i64 b0, i64 n, const ScanExtra& ca, i32 (&v)[kScanItems]) {
  static_assert(kScanItems == 8, "two 16-byte words");
  if (kMode == kScanSums) {
    const ulonglong2* p = reinterpret_cast<const ulonglong2*>(reinterpret_cast<const u64*>(in) + b0);
    u64 w[kScanItems];
#pragma unroll
    for (int i = 0; i < kScanItems; i += 2) {   // (the word array is padded to whole pairs)
      const ulonglong2 x = b0 + i < n ? p[i / 2] : make_ulonglong2(0, 0);
      w[i] = x.x;
      w[i + 1] = b0 + i + 1 < n ? x.y : 0;
    }
    i32 sum = 0;
    i32 wt[kScanItems];
#pragma unroll
    for (int i = 0; i < kScanItems; ++i) {
      v[i] = (i32)(u32)w[i];
      wt[i] = (i32)(u32)(w[i] >> 32);
      sum += v[i];
    }
    if (b0 + kScanItems < n) {   // (both arrays are the pool's: aligned)
      int4* pl = reinterpret_cast<int4*>(ca.length + b0);
      int4* pw = reinterpret_cast<int4*>(ca.weight + b0);
      pl[0] = make_int4(v[0], v[1], v[2], v[3]);
      pl[1] = make_int4(v[4], v[5], v[6], v[7]);
      pw[0] = make_int4(wt[0], wt[1], wt[2], wt[3]);
      pw[1] = make_int4(wt[4], wt[5], wt[6], wt[7]);
    } else {
#pragma unroll
      for (int i = 0; i < kScanItems; ++i) {
        if (b0 + i < n) ca.length[b0 + i] = v[i];
        if (b0 + i < n - 1) ca.weight[b0 + i] = wt[i];
        if (b0 + i == n - 1) ca.last[b0 + i] = 0;
      }
    }
    return sum;
  }
  if (b0 + kScanItems <= n && (reinterpret_cast<uintptr_t>(in) & 15) == 0) {
    const int4 x = *reinterpret_cast<const int4*>(in + b0), y = *reinterpret_cast<const int4*>(in + b0 + 4);
    v[0] = x.x, v[1] = x.y, v[2] = x.z, v[3] = x.w, v[4] = y.x, v[5] = y.y, v[6] = y.z, v[7] = y.w;
  } else {
#pragma unroll
    for (int i = 0; i < kScanItems; ++i) v[i] = (b0 + i < n) ? in[b0 + i] : 0;
  }
  if (kMode == kScanChunks) {
    i32 big = 0;
#pragma unroll
    for (int i = 0; i < kScanItems; ++i) big += v[i] > ca.cap ? v[i] : 0;
    const int lane = threadIdx.x & 31;
    i32 inc = big;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const i32 y = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += y;
    }
    i32 base = 0;
    if (lane == 31 && inc) base = atomicAdd(ca.mcounter, inc);
    base = __shfl_sync(0xffffffffu, base, 31) + inc - big;
#pragma unroll
    for (int i = 0; i < kScanItems; ++i) {
      if (v[i] > ca.cap) {
        ca.goff[b0 + i] = base;
        base += v[i];
        v[i] = (v[i] - 1) / ca.cap + 1;
      } else {
        v[i] = v[i] > 0;
      }
    }
  }
  i32 sum = 0;
#pragma unroll
  for (int i = 0; i < kScanItems; ++i) sum += v[i];
  return sum;
}

// kScanChunks: `size` holds the group sizes
template <int kMode>
__device__ __forceinline__ void scan_store(i32* out, i64 b0, i64 n, i32 run, const i32 (&v)[kScanItems],
                                           const i32* size) {
  if constexpr (kMode == kScanChunks) {   // (pairs of records, aligned as `out` is: the pool's)
    int4* rec = reinterpret_cast<int4*>(out) + b0 / 2;
#pragma unroll
    for (int i = 0; i < kScanItems; i += 2) {
      const i32 a = run, b = run + v[i];
      run = b + v[i + 1];
      if (b0 + i + 1 < n) rec[i / 2] = make_int4(size[b0 + i], a, size[b0 + i + 1], b);
      else if (b0 + i < n) reinterpret_cast<int2*>(out)[b0 + i] = make_int2(size[b0 + i], a);
    }
    return;
  } else {
    i32 r[kScanItems];
#pragma unroll
    for (int i = 0; i < kScanItems; ++i) {
      r[i] = run;
      run += v[i];
    }
    if (b0 + kScanItems <= n && (reinterpret_cast<uintptr_t>(out) & 15) == 0) {
      *reinterpret_cast<int4*>(out + b0) = make_int4(r[0], r[1], r[2], r[3]);
      *reinterpret_cast<int4*>(out + b0 + 4) = make_int4(r[4], r[5], r[6], r[7]);
    } else {
#pragma unroll
      for (int i = 0; i < kScanItems; ++i)
        if (b0 + i < n) out[b0 + i] = r[i];
    }
  }
}

// d_last: the scan ends with element *d_last (at most n - 1): a level's coarse
// arrays are sized by its fine vertices, and three of four of their tiles lie
// beyond n_c.
template <int kMode>
__global__ void __launch_bounds__(kScanThreads) k_scan_1pass(const i32* in, i32* out, i64 n, const i32* d_last,
                                                             i32* total, ScanState* ss, i32 ntiles, ScanExtra ca) {
  __shared__ i32 s_warp[33];
  __shared__ i32 s_tile;
  __shared__ i32 s_excl;
  __shared__ u32 s_epoch;
  if (threadIdx.x == 0) {
    s_tile = (i32)atomicAdd(&ss->ticket, 1u);
    s_epoch = *(volatile u32*)&ss->epoch;   // set by the previous scan, stream-ordered before this one
  }
  if (d_last) {
    const i64 last = *d_last;
    n = last + 1 < n ? last + 1 : n;
  }
  __syncthreads();
  const i32 tile = s_tile;
  const u64 epoch = s_epoch;
  const i64 b0 = (i64)tile * kScanTile + (i64)threadIdx.x * kScanItems;
  if ((i64)tile * kScanTile < n) {   // (no tile looks back at one beyond the end)
    i32 v[kScanItems];
    const i32 sum = scan_load<kMode>(in, b0, n, ca, v);
    i32 agg;
    const i32 off = block_exclusive_scan(sum, s_warp, agg);
    if (threadIdx.x < 32) {
      // warp 0 looks back 32 predecessors per step: every lane waits for its
      // predecessor's word, the nearest inclusive prefix ends the walk
      const int lane = threadIdx.x;
      unsigned long long* st = (unsigned long long*)ss->tiles;
      const u64 tag = epoch << 34;
      i32 excl = 0;
      if (tile == 0) {
        if (lane == 0) atomicExch(&st[0], (unsigned long long)(tag | (2ull << 32) | (u32)agg));
      } else {
        if (lane == 0) atomicExch(&st[tile], (unsigned long long)(tag | (1ull << 32) | (u32)agg));
        i64 hi = (i64)tile - 1;
        const long long t0 = clock64();
        for (;;) {
          const i64 j = hi - lane;
          u32 status = 2, val = 0;   // before tile 0: an empty prefix
          if (j >= 0) {
            for (;;) {
              const u64 w = ld_relaxed_gpu_u64(&st[j]);
              status = (w >> 34) == epoch ? (u32)((w >> 32) & 3u) : 0u;
              val = (u32)w;
              if (status != 0) break;
              if (clock64() - t0 > kScanSpinCycles) {
                atomicExch(&ss->err, 1);
                status = 2;
                val = 0;
                break;
              }
            }
          }
          const u32 m2 = __ballot_sync(0xffffffffu, status == 2);
          const int first2 = m2 ? __ffs(m2) - 1 : 32;   // nearest published prefix
          i32 add = lane <= first2 ? (i32)val : 0;
  #pragma unroll
          for (int o = 16; o > 0; o >>= 1) add += __shfl_xor_sync(0xffffffffu, add, o);
          excl += add;
          if (m2) break;
          hi -= 32;
        }
        if (lane == 0) atomicExch(&st[tile], (unsigned long long)(tag | (2ull << 32) | (u32)(excl + agg)));
      }
      if (lane == 0) {
        s_excl = excl;
        if (tile == (i32)((n - 1) / kScanTile) && total) *total = excl + agg;
      }
    }
    __syncthreads();
    scan_store<kMode>(out, b0, n, off + s_excl, v, in);
  }
  if (threadIdx.x == 0) {
    // the last tile to finish: every other tile has taken its ticket, read
    // the epoch and published; reset for the next scan
    __threadfence();
    if (atomicAdd(&ss->done, 1u) == (u32)ntiles - 1) {
      ss->ticket = 0;
      ss->done = 0;
      ss->epoch = (ss->epoch + 1) & kScanEpochMask;
      __threadfence();
    }
  }
}

__global__ void k_set_i32(i32* p, i32 v) { *p = v; }

// A scan that fits one tile: one CTA, no tickets, status words or look-back
// (the single-pass scan's bookkeeping is several dependent round trips to L2,
// most of a small scan's time).
template <int kMode>
__global__ void __launch_bounds__(kScanThreads) k_scan_small(const i32* in, i32* out, i32 n, const i32* d_last,
                                                             i32* total, ScanExtra ca) {
  __shared__ i32 s_warp[33];
  const i32 b0 = threadIdx.x * kScanItems;
  if (d_last) {
    const i32 last = *d_last;
    n = last < n ? last + 1 : n;
  }
  i32 v[kScanItems];
  const i32 sum = scan_load<kMode>(in, b0, n, ca, v);
  i32 agg;
  const i32 run = block_exclusive_scan(sum, s_warp, agg);
  scan_store<kMode>(out, b0, n, run, v, in);
  if (threadIdx.x == 0 && total) *total = agg;
}

template <int kMode>
static void scan_i32(Handle& h, const i32* in, i32* out, i64 n, i32* total, const i32* d_last, ScanExtra ca) {
  if (n <= 0) {
    if (total) launch(k_set_i32, 1, 1, 0, h.stream, total, 0);
    GKW_CHECK_LAUNCH();
    return;
  }
  if (n <= kScanTile) {
    launch(k_scan_small<kMode>, 1, kScanThreads, 0, h.stream, in, out, (i32)n, d_last, total, ca);
    GKW_CHECK_LAUNCH();
    return;
  }
  const i64 nt64 = (n + kScanTile - 1) / kScanTile;
  GKW_REQUIRE(nt64 < (i64)1 << 30, GKW_E_UNSUPPORTED, "scan too large");
  const i32 nt = (i32)nt64;
  // the device epoch wraps after 2^29 scans: before it could meet a status
  // word of the same epoch, start again from cleared state (never inside a
  // graph capture: a captured scan's epoch is read on the device)
  const bool fresh = h.scan_tiles_cap < nt || (h.scan_epoch >= kScanEpochMask - 4096 && !h.capturing);
  if (fresh) {
    GKW_REQUIRE(!h.capturing, GKW_E_INTERNAL, "scan state grown during a graph capture");
    // queued scans may still use the old state; the new state is cleared on
    // the handle's stream (which does not wait for the legacy stream), so the
    // scan below sees it cleared
    GKW_CUDA(cudaStreamSynchronize(h.stream));
    const i32 cap = std::max(nt, h.scan_tiles_cap < nt ? std::max(nt, 1024) : h.scan_tiles_cap);
    if (h.scan_tiles_cap < nt) {
      if (h.scan) GKW_CUDA(cudaFree(h.scan));
      h.scan = nullptr;
      GKW_CUDA(cudaMalloc(&h.scan, sizeof(ScanState) + sizeof(u64) * (size_t)cap));
      h.scan_tiles_cap = cap;
      graph_cache_clear(h);   // graphs hold the old state's address
    }
    GKW_CUDA(cudaMemsetAsync(h.scan, 0, sizeof(ScanState) + sizeof(u64) * (size_t)h.scan_tiles_cap, h.stream));
    h.scan_epoch = 0;
  }
  h.scan_epoch += 1;   // host mirror of the device epoch (wrap guard only)
  ++h.scans_enqueued;
  launch(k_scan_1pass<kMode>, nt, kScanThreads, 0, h.stream, in, out, n, d_last, total, h.scan, nt, ca);
  GKW_CHECK_LAUNCH();
}

void exclusive_scan_i32(Handle& h, const i32* in, i32* out, i64 n, i32* total, const i32* d_last) {
  scan_i32<kScanPlain>(h, in, out, n, total, d_last, ScanExtra{});
}

void scan_group_chunks(Handle& h, const i32* gsize, int2* grec, i32* goff, i32* mcounter, i64 n, i32 cap, i32* total) {
  ScanExtra x;
  x.cap = cap;
  x.goff = goff;
  x.mcounter = mcounter;
  scan_i32<kScanChunks>(h, gsize, reinterpret_cast<i32*>(grec), n, total, nullptr, x);
}

void scan_coarse_sums(Handle& h, const u64* sums, i32* ub, i32* rowlen, i32* cvwgt, i32* cnt, i64 n, i32* total,
                      const i32* d_last) {
  ScanExtra x;
  x.weight = cvwgt;
  x.length = rowlen;
  x.last = cnt;
  scan_i32<kScanSums>(h, reinterpret_cast<const i32*>(sums), ub, n, total, d_last, x);
}

namespace {
struct ClusterKey {
  const void* kern;
  i32 block;
  size_t smem;
  int device;
  bool operator<(const ClusterKey& o) const {
    if (kern != o.kern) return kern < o.kern;
    if (block != o.block) return block < o.block;
    if (smem != o.smem) return smem < o.smem;
    return device < o.device;
  }
};
std::mutex g_cluster_mu;
std::map<ClusterKey, i32> g_cluster_limit;
constexpr int kMaxDevices = 64;
std::mutex g_chain_mu[kMaxDevices];
cudaEvent_t g_chain_last[kMaxDevices] = {};
}  // namespace

i32 coop_cluster_limit(Handle& h, const void* kern, i32 block, size_t smem) {
  const ClusterKey key{kern, block, smem, h.device};
  {
    std::lock_guard<std::mutex> lk(g_cluster_mu);
    auto it = g_cluster_limit.find(key);
    if (it != g_cluster_limit.end()) return it->second;
  }
  i32 best = 1;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)
    cudaGetLastError();
  for (i32 c = 16; c >= 2; c >>= 1) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(c);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = c;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int nclusters = 0;
    if (cudaOccupancyMaxActiveClusters(&nclusters, kern, &cfg) == cudaSuccess && nclusters >= 1) {
      best = c;
      break;
    }
    cudaGetLastError();
  }
  std::lock_guard<std::mutex> lk(g_cluster_mu);
  g_cluster_limit[key] = best;
  return best;
}

i32 coop_grid(Handle& h, const void* kern, i32 want, i32 block, size_t smem) {
  want = std::max(want, 1);
  if (!h.narrow) return want;
  return std::min(want, coop_cluster_limit(h, kern, block, smem));
}

void launch_coop(Handle& h, const void* kern, i32 grid, i32 block, size_t smem, void** args) {
  GKW_REQUIRE(grid >= 1, GKW_E_INTERNAL, "empty grid");
  if (grid > 1 && grid <= coop_cluster_limit(h, kern, block, smem)) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = h.stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = grid;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    GKW_CUDA(cudaLaunchKernelExC(&cfg, kern, args));
    count_launch();
    return;
  }
  if (grid == 1) {   // one CTA waits on no other
    GKW_CUDA(cudaLaunchKernel(kern, dim3(1), dim3(block), args, smem, h.stream));
    count_launch();
    return;
  }
  GKW_REQUIRE(h.device >= 0 && h.device < kMaxDevices, GKW_E_UNSUPPORTED, "device index too large");
  if (h.capturing) {   // in a graph: graph_run chains the whole graph instead
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = h.stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    GKW_CUDA(cudaLaunchKernelExC(&cfg, kern, args));
    count_launch();
    h.capture_wide = true;
    return;
  }
  if (!h.coop_ev) GKW_CUDA(cudaEventCreateWithFlags(&h.coop_ev, cudaEventDisableTiming));
  std::lock_guard<std::mutex> lk(g_chain_mu[h.device]);
  if (g_chain_last[h.device] && g_chain_last[h.device] != h.coop_ev)
    GKW_CUDA(cudaStreamWaitEvent(h.stream, g_chain_last[h.device], 0));
  GKW_CUDA(cudaLaunchCooperativeKernel(kern, dim3(grid), dim3(block), args, smem, h.stream));
  count_launch();
  GKW_CUDA(cudaEventRecord(h.coop_ev, h.stream));
  g_chain_last[h.device] = h.coop_ev;
}

void graph_cache_clear(Handle& h) {
  for (Handle::GraphEntry& e : h.graphs)
    if (e.exec) cudaGraphExecDestroy(e.exec);
  h.graphs.clear();
}

bool graph_run(Handle& h, const std::string& key, const std::function<void()>& body) {
  if (!h.graphs_on || h.capturing) {
    body();
    return false;
  }
  Handle::GraphEntry* e = nullptr;
  for (Handle::GraphEntry& x : h.graphs)
    if (x.key == key) e = &x;
  if (!e) {   // first sight: run as is (pools grow, shapes settle)
    if (h.graphs.size() >= 64) graph_cache_clear(h);
    h.graphs.push_back(Handle::GraphEntry{key, 1});
    body();
    return false;
  }
  if (!e->exec) {   // second sight: capture, then run the graph
    const u64 l0 = launch_total(), s0 = h.scans_enqueued, ep0 = h.scan_epoch;
    cudaGraph_t g = nullptr;
    h.capture_wide = false;
    cudaError_t err = cudaStreamBeginCapture(h.stream, cudaStreamCaptureModeThreadLocal);
    if (err == cudaSuccess) {
      h.capturing = true;
      try {
        body();
      } catch (...) {
        h.capturing = false;
        cudaStreamEndCapture(h.stream, &g);
        if (g) cudaGraphDestroy(g);
        cudaGetLastError();
        uncount_launches(launch_total() - l0);
        h.scans_enqueued = s0;
        h.scan_epoch = ep0;
        h.graphs_on = false;   // the body needs something a capture cannot hold: run it plainly from now on
        body();
        return false;
      }
      h.capturing = false;
      err = cudaStreamEndCapture(h.stream, &g);
    }
    const u64 nl = launch_total() - l0, ns = h.scans_enqueued - s0;
    uncount_launches(nl);   // nothing ran yet
    h.scans_enqueued = s0;
    h.scan_epoch = ep0;
    if (err == cudaSuccess) err = cudaGraphInstantiate(&e->exec, g, 0);
    if (g) cudaGraphDestroy(g);
    if (err != cudaSuccess) {
      cudaGetLastError();
      e->exec = nullptr;
      h.graphs_on = false;
      body();
      return false;
    }
    e->launches = nl;
    e->scans = ns;
    e->wide = h.capture_wide;
  }
  if (e->wide) {   // wide launches of all handles take turns (launch_coop)
    GKW_REQUIRE(h.device >= 0 && h.device < kMaxDevices, GKW_E_UNSUPPORTED, "device index too large");
    if (!h.coop_ev) GKW_CUDA(cudaEventCreateWithFlags(&h.coop_ev, cudaEventDisableTiming));
    std::lock_guard<std::mutex> lk(g_chain_mu[h.device]);
    if (g_chain_last[h.device] && g_chain_last[h.device] != h.coop_ev)
      GKW_CUDA(cudaStreamWaitEvent(h.stream, g_chain_last[h.device], 0));
    GKW_CUDA(cudaGraphLaunch(e->exec, h.stream));
    GKW_CUDA(cudaEventRecord(h.coop_ev, h.stream));
    g_chain_last[h.device] = h.coop_ev;
  } else {
    GKW_CUDA(cudaGraphLaunch(e->exec, h.stream));
  }
  count_launches(e->launches);
  h.scans_enqueued += e->scans;
  h.scan_epoch += e->scans;
  return true;
}

// Drop a handle's chain event (the handle is going away).
void forget_coop_event(Handle& h) {
  if (!h.coop_ev) return;
  if (h.device >= 0 && h.device < kMaxDevices) {
    std::lock_guard<std::mutex> lk(g_chain_mu[h.device]);
    if (g_chain_last[h.device] == h.coop_ev) g_chain_last[h.device] = nullptr;
  }
  cudaEventDestroy(h.coop_ev);
  h.coop_ev = nullptr;
}

// ---------------------------------------------------------------------------
// Host memory.  A copy from pageable memory is staged by the driver on the
// calling thread (11.5 GB/s); here several threads fill pinned slots of 2 MB
// and queue one copy each, which the link takes at 40 GB/s and more: a batch
// of 256 graphs (349 MB) 65 -> 46 ms.  Small copies, pinned, managed or device
// pointers and the per-thread default stream take the plain call.  The buffer
// also holds a graph file's text: pinning memory for each 3.5 MB file cost 2.4
// of its 3.7 ms.
// ---------------------------------------------------------------------------
constexpr size_t kStageMin = size_t(8) << 20;   // below this the threads cost more than they save

// All handles of the process together keep at most kStageProcess bytes of
// buffers and run at most kStageHelpers threads beside their callers (a server
// has up to 256 slots).  A call that gets neither is an ordinary copy, or pins
// memory of its own for a file.
constexpr size_t kStageProcess = 4 * kStageBytes;
constexpr int kStageHelpers = 28;
static std::mutex g_stage_mu;
static size_t g_stage_bytes = 0;
static int g_stage_helpers = 0;

bool stage_reserve(size_t bytes) {
  std::lock_guard<std::mutex> lk(g_stage_mu);
  if (bytes > kStageProcess - g_stage_bytes) return false;
  g_stage_bytes += bytes;
  return true;
}

void stage_unreserve(size_t bytes) {
  std::lock_guard<std::mutex> lk(g_stage_mu);
  g_stage_bytes -= bytes;
}

int stage_take_helpers(int want) {
  const int all = std::min<int>(kStageHelpers, (int)(std::thread::hardware_concurrency() / 2));
  std::lock_guard<std::mutex> lk(g_stage_mu);
  const int n = std::max(0, std::min(want, all - g_stage_helpers));
  g_stage_helpers += n;
  return n;
}

void stage_return_helpers(int n) {
  std::lock_guard<std::mutex> lk(g_stage_mu);
  g_stage_helpers -= n;
}

// The helpers of one copy: up to seven, given back when it ends.
struct StageHelpers {
  int n;
  StageHelpers() : n(0) {}
  ~StageHelpers() {
    if (n) stage_return_helpers(n);
  }
  static int most() { return std::min(8, (int)(std::thread::hardware_concurrency() / 2)) - 1; }
  bool take() {
    n = stage_take_helpers(most());
    return n > 0;
  }
};

static bool pageable(const void* p) {
  cudaPointerAttributes at;
  if (cudaPointerGetAttributes(&at, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return at.type == cudaMemoryTypeUnregistered;
}

void free_stage(Handle& h) {
  for (cudaEvent_t& e : h.stage_ev) {
    if (e) cudaEventDestroy(e);
    e = nullptr;
  }
  if (h.stage) cudaFreeHost(h.stage);
  if (h.stage_cap) stage_unreserve(h.stage_cap);
  h.stage = nullptr;
  h.stage_cap = 0;
}

char* stage_buffer(Handle& h, size_t bytes) {
  if (bytes > kStageBytes) return nullptr;
  const bool grow = h.stage_cap < bytes;
  // small files keep a small buffer; a staged copy needs all the slots
  size_t cap = size_t(1) << 20;
  while (cap < bytes) cap <<= 1;
  if (grow && !stage_reserve(cap)) return nullptr;
  const cudaError_t e = cudaStreamSynchronize(h.stream);   // copies out of the old contents
  if (e != cudaSuccess) {
    if (grow) stage_unreserve(cap);
    GKW_CUDA(e);
  }
  if (grow) {
    free_stage(h);
    if (cudaHostAlloc((void**)&h.stage, cap, cudaHostAllocDefault) != cudaSuccess) {
      cudaGetLastError();
      h.stage = nullptr;
      stage_unreserve(cap);
      return nullptr;
    }
    h.stage_cap = cap;
  }
  h.stage_raw = true;
  return h.stage;
}

// The slots and their events; false if they cannot be had.
static bool stage_slots(Handle& h) {
  if (h.stage_cap < kStageBytes || h.stage_raw) {
    if (!stage_buffer(h, kStageBytes)) return false;   // (waits for the stream)
    h.stage_raw = false;
  }
  for (cudaEvent_t& e : h.stage_ev)
    if (!e && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) {
      cudaGetLastError();
      return false;
    }
  return true;
}

// Whether this call's copies can be queued by several threads: the per-thread
// default stream names another stream on each of them, and copies queued there
// would not be ordered with the caller's kernels.
static bool staged(const Handle& h, size_t bytes) {
  return bytes >= kStageMin && StageHelpers::most() > 0 && h.stream != cudaStreamPerThread;
}

// Runs work(t) on T threads (this one included) with the handle's device
// current; returns the first CUDA error.
template <class Work>
static cudaError_t on_threads(Handle& h, int T, Work work) {
  std::vector<cudaError_t> err((size_t)T, cudaSuccess);
  auto body = [&](int t) {
    err[t] = cudaSetDevice(h.device);
    if (err[t] == cudaSuccess) err[t] = work(t);
  };
  std::vector<std::thread> pool;
  int first = 1;   // workers that could not be started are run here
  try {
    for (; first < T; ++first) pool.emplace_back(body, first);
  } catch (const std::exception&) {
  }
  body(0);
  for (int t = first; t < T; ++t) body(t);
  for (std::thread& th : pool) th.join();
  for (cudaError_t e : err)
    if (e != cudaSuccess) return e;
  return cudaSuccess;
}

void copy_to_device(Handle& h, void* dst, const void* src, size_t bytes) {
  StageHelpers helpers;
  if (!staged(h, bytes) || !pageable(src) || !stage_slots(h) || !helpers.take()) {
    if (bytes) GKW_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, h.stream));
    return;
  }
  const int T = 1 + helpers.n;
  const size_t nchunk = (bytes + kStageChunk - 1) / kStageChunk;
  const int per = Handle::kStageSlots / T;   // slots of a thread
  const cudaError_t e = on_threads(h, T, [&](int t) {
    int use = 0;
    for (size_t c = (size_t)t; c < nchunk; c += (size_t)T, use = (use + 1) % per) {
      const int slot = t * per + use;
      cudaError_t er = cudaEventSynchronize(h.stage_ev[slot]);
      if (er != cudaSuccess) return er;
      char* p = h.stage + (size_t)slot * kStageChunk;
      const size_t off = c * kStageChunk, len = std::min(kStageChunk, bytes - off);
      memcpy(p, (const char*)src + off, len);
      er = cudaMemcpyAsync((char*)dst + off, p, len, cudaMemcpyHostToDevice, h.stream);
      if (er == cudaSuccess) er = cudaEventRecord(h.stage_ev[slot], h.stream);
      if (er != cudaSuccess) return er;
    }
    return cudaSuccess;
  });
  if (e != cudaSuccess) {
    cudaStreamSynchronize(h.stream);   // no queued copy may outlive the slots
    GKW_CUDA(e);
  }
}

void copy_to_host(Handle& h, void* dst, const void* src, size_t bytes) {
  StageHelpers helpers;
  if (!staged(h, bytes) || !pageable(dst) || !stage_slots(h) || !helpers.take()) {
    if (bytes) GKW_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, h.stream));
    GKW_CUDA(cudaStreamSynchronize(h.stream));
    return;
  }
  const int T = 1 + helpers.n;
  const size_t nchunk = (bytes + kStageChunk - 1) / kStageChunk;
  const int per = Handle::kStageSlots / T;
  const cudaError_t e = on_threads(h, T, [&](int t) {
    auto slot = [&](size_t i) { return t * per + (int)(i % (size_t)per); };
    auto range = [&](size_t i, size_t* off, size_t* len) {   // this thread's i-th chunk
      *off = ((size_t)t + i * (size_t)T) * kStageChunk;
      *len = *off < bytes ? std::min(kStageChunk, bytes - *off) : 0;
    };
    const size_t mine = (size_t)t < nchunk ? (nchunk - (size_t)t - 1) / (size_t)T + 1 : 0;
    for (size_t i = 0; i < mine + (size_t)per - 1; ++i) {
      size_t off, len;
      if (i < mine) {   // queue chunk i ...
        range(i, &off, &len);
        cudaError_t er = cudaMemcpyAsync(h.stage + (size_t)slot(i) * kStageChunk, (const char*)src + off, len,
                                         cudaMemcpyDeviceToHost, h.stream);
        if (er == cudaSuccess) er = cudaEventRecord(h.stage_ev[slot(i)], h.stream);
        if (er != cudaSuccess) return er;
      }
      if (i + 1 >= (size_t)per && i + 1 - (size_t)per < mine) {   // ... and empty the slot that is used next
        const size_t j = i + 1 - (size_t)per;
        const cudaError_t er = cudaEventSynchronize(h.stage_ev[slot(j)]);
        if (er != cudaSuccess) return er;
        range(j, &off, &len);
        memcpy((char*)dst + off, h.stage + (size_t)slot(j) * kStageChunk, len);
      }
    }
    return cudaSuccess;
  });
  const cudaError_t e2 = cudaStreamSynchronize(h.stream);
  GKW_CUDA(e);
  GKW_CUDA(e2);
}

float balance_cap(i64 total_vwgt, i32 k, double eps) {
  return (float)((1.0 + eps) * (double)total_vwgt / (double)k);
}

float max_part_weight(i64 total_vwgt, i32 k, double eps) {
  // graph_partitioner.hpp:230: (float)W/(float)k * (1.0f + IMBALANCE_RATIO) + 1,
  // IMBALANCE_RATIO a double literal, result stored as float.
  float q = (float)(u32)total_vwgt / (float)k;
  return (float)((double)q * (1.0 + eps) + 1);
}

}  // namespace gkw
