// kernels_select.cu -- greedy max-coverage building blocks for sm_100a.
//
// count_kernel      vertex-occurrence histogram over sets [0, S)
//                   (CountOccurrencies, include/ripples/counting.h:65-97;
//                   reference GPU kernel_count, src/gpu/find_most_influential.cc:56-63)
//                   with warp-aggregated atomics: __match_any_sync groups
//                   lanes holding the same vertex and one leader adds the
//                   group size.
// inverted_kernel   vertex -> sets index (a CSR transpose of the pool), built
//                   once per selection so each pick touches only the sets that
//                   contain the seed, instead of re-scanning the pool
//                   (update_mask_kernel + count_uncovered_kernel,
//                   src/gpu/find_most_influential.cc:74-98).
// cover_kernel      after a reference-heap pick: marks the seed's
//                   still-uncovered sets covered and decrements the counts of
//                   their members (UpdateCounters,
//                   include/ripples/counting.h:141-151).
// gather_counts     the counts of the heap items a reference-heap pick can
//                   examine, into mapped host memory.
// heap kernels      the selection max-heap built on the device, level by
//                   level, element for element the one std::make_heap builds.
// sel_* kernels     lowest-id picks entirely on the device (max count, lowest
//                   vertex id on ties, as thrust::max_element in
//                   src/gpu/find_most_influential.cc:65-72): cached chunk
//                   maxima, cover by decrement or recount.
//
// The per-set loops share one load balancing (block_elements): a warp takes up
// to 32 sets, scans their lengths and walks the concatenated elements, each
// lane finding its set with a 5-step shuffle search; long sets are spread over
// the whole block.
#include <algorithm>

#include <cooperative_groups.h>

#include "device.cuh"
#include "launch.h"

namespace rip {

namespace {

constexpr uint32_t NONE = 0xFFFFFFFFu;

// Sets of at least this many elements are walked by their whole block, 1024
// elements at a step; the others by the warp that met them.
constexpr uint32_t kLongSet = 512;
constexpr uint32_t kBlock = 256;  // threads of the per-set kernels

template <uint32_t THREADS>
struct LongSetsOf {  // shared: the long sets a block met in one step
  uint64_t set[THREADS], off[THREADS];
  uint32_t len[THREADS];
  uint32_t n;
};
using LongSets = LongSetsOf<kBlock>;

// Calls the grid over the elements of sets set_of(i), i in [lo, hi) (~0: none).
// A warp takes up to 32 sets a step -- fewer when that leaves warps idle: a
// pool of giant sets has fewer sets than the grid has warps -- scans their
// lengths and walks the concatenated elements, each lane finding its set with
// a shuffle search: mixed(set, vertex, valid) is called by all lanes of the
// warp, so it may use warp collectives.  Elements of a set of kLongSet or more
// are spread over the block: single(set, vertex), no collectives.  One warp
// walking a set of 40 000 elements alone took 0.5 ms; a block takes 15 us.
template <uint32_t THREADS, typename SetOf, typename Mixed, typename Single>
__device__ __forceinline__ void block_elements(const DevPool &P, uint64_t lo, uint64_t hi,
                                               LongSetsOf<THREADS> &sh, SetOf set_of,
                                               Mixed mixed, Single single) {
  constexpr uint32_t WARPS = THREADS / 32;
  const uint32_t lane = lane_id(), wid = threadIdx.x >> 5;
  if (hi <= lo) return;
  const uint64_t warps = (uint64_t)gridDim.x * WARPS;
  const uint64_t per = (hi - lo + warps - 1) / warps;
  const uint32_t take = per < 32 ? (uint32_t)per : 32u;  // sets a warp takes a step
  if (threadIdx.x == 0) sh.n = 0;
  __syncthreads();
  for (uint64_t base = lo + (uint64_t)blockIdx.x * WARPS * take; base < hi;
       base += warps * take) {
    const uint64_t i = base + wid * take + lane;
    uint64_t s = 0, off = 0;
    uint32_t len = 0;
    if (lane < take && i < hi) {
      s = set_of(i);
      if (s != ~0ull) {
        len = P.set_len[s];
        off = P.set_off[s];
      }
    }
    if (len >= kLongSet) {
      const uint32_t k = atomicAdd(&sh.n, 1u);
      sh.set[k] = s;
      sh.off[k] = off;
      sh.len[k] = len;
    }
    const bool any = __syncthreads_or(len >= kLongSet);
    if (len >= kLongSet) len = 0;
    const uint32_t incl = warp_incl_scan(len);
    const uint32_t total = __shfl_sync(FULL, incl, 31);
    for (uint32_t j0 = 0; j0 < total; j0 += 64) {
      uint64_t os[2];
      uint32_t v[2];
      bool valid[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const uint32_t j = j0 + 32 * h + lane;
        valid[h] = j < total;
        const uint32_t owner = warp_find_owner(incl, valid[h] ? j : total - 1);
        const uint64_t ooff = __shfl_sync(FULL, off, owner);
        const uint32_t oexcl = __shfl_sync(FULL, incl - len, owner);
        os[h] = __shfl_sync(FULL, s, owner);
        v[h] = valid[h] ? P.vtx[ooff + (j - oexcl)] : NONE;
      }
#pragma unroll
      for (int h = 0; h < 2; ++h)
        if (j0 + 32 * h < total) mixed(os[h], v[h], valid[h]);
    }
    if (any) {
      const uint32_t n = sh.n;
      for (uint32_t k = 0; k < n; ++k) {
        const uint64_t ks = sh.set[k];
        const uint32_t *vtx = P.vtx + sh.off[k];
        const uint32_t klen = sh.len[k];
        for (uint32_t j = threadIdx.x; j < klen; j += 4 * THREADS) {
          uint32_t v[4];
#pragma unroll
          for (int h = 0; h < 4; ++h)
            if (j + h * THREADS < klen) v[h] = vtx[j + h * THREADS];
#pragma unroll
          for (int h = 0; h < 4; ++h)
            if (j + h * THREADS < klen) single(ks, v[h]);
        }
      }
      __syncthreads();
      if (threadIdx.x == 0) sh.n = 0;
      __syncthreads();
    }
  }
}

// The set ids themselves, for walks over sets [0, S).
struct EverySet {
  __device__ __forceinline__ uint64_t operator()(uint64_t i) const { return i; }
};

// Iterates the elements of 32 sets per warp; `fn(set, vertex, valid)` is
// called by ALL lanes (valid says whether the lane holds an element) so it may
// use warp collectives.
template <typename SetOf, typename Fn>
__device__ __forceinline__ void for_each_element(const DevPool &P,
                                                 uint64_t window_base,
                                                 uint64_t limit, SetOf set_of,
                                                 Fn fn) {
  const uint32_t lane = lane_id();
  const uint64_t sidx = window_base + lane;
  uint64_t s = 0;
  uint32_t len = 0;
  uint64_t off = 0;
  if (sidx < limit) {
    s = set_of(sidx);
    if (s != ~0ull) {
      len = P.set_len[s];
      off = P.set_off[s];
    }
  }
  const uint32_t incl = warp_incl_scan(len);
  const uint32_t total = __shfl_sync(FULL, incl, 31);
  for (uint32_t base = 0; base < total; base += 32) {
    const uint32_t j = base + lane;
    const bool valid = j < total;
    const uint32_t owner = warp_find_owner(incl, valid ? j : total - 1);
    const uint64_t ooff = __shfl_sync(FULL, off, owner);
    const uint32_t oexcl =
        __shfl_sync(FULL, incl, owner) - __shfl_sync(FULL, len, owner);
    const uint64_t os = __shfl_sync(FULL, s, owner);
    const uint32_t v = valid ? P.vtx[ooff + (j - oexcl)] : NONE;
    fn(os, v, valid);
  }
}

// One occurrence per valid lane, called by all lanes of the warp.  When the
// warp's 32 elements come from one set they are distinct vertices (a set
// holds each vertex once) and every lane adds 1; otherwise lanes holding the
// same vertex are grouped with __match_any_sync and one leader adds the group
// size.  Lanes past the last element carry the last set's id.
__device__ __forceinline__ void add_occurrence(uint32_t *count, uint64_t s, uint32_t v,
                                               bool valid) {
  if (__shfl_sync(FULL, s, 0) == __shfl_sync(FULL, s, 31)) {
    if (valid) atomicAdd(count + v, 1u);
    return;
  }
  const uint32_t peers = __match_any_sync(FULL, v);
  if (valid && (__ffs(peers) - 1) == (int)lane_id())
    atomicAdd(count + v, (uint32_t)__popc(peers));
}

__global__ void __launch_bounds__(kBlock)
count_kernel(DevPool P, uint64_t S, uint32_t *count) {
  __shared__ LongSets sh;
  block_elements(
      P, 0, S, sh, EverySet(),
      [&](uint64_t s, uint32_t v, bool valid) { add_occurrence(count, s, v, valid); },
      [&](uint64_t, uint32_t v) { atomicAdd(count + v, 1u); });
}

// Sets of [0, S) holding at least one marked vertex (OPIM-C's FindCoverage,
// include/ripples/opimc.h:101-118): bit (s - window) of `hit` is set when a
// member of set s is marked; each warp adds the covered sets of its window.
__global__ void __launch_bounds__(256)
coverage_kernel(DevPool P, uint64_t S, const uint32_t *marked, unsigned long long *covered) {
  const uint64_t gw = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  unsigned long long mine = 0;
  for (uint64_t wb = gw * 32; wb < S; wb += nw * 32) {
    uint32_t hit = 0;
    for_each_element(
        P, wb, S, [](uint64_t i) { return i; },
        [&](uint64_t s, uint32_t v, bool valid) {
          const bool m = valid && ((__ldg(marked + (v >> 5)) >> (v & 31)) & 1u);
          hit |= __reduce_or_sync(FULL, m ? 1u << (uint32_t)(s - wb) : 0u);
        });
    mine += __popc(hit);
  }
  if (lane_id() == 0 && mine) atomicAdd(covered, mine);
}

__global__ void __launch_bounds__(kBlock)
inverted_kernel(DevPool P, uint64_t S, uint64_t *cursor, uint32_t *inv, uint64_t base) {
  __shared__ LongSets sh;
  unsigned long long *cur = reinterpret_cast<unsigned long long *>(cursor);
  block_elements(
      P, 0, S, sh, EverySet(),
      [&](uint64_t s, uint32_t v, bool valid) {
        if (__shfl_sync(FULL, s, 0) == __shfl_sync(FULL, s, 31)) {  // distinct vertices
          if (valid) inv[atomicAdd(cur + v, 1ull)] = (uint32_t)(base + s);
          return;
        }
        const uint32_t peers = __match_any_sync(FULL, v);
        const uint32_t leader = __ffs(peers) - 1;
        unsigned long long b = 0;
        if (valid && leader == lane_id())
          b = atomicAdd(cur + v, (unsigned long long)__popc(peers));
        b = __shfl_sync(FULL, b, leader);
        if (valid) inv[b + __popc(peers & lanes_below())] = (uint32_t)(base + s);
      },
      [&](uint64_t s, uint32_t v) { inv[atomicAdd(cur + v, 1ull)] = (uint32_t)(base + s); });
}

// A reference-heap pick: covers the vertex's uncovered sets and decrements
// their members with plain reductions (no result needed).  The vertex itself
// is a member of every one of them and ends at 0: it is written once instead
// of being decremented by every set at one address.
__device__ __forceinline__ void cover_sets(const CoverLaunch &C, LongSets &sh) {
  const uint64_t lo = C.inv_off[C.vertex], hi = C.inv_off[C.vertex + 1];
  block_elements(
      C.P, lo, hi, sh,
      [&](uint64_t i) -> uint64_t {
        const uint32_t s = C.inv[i];
        if (C.covered[s]) return ~0ull;  // covered by an earlier seed
        C.covered[s] = 1;                // s holds the vertex once: no other lane has s
        return s;
      },
      [&](uint64_t, uint32_t v, bool valid) {
        if (valid && v != C.vertex) atomicSub(C.count + v, 1u);
      },
      [&](uint64_t, uint32_t v) {
        if (v != C.vertex) atomicSub(C.count + v, 1u);
      });
  if (blockIdx.x == 0 && threadIdx.x == 0) C.count[C.vertex] = 0u;
}

__global__ void __launch_bounds__(kBlock) cover_kernel(CoverLaunch C) {
  __shared__ LongSets sh;
  cover_sets(C, sh);
}

// The pick of a sharded selection over the summed counts: the largest
// count << 32 | ~v, i.e. the largest count and the lowest vertex id among
// equal counts (thrust::max_element over the reduced counters,
// include/ripples/mpi/find_most_influential.h:505-511).
__device__ __forceinline__ unsigned long long pick_key(uint32_t c, uint32_t v) {
  return (unsigned long long)c << 32 | (uint32_t)~v;
}

// A sharded pick's cover with its decrements listed instead of applied:
// marks this shard's uncovered sets holding the vertex covered and appends
// their members to `out` (each entry: that vertex's summed count drops by
// one), a warp per set.  At most the shard's element count
// is written.
__global__ void __launch_bounds__(256) cover_list_kernel(CoverLaunch C, uint32_t *out,
                                                         unsigned long long *cursor) {
  const uint64_t gw = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  const uint32_t lane = lane_id();
  const uint64_t lo = C.inv_off[C.vertex], hi = C.inv_off[C.vertex + 1];
  for (uint64_t i = lo + gw; i < hi; i += nw) {
    const uint32_t s = C.inv[i];
    if (C.covered[s]) continue;  // warp-uniform
    const uint32_t len = C.P.set_len[s];
    const uint64_t off = C.P.set_off[s];
    unsigned long long b = 0;
    if (lane == 0) {
      C.covered[s] = 1;
      b = atomicAdd(cursor, (unsigned long long)len);
    }
    b = __shfl_sync(FULL, b, 0);
    for (uint32_t j = lane; j < len; j += 32) out[b + j] = C.P.vtx[off + j];
  }
}

// Summed counts minus the listed decrements; marks the chunks they touch for
// the next pick (entries >= n are skipped).
__global__ void __launch_bounds__(256) apply_decrements_kernel(uint32_t *count, uint32_t n,
                                                               const uint32_t *dec, uint64_t m,
                                                               uint8_t *dirty) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < m; i += stride) {
    const uint32_t v = dec[i];
    if (v < n) {
      atomicSub(count + v, 1u);
      dirty[v / kPickChunk] = 1;
    }
  }
}

// The pick key maximum of every dirty chunk of kPickChunk counts, one block
// per chunk (clean chunks return at once); clears the chunk's flag.
__global__ void __launch_bounds__(256) chunk_max_kernel(const uint32_t *__restrict__ count,
                                                        uint32_t n, uint8_t *dirty,
                                                        unsigned long long *cmax) {
  const uint32_t chunk = blockIdx.x;
  if (!dirty[chunk]) return;
  const uint32_t lo = chunk * kPickChunk;
  const uint32_t hi = min(n, lo + kPickChunk);
  unsigned long long key = 0;
  if (hi - lo == kPickChunk) {  // whole chunk: 16-byte loads (count 16-byte aligned)
    const uint4 *c4 = reinterpret_cast<const uint4 *>(count + lo);
    for (uint32_t i = threadIdx.x; i < kPickChunk / 4; i += blockDim.x) {
      const uint4 q = c4[i];
      const uint32_t v = lo + i * 4;
      key = max(key, pick_key(q.x, v));
      key = max(key, pick_key(q.y, v + 1));
      key = max(key, pick_key(q.z, v + 2));
      key = max(key, pick_key(q.w, v + 3));
    }
  } else {
    for (uint32_t v = lo + threadIdx.x; v < hi; v += blockDim.x) key = max(key, pick_key(count[v], v));
  }
  for (int o = 16; o; o >>= 1) key = max(key, __shfl_xor_sync(FULL, key, o));
  __shared__ unsigned long long s_key[8];
  const uint32_t warp = threadIdx.x >> 5;
  if (lane_id() == 0) s_key[warp] = key;
  __syncthreads();
  if (warp == 0) {
    key = lane_id() < (blockDim.x >> 5) ? s_key[lane_id()] : 0ull;
    for (int o = 4; o; o >>= 1) key = max(key, __shfl_xor_sync(FULL, key, o));
    if (lane_id() == 0) {
      cmax[chunk] = key;
      dirty[chunk] = 0;
    }
  }
}

// *best = the maximum of cmax[0, nchunks) (one block).
__global__ void __launch_bounds__(1024) cmax_max_kernel(const unsigned long long *cmax,
                                                        uint32_t nchunks,
                                                        unsigned long long *best) {
  unsigned long long key = 0;
  for (uint32_t i = threadIdx.x; i < nchunks; i += blockDim.x) key = max(key, cmax[i]);
  for (int o = 16; o; o >>= 1) key = max(key, __shfl_xor_sync(FULL, key, o));
  __shared__ unsigned long long s_key[32];
  const uint32_t warp = threadIdx.x >> 5;
  if (lane_id() == 0) s_key[warp] = key;
  __syncthreads();
  if (warp == 0) {
    key = lane_id() < (blockDim.x >> 5) ? s_key[lane_id()] : 0ull;
    for (int o = 16; o; o >>= 1) key = max(key, __shfl_xor_sync(FULL, key, o));
    if (lane_id() == 0) *best = key;
  }
}

// A reference-heap pick in one launch: cover_kernel's work, then the last
// block to finish (a completion ticket in *done) gathers the current counts of
// the host's candidates for the next pick into `out` (mapped host memory),
// resets the ticket and publishes `epoch` in *flag after a system-wide fence,
// so the host polls one word instead of synchronising the stream.
__global__ void __launch_bounds__(kBlock) cover_gather_kernel(CoverLaunch C, const uint32_t *ids,
                                                           uint32_t nids, uint32_t *out,
                                                           unsigned int *done,
                                                           volatile unsigned int *flag,
                                                           unsigned int epoch) {
  __shared__ LongSets sh;
  cover_sets(C, sh);
  __shared__ bool s_last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();  // this block's decrements before its ticket
    s_last = atomicAdd(done, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();  // every other block's decrements are visible from here
  // ids and out sit in mapped host memory (16-byte aligned): four ids a
  // read, so that a 2048-id gather is two rounds over the bus per thread
  const uint32_t n4 = nids >> 2;
  const uint4 *ids4 = reinterpret_cast<const uint4 *>(ids);
  uint4 *out4 = reinterpret_cast<uint4 *>(out);
  for (uint32_t i = threadIdx.x; i < n4; i += blockDim.x) {
    const uint4 v = ids4[i];
    out4[i] = make_uint4(__ldcg(C.count + v.x), __ldcg(C.count + v.y), __ldcg(C.count + v.z),
                         __ldcg(C.count + v.w));
  }
  for (uint32_t i = (n4 << 2) + threadIdx.x; i < nids; i += blockDim.x)
    out[i] = __ldcg(C.count + ids[i]);
  __syncthreads();
  if (threadIdx.x == 0) {
    *done = 0u;
    __threadfence_system();
    *flag = epoch;
  }
}

// ---- device-only picks (served queries) -----------------------------------
// Every kernel reads its buffers from a SelDesc in device memory, so one
// captured CUDA graph serves every round of a query: the host rewrites the
// descriptor (S, buffers) and replays the graph.  Picks keep the lowest-id
// tie-break: key(v) = count[v] << 32 | ~v, the maximum key wins.  The count
// array is split into chunks of SEL_CHUNK vertices with a cached maximum key
// each; a cover marks the chunks it decrements dirty and the next pick
// re-reads only those, then reduces the chunk maxima in the last block.
constexpr uint32_t SEL_CHUNK = 1024;
constexpr uint32_t kLoopCtas = 8, kLoopThreads = 512;
constexpr uint32_t kLoopChunks = 64;  // chunk maxima a block keeps
// A round is one cluster's if its chunks (kLoopCtas * kLoopChunks: 2^19 vertices)
// and elements are few enough; far above either, the chunks that covers touch
// (every one is read again, 4 KB) or the first covers alone keep eight SMs busy
// longer than the grid takes for all picks.  One cluster and grid-wide, lowest-id
// IMMs of 150 seeds on R-MAT graphs of degree 8, weighted cascade (LT): 2^19
// vertices 12.8 and 14.4 (7.2 and 8.3) ms, 2^20 20.5 and 16.2 (9.6 and 9.0), 2^21
// 28.7 and 22.6 (18.0 and 12.7), 2^22 48.7 and 27.9 (23.4 and 11.1).  Elements: the
// two rounds just below 8 M of a weighted-cascade query on Erdos-Renyi vertices 3.5
// and 3.7 ms.
constexpr double kLoopElements = 8.0 * (1 << 20);

__device__ __forceinline__ unsigned long long sel_key(uint32_t c, uint32_t v) {
  return ((unsigned long long)c << 32) | (unsigned long long)(~v);
}
__device__ __forceinline__ unsigned long long umax64(unsigned long long a,
                                                     unsigned long long b) {
  return a > b ? a : b;
}

__global__ void __launch_bounds__(256) sel_init_kernel(const SelDesc *__restrict__ dp) {
  const SelDesc d = *dp;
  const uint64_t tid = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  if (!d.keep_counts) {
    const uint64_t n4 = (uint64_t)d.nchunks * (SEL_CHUNK / 4);
    uint4 *c4 = reinterpret_cast<uint4 *>(d.count);
    for (uint64_t i = tid; i < n4; i += stride) c4[i] = make_uint4(0, 0, 0, 0);
    const uint64_t s16 = (d.S + 15) / 16;
    uint4 *cv = reinterpret_cast<uint4 *>(d.covered);
    for (uint64_t i = tid; i < s16; i += stride) cv[i] = make_uint4(0, 0, 0, 0);
  }
  for (uint64_t i = tid; i < d.nchunks; i += stride) d.dirty[i] = 1;
  for (uint64_t i = tid; i < d.k; i += stride) d.best[i] = 0ull;
  if (tid == 0) {
    *d.done_blocks = 0;
    d.acc[2] = d.keep_counts ? d.total_elems : 0ull;
    d.acc[3] = d.S;  // sets still uncovered
    d.acc[4] = 0ull;
  }
}

__global__ void __launch_bounds__(kBlock) sel_count_kernel(const SelDesc *__restrict__ dp) {
  __shared__ LongSets sh;
  const SelDesc d = *dp;
  unsigned long long elems = 0;
  block_elements(
      d.P, 0, d.S, sh, EverySet(),
      [&](uint64_t s, uint32_t v, bool valid) {
        add_occurrence(d.count, s, v, valid);
        elems += valid ? 1 : 0;
      },
      [&](uint64_t, uint32_t v) {
        atomicAdd(d.count + v, 1u);
        ++elems;
      });
  elems = warp_sum_u64(elems);
  if (lane_id() == 0 && elems) atomicAdd(d.acc + 2, elems);
}

// Whether a pick's cover recounts: its g sets hold about g x the mean
// uncovered set size; when that outweighs the rest, recounting the rest is
// less work than decrementing (either way the counts are exact).
__device__ __forceinline__ bool sel_recounts(unsigned long long g, unsigned long long left,
                                             unsigned long long sets, uint32_t n) {
  const unsigned long long est =
      sets ? (unsigned long long)((double)g * (double)left / (double)sets) : 0ull;
  return est > (left > est ? left - est : 0ull) + n / 4;
}

// The largest key of chunk c's counts (a warp).
__device__ __forceinline__ unsigned long long sel_chunk_max(const SelDesc &d, uint64_t c) {
  const uint32_t lane = lane_id();
  const uint4 *src = reinterpret_cast<const uint4 *>(d.count + c * SEL_CHUNK);
  unsigned long long key = 0;
#pragma unroll
  for (uint32_t j = 0; j < SEL_CHUNK / 128; ++j) {
    const uint32_t q = j * 32 + lane;
    const uint4 x = __ldcg(src + q);
    const uint32_t v = (uint32_t)(c * SEL_CHUNK) + 4 * q;
    key = umax64(key, umax64(umax64(sel_key(x.x, v), sel_key(x.y, v + 1)),
                             umax64(sel_key(x.z, v + 2), sel_key(x.w, v + 3))));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) key = umax64(key, __shfl_xor_sync(FULL, key, o));
  return key;
}

// Pick i: refresh the dirty chunk maxima (one warp per chunk), then the last
// block to finish reduces all chunk maxima into best[i].
__global__ void __launch_bounds__(256) sel_pick_kernel(const SelDesc *__restrict__ dp,
                                                       uint32_t i) {
  __shared__ unsigned long long s_red[8];
  __shared__ bool s_last;
  const SelDesc d = *dp;
  if (i > 0 && (d.best[i - 1] >> 32) == 0) return;  // everything covered
  const uint32_t lane = lane_id(), wid = threadIdx.x >> 5;
  const uint64_t gw = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  for (uint64_t c = gw; c < d.nchunks; c += nw) {
    if (!d.dirty[c]) continue;  // warp-uniform
    const unsigned long long key = sel_chunk_max(d, c);
    if (lane == 0) {
      d.cmax[c] = key;
      d.dirty[c] = 0;
    }
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(d.done_blocks, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  unsigned long long key = 0;
  for (uint64_t c = threadIdx.x; c < d.nchunks; c += blockDim.x)
    key = umax64(key, __ldcg(d.cmax + c));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) key = umax64(key, __shfl_xor_sync(FULL, key, o));
  if (lane == 0) s_red[wid] = key;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long b = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) b = umax64(b, s_red[w]);
    d.best[i] = b;
    *d.done_blocks = 0;
    const unsigned long long g = b >> 32, left = d.acc[2], sets = d.acc[3];
    d.acc[4] = sel_recounts(g, left, sets, d.n) ? 1ull : 0ull;  // how the cover of this pick runs
    d.acc[3] = sets > g ? sets - g : 0ull;
  }
}

// After pick i: mark the seed's still-uncovered sets in [0, S) covered (every
// index segment).  Decrement mode (the pick's choice in acc[4] = 0): one warp
// per set decrements its members and marks their chunks dirty.  Recount
// mode: the sets are only marked, every count is cleared and every chunk
// marked dirty, and sel_recount_kernel counts the sets left.  Both subtract
// the covered sets' elements from acc[2] (elements of uncovered sets).
constexpr uint32_t kDirtyShared = 4096;  // chunks whose dirty flags a block gathers first

// Decrement mode: marks v's uncovered sets in [0, S) covered and takes them out
// of the counts; adds their elements to `elems` (per thread).  The chunks a
// block touches are flagged in shared memory and written out once (one byte
// store per element otherwise).
template <uint32_t THREADS>
__device__ __forceinline__ void sel_cover_sets(const SelDesc *__restrict__ dp, const SelDesc &d,
                                               uint32_t v, LongSetsOf<THREADS> &sh,
                                               uint8_t *s_dirty, unsigned long long &elems) {
  const bool local = d.nchunks <= kDirtyShared;
  if (local)
    for (uint32_t x = threadIdx.x; x < d.nchunks; x += THREADS) s_dirty[x] = 0;
  auto take = [&](uint32_t u) {
    if (u == v) return;  // in every set of the list: written once, below
    atomicSub(d.count + u, 1u);
    if (local) s_dirty[u / SEL_CHUNK] = 1;
    else d.dirty[u / SEL_CHUNK] = 1;
  };
  for (uint32_t g = 0; g < d.nseg; ++g) {
    if (dp->seg_first[g] >= d.S) continue;  // the segment's sets are all >= S
    const uint64_t lo = dp->seg_off[g][v], hi = dp->seg_off[g][v + 1];
    const uint32_t *inv = dp->seg_inv[g];
    __syncthreads();
    block_elements(
        d.P, lo, hi, sh,
        [&](uint64_t j) -> uint64_t {
          const uint32_t s = inv[j];
          if (s >= d.S || __ldcg(d.covered + s)) return ~0ull;
          d.covered[s] = 1;  // s holds v once: no other lane has s
          elems += d.P.set_len[s];
          return s;
        },
        [&](uint64_t, uint32_t u, bool valid) {
          if (valid) take(u);
        },
        [&](uint64_t, uint32_t u) { take(u); });
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {  // every set of [0, S) that held v is covered now
    d.count[v] = 0u;
    d.dirty[v / SEL_CHUNK] = 1;
  }
  __syncthreads();
  if (local)
    for (uint32_t x = threadIdx.x; x < d.nchunks; x += THREADS)
      if (s_dirty[x]) d.dirty[x] = 1;
}

// Recount mode, first half: marks v's uncovered sets, clears the counts and
// flags every chunk.
__device__ __forceinline__ void sel_mark_sets(const SelDesc *__restrict__ dp, const SelDesc &d,
                                              uint32_t v, unsigned long long &elems) {
  const uint64_t tid = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  uint4 *c4 = reinterpret_cast<uint4 *>(d.count);
  const uint64_t n4 = (uint64_t)d.nchunks * (SEL_CHUNK / 4);
  for (uint64_t x = tid; x < n4; x += stride) c4[x] = make_uint4(0, 0, 0, 0);
  for (uint64_t x = tid; x < d.nchunks; x += stride) d.dirty[x] = 1;
  for (uint32_t g = 0; g < d.nseg; ++g) {
    if (dp->seg_first[g] >= d.S) continue;
    const uint64_t lo = dp->seg_off[g][v], hi = dp->seg_off[g][v + 1];
    for (uint64_t j = lo + tid; j < hi; j += stride) {  // one thread per entry: mark only
      const uint32_t s = dp->seg_inv[g][j];
      if (s < d.S && !__ldcg(d.covered + s)) {  // s holds v once: no other thread has s
        d.covered[s] = 1;
        elems += d.P.set_len[s];
      }
    }
  }
}

__global__ void __launch_bounds__(kBlock) sel_cover_kernel(const SelDesc *__restrict__ dp,
                                                           uint32_t i) {
  __shared__ LongSets sh;
  __shared__ uint8_t s_dirty[kDirtyShared];
  const SelDesc d = *dp;
  const unsigned long long b = d.best[i];
  if ((b >> 32) == 0) return;
  const uint32_t v = ~(uint32_t)(b & 0xFFFFFFFFull);
  unsigned long long elems = 0;
  if (d.acc[4] != 0ull) sel_mark_sets(dp, d, v, elems);
  else sel_cover_sets(dp, d, v, sh, s_dirty, elems);
  elems = warp_sum_u64(elems);
  if (lane_id() == 0 && elems) atomicAdd(d.acc + 2, (unsigned long long)0 - elems);  // acc[2] -= elems
}

// Every pick of a round in one launch: one cluster of kLoopCtas blocks, which
// meet at cluster barriers instead of kernel boundaries.  Small rounds spend
// their time between launches: a pick, its cover and the (idle) recount took
// some 25 us a pick, three launches of a captured graph; here a pick is two
// cluster barriers and about ten dependent reads, 15 us (twelve queries on six
// graphs of 4 K to 65 K vertices as one batch: 139 -> 130 ms).  A cluster's
// eight SMs cannot keep up with a round of many elements, which stays with the
// grid-wide kernels (kLoopElements).  A block keeps the maxima of every
// kLoopCtas-th chunk in
// shared memory and re-reads those a cover flagged.
__global__ void __cluster_dims__(kLoopCtas, 1, 1) __launch_bounds__(kLoopThreads, 2)
sel_loop_kernel(const SelDesc *__restrict__ dp) {
  namespace cg = cooperative_groups;
  constexpr uint32_t WARPS = kLoopThreads / 32;
  __shared__ LongSetsOf<kLoopThreads> sh;
  __shared__ uint8_t s_dirty[kDirtyShared];
  __shared__ unsigned long long s_cmax[kLoopChunks];
  __shared__ unsigned long long s_red[WARPS], s_key, s_elems;
  const SelDesc d = *dp;
  cg::cluster_group cluster = cg::this_cluster();
  const uint32_t rank = blockIdx.x, lane = lane_id(), wid = threadIdx.x >> 5;
  const uint32_t own = d.nchunks > rank ? (d.nchunks - rank + kLoopCtas - 1) / kLoopCtas : 0;
  // elements of the uncovered sets, and those sets: the same in every block
  unsigned long long left = __ldcg(d.acc + 2), sets = __ldcg(d.acc + 3);
  auto block_max = [&](unsigned long long key) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) key = umax64(key, __shfl_xor_sync(FULL, key, o));
    if (lane == 0) s_red[wid] = key;
    __syncthreads();
    if (wid == 0) {
      key = lane < WARPS ? s_red[lane] : 0ull;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) key = umax64(key, __shfl_xor_sync(FULL, key, o));
      if (lane == 0) s_key = key;
    }
  };
  for (uint32_t i = 0; i < d.k; ++i) {
    for (uint32_t j = wid; j < own; j += WARPS) {
      const uint32_t c = rank + j * kLoopCtas;
      if (!__ldcg(d.dirty + c)) continue;  // warp-uniform; all are at the start
      const unsigned long long key = sel_chunk_max(d, c);
      if (lane == 0) {
        s_cmax[j] = key;
        d.dirty[c] = 0;
      }
    }
    __syncthreads();
    unsigned long long key = 0;
    for (uint32_t j = threadIdx.x; j < own; j += kLoopThreads) key = umax64(key, s_cmax[j]);
    block_max(key);
    cluster.sync();
    key = lane < kLoopCtas ? *cluster.map_shared_rank(&s_key, lane) : 0ull;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) key = umax64(key, __shfl_xor_sync(FULL, key, o));
    if (rank == 0 && threadIdx.x == 0) d.best[i] = key;
    const unsigned long long g = key >> 32;
    if (g == 0 || i + 1 == d.k) break;  // the same in every block
    const uint32_t v = ~(uint32_t)(key & 0xFFFFFFFFull);
    unsigned long long elems = 0;
    if (threadIdx.x == 0) s_elems = 0;
    if (sel_recounts(g, left, sets, d.n)) {
      sel_mark_sets(dp, d, v, elems);
      cluster.sync();  // every set marked, every count cleared
      block_elements(
          d.P, 0, d.S, sh, [&](uint64_t x) -> uint64_t { return __ldcg(d.covered + x) ? ~0ull : x; },
          [&](uint64_t s, uint32_t u, bool valid) { add_occurrence(d.count, s, u, valid); },
          [&](uint64_t, uint32_t u) { atomicAdd(d.count + u, 1u); });
    } else {
      sel_cover_sets(dp, d, v, sh, s_dirty, elems);
    }
    __syncthreads();
    elems = warp_sum_u64(elems);
    if (lane == 0 && elems) atomicAdd(&s_elems, elems);
    cluster.sync();  // the cover is done
    elems = lane < kLoopCtas ? *cluster.map_shared_rank(&s_elems, lane) : 0ull;
    left -= warp_sum_u64(elems);
    sets = sets > g ? sets - g : 0ull;
  }
  cluster.sync();  // no block leaves while another may read its shared memory
}

// Recount mode only: count the members of every set in [0, S) still
// uncovered.
__global__ void __launch_bounds__(kBlock) sel_recount_kernel(const SelDesc *__restrict__ dp) {
  __shared__ LongSets sh;
  if (dp->acc[4] == 0ull) return;
  const SelDesc d = *dp;
  block_elements(
      d.P, 0, d.S, sh, [&](uint64_t x) -> uint64_t { return d.covered[x] ? ~0ull : x; },
      [&](uint64_t s, uint32_t v, bool valid) { add_occurrence(d.count, s, v, valid); },
      [&](uint64_t, uint32_t v) { atomicAdd(d.count + v, 1u); });
}

// out[i] = count[ids[i]] (ids and out may live in mapped host memory)
__global__ void gather_counts_kernel(const uint32_t *__restrict__ count,
                                     const uint32_t *ids, uint32_t m, uint32_t *out) {
  // ids and out in mapped host memory (16-byte aligned): four ids a read
  const uint32_t m4 = m >> 2;
  const uint4 *ids4 = reinterpret_cast<const uint4 *>(ids);
  uint4 *out4 = reinterpret_cast<uint4 *>(out);
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < m4; i += stride) {
    const uint4 v = ids4[i];
    out4[i] = make_uint4(count[v.x], count[v.y], count[v.z], count[v.w]);
  }
  for (uint32_t i = (m4 << 2) + blockIdx.x * blockDim.x + threadIdx.x; i < m; i += stride)
    out[i] = count[ids[i]];
}

// ---- exclusive scan of u32 counts into u64 offsets (n+1 outputs) ----------
constexpr int SCAN_THREADS = 1024;
constexpr int SCAN_ITEMS = 4;
constexpr uint32_t SCAN_TILE = SCAN_THREADS * SCAN_ITEMS;

__device__ unsigned long long block_excl_scan(unsigned long long x,
                                              unsigned long long *warp_tot,
                                              unsigned long long *total) {
  const uint32_t lane = lane_id(), wid = threadIdx.x >> 5;
  unsigned long long incl = x;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const unsigned long long y = __shfl_up_sync(FULL, incl, d);
    if (lane >= (uint32_t)d) incl += y;
  }
  if (lane == 31) warp_tot[wid] = incl;
  __syncthreads();
  if (wid == 0) {
    unsigned long long t = lane < (blockDim.x >> 5) ? warp_tot[lane] : 0;
    unsigned long long ti = t;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const unsigned long long y = __shfl_up_sync(FULL, ti, d);
      if (lane >= (uint32_t)d) ti += y;
    }
    warp_tot[lane] = ti - t;
    if (lane == 31) *total = ti;
  }
  __syncthreads();
  const unsigned long long r = warp_tot[wid] + incl - x;
  __syncthreads();
  return r;
}

__global__ void __launch_bounds__(SCAN_THREADS)
scan_tiles_kernel(const uint32_t *in, uint32_t n, uint64_t *tile_sums) {
  __shared__ unsigned long long wt[32];
  __shared__ unsigned long long tot;
  const uint64_t base = (uint64_t)blockIdx.x * SCAN_TILE + threadIdx.x * SCAN_ITEMS;
  unsigned long long s = 0;
#pragma unroll
  for (int i = 0; i < SCAN_ITEMS; ++i)
    if (base + i < n) s += in[base + i];
  block_excl_scan(s, wt, &tot);
  if (threadIdx.x == 0) tile_sums[blockIdx.x] = tot;
}

__global__ void __launch_bounds__(SCAN_THREADS)
scan_sums_kernel(uint64_t *tile_sums, uint32_t tiles) {
  __shared__ unsigned long long wt[32];
  __shared__ unsigned long long tot;
  unsigned long long carry = 0;
  for (uint32_t b = 0; b < tiles; b += SCAN_THREADS) {
    const uint32_t i = b + threadIdx.x;
    const unsigned long long x = i < tiles ? tile_sums[i] : 0;
    const unsigned long long ex = block_excl_scan(x, wt, &tot);
    if (i < tiles) tile_sums[i] = carry + ex;
    carry += tot;
    __syncthreads();
  }
  if (threadIdx.x == 0) tile_sums[tiles] = carry;
}

__global__ void __launch_bounds__(SCAN_THREADS)
scan_apply_kernel(const uint32_t *in, uint32_t n, const uint64_t *tile_sums,
                  uint64_t *out) {
  __shared__ unsigned long long wt[32];
  __shared__ unsigned long long tot;
  const uint64_t base = (uint64_t)blockIdx.x * SCAN_TILE + threadIdx.x * SCAN_ITEMS;
  uint32_t v[SCAN_ITEMS];
  unsigned long long s = 0;
#pragma unroll
  for (int i = 0; i < SCAN_ITEMS; ++i) {
    v[i] = base + i < n ? in[base + i] : 0u;
    s += v[i];
  }
  unsigned long long ex = block_excl_scan(s, wt, &tot) + tile_sums[blockIdx.x];
#pragma unroll
  for (int i = 0; i < SCAN_ITEMS; ++i) {
    if (base + i < n) out[base + i] = ex;
    ex += v[i];
  }
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) {
    const uint32_t tiles = gridDim.x;
    out[n] = tile_sums[tiles];
  }
}

// Heap items {vertex, count}: counts below K are all equally small (K = 0:
// every count is its own key).
__device__ __forceinline__ uint32_t heap_key(uint2 it, uint32_t K) { return it.y >= K ? it.y : 0u; }

// One stage of the heap build: levels [d0, d0 + L) of the heap as std::make_heap
// builds it (the parents of one level have disjoint subtrees, so any order
// within a level gives the same heap).  A block takes 2^g neighbouring subtrees
// rooted at level d0 and keeps their L levels in shared memory, each as a heap
// of its own (item i's children at 2i + 1, 2i + 2); a sift that goes deeper goes
// on in global memory, where the stages below have been built.  Small items
// need not be ordered among themselves (sparse_heap.h says why), so with K > 0
// a sift stops where both children are small.
// Latency-bound: a launch per level took 24 launches and 0.39 ms at n = 2^24
// (15 and 0.15 ms at 2^20); two stages keep all but the last sifts on chip.
__global__ void __launch_bounds__(1024)
heap_stage_kernel(const uint32_t *__restrict__ count, uint2 *heap, uint32_t len, uint32_t d0,
                  uint32_t L, uint32_t g, uint32_t K) {
  extern __shared__ uint2 s_item[];
  const uint64_t first = (uint64_t)blockIdx.x << g;  // the block's first root, within level d0
  // item i of subtree sub: its position in the heap
  auto index = [&](uint32_t sub, uint32_t i) -> uint64_t {
    const uint32_t j = 31u - __clz(i + 1);
    return (1ull << (d0 + j)) - 1 + ((first + sub) << j) + (i + 1 - (1u << j));
  };
  for (uint32_t j = 0; j < L; ++j)
    for (uint32_t x = threadIdx.x; x < (1u << (g + j)); x += blockDim.x) {
      const uint64_t p = (1ull << (d0 + j)) - 1 + (first << j) + x;
      if (p < len)
        s_item[((x >> j) << L) + (1u << j) - 1 + (x & ((1u << j) - 1))] =
            make_uint2((uint32_t)p, __ldg(count + p));
    }
  __syncthreads();
  const uint32_t inside = (1u << L) - 1;  // items of a subtree kept here
  for (int top = (int)L - 1; top >= 0; --top) {
    for (uint32_t x = threadIdx.x; x < (1u << (g + top)); x += blockDim.x) {
      const uint32_t sub = x >> top;
      uint2 *item = s_item + (sub << L);
      const uint32_t i0 = (1u << top) - 1 + (x & ((1u << top) - 1));
      uint64_t p = index(sub, i0);
      if (2 * p + 1 >= len) continue;  // a leaf, or past the end
      // libstdc++'s __adjust_heap: the hole sinks along the larger child (the
      // right one unless the left is strictly larger), then the value rises
      // while its parent is smaller
      const uint2 value = item[i0];
      uint32_t i = i0;
      while (2 * p + 1 < len) {
        const bool here = 2 * i + 1 < inside;  // both children are, or neither
        const uint64_t lp = 2 * p + 1;
        uint2 c = here ? item[2 * i + 1] : heap[lp];
        uint32_t right = 0;
        if (lp + 1 < len) {
          const uint2 r = here ? item[2 * i + 2] : heap[lp + 1];
          if (!(heap_key(r, K) < heap_key(c, K))) {
            c = r;
            right = 1;
          }
        }
        if (c.y < K) break;  // both small
        if (i < inside) item[i] = c;
        else heap[p] = c;
        i = 2 * i + 1 + right;
        p = lp + right;
      }
      while (i > i0) {
        const uint32_t pi = (i - 1) >> 1;
        const uint64_t pp = (p - 1) >> 1;
        const uint2 par = pi < inside ? item[pi] : heap[pp];
        if (!(heap_key(par, K) < heap_key(value, K))) break;
        if (i < inside) item[i] = par;
        else heap[p] = par;
        i = pi;
        p = pp;
      }
      if (i < inside) item[i] = value;
      else heap[p] = value;
    }
    __syncthreads();
  }
  for (uint32_t j = 0; j < L; ++j)
    for (uint32_t x = threadIdx.x; x < (1u << (g + j)); x += blockDim.x) {
      const uint64_t p = (1ull << (d0 + j)) - 1 + (first << j) + x;
      if (p < len) heap[p] = s_item[((x >> j) << L) + (1u << j) - 1 + (x & ((1u << j) - 1))];
    }
}

// hist[count_bucket(c)] += 1 over the counts.
__global__ void __launch_bounds__(256)
count_hist_kernel(const uint32_t *__restrict__ count, uint32_t n, uint32_t *hist) {
  __shared__ uint32_t s_hist[kCountBuckets];
  for (uint32_t i = threadIdx.x; i < kCountBuckets; i += blockDim.x) s_hist[i] = 0;
  __syncthreads();
  // most counts are small and equal: a warp adds each distinct bucket once
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t base = (uint64_t)blockIdx.x * blockDim.x; base < n; base += stride) {
    const uint64_t v = base + threadIdx.x;
    const uint32_t b = v < n ? count_bucket(count[v]) : kCountBuckets;
    const uint32_t peers = __match_any_sync(FULL, b);
    if (v < n && __ffs(peers) - 1 == (int)lane_id()) atomicAdd(&s_hist[b], __popc(peers));
  }
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < kCountBuckets; i += blockDim.x)
    if (s_hist[i]) atomicAdd(hist + i, s_hist[i]);
}

// count[v] = the count of every heap item.
__global__ void __launch_bounds__(256)
heap_counts_kernel(const uint2 *__restrict__ heap, uint32_t n, uint32_t *count) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t p = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; p < n; p += stride) {
    const uint2 it = heap[p];
    count[it.x] = it.y;
  }
}

// The heap's items of K or more, in any order: vertices, counts and positions,
// R of each.
__global__ void __launch_bounds__(256)
heap_list_kernel(const uint2 *__restrict__ heap, uint32_t n, uint32_t K, uint32_t R,
                 uint32_t *list, unsigned int *tail) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t base = (uint64_t)blockIdx.x * blockDim.x; base < n; base += stride) {
    const uint64_t p = base + threadIdx.x;
    const uint2 it = p < n ? heap[p] : make_uint2(0u, 0u);
    const bool want = p < n && it.y >= K;
    const uint32_t bal = __ballot_sync(FULL, want);
    if (!bal) continue;
    uint32_t at = 0;
    if (lane_id() == (uint32_t)(__ffs(bal) - 1)) at = atomicAdd(tail, (unsigned int)__popc(bal));
    at = __shfl_sync(FULL, at, __ffs(bal) - 1) + __popc(bal & lanes_below());
    if (want && at < R) {
      list[at] = it.x;
      list[(size_t)R + at] = it.y;
      list[2 * (size_t)R + at] = (uint32_t)p;
    }
  }
}

}  // namespace

cudaError_t launch_make_heap(const uint32_t *count, uint32_t n, uint2 *heap, uint32_t K,
                             cudaStream_t stream) {
  uint32_t depth = 0;  // levels of the heap
  while (depth < 32 && ((1ull << depth) - 1) < n) ++depth;
  // shared memory holds 2^11 items of a lower stage (16 KB, six blocks an SM)
  // and 2^14 of the top one (128 KB, one block): its sifts are the longest
  constexpr uint32_t kTop = 14, kStage = 11;
  // (per device: the limit belongs to the current one)
  const cudaError_t e = cudaFuncSetAttribute(
      heap_stage_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(sizeof(uint2) << kTop));
  if (e != cudaSuccess) return e;
  while (depth > 0) {
    const bool top = depth <= kTop;
    uint32_t d0 = 0, L = depth, g = 0;
    if (!top) {
      d0 = depth > kTop + kStage ? depth - kStage : kTop;
      L = depth - d0;
      g = std::min(kStage - L, d0);
    }
    // roots of level d0 that exist, 2^g of them a block
    const uint64_t roots = std::min<uint64_t>(1ull << d0, n - ((1ull << d0) - 1));
    const uint32_t blocks = (uint32_t)((roots + (1ull << g) - 1) >> g);
    const uint32_t threads = top ? (L >= 10 ? 1024 : 256) : 256;
    count_launches(1);
    heap_stage_kernel<<<blocks, threads, sizeof(uint2) << (L + g), stream>>>(count, heap, n, d0, L,
                                                                             g, K);
    depth = d0;
  }
  return cudaGetLastError();
}

void launch_count_hist(const uint32_t *count, uint32_t n, uint32_t *hist, cudaStream_t stream) {
  count_launches(1);
  cudaMemsetAsync(hist, 0, sizeof(uint32_t) * kCountBuckets, stream);
  const uint32_t blocks = std::min<uint32_t>(592, (n + 255) / 256);
  count_hist_kernel<<<blocks, 256, 0, stream>>>(count, n, hist);
}

void launch_heap_counts(const uint2 *heap, uint32_t n, uint32_t *count, cudaStream_t stream) {
  count_launches(1);
  heap_counts_kernel<<<1184, 256, 0, stream>>>(heap, n, count);
}

void launch_heap_list(const uint2 *heap, uint32_t n, uint32_t K, uint32_t R, uint32_t *list,
                      unsigned int *tail, cudaStream_t stream) {
  count_launches(1);
  cudaMemsetAsync(tail, 0, sizeof(*tail), stream);
  const uint32_t blocks = std::min<uint32_t>(1184, (n + 255) / 256);
  heap_list_kernel<<<blocks, 256, 0, stream>>>(heap, n, K, R, list, tail);
}

void launch_count(const DevPool &P, uint64_t num_sets, uint32_t *count,
                  int blocks, cudaStream_t stream) {
  count_launches(1);
  count_kernel<<<blocks, kBlock, 0, stream>>>(P, num_sets, count);
}

size_t scan_block_sums_needed(uint32_t n) {
  return (size_t)((uint64_t)n + SCAN_TILE - 1) / SCAN_TILE + 1;
}

void launch_exclusive_scan(const uint32_t *in, uint64_t *out, uint32_t n,
                           uint64_t *block_sums, cudaStream_t stream) {
  count_launches(3);
  const uint32_t tiles = (uint32_t)((n + (uint64_t)SCAN_TILE - 1) / SCAN_TILE);
  if (tiles == 0) {
    cudaMemsetAsync(out, 0, sizeof(uint64_t), stream);
    return;
  }
  scan_tiles_kernel<<<tiles, SCAN_THREADS, 0, stream>>>(in, n, block_sums);
  scan_sums_kernel<<<1, SCAN_THREADS, 0, stream>>>(block_sums, tiles);
  scan_apply_kernel<<<tiles, SCAN_THREADS, 0, stream>>>(in, n, block_sums, out);
}

void launch_build_inverted(const DevPool &P, uint64_t num_sets,
                           uint64_t *cursor, uint32_t *inv, int blocks,
                           cudaStream_t stream, uint64_t base) {
  count_launches(1);
  inverted_kernel<<<blocks, kBlock, 0, stream>>>(P, num_sets, cursor, inv, base);
}

void launch_cover(const CoverLaunch &C, cudaStream_t stream) {
  count_launches(1);
  cover_kernel<<<C.blocks, kBlock, 0, stream>>>(C);
}

void launch_cover_list(const CoverLaunch &C, uint32_t *out, unsigned long long *cursor,
                       cudaStream_t stream) {
  count_launches(1);
  cover_list_kernel<<<C.blocks, 256, 0, stream>>>(C, out, cursor);
}

void launch_apply_decrements(uint32_t *count, uint32_t n, const uint32_t *dec, uint64_t m,
                             uint8_t *dirty, int blocks, cudaStream_t stream) {
  count_launches(1);
  apply_decrements_kernel<<<blocks, 256, 0, stream>>>(count, n, dec, m, dirty);
}

void launch_chunk_pick(const uint32_t *count, uint32_t n, uint8_t *dirty,
                       unsigned long long *cmax, unsigned long long *best, cudaStream_t stream) {
  const uint32_t nchunks = (n + kPickChunk - 1) / kPickChunk;
  count_launches(2);
  chunk_max_kernel<<<nchunks, 256, 0, stream>>>(count, n, dirty, cmax);
  cmax_max_kernel<<<1, 1024, 0, stream>>>(cmax, nchunks, best);
}

void launch_cover_gather(const CoverLaunch &C, const uint32_t *ids, uint32_t nids,
                         uint32_t *out, unsigned int *done, unsigned int *flag,
                         unsigned int epoch, cudaStream_t stream) {
  count_launches(1);
  cover_gather_kernel<<<C.blocks, kBlock, 0, stream>>>(C, ids, nids, out, done, flag, epoch);
}

void launch_coverage(const DevPool &P, uint64_t S, const uint32_t *marked,
                     unsigned long long *covered, int blocks, cudaStream_t stream) {
  count_launches(1);
  coverage_kernel<<<blocks, 256, 0, stream>>>(P, S, marked, covered);
}

void launch_sel_init(const SelDesc *d, int blocks, cudaStream_t stream) {
  count_launches(1);
  sel_init_kernel<<<blocks, 256, 0, stream>>>(d);
}
void launch_sel_count(const SelDesc *d, int blocks, cudaStream_t stream) {
  count_launches(1);
  sel_count_kernel<<<blocks, kBlock, 0, stream>>>(d);
}
void launch_sel_pick(const SelDesc *d, uint32_t i, int blocks, cudaStream_t stream) {
  count_launches(1);
  sel_pick_kernel<<<blocks, 256, 0, stream>>>(d, i);
}
void launch_sel_cover(const SelDesc *d, uint32_t i, int blocks, cudaStream_t stream) {
  count_launches(2);
  sel_cover_kernel<<<blocks, kBlock, 0, stream>>>(d, i);
  sel_recount_kernel<<<blocks, kBlock, 0, stream>>>(d);
}
void launch_sel_loop(const SelDesc *d, cudaStream_t stream) {
  count_launches(1);
  sel_loop_kernel<<<kLoopCtas, kLoopThreads, 0, stream>>>(d);
}
bool sel_loop_fits(uint32_t nchunks, double elements) {
  return nchunks <= kLoopCtas * kLoopChunks && elements <= kLoopElements;
}
uint32_t sel_chunk_vertices() { return SEL_CHUNK; }

void launch_gather_counts(const uint32_t *count, const uint32_t *ids, uint32_t m,
                          uint32_t *out, cudaStream_t stream) {
  if (m == 0) return;
  count_launches(1);
  gather_counts_kernel<<<std::min<uint32_t>((m + 255) / 256, 148), 256, 0, stream>>>(count, ids,
                                                                                     m, out);
}


}  // namespace rip
