// device.cuh -- device data views and warp-level helpers shared by the kernels.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "philox.cuh"

namespace rip {

constexpr uint32_t FULL = 0xFFFFFFFFu;

// Backward CSR packed for the sampler.  edges[e] = {source vertex, threshold}:
//   IC: threshold = floor(p_e * 2^32)  (edge live iff coin < threshold)
//   LT: threshold = floor(cumulative in-weight up to e * 2^32)
// off has n+1 entries; edges is padded with {0, 0} records to a multiple of 4
// and 32-byte aligned so a 4-edge group is one aligned 32-byte read.
// vthr (IC graphs, optional): vthr[v] != 0 when every in-edge of v has the
// threshold vthr[v] (weighted cascade: p = 1/in-degree); the IC samplers then
// compare v's coins against it and read only the sources of live edges.
// 0 means "read each edge's own threshold" (a uniform threshold of 0, an
// in-list that never fires, is stored as 0 too: still exact, only slower).
struct DevGraph {
  uint32_t n;
  uint64_t m;
  const uint32_t *off;
  const uint2 *edges;
  const uint32_t *vthr = nullptr;
};

// Flat RRR pool: set s occupies vtx[set_off[s] .. set_off[s] + set_len[s]).
struct DevPool {
  uint32_t *vtx;
  unsigned long long *cursor;  // next free element (atomic bump pointer)
  uint64_t cap;                // element capacity
  uint64_t *set_off;
  uint32_t *set_len;
};

// Failure list for sets that did not fit their scratch or the pool; the host
// re-runs them with larger buffers (results do not depend on the retry).
struct FailList {
  uint32_t *ids;          // indices relative to the launch's first set
  unsigned int *count;
  unsigned long long *first_bad_base;  // lowest pool offset of a failed reservation
  // sets handed over for their edge work: a list of their own, downwards from
  // big_end (a launch with a work cap has one; it stays on the device)
  uint32_t *big_end = nullptr;
  unsigned int *big_count = nullptr;
};

// Counters for roofline accounting (see rip_pool_stats in ripples_b200.h).
struct Stats {
  unsigned long long *v;  // [8]
};

__device__ __forceinline__ uint32_t lane_id() { return threadIdx.x & 31u; }
__device__ __forceinline__ uint32_t lanes_below() {  // mask of the lanes before this one
  uint32_t m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}

__device__ __forceinline__ uint32_t warp_incl_scan(uint32_t x) {
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    uint32_t y = __shfl_up_sync(FULL, x, d);
    if (lane_id() >= (uint32_t)d) x += y;
  }
  return x;
}

__device__ __forceinline__ unsigned long long warp_sum_u64(unsigned long long x) {
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) x += __shfl_xor_sync(FULL, x, d);
  return x;
}

// Given an inclusive warp scan `incl` (held per lane) of per-lane item
// counts, returns the lane whose range holds item j (0 <= j < total):
// the smallest lane i with incl[i] > j.  Five shuffle steps.
__device__ __forceinline__ uint32_t warp_find_owner(uint32_t incl, uint32_t j) {
  uint32_t lo = 0;
#pragma unroll
  for (int step = 16; step > 0; step >>= 1) {
    uint32_t probe = __shfl_sync(FULL, incl, lo + step - 1);
    if (probe <= j) lo += step;
  }
  return lo;
}

// Whether any of a block's eight coarse coins is at most th (a uniform
// threshold's coarse half): when none is, no edge of the block is live and
// none ties.  Two three-way minima of 16-bit pairs clip every coin at th + 1;
// any smaller half changes the word.  (th = 0xFFFF: every coin is.)
__device__ __forceinline__ bool block_clipped(const u32x4 &c, uint32_t lim) {
  return __vimin3_u16x2(__vimin3_u16x2(c.x, c.y, c.z), c.w, lim) != lim;
}
__device__ __forceinline__ bool block_any_le(const u32x4 &c, uint32_t th) {
  return block_clipped(c, (th + 1) * 0x10001u) || th == 0xFFFFu;
}

// Number of 4-edge groups covering [beg, end).
__device__ __forceinline__ uint32_t group_count(uint32_t beg, uint32_t end) {
  return end > beg ? ((end - 1) >> 2) - (beg >> 2) + 1 : 0;
}

// Number of 8-edge coin blocks covering [beg, end).
__device__ __forceinline__ uint32_t block_count(uint32_t beg, uint32_t end) {
  return end > beg ? ((end - 1) >> 3) - (beg >> 3) + 1 : 0;
}

// Live edges (bit h: edge 8b + h) of 8-edge coin block b of the in-list
// [ob, oe) for set s, given the block's coarse coins c: compared with the
// list's uniform threshold ovt (a whole block usually cleared by its smallest
// coin) or, when ovt is 0, with each record's own threshold (records read two
// at a time; a pair past the list's end is not read: the record array ends
// on a 4-edge boundary, not an 8-edge one).  A coarse tie (one edge in
// 65 536) draws the fine half.
__device__ __forceinline__ uint32_t ic_block_live(const DevGraph &G, Key key, uint64_t s,
                                                  uint32_t b, uint32_t ob, uint32_t oe,
                                                  uint32_t ovt, const u32x4 &c) {
  uint32_t live = 0, tie = 0;
  if (ovt) {
    const uint32_t th = ovt >> 16;
    if (!block_any_le(c, th)) return 0u;
#pragma unroll
    for (int h = 0; h < 8; ++h) {
      const uint32_t cc = coarse_of(c, h), e = (b << 3) + h;
      if (cc <= th && e >= ob && e < oe) {
        if (cc < th) live |= 1u << h;
        else tie |= 1u << h;
      }
    }
  } else {
    const uint4 *rp = reinterpret_cast<const uint4 *>(G.edges + ((size_t)b << 3));
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const uint32_t e0 = (b << 3) + 2 * q;
      if (e0 < oe && e0 + 1 >= ob) {
        const uint4 r = __ldg(rp + q);
        const uint32_t c0 = coarse_of(c, 2 * q), c1 = coarse_of(c, 2 * q + 1);
        if (e0 >= ob) {
          if (c0 < (r.y >> 16)) live |= 1u << (2 * q);
          else if (c0 == (r.y >> 16)) tie |= 1u << (2 * q);
        }
        if (e0 + 1 < oe) {
          if (c1 < (r.w >> 16)) live |= 2u << (2 * q);
          else if (c1 == (r.w >> 16)) tie |= 2u << (2 * q);
        }
      }
    }
  }
  while (tie) {
    const uint32_t h = __ffs(tie) - 1;
    tie &= tie - 1;
    const uint32_t e = (b << 3) + h;
    const uint32_t thr = ovt ? ovt : __ldg(&G.edges[e].y);
    if (ic_fine_call(key, e, s) < (thr & 0xFFFFu)) live |= 1u << h;
  }
  return live;
}

// Live edges of the 32 consecutive coin blocks from b0 on of the in-list
// [ob, oe), whose records hold the thresholds; called by the whole warp.  A
// lane that reads its own block's records strides 64 bytes: 64 L1 wavefronts a
// tile, 256 issue cycles of a scheduler's share of L1 against 90 of coins.  So
// the lanes read the tile's records side by side, two edges a lane and step (16
// wavefronts), and pass each other the coins through shared memory: word w of
// the tile's coins belongs to its edges 2w and 2w + 1.  Bit 2i + j of the result
// is edge 8 b0 + 64 i + 2 lane + j.  `ahead` of the four steps' records are read before the coins are drawn.
template <int ahead, class RK, class Fine>
__device__ __forceinline__ uint32_t tile_live(const DevGraph &G, const RK &rk,
                                              const CoinSet &cs, uint32_t b0, uint32_t ob,
                                              uint32_t oe, uint4 *coins, Fine &&fine) {
  const uint32_t lane = lane_id(), e0 = (b0 << 3) + 2 * lane;
  const uint4 *rp = reinterpret_cast<const uint4 *>(G.edges + ((size_t)b0 << 3)) + lane;
  uint4 rec[4];
  auto read = [&](int i) {
    const uint32_t e = e0 + 64 * i;
    rec[i] = e < oe && e + 1 >= ob ? __ldg(rp + 32 * i) : make_uint4(0, 0, 0, 0);
  };
#pragma unroll
  for (int i = 0; i < ahead; ++i) read(i);
  const u32x4 c = coin_block(rk, cs, b0 + lane);
  __syncwarp();
  coins[lane] = make_uint4(c.x, c.y, c.z, c.w);
  __syncwarp();
#pragma unroll
  for (int i = ahead; i < 4; ++i) read(i);
  const uint32_t *word = reinterpret_cast<const uint32_t *>(coins) + lane;
  uint32_t live = 0, tie = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint32_t e = e0 + 64 * i, w = word[32 * i];
    const uint32_t c0 = w & 0xFFFFu, c1 = w >> 16;
    const uint32_t t0 = e >= ob ? rec[i].y >> 16 : 0u, t1 = e + 1 < oe ? rec[i].w >> 16 : 0u;
    if (c0 < t0) live |= 1u << (2 * i);
    else if (c0 == t0) tie |= 1u << (2 * i);
    if (c1 < t1) live |= 2u << (2 * i);
    else if (c1 == t1) tie |= 2u << (2 * i);
  }
  while (tie) {  // one edge in 65 536 (and those out of the list): the fine half decides
    const uint32_t h = __ffs(tie) - 1;
    tie &= tie - 1;
    const uint32_t e = e0 + 64 * (h >> 1) + (h & 1);
    if (e >= ob && e < oe && fine(e) < (__ldg(&G.edges[e].y) & 0xFFFFu)) live |= 1u << h;
  }
  return live;
}

// Loads the 4 edge records of group g (32-byte aligned).
__device__ __forceinline__ void load_group(const uint2 *edges, uint32_t g,
                                           uint2 rec[4]) {
  const uint4 *p = reinterpret_cast<const uint4 *>(edges + ((size_t)g << 2));
  uint4 a = __ldg(p), b = __ldg(p + 1);
  rec[0] = make_uint2(a.x, a.y);
  rec[1] = make_uint2(a.z, a.w);
  rec[2] = make_uint2(b.x, b.y);
  rec[3] = make_uint2(b.z, b.w);
}

}  // namespace rip
