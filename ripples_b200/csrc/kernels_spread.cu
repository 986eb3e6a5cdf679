// kernels_spread.cu -- forward Monte Carlo spread of a seed set (IC, LT).
//
// The reference measures the quality of a seed set with ripples::simulate
// (include/ripples/diffusion_simulation.h:73-178, driven replica by replica
// by tools/simulator.cc); the spread is the number of vertices reached,
// seeds included.  Here one CTA runs one replica at a time, level by level, as
// the one-CTA-per-heavy-set sampler grows a set: warps take 32 of the level's
// entries at a time and sweep their shorter out-lists through the concatenated
// 8-edge blocks (a warp scan and a shuffle search, no barrier); lists of
// kTileBlocks blocks or more are listed and dealt to all warps in 32-block
// tiles.  Small levels are packed over the whole CTA (kPackEntries).
//   IC: out-edge e of a reached vertex fires in replica r iff its coin
//       (coarse half from block e >> 3 of its CoinSet, fine half from
//       sim_ic_fine on a coarse tie) is below threshold(e) (BFS over live
//       edges, diffusion_simulation.h:73-127).
//   LT: the live-edge form of the threshold model (Kempe, Kleinberg, Tardos,
//       KDD'03): vertex v keeps at most one in-edge -- the first j of its
//       in-list with sim_lt_threshold(key, r, v) < cum[j], cum being the
//       fixed-point cumulative in-weights the LT sampler uses -- and v is
//       reached iff the source of that in-edge is reached.  The reached set
//       has the distribution of diffusion_simulation.h:129-178's.
// Either way a replica's reached set is a pure function of (seed, r),
// whatever the visiting order.
//
// What bounds it: latency.  IC draws 90 issue cycles of coins a warp and coin
// block; a live edge costs round trips.  The reached bitmap sits in shared memory
// where it fits and replicas grow (spread_shape), so a live edge costs none to L2
// and the bitmaps leave L2 to the graph.
#include <type_traits>

#include "device.cuh"
#include "launch.h"

namespace rip {

namespace {

constexpr uint32_t kTileBlocks = 128;  // lists of at least this many blocks go in tiles
// Levels of at most this many entries are packed, in the 512-thread form with the
// bitmap in shared memory: a warp's share of a small level leaves lanes without a
// block, and its passes over live edges wait for each other, which is what replicas
// of a few thousand vertices spend their time on.  R-MAT, p ~ U(0, 0.02), 5 hubs as
// seeds, 1500 replicas: 2^16 vertices 0.86 -> 0.755 ms, 2^18 3.67 -> 3.48.  Packing
// levels of up to 512 entries gains more there (0.73), but loses where the seeds are
// 178 hubs (0.68 -> 0.76 at p ~ U(0, 0.05)).  The larger forms lose by it (2^20
// vertices, p ~ U(0, 0.1), 50 hubs: 50.9 -> 53.5).
constexpr uint32_t kPackEntries = 128;
constexpr uint32_t kSimLong = 256;  // long lists a level may list

template <bool SHARED, int THREADS>
__global__ void __launch_bounds__(THREADS, THREADS == 1024 ? 1 : 4)
spread_ic_kernel(const __grid_constant__ SpreadLaunch L) {
  constexpr uint32_t WARPS = THREADS / 32;
  // the targets of a block's edges: kept in registers where there are 64 a
  // thread, else read again from L1
  constexpr bool KEEP = THREADS == 1024;
  constexpr bool PACK = SHARED && !KEEP;
  extern __shared__ uint4 s_dyn[];  // SHARED: the reached bitmap
  static_assert(kPackEntries <= kSimLong, "one room for both");
  __shared__ uint32_t s_beg[kSimLong], s_end[kSimLong];  // a packed level's entries, or long lists
  __shared__ uint32_t s_off[PACK ? kPackEntries : 1], s_warp[32];
  __shared__ uint32_t s_qlen, s_nlong, s_next;  // the last two zero between levels
  __shared__ unsigned long long s_rep;

  const uint32_t tid = threadIdx.x, lane = lane_id(), wid = tid >> 5;
  uint32_t *bm = SHARED ? reinterpret_cast<uint32_t *>(s_dyn)
                        : L.bitmaps + (size_t)blockIdx.x * L.bm_words;
  uint32_t *q = L.queues + (size_t)blockIdx.x * L.qcap;
  const uint32_t words4 = (uint32_t)((L.bm_words + 3) / 4);  // SHARED
  unsigned long long reached = 0;
  if (SHARED)
    for (uint32_t i = tid; i < words4; i += THREADS) s_dyn[i] = make_uint4(0, 0, 0, 0);

  for (;;) {
    if (tid == 0) {
      s_rep = atomicAdd(L.next, 1ull);
      s_qlen = 0;
      s_nlong = s_next = 0;
    }
    __syncthreads();
    const uint64_t r = s_rep;
    if (r >= L.replicas) break;
    // the seeds are the first level (a repeated seed is queued once)
    for (uint32_t i = tid; i < L.k; i += THREADS) {
      const uint32_t v = L.seeds[i];
      const uint32_t bit = 1u << (v & 31);
      if (!(atomicOr(&bm[v >> 5], bit) & bit)) {
        const uint32_t pos = atomicAdd(&s_qlen, 1u);
        if (pos < L.qcap) q[pos] = v;
      }
    }
    const CoinSet cs = coin_set(L.rk, r, DOM_SIM_IC);
    __syncthreads();
    // Queues this lane's vertex u (if any) unless it is reached already; all
    // lanes of the warp call it.
    auto reach = [&](bool want, uint32_t u) {
      const uint32_t bit = 1u << (u & 31);
      const bool isnew = want && !(atomicOr(&bm[u >> 5], bit) & bit);
      const uint32_t bal = __ballot_sync(FULL, isnew);
      if (!bal) return;
      uint32_t pos = 0;
      if (lane == (uint32_t)(__ffs(bal) - 1)) pos = atomicAdd(&s_qlen, (uint32_t)__popc(bal));
      pos = __shfl_sync(FULL, pos, __ffs(bal) - 1) + __popc(bal & lanes_below());
      if (isnew && pos < L.qcap) q[pos] = u;
    };
    // Draws 8-edge block b's edges in [ob, oe) (an empty range: none) and follows
    // those that fire: each lane its own, or (`together`) one a lane and pass, by
    // the whole warp.  Records are read two at a time (a pair past the list's end
    // is not read: the record array ends on a 4-edge boundary).
    auto expand_block = [&](auto together, uint32_t b, uint32_t ob, uint32_t oe) {
      const uint4 *rp = reinterpret_cast<const uint4 *>(L.G.edges + ((size_t)b << 3));
      const u32x4 c = coin_block(L.rk, cs, b);
      uint32_t u[8], live = 0, tie = 0;
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        const uint32_t e0 = (b << 3) + 2 * h;
        if (KEEP) u[2 * h] = u[2 * h + 1] = 0;
        if (e0 < oe && e0 + 1 >= ob) {
          const uint4 x = __ldg(rp + h);
          if (KEEP) {
            u[2 * h] = x.x;
            u[2 * h + 1] = x.z;
          }
          const uint32_t c0 = coarse_of(c, 2 * h), c1 = coarse_of(c, 2 * h + 1);
          if (e0 >= ob) {
            if (c0 < (x.y >> 16)) live |= 1u << (2 * h);
            else if (c0 == (x.y >> 16)) tie |= 1u << (2 * h);
          }
          if (e0 + 1 < oe) {
            if (c1 < (x.w >> 16)) live |= 2u << (2 * h);
            else if (c1 == (x.w >> 16)) tie |= 2u << (2 * h);
          }
        }
      }
      while (tie) {  // one edge in 65 536: the fine half decides
        const uint32_t h = __ffs(tie) - 1;
        tie &= tie - 1;
        const uint32_t e = (b << 3) + h;
        if (sim_ic_fine_call(L.key, e, r) < (__ldg(&L.G.edges[e].y) & 0xFFFFu)) live |= 1u << h;
      }
      while (together.value ? __any_sync(FULL, live != 0) : live != 0) {
        uint32_t x = 0;
        bool want = live != 0;
        if (want) {
          const uint32_t h = __ffs(live) - 1;
          live &= live - 1;
          if (KEEP) {
#pragma unroll
            for (int t = 0; t < 8; ++t)
              if (h == (uint32_t)t) x = u[t];
          } else {
            x = __ldg(&L.G.edges[(b << 3) + h].x);
          }
          // (bits are only set: a plain read spares the atomic where it is as near)
          if (SHARED && (!KEEP || !together.value)) want = !((bm[x >> 5] >> (x & 31)) & 1u);
        }
        if (together.value) {
          reach(want, x);
        } else if (want) {
          const uint32_t bit = 1u << (x & 31);
          if (!(atomicOr(&bm[x >> 5], bit) & bit)) {
            const uint32_t pos = atomicAdd(&s_qlen, 1u);
            if (pos < L.qcap) q[pos] = x;
          }
        }
      }
    };
    constexpr auto alone = std::false_type{};
    constexpr auto together = std::true_type{};
    uint32_t lo = 0, hi = min(s_qlen, L.qcap), levels = 0;
    __syncthreads();
    while (lo < hi) {
      ++levels;  // one BFS level (the seeds are the first)
      if (PACK && hi - lo <= kPackEntries) {
        // a small level: its blocks side by side over the whole CTA
        const uint32_t e = lo + tid;
        uint32_t nb = 0;
        if (tid < kPackEntries) {
          uint32_t beg = 0, end = 0;
          if (e < hi) {
            const uint32_t v = q[e];
            beg = __ldg(L.G.off + v);
            end = __ldg(L.G.off + v + 1);
          }
          s_beg[tid] = beg;
          s_end[tid] = end;
          nb = block_count(beg, end);
        }
        const uint32_t incl = warp_incl_scan(nb);
        if (lane == 31) s_warp[wid] = incl;
        __syncthreads();
        const uint32_t own = lane < WARPS ? s_warp[lane] : 0u, upto = warp_incl_scan(own);
        const uint32_t total = __shfl_sync(FULL, upto, 31);
        const uint32_t before = __shfl_sync(FULL, upto - own, wid);
        if (tid < kPackEntries) s_off[tid] = before + incl - nb;
        __syncthreads();
        for (uint32_t j = tid; j < total; j += THREADS) {
          uint32_t a = 0, z = hi - lo;  // entry a: s_off[a] <= j < s_off[a + 1]
          while (z - a > 1) {
            const uint32_t mid = (a + z) >> 1;
            if (s_off[mid] <= j) a = mid;
            else z = mid;
          }
          expand_block(alone, (s_beg[a] >> 3) + (j - s_off[a]), s_beg[a], s_end[a]);
        }
      } else {
        // 1. warps take the level's entries, up to 32 at a time
        const uint32_t share = min(32u, (hi - lo + WARPS - 1) / WARPS);
        for (;;) {
          uint32_t at = 0;
          if (lane == 0) at = atomicAdd(&s_next, share);
          at = __shfl_sync(FULL, at, 0);
          if (at >= hi - lo) break;
          const uint32_t e = lo + at + lane;
          uint32_t beg = 0, end = 0;
          if (lane < share && e < hi) {
            const uint32_t v = q[e];
            beg = __ldg(L.G.off + v);
            end = __ldg(L.G.off + v + 1);
          }
          uint32_t nb = block_count(beg, end);
          if (nb >= kTileBlocks) {
            const uint32_t pos = atomicAdd(&s_nlong, 1u);
            if (pos < kSimLong) {
              s_beg[pos] = beg;
              s_end[pos] = end;
              nb = 0;
            }  // (no room: this warp sweeps it with the others)
          }
          const uint32_t incl = warp_incl_scan(nb);
          const uint32_t total = __shfl_sync(FULL, incl, 31);
          for (uint32_t base = 0; base < total; base += 32) {
            const uint32_t j = base + lane;
            const uint32_t owner = warp_find_owner(incl, min(j, total - 1));
            const uint32_t ob = __shfl_sync(FULL, beg, owner);
            const uint32_t oe = __shfl_sync(FULL, end, owner);
            const uint32_t oexcl = __shfl_sync(FULL, incl - nb, owner);
            const bool valid = j < total;
            expand_block(together, valid ? (ob >> 3) + (j - oexcl) : 0u, valid ? ob : 0u,
                         valid ? oe : 0u);
          }
        }
        __syncthreads();
        // 2. the long lists, dealt to the warps a tile of 32 blocks at a time
        const uint32_t nlong = min(s_nlong, kSimLong);
        uint32_t deal = wid;  // (wid - tiles dealt so far) mod WARPS: this warp's next tile
        for (uint32_t a = 0; a < nlong; ++a) {
          const uint32_t ob = s_beg[a], oe = s_end[a];
          const uint32_t b_last = (oe - 1) >> 3;
          const uint32_t ntiles = ((b_last - (ob >> 3)) >> 5) + 1;
          for (uint32_t t = deal & (WARPS - 1); t < ntiles; t += WARPS) {
            const uint32_t b = (ob >> 3) + t * 32 + lane;
            const bool valid = b <= b_last;
            expand_block(together, valid ? b : 0u, valid ? ob : 0u, valid ? oe : 0u);
          }
          deal -= ntiles;
        }
      }
      __syncthreads();
      lo = hi;
      hi = min(s_qlen, L.qcap);
      if (tid == 0) s_nlong = s_next = 0;
      __syncthreads();
    }
    // every vertex is queued at most once, so qlen <= n = qcap
    const uint32_t qlen = hi;
    if (tid == 0) {
      if (L.sizes) L.sizes[r] = qlen;
      if (L.levels) L.levels[r] = levels;
      reached += qlen;
    }
    if (SHARED && qlen >= words4) {
      for (uint32_t i = tid; i < words4; i += THREADS) s_dyn[i] = make_uint4(0, 0, 0, 0);
    } else {
      for (uint32_t i = tid; i < qlen; i += THREADS) bm[q[i] >> 5] = 0u;
    }
    __syncthreads();
  }
  if (tid == 0 && reached) atomicAdd(L.total, reached);
}

// LT past 65536 vertices: four 512-thread CTAs per SM (32 registers a thread: 64 resident warps).
// The kernel waits on L2 latency, so replicas in flight are what move it:
// fewer and larger CTAs (one of 1024 threads, two of 768) were slower.
constexpr int SIM_THREADS = 512;
constexpr int SIM_WARPS = SIM_THREADS / 32;

__device__ uint32_t sim_block_scan(uint32_t x, uint32_t *warp_tot, uint32_t *total) {
  const uint32_t lane = lane_id(), wid = threadIdx.x >> 5;
  const uint32_t incl = warp_incl_scan(x);
  if (lane == 31) warp_tot[wid] = incl;
  __syncthreads();
  if (wid == 0) {
    const uint32_t t = lane < SIM_WARPS ? warp_tot[lane] : 0u;
    const uint32_t ti = warp_incl_scan(t);
    if (lane < SIM_WARPS) warp_tot[lane] = ti - t;
    if (lane == 31) *total = ti;
  }
  __syncthreads();
  const uint32_t r = warp_tot[wid] + incl - x;
  __syncthreads();
  return r;
}

constexpr uint32_t NO_VERTEX = 0xFFFFFFFFu;

// LT: the source of the in-edge vertex v keeps in replica r, or NO_VERTEX.
// cum is non-decreasing along the in-list, so the first j with t < cum[j] is
// found by binary search.
__device__ __forceinline__ uint32_t lt_kept_source(const DevGraph &B, Key key, uint64_t r,
                                                   uint32_t v) {
  const uint32_t lo = __ldg(B.off + v), hi = __ldg(B.off + v + 1);
  if (lo == hi) return NO_VERTEX;
  const uint32_t t = sim_lt_threshold(key, r, v);
  if (!(t < __ldg(B.edges + (hi - 1)).y)) return NO_VERTEX;  // keeps no in-edge
  uint32_t a = lo, b = hi - 1;  // cum[b] > t
  while (a < b) {
    const uint32_t mid = a + ((b - a) >> 1);  // edge ids reach 2^32: no a + b
    if (__ldg(B.edges + mid).y > t) b = mid;
    else a = mid + 1;
  }
  return __ldg(B.edges + a).x;
}

__global__ void __launch_bounds__(SIM_THREADS, 4)
spread_lt_kernel(SpreadLaunch L) {
  __shared__ uint32_t s_off[SIM_THREADS + 1];
  __shared__ uint32_t s_beg[SIM_THREADS], s_end[SIM_THREADS];
  __shared__ uint32_t s_v[SIM_THREADS];  // the entry's vertex
  __shared__ uint32_t s_warp[SIM_WARPS];
  __shared__ uint32_t s_qlen, s_total;
  __shared__ unsigned long long s_rep;

  const uint32_t tid = threadIdx.x;
  uint32_t *bm = L.bitmaps + (size_t)blockIdx.x * L.bm_words;
  uint32_t *q = L.queues + (size_t)blockIdx.x * L.qcap;
  unsigned long long reached = 0;

  for (;;) {
    if (tid == 0) {
      s_rep = atomicAdd(L.next, 1ull);
      s_qlen = 0;
    }
    __syncthreads();
    const uint64_t r = s_rep;
    if (r >= L.replicas) break;
    // the seeds are the first level (a repeated seed is queued once)
    for (uint32_t i = tid; i < L.k; i += SIM_THREADS) {
      const uint32_t v = L.seeds[i];
      const uint32_t bit = 1u << (v & 31);
      if (!(atomicOr(&bm[v >> 5], bit) & bit)) {
        const uint32_t pos = atomicAdd(&s_qlen, 1u);
        if (pos < L.qcap) q[pos] = v;
      }
    }
    __syncthreads();
    uint32_t lo = 0, hi = min(s_qlen, L.qcap), levels = 0;
    while (lo < hi) {
      ++levels;  // one BFS level (the seeds are the first)
      for (uint32_t cb = lo; cb < hi; cb += SIM_THREADS) {
        const uint32_t e = cb + tid;
        uint32_t beg = 0, end = 0;
        if (e < hi) {
          const uint32_t v = q[e];
          beg = __ldg(L.G.off + v);
          end = __ldg(L.G.off + v + 1);
          s_v[tid] = v;
        }
        s_beg[tid] = beg;
        s_end[tid] = end;
        const uint32_t ng = group_count(beg, end);
        s_off[tid] = sim_block_scan(ng, s_warp, &s_total);
        if (tid == 0) s_off[SIM_THREADS] = s_total;
        __syncthreads();
        const uint32_t total = s_off[SIM_THREADS];
        for (uint32_t j = tid; j < total; j += SIM_THREADS) {
          uint32_t a = 0, b = SIM_THREADS;  // entry a: s_off[a] <= j < s_off[a + 1]
          while (b - a > 1) {
            const uint32_t mid = (a + b) >> 1;
            if (s_off[mid] <= j) a = mid;
            else b = mid;
          }
          const uint32_t ob = s_beg[a], oe = s_end[a];
          const uint32_t g = (ob >> 2) + (j - s_off[a]);
          uint2 rec[4];
          load_group(L.G.edges, g, rec);
          const uint32_t from = s_v[a];
#pragma unroll
          for (int t = 0; t < 4; ++t) {
            const uint32_t ed = (g << 2) + t;
            if (ed < ob || ed >= oe) continue;
            const uint32_t u = rec[t].x;
            const uint32_t bit = 1u << (u & 31);
            // a plain read first: reached bits are only ever set
            if ((__ldcg(&bm[u >> 5]) & bit) || lt_kept_source(L.B, L.key, r, u) != from)
              continue;
            if (!(atomicOr(&bm[u >> 5], bit) & bit)) {
              const uint32_t pos = atomicAdd(&s_qlen, 1u);
              if (pos < L.qcap) q[pos] = u;
            }
          }
        }
        __syncthreads();
      }
      lo = hi;
      hi = min(s_qlen, L.qcap);
      __syncthreads();
    }
    // every vertex is queued at most once, so qlen <= n = qcap
    const uint32_t qlen = min(s_qlen, L.qcap);
    if (tid == 0) {
      if (L.sizes) L.sizes[r] = qlen;
      if (L.levels) L.levels[r] = levels;
      reached += qlen;
    }
    for (uint32_t i = tid; i < qlen; i += SIM_THREADS) bm[q[i] >> 5] = 0u;
    __syncthreads();
  }
  if (tid == 0 && reached) atomicAdd(L.total, reached);
}

// LT with vertex ids of 16 bits.  Sweeping the out-lists of reached vertices
// tries a vertex once for every reached in-neighbour, each try a search of its
// in-list by dependent L2 reads.  Once a replica's levels have more out-edges
// than n / kSweepShare, the in-edge every vertex keeps is drawn instead, once, and
// no out-list is read any more: a vertex is reached iff the chain of kept sources
// from it meets a reached vertex.
// The chains are halved round by round: a vertex whose source is not reached takes
// its source's source.  (Levels one by one are a pass over all vertices each, and
// sparse graphs have hundreds of them.)  The halving stops after a round that
// reaches nobody: of the vertices with a chain to a reached one, not reached yet,
// the one with the shortest chain has a reached source (sources never skip past
// the sweep's reached vertices) and joins in the next round.
// LEVELS: a vertex's level is its chain's length, so the sources are 32-bit words
// with it (length in the low half), in the queue's place in L2; lengths stay below
// 2^16 as chains have no vertex twice.
// 2000 replicas: an R-MAT graph's 20 hubs (2^16 vertices, 768 K edges) 26.1 ms by
// sweeps to the end, 8.2 by levels, 2.5 by halving; 2^16 Erdos-Renyi vertices of
// degree 10, 50 (5) seeds 20.6 (11.4), 47.5 (20.3), 3.0 (3.3).  What bounds it: half
// the issue slots are busy; the draw waits for the searches' reads, two of them in
// flight a thread, the halving at the CTA's barriers.
constexpr uint32_t kSweepShare = 64;  // (those 3.0 (3.3) ms: 4.3 (4.8) at 16, 14.6 (11.0) at 2)

template <int THREADS, bool LEVELS>
__global__ void __launch_bounds__(THREADS, THREADS == 1024 ? 1 : 3)
spread_lt_small_kernel(const __grid_constant__ SpreadLaunch L) {
  constexpr uint32_t WARPS = THREADS / 32;
  extern __shared__ uint4 s_dyn[];
  __shared__ uint32_t s_qlen, s_size, s_deep;
  __shared__ unsigned long long s_rep, s_work;
  const uint32_t tid = threadIdx.x, lane = lane_id(), wid = tid >> 5;
  const uint32_t n = L.G.n, words = (uint32_t)L.bm_words;
  volatile uint32_t *bm = reinterpret_cast<uint32_t *>(s_dyn);
  volatile uint16_t *kept = reinterpret_cast<uint16_t *>(reinterpret_cast<uint32_t *>(s_dyn) + words);
  uint32_t *q = L.queues + (size_t)blockIdx.x * L.qcap;
  auto is_reached = [&](uint32_t u) -> bool { return bm[u >> 5] >> (u & 31) & 1u; };
  unsigned long long reached = 0;
  for (;;) {
    if (tid == 0) {
      s_rep = atomicAdd(L.next, 1ull);
      s_qlen = s_size = s_deep = 0;
      s_work = 0;
    }
    for (uint32_t w = tid; w < words; w += THREADS) bm[w] = 0;
    __syncthreads();
    const uint64_t r = s_rep;
    if (r >= L.replicas) break;
    auto reach = [&](uint32_t u) {  // (every vertex is queued once at most: n = qcap)
      const uint32_t bit = 1u << (u & 31);
      if (atomicOr(const_cast<uint32_t *>(&bm[u >> 5]), bit) & bit) return;
      const uint32_t pos = atomicAdd(&s_qlen, 1u);
      if (pos < L.qcap) q[pos] = u;
    };
    for (uint32_t i = tid; i < L.k; i += THREADS) reach(L.seeds[i]);
    __syncthreads();
    uint32_t lo = 0, hi = min(s_qlen, L.qcap), levels = 0;
    bool scan = false;
    while (lo < hi) {
      ++levels;  // one BFS level (the seeds are the first)
      unsigned long long work = 0;
      for (uint32_t e = lo + tid; e < hi; e += THREADS) {
        const uint32_t v = q[e];
        work += __ldg(L.G.off + v + 1) - __ldg(L.G.off + v);
      }
      work = warp_sum_u64(work);
      if (lane == 0 && work) atomicAdd(&s_work, work);
      __syncthreads();
      if (s_work > n / kSweepShare) {
        scan = true;
        break;
      }
      for (uint32_t cb = lo + wid * 32; cb < hi; cb += WARPS * 32) {
        const uint32_t e = cb + lane;
        uint32_t beg = 0, end = 0, v = 0;
        if (e < hi) {
          v = q[e];
          beg = __ldg(L.G.off + v);
          end = __ldg(L.G.off + v + 1);
        }
        const uint32_t ng = group_count(beg, end), incl = warp_incl_scan(ng);
        const uint32_t total = __shfl_sync(FULL, incl, 31);
        for (uint32_t base = 0; base < total; base += 32) {
          const uint32_t j = base + lane;
          const uint32_t owner = warp_find_owner(incl, min(j, total - 1));
          const uint32_t ob = __shfl_sync(FULL, beg, owner), oe = __shfl_sync(FULL, end, owner);
          const uint32_t from = __shfl_sync(FULL, v, owner);
          const uint32_t g = (ob >> 2) + j - __shfl_sync(FULL, incl - ng, owner);
          if (j >= total) continue;
          uint2 rec[4];
          load_group(L.G.edges, g, rec);
#pragma unroll
          for (int t = 0; t < 4; ++t) {
            const uint32_t ed = (g << 2) + t, u = rec[t].x;
            if (ed < ob || ed >= oe) continue;
            if (!is_reached(u) && lt_kept_source(L.B, L.key, r, u) == from) reach(u);
          }
        }
      }
      __syncthreads();
      lo = hi;
      hi = min(s_qlen, L.qcap);
      __syncthreads();
    }
    if (scan) {
      uint32_t joined = 0, deep = 0;  // LEVELS: this thread's vertices reached, the longest chain
      bool grew = false;
      // the kept sources (none: the vertex itself), two vertices a thread in flight
      for (uint32_t v0 = tid; v0 < n; v0 += 2 * THREADS) {
        uint32_t a[2], b[2], t[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const uint32_t v = v0 + i * THREADS;
          a[i] = b[i] = 0;
          if (v < n) {
            a[i] = __ldg(L.B.off + v);
            b[i] = __ldg(L.B.off + v + 1);
          }
        }
        bool some[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          t[i] = sim_lt_threshold(L.key, r, v0 + i * THREADS);
          some[i] = a[i] < b[i] && t[i] < __ldg(&L.B.edges[b[i] - 1].y);
          b[i] = some[i] ? b[i] - 1 : a[i];  // cum[b] > t
        }
        while (a[0] < b[0] || a[1] < b[1]) {
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            if (a[i] >= b[i]) continue;
            const uint32_t mid = a[i] + ((b[i] - a[i]) >> 1);
            if (__ldg(&L.B.edges[mid].y) > t[i]) b[i] = mid;
            else a[i] = mid + 1;
          }
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const uint32_t v = v0 + i * THREADS;
          if (v >= n) continue;
          const uint32_t u = some[i] ? __ldg(&L.B.edges[a[i]].x) : v;
          if (LEVELS) {
            __stcg(q + v, u << 16 | (u != v));
            if (is_reached(u) && !is_reached(v)) {
              deep = 1;
              ++joined;
            }
          } else {
            kept[v] = (uint16_t)u;
          }
        }
      }
      if (LEVELS) {
        do {
          __syncthreads();
          grew = false;
          for (uint32_t v = tid; v < n; v += THREADS) {
            if (is_reached(v)) continue;
            const uint32_t x = __ldcg(q + v), u = x >> 16;
            if (u == v || is_reached(u)) continue;  // no source, or done
            const uint32_t y = __ldcg(q + u), len = (x + y) & 0xFFFFu;
            __stcg(q + v, (y & 0xFFFF0000u) | len);
            if (is_reached(y >> 16)) {
              grew = true;
              deep = max(deep, len);
              ++joined;
            }
          }
        } while (__syncthreads_or(grew));
        deep = __reduce_max_sync(FULL, deep);
        if (lane == 0 && deep) atomicMax(&s_deep, deep);
      } else {
        do {
          __syncthreads();
          grew = false;
          constexpr uint32_t U = 4;  // words in flight: three dependent reads each
          for (uint32_t w0 = wid; w0 < words; w0 += U * WARPS) {
            uint32_t was[U], u[U], to[U];
            bool open[U], joins[U];
#pragma unroll
            for (uint32_t i = 0; i < U; ++i) {
              const uint32_t w = w0 + i * WARPS;
              was[i] = FULL;
              if (w < words) was[i] = bm[w];
              open[i] = !(was[i] >> lane & 1u) && w * 32 + lane < n;
            }
#pragma unroll
            for (uint32_t i = 0; i < U; ++i)
              if (open[i]) u[i] = kept[(w0 + i * WARPS) * 32 + lane];
#pragma unroll
            for (uint32_t i = 0; i < U; ++i) {
              joins[i] = open[i] && is_reached(u[i]);
              if (open[i]) to[i] = kept[u[i]];
            }
#pragma unroll
            for (uint32_t i = 0; i < U; ++i) {
              const uint32_t w = w0 + i * WARPS;
              if (open[i] && !joins[i]) kept[w * 32 + lane] = (uint16_t)to[i];
              const uint32_t add = __ballot_sync(FULL, joins[i]);
              if (add && lane == 0) bm[w] = was[i] | add;
              grew = grew || add != 0;
            }
          }
        } while (__syncthreads_or(grew));
      }
      for (uint32_t w = tid; w < words; w += THREADS) joined += __popc(bm[w]);
      joined = __reduce_add_sync(FULL, joined);
      if (lane == 0 && joined) atomicAdd(&s_size, joined);
      __syncthreads();
      levels += s_deep;
    }
    if (tid == 0) {
      const uint32_t size = scan ? s_size : hi;
      if (L.sizes) L.sizes[r] = size;
      if (LEVELS) L.levels[r] = levels;
      reached += size;
    }
    __syncthreads();
  }
  if (tid == 0 && reached) atomicAdd(L.total, reached);
}

// Shared memory of an SM's CTAs, and what a spread CTA takes besides its dynamic
// part (static and reserved, rounded up).
constexpr size_t kSmShared = 227 * 1024;
constexpr size_t kSpreadStatic = 5120;
// Dynamic shared memory of the kernels below at most, by CTAs an SM.
constexpr size_t kIcShared4 = (kSmShared / 4 - kSpreadStatic) & ~(size_t)15;
constexpr size_t kIcShared1 = kSmShared - kSpreadStatic;
constexpr size_t lt_shared(size_t n) { return ((n + 31) / 32 * 4 + 2 * n + 15) & ~(size_t)15; }
constexpr size_t kLtLevels = 65536 / 8;
constexpr size_t kLtShared3 = kSmShared / 3 - 2048;
constexpr size_t kLtShared1 = lt_shared(65536);

// The limit set is the kernel's largest shape, not this launch's: it belongs to
// the kernel, and another thread may launch it for a larger graph meanwhile.
template <class Kernel>
cudaError_t launch_shared(Kernel kernel, const SpreadLaunch &L, int threads, size_t shared,
                          size_t limit, cudaStream_t stream) {
  const cudaError_t e =
      cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)limit);
  if (e != cudaSuccess) return e;
  kernel<<<L.blocks, threads, shared, stream>>>(L);
  return cudaGetLastError();
}

}  // namespace

// LT: up to 65536 vertices three 512-thread CTAs an SM where their bitmaps and
// 16-bit sources fit (n up to 34 K; with levels: always, the sources are in
// L2), else one of 1024; past that no shared form.
// IC: four 512-thread CTAs per SM with the bitmap in shared memory where four
// fit (n up to about 400 K), else one 1024-thread CTA with it where that fits (1.79
// million) and replicas grow (`super`: the branching factor of a traversal is above
// kSupercritical), else four with it in global memory.
// R-MAT, p ~ U(0, 0.1), 50 hubs as seeds, against block-wide scans of every
// level with the bitmap in global memory: 2^16 vertices, 1500 replicas 3.63 ->
// 3.50 ms; 2^18 14.9 -> 14.1 (four CTAs; one: 15.2); 2^20 62.9 -> 50.9 (one; in
// global memory: 59.8); 2^22, 300 replicas 77.7 -> 71.0 (global).  Replicas that
// end with a few vertices would wait for each other at one CTA an SM: 2^20
// Erdos-Renyi vertices, p ~ U(0, 0.06), 100 seeds, 1500 replicas 0.20 ms, 0.14 with
// four.
SpreadShape spread_shape(uint32_t n, bool lt, bool levels, bool super) {
  const size_t bitmap = (((size_t)n + 127) / 128) * 16;
  if (lt && n <= 65536) {  // the bitmap and the kept sources
    if (levels) return SpreadShape{512, 3, bitmap};
    const size_t bytes = lt_shared(n);
    return bytes <= kLtShared3 ? SpreadShape{512, 3, bytes} : SpreadShape{1024, 1, bytes};
  }
  if (lt) return SpreadShape{SIM_THREADS, 4, 0};
  if (bitmap <= kIcShared4) return SpreadShape{512, 4, bitmap};
  if (super && bitmap <= kIcShared1) return SpreadShape{1024, 1, bitmap};
  return SpreadShape{512, 4, 0};
}

cudaError_t launch_spread(const SpreadLaunch &L0, bool lt, const SpreadShape &s,
                          cudaStream_t stream) {
  count_launches(1);
  SpreadLaunch L = L0;
  L.rk = round_keys(L.key);
  if (lt && s.shared && L.levels)
    return launch_shared(spread_lt_small_kernel<512, true>, L, 512, s.shared, kLtLevels, stream);
  if (lt && s.shared && s.threads == 1024)
    return launch_shared(spread_lt_small_kernel<1024, false>, L, 1024, s.shared, kLtShared1, stream);
  if (lt && s.shared)
    return launch_shared(spread_lt_small_kernel<512, false>, L, 512, s.shared, kLtShared3, stream);
  if (!lt && s.shared && s.threads == 1024)
    return launch_shared(spread_ic_kernel<true, 1024>, L, 1024, s.shared, kIcShared1, stream);
  if (!lt && s.shared)
    return launch_shared(spread_ic_kernel<true, 512>, L, 512, s.shared, kIcShared4, stream);
  if (lt) spread_lt_kernel<<<L.blocks, SIM_THREADS, 0, stream>>>(L);
  else spread_ic_kernel<false, 512><<<L.blocks, 512, 0, stream>>>(L);
  return cudaGetLastError();
}

}  // namespace rip
