// kernels_sample.cu -- RRR-set sampling kernels for sm_100a.
//
// ic_plain_kernel   one IC set per warp: reverse BFS over live in-edges
//                   (semantics of include/ripples/add_rrrset.h:128-135, with
//                   the per-edge coin keyed on (set, edge) instead of drawn
//                   from a sequential trng stream).
// lt_walk_kernel    one LT set per warp: single-predecessor walk
//                   (include/ripples/add_rrrset.h:136-150) with no length cap
//                   and no host fallback (the reference GPU walk stops at 8
//                   vertices and redoes longer walks on the CPU,
//                   include/ripples/gpu/lt_kernel.h:59-130,
//                   streaming_rrr_generator.h:492-520).
//
// Both are persistent: each warp pulls set indices from an atomic counter
// until the range is exhausted.  A warp owns an n-bit visited bitmap and a
// queue (the set's members in discovery order) in global scratch; at the end
// of a set it reserves room in the pool with one atomicAdd, copies the queue
// out and clears exactly the bitmap words it touched.  A set that outgrows
// the queue, or does not fit in the pool, is recorded in the failure list and
// the host re-runs it with larger buffers -- the result does not change,
// because every draw is a pure function of (seed, set id, edge / vertex id).
#include "device.cuh"
#include "launch.h"
#include "ripples_b200.h"

namespace rip {

namespace {

// In-lists of at least this many 8-edge coin blocks are swept by a whole
// warp at a time instead of sharing it with other lists.
constexpr uint32_t kLongBlocks = 32;

struct WarpCtx {
  uint32_t *bm;  // visited bitmap, ceil(n/32) words
  uint32_t *q;   // queue, qcap entries
  uint32_t qcap;
  uint32_t *seen = nullptr;  // LT: the walk's revisit filter (shared memory)
  uint4 *coins = nullptr;    // IC: a tile's coins (shared memory)
  uint32_t *ev = nullptr;    // IC: live edges on their way to the queue (64, shared memory)
};

// Writes the finished set to the pool (unless it overflowed) and clears the
// warp's bitmap.  Returns true when the set was stored; on a pool overflow
// the reservation's offset is recorded in *first_bad.
__device__ bool store_set(const WarpCtx &W, uint32_t qlen, bool overflow, uint64_t s,
                          const DevPool &P, unsigned long long *first_bad,
                          bool clear_bitmap = true) {
  const uint32_t lane = lane_id();
  bool stored = false;
  if (!overflow) {
    unsigned long long b = 0;
    if (lane == 0) b = atomicAdd(P.cursor, (unsigned long long)qlen);
    b = __shfl_sync(FULL, b, 0);
    if (b + qlen <= P.cap) {
      for (uint32_t i = lane; i < qlen; i += 32) P.vtx[b + i] = W.q[i];
      if (lane == 0) {
        P.set_off[s] = b;
        P.set_len[s] = qlen;
      }
      stored = true;
    } else if (lane == 0) {
      atomicMin(first_bad, b);
    }
  }
  if (clear_bitmap)
    for (uint32_t i = lane; i < qlen; i += 32) W.bm[W.q[i] >> 5] = 0u;
  __syncwarp();
  return stored;
}

__device__ bool finish_set(const WarpCtx &W, uint32_t qlen, bool overflow,
                           uint64_t s, uint32_t rel, const DevPool &P,
                           const FailList &F, bool big = false, bool clear_bitmap = true) {
  const bool stored = store_set(W, qlen, overflow, s, P, F.first_bad_base, clear_bitmap);
  if (!stored && lane_id() == 0) {
    if (big) F.big_end[-1 - (int64_t)atomicAdd(F.big_count, 1u)] = rel;
    else F.ids[atomicAdd(F.count, 1u)] = rel;
  }
  __syncwarp();
  return stored;
}

struct SetOutcome {
  uint32_t qlen;
  bool overflow, big;
  unsigned long long exp, edges;  // per-set work (valid on lane 0 / summed over lanes)
  // IC, summed over lanes: in-edges of uniform-threshold lists (coins drawn,
  // records not read) and live edges of those lists (source id read)
  unsigned long long uedges = 0, usrc = 0;
};

// One IC set: reverse BFS from root(s) over live in-edges, warp-cooperative,
// members in discovery order in W.q.  Sets past `work_cap` in-edges (when
// nonzero) are abandoned with big = true.
template <class RK>
__device__ __forceinline__ SetOutcome ic_plain_set(const DevGraph &G, Key key, const RK &rk,
                                                   uint64_t s, const WarpCtx &W,
                                                   uint64_t work_cap) {
  const uint32_t lane = lane_id();
  const CoinSet cs = coin_set(rk, s, DOM_IC);
  const uint32_t root = root_of(key, s, G.n);
  if (lane == 0) {
    W.q[0] = root;
    atomicOr(&W.bm[root >> 5], 1u << (root & 31));
  }
  __syncwarp();
  uint32_t qlen = 1, head = 0;
  bool overflow = false, big = false;
  unsigned long long set_exp = 0, set_edges = 0, warp_edges = 0;
  uint32_t set_uedges = 0, set_usrc = 0;  // a set's edges are fewer than m < 2^32

  // Appends this lane's newly reached vertex (if any) to the queue,
  // warp-wide in lane order; on queue overflow the set is abandoned and the
  // bits of vertices that will never be queued cleared.
  auto append_one = [&](bool isnew, uint32_t nu) {
    const uint32_t bal = __ballot_sync(FULL, isnew);
    if (bal == 0) return;
    const uint32_t cnt = __popc(bal);
    if (overflow || qlen + cnt > W.qcap) {
      if (isnew) W.bm[nu >> 5] = 0u;
      overflow = true;
      return;
    }
    if (isnew) W.q[qlen + __popc(bal & lanes_below())] = nu;
    qlen += cnt;
  };
  auto block_live = [&](uint32_t b, uint32_t ob, uint32_t oe, uint32_t ovt) -> uint32_t {
    return ic_block_live(G, key, s, b, ob, oe, ovt, coin_block(rk, cs, b));
  };
  // Live edges are few (a block has none or one): following them as they come
  // would run the source read, the bitmap atomic and the append, round trips to
  // L2, for some lanes at a time.  They wait in the warp's buffer and are
  // followed 32 at a time, the last `cnt` of them here: sources new to the set
  // are marked and queued.  (2^14 vertices, p ~ U(0, 0.1): 0.67 -> 0.47 ms a
  // query's launches.)
  uint32_t nev = 0;
  auto follow = [&](uint32_t cnt) {
    __syncwarp();
    nev -= cnt;
    const uint32_t e = lane < cnt ? W.ev[nev + lane] : 0u;
    __syncwarp();
    bool isnew = false;
    uint32_t nu = 0;
    if (lane < cnt) {
      nu = __ldg(&G.edges[e].x);
      const uint32_t bit = 1u << (nu & 31);
      isnew = !(atomicOr(&W.bm[nu >> 5], bit) & bit);
    }
    append_one(isnew, nu);
    __syncwarp();
  };
  // Buffers a lane's live edges: bit h is edge at(h).
  auto take_live = [&](uint32_t live, bool uniform, auto &&at) {
    if (uniform) set_usrc += __popc(live);
    for (uint32_t bal; (bal = __ballot_sync(FULL, live != 0)) != 0;) {
      if (live) {
        W.ev[nev + __popc(bal & lanes_below())] = at((uint32_t)(__ffs(live) - 1));
        live &= live - 1;
      }
      nev += __popc(bal);
      if (nev >= 32) follow(32);
    }
  };

  while (!overflow) {
    if (nev && qlen - head < 32) {  // fill the next step first
      follow(min(nev, 32u));
      continue;
    }
    if (head == qlen) break;
    const uint32_t take = min(32u, qlen - head);
    uint32_t beg = 0, end = 0, nb = 0, vt = 0;
    if (lane < take) {
      const uint32_t v = W.q[head + lane];
      beg = __ldg(G.off + v);
      end = __ldg(G.off + v + 1);
      if (G.vthr) vt = __ldg(G.vthr + v);
      nb = block_count(beg, end);
      set_edges += end - beg;
      if (vt) set_uedges += end - beg;
    }
    set_exp += (lane == 0) ? take : 0;
    {
      const uint32_t all = warp_incl_scan(nb);
      warp_edges += (unsigned long long)__shfl_sync(FULL, all, 31) * 8;
    }
    if (work_cap && warp_edges > work_cap) {
      // too much edge work for one warp: leave the set to a whole CTA
      overflow = big = true;
      break;
    }
    // Long in-lists (hubs) are swept by the whole warp, one list at a time:
    // lane j takes coin blocks j, j + 32, ... of the list, no owner search.
    uint32_t longs = __ballot_sync(FULL, nb >= kLongBlocks);
    while (longs && !overflow) {
      const uint32_t L = __ffs(longs) - 1;
      longs &= longs - 1;
      const uint32_t lb = __shfl_sync(FULL, beg, L), le = __shfl_sync(FULL, end, L);
      const uint32_t lvt = __shfl_sync(FULL, vt, L);
      const uint32_t b_last = (le - 1) >> 3;
      for (uint32_t base = lb >> 3; base <= b_last && !overflow; base += 32) {
        if (lvt == 0) {
          const uint32_t live = tile_live<2>(G, rk, cs, base, lb, le, W.coins,
                                             [&](uint32_t e) { return ic_fine_call(key, e, s); });
          take_live(live, false, [&](uint32_t h) {
            return (base << 3) + 64 * (h >> 1) + 2 * lane + (h & 1);
          });
          continue;
        }
        const uint32_t b = base + lane;
        const uint32_t live = b <= b_last ? block_live(b, lb, le, lvt) : 0u;
        take_live(live, lvt != 0, [&](uint32_t h) { return (b << 3) + h; });
      }
    }
    // The shorter lists share the warp through their concatenated coin
    // blocks: block j belongs to the lane whose scanned range holds it.
    const uint32_t nbs = nb >= kLongBlocks ? 0u : nb;
    const uint32_t incl = warp_incl_scan(nbs);
    const uint32_t total = __shfl_sync(FULL, incl, 31);
    for (uint32_t base = 0; base < total && !overflow; base += 32) {
      const uint32_t j = base + lane;
      const bool valid = j < total;
      const uint32_t owner = warp_find_owner(incl, valid ? j : total - 1);
      const uint32_t ob = __shfl_sync(FULL, beg, owner);
      const uint32_t oe = __shfl_sync(FULL, end, owner);
      const uint32_t oexcl = __shfl_sync(FULL, incl, owner) - __shfl_sync(FULL, nbs, owner);
      const uint32_t ovt = __shfl_sync(FULL, vt, owner);
      const uint32_t b = (ob >> 3) + (j - oexcl);
      const uint32_t live = valid ? block_live(b, ob, oe, ovt) : 0u;
      take_live(live, ovt != 0, [&](uint32_t h) { return (b << 3) + h; });
    }
    head += take;
  }
  return SetOutcome{qlen, overflow, big, set_exp, set_edges, set_uedges, set_usrc};
}

// Revisit filter of a walk: kSeenBits bits per warp in shared memory.
constexpr uint32_t kSeenBits = 2048;
constexpr uint32_t kSeenWords = kSeenBits / 32;
constexpr uint32_t kProbe = 128;  // records a search step reads, four a lane

// One LT set: the single-predecessor walk from root(s) (see lt_walk_kernel).
// A step is a chain of two dependent reads: the vertex's offsets, then up to 128
// of its in-edge records, four a lane (most lists have at most 32: one).  Lists
// of up to 128 edges are read whole.
// A longer one is entered where the threshold would lie if the cumulative
// weights grew evenly: with weights drawn independently they stray from that
// by about sqrt(degree) / 3 edges, so consecutive records decide up to some
// thousand edges and points a few edges apart narrow a longer list to one more
// read; a list that strays further is split evenly in 128.  (A 32-way search
// took two steps past 32 edges, three past 1024, four past 32 768.)
// Revisits: the first 32 members are in registers, one a lane; a longer walk asks
// a bit of a small filter, which costs no memory latency, and scans the rest of
// the walk (the warp's queue) only when it is set.  The next vertex's offsets
// are on their way meanwhile.  (50 000 walks on Erdos-Renyi graphs of degree 16,
// 2^14, 2^18, 2^20, 2^21 vertices: 2.3, 11.2, 36, 70 ms; with every member in the
// filter, read back from the queue 32 at a time: 2.65, 14.7, 53.6, 113.7.)
__device__ __forceinline__ SetOutcome lt_walk_set(const DevGraph &G, Key key, uint64_t s,
                                                  const WarpCtx &W) {
  const uint32_t lane = lane_id();
  auto seen_hash = [](uint32_t v) { return (v * 0x9E3779B1u) >> 21; };  // 11 bits
  uint32_t cur = root_of(key, s, G.n);
  uint32_t member = lane == 0 ? cur : 0xFFFFFFFFu;  // lane j: the walk's vertex j
  if (lane == 0) W.q[0] = cur;
  uint32_t qlen = 1;
  bool overflow = false;
  uint32_t steps = 0, reads = 0;  // vertices expanded, records read
  uint32_t lo = __ldg(G.off + cur), hi = __ldg(G.off + cur + 1);
  for (;;) {
    const uint32_t t = lt_threshold(key, s, cur);
    ++steps;
    uint32_t u = 0;
    // The first of the `many` (at most kProbe) records from e on whose cumulative
    // threshold exceeds t, and its source u; kProbe: none.
    auto first_above = [&](uint32_t e, uint32_t many) -> uint32_t {
      const uint2 *ep = G.edges + e + lane;
      uint2 rec[kProbe / 32];
#pragma unroll
      for (uint32_t i = 0; i < kProbe / 32; ++i) {
        rec[i] = make_uint2(0u, 0u);
        if (i * 32 + lane < many) rec[i] = __ldg(ep + i * 32);
      }
      reads += many;
#pragma unroll
      for (uint32_t i = 0; i < kProbe / 32; ++i) {
        if (i * 32 >= many) break;
        const uint32_t bal = __ballot_sync(FULL, t < rec[i].y);
        if (bal) {
          const uint32_t at = __ffs(bal) - 1;
          u = __shfl_sync(FULL, rec[i].x, at);
          return i * 32 + at;
        }
      }
      return kProbe;
    };
    const uint32_t deg = hi - lo;
    bool found = false;
    if (deg <= 32) {
      uint2 rec = make_uint2(0u, 0u);
      if (lane < deg) rec = __ldg(G.edges + lo + lane);
      reads += deg;
      const uint32_t bal = __ballot_sync(FULL, t < rec.y);
      if (bal) u = __shfl_sync(FULL, rec.x, __ffs(bal) - 1);
      found = bal != 0;
    } else if (deg <= kProbe) {
      found = first_above(lo, deg) != kProbe;
    } else {
      // it is in [a, b)
      uint32_t a = lo, b = hi;
      for (bool guess = true; a < b; guess = false) {
        const uint32_t d = b - a;
        uint32_t start = a, stride = 1;
        if (d > kProbe && guess) {
          // points kept four standard deviations to either side
          if (d > 4096u) stride = 1u + (uint32_t)(sqrtf((float)d) * (2.5f / kProbe));
          const uint32_t at = __umulhi(t, d), half = stride * (kProbe / 2);
          start = a + min(at > half ? at - half : 0u, d - 1u - stride * (kProbe - 1));
        } else if (d > kProbe) {
          stride = (d + kProbe - 1) / kProbe;
          start = a + stride - 1;
        }
        uint32_t first = kProbe;  // the first point above t
        if (stride == 1) {
          const uint32_t many = min(kProbe, b - start);
          first = first_above(start, many);
          if (first == kProbe) {
            a = start + many;
            continue;
          }
          if (first || start == a) {
            found = true;
            break;
          }
          b = start + 1;
          continue;
        }
        uint32_t thr[kProbe / 32];
#pragma unroll
        for (uint32_t i = 0; i < kProbe / 32; ++i)
          thr[i] = __ldg(&G.edges[start + min((i * 32 + lane) * stride, b - 1 - start)].y);
        reads += kProbe;
#pragma unroll
        for (uint32_t i = 0; i < kProbe / 32; ++i) {
          const uint32_t bal = __ballot_sync(FULL, t < thr[i]);
          if (bal && first == kProbe) first = i * 32 + __ffs(bal) - 1;
        }
        if (first == kProbe) {  // every point at or below t
          a = start + min((kProbe - 1) * stride, b - 1 - start) + 1;
          continue;
        }
        const uint32_t p = start + min(first * stride, b - 1 - start);
        if (first) a = start + (first - 1) * stride + 1;  // first not ruled out
        b = p + 1;
      }
    }
    if (!found) break;  // no in-edge picked: the walk ends here
    lo = __ldg(G.off + u);
    hi = __ldg(G.off + u + 1);
    bool seen = __any_sync(FULL, member == u);
    const uint32_t h = seen_hash(u);
    if (!seen && qlen > 32 && (W.seen[h >> 5] >> (h & 31)) & 1u)
      for (uint32_t k = 32; k < qlen && !seen; k += 128) {
        bool mine = false;
#pragma unroll
        for (uint32_t i = 0; i < 4; ++i) {
          const uint32_t j = k + i * 32 + lane;
          if (j < qlen) mine |= W.q[j] == u;
        }
        seen = __any_sync(FULL, mine);
      }
    if (seen) break;
    if (qlen + 1 > W.qcap) {
      overflow = true;
      break;
    }
    if (qlen < 32) {
      if (lane == qlen) member = u;
    } else {
      __syncwarp();
      if (qlen == 32) {  // the filter holds the vertices from here on
#pragma unroll
        for (uint32_t i = 0; i < kSeenWords; i += 32) W.seen[i + lane] = 0u;
        __syncwarp();
      }
      if (lane == 0) W.seen[h >> 5] |= 1u << (h & 31);
    }
    if (lane == 0) W.q[qlen] = u;
    __syncwarp();
    ++qlen;
    cur = u;
  }
  __syncwarp();
  return SetOutcome{qlen, overflow, false, lane == 0 ? steps : 0u, lane == 0 ? reads : 0u};
}

}  // namespace

// MINB: resident blocks per SM the compiler must allow (4: at most 64
// registers, 32 warps per SM; 5: at most 48 registers, 40 warps per SM -- the
// autotuner picks per graph).
template <int MINB>
__global__ void __launch_bounds__(256, MINB)
ic_plain_kernel(DevGraph G, DevPool P, Key key, const __grid_constant__ RoundKeys rk,
                uint64_t first, uint32_t count,
                const uint32_t *ids, unsigned int *next, uint32_t *bitmaps,
                uint64_t bm_words, uint32_t *queues, uint32_t qcap,
                uint64_t work_cap, FailList F, Stats st) {
  const uint32_t lane = lane_id();
  const uint64_t w = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  __shared__ uint4 s_coin[256];
  __shared__ uint32_t s_ev[8][64];
  WarpCtx W{bitmaps + w * bm_words, queues + w * (uint64_t)qcap, qcap};
  W.coins = s_coin + (threadIdx.x & ~31u);
  W.ev = s_ev[threadIdx.x >> 5];
  unsigned long long n_exp = 0, n_edges = 0, n_sets = 0, n_elems = 0, n_uedges = 0, n_usrc = 0;

  for (;;) {
    uint32_t idx = 0;
    if (lane == 0) idx = atomicAdd(next, 1u);
    idx = __shfl_sync(FULL, idx, 0);
    if (idx >= count) break;
    const uint32_t rel = ids ? ids[idx] : idx;
    const uint64_t s = first + rel;
    const SetOutcome o = ic_plain_set(G, key, rk, s, W, work_cap);
    if (finish_set(W, o.qlen, o.overflow, s, rel, P, F, o.big)) {
      n_sets += (lane == 0);
      n_elems += (lane == 0) ? o.qlen : 0;
      n_exp += o.exp;
      n_edges += o.edges;
      n_uedges += o.uedges;
      n_usrc += o.usrc;
    }
  }
  n_exp = warp_sum_u64(n_exp);
  n_edges = warp_sum_u64(n_edges);
  n_sets = warp_sum_u64(n_sets);
  n_elems = warp_sum_u64(n_elems);
  n_uedges = warp_sum_u64(n_uedges);
  n_usrc = warp_sum_u64(n_usrc);
  if (lane == 0) {
    atomicAdd(st.v + 0, n_exp);
    atomicAdd(st.v + 1, n_edges);
    atomicAdd(st.v + 2, n_sets);
    atomicAdd(st.v + 3, n_elems);
    atomicAdd(st.v + 4, n_exp);
    atomicAdd(st.v + 5, n_edges);
    if (n_uedges) atomicAdd(st.v + 6, n_uedges);
    if (n_usrc) atomicAdd(st.v + 7, n_usrc);
  }
}

// One walk per warp (lt_walk_set).  Walks are chains of dependent loads; a
// launch lasts about as long as its longest walk, so the host launches 32 warps
// per SM and the free warp slots serve other queries' kernels.  Four blocks an SM
// (63 registers): with five (48, some spilled) small graphs' walks were 8% slower
// (50 000 on 2^12 R-MAT vertices, degree 30: 0.353 against 0.327 ms; twelve
// clients' IMMs the same, 15.3 against 15.6 M sets/s).
__global__ void __launch_bounds__(256, 4)
lt_walk_kernel(DevGraph G, DevPool P, Key key, uint64_t first, uint32_t count,
               const uint32_t *ids, unsigned int *next, uint32_t *bitmaps,
               uint64_t bm_words, uint32_t *queues, uint32_t qcap, FailList F,
               Stats st) {
  const uint32_t lane = lane_id();
  const uint64_t w = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  __shared__ uint32_t s_seen[8][kSeenWords];
  WarpCtx W{bitmaps + w * bm_words, queues + w * (uint64_t)qcap, qcap,
            s_seen[threadIdx.x >> 5]};
  unsigned long long n_exp = 0, n_edges = 0, n_sets = 0, n_elems = 0;

  for (;;) {
    uint32_t idx = 0;
    if (lane == 0) idx = atomicAdd(next, 1u);
    idx = __shfl_sync(FULL, idx, 0);
    if (idx >= count) break;
    const uint32_t rel = ids ? ids[idx] : idx;
    const uint64_t s = first + rel;
    const SetOutcome o = lt_walk_set(G, key, s, W);
    if (finish_set(W, o.qlen, o.overflow, s, rel, P, F, false, false)) {
      n_sets += (lane == 0);
      n_elems += (lane == 0) ? o.qlen : 0;
      n_exp += o.exp;
      n_edges += o.edges;
    }
  }
  n_exp = warp_sum_u64(n_exp);
  n_edges = warp_sum_u64(n_edges);
  n_sets = warp_sum_u64(n_sets);
  n_elems = warp_sum_u64(n_elems);
  if (lane == 0) {
    atomicAdd(st.v + 0, n_exp);
    atomicAdd(st.v + 1, n_edges);
    atomicAdd(st.v + 2, n_sets);
    atomicAdd(st.v + 3, n_elems);
    atomicAdd(st.v + 4, n_exp);
    atomicAdd(st.v + 5, n_edges);
  }
}

// Many IMM instances in one persistent launch: warps pull global work indices
// from one counter; index i belongs to the instance a with
// prefix[a] <= i < prefix[a+1] and is that instance's set first_a + i -
// prefix[a], grown with that instance's graph, model and seed into its pool.
// Four blocks an SM (64 registers, some spilled): the walks and sweeps wait for
// memory, and three blocks of 80 registers took 20.0 ms where four take 19.0
// (twelve queries' rounds as one batch).
__global__ void __launch_bounds__(256, 4)
multi_sample_kernel(MultiLaunch L) {
  const uint32_t lane = lane_id();
  const uint64_t w = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  __shared__ uint32_t s_seen[8][kSeenWords];
  __shared__ uint4 s_coin[256];
  __shared__ uint32_t s_ev[8][64];
  WarpCtx W{L.bitmaps + w * L.bm_words, L.queues + w * (uint64_t)L.qcap, L.qcap,
            s_seen[threadIdx.x >> 5]};
  W.coins = s_coin + (threadIdx.x & ~31u);
  W.ev = s_ev[threadIdx.x >> 5];
  // counters of the instance the warp is on, flushed when it moves on
  uint32_t cur = ~0u;
  unsigned long long n_exp = 0, n_edges = 0, n_sets = 0, n_elems = 0, n_uedges = 0, n_usrc = 0;
  auto flush = [&]() {
    const unsigned long long e = warp_sum_u64(n_exp), d = warp_sum_u64(n_edges);
    const unsigned long long ue = warp_sum_u64(n_uedges), us = warp_sum_u64(n_usrc);
    if (lane == 0 && cur != ~0u && n_sets) {
      unsigned long long *st = L.inst[cur].stats;
      atomicAdd(st + 0, e);
      atomicAdd(st + 1, d);
      atomicAdd(st + 2, n_sets);
      atomicAdd(st + 3, n_elems);
      atomicAdd(st + 4, e);
      atomicAdd(st + 5, d);
      if (ue) atomicAdd(st + 6, ue);
      if (us) atomicAdd(st + 7, us);
    }
    n_exp = n_edges = n_sets = n_elems = n_uedges = n_usrc = 0;
  };
  for (;;) {
    uint32_t idx = 0;
    if (lane == 0) idx = atomicAdd(L.next, 1u);
    idx = __shfl_sync(FULL, idx, 0);
    if (idx >= L.total) break;
    uint32_t a = 0, b = L.n_inst;  // prefix[a] <= idx < prefix[b]
    while (b - a > 1) {
      const uint32_t mid = (a + b) >> 1;
      if (L.prefix[mid] <= idx) a = mid;
      else b = mid;
    }
    if (a != cur) {
      flush();
      cur = a;
    }
    const InstanceDesc &D = L.inst[a];
    const uint32_t rel = idx - L.prefix[a];
    const uint64_t s = D.first + rel;
    const SetOutcome o = D.model == RIP_MODEL_IC ? ic_plain_set(D.G, D.key, KeyRounds{D.key}, s, W, D.work_cap)
                                                 : lt_walk_set(D.G, D.key, s, W);
    if (store_set(W, o.qlen, o.overflow, s, D.P, D.first_bad, D.model == RIP_MODEL_IC)) {
      n_sets += 1;
      n_elems += o.qlen;
      n_exp += o.exp;
      n_edges += o.edges;
      n_uedges += o.uedges;
      n_usrc += o.usrc;
    } else if (lane == 0) {
      const unsigned int f = atomicAdd(L.fail_count, 1u);
      L.fail[2 * f] = a;
      L.fail[2 * f + 1] = o.big ? (rel | FAIL_BIG) : rel;
    }
    __syncwarp();
  }
  flush();
}

void launch_multi_sample(const MultiLaunch &L, cudaStream_t stream) {
  count_launches(1);
  multi_sample_kernel<<<L.blocks, 256, 0, stream>>>(L);
}

void launch_ic_plain(const SampleLaunch &L, cudaStream_t stream) {
  count_launches(1);
  const RoundKeys rk = round_keys(L.key);
  if (L.occupancy == 5)
    ic_plain_kernel<5><<<L.blocks, L.threads, 0, stream>>>(
        L.G, L.P, L.key, rk, L.first, L.count, L.ids, L.next, L.bitmaps, L.bm_words,
        L.queues, L.qcap, L.work_cap, L.F, L.st);
  else
    ic_plain_kernel<4><<<L.blocks, L.threads, 0, stream>>>(
        L.G, L.P, L.key, rk, L.first, L.count, L.ids, L.next, L.bitmaps, L.bm_words,
        L.queues, L.qcap, L.work_cap, L.F, L.st);
}

void launch_lt_walk(const SampleLaunch &L, cudaStream_t stream) {
  count_launches(1);
  lt_walk_kernel<<<L.blocks, L.threads, 0, stream>>>(
      L.G, L.P, L.key, L.first, L.count, L.ids, L.next, L.bitmaps, L.bm_words,
      L.queues, L.qcap, L.F, L.st);
}

}  // namespace rip
