// kernels_bigset.cu -- IC sets with very large edge work, one CTA each.
//
// Under weighted-cascade probabilities on skewed graphs a few RRR sets reach
// many hubs and read millions of in-edge records each (on an R-MAT graph with
// 2^20 vertices 1% of the sets carry ~40% of the edge work).  One warp per set
// (ic_plain_kernel) or one warp per frontier entry (ic_fused_kernel) walks a
// hub's in-list alone, so those sets set the kernel's length.  Here one CTA
// grows one such set, level by level:
//   * every warp takes a share of the level's entries and sweeps their shorter
//     lists alone (a warp scan and a shuffle search over their concatenated
//     8-edge coin blocks: no block-wide scan);
//   * lists of at least kTileBlocks blocks are listed and dealt to all warps in
//     tiles of 32 blocks, round robin across lists;
//   * on a uniform-threshold list a block is only tested against the threshold;
//     the few that hold a live edge or a tie go to a shared list, and after the
//     level's barrier all threads take one each: the chain of coin, source
//     read, bitmap atomic and queue append runs once per level, not inside a
//     sweep.
// Coins are the same (set, edge)-keyed Philox draws as every other sampler.
// What bounds it: the integer-multiply pipe (18 wide multiplies of 4 cycles a
// coin block); the sweep is written to add as little as possible to them.
#include "device.cuh"
#include "launch.h"

namespace rip {

namespace {

// Block shapes: 128, 256, 512 or 1024 threads, kBigCtasPerSm of them
// resident per SM (10, 5, 2 or 1: at most 48, 48, 64 or 64 registers a
// thread), each growing its own set -- more resident CTAs let one set's
// barrier waits overlap another's work; the autotuner picks the shape per
// graph.

constexpr uint32_t kTileBlocks = 128;   // lists of at least this many blocks go in tiles
// The same for lists whose records are read: a full tile (600 heavy sets of a
// 2^14-vertex graph, 512 threads: 2.36 ms with 32, 2.66 with 16, 2.72 with 64,
// 2.74 with 128, 2.80 with a block's records read by its lane).
constexpr uint32_t kTileRecords = 32;
constexpr uint32_t kBigLong = 256;        // long lists a level may list
constexpr uint32_t kBigCandidates = 512;  // blocks a level may defer (the rest run in place)

template <int BIG_THREADS>
__global__ void __launch_bounds__(BIG_THREADS, kBigCtasPerSm(BIG_THREADS))
ic_bigset_kernel(const __grid_constant__ BigLaunch L) {
  constexpr uint32_t WARPS = BIG_THREADS / 32;
  // (48 registers a thread don't hold a tile's records: the spills cost the 2^24
  // weighted-cascade launches 3%, 148 -> 153 ms)
  constexpr bool TILES = BIG_THREADS >= 512;
  __shared__ uint4 s_cand[kBigCandidates];  // block, list begin, list end, threshold
  __shared__ uint32_t s_lbeg[kBigLong], s_lend[kBigLong], s_lvt[kBigLong];
  __shared__ uint4 s_coin[TILES ? BIG_THREADS : 32];  // tile_live's
  __shared__ uint32_t s_ev[WARPS][64];  // live edges on their way to the queue
  __shared__ uint32_t s_ncand[2], s_nlong[2];  // by the level's parity
  __shared__ uint32_t s_idx, s_qlen, s_overflow;
  __shared__ uint32_t s_edges, s_uedges, s_usrc;  // a set's in-edges are fewer than 2^32
  __shared__ unsigned long long s_base;

  const uint32_t tid = threadIdx.x, lane = lane_id(), wid = tid >> 5;
  uint32_t *bm = L.bitmaps + (size_t)blockIdx.x * L.bm_words;
  uint32_t *q = L.queues + (size_t)blockIdx.x * L.qcap;
  unsigned long long n_exp = 0, n_edges = 0, n_sets = 0, n_elems = 0, n_uedges = 0, n_usrc = 0;

  for (;;) {
    if (tid == 0) s_idx = atomicAdd(L.next, 1u);
    __syncthreads();
    const uint32_t idx = s_idx;
    if (idx >= L.count) break;
    const uint32_t rel = L.ids[idx];
    const uint64_t s = L.first + rel;
    if (tid == 0) {
      const uint32_t root = root_of(L.key, s, L.G.n);
      q[0] = root;
      atomicOr(&bm[root >> 5], 1u << (root & 31));
      s_qlen = 1;
      s_overflow = 0;
      s_ncand[0] = s_nlong[0] = 0;
      s_edges = 0;
      s_uedges = 0;
      s_usrc = 0;
    }
    __syncthreads();
    const CoinSet cs = coin_set(L.rk, s, DOM_IC);
    uint32_t my_edges = 0, my_uedges = 0, my_usrc = 0;
    // Source u of a live edge joins the set (and the queue) unless there.
    auto reach = [&](uint32_t u) {
      const uint32_t bit = 1u << (u & 31);
      if (!(atomicOr(&bm[u >> 5], bit) & bit)) {
        const uint32_t pos = atomicAdd(&s_qlen, 1u);
        if (pos < L.qcap) q[pos] = u;
        else s_overflow = 1;
      }
    };
    // The live edges of 8-edge coin block b of the in-list [ob, oe); their
    // sources are read then and reached.
    auto expand_block = [&](uint32_t b, uint32_t ob, uint32_t oe, uint32_t ovt) {
      uint32_t live = ic_block_live(L.G, L.key, s, b, ob, oe, ovt, coin_block(L.rk, cs, b));
      while (live) {
        const uint32_t ed = (b << 3) + (__ffs(live) - 1);
        live &= live - 1;
        if (ovt) ++my_usrc;
        reach(__ldg(&L.G.edges[ed].x));
      }
    };
    // Live edges of read records are followed 32 at a time, through the warp's
    // buffer: the bitmap atomic and the append are round trips to L2 (600 heavy
    // sets of a 2^14-vertex graph: 2.36 -> 1.82 ms).
    uint32_t nev = 0;
    uint32_t *ev = s_ev[wid];
    auto follow = [&](uint32_t cnt) {
      __syncwarp();
      nev -= cnt;
      if (lane < cnt) reach(__ldg(&L.G.edges[ev[nev + lane]].x));
      __syncwarp();
    };
    // Buffers a lane's live edges: bit h is edge at(h); called by the whole warp.
    auto take_live = [&](uint32_t live, auto &&at) {
      for (uint32_t bal; (bal = __ballot_sync(FULL, live != 0)) != 0;) {
        if (live) {
          ev[nev + __popc(bal & lanes_below())] = at((uint32_t)(__ffs(live) - 1));
          live &= live - 1;
        }
        nev += __popc(bal);
        if (nev >= 32) follow(32);
      }
    };
    uint32_t lo = 0, hi = 1, par = 0;
    bool full = false;  // the queue overflowed: every thread reads it between two barriers
    while (lo < hi && !full) {
      // A block of a uniform list that holds a live edge or a tie (or, past
      // the list's end, neither: the deferred pass looks).
      auto defer = [&](uint32_t b, uint32_t ob, uint32_t oe, uint32_t ovt) {
        const uint32_t pos = atomicAdd(&s_ncand[par], 1u);
        if (pos < kBigCandidates) s_cand[pos] = make_uint4(b, ob, oe, ovt);
        else expand_block(b, ob, oe, ovt);
      };
      // 1. Every warp takes a share of the level's entries: it sweeps their
      // shorter lists through their concatenated blocks (block j belongs to
      // the lane whose scanned range holds it) and lists the long ones.
      const uint32_t share = min(32u, (hi - lo + WARPS - 1) / WARPS);
      for (uint32_t cb = lo + wid * share; cb < hi; cb += WARPS * share) {
        const uint32_t e = cb + lane;
        uint32_t beg = 0, end = 0, vt = 0;
        if (lane < share && e < hi) {
          const uint32_t v = q[e];
          beg = __ldg(L.G.off + v);
          end = __ldg(L.G.off + v + 1);
          if (L.G.vthr) vt = __ldg(L.G.vthr + v);
          my_edges += end - beg;
          if (vt) my_uedges += end - beg;
        }
        uint32_t nb = block_count(beg, end);
        if (nb >= (vt || !TILES ? kTileBlocks : kTileRecords)) {
          const uint32_t pos = atomicAdd(&s_nlong[par], 1u);
          if (pos < kBigLong) {
            s_lbeg[pos] = beg;
            s_lend[pos] = end;
            s_lvt[pos] = vt;
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
          const uint32_t ovt = __shfl_sync(FULL, vt, owner);
          const uint32_t b = (ob >> 3) + (j - oexcl);
          const uint32_t live = j < total ? ic_block_live(L.G, L.key, s, b, ob, oe, ovt,
                                                          coin_block(L.rk, cs, b))
                                          : 0u;
          if (ovt) my_usrc += __popc(live);
          take_live(live, [&](uint32_t h) { return (b << 3) + h; });
        }
      }
      __syncthreads();
      // 2. The long lists, dealt to the warps a tile of 32 blocks at a time.
      const uint32_t nlong = min(s_nlong[par], kBigLong);
      uint32_t deal = wid;  // (wid - tiles dealt so far) mod WARPS: this warp's next tile
      for (uint32_t a = 0; a < nlong; ++a) {
        const uint32_t ob = s_lbeg[a], oe = s_lend[a], ovt = s_lvt[a];
        const uint32_t b_last = (oe - 1) >> 3;
        const uint32_t ntiles = ((b_last - (ob >> 3)) >> 5) + 1;
        uint32_t b = (ob >> 3) + (deal & (WARPS - 1)) * 32 + lane;
        const uint32_t b_stop = (ob >> 3) + ntiles * 32;  // first block past the tiles
        deal -= ntiles;
        const uint32_t th = ovt >> 16;
        if (ovt != 0 && th != 0xFFFFu) {
          // (blocks past the list's end draw coins nobody looks at: the
          // deferred pass drops edges outside [ob, oe))
          const uint32_t lim = (th + 1) * 0x10001u;
          for (; b + BIG_THREADS < b_stop; b += 2 * BIG_THREADS) {
            const bool h0 = block_clipped(coin_block(L.rk, cs, b), lim);
            const bool h1 = block_clipped(coin_block(L.rk, cs, b + BIG_THREADS), lim);
            if (h0 || h1) {
              if (h0) defer(b, ob, oe, ovt);
              if (h1) defer(b + BIG_THREADS, ob, oe, ovt);
            }
          }
          if (b < b_stop && block_clipped(coin_block(L.rk, cs, b), lim)) defer(b, ob, oe, ovt);
        } else if (!TILES || ovt != 0) {
          for (; b - lane < b_stop; b += BIG_THREADS) {
            const uint32_t live = b <= b_last ? ic_block_live(L.G, L.key, s, b, ob, oe, ovt,
                                                              coin_block(L.rk, cs, b))
                                              : 0u;
            if (ovt) my_usrc += __popc(live);
            take_live(live, [&](uint32_t h) { return (b << 3) + h; });
          }
        } else {
          for (b -= lane; b < b_stop; b += BIG_THREADS) {
            const uint32_t live = tile_live<4>(
                L.G, L.rk, cs, b, ob, oe, s_coin + (TILES ? wid * 32 : 0),
                [&](uint32_t e) { return ic_fine_call(L.key, e, s); });
            take_live(live, [&](uint32_t h) {
              return (b << 3) + 64 * (h >> 1) + 2 * lane + (h & 1);
            });
          }
        }
      }
      if (nev) follow(nev);
      __syncthreads();
      // 3. The deferred blocks, a thread each.
      const uint32_t ncand = min(s_ncand[par], kBigCandidates);
      if (tid == 0) s_ncand[par ^ 1] = s_nlong[par ^ 1] = 0;
      for (uint32_t i = tid; i < ncand; i += BIG_THREADS) {
        const uint4 c = s_cand[i];
        expand_block(c.x, c.y, c.z, c.w);
      }
      __syncthreads();
      lo = hi;
      hi = min(s_qlen, L.qcap);
      full = s_overflow != 0;
      par ^= 1;
      __syncthreads();
    }
    my_edges = __reduce_add_sync(FULL, my_edges);
    my_uedges = __reduce_add_sync(FULL, my_uedges);
    my_usrc = __reduce_add_sync(FULL, my_usrc);
    if (lane_id() == 0) {
      atomicAdd(&s_edges, my_edges);
      atomicAdd(&s_uedges, my_uedges);
      atomicAdd(&s_usrc, my_usrc);
    }
    const uint32_t qlen = min(s_qlen, L.qcap);
    bool stored = false;
    if (!s_overflow) {
      if (tid == 0) {
        const unsigned long long b = atomicAdd(L.P.cursor, (unsigned long long)qlen);
        if (b + qlen <= L.P.cap) {
          s_base = b;
          L.P.set_off[s] = b;
          L.P.set_len[s] = qlen;
        } else {
          atomicMin(L.F.first_bad_base, b);
          s_base = ~0ull;
        }
      }
      __syncthreads();
      stored = s_base != ~0ull;
      if (stored)
        for (uint32_t i = tid; i < qlen; i += BIG_THREADS) L.P.vtx[s_base + i] = q[i];
    }
    __syncthreads();
    // clear the bitmap: every set bit belongs to a queued vertex -- except on
    // queue overflow, where discovered vertices past the queue also set bits
    if (s_overflow) {
      for (uint64_t w = tid; w < L.bm_words; w += BIG_THREADS) bm[w] = 0u;
    } else {
      for (uint32_t i = tid; i < qlen; i += BIG_THREADS) bm[q[i] >> 5] = 0u;
    }
    if (tid == 0) {
      if (stored) {
        n_sets += 1;
        n_elems += qlen;
        n_exp += qlen;
        n_edges += s_edges;
        n_uedges += s_uedges;
        n_usrc += s_usrc;
      } else {
        L.F.ids[atomicAdd(L.F.count, 1u)] = rel;
      }
    }
    __syncthreads();
  }
  if (tid == 0) {
    atomicAdd(L.st.v + 0, n_exp);
    atomicAdd(L.st.v + 1, n_edges);
    atomicAdd(L.st.v + 2, n_sets);
    atomicAdd(L.st.v + 3, n_elems);
    atomicAdd(L.st.v + 4, n_exp);
    atomicAdd(L.st.v + 5, n_edges);
    if (n_uedges) atomicAdd(L.st.v + 6, n_uedges);
    if (n_usrc) atomicAdd(L.st.v + 7, n_usrc);
  }
}

}  // namespace

void launch_ic_bigset(const BigLaunch &L0, cudaStream_t stream) {
  count_launches(1);
  BigLaunch L = L0;
  L.rk = round_keys(L.key);
  if (L.threads == 128)
    ic_bigset_kernel<128><<<L.blocks, 128, 0, stream>>>(L);
  else if (L.threads == 256)
    ic_bigset_kernel<256><<<L.blocks, 256, 0, stream>>>(L);
  else if (L.threads == 512)
    ic_bigset_kernel<512><<<L.blocks, 512, 0, stream>>>(L);
  else
    ic_bigset_kernel<1024><<<L.blocks, 1024, 0, stream>>>(L);
}

}  // namespace rip
