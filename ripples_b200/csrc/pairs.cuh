// pairs.cuh -- (coin block, set) pairs of a multi-colour level, a lane each.
//
// In a traversal that grows up to 256 sets at once an entry is a vertex with
// the mask of the sets (colours) that reached it; its work is one Philox block
// per 8-edge coin block of its in-list and colour of its mask.  A warp lists
// the colours of a window of entries (up to kPairWindow pairs) and deals the
// pairs to its lanes, colours fastest: neighbouring lanes read the same records
// and every lane has one Philox block to do, however uneven masks and lists
// are.  A live edge is not followed on the spot: some 5% of the edges are live,
// so its reads and atomics would run for a few lanes at a time.  It goes to the
// warp's event buffer, which is handled 64 at a time, two a lane.  The records
// of a lane's next pair are on their way meanwhile.
#pragma once
#include "device.cuh"

namespace rip {

constexpr uint32_t kPairWindow = 1023;  // most pairs of a window
constexpr uint32_t kShortPairs = 512;   // entries with at most these share a window
constexpr uint32_t kPairTile = 16;      // coin blocks of a longer entry's tile, at least

struct PairWarp {        // a warp's shared memory
  uint4 own[33];         // list begin, end, first coin block, packed (below)
  uint2 ev[96];          // live edges: edge, colour
  uint32_t rcp[32];      // floor(2^20 / colours) + 1
  uint8_t list[1024];    // the entries' colours, one entry after the other
};
// packed: first pair (10 bits) | first colour in the list (10) | colours - 1 (8)

// Coin blocks of a tile of an entry with pc colours, and of a window of it.
__device__ __forceinline__ uint32_t window_blocks(uint32_t pc) { return kPairWindow / pc; }
__device__ __forceinline__ uint32_t tile_blocks(uint32_t pc) {
  return max(kPairTile, window_blocks(pc));
}

// The window of the warp's lanes with want (each an entry of nb * pc <=
// kShortPairs pairs, kPairWindow together); returns its pairs.
template <int CW>
__device__ __forceinline__ uint32_t fill_window(PairWarp &S, bool want, uint32_t beg, uint32_t end,
                                                uint32_t nb, uint32_t pc, const uint64_t *mask) {
  const uint32_t bal = __ballot_sync(FULL, want);
  const uint32_t mine = want ? (nb * pc) | (pc << 16) : 0u;  // both prefix sums at once
  const uint32_t incl = warp_incl_scan(mine);
  const uint32_t total = __shfl_sync(FULL, incl, 31) & 0xFFFFu;
  __syncwarp();
  if (want) {
    const uint32_t o = __popc(bal & lanes_below());
    uint32_t at = (incl - mine) >> 16;
    S.own[o] = make_uint4(beg, end, beg >> 3, ((incl - mine) & 0xFFFFu) | (at << 10) | ((pc - 1) << 20));
    S.rcp[o] = (1u << 20) / pc + 1;
#pragma unroll
    for (int w = 0; w < CW; ++w)
      for (uint64_t m = mask[w]; m; m &= m - 1)
        S.list[at++] = (uint8_t)(w * 64 + __ffsll((long long)m) - 1);
  }
  if (lane_id() == 0) S.own[__popc(bal)] = make_uint4(0, 0, 0, total);
  __syncwarp();
  return total;
}

// One entry's colours: lane w < 2 * CW holds the mask's 32-bit word w.
__device__ __forceinline__ void fill_colours(PairWarp &S, uint32_t word) {
  const uint32_t incl = warp_incl_scan(__popc(word));
  __syncwarp();
  uint32_t at = incl - __popc(word);
  for (; word; word &= word - 1) S.list[at++] = (uint8_t)(lane_id() * 32 + __ffs(word) - 1);
  __syncwarp();
}

// A window of that entry: nb coin blocks from b on.
__device__ __forceinline__ uint32_t fill_blocks(PairWarp &S, uint32_t beg, uint32_t end, uint32_t b,
                                                uint32_t nb, uint32_t pc) {
  __syncwarp();
  if (lane_id() == 0) {
    S.own[0] = make_uint4(beg, end, b, (pc - 1) << 20);
    S.own[1] = make_uint4(0, 0, 0, nb * pc);
    S.rcp[0] = (1u << 20) / pc + 1;
  }
  __syncwarp();
  return nb * pc;
}

// The records of coin block b of the list [beg, end): two at a time, none past
// the list's end (the record array ends on a 4-edge boundary).
__device__ __forceinline__ void pair_records(const DevGraph &G, uint32_t b, uint32_t beg,
                                             uint32_t end, uint4 *rec) {
  const uint4 *rp = reinterpret_cast<const uint4 *>(G.edges + ((size_t)b << 3));
#pragma unroll
  for (int h = 0; h < 4; ++h) {
    const uint32_t e = (b << 3) + 2 * h;
    if (e < end && e + 1 >= beg) rec[h] = __ldg(rp + h);
  }
}

// Draws the window's pairs; handle(edges, valid) takes two events {edge,
// colour} a lane and is called by all lanes, 64 events at a time (what is left
// over, nev of them, goes with the next window or drain_events).
template <class Handle>
__device__ __forceinline__ void sweep_pairs(PairWarp &S, uint32_t npairs, uint32_t &nev,
                                            const DevGraph &G, Key key, const RoundKeys &rk,
                                            const uint4 *cs, const uint64_t *set_ids,
                                            Handle &&handle) {
  const uint32_t lane = lane_id();
  uint32_t o = 0, b = 0, c = 0, beg = 0, end = 0;
  uint4 rec[4];
  auto start = [&](uint32_t j) {  // this lane's pair j: its block, colour and records
    if (j >= npairs) {
      end = 0;
      return;
    }
    while ((S.own[o + 1].w & 1023u) <= j) ++o;  // ends: the last is npairs
    const uint4 w = S.own[o];
    const uint32_t loc = j - (w.w & 1023u), pc = (w.w >> 20) + 1;
    // loc < 2^10 and pc <= 2^8: the quotient is exact
    const uint32_t blk = (loc * S.rcp[o]) >> 20;
    c = S.list[((w.w >> 10) & 1023u) + loc - blk * pc];
    b = w.z + blk;
    beg = w.x;
    end = w.y;
    pair_records(G, b, beg, end, rec);
  };
  start(lane);
  for (uint32_t p0 = 0; p0 < npairs; p0 += 32) {
    uint32_t live = 0;
    const uint32_t e0 = b << 3, pc = c;
    if (p0 + lane < npairs) {
      const uint4 k = cs[c];
      const u32x4 coin = coin_block(rk, CoinSet{k.x, k.y, k.z, k.w}, b);
      uint32_t tie = 0;
#pragma unroll
      for (int h = 0; h < 8; ++h) {
        const uint32_t th = (h & 1 ? rec[h >> 1].w : rec[h >> 1].y) >> 16, cc = coarse_of(coin, h);
        if (cc < th) live |= 1u << h;
        else if (cc == th) tie |= 1u << h;
      }
      const uint32_t in = (0xFFu << (beg > e0 ? beg - e0 : 0u)) & (0xFFu >> (end < e0 + 8 ? e0 + 8 - end : 0u));
      live &= in;
      tie &= in;
      while (tie) {  // one edge in 65 536: the fine half decides
        const uint32_t e = e0 + (__ffs(tie) - 1);
        tie &= tie - 1;
        if (ic_fine_call(key, e, set_ids[c]) < (__ldg(&G.edges[e].y) & 0xFFFFu))
          live |= 1u << (e - e0);
      }
    }
    start(p0 + 32 + lane);
    for (;;) {
      const uint32_t bal = __ballot_sync(FULL, live != 0);
      if (!bal) break;
      if (live) {
        S.ev[nev + __popc(bal & lanes_below())] = make_uint2(e0 + __ffs(live) - 1, pc);
        live &= live - 1;
      }
      nev += __popc(bal);
      if (nev >= 64) {
        nev -= 64;
        __syncwarp();
        const uint2 e[2] = {S.ev[nev + lane], S.ev[nev + 32 + lane]};
        const bool valid[2] = {true, true};
        __syncwarp();
        handle(e, valid);
      }
    }
  }
}

template <class Handle>
__device__ __forceinline__ void drain_events(PairWarp &S, uint32_t &nev, Handle &&handle) {
  __syncwarp();
  const uint2 e[2] = {S.ev[lane_id()], S.ev[32 + lane_id()]};
  const bool valid[2] = {lane_id() < nev, 32 + lane_id() < nev};
  __syncwarp();
  if (nev) handle(e, valid);
  nev = 0;
}

}  // namespace rip
