// kernels_giant.cu -- IC sets too large for one warp or one CTA, grown 64*CW
// at a time by the whole GPU.
//
// On graphs where IC is supercritical (R-MAT with p ~ U(0, 0.1) and average
// degree 16: a giant component), a tenth or more of all RRR sets each hold a
// sizeable fraction of the graph and overlap heavily.  A batch of up to 64*CW
// such sets is grown as one multi-colour reverse BFS spread over the whole
// grid: every vertex carries a visited and a pending colour mask, and each
// level runs as
//   prep    : the level's frontier entries take their pending masks (for the
//             colours that reached them last level); a warp's short entries
//             make windows, the (8-edge coin block, colour) pairs of a longer
//             one tiles: one list of work items;
//   expand  : a warp per item, a lane per pair (pairs.cuh); a live edge sets
//             its colour in the source's visited mask and, if it is new there,
//             in its pending mask, and puts the source on the next level's
//             frontier (once per level: a per-vertex level stamp).
// A hub's in-edge list is therefore split over the whole grid, and a vertex
// reached by many sets in the same level is read once for all of them.  When
// the frontier is empty the members are counted per colour, placed in the
// pool (host-reserved range), and the masks cleared -- only for vertices the
// batch touched (a first-touch list).  Coins are the same (set, edge) Philox
// draws as every other sampler, so the sets are bit-identical to theirs.
//
// What bounds expand: issue (58% of the slots busy, 45% of the warps resident);
// a pair is some 350 instructions, 75 of them its coins.  An IMM query (k = 20,
// eps = 0.5) on an R-MAT graph with 2^18 vertices, some 15 of 256 colours a
// vertex and level, expands in 20.9 ms; a thread per block looping over its
// colours took 20.3, but needed a scan of the blocks and an atomic per warp and
// append besides (prep 4.5 ms where the items take 1.06).
#include <algorithm>

#include "device.cuh"
#include "launch.h"
#include "pairs.cuh"

namespace rip {

namespace {

// Appends x (for lanes with want) to list[*tail ...], one atomic per warp.
__device__ __forceinline__ void warp_append(bool want, uint32_t x, uint32_t *list,
                                            unsigned int *tail) {
  const uint32_t bal = __ballot_sync(FULL, want);
  if (!bal) return;
  const uint32_t leader = __ffs(bal) - 1;
  uint32_t base = 0;
  if (lane_id() == leader) base = atomicAdd(tail, (unsigned int)__popc(bal));
  base = __shfl_sync(FULL, base, leader);
  if (want) list[base + __popc(bal & lanes_below())] = x;
}

template <int CW>
__global__ void __launch_bounds__(256) giant_seed_kernel(GiantLaunch L) {
  const uint32_t lane = lane_id();
  for (uint32_t base = blockIdx.x * blockDim.x; base < L.ncol; base += gridDim.x * blockDim.x) {
    const uint32_t c = base + threadIdx.x;
    const bool valid = c < L.ncol;
    uint32_t r = 0, old = 1;
    if (valid) {
      r = root_of(L.key, L.set_ids[c], L.G.n);
      const unsigned long long bit = 1ull << (c & 63);
      atomicOr((unsigned long long *)&L.vis[(size_t)r * CW + (c >> 6)], bit);
      atomicOr((unsigned long long *)&L.pend[(size_t)r * CW + (c >> 6)], bit);
      old = atomicExch(&L.pflag[r], 1u);
    }
    (void)lane;
    warp_append(valid && old == 0u, r, L.touched, L.ctr + 0);
    warp_append(valid && old != 1u, r, L.front, L.ctr + 1);
  }
}

// A work item: {first entry, kWindow | entries - 1} or {entry, first block of
// the list's}: the short entries among them, or a tile of a long one.
constexpr uint32_t kWindow = 0x80000000u;

// A vertex's mask of CW words in one access (a whole 32-byte sector for CW = 4).
template <int CW>
__device__ __forceinline__ void load_mask(const uint64_t *p, uint64_t *m) {
  if constexpr (CW == 4)
    asm volatile("ld.global.v4.u64 {%0, %1, %2, %3}, [%4];"
                 : "=l"(m[0]), "=l"(m[1]), "=l"(m[2]), "=l"(m[3]) : "l"(p) : "memory");
  else if constexpr (CW == 2)
    asm volatile("ld.global.v2.u64 {%0, %1}, [%2];" : "=l"(m[0]), "=l"(m[1]) : "l"(p) : "memory");
  else m[0] = *p;
}
template <int CW>
__device__ __forceinline__ void store_mask(uint64_t *p, const uint64_t *m) {
  if constexpr (CW == 4)
    asm volatile("st.global.v4.u64 [%0], {%1, %2, %3, %4};" ::"l"(p), "l"(m[0]), "l"(m[1]),
                 "l"(m[2]), "l"(m[3]) : "memory");
  else if constexpr (CW == 2)
    asm volatile("st.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(m[0]), "l"(m[1]) : "memory");
  else *p = m[0];
}

// Level prep: entry i of the frontier takes its vertex's pending colours; the
// warp's entries become work items.  Masks move a whole sector at a time and a
// block reserves its items with one atomic: with 8-byte accesses (each a partial
// sector write) and an atomic a warp the launch waited 33 us where it now takes
// 8 (57 000 entries a level on average).
template <int CW>
__global__ void __launch_bounds__(256) giant_prep_kernel(GiantLaunch L, uint32_t nf) {
  __shared__ unsigned long long s_sum[8][4];
  __shared__ uint32_t s_items[8], s_at;
  unsigned long long sum[4] = {0, 0, 0, 0};  // expansions, edges, both per set
  const uint32_t lane = lane_id(), wid = threadIdx.x >> 5;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t base = (uint64_t)blockIdx.x * blockDim.x; base < nf; base += stride) {
    const uint64_t i = base + threadIdx.x;
    uint32_t nt = 0, tb = 1, nb = 0, pc = 0;
    if (i < nf) {
      const uint32_t v = L.front[i];
      const uint32_t beg = __ldg(L.G.off + v), end = __ldg(L.G.off + v + 1);
      uint64_t m[CW], zero[CW];
      load_mask<CW>(L.pend + (size_t)v * CW, m);
#pragma unroll
      for (int w = 0; w < CW; ++w) {
        zero[w] = 0;
        pc += __popcll(m[w]);
      }
      store_mask<CW>(L.pend + (size_t)v * CW, zero);
      store_mask<CW>(L.masks + (size_t)i * CW, m);
      if (pc) {
        nb = block_count(beg, end);
        tb = tile_blocks(pc);
        if (nb > kShortPairs / pc) nt = (nb + tb - 1) / tb;
        sum[0] += 1;
        sum[1] += end - beg;
        sum[2] += pc;
        sum[3] += (unsigned long long)pc * (end - beg);
      }
    }
    // short entries that start in the same kShortPairs of the running sum
    // share a window: its first entry lists it
    const uint32_t pairs = nt ? 0u : nb * pc;
    const uint32_t psum = warp_incl_scan(pairs);
    const uint32_t win = pairs ? (psum - pairs) / kShortPairs : 0xFFFFFFFFu;
    const uint32_t peers = __match_any_sync(FULL, win);
    const bool heads = pairs && lane == (uint32_t)(__ffs(peers) - 1);
    const uint32_t mine = nt + heads;
    const uint32_t incl = warp_incl_scan(mine);
    if (lane == 31) s_items[wid] = incl;
    __syncthreads();
    if (threadIdx.x == 0) {
      uint32_t t = 0;
      for (int w = 0; w < 8; ++w) t += s_items[w];
      s_at = t ? atomicAdd(L.ctr + 2, t) : 0u;
    }
    __syncthreads();
    uint32_t at = s_at + incl - mine;
    for (uint32_t w = 0; w < wid; ++w) at += s_items[w];
    if (heads) L.items[at] = make_uint2((uint32_t)i, kWindow | (31u - __clz(peers) - lane));
    for (uint32_t t = 0; t < nt; ++t) L.items[at + t] = make_uint2((uint32_t)i, t * tb);
    __syncthreads();
  }
  // one atomic per block and counter
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const unsigned long long t = warp_sum_u64(sum[k]);
    if (lane == 0) s_sum[wid][k] = t;
  }
  __syncthreads();
  if (threadIdx.x < 4) {
    unsigned long long t = 0;
    for (int w = 0; w < 8; ++w) t += s_sum[w][threadIdx.x];
    const int slot[4] = {0, 1, 4, 5};
    if (t) atomicAdd(L.stats + slot[threadIdx.x], t);
  }
}

struct OutWarp {  // a warp's entries on their way to the lists
  uint32_t v[2][64];
};

template <int CW>
__global__ void __launch_bounds__(256, 4)
giant_expand_kernel(const __grid_constant__ GiantLaunch L, uint32_t level) {
  constexpr uint32_t NW = 2 * CW;  // 32-colour words of a vertex
  __shared__ uint4 s_cs[64 * CW];
  __shared__ PairWarp s_warp[8];
  __shared__ OutWarp s_out[8];
  __shared__ uint32_t s_nout[2][8], s_base[2];
  for (uint32_t c = threadIdx.x; c < L.ncol; c += blockDim.x) {
    const CoinSet t = coin_set(L.rk, L.set_ids[c], DOM_IC);
    s_cs[c] = make_uint4(t.x2, t.x0, t.y2, t.z2);
  }
  __syncthreads();
  const uint32_t lane = lane_id();
  PairWarp &S = s_warp[threadIdx.x >> 5];
  OutWarp &out = s_out[threadIdx.x >> 5];
  uint32_t *vis = reinterpret_cast<uint32_t *>(L.vis), *pend = reinterpret_cast<uint32_t *>(L.pend);
  const uint32_t *masks = reinterpret_cast<const uint32_t *>(L.masks);
  uint32_t nout[2] = {0, 0};
  // Appends to list k (0 touched, 1 next frontier) by way of the warp's buffer:
  // an atomic on the list's counter per 32 entries.
  auto append = [&](int k, bool want, uint32_t u) {
    const uint32_t bal = __ballot_sync(FULL, want);
    if (!bal) return;
    if (want) out.v[k][nout[k] + __popc(bal & lanes_below())] = u;
    nout[k] += __popc(bal);
    if (nout[k] < 32) return;
    nout[k] -= 32;
    __syncwarp();
    uint32_t base = 0;
    if (lane == 0) base = atomicAdd(L.ctr + k, 32u);
    base = __shfl_sync(FULL, base, 0);
    (k ? L.front_next : L.touched)[base + lane] = out.v[k][nout[k] + lane];
    __syncwarp();
  };
  // Live edges, two {edge, colour} a lane: the source joins the colour's set.
  auto handle = [&](const uint2 *ev, const bool *valid) {
    uint32_t u[2] = {0, 0}, oldf[2] = {level + 1, level + 1};
    bool added[2];
#pragma unroll
    for (int t = 0; t < 2; ++t)
      if (valid[t]) u[t] = __ldg(&L.G.edges[ev[t].x].x);
    // a plain read first: visited bits only get set, so colours it shows need
    // no atomic (most live edges late in a giant BFS)
#pragma unroll
    for (int t = 0; t < 2; ++t)
      added[t] = valid[t] && !(__ldcg(vis + (size_t)u[t] * NW + (ev[t].y >> 5)) >> (ev[t].y & 31) & 1u);
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      const uint32_t bit = 1u << (ev[t].y & 31);
      if (added[t]) added[t] = !(atomicOr(vis + (size_t)u[t] * NW + (ev[t].y >> 5), bit) & bit);
    }
#pragma unroll
    for (int t = 0; t < 2; ++t)
      if (added[t]) {
        atomicOr(pend + (size_t)u[t] * NW + (ev[t].y >> 5), 1u << (ev[t].y & 31));
        oldf[t] = atomicExch(&L.pflag[u[t]], level + 1);
      }
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      append(0, oldf[t] == 0u, u[t]);
      append(1, oldf[t] != level + 1, u[t]);
    }
  };
  uint32_t nev = 0;  // live edges in the warp's buffer
  auto sweep = [&](uint32_t npairs) {
    sweep_pairs(S, npairs, nev, L.G, L.key, L.rk, s_cs, L.set_ids, handle);
  };
  const uint32_t nitems = L.ctr[2];
  const uint32_t nw = gridDim.x * (blockDim.x >> 5);
  for (uint64_t t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); t < nitems; t += nw) {
    const uint2 item = L.items[t];
    if (item.y & kWindow) {
      uint64_t mask[CW];
      uint32_t beg = 0, end = 0, nb = 0, pc = 0;
      const uint32_t i = item.x + lane;
#pragma unroll
      for (int w = 0; w < CW; ++w) mask[w] = 0;
      if (lane <= (item.y & 31u)) {
        const uint32_t v = L.front[i];
        beg = __ldg(L.G.off + v);
        end = __ldg(L.G.off + v + 1);
        nb = block_count(beg, end);
#pragma unroll
        for (int w = 0; w < CW; ++w) {
          mask[w] = L.masks[(size_t)i * CW + w];
          pc += __popcll(mask[w]);
        }
      }
      sweep(fill_window<CW>(S, pc != 0 && nb != 0 && nb <= kShortPairs / pc, beg, end, nb, pc, mask));
    } else {
      const uint32_t v = L.front[item.x];
      const uint32_t beg = __ldg(L.G.off + v), end = __ldg(L.G.off + v + 1);
      const uint32_t word = lane < NW ? masks[(size_t)item.x * NW + lane] : 0u;
      const uint32_t pc = __reduce_add_sync(FULL, __popc(word));
      const uint32_t step = window_blocks(pc);
      uint32_t b = (beg >> 3) + item.y;
      const uint32_t b_end = min(b + tile_blocks(pc), ((end - 1) >> 3) + 1);
      fill_colours(S, word);
      for (; b < b_end; b += step) sweep(fill_blocks(S, beg, end, b, min(step, b_end - b), pc));
    }
  }
  drain_events(S, nev, handle);
  // what is left in the buffers: one atomic a block and list
  const uint32_t wid = threadIdx.x >> 5;
  if (lane == 0) {
    s_nout[0][wid] = nout[0];
    s_nout[1][wid] = nout[1];
  }
  __syncthreads();
  if (threadIdx.x < 2) {
    uint32_t t = 0;
    for (int w = 0; w < 8; ++w) t += s_nout[threadIdx.x][w];
    s_base[threadIdx.x] = t ? atomicAdd(L.ctr + threadIdx.x, t) : 0u;
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    uint32_t at = s_base[k];
    for (uint32_t w = 0; w < wid; ++w) at += s_nout[k][w];
    if (lane < nout[k]) (k ? L.front_next : L.touched)[at + lane] = out.v[k][lane];
  }
}

constexpr uint32_t GIANT_CHUNK = 512;  // touched vertices per block in compaction

// Members per colour (block-local histograms, one global add per colour).
template <int CW>
__global__ void __launch_bounds__(256) giant_sizes_kernel(GiantLaunch L, uint32_t nt) {
  __shared__ uint32_t s_cnt[64 * CW];
  for (uint32_t c = threadIdx.x; c < 64 * CW; c += blockDim.x) s_cnt[c] = 0;
  __syncthreads();
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nt; i += gridDim.x * blockDim.x) {
    const uint32_t v = L.touched[i];
#pragma unroll
    for (int w = 0; w < CW; ++w) {
      uint64_t m = L.vis[(size_t)v * CW + w];
      while (m) {
        const int bi = __ffsll((long long)m) - 1;
        m &= m - 1;
        atomicAdd(&s_cnt[w * 64 + bi], 1u);
      }
    }
  }
  __syncthreads();
  for (uint32_t c = threadIdx.x; c < L.ncol; c += blockDim.x)
    if (s_cnt[c]) atomicAdd(L.sizes + c, s_cnt[c]);
}

// Lane j's result: bit j of every lane's x (a 32 x 32 bit transpose).
__device__ __forceinline__ uint32_t warp_transpose(uint32_t x) {
  constexpr uint32_t keep[5] = {0x0000FFFFu, 0x00FF00FFu, 0x0F0F0F0Fu, 0x33333333u, 0x55555555u};
#pragma unroll
  for (int k = 0; k < 5; ++k) {
    const uint32_t s = 16u >> k, m = keep[k], y = __shfl_xor_sync(FULL, x, s);
    x = lane_id() & s ? (x & ~m) | ((y >> s) & m) : (x & m) | ((y & m) << s);
  }
  return x;
}

// Writes each member into its set's pool range and clears the batch's state.
// A block takes GIANT_CHUNK touched vertices: counts them per colour, reserves a
// slice of every colour's range with one atomic each, then places them;
// positions inside a set are arbitrary (set contents are compared as sets).  A
// warp has 32 vertices' masks, transposed: colour by colour, the lanes of its
// members write side by side.  (A thread that walked its vertex's mask wrote
// each member to a sector of its own: 0.51 ms for 256 sets of 45 000 members,
// 0.07 this way.)
template <int CW>
__global__ void __launch_bounds__(256) giant_scatter_kernel(GiantLaunch L, uint32_t nt) {
  constexpr uint32_t NW = 2 * CW, GROUPS = GIANT_CHUNK / 256;  // groups of 32 a warp
  __shared__ uint32_t s_cnt[64 * CW];
  __shared__ unsigned long long s_at[64 * CW];
  const uint32_t lane = lane_id(), wid = threadIdx.x >> 5;
  for (uint64_t c0 = (uint64_t)blockIdx.x * GIANT_CHUNK; c0 < nt;
       c0 += (uint64_t)gridDim.x * GIANT_CHUNK) {
    for (uint32_t c = threadIdx.x; c < 64 * CW; c += blockDim.x) s_cnt[c] = 0;
    __syncthreads();
    uint32_t v[GROUPS], has[GROUPS][NW], pos[GROUPS][NW];
#pragma unroll
    for (uint32_t g = 0; g < GROUPS; ++g) {
      const uint64_t i = c0 + (wid * GROUPS + g) * 32 + lane;
      uint64_t m[CW], zero[CW];
#pragma unroll
      for (int w = 0; w < CW; ++w) m[w] = zero[w] = 0;
      v[g] = 0;
      if (i < nt) {
        v[g] = L.touched[i];
        load_mask<CW>(L.vis + (size_t)v[g] * CW, m);
        store_mask<CW>(L.vis + (size_t)v[g] * CW, zero);
        L.pflag[v[g]] = 0u;
      }
#pragma unroll
      for (uint32_t w = 0; w < NW; ++w) {
        has[g][w] = warp_transpose((uint32_t)(m[w >> 1] >> (32 * (w & 1))));
        pos[g][w] = has[g][w] ? atomicAdd(&s_cnt[w * 32 + lane], (uint32_t)__popc(has[g][w])) : 0u;
      }
    }
    __syncthreads();
    for (uint32_t c = threadIdx.x; c < L.ncol; c += blockDim.x)
      s_at[c] = s_cnt[c] ? L.starts[c] + atomicAdd(L.fill + c, s_cnt[c]) : 0ull;
    __syncthreads();
#pragma unroll
    for (uint32_t g = 0; g < GROUPS; ++g) {
#pragma unroll
      for (uint32_t w = 0; w < NW; ++w) {
        for (uint32_t left = __ballot_sync(FULL, has[g][w] != 0); left; left &= left - 1) {
          const uint32_t j = __ffs(left) - 1;
          const uint32_t members = __shfl_sync(FULL, has[g][w], j);
          const uint32_t at = __shfl_sync(FULL, pos[g][w], j);
          if (members >> lane & 1u)
            L.P.vtx[s_at[w * 32 + j] + at + __popc(members & lanes_below())] = v[g];
        }
      }
    }
    __syncthreads();
  }
}

// set_off / set_len of the batch's sets (starts computed on the host).
__global__ void giant_meta_kernel(GiantLaunch L) {
  for (uint32_t c = blockIdx.x * blockDim.x + threadIdx.x; c < L.ncol;
       c += gridDim.x * blockDim.x) {
    const uint64_t s = L.set_ids[c];
    L.P.set_off[s] = L.starts[c];
    L.P.set_len[s] = L.sizes[c];
    L.fill[c] = 0;
    atomicAdd(L.stats + 2, 1ull);
    atomicAdd(L.stats + 3, (unsigned long long)L.sizes[c]);
  }
}

}  // namespace

template <int CW>
static void giant_launch(int what, const GiantLaunch &L, uint32_t n_items, uint32_t level,
                         int blocks, cudaStream_t s) {
  count_launches(1);
  switch (what) {
    case 0: giant_seed_kernel<CW><<<1, 256, 0, s>>>(L); break;
    case 1:
      giant_prep_kernel<CW><<<std::min<uint32_t>(blocks, (n_items + 255) / 256), 256, 0, s>>>(
          L, n_items);
      break;
    case 2: giant_expand_kernel<CW><<<blocks, 256, 0, s>>>(L, level); break;
    case 3: giant_sizes_kernel<CW><<<blocks, 256, 0, s>>>(L, n_items); break;
    case 4: giant_scatter_kernel<CW><<<blocks, 256, 0, s>>>(L, n_items); break;
    default: giant_meta_kernel<<<1, 256, 0, s>>>(L); break;
  }
}

void launch_giant(int what, int cw, const GiantLaunch &L0, uint32_t n_items, uint32_t level,
                  int blocks, cudaStream_t s) {
  GiantLaunch L = L0;
  L.rk = round_keys(L.key);
  if (cw == 1) giant_launch<1>(what, L, n_items, level, blocks, s);
  else if (cw == 2) giant_launch<2>(what, L, n_items, level, blocks, s);
  else giant_launch<4>(what, L, n_items, level, blocks, s);
}

}  // namespace rip
