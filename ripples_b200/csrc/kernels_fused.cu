// kernels_fused.cu -- fused multi-colour reverse BFS for IC sampling (sm_100a).
//
// One CTA grows a batch of W = 64*CW RRR sets (CW = 1, 2, 4 -> 64/128/256
// colours) in a single traversal: every vertex carries a W-bit colour mask, so
// a vertex reached by several sets in the same level reads its in-edge list
// once for all of them.  The reference's GPU sampler does the same colour
// batching (GPUBatchedBFSMultiColorFused, include/ripples/gpu/bfs.h:1338-1680;
// kernels include/ripples/gpu/bfs_kernels.h:442-666) but rescans all n
// vertices every level, syncs the host per level and copies the whole
// n x colour matrix back for a host-side scan after each batch.  Here:
//   * frontiers are sparse: a per-CTA log of (vertex) entries, one level
//     after the other; a vertex enters a level's list once, when its pending
//     mask first gains a colour for that level (per-vertex level flag); the
//     log's first kSharedLog entries are staged in shared memory (most
//     batches never leave it), the rest in the CTA's global log;
//   * levels are separated by __syncthreads only -- no grid sync, no host
//     round trip; CTAs are persistent and pull batches from an atomic counter;
//   * the coin of (set s, edge e) is the same pure function of (seed, s, e)
//     as every sampler's (coarse halves from an 8-edge Philox block, the fine
//     half on a tie), so the sets equal those of the one-set-per-warp kernel
//     and of the CPU restatement bit for bit;
//   * the (8-edge coin block, colour) pairs of a warp's entries are dealt to its
//     lanes (pairs.cuh); an entry of more than kShortPairs pairs is listed and
//     dealt to all warps in tiles after the level's barrier.  What bounds a
//     batch is its chain of dependent reads: with a lane per 4-edge group,
//     looping over its colours, a hub's list was one warp's and lanes waited for
//     the fullest mask (20 011 sets of a 2^14-vertex graph, 128 colours: 10.7
//     ms; with pairs 6.2, with two live edges a lane and the next records in
//     flight and no pilot launch 2.8);
//   * the finished batch is compacted straight into the flat pool: one
//     atomicAdd reserves all W sets, per-colour shared cursors place members,
//     and the same pass clears the colour masks (atomicExch) for the next
//     batch, touching only vertices the batch reached.
// A batch whose frontier log overflows is abandoned; the CTA marks its slot
// dirty and leaves, and the host clears the scratch and re-runs the batch's
// sets with the one-set-per-warp kernel (identical results).
#include "device.cuh"
#include "launch.h"
#include "pairs.cuh"

namespace rip {

namespace {

constexpr uint32_t kSharedLog = 4096;  // frontier-log entries staged in shared memory
constexpr uint32_t kFusedLong = 64;    // long entries a level may list

template <int CW, int FUSED_THREADS>
__global__ void __launch_bounds__(FUSED_THREADS, 1024 / FUSED_THREADS)
ic_fused_kernel(const __grid_constant__ FusedLaunch L) {
  constexpr int W = 64 * CW, FUSED_WARPS = FUSED_THREADS / 32;
  constexpr uint32_t NW = 2 * CW;  // 32-colour words of a vertex
  extern __shared__ uint4 s_dyn[];
  __shared__ uint64_t s_set[W];
  __shared__ uint4 s_cs[W];  // the sets' CoinSets
  __shared__ uint32_t s_lbeg[kFusedLong], s_lend[kFusedLong], s_lmask[kFusedLong * NW];
  __shared__ uint32_t s_nlong[2];  // by the level's parity
  __shared__ unsigned long long s_start[W];
  __shared__ uint32_t s_size[W];
  __shared__ uint32_t s_fill[W];
  __shared__ uint32_t s_batch, s_ncol, s_tail, s_overflow;
  __shared__ uint32_t s_log[kSharedLog];  // log entries [0, kSharedLog)
  __shared__ unsigned long long s_base, s_work;

  const uint32_t tid = threadIdx.x, lane = lane_id(), wid = tid >> 5;
  PairWarp &S = reinterpret_cast<PairWarp *>(s_dyn)[wid];
  const uint32_t slot = blockIdx.x;
  const uint32_t n = L.G.n;
  uint64_t *vis = L.vis + (size_t)slot * n * CW;
  uint64_t *pend = L.pend + (size_t)slot * n * CW;
  uint32_t *pflag = L.pflag + (size_t)slot * n;
  uint32_t *log = L.log + (size_t)slot * L.lcap;
  const uint32_t lcap = L.lcap;
  unsigned long long n_exp = 0, n_edges = 0, n_sexp = 0, n_sedges = 0,
                     n_sets = 0, n_elems = 0;
  // per-batch work, folded into the totals only when the batch is stored
  unsigned long long b_exp = 0, b_edges = 0, b_sexp = 0, b_sedges = 0;

  for (;;) {
    if (tid == 0) {
      s_batch = atomicAdd(L.next, 1u);
      s_tail = 0;
      s_overflow = 0;
      s_work = 0;
      s_nlong[0] = s_nlong[1] = 0;
    }
    __syncthreads();
    const uint32_t b = s_batch;
    if (b >= L.num_batches) break;
    const uint32_t c0 = b * W;
    const uint32_t ncol = min((uint32_t)W, L.count - c0);
    if (tid == 0) s_ncol = ncol;
    for (uint32_t c = tid; c < W; c += FUSED_THREADS) {
      s_size[c] = 0;
      s_fill[c] = 0;
      if (c < ncol) {
        const uint32_t rel = L.order ? L.order[c0 + c] : c0 + c;
        s_set[c] = L.first + rel;
        const CoinSet t = coin_set(L.rk, L.first + rel, DOM_IC);
        s_cs[c] = make_uint4(t.x2, t.x0, t.y2, t.z2);
      }
    }
    __syncthreads();
    // seed the roots: level 1
    for (uint32_t c = tid; c < ncol; c += FUSED_THREADS) {
      const uint32_t r = root_of(L.key, s_set[c], n);
      const uint64_t bit = 1ull << (c & 63);
      atomicOr((unsigned long long *)&vis[(size_t)r * CW + (c >> 6)], bit);
      atomicOr((unsigned long long *)&pend[(size_t)r * CW + (c >> 6)], bit);
      atomicAdd(&s_size[c], 1u);
      if (atomicExch(&pflag[r], 1u) != 1u) {
        const uint32_t pos = atomicAdd(&s_tail, 1u);
        if (pos < lcap) {
          if (pos < kSharedLog) s_log[pos] = r;
          else log[pos] = r;
        }
        else s_overflow = 1;
      }
    }
    __syncthreads();
    b_exp = b_edges = b_sexp = b_sedges = 0;
    uint32_t lvl_start = 0, lvl_end = min(s_tail, lcap), level = 1;
    uint32_t *vis32 = reinterpret_cast<uint32_t *>(vis), *pend32 = reinterpret_cast<uint32_t *>(pend);
    uint32_t nev = 0;  // live edges in the warp's buffer
    bool full = s_overflow != 0;
    __syncthreads();
    while (lvl_start < lvl_end && !full) {
      // Live edges, two {edge, colour} a lane: the source joins the colour's
      // set (and the next level).
      auto handle = [&](const uint2 *ev, const bool *valid) {
        uint32_t u[2] = {0, 0};
        bool push[2] = {false, false};
#pragma unroll
        for (int t = 0; t < 2; ++t)
          if (valid[t]) u[t] = __ldg(&L.G.edges[ev[t].x].x);
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          const uint32_t bit = 1u << (ev[t].y & 31);
          push[t] = valid[t] &&
                    !(atomicOr(vis32 + (size_t)u[t] * NW + (ev[t].y >> 5), bit) & bit);
        }
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          if (!push[t]) continue;
          atomicOr(pend32 + (size_t)u[t] * NW + (ev[t].y >> 5), 1u << (ev[t].y & 31));
          atomicAdd(&s_size[ev[t].y], 1u);
          push[t] = atomicExch(&pflag[u[t]], level + 1) != level + 1;
        }
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          const uint32_t bal = __ballot_sync(FULL, push[t]);
          if (!bal) continue;
          uint32_t pos = 0;
          if (lane == (uint32_t)(__ffs(bal) - 1)) pos = atomicAdd(&s_tail, __popc(bal));
          pos = __shfl_sync(FULL, pos, __ffs(bal) - 1) + __popc(bal & lanes_below());
          if (push[t]) {
            if (pos < lcap) {
              if (pos < kSharedLog) s_log[pos] = u[t];
              else log[pos] = u[t];
            }
            else s_overflow = 1;
          }
        }
      };
      auto sweep = [&](uint32_t npairs) {
        sweep_pairs(S, npairs, nev, L.G, L.key, L.rk, s_cs, s_set, handle);
      };
      // One tile of a long entry whose colours the warp has listed.
      auto sweep_tile = [&](uint32_t beg, uint32_t end, uint32_t b, uint32_t b_end, uint32_t pc) {
        const uint32_t step = window_blocks(pc);
        for (; b < b_end; b += step) sweep(fill_blocks(S, beg, end, b, min(step, b_end - b), pc));
      };
      // ---- expand level `level`: entries log[lvl_start, lvl_end) ----------
      const uint32_t share =
          min(32u, (lvl_end - lvl_start + FUSED_WARPS - 1) / FUSED_WARPS);
      for (uint32_t eb = lvl_start + wid * share; eb < lvl_end; eb += FUSED_WARPS * share) {
        const uint32_t ei = eb + lane;
        uint64_t mask[CW];
        uint32_t beg = 0, end = 0, nb = 0, pc = 0;
#pragma unroll
        for (int w = 0; w < CW; ++w) mask[w] = 0;
        if (lane < share && ei < lvl_end) {
          const uint32_t v = ei < kSharedLog ? s_log[ei] : log[ei];
#pragma unroll
          for (int w = 0; w < CW; ++w) {
            mask[w] = atomicExch((unsigned long long *)&pend[(size_t)v * CW + w], 0ull);
            pc += __popcll(mask[w]);
          }
          if (pc) {
            beg = __ldg(L.G.off + v);
            end = __ldg(L.G.off + v + 1);
            nb = block_count(beg, end);
            b_exp += 1;
            b_edges += end - beg;
            if (L.work_cap) atomicAdd(&s_work, (unsigned long long)(end - beg));
            b_sexp += pc;
            b_sedges += (unsigned long long)pc * (end - beg);
          }
        }
        const bool is_long = pc != 0 && nb > kShortPairs / pc;
        bool alone = false;  // long, and no room in the list
        if (is_long) {
          const uint32_t pos = atomicAdd(&s_nlong[level & 1], 1u);
          alone = pos >= kFusedLong;
          if (!alone) {
            s_lbeg[pos] = beg;
            s_lend[pos] = end;
#pragma unroll
            for (int w = 0; w < CW; ++w) {
              s_lmask[pos * NW + 2 * w] = (uint32_t)mask[w];
              s_lmask[pos * NW + 2 * w + 1] = (uint32_t)(mask[w] >> 32);
            }
          }
        }
        // short entries: those that start in the same kShortPairs of the
        // running sum share a window
        const uint32_t pairs = is_long ? 0u : nb * pc;
        const uint32_t incl = warp_incl_scan(pairs);
        const uint32_t total = __shfl_sync(FULL, incl, 31);
        for (uint32_t from = 0; from < total; from += kShortPairs)
          sweep(fill_window<CW>(S, pairs && (incl - pairs) - from < kShortPairs, beg, end, nb, pc,
                                mask));
        for (uint32_t left = __ballot_sync(FULL, alone); left; left &= left - 1) {
          const uint32_t o = __ffs(left) - 1;
          const uint32_t ob = __shfl_sync(FULL, beg, o), oe = __shfl_sync(FULL, end, o);
          const uint32_t opc = __shfl_sync(FULL, pc, o);
          uint32_t word = 0;
#pragma unroll
          for (int w = 0; w < CW; ++w) {
            const uint64_t m = __shfl_sync(FULL, mask[w], o);
            if ((lane >> 1) == (uint32_t)w) word = (uint32_t)(m >> (32 * (lane & 1)));
          }
          fill_colours(S, word);
          sweep_tile(ob, oe, ob >> 3, ((oe - 1) >> 3) + 1, opc);
        }
      }
      __syncthreads();
      // the long entries, a tile to a warp
      const uint32_t nlong = min(s_nlong[level & 1], kFusedLong);
      uint32_t deal = wid;  // (wid - tiles dealt so far) mod FUSED_WARPS: this warp's next tile
      for (uint32_t a = 0; a < nlong; ++a) {
        const uint32_t ob = s_lbeg[a], oe = s_lend[a];
        const uint32_t word = lane < NW ? s_lmask[a * NW + lane] : 0u;
        const uint32_t pc = __reduce_add_sync(FULL, __popc(word));
        const uint32_t tb = tile_blocks(pc), b0 = ob >> 3, nb = ((oe - 1) >> 3) - b0 + 1;
        const uint32_t ntiles = (nb + tb - 1) / tb;
        uint32_t t = deal & (FUSED_WARPS - 1);
        deal -= ntiles;
        if (t >= ntiles) continue;
        fill_colours(S, word);
        for (; t < ntiles; t += FUSED_WARPS)
          sweep_tile(ob, oe, b0 + t * tb, b0 + min(nb, (t + 1) * tb), pc);
      }
      drain_events(S, nev, handle);
      __syncthreads();
      // a batch that outgrows its edge budget goes to the CTA-per-set sampler;
      // every thread reads what ends the loop between two barriers
      const bool over = L.work_cap && s_work > L.work_cap;
      full = s_overflow != 0 || over;
      if (tid == 0) {
        s_nlong[level & 1] = 0;
        if (over && s_overflow == 0) s_overflow = 3;
      }
      lvl_start = lvl_end;
      lvl_end = min(s_tail, lcap);
      ++level;
      __syncthreads();
    }
    if (s_overflow == 1) {
      // Abandon: the scratch may now hold colours of vertices that never
      // reached the log.  Record the batch, mark the slot dirty and stop.
      if (tid == 0) {
        L.F.ids[atomicAdd(L.F.count, 1u)] = b;
        atomicAdd(L.dirty, 1u);
      }
      break;
    }
    // ---- compaction into the pool ----------------------------------------
    if (tid == 0 && s_overflow == 0) {
      unsigned long long tot = 0;
      for (uint32_t c = 0; c < ncol; ++c) tot += s_size[c];
      const unsigned long long base = atomicAdd(L.P.cursor, tot);
      s_base = base;
      if (base + tot > L.P.cap) {
        atomicMin(L.F.first_bad_base, base);
        s_overflow = 2;
      } else {
        unsigned long long run = base;
        for (uint32_t c = 0; c < ncol; ++c) {
          s_start[c] = run;
          run += s_size[c];
        }
      }
    }
    __syncthreads();
    const bool store = s_overflow == 0;
    if (store) {
      n_exp += b_exp;
      n_edges += b_edges;
      n_sexp += b_sexp;
      n_sedges += b_sedges;
      for (uint32_t c = tid; c < ncol; c += FUSED_THREADS) {
        L.P.set_off[s_set[c]] = s_start[c];
        L.P.set_len[s_set[c]] = s_size[c];
      }
    }
    const uint32_t tail = min(s_tail, lcap);
    const bool aborted = s_overflow == 3;  // frontier left unexpanded: clear pend too
    for (uint32_t i = tid; i < tail; i += FUSED_THREADS) {
      const uint32_t v = i < kSharedLog ? s_log[i] : log[i];
#pragma unroll
      for (int w = 0; w < CW; ++w) {
        if (aborted) pend[(size_t)v * CW + w] = 0ull;
        uint64_t mm = atomicExch((unsigned long long *)&vis[(size_t)v * CW + w], 0ull);
        while (mm && store) {
          const int bi = __ffsll((long long)mm) - 1;
          mm &= mm - 1;
          const uint32_t c = w * 64 + bi;
          const uint32_t pos = atomicAdd(&s_fill[c], 1u);
          L.P.vtx[s_start[c] + pos] = v;
        }
      }
      pflag[v] = 0;
    }
    if (tid == 0) {
      if (store) {
        unsigned long long tot = 0;
        for (uint32_t c = 0; c < ncol; ++c) tot += s_size[c];
        n_sets += ncol;
        n_elems += tot;
      } else {
        L.F.ids[atomicAdd(L.F.count, 1u)] = aborted ? (b | FAIL_BIG) : b;
      }
    }
    __syncthreads();
  }
  n_exp = warp_sum_u64(n_exp);
  n_edges = warp_sum_u64(n_edges);
  n_sexp = warp_sum_u64(n_sexp);
  n_sedges = warp_sum_u64(n_sedges);
  if (lane == 0) {
    atomicAdd(L.st.v + 0, n_exp);
    atomicAdd(L.st.v + 1, n_edges);
    atomicAdd(L.st.v + 4, n_sexp);
    atomicAdd(L.st.v + 5, n_sedges);
  }
  if (tid == 0) {
    atomicAdd(L.st.v + 2, n_sets);
    atomicAdd(L.st.v + 3, n_elems);
  }
}

}  // namespace

template <int CW, int THREADS>
static void fused_launch(const FusedLaunch &L, cudaStream_t stream) {
  constexpr size_t shared = THREADS / 32 * sizeof(PairWarp);
  cudaFuncSetAttribute(ic_fused_kernel<CW, THREADS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)shared);
  ic_fused_kernel<CW, THREADS><<<L.blocks, THREADS, shared, stream>>>(L);
}

template <int CW>
static void fused_launch(const FusedLaunch &L, cudaStream_t stream) {
  if (L.blocks <= L.num_sms) fused_launch<CW, 1024>(L, stream);
  else fused_launch<CW, 512>(L, stream);
}

void launch_ic_fused(const FusedLaunch &L0, cudaStream_t stream) {
  count_launches(1);
  FusedLaunch L = L0;
  L.rk = round_keys(L.key);
  if (L.colors == 64) fused_launch<1>(L, stream);
  else if (L.colors == 128) fused_launch<2>(L, stream);
  else fused_launch<4>(L, stream);
}

// ---- export gather: sets [first, first+count) -> out, in set-id order -----
namespace {
__global__ void __launch_bounds__(256)
gather_sets_kernel(DevPool P, uint64_t first, uint64_t count,
                   const uint64_t *csr, uint32_t *out) {
  const uint64_t gw = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  const uint32_t lane = lane_id();
  for (uint64_t i = gw; i < count; i += nw) {
    const uint64_t s = first + i;
    const uint64_t off = P.set_off[s];
    const uint32_t len = P.set_len[s];
    const uint64_t o = csr[i];
    for (uint32_t j = lane; j < len; j += 32) out[o + j] = P.vtx[off + j];
  }
}
}  // namespace

void launch_gather_sets(const DevPool &P, uint64_t first, uint64_t count,
                        const uint64_t *csr, uint32_t *out, cudaStream_t s) {
  count_launches(1);
  if (count == 0) return;
  gather_sets_kernel<<<1184, 256, 0, s>>>(P, first, count, csr, out);
}

}  // namespace rip
