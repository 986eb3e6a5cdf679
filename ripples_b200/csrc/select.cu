// select.cu -- greedy max-coverage seed selection behind include/ripples_b200.h
// (FindMostInfluentialSet, include/ripples/find_most_influential.h:176):
// counts, inverted index, the reference CPU heap (exact, host pops with
// device-fetched counts) and device-only lowest-id picks.
#include "host.h"

// ---------------------------------------------------------------------------
// selection
// ---------------------------------------------------------------------------
namespace {
// Bit-identical to std::make_heap(v.begin(), v.end(), CompareHeap{}), built
// level by level in parallel.  libstdc++'s make_heap runs __adjust_heap on
// every parent from (len-2)/2 down to 0; each call only touches the subtree
// under its parent, and all parents at one depth have disjoint subtrees and
// larger indices than every parent above them, so processing the depths from
// the deepest up -- each depth in any order -- performs the same operations on
// the same data.
void parallel_make_heap(std::vector<HeapItem> &v) {
  const std::ptrdiff_t len = (std::ptrdiff_t)v.size();
  if (len < 2) return;
  const std::ptrdiff_t last_parent = (len - 2) / 2;
  int dmax = 0;
  while ((((std::ptrdiff_t)2) << dmax) - 1 <= last_parent) ++dmax;
  for (int d = dmax; d >= 0; --d) {
    const std::ptrdiff_t lo = (((std::ptrdiff_t)1) << d) - 1;
    const std::ptrdiff_t hi = std::min(last_parent, (((std::ptrdiff_t)2) << d) - 2);
#pragma omp parallel for schedule(static) if (hi - lo > 8192)
    for (std::ptrdiff_t p = hi; p >= lo; --p) {
      HeapItem val = std::move(v[p]);
      std::__adjust_heap(v.begin(), p, len, std::move(val),
                         __gnu_cxx::__ops::_Iter_comp_iter<CompareHeap>(CompareHeap{}));
    }
  }
}
}  // namespace

// Diagnostic: the device heap build against std::make_heap on n random
// {vertex, count} items with counts in [0, max_count); 1 when identical.
extern "C" int rip_selftest_heap_device(rip_ctx *c, uint64_t n, uint32_t max_count,
                                        uint64_t seed) {
  if (!c || n == 0 || n >= 0xFFFFFFFFull) return RIP_ERR_INVALID;
  std::vector<uint32_t> cnt(n);
  uint64_t x = seed * 6364136223846793005ull + 1442695040888963407ull;
  for (uint64_t i = 0; i < n; ++i) {
    x = x * 6364136223846793005ull + 1442695040888963407ull;
    cnt[i] = (uint32_t)((x >> 33) % (max_count ? max_count : 1));
  }
  std::vector<HeapItem> ref(n), got(n);
  for (uint64_t i = 0; i < n; ++i) ref[i] = {(uint32_t)i, cnt[i]};
  std::make_heap(ref.begin(), ref.end(), CompareHeap{});
  DevMem d_cnt, d_heap;
  bool same = true;
  int rc = dalloc(c, d_cnt, 4 * n);
  if (!rc) rc = dalloc(c, d_heap, 8 * n);
  if (!rc) {
    cudaMemcpyAsync(d_cnt.p, cnt.data(), 4 * n, cudaMemcpyHostToDevice, c->stream);
    // the whole heap, then only the items of K or more in their places
    for (uint32_t K : {0u, 1u, max_count / 2, max_count}) {
      cudaError_t e = launch_make_heap(ptr<uint32_t>(d_cnt), (uint32_t)n, ptr<uint2>(d_heap), K,
                                       c->stream);
      cudaMemcpyAsync(got.data(), d_heap.p, 8 * n, cudaMemcpyDeviceToHost, c->stream);
      if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
      if (e == cudaSuccess) e = cudaGetLastError();
      if (e != cudaSuccess) {
        rc = set_err(c, RIP_ERR_CUDA, "heap selftest: %s", cudaGetErrorString(e));
        break;
      }
      for (uint64_t i = 0; i < n && same; ++i)
        same = (got[i].second >= K) == (ref[i].second >= K) &&
               (ref[i].second < K || got[i] == ref[i]);
    }
  }
  dfree(c, d_cnt);
  dfree(c, d_heap);
  if (rc) return rc;
  return same ? 1 : 0;
}

// Diagnostic: checks parallel_make_heap against std::make_heap on n random
// counts drawn from [0, max_count) (many ties); returns 1 when identical.
extern "C" int rip_selftest_heap(uint64_t n, uint32_t max_count, uint64_t seed) {
  std::vector<HeapItem> a(n), b;
  uint64_t x = seed * 6364136223846793005ull + 1442695040888963407ull;
  for (uint64_t i = 0; i < n; ++i) {
    x = x * 6364136223846793005ull + 1442695040888963407ull;
    a[i] = {(uint32_t)i, (uint32_t)((x >> 33) % (max_count ? max_count : 1))};
  }
  b = a;
  std::make_heap(b.begin(), b.end(), CompareHeap{});
  parallel_make_heap(a);
  if (!(a == b)) return 0;
  // pops and pushes on the items of K or more (0: the full heap) against the full
  // heap's
  for (uint32_t K : {0u, 1u, max_count / 2 + 1}) {
    std::vector<uint32_t> vtx, key, pos;
    std::vector<HeapItem> all = b;
    SparseHeap h;
    if (K == 0) {
      h.adopt(all.data(), n);
      for (uint64_t i = 0; i < n; ++i) vtx.push_back((uint32_t)i);
    } else {
      for (uint64_t i = 0; i < n; ++i)
        if (b[i].second >= K) {
          vtx.push_back(b[i].first);
          key.push_back(b[i].second);
          pos.push_back((uint32_t)i);
        }
      h.build(n, (uint32_t)vtx.size(), key.data(), pos.data());
    }
    a = b;
    for (int op = 0; op < 2000 && !a.empty(); ++op) {
      const HeapItem top = a.front();
      if (h.top_kept() != (top.second >= K)) return 0;
      if (top.second < K) break;
      const uint32_t id = h.top_id();
      if (vtx[id] != top.first || h.top_key() != top.second) return 0;
      std::pop_heap(a.begin(), a.end(), CompareHeap{});
      a.pop_back();
      h.pop();
      x = x * 6364136223846793005ull + 1442695040888963407ull;
      if ((x >> 40) % 5) {  // back with a smaller key
        const uint32_t k2 = (uint32_t)((x >> 33) % ((uint64_t)top.second + 1));
        a.push_back(HeapItem{top.first, k2});
        std::push_heap(a.begin(), a.end(), CompareHeap{});
        h.push(id, k2, k2 >= K);
      }
      if (a.size() != h.size()) return 0;
    }
  }
  return 1;
}

// Diagnostic: what a reference-heap selection keeps of counts with this histogram
// (kCountBuckets words) at first: the smallest count, and how many items that makes.
extern "C" int rip_selftest_keep(const uint32_t *hist, uint32_t *smallest, uint64_t *items) {
  *smallest = keep_from(hist, items);
  return RIP_OK;
}

// The counts left by the last selection still sit in the count buffer; bring
// them to the host before anything overwrites that buffer.
static int settle_last_counts(rip_pool *p) {
  if (!p->have_last_counts || !p->last_counts_on_device) return RIP_OK;
  rip_ctx *c = p->ctx;
  p->last_counts.resize(p->g->n);
  CK(c, cudaMemcpyAsync(p->last_counts.data(), p->count.p, sizeof(uint32_t) * (size_t)p->g->n,
                        cudaMemcpyDeviceToHost, c->stream));
  CK(c, cudaStreamSynchronize(c->stream));
  p->last_counts_on_device = false;
  return RIP_OK;
}

static int count_sets(rip_pool *p, uint64_t S) {
  rip_ctx *c = p->ctx;
  const uint32_t n = p->g->n;
  TRY(settle_last_counts(p));
  p->shard_sets = kNoShard;  // the count buffer no longer holds a shard's counts
  // padded to whole chunks of the device picks (the tail stays zero)
  const size_t chunk = sel_chunk_vertices();
  const size_t padded = ((size_t)n + chunk - 1) / chunk * chunk;
  TRY(dalloc(c, p->count, sizeof(uint32_t) * padded));
  CK(c, cudaMemsetAsync(p->count.p, 0, sizeof(uint32_t) * padded, c->stream));
  launch_count(p->view(), S, ptr<uint32_t>(p->count), c->num_sms * 8, c->stream);
  CK(c, cudaGetLastError());
  return RIP_OK;
}

extern "C" int rip_count(rip_pool *p, uint64_t num_sets, uint32_t *counts) {
  if (!p || !counts || num_sets > p->num_sets) return RIP_ERR_INVALID;
  rip_ctx *c = p->ctx;
  CK(c, cudaSetDevice(c->device));
  TRY(count_sets(p, num_sets));
  CK(c, cudaMemcpyAsync(counts, p->count.p, sizeof(uint32_t) * p->g->n,
                        cudaMemcpyDeviceToHost, c->stream));
  CK(c, cudaStreamSynchronize(c->stream));
  return RIP_OK;
}

// Counts left by the last rip_select (after its last update step).
extern "C" int rip_select_counts(rip_pool *p, uint32_t *counts) {
  if (!p || !counts) return RIP_ERR_INVALID;
  if (!p->have_last_counts)
    return set_err(p->ctx, RIP_ERR_STATE, "no selection has run on this pool");
  TRY(settle_last_counts(p));
  std::memcpy(counts, p->last_counts.data(), sizeof(uint32_t) * p->g->n);
  return RIP_OK;
}

// Counts sets [0, S) into `count`, builds the vertex -> sets index over them
// (inv_off, inv) and clears their covered flags; *P_out = index length.  hist
// (may be null): the counts by bucket, kCountBuckets words.
static int prepare_cover(rip_pool *p, uint64_t S, uint64_t *P_out, uint32_t *hist = nullptr) {
  rip_ctx *c = p->ctx;
  const uint32_t n = p->g->n;
  TRY(count_sets(p, S));
  TRY(dalloc(c, p->inv_off, sizeof(uint64_t) * ((size_t)n + 1)));
  TRY(dalloc(c, p->inv_cur, std::max(sizeof(uint64_t) * ((size_t)n + 1),
                                     sizeof(uint32_t) * kCountBuckets)));
  TRY(dalloc(c, p->scan_sums, sizeof(uint64_t) * scan_block_sums_needed(n)));
  launch_exclusive_scan(ptr<uint32_t>(p->count), ptr<uint64_t>(p->inv_off), n,
                        ptr<uint64_t>(p->scan_sums), c->stream);
  uint64_t P = 0;
  if (hist) {  // (in the cursors' room, before they are set)
    launch_count_hist(ptr<uint32_t>(p->count), n, ptr<uint32_t>(p->inv_cur), c->stream);
    CK(c, cudaMemcpyAsync(hist, p->inv_cur.p, sizeof(uint32_t) * kCountBuckets,
                          cudaMemcpyDeviceToHost, c->stream));
  }
  CK(c, cudaMemcpyAsync(&P, ptr<uint64_t>(p->inv_off) + n, sizeof(uint64_t),
                        cudaMemcpyDeviceToHost, c->stream));
  CK(c, cudaMemcpyAsync(p->inv_cur.p, p->inv_off.p, sizeof(uint64_t) * ((size_t)n + 1),
                        cudaMemcpyDeviceToDevice, c->stream));
  CK(c, cudaStreamSynchronize(c->stream));
  TRY(dalloc(c, p->inv, sizeof(uint32_t) * std::max<uint64_t>(P, 1)));
  launch_build_inverted(p->view(), S, ptr<uint64_t>(p->inv_cur), ptr<uint32_t>(p->inv),
                        c->num_sms * 8, c->stream);
  CK(c, cudaGetLastError());
  TRY(dalloc(c, p->covered, std::max<uint64_t>(S, 1)));
  CK(c, cudaMemsetAsync(p->covered.p, 0, std::max<uint64_t>(S, 1), c->stream));
  *P_out = P;
  return RIP_OK;
}

static CoverLaunch cover_launch(rip_pool *p) {
  CoverLaunch C;
  C.P = p->view();
  C.inv_off = ptr<uint64_t>(p->inv_off);
  C.inv = ptr<uint32_t>(p->inv);
  C.covered = ptr<uint8_t>(p->covered);
  C.count = ptr<uint32_t>(p->count);
  C.blocks = p->ctx->num_sms * 4;
  return C;
}

extern "C" int rip_select(rip_pool *p, uint64_t S, uint32_t k, int tiebreak,
                          uint32_t *seeds, uint64_t *gains, uint32_t *num_seeds,
                          double *f) {
  if (!p || (k && !seeds) || !num_seeds) return RIP_ERR_INVALID;
  rip_ctx *c = p->ctx;
  if (S > p->num_sets)
    return set_err(c, RIP_ERR_INVALID, "rip_select: %llu sets requested, pool has %llu",
                   (unsigned long long)S, (unsigned long long)p->num_sets);
  if (tiebreak != RIP_TIE_REF_HEAP && tiebreak != RIP_TIE_LOWEST_ID)
    return set_err(c, RIP_ERR_INVALID, "rip_select: unknown tie-break %d", tiebreak);
  if (S >= (1ull << 32))
    return set_err(c, RIP_ERR_LIMIT, "rip_select: at most 2^32-1 sets");
  CK(c, cudaSetDevice(c->device));
  const uint32_t n = p->g->n;
  *num_seeds = 0;
  if (f) *f = 0.0;
  CK(c, cudaEventRecord(c->ev0, c->stream));
  const auto t_sel0 = clk::now();
  // 1. histogram, 2. vertex -> sets index
  p->have_last_counts = false;  // superseded by this selection
  uint64_t P = 0;
  uint32_t hist[kCountBuckets];  // counts by size (reference-heap picks)
  TRY(prepare_cover(p, S, &P, tiebreak == RIP_TIE_REF_HEAP ? hist : nullptr));
  CoverLaunch C = cover_launch(p);

  // whole-array count fetches land in the context's page-locked buffer and
  // are read there (no second host copy)
  const uint32_t *hcount = nullptr;
  if (!c->h_cand) c->h_cand = new PinnedMem();
  if (!c->h_count) c->h_count = new PinnedMem();
  // mapped: candidate vertex ids in, their counts out (reference-heap picks)
  constexpr uint32_t CAND_CAP = 1u << 16;
  TRY(c->h_cand->ensure(c, 16 + 2 * sizeof(uint32_t) * (size_t)CAND_CAP, true));
  PinnedMem &h_cand = *c->h_cand, &h_count = *c->h_count;

  uint64_t uncovered = S;
  std::vector<uint32_t> out_seeds;
  std::vector<uint64_t> out_gains;

  p->sel_prof[0] += ms_since(t_sel0);
  p->sel_prof[6] += 1;
  const int max_blocks = c->num_sms * 4;
  unsigned char *hb = static_cast<unsigned char *>(h_cand.p);
  unsigned char *db = static_cast<unsigned char *>(h_cand.dev);
  // One pick: mark v's uncovered sets (`gain` of its inverted list) covered and
  // decrement their members, a warp for some of them at a time, a block for long
  // ones.
  auto cover = [&](uint32_t v, uint64_t gain) -> int {
    C.vertex = v;
    C.blocks = (int)std::min<uint64_t>(max_blocks * 4, std::max<uint64_t>(1, (gain + 7) / 8));
    launch_cover(C, c->stream);
    CK(c, cudaGetLastError());
    return RIP_OK;
  };

  if (tiebreak == RIP_TIE_REF_HEAP) {
    const auto t_h0 = clk::now();
    // InitHeapStorage + std::priority_queue(cmp, std::move(storage)), as the
    // reference builds its heap (streaming_find_most_influential.h:541-544;
    // counting.h:196-206), of which the host takes the items that can decide a
    // pick (sparse_heap.h): those whose count is at least K, up to kKeepFirst of
    // them (at n = 2^24 the whole heap was 128 MB over the bus a selection, 4.2 of
    // 14.5 ms, and every pop sank to a leaf 24 levels down).  If the gains fall
    // below K it takes the whole heap and repeats the pops so far on it, some
    // 16 000.  (Some eight times as many items at a time instead, in four steps,
    // repeated up to a million pops: an IMM on 2^21 Erdos-Renyi vertices, 100 seeds,
    // eps 0.2, 11.5 million pops: 4.2 s; the whole heap from the start, with
    // std::pop_heap: 3.15; so 2.05.)
    constexpr uint32_t kGone = 0xFFFFFFFFu;  // log: the popped item stayed out (a seed)
    SparseHeap &heap = c->heap;
    std::vector<uint32_t> ids;  // vertex by item id (of the full heap: the id itself)
    std::vector<uint32_t> log;  // per pop until then: the key it went back with, or kGone
    std::vector<rip_ctx::Fetched> &fetched = c->fetched;
    uint64_t kept = 0;
    uint32_t K = keep_from(hist, &kept);
    // the kept items come in the index cursors' room (the index is built)
    uint32_t *d_list = ptr<uint32_t>(p->inv_cur);
    if (3 * kept + 1 > 2 * ((uint64_t)n + 1)) K = 0;
    TRY(dalloc(c, p->d_heap, sizeof(uint2) * (size_t)n));
    if (!c->h_list) c->h_list = new PinnedMem();
    auto vertex_of = [&](uint32_t id) { return heap.all() ? id : ids[id]; };
    // The heap of these counts, of which the items of K or more are kept.
    auto build = [&](const uint32_t *d_count) -> int {
      CK(c, launch_make_heap(d_count, n, ptr<uint2>(p->d_heap), K, c->stream));
      const uint32_t R = (uint32_t)kept;
      const size_t words = K ? 3 * (size_t)R : 2 * (size_t)n;
      TRY(c->h_list->ensure(c, sizeof(uint32_t) * words));
      if (K) {
        launch_heap_list(ptr<uint2>(p->d_heap), n, K, R, d_list, d_list + words, c->stream);
        CK(c, cudaGetLastError());
      }
      CK(c, cudaMemcpyAsync(c->h_list->p, K ? (void *)d_list : p->d_heap.p, sizeof(uint32_t) * words,
                            cudaMemcpyDeviceToHost, c->stream));
      CK(c, cudaStreamSynchronize(c->stream));
      const size_t room = K ? R : n;
      if (fetched.size() < room) fetched.resize(room, rip_ctx::Fetched{0, 0});
      if (c->fetch > 0xF0000000u) {  // long before the numbers come round
        std::fill(fetched.begin(), fetched.end(), rip_ctx::Fetched{0, 0});
        c->fetch = 0;
      }
      ++c->fetch;  // (ids of another heap: no count is known)
      if (K) {
        const uint32_t *vtx = static_cast<const uint32_t *>(c->h_list->p);
        ids.assign(vtx, vtx + R);
        heap.build(n, R, vtx + R, vtx + 2 * (size_t)R);
      } else {
        heap.adopt(static_cast<HeapItem *>(c->h_list->p), n);
      }
      for (uint32_t key : log) {
        const uint32_t id = heap.top_id();
        heap.pop();
        if (key != kGone) heap.push(id, key, key >= K);
      }
      return RIP_OK;
    };
    TRY(build(ptr<uint32_t>(p->count)));
    p->sel_prof[1] += ms_since(t_h0);
    const auto t_p0 = clk::now();
    // The lazy pops of a pick only read the current counts of heap items keyed
    // at least the pick's gain m (keys are stale upper bounds of the counts and
    // m is the largest count).  After each cover the host fetches the counts
    // of the items keyed >= T for a guess T below the previous gain; if one of
    // them still counts >= T, then m >= T and the fetch covers every item the
    // pops can reach.  Otherwise their largest count c is a lower bound of m
    // and a second fetch with T = c is exact.  A pop outside the fetched items
    // (not expected) falls back to the whole count array.
    uint32_t *h_ids = reinterpret_cast<uint32_t *>(hb + 16);
    uint32_t *h_cnt = h_ids + CAND_CAP;
    const uint32_t *d_ids = reinterpret_cast<const uint32_t *>(db + 16);
    uint32_t *d_cnt = reinterpret_cast<uint32_t *>(db + 16) + CAND_CAP;
    std::vector<uint32_t> cand(CAND_CAP);  // the items whose vertices are in h_ids
    std::vector<uint32_t> stack;
    // First pick: every key is still exact.
    bool fresh_all = false, first = true;
    double ratio = 0.9;   // recent gain ratio g_i / g_{i-1}
    double margin = 0.9;  // guess = margin * ratio: lowered when a guess misses
    auto fetch_all = [&]() -> int {
      TRY(h_count.ensure(c, sizeof(uint32_t) * (size_t)n));
      CK(c, cudaMemcpyAsync(h_count.p, p->count.p, sizeof(uint32_t) * (size_t)n,
                            cudaMemcpyDeviceToHost, c->stream));
      CK(c, cudaStreamSynchronize(c->stream));
      hcount = static_cast<const uint32_t *>(h_count.p);
      fresh_all = true;
      p->sel_prof[8] += 1;
      return RIP_OK;
    };
    // The next pick's first candidate fetch rides on the cover: its items are
    // collected before the cover is launched (the heap and the last gain are
    // final once the seed is chosen) and, when few enough, the cover kernel's
    // last block gathers their counts and raises a flag the host polls.
    constexpr uint32_t FUSED_MAX = 2048;  // one block reads the ids over the bus
    TRY(dalloc(c, p->cg_done, sizeof(unsigned int)));
    if (!p->cg_done_zeroed) {
      CK(c, cudaMemsetAsync(p->cg_done.p, 0, sizeof(unsigned int), c->stream));
      p->cg_done_zeroed = true;
    }
    volatile unsigned int *h_flag = reinterpret_cast<volatile unsigned int *>(hb);
    unsigned int *d_flag = reinterpret_cast<unsigned int *>(db);
    bool prefetched = false;  // h_ids / h_cnt hold round 0 of the next pick
    uint32_t pre_T = 0, pre_nc = 0;
    auto first_T = [&](uint64_t g_prev) {
      const double guess = p->cand_fixed ? p->cand_fixed / 100.0 : margin * ratio;
      return (uint32_t)std::max<double>(1.0, std::floor((double)g_prev * guess));
    };
    auto collect = [&](uint32_t T) -> uint32_t {
      const auto t_c0 = clk::now();
      const uint32_t nc = heap.collect(T, CAND_CAP, heap.all() ? nullptr : ids.data(), cand.data(),
                                       h_ids, stack);
      p->sel_prof[10] += ms_since(t_c0);
      return nc;
    };
    // round-0 collect at T (raised once while too many items qualify);
    // returns the count, CAND_CAP + 1 when still too many
    auto collect0 = [&](uint64_t g_prev, uint32_t &T) -> uint32_t {
      for (;;) {
        const uint32_t nc = collect(T);
        if (nc > CAND_CAP && T < g_prev) {
          T = (uint32_t)std::min<uint64_t>(g_prev, (uint64_t)T + (g_prev - T + 1) / 2);
          continue;
        }
        return nc;
      }
    };
    // The counts the next pops can examine, after a cover.
    auto fetch_candidates = [&](uint64_t g_prev) -> int {
      uint32_t T = prefetched ? pre_T : first_T(g_prev);
      for (int round = 0;; ++round) {
        const bool have = round == 0 && prefetched;
        const uint32_t nc = have ? pre_nc : round == 0 ? collect0(g_prev, T) : collect(T);
        p->sel_prof[11] += 1;
        if (nc > CAND_CAP) {
          TRY(fetch_all());
          break;
        }
        if (!have) {
          launch_gather_counts(ptr<uint32_t>(p->count), d_ids, nc, d_cnt, c->stream);
          CK(c, cudaGetLastError());
          CK(c, cudaStreamSynchronize(c->stream));
        }
        p->sel_prof[5] += nc;
        const uint32_t fetch = ++c->fetch;
        uint32_t mc = 0;
        for (uint32_t i = 0; i < nc; ++i) {
          const uint32_t cv = *reinterpret_cast<volatile uint32_t *>(h_cnt + i);
          fetched[cand[i]] = rip_ctx::Fetched{cv, fetch};
          mc = std::max(mc, cv);
        }
        if (mc >= T || T <= 1) {
          if (round == 0) margin = std::min(0.97, margin + 0.01);
          break;
        }
        T = std::max<uint32_t>(mc, 1u);  // mc <= m < T: exact next round
        margin = std::max(0.5, margin - 0.05);
      }
      prefetched = false;
      return RIP_OK;
    };
    // The gains fell below K.  Every item's count at the start is still in the
    // heap array.
    auto keep_all = [&]() -> int {
      K = 0;
      launch_heap_counts(ptr<uint2>(p->d_heap), n, ptr<uint32_t>(p->inv_cur), c->stream);
      TRY(build(ptr<uint32_t>(p->inv_cur)));
      prefetched = false;
      return first || fresh_all ? RIP_OK : fetch_candidates(out_gains.back());
    };
    while (out_seeds.size() < k && uncovered != 0) {
      const auto t_g0 = clk::now();
      if (!first) TRY(fetch_candidates(out_gains.back()));
      p->sel_prof[7] += ms_since(t_g0);
      uint32_t id = 0, gain = 0;
      const auto t_q0 = clk::now();
      for (;;) {  // getNextSeed, streaming_find_most_influential.h:560-571
        if (!heap.top_kept()) {
          if (heap.all()) return set_err(c, RIP_ERR_STATE, "selection heap exhausted");
          TRY(keep_all());
          continue;
        }
        id = heap.top_id();
        const uint32_t key = heap.top_key();
        uint32_t cur = key;
        if (!first) {
          if (!fresh_all && fetched[id].at != c->fetch) TRY(fetch_all());
          cur = fresh_all ? hcount[vertex_of(id)] : fetched[id].count;
        }
        heap.pop();
        p->sel_prof[3] += 1;
        if (key > cur) {
          heap.push(id, cur, cur >= K);
          if (!heap.all()) log.push_back(cur);
          continue;
        }
        if (!heap.all()) log.push_back(kGone);
        gain = key;
        break;
      }
      p->sel_prof[9] += ms_since(t_q0);
      if (!out_gains.empty() && out_gains.back())
        ratio = std::min(1.0, (double)gain / (double)out_gains.back());
      uncovered -= gain;
      out_seeds.push_back(vertex_of(id));
      out_gains.push_back(gain);
      if (out_seeds.size() == k) break;
      const auto t_f0 = clk::now();
      pre_T = first_T(gain);
      pre_nc = collect0(gain, pre_T);
      if (pre_nc <= FUSED_MAX) {
        C.vertex = vertex_of(id);
        C.blocks = (int)std::min<uint64_t>(max_blocks * 4,
                                           std::max<uint64_t>(1, ((uint64_t)gain + 7) / 8));
        // epochs count per context: the mapped buffer is the context's
        const unsigned int epoch = ++c->cg_epoch;
        *h_flag = 0u;  // the buffer's first word may hold anything before this
        launch_cover_gather(C, d_ids, pre_nc, d_cnt, ptr<unsigned int>(p->cg_done), d_flag,
                            epoch, c->stream);
        CK(c, cudaGetLastError());
        // poll the flag; a stream synchronise covers the (unexpected) case of
        // a flag that does not arrive within a second
        const auto t_w0 = clk::now();
        while (*h_flag != epoch) {
          if (ms_since(t_w0) > 1000.0) {
            CK(c, cudaStreamSynchronize(c->stream));
            if (*h_flag != epoch)
              return set_err(c, RIP_ERR_DEVICE, "pick flag not raised after the cover");
            break;
          }
        }
        std::atomic_thread_fence(std::memory_order_acquire);
        prefetched = true;
      } else {
        TRY(cover(vertex_of(id), gain));
      }
      p->sel_prof[7] += ms_since(t_f0);
      fresh_all = first = false;
    }
    p->sel_prof[2] += ms_since(t_p0);
    p->sel_prof[4] += out_seeds.size();
  } else if (k > 0 && S > 0) {
    // Lowest-id picks entirely on the device: k pick launches (cached chunk
    // maxima, lowest id on ties) and k - 1 cover launches, one read-back.
    const uint32_t chunk = sel_chunk_vertices();
    const uint32_t nchunks = (uint32_t)(((uint64_t)n + chunk - 1) / chunk);
    TRY(dalloc(c, p->s_cmax, (size_t)nchunks * 8));
    TRY(dalloc(c, p->s_dirty, (size_t)nchunks));
    TRY(dalloc(c, p->s_best, (size_t)k * 8 + 256));
    TRY(dalloc(c, p->s_desc, sizeof(SelDesc)));
    TRY(p->h_best.ensure(c, (size_t)k * 8));
    SelDesc d{};
    d.P = p->view();
    d.seg_off[0] = ptr<uint64_t>(p->inv_off);
    d.seg_inv[0] = ptr<uint32_t>(p->inv);
    d.seg_first[0] = 0;
    d.nseg = 1;
    d.S = S;
    d.n = n;
    d.nchunks = nchunks;
    d.k = k;
    d.keep_counts = 1;
    d.count = ptr<uint32_t>(p->count);
    d.cmax = ptr<unsigned long long>(p->s_cmax);
    d.dirty = ptr<uint8_t>(p->s_dirty);
    d.covered = ptr<uint8_t>(p->covered);
    d.best = ptr<unsigned long long>(p->s_best);
    d.done_blocks = reinterpret_cast<unsigned int *>(ptr<uint8_t>(p->s_best) + (size_t)k * 8);
    d.acc = reinterpret_cast<unsigned long long *>(ptr<uint8_t>(p->s_best) + (size_t)k * 8 + 64);
    d.total_elems = P;
    CK(c, cudaMemcpyAsync(p->s_desc.p, &d, sizeof(d), cudaMemcpyHostToDevice, c->stream));
    const SelDesc *dd = ptr<SelDesc>(p->s_desc);
    const int pick_blocks = (int)std::max<uint32_t>(1, std::min<uint32_t>((nchunks + 7) / 8,
                                                                          c->num_sms * 4));
    if (sel_loop_fits(nchunks, (double)P)) {
      launch_sel_init(dd, c->num_sms, c->stream);
      launch_sel_loop(dd, c->stream);
      CK(c, cudaGetLastError());
      CK(c, cudaMemcpyAsync(p->h_best.p, p->s_best.p, (size_t)k * 8, cudaMemcpyDeviceToHost,
                            c->stream));
    } else {
      // The pick loop runs as one CUDA graph, captured once per (k, buffers):
      // kernels read everything through the descriptor; the final copy node
      // holds the best / h_best addresses, so moving those drops the graph.
      SelGraph &sg = p->sel_graph;
      if (sg.exec && (sg.k != k || sg.src != p->s_best.p || sg.dst != p->h_best.p ||
                      sg.desc != p->s_desc.p || sg.pick_blocks != pick_blocks)) {
        cudaGraphExecDestroy(sg.exec);
        sg.exec = nullptr;
      }
      if (!sg.exec) {
        const uint64_t before = launch_counter();
        cudaGraph_t graph = nullptr;
        CK(c, cudaStreamBeginCapture(c->stream, cudaStreamCaptureModeThreadLocal));
        launch_sel_init(dd, c->num_sms, c->stream);
        for (uint32_t i = 0; i < k; ++i) {
          launch_sel_pick(dd, i, pick_blocks, c->stream);
          if (i + 1 < k) launch_sel_cover(dd, i, max_blocks, c->stream);
        }
        cudaMemcpyAsync(p->h_best.p, p->s_best.p, (size_t)k * 8, cudaMemcpyDeviceToHost,
                        c->stream);
        const cudaError_t ce = cudaStreamEndCapture(c->stream, &graph);
        sg.nodes = launch_counter() - before;
        uncount_launches(sg.nodes);
        if (ce != cudaSuccess)
          return set_err(c, RIP_ERR_CUDA, "pick graph capture failed: %s", cudaGetErrorString(ce));
        const cudaError_t ie = cudaGraphInstantiate(&sg.exec, graph, 0);
        cudaGraphDestroy(graph);
        if (ie != cudaSuccess) {
          sg.exec = nullptr;
          return set_err(c, RIP_ERR_CUDA, "pick graph instantiate failed: %s",
                         cudaGetErrorString(ie));
        }
        sg.k = k;
        sg.src = p->s_best.p;
        sg.dst = p->h_best.p;
        sg.desc = p->s_desc.p;
        sg.pick_blocks = pick_blocks;
      }
      CK(c, cudaGraphLaunch(sg.exec, c->stream));
      count_launches(sg.nodes);
    }
    CK(c, cudaStreamSynchronize(c->stream));
    const unsigned long long *hb8 = static_cast<const unsigned long long *>(p->h_best.p);
    for (uint32_t i = 0; i < k && uncovered != 0; ++i) {
      const uint64_t cnt = hb8[i] >> 32;
      if (cnt == 0) break;
      uncovered -= cnt;
      out_seeds.push_back(~(uint32_t)(hb8[i] & 0xFFFFFFFFull));
      out_gains.push_back(cnt);
    }
  }
  CK(c, cudaEventRecord(c->ev1, c->stream));
  CK(c, cudaStreamSynchronize(c->stream));
  float sms = 0.f;
  cudaEventElapsedTime(&sms, c->ev0, c->ev1);
  p->select_kernel_ms += sms;
  p->have_last_counts = true;
  p->last_counts_on_device = true;  // read back on demand (rip_select_counts)
  for (size_t i = 0; i < out_seeds.size(); ++i) {
    seeds[i] = out_seeds[i];
    if (gains) gains[i] = out_gains[i];
  }
  *num_seeds = (uint32_t)out_seeds.size();
  if (f) *f = S ? double(S - uncovered) / (double)S : 0.0;
  return RIP_OK;
}

// ---------------------------------------------------------------------------
// sharded selection: one shard's part of a pick over sets split between
// devices or processes (MPI FindMostInfluentialSet,
// include/ripples/mpi/find_most_influential.h:449-690).  The caller sums the
// shards' counts into d_sum once (an all-reduce across ranks), then per pick
// either sums the shards' updated counts again (rip_shard_cover) or applies
// every shard's decrement list to d_sum (rip_shard_cover_list +
// rip_shard_apply).  Picks keep the maximum of each kPickChunk counts of
// d_sum; the next pick on the same array recomputes only the chunks that
// rip_shard_apply calls touched since, and all of them when none ran (the
// array may have been rewritten, or be a new one at the same address).
// ---------------------------------------------------------------------------

static int check_sum_buffer(rip_ctx *c, const void *d, const char *where) {
  if (!d || (reinterpret_cast<uintptr_t>(d) & 15))
    return set_err(c, RIP_ERR_INVALID, "%s: device array missing or not 16-byte aligned", where);
  return RIP_OK;
}

static int shard_state(rip_pool *p, const char *where) {
  if (p->shard_sets == kNoShard)
    return set_err(p->ctx, RIP_ERR_STATE, "%s: no rip_shard_begin on this pool's current counts",
                   where);
  return RIP_OK;
}

extern "C" int rip_shard_begin(rip_pool *p, uint64_t num_sets, uint32_t *d_sum,
                               uint64_t *elements) {
  if (!p) return RIP_ERR_INVALID;
  rip_ctx *c = p->ctx;
  TRY(check_sum_buffer(c, d_sum, "rip_shard_begin"));
  if (num_sets > p->num_sets)
    return set_err(c, RIP_ERR_INVALID, "rip_shard_begin: %llu sets requested, pool has %llu",
                   (unsigned long long)num_sets, (unsigned long long)p->num_sets);
  if (num_sets >= (1ull << 32))
    return set_err(c, RIP_ERR_LIMIT, "rip_shard_begin: at most 2^32-1 sets");
  CK(c, cudaSetDevice(c->device));
  p->have_last_counts = false;
  uint64_t P = 0;
  TRY(prepare_cover(p, num_sets, &P));
  const uint32_t nchunks = (p->g->n + kPickChunk - 1) / kPickChunk;
  TRY(dalloc(c, p->shard_cmax, (size_t)nchunks * 8));
  TRY(dalloc(c, p->shard_dirty, nchunks));
  TRY(dalloc(c, p->shard_meta, 16));
  TRY(p->h_shard_meta.ensure(c, 16));
  p->shard_sets = num_sets;
  p->shard_elems = P;
  p->shard_cache_ok = false;
  CK(c, cudaMemcpyAsync(d_sum, p->count.p, sizeof(uint32_t) * (size_t)p->g->n,
                        cudaMemcpyDeviceToDevice, c->stream));
  CK(c, cudaStreamSynchronize(c->stream));
  if (elements) *elements = P;
  return RIP_OK;
}

extern "C" int rip_shard_pick(rip_pool *p, const uint32_t *d_sum, uint32_t *vertex,
                              uint64_t *gain) {
  if (!p || !vertex || !gain) return RIP_ERR_INVALID;
  rip_ctx *c = p->ctx;
  TRY(check_sum_buffer(c, d_sum, "rip_shard_pick"));
  TRY(shard_state(p, "rip_shard_pick"));
  CK(c, cudaSetDevice(c->device));
  const uint32_t n = p->g->n;
  const uint32_t nchunks = (n + kPickChunk - 1) / kPickChunk;
  if (!p->shard_cache_ok || d_sum != p->shard_sum)
    CK(c, cudaMemsetAsync(p->shard_dirty.p, 1, nchunks, c->stream));
  unsigned long long *meta = ptr<unsigned long long>(p->shard_meta);
  launch_chunk_pick(d_sum, n, ptr<uint8_t>(p->shard_dirty), ptr<unsigned long long>(p->shard_cmax),
                    meta, c->stream);
  CK(c, cudaGetLastError());
  CK(c, cudaMemcpyAsync(p->h_shard_meta.p, meta, 8, cudaMemcpyDeviceToHost, c->stream));
  CK(c, cudaStreamSynchronize(c->stream));
  p->shard_sum = d_sum;
  p->shard_cache_ok = false;  // until a rip_shard_apply on this array
  const unsigned long long key = *static_cast<const unsigned long long *>(p->h_shard_meta.p);
  *vertex = ~(uint32_t)(key & 0xFFFFFFFFull);
  *gain = key >> 32;
  return RIP_OK;
}

static CoverLaunch shard_cover_launch(rip_pool *p, uint32_t vertex, uint64_t gain) {
  CoverLaunch C = cover_launch(p);
  C.vertex = vertex;
  C.blocks = (int)std::min<uint64_t>((uint64_t)p->ctx->num_sms * 16,
                                     std::max<uint64_t>(1, (gain + 7) / 8));
  return C;
}

extern "C" int rip_shard_cover(rip_pool *p, uint32_t vertex, uint64_t gain, uint32_t *d_sum) {
  if (!p) return RIP_ERR_INVALID;
  rip_ctx *c = p->ctx;
  TRY(check_sum_buffer(c, d_sum, "rip_shard_cover"));
  TRY(shard_state(p, "rip_shard_cover"));
  if (vertex >= p->g->n)
    return set_err(c, RIP_ERR_INVALID, "rip_shard_cover: vertex %u out of range", vertex);
  CK(c, cudaSetDevice(c->device));
  launch_cover(shard_cover_launch(p, vertex, gain), c->stream);
  CK(c, cudaGetLastError());
  CK(c, cudaMemcpyAsync(d_sum, p->count.p, sizeof(uint32_t) * (size_t)p->g->n,
                        cudaMemcpyDeviceToDevice, c->stream));
  CK(c, cudaStreamSynchronize(c->stream));
  p->shard_cache_ok = false;  // the caller rewrites d_sum with the new sums
  return RIP_OK;
}

extern "C" int rip_shard_cover_list(rip_pool *p, uint32_t vertex, uint64_t gain,
                                    uint32_t *d_dec, uint64_t capacity, uint64_t *count) {
  if (!p || !count) return RIP_ERR_INVALID;
  rip_ctx *c = p->ctx;
  TRY(shard_state(p, "rip_shard_cover_list"));
  if (vertex >= p->g->n)
    return set_err(c, RIP_ERR_INVALID, "rip_shard_cover_list: vertex %u out of range", vertex);
  if (capacity < p->shard_elems || (p->shard_elems && !d_dec))
    return set_err(c, RIP_ERR_INVALID,
                   "rip_shard_cover_list: capacity %llu below the shard's %llu elements",
                   (unsigned long long)capacity, (unsigned long long)p->shard_elems);
  CK(c, cudaSetDevice(c->device));
  unsigned long long *cursor = ptr<unsigned long long>(p->shard_meta) + 1;
  CK(c, cudaMemsetAsync(cursor, 0, 8, c->stream));
  if (p->shard_elems) {
    launch_cover_list(shard_cover_launch(p, vertex, gain), d_dec, cursor, c->stream);
    CK(c, cudaGetLastError());
  }
  unsigned long long *h = static_cast<unsigned long long *>(p->h_shard_meta.p);
  CK(c, cudaMemcpyAsync(h + 1, cursor, 8, cudaMemcpyDeviceToHost, c->stream));
  CK(c, cudaStreamSynchronize(c->stream));
  *count = h[1];
  return RIP_OK;
}

extern "C" int rip_shard_apply(rip_pool *p, uint32_t *d_sum, const uint32_t *d_dec,
                               uint64_t count) {
  if (!p || (count && !d_dec)) return RIP_ERR_INVALID;
  rip_ctx *c = p->ctx;
  TRY(check_sum_buffer(c, d_sum, "rip_shard_apply"));
  TRY(shard_state(p, "rip_shard_apply"));
  CK(c, cudaSetDevice(c->device));
  // the cached chunk maxima describe d_sum once this apply's chunks are marked
  p->shard_cache_ok = d_sum == p->shard_sum;
  if (count) {
    const int blocks = (int)std::min<uint64_t>((uint64_t)c->num_sms * 8, (count + 255) / 256);
    launch_apply_decrements(d_sum, p->g->n, d_dec, count, ptr<uint8_t>(p->shard_dirty), blocks,
                            c->stream);
    CK(c, cudaGetLastError());
  }
  CK(c, cudaStreamSynchronize(c->stream));
  return RIP_OK;
}
