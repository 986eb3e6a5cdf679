// kernels_graph.cu -- packs a backward CSR into the sampler's layout.
//
// The reference keeps index u64[n+1], edges u32[m], weights f32[m] as three
// arrays (include/ripples/graph.h:364-1086; device copy in
// src/gpu/gpu_graph.cc:48-84) and compares a fresh uniform01 draw with the
// float weight on every coin flip.  Here the weight is converted once into an
// integer threshold and interleaved with the source id, so one aligned 8-byte
// record serves an edge and the coin test is an integer compare:
//   IC : thr = clamp(floor(w * 2^32), 0, 2^32-1)   live iff coin < thr
//   LT : thr = min(min(sum_{i<=e} W_i, 2^41) >> 8, 2^32-1) over the vertex's
//        in-edges in CSR order, W_i = floor(clamp(w_i, 0, 2) * 2^40): exact
//        64-bit fixed point, so the prefix sum may run in any order (here a
//        warp-parallel scan) and still equal a left-to-right sum bit for bit
// Offsets shrink to u32 (m < 2^32 is required).
#include <atomic>

#include "device.cuh"
#include "launch.h"

namespace rip {

namespace {

__device__ __forceinline__ uint32_t prob_u32(double p) {
  const double y = p * 4294967296.0;
  if (!(y > 0.0)) return 0u;
  if (y >= 4294967295.0) return 0xFFFFFFFFu;
  return (uint32_t)floor(y);
}

__global__ void pack_off_kernel(const uint64_t *index, uint32_t n,
                                uint32_t *off) {
  for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v <= n;
       v += (uint64_t)gridDim.x * blockDim.x)
    off[v] = (uint32_t)index[v];
}

__global__ void pack_ic_kernel(const uint32_t *src, const float *w, uint64_t m,
                               uint64_t m_pad, uint2 *edges) {
  for (uint64_t e = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; e < m_pad;
       e += (uint64_t)gridDim.x * blockDim.x)
    edges[e] = e < m ? make_uint2(src[e], prob_u32((double)w[e]))
                     : make_uint2(0u, 0u);
}

__device__ __forceinline__ uint64_t lt_fixed(float w) {
  const double x = (double)w;
  if (!(x > 0.0)) return 0ull;
  if (x >= 2.0) return 2ull << 40;
  return (uint64_t)floor(x * 1099511627776.0);  // exact: w has a 24-bit mantissa
}

__device__ __forceinline__ uint64_t sat_add(uint64_t a, uint64_t b) {
  const uint64_t s = a + b;  // a, b <= 2^41: no wrap
  return s > (1ull << 41) ? (1ull << 41) : s;
}

__device__ __forceinline__ uint2 lt_record(uint32_t src, uint64_t sum) {
  const uint64_t c = sum >> 8;
  return make_uint2(src, c > 0xFFFFFFFFull ? 0xFFFFFFFFu : (uint32_t)c);
}

// In-lists of at least this many edges are scanned by their whole block.
constexpr uint32_t kPackLong = 1024;

// A warp takes 32 consecutive vertices, whose edges lie side by side: 32 edges
// a step, a saturating scan by shuffles that starts anew at every list's first
// edge.  Long lists are listed (*nlong, longs) for pack_lt_long_kernel.  One
// kernel that left a hub to its warp took 1.43 ms of the upload of an R-MAT graph
// with 2^18 vertices and 4 M edges (lists of 30 000, a dependent chain of 32-edge
// steps; hubs sit side by side); the two take 0.67 ms.
__global__ void __launch_bounds__(256)
pack_lt_kernel(const uint64_t *index, const uint32_t *src, const float *w, uint32_t n, uint64_t m,
               uint64_t m_pad, uint2 *edges, unsigned int *nlong, uint32_t *longs_out) {
  const uint32_t lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
  for (uint64_t v0 = (uint64_t)blockIdx.x * 256; v0 < n; v0 += (uint64_t)gridDim.x * 256) {
    const uint64_t v = v0 + threadIdx.x;
    uint64_t beg = 0, end = 0;
    if (v < n) {
      beg = index[v];
      end = index[v + 1];
    }
    const bool lng = end - beg >= kPackLong;
    if (lng) longs_out[atomicAdd(nlong, 1u)] = (uint32_t)v;
    // the warp's range, in steps of 32 edges between its long lists
    const uint64_t wv = v0 + wid * 32;
    const uint64_t first = __shfl_sync(0xFFFFFFFFu, beg, 0);
    const uint64_t last = wv < n ? __shfl_sync(0xFFFFFFFFu, end, (uint32_t)min((uint64_t)31, n - 1 - wv))
                                 : first;
    const uint32_t longs = __ballot_sync(0xFFFFFFFFu, lng);
    uint64_t carry = 0;
    for (uint64_t base = first; base < last;) {
      uint64_t stop = base + 32 < last ? base + 32 : last;
      bool skip = false;
      for (uint32_t l = longs; l; l &= l - 1) {  // (few warps have one)
        const uint64_t hb = __shfl_sync(0xFFFFFFFFu, beg, __ffs(l) - 1);
        const uint64_t he = __shfl_sync(0xFFFFFFFFu, end, __ffs(l) - 1);
        if (base >= hb && base < he) {
          base = he;
          skip = true;
          break;
        }
        if (hb > base && hb < stop) stop = hb;
      }
      if (skip) continue;
      const uint64_t e = base + lane;
      // bit i: edge base + i is the first of its list
      uint32_t head = 0;
      if (end > beg && beg >= base && beg < stop) head = 1u << (uint32_t)(beg - base);
      head = __reduce_or_sync(0xFFFFFFFFu, head);
      uint64_t x = e < stop ? lt_fixed(w[e]) : 0ull;
      // lanes back to this edge's list's first edge (or the step's)
      const uint32_t upto = head & (0xFFFFFFFFu >> (31 - lane));
      const uint32_t from = upto ? 31u - __clz(upto) : 0u;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const uint64_t y = __shfl_up_sync(0xFFFFFFFFu, x, d);
        if (lane >= from + (uint32_t)d) x = sat_add(x, y);
      }
      if (!upto) x = sat_add(x, carry);  // the list began in an earlier step
      if (e < stop) edges[e] = lt_record(src[e], x);
      carry = __shfl_sync(0xFFFFFFFFu, x, (uint32_t)(stop - base - 1));
      base = stop;
    }
  }
  const uint64_t tid = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t e = m + tid; e < m_pad; e += stride) edges[e] = make_uint2(0u, 0u);
}

// The long lists, a block each, 1024 edges a step.
__global__ void __launch_bounds__(256)
pack_lt_long_kernel(const uint64_t *index, const uint32_t *src, const float *w, uint2 *edges,
                    const unsigned int *nlong, const uint32_t *longs) {
  __shared__ uint64_t s_warp[8], s_carry;
  const uint32_t lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
  for (uint32_t k = blockIdx.x; k < *nlong; k += gridDim.x) {
    const uint64_t kb = index[longs[k]], ke = index[longs[k] + 1];
    if (threadIdx.x == 0) s_carry = 0;
    for (uint64_t base = kb; base < ke; base += 1024) {
      // four edges a thread, side by side
      const uint64_t e0 = base + 4 * threadIdx.x;
      uint64_t x[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        x[i] = e0 + i < ke ? lt_fixed(w[e0 + i]) : 0ull;
        if (i) x[i] = sat_add(x[i], x[i - 1]);
      }
      uint64_t t = x[3];
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const uint64_t y = __shfl_up_sync(0xFFFFFFFFu, t, d);
        if (lane >= (uint32_t)d) t = sat_add(t, y);
      }
      if (lane == 31) s_warp[wid] = t;
      __syncthreads();
      uint64_t before = s_carry;
      for (uint32_t i = 0; i < wid; ++i) before = sat_add(before, s_warp[i]);
      const uint64_t prev = __shfl_up_sync(0xFFFFFFFFu, t, 1);
      if (lane) before = sat_add(before, prev);
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (e0 + i < ke) edges[e0 + i] = lt_record(src[e0 + i], sat_add(before, x[i]));
      __syncthreads();
      if (threadIdx.x == 255) s_carry = sat_add(before, x[3]);
      __syncthreads();
    }
  }
}

}  // namespace

static std::atomic<uint64_t> g_launches{0};
uint64_t launch_counter() { return g_launches.load(); }
void count_launches(uint64_t n) { g_launches.fetch_add(n); }
void uncount_launches(uint64_t n) { g_launches.fetch_sub(n); }

static uint64_t pad4(uint64_t m) { return (m + 3) & ~uint64_t(3); }

void launch_pack_ic(const uint64_t *index, const float *w, uint32_t n,
                    uint64_t m, uint32_t *off, uint2 *edges, const uint32_t *src,
                    cudaStream_t stream) {
  count_launches(2);
  pack_off_kernel<<<1184, 256, 0, stream>>>(index, n, off);
  pack_ic_kernel<<<2368, 256, 0, stream>>>(src, w, m, pad4(m) + 4, edges);
}

// *bad = entries with index[v + 1] < index[v] plus sources >= n
__global__ void validate_csr_kernel(const uint64_t *index, const uint32_t *src, uint32_t n,
                                    uint64_t m, unsigned long long *bad) {
  const uint64_t tid = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  unsigned long long b = 0;
  for (uint64_t v = tid; v < n; v += stride) b += index[v + 1] < index[v];
  for (uint64_t e = tid; e < m; e += stride) b += src[e] >= n;
  for (int d = 16; d > 0; d >>= 1) b += __shfl_xor_sync(0xFFFFFFFFu, b, d);
  if ((threadIdx.x & 31u) == 0 && b) atomicAdd(bad, b);
}

void launch_validate_csr(const uint64_t *index, const uint32_t *src, uint32_t n, uint64_t m,
                         unsigned long long *bad, cudaStream_t stream) {
  count_launches(1);
  cudaMemsetAsync(bad, 0, sizeof(*bad), stream);
  validate_csr_kernel<<<2368, 256, 0, stream>>>(index, src, n, m, bad);
}

// vthr[v] = the threshold every in-edge of v shares, else 0; lam[v] = the
// expected number of live in-edges of v (sum of its thresholds / 2^32).  One
// warp per vertex.  sums[0] += in-degrees of the uniform vertices with at
// least two in-edges (the edge reads the IC samplers can skip).
__global__ void uniform_threshold_kernel(const uint32_t *off, const uint2 *edges, uint32_t n,
                                         uint32_t *vthr, float *lam, unsigned long long *sums) {
  const uint32_t lane = threadIdx.x & 31u;
  const uint64_t warp = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  const uint64_t warps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  unsigned long long cov = 0;
  for (uint64_t v = warp; v < n; v += warps) {
    const uint32_t beg = off[v], end = off[v + 1];
    const uint32_t t = end > beg ? edges[beg].y : 0u;
    bool same = true;
    unsigned long long tsum = 0;
    for (uint32_t e = beg + lane; e < end; e += 32) {
      const uint32_t x = edges[e].y;
      same = same && x == t;
      tsum += x;
    }
    same = __all_sync(0xFFFFFFFFu, same);
    for (int d = 16; d > 0; d >>= 1) tsum += __shfl_xor_sync(0xFFFFFFFFu, tsum, d);
    if (lane == 0) {
      vthr[v] = same ? t : 0u;
      lam[v] = (float)((double)tsum * (1.0 / 4294967296.0));
      if (same && t && end - beg >= 2) cov += end - beg;
    }
  }
  if (lane == 0 && cov) atomicAdd(sums, cov);
}

// *total (a double) += lam[source] over every edge: divided by m it is the
// branching factor of a reverse BFS (the expected live in-edges of the vertex
// an edge leads to).
__global__ void branching_kernel(const uint2 *edges, uint64_t m, const float *lam,
                                 double *total) {
  const uint64_t tid = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  double acc = 0.0;
  for (uint64_t e = tid; e < m; e += stride) acc += (double)lam[edges[e].x];
  for (int d = 16; d > 0; d >>= 1) acc += __shfl_xor_sync(0xFFFFFFFFu, acc, d);
  if ((threadIdx.x & 31u) == 0 && acc != 0.0) atomicAdd(total, acc);
}

void launch_uniform_threshold(const uint32_t *off, const uint2 *edges, uint32_t n, uint64_t m,
                              uint32_t *vthr, float *lam, unsigned long long *sums,
                              cudaStream_t stream) {
  count_launches(2);
  cudaMemsetAsync(sums, 0, 2 * sizeof(*sums), stream);
  uniform_threshold_kernel<<<2368, 256, 0, stream>>>(off, edges, n, vthr, lam, sums);
  branching_kernel<<<2368, 256, 0, stream>>>(edges, m, lam, reinterpret_cast<double *>(sums + 1));
}

void launch_pack_lt(const uint64_t *index, const float *w, uint32_t n,
                    uint64_t m, uint32_t *off, uint2 *edges, const uint32_t *src,
                    cudaStream_t stream) {
  count_launches(3);
  // the offsets' room (n + 1 words) holds the long lists' count and ids until they
  // are packed
  unsigned int *nlong = off;
  uint32_t *longs = off + 1;
  cudaMemsetAsync(nlong, 0, sizeof(*nlong), stream);
  pack_lt_kernel<<<2368, 256, 0, stream>>>(index, src, w, n, m, pad4(m) + 4, edges, nlong, longs);
  pack_lt_long_kernel<<<1184, 256, 0, stream>>>(index, src, w, edges, nlong, longs);
  pack_off_kernel<<<1184, 256, 0, stream>>>(index, n, off);
}

}  // namespace rip
