// Mixture-of-experts routing and token movement (sm_100a).
//
//   route        sigmoid scores, stable top-k (ties -> lower expert), gates = top / sum(top)
//   count/scan/place   a stable counting sort of the (token, slot) pairs by expert that gives
//                each pair its row in the expert-grouped buffer; expert segments start on
//                128-row boundaries so a segment is a whole number of GEMM row blocks
//   permute      gather token rows into the grouped buffer (optionally scaled by the gate: the
//                backward of combine), zeroing the padding rows
//   combine      out[t] = sum_s gate[t, s] * y[row(t, s)]  (gate = 1: backward of permute)
//   combine_bwd  dgate[t, s] = <y[row(t, s)], dout[t]>
//   route_bwd    gradient of the gates w.r.t. the router logits
//
// Row placement is a pure function of the expert ids (no atomics decide an order), so the
// grouped GEMMs and their weight gradients are bit-reproducible run to run.
//
// Reference semantics: model/__init__.py:485-598 of the reference (sigmoid router, top-k,
// gate normalisation with a 1e-9 floor); the grouped data path is this library's own.
#include "common.cuh"

namespace pb {
namespace moe {

// Tokens per block of the counting sort. One warp walks a block's pairs in order, 32 at a time, so more blocks are shorter
// walks, and more counts for the scan. 32 / 64 / 128 of them, us for the three kernels: 8192 tokens top-6 of 64 11.0 / 11.6 /
// 14.2, 32768 20.8 / 16.4 / 17.4, 4097 top-1 of 512 26.5 / 23.3 / 22.4 (256, and a scan of one thread an expert: 26.6, 39.1, 23.6).
constexpr int TOK_PER_BLOCK = 64;
constexpr int MAX_E = 512;
constexpr int MAX_K = 32;

// One warp per token. logits: [T, E] fp32. bias: [E] or null (selection only).
// PER = experts per lane the instantiation is unrolled for (2 covers 64 experts: a quarter of
// the compare / select work of the 512-expert form for the same result).
template <int PER>
__global__ void route_kernel(const float* __restrict__ logits, const float* __restrict__ bias,
                             int T, int E, int k, float* __restrict__ probs, int* __restrict__ ids,
                             float* __restrict__ gates) {
  after_previous_kernel();
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (warp >= T) return;
  const float* row = logits + static_cast<size_t>(warp) * E;
  float p[PER], s[PER];
  const int per = (E + 31) / 32;
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const int e = i * 32 + lane;
    if (i < per && e < E) {
      p[i] = 1.f / (1.f + expf(-row[e]));
      s[i] = p[i] + (bias ? bias[e] : 0.f);
      probs[static_cast<size_t>(warp) * E + e] = p[i];
    } else {
      p[i] = 0.f;
      s[i] = -INFINITY;
    }
  }
  float mine = 0.f;   // lane j keeps the probability of the j-th pick
  float sum = 0.f;
  for (int j = 0; j < k; ++j) {
    // best remaining (score, lowest index) of this lane, then across the warp
    float bv = -INFINITY;
    int be = 0x7fffffff;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int e = i * 32 + lane;
      if (i < per && s[i] > bv) { bv = s[i]; be = e; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
      const int oe = __shfl_xor_sync(0xffffffffu, be, o);
      if (ov > bv || (ov == bv && oe < be)) { bv = ov; be = oe; }
    }
    // owner lane retires the winner and reports its probability
    float pv = 0.f;
#pragma unroll
    for (int i = 0; i < PER; ++i)
      if (i * 32 + lane == be) { pv = p[i]; s[i] = -INFINITY; }
    pv = __shfl_sync(0xffffffffu, pv, be & 31);
    if (lane == j) mine = pv;
    sum += pv;
    if (lane == 0) ids[static_cast<size_t>(warp) * k + j] = be;
  }
  const float inv = 1.f / fmaxf(sum, 1e-9f);
  if (lane < k) gates[static_cast<size_t>(warp) * k + lane] = mine * inv;
}

// Gradient of gates w.r.t. logits. dgates, gates: [T, k]; probs: [T, E]; dlogits: [T, E] (zeroed
// here except at the selected experts).
__global__ void route_bwd_kernel(const float* __restrict__ dgates, const float* __restrict__ gates,
                                 const float* __restrict__ probs, const int* __restrict__ ids, int T,
                                 int E, int k, float* __restrict__ dlogits) {
  after_previous_kernel();
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (warp >= T) return;
  float* drow = dlogits + static_cast<size_t>(warp) * E;
  for (int e = lane; e < E; e += 32) drow[e] = 0.f;
  __syncwarp();
  if (lane == 0) {
    const size_t o = static_cast<size_t>(warp) * k;
    float sum = 0.f, dot = 0.f;
    for (int j = 0; j < k; ++j) {
      sum += probs[static_cast<size_t>(warp) * E + ids[o + j]];
      dot += dgates[o + j] * gates[o + j];
    }
    if (sum > 1e-9f) {
      const float inv = 1.f / sum;
      for (int j = 0; j < k; ++j) {
        const int e = ids[o + j];
        const float p = probs[static_cast<size_t>(warp) * E + e];
        drow[e] = (dgates[o + j] - dot) * inv * p * (1.f - p);
      }
    }
  }
}

// per-block histogram of expert ids. block_counts: [nblocks, E]
__global__ void count_kernel(const int* __restrict__ ids, int n_pairs, int pairs_per_block, int E,
                             int* __restrict__ block_counts) {
  after_previous_kernel();
  __shared__ int hist[MAX_E];
  for (int e = threadIdx.x; e < E; e += blockDim.x) hist[e] = 0;
  __syncthreads();
  const int lo = blockIdx.x * pairs_per_block;
  const int hi = min(lo + pairs_per_block, n_pairs);
  for (int i = lo + threadIdx.x; i < hi; i += blockDim.x) atomicAdd(&hist[ids[i]], 1);
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += blockDim.x)
    block_counts[static_cast<size_t>(blockIdx.x) * E + e] = hist[e];
}

// Segment starts from the experts' totals (one block; tot and off in shared memory):
//   expert_off[e] (128-aligned segment starts, expert_off[E] = rows in use), totals[e],
//   k_len[e] = padded segment length, mblk_group[m] for m < max_mblk (-1 beyond the data).
__device__ __forceinline__ void write_segments(const int* tot, int* off, int E, int* __restrict__ expert_off,
                                               int* __restrict__ totals, int* __restrict__ k_len,
                                               int* __restrict__ mblk_group, int max_mblk) {
  __syncthreads();
  if (threadIdx.x == 0) {
    int run = 0;
    for (int e = 0; e < E; ++e) {
      off[e] = run;
      run += (tot[e] + 127) / 128 * 128;
    }
    off[E] = run;
  }
  __syncthreads();
  for (int e = threadIdx.x; e <= E; e += blockDim.x) {
    expert_off[e] = off[e];
    if (e < E) {
      totals[e] = tot[e];
      k_len[e] = off[e + 1] - off[e];
    }
  }
  for (int m = threadIdx.x; m < max_mblk; m += blockDim.x) {
    const int row = m * 128;
    int g = -1;
    if (row < off[E]) {
      int lo = 0, hi = E;   // last e with off[e] <= row
      while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (off[mid] <= row) lo = mid; else hi = mid;
      }
      g = lo;
    }
    mblk_group[m] = g;
  }
}

constexpr int SCAN_THREADS = 512;
static_assert(SCAN_THREADS >= MAX_E, "a thread for every expert");
// One block. Turns block_counts into exclusive per-block bases and writes the segments.
__global__ void scan_kernel(int* __restrict__ block_counts, int nblocks, int E,
                            int* __restrict__ expert_off, int* __restrict__ totals,
                            int* __restrict__ k_len, int* __restrict__ mblk_group, int max_mblk) {
  after_previous_kernel();
  __shared__ int tot[MAX_E];
  __shared__ int off[MAX_E + 1];
  // A thread has one expert and a share of the blocks, eight counts in flight at a time: one thread an expert that
  // waited for each count took 10 us of 8192 tokens' 27.
  __shared__ int part[SCAN_THREADS];
  const int groups = SCAN_THREADS / E;   // at least one
  const int e = threadIdx.x % E, g = threadIdx.x / E;
  const int b0 = g < groups ? nblocks * g / groups : 0, b1 = g < groups ? nblocks * (g + 1) / groups : 0;
  int* mine = block_counts + e;
  auto walk = [&](int run, bool store) {
    for (int b = b0; b < b1; b += 8) {
      int c[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) c[u] = b + u < b1 ? mine[static_cast<size_t>(b + u) * E] : 0;
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        if (store && b + u < b1) mine[static_cast<size_t>(b + u) * E] = run;
        run += c[u];
      }
    }
    return run;
  };
  int base = 0;
  if (groups > 1) {
    part[threadIdx.x] = walk(0, false);
    __syncthreads();
    for (int q = 0; q < g && g < groups; ++q) base += part[q * E + e];
  }
  base = walk(base, true);
  if (g == groups - 1) tot[e] = base;
  write_segments(tot, off, E, expert_off, totals, k_len, mblk_group, max_mblk);
}

// One warp walks the pairs [lo, hi) in order; run[e] is the next row of expert e for them.
__device__ __forceinline__ void place_pairs(const int* __restrict__ ids, int lo, int hi, int* run,
                                            int* __restrict__ row_of, int lane) {
  int next = lo + lane < hi ? ids[lo + lane] : 0;
  for (int base = lo; base < hi; base += 32) {
    const int i = base + lane;
    const bool on = i < hi;
    const int e = on ? next : -1 - lane;
    if (i + 32 < hi) next = ids[i + 32];   // arrives while these are placed
    const unsigned same = __match_any_sync(0xffffffffu, e);
    const int rank = __popc(same & ((1u << lane) - 1u));
    int start = 0;
    if (on) start = run[e];
    __syncwarp();
    if (on) {
      row_of[i] = start + rank;
      if (rank == __popc(same) - 1) run[e] = start + rank + 1;   // last of its group advances
    }
    __syncwarp();
  }
}

// One warp per block of pairs; row_of[i] = expert_off + block base + rank.
__global__ void place_kernel(const int* __restrict__ ids, int n_pairs, int pairs_per_block, int E,
                             const int* __restrict__ block_base, const int* __restrict__ expert_off,
                             int* __restrict__ row_of) {
  after_previous_kernel();
  __shared__ int run[MAX_E];
  const int lane = threadIdx.x;
  for (int e = lane; e < E; e += 32)
    run[e] = expert_off[e] + block_base[static_cast<size_t>(blockIdx.x) * E + e];
  __syncwarp();
  const int lo = blockIdx.x * pairs_per_block;
  place_pairs(ids, lo, min(lo + pairs_per_block, n_pairs), run, row_of, lane);
}

// The whole sort in one block, each warp an eighth of the pairs: three launches less two for inputs whose
// kernels are shorter than a launch. Same placement (stable in the pair index).
// One / three, us: 1024 pairs of 8 experts 2.9 / 6.3, 2046 of 64 5.9 / 9.9, 4096 of 8 4.6 / 6.4, 4092 of 64 8.2 / 10.2.
constexpr int SORT_WARPS = 8, SORT_MAX = 4096;
__global__ void __launch_bounds__(SORT_WARPS * 32) sort_small_kernel(const int* __restrict__ ids, int n_pairs, int E,
                                                                     int* __restrict__ row_of,
                                                                     int* __restrict__ expert_off,
                                                                     int* __restrict__ totals,
                                                                     int* __restrict__ k_len,
                                                                     int* __restrict__ mblk_group, int max_mblk) {
  after_previous_kernel();
  __shared__ int run[SORT_WARPS][MAX_E];
  __shared__ int tot[MAX_E];
  __shared__ int off[MAX_E + 1];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int e = lane; e < E; e += 32) run[warp][e] = 0;
  __syncwarp();
  const int per = ((n_pairs + SORT_WARPS - 1) / SORT_WARPS + 31) / 32 * 32;
  const int lo = min(warp * per, n_pairs), hi = min(lo + per, n_pairs);
  for (int i = lo + lane; i < hi; i += 32) atomicAdd(&run[warp][ids[i]], 1);
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += blockDim.x) {
    int sum = 0;
#pragma unroll
    for (int w = 0; w < SORT_WARPS; ++w) {
      const int c = run[w][e];
      run[w][e] = sum;
      sum += c;
    }
    tot[e] = sum;
  }
  write_segments(tot, off, E, expert_off, totals, k_len, mblk_group, max_mblk);   // synchronises first
  for (int e = lane; e < E; e += 32) run[warp][e] += off[e];
  __syncwarp();
  place_pairs(ids, lo, hi, run[warp], row_of, lane);
}

constexpr int PAD_SPLIT = 8;   // blocks per expert that clear its padding rows
// zero rows [expert_off[e] + totals[e], expert_off[e + 1]), part of `parts` blocks
__device__ __forceinline__ void zero_pad_rows(bf16* __restrict__ buf, int d, int e, int part, int parts,
                                              const int* __restrict__ expert_off, const int* __restrict__ totals) {
  const int lo = expert_off[e] + totals[e], hi = expert_off[e + 1];
  const size_t n8 = static_cast<size_t>(hi - lo) * d / 8;
  bf16x8 z;
#pragma unroll
  for (int j = 0; j < 4; ++j) z.v[j] = __floats2bfloat162_rn(0.f, 0.f);
  bf16x8* p = reinterpret_cast<bf16x8*>(buf + static_cast<size_t>(lo) * d);
  for (size_t i = part * blockDim.x + threadIdx.x; i < n8; i += static_cast<size_t>(parts) * blockDim.x) p[i] = z;
}
__global__ void __launch_bounds__(256) zero_pad_kernel(bf16* __restrict__ buf, int d, const int* __restrict__ expert_off,
                                                       const int* __restrict__ totals) {
  after_previous_kernel();
  zero_pad_rows(buf, d, blockIdx.x, blockIdx.y, gridDim.y, expert_off, totals);
}
// the same rows of a quantised buffer: zero bytes, scale 1 (what the row quantiser makes of zeros)
__device__ __forceinline__ void zero_pad_q_rows(uint8_t* __restrict__ q, float* __restrict__ scales, int K, long rows,
                                                int e, int part, const int* __restrict__ expert_off,
                                                const int* __restrict__ totals) {
  const int lo = expert_off[e] + totals[e], n = expert_off[e + 1] - lo;
  const size_t first = part * blockDim.x + threadIdx.x, step = static_cast<size_t>(PAD_SPLIT) * blockDim.x;
  uint4* p = reinterpret_cast<uint4*>(q + static_cast<size_t>(lo) * K);
  for (size_t i = first; i < static_cast<size_t>(n) * K / 16; i += step) p[i] = make_uint4(0u, 0u, 0u, 0u);
  for (size_t i = first; i < static_cast<size_t>(n) * (K / 128); i += step)
    scales[(i / n) * rows + lo + i % n] = 1.f;
}

// dst[row_of[t, s]] = scale * src[t]; one warp per pair, up to 2048 columns in flight. d % 8 == 0.
// 65536 pairs x 2048: 92 -> 80 us (with the loads of one 256-column step at a time the warp waited
// once per step).
__global__ void __launch_bounds__(256) permute_kernel(const bf16* __restrict__ src, const int* __restrict__ row_of,
                                                      const float* __restrict__ scale, int n_pairs, int k, int d,
                                                      long ld_src, bf16* __restrict__ dst, long dst_rows,
                                                      int pair_blocks, const int* __restrict__ expert_off,
                                                      const int* __restrict__ totals) {
  after_previous_kernel();
  if (static_cast<int>(blockIdx.x) >= pair_blocks) {   // the blocks after the pairs' clear the padding rows
    const int i = blockIdx.x - pair_blocks;
    zero_pad_rows(dst, d, i / PAD_SPLIT, i % PAD_SPLIT, PAD_SPLIT, expert_off, totals);
    return;
  }
  const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (w >= n_pairs) return;
  const bf16* s = src + static_cast<size_t>(w / k) * ld_src;
  if (!PB_BOUNDS_OK(PB_K_MOE_PERMUTE, row_of[w], dst_rows)) return;
  bf16* o = dst + static_cast<size_t>(row_of[w]) * d;
  const float g = scale ? scale[w] : 1.f;
  for (int c0 = lane * 8; c0 < d; c0 += 2048) {
    bf16x8 v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (c0 + 256 * u < d) v[u] = *reinterpret_cast<const bf16x8*>(s + c0 + 256 * u);
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      if (c0 + 256 * u >= d) break;
      if (scale) {
        float f[8];
        unpack8(v[u], f);
#pragma unroll
        for (int j = 0; j < 8; ++j) f[j] *= g;
        v[u] = pack8(f);
      }
      *reinterpret_cast<bf16x8*>(o + c0 + 256 * u) = v[u];
    }
  }
}

// The same for rows that are already e4m3 with 1 x 128 scales: q [T, K] bytes and scales [K / 128, T] ->
// dq [rows, K], dscales [K / 128, rows]. A token is quantised once instead of once per expert it goes to,
// and the bf16 copy of its rows is never made. 65536 pairs x 2048 with the tokens' quantiser:
// permute + quantise 92 + 100 us -> 31 + 13 us.
__global__ void __launch_bounds__(256) permute_q_kernel(const uint8_t* __restrict__ q, const float* __restrict__ scales,
                                                        const int* __restrict__ row_of, int n_pairs, int k, int K,
                                                        int T, uint8_t* __restrict__ dq,
                                                        float* __restrict__ dscales, long dst_rows, int pair_blocks,
                                                        const int* __restrict__ expert_off,
                                                        const int* __restrict__ totals) {
  after_previous_kernel();
  if (static_cast<int>(blockIdx.x) >= pair_blocks) {
    const int i = blockIdx.x - pair_blocks;
    zero_pad_q_rows(dq, dscales, K, dst_rows, i / PAD_SPLIT, i % PAD_SPLIT, expert_off, totals);
    return;
  }
  const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (w >= n_pairs) return;
  const int t = w / k;
  if (!PB_BOUNDS_OK(PB_K_MOE_PERMUTE, row_of[w], dst_rows)) return;
  const size_t row = row_of[w];
  const uint8_t* s = q + static_cast<size_t>(t) * K;
  uint8_t* o = dq + row * K;
  for (int c0 = lane * 16; c0 < K; c0 += 2048) {
    uint4 v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (c0 + 512 * u < K) v[u] = *reinterpret_cast<const uint4*>(s + c0 + 512 * u);
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (c0 + 512 * u < K) *reinterpret_cast<uint4*>(o + c0 + 512 * u) = v[u];
  }
  for (int kb = lane; kb < K / 128; kb += 32)
    dscales[static_cast<size_t>(kb) * dst_rows + row] = scales[static_cast<size_t>(kb) * T + t];
}

// out[t] = sum_s gate[t, s] * y[row_of[t, s]] (+ add[t]); fp32 accumulate, slots in order. One warp
// per token and 512 columns, the rows of four slots in flight.
// 8192 tokens x 8 slots x 2048: 62.5 -> 61 us.
__global__ void __launch_bounds__(256) combine_kernel(const bf16* __restrict__ y, const int* __restrict__ row_of,
                                                      const float* __restrict__ gates, const bf16* __restrict__ add,
                                                      int T, int k, int d, bf16* __restrict__ out, long y_rows) {
  after_previous_kernel();
  const long w = (static_cast<long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31, parts = (d + 511) / 512;
  const long t = w / parts;
  if (t >= T) return;
  const int lo = static_cast<int>(w - t * parts) * 512, hi = min(d, lo + 512);
  for (int c = lo + lane * 8; c < hi; c += 256) {
    float acc[8];
    if (add != nullptr) unpack8(*reinterpret_cast<const bf16x8*>(add + static_cast<size_t>(t) * d + c), acc);
    else {
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[j] = 0.f;
    }
    for (int s0 = 0; s0 < k; s0 += 4) {
      bf16x8 v[4];
      float g[4];
      bool on[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const size_t i = static_cast<size_t>(t) * k + s0 + u;
        on[u] = s0 + u < k && PB_BOUNDS_OK(PB_K_MOE_COMBINE, row_of[i], y_rows);
        if (on[u]) {
          g[u] = gates ? gates[i] : 1.f;
          v[u] = *reinterpret_cast<const bf16x8*>(y + static_cast<size_t>(row_of[i]) * d + c);
        }
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (!on[u]) continue;
        float f[8];
        unpack8(v[u], f);
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[j] = fmaf(g[u], f[j], acc[j]);
      }
    }
    *reinterpret_cast<bf16x8*>(out + static_cast<size_t>(t) * d + c) = pack8(acc);
  }
}

// dgates[t, s] = <y[row_of[t, s]], dout[t]> ; one warp per pair
__global__ void combine_bwd_kernel(const bf16* __restrict__ y, const bf16* __restrict__ dout,
                                   const int* __restrict__ row_of, int n_pairs, int k, int d,
                                   float* __restrict__ dgates) {
  after_previous_kernel();
  const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (w >= n_pairs) return;
  const bf16* a = y + static_cast<size_t>(row_of[w]) * d;
  const bf16* b = dout + static_cast<size_t>(w / k) * d;
  float acc = 0.f;
  for (int c = lane * 8; c < d; c += 256) {
    float f[8], g[8];
    unpack8(*reinterpret_cast<const bf16x8*>(a + c), f);
    unpack8(*reinterpret_cast<const bf16x8*>(b + c), g);
#pragma unroll
    for (int j = 0; j < 8; ++j) acc = fmaf(f[j], g[j], acc);
  }
  acc = warp_sum(acc);
  if (lane == 0) dgates[w] = acc;
}

}  // namespace moe
}  // namespace pb

using namespace pb;

static inline int warps_grid(long warps, int threads) {
  return static_cast<int>((warps * 32 + threads - 1) / threads);
}

PB_API int pb_moe_route(const float* logits, const float* bias, int T, int E, int k, float* probs,
                        int* ids, float* gates, cudaStream_t st) {
  if (T <= 0 || E <= 0 || E > moe::MAX_E || k <= 0 || k > moe::MAX_K || k > E) return PB_BAD_ARG;
  const int per = (E + 31) / 32;
  const int grid = warps_grid(T, 256);
  if (per <= 2) pb::launch(moe::route_kernel<2>, grid, 256, 0, st, logits, bias, T, E, k, probs, ids, gates);
  else if (per <= 4) pb::launch(moe::route_kernel<4>, grid, 256, 0, st, logits, bias, T, E, k, probs, ids, gates);
  else if (per <= 8) pb::launch(moe::route_kernel<8>, grid, 256, 0, st, logits, bias, T, E, k, probs, ids, gates);
  else pb::launch(moe::route_kernel<moe::MAX_E / 32>, grid, 256, 0, st, logits, bias, T, E, k, probs, ids, gates);
  return static_cast<int>(cudaGetLastError());
}

PB_API int pb_moe_route_bwd(const float* dgates, const float* gates, const float* probs,
                            const int* ids, int T, int E, int k, float* dlogits, cudaStream_t st) {
  if (T <= 0 || E <= 0 || k <= 0) return PB_BAD_ARG;
  pb::launch(moe::route_bwd_kernel, warps_grid(T, 256), 256, 0, st, dgates, gates, probs, ids, T, E, k, dlogits);
  return static_cast<int>(cudaGetLastError());
}

PB_API int pb_moe_sort_nblocks(int n_pairs, int k) {
  const int per = moe::TOK_PER_BLOCK * k;
  return (n_pairs + per - 1) / per;
}

// Rows for the (token, slot) pairs grouped by expert. ids: [n_pairs] expert of each pair in
// token-major order; scratch: nblocks * E ints. Outputs: row_of [n_pairs]; expert_off [E + 1];
// totals [E]; k_len [E]; mblk_group [max_mblk].
PB_API int pb_moe_sort(const int* ids, int n_pairs, int k, int E, int* scratch, int* row_of,
                       int* expert_off, int* totals, int* k_len, int* mblk_group, int max_mblk,
                       cudaStream_t st) {
  if (n_pairs <= 0 || E <= 0 || E > moe::MAX_E || k <= 0) return PB_BAD_ARG;
  if (n_pairs <= moe::SORT_MAX) {
    pb::launch(moe::sort_small_kernel, 1, moe::SORT_WARPS * 32, 0, st, ids, n_pairs, E, row_of, expert_off, totals, k_len,
                                                               mblk_group, max_mblk);
    return static_cast<int>(cudaGetLastError());
  }
  const int per = moe::TOK_PER_BLOCK * k;
  const int nblocks = (n_pairs + per - 1) / per;
  pb::launch(moe::count_kernel, nblocks, 256, 0, st, ids, n_pairs, per, E, scratch);
  pb::launch(moe::scan_kernel, 1, moe::SCAN_THREADS, 0, st, scratch, nblocks, E, expert_off, totals, k_len, mblk_group,
                                      max_mblk);
  pb::launch(moe::place_kernel, nblocks, 32, 0, st, ids, n_pairs, per, E, scratch, expert_off, row_of);
  return static_cast<int>(cudaGetLastError());
}

PB_API int pb_moe_permute(const void* src, const int* row_of, const float* scale, int n_pairs, int k,
                          int d, long ld_src, void* dst, const int* expert_off, const int* totals,
                          int E, cudaStream_t st) {
  if (n_pairs <= 0 || d % 8 != 0) return PB_BAD_ARG;
  // rows of dst: the worst case the placement sizes its buffers for
  const long dst_rows = (static_cast<long>(n_pairs) + static_cast<long>(E > 0 ? E : 1) * 127 + 127) / 128 * 128;
  const int pair_blocks = warps_grid(n_pairs, 256);
  const int pad_blocks = expert_off != nullptr ? E * moe::PAD_SPLIT : 0;
  pb::launch(moe::permute_kernel, pair_blocks + pad_blocks, 256, 0, st, static_cast<const bf16*>(src), row_of, scale, n_pairs, k,
                                                                d, ld_src, static_cast<bf16*>(dst), dst_rows,
                                                                pair_blocks, expert_off, totals);
  return static_cast<int>(cudaGetLastError());
}

// Quantised token rows (q [T, K] e4m3 bytes, scales [K / 128, T]) into the grouped buffer dq [rows, K],
// dscales [K / 128, rows]; padding rows become zeros with scale 1. K a multiple of 128.
PB_API int pb_moe_permute_q(const void* q, const float* scales, const int* row_of, int T, int k, int K, void* dq,
                            float* dscales, long rows, const int* expert_off, const int* totals, int E,
                            cudaStream_t st) {
  if (T <= 0 || k <= 0 || K <= 0 || K % 128 != 0 || E <= 0) return PB_BAD_ARG;
  const int n_pairs = T * k;
  const int pair_blocks = warps_grid(n_pairs, 256);
  pb::launch(moe::permute_q_kernel, pair_blocks + E * moe::PAD_SPLIT, 256, 0, st,
      static_cast<const uint8_t*>(q), scales, row_of, n_pairs, k, K, T, static_cast<uint8_t*>(dq), dscales, rows,
      pair_blocks, expert_off, totals);
  return static_cast<int>(cudaGetLastError());
}

PB_API int pb_moe_zero_pad(void* buf, int d, const int* expert_off, const int* totals, int E,
                           cudaStream_t st) {
  if (E <= 0 || d % 8 != 0) return PB_BAD_ARG;
  pb::launch(moe::zero_pad_kernel, dim3(E, moe::PAD_SPLIT), 256, 0, st, static_cast<bf16*>(buf), d, expert_off, totals);
  return static_cast<int>(cudaGetLastError());
}

// y_rows: rows of y (the bound the debug build checks row_of against; 0 = unknown).
PB_API int pb_moe_combine(const void* y, const int* row_of, const float* gates, const void* add,
                          int T, int k, int d, void* out, long y_rows, cudaStream_t st) {
  if (T <= 0 || d % 8 != 0) return PB_BAD_ARG;
  pb::launch(moe::combine_kernel, warps_grid(static_cast<long>(T) * ((d + 511) / 512), 256), 256, 0, st,
      static_cast<const bf16*>(y), row_of, gates, static_cast<const bf16*>(add), T, k, d,
      static_cast<bf16*>(out), y_rows > 0 ? y_rows : (1L << 62));
  return static_cast<int>(cudaGetLastError());
}

PB_API int pb_moe_combine_bwd(const void* y, const void* dout, const int* row_of, int n_pairs, int k,
                              int d, float* dgates, cudaStream_t st) {
  if (n_pairs <= 0 || d % 8 != 0) return PB_BAD_ARG;
  pb::launch(moe::combine_bwd_kernel, warps_grid(n_pairs, 256), 256, 0, st,
      static_cast<const bf16*>(y), static_cast<const bf16*>(dout), row_of, n_pairs, k, d, dgates);
  return static_cast<int>(cudaGetLastError());
}

PB_DEFINE_BOUNDS_READER(moe)
