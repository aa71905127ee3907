// Causal softmax attention with grouped KV heads on tcgen05 (sm_100a), head dim 128.
//
// Forward (flash-style, one CTA per 256 query rows of one head, two tiles of 128):
//   S = Q K_j^T  (tensor memory, double-buffered)      P = exp2(S c - m)   (registers, one query row per
//   O += P V_j   (tensor memory)                       thread; back over S as the bf16 operand of P V)
// The running maximum is only raised when it would grow by more than 2^8 (the rescale of O is a
// tensor-memory read-modify-write, so it is skipped while the stale maximum is safe); the final
// O / l and the log-sum-exp use the maximum actually applied, which keeps the result exact.
//
// Backward, two kernels sharing one skeleton (no atomics, deterministic):
//   dQ  : CTA = 128 query rows; streams 64-key tiles   S = Q K^T, dP = dO V^T, dS = P (dP - delta) c
//         dQ += dS K
//   dKV : CTA = 128 key rows of one KV head; streams 64-query tiles of every query head of the
//         group  S^T = K Q^T, dP^T = V dO^T, dV += P^T dO, dK += dS^T Q
// Every streamed tile is used twice from the same shared-memory image: as the K-major B operand
// of the score product and as the MN-major B operand of the gradient product.
//
// Forward: warps 0-3 and 4-7 the rows of the two tiles, one tensor-memory lane (= row) per thread; warps 8 and 9 MMA
// issue, one tile each; warp 10 TMA producer. Backward: warps 0-7 rows, 8-10 MMA issue, 11 TMA producer.
// All tensors are token-major: Q/O/dO/dQ [batch * seq, ldq] with head h at columns 128 h,
// K/V/dK/dV [batch * seq, ldkv] with KV head g at columns 128 g. Any seq: the tensor maps are per batch entry,
// so the rows a last tile lacks read as zeros (no real query sees a key after itself, and a zero
// query with zero dO adds nothing) and are clipped from the stores. 3 x 1000 x 16/4 forward: 19.0 us; with
// padded copies of q, k, v and a cut of the result it took 48 us more.
//
// Reference semantics: model/__init__.py gqa/mla attention (softmax(q k^T / sqrt(d)) v with a
// causal mask) of the reference; the tiling is this library's own.
#include <cuda.h>

#include <climits>
#include <type_traits>

#include "common.cuh"

namespace pb {

int make_tmap_3d(CUtensorMap* tm, const void* base, int elem_bytes, uint64_t inner,
                 uint64_t outer, uint64_t batch, uint64_t ld_elems, uint64_t batch_stride_elems,
                 uint32_t box_inner, uint32_t box_outer);

namespace attn {

constexpr int D = 128;
constexpr float RESCALE_THRESHOLD = 8.f;  // log2 units

// Optional cycle accounting of the forward row warps (compile with -DPB_ATTN_PROF): thread 0 of
// each warpgroup adds the clocks it spent in each phase of a block to a device array.
#ifdef PB_ATTN_PROF
__device__ unsigned long long g_attn_prof[8];
#define PB_PROF_START long long prof_t = clock64();
#define PB_PROF(i)                                                                  \
  if (r == 0) {                                                                     \
    const long long prof_n = clock64();                                             \
    atomicAdd(&g_attn_prof[i], static_cast<unsigned long long>(prof_n - prof_t));  \
    prof_t = prof_n;                                                                \
  }
#else
#define PB_PROF_START
#define PB_PROF(i)
#endif

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// 16-byte store of 8 bf16 into a [rows][64] 128B-swizzled chunk (row pitch 128 bytes).
__device__ __forceinline__ void st_swz(uint8_t* chunk_base, int row, int c16, const bf16x8& v) {
  st_shared8(chunk_base + row * 128 + ((c16 ^ (row & 7)) << 4), v);
}
__device__ __forceinline__ bf16x8 pack_bf16x8(const float* f) {
  bf16x8 pk;
#pragma unroll
  for (int j = 0; j < 4; ++j) pk.v[j] = __floats2bfloat162_rn(f[2 * j], f[2 * j + 1]);
  return pk;
}
__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&v);
}
// Two fp32 operations in one instruction, each rounded as the scalar one.
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  float2 d;
  asm("{\n\t.reg .b64 pa, pb, pc;\n\tmov.b64 pa, {%2, %3};\n\tmov.b64 pb, {%4, %5};\n\tmov.b64 pc, {%6, %7};\n\t"
      "fma.rn.f32x2 pa, pa, pb, pc;\n\tmov.b64 {%0, %1}, pa;\n\t}"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return d;
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  float2 d;
  asm("{\n\t.reg .b64 pa, pb;\n\tmov.b64 pa, {%2, %3};\n\tmov.b64 pb, {%4, %5};\n\t"
      "add.rn.f32x2 pa, pa, pb;\n\tmov.b64 {%0, %1}, pa;\n\t}"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
  float2 d;
  asm("{\n\t.reg .b64 pa, pb;\n\tmov.b64 pa, {%2, %3};\n\tmov.b64 pb, {%4, %5};\n\t"
      "mul.rn.f32x2 pa, pa, pb;\n\tmov.b64 {%0, %1}, pa;\n\t}"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
__device__ __forceinline__ bool wait_all(uint64_t* bar, uint32_t parity, int* status) {
  return mbar_wait_spin_warp(bar, parity, status);
}

// Registers of a tensor-memory load are valid after the wait: no use of them may move above this.
__device__ __forceinline__ void tie32(uint32_t (&v)[32]) {
#pragma unroll
  for (int i = 0; i < 32; i += 8)
    asm volatile("" : "+r"(v[i]), "+r"(v[i + 1]), "+r"(v[i + 2]), "+r"(v[i + 3]), "+r"(v[i + 4]), "+r"(v[i + 5]),
                      "+r"(v[i + 6]), "+r"(v[i + 7]));
}

__device__ __forceinline__ void tie16(uint32_t (&v)[16]) {
#pragma unroll
  for (int i = 0; i < 16; i += 8)
    asm volatile("" : "+r"(v[i]), "+r"(v[i + 1]), "+r"(v[i + 2]), "+r"(v[i + 3]), "+r"(v[i + 4]), "+r"(v[i + 5]),
                      "+r"(v[i + 6]), "+r"(v[i + 7]));
}

// ------------------------------------------------------------------------------ forward
namespace fwd {
// shared memory: Q (two 128-row tiles, at the end the staging of O), five K/V stages of 64 keys
constexpr int Q_OFF = 0, KV_OFF = 65536, KV_STAGES = 5, KV_STAGE = 32768;
constexpr int BARS = KV_OFF + KV_STAGES * KV_STAGE;
constexpr int SMEM = BARS + 512 + 1024;
static_assert(SMEM <= 227 * 1024, "one CTA's shared memory");
// S[tile][buf] 64 columns, of which P takes the first 32 as packed bf16 operand; O[tile] 128
constexpr uint32_t COL_S = 0, COL_O = 256, TMEM_COLS = 512;

struct Params {
  int batch, seq, heads, kv_heads;   // seq: query rows per batch entry
  int seq_kv, q_off;          // key rows per batch entry; global position of query row 0
  float scale_log2;   // softmax scale * log2(e)
  float* lse2;        // [batch, heads, seq], log2 domain
  float* rowmax;      // [batch, heads, seq] largest scaled logit of the row, or null
  int* status;
};

// One CTA = 256 query rows of one head: two 128-row tiles, each owned by one warpgroup
// (warps 0-3 and 4-7) so that one group's exponentials overlap the other's tensor-core work.
// Keys and values arrive in blocks of 64. P goes back to tensor memory, over the scores it was made of, as the A
// operand of P V: 32 KB less shared-memory traffic per block and tile than an operand tile written and read
// there, and room for five K/V stages instead of three. A block of both tiles takes about 1650
// clocks: 1280 of products (Q K^T at N = 64 reads 6 KB of shared memory a step) and 1024 of exponentials, which overlap but for
// the latencies around them. P in tensor memory 4 x 4096 x 16/4 294 -> 280 us, products issued by a warp 280 -> 259 (1 x
// 8192 x 4/1 132.8 -> 112.7). Taken back: one exponential in eight as a polynomial on the FMA pipe, the same time, one in four
// slower; the next block's scores read before this one's exponentials 117; the groups' exponentials in turns 120.
// warps 8 and 9: MMA issue for tile 0 and tile 1, warp 10: TMA producer.
__global__ void __launch_bounds__(352, 1)
attn_fwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmO,
                const Params p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + BARS);
  uint64_t* q_full = bars;
  uint64_t* kv_full = bars + 1;    // [KV_STAGES]
  uint64_t* kv_empty = bars + 6;   // [KV_STAGES]
  uint64_t* s_done = bars + 11;    // [tile][buf]
  // [tile][buf], like the scores: these run two blocks ahead, so a warp may be done with block j + 1 while another still
  // rescales O in block j. With one barrier for both, its two arrivals and two of the others would complete block j's phase,
  // and P V would read the slow warp's raw scores as its P. Block j + 2 of a buffer comes after P V of j, that is after all.
  uint64_t* p_ready = bars + 15;
  uint64_t* o_done = bars + 19;    // [tile][buf]: P V of the block whose scores that buffer held
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 23);

  const int warp = warp_index(), lane = threadIdx.x & 31;
  // blocks start in index order, so the row block is the slowest index: the longest rows of all heads and
  // batch entries first, the shortest fill the gaps at the end. One grid dimension for all three: the others end
  // at 65535 blocks
  const int per = p.heads * p.batch;
  const int at = static_cast<int>(blockIdx.x % per);
  const int cb = static_cast<int>(gridDim.x / per) - 1 - static_cast<int>(blockIdx.x / per);
  const int b = at / p.heads, h = at - b * p.heads;
  const int g = h / (p.heads / p.kv_heads);
  const int gb = cb + p.q_off / 256;   // position of this CTA's rows among all keys
  const int row0 = cb * 256;           // first query row within the batch entry
  const int nj1 = 4 * gb + 4;     // 64-key blocks seen by tile 1; tile 0 sees nj1 - 2

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int i = 0; i < KV_STAGES; ++i) { mbar_init(&kv_full[i], 1); mbar_init(&kv_empty[i], 2); }
    for (int i = 0; i < 4; ++i) {
      mbar_init(&s_done[i], 1); mbar_init(&o_done[i], 1);
      mbar_init(&p_ready[i], 4);   // one arrival per warp
    }
    fence_barrier_init();
    tma_prefetch_desc(&tmQ); tma_prefetch_desc(&tmK); tma_prefetch_desc(&tmV);
  }
  if (warp == 8) {
    tmem_alloc(tmem_slot, TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  after_previous_kernel();

  if (warp == 10) {
    if (lane == 0) {
      mbar_arrive_expect_tx(q_full, 65536);
      for (int t = 0; t < 2; ++t) {
        tma_load_3d(smem + Q_OFF + t * 32768, &tmQ, q_full, h * D, row0 + t * 128, b);
        tma_load_3d(smem + Q_OFF + t * 32768 + 16384, &tmQ, q_full, h * D + 64, row0 + t * 128, b);
      }
      for (int j = 0; j < nj1; ++j) {
        const int s = j % KV_STAGES;
        const uint32_t ph = (j / KV_STAGES) & 1;
        const int krow = j * 64;
        if (!mbar_wait(&kv_empty[s], ph ^ 1, p.status)) break;
        mbar_arrive_expect_tx(&kv_full[s], KV_STAGE);
        uint8_t* st = smem + KV_OFF + s * KV_STAGE;
        tma_load_3d(st, &tmK, &kv_full[s], g * D, krow, b);
        tma_load_3d(st + 8192, &tmK, &kv_full[s], g * D + 64, krow, b);
        tma_load_3d(st + 16384, &tmV, &kv_full[s], g * D, krow, b);
        tma_load_3d(st + 16384 + 8192, &tmV, &kv_full[s], g * D + 64, krow, b);
      }
    }
  } else if (warp >= 8) {
    {
      const int t = warp - 8;                                     // the tile this warp issues for
      const int nj = nj1 - (t == 0 ? 2 : 0);
      const uint32_t id_s = make_idesc(1, 1, 128, 64, 0, 0);     // S = Q K^T, N = 64 keys
      const uint32_t id_o = make_idesc(1, 1, 128, 128, 0, 1);    // O += P V, V MN-major
      constexpr uint32_t HI = sdesc_hi_sw128(1024);
      // descriptor low words are kept in registers: one add per operand per MMA
      const uint32_t q_lo = sdesc_lo(smem_u32(smem + Q_OFF + t * 32768), 16);
      const uint32_t kv0 = smem_u32(smem + KV_OFF);
      const uint32_t d_o = tmem + COL_O + t * 128;
      bool ok = mbar_wait_spin_warp(q_full, 0, p.status);
      auto issue_s = [&](int j) -> bool {
        const int s = j % KV_STAGES;
        const int sb = t * 2 + (j & 1);
        if (!mbar_wait_spin_warp(&kv_full[s], (j / KV_STAGES) & 1, p.status)) return false;
        // the buffer still holds P of block j - 2 until its P V product is done
        if (j >= 2 && !mbar_wait_spin_warp(&o_done[sb], ((j - 2) >> 1) & 1, p.status)) return false;
        tc_fence_after();
        const uint32_t k_lo = sdesc_lo(kv0 + s * KV_STAGE, 16);
        const uint32_t d = tmem + COL_S + sb * 64;
#pragma unroll
        for (int jj = 0; jj < 8; ++jj)
          umma_f16_words_warp(d, q_lo + (((jj >> 2) * 16384 + (jj & 3) * 32) >> 4), HI,
                         k_lo + (((jj >> 2) * 8192 + (jj & 3) * 32) >> 4), HI, id_s, jj > 0);
        umma_commit_warp(&s_done[sb]);
        return true;
      };
      // the scores run two blocks ahead of the P V products, so neither the row warps nor
      // the P V issue ever wait for a K/V tile that is still in flight
      if (ok) ok = issue_s(0);
      if (ok && nj > 1) ok = issue_s(1);
      for (int j = 0; j < nj && ok; ++j) {
        const int s = j % KV_STAGES;
        if (!mbar_wait_spin_warp(&p_ready[t * 2 + (j & 1)], (j >> 1) & 1, p.status)) break;
        tc_fence_after();
        const uint32_t v_lo = sdesc_lo(kv0 + s * KV_STAGE + 16384, 8192);
        // 16 values of a bf16 operand row are eight tensor-memory columns
        const uint32_t p_col = tmem + COL_S + (t * 2 + (j & 1)) * 64;
#pragma unroll
        for (int jj = 0; jj < 4; ++jj)
          umma_f16_ts_warp(d_o, p_col + jj * 8, (static_cast<uint64_t>(HI) << 32) | (v_lo + ((jj * 2048) >> 4)), id_o,
                      (j > 0) || (jj > 0));
        umma_commit_warp(&o_done[t * 2 + (j & 1)]);
        umma_commit_warp(&kv_empty[s]);   // needs both tiles' commits (tile 0 skips the last two blocks,
                                     // whose stages are never refilled)
        if (j + 2 < nj && !issue_s(j + 2)) break;
      }
    }
  } else {
    const int t = warp >> 2;               // tile / warpgroup
    const int r = threadIdx.x & 127;       // query row of the tile = tensor-memory lane
    const uint32_t lane_addr = tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16);
    const int qpos = gb * 256 + t * 128 + r;     // global position (for the causal mask)
    const int q0 = gb * 256 + t * 128;
    const int nj = nj1 - (t == 0 ? 2 : 0);
    float m_used = -INFINITY, m_true = -INFINITY, l = 0.f;
    bool ok = true;
    for (int j = 0; j < nj && ok; ++j) {
      const int sb = t * 2 + (j & 1);
      const uint32_t ph = (j >> 1) & 1;
      const bool edge = j * 64 + 63 > q0;
      PB_PROF_START
      if (!wait_all(&s_done[sb], ph, p.status)) { ok = false; break; }
      tc_fence_after();
      PB_PROF(0)
      uint32_t v[64];
      tmem_ld_32x32b_x32(lane_addr + COL_S + sb * 64, v);
      tmem_ld_32x32b_x32(lane_addr + COL_S + sb * 64 + 32, v + 32);
      tmem_ld_wait();
      PB_PROF(1)
      if (edge) {   // only the blocks on the diagonal pay for the mask
#pragma unroll
        for (int i = 0; i < 64; ++i)
          if (j * 64 + i > qpos) v[i] = 0xff800000u;   // -inf
      }
      float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int i = 0; i < 64; i += 2)
        mx4[(i >> 1) & 3] = max3(mx4[(i >> 1) & 3], __uint_as_float(v[i]), __uint_as_float(v[i + 1]));
      const float mx = fmaxf(max3(mx4[0], mx4[1], mx4[2]), mx4[3]) * p.scale_log2;
      m_true = fmaxf(m_true, mx);
      PB_PROF(2)
      if (j == 0) {
        m_used = mx;
      } else if (__any_sync(0xffffffffu, mx > m_used + RESCALE_THRESHOLD)) {
        // raise the applied maximum: O of this tile must be idle (previous P V finished)
        if (!wait_all(&o_done[t * 2 + ((j - 1) & 1)], ((j - 1) >> 1) & 1, p.status)) { ok = false; break; }
        tc_fence_after();
        const float m_new = fmaxf(m_used, mx);
        const float alpha = ex2(m_used - m_new);
        l *= alpha;
#pragma unroll 1
        for (int c = 0; c < D; c += 32) {
          uint32_t o[32];
          tmem_ld_32x32b_x32(lane_addr + COL_O + t * 128 + c, o);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
          tmem_st_32x32b_x32(lane_addr + COL_O + t * 128 + c, o);
        }
        tmem_st_wait();
        m_used = m_new;
      }
      PB_PROF(3)
      const float2 neg_m = make_float2(-m_used, -m_used), mul = make_float2(p.scale_log2, p.scale_log2);
      float2 l01 = make_float2(0.f, 0.f), l23 = make_float2(0.f, 0.f);
      uint32_t pk[32];   // the row's P, two bf16 to a register
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        // one fused multiply-add and one exponential per score; masked entries are -inf -> 0
        const float2 ea = fma2(make_float2(__uint_as_float(v[4 * i]), __uint_as_float(v[4 * i + 1])), mul, neg_m);
        const float2 eb = fma2(make_float2(__uint_as_float(v[4 * i + 2]), __uint_as_float(v[4 * i + 3])), mul, neg_m);
        const float2 fa = make_float2(ex2(ea.x), ex2(ea.y)), fb = make_float2(ex2(eb.x), ex2(eb.y));
        l01 = add2(l01, fa);
        l23 = add2(l23, fb);
        pk[2 * i] = pack_bf16x2(fa.x, fa.y);
        pk[2 * i + 1] = pack_bf16x2(fb.x, fb.y);
      }
      tmem_st_32x32b_x32(lane_addr + COL_S + sb * 64, pk);
      l += (l01.x + l01.y) + (l23.x + l23.y);
      PB_PROF(4)
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_ready[sb]);
      PB_PROF(5)
#ifdef PB_ATTN_PROF
      if (r == 0) atomicAdd(&g_attn_prof[6], 1ull);
#endif
    }
    ok = ok && wait_all(&o_done[t * 2 + ((nj - 1) & 1)], ((nj - 1) >> 1) & 1, p.status);
    uint8_t* obuf = smem + Q_OFF + t * 32768;   // no product of the tile reads its Q any more
    if (ok) {
      tc_fence_after();
      const float inv = 1.f / l;
#pragma unroll 1
      for (int c = 0; c < D; c += 32) {
        uint32_t o[32];
        tmem_ld_32x32b_x32(lane_addr + COL_O + t * 128 + c, o);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          float f[8];
#pragma unroll
          for (int k = 0; k < 8; ++k) f[k] = __uint_as_float(o[8 * i + k]) * inv;
          const int col = c + 8 * i;
          st_swz(obuf + (col >> 6) * 16384, r, (col & 63) >> 3, pack_bf16x8(f));
        }
      }
      const int qrow = row0 + t * 128 + r;
      if (qrow < p.seq) {
        const size_t vi = (static_cast<size_t>(b) * p.heads + h) * p.seq + qrow;
        p.lse2[vi] = m_used + log2f(l);
        if (p.rowmax != nullptr) p.rowmax[vi] = m_true * 0.6931471805599453f;
      }
      fence_proxy_async_smem();
    }
    // a warp whose wait ran out arrives too: the group stores its tile or leaves together
    if (bar_sync_and(1 + t, 128, ok) && r == 0 && row0 + t * 128 < p.seq) {
      tma_store_3d(&tmO, obuf, h * D, row0 + t * 128, b);
      tma_store_3d(&tmO, obuf + 16384, h * D + 64, row0 + t * 128, b);
      tma_store_commit();
      tma_store_wait<0>();
    }
  }

  tc_fence_before();
  __syncthreads();
  if (p.status != nullptr && *reinterpret_cast<volatile int*>(p.status) != PB_OK) {
    for (int i = 0; i < 2000; ++i) __nanosleep(1000);  // let copies in flight land
    __syncthreads();
  }
  if (warp == 8) {
    tc_fence_after();
    tmem_dealloc(tmem, TMEM_COLS);
  }
}
}  // namespace fwd

// ----------------------------------------------------------------------------- backward
namespace bwd {
// Streamed tiles: T1 16 KB + T2 16 KB a stage. dQ copies its resident tiles into tensor memory and then
// streams through their shared memory too (stages 4 and 5); dK / dV keeps them, and has 512 bytes a stage of
// the streamed queries' log-sum-exp and delta.
constexpr int RA_OFF = 0, RB_OFF = 32768, ST_OFF = 65536;
template <bool DKV> struct Ring {
  static constexpr int STAGES = DKV ? 4 : 6;
  __device__ static int off(int s) { return s < 4 ? ST_OFF + s * 32768 : (s - 4) * 32768; }
};
constexpr int VEC_OFF = ST_OFF + 4 * 32768, BARS = VEC_OFF + 4 * 512;
constexpr int SMEM = BARS + 256 + 1024;
static_assert(SMEM <= 227 * 1024, "one CTA's shared memory");
// tensor memory: two score buffers of 128 columns (X1 at 0, X2 at 64), then the accumulators, and for dQ
// its resident tiles. Row warpgroup g works on columns 32 g .. 32 g + 31 of X1 and X2 and puts what it makes of
// them, packed bf16 operands (P^T over X1, dS over X2), over the first 16 of its own: no warp writes
// what another still reads.
constexpr uint32_t COL_X2 = 64, COL_ACC1 = 256, COL_ACC2 = 384, COL_R = 384, TMEM_COLS = 512;

struct Params {
  int batch, seq, heads, kv_heads, n_blk;  // seq: query rows per batch entry; n_blk: 128-row blocks of the grid
  int seq_kv, q_off;                // key rows per batch entry; global position of query row 0
  float scale_log2, scale;
  const float* lse2;    // [batch, heads, seq]
  // [batch, heads, ceil(seq / 64), 32 pairs of rows, {-lse2, -lse2, -delta, -delta}], delta = rowsum(dO * O), zeros
  // past seq: written by the dQ kernel, read by the other a tile (512 bytes) at a time
  float* vec;
  int* status;
};

// DKV = false: resident Q, dO (one head); streams K, V tiles; output dQ.
// DKV = true : resident K, V (one KV head); streams Q, dO tiles of the group; outputs dK, dV.
// Two warpgroups (warps 0-3, 4-7) share every streamed tile, half of its columns each: what a tile waits for is its
// score products, the rows' work on them and its gradient products one after the other, with two tiles on the
// way, and the rows' part of that chain halves.  MMA issue is spread over three warps, so that each
// waits only for what its own products need: warp 8 the first score product, warp 9 the second, warp 10 the gradient
// accumulations; warp 11: TMA producer. (One lane could not issue all 20+ products of a tile in time; whether one warp can
// was not measured.)
//
// Shared-memory bandwidth is what the products compete for: a 128 x 64 score product with both operands there reads
// 6 KB per 16-deep step, half as much again as the tensor core can use. So what can be kept off it is: P^T
// and dS go back to tensor memory as bf16 and are the gradient products' A operand there; dQ's resident
// tiles are A operands in tensor memory too (2 KB a step), and their shared memory holds two more stages of streamed
// tiles, whose loads were late with four (dK / dV has no tensor memory left for its own). The streamed queries'
// log-sum-exp and delta come with their tile, and a lane of the dK / dV rows reads 8 columns of them instead of 64.
// dS is rounded to bf16 once, with the softmax scale in it: P (dP - delta) scale costs two multiplications an
// element, so the rows' arithmetic is packed two elements to an instruction.
// 4 x 4096 x 16/4, clocks a 128 x 64 tile: dQ 1157 -> 1081 (768 of them MMAs), dK and dV 1908 -> 1500 (1280; 1644
// before a warp issued them); together 909 -> 811 us. A dQ block spends 10000 of 45000 clocks outside its loop: its
// resident tiles' arrival, delta, and the stores.
template <bool DKV>
__global__ void __launch_bounds__(384, 1)
attn_bwd_kernel(const __grid_constant__ CUtensorMap tmRA, const __grid_constant__ CUtensorMap tmRB,
                const __grid_constant__ CUtensorMap tmT1, const __grid_constant__ CUtensorMap tmT2,
                const __grid_constant__ CUtensorMap tmO1, const __grid_constant__ CUtensorMap tmO2,
                const __grid_constant__ CUtensorMap tmFO, const Params p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + BARS);
  uint64_t* r_full = bars;
  uint64_t* t_full = bars + 1;    // [STAGES]
  uint64_t* t_empty = bars + 7;   // [STAGES]
  uint64_t* x_done = bars + 13;   // [2] scores of a buffer
  uint64_t* x_free = bars + 15;   // [2] its gradient products
  uint64_t* pd_ready = bars + 17; // [2] its P^T and dS
  uint64_t* acc_done = bars + 19;
  uint64_t* o_full = bars + 20;   // dQ: the forward's output tile, in the last of the first four stages
  uint64_t* r_read = bars + 21;   // dQ: delta is taken from it and from the resident dO
  uint64_t* r_copied = bars + 22; // dQ: the resident tiles are in tensor memory
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 23);
  constexpr int STAGES = Ring<DKV>::STAGES, O_STAGE = 3;
  auto stage = [&](int s) { return smem + Ring<DKV>::off(s); };

  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int group = p.heads / p.kv_heads;
  // dQ: heavy blocks are the late query blocks; dKV: the early key blocks. Heavy blocks of all heads and
  // batch entries come first, in one grid dimension, as in the forward.
  const int rows_y = DKV ? p.kv_heads : p.heads, per = rows_y * p.batch;
  const int blk0 = static_cast<int>(blockIdx.x / per), at = static_cast<int>(blockIdx.x % per);
  const int blk = DKV ? blk0 : p.n_blk - 1 - blk0;
  const int b = at / rows_y;
  const int hy = at - b * rows_y;                  // query head (dQ) or KV head (dKV)
  const int g = DKV ? hy : hy / group;
  // dQ: blk is a local query block, streamed tiles are global key tiles 0 .. diagonal.
  // dKV: blk is a global key block, streamed tiles are the local query tiles at or after it.
  const int gblk = DKV ? blk : blk + p.q_off / 128;
  const int q_off64 = p.q_off / 64;
  const int t_first = DKV ? max(0, 2 * blk - q_off64) : 0;
  const int t_count = DKV ? max(0, (p.seq + 63) / 64 - t_first) : 2 * gblk + 2;
  const int n_it = DKV ? group * t_count : t_count;
  const int row0 = blk * 128;                      // within the batch entry

  if (threadIdx.x == 0) {
    mbar_init(r_full, 1);
    for (int i = 0; i < STAGES; ++i) { mbar_init(&t_full[i], 1); mbar_init(&t_empty[i], 1); }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&x_done[i], 2); mbar_init(&x_free[i], 1);    // two issuing warps
      mbar_init(&pd_ready[i], 8);                            // one arrival per row warp
    }
    mbar_init(acc_done, 1);
    mbar_init(o_full, 1); mbar_init(r_read, 8); mbar_init(r_copied, 8);
    fence_barrier_init();
    tma_prefetch_desc(&tmRA); tma_prefetch_desc(&tmRB);
    tma_prefetch_desc(&tmT1); tma_prefetch_desc(&tmT2);
  }
  if (warp == 8) {
    tmem_alloc(tmem_slot, TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  after_previous_kernel();

  if (warp == 11) {
    if (lane == 0) {
      const int rx = (DKV ? g : hy) * D;
      // A key block that no local query sees streams nothing: its resident tiles are not
      // loaded either, because their buffers are the staging of the all-zero stores and no one
      // would wait for the loads to land first.
      if (n_it > 0) {
        mbar_arrive_expect_tx(r_full, 65536);
        tma_load_3d(smem + RA_OFF, &tmRA, r_full, rx, row0, b);
        tma_load_3d(smem + RA_OFF + 16384, &tmRA, r_full, rx + 64, row0, b);
        tma_load_3d(smem + RB_OFF, &tmRB, r_full, rx, row0, b);
        tma_load_3d(smem + RB_OFF + 16384, &tmRB, r_full, rx + 64, row0, b);
      }
      if (!DKV) {
        mbar_arrive_expect_tx(o_full, 32768);
        tma_load_3d(stage(O_STAGE), &tmFO, o_full, rx, row0, b);
        tma_load_3d(stage(O_STAGE) + 16384, &tmFO, o_full, rx + 64, row0, b);
      }
      for (int it = 0; it < n_it; ++it) {
        const int s = it % STAGES;
        const uint32_t ph = (it / STAGES) & 1;
        const int t = t_first + (DKV ? it % t_count : it);
        const int th = DKV ? g * group + it / t_count : g, tx = th * D;
        const int trow = t * 64;
        if (!mbar_wait(&t_empty[s], ph ^ 1, p.status)) break;
        if (!DKV && it == O_STAGE && !mbar_wait(r_read, 0, p.status)) break;
        mbar_arrive_expect_tx(&t_full[s], DKV ? 32768 + 512 : 32768);
        uint8_t* st = stage(s);
        if (DKV)
          bulk_load(smem + VEC_OFF + s * 512,
                    p.vec + ((static_cast<size_t>(b) * p.heads + th) * ((p.seq + 63) / 64) + t) * 128, 512, &t_full[s]);
        tma_load_3d(st, &tmT1, &t_full[s], tx, trow, b);
        tma_load_3d(st + 8192, &tmT1, &t_full[s], tx + 64, trow, b);
        tma_load_3d(st + 16384, &tmT2, &t_full[s], tx, trow, b);
        tma_load_3d(st + 16384 + 8192, &tmT2, &t_full[s], tx + 64, trow, b);
      }
    }
  } else if (warp == 8 || warp == 9) {
    // score products: warp 8 issues X1 = RA T1^T, warp 9 issues X2 = RB T2^T
    {
      const int which = warp - 8;
      const uint32_t id_x = make_idesc(1, 1, 128, 64, 0, 0);     // A K-major, B K-major, N = 64
      constexpr uint32_t HI = sdesc_hi_sw128(1024);
      const uint32_t r_lo = sdesc_lo(smem_u32(smem + (which == 0 ? RA_OFF : RB_OFF)), 16);
      const uint32_t r_col = tmem + COL_R + which * 64;
      const uint32_t col = which == 0 ? 0 : COL_X2;
      bool ok = n_it == 0 || mbar_wait_spin_warp(DKV ? r_full : r_copied, 0, p.status);
      int ts = 0;
      uint32_t ph = 0;
      for (int it = 0; it < n_it && ok; ++it) {
        const int s = it & 1;
        if (!mbar_wait_spin_warp(&t_full[ts], ph, p.status)) break;
        if (!mbar_wait_spin_warp(&x_free[s], ((it >> 1) & 1) ^ 1, p.status)) break;
        tc_fence_after();
        const uint32_t t_lo = sdesc_lo(smem_u32(stage(ts)) + which * 16384, 16);
        const uint32_t d = tmem + col + s * 128;
#pragma unroll
        for (int jj = 0; jj < 8; ++jj) {
          const uint32_t b_lo = t_lo + (((jj >> 2) * 8192 + (jj & 3) * 32) >> 4);
          if (DKV)
            umma_f16_words_warp(d, r_lo + (((jj >> 2) * 16384 + (jj & 3) * 32) >> 4), HI, b_lo, HI, id_x, jj > 0);
          else
            umma_f16_ts_warp(d, r_col + jj * 8, (static_cast<uint64_t>(HI) << 32) | b_lo, id_x, jj > 0);
        }
        umma_commit_warp(&x_done[s]);
        if (++ts == STAGES) { ts = 0; ph ^= 1; }
      }
    }
  } else if (warp == 10) {
    // gradient accumulations, all from this one warp so that they stay ordered
    {
      const uint32_t id_acc = make_idesc(1, 1, 128, 128, 0, 1);  // A from tensor memory, B MN-major
      constexpr uint64_t HI = static_cast<uint64_t>(sdesc_hi_sw128(1024)) << 32;
      int it = 0, ts = 0;
      for (; it < n_it; ++it) {
        const int s = it & 1;
        if (!mbar_wait_spin_warp(&pd_ready[s], (it >> 1) & 1, p.status)) break;
        tc_fence_after();
        // the streamed tiles again, now as MN-major B operands (64-wide chunks 8 KB apart); 16
        // values of a bf16 operand row are eight tensor-memory columns, 32 of them to a warpgroup's part
        const uint32_t t1_mn = sdesc_lo(smem_u32(stage(ts)), 8192), t2_mn = t1_mn + (16384 >> 4);
        const uint32_t xb = tmem + s * 128;
        auto a_col = [](const int jj) { return static_cast<uint32_t>((jj >> 1) * 32 + (jj & 1) * 8); };
#pragma unroll
        for (int jj = 0; jj < 4; ++jj)
          umma_f16_ts_warp(tmem + COL_ACC1, xb + COL_X2 + a_col(jj), HI | (t1_mn + ((jj * 2048) >> 4)), id_acc,
                      (it > 0) || (jj > 0));
        if (DKV) {
#pragma unroll
          for (int jj = 0; jj < 4; ++jj)
            umma_f16_ts_warp(tmem + COL_ACC2, xb + a_col(jj), HI | (t2_mn + ((jj * 2048) >> 4)), id_acc,
                        (it > 0) || (jj > 0));
        }
        // the score products of this tile finished before the row warps could signal pd_ready,
        // so the completion of these MMAs releases the whole stage and the score buffer
        umma_commit_warp(&t_empty[ts]);
        umma_commit_warp(&x_free[s]);
        if (++ts == STAGES) ts = 0;
      }
      if (it == n_it) umma_commit_warp(acc_done);
    }
  } else {
    const int wg = warp >> 2;          // warpgroup = half of a tile's columns
    const int r = threadIdx.x & 127;
    const uint32_t lane_addr = tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16);
    float row_lse = 0.f, row_delta = 0.f;
    bool ok = true;
    if (!DKV) {
      const int q = blk * 128 + r;
      const size_t bh = static_cast<size_t>(b) * p.heads + hy;
      if (q < p.seq) row_lse = p.lse2[bh * p.seq + q];
      // delta of the row from the resident dO and the forward's output: a kernel of its own read both
      // again (268 MB, 45 us at 4 x 4096 x 16). Both groups need it, and add up half of it each.
      ok = wait_all(r_full, 0, p.status);
      if (ok) {
        // group 0 puts Q, group 1 dO where the score products read them, so that these run while delta is added up (3 x 1000 x 16/4,
        // both kernels: 91.6 -> 89.6 us, and 88.6 with delta halved): a row is 64 columns of bf16 pairs
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          uint32_t w[32];
#pragma unroll
          for (int i = 0; i < 8; ++i)
            *reinterpret_cast<uint4*>(w + 4 * i) = *reinterpret_cast<const uint4*>(
                smem + (wg == 0 ? RA_OFF : RB_OFF) + c * 16384 + r * 128 + ((i ^ (r & 7)) << 4));
          tmem_st_32x32b_x32(lane_addr + COL_R + wg * 64 + c * 32, w);
        }
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(r_copied);
        ok = wait_all(o_full, 0, p.status);
      }
      if (ok) {
        // Columns are added as a warp with four of them to a lane adds its lanes up (halves, quarters, ..):
        // dS, and with it the gradients' bf16 roundings, depend on the sum's last bit.
        auto lanes = [&](const int i) -> float2 {   // 16-byte piece i: two lanes' partial sums
          const int off = (i >> 3) * 16384 + r * 128 + (((i & 7) ^ (r & 7)) << 4);
          float x[8], y[8];
          unpack8(ld_shared8(smem + RB_OFF + off), x);
          unpack8(ld_shared8(stage(O_STAGE) + off), y);
          float t[4];   // products of bf16 values are exact
#pragma unroll
          for (int e = 0; e < 4; ++e) t[e] = fmaf(x[2 * e], y[2 * e], x[2 * e + 1] * y[2 * e + 1]);
          return add2(make_float2(t[0], t[2]), make_float2(t[1], t[3]));
        };
        auto half_sum = [&](const int i) { return add2(lanes(i), lanes(i + 8)); };
        auto quarter_sum = [&](const int i) { return add2(half_sum(i), half_sum(i + 4)); };
        // a group adds up half of the pieces and takes the other half from the other group
        float2* const swap = reinterpret_cast<float2*>(smem + VEC_OFF);   // 2 KB, unused by dQ
        const float2 mine = wg == 0 ? add2(quarter_sum(0), quarter_sum(2)) : add2(quarter_sum(1), quarter_sum(3));
        swap[threadIdx.x] = mine;
      }
      ok = bar_sync_and(3, 256, ok);
      if (ok) {
        const float2* const swap = reinterpret_cast<const float2*>(smem + VEC_OFF);
        const float2 mine = swap[threadIdx.x], theirs = swap[threadIdx.x ^ 128];
        const float2 sum = wg == 0 ? add2(mine, theirs) : add2(theirs, mine);
        row_delta = __fadd_rn(sum.x, sum.y);
        if (q < (p.seq + 63) / 64 * 64) {   // rows past seq have zeros in all four
          float* v = p.vec + (bh * ((p.seq + 63) / 64) + (q >> 6)) * 128 + ((q & 63) >> 1) * 4 + (q & 1);
          if (wg == 0) v[0] = -row_lse;
          else v[2] = -row_delta;
        }
      }
      fence_proxy_async_smem();   // the producer's next loads go over what was read here
      __syncwarp();
      if (ok && lane == 0) mbar_arrive(r_read);
    }
    const float2 log2_scale = make_float2(p.scale_log2, p.scale_log2), lin_scale = make_float2(p.scale, p.scale);
    // P and dS of two neighbouring columns of a row: nl, nd are the columns' (or the row's) -lse2 and -delta
    auto grad2 = [&](const uint32_t xa, const uint32_t xc, const uint32_t da, const uint32_t dc, const float2 nl,
                     const float2 nd, const bool mask_x, const bool mask_y, uint32_t& pk_p, uint32_t& pk_d) {
      const float2 e = fma2(make_float2(__uint_as_float(xa), __uint_as_float(xc)), log2_scale, nl);
      float2 pr = make_float2(ex2(e.x), ex2(e.y));
      if (mask_x) pr.x = 0.f;
      if (mask_y) pr.y = 0.f;
      const float2 dp = make_float2(__uint_as_float(da), __uint_as_float(dc));
      const float2 ds = mul2(pr, mul2(add2(dp, nd), lin_scale));   // the scale before the one rounding to bf16
      pk_d = pack_bf16x2(ds.x, ds.y);
      if (DKV) pk_p = pack_bf16x2(pr.x, pr.y);
    };
    int ts = 0, t = t_first;
    uint32_t t_ph = 0;
    for (int it = 0; it < n_it; ++it) {
      const int s = it & 1;
      // mask: dQ rows are queries, columns keys (key > query is masked);
      //       dKV rows are keys, columns queries (query < key is masked)
      const int tg = DKV ? t + q_off64 : t;     // global index of the streamed tile
      const bool edge = DKV ? (tg * 64 < gblk * 128 + 127) : (tg * 64 + 63 > gblk * 128);
      const uint32_t xb = lane_addr + s * 128 + wg * 32;
      const int col0 = tg * 64 + wg * 32;
      ok = ok && (!DKV || wait_all(&t_full[ts], t_ph, p.status)) && wait_all(&x_done[s], (it >> 1) & 1, p.status);
      if (!ok) break;
      tc_fence_after();
      if constexpr (DKV) {
        // Fragments of 16 rows x 8 columns: a lane has two neighbouring columns of eight, in rows lane / 4 and
        // lane / 4 + 8, so it needs the log-sum-exp and delta of 8 of its group's 32 columns, not of all: a
        // shared-memory read that all lanes share costs as much as one of 32 different words.
        uint32_t x1[2][16], x2[2][16], pk_p[2][8], pk_d[2][8];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          tmem_ld_16x256b_x4(xb + (static_cast<uint32_t>(16 * h) << 16), x1[h]);
          tmem_ld_16x256b_x4(xb + COL_X2 + (static_cast<uint32_t>(16 * h) << 16), x2[h]);
        }
        float4 v[4];   // -lse2 and -delta of the lane's columns
#pragma unroll
        for (int j = 0; j < 4; ++j)
          v[j] = *reinterpret_cast<const float4*>(smem + VEC_OFF + ts * 512 + (wg * 16 + j * 4 + (lane & 3)) * 16);
        tmem_ld_wait();
#pragma unroll
        for (int h = 0; h < 2; ++h) { tie16(x1[h]); tie16(x2[h]); }
        auto rows = [&](auto EDGE) {
#pragma unroll
          for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
              for (int u = 0; u < 2; ++u) {
                const int at = 4 * j + 2 * u, pos = gblk * 128 + (warp & 3) * 32 + h * 16 + u * 8 + (lane >> 2);
                const int q = col0 + 8 * j + 2 * (lane & 3);
                grad2(x1[h][at], x1[h][at + 1], x2[h][at], x2[h][at + 1], make_float2(v[j].x, v[j].y),
                      make_float2(v[j].z, v[j].w), decltype(EDGE)::value && q < pos,
                      decltype(EDGE)::value && q + 1 < pos, pk_p[h][2 * j + u], pk_d[h][2 * j + u]);
              }
        };
        if (edge) rows(std::true_type{});
        else rows(std::false_type{});
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          tmem_st_16x128b_x4(xb + (static_cast<uint32_t>(16 * h) << 16), pk_p[h]);
          tmem_st_16x128b_x4(xb + COL_X2 + (static_cast<uint32_t>(16 * h) << 16), pk_d[h]);
        }
      } else {
        uint32_t x1[32], x2[32], pk_d[16], none;
        tmem_ld_32x32b_x32(xb, x1);
        tmem_ld_32x32b_x32(xb + COL_X2, x2);
        tmem_ld_wait();
        tie32(x1);
        tie32(x2);
        const float2 nl = make_float2(-row_lse, -row_lse), nd = make_float2(-row_delta, -row_delta);
        const int pos = gblk * 128 + r;
        auto rows = [&](auto EDGE) {
#pragma unroll
          for (int i = 0; i < 16; ++i)
            grad2(x1[2 * i], x1[2 * i + 1], x2[2 * i], x2[2 * i + 1], nl, nd,
                  decltype(EDGE)::value && col0 + 2 * i > pos, decltype(EDGE)::value && col0 + 2 * i + 1 > pos, none,
                  pk_d[i]);
        };
        if (edge) rows(std::true_type{});
        else rows(std::false_type{});
        tmem_st_32x32b_x16(xb + COL_X2, pk_d);
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&pd_ready[s]);
      if (++ts == STAGES) { ts = 0; t_ph ^= 1; }
      if (++t == t_first + t_count) t = t_first;   // dKV: the next head of the group
    }
    // every row warp gets here, also one that gave up, so the group barrier below is safe
    ok = wait_all(acc_done, 0, p.status) && ok;
    // resident tiles are no longer read: reuse them as the staging for the TMA stores.
    // dKV: group 0 drains dK, group 1 drains dV.  dQ: each group drains 64 columns.
    uint8_t* out = smem + ((DKV && wg == 1) ? RB_OFF : RA_OFF);
    if (ok) {
      tc_fence_after();
      const uint32_t col0 = (DKV && wg == 1) ? COL_ACC2 : COL_ACC1;
      const int c_lo = DKV ? 0 : wg * 64, c_hi = DKV ? D : wg * 64 + 64;
#pragma unroll 1
      for (int c = c_lo; c < c_hi; c += 32) {
        uint32_t v[32];
        tmem_ld_32x32b_x32(lane_addr + col0 + c, v);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          float f[8];
#pragma unroll
          // a key block with no local query at or after it gets an all-zero gradient
          for (int k = 0; k < 8; ++k) f[k] = n_it > 0 ? __uint_as_float(v[8 * i + k]) : 0.f;
          const int col = c + 8 * i;
          st_swz(out + (col >> 6) * 16384, r, (col & 63) >> 3, pack_bf16x8(f));
        }
      }
      fence_proxy_async_smem();
    }
    if (bar_sync_and(1 + wg, 128, ok) && r == 0) {
      const int ox = (DKV ? g : hy) * D;
      if (DKV) {
        const CUtensorMap* tm = wg == 0 ? &tmO1 : &tmO2;
        tma_store_3d(tm, out, ox, row0, b);
        tma_store_3d(tm, out + 16384, ox + 64, row0, b);
      } else {
        tma_store_3d(&tmO1, out + wg * 16384, ox + wg * 64, row0, b);
      }
      tma_store_commit();
      tma_store_wait<0>();
    }
  }

  tc_fence_before();
  __syncthreads();
  if (p.status != nullptr && *reinterpret_cast<volatile int*>(p.status) != PB_OK) {
    for (int i = 0; i < 2000; ++i) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == 8) {
    tc_fence_after();
    tmem_dealloc(tmem, TMEM_COLS);
  }
}
}  // namespace bwd

// map of a token-major tensor [batch, seq, ld], 64-column boxes of box_rows rows of one batch entry
static int tok_map(CUtensorMap* tm, const void* base, uint64_t inner, int seq, int batch, int ld, int box_rows) {
  return make_tmap_3d(tm, base, 2, inner, seq, batch, ld, static_cast<uint64_t>(seq) * ld, 64, box_rows);
}

// CTAs of a grid of row blocks x heads x batch entries; more than a grid dimension holds is refused (-1)
static long grid_ctas(int rows, int block, int heads, int batch) {
  const long per = static_cast<long>(heads) * batch;
  const long blocks = (static_cast<long>(rows) + block - 1) / block;
  return per > INT_MAX || blocks > INT_MAX / per ? -1 : blocks * per;
}

static bool bad_geometry(int batch, int seq, int heads, int kv_heads, int ldq, int ldkv) {
  return batch <= 0 || seq <= 0 || heads <= 0 || kv_heads <= 0 ||
         heads % kv_heads != 0 || ldq < heads * D || ldkv < kv_heads * D || ldq % 8 != 0 ||
         ldkv % 8 != 0;
}

}  // namespace attn
}  // namespace pb

using namespace pb;

// out = softmax(scale * Q K^T + causal mask) V.  q/out: [batch * seq, ldq / ldo] bf16 with head h
// at columns [128 h, 128 h + 128); k/v: [batch * seq_kv, ldkv] with KV head g likewise.
// Query row i of a batch entry sits at global position q_off + i and sees keys 0 .. q_off + i
// (q_off = 0 and seq_kv = seq is ordinary causal attention; a context-parallel rank passes its
// slice of the queries, the gathered keys and its offset). q_off a multiple of 256, seq_kv >= q_off + seq.
// lse2: fp32 [batch, heads, seq], log2 of the softmax denominator plus the applied maximum.
// rowmax (optional): fp32 [batch, heads, seq], the largest scaled logit of each row.
PB_API int pb_attn_fwd_cp(const void* q, const void* k, const void* v, void* out, void* lse2,
                          void* rowmax, int batch, int seq, int seq_kv, int q_off, int heads,
                          int kv_heads, int ldq, int ldkv, int ldo, float scale, int* status,
                          cudaStream_t st) {
  using namespace attn;
  if (bad_geometry(batch, seq, heads, kv_heads, ldq, ldkv) || ldo < heads * D || ldo % 8 != 0 ||
      !(scale > 0.f) || q_off < 0 || q_off % 256 != 0 || seq_kv < q_off + seq)
    return PB_BAD_ARG;
  const long grid = grid_ctas(seq, 256, heads, batch);
  if (grid < 0) return PB_BAD_ARG;
  static pb::DeviceOnce attr_once;   // per device: the attribute belongs to the current GPU
  if (attr_once.need()) {
    cudaError_t e = cudaFuncSetAttribute(fwd::attn_fwd_kernel,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, fwd::SMEM);
    if (e != cudaSuccess) return static_cast<int>(e);
    attr_once.done();
  }
  CUtensorMap tQ, tK, tV, tO;
  int r = 0;
  r |= tok_map(&tQ, q, static_cast<uint64_t>(heads) * D, seq, batch, ldq, 128);
  r |= tok_map(&tK, k, static_cast<uint64_t>(kv_heads) * D, seq_kv, batch, ldkv, 64);
  r |= tok_map(&tV, v, static_cast<uint64_t>(kv_heads) * D, seq_kv, batch, ldkv, 64);
  r |= tok_map(&tO, out, static_cast<uint64_t>(heads) * D, seq, batch, ldo, 128);
  if (r != 0) return 1000 + r;
  fwd::Params p;
  p.batch = batch; p.seq = seq; p.heads = heads; p.kv_heads = kv_heads;
  p.seq_kv = seq_kv; p.q_off = q_off;
  p.scale_log2 = scale * 1.4426950408889634f;
  p.lse2 = static_cast<float*>(lse2);
  p.rowmax = static_cast<float*>(rowmax);
  p.status = status;
  pb::launch(fwd::attn_fwd_kernel, static_cast<unsigned>(grid), 352, fwd::SMEM, st, tQ, tK, tV, tO, p);
  return static_cast<int>(cudaGetLastError());
}

PB_API int pb_attn_fwd(const void* q, const void* k, const void* v, void* out, void* lse2,
                       void* rowmax, int batch, int seq, int heads, int kv_heads, int ldq, int ldkv,
                       int ldo, float scale, int* status, cudaStream_t st) {
  return pb_attn_fwd_cp(q, k, v, out, lse2, rowmax, batch, seq, seq, 0, heads, kv_heads, ldq, ldkv,
                        ldo, scale, status, st);
}

// Gradients of pb_attn_fwd_cp. delta: fp32 scratch [batch, heads, ceil(seq / 64), 128] (written here), 16-byte aligned.
// dq: [batch * seq, ldq]; dk, dv: [batch * seq_kv, ldkv] (all bf16, fully overwritten; key rows
// that no local query sees get zeros).
PB_API int pb_attn_bwd_cp(const void* q, const void* k, const void* v, const void* out,
                          const void* dout, const void* lse2, void* delta, void* dq, void* dk,
                          void* dv, int batch, int seq, int seq_kv, int q_off, int heads,
                          int kv_heads, int ldq, int ldkv, int ldo, float scale, int* status,
                          cudaStream_t st) {
  using namespace attn;
  if (bad_geometry(batch, seq, heads, kv_heads, ldq, ldkv) || ldo < heads * D || ldo % 8 != 0 ||
      !(scale > 0.f) || q_off < 0 || q_off % 128 != 0 || seq_kv < q_off + seq ||
      (reinterpret_cast<uintptr_t>(delta) & 15) != 0)
    return PB_BAD_ARG;
  const long grid_q = grid_ctas(seq, 128, heads, batch), grid_kv = grid_ctas(seq_kv, 128, kv_heads, batch);
  if (grid_q < 0 || grid_kv < 0) return PB_BAD_ARG;
  static pb::DeviceOnce attr_once;   // per device: the attribute belongs to the current GPU
  if (attr_once.need()) {
    cudaError_t e = cudaFuncSetAttribute(bwd::attn_bwd_kernel<false>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, bwd::SMEM);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(bwd::attn_bwd_kernel<true>,
                               cudaFuncAttributeMaxDynamicSharedMemorySize, bwd::SMEM);
    if (e != cudaSuccess) return static_cast<int>(e);
    attr_once.done();
  }
  const uint64_t qi = static_cast<uint64_t>(heads) * D, ki = static_cast<uint64_t>(kv_heads) * D;
  bwd::Params p;
  p.batch = batch; p.seq = seq; p.heads = heads; p.kv_heads = kv_heads;
  p.seq_kv = seq_kv; p.q_off = q_off;
  p.scale = scale; p.scale_log2 = scale * 1.4426950408889634f;
  p.lse2 = static_cast<const float*>(lse2);
  p.vec = static_cast<float*>(delta);
  p.status = status;
  int r = 0;
  {
    // dQ: resident Q, dO (128-row boxes); streamed K, V (64-row boxes)
    CUtensorMap tQ, tDO, tK, tV, tDQ, tO;
    r |= tok_map(&tO, out, qi, seq, batch, ldo, 128);
    r |= tok_map(&tQ, q, qi, seq, batch, ldq, 128);
    r |= tok_map(&tDO, dout, qi, seq, batch, ldo, 128);
    r |= tok_map(&tK, k, ki, seq_kv, batch, ldkv, 64);
    r |= tok_map(&tV, v, ki, seq_kv, batch, ldkv, 64);
    r |= tok_map(&tDQ, dq, qi, seq, batch, ldq, 128);
    if (r != 0) return 1000 + r;
    p.n_blk = (seq + 127) / 128;
    pb::launch(bwd::attn_bwd_kernel<false>, static_cast<unsigned>(grid_q), 384, bwd::SMEM, st,
        tQ, tDO, tK, tV, tDQ, tDQ, tO, p);
  }
  {
    // dK, dV: resident K, V (every key block of the gathered keys); streamed local Q, dO
    CUtensorMap tK, tV, tQ, tDO, tDK, tDV;
    r |= tok_map(&tK, k, ki, seq_kv, batch, ldkv, 128);
    r |= tok_map(&tV, v, ki, seq_kv, batch, ldkv, 128);
    r |= tok_map(&tQ, q, qi, seq, batch, ldq, 64);
    r |= tok_map(&tDO, dout, qi, seq, batch, ldo, 64);
    r |= tok_map(&tDK, dk, ki, seq_kv, batch, ldkv, 128);
    r |= tok_map(&tDV, dv, ki, seq_kv, batch, ldkv, 128);
    if (r != 0) return 2000 + r;
    p.n_blk = (seq_kv + 127) / 128;
    pb::launch(bwd::attn_bwd_kernel<true>, static_cast<unsigned>(grid_kv), 384, bwd::SMEM, st,
        tK, tV, tQ, tDO, tDK, tDV, tK, p);
  }
  return static_cast<int>(cudaGetLastError());
}

PB_API int pb_attn_bwd(const void* q, const void* k, const void* v, const void* out,
                       const void* dout, const void* lse2, void* delta, void* dq, void* dk,
                       void* dv, int batch, int seq, int heads, int kv_heads, int ldq, int ldkv,
                       int ldo, float scale, int* status, cudaStream_t st) {
  return pb_attn_bwd_cp(q, k, v, out, dout, lse2, delta, dq, dk, dv, batch, seq, seq, 0, heads,
                        kv_heads, ldq, ldkv, ldo, scale, status, st);
}

#ifdef PB_ATTN_PROF
PB_API int pb_attn_prof_read(unsigned long long* out8, int reset) {
  cudaError_t e = cudaMemcpyFromSymbol(out8, attn::g_attn_prof, sizeof(unsigned long long) * 8);
  if (e == cudaSuccess && reset) {
    unsigned long long z[8] = {};
    e = cudaMemcpyToSymbol(attn::g_attn_prof, z, sizeof z);
  }
  return static_cast<int>(e);
}
#endif
