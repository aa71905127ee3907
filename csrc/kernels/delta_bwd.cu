// Backward of the delta rule's chunk-local part in one kernel on tcgen05 (sm_100a): from what the state walks left
// (-dU, U, the bf16 states S entering and the state gradients dS' leaving every chunk of 64 tokens) and the inputs to
// dq, dk, dv and dbeta.
//
//   dW = (-dU) S^T      dM = tril(dO U^T)      dQ = dO S^T + dM K      dV = -(A'^T (-dU))
//   dA' = dW K^T - (-dU) V^T                   X = dA' A'^T            dA = -T^T X
//   dG = diag(beta) tril(dA, -1)               dK = U dS'^T + A'^T dW + (dG + dG^T) K + dM^T Q
//   dbeta_i = (dA'^T T)_ii + sum_{j<i} dA_ij (K K^T)_ij
//
// Bound by memory: 176 KB in and 48 KB out a chunk. As two kernels (delta_chunk.cu and the backward in delta_prep.cu,
// which stay as the parts that the tests check one by one) dW, dM and the two state products crossed memory in between,
// 112 KB a chunk more, and the latter two were rounded to bf16 on the way; here they stay in their accumulators. 4096
// chunks: 256 us as two kernels, 178 as one: 917 MB at 5.2 TB/s. What is left is the chain: about 9500 of a chunk's 10400
// clocks, with one chunk in flight in the 200 KB that its tiles take.
//
// One persistent CTA per SM. A chunk is a chain of products and conversions, so what does not depend on the chain is
// taken out of it: the next chunk's S, dS', dO, U and -dU arrive in a region of their own while this one is worked on,
// its dW and dM are multiplied during this chunk's last products, and the state products of dQ and dK run
// beside the conversion of dW.
//   warp 2: TMA producer   warp 3: MMA issue
//   warps 0, 1, 4, 5, 8, 9, 12, 13: rows 0..31 and 32..63 of the accumulators (a warp reads the tensor-memory lanes of its
//   quarter; the 64-row operands run as 128-row ones, whose upper rows are never read), a quarter of the columns each
//
// Reference semantics: kernels/__init__.py:357-376 of the reference (the recurrence this is a
// backward of); the chunked algebra and this kernel are this library's own.
#include <cuda.h>

#include "common.cuh"

namespace pb {

int make_tmap_3d(CUtensorMap* tm, const void* base, int elem_bytes, uint64_t inner,
                 uint64_t outer, uint64_t batch, uint64_t ld_elems, uint64_t batch_stride_elems,
                 uint32_t box_inner, uint32_t box_outer);
int num_sms();

namespace dbwd {

constexpr int C = 64, D = 128;
// what the walks left, prefetched a chunk ahead; then this chunk's operands, intermediates and results. A tile that is an
// A operand is read up to 16 KB past its start's last 8 KB: the results' staging lies behind all of them.
constexpr int NDU = 0, DO = 16384, UT = 32768, ST = 49152, DS = 81920;
constexpr int KT = 114688, VQ = 131072, DW = 147456, AP = 163840, TT = 172032, DM = 180224, TMP = 188416;
constexpr int OUTK = 196608, OUTV = 212992, BARS = 229376, SMEM = BARS + 256 + 1024;
static_assert(SMEM <= 227 * 1024, "one CTA's shared memory");
static_assert(TMP + 16384 <= OUTV, "A operands stay in bounds");
constexpr int THREADS = 448, ROW_WARPS = 8;
constexpr uint32_t COL_Q = 0, COL_K = 128, COL_W = 256, COL_A = 384, COL_B = 448, TMEM_COLS = 512;

struct Params {
  int n_chunks, heads, seq_len, total;   // chunks per sequence; chunk g = (b * heads + h) * n_chunks + n
  const void* beta;    // [batch, seq, heads]
  void* dbeta;         // like beta
  int beta_f32;
  int* status;
};

// Registers of tensor-memory loads are valid after the wait: no use of them may move above it.
template <int N>
__device__ __forceinline__ void tie(float (&f)[N]) {
#pragma unroll
  for (int i = 0; i < N; i += 8)
    asm volatile("" : "+f"(f[i]), "+f"(f[i + 1]), "+f"(f[i + 2]), "+f"(f[i + 3]), "+f"(f[i + 4]), "+f"(f[i + 5]),
                      "+f"(f[i + 6]), "+f"(f[i + 7]));
}
__device__ __forceinline__ void put8(uint8_t* tile, int row, int col, const float* f) {
  st_shared8(tile + (col >> 6) * 8192 + row * 128 + ((((col & 63) >> 3) ^ (row & 7)) << 4), pack8(f));
}

__global__ void __launch_bounds__(THREADS, 1)
delta_bwd_kernel(const __grid_constant__ CUtensorMap tmNDU, const __grid_constant__ CUtensorMap tmDO,
                 const __grid_constant__ CUtensorMap tmU, const __grid_constant__ CUtensorMap tmS,
                 const __grid_constant__ CUtensorMap tmDS, const __grid_constant__ CUtensorMap tmK,
                 const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmQ,
                 const __grid_constant__ CUtensorMap tmAP, const __grid_constant__ CUtensorMap tmT,
                 const __grid_constant__ CUtensorMap tmDQ, const __grid_constant__ CUtensorMap tmDK,
                 const __grid_constant__ CUtensorMap tmDV, const Params p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + BARS);
  // every barrier completes once a chunk, so the chunk's number picks the parity
  uint64_t* full0 = bars;        // -dU, dO, U, S, dS'
  uint64_t* full1 = bars + 1;    // K, V, A', T
  uint64_t* fullq = bars + 2;    // Q, in V's place
  uint64_t* states = bars + 3;   // the products of S, dS', dO and U are complete
  uint64_t* m0 = bars + 4;       // dW and dM
  uint64_t* m1 = bars + 5;       // dW K^T, (-dU) V^T
  uint64_t* mv = bars + 6;       // A'^T (-dU)
  uint64_t* m2 = bars + 7;       // X
  uint64_t* m3 = bars + 8;       // T^T X, dA'^T T, K K^T
  uint64_t* m4 = bars + 9;       // dQ and dK
  uint64_t* c0 = bars + 10;      // dW is an operand tile
  uint64_t* c1 = bars + 11;      // dA' and dM are
  uint64_t* dv_read = bars + 12; // dV's accumulator is in registers
  uint64_t* c2 = bars + 13;      // X is an operand tile
  uint64_t* c3 = bars + 14;      // dG is
  uint64_t* acc_read = bars + 15;  // dQ's and dK's accumulators are in registers
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 16);
  __shared__ float dbeta_part[4][C];

  const int warp = warp_index(), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    mbar_init(full0, 2);
    for (int i = 1; i < 10; ++i) mbar_init(bars + i, 1);
    for (int i = 10; i < 16; ++i) mbar_init(bars + i, ROW_WARPS);
    fence_barrier_init();
    tma_prefetch_desc(&tmNDU); tma_prefetch_desc(&tmDO); tma_prefetch_desc(&tmU); tma_prefetch_desc(&tmS);
    tma_prefetch_desc(&tmDS); tma_prefetch_desc(&tmK); tma_prefetch_desc(&tmV); tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmAP); tma_prefetch_desc(&tmT);
  }
  if (warp == 3) {
    tmem_alloc(tmem_slot, TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  after_previous_kernel();
  const int step = static_cast<int>(gridDim.x);

  if (warp == 2) {
    if (lane == 0) {
      auto place = [&](int g, int& x, int& t, int& b) {
        const int seq = g / p.n_chunks;
        t = (g - seq * p.n_chunks) * C;
        b = seq / p.heads;
        x = (seq - b * p.heads) * D;
      };
      auto load_q = [&](int g) {
        int x, t, b;
        place(g, x, t, b);
        mbar_arrive_expect_tx(fullq, 16384);
        tma_load_3d(smem + VQ, &tmQ, fullq, x, t, b);
        tma_load_3d(smem + VQ + 8192, &tmQ, fullq, x + 64, t, b);
      };
      uint32_t ph = 1;      // parity of the chunk before
      bool ok = true;
      int g = blockIdx.x;
      for (; g < p.total; g += step, ph ^= 1) {
        const bool first = g == static_cast<int>(blockIdx.x);
        int x, t, b;
        place(g, x, t, b);
        if (!first && !(ok = mbar_wait(states, ph, p.status))) break;
        mbar_arrive_expect_tx(full0, 2 * 32768 + 2 * 16384);
        for (int hf = 0; hf < 2; ++hf) {
          tma_load_3d(smem + ST + hf * 16384, &tmS, full0, hf * 64, g * D, 0);
          tma_load_3d(smem + DO + hf * 8192, &tmDO, full0, x + hf * 64, t, b);
          tma_load_3d(smem + UT + hf * 8192, &tmU, full0, hf * 64, g * C, 0);
          tma_load_3d(smem + DS + hf * 16384, &tmDS, full0, hf * 64, g * D, 0);
        }
        if (!first) {
          if (!(ok = mbar_wait(mv, ph, p.status))) break;
          load_q(g - step);
        }
        mbar_arrive_expect_tx(full0, 16384);
        tma_load_3d(smem + NDU, &tmNDU, full0, 0, g * C, 0);
        tma_load_3d(smem + NDU + 8192, &tmNDU, full0, 64, g * C, 0);
        if (!first && !(ok = mbar_wait(m4, ph, p.status))) break;
        mbar_arrive_expect_tx(full1, 2 * 16384 + 2 * 8192);
        tma_load_3d(smem + KT, &tmK, full1, x, t, b);
        tma_load_3d(smem + KT + 8192, &tmK, full1, x + 64, t, b);
        tma_load_3d(smem + VQ, &tmV, full1, x, t, b);
        tma_load_3d(smem + VQ + 8192, &tmV, full1, x + 64, t, b);
        tma_load_3d(smem + AP, &tmAP, full1, 0, g * C, 0);
        tma_load_3d(smem + TT, &tmT, full1, 0, g * C, 0);
      }
      if (ok && mbar_wait(mv, ph, p.status)) load_q(g - step);   // the last chunk's (the grid is at most the chunks)
    }
  } else if (warp == 3) {
    {
      const uint32_t id_kk = make_idesc(1, 1, 128, 128, 0, 0), id_kk64 = make_idesc(1, 1, 128, 64, 0, 0);
      const uint32_t id_mm = make_idesc(1, 1, 128, 128, 1, 1), id_mm64 = make_idesc(1, 1, 128, 64, 1, 1);
      const uint32_t id_kn = make_idesc(1, 1, 128, 128, 0, 1);
      const uint32_t base_k = sdesc_lo(smem_u32(smem), 16), base_mn = sdesc_lo(smem_u32(smem), 8192);
      auto kk = [&](int tile, int j) { return step_k(base_k + (tile >> 4), j); };
      auto mn = [&](int tile, int j) { return step_mn(base_mn + (tile >> 4), j); };
      // a [128, 128] tile is two halves of 16 KB
      auto kk128 = [&](int tile, int j) { return base_k + ((tile + (j >> 2) * 16384 + (j & 3) * 32) >> 4); };
      auto first_products = [&] {
#pragma unroll
        for (int j = 0; j < 8; ++j) umma_f16_lo_warp(tmem + COL_W, kk(NDU, j), kk128(ST, j), id_kk, j > 0);
#pragma unroll
        for (int j = 0; j < 8; ++j) umma_f16_lo_warp(tmem + COL_A, kk(DO, j), kk(UT, j), id_kk64, j > 0);
        umma_commit_warp(m0);
      };
      uint32_t ph = 0;
      if (static_cast<int>(blockIdx.x) < p.total && mbar_wait_spin_warp(full0, 0, p.status)) {
        tc_fence_after();
        first_products();
        for (int g = blockIdx.x; g < p.total; g += step, ph ^= 1) {
          if (!mbar_wait_spin_warp(acc_read, ph ^ 1, p.status)) break;
          tc_fence_after();
#pragma unroll
          for (int j = 0; j < 8; ++j) umma_f16_lo_warp(tmem + COL_Q, kk(DO, j), kk128(ST, j), id_kk, j > 0);
#pragma unroll
          for (int j = 0; j < 8; ++j) umma_f16_lo_warp(tmem + COL_K, kk(UT, j), kk128(DS, j), id_kk, j > 0);
          umma_commit_warp(states);
          if (!mbar_wait_spin_warp(full1, ph, p.status)) break;
          tc_fence_after();
#pragma unroll
          for (int j = 0; j < 8; ++j) umma_f16_lo_warp(tmem + COL_B, kk(NDU, j), kk(VQ, j), id_kk64, j > 0);
          if (!mbar_wait_spin_warp(c0, ph, p.status)) break;
          tc_fence_after();
#pragma unroll
          for (int j = 0; j < 8; ++j) umma_f16_lo_warp(tmem + COL_A, kk(DW, j), kk(KT, j), id_kk64, j > 0);
          umma_commit_warp(m1);
#pragma unroll
          for (int j = 0; j < 4; ++j) umma_f16_lo_warp(tmem + COL_W, mn(AP, j), mn(NDU, j), id_mm, j > 0);
          umma_commit_warp(mv);
          if (!mbar_wait_spin_warp(c1, ph, p.status)) break;
          tc_fence_after();
#pragma unroll
          for (int j = 0; j < 4; ++j) umma_f16_lo_warp(tmem + COL_A, kk(TMP, j), kk(AP, j), id_kk64, j > 0);
          umma_commit_warp(m2);
#pragma unroll
          for (int j = 0; j < 4; ++j) umma_f16_lo_warp(tmem + COL_B, mn(TMP, j), mn(TT, j), id_mm64, j > 0);
#pragma unroll
          for (int j = 0; j < 4; ++j) umma_f16_lo_warp(tmem + COL_K, mn(AP, j), mn(DW, j), id_mm, 1);
          if (!mbar_wait_spin_warp(dv_read, ph, p.status)) break;
          tc_fence_after();
#pragma unroll
          for (int j = 0; j < 8; ++j) umma_f16_lo_warp(tmem + COL_W, kk(KT, j), kk(KT, j), id_kk64, j > 0);
          if (!mbar_wait_spin_warp(c2, ph, p.status)) break;
          tc_fence_after();
#pragma unroll
          for (int j = 0; j < 4; ++j) umma_f16_lo_warp(tmem + COL_A, mn(TT, j), mn(OUTK, j), id_mm64, j > 0);
          umma_commit_warp(m3);
          if (!mbar_wait_spin_warp(fullq, ph, p.status) || !mbar_wait_spin_warp(c3, ph, p.status)) break;
          tc_fence_after();
#pragma unroll
          for (int j = 0; j < 4; ++j) umma_f16_lo_warp(tmem + COL_K, kk(TMP, j), mn(KT, j), id_kn, 1);
#pragma unroll
          for (int j = 0; j < 4; ++j) umma_f16_lo_warp(tmem + COL_K, mn(TMP, j), mn(KT, j), id_mm, 1);
#pragma unroll
          for (int j = 0; j < 4; ++j) umma_f16_lo_warp(tmem + COL_K, mn(DM, j), mn(VQ, j), id_mm, 1);
#pragma unroll
          for (int j = 0; j < 4; ++j) umma_f16_lo_warp(tmem + COL_Q, kk(DM, j), mn(KT, j), id_kn, 1);
          umma_commit_warp(m4);
          if (g + step < p.total) {
            // the next chunk's dW and dM: the row warps have read what those columns held
            if (!mbar_wait_spin_warp(full0, ph ^ 1, p.status)) break;
            tc_fence_after();
            first_products();
          }
        }
      }
    }
  } else if ((warp & 3) < 2) {
    const int cg = warp >> 2;                        // quarter of the columns
    const int r = (warp & 1) * 32 + lane;            // token row = tensor-memory lane
    const uint32_t taddr = tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16);
    const bool lead = threadIdx.x == 0;              // issues and tracks the bulk stores
    const int c16 = cg * 16, c32 = cg * 32;
    bool ok = true;
    auto wait = [&](uint64_t* bar, uint32_t parity) {
      ok = ok && mbar_wait_spin_warp(bar, parity, p.status);
      tc_fence_after();
    };
    auto arrive = [&](uint64_t* bar) {   // the warp's shared-memory writes and tensor-memory reads are done
      fence_proxy_async_smem();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar);
    };
    auto ask16 = [&](uint32_t col, float (&f)[16]) { tmem_ld_32x32b_x16(taddr + col, reinterpret_cast<uint32_t*>(f)); };
    auto ask32 = [&](uint32_t col, float (&f)[32]) { tmem_ld_32x32b_x32(taddr + col, reinterpret_cast<uint32_t*>(f)); };
    auto store32 = [&](uint8_t* tile, const float (&f)[32]) {
#pragma unroll
      for (int i = 0; i < 4; ++i) put8(tile, r, c32 + 8 * i, f + 8 * i);
    };
    auto load_beta = [&](int g) {
      const int seq = g / p.n_chunks, t = (g - seq * p.n_chunks) * C + r;
      const int b = seq / p.heads, h = seq - b * p.heads;
      if (g >= p.total || t >= p.seq_len) return 0.f;
      const size_t i = (static_cast<size_t>(b) * p.seq_len + t) * p.heads + h;
      return p.beta_f32 ? static_cast<const float*>(p.beta)[i] : bf16_to_f32(static_cast<const bf16*>(p.beta)[i]);
    };
    float beta_next = load_beta(blockIdx.x);
    uint32_t ph = 0;
    for (int g = blockIdx.x; g < p.total; g += step, ph ^= 1) {
      const float beta = beta_next;
      beta_next = load_beta(g + step);   // a chunk ahead: the load takes over 1000 clocks
      const int seq = g / p.n_chunks, n = g - seq * p.n_chunks;
      const int b = seq / p.heads, h = seq - b * p.heads;
      const int t0 = n * C, x0 = h * D;
      const bool valid = t0 + r < p.seq_len;
      const size_t bidx = (static_cast<size_t>(b) * p.seq_len + t0 + r) * p.heads + h;
      // ---- dW and tril(dM) -> operand tiles (what the chunk before had there is consumed: m4) ----
      wait(m0, ph);
      if (ok) {
        float f[32], m[16];
        ask32(COL_W + c32, f);
        ask16(COL_A + c16, m);
        tmem_ld_wait();
        tie(f);
        tie(m);
        store32(smem + DW, f);
        arrive(c0);
#pragma unroll
        for (int i = 0; i < 16; ++i) m[i] = c16 + i <= r ? m[i] : 0.f;
        put8(smem + DM, r, c16, m);
        put8(smem + DM, r, c16 + 8, m + 8);
        if (lead) tma_store_wait_read<0>();   // dq and dk of the chunk before have left the staging
      }
      // ---- dA' -> operand tile; dV ----
      wait(m1, ph);
      if (ok) {
        float a[16], s[16];
        ask16(COL_A + c16, a);
        ask16(COL_B + c16, s);
        tmem_ld_wait();
        tie(a);
        tie(s);
#pragma unroll
        for (int i = 0; i < 16; ++i) a[i] -= s[i];
        put8(smem + TMP, r, c16, a);
        put8(smem + TMP, r, c16 + 8, a + 8);
        arrive(c1);
      }
      // ---- X -> operand tile; dV meanwhile ----
      float dv[32];
      wait(mv, ph);
      if (ok) {
        ask32(COL_W + c32, dv);
        tmem_ld_wait();
        tie(dv);
        arrive(dv_read);
      }
      wait(m2, ph);
      if (ok) {
        float x[16];
        ask16(COL_A + c16, x);
        tmem_ld_wait();
        tie(x);
        put8(smem + OUTK, r, c16, x);       // dA'^T T may still be reading dA'; dk's staging is empty until the end
        put8(smem + OUTK, r, c16 + 8, x + 8);
        arrive(c2);
#pragma unroll
        for (int i = 0; i < 32; ++i) dv[i] = -dv[i];
        store32(smem + OUTV, dv);
        fence_proxy_async_smem();
      }
      ok = bar_sync_and(1, ROW_WARPS * 32, ok);
      if (!ok) break;
      if (lead) {
        tma_store_3d(&tmDV, smem + OUTV, x0, t0, b);
        tma_store_3d(&tmDV, smem + OUTV + 8192, x0 + 64, t0, b);
        tma_store_commit();
      }
      // ---- dG -> operand tile; dbeta ----
      wait(m3, ph);
      if (ok) {
        float na[16], gk[16], y[16], dbeta = 0.f;
        const int below = r - c16;
        ask16(COL_A + c16, na);
        ask16(COL_W + c16, gk);
        ask16(COL_B + c16, y);
        tmem_ld_wait();
        tie(na);
        tie(gk);
        tie(y);
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const bool low = i < below;
          if (low) dbeta = fmaf(-na[i], gk[i], dbeta);
          if (i == below) dbeta += y[i];
          na[i] = low ? -beta * na[i] : 0.f;
        }
        put8(smem + TMP, r, c16, na);
        put8(smem + TMP, r, c16 + 8, na + 8);
        dbeta_part[cg][r] = dbeta;
        if (lead) tma_store_wait_read<0>();   // dV has left the staging that dq takes
        arrive(c3);
      }
      // ---- dq, dk ----
      wait(m4, ph);
      if (ok) {
        float f[32], k[32];
        ask32(COL_Q + c32, f);
        ask32(COL_K + c32, k);
        tmem_ld_wait();
        tie(f);
        tie(k);
        arrive(acc_read);
        store32(smem + OUTV, f);
        store32(smem + OUTK, k);
        fence_proxy_async_smem();
      }
      ok = bar_sync_and(1, ROW_WARPS * 32, ok);
      if (!ok) break;
      if (lead) {
        tma_store_3d(&tmDQ, smem + OUTV, x0, t0, b);
        tma_store_3d(&tmDQ, smem + OUTV + 8192, x0 + 64, t0, b);
        tma_store_3d(&tmDK, smem + OUTK, x0, t0, b);
        tma_store_3d(&tmDK, smem + OUTK + 8192, x0 + 64, t0, b);
        tma_store_commit();
      }
      if (valid && cg == 0) {
        const float db = (dbeta_part[0][r] + dbeta_part[1][r]) + (dbeta_part[2][r] + dbeta_part[3][r]);
        if (p.beta_f32) static_cast<float*>(p.dbeta)[bidx] = db;
        else static_cast<bf16*>(p.dbeta)[bidx] = f32_to_bf16(db);
      }
    }
    if (lead) tma_store_wait<0>();
  }

  tc_fence_before();
  __syncthreads();
  if (p.status != nullptr && *reinterpret_cast<volatile int*>(p.status) != PB_OK) {
    for (int i = 0; i < 2000; ++i) __nanosleep(1000);  // let copies in flight land
    __syncthreads();
  }
  if (warp == 3) {
    tc_fence_after();
    tmem_dealloc(tmem, TMEM_COLS);
  }
}

}  // namespace dbwd
}  // namespace pb

using namespace pb;

// q, k, v, dO: bf16 [batch, seq_len, ld] with head h at columns [128 h, 128 h + 128); beta: [batch, seq_len, heads], fp32 or
// bf16. In chunk order, total = batch * heads * ceil(seq_len / 64): Ap, T [total, 64, 64] as pb_delta_prep_fwd made them; ndU
// (= -dU), U [total, 64, 128]; S, dS [total, 128, 128]. All bf16. Outputs dq, dk, dv like q, dbeta like beta.
PB_API int pb_delta_bwd(const void* q, const void* k, const void* v, const void* beta, int beta_f32, const void* Ap,
                        const void* T, const void* ndU, const void* dO, const void* U, const void* S, const void* dS,
                        void* dq, void* dk, void* dv, void* dbeta, int batch, int seq_len, int heads, int ld, int* status,
                        cudaStream_t st) {
  using namespace dbwd;
  if (batch <= 0 || heads <= 0 || seq_len <= 0 || ld < heads * D || ld % 8) return PB_BAD_ARG;
  static pb::DeviceOnce attr_once;   // per device: the attribute belongs to the current GPU
  if (attr_once.need()) {
    cudaError_t e = cudaFuncSetAttribute(delta_bwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
    if (e != cudaSuccess) return static_cast<int>(e);
    attr_once.done();
  }
  Params p;
  p.n_chunks = (seq_len + C - 1) / C; p.heads = heads; p.seq_len = seq_len;
  p.total = batch * heads * p.n_chunks;
  p.beta = beta; p.beta_f32 = beta_f32; p.dbeta = dbeta; p.status = status;
  const uint64_t hd = static_cast<uint64_t>(heads) * D, bstr = static_cast<uint64_t>(seq_len) * ld;
  const uint64_t rows = static_cast<uint64_t>(p.total) * C, srows = static_cast<uint64_t>(p.total) * D;
  auto tok = [&](CUtensorMap* tm, const void* base) {
    return make_tmap_3d(tm, base, 2, hd, seq_len, batch, ld, bstr, 64, C);
  };
  CUtensorMap tN, tO, tU, tS, tDS, tK, tV, tQ, tA, tT, tDQ, tDK, tDV;
  int r = 0;
  r |= make_tmap_3d(&tN, ndU, 2, D, rows, 1, D, 0, 64, C);
  r |= tok(&tO, dO);
  r |= make_tmap_3d(&tU, U, 2, D, rows, 1, D, 0, 64, C);
  r |= make_tmap_3d(&tS, S, 2, D, srows, 1, D, 0, 64, D);
  r |= make_tmap_3d(&tDS, dS, 2, D, srows, 1, D, 0, 64, D);
  r |= tok(&tK, k); r |= tok(&tV, v); r |= tok(&tQ, q);
  r |= make_tmap_3d(&tA, Ap, 2, C, rows, 1, C, 0, 64, C);
  r |= make_tmap_3d(&tT, T, 2, C, rows, 1, C, 0, 64, C);
  r |= tok(&tDQ, dq); r |= tok(&tDK, dk); r |= tok(&tDV, dv);
  if (r != 0) return 1000 + r;
  const int grid = p.total < num_sms() ? p.total : num_sms();
  pb::launch(delta_bwd_kernel, grid, THREADS, SMEM, st, tN, tO, tU, tS, tDS, tK, tV, tQ, tA, tT, tDQ, tDK, tDV, p);
  return static_cast<int>(cudaGetLastError());
}
