// Chunk-local WY operands of the delta rule on tcgen05 (sm_100a), one fused kernel.
//
// For every chunk of 64 tokens of one (batch, head) it forms, from the K / Q / V rows and
// the write strengths beta, everything the state walk consumes:
//
//   G = K K^T                      A  = diag(beta) tril(G, -1)       T = (I + A)^-1
//   A' = T diag(beta)              W  = A' K        U^ = A' V        M = tril(Q K^T)
//
// K, Q and V are read by TMA straight out of the projection outputs ([batch * seq,
// heads * 128], no per-chunk copies); G and Q K^T are two tcgen05.mma products with their
// accumulators in tensor memory; the unit-lower-triangular inverse is taken in fp32 by blocks (invert_unit_lower);
// A' goes back to shared memory as a 128-byte-swizzled bf16 operand for
// the two products W and U^; every result leaves by a TMA store. A chunk is one long chain of
// waits in two warps, so what counts is how many chunks an SM has in flight: four CTAs of 64
// threads, 49 KB and 128 tensor-memory columns each. V takes the place of the fp32 T once it is
// in registers, A' that of M once M is stored, U^ W's columns once W is in registers, and the next chunk's K and Q
// arrive while U^ is converted and stored.
// 4096 chunks: two CTAs with room for everything 165 us, three 141 us, four 129 us; with the inverse by blocks and
// the early loads 89 us (4.8 TB/s).
//
// Sequences need not be a multiple of 64 tokens: the token tensors are mapped per batch entry, so the
// rows the last chunk lacks load as zeros and are clipped from the stores; their beta counts as 0.
//
// Reference semantics: kernels/__init__.py:357-376 of the reference (per-token delta-rule
// recurrence); the chunked WY algebra and this kernel are this library's own.
#include <cuda.h>

#include "common.cuh"

namespace pb {

int make_tmap_3d(CUtensorMap* tm, const void* base, int elem_bytes, uint64_t inner,
                 uint64_t outer, uint64_t batch, uint64_t ld_elems, uint64_t batch_stride_elems,
                 uint32_t box_inner, uint32_t box_outer);

namespace dprep {

constexpr int C = 64, D = 128;
// A 64-row tile that serves as a 128-row A operand is read 8 KB past its end (A', the second halves of
// K and Q); what follows each of them is inside the allocation.
constexpr int KT = 0, QT = 16384, VA = 32768, BARS = 49152;   // Q, then M | T, then A' | T; A (fp32), then V
static_assert(KT + 24576 <= BARS && QT + 24576 <= BARS, "A operands stay in bounds");
constexpr int SMEM_BYTES = BARS + 256 + 1024;   // four CTAs per SM
constexpr int FWD_CTAS = 4, FWD_COLS = 128;
constexpr int TMEM_COLS = 256;   // backward

struct Params {
  int n_chunks;   // chunks per sequence
  int heads;
  int seq_len;    // tokens per sequence
  int total;      // batch * heads * n_chunks
  const void* beta;  // [batch, seq, heads]
  int beta_f32;
  int store_ta;   // 0: A' and T are not wanted (nothing will run backward)
  int* status;
};

__device__ __forceinline__ void st_swz(uint8_t* tile, int row, int c16, const bf16x8& v) {
  st_shared8(tile + row * 128 + ((c16 ^ (row & 7)) << 4), v);
}

// Row `row` of a 64-column fp32 accumulator block -> bf16 [64][64] swizzled tile, keeping
// columns <= limit (limit = 63 keeps all).
__device__ __forceinline__ void row_to_tile(uint32_t taddr, uint8_t* tile, int row, int limit) {
#pragma unroll 1
  for (int c = 0; c < 64; c += 32) {
    uint32_t v[32];
    tmem_ld_32x32b_x32(taddr + c, v);
    tmem_ld_wait();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float f[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) f[j] = (c + 8 * i + j <= limit) ? __uint_as_float(v[8 * i + j]) : 0.f;
      st_swz(tile, row, (c >> 3) + i, pack8(f));
    }
  }
}

// The fp32 matrix that is inverted: 64 rows of 16 pieces of 16 bytes, piece p of row i at p ^ (i & 15).
struct Square {
  float4* base;
  __device__ __forceinline__ float4& operator()(int row, int piece) const { return base[row * 16 + (piece ^ (row & 15))]; }
};
__device__ __forceinline__ void axpy(float4& acc, float a, const float4& b) {
  acc.x = fmaf(a, b.x, acc.x); acc.y = fmaf(a, b.y, acc.y);
  acc.z = fmaf(a, b.z, acc.z); acc.w = fmaf(a, b.w, acc.w);
}
// acc (R rows x 4 columns) = sum over k = 4 k_lo .. 4 k_hi - 1 of L(l_row + u, k from piece l_piece) R(r_row + k, r_piece)
template <int R>
__device__ __forceinline__ void block_mul(const Square m, float4 (&acc)[R], int l_row, int l_piece, int r_row,
                                          int r_piece, int k_lo, int k_hi) {
#pragma unroll
  for (int u = 0; u < R; ++u) acc[u] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 2
  for (int k4 = k_lo; k4 < k_hi; ++k4) {
    float4 a[R], b[4];
#pragma unroll
    for (int u = 0; u < R; ++u) a[u] = m(l_row + u, l_piece + k4);
#pragma unroll
    for (int j = 0; j < 4; ++j) b[j] = m(r_row + 4 * k4 + j, r_piece);
#pragma unroll
    for (int u = 0; u < R; ++u) {
      axpy(acc[u], a[u].x, b[0]); axpy(acc[u], a[u].y, b[1]);
      axpy(acc[u], a[u].z, b[2]); axpy(acc[u], a[u].w, b[3]);
    }
  }
}
// In place, 64 threads: the strictly lower A becomes T = (I + A)^-1. The 16 x 16 blocks on the diagonal by forward
// substitution, a column to a thread, then twice T21 = -T22 (A21 T11), a few rows and columns to a thread. What bounds
// it is the shared-memory port, 32 values a cycle whoever reads them: a substitution over all 64 rows, where a value
// serves one column a lane, takes 2752 cycles of it a chunk (for 1008 of multiply-adds), the blocks 1650.
__device__ __forceinline__ void invert_unit_lower(const Square m, int tid) {
  const int warp = tid >> 5, lane = tid & 31;
  {
    const int blk = tid >> 4, c = tid & 15;
    float t[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      float a0 = (i == c) ? 1.f : 0.f, a1 = 0.f, a2 = 0.f, a3 = 0.f;
#pragma unroll
      for (int q = 0; q < (i + 3) / 4; ++q) {
        const float4 a = m(16 * blk + i, 4 * blk + q);
        if (4 * q + 0 < i) a0 = fmaf(-a.x, t[4 * q + 0], a0);
        if (4 * q + 1 < i) a1 = fmaf(-a.y, t[4 * q + 1], a1);
        if (4 * q + 2 < i) a2 = fmaf(-a.z, t[4 * q + 2], a2);
        if (4 * q + 3 < i) a3 = fmaf(-a.w, t[4 * q + 3], a3);
      }
      t[i] = (a0 + a1) + (a2 + a3);
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 16; ++i) reinterpret_cast<float*>(&m(16 * blk + i, 4 * blk + (c >> 2)))[c & 3] = t[i];
    __syncwarp();
  }
  {   // 16 -> 32: a warp has one pair of blocks, a thread two rows and four columns
    const int row = 32 * warp + 16 + 2 * (lane >> 2), piece = 8 * warp + (lane & 3);
    float4 x[2];
    block_mul<2>(m, x, row, 8 * warp, 32 * warp, piece, 0, 4);
    __syncwarp();
    m(row, piece) = x[0]; m(row + 1, piece) = x[1];
    __syncwarp();
    block_mul<2>(m, x, row, 8 * warp + 4, 32 * warp + 16, piece, 0, 4);
    __syncwarp();
#pragma unroll
    for (int u = 0; u < 2; ++u) m(row + u, piece) = make_float4(-x[u].x, -x[u].y, -x[u].z, -x[u].w);
  }
  __syncthreads();
  {   // 32 -> 64: four rows and four columns to a thread; the zeros of T11 and T22 are left out by halves
    float4 x[4];
    int row = 32 + 4 * (lane >> 2), piece = 4 * warp + (lane & 3);
    block_mul<4>(m, x, row, 0, 0, piece, 4 * warp, 8);
    __syncthreads();
#pragma unroll
    for (int u = 0; u < 4; ++u) m(row + u, piece) = x[u];
    __syncthreads();
    row = 32 + 16 * warp + 4 * (lane >> 3); piece = lane & 7;
    block_mul<4>(m, x, row, 8, 32, piece, 0, 4 * warp + 4);
    __syncthreads();
#pragma unroll
    for (int u = 0; u < 4; ++u) m(row + u, piece) = make_float4(-x[u].x, -x[u].y, -x[u].z, -x[u].w);
  }
  __syncthreads();
}

__global__ void __launch_bounds__(64, FWD_CTAS)
delta_prep_fwd_kernel(const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmQ,
                      const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmW,
                      const __grid_constant__ CUtensorMap tmU, const __grid_constant__ CUtensorMap tmM,
                      const __grid_constant__ CUtensorMap tmAP, const __grid_constant__ CUtensorMap tmT,
                      const Params p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + BARS);
  uint64_t* full = bars;
  uint64_t* mma1 = bars + 1;
  uint64_t* mma2 = bars + 2;
  uint64_t* mma3 = bars + 3;
  uint64_t* fullv = bars + 4;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 5);
  float4* af4 = reinterpret_cast<float4*>(smem + VA);
  __shared__ float4 betas_[C / 4];
  float* betas = reinterpret_cast<float*>(betas_);

  const int r = threadIdx.x, warp = warp_index();
  if (r == 0) {
    mbar_init(full, 1); mbar_init(mma1, 1); mbar_init(mma2, 1); mbar_init(mma3, 1); mbar_init(fullv, 1);
    fence_barrier_init();
    tma_prefetch_desc(&tmK); tma_prefetch_desc(&tmQ); tma_prefetch_desc(&tmV);
  }
  if (warp == 0) {
    tmem_alloc(tmem_slot, FWD_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  after_previous_kernel();
  const uint32_t lane_addr = tmem + (static_cast<uint32_t>(warp * 32) << 16);
  const uint32_t id_kk64 = make_idesc(1, 1, 128, 64, 0, 0);    // A, B K-major, N = 64
  const uint32_t id_kn = make_idesc(1, 1, 128, 128, 0, 1);     // A K-major, B MN-major
  // descriptor words of the operands: an issue is one add for each
  const uint32_t k_k = sdesc_lo(smem_u32(smem + KT), 16), q_k = sdesc_lo(smem_u32(smem + QT), 16), ap_k = q_k;
  const uint32_t k_mn = sdesc_lo(smem_u32(smem + KT), 8192), v_mn = sdesc_lo(smem_u32(smem + VA), 8192);

  auto load_kq = [&](int g) {
    const int seq = g / p.n_chunks, t0 = (g - seq * p.n_chunks) * C;
    const int b = seq / p.heads, x0 = (seq - b * p.heads) * D;
    mbar_arrive_expect_tx(full, 2 * 16384);
    tma_load_3d(smem + KT, &tmK, full, x0, t0, b);
    tma_load_3d(smem + KT + 8192, &tmK, full, x0 + 64, t0, b);
    tma_load_3d(smem + QT, &tmQ, full, x0, t0, b);
    tma_load_3d(smem + QT + 8192, &tmQ, full, x0 + 64, t0, b);
  };
  if (r == 0 && static_cast<int>(blockIdx.x) < p.total) load_kq(blockIdx.x);
  uint32_t ph = 0;
  for (int g = blockIdx.x; g < p.total; g += gridDim.x, ph ^= 1) {
    const int seq = g / p.n_chunks, n = g - seq * p.n_chunks;
    const int b = seq / p.heads, h = seq - b * p.heads;
    const int t0 = n * C;                     // first token of the chunk
    const int x0 = h * D;
    float beta = 0.f;
    if (t0 + r < p.seq_len) {
      const size_t bidx = (static_cast<size_t>(b) * p.seq_len + t0 + r) * p.heads + h;
      beta = p.beta_f32 ? static_cast<const float*>(p.beta)[bidx]
                        : bf16_to_f32(static_cast<const bf16*>(p.beta)[bidx]);
    }
    bool ok = true;
    if (warp == 0) {
      ok = mbar_wait_warp(full, ph, p.status);
      if (ok) {
        tc_fence_after();
#pragma unroll
        for (int j = 0; j < 8; ++j)     // G = K K^T -> columns [0, 64)
          umma_f16_lo_warp(tmem, step_k(k_k, j), step_k(k_k, j), id_kk64, j > 0);
#pragma unroll
        for (int j = 0; j < 8; ++j)     // Q K^T -> columns [64, 128)
          umma_f16_lo_warp(tmem + 64, step_k(q_k, j), step_k(k_k, j), id_kk64, j > 0);
        umma_commit_warp(mma1);
      }
    }
    ok = mbar_wait_spin(mma1, ph, p.status) && ok;
    if (r == 0) tma_store_wait_read<0>();   // the previous chunk's U^ has left the tile that A goes into
    if (!__syncthreads_and(ok)) break;
    tc_fence_after();

    betas[r] = beta;
    // A = diag(beta) tril(G, -1), fp32
#pragma unroll 1
    for (int c = 0; c < 64; c += 32) {
      uint32_t v[32];
      tmem_ld_32x32b_x32(lane_addr + c, v);
      tmem_ld_wait();
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        float4 a;
        a.x = (c + 4 * i + 0 < r) ? beta * __uint_as_float(v[4 * i + 0]) : 0.f;
        a.y = (c + 4 * i + 1 < r) ? beta * __uint_as_float(v[4 * i + 1]) : 0.f;
        a.z = (c + 4 * i + 2 < r) ? beta * __uint_as_float(v[4 * i + 2]) : 0.f;
        a.w = (c + 4 * i + 3 < r) ? beta * __uint_as_float(v[4 * i + 3]) : 0.f;
        Square{af4}(r, (c >> 2) + i) = a;
      }
    }
    // M = tril(Q K^T) -> the Q tile's first half (the products that read Q are complete)
    row_to_tile(lane_addr + 64, smem + QT, r, r);
    fence_proxy_async_smem();
    __syncthreads();
    if (r == 0) {
      tma_store_3d(&tmM, smem + QT, 0, g * C, 0);
      tma_store_commit();
    }

    invert_unit_lower(Square{af4}, r);
    float4 t[16];   // row r of T
#pragma unroll
    for (int q = 0; q < 16; ++q) t[q] = Square{af4}(r, q);
    // T is in registers and M has left: V comes into T's place, A' goes into M's
    if (r == 0) tma_store_wait_read<0>();
    fence_proxy_async_smem();
    __syncthreads();
    if (r == 0) {
      mbar_arrive_expect_tx(fullv, 16384);
      tma_load_3d(smem + VA, &tmV, fullv, x0, t0, b);
      tma_load_3d(smem + VA + 8192, &tmV, fullv, x0 + 64, t0, b);
    }
    // T -> the Q tile's second half, A' = T diag(beta) -> its first
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const float4 lo = t[2 * q], hi = t[2 * q + 1];
      const float4 bl = reinterpret_cast<const float4*>(betas)[2 * q], bh = reinterpret_cast<const float4*>(betas)[2 * q + 1];
      const float ta[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
      const float aa[8] = {lo.x * bl.x, lo.y * bl.y, lo.z * bl.z, lo.w * bl.w,
                           hi.x * bh.x, hi.y * bh.y, hi.z * bh.z, hi.w * bh.w};
      st_swz(smem + QT, r, q, pack8(aa));
      if (p.store_ta) st_swz(smem + QT + 8192, r, q, pack8(ta));
    }
    fence_proxy_async_smem();
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
      tc_fence_after();
#pragma unroll
      for (int j = 0; j < 4; ++j)       // W = A' K -> columns [0, 128)
        umma_f16_lo_warp(tmem, step_k(ap_k, j), step_mn(k_mn, j), id_kn, j > 0);
      umma_commit_warp(mma2);
      if (r == 0 && p.store_ta) {
        tma_store_3d(&tmT, smem + QT + 8192, 0, g * C, 0);
        tma_store_3d(&tmAP, smem + QT, 0, g * C, 0);
        tma_store_commit();
      }
    }
    ok = mbar_wait_spin(mma2, ph, p.status);
    if (!__syncthreads_and(ok)) break;
    tc_fence_after();
    // W -> K tile (the product has finished reading it)
    row_to_tile(lane_addr + 0, smem + KT, r, 63);
    row_to_tile(lane_addr + 64, smem + KT + 8192, r, 63);
    fence_proxy_async_smem();
    tc_fence_before();
    __syncthreads();
    if (warp == 0 && (ok = mbar_wait_spin_warp(fullv, ph, p.status))) {
      tc_fence_after();
#pragma unroll
      for (int j = 0; j < 4; ++j)       // U^ = A' V -> the same columns
        umma_f16_lo_warp(tmem, step_k(ap_k, j), step_mn(v_mn, j), id_kn, j > 0);
      umma_commit_warp(mma3);
      if (r == 0) {
        tma_store_3d(&tmW, smem + KT, 0, g * C, 0);
        tma_store_3d(&tmW, smem + KT + 8192, 64, g * C, 0);
        tma_store_commit();
      }
    }
    ok = mbar_wait_spin(mma3, ph, p.status) && ok;
    if (!__syncthreads_and(ok)) break;
    tc_fence_after();
    if (r == 0 && g + static_cast<int>(gridDim.x) < p.total) {
      // nothing reads K, W, A' or T any more: the next chunk's K and Q arrive while U^ is converted and stored
      tma_store_wait_read<0>();
      load_kq(g + gridDim.x);
    }
    // U^ -> V tile
    row_to_tile(lane_addr + 0, smem + VA, r, 63);
    row_to_tile(lane_addr + 64, smem + VA + 8192, r, 63);
    fence_proxy_async_smem();
    tc_fence_before();
    __syncthreads();
    if (r == 0) {
      tma_store_3d(&tmU, smem + VA, 0, g * C, 0);
      tma_store_3d(&tmU, smem + VA + 8192, 64, g * C, 0);
      tma_store_commit();
    }
  }
  if (r == 0) tma_store_wait<0>();
  tc_fence_before();
  __syncthreads();
  if (p.status != nullptr && *reinterpret_cast<volatile int*>(p.status) != PB_OK) {
    for (int i = 0; i < 2000; ++i) __nanosleep(1000);  // let copies in flight land
    __syncthreads();
  }
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(tmem, FWD_COLS);
  }
}


// ------------------------------------------------------------------------------------
// Backward of the chunk-local part. Given, per chunk, the gradients the state walk hands
// back (dW, -dU, dM = dO U^T before masking, and the walk's own contributions to dQ and dK)
// it produces dq, dk, dv (token-major, like q / k / v) and dbeta:
//
//   dA' = dW K^T - (-dU) V^T... (dU^ = dU)          dV = A'^T dU          dK += A'^T dW
//   dbeta_j += sum_i dA'_ij T_ij                     dA = -T^T (dA' A'^T)
//   dbeta_i += sum_{j<i} dA_ij G_ij                  dG = diag(beta) tril(dA, -1)
//   dK += (dG + dG^T) K + tril(dM)^T Q               dQ += tril(dM) K
//
// Eleven tcgen05 products in four passes with 64-row operands; the 64 x 64 intermediates
// go through one shared-memory tile, re-used as K-major or MN-major operand as needed, so
// no transposes are materialised. The column sum for dbeta is the diagonal of dA'^T T,
// also a tensor-core product. The walk's dQ and dK come by TMA into the tiles the results leave from: read
// row by row from global memory at the end they were two thirds of all stalls. 4096 chunks: 297 -> 164 us.
namespace bwd {
constexpr int DW = 0, NDU = 16384, KTB = 32768, VQ = 49152, APB = 65536, TT = 73728, DM = 81920,
              TMP = 90112, BARSB = 98304;
constexpr int SMEM_BWD = 108 * 1024;
// Two warps cover the 64 rows (a warp reads the tensor-memory lanes of its quarter); warps 4 and 5 read the
// same lanes and take the other half of the columns, warps 2 and 3 only keep step. The conversions between two
// products are most of the chain, so halving them paid: 4096 chunks 162 -> 150 us.
constexpr int THREADS_BWD = 192;
}  // namespace bwd

struct BwdParams {
  int n_chunks, heads, seq_len, total;
  const void* beta;    // [batch, seq, heads]
  int beta_f32;
  int has_dq, has_dk;  // the walk's dQ = dO S^T and dK = U dS'^T are to be added
  void* dbeta;         // [batch, seq, heads], same type as beta
  int* status;
};

__device__ __forceinline__ void ld_row32(uint32_t taddr, float* f) {
  uint32_t v[32];
  tmem_ld_32x32b_x32(taddr, v);
  tmem_ld_wait();
#pragma unroll
  for (int i = 0; i < 32; ++i) f[i] = __uint_as_float(v[i]);
}

// Accumulator columns [c0, c0 + 64) of row `row`, times `sign`, -> two swizzled [64][64] bf16 tiles 8 KB apart;
// with `add` the tiles' present values are added first (each cell is this thread's alone)
__device__ __forceinline__ void row64_to_tile(uint32_t taddr, uint8_t* tiles, int row, int c0, float sign, bool add) {
#pragma unroll 1
  for (int c = c0; c < c0 + 64; c += 32) {
    float f[32];
    ld_row32(taddr + c, f);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int col = c + 8 * i;
      uint8_t* tile = tiles + (col >> 6) * 8192;
      const int c16 = (col & 63) >> 3;
      float o[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) o[j] = sign * f[8 * i + j];
      if (add) {
        float a[8];
        unpack8(ld_shared8(tile + row * 128 + ((c16 ^ (row & 7)) << 4)), a);
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] += a[j];
      }
      st_swz(tile, row, c16, pack8(o));
    }
  }
}

__global__ void __launch_bounds__(bwd::THREADS_BWD, 2)
delta_prep_bwd_kernel(const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmQ,
                      const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmDW,
                      const __grid_constant__ CUtensorMap tmNDU, const __grid_constant__ CUtensorMap tmDM,
                      const __grid_constant__ CUtensorMap tmAP, const __grid_constant__ CUtensorMap tmT,
                      const __grid_constant__ CUtensorMap tmDQ, const __grid_constant__ CUtensorMap tmDK,
                      const __grid_constant__ CUtensorMap tmDV, const __grid_constant__ CUtensorMap tmAQ,
                      const __grid_constant__ CUtensorMap tmAK, const BwdParams p) {
  using namespace bwd;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + BARSB);
  uint64_t* full = bars;
  uint64_t* fullq = bars + 1;
  uint64_t* mma = bars + 2;   // [4]
  uint64_t* fulla = bars + 6;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 8);

  __shared__ float dbeta_part[C];
  const int warp = threadIdx.x >> 5;
  const bool lead = threadIdx.x == 0;
  const bool active = (warp & 3) < 2;
  const int half = warp >> 2;                                   // which half of the columns
  const int r = (warp & 1) * 32 + (threadIdx.x & 31);           // row of the active warps
  if (lead) {
    mbar_init(full, 1); mbar_init(fullq, 1); mbar_init(fulla, 1);
    for (int i = 0; i < 4; ++i) mbar_init(&mma[i], 1);
    fence_barrier_init();
    tma_prefetch_desc(&tmK); tma_prefetch_desc(&tmQ); tma_prefetch_desc(&tmV);
    tma_prefetch_desc(&tmDW); tma_prefetch_desc(&tmNDU); tma_prefetch_desc(&tmDM);
    tma_prefetch_desc(&tmAP); tma_prefetch_desc(&tmT);
  }
  if (warp == 0) {
    tmem_alloc(tmem_slot, TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  after_previous_kernel();
  const uint32_t lane_addr = tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16);
  const int c32 = half * 32, c64 = half * 64;
  const uint32_t id_kk64 = make_idesc(1, 1, 128, 64, 0, 0);
  const uint32_t id_mm64 = make_idesc(1, 1, 128, 64, 1, 1);
  const uint32_t id_kn = make_idesc(1, 1, 128, 128, 0, 1);
  const uint32_t id_mm = make_idesc(1, 1, 128, 128, 1, 1);
  // operand descriptors, from words made once: K-major (8 steps over 128 columns, 4 over 64), MN-major (4 steps)
  const uint32_t base_k = sdesc_lo(smem_u32(smem), 16), base_mn = sdesc_lo(smem_u32(smem), 8192);
  auto kk = [&](int tile, int j) { return step_k(base_k + (tile >> 4), j); };
  auto mn = [&](int tile, int j) { return step_mn(base_mn + (tile >> 4), j); };

  uint32_t ph = 0;
  for (int g = blockIdx.x; g < p.total; g += gridDim.x, ph ^= 1) {
    const int seq = g / p.n_chunks, n = g - seq * p.n_chunks;
    const int b = seq / p.heads, h = seq - b * p.heads;
    const int t0 = n * C;
    const int x0 = h * D;
    const int crow = g * C;
    if (lead) {
      tma_store_wait_read<0>();
      mbar_arrive_expect_tx(full, 4 * 16384 + 3 * 8192);
      tma_load_3d(smem + DW, &tmDW, full, 0, crow, 0);
      tma_load_3d(smem + DW + 8192, &tmDW, full, 64, crow, 0);
      tma_load_3d(smem + NDU, &tmNDU, full, 0, crow, 0);
      tma_load_3d(smem + NDU + 8192, &tmNDU, full, 64, crow, 0);
      tma_load_3d(smem + KTB, &tmK, full, x0, t0, b);
      tma_load_3d(smem + KTB + 8192, &tmK, full, x0 + 64, t0, b);
      tma_load_3d(smem + VQ, &tmV, full, x0, t0, b);
      tma_load_3d(smem + VQ + 8192, &tmV, full, x0 + 64, t0, b);
      tma_load_3d(smem + APB, &tmAP, full, 0, crow, 0);
      tma_load_3d(smem + TT, &tmT, full, 0, crow, 0);
      tma_load_3d(smem + DM, &tmDM, full, 0, crow, 0);
    }
    const bool valid = active && t0 + r < p.seq_len;
    const size_t bidx = (static_cast<size_t>(b) * p.seq_len + t0 + r) * p.heads + h;
    float beta = 0.f;
    if (valid)
      beta = p.beta_f32 ? static_cast<const float*>(p.beta)[bidx]
                        : bf16_to_f32(static_cast<const bf16*>(p.beta)[bidx]);
    bool ok = true;
    // ---- pass 1: dA' parts and dV ----
    if (lead) {
      ok = mbar_wait(full, ph, p.status);
      if (ok) {
        tc_fence_after();
#pragma unroll
        for (int j = 0; j < 8; ++j) umma_f16_lo(tmem + 0, kk(DW, j), kk(KTB, j), id_kk64, j > 0);
#pragma unroll
        for (int j = 0; j < 8; ++j) umma_f16_lo(tmem + 64, kk(NDU, j), kk(VQ, j), id_kk64, j > 0);
#pragma unroll
        for (int j = 0; j < 4; ++j) umma_f16_lo(tmem + 128, mn(APB, j), mn(NDU, j), id_mm, j > 0);
        umma_commit(&mma[0]);
      }
    }
    ok = mbar_wait_spin(&mma[0], ph, p.status) && ok;
    if (!__syncthreads_and(ok)) break;
    tc_fence_after();
    if (lead) {   // V is consumed: bring Q into its place
      mbar_arrive_expect_tx(fullq, 16384);
      tma_load_3d(smem + VQ, &tmQ, fullq, x0, t0, b);
      tma_load_3d(smem + VQ + 8192, &tmQ, fullq, x0 + 64, t0, b);
    }
    if (active) {
      // dV = -(A'^T (-dU)) -> staged over the -dU tile
      row64_to_tile(lane_addr + 128, smem + NDU, r, c64, -1.f, false);
      // dA' = dW K^T - (-dU) V^T -> operand tile
      {
        float a[32], s[32];
        ld_row32(lane_addr + c32, a);
        ld_row32(lane_addr + 64 + c32, s);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          float o[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) o[j] = a[8 * i + j] - s[8 * i + j];
          st_swz(smem + TMP, r, (c32 >> 3) + i, pack8(o));
        }
      }
      // tril(dM) in place (row r keeps columns <= r)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int c16 = (c32 >> 3) + i;
        uint8_t* cell = smem + DM + r * 128 + ((c16 ^ (r & 7)) << 4);
        if (8 * c16 + 7 > r) {
          float f[8];
          unpack8(ld_shared8(cell), f);
#pragma unroll
          for (int j = 0; j < 8; ++j) if (8 * c16 + j > r) f[j] = 0.f;
          st_shared8(cell, pack8(f));
        }
      }
    }
    fence_proxy_async_smem();
    tc_fence_before();
    __syncthreads();
    // ---- pass 2: X = dA' A'^T, Y = dA'^T T (diagonal = dbeta part), dK = A'^T dW ----
    if (lead) {
      tc_fence_after();
      tma_store_3d(&tmDV, smem + NDU, x0, t0, b);
      tma_store_3d(&tmDV, smem + NDU + 8192, x0 + 64, t0, b);
      tma_store_commit();
#pragma unroll
      for (int j = 0; j < 4; ++j) umma_f16_lo(tmem + 0, kk(TMP, j), kk(APB, j), id_kk64, j > 0);
#pragma unroll
      for (int j = 0; j < 4; ++j) umma_f16_lo(tmem + 64, mn(TMP, j), mn(TT, j), id_mm64, j > 0);
#pragma unroll
      for (int j = 0; j < 4; ++j) umma_f16_lo(tmem + 128, mn(APB, j), mn(DW, j), id_mm, j > 0);
      umma_commit(&mma[1]);
    }
    ok = mbar_wait_spin(&mma[1], ph, p.status);
    if (!__syncthreads_and(ok)) break;
    tc_fence_after();
    if (lead && (p.has_dq || p.has_dk)) {
      // dW and dV's staging are done with: the walk's dQ and dK arrive in the tiles that dq and dk will
      // leave from, while the next two passes run
      tma_store_wait_read<0>();
      mbar_arrive_expect_tx(fulla, (p.has_dq ? 16384u : 0u) + (p.has_dk ? 16384u : 0u));
      if (p.has_dq) {
        tma_load_3d(smem + DW, &tmAQ, fulla, 0, crow, 0);
        tma_load_3d(smem + DW + 8192, &tmAQ, fulla, 64, crow, 0);
      }
      if (p.has_dk) {
        tma_load_3d(smem + NDU, &tmAK, fulla, 0, crow, 0);
        tma_load_3d(smem + NDU + 8192, &tmAK, fulla, 64, crow, 0);
      }
    }
    float dbeta = 0.f;
    if (active) {
      float x[32], y[32];
      ld_row32(lane_addr + c32, x);
      ld_row32(lane_addr + 64 + c32, y);
#pragma unroll
      for (int i = 0; i < 32; ++i) if (c32 + i == r) dbeta = y[i];
#pragma unroll
      for (int i = 0; i < 4; ++i) st_swz(smem + TMP, r, (c32 >> 3) + i, pack8(x + 8 * i));
    }
    fence_proxy_async_smem();
    tc_fence_before();
    __syncthreads();
    // ---- pass 3: -dA = T^T X, G = K K^T ----
    if (lead) {
      tc_fence_after();
#pragma unroll
      for (int j = 0; j < 4; ++j) umma_f16_lo(tmem + 0, mn(TT, j), mn(TMP, j), id_mm64, j > 0);
#pragma unroll
      for (int j = 0; j < 8; ++j) umma_f16_lo(tmem + 64, kk(KTB, j), kk(KTB, j), id_kk64, j > 0);
      umma_commit(&mma[2]);
    }
    ok = mbar_wait_spin(&mma[2], ph, p.status);
    if (!__syncthreads_and(ok)) break;
    tc_fence_after();
    if (active) {
      float na[32], gk[32];
      ld_row32(lane_addr + c32, na);
      ld_row32(lane_addr + 64 + c32, gk);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float o[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const bool low = c32 + 8 * i + j < r;
          const float da = low ? -na[8 * i + j] : 0.f;
          dbeta = fmaf(da, low ? gk[8 * i + j] : 0.f, dbeta);
          o[j] = beta * da;
        }
        st_swz(smem + TMP, r, (c32 >> 3) + i, pack8(o));
      }
      if (half == 1) dbeta_part[r] = dbeta;
    }
    fence_proxy_async_smem();
    tc_fence_before();
    __syncthreads();
    if (valid && half == 0) {
      dbeta += dbeta_part[r];
      if (p.beta_f32) static_cast<float*>(p.dbeta)[bidx] = dbeta;
      else static_cast<bf16*>(p.dbeta)[bidx] = f32_to_bf16(dbeta);
    }
    // ---- pass 4: dK += dG K + dG^T K + tril(dM)^T Q ; dQ = tril(dM) K ----
    if (lead) {
      ok = mbar_wait(fullq, ph, p.status);
      if (ok) {
        tc_fence_after();
#pragma unroll
        for (int j = 0; j < 4; ++j) umma_f16_lo(tmem + 128, kk(TMP, j), mn(KTB, j), id_kn, 1);
#pragma unroll
        for (int j = 0; j < 4; ++j) umma_f16_lo(tmem + 128, mn(TMP, j), mn(KTB, j), id_mm, 1);
#pragma unroll
        for (int j = 0; j < 4; ++j) umma_f16_lo(tmem + 128, mn(DM, j), mn(VQ, j), id_mm, 1);
#pragma unroll
        for (int j = 0; j < 4; ++j) umma_f16_lo(tmem + 0, kk(DM, j), mn(KTB, j), id_kn, j > 0);
        umma_commit(&mma[3]);
      }
      tma_store_wait_read<0>();   // dV has left the tile dK is staged in
    }
    if (p.has_dq || p.has_dk) ok = mbar_wait_spin(fulla, ph, p.status) && ok;
    ok = mbar_wait_spin(&mma[3], ph, p.status) && ok;
    if (!__syncthreads_and(ok)) break;
    tc_fence_after();
    if (active) {
      row64_to_tile(lane_addr + 0, smem + DW, r, c64, 1.f, p.has_dq != 0);
      row64_to_tile(lane_addr + 128, smem + NDU, r, c64, 1.f, p.has_dk != 0);
    }
    fence_proxy_async_smem();
    tc_fence_before();
    __syncthreads();
    if (lead) {
      tma_store_3d(&tmDQ, smem + DW, x0, t0, b);
      tma_store_3d(&tmDQ, smem + DW + 8192, x0 + 64, t0, b);
      tma_store_3d(&tmDK, smem + NDU, x0, t0, b);
      tma_store_3d(&tmDK, smem + NDU + 8192, x0 + 64, t0, b);
      tma_store_commit();
    }
  }
  if (lead) tma_store_wait<0>();
  tc_fence_before();
  __syncthreads();
  if (p.status != nullptr && *reinterpret_cast<volatile int*>(p.status) != PB_OK) {
    for (int i = 0; i < 2000; ++i) __nanosleep(1000);  // let copies in flight land
    __syncthreads();
  }
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(tmem, TMEM_COLS);
  }
}

}  // namespace dprep
}  // namespace pb

using namespace pb;

// q, k, v: bf16 [batch, seq_len, ld] row-major with head h at columns [128 h, 128 h + 128)
// (ld >= heads * 128, a multiple of 8); beta: [batch, seq_len, heads], fp32 or bf16.
// Outputs, chunk g = (b * heads + h) * n_chunks + n, n_chunks = ceil(seq_len / 64): W, U^ [g][64][128];
// M, A', T [g][64][64]. A' and T may both be null when nothing will run backward.
PB_API int pb_delta_prep_fwd(const void* q, const void* k, const void* v, const void* beta,
                             int beta_f32, void* W, void* Uhat, void* M, void* Ap, void* T,
                             int batch, int seq_len, int heads, int ld, int* status,
                             int max_ctas, cudaStream_t st) {
  using namespace dprep;
  if (batch <= 0 || heads <= 0 || seq_len <= 0 || ld < heads * D || ld % 8)
    return PB_BAD_ARG;
  static pb::DeviceOnce attr_once;   // per device: the attribute belongs to the current GPU
  if (attr_once.need()) {
    cudaError_t e = cudaFuncSetAttribute(delta_prep_fwd_kernel,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
    if (e != cudaSuccess) return static_cast<int>(e);
    attr_once.done();
  }
  Params p;
  p.n_chunks = (seq_len + C - 1) / C; p.heads = heads; p.seq_len = seq_len;
  p.total = batch * heads * p.n_chunks;
  p.beta = beta; p.beta_f32 = beta_f32; p.status = status;
  p.store_ta = Ap != nullptr;
  if (p.store_ta != (T != nullptr)) return PB_BAD_ARG;
  const uint64_t bstr = static_cast<uint64_t>(seq_len) * ld;   // batch stride of the token tensors
  const uint64_t rows = static_cast<uint64_t>(p.total) * C;
  CUtensorMap tK, tQ, tV, tW, tU, tM, tA, tT;
  int r = 0;
  r |= make_tmap_3d(&tK, k, 2, static_cast<uint64_t>(heads) * D, seq_len, batch, ld, bstr, 64, C);
  r |= make_tmap_3d(&tQ, q, 2, static_cast<uint64_t>(heads) * D, seq_len, batch, ld, bstr, 64, C);
  r |= make_tmap_3d(&tV, v, 2, static_cast<uint64_t>(heads) * D, seq_len, batch, ld, bstr, 64, C);
  r |= make_tmap_3d(&tW, W, 2, D, rows, 1, D, 0, 64, C);
  r |= make_tmap_3d(&tU, Uhat, 2, D, rows, 1, D, 0, 64, C);
  r |= make_tmap_3d(&tM, M, 2, C, rows, 1, C, 0, 64, C);
  tA = tT = tM;
  if (p.store_ta) {
    r |= make_tmap_3d(&tA, Ap, 2, C, rows, 1, C, 0, 64, C);
    r |= make_tmap_3d(&tT, T, 2, C, rows, 1, C, 0, 64, C);
  }
  if (r != 0) return 1000 + r;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  int grid = FWD_CTAS * sms;
  if (max_ctas > 0 && max_ctas < grid) grid = max_ctas;
  if (grid > p.total) grid = p.total;
  pb::launch(delta_prep_fwd_kernel, grid, 64, SMEM_BYTES, st, tK, tQ, tV, tW, tU, tM, tA, tT, p);
  return static_cast<int>(cudaGetLastError());
}

// Backward of pb_delta_prep_fwd. dW, ndU (= -dU), dq_add, dk_add: [total][64][128] bf16;
// dM (unmasked dO U^T), Ap, T: [total][64][64] bf16; dq, dk, dv: like q / k / v;
// dbeta: like beta. dq_add / dk_add may be null.
PB_API int pb_delta_prep_bwd(const void* q, const void* k, const void* v, const void* beta,
                             int beta_f32, const void* Ap, const void* T, const void* dW,
                             const void* ndU, const void* dM, const void* dq_add,
                             const void* dk_add, void* dq, void* dk, void* dv, void* dbeta,
                             int batch, int seq_len, int heads, int ld, int* status,
                             int max_ctas, cudaStream_t st) {
  using namespace dprep;
  if (batch <= 0 || heads <= 0 || seq_len <= 0 || ld < heads * D || ld % 8)
    return PB_BAD_ARG;
  static pb::DeviceOnce attr_once;   // per device: the attribute belongs to the current GPU
  if (attr_once.need()) {
    cudaError_t e = cudaFuncSetAttribute(delta_prep_bwd_kernel,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         bwd::SMEM_BWD);
    if (e != cudaSuccess) return static_cast<int>(e);
    attr_once.done();
  }
  BwdParams p;
  p.n_chunks = (seq_len + C - 1) / C; p.heads = heads; p.seq_len = seq_len;
  p.total = batch * heads * p.n_chunks;
  p.beta = beta; p.beta_f32 = beta_f32;
  p.has_dq = dq_add != nullptr; p.has_dk = dk_add != nullptr;
  p.dbeta = dbeta; p.status = status;
  const uint64_t bstr = static_cast<uint64_t>(seq_len) * ld;   // batch stride of the token tensors
  const uint64_t rows = static_cast<uint64_t>(p.total) * C;
  const uint64_t hd = static_cast<uint64_t>(heads) * D;
  CUtensorMap tK, tQ, tV, tDW, tNDU, tDM, tA, tT, tDQ, tDK, tDV, tAQ, tAK;
  int r = 0;
  r |= make_tmap_3d(&tK, k, 2, hd, seq_len, batch, ld, bstr, 64, C);
  r |= make_tmap_3d(&tQ, q, 2, hd, seq_len, batch, ld, bstr, 64, C);
  r |= make_tmap_3d(&tV, v, 2, hd, seq_len, batch, ld, bstr, 64, C);
  r |= make_tmap_3d(&tDW, dW, 2, D, rows, 1, D, 0, 64, C);
  r |= make_tmap_3d(&tNDU, ndU, 2, D, rows, 1, D, 0, 64, C);
  r |= make_tmap_3d(&tDM, dM, 2, C, rows, 1, C, 0, 64, C);
  r |= make_tmap_3d(&tA, Ap, 2, C, rows, 1, C, 0, 64, C);
  r |= make_tmap_3d(&tT, T, 2, C, rows, 1, C, 0, 64, C);
  r |= make_tmap_3d(&tDQ, dq, 2, hd, seq_len, batch, ld, bstr, 64, C);
  r |= make_tmap_3d(&tDK, dk, 2, hd, seq_len, batch, ld, bstr, 64, C);
  r |= make_tmap_3d(&tDV, dv, 2, hd, seq_len, batch, ld, bstr, 64, C);
  tAQ = tAK = tDW;
  if (dq_add != nullptr) r |= make_tmap_3d(&tAQ, dq_add, 2, D, rows, 1, D, 0, 64, C);
  if (dk_add != nullptr) r |= make_tmap_3d(&tAK, dk_add, 2, D, rows, 1, D, 0, 64, C);
  if (r != 0) return 1000 + r;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  int grid = 2 * sms;
  if (max_ctas > 0 && max_ctas < grid) grid = max_ctas;
  if (grid > p.total) grid = p.total;
  pb::launch(delta_prep_bwd_kernel, grid, bwd::THREADS_BWD, bwd::SMEM_BWD, st, tK, tQ, tV, tDW, tNDU, tDM, tA, tT, tDQ,
                                                           tDK, tDV, tAQ, tAK, p);
  return static_cast<int>(cudaGetLastError());
}
