// The chunk-local products of the delta rule's backward (sm_100a): what the state walks hand to the
// backward of the WY operands, four products per chunk of 64 tokens in one pass over their operands.
//
//   dW  = (-dU) S^T        dQ_s = dO S^T        dK_s = U dS'^T        dM = dO U^T
//
// The layer's backward runs delta_bwd.cu, which does this and pb_delta_prep_bwd's part in one kernel. These two are what its test
// compares it with, stage by stage.
//
// S is the bf16 state entering the chunk, dS' the gradient of the state leaving it, both
// [128, 128]; U, -dU and dO are [64, 128], dO read in place from its token-major layout.
//
// Bound by memory: 112 KB in and 56 KB out per chunk against about one microsecond of tensor-core
// time. As four batched GEMMs and a copy of dO into chunk order the same work moved 328 KB: S, U and
// dO were read by two products each. 4096 chunks: 281 us -> 110 us (6.3 TB/s).
//
// One persistent CTA per SM, two stages of all five operands (224 KB): while one chunk is
// multiplied, converted and stored, the next one's operands arrive. The results are staged in the
// stage's own S and dS' tiles, which the finished products no longer need.
//   warp 2: TMA producer   warp 3: MMA issue (one lane)
//   warp pairs (0,1) (4,5) (8,9) (12,13): rows 0..63 of one result each (a warp reads the
//   tensor-memory lanes of its quarter, so only the first two of four can serve 64 token rows)
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

namespace dchunk {

constexpr int C = 64, D = 128;
constexpr int NDU = 0, DO = 16384, UT = 32768, ST = 49152, DS = 81920, STAGE = 114688;
constexpr int BARS = 2 * STAGE, SMEM = BARS + 128 + 1024;
constexpr int THREADS = 448;
constexpr uint32_t COL_W = 0, COL_Q = 128, COL_K = 256, COL_M = 384, TMEM_COLS = 512;

struct Params {
  int n_chunks, heads, total;   // chunks per sequence; chunk g = (b * heads + h) * n_chunks + n
  int* status;
};

__global__ void __launch_bounds__(THREADS, 1)
delta_chunk_kernel(const __grid_constant__ CUtensorMap tmNDU, const __grid_constant__ CUtensorMap tmDO,
                   const __grid_constant__ CUtensorMap tmU, const __grid_constant__ CUtensorMap tmS,
                   const __grid_constant__ CUtensorMap tmDS, const __grid_constant__ CUtensorMap tmDW,
                   const __grid_constant__ CUtensorMap tmDQ, const __grid_constant__ CUtensorMap tmDK,
                   const __grid_constant__ CUtensorMap tmDM, const Params p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + BARS);
  uint64_t* full = bars;         // [2]
  uint64_t* empty = bars + 2;    // [2], one arrival per result
  uint64_t* acc_full = bars + 4;
  uint64_t* acc_free = bars + 5;   // one arrival per epilogue warp
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 6);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) { mbar_init(&full[i], 1); mbar_init(&empty[i], 4); }
    mbar_init(acc_full, 1);
    mbar_init(acc_free, 8);
    fence_barrier_init();
    tma_prefetch_desc(&tmNDU); tma_prefetch_desc(&tmDO); tma_prefetch_desc(&tmU);
    tma_prefetch_desc(&tmS); tma_prefetch_desc(&tmDS);
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

  if (warp == 2) {
    if (lane == 0) {
      uint32_t it = 0;
      for (int g = blockIdx.x; g < p.total; g += gridDim.x, ++it) {
        const int s = it & 1;
        if (!mbar_wait(&empty[s], ((it >> 1) & 1) ^ 1, p.status)) break;
        mbar_arrive_expect_tx(&full[s], STAGE);
        uint8_t* st = smem + s * STAGE;
        const int seq = g / p.n_chunks, n = g - seq * p.n_chunks;
        const int b = seq / p.heads, x0 = (seq - b * p.heads) * D;
        for (int hf = 0; hf < 2; ++hf) {
          tma_load_3d(st + NDU + hf * 8192, &tmNDU, &full[s], hf * 64, g * C, 0);
          tma_load_3d(st + ST + hf * 16384, &tmS, &full[s], hf * 64, g * D, 0);
          tma_load_3d(st + DO + hf * 8192, &tmDO, &full[s], x0 + hf * 64, n * C, b);
          tma_load_3d(st + UT + hf * 8192, &tmU, &full[s], hf * 64, g * C, 0);
          tma_load_3d(st + DS + hf * 16384, &tmDS, &full[s], hf * 64, g * D, 0);
        }
      }
    }
  } else if (warp == 3) {
    if (lane == 0) {
      const uint32_t id128 = make_idesc(1, 1, 128, 128, 0, 0), id64 = make_idesc(1, 1, 128, 64, 0, 0);
      uint32_t it = 0;
      for (int g = blockIdx.x; g < p.total; g += gridDim.x, ++it) {
        const int s = it & 1;
        if (!mbar_wait_spin(&full[s], (it >> 1) & 1, p.status)) break;
        if (!mbar_wait_spin(acc_free, (it & 1) ^ 1, p.status)) break;
        tc_fence_after();
        const uint32_t st = smem_u32(smem + s * STAGE);
        // 128-wide contraction, both operands K-major; a tile of R rows is two halves of R * 128 bytes.
        // The 64-row A tiles run as 128-row operands: accumulator lanes 64..127 are never read.
        auto mul = [&](uint32_t col, uint32_t a, uint32_t b, uint32_t b_half, uint32_t id) {
#pragma unroll
          for (int j = 0; j < 8; ++j)
            umma_f16(tmem + col, make_sdesc_sw128(st + a + (j >> 2) * 8192 + (j & 3) * 32, 16, 1024),
                     make_sdesc_sw128(st + b + (j >> 2) * b_half + (j & 3) * 32, 16, 1024), id, j > 0);
        };
        mul(COL_W, NDU, ST, 16384, id128);
        mul(COL_Q, DO, ST, 16384, id128);
        mul(COL_K, UT, DS, 16384, id128);
        mul(COL_M, DO, UT, 8192, id64);
        umma_commit(acc_full);
      }
    }
  } else if ((warp & 3) < 2) {
    const int res = warp >> 2;                     // 0 dW, 1 dQ, 2 dK, 3 dM
    const int r = (warp & 1) * 32 + lane;          // token row = tensor-memory lane
    const int cols = res == 3 ? 64 : 128;
    const uint32_t col = res == 0 ? COL_W : res == 1 ? COL_Q : res == 2 ? COL_K : COL_M;
    const uint32_t taddr = tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16) + col;
    const int stage_off = res < 2 ? ST + res * 16384 : DS + (res - 2) * 16384;
    const CUtensorMap* tm = res == 0 ? &tmDW : res == 1 ? &tmDQ : res == 2 ? &tmDK : &tmDM;
    uint32_t it = 0;
    for (int g = blockIdx.x; g < p.total; g += gridDim.x, ++it) {
      const int s = it & 1;
      const bool ok = mbar_wait_warp(acc_full, it & 1, p.status);
      tc_fence_after();
      uint8_t* out = smem + s * STAGE + stage_off;
#pragma unroll 1
      for (int c = 0; ok && c < cols; c += 64) {
        uint32_t v[64];
        tmem_ld_32x32b_x32(taddr + c, v);
        tmem_ld_32x32b_x32(taddr + c + 32, v + 32);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          bf16x8 pk;
#pragma unroll
          for (int j = 0; j < 4; ++j)
            pk.v[j] = __floats2bfloat162_rn(__uint_as_float(v[8 * i + 2 * j]), __uint_as_float(v[8 * i + 2 * j + 1]));
          st_shared8(out + (c >> 6) * 8192 + r * 128 + ((i ^ (r & 7)) << 4), pk);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (ok && lane == 0) mbar_arrive(acc_free);
      fence_proxy_async_smem();
      if (!bar_sync_and(1 + res, 64, ok)) break;   // both halves of the rows are staged
      if ((warp & 1) == 0 && lane == 0) {
        tma_store_3d(tm, out, 0, g * C, 0);
        if (cols == 128) tma_store_3d(tm, out + 8192, 64, g * C, 0);
        tma_store_commit();
        tma_store_wait_read<0>();
        mbar_arrive(&empty[s]);
      }
    }
    if ((warp & 1) == 0 && lane == 0) tma_store_wait<0>();
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

}  // namespace dchunk
}  // namespace pb

using namespace pb;

// ndU, U [total * 64, 128], S, dS [total * 128, 128] bf16 in chunk order; dO [batch, seq_len, ld] bf16
// with head h at columns 128 h (rows past seq_len count as zeros). Outputs in chunk order: dW, dQs, dKs
// [total * 64, 128], dM [total * 64, 64] bf16. total = batch * heads * ceil(seq_len / 64).
PB_API int pb_delta_chunk_products(const void* ndU, const void* dO, const void* U, const void* S,
                                   const void* dS, void* dW, void* dQs, void* dKs, void* dM, int batch,
                                   int seq_len, int heads, int ld, int* status, cudaStream_t st) {
  using namespace dchunk;
  if (batch <= 0 || heads <= 0 || seq_len <= 0 || ld < heads * D || ld % 8) return PB_BAD_ARG;
  static pb::DeviceOnce attr_once;   // per device: the attribute belongs to the current GPU
  if (attr_once.need()) {
    cudaError_t e = cudaFuncSetAttribute(delta_chunk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
    if (e != cudaSuccess) return static_cast<int>(e);
    attr_once.done();
  }
  Params p;
  p.n_chunks = (seq_len + C - 1) / C; p.heads = heads;
  p.total = batch * heads * p.n_chunks;
  p.status = status;
  const uint64_t rows = static_cast<uint64_t>(p.total) * C, srows = static_cast<uint64_t>(p.total) * D;
  CUtensorMap tN, tO, tU, tS, tD, tW, tQ, tK, tM;
  int r = 0;
  r |= make_tmap_3d(&tN, ndU, 2, D, rows, 1, D, 0, 64, C);
  r |= make_tmap_3d(&tO, dO, 2, static_cast<uint64_t>(heads) * D, seq_len, batch, ld,
                    static_cast<uint64_t>(seq_len) * ld, 64, C);
  r |= make_tmap_3d(&tU, U, 2, D, rows, 1, D, 0, 64, C);
  r |= make_tmap_3d(&tS, S, 2, D, srows, 1, D, 0, 64, D);
  r |= make_tmap_3d(&tD, dS, 2, D, srows, 1, D, 0, 64, D);
  r |= make_tmap_3d(&tW, dW, 2, D, rows, 1, D, 0, 64, C);
  r |= make_tmap_3d(&tQ, dQs, 2, D, rows, 1, D, 0, 64, C);
  r |= make_tmap_3d(&tK, dKs, 2, D, rows, 1, D, 0, 64, C);
  r |= make_tmap_3d(&tM, dM, 2, C, rows, 1, C, 0, 64, C);
  if (r != 0) return 1000 + r;
  const int grid = p.total < num_sms() ? p.total : num_sms();
  pb::launch(delta_chunk_kernel, grid, THREADS, SMEM, st, tN, tO, tU, tS, tD, tW, tQ, tK, tM, p);
  return static_cast<int>(cudaGetLastError());
}
