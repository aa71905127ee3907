// Block-scaled FP8 (e4m3) GEMM on tcgen05 and the quantisers that feed it (sm_100a).
//
//   C[M, N] (bf16) = sum over K-blocks kb of  sa[kb, m] * sb[n / 128, kb] * (Aq_kb . Bq_kb^T)
//
// Aq [M, K] e4m3 with one fp32 scale per row per 128 contraction elements (stored
// [K / 128, M] so a warp reads consecutive rows), Bq [N, K] e4m3 with one scale per
// 128 x 128 block. Exactly the arithmetic of quantise -> dequantise -> fp32 matmul, with the
// dequantisation applied to the 128-deep partial products instead of to the operands.
//
// Two kernels: on CTA pairs (gemm_fp8_pair_kernel below) and on single CTAs, for small or finely grouped products and
// for rows that are still arriving. The latter, one CTA per SM, persistent over 128 x 256 output tiles:
//   warp 0   TMA producer: per K-block a 128 x 128 B tile of A and a 256 x 128 B tile of B
//            (128 bytes per row = one swizzle atom), 4-stage ring
//   warp 1   MMA issuer: four kind::f8f6f4 MMAs (M 128, N 256, K 32) per K-block into one of
//            two 256-column tensor-memory accumulators, fresh (not accumulated) per K-block
//   warps 2-9  promotion + epilogue, two groups of four warps, one per 128-column half (one B
//            scale each): every thread owns one output row of its half; per K-block it reads
//            the 128 partial sums from tensor memory (two 64-column batches per wait), scales
//            them by sa * sb and adds them to 128 fp32 registers with packed two-wide FMAs
//            (fma.rn.f32x2: the promotion is bound by FMA issue slots); after the last K-block the
//            row goes out as bf16 through a swizzled staging slab and TMA stores
// Grouped mode (mixture-of-experts): row block m multiplies expert mblk_group[m] of a
// [groups, N, K] weight tensor with scales [groups, N / 128, K / 128]; negative = skip.
//
// Quantisers: pb_fp8_quant_rows (1 x 128 blocks, writes q and the [K / 128, M] scales) and
// pb_fp8_quant_blocks (128 x 128 blocks). scale = amax / 448, or 1 for an all-zero block.
//
// Reference semantics: kernels/__init__.py fp8_quantize / fp8_linear of the reference
// (block 128, e4m3, scale = amax / 448).
#include <cuda.h>
#include <cuda_fp8.h>

#include "common.cuh"

namespace pb {

int make_tmap_3d(CUtensorMap* tm, const void* base, int elem_bytes, uint64_t inner,
                 uint64_t outer, uint64_t batch, uint64_t ld_elems, uint64_t batch_stride_elems,
                 uint32_t box_inner, uint32_t box_outer);
int num_sms();

namespace f8 {

constexpr int BM = 128, BN = 256, BK = 128, HALF = 128;
constexpr int STAGES = 4;
constexpr int A_BYTES = BM * BK, B_BYTES = BN * BK, STAGE_BYTES = A_BYTES + B_BYTES;
constexpr int EPI_BYTES = 8 * 4096;
constexpr int THREADS = 320;
constexpr int SMEM_TOTAL = STAGES * STAGE_BYTES + EPI_BYTES + 1024 + 256;

struct Params {
  int M, N, K;
  const float* sa;     // [K / 128, M]
  const float* sb;     // [groups, ceil(N / 128), K / 128]
  const int* mblk_group;
  int* status;
  // Fused expert-parallel dispatch (null otherwise): the rows of A and their scales are being
  // stored into this GPU's memory by the other ranks' dispatch kernels while this kernel runs.
  // blk_arrived[m] counts the rows of 128-row block m that have landed (the senders add to it
  // with release semantics after each row), blk_expect[m] is how many will; the TMA producer
  // takes a block only once it is complete. TMA reads this GPU's own memory only.
  const uint32_t* blk_arrived;
  const int* blk_expect;
  uint64_t wait_budget_ns;
};

// Two fp32 FMAs in one instruction (fma.rn.f32x2): a0 += s * x0, a1 += s * x1, each rounded
// like fmaf. The promotion is bound by FMA issue slots, and this halves them.
__device__ __forceinline__ void fma2(float& a0, float& a1, float s, uint32_t x0, uint32_t x1) {
  asm("{\n\t.reg .b64 pa, pb, pc;\n\t"
      "mov.b64 pa, {%0, %1};\n\t"
      "mov.b64 pb, {%3, %4};\n\t"
      "mov.b64 pc, {%2, %2};\n\t"
      "fma.rn.f32x2 pa, pc, pb, pa;\n\t"
      "mov.b64 {%0, %1}, pa;\n\t}"
      : "+f"(a0), "+f"(a1)
      : "f"(s), "r"(x0), "r"(x1));
}

// PROBE 0 is the product. The others exist only in the debug build of the library and time
// parts of the kernel (their output is not the product's): 1 = no promotion (loads, MMAs and
// the per-K-block accumulator hand-over only), 2 = accumulation in place with one hand-over
// per tile (the ceiling of this tile shape and operand feed), 3 = promotion FMAs without the
// tensor-memory loads, 4 = tensor-memory loads without the FMAs.
template <int PROBE>
__global__ void __launch_bounds__(THREADS, 1)
gemm_fp8_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                const __grid_constant__ CUtensorMap tmC, const Params p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint8_t* smA = smem;
  uint8_t* smB = smem + STAGES * A_BYTES;
  uint8_t* smEpi = smem + STAGES * STAGE_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + STAGES * STAGE_BYTES + EPI_BYTES);
  uint64_t* full = bars;
  uint64_t* empty = bars + STAGES;
  uint64_t* tfull = bars + 2 * STAGES;
  uint64_t* tempty = bars + 2 * STAGES + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 4);

  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int num_m = (p.M + BM - 1) / BM, num_n = (p.N + BN - 1) / BN;
  const int nkb = p.K / BK;
  const long total = static_cast<long>(num_m) * num_n;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&tfull[a], 1);
      mbar_init(&tempty[a], 256);
    }
    fence_barrier_init();
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 2 * BN);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  after_previous_kernel();

  // n-major inside groups of 8 row blocks, like the bf16 kernel: B tiles stay in L2
  auto coords = [&](long t, int& m_blk, int& n_blk) {
    const int r = static_cast<int>(t);
    const int group = 8 * num_n;
    const int first_m = (r / group) * 8;
    const int gsz = min(num_m - first_m, 8);
    m_blk = first_m + (r % group) % gsz;
    n_blk = (r % group) / gsz;
  };
  auto group_of = [&](int m_blk) { return p.mblk_group ? p.mblk_group[m_blk] : 0; };

  if (warp == 0) {
    if (lane == 0) {
      int s = 0;
      uint32_t ph = 0;
      bool ok = true;
      for (long t = blockIdx.x; t < total && ok; t += gridDim.x) {
        int m_blk, n_blk;
        coords(t, m_blk, n_blk);
        const int g = group_of(m_blk);
        if (g < 0) continue;
        if (p.blk_arrived != nullptr) {
          const int want = p.blk_expect[m_blk];
          if (want > 0) {
            if (!wait_flag_ge(p.blk_arrived + m_blk, static_cast<uint32_t>(want), p.wait_budget_ns,
                              p.status)) { ok = false; break; }
            // the rows were written by peers' ordinary stores; the bulk loads below read
            // through the asynchronous proxy
            asm volatile("fence.proxy.async.global;" ::: "memory");
          }
        }
        for (int kb = 0; kb < nkb; ++kb) {
          if (!mbar_wait(&empty[s], ph ^ 1, p.status)) { ok = false; break; }
          mbar_arrive_expect_tx(&full[s], STAGE_BYTES);
          tma_load_3d(smA + s * A_BYTES, &tmA, &full[s], kb * BK, m_blk * BM, 0);
          tma_load_3d(smB + s * B_BYTES, &tmB, &full[s], kb * BK, n_blk * BN, g);
          if (++s == STAGES) { s = 0; ph ^= 1; }
        }
      }
    }
  } else if (warp == 1) {
    {
      const uint32_t idesc = make_idesc(0, 0, BM, BN, 0, 0);   // e4m3 x e4m3, both K-major
      int s = 0;
      uint32_t ph = 0;
      uint32_t it = 0;        // K-blocks issued so far: picks the accumulator and its phase
      bool ok = true;
      for (long t = blockIdx.x; t < total && ok; t += gridDim.x) {
        int m_blk, n_blk;
        coords(t, m_blk, n_blk);
        if (group_of(m_blk) < 0) continue;
        for (int kb = 0; kb < nkb; it += (PROBE == 2 ? (kb == nkb - 1) : 1), ++kb) {
          const int acc = it & 1;
          if ((PROBE != 2 || kb == 0) && !mbar_wait_warp(&tempty[acc], ((it >> 1) & 1) ^ 1, p.status)) { ok = false; break; }
          if (!mbar_wait_warp(&full[s], ph, p.status)) { ok = false; break; }
          tc_fence_after();
          const uint32_t a_addr = smem_u32(smA + s * A_BYTES);
          const uint32_t b_addr = smem_u32(smB + s * B_BYTES);
#pragma unroll
          for (int j = 0; j < BK / 32; ++j)
            umma_f8_warp(tmem_base + acc * BN, make_sdesc_sw128(a_addr + j * 32, 16, 1024),
                    make_sdesc_sw128(b_addr + j * 32, 16, 1024), idesc,
                    (j > 0 || (PROBE == 2 && kb > 0)) ? 1u : 0u);
          umma_commit_warp(&empty[s]);
          if (PROBE != 2 || kb == nkb - 1) umma_commit_warp(&tfull[acc]);
          if (++s == STAGES) { s = 0; ph ^= 1; }
        }
      }
    }
  } else {
    const int q = warp & 3;            // tensor-memory lane quarter of this warp
    const int half = (warp - 2) >> 2;  // which 128 columns of the tile
    const int n_sb = p.K / BK;
    const int n_sb_rows = (p.N + HALF - 1) / HALF;
    uint32_t it = 0;
    bool ok = true;
    uint8_t* buf = smEpi + (warp - 2) * 4096;
    for (long t = blockIdx.x; t < total && ok; t += gridDim.x) {
      int m_blk, n_blk;
      coords(t, m_blk, n_blk);
      const int g = group_of(m_blk);
      if (g < 0) continue;
      const int row = m_blk * BM + q * 32 + lane;
      const int srow = min(row, p.M - 1);
      const int sb_row = min(n_blk * 2 + half, n_sb_rows - 1);
      const float* sb = p.sb + (static_cast<size_t>(g) * n_sb_rows + sb_row) * n_sb;
      float acc[HALF];
#pragma unroll
      for (int i = 0; i < HALF; ++i) acc[i] = 0.f;
      // Scale of the K-block in hand, loaded one block ahead so its latency hides behind the
      // previous block's promotion. In the fused-dispatch mode a peer may still be writing the
      // scales when the tile starts: the first one is then read only after the first accumulator
      // is full, which implies that the whole row block (payload and scales) has landed.
      const float* sa_row = p.sa + srow;
      float scale_cur = 0.f;
      bool have = false;
      if (p.blk_arrived == nullptr) {
        scale_cur = __ldcg(sa_row) * sb[0];
        have = true;
      }
      for (int kb = 0; kb < (PROBE == 2 ? 1 : nkb); ++kb, ++it) {
        const int a = it & 1;
        if (!mbar_wait_warp(&tfull[a], (it >> 1) & 1, p.status)) { ok = false; break; }
        tc_fence_after();
        if (!have) scale_cur = __ldcg(sa_row + static_cast<size_t>(kb) * p.M) * sb[kb];
        const float scale = scale_cur;
        if (kb + 1 < nkb) {
          scale_cur = __ldcg(sa_row + static_cast<size_t>(kb + 1) * p.M) * sb[kb + 1];
          have = true;
        }
        const uint32_t t_addr =
            tmem_base + a * BN + half * HALF + (static_cast<uint32_t>(q * 32) << 16);
        if constexpr (PROBE == 0) {
#pragma unroll
          for (int c = 0; c < HALF; c += 64) {
            uint32_t r0[32], r1[32];
            tmem_ld_32x32b_x32(t_addr + c, r0);
            tmem_ld_32x32b_x32(t_addr + c + 32, r1);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; i += 2) {
              fma2(acc[c + i], acc[c + i + 1], scale, r0[i], r0[i + 1]);
              fma2(acc[c + 32 + i], acc[c + 32 + i + 1], scale, r1[i], r1[i + 1]);
            }
          }
        } else if constexpr (PROBE == 3) {
          const float v = __uint_as_float(0x3f800000u + (kb & 3));
#pragma unroll
          for (int i = 0; i < HALF; ++i) acc[i] = fmaf(scale, v + i, acc[i]);
        } else if constexpr (PROBE == 4) {
#pragma unroll
          for (int c = 0; c < HALF; c += 64) {
            uint32_t r0[32], r1[32];
            tmem_ld_32x32b_x32(t_addr + c, r0);
            tmem_ld_32x32b_x32(t_addr + c + 32, r1);
            tmem_ld_wait();
            acc[c] = fmaf(scale, __uint_as_float(r0[0]) + __uint_as_float(r1[31]), acc[c]);
          }
        } else {
          acc[0] += scale + __uint_as_float(t_addr & 1u);
        }
        tc_fence_before();
        mbar_arrive(&tempty[a]);
      }
      if (!ok) break;
      // row -> bf16 -> 64-column slabs in the TMA swizzle layout -> bulk tensor stores
      const int y0 = m_blk * BM + q * 32;
#pragma unroll
      for (int sl = 0; sl < 2; ++sl) {
        if (lane == 0) tma_store_wait_read<0>();
        __syncwarp();
        uint8_t* rowp = buf + lane * 128;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          bf16x8 pk;
#pragma unroll
          for (int j = 0; j < 4; ++j)
            pk.v[j] = __floats2bfloat162_rn(acc[sl * 64 + 8 * i + 2 * j], acc[sl * 64 + 8 * i + 2 * j + 1]);
          st_shared8(rowp + ((i ^ (lane & 7)) << 4), pk);
        }
        fence_proxy_async_smem();
        __syncwarp();
        const int x0 = n_blk * BN + half * HALF + sl * 64;
        if (lane == 0 && x0 < p.N && y0 < p.M) tma_store_3d(&tmC, buf, x0, y0, 0);
        if (lane == 0) tma_store_commit();
      }
    }
    if (lane == 0) tma_store_wait<0>();
  }

  tc_fence_before();
  __syncthreads();
  if (p.status != nullptr && *reinterpret_cast<volatile int*>(p.status) != PB_OK) {
    for (int i = 0; i < 2000; ++i) __nanosleep(1000);   // let copies in flight land
    __syncthreads();
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 2 * BN);
  }
}

// ---------------------------------------------------------------------------
// CTA-pair variant: a cluster of two CTAs computes a 256 x 256 tile with tcgen05.mma.cta_group::2, each loading its 128
// rows of A and 128 of the tile's 256 rows of B. A K-block of the single-CTA tile writes 48 KB to shared memory and
// reads them once, 768 clocks of it against 524 of tensor core; the pair's writes and reads 32 KB.
// Bound by the promotion and by handing the accumulators over (about 1090 clocks a K-block). Sixteen promotion warps,
// 64 columns each, so that a scheduler has four of them to hide tensor-memory reads, multiply-adds and waits behind one
// another, with what that takes: 104 registers (at 96, spilled, 8192^3 takes 616 us), eight columns read at a
// time (sixteen: 569 us), scales multiplied when they are used (as soon as they are asked for: 719 us), one arrival a
// warp with the scope of its CTA (released to the cluster 1228 us; what is handed over is tensor memory, which
// tcgen05.fence orders). Single-CTA / pair: 8192^3 705 / 555 us, 16384 x 2816 x 2048 154 / 124, 16384 x 2048 x 1408
// 86 / 70, 5000 x 2816 x 2048 56 / 48, 129 x 2816 x 2048 23.5 / 21.5.
// Row blocks of a pair may belong to two groups: then the pair makes two passes, one for each group's B, and in each the
// CTA whose rows are not of that group drops its half (at most once a group).
// Same arithmetic as the single-CTA kernel, bit for bit.
// ---------------------------------------------------------------------------
constexpr int P_STAGES = 5, P_OP = 128 * BK, P_STAGE = 2 * P_OP;      // A and B: 128 rows of 128 bytes each
constexpr int P_WARPS = 16, P_COLS = 64, P_THREADS = (4 + P_WARPS) * 32;   // warps 0 loads, 1 MMA, 2 and 3 idle
constexpr int P_EPI = P_STAGES * P_STAGE, P_BARS = P_EPI + P_WARPS * 4096, P_SMEM = P_BARS + 256 + 1024;
static_assert(P_SMEM <= 227 * 1024, "one CTA's shared memory");

__global__ void __launch_bounds__(P_THREADS, 1)
gemm_fp8_pair_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                     const __grid_constant__ CUtensorMap tmC, const Params p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + P_BARS);
  uint64_t* full = bars;                    // [P_STAGES], the even CTA's
  uint64_t* empty = bars + P_STAGES;        // [P_STAGES], both
  uint64_t* tfull = bars + 2 * P_STAGES;    // [2], both
  uint64_t* tempty = tfull + 2;             // [2], the even CTA's
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty + 2);

  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int rank = static_cast<int>(cluster_ctarank());   // 0: even CTA (issues the MMAs)
  const int pair = blockIdx.x >> 1, n_pairs = gridDim.x >> 1;
  const int num_m = (p.M + 255) / 256, num_n = (p.N + BN - 1) / BN;
  const int nkb = p.K / BK;
  const int total = num_m * num_n;

  if (threadIdx.x == 0) {
    for (int s = 0; s < P_STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&tfull[a], 1);
      mbar_init(&tempty[a], 2 * P_WARPS);
    }
    fence_barrier_init();
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 2 * BN);   // all columns: one address serves both CTAs
    tmem_relinquish();
  }
  tc_fence_before();
  cluster_sync_all();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  after_previous_kernel();

  // column-major inside groups of 8 pair rows: B tiles stay in L2
  auto coords = [&](int r, int& m_pair, int& n_blk) {
    const int first = (r / (8 * num_n)) * 8;
    const int gsz = min(num_m - first, 8);
    m_pair = first + (r % (8 * num_n)) % gsz;
    n_blk = (r % (8 * num_n)) / gsz;
  };
  const int n_blocks = (p.M + BM - 1) / BM;
  auto group_of = [&](int blk) { return p.mblk_group == nullptr ? 0 : blk < n_blocks ? p.mblk_group[blk] : -1; };
  // the groups whose B a pair of row blocks needs, in order, and this CTA's own (negative: padding)
  struct Passes {
    int first, second, n, own;
    __device__ int operator[](int i) const { return i == 0 ? first : second; }
  };
  auto passes = [&](int m_pair) {
    const int g0 = group_of(2 * m_pair), g1 = group_of(2 * m_pair + 1);
    Passes q;
    q.own = rank == 0 ? g0 : g1;
    q.first = g0 >= 0 ? g0 : g1;
    q.second = g1;
    q.n = (g0 >= 0 ? 1 : 0) + (g1 >= 0 && g1 != g0 ? 1 : 0);
    return q;
  };

  // 640 threads start with 96 registers: 128 x 56 + 512 x 104 are fewer than those 61440
  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
    if (warp == 0 && lane == 0) {
      int s = 0;
      uint32_t ph = 0;
      bool ok = true;
      for (int t = pair; t < total && ok; t += n_pairs) {
        int m_pair, n_blk;
        coords(t, m_pair, n_blk);
        const Passes q = passes(m_pair);
        const int m_blk = 2 * m_pair + rank;
        for (int i = 0; i < q.n && ok; ++i)
          for (int kb = 0; kb < nkb; ++kb) {
            if (!mbar_wait(&empty[s], ph ^ 1, p.status)) { ok = false; break; }
            if (rank == 0) mbar_arrive_expect_tx(&full[s], 2 * P_STAGE);
            const uint32_t bar = cluster_map(smem_u32(&full[s]), 0);
            uint8_t* st = smem + s * P_STAGE;
            tma_load_3d_pair(st, &tmA, bar, kb * BK, m_blk * BM, 0);
            tma_load_3d_pair(st + P_OP, &tmB, bar, kb * BK, n_blk * BN + rank * 128, q[i]);
            if (++s == P_STAGES) { s = 0; ph ^= 1; }
          }
      }
    }
    if (warp == 1 && rank == 0) {
      const uint32_t idesc = make_idesc(0, 0, 256, BN, 0, 0);   // e4m3 x e4m3, both K-major
      constexpr uint64_t HI = static_cast<uint64_t>(sdesc_hi_sw128(1024)) << 32;
      const uint32_t lo0 = sdesc_lo(smem_u32(smem), 16);
      int s = 0;
      uint32_t ph = 0, it = 0;   // it: K-blocks issued so far, picks the accumulator and its phase
      bool ok = true;
      for (int t = pair; t < total && ok; t += n_pairs) {
        int m_pair, n_blk;
        coords(t, m_pair, n_blk);
        const Passes q = passes(m_pair);
        for (int kb = 0; kb < q.n * nkb; ++kb, ++it) {
          const int acc = it & 1;
          if (!mbar_wait_spin_warp(&tempty[acc], ((it >> 1) & 1) ^ 1, p.status) ||
              !mbar_wait_spin_warp(&full[s], ph, p.status)) { ok = false; break; }
          tc_fence_after();
          const uint32_t a_lo = lo0 + s * (P_STAGE >> 4), b_lo = a_lo + (P_OP >> 4);
#pragma unroll
          for (int j = 0; j < BK / 32; ++j)
            umma_f8_pair_warp(tmem_base + acc * BN, HI | (a_lo + 2 * j), HI | (b_lo + 2 * j), idesc, j > 0 ? 1u : 0u);
          umma_commit_pair_warp(&empty[s], 3);
          umma_commit_pair_warp(&tfull[acc], 3);
          if (++s == P_STAGES) { s = 0; ph ^= 1; }
        }
      }
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 104;");
    const int q4 = warp & 3, cg = (warp - 4) >> 2;   // tensor-memory lane quarter, 64-column group
    const int n_sb_rows = (p.N + HALF - 1) / HALF;
    const uint32_t tempty0 = cluster_map(smem_u32(&tempty[0]), 0);
    uint8_t* buf = smem + P_EPI + (warp - 4) * 4096;
    uint32_t it = 0;
    bool ok = true;
    for (int t = pair; t < total && ok; t += n_pairs) {
      int m_pair, n_blk;
      coords(t, m_pair, n_blk);
      const Passes q = passes(m_pair);
      const int y0 = (2 * m_pair + rank) * BM + q4 * 32;
      const float* sa_row = p.sa + min(y0 + lane, p.M - 1);
      for (int i = 0; i < q.n && ok; ++i) {
        const bool mine = q[i] == q.own;
        const float* sb = p.sb + (static_cast<size_t>(q[i]) * n_sb_rows + min(n_blk * 2 + (cg >> 1), n_sb_rows - 1)) * nkb;
        float acc[P_COLS];
#pragma unroll
        for (int c = 0; c < P_COLS; ++c) acc[c] = 0.f;
        float sa_next = 0.f, sb_next = 0.f;   // scales, one K-block ahead
        if (mine) { sa_next = __ldcg(sa_row); sb_next = __ldg(sb); }
        for (int kb = 0; kb < nkb; ++kb, ++it) {
          const int a = it & 1;
          if (!mbar_wait_warp(&tfull[a], (it >> 1) & 1, p.status)) { ok = false; break; }
          tc_fence_after();
          if (mine) {
            const float scale = sa_next * sb_next;
            if (kb + 1 < nkb) {
              sa_next = __ldcg(sa_row + static_cast<size_t>(kb + 1) * p.M);
              sb_next = __ldg(sb + kb + 1);
            }
            const uint32_t t_addr = tmem_base + a * BN + cg * P_COLS + (static_cast<uint32_t>(q4 * 32) << 16);
#pragma unroll
            for (int c = 0; c < P_COLS; c += 8) {
              uint32_t v[8];
              tmem_ld_32x32b_x8(t_addr + c, v);
              tmem_ld_wait();
#pragma unroll
              for (int e = 0; e < 8; e += 2) fma2(acc[c + e], acc[c + e + 1], scale, v[e], v[e + 1]);
            }
          }
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive_peer(tempty0 + a * 8);
        }
        if (!ok || !mine) continue;
        if (lane == 0) tma_store_wait_read<0>();
        __syncwarp();
        uint8_t* rowp = buf + lane * 128;
#pragma unroll
        for (int c = 0; c < 8; ++c) st_shared8(rowp + ((c ^ (lane & 7)) << 4), pack8(acc + 8 * c));
        fence_proxy_async_smem();
        __syncwarp();
        const int x0 = n_blk * BN + cg * P_COLS;
        if (lane == 0 && x0 < p.N && y0 < p.M) tma_store_3d(&tmC, buf, x0, y0, 0);
        if (lane == 0) tma_store_commit();
      }
    }
    if (lane == 0) tma_store_wait<0>();
  }

  tc_fence_before();
  __syncthreads();
  if (p.status != nullptr && *reinterpret_cast<volatile int*>(p.status) != PB_OK) {
    for (int i = 0; i < 2000; ++i) __nanosleep(1000);   // let copies in flight land
  }
  // neither CTA leaves while its peer may still signal its barriers or read its operands
  cluster_sync_all();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 2 * BN);
  }
}

// ------------------------------------------------------------------------------ quantisers
__device__ __forceinline__ uint32_t to_e4m3x4(float a, float b, float c, float d) {
  const __nv_fp8x2_storage_t lo = __nv_cvt_float2_to_fp8x2(make_float2(a, b), __NV_SATFINITE, __NV_E4M3);
  const __nv_fp8x2_storage_t hi = __nv_cvt_float2_to_fp8x2(make_float2(c, d), __NV_SATFINITE, __NV_E4M3);
  return static_cast<uint32_t>(lo) | (static_cast<uint32_t>(hi) << 16);
}

// Every quantiser below gives a warp R consecutive rows x 256 columns: a lane covers 8 consecutive
// columns of each row (one 16-byte access of bf16), 16 lanes one 128-column block, and the R row
// loads are all in flight before the first use. What bounds them is memory once the arithmetic is
// out of the way: a warp per row with one 512-column step at a time left one load latency per step
// exposed, and a compiler division per element (about ten instructions) made the kernels
// issue-bound.
//
// e4m3(x / scale) must round as the correctly rounded quotient does (a reciprocal multiply moves
// some ties). Markstein (1990): with r = RN(1 / s) and q0 = RN(x r), the residual x - q0 s is exact in
// one FMA and RN(q0 + r residual) is RN(x / s): three operations. The range check keeps every
// quotient that does not round to zero clear of underflow and r clear of overflow; other scales
// take the division. The sign of a zero quotient is the numerator's. The tests compare the bytes of all
// 128 x 128 pairs of bf16 significands, at every exponent distance that does not round to zero, with the division's.
struct Quot {
  float s, r;
  bool fast;
  __device__ __forceinline__ explicit Quot(float scale)
      : s(scale), r(1.f / scale), fast(scale > 8.6736174e-19f && scale < 1.1529215e18f) {}
  __device__ __forceinline__ float markstein(float x) const {
    const float q0 = x * r;
    return copysignf(fmaf(fmaf(-q0, s, x), r, q0), x);
  }
  // e4m3 of 8 bf16 values
  __device__ __forceinline__ uint2 operator()(const bf16x8& p) const {
    float f[8];
    unpack8(p, f);
    if (fast) {
#pragma unroll
      for (int j = 0; j < 8; ++j) f[j] = markstein(f[j]);
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) f[j] = __fdiv_rn(f[j], s);
    }
    return make_uint2(to_e4m3x4(f[0], f[1], f[2], f[3]), to_e4m3x4(f[4], f[5], f[6], f[7]));
  }
};
// bf16(e4m3 * scale) of 8 values
__device__ __forceinline__ bf16x8 dequant8(uint2 q, float s) {
  const uint32_t w2[2] = {q.x, q.y};
  float f[8];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const __half2_raw h2 = __nv_cvt_fp8x2_to_halfraw2(
        static_cast<__nv_fp8x2_storage_t>((w2[j >> 1] >> (16 * (j & 1))) & 0xffffu), __NV_E4M3);
    const float2 v = __half22float2(*reinterpret_cast<const __half2*>(&h2));
    f[2 * j] = v.x * s;
    f[2 * j + 1] = v.y * s;
  }
  return pack8(f);
}
// largest magnitude of 8 bf16 values (exact; NaN is ignored, as fmaxf ignores it)
__device__ __forceinline__ bf16 amax8(const bf16x8& p) {
  const __nv_bfloat162 m = __hmax2(__hmax2(__habs2(p.v[0]), __habs2(p.v[1])),
                                   __hmax2(__habs2(p.v[2]), __habs2(p.v[3])));
  return __hmax(__hmax(__low2bfloat16(m), __high2bfloat16(m)), __ushort_as_bfloat16(0));
}
__device__ __forceinline__ float block_scale(float amax) { return amax > 0.f ? amax / 448.f : 1.f; }
__device__ __forceinline__ bf16x8 zero8() {
  bf16x8 z;
#pragma unroll
  for (int j = 0; j < 4; ++j) z.v[j] = __floats2bfloat162_rn(0.f, 0.f);
  return z;
}

// Quantises R rows x 256 columns held one bf16x8 per row and lane (zeros outside the matrix) and
// stores bytes and scales: row0 is the first row, c the lane's first column. Every lane takes part
// in the shuffles; two rows share one as a bf16 pair.
template <int R>
__device__ __forceinline__ void quant_tile(const bf16x8 (&v)[R], int row0, int m_eff, int M, int c, int K,
                                           int lane, uint8_t* __restrict__ q, float* __restrict__ scales) {
  float keep = 1.f;
#pragma unroll
  for (int i = 0; i < R; i += 2) {
    __nv_bfloat162 m = __halves2bfloat162(amax8(v[i]), amax8(v[i + 1]));
#pragma unroll
    for (int o = 1; o < 16; o <<= 1) m = __hmax2(m, __shfl_xor_sync(0xffffffffu, m, o));
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const float scale = block_scale(bf16_to_f32(h ? __high2bfloat16(m) : __low2bfloat16(m)));
      if ((lane & 15) == i + h) keep = scale;
      if (row0 + i + h < m_eff && c < K)
        *reinterpret_cast<uint2*>(q + static_cast<size_t>(row0 + i + h) * K + c) = Quot(scale)(v[i + h]);
    }
  }
  // lane j of a block's 16 holds the scale of row j: R consecutive floats of the table's row
  if ((lane & 15) < R && row0 + (lane & 15) < m_eff && c < K)
    scales[static_cast<size_t>(c >> 7) * M + row0 + (lane & 15)] = keep;
}

constexpr int QR = 8;       // rows of a warp in the plain row kernels
constexpr int QR_SWI = 4;   // two operands per element: half the rows for the same registers

// first row and column group of this warp; column groups of the same rows are neighbours
__device__ __forceinline__ bool warp_tile(int rows_per, int M, int K, int& row0, int& c, int lane) {
  const int ncg = (K + 255) >> 8;
  const long w = (static_cast<long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  row0 = static_cast<int>(w / ncg) * rows_per;
  c = static_cast<int>(w % ncg) * 256 + lane * 8;
  return w < static_cast<long>((M + rows_per - 1) / rows_per) * ncg;
}

// rows_dev (may be null): device-side count of the rows in use; the scale table keeps its row
// stride M whatever that count.
// 73984 x 2048: 132 us -> 100 us (read 2, write 1 byte an element: 4560 GB/s).
__global__ void __launch_bounds__(256) quant_rows_kernel(const bf16* __restrict__ x, long ld, int M,
                                                         int K, uint8_t* __restrict__ q,
                                                         float* __restrict__ scales,
                                                         const int* __restrict__ rows_dev) {
  after_previous_kernel();
  const int lane = threadIdx.x & 31;
  const int m_eff = rows_dev != nullptr ? min(M, *rows_dev) : M;
  int row0, c;
  if (!warp_tile(QR, M, K, row0, c, lane) || row0 >= m_eff) return;
  bf16x8 v[QR];
#pragma unroll
  for (int i = 0; i < QR; ++i)
    v[i] = row0 + i < m_eff && c < K
               ? *reinterpret_cast<const bf16x8*>(x + static_cast<size_t>(row0 + i) * ld + c)
               : zero8();
  quant_tile<QR>(v, row0, m_eff, M, c, K, lane, q, scales);
}

// SwiGLU fused with the row quantiser: h = silu(gate) * up is written as bf16 (the backward
// and the weight gradient of the next product need it) and, from those bf16 values, as e4m3 +
// 1 x 128 scales for the FP8 product that consumes it. One pass over gu instead of a SwiGLU
// pass and a quantiser pass. gu [rows, 2H] (gate | up), H a multiple of 128.
// 73984 rows, H = 1408, no bf16 copy: 199 us -> 194 us (the exponential and the gate's division bound it).
__global__ void __launch_bounds__(256) swiglu_quant_kernel(const bf16* __restrict__ gu,
                                                           bf16* __restrict__ h, int M, int H,
                                                           uint8_t* __restrict__ q,
                                                           float* __restrict__ scales,
                                                           const int* __restrict__ rows_dev) {
  after_previous_kernel();
  const int lane = threadIdx.x & 31;
  const int m_eff = rows_dev != nullptr ? min(M, *rows_dev) : M;
  int row0, c;
  if (!warp_tile(QR_SWI, M, H, row0, c, lane) || row0 >= m_eff) return;
  bf16x8 v[QR_SWI], up[QR_SWI];
#pragma unroll
  for (int i = 0; i < QR_SWI; ++i) {
    const bool in = row0 + i < m_eff && c < H;
    const bf16* src = gu + static_cast<size_t>(row0 + i) * 2 * H + c;
    v[i] = in ? *reinterpret_cast<const bf16x8*>(src) : zero8();
    up[i] = in ? *reinterpret_cast<const bf16x8*>(src + H) : zero8();
  }
#pragma unroll
  for (int i = 0; i < QR_SWI; ++i) {
    float g[8], u[8];
    unpack8(v[i], g);
    unpack8(up[i], u);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float s = 1.f / (1.f + __expf(-g[j]));
      g[j] = g[j] * s * u[j];
    }
    v[i] = pack8(g);   // what the bf16 copy holds is what is quantised, so both forms of h agree
    if (h != nullptr && row0 + i < m_eff && c < H)   // callers that keep only the e4m3 rows pass null
      *reinterpret_cast<bf16x8*>(h + static_cast<size_t>(row0 + i) * H + c) = v[i];
  }
  quant_tile<QR_SWI>(v, row0, m_eff, M, c, H, lane, q, scales);
}

// y[row, :] = bf16(e4m3(q[row, :]) * scale of its 1 x 128 block)
// 73984 x 2048 and 73984 x 1408 together: 475 us -> 122 us; 5000 rows of each: 48 us -> 13 us.
__global__ void __launch_bounds__(256) dequant_rows_kernel(const uint8_t* __restrict__ q,
                                                           const float* __restrict__ scales,
                                                           long ld_s, int M, int K,
                                                           bf16* __restrict__ y,
                                                           const int* __restrict__ rows_dev) {
  after_previous_kernel();
  const int lane = threadIdx.x & 31;
  const int m_eff = rows_dev != nullptr ? min(M, *rows_dev) : M;
  int row0, c;
  if (!warp_tile(QR, M, K, row0, c, lane) || row0 >= m_eff || c >= K) return;   // no shuffles below
  uint2 raw[QR];
  float sc[QR];
#pragma unroll
  for (int i = 0; i < QR; ++i) {
    if (row0 + i < m_eff) {
      raw[i] = *reinterpret_cast<const uint2*>(q + static_cast<size_t>(row0 + i) * K + c);
      sc[i] = scales[static_cast<size_t>(c >> 7) * ld_s + row0 + i];
    }
  }
#pragma unroll
  for (int i = 0; i < QR; ++i)
    if (row0 + i < m_eff)
      *reinterpret_cast<bf16x8*>(y + static_cast<size_t>(row0 + i) * K + c) = dequant8(raw[i], sc[i]);
}

// One CTA (256 threads) per 128 x 128 block of a [N, K] matrix (edges clipped).
// q / scales may be null when only `deq` is wanted. deq (may be null): bf16 [N, K] image of the
// quantised block, e4m3(w / scale) * scale: the operand the FP8 GEMM really multiplied, which is
// what the backward of an FP8 linear differentiates against.
// The block is read once and waits for the block-wide maximum as packed bf16 (32 registers a
// thread, so that four CTAs share an SM and one's loads cover another's arithmetic).
// 66 x (2816 x 2048 + 2048 x 1408), quantised and fake-quantised: 1372 us -> 674 us (610 at the copy rate).
__global__ void __launch_bounds__(256, 4)
quant_blocks_kernel(const bf16* __restrict__ w, long ld, int N, int K, uint8_t* __restrict__ q,
                    float* __restrict__ scales, bf16* __restrict__ deq) {
  after_previous_kernel();
  __shared__ float red[33];
  const int nb = blockIdx.y, kb = blockIdx.x;
  const int r0 = nb * 128 + (threadIdx.x >> 4), c = kb * 128 + (threadIdx.x & 15) * 8;
  const bool vec_ok = (ld % 8) == 0 && (reinterpret_cast<uintptr_t>(w) & 15) == 0;
  bf16x8 v[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int r = r0 + 16 * i;
    v[i] = zero8();
    if (r < N) {                               // K is a multiple of 128: the 8 columns are in range
      const bf16* src = w + static_cast<size_t>(r) * ld + c;
      if (vec_ok) {
        v[i] = *reinterpret_cast<const bf16x8*>(src);
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) v[i].v[j] = __halves2bfloat162(src[2 * j], src[2 * j + 1]);
      }
    }
  }
  bf16 m = amax8(v[0]);
#pragma unroll
  for (int i = 1; i < 8; ++i) m = __hmax(m, amax8(v[i]));
  const float scale = block_scale(block_max(bf16_to_f32(m), red));
  const Quot quot(scale);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int r = r0 + 16 * i;
    if (r >= N) continue;
    const uint2 pk = quot(v[i]);
    if (q != nullptr) *reinterpret_cast<uint2*>(q + static_cast<size_t>(r) * K + c) = pk;
    if (deq != nullptr)
      *reinterpret_cast<bf16x8*>(deq + static_cast<size_t>(r) * K + c) = dequant8(pk, scale);
  }
  if (threadIdx.x == 0 && scales != nullptr) scales[static_cast<size_t>(nb) * gridDim.x + kb] = scale;
}

// blocks of 8 warps that cover M rows, rows_per of them and 256 columns to a warp
inline unsigned tile_grid(int rows_per, int M, int K) {
  const long warps = static_cast<long>((M + rows_per - 1) / rows_per) * ((K + 255) / 256);
  return static_cast<unsigned>((warps + 7) / 8);
}

}  // namespace f8
}  // namespace pb

using namespace pb;

// x [M, K] bf16 (row stride ld, K % 128 == 0) -> q [M, K] e4m3, scales [K / 128, M] fp32.
PB_API int pb_fp8_quant_rows(const void* x, long ld, int M, int K, void* q, float* scales,
                             cudaStream_t st) {
  if (M <= 0 || K <= 0 || K % 128 != 0 || ld % 8 != 0 || (reinterpret_cast<uintptr_t>(x) & 15) != 0)
    return PB_BAD_ARG;
  pb::launch(f8::quant_rows_kernel, f8::tile_grid(f8::QR, M, K), 256, 0, st,
      static_cast<const bf16*>(x), ld, M, K, static_cast<uint8_t*>(q), scales, nullptr);
  return static_cast<int>(cudaGetLastError());
}
// The same over the first min(M, *rows_dev) rows (rows_dev: a device int).
PB_API int pb_fp8_quant_rows_dyn(const void* x, long ld, int M, int K, void* q, float* scales,
                                 const int* rows_dev, cudaStream_t st) {
  if (M <= 0 || K <= 0 || K % 128 != 0 || ld % 8 != 0 || (reinterpret_cast<uintptr_t>(x) & 15) != 0)
    return PB_BAD_ARG;
  pb::launch(f8::quant_rows_kernel, f8::tile_grid(f8::QR, M, K), 256, 0, st,
      static_cast<const bf16*>(x), ld, M, K, static_cast<uint8_t*>(q), scales, rows_dev);
  return static_cast<int>(cudaGetLastError());
}

// h [M, H] bf16 = silu(gu[:, :H]) * gu[:, H:], and its e4m3 rows q [M, H] with scales
// [H / 128, M], in one pass. H a multiple of 128; rows_dev (may be null): device row count.
PB_API int pb_swiglu_quant(const void* gu, void* h, int M, int H, void* q, float* scales,
                           const int* rows_dev, cudaStream_t st) {
  if (M <= 0 || H <= 0 || H % 128 != 0) return PB_BAD_ARG;
  pb::launch(f8::swiglu_quant_kernel, f8::tile_grid(f8::QR_SWI, M, H), 256, 0, st,
      static_cast<const bf16*>(gu), static_cast<bf16*>(h), M, H, static_cast<uint8_t*>(q), scales,
      rows_dev);
  return static_cast<int>(cudaGetLastError());
}

// q [M, K] e4m3 with scales [K / 128, ld_s] (ld_s >= M: the row stride of the scale table)
// -> y [M, K] bf16. The straight-through backward of an FP8 product uses these values.
PB_API int pb_fp8_dequant_rows(const void* q, const float* scales, long ld_s, int M, int K, void* y,
                               const int* rows_dev, cudaStream_t st) {
  if (M <= 0 || K <= 0 || K % 128 != 0 || ld_s < M) return PB_BAD_ARG;
  pb::launch(f8::dequant_rows_kernel, f8::tile_grid(f8::QR, M, K), 256, 0, st,
      static_cast<const uint8_t*>(q), scales, ld_s, M, K, static_cast<bf16*>(y), rows_dev);
  return static_cast<int>(cudaGetLastError());
}

// w [groups * N, K] bf16 (K % 128 == 0, N % 128 == 0 when groups > 1) -> q e4m3 same shape,
// scales [groups * ceil(N / 128), K / 128].
PB_API int pb_fp8_quant_blocks(const void* w, long ld, int rows, int K, void* q, float* scales,
                               cudaStream_t st) {
  if (rows <= 0 || K <= 0 || K % 128 != 0 || ld % 4 != 0) return PB_BAD_ARG;
  dim3 grid(K / 128, (rows + 127) / 128);
  pb::launch(f8::quant_blocks_kernel, grid, 256, 0, st, static_cast<const bf16*>(w), ld, rows, K,
                                                static_cast<uint8_t*>(q), scales, nullptr);
  return static_cast<int>(cudaGetLastError());
}

// out [rows, K] bf16 = the 128 x 128 block quantisation of w applied and undone (e4m3 rounding at
// the block's scale): the weight an FP8 linear really used. Same shape rules as
// pb_fp8_quant_blocks.
PB_API int pb_fp8_fakequant_blocks(const void* w, long ld, int rows, int K, void* out,
                                   cudaStream_t st) {
  if (rows <= 0 || K <= 0 || K % 128 != 0 || ld % 4 != 0 || out == nullptr) return PB_BAD_ARG;
  dim3 grid(K / 128, (rows + 127) / 128);
  pb::launch(f8::quant_blocks_kernel, grid, 256, 0, st, static_cast<const bf16*>(w), ld, rows, K, nullptr,
                                                nullptr, static_cast<bf16*>(out));
  return static_cast<int>(cudaGetLastError());
}

namespace pb {
namespace f8 {
// Whether a product runs on CTA pairs. Ungrouped they are the faster way at every size beyond one tile of the other
// kernel, equal within a microsecond where the contraction is 512 or less (above, and 1000 x 2816 x 2048 24.6 / 23.5 us,
// 4096 x 2048 x 1408 31.8 / 27.6, 1024 x 1024 x 512 13.4 / 14.4, 4096 x 512 x 256 13.2 / 13.2). With groups, every
// second group boundary costs a pass of which half is dropped; single / pair at row blocks a group, N = 2816,
// K = 2048: 3.9 blocks 290 / 309 us, 6.2 133 / 135, 8.2 584 / 534, 16 159 / 136. Rows that peers are still
// storing, and limited grids, stay on one CTA.
static bool takes_pairs(int M, int N, int groups, const Params& p, int max_ctas) {
  return M > BM && N > HALF && (max_ctas <= 0 || max_ctas >= num_sms()) && p.blk_arrived == nullptr &&
         (p.mblk_group == nullptr || (M + BM - 1) / BM >= 8L * groups);
}
static int launch_pair(const CUtensorMap& tmA, const CUtensorMap& tmB, const CUtensorMap& tmC, const Params& p,
                       cudaStream_t st) {
  static pb::DeviceOnce attr_once;   // per device: the attribute belongs to the current GPU
  static int max_pairs = 0;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;   // as pb::launch
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.blockDim = dim3(P_THREADS, 1, 1);
  cfg.dynamicSmemBytes = P_SMEM;
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  if (attr_once.need()) {
    cudaError_t e = cudaFuncSetAttribute(gemm_fp8_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, P_SMEM);
    if (e != cudaSuccess) return static_cast<int>(e);
    cfg.gridDim = dim3(num_sms() & ~1, 1, 1);
    int n = 0;
    e = cudaOccupancyMaxActiveClusters(&n, gemm_fp8_pair_kernel, &cfg);
    if (e != cudaSuccess) { cudaGetLastError(); n = num_sms() / 2; }
    max_pairs = n > 0 && n < num_sms() / 2 ? n : num_sms() / 2;
    attr_once.done();
  }
  const long tiles = static_cast<long>((p.M + 255) / 256) * ((p.N + BN - 1) / BN);
  cfg.gridDim = dim3(static_cast<unsigned>(2 * (tiles < max_pairs ? tiles : max_pairs)), 1, 1);
  const cudaError_t e = cudaLaunchKernelEx(&cfg, gemm_fp8_pair_kernel, tmA, tmB, tmC, p);
  return static_cast<int>(e != cudaSuccess ? e : cudaGetLastError());
}
}  // namespace f8
}  // namespace pb

// C [M, N] bf16 = block-scaled Aq [M, K] x Bq [groups, N, K]^T. K % 128 == 0, N % 8 == 0.
// sa [K / 128, M]; sb [groups, ceil(N / 128), K / 128]; mblk_group null (groups == 1) or one
// int per 128-row block of A / C.
template <int PROBE = 0>
static int gemm_fp8_launch(const void* Aq, const float* sa, const void* Bq, const float* sb,
                           void* C, int M, int N, int K, int groups, long ldc,
                           const int* mblk_group, int* status, int max_ctas,
                           const uint32_t* blk_arrived, const int* blk_expect, long budget_ns,
                           cudaStream_t st);

PB_API int pb_gemm_fp8_blockscaled(const void* Aq, const float* sa, const void* Bq, const float* sb,
                                   void* C, int M, int N, int K, int groups, long ldc,
                                   const int* mblk_group, int* status, int max_ctas,
                                   cudaStream_t st) {
  return gemm_fp8_launch(Aq, sa, Bq, sb, C, M, N, K, groups, ldc, mblk_group, status, max_ctas,
                         nullptr, nullptr, 0, st);
}

// The grouped product fused with the arrival of its rows: Aq / sa are a receive buffer that the
// other ranks' dispatch kernels are still filling. blk_arrived (uint32 per 128-row block, in
// memory the senders can reach, zero before the senders start) is incremented once per landed
// row; blk_expect (int per block) is the number of rows each block will receive. A row block is
// loaded only when complete; a block that does not complete within budget_ns latches
// PB_TIMEOUT_FLAG in *status and the kernel drains.
PB_API int pb_gemm_fp8_grouped_arrive(const void* Aq, const float* sa, const void* Bq, const float* sb,
                                      void* C, int M, int N, int K, int groups, long ldc,
                                      const int* mblk_group, const void* blk_arrived,
                                      const int* blk_expect, long budget_ns, int* status,
                                      cudaStream_t st) {
  if (blk_arrived == nullptr || blk_expect == nullptr || budget_ns <= 0 || mblk_group == nullptr)
    return PB_BAD_ARG;
  return gemm_fp8_launch(Aq, sa, Bq, sb, C, M, N, K, groups, ldc, mblk_group, status, 0,
                         static_cast<const uint32_t*>(blk_arrived), blk_expect, budget_ns, st);
}

#ifdef PB_DEBUG_BOUNDS
// Debug build only: the timing probes of gemm_fp8_kernel (1 no promotion, 2 accumulation in
// place, 3 FMAs only, 4 tensor-memory loads only). C receives values that are not the product.
PB_API int pb_gemm_fp8_probe(const void* Aq, const float* sa, const void* Bq, const float* sb,
                             void* C, int M, int N, int K, long ldc, int probe, int* status,
                             cudaStream_t st) {
  switch (probe) {
    case 1: return gemm_fp8_launch<1>(Aq, sa, Bq, sb, C, M, N, K, 1, ldc, nullptr, status, 0, nullptr, nullptr, 0, st);
    case 2: return gemm_fp8_launch<2>(Aq, sa, Bq, sb, C, M, N, K, 1, ldc, nullptr, status, 0, nullptr, nullptr, 0, st);
    case 3: return gemm_fp8_launch<3>(Aq, sa, Bq, sb, C, M, N, K, 1, ldc, nullptr, status, 0, nullptr, nullptr, 0, st);
    case 4: return gemm_fp8_launch<4>(Aq, sa, Bq, sb, C, M, N, K, 1, ldc, nullptr, status, 0, nullptr, nullptr, 0, st);
    default: return PB_BAD_ARG;
  }
}
#endif

template <int PROBE>
static int gemm_fp8_launch(const void* Aq, const float* sa, const void* Bq, const float* sb,
                           void* C, int M, int N, int K, int groups, long ldc,
                           const int* mblk_group, int* status, int max_ctas,
                           const uint32_t* blk_arrived, const int* blk_expect, long budget_ns,
                           cudaStream_t st) {
  using namespace f8;
  if (M <= 0 || N <= 0 || K <= 0 || K % BK != 0 || groups <= 0 || (ldc * 2) % 16 != 0)
    return PB_BAD_ARG;
  if (groups > 1 && (mblk_group == nullptr || N % HALF != 0)) return PB_BAD_ARG;
  if (groups == 1 && blk_arrived != nullptr && N % HALF != 0) return PB_BAD_ARG;
  if ((reinterpret_cast<uintptr_t>(Aq) & 15) || (reinterpret_cast<uintptr_t>(Bq) & 15) ||
      (reinterpret_cast<uintptr_t>(C) & 15))
    return PB_BAD_ARG;
  static pb::DeviceOnce attr_once;   // per device: the attribute belongs to the current GPU
  if (attr_once.need()) {
    cudaError_t e = cudaFuncSetAttribute(gemm_fp8_kernel<PROBE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         SMEM_TOTAL);
    if (e != cudaSuccess) return static_cast<int>(e);
    attr_once.done();
  }
  Params p;
  p.M = M; p.N = N; p.K = K;
  p.sa = sa; p.sb = sb; p.mblk_group = mblk_group; p.status = status;
  p.blk_arrived = blk_arrived; p.blk_expect = blk_expect;
  p.wait_budget_ns = static_cast<uint64_t>(budget_ns);
  const bool pair = PROBE == 0 && takes_pairs(M, N, groups, p, max_ctas);
  CUtensorMap tmA, tmB, tmC;
  int r = make_tmap_3d(&tmA, Aq, 1, K, M, 1, K, 0, BK, BM);
  if (r != 0) return 1000 + r;
  r = make_tmap_3d(&tmB, Bq, 1, K, N, groups, K, static_cast<uint64_t>(N) * K, BK, pair ? 128 : BN);
  if (r != 0) return 2000 + r;
  r = make_tmap_3d(&tmC, C, 2, N, M, 1, ldc, 0, 64, 32);
  if (r != 0) return 3000 + r;
  if (pair) return launch_pair(tmA, tmB, tmC, p, st);
  const long tiles = static_cast<long>((M + BM - 1) / BM) * ((N + BN - 1) / BN);
  int grid = num_sms();
  if (max_ctas > 0 && max_ctas < grid) grid = max_ctas;
  if (tiles < grid) grid = static_cast<int>(tiles);
  pb::launch(gemm_fp8_kernel<PROBE>, grid, THREADS, SMEM_TOTAL, st, tmA, tmB, tmC, p);
  return static_cast<int>(cudaGetLastError());
}
