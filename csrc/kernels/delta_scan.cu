// Chunked delta-rule state scan on tcgen05 (sm_100a), forward and backward.
//
// The chunk-local WY operands (W = T b K, U^ = T b V, M = tril(Q K^T)) do not depend
// on the running state; what is sequential is, per (batch, head), the walk over
// chunks of 64 tokens with the 128 x 128 fp32 state S:
//
//   forward   Y = W S            U = U^ - Y          O = Q S + M U      S += K^T U
//   backward  dU = M^T dO + K dS                     dS += Q^T dO - W^T dU
//
// A CTA walks one (batch, head) sequence, or one segment of it, with all 128 columns of the state or with 64. The
// state lives in tensor memory for the whole walk (fp32, 128 lanes); every product is a tcgen05.mma with
// M = 128, N = its columns; the bf16 image of the state and of U that the MMAs consume as
// their B operand is rewritten in shared memory each chunk in the 128-byte-swizzled
// layout TMA itself produces; Q/K/W/M and U^ (or dO) tiles arrive by TMA through a
// ring of two or three stages, and every output leaves by a TMA store from shared memory. Tiles with 64 token rows
// are used as 128-row A operands: the upper 64 accumulator rows are then meaningless and are never read. In the forward
// walk they are Q: W and Q are one operand of 128 rows, so that Y and O take eight products instead of sixteen (16
// sequences of 256 chunks 288 -> 272 us, 283 -> 259 where nothing is kept), and the warps without rows of Y stage O's.
//
// The walk is a serial chain per chunk (state image -> Y -> U -> state update), so its length is
// what counts, not throughput. Eight row warps share the conversions (two per tensor-memory lane
// quarter, 64 columns each); the state update is issued before the output product and has its own
// barrier; the output accumulator is double-buffered, so chunk n's output rows are staged while
// chunk n + 1's Y product runs; the part of the backward's Y that does not need the state is issued
// before the state image is ready. 64 sequences of 64 chunks: forward 96 us (1.5 us a chunk), backward 86 us, which is 5.1
// and 5.7 TB/s; 16 of 256 chunks 272 and 256 us. Four row warps that did all of it in order, in one CTA a sequence, took
// 230 and 133 us. What a chunk takes is the products' chain and the shared memory that they and the conversions share.
//
// The columns of the state never mix (U, O and dU have the same columns), so when the sequences or
// segments take at most half of the SMs, two CTAs walk each of them with 64 columns: the conversions
// and products between two waits are half as long. A forward walk that keeps the states stops eight sequences earlier, at 66 on
// 148 SMs, where its stores are what it waits for (figures at the rule in launch()). On both sides of the line, 64 chunks
// each: 74 sequences with 64 columns a CTA 79 us forward (nothing kept) and 104 us backward, 75 sequences with 128 columns 105
// and 110 us. With more CTAs than SMs it would be two waves of a chain that is not half as long.
//
// A forward summary walks every segment twice, once per map, over the same W and K. When the two CTAs a
// segment that takes are more than the SMs, one CTA does both, as two independent chains whose conversions
// and products fall into each other's waits: one wave and half of the operand reads. 16 sequences x 8
// segments x 32 chunks: 69 us; when it was built 86 us, against 104 us as two waves of a CTA for each map and 120 us as
// one chain of 256 columns, whose conversions and products take turns. With a CTA for each map on SMs of their own a chain is the
// shorter, so up to half of the SMs it stays so: 72 segments of 32 chunks 62 us, 80 segments in a CTA each 87 us.
// The initial state is read 16 bytes at a time: element by element the walk of those segments, 70 us, takes 6 us more.
//
// warps 0-7: tensor-memory <-> registers <-> shared/global (lane = state row or token)
// warp 8   : MMA issue                     warp 9: TMA producer (one lane)
// (two chains: 0-15 rows, 16 and 17 MMA issue, 18 TMA)
//
// Reference semantics: kernels/__init__.py:357-376 (per-token recurrence, post-update
// read) of the reference; the chunked algebra is this library's own.
#include <cuda.h>

#include "common.cuh"

namespace pb {

int make_tmap_3d(CUtensorMap* tm, const void* base, int elem_bytes, uint64_t inner,
                 uint64_t outer, uint64_t batch, uint64_t ld_elems, uint64_t batch_stride_elems,
                 uint32_t box_inner, uint32_t box_outer);
int num_sms();

namespace dscan {

constexpr int C = 64;    // tokens per chunk
constexpr int D = 128;   // head dim (keys and values)
constexpr int TMEM_COLS = 512;
constexpr uint32_t COL_X = 0;

struct Params {
  int n_chunks;        // chunks per sequence
  int n_seq;           // batch * heads
  int n_seg;           // segments per sequence: CTA (seq, seg) walks n_chunks / n_seg chunks from
                       //   x_init[seq * n_seg + seg] and leaves x_final[seq * n_seg + seg]
  int summary;         // 1: only the segment's affine map is wanted. Nothing but x_final is
                       //   written, the output products are skipped. Forward walks twice per
                       //   segment, in two CTAs (NC 128) or as the two chains of one (NC 256): from
                       //   zero (x_final <- R, the state the segment adds), and from the identity
                       //   with U^ = 0 (p_final <- P, the linear part). Backward only the first
                       //   (its linear part is P^T).
  float* p_final;      // [n_seq * n_seg, 128, 128], summary forward only
  int heads;           // > 0: Q, K, O and dO live in [batch, seq_len, ld] (head h at columns 128 h)
                       //      instead of the per-chunk layout; rows past seq_len in the last chunk
                       //      read as zeros and are not stored
  int store_ux;        // 0: U and the bf16 states are not wanted (nothing will run backward)
  const float* x_init; // [n_seq, 128, 128] or null (zeros)
  float* x_final;      // [n_seq, 128, 128] or null
  int* status;
};

// NC: state columns of a CTA. 128, or 64 (then two CTAs per segment, not in summary mode), or 256: both
// maps of a forward summary as two chains of 128 columns (0: R, 1: P), each with its own row warps, MMA
// warp and barriers, over the same W and K tiles; no Q, M and output staging.
template <int NC>
struct Shape {
  static constexpr bool BOTH = NC == 256;
  static constexpr int CHAINS = BOTH ? 2 : 1;
  static constexpr int CC = NC / CHAINS;                    // columns of a chain, and of each of its
  static constexpr int WC = CC / 2;                         //   eight row warps
  static constexpr int ROW_WARPS = 8 * CHAINS;
  static constexpr int THREADS = (ROW_WARPS + CHAINS + 1) * 32;
  static constexpr uint32_t COL_Y = BOTH ? 256 : 128, COL_O = 256;   // COL_O: two buffers of 128
  // Tiles sized for 64 columns leave room for a third stage, which hides the latency that memory has when many CTAs read
  // and write it. Two / three, 64 chunks, us: forward 16 sequences 79 / 72, 48 98 / 80, 64 112 / 98; backward 74 / 68, 88 / 73,
  // 99 / 86.
  // a stage: W, Q, K (16 KB each), M (8 KB), U^ or dO (16 KB). W's second half is followed by at
  // least 8 KB of the stage: as a 128-row A operand its upper rows are read from there.
  static constexpr int TILE_W = 0, TILE_Q = 16384, TILE_K = BOTH ? 16384 : 32768, TILE_M = 49152,
                       TILE_DO = BOTH ? 32768 : 57344, STAGE = TILE_DO + (NC == 64 ? 8192 : 16384);
  static constexpr int STAGES = NC == 64 ? 3 : 2;
  static constexpr int XB = STAGES * STAGE;
  static constexpr int UB = XB + 256 * NC;                  // state image, U and output staging: 128, 64 and 64 rows of NC
  static constexpr int OB = UB + 128 * NC;
  static constexpr int BARS = OB + (BOTH ? 0 : 128 * NC);
  static constexpr int TOTAL = BARS + 256 + 1024;
  static_assert(TOTAL <= 227 * 1024, "shared memory of a CTA");
};

template <bool BWD, int NC>
__global__ void __launch_bounds__(Shape<NC>::THREADS, 1)
delta_scan_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmQ,
                  const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmM,
                  const __grid_constant__ CUtensorMap tmDO, const __grid_constant__ CUtensorMap tmXB,
                  const __grid_constant__ CUtensorMap tmU, const __grid_constant__ CUtensorMap tmO,
                  const Params p) {
  using S = Shape<NC>;
  static_assert(!(BWD && S::BOTH), "both maps at once: forward summary only");
  constexpr int TILE_W = S::TILE_W, TILE_Q = S::TILE_Q, TILE_K = S::TILE_K, TILE_M = S::TILE_M, TILE_DO = S::TILE_DO;
  constexpr uint32_t COL_Y = S::COL_Y, COL_O = S::COL_O;
  // Forward walk: W and Q of a 64-column half lie one behind the other, 128 rows of one A operand, so that Y and O are one
  // product: Y in lanes 0 .. 63 and O in lanes 64 .. 127 of the output's buffer. (The backward's K, and W alone where a
  // summary wants no O, run as 128-row operands whose upper lanes are never read.)
  constexpr bool STACK = !BWD && !S::BOTH;
  constexpr int MMA_WARP = S::ROW_WARPS, TMA_WARP = MMA_WARP + S::CHAINS;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int chain = !S::BOTH ? 0 : (warp < MMA_WARP ? warp >> 3 : warp == MMA_WARP + 1);
  uint8_t* xb = smem + S::XB + chain * 32768;
  uint8_t* ub = smem + S::UB + chain * 16384;
  uint8_t* ob = smem + S::OB;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + S::BARS);
  constexpr int STAGES = S::STAGES;
  uint64_t* full = bars;          // [STAGES]
  uint64_t* empty = bars + 3;     // [STAGES]
  uint64_t* chain_bars = bars + 6 + 4 * chain;
  uint64_t* x_ready = chain_bars;
  uint64_t* y_done = chain_bars + 1;
  uint64_t* u_ready = chain_bars + 2;
  uint64_t* x_done = chain_bars + 3;    // the state update of a chunk
  // [2], by output buffer: a chunk's output product (forward). One barrier for both would be two phases ahead of a warp that
  // stages rows after U.
  uint64_t* o_done = bars + 6 + 4 * S::CHAINS;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(o_done + 2);

  const int n_units = p.n_seq * p.n_seg;
  constexpr int HALVES = NC == 64 ? 1 : 2;   // 64-column chunks of U^, dO and the outputs
  constexpr int WC = S::WC;                  // columns of a row warp
  const int half = static_cast<int>(blockIdx.x) / n_units;      // 1: the identity-start CTA, or the upper columns
  const int unit = static_cast<int>(blockIdx.x) % n_units;      // seq * n_seg + seg
  const int col0 = NC == 64 ? half * 64 : 0;                    // this CTA's first state column
  const int seq = unit / p.n_seg;
  const int N = p.n_chunks / p.n_seg;                           // chunks this CTA walks
  const int n0 = (unit % p.n_seg) * N;                          // its first chunk
  const int NT = p.n_chunks;
  const bool sum = S::BOTH || p.summary != 0;
  // linear part (U^ = 0): the second chain, or the identity-start CTA
  const bool lin = S::BOTH ? chain == 1 : NC == 128 && sum && half == 1;
  const bool store_ux = !sum && p.store_ux != 0;
  const bool tokmaj = p.heads > 0;
  // token tensors: batch entry, first row and first column of this sequence
  const int tb = tokmaj ? seq / p.heads : 0;
  const int tok0 = tokmaj ? 0 : seq * NT * C;
  const int tx = tokmaj ? (seq % p.heads) * D : 0;

  if (threadIdx.x == 0) {
#pragma unroll
    for (int s = 0; s < STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], S::CHAINS); }
#pragma unroll
    for (int c = 0; c < S::CHAINS; ++c) {
      uint64_t* b = bars + 6 + 4 * c;
      mbar_init(b, 8); mbar_init(b + 2, 4);   // x_ready, u_ready: one arrival per warp that takes part
      mbar_init(b + 1, 1); mbar_init(b + 3, 1);
    }
    mbar_init(&o_done[0], 1); mbar_init(&o_done[1], 1);
    fence_barrier_init();
    tma_prefetch_desc(&tmW); tma_prefetch_desc(&tmQ); tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmM);
    tma_prefetch_desc(&tmDO);
  }
  if (warp == MMA_WARP) {
    tmem_alloc(tmem_slot, TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot + chain * 128;
  after_previous_kernel();

  if (warp == TMA_WARP) {
    // ------------------------------- TMA producer -------------------------------
    if (lane == 0) {
      // a forward summary needs neither Q nor M (no output product), its linear half no U^
      const bool need_qm = BWD || !sum;
      const bool need_fifth = BWD || S::BOTH || !lin;
      const uint32_t stage_tx = 32768u + (need_qm ? 24576u : 0u) + (need_fifth ? HALVES * 8192u : 0u);
      for (int it = 0; it < N; ++it) {
        const int n = n0 + (BWD ? (N - 1 - it) : it);
        const int s = it % STAGES;
        const uint32_t ph = (it / STAGES) & 1;
        if (!mbar_wait(&empty[s], ph ^ 1, p.status)) break;
        mbar_arrive_expect_tx(&full[s], stage_tx);
        uint8_t* st = smem + s * S::STAGE;
        const int row = (seq * NT + n) * C;
        const int trow = tok0 + n * C;
        tma_load_3d(st + TILE_W, &tmW, &full[s], 0, row, 0);
        tma_load_3d(st + TILE_W + (STACK ? 16384 : 8192), &tmW, &full[s], 64, row, 0);
        tma_load_3d(st + TILE_K, &tmK, &full[s], tx, trow, tb);
        tma_load_3d(st + TILE_K + 8192, &tmK, &full[s], tx + 64, trow, tb);
        if (need_qm) {
          tma_load_3d(st + (STACK ? TILE_W + 8192 : TILE_Q), &tmQ, &full[s], tx, trow, tb);
          tma_load_3d(st + (STACK ? TILE_W + 24576 : TILE_Q + 8192), &tmQ, &full[s], tx + 64, trow, tb);
          tma_load_3d(st + TILE_M, &tmM, &full[s], 0, row, 0);
        }
        if (BWD) {
#pragma unroll
          for (int hf = 0; hf < HALVES; ++hf)
            tma_load_3d(st + TILE_DO + hf * 8192, &tmDO, &full[s], tx + col0 + hf * 64, trow, tb);
        } else if (need_fifth) {
#pragma unroll
          for (int hf = 0; hf < HALVES; ++hf)
            tma_load_3d(st + TILE_DO + hf * 8192, &tmDO, &full[s], col0 + hf * 64, row, 0);
        }
      }
    }
  } else if (warp >= MMA_WARP) {
    // -------------------------------- MMA issuer --------------------------------
    {
      const uint32_t id_kn = make_idesc(1, 1, 128, S::CC, 0, 1);  // A K-major, B MN-major
      const uint32_t id_nn = make_idesc(1, 1, 128, S::CC, 1, 1);  // A MN-major, B MN-major
      // descriptor words made once: an issue is one add for each operand
      const uint32_t xb_mn = sdesc_lo(smem_u32(xb), 16384), ub_mn = sdesc_lo(smem_u32(ub), 8192);
      const uint32_t st_k = sdesc_lo(smem_u32(smem), 16), st_mn = sdesc_lo(smem_u32(smem), 8192);
      for (int it = 0; it < N; ++it) {
        const int s = it % STAGES;
        const uint32_t ph = (it / STAGES) & 1, cph = it & 1;
        auto k_major = [&](int tile) { return st_k + ((s * S::STAGE + tile) >> 4); };
        auto mn_major = [&](int tile) { return st_mn + ((s * S::STAGE + tile) >> 4); };
        const uint32_t col_o = tmem + COL_O + (it & 1) * 128;
        if (!mbar_wait_spin_warp(&full[s], ph, p.status)) break;
        if (BWD) {
          // Y = M^T dO: the previous Y was in registers before its u_ready
          tc_fence_after();
#pragma unroll
          for (int j = 0; j < 4; ++j)
            umma_f16_lo_warp(tmem + COL_Y, step_mn(mn_major(TILE_M), j), step_mn(mn_major(TILE_DO), j), id_nn, j > 0);
        }
        if (!mbar_wait_spin_warp(x_ready, cph, p.status)) break;
        tc_fence_after();
        if (!BWD) {
          // Y = W X, and with W and Q stacked O = Q X too. The buffer's previous rows (chunk it - 2) were staged before
          // this x_ready
#pragma unroll
          for (int j = 0; j < 8; ++j)
            umma_f16_lo_warp(STACK ? col_o : tmem + COL_Y,
                             STACK ? k_major(TILE_W) + (((j >> 2) * 16384 + (j & 3) * 32) >> 4) : step_k(k_major(TILE_W), j),
                             step_mn(xb_mn, j), id_kn, j > 0);
          umma_commit_warp(y_done);
        } else {
          // Y += K X
#pragma unroll
          for (int j = 0; j < 8; ++j)
            umma_f16_lo_warp(tmem + COL_Y, step_k(k_major(TILE_K), j), step_mn(xb_mn, j), id_kn, 1);
          umma_commit_warp(y_done);
          // X += Q^T dO   (independent of dU: keeps the tensor core busy meanwhile)
#pragma unroll
          for (int j = 0; j < 4; ++j)
            umma_f16_lo_warp(tmem + COL_X, step_mn(mn_major(TILE_Q), j), step_mn(mn_major(TILE_DO), j), id_nn, 1);
        }
        if (!mbar_wait_spin_warp(u_ready, cph, p.status)) break;
        tc_fence_after();
        // X += K^T U  (forward), X += W^T (-dU)  (backward): what the next chunk waits for
#pragma unroll
        for (int j = 0; j < 4; ++j)
          umma_f16_lo_warp(tmem + COL_X, step_mn(mn_major(BWD ? TILE_W : TILE_K), j), step_mn(ub_mn, j), id_nn, 1);
        umma_commit_warp(x_done);
        if (!BWD && !sum) {
          // O += M U: M in the upper 64 rows; what the lower ones add to Y's lanes is never read
#pragma unroll
          for (int j = 0; j < 4; ++j)
            umma_f16_lo_warp(col_o, step_k(k_major(TILE_M) - (8192 >> 4), j), step_mn(ub_mn, j), id_kn, 1);
          umma_commit_warp(&o_done[it & 1]);
        }
        umma_commit_warp(&empty[s]);
      }
    }
  } else {
    // ------------------------- state / token row threads -------------------------
    // Every result leaves through shared memory and a TMA store (coalesced, asynchronous):
    // the bf16 state image is stored from the very tile the MMAs read, U / -dU from the
    // operand tile, O from a staging tile. Thread 0 issues and tracks the stores.
    const int r = (warp & 3) * 32 + lane;  // tensor-memory lane = state row (or token row < 64)
    const int ch = (warp >> 2) & 1, c0 = ch * WC;   // this warp's half of the chain's columns
    const int g0 = col0 + c0;                 // its first column in the state or map
    const bool tok_warp = (warp & 3) < 2;     // warps whose lanes are token rows
    const uint32_t lane_addr = tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16) + c0;
    auto sync_rows = [] { asm volatile("bar.sync 1, 256;" ::: "memory"); };
    auto sync_tok = [] { asm volatile("bar.sync 2, 128;" ::: "memory"); };
    // A lane whose wait ran out waits no more but stays in the loop to its end: whoever shares a barrier or a
    // collective instruction with it finds it there, and what is computed and stored meanwhile is reported as
    // invalid by the status word. 16 sequences x 8 segments x 32 chunks: 70.4 us, as with lanes that leave one by one
    // (69.9); a vote after each wait 72.5 us, and barriers that carry the result as well 75.5 us.
    bool ok = true;
    auto wait = [&](uint64_t* bar, uint32_t parity) {
      if (ok) ok = mbar_wait_spin(bar, parity, p.status);
      __syncwarp();   // lanes leave the spin one by one
      tc_fence_after();
    };
    auto arrive = [&](uint64_t* bar) {   // the warp's shared-memory writes and tensor-memory reads are done
      fence_proxy_async_smem();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar);
    };
    // this warp's accumulator columns from `col` of this lane
    auto load_cols = [&](uint32_t col, uint32_t (&v)[WC]) {
#pragma unroll
      for (int c = 0; c < WC; c += 32) tmem_ld_32x32b_x32(lane_addr + col + c, v + c);
      tmem_ld_wait();
    };
    // 16-byte piece i of this warp's columns in an operand image of `rows` rows per 64-column chunk
    auto piece = [&](uint8_t* tile, int rows, int i) -> uint8_t* {
      const int cc = c0 + 8 * i;
      return tile + (cc >> 6) * rows * 128 + r * 128 + ((((cc & 63) >> 3) ^ (r & 7)) << 4);
    };
    auto put_cols = [&](uint8_t* tile, int rows, const uint32_t (&v)[WC]) {
#pragma unroll
      for (int i = 0; i < WC / 8; ++i) {
        float f[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) f[j] = __uint_as_float(v[8 * i + j]);
        st_shared8(piece(tile, rows, i), pack8(f));
      }
    };
    {
      const float* x0 = (p.x_init && !sum) ? p.x_init + (static_cast<size_t>(unit) * D + r) * D + g0 : nullptr;
      const bool wide = (reinterpret_cast<uintptr_t>(x0) & 15) == 0;   // a caller's state may lie at any float
#pragma unroll 1
      for (int c = 0; c < WC; c += 32) {
        uint32_t v[32];
        if (wide) {
#pragma unroll
          for (int i = 0; i < 32; i += 4) {
            const uint4 w = x0 ? *reinterpret_cast<const uint4*>(x0 + c + i) : make_uint4(0u, 0u, 0u, 0u);
            v[i] = w.x; v[i + 1] = w.y; v[i + 2] = w.z; v[i + 3] = w.w;
          }
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] = __float_as_uint(x0[c + i]);
        }
        if (lin) {
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] = g0 + c + i == r ? __float_as_uint(1.f) : 0u;
        }
        tmem_st_32x32b_x32(lane_addr + COL_X + c, v);
      }
      tmem_st_wait();
    }
    // Rows of the previous chunk's output: tensor memory -> staging tile, by the warps that have no token rows of Y, while
    // the others make U.
    auto stage_rows = [&](int chunk) {   // the walk's chunk-th
      if (BWD || sum || tok_warp) return;
      const uint32_t buf = chunk & 1;
      wait(&o_done[buf], (chunk >> 1) & 1);
      uint32_t v[WC];
      load_cols(COL_O + buf * 128, v);
      put_cols(ob - C * 128, C, v);   // lanes 64 .. 127 are its rows
      fence_proxy_async_smem();
    };
    auto store_rows = [&](int n) {
#pragma unroll
      for (int hf = 0; hf < HALVES; ++hf) tma_store_3d(&tmO, ob + hf * 8192, tx + col0 + hf * 64, tok0 + n * C, tb);
    };
    for (int it = 0; it < N; ++it) {
      const int n = n0 + (BWD ? (N - 1 - it) : it);
      const uint32_t cph = it & 1;
      const int g = seq * NT + n;
      if (it > 0) wait(x_done, cph ^ 1);
      // bf16 image of the state entering this chunk
      {
        uint32_t v[WC];
        load_cols(COL_X, v);
        put_cols(xb, D, v);
      }
      arrive(x_ready);
      if (!sum) {
        if (r == 0 && ch == 0) tma_store_wait_read<0>();   // U of the previous chunk has left ub
        sync_rows();
        if (r == 0 && ch == 0) {
          if (store_ux) {
#pragma unroll
            for (int hf = 0; hf < HALVES; ++hf) tma_store_3d(&tmXB, xb + hf * 16384, col0 + hf * 64, g * D, 0);
          }
          tma_store_commit();
        }
      }
      if (tok_warp) {
        uint8_t* ut = smem + it % STAGES * S::STAGE + TILE_DO;
        bf16x8 uh[BWD ? 1 : WC / 8];   // this lane's U^, read while Y is computed
        if (!BWD && !lin) {
          wait(&full[it % STAGES], (it / STAGES) & 1);
#pragma unroll
          for (int i = 0; i < WC / 8; ++i) uh[BWD ? 0 : i] = ld_shared8(piece(ut, C, i));
        }
        wait(y_done, cph);
        constexpr int PART = S::BOTH ? 32 : WC;   // columns at a time: what the registers of two chains hold
#pragma unroll
        for (int c = 0; c < WC; c += PART) {
          uint32_t v[PART];
#pragma unroll
          for (int k = 0; k < PART; k += 32) tmem_ld_32x32b_x32(lane_addr + (STACK ? COL_O + cph * 128 : COL_Y) + c + k, v + k);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < PART / 8; ++i) {
            float y[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) y[j] = __uint_as_float(v[8 * i + j]);
            if (!BWD && !lin) {
              float uhv[8];
              unpack8(uh[BWD ? 0 : c / 8 + i], uhv);
#pragma unroll
              for (int j = 0; j < 8; ++j) y[j] = uhv[j] - y[j];  // U = U^ - W S
            } else {
#pragma unroll
              for (int j = 0; j < 8; ++j) y[j] = -y[j];          // operand (and output) is -dU
            }
            st_shared8(piece(ub, C, c / 8 + i), pack8(y));
          }
        }
        arrive(u_ready);
        if (store_ux) {
          sync_tok();
          if (r == 0 && ch == 0) {
#pragma unroll
            for (int hf = 0; hf < HALVES; ++hf) tma_store_3d(&tmU, ub + hf * 8192, col0 + hf * 64, g * C, 0);
            tma_store_commit();
          }
        }
      }
      if (it > 0) stage_rows(it - 1);
      if (!sum) {   // while the state is updated: the bulk stores before U's have read xb and ob, which are rewritten next
        if (r == 0 && ch == 0) {
          if (store_ux) tma_store_wait_read<1>();
          else tma_store_wait_read<0>();
        }
        sync_rows();
        if (!BWD && it > 0 && r == 0 && ch == 0) {   // read by the next chunk's first wait, before rows are staged again
          store_rows(n - 1);
          tma_store_commit();
        }
      }
    }
    // drain: last chunk's output rows and the final state
    if (N > 0) {
      wait(x_done, (N - 1) & 1);
      if (!BWD && !sum) {
        if (r == 0 && ch == 0) tma_store_wait_read<0>();
        sync_rows();
        stage_rows(N - 1);
        sync_rows();
        if (r == 0 && ch == 0) {
          store_rows(n0 + N - 1);
          tma_store_commit();
        }
      }
      float* fin = lin ? p.p_final : p.x_final;
      if (fin != nullptr) {
        float* xf = fin + (static_cast<size_t>(unit) * D + r) * D + g0;
        uint32_t v[WC];
        load_cols(COL_X, v);
#pragma unroll
        for (int i = 0; i < WC / 4; ++i)
          reinterpret_cast<float4*>(xf)[i] =
              make_float4(__uint_as_float(v[4 * i]), __uint_as_float(v[4 * i + 1]),
                          __uint_as_float(v[4 * i + 2]), __uint_as_float(v[4 * i + 3]));
      }
    }
    if (r == 0 && ch == 0) tma_store_wait<0>();
  }

  tc_fence_before();
  __syncthreads();
  if (p.status != nullptr && *reinterpret_cast<volatile int*>(p.status) != PB_OK) {
    for (int i = 0; i < 2000; ++i) __nanosleep(1000);  // let copies in flight land
    __syncthreads();
  }
  if (warp == MMA_WARP) {
    tc_fence_after();
    tmem_dealloc(tmem, TMEM_COLS);
  }
}

template <bool BWD, int NC>
int launch_cols(const CUtensorMap& tW, const CUtensorMap& tQ, const CUtensorMap& tK, const CUtensorMap& tM,
                const CUtensorMap& tD, const CUtensorMap& tXB, const CUtensorMap& tU, const CUtensorMap& tO,
                const Params& p, int ctas, cudaStream_t st) {
  static pb::DeviceOnce attr_once;   // per device: the attribute belongs to the current GPU
  if (attr_once.need()) {
    cudaError_t e = cudaFuncSetAttribute(delta_scan_kernel<BWD, NC>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         Shape<NC>::TOTAL);
    if (e != cudaSuccess) return static_cast<int>(e);
    attr_once.done();
  }
  pb::launch(delta_scan_kernel<BWD, NC>, ctas, Shape<NC>::THREADS, Shape<NC>::TOTAL, st, tW, tQ, tK, tM, tD, tXB, tU, tO, p);
  return static_cast<int>(cudaGetLastError());
}

template <bool BWD>
int launch(const void* W, const void* Q, const void* K, const void* M, const void* fifth,
           void* xb_out, void* u_out, void* o_out, int seq_len, int ld, const Params& p, cudaStream_t st) {
  const uint64_t G = static_cast<uint64_t>(p.n_seq) * p.n_chunks;
  const uint64_t rows = G * C;
  CUtensorMap tW, tQ, tK, tM, tD, tXB, tU, tO;
  int r = 0;
  // token-major tensors: [batch, seq_len, ld]; per-chunk tensors: [G * 64, 128]
  const bool tokmaj = p.heads > 0;
  const uint64_t batch = tokmaj ? static_cast<uint64_t>(p.n_seq) / p.heads : 1;
  auto tok_map = [&](CUtensorMap* tm, const void* base) {
    return tokmaj ? make_tmap_3d(tm, base, 2, static_cast<uint64_t>(p.heads) * D, seq_len, batch, ld,
                                 static_cast<uint64_t>(seq_len) * ld, 64, C)
                  : make_tmap_3d(tm, base, 2, D, rows, 1, D, 0, 64, C);
  };
  r |= make_tmap_3d(&tW, W, 2, D, rows, 1, D, 0, 64, C);
  r |= tok_map(&tQ, Q);
  r |= tok_map(&tK, K);
  r |= make_tmap_3d(&tM, M, 2, C, rows, 1, C, 0, 64, C);
  if (BWD) r |= tok_map(&tD, fifth);
  else r |= make_tmap_3d(&tD, fifth, 2, D, rows, 1, D, 0, 64, C);
  // outputs that are not stored still need a valid map: W stands in
  r |= make_tmap_3d(&tXB, p.store_ux ? xb_out : W, 2, D, p.store_ux ? G * D : rows, 1, D, 0, 64, p.store_ux ? D : C);
  r |= make_tmap_3d(&tU, p.store_ux ? u_out : W, 2, D, rows, 1, D, 0, 64, C);
  if (BWD) tO = tU;
  else r |= tok_map(&tO, o_out);
  if (r != 0) return 1000 + r;
  const int units = p.n_seq * p.n_seg;
  // A forward walk that keeps the states stays on 128 columns from 67 sequences on: with the last SMs writing too its stores
  // back up (seen on 148 SMs; the line is a measured one). 64 / 128 columns, 64 chunks, us: 60 sequences 91 / 120, 64 98 / 125, 68 141 / 127..131, 72 150 / 136, 74 150 / 129; nothing
  // kept 74 79 / 104, backward 74 104 / 109.
  const int most = BWD || p.store_ux == 0 ? num_sms() : num_sms() - 16;
  if (!p.summary && 2 * units <= most)
    return launch_cols<BWD, 64>(tW, tQ, tK, tM, tD, tXB, tU, tO, p, 2 * units, st);
  if constexpr (!BWD) {
    // both maps in one CTA where a CTA for each would be a second wave
    if (p.summary && 2 * units > num_sms())
      return launch_cols<false, 256>(tW, tQ, tK, tM, tD, tXB, tU, tO, p, units, st);
  }
  return launch_cols<BWD, 128>(tW, tQ, tK, tM, tD, tXB, tU, tO, p, units * ((p.summary && !BWD) ? 2 : 1), st);
}

}  // namespace dscan
}  // namespace pb

using namespace pb;

// Forward walk. All per-chunk tensors are row-major [(n_seq * n_chunks * 64), 128]
// bf16 (M: [.., 64]), chunk g = seq * n_chunks + n occupying rows [64 g, 64 g + 64).
// With heads > 0, Q, K and out (and dO in the backward walk) are instead token-major
// [batch, seq_len, ld] with head h = seq % heads at columns [128 h, 128 h + 128) and seq_len in
// (64 (n_chunks - 1), 64 n_chunks]: the rows the last chunk lacks read as zeros (k = q = 0 leave
// the state untouched) and are not written.
//   out   <- O            u_out <- U            xb_out[g] <- bf16(S entering chunk g)
//   x_init / x_final: fp32 [n_seq, 128, 128] (x_init may be null = zero state)
//   u_out and xb_out may both be null when nothing will run backward
static int scan_args_ok(int n_seq, int n_chunks, int heads, int seq_len, int ld, int n_seg) {
  if (heads > 0 && (seq_len <= (n_chunks - 1) * dscan::C || seq_len > n_chunks * dscan::C)) return 0;
  if (n_seq <= 0 || n_chunks <= 0 || heads < 0 || n_seg <= 0 || n_chunks % n_seg != 0) return 0;
  if (heads > 0 && (n_seq % heads != 0 || ld < heads * dscan::D || ld % 8 != 0)) return 0;
  return 1;
}
static dscan::Params scan_params(int n_seq, int n_chunks, int heads, int n_seg, int summary,
                                 const void* x_init, void* x_final, void* p_final, int* status,
                                 bool store_ux = true) {
  dscan::Params p;
  p.n_chunks = n_chunks; p.n_seq = n_seq; p.n_seg = n_seg; p.summary = summary;
  p.heads = heads; p.store_ux = store_ux ? 1 : 0;
  p.x_init = static_cast<const float*>(x_init);
  p.x_final = static_cast<float*>(x_final);
  p.p_final = static_cast<float*>(p_final);
  p.status = status;
  return p;
}

PB_API int pb_delta_scan_fwd(const void* W, const void* Uhat, const void* Q, const void* K,
                             const void* M, void* out, void* u_out, void* xb_out,
                             const void* x_init, void* x_final, int n_seq, int n_chunks,
                             int heads, int seq_len, int ld, int* status, cudaStream_t st) {
  if (!scan_args_ok(n_seq, n_chunks, heads, seq_len, ld, 1) || (u_out == nullptr) != (xb_out == nullptr))
    return PB_BAD_ARG;
  return dscan::launch<false>(W, Q, K, M, Uhat, xb_out, u_out, out, seq_len, ld,
                              scan_params(n_seq, n_chunks, heads, 1, 0, x_init, x_final, nullptr, status, u_out != nullptr), st);
}

// The same walk with every sequence cut into n_seg segments of n_chunks / n_seg chunks, one CTA
// per segment. x_init / x_final: fp32 [n_seq * n_seg, 128, 128], the state entering / leaving
// each segment (x_init comes from pb_delta_scan_summary_fwd + pb_delta_compose).
PB_API int pb_delta_scan_fwd_seg(const void* W, const void* Uhat, const void* Q, const void* K,
                                 const void* M, void* out, void* u_out, void* xb_out,
                                 const void* x_init, void* x_final, int n_seq, int n_chunks,
                                 int n_seg, int heads, int seq_len, int ld, int* status, cudaStream_t st) {
  if (!scan_args_ok(n_seq, n_chunks, heads, seq_len, ld, n_seg) || x_init == nullptr || (u_out == nullptr) != (xb_out == nullptr))
    return PB_BAD_ARG;
  return dscan::launch<false>(W, Q, K, M, Uhat, xb_out, u_out, out, seq_len, ld,
                              scan_params(n_seq, n_chunks, heads, n_seg, 0, x_init, x_final, nullptr, status, u_out != nullptr), st);
}

// Affine map of every segment, S_out = P S_in + R, without outputs: r_out, p_out fp32
// [n_seq * n_seg, 128, 128]. Three products per chunk and map instead of six, no stores but the
// two maps.
PB_API int pb_delta_scan_summary_fwd(const void* W, const void* Uhat, const void* K, void* r_out,
                                     void* p_out, int n_seq, int n_chunks, int n_seg, int heads,
                                     int seq_len, int ld, int* status, cudaStream_t st) {
  if (!scan_args_ok(n_seq, n_chunks, heads, seq_len, ld, n_seg) || r_out == nullptr || p_out == nullptr)
    return PB_BAD_ARG;
  // Q, M and the output maps are never touched in this mode; W stands in so that the tensor
  // maps are valid objects.
  return dscan::launch<false>(W, K, K, W, Uhat, const_cast<void*>(W), const_cast<void*>(W),
                              const_cast<void*>(K), seq_len, ld,
                              scan_params(n_seq, n_chunks, heads, n_seg, 1, nullptr, r_out, p_out, status), st);
}

// Backward walk (chunks in reverse). x_init = gradient of the final state (or null),
//   ndu_out <- -dU (note the sign)
//   dxb_out[g] <- bf16(dS leaving chunk g, i.e. before chunk g is applied)
//   x_final <- gradient of the initial state
PB_API int pb_delta_scan_bwd(const void* W, const void* Q, const void* K, const void* M,
                             const void* dO, void* ndu_out, void* dxb_out, const void* x_init,
                             void* x_final, int n_seq, int n_chunks, int heads, int seq_len, int ld,
                             int* status, cudaStream_t st) {
  if (!scan_args_ok(n_seq, n_chunks, heads, seq_len, ld, 1)) return PB_BAD_ARG;
  return dscan::launch<true>(W, Q, K, M, dO, dxb_out, ndu_out, nullptr, seq_len, ld,
                             scan_params(n_seq, n_chunks, heads, 1, 0, x_init, x_final, nullptr, status), st);
}

// Segmented backward walk: x_init = gradient of the state leaving each segment, x_final =
// gradient of the state entering it, both fp32 [n_seq * n_seg, 128, 128].
PB_API int pb_delta_scan_bwd_seg(const void* W, const void* Q, const void* K, const void* M,
                                 const void* dO, void* ndu_out, void* dxb_out, const void* x_init,
                                 void* x_final, int n_seq, int n_chunks, int n_seg, int heads,
                                 int seq_len, int ld, int* status, cudaStream_t st) {
  if (!scan_args_ok(n_seq, n_chunks, heads, seq_len, ld, n_seg) || x_init == nullptr) return PB_BAD_ARG;
  return dscan::launch<true>(W, Q, K, M, dO, dxb_out, ndu_out, nullptr, seq_len, ld,
                             scan_params(n_seq, n_chunks, heads, n_seg, 0, x_init, x_final, nullptr, status), st);
}

// What each segment's backward walk adds to the state gradient when it starts from zero
// (g_out fp32 [n_seq * n_seg, 128, 128]); the linear part is the transpose of the forward P.
PB_API int pb_delta_scan_summary_bwd(const void* W, const void* Q, const void* K, const void* M,
                                     const void* dO, void* g_out, int n_seq, int n_chunks,
                                     int n_seg, int heads, int seq_len, int ld, int* status, cudaStream_t st) {
  if (!scan_args_ok(n_seq, n_chunks, heads, seq_len, ld, n_seg) || g_out == nullptr) return PB_BAD_ARG;
  return dscan::launch<true>(W, Q, K, M, dO, const_cast<void*>(W), const_cast<void*>(W), nullptr, seq_len, ld,
                             scan_params(n_seq, n_chunks, heads, n_seg, 1, nullptr, g_out, nullptr, status), st);
}

// ---------------------------------------------------------------------------
// Sequential composition of the segments' affine maps (fp32 on the CUDA cores; 128^3 per step).
//   forward  S <- s0 (or 0); for j = 0 .. n_seg-1:  s_in[j] <- S;  S <- P_j S + R_j;   s_fin <- S
//            p_tot (optional) <- P_{n-1} ... P_0
//   reverse  G <- s0 (or 0); for j = n_seg-1 .. 0:  s_in[j] <- G;  G <- P_j^T G + R_j; s_fin <- G
// One CTA per (sequence, 16-column slab): columns of the state never mix.
// A step is 0.26 M multiply-adds per CTA and has to wait for the one before, so its latency is what
// counts. P_j comes by 16-byte asynchronous copies into one of two shared-memory images while
// step j - 1 is computed; a thread owns rows r and r + 64 and four columns, so an operand read from
// shared memory serves four (forward) or two to four (reverse) multiply-adds, and the image's row
// pitch of 132 floats keeps a warp's eight rows on different banks. Eight segments of 16
// sequences: 72 us -> 33 us (before: scalar transposing stores, one read per multiply-add, no
// overlap).
// ---------------------------------------------------------------------------
namespace pb {
namespace dcomp {
constexpr int D = 128, SLAB = 16, LDP = D + 4, LDC = SLAB + 4;
constexpr int SMEM = (2 * D * LDP + D * LDC) * 4;
__device__ __forceinline__ void copy16(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void fma4(float (&acc)[4], float p, const float4& c) {
  acc[0] = fmaf(p, c.x, acc[0]); acc[1] = fmaf(p, c.y, acc[1]);
  acc[2] = fmaf(p, c.z, acc[2]); acc[3] = fmaf(p, c.w, acc[3]);
}
__global__ void __launch_bounds__(256)
compose_kernel(const float* __restrict__ P, const float* __restrict__ R,
               const float* __restrict__ s0, float* __restrict__ s_in, float* __restrict__ s_fin,
               float* __restrict__ p_tot, int n_seg, int reverse, int slabs_state) {
  after_previous_kernel();
  extern __shared__ float sm[];
  float* cur = sm + 2 * D * LDP;                                    // cur[row * LDC + column]
  const int seq = blockIdx.y;
  const bool on_p = static_cast<int>(blockIdx.x) >= slabs_state;    // this CTA folds P itself
  const int col0 = (on_p ? blockIdx.x - slabs_state : blockIdx.x) * SLAB;
  const int r = threadIdx.x >> 2, c0 = (threadIdx.x & 3) * 4;       // rows r, r + 64; columns c0 .. c0 + 3
  const size_t mat = static_cast<size_t>(D) * D;
  auto seg = [&](int step) { return static_cast<size_t>(seq) * n_seg + (reverse ? n_seg - 1 - step : step); };
  auto fetch = [&](int step) {
    const float* Pj = P + seg(step) * mat;
    float* dst = sm + (step & 1) * D * LDP;
    for (int i = threadIdx.x; i < D * D / 4; i += 256) copy16(dst + (i >> 5) * LDP + (i & 31) * 4, Pj + i * 4);
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  fetch(0);
  float a[2][4];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int row = r + 64 * h;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      a[h][c] = 0.f;
      if (on_p) a[h][c] = (row == col0 + c0 + c) ? 1.f : 0.f;
      else if (s0 != nullptr) a[h][c] = s0[seq * mat + row * D + col0 + c0 + c];
    }
  }
  for (int step = 0; step < n_seg; ++step) {
    const size_t j = seg(step);
    // the state entering the segment: to shared memory for the product, and out
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int row = r + 64 * h;
      const float4 v = make_float4(a[h][0], a[h][1], a[h][2], a[h][3]);
      *reinterpret_cast<float4*>(cur + row * LDC + c0) = v;
      if (!on_p && s_in != nullptr) *reinterpret_cast<float4*>(s_in + j * mat + row * D + col0 + c0) = v;
      const float4 rv = on_p ? make_float4(0.f, 0.f, 0.f, 0.f)
                             : *reinterpret_cast<const float4*>(R + j * mat + row * D + col0 + c0);
      a[h][0] = rv.x; a[h][1] = rv.y; a[h][2] = rv.z; a[h][3] = rv.w;
    }
    if (step + 1 < n_seg) {   // its image was read in the previous step, whose closing barrier orders those reads before
      fetch(step + 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();          // P_j and cur are in place
    const float* pj = sm + (step & 1) * D * LDP;
    if (!reverse) {
#pragma unroll 4
      for (int k = 0; k < D; k += 4) {
        const float4 p0 = *reinterpret_cast<const float4*>(pj + r * LDP + k);
        const float4 p1 = *reinterpret_cast<const float4*>(pj + (r + 64) * LDP + k);
        float4 c[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) c[i] = *reinterpret_cast<const float4*>(cur + (k + i) * LDC + c0);
        fma4(a[0], p0.x, c[0]); fma4(a[1], p1.x, c[0]);
        fma4(a[0], p0.y, c[1]); fma4(a[1], p1.y, c[1]);
        fma4(a[0], p0.z, c[2]); fma4(a[1], p1.z, c[2]);
        fma4(a[0], p0.w, c[3]); fma4(a[1], p1.w, c[3]);
      }
    } else {
#pragma unroll 8
      for (int k = 0; k < D; ++k) {
        const float4 c = *reinterpret_cast<const float4*>(cur + k * LDC + c0);
        fma4(a[0], pj[k * LDP + r], c);
        fma4(a[1], pj[k * LDP + r + 64], c);
      }
    }
    __syncthreads();          // every thread has finished reading cur and P_j
  }
  float* fin = on_p ? p_tot : s_fin;
  if (fin != nullptr) {
#pragma unroll
    for (int h = 0; h < 2; ++h)
      *reinterpret_cast<float4*>(fin + seq * mat + (r + 64 * h) * D + col0 + c0) =
          make_float4(a[h][0], a[h][1], a[h][2], a[h][3]);
  }
}
}  // namespace dcomp
}  // namespace pb

PB_API int pb_delta_compose(const void* P, const void* R, const void* s0, void* s_in, void* s_fin,
                            void* p_tot, int n_seq, int n_seg, int reverse, cudaStream_t st) {
  if (n_seq <= 0 || n_seg <= 0 || P == nullptr || R == nullptr) return PB_BAD_ARG;
  if (p_tot != nullptr && reverse) return PB_BAD_ARG;
  const int slabs = pb::dcomp::D / pb::dcomp::SLAB;
  dim3 grid(p_tot != nullptr ? 2 * slabs : slabs, n_seq);
  static pb::DeviceOnce attr_once;
  if (attr_once.need()) {
    cudaError_t e = cudaFuncSetAttribute(pb::dcomp::compose_kernel,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, pb::dcomp::SMEM);
    if (e != cudaSuccess) return static_cast<int>(e);
    attr_once.done();
  }
  pb::launch(pb::dcomp::compose_kernel, grid, 256, pb::dcomp::SMEM, st,
      static_cast<const float*>(P), static_cast<const float*>(R), static_cast<const float*>(s0),
      static_cast<float*>(s_in), static_cast<float*>(s_fin), static_cast<float*>(p_tot), n_seg,
      reverse, slabs);
  return static_cast<int>(cudaGetLastError());
}
