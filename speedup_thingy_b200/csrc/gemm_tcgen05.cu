// Persistent warp-specialised bf16 GEMM for sm_100a:
//   C[M,N] = A[M,K] * B[N,K]^T, fp32 accumulation in tensor memory (TMEM),
//   operands staged by TMA into 128B-swizzled shared memory, MMAs issued by one
//   thread with tcgen05.mma.
//
// Two shapes of work unit (template parameter CTAS):
//   CTAS = 1: one CTA computes a 128 x BN tile (tcgen05.mma.cta_group::1, M = 128).
//   CTAS = 2: a cluster of two CTAs on neighbouring SMs computes a 256 x BN tile with
//             tcgen05.mma.cta_group::2 (M = 256): each CTA stages its own 128 rows of A and
//             its own HALF of the B tile (plain per-CTA TMA loads, no multicast), the MMA
//             of the leader CTA reads both halves, and each CTA's TMEM receives the
//             accumulators of its 128 rows.  Per FLOP this moves a third less operand
//             data from L2 into shared memory than two independent 128 x BN tiles,
//             which pays for long reductions; short products are bound by set-up, drain
//             and their stores and run in either shape within a few per cent.
//
// Roles per CTA (320 threads): warp 0 = TMA producer, warp 1 = TMEM owner + MMA
// issuer (the leader CTA's only, with CTAS = 2), warps 2..9 = epilogue: warp w may
// read the TMEM lane quadrant w % 4 (32 rows); the two warps of a quadrant split the
// tile's columns.  Every epilogue warp owns private staging slots in shared memory
// and hands its 32 x 64 (bf16) or 32 x 32 (fp32) pieces to the TMA by itself, so no
// barrier couples the epilogue warps.  Two accumulator buffers in TMEM let the
// epilogue of tile i overlap the main loop of tile i+1.  Every wait is bounded: on
// expiry the role records a code in the caller's status word and all roles drain to
// the common teardown, which frees TMEM.
//
// Either operand may be "MN-major" (stored with the reduction dimension as the
// slow axis), which is what the weight- and data-gradient GEMMs of the training
// step need; no transposed copies are ever made.

#include <stdlib.h>

#include "tcgen05_ptx.cuh"

namespace {

constexpr int BM = 128;         // rows of C per CTA (TMEM lanes)
constexpr int BK = 64;          // bf16 elements per k-block (= one 128-byte swizzle row)
constexpr int UMMA_K = 16;      // K per tcgen05.mma for 16-bit inputs
constexpr int NUM_THREADS = 320;   // warp 0 producer, warp 1 MMA issuer, warps 2..9 epilogue
constexpr int EPI_WARPS = 8;
constexpr int SLOT_BYTES = 4096;       // one epilogue staging slot: 32 rows x 128 bytes
constexpr int MAX_DYN_SMEM = 232448;   // 227 KB of dynamic shared memory per CTA

#ifdef RTE_GEMM_DIAG
constexpr bool DIAG = true;    // timing diagnostics: RTE_GEMM_DIAG_FLAGS bit 0 = no stores, 1 = no MMAs, 2 = no loads
#else
constexpr bool DIAG = false;
#endif

struct KParams {
  int diag;
  int M, N, K;
  int a_mn, b_mn;
  int epilogue;
  void* C; int ldc;
  const void* R; int ldr;
  void* C2; int ldc2;
  int pair_off;
  int splits; long long split_stride;
  int num_m_blocks, num_n_blocks, kblocks_total, kblocks_per_split;
  int tma_store;            // 1: outputs leave through shared-memory staging + TMA bulk stores
  int b_box_rows;           // K-major B: rows per TMA box
  const int* tile_group;    // grouped mode: group id of every 128-row block of A/C (< 0: block unused), else null
  int b_group_stride;       // grouped mode: rows of the stacked B between consecutive groups
  const int* split_kb;      // ragged split-K: k-block range [split_kb[s], split_kb[s+1]) of split s, else null
  int* status;
  const uint8_t* selected;  // MASK: [M, N] bytes, 0 where the gradient is zero; else null
  int as_two;               // MASK: the bits of a product with a bf16 result and the pass behind it (svd_ffn.cu)
};

// ------------------------------------------------------------------ epilogue helpers
__device__ __forceinline__ void store_bf16x32(__nv_bfloat16* dst, const float (&v)[32], int ncols_valid) {
  if (ncols_valid >= 32 && (reinterpret_cast<uintptr_t>(dst) & 15) == 0) {
    uint4* d4 = reinterpret_cast<uint4*>(dst);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      uint4 w;
      w.x = rte::pack_bf16x2(v[8 * q + 0], v[8 * q + 1]);
      w.y = rte::pack_bf16x2(v[8 * q + 2], v[8 * q + 3]);
      w.z = rte::pack_bf16x2(v[8 * q + 4], v[8 * q + 5]);
      w.w = rte::pack_bf16x2(v[8 * q + 6], v[8 * q + 7]);
      d4[q] = w;
    }
  } else {
#pragma unroll
    for (int j = 0; j < 32; ++j)
      if (j < ncols_valid) dst[j] = __float2bfloat16_rn(v[j]);
  }
}
__device__ __forceinline__ void store_f32x32(float* dst, const float (&v)[32], int ncols_valid) {
  if (ncols_valid >= 32 && (reinterpret_cast<uintptr_t>(dst) & 15) == 0) {
    float4* d4 = reinterpret_cast<float4*>(dst);
#pragma unroll
    for (int q = 0; q < 8; ++q) d4[q] = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
  } else {
#pragma unroll
    for (int j = 0; j < 32; ++j)
      if (j < ncols_valid) dst[j] = v[j];
  }
}
__device__ __forceinline__ void load_f32x32(const float* src, float (&v)[32], int ncols_valid) {
  if (ncols_valid >= 32 && (reinterpret_cast<uintptr_t>(src) & 15) == 0) {
    const float4* s4 = reinterpret_cast<const float4*>(src);
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      float4 t = s4[q];
      v[4 * q] = t.x; v[4 * q + 1] = t.y; v[4 * q + 2] = t.z; v[4 * q + 3] = t.w;
    }
  } else {
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = (j < ncols_valid) ? src[j] : 0.f;
  }
}
__device__ __forceinline__ void load_bf16x32(const __nv_bfloat16* src, float (&v)[32], int ncols_valid) {
  if (ncols_valid >= 32 && (reinterpret_cast<uintptr_t>(src) & 15) == 0) {
    const uint4* s4 = reinterpret_cast<const uint4*>(src);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      uint4 t = s4[q];
      float2 a = rte::unpack_bf16x2(t.x), b = rte::unpack_bf16x2(t.y), c = rte::unpack_bf16x2(t.z), d = rte::unpack_bf16x2(t.w);
      v[8 * q] = a.x; v[8 * q + 1] = a.y; v[8 * q + 2] = b.x; v[8 * q + 3] = b.y;
      v[8 * q + 4] = c.x; v[8 * q + 5] = c.y; v[8 * q + 6] = d.x; v[8 * q + 7] = d.y;
    }
  } else {
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = (j < ncols_valid) ? __bfloat162float(src[j]) : 0.f;
  }
}

template <int BN, int CTAS, bool SWB>
struct SmemLayout {
  static constexpr int A_BYTES = BM * BK * 2;            // this CTA's 128 rows of A: 16 KB
  static constexpr int B_ROWS = BN / CTAS;               // rows of the B tile this CTA stages
  static constexpr int B_BYTES = B_ROWS * BK * 2;
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  // staging slots per epilogue warp; with SWB two pairs: (up | gate) arrive there and (d up | d gate) leave from there
  static constexpr int SLOTS = SWB ? 4 : (BN == 256 && CTAS == 1) ? 1 : 2;
  static constexpr int STAGING_BYTES = EPI_WARPS * SLOTS * SLOT_BYTES;
  static constexpr int BAR_BYTES = 512;
  static constexpr int STAGES_FIT = (MAX_DYN_SMEM - 1024 - BAR_BYTES - STAGING_BYTES) / STAGE_BYTES;
  static constexpr int STAGES = STAGES_FIT > 8 ? 8 : STAGES_FIT;
  static constexpr int STAGING_OFFSET = STAGES * STAGE_BYTES;
  static constexpr int BAR_OFFSET = STAGING_OFFSET + STAGING_BYTES;
  static constexpr int TOTAL = BAR_OFFSET + BAR_BYTES + 1024;   // + slack for 1024-byte alignment
};

// ------------------------------------------------------------------ kernel
// SWB: the epilogue is SwiGLU's backward with its operands brought in by the TMA (see there); a kernel of its own because
// its staging slots take shared memory from the operand stages.
// MASK: gradients of the selected neurons only (zeros elsewhere).
template <int BN, int CTAS, bool SWB, bool MASK>
__global__ void __launch_bounds__(NUM_THREADS, 1)
gemm_tcgen05_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                    const __grid_constant__ CUtensorMap tmap_c, const __grid_constant__ CUtensorMap tmap_c2,
                    const __grid_constant__ CUtensorMap tmap_r, const __grid_constant__ CUtensorMap tmap_r2,
                    const KParams p) {
  using L = SmemLayout<BN, CTAS, SWB>;
  constexpr int STAGES = L::STAGES;
  constexpr uint32_t TMEM_COLS = 2 * BN;
  constexpr int HALF = BN / 2;               // columns of a tile per epilogue warp of a quadrant

  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t bar_base = smem_base + L::BAR_OFFSET;
  // barrier slots (8 bytes each): full[STAGES], empty[STAGES], tmem_full[2], tmem_empty[2]; then tmem ptr, error flag
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (STAGES + s); };
  auto tfull_bar = [&](int b) { return bar_base + 8u * (2 * STAGES + b); };
  auto tempty_bar = [&](int b) { return bar_base + 8u * (2 * STAGES + 2 + b); };
  const uint32_t tmem_slot = bar_base + 8u * (2 * STAGES + 4);
  volatile uint32_t* tmem_slot_ptr =
      reinterpret_cast<volatile uint32_t*>(smem_raw + (tmem_slot - smem_u32(smem_raw)));
  volatile uint32_t* err_flag = tmem_slot_ptr + 2;     // set by a role whose wait ran out
  auto operand_bar = [&](int epi_warp, uint32_t set) { return bar_base + 256u + uint32_t(epi_warp) * 16u + set * 8u; };   // SWB

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t cta_rank = (CTAS == 2) ? cluster_ctarank() : 0u;
  const bool leader = cta_rank == 0;
  const int unit = blockIdx.x / CTAS, n_units = gridDim.x / CTAS;    // work units = CTAs or CTA pairs

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(full_bar(s), 1); mbar_init(empty_bar(s), 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(tfull_bar(b), 1); mbar_init(tempty_bar(b), EPI_WARPS * CTAS); }
    if (SWB) for (int e = 0; e < EPI_WARPS; ++e) { mbar_init(operand_bar(e, 0), 1); mbar_init(operand_bar(e, 1), 1); }
    *err_flag = 0;
    fence_barrier_init();
    prefetch_tmap(&tmap_a);
    prefetch_tmap(&tmap_b);
  }
  if (warp == 1) {
    tmem_alloc<CTAS>(tmem_slot, TMEM_COLS);     // CTAS = 2: one warp of EACH CTA of the pair takes part
    tmem_relinquish<CTAS>();
  }
  rte::grid_dependency_wait();
  tc_fence_before();
  if (CTAS == 2) cluster_sync_all(); else __syncthreads();     // barriers of both CTAs are initialised beyond here
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot_ptr;
  rte::grid_dependents_launch();

  const int tiles = p.num_m_blocks * p.num_n_blocks;
  const int total_work = tiles * p.splits;

  if (warp == 0) {
    // ---------------- TMA producer (in both CTAs of a pair: each fills its own shared memory) ----------------
    // (the whole warp runs the loop; one elected lane issues -- see elect_one)
    {
      int stage = 0; uint32_t phase = 0; bool ok = true;
      for (int w = unit; w < total_work && ok; w += n_units) {
        const int split = w / tiles, t = w % tiles;
        const int mblk = t % p.num_m_blocks, nblk = t / p.num_m_blocks;
        const int m0 = (mblk * CTAS + int(cta_rank)) * BM, n0 = nblk * BN;
        int boff = 0;
        if (p.tile_group) {
          const int g = p.tile_group[mblk];
          if (g < 0) continue;
          boff = g * p.b_group_stride;
        }
        const int kb0 = p.split_kb ? p.split_kb[split] : split * p.kblocks_per_split;
        const int kb1 = p.split_kb ? p.split_kb[split + 1] : min(kb0 + p.kblocks_per_split, p.kblocks_total);
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!mbar_wait<CTAS>(empty_bar(stage), phase ^ 1u)) {
            if (p.status && lane == 0) atomicExch(p.status, RTE_DEV_WAIT_TIMEOUT_PRODUCER);
            *err_flag = 1;
            ok = false; break;
          }
          const uint32_t sa = smem_base + stage * L::STAGE_BYTES, sb = sa + L::A_BYTES;
          if (DIAG && (p.diag & 4)) {
            if (leader && lane == 0) mbar_arrive(full_bar(stage));
            if (++stage == STAGES) { stage = 0; phase ^= 1u; }
            continue;
          }
          if (elect_one()) {
          // the leader's barrier counts the bytes of both CTAs' loads of this stage
          if (leader) mbar_arrive_expect_tx(full_bar(stage), L::STAGE_BYTES * CTAS);
          const uint32_t fb = (CTAS == 2) ? mapa_cluster(full_bar(stage), 0) : full_bar(stage);
          const int k0 = kb * BK;
          if (!p.a_mn) {
            tma_load_2d<CTAS>(sa, &tmap_a, fb, k0, m0);
          } else {
#pragma unroll
            for (int j = 0; j < BM / 64; ++j) tma_load_2d<CTAS>(sa + j * 8192, &tmap_a, fb, m0 + 64 * j, k0);
          }
          // this CTA stages the tile's columns [c_lo, c_lo + B_ROWS)
          const int c_lo = int(cta_rank) * L::B_ROWS;
          if (!p.b_mn) {
            const int box = p.b_box_rows;
            for (int c = 0; c < L::B_ROWS; c += box) {
              const int tc = c_lo + c;               // column of the tile = row of B
              int brow;
              if (p.pair_off > 0 && p.epilogue == RTE_EPI_SWIGLU_FWD)     // tile = (up rows | matching gate rows)
                brow = (tc < HALF) ? nblk * HALF + tc : p.pair_off + nblk * HALF + (tc - HALF);
              else
                brow = n0 + tc;
              tma_load_2d<CTAS>(sb + uint32_t(c) * 128u, &tmap_b, fb, k0, boff + brow);
            }
          } else {
#pragma unroll
            for (int j = 0; j < L::B_ROWS / 64; ++j)
              tma_load_2d<CTAS>(sb + j * 8192, &tmap_b, fb, n0 + c_lo + 64 * j, boff + k0);
          }
          }
          if (++stage == STAGES) { stage = 0; phase ^= 1u; }
        }
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer (one thread; with CTAS = 2 the leader CTA's, for both CTAs) ----------------
    if (leader) {
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (uint32_t(p.a_mn) << 15) | (uint32_t(p.b_mn) << 16) |
                             (uint32_t(BN >> 3) << 17) | (uint32_t((BM * CTAS) >> 4) << 24);
      const uint32_t a_step = p.a_mn ? (UMMA_K * 128u) >> 4 : (UMMA_K * 2u) >> 4;
      const uint32_t b_step = p.b_mn ? (UMMA_K * 128u) >> 4 : (UMMA_K * 2u) >> 4;
      const uint64_t adesc0 = make_smem_desc(smem_base, p.a_mn != 0), bdesc0 = make_smem_desc(smem_base + L::A_BYTES, p.b_mn != 0);
      int stage = 0; uint32_t phase = 0; int acc = 0; uint32_t acc_phase = 0; bool ok = true;
      for (int w = unit; w < total_work && ok; w += n_units) {
        const int split = w / tiles;
        if (p.tile_group && p.tile_group[(w % tiles) % p.num_m_blocks] < 0) continue;
        const int kb0 = p.split_kb ? p.split_kb[split] : split * p.kblocks_per_split;
        const int kb1 = p.split_kb ? p.split_kb[split + 1] : min(kb0 + p.kblocks_per_split, p.kblocks_total);
        if (!mbar_wait<CTAS>(tempty_bar(acc), acc_phase ^ 1u)) {
          if (p.status && lane == 0) atomicExch(p.status, RTE_DEV_WAIT_TIMEOUT_MMA);
          *err_flag = 1;
          ok = false; break;
        }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * BN;
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!mbar_wait<CTAS>(full_bar(stage), phase)) {
            if (p.status && lane == 0) atomicExch(p.status, RTE_DEV_WAIT_TIMEOUT_MMA);
            *err_flag = 1;
            ok = false; break;
          }
          tc_fence_after();
          const uint64_t off = uint64_t(uint32_t(stage) * uint32_t(L::STAGE_BYTES >> 4));     // (addresses stay below the field's end)
          if (elect_one()) {
            if (!(DIAG && (p.diag & 2)))
#pragma unroll
            for (int k = 0; k < BK / UMMA_K; ++k)
              tc_mma_bf16<CTAS>(d_tmem, adesc0 + off + uint64_t(k * a_step), bdesc0 + off + uint64_t(k * b_step), idesc,
                                (kb > kb0 || k > 0) ? 1u : 0u);
            tc_commit<CTAS>(empty_bar(stage));       // frees the stage (in both CTAs) once these MMAs have read it
          }
          if (++stage == STAGES) { stage = 0; phase ^= 1u; }
        }
        if (!ok) break;
        if (elect_one()) tc_commit<CTAS>(tfull_bar(acc));           // accumulator complete -> epilogue (of both CTAs)
        if (++acc == 2) { acc = 0; acc_phase ^= 1u; }
      }
    }
  } else {
    // ---------------- epilogue (warps 2..9) ----------------
    // A warp may read the TMEM lane quadrant (warp % 4); warps 2..5 and 6..9 each cover all 128 rows and take one
    // half of the tile's columns.
    const int quad = warp & 3;               // TMEM lane quadrant this warp may read
    const int grp = (warp - 2) >> 2;         // 0 or 1: which half of the columns
    const uint32_t tempty_remote0 = (CTAS == 2) ? mapa_cluster(tempty_bar(0), 0) : 0u;
    const uint32_t tempty_remote1 = (CTAS == 2) ? mapa_cluster(tempty_bar(1), 0) : 0u;
    int acc = 0; uint32_t acc_phase = 0; bool ok = true;
    // TMA-store path: this warp's private staging slots; lane = row inside the warp's 32 rows.  A piece is written
    // into a slot with the 128-byte swizzle the store's tensor map expects, then lane 0 hands it to the TMA, which
    // clips rows / columns beyond M / N.  A slot is reused once the store that last read it has finished reading.
    const uint32_t wslots = smem_base + L::STAGING_OFFSET + uint32_t(warp - 2) * uint32_t(L::SLOTS * SLOT_BYTES);
    uint32_t job = 0;
    auto acquire = [&]() -> uint32_t {
      if (lane == 0) bulk_wait_read<L::SLOTS - 1>();
      __syncwarp();
      return wslots + (job % uint32_t(L::SLOTS)) * uint32_t(SLOT_BYTES);
    };
    auto submit = [&](const CUtensorMap* map, uint32_t slot, int x, int y, int z) {
      fence_proxy_async();
      __syncwarp();
      if (lane == 0 && !(DIAG && (p.diag & 32))) { tma_store_3d(map, slot, x, y, z); bulk_commit(); }
      ++job;
    };
    auto put16 = [&](uint32_t slot, uint32_t chunk, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
      st_shared_v4(slot + uint32_t(lane) * 128u + ((chunk ^ (uint32_t(lane) & 7u)) << 4), a, b, c, d);
    };

    auto epi_wait = [&](uint32_t bar, uint32_t parity) -> bool {
      return mbar_wait<CTAS>(bar, parity);
    };
    // ---- SWB: acc = dz; (d up | d gate) from the saved (up | gate), 64 columns at a time.  The pass is bound by the bytes
    // of (up | gate) in and (d up | d gate) out; read row by row by the lanes that own the rows, the operands cost more
    // than the product (8192 x 2048 x 512: 51 us, of which 18 are the product's).  So the TMA brings a piece's up and gate
    // into a pair of slots while the piece before is worked on, the results take their place there and leave from there:
    // 37 us (3.6 TB/s of the pass's own bytes); 16384 x 2048 x 512 89 -> 65, 8192 x 4096 x 1024 95 -> 85.
    // tmap_c / tmap_r view columns [0, F), tmap_c2 / tmap_r2 columns [F, 2F): each clips at its own edge, and a piece
    // outside the matrix reads zeros and is not written.
    uint32_t piece = 0;
    auto fetch_piece = [&](uint32_t q, int w, int c0) {
      if (w < total_work && lane == 0) {
        bulk_wait_read<0>();                   // the results that left from this pair two pieces ago
        const uint32_t pair = wslots + (q & 1u) * uint32_t(2 * SLOT_BYTES), bar = operand_bar(warp - 2, q & 1u);
        const int y = ((w % p.num_m_blocks) * CTAS + int(cta_rank)) * BM + quad * 32, x = (w / p.num_m_blocks) * BN + c0;
        mbar_arrive_expect_tx(bar, 2 * SLOT_BYTES);
        tma_load_3d(pair, &tmap_r, bar, x, y, 0);
        tma_load_3d(pair + SLOT_BYTES, &tmap_r2, bar, x, y, 0);
      }
      __syncwarp();
    };
    if (SWB) fetch_piece(0, unit, grp * HALF);

    for (int w = unit; w < total_work && ok; w += n_units) {
      const int split = w / tiles, t = w % tiles;
      const int mblk = t % p.num_m_blocks, nblk = t / p.num_m_blocks;
      const int m0 = (mblk * CTAS + int(cta_rank)) * BM, n0 = nblk * BN;
      if (p.tile_group && p.tile_group[mblk] < 0) continue;
      // a split with an empty k-range never touched its accumulator: its partial is all zeros
      const bool empty_acc = p.split_kb && p.split_kb[split + 1] <= p.split_kb[split];
      const int row = m0 + quad * 32 + lane;
      const bool row_ok = row < p.M;
      const int y0 = m0 + quad * 32;           // first row of this warp's pieces
      const bool warp_rows = y0 < p.M && !(DIAG && (p.diag & 1));   // any of this warp's rows inside the matrix
      const uint32_t t_row = tmem_base + (uint32_t(quad * 32) << 16) + acc * BN;
      uint32_t raw[32];

      if (SWB) {
        if (!epi_wait(tfull_bar(acc), acc_phase)) {
          if (p.status && lane == 0) atomicExch(p.status, RTE_DEV_WAIT_TIMEOUT_EPILOGUE);
          *err_flag = 1;
          ok = false; break;
        }
        tc_fence_after();
        for (int c0 = grp * HALF; c0 < (grp + 1) * HALF; c0 += 64, ++piece) {
          const bool last = c0 + 64 >= (grp + 1) * HALF;
          uint32_t sel[MASK ? 16 : 1];         // this row's 64 bytes, under way while the operands arrive
          if constexpr (MASK) {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              uint4 b = make_uint4(0u, 0u, 0u, 0u);
              if (row_ok && n0 + c0 + 16 * k < p.N) b = __ldg(reinterpret_cast<const uint4*>(p.selected + size_t(row) * p.N + n0 + c0 + 16 * k));
              sel[4 * k] = b.x; sel[4 * k + 1] = b.y; sel[4 * k + 2] = b.z; sel[4 * k + 3] = b.w;
            }
          }
          fetch_piece(piece + 1, last ? w + n_units : w, last ? grp * HALF : c0 + 64);
          if (!mbar_wait<1>(operand_bar(warp - 2, piece & 1u), (piece >> 1) & 1u)) {
            if (p.status && lane == 0) atomicExch(p.status, RTE_DEV_WAIT_TIMEOUT_EPILOGUE);
            *err_flag = 1;
            ok = false;
          }
          if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
          const int col = n0 + c0;
          if (!warp_rows || col >= p.N) continue;
          const uint32_t slot = wslots + (piece & 1u) * uint32_t(2 * SLOT_BYTES), slot2 = slot + uint32_t(SLOT_BYTES);
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            uint32_t u[16], g[16];
            tmem_ld32(t_row + c0 + 32 * h, raw);
#pragma unroll
            for (uint32_t c = 0; c < 4; ++c) {
              const uint32_t at = uint32_t(lane) * 128u + (((4u * h + c) ^ (uint32_t(lane) & 7u)) << 4);
              ld_shared_v4(slot + at, u[4 * c], u[4 * c + 1], u[4 * c + 2], u[4 * c + 3]);
              ld_shared_v4(slot2 + at, g[4 * c], g[4 * c + 1], g[4 * c + 2], g[4 * c + 3]);
            }
            tmem_ld_wait();
            auto form = [&](int j, float dz0, float dz1, float s0, float s1) {
              const float2 u_ = rte::unpack_bf16x2(u[j]), g_ = rte::unpack_bf16x2(g[j]);
              float du0 = dz0 * g_.x * s0, du1 = dz1 * g_.y * s1;
              float dg0 = dz0 * u_.x * s0 * (1.f + g_.x * (1.f - s0)), dg1 = dz1 * u_.y * s1 * (1.f + g_.y * (1.f - s1));
              if constexpr (MASK) {
                const uint32_t two = sel[8 * h + (j >> 1)] >> (16 * (j & 1));
                if ((two & 0xffu) == 0u) du0 = dg0 = 0.f;
                if ((two & 0xff00u) == 0u) du1 = dg1 = 0.f;
              }
              u[j] = rte::pack_bf16x2(du0, du1);
              g[j] = rte::pack_bf16x2(dg0, dg1);
            };
            if (MASK && p.as_two) {
#pragma unroll
              for (int j = 0; j < 16; ++j) {
                const float2 dz = rte::unpack_bf16x2(rte::pack_bf16x2(__uint_as_float(raw[2 * j]), __uint_as_float(raw[2 * j + 1])));
                const float2 g_ = rte::unpack_bf16x2(g[j]);
                form(j, dz.x, dz.y, rte::sigmoid_rn(g_.x), rte::sigmoid_rn(g_.y));
              }
            } else {
#pragma unroll
              for (int j = 0; j < 16; ++j) {
                const float2 g_ = rte::unpack_bf16x2(g[j]);
                form(j, __uint_as_float(raw[2 * j]), __uint_as_float(raw[2 * j + 1]), rte::fast_sigmoid(g_.x), rte::fast_sigmoid(g_.y));
              }
            }
#pragma unroll
            for (uint32_t c = 0; c < 4; ++c) {
              put16(slot, 4 * h + c, u[4 * c], u[4 * c + 1], u[4 * c + 2], u[4 * c + 3]);
              put16(slot2, 4 * h + c, g[4 * c], g[4 * c + 1], g[4 * c + 2], g[4 * c + 3]);
            }
          }
          fence_proxy_async();
          __syncwarp();
          if (lane == 0) { tma_store_3d(&tmap_c, slot, col, y0, 0); tma_store_3d(&tmap_c2, slot2, col, y0, 0); bulk_commit(); }
        }
        if (!ok) break;
      } else if (p.tma_store && p.epilogue == RTE_EPI_F32) {
        // ---- fp32 (+ residual): 32-column pieces; the residual of the next piece is fetched while this one is staged
        const float* Rf = reinterpret_cast<const float*>(p.R);
        float rres[32];
        const int c_first = grp * HALF;
        auto fetch_res = [&](int col) {
          if (Rf != nullptr) {
            if (row_ok && col < p.N) load_f32x32(Rf + size_t(row) * p.ldr + col, rres, p.N - col);
            else {
#pragma unroll
              for (int j = 0; j < 32; ++j) rres[j] = 0.f;
            }
          }
        };
        fetch_res(n0 + c_first);               // before the accumulator is complete
        if (!epi_wait(tfull_bar(acc), acc_phase)) {
          if (p.status && lane == 0) atomicExch(p.status, RTE_DEV_WAIT_TIMEOUT_EPILOGUE);
          *err_flag = 1;
          ok = false; break;
        }
        tc_fence_after();
        for (int c0 = c_first; c0 < c_first + HALF; c0 += 32) {
          const int col = n0 + c0;
          if (col >= p.N) break;
          tmem_ld32(t_row + c0, raw);
          tmem_ld_wait();
          float v[32];
          if (Rf != nullptr) {
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = rres[j] + __uint_as_float(raw[j]);
            if (c0 + 32 < c_first + HALF) fetch_res(col + 32);
          } else {
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = empty_acc ? 0.f : __uint_as_float(raw[j]);
          }
          if (warp_rows) {
            const uint32_t slot = acquire();
#pragma unroll
            for (uint32_t c = 0; c < 8; ++c)
              put16(slot, c, __float_as_uint(v[4 * c]), __float_as_uint(v[4 * c + 1]), __float_as_uint(v[4 * c + 2]),
                    __float_as_uint(v[4 * c + 3]));
            submit(&tmap_c, slot, col, y0, split);
          }
        }
      } else {
        if (!epi_wait(tfull_bar(acc), acc_phase)) {
          if (p.status && lane == 0) atomicExch(p.status, RTE_DEV_WAIT_TIMEOUT_EPILOGUE);
          *err_flag = 1;
          ok = false; break;
        }
        tc_fence_after();
        if (p.tma_store && p.epilogue == RTE_EPI_BF16) {
          // ---- bf16: 64-column pieces (128-byte rows)
          for (int c0 = grp * HALF; c0 < (grp + 1) * HALF; c0 += 64) {
            const int col = n0 + c0;
            if (col >= p.N) break;
            uint32_t raw2[32];
            tmem_ld32(t_row + c0, raw);
            tmem_ld32(t_row + c0 + 32, raw2);
            tmem_ld_wait();
            if (warp_rows) {
              const uint32_t slot = acquire();
#pragma unroll
              for (uint32_t c = 0; c < 4; ++c)
                put16(slot, c, rte::pack_bf16x2(__uint_as_float(raw[8 * c]), __uint_as_float(raw[8 * c + 1])),
                      rte::pack_bf16x2(__uint_as_float(raw[8 * c + 2]), __uint_as_float(raw[8 * c + 3])),
                      rte::pack_bf16x2(__uint_as_float(raw[8 * c + 4]), __uint_as_float(raw[8 * c + 5])),
                      rte::pack_bf16x2(__uint_as_float(raw[8 * c + 6]), __uint_as_float(raw[8 * c + 7])));
#pragma unroll
              for (uint32_t c = 0; c < 4; ++c)
                put16(slot, 4 + c, rte::pack_bf16x2(__uint_as_float(raw2[8 * c]), __uint_as_float(raw2[8 * c + 1])),
                      rte::pack_bf16x2(__uint_as_float(raw2[8 * c + 2]), __uint_as_float(raw2[8 * c + 3])),
                      rte::pack_bf16x2(__uint_as_float(raw2[8 * c + 4]), __uint_as_float(raw2[8 * c + 5])),
                      rte::pack_bf16x2(__uint_as_float(raw2[8 * c + 6]), __uint_as_float(raw2[8 * c + 7])));
              submit(&tmap_c, slot, col, y0, 0);
            }
          }
        } else if (p.tma_store && p.epilogue == RTE_EPI_SWIGLU_FWD) {
          // ---- the tile holds BN/2 (up, gate) column pairs: columns [0, BN/2) = up_j, [BN/2, BN) = gate_j for hidden
          // units j0 .. j0 + BN/2; this warp takes BN/4 = 64 of them: the rounded up and gate values and
          // z = up * silu(gate) leave as three 64-column pieces.
          const int pq = grp * (BN / 4);
          const int col = nblk * HALF + pq;
          if (col < p.pair_off) {
            uint32_t upk[32], gpk[32];
            uint32_t slot = acquire();
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              tmem_ld32(t_row + pq + 32 * h, raw);
              tmem_ld_wait();
#pragma unroll
              for (int j = 0; j < 16; ++j) upk[16 * h + j] = rte::pack_bf16x2(__uint_as_float(raw[2 * j]), __uint_as_float(raw[2 * j + 1]));
            }
#pragma unroll
            for (uint32_t c = 0; c < 8; ++c) put16(slot, c, upk[4 * c], upk[4 * c + 1], upk[4 * c + 2], upk[4 * c + 3]);
            if (warp_rows) submit(&tmap_c2, slot, col, y0, 0);
            slot = acquire();
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              tmem_ld32(t_row + HALF + pq + 32 * h, raw);
              tmem_ld_wait();
#pragma unroll
              for (int j = 0; j < 16; ++j) gpk[16 * h + j] = rte::pack_bf16x2(__uint_as_float(raw[2 * j]), __uint_as_float(raw[2 * j + 1]));
            }
#pragma unroll
            for (uint32_t c = 0; c < 8; ++c) put16(slot, c, gpk[4 * c], gpk[4 * c + 1], gpk[4 * c + 2], gpk[4 * c + 3]);
            if (warp_rows) submit(&tmap_c2, slot, p.pair_off + col, y0, 0);
            slot = acquire();
            // z from the ROUNDED up and gate: what backward re-reads must agree with what was multiplied here
#pragma unroll
            for (uint32_t c = 0; c < 8; ++c) {
              uint32_t zz[4];
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const float2 u_ = rte::unpack_bf16x2(upk[4 * c + i]), g_ = rte::unpack_bf16x2(gpk[4 * c + i]);
                zz[i] = rte::pack_bf16x2(u_.x * rte::fast_silu(g_.x), u_.y * rte::fast_silu(g_.y));
              }
              put16(slot, c, zz[0], zz[1], zz[2], zz[3]);
            }
            if (warp_rows) submit(&tmap_c, slot, col, y0, 0);
          }
        } else {
          // ---- direct stores (outputs whose addresses / strides the TMA cannot take): 32-column slices, the two
          // warps of a quadrant take alternate slices
          float v[32];
          if (p.epilogue == RTE_EPI_BF16) {
            for (int c = grp; c < BN / 32; c += 2) {
              tmem_ld32(t_row + c * 32, raw); tmem_ld_wait();
              const int col = n0 + c * 32;
              if (row_ok && col < p.N) {
#pragma unroll
                for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(raw[j]);
                store_bf16x32(reinterpret_cast<__nv_bfloat16*>(p.C) + size_t(row) * p.ldc + col, v, p.N - col);
              }
            }
          } else if (p.epilogue == RTE_EPI_F32) {
            float* Cf = reinterpret_cast<float*>(p.C) + size_t(split) * p.split_stride;
            for (int c = grp; c < BN / 32; c += 2) {
              tmem_ld32(t_row + c * 32, raw); tmem_ld_wait();
              const int col = n0 + c * 32;
              if (row_ok && col < p.N) {
                if (p.R != nullptr) {
                  load_f32x32(reinterpret_cast<const float*>(p.R) + size_t(row) * p.ldr + col, v, p.N - col);
#pragma unroll
                  for (int j = 0; j < 32; ++j) v[j] += __uint_as_float(raw[j]);
                } else {
#pragma unroll
                  for (int j = 0; j < 32; ++j) v[j] = empty_acc ? 0.f : __uint_as_float(raw[j]);
                }
                store_f32x32(Cf + size_t(row) * p.ldc + col, v, p.N - col);
              }
            }
          } else if (p.epilogue == RTE_EPI_SWIGLU_FWD) {
            const int j0 = nblk * HALF;
            uint32_t rawg[32];
            for (int c = grp; c < BN / 64; c += 2) {
              tmem_ld32(t_row + c * 32, raw);
              tmem_ld32(t_row + HALF + c * 32, rawg);
              tmem_ld_wait();
              const int col = j0 + c * 32;
              if (row_ok && col < p.pair_off) {
                __nv_bfloat16* ug = reinterpret_cast<__nv_bfloat16*>(p.C2) + size_t(row) * p.ldc2;
                float up[32], gt[32];
#pragma unroll
                for (int j = 0; j < 32; ++j) {
                  // round to bf16 first: the saved (up | gate) and z must agree with what backward re-reads
                  up[j] = __bfloat162float(__float2bfloat16_rn(__uint_as_float(raw[j])));
                  gt[j] = __bfloat162float(__float2bfloat16_rn(__uint_as_float(rawg[j])));
                  v[j] = up[j] * rte::fast_silu(gt[j]);
                }
                const int nv = p.pair_off - col;
                store_bf16x32(ug + col, up, nv);
                store_bf16x32(ug + p.pair_off + col, gt, nv);
                store_bf16x32(reinterpret_cast<__nv_bfloat16*>(p.C) + size_t(row) * p.ldc + col, v, nv);
              }
            }
          } else {  // RTE_EPI_SWIGLU_BWD
            const int F = p.pair_off;
            for (int c = grp; c < BN / 32; c += 2) {
              tmem_ld32(t_row + c * 32, raw); tmem_ld_wait();
              const int col = n0 + c * 32;
              if (row_ok && col < p.N) {
                const __nv_bfloat16* ug = reinterpret_cast<const __nv_bfloat16*>(p.R) + size_t(row) * p.ldr;
                float up[32], gt[32], dg[32];
                const int nv = p.N - col;
                load_bf16x32(ug + col, up, nv);
                load_bf16x32(ug + F + col, gt, nv);
#pragma unroll
                for (int j = 0; j < 32; ++j) {
                  const float dz = __uint_as_float(raw[j]);
                  const float sg = rte::fast_sigmoid(gt[j]);
                  v[j] = dz * gt[j] * sg;                                    // d up
                  dg[j] = dz * up[j] * sg * (1.f + gt[j] * (1.f - sg));      // d gate
                }
                __nv_bfloat16* out = reinterpret_cast<__nv_bfloat16*>(p.C) + size_t(row) * p.ldc;
                store_bf16x32(out + col, v, nv);
                store_bf16x32(out + F + col, dg, nv);
              }
            }
          }
        }
      }
      // the accumulator buffer is free once every epilogue warp (of both CTAs) has read its part
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if (CTAS == 2) mbar_arrive_cluster(acc ? tempty_remote1 : tempty_remote0);
        else mbar_arrive(tempty_bar(acc));
      }
      if (++acc == 2) { acc = 0; acc_phase ^= 1u; }
    }
    if (lane == 0) bulk_wait_read<0>();        // this warp's stores have left shared memory (the grid's end makes them visible)
  }

  // ---------------- teardown ----------------
  tc_fence_before();
  if (CTAS == 2) cluster_sync_all(); else __syncthreads();
  if (*err_flag != 0) {
    // a wait ran out: copies of this CTA (or, in a pair, of its peer) may still be in flight towards shared memory;
    // give them a bounded time to land before the CTA retires
    for (int i = 0; i < 64; ++i) __nanosleep(1000);
    if (CTAS == 2) cluster_sync_all(); else __syncthreads();
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc<CTAS>(tmem_base, TMEM_COLS);
  }
}

// ------------------------------------------------------------------ host side
// 3-D tensor map for the epilogue's bulk stores: [planes, rows, cols] with a box of 32 rows x 128 bytes
// (64 bf16 or 32 fp32 columns) and the 128-byte swizzle of the staging slots.
int make_store_tmap(CUtensorMap* map, const void* base, long long rows, long long cols, long long ld, long long planes,
                    long long plane_stride, bool f32) {
  EncodeTiledFn fn = get_encode_fn();
  if (!fn) return RTE_ERR_TENSOR_MAP;
  const unsigned long long es = f32 ? 4ull : 2ull;
  cuuint64_t dims[3] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows), static_cast<cuuint64_t>(planes)};
  cuuint64_t strides[2] = {static_cast<cuuint64_t>(ld) * es, static_cast<cuuint64_t>(plane_stride) * es};
  cuuint32_t box[3] = {f32 ? 32u : 64u, 32, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = encode_tiled(fn, map, f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, cuuint32_t(3), const_cast<void*>(base),
                  dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? RTE_OK : RTE_ERR_TENSOR_MAP;
}

// ------------------------------------------------------------------ which kernel, which tile
// Times in microseconds fitted to measurements (launches in a graph, operands in L2, M 64..16384, N 128..5000, K 64..8192):
// a launch costs a set-up and epilogue that depend on the tile and on what is written, plus a main loop whose k-blocks
// take longer once every SM pulls its operands from L2.  Picked by the sum: many tiles -> 256-row pairs (least operand
// traffic), one wave of tiles or less -> the smallest tile that still fits one wave, few tiles with a long reduction -> the
// reduction split over a cluster (gemm_tile.cu), a short reduction with few rows -> mma.sync tiles (gemm_small.cu).
// Against one fixed rule (256-column pairs above 128 rows), e.g. 512 x 384 x 128: 6.6 -> 2.6 us, 512 x 384 x 1152 with
// residual 17.3 -> 6.3 us, 1050 x 512 x 4096: 26.4 -> 12 us, 5000 x 384 x 384 with residual 13.9 -> 5.9 us.
struct TileConfig { int bn, ctas; };
struct Choice { int kernel; TileConfig tile; int ksplit; float us; };      // kernel: 0 persistent, 1 cluster tile, 2 mma.sync, 3 resident A

int persistent_ctas(const rte_gemm_args* a, int sms) { return a->max_ctas > 0 ? a->max_ctas : a->max_ctas < 0 ? -a->max_ctas : sms; }

float persistent_us(const rte_gemm_args* a, TileConfig t, int splits, int sms) {
  const int i = (t.bn == 256 ? 0 : 2) + (t.ctas == 2 ? 0 : 1);              // 256 pair | 256 | 128 pair | 128
  static const float base_bf16[4] = {5.2f, 4.0f, 4.5f, 3.2f}, base_f32[4] = {6.3f, 5.4f, 5.3f, 3.9f}, base_res[4] = {10.1f, 8.9f, 7.5f, 5.7f};
  static const float slope_idle[4] = {0.277f, 0.27f, 0.19f, 0.20f}, slope_busy[4] = {0.36f, 0.38f, 0.24f, 0.25f};
  static const float store_bf16[4] = {2.6f, 1.7f, 1.85f, 1.1f};             // a further tile's stores, when longer than its main loop
  const bool f32 = a->epilogue == RTE_EPI_F32, res = f32 && a->R != nullptr;
  const int cols = a->epilogue == RTE_EPI_SWIGLU_FWD ? 2 * a->b_pair_offset : a->N;
  const int units = rte::ceil_div(a->M, BM * t.ctas) * rte::ceil_div(cols, t.bn) * splits;
  const int conc = persistent_ctas(a, sms) / t.ctas, waves = rte::ceil_div(units, conc > 0 ? conc : 1);
  const float kb = float(rte::ceil_div(rte::ceil_div(a->K, BK), splits));
  const float slope = waves > 1 ? slope_busy[i] : slope_idle[i] + (slope_busy[i] - slope_idle[i]) * float(units) / float(conc);
  static const float store_swb[4] = {9.f, 9.f, 5.3f, 5.3f};                // SwiGLU's backward: (up | gate) in, (d up | d gate) out
  // (SwiGLU's forward writes three pieces per 64 hidden units instead of two and has no term of its own yet)
  const float store = a->epilogue == RTE_EPI_SWIGLU_BWD ? store_swb[i] : store_bf16[i] * (res ? 3.8f : f32 ? 2.f : 1.f);
  const float loop = kb * slope;
  return (res ? base_res[i] : f32 ? base_f32[i] : base_bf16[i]) + loop + float(waves - 1) * (loop > store ? loop : store);
}

// The kernels for few tiles launch a CTA per tile: under a positive `max_ctas` they are out for products that have more.
bool too_many(const rte_gemm_args* a, int ctas) { return a->max_ctas > 0 && ctas > a->max_ctas; }

float tile_us(const rte_gemm_args* a, int bn, int ksplit, int sms) {
  const int grid = rte::ceil_div(a->M, BM) * rte::ceil_div(a->N, bn) * ksplit, kb = rte::ceil_div(a->K, BK);
  const float full = float(persistent_ctas(a, sms)) / float(sms);
  // clusters of 2 / 4 / 8 that are resident together (a cluster sits inside one GPC)
  const int limit = int(full * (ksplit == 1 ? 148.f : ksplit == 2 ? 146.f : ksplit == 4 ? 132.f : 112.f));
  if (ksplit > kb || grid > 2 * limit || (ksplit > 1 && grid > limit) || too_many(a, grid)) return 1e9f;
  static const float base64[4] = {3.0f, 4.3f, 3.9f, 4.2f}, base128[4] = {4.1f, 6.2f, 5.4f, 5.4f};
  const float base = (bn == 64 ? base64 : base128)[ksplit == 1 ? 0 : ksplit == 2 ? 1 : ksplit == 4 ? 2 : 3];
  const float per = float(rte::ceil_div(kb, ksplit)) * 0.21f, f32 = a->epilogue == RTE_EPI_F32 ? (bn == 64 ? 0.2f : 0.5f) : 0.f;
  return base + f32 + (grid <= limit ? per : 1.f + 2.2f * per);
}

float small_us(const rte_gemm_args* a) {
  if (a->K % 8 != 0 || a->a_mn_major || (a->b_mn_major && a->N % 8 != 0)) return 1e9f;
  const int rows = rte::ceil_div(a->M, 64), wide = rte::ceil_div(a->N, 64) * rows, ctas = wide < 74 ? rte::ceil_div(a->N, 32) * rows : wide;
  if (ctas > 148 || too_many(a, ctas)) return 1e9f;
  const float kb = float(rte::ceil_div(a->K, BK));
  return 2.0f + (a->R != nullptr && a->epilogue == RTE_EPI_F32 ? 0.2f : 0.f) + kb * (wide < 74 ? 0.28f : 0.53f);
}

TileConfig pick_tile(const rte_gemm_args* a, int splits, int sms, float* us = nullptr) {
  const bool grouped = a->tile_group != nullptr || a->split_kblocks != nullptr;   // per-128-row-block bookkeeping
  const bool swb = a->epilogue == RTE_EPI_SWIGLU_BWD;
  TileConfig best = {swb ? 128 : 256, 1};
  float best_us = 1e30f;
  for (int bn = 128; bn <= 256; bn += 128)
    for (int ctas = 1; ctas <= 2; ++ctas) {
      if (ctas == 2 && (grouped || a->cta_pair == 1 || a->M <= BM)) continue;
      if (ctas == 1 && a->cta_pair == 2 && !grouped && a->M > BM) continue;
      if ((a->tile_n == 128 || a->tile_n == 256) && bn != a->tile_n) continue;
      if (a->epilogue == RTE_EPI_SWIGLU_FWD && bn != 256) continue;            // the paired epilogue takes 64 (up, gate) pairs per warp
      if (swb && bn == 256 && ctas == 1) continue;                             // two stages would be left of its shared memory
      const float t = persistent_us(a, {bn, ctas}, splits, sms);
      if (t < best_us) { best_us = t; best = {bn, ctas}; }
    }
  if (us) *us = best_us;
  return best;
}

// Short reductions with many tiles go to the kernel that keeps A in shared memory (gemm_resident.cu): three or more 256 x 256 tiles per
// CTA pair for plain results (two: 4096 x 1536 x 512 11.7 -> 12.3 us, three: 8192 x 1536 x 512 16.8 -> 15.5), any number with SwiGLU.  Not
// reductions of at most 256 (16384 x 1024 x 256 14.5 -> 14.8) nor more than 32 tiles along N (8192 x 16384 x 512 116 -> 119, 8192 x 32768
// x 512 237 -> 265), where every pair would stream all of a B that no longer stays in L2 beside the results.
bool resident(const rte_gemm_args* a, int splits, int sms) {
  const bool swiglu = a->epilogue == RTE_EPI_SWIGLU_FWD;
  if ((a->epilogue != RTE_EPI_BF16 && !swiglu) || a->K > 512 || a->a_mn_major || splits > 1 || a->tile_group != nullptr || a->split_kblocks != nullptr ||
      a->tile_n != 0 || a->cta_pair != 0 || a->M <= BM || ((reinterpret_cast<uintptr_t>(a->C) | reinterpret_cast<uintptr_t>(swiglu ? a->C2 : nullptr)) & 31) ||
      a->ldc % 16 || (swiglu && a->ldc2 % 16))
    return false;
  const int pairs = persistent_ctas(a, sms) / 2, n_blocks = rte::ceil_div(a->N, 256);
  if (pairs < 1) return false;
  return swiglu || (a->K > 256 && n_blocks <= 32 && (long long)rte::ceil_div(a->M, 256) * n_blocks > 2LL * pairs);
}

Choice choose(const rte_gemm_args* a, int splits, int sms) {
  Choice c = {0, {0, 0}, 1, 0.f};
  if (resident(a, splits, sms)) return {3, {0, 0}, 1, 0.f};
  c.tile = pick_tile(a, splits, sms, &c.us);
  if (a->tile_n != 0 || a->cta_pair != 0 || splits > 1 || a->tile_group != nullptr || a->split_kblocks != nullptr ||
      (a->epilogue != RTE_EPI_BF16 && a->epilogue != RTE_EPI_F32))
    return c;
  for (int bn = 64; bn <= 128; bn += 64)
    for (int ks = 1; ks <= 8; ks *= 2) {
      const float t = tile_us(a, bn, ks, sms);
      if (t < c.us) c = {1, {bn, 1}, ks, t};
    }
  const float t = small_us(a);
  if (t < c.us) c = {2, {0, 0}, 1, t};
  return c;
}

// Work units (CTAs or CTA pairs) that can run at the same time on `ctas` CTAs.
template <int BN, int CTAS, bool SWB = false, bool MASK = false>
int concurrent_units(int ctas, int sm_count) {
  using L = SmemLayout<BN, CTAS, SWB>;
  if (CTAS == 1) return ctas;
  static int max_clusters = -1;
  if (max_clusters < 0) {
    if (cudaFuncSetAttribute(gemm_tcgen05_kernel<BN, CTAS, SWB, MASK>, cudaFuncAttributeMaxDynamicSharedMemorySize, L::TOTAL) != cudaSuccess)
      return ctas / 2;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(unsigned(sm_count / 2 * 2));
    cfg.blockDim = dim3(NUM_THREADS);
    cfg.dynamicSmemBytes = L::TOTAL;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr; cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, gemm_tcgen05_kernel<BN, CTAS, SWB, MASK>, &cfg) == cudaSuccess && n > 0) max_clusters = n;
    else { (void)cudaGetLastError(); max_clusters = sm_count / 2; }
  }
  int units = ctas / 2;
  return units < max_clusters ? units : max_clusters;
}

template <int BN, int CTAS, bool SWB = false, bool MASK = false>
int launch(const rte_gemm_args* a, const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& tc,
           const CUtensorMap& tc2, const CUtensorMap& tr, const CUtensorMap& tr2, KParams& kp, int sm_count, cudaStream_t st) {
  using L = SmemLayout<BN, CTAS, SWB>;
  static_assert(L::STAGES >= 3, "too few pipeline stages fit");
  static bool attr_set = false;
  if (!attr_set) {
    if (cudaFuncSetAttribute(gemm_tcgen05_kernel<BN, CTAS, SWB, MASK>, cudaFuncAttributeMaxDynamicSharedMemorySize, L::TOTAL) != cudaSuccess)
      return RTE_ERR_LAUNCH;
    attr_set = true;
  }
  const int total = kp.num_m_blocks * kp.num_n_blocks * kp.splits;
  int units = concurrent_units<BN, CTAS, SWB, MASK>(persistent_ctas(a, sm_count), sm_count);
  if (units > total) units = total;
  if (units < 1) units = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(unsigned(units * CTAS));
  cfg.blockDim = dim3(NUM_THREADS);
  cfg.dynamicSmemBytes = L::TOTAL;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = CTAS; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr; cfg.numAttrs = (CTAS == 2) ? 2 : 1;
  if (cudaLaunchKernelEx(&cfg, gemm_tcgen05_kernel<BN, CTAS, SWB, MASK>, ta, tb, tc, tc2, tr, tr2, kp) != cudaSuccess) {
    (void)cudaGetLastError();
    return RTE_ERR_LAUNCH;
  }
  RTE_LAUNCH_CHECK();
  return RTE_OK;
}

}  // namespace

extern "C" int rte_device_sm_count(void) {
  static int cached = 0;
  if (cached > 0) return cached;
  int dev = 0, n = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return RTE_ERR_NO_DEVICE;
  if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return RTE_ERR_NO_DEVICE;
  cached = n;
  return n;
}

// us, separate -> fused.  Forward in the persistent kernel: 4096 x 576 -> 1152 19.4 -> 20.7, 8192 x 640 -> 512 20.3 -> 21.7, 4096 x 640 -> 1536 26.3 ->
// 26.5, 3000 x 768 -> 1536 21.3 -> 21.6, 8192 x 512 -> 1024 30.3 -> 31.3, 8192 x 512 -> 2048 53.8 -> 46.0 (with K = 1024 it would pay from 4 M: 4096 x 1024
// -> 2048 40.1 -> 34.3, but its z is not the separate pass's to the last bit, and with the exact quotient 4096 x 768 -> 1536 takes
// 30.7 against 28.4).  Backward (its operands come by TMA, so it pays
// earlier) 8192 x 512 -> 2048 53.7 -> 37.3, 8192 x 256 -> 1024 20.8 -> 17.3, 1000 x 256 -> 1024 7.8 -> 6.7; 512 x 128 -> 512 4.9 -> 6.0
extern "C" int64_t rte_swiglu_fuse_min(int32_t backward) { return backward ? 1000000 : 12000000; }

// The kernel that keeps A in shared memory (gemm_resident.cu) pays earlier, with the separate pass's bits: 8192 x 512 -> 512 18.4 -> 16.6, 4096 x 384
// -> 1536 21.2 -> 19.3, 5000 x 384 -> 1536 24.8 -> 24.1, 8192 x 320 -> 1024 25.1 -> 25.0, 8192 x 264 -> 512 18.4 -> 15.5; not 8192 x 256
// -> 1024 23.6 -> 24.8, 8192 x 128 -> 512 12.9 -> 14.0.
extern "C" int64_t rte_swiglu_fuse_min_fwd(int32_t K) { return K > 256 && K <= 512 ? 4000000 : rte_swiglu_fuse_min(0); }

extern "C" int rte_gemm_wgrad_splits(const rte_gemm_args* a, int32_t max_splits) {
  if (a == nullptr || a->M <= 0 || a->N <= 0 || a->K <= 0) return 1;
  const int sms = rte_device_sm_count(), kb = rte::ceil_div(a->K, BK);
  if (sms <= 0) return 1;
  float best = choose(a, 1, sms).us;
  int splits = 1;
  for (int s = 2; s <= max_splits && s * 4 <= kb; ++s) {
    if (rte::ceil_div(kb, rte::ceil_div(kb, s)) != s) continue;               // every split gets k-blocks
    float us;
    pick_tile(a, s, sms, &us);
    us += 1.8f + float(s + 1) * float(a->M) * float(a->N) * 4e-6f / 5.f;        // ... and one launch adds the partials (cautious: in a
                                                                                 // training step its traffic competes with the other stream's)
    if (us < best) { best = us; splits = s; }
  }
  return splits;
}

namespace {
// `selected` (SwiGLU's backward only): RTE_ERR_UNSUPPORTED where the epilogue that takes it does not serve
int run_gemm(const rte_gemm_args* a, const uint8_t* selected, bool as_two, rte_stream_t stream) {
  RTE_CHECK_ARG(a != nullptr && a->A && a->B && a->C);
  RTE_CHECK_ARG(a->M > 0 && a->N > 0 && a->K > 0);
  RTE_CHECK_ARG(a->epilogue >= RTE_EPI_BF16 && a->epilogue <= RTE_EPI_SWIGLU_BWD);
  const int splits = a->splits < 1 ? 1 : a->splits;
  RTE_CHECK_ARG(splits == 1 || (a->epilogue == RTE_EPI_F32 && a->R == nullptr));
  if ((reinterpret_cast<uintptr_t>(a->A) & 15) || (reinterpret_cast<uintptr_t>(a->B) & 15) || (a->lda % 8) || (a->ldb % 8))
    return RTE_ERR_ALIGNMENT;
  const bool swiglu_f = a->epilogue == RTE_EPI_SWIGLU_FWD, swiglu_b = a->epilogue == RTE_EPI_SWIGLU_BWD;
  if (swiglu_f) {
    RTE_CHECK_ARG(a->C2 != nullptr && a->b_pair_offset > 0 && a->N == 2 * a->b_pair_offset && !a->b_mn_major);
    RTE_CHECK_ARG(a->b_pair_offset % 64 == 0);
  }
  if (swiglu_b) RTE_CHECK_ARG(a->R != nullptr && a->b_pair_offset == a->N);

  const int sms = rte_device_sm_count();
  if (sms <= 0) return RTE_ERR_NO_DEVICE;
  const Choice c = choose(a, splits, sms);
  if (c.kernel == 1) return rte_gemm_bf16_tile(a, c.tile.bn, c.ksplit, stream);
  if (c.kernel == 2) return rte_gemm_bf16_small(a, stream);
  if (c.kernel == 3) return rte_gemm_bf16_resident(a, persistent_ctas(a, sms), stream);
  const int bn = c.tile.bn, ctas = c.tile.ctas;

  KParams kp;
  kp.diag = 0;
#ifdef RTE_GEMM_DIAG
  if (const char* e = getenv("RTE_GEMM_DIAG_FLAGS")) kp.diag = atoi(e);
#endif
  kp.M = a->M; kp.N = a->N; kp.K = a->K;
  kp.a_mn = a->a_mn_major ? 1 : 0; kp.b_mn = a->b_mn_major ? 1 : 0;
  kp.epilogue = a->epilogue;
  kp.C = a->C; kp.ldc = a->ldc; kp.R = a->R; kp.ldr = a->ldr; kp.C2 = a->C2; kp.ldc2 = a->ldc2;
  kp.pair_off = a->b_pair_offset;
  kp.splits = splits; kp.split_stride = a->split_stride;
  kp.num_m_blocks = rte::ceil_div(a->M, BM * ctas);
  kp.num_n_blocks = swiglu_f ? rte::ceil_div(a->b_pair_offset, bn / 2) : rte::ceil_div(a->N, bn);
  kp.kblocks_total = rte::ceil_div(a->K, BK);
  kp.kblocks_per_split = rte::ceil_div(kp.kblocks_total, splits);
  kp.status = a->status;
  kp.selected = selected;
  kp.as_two = as_two ? 1 : 0;
  kp.tile_group = a->tile_group;
  kp.b_group_stride = a->b_group_stride;
  kp.split_kb = a->split_kblocks;
  if (a->tile_group) {
    RTE_CHECK_ARG(a->n_groups >= 1 && a->b_group_stride > 0 && a->M % BM == 0);
    RTE_CHECK_ARG(!a->b_mn_major || a->K % BK == 0);          // a ragged k-block would read the next group's rows
  }
  if (a->split_kblocks) {
    RTE_CHECK_ARG(a->epilogue == RTE_EPI_F32 && a->R == nullptr && a->tile_group == nullptr);
  } else {
    kp.splits = rte::ceil_div(kp.kblocks_total, kp.kblocks_per_split);   // drop empty trailing splits
    // a dropped split would leave its partial unwritten: the caller reduces `splits` partials, so insist
    RTE_CHECK_ARG(kp.splits == splits);
  }

  CUtensorMap ta, tb;
  int rc;
  if (!kp.a_mn) rc = make_tmap(&ta, a->A, a->M, a->K, a->lda, BK, BM);
  else rc = make_tmap(&ta, a->A, a->K, a->M, a->lda, 64, BK);
  if (rc != RTE_OK) return rc;
  const long long b_groups = a->tile_group ? a->n_groups : 0;     // grouped mode: B is the stack of every group's matrix
  // K-major B: one TMA box holds up to 128 rows of this CTA's share of the tile; the paired (up | gate) tile never
  // lets a box straddle the two halves
  int box_rows = bn / ctas < 128 ? bn / ctas : 128;
  if (swiglu_f && box_rows > bn / 2) box_rows = bn / 2;
  kp.b_box_rows = box_rows;
  if (!kp.b_mn) {
    rc = make_tmap(&tb, a->B, b_groups ? b_groups * a->b_group_stride : a->N, a->K, a->ldb, BK, box_rows);
  } else {
    rc = make_tmap(&tb, a->B, b_groups ? b_groups * a->b_group_stride : a->K, a->N, a->ldb, 64, BK);
  }
  if (rc != RTE_OK) return rc;

  // Outputs through TMA bulk stores whenever their addresses and strides allow it (16-byte rules of the TMA);
  // otherwise the epilogue writes with plain vector stores.
  CUtensorMap tc = ta, tc2 = ta, tr = ta, tr2 = ta;
  const bool out_f32 = a->epilogue == RTE_EPI_F32;
  const long long es = out_f32 ? 4 : 2;
  auto aligned = [&](const void* ptr, long long ld) { return ptr && (reinterpret_cast<uintptr_t>(ptr) & 15) == 0 && (ld * es) % 16 == 0; };
  bool tma_ok = aligned(a->C, a->ldc) && a->M >= 1;
  if (splits > 1) tma_ok = tma_ok && (a->split_stride * es) % 16 == 0;
  if (out_f32 && a->R != nullptr) tma_ok = tma_ok && (reinterpret_cast<uintptr_t>(a->R) & 15) == 0 && (a->ldr % 4) == 0;
  if (swiglu_f) tma_ok = tma_ok && aligned(a->C2, a->ldc2);
  if (swiglu_b) tma_ok = tma_ok && a->tile_group == nullptr && (a->N % 8 == 0) && (reinterpret_cast<uintptr_t>(a->R) & 15) == 0 && (a->ldr % 8) == 0;
  if (tma_ok) {
    const long long plane = splits > 1 ? a->split_stride : (long long)a->M * a->ldc;
    if (swiglu_f) {
      rc = make_store_tmap(&tc, a->C, a->M, a->b_pair_offset, a->ldc, 1, (long long)a->M * a->ldc, false);
      if (rc == RTE_OK) rc = make_store_tmap(&tc2, a->C2, a->M, 2LL * a->b_pair_offset, a->ldc2, 1, (long long)a->M * a->ldc2, false);
    } else if (swiglu_b) {
      rc = make_store_tmap(&tc, a->C, a->M, a->N, a->ldc, 1, (long long)a->M * a->ldc, false);
      if (rc == RTE_OK)
        rc = make_store_tmap(&tc2, reinterpret_cast<const __nv_bfloat16*>(a->C) + a->N, a->M, a->N, a->ldc, 1, (long long)a->M * a->ldc, false);
      const __nv_bfloat16* r = reinterpret_cast<const __nv_bfloat16*>(a->R);
      if (rc == RTE_OK) rc = make_store_tmap(&tr, r, a->M, a->N, a->ldr, 1, (long long)a->M * a->ldr, false);
      if (rc == RTE_OK) rc = make_store_tmap(&tr2, r + a->N, a->M, a->N, a->ldr, 1, (long long)a->M * a->ldr, false);
    } else {
      rc = make_store_tmap(&tc, a->C, a->M, a->N, a->ldc, splits, plane, out_f32);
    }
    if (rc != RTE_OK) tma_ok = false;     // e.g. a stride the encoder rejects: use the direct path
  }
  kp.tma_store = tma_ok ? 1 : 0;
  if (DIAG && (kp.diag & 16)) kp.tma_store = 0;

  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const bool swb = swiglu_b && tma_ok && !(DIAG && (kp.diag & 16)) && !(bn == 256 && ctas == 1);
  if (selected != nullptr) {
    if (!swb || a->N % 16 != 0 || (reinterpret_cast<uintptr_t>(selected) & 15)) return RTE_ERR_UNSUPPORTED;
    if (ctas == 1) return launch<128, 1, true, true>(a, ta, tb, tc, tc2, tr, tr2, kp, sms, st);
    return bn == 256 ? launch<256, 2, true, true>(a, ta, tb, tc, tc2, tr, tr2, kp, sms, st)
                     : launch<128, 2, true, true>(a, ta, tb, tc, tc2, tr, tr2, kp, sms, st);
  }
  if (swb) {
    if (ctas == 1) return launch<128, 1, true>(a, ta, tb, tc, tc2, tr, tr2, kp, sms, st);
    return bn == 256 ? launch<256, 2, true>(a, ta, tb, tc, tc2, tr, tr2, kp, sms, st)
                     : launch<128, 2, true>(a, ta, tb, tc, tc2, tr, tr2, kp, sms, st);
  }
  if (swiglu_b) kp.tma_store = 0;
  if (ctas == 2)
    return bn == 256 ? launch<256, 2>(a, ta, tb, tc, tc2, tr, tr2, kp, sms, st) : launch<128, 2>(a, ta, tb, tc, tc2, tr, tr2, kp, sms, st);
  return bn == 256 ? launch<256, 1>(a, ta, tb, tc, tc2, tr, tr2, kp, sms, st) : launch<128, 1>(a, ta, tb, tc, tc2, tr, tr2, kp, sms, st);
}
}  // namespace

extern "C" int rte_gemm_bf16(const rte_gemm_args* a, rte_stream_t stream) { return run_gemm(a, nullptr, false, stream); }

extern "C" int rte_gemm_bf16_swiglu_bwd_selected(const rte_gemm_args* a, const uint8_t* selected, rte_stream_t stream) {
  RTE_CHECK_ARG(a != nullptr && selected != nullptr && a->epilogue == RTE_EPI_SWIGLU_BWD);
  return run_gemm(a, selected, false, stream);
}

extern "C" int rte_svd_ffn_hidden_bwd(const rte_gemm_args* a, const uint8_t* selected, rte_stream_t stream) {
  RTE_CHECK_ARG(a != nullptr && selected != nullptr && a->epilogue == RTE_EPI_SWIGLU_BWD);
  return run_gemm(a, selected, true, stream);
}
