// bf16 GEMM for many rows and a short reduction (K <= 512): C[M,N] = A[M,K] * B[N,K]^T with the A tile resident in shared memory.
//
// The products with a block's input (QKV, up | gate, logits, dz) have eight k-blocks per tile: the persistent kernel
// (gemm_tcgen05.cu) loads 48 KB per 128 x 256 tile and k-block, 400 MB from L2 for 8192 x 4096 x 512, and that traffic and the
// output's share one path: with the stores switched off the product takes 23.8 us, the stores alone 13.5, both 34.7.  Here a CTA
// pair (tcgen05.mma.cta_group::2, 256 x 256 tiles) keeps its 256 rows of A for a run of neighbouring tiles and streams B only,
// each CTA half of it: 16 KB per CTA and k-block, a third of the bytes.  The tiles are dealt out in equal runs along N, so a
// pair changes its rows once or twice; each k-block of A is replaced as soon as the last tile that reads it has issued its
// products.
//
// Sixteen epilogue warps (64 columns or 32 (up, gate) pairs of 32 rows each).  Plain results leave through a 2 KB slot per warp and
// the TMA (28.7 us against 31.4 with stores from the registers).  The three pieces of a SwiGLU tile do not: a piece takes
// 1.4 us from the slot's wait to its release, three of them longer than the tile's products (3 us), and larger slots have no room
// beside A; there a lane stores its row itself, whole 32-byte sectors at a time (st.global.v8; 41.8 -> 38.8 us).
//
// us on one B200, the persistent kernel against this one (operands rotating over more than L2; writing 96 MB alone takes 26 us):
//   8192 x 1536 x 512 16.9 -> 15.5   8192 x 4096 x 512 33.8 -> 29.0   16384 x 2048 x 512 35.1 -> 29.8   8192 x 3072 x 384 23.6 -> 20.4
//   SwiGLU: 8192 x 512 -> 2048 46.9 -> 39.0   16384 x 512 -> 2048 82.3 -> 76   8192 x 384 -> 1536 38 -> 34.5
//   with the exact quotient: 5000 x 384 -> 1536 29.6 -> 24.1 (21.4 without)   2048 x 512 -> 2048 19.5 -> 16.2 (15.0)   8192 x 512 -> 1024 31.3 -> 27.1 (24.5)
// What is left: stores and set-up.  8192 x 4096 x 512 keeps the tensor pipe active 63 % of the time, DRAM at 10 % (ncu).
//
// All waits are bounded (status word on expiry); plain per-CTA TMA loads, no multicast.

#include <stdlib.h>

#include "tcgen05_ptx.cuh"

namespace {

constexpr int BM = 128, BN = 256, BK = 64, UMMA_K = 16;
constexpr int EPI_WARPS = 16, THREADS = 32 * (2 + EPI_WARPS), MAX_KB = 8, MAX_STAGES = 8;
constexpr int BLOCK_BYTES = 16384;             // 128 rows x 64 columns: a k-block of A, a CTA's half of a k-block of B
constexpr int SLOT_BYTES = 2048;               // 32 rows x 32 bf16 columns
constexpr int MAX_DYN_SMEM = 232448;

__device__ __forceinline__ void st_global_v8(void* p, uint32_t a, uint32_t b, uint32_t c, uint32_t d, uint32_t e, uint32_t f, uint32_t g, uint32_t h) {
  asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
               ::"l"(p), "r"(a), "r"(b), "r"(c), "r"(d), "r"(e), "r"(f), "r"(g), "r"(h) : "memory");
}

struct ResidentParams {
  int M, N, b_mn, pair_off;
  __nv_bfloat16 *C, *C2;        // (SwiGLU)
  int ldc, ldc2;
  int m_blocks, n_blocks, kblocks, stages;
  int* status;
};

// EXACT: z has the bits of the separate pass (rte_swiglu_fwd), else those of the persistent kernel's epilogue.
template <int EPI, bool EXACT>
__global__ void __launch_bounds__(THREADS, 1)
gemm_resident_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b, const __grid_constant__ CUtensorMap tmap_c,
                     const ResidentParams p) {
  constexpr bool SWIGLU = EPI == RTE_EPI_SWIGLU_FWD;
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t bars[2 * MAX_KB + 2 * MAX_STAGES + 4];
  __shared__ uint32_t tmem_slot;
  __shared__ int err_flag;
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;      // A k-blocks, B stages, slots
  const uint32_t b_base = smem_base + uint32_t(p.kblocks) * BLOCK_BYTES, slot_base = b_base + uint32_t(p.stages) * BLOCK_BYTES;
  const uint32_t bar0 = smem_u32(bars);
  auto afull_bar = [&](int k) { return bar0 + 8u * k; };
  auto aempty_bar = [&](int k) { return bar0 + 8u * (MAX_KB + k); };
  auto full_bar = [&](int s) { return bar0 + 8u * (2 * MAX_KB + s); };
  auto empty_bar = [&](int s) { return bar0 + 8u * (2 * MAX_KB + MAX_STAGES + s); };
  auto tfull_bar = [&](int b) { return bar0 + 8u * (2 * MAX_KB + 2 * MAX_STAGES + b); };
  auto tempty_bar = [&](int b) { return bar0 + 8u * (2 * MAX_KB + 2 * MAX_STAGES + 2 + b); };

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const bool leader = rank == 0;

  if (threadIdx.x == 0) {
    for (int k = 0; k < MAX_KB; ++k) { mbar_init(afull_bar(k), 1); mbar_init(aempty_bar(k), 1); }
    for (int s = 0; s < MAX_STAGES; ++s) { mbar_init(full_bar(s), 1); mbar_init(empty_bar(s), 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(tfull_bar(b), 1); mbar_init(tempty_bar(b), 2 * EPI_WARPS); }
    err_flag = 0;
    fence_barrier_init();
    prefetch_tmap(&tmap_a);
    prefetch_tmap(&tmap_b);
  }
  if (warp == 1) {
    tmem_alloc<2>(smem_u32(&tmem_slot), 2 * BN);
    tmem_relinquish<2>();
  }
  rte::grid_dependency_wait();
  tc_fence_before();
  cluster_sync_all();
  tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(&tmem_slot);
  rte::grid_dependents_launch();

  // this pair's run of tiles: n fastest, so that neighbours share their rows
  const int pairs = gridDim.x / 2, pair = blockIdx.x / 2;
  const long long tiles = (long long)p.m_blocks * p.n_blocks;
  const int t_lo = int(tiles * pair / pairs), t_hi = int(tiles * (pair + 1) / pairs);
  auto give_up = [&](int code) {
    if (p.status && lane == 0) atomicExch(p.status, code);
    *reinterpret_cast<volatile int*>(&err_flag) = 1;
  };

  if (warp == 0) {
    // ---------------- TMA producer (both CTAs; the leader's barriers count the bytes of both)
    int stage = 0; uint32_t phase = 0, a_phase = 0; bool ok = true;
    for (int t = t_lo; t < t_hi && ok; ++t) {
      const int m = t / p.n_blocks, n = t - m * p.n_blocks, m0 = (m * 2 + int(rank)) * BM;
      const bool rows = t == t_lo || n == 0;
      for (int k = 0; k < p.kblocks && ok; ++k) {
        if (rows) {
          if (t != t_lo && !mbar_wait<2>(aempty_bar(k), a_phase ^ 1u)) { give_up(RTE_DEV_WAIT_TIMEOUT_PRODUCER); ok = false; break; }
          if (elect_one()) {
            if (leader) mbar_arrive_expect_tx(afull_bar(k), 2 * BLOCK_BYTES);
            tma_load_2d<2>(smem_base + uint32_t(k) * BLOCK_BYTES, &tmap_a, mapa_cluster(afull_bar(k), 0), k * BK, m0);
          }
        }
        if (!mbar_wait<2>(empty_bar(stage), phase ^ 1u)) { give_up(RTE_DEV_WAIT_TIMEOUT_PRODUCER); ok = false; break; }
        if (elect_one()) {
          if (leader) mbar_arrive_expect_tx(full_bar(stage), 2 * BLOCK_BYTES);
          const uint32_t fb = mapa_cluster(full_bar(stage), 0), sb = b_base + uint32_t(stage) * BLOCK_BYTES;
          // SwiGLU: the leader stages the tile's 128 up rows, its peer the matching gate rows
          const int col = SWIGLU ? int(rank) * p.pair_off + n * (BN / 2) : n * BN + int(rank) * (BN / 2);
          if (!p.b_mn) {
            tma_load_2d<2>(sb, &tmap_b, fb, k * BK, col);
          } else {
            tma_load_2d<2>(sb, &tmap_b, fb, col, k * BK);
            tma_load_2d<2>(sb + 8192, &tmap_b, fb, col + 64, k * BK);
          }
        }
        if (++stage == p.stages) { stage = 0; phase ^= 1u; }
      }
      if (rows) a_phase ^= 1u;
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer (the leader's, for both CTAs)
    if (leader) {
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (uint32_t(p.b_mn) << 16) | (uint32_t(BN >> 3) << 17) | (uint32_t((2 * BM) >> 4) << 24);
      const uint32_t b_step = p.b_mn ? (UMMA_K * 128u) >> 4 : (UMMA_K * 2u) >> 4;
      const uint64_t adesc0 = make_smem_desc(smem_base, false), bdesc0 = make_smem_desc(b_base, p.b_mn != 0);
      int stage = 0; uint32_t phase = 0, a_phase = 0, acc_phase = 0; int acc = 0; bool ok = true;
      for (int t = t_lo; t < t_hi && ok; ++t) {
        const int n = t % p.n_blocks;
        const bool first = t == t_lo || n == 0, last = n == p.n_blocks - 1 && t + 1 < t_hi;      // of the tiles on these rows; more rows follow
        if (!mbar_wait<2>(tempty_bar(acc), acc_phase ^ 1u)) { give_up(RTE_DEV_WAIT_TIMEOUT_MMA); break; }
        tc_fence_after();
        for (int k = 0; k < p.kblocks; ++k) {
          if ((first && !mbar_wait<2>(afull_bar(k), a_phase)) || !mbar_wait<2>(full_bar(stage), phase)) { give_up(RTE_DEV_WAIT_TIMEOUT_MMA); ok = false; break; }
          tc_fence_after();
          const uint64_t a = adesc0 + uint64_t(uint32_t(k) * (BLOCK_BYTES >> 4)), b = bdesc0 + uint64_t(uint32_t(stage) * (BLOCK_BYTES >> 4));
          if (elect_one()) {
#pragma unroll
            for (int j = 0; j < BK / UMMA_K; ++j)
              tc_mma_bf16<2>(tmem + acc * BN, a + uint64_t(j * ((UMMA_K * 2u) >> 4)), b + uint64_t(j * b_step), idesc, (k > 0 || j > 0) ? 1u : 0u);
            tc_commit<2>(empty_bar(stage));
            if (last) tc_commit<2>(aempty_bar(k));
          }
          if (++stage == p.stages) { stage = 0; phase ^= 1u; }
        }
        if (!ok) break;
        if (elect_one()) tc_commit<2>(tfull_bar(acc));
        if (++acc == 2) { acc = 0; acc_phase ^= 1u; }
        if (first) a_phase ^= 1u;
      }
    }
    __syncwarp();
  } else {
    // ---------------- epilogue: warp w reads the TMEM lanes of quadrant w % 4 (32 rows); the four warps of a quadrant take a
    // quarter of the tile's columns each
    const int quad = warp & 3, part = (warp - 2) >> 2;
    const uint32_t tempty_leader = mapa_cluster(tempty_bar(0), 0);
    uint32_t acc_phase = 0; int acc = 0;
    // 32 columns (16 packed words a lane): by way of this warp's slot, 64-byte rows with the 64-byte swizzle ...
    const uint32_t slot = slot_base + uint32_t(warp - 2) * SLOT_BYTES, mine = slot + uint32_t(lane) * 64u, swz = (uint32_t(lane) >> 1) & 3u;
    auto by_tma = [&](const uint32_t (&v)[16], int x, int y) {
      if (lane == 0) bulk_wait_read<0>();
      __syncwarp();
#pragma unroll
      for (uint32_t c = 0; c < 4; ++c) st_shared_v4(mine + ((c ^ swz) << 4), v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3]);
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) { tma_store_3d(&tmap_c, slot, x, y, 0); bulk_commit(); }
    };
    // ... or as two 32-byte sectors of this lane's row
    auto by_row = [&](__nv_bfloat16* to, const uint32_t (&v)[16]) {
      st_global_v8(to, v[0], v[1], v[2], v[3], v[4], v[5], v[6], v[7]);
      st_global_v8(to + 16, v[8], v[9], v[10], v[11], v[12], v[13], v[14], v[15]);
    };
    auto pack = [](const uint32_t (&raw)[32], uint32_t (&v)[16]) {
#pragma unroll
      for (int j = 0; j < 16; ++j) v[j] = rte::pack_bf16x2(__uint_as_float(raw[2 * j]), __uint_as_float(raw[2 * j + 1]));
    };
    for (int t = t_lo; t < t_hi; ++t) {
      const int m = t / p.n_blocks, n = t - m * p.n_blocks, y = (m * 2 + int(rank)) * BM + quad * 32;
      if (!mbar_wait<2>(tfull_bar(acc), acc_phase)) { give_up(RTE_DEV_WAIT_TIMEOUT_EPILOGUE); break; }
      tc_fence_after();
      const uint32_t at = tmem + (uint32_t(quad * 32) << 16) + acc * BN;
      uint32_t raw0[32], raw1[32], v0[16], v1[16];
      tmem_ld32(at + (SWIGLU ? 32 * part : 64 * part), raw0);
      tmem_ld32(at + (SWIGLU ? BN / 2 + 32 * part : 64 * part + 32), raw1);
      tmem_ld_wait();
      pack(raw0, v0);
      pack(raw1, v1);
      // (the accumulators are in registers: the next tile may have them)
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(tempty_leader + 8u * acc);
      if (++acc == 2) { acc = 0; acc_phase ^= 1u; }
      if (SWIGLU) {
        const int row = y + lane, col = n * (BN / 2) + 32 * part;
        if (row < p.M && col < p.pair_off) {
          __nv_bfloat16* ug = p.C2 + size_t(row) * p.ldc2 + col;
          by_row(ug, v0);
          by_row(ug + p.pair_off, v1);
          // z = up * silu(gate) from the ROUNDED up and gate: what backward re-reads must agree with what was multiplied here
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const float2 u = rte::unpack_bf16x2(v0[j]), g = rte::unpack_bf16x2(v1[j]);
            v0[j] = EXACT ? rte::pack_bf16x2(u.x * rte::silu_of_bf16(g.x), u.y * rte::silu_of_bf16(g.y))
                          : rte::pack_bf16x2(u.x * rte::fast_silu(g.x), u.y * rte::fast_silu(g.y));
          }
          by_row(p.C + size_t(row) * p.ldc + col, v0);
        }
      } else {
        const int col = n * BN + 64 * part;
        if (y < p.M && col < p.N) by_tma(v0, col, y);
        if (y < p.M && col + 32 < p.N) by_tma(v1, col + 32, y);
      }
      __syncwarp();                            // (lanes whose row lies outside stored nothing: the next tile's loads from TMEM want the whole warp)
    }
    if (lane == 0) bulk_wait_read<0>();
    __syncwarp();
  }

  tc_fence_before();
  if (*reinterpret_cast<volatile int*>(&err_flag) != 0) {      // a wait ran out: copies may still be in flight, a bounded time to land
    for (int i = 0; i < 64; ++i) __nanosleep(1000);
  }
  cluster_sync_all();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc<2>(tmem, 2 * BN);
  }
}

constexpr int fixed_bytes(int epi) { return 1024 + (epi == RTE_EPI_BF16 ? EPI_WARPS * SLOT_BYTES : 0); }
int resident_smem(int epi, int kblocks, int stages) { return (kblocks + stages) * BLOCK_BYTES + fixed_bytes(epi); }
int resident_stages(int epi, int kblocks) {
  const int fit = (MAX_DYN_SMEM - 1024 - fixed_bytes(epi)) / BLOCK_BYTES - kblocks;      // (1 KB for the static part)
  return fit < MAX_STAGES ? fit : MAX_STAGES;
}

template <int EPI, bool EXACT>
int max_pairs(int sms) {
  static int pairs = 0;
  if (pairs > 0) return pairs;
  if (cudaFuncSetAttribute(gemm_resident_kernel<EPI, EXACT>, cudaFuncAttributeMaxDynamicSharedMemorySize, resident_smem(EPI, MAX_KB, resident_stages(EPI, MAX_KB))) != cudaSuccess)
    return 0;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(unsigned(sms / 2 * 2));
  cfg.blockDim = dim3(THREADS);
  cfg.dynamicSmemBytes = resident_smem(EPI, MAX_KB, resident_stages(EPI, MAX_KB));
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr; cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, gemm_resident_kernel<EPI, EXACT>, &cfg) == cudaSuccess && n > 0) pairs = n;
  else { (void)cudaGetLastError(); pairs = sms / 2; }
  return pairs;
}

int store_tmap(CUtensorMap* map, const void* base, long long rows, long long cols, long long ld) {
  EncodeTiledFn fn = get_encode_fn();
  if (!fn) return RTE_ERR_TENSOR_MAP;
  cuuint64_t dims[3] = {cuuint64_t(cols), cuuint64_t(rows), 1};
  cuuint64_t strides[2] = {cuuint64_t(ld) * 2, cuuint64_t(ld) * 2 * cuuint64_t(rows)};
  cuuint32_t box[3] = {32, 32, 1}, estr[3] = {1, 1, 1};
  const CUresult r = encode_tiled(fn, map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, cuuint32_t(3), const_cast<void*>(base), dims, strides, box, estr,
                                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_NONE,
                                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? RTE_OK : RTE_ERR_TENSOR_MAP;
}

template <int EPI, bool EXACT>
int launch_resident(const rte_gemm_args* a, int ctas, cudaStream_t st) {
  ResidentParams p;
  p.M = a->M; p.N = a->N; p.b_mn = a->b_mn_major ? 1 : 0; p.pair_off = a->b_pair_offset;
  p.m_blocks = rte::ceil_div(a->M, 2 * BM);
  p.n_blocks = EPI == RTE_EPI_SWIGLU_FWD ? rte::ceil_div(a->b_pair_offset, BN / 2) : rte::ceil_div(a->N, BN);
  p.kblocks = rte::ceil_div(a->K, BK);
  p.stages = resident_stages(EPI, p.kblocks);
  p.status = a->status;
  CUtensorMap ta, tb;
  int rc = make_tmap(&ta, a->A, a->M, a->K, a->lda, BK, BM);
  if (rc != RTE_OK) return rc;
  rc = p.b_mn ? make_tmap(&tb, a->B, a->K, a->N, a->ldb, 64, BK) : make_tmap(&tb, a->B, a->N, a->K, a->ldb, BK, BN / 2);
  if (rc != RTE_OK) return rc;
  p.C = reinterpret_cast<__nv_bfloat16*>(a->C); p.C2 = reinterpret_cast<__nv_bfloat16*>(a->C2);
  p.ldc = a->ldc; p.ldc2 = a->ldc2;
  CUtensorMap tc = ta;
  if (EPI == RTE_EPI_BF16) rc = store_tmap(&tc, a->C, a->M, a->N, a->ldc);
  if (rc != RTE_OK) return rc;
  const int sms = rte_device_sm_count(), fit = max_pairs<EPI, EXACT>(sms);
  int pairs = ctas / 2 < fit ? ctas / 2 : fit;
  const long long tiles = (long long)p.m_blocks * p.n_blocks;
  if (tiles < pairs) pairs = int(tiles);
  if (pairs < 1) return RTE_ERR_LAUNCH;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(unsigned(2 * pairs));
  cfg.blockDim = dim3(THREADS);
  cfg.dynamicSmemBytes = resident_smem(EPI, p.kblocks, p.stages);
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = 2; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr; cfg.numAttrs = 2;
  if (cudaLaunchKernelEx(&cfg, gemm_resident_kernel<EPI, EXACT>, ta, tb, tc, p) != cudaSuccess) {
    (void)cudaGetLastError();
    return RTE_ERR_LAUNCH;
  }
  RTE_LAUNCH_CHECK();
  return RTE_OK;
}

}  // namespace

// What the kernel takes: rows of results that start on 32 bytes (SwiGLU's stores are whole sectors; plain results leave by the TMA and could do
// with 16, not measured), (up, gate) pairs in whole pieces.
extern "C" int rte_gemm_bf16_resident(const rte_gemm_args* a, int32_t ctas, rte_stream_t stream) {
  RTE_CHECK_ARG(a != nullptr && a->A && a->B && a->C && a->M > 0 && a->N > 0 && a->K > 0 && a->K <= MAX_KB * BK && ctas >= 2);
  RTE_CHECK_ARG(a->epilogue == RTE_EPI_BF16 || a->epilogue == RTE_EPI_SWIGLU_FWD);
  RTE_CHECK_ARG(!a->a_mn_major && a->splits <= 1 && a->tile_group == nullptr && a->split_kblocks == nullptr);
  if (((reinterpret_cast<uintptr_t>(a->A) | reinterpret_cast<uintptr_t>(a->B)) & 15) || (reinterpret_cast<uintptr_t>(a->C) & 31) || a->lda % 8 ||
      a->ldb % 8 || a->ldc % 16)
    return RTE_ERR_ALIGNMENT;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (a->epilogue == RTE_EPI_BF16) return launch_resident<RTE_EPI_BF16, false>(a, ctas, st);
  RTE_CHECK_ARG(a->C2 != nullptr && a->b_pair_offset > 0 && a->b_pair_offset % 32 == 0 && a->N == 2 * a->b_pair_offset && !a->b_mn_major);
  if ((reinterpret_cast<uintptr_t>(a->C2) & 31) || a->ldc2 % 16) return RTE_ERR_ALIGNMENT;
  // z by the bits of the route that a caller would otherwise take: the separate pass below the persistent kernel's line, that kernel above
  if ((long long)a->M * a->b_pair_offset < rte_swiglu_fuse_min(0)) return launch_resident<RTE_EPI_SWIGLU_FWD, true>(a, ctas, st);
  return launch_resident<RTE_EPI_SWIGLU_FWD, false>(a, ctas, st);
}
