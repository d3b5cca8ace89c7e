// bf16 GEMM for products that do not fill the GPU: C[M,N] = A[M,K] * B[N,K]^T, one 128 x BN tile per CTA
// (tcgen05.mma.cta_group::1, accumulators in TMEM), operands by TMA, the reduction optionally split over the CTAs of
// a thread-block cluster that add their partial tiles through distributed shared memory.
//
// The persistent kernel (gemm_tcgen05.cu) is built for many tiles per SM: 256-row tiles, an epilogue that hides behind
// the next tile's main loop, set-up paid once.  With fewer tiles than SMs none of that applies; what counts is how long
// ONE tile takes from launch to its last store.  So here
//   * tiles are small (128 x 128 or 128 x 64) and a long reduction is cut into up to eight pieces that run at the same
//     time; each CTA of a cluster leaves its fp32 partial tile in shared memory and adds, for its share of the rows,
//     the partials of all ranks in rank order (a fixed order: results are reproducible);
//   * several CTAs fit on an SM (about 100 KB and BN TMEM columns each), so that one's set-up and epilogue overlap
//     another's main loop when there are more tiles than SMs; with fewer, every k-block of the tile is in flight at once;
//   * the first loads are issued by the thread that initialised the barriers, before TMEM has been allocated;
//   * rows leave (and residual rows arrive) as whole-warp 256/512-byte accesses.
//
// Operand majors as in gemm_tcgen05.cu.  All waits are bounded (status word on expiry).

#include <stdlib.h>

#include "tcgen05_ptx.cuh"

namespace {

constexpr int BM = 128, BK = 64, UMMA_K = 16, THREADS = 256, MAX_STAGES = 8;
constexpr int MAX_SMEM = 8 * (16384 + 8192) + 1024;

struct TileParams {
  int M, N, a_mn, b_mn;
  void* C; int ldc;
  const float* R; int ldr;
  int out_f32, vec;             // vec: rows of C and R start on 16 bytes
  int m_blocks, kblocks, ksplit, stages;
  int* status;
};

__device__ __forceinline__ float4 ld_cluster_v4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}

template <int BN>
__global__ void __launch_bounds__(THREADS, 2)
gemm_tile_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b, const TileParams p) {
  constexpr int STAGE_BYTES = (BM + BN) * BK * 2;
  constexpr int LD = BN + 4;                       // floats per row of the fp32 tile in shared memory
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t bars[2 * MAX_STAGES + 1];
  __shared__ uint32_t tmem_ptr;
  __shared__ int failed;
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  float* tile = reinterpret_cast<float*>(smem_raw + (smem_base - smem_u32(smem_raw)));
  const uint32_t bar0 = smem_u32(bars);
  auto full_bar = [&](int s) { return bar0 + 8u * s; };
  auto empty_bar = [&](int s) { return bar0 + 8u * (MAX_STAGES + s); };
  const uint32_t done_bar = bar0 + 8u * (2 * MAX_STAGES);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = blockIdx.x % p.ksplit, t = blockIdx.x / p.ksplit;
  const int m0 = (t % p.m_blocks) * BM, n0 = (t / p.m_blocks) * BN;
  const int kb0 = p.kblocks * rank / p.ksplit, nk = p.kblocks * (rank + 1) / p.ksplit - kb0;
  const int stages = p.stages;

  auto load = [&](int i, int stage) {              // k-block kb0 + i into a stage (one elected lane)
    const uint32_t sa = smem_base + stage * STAGE_BYTES, sb = sa + BM * BK * 2, fb = full_bar(stage);
    const int k0 = (kb0 + i) * BK;
    mbar_arrive_expect_tx(fb, STAGE_BYTES);
    if (!p.a_mn) {
      tma_load_2d<1>(sa, &tmap_a, fb, k0, m0);
    } else {
      tma_load_2d<1>(sa, &tmap_a, fb, m0, k0);
      tma_load_2d<1>(sa + 8192, &tmap_a, fb, m0 + 64, k0);
    }
    if (!p.b_mn) {
      tma_load_2d<1>(sb, &tmap_b, fb, k0, n0);
    } else {
#pragma unroll
      for (int j = 0; j < BN / 64; ++j) tma_load_2d<1>(sb + j * 8192, &tmap_b, fb, n0 + 64 * j, k0);
    }
  };

  if (warp == 0) {
    if (elect_one()) {
      for (int s = 0; s < stages; ++s) { mbar_init(full_bar(s), 1); mbar_init(empty_bar(s), 1); }
      mbar_init(done_bar, 1);
      failed = 0;
      fence_barrier_init();
      prefetch_tmap(&tmap_a);
      prefetch_tmap(&tmap_b);
    }
    __syncwarp();
    rte::grid_dependency_wait();
    for (int i = 0; i < min(nk, stages); ++i)
      if (elect_one()) load(i, i);
  } else {
    if (warp == 1) {
      tmem_alloc<1>(smem_u32(&tmem_ptr), BN);
      tmem_relinquish<1>();
    }
    rte::grid_dependency_wait();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_ptr;
  rte::grid_dependents_launch();

  if (warp == 0) {
    int stage = 0; uint32_t phase = 0;
    for (int i = stages; i < nk; ++i) {
      if (!mbar_wait<1>(empty_bar(stage), phase)) {
        if (p.status && lane == 0) atomicExch(p.status, RTE_DEV_WAIT_TIMEOUT_PRODUCER);
        failed = 1;
        break;
      }
      if (elect_one()) load(i, stage);
      if (++stage == stages) { stage = 0; phase ^= 1u; }
    }
    __syncwarp();
  } else if (warp == 1) {
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (uint32_t(p.a_mn) << 15) | (uint32_t(p.b_mn) << 16) |
                           (uint32_t(BN >> 3) << 17) | (uint32_t(BM >> 4) << 24);
    const uint32_t a_step = p.a_mn ? (UMMA_K * 128u) >> 4 : (UMMA_K * 2u) >> 4;
    const uint32_t b_step = p.b_mn ? (UMMA_K * 128u) >> 4 : (UMMA_K * 2u) >> 4;
    const uint64_t adesc0 = make_smem_desc(smem_base, p.a_mn != 0), bdesc0 = make_smem_desc(smem_base + BM * BK * 2, p.b_mn != 0);
    int stage = 0; uint32_t phase = 0;
    for (int i = 0; i < nk; ++i) {
      if (!mbar_wait<1>(full_bar(stage), phase)) {
        if (p.status && lane == 0) atomicExch(p.status, RTE_DEV_WAIT_TIMEOUT_MMA);
        failed = 1;
        break;
      }
      tc_fence_after();
      const uint64_t off = uint64_t(uint32_t(stage) * uint32_t(STAGE_BYTES >> 4));     // (addresses stay below the field's end)
      if (elect_one()) {
#pragma unroll
        for (int k = 0; k < BK / UMMA_K; ++k)
          tc_mma_bf16<1>(tmem, adesc0 + off + uint64_t(k * a_step), bdesc0 + off + uint64_t(k * b_step), idesc, (i > 0 || k > 0) ? 1u : 0u);
        tc_commit<1>(empty_bar(stage));
      }
      if (++stage == stages) { stage = 0; phase ^= 1u; }
    }
    if (elect_one()) tc_commit<1>(done_bar);
    __syncwarp();
  }

  // ---------------- this rank's share of the rows: a row per BN / 4 lanes, one float4 each; the residual of the first
  // RB rows per thread is fetched while the main loop runs
  constexpr int CPR = BN / 4, RPP = THREADS / CPR, RB = 8;
  const int c4 = threadIdx.x % CPR, col = n0 + 4 * c4;
  const int valid = min(BM, p.M - m0), per = (valid + p.ksplit - 1) / p.ksplit;
  const int r_first = rank * per + threadIdx.x / CPR, r_hi = col < p.N ? min(valid, (rank + 1) * per) : 0;
  const bool whole = p.vec && col + 4 <= p.N, with_res = p.R != nullptr && whole;
  float4 res[RB];
  auto fetch = [&](int r0) {
#pragma unroll
    for (int j = 0; j < RB; ++j) {
      const int r = r0 + j * RPP;
      res[j] = (with_res && r < r_hi) ? *reinterpret_cast<const float4*>(p.R + (size_t)(m0 + r) * p.ldr + col) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  };
  fetch(r_first);

  // ---------------- the tile: TMEM -> shared memory (the stages are free once every MMA has completed)
  if (!mbar_wait<1>(done_bar, 0)) {
    if (p.status && lane == 0) atomicExch(p.status, RTE_DEV_WAIT_TIMEOUT_EPILOGUE);
    failed = 1;
  }
  tc_fence_after();
  {
    const int quad = warp & 3, row = quad * 32 + lane, c_lo = (warp >> 2) * (BN / 2);
    const uint32_t t_row = tmem + (uint32_t(quad * 32) << 16);
    float* out = tile + row * LD;
#pragma unroll
    for (int c = 0; c < BN / 2; c += 32) {
      uint32_t raw[32];
      tmem_ld32(t_row + c_lo + c, raw);
      tmem_ld_wait();
#pragma unroll
      for (int q = 0; q < 8; ++q)
        *reinterpret_cast<float4*>(out + c_lo + c + 4 * q) = make_float4(__uint_as_float(raw[4 * q]), __uint_as_float(raw[4 * q + 1]),
                                                                          __uint_as_float(raw[4 * q + 2]), __uint_as_float(raw[4 * q + 3]));
    }
  }
  tc_fence_before();
  if (p.ksplit > 1) cluster_sync_all(); else __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc<1>(tmem, BN);
  }

  // ---------------- sum of the ranks' partials in rank order (+ residual)
  const uint32_t tile_addr = smem_u32(tile) + 16u * c4;
  uint32_t peer[8];
#pragma unroll
  for (int s = 0; s < 8; ++s) peer[s] = s < p.ksplit ? mapa_cluster(tile_addr, s) : 0u;
  for (int r0 = r_first; r0 < r_hi; r0 += RB * RPP) {
    if (r0 != r_first) fetch(r0);
#pragma unroll
    for (int j = 0; j < RB; ++j) {
      const int r = r0 + j * RPP;
      if (r >= r_hi) break;
      const size_t row = (size_t)(m0 + r);
      float4 v;
      if (p.ksplit == 1) {
        v = *reinterpret_cast<const float4*>(tile + r * LD + 4 * c4);
      } else {
        v = ld_cluster_v4(peer[0] + r * (LD * 4));
#pragma unroll
        for (int s = 1; s < 8; ++s)
          if (s < p.ksplit) {
            const float4 w = ld_cluster_v4(peer[s] + r * (LD * 4));
            v.x += w.x; v.y += w.y; v.z += w.z; v.w += w.w;
          }
      }
      if (whole) {
        v.x += res[j].x; v.y += res[j].y; v.z += res[j].z; v.w += res[j].w;
        if (p.out_f32) *reinterpret_cast<float4*>(reinterpret_cast<float*>(p.C) + row * p.ldc + col) = v;
        else *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(p.C) + row * p.ldc + col) =
                 make_uint2(rte::pack_bf16x2(v.x, v.y), rte::pack_bf16x2(v.z, v.w));
      } else {
        const float e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (col + q < p.N) {
            const float x = e[q] + (p.R != nullptr ? p.R[row * p.ldr + col + q] : 0.f);
            if (p.out_f32) reinterpret_cast<float*>(p.C)[row * p.ldc + col + q] = x;
            else reinterpret_cast<__nv_bfloat16*>(p.C)[row * p.ldc + col + q] = __float2bfloat16_rn(x);
          }
      }
    }
  }
  if (p.ksplit > 1) cluster_sync_all();            // nobody leaves while a peer may still read its tile
  if (failed) {                                    // a wait ran out: give copies still in flight a bounded time to land
    for (int i = 0; i < 64; ++i) __nanosleep(1000);
    __syncthreads();
  }
}

template <int BN>
int launch_tile(const rte_gemm_args* a, int ksplit, cudaStream_t st) {
  TileParams p;
  p.M = a->M; p.N = a->N; p.a_mn = a->a_mn_major ? 1 : 0; p.b_mn = a->b_mn_major ? 1 : 0;
  p.out_f32 = a->epilogue == RTE_EPI_F32 ? 1 : 0;
  p.C = a->C; p.ldc = a->ldc; p.R = p.out_f32 ? reinterpret_cast<const float*>(a->R) : nullptr; p.ldr = a->ldr;      // (bf16 outputs take no R)
  const long long es = p.out_f32 ? 4 : 2;
  p.vec = (reinterpret_cast<uintptr_t>(a->C) & 15) == 0 && (a->ldc * es) % 16 == 0 &&
          (p.R == nullptr || ((reinterpret_cast<uintptr_t>(p.R) & 15) == 0 && p.ldr % 4 == 0));
  p.m_blocks = rte::ceil_div(a->M, BM);
  p.kblocks = rte::ceil_div(a->K, BK);
  p.ksplit = ksplit;
  p.status = a->status;
  const int tiles = p.m_blocks * rte::ceil_div(a->N, BN), grid = tiles * ksplit;
  // enough stages for every k-block of a CTA while one CTA per SM is all there is; otherwise what lets two share an SM
  constexpr int stage_bytes = (BM + BN) * BK * 2, deep = BN == 128 ? 6 : 8, shared = BN == 128 ? 3 : 4;
  const int per_cta = rte::ceil_div(p.kblocks, ksplit);
  p.stages = grid <= rte_device_sm_count() ? deep : shared;
  if (p.stages > per_cta) p.stages = per_cta;
  int smem = p.stages * stage_bytes;
  if (smem < BM * (BN + 4) * 4) smem = BM * (BN + 4) * 4;
  smem += 1024;
  CUtensorMap ta, tb;
  int rc = p.a_mn ? make_tmap(&ta, a->A, a->K, a->M, a->lda, 64, BK) : make_tmap(&ta, a->A, a->M, a->K, a->lda, BK, BM);
  if (rc != RTE_OK) return rc;
  rc = p.b_mn ? make_tmap(&tb, a->B, a->K, a->N, a->ldb, 64, BK) : make_tmap(&tb, a->B, a->N, a->K, a->ldb, BK, BN);
  if (rc != RTE_OK) return rc;
  static bool set = false;
  if (!set) {
    if (cudaFuncSetAttribute(gemm_tile_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, MAX_SMEM) != cudaSuccess) return RTE_ERR_LAUNCH;
    set = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(unsigned(grid));
  cfg.blockDim = dim3(THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = ksplit; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  if (ksplit == 1) attr[0] = attr[1];
  cfg.attrs = attr; cfg.numAttrs = ksplit > 1 ? 2 : 1;
  if (cudaLaunchKernelEx(&cfg, gemm_tile_kernel<BN>, ta, tb, p) != cudaSuccess) {
    (void)cudaGetLastError();
    return RTE_ERR_LAUNCH;
  }
  RTE_LAUNCH_CHECK();
  return RTE_OK;
}

}  // namespace

extern "C" int rte_gemm_bf16_tile(const rte_gemm_args* a, int32_t tile_n, int32_t ksplit, rte_stream_t stream) {
  RTE_CHECK_ARG(a != nullptr && a->A && a->B && a->C && a->M > 0 && a->N > 0 && a->K > 0);
  RTE_CHECK_ARG(a->epilogue == RTE_EPI_BF16 || a->epilogue == RTE_EPI_F32);
  RTE_CHECK_ARG(a->splits <= 1 && a->tile_group == nullptr && a->split_kblocks == nullptr);
  RTE_CHECK_ARG((tile_n == 64 || tile_n == 128) && ksplit >= 1 && ksplit <= 8 && ksplit <= rte::ceil_div(a->K, BK));
  if ((reinterpret_cast<uintptr_t>(a->A) & 15) || (reinterpret_cast<uintptr_t>(a->B) & 15) || (a->lda % 8) || (a->ldb % 8))
    return RTE_ERR_ALIGNMENT;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  return tile_n == 128 ? launch_tile<128>(a, ksplit, st) : launch_tile<64>(a, ksplit, st);
}
