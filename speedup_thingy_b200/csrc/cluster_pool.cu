// Static cluster-pool sparse SwiGLU FFN: the pieces around the grouped tensor-core GEMMs
// (reference layers.py:188-220, kernels/cluster_pool_ffn.py:90-241).
//
//   route  : token -> centre with the largest score (lowest index on ties), scores = q . centre
//            (the reference L2-normalises q first; a positive per-token scale cannot change the arg-max)
//   pack   : stable counting sort of the tokens by cluster into ONE packed row order in which every cluster
//            starts on a 128-row boundary, so each 128-row GEMM tile belongs to exactly one cluster and
//            no shape ever depends on the routing (the reference pads every cluster to the largest one and
//            reads that size back to the host).  Emits the tile -> cluster table and the per-cluster
//            k-block ranges the grouped GEMMs consume.
//   gather : row gather with conversion and zero fill (pack x / dY, un-pack Y / dX)
//   reduce : pool-gradient rows summed into dense FFN rows through a CSR built once per codebook: a
//            gather-reduce in fixed order instead of the reference's index_add_ scatter (no atomics,
//            bitwise reproducible).
//   transpose: [R, C] fp32 -> [C, R] bf16 / fp32 (W_down is stored [d, F]; its pool rows are rows of W_down^T)

#include "rte_common.cuh"

namespace {

constexpr int PACK_THREADS = 1024;
constexpr int MAX_CLUSTERS = 64;

// One warp per token.  Sixteen clusters' products are reduced together: every exchange of the butterfly halves the values a
// lane still carries, so a token takes 16 shuffles per 16 clusters instead of 80 in 16 dependent chains, with the sums of
// the plain butterfly bit for bit (8192 tokens, 16 clusters of 64: 15 -> 6 us).
__global__ void __launch_bounds__(256)
cluster_route_kernel(const float* __restrict__ q, int ldq, const float* __restrict__ centers, int32_t* __restrict__ assign,
                     float* __restrict__ scores_out, int n, int W, int C) {
  rte::after_previous_grid();
  extern __shared__ float sc[];              // centres [C][W] when they fit
  const bool in_smem = (size_t)C * W * sizeof(float) <= 96 * 1024;
  if (in_smem) {
    for (int i = threadIdx.x; i < C * W; i += blockDim.x) sc[i] = centers[i];
    __syncthreads();
  }
  const float* cen = in_smem ? sc : centers;
  const int lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  for (int tok = blockIdx.x * warps + (threadIdx.x >> 5); tok < n; tok += gridDim.x * warps) {
    const float* row = q + (size_t)tok * ldq;
    float best = -INFINITY;
    int best_c = 0;
    for (int c0 = 0; c0 < C; c0 += 16) {
      float v[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) v[i] = 0.f;
      for (int k = lane; k < W; k += 32) {
        const float x = row[k];
#pragma unroll
        for (int i = 0; i < 16; ++i)
          if (c0 + i < C) v[i] += x * cen[(size_t)(c0 + i) * W + k];
      }
      // after the exchange over 2h lanes a lane with that bit set keeps the upper half of its values
      int who = 0;
#pragma unroll
      for (int h = 8; h >= 1; h >>= 1) {
        const bool up = lane & (2 * h);
#pragma unroll
        for (int i = 0; i < h; ++i) {
          const float keep = up ? v[i + h] : v[i], give = up ? v[i] : v[i + h];
          v[i] = keep + __shfl_xor_sync(0xffffffffu, give, 2 * h);
        }
        who += up ? h : 0;
      }
      const float score = v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1);
      const int c = c0 + who;                                // (lanes 2j and 2j + 1 hold the same cluster)
      if (scores_out && !(lane & 1) && c < C) scores_out[(size_t)tok * C + c] = score;
      const bool counts = c < C && score == score;            // (a NaN is larger than nothing)
      float m = counts ? score : -INFINITY;
      int mc = counts ? c : 0x7fffffff;
#pragma unroll
      for (int o = 16; o >= 2; o >>= 1) {
        const float om = __shfl_xor_sync(0xffffffffu, m, o);
        const int oc = __shfl_xor_sync(0xffffffffu, mc, o);
        if (om > m || (om == m && oc < mc)) { m = om; mc = oc; }
      }
      if (m > best) { best = m; best_c = mc; }             // strict: the lowest index wins ties
    }
    if (lane == 0) assign[tok] = best_c;
  }
}

// Single CTA.  perm[p] = token packed at row p (-1: padding row); pos[token] = its packed row.  Every warp owns a contiguous
// range of tokens and walks it twice: once to count its tokens per cluster, once, after a scan of those counts over the
// warps, to place them, with nothing but its own counters in between (chunks of 1024 tokens with four barriers each:
// 8192 tokens 21 -> 9 us).
__global__ void __launch_bounds__(PACK_THREADS)
cluster_pack_kernel(const int32_t* __restrict__ assign, int n, int C, int cap, int32_t* __restrict__ perm,
                    int32_t* __restrict__ pos, int32_t* __restrict__ counts, int32_t* __restrict__ offsets,
                    int32_t* __restrict__ tile_group, int32_t* __restrict__ kblocks, int* status) {
  rte::after_previous_grid();
  constexpr int WARPS = PACK_THREADS / 32;
  __shared__ int total[MAX_CLUSTERS];
  __shared__ int base[MAX_CLUSTERS + 1];
  __shared__ int wc[WARPS][MAX_CLUSTERS];
  __shared__ int bad;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int i = tid; i < WARPS * MAX_CLUSTERS; i += PACK_THREADS) (&wc[0][0])[i] = 0;
  if (tid == 0) bad = 0;
  __syncthreads();
  const int per = (n + PACK_THREADS - 1) / PACK_THREADS * 32, lo = min(n, warp * per), hi = min(n, lo + per);
  for (int i0 = lo; i0 < hi; i0 += 256) {
    int a[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) a[u] = i0 + 32 * u + lane < hi ? assign[i0 + 32 * u + lane] : -1 - lane;      // (idle lanes: distinct dummies)
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      if (i0 + 32 * u >= hi) break;
      const bool in = i0 + 32 * u + lane < hi;
      if (in && (a[u] < 0 || a[u] >= C)) { bad = 1; a[u] = -1 - lane; }
      const unsigned peers = __match_any_sync(0xffffffffu, a[u]);
      if (a[u] >= 0 && (peers & ((1u << lane) - 1u)) == 0) wc[warp][a[u]] += __popc(peers);
      __syncwarp();
    }
  }
  for (int i = tid; i < cap; i += PACK_THREADS) perm[i] = -1;
  __syncthreads();
  for (int c = warp; c < C; c += WARPS) {            // a warp per cluster: exclusive scan of its counts over the warps
    const int mine = wc[lane][c];
    int sum = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, sum, o);
      if (lane >= o) sum += t;
    }
    wc[lane][c] = sum - mine;
    if (lane == 31) total[c] = sum;
  }
  __syncthreads();
  if (tid == 0) {
    int off = 0;
    for (int c = 0; c < C; ++c) {
      base[c] = off;
      off += (total[c] + 127) / 128 * 128;
    }
    base[C] = off;
    if (off > cap || bad) { if (status) atomicExch(status, off > cap ? RTE_DEV_CAPACITY_OVERFLOW : RTE_DEV_INDEX_OUT_OF_RANGE); bad = 1; }
  }
  __syncthreads();
  if (tid <= C) {
    offsets[tid] = base[tid];
    kblocks[tid] = base[tid] / 64;
    if (tid < C) counts[tid] = total[tid];
  }
  for (int b = tid; b < cap / 128; b += PACK_THREADS) {
    int g = -1;
    if (!bad)
      for (int c = 0; c < C; ++c)
        if (b * 128 >= base[c] && b * 128 < base[c + 1]) g = c;
    tile_group[b] = g;
  }
  if (bad) { for (int i = tid; i < n; i += PACK_THREADS) pos[i] = -1; return; }
  // stable placement: token order is kept inside every cluster
  for (int i0 = lo; i0 < hi; i0 += 256) {
    int a[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) a[u] = i0 + 32 * u + lane < hi ? assign[i0 + 32 * u + lane] : -1 - lane;
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      if (i0 + 32 * u >= hi) break;
      const unsigned peers = __match_any_sync(0xffffffffu, a[u]);
      if (a[u] >= 0) {
        const int i = i0 + 32 * u + lane, rank = __popc(peers & ((1u << lane) - 1u));
        const int p = base[a[u]] + wc[warp][a[u]] + rank;
        perm[p] = i;
        pos[i] = p;
      }
      __syncwarp();
      if (a[u] >= 0 && (peers & ((1u << lane) - 1u)) == 0) wc[warp][a[u]] += __popc(peers);
      __syncwarp();
    }
  }
}

template <typename T>
__device__ __forceinline__ float4 row4(const T* p, bool wide) {
  if constexpr (sizeof(T) == 2) {
    if (wide) {
      const uint2 w = *reinterpret_cast<const uint2*>(p);
      const float2 a = rte::unpack_bf16x2(w.x), b = rte::unpack_bf16x2(w.y);
      return make_float4(a.x, a.y, b.x, b.y);
    }
  } else {
    if (wide) return *reinterpret_cast<const float4*>(p);
  }
  return make_float4((float)p[0], (float)p[1], (float)p[2], (float)p[3]);
}
template <typename T>
__device__ __forceinline__ void put4(T* p, bool wide, const float4& v) {
  if constexpr (sizeof(T) == 2) {
    if (wide) { *reinterpret_cast<uint2*>(p) = make_uint2(rte::pack_bf16x2(v.x, v.y), rte::pack_bf16x2(v.z, v.w)); return; }
  } else {
    if (wide) { *reinterpret_cast<float4*>(p) = v; return; }
  }
  p[0] = (T)v.x; p[1] = (T)v.y; p[2] = (T)v.z; p[3] = (T)v.w;
}

// dst[i, :] = convert(src[idx[i], :]) or zeros when idx[i] < 0.  A warp per row, four columns per lane, four loads in flight
// (an element index divided by the width in 64 bits per four columns cost more than the copy).
template <typename TS, typename TD>
__global__ void __launch_bounds__(256)
gather_convert_kernel(const TS* __restrict__ src, const int32_t* __restrict__ idx, TD* __restrict__ dst, long long n_out, int d, int wide) {
  rte::after_previous_grid();
  const int lane = threadIdx.x & 31, d4 = d >> 2;
  for (long long r = blockIdx.x * 8LL + (threadIdx.x >> 5); r < n_out; r += gridDim.x * 8LL) {
    const int s = idx[r];
    const TS* p = src + (size_t)(s < 0 ? 0 : s) * d;
    TD* o = dst + (size_t)r * d;
#pragma unroll 4
    for (int c = lane; c < d4; c += 32) put4(o + 4 * c, wide, s < 0 ? make_float4(0.f, 0.f, 0.f, 0.f) : row4(p + 4 * c, wide));
  }
}

// dense[f, :] (+)= sum over k in [row_ptr[f], row_ptr[f+1]) of src[rows[k], :]     (fixed order).  A CTA of 128 threads per
// dense row, four columns per thread, the rows of four members requested together.
__global__ void __launch_bounds__(128)
csr_row_reduce_kernel(const float* __restrict__ src, const int32_t* __restrict__ row_ptr, const int32_t* __restrict__ rows,
                      float* __restrict__ dense, long long n_dense, int d, int accumulate) {
  rte::after_previous_grid();
  const int d4 = d >> 2;
  for (long long f = blockIdx.x; f < n_dense; f += gridDim.x) {
    const int k0 = row_ptr[f], k1 = row_ptr[f + 1];
    for (int c = threadIdx.x; c < d4; c += 128) {
      float4* out = reinterpret_cast<float4*>(dense + (size_t)f * d) + c;
      float4 acc = accumulate ? *out : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
      for (int k = k0; k < k1; ++k) {
        const float4 t = reinterpret_cast<const float4*>(src + (size_t)rows[k] * d)[c];
        acc.x += t.x; acc.y += t.y; acc.z += t.z; acc.w += t.w;
      }
      *out = acc;
    }
  }
}

template <typename TD>
__global__ void __launch_bounds__(256)
transpose_kernel(const float* __restrict__ src, TD* __restrict__ dst, int R, int C, int accumulate) {
  rte::after_previous_grid();
  __shared__ float tile[32][33];
  const int c0 = blockIdx.x * 32, r0 = blockIdx.y * 32;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;          // 32 x 8
  for (int j = ty; j < 32; j += 8) {
    const int r = r0 + j, c = c0 + tx;
    tile[j][tx] = (r < R && c < C) ? src[(size_t)r * C + c] : 0.f;
  }
  __syncthreads();
  for (int j = ty; j < 32; j += 8) {
    const int c = c0 + j, r = r0 + tx;
    if (r < R && c < C) {
      const size_t o = (size_t)c * R + r;
      const float v = tile[tx][j] + (accumulate ? (float)dst[o] : 0.f);
      dst[o] = (TD)v;
    }
  }
}

inline int grid_for(long long n, int block, int cap = 148 * 16) {
  long long g = (n + block - 1) / block;
  return (int)(g < 1 ? 1 : (g > cap ? cap : g));
}

}  // namespace

#define ST(s) reinterpret_cast<cudaStream_t>(s)

extern "C" int rte_cluster_route(const float* q, int32_t ldq, const float* centers, int32_t* assignments, float* scores_out,
                                 int32_t n_tokens, int32_t width, int32_t n_clusters, rte_stream_t stream) {
  RTE_CHECK_ARG(q && centers && assignments && n_tokens > 0 && width > 0 && n_clusters > 0 && ldq >= width);
  const size_t smem = (size_t)n_clusters * width * sizeof(float);
  const size_t use = smem <= 96 * 1024 ? smem : 0;
  if (use > 48 * 1024) {
    static bool set = false;
    if (!set) {
      if (cudaFuncSetAttribute(cluster_route_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 96 * 1024) != cudaSuccess)
        return RTE_ERR_LAUNCH;
      set = true;
    }
  }
  rte::launch(cluster_route_kernel, grid_for(n_tokens, 8, 148 * 8), 256, use, ST(stream), q, ldq, centers, assignments, scores_out, n_tokens,
                                                                            width, n_clusters);
  RTE_LAUNCH_CHECK();
  return RTE_OK;
}

extern "C" int rte_cluster_pack(const int32_t* assignments, int32_t n_tokens, int32_t n_clusters, int32_t capacity_rows,
                                int32_t* perm, int32_t* pos, int32_t* counts, int32_t* offsets, int32_t* tile_group,
                                int32_t* kblocks, int32_t* status, rte_stream_t stream) {
  RTE_CHECK_ARG(assignments && perm && pos && counts && offsets && tile_group && kblocks && n_tokens > 0 && n_clusters > 0);
  RTE_CHECK_ARG(capacity_rows > 0 && capacity_rows % 128 == 0);
  if (n_clusters > MAX_CLUSTERS) return RTE_ERR_UNSUPPORTED;
  rte::launch(cluster_pack_kernel, 1, PACK_THREADS, 0, ST(stream), assignments, n_tokens, n_clusters, capacity_rows, perm, pos, counts,
                                                          offsets, tile_group, kblocks, status);
  RTE_LAUNCH_CHECK();
  return RTE_OK;
}

extern "C" int rte_gather_rows_convert(const void* src, int32_t src_bf16, const int32_t* idx, void* dst, int32_t dst_bf16,
                                       int64_t n_out, int32_t d, rte_stream_t stream) {
  RTE_CHECK_ARG(src && idx && dst && n_out > 0 && d > 0 && d % 4 == 0);
  const int g = grid_for(n_out, 8, 148 * 16);
  using bf = __nv_bfloat16;
  const int wide = (reinterpret_cast<uintptr_t>(src) & (src_bf16 ? 7 : 15)) == 0 && (reinterpret_cast<uintptr_t>(dst) & (dst_bf16 ? 7 : 15)) == 0;
  if (src_bf16 && dst_bf16) rte::launch(gather_convert_kernel<bf, bf>, g, 256, 0, ST(stream), (const bf*)src, idx, (bf*)dst, n_out, d, wide);
  else if (src_bf16) rte::launch(gather_convert_kernel<bf, float>, g, 256, 0, ST(stream), (const bf*)src, idx, (float*)dst, n_out, d, wide);
  else if (dst_bf16) rte::launch(gather_convert_kernel<float, bf>, g, 256, 0, ST(stream), (const float*)src, idx, (bf*)dst, n_out, d, wide);
  else rte::launch(gather_convert_kernel<float, float>, g, 256, 0, ST(stream), (const float*)src, idx, (float*)dst, n_out, d, wide);
  RTE_LAUNCH_CHECK();
  return RTE_OK;
}

extern "C" int rte_csr_row_reduce_f32(const float* src, const int32_t* row_ptr, const int32_t* rows, float* dense,
                                      int64_t n_dense_rows, int32_t d, int32_t accumulate, rte_stream_t stream) {
  RTE_CHECK_ARG(src && row_ptr && rows && dense && n_dense_rows > 0 && d > 0 && d % 4 == 0);
  if ((reinterpret_cast<uintptr_t>(src) & 15) || (reinterpret_cast<uintptr_t>(dense) & 15)) return RTE_ERR_ALIGNMENT;
  rte::launch(csr_row_reduce_kernel, grid_for(n_dense_rows, 1, 148 * 16), 128, 0, ST(stream), src, row_ptr, rows, dense, n_dense_rows, d,
                                                                                     accumulate);
  RTE_LAUNCH_CHECK();
  return RTE_OK;
}

extern "C" int rte_transpose_f32(const float* src, void* dst, int32_t rows, int32_t cols, int32_t dst_bf16, int32_t accumulate,
                                 rte_stream_t stream) {
  RTE_CHECK_ARG(src && dst && rows > 0 && cols > 0);
  dim3 grid(rte::ceil_div(cols, 32), rte::ceil_div(rows, 32));
  if (dst_bf16) rte::launch(transpose_kernel<__nv_bfloat16>, grid, 256, 0, ST(stream), src, (__nv_bfloat16*)dst, rows, cols, accumulate);
  else rte::launch(transpose_kernel<float>, grid, 256, 0, ST(stream), src, (float*)dst, rows, cols, accumulate);
  RTE_LAUNCH_CHECK();
  return RTE_OK;
}
