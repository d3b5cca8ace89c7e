// Offline cluster-pool codebook build on the GPU: cosine k-means over the selector features, per-cluster score
// aggregation, per-neuron pool scores.  (Cluster assignment is rte_cluster_route, candidate selection
// rte_topk_lowest_index.)  Every reduction runs in a fixed order: the result is reproducible bit for bit.

#include "rte_common.cuh"

namespace {

#define ST(s) reinterpret_cast<cudaStream_t>(s)

// out[r, :] = x[r, :] / max(||x[r, :]||_2, 1e-12); one warp per row.
__global__ void __launch_bounds__(256)
normalize_rows_kernel(const float* __restrict__ x, float* __restrict__ out, int n, int W) {
  rte::after_previous_grid();
  const int lane = threadIdx.x & 31, row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= n) return;
  const float* xr = x + (size_t)row * W;
  float s = 0.f;
  for (int k = lane; k < W; k += 32) { const float v = xr[k]; s += v * v; }
  s = rte::warp_sum(s);
  const float inv = 1.f / fmaxf(sqrtf(s), 1e-12f);
  for (int k = lane; k < W; k += 32) out[(size_t)row * W + k] = xr[k] * inv;
}

// One CTA per (cluster, chunk of 256 columns): thread = column.  Members are visited in token order, so the sums do
// not depend on scheduling.  mode 0: centre update (mean of members, L2-normalised; an empty cluster keeps its old
// centre, normalised); mode 1: mean of the members' scores; mode 2: max (zeros when empty).
__global__ void __launch_bounds__(256)
cluster_reduce_kernel(const float* __restrict__ x, const int32_t* __restrict__ assign, const float* __restrict__ old,
                      float* __restrict__ out, int32_t* __restrict__ counts, int n, int W, int mode) {
  rte::after_previous_grid();
  __shared__ float red[32];
  __shared__ int32_t sa[1024];
  const int c = blockIdx.x, col = blockIdx.y * 256 + threadIdx.x;
  float acc = (mode == 2) ? -INFINITY : 0.f;
  int cnt = 0;
  for (int base = 0; base < n; base += 1024) {
    __syncthreads();
    for (int i = threadIdx.x; i < 1024; i += 256) sa[i] = (base + i < n) ? assign[base + i] : -1;
    __syncthreads();
    const int lim = min(1024, n - base);
    for (int i = 0; i < lim; ++i) {
      if (sa[i] == c) {
        ++cnt;
        if (col < W) {
          const float v = x[(size_t)(base + i) * W + col];
          acc = (mode == 2) ? fmaxf(acc, v) : acc + v;
        }
      }
    }
  }
  if (counts != nullptr && blockIdx.y == 0 && threadIdx.x == 0) counts[c] = cnt;
  if (mode != 0) {
    if (col < W) out[(size_t)c * W + col] = cnt > 0 ? (mode == 1 ? acc / (float)cnt : acc) : 0.f;
    return;
  }
  // centre update: the norm spans all columns, so mode 0 is launched with one column chunk per pass over W <= 256,
  // or (wider) normalised by a following normalize_rows launch; here W <= 256 is required by the host wrapper
  float v = (col < W) ? (cnt > 0 ? acc / (float)cnt : old[(size_t)c * W + col]) : 0.f;
  const float s = rte::block_sum(v * v, red);
  if (col < W) out[(size_t)c * W + col] = v / fmaxf(sqrtf(s), 1e-12f);
}

// Pool score of every (token, neuron) from the low-rank estimates of the up and gate pre-activations:
//   up = |up_hat| * wd_norm, gate = |silu(gate_hat)| * wd_norm, product = |up_hat * silu(gate_hat)| * wd_norm;
//   mode 0: up + gate + product ("sum"), 1: up + gate ("upgate"), 2: product.
__global__ void __launch_bounds__(256)
pool_scores_kernel(const float* __restrict__ up_hat, const float* __restrict__ gate_hat, const float* __restrict__ wd_norm,
                   float* __restrict__ out, long long total, int F, int mode) {
  rte::after_previous_grid();
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const float u = up_hat[i], g = gate_hat[i], w = wd_norm[i % F];
    const float ga = g / (1.f + expf(-g));
    const float us = fabsf(u) * w, gs = fabsf(ga) * w, ps = fabsf(u * ga) * w;
    out[i] = mode == 0 ? us + gs + ps : (mode == 1 ? us + gs : ps);
  }
}

}  // namespace

extern "C" int rte_normalize_rows_f32(const float* x, float* out, int32_t n, int32_t W, rte_stream_t stream) {
  RTE_CHECK_ARG(x && out && n > 0 && W > 0);
  rte::launch(normalize_rows_kernel, rte::ceil_div(n, 8), 256, 0, ST(stream), x, out, n, W);
  RTE_LAUNCH_CHECK();
  return RTE_OK;
}

extern "C" int rte_kmeans_update(const float* x_normed, const int32_t* assignments, const float* centers_old, float* centers_new,
                                 int32_t* counts, int32_t n, int32_t W, int32_t C, rte_stream_t stream) {
  RTE_CHECK_ARG(x_normed && assignments && centers_old && centers_new && n > 0 && W > 0 && C > 0);
  if (W > 256) return RTE_ERR_UNSUPPORTED;          // the centre's norm is taken inside one CTA
  rte::launch(cluster_reduce_kernel, dim3(C, 1), 256, 0, ST(stream), x_normed, assignments, centers_old, centers_new, counts, n, W, 0);
  RTE_LAUNCH_CHECK();
  return RTE_OK;
}

extern "C" int rte_cluster_aggregate(const float* scores, const int32_t* assignments, float* out, int32_t n, int32_t F, int32_t C,
                                     int32_t use_max, rte_stream_t stream) {
  RTE_CHECK_ARG(scores && assignments && out && n > 0 && F > 0 && C > 0);
  rte::launch(cluster_reduce_kernel, dim3(C, rte::ceil_div(F, 256)), 256, 0, ST(stream), scores, assignments, nullptr, out, nullptr, n, F,
                                                                               use_max ? 2 : 1);
  RTE_LAUNCH_CHECK();
  return RTE_OK;
}

extern "C" int rte_cluster_pool_scores(const float* up_hat, const float* gate_hat, const float* wd_norm, float* out, int64_t n,
                                       int32_t F, int32_t mode, rte_stream_t stream) {
  RTE_CHECK_ARG(up_hat && gate_hat && wd_norm && out && n > 0 && F > 0 && mode >= 0 && mode <= 2);
  const long long total = (long long)n * F;
  long long g = (total + 255) / 256;
  if (g > 148 * 16) g = 148 * 16;
  rte::launch(pool_scores_kernel, (int)g, 256, 0, ST(stream), up_hat, gate_hat, wd_norm, out, total, F, mode);
  RTE_LAUNCH_CHECK();
  return RTE_OK;
}
