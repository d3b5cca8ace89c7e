// Per-sample router of the recursive model and the backward pass of its auxiliary losses.
// One decision per SAMPLE from pooled = mean over the sequence of h0: two small MLPs
// (d -> hid -> R recipes, d -> hid -> K depths), softmaxes, arg-max ids with ties to the LOWEST
// index, per-pass recipe ids (logits + per-pass bias), entropies, expected depth.
// The matrices are tiny (hid x d floats, read once per sample from L2), so one CTA per sample.

#include "rte_common.cuh"

namespace {

constexpr int NTHR = 256;

__device__ __forceinline__ float4 load4(const float* p, bool wide) {
  return wide ? *reinterpret_cast<const float4*>(p) : make_float4(p[0], p[1], p[2], p[3]);
}

// pooled[b,c] = mean over s.  CTA = one sample x 128 columns; its eight warps take every eighth token, eight loads in flight
// each (a thread per column walking all S tokens: 32 x 256 x 1024 50 -> 19 us for 34 MB).
__global__ void __launch_bounds__(NTHR)
pool_kernel(const float* __restrict__ h0, float* __restrict__ pooled, int S, int d) {
  rte::after_previous_grid();
  __shared__ float4 part[NTHR];
  const int b = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, c = blockIdx.x * 128 + 4 * lane;
  const bool wide = (reinterpret_cast<uintptr_t>(h0) & 15) == 0;
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  if (c < d) {
    const float* p = h0 + (size_t)b * S * d + c;
#pragma unroll 8
    for (int s = warp; s < S; s += NTHR / 32) {
      const float4 x = load4(p + (size_t)s * d, wide);
      acc.x += x.x; acc.y += x.y; acc.z += x.z; acc.w += x.w;
    }
  }
  part[threadIdx.x] = acc;
  __syncthreads();
  if (threadIdx.x < 128) {
    const int col = blockIdx.x * 128 + threadIdx.x;
    const float* q = reinterpret_cast<const float*>(part) + threadIdx.x;
    float t = 0.f;
#pragma unroll
    for (int w = 0; w < NTHR / 32; ++w) t += q[128 * w];
    if (col < d) pooled[(size_t)b * d + col] = t / (float)S;
  }
}

__device__ __forceinline__ int argmax_lowest(const float* v, int n) {
  int best = 0;
  for (int i = 1; i < n; ++i) if (v[i] > v[best]) best = i;   // strict '>' keeps the lowest index on ties
  return best;
}
__device__ __forceinline__ void softmax_small(const float* logits, float* probs, int n) {
  float mx = logits[0];
  for (int i = 1; i < n; ++i) mx = fmaxf(mx, logits[i]);
  float s = 0.f;
  for (int i = 0; i < n; ++i) { probs[i] = expf(logits[i] - mx); s += probs[i]; }
  const float inv = 1.f / s;
  for (int i = 0; i < n; ++i) probs[i] *= inv;
}

// Hidden layer of one router MLP for 16 samples x 32 hidden rows per CTA: the samples' pooled vectors sit in shared memory
// and a warp dots its four weight rows with them together, so one shared read feeds four products (a row at a time the
// kernel was bound by those reads: 32 samples x 1024 -> 1024 46 -> 20 us).
constexpr int RH_SAMPLES = 16, RH_ROWS = 32, RH_PER_WARP = RH_ROWS / (NTHR / 32);
__global__ void __launch_bounds__(NTHR)
router_hidden_kernel(const float* __restrict__ pooled, const float* __restrict__ w0a, const float* __restrict__ b0a,
                     float* __restrict__ prea, const float* __restrict__ w0b, const float* __restrict__ b0b,
                     float* __restrict__ preb, int B, int d, int hid) {
  rte::after_previous_grid();
  extern __shared__ __align__(16) float xs[];                 // [RH_SAMPLES][d]
  const float* w0 = blockIdx.z == 0 ? w0a : w0b;
  const float* b0 = blockIdx.z == 0 ? b0a : b0b;
  float* pre = blockIdx.z == 0 ? prea : preb;
  const int s0 = blockIdx.y * RH_SAMPLES, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int d4 = d >> 2, n = min(RH_SAMPLES, B - s0) * d4;          // (the samples' vectors are contiguous)
  const bool wide = (reinterpret_cast<uintptr_t>(pooled) & 15) == 0;
  for (int i = threadIdx.x; i < RH_SAMPLES * d4; i += NTHR)
    reinterpret_cast<float4*>(xs)[i] = i < n ? load4(pooled + (size_t)s0 * d + 4 * (size_t)i, wide) : make_float4(0.f, 0.f, 0.f, 0.f);
  __syncthreads();
  const int j0 = blockIdx.x * RH_ROWS + warp * RH_PER_WARP;
  if (j0 >= hid) return;
  float acc[RH_PER_WARP][RH_SAMPLES];
#pragma unroll
  for (int r = 0; r < RH_PER_WARP; ++r)
#pragma unroll
    for (int q = 0; q < RH_SAMPLES; ++q) acc[r][q] = 0.f;
  const bool wide_w = (reinterpret_cast<uintptr_t>(w0) & 15) == 0;
  for (int c = lane; c < d4; c += 32) {
    float4 w[RH_PER_WARP];
#pragma unroll
    for (int r = 0; r < RH_PER_WARP; ++r) w[r] = load4(w0 + (size_t)min(j0 + r, hid - 1) * d + 4 * c, wide_w);
#pragma unroll
    for (int q = 0; q < RH_SAMPLES; ++q) {
      const float4 x = reinterpret_cast<const float4*>(xs)[q * d4 + c];
#pragma unroll
      for (int r = 0; r < RH_PER_WARP; ++r) acc[r][q] += w[r].x * x.x + w[r].y * x.y + w[r].z * x.z + w[r].w * x.w;
    }
  }
#pragma unroll
  for (int r = 0; r < RH_PER_WARP; ++r) {
    const int j = j0 + r;
    float mine = 0.f;
#pragma unroll
    for (int q = 0; q < RH_SAMPLES; ++q) {
      const float v = rte::warp_sum(acc[r][q]);
      if (lane == q) mine = v;
    }
    if (lane < RH_SAMPLES && s0 + lane < B && j < hid) pre[(size_t)(s0 + lane) * hid + j] = mine + b0[j];
  }
}

__device__ void head_logits(const float* __restrict__ pre, const float* __restrict__ w2, const float* __restrict__ b2,
                            float* hs, float* logits, int hid, int nout) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int j = threadIdx.x; j < hid; j += NTHR) hs[j] = rte::silu_f(pre[j]);
  __syncthreads();
  for (int r = warp; r < nout; r += NTHR / 32) {
    float acc = 0.f;
#pragma unroll 4
    for (int j = lane; j < hid; j += 32) acc += w2[(size_t)r * hid + j] * hs[j];
    acc = rte::warp_sum(acc);
    if (lane == 0) logits[r] = acc + b2[r];
  }
  __syncthreads();
}

__global__ void __launch_bounds__(NTHR)
router_fwd_kernel(rte_router_weights w, const int32_t* __restrict__ depth_values, rte_router_out o, int d, int hid,
                  int R, int K, int T, int fixed_recipe, int fixed_depth_id) {
  rte::after_previous_grid();
  extern __shared__ float sm[];   // hs[hid]
  __shared__ float rl[RTE_ROUTER_MAX_R], dl[RTE_ROUTER_MAX_K];
  float* hs = sm;
  const int b = blockIdx.x;
  head_logits(o.r_hidden_pre + (size_t)b * hid, w.r_w2, w.r_b2, hs, rl, hid, R);
  head_logits(o.d_hidden_pre + (size_t)b * hid, w.d_w2, w.d_b2, hs, dl, hid, K);
  if (threadIdx.x == 0) {
    float rp[RTE_ROUTER_MAX_R], dp[RTE_ROUTER_MAX_K];
    softmax_small(rl, rp, R);
    softmax_small(dl, dp, K);
    float rent = 0.f, dent = 0.f, ed = 0.f;
    for (int r = 0; r < R; ++r) {
      o.recipe_logits[(size_t)b * R + r] = rl[r];
      o.recipe_probs[(size_t)b * R + r] = rp[r];
      rent -= logf(fmaxf(rp[r], 1e-9f)) * rp[r];
    }
    for (int k = 0; k < K; ++k) {
      o.depth_probs[(size_t)b * K + k] = dp[k];
      dent -= logf(fmaxf(dp[k], 1e-9f)) * dp[k];
      ed += dp[k] * (float)depth_values[k];
    }
    o.expected_depth[b] = ed;
    o.router_entropy[b] = rent + dent;
    o.recipe_id[b] = fixed_recipe >= 0 ? fixed_recipe : argmax_lowest(rp, R);
    const int did = fixed_depth_id >= 0 ? fixed_depth_id : argmax_lowest(dp, K);
    o.depth_id[b] = did;
    o.depth[b] = depth_values[did];
  } else if (threadIdx.x >= 32) {              // a thread per pass, next to the sample's own softmaxes
    float tmp[RTE_ROUTER_MAX_R], tp[RTE_ROUTER_MAX_R];
    for (int t = threadIdx.x - 32; t < T; t += NTHR - 32) {
      int id = fixed_recipe;
      if (fixed_recipe < 0) {
        for (int r = 0; r < R; ++r) tmp[r] = rl[r] + w.pass_recipe_bias[t * R + r];
        softmax_small(tmp, tp, R);
        id = argmax_lowest(tp, R);
      }
      o.recipe_id_by_pass[(size_t)b * T + t] = id;
    }
  }
}

// aux losses and the batch-mean of the recipe probabilities
__global__ void __launch_bounds__(NTHR)
aux_kernel(const float* __restrict__ recipe_probs, const float* __restrict__ expected_depth, float lambda_load,
           float lambda_depth, float* __restrict__ aux, float* __restrict__ mean_prob, const float* __restrict__ mean_given,
           int B, int R) {
  rte::after_previous_grid();
  __shared__ float red[32];
  __shared__ float mp[RTE_ROUTER_MAX_R];
  for (int r = threadIdx.x; r < R; r += NTHR) {
    float acc = 0.f;
    if (mean_given != nullptr) {          // the batch mean over ALL data-parallel shards, reduced by the caller
      acc = mean_given[r];
    } else {
      for (int b = 0; b < B; ++b) acc += recipe_probs[(size_t)b * R + r];
      acc /= (float)B;
    }
    mp[r] = acc;
    mean_prob[r] = acc;
  }
  float ed = 0.f;
  for (int b = threadIdx.x; b < B; b += NTHR) ed += expected_depth[b];
  ed = rte::block_sum(ed, red);
  __syncthreads();
  if (threadIdx.x == 0) {
    float sq = 0.f;
    for (int r = 0; r < R; ++r) sq += mp[r] * mp[r];
    aux[0] = lambda_load * ((float)R * sq - 1.f);
    aux[1] = lambda_depth * ed / (float)B;
  }
}

// per-sample backward through softmax and both MLP heads; dh0 += dpooled / S
__device__ void mlp_backward_sample(const float* __restrict__ w2, const float* dlog, const float* __restrict__ pre, float* dpre_out, float* dhs,
                                    int hid, int nout) {
  for (int j = threadIdx.x; j < hid; j += NTHR) {
    float acc = 0.f;
    for (int r = 0; r < nout; ++r) acc += w2[(size_t)r * hid + j] * dlog[r];
    const float a = pre[j], sg = rte::sigmoid_f(a);
    const float v = acc * sg * (1.f + a * (1.f - sg));
    dhs[j] = v;
    dpre_out[j] = v;
  }
  __syncthreads();
}

__global__ void __launch_bounds__(NTHR)
router_bwd_sample_kernel(rte_router_weights w, rte_router_out o, const int32_t* __restrict__ depth_values,
                         const float* __restrict__ mean_prob, float lambda_load, float lambda_depth,
                         float* __restrict__ dpre_r, float* __restrict__ dpre_d, float* __restrict__ dlog_r,
                         float* __restrict__ dlog_d, float* __restrict__ dh0, int B, int S, int d, int hid, int R, int K) {
  rte::after_previous_grid();
  extern __shared__ float sm[];   // dhr[hid], dhd[hid]
  __shared__ float dlr[RTE_ROUTER_MAX_R], dld[RTE_ROUTER_MAX_K];
  float* dhr = sm;
  float* dhd = sm + hid;
  const int b = blockIdx.x;
  if (threadIdx.x == 0) {
    float dot = 0.f;
    for (int r = 0; r < R; ++r) dot += o.recipe_probs[(size_t)b * R + r] * (lambda_load * (float)R * 2.f * mean_prob[r] / (float)B);
    for (int r = 0; r < R; ++r) {
      const float p = o.recipe_probs[(size_t)b * R + r];
      const float v = p * (lambda_load * (float)R * 2.f * mean_prob[r] / (float)B - dot);
      dlr[r] = v;
      dlog_r[(size_t)b * R + r] = v;
    }
    float dotd = 0.f;
    for (int k = 0; k < K; ++k) dotd += o.depth_probs[(size_t)b * K + k] * (lambda_depth * (float)depth_values[k] / (float)B);
    for (int k = 0; k < K; ++k) {
      const float p = o.depth_probs[(size_t)b * K + k];
      const float v = p * (lambda_depth * (float)depth_values[k] / (float)B - dotd);
      dld[k] = v;
      dlog_d[(size_t)b * K + k] = v;
    }
  }
  __syncthreads();
  mlp_backward_sample(w.r_w2, dlr, o.r_hidden_pre + (size_t)b * hid, dpre_r + (size_t)b * hid, dhr, hid, R);
  mlp_backward_sample(w.d_w2, dld, o.d_hidden_pre + (size_t)b * hid, dpre_d + (size_t)b * hid, dhd, hid, K);
}

// dst[r,:] += sum_p vec[p][r / seg,:]   (nparts partial vectors, part_stride floats apart, added in fixed order).  CTA = 256
// float4 columns of one segment and 32 of its rows: the vector is added up once per thread, eight rows are in flight.
constexpr int BC_ROWS = 32;
__global__ void __launch_bounds__(NTHR)
bcast_add_kernel(float* __restrict__ dst, const float* __restrict__ vec, int rows, int seg, int d, int nparts, long long part_stride) {
  rte::after_previous_grid();
  const int d4 = d >> 2, b = blockIdx.z, c = blockIdx.x * NTHR + threadIdx.x;
  if (c >= d4) return;
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int p = 0; p < nparts; ++p) {
    const float4 t = reinterpret_cast<const float4*>(vec + p * part_stride)[(size_t)b * d4 + c];
    v.x += t.x; v.y += t.y; v.z += t.z; v.w += t.w;
  }
  const int r0 = blockIdx.y * BC_ROWS, r1 = min(min(seg, r0 + BC_ROWS), rows - b * seg);
  float4* q = reinterpret_cast<float4*>(dst) + (size_t)b * seg * d4 + c;
#pragma unroll 8
  for (int r = r0; r < r1; ++r) {
    float4 a = q[(size_t)r * d4];
    a.x += v.x; a.y += v.y; a.z += v.z; a.w += v.w;
    q[(size_t)r * d4] = a;
  }
}

// dpooled[part][b,:] = (dpre_r[b, J] @ W0r[J,:] + dpre_d[b, J] @ W0d[J,:]) / S over the part's slice J of the hidden
// dimension (blockIdx.y = part).  CTA = DP_SAMPLES samples x 128 columns (a float4 per lane); its eight warps take every
// eighth j and meet in shared memory in warp order.  The broadcast kernel adds the parts in fixed order.  32 samples x
// 1024 58 -> 20 us.
constexpr int DP_SAMPLES = 8, DP_WARPS = NTHR / 32;
__global__ void __launch_bounds__(NTHR)
router_dpooled_kernel(const float* __restrict__ w0r, const float* __restrict__ w0d, const float* __restrict__ dpre_r,
                      const float* __restrict__ dpre_d, float* __restrict__ dpooled, int B, int S, int d, int hid) {
  rte::after_previous_grid();
  extern __shared__ float sm[];            // sr[part_len][DP_SAMPLES], sd[part_len][DP_SAMPLES]
  __shared__ float4 comb[DP_WARPS / 2][DP_SAMPLES][32];
  const int cblocks = rte::ceil_div(d, 128), lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int b0 = (blockIdx.x / cblocks) * DP_SAMPLES, c = (blockIdx.x % cblocks) * 128 + 4 * lane;
  const int part_len = (hid + (int)gridDim.y - 1) / (int)gridDim.y;
  const int p_lo = min(hid, (int)blockIdx.y * part_len), len = min(hid, p_lo + part_len) - p_lo;
  float* sr = sm;
  float* sd = sm + part_len * DP_SAMPLES;
  dpooled += (size_t)blockIdx.y * B * d;
  for (int q = warp; q < DP_SAMPLES; q += DP_WARPS) {
    const int bb = b0 + q;
    for (int j = lane; j < len; j += 32) {
      sr[j * DP_SAMPLES + q] = bb < B ? dpre_r[(size_t)bb * hid + p_lo + j] : 0.f;
      sd[j * DP_SAMPLES + q] = bb < B ? dpre_d[(size_t)bb * hid + p_lo + j] : 0.f;
    }
  }
  __syncthreads();
  float4 acc[DP_SAMPLES];
#pragma unroll
  for (int q = 0; q < DP_SAMPLES; ++q) acc[q] = make_float4(0.f, 0.f, 0.f, 0.f);
  if (c < d) {
    const bool wide = ((reinterpret_cast<uintptr_t>(w0r) | reinterpret_cast<uintptr_t>(w0d)) & 15) == 0;
#pragma unroll 4
    for (int j = warp; j < len; j += DP_WARPS) {
      const float4 wr = load4(w0r + (size_t)(p_lo + j) * d + c, wide), wd = load4(w0d + (size_t)(p_lo + j) * d + c, wide);
#pragma unroll
      for (int q = 0; q < DP_SAMPLES; ++q) {
        const float r = sr[j * DP_SAMPLES + q], e = sd[j * DP_SAMPLES + q];
        acc[q].x += wr.x * r + wd.x * e;
        acc[q].y += wr.y * r + wd.y * e;
        acc[q].z += wr.z * r + wd.z * e;
        acc[q].w += wr.w * r + wd.w * e;
      }
    }
  }
  // warps 4-7 onto 0-3, then the rest of the tree
#pragma unroll
  for (int w = DP_WARPS / 2; w > 0; w >>= 1) {
    if (warp >= w && warp < 2 * w) {
#pragma unroll
      for (int q = 0; q < DP_SAMPLES; ++q) comb[warp - w][q][lane] = acc[q];
    }
    __syncthreads();
    if (warp < w) {
#pragma unroll
      for (int q = 0; q < DP_SAMPLES; ++q) {
        const float4 v = comb[warp][q][lane];
        acc[q].x += v.x; acc[q].y += v.y; acc[q].z += v.z; acc[q].w += v.w;
      }
    }
    __syncthreads();
  }
  if (warp == 0 && c < d) {
    const float inv = 1.f / (float)S;
#pragma unroll
    for (int q = 0; q < DP_SAMPLES; ++q) {
      if (b0 + q >= B) break;
      float* o = dpooled + (size_t)(b0 + q) * d + c;
      o[0] = acc[q].x * inv; o[1] = acc[q].y * inv; o[2] = acc[q].z * inv; o[3] = acc[q].w * inv;
    }
  }
}

// dW0[j,c] = sum_b dpre[b,j] * pooled[b,c];  db0[j] = sum_b dpre[b,j], for both MLPs (blockIdx.z).  CTA = 64 x 64 outputs, 16
// per thread, 16 samples at a time in shared memory (an output per thread read both operands from L1 for every product:
// 32 samples x 1024 x 1024, both MLPs 167 -> 13 us).
constexpr int W0_TILE = 64, W0_SAMPLES = 16;
struct Dw0Job { const float* dpre; float* dw0; float* db0; };
struct Dw0Jobs { Dw0Job job[2]; };
__global__ void __launch_bounds__(NTHR)
router_dw0_kernel(const Dw0Jobs jobs, const float* __restrict__ pooled, int B, int d, int hid) {
  rte::after_previous_grid();
  __shared__ __align__(16) float sj[W0_SAMPLES][W0_TILE], sc[W0_SAMPLES][W0_TILE];
  const Dw0Job& job = jobs.job[blockIdx.z];
  const int j0 = blockIdx.y * W0_TILE, c0 = blockIdx.x * W0_TILE, tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  float acc[4][4], accb = 0.f;
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int k = 0; k < 4; ++k) acc[i][k] = 0.f;
  for (int b0 = 0; b0 < B; b0 += W0_SAMPLES) {
    __syncthreads();
#pragma unroll
    for (int i = threadIdx.x; i < W0_SAMPLES * W0_TILE; i += NTHR) {
      const int b = b0 + i / W0_TILE, q = i % W0_TILE;
      sj[i / W0_TILE][q] = b < B && j0 + q < hid ? job.dpre[(size_t)b * hid + j0 + q] : 0.f;
      sc[i / W0_TILE][q] = b < B && c0 + q < d ? pooled[(size_t)b * d + c0 + q] : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int b = 0; b < W0_SAMPLES; ++b) {
      const float4 x = *reinterpret_cast<const float4*>(&sc[b][4 * tx]), v = *reinterpret_cast<const float4*>(&sj[b][4 * ty]);
      const float vv[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        acc[i][0] += vv[i] * x.x; acc[i][1] += vv[i] * x.y; acc[i][2] += vv[i] * x.z; acc[i][3] += vv[i] * x.w;
      }
      if (blockIdx.x == 0 && threadIdx.x < W0_TILE) accb += sj[b][threadIdx.x];
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (j0 + 4 * ty + i < hid && c0 + 4 * tx + k < d) job.dw0[(size_t)(j0 + 4 * ty + i) * d + c0 + 4 * tx + k] = acc[i][k];
  if (blockIdx.x == 0 && threadIdx.x < W0_TILE && j0 + threadIdx.x < hid) job.db0[j0 + threadIdx.x] = accb;
}
// dW2[r,j] = sum_b dlog[b,r] * silu(pre[b,j]);  db2[r] = sum_b dlog[b,r].  32 outputs x 8 sample groups per CTA.
__global__ void __launch_bounds__(NTHR)
router_dw2_kernel(const float* __restrict__ dlog, const float* __restrict__ pre, float* __restrict__ dw2,
                  float* __restrict__ db2, int B, int hid, int nout) {
  rte::after_previous_grid();
  __shared__ float sa[8][33], sb[8][33];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int i = blockIdx.x * 32 + tx;
  float acc = 0.f, accb = 0.f;
  if (i < nout * hid) {
    const int r = i / hid, j = i % hid;
#pragma unroll 4
    for (int b = ty; b < B; b += 8) {
      const float v = dlog[(size_t)b * nout + r];
      acc += v * rte::silu_f(pre[(size_t)b * hid + j]);
      accb += v;
    }
  }
  sa[ty][tx] = acc; sb[ty][tx] = accb;
  __syncthreads();
  if (ty == 0 && i < nout * hid) {
    float t = 0.f, u = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) { t += sa[k][tx]; u += sb[k][tx]; }
    dw2[i] = t;
    if (i % hid == 0) db2[i / hid] = u;
  }
}

}  // namespace

#define ST(s) reinterpret_cast<cudaStream_t>(s)

extern "C" int rte_router_fwd(const float* h0, const rte_router_weights* w, const int32_t* depth_values,
                              const rte_router_out* out, int32_t B, int32_t S, int32_t d, int32_t hid, int32_t R,
                              int32_t K, int32_t T, int32_t fixed_recipe, int32_t fixed_depth_id, rte_stream_t stream) {
  RTE_CHECK_ARG(h0 && w && depth_values && out && B > 0 && S > 0 && d > 0 && hid > 0);
  RTE_CHECK_ARG(R > 0 && R <= RTE_ROUTER_MAX_R && K > 0 && K <= RTE_ROUTER_MAX_K && T > 0 && T <= RTE_ROUTER_MAX_T);
  RTE_CHECK_ARG(fixed_recipe < R && fixed_depth_id < K);
  RTE_CHECK_ARG(out->pooled && out->r_hidden_pre && out->d_hidden_pre && out->recipe_logits && out->recipe_probs &&
                out->depth_probs && out->expected_depth && out->router_entropy && out->recipe_id &&
                out->recipe_id_by_pass && out->depth_id && out->depth);
  const size_t smem = (size_t)hid * sizeof(float);
  const size_t smem_h = (size_t)RH_SAMPLES * d * sizeof(float);
  if (smem > 48 * 1024 || d % 4 != 0) return RTE_ERR_UNSUPPORTED;
  if (smem_h > 48 * 1024) {
    static bool set = false;
    if (!set) {
      if (cudaFuncSetAttribute(router_hidden_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 128 * 1024) != cudaSuccess)
        return RTE_ERR_LAUNCH;
      set = true;
    }
  }
  rte::launch(pool_kernel, dim3(rte::ceil_div(d, 128), B), NTHR, 0, ST(stream), h0, out->pooled, S, d);
  RTE_LAUNCH_CHECK();
  rte::launch(router_hidden_kernel, dim3(rte::ceil_div(hid, RH_ROWS), rte::ceil_div(B, RH_SAMPLES), 2), NTHR, smem_h, ST(stream), out->pooled, w->r_w0, w->r_b0, out->r_hidden_pre, w->d_w0, w->d_b0, out->d_hidden_pre, B, d, hid);
  RTE_LAUNCH_CHECK();
  rte::launch(router_fwd_kernel, B, NTHR, smem, ST(stream), *w, depth_values, *out, d, hid, R, K, T, fixed_recipe, fixed_depth_id);
  RTE_LAUNCH_CHECK();
  return RTE_OK;
}

// out[r] = scale * sum_b recipe_probs[b, r]: with scale = 1 / (B * world) the SUM of `out` over the data-parallel ranks is
// the batch mean over the global batch, which rte_router_aux_bwd_data then takes as `mean_prob_in`.
__global__ void __launch_bounds__(NTHR)
mean_prob_kernel(const float* __restrict__ recipe_probs, float* __restrict__ out, float scale, int B, int R) {
  rte::after_previous_grid();
  for (int r = threadIdx.x; r < R; r += NTHR) {
    float acc = 0.f;
    for (int b = 0; b < B; ++b) acc += recipe_probs[(size_t)b * R + r];
    out[r] = acc * scale;
  }
}

extern "C" int rte_router_mean_prob(const float* recipe_probs, float* out, float scale, int32_t B, int32_t R, rte_stream_t stream) {
  RTE_CHECK_ARG(recipe_probs && out && B > 0 && R > 0 && R <= RTE_ROUTER_MAX_R);
  rte::launch(mean_prob_kernel, 1, NTHR, 0, ST(stream), recipe_probs, out, scale, B, R);
  RTE_LAUNCH_CHECK();
  return RTE_OK;
}

// Data-gradient half: the auxiliary losses, d(loss)/d(pre-activations) per sample (left in `scratch`), and
// dh0[b,s,:] += dpooled[b,:] / S -- what the rest of backward waits for.  None of it depends on an upstream
// gradient, so with dh0 == NULL everything but that last add can run as soon as the router's forward is done
// (rte_router_aux_add_dh0 performs the add later, from `scratch`).
extern "C" int rte_router_aux_bwd_data(const rte_router_weights* w, const rte_router_out* fwd, const int32_t* depth_values,
                                       float lambda_load, float lambda_depth, float* aux, float* dh0, float* scratch,
                                       const float* mean_prob_in, int32_t B, int32_t S, int32_t d, int32_t hid, int32_t R,
                                       int32_t K, rte_stream_t stream) {
  RTE_CHECK_ARG(w && fwd && depth_values && aux && scratch && B > 0 && S > 0 && d > 0 && hid > 0);
  RTE_CHECK_ARG(R > 0 && R <= RTE_ROUTER_MAX_R && K > 0 && K <= RTE_ROUTER_MAX_K);
  float* mean_prob = scratch;                       // [RTE_ROUTER_MAX_R]
  float* dpre_r = scratch + RTE_ROUTER_MAX_R;       // [B, hid]
  float* dpre_d = dpre_r + (size_t)B * hid;         // [B, hid]
  float* dlog_r = dpre_d + (size_t)B * hid;         // [B, R]
  float* dlog_d = dlog_r + (size_t)B * R;           // [B, K]
  float* dpooled = const_cast<float*>(rte::router_dpooled(scratch, B, hid, R, K));   // [B, d], 16-byte aligned
  if (reinterpret_cast<uintptr_t>(scratch) & 15) return RTE_ERR_ALIGNMENT;
  rte::launch(aux_kernel, 1, NTHR, 0, ST(stream), fwd->recipe_probs, fwd->expected_depth, lambda_load, lambda_depth, aux, mean_prob,
                                         mean_prob_in, B, R);
  RTE_LAUNCH_CHECK();
  const size_t smem = (size_t)2 * hid * sizeof(float);
  if (smem > 48 * 1024) return RTE_ERR_UNSUPPORTED;
  rte::launch(router_bwd_sample_kernel, B, NTHR, smem, ST(stream), *w, *fwd, depth_values, mean_prob, lambda_load, lambda_depth,
                                                          dpre_r, dpre_d, dlog_r, dlog_d, dh0, B, S, d, hid, R, K);
  RTE_LAUNCH_CHECK();
  const size_t smem_dp = (size_t)2 * rte::ceil_div(hid, RTE_ROUTER_DPOOLED_PARTS) * DP_SAMPLES * sizeof(float);
  if (smem_dp > 32 * 1024 &&
      cudaFuncSetAttribute(router_dpooled_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_dp) != cudaSuccess)
    return RTE_ERR_LAUNCH;
  rte::launch(router_dpooled_kernel, dim3(rte::ceil_div(B, DP_SAMPLES) * rte::ceil_div(d, 128), RTE_ROUTER_DPOOLED_PARTS), NTHR, smem_dp, ST(stream), w->r_w0, w->d_w0, dpre_r, dpre_d, dpooled, B, S, d, hid);
  RTE_LAUNCH_CHECK();
  if (d % 4 != 0) return RTE_ERR_UNSUPPORTED;
  if (dh0) {
    rte::launch(bcast_add_kernel, dim3(rte::ceil_div(d / 4, NTHR), rte::ceil_div(S, BC_ROWS), B), NTHR, 0, ST(stream), dh0, dpooled, B * S, S, d, RTE_ROUTER_DPOOLED_PARTS, (long long)B * d);
    RTE_LAUNCH_CHECK();
  }
  return RTE_OK;
}

int rte::add_router_dpooled(float* dh0, const float* dpooled, int B, int S, int d, cudaStream_t st) {
  rte::launch(bcast_add_kernel, dim3(rte::ceil_div(d / 4, NTHR), rte::ceil_div(S, BC_ROWS), B), NTHR, 0, st, dh0, dpooled, B * S, S, d, RTE_ROUTER_DPOOLED_PARTS, (long long)B * d);
  RTE_LAUNCH_CHECK();
  return RTE_OK;
}

// dh0[b,s,:] += dpooled[b,:] / S from the `scratch` a call of rte_router_aux_bwd_data(dh0 = NULL) left behind.
extern "C" int rte_router_aux_add_dh0(float* dh0, const float* scratch, int32_t B, int32_t S, int32_t d, int32_t hid, int32_t R,
                                      int32_t K, rte_stream_t stream) {
  RTE_CHECK_ARG(dh0 && scratch && B > 0 && S > 0 && d > 0 && hid > 0 && R > 0 && K > 0);
  if (d % 4 != 0) return RTE_ERR_UNSUPPORTED;
  if (reinterpret_cast<uintptr_t>(scratch) & 15) return RTE_ERR_ALIGNMENT;
  return rte::add_router_dpooled(dh0, rte::router_dpooled(scratch, B, hid, R, K), B, S, d, ST(stream));
}

// Parameter-gradient half of the auxiliary-loss backward: reads dpre / dlog left in `scratch` by the data half.
extern "C" int rte_router_aux_bwd_params(const rte_router_out* fwd, const rte_router_grads* grads, float* scratch, int32_t B,
                                         int32_t d, int32_t hid, int32_t R, int32_t K, rte_stream_t stream) {
  RTE_CHECK_ARG(fwd && grads && scratch && B > 0 && d > 0 && hid > 0 && R > 0 && K > 0);
  RTE_CHECK_ARG(grads->r_w0 && grads->r_b0 && grads->r_w2 && grads->r_b2 && grads->d_w0 && grads->d_b0 && grads->d_w2 && grads->d_b2);
  float* dpre_r = scratch + RTE_ROUTER_MAX_R;
  float* dpre_d = dpre_r + (size_t)B * hid;
  float* dlog_r = dpre_d + (size_t)B * hid;
  float* dlog_d = dlog_r + (size_t)B * R;
  const Dw0Jobs jobs = {{{dpre_r, grads->r_w0, grads->r_b0}, {dpre_d, grads->d_w0, grads->d_b0}}};
  rte::launch(router_dw0_kernel, dim3(rte::ceil_div(d, W0_TILE), rte::ceil_div(hid, W0_TILE), 2), NTHR, 0, ST(stream), jobs, fwd->pooled, B, d, hid);
  RTE_LAUNCH_CHECK();
  rte::launch(router_dw2_kernel, rte::ceil_div(R * hid, 32), NTHR, 0, ST(stream), dlog_r, fwd->r_hidden_pre, grads->r_w2, grads->r_b2, B, hid, R);
  RTE_LAUNCH_CHECK();
  rte::launch(router_dw2_kernel, rte::ceil_div(K * hid, 32), NTHR, 0, ST(stream), dlog_d, fwd->d_hidden_pre, grads->d_w2, grads->d_b2, B, hid, K);
  RTE_LAUNCH_CHECK();
  return RTE_OK;
}

// Both halves on one stream.
extern "C" int rte_router_aux_bwd(const rte_router_weights* w, const rte_router_out* fwd, const int32_t* depth_values,
                                  float lambda_load, float lambda_depth, float* aux, const rte_router_grads* grads,
                                  float* dh0, float* scratch, int32_t B, int32_t S, int32_t d, int32_t hid, int32_t R,
                                  int32_t K, rte_stream_t stream) {
  RTE_CHECK_ARG(grads != nullptr);
  const int rc = rte_router_aux_bwd_data(w, fwd, depth_values, lambda_load, lambda_depth, aux, dh0, scratch, nullptr, B, S, d, hid, R, K,
                                         stream);
  if (rc != RTE_OK) return rc;
  return rte_router_aux_bwd_params(fwd, grads, scratch, B, d, hid, R, K, stream);
}
