// Vocabulary shortlist of the `recursive_macro_shortlist` mode (reference output.py:72-136).
//
// rte_shortlist_build: per token, the first K distinct ids of the candidate sequence
//   [target | members of the top clusters | hard negatives | random negatives | filler | target + 0..2K-1 (mod V)]
// in order of first appearance -- the reference's scatter_reduce(amin) + topk(largest=False) over a [tokens, V]
// table, done here by one warp per token walking the sequence segment by segment with a per-warp "seen"
// bitmap in shared memory (no [tokens, V] table).  Candidates are generated from their position, never stored.
// Bit-exact given the same top clusters and random negatives; the target always lands in slot 0.
//
// rte_shortlist_ce: logits over the shortlist (gathered embedding rows . hidden), cross entropy against slot 0,
// and the gradient written as a dense, otherwise-zero [tokens, V] bf16 row so that the backward pass reuses the
// tensor-core GEMMs of the full-vocabulary path.

#include "rte_common.cuh"

namespace {

constexpr int SB_WARPS = 8;

struct ShortlistDims { int V, C, TC, HN, RN, K, mpc; };

// What bounds it: instructions of 32-lane steps, one chain per token (the lists are 1 % of the traffic HBM would carry in
// that time).  The sequence is walked by its segments, because each has a form cheaper than 32 arbitrary candidates:
//   * a cluster's members are distinct (c + j C; at most the last is padding), so a step needs no comparison of lanes;
//   * hard negatives, filler and target + 0..2K-1 are runs of consecutive ids: 32 words of the bitmap, 1024 candidates,
//     are one step -- fresh ids are the run's mask and not the bitmap;
//   * random negatives alone are compared with each other (__match_any_sync).
// 16384 tokens, 64 clusters (top 2), 32 + 32 negatives, K = 128, against 32 arbitrary candidates a step: vocabulary 2048
// (17 steps -> 8) 80.0 -> 13.7 us, K = 256 121.2 -> 13.7; 8192 tokens, vocabulary 8192 63.1 -> 11.8.
struct ShortlistWalk {
  uint32_t* seen;
  int32_t* out;
  int lane, K, n;                                                     // n: distinct ids so far (the first K are listed)

  // 32 candidates, one per lane; `first`: no lower lane holds the same id
  __device__ __forceinline__ void step(int id, bool first) {
    const bool fresh = first && ((seen[id >> 5] >> (id & 31)) & 1u) == 0u;
    const unsigned mask = __ballot_sync(0xffffffffu, fresh);
    if (fresh) {
      const int slot = n + __popc(mask & ((1u << lane) - 1u));
      if (slot < K) out[slot] = id;
      atomicOr(&seen[id >> 5], 1u << (id & 31));
    }
    __syncwarp();
    n += __popc(mask);
  }

  // the run of ids [lo, hi), 0 <= lo, hi <= V
  __device__ __forceinline__ void run(int lo, int hi) {
    if (lo >= hi) return;
    const int last = (hi - 1) >> 5;
    for (int w0 = lo >> 5; w0 <= last; w0 += 32) {
      const int w = w0 + lane;
      uint32_t fresh = 0u;
      if (w <= last) {
        uint32_t mask = 0xffffffffu;
        if (w == (lo >> 5)) mask &= 0xffffffffu << (lo & 31);
        if (w == last) mask &= 0xffffffffu >> (31 - ((hi - 1) & 31));
        const uint32_t have = seen[w];
        fresh = mask & ~have;
        if (fresh) seen[w] = have | mask;
      }
      unsigned words = __ballot_sync(0xffffffffu, fresh != 0u);
      int listed = n;
      while (words != 0u && listed < K) {                             // ascending ids: word after word
        const int src = __ffs(words) - 1;
        words &= words - 1u;
        const uint32_t bits = __shfl_sync(0xffffffffu, fresh, src);
        const int slot = listed + __popc(bits & ((1u << lane) - 1u));
        if (((bits >> lane) & 1u) != 0u && slot < K) out[slot] = ((w0 + src) << 5) + lane;
        listed += __popc(bits);
      }
      n += __reduce_add_sync(0xffffffffu, __popc(fresh));
    }
    __syncwarp();
  }

  // `count` consecutive ids from `start` < V, going on at 0 after V - 1
  __device__ __forceinline__ void ring(int start, long long count, int V) {
    if (count > V) count = V;                                         // (a second lap finds nothing new)
    const int hi = (int)min((long long)V, start + count);
    run(start, hi);
    run(0, (int)(start + count - hi));
  }
};

__global__ void __launch_bounds__(SB_WARPS * 32)
shortlist_build_kernel(const int64_t* __restrict__ targets, const int32_t* __restrict__ top_clusters,
                       const int32_t* __restrict__ random_negs, int32_t* __restrict__ shortlist,
                       int32_t* __restrict__ dup_count, int rows, ShortlistDims D, int* status) {
  rte::after_previous_grid();
  extern __shared__ uint32_t seen_all[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int row = blockIdx.x * SB_WARPS + warp;
  const int words = (D.V + 31) / 32;
  uint32_t* seen = seen_all + (size_t)warp * words;
  if (row >= rows) return;
  for (int i = lane; i < words; i += 32) seen[i] = 0u;
  __syncwarp();
  long long target = targets[row];
  if (target < 0 || target >= D.V) {
    if (status && lane == 0) atomicExch(status, RTE_DEV_INDEX_OUT_OF_RANGE);
    target = 0;
  }
  const int32_t* top = top_clusters + (size_t)row * D.TC;
  const int32_t* rnd = random_negs + (size_t)row * D.RN;
  ShortlistWalk walk{seen, shortlist + (size_t)row * D.K, lane, D.K, 0};
  const bool all = dup_count != nullptr;                              // the duplicates are counted over the whole sequence
  walk.step((int)target, lane == 0);
  for (int t = 0; t < D.TC && (all || walk.n < D.K); ++t) {
    const int c = top[t];                                             // cluster c owns ids c, c + C, c + 2C, ...
    for (int j0 = 0; j0 < D.mpc && (all || walk.n < D.K); j0 += 32) {
      const int j = j0 + lane;
      int id = c + j * D.C;
      bool valid = j < D.mpc;
      if (!valid || id >= D.V) id = 0;                                // (member table padded with id 0)
      if (id < 0) {                                                   // (a negative cluster)
        if (status && valid) atomicExch(status, RTE_DEV_INDEX_OUT_OF_RANGE);
        id = 0;
      }
      const unsigned zeros = __ballot_sync(0xffffffffu, valid && id == 0);
      if (id == 0) valid = valid && (zeros & ((1u << lane) - 1u)) == 0u;
      walk.step(id, valid);
    }
  }
  if (all || walk.n < D.K) walk.ring(0, D.HN, D.V);
  for (int p0 = 0; p0 < D.RN && (all || walk.n < D.K); p0 += 32) {
    const bool valid = p0 + lane < D.RN;
    int id = valid ? rnd[p0 + lane] : 0;
    if (id < 0 || id >= D.V) {
      if (status) atomicExch(status, RTE_DEV_INDEX_OUT_OF_RANGE);
      id = 0;
    }
    const unsigned same = __match_any_sync(0xffffffffu, valid ? id : -1 - lane);
    walk.step(id, valid && (same & ((1u << lane) - 1u)) == 0u);
  }
  if (all || walk.n < D.K) walk.ring(0, D.K, D.V);
  if (all || walk.n < D.K) walk.ring((int)target, 2LL * D.K, D.V);
  if (all && lane == 0) dup_count[row] = 1 + D.TC * D.mpc + D.HN + D.RN + 3 * D.K - walk.n;
}

// one CTA per token: logits over the shortlist, CE vs slot 0, dense gradient row
__global__ void __launch_bounds__(128)
shortlist_ce_kernel(const __nv_bfloat16* __restrict__ hidden, const __nv_bfloat16* __restrict__ W,
                    const int32_t* __restrict__ shortlist, const float* __restrict__ row_weight, int S,
                    float* __restrict__ loss_tok, __nv_bfloat16* __restrict__ logits_out,
                    __nv_bfloat16* __restrict__ dense, int d, int V, int K) {
  rte::after_previous_grid();
  extern __shared__ float sm[];          // hs[d], lg[K]
  __shared__ float red[32];
  float* hs = sm;
  float* lg = sm + d;
  const int row = blockIdx.x;
  for (int c = threadIdx.x; c < d; c += blockDim.x) hs[c] = __bfloat162float(hidden[(size_t)row * d + c]);
  if (dense != nullptr) {
    uint4* dr = reinterpret_cast<uint4*>(dense + (size_t)row * V);
    for (int i = threadIdx.x; i < V / 8; i += blockDim.x) dr[i] = make_uint4(0u, 0u, 0u, 0u);
  }
  __syncthreads();
  const int d8 = d >> 3;
  for (int k = threadIdx.x; k < K; k += blockDim.x) {
    const uint4* wr = reinterpret_cast<const uint4*>(W + (size_t)shortlist[(size_t)row * K + k] * d);
    float acc = 0.f;
#pragma unroll 4
    for (int c = 0; c < d8; ++c) {
      const uint4 pk = wr[c];
      const float2 a = rte::unpack_bf16x2(pk.x), b = rte::unpack_bf16x2(pk.y), e = rte::unpack_bf16x2(pk.z), f = rte::unpack_bf16x2(pk.w);
      const float* h = hs + 8 * c;
      acc += a.x * h[0] + a.y * h[1] + b.x * h[2] + b.y * h[3] + e.x * h[4] + e.y * h[5] + f.x * h[6] + f.y * h[7];
    }
    acc = __bfloat162float(__float2bfloat16_rn(acc));      // the reference's logits are bf16 under autocast
    lg[k] = acc;
    if (logits_out) logits_out[(size_t)row * K + k] = __float2bfloat16_rn(acc);
  }
  __syncthreads();
  float mx = -INFINITY;
  for (int k = threadIdx.x; k < K; k += blockDim.x) mx = fmaxf(mx, lg[k]);
  mx = rte::block_max(mx, red);
  float se = 0.f;
  for (int k = threadIdx.x; k < K; k += blockDim.x) se += __expf(lg[k] - mx);
  se = rte::block_sum(se, red);
  const float lse = mx + __logf(se);
  if (threadIdx.x == 0) loss_tok[row] = lse - lg[0];
  if (dense == nullptr) return;
  const float wgt = row_weight[row / S];
  for (int k = threadIdx.x; k < K; k += blockDim.x) {
    const float g = wgt * (__expf(lg[k] - lse) - (k == 0 ? 1.f : 0.f));
    dense[(size_t)row * V + shortlist[(size_t)row * K + k]] = __float2bfloat16_rn(g);
  }
}

// The same cross entropy when the FULL logits row already exists (one tcgen05 GEMM over the vocabulary costs less than
// gathering K weight rows per token while the vocabulary is small): reads the K shortlisted logits of the row, then
// overwrites the row in place with the dense gradient (zero outside the shortlist).  One CTA per token.
__global__ void __launch_bounds__(128)
shortlist_ce_logits_kernel(__nv_bfloat16* __restrict__ logits, const int32_t* __restrict__ shortlist,
                           const float* __restrict__ row_weight, int S, float* __restrict__ loss_tok, int V, int K) {
  rte::after_previous_grid();
  extern __shared__ float lg[];          // [K]
  __shared__ float red[32];
  const int row = blockIdx.x;
  __nv_bfloat16* lr = logits + (size_t)row * V;
  for (int k = threadIdx.x; k < K; k += blockDim.x) lg[k] = __bfloat162float(lr[shortlist[(size_t)row * K + k]]);
  __syncthreads();                        // every shortlisted logit has been read: the row may be overwritten
  uint4* dr = reinterpret_cast<uint4*>(lr);
  for (int i = threadIdx.x; i < V / 8; i += blockDim.x) dr[i] = make_uint4(0u, 0u, 0u, 0u);
  float mx = -INFINITY;
  for (int k = threadIdx.x; k < K; k += blockDim.x) mx = fmaxf(mx, lg[k]);
  mx = rte::block_max(mx, red);
  float se = 0.f;
  for (int k = threadIdx.x; k < K; k += blockDim.x) se += __expf(lg[k] - mx);
  se = rte::block_sum(se, red);           // (the reductions' barriers also order the zero fill before the scatter)
  const float lse = mx + __logf(se);
  if (threadIdx.x == 0) loss_tok[row] = lse - lg[0];
  const float wgt = row_weight[row / S];
  __syncthreads();
  for (int k = threadIdx.x; k < K; k += blockDim.x) {
    const float g = wgt * (__expf(lg[k] - lse) - (k == 0 ? 1.f : 0.f));
    lr[shortlist[(size_t)row * K + k]] = __float2bfloat16_rn(g);
  }
}

// dense[row, ids[row, k]] = vals[row, k], zero elsewhere (ids distinct within a row)
__global__ void __launch_bounds__(128)
scatter_cols_kernel(const __nv_bfloat16* __restrict__ vals, const int32_t* __restrict__ ids, __nv_bfloat16* __restrict__ dense,
                    int V, int K) {
  rte::after_previous_grid();
  const int row = blockIdx.x;
  uint4* dr = reinterpret_cast<uint4*>(dense + (size_t)row * V);
  for (int i = threadIdx.x; i < V / 8; i += blockDim.x) dr[i] = make_uint4(0u, 0u, 0u, 0u);
  __syncthreads();
  for (int k = threadIdx.x; k < K; k += blockDim.x) {
    const int id = ids[(size_t)row * K + k];
    if (id >= 0 && id < V) dense[(size_t)row * V + id] = vals[(size_t)row * K + k];
  }
}

// out[i] = hash(seed, i) mod vocab  (counter-based, reproducible; used when no host-drawn negatives are supplied)
__global__ void random_tokens_kernel(int32_t* __restrict__ out, long long n, int vocab, const int64_t* __restrict__ seed) {
  rte::after_previous_grid();
  const unsigned long long s = (unsigned long long)(*seed);
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    unsigned long long z = s * 0x9E3779B97F4A7C15ull + (unsigned long long)i + 0x632BE59BD9B4E019ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    z ^= z >> 31;
    out[i] = (int32_t)(z % (unsigned long long)vocab);
  }
}

}  // namespace

#define ST(s) reinterpret_cast<cudaStream_t>(s)

extern "C" int rte_shortlist_build(const int64_t* targets, const int32_t* top_clusters, const int32_t* random_negs,
                                   int32_t* shortlist, int32_t* dup_count, int32_t rows, int32_t V, int32_t C, int32_t TC,
                                   int32_t HN, int32_t RN, int32_t K, int32_t* status, rte_stream_t stream) {
  RTE_CHECK_ARG(targets && top_clusters && shortlist && rows > 0 && V > 0 && C > 0 && TC > 0 && TC <= C && HN >= 0 && RN >= 0 &&
                K > 0 && K <= V && (RN == 0 || random_negs != nullptr));
  ShortlistDims D{V, C, TC, HN, RN, K, (V + C - 1) / C};
  const size_t smem = (size_t)SB_WARPS * ((V + 31) / 32) * sizeof(uint32_t);
  if (smem > 200 * 1024) return RTE_ERR_UNSUPPORTED;
  if (smem > 48 * 1024) {
    static bool set = false;
    if (!set) {
      if (cudaFuncSetAttribute(shortlist_build_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024) != cudaSuccess)
        return RTE_ERR_LAUNCH;
      set = true;
    }
  }
  rte::launch(shortlist_build_kernel, rte::ceil_div(rows, SB_WARPS), SB_WARPS * 32, smem, ST(stream), targets, top_clusters, random_negs ? random_negs : top_clusters, shortlist, dup_count, rows, D, status);
  RTE_LAUNCH_CHECK();
  return RTE_OK;
}

extern "C" int rte_shortlist_ce(const void* hidden, const void* W, const int32_t* shortlist, const float* row_weight, int32_t S,
                                float* loss_tok, void* logits_out, void* dlogits_dense, int32_t rows, int32_t d, int32_t V,
                                int32_t K, rte_stream_t stream) {
  RTE_CHECK_ARG(hidden && W && shortlist && loss_tok && rows > 0 && d > 0 && d % 8 == 0 && V % 8 == 0 && K > 0 && S > 0);
  RTE_CHECK_ARG(dlogits_dense == nullptr || row_weight != nullptr);
  if ((reinterpret_cast<uintptr_t>(W) & 15) || (dlogits_dense && (reinterpret_cast<uintptr_t>(dlogits_dense) & 15))) return RTE_ERR_ALIGNMENT;
  const size_t smem = (size_t)(d + K) * sizeof(float);
  if (smem > 48 * 1024) return RTE_ERR_UNSUPPORTED;
  rte::launch(shortlist_ce_kernel, rows, 128, smem, ST(stream), reinterpret_cast<const __nv_bfloat16*>(hidden),
      reinterpret_cast<const __nv_bfloat16*>(W), shortlist, row_weight, S, loss_tok,
      reinterpret_cast<__nv_bfloat16*>(logits_out), reinterpret_cast<__nv_bfloat16*>(dlogits_dense), d, V, K);
  RTE_LAUNCH_CHECK();
  return RTE_OK;
}

extern "C" int rte_shortlist_ce_from_logits(void* logits_inout, const int32_t* shortlist, const float* row_weight, int32_t S,
                                           float* loss_tok, int32_t rows, int32_t V, int32_t K, rte_stream_t stream) {
  RTE_CHECK_ARG(logits_inout && shortlist && row_weight && loss_tok && rows > 0 && S > 0 && V > 0 && V % 8 == 0 && K > 0);
  if (reinterpret_cast<uintptr_t>(logits_inout) & 15) return RTE_ERR_ALIGNMENT;
  const size_t smem = (size_t)K * sizeof(float);
  if (smem > 48 * 1024) return RTE_ERR_UNSUPPORTED;
  rte::launch(shortlist_ce_logits_kernel, rows, 128, smem, ST(stream), reinterpret_cast<__nv_bfloat16*>(logits_inout), shortlist, row_weight,
                                                             S, loss_tok, V, K);
  RTE_LAUNCH_CHECK();
  return RTE_OK;
}

extern "C" int rte_scatter_cols_bf16(const void* vals, const int32_t* ids, void* dense, int32_t rows, int32_t V, int32_t K,
                                     rte_stream_t stream) {
  RTE_CHECK_ARG(vals && ids && dense && rows > 0 && V > 0 && V % 8 == 0 && K > 0);
  if (reinterpret_cast<uintptr_t>(dense) & 15) return RTE_ERR_ALIGNMENT;
  rte::launch(scatter_cols_kernel, rows, 128, 0, ST(stream), reinterpret_cast<const __nv_bfloat16*>(vals), ids,
                                                    reinterpret_cast<__nv_bfloat16*>(dense), V, K);
  RTE_LAUNCH_CHECK();
  return RTE_OK;
}

extern "C" int rte_random_tokens(int32_t* out, int64_t n, int32_t vocab, const int64_t* seed, rte_stream_t stream) {
  RTE_CHECK_ARG(out && seed && n > 0 && vocab > 0);
  long long g = (n + 255) / 256;
  if (g > 148 * 8) g = 148 * 8;
  rte::launch(random_tokens_kernel, (int)g, 256, 0, ST(stream), out, n, vocab, seed);
  RTE_LAUNCH_CHECK();
  return RTE_OK;
}
