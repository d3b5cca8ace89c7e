// HBM-bound kernels of the training step: embedding gather/scatter, RMSNorm forward/backward
// (with the recurrent core's FiLM), per-token cross entropy with its gradient, split-K reduction,
// fp32->bf16 weight shadows, fused multi-tensor AdamW and the global gradient norm.
// All loads/stores are 16-byte vectors along the contiguous axis; grids are sized from the data
// (one warp or one CTA per row), which at the step's sizes is many waves of 148 SMs.

#include "rte_common.cuh"

namespace {

using rte::block_max;
using rte::block_sum;
using rte::warp_sum;

// ------------------------------------------------------------------ embedding
__global__ void embed_fwd_kernel(const int64_t* __restrict__ tokens, const float* __restrict__ table,
                                 float* __restrict__ out, int n_tokens, int d, int vocab, int* status) {
  rte::after_previous_grid();
  const int d4 = d >> 2;
  const long long total = (long long)n_tokens * d4;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const int t = int(i / d4), c = int(i % d4);
    long long tok = tokens[t];
    if (tok < 0 || tok >= vocab) {
      if (status) atomicExch(status, RTE_DEV_INDEX_OUT_OF_RANGE);
      tok = 0;
    }
    reinterpret_cast<float4*>(out)[i] = reinterpret_cast<const float4*>(table)[tok * d4 + c];
  }
}

// The scatter-add of token-row gradients into the table is ORDER-FREE: every addend is converted to 64-bit fixed
// point (scale 2^40: resolution 9e-13, range +-8.4e6), integer atomics are associative, and the sum is converted
// back once per table element, so repeated runs produce the same bits whatever order the adds land in.
constexpr float EMBED_FX_SCALE = 1099511627776.f;          // 2^40

// (neighbouring lanes add to neighbouring words: an atomic per lane on 8 contiguous bytes each is one 256-byte access)
__global__ void __launch_bounds__(256)
embed_bwd_accum_kernel(const int64_t* __restrict__ tokens, const float* __restrict__ dx, unsigned long long* __restrict__ accum,
                       float* __restrict__ dtable, int n_tokens, int d, int vocab, int* status) {
  rte::after_previous_grid();
  for (int t = blockIdx.x; t < n_tokens; t += gridDim.x) {
    const long long tok = tokens[t];
    if (tok < 0 || tok >= vocab) {
      if (status && threadIdx.x == 0) atomicExch(status, RTE_DEV_INDEX_OUT_OF_RANGE);
      continue;
    }
#pragma unroll 4
    for (int c = threadIdx.x; c < d; c += blockDim.x) {
      const float x = dx[(size_t)t * d + c];
      const size_t at = (size_t)tok * d + c;
      if (!isfinite(x)) dtable[at] = x - x;                          // NaN stays NaN through the final add
      else atomicAdd(accum + at, (unsigned long long)__float2ll_rn(x * EMBED_FX_SCALE));
    }
  }
}

__global__ void embed_bwd_apply_kernel(const unsigned long long* __restrict__ accum, float* __restrict__ dtable, long long n) {
  rte::after_previous_grid();
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const long long q = (long long)accum[i];
    if (q != 0) dtable[i] += __ll2float_rn(q) * (1.f / EMBED_FX_SCALE);
  }
}

// A vocabulary larger than the batch: only the rows of the batch's tokens are cleared before and applied after, instead of
// the whole table (32768 x 1024 with 8192 tokens: 268 MB cleared and read again, 186 -> 114 us).  A token that occurs
// more than once is visited once per occurrence: clearing again is harmless, and the exchange hands the sum to one visitor.
__global__ void __launch_bounds__(256)
embed_bwd_rows_kernel(const int64_t* __restrict__ tokens, unsigned long long* __restrict__ accum, float* __restrict__ dtable, int n_tokens,
                      int d, int vocab, int apply) {
  rte::after_previous_grid();
  for (int t = blockIdx.x; t < n_tokens; t += gridDim.x) {
    const long long tok = tokens[t];
    if (tok < 0 || tok >= vocab) continue;
    const size_t row = (size_t)tok * d;
    if (apply) {
#pragma unroll 4
      for (int c = threadIdx.x; c < d; c += blockDim.x) {
        const long long q = (long long)atomicExch(accum + row + c, 0ull);
        if (q != 0) dtable[row + c] += __ll2float_rn(q) * (1.f / EMBED_FX_SCALE);
      }
    } else {
      if (d % 2 == 0)
        for (int c = threadIdx.x; c < d / 2; c += blockDim.x) reinterpret_cast<ulonglong2*>(accum + row)[c] = make_ulonglong2(0ull, 0ull);
      else
        for (int c = threadIdx.x; c < d; c += blockDim.x) accum[row + c] = 0ull;
    }
  }
}

// The same sums with the tokens grouped by id beforehand (the ids are known when a step begins, so a caller groups them beside
// its forward pass): a warp adds up to 16 rows of one id and 128 columns in registers, all its loads in flight at once, and writes
// the table once; the pieces of an id with more meet in 64-bit accumulators, and the last one to arrive converts.  Every sum is the integer it was,
// so the bits are the same.  Bound by the read of dx: one atomic per element and a pass over all accumulators are gone (us,
// accumulate and apply -> grouped: 8192 x 512 of 2048 ids 24.5 -> 10.9, 16384 x 512 45 -> 24, 8192 x 1024 of 32768 ids 80 -> 30; 512 x 128
// 5.3 -> 6.3, hence the line at 2^18 elements; the grouping itself takes 4..19 us beside other work).
constexpr int EG_THREADS = 1024, EG_PIECE = 16, EG_COLS = 128;
constexpr int EG_MAX_VOCAB = 48 * 1024;                      // one counter per id in shared memory, 192 KB (56 K would fit; the configurations here stop at 32768)
struct EmbedGroups {
  int* head;                 // [0]: pieces
  int4* piece;               // id, first entry of `order`, entries | pieces of the id << 8, row of `sums` (< 0: the id's only piece)
  int* order;                // token positions grouped by id
  int* ticket;               // per row of `sums` and column block: pieces that have arrived
  unsigned long long* sums;
};
inline size_t embed_groups_layout(void* scratch, int n, int d, EmbedGroups* g, size_t* clear_from = nullptr) {
  auto up = [](size_t x) { return (x + 15) & ~(size_t)15; };
  const size_t multi = (size_t)n / EG_PIECE, blocks = rte::ceil_div(d, EG_COLS);
  const size_t piece = 16, order = piece + 16 * (size_t)n, ticket = up(order + 4 * (size_t)n), sums = up(ticket + 4 * multi * blocks);
  char* at = reinterpret_cast<char*>(scratch);
  if (g) *g = {reinterpret_cast<int*>(at), reinterpret_cast<int4*>(at + piece), reinterpret_cast<int*>(at + order), reinterpret_cast<int*>(at + ticket),
               reinterpret_cast<unsigned long long*>(at + sums)};
  if (clear_from) *clear_from = ticket;
  return sums + 8 * multi * d;
}
inline bool embed_groups_fit(const void* scratch, const void* dtable, int n, int d, int vocab) {
  return d % 4 == 0 && (long long)n * d >= (1 << 18) && vocab <= EG_MAX_VOCAB && n < (1 << 23) && ((reinterpret_cast<uintptr_t>(scratch) | reinterpret_cast<uintptr_t>(dtable)) & 15) == 0 &&
         embed_groups_layout(nullptr, n, d, nullptr) <= (size_t)vocab * d * 8;
}

// One CTA: counts per id in shared memory, their running sums (ids dealt to the threads round robin), pieces, order.
__global__ void __launch_bounds__(EG_THREADS)
embed_group_kernel(const int64_t* __restrict__ tokens, int n, int vocab, EmbedGroups G, int* status) {
  rte::after_previous_grid();
  extern __shared__ int eg_count[];
  __shared__ int wsum[3][32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int v = tid; v < vocab; v += EG_THREADS) eg_count[v] = 0;
  __syncthreads();
#pragma unroll 4
  for (int t = tid; t < n; t += EG_THREADS) {
    const long long tok = tokens[t];
    if (tok >= 0 && tok < vocab) atomicAdd(&eg_count[tok], 1);
    else if (status) atomicExch(status, RTE_DEV_INDEX_OUT_OF_RANGE);
  }
  __syncthreads();
  int a[3] = {0, 0, 0};                                      // tokens, pieces, ids of several pieces
  for (int v = tid; v < vocab; v += EG_THREADS) {
    const int k = eg_count[v];
    a[0] += k; a[1] += (k + EG_PIECE - 1) / EG_PIECE; a[2] += k > EG_PIECE;
  }
  int upto[3];
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    int x = a[q];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const int y = __shfl_up_sync(0xffffffffu, x, o); if (lane >= o) x += y; }
    upto[q] = x;
    if (lane == 31) wsum[q][warp] = x;
  }
  __syncthreads();
  if (warp < 3) {
    int x = wsum[warp][lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const int y = __shfl_up_sync(0xffffffffu, x, o); if (lane >= o) x += y; }
    wsum[warp][lane] = x;
  }
  __syncthreads();
  int at[3];
#pragma unroll
  for (int q = 0; q < 3; ++q) at[q] = upto[q] - a[q] + (warp > 0 ? wsum[q][warp - 1] : 0);
  if (tid == 0) G.head[0] = wsum[1][31];
  for (int v = tid; v < vocab; v += EG_THREADS) {
    const int k = eg_count[v], pieces = (k + EG_PIECE - 1) / EG_PIECE;
    for (int q = 0; q < pieces; ++q)
      G.piece[at[1] + q] = make_int4(v, at[0] + q * EG_PIECE, min(EG_PIECE, k - q * EG_PIECE) | pieces << 8, pieces > 1 ? at[2] : -1);
    eg_count[v] = at[0];
    at[0] += k; at[1] += pieces; at[2] += pieces > 1;
  }
  __syncthreads();
#pragma unroll 4
  for (int t = tid; t < n; t += EG_THREADS) {
    const long long tok = tokens[t];
    if (tok >= 0 && tok < vocab) G.order[atomicAdd(&eg_count[tok], 1)] = t;
  }
}

__global__ void __launch_bounds__(256)
embed_sum_kernel(const float* __restrict__ dx, float* dtable, EmbedGroups G, int d) {
  rte::after_previous_grid();
  const int lane = threadIdx.x & 31, blocks = (d + EG_COLS - 1) / EG_COLS, d4 = d >> 2;
  const long long jobs = (long long)G.head[0] * blocks;
  for (long long j = blockIdx.x * 8LL + (threadIdx.x >> 5); j < jobs; j += gridDim.x * 8LL) {
    const int4 piece = G.piece[j / blocks];
    const int cb = int(j % blocks), c = cb * (EG_COLS / 4) + lane, count = piece.z & 255, pieces = piece.z >> 8;      // c: in float4
    const int mine = lane < count ? G.order[piece.y + lane] : 0;
    const bool in = c < d4;
    float4 x[EG_PIECE];
#pragma unroll
    for (int i = 0; i < EG_PIECE; ++i) {
      const int row = __shfl_sync(0xffffffffu, mine, i);
      x[i] = in && i < count ? reinterpret_cast<const float4*>(dx)[(size_t)row * d4 + c] : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    long long acc[4] = {0, 0, 0, 0};
    unsigned bad = 0;
#pragma unroll
    for (int i = 0; i < EG_PIECE; ++i) {
      if (i >= count) break;
      const float v[4] = {x[i].x, x[i].y, x[i].z, x[i].w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        if (isfinite(v[e])) acc[e] += __float2ll_rn(v[e] * EMBED_FX_SCALE);
        else bad |= 1u << e;
      }
    }
    float* out = dtable + (size_t)piece.x * d + 4 * c;
    const unsigned long long* sums = nullptr;
    if (piece.w >= 0) {                                       // one of several pieces
      unsigned long long* into = G.sums + (size_t)piece.w * d + 4 * c;
      if (in) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          if (bad >> e & 1) out[e] = __int_as_float(0x7fffffff);      // NaN stays NaN through the final add
          atomicAdd(into + e, (unsigned long long)acc[e]);
        }
      }
      __threadfence();
      __syncwarp();
      int arrived = 0;
      if (lane == 0) arrived = atomicAdd(&G.ticket[piece.w * blocks + cb], 1);
      if (__shfl_sync(0xffffffffu, arrived, 0) != pieces - 1) continue;
      __threadfence();
      sums = into;
      bad = 0;
    }
    if (!in) continue;
    float4 o = __ldcg(reinterpret_cast<float4*>(out));
    float* ov = &o.x;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const long long v = sums ? (long long)__ldcg(sums + e) : acc[e];
      if (bad >> e & 1) ov[e] = __int_as_float(0x7fffffff);
      else if (v != 0) ov[e] += __ll2float_rn(v) * (1.f / EMBED_FX_SCALE);
    }
    *reinterpret_cast<float4*>(out) = o;
  }
}

// ------------------------------------------------------------------ RMSNorm
// One warp per row, row held in registers (d <= 32 * 4 * RN_MAX_V4).
constexpr int RN_MAX_V4 = 16;   // d up to 2048

template <int NV>
__global__ void __launch_bounds__(256)
rmsnorm_fwd_kernel(const float* __restrict__ x, const float* __restrict__ w, const float* __restrict__ fg,
                   const float* __restrict__ fb, __nv_bfloat16* __restrict__ y16, float* __restrict__ y32,
                   float* __restrict__ rstd, int rows, int d, float eps) {
  rte::after_previous_grid();
  const int lane = threadIdx.x & 31;
  const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= rows) return;
  const int d4 = d >> 2;
  const float4* xr = reinterpret_cast<const float4*>(x + (size_t)row * d);
  float4 v[NV];
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = lane + 32 * i;
    if (c < d4) {
      v[i] = xr[c];
      ss += v[i].x * v[i].x + v[i].y * v[i].y + v[i].z * v[i].z + v[i].w * v[i].w;
    }
  }
  ss = warp_sum(ss);
  const float r = rsqrtf(ss / (float)d + eps);
  if (lane == 0 && rstd) rstd[row] = r;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = lane + 32 * i;
    if (c < d4) {
      float4 o = make_float4(v[i].x * r, v[i].y * r, v[i].z * r, v[i].w * r);
      if (w) {
        const float4 ww = reinterpret_cast<const float4*>(w)[c];
        o.x *= ww.x; o.y *= ww.y; o.z *= ww.z; o.w *= ww.w;
      }
      if (fg) {
        const float4 g = reinterpret_cast<const float4*>(fg)[c], b = reinterpret_cast<const float4*>(fb)[c];
        o.x = o.x * (1.f + g.x) + b.x; o.y = o.y * (1.f + g.y) + b.y;
        o.z = o.z * (1.f + g.z) + b.z; o.w = o.w * (1.f + g.w) + b.w;
      }
      if (y32) reinterpret_cast<float4*>(y32 + (size_t)row * d)[c] = o;
      if (y16) {
        uint2 pk = make_uint2(rte::pack_bf16x2(o.x, o.y), rte::pack_bf16x2(o.z, o.w));
        reinterpret_cast<uint2*>(y16 + (size_t)row * d)[c] = pk;
      }
    }
  }
}

// Residual update(s) fused in front of the norm (one warp per row):
//   x1 = (active == NULL || active[row / S]) ? base + *scale * branch : passthrough      -> x1_out (optional)
//   x  = add2 ? x1 + *scale2 * add2 : x1                                                  -> x_out
//   y  = rmsnorm(x) * w [* (1 + fg) + fb]
template <int NV>
__global__ void __launch_bounds__(256)
residual_rmsnorm_fwd_kernel(const float* __restrict__ base, const float* __restrict__ branch, const float* __restrict__ scale,
                            const int32_t* __restrict__ active, const float* __restrict__ passthrough, int S,
                            const float* __restrict__ add2, const float* __restrict__ scale2, float* __restrict__ x1_out,
                            float* __restrict__ x_out, const float* __restrict__ w, const float* __restrict__ fg,
                            const float* __restrict__ fb, __nv_bfloat16* __restrict__ y16, float* __restrict__ rstd, int rows, int d,
                            float eps, int branch_splits, long long branch_stride, float* __restrict__ branch_out) {
  rte::after_previous_grid();
  // branch_splits > 1: `branch` holds that many split-K partials of the branch, branch_stride floats apart; they are
  // summed here in split order (what rte_reduce_splits would have produced) and the sum is kept in branch_out.
  const int lane = threadIdx.x & 31;
  const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= rows) return;
  const int d4 = d >> 2;
  const size_t off = (size_t)row * d;
  const bool on = active == nullptr || active[row / S] != 0;
  const float s1 = *scale, s2 = add2 ? *scale2 : 0.f;
  float4 v[NV];
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = lane + 32 * i;
    if (c < d4) {
      float4 x;
      float4 b = make_float4(0.f, 0.f, 0.f, 0.f);
      if (on || branch_out) {
        b = reinterpret_cast<const float4*>(branch + off)[c];
        for (int s = 1; s < branch_splits; ++s) {
          const float4 t = reinterpret_cast<const float4*>(branch + (size_t)s * branch_stride + off)[c];
          b.x += t.x; b.y += t.y; b.z += t.z; b.w += t.w;
        }
        if (branch_out) reinterpret_cast<float4*>(branch_out + off)[c] = b;
      }
      if (on) {
        const float4 a = reinterpret_cast<const float4*>(base + off)[c];
        x = make_float4(a.x + s1 * b.x, a.y + s1 * b.y, a.z + s1 * b.z, a.w + s1 * b.w);
      } else {
        x = reinterpret_cast<const float4*>(passthrough + off)[c];
      }
      if (x1_out) reinterpret_cast<float4*>(x1_out + off)[c] = x;
      if (add2) {
        const float4 e = reinterpret_cast<const float4*>(add2 + off)[c];
        x.x += s2 * e.x; x.y += s2 * e.y; x.z += s2 * e.z; x.w += s2 * e.w;
      }
      reinterpret_cast<float4*>(x_out + off)[c] = x;
      v[i] = x;
      ss += x.x * x.x + x.y * x.y + x.z * x.z + x.w * x.w;
    }
  }
  ss = warp_sum(ss);
  const float r = rsqrtf(ss / (float)d + eps);
  if (lane == 0 && rstd) rstd[row] = r;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = lane + 32 * i;
    if (c < d4) {
      float4 o = make_float4(v[i].x * r, v[i].y * r, v[i].z * r, v[i].w * r);
      if (w) {
        const float4 ww = reinterpret_cast<const float4*>(w)[c];
        o.x *= ww.x; o.y *= ww.y; o.z *= ww.z; o.w *= ww.w;
      }
      if (fg) {
        const float4 g = reinterpret_cast<const float4*>(fg)[c], b = reinterpret_cast<const float4*>(fb)[c];
        o.x = o.x * (1.f + g.x) + b.x; o.y = o.y * (1.f + g.y) + b.y;
        o.z = o.z * (1.f + g.z) + b.z; o.w = o.w * (1.f + g.w) + b.w;
      }
      uint2 pk = make_uint2(rte::pack_bf16x2(o.x, o.y), rte::pack_bf16x2(o.z, o.w));
      reinterpret_cast<uint2*>(y16 + off)[c] = pk;
    }
  }
}

// RMSNorm(+FiLM) backward: dx = r * (g - xh * mean(g * xh)) + dres with xh = x * r, g = dy * (1 + gamma) * w, plus per-CTA
// column sums for the weight and FiLM gradients, written to row blockIdx.x of the partial buffers (deterministic, no
// atomics).  dy_splits > 1: dy32 holds that many split-K partials of dy, dy_stride floats apart, summed in split order.
//
// A thread owns four columns: blockDim.x threads span a row, blockDim.y rows run side by side, ROWS rows of each are in
// flight.  The column sums are then 4 (FiLM: 12) registers per thread whatever the width, so the loads of all ROWS rows
// (x, dy, residual gradient) fit ahead of the first use; a warp per row held d / 32 columns per lane and, beyond d = 512,
// one row at a time (with the column sums, us: 8192 x 1024 80 -> 34, 16384 x 512 42 -> 34, 8192 x 512 15.8 -> 13.9, 64 x
// 512 5.3 -> 3.4).  One barrier per ROWS rows joins the row sums of the warps.  FILM = false drops the FiLM accumulators.
constexpr int RN_ROWS = 4;
template <int N>
__device__ __forceinline__ void warp_sums(float (&v)[N]) {
#pragma unroll
  for (int u = 0; u < N; ++u) v[u] = warp_sum(v[u]);
}
// four sums at once: the first two exchanges halve the values a lane carries (6 shuffles + 4 to spread, not 20)
template <>
__device__ __forceinline__ void warp_sums<4>(float (&v)[4]) {
  const int lane = threadIdx.x & 31;
  const float a0 = lane & 16 ? v[2] : v[0], a1 = lane & 16 ? v[3] : v[1], b0 = lane & 16 ? v[0] : v[2], b1 = lane & 16 ? v[1] : v[3];
  const float c0 = a0 + __shfl_xor_sync(0xffffffffu, b0, 16), c1 = a1 + __shfl_xor_sync(0xffffffffu, b1, 16);
  float t = (lane & 8 ? c1 : c0) + __shfl_xor_sync(0xffffffffu, lane & 8 ? c0 : c1, 8);
  t += __shfl_xor_sync(0xffffffffu, t, 4);
  t += __shfl_xor_sync(0xffffffffu, t, 2);
  t += __shfl_xor_sync(0xffffffffu, t, 1);
#pragma unroll
  for (int u = 0; u < 4; ++u) v[u] = __shfl_sync(0xffffffffu, t, 8 * u);
}

template <int ROWS, bool FILM, int BLOCK>
__global__ void __launch_bounds__(BLOCK, ROWS == 1 ? 2 : 768 / BLOCK)
rmsnorm_bwd_kernel(const float* __restrict__ x, const float* __restrict__ w, const float* __restrict__ fg,
                   const float* __restrict__ rstd, const __nv_bfloat16* __restrict__ dy16,
                   const float* __restrict__ dy32, const float* __restrict__ dres, float* __restrict__ dx32,
                   __nv_bfloat16* __restrict__ dx16, float* __restrict__ dw_part, float* __restrict__ dg_part,
                   float* __restrict__ db_part, int rows, int d, int dy_splits, long long dy_stride) {
  rte::after_previous_grid();
  __shared__ float red[2][ROWS][BLOCK / 32];
  __shared__ float4 comb[BLOCK];
  const int c = threadIdx.x, d4 = d >> 2, nw = blockDim.x >> 5, gy = blockDim.y, warp0 = threadIdx.y * nw;
  const bool on = c < d4;
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  const float4 ww = !on ? zero : w ? reinterpret_cast<const float4*>(w)[c] : make_float4(1.f, 1.f, 1.f, 1.f);
  float4 f1 = make_float4(1.f, 1.f, 1.f, 1.f);
  if (FILM && fg && on) {
    const float4 t = reinterpret_cast<const float4*>(fg)[c];
    f1 = make_float4(1.f + t.x, 1.f + t.y, 1.f + t.z, 1.f + t.w);
  }
  const float4 wf = make_float4(ww.x * f1.x, ww.y * f1.y, ww.z * f1.z, ww.w * f1.w);
  float4 aw = zero, ag = zero, ab = zero;
  const int step = gridDim.x * gy;
  int buf = 0;
  for (int row0 = blockIdx.x * gy; row0 < rows; row0 += step * ROWS, buf ^= 1) {      // (the same trips for all rows of a CTA)
    float4 xh[ROWS], g[ROWS], res[ROWS];
    float r[ROWS], dot[ROWS];
#pragma unroll
    for (int u = 0; u < ROWS; ++u) {
      const int row = row0 + threadIdx.y + u * step;
      xh[u] = g[u] = res[u] = zero;
      r[u] = 0.f;
      if (row < rows && on) {
        const size_t at = (size_t)row * d4 + c;
        r[u] = rstd[row];
        xh[u] = reinterpret_cast<const float4*>(x)[at];
        if (dy16) {
          const uint2 pk = reinterpret_cast<const uint2*>(dy16)[at];
          const float2 a = rte::unpack_bf16x2(pk.x), b = rte::unpack_bf16x2(pk.y);
          g[u] = make_float4(a.x, a.y, b.x, b.y);
        } else {
          g[u] = reinterpret_cast<const float4*>(dy32)[at];
        }
        if (dres) res[u] = reinterpret_cast<const float4*>(dres)[at];
      }
    }
    if (dy_splits > 1) {
#pragma unroll
      for (int u = 0; u < ROWS; ++u) {
        const int row = row0 + threadIdx.y + u * step;
        if (row < rows && on)
          for (int s = 1; s < dy_splits; ++s) {
            const float4 t = reinterpret_cast<const float4*>(dy32 + (size_t)s * dy_stride)[(size_t)row * d4 + c];
            g[u].x += t.x; g[u].y += t.y; g[u].z += t.z; g[u].w += t.w;
          }
      }
    }
#pragma unroll
    for (int u = 0; u < ROWS; ++u) {
      float4& h = xh[u];
      const float4 dv = g[u];
      h.x *= r[u]; h.y *= r[u]; h.z *= r[u]; h.w *= r[u];
      const float4 p = make_float4(dv.x * h.x, dv.y * h.y, dv.z * h.z, dv.w * h.w);
      aw.x += p.x * f1.x; aw.y += p.y * f1.y; aw.z += p.z * f1.z; aw.w += p.w * f1.w;
      if constexpr (FILM) {
        ag.x += p.x * ww.x; ag.y += p.y * ww.y; ag.z += p.z * ww.z; ag.w += p.w * ww.w;
        ab.x += dv.x; ab.y += dv.y; ab.z += dv.z; ab.w += dv.w;
      }
      dot[u] = p.x * wf.x + p.y * wf.y + p.z * wf.z + p.w * wf.w;
      g[u] = make_float4(dv.x * wf.x, dv.y * wf.y, dv.z * wf.z, dv.w * wf.w);
    }
    warp_sums(dot);
    if (nw > 1) {
      if ((c & 31) == 0) {
#pragma unroll
        for (int u = 0; u < ROWS; ++u) red[buf][u][warp0 + (c >> 5)] = dot[u];
      }
      __syncthreads();                                                 // (two buffers: the next trip's writes need no second barrier)
#pragma unroll
      for (int u = 0; u < ROWS; ++u) {
        dot[u] = 0.f;
        for (int k = 0; k < nw; ++k) dot[u] += red[buf][u][warp0 + k];
      }
    }
#pragma unroll
    for (int u = 0; u < ROWS; ++u) {
      const int row = row0 + threadIdx.y + u * step;
      if (row < rows && on) {
        const size_t at = (size_t)row * d4 + c;
        const float mean = dot[u] / (float)d, q = r[u];
        const float4 o = make_float4(q * (g[u].x - xh[u].x * mean) + res[u].x, q * (g[u].y - xh[u].y * mean) + res[u].y,
                                     q * (g[u].z - xh[u].z * mean) + res[u].z, q * (g[u].w - xh[u].w * mean) + res[u].w);
        if (dx32) reinterpret_cast<float4*>(dx32)[at] = o;
        if (dx16) reinterpret_cast<uint2*>(dx16)[at] = make_uint2(rte::pack_bf16x2(o.x, o.y), rte::pack_bf16x2(o.z, o.w));
      }
    }
  }
  // column sums of the CTA's rows
  auto write = [&](float* part, const float4& sum) {
    float4 t = sum;
    if (gy > 1) {
      __syncthreads();
      comb[threadIdx.y * blockDim.x + c] = sum;
      __syncthreads();
      if (threadIdx.y == 0)
        for (int k = 1; k < gy; ++k) {
          const float4 v = comb[k * blockDim.x + c];
          t.x += v.x; t.y += v.y; t.z += v.z; t.w += v.w;
        }
    }
    if (threadIdx.y == 0 && on) reinterpret_cast<float4*>(part + (size_t)blockIdx.x * d)[c] = t;
  };
  if (dw_part) write(dw_part, aw);
  if (FILM && dg_part) {
    write(dg_part, ag);
    write(db_part, ab);
  }
}

// 32 columns x 32 row-groups per CTA: thirty-two partial sums per column, combined through shared memory in a
// fixed order (deterministic).
__global__ void __launch_bounds__(1024)
colsum_kernel(const float* __restrict__ part, int n_rows, int d, float* __restrict__ out, int accumulate) {
  rte::after_previous_grid();
  __shared__ float sm[32][33];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int c = blockIdx.x * 32 + tx;
  float s = 0.f;
  if (c < d) {
#pragma unroll 4
    for (int r = ty; r < n_rows; r += 32) s += part[(size_t)r * d + c];
  }
  sm[ty][tx] = s;
  __syncthreads();
  if (ty == 0 && c < d) {
    float t = 0.f;
#pragma unroll
    for (int k = 0; k < 32; ++k) t += sm[k][tx];
    out[c] = accumulate ? out[c] + t : t;
  }
}

// Up to three column sums of equally shaped partial buffers in one launch (blockIdx.y selects the buffer).
struct ColsumJob { const float* part; float* out; int accumulate; };
struct ColsumJobs { ColsumJob j[3]; };

__global__ void __launch_bounds__(1024)
colsum3_kernel(ColsumJobs jobs, int n_rows, int d) {
  rte::after_previous_grid();
  __shared__ float sm[32][33];
  const ColsumJob job = jobs.j[blockIdx.y];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int c = blockIdx.x * 32 + tx;
  float s = 0.f;
  if (c < d) {
#pragma unroll 4
    for (int r = ty; r < n_rows; r += 32) s += job.part[(size_t)r * d + c];
  }
  sm[ty][tx] = s;
  __syncthreads();
  if (ty == 0 && c < d) {
    float t = 0.f;
#pragma unroll
    for (int k = 0; k < 32; ++k) t += sm[k][tx];
    job.out[c] = job.accumulate ? job.out[c] + t : t;
  }
}

// Every sum of partials that the backward pass of the recurrent core leaves, in ONE launch: per pass and norm the FiLM
// vectors' columns, per norm the weight's columns over all passes (last pass first, as the passes accumulate), and the
// scalar parameters' segments.  What bounds it is the launch: 16 x 3 buffers of 128 rows at most.  Launch by launch (two per
// pass, three for the scalars) on the weight-gradient stream each waited 20..140 us for a place beside the hot pass, and
// the products behind them ran after everything else.  256 threads (8 x four columns, 32 rows): the same 32 partial sums
// per column in the same order as colsum_kernel, in a block that finds room beside the persistent products.
// Audited steps, us: 16384 x 512, 8 passes 2719 -> 2674; 8192 x 512, 4 passes 1415 -> 1404.
__global__ void __launch_bounds__(256)
core_sums_kernel(const __grid_constant__ rte_core_sums J, int T, int pr, int n_rows, int d, int P) {
  rte::after_previous_grid();
  __shared__ float sm[2][32][33];
  const int cols = rte::ceil_div(d, 32), tid = threadIdx.x;
  int job = blockIdx.x / cols;
  const int c = (blockIdx.x - job * cols) * 32 + (tid & 7) * 4, ty = tid >> 3;
  const int column_jobs = 2 + 4 * T;
  if (job < column_jobs) {
    // job 0, 1: weight of norm 2, 1; then (pass, norm, gamma or beta)
    const int norm = job < 2 ? job : ((job - 2) >> 1) & 1, buf = job < 2 ? 0 : 1 + ((job - 2) & 1);
    const int t_hi = job < 2 ? T - 1 : (job - 2) >> 2, t_lo = job < 2 ? 0 : t_hi;
    float* out = job < 2 ? J.dw[norm] : (buf == 1 ? J.dgamma[norm] : J.dbeta[norm]) + (size_t)t_hi * d;
    const int oc = (blockIdx.x - job * cols) * 32 + tid;
    float total = 0.f;
    for (int t = t_hi; t >= t_lo; --t) {
      const float* part = J.partials + ((size_t)(t * 2 + norm) * 3 + buf) * pr * d;
      float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
      if (c < d) {
#pragma unroll 4
        for (int r = ty; r < n_rows; r += 32) {
          const float4 v = *reinterpret_cast<const float4*>(part + (size_t)r * d + c);
          s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
        }
      }
      float* row = sm[t & 1][ty] + (tid & 7) * 4;
      row[0] = s.x; row[1] = s.y; row[2] = s.z; row[3] = s.w;
      __syncthreads();                      // (two buffers: warp 0 sums one while the others fill the next)
      if (tid < 32) {
        float v = 0.f;
#pragma unroll
        for (int k = 0; k < 32; ++k) v += sm[t & 1][k][tid];
        total = t == t_hi ? v : total + v;
      }
    }
    if (tid < 32 && oc < d) out[oc] = total;
    return;
  }
  // a segment of P partials per pass and scale, all T of them for alpha: threads 0..127, as segment_sum_kernel adds them
  const int seg = blockIdx.x - column_jobs * cols;
  const float* in = seg < T ? J.part_mlp + (size_t)seg * P : seg < 2 * T ? J.part_attn + (size_t)(seg - T) * P : J.part_alpha;
  const int len = seg < 2 * T ? P : T * P;
  float s = 0.f;
  if (tid < 128)
    for (int i = tid; i < len; i += 128) s += in[i];
  s = block_sum(s, &sm[0][0][0]);
  if (tid == 0) *(seg < T ? J.d_mlp_scale + seg : seg < 2 * T ? J.d_attn_scale + (seg - T) : J.d_alpha) = s;
}

// ------------------------------------------------------------------ cross entropy
// Rows are handled in 16-byte groups of W logits.  `off` is the number of elements between the 16-byte boundary at or
// before the row and the row itself: group g holds logits g * W - off ..., its slots outside [0, V) read as -inf and are
// never touched in memory, so rows of any width and alignment take the same kernels.  EVEN: every row starts on a
// boundary and has whole groups only (without the checks 8192 x 2048 takes 20.5 us instead of 26.6).
template <typename T>
struct CeVec;
template <>
struct CeVec<__nv_bfloat16> {
  static constexpr int W = 8;
  static __device__ __forceinline__ void unpack(const uint4& r, float (&v)[8]) {
    const float2 a = rte::unpack_bf16x2(r.x), b = rte::unpack_bf16x2(r.y), c = rte::unpack_bf16x2(r.z), d = rte::unpack_bf16x2(r.w);
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y; v[4] = c.x; v[5] = c.y; v[6] = d.x; v[7] = d.y;
  }
  static __device__ __forceinline__ uint4 pack(const float (&v)[8]) {
    return make_uint4(rte::pack_bf16x2(v[0], v[1]), rte::pack_bf16x2(v[2], v[3]), rte::pack_bf16x2(v[4], v[5]), rte::pack_bf16x2(v[6], v[7]));
  }
};
template <>
struct CeVec<float> {
  static constexpr int W = 4;
  static __device__ __forceinline__ void unpack(const uint4& r, float (&v)[4]) {
    v[0] = __uint_as_float(r.x); v[1] = __uint_as_float(r.y); v[2] = __uint_as_float(r.z); v[3] = __uint_as_float(r.w);
  }
  static __device__ __forceinline__ uint4 pack(const float (&v)[4]) {
    return make_uint4(__float_as_uint(v[0]), __float_as_uint(v[1]), __float_as_uint(v[2]), __float_as_uint(v[3]));
  }
};
__device__ __forceinline__ float to_f(float x) { return x; }
__device__ __forceinline__ float to_f(__nv_bfloat16 x) { return __bfloat162float(x); }

template <bool EVEN, typename T>
__device__ __forceinline__ uint4 ce_load(const T* row, int at, int V) {          // at = g * W - off
  constexpr int W = CeVec<T>::W;
  if (EVEN || (at >= 0 && at + W <= V)) return *reinterpret_cast<const uint4*>(row + at);
  float v[W];
#pragma unroll
  for (int j = 0; j < W; ++j) v[j] = at + j >= 0 && at + j < V ? to_f(row[at + j]) : -INFINITY;
  return CeVec<T>::pack(v);
}
template <bool EVEN, typename T>
__device__ __forceinline__ void ce_store(T* row, int at, int V, bool whole, const float (&v)[CeVec<T>::W]) {    // whole: a group of `row` is 16-byte aligned
  constexpr int W = CeVec<T>::W;
  if (EVEN || (whole && at >= 0 && at + W <= V)) { *reinterpret_cast<uint4*>(row + at) = CeVec<T>::pack(v); return; }
#pragma unroll
  for (int j = 0; j < W; ++j)
    if (at + j >= 0 && at + j < V) row[at + j] = (T)v[j];
}
template <typename T>
__device__ __forceinline__ int ce_offset(const T* row) { return int(reinterpret_cast<uintptr_t>(row) & 15) / (int)sizeof(T); }

__device__ __forceinline__ int ce_target(const int64_t* targets, int row, int V, int* status) {
  const long long t = targets[row];
  if (t >= 0 && t < V) return (int)t;
  if (status && threadIdx.x == 0) atomicExch(status, RTE_DEV_INDEX_OUT_OF_RANGE);
  return 0;
}
// Exponentials are taken relative to a maximum that may be -inf (columns masked out, or nothing but NaN, which a maximum
// passes over): relative to zero then, so that exp(-inf) is 0 and a NaN stays one and reaches the sum.
__device__ __forceinline__ float ce_reference(float m) { return m == -INFINITY ? 0.f : m; }

// (maximum, sum of exponentials) of the row from every warp's; a warp without a finite column brings 0, or NaN
template <int WARPS>
__device__ __forceinline__ float ce_lse(const float (&red_m)[WARPS], const float (&red_s)[WARPS]) {
  float mx = red_m[0], se = 0.f;
#pragma unroll
  for (int w = 1; w < WARPS; ++w) mx = fmaxf(mx, red_m[w]);
#pragma unroll
  for (int w = 0; w < WARPS; ++w) se += red_m[w] == -INFINITY ? red_s[w] : red_s[w] * __expf(red_m[w] - mx);
  return mx + __logf(se);
}

// One CTA of THREADS per row, the row in registers (at most NV groups per thread): logits are read once, maximum and sum
// of exponentials meet in one block reduction, the gradient is written from the exponentials.  Bound by HBM and, close
// behind, by the instructions per element, so the CTA is as small as the row allows (many rows in flight per SM) and only
// the group that holds the target looks for it.  With gradient, against a kernel that read a row three times with 256
// threads: bf16 8192 x 2048 38.9 -> 20.5 us (67 MB), 8192 x 8192 84.9 -> 61.4 us.
template <typename T, int THREADS, int NV, bool EVEN>
__global__ void __launch_bounds__(THREADS)
ce_row_kernel(const T* __restrict__ logits, int ldl, const int64_t* __restrict__ targets, const float* __restrict__ row_weight, int S,
              float* __restrict__ loss_tok, T* __restrict__ dlogits, int V, int* status) {
  rte::after_previous_grid();
  constexpr int W = CeVec<T>::W, WARPS = THREADS / 32;
  __shared__ float red_m[WARPS], red_s[WARPS], target_logit;
  const int row = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const T* lr = logits + (size_t)row * ldl;
  const int off = EVEN ? 0 : ce_offset(lr), groups = (V + off + W - 1) / W;
  float e[NV][W];
  {
    uint4 raw[NV];
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int g = int(threadIdx.x) + i * THREADS;
      if (g < groups) raw[i] = ce_load<EVEN>(lr, g * W - off, V);
    }
#pragma unroll
    for (int i = 0; i < NV; ++i)
      if (int(threadIdx.x) + i * THREADS < groups) CeVec<T>::unpack(raw[i], e[i]);
  }
  const int tgt = ce_target(targets, row, V, status), tg = (tgt + off) / W, tj = (tgt + off) % W;
  float m = -INFINITY;
#pragma unroll
  for (int i = 0; i < NV; ++i)
    if (int(threadIdx.x) + i * THREADS < groups) {
#pragma unroll
      for (int j = 0; j < W; ++j) m = fmaxf(m, e[i][j]);
    }
  m = rte::warp_max(m);
  const float ref = ce_reference(m);
  float s = 0.f;
#pragma unroll
  for (int i = 0; i < NV; ++i)
    if (int(threadIdx.x) + i * THREADS < groups) {
      if (int(threadIdx.x) + i * THREADS == tg) {
#pragma unroll
        for (int j = 0; j < W; ++j)
          if (j == tj) target_logit = e[i][j];
      }
#pragma unroll
      for (int j = 0; j < W; ++j) s += e[i][j] = __expf(e[i][j] - ref);
    }
  s = warp_sum(s);
  if (lane == 0) { red_m[warp] = m; red_s[warp] = s; }
  __syncthreads();
  const float lse = ce_lse(red_m, red_s);
  if (threadIdx.x == 0) loss_tok[row] = lse - target_logit;
  if (dlogits == nullptr) return;
  // (a warp without a finite column: zeros, whatever lse is, unless the whole row has none)
  const float wgt = row_weight[row / S], scale = m == -INFINITY ? wgt + (lse - lse) : wgt * __expf(m - lse);
  T* dr = dlogits + (size_t)row * ldl;
  const bool whole = EVEN || ce_offset(dr) == off;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int g = int(threadIdx.x) + i * THREADS;
    if (g < groups) {
#pragma unroll
      for (int j = 0; j < W; ++j) e[i][j] *= scale;
      if (g == tg) {
#pragma unroll
        for (int j = 0; j < W; ++j)
          if (j == tj) e[i][j] -= wgt;
      }
      ce_store<EVEN>(dr, g * W - off, V, whole, e[i]);
    }
  }
}

template <bool EVEN, int U, typename T>
__device__ __forceinline__ void ce_stream_gradient(const T* lr, T* dr, int off, int groups, int V, int tg, int tj, float wgt, float lse) {
  constexpr int W = CeVec<T>::W;
  const bool whole = EVEN || ce_offset(dr) == off;
  for (int g0 = threadIdx.x; g0 < groups; g0 += 256 * U) {
    uint4 raw[U];
#pragma unroll
    for (int i = 0; i < U; ++i)
      if (g0 + 256 * i < groups) raw[i] = ce_load<EVEN>(lr, (g0 + 256 * i) * W - off, V);
#pragma unroll
    for (int i = 0; i < U; ++i) {
      const int g = g0 + 256 * i;
      if (g < groups) {
        float v[W];
        CeVec<T>::unpack(raw[i], v);
#pragma unroll
        for (int j = 0; j < W; ++j) v[j] = wgt * __expf(v[j] - lse);
        if (g == tg) {
#pragma unroll
          for (int j = 0; j < W; ++j)
            if (j == tj) v[j] -= wgt;
        }
        ce_store<EVEN>(dr, g * W - off, V, whole, v);
      }
    }
  }
}

// Rows of more than 16 KB: a CTA that holds such a row leaves its SM waiting between its phases (8192 x 32768 bf16 took
// 369 us in registers of 1024 threads).  Five CTAs per SM stream their rows instead: one pass from HBM with a running
// maximum and sum, and, for the gradient, a second one that finds the row in L2 (148 x 5 rows of 64 KB are 48 MB).
// 8192 x 32768 with gradient: 299 -> 231 us (1.07 GB), loss alone 150 -> 133 us.
template <typename T, bool EVEN>
__global__ void __launch_bounds__(256, 5)
ce_stream_kernel(const T* __restrict__ logits, int ldl, const int64_t* __restrict__ targets, const float* __restrict__ row_weight, int S,
                 float* __restrict__ loss_tok, T* dlogits, int V, int* status, float* __restrict__ lse_out) {
  rte::after_previous_grid();
  constexpr int W = CeVec<T>::W, U = 4;
  __shared__ float red_m[8], red_s[8];
  const int row = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const T* lr = logits + (size_t)row * ldl;
  const int off = EVEN ? 0 : ce_offset(lr), groups = (V + off + W - 1) / W;
  const int tgt = ce_target(targets, row, V, status), tg = (tgt + off) / W, tj = (tgt + off) % W;
  const float tl = threadIdx.x == 0 ? to_f(lr[tgt]) : 0.f;           // (before the gradient may overwrite the row)
  float m = -INFINITY, s = 0.f;
  for (int g0 = threadIdx.x; g0 < groups; g0 += 256 * U) {
    uint4 raw[U];
#pragma unroll
    for (int i = 0; i < U; ++i)
      if (g0 + 256 * i < groups) raw[i] = ce_load<EVEN>(lr, (g0 + 256 * i) * W - off, V);
#pragma unroll
    for (int i = 0; i < U; ++i)
      if (g0 + 256 * i < groups) {
        float v[W];
        CeVec<T>::unpack(raw[i], v);
        float gm = v[0];
#pragma unroll
        for (int j = 1; j < W; ++j) gm = fmaxf(gm, v[j]);
        if (gm > m) { s *= __expf(m - gm); m = gm; }
        const float ref = ce_reference(m);
#pragma unroll
        for (int j = 0; j < W; ++j) s += __expf(v[j] - ref);
      }
  }
  const float wm = rte::warp_max(m);
  s = warp_sum(m == -INFINITY ? s : s * __expf(m - wm));
  if (lane == 0) { red_m[warp] = wm; red_s[warp] = s; }
  __syncthreads();
  const float lse = ce_lse(red_m, red_s);
  if (threadIdx.x == 0) {
    loss_tok[row] = lse - tl;
    if (lse_out != nullptr) lse_out[row] = lse;
  }
  if (dlogits == nullptr) return;
  ce_stream_gradient<EVEN, U>(lr, dlogits + (size_t)row * ldl, off, groups, V, tg, tj, row_weight[row / S], lse);
}

// The gradient of such rows from the sums that the loss's launch kept: one pass instead of two.  Bound by HBM: 4107 x 8192
// fp32 (269 MB) 51.7 -> 43.1 us, 8192 x 32768 bf16 (1.07 GB) 222.6 -> 164.7 (6.5 TB/s), 2000 x 9000 bf16 21.8 -> 10.8.
template <typename T, bool EVEN>
__global__ void __launch_bounds__(256, 6)
ce_gradient_kernel(const T* __restrict__ logits, int ldl, const int64_t* __restrict__ targets, const float* __restrict__ row_weight, int S,
                   const float* __restrict__ lse, T* dlogits, int V, int* status) {
  rte::after_previous_grid();
  constexpr int W = CeVec<T>::W;
  const int row = blockIdx.x;
  const T* lr = logits + (size_t)row * ldl;
  const int off = EVEN ? 0 : ce_offset(lr), groups = (V + off + W - 1) / W;
  const int tgt = ce_target(targets, row, V, status);
  ce_stream_gradient<EVEN, 4>(lr, dlogits + (size_t)row * ldl, off, groups, V, (tgt + off) / W, (tgt + off) % W, row_weight[row / S], lse[row]);
}

template <bool EVEN, typename T>
int ce_groups(int V) { return EVEN ? V / CeVec<T>::W : (V + 2 * (CeVec<T>::W - 1)) / CeVec<T>::W; }
constexpr int CE_ROW_GROUPS = 1024;            // groups of a row that ce_row_kernel still holds

template <bool EVEN, typename T>
int launch_ce_rows(const T* logits, int ldl, const int64_t* targets, const float* row_weight, int S, float* loss_tok, T* dlogits, int rows, int V,
                   int* status, cudaStream_t st) {
  const int groups = ce_groups<EVEN, T>(V);
#define RTE_CE(THREADS, NV) \
  rte::launch(ce_row_kernel<T, THREADS, NV, EVEN>, rows, THREADS, 0, st, logits, ldl, targets, row_weight, S, loss_tok, dlogits, V, status)
  if (groups <= 128) RTE_CE(64, 2);
  else if (groups <= 256) RTE_CE(64, 4);
  else if (groups <= 512) RTE_CE(128, 4);
  else if (groups <= CE_ROW_GROUPS) RTE_CE(256, 4);
  else rte::launch(ce_stream_kernel<T, EVEN>, rows, 256, 0, st, logits, ldl, targets, row_weight, S, loss_tok, dlogits, V, status, nullptr);
#undef RTE_CE
  RTE_LAUNCH_CHECK();
  return RTE_OK;
}
template <typename T>
int launch_ce(const T* logits, int ldl, const int64_t* targets, const float* row_weight, int S, float* loss_tok, T* dlogits, int rows, int V,
              int* status, cudaStream_t st) {
  constexpr int W = CeVec<T>::W;
  const bool even = V % W == 0 && ldl % W == 0 && ((reinterpret_cast<uintptr_t>(logits) | reinterpret_cast<uintptr_t>(dlogits)) & 15) == 0;
  return (even ? launch_ce_rows<true, T> : launch_ce_rows<false, T>)(logits, ldl, targets, row_weight, S, loss_tok, dlogits, rows, V, status, st);
}

// Loss with the rows' sums kept (dlogits null), or the gradient from kept sums: long rows only, shorter ones are read once as they are.
template <bool EVEN, typename T>
int launch_ce_lse(const T* logits, int ldl, const int64_t* targets, const float* row_weight, int S, float* loss_tok, float* lse, T* dlogits,
                  int rows, int V, int* status, cudaStream_t st) {
  if (ce_groups<EVEN, T>(V) <= CE_ROW_GROUPS) return RTE_ERR_UNSUPPORTED;
  if (dlogits == nullptr)
    rte::launch(ce_stream_kernel<T, EVEN>, rows, 256, 0, st, logits, ldl, targets, row_weight, S, loss_tok, dlogits, V, status, lse);
  else
    rte::launch(ce_gradient_kernel<T, EVEN>, rows, 256, 0, st, logits, ldl, targets, row_weight, S, (const float*)lse, dlogits, V, status);
  RTE_LAUNCH_CHECK();
  return RTE_OK;
}
template <typename T>
int launch_ce_lse(const void* logits, int ldl, const int64_t* targets, const float* row_weight, int S, float* loss_tok, float* lse, void* dlogits,
                  int rows, int V, int* status, cudaStream_t st) {
  constexpr int W = CeVec<T>::W;
  const bool even = V % W == 0 && ldl % W == 0 && ((reinterpret_cast<uintptr_t>(logits) | reinterpret_cast<uintptr_t>(dlogits)) & 15) == 0;
  return (even ? launch_ce_lse<true, T> : launch_ce_lse<false, T>)(reinterpret_cast<const T*>(logits), ldl, targets, row_weight, S, loss_tok, lse,
                                                                     reinterpret_cast<T*>(dlogits), rows, V, status, st);
}

__global__ void segment_sum_kernel(const float* __restrict__ in, float* __restrict__ out, int n_seg, int seg_len) {
  rte::after_previous_grid();
  __shared__ float red[32];
  const int seg = blockIdx.x;
  if (seg >= n_seg) return;
  float s = 0.f;
  for (int i = threadIdx.x; i < seg_len; i += blockDim.x) s += in[(size_t)seg * seg_len + i];
  s = block_sum(s, red);
  if (threadIdx.x == 0) out[seg] = s;
}

// ------------------------------------------------------------------ small vector kernels
// (up to eight partials of an element are requested together)
__global__ void __launch_bounds__(256)
reduce_splits_kernel(const float* __restrict__ ws, int splits, long long stride, long long n4, float* __restrict__ out, int accumulate) {
  rte::after_previous_grid();
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n4; i += (long long)gridDim.x * blockDim.x) {
    float4 acc = accumulate ? reinterpret_cast<float4*>(out)[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    for (int s0 = 0; s0 < splits; s0 += 8) {
      float4 t[8];
#pragma unroll
      for (int s = 0; s < 8; ++s)
        if (s0 + s < splits) t[s] = reinterpret_cast<const float4*>(ws + (size_t)(s0 + s) * stride)[i];
#pragma unroll
      for (int s = 0; s < 8; ++s)
        if (s0 + s < splits) { acc.x += t[s].x; acc.y += t[s].y; acc.z += t[s].z; acc.w += t[s].w; }
    }
    reinterpret_cast<float4*>(out)[i] = acc;
  }
}
__global__ void reduce_splits_tail_kernel(const float* __restrict__ ws, int splits, long long stride, long long start,
                                          long long n, float* __restrict__ out, int accumulate) {
  rte::after_previous_grid();
  const long long i = start + blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  float acc = accumulate ? out[i] : 0.f;
  for (int s = 0; s < splits; ++s) acc += ws[(size_t)s * stride + i];
  out[i] = acc;
}

__global__ void cast_kernel(const float* __restrict__ src, __nv_bfloat16* __restrict__ dst, long long n) {
  rte::after_previous_grid();
  const long long n4 = n >> 2;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n4; i += (long long)gridDim.x * blockDim.x) {
    const float4 t = reinterpret_cast<const float4*>(src)[i];
    reinterpret_cast<uint2*>(dst)[i] = make_uint2(rte::pack_bf16x2(t.x, t.y), rte::pack_bf16x2(t.z, t.w));
  }
  for (long long i = n4 * 4 + blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    dst[i] = __float2bfloat16_rn(src[i]);
}
__global__ void fill_kernel(float* __restrict__ dst, float value, long long n) {
  rte::after_previous_grid();
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) dst[i] = value;
}
// dst += src, one or two ranges (blockIdx.y).  Bound by HBM (12 bytes an element), so 16 bytes a load where the addresses
// allow: 17.8 M elements 46.9 -> 33.6 us (6.4 TB/s), 4 M 13.3 -> 9.2, 1 M 3.6 -> 2.6.
struct AddJob { float* dst; const float* src; long long n; };
struct AddJobs { AddJob j[2]; };
__global__ void __launch_bounds__(256)
add_kernel(const __grid_constant__ AddJobs jobs) {
  rte::after_previous_grid();
  const AddJob job = jobs.j[blockIdx.y];
  const long long first = blockIdx.x * (long long)blockDim.x + threadIdx.x, stride = (long long)gridDim.x * blockDim.x;
  const long long n4 = ((reinterpret_cast<uintptr_t>(job.dst) | reinterpret_cast<uintptr_t>(job.src)) & 15) == 0 ? job.n >> 2 : 0;
  for (long long i = first; i < n4; i += stride) {
    const float4 b = reinterpret_cast<const float4*>(job.src)[i];
    float4 a = reinterpret_cast<float4*>(job.dst)[i];
    a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w;
    reinterpret_cast<float4*>(job.dst)[i] = a;
  }
  for (long long i = 4 * n4 + first; i < job.n; i += stride) job.dst[i] += job.src[i];
}
__global__ void add_guarded_kernel(float* __restrict__ dst, const float* __restrict__ src, long long n, const int32_t* __restrict__ skip) {
  rte::after_previous_grid();
  if (*skip != 0) return;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) dst[i] += src[i];
}
__global__ void axpy_rows_kernel(float* __restrict__ dst, const float* __restrict__ vec, float alpha, int rows, int seg, int d) {
  rte::after_previous_grid();
  const long long total = (long long)rows * d;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const int r = int(i / d), c = int(i % d);
    dst[i] += alpha * vec[(size_t)(r / seg) * d + c];
  }
}

// ------------------------------------------------------------------ AdamW
// `skip` (optional device flag): non-zero turns the whole launch into a no-op -- parameters, moments, shadows and step
// counters stay as they are (the reference drops a step whose loss is not finite, training.py:448-452).
// Bound by HBM (30 bytes per parameter with a shadow): 67 M parameters 434 -> 327 us.
// `metric_partial` (optional, [chunks][2]): per-chunk sums of (grad_scale * g)^2 and of p^2 BEFORE the update, the
// raw material of the per-group gradient / parameter norms (training.py:386-443); reduced by adamw_finish_kernel.
__global__ void __launch_bounds__(256)
adamw_kernel(const rte_adamw_tensor* __restrict__ table, const int32_t* __restrict__ chunk_tensor,
             const int32_t* __restrict__ chunk_index, const float* __restrict__ lr_table,
             const int32_t* __restrict__ step_count, float beta1, float beta2, float eps, float wd,
             const float* __restrict__ grad_scale, const int32_t* __restrict__ skip, float* __restrict__ metric_partial,
             const int32_t* __restrict__ absent_flag, const uint8_t* __restrict__ absent_mask) {
  rte::after_previous_grid();
  __shared__ float red[32];
  const int ti = chunk_tensor[blockIdx.x];
  // dropped step, or a tensor that received no gradient in this step (torch.optim.AdamW skips `grad is None`: no decay,
  // no moment update, no step count)
  if ((skip != nullptr && *skip != 0) || (absent_flag != nullptr && *absent_flag != 0 && absent_mask[ti] != 0)) {
    if (metric_partial != nullptr && threadIdx.x == 0) { metric_partial[2 * blockIdx.x] = 0.f; metric_partial[2 * blockIdx.x + 1] = 0.f; }
    return;
  }
  const rte_adamw_tensor t = table[ti];
  const long long base = (long long)chunk_index[blockIdx.x] * RTE_ADAMW_CHUNK;
  // what the step count decides, once per CTA (two powf per thread were a fifth of the kernel's instructions)
  __shared__ float sstep[3];
  if (threadIdx.x == 0) {
    const float lr = lr_table[t.lr_group], step = (float)(step_count[t.step_slot] + 1);      // incremented by adamw_finish_kernel afterwards
    sstep[0] = lr / (1.f - powf(beta1, step));
    sstep[1] = rsqrtf(1.f - powf(beta2, step));
    sstep[2] = 1.f - lr * wd;
  }
  const float gs = grad_scale ? *grad_scale : 1.f;
  __nv_bfloat16* shadow = reinterpret_cast<__nv_bfloat16*>(t.bf16_shadow);
  float gsq = 0.f, psq = 0.f;
  auto update = [&](float g, float& p, float& m, float& v, float step_size, float inv_sqrt_bc2, float decay) {
    g *= gs;
    gsq += g * g; psq += p * p;
    m = beta1 * m + (1.f - beta1) * g;
    v = beta2 * v + (1.f - beta2) * g * g;
    p = p * decay - step_size * m / (sqrtf(v) * inv_sqrt_bc2 + eps);
  };
  if (base + RTE_ADAMW_CHUNK <= t.n &&
      ((reinterpret_cast<uintptr_t>(t.p) | reinterpret_cast<uintptr_t>(t.g) | reinterpret_cast<uintptr_t>(t.m) | reinterpret_cast<uintptr_t>(t.v) |
        (reinterpret_cast<uintptr_t>(t.bf16_shadow) << 1)) & 15) == 0) {
    // whole chunk: 16 elements per thread as float4, two per trip so that eight 16-byte loads are in flight
    constexpr int U = 2;
    bool ready = false;
    float step_size = 0.f, inv_sqrt_bc2 = 0.f, decay = 0.f;
#pragma unroll
    for (int j0 = 0; j0 < RTE_ADAMW_CHUNK / 1024; j0 += U) {
      float4 g[U], p[U], m[U], v[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const long long i4 = base / 4 + (j0 + u) * 256 + threadIdx.x;
        g[u] = reinterpret_cast<const float4*>(t.g)[i4];
        p[u] = reinterpret_cast<const float4*>(t.p)[i4];
        m[u] = reinterpret_cast<const float4*>(t.m)[i4];
        v[u] = reinterpret_cast<const float4*>(t.v)[i4];
      }
      if (!ready) {
        __syncthreads();
        step_size = sstep[0]; inv_sqrt_bc2 = sstep[1]; decay = sstep[2];
        ready = true;
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const long long i4 = base / 4 + (j0 + u) * 256 + threadIdx.x;
        update(g[u].x, p[u].x, m[u].x, v[u].x, step_size, inv_sqrt_bc2, decay);
        update(g[u].y, p[u].y, m[u].y, v[u].y, step_size, inv_sqrt_bc2, decay);
        update(g[u].z, p[u].z, m[u].z, v[u].z, step_size, inv_sqrt_bc2, decay);
        update(g[u].w, p[u].w, m[u].w, v[u].w, step_size, inv_sqrt_bc2, decay);
        reinterpret_cast<float4*>(t.p)[i4] = p[u];
        reinterpret_cast<float4*>(t.m)[i4] = m[u];
        reinterpret_cast<float4*>(t.v)[i4] = v[u];
        if (shadow) reinterpret_cast<uint2*>(shadow)[i4] = make_uint2(rte::pack_bf16x2(p[u].x, p[u].y), rte::pack_bf16x2(p[u].z, p[u].w));
      }
    }
  } else {
    __syncthreads();
    const float step_size = sstep[0], inv_sqrt_bc2 = sstep[1], decay = sstep[2];
#pragma unroll 4
    for (int j = threadIdx.x; j < RTE_ADAMW_CHUNK; j += blockDim.x) {
      const long long i = base + j;
      if (i >= t.n) break;
      float p = t.p[i], m = t.m[i], v = t.v[i];
      update(t.g[i], p, m, v, step_size, inv_sqrt_bc2, decay);
      t.p[i] = p; t.m[i] = m; t.v[i] = v;
      if (shadow) shadow[i] = __float2bfloat16_rn(p);
    }
  }
  if (metric_partial != nullptr) {       // uniform branch: every thread of the block takes part in the reductions
    gsq = block_sum(gsq, red);
    psq = block_sum(psq, red);
    if (threadIdx.x == 0) { metric_partial[2 * blockIdx.x] = gsq; metric_partial[2 * blockIdx.x + 1] = psq; }
  }
}
// What follows the update, in one launch (the step ends with it).  Blocks 0 .. n_groups - 1: out[2*g] = sum of grad^2, out[2*g+1] = sum
// of param^2 over the chunks of the tensors of metric group g (fixed summation order: reproducible); eight chunks a thread
// are requested together, a chain of loads per chunk took twice the time.  The blocks behind them: the step counts, unless
// the step is dropped.  Update of 17.8 M parameters with metrics (two launches behind it before) 92.3 -> 87.5 us.
__global__ void __launch_bounds__(256)
adamw_finish_kernel(const int32_t* __restrict__ chunk_tensor, const int32_t* __restrict__ metric_group, long long total_chunks,
                    const float* __restrict__ partial, float* __restrict__ out, int n_groups, const rte_adamw_tensor* __restrict__ table,
                    int n_tensors, int32_t* step_count, const int32_t* __restrict__ skip, const int32_t* __restrict__ absent_flag,
                    const uint8_t* __restrict__ absent_mask) {
  rte::after_previous_grid();
  if ((int)blockIdx.x >= n_groups) {
    if (skip != nullptr && *skip != 0) return;
    const int i = ((int)blockIdx.x - n_groups) * blockDim.x + threadIdx.x;
    if (i < n_tensors && !(absent_flag != nullptr && *absent_flag != 0 && absent_mask[i] != 0)) step_count[table[i].step_slot] += 1;
    return;
  }
  __shared__ float red[32];
  constexpr int U = 8;
  float a = 0.f, b = 0.f;
  for (long long c0 = threadIdx.x; c0 < total_chunks; c0 += U * blockDim.x) {
    int group[U];
    float2 v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const long long c = c0 + (long long)u * blockDim.x;
      group[u] = -1;
      v[u] = make_float2(0.f, 0.f);
      if (c < total_chunks) {
        group[u] = chunk_tensor[c];
        v[u] = make_float2(partial[2 * c], partial[2 * c + 1]);
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (group[u] >= 0) group[u] = metric_group[group[u]];
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (group[u] == (int)blockIdx.x) { a += v[u].x; b += v[u].y; }
  }
  a = block_sum(a, red);
  b = block_sum(b, red);
  if (threadIdx.x == 0) { out[2 * blockIdx.x] = a; out[2 * blockIdx.x + 1] = b; }
}
// skip = 1 (and flag_out = 1.0) when any of the listed values is not finite, else 0.
__global__ void __launch_bounds__(256)
nonfinite_guard_kernel(const float* __restrict__ a, int na, const float* __restrict__ b, int nb, const float* __restrict__ c, int nc,
                       int32_t* skip, float* flag_out) {
  rte::after_previous_grid();
  __shared__ int bad;
  if (threadIdx.x == 0) bad = 0;
  __syncthreads();
  int mine = 0;
  for (int i = threadIdx.x; i < na; i += blockDim.x) mine |= !isfinite(a[i]);
  for (int i = threadIdx.x; i < nb; i += blockDim.x) mine |= !isfinite(b[i]);
  for (int i = threadIdx.x; i < nc; i += blockDim.x) mine |= !isfinite(c[i]);
  if (mine) atomicOr(&bad, 1);
  __syncthreads();
  if (threadIdx.x == 0) { *skip = bad; if (flag_out) *flag_out = bad ? 1.f : 0.f; }
}

__global__ void __launch_bounds__(256)
gradnorm_partial_kernel(const rte_adamw_tensor* __restrict__ table, const int32_t* __restrict__ chunk_tensor,
                        const int32_t* __restrict__ chunk_index, float* __restrict__ partial) {
  rte::after_previous_grid();
  __shared__ float red[32];
  const rte_adamw_tensor t = table[chunk_tensor[blockIdx.x]];
  const long long base = (long long)chunk_index[blockIdx.x] * RTE_ADAMW_CHUNK;
  float s = 0.f;
  for (int j = threadIdx.x; j < RTE_ADAMW_CHUNK; j += blockDim.x) {
    const long long i = base + j;
    if (i < t.n) { const float g = t.g[i]; s += g * g; }
  }
  s = block_sum(s, red);
  if (threadIdx.x == 0) partial[blockIdx.x] = s;
}
__global__ void gradnorm_final_kernel(const float* __restrict__ partial, long long n, float* sumsq, float max_norm, float* clip_coef) {
  rte::after_previous_grid();
  __shared__ float red[32];
  float s = 0.f;
  for (long long i = threadIdx.x; i < n; i += blockDim.x) s += partial[i];
  s = block_sum(s, red);
  if (threadIdx.x == 0) {
    sumsq[0] = s;
    if (clip_coef) clip_coef[0] = max_norm > 0.f ? fminf(1.f, max_norm / (sqrtf(s) + 1e-6f)) : 1.f;
  }
}

// ------------------------------------------------------------------ built-in scratch for the no-allocation gradient norm
// Lives in the library image: every GPU that loads the library carries these 256 KB until the process ends.
// In HOST code the name `g_gradnorm_scratch` is only a stand-in for the symbol, not a device address, so the
// launcher below asks the runtime for the real address (once per device) and hands that to the kernels.
constexpr long long GRADNORM_STATIC_MAX_CHUNKS = 65536;   // 65536 chunks x 4096 elements = 268M gradient elements
static __device__ __align__(256) float g_gradnorm_scratch[GRADNORM_STATIC_MAX_CHUNKS];

constexpr int MAX_DEVICES = 64;
float* g_gradnorm_scratch_addr[MAX_DEVICES] = {nullptr};

// Returns the device address of the scratch array on the CURRENT device (looked up on first use).  The cache is
// written without a lock: two host threads that make the first call on a device at the same time both look the
// address up and store the same value, which is harmless.
int gradnorm_scratch_for_current_device(float** out) {
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= MAX_DEVICES) return RTE_ERR_NO_DEVICE;
  if (g_gradnorm_scratch_addr[dev] == nullptr) {
    float* ptr = nullptr;
    if (cudaGetSymbolAddress(reinterpret_cast<void**>(&ptr), g_gradnorm_scratch) != cudaSuccess || ptr == nullptr)
      return RTE_ERR_LAUNCH;
    g_gradnorm_scratch_addr[dev] = ptr;
  }
  *out = g_gradnorm_scratch_addr[dev];
  return RTE_OK;
}

// ------------------------------------------------------------------ top-k, ties to the lowest index
// One warp per row.  k rounds of a warp arg-max over (value desc, index asc); a selected entry is
// masked by remembering the previous winner's (value, index) and only admitting strictly "later"
// candidates in that order, so no scratch copy of the row is needed.
__global__ void __launch_bounds__(256)
topk_kernel(const float* __restrict__ scores, int ld, int rows, int n, int k, int32_t* __restrict__ idx, float* __restrict__ vals) {
  rte::after_previous_grid();
  const int lane = threadIdx.x & 31;
  const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= rows) return;
  const float* sr = scores + (size_t)row * ld;
  float pv = INFINITY; int pi = -1;      // previous winner; first round admits everything
  for (int r = 0; r < k; ++r) {
    float bv = -INFINITY; int bi = 0x7fffffff;
    for (int c = lane; c < n; c += 32) {
      const float v = sr[c];
      const bool after_prev = (v < pv) || (v == pv && c > pi);
      const bool better = (v > bv) || (v == bv && c < bi);
      if (after_prev && better) { bv = v; bi = c; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (ov > bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; }
    }
    if (lane == 0) {
      if (idx) idx[(size_t)row * k + r] = bi;
      if (vals) vals[(size_t)row * k + r] = bv;
    }
    pv = bv; pi = bi;
  }
}

inline int grid_for(long long n, int block, int cap = 148 * 16) {
  long long g = (n + block - 1) / block;
  if (g > cap) g = cap;
  if (g < 1) g = 1;
  return (int)g;
}

// SwiGLU as a pass of its own over a saved (up | gate) buffer: 8 hidden units per thread, 16-byte accesses.
__device__ __forceinline__ void unpack8(const uint4& t, float (&v)[8]) {
  const float2 a = rte::unpack_bf16x2(t.x), b = rte::unpack_bf16x2(t.y), c = rte::unpack_bf16x2(t.z), d = rte::unpack_bf16x2(t.w);
  v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y; v[4] = c.x; v[5] = c.y; v[6] = d.x; v[7] = d.y;
}
__device__ __forceinline__ uint4 pack8(const float (&v)[8]) {
  return make_uint4(rte::pack_bf16x2(v[0], v[1]), rte::pack_bf16x2(v[2], v[3]), rte::pack_bf16x2(v[4], v[5]), rte::pack_bf16x2(v[6], v[7]));
}
__global__ void __launch_bounds__(256)
swiglu_fwd_kernel(const __nv_bfloat16* __restrict__ ug, __nv_bfloat16* __restrict__ z, long long rows, int F) {
  rte::after_previous_grid();
  const int f8 = F >> 3;
  const long long total = rows * f8;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const long long r = i / f8;
    const int j = int(i % f8) << 3;
    float up[8], g[8], o[8];
    unpack8(*reinterpret_cast<const uint4*>(ug + r * 2 * F + j), up);
    unpack8(*reinterpret_cast<const uint4*>(ug + r * 2 * F + F + j), g);
#pragma unroll
    for (int k = 0; k < 8; ++k) o[k] = up[k] * rte::silu_f(g[k]);
    *reinterpret_cast<uint4*>(z + r * F + j) = pack8(o);
  }
}
__global__ void __launch_bounds__(256)
swiglu_bwd_kernel(const __nv_bfloat16* __restrict__ ug, const __nv_bfloat16* __restrict__ dz, __nv_bfloat16* __restrict__ dug,
                  long long rows, int F) {
  rte::after_previous_grid();
  const int f8 = F >> 3;
  const long long total = rows * f8;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const long long r = i / f8;
    const int j = int(i % f8) << 3;
    float up[8], g[8], d[8], du[8], dg[8];
    unpack8(*reinterpret_cast<const uint4*>(ug + r * 2 * F + j), up);
    unpack8(*reinterpret_cast<const uint4*>(ug + r * 2 * F + F + j), g);
    unpack8(*reinterpret_cast<const uint4*>(dz + r * F + j), d);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const float sg = rte::sigmoid_f(g[k]);
      du[k] = d[k] * g[k] * sg;
      dg[k] = d[k] * up[k] * sg * (1.f + g[k] * (1.f - sg));
    }
    *reinterpret_cast<uint4*>(dug + r * 2 * F + j) = pack8(du);
    *reinterpret_cast<uint4*>(dug + r * 2 * F + F + j) = pack8(dg);
  }
}

}  // namespace

#define ST(s) reinterpret_cast<cudaStream_t>(s)

extern "C" const char* rte_backend_name(void) { return "cuda_sm100a_ext"; }

extern "C" const char* rte_status_string(int code) {
  switch (code) {
    case RTE_OK: return "ok";
    case RTE_ERR_BAD_ARG: return "bad argument";
    case RTE_ERR_ALIGNMENT: return "pointer or stride not 16-byte aligned";
    case RTE_ERR_TENSOR_MAP: return "tensor map creation failed";
    case RTE_ERR_LAUNCH: return "kernel launch failed";
    case RTE_ERR_UNSUPPORTED: return "unsupported size";
    case RTE_ERR_NO_DEVICE: return "no CUDA device";
    case RTE_ERR_SCRATCH_CAPACITY: return "size exceeds the capacity of the library's built-in scratch array";
    case RTE_DEV_WAIT_TIMEOUT_PRODUCER: return "device: TMA producer wait ran out";
    case RTE_DEV_WAIT_TIMEOUT_MMA: return "device: MMA issuer wait ran out";
    case RTE_DEV_WAIT_TIMEOUT_EPILOGUE: return "device: epilogue wait ran out";
    case RTE_DEV_WAIT_TIMEOUT_PEER: return "device: wait for a data-parallel peer ran out";
    case RTE_DEV_INDEX_OUT_OF_RANGE: return "device: index out of range";
    case RTE_DEV_CAPACITY_OVERFLOW: return "device: packed rows exceed the caller's capacity";
    default: return "unknown";
  }
}

extern "C" int rte_embed_fwd(const int64_t* tokens, const float* table, float* out, int32_t n_tokens, int32_t d,
                             int32_t vocab, int32_t* status, rte_stream_t stream) {
  RTE_CHECK_ARG(tokens && table && out && n_tokens > 0 && d > 0 && d % 4 == 0);
  rte::launch(embed_fwd_kernel, grid_for((long long)n_tokens * (d / 4), 256), 256, 0, ST(stream), tokens, table, out, n_tokens, d, vocab, status);
  RTE_LAUNCH_CHECK();
  return RTE_OK;
}
extern "C" int rte_embed_bwd(const int64_t* tokens, const float* dx, float* dtable, int64_t* accum, int32_t n_tokens,
                             int32_t d, int32_t vocab, int32_t* status, rte_stream_t stream) {
  RTE_CHECK_ARG(tokens && dx && dtable && accum && n_tokens > 0 && d > 0 && vocab > 0);
  const long long n = (long long)vocab * d;
  auto* fx = reinterpret_cast<unsigned long long*>(accum);
  const bool rows = vocab >= 2 * (long long)n_tokens && (reinterpret_cast<uintptr_t>(accum) & 15) == 0;      // (two visits per token against two passes over the table)
  const int grid = n_tokens < 148 * 16 ? n_tokens : 148 * 16;
  if (rows) rte::launch(embed_bwd_rows_kernel, grid, 256, 0, ST(stream), tokens, fx, dtable, n_tokens, d, vocab, 0);
  else if (cudaMemsetAsync(accum, 0, (size_t)n * sizeof(int64_t), ST(stream)) != cudaSuccess) return RTE_ERR_LAUNCH;
  rte::launch(embed_bwd_accum_kernel, grid, 128, 0, ST(stream), tokens, dx, fx, dtable, n_tokens, d, vocab, status);
  if (rows) rte::launch(embed_bwd_rows_kernel, grid, 256, 0, ST(stream), tokens, fx, dtable, n_tokens, d, vocab, 1);
  else rte::launch(embed_bwd_apply_kernel, grid_for(n, 256), 256, 0, ST(stream), reinterpret_cast<const unsigned long long*>(accum), dtable, n);
  RTE_LAUNCH_CHECK();
  return RTE_OK;
}

extern "C" int rte_embed_bwd_group(const int64_t* tokens, const float* dtable, int64_t* accum, int32_t n_tokens, int32_t d, int32_t vocab,
                                   int32_t* status, rte_stream_t stream) {
  RTE_CHECK_ARG(tokens && dtable && accum && n_tokens > 0 && d > 0 && vocab > 0);
  if (!embed_groups_fit(accum, dtable, n_tokens, d, vocab)) return RTE_ERR_UNSUPPORTED;
  EmbedGroups g;
  size_t clear = 0;
  const size_t bytes = embed_groups_layout(accum, n_tokens, d, &g, &clear);
  if (bytes > clear && cudaMemsetAsync(reinterpret_cast<char*>(accum) + clear, 0, bytes - clear, ST(stream)) != cudaSuccess) return RTE_ERR_LAUNCH;
  const size_t smem = (size_t)vocab * sizeof(int);
  if (cudaFuncSetAttribute(embed_group_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, EG_MAX_VOCAB * (int)sizeof(int)) != cudaSuccess)
    return RTE_ERR_LAUNCH;
  rte::launch(embed_group_kernel, 1, EG_THREADS, smem, ST(stream), tokens, n_tokens, vocab, g, status);
  RTE_LAUNCH_CHECK();
  return RTE_OK;
}
extern "C" int rte_embed_bwd_grouped(const float* dx, float* dtable, int64_t* accum, int32_t n_tokens, int32_t d, int32_t vocab,
                                     rte_stream_t stream) {
  RTE_CHECK_ARG(dx && dtable && accum && n_tokens > 0 && d > 0 && vocab > 0);
  if (!embed_groups_fit(accum, dtable, n_tokens, d, vocab)) return RTE_ERR_UNSUPPORTED;
  if (reinterpret_cast<uintptr_t>(dx) & 15) return RTE_ERR_ALIGNMENT;
  EmbedGroups g;
  embed_groups_layout(accum, n_tokens, d, &g);
  const long long most = rte::ceil_div64((long long)n_tokens * rte::ceil_div(d, EG_COLS), 8);
  rte::launch(embed_sum_kernel, (int)(most < 148 * 16 ? most : 148 * 16), 256, 0, ST(stream), dx, dtable, g, d);
  RTE_LAUNCH_CHECK();
  return RTE_OK;
}

extern "C" int rte_rmsnorm_fwd(const float* x, const float* w, const float* film_gamma, const float* film_beta,
                               void* y_bf16, float* y_f32, float* rstd, int32_t rows, int32_t d, float eps,
                               rte_stream_t stream) {
  RTE_CHECK_ARG(x && rows > 0 && d > 0 && d % 4 == 0 && (y_bf16 || y_f32));
  RTE_CHECK_ARG((film_gamma == nullptr) == (film_beta == nullptr));
  if (d > 128 * RN_MAX_V4) return RTE_ERR_UNSUPPORTED;
#define RTE_RN_FWD(NV)                                                                            \
  rte::launch(rmsnorm_fwd_kernel<NV>, rte::ceil_div(rows, 8), 256, 0, ST(stream), x, w, film_gamma, film_beta, \
      reinterpret_cast<__nv_bfloat16*>(y_bf16), y_f32, rstd, rows, d, eps)
  if (d <= 128) RTE_RN_FWD(1);
  else if (d <= 256) RTE_RN_FWD(2);
  else if (d <= 512) RTE_RN_FWD(4);
  else if (d <= 1024) RTE_RN_FWD(8);
  else RTE_RN_FWD(16);
#undef RTE_RN_FWD
  RTE_LAUNCH_CHECK();
  return RTE_OK;
}

extern "C" int rte_residual_rmsnorm_fwd(const float* base, const float* branch, const float* scale, const int32_t* active,
                                        const float* passthrough, int32_t S, const float* add2, const float* scale2,
                                        float* x1_out, float* x_out, const float* w, const float* film_gamma,
                                        const float* film_beta, void* y_bf16, float* rstd, int32_t rows, int32_t d, float eps,
                                        rte_stream_t stream) {
  return rte_residual_rmsnorm_fwd_splits(base, branch, 1, 0, nullptr, scale, active, passthrough, S, add2, scale2, x1_out, x_out,
                                         w, film_gamma, film_beta, y_bf16, rstd, rows, d, eps, stream);
}

extern "C" int rte_residual_rmsnorm_fwd_splits(const float* base, const float* branch, int32_t branch_splits,
                                               int64_t branch_split_stride, float* branch_out, const float* scale,
                                               const int32_t* active, const float* passthrough, int32_t S, const float* add2,
                                               const float* scale2, float* x1_out, float* x_out, const float* w,
                                               const float* film_gamma, const float* film_beta, void* y_bf16, float* rstd,
                                               int32_t rows, int32_t d, float eps, rte_stream_t stream) {
  RTE_CHECK_ARG(base && branch && scale && x_out && y_bf16 && rows > 0 && d > 0 && d % 4 == 0 && S > 0);
  RTE_CHECK_ARG(branch_splits >= 1 && (branch_splits == 1 || (branch_split_stride % 4 == 0 && branch_split_stride >= (int64_t)rows * d)));
  RTE_CHECK_ARG((active == nullptr || passthrough != nullptr) && (add2 == nullptr || scale2 != nullptr));
  RTE_CHECK_ARG((film_gamma == nullptr) == (film_beta == nullptr));
  if (d > 128 * RN_MAX_V4) return RTE_ERR_UNSUPPORTED;
#define RTE_RRN_FWD(NV)                                                                                              \
  rte::launch(residual_rmsnorm_fwd_kernel<NV>, rte::ceil_div(rows, 8), 256, 0, ST(stream), base, branch, scale, active, passthrough, \
      S, add2, scale2, x1_out, x_out, w, film_gamma, film_beta, reinterpret_cast<__nv_bfloat16*>(y_bf16), rstd, rows, d, eps, \
      branch_splits, (long long)branch_split_stride, branch_out)
  if (d <= 128) RTE_RRN_FWD(1);
  else if (d <= 256) RTE_RRN_FWD(2);
  else if (d <= 512) RTE_RRN_FWD(4);
  else if (d <= 1024) RTE_RRN_FWD(8);
  else RTE_RRN_FWD(16);
#undef RTE_RRN_FWD
  RTE_LAUNCH_CHECK();
  return RTE_OK;
}

extern "C" int rte_rmsnorm_bwd(const float* x, const float* w, const float* film_gamma, const float* rstd,
                               const void* dy_bf16, const float* dy_f32, const float* dres, float* dx_f32,
                               void* dx_bf16, float* dw_partial, float* dgamma_partial, float* dbeta_partial,
                               int32_t rows, int32_t d, int32_t max_partials, int32_t* n_partials,
                               rte_stream_t stream) {
  return rte_rmsnorm_bwd_splits(x, w, film_gamma, rstd, dy_bf16, dy_f32, 1, 0, dres, dx_f32, dx_bf16, dw_partial, dgamma_partial,
                                dbeta_partial, rows, d, max_partials, n_partials, stream);
}

extern "C" int rte_rmsnorm_bwd_splits(const float* x, const float* w, const float* film_gamma, const float* rstd,
                                      const void* dy_bf16, const float* dy_f32, int32_t dy_splits, int64_t dy_split_stride,
                                      const float* dres, float* dx_f32, void* dx_bf16, float* dw_partial,
                                      float* dgamma_partial, float* dbeta_partial, int32_t rows, int32_t d,
                                      int32_t max_partials, int32_t* n_partials, rte_stream_t stream) {
  RTE_CHECK_ARG(x && rstd && rows > 0 && d > 0 && d % 4 == 0 && (dy_bf16 || dy_f32) && (dx_f32 || dx_bf16));
  RTE_CHECK_ARG(dy_splits >= 1 && (dy_splits == 1 || (dy_f32 && !dy_bf16 && dy_split_stride % 4 == 0 &&
                                                      dy_split_stride >= (int64_t)rows * d)));
  RTE_CHECK_ARG((dgamma_partial == nullptr) == (dbeta_partial == nullptr));
  if (d > 128 * RN_MAX_V4) return RTE_ERR_UNSUPPORTED;
  const bool film = film_gamma || dgamma_partial, grads = dw_partial || dgamma_partial;
  const int across = rte::ceil_div(d, 128) * 32, block = d <= 1024 ? 256 : 512, down = block / across;
  // ROWS rows in flight per thread once every SM has its CTAs; fewer rows spread over as many CTAs as there are
  const int most = 148 * (768 / block);
  const bool few = rows <= most * down;
  int grid = rte::ceil_div(rows, down * (few ? 1 : film ? 2 : RN_ROWS));
  if (grid > most) grid = most;
  if (grads) {
    RTE_CHECK_ARG(max_partials >= 1);
    if (grid > max_partials) grid = max_partials;
  }
  if (n_partials) *n_partials = grid;
#define RTE_RN_BWD(ROWS, FILM, BLOCK)                                                                            \
  rte::launch(rmsnorm_bwd_kernel<ROWS, FILM, BLOCK>, grid, dim3(across, down), 0, ST(stream), x, w, film_gamma, rstd, \
              reinterpret_cast<const __nv_bfloat16*>(dy_bf16), dy_f32, dres, dx_f32,                             \
              reinterpret_cast<__nv_bfloat16*>(dx_bf16), dw_partial, dgamma_partial, dbeta_partial, rows, d,     \
              dy_splits, (long long)dy_split_stride)
#define RTE_RN_BWD_B(ROWS, FILM) do { if (block == 256) RTE_RN_BWD(ROWS, FILM, 256); else RTE_RN_BWD(ROWS, FILM, 512); } while (0)
  if (few) { if (film) RTE_RN_BWD_B(1, true); else RTE_RN_BWD_B(1, false); }
  else { if (film) RTE_RN_BWD_B(2, true); else RTE_RN_BWD_B(RN_ROWS, false); }
#undef RTE_RN_BWD_B
#undef RTE_RN_BWD
  RTE_LAUNCH_CHECK();
  return RTE_OK;
}

extern "C" int rte_colsum_partials(const float* partial, int32_t n_rows, int32_t d, float* out, int32_t accumulate,
                                   rte_stream_t stream) {
  RTE_CHECK_ARG(partial && out && n_rows > 0 && d > 0);
  rte::launch(colsum_kernel, rte::ceil_div(d, 32), 1024, 0, ST(stream), partial, n_rows, d, out, accumulate);
  RTE_LAUNCH_CHECK();
  return RTE_OK;
}

extern "C" int rte_colsum_partials3(const float* const* partials, float* const* outs, const int32_t* accumulate, int32_t count,
                                    int32_t n_rows, int32_t d, rte_stream_t stream) {
  RTE_CHECK_ARG(partials && outs && accumulate && count >= 1 && count <= 3 && n_rows > 0 && d > 0);
  ColsumJobs jobs;
  for (int i = 0; i < 3; ++i) {
    const int k = i < count ? i : 0;
    RTE_CHECK_ARG(partials[k] && outs[k]);
    jobs.j[i] = ColsumJob{partials[k], outs[k], accumulate[k]};
  }
  rte::launch(colsum3_kernel, dim3(rte::ceil_div(d, 32), count), 1024, 0, ST(stream), jobs, n_rows, d);
  RTE_LAUNCH_CHECK();
  return RTE_OK;
}

extern "C" int rte_ce_fwd_bwd(const void* logits, int32_t ldl, const int64_t* targets, const float* row_weight,
                              int32_t S, float* loss_tok, void* dlogits, int32_t rows, int32_t V, int32_t* status,
                              rte_stream_t stream) {
  RTE_CHECK_ARG(logits && targets && loss_tok && rows > 0 && V > 0 && ldl >= V && S > 0);
  RTE_CHECK_ARG(dlogits == nullptr || row_weight != nullptr);
  return launch_ce(reinterpret_cast<const __nv_bfloat16*>(logits), ldl, targets, row_weight, S, loss_tok, reinterpret_cast<__nv_bfloat16*>(dlogits),
                   rows, V, status, ST(stream));
}

extern "C" int rte_ce_fwd_bwd_f32(const float* logits, int32_t ldl, const int64_t* targets, const float* row_weight, int32_t S,
                                  float* loss_tok, float* dlogits, int32_t rows, int32_t V, int32_t* status, rte_stream_t stream) {
  RTE_CHECK_ARG(logits && targets && loss_tok && rows > 0 && V > 0 && ldl >= V && S > 0);
  RTE_CHECK_ARG(dlogits == nullptr || row_weight != nullptr);
  return launch_ce(logits, ldl, targets, row_weight, S, loss_tok, dlogits, rows, V, status, ST(stream));
}

extern "C" int rte_ce_loss_lse(const void* logits, int32_t f32, int32_t ldl, const int64_t* targets, float* loss_tok, float* lse, int32_t rows,
                               int32_t V, int32_t* status, rte_stream_t stream) {
  RTE_CHECK_ARG(logits && targets && loss_tok && lse && rows > 0 && V > 0 && ldl >= V);
  return (f32 ? launch_ce_lse<float> : launch_ce_lse<__nv_bfloat16>)(logits, ldl, targets, nullptr, 1, loss_tok, lse, nullptr, rows, V, status, ST(stream));
}

extern "C" int rte_ce_gradient(const void* logits, int32_t f32, int32_t ldl, const int64_t* targets, const float* row_weight, int32_t S,
                               const float* lse, void* dlogits, int32_t rows, int32_t V, int32_t* status, rte_stream_t stream) {
  RTE_CHECK_ARG(logits && targets && row_weight && lse && dlogits && rows > 0 && V > 0 && ldl >= V && S > 0);
  return (f32 ? launch_ce_lse<float> : launch_ce_lse<__nv_bfloat16>)(logits, ldl, targets, row_weight, S, nullptr, const_cast<float*>(lse), dlogits, rows,
                                                                      V, status, ST(stream));
}

extern "C" int rte_core_gradient_sums(const rte_core_sums* sums, int32_t T, int32_t pr, int32_t n_rows, int32_t d, int32_t P,
                                      rte_stream_t stream) {
  RTE_CHECK_ARG(sums && T > 0 && pr > 0 && n_rows > 0 && n_rows <= pr && d > 0 && d % 4 == 0 && P > 0);
  RTE_CHECK_ARG(sums->partials && sums->part_mlp && sums->part_attn && sums->part_alpha && sums->d_mlp_scale && sums->d_attn_scale &&
                sums->d_alpha);
  for (int i = 0; i < 2; ++i) RTE_CHECK_ARG(sums->dw[i] && sums->dgamma[i] && sums->dbeta[i]);
  if (reinterpret_cast<uintptr_t>(sums->partials) & 15) return RTE_ERR_ALIGNMENT;
  const long long grid = (2 + 4 * (long long)T) * rte::ceil_div(d, 32) + 2 * (long long)T + 1;
  RTE_CHECK_ARG(grid < (1ll << 31) && (long long)T * P < (1ll << 31));
  rte::launch(core_sums_kernel, (int)grid, 256, 0, ST(stream), *sums, T, pr, n_rows, d, P);
  RTE_LAUNCH_CHECK();
  return RTE_OK;
}

extern "C" int rte_segment_sum(const float* in, float* out, int32_t n_seg, int32_t seg_len, rte_stream_t stream) {
  RTE_CHECK_ARG(in && out && n_seg > 0 && seg_len > 0);
  rte::launch(segment_sum_kernel, n_seg, 128, 0, ST(stream), in, out, n_seg, seg_len);
  RTE_LAUNCH_CHECK();
  return RTE_OK;
}

extern "C" int rte_reduce_splits(const float* ws, int32_t splits, int64_t split_stride, int64_t n, float* out,
                                 int32_t accumulate, rte_stream_t stream) {
  RTE_CHECK_ARG(ws && out && splits >= 1 && n > 0);
  const bool vec = (split_stride % 4 == 0) && ((reinterpret_cast<uintptr_t>(ws) & 15) == 0) &&
                   ((reinterpret_cast<uintptr_t>(out) & 15) == 0);
  const long long n4 = vec ? (n >> 2) : 0;
  if (n4 > 0) {
    rte::launch(reduce_splits_kernel, grid_for(n4, 256), 256, 0, ST(stream), ws, splits, split_stride, n4, out, accumulate);
    RTE_LAUNCH_CHECK();
  }
  const long long rest = n - n4 * 4;
  if (rest > 0) {
    rte::launch(reduce_splits_tail_kernel, (int)rte::ceil_div64(rest, 256), 256, 0, ST(stream), ws, splits, split_stride, n4 * 4, n, out, accumulate);
    RTE_LAUNCH_CHECK();
  }
  return RTE_OK;
}

extern "C" int rte_swiglu_fwd(const void* ug, void* z, int64_t rows, int32_t F, rte_stream_t stream) {
  RTE_CHECK_ARG(ug && z && rows > 0 && F > 0 && F % 8 == 0);
  if ((reinterpret_cast<uintptr_t>(ug) & 15) || (reinterpret_cast<uintptr_t>(z) & 15)) return RTE_ERR_ALIGNMENT;
  rte::launch(swiglu_fwd_kernel, grid_for(rows * (F / 8), 256), 256, 0, ST(stream), reinterpret_cast<const __nv_bfloat16*>(ug),
                                                                          reinterpret_cast<__nv_bfloat16*>(z), rows, F);
  RTE_LAUNCH_CHECK();
  return RTE_OK;
}
extern "C" int rte_swiglu_bwd(const void* ug, const void* dz, void* dug, int64_t rows, int32_t F, rte_stream_t stream) {
  RTE_CHECK_ARG(ug && dz && dug && rows > 0 && F > 0 && F % 8 == 0);
  if ((reinterpret_cast<uintptr_t>(ug) & 15) || (reinterpret_cast<uintptr_t>(dz) & 15) || (reinterpret_cast<uintptr_t>(dug) & 15))
    return RTE_ERR_ALIGNMENT;
  rte::launch(swiglu_bwd_kernel, grid_for(rows * (F / 8), 256), 256, 0, ST(stream), reinterpret_cast<const __nv_bfloat16*>(ug), reinterpret_cast<const __nv_bfloat16*>(dz), reinterpret_cast<__nv_bfloat16*>(dug), rows, F);
  RTE_LAUNCH_CHECK();
  return RTE_OK;
}

extern "C" int rte_cast_f32_bf16(const float* src, void* dst, int64_t n, rte_stream_t stream) {
  RTE_CHECK_ARG(src && dst && n > 0);
  if ((reinterpret_cast<uintptr_t>(src) & 15) || (reinterpret_cast<uintptr_t>(dst) & 7)) return RTE_ERR_ALIGNMENT;
  rte::launch(cast_kernel, grid_for(n / 4 + 1, 256), 256, 0, ST(stream), src, reinterpret_cast<__nv_bfloat16*>(dst), n);
  RTE_LAUNCH_CHECK();
  return RTE_OK;
}
extern "C" int rte_fill_f32(float* dst, float value, int64_t n, rte_stream_t stream) {
  RTE_CHECK_ARG(dst && n > 0);
  rte::launch(fill_kernel, grid_for(n, 256), 256, 0, ST(stream), dst, value, n);
  RTE_LAUNCH_CHECK();
  return RTE_OK;
}
namespace {
int launch_add(const AddJobs& jobs, int count, cudaStream_t st) {
  long long threads = 0;                       // of the larger range: four elements each, one where only scalars serve
  for (int i = 0; i < count; ++i) {
    const bool vec = ((reinterpret_cast<uintptr_t>(jobs.j[i].dst) | reinterpret_cast<uintptr_t>(jobs.j[i].src)) & 15) == 0;
    const long long t = vec ? (jobs.j[i].n + 3) / 4 : jobs.j[i].n;
    if (t > threads) threads = t;
  }
  rte::launch(add_kernel, dim3(grid_for(threads, 256), count), 256, 0, st, jobs);
  RTE_LAUNCH_CHECK();
  return RTE_OK;
}
}  // namespace

extern "C" int rte_add_f32(float* dst, const float* src, int64_t n, rte_stream_t stream) {
  RTE_CHECK_ARG(src && dst && n > 0);
  return launch_add(AddJobs{{{dst, src, n}, {dst, src, 0}}}, 1, ST(stream));
}
extern "C" int rte_add2_f32(float* dst0, const float* src0, int64_t n0, float* dst1, const float* src1, int64_t n1, rte_stream_t stream) {
  RTE_CHECK_ARG(dst0 && src0 && n0 > 0 && dst1 && src1 && n1 > 0);
  return launch_add(AddJobs{{{dst0, src0, n0}, {dst1, src1, n1}}}, 2, ST(stream));
}
extern "C" int rte_axpy_rows_f32(float* dst, const float* vec, float alpha, int32_t rows, int32_t seg, int32_t d,
                                 rte_stream_t stream) {
  RTE_CHECK_ARG(dst && vec && rows > 0 && seg > 0 && d > 0);
  rte::launch(axpy_rows_kernel, grid_for((long long)rows * d, 256), 256, 0, ST(stream), dst, vec, alpha, rows, seg, d);
  RTE_LAUNCH_CHECK();
  return RTE_OK;
}

extern "C" int rte_adamw_multi_tensor_ex(const rte_adamw_tensor* table, int32_t n_tensors, int64_t total_chunks,
                                         const int32_t* chunk_tensor, const int32_t* chunk_index, const float* lr_table,
                                         int32_t* step_count, float beta1, float beta2, float eps, float weight_decay,
                                         const float* grad_scale, const rte_adamw_extras* ex, rte_stream_t stream) {
  RTE_CHECK_ARG(table && chunk_tensor && chunk_index && lr_table && step_count && n_tensors > 0 && total_chunks > 0);
  const int32_t* skip = ex ? ex->skip : nullptr;
  const int32_t* absent_flag = ex ? ex->absent_flag : nullptr;
  const uint8_t* absent_mask = ex ? ex->absent_mask : nullptr;
  RTE_CHECK_ARG((absent_flag == nullptr) == (absent_mask == nullptr));
  float* mpart = nullptr;
  if (ex && ex->metric_out) {
    RTE_CHECK_ARG(ex->metric_partial && ex->metric_group && ex->n_metric_groups > 0);
    mpart = ex->metric_partial;
  }
  rte::launch(adamw_kernel, (unsigned)total_chunks, 256, 0, ST(stream), table, chunk_tensor, chunk_index, lr_table, step_count,
                                                               beta1, beta2, eps, weight_decay, grad_scale, skip, mpart,
                                                               absent_flag, absent_mask);
  RTE_LAUNCH_CHECK();
  const int groups = mpart ? ex->n_metric_groups : 0;
  rte::launch(adamw_finish_kernel, groups + rte::ceil_div(n_tensors, 256), 256, 0, ST(stream), chunk_tensor, mpart ? ex->metric_group : nullptr,
              total_chunks, (const float*)mpart, mpart ? ex->metric_out : nullptr, groups, table, n_tensors, step_count, skip, absent_flag, absent_mask);
  RTE_LAUNCH_CHECK();
  return RTE_OK;
}

extern "C" int rte_adamw_multi_tensor(const rte_adamw_tensor* table, int32_t n_tensors, int64_t total_chunks,
                                      const int32_t* chunk_tensor, const int32_t* chunk_index, const float* lr_table,
                                      int32_t* step_count, float beta1, float beta2, float eps, float weight_decay,
                                      const float* grad_scale, rte_stream_t stream) {
  return rte_adamw_multi_tensor_ex(table, n_tensors, total_chunks, chunk_tensor, chunk_index, lr_table, step_count, beta1,
                                   beta2, eps, weight_decay, grad_scale, nullptr, stream);
}

extern "C" int rte_add_f32_guarded(float* dst, const float* src, int64_t n, const int32_t* skip, rte_stream_t stream) {
  RTE_CHECK_ARG(dst && src && skip && n > 0);
  rte::launch(add_guarded_kernel, grid_for(n, 256), 256, 0, ST(stream), dst, src, n, skip);
  RTE_LAUNCH_CHECK();
  return RTE_OK;
}

extern "C" int rte_nonfinite_guard(const float* a, int32_t na, const float* b, int32_t nb, const float* c, int32_t nc,
                                   int32_t* skip, float* flag_out, rte_stream_t stream) {
  RTE_CHECK_ARG(skip && na >= 0 && nb >= 0 && nc >= 0 && (a || na == 0) && (b || nb == 0) && (c || nc == 0));
  rte::launch(nonfinite_guard_kernel, 1, 256, 0, ST(stream), a, na, b, nb, c, nc, skip, flag_out);
  RTE_LAUNCH_CHECK();
  return RTE_OK;
}

extern "C" int rte_grad_norm_multi_tensor(const rte_adamw_tensor* table, int64_t total_chunks, const int32_t* chunk_tensor,
                                          const int32_t* chunk_index, float* partial, float* sumsq, float max_norm,
                                          float* clip_coef, rte_stream_t stream) {
  RTE_CHECK_ARG(table && chunk_tensor && chunk_index && partial && sumsq && total_chunks > 0);
  rte::launch(gradnorm_partial_kernel, (unsigned)total_chunks, 256, 0, ST(stream), table, chunk_tensor, chunk_index, partial);
  RTE_LAUNCH_CHECK();
  rte::launch(gradnorm_final_kernel, 1, 1024, 0, ST(stream), partial, total_chunks, sumsq, max_norm, clip_coef);
  RTE_LAUNCH_CHECK();
  return RTE_OK;
}

// Same result as rte_grad_norm_multi_tensor, but the per-chunk partial sums go to the library's own
// built-in array instead of a caller-supplied buffer: nothing is allocated here or by the caller.
// The first call on a device looks up the array's device address (a host-side runtime query, not a launch).
// Each call first overwrites every slot it later reads, so nothing has to be cleared between calls; but all
// calls on one device share the one array, so two calls whose kernels overlap in time would corrupt each other.
extern "C" int rte_grad_norm_multi_tensor_static(const rte_adamw_tensor* table, int64_t total_chunks,
                                                 const int32_t* chunk_tensor, const int32_t* chunk_index, float* sumsq,
                                                 float max_norm, float* clip_coef, rte_stream_t stream) {
  RTE_CHECK_ARG(table && chunk_tensor && chunk_index && sumsq && total_chunks > 0);
  if (total_chunks > GRADNORM_STATIC_MAX_CHUNKS) return RTE_ERR_SCRATCH_CAPACITY;
  float* partial = nullptr;
  const int rc = gradnorm_scratch_for_current_device(&partial);
  if (rc != RTE_OK) return rc;
  rte::launch(gradnorm_partial_kernel, (unsigned)total_chunks, 256, 0, ST(stream), table, chunk_tensor, chunk_index, partial);
  RTE_LAUNCH_CHECK();
  rte::launch(gradnorm_final_kernel, 1, 1024, 0, ST(stream), partial, total_chunks, sumsq, max_norm, clip_coef);
  RTE_LAUNCH_CHECK();
  return RTE_OK;
}

extern "C" int rte_topk_lowest_index(const float* scores, int32_t ld, int32_t rows, int32_t n, int32_t k,
                                     int32_t* idx, float* vals, rte_stream_t stream) {
  RTE_CHECK_ARG(scores && rows > 0 && n > 0 && k > 0 && k <= n && ld >= n && (idx || vals));
  rte::launch(topk_kernel, rte::ceil_div(rows, 8), 256, 0, ST(stream), scores, ld, rows, n, k, idx, vals);
  RTE_LAUNCH_CHECK();
  return RTE_OK;
}
