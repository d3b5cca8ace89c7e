// SVD-factor sparse SwiGLU FFN (reference layers.py:342-643, mask mode; svd_sparse_ffn_triton.py:480-714):
// the per-token neuron selection.  Everything GEMM-shaped runs in the tcgen05 GEMM (selector factors, exact
// up/gate pre-activations of ALL neurons, the down projection over the masked activations); what remains is, per
// token, four "k largest of F" selections:
//   candidates = top up_m of |up_hat|*wn  U  top gate_m of |silu(gate_hat)|*wn  U  top product_m of |up_hat*silu(gate_hat)|*wn
//   selected   = top top_k of |z|*wn over the candidates,      z = up * silu(gate) (exact)
// and z_masked = selected ? z : 0, so the down projection is a dense GEMM whose zero rows cost nothing extra.
//
// One warp per token, persistent over tokens.  A selection needs only the threshold that separates the k largest from
// the rest, so it is a root search on count(key >= t) = k over order-preserving integer keys in shared memory: a
// secant step on log(count) that starts from the previous token's threshold, safeguarded by bisection.  It ends as
// soon as a probe counts exactly k, or once at most 32 keys are left between the brackets (they are then ranked
// against each other, one per lane); keys equal to the threshold are taken in ascending index order.  Results are
// bit-exact with a stable sort by (value descending, index ascending), the tie rule of this build.
//
// What bounds it: the latency of each warp's own search.  13 KB of shared memory per token leave 16 warps on an SM, four
// per scheduler, and each alternates a sweep over its keys with a reduction that it has to wait for: 47 % of the issue
// slots are used (per instruction issued 2.2 warps wait on fixed latencies, 1.9 on global loads, 1.0 on shared memory), HBM
// at 26 %.  The instructions executed would take 176 us of the 374.  16384 tokens, F = 2048, k = 256: 1092 us with four
// 8-bit radix passes per selection (shared-memory atomics whose bins are the few exponents a row holds, so they
// serialise) -> 379 us with this search.

#include "rte_common.cuh"

namespace {

constexpr int SEL_MAX_WARPS = 4;               // warps per CTA
constexpr int SEL_SMEM = 224 * 1024;           // shared memory an SM has for these CTAs
constexpr int SEL_LIST = 32;                   // keys left between the brackets when the search turns to ranking

// Scores are non-negative (magnitudes times norms), so their bits order like integers; one less keeps a NaN below the
// open upper bracket.  Neurons that are no candidates get NO_KEY, below every score.
constexpr int NO_KEY = -0x7fffffff - 1;
__device__ __forceinline__ int score_key(float v) { return __float_as_int(v) - 1; }
__device__ __forceinline__ float key_score(int k) { return __int_as_float(k + 1); }

// per warp: the keys of one selection, the exact z as bf16, candidate | selected bits per four neurons, the ranking list
__host__ __device__ constexpr size_t sel_list_offset(int F) { return ((size_t)F * 6 + (size_t)F / 4 + 15) / 16 * 16; }
__host__ __device__ constexpr size_t sel_warp_bytes(int F) { return sel_list_offset(F) + (SEL_LIST + 4 + 8) * 4; }      // + four Guess
static_assert(sel_warp_bytes(100) % 16 == 0 && sel_warp_bytes(2048) % 16 == 0 && (SEL_LIST + 12) % 4 == 0, "every warp's keys start on 16 bytes");

struct Cut { int t, need; };     // keys >= t are taken; need >= 0: of the keys == t only the first `need` by index

struct Guess { int t; float slope; };          // where the last search of this list ended, and d value / d log(count) there

__device__ __forceinline__ int warp_count_ge(const int4* k4, int n4, int t, int lane) {
  int c = 0;
#pragma unroll 4
  for (int i = lane; i < n4; i += 32) {
    const int4 v = k4[i];
    c += (v.x >= t) + (v.y >= t) + (v.z >= t) + (v.w >= t);
  }
  return __reduce_add_sync(0xffffffffu, c);
}

// Threshold of the k largest of the 4 * n4 keys, 0 < k < 4 * n4.  `list`: SEL_LIST + 4 ints of this warp's shared memory.
__device__ Cut warp_cut(const int4* k4, int n4, int k, Guess& guess, int* list, int lane) {
  int lo = NO_KEY, hi = 0x7fffffff, c_lo = 4 * n4, c_hi = 0;      // count(>= lo) > k > count(>= hi)
  int t = guess.t;
  float slope = guess.slope, x_prev = 0.f, l_prev = 0.f;
  Cut cut = {0, -1};
  for (int it = 0;; ++it) {
    const int c = warp_count_ge(k4, n4, t, lane);
    if (c == k) { cut.t = t; break; }
    if (c > k) { lo = t; c_lo = c; } else { hi = t; c_hi = c; }
    if (c_lo - c_hi <= SEL_LIST) {
      if (lane == 0) list[SEL_LIST] = 0;
      __syncwarp();
      const unsigned first = (unsigned)lo, span = (unsigned)hi - first;
#pragma unroll 4
      for (int i = lane; i < n4; i += 32) {
        const int4 v = k4[i];
        if ((unsigned)v.x - first < span) list[atomicAdd(&list[SEL_LIST], 1)] = v.x;
        if ((unsigned)v.y - first < span) list[atomicAdd(&list[SEL_LIST], 1)] = v.y;
        if ((unsigned)v.z - first < span) list[atomicAdd(&list[SEL_LIST], 1)] = v.z;
        if ((unsigned)v.w - first < span) list[atomicAdd(&list[SEL_LIST], 1)] = v.w;
      }
      __syncwarp();
      const int m = c_lo - c_hi, r = k - c_hi;             // the r-th largest of these m keys, 1 <= r <= m
      const int mine = lane < m ? list[lane] : NO_KEY;
      int gt = 0, ge = 0;
      for (int j = 0; j < m; ++j) { const int w = list[j]; gt += w > mine; ge += w >= mine; }
      const unsigned who = __ballot_sync(0xffffffffu, lane < m && gt < r && r <= ge);
      const int src = __ffs(who) - 1;
      cut.t = __shfl_sync(0xffffffffu, mine, src);
      const int taken = r - __shfl_sync(0xffffffffu, gt, src), equal = __shfl_sync(0xffffffffu, ge - gt, src);
      cut.need = taken == equal ? -1 : taken;
      __syncwarp();
      break;
    }
    if ((unsigned)hi - (unsigned)lo <= 1u) { cut.t = lo; cut.need = k - c_hi; break; }      // more than SEL_LIST equal keys
    // next probe: secant on log(count) from the last two probes; the middle of the bracket when that leaves it
    const float x = key_score(t), l = __logf(c > 0 ? (float)c : 0.5f);
    if (it > 0 && l != l_prev) { const float s = (x - x_prev) / (l_prev - l); if (s > 0.f) slope = s; }
    x_prev = x; l_prev = l;
    int next = score_key(x + slope * (l - __logf((float)k)));
    if (it >= 12 || next <= lo || next >= hi) next = (int)((unsigned)lo + (((unsigned)hi - (unsigned)lo) >> 1));
    t = next;
  }
  guess.t = cut.t;
  guess.slope = slope;
  return cut;
}

// ORs the selected keys' bits (bit j = element 4 i + j of the group i = it * 32 + lane) into flags[i] at `shift`.
__device__ void warp_flag(const int4* k4, int n4, Cut cut, uint8_t* flags, int shift, int lane) {
  if (cut.need < 0) {
#pragma unroll 4
    for (int i = lane; i < n4; i += 32) {
      const int4 v = k4[i];
      const int m = (v.x >= cut.t) | (v.y >= cut.t) << 1 | (v.z >= cut.t) << 2 | (v.w >= cut.t) << 3;
      flags[i] |= (uint8_t)(m << shift);
    }
  } else {
    int taken = 0;                                   // equal keys with lower indices so far
    for (int i0 = 0; i0 < n4; i0 += 32) {
      const int i = i0 + lane;
      int gt = 0, eq = 0;
      if (i < n4) {
        const int4 v = k4[i];
        gt = (v.x > cut.t) | (v.y > cut.t) << 1 | (v.z > cut.t) << 2 | (v.w > cut.t) << 3;
        eq = (v.x == cut.t) | (v.y == cut.t) << 1 | (v.z == cut.t) << 2 | (v.w == cut.t) << 3;
      }
      const int mine = __popc(eq);
      int upto = mine;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) { const int u = __shfl_up_sync(0xffffffffu, upto, o); if (lane >= o) upto += u; }
      int room = cut.need - (taken + upto - mine);   // how many of this lane's equal keys are still taken
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (eq >> j & 1) { if (room > 0) gt |= 1 << j; --room; }
      if (i < n4) flags[i] |= (uint8_t)(gt << shift);
      taken += __shfl_sync(0xffffffffu, upto, 31);
    }
  }
}

// (not inlined four times: the kernel's code then stays in the instruction cache)
__device__ __noinline__ void warp_take(const int4* k4, int n4, int k, Guess* start, int* list, uint8_t* flags, int shift, int lane) {
  Guess guess = *start;                              // this warp's shared memory
  __syncwarp();
  if (k > 0) {
    Cut cut = {NO_KEY, -1};                            // k >= F: everything
    if (k < 4 * n4) {
      if (guess.slope == 0.f) {                      // this warp's first token: the k / F quantile of 32 of its keys
        const int mine = k4[lane % n4].x, want = min(31, k * 8 / n4);
        int gt = 0;
        for (int j = 0; j < 32; ++j) { const int w = __shfl_sync(0xffffffffu, mine, j); gt += w > mine || (w == mine && j < lane); }
        guess.t = __shfl_sync(0xffffffffu, mine, __ffs(__ballot_sync(0xffffffffu, gt == want)) - 1);
        guess.slope = 0.3f * fabsf(key_score(guess.t)) + 1e-30f;
      }
      cut = warp_cut(k4, n4, k, guess, list, lane);
      if (lane == 0) *start = guess;
    }
    warp_flag(k4, n4, cut, flags, shift, lane);
  }
  __syncwarp();
}

// Calls f(i, a[i], b[i], w[i]) for this lane's groups of four neurons, the loads of Q groups issued before the first use.
template <int Q, typename T, typename Fn>
__device__ __forceinline__ void for_groups(const T* a, const T* b, const float4* w, int n4, int lane, Fn f) {
  for (int i0 = lane; i0 < n4; i0 += 32 * Q) {
    T av[Q], bv[Q];
    float4 wv[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int i = min(i0 + 32 * q, n4 - 1);
      av[q] = a[i]; bv[q] = b[i]; wv[q] = w[i];
    }
#pragma unroll
    for (int q = 0; q < Q; ++q)
      if (i0 + 32 * q < n4) f(i0 + 32 * q, av[q], bv[q], wv[q]);
  }
}
__device__ __forceinline__ void prefetch_l2(const void* p, int bytes, int lane) {
  for (int o = lane * 128; o < bytes; o += 32 * 128) asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const char*>(p) + o));
}

// hats f32 [rows, 2F] = (up_hat | gate_hat); ug bf16 [rows, 2F] = exact (up | gate); wn f32 [F], not negative
// z_masked bf16 [rows, F]; selected uint8 [rows, F] (1 = selected); cand_count int32 [rows] (optional)
__global__ void __launch_bounds__(SEL_MAX_WARPS * 32, 4)
svd_select_kernel(const float* __restrict__ hats, const __nv_bfloat16* __restrict__ ug, const float* __restrict__ wn,
                  __nv_bfloat16* __restrict__ z_masked, uint8_t* __restrict__ selected, int32_t* __restrict__ cand_count,
                  int rows, int F, int up_m, int gate_m, int product_m, int top_k) {
  rte::after_previous_grid();
  extern __shared__ __align__(16) uint8_t sm_raw[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5, n4 = F / 4;
  uint8_t* base = sm_raw + warp * sel_warp_bytes(F);
  int4* k4 = reinterpret_cast<int4*>(base);
  uint2* z4 = reinterpret_cast<uint2*>(k4 + n4);
  uint8_t* flags = reinterpret_cast<uint8_t*>(z4 + n4);
  int* list = reinterpret_cast<int*>(base + sel_list_offset(F));
  const float4* wn4 = reinterpret_cast<const float4*>(wn);
  Guess* guess = reinterpret_cast<Guess*>(list + SEL_LIST + 4);
  if (lane < 4) guess[lane] = Guess{0, 0.f};
  __syncwarp();
  for (int row = blockIdx.x * warps + warp; row < rows; row += gridDim.x * warps) {
    const float4* uh = reinterpret_cast<const float4*>(hats + (size_t)row * 2 * F);
    const float4* gh = uh + n4;
    const int next = row + gridDim.x * warps;          // the next token's inputs start on their way to L2
    if (next < rows) {
      prefetch_l2(hats + (size_t)next * 2 * F, 8 * F, lane);
      prefetch_l2(ug + (size_t)next * 2 * F, 4 * F, lane);
    }
    // --- three candidate lists
    for_groups<4>(uh, uh, wn4, n4, lane, [&](int i, float4 u, float4, float4 w) {
      k4[i] = make_int4(score_key(fabsf(u.x) * w.x), score_key(fabsf(u.y) * w.y), score_key(fabsf(u.z) * w.z), score_key(fabsf(u.w) * w.w));
      flags[i] = 0;
    });
    warp_take(k4, n4, up_m, guess + 0, list, flags, 0, lane);
    if (gate_m > 0) {
      for_groups<4>(gh, gh, wn4, n4, lane, [&](int i, float4 g, float4, float4 w) {
        k4[i] = make_int4(score_key(fabsf(rte::silu_f(g.x)) * w.x), score_key(fabsf(rte::silu_f(g.y)) * w.y),
                          score_key(fabsf(rte::silu_f(g.z)) * w.z), score_key(fabsf(rte::silu_f(g.w)) * w.w));
      });
      warp_take(k4, n4, gate_m, guess + 1, list, flags, 0, lane);
    }
    if (product_m > 0) {
      for_groups<2>(uh, gh, wn4, n4, lane, [&](int i, float4 u, float4 g, float4 w) {
        k4[i] = make_int4(score_key(fabsf(u.x * rte::silu_f(g.x)) * w.x), score_key(fabsf(u.y * rte::silu_f(g.y)) * w.y),
                          score_key(fabsf(u.z * rte::silu_f(g.z)) * w.z), score_key(fabsf(u.w * rte::silu_f(g.w)) * w.w));
      });
      warp_take(k4, n4, product_m, guess + 2, list, flags, 0, lane);
    }
    // --- exact re-rank over the candidates
    const uint2* up = reinterpret_cast<const uint2*>(ug + (size_t)row * 2 * F);
    int n_cand = 0;
    for_groups<2>(up, up + n4, wn4, n4, lane, [&](int i, uint2 u, uint2 g, float4 w) {
      const float2 u0 = rte::unpack_bf16x2(u.x), u1 = rte::unpack_bf16x2(u.y), g0 = rte::unpack_bf16x2(g.x), g1 = rte::unpack_bf16x2(g.y);
      const int m = flags[i];
      const float z0 = u0.x * rte::silu_f(g0.x), z1 = u0.y * rte::silu_f(g0.y), z2 = u1.x * rte::silu_f(g1.x), z3 = u1.y * rte::silu_f(g1.y);
      n_cand += __popc(m);
      k4[i] = make_int4(m & 1 ? score_key(fabsf(z0) * w.x) : NO_KEY, m & 2 ? score_key(fabsf(z1) * w.y) : NO_KEY,
                        m & 4 ? score_key(fabsf(z2) * w.z) : NO_KEY, m & 8 ? score_key(fabsf(z3) * w.w) : NO_KEY);
      z4[i] = make_uint2(rte::pack_bf16x2(z0, z1), rte::pack_bf16x2(z2, z3));
    });
    warp_take(k4, n4, top_k, guess + 3, list, flags, 4, lane);
    n_cand = __reduce_add_sync(0xffffffffu, n_cand);
    if (cand_count && lane == 0) cand_count[row] = n_cand;
    uint2* zo = reinterpret_cast<uint2*>(z_masked + (size_t)row * F);
    uint32_t* so = reinterpret_cast<uint32_t*>(selected + (size_t)row * F);
#pragma unroll 4
    for (int i = lane; i < n4; i += 32) {
      const int m = flags[i] >> 4;
      uint2 z = z4[i];
      z.x &= (m & 1 ? 0xffffu : 0u) | (m & 2 ? 0xffff0000u : 0u);
      z.y &= (m & 4 ? 0xffffu : 0u) | (m & 8 ? 0xffff0000u : 0u);
      zo[i] = z;
      if (selected) so[i] = (uint32_t)(m & 1) | (uint32_t)(m & 2) << 7 | (uint32_t)(m & 4) << 14 | (uint32_t)(m & 8) << 21;
    }
    __syncwarp();
  }
}

// dug = SwiGLU backward of dz over the selected neurons only (zeros elsewhere)
__device__ __forceinline__ void swiglu_grad(bool on, float u, float g, float d, float& du, float& dg) {
  const float sg = rte::sigmoid_f(g);
  du = on ? d * g * sg : 0.f;
  dg = on ? d * u * sg * (1.f + g * (1.f - sg)) : 0.f;
}

// Eight neurons per thread with 16-byte accesses: bound by HBM (11 bytes per neuron; 16384 x 2048: 166 us with one
// neuron per thread -> 67 us).
__global__ void __launch_bounds__(256)
svd_swiglu_bwd8_kernel(const __nv_bfloat16* __restrict__ ug, const __nv_bfloat16* __restrict__ dz, const uint8_t* __restrict__ selected,
                       __nv_bfloat16* __restrict__ dug, long long groups, int f8) {
  rte::after_previous_grid();
  const uint4* ug8 = reinterpret_cast<const uint4*>(ug);
  const uint4* dz8 = reinterpret_cast<const uint4*>(dz);
  const uint2* sel8 = reinterpret_cast<const uint2*>(selected);
  uint4* dug8 = reinterpret_cast<uint4*>(dug);
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < groups; i += (long long)gridDim.x * blockDim.x) {
    const long long r = i / f8, j = i - r * f8;
    const uint2 m = sel8[i];
    uint4 du = make_uint4(0u, 0u, 0u, 0u), dg = du;
    if (m.x | m.y) {
      const uint4 u = ug8[r * 2 * f8 + j], g = ug8[(r * 2 + 1) * f8 + j], d = dz8[i];
      const uint32_t uu[4] = {u.x, u.y, u.z, u.w}, gg[4] = {g.x, g.y, g.z, g.w}, dd[4] = {d.x, d.y, d.z, d.w};
      uint32_t a[4], b[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float2 u2 = rte::unpack_bf16x2(uu[q]), g2 = rte::unpack_bf16x2(gg[q]), d2 = rte::unpack_bf16x2(dd[q]);
        const uint32_t mm = (q < 2 ? m.x : m.y) >> (16 * (q & 1));
        float du0, dg0, du1, dg1;
        swiglu_grad(mm & 0xffu, u2.x, g2.x, d2.x, du0, dg0);
        swiglu_grad(mm & 0xff00u, u2.y, g2.y, d2.y, du1, dg1);
        a[q] = rte::pack_bf16x2(du0, du1);
        b[q] = rte::pack_bf16x2(dg0, dg1);
      }
      du = make_uint4(a[0], a[1], a[2], a[3]);
      dg = make_uint4(b[0], b[1], b[2], b[3]);
    }
    dug8[r * 2 * f8 + j] = du;
    dug8[(r * 2 + 1) * f8 + j] = dg;
  }
}

// F not a multiple of eight, or rows off the 16-byte grid
__global__ void __launch_bounds__(256)
svd_swiglu_bwd_kernel(const __nv_bfloat16* __restrict__ ug, const __nv_bfloat16* __restrict__ dz, const uint8_t* __restrict__ selected,
                      __nv_bfloat16* __restrict__ dug, long long rows, int F) {
  rte::after_previous_grid();
  const long long total = rows * F;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const long long r = i / F;
    const int j = int(i % F);
    float du, dg;
    swiglu_grad(selected[i], __bfloat162float(ug[r * 2 * F + j]), __bfloat162float(ug[r * 2 * F + F + j]), __bfloat162float(dz[i]), du, dg);
    dug[r * 2 * F + j] = __float2bfloat16_rn(du);
    dug[r * 2 * F + F + j] = __float2bfloat16_rn(dg);
  }
}

__global__ void row_norm_kernel(const float* __restrict__ w, float* __restrict__ out, int rows, int d) {
  rte::after_previous_grid();
  const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (row >= rows) return;
  float s = 0.f;
  for (int c = lane; c < d; c += 32) { const float x = w[(size_t)row * d + c]; s += x * x; }
  s = rte::warp_sum(s);
  if (lane == 0) out[row] = sqrtf(s);
}

}  // namespace

#define ST(s) reinterpret_cast<cudaStream_t>(s)

extern "C" int rte_svd_ffn_select(const float* hats, const void* ug, const float* wd_norm, void* z_masked, uint8_t* selected,
                                  int32_t* cand_count, int32_t rows, int32_t F, int32_t up_m, int32_t gate_m, int32_t product_m,
                                  int32_t top_k, rte_stream_t stream) {
  RTE_CHECK_ARG(hats && ug && wd_norm && z_masked && rows > 0 && F > 0 && top_k > 0 && top_k <= F);
  RTE_CHECK_ARG(up_m >= 0 && gate_m >= 0 && product_m >= 0);
  // with fewer candidates than top_k the reference's result depends on an unspecified ordering of non-candidates
  if (up_m < top_k && gate_m < top_k && product_m < top_k) return RTE_ERR_UNSUPPORTED;
  const size_t warp_bytes = sel_warp_bytes(F);
  if (warp_bytes > SEL_SMEM || F % 4) return RTE_ERR_UNSUPPORTED;
  if ((reinterpret_cast<uintptr_t>(hats) | reinterpret_cast<uintptr_t>(wd_norm)) & 15) return RTE_ERR_ALIGNMENT;
  if (((reinterpret_cast<uintptr_t>(ug) | reinterpret_cast<uintptr_t>(z_masked)) & 7) || (reinterpret_cast<uintptr_t>(selected) & 3)) return RTE_ERR_ALIGNMENT;
  static bool set = false;
  if (!set) {
    if (cudaFuncSetAttribute(svd_select_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SEL_SMEM) != cudaSuccess) return RTE_ERR_LAUNCH;
    set = true;
  }
  // as many warps per SM as their shared memory allows (1 KB of it goes to the system per CTA); fewer per CTA where that packs better
  int warps = 1, resident = 1;
  for (int w = 1; w <= SEL_MAX_WARPS; ++w) {
    const int ctas = (int)((SEL_SMEM + 3 * 1024) / (w * warp_bytes + 1024));
    if (ctas >= 1 && ctas * w >= warps * resident) { warps = w; resident = ctas; }
  }
  const int sms = rte_device_sm_count();
  int grid = rte::ceil_div(rows, warps);
  if (grid > sms * resident) grid = sms * resident;
  rte::launch(svd_select_kernel, grid, warps * 32, warps * warp_bytes, ST(stream), hats, reinterpret_cast<const __nv_bfloat16*>(ug), wd_norm, reinterpret_cast<__nv_bfloat16*>(z_masked), selected, cand_count,
      rows, F, up_m, gate_m, product_m, top_k);
  RTE_LAUNCH_CHECK();
  return RTE_OK;
}

extern "C" int rte_svd_ffn_swiglu_bwd(const void* ug, const void* dz, const uint8_t* selected, void* dug, int64_t rows, int32_t F,
                                      rte_stream_t stream) {
  RTE_CHECK_ARG(ug && dz && selected && dug && rows > 0 && F > 0);
  const auto *u = reinterpret_cast<const __nv_bfloat16*>(ug), *z = reinterpret_cast<const __nv_bfloat16*>(dz);
  auto* out = reinterpret_cast<__nv_bfloat16*>(dug);
  const bool wide = F % 8 == 0 && ((reinterpret_cast<uintptr_t>(ug) | reinterpret_cast<uintptr_t>(dz) | reinterpret_cast<uintptr_t>(dug)) & 15) == 0 &&
                    (reinterpret_cast<uintptr_t>(selected) & 7) == 0;
  long long g = ((wide ? rows * F / 8 : rows * F) + 255) / 256;
  if (g > 148 * 16) g = 148 * 16;
  if (wide)
    rte::launch(svd_swiglu_bwd8_kernel, (int)g, 256, 0, ST(stream), u, z, selected, out, rows * (F / 8), F / 8);
  else
    rte::launch(svd_swiglu_bwd_kernel, (int)g, 256, 0, ST(stream), u, z, selected, out, rows, F);
  RTE_LAUNCH_CHECK();
  return RTE_OK;
}

extern "C" int rte_row_norm_f32(const float* w, float* out, int32_t rows, int32_t d, rte_stream_t stream) {
  RTE_CHECK_ARG(w && out && rows > 0 && d > 0);
  rte::launch(row_norm_kernel, rte::ceil_div(rows, 8), 256, 0, ST(stream), w, out, rows, d);
  RTE_LAUNCH_CHECK();
  return RTE_OK;
}
