// SVD-factor sparse SwiGLU FFN (reference layers.py:342-643, mask mode; svd_sparse_ffn_triton.py:480-714):
// the per-token neuron selection.  Everything GEMM-shaped runs in the tcgen05 GEMM (selector factors, exact
// up/gate pre-activations of ALL neurons, the down projection over the masked activations); what remains is, per
// token, four "k largest of F" selections:
//   candidates = top up_m of |up_hat|*wn  U  top gate_m of |silu(gate_hat)|*wn  U  top product_m of |up_hat*silu(gate_hat)|*wn
//   selected   = top top_k of |z|*wn over the candidates,      z = up * silu(gate) (exact)
// and z_masked = selected ? z : 0, so the down projection is a dense GEMM whose zero rows cost nothing extra.
//
// One warp per token, persistent over tokens.  A selection needs only the threshold that separates the k largest from
// the rest, so it is a root search on count(key >= t) = k: a secant step on log(count) that starts from the previous token's
// threshold, safeguarded by bisection.  The keys are the upper halves of the scores, packed as bf16 pairs in shared memory and
// clamped into the normal range, so that one HSET2 and one HADD2 compare and count two of them.  The search ends as soon as a
// probe counts exactly k, or once at most 32 keys are left between the brackets; those are ranked against each other, one per
// lane, by their full scores, which are computed again, equal ones in ascending index order.  Should more than 32 share their upper
// half (a row of equal scores), the search goes on over the full scores.  Results are bit-exact with a stable sort by (value
// descending, index ascending), the tie rule of this build.
//
// What bounds it: 9.5 K instructions per token at 54 % of the issue slots, and the loads they wait for (24 warps on an SM, 9 KB of shared
// memory each; per instruction issued 3.2 warps wait on global loads, 2.0 on fixed latencies, 1.0 on shared memory; DRAM at 35 %).
// us, with 32-bit keys and a divide for every list -> now: 16384 tokens, F = 2048, k = 256 377 -> 271, 5000 x 2000, k = 200
// 172 -> 165, 3000 x 512, k = 60 44 -> 27.  The SiLU of the fp32 lists is the correctly rounded quotient, made once for two lists (302 us
// with a divide for each, 245 with an approximate reciprocal, which loses the order of gates below -87).  With all keys in
// registers and the three lists searched together it took 583: the unrolled code does not stay in the instruction cache.

#include "rte_common.cuh"

namespace {

constexpr int SEL_MAX_WARPS = 4;               // warps per CTA
constexpr int SEL_SMEM = 224 * 1024;           // shared memory an SM has for these CTAs
constexpr int SEL_LIST = 32;                   // keys left between the brackets when the search turns to ranking

// Scores are not negative (magnitudes times norms), so their bits order like integers, a NaN above infinity.  A key is the upper
// half, clamped and moved by KEY_MIN so that every candidate's is a normal bf16 number; 0: no candidate.
constexpr uint32_t KEY_MIN = 0x0080u, KEY_END = 0x7f80u;              // KEY_MIN <= key < KEY_END
__device__ __forceinline__ uint32_t pair_keys(float a, float b) {
  return __vminu2(__byte_perm(__float_as_uint(a), __float_as_uint(b), 0x7632), 0x7eff7effu) + 0x00800080u;
}
__device__ __forceinline__ float key_value(uint32_t t) { return __uint_as_float((t - KEY_MIN) << 16); }
__device__ __forceinline__ __nv_bfloat162 as_pair(uint32_t v) { return *reinterpret_cast<__nv_bfloat162*>(&v); }

// per warp: the keys of one selection, the exact z as bf16, candidate | selected bits per four neurons, the ranking list
__host__ __device__ constexpr int sel_pad(int F) { return (F + 7) / 8 * 8; }
__host__ __device__ constexpr size_t sel_list_offset(int F) { return ((size_t)sel_pad(F) * 4 + (size_t)sel_pad(F) / 4 + 15) / 16 * 16; }
__host__ __device__ constexpr size_t sel_warp_bytes(int F) { return sel_list_offset(F) + (SEL_LIST + 4 + 8) * 4; }      // + four Guess
static_assert(sel_warp_bytes(100) % 16 == 0 && sel_warp_bytes(2048) % 16 == 0 && (SEL_LIST + 12) % 4 == 0, "every warp's keys start on 16 bytes");

struct Guess { int t; float slope; };          // where the last search of this list ended, and d value / d log(count) there

// A token's inputs, for the scores of single neurons: list 0 |up_hat|, 1 |silu(gate_hat)|, 2 |up_hat * silu(gate_hat)|, 3 |z|, times wn.
struct Token { const float* hat; const __nv_bfloat16* ug; const float* wn; int F; };
__device__ __forceinline__ int full_score(const Token& x, int which, int i) {
  float v;
  if (which == 0) v = x.hat[i];
  else if (which == 1) v = rte::silu_f(x.hat[x.F + i]);
  else if (which == 2) v = x.hat[i] * rte::silu_f(x.hat[x.F + i]);
  else v = __bfloat162float(x.ug[i]) * rte::silu_of_bf16(__bfloat162float(x.ug[x.F + i]));
  return __float_as_int(fabsf(v) * x.wn[i]);
}

__device__ __forceinline__ int warp_count_ge(const uint4* k8, int n8, uint32_t t, int lane) {
  const __nv_bfloat162 t2 = as_pair(t | t << 16);
  int c = 0;
  for (int i0 = 0; i0 < n8; i0 += 32 * 32) {                          // (a half counts to at most 128 per round: exact in bf16)
    __nv_bfloat162 a = as_pair(0u), b = a;
#pragma unroll 4
    for (int i = i0 + lane; i < min(n8, i0 + 32 * 32); i += 32) {
      const uint4 v = k8[i];
      a = __hadd2(a, __hge2(as_pair(v.x), t2)); b = __hadd2(b, __hge2(as_pair(v.y), t2));
      a = __hadd2(a, __hge2(as_pair(v.z), t2)); b = __hadd2(b, __hge2(as_pair(v.w), t2));
    }
    const float2 fa = __bfloat1622float2(a), fb = __bfloat1622float2(b);
    c += int((fa.x + fa.y) + (fb.x + fb.y));
  }
  return __reduce_add_sync(0xffffffffu, c);
}
// bit j: key j of the eight >= t
__device__ __forceinline__ uint32_t ge_bits(const uint4& v, __nv_bfloat162 t2) {
  const uint32_t x = (__hge2_mask(as_pair(v.x), t2) & 0x00020001u) | (__hge2_mask(as_pair(v.y), t2) & 0x00080004u) |
                     (__hge2_mask(as_pair(v.z), t2) & 0x00200010u) | (__hge2_mask(as_pair(v.w), t2) & 0x00800040u);
  return (x | x >> 16) & 0xffu;
}

// ORs the k largest of a list into `flags` (a byte per four neurons) at `shift`, 0 < k < total keys that are not 0.
// (not inlined four times: the kernel's code then stays in the instruction cache)
__device__ __noinline__ void warp_take(const uint4* k8, int n8, int k, int total, Guess* start, int* list, uint16_t* flags, int shift, const Token x,
                                       int which, int lane) {
  Guess guess = *start;                              // this warp's shared memory
  __syncwarp();
  if (guess.slope == 0.f) {                          // this warp's first token: the k / total quantile of 32 keys, those that are candidates
    const uint32_t mine = k8[lane % n8].x & 0xffffu;
    const int some = __popc(__ballot_sync(0xffffffffu, mine != 0u)), want = min(max(some - 1, 0), (int)((long long)k * some / total));
    int gt = 0;
    for (int j = 0; j < 32; ++j) { const uint32_t w = __shfl_sync(0xffffffffu, mine, j); gt += w > mine || (w == mine && j < lane); }
    guess.t = max((int)__shfl_sync(0xffffffffu, mine, __ffs(__ballot_sync(0xffffffffu, gt == want)) - 1), (int)KEY_MIN + 1);
    guess.slope = 0.3f * key_value((uint32_t)guess.t) + 1e-30f;
  }
  uint32_t lo = KEY_MIN, hi = KEY_END, t = min(max((uint32_t)guess.t, KEY_MIN + 1), KEY_END - 1);
  int c_lo = total, c_hi = 0;                        // count(>= lo) > k > count(>= hi), or lo == hi: exactly k at or above
  float slope = guess.slope, x_prev = 0.f, l_prev = 0.f;
  const float l_below = __logf(fmaxf((float)k - 8.f, 0.5f)), l_above = __logf((float)k + 8.f);
  for (int it = 0; c_lo - c_hi > SEL_LIST && hi - lo > 1; ++it) {
    const int c = warp_count_ge(k8, n8, t, lane);
    if (c == k) { lo = hi = t; c_lo = c_hi = c; break; }
    if (c > k) { lo = t; c_lo = c; } else { hi = t; c_hi = c; }
    // next probe: secant on log(count) from the last two probes, aimed a few keys past k, so that the bracket closes around it;
    // bisection when that does not converge
    const float v = key_value(t), l = __logf(c > 0 ? (float)c : 0.5f);
    if (it > 0 && l != l_prev) { const float s = (v - x_prev) / (l_prev - l); if (s > 0.f) slope = s; }
    x_prev = v; l_prev = l;
    const float aim = v + slope * (l - (c > k ? l_below : l_above));
    const uint32_t next = aim > 0.f ? (__float_as_uint(aim) >> 16) + KEY_MIN : 0u;
    t = it >= 8 ? (lo + hi) >> 1 : min(max(next, lo + 1), hi - 1);
  }
  if (lane == 0) { start->t = (int)lo; start->slope = slope; list[SEL_LIST] = 0; }
  __syncwarp();
  // what lies above is taken; what lies between is listed
  const __nv_bfloat162 hi2 = as_pair(hi | hi << 16), lo2 = as_pair(lo | lo << 16);
  const int n = c_lo - c_hi, need = k - c_hi;
  const bool few = n <= SEL_LIST;
#pragma unroll 4
  for (int i = lane; i < n8; i += 32) {
    const uint4 v = k8[i];
    const uint32_t above = ge_bits(v, hi2);
    if (lo != hi && few) {
      for (uint32_t in = ge_bits(v, lo2) & ~above; in; in &= in - 1) list[atomicAdd(&list[SEL_LIST], 1)] = 8 * i + __ffs(in) - 1;
    }
    flags[i] |= (uint16_t)(((above & 15u) | (above & 240u) << 4) << shift);
  }
  if (lo == hi) { __syncwarp(); return; }
  __syncwarp();
  if (few) {
    const int who = lane < n ? list[lane] : 0x7fffffff, score = lane < n ? full_score(x, which, who) : -1;
    int above = 0;
    for (int j = 0; j < n; ++j) {
      const int s = __shfl_sync(0xffffffffu, score, j), i = __shfl_sync(0xffffffffu, who, j);
      above += s > score || (s == score && i < who);
    }
    if (lane < n && above < need) atomicOr(reinterpret_cast<unsigned*>(flags) + (who >> 4), 1u << (8 * (who >> 2 & 3) + (who & 3) + shift));
    return;
  }
  // more keys than the list holds share their upper half: the threshold among their full scores, then equal ones by index
  auto between = [&](int i) { const uint4 v = k8[i]; return ge_bits(v, lo2) & ~ge_bits(v, hi2); };
  int a = 0, b = 0x7fffffff;                         // count(score >= a) >= need; a becomes the largest such score
  while (a < b) {
    const int mid = a + (b - a) / 2 + 1;
    int c = 0;
    for (int i = lane; i < n8; i += 32)
      for (uint32_t in = between(i); in; in &= in - 1) c += full_score(x, which, 8 * i + __ffs(in) - 1) >= mid;
    if (__reduce_add_sync(0xffffffffu, c) >= need) a = mid; else b = mid - 1;
  }
  int c = 0;
  for (int i = lane; i < n8; i += 32)
    for (uint32_t in = between(i); in; in &= in - 1) c += full_score(x, which, 8 * i + __ffs(in) - 1) > a;
  int room = need - __reduce_add_sync(0xffffffffu, c);      // how many of the equal ones, in ascending index order
  for (int i0 = 0; i0 < n8; i0 += 32) {
    const int i = i0 + lane;
    uint32_t gt = 0u, eq = 0u;
    for (uint32_t in = i < n8 ? between(i) : 0u; in; in &= in - 1) {
      const int s = full_score(x, which, 8 * i + __ffs(in) - 1);
      const uint32_t bit = in & (0u - in);
      if (s > a) gt |= bit; else if (s == a) eq |= bit;
    }
    const int have = __popc(eq);
    int upto = have;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const int u = __shfl_up_sync(0xffffffffu, upto, o); if (lane >= o) upto += u; }
    int left = room - (upto - have);
    for (; eq && left > 0; eq &= eq - 1, --left) gt |= eq & (0u - eq);
    if (i < n8) flags[i] |= (uint16_t)(((gt & 15u) | (gt & 240u) << 4) << shift);
    room -= __shfl_sync(0xffffffffu, upto, 31);
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
__global__ void __launch_bounds__(SEL_MAX_WARPS * 32, 6)
svd_select_kernel(const float* __restrict__ hats, const __nv_bfloat16* __restrict__ ug, const float* __restrict__ wn,
                  __nv_bfloat16* __restrict__ z_masked, uint8_t* __restrict__ selected, int32_t* __restrict__ cand_count,
                  int rows, int F, int up_m, int gate_m, int product_m, int top_k) {
  rte::after_previous_grid();
  extern __shared__ __align__(16) uint8_t sm_raw[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5, n4 = F / 4, n8 = sel_pad(F) / 8;
  uint8_t* base = sm_raw + warp * sel_warp_bytes(F);
  uint2* key = reinterpret_cast<uint2*>(base);                       // four keys each
  uint2* z4 = key + 2 * n8;
  uint8_t* flags = reinterpret_cast<uint8_t*>(z4 + 2 * n8);
  int* list = reinterpret_cast<int*>(base + sel_list_offset(F));
  const uint4* k8 = reinterpret_cast<const uint4*>(key);
  uint16_t* flags16 = reinterpret_cast<uint16_t*>(flags);
  const float4* wn4 = reinterpret_cast<const float4*>(wn);
  Guess* guess = reinterpret_cast<Guess*>(list + SEL_LIST + 4);
  if (lane < 4) guess[lane] = Guess{0, 0.f};
  if (lane == 0 && n4 < 2 * n8) key[n4] = z4[n4] = make_uint2(0u, 0u);      // (the padding of an odd number of groups: no candidates)
  __syncwarp();
  for (int row = blockIdx.x * warps + warp; row < rows; row += gridDim.x * warps) {
    const Token tok = {hats + (size_t)row * 2 * F, ug + (size_t)row * 2 * F, wn, F};
    const float4* uh = reinterpret_cast<const float4*>(tok.hat);
    const float4* gh = uh + n4;
    const int next = row + gridDim.x * warps;          // the next token's inputs start on their way to L2
    if (next < rows) {
      prefetch_l2(hats + (size_t)next * 2 * F, 8 * F, lane);
      prefetch_l2(ug + (size_t)next * 2 * F, 4 * F, lane);
    }
    // --- three candidate lists
    auto take = [&](const uint4* keys, int k, int which) {
      __syncwarp();
      if (k >= F) { for (int i = lane; i < n8; i += 32) flags16[i] |= 0x0f0fu; }
      else if (k > 0) warp_take(keys, n8, k, F, guess + which, list, flags16, 0, tok, which, lane);
      __syncwarp();
    };
    for (int i = lane; i < n8; i += 32) flags16[i] = 0;
    for_groups<4>(uh, uh, wn4, n4, lane, [&](int i, float4 u, float4, float4 w) {
      key[i] = make_uint2(pair_keys(fabsf(u.x) * w.x, fabsf(u.y) * w.y), pair_keys(fabsf(u.z) * w.z, fabsf(u.w) * w.w));
    });
    take(k8, up_m, 0);
    if (gate_m > 0 || product_m > 0) {                // one divide per gate: the products' keys lie where z will
      for_groups<2>(uh, gh, wn4, n4, lane, [&](int i, float4 u, float4 g, float4 w) {
        g = make_float4(rte::silu_f(g.x), rte::silu_f(g.y), rte::silu_f(g.z), rte::silu_f(g.w));
        key[i] = make_uint2(pair_keys(fabsf(g.x) * w.x, fabsf(g.y) * w.y), pair_keys(fabsf(g.z) * w.z, fabsf(g.w) * w.w));
        z4[i] = make_uint2(pair_keys(fabsf(u.x * g.x) * w.x, fabsf(u.y * g.y) * w.y), pair_keys(fabsf(u.z * g.z) * w.z, fabsf(u.w * g.w) * w.w));
      });
      take(k8, gate_m, 1);
      take(reinterpret_cast<const uint4*>(z4), product_m, 2);
    }
    // --- exact re-rank over the candidates
    const uint2* up = reinterpret_cast<const uint2*>(tok.ug);
    int n_cand = 0;
    for_groups<2>(up, up + n4, wn4, n4, lane, [&](int i, uint2 u, uint2 g, float4 w) {
      const float2 u0 = rte::unpack_bf16x2(u.x), u1 = rte::unpack_bf16x2(u.y), g0 = rte::unpack_bf16x2(g.x), g1 = rte::unpack_bf16x2(g.y);
      const uint32_t m = flags[i];
      const float z0 = u0.x * rte::silu_of_bf16(g0.x), z1 = u0.y * rte::silu_of_bf16(g0.y), z2 = u1.x * rte::silu_of_bf16(g1.x), z3 = u1.y * rte::silu_of_bf16(g1.y);
      n_cand += __popc(m);
      key[i] = make_uint2(pair_keys(fabsf(z0) * w.x, fabsf(z1) * w.y) & ((m & 1u) * 0xffffu | (m & 2u) * 0x7fff8000u),
                          pair_keys(fabsf(z2) * w.z, fabsf(z3) * w.w) & ((m >> 2 & 1u) * 0xffffu | (m >> 2 & 2u) * 0x7fff8000u));
      z4[i] = make_uint2(rte::pack_bf16x2(z0, z1), rte::pack_bf16x2(z2, z3));
    });
    n_cand = __reduce_add_sync(0xffffffffu, n_cand);
    __syncwarp();
    if (lane == 0 && guess[3].slope == 0.f) guess[3] = guess[2];       // (a warp's first token: the products' scores estimate these)
    __syncwarp();
    if (top_k < n_cand) warp_take(k8, n8, top_k, n_cand, guess + 3, list, flags16, 4, tok, 3, lane);
    else for (int i = lane; i < n8; i += 32) flags16[i] |= (uint16_t)(flags16[i] << 4);
    __syncwarp();
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
