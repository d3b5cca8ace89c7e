// Tensor-core causal attention (forward and backward) for head sizes 32 / 64 / 128 and S <= 256.
//
// One CTA = one (sample, head).  Q, K (rotary embedding applied in place), V and -- in backward -- dO of the head sit in
// shared memory as bf16 rows of HD + 8 elements (the padding keeps ldmatrix free of bank conflicts); each warp owns
// 16-row tiles and issues mma.sync m16n8k16 (bf16 in, fp32 accumulate) on fragments fetched with ldmatrix.x4, transposed
// where the product wants it (V in P.V, K in dS.K, dO in P^T.dO, Q in dS^T.Q), so no transposed copy exists.  Scores
// never leave registers; backward recomputes the probabilities from the saved log-sum-exp in two sweeps (query-major
// for dQ, key-major for dK and dV), which keeps it free of atomics and bitwise reproducible.
//
// The contractions are far too small to bound these kernels (16 GFLOP at 32 x 256 x 16 heads x 64 with both sweeps);
// what does are the bytes of qkv / dqkv and, before that, latency: the loads of a head, then a dependent chain of small
// products.  So a head is loaded ONCE (a CTA per 64 rows would load K, V, Q and dO up to four times and leave one CTA of
// four warps per SM at S = 256), everything a CTA reads from global memory is requested before the first wait, causal
// work is balanced over the warps (tiles i and n-1-i in forward; sweep 1 of tile i costs i+1, its sweep 2 n-i), and
// results leave as 16-byte stores after a transpose inside each quad of lanes.
// 128 x 64 x 8 heads x 64: forward 24.6 -> 18.4 us, backward 49 -> 37 us; 32 x 256 x 16 x 64: forward 102 -> 45 us, backward
// 510 -> 102 us (34 / 67 and 134 / 268 MB; launch included).
#pragma once

#include "rte_common.cuh"

namespace attn_mma {

__device__ __forceinline__ void mma16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ldsm_x4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldsm_x4_trans(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ float inv_freq(int pair, int hd) { return 1.0f / powf(10000.0f, (float)(2 * pair) / (float)hd); }
// (without a table; a call, so that its registers do not burden the kernels that are given one)
__device__ __noinline__ float2 rope_value(int pos, int pair, int hd) {
  float2 v;
  sincosf((float)pos * inv_freq(pair, hd), &v.y, &v.x);
  return v;
}
// cos/sin of position `pos`, rotary pair `pair`: from the caller's table [S, hd/2, 2] when given, else computed.
__device__ __forceinline__ void rope_cs(const float* __restrict__ table, int pos, int pair, int hd, float& cs, float& sn) {
  if (table != nullptr) {
    const float2 v = *reinterpret_cast<const float2*>(table + ((size_t)pos * (hd / 2) + pair) * 2);
    cs = v.x; sn = v.y;
  } else {
    const float2 v = rope_value(pos, pair, hd);
    cs = v.x; sn = v.y;
  }
}

// ---- loads.  All tiles of a head are requested at once with cp.async (16-byte pieces straight into shared memory);
// every thread later rotates, scales or dots exactly the pieces it copied, so it only waits for its own copies.
__device__ __forceinline__ void cp_async16(void* smem_dst, const void* gsrc) {
  const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(smem_dst));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// rows [0, S) of one head -> smem rows [0, s_pad) (row stride HD + 8), rows past S zeroed
template <int HD, int NTHR>
__device__ __forceinline__ void tile_async(const __nv_bfloat16* __restrict__ src, int ld, int S, int s_pad, __nv_bfloat16* dst) {
  constexpr int LDS = HD + 8, CPR = HD / 8;      // 16-byte pieces per row
  for (int idx = threadIdx.x; idx < s_pad * CPR; idx += NTHR) {
    const int r = idx / CPR, ch = idx % CPR;
    __nv_bfloat16* d = dst + r * LDS + 8 * ch;
    if (r < S) cp_async16(d, src + (size_t)r * ld + 8 * ch);
    else *reinterpret_cast<uint4*>(d) = make_uint4(0u, 0u, 0u, 0u);
  }
}

struct Rot { float cs[4], sn[4]; };            // of the four rotary pairs of one piece
template <int HD>
__device__ __forceinline__ Rot rot_of(const float* __restrict__ rope, int r, int ch) {
  const float4* t4 = reinterpret_cast<const float4*>(rope + ((size_t)r * (HD / 2) + 4 * ch) * 2);
  const float4 a = t4[0], b = t4[1];
  return Rot{{a.x, a.z, b.x, b.z}, {a.y, a.w, b.y, b.w}};
}
__device__ __forceinline__ void rotate_piece(__nv_bfloat16* at, const Rot& o) {
  uint4* p = reinterpret_cast<uint4*>(at);
  const uint4 raw = *p;
  uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const float2 v = rte::unpack_bf16x2(w[q]);
    w[q] = rte::pack_bf16x2(v.x * o.cs[q] - v.y * o.sn[q], v.y * o.cs[q] + v.x * o.sn[q]);
  }
  *p = make_uint4(w[0], w[1], w[2], w[3]);
}
// Rotary embedding in place on q and k, NP pieces per thread, STEP at a time; PENDING: copy groups that may still be in
// flight when the first piece is touched (the table is read before that wait).
template <int HD, int NTHR, int NP, int STEP, int PENDING>
__device__ __forceinline__ void rotate_qk(__nv_bfloat16* q, __nv_bfloat16* k, int S, const float* __restrict__ rope) {
  constexpr int LDS = HD + 8, CPR = HD / 8;
  if (rope == nullptr) {
    cp_async_wait<PENDING>();
#pragma unroll 1
    for (int idx = threadIdx.x; idx < S * CPR; idx += NTHR) {
      const int r = idx / CPR, ch = idx % CPR;
      Rot rot;
#pragma unroll
      for (int j = 0; j < 4; ++j) rope_cs(nullptr, r, 4 * ch + j, HD, rot.cs[j], rot.sn[j]);
      rotate_piece(q + r * LDS + 8 * ch, rot);
      rotate_piece(k + r * LDS + 8 * ch, rot);
    }
    return;
  }
#pragma unroll
  for (int i0 = 0; i0 < NP; i0 += STEP) {
    Rot rot[STEP];
#pragma unroll
    for (int i = 0; i < STEP; ++i) {
      const int idx = threadIdx.x + (i0 + i) * NTHR;
      if (idx / CPR < S) rot[i] = rot_of<HD>(rope, idx / CPR, idx % CPR);
    }
    if (i0 == 0) cp_async_wait<PENDING>();
#pragma unroll
    for (int i = 0; i < STEP; ++i) {
      const int idx = threadIdx.x + (i0 + i) * NTHR, r = idx / CPR, at = r * LDS + 8 * (idx % CPR);
      if (r < S) {
        rotate_piece(q + at, rot[i]);
        rotate_piece(k + at, rot[i]);
      }
    }
  }
}

// ---- fragments.  Lane addresses inside a row-major tile: A operand and transposed B (rows 0-15, columns 0-15), plain B
// of 16 rows (n) by 16 columns (k).
template <int HD>
__device__ __forceinline__ uint32_t frag_at(const __nv_bfloat16* tile, int lane) {       // A, or B^T through .trans
  return static_cast<uint32_t>(__cvta_generic_to_shared(tile + (lane & 15) * (HD + 8) + (lane >> 4) * 8));
}
template <int HD>
__device__ __forceinline__ uint32_t frag_b_at(const __nv_bfloat16* tile, int lane) {     // [n0-7 k0-7][n0-7 k8-15][n8-15 k0-7][n8-15 k8-15]
  return static_cast<uint32_t>(__cvta_generic_to_shared(tile + ((lane & 7) + ((lane >> 4) << 3)) * (HD + 8) + ((lane >> 3) & 1) * 8));
}
template <int HD>
__host__ __device__ constexpr uint32_t rows_bytes(int rows) { return rows * (HD + 8) * 2; }

// acc[half] += A (16 rows) . B(16 rows, two halves of 8)^T over all HD columns
template <int HD>
__device__ __forceinline__ void product16(float (&acc)[2][4], const uint32_t (&a)[HD / 16][4], uint32_t b_at) {
#pragma unroll
  for (int h = 0; h < 2; ++h) acc[h][0] = acc[h][1] = acc[h][2] = acc[h][3] = 0.f;
#pragma unroll
  for (int ks = 0; ks < HD / 16; ++ks) {
    uint32_t b[4];
    ldsm_x4(b, b_at + ks * 32);
    mma16816(acc[0], a[ks], b[0], b[1]);
    mma16816(acc[1], a[ks], b[2], b[3]);
  }
}
// acc[nd] += A (16 x 16) . T where T is 16 rows of a row-major tile, all HD columns
template <int HD>
__device__ __forceinline__ void product_trans(float (&acc)[HD / 8][4], const uint32_t (&a)[4], uint32_t t_at) {
#pragma unroll
  for (int nd = 0; nd < HD / 8; nd += 2) {
    uint32_t b[4];
    ldsm_x4_trans(b, t_at + nd * 16);
    mma16816(acc[nd], a, b[0], b[1]);
    mma16816(acc[nd + 1], a, b[2], b[3]);
  }
}
// Four words per lane (word j = column pair of 8-column tile j) -> the four words of ONE tile, tile = lane's place in its
// quad: what a 16-byte store wants.
__device__ __forceinline__ uint4 quad_transpose(uint32_t w0, uint32_t w1, uint32_t w2, uint32_t w3, int t) {
  uint32_t r = __shfl_xor_sync(0xffffffffu, (t & 1) ? w0 : w1, 1);
  if (t & 1) w0 = r; else w1 = r;
  r = __shfl_xor_sync(0xffffffffu, (t & 1) ? w2 : w3, 1);
  if (t & 1) w2 = r; else w3 = r;
  const uint32_t x = __shfl_xor_sync(0xffffffffu, (t & 2) ? w0 : w2, 2), y = __shfl_xor_sync(0xffffffffu, (t & 2) ? w1 : w3, 2);
  return (t & 2) ? make_uint4(x, y, w2, w3) : make_uint4(w0, w1, x, y);
}

// ------------------------------------------------------------------ forward
// SMAX <= 64: a warp per 16-row tile.  Longer: half as many warps, each takes tiles n-1-p and p; the softmax runs over
// chunks of 64 keys with the usual rescaling.
template <int SMAX>
__host__ __device__ constexpr int fwd_warps() { return SMAX <= 64 ? SMAX / 16 : SMAX / 32; }
template <int HD, int SMAX>
__host__ __device__ constexpr int fwd_ctas() { return HD > 64 ? (SMAX <= 64 ? 3 : 1) : SMAX <= 64 ? 7 : SMAX <= 128 ? 4 : 2; }

template <int HD, int SMAX>
__global__ void __launch_bounds__(32 * fwd_warps<SMAX>(), fwd_ctas<HD, SMAX>())
fwd_kernel(const __nv_bfloat16* __restrict__ qkv, int ld, int sec, __nv_bfloat16* __restrict__ y, int ldy,
           float* __restrict__ lse, const float* __restrict__ rope, int S, int s_pad, int H,
           __nv_bfloat16* __restrict__ ym, const int32_t* __restrict__ mask_row, const float* __restrict__ mask_tab) {
  rte::after_previous_grid();
  constexpr int LDS = HD + 8, NTHR = 32 * fwd_warps<SMAX>(), CPR = HD / 8, NP = SMAX * CPR / NTHR, CK = SMAX < 64 ? SMAX : 64;
  constexpr bool PAIRS = SMAX > 64;
  extern __shared__ __align__(16) uint8_t smraw[];
  __nv_bfloat16* sq = reinterpret_cast<__nv_bfloat16*>(smraw);       // [s_pad][LDS] each
  __nv_bfloat16* sk = sq + s_pad * LDS;
  __nv_bfloat16* sv = sk + s_pad * LDS;
  const int b = blockIdx.x / H, h = blockIdx.x % H;
  const __nv_bfloat16* base = qkv + (size_t)b * S * ld + h * HD;
  tile_async<HD, NTHR>(base, ld, S, s_pad, sq);
  tile_async<HD, NTHR>(base + sec, ld, S, s_pad, sk);
  cp_async_commit();
  tile_async<HD, NTHR>(base + 2 * sec, ld, S, s_pad, sv);
  cp_async_commit();
  rotate_qk<HD, NTHR, NP, (NP < 4 ? NP : 4), 1>(sq, sk, S, rope);
  cp_async_wait<0>();
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3, n_tiles = s_pad / 16;
  const float scale = rsqrtf((float)HD), c2 = scale * 1.4426950408889634f;
  const uint32_t q_at = frag_at<HD>(sq, lane), k_at = frag_b_at<HD>(sk, lane), v_at = frag_at<HD>(sv, lane);
  // optional second output: the same rows times a per-sample column mask (ym = bf16(y) * mask_tab[mask_row[b]][col],
  // exactly what a separate pass over the stored y would give)
  const float* mt = ym ? mask_tab + (size_t)mask_row[b] * (H * HD) + h * HD : nullptr;
#pragma unroll 1
  for (int half = 0; half < (PAIRS ? 2 : 1); ++half) {
    const int tile = !PAIRS ? warp : half == 0 ? n_tiles - 1 - warp : warp;
    if (PAIRS ? (half == 0 ? tile < n_tiles - 1 - tile : tile >= n_tiles - 1 - tile) : tile >= n_tiles) break;
    const int row_a = tile * 16 + g, row_b = row_a + 8;
    float m0 = -INFINITY, m1 = -INFINITY, s0 = 0.f, s1 = 0.f;
    float o[HD / 8][4];
#pragma unroll
    for (int nd = 0; nd < HD / 8; ++nd) o[nd][0] = o[nd][1] = o[nd][2] = o[nd][3] = 0.f;
    int c0 = 0;
#pragma unroll 1
    do {
      const int n16 = min(CK / 16, tile + 1 - c0 / 16);               // key blocks of 16 in this chunk
      uint32_t pk[CK / 16][4];
      {
        float sc[CK / 8][4];
#pragma unroll
        for (int nb = 0; nb < CK / 8; ++nb) sc[nb][0] = sc[nb][1] = sc[nb][2] = sc[nb][3] = 0.f;
#pragma unroll
        for (int ks = 0; ks < HD / 16; ++ks) {
          uint32_t a[4];
          ldsm_x4(a, q_at + rows_bytes<HD>(tile * 16) + ks * 32);
#pragma unroll
          for (int j = 0; j < CK / 16; ++j)
            if (j < n16) {
              uint32_t kb[4];
              ldsm_x4(kb, k_at + rows_bytes<HD>(c0 + 16 * j) + ks * 32);
              mma16816(sc[2 * j], a, kb[0], kb[1]);
              mma16816(sc[2 * j + 1], a, kb[2], kb[3]);
            }
        }
        float n0 = m0, n1 = m1;
#pragma unroll
        for (int j = 0; j < CK / 16; ++j)
          if (j < n16) {
            if (c0 / 16 + j == tile) {                                // the diagonal block: later keys are masked
#pragma unroll
              for (int q = 0; q < 2; ++q) {
                const int c = 8 * q + 2 * t;
                if (c > g) sc[2 * j + q][0] = -INFINITY;
                if (c + 1 > g) sc[2 * j + q][1] = -INFINITY;
                if (c > g + 8) sc[2 * j + q][2] = -INFINITY;
                if (c + 1 > g + 8) sc[2 * j + q][3] = -INFINITY;
              }
            }
            n0 = fmaxf(n0, fmaxf(fmaxf(sc[2 * j][0], sc[2 * j][1]), fmaxf(sc[2 * j + 1][0], sc[2 * j + 1][1])));
            n1 = fmaxf(n1, fmaxf(fmaxf(sc[2 * j][2], sc[2 * j][3]), fmaxf(sc[2 * j + 1][2], sc[2 * j + 1][3])));
          }
        n0 = fmaxf(n0, __shfl_xor_sync(0xffffffffu, n0, 1)); n0 = fmaxf(n0, __shfl_xor_sync(0xffffffffu, n0, 2));
        n1 = fmaxf(n1, __shfl_xor_sync(0xffffffffu, n1, 1)); n1 = fmaxf(n1, __shfl_xor_sync(0xffffffffu, n1, 2));
        if (PAIRS && c0 > 0) {
          const float f0 = ex2((m0 - n0) * c2), f1 = ex2((m1 - n1) * c2);
          s0 *= f0; s1 *= f1;
#pragma unroll
          for (int nd = 0; nd < HD / 8; ++nd) { o[nd][0] *= f0; o[nd][1] *= f0; o[nd][2] *= f1; o[nd][3] *= f1; }
        }
        m0 = n0; m1 = n1;
        const float b0 = m0 * c2, b1 = m1 * c2;
#pragma unroll
        for (int j = 0; j < CK / 16; ++j)
          if (j < n16) {
#pragma unroll
            for (int q = 0; q < 2; ++q) {
              float* v = sc[2 * j + q];
              v[0] = ex2(fmaf(v[0], c2, -b0)); v[1] = ex2(fmaf(v[1], c2, -b0));
              v[2] = ex2(fmaf(v[2], c2, -b1)); v[3] = ex2(fmaf(v[3], c2, -b1));
              s0 += v[0] + v[1];
              s1 += v[2] + v[3];
              pk[j][2 * q] = rte::pack_bf16x2(v[0], v[1]);
              pk[j][2 * q + 1] = rte::pack_bf16x2(v[2], v[3]);
            }
          }
      }
#pragma unroll
      for (int j = 0; j < CK / 16; ++j)
        if (j < n16) product_trans<HD>(o, pk[j], v_at + rows_bytes<HD>(c0 + 16 * j));
      c0 += CK;
    } while (PAIRS && c0 <= tile * 16);
    s0 += __shfl_xor_sync(0xffffffffu, s0, 1); s0 += __shfl_xor_sync(0xffffffffu, s0, 2);
    s1 += __shfl_xor_sync(0xffffffffu, s1, 1); s1 += __shfl_xor_sync(0xffffffffu, s1, 2);
    const float i0 = 1.f / s0, i1 = 1.f / s1;
#pragma unroll
    for (int grp = 0; grp < HD / 32; ++grp) {
#pragma unroll
      for (int q = 0; q < 2; ++q) {                                   // rows a and b
        const float f = q ? i1 : i0;
        const uint4 w = quad_transpose(rte::pack_bf16x2(o[4 * grp][2 * q] * f, o[4 * grp][2 * q + 1] * f),
                                       rte::pack_bf16x2(o[4 * grp + 1][2 * q] * f, o[4 * grp + 1][2 * q + 1] * f),
                                       rte::pack_bf16x2(o[4 * grp + 2][2 * q] * f, o[4 * grp + 2][2 * q + 1] * f),
                                       rte::pack_bf16x2(o[4 * grp + 3][2 * q] * f, o[4 * grp + 3][2 * q + 1] * f), t);
        const int row = q ? row_b : row_a, col = (4 * grp + t) * 8;
        if (row < S) {
          *reinterpret_cast<uint4*>(y + (size_t)(b * S + row) * ldy + h * HD + col) = w;
          if (ym) {
            const float4 ma = reinterpret_cast<const float4*>(mt + col)[0], mb = reinterpret_cast<const float4*>(mt + col)[1];
            const float2 v0 = rte::unpack_bf16x2(w.x), v1 = rte::unpack_bf16x2(w.y), v2 = rte::unpack_bf16x2(w.z), v3 = rte::unpack_bf16x2(w.w);
            *reinterpret_cast<uint4*>(ym + (size_t)(b * S + row) * ldy + h * HD + col) =
                make_uint4(rte::pack_bf16x2(v0.x * ma.x, v0.y * ma.y), rte::pack_bf16x2(v1.x * ma.z, v1.y * ma.w),
                           rte::pack_bf16x2(v2.x * mb.x, v2.y * mb.y), rte::pack_bf16x2(v3.x * mb.z, v3.y * mb.w));
          }
        }
      }
    }
    if (t == 0 && row_a < S) lse[((size_t)b * H + h) * S + row_a] = m0 * scale + __logf(s0);
    if (t == 0 && row_b < S) lse[((size_t)b * H + h) * S + row_b] = m1 * scale + __logf(s1);
  }
}

// ------------------------------------------------------------------ backward
// rows a and b of a 16 x HD accumulator times `f` (and rotated back where rope-carrying) -> bf16 rows of `dst`
template <int HD, bool UNROPE>
__device__ __forceinline__ void store_tile(const float (&acc)[HD / 8][4], float f, __nv_bfloat16* dst, int ld, int row_a, int S,
                                           const float* __restrict__ rope, int t) {
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const int row = row_a + 8 * q, pos = min(row, S - 1);
#pragma unroll
    for (int grp = 0; grp < HD / 32; ++grp) {
      uint32_t w[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float x = acc[4 * grp + j][2 * q] * f, z = acc[4 * grp + j][2 * q + 1] * f;
        if constexpr (UNROPE) {
          float cs, sn;
          rope_cs(rope, pos, (4 * grp + j) * 4 + t, HD, cs, sn);
          const float u = x;
          x = u * cs + z * sn;
          z = z * cs - u * sn;
        }
        w[j] = rte::pack_bf16x2(x, z);
      }
      const uint4 v = quad_transpose(w[0], w[1], w[2], w[3], t);
      if (row < S) *reinterpret_cast<uint4*>(dst + (size_t)row * ld + (4 * grp + t) * 8) = v;
    }
  }
}

// A warp per 16-row tile: dQ of the tile's queries over key blocks <= tile, then dK and dV of its keys over query blocks
// >= tile.  MASKED: the upstream gradient is dy[row, c] * mask_tab[mask_row[sample]][c] (the banked core's recipe mask on
// the attention output, layers.py:702-728); the mask is applied to the dy tile in shared memory.  With few (sample, head)
// pairs the launch has two CTAs per head along z, one per sweep: half the latency.
template <int HD, int SMAX>
__host__ __device__ constexpr int bwd_ctas() { return HD > 64 ? 1 : SMAX <= 64 ? 4 : SMAX <= 128 ? 2 : 1; }

template <int HD, int SMAX, bool MASKED>
__global__ void __launch_bounds__(2 * SMAX, bwd_ctas<HD, SMAX>())
bwd_kernel(const __nv_bfloat16* __restrict__ qkv, int ld, int sec, const __nv_bfloat16* __restrict__ y,
           const __nv_bfloat16* __restrict__ dy, int ldy, const float* __restrict__ lse,
           __nv_bfloat16* __restrict__ dqkv, const float* __restrict__ rope, int S, int s_pad, int H,
           const int32_t* __restrict__ mask_row, const float* __restrict__ mask_tab) {
  rte::after_previous_grid();
  constexpr int LDS = HD + 8, NTHR = 2 * SMAX, CPR = HD / 8, NP = SMAX * CPR / NTHR;
  extern __shared__ __align__(16) uint8_t smraw[];
  __nv_bfloat16* sq = reinterpret_cast<__nv_bfloat16*>(smraw);       // [s_pad][LDS] each
  __nv_bfloat16* sk = sq + s_pad * LDS;
  __nv_bfloat16* sv = sk + s_pad * LDS;
  __nv_bfloat16* sdo = sv + s_pad * LDS;
  float* slse = reinterpret_cast<float*>(sdo + s_pad * LDS);         // log2 of the row sums
  float* sD = slse + s_pad;                                          // rowsum(dO * O)
  const int b = blockIdx.x / H, h = blockIdx.x % H;
  const __nv_bfloat16* base = qkv + (size_t)b * S * ld + h * HD;
  tile_async<HD, NTHR>(dy + (size_t)b * S * ldy + h * HD, ldy, S, s_pad, sdo);
  cp_async_commit();
  tile_async<HD, NTHR>(base, ld, S, s_pad, sq);
  tile_async<HD, NTHR>(base + sec, ld, S, s_pad, sk);
  tile_async<HD, NTHR>(base + 2 * sec, ld, S, s_pad, sv);
  cp_async_commit();
  {
    const __nv_bfloat16* yb = y + (size_t)b * S * ldy + h * HD;
    uint4 yv[NP];
#pragma unroll
    for (int i = 0; i < NP; ++i) {
      const int idx = threadIdx.x + i * NTHR, r = idx / CPR;
      yv[i] = r < S ? *reinterpret_cast<const uint4*>(yb + (size_t)r * ldy + 8 * (idx % CPR)) : make_uint4(0u, 0u, 0u, 0u);
    }
    if (threadIdx.x < s_pad)                                         // (rows past S: probability exp2(x - inf) = 0)
      slse[threadIdx.x] = threadIdx.x < S ? lse[((size_t)b * H + h) * S + threadIdx.x] * 1.4426950408889634f : INFINITY;
    cp_async_wait<1>();
#pragma unroll
    for (int i = 0; i < NP; ++i) {
      const int idx = threadIdx.x + i * NTHR, r = idx / CPR, ch = idx % CPR;
      if (r < s_pad) {                                               // (uniform over a row's threads: s_pad * CPR is a multiple of 32)
        uint4* at = reinterpret_cast<uint4*>(sdo + r * LDS + 8 * ch);
        const uint4 raw = *at;
        uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
        const uint32_t o4[4] = {yv[i].x, yv[i].y, yv[i].z, yv[i].w};
        float m8[8];
        if (MASKED) {
          const float4* m4 = reinterpret_cast<const float4*>(mask_tab + (size_t)mask_row[b] * (H * HD) + h * HD + 8 * ch);
          const float4 ma = m4[0], mb = m4[1];
          m8[0] = ma.x; m8[1] = ma.y; m8[2] = ma.z; m8[3] = ma.w; m8[4] = mb.x; m8[5] = mb.y; m8[6] = mb.z; m8[7] = mb.w;
        }
        float part = 0.f;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          if (MASKED) {
            const float2 v = rte::unpack_bf16x2(w[q]);
            w[q] = rte::pack_bf16x2(v.x * m8[2 * q], v.y * m8[2 * q + 1]);
          }
          const float2 x = rte::unpack_bf16x2(w[q]), z = rte::unpack_bf16x2(o4[q]);
          part += x.x * z.x + x.y * z.y;
        }
        if (MASKED) *at = make_uint4(w[0], w[1], w[2], w[3]);
#pragma unroll
        for (int o = 1; o < CPR; o <<= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
        if (ch == 0) sD[r] = part;
      }
    }
  }
  rotate_qk<HD, NTHR, NP, (NP < 4 ? NP : 4), 0>(sq, sk, S, rope);
  __syncthreads();
  const int lane = threadIdx.x & 31, tile = threadIdx.x >> 5, g = lane >> 2, t = lane & 3, n_tiles = s_pad / 16;
  if (tile >= n_tiles) return;
  const float scale = rsqrtf((float)HD), c2 = scale * 1.4426950408889634f;
  const int row_a = tile * 16 + g;
  __nv_bfloat16* dbase = dqkv + (size_t)b * S * ld + h * HD;
  const int only = gridDim.z == 2 ? (int)blockIdx.z : -1;

  // ---- sweep 1: dQ
  if (only != 1) {
    uint32_t qf[HD / 16][4], dof[HD / 16][4];
    const uint32_t q_at = frag_at<HD>(sq, lane) + rows_bytes<HD>(tile * 16), do_at = frag_at<HD>(sdo, lane) + rows_bytes<HD>(tile * 16);
#pragma unroll
    for (int ks = 0; ks < HD / 16; ++ks) {
      ldsm_x4(qf[ks], q_at + ks * 32);
      ldsm_x4(dof[ks], do_at + ks * 32);
    }
    const uint32_t k_at = frag_b_at<HD>(sk, lane), v_at = frag_b_at<HD>(sv, lane), kt_at = frag_at<HD>(sk, lane);
    const float la = slse[row_a], lb = slse[row_a + 8], Da = sD[row_a], Db = sD[row_a + 8];
    float dq[HD / 8][4];
#pragma unroll
    for (int nd = 0; nd < HD / 8; ++nd) dq[nd][0] = dq[nd][1] = dq[nd][2] = dq[nd][3] = 0.f;
#pragma unroll 1
    for (int j = 0; j <= tile; ++j) {
      float st[2][4], dp[2][4];
      product16<HD>(st, qf, k_at + rows_bytes<HD>(16 * j));
      product16<HD>(dp, dof, v_at + rows_bytes<HD>(16 * j));
      uint32_t a[4];
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        float d0 = ex2(fmaf(st[q][0], c2, -la)) * (dp[q][0] - Da), d1 = ex2(fmaf(st[q][1], c2, -la)) * (dp[q][1] - Da);
        float d2 = ex2(fmaf(st[q][2], c2, -lb)) * (dp[q][2] - Db), d3 = ex2(fmaf(st[q][3], c2, -lb)) * (dp[q][3] - Db);
        if (j == tile) {                                             // the diagonal block: keys after the query do not count
          const int c = 8 * q + 2 * t;
          if (c > g) d0 = 0.f;
          if (c + 1 > g) d1 = 0.f;
          if (c > g + 8) d2 = 0.f;
          if (c + 1 > g + 8) d3 = 0.f;
        }
        a[2 * q] = rte::pack_bf16x2(d0, d1);
        a[2 * q + 1] = rte::pack_bf16x2(d2, d3);
      }
      product_trans<HD>(dq, a, kt_at + rows_bytes<HD>(16 * j));
    }
    store_tile<HD, true>(dq, scale, dbase, ld, row_a, S, rope, t);
  }

  // ---- sweep 2: dK, dV (st and dp transposed: rows are keys, columns queries).  K and V fragments come from shared
  // memory again for every block: the two accumulators leave no registers for them.
  if (only != 0) {
    const uint32_t k_at = frag_at<HD>(sk, lane) + rows_bytes<HD>(tile * 16), v_at = frag_at<HD>(sv, lane) + rows_bytes<HD>(tile * 16);
    const uint32_t q_at = frag_b_at<HD>(sq, lane), do_at = frag_b_at<HD>(sdo, lane), qt_at = frag_at<HD>(sq, lane), dot_at = frag_at<HD>(sdo, lane);
    float dk[HD / 8][4], dv[HD / 8][4];
#pragma unroll
    for (int nd = 0; nd < HD / 8; ++nd) {
      dk[nd][0] = dk[nd][1] = dk[nd][2] = dk[nd][3] = 0.f;
      dv[nd][0] = dv[nd][1] = dv[nd][2] = dv[nd][3] = 0.f;
    }
#pragma unroll 1
    for (int j = tile; j < n_tiles; ++j) {
      float st[2][4], dp[2][4];
#pragma unroll
      for (int q = 0; q < 2; ++q) st[q][0] = st[q][1] = st[q][2] = st[q][3] = dp[q][0] = dp[q][1] = dp[q][2] = dp[q][3] = 0.f;
#pragma unroll
      for (int ks = 0; ks < HD / 16; ++ks) {
        uint32_t a[4], c[4];
        ldsm_x4(a, k_at + ks * 32);
        ldsm_x4(c, q_at + rows_bytes<HD>(16 * j) + ks * 32);
        mma16816(st[0], a, c[0], c[1]);
        mma16816(st[1], a, c[2], c[3]);
        ldsm_x4(a, v_at + ks * 32);
        ldsm_x4(c, do_at + rows_bytes<HD>(16 * j) + ks * 32);
        mma16816(dp[0], a, c[0], c[1]);
        mma16816(dp[1], a, c[2], c[3]);
      }
      uint32_t ap[4], ad[4];
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int c = 8 * q + 2 * t;
        const float2 l = *reinterpret_cast<const float2*>(slse + 16 * j + c), D = *reinterpret_cast<const float2*>(sD + 16 * j + c);
        float p0 = ex2(fmaf(st[q][0], c2, -l.x)), p1 = ex2(fmaf(st[q][1], c2, -l.y));
        float p2 = ex2(fmaf(st[q][2], c2, -l.x)), p3 = ex2(fmaf(st[q][3], c2, -l.y));
        if (j == tile) {                                             // queries before the key
          if (c < g) p0 = 0.f;
          if (c + 1 < g) p1 = 0.f;
          if (c < g + 8) p2 = 0.f;
          if (c + 1 < g + 8) p3 = 0.f;
        }
        ap[2 * q] = rte::pack_bf16x2(p0, p1);
        ap[2 * q + 1] = rte::pack_bf16x2(p2, p3);
        ad[2 * q] = rte::pack_bf16x2(p0 * (dp[q][0] - D.x), p1 * (dp[q][1] - D.y));
        ad[2 * q + 1] = rte::pack_bf16x2(p2 * (dp[q][2] - D.x), p3 * (dp[q][3] - D.y));
      }
      product_trans<HD>(dv, ap, dot_at + rows_bytes<HD>(16 * j));
      product_trans<HD>(dk, ad, qt_at + rows_bytes<HD>(16 * j));
    }
    store_tile<HD, true>(dk, scale, dbase + sec, ld, row_a, S, rope, t);
    store_tile<HD, false>(dv, 1.f, dbase + 2 * sec, ld, row_a, S, rope, t);
  }
}

// dynamic shared memory above 48 KB is granted once per kernel and device
template <typename Kernel>
int allow_smem(Kernel kernel, int bytes, uint64_t& granted) {
  if (bytes <= 48 * 1024) return RTE_OK;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return RTE_ERR_LAUNCH;
  if (dev < 64 && (granted >> dev & 1)) return RTE_OK;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess) return RTE_ERR_LAUNCH;
  if (dev < 64) granted |= 1ull << dev;
  return RTE_OK;
}

template <int HD, int SMAX>
int launch_fwd(const void* qkv, int ld, int sec, void* y, int ldy, float* lse, const float* rope, int B, int S, int H, cudaStream_t st,
               void* ym = nullptr, const int32_t* mask_row = nullptr, const float* mask_tab = nullptr) {
  static uint64_t granted = 0;
  const int rc = allow_smem(fwd_kernel<HD, SMAX>, 3 * SMAX * (HD + 8) * 2, granted);
  if (rc != RTE_OK) return rc;
  const int s_pad = (S + 15) & ~15;
  rte::launch(fwd_kernel<HD, SMAX>, B * H, 32 * fwd_warps<SMAX>(), 3 * s_pad * (HD + 8) * 2, st, reinterpret_cast<const __nv_bfloat16*>(qkv), ld, sec,
              reinterpret_cast<__nv_bfloat16*>(y), ldy, lse, rope, S, s_pad, H, reinterpret_cast<__nv_bfloat16*>(ym), mask_row, mask_tab);
  RTE_LAUNCH_CHECK();
  return RTE_OK;
}

template <int HD, int SMAX>
int launch_bwd(const void* qkv, int ld, int sec, const void* y, const void* dy, int ldy, const float* lse, void* dqkv,
               const float* rope, int B, int S, int H, cudaStream_t st, const int32_t* mask_row = nullptr,
               const float* mask_tab = nullptr) {
  static uint64_t granted[2] = {0, 0};
  constexpr int most = 4 * SMAX * (HD + 8) * 2 + 2 * SMAX * 4;
  const bool masked = mask_row != nullptr;
  const auto kernel = masked ? bwd_kernel<HD, SMAX, true> : bwd_kernel<HD, SMAX, false>;
  const int rc = allow_smem(kernel, most, granted[masked]);
  if (rc != RTE_OK) return rc;
  const int s_pad = (S + 15) & ~15;
  rte::launch(kernel, dim3(B * H, 1, B * H < 148 ? 2 : 1), 2 * SMAX, 4 * s_pad * (HD + 8) * 2 + 2 * s_pad * 4, st,
              reinterpret_cast<const __nv_bfloat16*>(qkv), ld, sec, reinterpret_cast<const __nv_bfloat16*>(y), reinterpret_cast<const __nv_bfloat16*>(dy), ldy, lse,
              reinterpret_cast<__nv_bfloat16*>(dqkv), rope, S, s_pad, H, mask_row, mask_tab);
  RTE_LAUNCH_CHECK();
  return RTE_OK;
}

}  // namespace attn_mma
