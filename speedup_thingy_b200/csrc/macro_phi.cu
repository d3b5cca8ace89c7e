// The macro operator Phi of the recursive model, forward and backward, on device:
//   out = h + s_cfg * scale * tanh(gain * h + silu(z @ v) @ u + bias),
//   z   = [rmsnorm(h), mean_S rmsnorm(h), h0],  h == h0 on the hot path (the consistency term applies Phi to a state
//   h != h0: the kernels that touch the h0 slice take it as a second pointer `hx`, equal to `h` on the hot path),
// with gain / v / u / bias / scale selected PER SAMPLE by (recipe id, stride id).
//
// The per-sample low-rank weights are small (3d x m and m x d, m <= 64), so these are SIMT kernels
// tiled through shared memory; the weight gather is pointer arithmetic, the concat `z` is never
// materialised (three K-slices; the pooled slice collapses to one m-vector per sample).
// Parameter gradients are produced per sample and then summed per (recipe, stride) key in sample
// order, so results are bitwise reproducible and keys no sample used receive exact zeros.

#include "rte_common.cuh"

namespace {

constexpr int TT = 32;        // tokens per CTA tile
constexpr int NTHR = 256;
constexpr int CH = 64;        // d-chunk staged in shared memory
constexpr int MMAX = 64;      // largest supported macro rank

struct PhiDims { int B, S, d, m, K; };

__device__ __forceinline__ size_t key_of(const int32_t* rid, const int32_t* sid, int b, int K) {
  return (size_t)rid[b] * K + sid[b];
}

// rstd per token, pooled = mean_S(rmsnorm(h0)) per sample, pa = pooled @ v[d:2d, :].
// A cluster of PREP_CTAS CTAs per sample: warps take tokens, a token stays in registers between its norm and the column
// sums (one pass over h0), the CTAs add their column sums and products through distributed shared memory in rank order.
// One CTA per sample left most SMs without work and read h0 twice: 32 x 256 x 1024 136 -> 29 us in the step (34 MB).
// PART 1 is what does not depend on the route (the pass over h0), which the caller may run beside the router; PART 2 is the product
// with the slice of v that the route picks, from the pooled rows in memory: the same sums in the same order as PART 0, both.
// Between the router and the operator's first product, transposed parameters included, 32 x 256 x 1024: 39 -> 6 us; 128 x 64 x 512
// in an audited step 26 -> 6.
constexpr int PREP_CTAS = 8;

__device__ __forceinline__ float dsmem_read(const float* p, int rank) {
  uint32_t a = static_cast<uint32_t>(__cvta_generic_to_shared(p)), r;
  float v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(r) : "memory");
  return v;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
}

// NV float4 per lane hold a token (d <= 128 * NV, d % 4 == 0)
template <int NV, int PART>
__global__ void __cluster_dims__(PREP_CTAS, 1, 1) __launch_bounds__(NTHR)
phi_prep_kernel(const float* __restrict__ h0, const float* __restrict__ v, const int32_t* __restrict__ rid,
                const int32_t* __restrict__ sid, float* __restrict__ rstd, float* __restrict__ pooled,
                float* __restrict__ pa, PhiDims D, float eps) {
  rte::after_previous_grid();
  extern __shared__ __align__(16) float sm[];            // warp sums [NTHR / 32][d] -> (row 0) this CTA's column sums; then pooled [d], products [m]
  constexpr int WARPS = NTHR / 32;
  float* ps = PART == 2 ? sm : sm + (size_t)WARPS * D.d;
  float* pj = ps + D.d;
  const int b = blockIdx.x / PREP_CTAS, rank = blockIdx.x % PREP_CTAS, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, d4 = D.d >> 2;
  // this CTA's slice of the columns
  const int per = rte::ceil_div(D.d, PREP_CTAS), c0 = rank * per, n = min(D.d, c0 + per) - c0;
  if constexpr (PART != 2) {
    const float4* hb = reinterpret_cast<const float4*>(h0 + (size_t)b * D.S * D.d);
    float4 acc[NV];
#pragma unroll
    for (int i = 0; i < NV; ++i) acc[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int s = rank * WARPS + warp; s < D.S; s += PREP_CTAS * WARPS) {
      float4 x[NV];
      float ss = 0.f;
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        const int c = lane + 32 * i;
        x[i] = c < d4 ? hb[(size_t)s * d4 + c] : make_float4(0.f, 0.f, 0.f, 0.f);
      }
#pragma unroll
      for (int i = 0; i < NV; ++i) ss += x[i].x * x[i].x + x[i].y * x[i].y + x[i].z * x[i].z + x[i].w * x[i].w;
      const float r = rsqrtf(rte::warp_sum(ss) / (float)D.d + eps);
      if (lane == 0) rstd[(size_t)b * D.S + s] = r;
#pragma unroll
      for (int i = 0; i < NV; ++i) { acc[i].x += x[i].x * r; acc[i].y += x[i].y * r; acc[i].z += x[i].z * r; acc[i].w += x[i].w * r; }
    }
#pragma unroll
    for (int i = 0; i < NV; ++i)
      if (lane + 32 * i < d4) reinterpret_cast<float4*>(sm + (size_t)warp * D.d)[lane + 32 * i] = acc[i];
    __syncthreads();
    for (int c = threadIdx.x; c < D.d; c += NTHR) {
      float t = sm[c];
#pragma unroll
      for (int w = 1; w < WARPS; ++w) t += sm[(size_t)w * D.d + c];
      sm[c] = t;
    }
    cluster_sync();
    // its sum over the cluster
    for (int c = threadIdx.x; c < n; c += NTHR) {
      float t = 0.f;
#pragma unroll
      for (int k = 0; k < PREP_CTAS; ++k) t += dsmem_read(sm + c0 + c, k);
      t /= (float)D.S;
      ps[c] = t;
      pooled[(size_t)b * D.d + c0 + c] = t;
    }
    if constexpr (PART == 1) {
      cluster_sync();                      // (no CTA leaves while another reads its shared memory)
      return;
    }
  } else {
    for (int c = threadIdx.x; c < n; c += NTHR) ps[c] = pooled[(size_t)b * D.d + c0 + c];
  }
  __syncthreads();
  // threads = column groups x ranks: neighbouring threads read neighbouring elements of v
  float* part = ps + rte::ceil_div(D.d, 4) * 4 + MMAX;                 // [NTHR]
  const int mw = D.m <= 32 ? 32 : 64, j = threadIdx.x % mw, cg = threadIdx.x / mw, groups = NTHR / mw;
  const float* v2 = v + (key_of(rid, sid, b, D.K) * 3 * D.d + D.d + c0) * D.m;
  float t = 0.f;
  if (j < D.m)
    for (int c = cg; c < n; c += groups) t += ps[c] * v2[(size_t)c * D.m + j];
  part[threadIdx.x] = t;
  __syncthreads();
  if (threadIdx.x < D.m) {
    t = 0.f;
    for (int k = 0; k < groups; ++k) t += part[k * mw + threadIdx.x];
    pj[threadIdx.x] = t;
  }
  cluster_sync();
  if (rank == 0 && threadIdx.x < D.m) {
    t = 0.f;
#pragma unroll
    for (int k = 0; k < PREP_CTAS; ++k) t += dsmem_read(pj + threadIdx.x, k);
    pa[(size_t)b * D.m + threadIdx.x] = t;
  }
  cluster_sync();                          // (no CTA leaves while another reads its shared memory)
}
inline size_t prep_product_smem(int d) { return ((size_t)d + 4 + MMAX + NTHR) * sizeof(float); }
inline size_t prep_smem(int d) { return ((size_t)(NTHR / 32 + 1) * d + 4 + MMAX + NTHR) * sizeof(float); }

// The same for widths the registers do not hold (d > 2048 or d % 4 != 0) or rows off 16 bytes: one CTA per sample.
__global__ void __launch_bounds__(NTHR)
phi_prep_any_kernel(const float* __restrict__ h0, const float* __restrict__ v, const int32_t* __restrict__ rid,
                const int32_t* __restrict__ sid, float* __restrict__ rstd, float* __restrict__ pooled,
                float* __restrict__ pa, PhiDims D, float eps) {
  rte::after_previous_grid();
  extern __shared__ __align__(16) float sm[];            // rstd_s[S] then pooled_s[d]
  float* rs = sm;
  float* ps = sm + D.S;
  const int b = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const float* hb = h0 + (size_t)b * D.S * D.d;
  for (int s = warp; s < D.S; s += NTHR / 32) {
    float ss = 0.f;
    for (int c = lane; c < D.d; c += 32) { const float x = hb[(size_t)s * D.d + c]; ss += x * x; }
    ss = rte::warp_sum(ss);
    if (lane == 0) { const float r = rsqrtf(ss / (float)D.d + eps); rs[s] = r; rstd[(size_t)b * D.S + s] = r; }
  }
  __syncthreads();
  for (int c = threadIdx.x; c < D.d; c += NTHR) {
    float acc = 0.f;
    for (int s = 0; s < D.S; ++s) acc += hb[(size_t)s * D.d + c] * rs[s];
    acc /= (float)D.S;
    ps[c] = acc;
    pooled[(size_t)b * D.d + c] = acc;
  }
  __syncthreads();
  const float* v2 = v + (key_of(rid, sid, b, D.K) * 3 * D.d + D.d) * D.m;
  for (int j = warp; j < D.m; j += NTHR / 32) {
    float acc = 0.f;
    for (int c = lane; c < D.d; c += 32) acc += ps[c] * v2[(size_t)c * D.m + j];
    acc = rte::warp_sum(acc);
    if (lane == 0) pa[(size_t)b * D.m + j] = acc;
  }
}

// act[tok, j] = pa[b, j] + sum_c (h0[tok,c] * rstd[tok] * v1[c,j] + hx[tok,c] * v3[c,j])      (hx == h0 on the hot path)
__global__ void __launch_bounds__(NTHR)
phi_act_kernel(const float* __restrict__ h0, const float* __restrict__ hx, const float* __restrict__ rstd,
               const float* __restrict__ pa, const float* __restrict__ v, const int32_t* __restrict__ rid,
               const int32_t* __restrict__ sid, float* __restrict__ act, PhiDims D) {
  rte::after_previous_grid();
  __shared__ float sx[TT][CH + 1];
  __shared__ float sv1[CH][MMAX];
  __shared__ float sv3[CH][MMAX];
  const int tiles = rte::ceil_div(D.S, TT);
  const int b = blockIdx.x / tiles, tok0 = (blockIdx.x % tiles) * TT;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const float* vb = v + key_of(rid, sid, b, D.K) * 3 * D.d * D.m;
  const bool own3 = hx != h0;                        // kernel-uniform
  float acc[4][2], rs[4];
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    const int s = tok0 + warp * 4 + t;
    rs[t] = (s < D.S) ? rstd[(size_t)b * D.S + s] : 0.f;
#pragma unroll
    for (int q = 0; q < 2; ++q) { const int j = lane + 32 * q; acc[t][q] = (j < D.m) ? pa[(size_t)b * D.m + j] : 0.f; }
  }
  for (int c0 = 0; c0 < D.d; c0 += CH) {
    for (int i = threadIdx.x; i < TT * CH; i += NTHR) {
      const int t = i / CH, c = i % CH, s = tok0 + t;
      sx[t][c] = (s < D.S && c0 + c < D.d) ? h0[((size_t)b * D.S + s) * D.d + c0 + c] : 0.f;
    }
    for (int i = threadIdx.x; i < CH * D.m; i += NTHR) {
      const int c = i / D.m, j = i % D.m;
      const bool ok = c0 + c < D.d;
      sv1[c][j] = ok ? vb[(size_t)(c0 + c) * D.m + j] : 0.f;
      sv3[c][j] = ok ? vb[(size_t)(2 * D.d + c0 + c) * D.m + j] : 0.f;
    }
    __syncthreads();
#pragma unroll 4
    for (int c = 0; c < CH; ++c) {
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int j = lane + 32 * q;
        if (j < D.m) {
          const float w1 = sv1[c][j], w3 = sv3[c][j];
#pragma unroll
          for (int t = 0; t < 4; ++t) { const float x = sx[warp * 4 + t][c]; acc[t][q] += own3 ? x * rs[t] * w1 : x * (rs[t] * w1 + w3); }
        }
      }
    }
    if (own3) {                                    // the v3 slice multiplies the injected state: second sweep over its tile
      __syncthreads();
      for (int i = threadIdx.x; i < TT * CH; i += NTHR) {
        const int t = i / CH, c = i % CH, s = tok0 + t;
        sx[t][c] = (s < D.S && c0 + c < D.d) ? hx[((size_t)b * D.S + s) * D.d + c0 + c] : 0.f;
      }
      __syncthreads();
#pragma unroll 4
      for (int c = 0; c < CH; ++c) {
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const int j = lane + 32 * q;
          if (j < D.m) {
            const float w3 = sv3[c][j];
#pragma unroll
            for (int t = 0; t < 4; ++t) acc[t][q] += sx[warp * 4 + t][c] * w3;
          }
        }
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    const int s = tok0 + warp * 4 + t;
    if (s < D.S) {
#pragma unroll
      for (int q = 0; q < 2; ++q) { const int j = lane + 32 * q; if (j < D.m) act[((size_t)b * D.S + s) * D.m + j] = acc[t][q]; }
    }
  }
}

// MODE 0 (forward):  out = h + s_cfg*scale*tanh(gain*h + silu(act) @ u + bias)
// MODE 1 (backward): dupd = dout*s_cfg*scale*(1 - tanh^2);  dh0 = dout + gain*dupd   (dupd -> scratch)
template <int MODE, int MP>
__global__ void __launch_bounds__(NTHR)
phi_out_kernel(const float* __restrict__ h0, const float* __restrict__ act, const float* __restrict__ gain,
               const float* __restrict__ u, const float* __restrict__ bias, const float* __restrict__ scale,
               const int32_t* __restrict__ rid, const int32_t* __restrict__ sid, float s_cfg,
               const float* __restrict__ dout, float* __restrict__ out, float* __restrict__ dupd, PhiDims D) {
  rte::after_previous_grid();
  __shared__ float ssa[TT][MMAX];
  const int tiles = rte::ceil_div(D.S, TT);
  const int b = blockIdx.x / tiles, tok0 = (blockIdx.x % tiles) * TT;
  const size_t key = key_of(rid, sid, b, D.K);
  for (int i = threadIdx.x; i < TT * MP; i += NTHR) {           // columns past the rank are zero (they meet ur[j] = 0)
    const int t = i / MP, j = i % MP, s = tok0 + t;
    ssa[t][j] = (s < D.S && j < D.m) ? rte::silu_f(act[((size_t)b * D.S + s) * D.m + j]) : 0.f;
  }
  __syncthreads();
  const float* ub = u + key * D.m * D.d;
  for (int c = threadIdx.x; c < D.d; c += NTHR) {
    float ur[MP];                 // MP = macro rank rounded up to 32 or 64
#pragma unroll
    for (int j = 0; j < MP; ++j) ur[j] = (j < D.m) ? ub[(size_t)j * D.d + c] : 0.f;
    const float g = gain[key * D.d + c], bs = bias[key * D.d + c], sc = s_cfg * scale[key * D.d + c];
    const int t_end = min(TT, D.S - tok0);
#pragma unroll 4
    for (int t = 0; t < t_end; ++t) {
      const int s = tok0 + t;
      float low = 0.f;
#pragma unroll
      for (int j = 0; j < MP; ++j) low += ssa[t][j] * ur[j];
      const size_t idx = ((size_t)b * D.S + s) * D.d + c;
      const float h = h0[idx];
      const float th = tanhf(g * h + low + bs);
      if (MODE == 0) {
        out[idx] = h + sc * th;
      } else {
        const float du = dout[idx] * sc * (1.f - th * th);
        dupd[idx] = du;
        out[idx] = dout[idx] + g * du;
      }
    }
  }
}

// da[tok, j] = silu'(act[tok,j]) * sum_c dupd[tok,c] * u[j,c]
__global__ void __launch_bounds__(NTHR)
phi_da_kernel(const float* __restrict__ dupd, const float* __restrict__ act, const float* __restrict__ u,
              const int32_t* __restrict__ rid, const int32_t* __restrict__ sid, float* __restrict__ da, PhiDims D) {
  rte::after_previous_grid();
  __shared__ float sd[TT][CH + 1];
  __shared__ float su[MMAX][CH + 1];
  const int tiles = rte::ceil_div(D.S, TT);
  const int b = blockIdx.x / tiles, tok0 = (blockIdx.x % tiles) * TT;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const float* ub = u + key_of(rid, sid, b, D.K) * D.m * D.d;
  float acc[4][2];
#pragma unroll
  for (int t = 0; t < 4; ++t) acc[t][0] = acc[t][1] = 0.f;
  for (int c0 = 0; c0 < D.d; c0 += CH) {
    for (int i = threadIdx.x; i < TT * CH; i += NTHR) {
      const int t = i / CH, c = i % CH, s = tok0 + t;
      sd[t][c] = (s < D.S && c0 + c < D.d) ? dupd[((size_t)b * D.S + s) * D.d + c0 + c] : 0.f;
    }
    for (int i = threadIdx.x; i < D.m * CH; i += NTHR) {
      const int j = i / CH, c = i % CH;
      su[j][c] = (c0 + c < D.d) ? ub[(size_t)j * D.d + c0 + c] : 0.f;
    }
    __syncthreads();
#pragma unroll 4
    for (int c = 0; c < CH; ++c) {
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int j = lane + 32 * q;
        if (j < D.m) {
          const float w = su[j][c];
#pragma unroll
          for (int t = 0; t < 4; ++t) acc[t][q] += sd[warp * 4 + t][c] * w;
        }
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    const int s = tok0 + warp * 4 + t;
    if (s < D.S) {
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int j = lane + 32 * q;
        if (j < D.m) {
          const size_t idx = ((size_t)b * D.S + s) * D.m + j;
          const float a = act[idx], sg = rte::sigmoid_f(a);
          da[idx] = acc[t][q] * sg * (1.f + a * (1.f - sg));
        }
      }
    }
  }
}

// ---- Tensor-core versions of the two data-gradient products (taken when d % 8 == 0): TF32 mma with the 3xTF32
// error compensation, so results stay at fp32 accuracy.
// Operand fragments of mma.m16n8k8 come straight from global memory: a quad of lanes reads 16 contiguous bytes of a
// row and the two k-halves of a step complete the 32-byte sector, so no shared-memory staging (and no barrier) is
// needed; the per-key weights stay in L1/L2.  Warp tile: 16 tokens; a CTA covers TT = 32 tokens of one sample.
__device__ __forceinline__ uint32_t to_tf32(float x) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return r;
}

__device__ __forceinline__ void mma_tf32(float (&c)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// fp32-accurate product from TF32 pieces: x = hi + lo with both representable in TF32, and
// a*b ~= a_lo*b_hi + a_hi*b_lo + a_hi*b_hi (the dropped lo*lo term is below fp32 rounding).
__device__ __forceinline__ void split_tf32(float x, uint32_t& hi, uint32_t& lo) {
  hi = to_tf32(x);
  lo = to_tf32(x - __uint_as_float(hi));
}

__device__ __forceinline__ void mma_3xtf32(float (&c)[4], const uint32_t (&ah)[4], const uint32_t (&al)[4],
                                           const uint32_t (&bh)[2], const uint32_t (&bl)[2]) {
  mma_tf32(c, al, bh);
  mma_tf32(c, ah, bl);
  mma_tf32(c, ah, bh);
}

// The kernels read their operands with 16-byte loads.  Inside a chunk of 32 reduction indices the mma's logical k-slot
// (step s, slot t or t+4) is mapped to a physical index, the same for A and B, so the sum is unchanged.  Where the
// reduction runs over columns (da, act) it is 4t+s or 16+4t+s: a quad reads 64 contiguous bytes per load, whole sectors
// (with 8t+s the two loads each touched every sector of the line).  Where it runs over the rank (out, dz) it is 8t+s or
// 8t+4+s.
struct Frag8 { float4 lo, hi; };     // the values of slots t and t+4, four steps each
__device__ __forceinline__ Frag8 load8(const float* p, bool ok) {
  Frag8 f;
  if (ok) { f.lo = *reinterpret_cast<const float4*>(p); f.hi = *reinterpret_cast<const float4*>(p + 4); }
  else { f.lo = make_float4(0.f, 0.f, 0.f, 0.f); f.hi = f.lo; }
  return f;
}
__device__ __forceinline__ float pick(const float4& v, int s) { return s == 0 ? v.x : s == 1 ? v.y : s == 2 ? v.z : v.w; }

__device__ __forceinline__ Frag8 load_k32(const float* row, int t, bool ok) {
  Frag8 f;
  if (ok) { f.lo = *reinterpret_cast<const float4*>(row + 4 * t); f.hi = *reinterpret_cast<const float4*>(row + 16 + 4 * t); }
  else { f.lo = make_float4(0.f, 0.f, 0.f, 0.f); f.hi = f.lo; }
  return f;
}
struct SplitA { uint32_t h[4][4], l[4][4]; };         // [step][fragment register]
__device__ __forceinline__ SplitA split_a(const Frag8& x0, const Frag8& x1) {
  SplitA a;
#pragma unroll
  for (int s = 0; s < 4; ++s) {
    split_tf32(pick(x0.lo, s), a.h[s][0], a.l[s][0]);
    split_tf32(pick(x1.lo, s), a.h[s][1], a.l[s][1]);
    split_tf32(pick(x0.hi, s), a.h[s][2], a.l[s][2]);
    split_tf32(pick(x1.hi, s), a.h[s][3], a.l[s][3]);
  }
  return a;
}
__device__ __forceinline__ void mma_chunk(float (&c)[4], const SplitA& a, const Frag8& w) {
#pragma unroll
  for (int s = 0; s < 4; ++s) {
    uint32_t f[2], fl[2];
    split_tf32(pick(w.lo, s), f[0], fl[0]);
    split_tf32(pick(w.hi, s), f[1], fl[1]);
    mma_3xtf32(c, a.h[s], a.l[s], f, fl);
  }
}

// The two products of 32 tokens with a key's weights over all d columns (d % 32 == 0): warps = 2 token tiles x 4 slices of
// the reduction (chunks of 32 columns, every fourth one), each with all ranks (NT tiles of 8), so a token's values are
// loaded and split once; the slices meet in shared memory in slice order.  (With the ranks divided over the warps instead,
// every warp read and split every token: bound by L1.)
constexpr int KSLICES = 4;
template <int NT>
__device__ __forceinline__ bool sum_slices(float (&acc)[NT][4], float (&red)[KSLICES - 1][2][NT * 4][32], int mt, int slice, int lane) {
  if (slice > 0) {
#pragma unroll
    for (int i = 0; i < NT; ++i)
#pragma unroll
      for (int e = 0; e < 4; ++e) red[slice - 1][mt][4 * i + e][lane] = acc[i][e];
  }
  __syncthreads();
  if (slice > 0) return false;
#pragma unroll
  for (int k = 0; k < KSLICES - 1; ++k)
#pragma unroll
    for (int i = 0; i < NT; ++i)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[i][e] += red[k][mt][4 * i + e][lane];
  return true;
}

// da[tok, j] = silu'(act[tok,j]) * sum_c dupd[tok,c] * u[j,c]:  M = tokens, N = rank, K = d.  32 x 256 x 1024, rank 32:
// 41 -> 27 us in the step.
template <int NT>
__global__ void __launch_bounds__(NTHR, 2)
phi_da_mma_kernel(const float* __restrict__ dupd, const float* __restrict__ act, const float* __restrict__ u,
                  const int32_t* __restrict__ rid, const int32_t* __restrict__ sid, float* __restrict__ da, PhiDims D) {
  rte::after_previous_grid();
  __shared__ float red[KSLICES - 1][2][NT * 4][32];
  const int tiles = rte::ceil_div(D.S, TT);
  const int b = blockIdx.x / tiles, tok0 = (blockIdx.x % tiles) * TT;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  const int mt = warp & 1, slice = warp >> 1;
  const float* ub = u + key_of(rid, sid, b, D.K) * D.m * D.d;
  const int r0 = tok0 + mt * 16 + g, r1 = r0 + 8;
  const bool ok0 = r0 < D.S, ok1 = r1 < D.S;
  const float* a0p = dupd + ((size_t)b * D.S + (ok0 ? r0 : 0)) * D.d;
  const float* a1p = dupd + ((size_t)b * D.S + (ok1 ? r1 : 0)) * D.d;
  float acc[NT][4];
#pragma unroll
  for (int i = 0; i < NT; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
  for (int k0 = 32 * slice; k0 < D.d; k0 += 32 * KSLICES) {
    const Frag8 x0 = load_k32(a0p + k0, t, ok0), x1 = load_k32(a1p + k0, t, ok1);
    Frag8 w[NT <= 4 ? NT : 1];
    if constexpr (NT <= 4) {                          // all weights requested ahead of the first product
#pragma unroll
      for (int i = 0; i < NT; ++i) w[i] = load_k32(ub + (size_t)min(8 * i + g, D.m - 1) * D.d + k0, t, 8 * i + g < D.m);
    }
    const SplitA a = split_a(x0, x1);
#pragma unroll
    for (int i = 0; i < NT; ++i) {
      if constexpr (NT <= 4) mma_chunk(acc[i], a, w[i]);
      else mma_chunk(acc[i], a, load_k32(ub + (size_t)min(8 * i + g, D.m - 1) * D.d + k0, t, 8 * i + g < D.m));
    }
  }
  if (!sum_slices<NT>(acc, red, mt, slice, lane)) return;
  auto put = [&](int row, int col, float x) {
    if (row < D.S && col < D.m) {
      const size_t idx = ((size_t)b * D.S + row) * D.m + col;
      const float av = act[idx], sg = rte::sigmoid_f(av);
      da[idx] = x * sg * (1.f + av * (1.f - sg));
    }
  };
#pragma unroll
  for (int i = 0; i < NT; ++i) {
    const int col = 8 * i + 2 * t;
    put(r0, col, acc[i][0]); put(r0, col + 1, acc[i][1]); put(r1, col, acc[i][2]); put(r1, col + 1, acc[i][3]);
  }
}

// ---- Forward products on tensor cores.  They need the reduction index contiguous per output column, i.e. the
// TRANSPOSED parameters: wt = vt [m][keys*3d] (vt[j][key*3d + c] = v[key][c][j]) followed by
// ut [d][keys*m] (ut[c][key*m + j] = u[key][j][c]), refreshed once per step by rte_macro_phi_prepare.

// act[tok, j] = pa[b, j] + rstd[tok] * (h0 @ v1)[tok, j] + (hx @ v3)[tok, j]:  M = tokens, N = rank, K = d.  With hx == h0,
// the hot path, both products share the token fragments.  32 x 256 x 1024, rank 32: 85 -> 47 us in the step.
template <int NT, bool OWN3>
__global__ void __launch_bounds__(NTHR, NT <= 4 ? 2 : 1)
phi_act_mma_kernel(const float* __restrict__ h0, const float* __restrict__ hx, const float* __restrict__ rstd,
                   const float* __restrict__ pa, const float* __restrict__ vt, long long vt_ld,
                   const int32_t* __restrict__ rid, const int32_t* __restrict__ sid, float* __restrict__ act, PhiDims D) {
  rte::after_previous_grid();
  __shared__ float red[KSLICES - 1][2][NT * 4][32];
  const int tiles = rte::ceil_div(D.S, TT);
  const int b = blockIdx.x / tiles, tok0 = (blockIdx.x % tiles) * TT;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  const int mt = warp & 1, slice = warp >> 1;
  const float* vk = vt + key_of(rid, sid, b, D.K) * 3 * D.d;
  const int r0 = tok0 + mt * 16 + g, r1 = r0 + 8;
  const bool ok0 = r0 < D.S, ok1 = r1 < D.S;
  const size_t row0 = ((size_t)b * D.S + (ok0 ? r0 : 0)) * D.d, row1 = ((size_t)b * D.S + (ok1 ? r1 : 0)) * D.d;
  float p1[NT][4], p3[NT][4];
#pragma unroll
  for (int i = 0; i < NT; ++i)
#pragma unroll
    for (int e = 0; e < 4; ++e) p1[i][e] = p3[i][e] = 0.f;
#pragma unroll 1
  for (int k0 = 32 * slice; k0 < D.d; k0 += 32 * KSLICES) {
    const SplitA a = split_a(load_k32(h0 + row0 + k0, t, ok0), load_k32(h0 + row1 + k0, t, ok1));
#pragma unroll
    for (int i = 0; i < NT; ++i) mma_chunk(p1[i], a, load_k32(vk + (size_t)min(8 * i + g, D.m - 1) * vt_ld + k0, t, 8 * i + g < D.m));
    if constexpr (OWN3) {
      const SplitA c = split_a(load_k32(hx + row0 + k0, t, ok0), load_k32(hx + row1 + k0, t, ok1));
#pragma unroll
      for (int i = 0; i < NT; ++i) mma_chunk(p3[i], c, load_k32(vk + (size_t)min(8 * i + g, D.m - 1) * vt_ld + 2 * D.d + k0, t, 8 * i + g < D.m));
    } else {
#pragma unroll
      for (int i = 0; i < NT; ++i) mma_chunk(p3[i], a, load_k32(vk + (size_t)min(8 * i + g, D.m - 1) * vt_ld + 2 * D.d + k0, t, 8 * i + g < D.m));
    }
  }
  const float rs0 = ok0 ? rstd[(size_t)b * D.S + r0] : 0.f, rs1 = ok1 ? rstd[(size_t)b * D.S + r1] : 0.f;
#pragma unroll
  for (int i = 0; i < NT; ++i) {
    p1[i][0] = rs0 * p1[i][0] + p3[i][0]; p1[i][1] = rs0 * p1[i][1] + p3[i][1];
    p1[i][2] = rs1 * p1[i][2] + p3[i][2]; p1[i][3] = rs1 * p1[i][3] + p3[i][3];
  }
  if (!sum_slices<NT>(p1, red, mt, slice, lane)) return;
  auto put = [&](int row, int col, float x) {
    if (row < D.S && col < D.m) act[((size_t)b * D.S + row) * D.m + col] = pa[(size_t)b * D.m + col] + x;
  };
#pragma unroll
  for (int i = 0; i < NT; ++i) {
    const int col = 8 * i + 2 * t;
    put(r0, col, p1[i][0]); put(r0, col + 1, p1[i][1]); put(r1, col, p1[i][2]); put(r1, col + 1, p1[i][3]);
  }
}

// MODE 0 (forward):  out = h + s_cfg*scale*tanh(gain*h + silu(act) @ u + bias)
// MODE 1 (backward): dupd = dout*s_cfg*scale*(1 - tanh^2);  out (= dh0) = dout + gain*dupd
// M = tokens, N = d, K = rank (d % 32 == 0, rank % 4 == 0); warp layout, operand permutations and float4 epilogue
// as in phi_dz_mma_kernel; the A operand is silu(act) of the warp's 16 tokens, held in registers.
template <int MODE, int KC>
__global__ void __launch_bounds__(NTHR, KC == 1 ? 2 : 1)
phi_out_mma_kernel(const float* __restrict__ h0, const float* __restrict__ act, const float* __restrict__ gain,
                   const float* __restrict__ ut, long long ut_ld, const float* __restrict__ bias,
                   const float* __restrict__ scale, const int32_t* __restrict__ rid, const int32_t* __restrict__ sid,
                   float s_cfg, const float* __restrict__ dout, float* __restrict__ out, float* __restrict__ dupd, PhiDims D) {
  rte::after_previous_grid();
  const int tiles = rte::ceil_div(D.S, TT);
  const int b = blockIdx.x / tiles, tok0 = (blockIdx.x % tiles) * TT;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  const int mt = warp & 1, cq = warp >> 1;
  const size_t key = key_of(rid, sid, b, D.K);
  const float* ub = ut + key * D.m;                 // row c of this key's u^T: ub + c * ut_ld
  const int r0 = tok0 + mt * 16 + g, r1 = r0 + 8;
  const bool ok0 = r0 < D.S, ok1 = r1 < D.S;
  const size_t row0 = (size_t)b * D.S + (ok0 ? r0 : 0), row1 = (size_t)b * D.S + (ok1 ? r1 : 0);
  uint32_t ah[KC][4][4], al[KC][4][4];
#pragma unroll
  for (int ch = 0; ch < KC; ++ch) {
    const int k = 32 * ch + 8 * t;
    Frag8 y0 = load8(act + row0 * D.m + k, ok0 && k + 8 <= D.m), y1 = load8(act + row1 * D.m + k, ok1 && k + 8 <= D.m);
    if (k < D.m && k + 8 > D.m) {
      if (ok0) y0.lo = *reinterpret_cast<const float4*>(act + row0 * D.m + k);
      if (ok1) y1.lo = *reinterpret_cast<const float4*>(act + row1 * D.m + k);
    }
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      const bool in_lo = k + s < D.m, in_hi = k + 4 + s < D.m;      // silu(0) = 0 anyway; keep padded slots exact zeros
      split_tf32(in_lo ? rte::silu_f(pick(y0.lo, s)) : 0.f, ah[ch][s][0], al[ch][s][0]);
      split_tf32(in_lo ? rte::silu_f(pick(y1.lo, s)) : 0.f, ah[ch][s][1], al[ch][s][1]);
      split_tf32(in_hi ? rte::silu_f(pick(y0.hi, s)) : 0.f, ah[ch][s][2], al[ch][s][2]);
      split_tf32(in_hi ? rte::silu_f(pick(y1.hi, s)) : 0.f, ah[ch][s][3], al[ch][s][3]);
    }
  }
  const int n_blocks = D.d / 32;
  const int pc0 = 8 * (g >> 1) + (g & 1);
  const float* gk = gain + key * D.d;
  const float* bk = bias + key * D.d;
  const float* sk = scale + key * D.d;
  for (int nb = cq; nb < n_blocks; nb += 4) {
    const int cb = nb * 32, col = cb + 8 * t;
    float c[4][4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      c[j][0] = c[j][1] = c[j][2] = c[j][3] = 0.f;
      const float* wr = ub + (size_t)(cb + pc0 + 2 * j) * ut_ld;
#pragma unroll
      for (int ch = 0; ch < KC; ++ch) {
        const int k = 32 * ch + 8 * t;
        Frag8 f = load8(wr + k, k + 8 <= D.m);
        if (k < D.m && k + 8 > D.m) f.lo = *reinterpret_cast<const float4*>(wr + k);
#pragma unroll
        for (int s = 0; s < 4; ++s) {
          uint32_t fh[2], fl[2];
          split_tf32(pick(f.lo, s), fh[0], fl[0]);
          split_tf32(pick(f.hi, s), fh[1], fl[1]);
          mma_3xtf32(c[j], ah[ch][s], al[ch][s], fh, fl);
        }
      }
    }
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      if (!(half ? ok1 : ok0)) continue;
      const size_t row = half ? row1 : row0;
      const float low[8] = {c[0][2 * half], c[0][2 * half + 1], c[1][2 * half], c[1][2 * half + 1],
                            c[2][2 * half], c[2][2 * half + 1], c[3][2 * half], c[3][2 * half + 1]};
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const size_t idx = row * D.d + col + 4 * q;
        const float4 h = *reinterpret_cast<const float4*>(h0 + idx);
        const float4 gv = *reinterpret_cast<const float4*>(gk + col + 4 * q);
        const float4 bv = *reinterpret_cast<const float4*>(bk + col + 4 * q);
        float4 sc = *reinterpret_cast<const float4*>(sk + col + 4 * q);
        sc.x *= s_cfg; sc.y *= s_cfg; sc.z *= s_cfg; sc.w *= s_cfg;
        const float t0 = tanhf(gv.x * h.x + low[4 * q] + bv.x), t1 = tanhf(gv.y * h.y + low[4 * q + 1] + bv.y);
        const float t2 = tanhf(gv.z * h.z + low[4 * q + 2] + bv.z), t3 = tanhf(gv.w * h.w + low[4 * q + 3] + bv.w);
        if (MODE == 0) {
          *reinterpret_cast<float4*>(out + idx) = make_float4(h.x + sc.x * t0, h.y + sc.y * t1, h.z + sc.z * t2, h.w + sc.w * t3);
        } else {
          const float4 dv = *reinterpret_cast<const float4*>(dout + idx);
          const float4 du = make_float4(dv.x * sc.x * (1.f - t0 * t0), dv.y * sc.y * (1.f - t1 * t1),
                                        dv.z * sc.z * (1.f - t2 * t2), dv.w * sc.w * (1.f - t3 * t3));
          *reinterpret_cast<float4*>(dupd + idx) = du;
          *reinterpret_cast<float4*>(out + idx) = make_float4(dv.x + gv.x * du.x, dv.y + gv.y * du.y, dv.z + gv.z * du.z, dv.w + gv.w * du.w);
        }
      }
    }
  }
}

// Per-sample parameter gradients, all of them in one launch over the tokens of a sample (M = columns c, K = tokens s):
//   pu[b][j, c]  = sum_s silu(act[s,j]) * dupd[s,c],   pg[b][c] = sum_s dupd[s,c] * h0[s,c],   pb[b][c] = sum_s dupd[s,c]
//   pv[b][c', j]: c' <  d  sum_s h0[s,c]*rstd[s] * da[s,j]
//                 c' < 2d  pooled[b,c] * sum_s da[s,j]
//                 else     sum_s hx[s,c] * da[s,j]                  (hx == h0 on the hot path: the operand is split once)
// 3xTF32 products: a warp owns 16 columns and all ranks (NT tiles of 8); its A operand is the transpose of [token, column]
// rows read straight from global memory (eight neighbouring columns per token: whole sectors), da and silu(act) of
// PG_TOK tokens at a time are staged in shared memory for the CTA's eight warps.  The scalar kernels this replaces were
// bound by four shared-memory reads per product term: 32 x 256 x 1024, rank 32: 307 -> 92 us in the step.
constexpr int PG_TOK = 64;

template <int NT, bool OWN3>
__global__ void __launch_bounds__(NTHR, NT <= 4 ? 2 : 1)
phi_param_grads_kernel(const float* __restrict__ h0, const float* __restrict__ hx, const float* __restrict__ rstd, const float* __restrict__ pooled,
                       const float* __restrict__ act, const float* __restrict__ dupd, const float* __restrict__ da, float* __restrict__ pu,
                       float* __restrict__ pg, float* __restrict__ pb, float* __restrict__ pv, PhiDims D) {
  rte::after_previous_grid();
  constexpr int LD = 8 * NT + 8;                                       // (+8: the four tokens of a fragment fall into different banks)
  __shared__ float sda[PG_TOK * LD], ssa[PG_TOK * LD], srs[PG_TOK];
  __shared__ float part[NTHR], stot[8 * NT];                           // column sums of da: per thread, then whole
  const int cblocks = rte::ceil_div(D.d, 128);
  const int b = blockIdx.x / cblocks, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  const int c0 = (blockIdx.x % cblocks) * 128 + warp * 16 + g, c1 = c0 + 8;      // this lane's rows of the products
  const bool ok0 = c0 < D.d, ok1 = c1 < D.d;
  const size_t base = (size_t)b * D.S * D.d;
  float uu[NT][4], v1[NT][4], v3[NT][4];
#pragma unroll
  for (int i = 0; i < NT; ++i)
#pragma unroll
    for (int e = 0; e < 4; ++e) uu[i][e] = v1[i][e] = v3[i][e] = 0.f;
  float ag0 = 0.f, ag1 = 0.f, ab0 = 0.f, ab1 = 0.f, colsum = 0.f;
  for (int s0 = 0; s0 < D.S; s0 += PG_TOK) {
    const int n = min(PG_TOK, D.S - s0);
    __syncthreads();
    for (int i = threadIdx.x; i < PG_TOK * 8 * NT; i += NTHR) {
      const int s = i / (8 * NT), j = i % (8 * NT);
      const bool in = s < n && j < D.m;
      const size_t at = ((size_t)b * D.S + s0 + s) * D.m + j;
      sda[s * LD + j] = in ? da[at] : 0.f;
      ssa[s * LD + j] = in ? rte::silu_f(act[at]) : 0.f;
    }
    for (int i = threadIdx.x; i < PG_TOK; i += NTHR) srs[i] = i < n ? rstd[(size_t)b * D.S + s0 + i] : 0.f;
    __syncthreads();
    for (int s = threadIdx.x / (8 * NT); s < n; s += NTHR / (8 * NT)) colsum += sda[s * LD + threadIdx.x % (8 * NT)];
#pragma unroll 2
    for (int k = 0; k < n; k += 8) {
      const int sa = s0 + k + t, sb = sa + 4;
      const bool ta = sa < D.S, tb = sb < D.S;
      float h[4], du[4], x3[4];
      const size_t ra = base + (size_t)sa * D.d, rb = base + (size_t)sb * D.d;
      h[0] = ta && ok0 ? h0[ra + c0] : 0.f;  h[1] = ta && ok1 ? h0[ra + c1] : 0.f;
      h[2] = tb && ok0 ? h0[rb + c0] : 0.f;  h[3] = tb && ok1 ? h0[rb + c1] : 0.f;
      du[0] = ta && ok0 ? dupd[ra + c0] : 0.f;  du[1] = ta && ok1 ? dupd[ra + c1] : 0.f;
      du[2] = tb && ok0 ? dupd[rb + c0] : 0.f;  du[3] = tb && ok1 ? dupd[rb + c1] : 0.f;
      if constexpr (OWN3) {
        x3[0] = ta && ok0 ? hx[ra + c0] : 0.f;  x3[1] = ta && ok1 ? hx[ra + c1] : 0.f;
        x3[2] = tb && ok0 ? hx[rb + c0] : 0.f;  x3[3] = tb && ok1 ? hx[rb + c1] : 0.f;
      }
      ag0 += du[0] * h[0] + du[2] * h[2];
      ag1 += du[1] * h[1] + du[3] * h[3];
      ab0 += du[0] + du[2];
      ab1 += du[1] + du[3];
      const float rsa = srs[k + t], rsb = srs[k + t + 4];
      uint32_t dh[4], dl[4], h1[4], l1[4], h3[4], l3[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        split_tf32(du[e], dh[e], dl[e]);
        split_tf32(h[e] * (e < 2 ? rsa : rsb), h1[e], l1[e]);
        if constexpr (OWN3) split_tf32(x3[e], h3[e], l3[e]);
        else split_tf32(h[e], h3[e], l3[e]);
      }
#pragma unroll
      for (int i = 0; i < NT; ++i) {
        uint32_t fh[2], fl[2];
        split_tf32(ssa[(k + t) * LD + 8 * i + g], fh[0], fl[0]);
        split_tf32(ssa[(k + t + 4) * LD + 8 * i + g], fh[1], fl[1]);
        mma_3xtf32(uu[i], dh, dl, fh, fl);
        split_tf32(sda[(k + t) * LD + 8 * i + g], fh[0], fl[0]);
        split_tf32(sda[(k + t + 4) * LD + 8 * i + g], fh[1], fl[1]);
        mma_3xtf32(v1[i], h1, l1, fh, fl);
        mma_3xtf32(v3[i], h3, l3, fh, fl);
      }
    }
  }
  part[threadIdx.x] = colsum;
  __syncthreads();
  if (threadIdx.x < 8 * NT) {
    float a = 0.f;
#pragma unroll
    for (int k = 0; k < NTHR / (8 * NT); ++k) a += part[k * 8 * NT + threadIdx.x];
    stot[threadIdx.x] = a;
  }
  __syncthreads();
  ag0 += __shfl_xor_sync(0xffffffffu, ag0, 1); ag0 += __shfl_xor_sync(0xffffffffu, ag0, 2);
  ag1 += __shfl_xor_sync(0xffffffffu, ag1, 1); ag1 += __shfl_xor_sync(0xffffffffu, ag1, 2);
  ab0 += __shfl_xor_sync(0xffffffffu, ab0, 1); ab0 += __shfl_xor_sync(0xffffffffu, ab0, 2);
  ab1 += __shfl_xor_sync(0xffffffffu, ab1, 1); ab1 += __shfl_xor_sync(0xffffffffu, ab1, 2);
  if (t == 0 && ok0) { pg[(size_t)b * D.d + c0] = ag0; pb[(size_t)b * D.d + c0] = ab0; }
  if (t == 0 && ok1) { pg[(size_t)b * D.d + c1] = ag1; pb[(size_t)b * D.d + c1] = ab1; }
  float* pvb = pv + (size_t)b * 3 * D.d * D.m;
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    const int c = half ? c1 : c0;
    if (!(half ? ok1 : ok0)) continue;
    const float pool = pooled[(size_t)b * D.d + c];
#pragma unroll
    for (int i = 0; i < NT; ++i)
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int j = 8 * i + 2 * t + q;
        if (j < D.m) {
          pu[((size_t)b * D.m + j) * D.d + c] = uu[i][2 * half + q];
          pvb[(size_t)c * D.m + j] = v1[i][2 * half + q];
          pvb[(size_t)(D.d + c) * D.m + j] = pool * stot[j];
          pvb[(size_t)(2 * D.d + c) * D.m + j] = v3[i][2 * half + q];
        }
      }
  }
}

// sda[b, j] = sum_s da[b,s,j]  ->  dpool[b, c] = (1/S) * sum_j sda[b,j] * v2[c,j]      (a CTA per sample and 256 columns)
__global__ void __launch_bounds__(NTHR)
phi_dpool_kernel(const float* __restrict__ da, const float* __restrict__ v, const int32_t* __restrict__ rid,
                 const int32_t* __restrict__ sid, float* __restrict__ dpool, PhiDims D) {
  rte::after_previous_grid();
  __shared__ float part[NTHR], ssum[MMAX];
  const int cblocks = rte::ceil_div(D.d, NTHR);
  const int b = blockIdx.x / cblocks, c = (blockIdx.x % cblocks) * NTHR + threadIdx.x;
  const int mw = D.m <= 32 ? 32 : 64, j = threadIdx.x % mw, groups = NTHR / mw;
  float a = 0.f;
  if (j < D.m) {
#pragma unroll 8
    for (int s = threadIdx.x / mw; s < D.S; s += groups) a += da[((size_t)b * D.S + s) * D.m + j];
  }
  part[threadIdx.x] = a;
  __syncthreads();
  if (threadIdx.x < D.m) {
    a = 0.f;
    for (int k = 0; k < groups; ++k) a += part[k * mw + threadIdx.x];
    ssum[threadIdx.x] = a;
  }
  __syncthreads();
  if (c >= D.d) return;
  const float* v2 = v + (key_of(rid, sid, b, D.K) * 3 * D.d + D.d + c) * D.m;
  a = 0.f;
  if (D.m % 4 == 0 && (reinterpret_cast<uintptr_t>(v) & 15) == 0) {
#pragma unroll 8
    for (int q = 0; q < D.m; q += 4) {
      const float4 w = *reinterpret_cast<const float4*>(v2 + q);
      a += ssum[q] * w.x + ssum[q + 1] * w.y + ssum[q + 2] * w.z + ssum[q + 3] * w.w;
    }
  } else {
    for (int q = 0; q < D.m; ++q) a += ssum[q] * v2[q];
  }
  dpool[(size_t)b * D.d + c] = a / (float)D.S;
}

// dhx[tok,:] += da @ v3^T;  dh0[tok,:] += rmsnorm_backward(da @ v1^T + dpool[b,:])     (one warp per token; dhx may be dh0)
__global__ void __launch_bounds__(NTHR)
phi_dz_kernel(const float* __restrict__ h0, const float* __restrict__ rstd, const float* __restrict__ da,
              const float* __restrict__ dpool, const float* __restrict__ v, const int32_t* __restrict__ rid,
              const int32_t* __restrict__ sid, float* dh0, float* dhx, PhiDims D) {
  rte::after_previous_grid();
  __shared__ float sv1[CH][MMAX + 1];
  __shared__ float sv3[CH][MMAX + 1];
  __shared__ float sda[TT][MMAX];
  const int tiles = rte::ceil_div(D.S, TT);
  const int b = blockIdx.x / tiles, tok0 = (blockIdx.x % tiles) * TT;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const float* vb = v + key_of(rid, sid, b, D.K) * 3 * D.d * D.m;
  for (int i = threadIdx.x; i < TT * D.m; i += NTHR) {
    const int t = i / D.m, j = i % D.m, s = tok0 + t;
    sda[t][j] = (s < D.S) ? da[((size_t)b * D.S + s) * D.m + j] : 0.f;
  }
  // pass 1: dh0 += da @ v3^T and the row dot products <dn, xhat>; pass 2 recomputes dn per chunk
  float dot[4] = {0.f, 0.f, 0.f, 0.f};
  const int nchunks = rte::ceil_div(D.d, CH);
  for (int ch = 0; ch < nchunks; ++ch) {
    const int c0 = ch * CH;
    __syncthreads();
    for (int i = threadIdx.x; i < CH * D.m; i += NTHR) {
      const int c = i / D.m, j = i % D.m;
      const bool ok = c0 + c < D.d;
      sv1[c][j] = ok ? vb[(size_t)(c0 + c) * D.m + j] : 0.f;
      sv3[c][j] = ok ? vb[(size_t)(2 * D.d + c0 + c) * D.m + j] : 0.f;
    }
    __syncthreads();
    float a1[4][2], a3[4][2];
#pragma unroll
    for (int t = 0; t < 4; ++t) a1[t][0] = a1[t][1] = a3[t][0] = a3[t][1] = 0.f;
#pragma unroll 4
    for (int j = 0; j < D.m; ++j) {
      const float w1a = sv1[lane][j], w1b = sv1[lane + 32][j], w3a = sv3[lane][j], w3b = sv3[lane + 32][j];
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const float dv = sda[warp * 4 + t][j];
        a1[t][0] += dv * w1a; a1[t][1] += dv * w1b;
        a3[t][0] += dv * w3a; a3[t][1] += dv * w3b;
      }
    }
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int cl = lane + 32 * q, c = c0 + cl;
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const int s = tok0 + warp * 4 + t;
        if (s < D.S && c < D.d) {
          const size_t idx = ((size_t)b * D.S + s) * D.d + c;
          const float dnv = a1[t][q] + dpool[(size_t)b * D.d + c];
          dhx[idx] += a3[t][q];
          dot[t] += dnv * h0[idx] * rstd[(size_t)b * D.S + s];
        }
      }
    }
  }
#pragma unroll
  for (int t = 0; t < 4; ++t) dot[t] = rte::warp_sum(dot[t]) / (float)D.d;
  // second pass: recompute dn per chunk and finish dx = rstd * (dn - xhat * dot)
  for (int ch = 0; ch < nchunks; ++ch) {
    const int c0 = ch * CH;
    __syncthreads();
    for (int i = threadIdx.x; i < CH * D.m; i += NTHR) {
      const int c = i / D.m, j = i % D.m;
      sv1[c][j] = (c0 + c < D.d) ? vb[(size_t)(c0 + c) * D.m + j] : 0.f;
    }
    __syncthreads();
    float a1[4][2];
#pragma unroll
    for (int t = 0; t < 4; ++t) a1[t][0] = a1[t][1] = 0.f;
#pragma unroll 4
    for (int j = 0; j < D.m; ++j) {
      const float w1a = sv1[lane][j], w1b = sv1[lane + 32][j];
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const float dv = sda[warp * 4 + t][j];
        a1[t][0] += dv * w1a; a1[t][1] += dv * w1b;
      }
    }
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int cl = lane + 32 * q, c = c0 + cl;
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const int s = tok0 + warp * 4 + t;
        if (s < D.S && c < D.d) {
          const size_t idx = ((size_t)b * D.S + s) * D.d + c;
          const float r = rstd[(size_t)b * D.S + s];
          const float dnv = a1[t][q] + dpool[(size_t)b * D.d + c];
          dh0[idx] += r * (dnv - h0[idx] * r * dot[t]);
        }
      }
    }
  }
}

// dhx[tok,:] += da @ v3^T;  dh0[tok,:] += rmsnorm_backward(da @ v1^T + dpool[b,:])  (dhx may be dh0):  M = tokens, N = d,
// K = rank (tensor-core form;
// d % 32 == 0, rank % 4 == 0).  Eight warps = 2 token tiles x 4 column groups; a group takes 32-column blocks
// cq, cq+4, ...  The A operand (16 tokens x rank) lives in registers (KC chunks of 32 rank indices, permuted as
// above).  Output columns are permuted too: mma tile j of a block holds, for lane t, the physical columns
// 8t+2j and 8t+2j+1, so a lane owns the eight consecutive columns [8t, 8t+8) of its two rows and the epilogue moves
// float4.  Pass 1 forms the row dot products <dn, xhat>; pass 2 recomputes the small products and finishes with one
// read-modify-write of dh0.
template <int KC>
__global__ void __launch_bounds__(NTHR, KC == 1 ? 2 : 1)
phi_dz_mma_kernel(const float* __restrict__ h0, const float* __restrict__ rstd, const float* __restrict__ da,
                  const float* __restrict__ dpool, const float* __restrict__ v, const int32_t* __restrict__ rid,
                  const int32_t* __restrict__ sid, float* dh0, float* dhx, const float* __restrict__ row_add, int parts, long long part_stride,
                  __nv_bfloat16* __restrict__ dh16, PhiDims D) {
  rte::after_previous_grid();
  __shared__ float sdot[TT][4];
  const int tiles = rte::ceil_div(D.S, TT);
  const int b = blockIdx.x / tiles, tok0 = (blockIdx.x % tiles) * TT;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  const int mt = warp & 1, cq = warp >> 1;
  const float* v1 = v + key_of(rid, sid, b, D.K) * 3 * D.d * D.m;
  const float* v3 = v1 + (size_t)2 * D.d * D.m;
  const int r0 = tok0 + mt * 16 + g, r1 = r0 + 8;
  const bool ok0 = r0 < D.S, ok1 = r1 < D.S;
  const size_t row0 = (size_t)b * D.S + (ok0 ? r0 : 0), row1 = (size_t)b * D.S + (ok1 ? r1 : 0);
  uint32_t ah[KC][4][4], al[KC][4][4];          // [chunk][k-step][fragment register]
#pragma unroll
  for (int ch = 0; ch < KC; ++ch) {
    const int k = 32 * ch + 8 * t;
    const bool in = k < D.m;                     // rank % 4 == 0 and 8-wide pieces: guard each half
    const Frag8 x0 = load8(da + row0 * D.m + k, ok0 && in && k + 8 <= D.m);
    const Frag8 x1 = load8(da + row1 * D.m + k, ok1 && in && k + 8 <= D.m);
    Frag8 y0 = x0, y1 = x1;
    if (in && k + 8 > D.m) {                     // only the first four of the eight exist
      if (ok0) y0.lo = *reinterpret_cast<const float4*>(da + row0 * D.m + k);
      if (ok1) y1.lo = *reinterpret_cast<const float4*>(da + row1 * D.m + k);
    }
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      split_tf32(pick(y0.lo, s), ah[ch][s][0], al[ch][s][0]);
      split_tf32(pick(y1.lo, s), ah[ch][s][1], al[ch][s][1]);
      split_tf32(pick(y0.hi, s), ah[ch][s][2], al[ch][s][2]);
      split_tf32(pick(y1.hi, s), ah[ch][s][3], al[ch][s][3]);
    }
  }
  const float rs0 = ok0 ? rstd[row0] : 0.f, rs1 = ok1 ? rstd[row1] : 0.f;
  const int n_blocks = D.d / 32;
  const float* dpb = dpool + (size_t)b * D.d;
  // rows of v this lane loads for mma tile j of a 32-column block: physical column 8*(g>>1) + 2j + (g&1)
  const int pc0 = 8 * (g >> 1) + (g & 1);

  auto product = [&](const float* w, int cb, float (&c)[4][4]) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      c[j][0] = c[j][1] = c[j][2] = c[j][3] = 0.f;
      const float* wr = w + (size_t)(cb + pc0 + 2 * j) * D.m;
#pragma unroll
      for (int ch = 0; ch < KC; ++ch) {
        const int k = 32 * ch + 8 * t;
        Frag8 f = load8(wr + k, k + 8 <= D.m);
        if (k < D.m && k + 8 > D.m) f.lo = *reinterpret_cast<const float4*>(wr + k);
#pragma unroll
        for (int s = 0; s < 4; ++s) {
          uint32_t fh[2], fl[2];
          split_tf32(pick(f.lo, s), fh[0], fl[0]);
          split_tf32(pick(f.hi, s), fh[1], fl[1]);
          mma_3xtf32(c[j], ah[ch][s], al[ch][s], fh, fl);
        }
      }
    }
  };
  // the lane's eight consecutive columns of row 0 / row 1 as two float4 each
  auto row_vals = [](const float (&c)[4][4], int half, float4& lo, float4& hi) {
    lo = make_float4(c[0][2 * half], c[0][2 * half + 1], c[1][2 * half], c[1][2 * half + 1]);
    hi = make_float4(c[2][2 * half], c[2][2 * half + 1], c[3][2 * half], c[3][2 * half + 1]);
  };
  auto dot4 = [](const float4& a, const float4& p, const float4& x) {
    return (a.x + p.x) * x.x + (a.y + p.y) * x.y + (a.z + p.z) * x.z + (a.w + p.w) * x.w;
  };

  float dot0 = 0.f, dot1 = 0.f;
  for (int nb = cq; nb < n_blocks; nb += 4) {
    const int cb = nb * 32, col = cb + 8 * t;
    float c1[4][4];
    product(v1, cb, c1);
    const float4 dpa = *reinterpret_cast<const float4*>(dpb + col), dpc = *reinterpret_cast<const float4*>(dpb + col + 4);
    float4 lo, hi;
    if (ok0) {
      row_vals(c1, 0, lo, hi);
      const float4 ha = *reinterpret_cast<const float4*>(h0 + row0 * D.d + col), hb = *reinterpret_cast<const float4*>(h0 + row0 * D.d + col + 4);
      dot0 += (dot4(lo, dpa, ha) + dot4(hi, dpc, hb)) * rs0;
    }
    if (ok1) {
      row_vals(c1, 1, lo, hi);
      const float4 ha = *reinterpret_cast<const float4*>(h0 + row1 * D.d + col), hb = *reinterpret_cast<const float4*>(h0 + row1 * D.d + col + 4);
      dot1 += (dot4(lo, dpa, ha) + dot4(hi, dpc, hb)) * rs1;
    }
  }
  dot0 += __shfl_xor_sync(0xffffffffu, dot0, 1); dot0 += __shfl_xor_sync(0xffffffffu, dot0, 2);
  dot1 += __shfl_xor_sync(0xffffffffu, dot1, 1); dot1 += __shfl_xor_sync(0xffffffffu, dot1, 2);
  if (t == 0) { sdot[mt * 16 + g][cq] = dot0; sdot[mt * 16 + g + 8][cq] = dot1; }
  __syncthreads();
  {
    const float* q0 = sdot[mt * 16 + g];
    const float* q1 = sdot[mt * 16 + g + 8];
    dot0 = (q0[0] + q0[1] + q0[2] + q0[3]) / (float)D.d;
    dot1 = (q1[0] + q1[1] + q1[2] + q1[3]) / (float)D.d;
  }
  const bool own3 = dhx != dh0;                      // kernel-uniform: the v3 slice's gradient has a buffer of its own
  auto finish = [&](float4& o, const float4& a1v, const float4& a3v, const float4& dp, const float4& hv, float rs, float dot) {
    o.x += a3v.x + rs * ((a1v.x + dp.x) - hv.x * rs * dot);
    o.y += a3v.y + rs * ((a1v.y + dp.y) - hv.y * rs * dot);
    o.z += a3v.z + rs * ((a1v.z + dp.z) - hv.z * rs * dot);
    o.w += a3v.w + rs * ((a1v.w + dp.w) - hv.w * rs * dot);
  };
  const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int nb = cq; nb < n_blocks; nb += 4) {
    const int cb = nb * 32, col = cb + 8 * t;
    float c1[4][4], c3[4][4];
    product(v1, cb, c1);
    product(v3, cb, c3);
    const float4 dpa = *reinterpret_cast<const float4*>(dpb + col), dpc = *reinterpret_cast<const float4*>(dpb + col + 4);
    float4 ra = zero4, rb = zero4;                   // what every token of the sample gets on top
    if (row_add)
      for (int k = 0; k < parts; ++k) {
        const float* r = row_add + k * part_stride + (size_t)b * D.d + col;
        const float4 xa = *reinterpret_cast<const float4*>(r), xb = *reinterpret_cast<const float4*>(r + 4);
        ra.x += xa.x; ra.y += xa.y; ra.z += xa.z; ra.w += xa.w;
        rb.x += xb.x; rb.y += xb.y; rb.z += xb.z; rb.w += xb.w;
      }
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const bool ok = half ? ok1 : ok0;
      if (!ok) continue;
      const size_t row = half ? row1 : row0;
      const float rs = half ? rs1 : rs0, dot = half ? dot1 : dot0;
      float4 l1, h1, l3, h3;
      row_vals(c1, half, l1, h1);
      row_vals(c3, half, l3, h3);
      const float4 ha = *reinterpret_cast<const float4*>(h0 + row * D.d + col), hb = *reinterpret_cast<const float4*>(h0 + row * D.d + col + 4);
      float4* q = reinterpret_cast<float4*>(dh0 + row * D.d + col);
      float4 oa = q[0], ob = q[1];
      finish(oa, l1, own3 ? zero4 : l3, dpa, ha, rs, dot);
      finish(ob, h1, own3 ? zero4 : h3, dpc, hb, rs, dot);
      if (row_add) {
        oa.x += ra.x; oa.y += ra.y; oa.z += ra.z; oa.w += ra.w;
        ob.x += rb.x; ob.y += rb.y; ob.z += rb.z; ob.w += rb.w;
      }
      q[0] = oa; q[1] = ob;
      if (dh16)
        *reinterpret_cast<uint4*>(dh16 + row * D.d + col) = make_uint4(rte::pack_bf16x2(oa.x, oa.y), rte::pack_bf16x2(oa.z, oa.w),
                                                                       rte::pack_bf16x2(ob.x, ob.y), rte::pack_bf16x2(ob.z, ob.w));
      if (own3) {
        float4* qx = reinterpret_cast<float4*>(dhx + row * D.d + col);
        float4 xa = qx[0], xb = qx[1];
        xa.x += l3.x; xa.y += l3.y; xa.z += l3.z; xa.w += l3.w;
        xb.x += h3.x; xb.y += h3.y; xb.z += h3.z; xb.w += h3.w;
        qx[0] = xa; qx[1] = xb;
      }
    }
  }
}

// out[key][e] = sum over samples b with key(b) == key, in sample order, of partial[b][e]   (blockIdx.y = key), for the
// four parameters in one launch.  The member list is compacted by ballots: one thread walking the samples' ids waited
// for memory B times before the first addition (32 samples x 1024, rank 32: four launches of 75 us together -> one of 17).
struct KeyJobs { const float* partial[4]; float* out[4]; long long elems[4]; int first_block[5]; };

__global__ void __launch_bounds__(NTHR)
phi_reduce_keys_kernel(const KeyJobs jobs, const int32_t* __restrict__ rid, const int32_t* __restrict__ sid, int B, int K) {
  rte::after_previous_grid();
  __shared__ int members[1024];
  __shared__ int warp_count[NTHR / 32];
  const int key = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int n = 0;
  for (int b0 = 0; b0 < B; b0 += NTHR) {
    const int b = b0 + threadIdx.x;
    const bool mine = b < B && rid[b] * K + sid[b] == key;
    const unsigned votes = __ballot_sync(0xffffffffu, mine);
    if (lane == 0) warp_count[warp] = __popc(votes);
    __syncthreads();
    int at = n + __popc(votes & ((1u << lane) - 1));
#pragma unroll
    for (int w = 0; w < NTHR / 32; ++w) {
      if (w < warp) at += warp_count[w];
      n += warp_count[w];
    }
    if (mine) members[at] = b;
    __syncthreads();
  }
  int q = 0;
  while (q < 3 && (int)blockIdx.x >= jobs.first_block[q + 1]) ++q;
  const long long elems = jobs.elems[q], e = ((long long)blockIdx.x - jobs.first_block[q]) * NTHR + threadIdx.x;
  const float* partial = jobs.partial[q];
  float* out = jobs.out[q] + (size_t)key * elems;
  if (e >= elems) return;          // (an element per thread: often one key has most samples, and only its CTAs work)
  float acc = 0.f;
#pragma unroll 16
  for (int i = 0; i < n; ++i) acc += partial[(size_t)members[i] * elems + e];
  out[e] = acc;
}

// Mean-squared-error pieces of the consistency term (macro.py:359): g[i] = coef * (a[i] - b[i]) and one partial sum of
// (a[i] - b[i])^2 per block (fixed grid, grid-stride: the summation order does not depend on anything but n).
constexpr int SQD_BLOCKS = 592;
__global__ void __launch_bounds__(256)
sqdiff_grad_kernel(const float* __restrict__ a, const float* __restrict__ b, long long n, float coef,
                   float* __restrict__ g, float* __restrict__ partial) {
  rte::after_previous_grid();
  __shared__ float red[32];
  float s = 0.f;
  for (long long i = blockIdx.x * 256LL + threadIdx.x; i < n; i += (long long)gridDim.x * 256) {
    const float dv = a[i] - b[i];
    g[i] = coef * dv;
    s += dv * dv;
  }
  s = rte::block_sum(s, red);
  if (threadIdx.x == 0) partial[blockIdx.x] = s;
}
__global__ void sqdiff_final_kernel(const float* __restrict__ partial, int n, float* __restrict__ out, int accumulate) {
  rte::after_previous_grid();
  __shared__ float red[32];
  float s = 0.f;
  for (int i = threadIdx.x; i < n; i += blockDim.x) s += partial[i];
  s = rte::block_sum(s, red);
  if (threadIdx.x == 0) out[0] = accumulate ? out[0] + s : s;
}

}  // namespace

#define ST(s) reinterpret_cast<cudaStream_t>(s)

namespace {
// The tensor-core forward / phi_out backward need the transposed parameters (p->wt, see rte_macro_phi_prepare),
// d % 32 == 0, rank % 4 == 0 and 16-byte aligned buffers; otherwise the scalar kernels run.
inline bool phi_tensor_path(const rte_phi_params* p, const void* a, const void* b, const void* c, int d, int m) {
  return p->wt != nullptr && p->n_keys > 0 && d % 32 == 0 && m % 4 == 0 &&
         ((reinterpret_cast<uintptr_t>(p->wt) | reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) |
           reinterpret_cast<uintptr_t>(c) | reinterpret_cast<uintptr_t>(p->gain) | reinterpret_cast<uintptr_t>(p->bias) |
           reinterpret_cast<uintptr_t>(p->scale)) & 15) == 0;
}
}  // namespace

// wt (n_keys*(3d*m + m*d) floats) = [ v^T as [m][n_keys*3d] | u^T as [d][n_keys*m] ]: once per optimiser step.
extern "C" int rte_macro_phi_prepare(const float* v, const float* u, float* wt, int32_t n_keys, int32_t d, int32_t m,
                                     rte_stream_t stream) {
  RTE_CHECK_ARG(v && u && wt && n_keys > 0 && d > 0 && m > 0);
  int rc = rte_transpose_f32(v, wt, n_keys * 3 * d, m, 0, 0, stream);
  if (rc != RTE_OK) return rc;
  return rte_transpose_f32(u, wt + (size_t)m * n_keys * 3 * d, n_keys * m, d, 0, 0, stream);
}

namespace {
// the cluster kernel's shapes; others take one CTA per sample
bool phi_rows_path(const float* h0, int d) { return d % 4 == 0 && d <= 2048 && (reinterpret_cast<uintptr_t>(h0) & 15) == 0; }

template <int PART>
int launch_prep(const float* h0, const float* v, const int32_t* recipe_id, const int32_t* stride_id, float* rstd, float* pooled,
                float* pa, PhiDims D, float eps, rte_stream_t stream) {
#define RTE_PREP(NV)                                                                                                         \
  do {                                                                                                                       \
    if (prep_smem(128 * NV) > 48 * 1024 &&                                                                                   \
        cudaFuncSetAttribute(phi_prep_kernel<NV, PART>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)prep_smem(128 * NV)) != cudaSuccess) \
      return RTE_ERR_LAUNCH;                                                                                                 \
    rte::launch(phi_prep_kernel<NV, PART>, D.B * PREP_CTAS, NTHR, prep_smem(D.d), ST(stream), h0, v, recipe_id, stride_id, rstd, pooled, pa, D, eps); \
  } while (0)
  if (D.d <= 128) RTE_PREP(1);
  else if (D.d <= 256) RTE_PREP(2);
  else if (D.d <= 512) RTE_PREP(4);
  else if (D.d <= 1024) RTE_PREP(8);
  else RTE_PREP(16);
#undef RTE_PREP
  return RTE_OK;
}

// `h0`: the state Phi is applied to (norm, pooled mean, gain and residual terms); `hx`: the injected state of the third
// slice of z (the same pointer on the hot path).
int phi_fwd_impl(const float* h0, const float* hx, const rte_phi_params* p, const int32_t* recipe_id,
                 const int32_t* stride_id, float s_cfg, float* out, float* rstd, float* pooled,
                 float* act, int32_t B, int32_t S, int32_t d, int32_t m, int32_t K_strides,
                 float eps, rte_stream_t stream, bool rows_done = false) {
  RTE_CHECK_ARG(h0 && hx && p && p->gain && p->v && p->u && p->bias && p->scale && recipe_id && stride_id && out && rstd &&
                pooled && act && B > 0 && S > 0 && d > 0 && m > 0 && K_strides > 0);
  if (m > MMAX) return RTE_ERR_UNSUPPORTED;
  PhiDims D{B, S, d, m, K_strides};
  const int tiles = rte::ceil_div(S, TT);
  // `act` doubles as the home of pa (B*m floats) is NOT safe; pa lives at the tail of `pooled`'s
  // companion: callers give pooled >= B*d + B*m floats.
  float* pa = pooled + (size_t)B * d;
  if (rows_done) {
    if (!phi_rows_path(h0, d)) return RTE_ERR_UNSUPPORTED;
    rte::launch(phi_prep_kernel<1, 2>, B * PREP_CTAS, NTHR, prep_product_smem(d), ST(stream), h0, p->v, recipe_id, stride_id, rstd, pooled, pa, D, eps);
  } else if (phi_rows_path(h0, d)) {
    const int rc = launch_prep<0>(h0, p->v, recipe_id, stride_id, rstd, pooled, pa, D, eps, stream);
    if (rc != RTE_OK) return rc;
  } else {
    rte::launch(phi_prep_any_kernel, B, NTHR, (size_t)(S + d) * sizeof(float), ST(stream), h0, p->v, recipe_id, stride_id, rstd, pooled, pa, D, eps);
  }
  RTE_LAUNCH_CHECK();
  if (phi_tensor_path(p, h0, out, act, d, m) && (reinterpret_cast<uintptr_t>(hx) & 15) == 0) {
    const long long vt_ld = (long long)p->n_keys * 3 * d, ut_ld = (long long)p->n_keys * m;
    const float* ut = p->wt + (size_t)m * vt_ld;
#define RTE_ACT(NT, OWN3) rte::launch(phi_act_mma_kernel<NT, OWN3>, B * tiles, NTHR, 0, ST(stream), h0, hx, rstd, pa, p->wt, vt_ld, recipe_id, stride_id, act, D)
    if (m <= 32) { if (hx != h0) RTE_ACT(4, true); else RTE_ACT(4, false); }
    else { if (hx != h0) RTE_ACT(8, true); else RTE_ACT(8, false); }
#undef RTE_ACT
    RTE_LAUNCH_CHECK();
    if (m <= 32)
      rte::launch(phi_out_mma_kernel<0, 1>, B * tiles, NTHR, 0, ST(stream), h0, act, p->gain, ut, ut_ld, p->bias, p->scale, recipe_id,
                                                                   stride_id, s_cfg, nullptr, out, nullptr, D);
    else
      rte::launch(phi_out_mma_kernel<0, 2>, B * tiles, NTHR, 0, ST(stream), h0, act, p->gain, ut, ut_ld, p->bias, p->scale, recipe_id,
                                                                   stride_id, s_cfg, nullptr, out, nullptr, D);
    RTE_LAUNCH_CHECK();
    return RTE_OK;
  }
  rte::launch(phi_act_kernel, B * tiles, NTHR, 0, ST(stream), h0, hx, rstd, pa, p->v, recipe_id, stride_id, act, D);
  RTE_LAUNCH_CHECK();
  if (m <= 32)
    rte::launch(phi_out_kernel<0, 32>, B * tiles, NTHR, 0, ST(stream), h0, act, p->gain, p->u, p->bias, p->scale, recipe_id, stride_id,
                                                              s_cfg, nullptr, out, nullptr, D);
  else
    rte::launch(phi_out_kernel<0, 64>, B * tiles, NTHR, 0, ST(stream), h0, act, p->gain, p->u, p->bias, p->scale, recipe_id, stride_id,
                                                              s_cfg, nullptr, out, nullptr, D);
  RTE_LAUNCH_CHECK();
  return RTE_OK;
}
}  // namespace

extern "C" int rte_macro_phi_fwd(const float* h0, const rte_phi_params* p, const int32_t* recipe_id,
                                 const int32_t* stride_id, float s_cfg, float* out, float* rstd, float* pooled,
                                 float* act, int32_t B, int32_t S, int32_t d, int32_t m, int32_t K_strides,
                                 float eps, rte_stream_t stream) {
  return phi_fwd_impl(h0, h0, p, recipe_id, stride_id, s_cfg, out, rstd, pooled, act, B, S, d, m, K_strides, eps, stream);
}

extern "C" int rte_macro_phi_rows(const float* h0, float* rstd, float* pooled, int32_t B, int32_t S, int32_t d, int32_t m, float eps,
                                  rte_stream_t stream) {
  RTE_CHECK_ARG(h0 && rstd && pooled && B > 0 && S > 0 && d > 0 && m > 0);
  if (m > MMAX || !phi_rows_path(h0, d)) return RTE_ERR_UNSUPPORTED;
  const int rc = launch_prep<1>(h0, nullptr, nullptr, nullptr, rstd, pooled, nullptr, PhiDims{B, S, d, m, 1}, eps, stream);
  if (rc != RTE_OK) return rc;
  RTE_LAUNCH_CHECK();
  return RTE_OK;
}

extern "C" int rte_macro_phi_fwd_from_rows(const float* h0, const rte_phi_params* p, const int32_t* recipe_id,
                                           const int32_t* stride_id, float s_cfg, float* out, float* rstd, float* pooled,
                                           float* act, int32_t B, int32_t S, int32_t d, int32_t m, int32_t K_strides,
                                           float eps, rte_stream_t stream) {
  return phi_fwd_impl(h0, h0, p, recipe_id, stride_id, s_cfg, out, rstd, pooled, act, B, S, d, m, K_strides, eps, stream, true);
}

extern "C" int rte_macro_phi_fwd_hx(const float* h, const float* h0, const rte_phi_params* p, const int32_t* recipe_id,
                                    const int32_t* stride_id, float s_cfg, float* out, float* rstd, float* pooled,
                                    float* act, int32_t B, int32_t S, int32_t d, int32_t m, int32_t K_strides,
                                    float eps, rte_stream_t stream) {
  return phi_fwd_impl(h, h0, p, recipe_id, stride_id, s_cfg, out, rstd, pooled, act, B, S, d, m, K_strides, eps, stream);
}

namespace {
struct PhiBwdScratch { float *dupd, *da, *dpool, *pu, *pg, *pb, *pv; };
// scratch layout (floats): dupd[M*d] | da[M*m] | dpool[B*d] | pu[B*m*d] | pg[B*d] | pb[B*d] | pv[B*3d*m]
inline PhiBwdScratch phi_scratch(float* scratch, int B, int S, int d, int m) {
  const size_t M = (size_t)B * S;
  PhiBwdScratch x;
  x.dupd = scratch;
  x.da = x.dupd + M * d;
  x.dpool = x.da + M * m;
  x.pu = x.dpool + (size_t)B * d;
  x.pg = x.pu + (size_t)B * m * d;
  x.pb = x.pg + (size_t)B * d;
  x.pv = x.pb + (size_t)B * d;
  return x;
}
}  // namespace

namespace {
// dh0 (overwritten): gradient wrt the state Phi was applied to; dhx (accumulated into; may be dh0): gradient wrt the
// injected state of z's third slice.
int phi_bwd_data_impl(const float* h0, const float* dout, const rte_phi_params* p, const int32_t* recipe_id,
                      const int32_t* stride_id, float s_cfg, const float* rstd, const float* act, float* dh0, float* dhx,
                      float* scratch, int32_t B, int32_t S, int32_t d, int32_t m, int32_t K_strides,
                      rte_stream_t stream, const float* row_add = nullptr, void* dh16 = nullptr) {
  RTE_CHECK_ARG(h0 && dhx && dout && p && recipe_id && stride_id && rstd && act && dh0 && scratch && B > 0 && S > 0 && d > 0 && m > 0 &&
                K_strides > 0);
  if (m > MMAX || B > 1024) return RTE_ERR_UNSUPPORTED;
  PhiDims D{B, S, d, m, K_strides};
  const int tiles = rte::ceil_div(S, TT);
  const PhiBwdScratch x = phi_scratch(scratch, B, S, d, m);
  if (phi_tensor_path(p, h0, dout, dh0, d, m) && (reinterpret_cast<uintptr_t>(scratch) & 15) == 0) {
    const long long vt_ld = (long long)p->n_keys * 3 * d, ut_ld = (long long)p->n_keys * m;
    const float* ut = p->wt + (size_t)m * vt_ld;
    if (m <= 32)
      rte::launch(phi_out_mma_kernel<1, 1>, B * tiles, NTHR, 0, ST(stream), h0, act, p->gain, ut, ut_ld, p->bias, p->scale, recipe_id,
                                                                   stride_id, s_cfg, dout, dh0, x.dupd, D);
    else
      rte::launch(phi_out_mma_kernel<1, 2>, B * tiles, NTHR, 0, ST(stream), h0, act, p->gain, ut, ut_ld, p->bias, p->scale, recipe_id,
                                                                   stride_id, s_cfg, dout, dh0, x.dupd, D);
  } else if (m <= 32)
    rte::launch(phi_out_kernel<1, 32>, B * tiles, NTHR, 0, ST(stream), h0, act, p->gain, p->u, p->bias, p->scale, recipe_id, stride_id,
                                                              s_cfg, dout, dh0, x.dupd, D);
  else
    rte::launch(phi_out_kernel<1, 64>, B * tiles, NTHR, 0, ST(stream), h0, act, p->gain, p->u, p->bias, p->scale, recipe_id, stride_id,
                                                              s_cfg, dout, dh0, x.dupd, D);
  RTE_LAUNCH_CHECK();
  // tensor-core (3xTF32) products with 16-byte operand loads; other shapes keep the scalar kernels
  const bool mma = d % 32 == 0 && m % 4 == 0 && ((reinterpret_cast<uintptr_t>(scratch) | reinterpret_cast<uintptr_t>(h0) |
                   reinterpret_cast<uintptr_t>(dh0) | reinterpret_cast<uintptr_t>(dhx) | reinterpret_cast<uintptr_t>(p->u) |
                   reinterpret_cast<uintptr_t>(p->v)) & 15) == 0;
  if (mma && m <= 32) rte::launch(phi_da_mma_kernel<4>, B * tiles, NTHR, 0, ST(stream), x.dupd, act, p->u, recipe_id, stride_id, x.da, D);
  else if (mma) rte::launch(phi_da_mma_kernel<8>, B * tiles, NTHR, 0, ST(stream), x.dupd, act, p->u, recipe_id, stride_id, x.da, D);
  else rte::launch(phi_da_kernel, B * tiles, NTHR, 0, ST(stream), x.dupd, act, p->u, recipe_id, stride_id, x.da, D);
  RTE_LAUNCH_CHECK();
  rte::launch(phi_dpool_kernel, B * rte::ceil_div(d, NTHR), NTHR, 0, ST(stream), x.da, p->v, recipe_id, stride_id, x.dpool, D);
  RTE_LAUNCH_CHECK();
  if (mma) {                       // (with the sum's last terms and its copy, where they are wanted: one pass over dh0 instead of three)
    const bool wide = ((reinterpret_cast<uintptr_t>(row_add) | reinterpret_cast<uintptr_t>(dh16)) & 15) == 0;
    const float* ra = wide ? row_add : nullptr;
    __nv_bfloat16* o16 = wide ? reinterpret_cast<__nv_bfloat16*>(dh16) : nullptr;
    if (m <= 32)
      rte::launch(phi_dz_mma_kernel<1>, B * tiles, NTHR, 0, ST(stream), h0, rstd, x.da, x.dpool, p->v, recipe_id, stride_id, dh0, dhx, ra,
                  RTE_ROUTER_DPOOLED_PARTS, (long long)B * d, o16, D);
    else
      rte::launch(phi_dz_mma_kernel<2>, B * tiles, NTHR, 0, ST(stream), h0, rstd, x.da, x.dpool, p->v, recipe_id, stride_id, dh0, dhx, ra,
                  RTE_ROUTER_DPOOLED_PARTS, (long long)B * d, o16, D);
    if (wide) { row_add = nullptr; dh16 = nullptr; }
  }
  else rte::launch(phi_dz_kernel, B * tiles, NTHR, 0, ST(stream), h0, rstd, x.da, x.dpool, p->v, recipe_id, stride_id, dh0, dhx, D);
  RTE_LAUNCH_CHECK();
  if (row_add) {
    const int rc = rte::add_router_dpooled(dh0, row_add, B, S, d, ST(stream));
    if (rc != RTE_OK) return rc;
  }
  return dh16 ? rte_cast_f32_bf16(dh0, dh16, (int64_t)B * S * d, stream) : RTE_OK;
}
}  // namespace

// Data-gradient half: dh0 (the chain the rest of backward waits for); leaves dupd and da in `scratch`.
extern "C" int rte_macro_phi_bwd_data(const float* h0, const float* dout, const rte_phi_params* p, const int32_t* recipe_id,
                                      const int32_t* stride_id, float s_cfg, const float* rstd, const float* act, float* dh0,
                                      float* scratch, int32_t B, int32_t S, int32_t d, int32_t m, int32_t K_strides,
                                      rte_stream_t stream) {
  return phi_bwd_data_impl(h0, dout, p, recipe_id, stride_id, s_cfg, rstd, act, dh0, dh0, scratch, B, S, d, m, K_strides, stream);
}

extern "C" int rte_macro_phi_bwd_data_finish(const float* h0, const float* dout, const rte_phi_params* p, const int32_t* recipe_id,
                                             const int32_t* stride_id, float s_cfg, const float* rstd, const float* act, float* dh0,
                                             float* scratch, const float* router_scratch, int32_t hid, int32_t R, void* dh0_bf16,
                                             int32_t B, int32_t S, int32_t d, int32_t m, int32_t K_strides, rte_stream_t stream) {
  RTE_CHECK_ARG(router_scratch == nullptr || (hid > 0 && R > 0));
  if (router_scratch && d % 4 != 0) return RTE_ERR_UNSUPPORTED;
  if (reinterpret_cast<uintptr_t>(router_scratch) & 15) return RTE_ERR_ALIGNMENT;
  return phi_bwd_data_impl(h0, dout, p, recipe_id, stride_id, s_cfg, rstd, act, dh0, dh0, scratch, B, S, d, m, K_strides, stream,
                           router_scratch ? rte::router_dpooled(router_scratch, B, hid, R, K_strides) : nullptr, dh0_bf16);
}

// Parameter-gradient half: reads dupd and da left in `scratch` by rte_macro_phi_bwd_data (may run on another
// stream, ordered after it); nothing downstream in backward depends on it.
namespace {
int phi_bwd_params_impl(const float* h0, const float* hx, const int32_t* recipe_id, const int32_t* stride_id, const float* rstd,
                        const float* pooled, const float* act, const rte_phi_grads* g, float* scratch,
                        int32_t B, int32_t S, int32_t d, int32_t m, int32_t R, int32_t K_strides,
                        rte_stream_t stream) {
  RTE_CHECK_ARG(h0 && hx && recipe_id && stride_id && rstd && pooled && act && g && scratch && B > 0 && S > 0 && d > 0 && m > 0 &&
                R > 0 && K_strides > 0);
  RTE_CHECK_ARG(g->gain && g->v && g->u && g->bias);
  if (m > MMAX || B > 1024) return RTE_ERR_UNSUPPORTED;
  PhiDims D{B, S, d, m, K_strides};
  const PhiBwdScratch x = phi_scratch(scratch, B, S, d, m);
  const int grid = B * rte::ceil_div(d, 128);
#define RTE_PG(NT, OWN3) rte::launch(phi_param_grads_kernel<NT, OWN3>, grid, NTHR, 0, ST(stream), h0, hx, rstd, pooled, act, x.dupd, x.da, x.pu, x.pg, x.pb, x.pv, D)
  if (m <= 32) { if (hx != h0) RTE_PG(4, true); else RTE_PG(4, false); }
  else { if (hx != h0) RTE_PG(8, true); else RTE_PG(8, false); }
#undef RTE_PG
  RTE_LAUNCH_CHECK();
  KeyJobs jobs = {{x.pv, x.pu, x.pg, x.pb}, {g->v, g->u, g->gain, g->bias}, {(long long)3 * d * m, (long long)m * d, d, d}, {0}};
  for (int q = 0; q < 4; ++q) jobs.first_block[q + 1] = jobs.first_block[q] + (int)rte::ceil_div64(jobs.elems[q], NTHR);
  rte::launch(phi_reduce_keys_kernel, dim3((unsigned)jobs.first_block[4], R * K_strides), NTHR, 0, ST(stream), jobs, recipe_id, stride_id, B, K_strides);
  RTE_LAUNCH_CHECK();
  return RTE_OK;
}
}  // namespace

extern "C" int rte_macro_phi_bwd_params(const float* h0, const int32_t* recipe_id, const int32_t* stride_id, const float* rstd,
                                        const float* pooled, const float* act, const rte_phi_grads* g, float* scratch,
                                        int32_t B, int32_t S, int32_t d, int32_t m, int32_t R, int32_t K_strides,
                                        rte_stream_t stream) {
  return phi_bwd_params_impl(h0, h0, recipe_id, stride_id, rstd, pooled, act, g, scratch, B, S, d, m, R, K_strides, stream);
}

// Phi applied to a state h that is not the injected h0 (macro.py:342-359, the consistency term's second application):
// dh (overwritten) and dh0 (ACCUMULATED into) are separate; parameter gradients as in rte_macro_phi_bwd.
extern "C" int rte_macro_phi_bwd_hx(const float* h, const float* h0, const float* dout, const rte_phi_params* p,
                                    const int32_t* recipe_id, const int32_t* stride_id, float s_cfg, const float* rstd,
                                    const float* pooled, const float* act, float* dh, float* dh0, const rte_phi_grads* g,
                                    float* scratch, int32_t B, int32_t S, int32_t d, int32_t m, int32_t R, int32_t K_strides,
                                    rte_stream_t stream) {
  RTE_CHECK_ARG(g != nullptr && R > 0 && dh != dh0);
  const int rc = phi_bwd_data_impl(h, dout, p, recipe_id, stride_id, s_cfg, rstd, act, dh, dh0, scratch, B, S, d, m, K_strides, stream);
  if (rc != RTE_OK) return rc;
  return phi_bwd_params_impl(h, h0, recipe_id, stride_id, rstd, pooled, act, g, scratch, B, S, d, m, R, K_strides, stream);
}

// Both halves on one stream.
extern "C" int rte_macro_phi_bwd(const float* h0, const float* dout, const rte_phi_params* p, const int32_t* recipe_id,
                                 const int32_t* stride_id, float s_cfg, const float* rstd, const float* pooled,
                                 const float* act, float* dh0, const rte_phi_grads* g, float* scratch, int32_t B,
                                 int32_t S, int32_t d, int32_t m, int32_t R, int32_t K_strides, float eps,
                                 rte_stream_t stream) {
  (void)eps;
  RTE_CHECK_ARG(g != nullptr && R > 0);
  const int rc = rte_macro_phi_bwd_data(h0, dout, p, recipe_id, stride_id, s_cfg, rstd, act, dh0, scratch, B, S, d, m, K_strides, stream);
  if (rc != RTE_OK) return rc;
  return rte_macro_phi_bwd_params(h0, recipe_id, stride_id, rstd, pooled, act, g, scratch, B, S, d, m, R, K_strides, stream);
}

// g = coef * (a - b);  sum_out (+)= sum (a - b)^2.  `partial`: >= 1024 floats of scratch.
extern "C" int rte_sqdiff_grad(const float* a, const float* b, int64_t n, float coef, float* g, float* partial, float* sum_out,
                               int32_t accumulate, rte_stream_t stream) {
  RTE_CHECK_ARG(a && b && g && partial && sum_out && n > 0);
  rte::launch(sqdiff_grad_kernel, SQD_BLOCKS, 256, 0, ST(stream), a, b, n, coef, g, partial);
  RTE_LAUNCH_CHECK();
  rte::launch(sqdiff_final_kernel, 1, 1024, 0, ST(stream), partial, SQD_BLOCKS, sum_out, accumulate);
  RTE_LAUNCH_CHECK();
  return RTE_OK;
}
