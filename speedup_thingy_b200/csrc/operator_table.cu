// Passes of the operator table (kernels.py) that turn whatever layout and type a caller's tensors have into what the
// compute kernels read, one launch per operator instead of one framework copy per tensor: fp32 -> bf16 of several tensors
// at once, RMSNorm on bf16 or fp32 rows, rotary embedding over strided [B, H, S, head_dim] views of q and k together, and
// q / k / v views packed into the attention kernels' row layout.  All of them are bound by memory for large tensors and
// by their launch for small ones (kernels reference.py:9-28,40-41).

#include "rte_common.cuh"

namespace {

// Bound by HBM (6 bytes an element).  Every CTA takes 4096 consecutive elements of one tensor, four 16-byte loads a thread before the
// first store: with the largest tensor's grid for each of them and one load a trip, small tensors left CTAs without work
// and a thread waited for each load: 4 M elements + two small tensors 17.5 -> 6.0 us, 8 M + three of 1 M 29.5 -> 12.4, 34 M alone
// 41.7 -> 33.2 (6.1 TB/s).
constexpr int CAST_CTA = 4096;
struct CastJobs { const float* src[4]; __nv_bfloat16* dst[4]; long long n4[4]; long long n[4]; int first[4]; int count; };

__global__ void __launch_bounds__(256) cast_many_kernel(const __grid_constant__ CastJobs jobs) {
  rte::after_previous_grid();
  int j = 0;
  while (j + 1 < jobs.count && (int)blockIdx.x >= jobs.first[j + 1]) ++j;
  const float* __restrict__ src = jobs.src[j];
  __nv_bfloat16* __restrict__ dst = jobs.dst[j];
  const long long n4 = jobs.n4[j], n = jobs.n[j], base = (long long)((int)blockIdx.x - jobs.first[j]) * CAST_CTA;
  if (n4 > 0) {
    const long long at = base / 4 + threadIdx.x;
    float4 v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (at + 256 * u < n4) v[u] = reinterpret_cast<const float4*>(src)[at + 256 * u];
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (at + 256 * u < n4) reinterpret_cast<uint2*>(dst)[at + 256 * u] = make_uint2(rte::pack_bf16x2(v[u].x, v[u].y), rte::pack_bf16x2(v[u].z, v[u].w));
    const long long rest = 4 * n4 + threadIdx.x;                       // (at most three elements: the last CTA's)
    if (base + CAST_CTA >= n && rest < n) dst[rest] = __float2bfloat16_rn(src[rest]);
  } else {
    for (long long i = base + threadIdx.x; i < n && i < base + CAST_CTA; i += 256) dst[i] = __float2bfloat16_rn(src[i]);
  }
}

__device__ __forceinline__ float4 load4(const void* p, int is_bf16, size_t i4) {
  if (!is_bf16) return reinterpret_cast<const float4*>(p)[i4];
  const uint2 w = reinterpret_cast<const uint2*>(p)[i4];
  const float2 a = rte::unpack_bf16x2(w.x), b = rte::unpack_bf16x2(w.y);
  return make_float4(a.x, a.y, b.x, b.y);
}
__device__ __forceinline__ void store4(void* p, int is_bf16, size_t i4, const float4& v) {
  if (is_bf16) reinterpret_cast<uint2*>(p)[i4] = make_uint2(rte::pack_bf16x2(v.x, v.y), rte::pack_bf16x2(v.z, v.w));
  else reinterpret_cast<float4*>(p)[i4] = v;
}

// One warp per row: y = x (+ res) in fp32 (kept for backward), out = y * rsqrt(mean y^2 + eps) * w.
template <int NV>
__global__ void __launch_bounds__(256)
rmsnorm_op_kernel(const void* __restrict__ x, int x16, const void* __restrict__ res, int res16, const void* __restrict__ w, int w16,
                  float* __restrict__ y, void* __restrict__ out, int out16, void* __restrict__ sum, int sum16, float* __restrict__ rstd,
                  float* __restrict__ w32, int rows, int d, float eps) {
  rte::after_previous_grid();
  const int lane = threadIdx.x & 31, row = blockIdx.x * 8 + (threadIdx.x >> 5), d4 = d >> 2;
  if (row >= rows) return;
  float4 v[NV];
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = lane + 32 * i;
    if (c < d4) {
      const size_t at = (size_t)row * d4 + c;
      v[i] = load4(x, x16, at);
      if (res) {
        const float4 r = load4(res, res16, at);
        v[i].x += r.x; v[i].y += r.y; v[i].z += r.z; v[i].w += r.w;
        store4(sum, sum16, at, v[i]);
      }
      if (y) reinterpret_cast<float4*>(y)[at] = v[i];
      ss += v[i].x * v[i].x + v[i].y * v[i].y + v[i].z * v[i].z + v[i].w * v[i].w;
    }
  }
  ss = rte::warp_sum(ss);
  const float r = rsqrtf(ss / (float)d + eps);
  if (lane == 0) rstd[row] = r;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = lane + 32 * i;
    if (c < d4) {
      const float4 ww = load4(w, w16, c);
      if (row == 0 && w32) reinterpret_cast<float4*>(w32)[c] = ww;
      store4(out, out16, (size_t)row * d4 + c, make_float4(v[i].x * r * ww.x, v[i].y * r * ww.y, v[i].z * r * ww.z, v[i].w * r * ww.w));
    }
  }
}

struct View4 { const void* p; long long sb, sh, ss; };          // [B, H, S, hd], unit stride along hd
struct View4Out { void* p; long long sb, sh, ss; };

// out = rotation (or its transpose) of adjacent pairs with caller's cos / sin [S, hd]; blockIdx.y: q | k.  I counts the
// pairs: 32 bits below 2^31 of them (a grid stride past the last one must not wrap), else 64.
template <typename T, typename I>
__global__ void __launch_bounds__(256)
rope_views_kernel(View4 q, View4 k, View4Out oq, View4Out ok, const float* __restrict__ cs, const float* __restrict__ sn, int H, int S, int hd,
                  I pairs, int adjoint) {
  rte::after_previous_grid();
  const View4& v = blockIdx.y == 0 ? q : k;
  const View4Out& o = blockIdx.y == 0 ? oq : ok;
  const unsigned hp = hd / 2;
  for (I i = blockIdx.x * blockDim.x + threadIdx.x; i < pairs; i += gridDim.x * blockDim.x) {
    // (pair, head, position, sample): neighbouring threads stay inside one token's row of a [B, S, H, hd] layout
    I r = i / hp;
    const unsigned pr = (unsigned)(i - r * hp), h = (unsigned)(r % (unsigned)H);
    r /= (unsigned)H;
    const unsigned s = (unsigned)(r % (unsigned)S), b = (unsigned)(r / (unsigned)S);
    const T* x = reinterpret_cast<const T*>(v.p) + b * v.sb + h * v.sh + s * v.ss + 2 * pr;
    T* y = reinterpret_cast<T*>(o.p) + b * o.sb + h * o.sh + s * o.ss + 2 * pr;
    const float a = (float)x[0], c = (float)x[1];
    const float c0 = cs[s * hd + 2 * pr], c1 = cs[s * hd + 2 * pr + 1], s0 = sn[s * hd + 2 * pr], s1 = sn[s * hd + 2 * pr + 1];
    y[0] = (T)(adjoint ? a * c0 + c * s1 : a * c0 - c * s0);
    y[1] = (T)(adjoint ? c * c1 - a * s0 : c * c1 + a * s1);
  }
}

// q | k | v views -> bf16 rows [B * S, 3 * H * hd], eight elements per thread
template <typename T>
__global__ void __launch_bounds__(256)
pack_qkv_kernel(View4 q, View4 k, View4 v, __nv_bfloat16* __restrict__ out, int H, int S, int hd, unsigned groups, int wide) {
  rte::after_previous_grid();
  const View4& src = blockIdx.y == 0 ? q : blockIdx.y == 1 ? k : v;
  const unsigned h8 = hd / 8;
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < groups; i += gridDim.x * blockDim.x) {
    unsigned r = i / h8;
    const unsigned c = (i - r * h8) * 8, h = r % (unsigned)H;
    r /= (unsigned)H;                                            // token b * S + s
    const unsigned s = r % (unsigned)S, b = r / (unsigned)S;
    const T* x = reinterpret_cast<const T*>(src.p) + b * src.sb + h * src.sh + s * src.ss + c;
    uint4 w;
    if constexpr (sizeof(T) == 2) {
      if (wide) {
        w = *reinterpret_cast<const uint4*>(x);
      } else {
        const uint16_t* u = reinterpret_cast<const uint16_t*>(x);
        w = make_uint4(u[0] | u[1] << 16, u[2] | u[3] << 16, u[4] | u[5] << 16, u[6] | u[7] << 16);
      }
    } else {
      float e[8];
      if (wide) {
        const float4 a = reinterpret_cast<const float4*>(x)[0], d = reinterpret_cast<const float4*>(x)[1];
        e[0] = a.x; e[1] = a.y; e[2] = a.z; e[3] = a.w; e[4] = d.x; e[5] = d.y; e[6] = d.z; e[7] = d.w;
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) e[j] = (float)x[j];
      }
      w = make_uint4(rte::pack_bf16x2(e[0], e[1]), rte::pack_bf16x2(e[2], e[3]), rte::pack_bf16x2(e[4], e[5]), rte::pack_bf16x2(e[6], e[7]));
    }
    *reinterpret_cast<uint4*>(out + ((size_t)r * 3 + blockIdx.y) * H * hd + h * hd + c) = w;
  }
}

inline int blocks_for(long long n, int cap) {
  const long long g = (n + 255) / 256;
  return (int)(g < 1 ? 1 : g > cap ? cap : g);
}
inline bool on16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

}  // namespace

#define ST(s) reinterpret_cast<cudaStream_t>(s)

extern "C" int rte_cast_many_f32_bf16(const float* const* src, void* const* dst, const int64_t* n, int32_t count, rte_stream_t stream) {
  RTE_CHECK_ARG(src && dst && n && count >= 1 && count <= 4);
  CastJobs jobs = {};
  long long ctas = 0;
  for (int j = 0; j < count; ++j) {
    RTE_CHECK_ARG(src[j] && dst[j] && n[j] > 0);
    jobs.src[j] = src[j];
    jobs.dst[j] = reinterpret_cast<__nv_bfloat16*>(dst[j]);
    jobs.n[j] = n[j];
    jobs.n4[j] = on16(src[j]) && (reinterpret_cast<uintptr_t>(dst[j]) & 7) == 0 ? n[j] / 4 : 0;
    jobs.first[j] = (int)ctas;
    ctas += (n[j] + CAST_CTA - 1) / CAST_CTA;
    RTE_CHECK_ARG(ctas < (1ll << 31));
  }
  jobs.count = count;
  rte::launch(cast_many_kernel, (unsigned)ctas, 256, 0, ST(stream), jobs);
  RTE_LAUNCH_CHECK();
  return RTE_OK;
}

extern "C" int rte_rmsnorm_op_fwd(const void* x, int32_t x_bf16, const void* res, int32_t res_bf16, const void* w, int32_t w_bf16, float* y,
                                  void* out, int32_t out_bf16, void* sum, int32_t sum_bf16, float* rstd, float* w_f32, int32_t rows, int32_t d,
                                  float eps, rte_stream_t stream) {
  RTE_CHECK_ARG(x && w && out && rstd && rows > 0 && d > 0 && d % 4 == 0 && (res == nullptr) == (sum == nullptr));
  if (d > 2048) return RTE_ERR_UNSUPPORTED;
  if (!on16(x) || !on16(w) || !on16(out) || !on16(y) || !on16(res) || !on16(sum) || !on16(w_f32)) return RTE_ERR_ALIGNMENT;
#define RTE_OP(NV) rte::launch(rmsnorm_op_kernel<NV>, rte::ceil_div(rows, 8), 256, 0, ST(stream), x, x_bf16, res, res_bf16, w, w_bf16, y, out, out_bf16, \
                               sum, sum_bf16, rstd, w_f32, rows, d, eps)
  if (d <= 128) RTE_OP(1);
  else if (d <= 256) RTE_OP(2);
  else if (d <= 512) RTE_OP(4);
  else if (d <= 1024) RTE_OP(8);
  else RTE_OP(16);
#undef RTE_OP
  RTE_LAUNCH_CHECK();
  return RTE_OK;
}

extern "C" int rte_rope_views(const void* q, const int64_t* q_strides, const void* k, const int64_t* k_strides, void* q_out, const int64_t* qo_strides,
                              void* k_out, const int64_t* ko_strides, const float* cos_tab, const float* sin_tab, int32_t B, int32_t H, int32_t S,
                              int32_t hd, int32_t is_bf16, int32_t adjoint, rte_stream_t stream) {
  RTE_CHECK_ARG(q && k && q_out && k_out && cos_tab && sin_tab && B > 0 && H > 0 && S > 0 && hd > 0 && hd % 2 == 0);
  const long long pairs = (long long)B * H * S * (hd / 2);
  const View4 vq = {q, q_strides[0], q_strides[1], q_strides[2]}, vk = {k, k_strides[0], k_strides[1], k_strides[2]};
  const View4Out oq = {q_out, qo_strides[0], qo_strides[1], qo_strides[2]}, ok = {k_out, ko_strides[0], ko_strides[1], ko_strides[2]};
#define RTE_ROPE(T, I) rte::launch(rope_views_kernel<T, I>, dim3(blocks_for(pairs, 148 * 8), 2), 256, 0, ST(stream), vq, vk, oq, ok, cos_tab, sin_tab, H, S, hd, \
                                   (I)pairs, adjoint)
  if (pairs < (1ll << 31)) { if (is_bf16) RTE_ROPE(__nv_bfloat16, unsigned); else RTE_ROPE(float, unsigned); }
  else { if (is_bf16) RTE_ROPE(__nv_bfloat16, unsigned long long); else RTE_ROPE(float, unsigned long long); }
#undef RTE_ROPE
  RTE_LAUNCH_CHECK();
  return RTE_OK;
}

extern "C" int rte_pack_qkv(const void* q, const int64_t* q_strides, const void* k, const int64_t* k_strides, const void* v, const int64_t* v_strides,
                            void* qkv, int32_t B, int32_t H, int32_t S, int32_t hd, int32_t is_bf16, rte_stream_t stream) {
  RTE_CHECK_ARG(q && k && v && qkv && B > 0 && H > 0 && S > 0 && hd > 0 && hd % 8 == 0);
  const long long groups = (long long)B * H * S * (hd / 8);
  RTE_CHECK_ARG(groups < (1ll << 32));
  const View4 views[3] = {{q, q_strides[0], q_strides[1], q_strides[2]}, {k, k_strides[0], k_strides[1], k_strides[2]}, {v, v_strides[0], v_strides[1], v_strides[2]}};
  const int per16 = is_bf16 ? 8 : 4;
  int wide = 1;
  for (const View4& x : views)
    if (!on16(x.p) || x.sb % per16 || x.sh % per16 || x.ss % per16) wide = 0;
  rte::launch(is_bf16 ? pack_qkv_kernel<__nv_bfloat16> : pack_qkv_kernel<float>, dim3(blocks_for(groups, 148 * 8), 3), 256, 0, ST(stream), views[0], views[1],
              views[2], reinterpret_cast<__nv_bfloat16*>(qkv), H, S, hd, (unsigned)groups, wide);
  RTE_LAUNCH_CHECK();
  return RTE_OK;
}
