// Pieces around the mixers of a post-norm decoder: the embedding with a sinusoidal position vector added, the
// residual update x += scale * RMSNorm(y) with a one-number norm weight and a per-feature layer scale, and the
// RMSNorm of a whole q or k projection (one statistic per token over all heads) with the store into the pages.
// Every statistic, angle and sum is float32 (the angle's product and its reduction to one turn are float64).
// These kernels take every size.
#include "common.cuh"
#include <math.h>

// ------------------------------------------------------------------------------------------
// out[n, 2i] = table[id, 2i] + sin(a), out[n, 2i+1] = table[id, 2i+1] + cos(a), a = position[n] * inv_freq[i].
// inv_freq is float64 (base^(-2i/width), made once on the host); the product is reduced to (-pi, pi] in float64
// before the float32 sine and cosine, so that a position in the hundreds of thousands loses nothing.
// half (may be null): the same row rounded to bfloat16, for the products that read the stream.
// An id outside the vocabulary reads nothing: the row is the position vector alone and the error word is set.
// ------------------------------------------------------------------------------------------
__global__ void embed_sinusoid_kernel(const void* __restrict__ table, int table_dtype, const int* __restrict__ ids,
                                      const int* __restrict__ positions, const double* __restrict__ inv_freq,
                                      float* __restrict__ out, __nv_bfloat16* __restrict__ half, int hidden, int vocab,
                                      int* __restrict__ err) {
  ifb_pdl_wait();
  ifb_pdl_trigger();
  const int n = blockIdx.x;
  const int id = ids[n];
  const bool bad = id < 0 || id >= vocab;
  if (bad && err && threadIdx.x == 0) atomicCAS(err, 0, IFB_DEV_ERR_TOKEN_ID);
  const size_t row = bad ? 0 : (size_t)id * hidden;
  const double p = (double)positions[n];
  const double two_pi = 6.283185307179586476925286766559;
  for (int i = threadIdx.x; 2 * i < hidden; i += blockDim.x) {
    double a = p * inv_freq[i];
    a -= two_pi * rint(a / two_pi);
    float s, c;
    sincosf((float)a, &s, &c);
    const int e0 = 2 * i, e1 = 2 * i + 1;
    const float v0 = (bad ? 0.f : load_as_f32(table, table_dtype, row + e0)) + s;
    out[(size_t)n * hidden + e0] = v0;
    if (half) half[(size_t)n * hidden + e0] = __float2bfloat16_rn(v0);
    if (e1 < hidden) {
      const float v1 = (bad ? 0.f : load_as_f32(table, table_dtype, row + e1)) + c;
      out[(size_t)n * hidden + e1] = v1;
      if (half) half[(size_t)n * hidden + e1] = __float2bfloat16_rn(v1);
    }
  }
}

IFB_EXPORT int ifb_embed_sinusoid(const void* table, int table_dtype, const int* ids, const int* positions,
                                  const double* inv_freq, float* out, void* half, int n, int hidden, int vocab, int* err,
                                  cudaStream_t stream) {
  if (n <= 0 || hidden <= 0) return IFB_OK;
  if (table_dtype != IFB_F32 && table_dtype != IFB_BF16) return IFB_ERR_DTYPE;
  const int pairs = (hidden + 1) / 2;
  const int threads = pairs >= 256 ? 256 : ((pairs + 31) / 32) * 32;
  return ifb_launch(embed_sinusoid_kernel, dim3(n), dim3(threads), 0, stream, table, table_dtype, ids, positions, inv_freq,
                    out, (__nv_bfloat16*)half, hidden, vocab, err);
}

// ------------------------------------------------------------------------------------------
// x[n, :] += y[n, :] / sqrt(mean(y[n, :]^2) + eps) * g * scale[:]      (g: one number; scale: per feature)
// half (may be null): the updated row rounded to bfloat16.  A block per row.  Rows of whole groups of four features at 16 bytes, up to
// 8,192 of them: the row, the stream's and the scale are requested together, four features at a time, the constants before the
// wait for the kernel before this one, and the sum over the block has one barrier (rows of 1,024: 2,043 of them 8.3 to 5.1 us, eight 3.4 to
// 1.5; bound by that chain of round trips for few rows and by the bytes for many).  Other rows: feature by feature; up to 2,048 features stay in
// registers between the two passes, longer rows are read twice.
// ------------------------------------------------------------------------------------------
// Four numbers of a float32 or bfloat16 array at index i, a multiple of 4; four numbers stored likewise.
__device__ __forceinline__ float4 sl_load4(const void* p, int dtype, size_t i) {
  if (dtype == IFB_F32) return *reinterpret_cast<const float4*>((const float*)p + i);
  const uint2 v = *reinterpret_cast<const uint2*>((const __nv_bfloat16*)p + i);
  return make_float4(__uint_as_float(v.x << 16), __uint_as_float(v.x & 0xffff0000u), __uint_as_float(v.y << 16), __uint_as_float(v.y & 0xffff0000u));
}
__device__ __forceinline__ void sl_store4(float* p, const float4& v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ void sl_store4(__nv_bfloat16* p, const float4& v) {
  __nv_bfloat162 lo = __floats2bfloat162_rn(v.x, v.y), hi = __floats2bfloat162_rn(v.z, v.w);
  *reinterpret_cast<uint2*>(p) = make_uint2(*reinterpret_cast<uint32_t*>(&lo), *reinterpret_cast<uint32_t*>(&hi));
}
__device__ __forceinline__ float sl_square(const float4& v, float s) { return fmaf(v.w, v.w, fmaf(v.z, v.z, fmaf(v.y, v.y, fmaf(v.x, v.x, s)))); }
// Sums of two numbers over a block of up to 256 threads, in a fixed order; one barrier.
__device__ __forceinline__ float2 sl_block_sum(float a, float b) {
  __shared__ float2 part[8];
  a = warp_sum(a);
  b = warp_sum(b);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = make_float2(a, b);
  __syncthreads();
  float2 t = part[0];
  for (int w = 1; w < (int)(blockDim.x >> 5); ++w) { t.x += part[w].x; t.y += part[w].y; }
  return t;
}
// Threads of a block whose threads take four features each, NV times.
static int sl_threads(int features, int nv) { return min(256, (((features + 3) / 4 + nv - 1) / nv + 31) / 32 * 32); }

template <int NV>
__global__ void __launch_bounds__(256)
residual_postnorm_vec_kernel(float* x, const float* y, const void* __restrict__ g, int g_dtype, const void* __restrict__ scale,
                             int scale_dtype, float eps, __nv_bfloat16* half, int hidden) {
  const size_t base = (size_t)blockIdx.x * hidden;
  float4 sc[NV], xv[NV], yv[NV];
  const float gain = load_as_f32(g, g_dtype, 0);
#pragma unroll
  for (int j = 0; j < NV; ++j) {
    const int e = (threadIdx.x + j * blockDim.x) * 4;
    sc[j] = e < hidden ? sl_load4(scale, scale_dtype, e) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  ifb_pdl_wait();
  ifb_pdl_trigger();
  float ss = 0.f;
#pragma unroll
  for (int j = 0; j < NV; ++j) {
    const int e = (threadIdx.x + j * blockDim.x) * 4;
    yv[j] = xv[j] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (e < hidden) {
      yv[j] = *reinterpret_cast<const float4*>(y + base + e);
      xv[j] = *reinterpret_cast<const float4*>(x + base + e);
    }
  }
#pragma unroll
  for (int j = 0; j < NV; ++j) ss = sl_square(yv[j], ss);
  const float r = gain / sqrtf(sl_block_sum(ss, 0.f).x / (float)hidden + eps);
#pragma unroll
  for (int j = 0; j < NV; ++j) {
    const int e = (threadIdx.x + j * blockDim.x) * 4;
    if (e >= hidden) continue;
    const float4 v = make_float4(xv[j].x + yv[j].x * r * sc[j].x, xv[j].y + yv[j].y * r * sc[j].y, xv[j].z + yv[j].z * r * sc[j].z,
                                 xv[j].w + yv[j].w * r * sc[j].w);
    sl_store4(x + base + e, v);
    if (half) sl_store4(half + base + e, v);
  }
}

constexpr int RP_THREADS = 256, RP_KEEP = 8;
__global__ void __launch_bounds__(RP_THREADS)
residual_postnorm_kernel(float* __restrict__ x, const float* __restrict__ y, const void* __restrict__ g, int g_dtype,
                         const void* __restrict__ scale, int scale_dtype, float eps, __nv_bfloat16* __restrict__ half,
                         int hidden) {
  __shared__ float scratch[33];
  ifb_pdl_wait();
  ifb_pdl_trigger();
  const size_t base = (size_t)blockIdx.x * hidden;
  const float* yr = y + base;
  float keep[RP_KEEP];
  float ss = 0.f;
  const bool held = hidden <= RP_KEEP * RP_THREADS;
  if (held) {
#pragma unroll
    for (int j = 0; j < RP_KEEP; ++j) {
      const int e = threadIdx.x + j * RP_THREADS;
      keep[j] = e < hidden ? yr[e] : 0.f;
      ss += keep[j] * keep[j];
    }
  } else {
    for (int e = threadIdx.x; e < hidden; e += RP_THREADS) { const float v = yr[e]; ss += v * v; }
  }
  ss = block_sum(ss, scratch);
  const float r = load_as_f32(g, g_dtype, 0) / sqrtf(ss / (float)hidden + eps);
  if (held) {
#pragma unroll
    for (int j = 0; j < RP_KEEP; ++j) {
      const int e = threadIdx.x + j * RP_THREADS;
      if (e < hidden) {
        const float v = x[base + e] + keep[j] * r * load_as_f32(scale, scale_dtype, e);
        x[base + e] = v;
        if (half) half[base + e] = __float2bfloat16_rn(v);
      }
    }
  } else {
    for (int e = threadIdx.x; e < hidden; e += RP_THREADS) {
      const float v = x[base + e] + yr[e] * r * load_as_f32(scale, scale_dtype, e);
      x[base + e] = v;
      if (half) half[base + e] = __float2bfloat16_rn(v);
    }
  }
}

IFB_EXPORT int ifb_residual_postnorm(float* x, const float* y, const void* g, int g_dtype, const void* scale, int scale_dtype,
                                     float eps, void* half, int n, int hidden, cudaStream_t stream) {
  if (n <= 0 || hidden <= 0) return IFB_OK;
  if ((g_dtype != IFB_F32 && g_dtype != IFB_BF16) || (scale_dtype != IFB_F32 && scale_dtype != IFB_BF16)) return IFB_ERR_DTYPE;
  if (hidden % 4 == 0 && hidden <= 8192 && (((uintptr_t)x | (uintptr_t)y | (uintptr_t)scale) & 15) == 0 && ((uintptr_t)half & 7) == 0) {
#define SL_VEC(NV)                                                                                                                  \
  if (hidden <= NV * 1024)                                                                                                          \
    return ifb_launch(residual_postnorm_vec_kernel<NV>, dim3(n), dim3(sl_threads(hidden, NV)), 0, stream, x, y, g, g_dtype, scale, scale_dtype, \
                      eps, (__nv_bfloat16*)half, hidden);
    SL_VEC(1) SL_VEC(2) SL_VEC(4) SL_VEC(8)
#undef SL_VEC
  }
  return ifb_launch(residual_postnorm_kernel, dim3(n), dim3(RP_THREADS), 0, stream, x, y, g, g_dtype, scale, scale_dtype, eps,
                    (__nv_bfloat16*)half, hidden);
}

// out = x rounded to bfloat16, element by element.
__global__ void cast_rows_kernel(const float* __restrict__ x, __nv_bfloat16* __restrict__ out, long long count) {
  ifb_pdl_wait();
  ifb_pdl_trigger();
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += (long long)gridDim.x * blockDim.x)
    out[i] = __float2bfloat16_rn(x[i]);
}

IFB_EXPORT int ifb_cast_rows(const float* x, void* out, long long count, cudaStream_t stream) {
  if (count <= 0) return IFB_OK;
  const long long blocks = (count + 255) / 256;
  return ifb_launch(cast_rows_kernel, dim3((unsigned)(blocks > 4096 ? 4096 : blocks)), dim3(256), 0, stream, x,
                    (__nv_bfloat16*)out, count);
}

// ------------------------------------------------------------------------------------------
// The q and k projections of a token, each normalised as ONE vector over all its heads:
//   q_out[n, :]  = q / sqrt(mean(q^2) + eps) * qw        (q: proj[n, 0 : q_width])
//   key page     = k / sqrt(mean(k^2) + eps) * kw        (k: proj[n, q_width : q_width + k_width])
//   value page   = k before its norm (values_are_keys), or proj[n, v_col : v_col + k_width]
// written at slot = page * page_size + offset of pages [pages][2][kv_heads][page_size][head_dim]; a negative slot
// stores nothing.  A null weight leaves that projection unnormalised.  proj is float32; T is the cache's type.
// Widths, columns and rows of whole groups of four at 16 bytes, up to 8,192 q and k features: q and k (neighbours in the row) stay in
// registers, requested with the values at once, both sums share a barrier (q 1,024, k 256: 2,043 rows 12.2 to 6.3 us, eight 4.9 to 2.1).
// Rows of more than 4,096 (NV 8) are held to the 128 registers with which two blocks share an SM: 32 bytes spill, and at 134 blocks of more than 192
// threads had an SM each (2,043 rows of q 6,144, k 1,024: 47 us feature by feature, 58 with one block, 33 so).
// ------------------------------------------------------------------------------------------
template <typename T, int NV>
__global__ void __launch_bounds__(256, NV == 8 ? 2 : 0)
wide_norm_store_vec_kernel(const float* proj, int ld, int q_width, int k_width, int v_col, int head_dim, const void* __restrict__ qw,
                           const void* __restrict__ kw, int w_dtype, float eps, T* q_out, const int* slots, T* pages, int page_size) {
  const int n = blockIdx.x, both = q_width + k_width;
  const float* row = proj + (size_t)n * ld;
  const float4 one = make_float4(1.f, 1.f, 1.f, 1.f);
  float4 wt[NV], v[NV], val[NV];
#pragma unroll
  for (int j = 0; j < NV; ++j) {
    const int e = (threadIdx.x + j * blockDim.x) * 4;
    wt[j] = one;
    if (e < q_width) { if (qw) wt[j] = sl_load4(qw, w_dtype, e); }
    else if (e < both && kw) wt[j] = sl_load4(kw, w_dtype, e - q_width);
  }
  ifb_pdl_wait();
  ifb_pdl_trigger();
  const int slot = slots ? slots[n] : -1;
  float sq = 0.f, sk = 0.f;
#pragma unroll
  for (int j = 0; j < NV; ++j) {
    const int e = (threadIdx.x + j * blockDim.x) * 4;
    v[j] = e < both ? *reinterpret_cast<const float4*>(row + e) : make_float4(0.f, 0.f, 0.f, 0.f);
    val[j] = v[j];
    if (v_col >= 0 && e >= q_width && e < both) val[j] = *reinterpret_cast<const float4*>(row + v_col + e - q_width);
  }
#pragma unroll
  for (int j = 0; j < NV; ++j) {
    const int e = (threadIdx.x + j * blockDim.x) * 4;
    if (e < q_width) sq = sl_square(v[j], sq);
    else sk = sl_square(v[j], sk);
  }
  const float2 sum = sl_block_sum(sq, sk);
  const float rq = qw ? 1.f / sqrtf(sum.x / (float)q_width + eps) : 1.f, rk = kw ? 1.f / sqrtf(sum.y / (float)k_width + eps) : 1.f;
  const int kv_heads = k_width / head_dim;
  const size_t head_stride = (size_t)page_size * head_dim;
  T* kp = slot < 0 ? nullptr : pages + (size_t)(slot / page_size) * 2 * kv_heads * head_stride + (size_t)(slot % page_size) * head_dim;
#pragma unroll
  for (int j = 0; j < NV; ++j) {
    const int e = (threadIdx.x + j * blockDim.x) * 4;
    if (e >= both) continue;
    const bool is_q = e < q_width;
    const float r = is_q ? rq : rk;
    const float4 o = make_float4(v[j].x * r * wt[j].x, v[j].y * r * wt[j].y, v[j].z * r * wt[j].z, v[j].w * r * wt[j].w);
    if (is_q) sl_store4(q_out + (size_t)n * q_width + e, o);
    else if (kp) {
      const int at = e - q_width;
      T* dst = kp + (size_t)(at / head_dim) * head_stride + at % head_dim;
      sl_store4(dst, o);
      sl_store4(dst + (size_t)kv_heads * head_stride, val[j]);
    }
  }
}

template <typename T>
__global__ void __launch_bounds__(256)
wide_norm_store_kernel(const float* __restrict__ proj, int ld, int q_width, int k_width, int v_col, int head_dim,
                       const void* __restrict__ qw, const void* __restrict__ kw, int w_dtype, float eps,
                       T* __restrict__ q_out, const int* __restrict__ slots, T* __restrict__ pages, int page_size) {
  __shared__ float scratch[33];
  ifb_pdl_wait();
  ifb_pdl_trigger();
  const int n = blockIdx.x;
  const float* row = proj + (size_t)n * ld;
  float sq = 0.f, sk = 0.f;
  if (qw) for (int e = threadIdx.x; e < q_width; e += blockDim.x) { const float v = row[e]; sq += v * v; }
  if (kw) for (int e = threadIdx.x; e < k_width; e += blockDim.x) { const float v = row[q_width + e]; sk += v * v; }
  const float rq = qw ? 1.f / sqrtf(block_sum(sq, scratch) / (float)q_width + eps) : 1.f;
  const float rk = kw ? 1.f / sqrtf(block_sum(sk, scratch) / (float)k_width + eps) : 1.f;
  for (int e = threadIdx.x; e < q_width; e += blockDim.x)
    q_out[(size_t)n * q_width + e] = from_f32<T>(qw ? row[e] * rq * load_as_f32(qw, w_dtype, e) : row[e]);
  const int slot = slots ? slots[n] : -1;
  if (slot < 0) return;
  const int kv_heads = k_width / head_dim;
  const size_t head_stride = (size_t)page_size * head_dim;
  T* kp = pages + (size_t)(slot / page_size) * 2 * kv_heads * head_stride + (size_t)(slot % page_size) * head_dim;
  T* vp = kp + (size_t)kv_heads * head_stride;
  for (int e = threadIdx.x; e < k_width; e += blockDim.x) {
    const int g = e / head_dim, d = e % head_dim;
    const float k = row[q_width + e];
    kp[(size_t)g * head_stride + d] = from_f32<T>(kw ? k * rk * load_as_f32(kw, w_dtype, e) : k);
    vp[(size_t)g * head_stride + d] = from_f32<T>(v_col < 0 ? k : row[v_col + e]);
  }
}

IFB_EXPORT int ifb_wide_norm_store(const float* proj, int ld, int q_width, int k_width, int v_col, int head_dim, const void* qw,
                                   const void* kw, int w_dtype, float eps, void* q_out, int out_dtype, const int* slots,
                                   void* pages, int page_size, int n, cudaStream_t stream) {
  if (n <= 0) return IFB_OK;
  if (head_dim < 1 || k_width % head_dim || q_width % head_dim || page_size < 1) return IFB_ERR_ARG;
  if (w_dtype != IFB_F32 && w_dtype != IFB_BF16) return IFB_ERR_DTYPE;
  const int both = q_width + k_width;
  if ((out_dtype == IFB_F32 || out_dtype == IFB_BF16) && both <= 8192 && q_width % 4 == 0 && k_width % 4 == 0 && head_dim % 4 == 0 && ld % 4 == 0 &&
      (v_col < 0 || v_col % 4 == 0) &&
      (((uintptr_t)proj | (uintptr_t)qw | (uintptr_t)kw | (uintptr_t)q_out | (uintptr_t)(slots ? pages : nullptr)) & 15) == 0) {
#define SL_VEC(T, NV)                                                                                                                \
  if (both <= NV * 1024)                                                                                                             \
    return ifb_launch(wide_norm_store_vec_kernel<T, NV>, dim3(n), dim3(sl_threads(both, NV)), 0, stream, proj, ld, q_width, k_width, v_col,     \
                      head_dim, qw, kw, w_dtype, eps, (T*)q_out, slots, (T*)pages, page_size);
    if (out_dtype == IFB_F32) { SL_VEC(float, 1) SL_VEC(float, 2) SL_VEC(float, 4) SL_VEC(float, 8) }
    else { SL_VEC(__nv_bfloat16, 1) SL_VEC(__nv_bfloat16, 2) SL_VEC(__nv_bfloat16, 4) SL_VEC(__nv_bfloat16, 8) }
#undef SL_VEC
  }
  if (out_dtype == IFB_F32)
    return ifb_launch(wide_norm_store_kernel<float>, dim3(n), dim3(256), 0, stream, proj, ld, q_width, k_width, v_col, head_dim,
                      qw, kw, w_dtype, eps, (float*)q_out, slots, (float*)pages, page_size);
  if (out_dtype == IFB_BF16)
    return ifb_launch(wide_norm_store_kernel<__nv_bfloat16>, dim3(n), dim3(256), 0, stream, proj, ld, q_width, k_width, v_col,
                      head_dim, qw, kw, w_dtype, eps, (__nv_bfloat16*)q_out, slots, (__nv_bfloat16*)pages, page_size);
  return IFB_ERR_DTYPE;
}
