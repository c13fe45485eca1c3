// Attention over the paged cache, plain float32 arithmetic, in two forms: float32 storage with heads of a multiple of four
// elements takes the shared-keys kernel below; bfloat16 storage and other head sizes one warp per (query token, query head).
// It serves every way a step can be cut (whole prompts, portions, single decoded tokens, mixed),
// any head size up to 256, any number of heads and groups, any page size, with or without a
// window, in float32 and in bfloat16 storage.  Scores, softmax and the weighted sum are float32.
//
// A query at position p reads the keys at positions first .. p from the pages its request's block
// table names, first = max(0, p - window + 1) with a window, else 0.  Block-table entries below
// `first` may be stale (-1): they are never read.
#include "common.cuh"
#include <math.h>
#include <type_traits>

#define ATT_MAX_D 256

template <typename T>
__global__ void __launch_bounds__(128)
paged_attention_simt_kernel(const T* __restrict__ qkv, int row_stride, const T* __restrict__ pages,
                            const int* __restrict__ block_tables, int bt_stride, const int* __restrict__ cu_q,
                            const int* __restrict__ seq_lens, T* __restrict__ out, int n_tokens, int n_req, int nq,
                            int nkv, int d, int page_size, float scale, int window) {
  extern __shared__ float sm[];
  ifb_pdl_wait();
  ifb_pdl_trigger();
  const int warps = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long item = (long long)blockIdx.x * warps + warp;
  if (item >= (long long)n_tokens * nq) return;
  const int tok = (int)(item / nq), h = (int)(item % nq);
  const int kvh = h / (nq / nkv);
  int lo = 0, hi = n_req;
  while (hi - lo > 1) { const int mid = (lo + hi) >> 1; if (cu_q[mid] <= tok) lo = mid; else hi = mid; }
  const int r = lo;
  T* o = out + (size_t)tok * nq * d + (size_t)h * d;
  if (tok >= cu_q[n_req]) { for (int i = lane; i < d; i += 32) o[i] = from_f32<T>(0.f); return; }
  const int q_len = cu_q[r + 1] - cu_q[r];
  const int p = seq_lens[r] - q_len + (tok - cu_q[r]);
  if (p < 0) { for (int i = lane; i < d; i += 32) o[i] = from_f32<T>(0.f); return; }
  const int first = window > 0 ? max(0, p - window + 1) : 0;
  float* qs = sm + (size_t)warp * d;
  const T* qp = qkv + (size_t)tok * row_stride + (size_t)h * d;
  for (int i = lane; i < d; i += 32) qs[i] = to_f32<T>(qp[i]);
  __syncwarp();
  const int* bt = block_tables + (size_t)r * bt_stride;
  const size_t head_stride = (size_t)page_size * d, page_stride = 2 * (size_t)nkv * head_stride;
  float m = -INFINITY, l = 0.f;
  float acc[ATT_MAX_D / 32];
#pragma unroll
  for (int c = 0; c < ATT_MAX_D / 32; ++c) acc[c] = 0.f;
  for (int kb = first; kb <= p; kb += 32) {
    const int key = kb + lane;
    const bool valid = key <= p;
    float s = -INFINITY;
    if (valid) {
      const int page = bt[key / page_size];
      const T* kp = pages + (size_t)page * page_stride + (size_t)kvh * head_stride + (size_t)(key % page_size) * d;
      float dot = 0.f;
      for (int i = 0; i < d; ++i) dot = fmaf(qs[i], to_f32<T>(kp[i]), dot);
      s = dot * scale;
    }
    const float m_new = fmaxf(m, warp_max(s));
    const float pj = valid ? expf(s - m_new) : 0.f;
    const float corr = expf(m - m_new);
    l = l * corr + warp_sum(pj);
#pragma unroll
    for (int c = 0; c < ATT_MAX_D / 32; ++c) acc[c] *= corr;
    const int count = min(32, p - kb + 1);
    for (int jj = 0; jj < count; ++jj) {
      const float pv = __shfl_sync(0xffffffffu, pj, jj);
      const int kj = kb + jj;
      const int page = bt[kj / page_size];
      const T* vp = pages + (size_t)page * page_stride + ((size_t)nkv + kvh) * head_stride + (size_t)(kj % page_size) * d;
#pragma unroll
      for (int c = 0; c < ATT_MAX_D / 32; ++c) {
        const int dim = lane + 32 * c;
        if (dim < d) acc[c] = fmaf(pv, to_f32<T>(vp[dim]), acc[c]);
      }
    }
    m = m_new;
  }
  const float inv = 1.f / l;
#pragma unroll
  for (int c = 0; c < ATT_MAX_D / 32; ++c) {
    const int dim = lane + 32 * c;
    if (dim < d) o[dim] = from_f32<T>(acc[c] * inv);
  }
}

// ---------------------------------------------------------------------------------------------------
// Float32 storage.  A CTA takes up to QT queries that share a key head (the heads of its group, and several consecutive
// tokens where a step has more tokens than requests).  Its W warps take the blocks of 32 keys in turn (block b goes to
// warp b mod W: which warp sums what depends on the keys' positions alone, so a query's result does not depend on the
// step it is part of), each warp with a softmax of its own, and the warps' results are merged in a fixed order.  Within a block a
// lane owns a key: the block goes through shared memory (rows padded by 16 bytes: conflict-free 16-byte reads) and each
// 16 bytes of it serve all queries; for the weighted sum a lane owns 4 (or 8) elements of the head and reads whole rows
// of values.  What bounds it is the chain of round trips of a block for few keys, and shared-memory reads for many.
// Eight queries (a prompt): the keys of a block come in pieces of 32 features, one piece ahead of the one that is being used: 9 KB of a warp
// whatever the head (whole rows take 16.5 KB at 128, 33 at 256, and 8.5 at 64 and less), so that two CTAs share an SM, and which queries see a
// row is a bit each, found with the scores.  Heads of 64 and less gain nothing in memory and as much in time by it.  Two queries and a CTA to an
// SM (AHEAD; a decoded token): whole rows at once, and all of a block's values are requested before its scores are formed, as a warp has one block or
// two and its time is that chain.  The registers that the CTAs of an SM leave do not hold all: eight queries spill 76 bytes (128 registers), with
// heads above 128 104 bytes (168), four queries with such heads 12.
// Us, 16 heads over 8, whole rows and now: 193 tokens 43 to 26 at heads of 64, 52 to 34 at 128, 83 to 44 at 192, 129 to 51 at 256; 1,000 tokens 446
// to 222, 540 to 291, 801 to 450, 1,444 to 524; one token at 195 keys 8.7 to 7.1, 10.0 to 8.3, 22.8 to 17.9, 24.8 to 20.1.  (A warp per query and
// head that read keys with a stride of a row took 156 for the 193 tokens and 155 for the one, at 128.)
// ---------------------------------------------------------------------------------------------------
constexpr int S32_PITCH = 36;                                   // floats of a row of a piece: 16-byte reads without conflicts
template <int QT, int DC, int W, bool AHEAD>
__global__ void __launch_bounds__(W * 32, AHEAD ? 1 : W == 8 ? 2 : QT == 8 ? 3 : 4)
paged_attention_shared32_kernel(const float* __restrict__ qkv, int row_stride, const float* __restrict__ pages,
                                const int* __restrict__ block_tables, int bt_stride, const int* __restrict__ cu_q,
                                const int* __restrict__ seq_lens, float* __restrict__ out, int n_tokens, int n_req, int nq,
                                int nkv, int d, int page_size, float scale, int window, int tokens_per_cta, int heads_per_cta) {
  extern __shared__ __align__(16) float sm[];
  ifb_pdl_wait();
  ifb_pdl_trigger();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  constexpr bool PIECES = QT == 8;
  constexpr int VB = AHEAD ? 32 : 8 / DC;                          // rows of values requested at a time
  const int pitch = d + 4, d4 = d / 4, row_step = 32 / d4, c_step = 32 % d4;
  float* qs = sm;                                               // [QT][d]
  float* ps = qs + QT * d;                                      // [W][QT][32]: a block's weights
  float* ml = ps + W * QT * 32;                                 // [W][QT][2]: maximum and sum of a warp, then its factor
  float* keys = ml + W * QT * 2;                                // [W][32][pitch] (PIECES: [W][2][32][S32_PITCH]), later [W][QT][d]: the warps' sums
  float* kr = keys + (size_t)warp * (PIECES ? 64 * S32_PITCH : 32 * pitch);
  const int rep = nq / nkv, chunks = (rep + heads_per_cta - 1) / heads_per_cta;
  const int kvh = blockIdx.y / chunks, hlo = (blockIdx.y % chunks) * heads_per_cta;
  const int nh = min(heads_per_cta, rep - hlo), h0 = kvh * rep + hlo;
  const size_t head_stride = (size_t)page_size * d, page_stride = 2 * (size_t)nkv * head_stride;
  const int t_end = min(n_tokens, ((int)blockIdx.x + 1) * tokens_per_cta);
  for (int t = blockIdx.x * tokens_per_cta; t < t_end;) {
    // the tokens t .. run - 1 belong to one request
    const bool padding = t >= cu_q[n_req];
    int r = 0;
    for (int hi = n_req; hi - r > 1;) { const int mid = (r + hi) >> 1; if (cu_q[mid] <= t) r = mid; else hi = mid; }
    const int run = padding ? t_end : min(t_end, cu_q[r + 1]);
    const int queries = (run - t) * nh;
    const int p0 = padding ? -QT : seq_lens[r] - (cu_q[r + 1] - t);      // position of token t; negative: sees nothing
    const int last = padding ? -1 : p0 + (run - t) - 1, first = window > 0 ? max(0, p0 - window + 1) : 0;
    __syncthreads();                                            // the shared memory of the tokens before is done with
    for (int i = tid; i < queries * d; i += W * 32) {
      const int j = i / d;
      qs[i] = qkv[(size_t)(t + j / nh) * row_stride + (size_t)(h0 + j % nh) * d + i % d];
    }
    for (int i = queries * d + tid; i < QT * d; i += W * 32) qs[i] = 0.f;
    __syncthreads();
    float m[QT], l[QT], acc[QT][DC * 4];
#pragma unroll
    for (int q = 0; q < QT; ++q) {
      m[q] = -INFINITY; l[q] = 0.f;
#pragma unroll
      for (int c = 0; c < DC * 4; ++c) acc[q][c] = 0.f;
    }
    const int* bt = block_tables + (size_t)r * bt_stride;
    const int b_first = first / 32;
    for (int b = b_first + (warp + W - b_first % W) % W; b * 32 <= last; b += W) {
      const int key = b * 32 + lane;
      const float* kp = nullptr;
      if (key >= first && key <= last)
        kp = pages + (size_t)bt[key / page_size] * page_stride + (size_t)kvh * head_stride + (size_t)(key % page_size) * d;
      const unsigned long long vp = (unsigned long long)(kp ? kp + (size_t)nkv * head_stride : nullptr);
      float4 v[VB][DC];
      auto values = [&](int j0) {
#pragma unroll
        for (int jj = 0; jj < VB; ++jj) {
          const float* row = (const float*)__shfl_sync(0xffffffffu, vp, j0 + jj);      // warp-uniform
#pragma unroll
          for (int c = 0; c < DC; ++c) {
            const int dim = (c * 32 + lane) * 4;
            v[jj][c] = row && dim < d ? *reinterpret_cast<const float4*>(row + dim) : make_float4(0.f, 0.f, 0.f, 0.f);
          }
        }
      };
      float s[QT];
#pragma unroll
      for (int q = 0; q < QT; ++q) s[q] = 0.f;
      // 16 bytes of this lane's key, at `at`, for all queries
      auto scores = [&](const float* at, int c) {
        const float4 k4 = *reinterpret_cast<const float4*>(at);
#pragma unroll
        for (int q = 0; q < QT; ++q) {
          const float4 q4 = *reinterpret_cast<const float4*>(qs + q * d + c * 4);
          s[q] = fmaf(q4.x, k4.x, s[q]);
          s[q] = fmaf(q4.y, k4.y, s[q]);
          s[q] = fmaf(q4.z, k4.z, s[q]);
          s[q] = fmaf(q4.w, k4.w, s[q]);
        }
      };
      if constexpr (PIECES) {
        const int pieces = (d4 + 7) / 8;
        auto piece = [&](int i) {                               // 8 lanes bring 128 bytes of a row, four rows at a time
          float* to = kr + (i & 1) * 32 * S32_PITCH + (lane & 7) * 4;
          const int c = i * 8 + (lane & 7);
#pragma unroll
          for (int it = 0; it < 8; ++it) {
            const int row = it * 4 + (lane >> 3);
            const float* src = (const float*)__shfl_sync(0xffffffffu, (unsigned long long)kp, row);
            if (src && c < d4) {
              const uint32_t dst = (uint32_t)__cvta_generic_to_shared(to + row * S32_PITCH);
              asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(src + c * 4) : "memory");
            }
          }
          asm volatile("cp.async.commit_group;\n" ::: "memory");
        };
        piece(0);
#pragma unroll 1
        for (int i = 0; i < pieces; ++i) {
          if (i + 1 < pieces) {
            piece(i + 1);
            asm volatile("cp.async.wait_group 1;\n" ::: "memory");
          } else {
            asm volatile("cp.async.wait_group 0;\n" ::: "memory");
          }
          __syncwarp();
          const float* at = kr + (i & 1) * 32 * S32_PITCH + lane * S32_PITCH;
          const int n = min(8, d4 - i * 8);
#pragma unroll 4
          for (int c = 0; c < n; ++c) scores(at + c * 4, i * 8 + c);
          __syncwarp();                                         // the piece after the next overwrites this one
        }
      } else {
        // 16 bytes per lane, row by row; lane's place moves on by 32 pieces at a time
        for (int it = 0, row = lane / d4, c = lane % d4; it < d4; ++it) {
          const float* src = (const float*)__shfl_sync(0xffffffffu, (unsigned long long)kp, row);
          if (src) {
            const uint32_t dst = (uint32_t)__cvta_generic_to_shared(kr + row * pitch + c * 4);
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(src + c * 4) : "memory");
          }
          row += row_step; c += c_step;
          if (c >= d4) { c -= d4; ++row; }
        }
        if (AHEAD) values(0);
        asm volatile("cp.async.wait_all;\n" ::: "memory");
        __syncwarp();
#pragma unroll 4
        for (int c = 0; c < d4; ++c) scores(kr + lane * pitch + c * 4, c);
      }
      uint32_t sees = 0;                                        // the queries that see this lane's key
      int p = p0, of = 0;
#pragma unroll
      for (int q = 0; q < QT; ++q) {
        const bool seen = q < queries && kp && key <= p && (window <= 0 || key > p - window);
        sees |= (seen ? 1u : 0u) << q;
        if (++of == nh) { of = 0; ++p; }
        const float sv = seen ? s[q] * scale : -INFINITY;
        const float m_new = fmaxf(m[q], warp_max(sv));
        // nothing seen so far, or scores of minus infinity alone (a block of them may be all that this warp sees): no weight, nothing
        // to rescale
        const float pj = seen && (sv != -INFINITY || m_new != -INFINITY) ? expf(sv - m_new) : 0.f;
        const float corr = m_new == -INFINITY ? 1.f : expf(m[q] - m_new);
        l[q] = l[q] * corr + warp_sum(pj);
        m[q] = m_new;
#pragma unroll
        for (int c = 0; c < DC * 4; ++c) acc[q][c] *= corr;
        ps[(warp * QT + q) * 32 + lane] = pj;
      }
      __syncwarp();
#pragma unroll 1
      for (int j0 = 0; j0 < 32; j0 += VB) {
        if (!AHEAD) values(j0);
        constexpr int G = 4;                                    // rows whose weights are read at once
        static_assert(VB % G == 0, "whole groups of rows");
#pragma unroll
        for (int g = 0; g < VB; g += G) {
          uint32_t row[G], any = 0, all = (1u << queries) - 1;
#pragma unroll
          for (int jj = 0; jj < G; ++jj) {
            row[jj] = __shfl_sync(0xffffffffu, sees, j0 + g + jj);
            any |= row[jj];
            all &= row[jj];
          }
          if (!any) continue;                                   // warp-uniform
          // a row that some query does not see is left out of that query's sum, not added with weight 0
          auto add = [&](auto every) {
#pragma unroll
            for (int q = 0; q < QT; ++q) {
              float pv[G];
              const float* at = ps + (warp * QT + q) * 32 + j0 + g;
              *reinterpret_cast<float4*>(pv) = *reinterpret_cast<const float4*>(at);
#pragma unroll
              for (int jj = 0; jj < G; ++jj) {
                if (!decltype(every)::value && !((row[jj] >> q) & 1)) continue;
#pragma unroll
                for (int c = 0; c < DC; ++c) {
                  const float4 x = v[g + jj][c];
                  acc[q][c * 4] = fmaf(pv[jj], x.x, acc[q][c * 4]);
                  acc[q][c * 4 + 1] = fmaf(pv[jj], x.y, acc[q][c * 4 + 1]);
                  acc[q][c * 4 + 2] = fmaf(pv[jj], x.z, acc[q][c * 4 + 2]);
                  acc[q][c * 4 + 3] = fmaf(pv[jj], x.w, acc[q][c * 4 + 3]);
                }
              }
            }
          };
          if (all == (1u << queries) - 1) add(std::true_type());
          else add(std::false_type());
        }
      }
      __syncwarp();                                             // the next block overwrites the keys and the weights
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < QT; ++q) {
#pragma unroll
      for (int c = 0; c < DC; ++c) {
        const int dim = (c * 32 + lane) * 4;
        if (dim < d)
          *reinterpret_cast<float4*>(keys + (size_t)(warp * QT + q) * d + dim) =
              make_float4(acc[q][c * 4], acc[q][c * 4 + 1], acc[q][c * 4 + 2], acc[q][c * 4 + 3]);
      }
      if (lane == 0) { ml[(warp * QT + q) * 2] = m[q]; ml[(warp * QT + q) * 2 + 1] = l[q]; }
    }
    __syncthreads();
    for (int i = tid; i < queries * d; i += W * 32) {
      const int q = i / d;
      float top = -INFINITY;
#pragma unroll
      for (int w = 0; w < W; ++w) top = fmaxf(top, ml[(w * QT + q) * 2]);
      float total = 0.f, sum = 0.f;
      if (top != -INFINITY) {
#pragma unroll
        for (int w = 0; w < W; ++w) {
          const float f = expf(ml[(w * QT + q) * 2] - top);      // 0 for a warp that saw no key, whose sums are 0
          total = fmaf(f, ml[(w * QT + q) * 2 + 1], total);
          sum = fmaf(f, keys[(size_t)(w * QT + q) * d + i % d], sum);
        }
      }
      const bool sees = p0 + q / nh >= 0;
      out[((size_t)(t + q / nh) * nq + h0 + q % nh) * d + i % d] = sees ? sum / total : 0.f;
    }
    t = run;
  }
}

template <int QT, int DC, int W, bool AHEAD = false>
static int shared32_launch(const float* qkv, int row_stride, const float* pages, const int* block_tables, int bt_stride, const int* cu_q,
                           const int* seq_lens, float* out, int n_tokens, int n_req, int nq, int nkv, int d, int page_size, float scale,
                           int window, int tokens, int heads, cudaStream_t stream) {
  const size_t keys = QT == 8 ? 64 * S32_PITCH : 32 * (size_t)(d + 4), sums = (size_t)QT * d;      // of a warp, in the same place
  const size_t smem = ((size_t)QT * d + W * QT * 34 + W * (keys > sums ? keys : sums)) * sizeof(float);
  IFB_ALLOW_SMEM((paged_attention_shared32_kernel<QT, DC, W, AHEAD>), smem);
  const int chunks = (nq / nkv + heads - 1) / heads;
  // the values ahead take the registers of a second CTA per SM: where one has an SM to itself, for want of CTAs or of shared memory
  // (16 heads of 64: 64 tokens at 300 keys, 1,024 CTAs, 73 us without, 111 so)
  if constexpr (QT == 2 && DC == 1 && !AHEAD)
    if ((long long)((n_tokens + tokens - 1) / tokens) * nkv * chunks <= ifb_sm_count() || smem > 113 * 1024)
      return shared32_launch<QT, DC, W, true>(qkv, row_stride, pages, block_tables, bt_stride, cu_q, seq_lens, out, n_tokens, n_req, nq, nkv, d,
                                              page_size, scale, window, tokens, heads, stream);
  return ifb_launch(paged_attention_shared32_kernel<QT, DC, W, AHEAD>, dim3((n_tokens + tokens - 1) / tokens, nkv * chunks), dim3(W * 32), smem,
                    stream, qkv, row_stride, pages, block_tables, bt_stride, cu_q, seq_lens, out, n_tokens, n_req, nq, nkv, d,
                    page_size, scale, window, tokens, heads);
}

IFB_EXPORT int ifb_paged_attention_simt(const void* qkv, int dtype, int row_stride, const void* pages,
                                        const int* block_tables, int bt_stride, const int* cu_q, const int* seq_lens,
                                        void* out, int n_tokens, int n_req, int nq, int nkv, int d, int page_size,
                                        float scale, int window, cudaStream_t stream) {
  if (n_tokens <= 0 || n_req <= 0) return IFB_OK;
  if (d < 1 || d > ATT_MAX_D) return IFB_ERR_SIZE;
  if (nkv < 1 || nq % nkv || page_size < 1 || window < 0) return IFB_ERR_ARG;
  if (dtype == IFB_F32 && d % 4 == 0 && row_stride % 4 == 0 && !(((uintptr_t)qkv | (uintptr_t)pages | (uintptr_t)out) & 15) &&
      (long long)nkv * ((nq / nkv + 7) / 8) <= 65535) {
    // one token per CTA where every request brings one (more would be one request after the other), else as many as make
    // eight queries; of large groups eight heads at a time
    const int heads = nq / nkv < 8 ? nq / nkv : 8, tokens = n_tokens <= n_req ? 1 : 8 / heads;
    const int queries = tokens * heads;
    const float *q = (const float*)qkv, *pg = (const float*)pages;
    float* o = (float*)out;
#define IFB_SHARED32(QT, DC, W) \
  return shared32_launch<QT, DC, W>(q, row_stride, pg, block_tables, bt_stride, cu_q, seq_lens, o, n_tokens, n_req, nq, nkv, d, page_size, \
                                    scale, window, tokens, heads, stream)
    if (d <= 128) {
      if (queries <= 2) IFB_SHARED32(2, 1, 8);
      if (queries <= 4) IFB_SHARED32(4, 1, 8);
      IFB_SHARED32(8, 1, 8);
    }
    if (queries <= 2) IFB_SHARED32(2, 2, 4);
    if (queries <= 4) IFB_SHARED32(4, 2, 4);
    IFB_SHARED32(8, 2, 4);
#undef IFB_SHARED32
  }
  const int warps = 4;
  const long long items = (long long)n_tokens * nq;
  const unsigned blocks = (unsigned)((items + warps - 1) / warps);
  const size_t smem = (size_t)warps * d * sizeof(float);
  if (dtype == IFB_F32)
    return ifb_launch(paged_attention_simt_kernel<float>, dim3(blocks), dim3(warps * 32), smem, stream, (const float*)qkv,
                      row_stride, (const float*)pages, block_tables, bt_stride, cu_q, seq_lens, (float*)out, n_tokens, n_req,
                      nq, nkv, d, page_size, scale, window);
  if (dtype == IFB_BF16)
    return ifb_launch(paged_attention_simt_kernel<__nv_bfloat16>, dim3(blocks), dim3(warps * 32), smem, stream,
                      (const __nv_bfloat16*)qkv, row_stride, (const __nv_bfloat16*)pages, block_tables, bt_stride, cu_q,
                      seq_lens, (__nv_bfloat16*)out, n_tokens, n_req, nq, nkv, d, page_size, scale, window);
  return IFB_ERR_DTYPE;
}
