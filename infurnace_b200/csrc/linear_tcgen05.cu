// Matrix product for many rows (prompts): out[n, o] = sum_k x[n, k] w[o, k], bfloat16 operands,
// float32 accumulation, on the fifth-generation tensor cores: tcgen05.mma issued by one thread, operands
// brought to shared memory by TMA (128-byte swizzle), the accumulator in tensor memory, read back with
// tcgen05.ld for the epilogue.
//
// A CTA of 320 threads takes one output tile:
//   warp 0: TMA producer.  Per 64-wide k block it waits for a free stage, arms the stage's "full" barrier with
//           the byte count and issues the loads of the x tile and the w tile(s).
//   warp 1: MMA issuer.  It waits for "full", issues the k=16 MMAs of the stage and commits them to the stage's
//           "empty" barrier, so the stage is reused as soon as the tensor core has read it.  After the last
//           k block it commits to the "accumulator ready" barrier.  Warp 1 also owns the tensor memory.
//   warps 2-9: epilogue.  A warp reads its quarter (warp index mod 4) of the accumulator's 128 lanes, one token per
//           thread and half; warps 2-5 take the first half of the tile's features and warps 6-9 the second.
// In warps 0 and 1 all lanes wait and one elected lane issues.
// Rows, features or k beyond the matrices are zero-filled by TMA and dropped at the store.
//
// Tile shapes (GemmCfg): MH halves of 128 tokens share the w tile of a stage; each half accumulates NACC
// columns in tensor memory with one MMA of N = NACC per k step.
//   narrow  MH 1, NACC 128: 128 tokens x 128 features, 3 stages of 32 KB, two CTAs per SM;
//   deep    the same with 6 stages, for grids of at most one CTA per SM (o and down projections of prompts of
//           a few thousand tokens): the stages in flight are what hides the latency of the loads;
//   wide    MH 2, NACC 256: 256 tokens x 256 features, 3 stages of 64 KB, all 512 columns of tensor memory:
//           half the bytes from L2 per product of the narrow shape.
// Epilogue 1 (silu_gate): w holds gate rows [0, O) and up rows [O, 2O).  A stage carries a gate tile and an up
// tile back to back as one B operand, the accumulator's first NACC/2 columns are gate and the rest up, and
// out = silu(gate) * up has NACC/2 features per CTA (narrow: NACC 256).
//
// Every wait on a barrier is bounded: after G_SPIN_LIMIT polls the thread writes a code to `*err`, raises
// the CTA's abort flag, and everything falls through to the common exit, which frees the tensor memory.
#include <cuda.h>
#include "common.cuh"

typedef __nv_bfloat16 bf16;
constexpr int G_BM = 128;          // tokens per half tile (MMA M)
constexpr int G_BK = 64;           // k per stage: 128 bytes, one swizzle row
constexpr int G_UK = 16;           // k per MMA
constexpr int G_THREADS = 320;      // producer warp, MMA warp, eight epilogue warps
constexpr uint32_t G_SPIN_LIMIT = 1u << 22;
constexpr int G_TILE_BYTES = G_BM * G_BK * 2;   // 16 KB: 128 rows of one k block

template <int EPI_, int MH_, int NACC_, int STAGES_> struct GemmCfg {
  static constexpr int EPI = EPI_, MH = MH_, NACC = NACC_, STAGES = STAGES_;
  static constexpr int FO = EPI ? NACC / 2 : NACC;            // output features per CTA
  static constexpr int A_BYTES = MH * G_TILE_BYTES;           // x rows of a stage
  static constexpr int B_BYTES = NACC * G_BK * 2;             // w rows of a stage
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int TMEM_COLS = MH * NACC;                 // 128, 256 or 512 columns of 32 bits
  static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 /* alignment */ + 256 /* barriers */;
  static constexpr bool SHARED_K = MH == 1 && FO == 128 && 2 * SMEM_BYTES > 226 * 1024;      // the deep shapes: the k range may be shared by a cluster
  // float32 accumulator, bfloat16 a and b, both K-major, M = 128, N = NACC
  static constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(NACC >> 3) << 17) | ((uint32_t)(G_BM >> 4) << 24);
};

__device__ __forceinline__ uint32_t g_smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint64_t* bar, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(g_smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(g_smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
               : "=r"(ok) : "r"(g_smem_u32(bar)), "r"(parity) : "memory");
  return ok != 0;
}
// Bounded wait.  False: gave up (the abort flag is up and *err says where).
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int* err, int code) {
  unsigned long long t0 = 0;
  for (uint32_t i = 0; i < G_SPIN_LIMIT; ++i) {
    if (mbar_try_wait(bar, parity)) return true;
    if (*abort_flag) return false;
    if (ifb_wait_expired(i, t0)) break;
  }
  *abort_flag = 1;
  atomicExch(err, code);
  return false;
}
__device__ __forceinline__ void tma_load_2d(void* smem, const CUtensorMap* map, uint64_t* bar, int x, int y) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];\n"
               ::"r"(g_smem_u32(smem)), "l"(map), "r"(g_smem_u32(bar)), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void tmem_alloc(uint32_t* slot, int cols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(g_smem_u32(slot)), "r"(cols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish() { asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory"); }
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, int cols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(taddr), "r"(cols) : "memory");
}
// True in exactly one lane of a converged warp.  Code under it is known to the compiler as single-threaded, which lets
// it keep the descriptors of the copies and products it issues in uniform registers.
__device__ __forceinline__ bool elect_one() {
  uint32_t pred;
  asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(pred));
  return pred != 0;
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void umma_bf16(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n"
               ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(g_smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
        "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),
        "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
        "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr) : "memory");
}
__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;\n" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float fast_rcp(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;\n" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory"); }

// All threads of all CTAs of the cluster: arrive (release) and wait (acquire).
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}
// Four floats at this CTA's shared address `addr`, read from the CTA of rank `rank` in the cluster.
__device__ __forceinline__ float4 ld_cluster_f4(uint32_t addr, int rank) {
  uint32_t remote;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(remote) : "r"(addr), "r"(rank));
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];\n" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(remote) : "memory");
  return v;
}

template <int N> struct TcInt { static constexpr int value = N; };

// Shared-memory matrix descriptor of a K-major tile in the 128-byte swizzle: rows of 128 bytes, groups of 8
// rows 1024 bytes apart (stride byte offset), leading byte offset unused (1), descriptor version 1.
__device__ __forceinline__ uint64_t make_smem_desc(uint32_t smem_addr) {
  return (uint64_t)((smem_addr >> 4) & 0x3FFF) | (1ull << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}

// The gate's function with the hardware's exp2 and reciprocal (relative error about 1e-6; the result is rounded to the
// output type): silu, or gelu in the tanh form, which is g * sigmoid(2 sqrt(2/pi) (g + 0.044715 g^3)); others exactly.
__device__ __forceinline__ float tc_gate(float g, int kind) {
  if (kind != IFB_UNARY_NONE && kind != IFB_UNARY_GELU_TANH) return ifb_unary(g, kind);
  const float z = kind ? 1.5957691216057308f * fmaf(0.044715f * g * g, g, g) : g;
  return g * fast_rcp(1.f + fast_exp2(-1.4426950408889634f * z));
}

// The unary function on every element of a row's piece.  The function is chosen once: chosen per element, 32 copies of every
// function's code lie between one element and the next, and a launch waits for its code (2,043 x 3,072 x 1,024 with relu^2: 49 us
// for 15).
template <int N>
__device__ __forceinline__ void tc_unary(float (&y)[N], int kind) {
#define IFB_TC_UNARY(KIND) \
  case KIND: \
    _Pragma("unroll") for (int j = 0; j < N; ++j) y[j] = ifb_unary(y[j], KIND); \
    break;
  switch (kind) {
    IFB_TC_UNARY(IFB_UNARY_RELU2)
    IFB_TC_UNARY(IFB_UNARY_SILU)
    IFB_TC_UNARY(IFB_UNARY_SIGMOID)
    IFB_TC_UNARY(IFB_UNARY_GELU_TANH)
    IFB_TC_UNARY(IFB_UNARY_TANH)
  }
#undef IFB_TC_UNARY
}
static_assert(IFB_UNARY_LAST == IFB_UNARY_TANH, "tc_unary names every function");
// A row's piece of gates times its ups, the gate's function likewise chosen once (64 rows of 3,072 x 1,024 with a gelu gate: chosen
// per element 11.5 us, chosen once 6.1, as with silu).
template <int N>
__device__ __forceinline__ void tc_gates(float (&y)[N], const uint32_t (&gate)[N], const uint32_t (&up)[N], float rfac, int kind) {
#define IFB_TC_GATES(ACT) \
  _Pragma("unroll") for (int j = 0; j < N; ++j) { \
    const float g = __uint_as_float(gate[j]) * rfac; \
    y[j] = (ACT) * (__uint_as_float(up[j]) * rfac); \
  }
  switch (kind) {
    case IFB_UNARY_NONE: IFB_TC_GATES(tc_gate(g, IFB_UNARY_NONE)) break;
    case IFB_UNARY_GELU_TANH: IFB_TC_GATES(tc_gate(g, IFB_UNARY_GELU_TANH)) break;
    default: {
      float act[N];
#pragma unroll
      for (int j = 0; j < N; ++j) act[j] = __uint_as_float(gate[j]) * rfac;
      tc_unary(act, kind);
#pragma unroll
      for (int j = 0; j < N; ++j) y[j] = act[j] * (__uint_as_float(up[j]) * rfac);
    }
  }
#undef IFB_TC_GATES
}

// A normalisation folded into the products around it (RMSNorm(v) = v * g * r with one r per row): the product that
// makes v (plain epilogue) adds the residual stream, writes v back to it, writes v * g as its output and leaves sums of
// v^2 over slices of the features; the product that reads v * g multiplies its rows by r, from those sums added in a
// fixed order, before its own epilogue.  No kernel runs for the norm itself.
struct TcFold {
  const float* rs_partials;   // reading side: [rs_parts][n_rows] sums of squares (null: rows are not scaled)
  int rs_parts;
  float rs_eps, rs_inv_width; // r = rsqrt(sum * inv_width + eps)
  float* res_x;               // making side: [n_rows][o_out] float32 residual stream, v = x + y in place (null: plain)
  const void* res_g;          // [o_out] norm weight
  int res_g_dtype;
  float* res_partials;        // [parts][n_rows], written; what a part covers depends on the launch (tc_fold_parts)
  int unary;                  // without res_x: the function of common.cuh applied to every element (0: none), or to the gates (0: silu)
  const float* bias;          // plain epilogue: [o_out], added to the product before the unary function (null: none)
  // The product is the fused q | k | v projection of an attention layer with heads of 128; a tile's 128 features (or each
  // 128 of its 256) are one head: the epilogue, or the sum over the cluster in the shared-k form, finishes what follows the
  // projection (RMSNorm over the q and k heads, rotation in the half-split pairing, q to its row, k and v to the token's
  // place in the pages).
  int qk_nq, qk_nkv;          // qk_nq > 0: on
  const void* qk_qw;          // [128] norm weights (null: no norm)
  const void* qk_kw;
  int qk_w_dtype;
  float qk_eps;
  const float2* qk_rope;      // [n_rows][64] (cos, sin) of each token's angles (null: no rotation)
  const int* qk_slots;        // [n_rows] page * page_size + offset, negative: store nothing (null: no store)
  bf16* qk_pages;             // [page][k | v][kv head][offset][128]
  int qk_page_size;
  // The grouped product of routed experts (one tile of 128 rows per CTA, no cluster): w holds the experts' matrices one
  // after the other, grp_w_rows rows each; the rows of x are sorted by expert in segments padded to 128, and tile t of rows
  // belongs to expert grp_tile_expert[t] (negative: the tile is unused and its CTAs return at once).
  const int* grp_tile_expert; // null: off
  int grp_w_rows;
};
__device__ __forceinline__ float tc_row_factor(const TcFold& f, int row, int n_rows) {
  if (!f.rs_partials || row >= n_rows) return 1.f;
  float sum = 0.f;
#pragma unroll 4
  for (int p = 0; p < f.rs_parts; ++p) sum += f.rs_partials[(size_t)p * n_rows + row];
  return rsqrtf(sum * f.rs_inv_width + f.rs_eps);
}
// v = x + y for 32 consecutive features of one row (x updated in place), y <- v * g; returns the sum of v^2.
__device__ __forceinline__ float tc_residual_chunk(const TcFold& f, float (&y)[32], int row, int n_rows, int col0, int o_out) {
  float ss = 0.f;
  if (row >= n_rows) return 0.f;
  float* xr = f.res_x + (size_t)row * o_out + col0;
  if (col0 + 32 <= o_out && (o_out & 3) == 0) {
#pragma unroll
    for (int j = 0; j < 32; j += 4) {
      float4 xv = *reinterpret_cast<float4*>(xr + j);
      xv.x += y[j]; xv.y += y[j + 1]; xv.z += y[j + 2]; xv.w += y[j + 3];
      *reinterpret_cast<float4*>(xr + j) = xv;
      ss += xv.x * xv.x + xv.y * xv.y + xv.z * xv.z + xv.w * xv.w;
      y[j] = xv.x * load_as_f32(f.res_g, f.res_g_dtype, col0 + j);
      y[j + 1] = xv.y * load_as_f32(f.res_g, f.res_g_dtype, col0 + j + 1);
      y[j + 2] = xv.z * load_as_f32(f.res_g, f.res_g_dtype, col0 + j + 2);
      y[j + 3] = xv.w * load_as_f32(f.res_g, f.res_g_dtype, col0 + j + 3);
    }
  } else {
#pragma unroll
    for (int j = 0; j < 32; ++j)
      if (col0 + j < o_out) {
        const float v = xr[j] + y[j];
        xr[j] = v;
        ss += v * v;
        y[j] = v * load_as_f32(f.res_g, f.res_g_dtype, col0 + j);
      }
  }
  return ss;
}

// 32 columns of the accumulator (a lane's row of them) times `f`, as float32 at `dst`.
__device__ __forceinline__ void tc_stage_rows(uint32_t taddr, unsigned char* dst, float f) {
  uint32_t v[32];
  tmem_ld32(taddr, v);
  tmem_ld_wait();
#pragma unroll
  for (int j = 0; j < 32; j += 4)
    *reinterpret_cast<float4*>(dst + j * 4) = make_float4(__uint_as_float(v[j]) * f, __uint_as_float(v[j + 1]) * f,
                                                          __uint_as_float(v[j + 2]) * f, __uint_as_float(v[j + 3]) * f);
}
// The end of a product with the residual addition, for a warp's 32 rows of CW features: v = x + y goes back to x, v * g to
// `out`, the sum of v^2 over the CW features to its part.  CW / 4 lanes share a row, so every access of the stream is a whole
// row segment (a lane with a row of its own touches 32 rows per instruction: for a prompt of 2,048 rows that epilogue cost
// what the separate norm did).  Eight warps per SM hide no latency by themselves, so the stream's rows are requested AHEAD
// passes at a time, the first of them before the product is there.
template <int CW, int AHEAD>
__device__ __forceinline__ void tc_residual_load(const TcFold& f, int row0, int n_rows, int col0, int o_out, int lane, float4 (&xv)[AHEAD]) {
  constexpr int LPR = CW / 4, RPP = 32 / LPR;
#pragma unroll
  for (int a = 0; a < AHEAD; ++a) {
    const int row = row0 + a * RPP + lane / LPR;
    xv[a] = row < n_rows ? *reinterpret_cast<const float4*>(f.res_x + (size_t)row * o_out + col0 + (lane % LPR) * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
}
// `xv`: the first AHEAD passes' rows, requested by the caller before it waited for the product.
template <int CW, int PITCH, int AHEAD, typename TO>
__device__ __forceinline__ void tc_finish_residual(const TcFold& f, const unsigned char* rows32, TO* out, int row0, int n_rows, int col0,
                                                   int o_out, int part, int lane, float4 (&xv)[AHEAD]) {
  constexpr int LPR = CW / 4, RPP = 32 / LPR;
  static_assert(32 % (RPP * AHEAD) == 0, "whole batches of passes");
  const int sub = lane / LPR, c = (lane % LPR) * 4;
  const bool whole = (((uintptr_t)out) & (4 * sizeof(TO) - 1)) == 0;
  float g[4], bias[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    g[j] = load_as_f32(f.res_g, f.res_g_dtype, col0 + c + j);
    bias[j] = f.bias ? __ldg(f.bias + col0 + c + j) : 0.f;
  }
  constexpr int GROUP = 4;                                       // passes whose reads precede all their stores
  static_assert(AHEAD % GROUP == 0, "whole groups");
#pragma unroll 1
  for (int r0 = 0; r0 < 32; r0 += RPP * AHEAD) {
    if (row0 + r0 >= n_rows) break;                              // warp-uniform
    if (r0) tc_residual_load<CW, AHEAD>(f, row0 + r0, n_rows, col0, o_out, lane, xv);
#pragma unroll
    for (int a0 = 0; a0 < AHEAD; a0 += GROUP) {
      float4 v[GROUP];
      float ss[GROUP];
#pragma unroll
      for (int a = 0; a < GROUP; ++a) v[a] = *reinterpret_cast<const float4*>(rows32 + (r0 + (a0 + a) * RPP + sub) * PITCH + c * 4);
#pragma unroll
      for (int a = 0; a < GROUP; ++a) {
        const float4 x = xv[a0 + a];
        v[a] = make_float4(x.x + (v[a].x + bias[0]), x.y + (v[a].y + bias[1]), x.z + (v[a].z + bias[2]), x.w + (v[a].w + bias[3]));
        ss[a] = v[a].x * v[a].x + v[a].y * v[a].y + v[a].z * v[a].z + v[a].w * v[a].w;
      }
#pragma unroll
      for (int d = LPR / 2; d > 0; d >>= 1)
#pragma unroll
        for (int a = 0; a < GROUP; ++a) ss[a] += __shfl_xor_sync(0xffffffffu, ss[a], d);
#pragma unroll
      for (int a = 0; a < GROUP; ++a) {
        const int row = row0 + r0 + (a0 + a) * RPP + sub;
        if (row < n_rows) {
          *reinterpret_cast<float4*>(f.res_x + (size_t)row * o_out + col0 + c) = v[a];
          TO* dst = out + (size_t)row * o_out + col0 + c;
          const float h[4] = {v[a].x * g[0], v[a].y * g[1], v[a].z * g[2], v[a].w * g[3]};
          if (!whole) {
#pragma unroll
            for (int j = 0; j < 4; ++j) dst[j] = from_f32<TO>(h[j]);
          } else if (sizeof(TO) == 2) {
            __nv_bfloat162 lo = __floats2bfloat162_rn(h[0], h[1]), hi = __floats2bfloat162_rn(h[2], h[3]);
            *reinterpret_cast<uint2*>(dst) = make_uint2(*reinterpret_cast<uint32_t*>(&lo), *reinterpret_cast<uint32_t*>(&hi));
          } else {
            *reinterpret_cast<float4*>(dst) = make_float4(h[0], h[1], h[2], h[3]);
          }
          if (lane % LPR == 0) f.res_partials[(size_t)part * n_rows + row] = ss[a];
        }
      }
    }
  }
}
// The end of the fused q | k | v projection for a warp's 32 tokens and NP of the 64 rotation pairs of one head (elements
// i0 .. i0 + NP - 1 and their partners 64 further on, staged one after the other, already divided by the head's rms): norm
// weight, rotation, the head's row of `out`, and for k and v heads the token's place in the pages.  NP / 4 lanes share a token.
template <int NP, int AHEAD>
__device__ __forceinline__ void tc_heads_load(const TcFold& f, int row0, int n_rows, int i0, bool rotate, bool store, int lane,
                                              float4 (&cs)[AHEAD][2], int (&slot)[AHEAD]) {
  constexpr int LPR = NP / 4, RPP = 32 / LPR;
#pragma unroll
  for (int a = 0; a < AHEAD; ++a) {
    const int row = row0 + a * RPP + lane / LPR;
    const float4* t = reinterpret_cast<const float4*>(f.qk_rope + (size_t)row * 64 + i0 + (lane % LPR) * 4);
    const bool in = rotate && row < n_rows;
    cs[a][0] = in ? t[0] : make_float4(1.f, 0.f, 1.f, 0.f);
    cs[a][1] = in ? t[1] : make_float4(1.f, 0.f, 1.f, 0.f);
    slot[a] = store && row < n_rows ? f.qk_slots[row] : -1;
  }
}
// `cs`, `slot`: the first AHEAD passes' angles and places, requested by the caller before it waited for the product.
template <int NP, int PITCH, int AHEAD>
__device__ __forceinline__ void tc_finish_heads(const TcFold& f, const unsigned char* rows32, bf16* out, int row0, int n_rows, int head,
                                                int i0, int o_out, const void* wn, bool is_v, bool rotate, bool store, int lane,
                                                float4 (&cs)[AHEAD][2], int (&slot)[AHEAD]) {
  constexpr int LPR = NP / 4, RPP = 32 / LPR, GROUP = 2;         // passes whose reads precede all their stores
  static_assert(32 % (RPP * AHEAD) == 0 && AHEAD % GROUP == 0, "whole batches of passes, whole groups");
  const int sub = lane / LPR, p = (lane % LPR) * 4, i = i0 + p;
  float wa[4] = {1.f, 1.f, 1.f, 1.f}, wb[4] = {1.f, 1.f, 1.f, 1.f};
  if (wn) {
#pragma unroll
    for (int j = 0; j < 4; ++j) { wa[j] = load_as_f32(wn, f.qk_w_dtype, i + j); wb[j] = load_as_f32(wn, f.qk_w_dtype, 64 + i + j); }
  }
  const int kvh = is_v ? head - f.qk_nq - f.qk_nkv : head - f.qk_nq;
  const int ps_shift = (f.qk_page_size & (f.qk_page_size - 1)) ? -1 : __ffs(f.qk_page_size) - 1;
#pragma unroll 1
  for (int r0 = 0; r0 < 32; r0 += RPP * AHEAD) {
    if (row0 + r0 >= n_rows) break;                              // warp-uniform
    if (r0) tc_heads_load<NP, AHEAD>(f, row0 + r0, n_rows, i0, rotate, store, lane, cs, slot);
#pragma unroll
    for (int a0 = 0; a0 < AHEAD; a0 += GROUP) {
      float4 x[GROUP], y[GROUP];
#pragma unroll
      for (int a = 0; a < GROUP; ++a) {
        const unsigned char* at = rows32 + (r0 + (a0 + a) * RPP + sub) * PITCH + p * 4;
        x[a] = *reinterpret_cast<const float4*>(at);
        y[a] = *reinterpret_cast<const float4*>(at + NP * 4);
      }
      uint2 lo[GROUP], hi[GROUP];
#pragma unroll
      for (int a = 0; a < GROUP; ++a) {
        const float4 c0 = cs[a0 + a][0], c1 = cs[a0 + a][1];
        const float u[4] = {x[a].x * wa[0], x[a].y * wa[1], x[a].z * wa[2], x[a].w * wa[3]};
        const float v[4] = {y[a].x * wb[0], y[a].y * wb[1], y[a].z * wb[2], y[a].w * wb[3]};
        const float co[4] = {c0.x, c0.z, c1.x, c1.z}, si[4] = {c0.y, c0.w, c1.y, c1.w};
        float s[4], t[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          s[j] = rotate ? u[j] * co[j] - v[j] * si[j] : u[j];
          t[j] = rotate ? v[j] * co[j] + u[j] * si[j] : v[j];
        }
        const __nv_bfloat162 s0 = __floats2bfloat162_rn(s[0], s[1]), s1 = __floats2bfloat162_rn(s[2], s[3]);
        const __nv_bfloat162 t0 = __floats2bfloat162_rn(t[0], t[1]), t1 = __floats2bfloat162_rn(t[2], t[3]);
        lo[a] = make_uint2(*reinterpret_cast<const uint32_t*>(&s0), *reinterpret_cast<const uint32_t*>(&s1));
        hi[a] = make_uint2(*reinterpret_cast<const uint32_t*>(&t0), *reinterpret_cast<const uint32_t*>(&t1));
      }
#pragma unroll
      for (int a = 0; a < GROUP; ++a) {
        const int row = row0 + r0 + (a0 + a) * RPP + sub, sl = slot[a0 + a];
        if (row < n_rows) {
          bf16* dst = out + (size_t)row * o_out + head * 128 + i;
          *reinterpret_cast<uint2*>(dst) = lo[a];
          *reinterpret_cast<uint2*>(dst + 64) = hi[a];
        }
        if (sl >= 0) {
          const int page = ps_shift >= 0 ? sl >> ps_shift : sl / f.qk_page_size;
          const size_t at = ((size_t)page * 2 + (is_v ? 1 : 0)) * f.qk_nkv + kvh;
          bf16* pg = f.qk_pages + (at * f.qk_page_size + sl - page * f.qk_page_size) * 128 + i;
          *reinterpret_cast<uint2*>(pg) = lo[a];
          *reinterpret_cast<uint2*>(pg + 64) = hi[a];
        }
      }
    }
  }
}

// (CTAs per SM by shared memory: left to itself the compiler aims for more and takes 64 registers, with spills)
template <typename Cfg, typename TO>
__global__ void __launch_bounds__(G_THREADS, 2 * Cfg::SMEM_BYTES <= 226 * 1024 ? 2 : 1)
linear_tcgen05_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_w,
                      TO* __restrict__ out, int n_rows, int o_out, int k_dim, int* __restrict__ err,
                      int splits, TcFold fold) {
  constexpr int EPI = Cfg::EPI, MH = Cfg::MH, NACC = Cfg::NACC, FO = Cfg::FO;
  extern __shared__ unsigned char g_smem_raw[];
  const uint32_t raw = g_smem_u32(g_smem_raw);
  unsigned char* smem = g_smem_raw + (((raw + 1023u) & ~1023u) - raw);      // tiles need 1024-byte alignment
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + Cfg::STAGES * Cfg::STAGE_BYTES);
  uint64_t* empty = full + Cfg::STAGES;
  uint64_t* accum = empty + Cfg::STAGES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(accum + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;     // warp-uniform
  const int m0 = blockIdx.y * (MH * G_BM), n0 = blockIdx.x * FO;
  int w0 = n0;                                                    // first row of this tile's w rows
  if (fold.grp_tile_expert) {
    ifb_pdl_wait();                                               // the list of tiles is the predecessor's
    const int e = fold.grp_tile_expert[blockIdx.y];
    if (e < 0) { ifb_pdl_trigger(); return; }                     // an unused tile: before any barrier or tensor memory exists
    w0 = e * fold.grp_w_rows + n0;
  }
  // With splits > 1 (plain epilogue, one 128-row tile per CTA) the CTAs of a tile are a cluster along z: CTA z
  // multiplies the z-th part of the k range, leaves its float32 tile in its shared memory, and after a cluster barrier
  // adds, in the order of z, a slice of the tile's rows over all CTAs' copies and stores it.
  const int kb_all = (k_dim + G_BK - 1) / G_BK;
  const int kb_per = (kb_all + splits - 1) / splits;
  const int kb0 = blockIdx.z * kb_per;
  const int kblocks = max(0, min(kb_all, kb0 + kb_per) - kb0);    // this CTA's k blocks are kb0 .. kb0 + kblocks - 1
  constexpr int RED_PITCH = NACC + 4;                             // floats per row of the tile left in shared memory

  if (threadIdx.x == 0) {
    for (int s = 0; s < Cfg::STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    mbar_init(accum, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
  }
  if (warp == 1) { tmem_alloc(tmem_slot, Cfg::TMEM_COLS); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  // What the sum over the cluster multiplies and adds per feature (a lane's four, the same for every row) is requested here:
  // requested behind the products it would come from memory after the weights of the next kernel.
  const int sum_c = lane * 4, qk_head = blockIdx.x;
  const bool qk_v = qk_head >= fold.qk_nq + fold.qk_nkv, qk_k = qk_head >= fold.qk_nq && !qk_v;
  const void* wn = fold.res_x ? fold.res_g : !fold.qk_nq || qk_v ? nullptr : qk_k ? fold.qk_kw : fold.qk_qw;
  float wv[4] = {1.f, 1.f, 1.f, 1.f}, bv[4] = {0.f, 0.f, 0.f, 0.f};
  if (Cfg::SHARED_K && !EPI && splits > 1) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (wn && n0 + sum_c + j < o_out)
        wv[j] = load_as_f32(wn, fold.res_x ? fold.res_g_dtype : fold.qk_w_dtype, (size_t)(fold.res_x ? n0 : 0) + sum_c + j);
      if (fold.bias && n0 + sum_c + j < o_out) bv[j] = __ldg(fold.bias + n0 + sum_c + j);
    }
  }

  if (warp == 0) {
    // The first fill of the stages: the w tiles, which no kernel of the step writes, are requested before this kernel
    // waits for its predecessor in the stream; the x tiles after.  (The other warps act only on what these loads
    // bring, so the wait of this warp orders the whole CTA behind the predecessor.)
    const int first = min(kblocks, Cfg::STAGES);
    if (elect_one()) {
      for (int kb = 0; kb < first; ++kb) {
        unsigned char* stage = smem + kb * Cfg::STAGE_BYTES;
        mbar_expect_tx(&full[kb], Cfg::STAGE_BYTES);
        tma_load_2d(stage + Cfg::A_BYTES, &tmap_w, &full[kb], (kb0 + kb) * G_BK, w0);       // FO rows of w
        if (EPI) tma_load_2d(stage + Cfg::A_BYTES + Cfg::B_BYTES / 2, &tmap_w, &full[kb], (kb0 + kb) * G_BK, o_out + w0);
      }
    }
    __syncwarp();
    ifb_pdl_wait();
    ifb_pdl_trigger();
    if (elect_one()) {
      for (int kb = 0; kb < first; ++kb)
        tma_load_2d(smem + kb * Cfg::STAGE_BYTES, &tmap_x, &full[kb], (kb0 + kb) * G_BK, m0);   // MH * 128 rows of x
    }
    __syncwarp();
    for (int kb = first; kb < kblocks; ++kb) {
      const int s = kb % Cfg::STAGES;
      const uint32_t ph = (kb / Cfg::STAGES) & 1;
      if (!mbar_wait(&empty[s], ph ^ 1, abort_flag, err, 1)) break;
      if (elect_one()) {
        unsigned char* stage = smem + s * Cfg::STAGE_BYTES;
        mbar_expect_tx(&full[s], Cfg::STAGE_BYTES);
        tma_load_2d(stage, &tmap_x, &full[s], (kb0 + kb) * G_BK, m0);
        tma_load_2d(stage + Cfg::A_BYTES, &tmap_w, &full[s], (kb0 + kb) * G_BK, w0);
        if (EPI) tma_load_2d(stage + Cfg::A_BYTES + Cfg::B_BYTES / 2, &tmap_w, &full[s], (kb0 + kb) * G_BK, o_out + w0);
      }
      __syncwarp();
    }
  } else if (warp == 1) {
    bool ok = true;
    for (int kb = 0; kb < kblocks && ok; ++kb) {
      const int s = kb % Cfg::STAGES;
      const uint32_t ph = (kb / Cfg::STAGES) & 1;
      ok = mbar_wait(&full[s], ph, abort_flag, err, 2);
      if (!ok) break;
      tc_fence_after();
      if (elect_one()) {
        const uint32_t a_addr = g_smem_u32(smem + s * Cfg::STAGE_BYTES);
        const uint64_t a_desc = make_smem_desc(a_addr);
        const uint64_t b_desc = make_smem_desc(a_addr + Cfg::A_BYTES);
#pragma unroll
        for (int k = 0; k < G_BK / G_UK; ++k) {
          const uint64_t step = (uint64_t)((k * G_UK * 2) >> 4);          // 32 bytes per k step, in 16-byte units
          const uint32_t acc = (kb | k) != 0;
#pragma unroll
          for (int hf = 0; hf < MH; ++hf)
            umma_bf16(tmem_base + hf * NACC, a_desc + (uint64_t)((hf * G_TILE_BYTES) >> 4) + step, b_desc + step, Cfg::IDESC, acc);
        }
        umma_commit(&empty[s]);
        if (kb == kblocks - 1) umma_commit(accum);
      }
      __syncwarp();
    }
  } else {
    // A warp's piece of the tile is 32 tokens (its lanes) by CW features.  A lane holds a token's row, so storing
    // from registers would send the 32 lanes of a store to 32 different rows of `out`; the piece goes through shared
    // memory instead (the stages, all consumed by now) and leaves in whole row segments, 512 bytes per store.
    constexpr int CW = FO / 2;
    // staged PW features at a time: all of the piece if eight warps' rows fit in the stages, else half of it
    constexpr int PW = 8 * 32 * (CW * (int)sizeof(TO) + 16) <= Cfg::STAGES * Cfg::STAGE_BYTES ? CW : CW / 2;
    constexpr int ROWB = PW * (int)sizeof(TO);                   // bytes of a row segment
    constexpr int PITCH = ROWB + 16;                             // an odd number of 16-byte units: no bank conflicts
    static_assert(8 * 32 * PITCH <= Cfg::STAGES * Cfg::STAGE_BYTES, "the staging rows must fit in the stages");
    const int q = warp & 3;                                      // this warp's quarter of the 128 lanes
    const int c_lo = ((warp - 2) >> 2) * CW;                     // and its half of the tile's features
    // What reads or finishes whole rows of float32 (tc_finish_residual, tc_finish_heads) gets its piece in float32 rows.
    const bool finish_res = !EPI && splits == 1 && fold.res_x && (o_out & 3) == 0 && n0 + c_lo + CW <= o_out;
    const bool finish_qk = !EPI && sizeof(TO) == 2 && splits == 1 && fold.qk_nq;
    constexpr int FPITCH = CW * 4 + 16;                          // bytes of a float32 row, padded
    static_assert(EPI || 8 * 32 * FPITCH <= Cfg::STAGES * Cfg::STAGE_BYTES, "the float32 rows must fit in the stages");
    // What the epilogue reads beside the product is requested while the product is being made.
    constexpr int AHEAD = (CW == 64 && Cfg::STAGES == 3) ? 8 : 16;       // (two CTAs per SM: half the registers)
    constexpr int AHEAD_H = AHEAD / 2;                           // passes over heads: twice the angles each
    float rfac_of[MH];
    float4 ahead[EPI ? 1 : AHEAD], angles[EPI ? 1 : AHEAD_H][2];      // rows of the stream, or angles
    int slot_of[EPI ? 1 : AHEAD_H];
    // finish_qk: CW 128: the warp has a head of its own; CW 64: the pairs [32 c, 32 c + 32) of the tile's one head
    const int qk_base = CW == 128 ? c_lo : 0, qk_i0 = CW == 128 ? 0 : c_lo / 2, qk_head = (n0 + qk_base) / 128;
    const bool qk_v = qk_head >= fold.qk_nq + fold.qk_nkv, qk_k = qk_head >= fold.qk_nq && !qk_v;
    const bool qk_rotate = finish_qk && !qk_v && fold.qk_rope, qk_store = finish_qk && (qk_v || qk_k) && fold.qk_slots;
    if (fold.rs_partials || fold.res_x || fold.qk_nq) ifb_pdl_wait();             // what the predecessor wrote is read here directly
#pragma unroll
    for (int hf = 0; hf < MH; ++hf) rfac_of[hf] = tc_row_factor(fold, m0 + hf * G_BM + q * 32 + lane, n_rows);
    if constexpr (!EPI) {
      if (finish_res) tc_residual_load<CW, AHEAD>(fold, m0 + q * 32, n_rows, n0 + c_lo, o_out, lane, ahead);
      else if (finish_qk) tc_heads_load<CW / 2, AHEAD_H>(fold, m0 + q * 32, n_rows, qk_i0, qk_rotate, qk_store, lane, angles, slot_of);
    }
    if (kblocks > 0 && mbar_wait(accum, 0, abort_flag, err, 3)) {
      tc_fence_after();
     if constexpr (!EPI) {
      if (finish_res || finish_qk) {
        unsigned char* rows32 = smem + (warp - 2) * (32 * FPITCH);
#pragma unroll
        for (int hf = 0; hf < MH; ++hf) {
          const int row0 = m0 + hf * G_BM + q * 32;
          if (row0 >= n_rows) break;                             // warp-uniform
          const uint32_t lane_base = tmem_base + ((uint32_t)(q * 32) << 16) + hf * NACC;
          float rfac = rfac_of[hf];
          if (finish_res) {
            if (hf) tc_residual_load<CW, AHEAD>(fold, row0, n_rows, n0 + c_lo, o_out, lane, ahead);
#pragma unroll 1
            for (int c0 = 0; c0 < CW; c0 += 32) tc_stage_rows(lane_base + c_lo + c0, rows32 + lane * FPITCH + c0 * 4, rfac);
            __syncwarp();
            tc_finish_residual<CW, FPITCH, AHEAD, TO>(fold, rows32, out, row0, n_rows, n0 + c_lo, o_out,
                                                      blockIdx.x * 2 + (c_lo ? 1 : 0), lane, ahead);
          } else if constexpr (sizeof(TO) == 2) {
            if (n0 + qk_base < o_out) {
              if (hf) tc_heads_load<CW / 2, AHEAD_H>(fold, row0, n_rows, qk_i0, qk_rotate, qk_store, lane, angles, slot_of);
              const void* wn = qk_v ? nullptr : qk_k ? fold.qk_kw : fold.qk_qw;
              if (wn) {
                float ss = 0.f;
#pragma unroll 1
                for (int c0 = 0; c0 < 128; c0 += 32) {
                  uint32_t v[32];
                  tmem_ld32(lane_base + qk_base + c0, v);
                  tmem_ld_wait();
#pragma unroll
                  for (int j = 0; j < 32; ++j) { const float f = __uint_as_float(v[j]) * rfac; ss = fmaf(f, f, ss); }
                }
                rfac *= rsqrtf(ss * (1.f / 128.f) + fold.qk_eps);
              }
              constexpr int NP = CW / 2;                         // pairs of the warp
#pragma unroll 1
              for (int c0 = 0; c0 < NP; c0 += 32) {
                tc_stage_rows(lane_base + qk_base + qk_i0 + c0, rows32 + lane * FPITCH + c0 * 4, rfac);
                tc_stage_rows(lane_base + qk_base + 64 + qk_i0 + c0, rows32 + lane * FPITCH + (NP + c0) * 4, rfac);
              }
              __syncwarp();
              tc_finish_heads<NP, FPITCH, AHEAD_H>(fold, rows32, reinterpret_cast<bf16*>(out), row0, n_rows, qk_head, qk_i0, o_out, wn, qk_v,
                                                   qk_rotate, qk_store, lane, angles, slot_of);
            }
          }
          __syncwarp();                                          // before the next rows overwrite the buffer
        }
      }
     }
     if (!finish_res && !finish_qk) {
      const bool vec = ((size_t)o_out * sizeof(TO)) % 16 == 0 && (((uintptr_t)out) & 15) == 0 && n0 + c_lo + CW <= o_out;
      unsigned char* buf = smem + (warp - 2) * (32 * PITCH);
#pragma unroll 1
      for (int hf = 0; hf < MH; ++hf) {
        const int row0 = m0 + hf * G_BM + q * 32;
        const uint32_t lane_base = tmem_base + ((uint32_t)(q * 32) << 16) + hf * NACC;
        const float rfac = MH == 1 || hf == 0 ? rfac_of[0] : rfac_of[MH - 1];
        float ss = 0.f;                                          // this row's v^2 over this warp's features
#pragma unroll 1
       for (int p0 = c_lo; p0 < c_lo + CW; p0 += PW) {
#pragma unroll 1
        for (int c0 = p0; c0 < p0 + PW; c0 += 32) {
          if (n0 + c0 >= o_out) break;                           // warp-uniform
          uint32_t v[32];
          float y[32];
          tmem_ld32(lane_base + c0, v);
          if (splits > 1) {
            // the part stays here for the cluster's sum (with the silu_gate epilogue: the gate columns, then the up
            // columns FO further on; the epilogue itself comes after the sum)
            float* dst = reinterpret_cast<float*>(smem) + (size_t)(hf * G_BM + q * 32 + lane) * RED_PITCH + c0;
            uint32_t u[32];
            if (EPI) tmem_ld32(lane_base + FO + c0, u);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 32; j += 4)
              *reinterpret_cast<float4*>(dst + j) = make_float4(__uint_as_float(v[j]) * rfac, __uint_as_float(v[j + 1]) * rfac,
                                                                __uint_as_float(v[j + 2]) * rfac, __uint_as_float(v[j + 3]) * rfac);
            if (EPI) {
#pragma unroll
              for (int j = 0; j < 32; j += 4)
                *reinterpret_cast<float4*>(dst + FO + j) = make_float4(__uint_as_float(u[j]) * rfac, __uint_as_float(u[j + 1]) * rfac,
                                                                       __uint_as_float(u[j + 2]) * rfac, __uint_as_float(u[j + 3]) * rfac);
            }
            continue;
          }
          if (EPI) {
            uint32_t u[32];
            tmem_ld32(lane_base + FO + c0, u);
            tmem_ld_wait();
            tc_gates(y, v, u, rfac, fold.unary);                 // (a warp-uniform choice)
          } else {
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 32; ++j) y[j] = __uint_as_float(v[j]) * rfac;
            if (fold.bias) {                                     // warp-uniform; every lane holds the same 32 features
#pragma unroll
              for (int j = 0; j < 32; ++j) y[j] += n0 + c0 + j < o_out ? __ldg(fold.bias + n0 + c0 + j) : 0.f;
            }
            if (fold.unary) {                                    // warp-uniform
              tc_unary(y, fold.unary);
            }
          }
          if (!EPI && fold.res_x) ss += tc_residual_chunk(fold, y, row0 + lane, n_rows, n0 + c0, o_out);
          if (vec) {
            unsigned char* dst = buf + lane * PITCH + (c0 - p0) * (int)sizeof(TO);
            if (sizeof(TO) == 2) {
#pragma unroll
              for (int j = 0; j < 32; j += 8) {
                uint4 pk;
                __nv_bfloat162 p0 = __floats2bfloat162_rn(y[j], y[j + 1]), p1 = __floats2bfloat162_rn(y[j + 2], y[j + 3]);
                __nv_bfloat162 p2 = __floats2bfloat162_rn(y[j + 4], y[j + 5]), p3 = __floats2bfloat162_rn(y[j + 6], y[j + 7]);
                pk.x = *reinterpret_cast<uint32_t*>(&p0); pk.y = *reinterpret_cast<uint32_t*>(&p1);
                pk.z = *reinterpret_cast<uint32_t*>(&p2); pk.w = *reinterpret_cast<uint32_t*>(&p3);
                *reinterpret_cast<uint4*>(dst + j * 2) = pk;
              }
            } else {
#pragma unroll
              for (int j = 0; j < 32; j += 4)
                *reinterpret_cast<float4*>(dst + j * 4) = make_float4(y[j], y[j + 1], y[j + 2], y[j + 3]);
            }
          } else if (row0 + lane < n_rows) {
            TO* dst = out + (size_t)(row0 + lane) * o_out + n0 + c0;
#pragma unroll
            for (int j = 0; j < 32; ++j)
              if (n0 + c0 + j < o_out) dst[j] = from_f32<TO>(y[j]);
          }
        }
        if (vec && splits == 1) {
          __syncwarp();
          unsigned char* obase = reinterpret_cast<unsigned char*>(out + (size_t)row0 * o_out + n0 + p0);
#pragma unroll 4
          for (int off = lane * 16; off < 32 * ROWB; off += 512) {
            const int r = off / ROWB, cb = off % ROWB;
            if (row0 + r < n_rows)
              *reinterpret_cast<uint4*>(obase + (size_t)r * o_out * sizeof(TO) + cb) = *reinterpret_cast<const uint4*>(buf + r * PITCH + cb);
          }
          __syncwarp();                                          // before the next rows overwrite the buffer
        }
       }
       if (!EPI && splits == 1 && fold.res_x && row0 + lane < n_rows)
         fold.res_partials[(size_t)(blockIdx.x * 2 + (c_lo ? 1 : 0)) * n_rows + row0 + lane] = ss;
      }
     }
    }
  }
  if constexpr (Cfg::SHARED_K) {
    if (splits > 1) {
      // The sum over the cluster: a warp adds a row of the tile at a time (a lane four features), from the row of each CTA
      // that had k blocks.  What bounds it is the round trip to the other CTAs' shared memory and the code's first run: the parts
      // of a row, and what else the epilogue reads for it, are requested before the first is used, but no more than two rows
      // at a time (with two and four rows unrolled a decode step of 64 rows of the 0.6B sizes took 1.73 ms, with one and two 1.64;
      // with the parts added one round trip after the other 1.67, and a prompt of 131 tokens 1.50 ms for 1.24).
      static_assert(FO == 128, "a lane of the sum has four of a row's features");
      constexpr int PARTS = EPI ? 2 : 1, ROWS_OF_8 = 1, ROWS_OF_4 = 2, WARPS = G_THREADS / 32;
      const int c = sum_c;
      const int rows = min(G_BM, n_rows - m0), cols = min(FO, o_out - n0);
      const int used = (kb_all + kb_per - 1) / kb_per;                     // CTAs that had k blocks
      const int per = (rows + splits - 1) / splits;
      const int r_lo = blockIdx.z * per + warp, r_hi = min(rows, ((int)blockIdx.z + 1) * per);
      const bool vec = ((size_t)o_out * sizeof(TO)) % 16 == 0 && (((uintptr_t)out) & 15) == 0 && cols == FO;
      cluster_sync_all();                      // every CTA's part is in its shared memory
      if (fold.res_x || fold.qk_nq) ifb_pdl_wait();
      const uint32_t tile_addr = g_smem_u32(smem);
      auto run = [&](auto z_max, auto rows_ahead) {
        constexpr int Z = decltype(z_max)::value, B = decltype(rows_ahead)::value;
        for (int rb = r_lo;; rb += B * WARPS) {
          float4 v[B][PARTS][Z], xr[EPI ? 1 : B], cs[EPI ? 1 : B][2];
          int slot[EPI ? 1 : B];
#pragma unroll
          for (int b = 0; b < B; ++b) {
            const int r = rb + b * WARPS;
            const uint32_t at = tile_addr + (uint32_t)((r * RED_PITCH + c) * 4);
#pragma unroll
            for (int e = 0; e < PARTS; ++e)
#pragma unroll
              for (int z = 0; z < Z; ++z)
                v[b][e][z] = r < r_hi && z < used ? ld_cluster_f4(at + e * FO * 4, z) : make_float4(0.f, 0.f, 0.f, 0.f);
            if (!EPI && fold.res_x) {
              const float* x = fold.res_x + (size_t)(m0 + r) * o_out + n0 + c;
              if (r >= r_hi) xr[b] = make_float4(0.f, 0.f, 0.f, 0.f);
              else if (cols == FO && (o_out & 3) == 0) xr[b] = *reinterpret_cast<const float4*>(x);
              else xr[b] = make_float4(c < cols ? x[0] : 0.f, c + 1 < cols ? x[1] : 0.f, c + 2 < cols ? x[2] : 0.f, c + 3 < cols ? x[3] : 0.f);
            }
            if (!EPI && fold.qk_nq) {
              const bool turn = !qk_v && fold.qk_rope && r < r_hi;
              const float4* t = reinterpret_cast<const float4*>(fold.qk_rope + (size_t)(m0 + r) * 64 + (c & 63));
              cs[b][0] = turn ? t[0] : make_float4(1.f, 0.f, 1.f, 0.f);
              cs[b][1] = turn ? t[1] : make_float4(1.f, 0.f, 1.f, 0.f);
              slot[b] = (qk_v || qk_k) && fold.qk_slots && r < r_hi ? fold.qk_slots[m0 + r] : -1;
            }
          }
          float4 sum[B][PARTS];
#pragma unroll
          for (int b = 0; b < B; ++b)
#pragma unroll
            for (int e = 0; e < PARTS; ++e) {
              float4 t = make_float4(0.f, 0.f, 0.f, 0.f);                  // in the order of the CTAs
#pragma unroll
              for (int z = 0; z < Z; ++z)
                if (z < used) { t.x += v[b][e][z].x; t.y += v[b][e][z].y; t.z += v[b][e][z].z; t.w += v[b][e][z].w; }
              sum[b][e] = t;
            }
          const bool last = rb + B * WARPS >= r_hi;
          // This warp has read all it reads of the other CTAs' shared memory, and its arrival lets them leave.  What has to hold is
          // that its reads are complete, that is, their values are in registers: the vote takes a part of every one of them, and the
          // arrival is predicated on the vote.  The predicate is always true (a count of lanes is above minus the number of rows),
          // but the number of rows is the launch's, so no compiler can know that and drop what the arrival waits for.  (A release
          // instead would wait for the stores of the rows before as well: 131 tokens of the 0.6B sizes 1,161 to 1,184 us, with the
          // sums kept in shared memory until all is read 1,199.)
          if (last) {
            float all = 0.f;
#pragma unroll
            for (int b = 0; b < B; ++b)
#pragma unroll
              for (int e = 0; e < PARTS; ++e) all += sum[b][e].x;
            const int votes = __popc(__ballot_sync(0xffffffffu, all != 0.f));
            asm volatile("{\n .reg .pred p;\n setp.gt.s32 p, %0, %1;\n @p barrier.cluster.arrive.relaxed.aligned;\n}\n" ::"r"(votes), "r"(-n_rows)
                         : "memory");
          }
#pragma unroll
          for (int b = 0; b < B; ++b) {
            const int r = rb + b * WARPS;
            if (r >= r_hi) break;                                          // warp-uniform
            float yv[4] = {sum[b][0].x, sum[b][0].y, sum[b][0].z, sum[b][0].w};
            if (EPI) {
              const float4 up = sum[b][PARTS - 1];
              yv[0] = tc_gate(yv[0], fold.unary) * up.x; yv[1] = tc_gate(yv[1], fold.unary) * up.y;
              yv[2] = tc_gate(yv[2], fold.unary) * up.z; yv[3] = tc_gate(yv[3], fold.unary) * up.w;
            } else {
              if (fold.bias) {
#pragma unroll
                for (int j = 0; j < 4; ++j) yv[j] += bv[j];
              }
              if (fold.unary) tc_unary(yv, fold.unary);
            }
            TO* dst = out + (size_t)(m0 + r) * o_out + n0 + c;
            if (!EPI && fold.res_x) {
              // v = x + y, x <- v, the output becomes v * g, the warp's sum of v^2 one part
              float* x = fold.res_x + (size_t)(m0 + r) * o_out + n0 + c;
              const float xo[4] = {xr[b].x, xr[b].y, xr[b].z, xr[b].w};
              float ss = 0.f;
#pragma unroll
              for (int j = 0; j < 4; ++j)
                if (c + j < cols) {
                  const float t = xo[j] + yv[j];
                  x[j] = t;
                  ss += t * t;
                  yv[j] = t * wv[j];
                }
#pragma unroll
              for (int d = 16; d > 0; d >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, d);
              if ((threadIdx.x & 31) == 0) fold.res_partials[(size_t)blockIdx.x * n_rows + m0 + r] = ss;
            }
            if (!EPI && sizeof(TO) == 2 && fold.qk_nq) {
              // the warp holds one head of one token (lane l its elements 4l .. 4l + 3; the rotation partner 16 lanes on)
              if (wn) {
                float ss = yv[0] * yv[0] + yv[1] * yv[1] + yv[2] * yv[2] + yv[3] * yv[3];
#pragma unroll
                for (int d = 16; d > 0; d >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, d);
                const float rn = rsqrtf(ss * (1.f / 128.f) + fold.qk_eps);
#pragma unroll
                for (int j = 0; j < 4; ++j) yv[j] = yv[j] * rn * wv[j];
              }
              if (!qk_v && fold.qk_rope) {
                const float co[4] = {cs[b][0].x, cs[b][0].z, cs[b][1].x, cs[b][1].z}, si[4] = {cs[b][0].y, cs[b][0].w, cs[b][1].y, cs[b][1].w};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                  const float o = __shfl_xor_sync(0xffffffffu, yv[j], 16);
                  yv[j] = (threadIdx.x & 31) < 16 ? yv[j] * co[j] - o * si[j] : yv[j] * co[j] + o * si[j];
                }
              }
              const __nv_bfloat162 lo = __floats2bfloat162_rn(yv[0], yv[1]), hi = __floats2bfloat162_rn(yv[2], yv[3]);
              const uint2 pk = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
              *reinterpret_cast<uint2*>(dst) = pk;
              if (slot[b] >= 0) {
                const int kvh = qk_v ? qk_head - fold.qk_nq - fold.qk_nkv : qk_head - fold.qk_nq;
                const size_t row = ((size_t)(slot[b] / fold.qk_page_size) * 2 + (qk_v ? 1 : 0)) * fold.qk_nkv + kvh;
                *reinterpret_cast<uint2*>(fold.qk_pages + (row * fold.qk_page_size + slot[b] % fold.qk_page_size) * 128 + c) = pk;
              }
              continue;
            }
            if (vec) {
              if (sizeof(TO) == 4) {
                *reinterpret_cast<float4*>(dst) = make_float4(yv[0], yv[1], yv[2], yv[3]);
              } else {
                const __nv_bfloat162 lo = __floats2bfloat162_rn(yv[0], yv[1]), hi = __floats2bfloat162_rn(yv[2], yv[3]);
                *reinterpret_cast<uint2*>(dst) = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
              }
            } else {
              for (int j = 0; j < 4; ++j)
                if (c + j < cols) dst[j] = from_f32<TO>(yv[j]);
            }
          }
          if (last) break;
        }
      };
      if (used > 4) run(TcInt<8>{}, TcInt<ROWS_OF_8>{});
      else run(TcInt<4>{}, TcInt<ROWS_OF_4>{});
      asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");      // nobody leaves while its shared memory is being read
    }
  }
  if (*abort_flag) {                         // a wait gave up: let copies in flight land before the CTA goes away
    for (int i = 0; i < 2000; ++i) __nanosleep(1000);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem_base, Cfg::TMEM_COLS); }
}


// ---------------------------------------------------------------------------------------------------
// A [rows, k] bfloat16 row-major matrix as a tensor map with boxes of 64 k x box_rows rows, 128-byte swizzle.
static int make_map(CUtensorMap* m, const void* ptr, int rows, int k, int box_rows) {
  const unsigned long long dims[2] = {(unsigned long long)k, (unsigned long long)rows};
  const unsigned long long strides[1] = {(unsigned long long)k * 2};
  const unsigned box[2] = {(unsigned)G_BK, (unsigned)box_rows};
  return ifb_tensor_map_bf16(m, ptr, 2, dims, strides, box);
}

// ---------------------------------------------------------------------------------------------------
// The persistent form.  A CTA per SM walks a list of output tiles (tile t of the list goes to CTA t mod grid), with two
// accumulators in tensor memory: while the epilogue warps read and store tile i from one, the issuer already
// multiplies tile i + 1 into the other, and the producer's ring of stages never drains between tiles.  Tiles are
// 128 tokens x NACC accumulator columns (128 or 256; with the silu_gate epilogue 128 gate + 128 up columns give 128
// features); consecutive tiles of the list share their w tile, so it is read from L2 by the CTAs of one round.
// The epilogue has its own staging rows in shared memory (the stages are busy with the next tile).
// ---------------------------------------------------------------------------------------------------
template <int EPI_, int NACC_, int STAGES_> struct PersistCfg {
  static constexpr int EPI = EPI_, NACC = NACC_, STAGES = STAGES_;
  static constexpr int FO = EPI ? NACC / 2 : NACC;            // output features per tile
  static constexpr int A_BYTES = G_TILE_BYTES;                // 128 x rows of a stage
  static constexpr int B_BYTES = NACC * G_BK * 2;             // w rows of a stage
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int TMEM_COLS = 2 * NACC;                  // two accumulators: 256 or 512 columns
  static constexpr int STAGING_PITCH = 128 + 16;              // a row segment of 128 bytes, padded against bank conflicts
  static constexpr int STAGING_BYTES = 8 * 32 * STAGING_PITCH;
  static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + STAGING_BYTES + 1024 /* alignment */ + 256 /* barriers */;
  static constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(NACC >> 3) << 17) | ((uint32_t)(G_BM >> 4) << 24);
};

// 32 columns of an accumulator (a lane's row of them) through the epilogue: y.  FO: columns from a gate to its up.
template <int EPI>
__device__ __forceinline__ void tc_epilogue_row(const TcFold& fold, uint32_t taddr, int fo, float rfac, int col, int o_out, float (&y)[32]) {
  uint32_t v[32];
  tmem_ld32(taddr, v);
  if (EPI) {
    uint32_t u[32];
    tmem_ld32(taddr + fo, u);
    tmem_ld_wait();
    tc_gates(y, v, u, rfac, fold.unary);                 // (a warp-uniform choice)
  } else {
    tmem_ld_wait();
#pragma unroll
    for (int j = 0; j < 32; ++j) y[j] = __uint_as_float(v[j]) * rfac;
    if (fold.bias) {                                     // warp-uniform; every lane holds the same 32 features
#pragma unroll
      for (int j = 0; j < 32; ++j) y[j] += col + j < o_out ? __ldg(fold.bias + col + j) : 0.f;
    }
    if (fold.unary) {                                    // warp-uniform
      tc_unary(y, fold.unary);
    }
  }
}
// 32 values in the output type at 16-byte aligned `dst`.
template <typename TO>
__device__ __forceinline__ void tc_pack_row(unsigned char* dst, const float (&y)[32]) {
  if (sizeof(TO) == 2) {
#pragma unroll
    for (int j = 0; j < 32; j += 8) {
      uint4 pk;
      __nv_bfloat162 h0 = __floats2bfloat162_rn(y[j], y[j + 1]), h1 = __floats2bfloat162_rn(y[j + 2], y[j + 3]);
      __nv_bfloat162 h2 = __floats2bfloat162_rn(y[j + 4], y[j + 5]), h3 = __floats2bfloat162_rn(y[j + 6], y[j + 7]);
      pk.x = *reinterpret_cast<uint32_t*>(&h0); pk.y = *reinterpret_cast<uint32_t*>(&h1);
      pk.z = *reinterpret_cast<uint32_t*>(&h2); pk.w = *reinterpret_cast<uint32_t*>(&h3);
      *reinterpret_cast<uint4*>(dst + j * 2) = pk;
    }
  } else {
#pragma unroll
    for (int j = 0; j < 32; j += 4) *reinterpret_cast<float4*>(dst + j * 4) = make_float4(y[j], y[j + 1], y[j + 2], y[j + 3]);
  }
}

template <typename Cfg, typename TO>
__global__ void __launch_bounds__(G_THREADS, 1)
linear_tcgen05_persistent_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_w,
                                 TO* __restrict__ out, int n_rows, int o_out, int k_dim, int tiles_m, int tiles_total,
                                 int* __restrict__ err, TcFold fold) {
  constexpr int EPI = Cfg::EPI, NACC = Cfg::NACC, FO = Cfg::FO, STAGES = Cfg::STAGES;
  extern __shared__ unsigned char g_smem_raw[];
  const uint32_t raw = g_smem_u32(g_smem_raw);
  unsigned char* smem = g_smem_raw + (((raw + 1023u) & ~1023u) - raw);      // tiles need 1024-byte alignment
  unsigned char* staging = smem + STAGES * Cfg::STAGE_BYTES;
  uint64_t* full = reinterpret_cast<uint64_t*>(staging + Cfg::STAGING_BYTES);
  uint64_t* empty = full + STAGES;
  uint64_t* acc_full = empty + STAGES;                         // [2]: the issuer has finished a tile in accumulator b
  uint64_t* acc_empty = acc_full + 2;                          // [2]: the eight epilogue warps have read accumulator b
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;     // warp-uniform
  const int kblocks = (k_dim + G_BK - 1) / G_BK;
  // this CTA's tiles: first, first + gridDim.x, ...; tile t covers tokens (t % tiles_m) * 128 and features (t / tiles_m) * FO
  const int first = blockIdx.x, step = gridDim.x;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(&acc_full[b], 1); mbar_init(&acc_empty[b], 8); }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
  }
  if (warp == 1) { tmem_alloc(tmem_slot, Cfg::TMEM_COLS); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    // ---- producer.  The w tiles of the first stages, which no kernel of the step writes, are requested before this
    // kernel waits for its predecessor in the stream; every x tile after.  (The other warps act only on what these
    // loads bring, so the wait of this warp orders the whole CTA behind the predecessor.)
    int g = 0;                                                  // k blocks issued so far, over all tiles
    bool waited = false, ok = true;
    for (int t = first; t < tiles_total && ok; t += step) {
      const int m0 = (t % tiles_m) * G_BM, n0 = (t / tiles_m) * FO;
      for (int kb = 0; kb < kblocks; ++kb, ++g) {
        const int s = g % STAGES;
        if (g >= STAGES && !mbar_wait(&empty[s], ((g / STAGES) - 1) & 1, abort_flag, err, 1)) { ok = false; break; }
        unsigned char* stage = smem + s * Cfg::STAGE_BYTES;
        if (elect_one()) {
          mbar_expect_tx(&full[s], Cfg::STAGE_BYTES);
          tma_load_2d(stage + Cfg::A_BYTES, &tmap_w, &full[s], kb * G_BK, n0);
          if (EPI) tma_load_2d(stage + Cfg::A_BYTES + Cfg::B_BYTES / 2, &tmap_w, &full[s], kb * G_BK, o_out + n0);
        }
        __syncwarp();
        if (!waited && (g == STAGES - 1 || (kb == kblocks - 1 && t + step >= tiles_total))) {
          // the ring is full of w tiles (or there are no more): now the predecessor, then the x tiles held back
          ifb_pdl_wait();
          ifb_pdl_trigger();
          waited = true;
          if (elect_one()) {
            int gg = 0;
            for (int tt = first; tt < tiles_total && gg <= g; tt += step)
              for (int kk = 0; kk < kblocks && gg <= g; ++kk, ++gg)
                tma_load_2d(smem + (gg % STAGES) * Cfg::STAGE_BYTES, &tmap_x, &full[gg % STAGES], kk * G_BK, (tt % tiles_m) * G_BM);
          }
          __syncwarp();
        } else if (waited) {
          if (elect_one()) tma_load_2d(stage, &tmap_x, &full[s], kb * G_BK, m0);
          __syncwarp();
        }
      }
    }
    if (!waited) { ifb_pdl_wait(); ifb_pdl_trigger(); }         // a CTA without tiles still orders itself behind the predecessor
  } else if (warp == 1) {
    // ---- issuer: tile i of this CTA accumulates in accumulator i & 1
    int g = 0, it = 0;
    bool ok = true;
    for (int t = first; t < tiles_total && ok; t += step, ++it) {
      const int b = it & 1;
      if (it >= 2) ok = mbar_wait(&acc_empty[b], ((it >> 1) - 1) & 1, abort_flag, err, 4);
      if (!ok) break;
      tc_fence_after();
      for (int kb = 0; kb < kblocks && ok; ++kb, ++g) {
        const int s = g % STAGES;
        ok = mbar_wait(&full[s], (g / STAGES) & 1, abort_flag, err, 2);
        if (!ok) break;
        tc_fence_after();
        if (elect_one()) {
          const uint32_t a_addr = g_smem_u32(smem + s * Cfg::STAGE_BYTES);
          const uint64_t a_desc = make_smem_desc(a_addr);
          const uint64_t b_desc = make_smem_desc(a_addr + Cfg::A_BYTES);
#pragma unroll
          for (int k = 0; k < G_BK / G_UK; ++k) {
            const uint64_t kstep = (uint64_t)((k * G_UK * 2) >> 4);          // 32 bytes per k step, in 16-byte units
            umma_bf16(tmem_base + b * NACC, a_desc + kstep, b_desc + kstep, Cfg::IDESC, (kb | k) != 0);
          }
          umma_commit(&empty[s]);
          if (kb == kblocks - 1) umma_commit(&acc_full[b]);
        }
        __syncwarp();
      }
    }
  } else {
    // ---- epilogue.  A warp's piece of a tile is 32 tokens (its lanes) by CW features, taken 128 bytes of a row at a
    // time: from tensor memory to registers, to the warp's staging rows, and from there in whole row segments to `out`.
    constexpr int CW = FO / 2;
    constexpr int PW = 128 / (int)sizeof(TO);                    // features per staged row segment
    constexpr int PITCH = Cfg::STAGING_PITCH;
    static_assert(CW % PW == 0, "a warp's features are whole row segments");
    const int q = warp & 3;                                      // this warp's quarter of the 128 lanes
    const int c_lo = ((warp - 2) >> 2) * CW;                     // and its half of the tile's features
    unsigned char* buf = staging + (warp - 2) * (32 * PITCH);
    int it = 0;
    bool ok = true;
    for (int t = first; t < tiles_total && ok; t += step, ++it) {
      const int b = it & 1;
      const int m0 = (t % tiles_m) * G_BM, n0 = (t / tiles_m) * FO;
      ok = mbar_wait(&acc_full[b], (it >> 1) & 1, abort_flag, err, 3);
      if (!ok) break;
      tc_fence_after();
      const bool vec = ((size_t)o_out * sizeof(TO)) % 16 == 0 && (((uintptr_t)out) & 15) == 0 && n0 + c_lo + CW <= o_out;
      const int row0 = m0 + q * 32;
      const uint32_t lane_base = tmem_base + ((uint32_t)(q * 32) << 16) + b * NACC;
      if (fold.rs_partials && it == 0) ifb_pdl_wait();             // the sums are the predecessor's: read them after it
      const float rfac = tc_row_factor(fold, row0 + lane, n_rows);
#pragma unroll 1
      for (int p0 = c_lo; p0 < c_lo + CW; p0 += PW) {
        if (n0 + p0 >= o_out) break;                             // warp-uniform
#pragma unroll
        for (int c0 = p0; c0 < p0 + PW; c0 += 32) {
          float y[32];
          tc_epilogue_row<EPI>(fold, lane_base + c0, FO, rfac, n0 + c0, o_out, y);
          if (vec) {
            tc_pack_row<TO>(buf + lane * PITCH + (c0 - p0) * (int)sizeof(TO), y);
          } else if (row0 + lane < n_rows) {
            TO* dst = out + (size_t)(row0 + lane) * o_out + n0 + c0;
#pragma unroll
            for (int j = 0; j < 32; ++j)
              if (n0 + c0 + j < o_out) dst[j] = from_f32<TO>(y[j]);
          }
        }
        if (vec) {
          __syncwarp();
          unsigned char* obase = reinterpret_cast<unsigned char*>(out + (size_t)row0 * o_out + n0 + p0);
#pragma unroll
          for (int off = lane * 16; off < 32 * 128; off += 512) {
            const int r = off >> 7, cb = off & 127;
            if (row0 + r < n_rows)
              *reinterpret_cast<uint4*>(obase + (size_t)r * o_out * sizeof(TO) + cb) = *reinterpret_cast<const uint4*>(buf + r * PITCH + cb);
          }
          __syncwarp();                                          // before the next segment overwrites the rows
        }
      }
      // this warp has read its part of accumulator b: the issuer may overwrite it (with the tile after next)
      tc_fence_before();
      __syncwarp();
      if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(g_smem_u32(&acc_empty[b])) : "memory");
    }
  }
  if (*abort_flag) {                         // a wait gave up: let copies in flight land before the CTA goes away
    for (int i = 0; i < 2000; ++i) __nanosleep(1000);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem_base, Cfg::TMEM_COLS); }
}

// ---------------------------------------------------------------------------------------------------
// The persistent form over pairs of SMs, for prompts.  A cluster of two CTAs takes a tile of 256 tokens x NACC accumulator
// columns: each CTA loads its own 128 rows of x and HALF of the tile's rows of w (with the silu_gate epilogue: one CTA the gate
// rows, the other the up rows), and one tcgen05.mma of the pair (cta_group::2, M = 256), issued by the first CTA, multiplies out
// of both CTAs' shared memory into both tensor memories, where each CTA finds its 128 tokens' full rows.  What bounds these
// products is the bytes that reach an SM from L2 (57 a cycle measured): per product of 128 x 256 the pair brings 32 KB to an SM
// per 64 of k where a CTA alone brings 48 KB, the same as a 256 x 256 tile of one CTA, but with a tile half as large, so that the other
// half of tensor memory holds a second accumulator and a tile's epilogue runs beside the next tile's products.
// Stages, barriers and epilogue are those of the persistent kernel above, except: the "full" barriers are the first CTA's and
// count both CTAs' bytes, the "empty" and "accumulator ready" barriers are each CTA's own and get a multicast commit, and the
// "accumulator read" barriers are the first CTA's and count both CTAs' epilogue warps.
// Measured at 2,048 rows against the best shape of one CTA: gate and up of 12,288 x 4,096 338 to 257 us (1.6 PFLOP/s),
// q | k | v of 6,144 x 4,096 82 to 70, gate and up of 3,072 x 1,024 22.4 to 20.3 (each alone, repeated; in a step it adds 23.3),
// 1,024 x 3,072 14.9 to 13.8.
// ROWS32: the epilogue stages 64 float32 features of a row at a time (tc_finish_residual, tc_finish_heads).
// HALVES: the tiles of a last round that has no more of them than half the pairs are halved, so that the round takes twice the pairs
// and 0.6 of a round's time (an SM gets 24 KB per 64 of k where it gets 32, and its epilogue is half as long).
// (Gate and up of 12,288 x 4,096 at 2,048 rows, 768 tiles for 74 pairs, 249 to 241 us; 3,072 x 1,024 at 2,048, 96 tiles, float32,
// 18.9 on one tile per CTA, 14.9 so.)
// ---------------------------------------------------------------------------------------------------
template <int EPI_, int NACC_, int STAGES_, bool ROWS32_, bool HALVES_ = false> struct PairCfg {
  static constexpr int EPI = EPI_, NACC = NACC_, STAGES = STAGES_;
  static constexpr bool ROWS32 = ROWS32_, HALVES = HALVES_;
  static constexpr int FO = EPI ? NACC / 2 : NACC;            // output features per tile
  static constexpr int W_ROWS = NACC / 2;                     // rows of w of a CTA's stage
  static constexpr int A_BYTES = G_TILE_BYTES, B_BYTES = W_ROWS * G_BK * 2, STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int TMEM_COLS = 2 * NACC;                  // two accumulators: 256 or 512 columns
  static constexpr int STAGING_PITCH = (ROWS32 ? 256 : 128) + 16;
  static constexpr int STAGING_BYTES = 8 * 32 * STAGING_PITCH;
  static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + STAGING_BYTES + 1024 /* alignment */ + 256 /* barriers */;
  // float32 accumulator, bfloat16 a and b, both K-major, M = 256 over the pair, N = NACC, or half of it
  static constexpr uint32_t IDESC_N0 = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(2 * G_BM >> 4) << 24);
  static constexpr uint32_t IDESC = IDESC_N0 | ((uint32_t)(NACC >> 3) << 17), IDESC_HALF = IDESC_N0 | ((uint32_t)(NACC >> 4) << 17);
  static_assert(SMEM_BYTES <= 227 * 1024, "stages and staging rows must fit in shared memory");
};

__device__ __forceinline__ uint32_t cluster_addr(const void* p, int rank) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(a) : "r"(g_smem_u32(p)), "r"(rank));
  return a;
}
// Into this CTA's shared memory; the bytes are counted by the barrier at `bar`, an address in the cluster (either CTA's).
__device__ __forceinline__ void tma_load_2d_pair(void* smem, const CUtensorMap* map, uint32_t bar, int x, int y) {
  asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];\n"
               ::"r"(g_smem_u32(smem)), "l"(map), "r"(bar), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void umma_bf16_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n}\n"
               ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
// Arrives at the barrier of this address in both CTAs once the products issued so far are done.
__device__ __forceinline__ void umma_commit_pair(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n"
               ::"r"(g_smem_u32(bar)), "h"((uint16_t)3) : "memory");
}

// Tile t of a launch over pairs: its tile of rows, and its first feature.  The first `whole` are whole, then come the two halves of
// tile `whole`, of the next, ...
template <bool HALVES>
__device__ __forceinline__ int tc_pair_place(int t, int whole, int tiles_m, int fo, int& n0) {
  if (!HALVES) { n0 = t / tiles_m * fo; return t % tiles_m; }
  const int half = t < whole ? 0 : (t - whole) & 1, tile = t < whole ? t : whole + ((t - whole) >> 1);
  n0 = tile / tiles_m * fo + half * (fo / 2);
  return tile % tiles_m;
}

// tiles_total: whole tiles and halves.  tmap_half: w in boxes of half a tile's rows (HALVES).
template <typename Cfg, typename TO>
__global__ void __launch_bounds__(G_THREADS, 1)
linear_tcgen05_pair_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_w,
                           const __grid_constant__ CUtensorMap tmap_half, TO* __restrict__ out, int n_rows, int o_out, int k_dim,
                           int tiles_m, int tiles_whole, int tiles_total, int* __restrict__ err, TcFold fold) {
  constexpr int EPI = Cfg::EPI, NACC = Cfg::NACC, FO = Cfg::FO, STAGES = Cfg::STAGES;
  extern __shared__ unsigned char g_smem_raw[];
  const uint32_t raw = g_smem_u32(g_smem_raw);
  unsigned char* smem = g_smem_raw + (((raw + 1023u) & ~1023u) - raw);      // the same offset in both CTAs
  unsigned char* staging = smem + STAGES * Cfg::STAGE_BYTES;
  uint64_t* full = reinterpret_cast<uint64_t*>(staging + Cfg::STAGING_BYTES);
  uint64_t* empty = full + STAGES;
  uint64_t* acc_full = empty + STAGES;                         // [2]: a tile's products are in accumulator b
  uint64_t* acc_empty = acc_full + 2;                          // [2], the first CTA's: the sixteen epilogue warps have read it
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;     // warp-uniform
  const int rank = blockIdx.x & 1;                             // the cluster is two neighbours along x
  const int kblocks = (k_dim + G_BK - 1) / G_BK;
  // this pair's tiles: first, first + step, ... (tc_pair_place)
  const int first = blockIdx.x >> 1, step = gridDim.x >> 1;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(&acc_full[b], 1); mbar_init(&acc_empty[b], 16); }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(g_smem_u32(tmem_slot)), "r"(Cfg::TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;\n" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();                                          // both CTAs' barriers exist before either CTA's copies count on them
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    // ---- producer, in both CTAs.  The w tiles of the first stages are requested before the wait for the predecessor.
    int g = 0;                                                  // k blocks issued so far, over all tiles
    bool waited = false, ok = true;
    for (int t = first; t < tiles_total && ok; t += step) {
      int n0;
      const int m0 = tc_pair_place<Cfg::HALVES>(t, tiles_whole, tiles_m, FO, n0) * (2 * G_BM) + rank * G_BM;
      const bool half = Cfg::HALVES && t >= tiles_whole;
      const int w0 = EPI ? rank * o_out + n0 : n0 + rank * (half ? Cfg::W_ROWS / 2 : Cfg::W_ROWS);
      for (int kb = 0; kb < kblocks; ++kb, ++g) {
        const int s = g % STAGES;
        if (g >= STAGES && !mbar_wait(&empty[s], ((g / STAGES) - 1) & 1, abort_flag, err, 1)) { ok = false; break; }
        unsigned char* stage = smem + s * Cfg::STAGE_BYTES;
        const uint32_t bar = cluster_addr(&full[s], 0);
        if (elect_one()) {
          if (rank == 0) mbar_expect_tx(&full[s], half ? 2 * Cfg::A_BYTES + Cfg::B_BYTES : 2 * Cfg::STAGE_BYTES);
          tma_load_2d_pair(stage + Cfg::A_BYTES, half ? &tmap_half : &tmap_w, bar, kb * G_BK, w0);
        }
        __syncwarp();
        if (!waited && (g == STAGES - 1 || (kb == kblocks - 1 && t + step >= tiles_total))) {
          // the ring is full of w tiles (or there are no more): now the predecessor, then the x tiles held back
          ifb_pdl_wait();
          ifb_pdl_trigger();
          waited = true;
          int gg = 0;
          for (int tt = first; tt < tiles_total && gg <= g; tt += step) {
            int nn;
            const int mm = tc_pair_place<Cfg::HALVES>(tt, tiles_whole, tiles_m, FO, nn) * (2 * G_BM) + rank * G_BM;
            for (int kk = 0; kk < kblocks && gg <= g; ++kk, ++gg) {
              const uint32_t bb = cluster_addr(&full[gg % STAGES], 0);
              if (elect_one()) tma_load_2d_pair(smem + (gg % STAGES) * Cfg::STAGE_BYTES, &tmap_x, bb, kk * G_BK, mm);
              __syncwarp();
            }
          }
        } else if (waited) {
          if (elect_one()) tma_load_2d_pair(stage, &tmap_x, bar, kb * G_BK, m0);
          __syncwarp();
        }
      }
    }
    if (!waited) { ifb_pdl_wait(); ifb_pdl_trigger(); }         // a CTA without tiles still orders itself behind the predecessor
  } else if (warp == 1) {
    // ---- issuer, in the first CTA: tile i of this pair accumulates in accumulator i & 1
    int g = 0, it = 0;
    bool ok = rank == 0;
    for (int t = first; t < tiles_total && ok; t += step, ++it) {
      const int b = it & 1;
      if (it >= 2) ok = mbar_wait(&acc_empty[b], ((it >> 1) - 1) & 1, abort_flag, err, 4);
      if (!ok) break;
      tc_fence_after();
      for (int kb = 0; kb < kblocks && ok; ++kb, ++g) {
        const int s = g % STAGES;
        ok = mbar_wait(&full[s], (g / STAGES) & 1, abort_flag, err, 2);
        if (!ok) break;
        tc_fence_after();
        if (elect_one()) {
          const uint32_t a_addr = g_smem_u32(smem + s * Cfg::STAGE_BYTES);
          const uint64_t a_desc = make_smem_desc(a_addr), b_desc = make_smem_desc(a_addr + Cfg::A_BYTES);
#pragma unroll
          for (int k = 0; k < G_BK / G_UK; ++k) {
            const uint64_t kstep = (uint64_t)((k * G_UK * 2) >> 4);          // 32 bytes per k step, in 16-byte units
            umma_bf16_pair(tmem_base + b * NACC, a_desc + kstep, b_desc + kstep, Cfg::HALVES && t >= tiles_whole ? Cfg::IDESC_HALF : Cfg::IDESC, (kb | k) != 0);
          }
          umma_commit_pair(&empty[s]);
          if (kb == kblocks - 1) umma_commit_pair(&acc_full[b]);
        }
        __syncwarp();
      }
    }
  } else {
    // ---- epilogue, in both CTAs, each its own 128 tokens.  A warp's piece of a tile is 32 tokens (its lanes) by CW features.
    constexpr int CW = FO / 2;
    constexpr int PITCH = Cfg::STAGING_PITCH;
    const int q = warp & 3;                                      // this warp's quarter of the 128 lanes
    const int c_lo = ((warp - 2) >> 2) * CW;                     // and its half of the tile's features
    unsigned char* buf = staging + (warp - 2) * (32 * PITCH);
    int it = 0;
    bool ok = true;
    if (fold.rs_partials || Cfg::ROWS32) ifb_pdl_wait();         // what the predecessors wrote is read here directly
    for (int t = first; t < tiles_total && ok; t += step, ++it) {
      const int b = it & 1;
      int n0;
      const int row0 = tc_pair_place<Cfg::HALVES>(t, tiles_whole, tiles_m, FO, n0) * (2 * G_BM) + rank * G_BM + q * 32;
      const uint32_t lane_base = tmem_base + ((uint32_t)(q * 32) << 16) + b * NACC;
      float rfac = tc_row_factor(fold, row0 + lane, n_rows);
      if constexpr (Cfg::ROWS32) {
        // whole rows of float32, 64 features at a time: the residual addition, or heads of 128
        constexpr int AHEAD = 16;
        float4 ahead[AHEAD], angles[AHEAD / 2][2];
        int slot_of[AHEAD / 2];
        const int head = (n0 + c_lo) / 128;
        const bool qk_v = head >= fold.qk_nq + fold.qk_nkv, qk_k = head >= fold.qk_nq && !qk_v;
        const bool heads = CW == 128 && sizeof(TO) == 2 && fold.qk_nq > 0;
        const bool rotate = !qk_v && fold.qk_rope, store = (qk_v || qk_k) && fold.qk_slots;
        if (heads) tc_heads_load<32, AHEAD / 2>(fold, row0, n_rows, 0, rotate, store, lane, angles, slot_of);
        else if (n0 + c_lo < o_out) tc_residual_load<64, AHEAD>(fold, row0, n_rows, n0 + c_lo, o_out, lane, ahead);
        ok = mbar_wait(&acc_full[b], (it >> 1) & 1, abort_flag, err, 3);
        if (!ok) break;
        tc_fence_after();
        if (row0 < n_rows && n0 + c_lo < o_out) {                // warp-uniform
          if (heads) {
            if constexpr (sizeof(TO) == 2 && CW == 128) {
              const void* wn = qk_v ? nullptr : qk_k ? fold.qk_kw : fold.qk_qw;
              if (wn) {
                float ss[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 1
                for (int c0 = 0; c0 < 128; c0 += 32) {
                  uint32_t v[32];
                  tmem_ld32(lane_base + c_lo + c0, v);
                  tmem_ld_wait();
#pragma unroll
                  for (int j = 0; j < 32; ++j) { const float f = __uint_as_float(v[j]) * rfac; ss[j & 3] = fmaf(f, f, ss[j & 3]); }
                }
                rfac *= rsqrtf(((ss[0] + ss[1]) + (ss[2] + ss[3])) * (1.f / 128.f) + fold.qk_eps);
              }
#pragma unroll 1
              for (int i0 = 0; i0 < 64; i0 += 32) {
                if (i0) tc_heads_load<32, AHEAD / 2>(fold, row0, n_rows, i0, rotate, store, lane, angles, slot_of);
                tc_stage_rows(lane_base + c_lo + i0, buf + lane * PITCH, rfac);
                tc_stage_rows(lane_base + c_lo + 64 + i0, buf + lane * PITCH + 128, rfac);
                __syncwarp();
                tc_finish_heads<32, PITCH, AHEAD / 2>(fold, buf, reinterpret_cast<bf16*>(out), row0, n_rows, head, i0, o_out, wn, qk_v, rotate,
                                                      store, lane, angles, slot_of);
                __syncwarp();
              }
            }
          } else {
#pragma unroll 1
            for (int c0 = c_lo; c0 < c_lo + CW && n0 + c0 < o_out; c0 += 64) {
              if (c0 != c_lo) tc_residual_load<64, AHEAD>(fold, row0, n_rows, n0 + c0, o_out, lane, ahead);
              tc_stage_rows(lane_base + c0, buf + lane * PITCH, rfac);
              tc_stage_rows(lane_base + c0 + 32, buf + lane * PITCH + 128, rfac);
              __syncwarp();
              tc_finish_residual<64, PITCH, AHEAD, TO>(fold, buf, out, row0, n_rows, n0 + c0, o_out, (n0 + c0) / 64, lane, ahead);
              __syncwarp();
            }
          }
        }
      } else {
        constexpr int LEAST = Cfg::HALVES ? CW / 2 : CW;         // features of a warp's piece of a half
        constexpr int PW = 128 / (int)sizeof(TO) < LEAST ? 128 / (int)sizeof(TO) : LEAST, SEG = PW * (int)sizeof(TO);   // per staged row segment
        static_assert(LEAST % PW == 0, "a warp's features are whole row segments");
        ok = mbar_wait(&acc_full[b], (it >> 1) & 1, abort_flag, err, 3);
        if (!ok) break;
        tc_fence_after();
        const bool half = Cfg::HALVES && t >= tiles_whole;
        const int cw = half ? CW / 2 : CW, c_at = half ? c_lo / 2 : c_lo, fo = half ? FO / 2 : FO;
        const bool vec = ((size_t)o_out * sizeof(TO)) % 16 == 0 && (((uintptr_t)out) & 15) == 0 && n0 + c_at + cw <= o_out;
#pragma unroll 1
        for (int p0 = c_at; p0 < c_at + cw; p0 += PW) {
          if (n0 + p0 >= o_out || row0 >= n_rows) break;         // warp-uniform
#pragma unroll
          for (int c0 = p0; c0 < p0 + PW; c0 += 32) {
            float y[32];
            tc_epilogue_row<EPI>(fold, lane_base + c0, fo, rfac, n0 + c0, o_out, y);
            if (vec) tc_pack_row<TO>(buf + lane * PITCH + (c0 - p0) * (int)sizeof(TO), y);
            else if (row0 + lane < n_rows) {
              TO* dst = out + (size_t)(row0 + lane) * o_out + n0 + c0;
#pragma unroll
              for (int j = 0; j < 32; ++j)
                if (n0 + c0 + j < o_out) dst[j] = from_f32<TO>(y[j]);
            }
          }
          if (vec) {
            __syncwarp();
            unsigned char* obase = reinterpret_cast<unsigned char*>(out + (size_t)row0 * o_out + n0 + p0);
#pragma unroll
            for (int off = lane * 16; off < 32 * SEG; off += 512) {
              const int r = off / SEG, cb = off % SEG;
              if (row0 + r < n_rows)
                *reinterpret_cast<uint4*>(obase + (size_t)r * o_out * sizeof(TO) + cb) = *reinterpret_cast<const uint4*>(buf + r * PITCH + cb);
            }
            __syncwarp();                                        // before the next segment overwrites the rows
          }
        }
      }
      // this warp has read its part of accumulator b: the issuer may overwrite it (with the tile after next)
      tc_fence_before();
      __syncwarp();
      if (lane == 0)
        asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];\n" ::"r"(cluster_addr(&acc_empty[b], 0)) : "memory");
    }
  }
  if (*abort_flag) {                         // a wait gave up: let copies in flight land before the CTA goes away
    for (int i = 0; i < 2000; ++i) __nanosleep(1000);
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();                        // neither CTA leaves while the other's products or arrivals need its memory
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(Cfg::TMEM_COLS) : "memory");
  }
}

// How many pairs of a kernel the device runs at a time (known once per device and kernel; 0 if it cannot say).
template <typename Cfg, typename TO>
static int tc_pairs() {
  static int known[IFB_MAX_DEVICES] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= IFB_MAX_DEVICES) return 0;
  if (!known[dev]) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2);
    cfg.blockDim = dim3(G_THREADS);
    cfg.dynamicSmemBytes = Cfg::SMEM_BYTES;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaFuncSetAttribute(linear_tcgen05_pair_kernel<Cfg, TO>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Cfg::SMEM_BYTES) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, linear_tcgen05_pair_kernel<Cfg, TO>, &cfg) != cudaSuccess || n < 1) {
      cudaGetLastError();
      return 0;
    }
    known[dev] = n;
  }
  return known[dev];
}

// Tiles of the last round that are halved: all of them, where whole rounds come before it and its halves find a pair each.  From a k of
// 512: below it the products of a round are shorter than its epilogue (gate and up of 3,072 features at 818 rows: k 256 7.3 us on the
// persistent kernel and 8.5 so, k 512 10.1 and 9.8; plain 2,304 x 256 at 5,000 rows 11.3 whole, 11.7 halved).
static int tc_pair_halved(int pairs, long long tiles, int k) {
  const int rest = (int)(tiles % pairs);
  return k >= 512 && tiles > pairs && 2 * rest <= pairs ? rest : 0;
}

template <typename Cfg, typename TO>
static int tc_launch_pair(const void* x, const void* w, void* out, int n, int o, int k, int* err, cudaStream_t s, const TcFold& fold) {
  CUtensorMap mx, mw;
  int st = make_map(&mx, x, n, k, G_BM);
  if (st) return st;
  st = make_map(&mw, w, Cfg::EPI ? 2 * o : o, k, Cfg::W_ROWS);
  if (st) return st;
  const int pairs = tc_pairs<Cfg, TO>();
  if (!pairs) return IFB_ERR_ARG;
  IFB_ALLOW_SMEM((linear_tcgen05_pair_kernel<Cfg, TO>), Cfg::SMEM_BYTES);
  const long long tiles_m = (n + 2 * G_BM - 1) / (2 * G_BM), tiles_n = (o + Cfg::FO - 1) / Cfg::FO;
  if (tiles_m * tiles_n > 0x3fffffffLL) return IFB_ERR_SIZE;
  int total = (int)(tiles_m * tiles_n);
  const int halved = tc_pair_halved(pairs, total, k), whole = total - (Cfg::HALVES ? halved : 0);
  CUtensorMap mh = mw;
  if constexpr (Cfg::HALVES) {
    total += halved;
    st = make_map(&mh, w, Cfg::EPI ? 2 * o : o, k, Cfg::W_ROWS / 2);
    if (st) return st;
  } else if constexpr (!Cfg::ROWS32 && Cfg::NACC == 256) {        // (a kernel of its own: the second epilogue costs the first registers)
    if (halved) return tc_launch_pair<PairCfg<Cfg::EPI, 256, Cfg::STAGES, false, true>, TO>(x, w, out, n, o, k, err, s, fold);
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * (total < pairs ? total : pairs));
  cfg.blockDim = dim3(G_THREADS);
  cfg.dynamicSmemBytes = Cfg::SMEM_BYTES;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = ifb_pdl_enabled() ? 2 : 1;
  cudaError_t e = cudaLaunchKernelEx(&cfg, linear_tcgen05_pair_kernel<Cfg, TO>, mx, mw, mh, (TO*)out, n, o, k, (int)tiles_m, whole, total, err, fold);
  if (e != cudaSuccess) { cudaGetLastError(); return -(int)e; }
  return IFB_OK;
}

template <typename Cfg, typename TO>
static int tc_launch_persistent(const void* x, const void* w, void* out, int n, int o, int k, int* err, int sm_count, cudaStream_t s,
                                const TcFold& fold) {
  CUtensorMap mx, mw;
  int st = make_map(&mx, x, n, k, G_BM);
  if (st) return st;
  st = make_map(&mw, w, Cfg::EPI ? 2 * o : o, k, Cfg::EPI ? Cfg::NACC / 2 : Cfg::NACC);
  if (st) return st;
  IFB_ALLOW_SMEM((linear_tcgen05_persistent_kernel<Cfg, TO>), Cfg::SMEM_BYTES);
  const long long tiles_m = (n + G_BM - 1) / G_BM, tiles_n = (o + Cfg::FO - 1) / Cfg::FO;
  if (tiles_m * tiles_n > 0x7fffffffLL) return IFB_ERR_SIZE;
  const int total = (int)(tiles_m * tiles_n);
  const int grid = total < sm_count ? total : sm_count;
  return ifb_launch(linear_tcgen05_persistent_kernel<Cfg, TO>, dim3(grid), dim3(G_THREADS), (size_t)Cfg::SMEM_BYTES, s, mx, mw, (TO*)out, n,
                    o, k, (int)tiles_m, total, err, fold);
}

template <typename Cfg, typename TO>
static int tc_launch_cfg(const void* x, const void* w, void* out, int n, int o, int k, int* err, cudaStream_t s, const TcFold& fold,
                         int splits = 1, long long w_rows = 0) {
  CUtensorMap mx, mw;
  int st = make_map(&mx, x, n, k, Cfg::MH * G_BM);
  if (st) return st;
  if (w_rows > 0x7fffffffLL) return IFB_ERR_SIZE;
  st = make_map(&mw, w, w_rows ? (int)w_rows : (Cfg::EPI ? 2 * o : o), k, Cfg::EPI ? Cfg::NACC / 2 : Cfg::NACC);
  if (st) return st;
  IFB_ALLOW_SMEM((linear_tcgen05_kernel<Cfg, TO>), Cfg::SMEM_BYTES);
  dim3 grid((o + Cfg::FO - 1) / Cfg::FO, (n + Cfg::MH * G_BM - 1) / (Cfg::MH * G_BM), splits);
  if (grid.y > 65535) return IFB_ERR_SIZE;
  if (splits == 1)
    return ifb_launch(linear_tcgen05_kernel<Cfg, TO>, grid, dim3(G_THREADS), (size_t)Cfg::SMEM_BYTES, s, mx, mw, (TO*)out, n, o, k, err, 1, fold);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(G_THREADS);
  cfg.dynamicSmemBytes = Cfg::SMEM_BYTES;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = splits;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = ifb_pdl_enabled() ? 2 : 1;
  cudaError_t e = cudaLaunchKernelEx(&cfg, linear_tcgen05_kernel<Cfg, TO>, mx, mw, (TO*)out, n, o, k, err, splits, fold);
  if (e != cudaSuccess) { cudaGetLastError(); return -(int)e; }
  return IFB_OK;
}

// The shape of the tiles: a wave of wide tiles does four 128 x 128 products per SM in little more time than a wave of
// narrow tiles (two CTAs per SM) does two, but only if there are enough wide tiles to fill the SMs.  shape: 0 chooses
// (see below), 1 narrow, 2 deep, 3 wide, 4 and 5 persistent, 6 the pairs (for tests and measurements).
// By measurement.  With the silu_gate epilogue: tiles of 64 features (64 gate and 64 up rows, one tile per CTA, a deep ring) where
// they are no more than the SMs: twice the SMs of tiles of 128, each with two thirds of the bytes.  Else the persistent kernel (its tile already accumulates 256 columns per
// product, and the heavy epilogue of one tile runs beside the products of the next).  Otherwise one tile per CTA:
// the wide shape when there are enough wide tiles to fill the SMs (a 256 x 256 tile reads half the operand bytes
// per product from shared memory, which is what bounds these kernels), else the deep or the narrow one.
static int tc_pick_shape(int epi, int n, int o, int sm_count) {
  if (epi) return (long long)((o + 63) / 64) * ((n + G_BM - 1) / G_BM) <= sm_count ? 7 : 4;
  const long long tn = (long long)((o + 127) / 128) * ((n + G_BM - 1) / G_BM);
  const long long tw = (long long)((o + 255) / 256) * ((n + 2 * G_BM - 1) / (2 * G_BM));
  const double cost_narrow = (double)((tn + 2 * sm_count - 1) / (2 * sm_count));
  const double cost_wide = (double)((tw + sm_count - 1) / sm_count) * 1.15;
  return (n > G_BM && cost_wide < cost_narrow) ? 3 : (tn <= sm_count ? 2 : 1);
}

// Whether the kernel over pairs of SMs takes a product (a rule on sizes and on the epilogue's kind alone, as the parts of a folded
// norm must agree with the launch): from 513 rows on (up to 512 few tiles share their k range in clusters), where its own tiles keep
// most pairs busy (four fifths over all rounds).
// `pairs`: of SMs; 0 where the device cannot run the largest of their kernels, or there is none: never.
static int tc_device_pairs() { return tc_pairs<PairCfg<0, 128, 6, true>, bf16>() > 0 ? ifb_sm_count() / 2 : 0; }
static int tc_pair_rounds(int pairs, int n, int o, int features) {
  const long long tiles = (long long)((n + 255) / 256) * ((o + features - 1) / features);
  return (int)((tiles + pairs - 1) / pairs);
}
enum TcKind { TC_PLAIN, TC_RESIDUAL, TC_HEADS, TC_GATED };     // the epilogues whose weight differs
static TcKind tc_kind(int epi, const TcFold& f) { return epi ? TC_GATED : f.res_x ? TC_RESIDUAL : f.qk_nq > 0 ? TC_HEADS : TC_PLAIN; }
// Features of the tiles of a launch over pairs: 128 with the silu_gate epilogue (their gate and up rows); two whole heads for the
// fused q | k | v product; else the quicker, a round of narrow tiles taking 0.7 of a wide one's time: an SM gets 24 KB per 64 of k
// where it gets 32 (2,048 x 1,024 x 2,048: one round of 64 narrow tiles 10.9 us).
static int tc_pair_features(int pairs, TcKind kind, int n, int o) {
  if (kind == TC_GATED) return 128;
  if (kind == TC_HEADS || pairs < 1) return 256;
  return 0.7 * tc_pair_rounds(pairs, n, o, 128) < tc_pair_rounds(pairs, n, o, 256) ? 128 : 256;
}
// The heads' epilogue is as long as the products of a k of 1,024, and in a single round there are no other tile's products to run
// it beside: steps of 850 and 1,000 rows of the 0.6B sizes (4,096 x 1,024, one round) 723 and 739 us for eight layers with it over
// pairs, 687 and 708 without, of 1,800 and 2,048 rows (two rounds) 930 and 978 against 911 and 967; six layers of the 8B sizes
// (6,144 x 4,096) at 513 rows (one round) 1,739 against 1,695, at 1,500 (two) 3,163 and 3,151, at 2,048 (three) 3,899 against 4,055.
static bool tc_pick_pair(int pairs, TcKind kind, int n, int o, int k) {
  if (o % 64 || n <= 512 || pairs < 1) return false;
  const int features = tc_pair_features(pairs, kind, n, o), rounds = tc_pair_rounds(pairs, n, o, features);
  if (kind == TC_HEADS && (rounds < 2 || k < 2048)) return false;
  const long long tiles = (long long)((n + 255) / 256) * ((o + features - 1) / features);
  return tiles * 10 >= (long long)pairs * 8 * rounds;
}
// Tiles of the last round that are halved, 0 for none.  A product with such a round takes the pairs even where whole tiles would leave
// more than a fifth of them idle, if the kernel it would go to needs a round more than the whole ones here: plain products that go to the wide
// tiles (0.62 to 0.92 of their time over 144 products of 512 to 12,288 features, k 512 to 4,096, 513 to 3,000 rows; against narrow tiles 0.92 to
// 1.31, most of them one round, 1,100 rows of 4,096 x 1,024 13.0 us and 16.3 so), gated ones from a k of 1,024 on with more rounds of the persistent kernel
// (0.71 to 1.0; with as many 0.93 to 1.36, 1,100 rows of 2,048 x 4,096 27.8 and 36.5, and below that k up to 1.12).  Gate and up of 3,072 x 1,024 at 818 rows
// 16.1 us on the persistent kernel, 12.9 so, at 1,600 rows 21.8 and 17.4; 6,144 x 2,048 at 818 rows 27.8 and 21.7, at 1,600 50 and 31.
static int tc_pick_halves(int pairs, TcKind kind, int n, int o, int k) {
  if (o % 64 || n <= 512 || pairs < 1 || (kind != TC_PLAIN && kind != TC_GATED)) return 0;
  const int features = tc_pair_features(pairs, kind, n, o), sms = 2 * pairs;
  if (features != (kind == TC_GATED ? 128 : 256)) return 0;
  const long long tiles = (long long)((n + 255) / 256) * ((o + features - 1) / features);
  const int halved = tc_pair_halved(pairs, tiles, k);
  if (!halved || tc_pick_pair(pairs, kind, n, o, k)) return halved;
  const int shape = tc_pick_shape(kind == TC_GATED, n, o, sms);
  if (kind == TC_PLAIN) return shape == 3 ? halved : 0;
  const long long alone = (long long)((n + G_BM - 1) / G_BM) * ((o + 127) / 128);
  return shape == 4 && k >= 1024 && (alone + sms - 1) / sms > tiles / pairs ? halved : 0;
}

template <int EPI, typename TO>
static int tc_launch(const void* x, const void* w, void* out, int n, int o, int k, int* err, int shape, int splits, const TcFold& fold,
                     cudaStream_t s) {
  using Narrow = GemmCfg<EPI, 1, EPI ? 256 : 128, EPI ? 2 : 3>;
  using Deep = GemmCfg<EPI, 1, EPI ? 256 : 128, EPI ? 4 : 6>;
  using Wide = GemmCfg<EPI, 2, 256, 3>;
  using P128 = PersistCfg<EPI, EPI ? 256 : 128, EPI ? 3 : 5>;      // 128 features per tile
  using P256 = PersistCfg<EPI, 256, 3>;                            // 256 features per tile (plain epilogue only)
  if (splits > 1) {
    static_assert(G_BM * (Deep::NACC + 4) * 4 <= Deep::STAGES * Deep::STAGE_BYTES, "the float32 tile must fit in the stages");
    if (splits > 8) return IFB_ERR_ARG;
    return tc_launch_cfg<Deep, TO>(x, w, out, n, o, k, err, s, fold, splits);
  }
  if (shape == 0) {
    const int pairs = tc_device_pairs();
    const TcKind kind = tc_kind(EPI, fold);
    shape = tc_pick_pair(pairs, kind, n, o, k) || tc_pick_halves(pairs, kind, n, o, k) > 0 ? 6 : tc_pick_shape(EPI, n, o, ifb_sm_count());
  }
  if (EPI && fold.res_x) return IFB_ERR_ARG;
  if (shape == 6) {
    using Pair = PairCfg<EPI, 256, 5, false>;
    if constexpr (!EPI) {
      using Rows256 = PairCfg<0, 256, 4, true>;
      using Rows128 = PairCfg<0, 128, 6, true>;
      using Pair128 = PairCfg<0, 128, 7, false>;
      const bool narrow = tc_pair_features(tc_device_pairs(), tc_kind(0, fold), n, o) == 128;
      if (fold.qk_nq || fold.res_x) {
        if (o % 64) return IFB_ERR_ARG;                              // (a forced shape: the rule asks for it)
        return narrow ? tc_launch_pair<Rows128, TO>(x, w, out, n, o, k, err, s, fold) : tc_launch_pair<Rows256, TO>(x, w, out, n, o, k, err, s, fold);
      }
      if (narrow) return tc_launch_pair<Pair128, TO>(x, w, out, n, o, k, err, s, fold);
    }
    return tc_launch_pair<Pair, TO>(x, w, out, n, o, k, err, s, fold);
  }
  if (fold.res_x && shape > 3) return IFB_ERR_ARG;        // the making side is the one-tile kernel's
  if (shape == 7) {
    if constexpr (EPI) return tc_launch_cfg<GemmCfg<1, 1, 128, 6>, TO>(x, w, out, n, o, k, err, s, fold);
    return IFB_ERR_ARG;
  }
  if (shape == 5 && !EPI) return tc_launch_persistent<P256, TO>(x, w, out, n, o, k, err, ifb_sm_count(), s, fold);
  if (shape == 4 || shape == 5) return tc_launch_persistent<P128, TO>(x, w, out, n, o, k, err, ifb_sm_count(), s, fold);
  if (shape == 3) return tc_launch_cfg<Wide, TO>(x, w, out, n, o, k, err, s, fold);
  if (shape == 2) return tc_launch_cfg<Deep, TO>(x, w, out, n, o, k, err, s, fold);
  return tc_launch_cfg<Narrow, TO>(x, w, out, n, o, k, err, s, fold);
}

// epilogue: 0 plain, 1 silu_gate, 16 * u: plain with the unary function u of common.cuh applied to every element,
// 1 + 16 * u: gated with u in silu's place.
// x [n_rows, k] and w [out_features (x2 for the silu_gate epilogue), k] bfloat16, 16-byte aligned, k a multiple of 8;
// out bfloat16 or float32.  `err` points to a device int that stays 0 unless a bounded wait gave up.  shape: 0 lets the
// library choose, 1-3 force the one-tile-per-CTA kernel narrow, deep or wide, 4 and 5 the persistent kernel with tiles of 128
// or 256 features, 6 the kernel over pairs of SMs, 7 (silu_gate) the one-tile kernel with 64 features.  splits 2 to 8: the k range of a tile of 128 x 128 is shared by a cluster of
// that many CTAs, whose parts are added in a fixed order; for few tiles of a long k (a step of some tens of tokens).
// scale_partials (may be null): [scale_parts][n_rows] sums of squares; output row n is multiplied by
// rsqrt(sum_p partials[p][n] / scale_width + scale_eps) before the epilogue.
// res_x (may be null; plain epilogue, shapes 0-3 and, with out_features a multiple of 64, 6): the residual stream [n_rows][out_features] float32: v = x + y is
// written back to it, out = v * res_g, and res_partials [ifb_linear_tcgen05_fold_parts(...)][n_rows] gets sums of v^2.
// bias (may be null; plain epilogue): float32 [out_features], added to the (scaled) product.
IFB_EXPORT int ifb_linear_tcgen05_ex(const void* x, const void* w, void* out, int out_dtype, int n_rows, int out_features,
                                     int k_dim, int epilogue, int shape, int splits, const float* scale_partials, int scale_parts,
                                     float scale_eps, int scale_width, float* res_x, const void* res_g, int res_g_dtype,
                                     float* res_partials, const float* bias, int* err, cudaStream_t stream) {
  if (n_rows <= 0 || out_features <= 0) return IFB_OK;
  if (k_dim < 8 || k_dim % 8) return IFB_ERR_SIZE;
  if (((uintptr_t)x & 15) || ((uintptr_t)w & 15)) return IFB_ERR_ALIGN;
  const int unary = epilogue >> 4;
  epilogue &= 15;
  if (epilogue > 1 || unary < 0 || unary > IFB_UNARY_LAST || (unary && res_x) || (bias && epilogue))
    return IFB_ERR_ARG;
  if (shape < 0 || shape > 7 || splits < 0 || splits > 8) return IFB_ERR_ARG;
  if (scale_partials && (scale_parts < 1 || scale_width < 1)) return IFB_ERR_ARG;
  if (res_x && (!res_g || !res_partials || ((uintptr_t)res_x & 15))) return IFB_ERR_ARG;
  TcFold fold = {};
  fold.rs_partials = scale_partials; fold.rs_parts = scale_parts; fold.rs_eps = scale_eps;
  fold.rs_inv_width = scale_partials ? 1.f / (float)scale_width : 0.f;
  fold.res_x = res_x; fold.res_g = res_g; fold.res_g_dtype = res_g_dtype; fold.res_partials = res_partials;
  fold.unary = unary;
  fold.bias = bias;
  if (out_dtype == IFB_BF16)
    return epilogue ? tc_launch<1, bf16>(x, w, out, n_rows, out_features, k_dim, err, shape, splits, fold, stream)
                    : tc_launch<0, bf16>(x, w, out, n_rows, out_features, k_dim, err, shape, splits, fold, stream);
  if (out_dtype == IFB_F32)
    return epilogue ? tc_launch<1, float>(x, w, out, n_rows, out_features, k_dim, err, shape, splits, fold, stream)
                    : tc_launch<0, float>(x, w, out, n_rows, out_features, k_dim, err, shape, splits, fold, stream);
  return IFB_ERR_DTYPE;
}

// The grouped product of routed experts.  x [rows, k]: the rows sorted by expert in segments padded to 128 (rows a multiple
// of 128); w [experts][out_features (x2 with the silu_gate epilogue)][k]; tile_expert [rows / 128]: the expert of each tile of
// rows, negative for unused tiles (device memory, written by a kernel before this one in the stream); out [rows, out_features].
IFB_EXPORT int ifb_linear_tcgen05_grouped(const void* x, const void* w, void* out, int out_dtype, int rows, int experts,
                                          int out_features, int k_dim, int epilogue, const int* tile_expert, int* err,
                                          cudaStream_t stream) {
  if (rows <= 0 || out_features <= 0) return IFB_OK;
  if (k_dim < 8 || k_dim % 8 || rows % G_BM || experts < 1) return IFB_ERR_SIZE;
  if (((uintptr_t)x & 15) || ((uintptr_t)w & 15)) return IFB_ERR_ALIGN;
  const int unary = epilogue >> 4;
  epilogue &= 15;
  if (epilogue > 1 || unary < 0 || unary > IFB_UNARY_LAST || (epilogue && unary) || !tile_expert) return IFB_ERR_ARG;
  TcFold fold = {};
  fold.unary = unary;
  fold.grp_tile_expert = tile_expert;
  fold.grp_w_rows = (epilogue ? 2 : 1) * out_features;
  const long long w_rows = (long long)experts * fold.grp_w_rows;
  using Plain = GemmCfg<0, 1, 128, 3>;
  using Gated = GemmCfg<1, 1, 256, 2>;
  if (out_dtype == IFB_BF16)
    return epilogue ? tc_launch_cfg<Gated, bf16>(x, w, out, rows, out_features, k_dim, err, stream, fold, 1, w_rows)
                    : tc_launch_cfg<Plain, bf16>(x, w, out, rows, out_features, k_dim, err, stream, fold, 1, w_rows);
  if (out_dtype == IFB_F32)
    return epilogue ? tc_launch_cfg<Gated, float>(x, w, out, rows, out_features, k_dim, err, stream, fold, 1, w_rows)
                    : tc_launch_cfg<Plain, float>(x, w, out, rows, out_features, k_dim, err, stream, fold, 1, w_rows);
  return IFB_ERR_DTYPE;
}

IFB_EXPORT int ifb_linear_tcgen05(const void* x, const void* w, void* out, int out_dtype, int n_rows, int out_features,
                                  int k_dim, int epilogue, int* err, int shape, cudaStream_t stream) {
  return ifb_linear_tcgen05_ex(x, w, out, out_dtype, n_rows, out_features, k_dim, epilogue, shape, 1, nullptr, 0, 0.f, 0, nullptr,
                               nullptr, 0, nullptr, nullptr, err, stream);
}

// The fused q | k | v projection of an attention layer with what follows it (see TcFold) in the epilogue of the one-tile
// kernel or of the pairs' (splits 1) or in the sum over the cluster of the shared-k form (splits 2 to 8): qkv [n_rows, (nq + 2 nkv) * 128] bfloat16 gets the normalised and rotated q heads (and the k and
// v heads as they are stored), the pages get k and v at slots[n].  Heads of 128, rotated whole in the half-split pairing
// (rope: [n_rows][64] pairs of cos and sin, 16-byte aligned, or null).  scale_*: as in ifb_linear_tcgen05_ex.
IFB_EXPORT int ifb_linear_tcgen05_qkv(const void* x, const void* w, void* qkv, int n_rows, int nq, int nkv, int head_dim, int k_dim,
                                      int splits, const float* scale_partials, int scale_parts, float scale_eps, int scale_width,
                                      const void* q_weight, const void* k_weight, int w_dtype, float eps, const float* rope,
                                      const int* slots, void* pages, int page_size, int* err, cudaStream_t stream) {
  if (n_rows <= 0) return IFB_OK;
  if (head_dim != 128 || nq < 1 || nkv < 1 || splits < 1 || splits > 8) return IFB_ERR_SIZE;
  if (k_dim < 8 || k_dim % 8) return IFB_ERR_SIZE;
  if (((uintptr_t)x & 15) || ((uintptr_t)w & 15) || ((uintptr_t)qkv & 15) || ((uintptr_t)pages & 15) || ((uintptr_t)rope & 15))
    return IFB_ERR_ALIGN;
  if ((q_weight || k_weight) && w_dtype != IFB_F32 && w_dtype != IFB_BF16) return IFB_ERR_DTYPE;
  if (scale_partials && (scale_parts < 1 || scale_width < 1)) return IFB_ERR_ARG;
  if (slots && (!pages || page_size < 1)) return IFB_ERR_ARG;
  TcFold fold = {};
  fold.rs_partials = scale_partials; fold.rs_parts = scale_parts; fold.rs_eps = scale_eps;
  fold.rs_inv_width = scale_partials ? 1.f / (float)scale_width : 0.f;
  fold.qk_nq = nq; fold.qk_nkv = nkv; fold.qk_qw = q_weight; fold.qk_kw = k_weight; fold.qk_w_dtype = w_dtype; fold.qk_eps = eps;
  fold.qk_rope = reinterpret_cast<const float2*>(rope); fold.qk_slots = slots; fold.qk_pages = (bf16*)pages;
  fold.qk_page_size = page_size;
  return tc_launch<0, bf16>(x, w, qkv, n_rows, (nq + 2 * nkv) * 128, k_dim, err, 0, splits, fold, stream);
}

// Features of the tiles with which a product of these sizes runs over pairs of SMs (shape 0, splits 1), or 0 where it runs on another
// kernel or over pairs for its halved tiles' sake alone.  kind: 0 plain, 1 with the residual addition, 2 the fused q | k | v product, 3 gated.  pairs: how many of them to answer
// for, 0: this device's.
IFB_EXPORT int ifb_linear_tcgen05_pair_tile(int kind, int n_rows, int out_features, int k_dim, int pairs) {
  if (kind < TC_PLAIN || kind > TC_GATED) return 0;
  if (!pairs) pairs = tc_device_pairs();
  return tc_pick_pair(pairs, (TcKind)kind, n_rows, out_features, k_dim) ? tc_pair_features(pairs, (TcKind)kind, n_rows, out_features) : 0;
}

// Tiles of a product's last round over pairs of SMs that are halved (shape 0, splits 1): 0 where none is, or another kernel takes it.
IFB_EXPORT int ifb_linear_tcgen05_pair_halved(int kind, int n_rows, int out_features, int k_dim, int pairs) {
  if (kind < TC_PLAIN || kind > TC_GATED) return 0;
  return tc_pick_halves(pairs ? pairs : tc_device_pairs(), (TcKind)kind, n_rows, out_features, k_dim);
}

// Parts of sums of squares that a product with res_x writes per row (the launch with shape 0 and these splits).
IFB_EXPORT int ifb_linear_tcgen05_fold_parts(int n_rows, int out_features, int splits) {
  if (splits > 1) return (out_features + 127) / 128;
  if (tc_pick_pair(tc_device_pairs(), TC_RESIDUAL, n_rows, out_features, 0)) return (out_features + 63) / 64;       // (whatever the k)
  return tc_pick_shape(0, n_rows, out_features, ifb_sm_count()) == 3 ? 2 * ((out_features + 255) / 256) : 2 * ((out_features + 127) / 128);
}

using SplitCfg = GemmCfg<0, 1, 128, 6>;

// How many clusters of `splits` CTAs of that kernel the device holds at a time (0 if it cannot say): a product whose
// tiles are no more than this runs in one wave.
IFB_EXPORT int ifb_linear_tcgen05_split_clusters(int splits) {
  static int cached_all[IFB_MAX_DEVICES][9] = {};
  static bool known_all[IFB_MAX_DEVICES][9] = {};
  int dev = 0;
  if (splits < 2 || splits > 8 || cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= IFB_MAX_DEVICES) return 0;
  int* cached = cached_all[dev];
  bool* known = known_all[dev];
  if (!known[splits]) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(1, 1, splits);
    cfg.blockDim = dim3(G_THREADS);
    cfg.dynamicSmemBytes = SplitCfg::SMEM_BYTES;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = splits;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int clusters = 0;
    if (cudaFuncSetAttribute(linear_tcgen05_kernel<SplitCfg, float>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)SplitCfg::SMEM_BYTES) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&clusters, linear_tcgen05_kernel<SplitCfg, float>, &cfg) != cudaSuccess) {
      cudaGetLastError();
      clusters = 0;
    }
    cached[splits] = clusters;
    known[splits] = true;
  }
  return cached[splits];
}
