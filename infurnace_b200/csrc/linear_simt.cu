// Matrix product out[n, o] = sum_k x[n, k] * w[o, k] with plain float32 multiply-adds: no tensor
// cores and no reduced-precision mode.  It is the product of the true 32-bit path and the
// fallback for operand dtypes or sizes that the tensor-core kernels refuse.  Any n, o, k.
//
// Three kernels.  Float32 operands: `rows32_kernel` up to 16 rows and `tile32_kernel` beyond; operands of which one is
// bfloat16: `linear_simt_kernel`.  The order in which an output's products are added depends on k alone, never on the
// number of rows or on the row's place, so a token's values are the same bits in every way of cutting the work:
// the bfloat16 combinations add them one after the other; float32 operands in S32_GROUPS consecutive parts of the k range,
// in each those of even and of odd k one after the other, and the parts as ((p0 + p1) + (p2 + p3)) + (p4 + p5) + (p6 + p7).  That is what lets several
// warps and CTAs share an output (and an eighth of the chain's length also leaves less rounding error than one chain).
#include "common.cuh"

#define TILE_N 64
#define TILE_O 64
#define TILE_K 16

constexpr int S32_GROUPS = 8;
constexpr int S32_BK = 16;                       // k of a stage of the tile kernel: groups are whole stages
// Length of each of the groups of the k range (the last ones may be shorter or empty).
__host__ __device__ __forceinline__ int s32_group(int k_dim) {
  return ((k_dim + S32_GROUPS - 1) / S32_GROUPS + S32_BK - 1) / S32_BK * S32_BK;
}
__device__ __forceinline__ float s32_total(const float (&p)[S32_GROUPS]) {
  return (((p[0] + p[1]) + (p[2] + p[3])) + (p[4] + p[5])) + (p[6] + p[7]);
}
// Two multiply-adds in one instruction (a and b: two neighbouring floats each): half the instructions at the rate of single ones
// (a warp's takes 2.2 cycles of a scheduler, a single one's 1.02).
__device__ __forceinline__ void s32_fma2(unsigned long long& acc, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;\n" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ float s32_pair_sum(unsigned long long v) {
  return __uint_as_float((uint32_t)v) + __uint_as_float((uint32_t)(v >> 32));
}
// VEC floats (4, or 1 where rows are not 16-byte aligned) from global to shared memory, or zeros where `in` is false.
template <bool VEC>
__device__ __forceinline__ void s32_copy(float* dst, const float* src, bool in) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  if (VEC) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src), "r"(in ? 16 : 0) : "memory");
  else asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(d), "l"(src), "r"(in ? 4 : 0) : "memory");
}
__device__ __forceinline__ void s32_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N> __device__ __forceinline__ void s32_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// ---------------------------------------------------------------------------------------------------
// Few rows (decoding): bound by the weights' bytes (one row, layers of the 0.6B sizes: 114 to 8.4 us for 4,096 x 1,024, 330 to 7.1
// us for 1,024 x 3,072 and, at 6.4 TB/s, 926 to 97 us for the head of 151,936 x 1,024, against a tile of 64 rows), so everything is about requesting them early and evenly.  A CTA of
// eight warps owns F rows of w and RB rows of x; warp g runs group g of the k range through its own ring of stages of 32 of
// k in shared memory, filled by 16-byte asynchronous copies (whole 128-byte pieces of a weight row), and lane l sums
// row l % F of w against the rows of x that its place gives it.  F = 8 puts enough CTAs on the device for the layers of a
// small model (1,024 features: 128 CTAs), F = 32 has more work per CTA where there are thousands of them (the LM head).
// EPI 1: the first F/2 rows of a CTA are gate rows, the others the up rows of the same features.
// The weights of the first stages are requested before the wait for the predecessor.
// ---------------------------------------------------------------------------------------------------
template <int F, int RB> struct Rows32 {
  static constexpr int NR = F == 32 ? RB : (RB + 3) / 4;          // rows of x per lane
  static constexpr int BK = 32, PITCH = 36;                       // 36 floats: eight lanes' 16-byte reads hit all banks once
  static constexpr int STAGES = F == 32 ? 3 : 6;
  static constexpr int STAGE = (F + RB) * PITCH;                  // floats
  static constexpr size_t SMEM = (size_t)S32_GROUPS * STAGES * STAGE * sizeof(float);
};

template <int F, int RB, int EPI, bool VEC, typename TO>
__global__ void __launch_bounds__(256)
rows32_kernel(const float* __restrict__ x, const float* __restrict__ w, TO* __restrict__ out, int n_rows, int o_out, int k_dim,
              int unary, const float* __restrict__ bias) {
  using C = Rows32<F, RB>;
  constexpr int STEP = VEC ? 4 : 1, PER = C::BK / STEP;           // copies per row of a stage
  extern __shared__ __align__(16) float s32_smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float* ring = s32_smem + (size_t)warp * C::STAGES * C::STAGE;
  constexpr int FO = EPI ? F / 2 : F;
  const int o0 = blockIdx.x * FO, n0 = blockIdx.y * RB;
  const int gl = s32_group(k_dim), kbeg = min(k_dim, warp * gl), kend = min(k_dim, kbeg + gl);
  const int steps = (kend - kbeg + C::BK - 1) / C::BK;
  auto load_w = [&](int st) {
    float* dst = ring + (st % C::STAGES) * C::STAGE;
    const int k0 = kbeg + st * C::BK;
#pragma unroll 4
    for (int i = lane; i < F * PER; i += 32) {
      const int r = i / PER, k = k0 + (i % PER) * STEP;
      const int o = o0 + (EPI ? r % FO : r);
      const bool in = o < o_out && k < kend;
      const size_t row = EPI && r >= FO ? (size_t)o_out + o : o;
      s32_copy<VEC>(dst + r * C::PITCH + (i % PER) * STEP, in ? w + row * k_dim + k : w, in);
    }
  };
  auto load_x = [&](int st) {
    float* dst = ring + (st % C::STAGES) * C::STAGE + F * C::PITCH;
    const int k0 = kbeg + st * C::BK;
#pragma unroll 2
    for (int i = lane; i < RB * PER; i += 32) {
      const int r = i / PER, k = k0 + (i % PER) * STEP;
      const bool in = n0 + r < n_rows && k < kend;
      s32_copy<VEC>(dst + r * C::PITCH + (i % PER) * STEP, in ? x + (size_t)(n0 + r) * k_dim + k : x, in);
    }
  };
#pragma unroll 1
  for (int st = 0; st < C::STAGES; ++st)
    if (st < steps) load_w(st);
  ifb_pdl_wait();
  ifb_pdl_trigger();
#pragma unroll 1
  for (int st = 0; st < C::STAGES; ++st) {
    if (st < steps) load_x(st);
    s32_commit();
  }
  const int f = lane % F, r0 = F == 32 ? 0 : (lane / F) * C::NR;
  unsigned long long acc[C::NR];                                  // sums over even and over odd k
#pragma unroll
  for (int r = 0; r < C::NR; ++r) acc[r] = 0;
#pragma unroll 1
  for (int st = 0; st < steps; ++st) {
    s32_wait<C::STAGES - 1>();
    __syncwarp();
    const float* ws = ring + (st % C::STAGES) * C::STAGE + f * C::PITCH;
    const float* xs = ring + (st % C::STAGES) * C::STAGE + F * C::PITCH;
#pragma unroll
    for (int k = 0; k < C::BK; k += 4) {
      const ulonglong2 wv = *reinterpret_cast<const ulonglong2*>(ws + k);
#pragma unroll
      for (int r = 0; r < C::NR; ++r) {
        const ulonglong2 xv = *reinterpret_cast<const ulonglong2*>(xs + min(r0 + r, RB - 1) * C::PITCH + k);
        s32_fma2(acc[r], xv.x, wv.x);
        s32_fma2(acc[r], xv.y, wv.y);
      }
    }
    __syncwarp();                                                 // the stage may be filled again
    if (st + C::STAGES < steps) { load_w(st + C::STAGES); load_x(st + C::STAGES); }
    s32_commit();
  }
  s32_wait<0>();
  __syncthreads();                                                // every ring is done with: the groups' sums go there
  float* red = s32_smem;                                          // [group][row][F]
#pragma unroll
  for (int r = 0; r < C::NR; ++r)
    if (r0 + r < RB) red[(warp * RB + r0 + r) * F + f] = s32_pair_sum(acc[r]);
  __syncthreads();
  for (int i = threadIdx.x; i < RB * FO; i += 256) {
    const int r = i / FO, c = i % FO, o = o0 + c, n = n0 + r;
    if (n >= n_rows || o >= o_out) continue;
    float p[S32_GROUPS];
#pragma unroll
    for (int g = 0; g < S32_GROUPS; ++g) p[g] = red[(g * RB + r) * F + c];
    float y = s32_total(p);
    if (EPI) {
#pragma unroll
      for (int g = 0; g < S32_GROUPS; ++g) p[g] = red[(g * RB + r) * F + FO + c];
      y = ifb_gate_act(y, unary) * s32_total(p);
    } else {
      if (bias) y += bias[o];
      if (unary) y = ifb_unary(y, unary);
    }
    out[(size_t)n * o_out + o] = from_f32<TO>(y);
  }
}

// ---------------------------------------------------------------------------------------------------
// Many rows: bound by the multiply-adds, of which two warps per scheduler keep one going every 3.5 cycles (2.5 is the least with
// operands in registers; four warps with half the outputs each, or single multiply-adds, are no faster).  The tile per thread is as large as
// the registers hold (a single chain per output had 22.5 TFLOP/s at 2,048 rows and, where 1,024 features
// leave most SMs without a tile, 4).  A cluster of two CTAs owns a tile of up to 64 rows of x by 64 rows of w; each of
// the eight slices of 64 threads (four per CTA) runs one group of the k range through its own ring of stages, a
// thread summing up to 8 x 8 outputs (16 16-byte reads of shared memory, free of bank conflicts, per 256 multiply-adds).  The
// groups' tiles then meet in the two CTAs' shared memory, each CTA adding half of the tile's rows.  EPI 1: the tile's first 32 rows of w are gate rows, the others the up rows of the same features.
// ALONE: where tiles are more than the pairs of SMs, a CTA takes a whole tile, each slice two groups one after the other in one run
// through its ring (of three stages; the first group's tile waits beside it).  Filling the ring and the sum at the end cost a CTA
// of a pair 17,000 of 37,000 cycles at a k of 1,024: 2,048 rows of 4,096 x 1,024 535 to 424 us (40 TFLOP/s), 193 rows of the LM head 2,371 to 1,837.
// RT: rows per thread, and an eighth of a tile's (tile32_form).  Eight take all 255 registers: a lone CTA spills 28 bytes (gated 128), single
// copies 188 to 592.
// ---------------------------------------------------------------------------------------------------
constexpr int T32 = 64, T32_SLICES = S32_GROUPS / 2, T32_PITCH = S32_BK + 4;      // 20 floats: conflict-free 16-byte reads
constexpr int T32_STAGE = 2 * T32 * T32_PITCH;                                    // floats: the rows of x, then those of w
constexpr int T32_LANES = 64, T32_TO = 8, T32_J = T32 / T32_TO;                   // threads of a slice, across features; features per thread
constexpr int T32_RED = T32 + 8;                                                  // floats per row of a group's tile
template <bool ALONE> struct Tile32 {
  static constexpr int STAGES = ALONE ? 3 : 4;
  static constexpr int RING = STAGES * T32_STAGE;                                 // floats of a slice's stages, then those of a first group's tile
  static constexpr int SLICE = RING + (ALONE ? T32 * T32_RED : 0);
  static constexpr size_t SMEM = (size_t)T32_SLICES * SLICE * sizeof(float);
  static_assert(T32 * T32_RED <= RING, "a group's tile goes where its stages were");
};

template <int EPI, bool VEC, bool ALONE, int RT, typename TO>
__global__ void __launch_bounds__(T32_SLICES * T32_LANES, 1)
tile32_kernel(const float* __restrict__ x, const float* __restrict__ w, TO* __restrict__ out, int n_rows, int o_out, int k_dim,
              int unary, const float* __restrict__ bias) {
  constexpr int STEP = VEC ? 4 : 1, PER = S32_BK / STEP, FO = EPI ? T32 / 2 : T32, T32_STAGES = Tile32<ALONE>::STAGES, ROWS = 8 * RT;
  extern __shared__ __align__(16) float s32_smem[];
  const int slice = threadIdx.x / T32_LANES, t = threadIdx.x % T32_LANES, to = t % T32_TO, tn = t / T32_TO;
  float* buf = s32_smem + (size_t)slice * Tile32<ALONE>::SLICE;
  uint32_t rank = 0;
  if (!ALONE) asm volatile("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(rank));
  const int o0 = (ALONE ? blockIdx.x : blockIdx.x >> 1) * FO, n0 = blockIdx.y * ROWS;
  const int gl = s32_group(k_dim), per = ALONE ? 2 : 1;           // groups of a slice
  const int kbeg = min(k_dim, ((int)rank * T32_SLICES + slice) * per * gl), kend = min(k_dim, kbeg + per * gl);
  const int steps = (kend - kbeg + S32_BK - 1) / S32_BK;
  auto load_w = [&](int st) {
    float* dst = buf + (st % T32_STAGES) * T32_STAGE + T32 * T32_PITCH;
#pragma unroll
    for (int i = t; i < T32 * PER; i += T32_LANES) {
      const int r = i / PER, k = kbeg + st * S32_BK + (i % PER) * STEP;
      const int o = o0 + (EPI ? r % FO : r);
      const bool in = o < o_out && k < kend;
      const size_t row = EPI && r >= FO ? (size_t)o_out + o : o;
      s32_copy<VEC>(dst + r * T32_PITCH + (i % PER) * STEP, in ? w + row * k_dim + k : w, in);
    }
  };
  auto load_x = [&](int st) {
    float* dst = buf + (st % T32_STAGES) * T32_STAGE;
#pragma unroll
    for (int i = t; i < ROWS * PER; i += T32_LANES) {
      const int r = i / PER, k = kbeg + st * S32_BK + (i % PER) * STEP;
      const bool in = n0 + r < n_rows && k < kend;
      s32_copy<VEC>(dst + r * T32_PITCH + (i % PER) * STEP, in ? x + (size_t)(n0 + r) * k_dim + k : x, in);
    }
  };
  auto slice_sync = [&]() { asm volatile("bar.sync %0, %1;\n" ::"r"(slice + 1), "n"(T32_LANES) : "memory"); };
#pragma unroll 1
  for (int st = 0; st < T32_STAGES - 1; ++st)
    if (st < steps) load_w(st);
  ifb_pdl_wait();
  ifb_pdl_trigger();
#pragma unroll 1
  for (int st = 0; st < T32_STAGES - 1; ++st) {
    if (st < steps) load_x(st);
    s32_commit();
  }
  unsigned long long acc[RT][T32_J];                                   // sums over even and over odd k
#pragma unroll
  for (int i = 0; i < RT; ++i)
#pragma unroll
    for (int j = 0; j < T32_J; ++j) acc[i][j] = 0;
  auto keep = [&](float* tile) {                                  // a group's sums, and from zero again
#pragma unroll
    for (int i = 0; i < RT; ++i)
#pragma unroll
      for (int j = 0; j < T32_J; ++j) {
        tile[(tn + 8 * i) * T32_RED + to + T32_TO * j] = s32_pair_sum(acc[i][j]);
        acc[i][j] = 0;
      }
  };
#pragma unroll 1
  for (int st = 0; st < steps; ++st) {
    s32_wait<T32_STAGES - 2>();
    slice_sync();                                                 // and the stage before this one may be filled again
    if (st + T32_STAGES - 1 < steps) { load_w(st + T32_STAGES - 1); load_x(st + T32_STAGES - 1); }
    s32_commit();
    const float* xs = buf + (st % T32_STAGES) * T32_STAGE + tn * T32_PITCH;
    const float* ws = buf + (st % T32_STAGES) * T32_STAGE + (T32 + to) * T32_PITCH;
#pragma unroll
    for (int k = 0; k < S32_BK; k += 4) {
      ulonglong2 wv[T32_J];
#pragma unroll
      for (int j = 0; j < T32_J; ++j) wv[j] = *reinterpret_cast<const ulonglong2*>(ws + T32_TO * j * T32_PITCH + k);
#pragma unroll
      for (int i = 0; i < RT; ++i) {
        const ulonglong2 xv = *reinterpret_cast<const ulonglong2*>(xs + 8 * i * T32_PITCH + k);
#pragma unroll
        for (int j = 0; j < T32_J; ++j) s32_fma2(acc[i][j], xv.x, wv[j].x);
#pragma unroll
        for (int j = 0; j < T32_J; ++j) s32_fma2(acc[i][j], xv.y, wv[j].y);
      }
    }
    if (ALONE && (st + 1) * S32_BK == gl) keep(buf + Tile32<ALONE>::RING);       // the first group is complete
  }
  s32_wait<0>();
  slice_sync();                                                   // no copy into the slice's stages is left, none is read
  if (ALONE && steps * S32_BK < gl) keep(buf + Tile32<ALONE>::RING);             // it was the last, and cut short
  keep(buf);
  if constexpr (ALONE) {
    __syncthreads();
    // the first groups of the slices, then the second ones
    auto total = [&](int r, int c) {
      float p[S32_GROUPS];
#pragma unroll
      for (int g = 0; g < S32_GROUPS; ++g) p[g] = s32_smem[(g / 2) * Tile32<ALONE>::SLICE + (g % 2 ? 0 : Tile32<ALONE>::RING) + r * T32_RED + c];
      return s32_total(p);
    };
#pragma unroll 2
    for (int i = threadIdx.x; i < ROWS * FO; i += T32_SLICES * T32_LANES) {
      const int r = i / FO, c = i % FO, o = o0 + c, n = n0 + r;
      if (n >= n_rows || o >= o_out) continue;
      float y = total(r, c);
      if (EPI) y = ifb_gate_act(y, unary) * total(r, FO + c);
      else {
        if (bias) y += bias[o];
        if (unary) y = ifb_unary(y, unary);
      }
      out[(size_t)n * o_out + o] = from_f32<TO>(y);
    }
    return;
  }
  asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
  // the tiles of groups 0-3 lie in CTA 0, those of 4-7 in CTA 1; this CTA adds the rows [32 * rank, 32 * rank + 32)
  uint32_t base[2];
  const uint32_t local = (uint32_t)__cvta_generic_to_shared(s32_smem);
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;\n" : "=r"(base[0]) : "r"(local));
  asm volatile("mapa.shared::cluster.u32 %0, %1, 1;\n" : "=r"(base[1]) : "r"(local));
  auto total = [&](int r, int c) {
    float p[S32_GROUPS];
#pragma unroll
    for (int g = 0; g < S32_GROUPS; ++g) {
      const uint32_t a = base[g / T32_SLICES] + (uint32_t)(((g % T32_SLICES) * Tile32<ALONE>::SLICE + r * T32_RED + c) * 4);
      asm volatile("ld.shared::cluster.f32 %0, [%1];\n" : "=f"(p[g]) : "r"(a) : "memory");
    }
    return s32_total(p);
  };
#pragma unroll 2
  for (int i = threadIdx.x; i < (ROWS / 2) * FO; i += T32_SLICES * T32_LANES) {
    const int r = (int)rank * (ROWS / 2) + i / FO, c = i % FO, o = o0 + c, n = n0 + r;
    if (n >= n_rows || o >= o_out) continue;
    float y = total(r, c);
    if (EPI) y = ifb_gate_act(y, unary) * total(r, FO + c);
    else {
      if (bias) y += bias[o];
      if (unary) y = ifb_unary(y, unary);
    }
    out[(size_t)n * o_out + o] = from_f32<TO>(y);
  }
  asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");      // nobody leaves while its tiles are being read
  asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}

template <int F, int RB, int EPI, bool VEC, typename TO>
static int rows32_launch(const float* x, const float* w, TO* out, int n, int o, int k, int unary, const float* bias, cudaStream_t s) {
  constexpr size_t smem = Rows32<F, RB>::SMEM;
  IFB_ALLOW_SMEM((rows32_kernel<F, RB, EPI, VEC, TO>), smem);
  const int fo = EPI ? F / 2 : F;
  return ifb_launch(rows32_kernel<F, RB, EPI, VEC, TO>, dim3((o + fo - 1) / fo, (n + RB - 1) / RB), dim3(256), smem, s, x, w, out, n, o, k,
                    unary, bias);
}

template <int EPI, bool VEC, bool ALONE, int RT, typename TO>
static int tile32_launch_as(const float* x, const float* w, TO* out, int n, int o, int k, int unary, const float* bias, cudaStream_t s) {
  constexpr size_t smem = Tile32<ALONE>::SMEM;
  constexpr int fo = EPI ? T32 / 2 : T32;
  IFB_ALLOW_SMEM((tile32_kernel<EPI, VEC, ALONE, RT, TO>), smem);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((ALONE ? 1 : 2) * ((o + fo - 1) / fo), (n + 8 * RT - 1) / (8 * RT));
  cfg.blockDim = dim3(T32_SLICES * T32_LANES);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = ifb_pdl_enabled() ? 1 : 0;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = 2;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = ALONE ? 1 : 2;
  cudaError_t e = cudaLaunchKernelEx(&cfg, tile32_kernel<EPI, VEC, ALONE, RT, TO>, x, w, out, n, o, k, unary, bias);
  if (e != cudaSuccess) { cudaGetLastError(); return -(int)e; }
  return IFB_OK;
}

// Rows per thread (a tile has eight times as many) and whether a CTA takes a tile alone: the form whose waves should take least
// time, a wave taking so many tenths of a microsecond and so many more for each 1,024 of k: what two CTAs share of a tile, filling the rings and
// the sum at the end, is most of a short k and little of a long one.  Over 66 products of 17 to 2,048 rows at each k of 256 to 4,096 within 0.2 % of the best
// form on average (0.6 to 2.5 % by the times of a k of 1,024 alone, which gave 300 rows of 2,500 x 4,096 203 us, now 182).  17 rows 18.8
// to 11.5 us for 4,096 x 1,024 and 31.9 to 16.4 for 1,024 x 2,048 against tiles of 64 rows by pairs, 193 rows 72 to 59 and 33.5 to 31.3.  The sums
// are the same in every form.  least: the fewest rows per thread that are compiled; vec: rows at 16 bytes.
static void tile32_form(int n, int k, int tiles, int sms, bool vec, int least, int* rows, bool* alone) {
  struct Wave { int begin, per_k; };                             // (six rows alone never take less than seven)
  static const Wave waves[2][9] = {{{0, 0}, {0, 0}, {30, 59}, {34, 74}, {35, 81}, {41, 100}, {40, 118}, {48, 127}, {47, 142}},
                                   {{0, 0}, {0, 0}, {26, 113}, {24, 166}, {27, 184}, {33, 205}, {0, 0}, {42, 252}, {49, 266}}};
  static const Wave scalar[2] = {{56, 222}, {44, 462}};
  long long best = 0;
  for (int rt = 8; rt >= least; --rt) {
    const long long all = (long long)tiles * ((n + 8 * rt - 1) / (8 * rt));
    for (int a = 0; a < 2; ++a) {
      const Wave w = vec ? waves[a][rt] : scalar[a];
      if (!w.per_k) continue;
      const int slots = a ? sms : sms / 2 > 1 ? sms / 2 : 1;
      const long long time = (all + slots - 1) / slots * (w.begin * 1024LL + (long long)w.per_k * k);
      if (!best || time < best) { best = time; *rows = rt; *alone = a; }
    }
  }
}
// Rows not at 16 bytes and bfloat16 outputs are rare: eight rows per thread.  So are more tiles of 16 rows than a grid holds.
static int tile32_least(int n, bool vec, size_t out_size) { return vec && out_size == 4 && n <= 65535 * 16 ? 2 : 8; }
template <int EPI, bool VEC, typename TO>
static int tile32_launch(const float* x, const float* w, TO* out, int n, int o, int k, int unary, const float* bias, cudaStream_t s) {
  const int fo = EPI ? T32 / 2 : T32;
  int rows = 8;
  bool alone = false;
  tile32_form(n, k, (o + fo - 1) / fo, ifb_sm_count(), VEC, tile32_least(n, VEC, sizeof(TO)), &rows, &alone);
#define IFB_T32(RT) \
  case RT: return alone ? tile32_launch_as<EPI, VEC, true, RT, TO>(x, w, out, n, o, k, unary, bias, s) \
                        : tile32_launch_as<EPI, VEC, false, RT, TO>(x, w, out, n, o, k, unary, bias, s);
  if constexpr (VEC && sizeof(TO) == 4)
    switch (rows) {
      IFB_T32(2) IFB_T32(3) IFB_T32(4) IFB_T32(5) IFB_T32(7)
      case 6: return tile32_launch_as<EPI, VEC, false, 6, TO>(x, w, out, n, o, k, unary, bias, s);      // alone, seven take less
    }
  switch (rows) { IFB_T32(8) }
#undef IFB_T32
  return IFB_ERR_ARG;
}
// The form of a product of more than S32_FEW_ROWS rows, for tests: twice the rows per thread, and 1 more where a CTA takes a tile alone.
// vec: rows at 16 bytes; sms: of the device.
IFB_EXPORT int ifb_linear_float32_form(int n_rows, int out_features, int k_dim, int epilogue, int vec, int out_dtype, int sms) {
  const int fo = (epilogue & 15) ? T32 / 2 : T32;
  int rows = 0;
  bool alone = false;
  tile32_form(n_rows, k_dim, (out_features + fo - 1) / fo, sms, vec != 0, tile32_least(n_rows, vec != 0, out_dtype == IFB_F32 ? 4 : 2), &rows, &alone);
  return 2 * rows + alone;
}

// Float32 operands.  Up to S32_FEW_ROWS rows the weights are streamed once per eight rows (from the second time on out of
// L2); beyond, tiles are the cheaper ones (4,096 x 1,024: 8 rows 9.6 us, 32 rows as four times eight 26 us, as a tile 12.8).
constexpr int S32_FEW_ROWS = 16;
template <int EPI, bool VEC, typename TO>
static int launch32_vec(const float* x, const float* w, TO* out, int n, int o, int k, int unary, const float* bias, cudaStream_t s) {
  if (n > S32_FEW_ROWS) return tile32_launch<EPI, VEC, TO>(x, w, out, n, o, k, unary, bias, s);
  const bool many = o >= 16384;                    // enough CTAs of 32 rows of w to fill the device several times
  if (n == 1) return many ? rows32_launch<32, 1, EPI, VEC, TO>(x, w, out, n, o, k, unary, bias, s)
                          : rows32_launch<8, 1, EPI, VEC, TO>(x, w, out, n, o, k, unary, bias, s);
  if (n <= 4) return many ? rows32_launch<32, 4, EPI, VEC, TO>(x, w, out, n, o, k, unary, bias, s)
                          : rows32_launch<8, 4, EPI, VEC, TO>(x, w, out, n, o, k, unary, bias, s);
  return many ? rows32_launch<32, 8, EPI, VEC, TO>(x, w, out, n, o, k, unary, bias, s)
              : rows32_launch<8, 8, EPI, VEC, TO>(x, w, out, n, o, k, unary, bias, s);
}

template <typename TO>
static int launch32(const void* x, const void* w, void* out, int n, int o, int k, int epi, const float* bias, cudaStream_t s) {
  const bool vec = k % 4 == 0 && !((uintptr_t)x & 15) && !((uintptr_t)w & 15);
  const float *xf = (const float*)x, *wf = (const float*)w;
  const int unary = epi >> 4;
  if ((epi & 15) == 0)
    return vec ? launch32_vec<0, true, TO>(xf, wf, (TO*)out, n, o, k, unary, bias, s)
               : launch32_vec<0, false, TO>(xf, wf, (TO*)out, n, o, k, unary, bias, s);
  return vec ? launch32_vec<1, true, TO>(xf, wf, (TO*)out, n, o, k, unary, nullptr, s)
             : launch32_vec<1, false, TO>(xf, wf, (TO*)out, n, o, k, unary, nullptr, s);
}

// EPI 0: out = unary(y + bias) (common.cuh: ifb_unary; 0 = y itself; bias null: none).  EPI 1 (silu_gate): w has 2*o_out rows, gate rows first;
// out[n, o] = act(y[n, o]) * y[n, o_out + o] with act = silu or the unary function.
template <typename TX, typename TW, typename TO, int EPI>
__global__ void __launch_bounds__(256)
linear_simt_kernel(const TX* __restrict__ x, const TW* __restrict__ w, TO* __restrict__ out, int n_rows, int o_out,
                   int k_dim, int unary, const float* __restrict__ bias) {
  __shared__ float xs[TILE_K][TILE_N + 1];
  __shared__ float ws[EPI ? 2 : 1][TILE_K][TILE_O + 1];
  ifb_pdl_wait();
  ifb_pdl_trigger();
  const int tid = threadIdx.x;
  const int tn = tid / 16, to = tid % 16;          // thread's 4x4 patch: rows tn*4.., columns to*4..
  const int n0 = blockIdx.y * TILE_N, o0 = blockIdx.x * TILE_O;
  float acc[EPI ? 2 : 1][4][4];
#pragma unroll
  for (int e = 0; e < (EPI ? 2 : 1); ++e)
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[e][i][j] = 0.f;

  for (int k0 = 0; k0 < k_dim; k0 += TILE_K) {
    // 64 rows x 16 k = 1024 elements per operand tile, 4 per thread
#pragma unroll
    for (int it = 0; it < 4; ++it) {
      const int idx = tid + it * 256;
      const int r = idx / TILE_K, kk = idx % TILE_K;
      const int k = k0 + kk;
      float xv = 0.f;
      if (n0 + r < n_rows && k < k_dim) xv = to_f32<TX>(x[(size_t)(n0 + r) * k_dim + k]);
      xs[kk][r] = xv;
#pragma unroll
      for (int e = 0; e < (EPI ? 2 : 1); ++e) {
        float wv = 0.f;
        if (o0 + r < o_out && k < k_dim) wv = to_f32<TW>(w[((size_t)e * o_out + o0 + r) * k_dim + k]);
        ws[e][kk][r] = wv;
      }
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < TILE_K; ++kk) {
      float xv[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) xv[i] = xs[kk][tn * 4 + i];
#pragma unroll
      for (int e = 0; e < (EPI ? 2 : 1); ++e) {
        float wv[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) wv[j] = ws[e][kk][to * 4 + j];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[e][i][j] = fmaf(xv[i], wv[j], acc[e][i][j]);
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int n = n0 + tn * 4 + i;
    if (n >= n_rows) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int o = o0 + to * 4 + j;
      if (o >= o_out) continue;
      float y = acc[0][i][j];
      if (EPI) y = ifb_gate_act(y, unary) * acc[EPI ? 1 : 0][i][j];
      else {
        if (bias) y += bias[o];
        if (unary) y = ifb_unary(y, unary);
      }
      out[(size_t)n * o_out + o] = from_f32<TO>(y);
    }
  }
}

template <typename TX, typename TW, typename TO>
static int launch(const void* x, const void* w, void* out, int n, int o, int k, int epi, const float* bias, cudaStream_t s) {
  dim3 grid((o + TILE_O - 1) / TILE_O, (n + TILE_N - 1) / TILE_N);
  const int unary = epi >> 4;
  if ((epi & 15) == 0)
    return ifb_launch(linear_simt_kernel<TX, TW, TO, 0>, grid, dim3(256), 0, s, (const TX*)x, (const TW*)w, (TO*)out, n, o, k, unary, bias);
  return ifb_launch(linear_simt_kernel<TX, TW, TO, 1>, grid, dim3(256), 0, s, (const TX*)x, (const TW*)w, (TO*)out, n, o, k, unary, (const float*)nullptr);
}

// out_features is the width of `out` (for the silu_gate epilogue, half of w's rows).  epilogue: 0 plain, 1 silu_gate,
// 16 * u: plain with the unary function u of common.cuh applied to every element, 1 + 16 * u: gated with u in silu's place.  bias (plain epilogue; may be null):
// float32 [out_features], added before the unary function.
IFB_EXPORT int ifb_linear_simt(const void* x, int x_dtype, const void* w, int w_dtype, void* out, int out_dtype,
                               int n_rows, int out_features, int k_dim, int epilogue, const float* bias, cudaStream_t stream) {
  if (n_rows <= 0 || out_features <= 0) return IFB_OK;
  if (k_dim < 1) return IFB_ERR_SIZE;
  if ((epilogue & 15) > 1 || (epilogue >> 4) > IFB_UNARY_LAST || epilogue < 0 ||
      (bias && (epilogue & 15)))
    return IFB_ERR_ARG;
  if ((n_rows + TILE_N - 1) / TILE_N > 65535) return IFB_ERR_SIZE;
  typedef __nv_bfloat16 bf;
  const int key = x_dtype * 4 + w_dtype * 2 + out_dtype;
  switch (key) {
    case 0: return launch32<float>(x, w, out, n_rows, out_features, k_dim, epilogue, bias, stream);
    case 1: return launch32<bf>(x, w, out, n_rows, out_features, k_dim, epilogue, bias, stream);
    case 2: return launch<float, bf, float>(x, w, out, n_rows, out_features, k_dim, epilogue, bias, stream);
    case 3: return launch<float, bf, bf>(x, w, out, n_rows, out_features, k_dim, epilogue, bias, stream);
    case 4: return launch<bf, float, float>(x, w, out, n_rows, out_features, k_dim, epilogue, bias, stream);
    case 5: return launch<bf, float, bf>(x, w, out, n_rows, out_features, k_dim, epilogue, bias, stream);
    case 6: return launch<bf, bf, float>(x, w, out, n_rows, out_features, k_dim, epilogue, bias, stream);
    case 7: return launch<bf, bf, bf>(x, w, out, n_rows, out_features, k_dim, epilogue, bias, stream);
  }
  return IFB_ERR_DTYPE;
}
