// y = x W^T for a handful of rows (decode batches, short prompts, verification), with W in 4-bit, 8-bit (MLX affine,
// group 64) or bf16, plain or grouped by expert, with SwiGLU, residual, fp32 output and the RMSNorm of x as options.
//
// What bounds it: the weights are read once, so at these sizes the time is the weights' trip from HBM, provided that
// enough of it is under way (about 50 KB per SM) and that turning codes into operands costs few enough issue slots. The
// 128-row tensor-core tile of xgemm_kernel.cuh keeps 16 KB of 4-bit weights in flight per SM and writes every expanded
// weight to shared memory; the per-row kernels unpack once per row of x. Here
//   * every warp streams rows of W through a private ring of cp.async stages (16 warps x 2 to 4 KB in flight), so there is no barrier
//     in the weight path and no producer to wait for;
//   * the rows of W are the M of mma.sync m16n8k16 and the rows of x its N: eight rows of x cost one instruction, and a
//     code becomes an operand in registers with 5 logic operations per 8 weights: a 4-bit or 8-bit code in the low bits of
//     an fp16 is the subnormal q x 2^-24, exactly (the nibble four bits up is 16 q, against x / 16);
//   * scale and bias are applied to the fp32 sums, once per group of 64: sum_k w x = s sum_k q x + b sum_k x, so weights
//     are never rounded;
//   * x is staged in shared memory in the order in which the fragments read it, as fp16 with one power of two per (row,
//     group) chosen from the group's maximum (exact for bf16 inputs), with the group's sum beside it. bf16 weights take x
//     as bf16, and x times a norm's weight (16 significant bits) as two bf16 terms, in two tiles that share the weights, and are
//     summed 64 of K at a time in the tensor cores, which cut what they add, and from there in fp32 (error of the fp32 result
//     at K = 14336 1.4e-7 of it, 2.0e-6 as one sum in the tensor cores; 28672 x 4096 at 8 rows 45.4 -> 44.9 us, with a norm
//     49.0 -> 50.2; adding the second terms up in the tensor cores: 50.9);
//   * a norm's 1 / rms multiplies the sums.
// Two kernels. Quantised weights run on narrow_even_kernel (further down), which splits a block's work over its warps by ring stages;
// narrow_gemm_kernel is for bf16 weights, four tiles of rows, and rows of W that are longer than 32768.
//
// narrow_gemm_kernel. An item is RT row tiles (16 rows of W each) of one expert against up to 8 T rows of x; the warps of a block are
// RT tiles x KS shares of K, whose sums meet in shared memory. A block takes a contiguous run of items, so x is staged again
// only when the expert or the rows change, if K fits the buffer (64 / T groups), else slab by slab. RT and KS are chosen so
// that the blocks' runs are even. The quantised forms are held to 80 registers for 24 warps.
//
// Reference counterparts: affine_qmm / gather_qmm for small M (crates/rmlx-core/src/ops/quantized.rs:2755,9634).
#include "../common/ptx.cuh"
#include "../common/launch.cuh"
#include "../common/gated.cuh"

namespace rb {

constexpr int kNwMaxExperts = 256;
constexpr int kNwUnits = 64;          // (tile of eight rows of x, group of 64) pieces of the x buffer: 1 KB each
constexpr int kNwKinds = 3;           // weight kinds: 0 bf16, 1 4-bit, 2 8-bit
constexpr int kNwCB = 128;            // bytes of a row of W per ring stage

template <int KIND, int T>
struct NwShape {
  // bf16 weights cost few instructions and three times the bytes: fewer warps, a deeper ring
  static constexpr int W = KIND ? 24 : 16, THREADS = W * 32, D = KIND ? 2 : 4;
  static constexpr int G = KIND == 1 ? 4 : KIND == 2 ? 2 : 1;    // groups of 64 weights per stage
  static constexpr int SLG = kNwUnits / T;                       // groups of K in the x buffer
  static constexpr int STAGE = 16 * kNwCB + (KIND ? 512 : 0);    // rows; then scales and biases, 16 bytes each per row
  static constexpr int RING = W * D * STAGE;
  static constexpr int X = kNwUnits * 1024;
  static constexpr int XS = KIND ? kNwUnits * 96 : 0;            // per row and group: scale; sum in two terms
  static constexpr bool kRedInX = T >= 4;                        // the shares' sums meet in the x buffer
  static constexpr int RED = kRedInX ? 0 : W * 512 * T;
  static constexpr int HEAD = (kNwMaxExperts + 2) * 8 + kNwUnits * 32 + 64;
  static constexpr int BYTES = RING + X + XS + RED + HEAD;
  static constexpr int KSMAX = SLG / G < 8 ? SLG / G : 8;        // shares of K: at least one stage per slab each
};

struct NwParams {
  const uint8_t* w;
  const __nv_bfloat16 *scales, *biases;
  const __nv_bfloat16* x;
  const int* order;          // position -> output row; null: the position itself
  const int* offsets;        // [E + 1] positions of every expert; null: all M rows, one expert
  const __nv_bfloat16 *norm, *residual;
  void* out;
  float eps;
  int x_stride, x_div;       // x row = output row / x_div
  int out_stride, out_f32, res_stride;
  int E, M, N, K, swiglu, RT, KS;
  int split;                 // bf16 weights and a norm: x times its weight goes in two terms, in two tiles of rows
};
// What the even split needs beside it. In a structure of its own: the other kernel keeps the registers that it has without these
// fields (bf16, one tile of rows, 92; with them 89, and 0.3 to 0.6 us more a launch: 1024 x 4096 at 5 rows 7.9 / 8.5, 6144 x 3072 at 24 18.9 / 19.8).
struct NeParams : NwParams {
  int CS, cs_log2, RL, xunits;   // blocks of a cluster that share K; tiles per run; units of x
  const int* choice;         // row i of E = M rows meets expert choice[i] (none outside [0, experts)); null: by offsets
  int experts;
};

__device__ __forceinline__ void nw_cp16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void nw_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void nw_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void nw_prefetch(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

__device__ __forceinline__ uint4 nw_lds128(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ uint2 nw_lds64(uint32_t a) {
  uint2 v;
  asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ uint32_t nw_lds32(uint32_t a) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
  return v;
}

template <bool F16>
__device__ __forceinline__ void nw_mma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                       uint32_t b1) {
  if constexpr (F16)
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
        "{%0, %1, %2, %3};" : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  else
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
        "{%0, %1, %2, %3};" : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// The first product of a sum: nothing to add to.
template <bool F16>
__device__ __forceinline__ void nw_mma0(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                        uint32_t b1) {
  if constexpr (F16)
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
  else
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}
__device__ __forceinline__ void nw_mma_tf32(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                            uint32_t b1) {
  asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ __forceinline__ uint64_t nw_pair(uint32_t lo, uint32_t hi) {
  uint64_t v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "r"(lo), "r"(hi));
  return v;
}
__device__ __forceinline__ void nw_unpair(uint64_t v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t nw_fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t v;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(v) : "l"(a), "l"(b), "l"(c));
  return v;
}
__device__ __forceinline__ uint64_t nw_mul2(uint64_t a, uint64_t b) {
  uint64_t v;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(a), "l"(b));
  return v;
}

__device__ __forceinline__ uint64_t nw_add2(uint64_t a, uint64_t b) {
  uint64_t v;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(a), "l"(b));
  return v;
}

// 16 values of a (row, group of 64), a quarter of the group per lane, as the operand words o that the products take: fp16 with one
// power of two for the group (down undoes it), chosen from its largest magnitude. sum: the group's sum of x times 2^-24. Codes enter
// the products as q x 2^-24: the sums are kept at that size and multiplied once, at the end.
template <int KIND>
__device__ __forceinline__ void nw_group_fp16(float (&f)[16], bool rounded, uint32_t (&o)[8], float& down, float& sum) {
  float m = 0.f;
  sum = 0.f;
#pragma unroll
  for (int i = 0; i < 16; ++i) { m = fmaxf(m, fabsf(f[i])); sum += f[i]; }
  m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 1));
  m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 2));
  // the group's largest magnitude goes to [2^14, 2^15): nothing overflows, and what fp16 loses is 2^-39 of it. The
  // exponents are held to where scale, inverse and the products with the weights' scales stay normal numbers.
  const uint32_t ex = min(max(__float_as_uint(m) >> 23, 60u), 230u);
  const float up = __uint_as_float((268u - ex) << 23);
  down = __uint_as_float((ex - 14u) << 23);
#pragma unroll
  for (int i = 0; i < 16; ++i) f[i] *= up;
  if (KIND == 1) {
    // word h of the lane holds nibbles 0..7: operand pairs (0, 4) (1, 5) (2, 6) (3, 7), odd ones 16 times too large
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float k = (i & 1) ? 0.0625f : 1.f;
        const __half2 v2 = __floats2half2_rn(f[8 * h + i] * k, f[8 * h + i + 4] * k);
        o[4 * h + i] = *reinterpret_cast<const uint32_t*>(&v2);
      }
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const __half2 v2 = __floats2half2_rn(f[2 * i], f[2 * i + 1]);
      o[i] = *reinterpret_cast<const uint32_t*>(&v2);
    }
  }
  if (rounded) {     // rounded to fp16: scale and bias have to see the same values, or a code's mean amplifies the rounding
    sum = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float2 v2 = __half22float2(*reinterpret_cast<const __half2*>(&o[i]));
      sum = fmaf(v2.x + v2.y, (KIND == 1 && (i & 1)) ? 16.f : 1.f, sum);
    }
    sum *= down;
  }
  sum += __shfl_xor_sync(0xffffffffu, sum, 1);
  sum += __shfl_xor_sync(0xffffffffu, sum, 2);
  sum *= 5.9604644775390625e-8f;
}

template <int KIND, int T>
__global__ void __launch_bounds__(NwShape<KIND, T>::THREADS, 1) narrow_gemm_kernel(const NwParams p) {
  using S = NwShape<KIND, T>;
  extern __shared__ __align__(128) char smem[];
  const uint32_t ring = smem_u32(smem), xbuf = ring + S::RING, xs = xbuf + S::X, xt = xs + kNwUnits * 32;
  float* red = reinterpret_cast<float*>(smem + S::RING + (S::kRedInX ? 0 : S::X + S::XS));
  int* s_off = reinterpret_cast<int*>(smem + S::RING + S::X + S::XS + S::RED);
  int* s_pre = s_off + kNwMaxExperts + 1;                // items before every expert
  float* s_ss = reinterpret_cast<float*>(s_pre + kNwMaxExperts + 3);   // [unit][8] sums of squares of what was staged there

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int rt = warp / p.KS, ks = warp % p.KS;
  const int rows = p.split ? 4 * T : 8 * T;              // rows of x per pass
  const int tiles = p.N / 16, blocks_n = (tiles + p.RT - 1) / p.RT;
  const int groups = p.K / 64, chunks = groups / S::G;
  const bool works = rt < p.RT && ks < chunks;           // the block may have warps to spare: they help to stage x
  const size_t row_bytes = size_t(p.K) * (KIND == 1 ? 1 : KIND == 2 ? 2 : 4) / 2;
  pdl_launch_dependents();

  if (p.offsets) {
    pdl_wait();
    for (int i = threadIdx.x; i <= p.E; i += S::THREADS) {
      const int o = p.offsets[i];
      s_off[i] = RB_BOUNDS(o, p.M + 1) ? o : 0;
    }
    __syncthreads();
    if (warp == 0) {       // items before every expert: a scan over 32 experts at a time
      int base = 0;
      for (int e0 = 0; e0 < p.E; e0 += 32) {
        const int e = e0 + lane;
        const int n = e < p.E ? s_off[e + 1] - s_off[e] : 0;
        const int mine = RB_BOUNDS(n, p.M + 1) ? (n + rows - 1) / rows * blocks_n : 0;
        int sum = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { const int v = __shfl_up_sync(0xffffffffu, sum, o); if (lane >= o) sum += v; }
        if (e < p.E) s_pre[e] = base + sum - mine;
        base += __shfl_sync(0xffffffffu, sum, 31);
      }
      if (lane == 0) s_pre[p.E] = base;
    }
  } else if (threadIdx.x == 0) {
    s_off[0] = 0; s_off[1] = p.M; s_pre[0] = 0; s_pre[1] = (p.M + rows - 1) / rows * blocks_n;
  }
  __syncthreads();
  const int total = s_pre[p.E];
  const int item0 = int((long long)blockIdx.x * total / gridDim.x), item1 = int((long long)(blockIdx.x + 1) * total / gridDim.x);
  if (item0 >= item1) return;

  // item -> (tile of rows of x, row block of W) and its expert; the rows of x vary fastest inside a row block, so that W is
  // found in L2 again
  auto locate = [&](int item, int& e) {
    while (s_pre[e + 1] <= item) ++e;
    const int mt = (s_off[e + 1] - s_off[e] + rows - 1) / rows, local = item - s_pre[e];
    return make_int2(local % mt, local / mt);
  };

  // ---------------------------------------------------------------- weight ring (one per warp)
  const uint32_t my_ring = ring + warp * (S::D * S::STAGE);
  // rows 8.. of a tile are `half` rows of W further (SwiGLU: the up rows)
  const int half = p.swiglu ? p.N / 2 : 8, per = p.swiglu ? 8 : 16;
  int p_item = works ? item0 : item1, p_e = 0, p_chunk = ks, p_stage = 0;
  const uint8_t* p_w = nullptr;                          // this lane's 16 bytes of row lane / 8 at chunk 0
  const uint8_t* p_s = nullptr;                          // lanes 0-15 the scales, 16-31 the biases, of row lane % 16
  auto p_locate = [&]() {                                // skips items in which this warp's tile does not exist
    while (p_item < item1) {
      const int tile = locate(p_item, p_e).y * p.RT + rt;
      if (tile < tiles) {
        // the first two lines of the rows of the next row block, whose stages are asked for only when this item's have run
        // (a row may have fewer)
        if (const int c = ks + (lane >> 4) * p.KS; tile + p.RT < tiles && c < chunks) {
          const size_t at = (size_t(p_e) * p.N + (tile + p.RT) * per + (lane & 7) + ((lane >> 3) & 1) * half) * row_bytes + c * kNwCB;
          if (RB_BOUNDS(at, size_t(p.E) * p.N * row_bytes)) nw_prefetch(p.w + at);
        }
        const size_t row = size_t(p_e) * p.N + tile * per;
        p_w = p.w + (row + (lane >> 3)) * row_bytes + (lane & 7) * 16;
        if (KIND)
          p_s = reinterpret_cast<const uint8_t*>((lane < 16 ? p.scales : p.biases) + (row + (lane & 7) + ((lane >> 3) & 1) * half) * groups);
        return;
      }
      ++p_item;
    }
  };
  p_locate();
  // where this lane's 16 bytes of row lane / 8 go: 32-byte (4-bit) or 64-byte (8-bit) groups, or 16-byte pieces (bf16), moved
  // by an exclusive or with the row, so that the fragments' reads of eight rows hit all banks once
  const uint32_t my_dst = [&]() {
    const int r = lane >> 3, c16 = lane & 7;
    const int off = KIND == 1 ? (((c16 >> 1) ^ r) << 5) + (c16 & 1) * 16
                    : KIND == 2 ? (((c16 >> 2) ^ (r & 1)) << 6) + (c16 & 3) * 16 : (c16 ^ (r & 1)) * 16;
    return uint32_t(r * kNwCB + off);
  }();
  const size_t half_b = half * row_bytes;
  auto issue = [&]() {
    if (p_item < item1) {
      const uint32_t st = my_ring + p_stage * S::STAGE;
      const uint8_t* src = p_w + size_t(p_chunk) * kNwCB;
      nw_cp16(st + my_dst, src);
      nw_cp16(st + my_dst + 4 * kNwCB, src + 4 * row_bytes);
      nw_cp16(st + my_dst + 8 * kNwCB, src + half_b);
      nw_cp16(st + my_dst + 12 * kNwCB, src + half_b + 4 * row_bytes);
      if (KIND) nw_cp16(st + 16 * kNwCB + lane * 16, p_s + (p_chunk * S::G * 2 & ~15));
      // the line of each row that the stage after next takes
      if ((lane & 7) < 4 && p_chunk + 2 * p.KS < chunks)
        nw_prefetch(src - (lane & 7) * 16 + size_t(2 * p.KS) * kNwCB + (lane & 1) * (4 * row_bytes) + ((lane >> 1) & 1) * half_b);
      p_chunk += p.KS;
      if (p_chunk >= chunks) { p_chunk = ks; ++p_item; p_locate(); }
      if (++p_stage == S::D) p_stage = 0;
    }
    nw_commit();
  };
#pragma unroll
  for (int i = 0; i < S::D - 1; ++i) issue();
  if (!p.offsets) pdl_wait();

  // ---------------------------------------------------------------- x
  // output row of the item's i-th row of x, -1: none
  auto out_row = [&](int e, int mt, int i) {
    const int pos = s_off[e] + mt * rows + i;
    if (i >= rows || pos >= s_off[e + 1]) return -1;
    if (!p.order) return pos;
    const int row = __ldg(p.order + pos);
    return RB_BOUNDS(row, p.M) ? row : -1;
  };
  // unit u of the buffer: tile u / SLG of the rows of x (split: the second half of the tiles repeats the first half's rows),
  // group u % SLG of the slab. A lane holds the 16 values that its fragments need: row g, share t.
  auto stage = [&](int e, int mt, int slab) {
    const int n = min(S::SLG, groups - slab * S::SLG);
    for (int u = warp; u < kNwUnits; u += S::W) {
      const int gi = u % S::SLG, tile = u / S::SLG;
      if (gi >= n) {
        if (slab == 0 && p.norm && t == 0) s_ss[u * 8 + g] = 0.f;
        continue;
      }
      const int group = slab * S::SLG + gi;
      const bool second = T > 1 && p.split && tile >= T / 2;
      uint4 lo = make_uint4(0u, 0u, 0u, 0u), hi = lo;
      const int row = out_row(e, mt, (second ? tile - T / 2 : tile) * 8 + g);
      const int at = group * 64 + (KIND == 0 ? t * 8 : t * 16);
      if (row >= 0) {
        const __nv_bfloat16* src = p.x + size_t(p.x_div > 1 ? row / p.x_div : row) * p.x_stride + at;
        lo = *reinterpret_cast<const uint4*>(src);
        hi = *reinterpret_cast<const uint4*>(src + (KIND == 0 ? 32 : 8));
      }
      const uint32_t dst = xbuf + u * 1024 + g * 64 + t * 16;
      uint32_t o[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
      if (KIND != 0 || p.norm) {
        float f[16];
#pragma unroll
        for (int i = 0; i < 8; ++i) { f[2 * i] = bf16lo(o[i]); f[2 * i + 1] = bf16hi(o[i]); }
        if (p.norm) {
          float ss = 0.f;
#pragma unroll
          for (int i = 0; i < 16; ++i) ss = fmaf(f[i], f[i], ss);
          ss += __shfl_xor_sync(0xffffffffu, ss, 1);
          ss += __shfl_xor_sync(0xffffffffu, ss, 2);
          if (t == 0) s_ss[u * 8 + g] = slab ? s_ss[u * 8 + g] + ss : ss;
          const uint4 n0 = *reinterpret_cast<const uint4*>(p.norm + at);
          const uint4 n1 = *reinterpret_cast<const uint4*>(p.norm + at + (KIND == 0 ? 32 : 8));
          const uint32_t nws[8] = {n0.x, n0.y, n0.z, n0.w, n1.x, n1.y, n1.z, n1.w};
#pragma unroll
          for (int i = 0; i < 8; ++i) { f[2 * i] *= bf16lo(nws[i]); f[2 * i + 1] *= bf16hi(nws[i]); }
        }
        if (KIND == 0) {
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            o[i] = pack_bf16(f[2 * i], f[2 * i + 1]);
            if (second) o[i] = pack_bf16(f[2 * i] - bf16lo(o[i]), f[2 * i + 1] - bf16hi(o[i]));
          }
        } else {
          float down, sum;
          nw_group_fp16<KIND>(f, p.norm != nullptr, o, down, sum);
          if (t == 0) {
            // the sum of x goes in two tf32 terms (2^-22 of it together), multiplied with the biases, which are exact in tf32
            const uint32_t s_hi = __float_as_uint(sum) & 0xffffe000u;
            const uint32_t s_lo = __float_as_uint(sum - __uint_as_float(s_hi)) & 0xffffe000u;
            asm volatile("st.shared.f32 [%0], %1;" ::"r"(xs + u * 32 + g * 4), "f"(down) : "memory");
            asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(xt + u * 64 + g * 8), "r"(s_hi), "r"(s_lo) : "memory");
          }
        }
      }
      asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(dst), "r"(o[0]), "r"(o[1]), "r"(o[2]), "r"(o[3]) : "memory");
      asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(dst + 512), "r"(o[4]), "r"(o[5]), "r"(o[6]), "r"(o[7]) : "memory");
    }
  };

  // ---------------------------------------------------------------- products
  float acc[T][4] = {};
  int c_stage = 0;
  // rows g and g + 8 of a stage, this lane's share of a group (the swizzle is an exclusive or with the group's number)
  const uint32_t my_src = KIND == 1 ? g * kNwCB + t * 8 + ((g & 3) << 5) : KIND == 2 ? g * kNwCB + t * 16 + ((g & 1) << 6)
                          : g * kNwCB + ((t ^ (g & 1)) << 4);
  auto compute = [&](int chunk, int unit0) {             // one ring stage against groups unit0 .. of the x buffer
    nw_wait<S::D - 2>();
    __syncwarp();
    issue();                                             // refills the stage that the previous call read
    const uint32_t st = my_ring + c_stage * S::STAGE;
    if (++c_stage == S::D) c_stage = 0;
    const uint32_t wa = st + my_src, xa = xbuf + unit0 * 1024 + lane * 16, qa = xs + unit0 * 32 + t * 8;
    uint32_t sw[2][2];                                    // scales of rows g, g + 8: two groups per word
    if constexpr (KIND != 0) {
      const uint32_t sa = st + 16 * kNwCB + g * 16 + (KIND == 1 ? (chunk & 1) * 8 : (chunk & 3) * 4);
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        if constexpr (KIND == 1) {
          const uint2 v = nw_lds64(sa + r * 128); sw[r][0] = v.x; sw[r][1] = v.y;
        } else {
          sw[r][0] = nw_lds32(sa + r * 128);
        }
      }
      // biases x sums of x, all groups of the stage in one product: k is (group t, first term), (group t, second term)
      uint32_t b0 = 0u, b1 = 0u;
      if (KIND == 1 || t < S::G) {
        const uint32_t ba = sa + 256 + (t & (S::G - 1)) * 2;
        asm volatile("{.reg .u16 h; ld.shared.u16 h, [%1]; cvt.u32.u16 %0, h;}" : "=r"(b0) : "r"(ba) : "memory");
        asm volatile("{.reg .u16 h; ld.shared.u16 h, [%1]; cvt.u32.u16 %0, h;}" : "=r"(b1) : "r"(ba + 128) : "memory");
        b0 <<= 16; b1 <<= 16;
      }
      const uint32_t ta = xt + (unit0 + (t & (S::G - 1))) * 64 + g * 8;
#pragma unroll
      for (int n = 0; n < T; ++n) {
        const uint2 v = nw_lds64(ta + n * (S::SLG * 64));
        nw_mma_tf32(acc[n], b0, b1, b0, b1, v.x, v.y);
      }
    }
#pragma unroll
    for (int j = 0; j < S::G; ++j) {
      uint32_t a[2][8];                                   // [row g, g + 8][operand words of the four products]
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        if constexpr (KIND == 1) {
          const uint2 v = nw_lds64((wa ^ (j << 5)) + 8 * r * kNwCB);
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const uint32_t w = h ? v.y : v.x, w8 = w >> 8;
            a[r][4 * h + 0] = w & 0x000f000fu; a[r][4 * h + 1] = w & 0x00f000f0u;
            a[r][4 * h + 2] = w8 & 0x000f000fu; a[r][4 * h + 3] = w8 & 0x00f000f0u;
          }
        } else if constexpr (KIND == 2) {
          const uint4 v = nw_lds128((wa ^ (j << 6)) + 8 * r * kNwCB);
          const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            a[r][2 * i] = __byte_perm(w[i], 0u, 0x4140u);
            a[r][2 * i + 1] = __byte_perm(w[i], 0u, 0x4342u);
          }
        } else {
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const uint4 v = nw_lds128((wa ^ (h << 6)) + 8 * r * kNwCB);
            a[r][4 * h] = v.x; a[r][4 * h + 1] = v.y; a[r][4 * h + 2] = v.z; a[r][4 * h + 3] = v.w;
          }
        }
      }
      uint32_t sc[2] = {};                                // as bits
      if constexpr (KIND != 0) {
#pragma unroll
        for (int r = 0; r < 2; ++r) sc[r] = (j & 1) ? sw[r][j >> 1] & 0xffff0000u : sw[r][j >> 1] << 16;
      }
#pragma unroll
      for (int n = 0; n < T; ++n) {
        const uint32_t un = n * S::SLG + j;
        const uint4 x0 = nw_lds128(xa + un * 1024), x1 = nw_lds128(xa + un * 1024 + 512);
        if constexpr (KIND == 0) {
          float c[4];
          nw_mma0<false>(c, a[0][0], a[1][0], a[0][1], a[1][1], x0.x, x0.y);
          nw_mma<false>(c, a[0][2], a[1][2], a[0][3], a[1][3], x0.z, x0.w);
          nw_mma<false>(c, a[0][4], a[1][4], a[0][5], a[1][5], x1.x, x1.y);
          nw_mma<false>(c, a[0][6], a[1][6], a[0][7], a[1][7], x1.z, x1.w);
#pragma unroll
          for (int r = 0; r < 2; ++r)
            nw_unpair(nw_add2(nw_pair(__float_as_uint(acc[n][2 * r]), __float_as_uint(acc[n][2 * r + 1])),
                              nw_pair(__float_as_uint(c[2 * r]), __float_as_uint(c[2 * r + 1]))), acc[n][2 * r], acc[n][2 * r + 1]);
        } else {
          const uint2 xq = nw_lds64(qa + un * 32);        // scales of rows 2t and 2t + 1
          float c[4];
          nw_mma0<true>(c, a[0][0], a[1][0], a[0][1], a[1][1], x0.x, x0.y);
          nw_mma<true>(c, a[0][2], a[1][2], a[0][3], a[1][3], x0.z, x0.w);
          nw_mma<true>(c, a[0][4], a[1][4], a[0][5], a[1][5], x1.x, x1.y);
          nw_mma<true>(c, a[0][6], a[1][6], a[0][7], a[1][7], x1.z, x1.w);
          // two columns per instruction: (scale x scale of x) c + acc
          const uint64_t xsc = nw_pair(xq.x, xq.y);
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            uint64_t d = nw_pair(__float_as_uint(acc[n][2 * r]), __float_as_uint(acc[n][2 * r + 1]));
            d = nw_fma2(nw_mul2(nw_pair(sc[r], sc[r]), xsc),
                        nw_pair(__float_as_uint(c[2 * r]), __float_as_uint(c[2 * r + 1])), d);
            nw_unpair(d, acc[n][2 * r], acc[n][2 * r + 1]);
          }
        }
      }
    }
  };

  auto put = [&](int row, int col, float v) {
    if (row < 0) return;
    if (p.residual) v += __bfloat162float(p.residual[size_t(row) * p.res_stride + col]);
    if (p.out_f32) static_cast<float*>(p.out)[size_t(row) * p.out_stride + col] = v;
    else static_cast<__nv_bfloat16*>(p.out)[size_t(row) * p.out_stride + col] = __float2bfloat16_rn(v);
  };
  // 1 / rms of row i of tile n: its units' shares, in order
  auto rstd = [&](int n, int i) {
    float ss = 0.f;
    for (int u = n * S::SLG; u < (n + 1) * S::SLG; ++u) ss += s_ss[u * 8 + i];
    return rsqrtf(ss / float(p.K) + p.eps);
  };
  auto finish = [&](int tile, int e, int mt) {
    const bool mine = works && tile < tiles;
    if (p.KS > 1) {
      __syncthreads();                                    // the previous item's sums have been read, the x buffer is free
      if (ks > 0 && mine) {
#pragma unroll
        for (int i = 0; i < T * 4; ++i) red[(warp * (T * 4) + i) * 32 + lane] = (&acc[0][0])[i];
      }
      __syncthreads();
      if (ks == 0 && mine) {
        for (int o = 1; o < min(p.KS, chunks); ++o)
#pragma unroll
          for (int i = 0; i < T * 4; ++i) (&acc[0][0])[i] += red[((warp + o) * (T * 4) + i) * 32 + lane];
      }
    }
    if (ks == 0 && mine) {
#pragma unroll
      for (int n = 0; n < T; ++n) {
        if (KIND == 0 && p.split && n >= T / 2) break;
        float* d = acc[n];
        if (KIND == 0 && p.split) {
#pragma unroll
          for (int i = 0; i < 4; ++i) d[i] += acc[(n + T / 2) % T][i];
        }
        const int row0 = out_row(e, mt, n * 8 + 2 * t), row1 = out_row(e, mt, n * 8 + 2 * t + 1);
        float r0 = KIND ? 16777216.f : 1.f, r1 = r0;
        if (p.norm) { r0 *= rstd(n, 2 * t); r1 *= rstd(n, 2 * t + 1); }
        d[0] *= r0; d[1] *= r1; d[2] *= r0; d[3] *= r1;
        if (p.swiglu) {
          put(row0, tile * 8 + g, gated_act(d[0], d[2], 0.f));
          put(row1, tile * 8 + g, gated_act(d[1], d[3], 0.f));
        } else {
          put(row0, tile * 16 + g, d[0]);
          put(row1, tile * 16 + g, d[1]);
          put(row0, tile * 16 + g + 8, d[2]);
          put(row1, tile * 16 + g + 8, d[3]);
        }
      }
    }
#pragma unroll
    for (int i = 0; i < T * 4; ++i) (&acc[0][0])[i] = 0.f;
  };

  const int nslab = (groups + S::SLG - 1) / S::SLG;
  const bool resident = nslab == 1 && !(S::kRedInX && p.KS > 1);
  int e = 0, key_e = -1, key_m = -1;
  for (int item = item0; item < item1; ++item) {
    const int2 at = locate(item, e);
    const int tile = at.y * p.RT + rt;
    const bool fresh = !resident || e != key_e || at.x != key_m;
    key_e = e; key_m = at.x;
    for (int s = 0; s < nslab; ++s) {
      if (fresh) {
        if (item > item0 || s > 0) __syncthreads();       // nobody reads the old rows (or the shares' sums) any more
        stage(e, at.x, s);
        __syncthreads();
      }
      if (works && tile < tiles) {
        const int c1 = min(chunks, (s + 1) * (S::SLG / S::G));
        for (int c = s * (S::SLG / S::G) + ks; c < c1; c += p.KS) compute(c, (c - s * (S::SLG / S::G)) * S::G);
      }
    }
    finish(tile, e, at.x);
  }
  nw_wait<0>();
}

// ------------------------------------------------------------------------------------------------
// Quantised weights, up to 16 rows of x per pass.
//
// What bounds it: above some 20 MB the weights' trip from HBM; below, a chain of latencies (x to shared memory 2 us, a few stages of 0.6 us,
// the sums of shared tiles, the launch). Both ask for the same thing, that every warp has as much to do as every other:
//   * a block takes a contiguous run of 16-row tiles of W that meet the same rows of x, and its 16 warps split the run's (tile, stage)
//     pairs evenly, to the stage (256 or 128 of K of 16 rows). A warp that did all stages of a tile writes its result; where a tile's
//     stages fall to several warps, their sums meet in shared memory, added by the warp that began the tile, in order.
//   * where x does not fit the buffer (64 units of eight rows and a group), or a block would have too little to do, the blocks of a
//     cluster take K apart: each holds its share of x, and every tile's sums are read out of all blocks' shared memory, in order.
//   * the loop has no work but its own: pointers that step, no plan kept in registers, no barrier. 16 warps of 128 registers spill nothing
//     and stage x with half the barrier's stragglers of 24 warps of 80 (151936 x 4096 at 8 rows 78 us with 24 warps, 71 with 16 and two
//     stages, 67 with three).
//   * few (row, slot) pairs need no lists: each is an expert of its own, whose number is read from the choices; x stays where it is from
//     one expert to the next if all pairs are of one row.
//   * only rows that exist are staged: a column of B that holds nothing is a column of results that nobody takes.
// Measured against narrow_gemm_kernel, chained launches, weights out of HBM, 4-bit (us, it / this; their bytes at the copy rate): 8
// rows, 4096 x 4096 8.5 / 8.4 (1.5), 9216 x 4096 14.1 / 11.8 (3.3), 28672 x 4096 25 / 19 (10), 4096 x 14336 21 / 14 (5), 151936 x 4096 103 /
// 67 (54); 16 rows, 9216 x 4096 20 / 16, 28672 x 4096 34 / 26, 4096 x 14336 35 / 21; 128 experts of 4096 x 1536 at 64 rows of 8
// choices, gate and up 250 / 170 (139), down 141 / 94 (70).
template <int KIND, int T>
struct NeShape {
  static constexpr int W = 16, THREADS = W * 32, D = T == 1 ? 3 : 2;
  static constexpr int G = KIND == 1 ? 4 : 2, PC = 8 / G;         // groups per stage; stages per 16-byte piece of scales
  static constexpr int STAGE = 16 * kNwCB, SLOT = 512;            // rows; scales and biases, 16 bytes per row
  static constexpr int UNIT = 1024 + 32 + 64;                     // x of eight rows and a group; its scales; its sums in two terms
  static constexpr int P = W * 512 * T;                           // sums of tiles that another warp began
  static constexpr int FIXED = W * D * (STAGE + SLOT) + P + (2 * kNwMaxExperts + 4) * 4 + 8 * T * 4;
  static constexpr int UNITS = 64;
  static constexpr int ROUNDS = (UNITS + W - 1) / W;
  static constexpr int LIMIT = 227 * 1024;
};

__device__ __forceinline__ void ne_cp16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global.L2::256B [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void ne_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float ne_remote(uint32_t addr, int rank) {
  float v;
  asm volatile("{.reg .u32 a; mapa.shared::cluster.u32 a, %1, %2; ld.shared::cluster.f32 %0, [a];}" : "=f"(v) : "r"(addr), "r"(rank) : "memory");
  return v;
}

template <int KIND, int T>
__global__ void __launch_bounds__(NeShape<KIND, T>::THREADS, 1) narrow_even_kernel(const NeParams p) {
  using S = NeShape<KIND, T>;
  extern __shared__ __align__(128) char smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  char* const slots = smem + S::W * S::D * S::STAGE;
  float* const part = reinterpret_cast<float*>(slots + S::W * S::D * S::SLOT);
  float* const s_ssq = part + S::P / 4;                  // [8 T] the block's sums of squares
  int* const s_off = reinterpret_cast<int*>(s_ssq + 8 * T);
  int* const s_pre = s_off + kNwMaxExperts + 1;          // items before every expert
  char* const xbuf = smem + S::FIXED;
  float* const s_ss = reinterpret_cast<float*>(xbuf + p.xunits * S::UNIT);   // [unit][8]
  float* const sums = s_ss + p.xunits * 8;               // [RL][T * 4][32] the block's sums of every tile (clusters)

  int rank = 0;
  if (p.CS > 1) asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  const int groups = p.K >> 6, tiles_n = p.N >> 4, k512 = p.K >> 9, k0 = k512 * rank >> p.cs_log2;
  const int gsh = ((k512 * (rank + 1) >> p.cs_log2) - k0) * 8;   // this block's groups
  const int C = gsh / S::G;                              // and stages per tile
  constexpr int rows = 8 * T;
  const size_t row_bytes = size_t(p.K) / (KIND == 1 ? 2 : 1);
  pdl_launch_dependents();
  if (p.norm && int(threadIdx.x) < gsh) nw_prefetch(p.norm + (k0 * 8 + threadIdx.x) * 64);

  int* const s_map = s_off + kNwMaxExperts / 2;          // the experts of single rows
  if (p.choice) {
    pdl_wait();
    if (warp == 0) {
      const int c = lane < p.E ? p.choice[lane] : -1;
      const unsigned is = __ballot_sync(0xffffffffu, unsigned(c) < unsigned(p.experts));
      s_off[lane] = lane;
      s_pre[lane] = __popc(is & ((1u << lane) - 1u)) * tiles_n;
      s_map[lane] = c;
      if (lane == 31) { s_off[32] = 32; s_pre[32] = __popc(is) * tiles_n; }
    }
  } else if (p.offsets) {
    pdl_wait();
    for (int i = threadIdx.x; i <= p.E; i += S::THREADS) {
      const int o = p.offsets[i];
      s_off[i] = RB_BOUNDS(o, p.M + 1) ? o : 0;
    }
    __syncthreads();
    if (warp == 0) {       // items before every expert: a scan over 32 experts at a time
      int base = 0;
      for (int e0 = 0; e0 < p.E; e0 += 32) {
        const int e = e0 + lane;
        const int n = e < p.E ? s_off[e + 1] - s_off[e] : 0;
        const int mine = RB_BOUNDS(n, p.M + 1) ? (n + rows - 1) / rows * tiles_n : 0;
        int sum = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { const int v = __shfl_up_sync(0xffffffffu, sum, o); if (lane >= o) sum += v; }
        if (e < p.E) s_pre[e] = base + sum - mine;
        base += __shfl_sync(0xffffffffu, sum, 31);
      }
      if (lane == 0) s_pre[p.E] = base;
    }
  } else if (threadIdx.x == 0) {
    s_off[0] = 0; s_off[1] = p.M; s_pre[0] = 0; s_pre[1] = (p.M + rows - 1) / rows * tiles_n;
  }
  __syncthreads();
  // the clusters' items: a contiguous run each, the first ones one more
  const int cl = int(blockIdx.x) >> p.cs_log2, ncl = int(gridDim.x) >> p.cs_log2;
  const int each = s_pre[p.E] / ncl, more = s_pre[p.E] - each * ncl;
  const int item0 = cl * each + min(cl, more), item1 = item0 + each + (cl < more ? 1 : 0);
  if (item0 >= item1) return;                            // all blocks of the cluster alike

  // A run: tiles of 16 rows of W that meet the same rows of x. (e, pass of the expert, first tile, tiles)
  auto run_at = [&](int item, int& e, int& mt, int& tile0) {
    while (s_pre[e + 1] <= item) ++e;
    const int local = item - s_pre[e];
    mt = local / tiles_n; tile0 = local - mt * tiles_n;
    return min(min(tiles_n - tile0, item1 - item), p.RL);
  };

  // ---------------------------------------------------------------- weight ring (one per warp)
  const int half = p.swiglu ? p.N / 2 : 8, per = p.swiglu ? 8 : 16;   // rows 8.. of a tile are `half` rows of W further
  const uint32_t my_ring = smem_u32(smem) + warp * (S::D * S::STAGE), my_slots = smem_u32(slots) + warp * (S::D * S::SLOT);
  const size_t half_b = half * row_bytes, row4_b = 4 * row_bytes;
  // where this lane's 16 bytes of row lane / 8 go: 32-byte (4-bit) or 64-byte (8-bit) groups, moved by an exclusive or with the
  // row, so that the fragments' reads of eight rows hit all banks once
  const uint32_t my_dst = [&]() {
    const int r = lane >> 3, c16 = lane & 7;
    const int off = KIND == 1 ? (((c16 >> 1) ^ r) << 5) + (c16 & 1) * 16 : (((c16 >> 2) ^ (r & 1)) << 6) + (c16 & 3) * 16;
    return uint32_t(r * kNwCB + off);
  }();
  int p_item = item0, p_e = 0, p_left = 0, p_c = 0, p_stage = 0, p_slot = 0;
  bool p_fresh = true;                                   // the stage begins a piece of scales
  const uint8_t* p_w = nullptr;                          // this lane's 16 bytes of row lane / 8
  const uint8_t* p_s = nullptr;                          // lanes 0-15 the scales, 16-31 the biases, of row lane % 16
  auto p_run = [&]() {                                   // the next run in which this warp has a share
#pragma unroll 1
    while (p_left == 0 && p_item < item1) {
      int mt, tile0;
      const int n = run_at(p_item, p_e, mt, tile0), u = n * C;
      const int u0 = warp * u / S::W, u1 = (warp + 1) * u / S::W;
      p_item += n;
      if (u1 > u0) {
        const int tile = u0 / C;
        p_left = u1 - u0; p_c = u0 - tile * C; p_fresh = true;
        const size_t row = size_t(p.choice ? s_map[p_e] : p_e) * p.N + (tile0 + tile) * per;
        p_w = p.w + (row + (lane >> 3)) * row_bytes + (k0 * S::PC + p_c) * kNwCB + (lane & 7) * 16;
        p_s = reinterpret_cast<const uint8_t*>((lane < 16 ? p.scales : p.biases) + (row + (lane & 7) + ((lane >> 3) & 1) * half) * groups +
                                               (k0 + p_c / S::PC) * 8);
      }
    }
  };
  auto issue = [&]() {
    if (p_left == 0) p_run();
    if (p_left > 0) {
      const uint32_t st = my_ring + p_stage * S::STAGE + my_dst;
      ne_cp16(st, p_w);
      ne_cp16(st + 4 * kNwCB, p_w + row4_b);
      ne_cp16(st + 8 * kNwCB, p_w + half_b);
      ne_cp16(st + 12 * kNwCB, p_w + half_b + row4_b);
      if (p_fresh) {
        nw_cp16(my_slots + p_slot * S::SLOT + lane * 16, p_s);
        p_s += 16;
        if (++p_slot == S::D) p_slot = 0;
      }
      if (++p_stage == S::D) p_stage = 0;
      p_w += kNwCB;
      if (++p_c == C) {
        p_c = 0;
        p_w += per * row_bytes - C * kNwCB;
        p_s += size_t(per) * groups * 2 - gsh * 2;
      }
      p_fresh = p_c % S::PC == 0;
      --p_left;
    }
    nw_commit();
  };
#pragma unroll 1
  for (int i = 0; i < S::D - 1; ++i) issue();
  if (!p.offsets && !p.choice) pdl_wait();

  // ---------------------------------------------------------------- x
  auto out_row = [&](int e, int mt, int i) {             // output row of the pass's i-th row of x, -1: none
    const int pos = s_off[e] + mt * rows + i;
    if (pos >= s_off[e + 1]) return -1;
    if (!p.order) return pos;
    const int row = __ldg(p.order + pos);
    return RB_BOUNDS(row, p.M) ? row : -1;
  };
  // Unit u: tile u / gsh of the rows of x, group u % gsh. Four lanes hold a row's part of it, 16 values each: share t. Rows that the
  // pass does not have are columns whose results nobody takes: they are left as they are.
  auto stage = [&](int e, int mt) {
    const int have = min(s_off[e + 1] - s_off[e] - mt * rows, 8), lg = have > 4 ? 3 : have > 2 ? 2 : have - 1;
    const int quads = T * gsh << lg;
    constexpr int kAtOnce = S::ROUNDS < 4 ? S::ROUNDS : 4;
#pragma unroll 1
    for (int b = 0; b < S::ROUNDS && (warp + b * S::W) * 8 < quads; b += kAtOnce) {
      uint4 v[kAtOnce][2], nv[kAtOnce][2];
#pragma unroll
      for (int j = 0; j < kAtOnce; ++j) {
        const int q = (warp + (b + j) * S::W) * 8 + g, u = q >> lg, tile = T > 1 && u >= gsh ? 1 : 0;
        v[j][0] = v[j][1] = nv[j][0] = nv[j][1] = make_uint4(0u, 0u, 0u, 0u);
        if (q < quads) {
          const int at = (k0 * 8 + u - tile * gsh) * 64 + t * 16;
          if (const int row = out_row(e, mt, tile * 8 + (q & ((1 << lg) - 1))); row >= 0) {
            const uint4* src = reinterpret_cast<const uint4*>(p.x + size_t(p.x_div > 1 ? row / p.x_div : row) * p.x_stride + at);
            v[j][0] = src[0]; v[j][1] = src[1];
          }
          if (p.norm) {
            const uint4* src = reinterpret_cast<const uint4*>(p.norm + at);
            nv[j][0] = src[0]; nv[j][1] = src[1];
          }
        }
      }
#pragma unroll
      for (int j = 0; j < kAtOnce; ++j) {
        if ((warp + (b + j) * S::W) * 8 >= quads) break;
        const int q = (warp + (b + j) * S::W) * 8 + g, u = q >> lg, row = q & ((1 << lg) - 1);
        const uint32_t w[8] = {v[j][0].x, v[j][0].y, v[j][0].z, v[j][0].w, v[j][1].x, v[j][1].y, v[j][1].z, v[j][1].w};
        float f[16];
#pragma unroll
        for (int i = 0; i < 8; ++i) { f[2 * i] = bf16lo(w[i]); f[2 * i + 1] = bf16hi(w[i]); }
        if (p.norm) {
          float ss = 0.f;
#pragma unroll
          for (int i = 0; i < 16; ++i) ss = fmaf(f[i], f[i], ss);
          ss += __shfl_xor_sync(0xffffffffu, ss, 1);
          ss += __shfl_xor_sync(0xffffffffu, ss, 2);
          if (t == 0 && q < quads) s_ss[u * 8 + row] = ss;
          const uint32_t nw[8] = {nv[j][0].x, nv[j][0].y, nv[j][0].z, nv[j][0].w, nv[j][1].x, nv[j][1].y, nv[j][1].z, nv[j][1].w};
#pragma unroll
          for (int i = 0; i < 8; ++i) { f[2 * i] *= bf16lo(nw[i]); f[2 * i + 1] *= bf16hi(nw[i]); }
        }
        uint32_t o[8];
        float down, sum;
        nw_group_fp16<KIND>(f, p.norm != nullptr, o, down, sum);
        if (q >= quads) continue;
        char* const dst = xbuf + u * S::UNIT;
        if (t == 0) {
          // the sum of x goes in two tf32 terms (2^-22 of it together), multiplied with the biases, which are exact in tf32
          const uint32_t s_hi = __float_as_uint(sum) & 0xffffe000u;
          const uint32_t s_lo = __float_as_uint(sum - __uint_as_float(s_hi)) & 0xffffe000u;
          *reinterpret_cast<float*>(dst + 1024 + row * 4) = down;
          *reinterpret_cast<uint2*>(dst + 1056 + row * 8) = make_uint2(s_hi, s_lo);
        }
        *reinterpret_cast<uint4*>(dst + row * 64 + t * 16) = make_uint4(o[0], o[1], o[2], o[3]);
        *reinterpret_cast<uint4*>(dst + 512 + row * 64 + t * 16) = make_uint4(o[4], o[5], o[6], o[7]);
      }
    }
  };

  // ---------------------------------------------------------------- results
  auto put = [&](int row, int col, float v) {
    if (row < 0) return;
    if (p.residual) v += __bfloat162float(p.residual[size_t(row) * p.res_stride + col]);
    if (p.out_f32) static_cast<float*>(p.out)[size_t(row) * p.out_stride + col] = v;
    else static_cast<__nv_bfloat16*>(p.out)[size_t(row) * p.out_stride + col] = __float2bfloat16_rn(v);
  };
  auto emit = [&](int e, int mt, int tile, const float (&d)[T][4], const float (&rs)[T]) {
#pragma unroll
    for (int n = 0; n < T; ++n) {
      const int row0 = out_row(e, mt, n * 8 + 2 * t), row1 = out_row(e, mt, n * 8 + 2 * t + 1);
      float r0 = 16777216.f, r1 = r0;
      if (p.norm) { r0 *= __shfl_sync(0xffffffffu, rs[n], 2 * t); r1 *= __shfl_sync(0xffffffffu, rs[n], 2 * t + 1); }
      const float a0 = d[n][0] * r0, a1 = d[n][1] * r1, b0 = d[n][2] * r0, b1 = d[n][3] * r1;
      if (p.swiglu) {
        put(row0, tile * 8 + g, gated_act(a0, b0, 0.f));
        put(row1, tile * 8 + g, gated_act(a1, b1, 0.f));
      } else {
        put(row0, tile * 16 + g, a0);
        put(row1, tile * 16 + g, a1);
        put(row0, tile * 16 + g + 8, b0);
        put(row1, tile * 16 + g + 8, b1);
      }
    }
  };

  // rows g and g + 8 of a stage, this lane's share of a group
  const int my_src = warp * (S::D * S::STAGE) + (KIND == 1 ? g * kNwCB + t * 8 + ((g & 3) << 5) : g * kNwCB + t * 16 + ((g & 1) << 6));
  const char* const slot_p = slots + warp * (S::D * S::SLOT) + g * 16;
  const int nstride = gsh * S::UNIT;
  int c_stage = 0, c_slot = S::D - 1, e = 0, key_e = -1, key_m = -1;
  for (int item = item0; item < item1;) {
    int mt, tile0;
    const int tiles = run_at(item, e, mt, tile0), u = tiles * C;
    const int u0 = warp * u / S::W, u1 = (warp + 1) * u / S::W;
    // single rows that are all the same row of x stay where they are
    if (const int x_of = p.choice && p.x_div >= p.M ? 0 : e; x_of != key_e || mt != key_m) { stage(e, mt); key_e = x_of; key_m = mt; }
    if (p.CS > 1) ne_cluster_sync(); else __syncthreads();

    float rs[T] = {};                                    // 1 / rms of row lane % 8 of the tile
    if (p.norm) {
#pragma unroll
      for (int n = 0; n < T; ++n) {
        float ss = 0.f;
        for (int gi = lane >> 3; gi < gsh; gi += 4) ss += s_ss[(n * gsh + gi) * 8 + (lane & 7)];
        ss += __shfl_xor_sync(0xffffffffu, ss, 8);
        ss += __shfl_xor_sync(0xffffffffu, ss, 16);
        if (p.CS > 1 && warp == 0 && lane < 8) s_ssq[n * 8 + lane] = ss;
        rs[n] = rsqrtf(ss / float(p.K) + p.eps);
      }
    }

    float acc[T][4] = {};
    int i = u0, tile = u0 / C, c = u0 - tile * C;
    bool began = c == 0, fresh = true;                   // whether this warp's share has the tile's first stage
    while (true) {
#pragma unroll 1
      for (; i < u1; ++i) {
        nw_wait<S::D - 2>();
        __syncwarp();
        issue();                                         // refills the stage that the previous round read
        const int wo = my_src + c_stage * S::STAGE;
        if (++c_stage == S::D) c_stage = 0;
        if (fresh || c % S::PC == 0) {
          fresh = false;
          if (++c_slot == S::D) c_slot = 0;
        }
        const char* const sp = slot_p + c_slot * S::SLOT + (KIND == 1 ? (c & 1) * 8 : (c & 3) * 4);
        uint32_t sc2[2][2];                              // scales of rows g, g + 8: two groups per word
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          if constexpr (KIND == 1) {
            const uint2 v = *reinterpret_cast<const uint2*>(sp + r * 128); sc2[r][0] = v.x; sc2[r][1] = v.y;
          } else {
            sc2[r][0] = *reinterpret_cast<const uint32_t*>(sp + r * 128);
          }
        }
        const char* const xp = xbuf + c * (S::G * S::UNIT);
        {   // biases x sums of x, all groups of the stage in one product: k is (group t, first term), (group t, second term)
          uint32_t b0 = 0u, b1 = 0u;
          if (KIND == 1 || t < S::G) {
            const char* const ba = sp + 256 + (t & (S::G - 1)) * 2;
            b0 = uint32_t(*reinterpret_cast<const uint16_t*>(ba)) << 16;
            b1 = uint32_t(*reinterpret_cast<const uint16_t*>(ba + 128)) << 16;
          }
#pragma unroll
          for (int n = 0; n < T; ++n) {
            const uint2 v = *reinterpret_cast<const uint2*>(xp + (t & (S::G - 1)) * S::UNIT + 1056 + g * 8 + n * nstride);
            nw_mma_tf32(acc[n], b0, b1, b0, b1, v.x, v.y);
          }
        }
#pragma unroll
        for (int j = 0; j < S::G; ++j) {
          uint32_t a[2][8];                               // [row g, g + 8][operand words of the four products]
          const char* const wj = smem + (wo ^ (KIND == 1 ? j << 5 : j << 6));    // the swizzle is an exclusive or with the group
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            if constexpr (KIND == 1) {
              const uint2 v = *reinterpret_cast<const uint2*>(wj + 8 * r * kNwCB);
#pragma unroll
              for (int h = 0; h < 2; ++h) {
                const uint32_t w = h ? v.y : v.x, w8 = w >> 8;
                a[r][4 * h + 0] = w & 0x000f000fu; a[r][4 * h + 1] = w & 0x00f000f0u;
                a[r][4 * h + 2] = w8 & 0x000f000fu; a[r][4 * h + 3] = w8 & 0x00f000f0u;
              }
            } else {
              const uint4 v = *reinterpret_cast<const uint4*>(wj + 8 * r * kNwCB);
              const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
              for (int k = 0; k < 4; ++k) {
                a[r][2 * k] = __byte_perm(w[k], 0u, 0x4140u);
                a[r][2 * k + 1] = __byte_perm(w[k], 0u, 0x4342u);
              }
            }
          }
          uint32_t sc[2];                                 // as bits
#pragma unroll
          for (int r = 0; r < 2; ++r) sc[r] = (j & 1) ? sc2[r][j >> 1] & 0xffff0000u : sc2[r][j >> 1] << 16;
#pragma unroll
          for (int n = 0; n < T; ++n) {
            const char* const xj = xp + j * S::UNIT + n * nstride;
            const uint4 x0 = *reinterpret_cast<const uint4*>(xj + lane * 16), x1 = *reinterpret_cast<const uint4*>(xj + 512 + lane * 16);
            const uint2 xq = *reinterpret_cast<const uint2*>(xj + 1024 + t * 8);    // scales of rows 2t and 2t + 1
            float d[4];
            nw_mma0<true>(d, a[0][0], a[1][0], a[0][1], a[1][1], x0.x, x0.y);
            nw_mma<true>(d, a[0][2], a[1][2], a[0][3], a[1][3], x0.z, x0.w);
            nw_mma<true>(d, a[0][4], a[1][4], a[0][5], a[1][5], x1.x, x1.y);
            nw_mma<true>(d, a[0][6], a[1][6], a[0][7], a[1][7], x1.z, x1.w);
            // two columns per instruction: (scale x scale of x) d + acc
            const uint64_t xsc = nw_pair(xq.x, xq.y);
#pragma unroll
            for (int r = 0; r < 2; ++r) {
              uint64_t s = nw_pair(__float_as_uint(acc[n][2 * r]), __float_as_uint(acc[n][2 * r + 1]));
              s = nw_fma2(nw_mul2(nw_pair(sc[r], sc[r]), xsc),
                          nw_pair(__float_as_uint(d[2 * r]), __float_as_uint(d[2 * r + 1])), s);
              nw_unpair(s, acc[n][2 * r], acc[n][2 * r + 1]);
            }
          }
        }
        if (++c == C) { ++i; break; }
      }
      // the tile, or this warp's share of it, is done
      const bool last = i == u1, open = c != C;
      if (!began && u1 > u0) {
#pragma unroll
        for (int k = 0; k < T * 4; ++k) part[(warp * (T * 4) + k) * 32 + lane] = (&acc[0][0])[k];
      }
      if (last) __syncthreads();
      if (began && u1 > u0) {
        if (open) {                                       // add the other warps' shares, in order
          const int end = (tile + 1) * C;
          for (int w = warp + 1; w < S::W; ++w) {
            const int w0 = w * u / S::W, w1 = (w + 1) * u / S::W;
            if (w0 >= end) break;
            if (w1 > w0) {
#pragma unroll
              for (int k = 0; k < T * 4; ++k) (&acc[0][0])[k] += part[(w * (T * 4) + k) * 32 + lane];
            }
          }
        }
        if (p.CS > 1) {
#pragma unroll
          for (int k = 0; k < T * 4; ++k) sums[(tile * (T * 4) + k) * 32 + lane] = (&acc[0][0])[k];
        } else {
          emit(e, mt, tile0 + tile, acc, rs);
        }
      }
      if (last) break;
      c = 0; ++tile; began = true;
#pragma unroll
      for (int k = 0; k < T * 4; ++k) (&acc[0][0])[k] = 0.f;
    }
    if (p.CS > 1) {                                       // every block adds up its tiles over the cluster, ranks in order
      ne_cluster_sync();
      for (int tl = rank + p.CS * warp; tl < tiles; tl += p.CS * S::W) {
        float d[T][4] = {}, q[T] = {};
        for (int r = 0; r < p.CS; ++r) {
#pragma unroll
          for (int k = 0; k < T * 4; ++k) (&d[0][0])[k] += ne_remote(smem_u32(sums + (tl * (T * 4) + k) * 32 + lane), r);
          if (p.norm)
#pragma unroll
            for (int n = 0; n < T; ++n) q[n] += ne_remote(smem_u32(s_ssq + n * 8 + (lane & 7)), r);
        }
#pragma unroll
        for (int n = 0; n < T; ++n) q[n] = rsqrtf(q[n] / float(p.K) + p.eps);
        emit(e, mt, tile0 + tl, d, q);
      }
    }
    item += tiles;
  }
  nw_wait<0>();
  if (p.CS > 1) ne_cluster_sync();                        // nobody leaves while its sums are read
}


// Pairs by expert in one block: counts, offsets [E + 1] (offsets[E]: all that chose an expert), and the pairs of an expert in their own
// order: a pair's place decides which pass takes it, and passes add up K in different shares, so that any other order would make
// results differ in their last bits from run to run. A warp counts a run of the pairs, 32 at a time. A choice outside [0, E) (a row of
// NaN logits has no largest one: decode_moe.cu) is in no expert's list, and the combination skips it.
__global__ void __launch_bounds__(1024) narrow_group_kernel(const int* __restrict__ idx, int pairs, int E,
                                                            int* __restrict__ offsets, int* __restrict__ order) {
  __shared__ int count[32][kNwMaxExperts], start[kNwMaxExperts + 1];   // [warp][expert]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  const int run = (pairs + 32 * warps - 1) / (32 * warps) * 32, i0 = warp * run, i1 = min(i0 + run, pairs);
  pdl_launch_dependents();
  for (int e = lane; e < E; e += 32) count[warp][e] = 0;
  __syncwarp();
  pdl_wait();
  // the lanes of a warp that chose the same expert: from a vote on each bit of its number, a third of __match_any_sync's time
  auto alike = [&](int e) {
    unsigned same = __ballot_sync(0xffffffffu, unsigned(e) < unsigned(E));
#pragma unroll
    for (int bit = 0; bit < 8; ++bit) {
      const unsigned set = __ballot_sync(0xffffffffu, e >> bit & 1);
      same &= e >> bit & 1 ? set : ~set;
    }
    return unsigned(e) < unsigned(E) ? same : 0u;
  };
  constexpr int kKept = 2;                               // of the first steps is kept what the second pass needs
  int e_of[kKept];
  unsigned same_of[kKept];
#pragma unroll
  for (int c = 0; c < kKept; ++c) {
    const int i = i0 + c * 32 + lane;
    e_of[c] = i < i1 ? idx[i] : -1;
  }
#pragma unroll
  for (int c = 0; c < kKept; ++c) {
    if (i0 + c * 32 >= i1) break;
    same_of[c] = alike(e_of[c]);
    if (same_of[c] && lane == __ffs(same_of[c]) - 1) count[warp][e_of[c]] += __popc(same_of[c]);
    __syncwarp();
  }
  for (int i = i0 + kKept * 32 + lane; i - lane < i1; i += 32) {
    const int e = i < i1 ? idx[i] : -1;
    const unsigned same = alike(e);
    if (same && lane == __ffs(same) - 1) count[warp][e] += __popc(same);
    __syncwarp();
  }
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += blockDim.x) {     // the warps' places within an expert
    int sum = 0;
#pragma unroll 8
    for (int w = 0; w < warps; ++w) { const int n = count[w][e]; count[w][e] = sum; sum += n; }
    start[e] = sum;
  }
  __syncthreads();
  if (warp == 0) {
    int base = 0;
    for (int e0 = 0; e0 < E; e0 += 32) {
      const int e = e0 + lane;
      const int mine = e < E ? start[e] : 0;
      int sum = mine;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) { const int v = __shfl_up_sync(0xffffffffu, sum, o); if (lane >= o) sum += v; }
      if (e < E) start[e] = base + sum - mine;
      base += __shfl_sync(0xffffffffu, sum, 31);
    }
    if (lane == 0) start[E] = base;
  }
  __syncthreads();
  for (int i = threadIdx.x; i <= E; i += blockDim.x) offsets[i] = start[i];
  auto place = [&](int i, int e, unsigned same) {
    const int at = same ? count[warp][e] : 0;
    __syncwarp();
    if (same) {
      order[start[e] + at + __popc(same & ((1u << lane) - 1u))] = i;
      if (lane == __ffs(same) - 1) count[warp][e] = at + __popc(same);
    }
    __syncwarp();
  };
#pragma unroll
  for (int c = 0; c < kKept; ++c) {
    if (i0 + c * 32 >= i1) break;
    place(i0 + c * 32 + lane, e_of[c], same_of[c]);
  }
  for (int i = i0 + kKept * 32 + lane; i - lane < i1; i += 32) {
    const int e = i < i1 ? idx[i] : -1;
    place(i, e, alike(e));
  }
}

// out[t] = residual[t] + sum_s w[t, s] y[t k + s], slots in order, y in fp32; slots whose choice idx[t, s] is no expert are
// skipped (nobody has written their y).
__global__ void __launch_bounds__(256) narrow_combine_kernel(const float* __restrict__ y, const int* __restrict__ idx, int E,
                                                             const float* __restrict__ wts,
                                                             const __nv_bfloat16* __restrict__ residual, int res_stride,
                                                             __nv_bfloat16* __restrict__ out, int out_stride, int top_k, int D) {
  const int row = blockIdx.y, c = (blockIdx.x * blockDim.x + threadIdx.x) * 4;
  pdl_launch_dependents();
  pdl_wait();
  if (c >= D) return;
  float a[4] = {0.f, 0.f, 0.f, 0.f};
  if (residual) {
    const uint2 r = *reinterpret_cast<const uint2*>(residual + size_t(row) * res_stride + c);
    a[0] = bf16lo(r.x); a[1] = bf16hi(r.x); a[2] = bf16lo(r.y); a[3] = bf16hi(r.y);
  }
#pragma unroll 8
  for (int s = 0; s < top_k; ++s) {
    if (unsigned(idx[row * top_k + s]) >= unsigned(E)) continue;
    const float w = wts[row * top_k + s];
    const float4 v = *reinterpret_cast<const float4*>(y + size_t(row * top_k + s) * D + c);
    a[0] = fmaf(w, v.x, a[0]); a[1] = fmaf(w, v.y, a[1]); a[2] = fmaf(w, v.z, a[2]); a[3] = fmaf(w, v.w, a[3]);
  }
  uint2 o;
  o.x = pack_bf16(a[0], a[1]); o.y = pack_bf16(a[2], a[3]);
  *reinterpret_cast<uint2*>(out + size_t(row) * out_stride + c) = o;
}

// Shares of K and row tiles per item: the blocks' runs of items should be even, an item costs its weights plus what is lost
// at its ends (reduction, barriers), every share must have a stage of each slab, and fewer than twelve working warps no longer
// keep an SM's issue slots and loads busy.
struct NwSplit { int ks, rt; };
static NwSplit nw_split(int warps, int tiles, int groups, int passes, int per_stage, int ks_max, int sms) {
  NwSplit best = {1, warps};
  double best_cost = 1e30;
  for (int ks = 1; ks <= ks_max && ks * per_stage <= groups; ks *= 2)
    for (int rt = warps / ks; rt >= 1; --rt) {
      const long long items = (long long)passes * ((tiles + rt - 1) / rt);
      const double busy = rt * ks >= 12 ? 1.0 : rt * ks / 12.0;
      const double cost = double((items + sms - 1) / sms) * (double(groups) * rt / busy + (ks > 1 ? 24.0 : 6.0));
      if (cost < best_cost * (1.0 - 1e-9)) { best = {ks, rt}; best_cost = cost; }
    }
  return best;
}

template <int KIND, int T>
static int launch_narrow(NwParams p, int passes, int ks_force, int pdl, cudaStream_t st) {
  using S = NwShape<KIND, T>;
  static_assert(S::BYTES <= 227 * 1024, "shared memory");
  static_assert(S::STAGE % 128 == 0, "the swizzle is an exclusive or with address bits");
  static_assert(!S::kRedInX || S::W * 512 * T <= S::X, "the shares' sums fit the x buffer");
  auto kern = narrow_gemm_kernel<KIND, T>;
  RB_CHECK(set_max_smem(kern, S::BYTES));
  const int sms = sm_count(), tiles = p.N / 16;
  NwSplit sp = nw_split(S::W, tiles, p.K / 64, passes, S::G, S::KSMAX, sms);
  if (ks_force > 0) { sp.ks = ks_force < S::KSMAX ? ks_force : S::KSMAX; sp.rt = S::W / sp.ks; }
  p.KS = sp.ks;
  p.RT = sp.rt;
  const long long items = (long long)passes * ((tiles + p.RT - 1) / p.RT);
  const int grid = p.offsets ? sms : int(items < sms ? items : sms);
  return launch(kern, dim3(grid), dim3(S::THREADS), size_t(S::BYTES), st, pdl != 0, p);
}

// Clusters of `cs` blocks of one per SM that can be resident at once.
template <class Kern>
static int ne_max_clusters(Kern kern, int cs, int threads, int smem) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(cs * 64);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cs; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr; cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) { (void)cudaGetLastError(); return 0; }
  return n;
}

// -2: not a shape of the even split.
template <int KIND, int T>
static int launch_even(NeParams p, int passes, int force, int pdl, cudaStream_t st) {
  using S = NeShape<KIND, T>;
  auto kern = narrow_even_kernel<KIND, T>;
  const int k512 = p.K / 512, tiles = p.N / 16, sms = sm_count();
  int dev = 0;
  RB_CHECK(cudaGetDevice(&dev));
  static int clusters[64][4] = {};                        // cs = 1 << i; 0: not asked yet
  const long long items = (long long)passes * tiles;
  double best = 1e30;
  int lg = -1, ncl = 0;
  for (int i = 0; i < 4; ++i) {
    const int c = 1 << i, share = (k512 + c - 1) / c * 8;
    if (c > k512 || T * share > S::UNITS) continue;
    int n = sms;
    if (c > 1) {
      int& known = clusters[dev & 63][i];
      if (known == 0) {
        RB_CHECK(set_max_smem(kern, S::LIMIT));
        const int m = ne_max_clusters(kern, c, S::THREADS, S::LIMIT);
        known = m > 0 ? m : -1;
      }
      if (known < 0) continue;
      n = known;
    }
    const double units = double((items + n - 1) / n) * share / S::G;
    double cost = units / S::W + T * share / 48.0 + (c > 1 ? 1.0 : 0.0);
    if (c == force) cost = -1.0;
    if (cost < best) { best = cost; lg = i; ncl = n; }
  }
  if (lg < 0) return -2;
  if (!p.offsets && items < ncl) ncl = int(items);
  p.CS = 1 << lg;
  p.cs_log2 = lg;
  p.xunits = T * ((k512 + p.CS - 1) / p.CS * 8);
  p.RL = tiles;
  int smem = S::FIXED + p.xunits * (S::UNIT + 32);
  if (lg) {
    const long long room = (S::LIMIT - smem) / (512 * T), want = (items + ncl - 1) / ncl;
    if (want < p.RL) p.RL = int(want);
    if (room < p.RL) p.RL = int(room);
    smem += p.RL * 512 * T;
  }
  RB_CHECK(set_max_smem(kern, S::LIMIT));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ncl << lg);
  cfg.blockDim = dim3(S::THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  int n = 0;
  if (lg) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = p.CS; attr[n].val.clusterDim.y = 1; attr[n].val.clusterDim.z = 1;
    ++n;
  }
  if (pdl) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n].val.programmaticStreamSerializationAllowed = 1;
    ++n;
    prefer_max_shared(kern);
  }
  cfg.attrs = attr;
  cfg.numAttrs = n;
  const cudaError_t err = cudaLaunchKernelEx(&cfg, kern, p);
  if (err != cudaSuccess) (void)cudaGetLastError();
  return static_cast<int>(err);
}

template <int KIND>
static int launch_narrow_t(const NwParams& p, int T, int passes, int ks, int pdl, cudaStream_t st) {
  switch (T) {
    case 1: return launch_narrow<KIND, 1>(p, passes, ks, pdl, st);
    case 2: return launch_narrow<KIND, 2>(p, passes, ks, pdl, st);
    case 4: return launch_narrow<KIND, 4>(p, passes, ks, pdl, st);
  }
  return -2;
}

}  // namespace rb

using namespace rb;
RB_BOUNDS_REGISTER("narrow_gemm.cu")

// Whether the kernel takes a weight of this kind, N rows (stacked gate and up rows included) and K columns: whole ring
// stages, 16-byte rows of scales, whole 16-row tiles.
extern "C" int rmlx_narrow_supported(int w_kind, int N, int K) {
  if (w_kind < 0 || w_kind >= kNwKinds || N < 16 || N % 16) return 0;
  return w_kind == 0 ? K >= 64 && K % 64 == 0 : K >= 512 && K % 512 == 0;
}

// tiles: rows of x per pass in units of eight (1, 2, 4; 0: chosen from rows, the expected rows per expert). ks: warps (quantised weights,
// even split: blocks) that share K, 0: chosen.
extern "C" int rmlx_narrow_gemm(int w_kind, const void* w, const void* scales, const void* biases, const void* x, int x_stride,
                                int x_div, const int* order, const int* offsets, int E, const void* norm, float eps,
                                const void* residual, int res_stride, void* out, int out_stride, int out_f32, int M, int N, int K,
                                int swiglu, int tiles, int ks, int pdl, cudaStream_t st) {
  if (!rmlx_narrow_supported(w_kind, N, K) || M < 1 || E < 1 || E > kNwMaxExperts || x_stride % 8 || x_div < 1) return -2;
  if (swiglu && residual) return -2;
  const int split = w_kind == 0 && norm != nullptr;      // twice the tiles for the same rows
  if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w)) & 15) return -2;
  if (norm && (reinterpret_cast<uintptr_t>(norm) & 15)) return -2;
  if (w_kind && (!scales || !biases || ((reinterpret_cast<uintptr_t>(scales) | reinterpret_cast<uintptr_t>(biases)) & 15))) return -2;
  if (ks < 0 || ks > 8 || (ks & (ks - 1))) return -2;
  NwParams p = {};
  p.w = static_cast<const uint8_t*>(w);
  p.scales = static_cast<const __nv_bfloat16*>(scales);
  p.biases = static_cast<const __nv_bfloat16*>(biases);
  p.x = static_cast<const __nv_bfloat16*>(x);
  p.order = order; p.offsets = offsets;
  p.norm = static_cast<const __nv_bfloat16*>(norm);
  p.residual = static_cast<const __nv_bfloat16*>(residual);
  p.out = out; p.eps = eps; p.x_stride = x_stride; p.x_div = x_div;
  p.out_stride = out_stride; p.out_f32 = out_f32; p.res_stride = res_stride;
  p.E = E; p.M = M; p.N = N; p.K = K; p.swiglu = swiglu;
  // rows of x per expert, and how many passes over the weights that makes (for the even split of the work)
  int T = tiles, hint;
  const bool even = w_kind && K <= 32768;
  if (offsets) {
    // 128 experts of 4096 x 1536 in 4 bits, both projections: one tile 273 us and two 413 at four rows per expert, 382 and 424 at
    // eight, 442 and 404 at ten, 654 and 577 at sixteen
    if (!T) T = even ? (M > 9 * E && K <= 16384 ? 2 : 1) : split || M > 6 * E ? 2 : 1;
    const int used = M < E ? M : E, rows = 8 * T >> split;
    hint = used > (M + rows - 1) / rows ? used : (M + rows - 1) / rows;
  } else {
    // two tiles expand a weight once for sixteen rows, but x fills twice the buffer: a third pass of one tile still beats a second of
    // two for wide or long projections (4-bit, 24 rows: 4096 x 14336 30 us against 37, 9216 x 4096 17 against 19, 4096 x 8192 22
    // against 19)
    if (!T && even) T = M <= 8 || K > 16384 || (M > 16 && M <= 24 && (N > 4096 || K > 8192)) ? 1 : 2;
    if (!T) T = (M <= 8 ? 1 : M <= 16 ? 2 : 4) << (split && M <= 16);
    hint = (M + (8 * T >> split) - 1) / (8 * T >> split);
  }
  if (split && T < 2) return -2;
  p.split = split;
  if (w_kind && T <= 2) {
    NeParams ne = {};
    static_cast<NwParams&>(ne) = p;
    const int rc = w_kind == 1 ? (T == 1 ? launch_even<1, 1>(ne, hint, ks, pdl, st) : launch_even<1, 2>(ne, hint, ks, pdl, st))
                               : (T == 1 ? launch_even<2, 1>(ne, hint, ks, pdl, st) : launch_even<2, 2>(ne, hint, ks, pdl, st));
    if (rc != -2) return rc;
  }
  switch (w_kind) {
    case 0: return launch_narrow_t<0>(p, T, hint, ks, pdl, st);
    case 1: return launch_narrow_t<1>(p, T, hint, ks, pdl, st);
    default: return launch_narrow_t<2>(p, T, hint, ks, pdl, st);
  }
}

// Single (row, slot) pairs, up to 32: output row i is row i / x_div of x through expert choice[i] of w [experts, N, K] (4- or 8-bit);
// rows whose choice is no expert are not written.
extern "C" int rmlx_narrow_pairs(int w_kind, const void* w, const void* scales, const void* biases, const void* x, int x_stride, int x_div,
                                 const int* choice, int experts, const void* norm, float eps, void* out, int out_stride, int out_f32,
                                 int pairs, int N, int K, int swiglu, int pdl, cudaStream_t st) {
  if (w_kind < 1 || !rmlx_narrow_supported(w_kind, N, K) || K > 32768 || pairs < 1 || pairs > 32 || experts < 1 || x_stride % 8 || x_div < 1 ||
      (swiglu && N % 32) || !choice || !scales || !biases)
    return -2;
  if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(scales) |
       reinterpret_cast<uintptr_t>(biases) | reinterpret_cast<uintptr_t>(norm)) & 15)
    return -2;
  NeParams p = {};
  p.w = static_cast<const uint8_t*>(w);
  p.scales = static_cast<const __nv_bfloat16*>(scales);
  p.biases = static_cast<const __nv_bfloat16*>(biases);
  p.x = static_cast<const __nv_bfloat16*>(x);
  p.norm = static_cast<const __nv_bfloat16*>(norm);
  p.out = out; p.eps = eps; p.x_stride = x_stride; p.x_div = x_div;
  p.out_stride = out_stride; p.out_f32 = out_f32;
  p.E = p.M = pairs; p.N = N; p.K = K; p.swiglu = swiglu;
  p.choice = choice; p.experts = experts;
  return w_kind == 1 ? launch_even<1, 1>(p, pairs, 0, pdl, st) : launch_even<2, 1>(p, pairs, 0, pdl, st);
}

extern "C" int rmlx_narrow_group(const int* idx, int pairs, int E, int* offsets, int* order, int pdl, cudaStream_t st) {
  if (pairs < 1 || E < 1 || E > kNwMaxExperts) return -2;
  const int threads = pairs >= 1024 ? 1024 : pairs <= 128 ? 128 : (pairs + 31) / 32 * 32;
  return launch(narrow_group_kernel, dim3(1), dim3(threads), 0, st, pdl != 0, idx, pairs, E, offsets, order);
}

extern "C" int rmlx_narrow_combine(const float* y, const int* idx, int E, const float* wts, const void* residual, int res_stride, void* out,
                                   int out_stride, int rows, int top_k, int D, int pdl, cudaStream_t st) {
  if (rows < 1 || D % 4) return -2;
  return launch(narrow_combine_kernel, dim3((D / 4 + 255) / 256, rows), dim3(256), 0, st, pdl != 0, y, idx, E, wts,
                static_cast<const __nv_bfloat16*>(residual), res_stride, static_cast<__nv_bfloat16*>(out), out_stride, top_k, D);
}
