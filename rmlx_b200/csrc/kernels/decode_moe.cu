// Decode-time mixture-of-experts kernels. Routing, offsets and expert selection never leave the
// device (the reference reads the routing result back to the host on every forward,
// crates/rmlx-nn/src/moe.rs:600-601).
//
//   moe_router        RMSNorm + gate projection + softmax + top-k + renormalise, one launch; a
//                     cluster of blocks takes eight rows and selects their experts
//                     (reference: moe_topk_route_f32, crates/rmlx-core/src/ops/topk_route.rs:212)
//   topk_route        the same selection over precomputed logits for many tokens, with the
//                     per-expert histogram; prefix offsets by moe_prefix_offsets
//                     (reference: moe_prefix_scan_u32, topk_route.rs:373)
//   moe_gate_up       per (token, slot): act = silu(Wg[e]·xn) * (Wu[e]·xn), RMSNorm folded in
//   moe_down          per token: out = residual + sum_slot w_slot * Wd[e_slot]·act[slot]
//                     (reference: gather_qmv_fast_*, crates/rmlx-core/src/ops/quantized.rs:9634 and
//                     ExpertGroup::grouped_forward, crates/rmlx-nn/src/expert_group.rs:308)
#include <cstdlib>
#include "../common/gemv_core.cuh"
#include "../common/launch.cuh"

namespace rb {

constexpr int kMaxExperts = 256;
constexpr int kMaxTopK = 8;

// Softmax over E logits held up to 8-per-lane, then k rounds of warp arg-max (ties: lowest index wins), weights renormalised to
// sum 1. Executed by one full warp for one token. The rounds are a chain: each is two warp reductions of integers (a probability's
// bits order as it does; 1 is added so that 0 is below all of them) instead of ten shuffles and their comparisons.
// NaN logits have no largest one: such a row's choices are numbers outside [0, E), which are not counted and which every user of
// the choices skips.
template <int V>
__device__ __forceinline__ void warp_topk_v(const float* logits, const float* bias, int E, int k, int* out_idx, float* out_w, int* counts) {
  const int lane = threadIdx.x & 31;
  float v[V];
  float m = -INFINITY;
#pragma unroll
  for (int i = 0; i < V; ++i) {
    const int e = i * 32 + lane;
    v[i] = (e < E) ? logits[e] + (bias ? bias[e] : 0.f) : -INFINITY;
    m = fmaxf(m, v[i]);
  }
  m = warp_max(m);
  float s = 0.f;
  uint32_t key[V];
#pragma unroll
  for (int i = 0; i < V; ++i) {
    const float p = (i * 32 + lane < E) ? __expf(v[i] - m) : 0.f;
    s += fmaxf(p, 0.f);
    const uint32_t bits = __float_as_uint(p);
    key[i] = (i * 32 + lane < E && bits <= 0x7f800000u) ? bits + 1u : 0u;   // neither absent nor NaN
  }
  s = warp_sum(s);
  const float inv = 1.f / s;
  float sel_w = 0.f;
  int sel_e = 0;
  float wsum = 0.f;
  for (int r = 0; r < k; ++r) {
    uint32_t best = key[0];
    int at = 0;
#pragma unroll
    for (int i = 1; i < V; ++i)
      if (key[i] > best) { best = key[i]; at = i; }
    const uint32_t top = __reduce_max_sync(0xffffffffu, best);
    const uint32_t e = __reduce_min_sync(0xffffffffu, best == top && top ? uint32_t(at * 32 + lane) : 0x7fffffffu);
#pragma unroll
    for (int i = 0; i < V; ++i)
      if (uint32_t(i * 32 + lane) == e) key[i] = 0u;
    const float p = (top ? __uint_as_float(top - 1u) : -2.f) * inv;
    wsum += p;
    if (lane == r) { sel_w = p; sel_e = int(e); }
  }
  if (lane < k) {
    out_idx[lane] = sel_e;
    out_w[lane] = sel_w / wsum;
    if (counts && unsigned(sel_e) < unsigned(E)) atomicAdd(counts + sel_e, 1);
  }
}

__device__ __forceinline__ void warp_topk(const float* logits, const float* bias, int E, int k, int* out_idx, float* out_w, int* counts) {
  if (E <= 32) warp_topk_v<1>(logits, bias, E, k, out_idx, out_w, counts);
  else if (E <= 128) warp_topk_v<4>(logits, bias, E, k, out_idx, out_w, counts);
  else warp_topk_v<kMaxExperts / 32>(logits, bias, E, k, out_idx, out_w, counts);
}

// One to four rows, where many blocks read the weights faster than one cluster (rule at the launch).
template <int B>
__global__ void __launch_bounds__(kGemvThreads)
moe_router_few_kernel(const __nv_bfloat16* __restrict__ gate_w, const __nv_bfloat16* __restrict__ x,
                  int x_stride, const __nv_bfloat16* __restrict__ norm_w, float eps,
                  const float* __restrict__ expert_bias, float* __restrict__ logits,
                  int* __restrict__ topk_idx, float* __restrict__ topk_w, int* __restrict__ counts,
                  unsigned int* __restrict__ ticket, int E, int K, int k) {
  // One block per expert row; the eight warps split K, so every lane has all of its weight bytes
  // in flight at once (a 4096-wide row is 2 x 16 bytes per lane) and the whole machine takes part.
  extern __shared__ __align__(16) char smem[];
  __shared__ float red[kGemvWarps];
  __shared__ float inv_rms[B];
  __shared__ float part[kGemvWarps][B];
  __shared__ unsigned int last;
  const size_t bstride = (XStage<WBf16>::bytes(K) + 15) & ~size_t(15);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nchunk = K >> 3;
  const int per_warp = (nchunk + kGemvWarps - 1) / kGemvWarps;
  for (int e = blockIdx.x; e < E; e += gridDim.x) {
    const __nv_bfloat16* wrow = gate_w + size_t(e) * K;
    // this warp's slice of the row: chunks [c_lo, c_hi)
    const int c_lo = warp * per_warp, c_hi = min(nchunk, c_lo + per_warp);
    uint4 wv[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int c = c_lo + u * 32 + lane;
      wv[u] = (c < c_hi) ? ldg_stream(wrow + (size_t(c) << 3)) : make_uint4(0, 0, 0, 0);
    }
    if (e == blockIdx.x) {
      pdl_launch_dependents();   // let the next kernel start its weight prefetch now; its own wait covers our completion
      pdl_wait();
#pragma unroll
      for (int b = 0; b < B; ++b) {
        const float ssq = XStage<WBf16>::stage(smem + b * bstride, x + size_t(b) * x_stride, norm_w,
                                               K, red, norm_w != nullptr);
        if (threadIdx.x == 0) inv_rms[b] = norm_w ? rsqrtf(ssq / float(K) + eps) : 1.f;
      }
      __syncthreads();
    }
    float acc[B];
#pragma unroll
    for (int b = 0; b < B; ++b) acc[b] = 0.f;
    for (int c0 = c_lo; c0 < c_hi; c0 += 128) {
      if (c0 != c_lo) {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int c = c0 + u * 32 + lane;
          wv[u] = (c < c_hi) ? ldg_stream(wrow + (size_t(c) << 3)) : make_uint4(0, 0, 0, 0);
        }
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int c = c0 + u * 32 + lane;
        if (c < c_hi) {
#pragma unroll
          for (int b = 0; b < B; ++b) {
            const float4* xs = reinterpret_cast<const float4*>(smem + b * bstride);
            const float4 x0 = xs[c], x1 = xs[nchunk + c];
            float a = acc[b];
            a = fmaf(bf16lo(wv[u].x), x0.x, a); a = fmaf(bf16hi(wv[u].x), x0.y, a);
            a = fmaf(bf16lo(wv[u].y), x0.z, a); a = fmaf(bf16hi(wv[u].y), x0.w, a);
            a = fmaf(bf16lo(wv[u].z), x1.x, a); a = fmaf(bf16hi(wv[u].z), x1.y, a);
            a = fmaf(bf16lo(wv[u].w), x1.z, a); a = fmaf(bf16hi(wv[u].w), x1.w, a);
            acc[b] = a;
          }
        }
      }
    }
#pragma unroll
    for (int b = 0; b < B; ++b) {
      const float v = warp_sum(acc[b]);
      if (lane == 0) part[warp][b] = v;
    }
    __syncthreads();
    if (threadIdx.x < B) {
      float v = 0.f;
#pragma unroll
      for (int w = 0; w < kGemvWarps; ++w) v += part[w][threadIdx.x];
      logits[size_t(threadIdx.x) * E + e] = v * inv_rms[threadIdx.x];
    }
    __syncthreads();
  }
  // Last block to arrive selects the experts for every token of this launch.
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = (atomicAdd(ticket, 1u) == gridDim.x - 1) ? 1u : 0u;
  __syncthreads();
  if (last) {
    __threadfence();
    for (int b = warp; b < B; b += kGemvWarps)
      warp_topk(logits + size_t(b) * E, expert_bias, E, k, topk_idx + size_t(b) * k,
                topk_w + size_t(b) * k, counts);
    if (threadIdx.x == 0) *ticket = 0u;  // ready for the next launch (graph replay included)
  }
  pdl_launch_dependents();
}

// The router of any number of rows: a cluster of 8 or 16 blocks per eight rows takes K apart, every warp 32 values at a time for all
// experts, 16 of them and eight rows to an instruction (mma m16n8k16; both operands come straight from global memory: a lane's 16
// bytes of a row of W, and the same values of x, are its operands of two instructions, the order of K being free). The sums of the
// warps, then of the blocks, meet in shared memory, and block r selects the experts of row r.
//
// Nothing is rounded on the way to the fp32 sums: x * g is a product of two bf16 numbers and has 16 bits, so a bf16 number and
// another bf16 remainder hold all of it; each instruction adds 16 products to zero and the sums between instructions are fp32
// additions. (Root mean square error of the logits of 128 experts of 4096, 64 rows, against 64 bits: 2.6e-8 of the largest; one fused
// multiply-add per product, as in the kernel above, 3.2e-8.)
//
// Bound by latency: 1 MB of weights (128 x 4096), of which a warp requests its first 32 columns before it waits for the rows, then two
// meetings of the warps and the selection. 128 x 4096, us: 5.7 for 8 rows (19 in two passes of the kernel above, whose every block
// stages all rows in fp32), 7.4 for 64 (26 as norm, GEMM and selection); 32 x 2048: 4.7 and 5.2 (14 and 19).
constexpr int kRtWarps = 8, kRtThreads = 32 * kRtWarps, kRtRows = 8, kRtTiles = 8, kRtGroup = 16 * kRtTiles, kRtPad = kRtGroup + 4;
constexpr int kRtMaxCluster = 16;

__device__ __forceinline__ void rt_mma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}
__device__ __forceinline__ float rt_remote(uint32_t addr, int rank) {
  float v;
  asm volatile("{.reg .u32 a; mapa.shared::cluster.u32 a, %1, %2; ld.shared::cluster.f32 %0, [a];}" : "=f"(v) : "r"(addr), "r"(rank) : "memory");
  return v;
}

template <int CS>
__global__ void __launch_bounds__(kRtThreads, 2)
moe_router_kernel(const __nv_bfloat16* __restrict__ gate_w, const __nv_bfloat16* __restrict__ x, int x_stride,
                  const __nv_bfloat16* __restrict__ norm_w, float eps, const float* __restrict__ expert_bias,
                  float* __restrict__ logits, int* __restrict__ topk_idx, float* __restrict__ topk_w, int* __restrict__ counts, int B,
                  int E, int K, int k) {
  __shared__ float red[kRtWarps][kRtRows][kRtPad];
  __shared__ float part[kRtRows][kMaxExperts];           // the block's sums, read by the cluster
  __shared__ float squares[kRtWarps][kRtRows], square[kRtRows];
  __shared__ float row_logits[kMaxExperts];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  int rank;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  const int row0 = blockIdx.x / CS * kRtRows, chunks = (K + 31) >> 5, chunk0 = rank * kRtWarps + warp;
  const __nv_bfloat16* const xr = x + size_t(min(row0 + g, B - 1)) * x_stride;
  const bool have = row0 + g < B;

  uint4 w[2 * kRtTiles];
  auto load_w = [&](int e0, int chunk) {
    const int c = chunk * 32 + t * 8;
#pragma unroll
    for (int j = 0; j < 2 * kRtTiles; ++j) {
      const int e = e0 + (j >> 1) * 16 + (j & 1) * 8 + g;
      w[j] = e < E && c < K ? ldg_stream(gate_w + size_t(e) * K + c) : make_uint4(0, 0, 0, 0);
    }
  };
  load_w(0, chunk0);
  pdl_launch_dependents();   // let the next kernel start its weight prefetch now; its own wait covers our completion
  pdl_wait();

  float ssq = 0.f;
  for (int e0 = 0; e0 < E; e0 += kRtGroup) {
    float acc[kRtTiles][4];
#pragma unroll
    for (int j = 0; j < kRtTiles; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f;
    for (int chunk = chunk0; chunk < chunks; chunk += CS * kRtWarps) {
      const int c = chunk * 32 + t * 8;
      const uint4 none = make_uint4(0, 0, 0, 0);
      const uint4 xv = have && c < K ? __ldcg(reinterpret_cast<const uint4*>(xr + c)) : none;
      const uint4 gv = norm_w && c < K ? *reinterpret_cast<const uint4*>(norm_w + c) : none;
      if (e0 != 0 || chunk != chunk0) load_w(e0, chunk);
      const uint32_t xs[4] = {xv.x, xv.y, xv.z, xv.w}, gs[4] = {gv.x, gv.y, gv.z, gv.w};
      uint32_t hi[4], lo[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float a = bf16lo(xs[i]), b = bf16hi(xs[i]);
        if (e0 == 0) ssq += a * a + b * b;
        hi[i] = xs[i]; lo[i] = 0;
        if (norm_w) {
          a *= bf16lo(gs[i]); b *= bf16hi(gs[i]);
          hi[i] = pack_bf16(a, b);
          // an infinite product has no remainder
          const float ra = a - bf16lo(hi[i]), rb = b - bf16hi(hi[i]);
          lo[i] = pack_bf16(isfinite(ra) ? ra : 0.f, isfinite(rb) ? rb : 0.f);
        }
      }
#pragma unroll
      for (int j = 0; j < kRtTiles; ++j) {
        if (e0 + j * 16 >= E) break;
        const uint4 p = w[2 * j], q = w[2 * j + 1];
        float d[4], f[4];
        rt_mma(d, p.x, q.x, p.y, q.y, hi[0], hi[1]);
        rt_mma(f, p.z, q.z, p.w, q.w, hi[2], hi[3]);
        if (norm_w) {
          float u[4], v[4];
          rt_mma(u, p.x, q.x, p.y, q.y, lo[0], lo[1]);
          rt_mma(v, p.z, q.z, p.w, q.w, lo[2], lo[3]);
#pragma unroll
          for (int i = 0; i < 4; ++i) { d[i] += u[i]; f[i] += v[i]; }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[j][i] += d[i] + f[i];
      }
    }
#pragma unroll
    for (int j = 0; j < kRtTiles; ++j) {
      red[warp][2 * t][j * 16 + g] = acc[j][0]; red[warp][2 * t + 1][j * 16 + g] = acc[j][1];
      red[warp][2 * t][j * 16 + 8 + g] = acc[j][2]; red[warp][2 * t + 1][j * 16 + 8 + g] = acc[j][3];
    }
    if (e0 == 0) {
      ssq += __shfl_xor_sync(0xffffffffu, ssq, 1);
      ssq += __shfl_xor_sync(0xffffffffu, ssq, 2);
      if (t == 0) squares[warp][g] = ssq;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kRtRows * kRtGroup / kRtThreads; ++i) {
      const int at = i * kRtThreads + threadIdx.x, r = at / kRtGroup, e = at % kRtGroup;
      float v[kRtWarps];
#pragma unroll
      for (int j = 0; j < kRtWarps; ++j) v[j] = red[j][r][e];
      part[r][e0 + e] = ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7]));
    }
    if (e0 == 0 && threadIdx.x < kRtRows) {
      float v = 0.f;
#pragma unroll
      for (int j = 0; j < kRtWarps; ++j) v += squares[j][threadIdx.x];
      square[threadIdx.x] = v;
    }
    if (e0 + kRtGroup < E) __syncthreads();
  }

  // block r: row r
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  const int row = row0 + rank;
  const bool mine = rank < kRtRows && row < B;
  if (mine) {
    const float sq = lane < CS ? rt_remote(smem_u32(&square[rank]), lane) : 0.f;
    const int e = threadIdx.x;
    float v[CS];
    if (e < E) {
#pragma unroll
      for (int j = 0; j < CS; ++j) v[j] = rt_remote(smem_u32(&part[rank][e]), j);
    }
    const float inv_rms = norm_w ? rsqrtf(warp_sum(sq) / float(K) + eps) : 1.f;
    if (e < E) {
#pragma unroll
      for (int o = CS / 2; o > 0; o >>= 1)
#pragma unroll
        for (int j = 0; j < o; ++j) v[j] += v[j + o];
      const float l = v[0] * inv_rms;
      row_logits[e] = l;
      if (logits) logits[size_t(row) * E + e] = l;
    }
  }
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  if (mine) {
    __syncthreads();
    if (warp == 0) warp_topk(row_logits, expert_bias, E, k, topk_idx + size_t(row) * k, topk_w + size_t(row) * k, counts);
  }
  __syncwarp();
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");   // nobody leaves while its sums are read
}

__global__ void __launch_bounds__(256)
topk_route_kernel(const float* __restrict__ logits, const float* __restrict__ expert_bias,
                  int* __restrict__ topk_idx, float* __restrict__ topk_w, int* __restrict__ counts,
                  int T, int E, int k) {
  const int t = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (t < T)
    warp_topk(logits + size_t(t) * E, expert_bias, E, k, topk_idx + size_t(t) * k,
              topk_w + size_t(t) * k, counts);
}

// offsets[e] = sum_{j<e} counts[j], offsets[E] = total. One warp.
__global__ void moe_prefix_offsets_kernel(const int* __restrict__ counts, int* __restrict__ offsets,
                                          int E) {
  const int lane = threadIdx.x;
  int carry = 0;
  for (int base = 0; base < E; base += 32) {
    const int e = base + lane;
    const int c = (e < E) ? counts[e] : 0;
    int inc = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int n = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += n;
    }
    if (e < E) offsets[e] = carry + inc - c;
    carry += __shfl_sync(0xffffffffu, inc, 31);
  }
  if (lane == 0) offsets[E] = carry;
}

// Stacked expert matrices [E, rows, K].
template <class WT>
struct ExpertMatrix;
template <>
struct ExpertMatrix<WBf16> {
  using Row = RowBf16;
  const __nv_bfloat16* w;
  int rows, K;
  __device__ Row row(int e, size_t n) const { return Row{w + (size_t(e) * rows + n) * size_t(K)}; }
};
template <>
struct ExpertMatrix<WQ4> {
  using Row = RowQ4;
  const uint32_t* w;
  const __nv_bfloat16* scales;
  const __nv_bfloat16* biases;
  int rows, K;
  __device__ Row row(int e, size_t n) const {
    const size_t r = size_t(e) * rows + n;
    return Row{w + r * size_t(K >> 3), scales + r * size_t(K >> 6), biases + r * size_t(K >> 6)};
  }
};

constexpr int kRowsPerWarpDown = 2;
constexpr int kGuPairsPerWarp = 2;  // (gate, up) row pairs in flight per warp

// grid = (row blocks, token*slot pairs). `i_begin`/`i_count` select a slice of the intermediate
// dimension (tensor-parallel shards own a slice of every expert).
template <class WT>
__global__ void __launch_bounds__(kGemvThreads, 2)
moe_gate_up_kernel(ExpertMatrix<WT> W /*rows = 2*I_full: gate then up*/,
                   const __nv_bfloat16* __restrict__ x, int x_stride,
                   const __nv_bfloat16* __restrict__ norm_w, float eps,
                   const int* __restrict__ topk_idx, __nv_bfloat16* __restrict__ act,
                   int act_stride, int I, int top_k, int expert_base, int experts_local) {
  extern __shared__ __align__(16) char smem[];
  __shared__ float red[kGemvWarps];
  __shared__ float inv_rms_s;
  const int K = W.K;
  const int pair = blockIdx.y, b = pair / top_k;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  pdl_launch_dependents();   // let the next kernel start its weight prefetch now; its own wait covers our completion
  pdl_wait();
  const int e = topk_idx[pair] - expert_base;
  if (e < 0 || e >= experts_local) return;  // expert lives on another rank
  using Row = typename ExpertMatrix<WT>::Row;
  constexpr int R = 2 * kGuPairsPerWarp;
  int i0 = (blockIdx.x * kGemvWarps + warp) * kGuPairsPerWarp;
  Row rows[R];
  Tile<Row, R> t0;
  auto set_rows = [&](int base) {
#pragma unroll
    for (int j = 0; j < kGuPairsPerWarp; ++j) {
      const int i = min(base + j, I - 1);
      rows[2 * j] = W.row(e, i);
      rows[2 * j + 1] = W.row(e, size_t(I) + i);
    }
  };
  if (i0 < I) { set_rows(i0); load_tile<R>(rows, K, 0, t0); }  // in flight during the staging
  const float ssq = XStage<WT>::stage(smem, x + size_t(b) * x_stride, norm_w, K, red,
                                      norm_w != nullptr);
  if (threadIdx.x == 0) inv_rms_s = norm_w ? rsqrtf(ssq / float(K) + eps) : 1.f;
  __syncthreads();
  const float inv_rms = inv_rms_s;
  for (bool first = true; i0 < I; i0 += gridDim.x * kGemvWarps * kGuPairsPerWarp, first = false) {
    if (!first) { set_rows(i0); load_tile<R>(rows, K, 0, t0); }
    float acc[R][1];
#pragma unroll
    for (int j = 0; j < R; ++j) acc[j][0] = 0.f;
    warp_dot<R, 1, Row>(rows, smem, 0, K, acc, t0);
#pragma unroll
    for (int j = 0; j < kGuPairsPerWarp; ++j) {
      const float g = warp_sum(acc[2 * j][0]) * inv_rms;
      const float u = warp_sum(acc[2 * j + 1][0]) * inv_rms;
      if (lane == j && i0 + j < I)
        act[size_t(pair) * act_stride + i0 + j] = __float2bfloat16_rn(g / (1.f + __expf(-g)) * u);
    }
  }
  pdl_launch_dependents();
}

// grid = (row blocks, tokens). Stages the token's top_k activation vectors, then every output row
// accumulates over the slots with the routing weight applied per slot. Slots whose expert is not
// local contribute nothing (the cross-rank sum happens in the caller's all-reduce).
template <class WT, bool OUT_F32>
__global__ void __launch_bounds__(kGemvThreads, 2)     // two blocks per SM: keeps more weight loads in flight
moe_down_kernel(ExpertMatrix<WT> W /*rows = N, K = I*/, const __nv_bfloat16* __restrict__ act,
                int act_stride, const int* __restrict__ topk_idx, const float* __restrict__ topk_w,
                const __nv_bfloat16* __restrict__ residual, int res_stride, void* __restrict__ out,
                int out_stride, int N, int top_k, int expert_base, int experts_local) {
  extern __shared__ __align__(16) char smem[];
  __shared__ int s_e[kMaxTopK];
  __shared__ float s_w[kMaxTopK];
  const int I = W.K;
  const size_t bstride = (XStage<WT>::bytes(I) + 15) & ~size_t(15);
  const int b = blockIdx.y;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  pdl_launch_dependents();   // let the next kernel start its weight prefetch now; its own wait covers our completion
  pdl_wait();
  if (threadIdx.x < top_k) {
    const int e = topk_idx[b * top_k + threadIdx.x] - expert_base;
    const bool local = e >= 0 && e < experts_local;
    s_e[threadIdx.x] = local ? e : -1;
    s_w[threadIdx.x] = local ? topk_w[b * top_k + threadIdx.x] : 0.f;
  }
  __syncthreads();
  using Row = typename ExpertMatrix<WT>::Row;
  constexpr int R = kRowsPerWarpDown;
  auto next_local = [&](int s) { while (s < top_k && s_e[s] < 0) ++s; return s; };
  int n0 = (blockIdx.x * kGemvWarps + warp) * R;
  const int s_first = next_local(0);
  Row rows[R];
  Tile<Row, R> cur;
  if (n0 < N && s_first < top_k) {  // first slot's weights fly while the activations are staged
#pragma unroll
    for (int r = 0; r < R; ++r) rows[r] = W.row(s_e[s_first], min(n0 + r, N - 1));
    load_tile<R>(rows, I, 0, cur);
  }
  for (int s = 0; s < top_k; ++s) {
    if (s_e[s] >= 0)
      XStage<WT>::stage(smem + s * bstride, act + size_t(b * top_k + s) * act_stride, nullptr, I,
                        nullptr, false);
  }
  __syncthreads();
  const int units = row_units(rows[0], I);
  for (bool first = true; n0 < N; n0 += gridDim.x * kGemvWarps * R, first = false) {
    float tot[R];
#pragma unroll
    for (int r = 0; r < R; ++r) tot[r] = 0.f;
    int s = s_first;
    if (!first && s < top_k) {
#pragma unroll
      for (int r = 0; r < R; ++r) rows[r] = W.row(s_e[s], min(n0 + r, N - 1));
      load_tile<R>(rows, I, 0, cur);
    }
    while (s < top_k) {
      // software pipeline over the slots: the next expert's first tile is requested before the
      // current one is consumed
      const int sn = next_local(s + 1);
      Row rows_n[R];
      Tile<Row, R> nxt;
      if (sn < top_k) {
#pragma unroll
        for (int r = 0; r < R; ++r) rows_n[r] = W.row(s_e[sn], min(n0 + r, N - 1));
        load_tile<R>(rows_n, I, 0, nxt);
      }
      float acc[R][1];
#pragma unroll
      for (int r = 0; r < R; ++r) acc[r][0] = 0.f;
      if (units <= 64) fma_tile<R, 1>(cur, 0, smem + s * bstride, 0, I, acc);
      else warp_dot<R, 1, Row>(rows, smem + s * bstride, 0, I, acc, cur);
      const float w = s_w[s];
#pragma unroll
      for (int r = 0; r < R; ++r) tot[r] = fmaf(w, acc[r][0], tot[r]);
      if (sn < top_k) {
        cur = nxt;
#pragma unroll
        for (int r = 0; r < R; ++r) rows[r] = rows_n[r];
      }
      s = sn;
    }
#pragma unroll
    for (int r = 0; r < kRowsPerWarpDown; ++r) {
      const float v = warp_sum(tot[r]);
      if (lane == r && n0 + r < N) {
        float o = v;
        if (residual) o += __bfloat162float(residual[size_t(b) * res_stride + n0 + r]);
        if (OUT_F32) reinterpret_cast<float*>(out)[size_t(b) * out_stride + n0 + r] = o;
        else reinterpret_cast<__nv_bfloat16*>(out)[size_t(b) * out_stride + n0 + r] =
                 __float2bfloat16_rn(o);
      }
    }
  }
  pdl_launch_dependents();
}

// Slot-parallel form of the expert down projection: warp s of a block takes routing slot s (its own
// expert), stages that slot's activation by itself and multiplies the block's kDownRows output rows;
// the block then adds the weighted partial sums of its warps. All experts' weight loads of a row
// set are in flight at once (the sequential form above walks the slots one after the other, which
// is the better shape only when a row is long enough to keep a warp busy).
constexpr int kDownRows = 4;

template <class WT, bool OUT_F32>
__global__ void __launch_bounds__(kGemvThreads, 2)
moe_down_par_kernel(ExpertMatrix<WT> W /*rows = N, K = I*/, const __nv_bfloat16* __restrict__ act,
                    int act_stride, const int* __restrict__ topk_idx, const float* __restrict__ topk_w,
                    const __nv_bfloat16* __restrict__ residual, int res_stride, void* __restrict__ out,
                    int out_stride, int N, int top_k, int expert_base, int experts_local) {
  extern __shared__ __align__(16) char smem[];
  __shared__ float s_part[kGemvWarps][kDownRows];
  const int I = W.K;
  const size_t bstride = (XStage<WT>::bytes(I) + 15) & ~size_t(15);
  const int b = blockIdx.y;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  using Row = typename ExpertMatrix<WT>::Row;
  pdl_launch_dependents();
  pdl_wait();
  float tot[kDownRows];
#pragma unroll
  for (int r = 0; r < kDownRows; ++r) tot[r] = 0.f;
  const int n0 = blockIdx.x * kDownRows;
  for (int s = warp; s < top_k; s += kGemvWarps) {      // top_k <= 8: one slot per warp
    const int e = topk_idx[b * top_k + s] - expert_base;
    if (e < 0 || e >= experts_local) continue;
    Row rows[kDownRows];
    Tile<Row, kDownRows> t0;
#pragma unroll
    for (int r = 0; r < kDownRows; ++r) rows[r] = W.row(e, min(n0 + r, N - 1));
    load_tile<kDownRows>(rows, I, 0, t0);               // in flight while the activation is staged
    XLoadBf16 ld{act + size_t(b * top_k + s) * act_stride, nullptr, 0.f};
    char* xs = smem + warp * bstride;
    XStage<WT>::stage_warp(xs, I, ld);
    float acc[kDownRows][1];
#pragma unroll
    for (int r = 0; r < kDownRows; ++r) acc[r][0] = 0.f;
    warp_dot<kDownRows, 1, Row>(rows, xs, 0, I, acc, t0);
    const float w = topk_w[b * top_k + s];
#pragma unroll
    for (int r = 0; r < kDownRows; ++r) tot[r] = fmaf(w, acc[r][0], tot[r]);
    __syncwarp();                                       // the staged vector is reused by the next slot
  }
#pragma unroll
  for (int r = 0; r < kDownRows; ++r) {
    const float v = warp_sum(tot[r]);
    if (lane == 0) s_part[warp][r] = v;
  }
  __syncthreads();
  if (threadIdx.x < kDownRows && n0 + threadIdx.x < N) {
    const int r = threadIdx.x;
    float o = 0.f;
#pragma unroll
    for (int w = 0; w < kGemvWarps; ++w) o += s_part[w][r];
    if (residual) o += __bfloat162float(residual[size_t(b) * res_stride + n0 + r]);
    if (OUT_F32) reinterpret_cast<float*>(out)[size_t(b) * out_stride + n0 + r] = o;
    else reinterpret_cast<__nv_bfloat16*>(out)[size_t(b) * out_stride + n0 + r] = __float2bfloat16_rn(o);
  }
}

template <class WT>
static ExpertMatrix<WT> make_expert_matrix(const void* w, const void* s, const void* b, int rows,
                                           int K);
template <>
ExpertMatrix<WBf16> make_expert_matrix<WBf16>(const void* w, const void*, const void*, int rows,
                                              int K) {
  return ExpertMatrix<WBf16>{static_cast<const __nv_bfloat16*>(w), rows, K};
}
template <>
ExpertMatrix<WQ4> make_expert_matrix<WQ4>(const void* w, const void* s, const void* b, int rows,
                                          int K) {
  return ExpertMatrix<WQ4>{static_cast<const uint32_t*>(w), static_cast<const __nv_bfloat16*>(s),
                           static_cast<const __nv_bfloat16*>(b), rows, K};
}

template <class WT>
static int launch_moe_gate_up(const void* w, const void* sc, const void* bi, const void* x,
                              int x_stride, const void* norm_w, float eps, const int* idx, void* act,
                              int act_stride, int B, int top_k, int I, int K, int expert_base,
                              int experts_local, int pdl, cudaStream_t st) {
  const size_t smem = (XStage<WT>::bytes(K) + 15) & ~size_t(15);
  auto kern = moe_gate_up_kernel<WT>;
  RB_CHECK(set_max_smem(kern, smem));
  int gx = (I + kGemvWarps * kGuPairsPerWarp - 1) / (kGemvWarps * kGuPairsPerWarp);
  if (gx < 1) gx = 1;
  return launch(kern, dim3(gx, B * top_k), dim3(kGemvThreads), smem, st, pdl != 0,
                make_expert_matrix<WT>(w, sc, bi, 2 * I, K), static_cast<const __nv_bfloat16*>(x),
                x_stride, static_cast<const __nv_bfloat16*>(norm_w), eps, idx,
                static_cast<__nv_bfloat16*>(act), act_stride, I, top_k, expert_base, experts_local);
}

// RMLX_MOE_DOWN=par selects the slot-parallel kernel. Default is the sequential-slot kernel: with
// its one-expert-ahead prefetch it measures the same or slightly better at full-width rows.
static bool moe_down_parallel_slots() {
  static const bool v = [] {
    const char* e = getenv("RMLX_MOE_DOWN");
    return e && e[0] == 'p';
  }();
  return v;
}

template <class WT, bool OUT_F32>
static int launch_moe_down(const void* w, const void* sc, const void* bi, const void* act,
                           int act_stride, const int* idx, const float* tw, const void* res,
                           int res_stride, void* out, int out_stride, int B, int top_k, int N, int I,
                           int expert_base, int experts_local, int pdl, cudaStream_t st) {
  if (moe_down_parallel_slots()) {
    const size_t psmem = ((XStage<WT>::bytes(I) + 15) & ~size_t(15)) * kGemvWarps;
    auto pk = moe_down_par_kernel<WT, OUT_F32>;
    RB_CHECK(set_max_smem(pk, psmem));
    return launch(pk, dim3((N + kDownRows - 1) / kDownRows, B), dim3(kGemvThreads), psmem, st, pdl != 0,
                  make_expert_matrix<WT>(w, sc, bi, N, I), static_cast<const __nv_bfloat16*>(act),
                  act_stride, idx, tw, static_cast<const __nv_bfloat16*>(res), res_stride, out,
                  out_stride, N, top_k, expert_base, experts_local);
  }
  const size_t smem = ((XStage<WT>::bytes(I) + 15) & ~size_t(15)) * top_k;
  auto kern = moe_down_kernel<WT, OUT_F32>;
  RB_CHECK(set_max_smem(kern, smem));
  int gx = (N + kGemvWarps * kRowsPerWarpDown - 1) / (kGemvWarps * kRowsPerWarpDown);
  const int cap = sm_count() * 4;
  if (gx > cap) gx = cap;
  return launch(kern, dim3(gx, B), dim3(kGemvThreads), smem, st, pdl != 0,
                make_expert_matrix<WT>(w, sc, bi, N, I), static_cast<const __nv_bfloat16*>(act),
                act_stride, idx, tw, static_cast<const __nv_bfloat16*>(res), res_stride, out,
                out_stride, N, top_k, expert_base, experts_local);
}

}  // namespace rb

using namespace rb;

template <int B>
static int launch_router_few(const void* gate_w, const void* x, int x_stride, const void* norm_w, float eps, const float* expert_bias,
                             float* logits, int* topk_idx, float* topk_w, int* counts, unsigned int* ticket, int E, int K, int k, int pdl,
                             cudaStream_t st) {
  const size_t smem = ((XStage<WBf16>::bytes(K) + 15) & ~size_t(15)) * B;
  auto kern = moe_router_few_kernel<B>;
  RB_CHECK(set_max_smem(kern, smem));
  return launch(kern, dim3(E), dim3(kGemvThreads), smem, st, pdl != 0, static_cast<const __nv_bfloat16*>(gate_w),
                static_cast<const __nv_bfloat16*>(x), x_stride, static_cast<const __nv_bfloat16*>(norm_w), eps, expert_bias, logits, topk_idx,
                topk_w, counts, ticket, E, K, k);
}

// Scratch: `logits` fp32 [B, E] and `ticket` one zero-initialised uint32 (left at zero on return); either may be null, few rows then
// take the cluster too. counts may be null; when given it must be zeroed by the caller and receives the histogram. x's rows, norm_w and gate_w at 16-byte
// addresses.
extern "C" int rmlx_moe_router(const void* gate_w, const void* x, int x_stride, const void* norm_w, float eps, const float* expert_bias,
                               float* logits, int* topk_idx, float* topk_w, int* counts, unsigned int* ticket, int B, int E, int K, int k,
                               int pdl, cudaStream_t st) {
  if (E > kMaxExperts || k > kMaxTopK || k > E || K % 8 || B < 1) return -2;
  // One row, and up to four where the cluster goes over the rows twice: a block per expert (us, blocks / cluster: 128 x 4096 4.6 / 5.0
  // for one row, 5.6 / 5.2 for two; 256 x 4096 6.5 / 9.8 for two, 8.7 / 9.7 for four; 256 x 7168 12 / 19 for four, 25 / 20 for eight,
  // which are two passes of blocks)
  if (logits && ticket && (B == 1 || (B <= 4 && E > kRtGroup))) {
#define RB_ROUTER(BB) return launch_router_few<BB>(gate_w, x, x_stride, norm_w, eps, expert_bias, logits, topk_idx, topk_w, counts, ticket, E, \
                                                   K, k, pdl, st)
    switch (B) {
      case 1: RB_ROUTER(1);
      case 2: RB_ROUTER(2);
      case 3: RB_ROUTER(3);
      default: RB_ROUTER(4);
    }
#undef RB_ROUTER
  }
  // sixteen blocks for rows of more than 2048: one 32-value step per warp at 4096
  const int cs = K > 2048 ? 16 : 8;
  auto kern = cs == 16 ? moe_router_kernel<16> : moe_router_kernel<8>;
  if (cs > 8) RB_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((B + kRtRows - 1) / kRtRows * cs);
  cfg.blockDim = dim3(kRtThreads);
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cs; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl ? 2 : 1;
  if (pdl) prefer_max_shared(kern);
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, static_cast<const __nv_bfloat16*>(gate_w), static_cast<const __nv_bfloat16*>(x), x_stride,
                                           static_cast<const __nv_bfloat16*>(norm_w), eps, expert_bias, logits, topk_idx, topk_w, counts, B, E,
                                           K, k);
  if (e != cudaSuccess) (void)cudaGetLastError();
  return static_cast<int>(e);
}

extern "C" int rmlx_topk_route(const float* logits, const float* expert_bias, int* topk_idx,
                               float* topk_w, int* counts, int* offsets, int T, int E, int k,
                               cudaStream_t st) {
  if (E > kMaxExperts || k > kMaxTopK || k > E || T < 1) return -2;
  if (counts) RB_CHECK(cudaMemsetAsync(counts, 0, sizeof(int) * E, st));
  topk_route_kernel<<<(T + 7) / 8, 256, 0, st>>>(logits, expert_bias, topk_idx, topk_w, counts, T, E, k);
  if (counts && offsets) moe_prefix_offsets_kernel<<<1, 32, 0, st>>>(counts, offsets, E);
  return static_cast<int>(cudaGetLastError());
}

extern "C" int rmlx_moe_gate_up(int w_kind, const void* w, const void* scales, const void* biases,
                                const void* x, int x_stride, const void* norm_w, float eps,
                                const int* topk_idx, void* act, int act_stride, int B, int top_k,
                                int I, int K, int expert_base, int experts_local, int pdl,
                                cudaStream_t st) {
  if (K % 8 || (w_kind == 1 && K % 64) || B < 1 || top_k < 1 || top_k > kMaxTopK) return -2;
  if (w_kind == 0)
    return launch_moe_gate_up<WBf16>(w, scales, biases, x, x_stride, norm_w, eps, topk_idx, act,
                                     act_stride, B, top_k, I, K, expert_base, experts_local, pdl, st);
  if (w_kind == 1)
    return launch_moe_gate_up<WQ4>(w, scales, biases, x, x_stride, norm_w, eps, topk_idx, act,
                                   act_stride, B, top_k, I, K, expert_base, experts_local, pdl, st);
  return -2;
}

extern "C" int rmlx_moe_down(int w_kind, const void* w, const void* scales, const void* biases,
                             const void* act, int act_stride, const int* topk_idx,
                             const float* topk_w, const void* residual, int res_stride, void* out,
                             int out_stride, int out_f32, int B, int top_k, int N, int I,
                             int expert_base, int experts_local, int pdl, cudaStream_t st) {
  if (I % 8 || (w_kind == 1 && I % 64) || B < 1 || top_k < 1 || top_k > kMaxTopK) return -2;
#define RB_DOWN(WT, F32)                                                                         \
  return launch_moe_down<WT, F32>(w, scales, biases, act, act_stride, topk_idx, topk_w, residual, \
                                  res_stride, out, out_stride, B, top_k, N, I, expert_base,      \
                                  experts_local, pdl, st)
  if (w_kind == 0) { if (out_f32) RB_DOWN(WBf16, true); else RB_DOWN(WBf16, false); }
  if (w_kind == 1) { if (out_f32) RB_DOWN(WQ4, true); else RB_DOWN(WQ4, false); }
#undef RB_DOWN
  return -2;
}
