// RoPE on Q and K plus the paged KV-cache append, one launch for every head of every token.
//
// Input is the merged QKV projection output [T, (Hq + 2*Hkv) * HD], bf16 or fp32 (decode rows: the
// projection's sums reach the rotation unrounded and are rounded once, after it). Q heads are rotated and
// written to q_out; K heads are rotated and written straight into their page slot; V heads are
// copied into theirs. Positions, block tables and the token->sequence map are device buffers, so
// the launch is shape-stable under CUDA graph replay while the cache grows.
//
// Replaces rope_qk(v)_batch_* + kv_cache_copy_batched_* (crates/rmlx-core/src/ops/rope.rs:500-870,
// crates/rmlx-core/src/ops/copy.rs:554) and PagedKvCache::append's host memcpy
// (crates/rmlx-nn/src/paged_kv_cache.rs:413-458).
// Rotation layouts: split-half (pairs i, i+HD/2; default) or traditional (pairs 2i, 2i+1), with
// cos/sin tables [max_pos, HD/2] as in crates/rmlx-core/src/ops/rope.rs:15-60.
#include "../common/ptx.cuh"
#include "../common/launch.cuh"

namespace rb {

__device__ __forceinline__ float rope_value(__nv_bfloat16 v) { return __bfloat162float(v); }
__device__ __forceinline__ float rope_value(float v) { return v; }

template <class T>
__global__ void rope_kv_write_kernel(const T* __restrict__ qkv,
                                     __nv_bfloat16* __restrict__ q_out,
                                     __nv_bfloat16* __restrict__ k_cache,
                                     __nv_bfloat16* __restrict__ v_cache,
                                     const int* __restrict__ block_table,
                                     const int* __restrict__ positions,
                                     const int* __restrict__ token_seq,
                                     const float* __restrict__ cos_t, const float* __restrict__ sin_t,
                                     int Hq, int Hkv, int HD, int max_blocks, int page,
                                     int traditional) {
  const int tkn = blockIdx.x, i = threadIdx.x;  // i in [0, HD/2)
  const int half = HD >> 1;
  pdl_launch_dependents();   // let the next kernel start its weight prefetch now; its own wait covers our completion
  pdl_wait();
  const int pos = positions[tkn];
  const int ia = traditional ? 2 * i : i, ib = traditional ? 2 * i + 1 : i + half;
  const float c = cos_t[size_t(pos) * half + i], s = sin_t[size_t(pos) * half + i];
  // a block takes every gridDim.y-th head of its token (one head each for decode-sized launches,
  // a strip of heads for prompts, where one block per head would be mostly launch overhead)
  for (int head = blockIdx.y; head < Hq + 2 * Hkv; head += gridDim.y) {
    const T* src = qkv + (size_t(tkn) * (Hq + 2 * Hkv) + head) * HD;
    const float a = rope_value(src[ia]), b = rope_value(src[ib]);
    __nv_bfloat16* dst;
    if (head < Hq) {
      dst = q_out + (size_t(tkn) * Hq + head) * HD;
    } else {
      const int seq = token_seq ? token_seq[tkn] : tkn;
      if (!RB_BOUNDS(pos / page, max_blocks)) continue;
      const int blk = block_table[size_t(seq) * max_blocks + pos / page];
      const bool is_k = head < Hq + Hkv;
      const int kvh = is_k ? head - Hq : head - Hq - Hkv;
      dst = (is_k ? k_cache : v_cache) + ((size_t(blk) * Hkv + kvh) * page + pos % page) * HD;
      if (!is_k) { dst[ia] = __float2bfloat16_rn(a); dst[ib] = __float2bfloat16_rn(b); continue; }
    }
    dst[ia] = __float2bfloat16_rn(a * c - b * s);
    dst[ib] = __float2bfloat16_rn(b * c + a * s);
  }
}

// The same in pieces of eight pairs: a thread takes 16 bytes of each half of a head (traditional: 32 bytes in a row), of
// every so many heads of its token, with the eight angles in registers. Bound by memory: 8192 tokens of 48 heads of 128 47 us (79 with one
// pair at a time; 4.0 TB/s), 2048 of 72 heads 15.5 us (28.6).
template <class T> struct RopePiece;                     // eight values
template <> struct RopePiece<__nv_bfloat16> {
  static __device__ __forceinline__ void load(const __nv_bfloat16* p, float (&v)[8]) {
    const uint4 u = *reinterpret_cast<const uint4*>(p);
    const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) { v[2 * i] = bf16lo(w[i]); v[2 * i + 1] = bf16hi(w[i]); }
  }
};
template <> struct RopePiece<float> {
  static __device__ __forceinline__ void load(const float* p, float (&v)[8]) {
    const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
  }
};
__device__ __forceinline__ void rope_store(__nv_bfloat16* p, const float (&v)[8]) {
  *reinterpret_cast<uint4*>(p) = make_uint4(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]), pack_bf16(v[4], v[5]), pack_bf16(v[6], v[7]));
}

template <class T>
__global__ void __launch_bounds__(256)
rope_kv_write_pieces_kernel(const T* __restrict__ qkv, __nv_bfloat16* __restrict__ q_out, __nv_bfloat16* __restrict__ k_cache,
                            __nv_bfloat16* __restrict__ v_cache, const int* __restrict__ block_table, const int* __restrict__ positions,
                            const int* __restrict__ token_seq, const float* __restrict__ cos_t, const float* __restrict__ sin_t, int Hq,
                            int Hkv, int HD, int max_blocks, int page, int traditional) {
  const int tkn = blockIdx.x, half = HD >> 1, pieces = half >> 3, heads = blockDim.x / pieces;
  const int mine = threadIdx.x / pieces, i0 = (threadIdx.x - mine * pieces) * 8, H = Hq + 2 * Hkv;
  pdl_launch_dependents();   // let the next kernel start its weight prefetch now; its own wait covers our completion
  pdl_wait();
  if (mine >= heads) return;
  const int pos = positions[tkn];
  float c[8], s[8];
  RopePiece<float>::load(cos_t + size_t(pos) * half + i0, c);
  RopePiece<float>::load(sin_t + size_t(pos) * half + i0, s);
  const int ia = traditional ? 2 * i0 : i0, ib = traditional ? 2 * i0 + 8 : i0 + half;
  size_t slot = 0;                                       // of the token in the caches, in heads of page x HD
  bool known = false, inside = false;
  for (int head = blockIdx.y * heads + mine; head < H; head += gridDim.y * heads) {
    const T* const src = qkv + (size_t(tkn) * H + head) * HD;
    float a[8], b[8];
    RopePiece<T>::load(src + ia, a);
    RopePiece<T>::load(src + ib, b);
    __nv_bfloat16* dst;
    if (head < Hq) {
      dst = q_out + (size_t(tkn) * Hq + head) * HD;
    } else {
      if (!known) {
        known = true;
        const int pg = pos / page;
        inside = RB_BOUNDS(pg, max_blocks);
        if (inside) slot = (size_t(block_table[size_t(token_seq ? token_seq[tkn] : tkn) * max_blocks + pg]) * Hkv * page + (pos - pg * page)) * HD;
      }
      if (!inside) continue;
      const bool is_k = head < Hq + Hkv;
      dst = (is_k ? k_cache : v_cache) + slot + size_t(is_k ? head - Hq : head - Hq - Hkv) * page * HD;
      if (!is_k) { rope_store(dst + ia, a); rope_store(dst + ib, b); continue; }
    }
    float x[8], y[8];
    if (traditional) {                                   // pairs side by side: a holds the first four, b the others
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        x[2 * i] = a[2 * i] * c[i] - a[2 * i + 1] * s[i]; x[2 * i + 1] = a[2 * i + 1] * c[i] + a[2 * i] * s[i];
        y[2 * i] = b[2 * i] * c[4 + i] - b[2 * i + 1] * s[4 + i]; y[2 * i + 1] = b[2 * i + 1] * c[4 + i] + b[2 * i] * s[4 + i];
      }
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i) { x[i] = a[i] * c[i] - b[i] * s[i]; y[i] = b[i] * c[i] + a[i] * s[i]; }
    }
    rope_store(dst + ia, x);
    rope_store(dst + ib, y);
  }
}

// Stand-alone RoPE over [T, H, HD] (used by tests and by attention variants that keep their own
// cache layout, e.g. latent attention's decoupled rope key).
__global__ void rope_kernel(const __nv_bfloat16* __restrict__ x, __nv_bfloat16* __restrict__ out,
                            const int* __restrict__ positions, const float* __restrict__ cos_t,
                            const float* __restrict__ sin_t, int H, int HD, int traditional,
                            int inverse) {
  const int tkn = blockIdx.x, head = blockIdx.y, i = threadIdx.x;
  const int half = HD >> 1;
  const int pos = positions[tkn];
  const size_t base = (size_t(tkn) * H + head) * HD;
  const int ia = traditional ? 2 * i : i, ib = traditional ? 2 * i + 1 : i + half;
  const float a = __bfloat162float(x[base + ia]), b = __bfloat162float(x[base + ib]);
  const float c = cos_t[size_t(pos) * half + i];
  const float s = inverse ? -sin_t[size_t(pos) * half + i] : sin_t[size_t(pos) * half + i];
  out[base + ia] = __float2bfloat16_rn(a * c - b * s);
  out[base + ib] = __float2bfloat16_rn(b * c + a * s);
}

}  // namespace rb

using namespace rb;
RB_BOUNDS_REGISTER("rope_kv.cu")


template <class T>
static int launch_rope_kv(const void* qkv, void* q_out, void* k_cache, void* v_cache, const int* block_table,
                          const int* positions, const int* token_seq, const float* cos_t, const float* sin_t, int tokens,
                          int Hq, int Hkv, int HD, int max_blocks, int page, int traditional, int pdl, cudaStream_t st) {
  const int H = Hq + 2 * Hkv;
  const uintptr_t all = reinterpret_cast<uintptr_t>(qkv) | reinterpret_cast<uintptr_t>(q_out) | reinterpret_cast<uintptr_t>(k_cache) |
                        reinterpret_cast<uintptr_t>(v_cache) | reinterpret_cast<uintptr_t>(cos_t) | reinterpret_cast<uintptr_t>(sin_t);
  auto kern = rope_kv_write_kernel<T>;
  int threads = HD / 2, gy = tokens >= 128 ? (H + 17) / 18 : H;         // prompts: ~18 heads per block
  // Prompts in whole pieces, up to three a thread. Decode batches keep a block per head: by itself the other kernel is as fast (1.8 us for
  // 8 tokens, 2.2 / 5.4 for 64), but whole steps gain nothing by it (8 rows 868 us / 857, 64 rows 1816 / 1809).
  if (tokens >= 128 && HD % 16 == 0 && HD <= 512 && all % 16 == 0) {
    kern = rope_kv_write_pieces_kernel<T>;
    threads = H * (HD / 16) < 256 ? (H * (HD / 16) + 31) / 32 * 32 : 256;        // no warps without a head (2048 tokens of 3 heads of 64: 6.4 us with)
    const int heads = threads / (HD / 16) * 3;
    gy = (H + heads - 1) / heads;
  }
  return launch(kern, dim3(tokens, gy), dim3(threads), 0, st, pdl != 0, static_cast<const T*>(qkv),
                static_cast<__nv_bfloat16*>(q_out), static_cast<__nv_bfloat16*>(k_cache),
                static_cast<__nv_bfloat16*>(v_cache), block_table, positions, token_seq, cos_t, sin_t, Hq, Hkv, HD,
                max_blocks, page, traditional);
}

// qkv bf16, or fp32 with qkv_f32.
extern "C" int rmlx_rope_kv_write(const void* qkv, int qkv_f32, void* q_out, void* k_cache, void* v_cache,
                                  const int* block_table, const int* positions, const int* token_seq,
                                  const float* cos_t, const float* sin_t, int T, int Hq, int Hkv,
                                  int HD, int max_blocks, int page, int traditional, int pdl,
                                  cudaStream_t st) {
  if (T < 1 || HD % 2 || HD / 2 > 1024) return -2;
  return qkv_f32 ? launch_rope_kv<float>(qkv, q_out, k_cache, v_cache, block_table, positions, token_seq, cos_t, sin_t, T,
                                         Hq, Hkv, HD, max_blocks, page, traditional, pdl, st)
                 : launch_rope_kv<__nv_bfloat16>(qkv, q_out, k_cache, v_cache, block_table, positions, token_seq, cos_t,
                                                 sin_t, T, Hq, Hkv, HD, max_blocks, page, traditional, pdl, st);
}

extern "C" int rmlx_rope(const void* x, void* out, const int* positions, const float* cos_t,
                         const float* sin_t, int T, int H, int HD, int traditional, int inverse,
                         cudaStream_t st) {
  if (T < 1 || HD % 2 || HD / 2 > 1024) return -2;
  rope_kernel<<<dim3(T, H), HD / 2, 0, st>>>(static_cast<const __nv_bfloat16*>(x),
                                             static_cast<__nv_bfloat16*>(out), positions, cos_t,
                                             sin_t, H, HD, traditional, inverse);
  return static_cast<int>(cudaGetLastError());
}
