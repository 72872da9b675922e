// 8-bit paged KV cache: RoPE + quantising append, and page expansion.
//
// Format (per layer): data uint8 [blocks, Hkv, 16, HD]; sb bf16 [blocks, Hkv, 16, HD/64, 2]
// holding (scale, bias) per token and group of 64 along the head dimension, x = q * scale + bias
// with q in 0..255: the affine group format of the reference's QuantizedKvCache
// (crates/rmlx-nn/src/attention.rs:4438-4680, bits = 8, group 64), which the reference keeps on
// the host and re-quantises on every append; here a new token's rows are quantised once, on the
// device, inside the kernel that rotates them, and the attention kernel (flash_decode.cu) expands
// pages in shared memory. Half the cache bytes per token at decode.
//
//   rope_kv_write_q8    merged QKV rows -> rotated Q (bf16), rotated K and V quantised into pages
//   kv_dequant_pages    the pages of one sequence -> contiguous bf16 pages (prompt attention over
//                       an 8-bit cache, tests)
#include "../common/ptx.cuh"
#include "../common/launch.cuh"

namespace rb {

constexpr int kKq8Warps = 4;

// A warp takes a head of a token, lane l the J = HD / 32 values from J l on, so that a row is one access of a warp each way, the other
// value of a pair is 16 lanes away (traditional: beside it) and a group of 64 is 64 / J lanes. Bound by latency (angles and page of the
// token, then the heads' values one ahead): 512 tokens of 48 heads of 128 7.2 us, 2048 16.9; 8.2 and 20.9 with values 32 apart in a lane
// and the angles read again for every head.
template <int J>
__global__ void __launch_bounds__(kKq8Warps * 32)
rope_kv_write_q8_kernel(const __nv_bfloat16* __restrict__ qkv, __nv_bfloat16* __restrict__ q_out,
                        uint8_t* __restrict__ k_q, __nv_bfloat16* __restrict__ k_sb,
                        uint8_t* __restrict__ v_q, __nv_bfloat16* __restrict__ v_sb,
                        const int* __restrict__ block_table, const int* __restrict__ positions,
                        const int* __restrict__ token_seq, const float* __restrict__ cos_t,
                        const float* __restrict__ sin_t, int Hq, int Hkv, int max_blocks, int page,
                        int traditional, int whole) {
  constexpr int HD = J * 32, G64 = HD / 64, half = HD / 2, kLanes = 64 / J;
  const int tkn = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  pdl_launch_dependents();
  pdl_wait();
  const int pos = positions[tkn];
  const int H = Hq + 2 * Hkv;
  const int pg = pos / page;
  const bool inside = RB_BOUNDS(pg, max_blocks);
  const int blk = inside ? block_table[size_t(token_seq ? token_seq[tkn] : tkn) * max_blocks + pg] : 0;
  float c[J], s[J];                             // the angles are the same for every head
#pragma unroll
  for (int j = 0; j < J; ++j) {
    const size_t i = size_t(pos) * half + (traditional ? (lane * J + j) >> 1 : (lane & 15) * J + j);
    c[j] = cos_t[i];
    s[j] = sin_t[i];
    if (!traditional && lane < 16) s[j] = -s[j];
  }
  uint32_t u[J / 2];
  auto load = [&](int head) {
    const __nv_bfloat16* const src = qkv + (size_t(tkn) * H + head) * HD + lane * J;
    if (whole) {                                // every table at a 16-byte address
      if constexpr (J == 2) u[0] = *reinterpret_cast<const uint32_t*>(src);
      if constexpr (J == 4) { const uint2 v = *reinterpret_cast<const uint2*>(src); u[0] = v.x; u[1] = v.y; }
      if constexpr (J == 8) { const uint4 v = *reinterpret_cast<const uint4*>(src); u[0] = v.x; u[1] = v.y; u[2] = v.z; u[3] = v.w; }
    } else {
#pragma unroll
      for (int j = 0; j < J / 2; ++j) u[j] = pack_bf16(__bfloat162float(src[2 * j]), __bfloat162float(src[2 * j + 1]));
    }
  };
  const int first = blockIdx.y * kKq8Warps + warp, step = gridDim.y * kKq8Warps;
  if (first < H) load(first);
  for (int head = first; head < H; head += step) {
    float x[J];
#pragma unroll
    for (int j = 0; j < J / 2; ++j) { x[2 * j] = bf16lo(u[j]); x[2 * j + 1] = bf16hi(u[j]); }
    if (head + step < H) load(head + step);     // on its way while this one is rotated
    if (head < Hq + Hkv) {                      // rotate Q and K
      if (!traditional) {
#pragma unroll
        for (int j = 0; j < J; ++j) {
          const float other = __shfl_xor_sync(0xffffffffu, x[j], 16);
          x[j] = x[j] * c[j] + other * s[j];
        }
      } else {
#pragma unroll
        for (int j = 0; j < J; j += 2) {
          const float a = x[j], b = x[j + 1];
          x[j] = a * c[j] - b * s[j];
          x[j + 1] = b * c[j] + a * s[j];
        }
      }
    }
    if (head < Hq) {
      __nv_bfloat16* const dst = q_out + (size_t(tkn) * Hq + head) * HD + lane * J;
      if (!whole) {
#pragma unroll
        for (int j = 0; j < J; ++j) dst[j] = __float2bfloat16_rn(x[j]);
        continue;
      }
      uint32_t o[J / 2];
#pragma unroll
      for (int j = 0; j < J / 2; ++j) o[j] = pack_bf16(x[2 * j], x[2 * j + 1]);
      if constexpr (J == 2) *reinterpret_cast<uint32_t*>(dst) = o[0];
      if constexpr (J == 4) *reinterpret_cast<uint2*>(dst) = make_uint2(o[0], o[1]);
      if constexpr (J == 8) *reinterpret_cast<uint4*>(dst) = make_uint4(o[0], o[1], o[2], o[3]);
      continue;
    }
    if (!inside) continue;
    const bool is_k = head < Hq + Hkv;
    const int kvh = is_k ? head - Hq : head - Hq - Hkv;
    const size_t row = (size_t(blk) * Hkv + kvh) * page + (pos - pg * page);
    uint8_t* dq = (is_k ? k_q : v_q) + row * HD;
    __nv_bfloat16* dsb = (is_k ? k_sb : v_sb) + row * G64 * 2;
    float mn = x[0], mx = x[0];
#pragma unroll
    for (int j = 1; j < J; ++j) { mn = fminf(mn, x[j]); mx = fmaxf(mx, x[j]); }
#pragma unroll
    for (int o = kLanes / 2; o > 0; o >>= 1) {
      mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    }
    // bias: the minimum rounded DOWN to bf16; scale: (max - stored bias) / 255 rounded UP to
    // bf16, so neither end of the range clips; the codes are computed against the stored pair
    const uint32_t mnb = __float_as_uint(mn);
    const float bi = __uint_as_float(mn >= 0.f ? (mnb & 0xFFFF0000u) : ((mnb + 0xFFFFu) & 0xFFFF0000u));
    const __nv_bfloat16 bb16 = __float2bfloat16_rn(bi);     // exact: bi is a bf16 value
    float span = fmaxf(mx - bi, 0.f) / 255.f;
    if (!(span > 0.f)) span = 1.f;
    const float sc = __uint_as_float((__float_as_uint(span) + 0xFFFFu) & 0xFFFF0000u);
    const __nv_bfloat16 sb16 = __float2bfloat16_rn(sc);     // exact: sc is a bf16 value
    const float inv = 1.f / sc;
    uint32_t code[(J + 3) / 4] = {};
#pragma unroll
    for (int j = 0; j < J; ++j) {
      const float q = rintf((x[j] - bi) * inv);
      code[j / 4] |= uint32_t(static_cast<uint8_t>(fminf(fmaxf(q, 0.f), 255.f))) << (8 * (j % 4));
    }
    if (whole) {
      if constexpr (J == 2) reinterpret_cast<uint16_t*>(dq)[lane] = uint16_t(code[0]);
      if constexpr (J == 4) reinterpret_cast<uint32_t*>(dq)[lane] = code[0];
      if constexpr (J == 8) reinterpret_cast<uint2*>(dq)[lane] = make_uint2(code[0], code[1]);
    } else {
#pragma unroll
      for (int j = 0; j < J; ++j) dq[lane * J + j] = uint8_t(code[j / 4] >> (8 * (j % 4)));
    }
    if (lane % kLanes == 0) { dsb[2 * (lane / kLanes)] = sb16; dsb[2 * (lane / kLanes) + 1] = bb16; }
  }
}

// out [n_pages, Hkv, page, HD] bf16: page i of the output is page table[i] of the cache. A thread expands 16 codes, which share a scale
// and a bias: 251 pages of 8 heads of 16 x 128 4.1 us, 10.2 one code at a time.
__global__ void __launch_bounds__(256)
kv_dequant_pages_kernel(const uint8_t* __restrict__ q, const __nv_bfloat16* __restrict__ sb,
                        const int* __restrict__ table, __nv_bfloat16* __restrict__ out, int Hkv,
                        int page, int HD, int whole) {
  pdl_launch_dependents();
  pdl_wait();
  const size_t src_page = size_t(table[blockIdx.x]) * Hkv + blockIdx.y;
  const size_t dst_page = size_t(blockIdx.x) * Hkv + blockIdx.y;
  const int n = page * HD;
  if (!whole) {                                 // tables at odd addresses
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
      const __nv_bfloat16* const s = sb + ((src_page * n + i) >> 6) * 2;
      out[dst_page * n + i] = __float2bfloat16_rn(float(q[src_page * n + i]) * __bfloat162float(s[0]) + __bfloat162float(s[1]));
    }
    return;
  }
  for (int i = threadIdx.x * 16; i < n; i += blockDim.x * 16) {
    const uint4 v = *reinterpret_cast<const uint4*>(q + src_page * n + i);
    const uint32_t both = *reinterpret_cast<const uint32_t*>(sb + ((src_page * n + i) >> 6) * 2);
    const float sc = bf16lo(both), bi = bf16hi(both);
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
    uint32_t o[8];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      o[2 * j] = pack_bf16(float(w[j] & 0xffu) * sc + bi, float(w[j] >> 8 & 0xffu) * sc + bi);
      o[2 * j + 1] = pack_bf16(float(w[j] >> 16 & 0xffu) * sc + bi, float(w[j] >> 24) * sc + bi);
    }
    uint4* const dst = reinterpret_cast<uint4*>(out + dst_page * n + i);
    dst[0] = make_uint4(o[0], o[1], o[2], o[3]);
    dst[1] = make_uint4(o[4], o[5], o[6], o[7]);
  }
}

// Every pointer on 16 bytes.
template <class... P>
static bool whole16(const P*... p) { return ((reinterpret_cast<uintptr_t>(p) | ...) % 16) == 0; }

}  // namespace rb

using namespace rb;
RB_BOUNDS_REGISTER("kv_q8.cu")

// Same contract as rmlx_rope_kv_write with the cache in the 8-bit format; head_dim 64, 128 or 256.
extern "C" int rmlx_rope_kv_write_q8(const void* qkv, void* q_out, void* k_q, void* k_sb, void* v_q,
                                     void* v_sb, const int* block_table, const int* positions,
                                     const int* token_seq, const float* cos_t, const float* sin_t,
                                     int T, int Hq, int Hkv, int HD, int max_blocks, int page,
                                     int traditional, int pdl, cudaStream_t st) {
  if (T < 1 || (HD != 64 && HD != 128 && HD != 256)) return -2;
  const int H = Hq + 2 * Hkv;
  const int per = T >= 1024 ? 12 * kKq8Warps : T >= 128 ? 4 * kKq8Warps : kKq8Warps;    // heads per block: prompts take several per warp, the next one's values on their way
  const dim3 grid(T, (H + per - 1) / per);
  const int whole = whole16(qkv, q_out, k_q, v_q);
#define RB_KQ8(J_)                                                                                 \
  return launch(rope_kv_write_q8_kernel<J_>, grid, dim3(kKq8Warps * 32), 0, st, pdl != 0,          \
                static_cast<const __nv_bfloat16*>(qkv), static_cast<__nv_bfloat16*>(q_out),        \
                static_cast<uint8_t*>(k_q), static_cast<__nv_bfloat16*>(k_sb),                     \
                static_cast<uint8_t*>(v_q), static_cast<__nv_bfloat16*>(v_sb), block_table,        \
                positions, token_seq, cos_t, sin_t, Hq, Hkv, max_blocks, page, traditional, whole);
  if (HD == 64) { RB_KQ8(2) }
  if (HD == 128) { RB_KQ8(4) }
  RB_KQ8(8)
#undef RB_KQ8
}

extern "C" int rmlx_kv_dequant_pages(const void* q, const void* sb, const int* table, void* out,
                                     int n_pages, int Hkv, int page, int HD, int pdl, cudaStream_t st) {
  if (n_pages < 1 || HD % 64) return -2;
  const int threads = page * HD >= 4096 ? 256 : 128;
  return launch(kv_dequant_pages_kernel, dim3(n_pages, Hkv), dim3(threads), 0, st, pdl != 0, static_cast<const uint8_t*>(q),
                static_cast<const __nv_bfloat16*>(sb), table, static_cast<__nv_bfloat16*>(out), Hkv, page, HD,
                whole16(q, out) && reinterpret_cast<uintptr_t>(sb) % 4 == 0);
}
