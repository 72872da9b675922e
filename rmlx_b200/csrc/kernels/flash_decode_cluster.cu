// Paged flash-decode attention: a cluster of 1 to 16 blocks per (sequence, kv head, 16 query heads) tile, its pages split evenly over the
// cluster's warps, merged once through distributed shared memory.
//
// What bounds it: the cache is read once, so with long contexts the time is its trip from HBM; with short ones, a chain of latencies
// (length, block table, page, products, merge) and of instructions fetched for the first time: code that runs once per block costs about a
// microsecond per hundred lines, so the merge is short loops. A grid of fixed splits per sequence loses both ways: 5 splits of 32 tiles are
// 160 blocks for 148 SMs, two waves, and their merge goes through global memory and a ticket (splitting all pages evenly over 148
// blocks kept the SMs even but paid 8 us for that merge). Here
//   * the cluster size is the one that needs the fewest rounds of clusters for its speed; with more tiles than clusters a cluster takes
//     a contiguous run of tiles of about its share of all pages, counted on the device from the lengths;
//   * each warp takes a contiguous run of the tile's pages through its own cp.async ring, which runs on into the next tile;
//   * a block's warps merge in its shared memory, and the blocks of a cluster through one another's: after one cluster barrier each
//     takes its share of the results and sums all blocks' parts of it, in order, so that results repeat (all warps' parts through the
//     cluster at once: four times the remote bytes, 19 us instead of 11 for one sequence of 4096);
//   * blocks are four warps and half an SM, so that one block's merge runs beside another's pages.
// With `early` the caller says that no kernel still running writes lengths, tables, or pages other than a sequence's last one (a decode step,
// whose predecessor appends one token): the first pages are then asked for before the predecessor has finished.
//
// 8-bit cache (x = q * scale + bias per token and group of 64): pages are not expanded. A byte in the low half of an fp16 is the subnormal
// q x 2^-24, exactly, so one byte permutation makes two operands; K's scale and bias are applied to the sums of a (head, token, group),
// V's scale to the probabilities and its bias to their sum. Neither K nor V is rounded, the query enters as fp16 with one power of two
// per (head, group), and probabilities times V's scale keep fp16's 11 bits.
//
// mma.sync on purpose: M is the 16 query heads of a tile and the kernel is bound by bytes and latency.
//
// Measured (us a launch, chained; before / this; the cache's bytes at the copy rate): 64 query and 4 kv heads of 128, one sequence of 4097
// 11.4 / 9.8 (1.3), 8 of 3474-3901 32.3 / 17.8 (9.4), 64 of 1548-2049 56.7 / 45.1 (36.8); 16 and 4 heads, 5 of 595-778 16.5 / 7.2 (1.1);
// 32 and 8 heads, 64 of 226-300 25.0 / 20.5 (10.7); 8-bit: 32 and 8 heads, 16 of 1513-2001 44.6 / 24.7 (9.5: some 600 instructions a
// page and two warps a scheduler); 4 and 2 heads of 64, 25 tokens 5.8 / 3.8. Error of the result against 64 bits: bf16 2.1e-3 before and now, 8-bit
// 3.1e-3 / 1.7e-3.
//
// Replaces sdpa_decode_batched_* over contiguous slabs (crates/rmlx-core/src/ops/sdpa.rs:810,1541); the 8-bit format is that of
// crates/rmlx-nn/src/attention.rs:4438-4680.
#include "../common/ptx.cuh"
#include "../common/launch.cuh"

namespace rb {

constexpr int kFcPage = 16, kFcWarps = 4, kFcThreads = kFcWarps * 32, kFcMaxBatch = 512, kFcMaxCluster = 16;

struct FcParams {
  const __nv_bfloat16* q;        // [B, Hq, HD]
  const char *k_cache, *v_cache; // [blocks, Hkv, 16, HD] bf16, or uint8 codes with
  const char *k_sb, *v_sb;       // [blocks, Hkv, 16, HD/64] (scale, bias) bf16 pairs
  const int* block_table;        // [B, max_blocks], rows table_stride apart (0: one row for all)
  const int* seq_lens;           // [B] tokens in the cache including the current one
  __nv_bfloat16* out;            // [B, Hq, HD]
  int B, max_blocks, table_stride, Hq, Hkv, G, gtiles, window, early, CS;
  float scale_log2;              // softmax scale * log2(e)
};

template <int HD, bool KVQ>
struct FcShape {
  static constexpr int NST = KVQ ? 4 : HD == 128 ? 2 : 3;
  static constexpr int PER_SM = 2;                                     // blocks
  static constexpr int PAGE = kFcPage * HD * (KVQ ? 1 : 2);            // bytes of a K (or V) page of one head
  static constexpr int SB = KVQ ? kFcPage * (HD / 64) * 4 : 0;         // bytes of its (scale, bias) pairs
  static constexpr int STAGE = 2 * (PAGE + SB);
  static constexpr int RING = kFcWarps * NST * STAGE;
  static constexpr int MERGE = kFcWarps * 16 * HD * 4;
  static constexpr int BYTES = RING + MERGE + kFcWarps * 32 * 4 + (kFcMaxBatch + 4) * 4;
};

__device__ __forceinline__ void fc_cp16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void fc_ldm4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void fc_ldm4t(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ float fc_exp2(float x) {      // 2 ulp, as exp2f; results below 2^-126 are zero
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ void fc_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
template <bool F16>
__device__ __forceinline__ void fc_mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  if constexpr (F16)
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  else
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t fc_half2(float lo, float hi) {
  const __half2 v = __floats2half2_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&v);
}

__device__ __forceinline__ float fc_remote(uint32_t addr, int rank) {
  float v;
  asm volatile("{.reg .u32 a; mapa.shared::cluster.u32 a, %1, %2; ld.shared::cluster.f32 %0, [a];}" : "=f"(v) : "r"(addr), "r"(rank) : "memory");
  return v;
}
__device__ __forceinline__ float2 fc_remote2(uint32_t addr, int rank) {
  float2 v;
  asm volatile("{.reg .u32 a; mapa.shared::cluster.u32 a, %2, %3; ld.shared::cluster.v2.f32 {%0, %1}, [a];}"
               : "=f"(v.x), "=f"(v.y) : "r"(addr), "r"(rank) : "memory");
  return v;
}

template <int HD, bool KVQ>
__global__ void __launch_bounds__(kFcThreads, FcShape<HD, KVQ>::PER_SM) flash_decode_cluster_kernel(const FcParams p) {
  using S = FcShape<HD, KVQ>;
  constexpr int KS = HD / 16, NT = HD / 8, G64 = HD / 64, CH = S::PAGE / kFcPage / 16;   // CH: 16-byte chunks per row
  extern __shared__ __align__(128) char smem[];
  float* const so = reinterpret_cast<float*>(smem + S::RING);            // [warp][16][HD] outputs
  float* const s_ml = so + S::MERGE / 4;                                 // [warp][16] (max, sum)
  int* const s_pre = reinterpret_cast<int*>(s_ml + kFcWarps * 32);       // pages before every sequence
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int heads = p.Hkv * p.gtiles, tiles = p.B * heads;
  int rank = 0;
  if (p.CS > 1) asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  const int cl = int(blockIdx.x) / p.CS, ncl = int(gridDim.x) / p.CS;
  const int W = p.CS * kFcWarps, wi = rank * kFcWarps + warp;            // warps of the cluster

  pdl_launch_dependents();
  if (!p.early) pdl_wait();
  // pages that a sequence's queries see, an empty sequence counted as one (its rows are zero)
  auto first_page = [&](int len) { return (p.window > 0 && len > p.window ? len - p.window : 0) / kFcPage; };
  auto pages_of = [&](int len) { return max(1, (len + kFcPage - 1) / kFcPage - first_page(len)); };
  int tile0 = cl, tile1 = min(cl + 1, tiles);            // tiles (b, yt) = b heads + yt of this cluster
  if (tiles > ncl) {
    if (warp == 0) {
      int base = 0;
      for (int b0 = 0; b0 < p.B; b0 += 32) {
        const int b = b0 + lane, n = b < p.B ? pages_of(p.seq_lens[b]) : 0;
        int sum = n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { const int v = __shfl_up_sync(0xffffffffu, sum, o); if (lane >= o) sum += v; }
        if (b < p.B) s_pre[b] = base + sum - n;
        base += __shfl_sync(0xffffffffu, sum, 31);
      }
      if (lane == 0) s_pre[p.B] = base;
    }
    __syncthreads();
    // the tile in whose first half the cluster's share of all pages begins, or the one after
    auto first_tile = [&](int c) {
      if (c >= ncl) return tiles;
      const int unit = int((long long)s_pre[p.B] * heads * c / ncl);
      int b = 0;
      for (int b0 = 0; b0 < p.B; b0 += 32)
        b += __popc(__ballot_sync(0xffffffffu, b0 + lane < p.B && s_pre[min(b0 + lane, p.B - 1) + 1] * heads <= unit));
      const int n = s_pre[b + 1] - s_pre[b], local = unit - s_pre[b] * heads, yt = local / n;
      return b * heads + yt + ((local - yt * n) * 2 > n ? 1 : 0);
    };
    tile0 = first_tile(cl); tile1 = first_tile(cl + 1);
  }
  if (tile0 >= tile1) return;                            // all blocks of the cluster alike

  // this warp's pages of a tile of n, counted from the first visible one
  auto share = [&](int n, int& from, int& to) {
    if (n >= W) { from = n * wi / W; to = n * (wi + 1) / W; }
    else { from = min(wi, n); to = min(wi + 1, n); }
  };

  // ---------------------------------------------------------------- page ring (one per warp)
  const uint32_t ring = smem_u32(smem) + warp * (S::NST * S::STAGE);
  struct { int tile, b, yt, n, at, to; } pw = {tile0 - 1, 0, 0, 1, 0, 0};
  int p_stage = 0, p_tab = 0, p_tab0 = -1;
  auto next_tile = [&]() {                               // to the next page of this warp: false if there is none
#pragma unroll 1
    while (pw.at >= pw.to) {
      if (++pw.tile >= tile1) { pw.tile = tile1; return false; }
      pw.b = pw.tile / heads; pw.yt = pw.tile - pw.b * heads;
      pw.n = pages_of(p.seq_lens[pw.b]);
      share(pw.n, pw.at, pw.to);
      p_tab0 = -1;
    }
    return true;
  };
  auto page = [&](int at) {                              // block number of a page of the producer's tile: 32 are looked up at a time
    if (p_tab0 < 0 || at >= p_tab0 + 32) {
      const int len = p.seq_lens[pw.b], pg = first_page(len) + min(at + lane, pw.n - 1);
      p_tab0 = at;
      p_tab = len > 0 && RB_BOUNDS(pg, p.max_blocks) ? p.block_table[size_t(pw.b) * p.table_stride + pg] : 0;   // page 0 is reserved
    }
    return __shfl_sync(0xffffffffu, p_tab, at - p_tab0);
  };
  bool waited = !p.early;
  auto issue = [&]() {
    if (next_tile()) {
      if (!waited && pw.at == pw.n - 1) { pdl_wait(); waited = true; }   // the predecessor writes to the last page
      const int blk = page(pw.at);
      const size_t at = size_t(blk) * p.Hkv + pw.yt / p.gtiles;
      const char *ks = p.k_cache + at * S::PAGE, *vs = p.v_cache + at * S::PAGE;
      const uint32_t kd = ring + p_stage * S::STAGE, vd = kd + S::PAGE;
#pragma unroll
      for (int i = 0; i < kFcPage * CH / 32; ++i) {
        const int idx = i * 32 + lane, r = idx / CH, c = idx % CH;
        int ko, vo;
        if (KVQ) {      // K is read 64 bytes of two tokens at a time, V 16 bytes of eight
          ko = r * HD + ((HD == 128 ? c ^ ((r & 1) << 2) : c) << 4);
          vo = r * HD + ((c ^ (HD == 128 ? r & 7 : (r >> 1) & 3)) << 4);
        } else {
          ko = vo = r * (HD * 2) + ((c ^ (r & 7)) << 4);
        }
        fc_cp16(kd + ko, ks + idx * 16);
        fc_cp16(vd + vo, vs + idx * 16);
      }
      if (KVQ && lane < 2 * S::SB / 16) {
        const bool v = lane >= S::SB / 16;
        const int o = (v ? lane - S::SB / 16 : lane) * 16;
        fc_cp16(vd + S::PAGE + lane * 16, (v ? p.v_sb : p.k_sb) + at * S::SB + o);
      }
      if (++p_stage == S::NST) p_stage = 0;
      ++pw.at;
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll 1
  for (int i = 0; i < S::NST; ++i) issue();
  if (!waited) {
    if (p_tab0 >= 0)     // what the ring has no room for yet, as far as the table was looked up
      for (int i = 0; i < 6 && pw.at + i < pw.to && pw.at + i < p_tab0 + 32; ++i) {
        const size_t at = size_t(page(pw.at + i)) * p.Hkv + pw.yt / p.gtiles;
        for (int l = lane * 128; l < S::PAGE; l += 32 * 128) {
          asm volatile("prefetch.global.L2 [%0];" ::"l"(p.k_cache + at * S::PAGE + l));
          asm volatile("prefetch.global.L2 [%0];" ::"l"(p.v_cache + at * S::PAGE + l));
        }
      }
    pdl_wait();
    waited = true;
  }

  int stage = 0;
#pragma unroll 1
  for (int tile = tile0; tile < tile1; ++tile) {
    struct { int b, yt; } s;
    s.b = tile / heads; s.yt = tile - s.b * heads;
    const int len = p.seq_lens[s.b], kvh = s.yt / p.gtiles, gt = s.yt - kvh * p.gtiles;
    int from, to;
    const int n = pages_of(len);
    share(n, from, to);
    const int first = p.window > 0 && len > p.window ? len - p.window : 0, pg_first = first / kFcPage;
    const __nv_bfloat16* const q0 = p.q + (size_t(s.b) * p.Hq + size_t(kvh) * p.G + gt * 16 + g) * HD;
    const bool v0 = gt * 16 + g < p.G, v1 = gt * 16 + g + 8 < p.G;       // query heads of this lane's two rows
    float o[NT][4];
#pragma unroll
    for (int j = 0; j < NT; ++j) o[j][0] = o[j][1] = o[j][2] = o[j][3] = 0.f;
    float m0 = -INFINITY, m1 = -INFINITY, l0 = 0.f, l1 = 0.f;
    // 8-bit: scale and sum of the query per (row, group); V's bias sums; the exponent at which o is kept
    float dn[2][G64], qs[2][G64], vb[2][G64];
    int vex[G64];
    uint32_t qa[KS][4];
    if constexpr (KVQ) {
#pragma unroll
      for (int gr = 0; gr < G64; ++gr) {
        vex[gr] = 0;
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          uint4 w[2] = {};
          if (r ? v1 : v0) {
            const uint4* src = reinterpret_cast<const uint4*>(q0 + r * 8 * HD + gr * 64 + t * 16);
            w[0] = src[0]; w[1] = src[1];
          }
          const uint32_t ww[8] = {w[0].x, w[0].y, w[0].z, w[0].w, w[1].x, w[1].y, w[1].z, w[1].w};
          float f[16], m = 0.f, sum = 0.f;
#pragma unroll
          for (int i = 0; i < 8; ++i) { f[2 * i] = bf16lo(ww[i]); f[2 * i + 1] = bf16hi(ww[i]); }
#pragma unroll
          for (int i = 0; i < 16; ++i) { m = fmaxf(m, fabsf(f[i])); sum += f[i]; }
          m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 1)); m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 2));
          sum += __shfl_xor_sync(0xffffffffu, sum, 1); sum += __shfl_xor_sync(0xffffffffu, sum, 2);
          // the largest magnitude goes to [2^14, 2^15), codes are q x 2^-24: scores are undone by 2^24 x 2^(ex - 141)
          const uint32_t ex = min(max(__float_as_uint(m) >> 23, 60u), 230u);
          const float up = __uint_as_float((268u - ex) << 23);
          dn[r][gr] = __uint_as_float((ex + 10u) << 23) * p.scale_log2;
          qs[r][gr] = sum * p.scale_log2;
          vb[r][gr] = 0.f;
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            qa[gr * 4 + i][r] = fc_half2(f[4 * i] * up, f[4 * i + 1] * up);
            qa[gr * 4 + i][2 + r] = fc_half2(f[4 * i + 2] * up, f[4 * i + 3] * up);
          }
        }
      }
    } else {
#pragma unroll
      for (int ks = 0; ks < KS; ++ks) {
        const int d = ks * 16 + t * 2;
        qa[ks][0] = v0 ? *reinterpret_cast<const uint32_t*>(q0 + d) : 0u;
        qa[ks][1] = v1 ? *reinterpret_cast<const uint32_t*>(q0 + 8 * HD + d) : 0u;
        qa[ks][2] = v0 ? *reinterpret_cast<const uint32_t*>(q0 + d + 8) : 0u;
        qa[ks][3] = v1 ? *reinterpret_cast<const uint32_t*>(q0 + 8 * HD + d + 8) : 0u;
      }
    }

#pragma unroll 1
    for (int pg = from; pg < to; ++pg) {
      asm volatile("cp.async.wait_group %0;" ::"n"(S::NST - 1) : "memory");
      __syncwarp();
      const uint32_t kbase = ring + stage * S::STAGE, vbase = kbase + S::PAGE;
      if (++stage == S::NST) stage = 0;
      // tokens of this lane's columns: 2t, 2t + 1, 2t + 8, 2t + 9 of the page
      bool ok[4];
      const int tok0 = (pg_first + pg) * kFcPage + t * 2;
#pragma unroll
      for (int i = 0; i < 4; ++i) { const int tk = tok0 + (i & 1) + (i >> 1) * 8; ok[i] = tk < len && tk >= first; }
      float sv[8];                                       // scores: row g of the four tokens, row g + 8
      if constexpr (KVQ) {
        const char* const raw = smem + (kbase - smem_u32(smem));
        const char* const sbk = raw + 2 * S::PAGE;
#pragma unroll
        for (int i = 0; i < 8; ++i) sv[i] = 0.f;
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
          uint32_t sb[2 * G64];                          // (scale, bias) of tokens 2t and 2t + 1, their groups
          if constexpr (G64 == 2) {
            const uint4 v = *reinterpret_cast<const uint4*>(sbk + (nt * 8 + 2 * t) * 8);
            sb[0] = v.x; sb[1] = v.y; sb[2] = v.z; sb[3] = v.w;
          } else {
            const uint2 v = *reinterpret_cast<const uint2*>(sbk + (nt * 8 + 2 * t) * 4);
            sb[0] = v.x; sb[1] = v.y;
          }
#pragma unroll
          for (int gr = 0; gr < G64; ++gr) {
            const int c = HD == 128 ? (gr * 4 + t) ^ ((g & 1) << 2) : t;
            const uint4 v = *reinterpret_cast<const uint4*>(raw + (nt * 8 + g) * HD + c * 16);
            const uint32_t w[4] = {v.x, v.y, v.z, v.w};
            float d[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int i = 0; i < 4; ++i)
              fc_mma<true>(d, qa[gr * 4 + i], __byte_perm(w[i], 0u, 0x4140u), __byte_perm(w[i], 0u, 0x4342u));
#pragma unroll
            for (int c2 = 0; c2 < 2; ++c2) {
              const float sc = __uint_as_float(sb[c2 * G64 + gr] << 16), bi = __uint_as_float(sb[c2 * G64 + gr] & 0xffff0000u);
#pragma unroll
              for (int r = 0; r < 2; ++r) {
                float& x = sv[r * 4 + nt * 2 + c2];
                x = fmaf(sc * dn[r][gr], d[r * 2 + c2], fmaf(bi, qs[r][gr], x));
              }
            }
          }
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) sv[i] = ok[i & 3] ? sv[i] : -INFINITY;
      } else {
        float s0[4] = {0.f, 0.f, 0.f, 0.f}, s1[4] = {0.f, 0.f, 0.f, 0.f};
        const int mi = lane >> 3, r = lane & 7, tok = (mi >> 1) * 8 + r;
#pragma unroll
        for (int ks = 0; ks < KS; ++ks) {
          const int c = 2 * ks + (mi & 1);
          uint32_t kb[4];
          fc_ldm4(kb, kbase + tok * (HD * 2) + ((c ^ r) << 4));
          fc_mma<false>(s0, qa[ks], kb[0], kb[1]);
          fc_mma<false>(s1, qa[ks], kb[2], kb[3]);
        }
        const float raw[8] = {s0[0], s0[1], s1[0], s1[1], s0[2], s0[3], s1[2], s1[3]};
#pragma unroll
        for (int i = 0; i < 8; ++i) sv[i] = ok[i & 3] ? raw[i] * p.scale_log2 : -INFINITY;
      }
      float mx0 = fmaxf(fmaxf(sv[0], sv[1]), fmaxf(sv[2], sv[3]));
      float mx1 = fmaxf(fmaxf(sv[4], sv[5]), fmaxf(sv[6], sv[7]));
      mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, 1));
      mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, 1));
      mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, 2));
      mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, 2));
      const float nm0 = fmaxf(m0, mx0), nm1 = fmaxf(m1, mx1);
      // a page holds at least one visible token, so nm is finite here (an empty sequence's only page is not looked at)
      if (__any_sync(0xffffffffu, nm0 != m0 || nm1 != m1)) {
        const float c0 = fc_exp2(m0 - nm0), c1 = fc_exp2(m1 - nm1);
        m0 = nm0; m1 = nm1;
        l0 *= c0; l1 *= c1;
#pragma unroll
        for (int j = 0; j < NT; ++j) { o[j][0] *= c0; o[j][1] *= c0; o[j][2] *= c1; o[j][3] *= c1; }
        if constexpr (KVQ)
#pragma unroll
          for (int gr = 0; gr < G64; ++gr) { vb[0][gr] *= c0; vb[1][gr] *= c1; }
      }
      float pr[8];
#pragma unroll
      for (int i = 0; i < 4; ++i) { pr[i] = fc_exp2(sv[i] - m0); pr[4 + i] = fc_exp2(sv[4 + i] - m1); }
      l0 += pr[0] + pr[1] + pr[2] + pr[3];
      l1 += pr[4] + pr[5] + pr[6] + pr[7];
      if constexpr (KVQ) {
        const char* const sbv = smem + (vbase - smem_u32(smem)) + S::PAGE + S::SB;
        uint32_t sb[4 * G64];                            // tokens 2t, 2t + 1, 2t + 8, 2t + 9
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
          if constexpr (G64 == 2) {
            const uint4 v = *reinterpret_cast<const uint4*>(sbv + (nt * 8 + 2 * t) * 8);
            sb[nt * 4] = v.x; sb[nt * 4 + 1] = v.y; sb[nt * 4 + 2] = v.z; sb[nt * 4 + 3] = v.w;
          } else {
            const uint2 v = *reinterpret_cast<const uint2*>(sbv + (nt * 8 + 2 * t) * 4);
            sb[nt * 2] = v.x; sb[nt * 2 + 1] = v.y;
          }
        }
#pragma unroll
        for (int gr = 0; gr < G64; ++gr) {
          float sc[4], big = 0.f;
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const uint32_t w = ok[i] ? sb[i * G64 + gr] : 0u;    // what lies behind the last token counts for nothing
            const float bi = __uint_as_float(w & 0xffff0000u);
            sc[i] = __uint_as_float(w << 16);
            big = fmaxf(big, fabsf(sc[i]));
            vb[0][gr] = fmaf(pr[i], bi, vb[0][gr]);
            vb[1][gr] = fmaf(pr[4 + i], bi, vb[1][gr]);
          }
          big = fmaxf(big, __shfl_xor_sync(0xffffffffu, big, 1));
          big = fmaxf(big, __shfl_xor_sync(0xffffffffu, big, 2));
          // the largest scale so far goes to [2^14, 2^15): probabilities times scales keep 11 bits down to 2^-28 of it
          const int ex = int(min(max(__float_as_uint(big) >> 23, 30u), 230u));
          if (ex > vex[gr]) {                            // the same in all lanes
            if (vex[gr]) {
              const float c = vex[gr] - ex < -100 ? 0.f : __uint_as_float(uint32_t(127 + vex[gr] - ex) << 23);
#pragma unroll
              for (int j = gr * 8; j < gr * 8 + 8; ++j) { o[j][0] *= c; o[j][1] *= c; o[j][2] *= c; o[j][3] *= c; }
            }
            vex[gr] = ex;
          }
          const float up = __uint_as_float(uint32_t(268 - vex[gr]) << 23);
#pragma unroll
          for (int i = 0; i < 4; ++i) sc[i] *= up;
          const uint32_t pa[4] = {fc_half2(pr[0] * sc[0], pr[1] * sc[1]), fc_half2(pr[4] * sc[0], pr[5] * sc[1]),
                                  fc_half2(pr[2] * sc[2], pr[3] * sc[3]), fc_half2(pr[6] * sc[2], pr[7] * sc[3])};
          // 16 dims of 16 tokens per pair of matrices: bytes (2g, 2g + 1) of tokens 2t and 2t + 1: an even and an odd tile
          const int mi = lane >> 3, r = lane & 7, tok = (mi & 1) * 8 + r;
#pragma unroll
          for (int j = 0; j < 4; j += 2) {
            const int c = gr * 4 + j + (mi >> 1);
            uint32_t w[4];
            fc_ldm4t(w, vbase + tok * HD + ((c ^ (HD == 128 ? tok & 7 : (tok >> 1) & 3)) << 4));
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
              for (int odd = 0; odd < 2; ++odd)
                fc_mma<true>(o[gr * 8 + (j + h) * 2 + odd], pa, __byte_perm(w[2 * h], 0u, odd ? 0x4341u : 0x4240u),
                             __byte_perm(w[2 * h + 1], 0u, odd ? 0x4341u : 0x4240u));
          }
        }
      } else {
        const uint32_t pa[4] = {pack_bf16(pr[0], pr[1]), pack_bf16(pr[4], pr[5]), pack_bf16(pr[2], pr[3]), pack_bf16(pr[6], pr[7])};
        const int mi = lane >> 3, r = lane & 7, tok = (mi & 1) * 8 + r;
#pragma unroll
        for (int j = 0; j < NT; j += 2) {
          const int c = j + (mi >> 1);
          uint32_t vv[4];
          fc_ldm4t(vv, vbase + tok * (HD * 2) + ((c ^ r) << 4));
          fc_mma<false>(o[j], pa, vv[0], vv[1]);
          fc_mma<false>(o[j + 1], pa, vv[2], vv[3]);
        }
      }
      __syncwarp();
      issue();                                           // the stage has been read
    }
    l0 += __shfl_xor_sync(0xffffffffu, l0, 1); l0 += __shfl_xor_sync(0xffffffffu, l0, 2);
    l1 += __shfl_xor_sync(0xffffffffu, l1, 1); l1 += __shfl_xor_sync(0xffffffffu, l1, 2);

    if constexpr (KVQ) {                                 // to true size, biases added
#pragma unroll
      for (int gr = 0; gr < G64; ++gr) {
        const float f = __uint_as_float(uint32_t(max(vex[gr], 1) + 10) << 23);      // 2^24 / 2^(141 - vex)
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          vb[r][gr] += __shfl_xor_sync(0xffffffffu, vb[r][gr], 1);
          vb[r][gr] += __shfl_xor_sync(0xffffffffu, vb[r][gr], 2);
        }
#pragma unroll
        for (int j = gr * 8; j < gr * 8 + 8; ++j)
#pragma unroll
          for (int i = 0; i < 4; ++i) o[j][i] = fmaf(o[j][i], f, vb[i >> 1][gr]);
      }
    }
    if (from < to) {
      if (t == 0) {
        float* const ml = s_ml + (warp * 16 + g) * 2;
        *reinterpret_cast<float2*>(ml) = make_float2(m0, l0);
        *reinterpret_cast<float2*>(ml + 16) = make_float2(m1, l1);
      }
      float* const mine = so + (warp * 16 + g) * HD;
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        if constexpr (KVQ) {
#pragma unroll
          for (int j = 0; j < NT; j += 2)
            *reinterpret_cast<float4*>(mine + r * 8 * HD + j * 8 + 4 * t) = make_float4(o[j][2 * r], o[j + 1][2 * r], o[j][2 * r + 1], o[j + 1][2 * r + 1]);
        } else {
#pragma unroll
          for (int j = 0; j < NT; ++j) *reinterpret_cast<float2*>(mine + r * 8 * HD + j * 8 + 2 * t) = make_float2(o[j][2 * r], o[j][2 * r + 1]);
        }
      }
    }
    // ---------------------------------------------------------------- merge
    __syncthreads();
    const int live = min(16, p.G - gt * 16);             // rows with a head
    const int mine_n = n >= W ? kFcWarps : min(kFcWarps, max(0, n - rank * kFcWarps));   // warps of the block, blocks with a page
    const int blocks = n >= W ? p.CS : (n + kFcWarps - 1) / kFcWarps;
    __nv_bfloat16* const dst = p.out + (size_t(s.b) * p.Hq + size_t(kvh) * p.G + gt * 16) * HD;
    constexpr int V = HD / 32;
    if (mine_n > 0) {                                    // the block's warps, into the first one's place
#pragma unroll 1
      for (int row = warp; row < live; row += kFcWarps) {
        float2 ml[kFcWarps];
        float M = -INFINITY, L = 0.f, acc[V] = {};
#pragma unroll
        for (int i = 0; i < kFcWarps; ++i) {
          ml[i] = i < mine_n ? *reinterpret_cast<const float2*>(s_ml + (i * 16 + row) * 2) : make_float2(-INFINITY, 0.f);
          M = fmaxf(M, ml[i].x);
        }
        float* const at = so + row * HD + lane * V;
#pragma unroll
        for (int i = 0; i < kFcWarps; ++i) {
          if (i >= mine_n) break;
          const float f = fc_exp2(ml[i].x - M);
          L = fmaf(ml[i].y, f, L);
#pragma unroll
          for (int x = 0; x < V; ++x) acc[x] = fmaf(at[i * 16 * HD + x], f, acc[x]);
        }
        if (p.CS == 1) {
          const float inv = 1.f / L;
          uint32_t* const out = reinterpret_cast<uint32_t*>(dst + row * HD + lane * V);
#pragma unroll
          for (int x = 0; x < V; x += 2) out[x / 2] = len > 0 ? pack_bf16(acc[x] * inv, acc[x + 1] * inv) : 0u;
        } else {
#pragma unroll
          for (int x = 0; x < V; ++x) at[x] = acc[x];
          __syncwarp();                                  // the row's maxima have been read by all lanes
          if (lane == 0) *reinterpret_cast<float2*>(s_ml + row * 2) = make_float2(M, L);
        }
      }
    }
    if (p.CS > 1) {                                      // the cluster's blocks: each the same share of the results
      fc_cluster_sync();
      const int each = (live * HD + p.CS - 1) / p.CS, end = min(live * HD, (rank + 1) * each);
#pragma unroll 1
      for (int e = rank * each + threadIdx.x; e < end; e += kFcThreads) {
        const uint32_t ml_at = smem_u32(s_ml + e / HD * 2), at = smem_u32(so + e);
        float M = -INFINITY, L = 0.f, acc = 0.f;
#pragma unroll 1
        for (int i0 = 0; i0 < blocks; i0 += 8) {         // loads first: what this costs is their latency
          float2 ml[8];
          float v[8], m = M;
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int r = min(i0 + i, blocks - 1);
            ml[i] = fc_remote2(ml_at, r);
            v[i] = fc_remote(at, r);
          }
#pragma unroll
          for (int i = 0; i < 8; ++i) m = fmaxf(m, ml[i].x);
          const float back = fc_exp2(M - m);
          M = m; L *= back; acc *= back;
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const float f = i0 + i < blocks ? fc_exp2(ml[i].x - M) : 0.f;
            L = fmaf(ml[i].y, f, L);
            acc = fmaf(v[i], f, acc);
          }
        }
        dst[e] = __float2bfloat16_rn(len > 0 ? acc / L : 0.f);
      }
    }
    // the partials are free, and nobody leaves while they are read
    if (p.CS > 1) fc_cluster_sync(); else if (tile + 1 < tile1) __syncthreads();
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
}

template <int HD, bool KVQ>
static cudaError_t fc_prepare(int cs) {
  auto kern = flash_decode_cluster_kernel<HD, KVQ>;
  cudaError_t e = set_max_smem(kern, FcShape<HD, KVQ>::BYTES);
  if (e == cudaSuccess && cs > 8) e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  return e;
}

static void fc_config(cudaLaunchConfig_t& cfg, cudaLaunchAttribute* attr, int grid, int cs, int smem, bool pdl, cudaStream_t st) {
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(kFcThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  int n = 0;
  if (cs > 1) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = cs; attr[n].val.clusterDim.y = 1; attr[n].val.clusterDim.z = 1;
    ++n;
  }
  if (pdl) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n].val.programmaticStreamSerializationAllowed = 1;
    ++n;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n;
}

template <int HD, bool KVQ>
static int fc_launch(const FcParams& p, int clusters, int pdl, cudaStream_t st) {
  using S = FcShape<HD, KVQ>;
  static_assert((S::BYTES + 1024) * S::PER_SM <= 228 * 1024, "blocks per SM");
  auto kern = flash_decode_cluster_kernel<HD, KVQ>;
  RB_CHECK((fc_prepare<HD, KVQ>(p.CS)));
  if (pdl) prefer_max_shared(kern);
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
  fc_config(cfg, attr, clusters * p.CS, p.CS, S::BYTES, pdl != 0, st);
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, p);
  if (e != cudaSuccess) (void)cudaGetLastError();
  return static_cast<int>(e);
}

// Clusters of cs blocks that can be resident at once.
template <int HD, bool KVQ>
static int fc_resident(int cs) {
  static int known[64][5] = {};                          // cs = 1 << i; 0: not asked yet
  int dev = 0, i = 0, n = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  while ((1 << i) < cs) ++i;
  if (cs == 1) return FcShape<HD, KVQ>::PER_SM * sm_count();
  if (known[dev][i] == 0) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[2];
    fc_config(cfg, attr, cs * 64, cs, FcShape<HD, KVQ>::BYTES, false, nullptr);
    if (fc_prepare<HD, KVQ>(cs) != cudaSuccess || cudaOccupancyMaxActiveClusters(&n, flash_decode_cluster_kernel<HD, KVQ>, &cfg) != cudaSuccess)
      n = 0;
    (void)cudaGetLastError();
    known[dev][i] = n > 0 ? n : -1;
  }
  return known[dev][i] > 0 ? known[dev][i] : 0;
}

}  // namespace rb

using namespace rb;
RB_BOUNDS_REGISTER("flash_decode_cluster.cu")

// Plan for `tiles` (= batch x kv heads x head tiles) tiles of at most `max_len` tokens, (cluster size << 16) | clusters: the size whose rounds
// of clusters, over the blocks that share a tile, are fewest; the smaller one of equals (a round costs a merge). 0: not a shape of this kernel.
// One block per tile from one tile per SM on, where clusters only add rounds (us, clusters of 1 / 2 blocks: 148 tiles of 16 heads 9.5 / 13 at 400
// tokens, 30 / 31 at 2000; 384 tiles of 4 heads 19 / 26 at 400), and where a tile has less than a page for each of sixteen warps (4 tiles of 16
// heads 6.4 / 8.9 at 150 tokens).
extern "C" int rmlx_flash_decode_cluster_plan(int batch, int tiles, int max_len, int HD, int kv_quant) {
  if (tiles < 1 || batch < 1 || batch > kFcMaxBatch || (HD != 64 && HD != 128)) return 0;
  const int pages = (max_len + kFcPage - 1) / kFcPage;
  if ((long long)pages * tiles > (1ll << 30)) return 0;
  const int largest = tiles >= sm_count() || pages < 4 * kFcWarps ? 1 : kFcMaxCluster;
  int best = 0;
  double best_cost = 1e30;
  for (int cs = 1; cs <= largest; cs *= 2) {
    if (cs > 1 && pages < cs * kFcWarps / 2) break;      // warps without a page
    const int n = HD == 128 ? (kv_quant ? fc_resident<128, true>(cs) : fc_resident<128, false>(cs))
                            : (kv_quant ? fc_resident<64, true>(cs) : fc_resident<64, false>(cs));
    if (n < 1) continue;
    const int rounds = (tiles + n - 1) / n;
    const double cost = rounds * (1.0 / cs + 0.15);      // a round's pages, and what its merge and first pages cost beside them
    if (cost < best_cost) { best_cost = cost; best = cs << 16 | (tiles < n ? tiles : n); }
  }
  return best;
}

// plan from rmlx_flash_decode_cluster_plan. k_sb null: bf16 cache, else the 8-bit one. `window` > 0: the last `window` tokens only.
extern "C" int rmlx_flash_decode_cluster(const void* q, const void* k_cache, const void* k_sb, const void* v_cache, const void* v_sb,
                                      const int* block_table, const int* seq_lens, void* out, int B, int Hq, int Hkv, int HD,
                                      int max_blocks, int table_stride, int plan, int window, float scale, int early, int pdl,
                                      cudaStream_t st) {
  const int cs = plan >> 16, clusters = plan & 0xffff;
  if (B < 1 || B > kFcMaxBatch || Hkv < 1 || Hq % Hkv || clusters < 1 || cs < 1 || cs > kFcMaxCluster || (cs & (cs - 1))) return -2;
  if ((k_sb == nullptr) != (v_sb == nullptr)) return -2;
  FcParams p = {};
  p.q = static_cast<const __nv_bfloat16*>(q);
  p.k_cache = static_cast<const char*>(k_cache); p.v_cache = static_cast<const char*>(v_cache);
  p.k_sb = static_cast<const char*>(k_sb); p.v_sb = static_cast<const char*>(v_sb);
  p.block_table = block_table; p.seq_lens = seq_lens;
  p.out = static_cast<__nv_bfloat16*>(out);
  p.B = B; p.max_blocks = max_blocks; p.table_stride = table_stride; p.Hq = Hq; p.Hkv = Hkv; p.G = Hq / Hkv; p.gtiles = (p.G + 15) / 16; p.window = window;
  p.early = early && pdl; p.CS = cs;
  p.scale_log2 = scale * 1.4426950408889634f;
  if (HD == 128) return k_sb ? fc_launch<128, true>(p, clusters, pdl, st) : fc_launch<128, false>(p, clusters, pdl, st);
  if (HD == 64) return k_sb ? fc_launch<64, true>(p, clusters, pdl, st) : fc_launch<64, false>(p, clusters, pdl, st);
  return -2;
}
