// C = A W^T for many rows on pairs of SMs (tcgen05 cta_group::2): the two blocks of a cluster hold 128 rows of A and 128 rows of
// W each and one product instruction multiplies both halves of A with both halves of W, a 256 x 256 tile with the accumulators of
// 128 rows in each block's tensor memory. W bf16 or MLX-affine 4-bit (expanded inside the main loop, as in xgemm_kernel.cuh), plain
// or grouped by expert, with SwiGLU or a residual in the epilogue.
//
// What bounds it: a one-SM tile of 128 x 256 is bound by shared memory (per 64 of K the products read 48 KB and 48 KB are written,
// at 128 bytes a cycle 750 cycles against 512 for the products; with 4-bit weights 112 KB, 875 cycles). A pair reads each half of W
// once for both: 64 KB (bf16) or 72 KB (4-bit) per SM, and each SM expands half as many weights per product.
//
// Roles per block (persistent, one pair per two SMs): warp 0 TMA producer of A (and bf16 W), warp 1 issues the products in the first
// block of the pair (in both it owns the tensor memory), warps 2-5 epilogue of the block's 128 rows; 4-bit weights: four groups of
// four dequant warps that take the k-blocks in turn, and a warp that asks for packed weights and scales. Packed weights come 128
// bytes of a row at a time, four k-blocks: the copy engine spends its time per row (32-byte pieces: 1300 cycles a k-block). Loads of
// both blocks count on the first one's barriers; the products' completion is committed to both. Every wait is bounded; both blocks
// meet before they leave, since each reads or signals the other's shared memory. Loads carry no cluster-broadcast qualifier.
#include "xgemm_kernel.cuh"

namespace rb {

constexpr int kPairRows = 128;        // rows of A and of W per block
constexpr int kPairN = 256;           // columns of the tile
constexpr int kPairDq = 16, kPairGroups = 4, kPairGroupWarps = kPairDq / kPairGroups;   // dequant warps, in groups

template <bool WQ4>
struct PairSmem {
  static constexpr int kStages = WQ4 ? 5 : 6;
  static constexpr int kRawStages = 3;
  static constexpr int kStageA = kPairRows * kXBK * 2, kStageB = kPairRows * kXBK * 2;
  static constexpr int kStageRaw = kPairRows * 128, kScaleSlot = 2 * kPairRows * 16;
  static constexpr int kBarBytes = 768;
  static constexpr int kBytes = kStages * (kStageA + kStageB) + (WQ4 ? kRawStages * kStageRaw + 2 * kScaleSlot : 0) + 1024 + kBarBytes +
                                (kXMaxExperts + 2) * 8;
  static constexpr int kThreads = 192 + (WQ4 ? 32 * kPairDq + 32 : 0);
};

__device__ __forceinline__ uint32_t pair_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void pair_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Address of the first block's copy of a shared-memory object.
__device__ __forceinline__ uint32_t pair_first(const void* p) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(a) : "r"(smem_u32(p)));
  return a;
}
// Signals and waits between the blocks have the default scope, the block's. That is a reliance, not something that the memory model
// gives: two of them order more than one block's accesses. What they order is what the tensor cores and the copy engine read or write
// (expanded weights behind each thread's proxy fence, accumulators behind the tcgen05 fences), in the memory of the SM whose threads
// wrote it, and no thread reads what the other block's threads stored; the pair tests compare every result bit for bit with the
// single-SM tiles over many runs. Release and acquire of cluster scope on the expanded weights' barrier alone cost a memory barrier
// per signal and an L1 invalidation per poll: 2048 rows of 28672 x 4096 336 -> 395 us, 4096 x 14336 173 -> 220.
__device__ __forceinline__ void pair_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
// A load into this block's shared memory that counts on a barrier of the pair's first block.
__device__ __forceinline__ void pair_load_2d(void* dst, const void* tmap, uint32_t bar, int32_t x, int32_t y) {
  asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
               ::"r"(smem_u32(dst)), "l"(tmap), "r"(bar), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void pair_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
               "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
               ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}
// Arrive on this barrier in both blocks once every product issued so far has completed.
__device__ __forceinline__ void pair_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(smem_u32(bar)), "h"(uint16_t(3)) : "memory");
}

template <bool WQ4, bool GROUPED, bool RESIDUAL>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(PairSmem<WQ4>::kThreads, 1)
pair_gemm_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_w,
                 const __grid_constant__ CUtensorMap tmap_s, const __grid_constant__ CUtensorMap tmap_b,
                 __nv_bfloat16* __restrict__ C, const __nv_bfloat16* __restrict__ residual, const int* __restrict__ offsets, int E,
                 int M, int N, int K, int ldc, int* __restrict__ status, int swiglu, float gate_limit) {
  using S = PairSmem<WQ4>;
  constexpr int STAGES = S::kStages, RAW = S::kRawStages;
  extern __shared__ char smem_raw[];
  char* smem = reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  char* sA = smem;
  char* sB = sA + STAGES * S::kStageA;
  char* sRaw = sB + STAGES * S::kStageB;
  char* sScale = sRaw + (WQ4 ? RAW * S::kStageRaw : 0);
  char* after = sScale + (WQ4 ? 2 * S::kScaleSlot : 0);
  uint64_t* full = reinterpret_cast<uint64_t*>(after);   // [STAGES] first block: the loads of both have landed
  uint64_t* empty = full + STAGES;                       // [STAGES] the products have read the stage
  uint64_t* bq_full = empty + STAGES;                    // [STAGES] first block: both halves of W expanded
  uint64_t* raw_full = bq_full + STAGES;                 // [RAW]
  uint64_t* raw_empty = raw_full + RAW;                  // [RAW]
  uint64_t* sc_full = raw_empty + RAW;                   // [2]
  uint64_t* sc_empty = sc_full + 2;                      // [2]
  uint64_t* acc_full = sc_empty + 2;                     // [2]
  uint64_t* acc_empty = acc_full + 2;                    // [2] first block: both epilogues have read the accumulators
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  volatile uint32_t* abort_flag = tmem_slot + 1;
  int* s_off = reinterpret_cast<int*>(after + S::kBarBytes);         // [E+1]
  int* s_tprefix = s_off + kXMaxExperts + 1;                         // [E+1]

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = int(pair_rank());
  const int tiles_n = (N + kPairN - 1) / kPairN, tiles_m = (M + 2 * kPairRows - 1) / (2 * kPairRows);
  const int num_kb = (K + kXBK - 1) / kXBK;

  if (threadIdx.x == 0) {
    for (int i = 0; i < STAGES; ++i) { mbar_init(full + i, 1); mbar_init(empty + i, 1); mbar_init(bq_full + i, 2 * kPairGroupWarps); }
    for (int i = 0; i < RAW; ++i) { mbar_init(raw_full + i, 1); mbar_init(raw_empty + i, kPairDq); }
    for (int i = 0; i < 2; ++i) {
      mbar_init(sc_full + i, 1); mbar_init(sc_empty + i, kPairDq);
      mbar_init(acc_full + i, 1); mbar_init(acc_empty + i, 8);
    }
    *abort_flag = 0u;
    fence_mbar_init();
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  pdl_wait();
  if (GROUPED)
    for (int i = threadIdx.x; i <= E; i += blockDim.x) {
      const int o = offsets[i];
      s_off[i] = RB_BOUNDS(o, M + 1) ? o : 0;
    }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  if (GROUPED) {
    if (threadIdx.x == 0) {
      int acc = 0;
      for (int e = 0; e < E; ++e) {
        s_tprefix[e] = acc;
        const int n = s_off[e + 1] - s_off[e];
        if (RB_BOUNDS(n, M + 1)) acc += ((n + 2 * kPairRows - 1) / (2 * kPairRows)) * tiles_n;
      }
      s_tprefix[E] = acc;
    }
    __syncthreads();
  }
  pair_sync();                                           // both blocks' barriers exist before either signals the other
  const int num_tiles = GROUPED ? s_tprefix[E] : tiles_m * tiles_n;
  const uint32_t tmem_base = *tmem_slot;
  const int first = blockIdx.x >> 1, step = gridDim.x >> 1;

  // tile -> this block's first rows of A, W and C. Column-major over row blocks, so that pairs working at the same time share W.
  // SwiGLU: the first block holds 128 gate rows of W, the second the matching up rows.
  auto locate = [&](int tile) {
    XTile t;
    int tm, tn, w0 = 0;
    if (!GROUPED) {
      tm = tile % tiles_m; tn = tile / tiles_m;
      t.a_row0 = tm * (2 * kPairRows); t.row_end = M;
    } else {
      int e = 0;
      while (s_tprefix[e + 1] <= tile) ++e;
      const int rows = s_off[e + 1] - s_off[e], mt = (rows + 2 * kPairRows - 1) / (2 * kPairRows), local = tile - s_tprefix[e];
      tm = local % mt; tn = local / mt; w0 = e * N;
      t.a_row0 = s_off[e] + tm * (2 * kPairRows); t.row_end = s_off[e + 1];
    }
    t.a_row0 += rank * kPairRows;
    t.w_row0 = w0 + (swiglu ? tn * kPairRows + rank * (N / 2) : tn * kPairN + rank * kPairRows);
    t.c_col0 = tn * (swiglu ? kPairRows : kPairN);
    return t;
  };

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (elect_one()) {
      tma_prefetch_desc(&tmap_a);
      tma_prefetch_desc(&tmap_w);
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int tile = first; tile < num_tiles && ok; tile += step) {
        const XTile t = locate(tile);
        for (int kb = 0; kb < num_kb; ++kb) {
          if (!mbar_wait(empty + stage, phase ^ 1u, abort_flag)) { ok = false; break; }
          if (rank == 0) mbar_arrive_expect_tx(full + stage, 2 * (S::kStageA + (WQ4 ? 0 : S::kStageB)));
          const uint32_t bar = pair_first(full + stage);
          pair_load_2d(sA + stage * S::kStageA, &tmap_a, bar, kb * kXBK, t.a_row0);
          if (!WQ4) pair_load_2d(sB + stage * S::kStageB, &tmap_w, bar, kb * kXBK, t.w_row0);
          if (++stage == STAGES) { stage = 0; phase ^= 1u; }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ products (first block)
    if (rank == 0 && elect_one()) {
      constexpr uint32_t idesc = umma_idesc_bf16_f32(2 * kPairRows, kPairN);
      int stage = 0, acc = 0;
      uint32_t phase = 0, acc_phase = 0;
      bool ok = true;
      for (int tile = first; tile < num_tiles && ok; tile += step) {
        if (!mbar_wait(acc_empty + acc, acc_phase ^ 1u, abort_flag)) { ok = false; break; }
        tc_fence_after_sync();
        const uint32_t d_tmem = tmem_base + acc * kPairN;
        for (int kb = 0; kb < num_kb; ++kb) {
          if (!mbar_wait(full + stage, phase, abort_flag)) { ok = false; break; }
          if (WQ4 && !mbar_wait(bq_full + stage, phase, abort_flag)) { ok = false; break; }
          tc_fence_after_sync();
          const uint32_t a_addr = smem_u32(sA + stage * S::kStageA), b_addr = smem_u32(sB + stage * S::kStageB);
#pragma unroll
          for (int k = 0; k < kXBK / 16; ++k)
            pair_mma(d_tmem, umma_desc_sw128_kmajor(a_addr + k * 32), umma_desc_sw128_kmajor(b_addr + k * 32), idesc,
                     (kb | k) != 0 ? 1u : 0u);
          pair_commit(empty + stage);
          if (++stage == STAGES) { stage = 0; phase ^= 1u; }
        }
        if (!ok) break;
        pair_commit(acc_full + acc);
        if (++acc == 2) { acc = 0; acc_phase ^= 1u; }
      }
    }
  } else if (warp < 6) {
    // ------------------------------------------------------------------ epilogue (warps 2..5) of this block's rows
    const int q = warp & 3;
    int acc = 0;
    uint32_t acc_phase = 0;
    for (int tile = first; tile < num_tiles; tile += step) {
      const XTile t = locate(tile);
      if (!mbar_wait(acc_full + acc, acc_phase, abort_flag)) break;
      tc_fence_after_sync();
      const int row = t.a_row0 + q * 32 + lane;
      const uint32_t t_row = tmem_base + acc * kPairN + (uint32_t(q * 32) << 16);
      const int n_out = swiglu ? N / 2 : N;
      if (swiglu) {
#pragma unroll 1
        for (int c = 0; c < kPairRows / 32; ++c) {
          uint32_t rg[32], ru[32];
          tmem_ld_32x32(t_row + c * 32, rg);
          tmem_ld_32x32(t_row + kPairRows + c * 32, ru);
          tmem_ld_wait();
          const int col0 = t.c_col0 + c * 32;
          if (row < t.row_end && col0 < n_out) {          // n_out is a multiple of 128
            __nv_bfloat16* dst = C + size_t(row) * ldc + col0;
#pragma unroll
            for (int v = 0; v < 4; ++v) {
              float f[8];
#pragma unroll
              for (int j = 0; j < 8; ++j)
                f[j] = gated_act_fast(__uint_as_float(rg[v * 8 + j]), __uint_as_float(ru[v * 8 + j]), gate_limit);
              uint4 o;
              o.x = pack_bf16(f[0], f[1]); o.y = pack_bf16(f[2], f[3]);
              o.z = pack_bf16(f[4], f[5]); o.w = pack_bf16(f[6], f[7]);
              *reinterpret_cast<uint4*>(dst + v * 8) = o;
            }
          }
        }
      } else {
#pragma unroll 1
        for (int c = 0; c < kPairN / 32; ++c) {
          uint32_t r[32];
          tmem_ld_32x32(t_row + c * 32, r);
          tmem_ld_wait();
          const int col0 = t.c_col0 + c * 32;
          if (row < t.row_end && col0 < n_out) {          // N is a multiple of 32
            __nv_bfloat16* dst = C + size_t(row) * ldc + col0;
            const __nv_bfloat16* res = RESIDUAL ? residual + size_t(row) * ldc + col0 : nullptr;
#pragma unroll
            for (int v = 0; v < 4; ++v) {
              float f[8];
#pragma unroll
              for (int j = 0; j < 8; ++j) f[j] = __uint_as_float(r[v * 8 + j]);
              if (RESIDUAL) {
                const uint4 rv = *reinterpret_cast<const uint4*>(res + v * 8);
                f[0] += bf16lo(rv.x); f[1] += bf16hi(rv.x); f[2] += bf16lo(rv.y); f[3] += bf16hi(rv.y);
                f[4] += bf16lo(rv.z); f[5] += bf16hi(rv.z); f[6] += bf16lo(rv.w); f[7] += bf16hi(rv.w);
              }
              uint4 o;
              o.x = pack_bf16(f[0], f[1]); o.y = pack_bf16(f[2], f[3]);
              o.z = pack_bf16(f[4], f[5]); o.w = pack_bf16(f[6], f[7]);
              *reinterpret_cast<uint4*>(dst + v * 8) = o;
            }
          }
        }
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) pair_arrive(pair_first(acc_empty + acc));
      if (++acc == 2) { acc = 0; acc_phase ^= 1u; }
    }
  } else if (WQ4 && warp == 6 + kPairDq) {
    // ------------------------------------------------------------------ packed weights, scales and biases of this block's half
    if (elect_one()) {
      int rstage = 0, sslot = 0;
      uint32_t rphase = 0, sphase = 0;
      bool ok = true;
      for (int tile = first; tile < num_tiles && ok; tile += step) {
        const XTile t = locate(tile);
        for (int kb = 0; kb < num_kb; ++kb) {
          if ((kb & 7) == 0) {
            if (!mbar_wait(sc_empty + sslot, sphase ^ 1u, abort_flag)) { ok = false; break; }
            mbar_arrive_expect_tx(sc_full + sslot, S::kScaleSlot);
            char* sd = sScale + sslot * S::kScaleSlot;
            tma_load_2d(sd, &tmap_s, sc_full + sslot, kb, t.w_row0);
            tma_load_2d(sd + kPairRows * 16, &tmap_b, sc_full + sslot, kb, t.w_row0);
            if (++sslot == 2) { sslot = 0; sphase ^= 1u; }
          }
          if ((kb & 3) == 0) {
            if (!mbar_wait(raw_empty + rstage, rphase ^ 1u, abort_flag)) { ok = false; break; }
            mbar_arrive_expect_tx(raw_full + rstage, S::kStageRaw);
            tma_load_2d(sRaw + rstage * S::kStageRaw, &tmap_w, raw_full + rstage, kb * 32, t.w_row0);
            if (++rstage == RAW) { rstage = 0; rphase ^= 1u; }
          }
        }
      }
    }
  } else if (WQ4) {
    // ------------------------------------------------------------------ dequant: a thread expands a row of the k-block
    // A k-block is a chain of some 200 dependent instructions, two waits and a fence: what hides it is k-blocks at the same time,
    // so four groups take them in turn (two groups of eight warps: 1350 cycles a k-block, however little of it each did).
    const int r = (threadIdx.x - 192) % (32 * kPairGroupWarps), group = (threadIdx.x - 192) / (32 * kPairGroupWarps);
    int stage = group, rstage = 0, sslot = 0;
    uint32_t phase = 0, rphase = 0, sphase = 0;
    bool ok = true;
    const uint32_t half_sel = (group & 1) ? 0x3232u : 0x1010u;
    for (int tile = first; tile < num_tiles && ok; tile += step) {
      for (int kb8 = 0; kb8 < num_kb && ok; kb8 += 8) {   // K % 512 == 0: whole groups of 8
        if (!mbar_wait(sc_full + sslot, sphase, abort_flag)) { ok = false; break; }
        const uint32_t scb = smem_u32(sScale) + sslot * S::kScaleSlot + r * 16 + (group >> 1) * 4;
        uint32_t sws[2], bws[2];                          // k-blocks kb8 + group and kb8 + 4 + group, each the half_sel half
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          sws[i] = x_lds32(scb + i * 8);
          bws[i] = x_lds32(scb + kPairRows * 16 + i * 8);
        }
#pragma unroll
        for (int k4 = 0; k4 < 2; ++k4) {
          if (!mbar_wait(raw_full + rstage, rphase, abort_flag)) { ok = false; break; }
          // this k-block's 32 bytes of the row's 128 (eight lanes, eight rows: with the swizzle every bank once)
          const uint32_t raw = smem_u32(sRaw) + rstage * S::kStageRaw + r * 128;
          const uint4 w0 = x_lds(raw + (((2 * group) ^ (r & 7)) << 4));
          const uint4 w1 = x_lds(raw + (((2 * group + 1) ^ (r & 7)) << 4));
          const uint32_t s2u = __byte_perm(sws[k4], 0u, half_sel), b2u = __byte_perm(bws[k4], 0u, half_sel);
          const __nv_bfloat162 s2 = *reinterpret_cast<const __nv_bfloat162*>(&s2u);
          const __nv_bfloat162 b2 = *reinterpret_cast<const __nv_bfloat162*>(&b2u);
          const uint32_t words[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
          if (!mbar_wait(empty + stage, phase ^ 1u, abort_flag)) { ok = false; break; }
          const uint32_t bst = smem_u32(sB) + stage * S::kStageB + r * 128;
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            uint32_t o[4];
            x_expand(words[j], s2, b2, o);
            x_sts(bst + ((j ^ (r & 7)) << 4), o);
          }
          fence_proxy_async_smem();     // generic-proxy stores -> visible to the tensor cores' reads
          __syncwarp();
          if (lane == 0) {
            pair_arrive(pair_first(bq_full + stage));
            mbar_arrive(raw_empty + rstage);
          }
          if (++rstage == RAW) { rstage = 0; rphase ^= 1u; }
          stage += kPairGroups;
          if (stage >= STAGES) { stage -= STAGES; phase ^= 1u; }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(sc_empty + sslot);     // only once the scales have been used (xgemm_kernel.cuh says why)
        if (++sslot == 2) { sslot = 0; sphase ^= 1u; }
      }
    }
  }

  tc_fence_before_sync();
  __syncthreads();
  pair_sync();                                           // the other block neither reads nor signals this one any more
  if (warp == 1) {
    tc_fence_after_sync();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
  }
  if (threadIdx.x == 0 && *abort_flag && status) atomicExch(status, kStatusMbarTimeout);
  pdl_launch_dependents();
}

template <bool WQ4, bool GROUPED, bool RESIDUAL>
static int launch_pair(const CUtensorMap& ta, const CUtensorMap& tw, const CUtensorMap& ts, const CUtensorMap& tb, void* C,
                       const void* residual, const int* offsets, int E, int M, int N, int K, int ldc, int* status, int swiglu,
                       float gate_limit, int pdl, cudaStream_t st) {
  using S = PairSmem<WQ4>;
  static_assert(S::kBytes <= 227 * 1024, "shared memory");
  static_assert((3 * S::kStages + 2 * S::kRawStages + 8) * 8 + 8 <= S::kBarBytes, "barriers");
  auto kern = pair_gemm_kernel<WQ4, GROUPED, RESIDUAL>;
  RB_CHECK(set_max_smem(kern, S::kBytes));
  const long long tiles = (GROUPED ? (M + 255) / 256 + E : (M + 255) / 256) * (long long)((N + kPairN - 1) / kPairN);
  const int pairs = sm_count() / 2;
  return launch(kern, dim3(2 * int(tiles < pairs ? tiles : pairs)), dim3(S::kThreads), size_t(S::kBytes), st, pdl != 0, ta, tw, ts, tb,
                static_cast<__nv_bfloat16*>(C), static_cast<const __nv_bfloat16*>(residual), offsets, E, M, N, K, ldc, status, swiglu,
                gate_limit);
}

}  // namespace rb

using namespace rb;
RB_BOUNDS_REGISTER("pair_gemm.cu")

// Shapes of the pair kernel: whole 32-column pieces (SwiGLU, grouped: whole tiles), 16-byte rows.
extern "C" int rmlx_pair_gemm_supported(int w_kind, int N, int K, int ldc, int grouped, int swiglu) {
  if (w_kind < 0 || w_kind > 1 || N % 32 || K % 8 || ldc % 8) return 0;
  if ((grouped || swiglu) && N % 256) return 0;
  return w_kind == 0 || K % 512 == 0;
}

// As rmlx_xgemm (bf16 or 4-bit weights, plain or grouped, residual or SwiGLU), on 256 x 256 tiles of SM pairs.
extern "C" int rmlx_pair_gemm(int w_kind, const void* A, const void* W, const void* scales, const void* biases, void* C,
                              const void* residual, const int* offsets, int E, int M, int N, int K, int lda, int ldc, int swiglu,
                              float gate_limit, int* status, int pdl, cudaStream_t st) {
  if (M < 1 || lda % 8 || !rmlx_pair_gemm_supported(w_kind, N, K, ldc, offsets != nullptr, swiglu)) return -2;
  const bool grouped = offsets != nullptr;
  if (grouped && (E < 1 || E > kXMaxExperts)) return -2;
  if (residual && (swiglu || grouped)) return -2;
  CUtensorMap ta, tw, ts, tb;
  int rc = make_tmap_2d_bf16(&ta, A, uint64_t(K), uint64_t(M), uint64_t(lda) * 2, kXBK, kPairRows);
  if (rc) return rc;
  const uint64_t rows_w = grouped ? uint64_t(E) * N : uint64_t(N);
  rc = x_weight_maps(w_kind, W, scales, biases, rows_w, K, kPairRows, &tw, &ts, &tb, 4);
  if (rc) return rc;
#define RB_PAIR(Q_, G_, R_)                                                                                                    \
  return launch_pair<Q_, G_, R_>(ta, tw, ts, tb, C, residual, offsets, E, M, N, K, ldc, status, swiglu, gate_limit, pdl, st)
  if (w_kind == 1) {
    if (grouped) RB_PAIR(true, true, false);
    if (residual) RB_PAIR(true, false, true);
    RB_PAIR(true, false, false);
  }
  if (grouped) RB_PAIR(false, true, false);
  if (residual) RB_PAIR(false, false, true);
  RB_PAIR(false, false, false);
#undef RB_PAIR
}
