// C = A W^T with 4-bit weights for a few to some hundred rows per weight matrix: experts of a prompt, decode batches, the LM head. The
// 128 rows of the products are rows of W, the columns rows of A, as many as there are (16 to 160 at a time).
//
// What bounds the other way round (xgemm_kernel.cuh, rows of A as the products' rows): a tile of 128 rows of A that is mostly
// padding costs as much as a full one, an expert of 130 rows two of them, each with all of W expanded again, and every expanded
// weight is written to shared memory and read from there, which at 128 bytes a cycle takes longer than the products. Here
//   * W is expanded once for up to 160 rows of A, and a tile costs what its rows need: the products' N is their number rounded up to 16;
//   * expanded weights go to tensor memory (tcgen05.st), from where the products take their A operand: shared memory carries the packed
//     weights and the rows of A only. A thread expands 64 values of one row of W and stores them as its lane's 32 columns: no swizzle;
//   * where one tile per SM would leave SMs idle (decode batches), the blocks of a cluster take K apart and add their sums through
//     distributed shared memory, in the order of their ranks.
//
// Roles per block (persistent): warp 0 asks for rows of A (TMA, 32 at a time), warp 1 issues the products and owns the tensor memory
// (two accumulators of 160 columns, three stages of 64 columns of expanded weights), warps 2-5 epilogue, three groups of four
// dequant warps that take the stages in turn, and a warp that asks for packed weights and scales, 128 bytes of a row at a time. A stage is
// 128 of K: a wait, a commit and a handover cost the one thread that issues products some 400 cycles however little there is to multiply (64
// of K a stage, four stages: 500 cycles each with 16 rows of A; rows of A and W counted on one barrier instead of two: 600 before).
// Every wait is bounded.
//
// Measured (us, single-SM or pair tiles / this): 128 experts of 4096 x 1536, gate and up 637 / 404 and down 415 / 264 at 128 rows each (the
// products' floor 250 + 125), 439 / 336 and 250 / 186 at 64, 429 / 324 and 242 / 167 at 16 (of which 75 the expansion's instructions and
// 210 what is left with neither expansion nor products); 4096 x 8192 at 64 rows 47 / 22, 9216 x 4096 27 / 24, 151936 x 4096 172 / 140.
// Six groups of dequant warps (64 registers) are faster below 32 rows each (283 for 324) and slower above (430 for 404).
#include "xgemm_kernel.cuh"

namespace rb {

constexpr int kRgRows = 128, kRgCols = 160;              // rows of W, rows of A per tile
constexpr int kRgStages = 3, kRgRawStages = 4, kRgBox = 32;   // a stage: two k-blocks of 64; packed weights: four
constexpr int kRgDq = 4 * kRgStages, kRgThreads = 192 + 32 * kRgDq + 32;
constexpr int kRgMaxSplit = 8;

struct RgParams {
  void* C;
  const __nv_bfloat16* residual;
  const int* offsets;            // [E + 1]; null: one matrix, all M rows
  int* status;
  int E, M, N, K, ldc, out_f32, swiglu, split;
  int boxes;                     // boxes of 32 rows of A per k-block
  float gate_limit;
};

struct RgSmem {
  static constexpr int kRaw = kRgRows * 128, kScale = 2 * kRgRows * 16, kBars = 512;
  static int bytes(int boxes, int split) {
    return kRgStages * 2 * boxes * kRgBox * 128 + kRgRawStages * kRaw + 2 * kScale + (split > 1 ? boxes * kRgBox * kRgRows * 4 : 0) + 1024 +
           kBars + (kXMaxExperts + 2) * 8;
  }
};

// D (+)= A B: A from tensor memory (a row of A per lane, two values per column), B from shared memory.
__device__ __forceinline__ void rg_mma(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
               "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
               ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}
// Arrive on a peer's copy of a barrier, releasing to the cluster; wait on this block's, acquiring.
__device__ __forceinline__ void rg_arrive(uint64_t* bar, int rank) {
  asm volatile("{.reg .u32 a; mapa.shared::cluster.u32 a, %0, %1; mbarrier.arrive.release.cluster.shared::cluster.b64 _, [a];}"
               ::"r"(smem_u32(bar)), "r"(rank) : "memory");
}
__device__ __forceinline__ bool rg_wait(uint64_t* bar, uint32_t parity, volatile uint32_t* abort_flag) {
  for (uint32_t i = 0; i < kMbarPollLimit; ++i) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    if (ok) return true;
    if ((i & 63u) == 63u && *abort_flag) return false;
  }
  *abort_flag = 1u;
  return false;
}
// A wait's outcome for the whole warp, whose next instructions are warp-wide.
__device__ __forceinline__ bool rg_all(bool ok) { return __all_sync(0xffffffffu, ok); }
__device__ __forceinline__ float rg_remote(uint32_t addr, int rank) {
  float v;
  asm volatile("{.reg .u32 a; mapa.shared::cluster.u32 a, %1, %2; ld.shared::cluster.f32 %0, [a];}" : "=f"(v) : "r"(addr), "r"(rank) : "memory");
  return v;
}

__global__ void __launch_bounds__(kRgThreads, 1)
row_gemm_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_w,
                const __grid_constant__ CUtensorMap tmap_s, const __grid_constant__ CUtensorMap tmap_b, const RgParams p) {
  extern __shared__ char smem_raw[];
  char* const smem = reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int half_a = p.boxes * kRgBox * 128, stage_a = 2 * half_a;
  char* const sA = smem;                                 // rows of A
  char* const sRaw = sA + kRgStages * stage_a;
  char* const sScale = sRaw + kRgRawStages * RgSmem::kRaw;
  float* const sRed = reinterpret_cast<float*>(sScale + 2 * RgSmem::kScale);   // [row of A][row of W] sums of this block's share of K
  char* const after = reinterpret_cast<char*>(sRed) + (p.split > 1 ? p.boxes * kRgBox * kRgRows * 4 : 0);
  uint64_t* const full = reinterpret_cast<uint64_t*>(after);   // [STAGES] rows of A have landed and W is expanded
  uint64_t* const empty = full + kRgStages;              // [STAGES] the products have read the stage
  uint64_t* const raw_full = empty + kRgStages;          // [RAW]
  uint64_t* const raw_empty = raw_full + kRgRawStages;   // [RAW]
  uint64_t* const sc_full = raw_empty + kRgRawStages;    // [2]
  uint64_t* const sc_empty = sc_full + 2;                // [2]
  uint64_t* const acc_full = sc_empty + 2;               // [2]
  uint64_t* const acc_empty = acc_full + 2;              // [2]
  uint64_t* const red_full = acc_empty + 2;              // all blocks of the cluster have put their sums
  uint64_t* const red_empty = red_full + 1;              // and have read this block's
  uint32_t* const tmem_slot = reinterpret_cast<uint32_t*>(red_empty + 1);
  volatile uint32_t* const abort_flag = tmem_slot + 1;
  int* const s_off = reinterpret_cast<int*>(after + RgSmem::kBars);   // [E + 1]
  int* const s_pre = s_off + kXMaxExperts + 1;           // [E + 1] tiles before every expert

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int rank = 0;
  if (p.split > 1) asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  const int tiles_n = p.N / kRgRows, kb8 = p.K / 512;
  const int kb_first = kb8 * rank / p.split * 8, kb_end = kb8 * (rank + 1) / p.split * 8;   // this block's k-blocks of 64

  if (threadIdx.x == 0) {
    for (int i = 0; i < kRgStages; ++i) { mbar_init(full + i, 1 + 4); mbar_init(empty + i, 1); }
    for (int i = 0; i < kRgRawStages; ++i) { mbar_init(raw_full + i, 1); mbar_init(raw_empty + i, 2 * 4); }
    for (int i = 0; i < 2; ++i) {
      mbar_init(sc_full + i, 1); mbar_init(sc_empty + i, 4 * 4);
      mbar_init(acc_full + i, 1); mbar_init(acc_empty + i, 4);
    }
    mbar_init(red_full, 4 * p.split); mbar_init(red_empty, 4 * p.split);
    *abort_flag = 0u;
    fence_mbar_init();
  }
  if (warp == 1) { tmem_alloc(tmem_slot, 512); tmem_relinquish(); }
  pdl_wait();
  if (p.offsets) {
    for (int i = threadIdx.x; i <= p.E; i += blockDim.x) {
      const int o = p.offsets[i];
      s_off[i] = RB_BOUNDS(o, p.M + 1) ? o : 0;
    }
  } else if (threadIdx.x == 0) {
    s_off[0] = 0; s_off[1] = p.M;
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  if (warp == 0) {       // tiles before every expert: a scan over 32 experts at a time
    int base = 0;
    for (int e0 = 0; e0 < p.E; e0 += 32) {
      const int e = e0 + lane;
      const int n = e < p.E ? s_off[e + 1] - s_off[e] : 0;
      const int mine = RB_BOUNDS(n, p.M + 1) ? (n + kRgCols - 1) / kRgCols * tiles_n : 0;
      int sum = mine;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) { const int v = __shfl_up_sync(0xffffffffu, sum, o); if (lane >= o) sum += v; }
      if (e < p.E) s_pre[e] = base + sum - mine;
      base += __shfl_sync(0xffffffffu, sum, 31);
    }
    if (lane == 0) s_pre[p.E] = base;
  }
  __syncthreads();
  if (p.split > 1) asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  const int num_tiles = s_pre[p.E];
  const uint32_t tmem_base = *tmem_slot, tmem_w = tmem_base + 2 * kRgCols;
  const int first = int(blockIdx.x) / p.split, step = int(gridDim.x) / p.split;

  // tile -> first row of A, their number, first rows of W (two runs of 64: with SwiGLU gate rows and the matching up rows), first
  // column of C. The rows of A vary fastest, so that blocks working at the same time share W. e: an expert at or before the tile's.
  struct Tile { int a_row0, rows, w0, w1, col0; };
  auto locate = [&](int tile, int& e) {
    while (s_pre[e + 1] <= tile) ++e;
    const int n = s_off[e + 1] - s_off[e], mt = (n + kRgCols - 1) / kRgCols, local = tile - s_pre[e];
    const int tn = local / mt, tm = local - tn * mt, per = ((n + mt - 1) / mt + 15) & ~15;
    Tile t;
    t.a_row0 = s_off[e] + tm * per;
    t.rows = min(per, n - tm * per);
    t.w0 = e * p.N + (p.swiglu ? tn * (kRgRows / 2) : tn * kRgRows);
    t.w1 = t.w0 + (p.swiglu ? p.N / 2 : kRgRows / 2);
    t.col0 = tn * (p.swiglu ? kRgRows / 2 : kRgRows);
    return t;
  };

  if (warp == 0) {
    // ------------------------------------------------------------------ rows of A
    if (elect_one()) {
      tma_prefetch_desc(&tmap_a);
      int stage = 0, e = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int tile = first; tile < num_tiles && ok; tile += step) {
        const Tile t = locate(tile, e);
        const int boxes = (t.rows + kRgBox - 1) / kRgBox;
        for (int kb = kb_first; kb < kb_end; kb += 2) {
          if (!mbar_wait(empty + stage, phase ^ 1u, abort_flag)) { ok = false; break; }
          mbar_arrive_expect_tx(full + stage, 2 * boxes * kRgBox * 128);
          for (int b = 0; b < boxes; ++b)
            for (int h = 0; h < 2; ++h)
              tma_load_2d(sA + stage * stage_a + h * half_a + b * kRgBox * 128, &tmap_a, full + stage, (kb + h) * kXBK, t.a_row0 + b * kRgBox);
          if (++stage == kRgStages) { stage = 0; phase ^= 1u; }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ products
    if (elect_one()) {
      // one thread, whose instructions follow one another: nothing is computed here that does not change
      const uint64_t desc = umma_desc_sw128_kmajor(smem_u32(sA));
      const uint32_t half_desc = uint32_t(half_a) >> 4;
      int acc = 0, e = 0, stage = 0;
      uint32_t phase = 0, acc_phase = 0;
      bool ok = true;
      for (int tile = first; tile < num_tiles && ok; tile += step) {
        const Tile t = locate(tile, e);
        const uint32_t idesc = umma_idesc_bf16_f32(kRgRows, (t.rows + 15) & ~15), d = tmem_base + acc * kRgCols;
        if (!mbar_wait(acc_empty + acc, acc_phase ^ 1u, abort_flag)) { ok = false; break; }
        tc_fence_after_sync();
        uint32_t more = 0;
        for (int kb = kb_first; kb < kb_end; kb += 2) {
          if (!mbar_wait(full + stage, phase, abort_flag)) { ok = false; break; }
          tc_fence_after_sync();
          const uint64_t b = desc + uint32_t(stage * 2) * half_desc;
          const uint32_t a = tmem_w + stage * 64;
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            rg_mma(d, a + k * 8, b + (k >> 2) * half_desc + (k & 3) * 2, idesc, more);
            more = 1u;
          }
          tc_commit(empty + stage);
          if (++stage == kRgStages) { stage = 0; phase ^= 1u; }
        }
        if (!ok) break;
        tc_commit(acc_full + acc);
        if (++acc == 2) { acc = 0; acc_phase ^= 1u; }
      }
    }
  } else if (warp < 6) {
    // ------------------------------------------------------------------ epilogue: a lane is a row of W
    const int q = warp & 3, half = lane >> 4;
    int acc = 0, e = 0;
    uint32_t acc_phase = 0, red_phase = 0;
    // the results v of this lane's row of W and rows of A a0 .. (those below `rows`); lanes 2i and 2i + 1 hold neighbouring columns
    auto put = [&](const Tile& t, int a0, const float* v, int count, int col) {
      if (p.out_f32) {
        float* const c = static_cast<float*>(p.C) + size_t(t.a_row0) * p.ldc + col;
#pragma unroll
        for (int i = 0; i < 32; ++i)
          if (i < count && a0 + i < t.rows) c[size_t(a0 + i) * p.ldc] = v[i];
      } else {
        const int odd = lane & 1;
        __nv_bfloat16* const c = static_cast<__nv_bfloat16*>(p.C) + size_t(t.a_row0) * p.ldc + (col - odd);
        const __nv_bfloat16* const r = p.residual ? p.residual + size_t(t.a_row0) * p.ldc + (col - odd) : nullptr;
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          if (i >= count) break;
          const float got = __shfl_xor_sync(0xffffffffu, odd ? v[i] : v[i + 1], 1);
          float lo = odd ? got : v[i], hi = odd ? v[i + 1] : got;
          const int row = a0 + i + odd;
          if (row < t.rows) {
            if (r) {
              const uint32_t w = *reinterpret_cast<const uint32_t*>(r + size_t(row) * p.ldc);
              lo += bf16lo(w); hi += bf16hi(w);
            }
            *reinterpret_cast<uint32_t*>(c + size_t(row) * p.ldc) = pack_bf16(lo, hi);
          }
        }
      }
    };
    for (int tile = first; tile < num_tiles; tile += step) {
      const Tile t = locate(tile, e);
      if (!rg_all(mbar_wait(acc_full + acc, acc_phase, abort_flag))) break;
      tc_fence_after_sync();
      const uint32_t t_row = tmem_base + acc * kRgCols + (uint32_t(q * 32) << 16);
      const int col = t.col0 + (p.swiglu ? q * 16 + (lane & 15) : q * 32 + lane);
      if (p.split > 1 && !rg_all(rg_wait(red_empty, red_phase ^ 1u, abort_flag))) break;
#pragma unroll 1
      for (int c = 0; c < t.rows; c += 32) {
        uint32_t r[32];
        tmem_ld_32x32(t_row + c, r);
        tmem_ld_wait();
        if (p.split > 1) {
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (c + i < t.rows) sRed[(c + i) * kRgRows + q * 32 + lane] = __uint_as_float(r[i]);
        } else if (p.swiglu) {
          // lanes 0-15 hold gate rows, 16-31 the matching up rows: each half takes sixteen rows of A
          float v[32];
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const uint32_t got = __shfl_xor_sync(0xffffffffu, half ? r[i] : r[16 + i], 16);
            const uint32_t gate = half ? got : r[i], up = half ? r[16 + i] : got;
            v[i] = gated_act_fast(__uint_as_float(gate), __uint_as_float(up), p.gate_limit);
          }
          put(t, c + half * 16, v, 16, col);
        } else {
          float v[32];
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
          put(t, c, v, 32, col);
        }
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(acc_empty + acc);
      if (++acc == 2) { acc = 0; acc_phase ^= 1u; }
      if (p.split > 1) {
        // every block adds up its share of the rows of A
        if (lane < p.split) rg_arrive(red_full, lane);
        if (!rg_all(rg_wait(red_full, red_phase, abort_flag))) break;
        const int per = ((t.rows + p.split - 1) / p.split + 1) & ~1, c1 = min(t.rows, (rank + 1) * per);
        const uint32_t mine = smem_u32(sRed + q * 32 + lane), pair = smem_u32(sRed + (q * 32 + (lane ^ 16)));
        // four rows of A at a time, all blocks' sums asked for before the first is added: what this costs is their latency
        auto sums = [&](uint32_t at, int c, float (&v)[32]) {
          float f[4][kRgMaxSplit];
#pragma unroll
          for (int k = 0; k < kRgMaxSplit; ++k)
            if (k < p.split) {
#pragma unroll
              for (int i = 0; i < 4; ++i) f[i][k] = rg_remote(at + min(c + i, c1 - 1) * (kRgRows * 4), k);
            }
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            float s = f[i][0];
#pragma unroll
            for (int k = 1; k < kRgMaxSplit; ++k)
              if (k < p.split) s += f[i][k];
            v[i] = s;
          }
        };
        Tile u = t;
        u.rows = (!p.swiglu || half == 0) ? c1 : 0;      // SwiGLU: both halves have the same results, one stores them
#pragma unroll 1
        for (int c = rank * per; c < c1; c += 4) {
          float v[32];
          sums(mine, c, v);
          if (p.swiglu) {
            float o[32];
            sums(pair, c, o);
#pragma unroll
            for (int i = 0; i < 4; ++i) v[i] = gated_act_fast(half ? o[i] : v[i], half ? v[i] : o[i], p.gate_limit);
          }
          put(u, c, v, 4, col);
        }
        __syncwarp();
        if (lane < p.split) rg_arrive(red_empty, lane);
        red_phase ^= 1u;
      }
    }
  } else if (warp == 6 + kRgDq) {
    // ------------------------------------------------------------------ packed weights, scales and biases
    if (elect_one()) {
      tma_prefetch_desc(&tmap_w);
      int rstage = 0, sslot = 0, e = 0;
      uint32_t rphase = 0, sphase = 0;
      bool ok = true;
      for (int tile = first; tile < num_tiles && ok; tile += step) {
        const Tile t = locate(tile, e);
        for (int kb = kb_first; kb < kb_end; kb += 4) {
          if ((kb & 7) == 0) {
            if (!mbar_wait(sc_empty + sslot, sphase ^ 1u, abort_flag)) { ok = false; break; }
            mbar_arrive_expect_tx(sc_full + sslot, RgSmem::kScale);
            char* const sd = sScale + sslot * RgSmem::kScale;
            tma_load_2d(sd, &tmap_s, sc_full + sslot, kb, t.w0);
            tma_load_2d(sd + 64 * 16, &tmap_s, sc_full + sslot, kb, t.w1);
            tma_load_2d(sd + 128 * 16, &tmap_b, sc_full + sslot, kb, t.w0);
            tma_load_2d(sd + 192 * 16, &tmap_b, sc_full + sslot, kb, t.w1);
            if (++sslot == 2) { sslot = 0; sphase ^= 1u; }
          }
          if (!mbar_wait(raw_empty + rstage, rphase ^ 1u, abort_flag)) { ok = false; break; }
          mbar_arrive_expect_tx(raw_full + rstage, RgSmem::kRaw);
          tma_load_2d(sRaw + rstage * RgSmem::kRaw, &tmap_w, raw_full + rstage, kb * 32, t.w0);
          tma_load_2d(sRaw + rstage * RgSmem::kRaw + 64 * 128, &tmap_w, raw_full + rstage, kb * 32, t.w1);
          if (++rstage == kRgRawStages) { rstage = 0; rphase ^= 1u; }
        }
      }
    }
  } else {
    // ------------------------------------------------------------------ dequant: a thread expands a row of the k-block
    // Group g takes stages g, g + 3, ... of the block's sequence. The barriers of packed weights and scales that it does not visit
    // every time cannot be a phase behind what it takes them for: at stage i, its own stage i - 3 was filled after the products of i - 6,
    // so that everything up to stage i - 6 had landed, the slot's former contents (six or more stages back) with it.
    const int group = (warp - 6) >> 2, q = warp & 3;
    const int r = !p.swiglu ? q * 32 + lane : lane < 16 ? q * 16 + lane : 64 + q * 16 + lane - 16;   // gate and up rows side by side
    const uint32_t dst = tmem_w + group * 64 + (uint32_t(q * 32) << 16);
    const uint32_t raw0 = smem_u32(sRaw) + r * 128, sc0 = smem_u32(sScale) + r * 16;
    uint32_t phase = 0;
    bool ok = true;
    const int per_tile = (kb_end - kb_first) / 2, mine = first < num_tiles ? (num_tiles - first + step - 1) / step : 0;
    const int total = mine * per_tile;                    // stages of this block; every tile has a multiple of four
    for (int i = group; i < total; i += kRgStages) {
      const int raw = i >> 1, slot = raw % kRgRawStages, sc = (i >> 2) & 1;
      if (!rg_all(mbar_wait(sc_full + sc, (i >> 3) & 1, abort_flag))) { ok = false; break; }
      const uint32_t s2w = x_lds32(sc0 + sc * RgSmem::kScale + (i & 3) * 4);          // of the stage's two k-blocks
      const uint32_t b2w = x_lds32(sc0 + sc * RgSmem::kScale + kRgRows * 16 + (i & 3) * 4);
      if (!rg_all(mbar_wait(raw_full + slot, (raw / kRgRawStages) & 1, abort_flag))) { ok = false; break; }
      uint4 w[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) w[c] = x_lds(raw0 + slot * RgSmem::kRaw + ((((i & 1) * 4 + c) ^ (r & 7)) << 4));
      uint32_t o[32];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const uint32_t s2u = __byte_perm(s2w, 0u, h ? 0x3232u : 0x1010u), b2u = __byte_perm(b2w, 0u, h ? 0x3232u : 0x1010u);
        const __nv_bfloat162 s2 = *reinterpret_cast<const __nv_bfloat162*>(&s2u);
        const __nv_bfloat162 b2 = *reinterpret_cast<const __nv_bfloat162*>(&b2u);
        const uint32_t words[8] = {w[2 * h].x, w[2 * h].y, w[2 * h].z, w[2 * h].w, w[2 * h + 1].x, w[2 * h + 1].y, w[2 * h + 1].z, w[2 * h + 1].w};
#pragma unroll
        for (int j = 0; j < 8; ++j) x_expand(words[j], s2, b2, *reinterpret_cast<uint32_t(*)[4]>(o + 4 * j));
        if (h == 0) {
          if (!rg_all(mbar_wait(empty + group, phase ^ 1u, abort_flag))) { ok = false; break; }
          tc_fence_after_sync();
        }
        tmem_st_32x32(dst + h * 32, o);
      }
      if (!ok) break;
      phase ^= 1u;
      tmem_st_wait();
      tc_fence_before_sync();
      __syncwarp();
      // what was read is given back only here, where its values have been used (xgemm_kernel.cuh says why)
      if (lane == 0) { mbar_arrive(full + group); mbar_arrive(sc_empty + sc); mbar_arrive(raw_empty + slot); }
    }
  }

  tc_fence_before_sync();
  __syncthreads();
  if (p.split > 1)       // nobody reads or signals another block's shared memory any more
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  if (warp == 1) { tc_fence_after_sync(); tmem_dealloc(tmem_base, 512); }
  if (threadIdx.x == 0 && *abort_flag && p.status) atomicExch(p.status, kStatusMbarTimeout);
  pdl_launch_dependents();
}

static void rg_config(cudaLaunchConfig_t& cfg, cudaLaunchAttribute* attr, int grid, int split, int smem, bool pdl, cudaStream_t st) {
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(kRgThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  int n = 0;
  if (split > 1) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = split; attr[n].val.clusterDim.y = 1; attr[n].val.clusterDim.z = 1;
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

// Clusters of `split` blocks that can be resident at once.
static int rg_resident(int split) {
  static int known[64][4] = {};                          // split = 1 << i; 0: not asked yet
  int dev = 0, i = 0, n = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  if (split == 1) return sm_count();
  while ((1 << i) < split) ++i;
  if (known[dev][i] == 0) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[2];
    rg_config(cfg, attr, split * 64, split, 200 * 1024, false, nullptr);
    if (set_max_smem(row_gemm_kernel, 227 * 1024) != cudaSuccess || cudaOccupancyMaxActiveClusters(&n, row_gemm_kernel, &cfg) != cudaSuccess) n = 0;
    (void)cudaGetLastError();
    known[dev][i] = n > 0 ? n : -1;
  }
  return known[dev][i] > 0 ? known[dev][i] : 0;
}

}  // namespace rb

using namespace rb;
RB_BOUNDS_REGISTER("row_gemm.cu")

// Whole tiles of 128 rows of W (SwiGLU: of 64 gate and 64 up rows), K in groups of 8 scales, even rows of C.
extern "C" int rmlx_row_gemm_supported(int N, int K, int lda, int ldc, int swiglu) {
  return N >= 128 && N % 128 == 0 && K >= 512 && K % 512 == 0 && lda % 8 == 0 && ldc % 2 == 0;
}

// As rmlx_xgemm with 4-bit weights; out_f32: the accumulators as they are. split: blocks that share K (1, 2, 4, 8; 0: chosen).
extern "C" int rmlx_row_gemm(const void* A, const void* W, const void* scales, const void* biases, void* C, int out_f32,
                             const void* residual, const int* offsets, int E, int M, int N, int K, int lda, int ldc, int swiglu,
                             float gate_limit, int split, int* status, int pdl, cudaStream_t st) {
  if (M < 1 || !rmlx_row_gemm_supported(N, K, lda, ldc, swiglu)) return -2;
  if (offsets && (E < 1 || E > kXMaxExperts)) return -2;
  if (residual && (swiglu || out_f32)) return -2;
  if ((reinterpret_cast<uintptr_t>(C) | reinterpret_cast<uintptr_t>(residual)) & 3) return -2;
  if (split < 0 || split > kRgMaxSplit || (split & (split - 1)) || (split > 1 && (offsets || split > K / 512))) return -2;
  RgParams p = {};
  p.C = C; p.residual = static_cast<const __nv_bfloat16*>(residual); p.offsets = offsets; p.status = status;
  p.E = offsets ? E : 1; p.M = M; p.N = N; p.K = K; p.ldc = ldc; p.out_f32 = out_f32; p.swiglu = swiglu; p.gate_limit = gate_limit;
  const int most = M < kRgCols ? M : kRgCols;
  p.boxes = (most + kRgBox - 1) / kRgBox;
  const long long tiles_n = N / kRgRows, mt = (M + kRgCols - 1) / kRgCols;
  const long long tiles = offsets ? tiles_n * (mt + E) : tiles_n * mt;
  if (!offsets && split == 0) {        // the split with the fewest k-blocks in a row, and what adding the sums costs beside them
    double best = 1e30;
    for (int s = 1; s <= kRgMaxSplit && s <= K / 512 && (s == 1 || RgSmem::bytes(p.boxes, s) <= 227 * 1024); s *= 2) {
      const int n = rg_resident(s);
      if (n < 1) continue;
      const double cost = double((tiles + n - 1) / n) * (double(K / 64) / s + (s > 1 ? 12.0 + M / 16 : 6.0));
      if (cost < best) { best = cost; split = s; }
    }
  }
  if (split < 1) split = 1;
  p.split = split;
  const int smem = RgSmem::bytes(p.boxes, split);
  if (smem > 227 * 1024) return -2;
  CUtensorMap ta, tw, ts, tb;
  int rc = make_tmap_2d_bf16(&ta, A, uint64_t(K), uint64_t(M), uint64_t(lda) * 2, kXBK, kRgBox);
  if (rc) return rc;
  rc = x_weight_maps(1, W, scales, biases, uint64_t(p.E) * N, K, 64, &tw, &ts, &tb, 4);
  if (rc) return rc;
  RB_CHECK(set_max_smem(row_gemm_kernel, 227 * 1024));
  const int n = rg_resident(split);
  if (n < 1) return -2;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
  rg_config(cfg, attr, int(tiles < n ? tiles : n) * split, split, smem, pdl != 0, st);
  const cudaError_t err = cudaLaunchKernelEx(&cfg, row_gemm_kernel, ta, tw, ts, tb, p);
  if (err != cudaSuccess) (void)cudaGetLastError();
  return static_cast<int>(err);
}
