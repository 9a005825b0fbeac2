// Products of weights that e4m3 holds exactly, on the fp8 tensor path without expanding them to bf16:
//     Y[T, N] = epilogue( X[T, K] · dequant(W[N, K])^T ),  bf16 activations, W in
//   * fp8 e4m3 with one fp32 scale per 128 x 128 block (plain and grouped by expert), or
//   * uint4 codes with a scale and a zero point per output channel (a byte 0..15 read as e4m3 is the code times 2^-9:
//     subnormals and the first binade are equally spaced).
//
// An activation becomes the sum of two e4m3 numbers: x / s_t = hi + lo / 16 with s_t a power of two per row.  A bf16 value has
// eight significant bits, hi takes four and lo the other four, so the sum is x itself down to 2^-13.8 of the row's maximum and off
// by at most 2^-21.8 of that maximum below (the scaled maximum lies between 224 and 448).  Both halves are columns of one
// `kind::f8f6f4` MMA (N = 2 BN), sums are fp32.  The expanding kernel (quant_gemm_sm100.cu, still used for int8 and nf4) rounds fp8 x
// scale to bf16 and spends about 100 instructions per weight byte row; here fp8 tiles go from TMA to the tensor core untouched, and uint4 costs one AND and half a
// shift per four codes.  Block scales multiply the fp32 sums of 128 k: two TMEM accumulators in turn, the epilogue warps fetch
// one and add it to registers while the next fills.
//
// The same pipeline carries W8A8 at decode sizes (int8 weights and activations, `kind::i8`, s32 sums; the parts of a cluster
// are added as integers).
//
// B200, us before (expanding kernel; W8A8: its own kernel, parts through global scratch) / here, with the split of X:
//   fp8 2 x 28672 x 8192, 16 rows 417 / 78 (6.0 TB/s); 4096 x 4096, 16 rows 21 / 8; uint4 2 x 28672 x 8192, 16 rows 165 / 82;
//   12288 x 4096, 32 rows 29 / 19.  Error against 64 bits (12288 x 4096, relative): fp8 1.6e-3 / 1e-7, uint4 1.4e-5 / 3e-7.
// bf16 operands (64 k per block) go the same way at decode sizes.  The kernels they had (gemm_sm100.cu, gemm_decode_sm100.cu) leave
// parts in global scratch or finish with four warps, a dependent chain that grows with the tokens: 2 x 11008 x 4096, 32 rows 58 us
// there, 36 here (27.6 at the copy rate); 12288 x 4096, 64 rows 40 and 27; 4096 x 4096, 32 rows 13.8 and 9.5; 8192 x 28672, 1 row
// 70 and 69.  The fused all-reduce and the rotary epilogue stay there.
//
// A CTA owns 128 features x BN tokens (BN = 16, 32, 64).  Small products are cut along K over a cluster: every CTA leaves its
// part in its own shared memory and finishes BN / cluster tokens from all parts.
#include "gemm_common.cuh"

#include <cuda_fp8.h>

namespace xft {

enum { kSrcFp8 = 0, kSrcU4 = 1, kSrcI8 = 2, kSrcBf16 = 3 };

struct E4Params {
  int N, T, K;
  int dual_off;
  void* out; int ldo; int out_fp32;
  const float* bias;
  const __nv_bfloat16* residual; int ldr; float res_scale;
  int act;
  int num_kb, n_tiles, t_tiles, splits;      // blocks of 128 k; CTAs of a cluster that share them
  int x_lo;                  // column of the lo halves in a row of split activations
  const float* x_scale;      // [rows] s_t
  const float* x_sum;        // [rows] sum over k (uint4)
  const float* scale;        // fp8: [N / 128, K / 128] blocks, row pitch scale_ld; uint4: [N]
  const float* zero;         // uint4: [N]
  int scale_ld;
  const int4* group_tiles; const int* num_group_tiles; int group_w_rows;      // see quant_gemm_sm100.cu
  const float* col_scale;
  const float* a_zero; const float* a_qsum; const float* w_sum;      // W8A8: [T], [T], [N]; x_scale, scale and zero as above
  // bf16: a folded RMSNorm (W carries its gain): sums are multiplied with 1 / rms of the rows of rms_x, which is X
  const __nv_bfloat16* rms_x; int rms_ldx; float rms_eps;
  const float* rms_ssq;      // [T] their sums of squares, or null: every CTA adds them up for itself
  int* status;
};

constexpr int kE4Threads = 320;              // producer, MMA, eight warps that fetch accumulators (and expand codes)

__device__ __forceinline__ void umma_f8(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n"
      "}\n"
      :
      : "r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t* v) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
               : "r"(taddr));
}
template <int C>
__device__ __forceinline__ void tmem_ld_cols(uint32_t taddr, uint32_t* v) {
  if constexpr (C == 8) tmem_ld8(taddr, v);
  else if constexpr (C == 16) tmem_ld16(taddr, *reinterpret_cast<uint32_t (*)[16]>(v));
  else tmem_ld32(taddr, *reinterpret_cast<uint32_t (*)[32]>(v));
}

// act(x) and act(x) * u, out of line but for what is common: every activation at every place makes code that a launch of a few
// microseconds waits for
__device__ __noinline__ float other_act(float x, int act, float param) { return apply_act(x, act, param); }
__device__ __noinline__ float other_gated(float x, float u, int act, float param) { return apply_gated(x, u, act, param); }
__device__ __forceinline__ float act_of(float x, int act, float param) {
  return act == 0 ? x : act == 2 ? apply_act(x, 2) : other_act(x, act, param);
}
__device__ __forceinline__ float gated_of(float x, float u, int act, float param) {
  return act == 2 ? apply_act(x, 2) * u : other_gated(x, u, act, param);
}

template <int BN, bool DUAL, int SRC>
struct E4Layout {
  // Gated uint4, up to 32 rows: 64 gate and 64 up rows stacked in one tile.  With a tile of each, the expanded codes left room for one
  // CTA per SM, and 2 x 11008 x 4096 kept 86 SMs busy.  us, so / stacked: 2 x 11008 x 4096 16 rows 20.9 / 19.5, 32 rows 23.0 / 22.0; 2 x
  // 4864 x 896 7.0 / 5.3, 8.4 / 6.5; 2 x 28672 x 8192 75.0 / 69.3, 80.4 / 77.2.  64 rows leave one CTA per SM in either form, and stacked
  // tiles read the rows twice as often: 26.9 / 35.6, 90.7 / 120.7.
  static constexpr bool STACK = DUAL && SRC == kSrcU4 && BN <= 32;
  static constexpr int FEAT = STACK ? 64 : 128;
  static constexpr int NACC = DUAL && !STACK ? 2 : 1;
  static constexpr int A_BYTES = 128 * 128 * NACC, RAW_BYTES = SRC == kSrcU4 ? 128 * 64 * NACC : 0, B_BYTES = (SRC == kSrcI8 || SRC == kSrcBf16 ? 1 : 2) * BN * 128;
  static constexpr int STAGE = (SRC == kSrcU4 ? RAW_BYTES : A_BYTES) + B_BYTES;       // what TMA fills
  static constexpr int A_RING = SRC == kSrcU4 ? 2 * A_BYTES : 0;                      // expanded codes, two buffers
  // two CTAs per SM where registers allow: one CTA's last accumulators and stores hide behind the other's stream
  static constexpr int CTAS = BN <= 32 && A_RING + 3 * STAGE <= 110 * 1024 ? 2 : 1;
  // Registers are left for the CTAs of the kernels behind: with programmatic launches those sit beside this one, their first weights
  // under way.  At 90 registers (16 rows, bf16) instead of 64 the products of a 7B layer were as fast one behind the other, but 31 steps
  // of one row over 16 layers took 48.3 ms instead of 46.3.
  static constexpr int MIN_CTAS = CTAS == 2 && (BN == 16 || SRC == kSrcI8) ? 3 : CTAS;
  static constexpr int FIT = ((CTAS == 2 ? 110 : 222) * 1024 - A_RING) / STAGE;
  static constexpr int STAGES = FIT > 8 ? 8 : FIT;
  static constexpr int SMEM = A_RING + STAGES * STAGE + 1024;
  static_assert(STAGES >= 3 && BN * NACC * 512 <= A_RING + STAGES * STAGE, "ring, and room for this CTA's part of the sums");
};

template <int BN, bool DUAL, int SRC>
__global__ void __launch_bounds__(kE4Threads, E4Layout<BN, DUAL, SRC>::MIN_CTAS)
    gemm_e4m3_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, const E4Params p) {
  using L = E4Layout<BN, DUAL, SRC>;
  constexpr int NACC = L::NACC, STAGES = L::STAGES, FEAT = L::FEAT, HALVES = DUAL ? 2 : 1;
  constexpr bool STACK = L::STACK;
  constexpr int NB = SRC == kSrcI8 || SRC == kSrcBf16 ? BN : 2 * BN;   // columns of an accumulator: hi [BN], lo [BN]
  constexpr int ACC = NB * NACC;
  // bf16: k in PARTS pieces with an accumulator each.  The tensor core drops bits below an accumulator's last one at every step, so
  // its error grows with the k it adds up: 12288 x 4096 against 64 bits 2.1e-6 (2 CTAs per tile) and 4.4e-6 (one) of the result with
  // one accumulator, 4.8e-7 and 1.0e-6 with four; the kernels that had these products, 1.4e-6.  It costs 0.1 to 0.3 us of a launch.
  constexpr int PARTS = SRC == kSrcBf16 ? 4 : 1;
  // 64 rows fetch an accumulator as soon as its k is through, beside the main loop; fewer rows all at once at the end, where a short
  // stream pays for one wait and not for four.
  constexpr bool EARLY = PARTS > 1 && BN == 64;
  constexpr int BUFS = SRC == kSrcFp8 ? 2 : PARTS;
  constexpr uint32_t TMEM_COLS = BUFS * ACC < 32 ? 32 : BUFS * ACC;
  static_assert(TMEM_COLS * L::CTAS <= 512, "accumulators of the resident CTAs");
  constexpr uint32_t IDESC = SRC == kSrcI8 ? umma_idesc(128, BN, 1, 1, 2) : SRC == kSrcBf16 ? umma_idesc(128, BN, 1, 1, 1) : umma_idesc(128, 2 * BN, 0, 0, 1);
  constexpr int HB = BN / 2;                                           // tokens per thread: two warps share a row of the tile
  constexpr int TILE_A = 128 * 128;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ uint64_t full_bar[STAGES], empty_bar[STAGES], tmem_full[PARTS > 2 ? PARTS : 2], tmem_empty[2], a_ready[2], a_empty[2];
  __shared__ uint32_t tmem_base_s;
  __shared__ int s_group[4];
  __shared__ float s_ssq[SRC == kSrcBf16 ? BN : 1];                    // bf16: sums of squares of the tokens over this CTA's k
  // what the finish needs per feature (gate rows, then up rows) and per token, fetched beside the main loop.  uint4: scale, zero; W8A8:
  // scale, zero, sum of codes
  constexpr int NCOL = SRC == kSrcI8 ? 3 : SRC == kSrcU4 ? 2 : 0, NROW = SRC == kSrcI8 ? 3 : SRC == kSrcBf16 ? 1 : 2;
  __shared__ alignas(16) float s_col[NCOL ? NCOL : 1][NACC][NCOL ? 128 : 4];
  __shared__ float s_row[NROW][BN];

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int tile_n, tile_t;
  {
    constexpr int GN = 16;                                             // feature tiles that walk the token tiles together
    const int per = GN * p.t_tiles, g = blockIdx.x / per, r = blockIdx.x % per, gn = min(GN, p.n_tiles - g * GN);
    tile_n = g * GN + r % gn;
    tile_t = r / gn;
  }
  const int rank = blockIdx.y;
  const int kb0 = rank * p.num_kb / p.splits, kb1 = (rank + 1) * p.num_kb / p.splits;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&tmem_full[a], 1);
      mbar_init(&tmem_empty[a], 8);
      mbar_init(&a_ready[a], 8);
      mbar_init(&a_empty[a], 1);
    }
    for (int a = 2; a < PARTS; ++a) mbar_init(&tmem_full[a], 1);
    fence_barrier_init();
    fence_proxy_async();
    tma_prefetch_desc(&tmW);
    tma_prefetch_desc(&tmX);
  }
  if (warp == 1) { tmem_alloc(&tmem_base_s, TMEM_COLS); tmem_relinquish(); }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem_base = tmem_base_s;
  grid_dep_launch();
  const bool grouped = p.group_tiles != nullptr;
  if (grouped) {
    grid_dep_wait();          // the tile table comes from the routing plan kernel
    if (threadIdx.x == 0) {
      int4 e = make_int4(0, 0, 0, 0);
      if (tile_t < *p.num_group_tiles) e = p.group_tiles[tile_t];
      s_group[0] = e.x; s_group[1] = e.y; s_group[2] = e.z;
    }
    __syncthreads();
  }
  const int w_row0 = (grouped ? s_group[0] * p.group_w_rows : 0) + tile_n * FEAT;
  const int x_row0 = grouped ? s_group[1] : tile_t * BN;
  const int x_rows = grouped ? s_group[2] : min(BN, p.T - x_row0);
  const int kend = x_rows > 0 ? kb1 : kb0;                             // nothing to do for a tile without rows
  // blocks per accumulator, and accumulators: up to 512 k stay in one
  const int part_kb = max((kb1 - kb0 + PARTS - 1) / PARTS, 8);
  const int parts = 1 + (kb1 - kb0 > part_kb) + (kb1 - kb0 > 2 * part_kb) + (kb1 - kb0 > 3 * part_kb);

  uint8_t* ring = smem + L::A_RING;
  if (warp == 0) {
    if (elect_one()) {
      constexpr int W_COLS = SRC == kSrcU4 ? 64 : 128;                 // bytes of a weight row per block of 128 k (bf16: 64 k)
      constexpr int W_TILE = 128 * W_COLS;
      constexpr int W_STEP = SRC == kSrcBf16 ? 64 : W_COLS;            // the same in elements of the tensor map
      const uint64_t hint_w = p.t_tiles == 1 || grouped ? kEvictFirst : kEvictNormal;
      auto load_w = [&](int s, int kb) {
        mbar_expect_tx(&full_bar[s], L::STAGE);
        uint8_t* st = ring + s * L::STAGE;
        tma_load_2d(st, &tmW, &full_bar[s], kb * W_STEP, w_row0, hint_w);
        if (DUAL) tma_load_2d(st + FEAT * W_COLS, &tmW, &full_bar[s], kb * W_STEP, p.dual_off + w_row0, hint_w);
      };
      auto load_x = [&](int s, int kb) {
        uint8_t* st = ring + s * L::STAGE + W_TILE * NACC;
        tma_load_2d(st, &tmX, &full_bar[s], SRC == kSrcBf16 ? kb * 64 : kb * 128, x_row0, kEvictLast);
        if (SRC != kSrcI8 && SRC != kSrcBf16) tma_load_2d(st + BN * 128, &tmX, &full_bar[s], p.x_lo + kb * 128, x_row0, kEvictLast);
      };
      // weights never depend on the previous kernel: the first round is requested before the grid dependency resolves
      const int pre = min(STAGES, kend - kb0);
      for (int i = 0; i < pre; ++i) load_w(i, kb0 + i);
      grid_dep_wait();
      for (int i = 0; i < pre; ++i) load_x(i, kb0 + i);
      Ring r = {0, 1};
      for (int kb = kb0 + pre; kb < kend; ++kb, r.next(STAGES)) {
        if (!mbar_wait(&empty_bar[r.s], r.ph ^ 1, p.status, XFT_ERR_WAIT_EMPTY)) break;
        load_w(r.s, kb);
        load_x(r.s, kb);
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      const uint64_t stage0 = umma_desc_k128(smem_u32(ring));
      const uint64_t bdesc0 = stage0 + (L::STAGE - L::B_BYTES) / 16;
      const uint64_t a0 = SRC == kSrcU4 ? umma_desc_k128(smem_u32(smem)) : stage0;
      Ring r = {0, 0}, b = {0, 0};                                     // stage; buffer of expanded codes or accumulator
      int in_part = 0, part = 0;                                       // blocks in this accumulator; which it is
      bool ok = true;
      for (int kb = kb0; kb < kend; ++kb, r.next(STAGES), b.next(2)) {
        if (SRC == kSrcFp8) ok = mbar_wait(&tmem_empty[b.s], b.ph ^ 1, p.status, XFT_ERR_WAIT_TMEM);
        ok = ok && mbar_wait(&full_bar[r.s], r.ph, p.status, XFT_ERR_WAIT_FULL);
        if (SRC == kSrcU4) ok = ok && mbar_wait(&a_ready[b.s], b.ph, p.status, XFT_ERR_WAIT_FULL);
        if (!ok) break;
        tcgen05_fence_after();
        const uint64_t bd = bdesc0 + (uint64_t)(r.s * (L::STAGE / 16));
        const uint64_t ad = a0 + (uint64_t)(SRC == kSrcU4 ? b.s * (L::A_BYTES / 16) : r.s * (L::STAGE / 16));
        const uint32_t acc = tmem_base + (SRC == kSrcFp8 ? b.s * ACC : PARTS > 1 ? part * ACC : 0);
#pragma unroll
        for (int k = 0; k < 4; ++k) {                                  // 4 x 32 k
          const uint32_t on = (SRC != kSrcFp8 && (PARTS > 1 ? in_part > 0 : kb > kb0)) || k > 0;
          auto mma = [&](uint32_t d, uint64_t a) {
            if constexpr (SRC == kSrcBf16) umma_bf16(d, a, bd + 2 * k, IDESC, on);
            else if constexpr (SRC == kSrcI8) umma_i8(d, a, bd + 2 * k, IDESC, on);
            else umma_f8(d, a, bd + 2 * k, IDESC, on);
          };
          mma(acc, ad + 2 * k);
          if (NACC == 2) mma(acc + NB, ad + TILE_A / 16 + 2 * k);
        }
        tcgen05_commit(&empty_bar[r.s]);
        if (PARTS > 1 && (++in_part == part_kb || kb + 1 == kend)) {
          if (EARLY) tcgen05_commit(&tmem_full[part]);
          ++part;
          in_part = 0;
        }
        if (SRC == kSrcU4) tcgen05_commit(&a_empty[b.s]);
        if (SRC == kSrcFp8) tcgen05_commit(&tmem_full[b.s]);
      }
      if (SRC != kSrcFp8 && !EARLY && kend > kb0 && ok) tcgen05_commit(&tmem_full[0]);
    }
  }

  // ---- warps 2..9: row = feature of the tile, tokens [c0, c0 + HB) of it
  const int q = warp & 3, row = q * 32 + lane, half = warp >= 6, c0 = half * HB;
  // the finish: warp w takes tokens w, w + 8, .. of this CTA's share of the tile, a lane four features of each (stacked tiles: half a
  // warp a token)
  constexpr int AT_ONCE = STACK ? 16 : 8;
  const int per = BN / p.splits, f0 = (STACK ? lane & 15 : lane) * 4, n = tile_n * FEAT + f0;
  const int tok0 = STACK ? 2 * (warp - 2) + (lane >> 4) : warp - 2;
  const bool vec = n + 4 <= p.N && (p.ldo & 3) == 0 && (reinterpret_cast<uintptr_t>(p.out) & (p.out_fp32 ? 15 : 7)) == 0;
  const bool vec_res = n + 4 <= p.N && (p.ldr & 3) == 0 && (reinterpret_cast<uintptr_t>(p.residual) & 7) == 0;
  constexpr int MINE = BN / AT_ONCE;
  auto residual_of = [&](int i) {                                      // of this thread's i-th token
    uint2 v = make_uint2(0, 0);
    const int c = rank * per + tok0 + AT_ONCE * i;
    if (p.residual && tok0 + AT_ONCE * i < per && c < x_rows) {
      const __nv_bfloat16* r = p.residual + (size_t)(x_row0 + c) * p.ldr + n;
      if (vec_res) {
        v = *reinterpret_cast<const uint2*>(r);
      } else {
        __nv_bfloat16* to = reinterpret_cast<__nv_bfloat16*>(&v);
#pragma unroll
        for (int f = 0; f < 4; ++f)
          if (n + f < p.N) to[f] = r[f];
      }
    }
    return v;
  };
  if (NCOL && warp >= 2) {                                             // weights' numbers depend on no earlier kernel
    const int e = threadIdx.x - 64, nn = tile_n * FEAT + (e & (FEAT - 1));
    if (e < 128 * NACC) {
      const int at = (e >= FEAT ? p.dual_off : 0) + nn;
      const float* from[3] = {p.scale, p.zero, p.w_sum};
#pragma unroll
      for (int i = 0; i < NCOL; ++i) s_col[i][e >> 7][e & 127] = nn < p.N && from[i] ? __ldg(from[i] + at) : 0.f;
    }
  }
  // residuals are asked for a token ahead, the first beside the main loop (all of them there cost every launch 0.4 us)
  uint2 next_res = make_uint2(0, 0);
  auto fetch_rows = [&]() {                                            // what earlier kernels leave per token
    next_res = residual_of(0);
    const int e = threadIdx.x - 64;
    if (e < BN) {
      const int t = x_row0 + e;
      const bool in = e < x_rows;
      if constexpr (SRC == kSrcBf16) {
        s_row[0][e] = in && p.rms_ssq ? p.rms_ssq[t] : 0.f;
      } else {
        s_row[0][e] = in ? p.x_scale[t] : 0.f;
        if constexpr (SRC == kSrcI8) { s_row[1][e] = in ? p.a_zero[t] : 0.f; s_row[2][e] = in ? p.a_qsum[t] : 0.f; }
        if constexpr (SRC == kSrcU4) s_row[1][e] = in ? p.x_sum[t] : 0.f;
        if constexpr (SRC == kSrcFp8) s_row[1][e] = in && p.col_scale ? p.col_scale[t] : 1.f;
      }
    }
  };
  float g[NACC][HB];
#pragma unroll
  for (int i = 0; i < NACC; ++i)
#pragma unroll
    for (int j = 0; j < HB; ++j) g[i][j] = 0.f;
  bool ok = x_rows > 0;
  if (warp >= 2) {
    const uint32_t taddr = tmem_base + (uint32_t(q * 32) << 16) + c0;
    auto fetch = [&](uint32_t col, float* to, float factor) {          // to += factor * (hi + lo / 16)
      uint32_t hi[HB], lo[HB];
      tmem_ld_cols<HB>(taddr + col, hi);
      tmem_ld_cols<HB>(taddr + col + BN, lo);
      tmem_ld_wait();
#pragma unroll
      for (int j = 0; j < HB; ++j)
        to[j] = fmaf(factor, fmaf(__uint_as_float(lo[j]), 0.0625f, __uint_as_float(hi[j])), to[j]);
    };
    if constexpr (SRC == kSrcFp8) {
      grid_dep_wait();
      fetch_rows();
      const float* sc = p.scale + (size_t)(w_row0 >> 7) * p.scale_ld;
      const float* sc_up = sc + (size_t)(p.dual_off >> 7) * p.scale_ld;
      Ring b = {0, 0};
      for (int kb = kb0; kb < kend && ok; ++kb, b.next(2)) {
        const float f0 = __ldg(sc + kb), f1 = DUAL ? __ldg(sc_up + kb) : 0.f;
        ok = mbar_wait(&tmem_full[b.s], b.ph, p.status, XFT_ERR_WAIT_TMEM);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tcgen05_fence_after();
        fetch(b.s * ACC, g[0], f0);
        if constexpr (DUAL) fetch(b.s * ACC + NB, g[1], f1);
        tcgen05_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&tmem_empty[b.s]);
      }
    } else if constexpr (SRC == kSrcI8 || SRC == kSrcBf16) {
      grid_dep_wait();
      fetch_rows();
      if (SRC == kSrcBf16 && p.rms_x && !p.rms_ssq) {                                // beside the main loop: 256 / BN threads per token
        constexpr int TPT = 256 / BN;
        const int e = threadIdx.x - 64, tok = e / TPT, sub = e % TPT;
        float acc = 0.f;
        if (tok < x_rows) {
          const __nv_bfloat16* xr = p.rms_x + (size_t)(x_row0 + tok) * p.rms_ldx;
          const int k1 = min(kb1 * 64, p.K);
#pragma unroll 4
          for (int k = kb0 * 64 + sub * 8; k < k1; k += TPT * 8) {
            const uint4 v = *reinterpret_cast<const uint4*>(xr + k);
            const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const float2 f = __bfloat1622float2(h[i]);
              acc += f.x * f.x + f.y * f.y;
            }
          }
        }
#pragma unroll
        for (int o = TPT / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if (sub == 0) s_ssq[tok] = acc;
      }
      ok = __all_sync(0xffffffffu, mbar_wait(&tmem_full[0], 0, p.status, XFT_ERR_WAIT_TMEM));
      tcgen05_fence_after();
      if (ok && (PARTS == 1 || EARLY)) {                               // s32 (or fp32), kept as they are
        tmem_ld_cols<HB>(taddr, reinterpret_cast<uint32_t*>(g[0]));
        if constexpr (DUAL) tmem_ld_cols<HB>(taddr + NB, reinterpret_cast<uint32_t*>(g[1]));
        tmem_ld_wait();
      }
      if constexpr (PARTS > 1 && !EARLY) {
        if (ok) {
#pragma unroll
          for (int a = 0; a < NACC; ++a) {
            uint32_t v[PARTS - 1][HB];
            tmem_ld_cols<HB>(taddr + a * NB, reinterpret_cast<uint32_t*>(g[a]));
#pragma unroll
            for (int i = 1; i < PARTS; ++i)
              if (i < parts) tmem_ld_cols<HB>(taddr + i * ACC + a * NB, v[i - 1]);
            tmem_ld_wait();
#pragma unroll
            for (int i = 1; i < PARTS; ++i)
#pragma unroll
              for (int j = 0; j < HB; ++j) g[a][j] += i < parts ? __uint_as_float(v[i - 1][j]) : 0.f;
          }
        }
      }
      if constexpr (EARLY) for (int i = 1; i < parts && ok; ++i) {
        ok = __all_sync(0xffffffffu, mbar_wait(&tmem_full[i], 0, p.status, XFT_ERR_WAIT_TMEM));
        tcgen05_fence_after();
        if (!ok) break;
        uint32_t v[NACC][HB];
        tmem_ld_cols<HB>(taddr + i * ACC, v[0]);
        if constexpr (DUAL) tmem_ld_cols<HB>(taddr + i * ACC + NB, v[1]);
        tmem_ld_wait();
#pragma unroll
        for (int a = 0; a < NACC; ++a)
#pragma unroll
          for (int j = 0; j < HB; ++j) g[a][j] += __uint_as_float(v[a][j]);
      }
    } else {
      // codes to bytes: a 16-byte piece holds 32 of them; the even ones go to one swizzled 16-byte piece of the operand row,
      // the odd ones to the next (the activations' k are in the same order)
      const int e = threadIdx.x - 64;
      Ring r = {0, 0}, b = {0, 0};
      bool alive = true;
      for (int kb = kb0; kb < kend; ++kb, r.next(STAGES), b.next(2)) {
        uint4 codes[2 * NACC];
        alive = alive && mbar_wait(&full_bar[r.s], r.ph, p.status, XFT_ERR_WAIT_FULL);
        if (alive) {
#pragma unroll
          for (int i = 0; i < 2 * NACC; ++i) codes[i] = *reinterpret_cast<const uint4*>(ring + r.s * L::STAGE + (e + 256 * i) * 16);
        }
        alive = alive && mbar_wait(&a_empty[b.s], b.ph ^ 1, p.status, XFT_ERR_WAIT_EMPTY);
        if (alive) {
          uint8_t* a = smem + b.s * L::A_BYTES;
#pragma unroll
          for (int i = 0; i < 2 * NACC; ++i) {
            const int ci = e + 256 * i, tr = ci >> 2, part = ci & 3;   // row of the stacked tiles, 32 codes of it
            const uint4 w = codes[i];
            constexpr uint32_t M = 0x0F0F0F0Fu;
            uint8_t* dst = a + tr * 128;
            *reinterpret_cast<uint4*>(dst + (((2 * part) ^ (tr & 7)) << 4)) = make_uint4(w.x & M, w.y & M, w.z & M, w.w & M);
            *reinterpret_cast<uint4*>(dst + (((2 * part + 1) ^ (tr & 7)) << 4)) =
                make_uint4((w.x >> 4) & M, (w.y >> 4) & M, (w.z >> 4) & M, (w.w >> 4) & M);
          }
          fence_proxy_async();
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&a_ready[b.s]);                     // per warp: with 256 arrivals a block 2 x 28672 x 8192 64 rows took 90.7 us, so 86
      }
      grid_dep_wait();
      fetch_rows();
      if (kend > kb0) {
        ok = __all_sync(0xffffffffu, mbar_wait(&tmem_full[0], 0, p.status, XFT_ERR_WAIT_TMEM));
        tcgen05_fence_after();
        if (ok) {
          fetch(0, g[0], 512.f);
          if constexpr (NACC == 2) fetch(NB, g[1], 512.f);
        }
      }
    }
  }
  // Every MMA has read its operands (the last accumulator is here), so the ring is free for this CTA's part of the sums, [column][128].
  // From there a lane takes four features of a token at once: residual and output move in 8-byte pieces, scales are already here, and
  // no load waits for the one before.  A thread per feature that walked its tokens waited for a global load in each:
  // us, so / now: bf16 12288 x 4096 with a folded norm 16 rows 21.8 / 20.1, 64 rows 36.8 / 23.6; 2 x 11008 x 4096 32 rows 38.3 / 34.3, 64
  // rows 52.3 / 37.2; 896 x 896 16 rows 5.8 / 4.1, 64 rows 12.0 / 6.0; W8A8 12288 x 4096 32 rows 15.9 / 13.8; one row is level (2 x 11008
  // x 4096 31.5 / 32.0, 4096 x 4096 8.4 / 8.5).
  float* part = reinterpret_cast<float*>(smem);
  if (warp >= 2) {
#pragma unroll
    for (int i = 0; i < NACC; ++i)
#pragma unroll
      for (int j = 0; j < HB; ++j) part[(i * BN + c0 + j) * 128 + row] = g[i][j];
  }
  __syncwarp();                                                        // the lanes behind the elected ones of warps 0 and 1
  if (p.splits > 1) {
    cluster_arrive();
    cluster_wait();
  } else if (warp >= 2) {
    named_bar_sync(1, 256);
  }
  if (warp >= 2 && n < p.N && (ok || p.splits > 1)) {
    float4 bias[HALVES];
#pragma unroll
    for (int a = 0; a < HALVES; ++a) {
      bias[a] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (p.bias) {
#pragma unroll
        for (int f = 0; f < 4; ++f)
          if (n + f < p.N) (&bias[a].x)[f] = __ldg(p.bias + a * p.dual_off + n + f);
      }
    }
#pragma unroll 1
    for (int i = 0; i < MINE; ++i) {
      const int mine = tok0 + AT_ONCE * i, c = rank * per + mine;
      if (mine >= per || c >= x_rows) break;
      const uint2 res = next_res;
      next_res = residual_of(i + 1);
      float4 y[HALVES];
      float ssq = SRC == kSrcBf16 ? s_row[0][c] : 0.f;
      const bool own_ssq = SRC == kSrcBf16 && p.rms_x && !p.rms_ssq;
      constexpr int UP = STACK ? 64 : BN * 128;                        // from a gate feature to its up feature
      const uint32_t at = smem_u32(part + c * 128 + f0), at_ssq = smem_u32(s_ssq + (SRC == kSrcBf16 ? c : 0));
      if (p.splits == 1) {
#pragma unroll
        for (int a = 0; a < HALVES; ++a) y[a] = *reinterpret_cast<const float4*>(part + c * 128 + f0 + a * UP);
        if (own_ssq) ssq += s_ssq[SRC == kSrcBf16 ? c : 0];
      } else {
        float q[8];
        if (own_ssq) {
#pragma unroll
          for (int r = 0; r < 8; ++r) q[r] = r < p.splits ? ld_dsmem(dsmem_addr(at_ssq, r)) : 0.f;
        }
#pragma unroll
        for (int a = 0; a < HALVES; ++a) {
          float4 v[8];
#pragma unroll
          for (int r = 0; r < 8; ++r) v[r] = r < p.splits ? ld_dsmem4(dsmem_addr(at + a * UP * 4, r)) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
          for (int f = 0; f < 4; ++f) {
            if constexpr (SRC == kSrcI8) {
              int sum = 0;
#pragma unroll
              for (int r = 0; r < 8; ++r) sum += __float_as_int((&v[r].x)[f]);
              (&y[a].x)[f] = __int_as_float(sum);
            } else {
              float sum = 0.f;
#pragma unroll
              for (int r = 0; r < 8; ++r) sum += (&v[r].x)[f];
              (&y[a].x)[f] = sum;
            }
          }
        }
        if (own_ssq) {
#pragma unroll
          for (int r = 0; r < 8; ++r) if (r < p.splits) ssq += q[r];
        }
      }
      const size_t t = x_row0 + c;
      const __nv_bfloat16* rv = reinterpret_cast<const __nv_bfloat16*>(&res);
      float ts = 1.f;
      if (SRC == kSrcBf16 && p.rms_x) ts = rsqrtf(ssq / (float)p.K + p.rms_eps);
      float out[4];
#pragma unroll
      for (int f = 0; f < 4; ++f) {
        float x = (&y[0].x)[f], u = DUAL ? (&y[HALVES - 1].x)[f] : 0.f;
        const float b = (&bias[0].x)[f], bu = (&bias[HALVES - 1].x)[f], r = __bfloat162float(rv[f]);
        if constexpr (SRC == kSrcBf16) {
          // Which multiply-adds are fused is spelled out: a last bit here moves every logit of a model with biases behind folded norms
          x = DUAL ? __fmaf_rn(x, ts, b) : __fadd_rn(__fmul_rn(x, ts), b);
          if (DUAL) x = gated_of(x, __fadd_rn(__fmul_rn(u, ts), bu), p.act, p.res_scale);
          else x = act_of(x, p.act, p.res_scale);
          if (p.residual) x = with_residual(x, r, p.res_scale, p.act);
        } else if constexpr (SRC == kSrcI8) {
          auto value = [&](float acc, int a, float to) {
            return w8a8_value((float)__float_as_int(acc), s_row[0][c], s_row[1][c], s_row[2][c], s_col[0][a][f0 + f], s_col[1][a][f0 + f],
                              s_col[2][a][f0 + f], p.K, to);
          };
          if (DUAL) x = act_of(bf16_round(value(x, 0, b)), p.act, 1.f) * bf16_round(value(u, NACC - 1, bu));
          else x = act_of(value(x, 0, b), p.act, 1.f);
          if (p.residual) x += p.res_scale * r;
        } else {
          const float st = s_row[0][c];
          if constexpr (SRC == kSrcU4) {
            const float xs = s_row[1][c];
            x = act_of(fmaf(x, st * s_col[0][0][f0 + f], b + s_col[1][0][f0 + f] * xs), p.act, 1.f);
            constexpr int AT = STACK ? 64 : 0;                         // up features of a stacked tile
            if (DUAL) x *= fmaf(u, st * s_col[0][NACC - 1][AT + f0 + f], bu + s_col[1][NACC - 1][AT + f0 + f] * xs);
          } else {
            x = act_of(fmaf(x, st, b), p.act, 1.f);
            if (DUAL) x *= fmaf(u, st, bu);
            if (p.col_scale) x *= s_row[1][c];
          }
          if (p.residual) x += p.res_scale * r;
        }
        out[f] = x;
      }
      if (p.out_fp32) {
        float* to = reinterpret_cast<float*>(p.out) + t * p.ldo + n;
        if (vec) {
          *reinterpret_cast<float4*>(to) = make_float4(out[0], out[1], out[2], out[3]);
        } else {
#pragma unroll
          for (int f = 0; f < 4; ++f)
            if (n + f < p.N) to[f] = out[f];
        }
      } else {
        __nv_bfloat16* to = reinterpret_cast<__nv_bfloat16*>(p.out) + t * p.ldo + n;
        if (vec) {
          const __nv_bfloat162 lo = __floats2bfloat162_rn(out[0], out[1]), hi = __floats2bfloat162_rn(out[2], out[3]);
          *reinterpret_cast<uint2*>(to) = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
        } else {
#pragma unroll
          for (int f = 0; f < 4; ++f)
            if (n + f < p.N) to[f] = __float2bfloat16(out[f]);
        }
      }
    }
  }
  if (p.splits > 1) {
    __syncwarp();
    cluster_arrive();                                                  // nobody leaves while its part is being read
    cluster_wait();
  }
  __syncwarp();
  tcgen05_fence_before();
  __syncthreads();
  if (warp == 1) { tcgen05_fence_after(); tmem_dealloc(tmem_base, TMEM_COLS); }
}

// Sums of squares of rows of X, a block per row.
__global__ void __launch_bounds__(256) row_ssq_kernel(const __nv_bfloat16* __restrict__ x, int ldx, int K, float* __restrict__ ssq) {
  __shared__ float s_sum[8];
  grid_dep_launch();
  grid_dep_wait();
  const __nv_bfloat16* row = x + (size_t)blockIdx.x * ldx;
  float sm = 0.f;
  for (int k = threadIdx.x * 8; k < K; k += 2048) {
    const uint4 v = *reinterpret_cast<const uint4*>(row + k);
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 f = __bfloat1622float2(h[i]);
      sm += f.x * f.x + f.y * f.y;
    }
  }
  for (int o = 16; o > 0; o >>= 1) sm += __shfl_xor_sync(0xffffffffu, sm, o);
  if ((threadIdx.x & 31) == 0) s_sum[threadIdx.x >> 5] = sm;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; ++w) sm += s_sum[w];
    ssq[blockIdx.x] = sm;
  }
}

// Row r of X (or row src[r]) -> [hi | lo] e4m3, its power-of-two scale and its sum.  `nibbles`: k in the order in which uint4
// codes expand, 16 even ones and 16 odd ones of every 32.  Rows from *rows_used on are left alone.  (Rows of more than 32768; others
// in quant_rows.cu.)
__global__ void __launch_bounds__(256) split_e4m3_kernel(const __nv_bfloat16* __restrict__ x, int ldx, const int* __restrict__ src,
                                                         const int* __restrict__ rows_used, int K, int Kp, int nibbles,
                                                         uint8_t* __restrict__ out, float* __restrict__ scale, float* __restrict__ sum) {
  __shared__ float s_mx[8], s_sum[8];
  grid_dep_launch();
  grid_dep_wait();
  const int r = blockIdx.x;
  if (rows_used && r >= *rows_used) return;
  const __nv_bfloat16* row = x + (size_t)(src ? src[r] : r) * ldx;
  float mx = 0.f, sm = 0.f;
  for (int k = threadIdx.x * 8; k < K; k += 2048) {
    const uint4 v = *reinterpret_cast<const uint4*>(row + k);
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 f = __bfloat1622float2(h[i]);
      sm += f.x + f.y;
      const float a = fabsf(f.x), b = fabsf(f.y);
      if (a <= 3.4e38f) mx = fmaxf(mx, a);                             // infinities and NaN have no part in the scale
      if (b <= 3.4e38f) mx = fmaxf(mx, b);
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    sm += __shfl_xor_sync(0xffffffffu, sm, o);
  }
  if ((threadIdx.x & 31) == 0) { s_mx[threadIdx.x >> 5] = mx; s_sum[threadIdx.x >> 5] = sm; }
  __syncthreads();
  mx = s_mx[0]; sm = s_sum[0];
  for (int w = 1; w < 8; ++w) { mx = fmaxf(mx, s_mx[w]); sm += s_sum[w]; }
  int e;
  const float f = frexpf(mx, &e);                                      // mx = f 2^e, 0.5 <= f < 1: at most 448 = 0.875 * 2^9
  e = mx == 0.f ? 0 : max(-100, e - 9 + (f > 0.875f));
  const float inv = exp2f((float)-e);
  if (threadIdx.x == 0) {
    scale[r] = exp2f((float)e);
    if (sum) sum[r] = sm;
  }
  uint8_t* hi_row = out + (size_t)r * 2 * Kp;
  for (int k = threadIdx.x * 8; k < Kp; k += 2048) {
    uint8_t hi[8], lo[8];
    if (k < K) {
      const uint4 v = *reinterpret_cast<const uint4*>(row + k);
      const __nv_bfloat16* b = reinterpret_cast<const __nv_bfloat16*>(&v);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float y = __bfloat162float(b[i]) * inv;
        const __nv_fp8_storage_t c = __nv_cvt_float_to_fp8(y, __NV_SATFINITE, __NV_E4M3);
        const float back = __half2float(__half(__nv_cvt_fp8_to_halfraw(c, __NV_E4M3)));
        hi[i] = fabsf(y) <= 3.4e38f ? c : 0x7F;                        // an infinity or NaN makes its row NaN
        lo[i] = fabsf(y) <= 3.4e38f ? __nv_cvt_float_to_fp8((y - back) * 16.f, __NV_SATFINITE, __NV_E4M3) : 0;
      }
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i) hi[i] = lo[i] = 0;                   // 0 x garbage of a padded column could be NaN
    }
    if (nibbles) {
      const int at = (k & ~31) + (k & 31) / 2;
#pragma unroll
      for (int o = 0; o < 2; ++o) {
        *reinterpret_cast<uchar4*>(hi_row + at + 16 * o) = make_uchar4(hi[o], hi[2 + o], hi[4 + o], hi[6 + o]);
        *reinterpret_cast<uchar4*>(hi_row + Kp + at + 16 * o) = make_uchar4(lo[o], lo[2 + o], lo[4 + o], lo[6 + o]);
      }
    } else {
      uint2 a, c;
      memcpy(&a, hi, 8);
      memcpy(&c, lo, 8);
      *reinterpret_cast<uint2*>(hi_row + k) = a;
      *reinterpret_cast<uint2*>(hi_row + Kp + k) = c;
    }
  }
}

int launch_split(const void* x, int ldx, const int* src, const int* rows_used, const float* gain, float eps, int rows, int K, int Kp,
                 int nibbles, void* out, float* scale, float* sum, cudaStream_t st);      // quant_rows.cu
int make_byte_map(CUtensorMap* out, const void* ptr, uint64_t rows, uint64_t row_bytes, uint64_t ld_bytes, uint32_t box_rows,
                  uint32_t box_bytes);                                 // gemm_sm100.cu: unswizzled bytes

// Parts of a tile's k: as many as one round of clusters holds, at least four blocks of k in each.  GPCs differ in their SMs, so what
// fits is not a division: clusters of 2, 4 and 8 CTAs that B200 takes at a time, with one and with two CTAs per SM.  us, gated uint4
// 2 x 11008 x 4096 (86 tiles of each half, one CTA per SM), 16 rows: 31.7 with two parts, 24.3 with one; e4m3 24 rows 33.9 and 24.8; bf16 4608 x
// 3584 (36 tiles) with its rotation behind it, 16 rows: 16.0 with eight parts, 12.4 with four, 48 rows 23.4 with four, 19.6 with two.
static int e4_splits(int tiles, int num_kb, int per_sm) {
  constexpr int kFit[2][3] = {{74, 33, 15}, {148, 71, 33}};
  int i = 0;
  while (i < 3 && tiles <= kFit[per_sm - 1][i] && num_kb >> (i + 1) >= 4) ++i;
  return 1 << i;
}

template <int BN, bool DUAL, int SRC>
static int launch_e4(const CUtensorMap& tmW, const CUtensorMap& tmX, E4Params p, cudaStream_t st) {
  using L = E4Layout<BN, DUAL, SRC>;
  const auto kernel = gemm_e4m3_kernel<BN, DUAL, SRC>;
  static bool attr_set = false;
  if (!attr_set) {
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, L::SMEM) != cudaSuccess)
      return 3000 + (int)cudaGetLastError();
    attr_set = true;
  }
  // stacked tiles: as many parts as tiles of 128 features on an SM each would have (64 rows have those), so a row's sums do not depend on
  // how many rows stand beside it
  p.splits = p.group_tiles ? 1 : L::STACK ? e4_splits((p.n_tiles + 1) / 2 * p.t_tiles, p.num_kb, 1)
                                          : e4_splits(p.n_tiles * p.t_tiles, p.num_kb, L::CTAS);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(p.n_tiles * p.t_tiles, p.splits);
  cfg.blockDim = dim3(kE4Threads);
  cfg.dynamicSmemBytes = L::SMEM;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = attr[0].val.clusterDim.z = 1;
  attr[0].val.clusterDim.y = p.splits;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = g_xft_pdl ? 2 : 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, tmW, tmX, p);
  return e != cudaSuccess ? (int)e : (int)cudaGetLastError();
}

}  // namespace xft

using namespace xft;

// Columns of a row of split activations: hi and lo halves are this many bytes each.
extern "C" int xft_split_e4m3_cols(int K) { return (K + 31) / 32 * 32; }

// X [.., ldx] bf16 -> out [rows, 2 * cols], scale [rows], sum [rows] (or null); K, ldx multiples of 8, 16-byte aligned rows.
extern "C" int xft_split_e4m3(const void* x, int ldx, const int* src, const int* rows_used, int rows, int K, int nibbles, void* out,
                              float* scale, float* sum, cudaStream_t st) {
  if (rows <= 0) return 0;
  if ((K & 7) || (ldx & 7) || ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(out)) & 15)) return -2;
  const int rc = launch_split(x, ldx, src, rows_used, nullptr, 0.f, rows, K, xft_split_e4m3_cols(K), nibbles, out, scale, sum, st);
  if (rc != -1) return rc;
  const cudaError_t e = launch_pdl(split_e4m3_kernel, dim3(rows), dim3(256), 0, st, (const __nv_bfloat16*)x, ldx, src, rows_used, K,
                                   xft_split_e4m3_cols(K), nibbles, (uint8_t*)out, scale, sum);
  return e != cudaSuccess ? (int)e : (int)cudaGetLastError();
}

// src: 0 = e4m3 weights [w_rows, K] with block scales, 1 = uint4 [w_rows, K / 2] with scale / zero per row.  xs, x_scale, x_sum
// from xft_split_e4m3 (`nibbles` = src).  Grouped (fp8): tiles of `bn` rows as in xft_qgemm_grouped; plain: group_tiles null.
extern "C" int xft_gemm_e4m3(const void* xs, int x_rows, const float* x_scale, const float* x_sum, const void* W, int w_rows,
                             int ldw_bytes, int src, void* Y, int ldo, int out_fp32, int T, int N, int K, int gated, int dual_off,
                             const float* scale, const float* zero, int scale_ld, const float* bias, const void* residual, int ldr,
                             float res_scale, int act, const void* group_tiles, const int* num_group_tiles, int group_w_rows,
                             int max_tiles, int bn, const float* col_scale, int* status, cudaStream_t st) {
  if (T <= 0 || N <= 0 || K <= 0) return 0;
  if (K & 7) return -2;
  if (src == kSrcFp8 && ((gated && (dual_off & 127)) || (group_tiles && (group_w_rows & 127)))) return -4;
  if (src == kSrcU4 && (group_tiles || !zero || !x_sum)) return -4;
  E4Params p{};
  p.N = N; p.T = T; p.K = K; p.dual_off = dual_off; p.out = Y; p.ldo = ldo; p.out_fp32 = out_fp32; p.bias = bias;
  p.residual = (const __nv_bfloat16*)residual; p.ldr = ldr; p.res_scale = res_scale; p.act = act; p.x_scale = x_scale;
  p.x_sum = x_sum; p.scale = scale; p.zero = zero; p.scale_ld = scale_ld; p.status = status; p.col_scale = col_scale;
  p.group_tiles = reinterpret_cast<const int4*>(group_tiles); p.num_group_tiles = num_group_tiles; p.group_w_rows = group_w_rows;
  p.x_lo = xft_split_e4m3_cols(K);
  if (!group_tiles) bn = T <= 16 ? 16 : T <= 32 ? 32 : 64;
  const int feat = src == kSrcU4 && gated && bn <= 32 ? 64 : 128;                  // E4Layout::FEAT
  p.num_kb = (K + 127) / 128;
  p.n_tiles = (N + feat - 1) / feat;
  p.t_tiles = group_tiles ? max_tiles : (T + bn - 1) / bn;
  CUtensorMap tmW, tmX;
  int r = src == kSrcU4 ? make_byte_map(&tmW, W, (uint64_t)w_rows, (uint64_t)K / 2, (uint64_t)ldw_bytes, (uint32_t)feat, 64)
                        : make_tensor_map(&tmW, W, (uint64_t)w_rows, (uint64_t)K, (uint64_t)ldw_bytes, 128, 1);
  if (r) return 1000 - r;
  r = make_tensor_map(&tmX, xs, (uint64_t)x_rows, (uint64_t)2 * p.x_lo, (uint64_t)2 * p.x_lo, (uint32_t)bn, 1);
  if (r) return 2000 - r;
#define XFT_E4(BN_)                                                                                     \
  case BN_:                                                                                             \
    if (src == kSrcU4) return gated ? launch_e4<BN_, true, kSrcU4>(tmW, tmX, p, st) : launch_e4<BN_, false, kSrcU4>(tmW, tmX, p, st); \
    return gated ? launch_e4<BN_, true, kSrcFp8>(tmW, tmX, p, st) : launch_e4<BN_, false, kSrcFp8>(tmW, tmX, p, st);
  switch (bn) { XFT_E4(16) XFT_E4(32) XFT_E4(64) }
#undef XFT_E4
  return -1;
}

namespace xft {
// W8A8 at decode sizes (T <= 64), see xft_w8a8_gemm; gated: act(gate) * up, gate rows [0, N) and up rows from dual_off on.
int launch_w8a8_decode(const void* qx, int ldqx, const void* Wq, int w_rows, int ldw, void* Y, int ldo, int out_fp32, int T, int N, int K,
                       int gated, int dual_off, const float* a_scale, const float* a_zero, const float* a_qsum, const float* w_scale,
                       const float* w_zero, const float* w_sum, const float* bias, const void* residual, int ldr, float res_scale,
                       int act, int* status, cudaStream_t st) {
  E4Params p{};
  p.N = N; p.T = T; p.K = K; p.dual_off = dual_off; p.out = Y; p.ldo = ldo; p.out_fp32 = out_fp32; p.bias = bias;
  p.residual = (const __nv_bfloat16*)residual; p.ldr = ldr; p.res_scale = res_scale; p.act = act; p.x_scale = a_scale;
  p.a_zero = a_zero; p.a_qsum = a_qsum; p.scale = w_scale; p.zero = w_zero; p.w_sum = w_sum; p.status = status;
  const int bn = T <= 16 ? 16 : T <= 32 ? 32 : 64;
  p.num_kb = (K + 127) / 128;
  p.n_tiles = (N + 127) / 128;
  p.t_tiles = (T + bn - 1) / bn;
  CUtensorMap tmW, tmX;
  int r = make_tensor_map(&tmW, Wq, (uint64_t)w_rows, (uint64_t)K, (uint64_t)ldw, 128, 1);
  if (r) return 1000 - r;
  r = make_tensor_map(&tmX, qx, (uint64_t)T, (uint64_t)K, (uint64_t)ldqx, (uint32_t)bn, 1);
  if (r) return 2000 - r;
#define XFT_I8(BN_) \
  case BN_: return gated ? launch_e4<BN_, true, kSrcI8>(tmW, tmX, p, st) : launch_e4<BN_, false, kSrcI8>(tmW, tmX, p, st);
  switch (bn) { XFT_I8(16) XFT_I8(32) XFT_I8(64) }
#undef XFT_I8
  return -1;
}

int launch_w8a8_prompt(const void* qx, int ldqx, const void* Wq, int w_rows, int ldw, void* Y, int ldo, int out_fp32, int T, int N, int K,
                       int gated, int dual_off, const float* a_scale, const float* a_zero, const float* a_qsum, const float* w_scale,
                       const float* w_zero, const float* w_sum, const float* bias, const void* residual, int ldr, float res_scale,
                       int act, int* status, cudaStream_t st);      // gemm_prefill_sm100.cu
}  // namespace xft

// Y = epi(dequant(qx) · dequant(Wq)^T): qx int8 [T, K] with a_scale/a_zero/a_qsum from xft_quant_act, one scale and zero point per
// weight row; y = sa sw acc + sa zw sum(qx) + za sw sum(qw) + K za zw, then bias, activation, residual.  gated: act(gate) * up of
// gate rows [0, N) and up rows [dual_off, dual_off + N).  Up to 64 tokens the kernel above, then the
// token-major one of gemm_prefill_sm100.cu.
static int w8a8(const void* qx, int ldqx, const void* Wq, int ldw, void* Y, int ldo, int out_fp32, int T, int N, int K, int gated,
                int dual_off, const float* a_scale, const float* a_zero, const float* a_qsum, const float* w_scale, const float* w_zero,
                const float* w_sum, const float* bias, const void* residual, int ldr, float res_scale, int act, int* status,
                cudaStream_t st) {
  if (T <= 0 || N <= 0 || K <= 0) return 0;
  if (K % 16) return -4;
  const int w_rows = gated ? dual_off + N : N;
  return (T <= 64 ? launch_w8a8_decode : launch_w8a8_prompt)(qx, ldqx, Wq, w_rows, ldw, Y, ldo, out_fp32, T, N, K, gated, dual_off,
                                                             a_scale, a_zero, a_qsum, w_scale, w_zero, w_sum, bias, residual, ldr,
                                                             res_scale, act, status, st);
}

extern "C" int xft_w8a8_gemm(const void* qx, int ldqx, const void* Wq, int ldw, void* Y, int ldo, int out_fp32, int T, int N, int K,
                             const float* a_scale, const float* a_zero, const float* a_qsum, const float* w_scale, const float* w_zero,
                             const float* w_sum, const float* bias, const void* residual, int ldr, float res_scale, int act, float*,
                             size_t, int*, int, int* status, cudaStream_t st) {
  return w8a8(qx, ldqx, Wq, ldw, Y, ldo, out_fp32, T, N, K, 0, 0, a_scale, a_zero, a_qsum, w_scale, w_zero, w_sum, bias, residual, ldr,
              res_scale, act, status, st);
}

extern "C" int xft_w8a8_gemm_gated(const void* qx, int ldqx, const void* Wq, int ldw, void* Y, int ldo, int T, int N, int K, int dual_off,
                                   const float* a_scale, const float* a_zero, const float* a_qsum, const float* w_scale,
                                   const float* w_zero, const float* w_sum, const float* bias, int act, int* status, cudaStream_t st) {
  return w8a8(qx, ldqx, Wq, ldw, Y, ldo, 0, T, N, K, 1, dual_off, a_scale, a_zero, a_qsum, w_scale, w_zero, w_sum, bias, nullptr, 0, 1.f,
              act, status, st);
}

// Y = epi(X W^T) for T <= 64, bf16 operands on the same pipeline; arguments as xft_gemm_bf16 (gemm_sm100.cu), rms_eps as in xft_gemm_sk.
// rms_ssq: room for T floats, or null.  With it the rows' sums of squares are a launch of their own (2 us); without it every CTA adds
// them up beside its weight stream, which at 64 rows costs more than the stream hides (12288 x 4096: 10 us, at 16 rows 1 us).
extern "C" int xft_gemm_bf16_cluster(const void* X, int ldx, const void* W, int w_rows, int ldw, void* Y, int ldo, int out_fp32, int T,
                                     int N, int K, int gated, int dual_off, const float* bias, const void* residual, int ldr,
                                     float res_scale, int act, const float* rms_eps, float* rms_ssq, int* status, cudaStream_t st) {
  if (T <= 0 || N <= 0 || K <= 0) return 0;
  if (T > 64 || (K & 7) || (ldx & 7) || (ldw & 7)) return -2;
  E4Params p{};
  if (rms_eps) { p.rms_x = (const __nv_bfloat16*)X; p.rms_ldx = ldx; p.rms_eps = *rms_eps; p.rms_ssq = rms_ssq; }
  p.N = N; p.T = T; p.K = K; p.dual_off = dual_off; p.out = Y; p.ldo = ldo; p.out_fp32 = out_fp32; p.bias = bias;
  p.residual = (const __nv_bfloat16*)residual; p.ldr = ldr; p.res_scale = res_scale; p.act = act; p.status = status;
  const int bn = T <= 16 ? 16 : T <= 32 ? 32 : 64;
  p.num_kb = (K + 63) / 64;
  p.n_tiles = (N + 127) / 128;
  p.t_tiles = (T + bn - 1) / bn;
  CUtensorMap tmW, tmX;
  int r = make_tensor_map(&tmW, W, (uint64_t)w_rows, (uint64_t)K, (uint64_t)ldw, 128, 2);
  if (r) return 1000 - r;
  r = make_tensor_map(&tmX, X, (uint64_t)T, (uint64_t)K, (uint64_t)ldx, (uint32_t)bn, 2);
  if (r) return 2000 - r;
  if (rms_eps && rms_ssq) {
    const cudaError_t e = launch_pdl(row_ssq_kernel, dim3(T), dim3(256), 0, st, p.rms_x, ldx, K, rms_ssq);
    if (e != cudaSuccess) return (int)e;
  }
#define XFT_BF(BN_) \
  case BN_: return gated ? launch_e4<BN_, true, kSrcBf16>(tmW, tmX, p, st) : launch_e4<BN_, false, kSrcBf16>(tmW, tmX, p, st);
  switch (bn) { XFT_BF(16) XFT_BF(32) XFT_BF(64) }
#undef XFT_BF
  return -1;
}
