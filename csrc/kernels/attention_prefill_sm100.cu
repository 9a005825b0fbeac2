// Prefill attention for sm_100a on the 5th-generation tensor cores: causal flash attention over the paged KV cache,
// head_dim 128, bf16 cache, GQA.
//
// Replaces the reference's prompt-phase attention (src/kernels/attention_kernels.h:142-552 crossAttnByHead /
// selfAttention with its small-GEMM softmax loop, and the flash variant at :1285-1408) with one kernel per
// (128 query rows, head, sequence):
//
//   S = Q K^T   tcgen05.mma, A = the query tile [128 rows x 128] (K-major, shared memory, loaded once by TMA),
//               B = 128 keys of the cache (two 64-token blocks of the block table, K-major), D = S in TMEM (fp32, 128 columns)
//   P = softmax row by row: four warps, one query row (= one TMEM lane) per thread, read S with tcgen05.ld, keep the
//               running maximum and sum in registers, write P as bf16 over S
//   O = P V     tcgen05.mma, A = P (TMEM), B = the same 128 cache rows of V used as an MN-major operand
//               (rows = keys = the contraction dimension, the 128 head features contiguous: no transpose is needed),
//               D = the tile's contribution in TMEM; the four warps add it to their fp32 accumulator rows in registers
//               with the usual exp(m_old - m_new) correction
//
// Bound by the chain S -> softmax -> P -> O of a tile: the products are 1024 cycles of it, the exponentials 1024 at least (16 per
// cycle and SM).  Two CTAs share an SM (96 KB, 256 TMEM columns, 256 x 128 registers each), so that one's products run beside the
// other's softmax and one's start and finish beside the other's tiles; two query tiles in one CTA with shared K and V were no faster
// (their CTAs start alone).  Each product is issued in halves as soon as its half of P is written, a chunk of S is on its way from
// TMEM while the one before is worked on, and exponentials are interleaved with the rounding of the chunk before.  The order of
// every sum is that of one tile of 128 keys after the other.  us, one tile per SM and P through shared memory / now: 4 x 2048
// tokens, 64 and 8 heads 735 / 375; 8 x 950, 32 heads 231 / 139; 32 x 128 59 / 45; int8 cache, 2 x 2880, 32 and 8 heads 726 / 255.
//
// CTAs with the most keys to visit (the last query rows of a causal prompt) are scheduled first, over all heads and sequences.
//
// Warp roles: warp 0 = TMA producer, warp 1 = TMEM owner + MMA issuer, warps 4-7 = softmax / output.
// Every wait is bounded and reports through the status word.
//
// attn_prefill_ext_kernel adds, each with its constants as launch parameters: a sliding window with kept first keys (only
// the key tiles that hold a visible key are visited: first those of the kept keys, then those of the window), a tanh cap
// on the scores, and one sink per query head (a term of the softmax denominator without key or value).
#include "ptx.cuh"

namespace xft {

int make_tensor_map(CUtensorMap* out, const void* ptr, uint64_t rows, uint64_t cols, uint64_t ld, uint32_t box_rows,
                    uint32_t esize);

struct PrefillAttnParams {
  __nv_bfloat16* out;        // [T, hq, 128]
  const int* block_table; int bt_stride;
  const int* cu_q; const int* kv_lens;
  int hq, hkv, group, q_off;  // kv head of query head h = (h + q_off) / group
  int bs;                     // tokens per cache block (64)
  float scale_log2;           // softmax scale * log2(e)
  // attn_prefill_ext_kernel
  float cap_log2, inv_cap;    // softcap * log2(e), scale / softcap (cap_log2 0: no cap)
  int window, keep;           // keys within `window` positions and the first `keep` are visible (window 2^30: all)
  const float* sinks;         // [hq] or null
  int num_blocks;
  // INT8 only: the scales of the int8 cache [num_blocks, hkv, bs]; the K / V tiles come from a copy of the codes in bf16, where
  // block j of sequence b is at b * copy_w + j
  const float* ks; const float* vs;
  int copy_w;
  int* status;
};

constexpr int kPfTile = 128;                 // keys per tile = two cache blocks
constexpr int kPfQ = 128;                    // query rows of a tile
constexpr int kPfHalf = kPfTile * 128;       // bytes of one 64-feature half of a 128-row tile (128 rows x 128 B)
constexpr int kPfTileBytes = 2 * kPfHalf;    // 32 KB: each Q tile, each K / V stage

constexpr int kPfScales = 2 * kPfTile * 4;   // int8 cache: scales of a tile's keys and values, in a ring of two
constexpr int kPfSmem = 3 * kPfTileBytes + 1024, kPfSmemInt8 = kPfSmem + 2 * kPfScales;
constexpr int kPfThreads = 256;
constexpr int kPfExtSmem = 6 * kPfTileBytes + 1024;      // attn_prefill_ext_kernel: Q, P, K x 2, V x 2

__device__ __forceinline__ float fmax3(float a, float b, float c) {
  float d;
  asm("max.ftz.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
// Two products or sums in one instruction
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  float2 d;
  asm("fma.rn.ftz.f32x2 %0, %1, %2, %3;"
      : "=l"(reinterpret_cast<unsigned long long&>(d))
      : "l"(reinterpret_cast<unsigned long long&>(a)), "l"(reinterpret_cast<unsigned long long&>(b)), "l"(reinterpret_cast<unsigned long long&>(c)));
  return d;
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  float2 d;
  asm("add.rn.ftz.f32x2 %0, %1, %2;"
      : "=l"(reinterpret_cast<unsigned long long&>(d))
      : "l"(reinterpret_cast<unsigned long long&>(a)), "l"(reinterpret_cast<unsigned long long&>(b)));
  return d;
}
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  const __nv_bfloat162 b = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&b);
}

// INT8: K and V are the codes of an int8 cache (exact in bf16); a key's scale multiplies its score and its weight in fp32, as in the
// kernel for other head sizes (attention.cu).
template <bool INT8>
__global__ void __launch_bounds__(kPfThreads, 2)
    attn_prefill_tc_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                           const __grid_constant__ CUtensorMap tmV, const PrefillAttnParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem;
  uint8_t* sK = smem + kPfTileBytes;
  uint8_t* sV = smem + 2 * kPfTileBytes;
  float* s_scales = reinterpret_cast<float*>(smem + 3 * kPfTileBytes);
  __shared__ uint64_t q_full, k_full, k_empty, v_full, v_empty, s_full, p_half, p_full, o_full, c_full[2], c_empty[2];
  __shared__ uint32_t tmem_base_s;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int h = blockIdx.x, b = blockIdx.y;
  const int q0 = p.cu_q[b], q_len = p.cu_q[b + 1] - q0, kv_len = p.kv_lens[b];
  // heavy rows first, over all heads and sequences: the last query rows of a causal prompt visit the most keys
  const int n_qt = (q_len + kPfQ - 1) / kPfQ;
  if ((int)blockIdx.z >= n_qt) return;
  const int row0 = (n_qt - 1 - (int)blockIdx.z) * kPfQ;
  const int past = kv_len - q_len;            // keys before this call's first query
  const int last_row = min(row0 + kPfQ, q_len) - 1;
  const int n_tiles = (min(kv_len, past + last_row + 1) + kPfTile - 1) / kPfTile;
  const int kvh = (h + p.q_off) / p.group;

  if (threadIdx.x == 0) {
    mbar_init(&q_full, 1);
    mbar_init(&k_full, 1); mbar_init(&k_empty, 1);
    mbar_init(&v_full, 1); mbar_init(&v_empty, 1);
    mbar_init(&s_full, 1); mbar_init(&o_full, 1);
    mbar_init(&p_half, 4); mbar_init(&p_full, 4);        // one arrival per softmax warp
    for (int s = 0; s < 2; ++s) { mbar_init(&c_full[s], 1); mbar_init(&c_empty[s], 4); }
    fence_barrier_init();
    fence_proxy_async();
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
  }
  if (warp == 1) {
    tmem_alloc(&tmem_base_s, 256);             // S, whose first half becomes P, and O
    tmem_relinquish();
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem_base = tmem_base_s;
  grid_dep_launch();
  grid_dep_wait();

  // registers: 256 x 128 at launch, 128 x 40 + 128 x 216 from here on
  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
    if (warp == 0) {
      // ------------------------------------------------------------------ TMA producer
      if (elect_one()) {
        mbar_expect_tx(&q_full, kPfTileBytes);
        // q is [T, hq * 128]: rows past the end of the tensor read as zero, rows of the next sequence are never stored
        tma_load_2d(sQ, &tmQ, &q_full, h * 128, q0 + row0, kEvictFirst);
        tma_load_2d(sQ + kPfHalf, &tmQ, &q_full, h * 128 + 64, q0 + row0, kEvictFirst);
        const int* bt = p.block_table + (size_t)b * p.bt_stride;
        const int n_blocks = (kv_len + p.bs - 1) / p.bs;
        for (int j = 0; j < n_tiles; ++j) {
          // cache rows of the two blocks of this tile; past the sequence's last block the last one is read again
          // (finite values; those keys are masked)
          int rowk[2], rowc[2];
          bool bad = false;
          for (int i = 0; i < 2; ++i) {
            int blk = bt[min(2 * j + i, n_blocks - 1)];
            if (blk < 0 || blk >= p.num_blocks) { bad = true; blk = 0; }
            rowc[i] = (blk * p.hkv + kvh) * p.bs;
            if (INT8) blk = b * p.copy_w + min(2 * j + i, n_blocks - 1);
            rowk[i] = (blk * p.hkv + kvh) * p.bs;
          }
          if (bad && p.status) atomicCAS(p.status, 0, XFT_ERR_BOUNDS);
          if (!mbar_wait(&k_empty, (j & 1) ^ 1, p.status, XFT_ERR_WAIT_EMPTY)) break;
          mbar_expect_tx(&k_full, kPfTileBytes);
          for (int i = 0; i < 2; ++i) {
            tma_load_2d(sK + i * 8192, &tmK, &k_full, 0, rowk[i], kEvictNormal);
            tma_load_2d(sK + kPfHalf + i * 8192, &tmK, &k_full, 64, rowk[i], kEvictNormal);
          }
          if constexpr (INT8) {
            const int s = j & 1;
            if (!mbar_wait(&c_empty[s], ((j >> 1) & 1) ^ 1, p.status, XFT_ERR_WAIT_EMPTY)) break;
            mbar_expect_tx(&c_full[s], kPfScales);
            float* to = s_scales + s * 2 * kPfTile;
            for (int i = 0; i < 2; ++i) {
              bulk_load(to + i * 64, p.ks + rowc[i], 256, &c_full[s]);
              bulk_load(to + kPfTile + i * 64, p.vs + rowc[i], 256, &c_full[s]);
            }
          }
          if (!mbar_wait(&v_empty, (j & 1) ^ 1, p.status, XFT_ERR_WAIT_EMPTY)) break;
          mbar_expect_tx(&v_full, kPfTileBytes);
          for (int i = 0; i < 2; ++i) {
            tma_load_2d(sV + i * 8192, &tmV, &v_full, 0, rowk[i], kEvictNormal);
            tma_load_2d(sV + kPfHalf + i * 8192, &tmV, &v_full, 64, rowk[i], kEvictNormal);
          }
        }
      }
    } else if (warp == 1) {
      // ------------------------------------------------------------------ MMA issuer
      if (elect_one()) {
        // S = Q K^T: both operands K-major, M = 128 query rows, N = 128 keys, K = 128 features in 8 steps of 16
        constexpr uint32_t IDESC_S = umma_idesc(128, 128, 1, 1, 1);
        // O = P V: A = P (tensor memory), B = V MN-major (bit 16), N = 128 features, K = 128 keys
        constexpr uint32_t IDESC_O = umma_idesc(128, 128, 1, 1, 1) | (1u << 16);
        const uint64_t qd = umma_desc_k128(smem_u32(sQ)), kd = umma_desc_k128(smem_u32(sK));
        const uint64_t vd = umma_desc_mn128(smem_u32(sV), kPfHalf);
        bool ok = mbar_wait(&q_full, 0, p.status, XFT_ERR_WAIT_FULL);
        for (int j = 0; j <= n_tiles && ok; ++j) {
          if (j > 0) {                                                   // 16 keys = 8 columns of P, 16 rows of 128 bytes of V
            const uint32_t ph = (j - 1) & 1;
            ok = mbar_wait(&v_full, ph, p.status, XFT_ERR_WAIT_FULL) && mbar_wait(&p_half, ph, p.status, XFT_ERR_WAIT_TMEM);
            if (!ok) break;
            tcgen05_fence_after();
#pragma unroll
            for (int kk = 0; kk < 4; ++kk)
              umma_bf16_ta(tmem_base + 128, tmem_base + kk * 8, vd + kk * (2048 / 16), IDESC_O, kk > 0);
            ok = mbar_wait(&p_full, ph, p.status, XFT_ERR_WAIT_TMEM);
            if (!ok) break;
            tcgen05_fence_after();
#pragma unroll
            for (int kk = 4; kk < 8; ++kk)
              umma_bf16_ta(tmem_base + 128, tmem_base + kk * 8, vd + kk * (2048 / 16), IDESC_O, 1);
            tcgen05_commit(&v_empty);
            tcgen05_commit(&o_full);
          }
          if (j == n_tiles) break;
          // the next S is written over P: issued behind the product that reads P, it is carried out behind it
          ok = mbar_wait(&k_full, j & 1, p.status, XFT_ERR_WAIT_FULL);
          if (!ok) break;
          tcgen05_fence_after();
#pragma unroll
          for (int kk = 0; kk < 8; ++kk) {
            const uint32_t off = ((kk >> 2) * kPfHalf + (kk & 3) * 32) / 16;     // feature half, then 16 features = 32 bytes
            umma_bf16(tmem_base, qd + off, kd + off, IDESC_S, kk > 0);
          }
          tcgen05_commit(&k_empty);
          tcgen05_commit(&s_full);
        }
      }
    }
  } else {
    // ------------------------------------------------------------------ softmax + output: one query row per thread
    asm volatile("setmaxnreg.inc.sync.aligned.u32 216;");
    const int qd = warp & 3;
    const int r = qd * 32 + lane;                          // row of the tile = TMEM lane
    const int qrow = row0 + r;
    // rows past the sequence's end attend like its last row (finite numbers, never stored)
    const int qpos = past + min(qrow, q_len - 1);
    const uint32_t sa = tmem_base + (uint32_t(qd * 32) << 16), oa = sa + 128;
    float2 o[64];
#pragma unroll
    for (int i = 0; i < 64; ++i) o[i] = make_float2(0.f, 0.f);
    float m = -INFINITY, l = 0.f;
    bool ok = true;
    for (int j = 0; j < n_tiles; ++j) {
      if (INT8 && !mbar_wait(&c_full[j & 1], (j >> 1) & 1, p.status, XFT_ERR_WAIT_FULL)) { ok = false; break; }
      if (!mbar_wait(&s_full, j & 1, p.status, XFT_ERR_WAIT_TMEM)) { ok = false; break; }
      tcgen05_fence_after();
      const int k0 = j * kPfTile;
      const int nvalid = min(qpos, kv_len - 1) - k0 + 1;    // keys [k0, k0 + nvalid) are visible to this row
      float* scales = s_scales + (j & 1) * 2 * kPfTile;     // INT8: of the tile's keys, then of its values
      const bool whole = __all_sync(0xffffffffu, nvalid >= 128);
      int chunks = 8;                                        // chunks of 16 keys, in twos, that hold all that the rows of this warp see
      if (!whole) {
        chunks = 0;
#pragma unroll
        for (int c = 0; c < 128; c += 32)
          if (__any_sync(0xffffffffu, nvalid > c)) chunks = (c >> 4) + 2;
        if (INT8 && k0 + kPfTile > kv_len) {                 // slots that no one has written since their last owner: 0 x their scale can be NaN
          for (int i = lane; i < kPfTile; i += 32)
            if (k0 + i >= kv_len) scales[i] = scales[kPfTile + i] = 0.f;
          fence_proxy_async();
          __syncwarp();
        }
      }
      // pass 1: row maximum of the visible raw scores (the scale is positive).  Scores of hidden keys become -inf and those of an int8
      // cache are scaled, back in tensor memory.  Of both passes' chunks the next is on its way while one is worked on.
      float mc[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
      uint32_t v[3][16];
      auto largest = [&](const uint32_t (&x)[16]) {
#pragma unroll
        for (int i = 0; i < 16; i += 2) mc[(i >> 1) & 3] = fmax3(mc[(i >> 1) & 3], __uint_as_float(x[i]), __uint_as_float(x[i + 1]));
      };
      auto hide = [&](uint32_t (&x)[16], int c) {
#pragma unroll
        for (int i = 0; i < 16; ++i)
          if (c + i >= nvalid) x[i] = 0xff800000u;
      };
      if constexpr (INT8) {
        float4 f[2][4];                                      // scales of a chunk's keys
        auto fetch = [&](int k) {
#pragma unroll
          for (int i = 0; i < 4; ++i) f[k & 1][i] = *reinterpret_cast<const float4*>(scales + 16 * k + 4 * i);
        };
        tmem_ld16(sa, v[0]);
        fetch(0);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          uint32_t (&x)[16] = v[k & 1];
          if (k < chunks) {
            tmem_ld_wait(x);
            if (k < 7) {
              tmem_ld16(sa + 16 * k + 16, v[(k + 1) & 1]);
              fetch(k + 1);
            }
#pragma unroll
            for (int i = 0; i < 16; ++i) x[i] = __float_as_uint(__uint_as_float(x[i]) * (&f[k & 1][i >> 2].x)[i & 3]);
            if (!whole) hide(x, 16 * k);
            tmem_st16(sa + 16 * k, x);
            largest(x);
          }
        }
        tmem_ld_wait(v[0]);
        tmem_st_wait();
      } else {
        if (!whole) {
#pragma unroll 1
          for (int c = 0; c < 16 * chunks; c += 16) {
            tmem_ld16(sa + c, v[0]);
            tmem_ld_wait(v[0]);
            hide(v[0], c);
            tmem_st16(sa + c, v[0]);
          }
          tmem_st_wait();
        }
        tmem_ld16(sa, v[0]);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          tmem_ld_wait(v[k & 1]);
          if (k < 7) tmem_ld16(sa + 16 * k + 16, v[(k + 1) & 1]);
          if (k < chunks) largest(v[k & 1]);
        }
      }
      // raw maximum -inf: nothing visible in this tile.  m = -inf on the first tile: alpha = 0, o and l are 0
      const float mx = fmaxf(m, fmaxf(fmaxf(mc[0], mc[1]), fmaxf(mc[2], mc[3])) * p.scale_log2);
      const float alpha = exp2f(m - mx);
      m = mx;
      // pass 2: P = exp2(s - m) as bf16 over the scores, 16 of which become 8 columns; row sum.  A chunk's exponentials are taken while
      // those of the one before are rounded, added and stored: one warp's instructions issue in order, and one behind an exponential
      // waits for the eight cycles that each of these takes.
      float sum = 0.f;
      auto exponentials = [&](uint32_t (&x)[16], int i) {    // of keys i .. i + 3 of the chunk
#pragma unroll
        for (int e = i; e < i + 4; e += 2) {
          const float2 s2 = fma2(make_float2(__uint_as_float(x[e]), __uint_as_float(x[e + 1])), make_float2(p.scale_log2, p.scale_log2), make_float2(-m, -m));
          x[e] = __float_as_uint(exp2f(s2.x));
          x[e + 1] = __float_as_uint(exp2f(s2.y));
        }
      };
      auto rounded = [&](const uint32_t (&x)[16], uint32_t (&w)[8], int i, int k) {
        const float e0 = __uint_as_float(x[i]), e1 = __uint_as_float(x[i + 1]), e2 = __uint_as_float(x[i + 2]), e3 = __uint_as_float(x[i + 3]);
        uint32_t& w0 = w[i >> 1];
        uint32_t& w1 = w[(i >> 1) + 1];
        float2 add;
        if constexpr (INT8) {                                // the value's scale belongs to the product, not to the sum
          const float4 f = *reinterpret_cast<const float4*>(scales + kPfTile + 16 * k + i);
          w0 = pack_bf16(e0 * f.x, e1 * f.y);
          w1 = pack_bf16(e2 * f.z, e3 * f.w);
          add = add2(make_float2(e0, e2), make_float2(e1, e3));
        } else {                                             // the sum uses the rounded values, as the product does
          w0 = pack_bf16(e0, e1);
          w1 = pack_bf16(e2, e3);
          add = add2(make_float2(__uint_as_float(w0 << 16), __uint_as_float(w1 << 16)),
                     make_float2(__uint_as_float(w0 & 0xffff0000u), __uint_as_float(w1 & 0xffff0000u)));
        }
        sum += add.x;
        sum += add.y;
      };
      if (chunks > 0) {
        tmem_ld16(sa, v[0]);
        tmem_ld_wait(v[0]);
        tmem_ld16(sa + 16, v[1]);
#pragma unroll
        for (int i = 0; i < 16; i += 4) exponentials(v[0], i);
      }
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        uint32_t (&now)[16] = v[k % 3];
        uint32_t (&next)[16] = v[(k + 1) % 3];
        uint32_t w[8] = {};
        if (k < chunks) {
          if (k + 1 < 8) {
            tmem_ld_wait(next);
            if (k + 2 < 8) tmem_ld16(sa + 16 * k + 32, v[(k + 2) % 3]);
#pragma unroll
            for (int i = 0; i < 16; i += 4) {
              exponentials(next, i);
              rounded(now, w, i, k);
            }
          } else {
#pragma unroll
            for (int i = 0; i < 16; i += 4) rounded(now, w, i, k);
          }
        }
        tmem_st8(sa + 8 * k, w);
        if (k == 3) {                                        // the product may begin with the first 64 keys
          tmem_st_wait();
          tcgen05_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&p_half);
        }
      }
      l = l * alpha + sum;
      // P is complete
      tmem_st_wait();
      tcgen05_fence_before();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(&p_full);
        if (INT8) mbar_arrive(&c_empty[j & 1]);
      }
      // this tile's P V, added to the row's accumulator with the correction for the new maximum
      if (!mbar_wait(&o_full, j & 1, p.status, XFT_ERR_WAIT_TMEM)) { ok = false; break; }
      tcgen05_fence_after();
      {
        uint32_t v[2][16];
        tmem_ld16(oa, v[0]);
#pragma unroll
        for (int c = 0; c < 128; c += 16) {
          tmem_ld_wait(v[(c >> 4) & 1]);
          if (c < 112) tmem_ld16(oa + c + 16, v[((c >> 4) + 1) & 1]);
          const uint32_t (&x)[16] = v[(c >> 4) & 1];
#pragma unroll
          for (int i = 0; i < 16; i += 2)
            o[(c + i) >> 1] = fma2(o[(c + i) >> 1], make_float2(alpha, alpha), make_float2(__uint_as_float(x[i]), __uint_as_float(x[i + 1])));
        }
      }
      tcgen05_fence_before();
    }
    if (ok && qrow < q_len) {
      const float inv = l > 0.f ? 1.f / l : 0.f;
      __nv_bfloat16* dst = p.out + ((size_t)(q0 + qrow) * p.hq + h) * 128;
#pragma unroll
      for (int c = 0; c < 128; c += 8) {
        uint32_t w[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) w[i] = pack_bf16(o[c / 2 + i].x * inv, o[c / 2 + i].y * inv);
        *reinterpret_cast<uint4*>(dst + c) = make_uint4(w[0], w[1], w[2], w[3]);
      }
    }
  }
  __syncwarp();
  tcgen05_fence_before();
  __syncthreads();
  if (warp == 1) {
    tcgen05_fence_after();
    tmem_dealloc(tmem_base, 256);
  }
}

// Capped score in log2 units, cap * tanh(z) with z = raw * scale / cap: tanh(z) = 1 - 2 / (1 + exp(2z)).
__device__ __forceinline__ float capped_log2(const PrefillAttnParams& p, float raw) {
  return p.cap_log2 - __fdividef(2.f * p.cap_log2, 1.f + exp2f(fminf(raw * p.inv_cap * 2.8853900817779268f, 120.f)));
}
// The same for |z| <= 1 without the special-function unit: tanh(z) / z as a polynomial in z^2, fitted with minimax
// weights on [0, 1] (relative error below 2e-7, the size of the rounding).
__device__ __forceinline__ float capped_log2_small(const PrefillAttnParams& p, float raw) {
  const float z = raw * p.inv_cap, t = z * z;
  float q = 0.0010410224785f;
  q = fmaf(q, t, -0.0062033790164f);
  q = fmaf(q, t, 0.020289981738f);
  q = fmaf(q, t, -0.053457029164f);
  q = fmaf(q, t, 0.13325203957f);
  q = fmaf(q, t, -0.33332839608f);
  q = fmaf(q, t, 0.99999994040f);
  return z * p.cap_log2 * q;
}

// Windows, kept first keys, caps and sinks: one tile of queries per SM whose softmax and products take turns, P through shared memory.
// Chunks of keys that no row sees are skipped wherever they lie, in loops: the straight-line code of the kernel above, in the versions
// that the cap needs, does not stay in the instruction cache (4 x 2048 tokens, 32 heads, cap and window: 451 us here, 578 there).
__global__ void __launch_bounds__(192, 1) attn_prefill_ext_kernel(const __grid_constant__ CUtensorMap tmQ,
                                                                  const __grid_constant__ CUtensorMap tmK,
                                                                  const __grid_constant__ CUtensorMap tmV,
                                                                  const PrefillAttnParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem;
  uint8_t* sP = smem + kPfTileBytes;
  uint8_t* sK = smem + 2 * kPfTileBytes;      // two stages
  uint8_t* sV = smem + 4 * kPfTileBytes;      // two stages
  __shared__ uint64_t q_full, k_full[2], k_empty[2], v_full[2], v_empty[2], s_full[2], p_full, o_full;
  __shared__ uint32_t tmem_base_s;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int b = blockIdx.z, h = blockIdx.y;
  const int q0 = p.cu_q[b], q_len = p.cu_q[b + 1] - q0, kv_len = p.kv_lens[b];
  // heavy tiles first: the last query rows of a causal prompt visit the most keys
  const int n_qt = (q_len + kPfQ - 1) / kPfQ;
  if ((int)blockIdx.x >= n_qt) return;
  const int row0 = (n_qt - 1 - (int)blockIdx.x) * kPfQ;
  const int past = kv_len - q_len;            // keys before this call's first query
  const int last_row = min(row0 + kPfQ, q_len) - 1;
  const int end_tile = (min(kv_len, past + last_row + 1) + kPfTile - 1) / kPfTile;
  // the tiles to visit: [0, keep_tiles) and [lo_tile, end_tile)
  const int lo_tile = min(max(0, past + row0 - p.window + 1) / kPfTile, end_tile);
  const int keep_tiles = min((p.keep + kPfTile - 1) / kPfTile, lo_tile);
  const int n_tiles = keep_tiles + end_tile - lo_tile;
  auto tile_of = [&](int j) { return j < keep_tiles ? j : j - keep_tiles + lo_tile; };
  const int kvh = (h + p.q_off) / p.group;

  if (threadIdx.x == 0) {
    mbar_init(&q_full, 1);
    for (int s = 0; s < 2; ++s) {
      mbar_init(&k_full[s], 1); mbar_init(&k_empty[s], 1);
      mbar_init(&v_full[s], 1); mbar_init(&v_empty[s], 1);
      mbar_init(&s_full[s], 1);
    }
    mbar_init(&p_full, 4);                     // one arrival per softmax warp
    mbar_init(&o_full, 1);
    fence_barrier_init();
    fence_proxy_async();
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
  }
  if (warp == 1) {
    tmem_alloc(&tmem_base_s, 512);             // S x 2 (256 columns) + O tile (128), rounded up to a power of two
    tmem_relinquish();
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem_base = tmem_base_s;
  grid_dep_launch();
  grid_dep_wait();

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (elect_one()) {
      mbar_expect_tx(&q_full, kPfTileBytes);
      // q is [T, hq * 128]: rows past the end of the tensor read as zero, rows of the next sequence are never stored
      tma_load_2d(sQ, &tmQ, &q_full, h * 128, q0 + row0, kEvictFirst);
      tma_load_2d(sQ + kPfHalf, &tmQ, &q_full, h * 128 + 64, q0 + row0, kEvictFirst);
      const int* bt = p.block_table + (size_t)b * p.bt_stride;
      const int n_blocks = (kv_len + p.bs - 1) / p.bs;
      for (int j = 0; j < n_tiles; ++j) {
        const int s = j & 1;
        const uint32_t ph = (j >> 1) & 1;
        // cache rows of the two blocks of this tile; past the sequence's last block the last one is read again
        // (finite values; those keys are masked)
        int rowk[2];
        bool bad = false;
        for (int i = 0; i < 2; ++i) {
          int blk = bt[min(2 * tile_of(j) + i, n_blocks - 1)];
          if (blk < 0 || blk >= p.num_blocks) { bad = true; blk = 0; }
          rowk[i] = (blk * p.hkv + kvh) * p.bs;
        }
        if (bad && p.status) atomicCAS(p.status, 0, XFT_ERR_BOUNDS);
        if (!mbar_wait(&k_empty[s], ph ^ 1, p.status, XFT_ERR_WAIT_EMPTY)) break;
        mbar_expect_tx(&k_full[s], kPfTileBytes);
        uint8_t* k = sK + s * kPfTileBytes;
        for (int i = 0; i < 2; ++i) {
          tma_load_2d(k + i * 8192, &tmK, &k_full[s], 0, rowk[i], kEvictNormal);
          tma_load_2d(k + kPfHalf + i * 8192, &tmK, &k_full[s], 64, rowk[i], kEvictNormal);
        }
        if (!mbar_wait(&v_empty[s], ph ^ 1, p.status, XFT_ERR_WAIT_EMPTY)) break;
        mbar_expect_tx(&v_full[s], kPfTileBytes);
        uint8_t* v = sV + s * kPfTileBytes;
        for (int i = 0; i < 2; ++i) {
          tma_load_2d(v + i * 8192, &tmV, &v_full[s], 0, rowk[i], kEvictNormal);
          tma_load_2d(v + kPfHalf + i * 8192, &tmV, &v_full[s], 64, rowk[i], kEvictNormal);
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (elect_one()) {
      // S = Q K^T: both operands K-major, M = 128 query rows, N = 128 keys, K = 128 features in 8 steps of 16
      constexpr uint32_t IDESC_S = umma_idesc(128, 128, 1, 1, 1);
      // O = P V: A = P K-major (keys contiguous), B = V MN-major (bit 16), N = 128 features, K = 128 keys
      constexpr uint32_t IDESC_O = umma_idesc(128, 128, 1, 1, 1) | (1u << 16);
      auto issue_s = [&](int j) -> bool {
        const int s = j & 1;
        if (!mbar_wait(&k_full[s], (j >> 1) & 1, p.status, XFT_ERR_WAIT_FULL)) return false;
        tcgen05_fence_after();
        const uint32_t qa = smem_u32(sQ), ka = smem_u32(sK + s * kPfTileBytes);
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {
          const uint32_t off = (kk >> 2) * kPfHalf + (kk & 3) * 32;       // feature half, then 16 features = 32 bytes
          umma_bf16(tmem_base + (uint32_t)(s * 128), umma_desc_k128(qa + off), umma_desc_k128(ka + off), IDESC_S, kk > 0);
        }
        tcgen05_commit(&k_empty[s]);
        tcgen05_commit(&s_full[s]);
        return true;
      };
      bool ok = mbar_wait(&q_full, 0, p.status, XFT_ERR_WAIT_FULL) && issue_s(0);
      for (int j = 0; j < n_tiles && ok; ++j) {
        if (j + 1 < n_tiles) ok = issue_s(j + 1);          // runs while the softmax warps work on tile j
        if (!ok) break;
        const int s = j & 1;
        if (!mbar_wait(&p_full, j & 1, p.status, XFT_ERR_WAIT_TMEM)) break;
        if (!mbar_wait(&v_full[s], (j >> 1) & 1, p.status, XFT_ERR_WAIT_FULL)) break;
        tcgen05_fence_after();
        const uint32_t pa = smem_u32(sP), va = smem_u32(sV + s * kPfTileBytes);
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {
          // A: 16 keys = 32 bytes inside the 64-key half; B: 16 keys = 16 rows of 128 bytes
          const uint32_t aoff = (kk >> 2) * kPfHalf + (kk & 3) * 32;
          umma_bf16(tmem_base + 256, umma_desc_k128(pa + aoff), umma_desc_mn128(va + kk * 2048, kPfHalf), IDESC_O, kk > 0);
        }
        tcgen05_commit(&v_empty[s]);
        tcgen05_commit(&o_full);
      }
    }
  } else {
    // ------------------------------------------------------------------ softmax + output: one query row per thread
    const int qd = warp & 3;
    const int r = qd * 32 + lane;                          // row of the tile = TMEM lane
    const int qrow = row0 + r;
    // rows past the sequence's end attend like its last row (finite numbers, never stored)
    const int qpos = past + min(qrow, q_len - 1);
    const uint32_t lane_addr = tmem_base + (uint32_t(qd * 32) << 16);
    float o[128];
#pragma unroll
    for (int i = 0; i < 128; ++i) o[i] = 0.f;
    float m = -INFINITY, l = 0.f;
    if (p.sinks) { m = p.sinks[h] * 1.4426950408889634f; l = 1.f; }
    bool ok = true;
    for (int j = 0; j < n_tiles; ++j) {
      const int s = j & 1;
      if (!mbar_wait(&s_full[s], (j >> 1) & 1, p.status, XFT_ERR_WAIT_TMEM)) { ok = false; break; }
      tcgen05_fence_after();
      const uint32_t sa = lane_addr + (uint32_t)(s * 128);
      const int k0 = tile_of(j) * kPfTile;
      const int nvalid = min(qpos, kv_len - 1) - k0 + 1;    // keys [k0, k0 + nvalid) are visible to this row
      // of these, the ones from k0 + first on and the ones below k0 + kept
      const int first = qpos - p.window + 1 - k0, kept = p.keep - k0;
      auto visible = [&](int i) { return i < nvalid && (i >= first || i < kept); };
      // pass 1: row maximum of the visible scores
      float mx = -INFINITY;
      float big = 0.f;                                       // largest |raw score| of the row
      // which of the four 32-key chunks hold no key visible to any row of this warp, and which only visible ones
      uint32_t none = 0, whole = 0;
#pragma unroll
      for (int c = 0; c < 128; c += 32) {
        if (__all_sync(0xffffffffu, nvalid <= c || (first >= c + 32 && kept <= c))) none |= 1u << (c >> 5);
        if (__all_sync(0xffffffffu, nvalid >= c + 32 && (first <= c || kept >= c + 32))) whole |= 1u << (c >> 5);
      }
#pragma unroll 1
      for (int c = 0; c < 128; c += 32) {
        if (none >> (c >> 5) & 1) continue;
        uint32_t v[32];
        tmem_ld32(sa + c, v);
        tmem_ld_wait();
        if (whole >> (c >> 5) & 1) {
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            mx = fmaxf(mx, __uint_as_float(v[i]));
            big = fmaxf(big, fabsf(__uint_as_float(v[i])));
          }
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            if (visible(c + i)) mx = fmaxf(mx, __uint_as_float(v[i]));
            big = fmaxf(big, fabsf(__uint_as_float(v[i])));
          }
        }
      }
      // the maximum was taken over the raw scores (the cap is increasing); m = -inf: nothing visible so far
      mx = fmaxf(m, mx == -INFINITY ? -INFINITY : p.cap_log2 > 0.f ? capped_log2(p, mx) : mx * p.scale_log2);
      // m = -inf on the first tile: alpha = 0, o and l are 0
      const float alpha = mx == -INFINITY ? 1.f : exp2f(m - mx);
      m = mx;
      // pass 2: P = exp2(s - m) as bf16 into the swizzled K-major tile, row sum
      float sum = 0.f;
      auto weights = [&](auto score) {
#pragma unroll 1
        for (int c = 0; c < 128; c += 32) {
          uint8_t* prow = sP + (c >> 6) * kPfHalf + r * 128;
          const int chunk0 = (c & 63) >> 3;                  // 16-byte chunk of the 128-byte row
          if (none >> (c >> 5) & 1) {
#pragma unroll
            for (int g8 = 0; g8 < 4; ++g8)
              *reinterpret_cast<uint4*>(prow + (((chunk0 + g8) ^ (r & 7)) << 4)) = make_uint4(0, 0, 0, 0);
            continue;
          }
          uint32_t v[32];
          tmem_ld32(sa + c, v);
          tmem_ld_wait();
            auto store = [&](auto seen) {
#pragma unroll
            for (int g8 = 0; g8 < 4; ++g8) {
              uint32_t w[4];
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const int e = g8 * 8 + 2 * i;
                const float p0 = seen(c + e) ? exp2f(score(__uint_as_float(v[e])) - m) : 0.f;
                const float p1 = seen(c + e + 1) ? exp2f(score(__uint_as_float(v[e + 1])) - m) : 0.f;
                const __nv_bfloat162 pb = __floats2bfloat162_rn(p0, p1);
                // the sum uses the rounded values, as the product does
                sum += __low2float(pb) + __high2float(pb);
                w[i] = *reinterpret_cast<const uint32_t*>(&pb);
              }
              *reinterpret_cast<uint4*>(prow + (((chunk0 + g8) ^ (r & 7)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
            }
          };
          if (whole >> (c >> 5) & 1) store([](int) { return true; });
          else store(visible);
        }
      };
      auto plain = [&](float x) { return x * p.scale_log2; };
      if (p.cap_log2 > 0.f) {
        if (__all_sync(0xffffffffu, big * fabsf(p.inv_cap) <= 1.f))
          weights([&](float x) { return capped_log2_small(p, x); });
        else
          weights([&](float x) { return capped_log2(p, x); });
      } else {
        weights(plain);
      }
      l = l * alpha + sum;
      // P is complete: make the generic-proxy stores visible to the tensor core, then tell the MMA warp
      fence_proxy_async();
      tcgen05_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_full);
      // this tile's P V, added to the row's accumulator with the correction for the new maximum
      if (!mbar_wait(&o_full, j & 1, p.status, XFT_ERR_WAIT_TMEM)) { ok = false; break; }
      tcgen05_fence_after();
#pragma unroll
      for (int c = 0; c < 128; c += 32) {
        uint32_t v[32];
        tmem_ld32(lane_addr + 256 + c, v);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 32; ++i) o[c + i] = o[c + i] * alpha + __uint_as_float(v[i]);
      }
      tcgen05_fence_before();
    }
    if (ok && qrow < q_len) {
      const float inv = l > 0.f ? 1.f / l : 0.f;
      __nv_bfloat16* dst = p.out + ((size_t)(q0 + qrow) * p.hq + h) * 128;
#pragma unroll
      for (int c = 0; c < 128; c += 8) {
        uint32_t w[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const __nv_bfloat162 ob = __floats2bfloat162_rn(o[c + 2 * i] * inv, o[c + 2 * i + 1] * inv);
          w[i] = *reinterpret_cast<const uint32_t*>(&ob);
        }
        *reinterpret_cast<uint4*>(dst + c) = make_uint4(w[0], w[1], w[2], w[3]);
      }
    }
  }
  tcgen05_fence_before();
  __syncthreads();
  if (warp == 1) {
    tcgen05_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// Codes of an int8 cache as bf16: block j, head h of sequence b -> copy[(b * w + j) * hkv + h], keys and values.
__global__ void __launch_bounds__(256) expand_codes_kernel(const int8_t* __restrict__ kc, const int8_t* __restrict__ vc,
                                                           __nv_bfloat16* __restrict__ k, __nv_bfloat16* __restrict__ v,
                                                           const int* __restrict__ block_table, int bt_stride,
                                                           const int* __restrict__ kv_lens, int hkv, int num_blocks, int* status) {
  const int j = blockIdx.x, h = blockIdx.y, b = blockIdx.z, w = gridDim.x;
  grid_dep_launch();
  grid_dep_wait();
  if (j * 64 >= kv_lens[b]) return;
  int blk = block_table[(size_t)b * bt_stride + j];
  if (blk < 0 || blk >= num_blocks) { if (threadIdx.x == 0 && status) atomicCAS(status, 0, XFT_ERR_BOUNDS); blk = 0; }
  const size_t from = ((size_t)blk * hkv + h) * 8192, to = ((size_t)(b * w + j) * hkv + h) * 8192;
  uint4 raw[4];
#pragma unroll
  for (int i = 0; i < 4; ++i)                                          // 16 codes each: two of K, two of V
    raw[i] = *reinterpret_cast<const uint4*>((i < 2 ? kc : vc) + from + (threadIdx.x + 256 * (i & 1)) * 16);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int8_t* c = reinterpret_cast<const int8_t*>(&raw[i]);
    uint32_t o[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const __nv_bfloat162 x = __floats2bfloat162_rn((float)c[2 * e], (float)c[2 * e + 1]);
      o[e] = *reinterpret_cast<const uint32_t*>(&x);
    }
    uint4* dst = reinterpret_cast<uint4*>((i < 2 ? k : v) + to + (threadIdx.x + 256 * (i & 1)) * 16);
    dst[0] = make_uint4(o[0], o[1], o[2], o[3]);
    dst[1] = make_uint4(o[4], o[5], o[6], o[7]);
  }
}

template <bool INT8>
static int launch_prefill(const CUtensorMap& tmQ, const CUtensorMap& tmK, const CUtensorMap& tmV, const PrefillAttnParams& p, int B,
                          int max_q, cudaStream_t st) {
  constexpr int SMEM = INT8 ? kPfSmemInt8 : kPfSmem;
  const auto kernel = attn_prefill_tc_kernel<INT8>;
  static bool attr_set = false;
  if (!attr_set) {
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM) != cudaSuccess)
      return 3000 + (int)cudaGetLastError();
    attr_set = true;
  }
  const cudaError_t e = launch_pdl(kernel, dim3(p.hq, B, (max_q + kPfQ - 1) / kPfQ), dim3(kPfThreads), (size_t)SMEM, st, tmQ, tmK, tmV, p);
  return e != cudaSuccess ? (int)e : (int)cudaGetLastError();
}

}  // namespace xft

using namespace xft;

extern "C" int xft_paged_attention_ext(const void* q, void* out, const void* kc, const void* vc, const float* ks, const float* vs,
                                       const int* block_table, int bt_stride, const int* cu_q, const int* kv_lens, int B, int max_q,
                                       int hq, int hkv, int group, int q_off, int HD, int bs, int num_blocks, float scale,
                                       const float* slopes, const int* prefix_lens, int decode, int nsplit, float* part_o,
                                       float* part_ml, int* split_counters, int* status, float softcap, int window, int keep,
                                       const float* sinks, cudaStream_t st);      // attention.cu

// Causal prefill attention over the paged bf16 cache, head_dim 128 (see the file comment).  q, out: [T, hq, 128];
// caches [num_blocks, hkv, bs, 128] with bs = 64; cu_q [B + 1], kv_lens [B] (keys visible after this call's append).
// softcap > 0: scores become softcap * tanh(score / softcap).  window > 0: position i sees the keys j <= i with
// i - j < window or j < keep.  sinks [hq]: exp(sinks[h]) joins the softmax denominator of head h.
// Returns 0, -1 for an unsupported shape, or a CUDA / tensor-map error.
extern "C" int xft_attn_prefill_tc(const void* q, void* out, const void* kc, const void* vc, const int* block_table,
                                   int bt_stride, const int* cu_q, const int* kv_lens, int B, int T, int max_q, int hq,
                                   int hkv, int group, int q_off, int bs, int num_blocks, float scale, float softcap,
                                   int window, int keep, const float* sinks, int* status, cudaStream_t st) {
  if (B <= 0 || T <= 0 || max_q <= 0) return 0;
  if (bs != 64 || hq <= 0 || hkv <= 0 || softcap < 0.f || window < 0 || keep < 0) return -1;
  const bool ext = softcap > 0.f || window > 0 || sinks;
  if (!ext && !(scale > 0.f))                  // attn_prefill_tc_kernel takes the maximum before scores are scaled, and hides keys there
    return xft_paged_attention_ext(q, out, kc, vc, nullptr, nullptr, block_table, bt_stride, cu_q, kv_lens, B, max_q, hq, hkv, group, q_off,
                                   128, bs, num_blocks, scale, nullptr, nullptr, 0, 1, nullptr, nullptr, nullptr, status, 0.f, 0, 0, nullptr,
                                   st);
  PrefillAttnParams p{};
  p.out = (__nv_bfloat16*)out; p.block_table = block_table; p.bt_stride = bt_stride; p.cu_q = cu_q; p.kv_lens = kv_lens;
  p.hq = hq; p.hkv = hkv; p.group = group; p.q_off = q_off; p.bs = bs; p.scale_log2 = scale * 1.4426950408889634f;
  p.num_blocks = num_blocks; p.status = status;
  p.window = window > 0 ? min(window, 1 << 30) : 1 << 30; p.keep = window > 0 ? keep : 0; p.sinks = sinks;
  p.cap_log2 = softcap * 1.4426950408889634f;
  p.inv_cap = softcap > 0.f ? scale / softcap : 0.f;
  CUtensorMap tmQ, tmK, tmV;
  const uint64_t rows = (uint64_t)num_blocks * hkv * bs;
  int r = make_tensor_map(&tmQ, q, (uint64_t)T, (uint64_t)hq * 128, (uint64_t)hq * 128, 128, 2);
  if (r) return 1000 - r;
  if (make_tensor_map(&tmK, kc, rows, 128, 128, 64, 2) || make_tensor_map(&tmV, vc, rows, 128, 128, 64, 2)) return -4;
  if (!ext) return launch_prefill<false>(tmQ, tmK, tmV, p, B, max_q, st);
  static bool attr_set = false;
  if (!attr_set) {
    if (cudaFuncSetAttribute(attn_prefill_ext_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kPfExtSmem) != cudaSuccess)
      return 3000 + (int)cudaGetLastError();
    attr_set = true;
  }
  const cudaError_t e = launch_pdl(attn_prefill_ext_kernel, dim3((max_q + kPfQ - 1) / kPfQ, hq, B), dim3(192), (size_t)kPfExtSmem, st, tmQ,
                                   tmK, tmV, p);
  return e != cudaSuccess ? (int)e : (int)cudaGetLastError();
}

// The same over an int8 cache with one scale per key and head; copy: bf16 [2, B * copy_w, hkv, 64, 128] for the codes, copy_w blocks
// (at least kv_len / 64 of the longest sequence) each.
extern "C" int xft_attn_prefill_tc_int8(const void* q, void* out, const void* kc, const void* vc, const float* ks, const float* vs,
                                        void* copy, int copy_w, const int* block_table, int bt_stride, const int* cu_q,
                                        const int* kv_lens, int B, int T, int max_q, int hq, int hkv, int group, int q_off, int bs,
                                        int num_blocks, float scale, int* status, cudaStream_t st) {
  if (B <= 0 || T <= 0 || max_q <= 0) return 0;
  if (bs != 64 || hq <= 0 || hkv <= 0 || copy_w <= 0 || ((reinterpret_cast<uintptr_t>(ks) | reinterpret_cast<uintptr_t>(vs)) & 15)) return -1;
  if (!(scale > 0.f))
    return xft_paged_attention_ext(q, out, kc, vc, ks, vs, block_table, bt_stride, cu_q, kv_lens, B, max_q, hq, hkv, group, q_off, 128, bs,
                                   num_blocks, scale, nullptr, nullptr, 0, 1, nullptr, nullptr, nullptr, status, 0.f, 0, 0, nullptr, st);
  PrefillAttnParams p{};
  p.out = (__nv_bfloat16*)out; p.block_table = block_table; p.bt_stride = bt_stride; p.cu_q = cu_q; p.kv_lens = kv_lens;
  p.hq = hq; p.hkv = hkv; p.group = group; p.q_off = q_off; p.bs = bs; p.scale_log2 = scale * 1.4426950408889634f;
  p.num_blocks = num_blocks; p.status = status; p.window = 1 << 30; p.ks = ks; p.vs = vs; p.copy_w = copy_w;
  __nv_bfloat16* k = (__nv_bfloat16*)copy;
  const uint64_t rows = (uint64_t)B * copy_w * hkv * bs;
  __nv_bfloat16* v = k + rows * 128;
  CUtensorMap tmQ, tmK, tmV;
  int r = make_tensor_map(&tmQ, q, (uint64_t)T, (uint64_t)hq * 128, (uint64_t)hq * 128, 128, 2);
  if (r) return 1000 - r;
  if (make_tensor_map(&tmK, k, rows, 128, 128, 64, 2) || make_tensor_map(&tmV, v, rows, 128, 128, 64, 2)) return -4;
  const cudaError_t e = launch_pdl(expand_codes_kernel, dim3(copy_w, hkv, B), dim3(256), 0, st, (const int8_t*)kc, (const int8_t*)vc, k, v,
                                   block_table, bt_stride, kv_lens, hkv, num_blocks, status);
  if (e != cudaSuccess) return (int)e;
  return launch_prefill<true>(tmQ, tmK, tmV, p, B, max_q, st);
}
