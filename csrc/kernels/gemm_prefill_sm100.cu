// Persistent prefill GEMM for sm_100a with the tensor-parallel reduction fused in:
//     Y[T, N] = act( sum over ranks ( X_r[T, K_r] · W_r[N, K_r]^T ) + bias ) + res_scale * residual        (bf16 in / out)
//
// The reference runs a row-parallel linear and then a separate collective (o_proj / down_proj followed by
// Messenger::reduceAdd, src/layers/decoder_block.h:122-134; DistLinear in src/layers/dist_linear.h).  At prefill sizes
// that collective moves T x N values per layer twice and leaves the tensor cores idle while it runs.  Here one kernel
// does both, tile by tile:
//
//   * One CTA per SM walks a list of 128-feature x BN-token output tiles.  Warp 0 streams operands with TMA into a
//     shared-memory ring, warp 1 issues tcgen05.mma into one of TWO TMEM accumulators, warps 2-5 drain the other one:
//     the epilogue of tile i (conversion, NVLink stores, waits on peers) overlaps the main loop of tile i + 1.
//   * Token blocks are owned round-robin by the ranks (block j belongs to rank j % world).  A rank that finishes a tile
//     of a block it does not own stores its bf16 partial straight into the owner's memory (reduce-scatter half) and
//     raises a flag there; the owner adds the partials of all ranks to its own fp32 accumulator in rank order, applies
//     bias / activation / residual and stores the finished tile into the output buffer of EVERY rank (all-gather half),
//     again followed by a flag.  The kernel ends on a rank when the finished tiles of all other owners have arrived,
//     so its output is complete in local memory and the next kernel needs no collective.
//   * Each rank visits the blocks it owns a few positions late (the host passes the visiting order), so the partials
//     of its peers are normally there when it gets to them and the waits cost nothing.
//
// Peer memory is touched with plain global stores only (no TMA, no multicast); the operands of the MMA always come
// from this GPU's own memory.  Ordering: data stores, __threadfence_system() by every storing thread, a CTA barrier,
// then one st.release.sys of the flag; the consumer polls with ld.acquire.sys.  Every wait is bounded and reports
// through the status word.  With world == 1 the same kernel is a plain persistent GEMM with a double-buffered
// accumulator.
#include "gemm_common.cuh"

#include <cstdlib>

namespace xft {

int make_tensor_map(CUtensorMap* out, const void* ptr, uint64_t rows, uint64_t cols, uint64_t ld, uint32_t box_rows,
                    uint32_t esize);

struct BulkArParams {
  int world, rank;
  __nv_bfloat16* part[8];     // rank r's partial area as mapped here: [world source slots][part_stride]
  unsigned* flag_part[8];     // rank r's arrival flags: [owned tile][world]
  __nv_bfloat16* out[8];      // rank r's output buffer [T, ldo] (out[rank] is this rank's own)
  unsigned* flag_res[8];      // rank r's result flags: [tile]
  int* epoch;                 // local: completed launches
  int* done;                  // local: CTAs of the current launch that have finished their tiles
  long long part_stride;      // elements per source slot of the partial area
  long long wait_cycles;      // bound of every wait on a peer
};

struct PrefillParams {
  int N, T, K;
  __nv_bfloat16* out;
  int ldo;
  const float* bias;
  const __nv_bfloat16* residual;
  int ldr;
  float res_scale;
  int act;
  int n_tiles, t_tiles, num_kb, stages;
  int gn;                     // feature tiles per group: a group sweeps all token blocks before the next one starts
  int dual_off;               // gated form: W row of the first "up" feature (gate rows are [0, dual_off)); bias likewise
  const int* order;           // optional: i-th visited token block (a permutation of 0..t_tiles-1)
  int wide;                   // != 0: bf16 rows leave through shared memory as 256-byte runs (full 128-feature tiles)
  int* status;
  // token-major kernel only: fp32 rows out, and the grouped form (experts): token tile i is group_tiles[i] = {group, first
  // row, rows, -} of num_group_tiles[0] tiles, and a group's weight rows start at group * group_w_rows
  int out_fp32;
  const int4* group_tiles; const int* num_group_tiles;
  int group_w_rows, group_rows;          // weight rows of a group, token rows of a tile of the table (128 or 256)
  // W8A8: int8 X and W, see xft_w8a8_gemm (all per token or per weight row)
  const float* a_scale; const float* a_zero; const float* a_qsum; const float* w_scale; const float* w_zero; const float* w_sum;
  int dual_rows;                         // weight rows between a gate feature and its up feature (ungated: all)
  // weights of codes in bf16: w_scale and w_zero per weight row, and the rows' sums of X
  const float* x_sum;
  BulkArParams ar;
};

// An activation code with this bit set: the residual operand multiplies the activated value instead of being added to it.
constexpr int kPrefillTimes = 16;
__device__ __forceinline__ float prefill_residual(float x, float r, float scale, int act) {
  return act & kPrefillTimes ? x * r : x + scale * r;
}


__device__ __forceinline__ unsigned ld_acquire_sys(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release_sys(unsigned* p, unsigned v) {
  asm volatile("st.release.sys.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
// Bounded poll of a flag another GPU writes; false on time-out.
__device__ __forceinline__ bool wait_flag(const unsigned* p, unsigned want, long long limit) {
  if (ld_acquire_sys(p) == want) return true;
  const long long t0 = clock64();
  while (ld_acquire_sys(p) != want) {
    if (clock64() - t0 > limit) return false;
  }
  return true;
}

// work item -> (feature tile, visited block index)
__device__ __forceinline__ void decode_item(const PrefillParams& p, int item, int& nt, int& blk) {
  const int per_group = p.gn * p.t_tiles;
  const int g = item / per_group, r = item % per_group;
  const int gn = min(p.gn, p.n_tiles - g * p.gn);
  nt = g * p.gn + r % gn;
  const int bi = r / gn;
  blk = p.order ? p.order[bi] : bi;
}

// mbarrier wait that also gives up as soon as another role of this CTA has raised the abort flag
// (CLUSTER: the phase is completed by another CTA of the cluster too)
template <bool CLUSTER = false>
__device__ __forceinline__ bool mbar_wait_or_abort(uint64_t* bar, uint32_t parity, int* status, int code,
                                                   volatile int* abort_flag) {
  auto done = [&] { return CLUSTER ? mbar_try_wait_cluster(bar, parity) : mbar_try_wait(bar, parity); };
  if (done()) return true;
  const long long t0 = clock64();
  while (!done()) {
    if (*abort_flag) return false;
    if (clock64() - t0 > kWaitCycles) {
      if (status) atomicCAS(status, 0, code);
      *abort_flag = 1;
      return false;
    }
  }
  return true;
}

constexpr int kPrefillMaxStages = 8;

// DUAL: gated form (column-parallel gate ‖ up projection, no reduction over ranks): two weight tiles, gate rows n and up
// rows dual_off + n, share one token tile and feed two accumulators; the epilogue stores act(gate) * up.  With BN = 128
// the four accumulators (2 x double buffer) fill the 512 TMEM columns and a stage moves the same bytes per FLOP as the
// plain 128 x 256 tile.
template <int BN, bool DUAL>
__global__ void __launch_bounds__(192, 1) gemm_prefill_kernel(const __grid_constant__ CUtensorMap tmW,
                                                              const __grid_constant__ CUtensorMap tmX,
                                                              const PrefillParams p) {
  constexpr int A_BYTES = 128 * 64 * 2;
  constexpr int B_BYTES = BN * 64 * 2;
  constexpr int NACC = DUAL ? 2 : 1;
  constexpr int STAGE_BYTES = A_BYTES * NACC + B_BYTES;
  constexpr uint32_t TMEM_COLS = 2 * BN * NACC;          // double-buffered accumulators of BN fp32 columns each
  constexpr uint32_t IDESC = umma_idesc(128, BN, 1, 1, 1);
  static_assert(BN == 128 || (BN == 256 && !DUAL), "token tile of the prefill kernel");

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ uint64_t full_bar[kPrefillMaxStages], empty_bar[kPrefillMaxStages], tmem_full[2], tmem_empty[2];
  __shared__ uint32_t tmem_base_s;
  __shared__ int s_abort_mem, s_epoch, s_last;
  // wide stores: 16 token rows x 128 features of bf16, rows padded by 8 elements so that both the per-feature writes
  // and the 16-byte row reads spread over the banks
  constexpr int kStageLd = 128 + 8;
  __shared__ __align__(16) __nv_bfloat16 s_stage[16 * kStageLd];
  volatile int* s_abort = &s_abort_mem;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int stages = p.stages;
  const int total = p.n_tiles * p.t_tiles;
  const int world = p.ar.world, rank = p.ar.rank;

  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&tmem_full[a], 1);
      mbar_init(&tmem_empty[a], 4);          // one arrival per epilogue warp
    }
    s_abort_mem = 0;
    s_last = 0;
    s_epoch = world > 1 ? *reinterpret_cast<volatile int*>(p.ar.epoch) + 1 : 0;
    fence_barrier_init();
    fence_proxy_async();
    tma_prefetch_desc(&tmW);
    tma_prefetch_desc(&tmX);
  }
  if (warp == 1) {
    tmem_alloc(&tmem_base_s, TMEM_COLS);
    tmem_relinquish();
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem_base = tmem_base_s;
  const unsigned epoch = (unsigned)s_epoch;

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      const uint64_t hint = kEvictNormal;          // both operands are re-read by other CTAs out of L2
      int it = 0;
      bool ok = true;
      for (int item = blockIdx.x; item < total && ok; item += gridDim.x) {
        int nt, blk;
        decode_item(p, item, nt, blk);
        for (int kb = 0; kb < p.num_kb; ++kb, ++it) {
          const int s = it % stages;
          const uint32_t ph = (it / stages) & 1;
          if (*s_abort || !mbar_wait_or_abort(&empty_bar[s], ph ^ 1, p.status, XFT_ERR_WAIT_EMPTY, s_abort)) {
            ok = false;
            break;
          }
          mbar_expect_tx(&full_bar[s], STAGE_BYTES);
          uint8_t* a = smem + s * STAGE_BYTES;
          tma_load_2d(a, &tmW, &full_bar[s], kb * 64, nt * 128, hint);
          if (DUAL) tma_load_2d(a + A_BYTES, &tmW, &full_bar[s], kb * 64, p.dual_off + nt * 128, hint);
          tma_load_2d(a + A_BYTES * NACC, &tmX, &full_bar[s], kb * 64, blk * BN, hint);
        }
      }
      if (!ok) {
        // loads already issued still write into this CTA's shared memory: give them time to land before the CTA exits
        const long long t0 = clock64();
        while (clock64() - t0 < 2000000LL) {}
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (lane == 0) {
      int it = 0, lt = 0;
      bool ok = true;
      for (int item = blockIdx.x; item < total && ok; item += gridDim.x, ++lt) {
        const int a = lt & 1;
        const uint32_t aph = (lt >> 1) & 1;
        if (*s_abort || !mbar_wait_or_abort(&tmem_empty[a], aph ^ 1, p.status, XFT_ERR_WAIT_TMEM, s_abort)) break;
        tcgen05_fence_after();
        const uint32_t acc = tmem_base + (uint32_t)(a * BN * NACC);
        for (int kb = 0; kb < p.num_kb; ++kb, ++it) {
          const int s = it % stages;
          const uint32_t ph = (it / stages) & 1;
          if (!mbar_wait_or_abort(&full_bar[s], ph, p.status, XFT_ERR_WAIT_FULL, s_abort)) {
            ok = false;
            break;
          }
          tcgen05_fence_after();
          const uint32_t a_addr = smem_u32(smem + s * STAGE_BYTES);
          const uint64_t adesc = umma_desc_k128(a_addr);
          const uint64_t bdesc = umma_desc_k128(a_addr + A_BYTES * NACC);
#pragma unroll
          for (int k = 0; k < 4; ++k) {        // 4 x (K = 16) per 64-wide k-block; +32 B = +2 in the address field
            umma_bf16(acc, adesc + 2 * k, bdesc + 2 * k, IDESC, (kb > 0 || k > 0) ? 1u : 0u);
            if (DUAL) {
              const uint64_t a1desc = umma_desc_k128(a_addr + A_BYTES);
              umma_bf16(acc + BN, a1desc + 2 * k, bdesc + 2 * k, IDESC, (kb > 0 || k > 0) ? 1u : 0u);
            }
          }
          tcgen05_commit(&empty_bar[s]);
        }
        if (ok) tcgen05_commit(&tmem_full[a]);
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue (4 warps, one TMEM lane per thread)
    const int q = warp & 3;
    const int row = q * 32 + lane;
    const int et = threadIdx.x - 64;
    int lt = 0;
    for (int item = blockIdx.x; item < total; item += gridDim.x, ++lt) {
      int nt, blk;
      decode_item(p, item, nt, blk);
      const int a = lt & 1;
      const uint32_t aph = (lt >> 1) & 1;
      mbar_wait_or_abort(&tmem_full[a], aph, p.status, XFT_ERR_WAIT_TMEM, s_abort);
      const int owner = world > 1 ? blk % world : 0;
      const bool owned = world <= 1 || owner == rank;
      const int own_idx = world > 1 ? blk / world : 0;          // index of this block among its owner's blocks
      if (world > 1 && owned && et < world && et != rank && !*s_abort) {
        // the partial of rank `et` for this tile must have landed in this rank's memory
        const unsigned* f = p.ar.flag_part[rank] + ((size_t)own_idx * p.n_tiles + nt) * world + et;
        if (!wait_flag(f, epoch, p.ar.wait_cycles)) {
          if (p.status) atomicCAS(p.status, 0, XFT_ERR_WAIT_PEER);
          *s_abort = 1;
        }
      }
      // one answer for all 128 epilogue threads: a flag read per thread could change between two reads (the other
      // roles raise it too) and leave part of the group in front of a barrier the rest never reaches
      if (named_bar_or(1, 128, *s_abort != 0)) break;
      tcgen05_fence_after();
      const uint32_t taddr = tmem_base + (uint32_t(q * 32) << 16) + (uint32_t)(a * BN * NACC);
      const int n = nt * 128 + row;
      const bool n_ok = n < p.N;
      const int t0 = blk * BN;
      const float bias = (p.bias && n_ok) ? p.bias[n] : 0.f;
      const float bias_u = (DUAL && p.bias && n_ok) ? p.bias[p.dual_off + n] : 0.f;
#pragma unroll 1
      for (int c = 0; c < BN; c += 16) {
        uint32_t v[16];
        uint32_t vu[DUAL ? 16 : 1];
        tmem_ld16(taddr + c, v);
        if constexpr (DUAL) tmem_ld16(taddr + BN + c, vu);
        tmem_ld_wait();
        if (c + 16 >= BN) {
          // the accumulator is in registers: hand the TMEM buffer back to the MMA warp before the stores
          tcgen05_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&tmem_empty[a]);
        }
        // full 128-feature tile and the caller asked for it: rows go out as 256-byte runs through shared memory.
        // Uniform over the 128 epilogue threads (it depends on the tile only), so the barriers inside are safe.
        const bool wide = p.wide && (nt * 128 + 128 <= p.N) && (p.N % 8 == 0) && (p.ldo % 8 == 0);
        if (!owned && wide) {
#pragma unroll
          for (int j = 0; j < 16; ++j) s_stage[j * kStageLd + row] = __float2bfloat16(__uint_as_float(v[j]));
          named_bar_sync(1, 128);
          __nv_bfloat16* base = p.ar.part[owner] + (size_t)rank * p.ar.part_stride +
                                ((size_t)own_idx * BN + c) * p.N + nt * 128;
#pragma unroll
          for (int it = 0; it < 2; ++it) {
            const int j = (et >> 4) + 8 * it, seg = et & 15;          // 16 threads write one 256-byte row
            if (t0 + c + j < p.T)
              *reinterpret_cast<uint4*>(base + (size_t)j * p.N + seg * 8) =
                  *reinterpret_cast<const uint4*>(&s_stage[j * kStageLd + seg * 8]);
          }
          named_bar_sync(1, 128);                                      // the buffer is reused by the next chunk
          continue;
        }
        if (!n_ok) continue;
        if (!owned) {
          __nv_bfloat16* dst = p.ar.part[owner] + (size_t)rank * p.ar.part_stride +
                               ((size_t)own_idx * BN + c) * p.N + n;
#pragma unroll
          for (int j = 0; j < 16; ++j)
            if (t0 + c + j < p.T) dst[(size_t)j * p.N] = __float2bfloat16(__uint_as_float(v[j]));
          continue;
        }
        float x[16];
        if (world > 1) {
          // sum in rank order; this rank's own term is its fp32 accumulator, the others arrive rounded to bf16
#pragma unroll
          for (int j = 0; j < 16; ++j) x[j] = 0.f;
          for (int r = 0; r < world; ++r) {
            if (r == rank) {
#pragma unroll
              for (int j = 0; j < 16; ++j) x[j] += __uint_as_float(v[j]);
            } else {
              const __nv_bfloat16* src = p.ar.part[rank] + (size_t)r * p.ar.part_stride +
                                         ((size_t)own_idx * BN + c) * p.N + n;
#pragma unroll
              for (int j = 0; j < 16; ++j)
                if (t0 + c + j < p.T) x[j] += __bfloat162float(__ldcg(src + (size_t)j * p.N));
            }
          }
        } else {
#pragma unroll
          for (int j = 0; j < 16; ++j) x[j] = __uint_as_float(v[j]);
        }
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const int t = t0 + c + j;
          if (t < p.T) {
            float y = x[j] + bias;
            if constexpr (DUAL) y = apply_gated(y, __uint_as_float(vu[j]) + bias_u, p.act, p.res_scale);
            else y = apply_act(y, p.act, p.res_scale);
            if (p.residual) y = prefill_residual(y, __bfloat162float(p.residual[(size_t)t * p.ldr + n]), p.res_scale, p.act);
            const __nv_bfloat16 yb = __float2bfloat16(y);
            if (wide) {
              s_stage[j * kStageLd + row] = yb;
            } else if (world > 1) {
              for (int r = 0; r < world; ++r) p.ar.out[r][(size_t)t * p.ldo + n] = yb;
            } else {
              p.out[(size_t)t * p.ldo + n] = yb;
            }
          }
        }
        if (wide) {
          named_bar_sync(1, 128);
#pragma unroll
          for (int it = 0; it < 2; ++it) {
            const int j = (et >> 4) + 8 * it, seg = et & 15;
            const int t = t0 + c + j;
            if (t < p.T) {
              const uint4 val = *reinterpret_cast<const uint4*>(&s_stage[j * kStageLd + seg * 8]);
              const size_t off = (size_t)t * p.ldo + nt * 128 + seg * 8;
              if (world > 1) {
                for (int r = 0; r < world; ++r) *reinterpret_cast<uint4*>(p.ar.out[r] + off) = val;
              } else {
                *reinterpret_cast<uint4*>(p.out + off) = val;
              }
            }
          }
          named_bar_sync(1, 128);
        }
      }
      if (world > 1) {
        __threadfence_system();               // this thread's stores to peer memory, before the flag below
        named_bar_sync(1, 128);
        if (!owned) {
          if (et == 0)
            st_release_sys(p.ar.flag_part[owner] + ((size_t)own_idx * p.n_tiles + nt) * world + rank, epoch);
        } else if (et < world && et != rank) {
          st_release_sys(p.ar.flag_res[et] + (size_t)blk * p.n_tiles + nt, epoch);
        }
      }
    }
    if (world > 1) {
      // The launch is complete on this rank when the finished tiles of every other owner are here.  The CTA that
      // finishes last checks them all, then opens the next epoch.
      named_bar_sync(1, 128);
      if (et == 0) {
        __threadfence();
        s_last = (atomicAdd(p.ar.done, 1) == (int)gridDim.x - 1);
      }
      named_bar_sync(1, 128);
      if (s_last) {
        bool ok = !*s_abort;
        for (int idx = et; idx < total && ok; idx += 128) {
          const int blk = idx / p.n_tiles;
          if (blk % world == rank) continue;
          if (!wait_flag(p.ar.flag_res[rank] + idx, epoch, p.ar.wait_cycles)) {
            if (p.status) atomicCAS(p.status, 0, XFT_ERR_WAIT_PEER);
            ok = false;
          }
        }
        named_bar_sync(1, 128);
        if (et == 0) {
          *reinterpret_cast<volatile int*>(p.ar.done) = 0;
          __threadfence();
          atomicAdd(p.ar.epoch, 1);
        }
      }
    }
  }
  tcgen05_fence_before();
  __syncthreads();
  if (warp == 1) {
    tcgen05_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

// ------------------------------------------------------------------------------------------------------------------
// Token-major form (one GPU, or the local product in front of a library collective).  Same pipeline, but the operands
// trade places: the rows of the MMA are TOKENS (A = the activation tile) and its columns are output features
// (B = the weight tile), so the accumulator is [token lane][feature column] — the layout of Y itself.  Each epilogue
// thread owns one token row and handles 32 consecutive features per step: bias and residual arrive as 16-byte vectors
// and the result leaves as 16-byte stores, instead of one 2-byte store per element in the feature-major form, whose
// epilogue (a dependent chain per element on four warps) took ten times longer than the main loop of the short-K
// row-parallel products.  Gated form: gate and up accumulators side by side, act(gate) * up on the way out.
//
// CG = 2: the two CTAs of a cluster work on one tile of 256 tokens with `cta_group::2` MMAs issued by the first of them.
// Each CTA keeps its 128 tokens (A, and their accumulator rows in its own TMEM) and HALF of the tile's weight rows, which
// the tensor cores of both read: per MMA an SM then takes 128 + NCOL / 2 rows from shared memory instead of 128 + NCOL,
// and as many fewer arrive by TMA.  With 128 x 256 tiles of single CTAs those reads and writes together (192 bytes per
// cycle) were more than shared memory delivers.  In the gated form the first CTA holds the gate rows and the second the
// up rows.  Both producers signal the first CTA's full barrier; a commit frees the stage in both.
//
// NCOL: accumulator columns of a tile (gated: half of them gate, half up).
// SRC: bf16 operands; int8 operands of W8A8; bf16 activations and int8 codes (exact in bf16, see xft_gemm_codes_tm), whose
// scale and zero point per weight row come in with the epilogue.
enum { kTmBf16 = 0, kTmI8 = 1, kTmCodes = 2 };
constexpr int kPrefillTmThreads = 320;      // producer, MMA, two epilogue warps per quarter of the accumulator's rows
__host__ __device__ constexpr int prefill_tm_stages(int stage_bytes) { return 196 * 1024 / stage_bytes < kPrefillMaxStages ? 196 * 1024 / stage_bytes : kPrefillMaxStages; }

template <int NCOL, bool DUAL, int CG, int SRC = kTmBf16>
__global__ void __launch_bounds__(kPrefillTmThreads, 1) gemm_prefill_tm_kernel(const __grid_constant__ CUtensorMap tmX,
                                                                 const __grid_constant__ CUtensorMap tmW,
                                                                 const PrefillParams p) {
  constexpr int FEAT = DUAL ? NCOL / 2 : NCOL;           // features of an output tile
  constexpr int TOK = 128 * CG;                          // tokens of an output tile
  constexpr int A_BYTES = 128 * 64 * 2;                  // this CTA's 128 tokens x 64 k
  constexpr int B_BYTES = NCOL / CG * 64 * 2;            // this CTA's weight rows x 64 k
  constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  constexpr int STAGES = prefill_tm_stages(STAGE_BYTES);
  constexpr uint32_t TMEM_COLS = 2 * NCOL;               // double-buffered accumulators
  constexpr bool I8 = SRC == kTmI8, CODES = SRC == kTmCodes;
  constexpr int KEL = I8 ? 128 : 64;                     // k of a step: 128 bytes of a row
  constexpr uint32_t IDESC = umma_idesc(TOK, NCOL, 1, 1, I8 ? 2 : 1);
  constexpr int CW = DUAL || SRC != kTmBf16 ? 16 : 32;               // columns of an epilogue step: registers for what it holds at once
  static_assert((NCOL == 256 || NCOL == 128) && (CG == 1 || CG == 2), "tile of the token-major kernel");

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ uint64_t full_bar[STAGES], empty_bar[STAGES], tmem_full[2], tmem_empty[2];
  __shared__ uint32_t tmem_base_s;
  __shared__ int s_abort_mem;
  volatile int* s_abort = &s_abort_mem;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int half = CG == 2 ? (int)cluster_ctarank() : 0;      // which 128 tokens of a tile are this CTA's
  const int first = blockIdx.x / CG, step = gridDim.x / CG;
  // n_tiles: feature tiles of FEAT, t_tiles: token blocks of TOK (grouped: at most so many)
  const int total = p.n_tiles * (p.group_tiles ? min(*p.num_group_tiles, p.t_tiles) : p.t_tiles);
  // an item's feature tile, first token row, number of rows and first weight row of its group
  struct Item { int nt, row0, rows, w0; };
  auto item_of = [&](int item) {
    Item r;
    if (p.group_tiles) {
      const int4 e = p.group_tiles[item / p.n_tiles];
      r = {item % p.n_tiles, e.y, e.z, e.x * p.group_w_rows};
    } else {
      int blk;
      decode_item(p, item, r.nt, blk);
      r.row0 = blk * TOK;
      r.rows = p.T - r.row0;
      r.w0 = 0;
    }
    r.row0 += half * 128;
    r.rows -= half * 128;
    return r;
  };

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&tmem_full[a], 1);
      mbar_init(&tmem_empty[a], 8 * CG);
    }
    s_abort_mem = 0;
    fence_barrier_init();
    fence_proxy_async();
    tma_prefetch_desc(&tmW);
    tma_prefetch_desc(&tmX);
  }
  if (warp == 1) {
    if constexpr (CG == 2) {
      tmem_alloc_pair(&tmem_base_s, TMEM_COLS);
      tmem_relinquish_pair();
    } else {
      tmem_alloc(&tmem_base_s, TMEM_COLS);
      tmem_relinquish();
    }
  }
  tcgen05_fence_before();
  __syncthreads();
  if constexpr (CG == 2) {              // both CTAs' barriers and accumulators exist before either touches the other's
    cluster_arrive();
    cluster_wait();
  }
  tcgen05_fence_after();
  const uint32_t tmem_base = tmem_base_s;

  // The two issuing threads are the kernel's critical path when a step's MMAs are short, so their loops carry stage, phase
  // and descriptors along instead of dividing, and look at the abort flag only when a wait does not succeed at once.
  if (warp == 0) {
    if (elect_one()) {
      const uint64_t hint = kEvictNormal;
      const uint32_t lead_bar = CG == 2 ? dsmem_addr(smem_u32(full_bar), 0) : 0;      // the first CTA's full barriers
      int s = 0;
      uint32_t ph = 0;
      bool ok = true;
      auto step_stage = [&] { if (++s == STAGES) { s = 0; ph ^= 1; } };
      for (int item = first; item < total && ok; item += step) {
        const Item im = item_of(item);
        const int wrow = im.w0 + im.nt * FEAT + half * (DUAL ? p.dual_off : NCOL / 2);
        for (int kb = 0; kb < p.num_kb; ++kb, step_stage()) {
          if (!mbar_wait_or_abort<CG == 2>(&empty_bar[s], ph ^ 1, p.status, XFT_ERR_WAIT_EMPTY, s_abort)) {
            ok = false;
            break;
          }
          uint8_t* a = smem + s * STAGE_BYTES;
          if constexpr (CG == 2) {
            if (half == 0) mbar_expect_tx(&full_bar[s], 2 * STAGE_BYTES);
            tma_load_2d_pair(a, &tmX, lead_bar + 8 * s, kb * KEL, im.row0, hint);
            tma_load_2d_pair(a + A_BYTES, &tmW, lead_bar + 8 * s, kb * KEL, wrow, hint);
          } else {
            mbar_expect_tx(&full_bar[s], STAGE_BYTES);
            tma_load_2d(a, &tmX, &full_bar[s], kb * KEL, im.row0, hint);
            tma_load_2d(a + A_BYTES, &tmW, &full_bar[s], kb * KEL, wrow, hint);
            if (DUAL) tma_load_2d(a + A_BYTES + FEAT * 128, &tmW, &full_bar[s], kb * KEL, wrow + p.dual_off, hint);
          }
        }
      }
      if (!ok) {
        const long long t0 = clock64();
        while (clock64() - t0 < 2000000LL) {}
      } else if (CG == 2) {
        // the first CTA's commits also arrive here: stay until every stage has been given back
        for (int k = 0; k < STAGES; ++k, step_stage())
          if (!mbar_wait_or_abort<true>(&empty_bar[s], ph ^ 1, p.status, XFT_ERR_WAIT_EMPTY, s_abort)) break;
      }
    }
  } else if (warp == 1) {
    if (half == 0 && elect_one()) {
      const uint64_t adesc0 = umma_desc_k128(smem_u32(smem));                      // tokens
      const uint64_t bdesc0 = umma_desc_k128(smem_u32(smem) + A_BYTES);            // features (gated: gate rows, then up rows)
      int s = 0, lt = 0;
      uint32_t ph = 0;
      bool ok = true;
      for (int item = first; item < total && ok; item += step, ++lt) {
        const int a = lt & 1;
        const uint32_t aph = (lt >> 1) & 1;
        if (!mbar_wait_or_abort<CG == 2>(&tmem_empty[a], aph ^ 1, p.status, XFT_ERR_WAIT_TMEM, s_abort)) break;
        tcgen05_fence_after();
        const uint32_t acc = tmem_base + (uint32_t)(a * NCOL);
        for (int kb = 0; kb < p.num_kb; ++kb) {
          if (!mbar_wait_or_abort<CG == 2>(&full_bar[s], ph, p.status, XFT_ERR_WAIT_FULL, s_abort)) {
            ok = false;
            break;
          }
          tcgen05_fence_after();
          const uint64_t off = (uint64_t)(s * (STAGE_BYTES / 16));
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const uint32_t acc_on = (kb > 0 || k > 0) ? 1u : 0u;
            if constexpr (CG == 2 && I8) umma_i8_pair(acc, adesc0 + off + 2 * k, bdesc0 + off + 2 * k, IDESC, acc_on);
            else if constexpr (CG == 2) umma_bf16_pair(acc, adesc0 + off + 2 * k, bdesc0 + off + 2 * k, IDESC, acc_on);
            else umma_bf16(acc, adesc0 + off + 2 * k, bdesc0 + off + 2 * k, IDESC, acc_on);
          }
          if constexpr (CG == 2) tcgen05_commit_pair(&empty_bar[s]);
          else tcgen05_commit(&empty_bar[s]);
          if (++s == STAGES) { s = 0; ph ^= 1; }
        }
        if (ok) {
          if constexpr (CG == 2) tcgen05_commit_pair(&tmem_full[a]);
          else tcgen05_commit(&tmem_full[a]);
        }
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue: one token row and half the features per thread
    const int q = warp & 3;
    const int c_begin = warp < 6 ? 0 : FEAT / 2, c_end = c_begin + FEAT / 2;
    const int row = q * 32 + lane;
    // 16-byte pieces where every row of output and residual starts on one (a residual may be a slice of a wider tensor)
    const bool vec = (p.N % 8 == 0) && (p.ldo % 8 == 0) && (!p.residual || p.ldr % 8 == 0) &&
                     ((reinterpret_cast<uintptr_t>(p.out) | reinterpret_cast<uintptr_t>(p.residual)) & 15) == 0;
    // 32-byte rows' pieces: every store fills a whole sector
    const bool vec32 = vec && p.ldo % 16 == 0 && (reinterpret_cast<uintptr_t>(p.out) & 31) == 0;
    const bool bias16 = (reinterpret_cast<uintptr_t>(p.bias) & 15) == 0;
    int lt = 0;
    for (int item = first; item < total; item += step, ++lt) {
      const Item im = item_of(item);
      const int a = lt & 1;
      const uint32_t aph = (lt >> 1) & 1;
      mbar_wait_or_abort(&tmem_full[a], aph, p.status, XFT_ERR_WAIT_TMEM, s_abort);
      if (named_bar_or(1, 256, *s_abort != 0)) break;
      tcgen05_fence_after();
      const uint32_t taddr = tmem_base + (uint32_t(q * 32) << 16) + (uint32_t)(a * NCOL);
      const int t = im.row0 + row;
      const bool t_ok = row < im.rows;
      __nv_bfloat16* orow = p.out + (size_t)t * p.ldo;
      const __nv_bfloat16* rrow = p.residual ? p.residual + (size_t)t * p.ldr : nullptr;
      auto load_cols = [&](uint32_t at, uint32_t* to) {
        if constexpr (CW == 16) tmem_ld16(at, *reinterpret_cast<uint32_t (*)[16]>(to));
        else tmem_ld32(at, *reinterpret_cast<uint32_t (*)[32]>(to));
      };
      // W8A8: integer sums of 16 features from weight row nn on -> values
      float sa = 0.f, za = 0.f, qs = 0.f;
      if constexpr (I8) {
        if (t_ok) { sa = __ldg(p.a_scale + t); za = __ldg(p.a_zero + t); qs = __ldg(p.a_qsum + t); }
      }
      float xs = 0.f;
      if constexpr (CODES) {
        if (t_ok && p.w_zero) xs = __ldg(p.x_sum + t);
      }
      auto dequant = [&](const uint32_t* acc, int nn, bool whole, float* to) {
        if constexpr (CODES) {
#pragma unroll
          for (int j = 0; j < CW; ++j) {
            const int m = whole || nn % p.dual_rows + j < p.N ? nn + j : nn;
            // the roundings of qgemm_kernel (quant_gemm_sm100.cu), spelled out
            const float y = __fmul_rn(__uint_as_float(acc[j]), __ldg(p.w_scale + m));
            to[j] = __fadd_rn(p.w_zero ? __fmaf_rn(__ldg(p.w_zero + m), xs, y) : y, p.bias ? __ldg(p.bias + m) : 0.f);
          }
          return;
        }
#pragma unroll
        for (int j = 0; j < CW; ++j) {
          const int m = whole || nn % p.dual_rows + j < p.N ? nn + j : nn;
          const float y = w8a8_value((float)(int)acc[j], sa, za, qs, __ldg(p.w_scale + m), p.w_zero ? __ldg(p.w_zero + m) : 0.f,
                                     p.w_sum ? __ldg(p.w_sum + m) : 0.f, p.K, p.bias ? __ldg(p.bias + m) : 0.f);
          to[j] = DUAL ? bf16_round(y) : y;
        }
      };
#pragma unroll 1
      for (int c = c_begin; c < c_end; c += CW) {
        const int n0 = im.nt * FEAT + c;
        const bool full = vec && n0 + CW <= p.N;
        uint32_t v[CW];
        uint32_t vu[DUAL ? CW : 1];
        load_cols(taddr + c, v);
        if constexpr (DUAL) load_cols(taddr + FEAT + c, vu);
        uint4 res[CW / 8];
        const bool take = rrow && full && t_ok;
        if (take) {
#pragma unroll
          for (int j = 0; j < CW / 8; ++j) res[j] = *reinterpret_cast<const uint4*>(rrow + n0 + 8 * j);
        }
        tmem_ld_wait();
        if (c + CW >= c_end) {
          tcgen05_fence_before();
          __syncwarp();
          if (lane == 0) {
            if constexpr (CG == 2) mbar_arrive_cluster(dsmem_addr(smem_u32(&tmem_empty[a]), 0));
            else mbar_arrive(&tmem_empty[a]);
          }
        }
        if (!t_ok || n0 >= p.N) continue;
        float x[CW];
        if constexpr (I8 || CODES) {
          dequant(v, n0, full, x);
        } else {
#pragma unroll
          for (int j = 0; j < CW; ++j) x[j] = __uint_as_float(v[j]);
        }
        if (I8 || CODES) {                         // the bias is in already
        } else if (p.bias && full && bias16) {
#pragma unroll
          for (int j = 0; j < CW / 4; ++j) {
            const float4 w = __ldg(reinterpret_cast<const float4*>(p.bias + n0) + j);
            x[4 * j] += w.x; x[4 * j + 1] += w.y; x[4 * j + 2] += w.z; x[4 * j + 3] += w.w;
          }
        } else if (p.bias) {
#pragma unroll
          for (int j = 0; j < CW; ++j) if (full || n0 + j < p.N) x[j] += __ldg(p.bias + n0 + j);
        }
        // one branch for the whole row: a branch per element cost more than the arithmetic
        switch (p.act & (kPrefillTimes - 1)) {
          case 1:
#pragma unroll
            for (int j = 0; j < CW; ++j) x[j] = apply_act(x[j], 1);
            break;
          case 2:
#pragma unroll
            for (int j = 0; j < CW; ++j) x[j] = apply_act(x[j], 2);
            break;
          case 3:
#pragma unroll
            for (int j = 0; j < CW; ++j) x[j] = apply_act(x[j], 3);
            break;
          case 4:
#pragma unroll
            for (int j = 0; j < CW; ++j) x[j] = apply_act(x[j], 4);
            break;
          case kActGeluErf:
#pragma unroll
            for (int j = 0; j < CW; ++j) x[j] = gelu_erf(x[j]);
            break;
          case kActTanh:
          case kActSoftcap:
#pragma unroll
            for (int j = 0; j < CW; ++j) x[j] = apply_act(x[j], p.act, p.res_scale);
            break;
          default: break;
        }
        if constexpr (DUAL) {
          float up[CW];
          if constexpr (I8 || CODES) {
            dequant(vu, p.dual_off + n0, full, up);
          } else {
#pragma unroll
            for (int j = 0; j < CW; ++j) up[j] = __uint_as_float(vu[j]);
          }
#pragma unroll
          for (int j = 0; j < CW; ++j) {
            float u = up[j];
            if (!I8 && !CODES && p.bias && (full || n0 + j < p.N)) u += __ldg(p.bias + p.dual_off + n0 + j);
            x[j] = p.act == kActClamped ? clamped_glu(x[j], u, p.res_scale) : x[j] * u;
          }
        }
        if (take) {
          const __nv_bfloat162* r2 = reinterpret_cast<const __nv_bfloat162*>(res);
          if (p.act & kPrefillTimes) {
#pragma unroll
            for (int j = 0; j < CW / 2; ++j) {
              const float2 f = __bfloat1622float2(r2[j]);
              x[2 * j] *= f.x; x[2 * j + 1] *= f.y;
            }
          } else {
#pragma unroll
            for (int j = 0; j < CW / 2; ++j) {
              const float2 f = __bfloat1622float2(r2[j]);
              x[2 * j] += p.res_scale * f.x; x[2 * j + 1] += p.res_scale * f.y;
            }
          }
        } else if (rrow) {
#pragma unroll
          for (int j = 0; j < CW; ++j)
            if (n0 + j < p.N) x[j] = prefill_residual(x[j], __bfloat162float(rrow[n0 + j]), p.res_scale, p.act);
        }
        if (p.out_fp32) {
          float* frow = reinterpret_cast<float*>(p.out) + (size_t)t * p.ldo + n0;
          if (full) {
#pragma unroll
            for (int j = 0; j < CW / 4; ++j)
              reinterpret_cast<float4*>(frow)[j] = make_float4(x[4 * j], x[4 * j + 1], x[4 * j + 2], x[4 * j + 3]);
          } else {
#pragma unroll
            for (int j = 0; j < CW; ++j) if (n0 + j < p.N) frow[j] = x[j];
          }
        } else if (full) {
          uint32_t w[CW / 2];
#pragma unroll
          for (int j = 0; j < CW / 2; ++j) {
            const __nv_bfloat162 b = __floats2bfloat162_rn(x[2 * j], x[2 * j + 1]);
            w[j] = *reinterpret_cast<const uint32_t*>(&b);
          }
          if (vec32) {
#pragma unroll
            for (int i = 0; i < CW / 16; ++i) st_global_256(orow + n0 + 16 * i, w + 8 * i);
          } else {
#pragma unroll
            for (int i = 0; i < CW / 8; ++i)
              *reinterpret_cast<uint4*>(orow + n0 + 8 * i) = make_uint4(w[4 * i], w[4 * i + 1], w[4 * i + 2], w[4 * i + 3]);
          }
        } else {
#pragma unroll
          for (int j = 0; j < CW; ++j) {
            if (n0 + j < p.N) orow[n0 + j] = __float2bfloat16(x[j]);
          }
        }
      }
    }
  }
  __syncwarp();
  tcgen05_fence_before();
  __syncthreads();
  if constexpr (CG == 2) {              // neither CTA's shared memory or accumulator goes while the other may still use it
    cluster_arrive();
    cluster_wait();
  }
  if (warp == 1) {
    tcgen05_fence_after();
    if constexpr (CG == 2) tmem_dealloc_pair(tmem_base, TMEM_COLS);
    else tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

template <int NCOL, bool DUAL, int CG, int SRC = kTmBf16>
static int launch_prefill_tm(const void* X, int ldx, const void* W, int w_rows, int ldw, PrefillParams& p, int num_ctas,
                             cudaStream_t st) {
  constexpr bool I8 = SRC == kTmI8;
  constexpr int STAGE_BYTES = 128 * 64 * 2 + NCOL / CG * 64 * 2;
  constexpr int FEAT = DUAL ? NCOL / 2 : NCOL;
  p.n_tiles = (p.N + FEAT - 1) / FEAT;
  if (!p.group_tiles) p.t_tiles = (p.T + 128 * CG - 1) / (128 * CG);
  CUtensorMap tmW, tmX;
  int r = make_tensor_map(&tmW, W, (uint64_t)w_rows, (uint64_t)p.K, (uint64_t)ldw, (uint32_t)(DUAL ? FEAT : NCOL / CG), I8 ? 1 : 2);
  if (r) return 1000 - r;
  r = make_tensor_map(&tmX, X, (uint64_t)p.T, (uint64_t)p.K, (uint64_t)ldx, 128, I8 ? 1 : 2);
  if (r) return 2000 - r;
  const size_t smem = (size_t)prefill_tm_stages(STAGE_BYTES) * STAGE_BYTES + 1024;
  static bool attr_set = false;
  if (!attr_set) {
    if (cudaFuncSetAttribute(gemm_prefill_tm_kernel<NCOL, DUAL, CG, SRC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
        cudaSuccess)
      return 3000 + (int)cudaGetLastError();
    attr_set = true;
  }
  const int total = p.n_tiles * p.t_tiles, slots = num_ctas / CG > 0 ? num_ctas / CG : 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((total < slots ? total : slots) * CG);
  cfg.blockDim = dim3(kPrefillTmThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = CG;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = CG > 1 ? 1 : 0;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, gemm_prefill_tm_kernel<NCOL, DUAL, CG, SRC>, tmX, tmW, (const PrefillParams)p);
  return e != cudaSuccess ? (int)e : (int)cudaGetLastError();
}

template <int BN, bool DUAL>
static int launch_prefill(const CUtensorMap& tmW, const CUtensorMap& tmX, PrefillParams& p, int num_ctas,
                          cudaStream_t st) {
  constexpr int STAGE_BYTES = 128 * 64 * 2 * (DUAL ? 2 : 1) + BN * 64 * 2;
  int stages = (220 * 1024) / STAGE_BYTES;
  if (stages > kPrefillMaxStages) stages = kPrefillMaxStages;
  p.stages = stages;
  const size_t smem = (size_t)stages * STAGE_BYTES + 1024;
  static bool attr_set = false;
  if (!attr_set) {
    // the request is the ring itself: the kernel's static shared memory (barriers, the 4 KB store staging tile)
    // counts against the same 227 KB, so asking for more than the ring needs can be refused
    if (cudaFuncSetAttribute(gemm_prefill_kernel<BN, DUAL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
        cudaSuccess)
      return 3000 + (int)cudaGetLastError();
    attr_set = true;
  }
  const int total = p.n_tiles * p.t_tiles;
  const int grid = total < num_ctas ? total : num_ctas;
  gemm_prefill_kernel<BN, DUAL><<<grid, 192, smem, st>>>(tmW, tmX, p);
  return (int)cudaGetLastError();
}

}  // namespace xft

using namespace xft;

// Elements of one source slot of the partial area and the flag counts a launch of (T, N) needs at `world` ranks.
extern "C" void xft_prefill_ar_sizes(int T, int N, int world, long long* part_elems_per_slot, long long* n_flag_part,
                                     long long* n_flag_res) {
  const int bn = T > 128 ? 256 : 128;
  const long long t_tiles = (T + bn - 1) / bn, n_tiles = (N + 127) / 128;
  const long long own = (t_tiles + world - 1) / world;
  *part_elems_per_slot = own * bn * (long long)N;
  *n_flag_part = own * n_tiles * world;
  *n_flag_res = t_tiles * n_tiles;
}

// Y = act(X W^T (+ the same product of every other rank) + bias) + res_scale * residual, bf16.  ar == nullptr or
// ar->world <= 1: plain persistent GEMM.  order: optional device array, the order in which token blocks are visited
// (with ar it must hold the same multiset on every rank, see the file comment).  Returns 0, a negative argument
// error, or a CUDA error code.
extern "C" int xft_gemm_bf16_prefill(const void* X, int ldx, const void* W, int w_rows, int ldw, void* Y, int ldo, int T,
                                     int N, int K, const float* bias, const void* residual, int ldr, float res_scale,
                                     int act, const int* order, int* status, const BulkArParams* ar, int num_ctas,
                                     cudaStream_t st) {
  if (T <= 0 || N <= 0 || K <= 0) return 0;
  if ((K & 7) || (ldx & 7) || (ldw & 7)) return -2;
  PrefillParams p{};
  p.N = N; p.T = T; p.K = K; p.out = reinterpret_cast<__nv_bfloat16*>(Y); p.ldo = ldo; p.bias = bias;
  p.residual = reinterpret_cast<const __nv_bfloat16*>(residual); p.ldr = ldr; p.res_scale = res_scale; p.act = act;
  p.order = order; p.status = status;
  static const int wide_env = [] { const char* v = getenv("XFT_PREFILL_WIDE_STORES"); return v && v[0] == '1' ? 1 : 0; }();
  p.wide = wide_env;
  const int bn = T > 128 ? 256 : 128;
  p.n_tiles = (N + 127) / 128;
  p.t_tiles = (T + bn - 1) / bn;
  p.num_kb = (K + 63) / 64;
  p.gn = 16;
  if (ar && ar->world > 1) {
    if (ar->world > 8 || ar->rank < 0 || ar->rank >= ar->world) return -3;
    long long need_part, nfp, nfr;
    xft_prefill_ar_sizes(T, N, ar->world, &need_part, &nfp, &nfr);
    if (ar->part_stride < need_part) return -4;
    if (ar->out[ar->rank] != p.out) return -5;
    p.ar = *ar;
    p.gn = p.n_tiles;                 // block-major: all feature tiles of a token block are visited together
  }
  if (num_ctas <= 0) {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    num_ctas = sms > 0 ? sms : 148;
  }
  CUtensorMap tmW, tmX;
  int r = make_tensor_map(&tmW, W, (uint64_t)w_rows, (uint64_t)K, (uint64_t)ldw, 128, 2);
  if (r) return 1000 - r;
  r = make_tensor_map(&tmX, X, (uint64_t)T, (uint64_t)K, (uint64_t)ldx, (uint32_t)bn, 2);
  if (r) return 2000 - r;
  return bn == 256 ? launch_prefill<256, false>(tmW, tmX, p, num_ctas, st)
                   : launch_prefill<128, false>(tmW, tmX, p, num_ctas, st);
}

// Gated form: Y[T, N] = act(X Wg^T + bias_g) * (X Wu^T + bias_u), W holds gate rows [0, N) and up rows
// [dual_off, dual_off + N) (bias likewise).  Token tiles of 128.
extern "C" int xft_gemm_bf16_prefill_gated(const void* X, int ldx, const void* W, int w_rows, int ldw, void* Y, int ldo,
                                           int T, int N, int K, int dual_off, const float* bias, int act, int* status,
                                           int num_ctas, cudaStream_t st) {
  if (T <= 0 || N <= 0 || K <= 0) return 0;
  if ((K & 7) || (ldx & 7) || (ldw & 7)) return -2;
  PrefillParams p{};
  p.N = N; p.T = T; p.K = K; p.out = reinterpret_cast<__nv_bfloat16*>(Y); p.ldo = ldo; p.bias = bias; p.act = act;
  p.status = status; p.dual_off = dual_off;
  static const int wide_env = [] { const char* v = getenv("XFT_PREFILL_WIDE_STORES"); return v && v[0] == '1' ? 1 : 0; }();
  p.wide = wide_env;
  p.n_tiles = (N + 127) / 128;
  p.t_tiles = (T + 127) / 128;
  p.num_kb = (K + 63) / 64;
  p.gn = 16;
  if (num_ctas <= 0) {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    num_ctas = sms > 0 ? sms : 148;
  }
  CUtensorMap tmW, tmX;
  int r = make_tensor_map(&tmW, W, (uint64_t)w_rows, (uint64_t)K, (uint64_t)ldw, 128, 2);
  if (r) return 1000 - r;
  r = make_tensor_map(&tmX, X, (uint64_t)T, (uint64_t)K, (uint64_t)ldx, 128, 2);
  if (r) return 2000 - r;
  return launch_prefill<128, true>(tmW, tmX, p, num_ctas, st);
}

// Size and field offsets of BulkArParams, for the layout check of the Python mirror.
extern "C" int xft_bulk_ar_layout(long long* out, int n) {
  const long long v[] = {sizeof(BulkArParams),           offsetof(BulkArParams, world),       offsetof(BulkArParams, rank),
                         offsetof(BulkArParams, part),   offsetof(BulkArParams, flag_part),   offsetof(BulkArParams, out),
                         offsetof(BulkArParams, flag_res), offsetof(BulkArParams, epoch),     offsetof(BulkArParams, done),
                         offsetof(BulkArParams, part_stride), offsetof(BulkArParams, wait_cycles)};
  const int m = (int)(sizeof(v) / sizeof(v[0]));
  for (int i = 0; i < m && i < n; ++i) out[i] = v[i];
  return m;
}

// Token-major persistent GEMM (see gemm_prefill_tm_kernel): Y[T, N] = act(X W^T + bias) [* (X Wu^T + bias_u)] +
// res_scale * residual, bf16.  gated != 0: gate rows [0, N) and up rows [dual_off, dual_off + N) of W.
static int prefill_tm(const void* X, int ldx, const void* W, int w_rows, int ldw, PrefillParams& p, int gated, int num_ctas,
                      cudaStream_t st) {
  const bool i8 = p.a_scale != nullptr;
  p.num_kb = i8 ? (p.K + 127) / 128 : (p.K + 63) / 64;
  p.gn = 8;
  if (num_ctas <= 0) {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    num_ctas = sms > 0 ? sms : 148;
  }
#define XFT_TM(NCOL, CG)                                                                    \
  (gated ? launch_prefill_tm<NCOL, true, CG>(X, ldx, W, w_rows, ldw, p, num_ctas, st)       \
         : launch_prefill_tm<NCOL, false, CG>(X, ldx, W, w_rows, ldw, p, num_ctas, st))
  if (p.group_tiles) return p.group_rows == 256 ? XFT_TM(256, 2) : XFT_TM(256, 1);
  // Which tile: the number of rounds that the SMs need, times what a 64-deep step of one tile takes, plus what a launch costs
  // beside its steps (accumulator on its way out, start of a cluster), all in steps of the largest tile (about 0.33 us).
  // Fitted to a sweep of 25 shapes on B200.  T x N x K, us with 256 x 256 (pair) / 256 x 128 (pair) / 128 x 128 tiles:
  // 8192 x 8192 x 8192: 757 / 953 / 1016; 2048 x 4096 x 4096: 59 / 66 / 70; 512 x 12288 x 4096: 49 / 48 / 52;
  // 512 x 4096 x 11008: 66 / 43 / 47; 778 x 2560 x 2048: 31 / 23 / 21; 200 x 3072 x 1024: 19 / 14 / 12.
  const int feats = gated ? 2 * p.N : p.N, pairs = num_ctas / 2 > 0 ? num_ctas / 2 : 1;
  auto rounds = [&](int tok, int ncol, int slots) {
    const long long tiles = (long long)((p.T + tok - 1) / tok) * ((feats + ncol - 1) / ncol);
    return (float)((tiles + slots - 1) / slots) * (float)p.num_kb;
  };
  const float wide = rounds(256, 256, pairs) + 8.f, pair = 0.6f * rounds(256, 128, pairs) + 9.f,
              single = 0.65f * rounds(128, 128, num_ctas) + 3.f;
  // W8A8 and codes: pairs only, the same line between wide and narrow tiles
#define XFT_TM_SRC(NCOL, SRC)                                                                       \
  (gated ? launch_prefill_tm<NCOL, true, 2, SRC>(X, ldx, W, w_rows, ldw, p, num_ctas, st)           \
         : launch_prefill_tm<NCOL, false, 2, SRC>(X, ldx, W, w_rows, ldw, p, num_ctas, st))
  if (i8) return wide <= pair ? XFT_TM_SRC(256, kTmI8) : XFT_TM_SRC(128, kTmI8);
  if (p.w_scale) return wide <= pair ? XFT_TM_SRC(256, kTmCodes) : XFT_TM_SRC(128, kTmCodes);
#undef XFT_TM_SRC
  if (wide <= pair && wide <= single) return XFT_TM(256, 2);
  return pair < single ? XFT_TM(128, 2) : XFT_TM(128, 1);
#undef XFT_TM
}

extern "C" int xft_gemm_bf16_prefill_tm(const void* X, int ldx, const void* W, int w_rows, int ldw, void* Y, int ldo, int T,
                                        int N, int K, int gated, int dual_off, const float* bias, const void* residual,
                                        int ldr, float res_scale, int act, int* status, int num_ctas, cudaStream_t st) {
  if (T <= 0 || N <= 0 || K <= 0) return 0;
  if ((K & 7) || (ldx & 7) || (ldw & 7)) return -2;
  PrefillParams p{};
  p.N = N; p.T = T; p.K = K; p.out = reinterpret_cast<__nv_bfloat16*>(Y); p.ldo = ldo; p.bias = bias;
  p.residual = reinterpret_cast<const __nv_bfloat16*>(residual); p.ldr = ldr; p.res_scale = res_scale; p.act = act;
  p.status = status; p.dual_off = dual_off;
  return prefill_tm(X, ldx, W, w_rows, ldw, p, gated, num_ctas, st);
}

// The same with fp32 rows: Y[T, N] = act(X W^T + bias).
extern "C" int xft_gemm_bf16_prefill_tm_f32(const void* X, int ldx, const void* W, int w_rows, int ldw, float* Y, int ldo, int T,
                                            int N, int K, const float* bias, int act, float param, int* status, cudaStream_t st) {
  if (T <= 0 || N <= 0 || K <= 0) return 0;
  if ((K & 7) || (ldx & 7) || (ldw & 7)) return -2;
  PrefillParams p{};
  p.N = N; p.T = T; p.K = K; p.out = reinterpret_cast<__nv_bfloat16*>(Y); p.ldo = ldo; p.bias = bias; p.res_scale = param; p.act = act;
  p.status = status; p.out_fp32 = 1;
  return prefill_tm(X, ldx, W, w_rows, ldw, p, 0, 0, st);
}

// Rows sorted by group (experts at prompt sizes): token tiles of `tile_rows` (128 or 256) rows from xft_moe_plan, W [groups * group_w_rows, K];
// gated: a group's rows are gate [0, N), up [dual_off, dual_off + N).  bf16 rows out.
extern "C" int xft_gemm_bf16_grouped_tm(const void* X, int ldx, int x_rows, const void* W, int w_rows, int ldw, void* Y, int ldo,
                                        int N, int K, int gated, int dual_off, int group_w_rows, const void* group_tiles,
                                        const int* num_group_tiles, int max_tiles, int tile_rows, int act, int* status, cudaStream_t st) {
  if (x_rows <= 0 || N <= 0 || K <= 0 || max_tiles <= 0) return 0;
  if ((K & 7) || (ldx & 7) || (ldw & 7) || !group_tiles || !num_group_tiles || (tile_rows != 128 && tile_rows != 256)) return -2;
  PrefillParams p{};
  p.N = N; p.T = x_rows; p.K = K; p.out = reinterpret_cast<__nv_bfloat16*>(Y); p.ldo = ldo; p.res_scale = 1.f; p.act = act;
  p.status = status; p.dual_off = dual_off;
  p.group_tiles = reinterpret_cast<const int4*>(group_tiles); p.num_group_tiles = num_group_tiles; p.group_w_rows = group_w_rows;
  p.t_tiles = max_tiles; p.group_rows = tile_rows;
  return prefill_tm(X, ldx, W, w_rows, ldw, p, gated, 0, st);
}

namespace xft {
// int8 codes of weights as bf16, four rows per block, 16 codes of each per thread.  Bound by the stores.
constexpr int kCodeRows = 4;
__global__ void __launch_bounds__(256) codes_bf16_kernel(const uint8_t* __restrict__ w, long long ldw, int rows, int K,
                                                         __nv_bfloat16* __restrict__ out) {
  grid_dep_launch();
  const int k = (blockIdx.y * 256 + threadIdx.x) * 16, r0 = blockIdx.x * kCodeRows;
  uint4 raw[kCodeRows];
#pragma unroll
  for (int i = 0; i < kCodeRows; ++i)
    if (k < K && r0 + i < rows) raw[i] = *reinterpret_cast<const uint4*>(w + (size_t)(r0 + i) * ldw + k);
  grid_dep_wait();                                                     // the buffer may still be read by the product before
#pragma unroll
  for (int i = 0; i < kCodeRows; ++i) {
    if (k >= K || r0 + i >= rows) return;
    const int8_t* c = reinterpret_cast<const int8_t*>(&raw[i]);
    uint32_t o[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const __nv_bfloat162 x = __floats2bfloat162_rn((float)c[2 * j], (float)c[2 * j + 1]);
      o[j] = *reinterpret_cast<const uint32_t*>(&x);
    }
    __nv_bfloat16* dst = out + (size_t)(r0 + i) * K + k;
    if ((reinterpret_cast<uintptr_t>(dst) & 31) == 0 && k + 8 < K) {
      st_global_256(dst, o);
    } else {
      reinterpret_cast<uint4*>(dst)[0] = make_uint4(o[0], o[1], o[2], o[3]);
      if (k + 8 < K) reinterpret_cast<uint4*>(dst)[1] = make_uint4(o[4], o[5], o[6], o[7]);
    }
  }
}
}  // namespace xft

// Prompts over int8 weights: the codes of all w_rows rows as bf16 into `codes` [w_rows, K], which holds them exactly, then the
// token-major product; y = scale (X codes^T) + zero sum(X) per weight row, then bias, activation, residual as in
// xft_gemm_bf16_prefill_tm.  x_sum: the rows' sums of X, where zero is given.  K a multiple of 8, rows of W on 16 bytes.
extern "C" int xft_gemm_codes_tm(const void* X, int ldx, const void* W, int w_rows, int ldw_bytes, void* codes, void* Y, int ldo,
                                 int out_fp32, int T, int N, int K, int gated, int dual_off, const float* scale, const float* zero,
                                 const float* x_sum, const float* bias, const void* residual, int ldr, float res_scale, int act,
                                 int* status, cudaStream_t st) {
  if (T <= 0 || N <= 0 || K <= 0) return 0;
  if ((K & 7) || (ldx & 7) || (ldw_bytes & 15) || ldw_bytes < K || !scale || (zero && !x_sum) ||
      ((reinterpret_cast<uintptr_t>(W) | reinterpret_cast<uintptr_t>(codes)) & 15))
    return -2;
  const cudaError_t e = launch_pdl(codes_bf16_kernel, dim3((w_rows + kCodeRows - 1) / kCodeRows, (K + 4095) / 4096), dim3(256), 0, st,
                                   (const uint8_t*)W, (long long)ldw_bytes, w_rows, K, (__nv_bfloat16*)codes);
  if (e != cudaSuccess) return (int)e;
  PrefillParams p{};
  p.N = N; p.T = T; p.K = K; p.out = reinterpret_cast<__nv_bfloat16*>(Y); p.ldo = ldo; p.out_fp32 = out_fp32; p.bias = bias;
  p.residual = reinterpret_cast<const __nv_bfloat16*>(residual); p.ldr = ldr; p.res_scale = res_scale; p.act = act;
  p.status = status; p.dual_off = dual_off; p.dual_rows = gated ? dual_off : 0x7fffffff;
  p.w_scale = scale; p.w_zero = zero; p.x_sum = x_sum;
  return prefill_tm(X, ldx, codes, w_rows, K, p, gated, 0, st);
}

// W8A8 above 64 tokens, see xft_w8a8_gemm (gemm_e4m3_sm100.cu)
namespace xft {
int launch_w8a8_prompt(const void* qx, int ldqx, const void* Wq, int w_rows, int ldw, void* Y, int ldo, int out_fp32, int T, int N, int K,
                       int gated, int dual_off, const float* a_scale, const float* a_zero, const float* a_qsum, const float* w_scale,
                       const float* w_zero, const float* w_sum, const float* bias, const void* residual, int ldr, float res_scale,
                       int act, int* status, cudaStream_t st) {
  PrefillParams p{};
  p.N = N; p.T = T; p.K = K; p.out = reinterpret_cast<__nv_bfloat16*>(Y); p.ldo = ldo; p.out_fp32 = out_fp32; p.bias = bias;
  p.residual = reinterpret_cast<const __nv_bfloat16*>(residual); p.ldr = ldr; p.res_scale = res_scale; p.act = act;
  p.status = status; p.dual_off = dual_off; p.dual_rows = gated ? dual_off : 0x7fffffff;
  p.a_scale = a_scale; p.a_zero = a_zero; p.a_qsum = a_qsum; p.w_scale = w_scale; p.w_zero = w_zero; p.w_sum = w_sum;
  return prefill_tm(qx, ldqx, Wq, w_rows, ldw, p, gated, 0, st);
}
}  // namespace xft
