// Activations on their way into an 8-bit product, a block per row: int8 codes with scale, zero point and sum of codes (W8A8), or the
// two e4m3 halves of gemm_e4m3_sm100.cu with scale and sum; with `gain`, of the row's RMSNorm.
//
// A row stays in registers: it is read once, and its norm, its range and its codes follow one another without another pass over
// memory.  Bound by that chain (fetch, one or two reductions over the block, store), which decode steps pay in front of every product;
// the norm in the same launch takes one more out of it.  us for 32 rows of 4096 in a chain of launches: codes alone 2.1 (quant_act_kernel
// and split_e4m3_kernel, which read their rows twice, 3.6 in a 7B layer), norm and codes in two launches 4.2, in one 2.9.
// Values, roundings and the order of the sums are those of the separate kernels.
#include "gemm_common.cuh"

#include <cuda_fp8.h>

namespace xft {

enum { kRowsInt8 = 0, kRowsSplit = 1, kRowsNibbles = 2 };              // the last: the halves in the order in which uint4 codes expand
constexpr int kRowThreads = 256;

struct RowsParams {
  const __nv_bfloat16* x; int ldx;
  const int* src; const int* rows_used;      // row r is row src[r] of x; rows from *rows_used on are left alone
  const float* gain; float eps;              // NORM
  int K, Kp;                                 // Kp: columns of one half of a split row
  uint8_t* out; long long ldo;
  float* scale; float* zero; float* sum;
};

__device__ __forceinline__ float rows_block_sum(float v, float* s) {   // block_sum of elementwise.cu
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = v;
  __syncthreads();
  float t = 0.f;
#pragma unroll
  for (int w = 0; w < kRowThreads / 32; ++w) t += s[w];
  return t;
}

template <int CH, bool NORM, int MODE>
__global__ void __launch_bounds__(kRowThreads) quant_rows_kernel(const RowsParams p) {
  __shared__ float s_ss[8], s_a[8], s_b[8];
  grid_dep_launch();
  grid_dep_wait();
  const int r = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (p.rows_used && r >= *p.rows_used) return;
  const uint4* row = reinterpret_cast<const uint4*>(p.x + (size_t)(p.src ? p.src[r] : r) * p.ldx);
  const int nch = p.K / 8;
  uint4 v[CH];
#pragma unroll
  for (int c = 0; c < CH; ++c) {
    const int i = tid + c * kRowThreads;
    v[c] = i < nch ? row[i] : make_uint4(0, 0, 0, 0);
  }
  auto pair = [&](int c, int j) { return __bfloat1622float2(reinterpret_cast<const __nv_bfloat162*>(&v[c])[j]); };
  if constexpr (NORM) {
    float ss = 0.f;
#pragma unroll
    for (int c = 0; c < CH; ++c)
      if (tid + c * kRowThreads < nch)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 f = pair(c, j);
          ss += f.x * f.x;
          ss += f.y * f.y;
        }
    ss = rows_block_sum(ss, s_ss);
    const float inv = rsqrtf(ss / p.K + p.eps);
#pragma unroll
    for (int c = 0; c < CH; ++c) {
      const int i = tid + c * kRowThreads;
      if (i >= nch) continue;
      const float4 w0 = __ldg(reinterpret_cast<const float4*>(p.gain) + 2 * i), w1 = __ldg(reinterpret_cast<const float4*>(p.gain) + 2 * i + 1);
      const float w[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 f = pair(c, j);
        reinterpret_cast<__nv_bfloat162*>(&v[c])[j] = __floats2bfloat162_rn(f.x * inv * w[2 * j], f.y * inv * w[2 * j + 1]);
      }
    }
  }
  if constexpr (MODE == kRowsInt8) {
    float mx = -INFINITY, mn = INFINITY;
#pragma unroll
    for (int c = 0; c < CH; ++c)
      if (tid + c * kRowThreads < nch)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 f = pair(c, j);
          mx = fmaxf(mx, fmaxf(f.x, f.y));
          mn = fminf(mn, fminf(f.x, f.y));
        }
    for (int o = 16; o > 0; o >>= 1) { mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o)); mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o)); }
    if (lane == 0) { s_a[warp] = mx; s_b[warp] = mn; }
    __syncthreads();
    mx = s_a[0]; mn = s_b[0];
#pragma unroll
    for (int w = 1; w < 8; ++w) { mx = fmaxf(mx, s_a[w]); mn = fminf(mn, s_b[w]); }
    const float z = 0.5f * (mx + mn);
    const float s = fmaxf(fmaxf(mx - z, z - mn) / 127.f, 1e-10f);
    const float inv = 1.f / s;
    float acc = 0.f;
    auto code = [&](float x) {
      const float q = fminf(fmaxf(rintf((x - z) * inv), -127.f), 127.f);
      acc += q;
      return (int8_t)q;
    };
#pragma unroll
    for (int c = 0; c < CH; ++c) {
      const int i = tid + c * kRowThreads;
      if (i >= nch) continue;
      int8_t q[8];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 f = pair(c, j);
        q[2 * j] = code(f.x);
        q[2 * j + 1] = code(f.y);
      }
      uint2 w;
      memcpy(&w, q, 8);
      *reinterpret_cast<uint2*>(p.out + (size_t)r * p.ldo + 8 * i) = w;
    }
    acc = rows_block_sum(acc, s_ss);
    if (tid == 0) { p.scale[r] = s; p.zero[r] = z; p.sum[r] = acc; }
  } else {
    float mx = 0.f, sm = 0.f;
#pragma unroll
    for (int c = 0; c < CH; ++c)
      if (tid + c * kRowThreads < nch)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 f = pair(c, j);
          sm += f.x + f.y;
          const float a = fabsf(f.x), b = fabsf(f.y);
          if (a <= 3.4e38f) mx = fmaxf(mx, a);                         // infinities and NaN have no part in the scale
          if (b <= 3.4e38f) mx = fmaxf(mx, b);
        }
    for (int o = 16; o > 0; o >>= 1) {
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
      sm += __shfl_xor_sync(0xffffffffu, sm, o);
    }
    if (lane == 0) { s_a[warp] = mx; s_b[warp] = sm; }
    __syncthreads();
    mx = s_a[0]; sm = s_b[0];
#pragma unroll
    for (int w = 1; w < 8; ++w) { mx = fmaxf(mx, s_a[w]); sm += s_b[w]; }
    int e;
    const float f = frexpf(mx, &e);                                    // mx = f 2^e, 0.5 <= f < 1: at most 448 = 0.875 * 2^9
    e = mx == 0.f ? 0 : max(-100, e - 9 + (f > 0.875f));
    const float inv = exp2f((float)-e);
    if (tid == 0) {
      p.scale[r] = exp2f((float)e);
      if (p.sum) p.sum[r] = sm;
    }
    uint8_t* hi_row = p.out + (size_t)r * p.ldo;
#pragma unroll
    for (int c = 0; c < CH; ++c) {
      const int k = (tid + c * kRowThreads) * 8;
      if (k >= p.Kp) continue;
      uint8_t hi[8], lo[8];
      if (k < p.K) {
        const __nv_bfloat16* b = reinterpret_cast<const __nv_bfloat16*>(&v[c]);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float y = __bfloat162float(b[i]) * inv;
          const __nv_fp8_storage_t q = __nv_cvt_float_to_fp8(y, __NV_SATFINITE, __NV_E4M3);
          const float back = __half2float(__half(__nv_cvt_fp8_to_halfraw(q, __NV_E4M3)));
          hi[i] = fabsf(y) <= 3.4e38f ? q : 0x7F;                      // an infinity or NaN makes its row NaN
          lo[i] = fabsf(y) <= 3.4e38f ? __nv_cvt_float_to_fp8((y - back) * 16.f, __NV_SATFINITE, __NV_E4M3) : 0;
        }
      } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) hi[i] = lo[i] = 0;                 // 0 x garbage of a padded column could be NaN
      }
      if constexpr (MODE == kRowsNibbles) {
        const int at = (k & ~31) + (k & 31) / 2;
#pragma unroll
        for (int o = 0; o < 2; ++o) {
          *reinterpret_cast<uchar4*>(hi_row + at + 16 * o) = make_uchar4(hi[o], hi[2 + o], hi[4 + o], hi[6 + o]);
          *reinterpret_cast<uchar4*>(hi_row + p.Kp + at + 16 * o) = make_uchar4(lo[o], lo[2 + o], lo[4 + o], lo[6 + o]);
        }
      } else {
        uint2 a, b;
        memcpy(&a, hi, 8);
        memcpy(&b, lo, 8);
        *reinterpret_cast<uint2*>(hi_row + k) = a;
        *reinterpret_cast<uint2*>(hi_row + p.Kp + k) = b;
      }
    }
  }
}

template <bool NORM, int MODE>
static int launch_rows(const RowsParams& p, int rows, cudaStream_t st) {
  const int span = MODE == kRowsInt8 ? p.K : p.Kp;
  const auto kernel = [&] {
    if constexpr (!NORM) {                                             // with a norm up to 8192, see xft_rms_quant_act
      if (span > 16384) return quant_rows_kernel<16, NORM, MODE>;
      if (span > 8192) return quant_rows_kernel<8, NORM, MODE>;
    }
    return span > 4096 ? quant_rows_kernel<4, NORM, MODE> : quant_rows_kernel<2, NORM, MODE>;
  }();
  const cudaError_t e = launch_pdl(kernel, dim3(rows), dim3(kRowThreads), 0, st, p);
  return e != cudaSuccess ? (int)e : (int)cudaGetLastError();
}

// -1: not a form of these kernels (rows that do not start on 16 bytes, longer than 32768), see xft_quant_act and xft_split_e4m3.
int launch_quant_act(const void* x, int ldx, const float* gain, float eps, void* q, int ldq, float* scale, float* zero, float* sum,
                     int rows, int K, cudaStream_t st) {
  if ((K & 7) || (ldx & 7) || (ldq & 7) || K > 32768 ||
      ((reinterpret_cast<uintptr_t>(x) & 15) | (reinterpret_cast<uintptr_t>(q) & 7) | (reinterpret_cast<uintptr_t>(gain) & 15)))
    return -1;
  RowsParams p{};
  p.x = (const __nv_bfloat16*)x; p.ldx = ldx; p.gain = gain; p.eps = eps; p.K = K; p.out = (uint8_t*)q; p.ldo = ldq;
  p.scale = scale; p.zero = zero; p.sum = sum;
  return gain ? launch_rows<true, kRowsInt8>(p, rows, st) : launch_rows<false, kRowsInt8>(p, rows, st);
}

int launch_split(const void* x, int ldx, const int* src, const int* rows_used, const float* gain, float eps, int rows, int K, int Kp,
                 int nibbles, void* out, float* scale, float* sum, cudaStream_t st) {
  if ((K & 7) || (ldx & 7) || Kp > 32768 ||
      ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(gain)) & 15))
    return -1;
  RowsParams p{};
  p.x = (const __nv_bfloat16*)x; p.ldx = ldx; p.src = src; p.rows_used = rows_used; p.gain = gain; p.eps = eps; p.K = K; p.Kp = Kp;
  p.out = (uint8_t*)out; p.ldo = 2 * Kp; p.scale = scale; p.sum = sum;
  if (gain) return nibbles ? launch_rows<true, kRowsNibbles>(p, rows, st) : launch_rows<true, kRowsSplit>(p, rows, st);
  return nibbles ? launch_rows<false, kRowsNibbles>(p, rows, st) : launch_rows<false, kRowsSplit>(p, rows, st);
}

}  // namespace xft

using namespace xft;

// RMSNorm(x; gain, eps) as bf16 rows would hold it, then what xft_quant_act / xft_split_e4m3 make of it.  2048 <= K <= 8192: the sizes at
// which xft_rmsnorm adds a row's squares in this order.
extern "C" int xft_rms_quant_act(const void* x, int ldx, const float* gain, float eps, void* q, int ldq, float* scale, float* zero,
                                 float* qsum, int T, int K, cudaStream_t st) {
  if (T <= 0) return 0;
  if (K < 2048 || K > 8192 || !gain) return -1;
  return launch_quant_act(x, ldx, gain, eps, q, ldq, scale, zero, qsum, T, K, st);
}

extern "C" int xft_rms_split_e4m3(const void* x, int ldx, const float* gain, float eps, int rows, int K, int nibbles, void* out,
                                  float* scale, float* sum, cudaStream_t st) {
  if (rows <= 0) return 0;
  if (K < 2048 || K > 8192 || !gain) return -1;
  return launch_split(x, ldx, nullptr, nullptr, gain, eps, rows, K, (K + 31) / 32 * 32, nibbles, out, scale, sum, st);
}
