// RMSNorm, residual add + RMSNorm, and the NeoX rotary embedding for sm_100: the operators that sit
// in front of the quantise + GEMM path in a transformer block (reference kernels/rmsnorm.cu:21-59,
// kernels/rope.cu:19-41; CPU golden reference/reference.cpp:11-53).  All three are HBM-bound:
// every element is read once and written once.
//
//   * rmsnorm16_kernel, rmsnorm_vec_kernel (fp32, and 16-bit rows that are no whole 32-byte pieces): a row lives in registers
//     between the two passes the reference makes over it, so it is read from memory once; 32 to 256
//     threads per row depending on its length, several rows per CTA when rows are short.
//   * rope_kernel: the angle of (position, i) does not depend on the head, so a CTA computes the
//     cos / sin table of its token once and applies it to a block of heads with 16-byte accesses.
//     The frequencies come from the host (the C library's powf, as in the CPU golden: at position
//     100 000 two units in the last place of a device powf would be 0.02 rad).
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "internal.h"
#include "quant_math.cuh"

namespace ib200 {
namespace {

constexpr int kThreads = 256;
constexpr int kNormThreads = 128;   // rmsnorm16_kernel: per part of a row
constexpr int kMaxVec = 8;   // 16-byte vectors of a row that one thread keeps in registers

template <typename T>
struct VecOf {
  static constexpr int N = 16 / sizeof(T);
};

template <typename T>
__device__ __forceinline__ float to_f32(T v);
template <>
__device__ __forceinline__ float to_f32(float v) { return v; }
template <>
__device__ __forceinline__ float to_f32(__half v) { return __half2float(v); }
template <>
__device__ __forceinline__ float to_f32(__nv_bfloat16 v) { return __bfloat162float(v); }
template <typename T>
__device__ __forceinline__ T from_f32(float v);
template <>
__device__ __forceinline__ float from_f32(float v) { return v; }
template <>
__device__ __forceinline__ __half from_f32(float v) { return __float2half_rn(v); }
template <>
__device__ __forceinline__ __nv_bfloat16 from_f32(float v) { return __float2bfloat16_rn(v); }

template <typename T>
__device__ __forceinline__ void unpack(const uint4& raw, float (&f)[VecOf<T>::N]) {
  const T* e = reinterpret_cast<const T*>(&raw);
#pragma unroll
  for (int i = 0; i < VecOf<T>::N; ++i) f[i] = to_f32<T>(e[i]);
}
template <typename T>
__device__ __forceinline__ uint4 pack(const float (&f)[VecOf<T>::N]) {
  uint4 raw;
  T* e = reinterpret_cast<T*>(&raw);
#pragma unroll
  for (int i = 0; i < VecOf<T>::N; ++i) e[i] = from_f32<T>(f[i]);
  return raw;
}

// kAdd: residual[r, :] += x[r, :] first (stored in T), then the norm of the sum.  As in the
// reference's kernel the sum of squares uses the unrounded sums and the output the stored ones.
// tpr = threads per row (a power of two, 32 .. 256); rows per CTA = 256 / tpr; NV = 16-byte
// vectors of the row per thread, kept packed in registers between the two passes.
template <typename T, bool kAdd, int NV>
__global__ void __launch_bounds__(kThreads)
rmsnorm_vec_kernel(T* __restrict__ out, T* __restrict__ residual, const T* __restrict__ in,
                   const T* __restrict__ weight, float eps, int64_t rows, int cols, int tpr) {
  constexpr int V = VecOf<T>::N;
  __shared__ float red[kThreads / 32];
  const int lane_in_row = threadIdx.x & (tpr - 1);
  const int64_t row = static_cast<int64_t>(blockIdx.x) * (kThreads / tpr) + (threadIdx.x / tpr);
  const bool live = row < rows;
  const int nvec = cols / V;
  const uint4* src = reinterpret_cast<const uint4*>(in + (live ? row : 0) * cols);
  uint4* res = kAdd ? reinterpret_cast<uint4*>(residual + (live ? row : 0) * cols) : nullptr;

  uint4 raw[NV], rraw[kAdd ? NV : 1];
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    const int j = lane_in_row + k * tpr;
    const bool have = live && j < nvec;
    raw[k] = have ? __ldg(src + j) : make_uint4(0u, 0u, 0u, 0u);
    if constexpr (kAdd) rraw[k] = have ? res[j] : make_uint4(0u, 0u, 0u, 0u);
  }
  float partial = 0.0f;
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    float v[V];
    unpack<T>(raw[k], v);
    if constexpr (kAdd) {
      float r[V];
      unpack<T>(rraw[k], r);
#pragma unroll
      for (int i = 0; i < V; ++i) r[i] = __fadd_rn(r[i], v[i]);
#pragma unroll
      for (int i = 0; i < V; ++i) partial = fmaf(r[i], r[i], partial);
      raw[k] = pack<T>(r);   // what is stored; the output is computed from it
      const int j = lane_in_row + k * tpr;
      if (live && j < nvec) res[j] = raw[k];
    } else {
#pragma unroll
      for (int i = 0; i < V; ++i) partial = fmaf(v[i], v[i], partial);
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) partial += __shfl_xor_sync(0xFFFFFFFFu, partial, o);
  if (tpr > 32) {
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = partial;
    __syncthreads();
    const int w0 = (threadIdx.x / tpr) * (tpr >> 5);
    partial = 0.0f;
    for (int w = 0; w < (tpr >> 5); ++w) partial += red[w0 + w];
  }
  const float inv = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(partial, static_cast<float>(cols)), eps)));
  uint4* dst = reinterpret_cast<uint4*>(out + (live ? row : 0) * cols);
  const uint4* wv = reinterpret_cast<const uint4*>(weight);
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    const int j = lane_in_row + k * tpr;
    if (live && j < nvec) {
      float v[V], w[V], y[V];
      unpack<T>(raw[k], v);
      unpack<T>(__ldg(wv + j), w);
#pragma unroll
      for (int i = 0; i < V; ++i) y[i] = __fmul_rn(__fmul_rn(v[i], inv), w[i]);
      dst[j] = pack<T>(y);
    }
  }
}

// Two sums of a 32-bit word of 16-bit elements rounded back to it
template <typename T>
__device__ __forceinline__ uint32_t narrow2(float2 f) {
  if constexpr (std::is_same<T, __half>::value) {
    const __half2 h = __floats2half2_rn(f.x, f.y);
    return *reinterpret_cast<const uint32_t*>(&h);
  } else {
    const __nv_bfloat162 h = __floats2bfloat162_rn(f.x, f.y);
    return *reinterpret_cast<const uint32_t*>(&h);
  }
}
template <bool kWide>
__device__ __forceinline__ Words8 load32(const void* p) {   // (not through the read-only path: written by this kernel)
  Words8 v;
  if constexpr (kWide) {
    asm volatile("ld.global.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(v.w[0]), "=r"(v.w[1]), "=r"(v.w[2]), "=r"(v.w[3]), "=r"(v.w[4]), "=r"(v.w[5]), "=r"(v.w[6]), "=r"(v.w[7])
                 : "l"(p)
                 : "memory");
  } else {
    const uint4 a = static_cast<const uint4*>(p)[0], b = static_cast<const uint4*>(p)[1];
    v.w[0] = a.x, v.w[1] = a.y, v.w[2] = a.z, v.w[3] = a.w;
    v.w[4] = b.x, v.w[5] = b.y, v.w[6] = b.z, v.w[7] = b.w;
  }
  return v;
}
template <bool kWide>
__device__ __forceinline__ void store32(void* p, const Words8& v) {
  if constexpr (kWide) {
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(v.w[0]), "r"(v.w[1]), "r"(v.w[2]),
                 "r"(v.w[3]), "r"(v.w[4]), "r"(v.w[5]), "r"(v.w[6]), "r"(v.w[7])
                 : "memory");
  } else {
    static_cast<uint4*>(p)[0] = make_uint4(v.w[0], v.w[1], v.w[2], v.w[3]);
    static_cast<uint4*>(p)[1] = make_uint4(v.w[4], v.w[5], v.w[6], v.w[7]);
  }
}

// 16-bit types, rows of whole 32-byte pieces: RMSNorm, or residual add + RMSNorm (kAdd, as above), whose result is stored
// (out = T [rows, cols]) or, kQuant, quantised in the same pass (out = E4M3 [rows, cols], one scale per 128; cols % 128
// == 0): the normalised value is rounded to T first and quantised by the quantiser's own functions, so q / scales are what
// quant_fp8_per_token_group gives on the norm's output, bit for bit, and the 16-bit matrix between the two never exists.
//
// A lane owns pieces of sixteen elements (quant_math.cuh), NV of them; eight lanes own a group.  The squares are added in the
// order of rmsnorm_vec_kernel, so that a row's bits depend neither on the kernel nor on the alignment that chose it: a
// piece is two vectors of it, so `lanes` (16 .. 128) lanes, half as many as it has threads per row, hold what two
// neighbouring threads of it hold, as two sums.  kParts = 1: a lane adds all of it.  kParts = 2: it adds the first half of it
// and hands the two sums to a lane that holds the second half.
// Bound by HBM; what is left over it are the barriers between the two passes over a row, hidden by the other CTAs of the SM.
// Norm + quantisation with residual, bf16, us, rmsnorm_vec_kernel's layout (16 bytes per access) -> this one, behind a flush
// of L2: 4096 x 7168 47.2 -> 38.9, 16000 x 5120 149 -> 109, 64 x 7168 5.9 -> 4.4, 65536 x 128 27.1 -> 23.5; without residual
// 4096 x 7168 34.7 -> 28.2; the norm alone with residual 46.4 -> 37.7, without 25.4 -> 23.3.
template <typename T, bool kAdd, bool kQuant, int kParts, int NV, bool kWide>
__global__ void __launch_bounds__(kNormThreads * kParts, kParts == 2 ? 2 : kQuant && !kAdd ? 5 : 4)
rmsnorm16_kernel(void* __restrict__ out, float* __restrict__ scales, T* __restrict__ residual, const T* __restrict__ in,
                 const T* __restrict__ weight, float eps, int64_t rows, int cols, int lanes) {
  __shared__ float2 handed[kParts == 2 ? kNormThreads : 1];
  __shared__ float red[kNormThreads / 16];
  const int slot = threadIdx.x & (kNormThreads - 1);   // lane among those of the CTA's first (second) parts
  const int part = threadIdx.x / kNormThreads;
  const int lane_in_row = slot & (lanes - 1);
  const int64_t row = static_cast<int64_t>(blockIdx.x) * (kNormThreads / lanes) + slot / lanes;
  const bool live = row < rows;
  const int pieces = cols / 16;
  const int64_t at = (live ? row : 0) * cols;
  const int first = lane_in_row + part * NV * lanes;   // piece k of this lane is first + k * lanes

  Words8 x[NV], r[kAdd ? NV : 1];
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    const int j = first + k * lanes;
    const bool have = live && j < pieces;
    x[k] = have ? load_nc32<kWide>(in + at + j * 16) : zero_words();
    if constexpr (kAdd) r[k] = have ? load32<kWide>(residual + at + j * 16) : zero_words();
  }
  float2 squares = make_float2(0.0f, 0.0f);   // of the first and of the second vectors of the pieces
#pragma unroll 1
  for (int turn = 0; turn < kParts; ++turn) {
    if (part == turn) {
#pragma unroll
      for (int k = 0; k < NV; ++k) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float2 a = widen2<T>(x[k].w[i]), b = widen2<T>(x[k].w[i + 4]);
          float2 lo = make_float2(a.x, b.x), hi = make_float2(a.y, b.y);
          if constexpr (kAdd) {
            const float2 ra = widen2<T>(r[k].w[i]), rb = widen2<T>(r[k].w[i + 4]);
            lo = __fadd2_rn(make_float2(ra.x, rb.x), lo);
            hi = __fadd2_rn(make_float2(ra.y, rb.y), hi);
            x[k].w[i] = narrow2<T>(make_float2(lo.x, hi.x));   // what is stored; the output is computed from it
            x[k].w[i + 4] = narrow2<T>(make_float2(lo.y, hi.y));
          }
          squares = __ffma2_rn(lo, lo, squares);
          squares = __ffma2_rn(hi, hi, squares);
        }
        const int j = first + k * lanes;
        if (kAdd && live && j < pieces) store32<kWide>(residual + at + j * 16, x[k]);
      }
    }
    if (kParts == 2 && turn == 0) {
      if (part == 0) handed[slot] = squares;
      __syncthreads();
      if (part == 1) squares = handed[slot];
    }
  }
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) {
    squares.x += __shfl_xor_sync(0xFFFFFFFFu, squares.x, o);
    squares.y += __shfl_xor_sync(0xFFFFFFFFu, squares.y, o);
  }
  float partial = squares.x + squares.y;   // (last part) of sixteen lanes: a warp of rmsnorm_vec_kernel
  if (kParts == 2 || lanes > 16) {
    if (part == kParts - 1 && (slot & 15) == 0) red[slot >> 4] = partial;
    __syncthreads();
    const int w0 = (slot / lanes) * (lanes >> 4);
    partial = 0.0f;
    for (int w = 0; w < (lanes >> 4); ++w) partial += red[w0 + w];
  }
  const float inv = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(partial, static_cast<float>(cols)), eps)));
  const float2 inv2 = make_float2(inv, inv);
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    const int j = first + k * lanes;
    const bool have = live && j < pieces;   // kQuant: the same for the eight lanes of a group (pieces % 8 == 0)
    const Words8 w = have ? load_nc32<kWide>(weight + j * 16) : zero_words();
    Words8 y;
#pragma unroll
    for (int i = 0; i < 8; ++i)
      y.w[i] = narrow2<T>(__fmul2_rn(__fmul2_rn(widen2<T>(x[k].w[i]), inv2), widen2<T>(w.w[i])));
    if constexpr (kQuant) {
      float amax = absmax16<T>(y);
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, o));
      const float scale = group_scale(amax);
      if (have) {
        store16<kWide>(static_cast<uint8_t*>(out) + at + j * 16, quantise16<T>(y, amax, scale));
        if ((threadIdx.x & 7) == 0) scales[(live ? row : 0) * (cols >> 7) + (j >> 3)] = scale;
      }
    } else {
      if (have) store32<kWide>(static_cast<T*>(out) + at + j * 16, y);
    }
  }
}

// (cols <= 16 * 128 * kMaxPieces; pointers 16-byte aligned, q 8-byte; wide: 32, q 16)
constexpr int kMaxPieces = 8;
// Up to so many rows take two parts, since what counts is how long a lane is busy (norm + quantisation with residual of 64 x
// 7168: 4.4 us, 5.6 in one part).  More rows take one part, which holds a row in half as many threads and one barrier less
// (512 x 7168 8.0 us, 9.6 in two parts, 4096 x 7168 38.9 and 48.9).  More than eight vectors per chain would not fit one lane.
constexpr int64_t kNormFewRows = 256;
template <typename T, bool kAdd, bool kQuant>
int launch_rmsnorm16(void* out, void* scales, void* residual, const void* in, const void* weight, int64_t rows, int64_t cols,
                     float eps, cudaStream_t stream) {
  const int64_t pieces = cols / 16;
  int lanes = 16;   // half of what launch_rmsnorm_t gives rmsnorm_vec_kernel
  while (lanes < kNormThreads && static_cast<int64_t>(lanes) * 4 < pieces) lanes <<= 1;
  const int rows_per_cta = kNormThreads / lanes;
  const int64_t grid = (rows + rows_per_cta - 1) / rows_per_cta;
  if (grid > 0x7FFFFFFFLL) return INFEROP_ERR_LIMIT;
  const uintptr_t all = reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(weight) | reinterpret_cast<uintptr_t>(residual);
  const bool wide = all % 32 == 0 && reinterpret_cast<uintptr_t>(out) % (kQuant ? 16 : 32) == 0;
  const int64_t per_lane = (pieces + lanes - 1) / lanes;
  const bool halves = per_lane > 4 || rows <= kNormFewRows;
  const auto launch = [&](auto* kernel) {
    kernel<<<static_cast<unsigned>(grid), halves ? 2 * kNormThreads : kNormThreads, 0, stream>>>(
        out, static_cast<float*>(scales), static_cast<T*>(residual), static_cast<const T*>(in), static_cast<const T*>(weight), eps,
        rows, static_cast<int>(cols), lanes);
  };
  if (per_lane > 4) launch(wide ? rmsnorm16_kernel<T, kAdd, kQuant, 2, 4, true> : rmsnorm16_kernel<T, kAdd, kQuant, 2, 4, false>);
  else if (halves) launch(wide ? rmsnorm16_kernel<T, kAdd, kQuant, 2, 2, true> : rmsnorm16_kernel<T, kAdd, kQuant, 2, 2, false>);
  else if (per_lane > 2) launch(wide ? rmsnorm16_kernel<T, kAdd, kQuant, 1, 4, true> : rmsnorm16_kernel<T, kAdd, kQuant, 1, 4, false>);
  else launch(wide ? rmsnorm16_kernel<T, kAdd, kQuant, 1, 2, true> : rmsnorm16_kernel<T, kAdd, kQuant, 1, 2, false>);
  return check_launch();
}

// Any shape and alignment: one CTA per row, two strided passes (the reference's own scheme).
template <typename T, bool kAdd>
__global__ void __launch_bounds__(kThreads)
rmsnorm_any_kernel(T* __restrict__ out, T* __restrict__ residual, const T* __restrict__ in,
                   const T* __restrict__ weight, float eps, int cols) {
  __shared__ float red[kThreads / 32];
  const int64_t row = blockIdx.x;
  const T* x = in + row * cols;
  T* res = kAdd ? residual + row * cols : nullptr;
  float partial = 0.0f;
  for (int i = threadIdx.x; i < cols; i += kThreads) {
    float v = to_f32<T>(x[i]);
    if constexpr (kAdd) {
      v = __fadd_rn(to_f32<T>(res[i]), v);
      res[i] = from_f32<T>(v);   // the same thread reads it back below
    }
    partial = fmaf(v, v, partial);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) partial += __shfl_xor_sync(0xFFFFFFFFu, partial, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = partial;
  __syncthreads();
  partial = 0.0f;
  for (int w = 0; w < kThreads / 32; ++w) partial += red[w];
  const float inv = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(partial, static_cast<float>(cols)), eps)));
  T* y = out + row * cols;
  for (int i = threadIdx.x; i < cols; i += kThreads) {
    const float v = to_f32<T>(kAdd ? res[i] : x[i]);
    y[i] = from_f32<T>(__fmul_rn(__fmul_rn(v, inv), to_f32<T>(weight[i])));
  }
}

template <typename T, bool kAdd>
int launch_rmsnorm_t(void* out, void* residual, const void* in, const void* weight, int64_t rows, int64_t cols,
                     float eps, cudaStream_t stream) {
  constexpr int V = VecOf<T>::N;
  const bool aligned = ((reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(in) |
                         reinterpret_cast<uintptr_t>(weight) | reinterpret_cast<uintptr_t>(residual)) & 15u) == 0;
  const int64_t nvec = cols / V;
  if constexpr (sizeof(T) == 2) {
    if (aligned && cols % 16 == 0 && cols / 16 <= static_cast<int64_t>(kNormThreads) * kMaxPieces)
      return launch_rmsnorm16<T, kAdd, false>(out, nullptr, residual, in, weight, rows, cols, eps, stream);
  }
  if (aligned && cols % V == 0 && nvec <= static_cast<int64_t>(kThreads) * kMaxVec) {
    int tpr = 32;
    while (tpr < kThreads && static_cast<int64_t>(tpr) * 4 < nvec) tpr <<= 1;   // about four vectors per thread
    const int per_thread = static_cast<int>((nvec + tpr - 1) / tpr);
    const int rows_per_cta = kThreads / tpr;
    const int64_t grid = (rows + rows_per_cta - 1) / rows_per_cta;
    if (grid > 0x7FFFFFFFLL) return INFEROP_ERR_LIMIT;
    T* o = static_cast<T*>(out);
    T* r = static_cast<T*>(residual);
    const T* i = static_cast<const T*>(in);
    const T* w = static_cast<const T*>(weight);
    const unsigned g = static_cast<unsigned>(grid);
    const int c = static_cast<int>(cols);
    if (per_thread <= 1) rmsnorm_vec_kernel<T, kAdd, 1><<<g, kThreads, 0, stream>>>(o, r, i, w, eps, rows, c, tpr);
    else if (per_thread <= 2) rmsnorm_vec_kernel<T, kAdd, 2><<<g, kThreads, 0, stream>>>(o, r, i, w, eps, rows, c, tpr);
    else if (per_thread <= 4) rmsnorm_vec_kernel<T, kAdd, 4><<<g, kThreads, 0, stream>>>(o, r, i, w, eps, rows, c, tpr);
    else rmsnorm_vec_kernel<T, kAdd, kMaxVec><<<g, kThreads, 0, stream>>>(o, r, i, w, eps, rows, c, tpr);
  } else {
    if (rows > 0x7FFFFFFFLL || cols > 0x7FFFFFFFLL) return INFEROP_ERR_LIMIT;
    rmsnorm_any_kernel<T, kAdd><<<static_cast<unsigned>(rows), kThreads, 0, stream>>>(
        static_cast<T*>(out), static_cast<T*>(residual), static_cast<const T*>(in), static_cast<const T*>(weight),
        eps, static_cast<int>(cols));
  }
  return check_launch();
}

// ------------------------------------------------------------------------------------- rotary embedding
constexpr int kRopeThreads = 128;
constexpr int kRopeMaxHalf = 512;   // rotary_dim up to 1024

// The frequencies base^(-2 i / rotary_dim) * yarn depend on i only: the launcher computes them on the
// host with the C library's powf, the very function the CPU golden calls, and passes them in the
// kernel's parameter block.
struct RopeFreq {
  float f[kRopeMaxHalf];
};

// grid (tokens, ceil(heads / heads_per_cta)).  kVec: 16-byte accesses (rotary_dim / 2 a multiple of the
// vector length, rows 16-byte aligned); otherwise element by element.
template <typename T, bool kVec>
__global__ void __launch_bounds__(kRopeThreads)
rope_kernel(T* __restrict__ qkv, const int64_t* __restrict__ positions, int heads, int head_dim, int rotary_dim,
            int heads_per_cta, const __grid_constant__ RopeFreq freq) {
  constexpr int V = VecOf<T>::N;
  constexpr int kItems = 4;             // vector pairs a thread handles per CTA (the launcher sizes the head block so)
  __shared__ float2 cs[kRopeMaxHalf];   // (cos, sin) of this token's angles
  const int half = rotary_dim >> 1;
  const int64_t t = blockIdx.x;
  const int h0 = blockIdx.y * heads_per_cta;
  const int h1 = min(heads, h0 + heads_per_cta);
  T* tok = qkv + t * heads * head_dim;
  // the operands are requested before the table is computed, so that the two latencies overlap
  uint4 r0[kVec ? kItems : 1], r1[kVec ? kItems : 1];
  if constexpr (kVec) {
    const int vec_per_head = half / V;
    const int work = (h1 - h0) * vec_per_head;
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
      const int wi = threadIdx.x + k * kRopeThreads;
      if (wi < work) {
        const int h = h0 + wi / vec_per_head, j = wi % vec_per_head;
        r0[k] = *(reinterpret_cast<const uint4*>(tok + h * head_dim) + j);
        r1[k] = *(reinterpret_cast<const uint4*>(tok + h * head_dim + half) + j);
      }
    }
  }
  const float pos = static_cast<float>(__ldg(positions + t));
  for (int i = threadIdx.x; i < half; i += kRopeThreads) {
    float sn, c;
    sincosf(__fmul_rn(pos, freq.f[i]), &sn, &c);   // the accurate version: angles reach 1e5 rad
    cs[i] = make_float2(c, sn);
  }
  __syncthreads();
  if constexpr (kVec) {
    const int vec_per_head = half / V;
    const int work = (h1 - h0) * vec_per_head;
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
      const int wi = threadIdx.x + k * kRopeThreads;
      if (wi < work) {
        const int h = h0 + wi / vec_per_head, j = wi % vec_per_head;
        float x0[V], x1[V], y0[V], y1[V];
        unpack<T>(r0[k], x0);
        unpack<T>(r1[k], x1);
#pragma unroll
        for (int i = 0; i < V; ++i) {
          const float2 a = cs[j * V + i];
          y0[i] = __fsub_rn(__fmul_rn(x0[i], a.x), __fmul_rn(x1[i], a.y));
          y1[i] = __fadd_rn(__fmul_rn(x1[i], a.x), __fmul_rn(x0[i], a.y));
        }
        *(reinterpret_cast<uint4*>(tok + h * head_dim) + j) = pack<T>(y0);
        *(reinterpret_cast<uint4*>(tok + h * head_dim + half) + j) = pack<T>(y1);
      }
    }
  } else {
    const int work = (h1 - h0) * half;
    for (int wi = threadIdx.x; wi < work; wi += kRopeThreads) {
      const int h = h0 + wi / half, i = wi % half;
      T* p = tok + h * head_dim;
      const float x0 = to_f32<T>(p[i]), x1 = to_f32<T>(p[i + half]);
      const float2 a = cs[i];
      p[i] = from_f32<T>(__fsub_rn(__fmul_rn(x0, a.x), __fmul_rn(x1, a.y)));
      p[i + half] = from_f32<T>(__fadd_rn(__fmul_rn(x1, a.x), __fmul_rn(x0, a.y)));
    }
  }
}

template <typename T>
int launch_rope_t(void* qkv, const int64_t* positions, int64_t tokens, int heads, int head_dim, int rotary_dim,
                  float base, float yarn, cudaStream_t stream) {
  constexpr int V = VecOf<T>::N;
  const int half = rotary_dim / 2;
  RopeFreq freq;
  for (int i = 0; i < half; ++i) {
    // reference/reference.cpp:44: std::pow(base, -2.0f * float(i) / float(rotary_dim)) * yarn_factor
    volatile float e = -2.0f * static_cast<float>(i) / static_cast<float>(rotary_dim);
    volatile float pw = powf(base, e);
    freq.f[i] = pw * yarn;
  }
  for (int i = half; i < kRopeMaxHalf; ++i) freq.f[i] = 0.0f;
  const bool vec = (reinterpret_cast<uintptr_t>(qkv) & 15u) == 0 && half % V == 0 &&
                   (static_cast<int64_t>(head_dim) * sizeof(T)) % 16 == 0;
  // at most four work items per thread and CTA (the vector kernel holds that many in registers);
  // a token's table is computed once per CTA
  const int items_per_head = vec ? half / V : half;
  int hpc = 4 * kRopeThreads / items_per_head;
  if (hpc > heads) hpc = heads;
  if (hpc < 1) hpc = 1;
  const int chunks = (heads + hpc - 1) / hpc;
  if (chunks > 65535) return INFEROP_ERR_LIMIT;
  const dim3 grid(static_cast<unsigned>(tokens), static_cast<unsigned>(chunks));
  if (vec) {
    rope_kernel<T, true><<<grid, kRopeThreads, 0, stream>>>(static_cast<T*>(qkv), positions, heads, head_dim,
                                                            rotary_dim, hpc, freq);
  } else {
    rope_kernel<T, false><<<grid, kRopeThreads, 0, stream>>>(static_cast<T*>(qkv), positions, heads, head_dim,
                                                             rotary_dim, hpc, freq);
  }
  return check_launch();
}

}  // namespace

int launch_rmsnorm(void* out, void* residual, const void* in, const void* weight, int32_t dt, int64_t rows,
                   int64_t cols, float eps, cudaStream_t stream) {
  const bool add = residual != nullptr;
  switch (dt) {
    case 0: return add ? launch_rmsnorm_t<float, true>(out, residual, in, weight, rows, cols, eps, stream)
                       : launch_rmsnorm_t<float, false>(out, nullptr, in, weight, rows, cols, eps, stream);
    case 1: return add ? launch_rmsnorm_t<__half, true>(out, residual, in, weight, rows, cols, eps, stream)
                       : launch_rmsnorm_t<__half, false>(out, nullptr, in, weight, rows, cols, eps, stream);
    case 2: return add ? launch_rmsnorm_t<__nv_bfloat16, true>(out, residual, in, weight, rows, cols, eps, stream)
                       : launch_rmsnorm_t<__nv_bfloat16, false>(out, nullptr, in, weight, rows, cols, eps, stream);
    default: return INFEROP_ERR_DTYPE;
  }
}

int launch_rmsnorm_quant(void* q, void* scales, void* residual, const void* in, const void* weight, int32_t dt,
                         int64_t rows, int64_t cols, float eps, cudaStream_t stream) {
  if (cols % 128 != 0 || cols / 16 > static_cast<int64_t>(kNormThreads) * kMaxPieces) return INFEROP_ERR_SHAPE;
  const bool add = residual != nullptr;
  switch (dt) {
    case 1: return add ? launch_rmsnorm16<__half, true, true>(q, scales, residual, in, weight, rows, cols, eps, stream)
                       : launch_rmsnorm16<__half, false, true>(q, scales, nullptr, in, weight, rows, cols, eps, stream);
    case 2: return add ? launch_rmsnorm16<__nv_bfloat16, true, true>(q, scales, residual, in, weight, rows, cols, eps, stream)
                       : launch_rmsnorm16<__nv_bfloat16, false, true>(q, scales, nullptr, in, weight, rows, cols, eps, stream);
    default: return INFEROP_ERR_DTYPE;
  }
}

int launch_rope_neox(void* qkv, const int64_t* positions, int32_t dt, int64_t tokens, int heads, int head_dim,
                     int rotary_dim, float base, float yarn, cudaStream_t stream) {
  if (rotary_dim / 2 > kRopeMaxHalf) return INFEROP_ERR_LIMIT;
  if (tokens > 0x7FFFFFFFLL) return INFEROP_ERR_LIMIT;
  switch (dt) {
    case 0: return launch_rope_t<float>(qkv, positions, tokens, heads, head_dim, rotary_dim, base, yarn, stream);
    case 1: return launch_rope_t<__half>(qkv, positions, tokens, heads, head_dim, rotary_dim, base, yarn, stream);
    case 2: return launch_rope_t<__nv_bfloat16>(qkv, positions, tokens, heads, head_dim, rotary_dim, base, yarn, stream);
    default: return INFEROP_ERR_DTYPE;
  }
}

}  // namespace ib200
