// Per-token-group FP8 (E4M3) quantisation and its inverse for sm_100a.
//
// Replaces the reference's kernels/quant.cu (quant_fp8_kernel :16-35,
// dequant_fp8_kernel :37-46) and must reproduce reference/reference.cpp:65-80
// bit for bit:
//     amax  = max |x| over the group (NaN never wins)
//     scale = amax * fl(1/448), exactly 1 for an all-zero group
//     q     = e4m3_rn_sat(x / scale)       <- IEEE fp32 division
//
// Layout.  With cols % 128 == 0 and row-major storage, group g of the
// flattened [rows * cols/128] group index space starts at element g*128 of x
// and q and at scales[g]; the kernel therefore treats the tensor as a flat
// array of 128-element groups.  A lane owns 32 bytes of a group, one 256-bit load: eight lanes per
// group of a 16-bit type, sixteen of fp32.  The absmax is reduced by xor-shuffles among them, each
// lane converts its values with cvt.rn.satfinite.e4m3x2.f32 and writes them with one store.
// Every thread has kUnroll groups in flight, and a CTA is done after them: the hardware keeps the SMs
// full of loads as CTAs come and go.
//
// HBM traffic per element (16-bit): 2 B read + 1 B written + 4/128 B of scale = 3.03 B.  Measured, bf16, cold,
// graph replay, 16 bytes per lane in a persistent loop -> now: 4096 x 7168 17.5 -> 14.6 us (6.1 TB/s), 16384 x 7168
// 62.0 -> 51.5, 16384 x 18432 153 -> 129 (7.1 TB/s), 1000 x 7168 6.4 -> 5.2, 64 x 7168 2.0 -> 1.7.  The old form was bound by
// the instructions that all lanes of a group repeat, and by its second wave.  32 bytes in a persistent loop: 15.4, 55, 140; a
// loop with the next loads in flight: 22, 84, 214; one or four groups per thread: 15.1, 54.8, 137 and 14.9, 52.4, 131.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "inferop/fp8.h"
#include "internal.h"
#include "quant_math.cuh"

namespace ib200 {
namespace {

constexpr int kThreads = 256;
constexpr int kUnroll = 2;    // groups in flight per lane
// resident CTAs per SM the register budget allows.  At six the 16-bit forms spill (bf16 4-12 bytes, fp16 12-44), at four not;
// bf16 4096 x 7168 / 16384 x 18432 / 1000 x 7168, us: six 16.9 / 133.7 / 6.4, five 16.9 / 137.5 / 6.2, four 17.2 / 140.9 / 5.9;
// fp16: six 17.6 / 135.9 / 6.9, five 16.4 / 132.6 / 6.2, four 16.7 / 138.0 / 6.0; fp32: six 26.1 / 219.8 / 8.9, five 28.4 / 233.2 / 9.0
constexpr int kMinCtas = 6;

// kWide: x 32-byte and (16-bit types) q 16-byte aligned
template <typename T, bool kWide>
__global__ void __launch_bounds__(kThreads, kMinCtas)
quant128_kernel(uint8_t* __restrict__ q, float* __restrict__ scales, const T* __restrict__ x,
                int64_t groups) {
  // a GEMM queued behind this kernel may begin its preamble (barriers, tensor memory, weight
  // prefetch); it waits for this kernel's completion before it reads q or scales
  pdl_launch_dependents();
  // launched with programmatic stream serialisation this kernel may itself have started under the
  // tail of the kernel before it (a GEMM that still reads q and scales, or the producer of x):
  // nothing is read or written before that kernel has completed (a no-op after an ordinary launch)
  pdl_wait();
  constexpr int kElems = 32 / sizeof(T);   // per lane
  constexpr int kLanes = 128 / kElems;     // of a group
  constexpr int kStep = kThreads / kLanes; // groups of a CTA per unrolled step
  const int sub = threadIdx.x % kLanes;
  const int64_t first = static_cast<int64_t>(blockIdx.x) * (kStep * kUnroll) + threadIdx.x / kLanes;
  const int left = static_cast<int>(groups - first < kStep * kUnroll ? groups - first : kStep * kUnroll);   // from `first` on
  x += first * 128 + sub * kElems;
  q += first * 128 + sub * kElems;
  scales += first;
  Words8 v[kUnroll];
#pragma unroll
  for (int u = 0; u < kUnroll; ++u) v[u] = u * kStep < left ? load_nc32<kWide>(x + u * kStep * 128) : zero_words();
#pragma unroll
  for (int u = 0; u < kUnroll; ++u) {   // (all 32 lanes take part in the shuffles)
    float f[8], amax;
    if constexpr (sizeof(T) == 2) {
      amax = absmax16<T>(v[u]);
    } else {
      amax = 0.0f;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        f[i] = __uint_as_float(v[u].w[i]);
        amax = fmaxf(amax, fabsf(f[i]));
      }
    }
#pragma unroll
    for (int o = kLanes / 2; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, o));
    const float scale = group_scale(amax);
    if (u * kStep < left) {
      uint8_t* dst = q + u * kStep * 128;
      // 16-bit inputs whose group maximum is far from the ends of the fp32 range divide through the reciprocal, two
      // elements per instruction; everything else uses IEEE division
      if constexpr (sizeof(T) == 2) store16<kWide>(dst, quantise16<T>(v[u], amax, scale));
      else *reinterpret_cast<uint2*>(dst) = quantise8<false>(f, scale, 0.0f);
      if (sub == 0) scales[u * kStep] = scale;
    }
  }
}

template <typename T>
cudaError_t launch_quant128(const cudaLaunchConfig_t& cfg, bool wide, uint8_t* q, float* scales, const void* x, int64_t groups) {
  const T* xt = static_cast<const T*>(x);
  return wide ? cudaLaunchKernelEx(&cfg, quant128_kernel<T, true>, q, scales, xt, groups)
              : cudaLaunchKernelEx(&cfg, quant128_kernel<T, false>, q, scales, xt, groups);
}

// Any other group size: one warp per group, strided lanes.  Correctness path
// only; the library's hot path always uses 128.
template <typename T>
__device__ __forceinline__ float widen(T v);
template <>
__device__ __forceinline__ float widen(float v) { return v; }
template <>
__device__ __forceinline__ float widen(__half v) { return __half2float(v); }
template <>
__device__ __forceinline__ float widen(__nv_bfloat16 v) { return __bfloat162float(v); }

template <typename T>
__global__ void __launch_bounds__(kThreads)
quant_any_kernel(uint8_t* __restrict__ q, float* __restrict__ scales, const T* __restrict__ x,
                 int64_t groups, int gs) {
  const int lane = threadIdx.x & 31;
  const int64_t warp = (static_cast<int64_t>(blockIdx.x) * kThreads + threadIdx.x) >> 5;
  const int64_t warps = (static_cast<int64_t>(gridDim.x) * kThreads) >> 5;
  for (int64_t g = warp; g < groups; g += warps) {
    const T* gx = x + g * gs;
    float amax = 0.0f;
    for (int i = lane; i < gs; i += 32) amax = fmaxf(amax, fabsf(widen(gx[i])));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, o));
    const float scale = group_scale(amax);
    if (lane == 0) scales[g] = scale;
    for (int i = lane; i < gs; i += 32) {
      const float xv = widen(gx[i]);
      const float r = __fdiv_rn(xv, scale);
      uint32_t b = cvt2(r, 0.0f) & 0xFFu;
      if (r != r) b = nan_byte(xv);
      q[g * gs + i] = static_cast<uint8_t>(b);
    }
  }
}

// E4M3 byte -> fp32, exact (hardware e4m3x2 -> f16x2 conversion, then widen).
__device__ __forceinline__ float decode_e4m3(uint8_t b) {
  const __half_raw h = __nv_cvt_fp8_to_halfraw(b, __NV_E4M3);
  return __half2float(*reinterpret_cast<const __half*>(&h));
}
template <typename T>
__device__ __forceinline__ T narrow(float v);
template <>
__device__ __forceinline__ float narrow(float v) { return v; }
template <>
__device__ __forceinline__ __half narrow(float v) { return __float2half_rn(v); }
template <>
__device__ __forceinline__ __nv_bfloat16 narrow(float v) { return __float2bfloat16_rn(v); }

template <typename T>
__global__ void __launch_bounds__(kThreads)
dequant_kernel(T* __restrict__ x, const uint8_t* __restrict__ q, const float* __restrict__ scales,
               int64_t total, int gs) {
  const int64_t stride = static_cast<int64_t>(gridDim.x) * kThreads;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * kThreads + threadIdx.x; i < total;
       i += stride) {
    x[i] = narrow<T>(__fmul_rn(decode_e4m3(q[i]), __ldg(scales + i / gs)));
  }
}

// Self-test: hardware converter against the software encoder of
// include/inferop/fp8.h on every fp32 bit pattern in [lo, hi).  NaN inputs are
// counted separately (the hardware drops their sign; quantise8 restores it).
__global__ void __launch_bounds__(kThreads)
cvt_selftest_kernel(uint64_t lo, uint64_t hi, unsigned long long* counts) {
  unsigned long long bad = 0, bad_nan = 0;
  const uint64_t stride = static_cast<uint64_t>(gridDim.x) * kThreads;
  for (uint64_t u = lo + static_cast<uint64_t>(blockIdx.x) * kThreads + threadIdx.x; u < hi;
       u += stride) {
    const float f = __uint_as_float(static_cast<uint32_t>(u));
    const uint32_t hw = cvt2(f, 0.0f) & 0xFFu;
    const uint32_t sw = inferop::fp8::float_to_e4m3_rn_sat(f);
    if (hw != sw) {
      if (f != f) ++bad_nan; else ++bad;
    }
  }
  if (bad) atomicAdd(&counts[0], bad);
  if (bad_nan) atomicAdd(&counts[1], bad_nan);
}

// Self-test of div_by_rcp: for every finite positive 16-bit group maximum (bf16 when
// is_bf16, else fp16) that takes the fast path, and every 16-bit element value no larger in
// magnitude, the E4M3 byte from the reciprocal path must equal the byte from __fdiv_rn.
__global__ void __launch_bounds__(kThreads)
div_selftest_kernel(int is_bf16, unsigned long long* counts) {
  unsigned long long bad = 0, pairs = 0;
  for (uint32_t a = blockIdx.x; a < 0x8000u; a += gridDim.x) {   // a == 0: the all-zero group
    const float amax = is_bf16 ? __uint_as_float(a << 16)
                               : __half2float(__ushort_as_half(static_cast<unsigned short>(a)));
    if (!(amax == amax) || !fast_div_ok(amax)) continue;  // NaN / Inf / out of the fast range
    const float scale = group_scale(amax);
    const float rcp = __frcp_rn(scale);
    for (uint32_t xb = threadIdx.x; xb < 0x10000u; xb += kThreads) {
      const float x = is_bf16 ? __uint_as_float(xb << 16)
                              : __half2float(__ushort_as_half(static_cast<unsigned short>(xb)));
      if (!(fabsf(x) <= amax)) continue;
      ++pairs;
      // the kernels' fast path, element 0 of the eight (the other seven are zeros)
      const uint4 raw = make_uint4(xb, 0u, 0u, 0u);
      const float f8[8] = {x, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
      const uint32_t fast = quantise8_fast16(raw, f8, scale, rcp).x & 0xFFu;
      const uint32_t slow = cvt2(__fdiv_rn(x, scale), 0.0f) & 0xFFu;
      if (fast != slow) {
        ++bad;
        counts[2] = (static_cast<unsigned long long>(a) << 32) | xb;  // one example: group maximum, element
      }
    }
  }
  if (bad) atomicAdd(&counts[0], bad);
  atomicAdd(&counts[1], pairs);
}

int grid_for(int64_t work_items_per_thread_block, int sms) {
  int64_t want = work_items_per_thread_block;
  int64_t cap = static_cast<int64_t>(sms) * 8;  // 8 resident 256-thread CTAs per SM
  if (want > cap) want = cap;
  if (want < 1) want = 1;
  return static_cast<int>(want);
}

}  // namespace

int launch_quant(void* q, void* scales, const void* x, int32_t dt, int64_t rows, int64_t cols,
                 int32_t gs, cudaStream_t stream, int sms) {
  const int64_t groups = rows * (cols / gs);
  uint8_t* qp = static_cast<uint8_t*>(q);
  float* sp = static_cast<float*>(scales);
  const bool vec_ok = gs == 128 && (reinterpret_cast<uintptr_t>(x) % 16 == 0) &&
                      (reinterpret_cast<uintptr_t>(q) % 8 == 0);
  if (vec_ok) {
    const int64_t groups_per_block = kThreads / (dt == 0 ? 16 : 8) * kUnroll;
    const int64_t blocks = groups > 0 ? (groups + groups_per_block - 1) / groups_per_block : 1;
    if (blocks > 0x7FFFFFFF) return INFEROP_ERR_LIMIT;   // (more than 2^37 groups)
    const bool wide = reinterpret_cast<uintptr_t>(x) % 32 == 0 && reinterpret_cast<uintptr_t>(q) % 16 == 0;
    // programmatic stream serialisation: the launch itself may overlap the tail of the kernel
    // queued before it when that kernel lets its dependents start early (the small-M GEMM does)
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(blocks));
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = options().quant_pdl ? 1 : 0;
    cudaError_t e;
    switch (dt) {
      case 0: e = launch_quant128<float>(cfg, wide, qp, sp, x, groups); break;
      case 1: e = launch_quant128<__half>(cfg, wide, qp, sp, x, groups); break;
      case 2: e = launch_quant128<__nv_bfloat16>(cfg, wide, qp, sp, x, groups); break;
      default: return INFEROP_ERR_DTYPE;
    }
    if (e != cudaSuccess) return note_cuda_error(e);
  } else {
    const int64_t groups_per_block = kThreads / 32;
    const int grid = grid_for((groups + groups_per_block - 1) / groups_per_block, sms);
    switch (dt) {
      case 0: quant_any_kernel<float><<<grid, kThreads, 0, stream>>>(qp, sp, static_cast<const float*>(x), groups, gs); break;
      case 1: quant_any_kernel<__half><<<grid, kThreads, 0, stream>>>(qp, sp, static_cast<const __half*>(x), groups, gs); break;
      case 2: quant_any_kernel<__nv_bfloat16><<<grid, kThreads, 0, stream>>>(qp, sp, static_cast<const __nv_bfloat16*>(x), groups, gs); break;
      default: return INFEROP_ERR_DTYPE;
    }
  }
  return check_launch();
}

int run_cvt_selftest(uint64_t lo, uint64_t hi, uint64_t* out2, int sms) {
  unsigned long long* d = nullptr;
  cudaError_t e = cudaMalloc(&d, 16);
  if (e != cudaSuccess) return note_cuda_error(e);
  cudaMemset(d, 0, 16);
  cvt_selftest_kernel<<<sms * 8, kThreads>>>(lo, hi, d);
  e = cudaMemcpy(out2, d, 16, cudaMemcpyDeviceToHost);
  cudaFree(d);
  return e == cudaSuccess ? INFEROP_OK : note_cuda_error(e);
}

int run_div_selftest(int is_bf16, uint64_t* out3, int sms) {
  unsigned long long* d = nullptr;
  cudaError_t e = cudaMalloc(&d, 24);
  if (e != cudaSuccess) return note_cuda_error(e);
  cudaMemset(d, 0, 24);
  div_selftest_kernel<<<sms * 8, kThreads>>>(is_bf16, d);
  e = cudaMemcpy(out3, d, 24, cudaMemcpyDeviceToHost);
  cudaFree(d);
  return e == cudaSuccess ? INFEROP_OK : note_cuda_error(e);
}

int launch_dequant(void* x, int32_t dt, const void* q, const void* scales, int64_t rows,
                   int64_t cols, int32_t gs, cudaStream_t stream, int sms) {
  const int64_t total = rows * cols;
  const int grid = grid_for((total + kThreads - 1) / kThreads, sms);
  const uint8_t* qp = static_cast<const uint8_t*>(q);
  const float* sp = static_cast<const float*>(scales);
  switch (dt) {
    case 0: dequant_kernel<float><<<grid, kThreads, 0, stream>>>(static_cast<float*>(x), qp, sp, total, gs); break;
    case 1: dequant_kernel<__half><<<grid, kThreads, 0, stream>>>(static_cast<__half*>(x), qp, sp, total, gs); break;
    case 2: dequant_kernel<__nv_bfloat16><<<grid, kThreads, 0, stream>>>(static_cast<__nv_bfloat16*>(x), qp, sp, total, gs); break;
    default: return INFEROP_ERR_DTYPE;
  }
  return check_launch();
}

}  // namespace ib200
