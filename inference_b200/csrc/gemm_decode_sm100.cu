// Small-M ("decode") variant of the blockwise-FP8 W8A8 GEMM for sm_100a.
//
// Same arithmetic contract as gemm_sm100.cu (reference kernels/gemm/w8a8_block_fp8.cu:100-114,
// reference/reference.cpp:93-110), different mapping.  With a handful of tokens the work is a
// pure stream of the weight matrix from HBM, so:
//   * operands are swapped: a 128-row weight tile is the M side of tcgen05.mma (UMMA M=128)
//     and the tokens, padded to MP in {16, 32, 64, 128}, are its N side.  The accumulator of one
//     K block is a [128 weight rows] x [MP tokens] slice of tensor memory; 512 / MP (at most 8)
//     slices are in flight, so the MMA -> promotion -> MMA round trip never limits the stream.
//   * work is dealt in whole pieces: with at least as many weight tiles as CTAs every CTA takes
//     a contiguous run of whole tiles; with fewer, every tile's K range is cut into `splits`
//     equal parts, one CTA each (split-K).  A CTA of a split tile writes an fp32 partial to a
//     workspace; the last CTA to finish the tile adds the parts in a fixed order
//     (deterministic) and writes the output.  HBM, not the SM count, bounds this kernel, so
//     leaving a few SMs idle costs nothing, while ragged pieces would cost a second partial
//     flush per CTA.
//
// CTA layout (256 threads, one CTA per SM):
//   warp 0  allocates / frees tensor memory; one thread is the TMA producer: weight tile
//           [128 x 128 B] + token tile [MP x 128 B] per K block into a deep ring
//   warps 1, 3  MMA issuers (warp-uniform loops, one elected lane each, alternating units):
//           4 x tcgen05.mma (M=128, N=MP, K=32) per unit
//   warp 2  scale warp: writes sa[m, kb] * sb[tile, kb] for the MP tokens of each unit to a
//           small shared ring, one vector per TMEM slice
//   warps 4-7  promotion + epilogue: thread = one weight row (= output column), MP accumulators
//
// HBM traffic (algorithmic): N*K weight bytes + M*K token bytes + scales + 2*M*N output bytes;
// split tiles add 2 x 4*128*MP bytes of workspace traffic per extra segment.
//
// Every wait is bounded (ptx.cuh: mbar_wait); see gemm_sm100.cu for the wind-down rules.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <mutex>
#include <type_traits>

#include "internal.h"
#include "quant_math.cuh"

namespace ib200 {
namespace {

constexpr int TN = 128;   // weight rows per tile (UMMA M)
constexpr int BK = 128;
constexpr int kThreads = 256;
constexpr int kFusedThreads = 384;   // fused prologue: four more warps that quantise the token tile
constexpr int kBytesW = TN * BK;
constexpr uint32_t kAhead = 6;       // K blocks of weights per CTA that are asked into L2 before the wait for the kernel before
constexpr int kMaxStages = 12;       // barrier slots of the ring
constexpr int kFusedMaxSmem = 227 * 1024;   // fused prologue: dynamic shared memory the launcher may ask for
constexpr int kMaxSlots = 16;        // fused prologue: barrier slots of the token-tile ring

template <int MP>
struct DCfg {
  static constexpr int kBytesA = MP * BK;
  static constexpr int kStageBytes = kBytesW + kBytesA;
  // (twelve stages of 18 KiB fit too and measured 3 % slower than ten)
  static constexpr int kStages = (200 * 1024 / kStageBytes) < 10 ? (200 * 1024 / kStageBytes) : 10;
  static_assert(kStages % 2 == 0, "the two MMA issuer warps alternate units: a stage must always belong to the same warp");
  static_assert(kStages % 2 == 0, "the two MMA issuer warps alternate units: a stage must always belong to the same warp");
  static constexpr int kBufs = (512 / MP) < 8 ? (512 / MP) : 8;
  static constexpr int kTmemCols = (kBufs * MP) < 32 ? 32 : (kBufs * MP);
  static constexpr int kScaleBytes = kBufs * MP * 4;
  static constexpr int kBarrierBytes = 512;
  static constexpr int kSmemBytes = kStages * kStageBytes + kScaleBytes + kBarrierBytes + 1024;
};

struct DecodeParams {
  const float* a_scales;   // [M, KB]
  const void* a_src;       // fused prologue only: unquantised activations [M, K] (bf16 / fp16)
  const float* b_scales;   // [ceil(N/128), KB]
  // Output: the [M, N] result goes to columns [col0, col0 + N) of n_dst row-major buffers with
  // row pitch ldc elements.  A plain call has one destination (c, ldc = N, col0 = 0); the
  // all-gather form lists every rank's buffer (peer-mapped addresses, plain stores).
  void* dst[8];
  int n_dst, ldc, col0;
  float* workspace;        // [gridDim.x][2][MP][128] fp32 partials (slot 0: the CTA's first tile, slot 1: its last)
  int splits;              // 0: units dealt evenly (below); else K parts per tile (1 = runs of whole tiles)
  int stages, a_slots;     // fused prologue: depth of the weight ring and of the token-tile ring
  int* counters;           // [n_tiles], zero between launches
  int m, n, kb, n_tiles;
  long long units;         // n_tiles * kb
  int no_loads;            // test hook: the producer issues no load
  int trigger;    // let kernels queued behind this one with programmatic stream serialisation start early
  DeviceStatus* status;
};

enum : uint32_t {
  kSiteDProducerEmpty = 0x111,
  kSiteDMmaFull = 0x211,
  kSiteDMmaTmemEmpty = 0x212,
  kSiteDScaleEmpty = 0x411,
  kSiteDPromoFull = 0x311,
  kSiteDPromoScale = 0x312,
  kSiteDQuantEmpty = 0x511,
  kSiteDQuantTmem = 0x512,
};

template <typename OutT>
__device__ __forceinline__ OutT cvt_out(float v);

template <>
__device__ __forceinline__ float cvt_out<float>(float v) { return v; }
template <>
__device__ __forceinline__ __half cvt_out<__half>(float v) { return __float2half_rn(v); }
template <>
__device__ __forceinline__ __nv_bfloat16 cvt_out<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }

// Column gn of the result (MP values, one per token, in registers) to every destination.  The
// destination loop is the outer one so that the token loop stays fully unrolled over registers;
// with the usual single destination it runs once.
template <int MP, typename OutT>
__device__ __forceinline__ void store_column(const DecodeParams& p, int gn, const float (&v)[MP]) {
  for (int d = 0; d < p.n_dst; ++d) {
    OutT* col = static_cast<OutT*>(p.dst[d]) + p.col0 + gn;
#pragma unroll
    for (int m = 0; m < MP; ++m)
      if (m < p.m) col[static_cast<int64_t>(m) * p.ldc] = cvt_out<OutT>(v[m]);
  }
}

template <int N>
__device__ __forceinline__ void tmem_ld_cols(uint32_t taddr, uint32_t (&r)[N]);
template <>
__device__ __forceinline__ void tmem_ld_cols<16>(uint32_t taddr, uint32_t (&r)[16]) { tmem_ld_32x16(taddr, r); }
template <>
__device__ __forceinline__ void tmem_ld_cols<32>(uint32_t taddr, uint32_t (&r)[32]) { tmem_ld_32x32(taddr, r); }

template <int N>
__device__ __forceinline__ void tmem_wait_pin(uint32_t (&r)[N]) {
  tmem_ld_wait();
#pragma unroll
  for (int i = 0; i < N; ++i) asm volatile("" : "+r"(r[i])::"memory");
}

// 8 consecutive 16-bit activations -> 8 floats
template <typename AT>
__device__ __forceinline__ void unpack8(const uint4& raw, float (&f)[8]);
template <>
__device__ __forceinline__ void unpack8<__nv_bfloat16>(const uint4& raw, float (&f)[8]) {
  const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    f[2 * i] = __uint_as_float(w[i] << 16);
    f[2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u);
  }
}
template <>
__device__ __forceinline__ void unpack8<__half>(const uint4& raw, float (&f)[8]) {
  const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 t = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}
template <>
__device__ __forceinline__ void unpack8<void>(const uint4&, float (&)[8]) {}

// AT = void: the token tile arrives quantised through TMA and a scale warp prepares the scale
// vectors.  AT = bf16 / fp16 (the fused prologue): warps 8-11 quantise the token tile of every
// unit themselves, straight from the unquantised activations, into a ring of their own in
// shared memory (swizzled [MP x 128 B] tiles, the layout a TMA load would have produced, plus
// the group scales), running ahead of the weight stream by up to the ring's depth; the producer
// streams weights only.  The stand-alone quantisation kernel, its launch and its q / scales
// round trip through HBM disappear.
template <int MP, typename OutT, typename AT>
__global__ void __launch_bounds__(std::is_same<AT, void>::value ? kThreads : kFusedThreads, 1)
w8a8_decode_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_a,
                   const DecodeParams p) {
  using C = DCfg<MP>;
  constexpr bool kFused = !std::is_same<AT, void>::value;
  constexpr int kQuantWarps = 4;
  constexpr int CH = (MP < 32) ? MP : 32;   // columns per tensor-memory load
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~uintptr_t(1023));
  // ring stages: weight tile + token tile; fused: weight tile only, depth chosen by the launcher
  const uint32_t nst = kFused ? static_cast<uint32_t>(p.stages) : static_cast<uint32_t>(C::kStages);
  constexpr uint32_t kStride = kFused ? kBytesW : C::kStageBytes;
  const uint32_t a_slots = kFused ? static_cast<uint32_t>(p.a_slots) : 0u;  // fused: ring of quantised token tiles (a power of two)
  const uint32_t a_mask = a_slots - 1u, a_shift = 31u - static_cast<uint32_t>(__clz(static_cast<int>(a_slots | 1u)));
  uint8_t* a_res = smem + nst * kStride;                                    // [a_slots][MP x 128 B], swizzled
  float* sa_res = reinterpret_cast<float*>(a_res + a_slots * (MP * BK));     // [a_slots][MP] group scales
  float* sv = sa_res + a_slots * MP;                                         // [kBufs][MP]
  uint64_t* bars = reinterpret_cast<uint64_t*>(reinterpret_cast<uint8_t*>(sv) + C::kScaleBytes);
  uint64_t* full = bars;                         // [kMaxStages] TMA -> MMA
  uint64_t* empty = full + kMaxStages;           // [kMaxStages] MMA -> TMA
  uint64_t* tmem_full = empty + kMaxStages;      // [kBufs]   MMA -> promotion
  uint64_t* tmem_empty = tmem_full + C::kBufs;   // [kBufs]   promotion -> MMA, scale warp
  uint64_t* sv_full = tmem_empty + C::kBufs;     // [kBufs]   scale warp -> promotion
  uint64_t* a_full = sv_full + C::kBufs;         // [a_slots] fused: quantising warps -> MMA, scale warp
  uint64_t* a_empty = a_full + (kFused ? kMaxSlots : 0);   // [a_slots] fused: MMA + scale warp -> quantising warps
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(a_empty + (kFused ? kMaxSlots : 0));
  volatile uint32_t* abort_flag = tmem_slot + 1;
  volatile uint32_t* last_flag = tmem_slot + 2;

  const int warp = __shfl_sync(0xFFFFFFFFu, static_cast<int>(threadIdx.x >> 5), 0);
  const int lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (uint32_t s = 0; s < nst; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (uint32_t j = 0; j < a_slots; ++j) {
      mbar_init(&a_full[j], 1);
      mbar_init(&a_empty[j], 2);   // the unit's MMAs have read the tile, the scale warp its scales
    }
    for (int b = 0; b < C::kBufs; ++b) {
      mbar_init(&tmem_full[b], 1);
      mbar_init(&tmem_empty[b], 4);
      mbar_init(&sv_full[b], 1);
    }
    *abort_flag = 0u;
    mbar_init_fence();
    tma_prefetch_desc(&map_w);
    if (!kFused) tma_prefetch_desc(&map_a);
  }
  if (warp == 0) {
    tmem_alloc(tmem_slot, C::kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = __shfl_sync(0xFFFFFFFFu, *tmem_slot, 0);
  // A kernel queued behind this one with programmatic stream serialisation (the quantiser of the
  // next step, and behind it the next GEMM) may be launched from now on: it takes SMs as this
  // grid's CTAs leave them and waits for this grid's completion before it touches memory.
  if (p.trigger) pdl_launch_dependents();

  // This CTA's piece: tiles [t_first, ...) from K block kb_first, `count` units in all.  A unit
  // is one (weight tile, K block) pair = 16 KiB of weights.  Default: the n_tiles * kb units are
  // dealt evenly, CTA c takes units [c U / G, (c + 1) U / G), so every SM streams the same number
  // of bytes whatever the tile count; a piece may start and end inside a tile, and the K parts of
  // a tile are then added in CTA order by the last CTA to finish (deterministic).
  int t_first, kb_first;
  uint32_t count;
  if (p.splits == 0) {
    const long long g = gridDim.x, c = blockIdx.x;
    const long long u0 = c * p.units / g, u1 = (c + 1) * p.units / g;
    t_first = static_cast<int>(u0 / p.kb);
    kb_first = static_cast<int>(u0 - static_cast<long long>(t_first) * p.kb);
    count = static_cast<uint32_t>(u1 - u0);
  } else if (p.splits == 1) {
    const long long g = gridDim.x, c = blockIdx.x;
    t_first = static_cast<int>(c * p.n_tiles / g);
    kb_first = 0;
    count = static_cast<uint32_t>(((c + 1) * p.n_tiles / g - t_first) * p.kb);
  } else {
    const int part = blockIdx.x % p.splits;
    t_first = blockIdx.x / p.splits;
    kb_first = part * p.kb / p.splits;
    count = static_cast<uint32_t>((part + 1) * p.kb / p.splits - kb_first);
  }

  if (warp == 0) {
    // ------------------------------ TMA producer (warp-uniform loop) ------
    // The kernel may have started under the one queued before it (programmatic dependent launch), which may have
    // written anything that this one reads, the weights too: nothing is loaded before the wait (a no-op after an
    // ordinary launch).  The first weight tiles are asked into L2 meanwhile, where a later write reaches them.  Quantiser +
    // GEMM in a graph, cold weights, us, asking for 0 / 6 / 10 / 16 blocks: 1 x 18432 x 7168 26.0 / 25.6 / 25.9 / 25.9, 3 x 4096
    // x 7168 10.7 / 10.3 / 10.5 / 10.7, 16 x 24576 x 1536 13.5 / 12.7 / 12.7 / 12.7 (loaded into shared memory, which a write
    // by the kernel before would not reach: 25.3, 9.6, 11.5).
    int t = t_first, kb = kb_first;
    uint32_t armed = 0;
    bool ok = true;
    if (!p.no_loads) {   // (test hook: nothing is ever loaded, so every other role's wait runs out)
      int th = t, kh = kb;
      for (uint32_t i = 0; i < count && i < kAhead; ++i) {
        if (elect_one()) tma_prefetch_2d(&map_w, kh * BK, th * TN);
        __syncwarp();
        if (++kh == p.kb) {
          kh = 0;
          ++th;
        }
      }
      pdl_wait();
    }
    for (uint32_t i = 0; i < count && !p.no_loads; ++i) {
      const uint32_t stage = i % nst;
      const uint32_t phase = (i / nst) & 1u;
      if (!mbar_wait(&empty[stage], phase ^ 1u, abort_flag, p.status, kSiteDProducerEmpty)) {
        ok = false;
        break;
      }
      __syncwarp();
      uint8_t* dst = smem + stage * kStride;
      if (elect_one()) {
        mbar_arrive_expect_tx(&full[stage], kStride);
        tma_load_2d(dst, &map_w, &full[stage], kb * BK, t * TN);
        if (!kFused) tma_load_2d(dst + kBytesW, &map_a, &full[stage], kb * BK, 0);
      }
      __syncwarp();
      armed = i + 1;
      if (++kb == p.kb) {
        kb = 0;
        ++t;
      }
    }
    if (!ok && lane == 0) {
      // wind-down: let the copies this warp started land before the CTA exits
      const uint32_t lo = armed > nst ? armed - nst : 0u;
      for (uint32_t i = lo; i < armed; ++i) {
        const long long t0 = clock64();
        while (!mbar_test_wait(&full[i % nst], (i / nst) & 1u)) {
          if (clock64() - t0 > kWaitBudgetCycles) break;
        }
      }
    }
  } else if (warp == 1 || warp == 3) {
    // ------------------------------ MMA issuers (warp-uniform) ------------
    // warp 1 issues the even units of the range, warp 3 the odd ones: waiting, building
    // descriptors, 4 MMAs and 2 commits cost one thread about 650 cycles per unit, more than
    // the time the unit's 18 KiB take to arrive from HBM
    constexpr uint32_t idesc = umma_idesc_e4m3_f32(TN, MP);
    const uint32_t smem_base = smem_u32(smem);
    for (uint32_t i = (warp == 3) ? 1u : 0u; i < count; i += 2) {
      const uint32_t stage = i % nst;
      const uint32_t phase = (i / nst) & 1u;
      const uint32_t buf = i % C::kBufs;
      const uint32_t use = i / C::kBufs;
      const uint32_t slot = kFused ? (i & a_mask) : 0u;   // fused: the unit's slot in the token-tile ring
      if (!mbar_wait(&full[stage], phase, abort_flag, p.status, kSiteDMmaFull)) break;
      if (kFused && !mbar_wait(&a_full[slot], (i >> a_shift) & 1u, abort_flag, p.status, kSiteDQuantEmpty)) break;
      if (!mbar_wait(&tmem_empty[buf], (use & 1u) ^ 1u, abort_flag, p.status, kSiteDMmaTmemEmpty)) break;
      __syncwarp();
      tc_fence_after_sync();
      const uint32_t w_addr = smem_base + stage * kStride;
      const uint64_t dw = umma_desc_k_sw128(w_addr);
      const uint64_t da = umma_desc_k_sw128(kFused ? smem_u32(a_res) + slot * (MP * BK) : w_addr + kBytesW);
      const uint32_t d_tmem = tmem_base + buf * MP;
      if (elect_one()) {
#pragma unroll
        for (int k4 = 0; k4 < BK / 32; ++k4) {
          umma_f8_ss(d_tmem, dw + 2u * k4, da + 2u * k4, idesc, k4 > 0 ? 1u : 0u);
        }
        umma_commit(&tmem_full[buf]);
        umma_commit(&empty[stage]);
        if (kFused) umma_commit(&a_empty[slot]);
      }
      __syncwarp();
    }
  } else if (kFused && warp >= 8) {
    // ------------------------------ quantising prologue (fused) -----------
    // Warp w takes the units w, w + 4, ...: all token rows of the unit's K block, two per step (a
    // half warp owns one row's 128-wide group: 16 lanes x 8 elements), the next unit's
    // activations in flight while the current one is quantised.  Rows beyond M are zero: they are
    // written once, before the loop, and never touched again.
    if constexpr (kFused) {
      constexpr int STEPS = MP / 2;
      const int qw = warp - 8, hw = lane >> 4, sub = lane & 15;
      const AT* src = static_cast<const AT*>(p.a_src);
      const int64_t ld = static_cast<int64_t>(p.kb) * BK;
      const int live_steps = (p.m + 1) >> 1;   // steps that hold at least one real row
      for (uint32_t j = qw; j < a_slots; j += kQuantWarps) {
#pragma unroll
        for (int s2 = 0; s2 < STEPS; ++s2) {
          const int r = 2 * s2 + hw;
          if (r >= p.m) {
            *reinterpret_cast<uint2*>(a_res + j * (MP * BK) + r * 128 + (((sub >> 1) ^ (r & 7)) << 4) + ((sub & 1) << 3)) =
                make_uint2(0u, 0u);
            if (sub == 0) sa_res[j * MP + r] = 0.0f;
          }
        }
      }
      uint4 cur[STEPS], nxt[STEPS];
      pdl_wait();   // the activations may come from the kernel queued before this one
      auto fetch = [&](uint4 (&dst)[STEPS], uint32_t unit) {
        const int kbx = static_cast<int>((static_cast<uint32_t>(kb_first) + unit) % static_cast<uint32_t>(p.kb));
#pragma unroll
        for (int s2 = 0; s2 < STEPS; ++s2) {
          const int r = 2 * s2 + hw;
          if (s2 < live_steps) {
            dst[s2] = (r < p.m && unit < count)
                          ? __ldg(reinterpret_cast<const uint4*>(src + r * ld + kbx * BK + sub * 8))
                          : make_uint4(0u, 0u, 0u, 0u);
          }
        }
      };
      fetch(cur, qw);
      for (uint32_t i = qw; i < count; i += kQuantWarps) {
        fetch(nxt, i + kQuantWarps);
        const uint32_t slot = (i & a_mask);
        if (!mbar_wait(&a_empty[slot], ((i >> a_shift) & 1u) ^ 1u, abort_flag, p.status, kSiteDQuantEmpty)) break;
        __syncwarp();
        uint8_t* tile = a_res + slot * (MP * BK);
#pragma unroll
        for (int s2 = 0; s2 < STEPS; ++s2) {
          if (s2 < live_steps) {
            const int r = 2 * s2 + hw;
            float f[8];
            unpack8<AT>(cur[s2], f);
            float amax = 0.0f;
#pragma unroll
            for (int e = 0; e < 8; ++e) amax = fmaxf(amax, fabsf(f[e]));
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, o));
            const float scale = group_scale(amax);
            const uint2 bytes = fast_div_ok(amax) ? quantise8_fast16(cur[s2], f, scale, __frcp_rn(scale))
                                                  : quantise8<false>(f, scale, 0.0f);
            if (r < p.m) {
              // swizzled K-major layout of a TMA SWIZZLE_128B load: 16-byte chunk c of row r sits at
              // chunk c ^ (r & 7); this lane's 8 bytes are half of chunk sub / 2
              *reinterpret_cast<uint2*>(tile + r * 128 + (((sub >> 1) ^ (r & 7)) << 4) + ((sub & 1) << 3)) = bytes;
              if (sub == 0) sa_res[slot * MP + r] = scale;
            }
          }
        }
        fence_proxy_async_smem();   // the tensor core reads the tile through the async proxy
        __syncwarp();
        if (lane == 0) mbar_arrive(&a_full[slot]);
#pragma unroll
        for (int s2 = 0; s2 < STEPS; ++s2) cur[s2] = nxt[s2];
      }
    }
  } else if (warp == 2) {
    // ------------------------------ scale warp ----------------------------
    pdl_wait();   // the scales may come from the kernel queued before this one
    int t = t_first, kb = kb_first;
    for (uint32_t i = 0; i < count; ++i) {
      const uint32_t buf = i % C::kBufs;
      const uint32_t use = i / C::kBufs;
      if (!mbar_wait(&tmem_empty[buf], (use & 1u) ^ 1u, abort_flag, p.status, kSiteDScaleEmpty)) break;
      const float sb = __ldg(p.b_scales + static_cast<int64_t>(t) * p.kb + kb);
      // fused: the group scales of this unit are in shared memory once its tile is published
      const uint32_t slot = kFused ? (i & a_mask) : 0u;
      if (kFused && !mbar_wait(&a_full[slot], (i >> a_shift) & 1u, abort_flag, p.status, kSiteDQuantTmem)) break;
#pragma unroll
      for (int m0 = 0; m0 < MP; m0 += 32) {
        const int m = m0 + lane;
        if (m < MP) {
          float sa;
          if (kFused) sa = sa_res[slot * MP + m];
          else sa = (m < p.m) ? __ldg(p.a_scales + static_cast<int64_t>(m) * p.kb + kb) : 0.0f;
          sv[buf * MP + m] = sa * sb;
        }
      }
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(&sv_full[buf]);
        if (kFused) mbar_arrive(&a_empty[slot]);
      }
      if (++kb == p.kb) {
        kb = 0;
        ++t;
      }
    }
  } else if (warp >= 4 && warp < 8) {
    // ------------------------------ promotion + epilogue ------------------
    const int quarter = warp - 4;            // == warp % 4: TMEM lane quarter
    const int row = quarter * 32 + lane;     // weight row inside the tile
    const int ct = threadIdx.x - 128;        // 0..127 among the promotion threads
    const uint32_t lane_base = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
    float acc[MP];
#pragma unroll
    for (int j = 0; j < MP; ++j) acc[j] = 0.0f;
    pdl_wait();   // the output, workspace and counters may still be in use by the preceding kernel
    int t = t_first, kb = kb_first, seg_kb0 = kb_first;
    bool ok = true;
    for (uint32_t i = 0; i < count; ++i) {
      const uint32_t buf = i % C::kBufs;
      const uint32_t par = (i / C::kBufs) & 1u;
      // a warp whose wait ran out skips the work of the remaining units of its segment (without
      // waiting) and meets its siblings at the segment's end, where the four warps agree to leave
      if (ok && (!mbar_wait(&tmem_full[buf], par, abort_flag, p.status, kSiteDPromoFull) ||
                 !mbar_wait(&sv_full[buf], par, abort_flag, p.status, kSiteDPromoScale))) {
        ok = false;
      }
      if (ok) {
        __syncwarp();
        tc_fence_after_sync();
        const float4* svb = reinterpret_cast<const float4*>(sv + buf * MP);
        // all loads of up to 64 columns are issued before the single wait, so that their
        // latencies overlap; 128 columns go in two such halves (register budget)
        constexpr int HALF = (MP < 64) ? MP : 64;
#pragma unroll
        for (int h0 = 0; h0 < MP; h0 += HALF) {
          uint32_t v[HALF / CH][CH];
#pragma unroll
          for (int q = 0; q < HALF / CH; ++q) tmem_ld_cols<CH>(lane_base + buf * MP + h0 + q * CH, v[q]);
          tmem_ld_wait();
#pragma unroll
          for (int q = 0; q < HALF / CH; ++q) {
#pragma unroll
            for (int j = 0; j < CH; ++j) asm volatile("" : "+r"(v[q][j])::"memory");
          }
#pragma unroll
          for (int q = 0; q < HALF / CH; ++q) {
#pragma unroll
            for (int j = 0; j < CH; j += 4) {
              const int c = h0 + q * CH + j;
              const float4 s4 = svb[c >> 2];
              acc[c + 0] = fmaf(__uint_as_float(v[q][j + 0]), s4.x, acc[c + 0]);
              acc[c + 1] = fmaf(__uint_as_float(v[q][j + 1]), s4.y, acc[c + 1]);
              acc[c + 2] = fmaf(__uint_as_float(v[q][j + 2]), s4.z, acc[c + 2]);
              acc[c + 3] = fmaf(__uint_as_float(v[q][j + 3]), s4.w, acc[c + 3]);
            }
          }
        }
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(&tmem_empty[buf]);
      }

      const bool seg_end = (kb == p.kb - 1) || (i + 1 == count);
      if (seg_end) {
        if (named_bar_or(2, 128, !ok)) break;   // agreed: the piece is abandoned, nobody waits at the barriers below
        const int gn = t * TN + row;
        const bool whole = (seg_kb0 == 0 && kb == p.kb - 1);
        if (whole) {
          if (gn < p.n) store_column<MP, OutT>(p, gn, acc);
        } else {
          // one K part of a split tile: a slot of this CTA in the workspace (slot 0 for the tile
          // the piece starts in, slot 1 for the tile it ends in)
          const int64_t my_slot = p.splits == 0 ? static_cast<int64_t>(blockIdx.x) * 2 + (t == t_first ? 0 : 1)
                                                : static_cast<int64_t>(blockIdx.x);
          float* wp = p.workspace + my_slot * (MP * TN);
#pragma unroll
          for (int m = 0; m < MP; ++m) __stcg(wp + m * TN + row, acc[m]);
          __threadfence();
          // which CTAs hold parts of tile t: with even dealing, the CTA that owns unit u is
          // ceil((u + 1) G / U) - 1
          int c_lo = 0, c_hi = 0;
          if (p.splits == 0) {
            const long long g = gridDim.x;
            c_lo = static_cast<int>(((static_cast<long long>(t) * p.kb + 1) * g + p.units - 1) / p.units) - 1;
            c_hi = static_cast<int>(((static_cast<long long>(t + 1) * p.kb) * g + p.units - 1) / p.units) - 1;
          }
          const int parts = p.splits == 0 ? c_hi - c_lo + 1 : p.splits;
          named_bar_sync(1, 128);
          if (ct == 0) {
            const int prev = atomicAdd(p.counters + t, 1);
            *last_flag = (prev == parts - 1) ? 1u : 0u;
          }
          named_bar_sync(1, 128);
          if (*last_flag != 0u) {
            __threadfence();
            float sum[MP];
#pragma unroll
            for (int m = 0; m < MP; ++m) sum[m] = 0.0f;
            for (int part = 0; part < parts; ++part) {   // fixed order: the result does not depend on arrival order
              int64_t slot;
              if (p.splits == 0) {
                const long long c2 = c_lo + part;
                const int tf = static_cast<int>((c2 * p.units / gridDim.x) / p.kb);   // the tile CTA c2 starts in
                slot = c2 * 2 + (tf == t ? 0 : 1);
              } else {
                slot = static_cast<int64_t>(t) * p.splits + part;
              }
              const float* rp = p.workspace + slot * (MP * TN);
#pragma unroll
              for (int m = 0; m < MP; ++m) sum[m] += __ldcg(rp + m * TN + row);
            }
            if (gn < p.n) store_column<MP, OutT>(p, gn, sum);
            if (ct == 0) p.counters[t] = 0;   // ready for the next launch
          }
          named_bar_sync(1, 128);   // last_flag may be rewritten only after everyone has read it
        }
#pragma unroll
        for (int j = 0; j < MP; ++j) acc[j] = 0.0f;
        seg_kb0 = 0;
      }
      if (++kb == p.kb) {
        kb = 0;
        ++t;
      }
    }
  }

  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  if (warp == 0) tmem_dealloc(tmem_base, C::kTmemCols);
}

template <int MP, typename OutT, typename AT = void>
int launch_decode_t(const CUtensorMap& mw, const CUtensorMap& ma, const DecodeParams& p, int ctas,
                    cudaStream_t stream, int smem_bytes = 0) {
  using C = DCfg<MP>;
  constexpr bool kFused = !std::is_same<AT, void>::value;
  if (!kFused) smem_bytes = C::kSmemBytes;
  static bool attr_done[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !attr_done[dev]) {
    cudaError_t e = cudaFuncSetAttribute(w8a8_decode_kernel<MP, OutT, AT>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         kFused ? kFusedMaxSmem : C::kSmemBytes);
    if (e != cudaSuccess) return note_cuda_error(e);
    attr_done[dev] = true;
  }
  // programmatic dependent launch: the preamble and the weight prefetch (into L2) of this kernel may
  // overlap the tail of the kernel queued before it (in practice the quantisation kernel)
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ctas);
  cfg.blockDim = dim3(std::is_same<AT, void>::value ? kThreads : kFusedThreads);
  cfg.dynamicSmemBytes = smem_bytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = options().decode_pdl ? 1 : 0;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, w8a8_decode_kernel<MP, OutT, AT>, mw, ma, p);
  if (e != cudaSuccess) return note_cuda_error(e);
  return check_launch();
}

template <typename OutT, typename AT>
int launch_decode_fused_mp(int mp, const CUtensorMap& mw, const DecodeParams& p, int ctas,
                           cudaStream_t stream, int smem_bytes) {
  return mp == 16 ? launch_decode_t<16, OutT, AT>(mw, mw, p, ctas, stream, smem_bytes)
                  : launch_decode_t<32, OutT, AT>(mw, mw, p, ctas, stream, smem_bytes);
}
template <typename AT>
int launch_decode_fused_out(int out_dt, int mp, const CUtensorMap& mw, const DecodeParams& p, int ctas,
                            cudaStream_t stream, int smem_bytes) {
  switch (out_dt) {
    case 0: return launch_decode_fused_mp<float, AT>(mp, mw, p, ctas, stream, smem_bytes);
    case 1: return launch_decode_fused_mp<__half, AT>(mp, mw, p, ctas, stream, smem_bytes);
    case 2: return launch_decode_fused_mp<__nv_bfloat16, AT>(mp, mw, p, ctas, stream, smem_bytes);
    default: return INFEROP_ERR_DTYPE;
  }
}

template <typename OutT>
int launch_decode_mp(int mp, const CUtensorMap& mw, const CUtensorMap& ma, const DecodeParams& p,
                     int ctas, cudaStream_t stream) {
  switch (mp) {
    case 16: return launch_decode_t<16, OutT>(mw, ma, p, ctas, stream);
    case 32: return launch_decode_t<32, OutT>(mw, ma, p, ctas, stream);
    case 64: return launch_decode_t<64, OutT>(mw, ma, p, ctas, stream);
    default: return launch_decode_t<128, OutT>(mw, ma, p, ctas, stream);
  }
}

// ------------------------------ K parts over a cluster --------------------------------------
// The form for few tiles (parts_for), at most one wave of them, whatever M.  With few output tiles one CTA per tile leaves most SMs
// idle while the weights could stream from HBM through all of them.  Here the `parts` CTAs of a cluster own one
// 128 x 128 tile of C and an equal share of its K blocks each; at the end each CTA leaves its fp32 partial tile in its own
// shared memory, and after a cluster barrier every CTA adds one slice of the rows over all parts, in K order, through
// distributed shared memory, rounds once and stores.  No partial touches global memory, nothing is counted or fenced
// there, and the call needs no scratch.  What it replaces, quantiser + GEMM in a graph on cold weights, before -> after (us):
// 16 x 7168 x 18432 30.4 -> 26.8, 64 x 4096 x 7168 19.5 -> 13.0, 64 x 7168 x 18432 47.8 -> 32.6, 32 x 1024 x 1024 9.6 -> 5.7
// (parts added through a workspace by the kernel above).  What is left over the weights' time at the HBM rate is about
// 5 us: set-up, first round trip, merge and drain.
//
// Per CTA (384 threads, one CTA per SM):
//   warps 0, 2  tensor memory; TMA producers: weight rows [128 x 128 B] and activation rows [ROWS x 128 B] per K block
//   warps 1, 3  MMA issuers (even / odd K blocks): 4 x tcgen05.mma (K = 32) into one of four accumulator buffers
//   warps 4-11  promotion
// More than 64 rows (ROWS = 128): the activations are the M side, as in gemm_sm100.cu; a promotion thread owns a row
// and 64 columns and has one scale per K block in a register.  Up to 64 rows the weights are the M side (M = 128) and the
// rows, rounded up to 16, the N side, as above: a promotion thread owns one column and half of ROWS rows, whose scales the
// warp hands around through shared memory.  128 rows of products per weight byte would put a stream of weights at 5 TB/s
// on the power cap: 16 x 7168 x 18432, a second of calls, 30.6 us with 128 rows multiplied although a graph of a few
// milliseconds took 26.3.
// Warps whose rows lie beyond M have no part in it.  A CTA that gave up a wait says so in its shared memory, all CTAs of
// the cluster still meet at both barriers, and a tile with such a part is not stored.
namespace split {

constexpr int TM = 128;                 // rows of C per tile (UMMA M)
constexpr int kPromoWarps = 8;
constexpr int kThreads = 128 + 32 * kPromoWarps;
constexpr int kBufs = 4;                // accumulator buffers of TN columns
constexpr int CT = TN / 2;              // columns per promotion thread
constexpr int kMaxParts = 8;            // portable cluster size

template <int ROWS>
struct SCfg {
  static constexpr int kBytesA = ROWS * BK;
  static constexpr int kStageBytes = kBytesA + kBytesW;
  static constexpr int kStages = (ROWS == 32) ? 10 : (ROWS == 64) ? 8 : 6;
  static constexpr bool kSwapped = ROWS < TM;      // the weights are the M side of the MMA
  static constexpr int kBarrierBytes = 256;
  static constexpr int kScaleBytes = kPromoWarps * 32 * 4;   // swapped: the rows' scales of a K block, per promotion warp
  static constexpr int kSmemBytes = kStages * kStageBytes + kBarrierBytes + kScaleBytes + 1024;
  static_assert(kStages % 2 == 0, "a stage always belongs to the same MMA issuer");
  static_assert(kStages * kStageBytes >= TM * TN * 4, "the partial tile takes the place of the ring");
  static_assert((2 * kStages + 2 * kBufs) * 8 + 8 <= kBarrierBytes, "barriers, tensor-memory slot, flag");
  static_assert(kSmemBytes <= 232448, "shared memory of one CTA");
};

struct SplitParams {
  const float* a_scales;
  const float* b_scales;
  void* dst[8];    // as in DecodeParams
  int n_dst, ldc, col0;
  int m, n, kb;
  int tiles_m, parts;
  int vec_store;   // the rows of C start on 4-element boundaries in every destination
  int no_loads;    // test hook: the producers issue no load
  int trigger;     // let kernels queued behind this one with programmatic stream serialisation start early
  DeviceStatus* status;
};

enum : uint32_t {
  kSiteSProducerEmpty = 0x131,
  kSiteSMmaFull = 0x231,
  kSiteSMmaTmemEmpty = 0x232,
  kSiteSPromoTmemFull = 0x331,
};

__device__ __forceinline__ void pin32(uint32_t (&r)[32]) {
#pragma unroll
  for (int i = 0; i < 32; ++i) asm volatile("" : "+r"(r[i])::"memory");
}

__device__ __forceinline__ float4 ld_cluster_f4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(addr)
               : "memory");
  return v;
}
__device__ __forceinline__ uint32_t ld_cluster_u32(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
  return v;
}

template <typename OutT, int ROWS>
__global__ void __launch_bounds__(kThreads, 1)
w8a8_split_gemm_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w,
                       const SplitParams p) {
  using C = SCfg<ROWS>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::kStages * C::kStageBytes);
  uint64_t* full = bars;                        // [kStages] TMA -> MMA
  uint64_t* empty = full + C::kStages;          // [kStages] MMA -> TMA
  uint64_t* tmem_full = empty + C::kStages;     // [kBufs]   MMA -> promotion
  uint64_t* tmem_empty = tmem_full + kBufs;     // [kBufs]   promotion -> MMA
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tmem_empty + kBufs);
  volatile uint32_t* abort_flag = tmem_slot + 1;

  const int warp = __shfl_sync(0xFFFFFFFFu, static_cast<int>(threadIdx.x >> 5), 0);
  const int lane = threadIdx.x & 31;
  const int part = static_cast<int>(cluster_ctarank());
  // M-tiles of one weight tile lie next to each other, so that its weights are read from HBM once
  const int tile = (blockIdx.x / p.parts) / p.tiles_m;
  const int row0 = (blockIdx.x / p.parts) % p.tiles_m * TM;
  const int rows = min(p.m - row0, ROWS);   // live rows of this tile
  const int kb0 = part * p.kb / p.parts;
  const uint32_t count = static_cast<uint32_t>((part + 1) * p.kb / p.parts - kb0);
  // which promotion warps have rows: lane quarters of both column halves, or (swapped) halves of ROWS
  constexpr int kHalfRows = ROWS / 2;
  const int live_quarters = C::kSwapped ? 4 : (rows + 31) >> 5;
  const int live_halves = C::kSwapped && rows <= kHalfRows ? 1 : 2;

  if (threadIdx.x == 0) {
    for (int s = 0; s < C::kStages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < kBufs; ++b) {
      mbar_init(&tmem_full[b], 1);
      mbar_init(&tmem_empty[b], live_halves * live_quarters);
    }
    *abort_flag = 0u;
    mbar_init_fence();
    tma_prefetch_desc(&map_w);
    tma_prefetch_desc(&map_a);
  }
  if (warp == 0) {
    tmem_alloc(tmem_slot, kBufs * TN);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = __shfl_sync(0xFFFFFFFFu, *tmem_slot, 0);
  if (p.trigger) pdl_launch_dependents();

  if (warp == 0 || warp == 2) {
    // ------------------------------ TMA producers ------------------------------
    // warp 0 arms the stages and loads the weights, warp 2 the activations; neither before the wait, as above
    const bool weights = warp == 0;
    const CUtensorMap* map = weights ? &map_w : &map_a;
    const uint32_t off = weights ? C::kBytesA : 0u;
    const int y = weights ? tile * TN : row0;
    uint32_t stage = 0, phase = 0, armed = 0;
    bool ok = true;
    if (weights && !p.no_loads) {
      for (uint32_t i = 0; i < count && i < kAhead; ++i) {
        if (elect_one()) tma_prefetch_2d(map, (kb0 + static_cast<int>(i)) * BK, y);
        __syncwarp();
      }
    }
    pdl_wait();
    for (uint32_t i = 0; i < count && !p.no_loads; ++i) {
      if (!mbar_wait(&empty[stage], phase ^ 1u, abort_flag, p.status, kSiteSProducerEmpty)) {
        ok = false;
        break;
      }
      __syncwarp();
      if (elect_one()) {
        if (weights) mbar_arrive_expect_tx(&full[stage], C::kStageBytes);
        tma_load_2d(smem + stage * C::kStageBytes + off, map, &full[stage], (kb0 + static_cast<int>(i)) * BK, y);
      }
      __syncwarp();
      armed = i + 1;
      if (++stage == static_cast<uint32_t>(C::kStages)) {
        stage = 0;
        phase ^= 1u;
      }
    }
    if (!ok && lane == 0) {
      // wind-down: let the copies this warp started land before the CTA exits
      const uint32_t lo = armed > static_cast<uint32_t>(C::kStages) ? armed - C::kStages : 0u;
      for (uint32_t i = lo; i < armed; ++i) {
        const long long t0 = clock64();
        while (!mbar_test_wait(&full[i % C::kStages], (i / C::kStages) & 1u)) {
          if (clock64() - t0 > kWaitBudgetCycles) break;
        }
      }
    }
  } else if (warp == 1 || warp == 3) {
    // ------------------------------ MMA issuers (warp-uniform) ----------------
    const uint32_t idesc =
        C::kSwapped ? umma_idesc_e4m3_f32(TN, static_cast<uint32_t>((rows + 15) & ~15)) : umma_idesc_e4m3_f32(TM, TN);
    const uint32_t smem_base = smem_u32(smem);
    for (uint32_t i = warp >> 1; i < count; i += 2) {
      const uint32_t stage = i % C::kStages, phase = (i / C::kStages) & 1u;
      const uint32_t buf = i % kBufs, use = i / kBufs;
      if (!mbar_wait(&full[stage], phase, abort_flag, p.status, kSiteSMmaFull)) break;
      if (!mbar_wait(&tmem_empty[buf], (use & 1u) ^ 1u, abort_flag, p.status, kSiteSMmaTmemEmpty)) break;
      __syncwarp();
      tc_fence_after_sync();
      const uint32_t a_addr = smem_base + stage * C::kStageBytes;
      const uint64_t da = umma_desc_k_sw128(a_addr);
      const uint64_t dw = umma_desc_k_sw128(a_addr + C::kBytesA);
      if (elect_one()) {
#pragma unroll
        for (int k4 = 0; k4 < BK / 32; ++k4)
          umma_f8_ss(tmem_base + buf * TN, (C::kSwapped ? dw : da) + 2u * k4, (C::kSwapped ? da : dw) + 2u * k4, idesc,
                     k4 > 0 ? 1u : 0u);
        umma_commit(&tmem_full[buf]);
        umma_commit(&empty[stage]);
      }
      __syncwarp();
    }
  } else if (warp >= 4) {
    // ------------------------------ promotion ---------------------------------
    const int quarter = warp & 3;        // == warp % 4: the lane quarter this warp may read
    const int half = (warp - 4) >> 2;    // column half of the tile; swapped: half of ROWS
    pdl_wait();   // a_scales come from the kernel queued before this one, which may also still read C
    if (quarter < live_quarters && half < live_halves) {
      // columns of the accumulator per thread: 64 columns of C of one row, or the rows of one column of C
      constexpr int kCols = C::kSwapped ? kHalfRows : CT;
      const uint32_t lane_base = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + half * kCols;
      const int scale_row = C::kSwapped ? half * kHalfRows + lane : quarter * 32 + lane;   // whose scale this lane fetches
      const bool have = scale_row < rows && (!C::kSwapped || lane < kHalfRows);
      const float* sa_ptr = p.a_scales + static_cast<int64_t>(row0 + (have ? scale_row : 0)) * p.kb + kb0;
      const float* sb_ptr = p.b_scales + static_cast<int64_t>(tile) * p.kb + kb0;
      float* my_scales = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(bars) + C::kBarrierBytes) + (warp - 4) * 32;
      const int units = static_cast<int>(count);
      float2 acc[kCols / 2];
#pragma unroll
      for (int j = 0; j < kCols / 2; ++j) acc[j] = make_float2(0.0f, 0.0f);
      // the row's scales are requested three blocks ahead; lane l holds the weight block's scale of block l of the
      // current 32
      float s0 = have ? ld_nc_f32_pinned(sa_ptr) : 0.0f;
      float s1 = have && 1 < units ? ld_nc_f32_pinned(sa_ptr + 1) : 0.0f;
      float s2 = have && 2 < units ? ld_nc_f32_pinned(sa_ptr + 2) : 0.0f;
      float sb_c = lane < units ? ld_nc_f32_pinned(sb_ptr + lane) : 0.0f;
      float sb_n = lane + 32 < units ? ld_nc_f32_pinned(sb_ptr + lane + 32) : 0.0f;
      bool ok = true;
      for (int i = 0; i < units; ++i) {
        if (i > 0 && (i & 31) == 0) {
          sb_c = sb_n;
          sb_n = i + 32 + lane < units ? ld_nc_f32_pinned(sb_ptr + i + 32 + lane) : 0.0f;
        }
        const float s = s0 * __shfl_sync(0xFFFFFFFFu, sb_c, i & 31);
        if constexpr (C::kSwapped) my_scales[lane] = s;
        s0 = s1;
        s1 = s2;
        if (have && i + 3 < units) s2 = ld_nc_f32_pinned(sa_ptr + i + 3);
        const int buf = i % kBufs;
        if (!mbar_wait(&tmem_full[buf], (i / kBufs) & 1u, abort_flag, p.status, kSiteSPromoTmemFull)) {
          ok = false;
          break;
        }
        __syncwarp();
        tc_fence_after_sync();
        if constexpr (C::kSwapped) {
          uint32_t v[kCols];
          tmem_ld_cols<kCols>(lane_base + buf * TN, v);
          tmem_wait_pin<kCols>(v);
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive(&tmem_empty[buf]);
          const float4* s4 = reinterpret_cast<const float4*>(my_scales);
#pragma unroll
          for (int j = 0; j < kCols / 4; ++j) {
            const float4 f = s4[j];
            acc[2 * j] = __ffma2_rn(make_float2(__uint_as_float(v[4 * j]), __uint_as_float(v[4 * j + 1])),
                                    make_float2(f.x, f.y), acc[2 * j]);
            acc[2 * j + 1] = __ffma2_rn(make_float2(__uint_as_float(v[4 * j + 2]), __uint_as_float(v[4 * j + 3])),
                                        make_float2(f.z, f.w), acc[2 * j + 1]);
          }
          __syncwarp();   // every lane has read the scales: the slot may be written again
        } else {
          uint32_t v0[32], v1[32];
          tmem_ld_32x32(lane_base + buf * TN, v0);
          tmem_ld_32x32(lane_base + buf * TN + 32, v1);
          tmem_ld_wait();
          pin32(v0);
          pin32(v1);
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive(&tmem_empty[buf]);
          const float2 ss = make_float2(s, s);
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            acc[j] = __ffma2_rn(make_float2(__uint_as_float(v0[2 * j]), __uint_as_float(v0[2 * j + 1])), ss, acc[j]);
            acc[16 + j] =
                __ffma2_rn(make_float2(__uint_as_float(v1[2 * j]), __uint_as_float(v1[2 * j + 1])), ss, acc[16 + j]);
          }
        }
      }
      // The partial tile takes the place of the ring: this warp has waited for every unit's products, so the tensor
      // core has read every stage and no copy is in flight.  Row r = 512 bytes, 16-byte chunk j at j ^ (r & 31).
      if (ok) {
        const float* a = reinterpret_cast<const float*>(acc);
        if constexpr (C::kSwapped) {
          const int col = quarter * 32 + lane;
#pragma unroll
          for (int j = 0; j < kCols; ++j) {
            const int row = half * kHalfRows + j;
            *reinterpret_cast<float*>(smem + row * (TN * 4) + (((col >> 2) ^ (row & 31)) << 4) + (col & 3) * 4) = a[j];
          }
        } else {
          const int row = quarter * 32 + lane;
#pragma unroll
          for (int j = 0; j < kCols / 4; ++j) {
            const int chunk = half * (kCols / 4) + j;
            *reinterpret_cast<float4*>(smem + row * (TN * 4) + ((chunk ^ (row & 31)) << 4)) =
                make_float4(a[4 * j], a[4 * j + 1], a[4 * j + 2], a[4 * j + 3]);
          }
        }
      }
    }
  }
  __syncwarp();
  tc_fence_before_sync();
  cluster_sync_all();
  tc_fence_after_sync();
  if (warp == 0) tmem_dealloc(tmem_base, kBufs * TN);

  // ------------------------------ merge -----------------------------------------
  // float4 e of the tile's live rows, in row order: this CTA adds [part, part + 1) * total / parts
  {
    const uint32_t my_base = smem_u32(smem), my_flag = smem_u32(tmem_slot + 1);
    const int total = rows * (TN / 4);
    const int lo = part * total / p.parts, hi = (part + 1) * total / p.parts;
    uint32_t bad = 0;
    for (int q = 0; q < p.parts; ++q) bad |= ld_cluster_u32(mapa_shared(my_flag, q));
    if (bad == 0) {
      for (int e = lo + static_cast<int>(threadIdx.x); e < hi; e += kThreads) {
        const int row = e / (TN / 4), chunk = e % (TN / 4);
        const uint32_t at = my_base + row * (TN * 4) + ((chunk ^ (row & 31)) << 4);
        float4 v[kMaxParts];
#pragma unroll
        for (int q = 0; q < kMaxParts; ++q)
          if (q < p.parts) v[q] = ld_cluster_f4(mapa_shared(at, q));
        float4 sum = v[0];
#pragma unroll
        for (int q = 1; q < kMaxParts; ++q)
          if (q < p.parts) {
            sum.x += v[q].x;
            sum.y += v[q].y;
            sum.z += v[q].z;
            sum.w += v[q].w;
          }
        const int col = tile * TN + chunk * 4;
        alignas(16) OutT o[4] = {cvt_out<OutT>(sum.x), cvt_out<OutT>(sum.y), cvt_out<OutT>(sum.z), cvt_out<OutT>(sum.w)};
        const int64_t to = static_cast<int64_t>(row0 + row) * p.ldc + p.col0 + col;
#pragma unroll 1
        for (int d = 0; d < p.n_dst; ++d) {
          OutT* dst = static_cast<OutT*>(p.dst[d]) + to;
          if (p.vec_store && col + 4 <= p.n) {
            if constexpr (sizeof(OutT) == 4) *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<const uint4*>(o);
            else *reinterpret_cast<uint2*>(dst) = *reinterpret_cast<const uint2*>(o);
          } else {
#pragma unroll
            for (int j = 0; j < 4; ++j)
              if (col + j < p.n) dst[j] = o[j];
          }
        }
      }
    }
  }
  // nobody leaves while a peer may still read its partial tile
  cluster_sync_all();
}

template <int ROWS>
cudaLaunchConfig_t config(cudaLaunchAttribute (&attr)[2], int tiles, int parts, bool pdl, cudaStream_t stream) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(tiles * parts);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = SCfg<ROWS>::kSmemBytes;
  cfg.stream = stream;
  int n = 0;
  if (parts > 1) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = parts;
    attr[n].val.clusterDim.y = 1;
    attr[n++].val.clusterDim.z = 1;
  }
  if (pdl) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n++].val.programmaticStreamSerializationAllowed = 1;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n;
  return cfg;
}

template <typename OutT, int ROWS>
int launch_t(const CUtensorMap& ma, const CUtensorMap& mw, const SplitParams& p, int tiles, cudaStream_t stream) {
  static bool attr_done[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !attr_done[dev]) {
    cudaError_t e = cudaFuncSetAttribute(w8a8_split_gemm_kernel<OutT, ROWS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         SCfg<ROWS>::kSmemBytes);
    if (e != cudaSuccess) return note_cuda_error(e);
    attr_done[dev] = true;
  }
  cudaLaunchAttribute attr[2];
  const cudaLaunchConfig_t cfg = config<ROWS>(attr, tiles, p.parts, options().decode_pdl != 0, stream);
  const cudaError_t e = cudaLaunchKernelEx(&cfg, w8a8_split_gemm_kernel<OutT, ROWS>, ma, mw, p);
  if (e != cudaSuccess) return note_cuda_error(e);
  return check_launch();
}

template <typename OutT>
int launch_rows(int rows, const CUtensorMap& ma, const CUtensorMap& mw, const SplitParams& p, int tiles, cudaStream_t stream) {
  switch (rows) {
    case 32: return launch_t<OutT, 32>(ma, mw, p, tiles, stream);
    case 64: return launch_t<OutT, 64>(ma, mw, p, tiles, stream);
    default: return launch_t<OutT, 128>(ma, mw, p, tiles, stream);
  }
}

// [s]: clusters of s CTAs (1..kMaxParts) that the current device holds at once, 0 where that cannot be learned
// (inferop_last_cuda_error says why); asked once per device.
const int* active_clusters() {
  static int known[64][kMaxParts + 1] = {};
  static std::once_flag once[64];
  static const int none[kMaxParts + 1] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return none;
  std::call_once(once[dev], [dev] {
    const auto ok = [](cudaError_t e) {
      if (e == cudaSuccess) return true;
      note_cuda_error(e);
      cudaGetLastError();
      return false;
    };
    const auto kernel = w8a8_split_gemm_kernel<float, 32>;   // (the largest shared memory of the three)
    if (!ok(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SCfg<32>::kSmemBytes))) return;
    // one part is launched without the cluster attribute, of which the cluster query wants to see one
    int sms = 0, n = 0;
    if (ok(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) &&
        ok(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, kThreads, SCfg<32>::kSmemBytes))) {
      known[dev][1] = sms * n;
    }
    for (int s = 2; s <= kMaxParts; ++s) {
      cudaLaunchAttribute attr[2];
      const cudaLaunchConfig_t cfg = config<32>(attr, 1, s, false, nullptr);
      if (ok(cudaOccupancyMaxActiveClusters(&n, kernel, &cfg))) known[dev][s] = n;
    }
  });
  return known[dev];
}

// Over how many CTAs the K range of a tile goes (0: another kernel serves the call).  As many as still leave every cluster of the
// launch an SM set of its own (8 at most; fewer, smaller clusters fill more of the chip: 33 of 4, 45 of 3, 74 of 2 on 148
// SMs), since a second wave costs a whole pass.  Quantiser + GEMM, us in a graph, cold weights, parts 1 / 2 / 3 / 4 / 8: 16
// tiles (32 x 2048 x 1024) 7.4 / 6.2 / 6.6 / 5.9 / 10.1 (two waves), 24 tiles (64 x 3072 x 3072) 12.2 / 9.0 / 8.7 / 7.8 / 13.5,
// 8 tiles (32 x 1024 x 4096) 13.6 / 9.4 / 8.7 / 7.6 / 6.8.
// From 65 rows on one part: there the other kernels add along K in one chain, so a row's bits do not depend on the
// rows that share its call, and that stays so although parts would be faster (129 x 4096 x 7168: 23.2 at one part, 16.4 at two).
// One part where it is the faster kernel, same bits either way.  Quantiser + GEMM, us, the other kernels / one part: 256 x 7168 x
// 18432 68.0 / 51.5, 1000 x 2048 x 7168 31.7 / 26.1, 129 x 4096 x 7168 29.0 / 23.2, 65 x 7168 x 18432 50.7 / 45.7, 64 x 10240 x 7168
// 34.3 / 24.9, 16 x 9600 x 7168 21.2 / 19.2.  Not for a short K of up to 128 rows (128 x 18432 x 1024 11.0 / 12.0, 32 x 18432 x 1024
// 7.7 / 7.8) or of very many (18900 x 128 x 1024 17.8 / 18.8), nor for a few rows on nearly a wave of tiles, which the kernel with a
// workspace streams at the rate of HBM (1 x 18432 x 7168 25.5 / 26.2; 1 x 16384 x 7168 23.5 / 23.5).
int parts_for(int64_t m, int64_t tiles, int64_t kb) {
  const int* const clusters = active_clusters();
  for (int s = m <= 64 ? kMaxParts : 1; s > 1; --s)
    if (s <= kb && tiles <= clusters[s]) return s;
  if (tiles > clusters[1]) return 0;
  if (m <= 128 ? kb < 32 : kb < 32 && m > 4096) return 0;
  return m <= 16 && tiles * 8 > static_cast<int64_t>(clusters[1]) * 7 ? 0 : 1;
}

}  // namespace split

// How the kernel with a workspace deals a call: DecodeParams::splits and the number of CTAs.  The K parts of a split tile are
// those of the cluster form, so that both give the same bits (the one-launch form of quantise + GEMM, the options
// gemm_path and gemm_split).  More rows and a limited number of CTAs cut as finely as there are CTAs.
struct Cut {
  int splits, ctas;
};
Cut decode_cut(int sm_count, int64_t m, int64_t n, int64_t k, bool fused) {
  const Options& opt = options();
  int max_ctas = opt.gemm_ctas > 0 ? opt.gemm_ctas : sm_count;
  if (max_ctas > sm_count) max_ctas = sm_count;   // the workspace is sized for one CTA per SM
  const int64_t tiles = (n + TN - 1) / TN, kb = k / BK;
  if (opt.decode_deal == 0 && !fused) {
    // every (tile, K block) unit dealt evenly over one CTA per SM
    return {0, static_cast<int>(tiles * kb < max_ctas ? tiles * kb : max_ctas)};
  }
  if (tiles >= max_ctas) return {1, max_ctas};
  int parts = static_cast<int>(max_ctas / tiles);
  if (parts > kb) parts = static_cast<int>(kb);
  if (opt.decode_splits > 0) {
    if (opt.decode_splits <= parts) parts = opt.decode_splits;
  } else if (m <= 64 && opt.gemm_ctas == 0) {
    const int cluster = split::parts_for(m, tiles, kb);
    if (cluster > 0 && cluster < parts) parts = cluster;
  }
  return {parts, static_cast<int>(tiles) * parts};
}

}  // namespace

// More tiles than one wave are for the other kernels: here they would take two (300 x 7168 x 2048, 168 tiles: 21.3 against 15.5 of
// the pair kernel).
int split_gemm_parts(int64_t m, int64_t n, int64_t k) {
  const Options& opt = options();
  if (opt.gemm_split < 0 || opt.gemm_path != 0 || opt.gemm_pair == 1 || opt.gemm_block_n != 0 || opt.gemm_ctas != 0 ||
      opt.decode_deal == 0 || opt.decode_splits != 0) {
    return 0;
  }
  const int64_t tiles_m = (m + split::TM - 1) / split::TM, tiles_n = (n + TN - 1) / TN, kb = k / BK;
  if (tiles_m > (1 << 15) || tiles_n > (1 << 15)) return 0;
  if (opt.gemm_split > 0) return opt.gemm_split <= kb ? opt.gemm_split : 0;
  return split::parts_for(m, tiles_m * tiles_n, kb);
}

int launch_gemm_split_to(DeviceCtx* ctx, int parts, void* const* dst, int n_dst, int64_t ldc, int64_t col0, const void* a_q,
                         const void* a_scales, const void* b_q, const void* b_scales, int64_t m, int64_t n, int64_t k,
                         int32_t out_dt, bool trigger, cudaStream_t stream) {
  if (n_dst < 1 || n_dst > 8) return INFEROP_ERR_SHAPE;
  const int rows = m <= 32 ? 32 : m <= 64 ? 64 : 128;
  const int out_bytes = out_dt == 0 ? 4 : 2;
  split::SplitParams p;
  p.a_scales = static_cast<const float*>(a_scales);
  p.b_scales = static_cast<const float*>(b_scales);
  uintptr_t all = 0;
  for (int d = 0; d < 8; ++d) {
    p.dst[d] = dst[d < n_dst ? d : 0];
    all |= reinterpret_cast<uintptr_t>(p.dst[d]);
  }
  p.n_dst = n_dst;
  p.ldc = static_cast<int>(ldc);
  p.col0 = static_cast<int>(col0);
  p.m = static_cast<int>(m);
  p.n = static_cast<int>(n);
  p.kb = static_cast<int>(k / BK);
  p.tiles_m = static_cast<int>((m + split::TM - 1) / split::TM);
  p.parts = parts;
  p.vec_store = ldc % 4 == 0 && col0 % 4 == 0 && all % (4 * out_bytes) == 0;
  p.no_loads = options().debug_no_loads;
  p.trigger = trigger && options().pdl_trigger;
  p.status = ctx->status;
  CUtensorMap ma, mw;
  int rc = make_tensor_map_2d(&ma, a_q, 1, m, k, k, rows, BK, true);
  if (rc != INFEROP_OK) return rc;
  rc = make_tensor_map_2d(&mw, b_q, 1, n, k, k, TN, BK, true);
  if (rc != INFEROP_OK) return rc;
  const int tiles = static_cast<int>((n + TN - 1) / TN) * p.tiles_m;
  switch (out_dt) {
    case 0: return split::launch_rows<float>(rows, ma, mw, p, tiles, stream);
    case 1: return split::launch_rows<__half>(rows, ma, mw, p, tiles, stream);
    case 2: return split::launch_rows<__nv_bfloat16>(rows, ma, mw, p, tiles, stream);
    default: return INFEROP_ERR_DTYPE;
  }
}

bool decode_needs_scratch(int sm_count, int64_t m, int64_t n, int64_t k, bool fused) {
  return decode_cut(sm_count, m, n, k, fused).splits != 1;   // (whole tiles leave workspace and counters alone)
}

size_t decode_workspace_bytes(int ctas) { return static_cast<size_t>(ctas) * 2 * kDecodeMaxM * TN * 4; }

int launch_gemm_decode_fused(DeviceCtx* ctx, float* workspace, int* counters, void* c, const void* a,
                             int32_t a_dt, const void* b_q, const void* b_scales, int64_t m, int64_t n,
                             int64_t k, int32_t out_dt, cudaStream_t stream) {
  const int mp = m <= 16 ? 16 : 32;
  DecodeParams p;
  p.a_scales = nullptr;
  p.a_src = a;
  p.b_scales = static_cast<const float*>(b_scales);
  p.dst[0] = c;
  p.n_dst = 1;
  p.ldc = static_cast<int>(n);
  p.col0 = 0;
  p.workspace = workspace;
  p.counters = counters;
  p.m = static_cast<int>(m);
  p.n = static_cast<int>(n);
  p.kb = static_cast<int>(k / 128);
  p.n_tiles = static_cast<int>((n + TN - 1) / TN);
  p.units = static_cast<long long>(p.n_tiles) * p.kb;
  p.no_loads = options().debug_no_loads;
  p.trigger = options().pdl_trigger;
  p.status = ctx->status;
  CUtensorMap mw;
  const int rc = make_tensor_map_2d(&mw, b_q, 1, n, k, k, TN, BK, true);
  if (rc != INFEROP_OK) return rc;
  const Cut cut = decode_cut(ctx->sm_count, m, n, k, true);
  if (cut.splits != 1 && !workspace) return INFEROP_ERR_LIMIT;   // (an option changed since decode_needs_scratch)
  p.splits = cut.splits;
  // token-tile ring of 32 KiB beside a full-depth weight ring
  p.a_slots = 32 * 1024 / (mp * BK);
  if (p.a_slots > kMaxSlots) p.a_slots = kMaxSlots;
  const int bufs = (512 / mp) < 8 ? (512 / mp) : 8;
  const int fixed = p.a_slots * mp * (BK + 4) + bufs * mp * 4 + 1024 /* barriers */ + 1024 /* alignment slack */;
  p.stages = 10;
  const int smem_bytes = p.stages * kBytesW + fixed;
  if (a_dt == 2) return launch_decode_fused_out<__nv_bfloat16>(out_dt, mp, mw, p, cut.ctas, stream, smem_bytes);
  if (a_dt == 1) return launch_decode_fused_out<__half>(out_dt, mp, mw, p, cut.ctas, stream, smem_bytes);
  return INFEROP_ERR_DTYPE;
}

int launch_gemm_decode(DeviceCtx* ctx, float* workspace, int* counters, void* c, const void* a_q,
                       const void* a_scales, const void* b_q, const void* b_scales, int64_t m,
                       int64_t n, int64_t k, int32_t out_dt, cudaStream_t stream, int clear_counters) {
  void* const dst[1] = {c};
  return launch_gemm_decode_to(ctx, workspace, counters, dst, 1, n, 0, a_q, a_scales, b_q, b_scales, m, n,
                               k, out_dt, stream, clear_counters);
}

int launch_gemm_decode_to(DeviceCtx* ctx, float* workspace, int* counters, void* const* dst, int n_dst,
                          int64_t ldc, int64_t col0, const void* a_q, const void* a_scales,
                          const void* b_q, const void* b_scales, int64_t m, int64_t n, int64_t k,
                          int32_t out_dt, cudaStream_t stream, int clear_counters) {
  const int mp = m <= 16 ? 16 : m <= 32 ? 32 : m <= 64 ? 64 : 128;
  DecodeParams p;
  p.a_src = nullptr;
  p.stages = 0;
  p.a_slots = 0;
  p.a_scales = static_cast<const float*>(a_scales);
  p.b_scales = static_cast<const float*>(b_scales);
  if (n_dst < 1 || n_dst > 8) return INFEROP_ERR_SHAPE;
  for (int d = 0; d < 8; ++d) p.dst[d] = dst[d < n_dst ? d : 0];
  p.n_dst = n_dst;
  p.ldc = static_cast<int>(ldc);
  p.col0 = static_cast<int>(col0);
  p.workspace = workspace;
  p.counters = counters;
  p.m = static_cast<int>(m);
  p.n = static_cast<int>(n);
  p.kb = static_cast<int>(k / 128);
  p.n_tiles = static_cast<int>((n + TN - 1) / TN);
  p.units = static_cast<long long>(p.n_tiles) * p.kb;
  p.no_loads = options().debug_no_loads;
  p.trigger = options().pdl_trigger;
  p.status = ctx->status;

  CUtensorMap mw, ma;
  int rc = make_tensor_map_2d(&mw, b_q, 1, n, k, k, TN, BK, true);
  if (rc != INFEROP_OK) return rc;
  rc = make_tensor_map_2d(&ma, a_q, 1, m, k, k, mp, BK, true);
  if (rc != INFEROP_OK) return rc;
  if (out_dt < 0 || out_dt > 2) return INFEROP_ERR_DTYPE;
  if (clear_counters > 0) {
    // everything that can reject the call has been checked: nothing is left on the stream by a rejected call
    const cudaError_t e = cudaMemsetAsync(counters, 0, static_cast<size_t>(clear_counters) * sizeof(int), stream);
    if (e != cudaSuccess) return note_cuda_error(e);
  }
  const Cut cut = decode_cut(ctx->sm_count, m, n, k, false);
  if (cut.splits != 1 && !workspace) return INFEROP_ERR_LIMIT;   // (an option changed since decode_needs_scratch)
  p.splits = cut.splits;
  switch (out_dt) {
    case 0: return launch_decode_mp<float>(mp, mw, ma, p, cut.ctas, stream);
    case 1: return launch_decode_mp<__half>(mp, mw, ma, p, cut.ctas, stream);
    case 2: return launch_decode_mp<__nv_bfloat16>(mp, mw, ma, p, cut.ctas, stream);
    default: return INFEROP_ERR_DTYPE;
  }
}

}  // namespace ib200

// ---------------------------------------------------------------------------
// Entry point that allocates nothing.
//
// Some callers cannot let a library call cudaMalloc on their behalf: a serving process that
// handed all of the device's memory to its own pool at start-up (weights, KV cache) has none
// left for the driver to give out, and a latency-critical loop cannot afford an allocation
// call that may take driver locks or synchronise the device.  For them the split-tile scratch
// of the small-M kernel lives in a fixed array inside the library image instead of in memory
// obtained at run time.  Every GPU that loads the library carries the array (about 5.3 MB)
// until the process exits, which is why it is kept small: M <= 32 tokens, at most 4096 weight
// tiles (N <= 524288) and at most 160 SMs.
// ---------------------------------------------------------------------------
namespace ib200 {
namespace {

constexpr int kFixedMaxM = 32;
constexpr int kFixedMaxCtas = 160;
constexpr int kFixedMaxTiles = 4096;

struct FixedScratch {
  float partials[kFixedMaxCtas * 2 * kFixedMaxM * TN];  // two K parts of split tiles per CTA
  int counters[kFixedMaxTiles];                     // arrivals per tile; zero between launches
  DeviceStatus status;                              // bounded-wait record of this entry point
};

// The scratch itself.  In host code this name is only a handle for cudaGetSymbolAddress; the
// device address obtained from it is what the kernel receives.
static __device__ __align__(256) unsigned char g_fixed_scratch[sizeof(FixedScratch)];

struct FixedScratchPtr {
  FixedScratch* ptr = nullptr;
  int sm_count = 0;
  int sm_version = 0;
};

FixedScratchPtr g_fixed_cache[64];
std::mutex g_fixed_mutex;

FixedScratch* fixed_scratch_cached(int dev) {
  std::lock_guard<std::mutex> lock(g_fixed_mutex);
  return g_fixed_cache[dev].ptr;
}

// Device address of the scratch on the current device, resolved once per device.
int fixed_scratch_for_current_device(FixedScratchPtr* out) {
  FixedScratchPtr* cache = g_fixed_cache;
  std::mutex& m = g_fixed_mutex;
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return note_cuda_error(e);
  if (dev < 0 || dev >= 64) return INFEROP_ERR_LIMIT;
  std::lock_guard<std::mutex> lock(m);
  if (!cache[dev].ptr) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_fixed_scratch);
    if (e != cudaSuccess || !p) return note_cuda_error(e == cudaSuccess ? cudaErrorInvalidSymbol : e);
    int major = 0, minor = 0, sms = 0;
    if ((e = cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev)) != cudaSuccess ||
        (e = cudaDeviceGetAttribute(&minor, cudaDevAttrComputeCapabilityMinor, dev)) != cudaSuccess ||
        (e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) {
      return note_cuda_error(e);
    }
    cache[dev].sm_version = major * 10 + minor;
    cache[dev].sm_count = sms;
    cache[dev].ptr = static_cast<FixedScratch*>(p);
  }
  *out = cache[dev];
  return INFEROP_OK;
}

}  // namespace
}  // namespace ib200

extern "C" int inferop_w8a8_block_fp8_gemm_fixed_scratch(void* c, const void* a_q, const void* a_scales,
                                                         const void* b_q, const void* b_scales, int64_t m,
                                                         int64_t n, int64_t k, int32_t group_size,
                                                         int32_t block_n, int32_t out_dt, void* stream) {
  using namespace ib200;
  if (group_size != 128 || block_n != 128 || k < 0 || k % 128 != 0 || m <= 0 || n <= 0) {
    return INFEROP_ERR_SHAPE;
  }
  if (out_dt < 0 || out_dt > 2) return INFEROP_ERR_DTYPE;
  if (m > kFixedMaxM || (n + TN - 1) / TN > kFixedMaxTiles || k > 0x7FFFFF00LL) return INFEROP_ERR_LIMIT;
  if (!c) return INFEROP_ERR_POINTER;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (k == 0) {  // empty sum: zeros, as the regular entry point (and the reference's kernel) stores
    const cudaError_t e = cudaMemsetAsync(c, 0, static_cast<size_t>(m) * n * (out_dt == 0 ? 4 : 2), s);
    return e == cudaSuccess ? INFEROP_OK : note_cuda_error(e);
  }
  if (!a_q || !a_scales || !b_q || !b_scales) return INFEROP_ERR_POINTER;
  if ((reinterpret_cast<uintptr_t>(a_q) & 15u) || (reinterpret_cast<uintptr_t>(b_q) & 15u)) {
    return INFEROP_ERR_POINTER;
  }
  FixedScratchPtr fs;
  const int rc = fixed_scratch_for_current_device(&fs);
  if (rc != INFEROP_OK) return rc;
  if (fs.sm_version != 100) return INFEROP_ERR_ARCH;
  if (fs.sm_count > kFixedMaxCtas) return INFEROP_ERR_LIMIT;
  DeviceCtx local;  // carries the SM count and the status slot to the launcher; owns nothing
  local.ordinal = 0;
  local.sm_version = fs.sm_version;
  local.sm_count = fs.sm_count;
  local.status = &fs.ptr->status;
  // the array keeps whatever the last call left: where tiles are split, the launcher zeroes the arrival counters of
  // this call's tiles on the stream, after its last check and before the kernel
  const int tiles = decode_needs_scratch(fs.sm_count, m, n, k, false) ? static_cast<int>((n + TN - 1) / TN) : 0;
  if (const int parts = split_gemm_parts(m, n, k))   // needs no scratch
    return launch_gemm_split_to(&local, parts, &c, 1, n, 0, a_q, a_scales, b_q, b_scales, m, n, k, out_dt, true, s);
  return launch_gemm_decode(&local, fs.ptr->partials, fs.ptr->counters, c, a_q, a_scales, b_q, b_scales,
                            m, n, k, out_dt, s, tiles);
}

// The bounded-wait record of the fixed-scratch entry point on the current device, for
// inferop_device_status: nothing is read (and *used = false) when that entry point has not
// run on this device yet.  Allocates nothing.
int ib200::fixed_scratch_status(DeviceStatus* out, bool reset, bool* used) {
  *used = false;
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return note_cuda_error(e);
  if (dev < 0 || dev >= 64) return INFEROP_OK;
  FixedScratch* ptr = fixed_scratch_cached(dev);
  if (!ptr) return INFEROP_OK;
  e = cudaMemcpy(out, &ptr->status, kStatusRecordBytes, cudaMemcpyDeviceToHost);
  if (e != cudaSuccess) return note_cuda_error(e);
  if (reset) {
    e = cudaMemset(&ptr->status, 0, kStatusRecordBytes);
    if (e != cudaSuccess) return note_cuda_error(e);
  }
  *used = true;
  return INFEROP_OK;
}
