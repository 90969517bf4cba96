// Paged attention, single-token decode with grouped-query heads, 16-bit types, on the tensor cores
// (same contract as attention.cu; reference kernels/attention/paged_attn_decode.cu:26-118).
//
// The step is a stream of the sequences' K and V rows from HBM; what has to be kept small is
// everything else that an SM does per row.
//   * Scores and the weighted sum are matrix products (mma.sync m16n8k16): up to eight query heads
//     that share a KV head are rows 0-7 of the A operand, 16 tokens at a time the other side.  The
//     CUDA-core form of this step spent 4 x 2 FMAs per element of K and V and a shuffle tree per
//     token and was bound by instruction issue (72 % of the slots at 4.6 TB/s).
//   * The probabilities keep their fp32 value: p = hi + lo + rest in the 16-bit type, hi in rows 0-7 and
//     the remainders in rows 8-15 of two MMAs (rows 8-15 would be idle otherwise): 24 bits, in fp16 of
//     p 2^15, so that they hold from 1 down to 2^-15 and an absolute step of 2^-39 remains below.  Their sums
//     over the steps are fp32 additions, of hi by itself: an infinity of V is an infinity of that sum (join_parts).
//   * Every warp streams 16-token blocks of its own through a cp.async ring in shared memory
//     (16-byte chunks, chunk index xor row, so that ldmatrix is free of bank conflicts); no
//     block-wide synchronisation inside a sequence.
//   * The work is cut evenly: the 64-token units of all (sequence, head group) pairs form one list,
//     and CTA c takes units [c S, (c + 1) S) of it, whatever the lengths of the sequences.  The
//     lengths are read on the device (no host step).  A pair that spans CTAs leaves partial
//     states in the workspace; the CTA that finishes last adds them in list order (the result does
//     not depend on arrival order) -- no second launch.
//
// Bound by HBM for large batches.  Measured (bf16, 32 heads over 8 KV heads of 128, blocks of 16 in
// random order; the CUDA-core form in brackets): 64 x 4096 tokens 173.5 us = 6.2 TB/s (224 us), 128
// sequences of 500-2000 tokens 120 us = 5.5 TB/s (176 us), one sequence of 65536 58 us (75 us), 3 of
// 5000-20000 36.5 us (60 us); 28 heads over 4 KV heads, 64 x 2048: 55 us (232 us).  ncu on the first: DRAM bytes =
// the cache, issue slots 37 % busy (72 % in the CUDA-core form), tensor pipe 28 %.  Calls that it does not
// gain on take the other form: paged_attn_on_tensor_cores.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "internal.h"

namespace ib200 {
namespace {

constexpr int kWarps = 4;
constexpr int kThreads = 32 * kWarps;
constexpr int kTok = 16;              // tokens of a warp per step
constexpr int kUnit = kWarps * kTok;  // tokens of the CTA per step: the unit the work is cut in
constexpr int kRows = 8;              // query heads per CTA at most
// Up to so many sequences the pairs are cut evenly.  More balance by themselves, and every CTA searches all
// lengths: 1030 to 4000 sequences, 3 % of them sixteen times as long as the rest or all equal, were 0.7 to 1.07
// times as fast when cut.
constexpr int kMaxBatchCut = 1024;
constexpr int kSms = 148;             // of a B200: the CTAs that workspace, weights and counters are laid out for

template <int D>
struct MCfg {
  static constexpr int kRowBytes = 2 * D;
  static constexpr int kChunks = D / 8;                 // 16-byte chunks of a row
  static constexpr int kTileBytes = kTok * kRowBytes;   // a warp step's K (or V) rows
  static constexpr int kStageBytes = 2 * kTileBytes;
  static constexpr int kStages = D == 64 ? 6 : 3;
  static constexpr int kCtasPerSm = D == 256 ? 1 : 2;
  static constexpr int kRec = D + 2;                    // a warp's state of a head: accumulator, maximum (base 2), denominator
  static constexpr int kPart = kRows * (D + 2);         // a CTA's part of a pair: [kRows][D] sums, [kRows][2] maximum and denominator
  static constexpr int kRingBytes = kWarps * kStages * kStageBytes;
  static constexpr int kStateFloats = kWarps * kRows * kRec;
  static constexpr int kWeightFloats = kRows * kSms * kCtasPerSm;
  static constexpr int kMergeBytes = 4 * (kStateFloats > kWeightFloats ? kStateFloats : kWeightFloats);
  static constexpr int kSmemBytes = kRingBytes + kMergeBytes;
};
// (1 KiB per CTA is the system's; the kernel's static variables take less than 256 bytes)
static_assert(2 * (MCfg<64>::kSmemBytes + 1280) <= 233472 && 2 * (MCfg<128>::kSmemBytes + 1280) <= 233472, "two CTAs per SM");
static_assert(kSms * MCfg<64>::kCtasPerSm <= AttnSet::kCounters && kSms * MCfg<128>::kCtasPerSm <= AttnSet::kCounters,
              "a counter per CTA");
static_assert(MCfg<256>::kSmemBytes + 256 <= 232448, "one CTA per SM");

struct MmaAttnParams {
  void* out;
  const void* q;
  const void* k_cache;
  const void* v_cache;
  const int32_t* block_tables;
  const int32_t* seq_lens;
  float* partial;      // [CTA][2] parts of kPart floats
  int* counters;       // [CTA], zero at the start, this launch's alone
  int batch, num_heads, num_kv_heads, block_size, block_shift, max_blocks;   // block_shift: log2(block_size) or -1
  int gt, groups;      // query heads per CTA, head groups per sequence
  int whole;           // 1: no workspace, CTA i takes the whole of pair i
  int q_words;         // q may be read in 32-bit words
  float scale_log2e;
};

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// What exponents are taken relative to: 0 as long as every score was -inf (their p is 0, not NaN).
__device__ __forceinline__ float finite_max(float m) { return m == -INFINITY ? 0.0f : m; }

// The sum of a head's leading parts and that of the remainders.  An infinite V makes the second
// NaN (a remainder is often zero or negative) while the first has the infinity that p V has.
__device__ __forceinline__ float join_parts(float lead, float remainder) {
  return fabsf(lead) < INFINITY ? lead + remainder : lead;
}

// a += b, two sums per instruction where kPairs
template <bool kPairs>
__device__ __forceinline__ void add4(float (&a)[4], const float (&b)[4]) {
#pragma unroll
  for (int i = 0; i < 4; i += 2) {
    if (kPairs) {
      asm("{\n\t.reg .b64 x, y;\n\tmov.b64 x, {%0, %1};\n\tmov.b64 y, {%2, %3};\n\tadd.rn.f32x2 x, x, y;\n\tmov.b64 {%0, %1}, x;\n\t}"
          : "+f"(a[i]), "+f"(a[i + 1])
          : "f"(b[i]), "f"(b[i + 1]));
    } else {
      a[i] += b[i];
      a[i + 1] += b[i + 1];
    }
  }
}

template <typename T>
struct Ops16;
template <>
struct Ops16<__nv_bfloat16> {
  static constexpr float kScale = 1.0f;   // the exponent range of fp32
  static __device__ __forceinline__ float floor_of(float p) { return p; }
  static __device__ __forceinline__ uint32_t pack(float a, float b) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
  }
  static __device__ __forceinline__ float2 unpack(uint32_t w) {
    return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xFFFF0000u));
  }
  static __device__ __forceinline__ __nv_bfloat16 narrow(float v) { return __float2bfloat16_rn(v); }
  // (the product alone)
  static __device__ __forceinline__ void mma_first(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                                   uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.0f));
  }
  static __device__ __forceinline__ void mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                             uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  }
};
template <>
struct Ops16<__half> {
  // p <= 1 is summed as p 2^15: the parts have steps of 2^-39 then.  Without it the steps are 2^-24, and tokens
  // of 2^-25 and less are lost from the sum while the denominator has them.
  static constexpr float kScale = 32768.0f;
  // no leading part of a positive p is zero (2 x 2^-24; the remainder takes the difference back)
  static __device__ __forceinline__ float floor_of(float p) { return p > 0.0f ? fmaxf(p, 1.1920929e-7f) : p; }
  static __device__ __forceinline__ uint32_t pack(float a, float b) {
    const __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
  }
  static __device__ __forceinline__ float2 unpack(uint32_t w) { return __half22float2(*reinterpret_cast<const __half2*>(&w)); }
  static __device__ __forceinline__ __half narrow(float v) { return __float2half_rn(v); }
  // (the product alone)
  static __device__ __forceinline__ void mma_first(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                                   uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.0f));
  }
  static __device__ __forceinline__ void mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                             uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  }
};

__device__ __forceinline__ void ldsm4(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}
__device__ __forceinline__ void ldsm4_trans(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}

__device__ __forceinline__ int clamped_len(const MmaAttnParams& p, int b) {
  const int len = __ldg(p.seq_lens + b);
  const int cap = p.max_blocks * p.block_size;
  return len < 0 ? 0 : (len > cap ? cap : len);
}
// an empty sequence counts one unit: its zeros have to be written by somebody
__device__ __forceinline__ int units_of(int len) { return len <= 0 ? 1 : (len + kUnit - 1) / kUnit; }

// A place in the CTA's run of units: pair (b, gi), first token of the unit, end of the sequence.
struct Cursor {
  int b, gi, t, len;
  int left;   // units of the CTA from here on
  __device__ __forceinline__ void next(const MmaAttnParams& p) {
    --left;
    t += kUnit;
    if (t >= len && left > 0) {
      t = 0;
      if (++gi == p.groups) {
        gi = 0;
        ++b;
        len = clamped_len(p, b);
      }
    }
  }
};

template <typename T, int D>
__global__ void __launch_bounds__(kThreads, MCfg<D>::kCtasPerSm)
paged_attn_mma_kernel(const MmaAttnParams p) {
  using C = MCfg<D>;
  using O = Ops16<T>;
  extern __shared__ __align__(128) uint8_t smem[];
  float* states = reinterpret_cast<float*>(smem + C::kRingBytes);
  __shared__ int sh_last;
  const int lane = threadIdx.x & 31;
  const int warp = __shfl_sync(0xFFFFFFFFu, static_cast<int>(threadIdx.x >> 5), 0);
  const int row = lane >> 2;        // head row of this lane's accumulators
  const int quad = lane & 3;

  // q, the cache, the tables and the lengths may come from the kernel queued before this one; dependents are
  // not signalled early: the outputs are whole when a kernel behind this one starts, however it is launched
  pdl_wait();

  // ---- this CTA's run of units
  long long share = 0, u0 = 0;   // (whole: unused)
  Cursor use;
  if (p.whole) {
    use.b = blockIdx.x / p.groups;
    use.gi = blockIdx.x % p.groups;
    use.t = 0;
    use.len = clamped_len(p, use.b);
    use.left = units_of(use.len);
  } else {
    // every warp on its own, no barrier: the lengths are a few cache lines, and the first of them
    // stay in registers between the sum and the search
    const int mine0 = lane < p.batch ? units_of(clamped_len(p, lane)) : 0;
    long long sum = mine0;
    int longest = mine0;
    for (int b = lane + 32; b < p.batch; b += 32) {
      const int ub = units_of(clamped_len(p, b));
      sum += ub;
      longest = max(longest, ub);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      sum += __shfl_xor_sync(0xFFFFFFFFu, sum, o);
      longest = max(longest, __shfl_xor_sync(0xFFFFFFFFu, longest, o));
    }
    const long long total = sum * p.groups;
    share = (total + gridDim.x - 1) / gridDim.x;
    // The CTA that merges a pair reads its parts one batch after another, so a pair of U units goes to no more
    // than about sqrt(5 U) CTAs, where a unit's time and a part's balance.  One sequence of 16384 tokens, 8 heads
    // over one KV head of 128: 118 us on 256 CTAs, 20 us on 32 (with the merge below); 65536 tokens: 115 us on
    // 256, 33 us on 69.  sqrt(2 U) CTAs were up to a third slower, sqrt(10 U) between 30 % faster and 25 %
    // slower.  With a dozen pairs and more the even share is the larger one.
    share = max(share, static_cast<long long>(ceilf(sqrtf(0.2f * static_cast<float>(longest)))));
    u0 = share * blockIdx.x;
    if (u0 >= total) return;   // (the whole CTA)
    // the sequence that unit u0 belongs to: an inclusive scan over the lengths, 32 at a time
    long long before = 0;
    for (int b0 = 0;; b0 += 32) {
      const int b = b0 + lane;
      const int ub = b0 == 0 ? mine0 : (b < p.batch ? units_of(clamped_len(p, b)) : 0);
      const long long mine = static_cast<long long>(ub) * p.groups;
      long long inc = mine;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const long long v = __shfl_up_sync(0xFFFFFFFFu, inc, o);
        if (lane >= o) inc += v;
      }
      const unsigned hit = __ballot_sync(0xFFFFFFFFu, u0 < before + inc);
      if (hit != 0u) {
        const int src = __ffs(hit) - 1;
        const int r = static_cast<int>(u0 - before - __shfl_sync(0xFFFFFFFFu, inc - mine, src));
        const int units = __shfl_sync(0xFFFFFFFFu, ub, src);
        use.b = b0 + src;
        use.gi = r / units;
        use.t = (r - use.gi * units) * kUnit;
        break;
      }
      before += __shfl_sync(0xFFFFFFFFu, inc, 31);
    }
    use.len = clamped_len(p, use.b);
    use.left = static_cast<int>(min(share, total - u0));
  }

  const int my_units = use.left;

  // ---- producer: rows of one step of this warp, 16 tokens of K and of V
  const uint32_t ring = smem_u32(smem) + warp * (C::kStages * C::kStageBytes);
  const int gpk = (p.num_heads / p.num_kv_heads) / p.gt;   // head groups per KV head
  const int64_t row_elems = static_cast<int64_t>(p.num_kv_heads) * D;
  Cursor pre = use;
  // lane l looks up the row of token l (mod 16) of a step, one step before its copies are issued
  auto lookup = [&](const Cursor& c) -> uint32_t {
    const int t = c.t + warp * kTok + (lane & (kTok - 1));
    if (c.left <= 0 || t >= c.len) return 0xFFFFFFFFu;
    const int bi = p.block_shift >= 0 ? t >> p.block_shift : t / p.block_size;
    const int off = t - bi * p.block_size;
    return static_cast<uint32_t>(__ldg(p.block_tables + static_cast<int64_t>(c.b) * p.max_blocks + bi)) *
               static_cast<uint32_t>(p.block_size) + static_cast<uint32_t>(off);
  };
  uint32_t rows = lookup(pre);
  auto issue = [&](int slot) {
    const uint32_t dst = ring + slot * C::kStageBytes;
    const int kvh = pre.gi / gpk;
    const T* kb = static_cast<const T*>(p.k_cache) + kvh * D;
    const T* vb = static_cast<const T*>(p.v_cache) + kvh * D;
    const bool any = pre.left > 0 && pre.t + warp * kTok < pre.len;   // warp-uniform
    const uint32_t now = rows;
    if (pre.left > 0) {
      pre.next(p);
      rows = lookup(pre);
    }
    if (any) {
#pragma unroll
      for (int i = 0; i < kTok * C::kChunks / 32; ++i) {
        const int c = i * 32 + lane;
        const int r = c / C::kChunks, col = c % C::kChunks;
        const uint32_t token = __shfl_sync(0xFFFFFFFFu, now, r);
        // tokens beyond the sequence are zeros (never stale bytes: 0 x NaN would reach the sums)
        const int bytes = token == 0xFFFFFFFFu ? 0 : 16;
        const int64_t at = static_cast<int64_t>(bytes ? token : 0u) * row_elems + col * 8;
        const uint32_t d = dst + r * C::kRowBytes + ((col ^ (r & 7)) << 4);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(kb + at), "r"(bytes) : "memory");
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d + C::kTileBytes), "l"(vb + at), "r"(bytes)
                     : "memory");
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // the query rows of a pair as A fragments; requested before anything waits for them
  uint32_t qa[D / 16][2];
  auto load_q = [&](const Cursor& c) {
    const int kvh = c.gi / gpk;
    const int head0 = kvh * (p.num_heads / p.num_kv_heads) + (c.gi - kvh * gpk) * p.gt;
    const uint16_t* qrow = static_cast<const uint16_t*>(p.q) + (static_cast<int64_t>(c.b) * p.num_heads + head0 + row) * D;
#pragma unroll
    for (int kk = 0; kk < D / 16; ++kk) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int e = kk * 16 + h * 8 + quad * 2;
        uint32_t w = 0;
        if (row < p.gt) {
          if (p.q_words) w = __ldg(reinterpret_cast<const uint32_t*>(qrow + e));
          else w = static_cast<uint32_t>(qrow[e]) | (static_cast<uint32_t>(qrow[e + 1]) << 16);
        }
        qa[kk][h] = w;
      }
    }
  };
  load_q(use);
#pragma unroll
  for (int s = 0; s < C::kStages - 1; ++s) issue(s);

  // ldmatrix addresses inside a tile: K rows as they are (n = token), V transposed (k = token)
  const int mi = lane >> 3, mr = lane & 7;
  const uint32_t k_row = ((mi >> 1) * 8 + mr) * C::kRowBytes;
  const uint32_t v_row = C::kTileBytes + ((mi & 1) * 8 + mr) * C::kRowBytes;

  int slot = 0;
  while (use.left > 0) {
    // ---- a pair (or the part of it that is this CTA's)
    const int b = use.b, gi = use.gi, len = use.len, t_first = use.t;
    const int kvh = gi / gpk;
    const int head0 = kvh * (p.num_heads / p.num_kv_heads) + (gi - kvh * gpk) * p.gt;
    float acc[D / 8][4];
#pragma unroll
    for (int j = 0; j < D / 8; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.0f;
    float m = -INFINITY, l = 0.0f;
    const long long seg_u = u0 + (my_units - use.left);   // unit index of this segment's first unit
    int t_last;
    bool end;
    do {
      __syncwarp();   // every lane has read the slot that is filled next
      {
        int ahead = slot + C::kStages - 1;
        if (ahead >= C::kStages) ahead -= C::kStages;
        issue(ahead);
      }
      asm volatile("cp.async.wait_group %0;" ::"n"(C::kStages - 1) : "memory");
      __syncwarp();   // the other lanes' copies of this step are there too
      const int tw = use.t + warp * kTok;
      if (tw < len) {
        const uint32_t base = ring + slot * C::kStageBytes;
        float sc[2][4] = {};
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
          uint32_t kf[4];
          ldsm4(base + k_row + (((2 * kk + (mi & 1)) ^ mr) << 4), kf);
          O::mma(sc[0], qa[kk][0], 0u, qa[kk][1], 0u, kf[0], kf[1]);
          O::mma(sc[1], qa[kk][0], 0u, qa[kk][1], 0u, kf[2], kf[3]);
        }
        // scores of head `row` for tokens 2 quad, + 1 of either half of the block
        float s[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int t = tw + (i >> 1) * 8 + quad * 2 + (i & 1);
          s[i] = t < len ? sc[i >> 1][i & 1] * p.scale_log2e : -INFINITY;
        }
        float mx = fmaxf(fmaxf(s[0], s[1]), fmaxf(s[2], s[3]));
        mx = fmaxf(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, 1));
        mx = fmaxf(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, 2));
        if (__any_sync(0xFFFFFFFFu, mx > m)) {
          // a new maximum (always in the first step, rare later): the state is rescaled
          const float m_new = fmaxf(m, mx);
          const float alpha = ex2(m - finite_max(m_new));
          m = m_new;
          l *= alpha;
#pragma unroll
          for (int j = 0; j < D / 8; ++j) {
            acc[j][0] *= alpha;
            acc[j][1] *= alpha;
            acc[j][2] *= alpha;
            acc[j][3] *= alpha;
          }
        }
        float pr[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) pr[i] = ex2(s[i] - finite_max(m));   // 0 for a missing token
        l += (pr[0] + pr[1]) + (pr[2] + pr[3]);
#pragma unroll
        for (int i = 0; i < 4; ++i) pr[i] *= O::kScale;
        // rows 0-7 take the leading part of p, half of it in either MMA (zeros in the second would be 0 x inf
        // under an infinite V), rows 8-15 the two remainders
        uint32_t hi[2], lo[2], rest[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          hi[h] = O::pack(0.5f * O::floor_of(pr[2 * h]), 0.5f * O::floor_of(pr[2 * h + 1]));
          const float2 a = O::unpack(hi[h]);
          const float r0 = fmaf(a.x, -2.0f, pr[2 * h]), r1 = fmaf(a.y, -2.0f, pr[2 * h + 1]);   // exact
          lo[h] = O::pack(r0, r1);
          const float2 c = O::unpack(lo[h]);
          rest[h] = O::pack(r0 - c.x, r1 - c.y);
        }
#pragma unroll
        for (int j = 0; j < D / 8; j += 2) {
          uint32_t vf[4];
          ldsm4_trans(base + v_row + (((j + (mi >> 1)) ^ mr) << 4), vf);
          // The tensor cores truncate their sums, fp32 additions round: products of a step are summed there, the
          // steps by additions (a chain of MMAs left 6e-6 of a sum of 20000 tokens, 40 times the error of fp32
          // additions; 171.5 -> 173.5 us at 64 x 4096 tokens).
          float p0[4], p1[4];
          O::mma_first(p0, hi[0], lo[0], hi[1], lo[1], vf[0], vf[1]);
          O::mma_first(p1, hi[0], lo[0], hi[1], lo[1], vf[2], vf[3]);
          O::mma(p0, hi[0], rest[0], hi[1], rest[1], vf[0], vf[1]);
          O::mma(p1, hi[0], rest[0], hi[1], rest[1], vf[2], vf[3]);
          add4<D <= 128>(acc[j], p0);   // (size 256 has no registers for the pairs: 97 us for 88)
          add4<D <= 128>(acc[j + 1], p1);
        }
      }
      if (++slot == C::kStages) slot = 0;
      t_last = use.t;
      end = use.t + kUnit >= len || use.left == 1;
      use.next(p);
    } while (!end);

    if (use.left > 0) load_q(use);

    // ---- the four warps' states -> one
    l += __shfl_xor_sync(0xFFFFFFFFu, l, 1);
    l += __shfl_xor_sync(0xFFFFFFFFu, l, 2);
    if (row < p.gt) {
      float* st = states + (warp * kRows + row) * C::kRec;
#pragma unroll
      for (int j = 0; j < D / 8; ++j)
        *reinterpret_cast<float2*>(st + j * 8 + quad * 2) =
            make_float2(join_parts(acc[j][0], acc[j][2]) * (1.0f / O::kScale), join_parts(acc[j][1], acc[j][3]) * (1.0f / O::kScale));
      if (quad == 0) {
        st[D] = m;
        st[D + 1] = l;
      }
    }
    __syncthreads();
    const bool before = t_first > 0;                                            // the pair began in an earlier CTA
    const bool after = use.left == 0 && t_last + kUnit < len;                    // ... goes on in a later one
    const bool split = before || after;
    float* rec = p.partial + (static_cast<int64_t>(blockIdx.x) * 2 + (before ? 0 : 1)) * C::kPart;
    for (int idx = threadIdx.x; idx < p.gt * D; idx += kThreads) {
      const int g = idx / D, d = idx % D;
      const float* st = states + g * C::kRec;
      float mm = -INFINITY;
#pragma unroll
      for (int w = 0; w < kWarps; ++w) mm = fmaxf(mm, st[w * kRows * C::kRec + D]);
      float a = 0.0f, ll = 0.0f;
#pragma unroll
      for (int w = 0; w < kWarps; ++w) {
        const float mw = st[w * kRows * C::kRec + D];
        const float f = mw == -INFINITY ? 0.0f : exp2f(mw - mm);
        a = fmaf(st[w * kRows * C::kRec + d], f, a);
        ll = fmaf(st[w * kRows * C::kRec + D + 1], f, ll);
      }
      if (!split) {
        static_cast<T*>(p.out)[(static_cast<int64_t>(b) * p.num_heads + head0 + g) * D + d] = O::narrow(len <= 0 ? 0.0f : a / ll);
      } else {
        __stcg(rec + idx, a);
        if (d == 0) __stcg(reinterpret_cast<float2*>(rec + kRows * D) + g, make_float2(mm, ll));
      }
    }
    if (split) {
      // the pair's CTAs: c_lo (its last segment, record 1) ... c_hi (its first, record 0 like those between)
      const long long pair_u = seg_u - t_first / kUnit;
      const int c_lo = static_cast<int>(pair_u / share);
      const int c_hi = static_cast<int>((pair_u + units_of(len) - 1) / share);
      const int parts = c_hi - c_lo + 1;
      __threadfence();
      __syncthreads();
      if (threadIdx.x == 0) sh_last = atomicAdd(p.counters + c_lo, 1) == parts - 1;
      __syncthreads();
      if (sh_last) {
        __threadfence();
        const float* first = p.partial + (static_cast<int64_t>(c_lo) * 2 + 1) * C::kPart;   // part i > 0: 2 i - 1 records on
        auto part = [&](int i) { return first + (i == 0 ? 0 : 2 * i - 1) * C::kPart; };
        // weights of the parts, two heads per warp: states[head * parts + part]
        {
          float mm[2] = {-INFINITY, -INFINITY}, ll[2] = {0.0f, 0.0f};
          for (int i = lane; i < parts; i += 32) {
            float2 v[2];
#pragma unroll
            for (int e = 0; e < 2; ++e)
              if (warp + e * kWarps < p.gt) v[e] = __ldcg(reinterpret_cast<const float2*>(part(i) + kRows * D) + warp + e * kWarps);
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              if (warp + e * kWarps >= p.gt) break;
              const float m_new = fmaxf(mm[e], v[e].x), ref = finite_max(m_new);
              ll[e] = fmaf(ll[e], exp2f(mm[e] - ref), v[e].y * exp2f(v[e].x - ref));
              mm[e] = m_new;
              states[(warp + e * kWarps) * parts + i] = v[e].x;
            }
          }
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int g = warp + e * kWarps;
            if (g >= p.gt) break;
            float m_all = mm[e];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) m_all = fmaxf(m_all, __shfl_xor_sync(0xFFFFFFFFu, m_all, o));
            m_all = finite_max(m_all);
            float l_all = ll[e] * exp2f(mm[e] - m_all);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) l_all += __shfl_xor_sync(0xFFFFFFFFu, l_all, o);
            const float inv = 1.0f / l_all;
            for (int i = lane; i < parts; i += 32) states[g * parts + i] = exp2f(states[g * parts + i] - m_all) * inv;
          }
        }
        __syncthreads();
        // the sums: a thread's four-element columns side by side, eight loads in flight (sixteen make the stream spill)
        constexpr int kCols = kRows * D / 4 / kThreads;
        constexpr int kBatch = 8 / kCols;
        float4 a[kCols];
#pragma unroll
        for (int j = 0; j < kCols; ++j) a[j] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        for (int i0 = 0; i0 < parts; i0 += kBatch) {
          float4 v[kCols][kBatch];
#pragma unroll
          for (int j = 0; j < kCols; ++j) {
            const int idx = threadIdx.x + j * kThreads;
            if (idx >= p.gt * D / 4) break;
#pragma unroll
            for (int e = 0; e < kBatch; ++e) {
              asm volatile("ld.global.cg.v4.f32 {%0, %1, %2, %3}, [%4];"
                           : "=f"(v[j][e].x), "=f"(v[j][e].y), "=f"(v[j][e].z), "=f"(v[j][e].w)
                           : "l"(part(min(i0 + e, parts - 1)) + idx * 4));
            }
          }
#pragma unroll
          for (int j = 0; j < kCols; ++j) {
            const int idx = threadIdx.x + j * kThreads;
            if (idx >= p.gt * D / 4) break;
            const float* wg = states + idx / (D / 4) * parts;
#pragma unroll
            for (int e = 0; e < kBatch; ++e) {
              if (i0 + e >= parts) break;   // (not a weight of zero: the sum may be infinite)
              const float w = wg[i0 + e];
              a[j].x = fmaf(v[j][e].x, w, a[j].x);
              a[j].y = fmaf(v[j][e].y, w, a[j].y);
              a[j].z = fmaf(v[j][e].z, w, a[j].z);
              a[j].w = fmaf(v[j][e].w, w, a[j].w);
            }
          }
        }
#pragma unroll
        for (int j = 0; j < kCols; ++j) {
          const int idx = threadIdx.x + j * kThreads;
          if (idx >= p.gt * D / 4) break;
          T* dst = static_cast<T*>(p.out) + (static_cast<int64_t>(b) * p.num_heads + head0) * D + idx * 4;
          dst[0] = O::narrow(a[j].x);
          dst[1] = O::narrow(a[j].y);
          dst[2] = O::narrow(a[j].z);
          dst[3] = O::narrow(a[j].w);
        }
      }
    }
    __syncthreads();   // the states may be overwritten now
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// the largest divisor of the group that fits the rows
int heads_per_pair(int group) {
  int gt = kRows;
  while (group % gt != 0) --gt;
  return gt;
}

template <typename T, int D>
int launch_d(MmaAttnParams p, int sm_count, bool pdl, cudaStream_t stream) {
  using C = MCfg<D>;
  static bool attr_done[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !attr_done[dev]) {
    const cudaError_t e = cudaFuncSetAttribute(paged_attn_mma_kernel<T, D>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               C::kSmemBytes);
    if (e != cudaSuccess) return note_cuda_error(e);
    attr_done[dev] = true;
  }
  const int64_t pairs = static_cast<int64_t>(p.batch) * p.groups;
  int64_t ctas = pairs;
  if (!p.whole) {
    // as many CTAs as are resident at once, but no more than the tables could fill
    const int64_t most = pairs * ((static_cast<int64_t>(p.max_blocks) * p.block_size + kUnit - 1) / kUnit);
    ctas = static_cast<int64_t>(sm_count < kSms ? sm_count : kSms) * C::kCtasPerSm;
    if (ctas > most) ctas = most;   // (two units per CTA at least: 7.8 instead of 5.2 us for one sequence of 64 tokens)
  }
  if (ctas > 0x7FFFFFFF) return INFEROP_ERR_LIMIT;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(ctas));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = C::kSmemBytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl ? 1 : 0;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, paged_attn_mma_kernel<T, D>, p);
  if (e != cudaSuccess) return note_cuda_error(e);
  return check_launch();
}

template <typename T>
int launch_t(const MmaAttnParams& p, int head_dim, int sm_count, bool pdl, cudaStream_t stream) {
  switch (head_dim) {
    case 64: return launch_d<T, 64>(p, sm_count, pdl, stream);
    case 128: return launch_d<T, 128>(p, sm_count, pdl, stream);
    case 256: return launch_d<T, 256>(p, sm_count, pdl, stream);
    default: return INFEROP_ERR_SHAPE;
  }
}

}  // namespace

// Which 16-bit calls come here; the others take attention.cu.  Both forms were timed on 550 shapes per type: head
// sizes 64, 128 and 256, one to eight query heads per KV head, 1 to 4000 sequences of 64 to 65536 tokens, all
// equal or ragged down to a quarter.  The figures are the other form's time over this one's, equal / ragged.  A pair
// costs this form about 5 us whatever its length, with two in flight per SM (one at head size 256) where the
// other has four; its gain is that a K / V row is read and multiplied once for up to eight heads.  So:
//   * where the other form (4, 2 or 1 heads per CTA) would fetch rows more than once: from 256 pairs or 1024
//     units on, 1.1 to 2.5 / 0.9 to 2.4 (below: 0.6 to 1.4); at head size 256 from 1024 tokens and 2048 units on,
//     1.4 to 1.9 / 1.3 to 1.9 (below: 0.5 to 1.4);
//   * four heads in either form: at head size 128 from 512 tokens and 2048 units on, or 1024 with 32 pairs and
//     more, 1.0 to 1.6 / 0.9 to 1.5 (the lower figures below 2048 units, and there the other form's second launch
//     comes on top: 8 x 1024 tokens called one by one 22.8 us, 13.4 / 16.3 here; with fewer pairs down to 0.7; 256
//     tokens and many pairs 0.8 to 1.1); at 64 from 512 tokens and 4096 units on, 1.0 to 1.35; at 256 from 4096
//     tokens and 4096 units on, 1.02 to 1.2;
//   * two heads, or one with 32 to 256 pairs: at head size 128 from 4096 tokens and 4096 units on, 1.0 to 1.3;
//     at 64 the other form is as fast or faster (0.5 to 1.1), at 256 faster (0.2 to 0.95).
bool paged_attn_on_tensor_cores(int batch, int num_heads, int num_kv_heads, int head_dim, int64_t tokens) {
  const Options& opt = options();
  if (opt.attn_path != 0) return opt.attn_path == 2;
  if (opt.attn_splits > 0 || opt.attn_heads_per_cta > 0) return false;
  const int group = num_heads / num_kv_heads;
  const int gt = heads_per_pair(group);
  const int other = group % 4 == 0 ? 4 : (group % 2 == 0 ? 2 : 1);
  const int64_t pairs = static_cast<int64_t>(batch) * (num_heads / gt);
  const int64_t units = pairs * ((tokens + kUnit - 1) / kUnit);
  if (2 * gt >= 3 * other) return head_dim <= 128 ? pairs >= 256 || units >= 1024 : tokens >= 1024 && units >= 2048;
  if (gt >= 4) {
    if (head_dim == 64) return tokens >= 512 && units >= 4096 && batch <= kMaxBatchCut;   // (uncut: 0.96 / 0.94)
    return head_dim == 128 ? tokens >= 512 && units >= (pairs >= 32 ? 1024 : 2048) : tokens >= 4096 && units >= 4096;
  }
  return head_dim == 128 && tokens >= 4096 && units >= 4096 && (gt > 1 || (pairs >= 32 && pairs <= 256));
}

size_t paged_attn_mma_workspace_bytes() {
  const size_t a = static_cast<size_t>(kSms) * MCfg<128>::kCtasPerSm * 2 * MCfg<128>::kPart * sizeof(float);
  const size_t b = static_cast<size_t>(kSms) * MCfg<256>::kCtasPerSm * 2 * MCfg<256>::kPart * sizeof(float);
  return a > b ? a : b;
}

int launch_paged_attn_mma(void* out, const void* q, const void* k_cache, const void* v_cache, const int32_t* block_tables,
                          const int32_t* seq_lens, int32_t dt, int batch, int num_heads, int num_kv_heads, int head_dim,
                          int block_size, int max_blocks_per_seq, float scale, int sm_count, float* workspace, int* counters,
                          bool pdl, cudaStream_t stream) {
  MmaAttnParams p;
  p.out = out;
  p.q = q;
  p.k_cache = k_cache;
  p.v_cache = v_cache;
  p.block_tables = block_tables;
  p.seq_lens = seq_lens;
  p.partial = workspace;
  p.counters = counters;
  p.batch = batch;
  p.num_heads = num_heads;
  p.num_kv_heads = num_kv_heads;
  p.block_size = block_size;
  p.block_shift = -1;
  for (int sh = 0; sh < 31; ++sh)
    if ((1 << sh) == block_size) p.block_shift = sh;
  p.max_blocks = max_blocks_per_seq;
  const int group = num_heads / num_kv_heads;
  p.gt = heads_per_pair(group);
  p.groups = num_heads / p.gt;

  p.whole = workspace == nullptr || batch > kMaxBatchCut ? 1 : 0;
  p.q_words = (reinterpret_cast<uintptr_t>(q) & 3u) == 0 ? 1 : 0;
  p.scale_log2e = scale * 1.4426950408889634f;
  return dt == 1 ? launch_t<__half>(p, head_dim, sm_count, pdl, stream) : launch_t<__nv_bfloat16>(p, head_dim, sm_count, pdl, stream);
}

}  // namespace ib200
