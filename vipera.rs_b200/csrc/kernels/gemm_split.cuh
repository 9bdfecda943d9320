// 32-bit matrix products of many rows on the fifth-generation tensor cores: out[M, N] = A[M, K] . W[N, K]^T with A, W
// and the sums in 32 bits.
//
// A 32-bit number is the exact sum of three bfloat16 numbers (its first 8 bits rounded to nearest, the remainder's, and
// what is left, at most 7 bits), and a product of two bfloat16 numbers is exact in 32 bits.  So a . w is a1 w1 + (a1 w2 + a2 w1
// + a2 w2 + a1 w3 + a3 w1), six products in place of one, and a2 w3 + a3 w2 + a3 w3, left out: some 2^-24 of |a w| at most, 2^-28
// on average, of either sign (parts cut off instead of rounded leave out up to 2^-21, always towards zero).  Of a number below
// 2^-110 the last part has no place in bfloat16 any more: it is held to 2^-134.  The tensor cores round
// every step of their sums towards zero, which over a long K would cost more than 32-bit multiply-adds do: so the
// leading product and the five small ones have accumulators of their own, both are read after every 64 values of K
// and added to the tile's sums in registers, rounded to nearest.  Against 64 bits the result is closer than a chain of
// fused multiply-adds over K (1,024 rows through a model of two layers and K up to 4,864: 4.3e-7 against 2.1e-6).
// An infinity or a NaN has no such parts (its products with their zeros would be NaN), nor has a number above bfloat16's
// largest.  No other row reads such a row of A or W: a block notes which of its rows hold one, writes NaN where a row holds a
// NaN, and computes the outputs of the others with multiply-adds, a warp an output.
//
// A block computes a tile of 128 x 128: eight warps read 64 values of K, split them and leave the parts in shared
// memory (three images of 128 rows each, 128-byte swizzle, two stages of 96 KB); eight warps add up, the first of which
// issues 24 products of 16 values a stage (a warp of its own for that would leave too few registers).  The left
// operand's images are written once by a kernel ahead and copied in bulk where that pays (parts_bytes), else the same
// warps split both.  Two pairs of accumulators fill tensor memory.  K is cut into up to four groups, each
// summed on its own; where the tiles are too few to fill the chip, the blocks of a cluster share the groups and add their sums
// through distributed shared memory.
// What bounds it: a stage's 24 products of 64 clocks read shared memory for all of these 1,536 clocks, and the
// images' 96 KB are written there beside them; 3,400 clocks a stage are left of that in long K, and what a block costs
// before its first and after its last stage (about six stages).  1,024 x 9,728 of 896: 188 us (multiply-adds: 503; parts
// cut off instead of rounded: 185), the left operand split in every block: 279; 8,192 x 4,096 of 4,096: 1,860 us, 148 TFLOP/s (the
// CUDA cores' own peak is 74).
#pragma once

#include "tcgen05.cuh"

namespace gemm_split {

using namespace tcgen05;

constexpr int kTile = 128, kDepth = 64, kStages = 2, kParts = 3;
constexpr int kImageBytes = kTile * kDepth * 2, kStageBytes = 2 * kParts * kImageBytes;
constexpr int kSumWarps = 8, kIssuer = 0, kFirstSplitter = 8, kSplitters = 256;   // (the first of the adding warps issues)
constexpr int kThreads = (kFirstSplitter + 8) * 32;
constexpr int kSumPitch = kTile + 4;
constexpr int kRowWords = kTile / 32;   // words of a bit per row
enum { WAIT_EXPIRED = 6 };

struct Args {
  const float* A;
  const float* W;
  int M, N, K;
  int groups, share, cluster;    // groups of `share` stages of K that are summed on their own, and how many blocks share them
  const float* bias;
  void* out;
  float* resid;
  int activation, epilogue, out_bf16;
  int* status;
  uint8_t* parts;            // the left operand's images, written ahead: [tile of rows][64 of K][part], or null
  uint32_t* odd;             // of each of those threes of images: a bit for each row with something that is not finite
  long long parts_bytes;     // what `parts` has room for (the flags lie behind the images)
};

struct Shared {
  uint64_t full[kStages], empty[kStages], sums_full[2], sums_empty[2];
  uint32_t tmem_base;
  int abort_flag;
  uint32_t odd[2 * kRowWords];   // rows of A, then of W, that hold something that is not finite
  uint32_t nan[2 * kRowWords];   // of those, the ones that hold a NaN
};
constexpr int kSharedBytes = kStages * kStageBytes + static_cast<int>(sizeof(Shared)) + 1024;
static_assert(2 * kTile * kSumPitch * 4 <= kStages * kStageBytes, "the tile's sums, of two groups, take the stages' place");

#define GEMM_SPLIT_8(r, o) "=r"(r[o]), "=r"(r[o + 1]), "=r"(r[o + 2]), "=r"(r[o + 3]), "=r"(r[o + 4]), "=r"(r[o + 5]), "=r"(r[o + 6]), "=r"(r[o + 7])
__device__ __forceinline__ void tmem_load_16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : GEMM_SPLIT_8(r, 0), GEMM_SPLIT_8(r, 8) : "r"(taddr));
}
#undef GEMM_SPLIT_8
// An image as an operand: rows of 64 values (128 bytes, 128-byte swizzle), groups of eight rows 1024 bytes apart, the
// contraction along the rows.
__device__ __forceinline__ uint64_t descriptor(uint32_t saddr) {
  return static_cast<uint64_t>((saddr & 0x3FFFFu) >> 4) | (static_cast<uint64_t>(1) << 16) | (static_cast<uint64_t>(1024 >> 4) << 32) |
         (static_cast<uint64_t>(1) << 46) | (static_cast<uint64_t>(2) << 61);
}
// Two numbers in one 64-bit register: what rounding both to bfloat16 gives, packed (ties away from zero; a NaN's may end as a
// zero's, and its remainder is NaN all the same), and what it leaves of them.
__device__ __forceinline__ uint32_t take_leading(unsigned long long& two) {
  const uint32_t lo = static_cast<uint32_t>(two) + 0x8000u, hi = static_cast<uint32_t>(two >> 32) + 0x8000u;
  const uint32_t minus_lo = (lo & 0xffff0000u) ^ 0x80000000u, minus_hi = (hi & 0xffff0000u) ^ 0x80000000u;
  asm("add.rn.f32x2 %0, %0, %1;" : "+l"(two) : "l"(static_cast<unsigned long long>(minus_hi) << 32 | minus_lo));
  return __byte_perm(lo, hi, 0x7632);
}

// Eight values' pieces of the three images; odd(): one of them is not finite (its remainder is NaN), or so large that its
// leading part is not.
struct Pieces {
  uint32_t first[4], second[4], third[4];
  unsigned long long sums;
  __device__ __forceinline__ bool odd() const { return sum_of_pair(sums) != 0.0f; }
  __device__ __forceinline__ Pieces(const float4& lo, const float4& hi) : sums(0ull) {
    const float v[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
    for (int e = 0; e < 8; e += 2) {
      unsigned long long two = static_cast<unsigned long long>(__float_as_uint(v[e + 1])) << 32 | __float_as_uint(v[e]);
      first[e >> 1] = take_leading(two);
      fma_pair(sums, two, 0ull);   // (0, or NaN)
      second[e >> 1] = take_leading(two);
      third[e >> 1] = __byte_perm(static_cast<uint32_t>(two), static_cast<uint32_t>(two >> 32), 0x7632);
    }
  }
  __device__ __forceinline__ void store(uint8_t* at) const {
    *reinterpret_cast<uint4*>(at) = make_uint4(first[0], first[1], first[2], first[3]);
    *reinterpret_cast<uint4*>(at + kImageBytes) = make_uint4(second[0], second[1], second[2], second[3]);
    *reinterpret_cast<uint4*>(at + 2 * kImageBytes) = make_uint4(third[0], third[1], third[2], third[3]);
  }
};

// The left operand's parts, a block 128 rows and 64 values of K: the images as the products' blocks want them in shared
// memory.  Every block along N would split the same rows again.
__global__ void __launch_bounds__(kSplitters)
gemm_split_left_kernel(const Args p) {
  const int t = threadIdx.x, piece = t & 7, sub = t >> 3, k = blockIdx.x * kDepth + piece * 8, m0 = blockIdx.y * kTile;
  const int three = blockIdx.y * gridDim.x + blockIdx.x;
  pdl_launch_dependents();
  pdl_wait();
  float4 lo[4], hi[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int m = m0 + sub + 32 * i;
    const float* src = p.A + static_cast<size_t>(m) * p.K + k;
    lo[i] = hi[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (m < p.M && k < p.K) lo[i] = *reinterpret_cast<const float4*>(src);
    if (m < p.M && k + 4 < p.K) hi[i] = *reinterpret_cast<const float4*>(src + 4);
  }
  uint8_t* dst = p.parts + static_cast<size_t>(three) * (kParts * kImageBytes) + sub * 128 + ((piece ^ (sub & 7)) << 4);
  __shared__ uint32_t rows[kRowWords];
  if (t < kRowWords) rows[t] = 0u;
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const Pieces pieces(lo[i], hi[i]);
    pieces.store(dst + i * 32 * 128);
    if (pieces.odd()) atomicOr(&rows[i], 1u << sub);
  }
  __syncthreads();
  if (t < kRowWords) p.odd[three * kRowWords + t] = rows[t];
}

// AHEAD: the left operand's images lie in p.parts and are copied; else this block splits both operands.
template <bool AHEAD>
__global__ void __launch_bounds__(kThreads, 1)
gemm_split_kernel(const Args p) {
  extern __shared__ uint8_t split_raw[];
  uint8_t* stages = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(split_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  Shared& s = *reinterpret_cast<Shared*>(stages + kStages * kStageBytes);
  float* sums = reinterpret_cast<float*>(stages);   // [128][kSumPitch], once the stages are read out
  volatile int* abort_flag = &s.abort_flag;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int rank = blockIdx.x % p.cluster, n0 = blockIdx.x / p.cluster * kTile, m0 = blockIdx.y * kTile;
  const int own_groups = p.groups / p.cluster, group_depth = p.share * kDepth;
  const int k_begin = min(rank * own_groups * group_depth, p.K), k_end = min(k_begin + own_groups * group_depth, p.K);
  const int count = (k_end - k_begin + kDepth - 1) / kDepth;
  // The groups' sums are added in their order: the first block of a cluster adds its own up as it goes; the others keep
  // theirs apart, one tile each in shared memory (there are two at most: four groups in two blocks).
  const bool apart = rank > 0 && own_groups > 1;
  pdl_launch_dependents();
  if (tid == 0) {
    for (int i = 0; i < kStages; ++i) {
      bar_init(&s.full[i], kSplitters + (AHEAD ? 1 : 0));
      bar_init(&s.empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      bar_init(&s.sums_full[i], 1);
      bar_init(&s.sums_empty[i], kSumWarps * 32);
    }
    s.abort_flag = 0;
    for (int i = 0; i < 2 * kRowWords; ++i) s.odd[i] = s.nan[i] = 0u;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kIssuer) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(shared_address(&s.tmem_base)), "r"(512));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = s.tmem_base;

  if (warp < kSumWarps) {
    // ---------------- sums: a row and 64 columns a thread; the first warp issues the products ----------------
    const int row = (warp & 3) * 32 + lane, column0 = (warp >> 2) * 64;
    const uint32_t taddr = tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16) + column0;
    float total[64];
#pragma unroll
    for (int j = 0; j < 64; ++j) total[j] = 0.0f;
    volatile float before[64];   // the groups before this one; in local memory, registers are short
    bool some_before = false;
    constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(kTile >> 4) << 24) | (static_cast<uint32_t>(kTile >> 3) << 17);
    const uint32_t base = shared_address(stages);
    auto products = [&](int c) {
      const uint32_t stage = c & 1, parity = (c >> 1) & 1;
      if (lane == 0) {
        if (c >= 2) bar_wait<WAIT_EXPIRED>(&s.sums_empty[stage], parity ^ 1u, abort_flag, p.status);
        bar_wait<WAIT_EXPIRED>(&s.full[stage], parity, abort_flag, p.status);
      }
      __syncwarp();
      fence_after();
      const uint64_t a = descriptor(base + stage * kStageBytes), w = descriptor(base + stage * kStageBytes + kParts * kImageBytes);
      constexpr uint64_t kNext = kImageBytes >> 4;   // the next part's image
      const uint32_t large = tmem + stage * 256, small = large + 128;
#pragma unroll
      for (int ks = 0; ks < kDepth / 16; ++ks) {
        const uint64_t x = a + 2 * ks, y = w + 2 * ks;
        mma_shared(small, x + 2 * kNext, y, kIdesc, ks > 0 ? 1u : 0u);
        mma_shared(small, x, y + 2 * kNext, kIdesc, 1u);
        mma_shared(small, x + kNext, y + kNext, kIdesc, 1u);
        mma_shared(small, x + kNext, y, kIdesc, 1u);
        mma_shared(small, x, y + kNext, kIdesc, 1u);
        mma_shared(large, x, y, kIdesc, ks > 0 ? 1u : 0u);
      }
      commit(&s.empty[stage]);
      commit(&s.sums_full[stage]);
    };
    if (warp == kIssuer && count > 0) products(0);
    for (int c = 0; c < count;) {
      const int group_end = min(c + p.share, count);
#pragma unroll 1
      for (; c < group_end; ++c) {
        if (warp == kIssuer && c + 1 < count) products(c + 1);   // (on their way while this warp adds)
        const uint32_t pair = taddr + (c & 1) * 256;
        bar_wait<WAIT_EXPIRED>(&s.sums_full[c & 1], (c >> 1) & 1, abort_flag, p.status);
        fence_after();
#pragma unroll
        for (int j = 0; j < 64; j += 16) {
          uint32_t large[16], small[16];
          tmem_load_16(pair + j, large);
          tmem_load_16(pair + 128 + j, small);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int e = 0; e < 16; ++e) total[j + e] = (total[j + e] + __uint_as_float(small[e])) + __uint_as_float(large[e]);
        }
        fence_before();
        bar_arrive(&s.sums_empty[c & 1]);
      }
      if (own_groups == 1) break;
      if (some_before && !apart) {
#pragma unroll
        for (int j = 0; j < 64; ++j) total[j] = before[j] + total[j];
      }
      if (c < count) {
#pragma unroll
        for (int j = 0; j < 64; ++j) {
          before[j] = total[j];
          total[j] = 0.0f;
        }
        some_before = true;
      }
    }
    // (the last sums are complete, so every product that read the stages is)
    float* own = sums + row * kSumPitch + column0;
    if (apart) {   // the first group's tile, then the second's
      if (!some_before) {
#pragma unroll
        for (int j = 0; j < 64; ++j) {
          before[j] = total[j];
          total[j] = 0.0f;
        }
      }
#pragma unroll
      for (int j = 0; j < 64; j += 4) *reinterpret_cast<float4*>(own + j) = make_float4(before[j], before[j + 1], before[j + 2], before[j + 3]);
      own += kTile * kSumPitch;
    }
#pragma unroll
    for (int j = 0; j < 64; j += 4) *reinterpret_cast<float4*>(own + j) = make_float4(total[j], total[j + 1], total[j + 2], total[j + 3]);
  } else {
    // ---------------- operands: runs of eight values, four a thread and stage of either operand ----------------
    constexpr int kRuns = AHEAD ? 4 : 8, kFirstW = kRuns - 4;
    const int t = tid - kFirstSplitter * 32, piece = t & 7, sub = t >> 3;   // rows sub + 32 i
    float4 lo[kRuns], hi[kRuns];
    // where this thread's runs start, and which of its rows exist
    const float* a_rows = p.A + static_cast<size_t>(m0 + sub) * p.K + k_begin + piece * 8;
    const float* w_rows = p.W + static_cast<size_t>(n0 + sub) * p.K + k_begin + piece * 8;
    const size_t step = static_cast<size_t>(32) * p.K;
    unsigned live = 0;
#pragma unroll
    for (int i = 0; i < kRuns; ++i)
      live |= (i < kFirstW ? m0 + sub + 32 * i < p.M : n0 + sub + 32 * (i - kFirstW) < p.N) ? 1u << i : 0u;
    const int whole = (k_end - k_begin) / kDepth;   // stages that lie within K
    auto ask = [&](int i, int c) {
      const float* src = (i < kFirstW ? a_rows + i * step : w_rows + (i - kFirstW) * step) + c * kDepth;
      lo[i] = hi[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      if (live >> i & 1u) {
        // (K is a multiple of four: each half of the run lies within it or not)
        if (c < whole || k_begin + c * kDepth + piece * 8 < k_end) lo[i] = *reinterpret_cast<const float4*>(src);
        if (c < whole || k_begin + c * kDepth + piece * 8 + 4 < k_end) hi[i] = *reinterpret_cast<const float4*>(src + 4);
      }
    };
    // the weights of the first stage are asked for before the kernel ahead has ended
#pragma unroll
    for (int i = kFirstW; i < kRuns; ++i)
      if (count > 0) ask(i, 0);
    pdl_wait();
#pragma unroll
    for (int i = 0; i < kFirstW; ++i)
      if (count > 0) ask(i, 0);
    const int three = blockIdx.y * ((p.K + kDepth - 1) / kDepth) + k_begin / kDepth;   // the first images of this block
    if (AHEAD)
      for (int i = t; i < count * kRowWords; i += kSplitters)
        if (const uint32_t rows = p.odd[three * kRowWords + i]) atomicOr(&s.odd[i % kRowWords], rows);
    for (int c = 0; c < count; ++c) {
      const int stage = c & 1;
      if (c >= 2) bar_wait<WAIT_EXPIRED>(&s.empty[stage], ((c >> 1) & 1) ^ 1, abort_flag, p.status);
      if (AHEAD && t == 0) {
        const uint32_t bytes = *abort_flag ? 0 : kParts * kImageBytes, bar = shared_address(&s.full[stage]);
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
        if (bytes)
          asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                           shared_address(stages + stage * kStageBytes)),
                       "l"(p.parts + static_cast<size_t>(three + c) * (kParts * kImageBytes)), "r"(bytes), "r"(bar)
                       : "memory");
      }
      uint8_t* dst = stages + stage * kStageBytes + sub * 128 + ((piece ^ (sub & 7)) << 4);   // (rows 32 apart are swizzled alike)
#pragma unroll
      for (int i = 0; i < kRuns; ++i) {
        const Pieces pieces(lo[i], hi[i]);
        if (c + 1 < count) ask(i, c + 1);   // the next stage's run takes this one's registers
        if (pieces.odd()) atomicOr(&s.odd[i < kFirstW ? i : kRowWords + i - kFirstW], 1u << sub);
        pieces.store(dst + (i < kFirstW ? 0 : kParts * kImageBytes) + ((i - kFirstW) & 3) * 32 * 128);
      }
      fence_async();
      bar_arrive(&s.full[stage]);
    }
    if (AHEAD && t == 0 && *abort_flag) {   // a copy may be on its way still: it ends long before this does
      for (int i = 0; i < 1000; ++i) __nanosleep(1000);
    }
  }
  fence_before();
  __syncthreads();
  if (warp == kIssuer) {
    fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
  }
  pdl_wait();   // (every thread may read A or the residual stream from here on)
  uint32_t any = 0u;
#pragma unroll
  for (int i = 0; i < 2 * kRowWords; ++i) any |= s.odd[i];
  if (any) {
    // which of these rows hold a NaN within this block's share of K: a warp a row (one that holds something exists)
    for (int r = warp; r < 2 * kTile; r += kThreads / 32) {
      if (!(s.odd[r >> 5] >> (r & 31) & 1u)) continue;
      const float* row = r < kTile ? p.A + static_cast<size_t>(m0 + r) * p.K : p.W + static_cast<size_t>(n0 + r - kTile) * p.K;
      bool nan = false;
#pragma unroll 4
      for (int k = k_begin + lane; k < k_end; k += 32) nan |= row[k] != row[k];
      if (__any_sync(0xffffffffu, nan) && lane == 0) atomicOr(&s.nan[r >> 5], 1u << (r & 31));
    }
    __syncthreads();
    // their outputs: row r of A against all of W's, then row r of W against all of A's
    for (int word = 0; word < 2 * kRowWords; ++word) {
      for (uint32_t left = s.odd[word]; left; left &= left - 1u) {
        const int r = word % kRowWords * 32 + __ffs(static_cast<int>(left)) - 1;
        const bool of_a = word < kRowWords, nan = s.nan[word] & left & -left;
        const float* own = of_a ? p.A + static_cast<size_t>(m0 + r) * p.K : p.W + static_cast<size_t>(n0 + r) * p.K;
        const float* others = of_a ? p.W + static_cast<size_t>(n0) * p.K : p.A + static_cast<size_t>(m0) * p.K;
        const int count_others = min(kTile, of_a ? p.N - n0 : p.M - m0);
        for (int i = warp; i < count_others; i += kThreads / 32) {
          float* at = sums + (of_a ? r : i) * kSumPitch + (of_a ? i : r);
          float all = nan ? NAN : 0.0f;
          for (int group = 0; group < own_groups; ++group) {
            const int begin = min(k_begin + group * group_depth, k_end), end = min(begin + group_depth, k_end);
            float sum = 0.0f;
            if (!nan) {
#pragma unroll 4
              for (int k = begin + lane; k < end; k += 32) sum = fmaf(own[k], others[static_cast<size_t>(i) * p.K + k], sum);
              sum = warp_sum(sum);
            }
            if (apart && group == 0) {
              if (lane == 0) at[0] = all + sum;
              all = 0.0f;
            } else {
              all += sum;
            }
          }
          if (lane == 0) at[apart ? kTile * kSumPitch : 0] = all;
        }
      }
    }
    __syncthreads();
  }
  if (p.cluster > 1) cluster_sync();

  // The ending.  In a cluster each block finishes every cluster-th row of the tile.  A thread keeps one column.
  auto total = [&](int m, int n) {
    float* own = sums + m * kSumPitch + n;
    if (p.cluster == 1) return *own;
    // (every part is asked for before the first is added)
    const uint32_t at = shared_address(own);
    float part[4], second = 0.0f;
#pragma unroll
    for (int r = 0; r < 4; ++r) part[r] = r < p.cluster ? remote_float(at, r) : 0.0f;
    if (own_groups > 1) second = remote_float(at + kTile * kSumPitch * 4, 1);   // (four groups in two blocks)
    if (p.cluster == 2) return own_groups > 1 ? (part[0] + part[1]) + second : part[0] + part[1];
    return ((part[0] + part[1]) + part[2]) + part[3];
  };
  const bool gated = p.epilogue == 2;
  const int columns = gated ? kTile / 2 : kTile, column_bits = gated ? 6 : 7, row_step = 512 >> column_bits;
  const int c = tid & (columns - 1), n = gated ? (c / 16) * 32 + c % 16 : c;   // gated: the gate's column; the up value is 16 further
  if (tid < 512 && n0 + n + (gated ? 16 : 0) < p.N && !*abort_flag) {
    const float bias = p.bias ? p.bias[n0 + n] : 0.0f, up_bias = p.bias && gated ? p.bias[n0 + n + 16] : 0.0f;
    const int pitch = gated ? p.N / 2 : p.N, column = gated ? n0 / 2 + c : n0 + c;
    for (int row = tid >> column_bits; row < kTile / p.cluster; row += 4 * row_step) {
      float value[4], before[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int m = (row + i * row_step) * p.cluster + rank;
        if (m >= kTile || m0 + m >= p.M) continue;
        if (p.epilogue == 1) before[i] = p.resid[static_cast<size_t>(m0 + m) * pitch + column];
        value[i] = total(m, n) + bias;
        if (gated) value[i] = (total(m, n + 16) + up_bias) * gate_activation(value[i], p.activation);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int m = (row + i * row_step) * p.cluster + rank;
        if (m >= kTile || m0 + m >= p.M) continue;
        const size_t at = static_cast<size_t>(m0 + m) * pitch + column;
        if (p.epilogue == 1) p.resid[at] = before[i] + value[i];
        else if (p.out_bf16) static_cast<__nv_bfloat16*>(p.out)[at] = __float2bfloat16_rn(value[i]);
        else static_cast<float*>(p.out)[at] = value[i];
      }
    }
  }
  if (p.cluster > 1) cluster_sync();   // no block leaves while another reads its part
}

// How K is cut.  A call costs about (waves of blocks) x (stages of a block + what it costs besides).  The groups that are
// summed on their own are as many as blocks would share K with a single tile of rows: they follow from N and K alone, so that
// a row's sums have one order whatever the step's other rows are.  The blocks of a cluster share the groups where that is
// faster for the rows there are.  (As many blocks for every count of rows, those that lose least on average: 256 x 896 of 896
// 35 us, 2,048 x 896 of 4,864 192; so 26 and 166.)
constexpr long long kSms = 148;   // (not asked of the device: the groups follow from it)
static double cost_of(long long tiles, int blocks, int stages) { return static_cast<double>((tiles * blocks + kSms - 1) / kSms) * (stages + 4); }
static void share_out(int M, int N, int K, int* groups, int* share, int* cluster) {
  const long long tiles_n = (N + kTile - 1) / kTile, tiles = tiles_n * ((M + kTile - 1) / kTile);
  const int depth = (K + kDepth - 1) / kDepth;
  *groups = *cluster = 1;
  for (int n = 2; n <= 4; n *= 2)
    if (cost_of(tiles_n, n, (depth + n - 1) / n) < cost_of(tiles_n, *groups, (depth + *groups - 1) / *groups)) *groups = n;
  *share = (depth + *groups - 1) / *groups;
  for (int n = 2; n <= *groups; n *= 2)
    if (cost_of(tiles, n, *groups / n * *share) < cost_of(tiles, *cluster, *groups / *cluster * *share)) *cluster = n;
}

static int launch_rows(const Args& args, cudaStream_t s) {
  Args p = args;
  const long long tiles_n = (p.N + kTile - 1) / kTile, tiles_m = (p.M + kTile - 1) / kTile, depth = (p.K + kDepth - 1) / kDepth;
  if (tiles_m > 65535) return VIPERA_BAD_SHAPE;
  share_out(p.M, p.N, p.K, &p.groups, &p.share, &p.cluster);
  const dim3 grid(static_cast<unsigned>(tiles_n * p.cluster), static_cast<unsigned>(tiles_m));
  if (!p.parts) return launch_in_clusters(gemm_split_kernel<false>, p.cluster, grid, dim3(kThreads), kSharedBytes, s, p);
  const int status = vipera_launch(gemm_split_left_kernel, dim3(static_cast<unsigned>(depth), static_cast<unsigned>(tiles_m)),
                                   dim3(kSplitters), 0, s, p);
  if (status) return status;
  return launch_in_clusters(gemm_split_kernel<true>, p.cluster, grid, dim3(kThreads), kSharedBytes, s, p);
}

// Room for the left operand's parts, or 0 where splitting them ahead does not pay: a launch more, and each stage shorter
// (5,500 clocks to 3,400).  Not more room than the L2 holds well: more rows are taken in turns.  Both operands split in the
// block / the left one ahead: 80 x 896 of 896, seven stages in a row: 17.5 / 18.5 us; 1,024 x 1,152 of 896, seven: 30.6 / 31.2;
// 256 x 256 of 2,048, eight: 33.9 / 27.0 (these three with parts cut off); 128 x 9,728 of 896, fourteen: 57.9 / 41.2; 8,192 x 4,096
// of 4,096: 3,057 / 1,860.
constexpr long long kMostParts = 96ll << 20, kTileExtra = kRowWords * 4;   // (bytes beside each three of images: its rows' bits)
static int parts_bytes(int M, int N, int K) {
  if (M <= 64 || N <= kTile || K % 4 != 0) return 0;   // (one tile along N: nobody else would split the same rows)
  const long long tiles_m = (M + kTile - 1) / kTile, tiles_n = (N + kTile - 1) / kTile;
  int groups, share, cluster;
  share_out(M, N, K, &groups, &share, &cluster);
  if ((tiles_m * tiles_n * cluster + kSms - 1) / kSms * (groups / cluster * share) < 8) return 0;   // stages in a row
  const long long of_tile = (K + kDepth - 1) / kDepth * (kParts * kImageBytes + kTileExtra);
  const long long tiles = kMostParts / of_tile;
  return static_cast<int>((tiles < tiles_m ? tiles : tiles_m) * of_tile);
}

static int launch(const Args& args, cudaStream_t s) {
  static SharedMemoryOptIn opt_in, opt_in_ahead;
  int status = opt_in.ask(reinterpret_cast<const void*>(gemm_split_kernel<false>), kSharedBytes);
  if (!status) status = opt_in_ahead.ask(reinterpret_cast<const void*>(gemm_split_kernel<true>), kSharedBytes);
  if (status) return status;
  const long long of_tile = static_cast<long long>((args.K + kDepth - 1) / kDepth) * (kParts * kImageBytes + kTileExtra);
  const long long tiles = args.parts ? args.parts_bytes / of_tile : 0;
  if (tiles < 1) {
    Args p = args;
    p.parts = nullptr;
    return launch_rows(p, s);
  }
  const size_t out_pitch = static_cast<size_t>(args.epilogue == 2 ? args.N / 2 : args.N);
  for (long long m = 0; m < args.M && !status; m += tiles * kTile) {
    Args p = args;
    p.M = static_cast<int>(args.M - m < tiles * kTile ? args.M - m : tiles * kTile);
    p.odd = reinterpret_cast<uint32_t*>(p.parts + tiles * ((p.K + kDepth - 1) / kDepth) * (kParts * kImageBytes));
    p.A += static_cast<size_t>(m) * p.K;
    if (p.epilogue == 1) p.resid += m * out_pitch;
    else p.out = static_cast<char*>(p.out) + m * out_pitch * (p.out_bf16 ? 2 : 4);
    status = launch_rows(p, s);
  }
  return status;
}

}  // namespace gemm_split
