// The fold over latents on the fifth-generation tensor cores (tcgen05, accumulators in tensor memory), for steps
// of many (token, head) rows in the head-major form (bfloat16 caches).
//
// A block takes 128 rows (numbered token by token, so that a tile's heads share its keys) and a slice of up to
// 256 of the latent's columns, and walks the keys 64 at a time:
//
//   S = Q [c | kr]^T     tcgen05.mma 128 x 64 over rank + rot values, from shared memory, into tensor memory
//   softmax              a row a thread; weights rounded to bfloat16 go back to tensor memory, where the
//                        output product takes them from; their sum is that of the rounded weights
//   O += P C             tcgen05.mma 128 x 128 columns x 64 keys per part of 128 columns (64 where a slice has one more half), in tensor memory
//
// Two score and two weight buffers let the scores of one tile run while the softmax of the one before is
// computed.  Keys and values are the same rows: a tile comes as parts of [64 keys][128 columns] (two halves of 64
// columns, 8 KB, 128-byte swizzle), read along the columns for the scores and along the keys for the output.  The
// queries fill 144 KB of shared memory, which leaves five slots for parts: a ring of two for those that only the
// scores read, and one of three for those the output product reads too (a tile's two and the next one's first).  The
// scores are computed in the block of each slice: with 512 columns of output beside them, tensor memory would not do
// (512 columns an SM).
//
// Roles: warps 0-3 softmax and ending, warp 4 issues the products, then a warp per half of a slot, which brings one
// half part after another through the block table (cp.async; first of all each brings a half part of the queries).
// What bounds it is the issuing warp: a product of 16 values' depth keeps the tensor cores for 48 to 64 clocks and its
// issue takes 35 (77 from a single lane in a diverged branch, whose operands travel one by one), a wait or a commit
// about 100; hence the elected lane, the parts of 128 columns and the output products of 128.
// Measured: 2,048 tokens, 12 heads, window 1,024: 197 us, the mixer 543 -> 290 us; 1,024 tokens behind 2,000, 12 heads: the mixer
// 781 -> 362 us, 32 heads: 1,813 -> 759 (before: mma.sync, a block 16 or 32 rows).
// Tokens of several requests in a tile are folded one request after another.
// Every wait is bounded; one that runs out leaves a code in the status word and the rows unwritten.
#pragma once

#include "tcgen05.cuh"

namespace latent_tc {

using namespace tcgen05;

constexpr int kRows = 128, kKeys = 64, kHalf = 64, kPart = 128;   // rows, keys of a tile, columns of a half part and of a part
constexpr int kHalfBytes = kKeys * kHalf * 2, kQueryBytes = kRows * kHalf * 2;
constexpr int kScoreSlots = 2, kValueSlots = 3, kSlots = kScoreSlots + kValueSlots;
constexpr int kMostHalves = 9;                       // 512 / 64 and the rotated part
constexpr int kSoftmaxWarps = 4, kIssuer = 4, kFirstLoader = 5, kLoaders = 2 * kSlots;
constexpr int kThreads = (kFirstLoader + kLoaders) * 32;
constexpr uint32_t kColsO = 0, kColsS = 256, kColsP = 384, kTmemCols = 512;   // O 256, S 2 x 64, P 2 x 32
constexpr float kLog2e = 1.4426950408889634f;
enum { WAIT_EXPIRED = 5 };
static_assert(kLoaders >= kMostHalves, "a loading warp brings at most one half part of the queries");

struct Params {
  const float* qa_heads;           // [heads, padded_tokens, rank], unscaled
  const float* q_rot;              // [tokens, heads, rot], scaled
  const __nv_bfloat16* k_pool;     // latents
  const __nv_bfloat16* v_pool;     // rotated key parts
  const int* token_entry;
  const int* positions;
  const int* block_table;
  __nv_bfloat16* l_heads;          // [heads, padded_tokens, rank]
  int num_tokens, heads, rank, rot, table_width, page_size, padded_tokens, window;
  float scale;
  const float* sink;
  int* status;
};

struct Shared {
  uint64_t full[kSlots], empty[kSlots], query[kMostHalves], score[2], weight[2], done;
  uint32_t tmem_base;
  int abort_flag;
  int entry[kRows], position[kRows];   // of the tile's tokens
};

constexpr int kSharedBytes = kMostHalves * kQueryBytes + 2 * kSlots * kHalfBytes + static_cast<int>(sizeof(Shared)) + 1024;
static_assert(kSharedBytes <= 227 * 1024, "a block's shared memory");

__device__ __forceinline__ void mma_tensor(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p, leader;\n elect.sync _|leader, 0xffffffff;\n setp.ne.b32 p, %4, 0;\n"
      " @leader tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}\n" ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}
#define LATENT_TC_8(r, o) "=r"(r[o]), "=r"(r[o + 1]), "=r"(r[o + 2]), "=r"(r[o + 3]), "=r"(r[o + 4]), "=r"(r[o + 5]), "=r"(r[o + 6]), "=r"(r[o + 7])
__device__ __forceinline__ void tmem_load(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : LATENT_TC_8(r, 0), LATENT_TC_8(r, 8), LATENT_TC_8(r, 16), LATENT_TC_8(r, 24)
      : "r"(taddr));
}
#undef LATENT_TC_8
__device__ __forceinline__ void tmem_load_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
#define LATENT_TC_8(r, o) "r"(r[o]), "r"(r[o + 1]), "r"(r[o + 2]), "r"(r[o + 3]), "r"(r[o + 4]), "r"(r[o + 5]), "r"(r[o + 6]), "r"(r[o + 7])
__device__ __forceinline__ void tmem_store(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
      ::"r"(taddr), LATENT_TC_8(r, 0), LATENT_TC_8(r, 8), LATENT_TC_8(r, 16), LATENT_TC_8(r, 24)
      : "memory");
}
#undef LATENT_TC_8
__device__ __forceinline__ void tmem_store_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// 2^x with the hardware's approximation (the weights are rounded to bfloat16); 2^(-inf) = 0
__device__ __forceinline__ float power_of_two(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// 16-byte piece `piece` (0..7) of row `row` of a half part, swizzled
__device__ __forceinline__ uint32_t piece_offset(int row, int piece) { return static_cast<uint32_t>(row * 128 + ((piece ^ (row & 7)) << 4)); }
// A half part as an operand: 128-byte rows, 128-byte swizzle, groups of eight rows 1024 bytes apart, read with the
// contraction along the rows' bytes or (`down`) down the rows; in the latter the second 64 of an operand's columns are
// one half part further.
__device__ __forceinline__ uint64_t descriptor(uint32_t saddr, bool down) {
  return static_cast<uint64_t>((saddr & 0x3FFFFu) >> 4) | (static_cast<uint64_t>(down ? kHalfBytes >> 4 : 1) << 16) |
         (static_cast<uint64_t>(1024 >> 4) << 32) | (static_cast<uint64_t>(1) << 46) | (static_cast<uint64_t>(2) << 61);
}

// One request's tokens that follow one another in the tile, and the keys any of them sees.
struct Segment { int begin, end, entry, first_key, end_key, first_tile, tiles; };
__device__ __forceinline__ Segment segment_from(const Shared& s, int begin, int tokens, int window) {
  Segment g{begin, begin, s.entry[begin], 0, 0, 0, 0};
  int low = 0x7fffffff, high = -1;
  while (g.end < tokens && s.entry[g.end] == g.entry) {
    low = min(low, s.position[g.end]);
    high = max(high, s.position[g.end]);
    ++g.end;
  }
  g.first_key = window > 0 ? max(0, low - window + 1) : 0;
  g.end_key = high + 1;
  g.first_tile = g.first_key / kKeys;
  g.tiles = (g.end_key + kKeys - 1) / kKeys - g.first_tile;
  return g;
}

__global__ void __launch_bounds__(kThreads, 1)
latent_fold_tc_kernel(const Params p) {
  extern __shared__ uint8_t latent_tc_raw[];
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(latent_tc_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint8_t* queries = base;                                   // half parts of [128 rows][64 columns]
  uint8_t* slots = base + kMostHalves * kQueryBytes;         // half parts of [64 keys][64 columns], two a slot
  Shared& s = *reinterpret_cast<Shared*>(slots + 2 * kSlots * kHalfBytes);
  volatile int* abort_flag = &s.abort_flag;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int slices = (p.rank + 255) / 256;
  const int tile = (static_cast<int>(gridDim.x) - 1 - static_cast<int>(blockIdx.x)) / slices;   // the longest histories of a prompt first
  const int slice = static_cast<int>(blockIdx.x) % slices;
  // The columns in the order they are read: those only the scores need (the other slice's), the rotated part, this
  // slice's.  Counted in half parts: others, then one, then own; in parts: others_parts, one, own_parts.
  const int own = min(256, p.rank - 256 * slice) / kHalf, others = p.rank / kHalf - own, halves = others + 1 + own;
  const int others_parts = (others + 1) / 2, own_parts = (own + 1) / 2, score_parts = others_parts + 1;
  auto column_of = [&](int half) { return half > others ? 256 * slice + (half - others - 1) * kHalf : (slice ? 0 : 256) + half * kHalf; };
  const int total_rows = p.num_tokens * p.heads, row0 = tile * kRows, rows = min(kRows, total_rows - row0);
  const int token0 = row0 / p.heads, tokens = (row0 + rows - 1) / p.heads - token0 + 1;

  pdl_launch_dependents();
  if (tid == 0) {
    for (int i = 0; i < kSlots; ++i) {
      bar_init(&s.full[i], 64);
      bar_init(&s.empty[i], 1);
    }
    for (int i = 0; i < kMostHalves; ++i) bar_init(&s.query[i], 32);
    for (int i = 0; i < 2; ++i) {
      bar_init(&s.score[i], 1);
      bar_init(&s.weight[i], kSoftmaxWarps * 32);
    }
    bar_init(&s.done, 1);
    s.abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kIssuer) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(shared_address(&s.tmem_base)), "r"(kTmemCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  // (the step's tokens are the host's, written before the step)
  for (int i = tid; i < tokens; i += kThreads) {
    s.entry[i] = p.token_entry[token0 + i];
    s.position[i] = p.positions[token0 + i];
  }
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = s.tmem_base;

  if (warp < kSoftmaxWarps) {
    // ---------------- softmax, ending: thread = row ----------------
    pdl_wait();   // the output belongs to earlier kernels until now
    const int row = tid, own_token = (row0 + min(row, rows - 1)) / p.heads - token0;
    const int head = (row0 + min(row, rows - 1)) % p.heads;
    const uint32_t lanes = tmem + (static_cast<uint32_t>(warp * 32) << 16);
    int count = 0, passes = 0;   // tiles, and requests, so far
    for (int begin = 0; begin < tokens; ++passes) {
      const Segment g = segment_from(s, begin, tokens, p.window);
      begin = g.end;
      const bool mine = row < rows && own_token >= g.begin && own_token < g.end;
      const int last = mine ? s.position[own_token] : -1;
      const int first = mine && p.window > 0 ? last - p.window + 1 : 0;
      float row_max = -INFINITY, row_sum = 0.0f;   // the max in powers of two
      for (int t = 0; t < g.tiles; ++t, ++count) {
        const uint32_t buffer = count & 1, parity = (count >> 1) & 1;
        bar_wait<WAIT_EXPIRED>(&s.score[buffer], parity, abort_flag, p.status);
        fence_after();
        uint32_t v[64];
        tmem_load(lanes + kColsS + buffer * kKeys, *reinterpret_cast<uint32_t(*)[32]>(&v[0]));
        tmem_load(lanes + kColsS + buffer * kKeys + 32, *reinterpret_cast<uint32_t(*)[32]>(&v[32]));
        tmem_load_wait();
        const int key0 = (g.first_tile + t) * kKeys;
        if (key0 < first || key0 + kKeys - 1 > last) {
#pragma unroll
          for (int k = 0; k < kKeys; ++k)
            if (key0 + k < first || key0 + k > last) v[k] = __float_as_uint(-INFINITY);
        }
        float m0 = -INFINITY, m1 = -INFINITY, m2 = -INFINITY, m3 = -INFINITY;
#pragma unroll
        for (int k = 0; k < kKeys; k += 4) {
          m0 = fmaxf(m0, __uint_as_float(v[k]));
          m1 = fmaxf(m1, __uint_as_float(v[k + 1]));
          m2 = fmaxf(m2, __uint_as_float(v[k + 2]));
          m3 = fmaxf(m3, __uint_as_float(v[k + 3]));
        }
        const float tile_max = fmaxf(fmaxf(m0, m1), fmaxf(m2, m3)) * kLog2e;
        // (the running max follows at once, so that the largest weight is exactly 1: one that lags by up to 2^8 saves some
        // passes over the output, 2 us of 290, and rounds it: 4.99e-3 from 64 bits instead of 4.93e-3, mma.sync's)
        const float new_max = fmaxf(row_max, tile_max);
        const float alpha = new_max == row_max ? 1.0f : power_of_two(row_max - new_max);
        row_max = new_max;
        row_sum *= alpha;
        // (these scores are complete, so the output product of the tile before is)
        if (t > 0 && __any_sync(0xffffffffu, alpha != 1.0f)) {
#pragma unroll 1
          for (int c = 0; c < own * kHalf; c += 32) {
            uint32_t o[32];
            tmem_load(lanes + kColsO + c, o);
            tmem_load_wait();
#pragma unroll
            for (int k = 0; k < 32; ++k) o[k] = __float_as_uint(__uint_as_float(o[k]) * alpha);
            tmem_store(lanes + kColsO + c, o);
          }
        }
        const float shift = row_max == -INFINITY ? 0.0f : row_max;
        float sum0 = 0.0f, sum1 = 0.0f;
        uint32_t packed[32];
#pragma unroll
        for (int k = 0; k < kKeys; k += 2) {
          const __nv_bfloat162 w = __floats2bfloat162_rn(power_of_two(fmaf(__uint_as_float(v[k]), kLog2e, -shift)),
                                                         power_of_two(fmaf(__uint_as_float(v[k + 1]), kLog2e, -shift)));
          const float2 rounded = __bfloat1622float2(w);
          sum0 += rounded.x;
          sum1 += rounded.y;
          packed[k >> 1] = *reinterpret_cast<const uint32_t*>(&w);
        }
        row_sum += sum0 + sum1;
        tmem_store(lanes + kColsP + buffer * (kKeys / 2), packed);
        tmem_store_wait();
        fence_before();
        bar_arrive(&s.weight[buffer]);
      }
      // the ending: the request's rows
      bar_wait<WAIT_EXPIRED>(&s.done, static_cast<uint32_t>(passes) & 1u, abort_flag, p.status);
      fence_after();
      float total = row_sum;
      if (p.sink) total += exp2f(p.sink[head] * kLog2e - row_max);
      const float inverse = 1.0f / total;
      __nv_bfloat16* out = p.l_heads + (static_cast<size_t>(head) * p.padded_tokens + token0 + own_token) * p.rank + slice * 256;
#pragma unroll 1
      for (int c = 0; c < own * kHalf; c += 32) {
        uint32_t o[32];
        tmem_load(lanes + kColsO + c, o);
        tmem_load_wait();
        if (mine && !*abort_flag) {
#pragma unroll
          for (int k = 0; k < 32; k += 8) {
            uint4 packed;
            __nv_bfloat162* pairs = reinterpret_cast<__nv_bfloat162*>(&packed);
#pragma unroll
            for (int e = 0; e < 4; ++e)
              pairs[e] = __floats2bfloat162_rn(__uint_as_float(o[k + 2 * e]) * inverse, __uint_as_float(o[k + 2 * e + 1]) * inverse);
            *reinterpret_cast<uint4*>(out + c + k) = packed;
          }
        }
      }
      fence_before();
      asm volatile("bar.sync 1, 160;" ::: "memory");   // with the issuer: the next request's products overwrite O
    }
  } else if (warp == kIssuer) {
    // ---------------- the products: a warp that walks together, one elected lane issues ----------------
    constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(kRows >> 4) << 24);
    constexpr uint32_t kIdescScores = kIdesc | (static_cast<uint32_t>(kKeys >> 3) << 17);
    constexpr uint32_t kIdescValues = kIdesc | (1u << 16) | (static_cast<uint32_t>(kPart >> 3) << 17);       // B read down its rows
    constexpr uint32_t kIdescHalf = kIdesc | (1u << 16) | (static_cast<uint32_t>(kHalf >> 3) << 17);
    const uint32_t query_addr = shared_address(queries), slot_addr = shared_address(slots);
    uint32_t score_slot = 0, score_parity = 0, value_slot = 0, value_parity = 0;   // of the next part of either ring
    int count = 0;                                                                // tiles issued
    const int rot_steps = (p.rot + 15) / 16;
    auto wait = [&](uint64_t* bar, uint32_t parity) {
      if (lane == 0) bar_wait<WAIT_EXPIRED>(bar, parity, abort_flag, p.status);
      __syncwarp();
      fence_after();
    };
    // `steps` products of 16 columns of a half part
    auto scores_of = [&](int half, uint32_t keys, uint32_t buffer, int steps) {
      const uint64_t a = descriptor(query_addr + half * kQueryBytes, false), b = descriptor(keys, false);
      const uint32_t d = tmem + kColsS + buffer * kKeys;
      if (steps == 4) {
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) mma_shared(d, a + 2 * ks, b + 2 * ks, kIdescScores, half > 0 || ks > 0 ? 1u : 0u);
      } else {
        for (int ks = 0; ks < steps; ++ks) mma_shared(d, a + 2 * ks, b + 2 * ks, kIdescScores, half > 0 || ks > 0 ? 1u : 0u);
      }
    };
    auto score_part = [&](int i, uint32_t buffer, bool very_first) {   // a part that only the scores read (the last: the rotated one)
      const int half = i == score_parts - 1 ? others : 2 * i, more = i < score_parts - 1 && half + 1 < others;
      if (very_first) {
        wait(&s.query[half], 0);
        if (more) wait(&s.query[half + 1], 0);
      }
      wait(&s.full[score_slot], score_parity);
      const uint32_t keys = slot_addr + score_slot * 2 * kHalfBytes;
      scores_of(half, keys, buffer, i == score_parts - 1 ? rot_steps : 4);
      if (more) scores_of(half + 1, keys + kHalfBytes, buffer, 4);
      commit(&s.empty[score_slot]);
      if (++score_slot == kScoreSlots) score_slot = 0, score_parity ^= 1;
    };
    for (int begin = 0; begin < tokens;) {
      const Segment g = segment_from(s, begin, tokens, p.window);
      begin = g.end;
      uint32_t values_slot = 0;   // of the first value part of the tile before
      for (int t = 0; t <= g.tiles; ++t) {
        // scores of tile t, and in their midst the output product of tile t - 1
        const int number = count + t;
        const uint32_t buffer = number & 1;
        const bool very_first = number == 0;   // the queries may still be on their way
        if (t < g.tiles) {
          score_part(0, buffer, very_first);
          if (score_parts > 2) score_part(1, buffer, very_first);
        }
        if (t > 0) {
          const int before = number - 1;
          wait(&s.weight[before & 1], (before >> 1) & 1);
          const uint32_t weights = tmem + kColsP + (before & 1) * (kKeys / 2);
          uint32_t slot = values_slot;
          for (int v = 0; v < own_parts; ++v) {
            const uint64_t b = descriptor(slot_addr + (kScoreSlots + slot) * 2 * kHalfBytes, true);
            const uint32_t idesc = 2 * v + 1 < own ? kIdescValues : kIdescHalf;
#pragma unroll
            for (int ks = 0; ks < kKeys / 16; ++ks)
              mma_tensor(tmem + kColsO + v * kPart, weights + ks * 8, b + ks * (2048 >> 4), idesc, t > 1 || ks > 0 ? 1u : 0u);
            commit(&s.empty[kScoreSlots + slot]);
            if (++slot == kValueSlots) slot = 0;
          }
          if (t == g.tiles) commit(&s.done);
        }
        if (t < g.tiles) {
          for (int i = score_parts > 2 ? 2 : 1; i < score_parts; ++i) score_part(i, buffer, very_first);
          values_slot = value_slot;
          for (int v = 0; v < own_parts; ++v) {
            const int half = others + 1 + 2 * v;
            const bool more = 2 * v + 1 < own;
            if (very_first) {
              wait(&s.query[half], 0);
              if (more) wait(&s.query[half + 1], 0);
            }
            wait(&s.full[kScoreSlots + value_slot], value_parity);
            const uint32_t keys = slot_addr + (kScoreSlots + value_slot) * 2 * kHalfBytes;
            scores_of(half, keys, buffer, 4);
            if (more) scores_of(half + 1, keys + kHalfBytes, buffer, 4);
            if (++value_slot == kValueSlots) value_slot = 0, value_parity ^= 1;
          }
          commit(&s.score[buffer]);
        }
      }
      count += g.tiles;
      fence_before();
      asm volatile("bar.sync 1, 160;" ::: "memory");
      fence_after();
    }
  } else {
    // ---------------- a warp per half of a slot: the half parts that come to it, one after another ----------------
    const int loader = warp - kFirstLoader, slot = loader >> 1, second = loader & 1;
    const bool of_values = slot >= kScoreSlots;
    const int ring = of_values ? kValueSlots : kScoreSlots, each = of_values ? own_parts : score_parts;   // slots, parts a tile
    const int piece = lane & 7, sub = lane >> 3;
    const uint32_t dst = shared_address(slots + loader * kHalfBytes);
    int number = of_values ? slot - kScoreSlots : slot, round = 0, count = 0;   // of the part, of the slot's use; tiles before this request
    // where keys lane and lane + 32 of a tile lie in the pools, -1: nowhere (zeros)
    int place_lo = -1, place_hi = -1;
    auto look_up = [&](const Segment& g, int tile_index) {
      const int* table = p.block_table + static_cast<size_t>(g.entry) * p.table_width;
      const int lo = (g.first_tile + tile_index) * kKeys + lane, hi = lo + 32;
      place_lo = place_hi = -1;
      if (lo >= g.first_key && lo < g.end_key) {
        const int page = table[lo / p.page_size];
        if (page >= 0) place_lo = page * p.page_size + lo % p.page_size;
      }
      if (hi >= g.first_key && hi < g.end_key) {
        const int page = table[hi / p.page_size];
        if (page >= 0) place_hi = page * p.page_size + hi % p.page_size;
      }
    };
    auto copy = [&](int i) {   // this warp's half of the i-th part of its ring's in a tile
      const bool rotated = !of_values && i == score_parts - 1;
      const int half = rotated ? others : (of_values ? others + 1 : 0) + 2 * i + second;
      // (a part may have one half only; the rotated one does)
      const bool there = rotated ? second == 0 : 2 * i + second < (of_values ? own : others);
      if (!there) return;
      const __nv_bfloat16* pool = (rotated ? p.v_pool : p.k_pool + column_of(half)) + piece * 8;
      const int stride = rotated ? p.rot : p.rank;
      const bool column = !rotated || piece * 8 < p.rot;
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const int r = sub + 4 * j;   // (rows 32 and on from j = 8 on)
        const int place = __shfl_sync(0xffffffffu, j < 8 ? place_lo : place_hi, r & 31);
        const bool valid = place >= 0 && column;
        copy_16(dst + piece_offset(r, piece), valid ? pool + static_cast<size_t>(place) * stride : p.k_pool, valid);
      }
      copy_commit();
    };
    bool queries_due = loader < halves;
    auto bring_queries = [&]() {   // half part `loader` of the queries, 32 rows of it at a time
      queries_due = false;
      const bool rotated = loader == others;
      const float f = rotated ? 1.0f : p.scale;
      const int column = rotated ? 0 : column_of(loader);
      const int c = piece * 8;
#pragma unroll 1
      for (int r0 = 0; r0 < kRows; r0 += 32) {
        float4 lo[8], hi[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int r = r0 + sub + 4 * j, global = row0 + r;
          lo[j] = hi[j] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
          if (r < rows && (!rotated || c < p.rot)) {
            const float* src = rotated ? p.q_rot + static_cast<size_t>(global) * p.rot + c
                : p.qa_heads + (static_cast<size_t>(global % p.heads) * p.padded_tokens + global / p.heads) * p.rank + column + c;
            lo[j] = *reinterpret_cast<const float4*>(src);
            hi[j] = *reinterpret_cast<const float4*>(src + 4);
          }
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          uint4 packed;
          __nv_bfloat162* pairs = reinterpret_cast<__nv_bfloat162*>(&packed);
          pairs[0] = __floats2bfloat162_rn(lo[j].x * f, lo[j].y * f);
          pairs[1] = __floats2bfloat162_rn(lo[j].z * f, lo[j].w * f);
          pairs[2] = __floats2bfloat162_rn(hi[j].x * f, hi[j].y * f);
          pairs[3] = __floats2bfloat162_rn(hi[j].z * f, hi[j].w * f);
          *reinterpret_cast<uint4*>(queries + loader * kQueryBytes + piece_offset(r0 + sub + 4 * j, piece)) = packed;
        }
      }
      fence_async();
      bar_arrive(&s.query[loader]);
    };
    bool waited = false;
    for (int begin = 0; begin < tokens;) {
      const Segment g = segment_from(s, begin, tokens, p.window);
      begin = g.end;
      if (number < (count + g.tiles) * each) look_up(g, number / each - count);
      if (!waited) {
        pdl_wait();   // (the block table is the host's)
        waited = true;
      }
      for (; number < (count + g.tiles) * each; number += ring, ++round) {
        if (round > 0) bar_wait<WAIT_EXPIRED>(&s.empty[slot], (round - 1) & 1, abort_flag, p.status);
        copy(number % each);
        if (number + ring < (count + g.tiles) * each) look_up(g, (number + ring) / each - count);
        if (queries_due) bring_queries();
        copy_wait<0>();
        fence_async();
        bar_arrive(&s.full[slot]);
      }
      count += g.tiles;
    }
    if (queries_due) bring_queries();   // (a slot that no part comes to)
  }
  fence_before();
  __syncthreads();
  if (warp == kIssuer) {
    fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols));
  }
}

}  // namespace latent_tc
