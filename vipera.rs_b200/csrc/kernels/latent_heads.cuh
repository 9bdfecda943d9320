// Attention over cached latents for steps that share their keys between many tokens: every head's keys and values are
// expanded once (bfloat16 caches, heads of 128 values and 64 rotated ones, values of 128), then the heads attend plainly.
//
//   rows      the keys any token of the step sees, request by request, copied out of their pages into runs of rows
//             (latent_gather_kernel); a request's run starts on a multiple of 128 rows, and what it is short of one is zero
//   expand    [k_h | v_h] = rows . [U_h | V_h]^T, one plain product over all heads (gemm_tc.cu)
//   attend    latent_heads_kernel: 128 queries of a request and a head to a block, which walks its keys
//
// A (query, key) pair costs a head 2 (128 + 64 + 128) operations here and 2 (2 rank + 64) over the latents themselves, 3.4
// times as many at a rank of 512; against that every key costs 2 x 256 rank operations once for all of the step's queries.
//
// The block: S = Q [k | kr]^T in tensor memory (tcgen05.mma 128 x 64 x 192, operands in shared memory), a softmax whose
// threads have a row each and leave the weights, rounded to bfloat16, in the columns the scores were in, O += P V with P
// read from there.  Tiles of 64 keys are dealt to two groups of four softmax warps, each with two score buffers, an output
// accumulator, two buffers for keys and two for values, an issuing warp and two loading warps of its own: a group's next
// scores are computed under its softmax, the two groups drift against one another, and the ending joins them.  208 KB of
// shared memory: Q 48, keys 4 x 24, values 4 x 16 (weights that stay in tensor memory are what makes room for these).
// The queries and, for the ending, the rows of the gate come by TMA as they are, in 32 bits, into space that the keys do not need
// yet or any more.  (The gate read from memory by the ending's threads held it up by some 9,000 clocks: 327 us below.)
// What bounds it: a block's start (set-up, queries: some 8 K clocks) and its softmax, 2.4 K clocks per 64 keys and group, of
// which the exponentials are 512 and scaling the output to a new maximum some 400; tensor cores are busy a third of the time.
// Measured: 2,048 tokens, 12 heads, rank 512, window 1,024: the mixer 287 -> 108 us; 1,748 tokens of four requests behind up
// to 3,000, 32 heads, a gate: 663 -> 306 us (over the latents, latent_tc.cuh, before; the same inputs again, in L2: with inputs
// that change 290 -> 113 and 668 -> 352).
// A value that is not finite shows in the outputs of the queries that see its key, and in no others: out of the tiles that some query
// of a block sees and another does not, such values are taken before the product and given back at the end.  Looking through these
// tiles costs 0.4 us of 112; with the product's own zeros times infinities up to 127 earlier tokens lost their outputs.
// Every wait is bounded; one that runs out leaves a code in the status word.
#pragma once

#include <cuda.h>

#include "latent_tc.cuh"

namespace latent_heads {

using namespace tcgen05;
using latent_tc::mma_tensor;
using latent_tc::piece_offset;
using latent_tc::power_of_two;
using latent_tc::tmem_load;
using latent_tc::tmem_load_wait;
using latent_tc::tmem_store;
using latent_tc::tmem_store_wait;

constexpr int kDim = 128, kRot = 64, kValues = 128;
constexpr int kQ = 128, kKeys = 64;                  // queries of a block, keys of a tile
constexpr int kRunRows = 128;                        // a request's run of rows starts on a multiple of this
constexpr int kQueryHalf = kQ * 128, kHalf = kKeys * 128;   // bytes of [rows][64 values]
constexpr int kQueryBytes = 3 * kQueryHalf, kKeyBytes = 3 * kHalf, kValueBytes = 2 * kHalf;
constexpr int kStagedPitch = kValues + 4;            // floats between rows of the ending's tile
constexpr int kRawPitch = kDim + kRot;               // and of the queries as they come
constexpr int kGroupThreads = 128, kSoftmaxThreads = 2 * kGroupThreads;
constexpr int kIssuer = 8, kLoader = 12, kThreads = 16 * 32;   // (two warps idle: register shares go by four warps)
constexpr int kSoftmaxRegisters = 184, kOtherRegisters = 72;
static_assert(256 * (kSoftmaxRegisters + kOtherRegisters) <= 65536, "the block's registers");
constexpr uint32_t kColsS = 0, kColsO = 256, kTmemCols = 512;   // scores 2 x 2 x 64, outputs 2 x 128
constexpr float kLog2e = 1.4426950408889634f;
enum { WAIT_EXPIRED = 6 };

struct Params {
  const float* q;                  // [tokens, q_width], from column q_off on head by head [128 | 64 not yet rotated]
  long long q_width;
  int q_off;
  const float* gate;               // pre-activations of the output gate, [tokens, gate_width], or null
  long long gate_width;
  const float* cos_table;          // [positions, 32]
  const float* sin_table;
  const float* sink;               // [heads] or null
  const int* entry_starts;         // [requests + 1]
  const int* entry_pos0;           // [requests]
  const int* block_table;
  const __nv_bfloat16* k_pool;     // latents
  const __nv_bfloat16* v_pool;     // rotated key parts
  __nv_bfloat16* rows;             // [row_capacity, rank]
  __nv_bfloat16* rot_rows;         // [row_capacity, 64]
  __nv_bfloat16* out;              // [tokens, heads * 128]
  int requests, heads, rank, table_width, page_size, window, pairing, row_capacity;
  float scale;
  int* status;
};

// A request's run of rows: its first key, how many keys, and the row it starts in.
struct Run { int entry, token0, count, pos0, first_key, keys, row0; };

// The request to which block of 128 rows, or tile of 128 queries, number `number` belongs, with `number` within it left
// in `within`; entry < 0: none.  A warp looks at 32 requests at a time, a lane each.
template <bool QUERIES>
__device__ __forceinline__ Run find_run(const Params& p, int number, int lane, int& within) {
  Run run{-1, 0, 0, 0, 0, 0, 0};
  int key_tiles_before = 0;
  within = number;
  for (int e0 = 0; e0 < p.requests; e0 += 32) {
    const int e = e0 + lane;
    int start = 0, count = 0, pos0 = 0;
    if (e < p.requests) {
      start = p.entry_starts[e];
      count = p.entry_starts[e + 1] - start;
      pos0 = p.entry_pos0[e];
    }
    const int first_key = p.window > 0 ? max(0, pos0 - p.window + 1) : 0;
    const int keys = count > 0 ? pos0 + count - first_key : 0;
    const int key_tiles = (keys + kRunRows - 1) / kRunRows, things = QUERIES ? (max(count, 0) + kQ - 1) / kQ : key_tiles;
    int before = things, key_before = key_tiles;
#pragma unroll
    for (int step = 1; step < 32; step <<= 1) {
      const int a = __shfl_up_sync(0xffffffffu, before, step), b = __shfl_up_sync(0xffffffffu, key_before, step);
      if (lane >= step) before += a, key_before += b;
    }
    const int all = __shfl_sync(0xffffffffu, before, 31), key_all = __shfl_sync(0xffffffffu, key_before, 31);
    before -= things;
    key_before -= key_tiles;
    const unsigned found = __ballot_sync(0xffffffffu, within >= before && within < before + things);
    if (found) {
      const int owner = __ffs(found) - 1;
      within -= __shfl_sync(0xffffffffu, before, owner);
      run.entry = e0 + owner;
      run.token0 = __shfl_sync(0xffffffffu, start, owner);
      run.count = __shfl_sync(0xffffffffu, count, owner);
      run.pos0 = __shfl_sync(0xffffffffu, pos0, owner);
      run.first_key = __shfl_sync(0xffffffffu, first_key, owner);
      run.keys = __shfl_sync(0xffffffffu, keys, owner);
      run.row0 = (key_tiles_before + __shfl_sync(0xffffffffu, key_before, owner)) * kRunRows;
      return run;
    }
    within -= all;
    key_tiles_before += key_all;
  }
  return run;
}

// 32 rows a block, in pieces of 16 bytes: the latents and the rotated parts of a run's keys, zeros behind its end.
constexpr int kGatherThreads = 256, kGatherRows = 32;

__global__ void __launch_bounds__(kGatherThreads)
latent_gather_kernel(const Params p) {
  __shared__ Run run_s;
  __shared__ int within_s;
  pdl_launch_dependents();
  if (threadIdx.x < 32) {   // (the step's requests are the host's, written before the step)
    int within;
    const Run run = find_run<false>(p, blockIdx.x / (kRunRows / kGatherRows), threadIdx.x, within);
    if (threadIdx.x == 0) run_s = run, within_s = within;
  }
  __syncthreads();
  const Run run = run_s;
  if (run.entry < 0) return;
  const int first = within_s * kRunRows + (blockIdx.x % (kRunRows / kGatherRows)) * kGatherRows;   // of the run
  const size_t row0 = static_cast<size_t>(run.row0) + first;
  const int pieces = p.rank / 8, each = pieces + kRot / 8;
  const int* table = p.block_table + static_cast<size_t>(run.entry) * p.table_width;
  pdl_wait();
  for (int i = threadIdx.x; i < kGatherRows * each; i += kGatherThreads) {
    const int r = i / each, piece = i % each;
    uint4 value = make_uint4(0, 0, 0, 0);
    if (first + r < run.keys) {
      const int key = run.first_key + first + r;
      const size_t slot = static_cast<size_t>(table[key / p.page_size]) * p.page_size + key % p.page_size;
      value = piece < pieces ? *reinterpret_cast<const uint4*>(p.k_pool + slot * p.rank + piece * 8)
                             : *reinterpret_cast<const uint4*>(p.v_pool + slot * kRot + (piece - pieces) * 8);
    }
    __nv_bfloat16* to = piece < pieces ? p.rows + (row0 + r) * p.rank + piece * 8 : p.rot_rows + (row0 + r) * kRot + (piece - pieces) * 8;
    *reinterpret_cast<uint4*>(to) = value;
  }
}

constexpr int kMostTakenOut = 6 * kKeys;
struct Shared {
  // per group and, but for the output's, per buffer
  uint64_t raw, query, scored, gate, key_full[2][2], key_empty[2][2], value_landed[2][2], value_looked[2][2], value_empty[2][2], score[2][2], weight[2][2], done[2], finished[2];
  uint32_t tmem_base;
  int abort_flag;
  int taken_out;
  int taken_out_key[kMostTakenOut];
  Run run;
  int tile;
  float2 told[2][kQ];   // a group's maxima and sums, for the other
};
constexpr int kGateBytes = kQ * kValues * 4;
constexpr int kSharedBytes = kQueryBytes + 4 * kKeyBytes + 4 * kValueBytes + static_cast<int>(sizeof(Shared)) + 1024;
static_assert(kSharedBytes <= 227 * 1024, "a block's shared memory");
static_assert(kGateBytes + kQ * kStagedPitch * 4 <= kQueryBytes + 4 * kKeyBytes && kQ * kRawPitch * 4 <= 4 * kKeyBytes, "what lies where queries and keys did, or will");

__device__ __forceinline__ void expect_bytes(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(shared_address(bar)), "r"(bytes) : "memory");
}
// a box [64 rows][64 columns]
__device__ __forceinline__ void load_box(void* dst, const CUtensorMap* map, uint64_t* bar, int column, int row) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(shared_address(dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(shared_address(bar)), "r"(column), "r"(row)
      : "memory");
}
// Halves of [rows][128 bytes], 128-byte swizzle, read with the contraction along the rows' bytes or (`down`) down the rows,
// the second 64 of an operand's columns one half further.
__device__ __forceinline__ uint64_t descriptor(uint32_t saddr, bool down) {
  return static_cast<uint64_t>((saddr & 0x3FFFFu) >> 4) | (static_cast<uint64_t>(down ? kHalf >> 4 : 1) << 16) |
         (static_cast<uint64_t>(1024 >> 4) << 32) | (static_cast<uint64_t>(1) << 46) | (static_cast<uint64_t>(2) << 61);
}
__device__ __forceinline__ uint32_t packed_pair(float a, float b) {
  const __nv_bfloat162 pair = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&pair);
}

// Pairs of bfloat16 numbers times zero: what was not finite leaves a number that is none.
__device__ __forceinline__ void times_zero(uint32_t& sum, const uint4& v) {
  asm("fma.rn.bf16x2 %0, %1, %5, %0;\nfma.rn.bf16x2 %0, %2, %5, %0;\nfma.rn.bf16x2 %0, %3, %5, %0;\nfma.rn.bf16x2 %0, %4, %5, %0;"
      : "+r"(sum) : "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w), "r"(0u));
}
__device__ __forceinline__ uint32_t without_wrong(uint32_t pair) {
  if ((pair & 0x7f80u) == 0x7f80u) pair &= 0xffff0000u;
  if ((pair & 0x7f800000u) == 0x7f800000u) pair &= 0x0000ffffu;
  return pair;
}

// Out of a tile of values [64 keys][128], its first key at position `key0`, go rows that no query of the block sees, whole, and of
// the others what is not finite.
__device__ __forceinline__ void take_out(Shared& s, uint8_t* tile, int lane, int key0, int first_key, int end_key) {
  for (int r = lane; r < kKeys; r += 32) {
    auto at = [&](int piece) { return reinterpret_cast<uint4*>(tile + (piece >> 3) * kHalf + piece_offset(r, piece & 7)); };
    if (key0 + r < first_key || key0 + r >= end_key) {   // it may be anything
#pragma unroll
      for (int piece = 0; piece < 16; ++piece) *at(piece) = make_uint4(0, 0, 0, 0);
      continue;
    }
    uint32_t sums[2] = {0u, 0u};
#pragma unroll
    for (int piece = 0; piece < 16; ++piece) times_zero(sums[piece & 1], *at(piece));
    if (((sums[0] | sums[1]) & 0x7f807f80u) != 0u) {
      for (int piece = 0; piece < 16; ++piece) {
        const uint4 v = *at(piece);
        *at(piece) = make_uint4(without_wrong(v.x), without_wrong(v.y), without_wrong(v.z), without_wrong(v.w));
      }
      const int place = atomicAdd(&s.taken_out, 1);
      if (place < kMostTakenOut) s.taken_out_key[place] = key0 + r;
    }
  }
}
// A query's 64 outputs get back what was taken out of the values from column `column` on of the keys that it sees.
__device__ __noinline__ void give_back(const Shared& s, const Params& p, const __nv_bfloat16* expanded, float* y, int column, int position) {
  const int first = p.window > 0 ? max(0, position - p.window + 1) : 0;
  for (int i = 0; i < min(s.taken_out, kMostTakenOut); ++i) {
    const int key = s.taken_out_key[i];
    if (key < first || key > position) continue;
    const __nv_bfloat16* v = expanded + static_cast<size_t>(s.run.row0 + key - s.run.first_key) * (2 * p.heads * kDim) + p.heads * kValues + column;
    for (int k = 0; k < 64; ++k) {
      const float value = __bfloat162float(v[k]);
      if (!isfinite(value)) y[k] += value;
    }
  }
}

// The largest of a row's 64 scores, three at a time.
__device__ __forceinline__ float largest_of(const uint32_t (&v)[kKeys]) {
  float m[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) m[j] = fmaxf(__uint_as_float(v[j]), __uint_as_float(v[4 + j]));
#pragma unroll
  for (int k = 8; k < kKeys; k += 8)
#pragma unroll
    for (int j = 0; j < 4; ++j) asm("max.f32 %0, %0, %1, %2;" : "+f"(m[j]) : "f"(__uint_as_float(v[k + j])), "f"(__uint_as_float(v[k + 4 + j])));
  return fmaxf(fmaxf(m[0], m[1]), fmaxf(m[2], m[3]));
}
// 2^(a * scale + shift) and the same of b, rounded to bfloat16 and packed; the rounded values join `sums`.
__device__ __forceinline__ uint32_t weights_of(uint32_t a, uint32_t b, float scale, float shift, unsigned long long& sums) {
  float x, y;
  asm("{\n .reg .b64 v, f, s;\n mov.b64 v, {%2, %3};\n mov.b64 f, {%4, %4};\n mov.b64 s, {%5, %5};\n fma.rn.f32x2 v, v, f, s;\n mov.b64 {%0, %1}, v;\n}\n"
      : "=f"(x), "=f"(y) : "r"(a), "r"(b), "f"(scale), "f"(shift));
  const __nv_bfloat162 pair = __floats2bfloat162_rn(power_of_two(x), power_of_two(y));
  const uint32_t packed = *reinterpret_cast<const uint32_t*>(&pair);
  asm("{\n .reg .b64 v;\n mov.b64 v, {%1, %2};\n add.rn.f32x2 %0, %0, v;\n}\n" : "+l"(sums) : "r"(packed << 16), "r"(packed & 0xffff0000u));
  return packed;
}

__global__ void __launch_bounds__(kThreads, 1)
latent_heads_kernel(const __grid_constant__ CUtensorMap expanded_map, const __grid_constant__ CUtensorMap rot_map,
                    const __grid_constant__ CUtensorMap query_map, const __grid_constant__ CUtensorMap gate_map, const __nv_bfloat16* __restrict__ expanded, const Params p) {
  extern __shared__ uint8_t latent_heads_raw[];
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(latent_heads_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint8_t* queries = base;                          // three halves
  uint8_t* keys = base + kQueryBytes;               // [group][buffer] of three halves
  uint8_t* values = keys + 4 * kKeyBytes;           // [group][buffer] of two
  Shared& s = *reinterpret_cast<Shared*>(values + 4 * kValueBytes);
  volatile int* abort_flag = &s.abort_flag;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, head = blockIdx.x;
  pdl_launch_dependents();
  // Blocks are numbered from the back and heads run along x, so that the longest histories of a prompt start first.
  // (The step's requests are the host's: they may be read before the wait.)
  if (warp == 0) {
    int tile;
    const Run run = find_run<true>(p, static_cast<int>(gridDim.y) - 1 - static_cast<int>(blockIdx.y), lane, tile);
    if (lane == 0) s.run = run, s.tile = tile;
  }
  __syncthreads();
  const Run run = s.run;
  if (run.entry < 0) return;
  const int token0 = run.token0 + s.tile * kQ, tokens = min(kQ, run.token0 + run.count - token0);
  const int pos0 = run.pos0 + s.tile * kQ;                                    // of the tile's first query
  const int first_key = p.window > 0 ? max(0, pos0 - p.window + 1) : 0;       // that any of its queries sees
  const int end_key = pos0 + tokens;
  const int first_tile = (first_key - run.first_key) / kKeys;                 // within the run
  const int num_tiles = (end_key - run.first_key + kKeys - 1) / kKeys - first_tile;
  const int key_base = run.first_key + first_tile * kKeys;                    // position of the first tile's first key

  if (tid == 0) {
    bar_init(&s.raw, 1);
    bar_init(&s.query, kSoftmaxThreads);
    bar_init(&s.scored, 2);
    bar_init(&s.gate, 1);
    for (int g = 0; g < 2; ++g) {
      for (int b = 0; b < 2; ++b) {
        bar_init(&s.key_full[g][b], 1);
        bar_init(&s.key_empty[g][b], 1);
        bar_init(&s.value_landed[g][b], 1);
        bar_init(&s.value_looked[g][b], 32);
        bar_init(&s.value_empty[g][b], 1);
        bar_init(&s.score[g][b], 1);
        bar_init(&s.weight[g][b], kGroupThreads);
      }
      bar_init(&s.done[g], 1);
      bar_init(&s.finished[g], 2);   // the last product's end, and its issuer's word that what was taken out stands written
    }
    s.abort_flag = s.taken_out = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kIssuer) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(shared_address(&s.tmem_base)), "r"(kTmemCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = s.tmem_base;
  // a value tile with rows that no query of the block may see: their weights are zero, but what they hold may be anything
  auto bounded = [&](int j) { const int key0 = key_base + j * kKeys; return key0 + kKeys - 1 > pos0 || (p.window > 0 && key0 < end_key - p.window); };

  if (warp < kIssuer) {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kSoftmaxRegisters));
    // ---------------- queries, then softmax and ending: thread = query, group = every other tile ----------------
    // The queries come as they are, 32-bit rows of 192 values, where the keys will be; each thread then takes four pieces of
    // eight rotated values and eight of the others into bfloat16.  The angles' tables are no kernel's result.
    const int own_piece = tid & 7;
    float4 c[4][2], n[4][2];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int row = (j * kSoftmaxThreads + tid) >> 3;
      const size_t at = static_cast<size_t>(pos0 + min(row, tokens - 1)) * (kRot / 2);
      const float4* cs = reinterpret_cast<const float4*>(p.cos_table + at);
      const float4* sn = reinterpret_cast<const float4*>(p.sin_table + at);
      if (p.pairing) {
        c[j][0] = cs[2 * (own_piece & 3)], c[j][1] = cs[2 * (own_piece & 3) + 1];
        n[j][0] = sn[2 * (own_piece & 3)], n[j][1] = sn[2 * (own_piece & 3) + 1];
      } else {
        c[j][0] = cs[own_piece], n[j][0] = sn[own_piece];
        c[j][1] = n[j][1] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      }
    }
    pdl_wait();
    if (tid == 0) {
      expect_bytes(&s.raw, kQ * kRawPitch * 4);
      load_box(keys, &query_map, &s.raw, p.q_off + head * (kDim + kRot), token0);
    }
    __syncwarp();
    bar_wait<WAIT_EXPIRED>(&s.raw, 0, abort_flag, p.status);
    const float* raw = reinterpret_cast<const float*>(keys);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int row = (j * kSoftmaxThreads + tid) >> 3, piece = own_piece;
      uint4 to = make_uint4(0u, 0u, 0u, 0u);
      if (row < tokens) {
        const float4* src = reinterpret_cast<const float4*>(raw + row * kRawPitch + kDim);
        const float4 q0 = src[2 * piece], q1 = src[2 * piece + 1];
        if (p.pairing) {   // values half of the part apart turn together
          const float4 o0 = src[2 * (piece ^ 4)], o1 = src[2 * (piece ^ 4) + 1];
          const float f = piece < 4 ? -1.0f : 1.0f;
          to.x = packed_pair(q0.x * c[j][0].x + f * (o0.x * n[j][0].x), q0.y * c[j][0].y + f * (o0.y * n[j][0].y));
          to.y = packed_pair(q0.z * c[j][0].z + f * (o0.z * n[j][0].z), q0.w * c[j][0].w + f * (o0.w * n[j][0].w));
          to.z = packed_pair(q1.x * c[j][1].x + f * (o1.x * n[j][1].x), q1.y * c[j][1].y + f * (o1.y * n[j][1].y));
          to.w = packed_pair(q1.z * c[j][1].z + f * (o1.z * n[j][1].z), q1.w * c[j][1].w + f * (o1.w * n[j][1].w));
        } else {           // neighbours do
          to.x = packed_pair(q0.x * c[j][0].x - q0.y * n[j][0].x, q0.y * c[j][0].x + q0.x * n[j][0].x);
          to.y = packed_pair(q0.z * c[j][0].y - q0.w * n[j][0].y, q0.w * c[j][0].y + q0.z * n[j][0].y);
          to.z = packed_pair(q1.x * c[j][0].z - q1.y * n[j][0].z, q1.y * c[j][0].z + q1.x * n[j][0].z);
          to.w = packed_pair(q1.z * c[j][0].w - q1.w * n[j][0].w, q1.w * c[j][0].w + q1.z * n[j][0].w);
        }
      }
      *reinterpret_cast<uint4*>(queries + 2 * kQueryHalf + piece_offset(row, piece)) = to;
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int i = j * kSoftmaxThreads + tid, row = i >> 4, piece = i & 15;
      const float4* src = reinterpret_cast<const float4*>(raw + row * kRawPitch) + 2 * piece;
      const float4 q0 = src[0], q1 = src[1];
      *reinterpret_cast<uint4*>(queries + (piece >> 3) * kQueryHalf + piece_offset(row, piece & 7)) =
          row < tokens ? make_uint4(packed_pair(q0.x, q0.y), packed_pair(q0.z, q0.w), packed_pair(q1.x, q1.y), packed_pair(q1.z, q1.w)) : make_uint4(0u, 0u, 0u, 0u);
    }
    fence_async();
    bar_arrive(&s.query);

    const int quarter = warp & 3, group = warp >> 2, row = quarter * 32 + lane, position = pos0 + row;
    const int last = row < tokens ? position : -1, first = p.window > 0 ? max(0, position - p.window + 1) : 0;
    const float scale_log2 = p.scale * kLog2e;
    const uint32_t lanes = tmem + (static_cast<uint32_t>(quarter * 32) << 16);
    const uint32_t o_addr = lanes + kColsO + group * 128;
    const int group_tiles = (num_tiles - group + 1) / 2;   // tiles group, group + 2, ...
    float row_max = -INFINITY, row_sum = 0.0f;             // the max in powers of two
    for (int i = 0; i < group_tiles; ++i) {
      const int key0 = key_base + (2 * i + group) * kKeys, buffer = i & 1;
      const uint32_t s_addr = lanes + kColsS + (2 * group + buffer) * kKeys;
      bar_wait<WAIT_EXPIRED>(&s.score[group][buffer], (i >> 1) & 1, abort_flag, p.status);
      fence_after();
      uint32_t v[kKeys];
      tmem_load(s_addr, *reinterpret_cast<uint32_t(*)[32]>(&v[0]));
      tmem_load(s_addr + 32, *reinterpret_cast<uint32_t(*)[32]>(&v[32]));
      tmem_load_wait();
      if (key0 + kKeys - 1 > pos0 || (p.window > 0 && key0 < end_key - p.window) || tokens < kQ) {   // some row needs a mask
#pragma unroll
        for (int k = 0; k < kKeys; ++k)
          if (key0 + k < first || key0 + k > last) v[k] = __float_as_uint(-INFINITY);
      }
      const float new_max = fmaxf(row_max, largest_of(v) * scale_log2);
      const float alpha = new_max == row_max ? 1.0f : power_of_two(row_max - new_max);
      row_max = new_max;
      row_sum *= alpha;
      if (i > 0 && __any_sync(0xffffffffu, alpha != 1.0f)) {
        bar_wait<WAIT_EXPIRED>(&s.done[group], (i - 1) & 1, abort_flag, p.status);
        fence_after();
#pragma unroll 1
        for (int c = 0; c < kValues; c += 64) {
          uint32_t o[64];
          tmem_load(o_addr + c, *reinterpret_cast<uint32_t(*)[32]>(&o[0]));
          tmem_load(o_addr + c + 32, *reinterpret_cast<uint32_t(*)[32]>(&o[32]));
          tmem_load_wait();
#pragma unroll
          for (int k = 0; k < 64; ++k) o[k] = __float_as_uint(__uint_as_float(o[k]) * alpha);
          tmem_store(o_addr + c, *reinterpret_cast<const uint32_t(*)[32]>(&o[0]));
          tmem_store(o_addr + c + 32, *reinterpret_cast<const uint32_t(*)[32]>(&o[32]));
        }
      }
      // weights 2^(s * scale * log2 e - max), rounded to bfloat16, over scores that are in registers by now; their sum is
      // that of the rounded ones
      const float shift = row_max == -INFINITY ? 0.0f : row_max;   // (a row that has seen no key: 2^-inf = 0)
      unsigned long long sums = 0;
      uint32_t packed[32];
#pragma unroll
      for (int k = 0; k < 32; ++k) packed[k] = weights_of(v[2 * k], v[2 * k + 1], scale_log2, -shift, sums);
      tmem_store(s_addr, packed);
      row_sum += sum_of_pair(sums);
      tmem_store_wait();
      fence_before();
      bar_arrive(&s.weight[group][buffer]);
    }
    // ---------------- the two groups' folds are joined ----------------
    // (`done` would not do: the last scores tell only that the third product from the end is done, whose parity is the last's)
    if (group_tiles > 0) bar_wait<WAIT_EXPIRED>(&s.finished[group], 0, abort_flag, p.status);
    fence_after();
    s.told[group][row] = make_float2(row_max, row_sum);
    fence_before();
    asm volatile("bar.sync %0, 64;" ::"r"(1 + quarter) : "memory");
    fence_after();
    const float2 other = s.told[group ^ 1][row];
    const bool own_counts = group_tiles > 0, other_counts = group == 1 || num_tiles > 1;   // (an accumulator never written holds anything)
    const float joint_max = fmaxf(row_max, other.x);
    const float own_weight = row_max == -INFINITY ? 0.0f : power_of_two(row_max - joint_max);
    const float other_weight = other.x == -INFINITY ? 0.0f : power_of_two(other.x - joint_max);
    float joint_sum = row_sum * own_weight + other.y * other_weight;
    if (p.sink != nullptr && joint_max > -INFINITY) joint_sum += exp2f(p.sink[head] * kLog2e - joint_max);
    const float inverse = joint_sum > 0.0f ? 1.0f / joint_sum : 0.0f;
    const float own_factor = own_weight * inverse, other_factor = other_weight * inverse;
    const uint32_t other_o = lanes + kColsO + (group ^ 1) * 128;
    // each group lays out half of the columns behind the gate, where keys were (every product that read them is done)
    float* staged = reinterpret_cast<float*>(base + kGateBytes);
#pragma unroll 1
    for (int c = group * 64; c < group * 64 + 64; c += 32) {
      uint32_t a[32], b[32];
      if (own_counts) tmem_load(o_addr + c, a);
      if (other_counts) tmem_load(other_o + c, b);
      tmem_load_wait();
      float y[32];
#pragma unroll
      for (int k = 0; k < 32; ++k) {
        y[k] = own_counts ? __uint_as_float(a[k]) * own_factor : 0.0f;
        if (other_counts) y[k] = fmaf(__uint_as_float(b[k]), other_factor, y[k]);
      }
#pragma unroll
      for (int k = 0; k < 32; k += 4) *reinterpret_cast<float4*>(staged + row * kStagedPitch + c + k) = make_float4(y[k], y[k + 1], y[k + 2], y[k + 3]);
    }
    if (s.taken_out > 0 && row < tokens) give_back(s, p, expanded, staged + row * kStagedPitch + group * 64, head * kValues + group * 64, pos0 + row);
    asm volatile("bar.sync 6, 256;" ::: "memory");
    if (p.gate != nullptr) bar_wait<WAIT_EXPIRED>(&s.gate, 0, abort_flag, p.status);
    if (!*abort_flag) {   // neighbouring threads write a row
      const int piece = tid & 15;
      auto opened = [](float y, float z) { return y * sigmoid(z); };
      // (a row at a time: unrolled, this takes registers from the softmax above, 111.5 us for 108.3)
#pragma unroll 1
      for (int j = 0; j < 8; ++j) {
        const int r = (j * kSoftmaxThreads + tid) >> 4;
        const float4* from = reinterpret_cast<const float4*>(staged + r * kStagedPitch + piece * 8);
        float4 lo = from[0], hi = from[1];
        if (p.gate != nullptr) {
          const float4* z = reinterpret_cast<const float4*>(base) + r * (kValues / 4) + 2 * piece;
          const float4 a = z[0], b = z[1];
          lo = make_float4(opened(lo.x, a.x), opened(lo.y, a.y), opened(lo.z, a.z), opened(lo.w, a.w));
          hi = make_float4(opened(hi.x, b.x), opened(hi.y, b.y), opened(hi.z, b.z), opened(hi.w, b.w));
        }
        if (r < tokens)
          *reinterpret_cast<uint4*>(p.out + (static_cast<size_t>(token0 + r) * p.heads + head) * kValues + piece * 8) =
              make_uint4(packed_pair(lo.x, lo.y), packed_pair(lo.z, lo.w), packed_pair(hi.x, hi.y), packed_pair(hi.z, hi.w));
      }
    }
  } else if (warp < kLoader) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kOtherRegisters));
    // ---------------- products: a warp a group ----------------
    if (warp < kIssuer + 2) {
      const int g = warp - kIssuer, group_tiles = (num_tiles - g + 1) / 2;
      constexpr uint32_t kCommon = (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(kQ >> 4) << 24);
      constexpr uint32_t kScores = kCommon | (static_cast<uint32_t>(kKeys >> 3) << 17);
      constexpr uint32_t kOutputs = kCommon | (static_cast<uint32_t>(kValues >> 3) << 17) | (1u << 16);
      const uint32_t q_addr = shared_address(queries), k_addr = shared_address(keys + 2 * g * kKeyBytes), v_addr = shared_address(values + 2 * g * kValueBytes);
      const uint32_t s_tmem = tmem + kColsS + 2 * g * kKeys, o_tmem = tmem + kColsO + g * 128;
      uint32_t looked = 0;   // the bounded tiles' parities, a bit per buffer
      auto scores = [&](int i) {
        const uint32_t buffer = i & 1;
        bar_wait<WAIT_EXPIRED>(&s.key_full[g][buffer], (i >> 1) & 1, abort_flag, p.status);
        fence_after();
#pragma unroll
        for (int k = 0; k < (kDim + kRot) / 16; ++k) {
          const uint32_t step = (k & 3) * 32;
          mma_shared(s_tmem + buffer * kKeys, descriptor(q_addr + (k >> 2) * kQueryHalf + step, false),
                     descriptor(k_addr + buffer * kKeyBytes + (k >> 2) * kHalf + step, false), kScores, k > 0 ? 1u : 0u);
        }
        commit(&s.score[g][buffer]);
        commit(&s.key_empty[g][buffer]);
      };
      if (group_tiles > 0) {
        bar_wait<WAIT_EXPIRED>(&s.query, 0, abort_flag, p.status);
        scores(0);
      }
      if (group_tiles > 1) scores(1);
      for (int i = 0; i < group_tiles; ++i) {
        const uint32_t buffer = i & 1;
        if (bounded(2 * i + g)) {
          bar_wait<WAIT_EXPIRED>(&s.value_looked[g][buffer], (looked >> buffer) & 1, abort_flag, p.status);
          looked ^= 1u << buffer;
        } else {
          bar_wait<WAIT_EXPIRED>(&s.value_landed[g][buffer], (i >> 1) & 1, abort_flag, p.status);
        }
        bar_wait<WAIT_EXPIRED>(&s.weight[g][buffer], (i >> 1) & 1, abort_flag, p.status);
        fence_after();
#pragma unroll
        for (int k = 0; k < kKeys / 16; ++k)
          mma_tensor(o_tmem, s_tmem + buffer * kKeys + 8 * k, descriptor(v_addr + buffer * kValueBytes + k * 2048, true), kOutputs, (i > 0 || k > 0) ? 1u : 0u);
        commit(&s.done[g]);
        if (i + 1 == group_tiles) {
          commit(&s.finished[g]);
          if (lane == 0) bar_arrive(&s.finished[g]);
        }
        commit(&s.value_empty[g][buffer]);
        if (i + 2 < group_tiles) {
          bar_wait<WAIT_EXPIRED>(&s.done[g], i & 1, abort_flag, p.status);   // (it reads the weights from the scores' columns)
          scores(i + 2);
        }
      }
    }
  } else {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kOtherRegisters));
    // ---------------- loads: a warp for either group's keys and values ----------------
    const int g = (warp - kLoader) >> 1, group_tiles = (num_tiles - g + 1) / 2;
    const bool brings_values = ((warp - kLoader) & 1) != 0;
    pdl_wait();
    if (!brings_values) bar_wait<WAIT_EXPIRED>(&s.query, 0, abort_flag, p.status);   // the queries lay where the keys go
    // (a bounded tile's values are looked through behind the request for the next tile)
    for (int i = 0; i <= group_tiles; ++i) {
      if (i < group_tiles) {
        const int j = 2 * i + g, buffer = i & 1, row = run.row0 + (first_tile + j) * kKeys;
        uint8_t* tile = brings_values ? values + (2 * g + buffer) * kValueBytes : keys + (2 * g + buffer) * kKeyBytes;
        if (i > 1)
          bar_wait<WAIT_EXPIRED>(brings_values ? &s.value_empty[g][buffer] : &s.key_empty[g][buffer], ((i >> 1) - 1) & 1, abort_flag, p.status);
        if (__any_sync(0xffffffffu, *abort_flag)) break;   // (what is in flight is waited for below)
        if (lane == 0) {
          uint64_t* full = brings_values ? &s.value_landed[g][buffer] : &s.key_full[g][buffer];
          const int column = brings_values ? (p.heads + head) * kValues : head * kDim;
          expect_bytes(full, brings_values ? kValueBytes : kKeyBytes);
          for (int h = 0; h < 2; ++h) load_box(tile + h * kHalf, &expanded_map, full, column + 64 * h, row);
          if (!brings_values) load_box(tile + 2 * kHalf, &rot_map, full, 0, row);
        }
        __syncwarp();
      }
      const int before = i - 1, j = 2 * before + g, buffer = before & 1;
      if (brings_values && before >= 0 && bounded(j)) {
        bar_wait<WAIT_EXPIRED>(&s.value_landed[g][buffer], (before >> 1) & 1, abort_flag, p.status);
        take_out(s, values + (2 * g + buffer) * kValueBytes, lane, key_base + j * kKeys, first_key, end_key);
        fence_async();
        bar_arrive(&s.value_looked[g][buffer]);
      }
    }
    // The gate's rows come where the queries and the first keys were, behind the last scores of both groups: the last softmax
    // and product run meanwhile.  (Loaded by the ending's threads they held it up by 9,000 clocks.)
    if (!brings_values && p.gate != nullptr) {
      if (group_tiles > 0) bar_wait<WAIT_EXPIRED>(&s.key_empty[g][(group_tiles - 1) & 1], ((group_tiles - 1) >> 1) & 1, abort_flag, p.status);
      if (lane == 0) bar_arrive(&s.scored);
      if (g == 0) bar_wait<WAIT_EXPIRED>(&s.scored, 0, abort_flag, p.status);
      if (g == 0 && lane == 0 && !*abort_flag) {
        expect_bytes(&s.gate, kGateBytes);
        load_box(base, &gate_map, &s.gate, head * kValues, token0);
      }
      __syncwarp();
    }
  }
  fence_before();
  __syncthreads();
  if (*abort_flag && tid == 0)
    for (int i = 0; i < 1000; ++i) __nanosleep(1000);   // loads may still be landing in this block's shared memory
  __syncthreads();
  if (warp == kIssuer) {
    fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols));
  }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// [rows, columns] of bfloat16 in boxes of 64 rows x 64 columns, 128-byte swizzle; or of 32-bit numbers (queries, gate)
// in boxes of 128 rows x `raw_columns`, as they are, rows `pitch` apart
inline int make_map(CUtensorMap* map, const void* base, int rows, long long columns, int raw_columns = 0, long long pitch = 0) {
  void* entry = nullptr;
  cudaDriverEntryPointQueryResult result;
  if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &entry, cudaEnableDefault, &result) != cudaSuccess ||
      result != cudaDriverEntryPointSuccess || !entry)
    return VIPERA_NO_DRIVER_ENTRY;
  cuuint64_t dims[2] = {static_cast<cuuint64_t>(columns), static_cast<cuuint64_t>(rows)};
  const bool raw = raw_columns > 0;
  cuuint64_t strides[1] = {static_cast<cuuint64_t>(raw ? pitch * 4 : columns * 2)};
  cuuint32_t box[2] = {static_cast<cuuint32_t>(raw ? raw_columns : 64), static_cast<cuuint32_t>(raw ? kQ : kKeys)}, elem[2] = {1, 1};
  const CUresult r = reinterpret_cast<EncodeTiledFn>(entry)(
      map, raw ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, elem,
      CU_TENSOR_MAP_INTERLEAVE_NONE, raw ? CU_TENSOR_MAP_SWIZZLE_NONE : CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? VIPERA_OK : VIPERA_BAD_ARGUMENT;
}

// stage 1: the rows; stage 2 (behind the product that leaves `expanded` [row_capacity, 2 * heads * 128]): the attention
inline int launch(const Params& p, const void* expanded, int num_tokens, int stage, cudaStream_t s) {
  const uintptr_t bases = reinterpret_cast<uintptr_t>(p.k_pool) | reinterpret_cast<uintptr_t>(p.v_pool) | reinterpret_cast<uintptr_t>(p.rows) |
                          reinterpret_cast<uintptr_t>(p.rot_rows) | reinterpret_cast<uintptr_t>(p.out) | reinterpret_cast<uintptr_t>(p.q) |
                          reinterpret_cast<uintptr_t>(p.gate) | reinterpret_cast<uintptr_t>(expanded) | reinterpret_cast<uintptr_t>(p.cos_table) | reinterpret_cast<uintptr_t>(p.sin_table);
  if ((bases & 15) || (p.q_width & 3) || (p.q_off & 3) || (p.gate_width & 3)) return VIPERA_BAD_ARGUMENT;
  if (p.row_capacity % kRunRows != 0 || p.rank % 8 != 0 || p.requests <= 0 || !p.status) return VIPERA_BAD_ARGUMENT;
  if (stage == 1)
    return vipera_launch(latent_gather_kernel, dim3(p.row_capacity / kGatherRows), dim3(kGatherThreads), 0, s, p);
  CUtensorMap expanded_map, rot_map, query_map, gate_map;
  int status = make_map(&expanded_map, expanded, p.row_capacity, 2 * p.heads * kDim);
  if (status == VIPERA_OK) status = make_map(&rot_map, p.rot_rows, p.row_capacity, kRot);
  if (status == VIPERA_OK) status = make_map(&query_map, p.q, num_tokens, p.q_width, kRawPitch, p.q_width);
  if (status == VIPERA_OK)   // (without a gate any valid map)
    status = p.gate != nullptr ? make_map(&gate_map, p.gate, num_tokens, p.heads * kValues, kValues, p.gate_width)
                               : make_map(&gate_map, p.rot_rows, p.row_capacity, kRot);
  if (status != VIPERA_OK) return status;
  static SharedMemoryOptIn opt_in;
  if ((status = opt_in.ask(reinterpret_cast<const void*>(latent_heads_kernel), kSharedBytes)) != 0) return status;
  // at most one partly filled tile per request beyond the full ones
  return vipera_launch(latent_heads_kernel, dim3(p.heads, (num_tokens + kQ - 1) / kQ + p.requests), dim3(kThreads), kSharedBytes, s,
                       expanded_map, rot_map, query_map, gate_map, static_cast<const __nv_bfloat16*>(expanded), p);
}

}  // namespace latent_heads
