// The chunked form of linear attention whose state decays, in 32 bits on the CUDA cores: two products
// per chunk of kLinearChunk tokens instead of a walk over its tokens.
//
// Per head S [d, dv] with S_t = diag(a_t) S_(t-1) + k_t v_t^T and o_t = S_t^T q_t.  With B_t the sum of the
// chunk's log decays up to and with token t, and S the state at the chunk's start,
//
//   E       = sum_s (e^(B_end - B_s) k_s) v_s^T                          (linear_ends_kernel)
//   o_t     = (e^(B_t) q_t) S + sum_(s <= t) A_ts v_s,   A_ts = sum_c q_tc k_sc e^(B_tc - B_sc)   (linear_outputs_kernel)
//
// and the caller walks the chunks in between (start' = e^(B_end) start + E).  CHANNEL: a decay per key
// channel, its logarithms in `log_decay`; A is then a plain product of q e^(B_t - B_m) and k e^(B_m - B_s)
// with B_m in the chunk's middle, as long as no channel decays by more than e^-60 over the chunk (the
// factors stay in range).  Else the chunk is taken as four of 16 tokens: q against its sixteen's start, k against its
// end, each at most 1, and what lies between (or, within a sixteen, is too much) as a factor of its own; where some
// channel decays by more than e^-60 within a sixteen, that sixteen's decays are multiplied up token by token.  4 heads of
// 128 x 256, 400 tokens, every channel far: 126 us the mixer (walks: 135, multiplied up through whole chunks: 378), 120 with
// none.  Otherwise a constant decay per head: A = (q k) a^(t - s) from a table of powers, whatever the decay, and q, k and v are
// the silu of what `proj` holds.
//
// What bounds it: multiply-adds, and the instructions around them.  A walk pays five
// instructions per state element and token (three with outputs, two for the chunks' ends); the
// products pay 2.4 multiply-adds, in register tiles of 8 x 8, sixteen warps a multiprocessor (tiles of 8 x 16 with
// half as many warps read less but waited longer for their loads).
// 6 heads of 128 x 256, 2,048 tokens: 46 and 67 us instead of walks of 113 and 153 us (and of 28 us that
// applied the silu in place); 8 heads of 128 x 256, 2,002 tokens, decays per channel: 45 and 79 us
// instead of 119 and 153 us, and one share of partial outputs instead of eight (84 -> 19 us to add and norm them).
#pragma once

#include "simt.cuh"

constexpr int kLinearChunk = 64;
constexpr int kLinearPitch = kLinearChunk + 4;
constexpr float kLinearMostDecay = 60.0f;

struct LinearArgs {
  const float* proj;        // [tokens, proj_width]
  long long proj_width;
  int q_off, k_off, v_off;
  const float* log_decay;   // CHANNEL: [tokens, heads * d]
  const float* alpha;       // CHANNEL: the decays themselves, the same shape
  const float* decay;       // otherwise: [heads]
  const int* entry_starts;  // [entries + 1]
  float* chunk_state;       // [jobs, heads * d * dv]
  float* chunk_decay;       // CHANNEL: [jobs, heads * d] receives B_end
  float* out;               // [tokens, heads * dv]
  int num_entries, heads, d, dv;
  float q_scale;
};

// What the chunked form takes: rows of whole 16-byte pieces, heads of up to 256 key channels.
static inline bool linear_chunks_take(const LinearArgs& p) {
  const uintptr_t bases = reinterpret_cast<uintptr_t>(p.proj) | reinterpret_cast<uintptr_t>(p.chunk_state) | reinterpret_cast<uintptr_t>(p.out) |
                          reinterpret_cast<uintptr_t>(p.alpha);
  return p.d % 4 == 0 && p.dv % 4 == 0 && p.d <= 256 && p.proj_width % 4 == 0 && p.v_off % 4 == 0 && (bases & 15) == 0;
}

__device__ __forceinline__ float linear_silu(float z) { return z / (1.0f + expf(-z)); }

// The chunk a job index names, for the whole block: its first token and how many it has (0: none).
__device__ __forceinline__ int2 linear_chunk_of(const int* __restrict__ entry_starts, int num_entries, int job) {
  __shared__ int2 found;
  if (threadIdx.x == 0) {
    found = make_int2(0, 0);
    int before = 0;
    for (int e = 0; e < num_entries; ++e) {
      const int begin = entry_starts[e], count = entry_starts[e + 1] - begin;
      const int chunks = (count + kLinearChunk - 1) / kLinearChunk;
      if (job < before + chunks) {
        const int first = (job - before) * kLinearChunk;
        found = make_int2(begin + first, min(kLinearChunk, count - first));
        break;
      }
      before += chunks;
    }
  }
  __syncthreads();
  return found;
}

// ---------------------------------------------------------------------------------------
// E for 128 key channels and 128 values of a (chunk, head).
// ---------------------------------------------------------------------------------------
constexpr int kEndRows = 128, kEndColumns = 128, kEndThreads = 256;
constexpr int kEndBytes = kLinearChunk * (kEndRows + kEndColumns) * 4;

template <bool CHANNEL>
__global__ void __launch_bounds__(kEndThreads, 2)
linear_ends_kernel(const LinearArgs p) {
  extern __shared__ __align__(16) float ends_shared[];
  float* ks = ends_shared;                                // [token][kEndRows]
  float* vs = ends_shared + kLinearChunk * kEndRows;      // [token][kEndColumns]
  __shared__ float power[kLinearChunk];
  __shared__ float later[kEndRows];   // what the second half of the chunk decays by
  pdl_launch_dependents();
  const int tid = threadIdx.x, h = blockIdx.y, job = blockIdx.z;
  const int column_tiles = (p.dv + kEndColumns - 1) / kEndColumns;
  const int row0 = blockIdx.x / column_tiles * kEndRows, column0 = blockIdx.x % column_tiles * kEndColumns;
  const int2 chunk = linear_chunk_of(p.entry_starts, p.num_entries, job);
  const int first = chunk.x, count = chunk.y;
  if (count == 0) return;
  pdl_wait();
  // keys: a channel and half of the chunk's tokens a thread
  constexpr int kHalf = kLinearChunk / 2;
  const int own = tid % kEndRows, part = tid / kEndRows, c = row0 + own;
  const bool live = c < p.d;
  const int t0 = part * kHalf, mine = min(max(count - t0, 0), kHalf);
  float x[kHalf], y[kHalf];
  {
    const float* k = p.proj + p.k_off + static_cast<size_t>(h) * p.d + (live ? c : 0);
    const float* b = CHANNEL ? p.log_decay + static_cast<size_t>(h) * p.d + (live ? c : 0) : nullptr;
#pragma unroll
    for (int j = 0; j < kHalf; ++j) {
      const size_t t = first + min(t0 + j, count - 1);
      x[j] = live && j < mine ? k[t * p.proj_width] : 0.0f;
      y[j] = CHANNEL && live && j < mine ? b[t * p.heads * p.d] : 0.0f;
    }
  }
  if (!CHANNEL && tid < kLinearChunk) {
    // by repeated multiplication, a thread a power
    float w = 1.0f;
    const float a = p.decay[h];
    for (int i = 0; i < tid; ++i) w *= a;
    power[tid] = w;
  }
  float left = 0.0f;   // from the last token back: what is left of each at the chunk's end
  if (CHANNEL) {
#pragma unroll
    for (int j = kHalf - 1; j >= 0; --j) left += y[j];
    if (part == 1) later[own] = left;
  }
  __syncthreads();
  if (CHANNEL) {
    if (part == 0 && live && column0 == 0) p.chunk_decay[(static_cast<size_t>(job) * p.heads + h) * p.d + c] = left + later[own];
    left = part == 0 ? later[own] : 0.0f;
  }
#pragma unroll
  for (int j = kHalf - 1; j >= 0; --j) {
    if (j < mine) ks[(t0 + j) * kEndRows + own] = CHANNEL ? x[j] * expf(left) : linear_silu(x[j]) * power[count - 1 - (t0 + j)];
    if (CHANNEL) left += y[j];
  }
  {
    // values: four neighbours a thread
    const float* v = p.proj + p.v_off + static_cast<size_t>(h) * p.dv + column0;
#pragma unroll 8
    for (int i = tid; i < count * (kEndColumns / 4); i += kEndThreads) {
      const int s = i / (kEndColumns / 4), e = i % (kEndColumns / 4) * 4;
      float4 z = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      if (column0 + e < p.dv) z = *reinterpret_cast<const float4*>(v + static_cast<size_t>(first + s) * p.proj_width + e);
      if (!CHANNEL) z = make_float4(linear_silu(z.x), linear_silu(z.y), linear_silu(z.z), linear_silu(z.w));
      *reinterpret_cast<float4*>(vs + s * kEndColumns + e) = z;
    }
  }
  __syncthreads();
  const int rows = (tid >> 4) * 8, columns = (tid & 15) * 4;   // rows .. + 7; columns + 64 j
  float acc[8][8];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = 0.0f;
#pragma unroll 2
  for (int s = 0; s < count; ++s) {
    const float4 lo = *reinterpret_cast<const float4*>(ks + s * kEndRows + rows), hi = *reinterpret_cast<const float4*>(ks + s * kEndRows + rows + 4);
    const float a[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const float4 v = *reinterpret_cast<const float4*>(vs + s * kEndColumns + columns + 64 * j);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        acc[i][4 * j] = fmaf(a[i], v.x, acc[i][4 * j]);
        acc[i][4 * j + 1] = fmaf(a[i], v.y, acc[i][4 * j + 1]);
        acc[i][4 * j + 2] = fmaf(a[i], v.z, acc[i][4 * j + 2]);
        acc[i][4 * j + 3] = fmaf(a[i], v.w, acc[i][4 * j + 3]);
      }
    }
  }
  float* out = p.chunk_state + ((static_cast<size_t>(job) * p.heads + h) * p.d + row0 + rows) * p.dv + column0 + columns;
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j)
      if (row0 + rows + i < p.d && column0 + columns + 64 * j < p.dv)
        *reinterpret_cast<float4*>(out + static_cast<size_t>(i) * p.dv + 64 * j) =
            make_float4(acc[i][4 * j], acc[i][4 * j + 1], acc[i][4 * j + 2], acc[i][4 * j + 3]);
}

// ---------------------------------------------------------------------------------------
// The outputs of a (chunk, head) for COLUMNS values, a thread per value column of the tile (8 x 8 outputs each).  q and
// k lie transposed in shared memory, [channel][token]; A goes beside them, [s][t]; then one product runs over the d rows
// of the state and the chunk's values, staged sixteen rows at a time where the keys were, the next rows in registers
// while these are used.
// ---------------------------------------------------------------------------------------
constexpr int kStageRows = 16;
constexpr int kSixteen = 16, kSixteens = kLinearChunk / kSixteen;

template <int COLUMNS>
static inline int linear_outputs_bytes(int d) {
  const int keys = d * kLinearPitch, ring = 2 * kStageRows * COLUMNS;
  return (d * kLinearPitch + (keys > ring ? keys : ring) + kLinearChunk * kLinearPitch + 2 * kSixteens * d + kLinearChunk + 1) * 4;
}

template <bool CHANNEL, int COLUMNS>
__global__ void __launch_bounds__(COLUMNS, 2)
linear_outputs_kernel(const LinearArgs p) {
  extern __shared__ __align__(16) float outputs_shared[];
  const int keys_floats = max(p.d * kLinearPitch, 2 * kStageRows * COLUMNS);
  float* qt = outputs_shared;                               // [d][kLinearPitch]
  float* kt = qt + p.d * kLinearPitch;                      // [d][kLinearPitch], then two stages [kStageRows][COLUMNS]
  float* at = kt + keys_floats;                             // [s][kLinearPitch]
  float* middle = at + kLinearChunk * kLinearPitch;         // CHANNEL: [d] B_m; or [sixteen][d] what each decays by, and 1 over it
  float* power = middle + 2 * kSixteens * p.d;              // otherwise: a^0 .. a^64
  pdl_launch_dependents();
  const int tid = threadIdx.x, h = blockIdx.y, job = blockIdx.z;
  const int column0 = blockIdx.x * COLUMNS;
  const int2 chunk = linear_chunk_of(p.entry_starts, p.num_entries, job);
  const int first = chunk.x, count = chunk.y;
  if (count == 0) return;
  pdl_wait();
  constexpr int kThreads = COLUMNS, kGroups = 2, kAcross = COLUMNS / 8;   // threads a row of tiles takes
  const int group_t = tid / kAcross * 8, group_n = tid % kAcross * 4;     // tokens group_t .. + 7; values group_n + COLUMNS / 2 j

  // rows of the long product: the state's, then the values'
  const float* state = p.chunk_state + (static_cast<size_t>(job) * p.heads + h) * p.d * p.dv + column0;
  const float* values = p.proj + p.v_off + static_cast<size_t>(h) * p.dv + column0 + static_cast<size_t>(first) * p.proj_width;
  constexpr int kPieces = kStageRows * COLUMNS / 4 / kThreads;
  const int stages_state = (p.d + kStageRows - 1) / kStageRows, stages = stages_state + (count + kStageRows - 1) / kStageRows;
  float4 ahead[kPieces];
  auto ask = [&](int stage) {
#pragma unroll
    for (int j = 0; j < kPieces; ++j) {
      const int i = tid + j * kThreads, r = i / (COLUMNS / 4), c = i % (COLUMNS / 4) * 4;
      const bool of_state = stage < stages_state;
      const int row = (of_state ? stage : stage - stages_state) * kStageRows + r;
      const bool live = row < (of_state ? p.d : count) && column0 + c < p.dv;
      const float* src = of_state ? state + static_cast<size_t>(row) * p.dv + c : values + static_cast<size_t>(row) * p.proj_width + c;
      ahead[j] = live ? *reinterpret_cast<const float4*>(src) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
  };
  auto put = [&](int stage) {
    float* dst = kt + (stage & 1) * kStageRows * COLUMNS;
    const bool activate = !CHANNEL && stage >= stages_state;
#pragma unroll
    for (int j = 0; j < kPieces; ++j) {
      float4 x = ahead[j];
      if (activate) x = make_float4(linear_silu(x.x), linear_silu(x.y), linear_silu(x.z), linear_silu(x.w));
      *reinterpret_cast<float4*>(dst + (tid + j * kThreads) * 4) = x;
    }
  };

  if (!CHANNEL && tid <= kLinearChunk) {
    // by repeated multiplication, a thread a power
    float w = 1.0f;
    const float a = p.decay[h];
    for (int i = 0; i < tid; ++i) w *= a;
    power[tid] = w;
  }
  // q and k: a channel and half of the chunk's tokens a thread (where there are threads enough), the reference B_m
  // at the first half's end
  constexpr int kHalf = kLinearChunk / 2;
  const int parts = kThreads >= 2 * p.d ? 2 : 1, per = kLinearChunk / parts;
  bool far = false;
  if (CHANNEL) {
    for (int i = tid; i < p.d; i += kThreads) {
      const float* b = p.log_decay + (static_cast<size_t>(first) * p.heads + h) * p.d + i;
      float to_middle = 0.0f, sum = 0.0f;
#pragma unroll 2
      for (int t0 = 0; t0 < kLinearChunk; t0 += kHalf) {
        float z[kHalf];
#pragma unroll
        for (int j = 0; j < kHalf; ++j) z[j] = t0 + j < count ? b[static_cast<size_t>(t0 + j) * p.heads * p.d] : 0.0f;
#pragma unroll
        for (int j = 0; j < kHalf; ++j) sum += z[j];
        if (t0 == 0) to_middle = sum;
      }
      far |= !(sum > -kLinearMostDecay);
      middle[i] = to_middle;
    }
  }
  far = __syncthreads_or(far);   // some channel decays too far for the factors: q and k stay as they are, for now
  for (int i = tid; i < p.d * parts; i += kThreads) {
    const int c = i % p.d, from = i / p.d * per;
    const float* q = p.proj + p.q_off + static_cast<size_t>(h) * p.d + c + static_cast<size_t>(first) * p.proj_width;
    const float* k = p.proj + p.k_off + static_cast<size_t>(h) * p.d + c + static_cast<size_t>(first) * p.proj_width;
    const float* b = CHANNEL ? p.log_decay + (static_cast<size_t>(first) * p.heads + h) * p.d + c : nullptr;
    const float to_middle = CHANNEL ? middle[c] : 0.0f;
    float sum = from ? to_middle : 0.0f;   // (a second half starts where the first one ends)
#pragma unroll 1
    for (int t0 = from; t0 < from + per; t0 += 16) {
      float x[16], y[16], z[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const size_t t = min(t0 + j, count - 1);
        x[j] = q[t * p.proj_width];
        y[j] = k[t * p.proj_width];
        if (CHANNEL) z[j] = b[t * p.heads * p.d];
      }
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        if (CHANNEL) {
          sum += z[j];
          x[j] *= p.q_scale;
          if (!far) {
            x[j] *= expf(sum - to_middle);
            y[j] *= expf(to_middle - sum);
          }
        } else {
          x[j] = linear_silu(x[j]) * p.q_scale;
          y[j] = linear_silu(y[j]);
        }
        if (t0 + j >= count) x[j] = y[j] = 0.0f;
      }
#pragma unroll
      for (int j = 0; j < 16; j += 4) {
        *reinterpret_cast<float4*>(qt + c * kLinearPitch + t0 + j) = make_float4(x[j], x[j + 1], x[j + 2], x[j + 3]);
        *reinterpret_cast<float4*>(kt + c * kLinearPitch + t0 + j) = make_float4(y[j], y[j + 1], y[j + 2], y[j + 3]);
      }
    }
  }
  __syncthreads();
  ask(0);
  if (!CHANNEL || !far) {
    constexpr int kRowsA = kLinearChunk * kLinearChunk / 4 / kThreads;   // tokens x 4 keys a thread: 4 or 8
    const int row = tid / 16 * kRowsA, key = tid % 16 * 4;
    float a[kRowsA][4];
#pragma unroll
    for (int i = 0; i < kRowsA; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) a[i][j] = 0.0f;
#pragma unroll 4
    for (int c = 0; c < p.d; ++c) {
      const float4 k = *reinterpret_cast<const float4*>(kt + c * kLinearPitch + key);
#pragma unroll
      for (int i4 = 0; i4 < kRowsA; i4 += 4) {
        const float4 q = *reinterpret_cast<const float4*>(qt + c * kLinearPitch + row + i4);
        const float x[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          a[i4 + i][0] = fmaf(x[i], k.x, a[i4 + i][0]);
          a[i4 + i][1] = fmaf(x[i], k.y, a[i4 + i][1]);
          a[i4 + i][2] = fmaf(x[i], k.z, a[i4 + i][2]);
          a[i4 + i][3] = fmaf(x[i], k.w, a[i4 + i][3]);
        }
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int s = key + j;
#pragma unroll
      for (int i4 = 0; i4 < kRowsA; i4 += 4) {
        float w[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int t = row + i4 + i;
          w[i] = s > t ? 0.0f : (CHANNEL ? a[i4 + i][j] : a[i4 + i][j] * power[t - s]);   // (what lies ahead may be out of range)
        }
        *reinterpret_cast<float4*>(at + s * kLinearPitch + row + i4) = make_float4(w[0], w[1], w[2], w[3]);
      }
    }
  } else {
    constexpr int kShares = kThreads / kLinearChunk;
    bool deep = false;   // some channel decays too far over sixteen tokens
    for (int i = tid; i < p.d * kSixteens; i += kThreads) {
      const int c = i % p.d, t0 = i / p.d * kSixteen;
      const float* b = p.log_decay + (static_cast<size_t>(first) * p.heads + h) * p.d + c;
      float sum = 0.0f;
#pragma unroll
      for (int j = 0; j < kSixteen; ++j) sum += t0 + j < count ? b[static_cast<size_t>(t0 + j) * p.heads * p.d] : 0.0f;
      deep |= !(sum > -kLinearMostDecay);
    }
    deep = __syncthreads_or(deep);
    if (deep) {
      // within a sixteen: a thread a key token and a part of the channels, its keys decay token by token
      const int s = tid % kLinearChunk, share = tid / kLinearChunk, t0 = s / kSixteen * kSixteen;
      float a[kSixteen];
#pragma unroll
      for (int j = 0; j < kSixteen; ++j) a[j] = 0.0f;
      const float* alpha = p.alpha + (static_cast<size_t>(first) * p.heads + h) * p.d;
      // two channels at a time: sixteen reads in flight bound this
#pragma unroll 1
      for (int c = 2 * share; c < p.d; c += 2 * kShares) {
        float2 decay[kSixteen];
#pragma unroll
        for (int j = 0; j < kSixteen; ++j)
          decay[j] = *reinterpret_cast<const float2*>(alpha + static_cast<size_t>(min(t0 + j, count - 1)) * p.heads * p.d + c);
        float lo = kt[c * kLinearPitch + s], hi = kt[(c + 1) * kLinearPitch + s];
        const float* x = qt + c * kLinearPitch + t0;
#pragma unroll
        for (int j = 0; j < kSixteen; ++j) {
          if (t0 + j > s) lo *= decay[j].x, hi *= decay[j].y;
          if (t0 + j >= s) a[j] = fmaf(x[kLinearPitch + j], hi, fmaf(x[j], lo, a[j]));
        }
      }
      for (int turn = 0; turn < kShares; ++turn) {
        if (share == turn) {
#pragma unroll
          for (int j = 0; j < kSixteen; ++j) at[s * kLinearPitch + t0 + j] = turn == 0 ? a[j] : at[s * kLinearPitch + t0 + j] + a[j];
        }
        __syncthreads();
      }
    }
    // q from its sixteen's start on, k to its sixteen's end, and what a sixteen decays by
    for (int i = tid; i < p.d * kSixteens; i += kThreads) {
      const int c = i % p.d, sixteen = i / p.d, t0 = sixteen * kSixteen;
      const float* b = p.log_decay + (static_cast<size_t>(first) * p.heads + h) * p.d + c;
      float z[kSixteen], sum = 0.0f, rest = 0.0f;
#pragma unroll
      for (int j = 0; j < kSixteen; ++j) z[j] = t0 + j < count ? b[static_cast<size_t>(t0 + j) * p.heads * p.d] : 0.0f;
#pragma unroll
      for (int j = 0; j < kSixteen; ++j) qt[c * kLinearPitch + t0 + j] *= expf(sum += z[j]);
#pragma unroll
      for (int j = kSixteen - 1; j >= 0; --j) {
        kt[c * kLinearPitch + t0 + j] *= expf(rest);
        rest += z[j];
      }
      middle[sixteen * p.d + c] = expf(sum);
      middle[(kSixteens + sixteen) * p.d + c] = expf(-sum);   // (used where it stays in range)
    }
    __syncthreads();
    // between sixteens, and within one where its own decay is a factor: tokens x 4 keys a thread
    constexpr int kRowsA = kLinearChunk * kLinearChunk / 4 / kThreads;   // 4 or 8
    const int row = tid / 16 * kRowsA, key = tid % 16 * 4, to = row / kSixteen, from = key / kSixteen;
    if (from != to || !deep) {
      float a[kRowsA][4];
#pragma unroll
      for (int i = 0; i < kRowsA; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) a[i][j] = 0.0f;
      if (from <= to) {
        // the factor between: of the second and third sixteen where they lie between, 1 over its own within one
        const float* second = middle + (from == to ? kSixteens + to : 1) * p.d;
        const bool by_second = from == to || (from < 1 && to > 1), by_third = from < 2 && to > 2;
#pragma unroll 4
        for (int c = 0; c < p.d; ++c) {
          float4 k = *reinterpret_cast<const float4*>(kt + c * kLinearPitch + key);
          const float m1 = second[c], m2 = middle[2 * p.d + c];
          const float between = (by_second ? m1 : 1.0f) * (by_third ? m2 : 1.0f);
          k = make_float4(k.x * between, k.y * between, k.z * between, k.w * between);
#pragma unroll
          for (int i4 = 0; i4 < kRowsA; i4 += 4) {
            const float4 q = *reinterpret_cast<const float4*>(qt + c * kLinearPitch + row + i4);
            const float x[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              a[i4 + i][0] = fmaf(x[i], k.x, a[i4 + i][0]);
              a[i4 + i][1] = fmaf(x[i], k.y, a[i4 + i][1]);
              a[i4 + i][2] = fmaf(x[i], k.z, a[i4 + i][2]);
              a[i4 + i][3] = fmaf(x[i], k.w, a[i4 + i][3]);
            }
          }
        }
      }
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int i = 0; i < kRowsA; ++i) at[(key + j) * kLinearPitch + row + i] = key + j > row + i ? 0.0f : a[i][j];
    }
  }
  __syncthreads();   // the keys are read out; A is there
  if (CHANNEL) {
    // q against the state at the chunk's start: e^(B_t) q
    for (int c = tid; c < p.d; c += kThreads) {
      if (!far) {
        const float factor = expf(middle[c]);
        for (int t = 0; t < kLinearChunk; t += 4) {
          float4* x = reinterpret_cast<float4*>(qt + c * kLinearPitch + t);
          *x = make_float4(x->x * factor, x->y * factor, x->z * factor, x->w * factor);
        }
      } else {
        float before = 1.0f;   // what the sixteens before decay by
        for (int t0 = 0; t0 < kLinearChunk; t0 += kSixteen) {
          for (int t = t0; t < t0 + kSixteen; t += 4) {
            float4* x = reinterpret_cast<float4*>(qt + c * kLinearPitch + t);
            *x = make_float4(x->x * before, x->y * before, x->z * before, x->w * before);
          }
          before *= middle[t0 / kSixteen * p.d + c];
        }
      }
    }
  }
  float acc[8][4 * kGroups];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4 * kGroups; ++j) acc[i][j] = 0.0f;
  put(0);
  for (int stage = 0; stage < stages; ++stage) {
    if (stage + 1 < stages) ask(stage + 1);
    __syncthreads();   // this stage is there (and, before the first, e^(B_t) q); the one before is read out
    if (!CHANNEL && stage == stages_state) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float w = power[group_t + i + 1];
#pragma unroll
        for (int j = 0; j < 4 * kGroups; ++j) acc[i][j] *= w;
      }
    }
    const bool of_state = stage < stages_state;
    const int row0 = (of_state ? stage : stage - stages_state) * kStageRows;
    const float* x_rows = (of_state ? qt : at) + row0 * kLinearPitch + group_t;
    const float* y_rows = kt + (stage & 1) * kStageRows * COLUMNS + group_n;
    const int rows = min(kStageRows, (of_state ? p.d : count) - row0);
    // (of the chunk's values: those of the tokens before this thread's eight, whole, then its eight's own: a token takes no
    // part of a value behind it, whatever that holds)
    const int whole = of_state ? rows : min(max(group_t - row0, 0), rows);
#pragma unroll 2
    for (int r = 0; r < whole; ++r) {
      const float4 lo = *reinterpret_cast<const float4*>(x_rows + r * kLinearPitch), hi = *reinterpret_cast<const float4*>(x_rows + r * kLinearPitch + 4);
      const float x[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
      for (int j = 0; j < kGroups; ++j) {
        const float4 y = *reinterpret_cast<const float4*>(y_rows + r * COLUMNS + COLUMNS / 2 * j);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          acc[i][4 * j] = fmaf(x[i], y.x, acc[i][4 * j]);
          acc[i][4 * j + 1] = fmaf(x[i], y.y, acc[i][4 * j + 1]);
          acc[i][4 * j + 2] = fmaf(x[i], y.z, acc[i][4 * j + 2]);
          acc[i][4 * j + 3] = fmaf(x[i], y.w, acc[i][4 * j + 3]);
        }
      }
    }
    if (!of_state && group_t >= row0 && group_t < row0 + rows) {
      const int own = min(8, row0 + rows - group_t);
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        if (e >= own) break;
        const float* at_x = x_rows + (group_t - row0 + e) * kLinearPitch;
        const float4 lo = *reinterpret_cast<const float4*>(at_x), hi = *reinterpret_cast<const float4*>(at_x + 4);
        const float x[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
        for (int j = 0; j < kGroups; ++j) {
          const float4 y = *reinterpret_cast<const float4*>(y_rows + (group_t - row0 + e) * COLUMNS + COLUMNS / 2 * j);
#pragma unroll
          for (int i = e; i < 8; ++i) {
            acc[i][4 * j] = fmaf(x[i], y.x, acc[i][4 * j]);
            acc[i][4 * j + 1] = fmaf(x[i], y.y, acc[i][4 * j + 1]);
            acc[i][4 * j + 2] = fmaf(x[i], y.z, acc[i][4 * j + 2]);
            acc[i][4 * j + 3] = fmaf(x[i], y.w, acc[i][4 * j + 3]);
          }
        }
      }
    }
    if (stage + 1 < stages) put(stage + 1);   // (the half read in the pass before; every thread is past it)
  }
  float* out = p.out + (static_cast<size_t>(first + group_t) * p.heads + h) * p.dv + column0 + group_n;
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < kGroups; ++j)
      if (group_t + i < count && column0 + group_n + COLUMNS / 2 * j < p.dv)
        *reinterpret_cast<float4*>(out + static_cast<size_t>(i) * p.heads * p.dv + COLUMNS / 2 * j) =
            make_float4(acc[i][4 * j], acc[i][4 * j + 1], acc[i][4 * j + 2], acc[i][4 * j + 3]);
}

template <bool CHANNEL>
static int launch_linear_ends(const LinearArgs& p, int jobs, cudaStream_t s) {
  static SharedMemoryOptIn opt_in;
  const int opted = opt_in.ask(reinterpret_cast<const void*>(linear_ends_kernel<CHANNEL>), kEndBytes);
  if (opted) return opted;
  const dim3 grid((p.d + kEndRows - 1) / kEndRows * ((p.dv + kEndColumns - 1) / kEndColumns), p.heads, jobs);
  return vipera_launch(linear_ends_kernel<CHANNEL>, grid, dim3(kEndThreads), kEndBytes, s, p);
}

template <bool CHANNEL, int COLUMNS>
static int launch_linear_outputs_as(const LinearArgs& p, int jobs, cudaStream_t s) {
  static SharedMemoryOptIn opt_in;
  const int opted = opt_in.ask(reinterpret_cast<const void*>(linear_outputs_kernel<CHANNEL, COLUMNS>), linear_outputs_bytes<COLUMNS>(256));
  if (opted) return opted;
  return vipera_launch(linear_outputs_kernel<CHANNEL, COLUMNS>, dim3((p.dv + COLUMNS - 1) / COLUMNS, p.heads, jobs), dim3(COLUMNS),
                       linear_outputs_bytes<COLUMNS>(p.d), s, p);
}

// Values of up to 128 numbers fill half of the wider tile only.
template <bool CHANNEL>
static int launch_linear_outputs(const LinearArgs& p, int jobs, cudaStream_t s) {
  return p.dv <= 128 ? launch_linear_outputs_as<CHANNEL, 128>(p, jobs, s) : launch_linear_outputs_as<CHANNEL, 256>(p, jobs, s);
}
