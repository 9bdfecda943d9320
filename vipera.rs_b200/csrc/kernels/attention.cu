// Causal grouped-query attention over the paged cache, for any mix of prompt portions and
// single decode tokens, with 32-bit scores, softmax and accumulation.
//
// Definition (crates/vipera-backend-cpu/src/model.rs:1804-1859): query head h reads KV head
// h / group; s_j = (q . k_j) * scale; a query at position p sees keys 0..p (with a window w,
// keys p-w+1..p); weights exp(s_j - max) over their sum; output = weighted sum of v_j.
// Traversal: a block folds the keys 64 at a time with a running (max, sum, output) per row, the online
// form of the reference's chunk fold (model.rs:2752-2857) and of its device kernels' partials
// (crates/vipera-backend-gpu/src/layer.cu:307-467); few tokens split their keys between the blocks of a
// cluster, more share what they read in tiles, and where few keys are visible a warp folds those of a (token, head) (see the three kernels).
// Keys are found through the block table: position j lives in page table[j / page], slot
// j % page (model.rs:1507-1542).
//
// Three options beyond that definition, each a parameter: values of another size than keys
// (`value_dim`); with a window, the first `keep_first` keys of a request stay visible to every
// later query, at their true positions; and a sink, an extra key of score 0 without a value,
// which adds exp(0 - max) to the softmax's denominator (p_j = e^{s_j} / (1 + sum e^{s_j})).
// Instead of a window the mask may be one of chunks (`chunk`): position i sees j <= i with
// floor(i / chunk) = floor(j / chunk).  `out_scale` multiplies the output.  The sink's score may be
// learned, one per query head (`sink_values`: exp(sink_h - max) joins the denominator, unscaled), and
// the output may be gated: out[t, h, e] *= sigmoid(gate[t * gate_stride + h * value_dim + e]), the gate
// a 32-bit pre-activation (`gate_per_head`: one per head, gate[t * gate_stride + h]).
//
// This is the attention of the 32-bit path and of bfloat16 head sizes without tensor-core kernels.  It takes
// every head size up to 256 (keys and values each; rows that are not whole 16-byte pieces are read value by
// value), any number of heads and groups, any page size.
#include <algorithm>

#include "simt.cuh"

constexpr int kMaxHeadDim = 256;
constexpr int kTileKeys = 64;       // keys a block holds at a time
constexpr int kAttentionThreads = 128;

struct AttentionParams {
  const void* q;
  void* out;
  const void* k_pool;
  const void* v_pool;
  const int* token_seq;
  const int* positions;
  const int* block_table;
  int table_width, page_size, num_tokens, num_heads, num_kv_heads, head_dim, value_dim;
  float scale;
  int window, keep_first, sink, chunk;
  float out_scale;
  const float* sink_values;
  const float* gate;
  long long gate_stride;
  int gate_per_head;
  int singles;   // tokens that stand alone among their neighbours have a launch of their own
};

// What a query at `position` sees: keys 0 .. kept - 1 and first .. position.
__device__ __forceinline__ void visible_keys(const AttentionParams& p, int position, int* kept, int* first) {
  // a mask of chunks: a query sees the keys of its own chunk of `chunk` positions, counted from 0
  *first = p.chunk > 0 ? position / p.chunk * p.chunk : (p.window > 0 ? max(0, position - p.window + 1) : 0);
  *kept = p.window > 0 ? min(p.keep_first, *first) : 0;
}

// Rows of a pool (row r's place in place[r], -1: zeros) into shared memory as floats, `pitch` apart.  VEC: rows of
// whole 16-byte pieces on 16-byte boundaries (32-bit ones are copied asynchronously: the caller waits).
template <typename T, bool VEC, int THREADS = kAttentionThreads>
__device__ __forceinline__ void stage_keys(float* dst, int pitch, const T* __restrict__ pool, size_t row_stride, int size,
                                           const int* place, int rows) {
  constexpr int kPiece = VEC ? 16 / static_cast<int>(sizeof(T)) : 1;
  const int pieces = size / kPiece;
#pragma unroll 4
  for (int i = threadIdx.x; i < rows * pieces; i += THREADS) {
    const int r = i / pieces, c = (i - r * pieces) * kPiece;
    const int at = place[r];
    const T* src = pool + (at >= 0 ? static_cast<size_t>(at) * row_stride + c : 0);
    float* to = dst + r * pitch + c;
    if constexpr (!VEC) {
      *to = at >= 0 ? to_float<T>(*src) : 0.0f;
    } else if constexpr (sizeof(T) == 4) {
      copy_16(shared_address(to), src, at >= 0);
    } else {
      const uint4 raw = at >= 0 ? *reinterpret_cast<const uint4*>(src) : make_uint4(0u, 0u, 0u, 0u);
      const __nv_bfloat162* pairs = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
      for (int e = 0; e < 4; ++e) *reinterpret_cast<float2*>(to + 2 * e) = __bfloat1622float2(pairs[e]);
    }
  }
}

// The output gate's factor for (token, head, value e).
__device__ __forceinline__ float gate_factor(const AttentionParams& p, int t, int h, int e) {
  if (!p.gate) return 1.0f;
  const float* row = p.gate + static_cast<size_t>(t) * p.gate_stride;
  return 1.0f / (1.0f + expf(-(p.gate_per_head ? row[h] : row[static_cast<size_t>(h) * p.value_dim + e])));
}
// Folds the sink (a key of score 0, or of a learned one, whose value is zero) into (max, sum); returns the factor
// of the accumulated output, 1 / sum and out_scale included.
__device__ __forceinline__ float ending_factor(const AttentionParams& p, int h, float row_max, float row_sum) {
  if (p.sink || p.sink_values) {
    const float sink_score = p.sink_values ? p.sink_values[h] : 0.0f;
    const float top = fmaxf(row_max, sink_score);
    const float alpha = row_max == top ? 1.0f : expf(row_max - top);
    return alpha * (p.out_scale / (row_sum * alpha + expf(sink_score - top)));
  }
  return p.out_scale / row_sum;
}

// ---------------------------------------------------------------------------------------
// Steps of few tokens: a cluster of eight blocks per (token, up to eight query heads of one KV head), an eighth of
// the visible keys each, joined through distributed shared memory.  A tile of 64 keys and their values is
// staged; a thread scores one key against four heads (packed multiply-adds), a warp takes the softmax of two heads,
// a thread then owns value columns of all eight heads.  DP: head and value sizes up to 64, 128 or 256.
// What bounds it is the trips to memory of a block's few tiles, so the keys of a (token, KV head) are read once
// for its heads and by eight multiprocessors.  8 tokens, 12 heads of 128 on 2, 1,000 keys, 32-bit: 23 us (a warp
// per (token, head): 1,117 us).
// ---------------------------------------------------------------------------------------
constexpr int kSplits = 8, kRows = 8, kScorePitch = 12;

// The `index`-th token that stands alone (another request's before it and behind it), for the whole block; -1: none.
__device__ __forceinline__ int single_token(const int* __restrict__ seq, int tokens, int index) {
  __shared__ int counts[kAttentionThreads / 32], found;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) found = -1;
  int before = 0;
  for (int base = 0; base < tokens; base += kAttentionThreads) {
    const int t = base + threadIdx.x;
    const bool alone = t < tokens && (t == 0 || seq[t - 1] != seq[t]) && (t + 1 == tokens || seq[t + 1] != seq[t]);
    const unsigned votes = __ballot_sync(0xffffffffu, alone);
    __syncthreads();   // the counts before are read
    if (lane == 0) counts[warp] = __popc(votes);
    __syncthreads();
    int own = before + __popc(votes & ((1u << lane) - 1u));
    for (int w = 0; w < kAttentionThreads / 32; ++w) {
      if (w < warp) own += counts[w];
      before += counts[w];
    }
    if (alone && own == index) found = t;
    if (before > index) break;
  }
  __syncthreads();
  return found;
}

template <int DP>
struct SplitShared {
  float q[kRows][DP];
  float k[kTileKeys][DP + 4];
  float v[kTileKeys][DP];
  float score[kTileKeys][kScorePitch];   // [key][head]
  float out[kRows][DP];
  float top[kRows], sum[kRows], alpha[kRows];
  int place[kTileKeys];
};

template <typename T, int DP, bool VEC>
__global__ void __launch_bounds__(kAttentionThreads)
attention_split_kernel(const AttentionParams p) {
  extern __shared__ __align__(16) unsigned char split_raw[];
  SplitShared<DP>& s = *reinterpret_cast<SplitShared<DP>*>(split_raw);
  pdl_launch_dependents();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int split = blockIdx.x;
  const int group = p.num_heads / p.num_kv_heads, parts = (group + kRows - 1) / kRows;
  const int kv_head = blockIdx.y / parts, h0 = kv_head * group + (blockIdx.y % parts) * kRows;
  const int heads = min(kRows, (kv_head + 1) * group - h0);
  const int d = p.head_dim, dv = p.value_dim;
  // columns that no row of a pool fills are read with the others: zeros
  for (int i = tid; i < kTileKeys * (DP + 4 - d); i += kAttentionThreads) s.k[i / (DP + 4 - d)][d + i % (DP + 4 - d)] = 0.0f;
  pdl_wait();
  // a token a cluster; or the tokens that stand alone, as many clusters as there are requests (nearly always one round)
  for (int turn = blockIdx.z;; turn += gridDim.z) {
  const int t = p.singles ? single_token(p.token_seq, p.num_tokens, turn) : turn;
  if (t < 0 || t >= p.num_tokens) return;   // (the same for every block of the cluster)
  const int position = p.positions[t];
  const int* table = p.block_table + static_cast<size_t>(p.token_seq[t]) * p.table_width;
  int kept, first;
  visible_keys(p, position, &kept, &first);
  const int keys = kept + max(position - first + 1, 0);
  const int share = (keys + kSplits - 1) / kSplits;
  const int begin = min(split * share, keys), end = min(begin + share, keys);
  auto look_up = [&](int base) {   // where the key of this thread lies in the tile from `base` on
    const int index = min(base + (tid & (kTileKeys - 1)), end - 1);
    const int key = index < kept ? index : first + index - kept;
    return table[key / p.page_size] * p.page_size + key % p.page_size;
  };
  int ahead = begin < end ? look_up(begin) : 0;
  for (int i = tid; i < kRows * DP; i += kAttentionThreads) {
    const int r = i / DP, c = i % DP;
    s.q[r][c] = r < heads && c < d ? to_float<T>(static_cast<const T*>(p.q)[(static_cast<size_t>(t) * p.num_heads + h0 + r) * d + c]) : 0.0f;
  }
  if (tid < kRows) {
    s.top[tid] = -INFINITY;
    s.sum[tid] = 0.0f;
  }
  constexpr int kColumns = (DP + kAttentionThreads - 1) / kAttentionThreads;
  float acc[kRows][kColumns];
#pragma unroll
  for (int r = 0; r < kRows; ++r)
#pragma unroll
    for (int j = 0; j < kColumns; ++j) acc[r][j] = 0.0f;

  for (int base = begin; base < end; base += kTileKeys) {
    const int count = min(kTileKeys, end - base);
    __syncthreads();   // the tile before is read out
    if (tid < kTileKeys) s.place[tid] = ahead;
    __syncthreads();
    stage_keys<T, VEC>(&s.k[0][0], DP + 4, static_cast<const T*>(p.k_pool) + static_cast<size_t>(kv_head) * d,
                       static_cast<size_t>(p.num_kv_heads) * d, d, s.place, count);
    stage_keys<T, VEC>(&s.v[0][0], DP, static_cast<const T*>(p.v_pool) + static_cast<size_t>(kv_head) * dv,
                       static_cast<size_t>(p.num_kv_heads) * dv, dv, s.place, count);
    copy_commit();
    if (base + kTileKeys < end) ahead = look_up(base + kTileKeys);
    copy_wait<0>();
    __syncthreads();
    {
      const int key = tid & (kTileKeys - 1), r0 = (tid / kTileKeys) * 4;
      unsigned long long dot[4] = {0ull, 0ull, 0ull, 0ull};
      if (key < count) {
#pragma unroll 8
        for (int c = 0; c < DP; c += 4) {
          const ulonglong2 kk = *reinterpret_cast<const ulonglong2*>(&s.k[key][c]);
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            const ulonglong2 qq = *reinterpret_cast<const ulonglong2*>(&s.q[r0 + r][c]);
            fma_pair(dot[r], qq.x, kk.x);
            fma_pair(dot[r], qq.y, kk.y);
          }
        }
      }
#pragma unroll
      for (int r = 0; r < 4; ++r) s.score[key][r0 + r] = key < count ? sum_of_pair(dot[r]) * p.scale : -INFINITY;
    }
    __syncthreads();
#pragma unroll
    for (int own = 0; own < 2; ++own) {
      const int r = 2 * warp + own;
      const float a = s.score[lane][r], b = s.score[lane + 32][r];
      const float before = s.top[r], top = fmaxf(before, warp_max(fmaxf(a, b)));
      const float shift = top == -INFINITY ? 0.0f : top;
      const float wa = lane < count ? expf(a - shift) : 0.0f, wb = lane + 32 < count ? expf(b - shift) : 0.0f;
      s.score[lane][r] = wa;
      s.score[lane + 32][r] = wb;
      const float sum = warp_sum(wa + wb);
      if (lane == 0) {
        const float alpha = before == top ? 1.0f : expf(before - top);
        s.top[r] = top;
        s.alpha[r] = alpha;
        s.sum[r] = s.sum[r] * alpha + sum;
      }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kRows; ++r)
#pragma unroll
      for (int j = 0; j < kColumns; ++j) acc[r][j] *= s.alpha[r];
#pragma unroll
    for (int j = 0; j < kColumns; ++j) {
      const int c = tid + j * kAttentionThreads;
      if (c >= dv) continue;
#pragma unroll 8
      for (int key = 0; key < count; ++key) {
        const float v = s.v[key][c];
        const float4 lo = *reinterpret_cast<const float4*>(&s.score[key][0]), hi = *reinterpret_cast<const float4*>(&s.score[key][4]);
        acc[0][j] = fmaf(lo.x, v, acc[0][j]);
        acc[1][j] = fmaf(lo.y, v, acc[1][j]);
        acc[2][j] = fmaf(lo.z, v, acc[2][j]);
        acc[3][j] = fmaf(lo.w, v, acc[3][j]);
        acc[4][j] = fmaf(hi.x, v, acc[4][j]);
        acc[5][j] = fmaf(hi.y, v, acc[5][j]);
        acc[6][j] = fmaf(hi.z, v, acc[6][j]);
        acc[7][j] = fmaf(hi.w, v, acc[7][j]);
      }
    }
  }
#pragma unroll
  for (int j = 0; j < kColumns; ++j) {
    const int c = tid + j * kAttentionThreads;
    if (c < DP) {
#pragma unroll
      for (int r = 0; r < kRows; ++r) s.out[r][c] = acc[r][j];
    }
  }
  cluster_sync();
  // block r of the cluster joins head r
  if (split < heads) {
    const int h = h0 + split;
    float tops[kSplits], sums[kSplits], top = -INFINITY;
#pragma unroll
    for (int b = 0; b < kSplits; ++b) {
      tops[b] = remote_float(shared_address(&s.top[split]), b);
      sums[b] = remote_float(shared_address(&s.sum[split]), b);
      top = fmaxf(top, tops[b]);
    }
    float sum = 0.0f;
#pragma unroll
    for (int b = 0; b < kSplits; ++b) {
      tops[b] = tops[b] == top ? 1.0f : expf(tops[b] - top);   // (0 where a block saw no key)
      sum += sums[b] * tops[b];
    }
    const float factor = ending_factor(p, h, top, sum);
    for (int c = tid; c < dv; c += kAttentionThreads) {
      float part[kSplits], value = 0.0f;
#pragma unroll
      for (int b = 0; b < kSplits; ++b) part[b] = remote_float(shared_address(&s.out[split][c]), b);
#pragma unroll
      for (int b = 0; b < kSplits; ++b) value = fmaf(part[b], tops[b], value);
      static_cast<T*>(p.out)[(static_cast<size_t>(t) * p.num_heads + h) * dv + c] = from_float<T>(value * factor * gate_factor(p, t, h, c));
    }
  }
  cluster_sync();   // no block goes on while another reads its part
  }
}

// ---------------------------------------------------------------------------------------
// Steps of more tokens: a block takes 64 neighbouring tokens and one head and walks the keys 64 at a time.  A
// thread owns 4 rows x 4 keys of the scores (packed multiply-adds) and 4 rows x DP / 16 values of the output;
// sixteen lanes share a row, a warp eight rows, so that a row's weights pass through shared memory
// within its warp.  Tokens of several requests in one tile are folded one request after another, the
// others' rows masked.  Bound by the multiply-adds and the reads of shared memory that feed them: 64 x 64 tiles
// read a key 64 times less often than a warp per row.  The longest walk bounds a step of few tiles: blocks of a cluster then
// share a tile's keys (tile_members).  1,024 tokens of three requests (700, 1 and 323, histories 0, 900, 40), 14 heads of 64 on 2,
// 32-bit, with 21 us for the one alone: 95 us by two blocks, 128 by one (four warps of twice the rows: 154; a warp per (token,
// head): 1,146 us).  (The next keys asked for ahead, with a place for the weights beside them: no faster.)
// ---------------------------------------------------------------------------------------
constexpr int kTileRows = 64, kTileThreads = 256, kOwn = kTileRows * 16 / kTileThreads;   // (sixteen lanes a row; kOwn rows a thread)

template <int DP>
struct TileShared {
  float q[kTileRows][DP + 4];
  float k[kTileKeys][DP + 4];   // then the tile's weights, [row][kTileKeys + 4]
  float v[kTileKeys][DP];
  int place[kTileKeys];
  int seq[kTileRows], last[kTileRows], first[kTileRows], kept[kTileRows];
  float top[kTileRows], sum[kTileRows];   // JOIN: a block's, for the others of its cluster (its outputs take the values' place)
};
constexpr int kMostMembers = 4;

// JOIN: the `members` blocks of a cluster share a tile's keys, each every members-th 64 of them, and join their outputs.
template <typename T, int DP, bool VEC, bool JOIN>
__global__ void __launch_bounds__(kTileThreads)
attention_tile_kernel(const AttentionParams p, int members) {
  extern __shared__ __align__(16) unsigned char tile_raw[];
  TileShared<DP>& s = *reinterpret_cast<TileShared<DP>*>(tile_raw);
  constexpr int kWeightPitch = kTileKeys + 4;
  static_assert(kTileRows * kWeightPitch <= kTileKeys * (DP + 4), "the weights take the keys' place");
  float* weights = &s.k[0][0];
  pdl_launch_dependents();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int h = JOIN ? blockIdx.x / members : blockIdx.x, member = JOIN ? blockIdx.x % members : 0, stride = JOIN ? members * kTileKeys : kTileKeys;
  const int kv_head = h / (p.num_heads / p.num_kv_heads);
  const int t0 = (gridDim.y - 1 - blockIdx.y) * kTileRows;   // the longest histories of a prompt first
  const int rows = min(kTileRows, p.num_tokens - t0);
  const int d = p.head_dim, dv = p.value_dim;
  pdl_wait();
  if (tid < kTileRows) {
    const bool valid = tid < rows;
    s.seq[tid] = valid ? p.token_seq[t0 + tid] : -1;
    s.last[tid] = valid ? p.positions[t0 + tid] : -1;
    s.first[tid] = 0;
    s.kept[tid] = 0;
    if (valid) visible_keys(p, s.last[tid], &s.kept[tid], &s.first[tid]);
  }
#pragma unroll 4
  for (int i = tid; i < kTileRows * d; i += kTileThreads) {
    const int r = i / d, c = i - r * d;
    s.q[r][c] = r < rows ? to_float<T>(static_cast<const T*>(p.q)[(static_cast<size_t>(t0 + r) * p.num_heads + h) * d + c]) : 0.0f;
  }
  if (d < DP) {
    const int spare = DP - d;
    for (int i = tid; i < kTileRows * spare; i += kTileThreads) s.q[i / spare][d + i % spare] = 0.0f;
  }
  if (dv < DP) {
    const int spare = DP - dv;
    for (int i = tid; i < kTileKeys * spare; i += kTileThreads) s.v[i / spare][dv + i % spare] = 0.0f;
  }
  __syncthreads();

  const int row0 = warp * 2 * kOwn + (lane >> 4), column0 = lane & 15;   // rows row0 + 2 i; keys column0 + 16 j; values 4 column0 + 64 j
  constexpr int kGroups = DP / 64;
  float out[kOwn][kGroups][4];
  float row_max[kOwn], row_sum[kOwn];
#pragma unroll
  for (int i = 0; i < kOwn; ++i) {
    row_max[i] = -INFINITY;
    row_sum[i] = 0.0f;
#pragma unroll
    for (int j = 0; j < kGroups; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) out[i][j][e] = 0.0f;
  }

  for (int seg = 0; seg < rows;) {
    // the rows of one request that follow one another, and the keys any of them sees
    const int seq = s.seq[seg];
    int seg_end = seg, low = 0x7fffffff, high = -1, most_kept = 0;
    while (seg_end < rows && s.seq[seg_end] == seq) {
      low = min(low, s.first[seg_end]);
      high = max(high, s.last[seg_end]);
      most_kept = max(most_kept, s.kept[seg_end]);
      ++seg_end;
    }
    if (p.singles && seg_end - seg == 1 && (t0 + seg == 0 || p.token_seq[t0 + seg - 1] != seq) &&
        (t0 + seg_end == p.num_tokens || p.token_seq[t0 + seg_end] != seq)) {
      if (tid == 0) s.last[seg] = -2;   // no row of this launch's
      __syncthreads();
      seg = seg_end;
      continue;
    }
    const int* table = p.block_table + static_cast<size_t>(seq) * p.table_width;
    for (int run = 0; run < 2; ++run) {
      const int run_first = (run == 0 ? 0 : low) + member * kTileKeys, run_end = run == 0 ? most_kept : high + 1;
      auto look_up = [&](int base) {   // where the key of this thread lies in the tile from `base` on, -1: nowhere
        const int key = base + (tid & (kTileKeys - 1));
        if (key >= run_end) return -1;
        const int page = table[key / p.page_size];   // (a page that no row sees may be gone)
        return page >= 0 ? page * p.page_size + key % p.page_size : -1;
      };
      int ahead = run_first < run_end ? look_up(run_first) : -1;
      for (int base = run_first; base < run_end; base += stride) {
        const int count = min(kTileKeys, run_end - base);
        __syncthreads();   // the tile before is read out
        if (tid < kTileKeys) s.place[tid] = ahead;
        if (d < DP) {   // the weights were here
          const int spare = DP - d;
          for (int i = tid; i < kTileKeys * spare; i += kTileThreads) s.k[i / spare][d + i % spare] = 0.0f;
        }
        __syncthreads();
        stage_keys<T, VEC, kTileThreads>(&s.k[0][0], DP + 4, static_cast<const T*>(p.k_pool) + static_cast<size_t>(kv_head) * d,
                           static_cast<size_t>(p.num_kv_heads) * d, d, s.place, kTileKeys);
        copy_commit();
        stage_keys<T, VEC, kTileThreads>(&s.v[0][0], DP, static_cast<const T*>(p.v_pool) + static_cast<size_t>(kv_head) * dv,
                           static_cast<size_t>(p.num_kv_heads) * dv, dv, s.place, kTileKeys);
        copy_commit();
        if (base + stride < run_end) ahead = look_up(base + stride);
        copy_wait<1>();
        __syncthreads();
        unsigned long long dot[kOwn][4];
#pragma unroll
        for (int i = 0; i < kOwn; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) dot[i][j] = 0ull;
#pragma unroll 2
        for (int c = 0; c < DP; c += 4) {
          ulonglong2 kk[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) kk[j] = *reinterpret_cast<const ulonglong2*>(&s.k[column0 + 16 * j][c]);
#pragma unroll
          for (int i = 0; i < kOwn; ++i) {
            const ulonglong2 qq = *reinterpret_cast<const ulonglong2*>(&s.q[row0 + 2 * i][c]);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              fma_pair(dot[i][j], qq.x, kk[j].x);
              fma_pair(dot[i][j], qq.y, kk[j].y);
            }
          }
        }
        copy_wait<0>();
        __syncthreads();   // the keys are read out (the weights take their place), and the values are there
        bool some_hidden = false;
#pragma unroll
        for (int i = 0; i < kOwn; ++i) {
          const int row = row0 + 2 * i;
          const int from = run == 0 ? 0 : s.first[row], to = run == 0 ? s.kept[row] : s.last[row] + 1;
          const bool mine = row >= seg && row < seg_end;
          float score[4];
          bool seen[4];
          float top = row_max[i];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int key = base + column0 + 16 * j;
            seen[j] = mine && key >= from && key < to;
            some_hidden |= !seen[j];
            score[j] = sum_of_pair(dot[i][j]) * p.scale;
            if (seen[j]) top = fmaxf(top, score[j]);
          }
#pragma unroll
          for (int offset = 8; offset > 0; offset >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, offset));
          const float shift = top == -INFINITY ? 0.0f : top;
          float sum = 0.0f;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float w = expf(score[j] - shift);
            if (seen[j]) sum += w;
            weights[row * kWeightPitch + column0 + 16 * j] = seen[j] ? w : -1.0f;   // below 0: not seen at all
          }
#pragma unroll
          for (int offset = 8; offset > 0; offset >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, offset);
          const float alpha = row_max[i] == top ? 1.0f : expf(row_max[i] - top);
          row_max[i] = top;
          row_sum[i] = row_sum[i] * alpha + sum;
#pragma unroll
          for (int j = 0; j < kGroups; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) out[i][j][e] *= alpha;
        }
        const bool edge = __any_sync(0xffffffffu, some_hidden);
        __syncwarp();   // a warp's rows and their weights are its own
        if (!edge) {
#pragma unroll 2
          for (int key = 0; key < kTileKeys; key += 2) {
            float2 w[kOwn];
#pragma unroll
            for (int i = 0; i < kOwn; ++i) w[i] = *reinterpret_cast<const float2*>(weights + (row0 + 2 * i) * kWeightPitch + key);
#pragma unroll
            for (int j = 0; j < kGroups; ++j) {
              const float4 a = *reinterpret_cast<const float4*>(&s.v[key][4 * column0 + 64 * j]);
              const float4 b = *reinterpret_cast<const float4*>(&s.v[key + 1][4 * column0 + 64 * j]);
#pragma unroll
              for (int i = 0; i < kOwn; ++i) {
                out[i][j][0] = fmaf(w[i].y, b.x, fmaf(w[i].x, a.x, out[i][j][0]));
                out[i][j][1] = fmaf(w[i].y, b.y, fmaf(w[i].x, a.y, out[i][j][1]));
                out[i][j][2] = fmaf(w[i].y, b.z, fmaf(w[i].x, a.z, out[i][j][2]));
                out[i][j][3] = fmaf(w[i].y, b.w, fmaf(w[i].x, a.w, out[i][j][3]));
              }
            }
          }
        } else {
          // a value a row does not see is left out, whatever it holds (0 times infinity is not 0)
#pragma unroll 2
          for (int key = 0; key < count; ++key) {
            float w[kOwn];
#pragma unroll
            for (int i = 0; i < kOwn; ++i) w[i] = weights[(row0 + 2 * i) * kWeightPitch + key];
#pragma unroll
            for (int j = 0; j < kGroups; ++j) {
              const float4 a = *reinterpret_cast<const float4*>(&s.v[key][4 * column0 + 64 * j]);
#pragma unroll
              for (int i = 0; i < kOwn; ++i) {
                if (!(w[i] < 0.0f)) {
                  out[i][j][0] = fmaf(w[i], a.x, out[i][j][0]);
                  out[i][j][1] = fmaf(w[i], a.y, out[i][j][1]);
                  out[i][j][2] = fmaf(w[i], a.z, out[i][j][2]);
                  out[i][j][3] = fmaf(w[i], a.w, out[i][j][3]);
                }
              }
            }
          }
        }
      }
    }
    seg = seg_end;
  }
  if constexpr (JOIN) {
    __syncthreads();   // the values are read out
#pragma unroll
    for (int i = 0; i < kOwn; ++i) {
      const int row = row0 + 2 * i;
      if (column0 == 0) s.top[row] = row_max[i], s.sum[row] = row_sum[i];
#pragma unroll
      for (int j = 0; j < kGroups; ++j) *reinterpret_cast<float4*>(&s.v[row][4 * column0 + 64 * j]) = make_float4(out[i][j][0], out[i][j][1], out[i][j][2], out[i][j][3]);
    }
    cluster_sync();
    // an even share of the rows a block, sixteen lanes a row
    const int share = kTileRows / members;
    for (int row = member * share + (tid >> 4); row < min(rows, (member + 1) * share); row += kTileThreads / 16) {
      if (s.last[row] == -2) continue;
      const int t = t0 + row;
      float weight[kMostMembers], sums[kMostMembers], most = -INFINITY, sum = 0.0f;
#pragma unroll
      for (int b = 0; b < kMostMembers; ++b) {
        weight[b] = b < members ? remote_float(shared_address(&s.top[row]), b) : -INFINITY;
        sums[b] = b < members ? remote_float(shared_address(&s.sum[row]), b) : 0.0f;
      }
#pragma unroll
      for (int b = 0; b < kMostMembers; ++b) most = fmaxf(most, weight[b]);
#pragma unroll
      for (int b = 0; b < kMostMembers; ++b) {
        weight[b] = weight[b] == -INFINITY ? 0.0f : expf(weight[b] - most);
        sum = fmaf(sums[b], weight[b], sum);
      }
      const float factor = ending_factor(p, h, most, sum);
      T* out_row = static_cast<T*>(p.out) + (static_cast<size_t>(t) * p.num_heads + h) * dv;
#pragma unroll
      for (int e = 0; e < 4 * kGroups; ++e) {
        const int c = column0 + 16 * e;
        float part[kMostMembers], value = 0.0f;
#pragma unroll
        for (int b = 0; b < kMostMembers; ++b) part[b] = b < members ? remote_float(shared_address(&s.v[row][c]), b) : 0.0f;
#pragma unroll
        for (int b = 0; b < kMostMembers; ++b)
          if (b < members) value = fmaf(part[b], weight[b], value);
        if (c < dv) out_row[c] = from_float<T>(value * factor * gate_factor(p, t, h, c));
      }
    }
    cluster_sync();   // no block leaves while another reads its part
  } else {
#pragma unroll
    for (int i = 0; i < kOwn; ++i) {
      const int row = row0 + 2 * i;
      if (row >= rows || s.last[row] == -2) continue;
      const int t = t0 + row;
      const float factor = ending_factor(p, h, row_max[i], row_sum[i]);
      T* out_row = static_cast<T*>(p.out) + (static_cast<size_t>(t) * p.num_heads + h) * dv;
#pragma unroll
      for (int j = 0; j < kGroups; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int c = 4 * column0 + 64 * j + e;
          if (c < dv) out_row[c] = from_float<T>(out[i][j][e] * factor * gate_factor(p, t, h, c));
        }
    }
  }
}

// ---------------------------------------------------------------------------------------
// Few visible keys: a warp per (token, head) folds them 32 at a time, a lane's score from its own key's row, the weights
// handed round by shuffles.  Nothing is staged or shared, so many warps fit a multiprocessor; what bounds it is a warp's
// chain of reads, some 16 us per 32 keys.
// ---------------------------------------------------------------------------------------
constexpr int kWarpsPerBlock = 4;

// Dot product of `n` floats in shared memory with a row of T in memory.
template <typename T, bool VEC>
__device__ __forceinline__ float dot_row(const float* q, const T* __restrict__ row, int n) {
  float sum = 0.0f;
  if constexpr (!VEC) {
    for (int i = 0; i < n; ++i) sum = fmaf(q[i], to_float<T>(row[i]), sum);
  } else if constexpr (sizeof(T) == 4) {
#pragma unroll 4
    for (int i = 0; i < n; i += 4) {
      const float4 f = *reinterpret_cast<const float4*>(row + i);
      sum = fmaf(q[i], f.x, sum);
      sum = fmaf(q[i + 1], f.y, sum);
      sum = fmaf(q[i + 2], f.z, sum);
      sum = fmaf(q[i + 3], f.w, sum);
    }
  } else {
#pragma unroll 4
    for (int i = 0; i < n; i += 8) {
      const uint4 raw = *reinterpret_cast<const uint4*>(row + i);
      const __nv_bfloat162* pairs = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 f = __bfloat1622float2(pairs[e]);
        sum = fmaf(q[i + 2 * e], f.x, sum);
        sum = fmaf(q[i + 2 * e + 1], f.y, sum);
      }
    }
  }
  return sum;
}

template <typename T, bool VEC>
__global__ void __launch_bounds__(kWarpsPerBlock * 32)
attention_warp_kernel(const AttentionParams p) {
  __shared__ float q_shared[kWarpsPerBlock][kMaxHeadDim];
  pdl_launch_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int t = blockIdx.x, h = blockIdx.y * kWarpsPerBlock + warp;
  if (h >= p.num_heads) return;
  const int kv_head = h / (p.num_heads / p.num_kv_heads), d = p.head_dim, dv = p.value_dim;
  pdl_wait();
  const int position = p.positions[t];
  const int* table = p.block_table + static_cast<size_t>(p.token_seq[t]) * p.table_width;
  int kept, first;
  visible_keys(p, position, &kept, &first);
  const T* q_row = static_cast<const T*>(p.q) + (static_cast<size_t>(t) * p.num_heads + h) * d;
  float* qs = q_shared[warp];
  for (int i = lane; i < d; i += 32) qs[i] = to_float<T>(q_row[i]);
  __syncwarp();
  const T* k_head = static_cast<const T*>(p.k_pool) + static_cast<size_t>(kv_head) * d;
  const T* v_head = static_cast<const T*>(p.v_pool) + static_cast<size_t>(kv_head) * dv;
  const size_t k_stride = static_cast<size_t>(p.num_kv_heads) * d, v_stride = static_cast<size_t>(p.num_kv_heads) * dv;

  constexpr int kColumns = kMaxHeadDim / 32;
  float acc[kColumns];
#pragma unroll
  for (int i = 0; i < kColumns; ++i) acc[i] = 0.0f;
  float row_max = -INFINITY, row_sum = 0.0f;
  // two runs of keys: the kept first ones that the window has left behind, then the window
  for (int run = 0; run < 2; ++run) {
    const int begin = run == 0 ? 0 : first, end = run == 0 ? kept : position + 1;
    for (int base = begin; base < end; base += 32) {
      const int count = min(32, end - base);
      int place = 0;
      float score = -INFINITY;
      if (lane < count) {
        const int key = base + lane;
        place = table[key / p.page_size] * p.page_size + key % p.page_size;
        score = dot_row<T, VEC>(qs, k_head + static_cast<size_t>(place) * k_stride, d) * p.scale;
      }
      const float top = fmaxf(row_max, warp_max(score)), shift = top == -INFINITY ? 0.0f : top;
      const float alpha = row_max == top ? 1.0f : expf(row_max - top);
      const float weight = lane < count ? expf(score - shift) : 0.0f;
      row_sum = row_sum * alpha + warp_sum(weight);
      row_max = top;
#pragma unroll
      for (int i = 0; i < kColumns; ++i) acc[i] *= alpha;
#pragma unroll 4
      for (int k = 0; k < count; ++k) {
        const float w = __shfl_sync(0xffffffffu, weight, k);
        const T* v_row = v_head + static_cast<size_t>(__shfl_sync(0xffffffffu, place, k)) * v_stride;
#pragma unroll
        for (int i = 0; i < kColumns; ++i)
          if (lane + 32 * i < dv) acc[i] = fmaf(w, to_float<T>(v_row[lane + 32 * i]), acc[i]);
      }
    }
  }
  const float factor = ending_factor(p, h, row_max, row_sum);
  T* out_row = static_cast<T*>(p.out) + (static_cast<size_t>(t) * p.num_heads + h) * dv;
#pragma unroll
  for (int i = 0; i < kColumns; ++i)
    if (lane + 32 * i < dv) out_row[lane + 32 * i] = from_float<T>(acc[i] * factor * gate_factor(p, t, h, lane + 32 * i));
}

// Whether a warp per (token, head) is the faster one: only where no token sees more than 128 keys (of the block table's
// width, a window or a chunk), by what the forms take, in microseconds (largest errors a third).  A warp: 14 + d / 32 per 32 keys
// and 3 besides, 4 + d / 36 at least, or 450 / d pairs of a query and a key per nanosecond, whichever is more.  Split: a start, and a cluster
// after the other.  Tiles: the 64 x 64 tiles of keys that a tile's requests walk one after another.  Warps / before: 100 tokens
// of one request each with a window of 32, 14 heads of 64 on 2 in 32 bits 23 / 48 us, 8 heads of 96 21 / 216, 4 of 256 on 1
// 25 / 94; 30 portions of 7 behind 100: 72 / 133, 68 / 310, 82 / 363; 64 tokens of one prompt: 36 / 17, 35 / 109, 42 / 43.
static bool warps_win(const AttentionParams& p, int dp, bool vec, bool narrow, int requests) {
  long long most = static_cast<long long>(p.table_width) * p.page_size;
  if (p.window > 0) most = std::min<long long>(most, static_cast<long long>(p.window) + p.keep_first);
  if (p.chunk > 0) most = std::min<long long>(most, p.chunk);
  const double run = static_cast<double>(p.num_tokens) / std::max(requests, 1);   // tokens of a request, on average
  // (many requests of a token each in bfloat16: the split form's clusters are worth more keys; 100 behind 300, 8 heads of 96: 220 / 380 us)
  if (most > (narrow && run < 2 ? 512 : 128) || (p.num_tokens > kTileRows && requests <= 1)) return false;
  const int group = p.num_heads / p.num_kv_heads;
  // the keys there probably are: widths are in whole pages, and an engine's in powers of two from eight pages on
  const double keys = most >= 128 ? 0.7 * most : most - 0.5 * p.page_size, d = std::max(p.head_dim, p.value_dim);
  const double warps = std::max({3.0 + (14.0 + d / 32) * keys / 32, 4.0 + d / 36,
                                 static_cast<double>(p.num_tokens) * p.num_heads * keys * std::max(d, 90.0) / 450e3});
  const double start = dp == 64 ? 7.0 : dp == 128 ? 8.0 : 10.0, cluster = dp == 64 ? 0.11 : dp == 128 ? 0.21 : 0.6;
  const double split = start + static_cast<double>(p.num_tokens) * p.num_kv_heads * ((group + kRows - 1) / kRows) * cluster *
                                   (1.0 + std::max(keys - 128.0, 0.0) / 600);
  if (p.num_tokens <= kTileRows) return warps < split;
  if (run < 2) return warps < 8.0 + split;
  const double walked = std::min(kTileRows / run + 1, static_cast<double>(requests)) * ((most + kTileKeys - 1) / kTileKeys);
  return warps < 8.0 + walked * (dp == 64 ? (vec ? 7.0 : 10.0) : dp == 128 ? 12.0 : 19.0);
}

// Up to this many tokens (a tile's rows) a step's keys are split between blocks: a single tile per head would leave
// the chip idle.  With more, tiles of 64 tokens share what they read.
constexpr int kSplitTokens = 64;

template <typename T, int DP, bool VEC>
static int launch_split(const AttentionParams& p, int clusters, cudaStream_t s) {
  static SharedMemoryOptIn opt_in;
  constexpr int kBytes = static_cast<int>(sizeof(SplitShared<DP>));
  const int opted = opt_in.ask(reinterpret_cast<const void*>(attention_split_kernel<T, DP, VEC>), kBytes);
  if (opted) return opted;
  const int group = p.num_heads / p.num_kv_heads;
  return launch_in_clusters(attention_split_kernel<T, DP, VEC>, kSplits, dim3(kSplits, p.num_kv_heads * ((group + kRows - 1) / kRows), clusters),
                            dim3(kAttentionThreads), kBytes, s, p);
}

// Among how many blocks a tile's keys are cut: 1, 2 or 4, by the longest of what a block walks and what all of them cost a
// multiprocessor, in microseconds: a tile of 64 keys `tile`, a block's start and ending `start`, joining 4.  The keys are those the
// block table, a window or a chunk leaves room for; several requests see half of them on average (the longest history may be
// a lone token's, whose launch is another), and below 128 tokens of several requests it may be a lone token's alone.  `longest`: the
// keys of the longest of the requests that bring several tokens, where the caller knows (0: not): short requests in a wide table
// have none to share (eight portions of 60 tokens, room for 512, a 32-bit step of four layers: 1,220 us shared, 1,142 not).  1 / 2 / 4
// blocks: 14 heads of 64 on 2, 200 tokens 28 / 25 / 21 us, 800 106 / 75 / 85, 2,048 299 / 292 / 342, 800 under a window of 256 55 / 60 / 72,
// 100 behind 1,000 119 / 68 / 52; 12 heads of 128 on 2, 1,024 tokens of three requests 206 / 138 / 146, 100 behind 3,000 556 / 285 /
// 190; 4 heads of 256 on 1, 800 tokens 245 / 146 / 109; two tiles of keys: 65 tokens, 14 heads of 64 14.8 / 17.2.
static int tile_members(const AttentionParams& p, int dp, int requests, int longest) {
  long long most = static_cast<long long>(p.table_width) * p.page_size;
  if (longest > 0) most = std::min<long long>(most, longest);
  if (p.window > 0) most = std::min<long long>(most, static_cast<long long>(p.window) + kTileRows + p.keep_first);
  if (p.chunk > 0) most = std::min<long long>(most, p.chunk);
  const long long walked = (most + kTileKeys - 1) / kTileKeys;
  if (walked < 3 || (requests > 1 && p.num_tokens < 2 * kTileRows)) return 1;
  const double run = static_cast<double>(p.num_tokens) / std::max(requests, 1);
  const double in_tile = requests > 1 ? std::min(kTileRows / run + 1.0, static_cast<double>(requests)) : 1.0;
  const double seen = requests > 1 ? 0.5 * most : p.window > 0 || p.chunk > 0 ? most : most - 0.5 * std::min<double>(run, most);
  const double tile = dp == 64 ? 6.2 : dp == 128 ? 11.8 : 18.5, start = dp == 64 ? 4.7 : dp == 128 ? 7.0 : 12.0;
  const double blocks = static_cast<double>(p.num_heads) * ((p.num_tokens + kTileRows - 1) / kTileRows);
  double best = 0.0;
  int members = 1;
  for (int m = 1; m <= kMostMembers; m *= 2) {
    const double longest = start + tile * in_tile * ((walked + m - 1) / m);
    const double all = blocks * (m * start + in_tile * seen / kTileKeys * tile) / multiprocessors();
    const double cost = (m > 1 ? 4.0 : 0.0) + std::max(longest, all);
    if (m == 1 || cost < best) best = cost, members = m;
  }
  return members;
}

// In a step of portions beside tokens that stand alone (other requests' decode tokens) those would walk their whole
// histories in a tile's rows that they do not fill, behind the tile's other requests: they go to the split form, a launch
// of their own (1,024 tokens, one of them alone behind 900 keys: 270 us in the tiles alone, 133 + 21 us).
template <typename T, int DP, bool VEC>
static int launch_attention(const AttentionParams& asked, int requests, int longest, cudaStream_t s) {
  AttentionParams p = asked;
  if (warps_win(p, DP, VEC, sizeof(T) == 2, requests))
    return vipera_launch(attention_warp_kernel<T, VEC>, dim3(p.num_tokens, (p.num_heads + kWarpsPerBlock - 1) / kWarpsPerBlock),
                         dim3(kWarpsPerBlock * 32), 0, s, p);
  if (p.num_tokens <= kSplitTokens) return launch_split<T, DP, VEC>(p, p.num_tokens, s);
  if (requests > 1) {
    p.singles = 1;
    const int status = launch_split<T, DP, VEC>(p, requests < 65535 ? requests : 65535, s);
    if (status) return status;
  }
  static SharedMemoryOptIn opt_in, opt_in_join;
  constexpr int kBytes = static_cast<int>(sizeof(TileShared<DP>));
  const dim3 grid(p.num_heads, (p.num_tokens + kTileRows - 1) / kTileRows);
  const int members = tile_members(p, DP, requests, longest);
  if (members == 1) {
    const int opted = opt_in.ask(reinterpret_cast<const void*>(attention_tile_kernel<T, DP, VEC, false>), kBytes);
    return opted ? opted : vipera_launch(attention_tile_kernel<T, DP, VEC, false>, grid, dim3(kTileThreads), kBytes, s, p, 1);
  }
  const int opted = opt_in_join.ask(reinterpret_cast<const void*>(attention_tile_kernel<T, DP, VEC, true>), kBytes);
  return opted ? opted : launch_in_clusters(attention_tile_kernel<T, DP, VEC, true>, members, dim3(grid.x * members, grid.y), dim3(kTileThreads), kBytes, s, p, members);
}

template <typename T>
static int launch_sizes(const AttentionParams& p, int requests, int longest, cudaStream_t s) {
  constexpr int kPiece = 16 / static_cast<int>(sizeof(T));
  const bool vec = p.head_dim % kPiece == 0 && p.value_dim % kPiece == 0 &&
                   ((reinterpret_cast<uintptr_t>(p.k_pool) | reinterpret_cast<uintptr_t>(p.v_pool)) & 15) == 0;
  const int largest = p.head_dim > p.value_dim ? p.head_dim : p.value_dim;
  if (largest <= 64) return vec ? launch_attention<T, 64, true>(p, requests, longest, s) : launch_attention<T, 64, false>(p, requests, longest, s);
  if (largest <= 128) return vec ? launch_attention<T, 128, true>(p, requests, longest, s) : launch_attention<T, 128, false>(p, requests, longest, s);
  return vec ? launch_attention<T, 256, true>(p, requests, longest, s) : launch_attention<T, 256, false>(p, requests, longest, s);
}

// q is [tokens, heads, d] and out [tokens, heads, value_dim]; the key pool is
// [pages, page_size, kv_heads, d] and the value pool the same with value_dim last.
// token_seq[t] is the row of block_table (width table_width) of token t's request and
// positions[t] its position.  The keys and values of this step's tokens must already be
// in the cache.  window = 0 means every earlier key is visible; keep_first counts only with a
// window; sink != 0 adds the sink to the denominator.
// sink_values (null: none) holds a learned sink score per query head; gate (null: none) the output
// gate's 32-bit pre-activations, row t at gate + t * gate_stride, [heads * value_dim] values ([heads] with
// gate_per_head).
// `requests`: the rows of block_table (1: not known; every token then takes the tiles).
VIPERA_API int vipera_attention_step(const void* q, void* out, int dtype, const void* k_pool, const void* v_pool,
                                      const int* token_seq, const int* positions, const int* block_table,
                                      int table_width, int page_size, int num_tokens, int num_heads,
                                      int num_kv_heads, int head_dim, int value_dim, float scale, int window,
                                      int keep_first, int sink, int chunk, float out_scale, const float* sink_values,
                                      const float* gate, long long gate_stride, int gate_per_head, int requests, int longest, void* stream) {
  if (num_tokens <= 0) return VIPERA_OK;
  if (chunk < 0 || (chunk > 0 && window > 0)) return VIPERA_BAD_ARGUMENT;
  if (head_dim <= 0 || head_dim > kMaxHeadDim) return VIPERA_BAD_SHAPE;
  if (value_dim <= 0 || value_dim > kMaxHeadDim || keep_first < 0) return VIPERA_BAD_SHAPE;
  if (num_heads <= 0 || num_kv_heads <= 0 || num_heads % num_kv_heads != 0) return VIPERA_BAD_SHAPE;
  if (page_size <= 0 || table_width <= 0 || window < 0) return VIPERA_BAD_ARGUMENT;
  if (num_heads > 65535) return VIPERA_BAD_SHAPE;
  const AttentionParams p{q, out, k_pool, v_pool, token_seq, positions, block_table, table_width, page_size, num_tokens, num_heads,
                          num_kv_heads, head_dim, value_dim, scale, window, keep_first, sink, chunk, out_scale, sink_values, gate,
                          gate_stride, gate_per_head, 0};
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (dtype == VIPERA_F32) return launch_sizes<float>(p, requests, longest, s);
  if (dtype == VIPERA_BF16) return launch_sizes<__nv_bfloat16>(p, requests, longest, s);
  return VIPERA_BAD_DTYPE;
}

VIPERA_API const char* vipera_attention_status_text(int status) { return vipera_status_text(status); }
