// Linear attention with one constant decay per head.
//
// Per head a matrix S [d, dv] of 32-bit floats, zero at a request's start.  With q, k, v the silu
// of their projections, for each token
//
//     S = lambda_h S + k v^T        o = S^T q
//
// and the concatenated heads' o is divided by its root mean square over the whole row, multiplied by a
// weight per value and by sigmoid(gate) (lightning_finish_kernel).
//
// A block owns 32 value columns of a head's state for one job; a lane a column, a warp a run of
// neighbouring rows (so that a thread reads its rows' k and q four at a time from shared memory),
// each thread's share of S in registers.  The operands of kStage
// tokens (silu applied) are staged in shared memory; the four warps' partial outputs are added in
// a fixed order.  Three kinds of job (own notation; a chunk is kChunk tokens of one entry, cut
// where the entry's tokens start in the step):
//   walk     a job is an entry: from the request's state (zero if fresh) over all its tokens,
//            with outputs, leaving the new state.  Steps of few tokens and of single tokens.
//   ends     a job is a chunk: from zero over the chunk, no outputs, leaving E_c = sum_s
//            lambda^(len - 1 - s) k_s v_s^T in the chunk's scratch row.
//   outputs  a job is a chunk: from the state at the chunk's start (the scratch row), with outputs.
// (The two kinds of chunk jobs run as products, linear_chunks.cuh, where its rows are whole 16-byte pieces.)
// Between ends and outputs, lightning_carry_kernel walks each entry's chunks: start_c = S;
// S = lambda^len_c S + E_c; the request's new state is the last S.  Another cut of a prompt only
// re-associates 32-bit sums.
#include "linear_chunks.cuh"

constexpr int kChunk = 64;
constexpr int kStage = 16;
constexpr int kColumns = 32;
constexpr int kRowWarps = 4;

enum LightningMode { MODE_WALK = 0, MODE_ENDS = 1, MODE_OUTPUTS = 2 };

struct LightningParams {
  const float* proj;        // [tokens, proj_width] 32-bit pre-activations of q, k, v and the gate
  long long proj_width;
  int q_off, k_off, v_off, g_off;
  const float* decay;       // [heads]
  float* state;             // [slots, heads * d * dv]
  const int* entry_starts;  // [entries + 1]
  const int* state_slots;   // [entries]
  const int* fresh;         // [entries]
  float* raw;               // [tokens, heads * dv] outputs before the norm
  const float* norm_weight; // [heads * dv]
  void* out;                // [tokens, heads * dv]
  float* chunk_state;       // [jobs, heads * d * dv] (chunked form only)
  int heads, d, dv, num_entries, num_tokens, num_jobs;
  float eps;
  int activated;            // 1: q, k and v in proj are past their silu already (the chunked form's first kernel)
};

__device__ __forceinline__ float silu(float z) { return z / (1.0f + expf(-z)); }

// The chunk a job index names: (entry, first token, one past the last), or entry -1 past the last chunk.
__device__ __forceinline__ void find_chunk(const int* __restrict__ entry_starts, int num_entries, int job, int* entry,
                                           int* begin, int* end) {
  int base = 0;
  *entry = -1;
  for (int e = 0; e < num_entries; ++e) {
    const int start = entry_starts[e], stop = entry_starts[e + 1];
    const int chunks = (stop - start + kChunk - 1) / kChunk;
    if (job < base + chunks) {
      *entry = e;
      *begin = start + (job - base) * kChunk;
      *end = min(*begin + kChunk, stop);
      return;
    }
    base += chunks;
  }
}

// The chunked form reads every token's q and k in each block of its head's columns, twice: the silu
// is applied once, in place (the gate's columns stay as they are).
__global__ void __launch_bounds__(256)
lightning_activate_kernel(LightningParams p) {
  pdl_launch_dependents();
  pdl_wait();
  const int per_token = p.heads * (2 * p.d + p.dv);
  const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= static_cast<long long>(p.num_tokens) * per_token) return;
  const long long t = i / per_token;
  int c = static_cast<int>(i % per_token);
  int column;
  if (c < p.heads * p.d) column = p.q_off + c;
  else if ((c -= p.heads * p.d) < p.heads * p.d) column = p.k_off + c;
  else column = p.v_off + c - p.heads * p.d;
  float* at = const_cast<float*>(p.proj) + t * p.proj_width + column;
  *at = silu(*at);
}

template <int RPT, int MODE>
__global__ void __launch_bounds__(kRowWarps * 32)
lightning_scan_kernel(LightningParams p) {
  extern __shared__ __align__(16) float shared[];
  float* q_s = shared;                       // [kStage][d]
  float* k_s = q_s + kStage * p.d;           // [kStage][d]
  float* v_s = k_s + kStage * p.d;           // [kStage][kColumns]
  float* part = v_s + kStage * kColumns;     // [kStage][kRowWarps][kColumns]
  __shared__ int job_info[3];
  pdl_launch_dependents();
  pdl_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int h = blockIdx.y, job = blockIdx.z;
  const int column = blockIdx.x * kColumns + lane;
  const bool live = column < p.dv;
  int entry, begin, end;
  if (MODE == MODE_WALK) {
    entry = job;
    begin = p.entry_starts[entry];
    end = p.entry_starts[entry + 1];
  } else {
    if (threadIdx.x == 0) find_chunk(p.entry_starts, p.num_entries, job, &job_info[0], &job_info[1], &job_info[2]);
    __syncthreads();
    entry = job_info[0], begin = job_info[1], end = job_info[2];
    if (entry < 0) return;
  }
  if (end <= begin) return;
  const float lambda = p.decay[h];
  const size_t state_size = static_cast<size_t>(p.heads) * p.d * p.dv;
  float* own = MODE == MODE_WALK ? p.state + static_cast<size_t>(p.state_slots[entry]) * state_size
                                 : p.chunk_state + static_cast<size_t>(job) * state_size;
  own += static_cast<size_t>(h) * p.d * p.dv;
  float s[RPT];
  const bool load = MODE == MODE_OUTPUTS || (MODE == MODE_WALK && !p.fresh[entry]);
#pragma unroll
  for (int i = 0; i < RPT; ++i) {
    const int row = warp * RPT + i;
    s[i] = (load && live && row < p.d) ? own[static_cast<size_t>(row) * p.dv + column] : 0.0f;
  }
  for (int base = begin; base < end; base += kStage) {
    const int count = min(kStage, end - base);
    __syncthreads();
    for (int i = threadIdx.x; i < count * p.d; i += blockDim.x) {
      const int tt = i / p.d, e = i % p.d;
      const float* row = p.proj + static_cast<size_t>(base + tt) * p.proj_width;
      const float q_raw = MODE != MODE_ENDS ? row[p.q_off + h * p.d + e] : 0.0f, k_raw = row[p.k_off + h * p.d + e];
      if (MODE != MODE_ENDS) q_s[tt * p.d + e] = (MODE != MODE_WALK && p.activated) ? q_raw : silu(q_raw);
      k_s[tt * p.d + e] = (MODE != MODE_WALK && p.activated) ? k_raw : silu(k_raw);
    }
    for (int i = threadIdx.x; i < count * kColumns; i += blockDim.x) {
      const int tt = i / kColumns, c = blockIdx.x * kColumns + i % kColumns;
      const float v_raw = c < p.dv ? p.proj[static_cast<size_t>(base + tt) * p.proj_width + p.v_off + h * p.dv + c] : 0.0f;
      v_s[i] = (MODE != MODE_WALK && p.activated) ? v_raw : silu(v_raw);
    }
    __syncthreads();
    const bool whole_rows = (p.d & 3) == 0 && (warp + 1) * RPT <= p.d;   // this warp's rows all exist, in fours
    for (int tt = 0; tt < count; ++tt) {
      const float v = v_s[tt * kColumns + lane];
      float o = 0.0f;
      if (RPT % 4 == 0 && whole_rows) {
        const float4* k4 = reinterpret_cast<const float4*>(k_s + tt * p.d + warp * RPT);
        const float4* q4 = reinterpret_cast<const float4*>(q_s + tt * p.d + warp * RPT);
#pragma unroll
        for (int i = 0; i < RPT / 4; ++i) {
          const float4 kk = k4[i];
          s[4 * i] = fmaf(lambda, s[4 * i], kk.x * v);
          s[4 * i + 1] = fmaf(lambda, s[4 * i + 1], kk.y * v);
          s[4 * i + 2] = fmaf(lambda, s[4 * i + 2], kk.z * v);
          s[4 * i + 3] = fmaf(lambda, s[4 * i + 3], kk.w * v);
          if (MODE != MODE_ENDS) {
            const float4 qq = q4[i];
            o = fmaf(s[4 * i], qq.x, o);
            o = fmaf(s[4 * i + 1], qq.y, o);
            o = fmaf(s[4 * i + 2], qq.z, o);
            o = fmaf(s[4 * i + 3], qq.w, o);
          }
        }
      } else {
#pragma unroll
        for (int i = 0; i < RPT; ++i) {
          const int row = warp * RPT + i;
          if (row < p.d) {
            s[i] = fmaf(lambda, s[i], k_s[tt * p.d + row] * v);
            if (MODE != MODE_ENDS) o = fmaf(s[i], q_s[tt * p.d + row], o);
          }
        }
      }
      if (MODE != MODE_ENDS) part[(tt * kRowWarps + warp) * kColumns + lane] = o;
    }
    if (MODE != MODE_ENDS) {
      __syncthreads();
      for (int i = threadIdx.x; i < count * kColumns; i += blockDim.x) {
        const int tt = i / kColumns, l = i % kColumns, c = blockIdx.x * kColumns + l;
        if (c < p.dv) {
          const float* o = part + tt * kRowWarps * kColumns + l;
          p.raw[static_cast<size_t>(base + tt) * (p.heads * p.dv) + h * p.dv + c] =
              ((o[0] + o[kColumns]) + o[2 * kColumns]) + o[3 * kColumns];
        }
      }
    }
  }
  if (MODE != MODE_OUTPUTS && live) {
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
      const int row = warp * RPT + i;
      if (row < p.d) own[static_cast<size_t>(row) * p.dv + column] = s[i];
    }
  }
}

// A thread N neighbouring values of a head's state and entry (where rows are whole pieces of N): the entry's chunks in a row,
// `AHEAD` of them asked for together, then walked in order.  What bounds it: the chunks' states, read and written; the powers of
// lambda, which every thread computed for itself, were most of its instructions (28 us of ten requests of 100 tokens, 6 heads of
// 128 x 256, where the bytes are 6; two values and sixteen ahead with them 46).  The mixer, cold, us by one value and eight ahead, each
// with its powers / two and sixteen / four and four: 6 heads of 128 x 256, 2,048 tokens 156.6 / 148.5 / 156.5, 1,030 124.0 / 123.2 /
// 127.9, ten requests of 100 119.9 / 130.7 / 124.6, twenty of 20 124 / 117 / 106, forty of 50 276 / 206 / 177; of 64 x 128, three of 700
// 132 / 128 / 122, eight of 256 114 / 124 / 122.  So requests of few chunks take four and four.
constexpr int kCarryThreads = 128;
constexpr int kCarryShort = 12;   // chunks of a request on average, up to which it takes four values and four ahead

template <int N, int AHEAD>
__global__ void __launch_bounds__(kCarryThreads)
lightning_carry_kernel(LightningParams p) {
  // lambda^kChunk of each head of the block's values, and what the request's last chunk leaves: by repeated multiplication, the same
  // way the scan applies it, a thread a head (each of the block's threads for itself they were most of this kernel's instructions)
  __shared__ float whole[kCarryThreads * N + 2], ends_with[kCarryThreads * N + 2];
  __shared__ int first_job;
  pdl_launch_dependents();
  pdl_wait();
  const int entry = blockIdx.y, head_size = p.d * p.dv;
  const size_t state_size = static_cast<size_t>(p.heads) * head_size, first = static_cast<size_t>(blockIdx.x) * (kCarryThreads * N);
  const size_t element = first + threadIdx.x * N;
  const int start = p.entry_starts[entry], stop = p.entry_starts[entry + 1];
  if (stop <= start) return;
  const int head0 = static_cast<int>(first / head_size), heads = min(p.heads - head0, static_cast<int>((first % head_size + kCarryThreads * N - 1) / head_size) + 1);
  if (threadIdx.x >= kCarryThreads - 32) {
    const int lane = threadIdx.x & 31;
    int jobs = 0;
    for (int e = lane; e < entry; e += 32) jobs += (p.entry_starts[e + 1] - p.entry_starts[e] + kChunk - 1) / kChunk;
    jobs = __reduce_add_sync(0xffffffffu, jobs);
    if (lane == 0) first_job = jobs;
  }
  for (int i = threadIdx.x; i < heads; i += kCarryThreads) {
    const float lambda = p.decay[head0 + i];
    const int tail = (stop - start - 1) % kChunk + 1;
    float power = 1.0f, ends = 1.0f;
#pragma unroll
    for (int k = 1; k <= kChunk; ++k) {
      power *= lambda;
      if (k == tail) ends = power;
    }
    whole[i] = power;
    ends_with[i] = ends;
  }
  struct alignas(4 * N) Values { float v[N]; };
  const bool valid = element < state_size;
  Values* own = reinterpret_cast<Values*>(p.state + static_cast<size_t>(p.state_slots[entry]) * state_size + element);
  Values s{};
  if (valid && !p.fresh[entry]) s = *own;
  __syncthreads();
  if (!valid) return;
  const int at = static_cast<int>(static_cast<unsigned>(element) / static_cast<unsigned>(head_size)) - head0;   // (a state of 4 G elements does not exist)
  const float factor = whole[at], last_factor = ends_with[at];
  Values* states = reinterpret_cast<Values*>(p.chunk_state + static_cast<size_t>(first_job) * state_size + element);
  const size_t step = state_size / N;   // (a row of the state is whole pieces)
  const int chunks = (stop - start + kChunk - 1) / kChunk;
  for (int c0 = 0; c0 < chunks; c0 += AHEAD, states += AHEAD * step) {
    Values ending[AHEAD];
#pragma unroll
    for (int c = 0; c < AHEAD; ++c)
      if (c0 + c < chunks) ending[c] = states[c * step];
#pragma unroll
    for (int c = 0; c < AHEAD; ++c) {
      if (c0 + c >= chunks) break;
      states[c * step] = s;
      const float power = c0 + c + 1 < chunks ? factor : last_factor;
#pragma unroll
      for (int j = 0; j < N; ++j) s.v[j] = fmaf(power, s.v[j], ending[c].v[j]);
    }
  }
  *own = s;
}

// The norm over the concatenated heads, the norm's weight and the output gate; a block per token.  What bounds it: memory.
// KEPT: pieces of four values a thread keeps of a row (0: rows that are read again, a value at a time).  Narrow rows take blocks of no
// more threads than they have pieces: 2,048 rows of 768 values 6.5 us, by 256 threads of four pieces 8.4, a value at a time 10.8.
constexpr int kFinishKept = 4;

template <typename TO, int KEPT>
__global__ void __launch_bounds__(256)
lightning_finish_kernel(LightningParams p) {
  __shared__ float scratch[32];
  pdl_launch_dependents();
  pdl_wait();
  const int t = blockIdx.x;
  const int width = p.heads * p.dv;
  const float* raw = p.raw + static_cast<size_t>(t) * width;
  const float* gate = p.proj + static_cast<size_t>(t) * p.proj_width + p.g_off;
  if constexpr (KEPT > 0) {
    // rows of whole 16-byte pieces that fit the block's registers: read once, all of it at the same time
    float4 o[KEPT], g[KEPT];
    float sum = 0.0f;
#pragma unroll
    for (int j = 0; j < KEPT; ++j) {
      const int i = (threadIdx.x + blockDim.x * j) * 4;
      o[j] = g[j] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      if (i < width) o[j] = *reinterpret_cast<const float4*>(raw + i), g[j] = *reinterpret_cast<const float4*>(gate + i);
    }
#pragma unroll
    for (int j = 0; j < KEPT; ++j) sum += o[j].x * o[j].x + o[j].y * o[j].y + o[j].z * o[j].z + o[j].w * o[j].w;
    const float inverse = 1.0f / sqrtf(block_sum(sum, scratch) / static_cast<float>(width) + p.eps);
    TO* out = static_cast<TO*>(p.out) + static_cast<size_t>(t) * width;
#pragma unroll
    for (int j = 0; j < KEPT; ++j) {
      const int i = (threadIdx.x + blockDim.x * j) * 4;
      if (i >= width) break;
      const float4 w = *reinterpret_cast<const float4*>(p.norm_weight + i);
      store_four_as<TO>(out + i, o[j].x * inverse * w.x * sigmoid(g[j].x), o[j].y * inverse * w.y * sigmoid(g[j].y),
                        o[j].z * inverse * w.z * sigmoid(g[j].z), o[j].w * inverse * w.w * sigmoid(g[j].w));
    }
  } else {
    float sum = 0.0f;
    for (int i = threadIdx.x; i < width; i += blockDim.x) sum += raw[i] * raw[i];
    const float inverse = 1.0f / sqrtf(block_sum(sum, scratch) / static_cast<float>(width) + p.eps);
    TO* out = static_cast<TO*>(p.out) + static_cast<size_t>(t) * width;
    for (int i = threadIdx.x; i < width; i += blockDim.x)
      out[i] = from_float<TO>(raw[i] * inverse * p.norm_weight[i] * sigmoid(gate[i]));
  }
}

template <typename TO>
static int launch_finish(const LightningParams& p, cudaStream_t s) {
  const int width = p.heads * p.dv, pieces = (width + 3) / 4;
  const uintptr_t bases = reinterpret_cast<uintptr_t>(p.raw) | reinterpret_cast<uintptr_t>(p.proj) | reinterpret_cast<uintptr_t>(p.norm_weight) | reinterpret_cast<uintptr_t>(p.out);
  if (pieces > kFinishKept * 256 || width % 4 || p.proj_width % 4 || p.g_off % 4 || (bases & 15))
    return vipera_launch(lightning_finish_kernel<TO, 0>, p.num_tokens, 256, 0, s, p);
  const int threads = pieces < 256 ? (pieces + 31) / 32 * 32 : 256;
  if (pieces <= 256) return vipera_launch(lightning_finish_kernel<TO, 1>, p.num_tokens, threads, 0, s, p);
  return vipera_launch(lightning_finish_kernel<TO, kFinishKept>, p.num_tokens, threads, 0, s, p);
}

template <int N, int AHEAD>
static int launch_carry_as(const LightningParams& p, cudaStream_t s) {
  const size_t threads = static_cast<size_t>(p.heads) * p.d * p.dv / N;
  return vipera_launch(lightning_carry_kernel<N, AHEAD>, dim3(static_cast<unsigned>((threads + kCarryThreads - 1) / kCarryThreads), p.num_entries), kCarryThreads, 0, s, p);
}
static int launch_carry(const LightningParams& p, cudaStream_t s) {
  const uintptr_t bases = reinterpret_cast<uintptr_t>(p.state) | reinterpret_cast<uintptr_t>(p.chunk_state);
  if (p.dv % 4 == 0 && (bases & 15) == 0 && p.num_tokens <= static_cast<long long>(kCarryShort) * kChunk * p.num_entries) return launch_carry_as<4, 4>(p, s);
  return p.dv % 2 == 0 && (bases & 7) == 0 ? launch_carry_as<2, 16>(p, s) : launch_carry_as<1, 16>(p, s);
}

template <int RPT>
static int launch_scans(const LightningParams& params, bool chunked, cudaStream_t s) {
  LightningParams p = params;
  p.activated = 0;
  const size_t shared = (static_cast<size_t>(2 * kStage) * p.d + kStage * kColumns + kStage * kRowWarps * kColumns) * sizeof(float);
  const int tiles = (p.dv + kColumns - 1) / kColumns;
  if (!chunked)
    return vipera_launch(lightning_scan_kernel<RPT, MODE_WALK>, dim3(tiles, p.heads, p.num_entries), kRowWarps * 32, shared, s, p);
  // Rows that are not whole 16-byte pieces walk their chunks, and so do small heads (up to 64 key channels): a walk's
  // block holds their state in few registers, and the products' tiles are not filled.  Walks / products, the mixer: 4 heads of
  // 64 x 128, 400 and 800 tokens: 75 / 86 and 81 / 95 us; 8 heads: 82 / 81 and 95 / 100; 4 heads of 128 x 256: 134 / 95 and 146 / 121.
  const LinearArgs chunks{p.proj, p.proj_width, p.q_off, p.k_off, p.v_off, nullptr, nullptr, p.decay, p.entry_starts, p.chunk_state,
                          nullptr, p.raw, p.num_entries, p.heads, p.d, p.dv, 1.0f};
  if (p.d > 64 && linear_chunks_take(chunks)) {
    int status = launch_linear_ends<false>(chunks, p.num_jobs, s);
    if (status) return status;
    status = launch_carry(p, s);
    if (status) return status;
    return launch_linear_outputs<false>(chunks, p.num_jobs, s);
  }
  p.activated = 1;
  const long long values = static_cast<long long>(p.num_tokens) * p.heads * (2 * p.d + p.dv);
  int status = vipera_launch(lightning_activate_kernel, static_cast<unsigned>((values + 255) / 256), 256, 0, s, p);
  if (status) return status;
  status = vipera_launch(lightning_scan_kernel<RPT, MODE_ENDS>, dim3(tiles, p.heads, p.num_jobs), kRowWarps * 32, shared, s, p);
  if (status) return status;
  status = launch_carry(p, s);
  if (status) return status;
  return vipera_launch(lightning_scan_kernel<RPT, MODE_OUTPUTS>, dim3(tiles, p.heads, p.num_jobs), kRowWarps * 32, shared, s, p);
}

// num_jobs > 0 (with chunk_state): the chunked form, num_jobs at least the step's count of chunks.
VIPERA_API int vipera_lightning(const LightningParams* params, int out_dtype, void* stream) {
  const LightningParams& p = *params;
  if (p.num_tokens <= 0 || p.num_entries <= 0) return VIPERA_OK;
  if (p.heads <= 0 || p.d <= 0 || p.d > 256 || p.dv <= 0 || p.heads > 65535 || p.num_entries > 65535) return VIPERA_BAD_SHAPE;
  const bool chunked = p.num_jobs > 0;
  if (chunked && (p.chunk_state == nullptr || p.num_jobs > 65535)) return VIPERA_BAD_ARGUMENT;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  int status;
  if (p.d <= 32) status = launch_scans<8>(p, chunked, s);
  else if (p.d <= 64) status = launch_scans<16>(p, chunked, s);
  else if (p.d <= 128) status = launch_scans<32>(p, chunked, s);
  else status = launch_scans<64>(p, chunked, s);
  if (status) return status;
  if (out_dtype == VIPERA_F32) return launch_finish<float>(p, s);
  if (out_dtype == VIPERA_BF16) return launch_finish<__nv_bfloat16>(p, s);
  return VIPERA_BAD_DTYPE;
}

VIPERA_API int vipera_lightning_params_size() { return static_cast<int>(sizeof(LightningParams)); }
VIPERA_API int vipera_lightning_chunk() { return kChunk; }
VIPERA_API const char* vipera_lightning_status_text(int status) { return vipera_status_text(status); }
