// Matrix products with 32-bit accumulation: out[M, N] = A[M, K] . W[N, K]^T.
//
// This is the product kernel of the true 32-bit path (no reduced-precision mode) and the fallback of the bfloat16 path for sizes the tensor-core kernel refuses.
// The reference multiplies one weight matrix by all B activation rows in one pass over the
// weights (crates/vipera-backend-cpu/src/model.rs:1005-1025) and promises that a row's
// result does not depend on its neighbours in the batch (model.rs:881-882); here every output
// element sums over K in an order that is fixed by N, K and the class of row counts: up to eight rows, up to 64, or more (one
// class for values that are widened and for rows off 16 bytes).
//
// Up to eight rows the stream of W bounds the product (gemv_rows_kernel): a warp reads eight rows of W
// through a ring of its own, 512 neighbouring bytes of a row at a time, a lane's four values against all
// rows of A, and adds its lanes' sums at the end.
// A K of up to 320 lies in shared memory whole (gemm_short_kernel).
// 32-bit products of more than 64 rows (whole rows of 16-byte pieces) run on the tensor cores, three bfloat16 parts of every
// number: gemm_split.cuh.  Multiply-adds / tensor cores: 65 rows, W 896 x 896: 17.4 / 17.3 us; W 9,728 x 896: 106 / 38; 128
// rows, W 896 x 4,864: 70 / 47; W 512 x 128, in shared memory whole / tensor cores: 10.5 / 16.8.
// The others of more rows (gemm_simt_kernel): the multiply-add units and the reads of shared memory that feed them.  K is
// cut into eight slabs (of whole chunks of 32), a slab's even and odd places are two chains of fused
// multiply-adds (the two halves of a packed 32-bit pair) whose ends are added, and the slabs are added in
// their order.  A block takes a tile of rows and columns through a ring of cp.async
// stages (rows of 32 values, 16 bytes of padding so that neighbouring rows' 16-byte reads meet no bank
// twice), and where the tiles are too few to fill the chip the eight slabs of a tile go to the eight
// blocks of a cluster, which add their parts through distributed shared memory: one launch and no
// scratch either way.
//
// Measured (B200; a 64 x 64 tile staged value by value before): 8 rows, W 17,920 x 1,536: 166 -> 30 us (3.7 TB/s);
// 8 rows, W 1,536 x 1,536 and 1,536 x 8,960: 461 -> 16 us on average; 1,024 rows, W 9,728 x 896: 758 -> 503 us
// here, 183 us on the tensor cores.  Sums in parts are also closer to 64-bit ones: 8e-7 instead of 3e-6 on a decode step's logits.
//
// Epilogues:
//   STORE     out[m, n] = acc (+ bias[n]), stored as float or bfloat16
//   RESIDUAL  resid[m, n] += acc (+ bias[n])  (32-bit residual stream)
//   SWIGLU    (a gated unit) W holds gate and up rows interleaved in groups of 16 (16 gate rows,
//             then the 16 up rows of the same features, and the bias likewise);
//             out[m, f] = (up + bias) * act(gate + bias), act = silu, silu(z) = z/(1+exp(-z))
//             (model.rs:4368-4374), or the tanh form of gelu,
//             0.5 z (1 + tanh(sqrt(2/pi) (z + 0.044715 z^3)))
#include "gemm_split.cuh"

enum GemmEpilogue { EPI_STORE = 0, EPI_RESIDUAL = 1, EPI_SWIGLU = 2 };

constexpr int kSlabs = 8;          // parts of K with sums of their own
constexpr int kChunk = 32;         // values of K a stage holds
constexpr int kPitch = kChunk + 4; // floats per staged row

// The tiles.  A warp's lanes are LM x LN; a thread owns TM x TN outputs, LM rows and LN columns apart.
template <int BM_, int BN_, int WM_, int WN_, int LM_, int LN_, int TM_, int TN_, int STAGES_>
struct Tile {
  static constexpr int BM = BM_, BN = BN_, WM = WM_, WN = WN_, LM = LM_, LN = LN_, TM = TM_, TN = TN_, STAGES = STAGES_;
  static constexpr int kThreads = WM * WN * 32;
  static constexpr int kSumPitch = BN + 8;
  static constexpr int kStageFloats = (BM + BN) * kPitch;
  static constexpr int kSharedBytes = (STAGES * kStageFloats + BM * kSumPitch) * 4;
  static_assert(LM * LN == 32 && WM * LM * TM == BM && WN * LN * TN == BN, "the tile is covered once");
};
using TileSome = Tile<32, 128, 4, 1, 1, 32, 8, 4, 3>;
using TileMid = Tile<64, 128, 2, 2, 4, 8, 8, 8, 3>;
using TileLow = Tile<64, 64, 4, 2, 4, 8, 4, 4, 2>;   // little shared memory: four blocks an SM hide the staging through registers

struct GemmArgs {
  const void* A;
  const void* W;
  int M, N, K, slab;   // slab: values of K per slab, a multiple of kChunk
  const float* bias;
  void* out;
  float* resid;
  int activation, epilogue, out_bf16;
  int wide;            // rows of whole pieces of eight values on 16-byte boundaries
  int* status;         // for the bounded waits of the tensor-core form
  void* parts;         // room for its left operand's parts, or null
  long long parts_bytes;
};

__device__ __forceinline__ void load_eight(const float* src, float (&v)[8]) {
  const float4 lo = *reinterpret_cast<const float4*>(src), hi = *reinterpret_cast<const float4*>(src + 4);
  v[0] = lo.x, v[1] = lo.y, v[2] = lo.z, v[3] = lo.w, v[4] = hi.x, v[5] = hi.y, v[6] = hi.z, v[7] = hi.w;
}
__device__ __forceinline__ void load_eight(const __nv_bfloat16* src, float (&v)[8]) {
  const uint4 raw = *reinterpret_cast<const uint4*>(src);
  const __nv_bfloat162* pairs = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const float2 f = __bfloat1622float2(pairs[e]);
    v[2 * e] = f.x, v[2 * e + 1] = f.y;
  }
}

// `rows` rows of [extent, K] from row0 on, values k0 .. k0 + kChunk - 1, into shared memory as floats; zeros outside.
// DIRECT: 32-bit rows of whole 16-byte pieces, copied without passing through registers.
template <typename T, bool DIRECT, int ROWS, int THREADS>
__device__ __forceinline__ void stage_rows(float* dst, const T* __restrict__ src, int row0, int extent, int k0, int k_end, int K, bool wide) {
  if (DIRECT) {
#pragma unroll
    for (int i = threadIdx.x; i < ROWS * (kChunk / 4); i += THREADS) {
      const int r = i / (kChunk / 4), piece = (i % (kChunk / 4)) * 4;
      const bool valid = row0 + r < extent && k0 + piece < k_end;
      copy_16(shared_address(dst + r * kPitch + piece),
              reinterpret_cast<const float*>(src) + (valid ? static_cast<size_t>(row0 + r) * K + k0 + piece : 0), valid);
    }
  } else if (wide) {
    // rows of whole pieces of eight values
#pragma unroll 4
    for (int i = threadIdx.x; i < ROWS * (kChunk / 8); i += THREADS) {
      const int r = i / (kChunk / 8), piece = (i % (kChunk / 8)) * 8;
      float v[8] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
      if (row0 + r < extent && k0 + piece < k_end) load_eight(src + static_cast<size_t>(row0 + r) * K + k0 + piece, v);
      *reinterpret_cast<float4*>(dst + r * kPitch + piece) = make_float4(v[0], v[1], v[2], v[3]);
      *reinterpret_cast<float4*>(dst + r * kPitch + piece + 4) = make_float4(v[4], v[5], v[6], v[7]);
    }
  } else {
#pragma unroll 4
    for (int i = threadIdx.x; i < ROWS * kChunk; i += THREADS) {
      const int r = i / kChunk, k = i % kChunk;
      const bool valid = row0 + r < extent && k0 + k < k_end;
      dst[r * kPitch + k] = valid ? to_float<T>(src[static_cast<size_t>(row0 + r) * K + k0 + k]) : 0.0f;
    }
  }
}

template <typename TA, typename TW, typename T, bool DIRECT, bool CLUSTER>
__global__ void __launch_bounds__(T::kThreads)
gemm_simt_kernel(const GemmArgs p) {
  extern __shared__ __align__(16) float gemm_shared[];
  float* sums = gemm_shared;                                 // [BM][kSumPitch]
  float* ring = gemm_shared + T::BM * T::kSumPitch;          // as many stages as there are chunks, STAGES at most
  const TA* A = static_cast<const TA*>(p.A);
  const TW* W = static_cast<const TW*>(p.W);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tile_n = CLUSTER ? blockIdx.x / kSlabs : blockIdx.x;
  const int own_slab = CLUSTER ? blockIdx.x % kSlabs : 0;
  const int m0 = blockIdx.y * T::BM, n0 = tile_n * T::BN;
  const int first_m = (warp / T::WN) * (T::LM * T::TM) + lane / T::LN;
  const int first_n = (warp % T::WN) * (T::LN * T::TN) + lane % T::LN;
  const int begin = own_slab * p.slab, end = CLUSTER ? min(p.K, begin + p.slab) : p.K;
  const int chunks = end > begin ? (end - begin + kChunk - 1) / kChunk : 0;   // (slabs are whole chunks)
  const int slab_chunks = p.slab / kChunk;

  auto stage_w = [&](int chunk) {
    if (chunk < chunks)
      stage_rows<TW, DIRECT, T::BN, T::kThreads>(ring + (chunk % T::STAGES) * T::kStageFloats + T::BM * kPitch, W, n0, p.N,
                                                 begin + chunk * kChunk, end, p.K, p.wide != 0);
  };
  auto stage_a = [&](int chunk) {
    if (chunk < chunks)
      stage_rows<TA, DIRECT, T::BM, T::kThreads>(ring + (chunk % T::STAGES) * T::kStageFloats, A, m0, p.M,
                                                 begin + chunk * kChunk, end, p.K, p.wide != 0);
    copy_commit();
  };
  pdl_launch_dependents();
  // the weights of the first stages are asked for before the kernel ahead has ended
#pragma unroll
  for (int c = 0; c < T::STAGES - 1; ++c) stage_w(c);
  pdl_wait();
#pragma unroll
  for (int c = 0; c < T::STAGES - 1; ++c) stage_a(c);

  unsigned long long acc[T::TM][T::TN];   // (sum over even places, sum over odd places)
#pragma unroll
  for (int i = 0; i < T::TM; ++i)
#pragma unroll
    for (int j = 0; j < T::TN; ++j) acc[i][j] = 0ull;

  int in_slab = 0;
  bool summed = false;
  for (int chunk = 0; chunk < chunks; ++chunk) {
    copy_wait<T::STAGES - 2>();
    __syncthreads();   // this chunk has landed for every thread, and the one before is read out
    stage_w(chunk + T::STAGES - 1);
    stage_a(chunk + T::STAGES - 1);
    const float* a_s = ring + (chunk % T::STAGES) * T::kStageFloats + first_m * kPitch;
    const float* w_s = ring + (chunk % T::STAGES) * T::kStageFloats + (T::BM + first_n) * kPitch;
#pragma unroll
    for (int k = 0; k < kChunk; k += 4) {
      ulonglong2 a[T::TM];
#pragma unroll
      for (int i = 0; i < T::TM; ++i) a[i] = *reinterpret_cast<const ulonglong2*>(a_s + i * T::LM * kPitch + k);
#pragma unroll
      for (int j = 0; j < T::TN; ++j) {
        const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(w_s + j * T::LN * kPitch + k);
#pragma unroll
        for (int i = 0; i < T::TM; ++i) {
          fma_pair(acc[i][j], a[i].x, w.x);
          fma_pair(acc[i][j], a[i].y, w.y);
        }
      }
    }
    if (++in_slab == slab_chunks || chunk + 1 == chunks) {
      // a slab's end: its sums join the tile's (a thread's own places)
#pragma unroll
      for (int i = 0; i < T::TM; ++i)
#pragma unroll
        for (int j = 0; j < T::TN; ++j) {
          float* at = sums + (first_m + i * T::LM) * T::kSumPitch + first_n + j * T::LN;
          const float slab_sum = sum_of_pair(acc[i][j]);
          *at = summed ? *at + slab_sum : slab_sum;
          acc[i][j] = 0ull;
        }
      in_slab = 0;
      summed = true;
    }
  }
  if (CLUSTER) cluster_sync();
  else __syncthreads();

  // The ending.  In a cluster each block finishes every eighth row of the tile.
  const int used_slabs = CLUSTER ? (p.K + p.slab - 1) / p.slab : 1;
  auto total = [&](int m, int n) {
    if (!CLUSTER) return sums[m * T::kSumPitch + n];
    const uint32_t at = shared_address(sums + m * T::kSumPitch + n);
    float part[kSlabs];   // (what a block without values of K holds is not used)
#pragma unroll
    for (int s = 0; s < kSlabs; ++s) part[s] = remote_float(at, s);
    float sum = part[0];
#pragma unroll
    for (int s = 1; s < kSlabs; ++s) sum = s < used_slabs ? sum + part[s] : sum;
    return sum;
  };
  const bool gated = p.epilogue == EPI_SWIGLU;
  const int columns = gated ? T::BN / 2 : T::BN;   // (powers of two)
  const int column_bits = 31 - __clz(columns), blocks = CLUSTER ? kSlabs : 1;
  auto store = [&](size_t at, float value) {
    if (p.out_bf16) static_cast<__nv_bfloat16*>(p.out)[at] = __float2bfloat16_rn(value);
    else static_cast<float*>(p.out)[at] = value;
  };
  // A thread keeps one column (a block has at least as many threads as columns) and takes four rows at a time, whose
  // reads are all on their way before the first store.
  static_assert(T::kThreads >= T::BN, "a thread keeps one column");
  const int c = threadIdx.x & (columns - 1), row_step = T::kThreads >> column_bits;
  const int n = gated ? (c / 16) * 32 + c % 16 : c;   // gated: the gate's column; the feature's up value is 16 further
  if (n0 + n + (gated ? 16 : 0) < p.N) {
    const float bias = p.bias ? p.bias[n0 + n] : 0.0f, up_bias = p.bias && gated ? p.bias[n0 + n + 16] : 0.0f;
    const int pitch = gated ? p.N / 2 : p.N, column = gated ? n0 / 2 + c : n0 + c;
    for (int row = threadIdx.x >> column_bits; row < T::BM / blocks; row += 4 * row_step) {
      float value[4], before[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int m = (row + i * row_step) * blocks + own_slab;
        if (row + i * row_step >= T::BM / blocks || m0 + m >= p.M) continue;
        if (p.epilogue == EPI_RESIDUAL) before[i] = p.resid[static_cast<size_t>(m0 + m) * pitch + column];
        value[i] = total(m, n) + bias;
        if (gated) value[i] = (total(m, n + 16) + up_bias) * gate_activation(value[i], p.activation);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int m = (row + i * row_step) * blocks + own_slab;
        if (row + i * row_step >= T::BM / blocks || m0 + m >= p.M) continue;
        const size_t at = static_cast<size_t>(m0 + m) * pitch + column;
        if (p.epilogue == EPI_RESIDUAL) p.resid[at] = before[i] + value[i];
        else store(at, value[i]);
      }
    }
  }
  if (CLUSTER) cluster_sync();   // no block leaves while another reads its part
}

// ---------------------------------------------------------------------------------------
// Up to eight rows.  `members` (1, 2, 4 or 8, as many as it takes to give every multiprocessor a dozen warps of eight rows of
// W) share rows of W, each every `members`-th run of 128 values of K; a lane adds its places in one chain, the lanes' sums and
// then the members' are added in their order.  Two runs are in flight while one is used, the first two of W before the kernel
// ahead has ended.  MR: rows of A computed (1, 2, 4 or 8).  No sum's order depends on MR, nor on which of two forms runs:
//   gemv_rows_kernel         the members are warps of a block, each with eight rows of W; a warp reads its runs of A itself.
//   gemv_rows_shared_kernel  the members are blocks of a cluster, a block has eight rows of W for each of its eight warps, and
//                            a run of A comes once for all of them.
// Eight rows of A read by every warp are as many bytes from L2 as its rows of W, which bounds the first form at half of the
// memory's rate; the cluster's two barriers cost the second 1.2 us.  8 rows, us in warps / shared: W 32,000 x 1,536 50.6 / 41.2
// (4.8 TB/s), 17,920 x 1,536 27.1 / 22.2, 1,536 x 8,960 20.0 / 16.3, 896 x 4,864 11.2 / 9.5; 2,048 x 1,536 6.1 / 7.6.  4 rows:
// 32,000 x 1,536 37.5 / 35.5, but 1,536 x 8,960 in eight parts 11.9 / 12.9.  (Pairs of chains with packed multiply-adds and four
// rows a warp: 42.4 and 24.3 us where these take 41.2 and 22.2: what bounds it now is shared memory, which feeds W and A.)
// ---------------------------------------------------------------------------------------
constexpr int kFewRows = 8;     // rows of A, and rows of W a warp holds
constexpr int kFewWarps = 8;    // of a block
constexpr int kFewStages = 3;   // runs of a warp's ring
constexpr int kFewRun = 128;    // values of K
constexpr int kFewSplit = 8;    // most members
constexpr long long kSharedFrom = 4000000;   // numbers of W
// Runs of a member, below which the cluster's barriers and a run of A that is asked for behind the wait are not made up for, by
// more than four rows and by up to four.  8 rows, inputs out of L2, us in warps / shared: 2,048 x 2,048 (two runs) 6.5 / 7.8, 8,000 x
// 512 (two) 6.4 / 7.5, 3,072 x 2,048 (two) 12.4 / 13.3, 9,728 x 896 (three and a half) 18.1 / 15.7, 1,024 x 4,096 (four) 9.8 / 8.2.
// 4 rows: 16,384 x 256 (two) 4.6 / 5.0, 32,000 x 896 (seven) 21.8 / 22.1, 17,920 x 1,536 (twelve) 19.6 / 18.8.
constexpr int kSharedRuns = 3, kSharedRunsFour = 8;

// The lanes' sums of N values: at each step a lane keeps one half of the values it holds and hands over the other, until
// it holds one or two; then every lane holds the same value's.  Returns the first value a lane ends with, and how many.
template <int N>
__device__ __forceinline__ int sum_lanes(float (&acc)[N], int lane, int& held) {
  int first = 0;
  held = N;
#pragma unroll
  for (int offset = 16; offset > 0; offset >>= 1) {
    const bool upper = (lane & offset) != 0;
    if (held > 1) {
      held >>= 1;
#pragma unroll
      for (int i = 0; i < N / 2; ++i) {
        if (i < held) {
          const float keep = upper ? acc[i + held] : acc[i], give = upper ? acc[i] : acc[i + held];
          acc[i] = keep + __shfl_xor_sync(0xffffffffu, give, offset);
        }
      }
      if (upper) first += held;
    } else {
      acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], offset);
    }
  }
  return first;
}

template <int MR>
__global__ void __launch_bounds__(kFewWarps * 32, 2)
gemv_rows_kernel(const GemmArgs p, int warps) {
  __shared__ float parts[kFewWarps][kFewRows * MR];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int group = (blockIdx.x * kFewWarps + warp) / warps, member = warp % warps;
  const float* A = static_cast<const float*>(p.A);
  const float* W = static_cast<const float*>(p.W);
  const bool gated = p.epilogue == EPI_SWIGLU;
  // the group's rows: eight neighbours, or the gates and the ups of four neighbouring features
  auto row_of = [&](int r) {
    if (!gated) return group * kFewRows + r;
    const int feature = group * (kFewRows / 2) + r % (kFewRows / 2);
    return feature / 16 * 32 + feature % 16 + (r >= kFewRows / 2 ? 16 : 0);
  };
  // A lane copies the 16 bytes of each row that it will use itself, so a wait for its own copies is all it needs.
  extern __shared__ __align__(16) float few_shared[];
  float* ring = few_shared + (warp * kFewStages * kFewRows * 32 + lane) * 4;
  const float* rows[kFewRows];
  bool live[kFewRows];
#pragma unroll
  for (int r = 0; r < kFewRows; ++r) {
    const int n = row_of(r);
    live[r] = n < p.N;
    rows[r] = W + (live[r] ? static_cast<size_t>(n) * p.K : 0);
  }
  const int step = warps * 128;
  auto ask = [&](int stage, int k) {
#pragma unroll
    for (int r = 0; r < kFewRows; ++r) {
      const bool valid = live[r] && k < p.K;
      copy_16(shared_address(ring + (stage * kFewRows + r) * 128), rows[r] + (valid ? k : 0), valid);
    }
    copy_commit();
  };
  int k = member * 128 + lane * 4;
  pdl_launch_dependents();
#pragma unroll
  for (int stage = 0; stage < kFewStages - 1; ++stage) ask(stage, k + stage * step);
  pdl_wait();
  float acc[kFewRows * MR];
#pragma unroll
  for (int i = 0; i < kFewRows * MR; ++i) acc[i] = 0.0f;
  int stage = 0;
  for (int k0 = member * 128; k0 < p.K; k0 += step, k += step) {
    float4 a[MR];
#pragma unroll
    for (int m = 0; m < MR; ++m)
      a[m] = k < p.K && m < p.M ? *reinterpret_cast<const float4*>(A + static_cast<size_t>(m) * p.K + k) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    copy_wait<kFewStages - 2>();
    const int last = stage == 0 ? kFewStages - 1 : stage - 1;
    ask(last, k + (kFewStages - 1) * step);   // (the stage read out in the pass before)
#pragma unroll
    for (int r = 0; r < kFewRows; ++r) {
      const float4 w = *reinterpret_cast<const float4*>(ring + (stage * kFewRows + r) * 128);
#pragma unroll
      for (int m = 0; m < MR; ++m) {
        float& sum = acc[m * kFewRows + r];
        sum = fmaf(a[m].x, w.x, sum);
        sum = fmaf(a[m].y, w.y, sum);
        sum = fmaf(a[m].z, w.z, sum);
        sum = fmaf(a[m].w, w.w, sum);
      }
    }
    stage = stage == kFewStages - 1 ? 0 : stage + 1;
  }
  int held;
  const int first = sum_lanes<kFewRows * MR>(acc, lane, held);
#pragma unroll
  for (int i = 0; i < kFewRows * MR / 2; ++i)
    if (i < held) parts[warp][first + i] = acc[i];
  __syncthreads();
  auto total = [&](int own, int i) {   // value i of the block's group `own`, its warps in their order
    float sum = parts[own * warps][i];
    for (int o = 1; o < warps; ++o) sum += parts[own * warps + o][i];
    return sum;
  };
  auto store = [&](size_t at, float value) {
    if (p.out_bf16) static_cast<__nv_bfloat16*>(p.out)[at] = __float2bfloat16_rn(value);
    else static_cast<float*>(p.out)[at] = value;
  };
  const int per_group = (gated ? kFewRows / 2 : kFewRows) * MR;
  for (int i = threadIdx.x; i < kFewWarps / warps * per_group; i += kFewWarps * 32) {
    const int own = i / per_group, item = i % per_group;
    const int r = item % (per_group / MR), m = item / (per_group / MR);
    const int first_row = (blockIdx.x * (kFewWarps / warps) + own) * kFewRows;
    if (m >= p.M) continue;
    if (gated) {
      const int feature = first_row / 2 + r, n = feature / 16 * 32 + feature % 16;
      if (n + 16 >= p.N) continue;
      float gate = total(own, m * kFewRows + r), up = total(own, m * kFewRows + r + kFewRows / 2);
      if (p.bias) {
        gate += p.bias[n];
        up += p.bias[n + 16];
      }
      store(static_cast<size_t>(m) * (p.N / 2) + feature, up * gate_activation(gate, p.activation));
    } else {
      const int n = first_row + r;
      if (n >= p.N) continue;
      float value = total(own, m * kFewRows + r);
      if (p.bias) value += p.bias[n];
      const size_t at = static_cast<size_t>(m) * p.N + n;
      if (p.epilogue == EPI_STORE) store(at, value);
      else p.resid[at] += value;
    }
  }
}

template <int MR>
__global__ void __launch_bounds__(kFewWarps * 32, 2)
gemv_rows_shared_kernel(const GemmArgs p, int split) {
  constexpr int R = kFewRows;
  __shared__ float parts[kFewWarps][R * MR];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tile = static_cast<int>(blockIdx.x) / split, member = static_cast<int>(blockIdx.x) % split;
  const int group = tile * kFewWarps + warp;
  const float* A = static_cast<const float*>(p.A);
  const float* W = static_cast<const float*>(p.W);
  const bool gated = p.epilogue == EPI_SWIGLU;
  // the warp's rows: neighbours, or the gates and the ups of neighbouring features
  auto row_of = [&](int r) {
    if (!gated) return group * R + r;
    const int feature = group * (R / 2) + r % (R / 2);
    return feature / 16 * 32 + feature % 16 + (r >= R / 2 ? 16 : 0);
  };
  // A lane copies the 16 bytes of each row of W that it will use itself; the run of A is everyone's.
  extern __shared__ __align__(16) float few_shared[];
  float* ring = few_shared + (warp * kFewStages * R * 32 + lane) * 4;
  float* shared_rows = few_shared + kFewWarps * kFewStages * R * kFewRun;   // [stage][MR][run]
  const float* rows[R];
  bool live[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int n = row_of(r);
    live[r] = n < p.N;
    rows[r] = W + (live[r] ? static_cast<size_t>(n) * p.K : 0);
  }
  const int step = split * kFewRun;
  auto ask = [&](int stage, int k) {
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const bool valid = live[r] && k < p.K;
      copy_16(shared_address(ring + (stage * R + r) * kFewRun), rows[r] + (valid ? k : 0), valid);
    }
  };
  auto ask_a = [&](int stage, int k) {
    if (warp < MR) {
      const bool valid = warp < p.M && k < p.K;
      copy_16(shared_address(shared_rows + (stage * MR + warp) * kFewRun + lane * 4), A + (valid ? static_cast<size_t>(warp) * p.K + k : 0), valid);
    }
  };
  int k = member * kFewRun + lane * 4;
  pdl_launch_dependents();
#pragma unroll
  for (int stage = 0; stage < kFewStages - 1; ++stage) ask(stage, k + stage * step);
  pdl_wait();
#pragma unroll
  for (int stage = 0; stage < kFewStages - 1; ++stage) {
    ask_a(stage, k + stage * step);
    copy_commit();   // (with the first, all that was asked for before the wait)
  }
  float acc[R * MR];
#pragma unroll
  for (int i = 0; i < R * MR; ++i) acc[i] = 0.0f;
  int stage = 0;
  for (int k0 = member * kFewRun; k0 < p.K; k0 += step, k += step) {
    copy_wait<kFewStages - 2>();
    __syncthreads();   // this run of A is there, the one before is read out
    const int last = stage == 0 ? kFewStages - 1 : stage - 1;
    ask(last, k + (kFewStages - 1) * step);
    ask_a(last, k + (kFewStages - 1) * step);
    copy_commit();
    float4 a[MR];
#pragma unroll
    for (int m = 0; m < MR; ++m) a[m] = *reinterpret_cast<const float4*>(shared_rows + (stage * MR + m) * kFewRun + lane * 4);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const float4 w = *reinterpret_cast<const float4*>(ring + (stage * R + r) * kFewRun);
#pragma unroll
      for (int m = 0; m < MR; ++m) {
        float& sum = acc[m * R + r];
        sum = fmaf(a[m].x, w.x, sum);
        sum = fmaf(a[m].y, w.y, sum);
        sum = fmaf(a[m].z, w.z, sum);
        sum = fmaf(a[m].w, w.w, sum);
      }
    }
    stage = stage == kFewStages - 1 ? 0 : stage + 1;
  }
  int held;
  const int first = sum_lanes<R * MR>(acc, lane, held);
#pragma unroll
  for (int i = 0; i < R * MR / 2; ++i)
    if (i < held) parts[warp][first + i] = acc[i];
  if (split > 1) cluster_sync();
  else __syncthreads();
  auto total = [&](int own, int i) {   // value i of warp `own`, the cluster's blocks in their order
    if (split == 1) return parts[own][i];
    const uint32_t at = shared_address(&parts[own][i]);
    float each[kFewSplit];
#pragma unroll
    for (int o = 0; o < kFewSplit; ++o) each[o] = o < split ? remote_float(at, o) : 0.0f;
    float sum = each[0];
#pragma unroll
    for (int o = 1; o < kFewSplit; ++o)
      if (o < split) sum += each[o];
    return sum;
  };
  auto store = [&](size_t at, float value) {
    if (p.out_bf16) static_cast<__nv_bfloat16*>(p.out)[at] = __float2bfloat16_rn(value);
    else static_cast<float*>(p.out)[at] = value;
  };
  // the tile's outputs, row of A by row of A, an even share a block
  const int columns = kFewWarps * (gated ? R / 2 : R), items = columns * MR, share = (items + split - 1) / split;
  for (int i = member * share + static_cast<int>(threadIdx.x); i < min(items, (member + 1) * share); i += kFewWarps * 32) {
    const int m = i / columns, column = i % columns;
    if (m >= p.M) break;
    if (gated) {
      const int own = column / (R / 2), r = column % (R / 2);
      const int feature = tile * columns + column, n = feature / 16 * 32 + feature % 16;
      if (n + 16 >= p.N) continue;
      float gate = total(own, m * R + r), up = total(own, m * R + r + R / 2);
      if (p.bias) {
        gate += p.bias[n];
        up += p.bias[n + 16];
      }
      store(static_cast<size_t>(m) * (p.N / 2) + feature, up * gate_activation(gate, p.activation));
    } else {
      const int n = tile * columns + column;
      if (n >= p.N) continue;
      float value = total(column / R, m * R + column % R);
      if (p.bias) value += p.bias[n];
      const size_t at = static_cast<size_t>(m) * p.N + n;
      if (p.epilogue == EPI_STORE) store(at, value);
      else p.resid[at] += value;
    }
  }
  if (split > 1) cluster_sync();   // no block leaves while another reads its sums
}

template <int MR>
static int launch_few_rows(const GemmArgs& p, int members, cudaStream_t s) {
  constexpr int kBytes = kFewWarps * kFewStages * kFewRows * kFewRun * 4;
  static SharedMemoryOptIn opt_in;
  const int opted = opt_in.ask(reinterpret_cast<const void*>(gemv_rows_kernel<MR>), kBytes);
  const long long groups = (p.N + kFewRows - 1) / kFewRows;
  const dim3 grid(static_cast<unsigned>((groups * members + kFewWarps - 1) / kFewWarps));
  return opted ? opted : vipera_launch(gemv_rows_kernel<MR>, grid, dim3(kFewWarps * 32), kBytes, s, p, members);
}

template <int MR>
static int launch_few_shared(const GemmArgs& p, int members, cudaStream_t s) {
  constexpr int kBytes = (kFewWarps * kFewRows + MR) * kFewStages * kFewRun * 4;
  static SharedMemoryOptIn opt_in;
  const int opted = opt_in.ask(reinterpret_cast<const void*>(gemv_rows_shared_kernel<MR>), kBytes);
  const long long tiles = (static_cast<long long>(p.N) + kFewWarps * kFewRows - 1) / (kFewWarps * kFewRows);
  return opted ? opted : launch_in_clusters(gemv_rows_shared_kernel<MR>, members, dim3(static_cast<unsigned>(tiles * members)), dim3(kFewWarps * 32), kBytes, s, p, members);
}

static int launch_few(const GemmArgs& p, cudaStream_t s) {
  constexpr int kWarpsWanted = 148 * 12;
  const long long groups = (p.N + kFewRows - 1) / kFewRows;
  int members = 1;
  while (members < kFewSplit && groups * members < kWarpsWanted) members *= 2;
  if (p.M == 1) return launch_few_rows<1>(p, members, s);
  if (p.M == 2) return launch_few_rows<2>(p, members, s);
  const bool large = static_cast<long long>(p.N) * p.K >= kSharedFrom;
  const int runs = p.K / (kFewRun * members);
  if (p.M <= 4) return members == 1 && large && runs >= kSharedRunsFour ? launch_few_shared<4>(p, members, s) : launch_few_rows<4>(p, members, s);
  return large && (members == 1 || runs >= kSharedRuns) ? launch_few_shared<8>(p, members, s) : launch_few_rows<8>(p, members, s);
}

template <typename TA, typename TW, typename T, bool DIRECT, bool CLUSTER>
static int launch_form(const GemmArgs& p, cudaStream_t s) {
  auto kernel = gemm_simt_kernel<TA, TW, T, DIRECT, CLUSTER>;
  static SharedMemoryOptIn opt_in;   // one per form of the kernel
  const int opted = opt_in.ask(reinterpret_cast<const void*>(kernel), T::kSharedBytes);
  if (opted) return opted;
  const unsigned tiles_n = (p.N + T::BN - 1) / T::BN, tiles_m = (p.M + T::BM - 1) / T::BM;
  if (tiles_m > 65535u) return VIPERA_BAD_SHAPE;
  const int chunks = ((CLUSTER ? p.slab : p.K) + kChunk - 1) / kChunk;
  const int bytes = T::kSharedBytes - (chunks < T::STAGES ? T::STAGES - chunks : 0) * T::kStageFloats * 4;
  return launch_in_clusters(kernel, CLUSTER ? kSlabs : 1, dim3(CLUSTER ? tiles_n * kSlabs : tiles_n, tiles_m), dim3(T::kThreads), bytes, s, p);
}

// A tile's slabs go to a cluster where whole tiles would leave much of the chip idle: fewer small tiles
// than multiprocessors, or a last wave that is mostly empty for the large ones (a block a multiprocessor).  The tiles
// of rows that are staged through registers go to clusters up to a count that grows with K: in bfloat16, whole / cluster, 140
// tiles of K = 896: 51.5 / 55.6 us, 70: 51.5 / 33.5; 320 of 2,048: 217 / 202, 512: 305 / 316; 64 of 300: 26.9 / 20.7.
// (Tiles of 64 x 128 took 78.7, 47.4, 283, 338 and 20.6 us there, tiles of 64 x 64 with one chain over K
// 72, 72, 313, 419 and 24.9.)
template <typename TA, typename TW, typename T, bool DIRECT>
static int launch_tile(const GemmArgs& p, cudaStream_t s) {
  constexpr long long kSms = 148;
  const long long tiles = static_cast<long long>((p.N + T::BN - 1) / T::BN) * ((p.M + T::BM - 1) / T::BM);
  bool cluster;
  if (T::BM <= 32) cluster = tiles < kSms;
  else if (!DIRECT) cluster = tiles <= (p.K / 6 > 80 ? p.K / 6 : 80);
  else cluster = tiles * 5 < (tiles + kSms - 1) / kSms * kSms * 4;
  // a slab of less than three chunks is all start and ending
  if (cluster && (p.slab >= 3 * kChunk || (T::BM > 32 && !DIRECT))) return launch_form<TA, TW, T, DIRECT, true>(p, s);
  return launch_form<TA, TW, T, DIRECT, false>(p, s);
}

// A short inner size: the trip to memory and the output's stores bound the product, and what the forms of long K keep for
// it (rings, slabs, tensor memory) only delays the start.  A block takes 32 rows and 128 columns with all of K in shared
// memory, a thread four rows and four columns a warp apart; a sum has two chains, even and odd places.  VEC: rows of whole
// pieces of four values.  Tiles through slabs or the tensor cores / this: bfloat16, 300 rows, W 256 x 100: 24.9 / 10.6 us, W 512
// x 256: 31.0 / 18.7; 32-bit, 300 rows, W 128 x 128: 18.7 / 8.5.
constexpr int kShortRows = 32, kShortColumns = 128, kShortThreads = 256;
constexpr int kShortInner = 320, kShortInnerParts = 128;   // the longest K, and where the tensor cores could take over

__device__ __forceinline__ float4 load_four(const float* src) { return *reinterpret_cast<const float4*>(src); }
__device__ __forceinline__ float4 load_four(const __nv_bfloat16* src) {
  const uint2 raw = *reinterpret_cast<const uint2*>(src);
  const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x));
  const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
  return make_float4(a.x, a.y, b.x, b.y);
}
// fours of a row in shared memory: odd, so that neighbouring rows' 16-byte reads meet no bank twice
__host__ __device__ __forceinline__ int short_pitch(int K) { return ((K + 3) / 4) | 1; }

// `rows` rows from row0 on; zeros outside.
template <typename T, bool VEC>
__device__ __forceinline__ void stage_short(float4* dst, int pitch, const T* __restrict__ src, int row0, int extent, int rows, int K) {
  const int pieces = (K + 3) / 4;
#pragma unroll 8
  for (int i = threadIdx.x; i < rows * pieces; i += kShortThreads) {
    const int r = i / pieces, c = i - r * pieces;
    float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (row0 + r < extent) {
      const T* at = src + static_cast<size_t>(row0 + r) * K + 4 * c;
      if (VEC) {
        v = load_four(at);
      } else {
        v.x = to_float<T>(at[0]);
        if (4 * c + 1 < K) v.y = to_float<T>(at[1]);
        if (4 * c + 2 < K) v.z = to_float<T>(at[2]);
        if (4 * c + 3 < K) v.w = to_float<T>(at[3]);
      }
    }
    dst[r * pitch + c] = v;
  }
}

template <typename TA, typename TW, bool VEC>
__global__ void __launch_bounds__(kShortThreads)
gemm_short_kernel(const GemmArgs p) {
  extern __shared__ float4 short_shared[];
  pdl_launch_dependents();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, m0 = blockIdx.y * kShortRows, n0 = blockIdx.x * kShortColumns;
  const int pitch = short_pitch(p.K), pieces = (p.K + 3) / 4;
  float4* w_s = short_shared;                       // [kShortColumns][pitch]
  float4* a_s = w_s + kShortColumns * pitch;        // [kShortRows][pitch]
  stage_short<TW, VEC>(w_s, pitch, static_cast<const TW*>(p.W), n0, p.N, kShortColumns, p.K);
  pdl_wait();
  stage_short<TA, VEC>(a_s, pitch, static_cast<const TA*>(p.A), m0, p.M, min(kShortRows, p.M - m0), p.K);
  __syncthreads();
  if (m0 + warp * 4 >= p.M) return;
  unsigned long long sums[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) sums[i][j] = 0ull;
  for (int c = 0; c < pieces; ++c) {   // (rows of A that do not exist: whatever lies there, never stored)
    ulonglong2 w[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) w[j] = *reinterpret_cast<const ulonglong2*>(w_s + (lane + 32 * j) * pitch + c);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(a_s + (warp * 4 + i) * pitch + c);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        fma_pair(sums[i][j], a.x, w[j].x);
        fma_pair(sums[i][j], a.y, w[j].y);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int m = m0 + warp * 4 + i, n = n0 + lane + 32 * j;
      float value = sum_of_pair(sums[i][j]) + (p.bias && n < p.N ? p.bias[n] : 0.0f);
      int column = n, columns = p.N;
      if (p.epilogue == EPI_SWIGLU) {   // the feature's up value is 16 columns, and lanes, further
        const float up = __shfl_down_sync(0xffffffffu, value, 16);
        value = up * gate_activation(value, p.activation);
        column = n / 32 * 16 + n % 32, columns = p.N / 2;
        if (lane >= 16) continue;
      }
      if (m >= p.M || n >= p.N) continue;
      const size_t at = static_cast<size_t>(m) * columns + column;
      if (p.epilogue == EPI_RESIDUAL) p.resid[at] += value;
      else if (p.out_bf16) static_cast<__nv_bfloat16*>(p.out)[at] = __float2bfloat16_rn(value);
      else static_cast<float*>(p.out)[at] = value;
    }
}

template <typename TA, typename TW, bool VEC>
static int launch_short(const GemmArgs& p, cudaStream_t s) {
  constexpr int kRowsHeld = kShortColumns + kShortRows;
  static SharedMemoryOptIn opt_in;
  const int opted = opt_in.ask(reinterpret_cast<const void*>(gemm_short_kernel<TA, TW, VEC>), kRowsHeld * ((kShortInner / 4) | 1) * 16);
  if (opted) return opted;
  const dim3 grid(static_cast<unsigned>((p.N + kShortColumns - 1) / kShortColumns), static_cast<unsigned>((p.M + kShortRows - 1) / kShortRows));
  return vipera_launch(gemm_short_kernel<TA, TW, VEC>, grid, dim3(kShortThreads), kRowsHeld * short_pitch(p.K) * 16, s, p);
}

template <typename TA, typename TW>
static int launch_sizes(const GemmArgs& p, cudaStream_t s) {
  constexpr bool kBothFloat = sizeof(TA) == 4 && sizeof(TW) == 4;
  const bool direct = kBothFloat && p.K % 4 == 0 && ((reinterpret_cast<uintptr_t>(p.A) | reinterpret_cast<uintptr_t>(p.W)) & 15) == 0;
  const bool parts = direct && p.M > TileMid::BM;   // many rows: three parts of every number on the tensor cores
  if (p.K <= (parts ? kShortInnerParts : kShortInner) && (p.M > kFewRows || !direct) && (p.M + kShortRows - 1) / kShortRows <= 65535) {
    const bool vec = p.K % 4 == 0 && reinterpret_cast<uintptr_t>(p.A) % (4 * sizeof(TA)) == 0 &&
                     reinterpret_cast<uintptr_t>(p.W) % (4 * sizeof(TW)) == 0;
    return vec ? launch_short<TA, TW, true>(p, s) : launch_short<TA, TW, false>(p, s);
  }
  if constexpr (kBothFloat) {
    if (direct) {
      if (p.M <= kFewRows) return launch_few(p, s);
      if (p.M <= TileSome::BM) return launch_tile<TA, TW, TileSome, true>(p, s);
      if (p.M <= TileMid::BM) return launch_tile<TA, TW, TileMid, true>(p, s);
      if (p.status)
        return gemm_split::launch({static_cast<const float*>(p.A), static_cast<const float*>(p.W), p.M, p.N, p.K, 1, 0, 1, p.bias, p.out,
                                   p.resid, p.activation, p.epilogue, p.out_bf16, p.status,
                                   static_cast<uint8_t*>(p.parts), nullptr, p.parts_bytes}, s);
      return VIPERA_BAD_ARGUMENT;
    }
  }
  // rows that do not start on 16 bytes, or values that are widened on the way
  if (p.M <= TileMid::BM) return launch_tile<TA, TW, TileSome, false>(p, s);
  return launch_tile<TA, TW, TileLow, false>(p, s);
}

template <typename TA, typename TW>
static int launch_typed(const TA* A, const TW* W, int M, int N, int K, int epilogue, const float* bias,
                        void* out, int out_dtype, float* resid, int activation, int* status, void* parts, long long parts_bytes, cudaStream_t s) {
  const int slab = ((K + kSlabs - 1) / kSlabs + kChunk - 1) / kChunk * kChunk;
  if (epilogue != EPI_STORE && epilogue != EPI_RESIDUAL && epilogue != EPI_SWIGLU) return VIPERA_BAD_ARGUMENT;
  if (epilogue == EPI_RESIDUAL ? !resid : !out) return VIPERA_BAD_ARGUMENT;
  if (epilogue == EPI_SWIGLU && N % 32 != 0) return VIPERA_BAD_SHAPE;  // gate/up groups of 16 must pair up
  if (epilogue != EPI_RESIDUAL && out_dtype != VIPERA_F32 && out_dtype != VIPERA_BF16) return VIPERA_BAD_DTYPE;
  const int wide = K % 8 == 0 && ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(W)) & 15) == 0;
  const GemmArgs p{A, W, M, N, K, slab, bias, out, resid, activation, epilogue, out_dtype == VIPERA_BF16, wide, status, parts, parts_bytes};
  return launch_sizes<TA, TW>(p, s);
}

// A is [M, K] and W is [N, K], both row-major and contiguous.  For SWIGLU, N counts the
// interleaved gate and up rows (twice the intermediate size) and out is [M, N/2].
static int run_simt(const void* A, int a_dtype, const void* W, int w_dtype, int M, int N, int K, int epilogue,
                    const float* bias, void* out, int out_dtype, float* resid, int activation, int* status, void* parts,
                    long long parts_bytes, void* stream) {
  if (M <= 0) return VIPERA_OK;
  if (N <= 0 || K <= 0) return VIPERA_BAD_SHAPE;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (a_dtype == VIPERA_F32 && w_dtype == VIPERA_F32)
    return launch_typed(static_cast<const float*>(A), static_cast<const float*>(W), M, N, K, epilogue, bias, out, out_dtype, resid, activation, status,
                        parts, parts_bytes, s);
  if (a_dtype == VIPERA_BF16 && w_dtype == VIPERA_BF16)
    return launch_typed(static_cast<const __nv_bfloat16*>(A), static_cast<const __nv_bfloat16*>(W), M, N, K, epilogue, bias, out, out_dtype, resid, activation, status,
                        parts, parts_bytes, s);
  if (a_dtype == VIPERA_F32 && w_dtype == VIPERA_BF16)
    return launch_typed(static_cast<const float*>(A), static_cast<const __nv_bfloat16*>(W), M, N, K, epilogue, bias, out, out_dtype, resid, activation, status,
                        parts, parts_bytes, s);
  return VIPERA_BAD_DTYPE;
}

// A bias counts in every ending; `activation` is the gated unit's (ACT_SILU, ACT_GELU_TANH).  `status`: a device word that must
// be 0 before the launch and is not afterwards where a bounded wait ran out; only 32-bit products of more than 64 rows need it.
// `parts`: room of vipera_gemm_simt_parts bytes (16-byte aligned), or null.
VIPERA_API int vipera_gemm_simt_status(const void* A, int a_dtype, const void* W, int w_dtype, int M, int N, int K,
                                       int epilogue, const float* bias, void* out, int out_dtype, float* resid,
                                       int activation, int* status, void* parts, long long parts_bytes, void* stream) {
  if (activation != ACT_SILU && activation != ACT_GELU_TANH) return VIPERA_BAD_ARGUMENT;
  return run_simt(A, a_dtype, W, w_dtype, M, N, K, epilogue, bias, out, out_dtype, resid, activation, status, parts,
                  parts_bytes, stream);
}

// The bytes that 32-bit products of such sizes want for the parts of their left operand (0: none).
VIPERA_API int vipera_gemm_simt_parts(int M, int N, int K) { return K <= kShortInnerParts ? 0 : gemm_split::parts_bytes(M, N, K); }

VIPERA_API const char* vipera_gemm_simt_status_text(int status) { return vipera_status_text(status); }
