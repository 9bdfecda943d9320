// The cell's portions as a walk whose blocks keep their part of the state in registers, with all that does not depend on the
// state computed ahead of it (bfloat16 runs; included by mlstm.cu, whose names it uses).
//
//   1. mlstm_prepare_kernel, a block per (head, chunk of 64 tokens): q and k rounded to bfloat16, the chunk's weights
//      w_ts = (q_t . k_s) exp(a_s - top_t) with top_t = max_(s <= t) a_s, their row sums, the chunk's own part of n, its A and B;
//   2. mlstm_nm_kernel, a block per (head, request): n and m at the start of every chunk;
//   3. mlstm_factors_kernel, a block per (head, chunk, 128 value columns): q . n, the denominators, and what the two parts of
//      an output are multiplied by, exp(m_0 - M_t) and exp(top_t - M_t), each over the denominator; v in bfloat16, as it is
//      and as it enters the state;
//   4. mlstm_walk_kernel, a block per (32 value columns, head, request): chunk by chunk
//        o^T = f (S^T q^T) + f' (v^T w^T),  S^T = keep S^T + (v exp(a - M_L))^T k
//      A warp has 16 columns and a quarter of the channels of S^T as the accumulators of its update product.  What they hold is
//      laid out as the left operand of the next chunk's S^T q^T wants it, so the state never leaves the registers (it enters
//      that product rounded to bfloat16, as in the other forms); the four quarters' outputs are added in shared memory.
//
// What a block reads of a chunk lies in memory as it lies in shared memory, rows padded by 16 bytes, and comes as five bulk
// copies, two chunks ahead.
//
// What bounds the walk: a chunk's 72 products of 16 x 8 x 16 a warp and their fragments, two warps a scheduler, and two
// barriers; 2.2 us a chunk at 256 channels (3.2 where blocks brought q, k and v themselves and converted v).  2,048 tokens, 8
// heads of 256 x 512: prepare 15, n and m 8, factors 22, walk 73, ending 24 us; all chunks at once, through the states of 32
// bits at every chunk's start: 60, 62, 151 and 27 us.
#pragma once

constexpr int kWalkCols = 32, kWalkThreads = 256;

// What is prepared of a (chunk, head), in bytes.
template <int D>
struct WalkLayout {
  static constexpr int kQS = D + 8, kWS = kTcChunk + 8, kVS = kWalkCols + 8, kOS = kTcChunk + 4;
  static constexpr int kRows = kTcChunk * kQS * 2;                   // q, or k
  static constexpr int kWeights = kTcChunk * kWS * 2;
  static constexpr int kValues = 2 * kTcChunk * kVS * 2;             // 32 columns of v, and the same as they enter the state
  static constexpr int kFactors = (2 * kTcChunk + 4) * 4;            // f, f', keep
  static constexpr int kStage = 2 * kRows + kWeights + kValues + kFactors;
  static constexpr int kBytes = 2 * kStage + 8 * 16 * kOS * 4;
  static_assert(kRows % 16 == 0 && kWeights % 16 == 0 && kValues % 16 == 0 && kFactors % 16 == 0, "whole bulk copies");
};
struct WalkBuffers {
  __nv_bfloat16* q;      // [jobs, heads, 64, d + 8]
  __nv_bfloat16* k;
  __nv_bfloat16* w;      // [jobs, heads, 64, 72]
  __nv_bfloat16* v;      // [jobs, heads, vdim / 32, 2, 64, 40]
  float* token;          // [jobs, heads, 4, 64]: a, b, top, row sum
  float* factors;        // [jobs, heads, 132]
  int* status;
};
enum { WALK_A, WALK_B, WALK_TOP, WALK_SUM, WALK_ROWS };
enum { WALK_WAIT_EXPIRED = 7 };

template <int D>
struct PrepareLayout {
  static constexpr int kQS = D + 8, kWS = kTcChunk + 8;
  static constexpr size_t kBytes = (2 * static_cast<size_t>(kTcChunk) * kQS + kTcChunk * kWS) * 2 + (7 * kTcChunk + 8) * 4;
};

template <int D>
__global__ void __launch_bounds__(kTcThreads)
mlstm_prepare_kernel(const MlstmParams p, const WalkBuffers buffers) {
  constexpr int L = kTcChunk, QS = PrepareLayout<D>::kQS, WS = PrepareLayout<D>::kWS;
  pdl_launch_dependents();
  int e, chunk;
  const int h = blockIdx.x, job = blockIdx.y;
  if (!find_job(p, job, &e, &chunk)) return;   // (the step's requests are the host's, written before the step)
  pdl_wait();
  extern __shared__ __align__(16) unsigned char raw[];
  __nv_bfloat16* Qs = reinterpret_cast<__nv_bfloat16*>(raw);   // [L][QS]
  __nv_bfloat16* Ks = Qs + L * QS;
  __nv_bfloat16* Ws = Ks + L * QS;                             // [L][WS]
  float* lis = reinterpret_cast<float*>(Ws + L * WS);
  float* lfs = lis + L;
  float* av = lfs + L;
  float* bv = av + L;
  float* tops = bv + L;
  float* rs = tops + L;      // [2][L]
  float* scal = rs + 2 * L;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, tq = lane & 3, rm = warp & 3, cn = warp >> 2;
  const int t0 = p.entry_starts[e], count = p.entry_starts[e + 1] - t0, start = chunk * L, len = min(L, count - start);
  const float* rows = p.proj + static_cast<size_t>(t0 + start) * p.proj_width;
  const size_t at = static_cast<size_t>(job) * p.heads + h;
#pragma unroll 4
  for (int item = tid; item < L * (D / 8); item += kTcThreads) {
    const int t = item / (D / 8), dd = (item % (D / 8)) * 8;
    float4 q[2], k[2];
    q[0] = q[1] = k[0] = k[1] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (t < len) {
      const float* row = rows + static_cast<size_t>(t) * p.proj_width + h * D + dd;
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        q[i] = *reinterpret_cast<const float4*>(row + p.q_off + 4 * i);
        k[i] = *reinterpret_cast<const float4*>(row + p.k_off + 4 * i);
      }
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      store_four(Qs + t * QS + dd + 4 * i, make_float4(q[i].x * p.q_scale, q[i].y * p.q_scale, q[i].z * p.q_scale, q[i].w * p.q_scale));
      store_four(Ks + t * QS + dd + 4 * i, k[i]);
    }
    const size_t to = (at * L + t) * QS + dd;
    *reinterpret_cast<uint4*>(buffers.q + to) = *reinterpret_cast<const uint4*>(Qs + t * QS + dd);
    *reinterpret_cast<uint4*>(buffers.k + to) = *reinterpret_cast<const uint4*>(Ks + t * QS + dd);
  }
  if (tid < L) {
    float li = 0.0f, lf = 0.0f;
    if (tid < len) {
      const float* row = rows + static_cast<size_t>(tid) * p.proj_width;
      li = capped(row[p.i_off + h], p.gate_cap);
      lf = log_sigmoid(capped(row[p.f_off + h], p.gate_cap));
    }
    lis[tid] = li;
    lfs[tid] = lf;
  }
  __syncthreads();
  if (warp == 0) {
    // two tokens a lane: b, a = li - b, the running maxima of a; the largest; the sum of the log forget gates
    const float first = lfs[2 * lane], second = lfs[2 * lane + 1], pair = first + second;
    float before = pair;
#pragma unroll
    for (int offset = 1; offset < 32; offset <<= 1) {
      const float other = __shfl_up_sync(0xffffffffu, before, offset);
      if (lane >= offset) before += other;
    }
    const float b0 = before - pair + first, b1 = before;
    const float a0 = 2 * lane < len ? lis[2 * lane] - b0 : -INFINITY, a1 = 2 * lane + 1 < len ? lis[2 * lane + 1] - b1 : -INFINITY;
    float scan = fmaxf(a0, a1);
#pragma unroll
    for (int offset = 1; offset < 32; offset <<= 1) {
      const float other = __shfl_up_sync(0xffffffffu, scan, offset);
      if (lane >= offset) scan = fmaxf(scan, other);
    }
    float earlier = __shfl_up_sync(0xffffffffu, scan, 1);
    if (lane == 0) earlier = -INFINITY;
    av[2 * lane] = a0, av[2 * lane + 1] = a1;
    bv[2 * lane] = b0, bv[2 * lane + 1] = b1;
    tops[2 * lane] = fmaxf(earlier, a0), tops[2 * lane + 1] = scan;
    const float most = __shfl_sync(0xffffffffu, scan, 31);
    lis[2 * lane] = expf(a0 - most), lis[2 * lane + 1] = expf(a1 - most);   // what a token enters the chunk's own n with
    if (lane == 31) scal[0] = scan, scal[1] = before;
  }
  __syncthreads();
  {
    float G[4][4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int i = 0; i < 4; ++i) G[j][i] = 0.0f;
#pragma unroll 4
    for (int kk = 0; kk < D / 16; ++kk) {
      uint32_t a[4], b[4];
      left(a, Qs, QS, rm * 16, kk * 16, lane);
#pragma unroll
      for (int j = 0; j < 4; j += 2) {
        right(b, Ks, QS, cn * 32 + j * 8, kk * 16, lane);
        mma_bf16(G[j], a, b[0], b[1]);
        mma_bf16(G[j + 1], a, b[2], b[3]);
      }
    }
    float sums[2] = {0.0f, 0.0f};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const int t = rm * 16 + g + 8 * r, s0 = cn * 32 + j * 8 + 2 * tq;
        float w[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          w[i] = s0 + i <= t && t < len ? G[j][2 * r + i] * expf(av[s0 + i] - tops[t]) : 0.0f;
          sums[r] += w[i];
        }
        *reinterpret_cast<__nv_bfloat162*>(Ws + t * WS + s0) = __floats2bfloat162_rn(w[0], w[1]);
      }
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      sums[r] += __shfl_xor_sync(0xffffffffu, sums[r], 1);
      sums[r] += __shfl_xor_sync(0xffffffffu, sums[r], 2);
      if (tq == 0) rs[cn * L + rm * 16 + g + 8 * r] = sums[r];
    }
  }
  // the chunk's own part of n
  if (tid < D) {
    float acc = 0.0f;
    for (int t = 0; t < len; ++t) acc = fmaf(lis[t], __bfloat162float(Ks[t * QS + tid]), acc);
    p.chunk_n[at * D + tid] = acc;
  }
  __syncthreads();
  for (int item = tid; item < L * (L / 8); item += kTcThreads)
    *reinterpret_cast<uint4*>(buffers.w + at * L * WS + item / (L / 8) * WS + item % (L / 8) * 8) = *reinterpret_cast<const uint4*>(Ws + item / (L / 8) * WS + item % (L / 8) * 8);
  float* token = buffers.token + at * WALK_ROWS * L;
  if (tid < L) {
    token[WALK_A * L + tid] = av[tid];
    token[WALK_B * L + tid] = bv[tid];
    token[WALK_TOP * L + tid] = tops[tid];
    token[WALK_SUM * L + tid] = rs[tid] + rs[L + tid];
  }
  if (tid == 0) {
    p.chunk_aux[at * 4] = scal[0];
    p.chunk_aux[at * 4 + 1] = scal[1];
  }
}

// n and m at the start of every chunk take the place of the chunk's own n and join its A and B; the last ones go to the scratch row.
__global__ void __launch_bounds__(256)
mlstm_nm_kernel(const MlstmParams p) {
  pdl_launch_dependents();
  pdl_wait();
  const int h = blockIdx.x, e = blockIdx.y, d = p.dim, dd = threadIdx.x;
  const int count = p.entry_starts[e + 1] - p.entry_starts[e];
  if (count <= 0) return;
  const int chunks = (count + kTcChunk - 1) / kTcChunk;
  int job0 = 0;
  for (int other = 0; other < e; ++other) job0 += (p.entry_starts[other + 1] - p.entry_starts[other] + kTcChunk - 1) / kTcChunk;
  const float* state = p.state + static_cast<long long>(p.state_slots[e]) * p.state_stride + static_cast<size_t>(p.heads) * d * p.vdim;
  const bool fresh = p.fresh[e] != 0;
  float m = fresh ? 0.0f : state[static_cast<size_t>(p.heads) * d + h];
  float n = fresh || dd >= d ? 0.0f : state[static_cast<size_t>(h) * d + dd];
  constexpr int kAhead = 8;
  for (int c0 = 0; c0 < chunks; c0 += kAhead) {
    float own[kAhead], tops[kAhead], sums[kAhead];
#pragma unroll
    for (int j = 0; j < kAhead; ++j) {
      const size_t at = static_cast<size_t>(job0 + min(c0 + j, chunks - 1)) * p.heads + h;
      own[j] = dd < d ? p.chunk_n[at * d + dd] : 0.0f;
      tops[j] = p.chunk_aux[at * 4];
      sums[j] = p.chunk_aux[at * 4 + 1];
    }
#pragma unroll
    for (int j = 0; j < kAhead; ++j) {
      if (c0 + j >= chunks) break;
      const size_t at = static_cast<size_t>(job0 + c0 + j) * p.heads + h;
      const float M = fmaxf(m, tops[j]), keep = expf(m - M), take = expf(tops[j] - M);
      if (dd < d) p.chunk_n[at * d + dd] = n;
      if (dd == 0) {
        p.chunk_aux[at * 4 + 2] = m;
        p.chunk_aux[at * 4 + 3] = keep;
      }
      n = keep * n + take * own[j];
      m = sums[j] + M;
    }
  }
  float* scratch = p.nm_scratch + (static_cast<size_t>(e) * p.heads + h) * (d + 1);
  if (dd < d) scratch[dd] = n;
  if (dd == 0) scratch[d] = m;
}

// What a token's two parts of the output are multiplied by, and the values, as they are and as they enter the state.
constexpr int kFactorCols = 128;

template <int D>
__global__ void __launch_bounds__(256)
mlstm_factors_kernel(const MlstmParams p, const WalkBuffers buffers) {
  using Layout = WalkLayout<D>;
  constexpr int L = kTcChunk, VS = Layout::kVS;
  __shared__ float enters[L];
  pdl_launch_dependents();
  int e, chunk;
  const int h = blockIdx.x, job = blockIdx.y, c0 = blockIdx.z * kFactorCols, cols = min(kFactorCols, p.vdim - c0);
  if (!find_job(p, job, &e, &chunk)) return;
  pdl_wait();
  const size_t at = static_cast<size_t>(job) * p.heads + h;
  const int t0 = p.entry_starts[e], count = p.entry_starts[e + 1] - t0, len = min(L, count - chunk * L);
  const float* token = buffers.token + at * WALK_ROWS * L;
  const float A = p.chunk_aux[at * 4], m0 = p.chunk_aux[at * 4 + 2];
  if (threadIdx.x < L) enters[threadIdx.x] = expf(token[WALK_A * L + threadIdx.x] - fmaxf(m0, A));   // (0 behind the last token)
  if (blockIdx.z == 0) {
    const int t = threadIdx.x >> 2, part = threadIdx.x & 3;
    const __nv_bfloat16* q = buffers.q + (at * L + t) * Layout::kQS;
    const float* n = p.chunk_n + at * D;
    float qn = 0.0f;
#pragma unroll
    for (int i = 0; i < D / 32; ++i) {
      const int dd = (i * 4 + part) * 8;
      const uint4 packed = *reinterpret_cast<const uint4*>(q + dd);
      const __nv_bfloat162* pairs = reinterpret_cast<const __nv_bfloat162*>(&packed);
      const float4 lo = *reinterpret_cast<const float4*>(n + dd), hi = *reinterpret_cast<const float4*>(n + dd + 4);
      const float values[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        qn = fmaf(__low2float(pairs[j]), values[2 * j], qn);
        qn = fmaf(__high2float(pairs[j]), values[2 * j + 1], qn);
      }
    }
    qn += __shfl_xor_sync(0xffffffffu, qn, 1);
    qn += __shfl_xor_sync(0xffffffffu, qn, 2);
    if (part == 0) {
      const float top = token[WALK_TOP * L + t], M = fmaxf(m0, top);
      const float inter = expf(m0 - M), own = expf(top - M);
      const float total = own * token[WALK_SUM * L + t] + inter * qn;
      const float denominator = fmaxf(fabsf(total), expf(-(token[WALK_B * L + t] + M))) + p.denom_eps;
      float* factors = buffers.factors + at * (Layout::kFactors / 4);
      factors[t] = inter / denominator;
      factors[L + t] = own / denominator;
      if (t == 0) factors[2 * L] = p.chunk_aux[at * 4 + 3];
    }
  }
  __syncthreads();
  const float* rows = p.proj + static_cast<size_t>(t0 + chunk * L) * p.proj_width + p.v_off + h * p.vdim + c0;
  __nv_bfloat16* to = buffers.v + (at * (p.vdim / kWalkCols) + c0 / kWalkCols) * (2 * L * VS);
#pragma unroll 4
  for (int item = threadIdx.x; item < L * (cols / 4); item += 256) {
    const int t = item / (cols / 4), c = item % (cols / 4) * 4;
    float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (t < len) v = *reinterpret_cast<const float4*>(rows + static_cast<size_t>(t) * p.proj_width + c);
    __nv_bfloat16* tile = to + c / kWalkCols * (2 * L * VS) + t * VS + c % kWalkCols;
    const float f = enters[t];
    store_four(tile, v);
    store_four(tile + L * VS, make_float4(v.x * f, v.y * f, v.z * f, v.w * f));
  }
}

template <int D>
__global__ void __launch_bounds__(kWalkThreads, 1)
mlstm_walk_kernel(const MlstmParams p, const WalkBuffers buffers) {
  using Layout = WalkLayout<D>;
  constexpr int L = kTcChunk, QS = Layout::kQS, WS = Layout::kWS, VS = Layout::kVS, OS = Layout::kOS;
  constexpr int kQuarter = D / 4, kSteps = kQuarter / 16, kTiles = kQuarter / 8;   // of the channels of a warp
  pdl_launch_dependents();
  const int h = blockIdx.y, e = blockIdx.z, c0 = blockIdx.x * kWalkCols, dv = p.vdim;
  const int t0 = p.entry_starts[e], count = p.entry_starts[e + 1] - t0;
  if (count <= 0) return;
  const int chunks = (count + L - 1) / L;
  int job0 = 0;
  for (int other = 0; other < e; ++other) job0 += (p.entry_starts[other + 1] - p.entry_starts[other] + L - 1) / L;
  extern __shared__ __align__(16) unsigned char raw[];
  __shared__ uint64_t full[2];
  __shared__ int gave_up;
  volatile int* abort_flag = &gave_up;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, tq = lane & 3;
  const int group = warp & 1, quarter = warp >> 1;   // sixteen columns, a quarter of the channels
  float* Os = reinterpret_cast<float*>(raw + 2 * Layout::kStage);   // [group][quarter][16 columns][OS]
  if (tid == 0) {
    for (int i = 0; i < 2; ++i) tcgen05::bar_init(&full[i], 1);
    gave_up = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\nfence.proxy.async.shared::cta;" ::: "memory");
  }
  auto bring = [&](int chunk) {   // by one thread
    const size_t at = static_cast<size_t>(job0 + chunk) * p.heads + h;
    uint64_t* bar = &full[chunk & 1];
    uint32_t to = shared_address(raw + (chunk & 1) * Layout::kStage);
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(shared_address(bar)), "r"(Layout::kStage) : "memory");
    auto copy = [&](const void* from, int bytes) {
      asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                   ::"r"(to), "l"(from), "r"(bytes), "r"(shared_address(bar)) : "memory");
      to += bytes;
    };
    copy(buffers.q + at * (L * QS), Layout::kRows);
    copy(buffers.k + at * (L * QS), Layout::kRows);
    copy(buffers.w + at * (L * WS), Layout::kWeights);
    copy(buffers.v + (at * (dv / kWalkCols) + blockIdx.x) * (2 * L * VS), Layout::kValues);
    copy(buffers.factors + at * (Layout::kFactors / 4), Layout::kFactors);
  };
  pdl_wait();
  if (tid == 0) {
    bring(0);
    if (chunks > 1) bring(1);
  }
  // S^T: column c0 + 16 group + g (+ 8), channel quarter * kQuarter + 8 j + 2 tq (+ 1)
  float* S_state = p.state + static_cast<long long>(p.state_slots[e]) * p.state_stride + static_cast<size_t>(h) * D * dv;
  const int column = c0 + 16 * group + g, channel = quarter * kQuarter + 2 * tq;
  float S[kTiles][4];
  const bool fresh = p.fresh[e] != 0;
#pragma unroll
  for (int j = 0; j < kTiles; ++j)
#pragma unroll
    for (int i = 0; i < 4; ++i)
      S[j][i] = fresh ? 0.0f : S_state[static_cast<size_t>(channel + 8 * j + (i & 1)) * dv + column + 8 * (i >> 1)];
  __syncthreads();   // the barriers are set up

  for (int chunk = 0; chunk < chunks; ++chunk) {
    const __nv_bfloat16* Qs = reinterpret_cast<const __nv_bfloat16*>(raw + (chunk & 1) * Layout::kStage);
    const __nv_bfloat16 *Ks = Qs + L * QS, *Ws = Ks + L * QS, *Vs = Ws + L * WS, *Us = Vs + L * VS;
    const float* factors = reinterpret_cast<const float*>(Us + L * VS);
    tcgen05::bar_wait<WALK_WAIT_EXPIRED>(&full[chunk & 1], (chunk >> 1) & 1, abort_flag, buffers.status);
    // outputs: what the state gives, over this warp's channels
    float O[8][4];
#pragma unroll
    for (int n = 0; n < 8; ++n)
#pragma unroll
      for (int i = 0; i < 4; ++i) O[n][i] = 0.0f;
#pragma unroll
    for (int kk = 0; kk < kSteps; ++kk) {
      uint32_t a[4];
#pragma unroll
      for (int half = 0; half < 2; ++half)
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const __nv_bfloat162 pair = __floats2bfloat162_rn(S[2 * kk + half][2 * r], S[2 * kk + half][2 * r + 1]);
          a[2 * half + r] = *reinterpret_cast<const uint32_t*>(&pair);
        }
#pragma unroll
      for (int n = 0; n < 8; n += 2) {
        uint32_t b[4];
        right(b, Qs, QS, n * 8, quarter * kQuarter + kk * 16, lane);
        mma_bf16(O[n], a, b[0], b[1]);
        mma_bf16(O[n + 1], a, b[2], b[3]);
      }
    }
    // and what the chunk's own earlier tokens give, sixteen of them a warp
    {
      uint32_t a[4];
      left_turned(a, Vs, VS, 16 * group, quarter * 16, lane);
      float* mine = Os + (group * 4 + quarter) * 16 * OS;
#pragma unroll
      for (int n = 0; n < 8; n += 2) {
        float P[2][4] = {{0.0f, 0.0f, 0.0f, 0.0f}, {0.0f, 0.0f, 0.0f, 0.0f}};
        if (n * 8 + 15 >= quarter * 16) {   // (else tokens before these)
          uint32_t b[4];
          right(b, Ws, WS, n * 8, quarter * 16, lane);
          mma_bf16(P[0], a, b[0], b[1]);
          mma_bf16(P[1], a, b[2], b[3]);
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int t = (n + i) * 8 + 2 * tq;
          const float2 f = *reinterpret_cast<const float2*>(factors + t), own = *reinterpret_cast<const float2*>(factors + L + t);
          *reinterpret_cast<float2*>(mine + g * OS + t) = make_float2(fmaf(P[i][0], own.x, O[n + i][0] * f.x), fmaf(P[i][1], own.y, O[n + i][1] * f.y));
          *reinterpret_cast<float2*>(mine + (g + 8) * OS + t) = make_float2(fmaf(P[i][2], own.x, O[n + i][2] * f.x), fmaf(P[i][3], own.y, O[n + i][3] * f.y));
        }
      }
    }
    asm volatile("bar.sync %0, 128;" ::"r"(1 + group) : "memory");   // a group's four warps have their parts there
    // the state
    const float keep = factors[2 * L];
#pragma unroll
    for (int j = 0; j < kTiles; ++j)
#pragma unroll
      for (int i = 0; i < 4; ++i) S[j][i] *= keep;
#pragma unroll
    for (int kk = 0; kk < L / 16; ++kk) {
      uint32_t a[4];
      left_turned(a, Us, VS, 16 * group, kk * 16, lane);
#pragma unroll
      for (int j = 0; j < kTiles; j += 2) {
        uint32_t b[4];
        right_turned(b, Ks, QS, quarter * kQuarter + j * 8, kk * 16, lane);
        mma_bf16(S[j], a, b[0], b[1]);
        mma_bf16(S[j + 1], a, b[2], b[3]);
      }
    }
    // sixteen tokens a warp: the four quarters' outputs, neighbouring lanes neighbouring columns
    {
      const float* parts = Os + group * 4 * 16 * OS + (lane & 15) * OS;
      const int len = count - chunk * L;
      float* out = p.o_raw + (static_cast<size_t>(t0 + chunk * L) * p.heads + h) * dv + c0 + 16 * group + (lane & 15);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int t = quarter * 16 + 2 * i + (lane >> 4);
        const float sum = (parts[t] + parts[16 * OS + t]) + (parts[32 * OS + t] + parts[48 * OS + t]);
        if (t < len) out[static_cast<size_t>(t) * p.heads * dv] = sum;
      }
    }
    __syncthreads();   // the stage and the outputs' parts are read
    if (tid == 0 && chunk + 2 < chunks && !*abort_flag) bring(chunk + 2);
  }
#pragma unroll
  for (int j = 0; j < kTiles; ++j)
#pragma unroll
    for (int i = 0; i < 4; ++i) S_state[static_cast<size_t>(channel + 8 * j + (i & 1)) * dv + column + 8 * (i >> 1)] = S[j][i];
  if (*abort_flag && tid == 0)
    for (int i = 0; i < 1000; ++i) __nanosleep(1000);   // copies may still be landing in this block's shared memory
}
