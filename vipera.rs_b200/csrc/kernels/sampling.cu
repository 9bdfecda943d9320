// Sampling on the device: penalties, greedy argmax, and temperature sampling with top-k,
// top-p and min-p, a cluster of blocks per row of logits.
//
// Semantics are those of the reference's sampler crate.  Greedy: the best finite logit,
// ties to the lowest id (crates/vipera-sampler/src/lib.rs:135-156).  Temperature: the k best
// candidates, best first with ties by ascending id (lib.rs:440-527); peak = best/T; total =
// sum over every finite logit of exp(x/T - peak); candidate weights exp(x/T - peak); the
// shortest head whose weights reach top_p * total; drop weights below min_p * best weight;
// target = uniform * mass, first candidate whose running sum (64-bit) exceeds it
// (lib.rs:172-247).  Penalties: for ids seen recently, logit > 0 ? logit / f : logit * f,
// minus presence + frequency * count; then the bias of the id (lib.rs:596-616).  The
// uniform number is drawn on the host from the request's own generator.
//
// With top_k = 0 the reference keeps a head of 4096 and sorts the whole vocabulary only if
// top-p reaches past it (lib.rs:437, 206-216); this kernel reports that case in `status`
// (SAMPLE_NEEDS_HOST) and the caller draws that row with the host sampler.
#include "simt.cuh"

enum SampleStatus { SAMPLE_OK = 0, SAMPLE_NO_FINITE = 1, SAMPLE_NO_MASS = 2, SAMPLE_NEEDS_HOST = 3 };

constexpr int kMaxCandidates = 4096;

__device__ __forceinline__ uint32_t ordered_key(float v) {
  const uint32_t bits = __float_as_uint(v);
  return (bits & 0x80000000u) ? ~bits : (bits | 0x80000000u);
}
__device__ __forceinline__ float key_value(uint32_t key) {
  return __uint_as_float((key & 0x80000000u) ? (key & 0x7fffffffu) : ~key);
}
__device__ __forceinline__ bool finite(float v) { return fabsf(v) <= 3.402823466e38f; }

// ---------------------------------------------------------------------------------------
// penalties: one thread per (row, id) entry
// ---------------------------------------------------------------------------------------
__global__ void penalty_kernel(float* __restrict__ logits, int vocab, int entries,
                               const int* __restrict__ entry_row, const int* __restrict__ entry_id,
                               const int* __restrict__ entry_count, const float* __restrict__ entry_bias,
                               const float* __restrict__ repetition, const float* __restrict__ presence,
                               const float* __restrict__ frequency) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= entries) return;
  const int row = entry_row[e], id = entry_id[e];
  if (id < 0 || id >= vocab) return;
  float* cell = logits + static_cast<size_t>(row) * vocab + id;
  float value = *cell;
  if (!finite(value)) return;
  const int count = entry_count[e];
  if (count > 0) {
    const float f = repetition[row];
    if (f != 1.0f) value = value > 0.0f ? value / f : value * f;
    value -= presence[row] + frequency[row] * static_cast<float>(count);
  }
  value += entry_bias[e];
  *cell = value;
}

VIPERA_API int vipera_apply_penalties(float* logits, int vocab, int entries, const int* entry_row,
                                      const int* entry_id, const int* entry_count, const float* entry_bias,
                                      const float* repetition, const float* presence, const float* frequency,
                                      void* stream) {
  if (entries <= 0) return VIPERA_OK;
  penalty_kernel<<<(entries + 127) / 128, 128, 0, static_cast<cudaStream_t>(stream)>>>(
      logits, vocab, entries, entry_row, entry_id, entry_count, entry_bias, repetition, presence, frequency);
  return vipera_launch_status();
}

// ---------------------------------------------------------------------------------------
// argmax with ties to the lowest id
// ---------------------------------------------------------------------------------------
struct Best {
  float value;
  int id;  // -1: nothing finite seen
};
__device__ __forceinline__ Best better_of(Best a, Best b) {
  if (a.id < 0) return b;
  if (b.id < 0) return a;
  if (a.value > b.value) return a;
  if (b.value > a.value) return b;
  return a.id < b.id ? a : b;
}
// Greedy over a wide vocabulary in two stages, so that many blocks read each row at once:
// every block finds the best of its slice of the row (eight independent loads in flight per
// thread), then one warp per row picks the best of the slices.  Ties still go to the lowest id.
constexpr int kArgmaxSlices = 32;
constexpr int kArgmaxThreads = 256;

__global__ void __launch_bounds__(kArgmaxThreads)
argmax_slice_kernel(const float* __restrict__ logits, int vocab, float* __restrict__ slice_value,
                    int* __restrict__ slice_id) {
  __shared__ Best scratch[32];
  const int row = blockIdx.x, slice = blockIdx.y;
  const int per = (vocab + kArgmaxSlices - 1) / kArgmaxSlices;
  const int begin = slice * per, end = min(vocab, begin + per);
  const float* src = logits + static_cast<size_t>(row) * vocab;
  Best best{0.0f, -1};
  for (int base = begin + threadIdx.x; base < end; base += 8 * kArgmaxThreads) {
    float v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int i = base + u * kArgmaxThreads;
      v[u] = i < end ? src[i] : NAN;
    }
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (finite(v[u])) best = better_of(best, Best{v[u], base + u * kArgmaxThreads});
  }
#pragma unroll
  for (int offset = 16; offset > 0; offset >>= 1) {
    Best other;
    other.value = __shfl_xor_sync(0xffffffffu, best.value, offset);
    other.id = __shfl_xor_sync(0xffffffffu, best.id, offset);
    best = better_of(best, other);
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) scratch[warp] = best;
  __syncthreads();
  if (warp == 0) {
    best = lane < kArgmaxThreads / 32 ? scratch[lane] : Best{0.0f, -1};
#pragma unroll
    for (int offset = 16; offset > 0; offset >>= 1) {
      Best other;
      other.value = __shfl_xor_sync(0xffffffffu, best.value, offset);
      other.id = __shfl_xor_sync(0xffffffffu, best.id, offset);
      best = better_of(best, other);
    }
    if (lane == 0) {
      slice_value[row * kArgmaxSlices + slice] = best.value;
      slice_id[row * kArgmaxSlices + slice] = best.id;
    }
  }
}

__global__ void argmax_final_kernel(const float* __restrict__ slice_value, const int* __restrict__ slice_id,
                                    int* __restrict__ tokens, int* __restrict__ status) {
  const int row = blockIdx.x, lane = threadIdx.x;
  Best best{slice_value[row * kArgmaxSlices + lane], slice_id[row * kArgmaxSlices + lane]};
#pragma unroll
  for (int offset = 16; offset > 0; offset >>= 1) {
    Best other;
    other.value = __shfl_xor_sync(0xffffffffu, best.value, offset);
    other.id = __shfl_xor_sync(0xffffffffu, best.id, offset);
    best = better_of(best, other);
  }
  if (lane == 0) {
    tokens[row] = best.id < 0 ? 0 : best.id;
    if (status) status[row] = best.id < 0 ? SAMPLE_NO_FINITE : SAMPLE_OK;
  }
}

// `scratch` holds 64 * rows 32-bit words (a value and an id for each of 32 slices of a row).
VIPERA_API int vipera_argmax(const float* logits, int rows, int vocab, int* tokens, int* status, void* scratch,
                             void* stream) {
  if (rows <= 0) return VIPERA_OK;
  if (vocab <= 0) return VIPERA_BAD_SHAPE;
  if (!scratch) return VIPERA_BAD_ARGUMENT;
  static_assert(kArgmaxSlices == 32, "the final stage is one warp");
  float* slice_value = static_cast<float*>(scratch);
  int* slice_id = reinterpret_cast<int*>(slice_value + static_cast<size_t>(rows) * kArgmaxSlices);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  argmax_slice_kernel<<<dim3(rows, kArgmaxSlices), kArgmaxThreads, 0, s>>>(logits, vocab, slice_value, slice_id);
  int launched = vipera_launch_status();
  if (launched != VIPERA_OK) return launched;
  argmax_final_kernel<<<rows, 32, 0, s>>>(slice_value, slice_id, tokens, status);
  return vipera_launch_status();
}

// ---------------------------------------------------------------------------------------
// temperature sampling
//
// A cluster of eight blocks takes a row.  Block b keeps the logits whose index modulo 1024 is in [128 b, 128 b + 128)
// in shared memory (one trip to memory for the whole draw), so that each of 1024 chains of the softmax sum lies in one
// block.  Four threads of a chain compute weights ahead and add them in turn.  Then a histogram over 2,048 equal steps
// below the best value (few ids meet in a bin, unlike the leading bits of the values; the upper bins first, which most
// draws do not look beyond) tells the first block how far down it has to go: to the bound-th largest, or to where the
// weights' sum is past top-p with a margin.  If what lies above is at most 4,096 ids, it goes to the first block, which
// puts it in order bin by bin, a bin's few by counting, and draws; the others leave.  Otherwise the bound-th largest
// (value, lowest id first) is found digit by digit, and sorted.  The weights' sum that top-p cuts and the mass are added
// in order, best first, by one thread from weights in shared memory, and what the floor leaves is read off on the way.
// What bounds it: instructions, two blocks of 512 threads an SM (clocks of a row with top-p, of 57 K: load 3, best 6,
// weights 8, bins 13, gathering and order 8, sum of 1,219 weights 10, draw 3), and 64 rows being two waves.  64 rows of
// 151,936 (a quarter each top-k 50, top-p alone, min-p, greedy): 48 us, 8 of 128,256: 24 us (with one thread a chain, a
// sort, two sums in order and every bin filled: 102 and 60; one block a row and a pass over memory per step: 440).
// ---------------------------------------------------------------------------------------
constexpr int kSampleBlocks = 8, kSampleThreads = 512;
constexpr int kChains = 1024, kOwnChains = kChains / kSampleBlocks;
constexpr int kBins = 2048;
constexpr int kFirstBins = 576;         // the bins that are filled first: far more than most draws look down to
constexpr int kAhead = 20;              // weights a thread has computed ahead of its turn in a chain
constexpr int kMostInBin = 64;          // of the candidates; more are sorted without the bins
constexpr int kMostKept = 200 * 1024;   // bytes of logits a block keeps; longer rows are read again for each step

struct SampleShared {
  unsigned int histogram[kBins];
  int ids[kMaxCandidates];              // the first block's candidates, then its weights
  float least[kSampleThreads / 32];
  // what every block found of the row, and its chains' sums, told by each to all
  Best block_best[kSampleBlocks];
  float block_least[kSampleBlocks];
  unsigned int block_finite[kSampleBlocks];
  float chain_sums[kSampleBlocks * kOwnChains / 32];
  int best_item;
  float scan_float[kSampleThreads / 32];
  float partial[kOwnChains];            // the chains' sums so far
  unsigned int count, bin, seen, listed, place;
  unsigned int scan[kSampleThreads / 32];
  double scan_double[kSampleThreads / 32];
  int cut, chosen, last;
  float mass;
};

__device__ __forceinline__ uint32_t cluster_address(const void* p, uint32_t block) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(shared_address(p)), "r"(block));
  return r;
}
__device__ __forceinline__ unsigned int remote_word(const void* p, uint32_t block) {
  unsigned int v;
  asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(cluster_address(p, block)) : "memory");
  return v;
}
__device__ __forceinline__ void remote_add(const void* p, uint32_t block, unsigned int value) {
  asm volatile("red.relaxed.cluster.shared::cluster.add.u32 [%0], %1;" ::"r"(cluster_address(p, block)), "r"(value) : "memory");
}
__device__ __forceinline__ unsigned int remote_fetch_add(const void* p, uint32_t block, unsigned int value) {
  unsigned int v;
  asm volatile("atom.relaxed.cluster.shared::cluster.add.u32 %0, [%1], %2;" : "=r"(v) : "r"(cluster_address(p, block)), "r"(value) : "memory");
  return v;
}
__device__ __forceinline__ void remote_store(const void* p, uint32_t block, unsigned int value) {
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(cluster_address(p, block)), "r"(value) : "memory");
}

// (value, id) as one number: larger is better, equal values best by the lowest id
__device__ __forceinline__ unsigned long long ranked(float v, int id) {
  return (static_cast<unsigned long long>(ordered_key(v)) << 32) | (0xffffffffu - static_cast<unsigned int>(id));
}

template <bool KEPT>
__global__ void __launch_bounds__(kSampleThreads, 2)
sample_kernel(const float* __restrict__ logits, int vocab, const float* __restrict__ temperature,
              const int* __restrict__ top_k, const float* __restrict__ top_p, const float* __restrict__ min_p,
              const double* __restrict__ uniform, int* __restrict__ tokens, int* __restrict__ status) {
  extern __shared__ __align__(16) unsigned char sample_raw[];
  SampleShared& s = *reinterpret_cast<SampleShared*>(sample_raw);
  float* kept = reinterpret_cast<float*>(sample_raw + (sizeof(SampleShared) + 15) / 16 * 16);   // [runs][kOwnChains]
  // (nothing is stored into another block before that has begun: the wait is ahead of the first such store)
  asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int own = blockIdx.x, r = blockIdx.y;
  const float* row = logits + static_cast<size_t>(r) * vocab;
  const int runs = (vocab + kChains - 1) / kChains, items = runs * kOwnChains;
  auto id_of = [&](int item) { return item / kOwnChains * kChains + own * kOwnChains + item % kOwnChains; };
  auto value_of = [&](int item) {
    if (KEPT) return kept[item];
    const int id = id_of(item);
    return id < vocab ? row[id] : NAN;
  };
  // every item of this thread: four neighbours at a time where the row is kept
  auto each_value = [&](auto take) {
    if (KEPT) {
#pragma unroll 2
      for (int i = tid * 4; i < items; i += kSampleThreads * 4) {
        const float4 v = *reinterpret_cast<const float4*>(kept + i);
        take(v.x, i), take(v.y, i + 1), take(v.z, i + 2), take(v.w, i + 3);
      }
    } else {
#pragma unroll 4
      for (int i = tid; i < items; i += kSampleThreads) take(value_of(i), i);
    }
  };
  for (int i = tid; i < kBins; i += kSampleThreads) s.histogram[i] = 0;
  if (tid < kOwnChains) s.partial[tid] = 0.0f;
  if (tid == 0) s.count = s.listed = 0;
  pdl_wait();
  if (KEPT) {
    if ((vocab & 3) == 0 && (reinterpret_cast<uintptr_t>(logits) & 15) == 0) {
#pragma unroll 4
      for (int i = tid * 4; i < items; i += kSampleThreads * 4) {
        const int id = id_of(i);
        if (id < vocab) copy_16(shared_address(kept + i), row + id, true);
        else kept[i] = kept[i + 1] = kept[i + 2] = kept[i + 3] = NAN;
      }
      copy_commit();
      copy_wait<0>();
    } else {
#pragma unroll 4
      for (int i = tid; i < items; i += kSampleThreads) kept[i] = id_of(i) < vocab ? row[id_of(i)] : NAN;
    }
  }
  __syncthreads();

  // the best finite logit of the row, ties to the lowest id, and how many are finite
  {
    float most = -INFINITY, least = INFINITY;
    unsigned int own_finite = 0;
    auto one = [&](float v) {
      if (!finite(v)) return;
      most = fmaxf(most, v);
      least = fminf(least, v);
      ++own_finite;
    };
    if (KEPT) {
      // (twice a number's bits are at least 0xff000000 where it is none)
#pragma unroll 2
      for (int i = tid * 4; i < items; i += kSampleThreads * 4) {
        const float4 v = *reinterpret_cast<const float4*>(kept + i);
        const unsigned int bits = max(max(__float_as_uint(v.x) << 1, __float_as_uint(v.y) << 1), max(__float_as_uint(v.z) << 1, __float_as_uint(v.w) << 1));
        if (bits < 0xff000000u) {
          most = fmaxf(most, fmaxf(fmaxf(v.x, v.y), fmaxf(v.z, v.w)));
          least = fminf(least, fminf(fminf(v.x, v.y), fminf(v.z, v.w)));
          own_finite += 4;
        } else {
          one(v.x), one(v.y), one(v.z), one(v.w);
        }
      }
    } else {
#pragma unroll 4
      for (int i = tid; i < items; i += kSampleThreads) one(value_of(i));
    }
    const float warp_most = warp_max(most);
    least = -warp_max(-least);
    own_finite = __reduce_add_sync(0xffffffffu, own_finite);
    if (lane == 0) {
      s.scan_float[warp] = warp_most;
      s.least[warp] = least;
      s.scan[warp] = own_finite;
    }
    if (tid == 0) s.best_item = 0x7fffffff;
    __syncthreads();
    float block_most = -INFINITY;
    for (int w = 0; w < kSampleThreads / 32; ++w) block_most = fmaxf(block_most, s.scan_float[w]);
    if (most == block_most && block_most > -INFINITY) {   // who has it looks for where it is first
      int where = 0x7fffffff;
      each_value([&](float v, int i) {
        if (v == block_most) where = min(where, i);
      });
      atomicMin(&s.best_item, where);
    }
    __syncthreads();
    asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
    if (tid < kSampleBlocks) {   // told to every block
      least = INFINITY, own_finite = 0;
      for (int w = 0; w < kSampleThreads / 32; ++w) least = fminf(least, s.least[w]), own_finite += s.scan[w];
      const int id = block_most > -INFINITY ? id_of(s.best_item) : -1;
      remote_store(&s.block_best[own].value, tid, __float_as_uint(block_most));
      remote_store(&s.block_best[own].id, tid, static_cast<unsigned int>(id));
      remote_store(&s.block_least[own], tid, __float_as_uint(least));
      remote_store(&s.block_finite[own], tid, own_finite);
    }
  }
  cluster_sync();
  Best best{0.0f, -1};
  unsigned int finite_total = 0;
  float least = INFINITY;
#pragma unroll
  for (int b = 0; b < kSampleBlocks; ++b) {
    least = fminf(least, s.block_least[b]);
    best = better_of(best, s.block_best[b]);
    finite_total += s.block_finite[b];
  }
  const float temp = temperature[r];
  if (best.id < 0 || temp == 0.0f) {
    if (own == 0 && tid == 0) {
      tokens[r] = best.id < 0 ? 0 : best.id;
      status[r] = best.id < 0 ? SAMPLE_NO_FINITE : SAMPLE_OK;
    }
    return;
  }
  const float scale = 1.0f / temp;
  const float peak = best.value * scale;

  // softmax mass over every finite logit: chain t adds the weights of ids t, t + 1024, ... in order.  Four threads a chain:
  // all compute the weights of their next runs at once, then each in its turn adds them to what the ones before have.
  {
    constexpr int kTurns = kSampleThreads / kOwnChains;
    const int chain = tid % kOwnChains, turn = tid / kOwnChains;
    for (int first = 0; first < runs; first += kTurns * kAhead) {
      float weight[kAhead];
#pragma unroll
      for (int j = 0; j < kAhead; ++j) {
        const int run = first + turn * kAhead + j;
        const float v = run < runs ? value_of(run * kOwnChains + chain) : NAN;
        weight[j] = finite(v) ? expf(v * scale - peak) : 0.0f;
      }
      for (int now = 0; now < kTurns; ++now) {
        if (turn == now) {
          float partial = s.partial[chain];
#pragma unroll
          for (int j = 0; j < kAhead; ++j) partial += weight[j];
          s.partial[chain] = partial;
        }
        __syncthreads();
      }
    }
    if (tid < kOwnChains) {
      const float partial = warp_sum(s.partial[tid]);
      if (lane < kSampleBlocks) remote_store(&s.chain_sums[own * (kOwnChains / 32) + warp], lane, __float_as_uint(partial));
    }
  }
  cluster_sync();
  static_assert(kSampleBlocks * kOwnChains / 32 == 32, "a lane has 32 chains' sum");
  const float total = warp_sum(s.chain_sums[lane]);
  const int requested = top_k[r];
  const bool uncut = requested == 0;
  if (!(total > 0.0f) || !finite(total) || requested > kMaxCandidates) {
    if (own == 0 && tid == 0) {
      tokens[r] = 0;
      status[r] = !(total > 0.0f) || !finite(total) ? SAMPLE_NO_MASS : SAMPLE_NEEDS_HOST;
    }
    return;
  }
  const unsigned int bound = min(min(uncut ? static_cast<unsigned int>(kMaxCandidates) : static_cast<unsigned int>(requested),
                                     static_cast<unsigned int>(kMaxCandidates)), finite_total);

  // Bins of equal steps below the best value, and how many of them are needed.
  const float step = (best.value - least) / (kBins - 0.5f), per_step = 1.0f / step;
  const bool spread = step > 0.0f && finite(step) && finite(per_step);
  auto bin_of = [&](float v) { return min(static_cast<int>((best.value - v) * per_step), kBins - 1); };
  int last_bin = -1;   // ids up to this bin go to the first block; below 0: bins cannot tell
  // The upper bins first; the others only where these do not reach far enough.
  const float floor_value = best.value - (kFirstBins + 2) * step;   // (no value of the upper bins is below)
  unsigned long long upper = 0;   // which of this thread's items, the first 64 of them, may lie in the upper bins
  for (int pass = 0; spread && pass < 2; ++pass) {
    const int from = pass ? kFirstBins : 0, to = pass ? kBins : kFirstBins;
    int number_of = 0;
    each_value([&](float v, int) {
      if (pass || v >= floor_value) {
        const int bin = finite(v) ? bin_of(v) : kBins;
        if (bin >= from && bin < to) {
          atomicAdd(&s.histogram[bin], 1u);
          if (number_of < 64) upper |= 1ull << number_of;
        }
      }
      ++number_of;
    });
    if (tid == 0) s.bin = kBins;
    cluster_sync();
    if (own == 0) {
      constexpr int kPer = kBins / kSampleThreads;
      static_assert(kPer == 4, "a thread's bins are one 16-byte read");
      uint4 n = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
      for (int b = 0; b < kSampleBlocks; ++b) {
        uint4 other;
        asm volatile("ld.shared::cluster.v4.u32 {%0, %1, %2, %3}, [%4];"
                     : "=r"(other.x), "=r"(other.y), "=r"(other.z), "=r"(other.w) : "r"(cluster_address(&s.histogram[tid * kPer], b)) : "memory");
        n.x += other.x, n.y += other.y, n.z += other.z, n.w += other.w;
      }
      const unsigned int mine[kPer] = {n.x, n.y, n.z, n.w};
      // what the bins hold at least: their count times the weight a little below their lower end
      const float top_weight = fmaf(best.value, scale, -peak);   // (0 but for the peak's rounding)
      unsigned int number = 0;
      float weight = 0.0f, lower[kPer];
#pragma unroll
      for (int j = 0; j < kPer; ++j) {
        lower[j] = static_cast<float>(mine[j]) * expf(top_weight - (tid * kPer + j + 1.01f) * (step * scale));
        number += mine[j];
        weight += lower[j];
      }
      unsigned int number_before = number;
      float weight_before = weight;
#pragma unroll
      for (int offset = 1; offset < 32; offset <<= 1) {
        const unsigned int other = __shfl_up_sync(0xffffffffu, number_before, offset);
        const float other_weight = __shfl_up_sync(0xffffffffu, weight_before, offset);
        if (lane >= offset) number_before += other, weight_before += other_weight;
      }
      if (lane == 31) s.scan[warp] = number_before, s.scan_float[warp] = weight_before;
      __syncthreads();
      number_before -= number, weight_before -= weight;
      for (int w = 0; w < warp; ++w) number_before += s.scan[w], weight_before += s.scan_float[w];
      // 4,096 roundings of 2^-24 and the exponentials' own stay far within a thousandth
      const float enough = top_p[r] * total * 1.001f;
      int found = kBins;
      unsigned int found_number = 0, upto = number_before;
#pragma unroll
      for (int j = 0; j < kPer; ++j) {
        upto += mine[j], weight_before += lower[j];
        if (found == kBins && (upto >= bound || weight_before >= enough)) found = tid * kPer + j, found_number = upto;
      }
      if (found < to) atomicMin(&s.bin, static_cast<unsigned int>(found));
      __syncthreads();
      if (found < kBins && s.bin == static_cast<unsigned int>(found)) s.seen = found_number;
      // where each bin's candidates begin
      if (s.bin < kBins) {
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
          s.histogram[tid * kPer + j] = number_before;
          number_before += mine[j];
        }
      }
    }
    cluster_sync();
    const unsigned int reached = remote_word(&s.bin, 0);
    if (reached >= kBins) {
      cluster_sync();   // the answer is read before the next one is begun
      continue;
    }
    if (remote_word(&s.seen, 0) <= kMaxCandidates) last_bin = static_cast<int>(reached);
    else {
      for (int i = tid; i < kBins; i += kSampleThreads) s.histogram[i] = 0;
      cluster_sync();   // the answer is read and every histogram is empty before anything is added to the first
    }
    break;
  }

  // The bound-th largest of (value, id): digits of its number from the highest on.  After each digit, everything
  // above the digits found is in, and `remaining` of those that share them.
  unsigned long long prefix = 0;
  unsigned int remaining = bound;
  int shift = 64;
#pragma unroll 1
  while (last_bin < 0) {
    const int width = shift == 42 || shift == 10 ? 10 : 11;   // 11, 11, 10 bits of the value, the same of the id
    const int next = shift - width;
    for (int i = tid; i < items; i += kSampleThreads) {
      const float v = value_of(i);
      if (!finite(v)) continue;
      const unsigned long long number = ranked(v, id_of(i));
      if (shift == 64 || (number >> shift) == prefix) atomicAdd(&s.histogram[(number >> next) & (kBins - 1) & ((1u << width) - 1u)], 1u);
    }
    __syncthreads();
    if (own != 0)
      for (int i = tid; i < kBins; i += kSampleThreads)
        if (const unsigned int n = s.histogram[i]) remote_add(&s.histogram[i], 0, n);
    cluster_sync();
    if (own == 0) {
      // from the highest bin down: a thread's four bins, then the threads before it
      constexpr int kPer = kBins / kSampleThreads;
      unsigned int mine[kPer], sum = 0;
#pragma unroll
      for (int j = 0; j < kPer; ++j) sum += mine[j] = s.histogram[kBins - 1 - (tid * kPer + j)];
      unsigned int before = sum;
#pragma unroll
      for (int offset = 1; offset < 32; offset <<= 1) {
        const unsigned int other = __shfl_up_sync(0xffffffffu, before, offset);
        if (lane >= offset) before += other;
      }
      if (lane == 31) s.scan[warp] = before;
      __syncthreads();
      for (int w = 0; w < warp; ++w) before += s.scan[w];
      before -= sum;
      if (before < remaining && before + sum >= remaining) {
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
          if (before + mine[j] >= remaining) {
            s.bin = kBins - 1 - (tid * kPer + j);
            s.seen = before | (before + mine[j] == remaining ? 0x80000000u : 0u);   // the bin is taken whole
            break;
          }
          before += mine[j];
        }
      }
    }
    cluster_sync();
    const unsigned int bin = remote_word(&s.bin, 0), seen = remote_word(&s.seen, 0);
    prefix = (shift == 64 ? 0ull : prefix << width) | bin;
    remaining -= seen & 0x7fffffffu;
    shift = next;
    if ((seen & 0x80000000u) || shift == 0) break;
    for (int i = tid; i < kBins; i += kSampleThreads) s.histogram[i] = 0;
    cluster_sync();   // the answer is read and every histogram is empty before anything is added to the first
  }

  // what is good enough goes to the first block
  {
    auto taken = [&](float v, int i) { return finite(v) && (last_bin >= 0 ? bin_of(v) <= last_bin : (ranked(v, id_of(i)) >> shift) >= prefix); };
    // The other blocks list theirs where their bins were (the first block has read them) and hand the list over at once.
    auto give = [&](float v, int i) {
      if (!taken(v, i)) return;
      const unsigned int id = static_cast<unsigned int>(id_of(i));
      if (own == 0) {
        const unsigned int at = atomicAdd(&s.count, 1u);
        if (at < kMaxCandidates) s.ids[at] = static_cast<int>(id);
        return;
      }
      const unsigned int place = atomicAdd(&s.listed, 1u);
      if (place < kBins) {
        s.histogram[place] = id;
      } else {
        const unsigned int at = remote_fetch_add(&s.count, 0, 1u);
        if (at < kMaxCandidates) remote_store(&s.ids[at], 0, id);
      }
    };
    if (KEPT && last_bin >= 0) {   // (what the bins hold was noted as it was counted)
      for (; upper; upper &= upper - 1) {
        const int number = __ffsll(static_cast<long long>(upper)) - 1, i = tid * 4 + number / 4 * (kSampleThreads * 4) + number % 4;
        give(kept[i], i);
      }
      for (int i = tid * 4 + 16 * (kSampleThreads * 4); i < items; i += kSampleThreads * 4)
        for (int j = 0; j < 4; ++j) give(kept[i + j], i + j);
    } else {
      each_value(give);
    }
    __syncthreads();
    const unsigned int listed = min(s.listed, static_cast<unsigned int>(kBins));
    if (tid == 0 && listed) s.place = remote_fetch_add(&s.count, 0, listed);
    __syncthreads();
    for (unsigned int i = tid; i < listed; i += kSampleThreads)
      if (s.place + i < kMaxCandidates) remote_store(&s.ids[s.place + i], 0, s.histogram[i]);
  }
  cluster_sync();
  if (own != 0) return;

  const unsigned int gathered = min(s.count, static_cast<unsigned int>(kMaxCandidates)), count = min(gathered, bound);
  // the candidates' numbers take the place of the logits (and, where those are not kept, room of their own)
  unsigned long long* candidates = reinterpret_cast<unsigned long long*>(kept);
  bool ordered = last_bin >= 0;
  if (ordered) {
    // Each goes among its bin's, and there behind those that are better.  (gathered is what the bins hold up to the last.)
    unsigned long long* grouped = candidates + kMaxCandidates;
    auto bin_at = [&](unsigned long long number) { return bin_of(key_value(static_cast<uint32_t>(number >> 32))); };
    for (unsigned int i = tid; i < gathered; i += kSampleThreads) {
      const unsigned long long number = ranked(row[s.ids[i]], s.ids[i]);
      grouped[min(atomicAdd(&s.histogram[bin_at(number)], 1u), static_cast<unsigned int>(kMaxCandidates - 1))] = number;
    }
    __syncthreads();
    bool crowded = false;
    for (unsigned int i = tid; i < gathered; i += kSampleThreads) {
      const unsigned long long number = grouped[i];
      const int bin = bin_at(number);
      const unsigned int begin = bin ? s.histogram[bin - 1] : 0, end = s.histogram[bin];
      if (end - begin > kMostInBin) {
        crowded = true;
        continue;
      }
      unsigned int place = begin;
      for (unsigned int j = begin; j < end; ++j) place += grouped[j] > number;
      candidates[place] = number;
    }
    ordered = !__syncthreads_or(crowded);
  }
  if (!ordered) {
    unsigned int padded = 1;
    while (padded < gathered) padded <<= 1;
    for (unsigned int i = tid; i < padded; i += kSampleThreads) candidates[i] = i < gathered ? ranked(row[s.ids[i]], s.ids[i]) : 0ull;
    __syncthreads();
    // bitonic sort, descending
    for (unsigned int size = 2; size <= padded; size <<= 1) {
      for (unsigned int stride = size >> 1; stride > 0; stride >>= 1) {
        for (unsigned int pair = tid; pair < padded / 2; pair += kSampleThreads) {
          const unsigned int i = 2 * pair - (pair & (stride - 1)), partner = i + stride;
          const bool descending = (i & size) == 0;
          const unsigned long long a = candidates[i], b = candidates[partner];
          if (descending ? a < b : a > b) { candidates[i] = b; candidates[partner] = a; }
        }
        __syncthreads();
      }
    }
  }
  auto id_at = [&](unsigned int i) { return static_cast<int>(0xffffffffu - static_cast<unsigned int>(candidates[i] & 0xffffffffull)); };
  float* weights = reinterpret_cast<float*>(s.ids);
  for (unsigned int i = tid; i < kMaxCandidates; i += kSampleThreads)
    weights[i] = i < count ? expf(key_value(static_cast<uint32_t>(candidates[i] >> 32)) * scale - peak) : 0.0f;
  __syncthreads();
  const float best_weight = weights[0], floor_weight = min_p[r] * best_weight;
  // How many are not below the floor, and whether these are the first ones (weights fall, but for an exponential's last bit).
  unsigned int above = 0, behind = 0;
  for (unsigned int i0 = 0; i0 < count; i0 += kSampleThreads) {
    const unsigned int i = i0 + tid;
    const bool in = i < count && weights[i] >= floor_weight;
    above += __syncthreads_count(in);
    behind += __syncthreads_count(in && i > 0 && !(weights[i - 1] >= floor_weight));
  }
  if (tid == 0) {
    // The top-p cut: weights added in order, best first, 32 at a time with nothing between the additions, then again within
    // the 32 that the cut, or the floor, falls in.  What the floor leaves has the sum the weights had when it was met.
    const float target_mass = top_p[r] * total;
    float* upto = reinterpret_cast<float*>(s.histogram);   // before each 32
    float cumulative = 0.0f, mass = 0.0f;
    int cut = -1;
    unsigned int reached = 0;
#pragma unroll 1
    for (unsigned int i = 0; i < count; i += 32) {
      float w[32];
#pragma unroll
      for (int j = 0; j < 32; j += 4) *reinterpret_cast<float4*>(w + j) = *reinterpret_cast<const float4*>(weights + i + j);
      upto[i / 32] = cumulative;
#pragma unroll
      for (int j = 0; j < 32; ++j) cumulative += w[j];
      reached = i;
      if (cumulative >= target_mass) break;
    }
    if (cumulative >= target_mass) {
      float again = upto[reached / 32];
      for (unsigned int i = reached; cut < 0; ++i) {
        again += weights[i];
        if (again >= target_mass) cut = static_cast<int>(i) + 1;
      }
    }
    const unsigned int end = cut >= 0 ? min(above, static_cast<unsigned int>(cut)) : above;
    if (end > 0) {
      mass = upto[(end - 1) / 32];
      for (unsigned int i = (end - 1) / 32 * 32; i < end; ++i) mass += weights[i];
    }
    if (behind) {
      const unsigned int kept_end = cut >= 0 ? static_cast<unsigned int>(cut) : count;
      mass = 0.0f;
      for (unsigned int i = 0; i < kept_end; ++i)
        if (weights[i] >= floor_weight) mass += weights[i];
    }
    s.cut = cut;
    s.mass = mass;
    s.chosen = kMaxCandidates;
    s.last = -1;
  }
  __syncthreads();
  if (uncut && s.cut < 0 && count < finite_total) {
    if (tid == 0) { tokens[r] = 0; status[r] = SAMPLE_NEEDS_HOST; }
    return;
  }
  const unsigned int kept_end = s.cut >= 0 ? static_cast<unsigned int>(s.cut) : count;
  const double target = uniform[r] * static_cast<double>(s.mass);
  // the first candidate whose running sum (64-bit) exceeds the target: eight neighbours a thread, then the threads before it
  constexpr int kPer = kMaxCandidates / kSampleThreads;
  double running[kPer], sum = 0.0;
  bool counts[kPer];
#pragma unroll
  for (int j = 0; j < kPer; ++j) {
    const unsigned int i = tid * kPer + j;
    counts[j] = i < kept_end && weights[i] >= floor_weight;
    if (counts[j]) sum += static_cast<double>(weights[i]);
    running[j] = sum;
  }
  double before = sum;
#pragma unroll
  for (int offset = 1; offset < 32; offset <<= 1) {
    const double other = __shfl_up_sync(0xffffffffu, before, offset);
    if (lane >= offset) before += other;
  }
  if (lane == 31) s.scan_double[warp] = before;
  __syncthreads();
  before -= sum;
  for (int w = 0; w < warp; ++w) before += s.scan_double[w];
#pragma unroll
  for (int j = kPer - 1; j >= 0; --j) {
    if (!counts[j]) continue;
    if (target < before + running[j]) atomicMin(&s.chosen, tid * kPer + j);
    atomicMax(&s.last, tid * kPer + j);
  }
  __syncthreads();
  if (tid == 0) {
    tokens[r] = s.chosen < kMaxCandidates ? id_at(s.chosen) : (s.last >= 0 ? id_at(s.last) : best.id);
    status[r] = SAMPLE_OK;
  }
}

// One row of `logits` per request; rows with temperature 0 are drawn greedily.  `status`
// gets a SampleStatus per row.
VIPERA_API int vipera_sample(const float* logits, int rows, int vocab, const float* temperature,
                             const int* top_k, const float* top_p, const float* min_p,
                             const double* uniform, int* tokens, int* status, void* stream) {
  if (rows <= 0) return VIPERA_OK;
  if (vocab <= 0) return VIPERA_BAD_SHAPE;
  if (!status || !tokens) return VIPERA_BAD_ARGUMENT;
  constexpr int kHead = static_cast<int>((sizeof(SampleShared) + 15) / 16 * 16), kRanks = 2 * kMaxCandidates * 8;
  const long long logits_bytes = (static_cast<long long>(vocab) + kChains - 1) / kChains * kOwnChains * 4;
  const bool keep = logits_bytes <= kMostKept;
  const int bytes = kHead + static_cast<int>(keep && logits_bytes > kRanks ? logits_bytes : kRanks);
  static SharedMemoryOptIn opt_in_kept, opt_in_read;
  const int opted = keep ? opt_in_kept.ask(reinterpret_cast<const void*>(sample_kernel<true>), kHead + kMostKept)
                         : opt_in_read.ask(reinterpret_cast<const void*>(sample_kernel<false>), kHead + kMostKept);
  if (opted) return opted;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  for (int first = 0; first < rows; first += 65535) {   // a grid's extent along y
    const int count = rows - first < 65535 ? rows - first : 65535;
    const int launched = launch_in_clusters(keep ? sample_kernel<true> : sample_kernel<false>, kSampleBlocks, dim3(kSampleBlocks, count),
                                            dim3(kSampleThreads), bytes, s, logits + static_cast<size_t>(first) * vocab, vocab,
                                            temperature + first, top_k + first, top_p + first, min_p + first, uniform + first,
                                            tokens + first, status + first);
    if (launched) return launched;
  }
  return VIPERA_OK;
}

// ---------------------------------------------------------------------------------------
// Log-probabilities of drawn tokens (crates/vipera-sampler/src/lib.rs:319-378): over every
// finite logit (penalties already applied), x = logit / temperature (1 where the row is drawn
// greedily), logprob(id) = x_id - max - ln(sum exp(x - max)); the drawn token's, and the top_n
// most likely ids with theirs, best first, ties to the lowest id.  One block per asked row.
// ---------------------------------------------------------------------------------------
constexpr int kLogprobThreads = 256;

__global__ void __launch_bounds__(kLogprobThreads)
logprob_kernel(const float* __restrict__ logits, int vocab, const int* __restrict__ rows, const int* __restrict__ tokens,
               const float* __restrict__ temperature, int top_n, float* __restrict__ chosen, int* __restrict__ top_ids,
               float* __restrict__ top_values) {
  __shared__ float scratch[32];
  __shared__ float best_value[kLogprobThreads];
  __shared__ int best_id[kLogprobThreads];
  const int item = blockIdx.x;
  const float* row = logits + static_cast<size_t>(rows[item]) * vocab;
  const float t = temperature[item] > 0.0f ? temperature[item] : 1.0f;
  float peak = -INFINITY;
  for (int i = threadIdx.x; i < vocab; i += kLogprobThreads) {
    const float v = row[i];
    if (finite(v)) peak = fmaxf(peak, v / t);
  }
  peak = block_max(peak, scratch);
  float mass = 0.0f;
  for (int i = threadIdx.x; i < vocab; i += kLogprobThreads) {
    const float v = row[i];
    if (finite(v)) mass += expf(v / t - peak);
  }
  mass = block_sum(mass, scratch);
  const float log_mass = logf(mass);
  if (threadIdx.x == 0) {
    const float v = row[tokens[item]];
    chosen[item] = finite(peak) && finite(v) ? v / t - peak - log_mass : -INFINITY;
  }
  // the top_n: each round takes the best (value, then lowest id) that comes after the one before
  float last_value = INFINITY;
  int last_id = -1;
  for (int k = 0; k < top_n; ++k) {
    float mine = -INFINITY;
    int mine_id = -1;
    for (int i = threadIdx.x; i < vocab; i += kLogprobThreads) {
      const float v = row[i];
      if (!finite(v)) continue;
      const float x = v / t;
      const bool after = x < last_value || (x == last_value && i > last_id);
      if (after && (x > mine || mine_id < 0)) {   // ids rise within a thread, so the first of equals stays
        mine = x;
        mine_id = i;
      }
    }
    best_value[threadIdx.x] = mine;
    best_id[threadIdx.x] = mine_id;
    __syncthreads();
    for (int stride = kLogprobThreads / 2; stride > 0; stride >>= 1) {
      if (threadIdx.x < stride) {
        const float a = best_value[threadIdx.x], b = best_value[threadIdx.x + stride];
        const int ia = best_id[threadIdx.x], ib = best_id[threadIdx.x + stride];
        const bool take_b = ib >= 0 && (ia < 0 || b > a || (b == a && ib < ia));
        if (take_b) {
          best_value[threadIdx.x] = b;
          best_id[threadIdx.x] = ib;
        }
      }
      __syncthreads();
    }
    last_value = best_value[0];
    last_id = best_id[0];
    __syncthreads();
    if (threadIdx.x == 0) {
      top_ids[static_cast<size_t>(item) * top_n + k] = last_id;
      top_values[static_cast<size_t>(item) * top_n + k] = last_id >= 0 ? last_value - peak - log_mass : -INFINITY;
    }
    if (last_id < 0) last_value = -INFINITY;   // nothing left: the remaining places stay empty
  }
}

// chosen[i] = log-probability of tokens[i] in row rows[i] of `logits` at temperature[i]; with
// top_n > 0 also the top_n most likely ids of that row and their log-probabilities (-1 and
// -inf where the row has fewer finite logits).
VIPERA_API int vipera_logprobs(const float* logits, int vocab, int count, const int* rows, const int* tokens,
                               const float* temperature, int top_n, float* chosen, int* top_ids, float* top_values,
                               void* stream) {
  if (count <= 0) return VIPERA_OK;
  if (vocab <= 0 || top_n < 0) return VIPERA_BAD_SHAPE;
  if (!logits || !rows || !tokens || !temperature || !chosen || (top_n > 0 && (!top_ids || !top_values)))
    return VIPERA_BAD_ARGUMENT;
  logprob_kernel<<<count, kLogprobThreads, 0, static_cast<cudaStream_t>(stream)>>>(logits, vocab, rows, tokens, temperature,
                                                                                   top_n, chosen, top_ids, top_values);
  return vipera_launch_status();
}

VIPERA_API const char* vipera_sampling_status_text(int status) { return vipera_status_text(status); }

// ---------------------------------------------------------------------------------------
// greedy argmax for callers that cannot allocate (see no_alloc.h)
// ---------------------------------------------------------------------------------------
#include "no_alloc.h"

// The scratch of the two argmax stages, inside the library image itself.  In host code this
// name is only a handle for the symbol, not a device address: the address comes from
// cudaGetSymbolAddress below.
static __device__ __align__(256) unsigned int argmax_static_scratch[64 * VIPERA_ARGMAX_STATIC_MAX_ROWS];

// Device address of the array on each device, looked up on the first call there.
static void* argmax_static_address[64] = {nullptr};

extern "C" __attribute__((visibility("default")))
int vipera_argmax_static(const float* logits, int rows, int vocab, int* tokens, int* status, void* stream) {
  if (rows <= 0) return VIPERA_OK;
  if (rows > VIPERA_ARGMAX_STATIC_MAX_ROWS || vocab <= 0) return VIPERA_BAD_SHAPE;
  if (!logits || !tokens) return VIPERA_BAD_ARGUMENT;
  int device = 0;
  cudaError_t error = cudaGetDevice(&device);
  if (error != cudaSuccess) return static_cast<int>(error);
  if (device < 0 || device >= 64) return VIPERA_BAD_ARGUMENT;
  if (argmax_static_address[device] == nullptr) {
    // set-up, once per device, with that device current
    void* address = nullptr;
    error = cudaGetSymbolAddress(&address, argmax_static_scratch);
    if (error != cudaSuccess) return static_cast<int>(error);
    argmax_static_address[device] = address;
  }
  float* slice_value = static_cast<float*>(argmax_static_address[device]);
  int* slice_id = reinterpret_cast<int*>(slice_value + static_cast<size_t>(rows) * kArgmaxSlices);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  // Every (row, slice) word is written by the first kernel before the second reads it, so
  // nothing left by an earlier call is ever read and nothing needs clearing.
  argmax_slice_kernel<<<dim3(rows, kArgmaxSlices), kArgmaxThreads, 0, s>>>(logits, vocab, slice_value, slice_id);
  int launched = vipera_launch_status();
  if (launched != VIPERA_OK) return launched;
  argmax_final_kernel<<<rows, 32, 0, s>>>(slice_value, slice_id, tokens, status);
  return vipera_launch_status();
}

// The tokens a step has drawn become the next step's input without a trip to the host:
// dst[i] = src[i] for the step's own entries; the entries a captured graph adds to fill its
// size repeat entry 0, as they do in every other input.
__global__ void feed_tokens_kernel(const int* __restrict__ src, int* __restrict__ dst, int own, int total) {
  pdl_launch_dependents();
  pdl_wait();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < total) dst[i] = src[i < own ? i : 0];
}

VIPERA_API int vipera_feed_tokens(const int* src, int* dst, int own, int total, void* stream) {
  if (own <= 0 || total < own) return VIPERA_BAD_SHAPE;
  return vipera_launch(feed_tokens_kernel, dim3((total + 255) / 256), dim3(256), 0, static_cast<cudaStream_t>(stream), src, dst,
                       own, total);
}

// Wait until everything queued on `stream` so far has run.
VIPERA_API int vipera_stream_synchronize(void* stream) {
  const cudaError_t error = cudaStreamSynchronize(static_cast<cudaStream_t>(stream));
  return error == cudaSuccess ? VIPERA_OK : static_cast<int>(error);
}
