// Device-side token sampler: top-k / top-p selection with a per-request xorshift64 generator,
// replacing the host `Sampler` (tuisko-engine/src/sampling.rs:76-231) and the device -> host copy
// of a 248 320-wide logit row that feeds it.
//
// One launch for a decode batch of up to 8 rows.  A row of BF16 logits (0.5 MB) is cut into slices of
// about 8000 values, one CTA each, 32 values per thread, all requested before the first is used.  The
// top_k-th largest of the 256 thread maxima is a bound that at most top_k threads reach: only they
// write candidates (about as many as top_k, never more than 32 per thread) to shared memory, and one
// warp sorts those.  Inside a CTA a candidate is 32 bits, its order above its position in the slice;
// sorts and merges run on one key per lane with warp shuffles.  The CTAs leave their 32 keys in a
// caller-owned scratch and take a ticket; the CTA that draws a row's last ticket merges them and runs
// the reference's scalar selection on the k survivors (same float / double operations in the same
// order), so no second launch and no host hop follow.
//
// What bounds it is this chain of latencies, not the 4 MB of eight rows: 8.7 us for eight rows of
// 248 320 values, against 20.4 us with sorted 64-bit lists kept by every warp, whose shuffles (two per
// exchange, 330 per warp before the first value was dropped) filled the issue slots.
#include <math.h>

#include "common.cuh"
#include "kernels.h"
#include "ptx.cuh"

namespace tk100 {
namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kList = 32;  // keys a list keeps = the largest admitted top_k
constexpr int kPerThread = 32;                           // values of a block per thread
constexpr int kBlockChunks = kThreads * kPerThread / 8;  // 8192 values: positions fit 16 bits

// Larger order = earlier in the reference's order: value descending under the IEEE total order
// (+0 above -0); of equal ones the lower index (sampling.rs:219-224: only a strictly greater value
// displaces a retained one).
__device__ __forceinline__ uint32_t order_of(uint32_t bf16_bits) {
  return (bf16_bits & 0x8000u) ? (~bf16_bits & 0xffffu) : (bf16_bits | 0x8000u);
}
__device__ __forceinline__ uint32_t key_index(uint64_t key) { return ~static_cast<uint32_t>(key); }
__device__ __forceinline__ float key_value(uint64_t key) {
  const uint32_t ord = static_cast<uint32_t>(key >> 32);
  const uint32_t bits = (ord & 0x8000u) ? (ord & 0x7fffu) : (~ord & 0xffffu);
  return __uint_as_float(bits << 16);
}

// exp of a non-positive f32 argument as the f32 nearest to the exact value, returned as a double:
// the reference's `((v - max) / temperature).exp() as f64`.  Evaluated in double (argument
// reduction by ln 2 in two pieces, degree-13 Taylor polynomial on |r| <= 0.347: relative error
// below 1e-16), so the rounding to f32 is the correctly rounded result except within 1e-9 of a
// rounding boundary.  Written out here rather than calling the library exponential, whose slow
// path is a function call.
__device__ __forceinline__ double softmax_weight(float scaled) {
  const double x = static_cast<double>(scaled);
  if (!(x >= -104.0)) return 0.0;  // below half of the smallest f32 denormal (e^-103.97)
  const double n = rint(x * 1.4426950408889634);
  double r = fma(n, -6.93147180369123816490e-01, x);
  r = fma(n, -1.90821492927058770002e-10, r);
  double p = 1.0 / 6227020800.0;
  p = fma(p, r, 1.0 / 479001600.0);
  p = fma(p, r, 1.0 / 39916800.0);
  p = fma(p, r, 1.0 / 3628800.0);
  p = fma(p, r, 1.0 / 362880.0);
  p = fma(p, r, 1.0 / 40320.0);
  p = fma(p, r, 1.0 / 5040.0);
  p = fma(p, r, 1.0 / 720.0);
  p = fma(p, r, 1.0 / 120.0);
  p = fma(p, r, 1.0 / 24.0);
  p = fma(p, r, 1.0 / 6.0);
  p = fma(p, r, 0.5);
  p = fma(p, r, 1.0);
  p = fma(p, r, 1.0);
  const double scale = __longlong_as_double((static_cast<long long>(n) + 1023) << 52);  // 2^n, n >= -151
  return static_cast<double>(static_cast<float>(p * scale));
}

__device__ __forceinline__ uint64_t shfl64(uint64_t v, int src) {
  return __shfl_sync(0xffffffffu, v, src);
}

template <class Key>
__device__ __forceinline__ Key greater_of(Key a, Key b) { return a > b ? a : b; }
template <class Key>
__device__ __forceinline__ Key lesser_of(Key a, Key b) { return a < b ? a : b; }

// Bitonic sort of one key per lane into descending order (lane 0 the largest): 15 exchanges.
template <class Key>
__device__ __forceinline__ Key sort_descending(Key v, int lane) {
#pragma unroll
  for (int k = 2; k <= 32; k <<= 1) {
#pragma unroll
    for (int j = k >> 1; j > 0; j >>= 1) {
      const Key other = __shfl_xor_sync(0xffffffffu, v, j);
      const bool keep_max = ((lane & j) == 0) == ((lane & k) == 0);
      v = keep_max ? greater_of(v, other) : lesser_of(v, other);
    }
  }
  return v;
}

// The 32 largest of two descending lists (one key per lane each), descending: reversing one list
// makes the lane-wise maxima a bitonic sequence of exactly those keys; 5 exchanges sort it.
template <class Key>
__device__ __forceinline__ Key merge_descending(Key a, Key b, int lane) {
  Key v = greater_of(a, __shfl_sync(0xffffffffu, b, 31 - lane));
#pragma unroll
  for (int j = 16; j > 0; j >>= 1) {
    const Key other = __shfl_xor_sync(0xffffffffu, v, j);
    v = ((lane & j) == 0) ? greater_of(v, other) : lesser_of(v, other);
  }
  return v;
}

// Warp 0 ends with the 32 largest keys of the CTA's eight descending lists (one per warp).
template <class Key>
__device__ __forceinline__ Key fold_warps(Key held, Key (*lists)[kList], int warp, int lane) {
#pragma unroll
  for (int half = kWarps / 2; half > 0; half >>= 1) {
    if (warp >= half && warp < 2 * half) lists[warp][lane] = held;
    __syncthreads();
    if (warp < half) held = merge_descending(held, lists[warp + half][lane], lane);
  }
  return held;
}

__global__ void __launch_bounds__(kThreads, 1) sampler_kernel(SamplerParams p) {
  __shared__ union {
    uint32_t local[kWarps][kList];  // thread maxima, folded
    uint32_t candidates[kList * kPerThread];
    uint64_t global[kWarps][kList];  // slices' lists, folded
  } lists;
  __shared__ uint32_t bound, candidate_count;
  __shared__ int is_last;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int row = blockIdx.y, slice = blockIdx.x, slices = gridDim.x;
  const int top_k = p.top_k[row];
  const uint16_t* logits = p.logits + static_cast<size_t>(row) * p.vocab;
  uint64_t* row_scratch = p.scratch + static_cast<size_t>(row) * (slices * kList);
  unsigned int* ticket = reinterpret_cast<unsigned int*>(p.scratch + static_cast<size_t>(p.rows) * slices * kList) + row;

  pdl_trigger();
  pdl_wait();

  // 8-value chunks of the row, dealt to the slices in contiguous runs and walked in blocks of
  // kBlockChunks (one block while the vocabulary has at most 32 * 8192 values).
  const int chunks = p.vocab / 8;
  const int begin = static_cast<int>(static_cast<long long>(chunks) * slice / slices);
  const int end = static_cast<int>(static_cast<long long>(chunks) * (slice + 1) / slices);

  uint64_t held = 0;
  bool nonfinite = false;
  for (int base = begin; base < end; base += kBlockChunks) {
    uint4 w[kPerThread / 8];
#pragma unroll
    for (int i = 0; i < kPerThread / 8; ++i) {
      const int chunk = base + i * kThreads + tid;
      w[i] = chunk < end ? __ldg(reinterpret_cast<const uint4*>(logits) + chunk) : make_uint4(0u, 0u, 0u, 0u);
    }
    // Keys of this block: order above 0xffff - position, so a lower index wins a tie; 0 is no value
    // (the lowest order with the highest position is still above it).
    uint32_t key[kPerThread];
    uint32_t best = 0;
#pragma unroll
    for (int i = 0; i < kPerThread / 8; ++i) {
      const bool live = base + i * kThreads + tid < end;
      const uint32_t words[4] = {w[i].x, w[i].y, w[i].z, w[i].w};
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const uint32_t bits = (words[j >> 1] >> ((j & 1) * 16)) & 0xffffu;
        nonfinite |= (bits & 0x7f80u) == 0x7f80u;
        const uint32_t position = static_cast<uint32_t>((i * kThreads + tid) * 8 + j);
        key[i * 8 + j] = live ? (order_of(bits) << 16) | (0xffffu - position) : 0u;
        best = greater_of(best, key[i * 8 + j]);
      }
    }
    const uint32_t maxima = fold_warps(sort_descending(best, lane), lists.local, warp, lane);
    if (warp == 0) {
      const uint32_t kth = __shfl_sync(0xffffffffu, maxima, top_k - 1);
      if (lane == 0) {
        bound = greater_of(kth, 1u);  // fewer than top_k threads have values: all of theirs
        candidate_count = 0;
      }
    }
    __syncthreads();
    const uint32_t least = bound;
    if (best >= least) {  // at most top_k threads: keys are distinct
#pragma unroll
      for (int i = 0; i < kPerThread; ++i) {
        if (key[i] >= least) lists.candidates[atomicAdd(&candidate_count, 1u)] = key[i];
      }
    }
    __syncthreads();
    if (warp == 0) {
      const int count = static_cast<int>(candidate_count);
      uint32_t top = 0;
      for (int c = 0; c < count; c += kList) {
        const uint32_t sorted = sort_descending(c + lane < count ? lists.candidates[c + lane] : 0u, lane);
        top = c == 0 ? sorted : merge_descending(top, sorted, lane);
      }
      const uint32_t index = static_cast<uint32_t>(base) * 8u + (0xffffu - (top & 0xffffu));
      const uint64_t wide = top == 0u ? 0ull : (static_cast<uint64_t>(top >> 16) << 32) | static_cast<uint64_t>(~index);
      held = base == begin ? wide : merge_descending(held, wide, lane);
    }
    __syncthreads();  // the shared lists are free again
  }
  if (nonfinite) atomicOr(p.status, STATUS_NONFINITE_LOGIT);

  if (warp == 0) {
    row_scratch[slice * kList + lane] = held;
    __threadfence();
    __syncwarp();
    if (lane == 0) is_last = atomicAdd(ticket, 1u) == static_cast<unsigned int>(slices - 1);
  }
  __syncthreads();
  if (!is_last) return;
  __threadfence();

  // The row's last CTA: every warp merges its share of the slices' lists, then the tree over the warps.
  {
    // at most 32 slices: four lists per warp, all requested before the first merge
    uint64_t other[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int s = warp + i * kWarps;
      other[i] = s < slices ? *reinterpret_cast<volatile uint64_t*>(row_scratch + s * kList + lane) : 0ull;
    }
    held = merge_descending(merge_descending(other[0], other[1], lane), merge_descending(other[2], other[3], lane), lane);
  }
  held = fold_warps(held, lists.global, warp, lane);
  if (warp != 0) return;
  if (lane == 0) *ticket = 0;  // ready for the next launch

  if (p.top_out != nullptr && lane < top_k) {
    p.top_out[(row * kList + lane) * 2] = __float_as_uint(key_value(held));
    p.top_out[(row * kList + lane) * 2 + 1] = key_index(held);
  }

  // sampling.rs:102-108: temperature 0 or top_k 1 is the greedy route and draws no random number.
  const float temperature = p.temperature[row];
  uint32_t token = key_index(shfl64(held, 0));
  if (!(temperature == 0.0f || top_k == 1)) {
    // sampling.rs:175-210, evaluated by every lane on the same values.
    // Lane i evaluates the weight of survivor i (the exponentials run side by side); the sums
    // below then walk the lanes in the reference's order.
    const float maximum = key_value(shfl64(held, 0));
    const float scaled = __fdiv_rn(key_value(held) - maximum, temperature);
    const double my_weight = lane < top_k ? softmax_weight(scaled) : 0.0;
    // Lane i ends with the running sum over survivors 0..i, added in survivor order (the
    // reference's three loops walk this same sequence).
    double running = 0.0;
#pragma unroll 4
    for (int i = 0; i < top_k; ++i) {
      const double w = __shfl_sync(0xffffffffu, my_weight, i);
      if (i <= lane) running += w;
    }
    const double total = __shfl_sync(0xffffffffu, running, top_k - 1);
    const double cutoff = static_cast<double>(fmaxf(p.top_p[row], 1.17549435e-38f)) * total;
    // first survivor whose running sum reaches the cut-off (all of them if none does)
    int retained = __popc(__ballot_sync(0xffffffffu, lane < top_k && !(running >= cutoff))) + 1;
    retained = retained > top_k ? top_k : retained;
    const double retained_total = __shfl_sync(0xffffffffu, running, retained - 1);
    // xorshift64 (sampling.rs:244-260); the state advances once per sampled token.
    uint64_t state = p.rng_state[row];
    state ^= state << 13;
    state ^= state >> 7;
    state ^= state << 17;
    const double unit = static_cast<double>(state >> 11) * (1.0 / 9007199254740992.0);
    const double threshold = unit * retained_total;
    int chosen = __popc(__ballot_sync(0xffffffffu, lane < retained && !(running >= threshold)));
    chosen = chosen >= retained ? retained - 1 : chosen;
    token = key_index(shfl64(held, chosen));
    if (lane == 0) p.rng_state[row] = state;
    if (!(retained_total > 0.0) || isinf(retained_total)) atomicOr(p.status, STATUS_NONFINITE_LOGIT);
  }
  if (lane == 0) {
    p.decisions[row * 2] = token;
    p.decisions[row * 2 + 1] = (token == p.stop_ids[row * 2] || token == p.stop_ids[row * 2 + 1]) ? 1u : 0u;
  }
}

}  // namespace

int sampler_slices(int vocab) {
  // About 1000 values per warp: 31 slices at the 248 320-wide vocabulary, fewer for small rows.
  int slices = (vocab + 8 * 1024 - 1) / (8 * 1024);
  return slices < 1 ? 1 : slices > 32 ? 32 : slices;
}

size_t sampler_scratch_bytes(int rows, int vocab) {
  return static_cast<size_t>(rows) * sampler_slices(vocab) * kList * sizeof(uint64_t) +
         static_cast<size_t>(rows) * sizeof(unsigned int) + 8;
}

cudaError_t launch_sampler(cudaStream_t stream, const SamplerParams& p) {
  return launch_kernel(sampler_kernel, dim3(sampler_slices(p.vocab), p.rows), dim3(kThreads), 0,
                       stream, p);
}

}  // namespace tk100
