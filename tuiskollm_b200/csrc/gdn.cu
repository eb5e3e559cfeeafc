// Gated-delta-net decode step either side of the FP8 GDN projections: the control mat-vecs and
// the width-4 causal convolution ("prepare"), and the FP32 state recurrence with its gated
// RMSNorm.  Replaces tuisko-kernels-sm120/src/gdn/prepare.rs:41-102 (bodies
// src/device/gdn_prepare.rs:34-142) and src/gdn/recurrence.rs:41-88 (body
// src/device/gdn_recurrence.rs:42-186).
//
// Both steps are HBM- and latency-bound byte movers (0.98 MB of control weights, 6.29 MB of
// state per token), so the work here is in how the bytes move:
//   * prepare is ONE launch: CTAs [0, 96) each own one control row for all tokens of the batch
//     (the weight row is read once, 16 bytes per load), the remaining CTAs run the convolution
//     on 8 channels per thread (history, weights, input and output as 16-byte accesses).  Tokens and columns
//     that do not exist are skipped (multiplied as zeros they were most of a one-token launch), products run
//     on fp32 pairs and eight tokens' sums are reduced together: batch 1 3.0 -> 2.3 us, 8 4.5 -> 2.7;
//   * the recurrence gives every (token, value head) a CTA, whose warps own its state rows.  Where every head has
//     an SM to itself (batches up to 3) the rows pass through registers; beyond that through shared memory, as bulk
//     copies that each warp issues, waits for and sends back for itself, so bytes in flight cost no registers.  q
//     and k are normalised by each warp for itself (no barrier in front of the state math), and the one value that
//     couples the rows -- the mean square of the 128 recurrent outputs -- meets at a CTA barrier.
#include "common.cuh"
#include "kernels.h"
#include "ptx.cuh"

namespace tk100 {
namespace {

constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLn2 = 0.6931471805599453f;

__device__ __forceinline__ float ex2_approx(float v) {
  float r;
  asm("ex2.approx.f32 %0, %1;" : "=f"(r) : "f"(v));
  return r;
}
__device__ __forceinline__ float lg2_approx(float v) {
  float r;
  asm("lg2.approx.f32 %0, %1;" : "=f"(r) : "f"(v));
  return r;
}
__device__ __forceinline__ float rsqrt_approx(float v) {
  float r;
  asm("rsqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(v));
  return r;
}
// The reference's forms (device/gdn_prepare.rs:14-31): exp through ex2.approx, an IEEE divide.
__device__ __forceinline__ float fast_exp(float v) { return ex2_approx(v * kLog2e); }
__device__ __forceinline__ float sigmoid_ref(float v) { return __fdiv_rn(1.0f, 1.0f + fast_exp(-v)); }
__device__ __forceinline__ float softplus_ref(float v) {
  return v > 20.0f ? v : lg2_approx(1.0f + fast_exp(v)) * kLn2;
}

__device__ __forceinline__ uint4 ldg16(const void* p) {
  return __ldg(reinterpret_cast<const uint4*>(p));
}

// Dot product of the 8 values packed in a uint4 with 8 widened ones, even and odd columns apart.
__device__ __forceinline__ F32x2 dot8(const uint4& x, const F32x2 (&w)[4], F32x2 acc) {
  acc = fma2(bf16x2_to_f32x2(x.x), w[0], acc);
  acc = fma2(bf16x2_to_f32x2(x.y), w[1], acc);
  acc = fma2(bf16x2_to_f32x2(x.z), w[2], acc);
  return fma2(bf16x2_to_f32x2(x.w), w[3], acc);
}

constexpr int kPrepThreads = 320;
constexpr int kPrepWarps = kPrepThreads / 32;
constexpr int kMaxChunksPerThread = 4;  // hidden <= 320 * 4 * 8 = 10240

// --------------------------------------------------------------------------- prepare
// CTAs [0, 2 * control_rows): one fused control row each, all tokens.
// CTAs beyond: the convolution, 8 channels per thread.
__global__ void __launch_bounds__(kPrepThreads) gdn_prepare_kernel(GdnPrepareParams p) {
  __shared__ float partial[kPrepWarps][kGdnMaxBatch];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int control_ctas = 2 * p.control_rows;

  if (static_cast<int>(blockIdx.x) < control_ctas) {
    const int row = blockIdx.x;
    const int chunks = p.hidden / 8;
    // Weights do not depend on the predecessor: request them before waiting for it.
    uint4 w[kMaxChunksPerThread];
#pragma unroll
    for (int c = 0; c < kMaxChunksPerThread; ++c) {
      const int chunk = tid + c * kPrepThreads;
      w[c] = chunk < chunks ? ldg16(p.control_weights + static_cast<size_t>(row) * p.hidden + chunk * 8)
                            : make_uint4(0, 0, 0, 0);
    }
    pdl_wait();
    pdl_trigger();
    // Two chunk columns at a time: all tokens' loads of a column pair are requested before the
    // first FMA on them, so a batch of 8 costs one round trip to L2 per pair, not eight.  Columns and tokens
    // that do not exist cost nothing (multiplied as zeros they were most of a one-token launch).
    F32x2 acc2[kGdnMaxBatch];
#pragma unroll
    for (int t = 0; t < kGdnMaxBatch; ++t) acc2[t] = f32x2_splat(0.0f);
#pragma unroll
    for (int c0 = 0; c0 < kMaxChunksPerThread; c0 += 2) {
      if (c0 * kPrepThreads >= chunks) break;
      uint4 x[kGdnMaxBatch][2];
#pragma unroll
      for (int t = 0; t < kGdnMaxBatch; ++t) {
        if (t < p.batch) {
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            const int chunk = tid + (c0 + c) * kPrepThreads;
            x[t][c] = chunk < chunks ? ldg16(p.input + static_cast<size_t>(t) * p.hidden + chunk * 8)
                                     : make_uint4(0, 0, 0, 0);
          }
        }
      }
      F32x2 wf[2][4];
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        wf[c][0] = bf16x2_to_f32x2(w[c0 + c].x);
        wf[c][1] = bf16x2_to_f32x2(w[c0 + c].y);
        wf[c][2] = bf16x2_to_f32x2(w[c0 + c].z);
        wf[c][3] = bf16x2_to_f32x2(w[c0 + c].w);
      }
#pragma unroll
      for (int t = 0; t < kGdnMaxBatch; ++t) {
        if (t < p.batch) acc2[t] = dot8(x[t][1], wf[1], dot8(x[t][0], wf[0], acc2[t]));
      }
    }
    float acc[kGdnMaxBatch];
#pragma unroll
    for (int t = 0; t < kGdnMaxBatch; ++t) {
      const float2 halves = f32x2_parts(acc2[t]);
      acc[t] = halves.x + halves.y;
    }
    if (p.batch == 1) {
      const float sum = warp_sum(acc[0]);
      if (lane == 0) partial[warp][0] = sum;
    } else {
      static_assert(kGdnMaxBatch == 8, "the exchanges below are for eight sums");
      // Eight sums over 32 lanes in nine exchanges: at offsets 16, 8 and 4 a lane hands half of its tokens to
      // its partner, and lane l ends with token l / 4.
#pragma unroll
      for (int o = 16, count = 4; o > 2; o >>= 1, count >>= 1) {
        const bool upper = (lane & o) != 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          if (j < count) {
            const float give = upper ? acc[j] : acc[j + count], keep = upper ? acc[j + count] : acc[j];
            acc[j] = keep + __shfl_xor_sync(0xffffffffu, give, o);
          }
        }
      }
      acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], 2);
      acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], 1);
      if ((lane & 3) == 0) partial[warp][lane >> 2] = acc[0];
    }
    __syncthreads();
    if (tid < p.batch) {
      float sum = partial[0][tid];
#pragma unroll
      for (int i = 1; i < kPrepWarps; ++i) sum += partial[i][tid];
      if (row < p.control_rows) {
        const float control = sum + bf16_bits_to_f32(p.dt_bias[row]);
        p.log_decay[tid * p.control_rows + row] =
            -fast_exp(bf16_bits_to_f32(p.a_log[row])) * softplus_ref(control);
      } else {
        p.beta[tid * p.control_rows + row - p.control_rows] = sigmoid_ref(sum);
      }
    }
    return;
  }

  // Convolution: 8 adjacent channels of one token per thread.
  const int groups = p.qkv_rows / 8;
  const int index = (static_cast<int>(blockIdx.x) - control_ctas) * kPrepThreads + tid;
  pdl_wait();
  pdl_trigger();
  if (index >= p.batch * groups) return;
  const int token = index / groups;
  const int channel = (index - token * groups) * 8;
  const size_t state_row = p.state_rows[token];
  uint16_t* hist = p.history + (state_row * p.qkv_rows + channel) * 3;  // 48 bytes, 16-aligned
  const uint4 cur4 = ldg16(p.projected + static_cast<size_t>(token) * p.input_rows + channel);
  const uint4 h4[3] = {*reinterpret_cast<const uint4*>(hist), *reinterpret_cast<const uint4*>(hist + 8),
                       *reinterpret_cast<const uint4*>(hist + 16)};
  uint4 w4[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) w4[i] = ldg16(p.convolution_weights + static_cast<size_t>(channel) * 4 + i * 8);

  const uint32_t hw[12] = {h4[0].x, h4[0].y, h4[0].z, h4[0].w, h4[1].x, h4[1].y,
                           h4[1].z, h4[1].w, h4[2].x, h4[2].y, h4[2].z, h4[2].w};
  const uint32_t ww[16] = {w4[0].x, w4[0].y, w4[0].z, w4[0].w, w4[1].x, w4[1].y, w4[1].z, w4[1].w,
                           w4[2].x, w4[2].y, w4[2].z, w4[2].w, w4[3].x, w4[3].y, w4[3].z, w4[3].w};
  const uint32_t cw[4] = {cur4.x, cur4.y, cur4.z, cur4.w};
  auto half_of = [](const uint32_t* words, int i) -> uint32_t {
    return (words[i >> 1] >> ((i & 1) * 16)) & 0xffffu;
  };
  uint32_t new_hist[24];
  uint32_t out_bits[8];
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    const uint32_t h0 = half_of(hw, 3 * c), h1 = half_of(hw, 3 * c + 1), h2 = half_of(hw, 3 * c + 2);
    const uint32_t cur = half_of(cw, c);
    new_hist[3 * c] = h1;
    new_hist[3 * c + 1] = h2;
    new_hist[3 * c + 2] = cur;
    // Same association as the reference: w0*h0 + (w1*h1 + (w2*h2 + w3*cur)), each step one FMA.
    const float sum = fmaf(
        bf16_bits_to_f32(half_of(ww, 4 * c)), bf16_bits_to_f32(h0),
        fmaf(bf16_bits_to_f32(half_of(ww, 4 * c + 1)), bf16_bits_to_f32(h1),
             fmaf(bf16_bits_to_f32(half_of(ww, 4 * c + 2)), bf16_bits_to_f32(h2),
                  bf16_bits_to_f32(half_of(ww, 4 * c + 3)) * bf16_bits_to_f32(cur))));
    out_bits[c] = f32_to_bf16_bits(sum * sigmoid_ref(sum));
  }
  uint4 s[3];
  uint32_t* sw = reinterpret_cast<uint32_t*>(s);
#pragma unroll
  for (int i = 0; i < 12; ++i) sw[i] = new_hist[2 * i] | (new_hist[2 * i + 1] << 16);
  *reinterpret_cast<uint4*>(hist) = s[0];
  *reinterpret_cast<uint4*>(hist + 8) = s[1];
  *reinterpret_cast<uint4*>(hist + 16) = s[2];
  uint4 o;
  o.x = out_bits[0] | (out_bits[1] << 16);
  o.y = out_bits[2] | (out_bits[3] << 16);
  o.z = out_bits[4] | (out_bits[5] << 16);
  o.w = out_bits[6] | (out_bits[7] << 16);
  *reinterpret_cast<uint4*>(p.convolved + static_cast<size_t>(token) * p.qkv_rows + channel) = o;
}

// ------------------------------------------------------------------------ recurrence
constexpr int kHeadDim = 128;
constexpr int kKeyHeads = 16;
constexpr int kValueHeads = 48;
constexpr int kQkWidth = kKeyHeads * kHeadDim;
constexpr int kRecWarps = 16;
constexpr int kRecThreads = 32 * kRecWarps;
constexpr int kRecRows = kHeadDim / kRecWarps;  // state rows of a warp
constexpr int kRecGroup = 4;                    // rows whose reductions run side by side
constexpr int kRecTileBytes = kHeadDim * kHeadDim * 4;
constexpr float kRmsEpsilon = 1.0e-6f;
constexpr float kDeltaScale = 0.08838835f;  // 1 / sqrt(128)

__device__ __forceinline__ float dot4(const float4& a, const float4& b) {
  return fmaf(a.x, b.x, fmaf(a.y, b.y, fmaf(a.z, b.z, a.w * b.w)));
}

// Four BF16 values at p (8-byte aligned) as floats.
__device__ __forceinline__ float4 load_bf16x4(const uint16_t* p) {
  const uint2 w = __ldg(reinterpret_cast<const uint2*>(p));
  return make_float4(bf16x2_lo(w.x), bf16x2_hi(w.x), bf16x2_lo(w.y), bf16x2_hi(w.y));
}

// One CTA per (token, value head); a warp owns kRecRows consecutive state rows.  THROUGH_SHARED: it brings them to
// shared memory with one bulk copy, updates them there and sends them back with another, so no register holds a
// state byte in flight and two CTAs share an SM.  Otherwise the rows go through registers: no barrier and no trip
// through shared memory on the chain, but one CTA per SM, so it is taken where every head has an SM to itself.
// The value that couples the rows, the mean square of the head's outputs, meets at a CTA barrier.
template <bool THROUGH_SHARED>
__global__ void __launch_bounds__(kRecThreads, THROUGH_SHARED ? 2 : 1) gdn_recurrence_kernel(GdnRecurrenceParams p) {
  constexpr uint32_t kBytes = kRecRows * kHeadDim * 4;
  extern __shared__ __align__(128) float tile[];  // THROUGH_SHARED: the head's state
  __shared__ float squares[kRecWarps];
  __shared__ float recurrent[kHeadDim];
  __shared__ uint64_t landed[kRecWarps];

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int token = blockIdx.x / kValueHeads;
  const int value_head = blockIdx.x - token * kValueHeads;
  const int key_head = value_head / (kValueHeads / kKeyHeads);
  const int row0 = warp * kRecRows;
  float* rows = tile + row0 * kHeadDim;

  if (THROUGH_SHARED && lane == 0) {
    mbar_init(&landed[warp], 1);
    fence_mbar_init();
  }
  pdl_wait();
  pdl_trigger();

  const size_t state_row = p.state_rows[token];
  float* state = p.state + ((state_row * kValueHeads + value_head) * kHeadDim + row0) * kHeadDim;
  float4 old[THROUGH_SHARED ? 1 : kRecRows];
  if constexpr (THROUGH_SHARED) {
    if (lane == 0) {
      mbar_arrive_expect_tx(&landed[warp], kBytes);
      // No L2 policy: the rows are not read again before the next token.  Over eight layers in turn (920 MB of
      // weights, up to 25 MB of state each) evict_first and evict_last gave the same times within 1.5 %.
      bulk_load_1d(rows, state, kBytes, &landed[warp]);
    }
    __syncwarp();
  } else {
#pragma unroll
    for (int i = 0; i < kRecRows; ++i) old[i] = *reinterpret_cast<const float4*>(state + i * kHeadDim + lane * 4);
  }

  const uint16_t* token_qkv = p.qkv + static_cast<size_t>(token) * p.qkv_rows;
  float4 q = load_bf16x4(token_qkv + key_head * kHeadDim + lane * 4);
  float4 k = load_bf16x4(token_qkv + kQkWidth + key_head * kHeadDim + lane * 4);
  // lane i holds the value of the warp's row i
  const uint16_t* values = token_qkv + 2 * kQkWidth + value_head * kHeadDim + row0;
  const float my_value = lane < kRecRows ? bf16_bits_to_f32(__ldg(values + lane)) : 0.0f;
  const int control = token * kValueHeads + value_head;
  const float decay = ex2_approx(__ldg(p.log_decay + control) * kLog2e);
  const float beta = __ldg(p.beta + control);

  // The first kHeadDim threads finish the outputs; what they need for that is asked for before the state math.
  float weight = 0.0f, gate = 0.0f;
  if (tid < kHeadDim) {
    weight = bf16_bits_to_f32(__ldg(p.norm_weight + tid));
    gate = bf16_bits_to_f32(__ldg(
        p.projected + static_cast<size_t>(token) * p.input_rows + p.qkv_rows + value_head * kHeadDim + tid));
  }

  // L2 normalisation of q and k over the head (device/gdn_recurrence.rs:79-105); each warp for itself.
  const float q_norm = rsqrt_approx(warp_sum(dot4(q, q)) + kRmsEpsilon);
  const float k_norm = rsqrt_approx(warp_sum(dot4(k, k)) + kRmsEpsilon);
  q.x *= q_norm; q.y *= q_norm; q.z *= q_norm; q.w *= q_norm;
  k.x *= k_norm; k.y *= k_norm; k.z *= k_norm; k.w *= k_norm;

  // One verdict for the warp: every lane updates columns of all its rows, and lane 0 alone sends them back.
  bool ok = true;
  if constexpr (THROUGH_SHARED) ok = __all_sync(0xffffffffu, mbar_wait(&landed[warp], 0, p.status));
  float square = 0.0f;
#pragma unroll
  for (int i0 = 0; i0 < kRecRows; i0 += kRecGroup) {
    float4 s[kRecGroup];
    float sum[kRecGroup];
#pragma unroll
    for (int i = 0; i < kRecGroup; ++i) {
      if constexpr (THROUGH_SHARED) s[i] = *reinterpret_cast<const float4*>(rows + (i0 + i) * kHeadDim + lane * 4);
      else s[i] = old[i0 + i];
      sum[i] = dot4(s[i], k);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
      for (int i = 0; i < kRecGroup; ++i) sum[i] += __shfl_xor_sync(0xffffffffu, sum[i], o);
    }
#pragma unroll
    for (int i = 0; i < kRecGroup; ++i) {
      const float update = beta * (__shfl_sync(0xffffffffu, my_value, i0 + i) - decay * sum[i]);
      s[i].x = fmaf(s[i].x, decay, k.x * update);
      s[i].y = fmaf(s[i].y, decay, k.y * update);
      s[i].z = fmaf(s[i].z, decay, k.z * update);
      s[i].w = fmaf(s[i].w, decay, k.w * update);
      *reinterpret_cast<float4*>((THROUGH_SHARED ? rows : state) + (i0 + i) * kHeadDim + lane * 4) = s[i];
      sum[i] = dot4(s[i], q);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
      for (int i = 0; i < kRecGroup; ++i) sum[i] += __shfl_xor_sync(0xffffffffu, sum[i], o);
    }
#pragma unroll
    for (int i = 0; i < kRecGroup; ++i) {
      sum[i] *= kDeltaScale;
      square = fmaf(sum[i], sum[i], square);
      if (lane == i) recurrent[row0 + i0 + i] = sum[i];
    }
  }
  if (lane == 0) squares[warp] = square;
  // The new rows leave while the head's outputs are finished.
  if constexpr (THROUGH_SHARED) {
    fence_proxy_async_smem();
    __syncwarp();
    if (lane == 0 && ok) {
      bulk_store_1d(state, rows, kBytes);
      bulk_store_commit();
    }
  }
  __syncthreads();

  if (tid < kHeadDim) {
    float total = 0.0f;
#pragma unroll
    for (int i = 0; i < kRecWarps; ++i) total += squares[i];
    const float inverse_rms = rsqrt_approx(total / static_cast<float>(kHeadDim) + kRmsEpsilon);
    const float normalized = recurrent[tid] * inverse_rms * weight;
    const float silu = __fdiv_rn(gate, 1.0f + ex2_approx(-gate * kLog2e));
    p.output[static_cast<size_t>(token) * (kValueHeads * kHeadDim) + value_head * kHeadDim + tid] =
        static_cast<uint16_t>(f32_to_bf16_bits(normalized * silu));
  }
  if (THROUGH_SHARED && lane == 0) {
    bulk_store_wait();  // shared memory stays until the rows are in global memory
    // a wait that gave up: give the copy in flight time to land before shared memory is released
    for (int i = 0; i < 64 && !ok; ++i) __nanosleep(1000);
  }
}

}  // namespace

bool gdn_geometry_ok(int hidden, int control_rows, int qkv_rows, int input_rows) {
  return hidden > 0 && hidden % 8 == 0 && hidden <= kPrepThreads * kMaxChunksPerThread * 8 &&
         control_rows == kValueHeads && qkv_rows == 2 * kQkWidth + kValueHeads * kHeadDim &&
         input_rows == qkv_rows + kValueHeads * kHeadDim;
}

cudaError_t launch_gdn_prepare(cudaStream_t stream, const GdnPrepareParams& p) {
  const int conv_threads = p.batch * (p.qkv_rows / 8);
  const int grid = 2 * p.control_rows + (conv_threads + kPrepThreads - 1) / kPrepThreads;
  return launch_kernel(gdn_prepare_kernel, dim3(grid), dim3(kPrepThreads), 0, stream, p);
}

cudaError_t gdn_recurrence_prepare() {
  return cudaFuncSetAttribute(gdn_recurrence_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kRecTileBytes);
}

cudaError_t launch_gdn_recurrence(cudaStream_t stream, const GdnRecurrenceParams& p, int sm_count) {
  const dim3 grid(p.batch * kValueHeads), block(kRecThreads);
  // Registers / shared memory, prepare and recurrence in sequence: batch 1 5.9 / 6.5 us, 2 6.4 / 8.5, 3 7.0 / 9.0,
  // 4 10.3 / 9.6, 8 14.9 / 13.4 (the recurrence alone 3.6 / 4.2, 3.8 / 4.3, 4.2 / 4.5, 7.4 / 6.8, 11.9 / 10.7).
  if (static_cast<int>(grid.x) <= sm_count)
    return launch_kernel(gdn_recurrence_kernel<false>, grid, block, 0, stream, p);
  return launch_kernel(gdn_recurrence_kernel<true>, grid, block, kRecTileBytes, stream, p);
}

}  // namespace tk100
