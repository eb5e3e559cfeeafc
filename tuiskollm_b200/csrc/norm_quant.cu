// Fused residual-add + zero-centred RMSNorm + per-token activation quantisation.
//
// One CTA owns one token row and keeps it in registers from the first load to the
// last store: x (+ branch) is read once, the rounded residual, the normalised row,
// the E4M3 codes and the fp32 scale are written once.  The reference runs this as
// three launches that each re-read the row from global memory
// (tuisko-kernels-sm120/src/residual_norm.rs:155-226 followed by
// tuisko-kernels-sm120/src/device/fp8_projection.rs:54-126).
//
// Instruction issue bounds it beyond one wave of rows (2048 rows with both quantised forms: 12.7 M warp
// instructions, two thirds of the issue slots, 21.3 us where the 98 MB take 15.3 at the copy rate); below that
// its chain of load, two block reductions and store does (one row 2.6 us).  So every quotient is two operations
// on fp32 pairs (reciprocal_parts), maxima are packed BF16 and reduced as integers, a reduction has one barrier,
// and a row's values stay widened.
//
// Numeric contract (bit-exact parts marked *):
//   res  = bf16_rn(f32(x) + f32(branch))                                  *
//   r    = 1/sqrt(sum(res^2)/H + eps), fp32, fixed summation order
//   y    = bf16_rn(res * r * (1 + w)), evaluated left to right in fp32
//   amax = max |y|; scale = amax == 0 ? 1 : amax / 448   (as the fp32 divide rounds) *
//   code = e4m3_rn_satfinite(y / scale)                  (likewise)          *
// The starred results are bit-exact functions of their inputs; `codes`/`scale`
// are exact with respect to the normalised row this same kernel wrote.
#include <cstdlib>
#include <type_traits>

#include "common.cuh"
#include "kernels.h"
#include "ptx.cuh"

namespace tk100 {

namespace {

constexpr int kMaxChunks = 4;  // 16-byte chunks (8 BF16) per thread

struct alignas(16) Chunk {
  uint32_t w[4];
};

// Optional NVFP4 side output of the fused producer (all null/zero when unused).  `rows` is for PADDED kernels and lies
// here because 4 bytes are free: an argument of its own made 100 bytes of parameters out of 96, with which a launch
// outside a graph takes 3.0 us instead of 2.6.
struct Nvfp4Out {
  uint8_t* codes;   // [rows, hidden/2]
  uint8_t* scales;  // 128-row x 4-group tiles, row = token
  float divisor;    // input global divisor
  int rows;         // of the launch
};

// Sum and max over the CTA, one barrier each.  The sum has a fixed order: a butterfly inside each warp, then
// every thread adds the warps' values in warp order (the zeros behind the last do not change it).  The max is
// over magnitudes as integers (bf16x2_fold).
__device__ __forceinline__ float row_sum(float v, float* scratch) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int warps = (blockDim.x + 31) >> 5;
  v = warp_sum(v);
  if (lane == 0) scratch[warp] = v;
  if (threadIdx.x >= warps && threadIdx.x < 32) scratch[threadIdx.x] = 0.0f;
  __syncthreads();
  float4 f = *reinterpret_cast<const float4*>(scratch);
  float r = __fadd_rn(__fadd_rn(__fadd_rn(f.x, f.y), f.z), f.w);
  for (int i = 4; i < warps; i += 4) {
    f = *reinterpret_cast<const float4*>(scratch + i);
    r = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(r, f.x), f.y), f.z), f.w);
  }
  return r;
}
__device__ __forceinline__ uint32_t row_max(uint32_t v, uint32_t* scratch) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int warps = (blockDim.x + 31) >> 5;
  v = __reduce_max_sync(0xffffffffu, v);
  if (lane == 0) scratch[warp] = v;
  __syncthreads();
  return __reduce_max_sync(0xffffffffu, lane < warps ? scratch[lane] : 0u);
}

// A pair of BF16 values that a thread keeps: in fp32, or packed where the registers do not allow that.
__device__ __forceinline__ void keep_pair(F32x2& v, uint32_t w) { v = bf16x2_to_f32x2(w); }
__device__ __forceinline__ void keep_pair(uint32_t& v, uint32_t w) { v = w; }
__device__ __forceinline__ F32x2 pair_f32(F32x2 v) { return v; }
__device__ __forceinline__ F32x2 pair_f32(uint32_t v) { return bf16x2_to_f32x2(v); }

// PADDED: the grid is filled up to whole clusters (launch_chunks).
template <bool HAS_BRANCH, bool DO_NORM, bool DO_QUANT, int CHUNKS, bool PADDED>
__global__ void __launch_bounds__(CHUNKS == 3 ? 704 : 1024)  // norm_geometry: three chunks on at most 704
    resnorm_quant_kernel(const uint16_t* __restrict__ x, const uint16_t* __restrict__ branch,
                         const uint16_t* __restrict__ weight, uint16_t* __restrict__ residual_out,
                         uint16_t* __restrict__ normalized_out, uint8_t* __restrict__ codes,
                         float* __restrict__ scales, int hidden, float eps, uint32_t* status,
                         const Nvfp4Out nv) {
  __shared__ __align__(16) float sums[32];
  __shared__ uint32_t maxima[32];
  pdl_trigger();
  pdl_wait();  // x / branch may be the predecessor's output
  const int row = blockIdx.x;
  if (PADDED && row >= nv.rows) return;
  const int chunks_per_row = hidden >> 3;
  const size_t row_off = static_cast<size_t>(row) * hidden;

  using Pair = std::conditional_t<CHUNKS <= 2, F32x2, uint32_t>;
  Pair v[CHUNKS][4];  // the row: rounded residual, later the normalised row
  // The norm weight of this thread's columns is requested together with the row (one memory
  // latency less on the chain load -> reduce -> scale -> reduce -> store); with three or four
  // chunks per thread the registers do not allow it and the weight is loaded where it is used.
  constexpr bool EARLY_WEIGHT = DO_NORM && CHUNKS <= 2;
  Chunk wreg[EARLY_WEIGHT ? CHUNKS : 1];
  F32x2 sum = f32x2_splat(0.0f);
  uint32_t m[CHUNKS];  // largest magnitudes of the row to quantise
#pragma unroll
  for (int i = 0; i < CHUNKS; ++i) {
    const int c = threadIdx.x + i * blockDim.x;
    m[i] = 0u;
    if (c < chunks_per_row) {
      if constexpr (EARLY_WEIGHT) wreg[i] = *reinterpret_cast<const Chunk*>(weight + c * 8);
      Chunk a = *reinterpret_cast<const Chunk*>(x + row_off + c * 8);
      if (HAS_BRANCH) {
        Chunk b = *reinterpret_cast<const Chunk*>(branch + row_off + c * 8);
        Chunk r;
#pragma unroll
        for (int j = 0; j < 4; ++j) r.w[j] = f32x2_to_bf16x2(add2(bf16x2_to_f32x2(a.w[j]), bf16x2_to_f32x2(b.w[j])));
        *reinterpret_cast<Chunk*>(residual_out + row_off + c * 8) = r;
        a = r;  // the norm consumes the rounded residual
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        keep_pair(v[i][j], a.w[j]);
        if (DO_NORM) {
          const F32x2 f = pair_f32(v[i][j]);
          sum = fma2(f, f, sum);
        } else {
          m[i] = bf16x2_absmax(m[i], a.w[j]);
        }
      }
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j) keep_pair(v[i][j], 0u);
    }
  }

  if (DO_NORM) {
    const float2 halves = f32x2_parts(sum);
    const float total = row_sum(__fadd_rn(halves.x, halves.y), sums);
    const float mean = __fdiv_rn(total, static_cast<float>(hidden));
    const F32x2 inv_rms = f32x2_splat(__frsqrt_rn(__fadd_rn(mean, eps)));
    const F32x2 one = f32x2_splat(1.0f);
#pragma unroll
    for (int i = 0; i < CHUNKS; ++i) {
      const int c = threadIdx.x + i * blockDim.x;
      if (c < chunks_per_row) {
        Chunk wv;
        if constexpr (EARLY_WEIGHT) wv = wreg[i];
        else wv = *reinterpret_cast<const Chunk*>(weight + c * 8);
        Chunk o;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          o.w[j] = f32x2_to_bf16x2(mul2(mul2(pair_f32(v[i][j]), inv_rms), add2(one, bf16x2_to_f32x2(wv.w[j]))));
          m[i] = bf16x2_absmax(m[i], o.w[j]);
          keep_pair(v[i][j], o.w[j]);  // keep the rounded value for the quantiser
        }
        *reinterpret_cast<Chunk*>(normalized_out + row_off + c * 8) = o;
      }
    }
  }

  if (nv.codes != nullptr) {
    // NVFP4 codes of the (rounded) row for the W4A4 MLP: a 16-column block is the two 8-value
    // chunks of an even/odd thread pair; same arithmetic as nvfp4_quantize_kernel.
    const int groups = hidden >> 4;
#pragma unroll
    for (int i = 0; i < CHUNKS; ++i) {
      const int c = threadIdx.x + i * blockDim.x;  // chunk index; block g = c / 2
      const uint32_t block = bf16x2_absmax(m[i], __shfl_xor_sync(0xffffffffu, m[i], 1));
      if (c < chunks_per_row) {
        const uint32_t sc = nvfp4_scale_code(__uint_as_float(bf16x2_fold(block) << 16), nv.divisor);
        const F32x2 f[4] = {pair_f32(v[i][0]), pair_f32(v[i][1]), pair_f32(v[i][2]), pair_f32(v[i][3])};
        uint32_t packed[1];
        nvfp4_codes(f, nv.divisor, e4m3_to_f32(sc), packed);
        *reinterpret_cast<uint32_t*>(nv.codes + static_cast<size_t>(row) * (hidden >> 1) + c * 4) = packed[0];
        if ((c & 1) == 0) {
          const int g = c >> 1;
          const size_t off = (static_cast<size_t>(row >> 7) * (groups >> 2) + (g >> 2)) * 512 +
                             static_cast<size_t>(row & 31) * 16 + ((row & 127) >> 5) * 4 + (g & 3);
          nv.scales[off] = static_cast<uint8_t>(sc);
        }
      }
    }
  }

  if (DO_QUANT) {
    uint32_t all = m[0];
#pragma unroll
    for (int i = 1; i < CHUNKS; ++i) all = bf16x2_absmax(all, m[i]);
    const float amax = __uint_as_float(row_max(bf16x2_fold(all), maxima) << 16);
    auto store_codes = [&](auto&& pair) {
#pragma unroll
      for (int i = 0; i < CHUNKS; ++i) {
        const int c = threadIdx.x + i * blockDim.x;
        if (c < chunks_per_row) {
          uint32_t q[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) q[j] = pair(pair_f32(v[i][j]));
          *reinterpret_cast<uint2*>(codes + row_off + c * 8) = make_uint2(q[0] | (q[1] << 16), q[2] | (q[3] << 16));
        }
      }
    };
    if (e4m3_amax_is_ordinary(amax)) {
      const float scale = e4m3_scale_ordinary(amax);
      const Reciprocal r = reciprocal_parts(scale);
      const F32x2 hi = f32x2_splat(r.hi), lo = f32x2_splat(r.lo);
      if (threadIdx.x == 0) scales[row] = scale;
      store_codes([&](F32x2 p) { return e4m3_pair_ordinary(p, hi, lo); });
    } else {
      const float scale = e4m3_scale(amax);
      if (threadIdx.x == 0) {
        if (!(amax <= 3.0e38f)) atomicOr(status, STATUS_NONFINITE_INPUT);
        scales[row] = scale;
      }
      store_codes([&](F32x2 p) { return e4m3_pair(p, scale); });
    }
  }
}

template <bool HAS_BRANCH, bool DO_NORM, bool DO_QUANT>
cudaError_t launch_chunks(cudaStream_t stream, int rows, int hidden, int threads, int chunks,
                          const uint16_t* x, const uint16_t* branch, const uint16_t* weight,
                          uint16_t* residual_out, uint16_t* normalized_out, uint8_t* codes,
                          float* scales, float eps, uint32_t* status, const Nvfp4Out& nv) {
  // Norms with a quantiser: 13 to 32 rows in clusters of four, whose CTAs have an SM each.  Alone they pile up on the SMs
  // that the kernel in front frees first, three to an SM, and share what it can load.  Without / with, us:
  //   12288 x 5120 FP8 behind it, 14 / 16 / 24 / 32 rows 13.9 / 14.1 / 15.4 / 15.8, so 13.5 / 13.4 / 14.2 / 15.1 (8192
  //     rows of weights, 16: 10.9, so 11.1); 8192 x 2048, 32 rows 8.4, so 8.1; 12288 x 4096 14.1, 13.0; x 6144 18.4, 17.1;
  //   NVFP4 MLP of 5120 columns, 14 / 16 / 24 / 32 tokens 32.3 / 32.8 / 33.6 / 34.3, so 30.8 / 31.1 / 32.3 / 32.9.
  // Not with fewer rows (8192 x 5120, 12 rows 10.0, so 10.4) or more (48 rows 12.4, so 13.2: clusters share SMs too, and
  // beside another stream's kernel wait for four places), not with wider rows (10240 x 8192 equal, 8192 x 16384, 32 rows
  // 32, so 37) or narrower ones (the norm itself, 512 columns, 1.42, so 1.45).  Shared memory asked for and not used
  // spreads up to a wave of rows, but such a norm waits for a free SM: 32 rows beside another stream's FP8 gate/up 14,
  // so 27, 100 rows beside attention 18, so 34; and 10240 x 8192 behind 32 rows took 23.4 for 20.4.
  if constexpr (DO_NORM && DO_QUANT) {
    if (rows >= 13 && rows <= 32 && hidden >= 2048 && hidden <= 6144 && chunks <= 2) {
      const auto kernel = chunks == 1 ? resnorm_quant_kernel<HAS_BRANCH, DO_NORM, DO_QUANT, 1, true>
                                      : resnorm_quant_kernel<HAS_BRANCH, DO_NORM, DO_QUANT, 2, true>;
      return launch_kernel_cluster(kernel, dim3((rows + 3) & ~3), dim3(threads), 0, stream, dim3(4), x, branch, weight,
                                   residual_out, normalized_out, codes, scales, hidden, eps, status, nv);
    }
  }
#define TK100_LAUNCH(C)                                                                       \
  launch_kernel(resnorm_quant_kernel<HAS_BRANCH, DO_NORM, DO_QUANT, C, false>, dim3(rows), dim3(threads), \
                0, stream, x, branch, weight, residual_out, normalized_out, codes, scales, hidden, \
                eps, status, nv)
  switch (chunks) {
    case 1: return TK100_LAUNCH(1);
    case 2: return TK100_LAUNCH(2);
    case 3: return TK100_LAUNCH(3);
    default: return TK100_LAUNCH(4);
  }
#undef TK100_LAUNCH
}

}  // namespace

namespace {
bool g_pdl = true;
uint32_t g_debug = 0;
unsigned long long* g_stamps = nullptr;
}  // namespace

void read_process_switches() {
  const char* v = std::getenv("TK100_PDL");
  g_pdl = !(v && v[0] == '0');
#ifdef TK100_EXPERIMENT
  const char* d = std::getenv("TK100_DEBUG");
  g_debug = d ? static_cast<uint32_t>(std::atoi(d)) : 0u;
  const char* sp = std::getenv("TK100_STAMPS_PTR");
  g_stamps = sp ? reinterpret_cast<unsigned long long*>(std::strtoull(sp, nullptr, 0)) : nullptr;
#endif
}

bool pdl_enabled() { return g_pdl; }

uint32_t debug_flags() { return g_debug; }

unsigned long long* debug_stamps() { return g_stamps; }

bool norm_geometry(int hidden, int* threads, int* chunks) {
  if (hidden <= 0 || (hidden & 7) != 0) return false;
  const int row_chunks = hidden >> 3;
  // One chunk per thread while the row fits a 1024-thread CTA, warp-multiple CTAs.
  int c = (row_chunks + 1023) / 1024;
  if (c > kMaxChunks) return false;
  // Prefer CTAs of at most 640 threads (three co-resident per SM) when that costs
  // no extra chunk, e.g. 5120 -> 640 x 1, 17408 -> 544 x 4.
  int t = (row_chunks + c - 1) / c;
  if (t > 704 && c < kMaxChunks) {
    c = (row_chunks + 639) / 640;
    if (c > kMaxChunks) c = kMaxChunks;
    t = (row_chunks + c - 1) / c;
  }
  t = (t + 31) & ~31;
  if (t > 1024) return false;
  *threads = t;
  *chunks = c;
  return true;
}

cudaError_t launch_resnorm_quant(cudaStream_t stream, int rows, int hidden, const uint16_t* x,
                                 const uint16_t* branch, const uint16_t* weight,
                                 uint16_t* residual_out, uint16_t* normalized_out, uint8_t* codes,
                                 float* scales, float eps, uint32_t* status, uint8_t* nvfp4_codes,
                                 uint8_t* nvfp4_scales, float nvfp4_divisor) {
  const Nvfp4Out nv{nvfp4_codes, nvfp4_scales, nvfp4_divisor, rows};
  int threads = 0, chunks = 0;
  if (!norm_geometry(hidden, &threads, &chunks)) return cudaErrorInvalidValue;
  const bool has_branch = branch != nullptr;
  const bool do_norm = normalized_out != nullptr;
  const bool do_quant = codes != nullptr;
  // A row per CTA.  Rows beyond one wave of CTAs run better on more of them with fewer threads and more chunks,
  // which are in different phases at once.  The quantiser alone takes four chunks there: 6144 columns (384 threads
  // x 2, four CTAs per SM at 40 registers), two / four chunks: 600 rows 4.6 / 3.8 us, 740 5.4 / 4.1, 2048 10.8 / 7.9;
  // 5120 columns, one / two / four: 600 rows 4.1 / 4.5 / 3.6, 2048 9.4 / 10.0 / 6.8.  With the norm the chunks
  // double; 5120 columns, one / two / four: 512 rows 7.0 / 6.5 / 8.7, 800 9.2 / 9.5 / 10.5, 1024 rows and
  // more equal; 10240 columns, two / four: 600 rows 13.9 / 15.1, 1024 21.8 / 20.5, 2048 38.9 / 36.9.
  if (chunks <= 2) {
    static int sms = 0;
    if (sms == 0) {
      int device = 0;
      if (cudaGetDevice(&device) != cudaSuccess ||
          cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) {
        sms = 148;
      }
    }
    const int resident = !do_norm && chunks == 2 ? 1536 : 2048;  // threads of an SM
    const int wide = do_norm ? 2 * chunks : 4;
    const int narrow = (((hidden >> 3) + wide - 1) / wide + 31) & ~31;
    if (rows > sms * (resident / threads) && narrow >= (do_norm ? 128 : 64)) {
      chunks = wide;
      threads = narrow;
    }
  }
#define TK100_CASE(B, N, Q)                                                                      \
  if (has_branch == B && do_norm == N && do_quant == Q)                                          \
  return launch_chunks<B, N, Q>(stream, rows, hidden, threads, chunks, x, branch, weight,        \
                                residual_out, normalized_out, codes, scales, eps, status, nv)
  TK100_CASE(true, true, true);
  TK100_CASE(true, true, false);
  TK100_CASE(false, true, true);
  TK100_CASE(false, true, false);
  TK100_CASE(false, false, true);
#undef TK100_CASE
  return cudaErrorInvalidValue;
}

}  // namespace tk100
