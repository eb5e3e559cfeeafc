// Contractions of more than a few dozen tokens on persistent CTA pairs (tcgen05 cta_group::2):
// FP8 projection, FP8 gate/up + SwiGLU, NVFP4 projection, NVFP4 gate/up + SwiGLU (+ NVFP4 form).
//
// A pair tile is 256 weight rows (128 per CTA, the UMMA "A" operand) x N tokens, N chosen per launch: a
// multiple of 32 up to 256 for FP8 (a ragged token count costs at most 31 padded tokens a tile), 128 or
// 256 for NVFP4: activation scales are stored, copied and addressed in whole tiles of 128 tokens.  Each
// CTA loads its 128 weight rows and half of the tokens; one pair per two SMs stays resident and walks
// its share of the tiles (token tiles fastest: the pairs that run together read the same weights).
//
//   warp 0     TMA producer, one ring across all tiles of the pair (as many stages as fit 209 KB, FP8 with one tile per pair 225)
//   warp 1     even CTA: scale copies (NVFP4) and MMAs for both CTAs
//   warps 2-   epilogue: two (NVFP4 SwiGLU: four) warps per TMEM lane quadrant, alternate 32-token batches
//
// Two accumulators in TMEM let the epilogue of one tile run under the MMAs of the next.  FP8: two times
// 256 columns.  NVFP4 keeps 128 columns for scale factors (two stages of 4 x 16), which leaves 384: two
// 256-token accumulators overlap by 128 columns, and the epilogue drains those first and hands them
// over while it still works on the rest.
//
// SwiGLU: a CTA's 128 rows are 64 gate and 64 up rows of the same outputs, 16 gate + 16 up rows in
// every 32-lane quadrant (a 4-D tensor map gathers them, the scale map does the same with the lanes
// of a scale chunk).  Read back as 16-lane fragments, gate and up of an output land in the same thread,
// and the 16 outputs a quadrant makes per token are one NVFP4 block, so their quantisation is local to
// one thread after the transposition through 2 KB of shared memory that the 16-byte output stores
// need anyway (stmatrix.trans; with 2-byte shared stores and a scale load per value the epilogue of a
// 256-token tile took 6.1 us instead of ~2).
//
// Few tiles (T tiles on P pairs, T <= P / 2), or with NVFP4 few left over by rounds of whole tiles: the S pairs
// of a cluster split K of one; each CTA parks the token batches other splits finish in its own ring, one cluster
// barrier, and every split adds its batches over distributed shared memory in split order (fixed, so
// bit-reproducible).  No global scratch, so launches on several streams of one context stay independent.
//
// No load is shared through multicast: every CTA fetches its own operands.
#include <type_traits>

#include "common.cuh"
#include "kernels.h"
#include "ptx.cuh"

namespace tk100 {

namespace {

constexpr int kRows = 128;         // weight rows per CTA
constexpr int kStageKBytes = 128;  // K bytes per row and stage (128 FP8 or 256 FP4 elements)
constexpr int kWTile = kRows * kStageKBytes;
constexpr int kSfTile = 2048;      // scales of 128 rows x 16 groups
constexpr int kMaxStages = 12;
constexpr int kBatch = 32;         // tokens an epilogue warp handles at a time
// Epilogue warps.  SwiGLU with the quantisation behind it is a long dependent chain per value, and eight warps
// did not get through a 256-token NVFP4 tile under the next tile's MMAs: gate/up of 512 tokens 47.5 -> 44.7 us
// with sixteen, 301 tokens 45.2 -> 41.1, 2048 tokens 160.5 -> 157.5.  FP8 tiles have twice the MMA time per value;
// there sixteen warps and the 96 registers they leave were slower (512 tokens 66.0 -> 68.6 us).
__host__ __device__ constexpr int epilogue_warps(bool nv, bool swiglu) { return nv && swiglu ? 16 : 8; }
__host__ __device__ constexpr int block_threads(bool nv, bool swiglu) { return 64 + 32 * epilogue_warps(nv, swiglu); }
// transposition space of a warp: 32 rows (SwiGLU: 16 outputs) of 2 bytes per token
__host__ __device__ constexpr int staging_per_warp(bool swiglu) { return kBatch * (swiglu ? 32 : 64); }
constexpr int kStagingBytes = epilogue_warps(false, false) * staging_per_warp(false);
static_assert(epilogue_warps(true, true) * staging_per_warp(true) == kStagingBytes, "one ring size for all kernels");
constexpr uint32_t kTmemCols = 512;
constexpr uint32_t kSfCols = 128;      // NVFP4: two stages of scale columns
constexpr uint32_t kSfStageCols = 64;  // per stage: 4 K steps x 16 (4 weight + up to 8 token columns)
constexpr size_t kSmemLimit = 227 * 1024;

struct Control {
  uint64_t full[kMaxStages];
  uint64_t empty[kMaxStages];
  uint64_t acc_full[2];
  uint64_t acc_empty[2];
  uint32_t tmem_base;
  uint32_t pad;
};

// Ring and transposition space.  With one tile per pair the space lies over the ring's end: the epilogue starts
// when every stage has been read.
constexpr size_t kRingBytes = (kSmemLimit - 1024 - sizeof(Control)) / 1024 * 1024;

__device__ __forceinline__ uint4 lds128(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
  return v;
}
__device__ __forceinline__ void sts128(uint32_t addr, const uint4& v) {
  asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}

template <int N>
using Int = std::integral_constant<int, N>;

// SPLIT: the pairs of a cluster split K, of every tile or of those that rounds of whole ones leave (SwiGLU never does).  A
// kernel of its own: with that code in it (158 registers instead of 96) unsplit launches took 0.2 to 0.6 us longer (NVFP4
// down, K 4352, 301 / 777 tokens 9.9 / 15.6 us, 10.4 / 16.2 with it; FP8 5120 x 6144, 301 tokens 12.9, 13.2).
template <bool NV, bool SWIGLU, bool SPLIT>
__global__ void __launch_bounds__(block_threads(NV, SWIGLU), 1)
    pair_gemm_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_a,
                     const __grid_constant__ CUtensorMap map_wsf, const __grid_constant__ CUtensorMap map_asf,
                     const __grid_constant__ PairGemmParams p) {
  constexpr int EW = epilogue_warps(NV, SWIGLU);
  constexpr int PARTS = EW / 4;  // warps that share a TMEM lane quadrant, on alternate batches
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  Control* ctl = reinterpret_cast<Control*>(smem + kRingBytes);

  const int warp = warp_index(), lane = threadIdx.x & 31;
  const uint32_t cta = cluster_cta_rank();
  const uint32_t rank = cta & 1u;        // 0 = even CTA of its pair (issues the MMAs)
  const uint32_t leader = cta & ~1u;     // the pair's even CTA
  const int split = static_cast<int>(cta >> 1);
  // With SwiGLU p.splits is 1.  As a constant it brings the first weight requests forward by 0.2 us, in front of the rows
  // of a norm that ran before: NVFP4 MLP of 100 tokens 39.7 us, constant 40.0; layer slice of 48 tokens 61.2 and 60.6.
  const int splits = SPLIT || SWIGLU ? p.splits : 1;
  const int worker = static_cast<int>(blockIdx.x) / (2 * splits);
  const int workers = static_cast<int>(gridDim.x) / (2 * splits);
  const int tok_tile = p.tok_tile;
  const int tiles = p.tiles_m * p.row_units;
  const int k0 = static_cast<int>(static_cast<long long>(split) * p.nkb / splits);
  const int k1 = static_cast<int>(static_cast<long long>(split + 1) * p.nkb / splits);
  // NVFP4 projections: behind `rounds` rounds of whole tiles on all pairs the cluster's pairs split K of one more.
  constexpr bool TAILS = NV && SPLIT;
  const int rounds = TAILS ? p.rounds : 0;
  const int whole = rounds * workers * splits;
  // The n-th tile of this pair: index and blocks of K.
  auto tile_at = [&](int n, int& t, int& first_kb, int& last_kb) {
    first_kb = k0;
    last_kb = k1;
    if (TAILS && n < rounds) {
      t = static_cast<int>(blockIdx.x >> 1) + n * workers * splits;
      first_kb = 0;
      last_kb = p.nkb;
      return true;
    }
    t = TAILS ? whole + worker : worker + n * workers;
    return t < tiles && (!TAILS || n == rounds);
  };
  const int stages = p.stages;
  const uint32_t stage_bytes = static_cast<uint32_t>(p.stage_bytes);
  const uint32_t off_b = kWTile;
  const uint32_t off_sfa = off_b + static_cast<uint32_t>(tok_tile) * 64u;
  const uint32_t off_sfb = off_sfa + kSfTile;
  const int chunks_per_tile = p.chunks_per_tile;
  // overlapping accumulators: the second starts where the first has been handed over
  const bool overlap = NV && 2 * tok_tile > static_cast<int>(kTmemCols - kSfCols);
  const uint32_t acc_stride =
      NV ? (overlap ? kTmemCols - kSfCols - static_cast<uint32_t>(tok_tile) : 128u) : 256u;
  const int overlap_batches = overlap ? (tok_tile - static_cast<int>(acc_stride)) / kBatch : 0;

  if (warp == 0 && elect_one()) {
    for (int s = 0; s < stages; ++s) {
      mbar_init(&ctl->full[s], 1);
      mbar_init(&ctl->empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&ctl->acc_full[b], 1);
      mbar_init(&ctl->acc_empty[b], 2 * EW);
    }
    fence_mbar_init();
    prefetch_tensormap(&map_w);
    prefetch_tensormap(&map_a);
    if (NV) {
      prefetch_tensormap(&map_wsf);
      prefetch_tensormap(&map_asf);
    }
  }
  if (warp == 1) {
    tmem_alloc_pair(&ctl->tmem_base, kTmemCols);
    tmem_relinquish_pair();
  }
  tc_fence_before_sync();
  __syncthreads();
  // every CTA's barriers exist before another touches them
  cluster_arrive();
  cluster_wait();
  tc_fence_after_sync();
  const uint32_t tmem = ctl->tmem_base;
  pdl_trigger();

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer
    if (elect_one()) {
      const uint64_t pol_a = l2_policy_evict_last();
      const uint64_t pol_w = p.tiles_m == 1 ? l2_policy_evict_first() : pol_a;
      const uint32_t bar0 = mapa_u32(smem_u32(&ctl->full[0]), leader);
      const int half_tok = tok_tile / 2;
      auto load_w = [&](int s, int kb, int unit) {
        uint8_t* stage = smem + static_cast<uint32_t>(s) * stage_bytes;
        const uint32_t bar = bar0 + static_cast<uint32_t>(s) * 8u;
        if (SWIGLU) {
          tma_load_4d_pair(stage, &map_w, bar, kb * kStageKBytes, static_cast<int>(rank) * 16, 0, unit * 4, pol_w);
          if (NV) {
            tma_load_4d_pair(stage + off_sfa, &map_wsf, bar, 0, static_cast<int>(rank), 0,
                             unit * chunks_per_tile + kb * 4, pol_w);
          }
        } else {
          const int w_tile = 2 * unit + static_cast<int>(rank);
          tma_load_2d_pair(stage, &map_w, bar, kb * kStageKBytes, w_tile * kRows, pol_w);
          if (NV) tma_load_2d_pair(stage + off_sfa, &map_wsf, bar, 0, w_tile * chunks_per_tile + kb * 4, pol_w);
        }
      };
      const int sf_tiles = NV ? tok_tile / kRows : 0;  // 128-token scale tiles of a token tile
      const uint32_t bytes = 2u * (kWTile + static_cast<uint32_t>(tok_tile) * 64u +
                                   (NV ? kSfTile * static_cast<uint32_t>(1 + sf_tiles) : 0u));
      auto load_b = [&](int s, int kb, int tok0) {
        uint8_t* stage = smem + static_cast<uint32_t>(s) * stage_bytes;
        const uint32_t bar = bar0 + static_cast<uint32_t>(s) * 8u;
        tma_load_2d_pair(stage + off_b, &map_a, bar, kb * kStageKBytes, tok0 + static_cast<int>(rank) * half_tok,
                         pol_a);
        if (NV) {
          const int first = tok0 / kRows;
          for (int c = 0; c < sf_tiles; ++c) {
            tma_load_2d_pair(stage + off_sfb + c * kSfTile, &map_asf, bar, 0,
                             (first + c) * chunks_per_tile + kb * 4, pol_a);
          }
        }
      };
      bool ok = true, first = true;
      int s = 0, t = 0, kb = 0, kb_end = 0;
      uint32_t phase = 0;
      for (int n = 0; ok && tile_at(n, t, kb, kb_end); ++n) {
        const int unit = t / p.tiles_m;
        const int tok0 = (t - unit * p.tiles_m) * tok_tile;
        if (first) {
          // First pass over the ring: the weights do not depend on the predecessor kernel and are
          // requested before pdl_wait(), the tokens of the same stages follow it.
          const int pre = min(stages, kb_end - kb);
          for (int i = 0; i < pre; ++i) {
            if (rank == 0) mbar_arrive_expect_tx(&ctl->full[i], bytes);
            load_w(i, kb + i, unit);
          }
          pdl_wait();
          for (int i = 0; i < pre; ++i) load_b(i, kb + i, tok0);
          first = false;
          kb += pre;
          s = pre == stages ? 0 : pre;
          phase = pre == stages ? 1u : 0u;
        }
        for (; kb < kb_end; ++kb) {
          ok = mbar_wait(&ctl->empty[s], phase ^ 1u, p.status);
          if (!ok) break;
          if (rank == 0) mbar_arrive_expect_tx(&ctl->full[s], bytes);
          load_w(s, kb, unit);
          load_b(s, kb, tok0);
          if (++s == stages) {
            s = 0;
            phase ^= 1u;
          }
        }
      }
      if (!ok) {
        // Give copies already in flight time to land before shared memory is released.
        for (int i = 0; i < 64; ++i) __nanosleep(1000);
      }
    }
  } else if (warp == 1) {
    // -------------------------------------------------------------- UMMA issuer
    if (rank == 0 && elect_one()) {
      const uint32_t idesc = NV ? umma_idesc_nvfp4(2 * kRows, static_cast<uint32_t>(tok_tile))
                                : umma_idesc_e4m3(2 * kRows, static_cast<uint32_t>(tok_tile));
      const uint16_t both = static_cast<uint16_t>(3u << leader);
      const uint32_t base0 = smem_u32(smem);
      const uint64_t desc_w0 = umma_desc_sw128(base0);
      const uint64_t desc_b0 = umma_desc_sw128(base0 + off_b);
      const uint64_t desc_sfa0 = umma_desc_noswizzle_rows16(base0 + off_sfa);
      const uint64_t desc_sfb0 = umma_desc_noswizzle_rows16(base0 + off_sfb);
      const uint32_t stage_step = stage_bytes >> 4;
      bool ok = true;
      int s = 0, t = 0, kb0 = 0, kb_end = 0;
      uint32_t phase = 0, sf_parity = 0;
      for (int n = 0; ok && tile_at(n, t, kb0, kb_end); ++n) {
        const int b = n & 1;
        // the columns this tile accumulates into have been read: overlapping accumulators wait for
        // the shared columns of the tile before, disjoint ones for the tile two before
        if (overlap ? n >= 1 : n >= 2) {
          ok = overlap ? mbar_wait_cluster(&ctl->acc_empty[b ^ 1], ((n - 1) >> 1) & 1, p.status)
                       : mbar_wait_cluster(&ctl->acc_empty[b], ((n >> 1) - 1) & 1, p.status);
          if (!ok) break;
          tc_fence_after_sync();
        }
        const uint32_t acc = tmem + static_cast<uint32_t>(b) * acc_stride;
        for (int kb = kb0; kb < kb_end; ++kb) {
          ok = mbar_wait(&ctl->full[s], phase, p.status);
          if (!ok) break;
          tc_fence_after_sync();
          const uint64_t step = static_cast<uint64_t>(static_cast<uint32_t>(s) * stage_step);
          const uint64_t desc_w = desc_w0 + step, desc_b = desc_b0 + step;
          if (NV) {
            const uint64_t desc_sfa = desc_sfa0 + step, desc_sfb = desc_sfb0 + step;
            const uint32_t sf = tmem + (kTmemCols - kSfCols) + sf_parity * kSfStageCols;
            sf_parity ^= 1u;
            const int steps = min(4, (p.k - kb * 256) / 64);
#pragma unroll
            for (int k4 = 0; k4 < 4; ++k4) {
              if (k4 < steps) {
                const uint32_t slot = sf + k4 * 16;
                tmem_cp_32x128b_warpx4_pair(slot, desc_sfa + k4 * 32);
                tmem_cp_32x128b_warpx4_pair(slot + 4, desc_sfb + k4 * 32);
                if (tok_tile > kRows) tmem_cp_32x128b_warpx4_pair(slot + 8, desc_sfb + 128 + k4 * 32);
                umma_nvfp4_pair(acc, desc_w + 2 * k4, desc_b + 2 * k4, idesc, slot, slot + 4,
                                (kb > kb0 || k4 > 0) ? 1u : 0u);
              }
            }
          } else {
#pragma unroll
            for (int k4 = 0; k4 < 4; ++k4) {
              umma_f8f6f4_pair(acc, desc_w + 2 * k4, desc_b + 2 * k4, idesc, (kb > kb0 || k4 > 0) ? 1u : 0u);
            }
          }
          umma_commit_pair(&ctl->empty[s], both);
          if (++s == stages) {
            s = 0;
            phase ^= 1u;
          }
        }
        umma_commit_pair(&ctl->acc_full[b], both);  // also releases both epilogues after a failed wait
      }
    }
  } else {
    // ----------------------------------------------------------------- epilogue
    const int ew = warp - 2;
    const int quad = warp & 3;   // TMEM lane quadrant this warp may read
    const int part = ew >> 2;    // which of the quadrant's warps
    const uint32_t stg = smem_u32(smem + kRingBytes - kStagingBytes + ew * staging_per_warp(SWIGLU));
    const uint32_t acc_empty0 = mapa_u32(smem_u32(&ctl->acc_empty[0]), leader);
    const int batches = tok_tile / kBatch;

    pdl_wait();  // activation scales and the output planes belong to the predecessor until now

    // A batch of 32 tokens of this warp's 32 accumulator lanes, as two 16-lane fragments: f[h][4 i + e] is
    // lane 16 h + lane / 4 + 8 (e / 2), token 8 i + 2 (lane % 4) + e % 2.  SwiGLU: h = 0 gate, 1 up.
    const int frow = lane >> 2, fcol = 2 * (lane & 3);

    // Dequantisation scales of this thread's weight rows.
    auto row_scales = [&](int unit, float (&ws)[4]) {
      if (NV) {
#pragma unroll
        for (int m = 0; m < 4; ++m) ws[m] = p.out_scale;
      } else {
#pragma unroll
        for (int m = 0; m < 4; ++m) {
          if (SWIGLU) {
            const int o = unit * kRows + quad * 32 + static_cast<int>(rank) * 16 + frow + 8 * (m & 1);
            ws[m] = bf16_bits_to_f32(p.w_scales[(m >> 1) * p.out_rows + o]);
          } else {
            const int o = (2 * unit + static_cast<int>(rank)) * kRows + quad * 32 + frow + 8 * m;
            ws[m] = o < p.out_rows ? bf16_bits_to_f32(p.w_scales[o]) : 0.0f;
          }
        }
      }
    };

    auto store16 = [&](uint16_t* dst, const uint4& v) {
      if (p.vector_out) {
        *reinterpret_cast<uint4*>(dst) = v;
      } else {
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int q = 0; q < 8; ++q) dst[q] = static_cast<uint16_t>(w[q >> 1] >> ((q & 1) * 16));
      }
    };

    // Scales of this thread's tokens in [t0, t0 + 32); NVFP4 has none.
    auto token_scales = [&](int t0, float2 (&as)[4]) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int tok = t0 + 8 * i + fcol;
        as[i].x = !NV && tok < p.rows ? __ldg(p.act_scales + tok) : 0.0f;
        as[i].y = !NV && tok + 1 < p.rows ? __ldg(p.act_scales + tok + 1) : 0.0f;
      }
    };

    // Finishes tokens [t0, t0 + 32).
    auto finish = [&](const uint32_t (&f)[2][16], int unit, int t0, const float (&ws)[4], const float2 (&as)[4]) {
      const int valid = p.rows - t0;  // > 0
      auto value = [&](int h, int i, int e) {
        const float acc = __uint_as_float(f[h][4 * i + e]);
        const float w = ws[2 * h + (e >> 1)];
        return NV ? __fmul_rn(acc, w) : __fmul_rn(__fmul_rn(acc, (e & 1) ? as[i].y : as[i].x), w);
      };
      if (!SWIGLU) {
        const int col0 = (2 * unit + static_cast<int>(rank)) * kRows + quad * 32;
        if (NV && p.out_f32 != nullptr) {
#pragma unroll
          for (int h = 0; h < 2; ++h) {
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              const int tok = 8 * (j >> 2) + fcol + (j & 1), col = col0 + 16 * h + frow + 8 * ((j >> 1) & 1);
              if (tok < valid && col < p.out_rows) {
                p.out_f32[static_cast<size_t>(t0 + tok) * p.out_rows + col] = value(h, j >> 2, j & 3);
              }
            }
          }
          return;
        }
        // [token][32 rows] through 2 KB of shared memory; the 16-byte pieces of a token are rotated so
        // that eight tokens of one piece fall into different banks
        const uint32_t dst = stg + (lane & 7) * 64 + (((lane >> 3) ^ ((lane >> 1) & 3)) << 4);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          stmatrix_x4_trans(dst + i * 512, pack_bf16x2(value(0, i, 0), value(0, i, 1)),
                            pack_bf16x2(value(0, i, 2), value(0, i, 3)), pack_bf16x2(value(1, i, 0), value(1, i, 1)),
                            pack_bf16x2(value(1, i, 2), value(1, i, 3)));
        }
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int tok = i * 8 + (lane >> 2), c = lane & 3;
          const uint4 v = lds128(stg + tok * 64 + ((c ^ ((tok >> 1) & 3)) << 4));
          const int col = col0 + c * 8;
          if (tok < valid && col < p.out_rows) {  // out_rows is a multiple of 16
            store16(p.out + static_cast<size_t>(t0 + tok) * p.out_rows + col, v);
          }
        }
        __syncwarp();
      } else {
        const int col0 = unit * kRows + quad * 32 + static_cast<int>(rank) * 16;
        uint32_t y[4][2];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
#pragma unroll
          for (int m = 0; m < 2; ++m) {
            float o[2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const float g = value(0, i, 2 * m + e), u = value(1, i, 2 * m + e);
              o[e] = __fmul_rn(NV ? silu_stable(g) : silu_fp8_path(g), u);
            }
            y[i][m] = pack_bf16x2(o[0], o[1]);
          }
        }
        // [token][16 outputs], the two 16-byte pieces of tokens 4..7 of every eight swapped
        const int wt = 8 * (lane >> 4) + (lane & 7);
        const uint32_t dst = stg + wt * 32 + ((((lane >> 3) & 1) ^ ((wt >> 2) & 1)) << 4);
        stmatrix_x4_trans(dst, y[0][0], y[0][1], y[1][0], y[1][1]);
        stmatrix_x4_trans(dst + 512, y[2][0], y[2][1], y[3][0], y[3][1]);
        __syncwarp();
        if (p.out != nullptr) {
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const int tok = i * 16 + (lane >> 1), c = lane & 1;
            const uint4 v = lds128(stg + tok * 32 + ((c ^ ((tok >> 2) & 1)) << 4));
            if (tok < valid) store16(p.out + static_cast<size_t>(t0 + tok) * p.out_rows + col0 + c * 8, v);
          }
        }
        if (NV && p.q_codes != nullptr && lane < valid) {
          // a lane owns one token's block of 16 outputs
          const uint32_t flip = ((lane >> 2) & 1) << 4;
          const uint4 lo = lds128(stg + lane * 32 + flip), hi = lds128(stg + lane * 32 + (flip ^ 16u));
          const uint32_t w[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
          uint32_t scale_code;
          const uint2 codes = nvfp4_quantize_block(w, p.q_divisor, &scale_code);
          const int tok = t0 + lane, groups = p.out_rows >> 4, g = col0 >> 4;
          *reinterpret_cast<uint2*>(p.q_codes + static_cast<size_t>(tok) * (p.out_rows >> 1) + (col0 >> 1)) = codes;
          const size_t off = (static_cast<size_t>(tok >> 7) * (groups >> 2) + (g >> 2)) * 512 +
                             static_cast<size_t>(tok & 31) * 16 + ((tok & 127) >> 5) * 4 + (g & 3);
          p.q_scales[off] = static_cast<uint8_t>(scale_code);
        }
        __syncwarp();
      }
    };

    // parked batches: [batch][quadrant][four 16-byte pieces of both fragments][lane]
    const uint32_t parked = smem_u32(smem) + static_cast<uint32_t>(quad * 4096 + lane * 16);
    constexpr uint32_t kParkedBatch = 16384;
    int t = 0, kb0 = 0, kb_end = 0;
    for (int n = 0; tile_at(n, t, kb0, kb_end); ++n) {
      const int unit = t / p.tiles_m;
      const int tok0 = (t - unit * p.tiles_m) * tok_tile;
      const int b = n & 1;
      // Batches part, part + PARTS, ... in the order in which columns are due.  Token scales are requested a
      // batch ahead: behind the wait every batch of a pair's last tile paid an L2 round trip for them (12288 rows,
      // 256 tokens 20.4 -> 20.1 us, 8192 rows, 301 tokens 15.2 -> 15.0).  A warp's last batch asks for a batch
      // outside the tile: the tokens behind it (checked against the row count, then dropped), and never those in front
      // of the first tile, because only NVFP4 has overlapping accumulators and it reads no token scales.
      auto batch_of = [&](int o) { return (overlap && b == 0) ? batches - 1 - o : o; };
      float ws[4];
      float2 as[4];
      row_scales(unit, ws);
      const bool shared = SPLIT && n == rounds;  // the tile whose K the cluster's pairs split
      if (!shared) token_scales(tok0 + batch_of(part) * kBatch, as);
      if (!mbar_wait(&ctl->acc_full[b], (n >> 1) & 1, p.status)) break;
      tc_fence_after_sync();
      const uint32_t taddr = tmem + (static_cast<uint32_t>(quad * 32) << 16) + static_cast<uint32_t>(b) * acc_stride;
      if (shared) {
        // park the batches other splits finish over the ring, whose loads and reads are all done
        for (int o = part; o < batches; o += PARTS) {
          if (o % splits == split || tok0 + o * kBatch >= p.rows) continue;
          uint32_t f[2][16];
          tmem_ld_16x256b_x4(taddr + o * kBatch, f[0]);
          tmem_ld_16x256b_x4(taddr + (16u << 16) + o * kBatch, f[1]);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const uint32_t* v = &f[j >> 2][4 * (j & 3)];
            sts128(parked + o * kParkedBatch + j * 512, make_uint4(v[0], v[1], v[2], v[3]));
          }
        }
        break;  // the cluster's last tile; finished behind the barrier below
      }
      const int due = overlap ? overlap_batches : batches;  // columns the next tile waits for
      if (part >= due) {
        __syncwarp();
        if (lane == 0) mbar_arrive_remote(acc_empty0 + static_cast<uint32_t>(b) * 8u);
      }
      for (int o = part; o < batches; o += PARTS) {
        const int batch = batch_of(o);
        uint32_t f[2][16];
        tmem_ld_16x256b_x4(taddr + batch * kBatch, f[0]);
        tmem_ld_16x256b_x4(taddr + (16u << 16) + batch * kBatch, f[1]);
        float2 next[4];
        token_scales(tok0 + batch_of(o + PARTS) * kBatch, next);
        tmem_ld_wait();
        if (o < due && o + PARTS >= due) {
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive_remote(acc_empty0 + static_cast<uint32_t>(b) * 8u);
        }
        const int t0 = tok0 + batch * kBatch;
        if (t0 < p.rows) finish(f, unit, t0, ws, as);
#pragma unroll
        for (int i = 0; i < 4; ++i) as[i] = next[i];
      }
    }

    if constexpr (SPLIT) {
      cluster_arrive();
      cluster_wait();
      t = whole + worker;
      if (t < tiles) {
        const int unit = t / p.tiles_m;
        const int tok0 = (t - unit * p.tiles_m) * tok_tile;
        float ws[4];
        row_scales(unit, ws);
        const uint32_t taddr =
            tmem + (static_cast<uint32_t>(quad * 32) << 16) + static_cast<uint32_t>(rounds & 1) * acc_stride;
        // This split's batches are split, split + splits, ...; the quadrant's warps alternate.  All that the S - 1
        // other splits parked of a batch is requested before the first sum (instead of one split after the other;
        // three splits, 256 tokens: NVFP4 down 18.4 -> 18.0 us, FP8 5120 x 6144 16.1 -> 15.8).  The sums run in split
        // order; own values come at place POS of it (addition commutes, so the first two places are one).
        auto add_parts = [&](auto s_const, auto pos_const) {
          constexpr int S = decltype(s_const)::value, POS = decltype(pos_const)::value;
          for (int o = split + part * S; o < batches; o += PARTS * S) {
            const int t0 = tok0 + o * kBatch;
            if (t0 >= p.rows) break;
            uint32_t own[2][16];
            tmem_ld_16x256b_x4(taddr + o * kBatch, own[0]);
            tmem_ld_16x256b_x4(taddr + (16u << 16) + o * kBatch, own[1]);
            float4 parts[S - 1][8];
#pragma unroll
            for (int i = 0; i < S - 1; ++i) {
              const int q = i + (i >= split ? 1 : 0);
              const uint32_t from =
                  mapa_u32(parked, static_cast<uint32_t>(2 * q) + rank) + static_cast<uint32_t>(o) * kParkedBatch;
#pragma unroll
              for (int j = 0; j < 8; ++j) parts[i][j] = ld_cluster_f32x4(from + j * 512);
            }
            float2 as[4];
            token_scales(t0, as);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 32; ++j) {
              const float mine = __uint_as_float(own[j >> 4][j & 15]);
              float acc = 0.0f;
#pragma unroll
              for (int i = 0; i < S; ++i) {
                if (i == POS) acc = __fadd_rn(acc, mine);
                if (i < S - 1) {
                  const float4& v = parts[i][j >> 2];
                  acc = __fadd_rn(acc, (j & 3) == 0 ? v.x : (j & 3) == 1 ? v.y : (j & 3) == 2 ? v.z : v.w);
                }
              }
              own[j >> 4][j & 15] = __float_as_uint(acc);
            }
            finish(own, unit, t0, ws, as);
          }
        };
        static_assert(kPairGemmMaxSplits == 4, "");
        if (splits == 2) add_parts(Int<2>{}, Int<0>{});
        else if (splits == 3 && split < 2) add_parts(Int<3>{}, Int<0>{});
        else if (splits == 3) add_parts(Int<3>{}, Int<2>{});
        else if (split < 2) add_parts(Int<4>{}, Int<0>{});
        else if (split == 2) add_parts(Int<4>{}, Int<2>{});
        else add_parts(Int<4>{}, Int<3>{});
      }
    }
  }
  if (SPLIT && warp < 2) {
    __syncwarp();
    cluster_arrive();
    cluster_wait();
  }

  // Neither CTA of a pair may release shared memory or TMEM while the pair still works on it, nor a
  // split while a peer reads its parked batches (execution order only: nothing here waits for the
  // epilogue's global stores).
  __syncwarp();
  tc_fence_before_sync();
  cluster_arrive_relaxed();
  cluster_wait_relaxed();
  if (warp == 1) {
    __syncwarp();
    tmem_dealloc_pair(tmem, kTmemCols);
  }
}

template <bool NV, bool SWIGLU>
cudaError_t pg_launch(cudaStream_t stream, int workers, const CUtensorMap& w, const CUtensorMap& a,
                      const CUtensorMap& wsf, const CUtensorMap& asf, const PairGemmParams& p) {
  const auto kernel = !SWIGLU && p.splits > 1 ? pair_gemm_kernel<NV, SWIGLU, !SWIGLU> : pair_gemm_kernel<NV, SWIGLU, false>;
  return launch_kernel_cluster(kernel, dim3(2 * p.splits * workers), dim3(block_threads(NV, SWIGLU)), kSmemLimit, stream,
                               dim3(2 * p.splits), w, a, wsf, asf, p);
}

template <bool NV, bool SWIGLU, bool SPLIT>
cudaError_t pg_prepare() {
  return cudaFuncSetAttribute(pair_gemm_kernel<NV, SWIGLU, SPLIT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              static_cast<int>(kSmemLimit));
}

}  // namespace

int pair_gemm_stage_bytes(bool nvfp4, int tok_tile) {
  return kWTile + tok_tile * 64 + (nvfp4 ? kSfTile * (1 + tok_tile / kRows) : 0);
}

int pair_gemm_stages(int stage_bytes, bool one_tile) {
  const int n = static_cast<int>(kRingBytes - (one_tile ? 0 : kStagingBytes)) / stage_bytes;
  return n < kMaxStages ? n : kMaxStages;
}

cudaError_t pair_gemm_prepare(int* max_clusters) {
  cudaError_t e;
  if ((e = pg_prepare<false, false, false>()) != cudaSuccess) return e;
  if ((e = pg_prepare<false, false, true>()) != cudaSuccess) return e;
  if ((e = pg_prepare<false, true, false>()) != cudaSuccess) return e;
  if ((e = pg_prepare<true, false, false>()) != cudaSuccess) return e;
  if ((e = pg_prepare<true, false, true>()) != cudaSuccess) return e;
  if ((e = pg_prepare<true, true, false>()) != cudaSuccess) return e;
  // clusters of 2, 4, 6 and 8 CTAs (one CTA per SM) that are resident at once
  for (int s = 1; s <= kPairGemmMaxSplits; ++s) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * s * 512, 1, 1);
    cfg.blockDim = dim3(block_threads(true, true));
    cfg.dynamicSmemBytes = kSmemLimit;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2 * s;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int clusters = 0;
    e = cudaOccupancyMaxActiveClusters(&clusters, pair_gemm_kernel<true, true, false>, &cfg);
    if (e != cudaSuccess) {
      (void)cudaGetLastError();
      clusters = 0;
    }
    if (clusters <= 0 && s == 1) {  // no answer: one pair per two SMs
      int device = 0, sms = 0;
      if ((e = cudaGetDevice(&device)) != cudaSuccess) return e;
      if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device)) != cudaSuccess) return e;
      clusters = sms / 2;
    }
    max_clusters[s] = clusters;
  }
  return cudaSuccess;
}

cudaError_t launch_pair_gemm(cudaStream_t stream, bool nvfp4, bool swiglu, int workers, const CUtensorMap& map_w,
                             const CUtensorMap& map_a, const CUtensorMap& map_wsf, const CUtensorMap& map_asf,
                             const PairGemmParams& p) {
  if (nvfp4) {
    return swiglu ? pg_launch<true, true>(stream, workers, map_w, map_a, map_wsf, map_asf, p)
                  : pg_launch<true, false>(stream, workers, map_w, map_a, map_wsf, map_asf, p);
  }
  return swiglu ? pg_launch<false, true>(stream, workers, map_w, map_a, map_wsf, map_asf, p)
                : pg_launch<false, false>(stream, workers, map_w, map_a, map_wsf, map_asf, p);
}

}  // namespace tk100
