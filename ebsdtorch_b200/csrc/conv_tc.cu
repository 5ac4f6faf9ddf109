// 3x3 / stride 2 / padding 1 convolution of NHWC bf16 activations on the
// tensor cores without an im2col pass (the proposal network's layers 2-5,
// forward). The patches of a tap are a strided box of the input: for output
// rows h0 .. and all columns, tap (ky, kx) reads input rows 2 h - 1 + ky and
// columns 2 w - 1 + kx, which one 4-D TMA copy with traversal stride 2 gathers
// straight into the swizzled operand tile, zeros outside the image included.
//
// With 32 channels a copy moves 64 bytes a row and the rows are what costs
// (about 5 cycles each), so there, for even sizes, a row is a pair of pixels
// (even and odd column, 128 bytes): one copy per ky of the pairs left of, at and
// between the output columns holds all three kx, kx = 1 and 2 one row below
// kx = 0. Odd sizes take the strided copies.
//
// D[pixel, channel] = sum over taps and channel chunks: A = 128 output pixels
// x 32 or 64 input channels of one tap, B = the weights of that tap (all COUT
// channels on the N side, so no MMA row or column is padding), FP32
// accumulators double-buffered in TMEM; K runs over (tap, channel) in the order
// of the im2col GEMM, 16 at a time, so the results are the same bits. Weights
// that fit stay in shared memory for all of a CTA's tiles.
//   warp 0 TMA producer, warp 1 TMEM and MMAs, warps 2-5 epilogue (bias, ReLU,
//   bf16 and optional FP32 rows; a thread owns one pixel, so its channels are
//   contiguous stores). One persistent CTA per SM over the pixel tiles. Waits
//   and give-up as in gemm_tc.cu.
//
// The im2col route wrote and re-read 9/4 of every activation and padded layer
// 2's 64 channels to 128 rows. Batch 4,096 at 128 x 128 px: layers 2-5 3.49 ms
// with im2col, 0.92 ms here (32 -> 64 channels 0.43, with strided copies 0.66;
// 64 -> 128 0.23, 660 TFLOP/s; 128 -> 256 0.15, 1,059; 256 -> 256 0.11 with its
// FP32 copy, 0.07 without).
#include <algorithm>

#include "common.cuh"

namespace ebsd {

constexpr int CV_THREADS = 192;
constexpr int CV_MAX_STAGES = 16;

// RB: bytes of a row of a weight tile (32 or 64 channels); BN: output channels;
// RES: weights resident in shared memory; PAIR: a row of A holds a pair of
// input pixels (even, odd column) of 32 channels each.
template <int RB, int BN, bool RES, bool PAIR>
struct ConvTile {
  static constexpr int KC = RB / 2;
  static constexpr int A_BYTES = 128 * (PAIR ? 2 * RB : RB), B_BYTES = BN * RB;
  static constexpr int STAGE = A_BYTES + (RES ? 0 : B_BYTES);
  static constexpr int W_BYTES = RES ? 9 * B_BYTES : 0;  // one channel chunk per tap
  static constexpr int FIT = (220 * 1024 - W_BYTES) / STAGE;
  static constexpr int STAGES = FIT < CV_MAX_STAGES ? FIT : CV_MAX_STAGES;
  static constexpr int BARS = 2 * CV_MAX_STAGES + 6;
  static constexpr int SMEM = 1024 + W_BYTES + STAGES * STAGE + 8 * BARS + 16 + BN * 4;
  static_assert(SMEM <= 232448, "shared memory budget");
  static_assert(STAGES >= 3, "pipeline depth");
};

struct ConvParams {
  int tiles, tiles_h;  // pixel tiles; of them per image block
  int wt, ht, nt;      // tile rows per output row, output rows and images of a tile
  int Wo, Ho, B;
  int chunks;          // channel chunks of a tap
  int cin, paired;     // paired: the input map splits rows and columns by parity
  const float* bias;
  __nv_bfloat16* out16;
  float* out32;
  int relu;
  int* status;
  uint64_t wait_ns;
};

__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap* map, int c, int w, int h, int n,
                                            uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(c), "r"(w), "r"(h), "r"(n), "r"(bar)
      : "memory");
}

__device__ __forceinline__ void tma_load_5d(uint32_t dst, const CUtensorMap* map, int c, int w, int hp, int h, int n,
                                            uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.5d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%2, %3, %4, %5, %6}], [%7];" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(c), "r"(w), "r"(hp), "r"(h), "r"(n), "r"(bar)
      : "memory");
}

// As smem_desc_sw128, for rows of 64 bytes with 64-byte swizzling (8-row
// groups 512 bytes apart).
template <int RB>
__device__ __forceinline__ uint64_t conv_desc(uint32_t saddr) {
  if constexpr (RB == 128) return smem_desc_sw128(saddr);
  return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(512 >> 4) << 32) |
         ((uint64_t)1 << 46) | ((uint64_t)4 << 61);
}

// 128-byte rows starting `row` rows into a tile: the swizzle follows the shared
// memory address, so a tile may be entered at any row.
__device__ __forceinline__ uint64_t pair_desc(uint32_t tile, int row, int byte) {
  return smem_desc_sw128(tile + row * 128 + byte);
}

template <int RB, int BN, bool RES, bool PAIR>
__global__ void __launch_bounds__(CV_THREADS, 1)
    k_conv_tc(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmW, const ConvParams p) {
  using T = ConvTile<RB, BN, RES, PAIR>;
  constexpr int STAGES = T::STAGES;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_s = smem_u32(smem_raw);
  uint8_t* smem = smem_raw + ((1024u - (raw_s & 1023u)) & 1023u);
  const uint32_t wbase = smem_u32(smem), sbase = wbase + T::W_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + T::W_BYTES + STAGES * T::STAGE);
  const uint32_t bar0 = smem_u32(bars);
  auto full_bar = [&](int s) { return bar0 + 8u * s; };
  auto empty_bar = [&](int s) { return bar0 + 8u * (CV_MAX_STAGES + s); };
  auto accf_bar = [&](int a) { return bar0 + 8u * (2 * CV_MAX_STAGES + a); };
  auto acce_bar = [&](int a) { return bar0 + 8u * (2 * CV_MAX_STAGES + 2 + a); };
  const uint32_t w_bar = bar0 + 8u * (2 * CV_MAX_STAGES + 4), drain_bar = w_bar + 8u;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + T::BARS);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  float* bias_s = reinterpret_cast<float*>(tmem_slot + 4);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rows = p.wt * p.ht * p.nt, k_iters = PAIR ? 3 : 9 * p.chunks;
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(accf_bar(a), 1);
      mbar_init(acce_bar(a), 128);
    }
    mbar_init(w_bar, 1);
    mbar_init(drain_bar, 1);
    *abort_flag = 0;
    fence_mbar_init();
  }
  for (int c = threadIdx.x; c < BN; c += CV_THREADS) bias_s[c] = p.bias ? p.bias[c] : 0.0f;
  if (warp == 0 && lane == 0) {
    prefetch_tmap(&tmX);
    prefetch_tmap(&tmW);
  }
  if (warp == 1) tmem_alloc(smem_u32(tmem_slot), 2 * BN);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(tmem_slot);
  const uint64_t wait_ns = p.wait_ns;
  int prod_stage = 0;
  uint32_t prod_phase = 0;
  int64_t issued = 0;
  bool any_mma = false, w_issued = false;
  auto give_up = [&]() {
    *abort_flag = 1;
    atomicExch(p.status, EBSD_DEVICE_TIMEOUT);
  };

  if (warp == 0) {
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      if constexpr (RES) {
        mbar_arrive_expect_tx(w_bar, T::W_BYTES);
        for (int k = 0; k < 9; ++k) tma_load_2d(wbase + k * T::B_BYTES, &tmW, k * T::KC, 0, w_bar);
        w_issued = true;
      }
      const uint32_t bytes = (uint32_t)rows * (T::A_BYTES / 128) + (RES ? 0 : T::B_BYTES);
      for (int t = blockIdx.x; t < p.tiles && ok; t += gridDim.x) {
        const int nb = t / p.tiles_h, n0 = nb * p.nt, h0 = (t - nb * p.tiles_h) * p.ht;
        for (int tap = 0; tap < (PAIR ? 3 : 9) && ok; ++tap) {
          const int ky = PAIR ? tap : tap / 3, kx = tap - 3 * ky;
          for (int c = 0; c < p.chunks; ++c) {
            if (!mbar_wait(empty_bar(stage), phase ^ 1u, abort_flag, wait_ns)) {
              ok = false;
              break;
            }
            const uint32_t dst = sbase + (uint32_t)stage * T::STAGE;
            mbar_arrive_expect_tx(full_bar(stage), bytes);
            if constexpr (PAIR)
              tma_load_5d(dst, &tmX, 0, -1, ky != 1 ? 1 : 0, ky == 0 ? h0 - 1 : h0, n0, full_bar(stage));
            else if (p.paired)
              tma_load_5d(dst, &tmX, c * T::KC + (kx != 1 ? p.cin : 0), kx == 0 ? -1 : 0, ky != 1 ? 1 : 0,
                          ky == 0 ? h0 - 1 : h0, n0, full_bar(stage));
            else
              tma_load_4d(dst, &tmX, c * T::KC, kx - 1, 2 * h0 - 1 + ky, n0, full_bar(stage));
            if constexpr (!RES)
              tma_load_2d(dst + T::A_BYTES, &tmW, (tap * p.chunks + c) * T::KC, 0, full_bar(stage));
            ++issued;
            if (++stage == STAGES) {
              stage = 0;
              phase ^= 1u;
            }
          }
        }
      }
      if (!ok) give_up();
      prod_stage = stage;
      prod_phase = phase;
    }
    __syncwarp();
  } else if (warp == 1) {
    if (lane == 0) {
      int stage = 0, acc = 0;
      uint32_t phase = 0, acc_phase = 0;
      bool ok = true;
      // FP32 accumulators, bf16 operands, both K-major, N = BN, M = 128
      constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | (8u << 24);
      if constexpr (RES) ok = mbar_wait(w_bar, 0, abort_flag, wait_ns);
      for (int t = blockIdx.x; t < p.tiles && ok; t += gridDim.x) {
        if (!mbar_wait(acce_bar(acc), acc_phase ^ 1u, abort_flag, wait_ns)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t d = tmem_base + (uint32_t)(acc * BN);
        for (int k = 0; k < k_iters; ++k) {
          if (!mbar_wait(full_bar(stage), phase, abort_flag, wait_ns)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t a = sbase + (uint32_t)stage * T::STAGE;
          if constexpr (PAIR) {
            // row r of the tile is the pair left of output column r: kx = 0 is
            // its odd pixel, kx = 1 and 2 the pixels of the next row's pair
#pragma unroll
            for (int kx = 0; kx < 3; ++kx)
#pragma unroll
              for (int kk = 0; kk < RB / 32; ++kk)
                tc_mma<0>(d, pair_desc(a, kx ? 1 : 0, (kx == 1 ? 0 : RB) + kk * 32),
                          conv_desc<RB>(wbase + (uint32_t)(3 * k + kx) * T::B_BYTES + kk * 32), idesc,
                          (k | kx | kk) != 0 ? 1u : 0u);
          } else {
            const uint32_t b = RES ? wbase + (uint32_t)k * T::B_BYTES : a + T::A_BYTES;
#pragma unroll
            for (int kk = 0; kk < RB / 32; ++kk)
              tc_mma<0>(d, conv_desc<RB>(a + kk * 32), conv_desc<RB>(b + kk * 32), idesc, (k | kk) != 0 ? 1u : 0u);
          }
          any_mma = true;
          tc_commit(empty_bar(stage));
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1u;
          }
        }
        if (!ok) break;
        tc_commit(accf_bar(acc));
        if (++acc == 2) {
          acc = 0;
          acc_phase ^= 1u;
        }
      }
      if (!ok) give_up();
    }
    __syncwarp();
  } else {
    const int wq = warp & 3, row = wq * 32 + lane;
    const uint32_t lane_addr = (uint32_t)(wq * 32) << 16;
    const int rw = row % p.wt, rh = (row / p.wt) % p.ht, rn = row / (p.wt * p.ht);
    int acc = 0;
    uint32_t acc_phase = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < p.tiles; t += gridDim.x) {
      ok = __all_sync(0xffffffffu, mbar_wait_epilogue(accf_bar(acc), acc_phase, abort_flag, wait_ns));
      if (!ok) break;
      tc_fence_after();
      const int nb = t / p.tiles_h, n = nb * p.nt + rn, h = (t - nb * p.tiles_h) * p.ht + rh;
      const bool live = row < rows && rw < p.Wo && h < p.Ho && n < p.B;
      const int64_t pix = ((int64_t)n * p.Ho + h) * p.Wo + rw;
#pragma unroll 1
      for (int c = 0; c < BN; c += 32) {
        __syncwarp();
        float v[32];
        tmem_ld32(tmem_base + lane_addr + (uint32_t)(acc * BN + c), v);
        const float4* b4 = reinterpret_cast<const float4*>(bias_s + c);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float4 b = b4[j];
          v[4 * j + 0] += b.x;
          v[4 * j + 1] += b.y;
          v[4 * j + 2] += b.z;
          v[4 * j + 3] += b.w;
        }
        if (p.relu) {
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = fmaxf(v[j], 0.0f);
        }
        if (live) {
          __align__(16) __nv_bfloat16 o[32];
#pragma unroll
          for (int j = 0; j < 32; ++j) o[j] = __float2bfloat16_rn(v[j]);
          uint4* d16 = reinterpret_cast<uint4*>(p.out16 + pix * BN + c);
#pragma unroll
          for (int j = 0; j < 4; ++j) d16[j] = reinterpret_cast<const uint4*>(o)[j];
          if (p.out32) {
            float4* d32 = reinterpret_cast<float4*>(p.out32 + pix * BN + c);
#pragma unroll
            for (int j = 0; j < 8; ++j) d32[j] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
          }
        }
      }
      tc_fence_before();
      mbar_arrive(acce_bar(acc));
      if (++acc == 2) {
        acc = 0;
        acc_phase ^= 1u;
      }
    }
    if (!ok && lane == 0) give_up();
  }

  // as in k_tc_gemm: after a give-up, wait for the copies and MMAs in flight
  __syncthreads();
  if (*abort_flag) {
    volatile int never = 0;
    if (warp == 0 && lane == 0) {
      if (w_issued) mbar_wait(w_bar, 0, &never);
      const int64_t inflight = issued < STAGES ? issued : (int64_t)STAGES;
      int s = prod_stage;
      uint32_t ph = prod_phase;
      for (int64_t i = 0; i < inflight; ++i) {
        if (s == 0) {
          s = STAGES - 1;
          ph ^= 1u;
        } else {
          --s;
        }
        mbar_wait(full_bar(s), ph, &never);
      }
    } else if (warp == 1 && lane == 0 && any_mma) {
      tc_commit(drain_bar);
      mbar_wait(drain_bar, 0, &never);
    }
  } else if (RES && warp == 0 && lane == 0 && w_issued) {
    // a CTA without tiles must not exit under its weight copies
    volatile int never = 0;
    mbar_wait(w_bar, 0, &never);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 2 * BN);
  }
}

// The operand shapes the kernel is built for (the network's layers) and the
// images a tile can cover: an output row fits the tile's 128 pixels. Other
// shapes take im2col + ebsd_cnn_conv_fwd.
static bool conv_rule(int cin, int cout, int Wo) {
  const bool shape = (cin == 32 && cout == 64) || (cin == 64 && cout == 128) ||
                     (cin % 64 == 0 && cin <= 1024 && cout == 256);
  return shape && Wo >= 1 && Wo <= 128;
}

template <int RB, int BN, bool RES, bool PAIR>
static int launch_conv(const CUtensorMap& tx, const CUtensorMap& tw, const ConvParams& p, cudaStream_t s) {
  using T = ConvTile<RB, BN, RES, PAIR>;
  const auto kern = k_conv_tc<RB, BN, RES, PAIR>;
  EBSD_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, T::SMEM));
  kern<<<std::min(p.tiles, device_sm_count()), CV_THREADS, T::SMEM, s>>>(tx, tw, p);
  EBSD_LAUNCH_CHECK();
  return 0;
}

}  // namespace ebsd

using namespace ebsd;

extern "C" int ebsd_cnn_conv_supported(int cin, int cout, int width) {
  return conv_rule(cin, cout, (width + 1) / 2) ? 1 : 0;
}

extern "C" int ebsd_cnn_conv_tc(const void* x, int batch, int height, int width, int cin, const void* w16,
                                int64_t ldw, const float* bias, int cout, int relu, void* out16, float* out32,
                                int* d_status, void* stream) {
  EBSD_ARG_CHECK(x && w16 && out16 && d_status, "ebsd_cnn_conv_tc: null pointer");
  EBSD_ARG_CHECK(batch >= 1 && height >= 1 && width >= 1, "ebsd_cnn_conv_tc: bad shape");
  const int Ho = (height + 1) / 2, Wo = (width + 1) / 2;
  EBSD_ARG_CHECK(conv_rule(cin, cout, Wo), "ebsd_cnn_conv_tc: %d -> %d channels at width %d not supported", cin, cout,
                 width);
  EBSD_ARG_CHECK(ldw >= 9 * cin && ldw % 8 == 0, "ebsd_cnn_conv_tc: weight rows too short or not 16-byte multiples");
  EBSD_ARG_CHECK(((uintptr_t)x & 15) == 0 && ((uintptr_t)w16 & 15) == 0 && ((uintptr_t)out16 & 15) == 0 &&
                     ((uintptr_t)out32 & 15) == 0,
                 "ebsd_cnn_conv_tc: pointers must be 16-byte aligned");
  ConvParams p{};
  p.paired = height % 2 == 0 && width % 2 == 0;
  // pairs of 32-channel pixels as rows, with the pair left of the image
  const bool pair_rows = cin == 32 && p.paired && Wo < 128;
  p.Wo = Wo;
  p.wt = pair_rows ? Wo + 1 : Wo;
  const int ht_max = std::min(Ho, 128 / p.wt);
  p.tiles_h = ceil_div(Ho, ht_max);
  p.ht = ceil_div(Ho, p.tiles_h);
  p.nt = p.tiles_h == 1 ? std::min(batch, 128 / (p.wt * p.ht)) : 1;
  const int64_t tiles = (int64_t)ceil_div(batch, p.nt) * p.tiles_h;
  EBSD_ARG_CHECK(tiles < INT32_MAX, "ebsd_cnn_conv_tc: too many tiles");
  p.tiles = (int)tiles;
  p.Ho = Ho;
  p.B = batch;
  p.bias = bias;
  p.out16 = reinterpret_cast<__nv_bfloat16*>(out16);
  p.out32 = out32;
  p.relu = relu;
  p.status = d_status;
  p.wait_ns = wait_limit_ns();
  const int kc = std::min(cin, 64);
  p.chunks = cin / kc;
  p.cin = cin;
  const CUtensorMapSwizzle sw = kc == 32 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B;
  CUtensorMap tx, tw;
  {
    const cuuint64_t c = (cuuint64_t)cin, w = (cuuint64_t)width, h = (cuuint64_t)height;
    int rc;
    if (p.paired) {
      const cuuint64_t dims[5] = {2 * c, w / 2, 2, h / 2, (cuuint64_t)batch};
      const cuuint64_t str[4] = {4 * c, 2 * c * w, 4 * c * w, 2 * c * w * h};
      const cuuint32_t box[5] = {(cuuint32_t)(pair_rows ? 64 : kc), (cuuint32_t)p.wt, 1, (cuuint32_t)p.ht, (cuuint32_t)p.nt};
      const cuuint32_t step[5] = {1, 1, 1, 1, 1};
      rc = encode_tensor_map(&tx, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, x, dims, str, box, step,
                             pair_rows ? CU_TENSOR_MAP_SWIZZLE_128B : sw);
    } else {
      const cuuint64_t dims[4] = {c, w, h, (cuuint64_t)batch};
      const cuuint64_t str[3] = {2 * c, 2 * c * w, 2 * c * w * h};
      // a box of 2 n elements walked with stride 2 loads n of them
      const cuuint32_t box[4] = {(cuuint32_t)kc, (cuuint32_t)(2 * p.wt), (cuuint32_t)(2 * p.ht), (cuuint32_t)p.nt};
      const cuuint32_t step[4] = {1, 2, 2, 1};
      rc = encode_tensor_map(&tx, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, x, dims, str, box, step, sw);
    }
    if (rc) return rc;
  }
  {
    const cuuint64_t dims[2] = {(cuuint64_t)(9 * cin), (cuuint64_t)cout};
    const cuuint64_t str[1] = {(cuuint64_t)ldw * 2};
    const cuuint32_t box[2] = {(cuuint32_t)kc, (cuuint32_t)cout};
    const cuuint32_t step[2] = {1, 1};
    if (int rc = encode_tensor_map(&tw, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, w16, dims, str, box, step, sw)) return rc;
  }
  cudaStream_t s = as_stream(stream);
  if (pair_rows) return launch_conv<64, 64, true, true>(tx, tw, p, s);
  if (cin == 32) return launch_conv<64, 64, true, false>(tx, tw, p, s);
  if (cout == 128) return launch_conv<128, 128, true, false>(tx, tw, p, s);
  return launch_conv<128, 256, false, false>(tx, tw, p, s);
}
