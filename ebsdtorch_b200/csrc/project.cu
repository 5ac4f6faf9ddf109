// K1: dictionary projector and K2: pattern preparation.
//
// K1 follows ebsdtorch/ebsd/indexing.py:117-143: rotate each unit detector
// ray by the orientation (qu_apply, quaternions.py:186-213), map it to the
// side-by-side square Lambert projection (rosca_lambert_side_by_side,
// sphere.py:145-185), sample the (H, 2W) master pattern bilinearly with
// grid_sample semantics (align_corners=False, padding_mode="border";
// master_pattern.py:197-206), then subtract the row mean.
// K2 follows experiment_pats.py:318-346 (avg-pool binning) and
// indexing.py:175-187 (mask select, row mean subtraction).
//
// Both end in the same row finaliser: the zero-mean FP32 row, its L2 norm, and
// a unit-norm copy in the low-precision matching type (bf16, or e4m3 with a
// per-row absmax scale), zero padded to the GEMM row length.
#include <algorithm>
#include <cstring>
#include <type_traits>

#include "common.cuh"
#include "sampling.cuh"

namespace ebsd {

// Rows up to this length take 256-thread CTAs, six of which fit an SM beside an
// L1 that still holds the rays; longer rows 512-thread CTAs (two to an SM).
constexpr int kSmallRowPix = 6656;
constexpr int kMaxRowPix = 57344;  // 224 KiB of fp32 in shared memory

struct RowOut {
  float* f32;
  int64_t ld_f32;
  void* lp;
  int lp_dtype;
  int64_t ld_lp;
  float* norm;
  float* lp_scale;
};

// Sum of the 2^k lane-group values red[0 .. n_warps) in every thread, n_warps
// a power of two up to 32.
template <typename T>
__device__ __forceinline__ T sum_of_warps(const T* red, int n_warps) {
  T v = red[threadIdx.x & (n_warps - 1)];
  for (int o = n_warps >> 1; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// sqrt of an FP64 sum, rounded to FP32: two Newton steps in FP64 from the FP32
// reciprocal root (relative errors 2^-22, 2^-43, then FP64's own), instead of the
// FP64 square root's long dependent chain in every thread of the block.
__device__ __forceinline__ float root_of_sum(double x) {
  if (!(x >= 1e-30 && x <= 1e30)) return (float)sqrt(x);
  const float r = rsqrtf((float)x);
  const double h = 0.5 * (double)r;
  double y = x * (double)r;
  y = fma(h, fma(-y, y, x), y);
  return (float)fma(h, fma(-y, y, x), y);
}

// Two FP32 values as e4m3 (round to nearest even, saturating) in 16 bits.
__device__ __forceinline__ uint32_t e4m3x2(float lo, float hi) {
  return __nv_cvt_float2_to_fp8x2(make_float2(lo, hi), __NV_SATFINITE, __NV_E4M3);
}

// Scratch of one block's row reductions.
struct RowScratch {
  double sum[16], sq[16];
  float amax[16];
};

// FP32 partial sums of a thread, added in FP64: with 512 of them in a block of any
// size, each takes at most ceil(n / 512) of a row's n values. Fewer and longer
// ones would round more; FP64 ones (a conversion a value, 16 a clock on an SM)
// take K2 from 332 to 365 us for 32,768 patterns of 80^2 px.
template <int THREADS>
constexpr int kChains = 512 / THREADS;
template <int N>
__device__ __forceinline__ double sum_of_chains(const float (&c)[N]) {
  if constexpr (N == 4) return ((double)c[0] + c[1]) + ((double)c[2] + c[3]);
  if constexpr (N == 2) return (double)c[0] + c[1];
  return c[0];
}

// The next value of a thread's chains in turn.
template <int N>
__device__ __forceinline__ void add_in_turn(float (&c)[N], float v) {
  const float s = c[0] + v;
#pragma unroll
  for (int i = 0; i + 1 < N; ++i) c[i] = c[i + 1];
  c[N - 1] = s;
}

// Row values are in row[0..n); part_sum is the sum of the values this thread
// wrote. Finalise and write the outputs of row `r` (the shared row itself is
// left as it was): the mean (FP64 sum over the threads), then, where a norm or
// low-precision row is wanted, the norm and absmax of the zero-mean row, then the
// rows, in 16-byte stores where length and strides allow. The caller's block has
// not synchronised since writing the row, and synchronises before the row or the
// scratch are written again. The loops are short and kept rolled: unrolled by
// four they hold 48 to 64 registers instead of 32 to 40, which costs K2 CTAs on
// an SM (65,536 uint16 patterns of 60^2 px 397 us, 348 rolled; half of the pixels
// masked 294 and 218; 32,768 of 80^2 px 357 and 315).
template <int THREADS>
__device__ __forceinline__ void finalize_row(const float* row, int n, double inv_n, int subtract_mean,
                                             double part_sum, int64_t r, const RowOut& o, RowScratch& red) {
  constexpr int nt = THREADS, n_warps = nt / 32, C = kChains<THREADS>;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  part_sum = warp_sum(part_sum);
  if (lane == 0) red.sum[wid] = part_sum;
  __syncthreads();
  const float meanf = subtract_mean ? (float)(sum_of_warps(red.sum, n_warps) * inv_n) : 0.0f;
  const float4* row4 = reinterpret_cast<const float4*>(row);
  float* f32 = o.f32 ? o.f32 + r * o.ld_f32 : nullptr;
  const bool vec_f32 = (n & 3) == 0 && (reinterpret_cast<uintptr_t>(f32) & 15) == 0;
  if (!o.lp && !o.norm && !o.lp_scale) {
    if (vec_f32) {
#pragma unroll 1
      for (int c = tid; c < n / 4; c += nt) {
        const float4 a = row4[c];
        reinterpret_cast<float4*>(f32)[c] = make_float4(a.x - meanf, a.y - meanf, a.z - meanf, a.w - meanf);
      }
    } else {
#pragma unroll 1
      for (int p = tid; p < n; p += nt) f32[p] = row[p] - meanf;
    }
    return;
  }
  float ss[C] = {}, amax = 0.0f;
#pragma unroll 2
  for (int c = tid; c < n / 4; c += nt) {
    const float4 a = row4[c];
    const float v[4] = {a.x - meanf, a.y - meanf, a.z - meanf, a.w - meanf};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      ss[e % C] = fmaf(v[e], v[e], ss[e % C]);
      amax = fmaxf(amax, fabsf(v[e]));
    }
  }
  // the last threads, which have the fewest groups of four
  for (int p = (n & ~3) + nt - 1 - tid; p < n; p += nt) {
    const float v = row[p] - meanf;
    ss[0] = fmaf(v, v, ss[0]);
    amax = fmaxf(amax, fabsf(v));
  }
  const bool e4m3 = o.lp && o.lp_dtype == EBSD_DT_E4M3;
  const double wss = warp_sum(sum_of_chains(ss));
  if (e4m3) amax = warp_max(amax);
  if (lane == 0) {
    red.sq[wid] = wss;
    red.amax[wid] = amax;
  }
  __syncthreads();
  const float nrm = root_of_sum(sum_of_warps(red.sq, n_warps));
  const float inv = nrm > 0.0f ? 1.0f / nrm : 0.0f;
  float qscale = 1.0f;
  if (e4m3) {
    const float m = warp_max(red.amax[lane & (n_warps - 1)]) * inv;  // absmax of the unit row
    qscale = m > 0.0f ? m / 448.0f : 1.0f;
  }
  if (tid == 0) {
    if (o.norm) o.norm[r] = nrm;
    if (o.lp_scale) o.lp_scale[r] = qscale;
  }
  if (f32 && !vec_f32) {
#pragma unroll 1
    for (int p = tid; p < n; p += nt) f32[p] = row[p] - meanf;
  }
  if (!o.lp) {
    if (f32 && vec_f32)
#pragma unroll 1
      for (int c = tid; c < n / 4; c += nt) {
        const float4 a = row4[c];
        reinterpret_cast<float4*>(f32)[c] = make_float4(a.x - meanf, a.y - meanf, a.z - meanf, a.w - meanf);
      }
    return;
  }
  // eight values per thread and step: two float4 loads, the FP32 stores, one
  // 16-byte bf16 or 8-byte e4m3 store; zero from n to the row stride
  const int ld_lp = (int)o.ld_lp;
  const float sc = e4m3 ? inv / qscale : inv;
  uint8_t* lp = static_cast<uint8_t*>(o.lp) + r * o.ld_lp * (e4m3 ? 1 : 2);
  const bool vec_lp = (ld_lp & 7) == 0 && (reinterpret_cast<uintptr_t>(o.lp) & 15) == 0;
#pragma unroll 1
  for (int c = tid; c < (ld_lp + 7) / 8; c += nt) {
    float v[8];
    if (8 * c + 8 <= n) {
      const float4 a = row4[2 * c], b = row4[2 * c + 1];
      v[0] = a.x - meanf;
      v[1] = a.y - meanf;
      v[2] = a.z - meanf;
      v[3] = a.w - meanf;
      v[4] = b.x - meanf;
      v[5] = b.y - meanf;
      v[6] = b.z - meanf;
      v[7] = b.w - meanf;
      if (f32 && vec_f32) {
        reinterpret_cast<float4*>(f32)[2 * c] = make_float4(v[0], v[1], v[2], v[3]);
        reinterpret_cast<float4*>(f32)[2 * c + 1] = make_float4(v[4], v[5], v[6], v[7]);
      }
    } else {
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const int p = 8 * c + e;
        v[e] = p < n ? row[p] - meanf : 0.0f;
        if (f32 && vec_f32 && p < n) f32[p] = v[e];
      }
    }
    if (e4m3) {
      uint2 h;
      h.x = e4m3x2(v[0] * sc, v[1] * sc) | (e4m3x2(v[2] * sc, v[3] * sc) << 16);
      h.y = e4m3x2(v[4] * sc, v[5] * sc) | (e4m3x2(v[6] * sc, v[7] * sc) << 16);
      if (vec_lp) {
        reinterpret_cast<uint2*>(lp)[c] = h;
      } else {
        for (int e = 0; e < 8 && 8 * c + e < ld_lp; ++e) lp[8 * c + e] = (uint8_t)((e < 4 ? h.x : h.y) >> (8 * (e & 3)));
      }
    } else {
      __align__(16) __nv_bfloat16 h[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) h[e] = __float2bfloat16_rn(v[e] * sc);
      if (vec_lp) {
        reinterpret_cast<uint4*>(lp)[c] = *reinterpret_cast<const uint4*>(h);
      } else {
        for (int e = 0; e < 8 && 8 * c + e < ld_lp; ++e) reinterpret_cast<__nv_bfloat16*>(lp)[8 * c + e] = h[e];
      }
    }
  }
}

// quads[y][x] = the four values a bilinear sample with lower tap (x, y)
// blends, upper taps clamped to the border.
__global__ void k_sampling_quads(const float* __restrict__ mp, int h, int w, float4* __restrict__ quads) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y;
  if (x >= w) return;
  const int x1 = min(x + 1, w - 1);
  const float* lo = mp + (int64_t)y * w;
  const float* hi = mp + (int64_t)min(y + 1, h - 1) * w;
  quads[(int64_t)y * w + x] = make_float4(__ldg(lo + x), __ldg(lo + x1), __ldg(hi + x), __ldg(hi + x1));
}

// One CTA per dictionary row, grid-stride; each thread computes the taps of
// its next pixel while the gather of the current one is in flight. QUADS:
// `img` holds the four taps of every pixel as one float4, so a sample is one
// 16-byte gather instead of four 4-byte ones: neighbouring rays fall on
// different image rows, so each gather of a warp touches up to 32 lines, and
// those accesses bound the plain route. Bound by instruction issue now (issue
// slots 0.61 busy with two unpipelined pixels a thread and half the warps).
// 36,829 rows of 60^2 px: 98.5 G samples/s with IEEE-rounded divisions by two,
// floors and four gathers, 125 with lambert_tap and the table, 150 pipelined
// with 48 warps on an SM; 16,384 rows of 128^2: 97.7, 132, 150; 8,192 of
// 160^2: 52, 93, 115. All bit for bit the same rows.
// Both thread counts add pixels p = c (mod 512) in ascending order into one
// FP32 partial sum per class c, so the row mean does not depend on the count.
template <int THREADS, bool QUADS>
__global__ void __launch_bounds__(THREADS, THREADS == 256 ? 6 : 2) k_project(
    const float* __restrict__ img, int mp_h, const LambertGrid g, const float* __restrict__ rays, int n_pix,
    double inv_n, const float4* __restrict__ quats, int64_t n_rows, int subtract_mean, RowOut o) {
  static_assert(THREADS == 512 || THREADS == 256, "partial sums by pixel modulo 512");
  extern __shared__ __align__(16) float row[];
  __shared__ RowScratch red;
  const float* rx = rays;
  const float* ry = rays + n_pix;
  const float* rz = rays + 2 * (int64_t)n_pix;
  for (int64_t r = blockIdx.x; r < n_rows; r += gridDim.x) {
    const float4 q = quats[r];
    const float3 q2 = make_float3(2.0f * q.y, 2.0f * q.z, 2.0f * q.w);
    float part[kChains<THREADS>] = {};
    int p = threadIdx.x;
    LambertTap<QUADS> t{};
    float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (p < n_pix) {
      t = lambert_tap<false, QUADS>(g, q, q2, __ldg(rx + p), __ldg(ry + p), __ldg(rz + p));
      v = load_taps(img, mp_h, g, t);
    }
#pragma unroll 2
    for (; p < n_pix; p += THREADS) {
      const int pn = min(p + THREADS, n_pix - 1);
      const LambertTap<QUADS> tn = lambert_tap<false, QUADS>(g, q, q2, __ldg(rx + pn), __ldg(ry + pn), __ldg(rz + pn));
      const float4 vn = load_taps(img, mp_h, g, tn);
      const float val = blend(t, v);
      row[p] = val;
      add_in_turn(part, val);
      t = tn;
      v = vn;
    }
    finalize_row<THREADS>(row, n_pix, inv_n, subtract_mean, sum_of_chains(part), r, o, red);
    __syncthreads();
  }
}

__device__ __forceinline__ float as_float(float v) { return v; }
__device__ __forceinline__ float as_float(uint16_t v) { return (float)v; }
__device__ __forceinline__ float as_float(uint8_t v) { return (float)v; }
__device__ __forceinline__ float as_float(__half v) { return __half2float(v); }
template <typename T>
__device__ __forceinline__ float load_pixel(const T* p, int64_t i) {
  return as_float(__ldg(p + i));
}

// Four consecutive values, loaded as one word of their size.
template <typename T>
struct alignas(4 * sizeof(T)) Vec4 {
  T v[4];
};
template <typename T>
__device__ __forceinline__ Vec4<T> load_vec4(const Vec4<T>* p) {
  using Word = std::conditional_t<sizeof(T) == 4, float4, std::conditional_t<sizeof(T) == 2, uint2, unsigned>>;
  const Word x = __ldg(reinterpret_cast<const Word*>(p));
  Vec4<T> r;
  memcpy(&r, &x, sizeof(r));
  return r;
}

// Patterns of type T (fp32, uint16 or uint8 detector counts, fp16) -> rows.
// Bound by HBM: one CTA per row, several rows' loads in flight per SM. vec4:
// whole unbinned patterns whose length, stride and base allow loads of four
// values.
template <typename T, int THREADS>
__global__ void __launch_bounds__(THREADS) k_prep(const T* __restrict__ pats, int64_t n_rows,
                                                  int h, int w, int64_t stride, int b,
                                                  const int32_t* __restrict__ pix, int n_pix, double inv_n,
                                                  int vec4, int subtract_mean, RowOut o) {
  extern __shared__ __align__(16) float row[];
  __shared__ RowScratch red;
  constexpr int C = kChains<THREADS>;
  const int wb = w / b;
  const float cnt = (float)(b * b);
  for (int64_t r = blockIdx.x; r < n_rows; r += gridDim.x) {
    const T* img = pats + r * stride;
    float part[C] = {};
    if (vec4) {
      const Vec4<T>* img4 = reinterpret_cast<const Vec4<T>*>(img);
      float4* row4 = reinterpret_cast<float4*>(row);
#pragma unroll 4
      for (int c = threadIdx.x; c < n_pix / 4; c += THREADS) {
        const Vec4<T> x = load_vec4(img4 + c);
        const float4 f = make_float4(as_float(x.v[0]), as_float(x.v[1]), as_float(x.v[2]), as_float(x.v[3]));
        row4[c] = f;
        if constexpr (C == 4) {
          part[0] += f.x;
          part[1] += f.y;
          part[2] += f.z;
          part[3] += f.w;
        } else {
          part[0] += f.x + f.y;
          part[C - 1] += f.z + f.w;
        }
      }
    } else if (b == 1) {
#pragma unroll 4
      for (int p = threadIdx.x; p < n_pix; p += THREADS) {
        const float v = load_pixel(img, pix ? __ldg(pix + p) : p);
        row[p] = v;
        add_in_turn(part, v);
      }
    } else {
      for (int p = threadIdx.x; p < n_pix; p += THREADS) {
        const int idx = pix ? __ldg(pix + p) : p;
        const int i = idx / wb, j = idx - i * wb;
        const int64_t src = (int64_t)(i * b) * w + j * b;
        float s = 0.0f;
        for (int a = 0; a < b; ++a) {
          const T* line = img + src + (int64_t)a * w;
#pragma unroll 2  // by 4 it costs uint8 rows a quarter (500 of 480 x 640 binned by 8: 94 and 126 us)
          for (int c = 0; c < b; ++c) s += as_float(__ldg(line + c));
        }
        const float v = s / cnt;
        row[p] = v;
        add_in_turn(part, v);
      }
    }
    finalize_row<THREADS>(row, n_pix, inv_n, subtract_mean, sum_of_chains(part), r, o, red);
    __syncthreads();
  }
}

__global__ void k_sample_points(const float* __restrict__ mp, int mp_h, int mp_w2,
                                const float* __restrict__ xyz, int64_t n, int normalize,
                                float* __restrict__ out) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    float x = xyz[3 * i], y = xyz[3 * i + 1], z = xyz[3 * i + 2];
    if (normalize) {
      const float nrm = sqrtf(x * x + y * y + z * z);
      x /= nrm;
      y /= nrm;
      z /= nrm;
    }
    const float2 uv = lambert_side_by_side(x, y, z);
    out[i] = sample_border(mp, mp_h, mp_w2, uv.x, uv.y);
  }
}

static int check_row_out(const RowOut& o, int n_pix) {
  EBSD_ARG_CHECK(!o.f32 || o.ld_f32 >= n_pix, "ld_f32 (%lld) < row length (%d)", (long long)o.ld_f32,
                 n_pix);
  if (o.lp) {
    EBSD_ARG_CHECK(o.lp_dtype == EBSD_DT_BF16 || o.lp_dtype == EBSD_DT_E4M3,
                   "lp_dtype must be EBSD_DT_BF16 or EBSD_DT_E4M3");
    EBSD_ARG_CHECK(o.ld_lp >= n_pix, "ld_lp (%lld) < row length (%d)", (long long)o.ld_lp, n_pix);
  }
  return 0;
}

// Every output may be NULL; with none wanted nothing is launched (finalize_row
// writes FP32 rows when it is asked for nothing else).
static bool no_output(const RowOut& o) { return !o.f32 && !o.lp && !o.norm && !o.lp_scale; }

static int row_grid(int64_t n_rows, size_t smem, const void* fn, int threads) {
  int per_sm = 1;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, smem) != cudaSuccess ||
      per_sm < 1)
    per_sm = 1;
  const int64_t cap = (int64_t)device_sm_count() * per_sm * 8;
  return (int)std::min<int64_t>(n_rows, cap);
}

template <int THREADS, bool QUADS>
static int launch_project(const float* img, int mp_h, int mp_w2, const float* rays, int n_pix, const float4* quats,
                          int64_t n_rows, int subtract_mean, const RowOut& o, cudaStream_t s) {
  const size_t smem = (size_t)n_pix * sizeof(float);
  const auto fn = k_project<THREADS, QUADS>;
  EBSD_CUDA_CHECK(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int grid = row_grid(n_rows, smem, (const void*)fn, THREADS);
  fn<<<grid, THREADS, smem, s>>>(img, mp_h, lambert_grid(mp_h, mp_w2), rays, n_pix, 1.0 / n_pix, quats, n_rows, subtract_mean, o);
  EBSD_LAUNCH_CHECK();
  return 0;
}

}  // namespace ebsd

using namespace ebsd;

template <bool QUADS>
static int project_rows(const float* img, int mp_h, int mp_w2, const float* rays_soa, int n_pix, const float* quats,
                        int64_t n_rows, int subtract_mean, const RowOut& o, void* stream) {
  EBSD_ARG_CHECK(img && rays_soa && quats, "ebsd_project_dictionary: null input");
  EBSD_ARG_CHECK(mp_h >= 1 && mp_w2 >= 1, "master pattern shape (%d, %d) invalid", mp_h, mp_w2);
  EBSD_ARG_CHECK(n_pix >= 1 && n_pix <= kMaxRowPix, "row length %d outside [1, %d]", n_pix,
                 kMaxRowPix);
  EBSD_ARG_CHECK(n_rows >= 0, "n_rows < 0");
  EBSD_ARG_CHECK((reinterpret_cast<uintptr_t>(quats) & 15) == 0, "quats must be 16-byte aligned");
  EBSD_ARG_CHECK(!QUADS || (reinterpret_cast<uintptr_t>(img) & 15) == 0, "quads must be 16-byte aligned");
  EBSD_ARG_CHECK(!QUADS || quads_fit(mp_h, mp_w2), "master pattern shape (%d, %d) too large for quads", mp_h, mp_w2);
  if (int rc = check_row_out(o, n_pix)) return rc;
  if (n_rows == 0 || no_output(o)) return 0;
  const float4* q = reinterpret_cast<const float4*>(quats);
  cudaStream_t s = as_stream(stream);
  if (n_pix <= kSmallRowPix)
    return launch_project<256, QUADS>(img, mp_h, mp_w2, rays_soa, n_pix, q, n_rows, subtract_mean, o, s);
  return launch_project<512, QUADS>(img, mp_h, mp_w2, rays_soa, n_pix, q, n_rows, subtract_mean, o, s);
}

extern "C" int ebsd_project_dictionary(const float* master_pattern, int mp_h, int mp_w2,
                                       const float* rays_soa, int n_pix, const float* quats,
                                       int64_t n_rows, int subtract_mean, float* out_f32,
                                       int64_t ld_f32, void* out_lp, int lp_dtype, int64_t ld_lp,
                                       float* out_norm, float* out_lp_scale, void* stream) {
  const RowOut o{out_f32, ld_f32, out_lp, lp_dtype, ld_lp, out_norm, out_lp_scale};
  return project_rows<false>(master_pattern, mp_h, mp_w2, rays_soa, n_pix, quats, n_rows, subtract_mean, o, stream);
}

extern "C" int ebsd_sampling_quads(const float* master_pattern, int mp_h, int mp_w2, float* quads, void* stream) {
  EBSD_ARG_CHECK(master_pattern && quads, "ebsd_sampling_quads: null pointer");
  EBSD_ARG_CHECK(mp_h >= 1 && mp_w2 >= 1 && quads_fit(mp_h, mp_w2), "master pattern shape (%d, %d) invalid", mp_h, mp_w2);
  EBSD_ARG_CHECK((reinterpret_cast<uintptr_t>(quads) & 15) == 0, "quads must be 16-byte aligned");
  k_sampling_quads<<<dim3(ceil_div(mp_w2, 256), mp_h), 256, 0, as_stream(stream)>>>(
      master_pattern, mp_h, mp_w2, reinterpret_cast<float4*>(quads));
  EBSD_LAUNCH_CHECK();
  return 0;
}

extern "C" int ebsd_project_dictionary_quads(const float* quads, int mp_h, int mp_w2, const float* rays_soa,
                                             int n_pix, const float* quats, int64_t n_rows, int subtract_mean,
                                             float* out_f32, int64_t ld_f32, void* out_lp, int lp_dtype,
                                             int64_t ld_lp, float* out_norm, float* out_lp_scale, void* stream) {
  const RowOut o{out_f32, ld_f32, out_lp, lp_dtype, ld_lp, out_norm, out_lp_scale};
  return project_rows<true>(quads, mp_h, mp_w2, rays_soa, n_pix, quats, n_rows, subtract_mean, o, stream);
}

template <typename T, int THREADS>
static int launch_prep_threads(const T* patterns, int64_t n_rows, int height, int width, int64_t pattern_stride,
                               int binning, const int32_t* pix_index, int n_pix, int subtract_mean, const RowOut& o,
                               cudaStream_t s) {
  const size_t smem = (size_t)n_pix * sizeof(float);
  const auto fn = k_prep<T, THREADS>;
  EBSD_CUDA_CHECK(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  // No more CTAs on an SM than leave L1 room for their loads in flight: rows of
  // 3,840 to 4,096 FP32 pixels with 12 CTAs and 28 KB of L1 take 113 us for 240 MB
  // in, 360 MB out; with 164 KB for the rows 99
  if (THREADS == 128)
    EBSD_CUDA_CHECK(cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, 72));
  const int grid = row_grid(n_rows, smem, (const void*)fn, THREADS);
  const int vec4 = binning == 1 && !pix_index && n_pix % 4 == 0 && pattern_stride % 4 == 0 &&
                   reinterpret_cast<uintptr_t>(patterns) % (4 * sizeof(T)) == 0;
  fn<<<grid, THREADS, smem, s>>>(patterns, n_rows, height, width, pattern_stride, binning, pix_index, n_pix,
                                 1.0 / n_pix, vec4, subtract_mean, o);
  EBSD_LAUNCH_CHECK();
  return 0;
}

template <typename T>
static int launch_prep(const T* patterns, int64_t n_rows, int height, int width, int64_t pattern_stride,
                       int binning, const int32_t* pix_index, int n_pix, int subtract_mean, const RowOut& o,
                       void* stream) {
  // Threads for a row: enough CTAs on an SM to keep HBM busy, enough threads
  // for a long row. 60^2 px: 128 threads 6.03, 256 5.18 TB/s; 80^2 (e4m3):
  // 5.34, 5.96; 128^2: 256 threads 5.44, 512 5.12; 160^2: 4.88, 5.31 (with the
  // finaliser's loops unrolled; rolled, what it takes now is 0 to 30 % faster).
#define EBSD_PREP(THREADS)                                                                                       \
  launch_prep_threads<T, THREADS>(patterns, n_rows, height, width, pattern_stride, binning, pix_index, n_pix, \
                                  subtract_mean, o, as_stream(stream))
  // Binned rows by their loads: with the threads of an unbinned row of their length
  // 1,000 patterns of 240^2 px binned by 2 took 237 us (uint16), now 130, and 100 of
  // 1,024^2 binned by 16 388 and 160 (512 threads for all: 155, 164).
  const int64_t loads = (int64_t)n_pix * binning * binning;
  return loads <= 4096 ? EBSD_PREP(128) : loads <= 16384 ? EBSD_PREP(256) : EBSD_PREP(512);
#undef EBSD_PREP
}

extern "C" int ebsd_prep_patterns_typed(const void* patterns, int pattern_dtype, int64_t n_rows, int height,
                                        int width, int64_t pattern_stride, int binning, const int32_t* pix_index,
                                        int n_pix, int subtract_mean, float* out_f32, int64_t ld_f32, void* out_lp,
                                        int lp_dtype, int64_t ld_lp, float* out_norm, float* out_lp_scale,
                                        void* stream) {
  EBSD_ARG_CHECK(patterns != nullptr, "ebsd_prep_patterns: null patterns");
  EBSD_ARG_CHECK(pattern_dtype >= EBSD_PAT_F32 && pattern_dtype <= EBSD_PAT_F16, "unknown pattern_dtype %d",
                 pattern_dtype);
  EBSD_ARG_CHECK(binning >= 1 && height % binning == 0 && width % binning == 0,
                 "binning %d must divide the pattern shape (%d, %d)", binning, height, width);
  const int n_binned = (height / binning) * (width / binning);
  EBSD_ARG_CHECK(n_pix >= 1 && n_pix <= kMaxRowPix, "row length %d outside [1, %d]", n_pix,
                 kMaxRowPix);
  EBSD_ARG_CHECK(pix_index || n_pix == n_binned,
                 "without a pixel index the row length must equal the binned pixel count");
  EBSD_ARG_CHECK(pattern_stride >= (int64_t)height * width, "pattern_stride too small");
  RowOut o{out_f32, ld_f32, out_lp, lp_dtype, ld_lp, out_norm, out_lp_scale};
  if (int rc = check_row_out(o, n_pix)) return rc;
  if (n_rows == 0 || no_output(o)) return 0;
  switch (pattern_dtype) {
    case EBSD_PAT_U16:
      return launch_prep(static_cast<const uint16_t*>(patterns), n_rows, height, width, pattern_stride, binning,
                         pix_index, n_pix, subtract_mean, o, stream);
    case EBSD_PAT_U8:
      return launch_prep(static_cast<const uint8_t*>(patterns), n_rows, height, width, pattern_stride, binning,
                         pix_index, n_pix, subtract_mean, o, stream);
    case EBSD_PAT_F16:
      return launch_prep(static_cast<const __half*>(patterns), n_rows, height, width, pattern_stride, binning,
                         pix_index, n_pix, subtract_mean, o, stream);
    default:
      return launch_prep(static_cast<const float*>(patterns), n_rows, height, width, pattern_stride, binning,
                         pix_index, n_pix, subtract_mean, o, stream);
  }
}

extern "C" int ebsd_prep_patterns(const float* patterns, int64_t n_rows, int height, int width,
                                  int64_t pattern_stride, int binning, const int32_t* pix_index,
                                  int n_pix, int subtract_mean, float* out_f32, int64_t ld_f32,
                                  void* out_lp, int lp_dtype, int64_t ld_lp, float* out_norm,
                                  float* out_lp_scale, void* stream) {
  return ebsd_prep_patterns_typed(patterns, EBSD_PAT_F32, n_rows, height, width, pattern_stride, binning,
                                  pix_index, n_pix, subtract_mean, out_f32, ld_f32, out_lp, lp_dtype, ld_lp,
                                  out_norm, out_lp_scale, stream);
}

extern "C" int ebsd_sample_master_pattern(const float* master_pattern, int mp_h, int mp_w2,
                                          const float* xyz, int64_t n, int normalize, float* out,
                                          void* stream) {
  EBSD_ARG_CHECK(master_pattern && xyz && out, "ebsd_sample_master_pattern: null pointer");
  EBSD_ARG_CHECK(mp_h >= 1 && mp_w2 >= 1 && n >= 0, "ebsd_sample_master_pattern: bad sizes");
  if (n == 0) return 0;
  const int blocks = (int)std::min<int64_t>((n + 255) / 256, (int64_t)device_sm_count() * 16);
  k_sample_points<<<blocks, 256, 0, as_stream(stream)>>>(master_pattern, mp_h, mp_w2, xyz, n,
                                                         normalize, out);
  EBSD_LAUNCH_CHECK();
  return 0;
}
