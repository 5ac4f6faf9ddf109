// Experimental-pattern preprocessing: overall background subtraction,
// per-pattern normalisation, CLAHE (optionally fused with the background
// subtraction and the two min-max passes of standard_clean) and the two
// scan-neighbourhood passes of NLPAR.
//
// Follows ebsdtorch/ebsd/experiment_pats.py:223-316 (subtract_overall_
// background, contrast_enhance_clahe, normalize_per_pattern, standard_clean,
// do_nlpar), ebsdtorch/preprocessing/clahe.py:17-130 and
// ebsdtorch/preprocessing/nlpar.py:19-192 (Brewick et al. 2019). Every pass
// here is an image pass over FP32 patterns: HBM-bound (mean, subtract,
// normalise, CLAHE) or bound on the SM (the NLPAR window passes, whose scan
// tile and halo are staged in shared memory once per pixel chunk).
#include <algorithm>
#include <climits>

#include "common.cuh"

namespace ebsd {

// ---------------------------------------------------------------- background

// partial[s][c] = sum of X[r, c] over the rows r of split s (FP64)
__global__ void k_colsum_partial(const float* __restrict__ X, int64_t n, int n_cols, int64_t ld, int n_splits,
                                 double* __restrict__ partial) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  const int s = blockIdx.y;
  if (c >= n_cols) return;
  const int64_t r0 = (int64_t)s * n / n_splits, r1 = (int64_t)(s + 1) * n / n_splits;
  double acc = 0.0;
#pragma unroll 8
  for (int64_t r = r0; r < r1; ++r) acc += __ldg(X + r * ld + c);
  partial[(int64_t)s * n_cols + c] = acc;
}

__device__ __forceinline__ float count_value(uint16_t v) { return (float)v; }
__device__ __forceinline__ float count_value(uint8_t v) { return (float)v; }
__device__ __forceinline__ float count_value(__half v) { return __half2float(v); }

// FP32 rows of patterns in their detector type, and the column sums of
// k_colsum_partial on the way. Bound by HBM (read once, written once): a thread
// takes VEC columns, so that the 2- and 1-byte types load 8 and 4 bytes. 65,536
// uint16 patterns of 60^2 px with the mean: 0.82 ms for a conversion and a pass
// over its result, 0.34 here (4.4 TB/s).
template <typename T, int VEC>
__global__ void k_rows_colsum(const T* __restrict__ X, int64_t n, int n_cols, int64_t ld, int n_splits,
                              float* __restrict__ rows, double* __restrict__ partial) {
  struct alignas(VEC * sizeof(T)) In {
    T v[VEC];
  };
  struct alignas(VEC * sizeof(float)) Out {
    float v[VEC];
  };
  const int c = (blockIdx.x * blockDim.x + threadIdx.x) * VEC;
  const int s = blockIdx.y;
  if (c >= n_cols) return;
  const int64_t r0 = (int64_t)s * n / n_splits, r1 = (int64_t)(s + 1) * n / n_splits;
  double acc[VEC] = {};
#pragma unroll 8
  for (int64_t r = r0; r < r1; ++r) {
    const In x = *reinterpret_cast<const In*>(X + r * ld + c);
    Out y;
#pragma unroll
    for (int k = 0; k < VEC; ++k) {
      y.v[k] = count_value(x.v[k]);
      acc[k] += y.v[k];
    }
    *reinterpret_cast<Out*>(rows + r * n_cols + c) = y;
  }
#pragma unroll
  for (int k = 0; k < VEC; ++k) partial[(int64_t)s * n_cols + c + k] = acc[k];
}

__global__ void k_colsum_final(const double* __restrict__ partial, int n_splits, int n_cols, int64_t n,
                               float* __restrict__ mean) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= n_cols) return;
  double s = 0.0;
  for (int k = 0; k < n_splits; ++k) s += partial[(int64_t)k * n_cols + c];
  mean[c] = (float)(s / (double)n);
}

template <typename T>
static int rows_and_mean(const void* patterns, int64_t n, int n_pix, int64_t ld, float* rows, double* partial,
                         int n_splits, float* mean, cudaStream_t s) {
  const T* x = static_cast<const T*>(patterns);
  EBSD_ARG_CHECK(reinterpret_cast<uintptr_t>(x) % sizeof(T) == 0, "ebsd_pattern_rows_mean: misaligned patterns");
  // four columns a thread where no load or store straddles its own size
  if (n_pix % 4 == 0 && ld % 4 == 0 && reinterpret_cast<uintptr_t>(x) % (4 * sizeof(T)) == 0 &&
      reinterpret_cast<uintptr_t>(rows) % 16 == 0) {
    k_rows_colsum<T, 4><<<dim3(ceil_div(n_pix, 256), n_splits), 64, 0, s>>>(x, n, n_pix, ld, n_splits, rows, partial);
  } else {
    k_rows_colsum<T, 1><<<dim3(ceil_div(n_pix, 256), n_splits), 256, 0, s>>>(x, n, n_pix, ld, n_splits, rows, partial);
  }
  EBSD_LAUNCH_CHECK();
  k_colsum_final<<<ceil_div(n_pix, 256), 256, 0, s>>>(partial, n_splits, n_pix, n, mean);
  EBSD_LAUNCH_CHECK();
  return 0;
}

__global__ void k_sub_vector(float* __restrict__ X, int64_t n, int n_cols, int64_t ld, const float* __restrict__ v) {
  const int64_t total = n * n_cols;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = t / n_cols;
    const int c = (int)(t - r * n_cols);
    X[r * ld + c] -= __ldg(v + c);
  }
}

// ------------------------------------------------------------- normalisation

constexpr int kNormThreads = 256;

__device__ __forceinline__ void cp_async4(float* dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async16(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// mode 0 min-max: (x - min) / ((1e-4 + max) - min); 1 zero mean; 2 zero mean
// and unit unbiased standard deviation (torch.std). One CTA per pattern; with
// PER > 0 a row of up to PER * 256 values is held in registers (one read, one
// write), otherwise it is re-read from global memory (L2) per pass.
template <int PER>
__global__ void __launch_bounds__(kNormThreads) k_normalize(float* __restrict__ X, int64_t n, int n_cols,
                                                           int64_t ld, int mode) {
  __shared__ float fred[32];
  __shared__ double dred[32];
  constexpr int R = PER > 0 ? PER : 1;
  float v[R];
  for (int64_t r = blockIdx.x; r < n; r += gridDim.x) {
    float* row = X + r * ld;
    auto at = [&](int k, int c) -> float {
      if constexpr (PER > 0) {
        return v[k];
      } else {
        return row[c];
      }
    };
    if constexpr (PER > 0) {
#pragma unroll
      for (int k = 0; k < PER; ++k) {
        const int c = threadIdx.x + k * kNormThreads;
        v[k] = c < n_cols ? row[c] : 0.f;
      }
    }
    if (mode == 0) {
      float mn = INFINITY, mx = -INFINITY;
#pragma unroll
      for (int k = 0; k < R; ++k)
        for (int c = threadIdx.x + k * kNormThreads; c < n_cols; c += R * kNormThreads) {
          const float x = at(k, c);
          mn = fminf(mn, x);
          mx = fmaxf(mx, x);
          if constexpr (PER > 0) break;
        }
      mx = block_max(mx, fred);
      mn = -block_max(-mn, fred);
      const float den = (1e-4f + mx) - mn;
#pragma unroll
      for (int k = 0; k < R; ++k)
        for (int c = threadIdx.x + k * kNormThreads; c < n_cols; c += R * kNormThreads) {
          row[c] = (at(k, c) - mn) / den;
          if constexpr (PER > 0) break;
        }
    } else {
      double s = 0.0;
#pragma unroll
      for (int k = 0; k < R; ++k)
        for (int c = threadIdx.x + k * kNormThreads; c < n_cols; c += R * kNormThreads) {
          s += at(k, c);
          if constexpr (PER > 0) break;
        }
      const float mean = (float)(block_sum(s, dred) / n_cols);
      float sd = 1.0f;
      if (mode == 2) {
        double ss = 0.0;
#pragma unroll
        for (int k = 0; k < R; ++k)
          for (int c = threadIdx.x + k * kNormThreads; c < n_cols; c += R * kNormThreads) {
            const double d = (double)(at(k, c) - mean);
            ss += d * d;
            if constexpr (PER > 0) break;
          }
        sd = (float)sqrt(block_sum(ss, dred) / (double)(n_cols - 1));
      }
#pragma unroll
      for (int k = 0; k < R; ++k)
        for (int c = threadIdx.x + k * kNormThreads; c < n_cols; c += R * kNormThreads) {
          const float x = at(k, c) - mean;
          row[c] = mode == 2 ? x / sd : x;
          if constexpr (PER > 0) break;
        }
    }
    __syncthreads();
  }
}

// --------------------------------------------------------------------- CLAHE

constexpr int kClaheThreads = 256;
// dynamic shared memory of one CTA: the CDF and histogram table, the
// coordinate tables, plus two image buffers when they fit (then each image
// is read once, prefetched while the previous one is equalised, and written
// once)
constexpr size_t kClaheSmemCap = 220 * 1024;

__device__ __forceinline__ int reflect_index(int i, int n) { return i < n ? i : 2 * (n - 1) - i; }

// redux.sync on FP32 values (sm_100): a NaN operand is ignored, as in fminf.
__device__ __forceinline__ float warp_redux_max(float v) {
  float r;
  asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
  return r;
}
__device__ __forceinline__ float warp_redux_min(float v) {
  float r;
  asm volatile("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
  return r;
}

// Block-wide min and max (all threads get both); synchronises the block.
__device__ __forceinline__ float2 block_minmax(float mn, float mx, float2* red) {
  const int lane = threadIdx.x & 31, n_warps = blockDim.x >> 5;
  mn = warp_redux_min(mn);
  mx = warp_redux_max(mx);
  __syncthreads();
  if (lane == 0) red[threadIdx.x >> 5] = make_float2(mn, mx);
  __syncthreads();
  const float2 v = lane < n_warps ? red[lane] : make_float2(INFINITY, -INFINITY);
  return make_float2(warp_redux_min(v.x), warp_redux_max(v.y));
}

// Exactly rounded x / den for many x of one den: x times the rounded reciprocal,
// corrected twice by its remainder (Markstein, IBM J. Res. Dev. 34, 1990: with a
// correctly rounded reciprocal and a quotient within one unit in the last place,
// one remainder correction rounds correctly; the first step brings it there).
// Asks for a den in [2^-60, 2^60] and remainders that do not underflow.
struct Quotient {
  float den, rcp;
  __device__ __forceinline__ explicit Quotient(float d) : den(d), rcp(1.0f / d) {}
  __device__ __forceinline__ bool reaches() const { return fabsf(den) >= 0x1p-60f && fabsf(den) <= 0x1p60f; }
  __device__ __forceinline__ float of(float x) const {
    float q = __fmul_rn(x, rcp);
    q = __fmaf_rn(__fmaf_rn(-q, den, x), rcp, q);
    return __fmaf_rn(__fmaf_rn(-q, den, x), rcp, q);
  }
};

// floor(x) of x in [0, 2^22) as a float and an integer, by adding 2^23 rounding down
__device__ __forceinline__ int small_floor(float x, float& f) {
  const float b = __fadd_rd(x, 8388608.0f);
  f = __fadd_rn(b, -8388608.0f);
  return (int)(__float_as_uint(b) - 0x4B000000u);
}

struct ClaheArgs {
  const float* X;
  int64_t n, ld;
  int H, W;
  const float* sub;  // optional pattern subtracted first (background)
  int minmax_in, minmax_out;
  float limit;
  int clip, nb, gh, gw;
  int vec_in, vec_sub, vec_out;  // whole float4s: H * W % 4 == 0 and rows of X, sub, rows of out 16-byte aligned
  float* out;
  int64_t ld_out;
};

// Shared-memory layout of k_clahe (bytes), shared with the host.
struct ClaheLayout {
  size_t table, coltile, rowtile, row, img, img_stride, total_tables;
  __host__ __device__ ClaheLayout(int H, int W, int gh, int gw, int nb) {
    const int th = (H + gh - 1) / gh, tw = (W + gw - 1) / gw;
    size_t o = 0;
    table = o;
    o += (size_t)gh * gw * nb * 8;
    row = o;
    o += (size_t)H * 8;
    coltile = o;
    o += (size_t)gw * tw * 4;
    rowtile = o;
    o += (size_t)gh * th * 4;
    img = (o + 15) / 16 * 16;
    img_stride = ((size_t)H * W + 3) / 4 * 4;  // floats
    total_tables = img;
  }
};

// One CTA per image. Optional pre-pass (x - sub, then min-max); tile
// histograms of floor(x (n_bins - 1)) over the bottom/right reflect-padded
// image; per tile (one warp) clip at `limit`, spread the excess evenly and
// the remainder one count to each of the first bins, cumulate into a CDF;
// then each pixel reads the (tile-y, tile-x, bin) CDF volume by trilinear
// interpolation with grid_sample's align_corners=False / border rules;
// optional post min-max. STAGED keeps the image in shared memory, the next
// image arriving by cp.async while this one is processed; otherwise every
// pass reads global memory (L2).
// Bound by instruction issue (0.72 of the slots at 250 instructions per 32
// pixels before), so instructions are what the passes save: a lane keeps its
// column and a warp takes every eighth row (one quarter of the addressing), the
// flat passes move four pixels at a time, scaling and histogram are one pass,
// quotients by a range or a count take five instructions (Quotient), and a
// tile's CDF is stored as pairs (value at b, value at b + 1), one 8-byte read per
// tile and pixel. Four CTAs per SM (64 registers): 1.48 ms for 65,536 patterns of
// 60^2 px with background and both min-max passes, 1.83 with two (118), 1.47
// with five (48), where 128^2 loses; 2.29 ms before. 16,384 of 128^2 px: 3.73 ms
// before, 1.85 now. The same bits.
// A tile's 8 n_bins bytes hold its counts in the lower half, then its clipped
// counts in the upper half, then the pairs.
template <bool STAGED>
__global__ void __launch_bounds__(kClaheThreads, 4) k_clahe(const ClaheArgs a) {
  extern __shared__ __align__(16) uint8_t smraw[];
  __shared__ float2 red[kClaheThreads / 32];
  const int n_tiles = a.gh * a.gw, nb = a.nb, H = a.H, W = a.W, P = H * W;
  const ClaheLayout L(H, W, a.gh, a.gw, nb);
  float2* table = reinterpret_cast<float2*>(smraw + L.table);
  int* coltile = reinterpret_cast<int*>(smraw + L.coltile);
  int* rowtile = reinterpret_cast<int*>(smraw + L.rowtile);
  // .x: table offset (bytes) of the lower tile's row, .y: weight of the upper one
  int2* row = reinterpret_cast<int2*>(smraw + L.row);
  float* img_s = reinterpret_cast<float*>(smraw + L.img);  // 2 images (STAGED)
  const int th = (H + a.gh - 1) / a.gh, tw = (W + a.gw - 1) / a.gw;
  const int hp = a.gh * th, wp = a.gw * tw, vpt = th * tw;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, n_warps = blockDim.x >> 5;
  const Quotient per_vpt((float)vpt);

  const Quotient per_nb((float)nb);

  // coordinate tables: padded pixel -> its tile's counts; output row
  // -> CDF cells and weight (torch.linspace(-1, 1, n) grids unnormalised
  // with align_corners=False, clamped at the border)
  const int row_bytes = a.gw * nb * 8, last_row = (a.gh - 1) * row_bytes;
  auto cell = [](int i, int n, int tiles) {
    const float c = -1.0f + 2.0f * (float)i / (float)(n - 1);
    return fminf(fmaxf(((c + 1.0f) * tiles - 1.0f) / 2.0f, 0.0f), (float)(tiles - 1));
  };
  for (int x = threadIdx.x; x < wp; x += blockDim.x) coltile[x] = x / tw * nb * 2;
  for (int y = threadIdx.x; y < hp; y += blockDim.x) rowtile[y] = y / th * a.gw * nb * 2;
  for (int y = threadIdx.x; y < H; y += blockDim.x) {
    const float f = cell(y, H, a.gh);
    row[y] = make_int2((int)f * row_bytes, __float_as_int(f - (int)f));
  }

  auto prefetch = [&](int64_t r, float* buf) {
    const float* src = a.X + r * a.ld;
    if (a.vec_in) {
      for (int t = threadIdx.x; t < P / 4; t += blockDim.x) cp_async16(buf + 4 * t, src + 4 * t);
    } else {
      for (int t = threadIdx.x; t < P; t += blockDim.x) cp_async4(buf + t, src + t);
    }
  };
  if constexpr (STAGED) {
    if (blockIdx.x < a.n) prefetch(blockIdx.x, img_s);
    cp_async_commit();
  }
  int it = 0;
  for (int64_t r = blockIdx.x; r < a.n; r += gridDim.x, ++it) {
    const float* img = a.X + r * a.ld;
    float* dst = a.out + r * a.ld_out;
    float* buf = img_s + (it & 1) * L.img_stride;
    if constexpr (STAGED) {
      if (r + gridDim.x < a.n) prefetch(r + gridDim.x, img_s + ((it + 1) & 1) * L.img_stride);
      cp_async_commit();
      cp_async_wait<1>();
    }
    for (int t = threadIdx.x; t < n_tiles * nb; t += blockDim.x) table[t] = make_float2(0.f, 0.f);
    __syncthreads();
    // pre-pass: x - sub, min / max (in place in shared memory when staged)
    float mn = INFINITY, mx = -INFINITY;
    if (a.sub || a.minmax_in) {
      if (STAGED && (!a.sub || a.vec_sub)) {
        float4* buf4 = reinterpret_cast<float4*>(buf);
        for (int t = threadIdx.x; t < P / 4; t += blockDim.x) {
          float4 v = buf4[t];
          if (a.sub) {
            const float4 s = __ldg(reinterpret_cast<const float4*>(a.sub) + t);
            v = make_float4(v.x - s.x, v.y - s.y, v.z - s.z, v.w - s.w);
            buf4[t] = v;
          }
          mn = fminf(mn, fminf(fminf(v.x, v.y), fminf(v.z, v.w)));
          mx = fmaxf(mx, fmaxf(fmaxf(v.x, v.y), fmaxf(v.z, v.w)));
        }
      }
      for (int t = (STAGED && (!a.sub || a.vec_sub) ? P / 4 * 4 : 0) + threadIdx.x; t < P; t += blockDim.x) {
        float v = STAGED ? buf[t] : img[t];
        if (a.sub) v -= __ldg(a.sub + t);
        if constexpr (STAGED) buf[t] = v;
        mn = fminf(mn, v);
        mx = fmaxf(mx, v);
      }
    }
    float in_mn = 0.f, in_den = 1.f;
    if (a.minmax_in) {
      const float2 m = block_minmax(mn, mx, red);
      in_mn = m.x;
      in_den = (1e-4f + m.y) - m.x;
    } else {
      __syncthreads();
    }
    // the value CLAHE sees at pixel t, `raw`: before its scaling. Remainders that
    // underflow belong to scaled values below 2^-26, which change neither a bin
    // nor a CDF coordinate (2 v - 1 is -1).
    const Quotient per_range(in_den);
    const int scaling = !a.minmax_in ? 0 : per_range.reaches() ? 1 : 2;
    auto raw = [&](int t) -> float {
      if constexpr (STAGED) {
        return buf[t];
      } else {
        float v = img[t];
        if (a.sub) v -= __ldg(a.sub + t);
        return v;
      }
    };
    auto scaled = [&](float v) -> float {
      return scaling == 0 ? v : scaling == 1 ? per_range.of(v - in_mn) : (v - in_mn) / in_den;
    };
    int* hist = reinterpret_cast<int*>(table);
    auto count = [&](int tile, float v) {
      float f;
      atomicAdd(hist + tile + small_floor(fminf(fmaxf(v * (float)(nb - 1), 0.0f), (float)(nb - 1)), f), 1);
    };
    // a lane keeps its column, a warp takes every eighth row
    auto scale_and_count = [&](auto scale) {
      for (int x = lane; x < W; x += 32) {
        const int tile_col = coltile[x];
#pragma unroll 4
        for (int y = wid; y < H; y += n_warps) {
          const int t = y * W + x;
          const float v = scale(raw(t));
          if constexpr (STAGED) buf[t] = v;
          count(rowtile[y] + tile_col, v);
        }
      }
    };
    if (scaling == 1) {  // without a branch per pixel
      scale_and_count([&](float v) { return per_range.of(v - in_mn); });
    } else {
      scale_and_count(scaled);
    }
    // the reflected pixels right of and below the image
    if (hp > H || wp > W) {
      __syncthreads();
      const int n_right = H * (wp - W), n_pad = hp * wp - P;
      for (int t = threadIdx.x; t < n_pad; t += blockDim.x) {
        const bool right = t < n_right;
        const int k = right ? t : t - n_right, w = right ? wp - W : wp;
        const int y = right ? k / w : H + k / w, x = (right ? W : 0) + k % w;
        const float v = raw(reflect_index(y, H) * W + reflect_index(x, W));
        count(rowtile[y] + coltile[x], STAGED ? v : scaled(v));
      }
    }
    __syncthreads();
    for (int tile = wid; tile < n_tiles; tile += n_warps) {
      float2* pairs = table + tile * nb;
      const int* h = reinterpret_cast<const int*>(pairs);
      float* c = reinterpret_cast<float*>(pairs) + nb;
      // pixel counts as the reference forms them (count / total * voxels)
      float part = 0.f;
      for (int b = lane; b < nb; b += 32) {
        float v = per_vpt.of((float)h[b]) * (float)vpt;
        if (a.clip) v = fminf(v, a.limit);
        c[b] = v;
        part += v;
      }
      const float sum = warp_sum(part);
      float residual = 0.f, redist = 0.f;
      if (a.clip) {
        const float clipped = (float)vpt - sum;
        residual = clipped - (float)nb * floorf(per_nb.of(clipped));  // torch.remainder
        redist = per_nb.of(clipped - residual);
      }
      __syncwarp();
      // the pairs of 32 bins are written when the next 32 CDF values are known;
      // pair b covers c[2 b - nb] and c[2 b - nb + 1], all read by then
      float carry = 0.f, prev = 0.f;
      for (int b0 = 0; b0 < nb; b0 += 32) {
        const int b = b0 + lane;
        float v = 0.f;
        if (b < nb) {
          v = c[b];
          if (a.clip) v = v + redist + ((float)b < residual ? 1.f : 0.f);
        }
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const float u = __shfl_up_sync(0xffffffffu, v, o);
          if (lane >= o) v += u;
        }
        v += carry;
        carry = __shfl_sync(0xffffffffu, v, 31);
        v = fminf(fmaxf(per_vpt.of(v), 0.f), 1.f);
        const float right = __shfl_down_sync(0xffffffffu, prev, 1), first = __shfl_sync(0xffffffffu, v, 0);
        __syncwarp();
        if (b0 > 0) pairs[b - 32] = make_float2(prev, lane < 31 ? right : first);
        prev = v;
      }
      const int b = (nb - 1) / 32 * 32 + lane;
      const float right = __shfl_down_sync(0xffffffffu, prev, 1);
      __syncwarp();
      if (b < nb) pairs[b] = make_float2(prev, b < nb - 1 ? right : prev);
    }
    __syncthreads();
    mn = INFINITY;
    mx = -INFINITY;
    const float half_nb = 0.5f * (float)nb, last_bin = (float)(nb - 1);
    for (int x = lane; x < W; x += 32) {
      const float f = cell(x, W, a.gw);
      const int x0 = (int)f, right = x0 + 1 < a.gw ? nb * 8 : 0;
      const float wx1 = f - x0, wx0 = 1.f - wx1;
      const uint8_t* column = smraw + L.table + (size_t)x0 * nb * 8;
#pragma unroll 4
      for (int y = wid; y < H; y += n_warps) {
        const int t = y * W + x;
        const int2 ry = row[y];
        const float wy1 = __int_as_float(ry.y), wy0 = 1.f - wy1;
        const float v = STAGED ? buf[t] : scaled(raw(t));
        // value coordinate: ((2 v - 1) + 1) n_bins - 1) / 2, as grid_sample
        // unnormalises the reference's v * 2 - 1
        const float fb = fminf(
            fmaxf(__fmaf_rn(__fadd_rn(__fmaf_rn(v, 2.0f, -1.0f), 1.0f), half_nb, -0.5f), 0.0f), last_bin);
        float fb0;
        const uint8_t* cell00 = column + ry.x + 8 * small_floor(fb, fb0);
        const uint8_t* cell10 = cell00 + (ry.x < last_row ? row_bytes : 0);
        const float wb1 = fb - fb0, wb0 = 1.f - wb1;
        const float2 c00 = *reinterpret_cast<const float2*>(cell00);
        const float2 c01 = *reinterpret_cast<const float2*>(cell00 + right);
        const float2 c10 = *reinterpret_cast<const float2*>(cell10);
        const float2 c11 = *reinterpret_cast<const float2*>(cell10 + right);
        const float v00 = c00.x * wb0 + c00.y * wb1;
        const float v01 = c01.x * wb0 + c01.y * wb1;
        const float v10 = c10.x * wb0 + c10.y * wb1;
        const float v11 = c11.x * wb0 + c11.y * wb1;
        const float o = (v00 * wx0 + v01 * wx1) * wy0 + (v10 * wx0 + v11 * wx1) * wy1;
        mn = fminf(mn, o);
        mx = fmaxf(mx, o);
        if (STAGED && a.minmax_out) {
          buf[t] = o;  // pixel t is read and written by this thread only
        } else {
          dst[t] = o;
        }
      }
    }
    if (a.minmax_out) {
      const float2 m = block_minmax(mn, mx, red);  // synchronises the block
      // the equalised values lie in [0, 1], each a sum of products of three
      // weights of 24 bits and a CDF: no remainder underflows
      const Quotient per_out((1e-4f + m.y) - m.x);
      if (STAGED && a.vec_out) {
        for (int t = threadIdx.x; t < P / 4; t += blockDim.x) {
          const float4 v = reinterpret_cast<const float4*>(buf)[t];
          reinterpret_cast<float4*>(dst)[t] = make_float4(per_out.of(v.x - m.x), per_out.of(v.y - m.x),
                                                          per_out.of(v.z - m.x), per_out.of(v.w - m.x));
        }
      } else {
        for (int t = threadIdx.x; t < P; t += blockDim.x) dst[t] = per_out.of((STAGED ? buf[t] : dst[t]) - m.x);
      }
    }
    __syncthreads();
  }
  if constexpr (STAGED) cp_async_wait<0>();
}

// --------------------------------------------------------------------- NLPAR

constexpr int kNlTile = 8;          // scan points per row segment (and rows) of an averaging CTA
constexpr int kNlMaxRad = 7;
constexpr int kNlMaxCells = (2 * kNlMaxRad + 1) * (2 * kNlMaxRad + 1);
constexpr int kNlMaxOffsets = kNlMaxCells;  // offsets per launch
constexpr int kNlBlockOffsets = 128;        // of the entry points that take a block of offsets

// Two FP32 values in one 64-bit register pair: the packed FP32 instructions
// issue two lanes' worth of FADD / FFMA at a time, each value rounded as usual.
using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float2 unpack2(f32x2 v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

// The window passes stage scan points in shared memory, kNlPix pixels of each
// at a time, several chunks ahead (cp.async); a lane owns pixels 2 lane and
// 2 lane + 1 of each half of a chunk.
constexpr int kNlPix = 64;

// T[i * kNlPix + q] = pixel p0 + q of staged point i, the pattern at
// data + src[i], or zeros where src[i] is negative (the reference pads the scan
// with zeros) and beyond the last pixel. VEC: 16-byte copies; a thread copies
// the same pixels of every point it takes.
template <bool VEC, int POINTS, int THREADS>
__device__ __forceinline__ void nl_stage(float* T, const float* __restrict__ data, const int64_t* src, int p0,
                                         int n_pix) {
  constexpr int kBytes = VEC ? 16 : 4, kPer = kNlPix * 4 / kBytes;
  static_assert(THREADS % 32 == 0 && kNlPix % 32 == 0, "whole warps per point");
  constexpr int kStep = THREADS >= kPer ? THREADS / kPer : 1;  // points per pass (whole points only)
  constexpr int kUsed = kStep * kPer;
  const int q = (int)threadIdx.x % kPer, p = p0 + q * (kBytes / 4);
  const float* base = data + p;
  uint32_t dst = smem_u32(T + ((int)threadIdx.x / kPer) * kNlPix) + q * kBytes;
  if ((int)threadIdx.x < kUsed) {
#pragma unroll 4
    for (int i = (int)threadIdx.x / kPer; i < POINTS; i += kStep, dst += kStep * kNlPix * 4) {
      const int64_t o = src[i];
      const bool ok = o >= 0 && p < n_pix;
      const float* g = ok ? base + o : data;
      if constexpr (VEC)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(g), "r"(ok ? 16 : 0) : "memory");
      else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(g), "r"(ok ? 4 : 0) : "memory");
    }
  }
}

__device__ __forceinline__ f32x2 nl_px(const float* point, int lane) {
  return reinterpret_cast<const f32x2*>(point)[lane];
}

// Shape of the distance kernel for a window radius: PT scan points of one row
// per warp, ROWS rows and all H + 1 row offsets of the half window per CTA,
// STAGES chunks in flight. Registers hold PT (2 H + 1) packed accumulators, so
// PT is halved for wide windows.
template <int H>
struct NlShape {
  static constexpr int PT = H <= 3 ? 8 : 4;
  static constexpr int ROWS = H <= 1 ? 6 : H == 2 ? 4 : H <= 4 ? 3 : H <= 6 ? 2 : 1;
  static constexpr int WARPS = ROWS * (H + 1);
  static constexpr int THREADS = 32 * WARPS;
  static constexpr int SIDE = PT + 2 * H, POINTS = (ROWS + H) * SIDE;
  static constexpr int STAGES = 4;
  static constexpr size_t SMEM = (size_t)STAGES * POINTS * kNlPix * sizeof(float);
};

// v[i] of 32 values summed over the warp's lanes; lane i gets value i.
__device__ __forceinline__ float transpose_sum(float (&v)[32], int lane) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int i = 0; i < o; ++i) {
      const float send = up ? v[i] : v[i + o], keep = up ? v[i + o] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
  return v[0];
}

// The (di, dj) -> offset lookup of one launch's offsets: first offset of a
// window cell (-1: none), the next offset of the same cell, and whether any
// offset lies outside the window.
struct NlMap {
  short first[kNlMaxCells];
  short next[kNlMaxOffsets];
  signed char di[kNlMaxOffsets], dj[kNlMaxOffsets];
  int any_bad;
};

template <int H>
__device__ __forceinline__ void nl_map(NlMap& m, const int* __restrict__ offsets, int o0, int n_off) {
  constexpr int w2 = 2 * H + 1;
  for (int c = threadIdx.x; c < w2 * w2; c += blockDim.x) m.first[c] = -1;
  if (threadIdx.x == 0) m.any_bad = 0;
  __syncthreads();
  for (int o = threadIdx.x; o < n_off; o += blockDim.x) {
    const int di = offsets[2 * (o0 + o)], dj = offsets[2 * (o0 + o) + 1];
    const bool ok = di >= -H && di <= H && dj >= -H && dj <= H;
    m.di[o] = (signed char)(ok ? di : 127);
    m.dj[o] = (signed char)(ok ? dj : 127);
    m.next[o] = -1;
    if (!ok) m.any_bad = 1;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int o = n_off - 1; o >= 0; --o) {
      if (m.di[o] == 127) continue;
      short& f = m.first[(m.di[o] + H) * w2 + m.dj[o] + H];
      m.next[o] = f;
      f = (short)o;
    }
  }
  __syncthreads();
}

// One chunk of one warp's pairs: ZERO (row offset 0) the offsets dj = 0..H and
// the squared norms, else dj = -H..H. own: the staged row of the warp's points,
// starting at column -H; nb: the row dy below it.
template <int H, bool ZERO, int N>
__device__ __forceinline__ void nl_pairs(f32x2 (&acc)[N], const float* own, const float* nb, int lane) {
  constexpr int PT = NlShape<H>::PT;
  f32x2 c[PT];  // the points, negated
#pragma unroll
  for (int j = 0; j < PT; ++j) c[j] = nl_px(own + (j + H) * kNlPix, lane) ^ 0x8000000080000000ull;
#pragma unroll
  for (int k = ZERO ? 0 : -H; k < PT + H; ++k) {
    const f32x2 v = nl_px(nb + (k + H) * kNlPix, lane);
#pragma unroll
    for (int j = 0; j < PT; ++j) {
      const int dj = k - j;
      if (dj < (ZERO ? 0 : -H) || dj > H) continue;
      f32x2& s = acc[(ZERO ? dj : dj + H) * PT + j];
      const f32x2 e = add2(v, c[j]);
      s = fma2(e, e, s);
    }
    if (ZERO && k < PT) {
      f32x2& s = acc[(H + 1) * PT + (k < PT && k >= 0 ? k : 0)];
      s = fma2(v, v, s);
    }
  }
}

// dists[pt, o0 + o] = sum_p (x[pt + off[o]] - x[pt])^2. A distance belongs to
// both points of a pair, so only the half window (di, dj) >= (0, 0) is
// computed and each sum is stored twice; offsets that leave the scan (zeros
// there) get the point's squared norm. Warp: PT points of one row against row
// offset di; lanes: pattern pixels, so the pixels of a point are read once
// from shared memory for all column offsets, two packed operations per pair
// and pixel pair. Each lane sums its own pixels, the lanes are added at the end
// (so the sums are also closer to 64 bits, 5e-8 against 1e-6).
// Near the FP32 pipe's bound for wide windows and large scans: 65,536 patterns
// of 60^2 px, k_rad 3: 2.70 -> 1.00 ms; 2,867 of 128^2 px, k_rad 5: 4.54 ->
// 0.61 ms; 36,000 of 40^2, k_rad 1: 0.40 -> 0.10 ms. Bounded before by one
// shared-memory load a pair and pixel, and by 256-thread CTAs of 64 points that
// left a small scan on a third of the SMs.
template <int H, bool VEC>
__global__ void __launch_bounds__(NlShape<H>::THREADS, 1)
    k_nlpar_dists(const float* __restrict__ data, int hs, int ws, int n_pix, int64_t ld,
                  const int* __restrict__ offsets, int o0, int n_off, int n_off_total, float* __restrict__ dists) {
  using S = NlShape<H>;
  constexpr int PT = S::PT, w2 = 2 * H + 1;
  constexpr int N = PT * (w2 > H + 2 ? w2 : H + 2), NB = (N + 31) / 32;
  extern __shared__ __align__(16) float T[];
  __shared__ NlMap map;
  __shared__ int64_t src[S::POINTS];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int segs = (ws + PT - 1) / PT;
  const int y0 = (int)(blockIdx.x / segs) * S::ROWS, x0 = (int)(blockIdx.x % segs) * PT;
  const int ry = wid / (H + 1), dy = wid % (H + 1), y = y0 + ry;
  for (int i = threadIdx.x; i < S::POINTS; i += S::THREADS) {
    const int py = y0 + i / S::SIDE, px = x0 - H + i % S::SIDE;
    src[i] = py < hs && px >= 0 && px < ws ? ((int64_t)py * ws + px) * ld : -1;
  }
  nl_map<H>(map, offsets, o0, n_off);  // synchronises
  const int n_chunks = (n_pix + kNlPix - 1) / kNlPix;
#pragma unroll
  for (int c = 0; c < S::STAGES - 1; ++c) {
    if (c < n_chunks)
      nl_stage<VEC, S::POINTS, S::THREADS>(T + c * S::POINTS * kNlPix, data, src, c * kNlPix, n_pix);
    cp_async_commit();
  }
  f32x2 acc[N];
#pragma unroll
  for (int i = 0; i < N; ++i) acc[i] = 0ull;
  for (int c = 0; c < n_chunks; ++c) {
    cp_async_wait<S::STAGES - 2>();
    __syncthreads();
    const int ahead = c + S::STAGES - 1;
    if (ahead < n_chunks)
      nl_stage<VEC, S::POINTS, S::THREADS>(T + (ahead % S::STAGES) * S::POINTS * kNlPix, data, src, ahead * kNlPix,
                                           n_pix);
    cp_async_commit();
    const float* own = T + ((c % S::STAGES) * S::POINTS + ry * S::SIDE) * kNlPix;
    if (dy == 0)
      nl_pairs<H, true>(acc, own, own, lane);
    else
      nl_pairs<H, false>(acc, own, own + dy * S::SIDE * kNlPix, lane);
  }
  cp_async_wait<0>();
  if (y >= hs) return;

  const int n_val = dy == 0 ? PT * (H + 2) : PT * w2;
#pragma unroll
  for (int b = 0; b < NB; ++b) {
    float v[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) {
      v[i] = 0.f;
      if (32 * b + i < N) {
        const float2 s = unpack2(acc[32 * b + i < N ? 32 * b + i : 0]);
        v[i] = s.x + s.y;
      }
    }
    const float val = transpose_sum(v, lane);
    const int i = 32 * b + lane, t = i / PT, px = x0 + i % PT;
    if (i >= n_val || px >= ws) continue;
    const int64_t pt = (int64_t)y * ws + px;
    if (dy == 0 && t == H + 1) {
      // offsets out of the scan: the neighbour is zero; out of the window: NaN
      if (px >= H && px + H < ws && y >= H && y + H < hs && !map.any_bad) continue;
      for (int o = 0; o < n_off; ++o) {
        const bool bad = map.di[o] == 127;
        const int qy = y + map.di[o], qx = px + map.dj[o];
        if (bad || qy < 0 || qy >= hs || qx < 0 || qx >= ws) dists[pt * n_off_total + o0 + o] = bad ? NAN : val;
      }
      continue;
    }
    const int dj = dy == 0 ? t : t - H, qx = px + dj, qy = y + dy;
    if (qx < 0 || qx >= ws || qy >= hs) continue;
    const int64_t q = (int64_t)qy * ws + qx;
    for (int o = map.first[(dy + H) * w2 + dj + H]; o >= 0; o = map.next[o]) dists[pt * n_off_total + o0 + o] = val;
    if (q != pt)
      for (int o = map.first[(H - dy) * w2 + H - dj]; o >= 0; o = map.next[o]) dists[q * n_off_total + o0 + o] = val;
  }
}

// Shape of the averaging kernel: warp = kNlTile points of one of ROWS rows.
template <int H>
struct NlAvg {
  static constexpr int ROWS = H <= 5 ? 8 : 4, THREADS = 32 * ROWS;
  static constexpr int SIDE = kNlTile + 2 * H, POINTS = (ROWS + 2 * H) * SIDE;
  static constexpr size_t WEIGHTS = (size_t)(2 * H + 1) * SIDE * ROWS * kNlTile * sizeof(float);
  static constexpr size_t STAGE = (size_t)POINTS * kNlPix * sizeof(float);
  static constexpr int STAGES = WEIGHTS + 3 * STAGE <= 224 * 1024 ? 3 : WEIGHTS + 2 * STAGE <= 224 * 1024 ? 2 : 1;
  static constexpr size_t SMEM = WEIGHTS + STAGES * STAGE;
};

// out[pt] (+)= sum_o w[pt, o0 + o] x[pt + off[o]]. Warp: 8 scan points of one
// row, lanes: pairs of pattern pixels. The window is walked by row di; a
// neighbour's pixels are read from shared memory once and used for every point
// whose window reaches it. The weights sit in shared memory in the order of use,
// [di][neighbour column][row][point], four points a read. Each (di, dj) may
// appear at most once per call; an offset outside the window makes the outputs
// NaN. WHOLE: the call's offsets fill the window; otherwise cells that are none of
// them are skipped, since a zero weight would let a non-finite value there
// through (both loops in one kernel: 1.40 instead of 1.34 ms for an NLPAR call of
// 2,867 patterns of 128^2 px, k_rad 5).
// Bound by shared-memory reads with one CTA per SM (window of points and
// weights), so weights are kept as single values: as (w, w) pairs for the packed
// FFMA they take two points a read. 65,536 patterns of 60^2 px, k_rad 3: 1.54 ms
// with pairs, 1.26 now (2.37 per-offset reads); 2,867 of 128^2 px, k_rad 5:
// 0.78, 0.63 (1.47). The same sums in the same order.
template <int H, bool VEC, bool WHOLE>
__global__ void __launch_bounds__(NlAvg<H>::THREADS) k_nlpar_average(const float* __restrict__ data, int hs, int ws,
                                                             int n_pix, int pix_per_split, int64_t ld,
                                                             const int* __restrict__ offsets, int o0, int n_off,
                                                             int n_off_total, const float* __restrict__ weights,
                                                             int accumulate, float* __restrict__ out,
                                                             int64_t ld_out) {
  using S = NlAvg<H>;
  constexpr int side = S::SIDE, w2 = 2 * H + 1, PTS = S::ROWS * kNlTile;
  extern __shared__ __align__(16) float w_s[];
  float* T = w_s + w2 * side * PTS;
  __shared__ int any_bad;
  __shared__ unsigned present[w2];  // !WHOLE: per window row, the columns among this call's offsets
  __shared__ int64_t src[S::POINTS];
  const int tiles_x = (ws + kNlTile - 1) / kNlTile;
  const int y0 = (blockIdx.x / tiles_x) * S::ROWS, x0 = (blockIdx.x % tiles_x) * kNlTile;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  // this CTA's range of pattern pixels (blockIdx.y); outputs are disjoint
  const int pix_begin = blockIdx.y * pix_per_split, pix_end = min(n_pix, pix_begin + pix_per_split);
  if (threadIdx.x == 0) any_bad = 0;
  if (!WHOLE && threadIdx.x < w2) present[threadIdx.x] = 0u;
  for (int i = threadIdx.x; i < S::POINTS; i += S::THREADS) {
    const int py = y0 - H + i / side, px = x0 - H + i % side;
    src[i] = py >= 0 && py < hs && px >= 0 && px < ws ? ((int64_t)py * ws + px) * ld : -1;
  }
  __syncthreads();
  const int n_chunks = (pix_end - pix_begin + kNlPix - 1) / kNlPix;
#pragma unroll
  for (int c = 0; c < S::STAGES - 1; ++c) {
    if (c < n_chunks)
      nl_stage<VEC, S::POINTS, S::THREADS>(T + c * S::POINTS * kNlPix, data, src, pix_begin + c * kNlPix, pix_end);
    cp_async_commit();
  }
  for (int i = threadIdx.x; i < w2 * side * PTS; i += S::THREADS) w_s[i] = 0.f;
  __syncthreads();
  for (int i = threadIdx.x; i < PTS * n_off; i += S::THREADS) {
    const int o = i / PTS, pt = i % PTS;
    const int di = offsets[2 * (o0 + o)], dj = offsets[2 * (o0 + o) + 1];
    if (di < -H || di > H || dj < -H || dj > H) {
      any_bad = 1;
      continue;
    }
    if (!WHOLE && pt == 0) atomicOr(&present[di + H], 1u << (dj + H));
    const int y = y0 + pt / kNlTile, x = x0 + pt % kNlTile;
    const float w = y < hs && x < ws ? weights[((int64_t)y * ws + x) * n_off_total + o0 + o] : 0.f;
    w_s[((di + H) * side + pt % kNlTile + dj + H) * PTS + pt] = w;
  }
  const int y = y0 + wid;
  for (int c = 0; c < n_chunks; ++c) {
    const int p0 = pix_begin + c * kNlPix;
    if constexpr (S::STAGES > 1) {
      cp_async_wait<S::STAGES - 2>();
      __syncthreads();
      const int ahead = c + S::STAGES - 1;
      if (ahead < n_chunks)
        nl_stage<VEC, S::POINTS, S::THREADS>(T + (ahead % S::STAGES) * S::POINTS * kNlPix, data, src,
                                             pix_begin + ahead * kNlPix, pix_end);
      cp_async_commit();
    } else {
      __syncthreads();
      nl_stage<VEC, S::POINTS, S::THREADS>(T, data, src, p0, pix_end);
      cp_async_commit();
      cp_async_wait<0>();
      __syncthreads();
    }
    if (y >= hs) continue;
    float2 s[kNlTile];
#pragma unroll
    for (int j = 0; j < kNlTile; ++j) s[j] = make_float2(0.f, 0.f);
    const float* row = T + ((c % S::STAGES) * S::POINTS + wid * side) * kNlPix;
    const float* wr = w_s + wid * kNlTile;
#pragma unroll 1
    for (int a = 0; a < w2; ++a, row += side * kNlPix, wr += side * PTS) {
      const unsigned cells = WHOLE ? 0u : present[a];
#pragma unroll
      for (int k = 0; k < side; ++k) {
        const float2 v = unpack2(nl_px(row + k * kNlPix, lane));
        const float4* w4 = reinterpret_cast<const float4*>(wr + k * PTS);
#pragma unroll
        for (int j = 0; j < kNlTile; j += 4) {
          if (k - j < 0 || k - j - 3 > 2 * H) continue;
          const float4 w = w4[j / 4];
          auto add = [&](int i, float wi) {
            if (k - i < 0 || k - i > 2 * H) return;
            if (!WHOLE && !(cells >> (k - i) & 1u)) return;
            s[i].x = fmaf(wi, v.x, s[i].x);
            s[i].y = fmaf(wi, v.y, s[i].y);
          };
          add(j, w.x);
          add(j + 1, w.y);
          add(j + 2, w.z);
          add(j + 3, w.w);
        }
      }
    }
#pragma unroll
    for (int j = 0; j < kNlTile; ++j) {
      if (x0 + j >= ws) break;
      float* dp = out + ((int64_t)y * ws + x0 + j) * ld_out + p0 + 2 * lane;
      float2 r = s[j];
      if (any_bad) r.x = r.y = NAN;
      if (VEC) {
        if (p0 + 2 * lane < pix_end) {
          float2* d = reinterpret_cast<float2*>(dp);
          if (accumulate) r = make_float2(d->x + r.x, d->y + r.y);
          *d = r;
        }
      } else {
        if (p0 + 2 * lane < pix_end) dp[0] = accumulate ? dp[0] + r.x : r.x;
        if (p0 + 2 * lane + 1 < pix_end) dp[1] = accumulate ? dp[1] + r.y : r.y;
      }
    }
  }
  cp_async_wait<0>();
}

// ---- NLPAR weights (nlpar.py:122-183): noise estimate, normalised
// distances, Newton fit of the global coefficient, masked softmax

constexpr int kNlWThreads = 256;
constexpr int kNlFitBlocks = 592;  // partial sums of one fit iteration

struct NlFitState {
  double g;       // the coefficient (the reference's guess_coeff)
  int done;       // |obj| fell below the tolerance in an earlier iteration
  unsigned ticket;
};

__global__ void k_nlpar_fit_init(NlFitState* st) {
  st->g = 1.0;
  st->done = 0;
  st->ticket = 0u;
}

// sigma[pt] = sqrt(min(d[pt, 1..8]) / (2 P))
__global__ void k_nlpar_sigma(const float* __restrict__ d, int64_t n_pts, int K, int n_pix,
                              float* __restrict__ sigma) {
  const int64_t pt = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (pt >= n_pts) return;
  float m = INFINITY;
  for (int o = 1; o < 9; ++o) m = fminf(m, d[pt * K + o]);
  sigma[pt] = sqrtf(m / (float)(2 * n_pix));
}

// w[pt, o] = -max((d - P s2) / (sqrt(2) sqrt(P) s2), 0), s2 = sigma^2 +
// sigma_other^2 (sigma_other = 1 outside the scan), in place over d
__global__ void k_nlpar_logits(float* __restrict__ d, int hs, int ws, int K, int n_pix,
                               const int* __restrict__ offsets, const float* __restrict__ sigma) {
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= (int64_t)hs * ws * K) return;
  const int64_t pt = t / K;
  const int o = (int)(t - pt * K);
  const int y = (int)(pt / ws) + offsets[2 * o], x = (int)(pt % ws) + offsets[2 * o + 1];
  const float so = (y >= 0 && y < hs && x >= 0 && x < ws) ? sigma[(int64_t)y * ws + x] : 1.0f;
  const float sp = sigma[pt];
  const float s2 = sp * sp + so * so;
  const float scale = (float)(1.4142135623730951 * sqrt((double)n_pix));  // 2**0.5 * n_pix**0.5
  const float v = (d[t] - (float)n_pix * s2) / (scale * s2);
  d[t] = -fmaxf(v, 0.0f);
}

// One Newton iteration: per point e_o = exp(w_o / g^2) over offsets 0..8,
// S = sum e_o; obj = mean(e_0 / S) - coeff, grad = mean(-2 e_0 (w_0 S -
// sum w_o e_o) / (g^3 S^2)); the last block to finish updates g (FP64 sums).
__global__ void __launch_bounds__(kNlWThreads) k_nlpar_fit(const float* __restrict__ w, int64_t n_pts, int K,
                                                          double coeff, double tol, NlFitState* st,
                                                          double2* __restrict__ partial) {
  __shared__ double red[32];
  __shared__ bool last;
  if (st->done) return;  // uniform: the state is written only by the previous launch
  const double g = st->g;
  const float g2 = (float)(g * g), g3 = (float)(g * g * g);
  double so = 0.0, sg = 0.0;
  for (int64_t pt = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; pt < n_pts;
       pt += (int64_t)gridDim.x * blockDim.x) {
    const float* r = w + pt * K;
    const float w0 = r[0];
    const float e0 = expf(w0 / g2);
    float S = e0, Swe = w0 * e0;
    for (int o = 1; o < 9; ++o) {
      const float wo = r[o];
      const float e = expf(wo / g2);
      S += e;
      Swe += wo * e;
    }
    so += e0 / S;
    sg += -2.0f * e0 * (w0 * S - Swe) / (g3 * S * S);
  }
  so = block_sum(so, red);
  sg = block_sum(sg, red);
  if (threadIdx.x == 0) {
    partial[blockIdx.x] = make_double2(so, sg);
    __threadfence();
    last = atomicAdd(&st->ticket, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  double a = 0.0, b = 0.0;
  for (int i = threadIdx.x; i < (int)gridDim.x; i += blockDim.x) {
    const double2 v = __ldcg(partial + i);
    a += v.x;
    b += v.y;
  }
  a = block_sum(a, red);
  b = block_sum(b, red);
  if (threadIdx.x == 0) {
    const double obj = a / (double)n_pts - coeff, grad = b / (double)n_pts;
    st->g = g - obj / grad;
    st->done = fabs(obj) < tol ? 1 : 0;
    st->ticket = 0;
  }
}

// weights[pt, :] = softmax over o of (w / g^2, + bias at o = 0; -inf for
// neighbours outside the scan), in place. One warp per point.
__global__ void k_nlpar_softmax(float* __restrict__ w, int hs, int ws, int K, const int* __restrict__ offsets,
                                const NlFitState* st, float bias) {
  const int64_t pt = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (pt >= (int64_t)hs * ws) return;
  const float g2 = (float)(st->g * st->g);
  const int py = (int)(pt / ws), px = (int)(pt % ws);
  float* r = w + pt * K;
  float mx = -INFINITY;
  for (int o = lane; o < K; o += 32) {
    const int y = py + offsets[2 * o], x = px + offsets[2 * o + 1];
    float v = r[o] / g2;
    if (o == 0 && bias > 0.0f) v += bias;
    if (y < 0 || y >= hs || x < 0 || x >= ws) v = -INFINITY;
    r[o] = v;
    mx = fmaxf(mx, v);
  }
  mx = warp_max(mx);
  float sum = 0.f;
  for (int o = lane; o < K; o += 32) sum += expf(r[o] - mx);
  sum = warp_sum(sum);
  for (int o = lane; o < K; o += 32) r[o] = expf(r[o] - mx) / sum;
}

// Pixel ranges of the average (second grid dimension), so that small scans
// still fill the GPU: about `waves` waves at the kernel's occupancy.
static int nl_splits(const void* func, int threads, size_t smem, int tiles, int max_splits, int waves) {
  int per_sm = 1;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, func, threads, smem) != cudaSuccess || per_sm < 1)
    per_sm = 1;
  const int64_t want = (int64_t)waves * device_sm_count() * per_sm;
  return (int)std::max<int64_t>(1, std::min<int64_t>(max_splits, (want + tiles - 1) / tiles));
}

template <int H, bool VEC>
static int nl_launch(bool average, const float* data, int hs, int ws, int n_pix, int64_t ld, const int* offsets,
                     int o0, int n_off, int n_off_total, float* dists, const float* weights, int accumulate,
                     float* out, int64_t ld_out, cudaStream_t s) {
  if (!average) {
    using S = NlShape<H>;
    const auto fn = k_nlpar_dists<H, VEC>;
    EBSD_CUDA_CHECK(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::SMEM));
    fn<<<ceil_div(hs, S::ROWS) * ceil_div(ws, S::PT), S::THREADS, S::SMEM, s>>>(data, hs, ws, n_pix, ld, offsets, o0,
                                                                               n_off, n_off_total, dists);
  } else {
    using S = NlAvg<H>;
    const int tiles = ceil_div(hs, S::ROWS) * ceil_div(ws, kNlTile);
    const bool whole = n_off == (2 * H + 1) * (2 * H + 1);
    const auto fn = whole ? k_nlpar_average<H, VEC, true> : k_nlpar_average<H, VEC, false>;
    EBSD_CUDA_CHECK(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::SMEM));
    // ranges of whole chunks, at least 8 chunks each
    const int n_chunks = ceil_div(n_pix, kNlPix);
    const int splits = nl_splits((const void*)fn, S::THREADS, S::SMEM, tiles, std::max(1, n_chunks / 8), 3);
    const int pix_per_split = ceil_div(n_chunks, splits) * kNlPix;
    fn<<<dim3(tiles, ceil_div(n_pix, pix_per_split)), S::THREADS, S::SMEM, s>>>(
        data, hs, ws, n_pix, pix_per_split, ld, offsets, o0, n_off, n_off_total, weights, accumulate, out, ld_out);
  }
  EBSD_LAUNCH_CHECK();
  return 0;
}

static int nl_dispatch(bool average, const float* data, int hs, int ws, int n_pix, int64_t ld, int k_rad,
                       const int* offsets, int o0, int n_off, int n_off_total, float* dists, const float* weights,
                       int accumulate, float* out, int64_t ld_out, cudaStream_t s) {
  // 16-byte accesses to every pattern
  const bool vec = n_pix % 4 == 0 && ld % 4 == 0 && reinterpret_cast<uintptr_t>(data) % 16 == 0 &&
                   (!average || (ld_out % 4 == 0 && reinterpret_cast<uintptr_t>(out) % 16 == 0));
  switch (k_rad) {
#define EBSD_NL_CASE(R)                                                                                         \
  case R:                                                                                                       \
    return vec ? nl_launch<R, true>(average, data, hs, ws, n_pix, ld, offsets, o0, n_off, n_off_total, dists,   \
                                    weights, accumulate, out, ld_out, s)                                        \
               : nl_launch<R, false>(average, data, hs, ws, n_pix, ld, offsets, o0, n_off, n_off_total, dists,  \
                                     weights, accumulate, out, ld_out, s);
    EBSD_NL_CASE(0)
    EBSD_NL_CASE(1)
    EBSD_NL_CASE(2)
    EBSD_NL_CASE(3)
    EBSD_NL_CASE(4)
    EBSD_NL_CASE(5)
    EBSD_NL_CASE(6)
    EBSD_NL_CASE(7)
#undef EBSD_NL_CASE
    default:
      EBSD_ARG_CHECK(false, "NLPAR: kernel radius must be in [0, %d]", kNlMaxRad);
  }
}

}  // namespace ebsd

using namespace ebsd;

extern "C" int ebsd_pattern_mean(const float* patterns, int64_t n, int n_pix, int64_t ld, double* partial,
                                 int n_splits, float* mean, void* stream) {
  EBSD_ARG_CHECK(patterns && partial && mean, "ebsd_pattern_mean: null pointer");
  EBSD_ARG_CHECK(n >= 1 && n_pix >= 1 && ld >= n_pix, "ebsd_pattern_mean: bad sizes");
  EBSD_ARG_CHECK(n_splits >= 1 && n_splits <= 65535, "n_splits must be in [1, 65535]");
  cudaStream_t s = as_stream(stream);
  k_colsum_partial<<<dim3(ceil_div(n_pix, 256), n_splits), 256, 0, s>>>(patterns, n, n_pix, ld, n_splits, partial);
  EBSD_LAUNCH_CHECK();
  k_colsum_final<<<ceil_div(n_pix, 256), 256, 0, s>>>(partial, n_splits, n_pix, n, mean);
  EBSD_LAUNCH_CHECK();
  return 0;
}

extern "C" int ebsd_pattern_rows_mean(const void* patterns, int pattern_dtype, int64_t n, int n_pix, int64_t ld,
                                      float* rows, double* partial, int n_splits, float* mean, void* stream) {
  EBSD_ARG_CHECK(patterns && rows && partial && mean, "ebsd_pattern_rows_mean: null pointer");
  EBSD_ARG_CHECK(n >= 1 && n_pix >= 1 && ld >= n_pix, "ebsd_pattern_rows_mean: bad sizes");
  EBSD_ARG_CHECK(n_splits >= 1 && n_splits <= 65535, "n_splits must be in [1, 65535]");
  cudaStream_t s = as_stream(stream);
  switch (pattern_dtype) {
    case EBSD_PAT_U16:
      return rows_and_mean<uint16_t>(patterns, n, n_pix, ld, rows, partial, n_splits, mean, s);
    case EBSD_PAT_U8:
      return rows_and_mean<uint8_t>(patterns, n, n_pix, ld, rows, partial, n_splits, mean, s);
    case EBSD_PAT_F16:
      return rows_and_mean<__half>(patterns, n, n_pix, ld, rows, partial, n_splits, mean, s);
  }
  EBSD_ARG_CHECK(false, "ebsd_pattern_rows_mean: pattern_dtype %d is not uint16, uint8 or half", pattern_dtype);
  return 0;
}

extern "C" int ebsd_subtract_pattern(float* patterns, int64_t n, int n_pix, int64_t ld, const float* v,
                                     void* stream) {
  EBSD_ARG_CHECK(patterns && v && n >= 0 && n_pix >= 1 && ld >= n_pix, "ebsd_subtract_pattern: bad arguments");
  if (n == 0) return 0;
  const int blocks = (int)std::min<int64_t>((n * n_pix + 255) / 256, (int64_t)device_sm_count() * 32);
  k_sub_vector<<<blocks, 256, 0, as_stream(stream)>>>(patterns, n, n_pix, ld, v);
  EBSD_LAUNCH_CHECK();
  return 0;
}

extern "C" int ebsd_normalize_patterns(float* patterns, int64_t n, int n_pix, int64_t ld, int mode, void* stream) {
  EBSD_ARG_CHECK(patterns && n >= 0 && n_pix >= 2 && ld >= n_pix, "ebsd_normalize_patterns: bad arguments");
  EBSD_ARG_CHECK(mode >= 0 && mode <= 2, "mode must be 0 (minmax), 1 (zeromean) or 2 (standard)");
  if (n == 0) return 0;
  const int blocks = (int)std::min<int64_t>(n, (int64_t)device_sm_count() * 8);
  cudaStream_t s = as_stream(stream);
  if (n_pix <= 4 * kNormThreads)
    k_normalize<4><<<blocks, kNormThreads, 0, s>>>(patterns, n, n_pix, ld, mode);
  else if (n_pix <= 8 * kNormThreads)
    k_normalize<8><<<blocks, kNormThreads, 0, s>>>(patterns, n, n_pix, ld, mode);
  else if (n_pix <= 16 * kNormThreads)
    k_normalize<16><<<blocks, kNormThreads, 0, s>>>(patterns, n, n_pix, ld, mode);
  else
    k_normalize<0><<<blocks, kNormThreads, 0, s>>>(patterns, n, n_pix, ld, mode);
  EBSD_LAUNCH_CHECK();
  return 0;
}

extern "C" int ebsd_clahe(const float* images, int64_t n, int height, int width, int64_t ld, const float* subtract,
                          int minmax_in, float clip_limit, int n_bins, int grid_h, int grid_w, int minmax_out,
                          float* out, int64_t ld_out, void* stream) {
  EBSD_ARG_CHECK(images && out && n >= 0, "ebsd_clahe: bad arguments");
  EBSD_ARG_CHECK(height >= 2 && width >= 2 && ld >= (int64_t)height * width && ld_out >= (int64_t)height * width,
                 "ebsd_clahe: bad image shape");
  EBSD_ARG_CHECK(grid_h >= 1 && grid_w >= 1 && grid_h <= height && grid_w <= width, "ebsd_clahe: bad grid");
  EBSD_ARG_CHECK(n_bins >= 2 && n_bins <= 2048, "n_bins must be in [2, 2048]");
  const int th = (height + grid_h - 1) / grid_h, tw = (width + grid_w - 1) / grid_w;
  // reflect padding needs the pad to be smaller than the image
  EBSD_ARG_CHECK(grid_h * th - height < height && grid_w * tw - width < width, "ebsd_clahe: padding too large");
  const ClaheLayout lay(height, width, grid_h, grid_w, n_bins);
  EBSD_ARG_CHECK(lay.total_tables <= kClaheSmemCap, "ebsd_clahe: grid x bins too large for shared memory");
  EBSD_ARG_CHECK(images != out || ld == ld_out, "ebsd_clahe: in place needs ld == ld_out");
  if (n == 0) return 0;
  ClaheArgs a;
  a.X = images;
  a.n = n;
  a.ld = ld;
  a.H = height;
  a.W = width;
  a.sub = subtract;
  a.minmax_in = minmax_in ? 1 : 0;
  a.minmax_out = minmax_out ? 1 : 0;
  // clip limit as the reference computes it: max(clip * voxels // bins, 1)
  a.limit = (float)std::max(std::floor((double)clip_limit * th * tw / n_bins), 1.0);
  a.clip = clip_limit > 0.0f ? 1 : 0;
  a.nb = n_bins;
  a.gh = grid_h;
  a.gw = grid_w;
  const int n_pix = height * width;
  auto whole_vec4 = [&](const void* p, int64_t stride) {
    return reinterpret_cast<uintptr_t>(p) % 16 == 0 && stride % 4 == 0 && n_pix % 4 == 0 ? 1 : 0;
  };
  a.vec_in = whole_vec4(images, ld);
  a.vec_sub = whole_vec4(subtract, 0);
  a.vec_out = whole_vec4(out, ld_out);
  a.out = out;
  a.ld_out = ld_out;
  const size_t staged_smem = lay.total_tables + 2 * lay.img_stride * sizeof(float);
  const bool staged = staged_smem <= kClaheSmemCap;
  const size_t smem = staged ? staged_smem : lay.total_tables;
  cudaStream_t s = as_stream(stream);
  if (staged) {
    EBSD_CUDA_CHECK(cudaFuncSetAttribute(k_clahe<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int per_sm = 0;
    EBSD_CUDA_CHECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_clahe<true>, kClaheThreads, smem));
    const int blocks = (int)std::min<int64_t>(n, (int64_t)device_sm_count() * std::max(per_sm, 1));
    k_clahe<true><<<blocks, kClaheThreads, smem, s>>>(a);
  } else {
    EBSD_CUDA_CHECK(cudaFuncSetAttribute(k_clahe<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int per_sm = 0;
    EBSD_CUDA_CHECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_clahe<false>, kClaheThreads, smem));
    const int blocks = (int)std::min<int64_t>(n, (int64_t)device_sm_count() * std::max(per_sm, 1));
    k_clahe<false><<<blocks, kClaheThreads, smem, s>>>(a);
  }
  EBSD_LAUNCH_CHECK();
  return 0;
}

static int nl_check(const float* data, int hs, int ws, int n_pix, int64_t ld, int halo, const int* offsets, int o0,
                    int n_off, int n_off_total, int max_off = kNlBlockOffsets) {
  EBSD_ARG_CHECK(data && offsets, "NLPAR: null pointer");
  EBSD_ARG_CHECK(hs >= 1 && ws >= 1 && n_pix >= 1 && ld >= n_pix, "NLPAR: bad sizes");
  EBSD_ARG_CHECK(halo >= 0 && halo <= kNlMaxRad, "NLPAR: kernel radius must be in [0, %d]", kNlMaxRad);
  EBSD_ARG_CHECK(n_off >= 1 && n_off <= max_off && o0 >= 0 && o0 + n_off <= n_off_total,
                 "NLPAR: an offset block holds 1..%d offsets", max_off);
  // the distance kernel's smallest tile: one row of four points
  EBSD_ARG_CHECK((int64_t)hs * ceil_div(ws, 4) <= INT_MAX, "NLPAR: scan too large");
  return 0;
}

extern "C" int ebsd_nlpar_dists(const float* data, int scan_h, int scan_w, int n_pix, int64_t ld, int k_rad,
                                const int* offsets, int o0, int n_off, int n_off_total, float* dists, void* stream) {
  if (int rc = nl_check(data, scan_h, scan_w, n_pix, ld, k_rad, offsets, o0, n_off, n_off_total)) return rc;
  EBSD_ARG_CHECK(dists != nullptr, "NLPAR: null output");
  return nl_dispatch(false, data, scan_h, scan_w, n_pix, ld, k_rad, offsets, o0, n_off, n_off_total, dists, nullptr,
                     0, nullptr, 0, as_stream(stream));
}

extern "C" int ebsd_nlpar_average(const float* data, int scan_h, int scan_w, int n_pix, int64_t ld, int k_rad,
                                  const int* offsets, int o0, int n_off, int n_off_total, const float* weights,
                                  int accumulate, float* out, int64_t ld_out, void* stream) {
  if (int rc = nl_check(data, scan_h, scan_w, n_pix, ld, k_rad, offsets, o0, n_off, n_off_total)) return rc;
  EBSD_ARG_CHECK(weights && out && ld_out >= n_pix, "NLPAR: bad output");
  EBSD_ARG_CHECK(out != data, "NLPAR: the average cannot be written in place");
  return nl_dispatch(true, data, scan_h, scan_w, n_pix, ld, k_rad, offsets, o0, n_off, n_off_total, nullptr, weights,
                     accumulate, out, ld_out, as_stream(stream));
}

extern "C" int ebsd_nlpar_dists_window(const float* data, int scan_h, int scan_w, int n_pix, int64_t ld, int k_rad,
                                       const int* offsets, int n_off, float* dists, void* stream) {
  if (int rc = nl_check(data, scan_h, scan_w, n_pix, ld, k_rad, offsets, 0, n_off, n_off, kNlMaxOffsets)) return rc;
  EBSD_ARG_CHECK(dists != nullptr, "NLPAR: null output");
  return nl_dispatch(false, data, scan_h, scan_w, n_pix, ld, k_rad, offsets, 0, n_off, n_off, dists, nullptr, 0,
                     nullptr, 0, as_stream(stream));
}

extern "C" int ebsd_nlpar_average_window(const float* data, int scan_h, int scan_w, int n_pix, int64_t ld, int k_rad,
                                         const int* offsets, int n_off, const float* weights, float* out,
                                         int64_t ld_out, void* stream) {
  if (int rc = nl_check(data, scan_h, scan_w, n_pix, ld, k_rad, offsets, 0, n_off, n_off, kNlMaxOffsets)) return rc;
  EBSD_ARG_CHECK(weights && out && ld_out >= n_pix, "NLPAR: bad output");
  EBSD_ARG_CHECK(out != data, "NLPAR: the average cannot be written in place");
  return nl_dispatch(true, data, scan_h, scan_w, n_pix, ld, k_rad, offsets, 0, n_off, n_off, nullptr, weights, 0, out,
                     ld_out, as_stream(stream));
}

extern "C" size_t ebsd_nlpar_workspace_bytes(int scan_h, int scan_w) {
  return 64 + (size_t)kNlFitBlocks * sizeof(double2) + (size_t)scan_h * scan_w * sizeof(float);
}

extern "C" int ebsd_nlpar_weights(float* dists, int scan_h, int scan_w, int n_pix, const int* offsets, int n_off,
                                  float coeff, float coeff_fit_tol, float center_logit_bias, void* workspace,
                                  size_t workspace_bytes, void* stream) {
  EBSD_ARG_CHECK(dists && offsets && workspace, "ebsd_nlpar_weights: null pointer");
  EBSD_ARG_CHECK(scan_h >= 1 && scan_w >= 1 && n_pix >= 1, "ebsd_nlpar_weights: bad sizes");
  EBSD_ARG_CHECK(n_off >= 9, "ebsd_nlpar_weights: the window needs at least 9 offsets (k_rad >= 1)");
  EBSD_ARG_CHECK(workspace_bytes >= ebsd_nlpar_workspace_bytes(scan_h, scan_w),
                 "ebsd_nlpar_weights: workspace too small");
  EBSD_ARG_CHECK(reinterpret_cast<uintptr_t>(workspace) % 16 == 0, "ebsd_nlpar_weights: workspace not 16-byte aligned");
  cudaStream_t s = as_stream(stream);
  auto* st = reinterpret_cast<NlFitState*>(workspace);
  auto* partial = reinterpret_cast<double2*>(static_cast<uint8_t*>(workspace) + 64);
  float* sigma = reinterpret_cast<float*>(partial + kNlFitBlocks);
  const int64_t n_pts = (int64_t)scan_h * scan_w;
  k_nlpar_fit_init<<<1, 1, 0, s>>>(st);
  EBSD_LAUNCH_CHECK();
  k_nlpar_sigma<<<ceil_div(n_pts, 256), 256, 0, s>>>(dists, n_pts, n_off, n_pix, sigma);
  EBSD_LAUNCH_CHECK();
  k_nlpar_logits<<<ceil_div(n_pts * n_off, 256), 256, 0, s>>>(dists, scan_h, scan_w, n_off, n_pix, offsets, sigma);
  EBSD_LAUNCH_CHECK();
  const int fit_blocks = (int)std::min<int64_t>(kNlFitBlocks, ceil_div(n_pts, kNlWThreads));
  for (int i = 0; i < 10; ++i) {
    k_nlpar_fit<<<fit_blocks, kNlWThreads, 0, s>>>(dists, n_pts, n_off, (double)coeff, (double)coeff_fit_tol, st,
                                                   partial);
    EBSD_LAUNCH_CHECK();
  }
  k_nlpar_softmax<<<ceil_div(n_pts * 32, 256), 256, 0, s>>>(dists, scan_h, scan_w, n_off, offsets, st,
                                                            center_logit_bias);
  EBSD_LAUNCH_CHECK();
  return 0;
}
