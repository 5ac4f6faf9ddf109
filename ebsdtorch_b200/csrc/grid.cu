// K0: FP64 cubochoric SO(3) grid -> quaternions -> Laue fundamental-zone
// filter -> order-preserving compaction.
//
// Follows ebsdtorch/s2_and_so3/laue_fz_ori.py:516-557 (grid size rule and
// filter), sampling.py:179-205 (grid coordinates, 'ij' order), cu2ho
// orientations.py:293-349, ho2ax :419-517, ax2qu :730-746, qu_std
// quaternions.py:27-38, ori_in_fz_laue laue_fz_ori.py:144-239.
//
// Differences from the reference, by design: everything is FP64 (the
// reference works in FP32 and fits cos(w/2) with a polynomial); the rotation
// angle is obtained by solving |h|^3 = 3/4 (w - sin w) with Newton's method.
// The output set and order equal the reference's for every grid checked.
#include <algorithm>
#include <cmath>

#include "common.cuh"
#include "cubochoric.cuh"

namespace ebsd {

constexpr int kGridBlock = 1024;      // threads of a large grid's blocks
constexpr int kSmallGridBlock = 256;  // of one below kSmallGrid points, so that it covers the SMs
constexpr int64_t kSmallGrid = 1 << 20;

__device__ __forceinline__ bool in_fz(const double q[4], int laue) {
  const double w = q[0], x = fabs(q[1]), y = fabs(q[2]), z = fabs(q[3]);
  const double kR2M1 = 0.41421356237309504880, kR3 = 1.73205080756887729353;
  switch (laue) {
    case 11: return (fmax(fmax(x, y), z) <= w * kR2M1) && (x + y + z <= w);
    case 10: return x + y + z <= w;
    case 9: {
      const double mm = fmax(x, y), nn = fmin(x, y);
      const double rot = (mm > (2.0 + kR3) * nn) ? mm : (kR3 / 2.0) * mm + 0.5 * nn;
      return (z <= (2.0 - kR3) * w) && (rot <= w);
    }
    case 8: return z <= (2.0 - kR3) * w;
    case 7: {
      const double rot = (x >= y * kR3) ? x : (kR3 / 2.0) * y + 0.5 * x;
      return (z <= (1.0 / kR3) * w) && (rot <= w);
    }
    case 6: return z <= (1.0 / kR3) * w;
    case 5: {
      const double mm = fmax(x, y), nn = fmin(x, y);
      const double rot = (mm > (kR2M1 + 2.0) * nn) ? mm : 0.70710678118654752440 * (mm + nn);
      return (z <= kR2M1 * w) && (rot <= w);
    }
    case 4: return z <= kR2M1 * w;
    case 3: return fmax(fmax(x, y), z) <= w;
    case 2: return z <= w;
    default: return true;
  }
}

// Grid coordinate i of `edge` along each axis: the edge + 1 points spanning
// [-a/2, a/2] with the last dropped, i.e. a/2 * (2i - edge) / edge. This form
// is exactly 0 at i = edge / 2 and exactly antisymmetric, as the reference's
// symmetric linspace is; the FZ test of 180-degree rotations about in-plane
// axes (z exactly 0) depends on that. grid.cu is compiled without FMA
// contraction so the FP64 arithmetic rounds like the CPU oracle.
__device__ __forceinline__ void grid_point(int ia, int ib, int ic, int edge, double c[3]) {
  const double kHalf = 1.0725146985555127;  // 0.5 * pi^(2/3)
  c[0] = kHalf * (double)(2 * ia - edge) / (double)edge;
  c[1] = kHalf * (double)(2 * ib - edge) / (double)edge;
  c[2] = kHalf * (double)(2 * ic - edge) / (double)edge;
}

// The grid indices [lo, lo + side) an axis that can hold points of the
// fundamental zone. The cube's nested shells max|c_i| = m map to spheres of
// homochoric radius proportional to m, so a zone whose rotation angles stay
// below a limit lies in a smaller cube: for m-3m (62.8 degrees) 6.6 % of the
// grid, for 4/mmm 23 %. The points keep their order, so the output does too.
// Bound by FP64 instructions in both passes: at m-3m 1 degree (edge 96) 469 us
// for the two over the whole cube, 57 us over the box; 4/mmm 1.2 degrees
// (edge 115) 777 and 191 us. Below a few thousand points the dependent chain
// of one point, 25 us a pass, is what remains.
struct GridBox {
  int lo, side;
};

static GridBox grid_box(int laue, int edge) {
  const double k = std::sqrt(2.0) - 1.0, s3 = std::sqrt(3.0), pi = 3.14159265358979323846;
  const auto prism = [&](int n) { return 1.0 / (std::cos(pi / (2 * n)) * std::cos(pi / (2 * n))); };
  double r2 = 0.0;  // largest squared Rodrigues vector of the zone's corners, 0: unbounded
  switch (laue) {
    case 11: r2 = 2 * k * k + (1 - 2 * k) * (1 - 2 * k); break;
    case 10: r2 = 1.0; break;
    case 9: r2 = prism(6) + (2 - s3) * (2 - s3); break;
    case 7: r2 = prism(3) + 1.0 / 3.0; break;
    case 5: r2 = prism(4) + k * k; break;
    case 3: r2 = 3.0; break;
    default: return {0, edge};
  }
  const double w = 2.0 * std::atan(std::sqrt(r2)) + 1e-6;
  const double reach = std::cbrt((w - std::sin(w)) / pi) * edge + 1e-3;  // bound on |2 i - edge|
  const int lo = std::max(0, (int)std::ceil((edge - reach) / 2));
  const int hi = std::min(edge - 1, (int)std::floor((edge + reach) / 2));
  return {lo, hi - lo + 1};
}

__device__ __forceinline__ bool box_point(int64_t i, int laue, int edge, GridBox box, double q[4], int* cell) {
  const unsigned side = (unsigned)box.side, u = (unsigned)i;  // side^3 < 2^32 for edges up to 1,625
  unsigned ia, ib, ic;
  if ((int64_t)side * side * side <= 0xffffffffll) {
    ic = u % side;
    ib = (u / side) % side;
    ia = u / (side * side);
  } else {
    ic = (unsigned)(i % side);
    ib = (unsigned)((i / side) % side);
    ia = (unsigned)(i / ((int64_t)side * side));
  }
  const int a = box.lo + (int)ia, b = box.lo + (int)ib, c2 = box.lo + (int)ic;
  double c[3];
  grid_point(a, b, c2, edge, c);
  cu_to_qu(c, q);
  *cell = (int)(((int64_t)a * edge + b) * edge + c2);
  return in_fz(q, laue);
}

__global__ void __launch_bounds__(kGridBlock) k_grid_count(int laue, int edge, GridBox box, int64_t n_total,
                                                           int32_t* __restrict__ block_counts) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  int flag = 0;
  if (i < n_total) {
    double q[4];
    int cell;
    flag = box_point(i, laue, edge, box, q, &cell) ? 1 : 0;
  }
  const int cnt = __syncthreads_count(flag);
  if (threadIdx.x == 0) block_counts[blockIdx.x] = cnt;
}

__global__ void __launch_bounds__(1024) k_grid_scan(const int32_t* __restrict__ block_counts,
                                                    int n_blocks, int64_t* __restrict__ offsets,
                                                    int64_t* __restrict__ d_count) {
  __shared__ int64_t red[32];
  __shared__ int64_t carry;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (int base = 0; base < n_blocks; base += 1024) {
    const int j = base + threadIdx.x;
    const int64_t v = (j < n_blocks) ? block_counts[j] : 0;
    // inclusive warp scan
    int64_t x = v;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int64_t y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) red[wid] = x;
    __syncthreads();
    if (wid == 0) {
      int64_t w = red[lane];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int64_t y = __shfl_up_sync(0xffffffffu, w, o);
        if (lane >= o) w += y;
      }
      red[lane] = w;
    }
    __syncthreads();
    const int64_t incl = x + (wid > 0 ? red[wid - 1] : 0);
    if (j < n_blocks) offsets[j] = carry + incl - v;
    __syncthreads();
    if (threadIdx.x == 1023) carry += incl;
    __syncthreads();
  }
  if (threadIdx.x == 0) *d_count = carry;
}

__global__ void __launch_bounds__(kGridBlock) k_grid_write(int laue, int edge, GridBox box, int64_t n_total,
                                                           const int64_t* __restrict__ offsets,
                                                           float* __restrict__ out_f32,
                                                           double* __restrict__ out_f64,
                                                           int32_t* __restrict__ out_cells) {
  __shared__ int warp_cnt[kGridBlock / 32];
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  double q[4] = {0, 0, 0, 0};
  int cell = 0;
  const bool flag = i < n_total && box_point(i, laue, edge, box, q, &cell);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const unsigned bal = __ballot_sync(0xffffffffu, flag);
  if (lane == 0) warp_cnt[wid] = __popc(bal);
  __syncthreads();
  int before = 0;
  for (int w = 0; w < wid; ++w) before += warp_cnt[w];
  if (flag) {
    const int64_t r = offsets[blockIdx.x] + before + __popc(bal & ((1u << lane) - 1u));
    reinterpret_cast<float4*>(out_f32)[r] =
        make_float4((float)q[0], (float)q[1], (float)q[2], (float)q[3]);
    if (out_cells) out_cells[r] = cell;
    if (out_f64) {
      out_f64[4 * r + 0] = q[0];
      out_f64[4 * r + 1] = q[1];
      out_f64[4 * r + 2] = q[2];
      out_f64[4 * r + 3] = q[3];
    }
  }
}

// Launch of the passes over a zone's box.
struct GridPlan {
  GridBox box;
  int64_t n;
  int threads, blocks;
};

static GridPlan grid_plan(int laue, int edge) {
  GridPlan p;
  p.box = grid_box(laue, edge);
  p.n = (int64_t)p.box.side * p.box.side * p.box.side;
  p.threads = p.n < kSmallGrid ? kSmallGridBlock : kGridBlock;
  p.blocks = (int)std::max<int64_t>(1, (p.n + p.threads - 1) / p.threads);
  return p;
}

}  // namespace ebsd

using namespace ebsd;

extern "C" size_t ebsd_grid_workspace_bytes(int edge_length) {
  if (edge_length <= 0) return 0;
  // blocks of any Laue group's plan
  const int64_t n = (int64_t)edge_length * edge_length * edge_length;
  const size_t nb = (size_t)std::max((n + kGridBlock - 1) / kGridBlock,
                                     (std::min(n, kSmallGrid) + kSmallGridBlock - 1) / kSmallGridBlock);
  return nb * sizeof(int64_t) + nb * sizeof(int32_t) + 256;
}

static int grid_check(int laue_id, int edge, const void* ws, size_t ws_bytes) {
  EBSD_ARG_CHECK(laue_id >= 1 && laue_id <= 11, "Laue group %d is not supported", laue_id);
  EBSD_ARG_CHECK(edge >= 1 && edge <= 2048, "grid edge length %d out of range [1, 2048]", edge);
  EBSD_ARG_CHECK(ws != nullptr, "grid workspace is null");
  EBSD_ARG_CHECK(ws_bytes >= ebsd_grid_workspace_bytes(edge),
                 "grid workspace too small: %zu < %zu bytes", ws_bytes,
                 ebsd_grid_workspace_bytes(edge));
  return 0;
}

extern "C" int ebsd_grid_fz_count(int laue_id, int edge_length, void* workspace,
                                  size_t workspace_bytes, int64_t* d_count, void* stream) {
  if (int rc = grid_check(laue_id, edge_length, workspace, workspace_bytes)) return rc;
  EBSD_ARG_CHECK(d_count != nullptr, "d_count is null");
  const GridPlan p = grid_plan(laue_id, edge_length);
  int64_t* offsets = reinterpret_cast<int64_t*>(workspace);
  int32_t* counts = reinterpret_cast<int32_t*>(offsets + p.blocks);
  cudaStream_t s = as_stream(stream);
  k_grid_count<<<p.blocks, p.threads, 0, s>>>(laue_id, edge_length, p.box, p.n, counts);
  EBSD_LAUNCH_CHECK();
  k_grid_scan<<<1, 1024, 0, s>>>(counts, p.blocks, offsets, d_count);
  EBSD_LAUNCH_CHECK();
  return 0;
}

extern "C" int ebsd_grid_fz_write(int laue_id, int edge_length, const void* workspace,
                                  size_t workspace_bytes, float* out_f32, double* out_f64,
                                  int32_t* out_cells, void* stream) {
  if (int rc = grid_check(laue_id, edge_length, workspace, workspace_bytes)) return rc;
  EBSD_ARG_CHECK(out_f32 != nullptr, "out_f32 is null");
  EBSD_ARG_CHECK((reinterpret_cast<uintptr_t>(out_f32) & 15) == 0, "out_f32 must be 16-byte aligned");
  const GridPlan p = grid_plan(laue_id, edge_length);
  const int64_t* offsets = reinterpret_cast<const int64_t*>(workspace);
  k_grid_write<<<p.blocks, p.threads, 0, as_stream(stream)>>>(laue_id, edge_length, p.box, p.n, offsets, out_f32,
                                                              out_f64, out_cells);
  EBSD_LAUNCH_CHECK();
  return 0;
}
