// Grid previews and clean-up outside the render path:
//  - the point-splat preview of src/visualization.py:157-232 (visulize_3d_in_2d_fast):
//    every cell with alpha above a floor projects to a pixel; the nearest one paints it
//    (the reference sorts far to near and lets the last write win), white elsewhere;
//  - the stray-voxel clean-up of src/grid_functions.py:260-280
//    (convolve_grid_to_remove_noise): repeatedly, the alpha of each cell's neighbours
//    within `radius` (a filled-ball kernel without its centre, zero padding) is summed and
//    cells whose sum is below the threshold are cleared (all four channels).
#include <algorithm>
#include <cmath>

#include "pgb_host.h"
#include "pgb_device.cuh"

namespace pgb {
namespace {

struct SplatCam {
  float T[12];  // rows 0..2 of the camera-to-world matrix
  float fov, aspect, pd;
  int xs, ys;
  float hx, hy, hz;  // ceil(shape / 2)
  float alpha_min;
};

__device__ __forceinline__ float dot3_ref(float a0, float a1, float a2, float b0, float b1, float b2) {
  return radd(radd(rmul(a0, b0), rmul(a1, b1)), rmul(a2, b2));
}

__global__ void splat_kernel(const float4* __restrict__ cells, int X, int Y, int Z, SplatCam k,
                             unsigned long long* __restrict__ keys) {
  const int64_t G = (int64_t)X * Y * Z;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < G;
       i += (int64_t)gridDim.x * blockDim.x) {
    const float4 c = __ldg(cells + i);
    if (!(c.w > k.alpha_min)) continue;
    const int iz = (int)(i % Z);
    const int64_t ij = i / Z;
    const int iy = (int)(ij % Y), ix = (int)(ij / Y);
    // world position ((index - ceil(shape/2)) + 1) * pd, then relative to the camera
    const float px = rmul(radd(rsub((float)ix, k.hx), 1.f), k.pd);
    const float py = rmul(radd(rsub((float)iy, k.hy), 1.f), k.pd);
    const float pz = rmul(radd(rsub((float)iz, k.hz), 1.f), k.pd);
    const float cx = rsub(px, k.T[3]), cy = rsub(py, k.T[7]), cz = rsub(pz, k.T[11]);
    // camera axes: x axis = column 0 (the "yz plane normal"), y axis = column 1
    const float dyz = dot3_ref(cx, cy, cz, k.T[0], k.T[4], k.T[8]);
    const float dxz = dot3_ref(cx, cy, cz, k.T[1], k.T[5], k.T[9]);
    const float dist = rsqrt_exact(rfma(cz, cz, rfma(cy, cy, rmul(cx, cx))));
    const float nyz = rsqrt_exact(radd(radd(rmul(k.T[0], k.T[0]), rmul(k.T[4], k.T[4])), rmul(k.T[8], k.T[8])));
    const float norms = rmul(dist, nyz);
    const float ax = rdiv(dyz, norms), ay = rdiv(dxz, norms);
    const float xn = radd(0.5f, rdiv(ay, -k.fov));
    const float yn = radd(0.5f, rdiv(ax, rdiv(k.fov, k.aspect)));
    if (!(xn < 1.f && xn >= 0.f && yn < 1.f && yn >= 0.f)) continue;
    const int xx = (int)fminf(fmaxf(rintf(rmul((float)k.xs, xn)), 0.f), (float)(k.xs - 1));
    const int yy = (int)fminf(fmaxf(rintf(rmul((float)k.ys, yn)), 0.f), (float)(k.ys - 1));
    // nearest point wins; among equal distances the later cell in row-major order
    const unsigned long long key = ((unsigned long long)__float_as_uint(dist) << 32) |
                                   (unsigned long long)(0xffffffffu - (uint32_t)i);
    atomicMin(keys + (int64_t)xx * k.ys + yy, key);
  }
}

__global__ void splat_resolve_kernel(const float4* __restrict__ cells,
                                     const unsigned long long* __restrict__ keys, int64_t npix,
                                     float* __restrict__ img) {
  for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < npix;
       p += (int64_t)gridDim.x * blockDim.x) {
    const unsigned long long key = keys[p];
    float r = 1.f, g = 1.f, b = 1.f;  // white background
    if (key != ~0ull) {
      const uint32_t i = 0xffffffffu - (uint32_t)(key & 0xffffffffull);
      const float4 c = __ldg(cells + i);
      r = c.x; g = c.y; b = c.z;
    }
    img[3 * p + 0] = r;
    img[3 * p + 1] = g;
    img[3 * p + 2] = b;
  }
}

__global__ void fill_u64_kernel(unsigned long long* p, int64_t n, unsigned long long v) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    p[i] = v;
}

// Offsets of the filled-ball kernel (src/grid_functions.py:260-267), decided on the host
// in double precision as the reference decides them, in the order of x, y, z. A list, since a
// ball holds few of its cube's offsets (radius 1: 6 of 26, 124 or 342) and a pass that
// walked the cube and tested a bit for each spent its time on the others.
struct BallList {
  int count;
  uint32_t at[343];  // kernel_size <= 7; (dx + 8) | (dy + 8) << 8 | (dz + 8) << 16
};

// neighbour sums over the ball offsets, zero padding, of ROWS cells at consecutive x (their
// loads do not wait for one another); value(i): alpha of flat cell i
template <int ROWS, typename F>
__device__ __forceinline__ void ball_sums(int x, int y, int z, int X, int Y, int Z, const BallList& ball,
                                          F value, float s[ROWS]) {
#pragma unroll
  for (int u = 0; u < ROWS; ++u) s[u] = 0.f;
  for (int k = 0; k < ball.count; ++k) {
    const uint32_t at = ball.at[k];
    const int xx = x + (int)(at & 0xffu) - 8, yy = y + (int)((at >> 8) & 0xffu) - 8,
              zz = z + (int)(at >> 16) - 8;
    if (!((unsigned)yy < (unsigned)Y && (unsigned)zz < (unsigned)Z)) continue;
    const int64_t i = ((int64_t)xx * Y + yy) * Z + zz;
#pragma unroll
    for (int u = 0; u < ROWS; ++u)
      if ((unsigned)(xx + u) < (unsigned)X) s[u] += value(i + (int64_t)u * Y * Z);
  }
}

__global__ void ball_sum_kernel(const float4* __restrict__ cells, int X, int Y, int Z,
                                const __grid_constant__ BallList ball, float* __restrict__ out) {
  const int z = blockIdx.x * blockDim.x + threadIdx.x;
  if (z >= Z) return;
  const int y = blockIdx.y, x = blockIdx.z;
  float s[1];
  ball_sums<1>(x, y, z, X, Y, Z, ball, [&](int64_t i) { return __ldg(cells + i).w; }, s);
  out[((int64_t)x * Y + y) * Z + z] = s[0];
}

// Clean-up on a copy of the alphas (two planes of 4 bytes a cell, taking turns: 134 MB for
// 256^3, about the L2) instead of the cells: each repeat reads one plane and writes the
// other, and the cells are touched twice in all. -0 in a plane marks a cleared cell (it adds
// nothing to a sum; a stored -0 becomes 0 when the plane is filled). A repeat after one that
// changed no alpha would decide every cell as that one did, so it returns at once.
// 256^3, kernel 5, radius 1, 20 repeats: 77.6 -> 2.3 ms; 128^3, kernel 3: 1.86 -> 0.19 ms.
struct NoiseState {
  int plane;       // the plane written last
  int pad;
  int changed[1];  // [repeats] whether the repeat cleared a cell whose alpha was not 0
};
constexpr int kNoiseRows = 4;  // consecutive x per block

__global__ void noise_fill_kernel(const float4* __restrict__ cells, int64_t G, float* __restrict__ plane) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < G;
       i += (int64_t)gridDim.x * blockDim.x)
    plane[i] = radd(__ldg(&cells[i].w), 0.f);
}

__global__ void noise_step_kernel(const float* __restrict__ in, float* __restrict__ out, int X, int Y,
                                  int Z, const __grid_constant__ BallList ball, float threshold,
                                  NoiseState* state, int repeat) {
  // (the last launch wrote it: a load through L1, since one past it by every warp queues at one
  // L2 address, 0.1 ms a launch at 256^3)
  if (repeat > 0 && state->changed[repeat - 1] == 0) return;
  const int z = blockIdx.x * blockDim.x + threadIdx.x;
  const int y = blockIdx.y;
  bool changed = false;
  if (z < Z) {
    const int x = blockIdx.z * kNoiseRows;
    float s[kNoiseRows];
    ball_sums<kNoiseRows>(x, y, z, X, Y, Z, ball, [&](int64_t j) { return __ldg(in + j); }, s);
#pragma unroll
    for (int u = 0; u < kNoiseRows; ++u) {
      if (x + u >= X) break;
      const int64_t i = ((int64_t)(x + u) * Y + y) * Z + z;
      const float v = __ldg(in + i);
      const bool clear = s[u] < threshold;
      changed |= clear && v != 0.f;
      out[i] = clear ? -0.f : v;
    }
  }
  if (__syncthreads_or(changed) && threadIdx.x == 0) state->changed[repeat] = 1;
  if (threadIdx.x == 0 && (blockIdx.x | blockIdx.y | blockIdx.z) == 0) state->plane = (repeat + 1) & 1;
}

__global__ void noise_clear_kernel(float4* __restrict__ cells, const float* __restrict__ planes, int64_t G,
                                   const NoiseState* __restrict__ state) {
  const float* plane = planes + (int64_t)state->plane * G;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < G;
       i += (int64_t)gridDim.x * blockDim.x)
    if (__float_as_uint(__ldg(plane + i)) == 0x80000000u) cells[i] = make_float4(0.f, 0.f, 0.f, 0.f);
}

__global__ void clear_below_kernel(float4* __restrict__ cells, const float* __restrict__ sums, int64_t G,
                                   float threshold) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < G;
       i += (int64_t)gridDim.x * blockDim.x)
    if (sums[i] < threshold) cells[i] = make_float4(0.f, 0.f, 0.f, 0.f);
}

inline unsigned nblocks(int64_t n) {
  return (unsigned)std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, 152 * 32));
}

// The arguments of a clean-up, and its ball. A ball with no cell besides the centre: the
// reference's normalised kernel is 0/0 (NaN) and no sum compares below the threshold, so
// nothing is cleared.
int check_noise(const float* cells, const int32_t dims[3], int32_t kernel_size, double radius,
                int32_t repeats, const void* scratch, BallList& ball) {
  ball.count = 0;
  if (!cells || !dims || !scratch || repeats < 0) return PGB_ERR_ARG;
  if (kernel_size < 1 || kernel_size % 2 == 0 || kernel_size > 7) return PGB_ERR_ARG;
  if (dims[0] <= 0 || dims[1] <= 0 || dims[2] <= 0) return PGB_ERR_ARG;
  if (dims[0] > 65535 || dims[1] > 65535) return PGB_ERR_UNSUPPORTED;
  if ((uintptr_t)cells % 16) return PGB_ERR_ALIGN;
  const int h = kernel_size / 2;
  for (int dx = -h; dx <= h; ++dx)
    for (int dy = -h; dy <= h; ++dy)
      for (int dz = -h; dz <= h; ++dz) {
        const int d2 = dx * dx + dy * dy + dz * dz;
        if (d2 != 0 && std::sqrt((double)d2) <= radius)
          ball.at[ball.count++] = (uint32_t)(dx + 8) | (uint32_t)(dy + 8) << 8 | (uint32_t)(dz + 8) << 16;
      }
  return PGB_OK;
}

// Host fp32 arithmetic, rounded op by op (this file is compiled without FMA contraction).
inline float norm3_plain(float x, float y, float z) {
  const float xx = x * x, yy = y * y, zz = z * z;
  const float s = xx + yy;
  return std::sqrt(s + zz);
}

}  // namespace
}  // namespace pgb

using namespace pgb;

extern "C" {

int pgb_splat_size(const float* transform, int32_t size_y, int32_t* width_out) {
  if (!transform || !width_out || size_y <= 0) return PGB_ERR_ARG;
  const float aspect = norm3_plain(transform[0], transform[4], transform[8]) /
                       norm3_plain(transform[1], transform[5], transform[9]);
  const float w = (float)size_y * aspect;
  if (!(w >= 1.f) || w > 1.0e6f) return PGB_ERR_ARG;
  *width_out = (int32_t)w;
  return PGB_OK;
}

int pgb_splat_preview(const float* cells, const int32_t dims[3], float points_distance,
                      const float* transform, float camera_angle_x, int32_t size_y, float alpha_min,
                      unsigned long long* keys_scratch, float* image_out, pgb_stream_t stream) {
  if (!cells || !dims || !transform || !keys_scratch || !image_out) return PGB_ERR_ARG;
  if (dims[0] <= 0 || dims[1] <= 0 || dims[2] <= 0) return PGB_ERR_ARG;
  const int64_t G = (int64_t)dims[0] * dims[1] * dims[2];
  if (G > 0xffffffffll) return PGB_ERR_UNSUPPORTED;
  if (((uintptr_t)cells % 16) || ((uintptr_t)keys_scratch % 8)) return PGB_ERR_ALIGN;
  int32_t xs = 0;
  int st = pgb_splat_size(transform, size_y, &xs);
  if (st) return st;
  SplatCam k;
  for (int r = 0; r < 3; ++r)
    for (int c = 0; c < 4; ++c) k.T[4 * r + c] = transform[4 * r + c];
  k.fov = camera_angle_x;
  k.aspect = norm3_plain(transform[0], transform[4], transform[8]) /
             norm3_plain(transform[1], transform[5], transform[9]);
  k.pd = points_distance;
  k.xs = xs;
  k.ys = size_y;
  k.hx = std::ceil((float)dims[0] / 2.f);
  k.hy = std::ceil((float)dims[1] / 2.f);
  k.hz = std::ceil((float)dims[2] / 2.f);
  k.alpha_min = alpha_min;
  const int64_t npix = (int64_t)xs * size_y;
  fill_u64_kernel<<<nblocks(npix), 256, 0, stream>>>(keys_scratch, npix, ~0ull);
  if ((st = after_launch())) return st;
  splat_kernel<<<nblocks(G), 256, 0, stream>>>(reinterpret_cast<const float4*>(cells), dims[0], dims[1],
                                               dims[2], k, keys_scratch);
  if ((st = after_launch())) return st;
  splat_resolve_kernel<<<nblocks(npix), 256, 0, stream>>>(reinterpret_cast<const float4*>(cells),
                                                          keys_scratch, npix, image_out);
  return after_launch();
}

int pgb_remove_noise(float* cells, const int32_t dims[3], int32_t kernel_size, double radius,
                     float threshold, int32_t repeats, float* sums_scratch, pgb_stream_t stream) {
  BallList ball;
  int st = check_noise(cells, dims, kernel_size, radius, repeats, sums_scratch, ball);
  if (st || ball.count == 0) return st;
  const int64_t G = (int64_t)dims[0] * dims[1] * dims[2];
  const dim3 grid((dims[2] + 127) / 128, dims[1], dims[0]);
  for (int it = 0; it < repeats; ++it) {
    ball_sum_kernel<<<grid, 128, 0, stream>>>(reinterpret_cast<const float4*>(cells), dims[0], dims[1],
                                              dims[2], ball, sums_scratch);
    if ((st = after_launch())) return st;
    clear_below_kernel<<<nblocks(G), 256, 0, stream>>>(reinterpret_cast<float4*>(cells), sums_scratch, G,
                                                       threshold);
    if ((st = after_launch())) return st;
  }
  return PGB_OK;
}

int64_t pgb_remove_noise_scratch_bytes(const int32_t dims[3], int32_t repeats) {
  if (!dims || dims[0] <= 0 || dims[1] <= 0 || dims[2] <= 0 || repeats < 0) return 0;
  return 8 * (int64_t)dims[0] * dims[1] * dims[2] + (int64_t)sizeof(NoiseState) + 4 * (int64_t)repeats;
}

int pgb_remove_noise_planes(float* cells, const int32_t dims[3], int32_t kernel_size, double radius,
                            float threshold, int32_t repeats, void* scratch, pgb_stream_t stream) {
  BallList ball;
  int st = check_noise(cells, dims, kernel_size, radius, repeats, scratch, ball);
  if (st || ball.count == 0 || repeats == 0) return st;
  if ((uintptr_t)scratch % 16) return PGB_ERR_ALIGN;
  const int X = dims[0], Y = dims[1], Z = dims[2];
  const int64_t G = (int64_t)X * Y * Z;
  float* planes = reinterpret_cast<float*>(scratch);
  NoiseState* state = reinterpret_cast<NoiseState*>(planes + 2 * G);
  if (cudaMemsetAsync(state, 0, sizeof(NoiseState) + 4 * (size_t)repeats, stream) != cudaSuccess)
    return PGB_ERR_LAUNCH;
  float4* c = reinterpret_cast<float4*>(cells);
  noise_fill_kernel<<<nblocks(G), 256, 0, stream>>>(c, G, planes);
  if ((st = after_launch())) return st;
  const dim3 grid((Z + 127) / 128, Y, (X + kNoiseRows - 1) / kNoiseRows);
  for (int it = 0; it < repeats; ++it) {
    noise_step_kernel<<<grid, 128, 0, stream>>>(planes + (it & 1) * G, planes + ((it + 1) & 1) * G, X, Y, Z, ball,
                                                threshold, state, it);
    if ((st = after_launch())) return st;
  }
  noise_clear_kernel<<<nblocks(G), 256, 0, stream>>>(c, planes, G, state);
  return after_launch();
}

}  // extern "C"
