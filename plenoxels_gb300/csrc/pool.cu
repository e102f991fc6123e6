// Average pooling of the grid for coarse-to-fine training (src/grid_functions.py:173-181,
// average_pool3d_grid: avg_pool3d of the channels-last grid with a cubic window of r
// cells and stride s, no padding), and its adjoint.
//
// The window sum is separable, so both directions run as three 1-D passes over the
// channels-last layout (z, then y, then x forward; x, then y, then z backward), each
// thread producing one float4 cell. The last backward pass writes every cell of the full
// gradient (cells under no window get 0), so it also clears it.
#include <algorithm>

#include "pgb_host.h"
#include "adam.cuh"

namespace pgb {
namespace {

inline unsigned blocks_of(int64_t n) {
  return (unsigned)std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, 1 << 20));
}

// out[a, o, b] = scale * sum_{k<r} in[a, o*s + k, b] for a [A, N, B] float4 view. Index: the
// type of a flat index (the 64-bit divisions of one cost more than the sums here).
template <typename Index>
__global__ void pool_axis_kernel(const float4* __restrict__ in, float4* __restrict__ out, Index A,
                                 int N, Index B, int No, int r, int s, float scale) {
  const Index total = A * No * B, step = (Index)gridDim.x * blockDim.x;
  for (Index i = (Index)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += step) {
    const Index b = i % B;
    const Index ao = i / B;
    const int o = (int)(ao % No);
    const Index a = ao / No;
    const float4* p = in + ((int64_t)a * N + (int64_t)o * s) * B + b;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int k = 0; k < r; ++k) acc = add4(acc, __ldg(p + (int64_t)k * B));
    acc.x *= scale; acc.y *= scale; acc.z *= scale; acc.w *= scale;
    out[i] = acc;
  }
}

__device__ __forceinline__ float4 shfl_down4(const float4& v, int d) {
  return make_float4(__shfl_down_sync(kFull, v.x, d), __shfl_down_sync(kFull, v.y, d),
                     __shfl_down_sync(kFull, v.z, d), __shfl_down_sync(kFull, v.w, d));
}

// pool_axis along contiguous rows (B = 1, no scale), for windows of q = r / s <= kPoolBlocks
// strides: lane j sums the s cells of block j and the first r mod s of them, each cell once,
// and window o is blocks o .. o + q - 1 and the head of block o + q, from the lanes behind. A
// window-by-window pass reads every cell r / s times over (256^3, window 21, stride 5: the
// three passes took 99 us, now 77 us, 55 of them here; reading the grid alone takes 40).
// Windows of one stride (no overlap) and wider ones keep that pass.
constexpr int kPoolBlocks = 8;

__global__ void __launch_bounds__(256) pool_rows_kernel(const float4* __restrict__ in,
                                                        float4* __restrict__ out, int64_t rows, int N,
                                                        int No, int r, int s) {
  const int lane = threadIdx.x & 31;
  const int q = r / s, head = r - q * s;
  const int given = kWarp - (q - 1) - (head > 0 ? 1 : 0);  // windows per warp
  const int parts = (No + given - 1) / given;
  const int64_t total = rows * parts;
  for (int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < total;
       w += ((int64_t)gridDim.x * blockDim.x) >> 5) {
    const int64_t row = w / parts;
    const int o = (int)(w - row * parts) * given + lane;
    const float4* p = in + row * N + (int64_t)o * s;
    const int left = N - o * s;  // cells of the row from this block on
    float4 sum = make_float4(0.f, 0.f, 0.f, 0.f), first = sum;
#pragma unroll 4
    for (int k = 0; k < s; ++k) {
      if (k == head) first = sum;
      if (k < left) sum = add4(sum, __ldg(p + k));
    }
    float4 acc = sum;
    for (int d = 1; d < q; ++d) acc = add4(acc, shfl_down4(sum, d));
    if (head > 0) acc = add4(acc, shfl_down4(first, q));
    if (lane < given && o < No) out[row * No + o] = acc;
  }
}

// The sum over the windows o that contain n of dout[o * B] (the adjoint of pool_axis at n).
__device__ __forceinline__ float4 unpool_sum(const float4* __restrict__ dout, int64_t B, int n, int No,
                                             int r, int s) {
  // windows o with o*s <= n < o*s + r
  const int hi = min(No - 1, n / s);
  const int lo = n - r + 1 <= 0 ? 0 : (n - r + 1 + s - 1) / s;
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int o = lo; o <= hi; ++o) acc = add4(acc, __ldg(dout + o * B));
  return acc;
}

// adjoint of pool_axis: din[a, n, b] = scale * sum over windows o containing n of dout[a, o, b]
template <typename Index>
__global__ void unpool_axis_kernel(const float4* __restrict__ dout, float4* __restrict__ din, Index A,
                                   int N, Index B, int No, int r, int s, float scale) {
  const Index total = A * N * B, step = (Index)gridDim.x * blockDim.x;
  for (Index i = (Index)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += step) {
    const Index b = i % B;
    const Index an = i / B;
    const int n = (int)(an % N);
    const Index a = an / N;
    float4 acc = unpool_sum(dout + (int64_t)a * No * B + b, (int64_t)B, n, No, r, s);
    acc.x *= scale; acc.y *= scale; acc.z *= scale; acc.w *= scale;
    din[i] = acc;
  }
}

// The last adjoint pass (along the rows) and Adam in one: the full gradient is formed in
// registers, used and dropped, where it was written (16 bytes a cell), read and zeroed again
// by Adam. Bound by HBM: 128 bytes a cell (256^3, window 21: 399 us for Adam alone -> 335 us for both).
template <typename Index>
__global__ void __launch_bounds__(256) unpool_adam_kernel(
    const float4* __restrict__ dout, float4* __restrict__ p, float4* __restrict__ m,
    float4* __restrict__ s2, float4* __restrict__ acc, Index rows, int N, int No, int r, int s,
    AdamConst k) {
  const Index total = rows * N, step = (Index)gridDim.x * blockDim.x;
  for (Index i = (Index)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += step) {
    float4 M = m[i], S = s2[i], P = p[i], C = make_float4(0.f, 0.f, 0.f, 0.f);
    if (acc) C = acc[i];
    const Index a = i / N;
    const int n = (int)(i - a * N);
    const float4 G = unpool_sum(dout + (int64_t)a * No, 1, n, No, r, s);
    const float4 d = adam_cell(P, G, M, S, k);
    p[i] = P;
    m[i] = M;
    s2[i] = S;
    if (acc) acc[i] = add4(C, d);
  }
}

// Launches of the passes with 32-bit indices where a flat index (and a grid stride past it)
// fits.
inline bool small_index(int64_t total) { return total < ((int64_t)1 << 31); }

int pool_axis(const float4* in, float4* out, int64_t A, int N, int64_t B, int No, int r, int s,
              float scale, cudaStream_t st) {
  const int64_t total = A * No * B;
  if (small_index(total) && small_index(A) && small_index(B))
    pool_axis_kernel<uint32_t><<<blocks_of(total), 256, 0, st>>>(in, out, (uint32_t)A, N, (uint32_t)B, No,
                                                                r, s, scale);
  else
    pool_axis_kernel<int64_t><<<blocks_of(total), 256, 0, st>>>(in, out, A, N, B, No, r, s, scale);
  return after_launch();
}

int unpool_axis(const float4* dout, float4* din, int64_t A, int N, int64_t B, int No, int r, int s,
                float scale, cudaStream_t st) {
  const int64_t total = A * N * B;
  if (small_index(total) && small_index(A) && small_index(B))
    unpool_axis_kernel<uint32_t><<<blocks_of(total), 256, 0, st>>>(dout, din, (uint32_t)A, N, (uint32_t)B,
                                                                  No, r, s, scale);
  else
    unpool_axis_kernel<int64_t><<<blocks_of(total), 256, 0, st>>>(dout, din, A, N, B, No, r, s, scale);
  return after_launch();
}

// The adjoint passes along x and y: the gradient of the rows, [X, Y, Zo] in the scratch.
int unpool_to_rows(const float* d_out, const int32_t dims[3], const int32_t od[3], int window, int stride,
                   void* scratch, float4** rows, cudaStream_t s) {
  const int X = dims[0], Y = dims[1];
  float4* t1 = reinterpret_cast<float4*>(scratch);  // [X,Y,Zo]
  float4* t2 = reinterpret_cast<float4*>((char*)scratch +
                                         (((int64_t)X * Y * od[2] * 16 + 255) / 256) * 256);  // [X,Yo,Zo]
  const float inv = 1.0f / ((float)window * (float)window * (float)window);
  const int st = unpool_axis(reinterpret_cast<const float4*>(d_out), t2, 1, X, (int64_t)od[1] * od[2], od[0],
                             window, stride, inv, s);
  if (st) return st;
  *rows = t1;
  return unpool_axis(t2, t1, X, Y, od[2], od[1], window, stride, 1.f, s);
}

int out_size(int n, int r, int s) { return n < r ? 0 : (n - r) / s + 1; }

}  // namespace
}  // namespace pgb

using namespace pgb;

extern "C" {

int pgb_avg_pool3d_shape(const int32_t dims[3], int32_t window, int32_t stride, int32_t out_dims[3],
                         int64_t* scratch_bytes) {
  if (!dims || !out_dims || window < 1 || stride < 1) return PGB_ERR_ARG;
  for (int a = 0; a < 3; ++a) {
    if (dims[a] <= 0) return PGB_ERR_ARG;
    out_dims[a] = out_size(dims[a], window, stride);
    if (out_dims[a] <= 0) return PGB_ERR_UNSUPPORTED;  // window larger than the grid
  }
  if (scratch_bytes) {
    // two intermediates: [X,Y,Zo,4] and [X,Yo,Zo,4] floats
    const int64_t t1 = (int64_t)dims[0] * dims[1] * out_dims[2] * 16;
    const int64_t t2 = (int64_t)dims[0] * out_dims[1] * out_dims[2] * 16;
    *scratch_bytes = ((t1 + 255) / 256) * 256 + t2;
  }
  return PGB_OK;
}

int pgb_avg_pool3d_fwd(const float* cells, const int32_t dims[3], int32_t window, int32_t stride,
                       void* scratch, float* out, pgb_stream_t s) {
  int32_t od[3];
  int64_t bytes = 0;
  int st = pgb_avg_pool3d_shape(dims, window, stride, od, &bytes);
  if (st) return st;
  if (!cells || !scratch || !out) return PGB_ERR_ARG;
  if (((uintptr_t)cells | (uintptr_t)scratch | (uintptr_t)out) % 16) return PGB_ERR_ALIGN;
  const int X = dims[0], Y = dims[1], Z = dims[2];
  float4* t1 = reinterpret_cast<float4*>(scratch);
  float4* t2 = reinterpret_cast<float4*>((char*)scratch +
                                         (((int64_t)X * Y * od[2] * 16 + 255) / 256) * 256);
  const float inv = 1.0f / ((float)window * (float)window * (float)window);
  const float4* in = reinterpret_cast<const float4*>(cells);
  const int q = window / stride;
  if (q >= 2 && q <= kPoolBlocks) {
    pool_rows_kernel<<<blocks_of((int64_t)X * Y * (od[2] + 24)), 256, 0, s>>>(in, t1, (int64_t)X * Y, Z, od[2],
                                                                             window, stride);
    st = after_launch();
  } else {
    st = pool_axis(in, t1, (int64_t)X * Y, Z, 1, od[2], window, stride, 1.f, s);
  }
  if (st) return st;
  if ((st = pool_axis(t1, t2, X, Y, od[2], od[1], window, stride, 1.f, s))) return st;
  return pool_axis(t2, reinterpret_cast<float4*>(out), 1, X, (int64_t)od[1] * od[2], od[0], window, stride,
                   inv, s);
}

int pgb_avg_pool3d_bwd(const float* d_out, const int32_t dims[3], int32_t window, int32_t stride,
                       void* scratch, float* d_cells, pgb_stream_t s) {
  int32_t od[3];
  int64_t bytes = 0;
  int st = pgb_avg_pool3d_shape(dims, window, stride, od, &bytes);
  if (st) return st;
  if (!d_out || !scratch || !d_cells) return PGB_ERR_ARG;
  if (((uintptr_t)d_out | (uintptr_t)scratch | (uintptr_t)d_cells) % 16) return PGB_ERR_ALIGN;
  float4* rows = nullptr;
  if ((st = unpool_to_rows(d_out, dims, od, window, stride, scratch, &rows, s))) return st;
  return unpool_axis(rows, reinterpret_cast<float4*>(d_cells), (int64_t)dims[0] * dims[1], dims[2], 1, od[2],
                     window, stride, 1.f, s);
}

int pgb_avg_pool3d_bwd_adam(const float* d_out, const int32_t dims[3], int32_t window, int32_t stride,
                            void* scratch, float* param, float* exp_avg, float* exp_avg_sq,
                            float* abs_grad_accum, double lr, double beta1, double beta2, double eps,
                            int64_t step, pgb_stream_t s) {
  int32_t od[3];
  int64_t bytes = 0;
  int st = pgb_avg_pool3d_shape(dims, window, stride, od, &bytes);
  if (st) return st;
  if (!d_out || !scratch || !param || !exp_avg || !exp_avg_sq || step < 1) return PGB_ERR_ARG;
  if (((uintptr_t)d_out | (uintptr_t)scratch | (uintptr_t)param | (uintptr_t)exp_avg |
       (uintptr_t)exp_avg_sq | (uintptr_t)abs_grad_accum) % 16)
    return PGB_ERR_ALIGN;
  float4* rows = nullptr;
  if ((st = unpool_to_rows(d_out, dims, od, window, stride, scratch, &rows, s))) return st;
  const int64_t n = (int64_t)dims[0] * dims[1], total = n * dims[2];
  const unsigned blocks = (unsigned)std::max<int64_t>(1, std::min<int64_t>((total + 255) / 256, 152 * 16));
  float4 *p = (float4*)param, *m = (float4*)exp_avg, *v = (float4*)exp_avg_sq, *a = (float4*)abs_grad_accum;
  const AdamConst k = adam_const(lr, beta1, beta2, eps, step);
  if (small_index(total))
    unpool_adam_kernel<uint32_t><<<blocks, 256, 0, s>>>(rows, p, m, v, a, (uint32_t)n, dims[2], od[2], window,
                                                       stride, k);
  else
    unpool_adam_kernel<int64_t><<<blocks, 256, 0, s>>>(rows, p, m, v, a, n, dims[2], od[2], window, stride, k);
  return after_launch();
}

}  // extern "C"
