// Fused render kernels: ray sampling -> voxel lookup -> front-to-back compositing, and the
// hand-written adjoint, one warp per ray.
//
// What one launch replaces (paths relative to the reference repository):
//   src/ray_sampling.py:195-264  generate_rays_batched       (in-kernel when cameras are given)
//   src/ray_sampling.py:161-167  sample positions o + d * (delta * k)
//   src/ray_sampling.py:12-13    normalisation (p - min) / points_distance
//   src/grid_functions.py:103-114 nearest lookup / :7-44, :220-246 trilinear lookup
//   scripts/train.py:146-147     grid.clip(0, 1) and the in-bounds mask
//   src/ray_sampling.py:172-192  compute_alpha_weighted_pixels
//   scripts/train.py:156, 181    mse_loss and its backward through all of the above
//
// Work layout: a warp owns one ray at a time. Samples are dealt to lanes in "slots":
// slot k of lane l is sample 32*k + l, so each load instruction of a warp touches 32
// consecutive samples of one ray (a compact run of cells). A chunk is K slots (32*K
// samples). The transmittance is an exclusive prefix product, computed per slot with a
// warp scan and carried across slots and chunks. The adjoint needs, per sample,
//     d alpha_s = T_s * (G_s - S_{s+1}),   G_s = <g_rgb, c_s> + g_A,
//     S_s = G_s * alpha_s + (1 - alpha_s) * S_{s+1},  S_{end} = 0,
// a suffix recurrence of affine maps evaluated with a second warp scan. It contains no
// division, so alpha == 1 (transmittance exactly 0 after the clip) is exact. Per-sample
// values of the current chunk stay in registers; in the reverse pass the chunks before the
// last come back from the warp's shared-memory stage (the last few chunks) or are gathered
// again from the grid (the transmittance at each chunk start is kept in lane c).
#pragma once

#include <type_traits>

#include "pgb_device.cuh"

namespace pgb {

enum Phase { kForward = 0, kBackward = 1, kTrain = 2 };

template <typename Real>
struct GridP {
  const void* cells;
  int X, Y, Z;
  Real fX, fY, fZ;
  Real ox, oy, oz;
  Real pd;
  int clip;
  float alpha_floor;  // >0: clamped alpha below it reads as 0 (inference threshold)
  Real inv_pd;        // 1 / pd, rounded to nearest
  Real box_lo[3], box_hi[3];  // the box of ray_span (set_box)
  int quick;          // the grid is in the range of the quick index arithmetic (quick_grid)
};

// Which index arithmetic a kernel is compiled with: the general one (any grid), the quick
// one (fp32 grids for which quick_grid holds), or either, by GridP::quick at run time.
enum Arith { kGeneral = 0, kQuick = 1, kByGrid = 2 };

template <int A, typename Real>
__device__ __forceinline__ bool use_quick(const GridP<Real>& g) {
  if constexpr (sizeof(Real) != 4 || A == kGeneral) return false;
  else if constexpr (A == kQuick) return true;
  else return g.quick != 0;
}

// Whether an fp32 grid is in the range of the quick index arithmetic:
//  - indices: every dimension at most 2^21, so that adding 2^23 or 1.5 * 2^23 leaves the
//    rounded coordinate in the low mantissa bits (of any coordinate that is in bounds; all
//    others still compare out of bounds), and fewer than 2^32 cells, so that a cell index
//    is one 32-bit word;
//  - the division by pd as a multiplication by its reciprocal with two fused corrections
//    (div_pd): needs quotients and remainders clear of underflow. With |origin| >= 2^-20
//    the difference p - origin is 0 or at least 2^-45 in magnitude (below a factor of two
//    it is a multiple of an ulp of the smaller operand, beyond that it is at least half of
//    |origin|), and pd within 2^+-40 keeps the rest normal.
// Grids outside (an axis of one or two cells has origin 0, and a caller may give it) take the
// general arithmetic.
constexpr float kQuickMinOrigin = 9.5367431640625e-07f;  // 2^-20

__host__ __device__ inline bool quick_grid(int X, int Y, int Z, float ox, float oy, float oz,
                                           float pd) {
  const auto fits = [](float o) {
    const float m = o < 0.f ? -o : o;
    return m >= kQuickMinOrigin && m <= 1.0995116e12f;
  };
  constexpr int kMaxDim = 1 << 21;
  return X <= kMaxDim && Y <= kMaxDim && Z <= kMaxDim &&
         (uint64_t)X * (uint64_t)Y * (uint64_t)Z < (1ull << 32) && fits(ox) && fits(oy) && fits(oz) &&
         pd >= 9.094947e-13f && pd <= 1.0995116e12f;
}

// A sum of fp32 numbers kept exactly, so that it comes out the same in whatever order rays
// are taken: each term's 24-bit mantissa is added as an integer to the bin of its exponent
// (bin b: exponents 8 b .. 8 b + 7, worth 2^(8 b - 150)), 31 bits a term in a 64-bit bin.
// Lane b of a warp holds bin b; infinities and NaN are flags beside them.
struct BinSum {
  long long bin = 0;
  unsigned special = 0u;  // bit 0: +inf, 1: -inf, 2: NaN
  __device__ __forceinline__ void add(float x, int lane) {  // the same x in every lane
    const uint32_t u = __float_as_uint(x), e = (u >> 23) & 0xffu, m = u & 0x7fffffu;
    if (e == 0xffu) {
      special |= m != 0u ? 4u : (u >> 31) ? 2u : 1u;
      return;
    }
    const uint32_t ex = e != 0u ? e : 1u;
    const long long t = (long long)(e != 0u ? m | 0x800000u : m) << (ex & 7u);
    if ((uint32_t)lane == ex >> 3) bin += (u >> 31) ? -t : t;
  }
  // the value over all lanes' bins
  __device__ __forceinline__ double value(int lane) const {
    const double unit = __longlong_as_double((long long)(1023 + 8 * lane - 150) << 52);
    const double sum = warp_sum((double)bin * unit);
    const double inf = __longlong_as_double(0x7ff0000000000000ll);
    if (special == 0u) return sum;
    return (special & 4u) || (special & 3u) == 3u ? inf - inf : (special & 1u) ? inf : -inf;
  }
};

// What the warps of a training launch share (fp32). All zero between launches.
struct TrainState {
  unsigned long long bins[2][kWarp];  // squared errors, beta terms
  unsigned special[2];
  unsigned blocks_done;
};

template <typename Real>
struct RenderArgs {
  GridP<Real> g;
  // explicit rays
  const Real* origins;
  const Real* dirs;
  // in-kernel camera rays
  int use_cameras;
  const float* transforms;
  const float* images;
  int C, H, W;
  float fov, near_dist;
  uint64_t cam_seed;
  // sampling
  int64_t R;
  int S;
  Real delta, inv_delta;
  int stratified;
  uint64_t strat_seed;
  int64_t first_ray;  // index of ray 0 in the stratification stream
  float term_thr;
  int chunk_samples;  // host-side chunk request (pick_slots)
  int long_ray;    // the ray would be one long chunk (rounding of the suffix scan)
  int group_log2;  // a block's rays come in groups of 2^group_log2 consecutive ones
  int use_bg;      // rgb += (1 - A) * bg after compositing
  float bg[3];
  // outputs / adjoint inputs
  Real* rgba_out;
  const Real* d_rgba;
  const Real* target;
  Real* grad;
  uint32_t* grad_marks;  // optional: units of written gradient cells are marked here
  // optional (fp32 training): another gradient buffer whose marked units are zeroed (without
  // marks: the whole of it)
  uint4* clear_grad;
  int64_t clear_total16;
  uint32_t* clear_marks;
  int64_t clear_words;
  int clear_early;  // some warps begin with the clear
  Real* loss_out;
  double* partials;  // fp64: block loss partials, and the block counter
  unsigned* counter;
  TrainState* state;  // fp32
  double loss_w;
  double inv_count;
  // beta loss of scripts/train.py:170-177: beta_w * mean over all R*S samples of
  // log(alpha + eps) - log(1 - alpha + eps) (0: off)
  double beta_w;
  float beta_eps;
  double inv_samples;
  double* partials_beta;
  // derived on the host (finish_args): GB300's fp64 rate is low, and every warp would
  // otherwise evaluate these double expressions at its start
  int use_beta;       // beta_w != 0
  Real grad_scale;    // 2 * loss_w * inv_count: d(weighted MSE)/d pixel
  Real beta_scale;    // beta_w * inv_samples * (1 + 2 eps)
  Real beta_zero;     // log(eps) - log(1 + eps): the beta term of a sample of alpha 0
};

template <typename Real>
struct Ray {
  Real ox, oy, oz, dx, dy, dz;
  Real tgt;    // channel (lane % 4) of the target pixel
  uint64_t h;  // stratification stream of this ray
};

// Euclidean norm of a 3-vector as the reference's CPU torch.norm evaluates it. Over a
// contiguous last dimension (the direction tensor) it accumulates with FMAs:
// sqrt(fma(z, z, fma(y, y, x * x))); over a strided view (the camera axes T[:, :3, i])
// it rounds every product and sum: sqrt((x*x + y*y) + z*z).
__device__ __forceinline__ float norm3_ref(float x, float y, float z) {
  return rsqrt_exact(rfma(z, z, rfma(y, y, rmul(x, x))));
}
__device__ __forceinline__ float norm3_strided_ref(float x, float y, float z) {
  return rsqrt_exact(radd(radd(rmul(x, x), rmul(y, y)), rmul(z, z)));
}

// Direction of a camera ray from uniforms (u, v), src/ray_sampling.py:215-262, rounded
// op by op as the reference's fp32 tensor program.
__device__ __forceinline__ void camera_direction(const float* T, float fov, float u, float v,
                                                 float d[3]) {
  // T is row-major 4x4: column 0 = x axis, column 1 = y axis, column 2 = back axis.
  const float xa0 = T[0], xa1 = T[4], xa2 = T[8];
  const float ya0 = T[1], ya1 = T[5], ya2 = T[9];
  const float za0 = -T[2], za1 = -T[6], za2 = -T[10];
  const float aspect = rdiv(norm3_strided_ref(xa0, xa1, xa2), norm3_strided_ref(ya0, ya1, ya2));
  const float ru = rmul(fov, rsub(u, 0.5f));
  const float rv = -rmul(rmul(fov, rdiv(1.0f, aspect)), rsub(v, 0.5f));
  const float e0 = radd(radd(rmul(ru, xa0), rmul(rv, ya0)), za0);
  const float e1 = radd(radd(rmul(ru, xa1), rmul(rv, ya1)), za1);
  const float e2 = radd(radd(rmul(ru, xa2), rmul(rv, ya2)), za2);
  const float n = norm3_ref(e0, e1, e2);
  d[0] = rdiv(e0, n);
  d[1] = rdiv(e1, n);
  d[2] = rdiv(e2, n);
}

// Pixel of a ray (src/ray_sampling.py:238-248): column from u scaled by H, row from v
// scaled by W, round half to even, clamp to the last index.
__device__ __forceinline__ void camera_pixel(int H, int W, float u, float v, int& row, int& col) {
  col = (int)fminf(rintf(rmul((float)H, u)), (float)(H - 1));
  row = (int)fminf(rintf(rmul((float)W, v)), (float)(W - 1));
}

template <typename Real>
__device__ __forceinline__ void load_ray(const RenderArgs<Real>& a, int64_t r, Ray<Real>& ray,
                                         bool need_target) {
  if (a.use_cameras) {
    // cameras get contiguous runs of rays (camera-major, src/ray_sampling.py:243)
    // floor(r * C / R), in 32-bit arithmetic when r * C fits (the 64-bit divide is a long
    // instruction sequence)
    const uint64_t rc = (uint64_t)r * (uint64_t)a.C;
    const int c = (rc >> 32) == 0 && ((uint64_t)a.R >> 32) == 0
                      ? (int)((uint32_t)rc / (uint32_t)a.R)
                      : (int)(rc / (uint64_t)a.R);
    const float* T = a.transforms + 16 * (int64_t)c;
    const uint64_t h = hash_stream(a.cam_seed, (uint64_t)r);
    const float u = hash_to_unit(h, 0u), v = hash_to_unit(h, 1u);
    float d[3];
    camera_direction(T, a.fov, u, v, d);
    ray.dx = d[0]; ray.dy = d[1]; ray.dz = d[2];
    ray.ox = radd(T[3], rmul(a.near_dist, d[0]));
    ray.oy = radd(T[7], rmul(a.near_dist, d[1]));
    ray.oz = radd(T[11], rmul(a.near_dist, d[2]));
    if (need_target) {
      int row, col;
      camera_pixel(a.H, a.W, u, v, row, col);
      ray.tgt = __ldg(a.images + 4 * (((int64_t)c * a.H + row) * a.W + col) + (threadIdx.x & 3));
    }
  } else {
    ray.ox = a.origins[3 * r + 0]; ray.oy = a.origins[3 * r + 1]; ray.oz = a.origins[3 * r + 2];
    ray.dx = a.dirs[3 * r + 0];    ray.dy = a.dirs[3 * r + 1];    ray.dz = a.dirs[3 * r + 2];
    if (need_target) ray.tgt = a.target[4 * r + (threadIdx.x & 3)];
  }
  ray.h = a.stratified ? hash_stream(a.strat_seed, (uint64_t)(r + a.first_ray)) : 0ull;
}

// Normalised grid coordinates of sample s (0-based) of a ray:
//   t = delta * (s + 1) [- jitter],  p = o + d * t,  n = (p - origin) / pd
// each op rounded separately (src/ray_sampling.py:161-167, :13).
//
// div_pd is x / pd rounded to nearest for a grid with `quick` set: from the rounded
// reciprocal y = 1 / pd, two corrections q += (x - q * pd) * y with fused multiply-adds. The
// first brings q within one unit in the last place, where the remainder is exact; the
// second then gives the correctly rounded quotient (P. Markstein, "Computation of
// elementary functions on the IBM RISC System/6000 processor", IBM J. Res. Dev. 34, 1990).
// Five multiply-adds and no special-case branch per quotient instead of an IEEE division.
__device__ __forceinline__ float div_pd(float x, float pd, float y) {
  float q = rmul(x, y);
  q = rfma(rfma(-q, pd, x), y, q);
  return rfma(rfma(-q, pd, x), y, q);
}

template <int A, typename Real>
__device__ __forceinline__ void sample_coords(const RenderArgs<Real>& a, const Ray<Real>& ray,
                                              int s, Real& nx, Real& ny, Real& nz) {
  Real k = (Real)(s + 1);
  if (a.stratified) k = rsub(k, (Real)hash_to_unit(ray.h, (uint32_t)s));
  const Real t = rmul(a.delta, k);
  const Real px = radd(ray.ox, rmul(ray.dx, t));
  const Real py = radd(ray.oy, rmul(ray.dy, t));
  const Real pz = radd(ray.oz, rmul(ray.dz, t));
  const Real x = rsub(px, a.g.ox), y = rsub(py, a.g.oy), z = rsub(pz, a.g.oz);
  if (use_quick<A>(a.g)) {
    if constexpr (sizeof(Real) == 4) {
      nx = div_pd(x, a.g.pd, a.g.inv_pd);
      ny = div_pd(y, a.g.pd, a.g.inv_pd);
      nz = div_pd(z, a.g.pd, a.g.inv_pd);
      if constexpr (A == kByGrid) {
        // the views report the quotient also where it is not finite (the corrections make NaN of
        // an infinity, which is as much out of bounds)
        if (isinf(rdiv(x, a.g.pd))) nx = rdiv(x, a.g.pd);
        if (isinf(rdiv(y, a.g.pd))) ny = rdiv(y, a.g.pd);
        if (isinf(rdiv(z, a.g.pd))) nz = rdiv(z, a.g.pd);
      }
    }
  } else {
    nx = rdiv(x, a.g.pd);
    ny = rdiv(y, a.g.pd);
    nz = rdiv(z, a.g.pd);
  }
}

template <typename Real>
__device__ __forceinline__ uint64_t cell_index(const GridP<Real>& g, int i, int j, int k) {
  return ((uint64_t)i * (uint64_t)g.Y + (uint64_t)j) * (uint64_t)g.Z + (uint64_t)k;
}

// The samples [first, end) of a ray outside of which every sample is out of bounds (value
// 0, no gradient): the ray against the grid's box, grown by a hundredth of a cell and by
// 2^-18 of the coordinates' magnitude (64 times what the rounding of a position or of the
// arithmetic here can move it), and two samples more at both ends (the jitter of stratified
// samples and the rounding of the quotients). An axis whose bounds come out NaN restricts
// nothing, and neither does a step that is not a positive normal number. `first` is a multiple of
// 32: the scans of a slot then run over the samples that they would without the cut, with the
// same rounding. Rays enter and leave the grid well inside their [near, far] range, so this
// spares a quarter of the benchmark's samples: their chunks ran the coordinate arithmetic and
// both scans for zeros. A ray of a few chunks may spare none, so the box and 1 / delta are
// made once and the reciprocals are approximate ones.
constexpr float kSpanSlack = 3.8147e-6f;  // 2^-18

template <typename Real>
__host__ __device__ inline void set_box(GridP<Real>& g) {
  const Real org[3] = {g.ox, g.oy, g.oz}, dim[3] = {g.fX, g.fY, g.fZ};
  const auto mag = [](Real x) { return x < Real(0) ? -x : x; };
  for (int ax = 0; ax < 3; ++ax) {
    const Real lo = org[ax] - Real(0.5) * g.pd, hi = org[ax] + dim[ax] * g.pd;
    const Real grow = Real(0.01) * g.pd + Real(kSpanSlack) * (mag(lo) + mag(hi));
    g.box_lo[ax] = lo - grow;
    g.box_hi[ax] = hi + grow;
  }
}

template <typename Real>
__device__ __forceinline__ void ray_span(const RenderArgs<Real>& a, const Ray<Real>& ray, int& first,
                                         int& end) {
  first = 0;
  end = a.S;
  if constexpr (sizeof(Real) == 4) {
    if (!(a.delta >= 1e-30f) || !(a.g.pd > 0.f)) return;
    const float o[3] = {ray.ox, ray.oy, ray.oz}, d[3] = {ray.dx, ray.dy, ray.dz};
    float t0 = 0.f, t1 = __int_as_float(0x7f800000);
#pragma unroll
    for (int ax = 0; ax < 3; ++ax) {
      const float slack = kSpanSlack * fabsf(o[ax]);
      float inv;
      asm("rcp.approx.f32 %0, %1;" : "=f"(inv) : "f"(d[ax]));
      const float ta = (a.g.box_lo[ax] - o[ax] - slack) * inv, tb = (a.g.box_hi[ax] - o[ax] + slack) * inv;
      t0 = fmaxf(t0, fminf(ta, tb));  // fminf and fmaxf pass the other operand of a NaN
      t1 = fminf(t1, fmaxf(ta, tb));
    }
    // t of sample s lies in [delta * s, delta * (s + 1)]
    const float most = (float)a.S;
    first = (int)fminf(fmaxf(t0 * a.inv_delta - 3.f, 0.f), most) & ~(kWarp - 1);
    end = max(first, (int)fminf(fmaxf(t1 * a.inv_delta + 3.f, 0.f), most));
  }
}

// Nearest cell of normalised coordinates: false outside the grid. Quick form: adding
// 1.5 * 2^23 rounds to the nearest integer, ties to even, into the low mantissa bits; one
// unsigned comparison of those bits tests both bounds (every coordinate that is not in
// bounds, infinities and NaN included, leaves a value of 2^22 or more). Rounding and
// converting through the conversion unit took a quarter-rate instruction each.
template <int A, typename Real>
__device__ __forceinline__ bool nearest_cell(const GridP<Real>& g, Real nx, Real ny, Real nz,
                                             uint64_t& cell) {
  if (use_quick<A>(g)) {
    constexpr float kRound = 12582912.0f;  // 1.5 * 2^23
    constexpr int kBits = 0x4B400000;
    const uint32_t i = (uint32_t)(__float_as_int(radd((float)nx, kRound)) - kBits);
    const uint32_t j = (uint32_t)(__float_as_int(radd((float)ny, kRound)) - kBits);
    const uint32_t k = (uint32_t)(__float_as_int(radd((float)nz, kRound)) - kBits);
    if (!(i < (uint32_t)g.X && j < (uint32_t)g.Y && k < (uint32_t)g.Z)) return false;
    cell = (i * (uint32_t)g.Y + j) * (uint32_t)g.Z + k;
    return true;
  }
  const Real rx = rround(nx), ry = rround(ny), rz = rround(nz);
  if (!(rx >= Real(0) && rx < g.fX && ry >= Real(0) && ry < g.fY && rz >= Real(0) && rz < g.fZ))
    return false;
  cell = cell_index(g, (int)rx, (int)ry, (int)rz);
  return true;
}

// Trilinear corner geometry of an in-bounds sample: wrapped ceil/floor indices per axis
// and the fractional weights (src/grid_functions.py:29, :230-244, :75-77). For an
// in-bounds coordinate 0 <= n < dim, only ceil can leave the grid (n in (dim-1, dim)),
// and it wraps to 0.
template <typename Real>
struct Corners {
  int c[3], f[3];
  Real w[3];  // frac(n) per axis
};

//
// Quick form: adding 2^23 rounding down leaves floor(n) in the low mantissa bits of an
// in-bounds coordinate, and ceil is one more unless n is whole.
template <int A, typename Real>
__device__ __forceinline__ bool trilinear_corners(const GridP<Real>& g, Real nx, Real ny, Real nz,
                                                  Corners<Real>& q) {
  if (!(nx >= Real(0) && nx < g.fX && ny >= Real(0) && ny < g.fY && nz >= Real(0) && nz < g.fZ))
    return false;
  const Real n[3] = {nx, ny, nz};
  const int dim[3] = {g.X, g.Y, g.Z};
#pragma unroll
  for (int ax = 0; ax < 3; ++ax) {
    if (use_quick<A>(g)) {
      if constexpr (sizeof(Real) == 4) {
        constexpr float kTwo23 = 8388608.0f;
        const float m = __fadd_rd(n[ax], kTwo23);
        q.f[ax] = __float_as_int(m) & 0x7fffff;
        q.w[ax] = rsub(n[ax], rsub(m, kTwo23));
        const int ce = q.f[ax] + (q.w[ax] > 0.f ? 1 : 0);
        q.c[ax] = ce == dim[ax] ? 0 : ce;
      }
    } else {
      const Real fl = rfloor(n[ax]);
      q.f[ax] = (int)fl;
      const int ce = (int)rceil(n[ax]);
      q.c[ax] = ce >= dim[ax] ? ce - dim[ax] : ce;
      q.w[ax] = rsub(n[ax], fl);  // == n - trunc(n) for n >= 0
    }
  }
  return true;
}

// The eight corner cells of a sample (corner order of src/grid_functions.py:16-24), as
// 32-bit indices in the quick form.
template <int A, typename Real>
struct CornerCells {
  using Index = typename std::conditional<A == kQuick && sizeof(Real) == 4, uint32_t, uint64_t>::type;
  Index row[4];  // (x, y) rows: ceil/ceil, ceil/floor, floor/ceil, floor/floor
  Index zc, zf;
  __device__ __forceinline__ CornerCells(const GridP<Real>& g, const Corners<Real>& q) {
    const Index Y = (Index)g.Y, Z = (Index)g.Z;
    const Index xc = (Index)q.c[0] * Y, xf = (Index)q.f[0] * Y;
    row[0] = (xc + (Index)q.c[1]) * Z;
    row[1] = (xc + (Index)q.f[1]) * Z;
    row[2] = (xf + (Index)q.c[1]) * Z;
    row[3] = (xf + (Index)q.f[1]) * Z;
    zc = (Index)q.c[2];
    zf = (Index)q.f[2];
  }
  __device__ __forceinline__ Index operator()(int corner) const {
    return row[corner >> 1] + ((corner & 1) ? zf : zc);
  }
};

// Two fp32 values in one register pair, for the paired fp32 instructions (one issue slot
// for two operations, each rounded as the scalar one).
struct F2 {
  unsigned long long v;
  __device__ __forceinline__ static F2 of(float lo, float hi) {
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(lo), "f"(hi));
    return r;
  }
  __device__ __forceinline__ void get(float& lo, float& hi) const {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
  }
};
__device__ __forceinline__ F2 sub2(F2 a, F2 b) {
  F2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 add2(F2 a, F2 b) {
  F2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 mul2(F2 a, F2 b) {
  F2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}

// clamp01 of a sample's N cells and (BITS) the flags of the values inside [0, 1], which the
// clamp lets the gradient through. Kernels are bound by the logic pipe here (it runs at half
// the rate of the multiply-add pipe), so the clamp is the saturating add of the latter, and
// a flag is one unsigned comparison: negative values and NaN compare above 1's bits, and
// -0 is inside once 0 is added to it. Saturation turns NaN into 0 where the reference's
// clamp keeps it; returns the channels in which a cell is NaN (a sum of all values finds
// that there may be one: also of infinities of both signs).
template <bool BITS, int N>
__device__ __forceinline__ uint32_t clamp_cells(float cv[N][4], uint32_t& bits) {
  F2 sum = F2::of(cv[0][0], cv[0][1]);
  sum = add2(sum, F2::of(cv[0][2], cv[0][3]));
#pragma unroll
  for (int i = 1; i < N; ++i)
    sum = add2(add2(sum, F2::of(cv[i][0], cv[i][1])), F2::of(cv[i][2], cv[i][3]));
  float lo, hi;
  sum.get(lo, hi);
  uint32_t nan = 0u;
  if (!(lo + hi == lo + hi)) {
#pragma unroll
    for (int i = 0; i < 4 * N; ++i) nan |= cv[i / 4][i % 4] != cv[i / 4][i % 4] ? 1u << (i % 4) : 0u;
  }
#pragma unroll
  for (int i = 0; i < 4 * N; ++i) {
    if (BITS && i % 2 == 0) {
      float& x = cv[i / 4][i % 4];
      float& y = cv[i / 4][i % 4 + 1];
      add2(F2::of(x, y), F2::of(0.f, 0.f)).get(x, y);
    }
    const float x = cv[i / 4][i % 4];
    if (BITS) bits |= __float_as_uint(x) <= 0x3f800000u ? 1u << i : 0u;
    cv[i / 4][i % 4] = __saturatef(x);
  }
  return nan;
}

// What the quick index arithmetic, the cut of a ray (ray_span), these clamps and the paired
// blend gave together (the forward kernel spent 69 % of the logic pipe's cycles and 1800
// warp instructions per ray): three 400 x 400 pictures of a 256^3 grid 1.23 -> 0.98 ms, the
// 512^3 BF16 log-sum step of 65,536 rays 0.464 -> 0.372 ms, the batched step of 16 scenes
// 1.54 -> 1.31 ms, the 8192-ray trilinear step of 256^3 0.100 -> 0.092 ms.
//
// Value of one sample, masked to zero outside the grid. bits: gradient-pass flags of
// the clamp, bit 4*corner + channel (trilinear; corner order of
// src/grid_functions.py:16-24) or bit channel (nearest). Zero when out of bounds; not
// written without BITS (a forward pass needs none).
template <typename Real, typename Store, int MODE, int A, bool BITS>
__device__ __forceinline__ void sample_value(const GridP<Real>& g, Real nx, Real ny, Real nz,
                                             Real v[4], uint32_t& bits) {
  constexpr int N = MODE == PGB_NEAREST ? 1 : 8;  // cells of a sample
  bits = 0u;
  v[0] = v[1] = v[2] = v[3] = Real(0);
  Real cv[N][4];
  Real wx = Real(0), wy = Real(0), wz = Real(0);
  if constexpr (MODE == PGB_NEAREST) {
    uint64_t cell;
    if (!nearest_cell<A>(g, nx, ny, nz, cell)) return;
    CellIO<Store>::load(g.cells, cell, cv[0]);
  } else {
    Corners<Real> q;
    if (!trilinear_corners<A>(g, nx, ny, nz, q)) return;
    const CornerCells<A, Real> cells(g, q);
#pragma unroll
    for (int corner = 0; corner < N; ++corner) CellIO<Store>::load(g.cells, cells(corner), cv[corner]);
    wx = q.w[0];
    wy = q.w[1];
    wz = q.w[2];
  }
  uint32_t nan = 0u;  // channels with a NaN cell (fp32)
  if (g.clip) {
    if constexpr (sizeof(Real) == 4) {
      nan = clamp_cells<BITS, N>(cv, bits);
    } else {
#pragma unroll
      for (int i = 0; i < 4 * N; ++i) {
        Real& x = cv[i / 4][i % 4];
        bits |= (in01(x) ? 1u : 0u) << i;
        x = clamp01(x);
      }
    }
  } else {
    bits = MODE == PGB_NEAREST ? 0xfu : 0xffffffffu;
  }
  if (g.alpha_floor > 0.0f) {
#pragma unroll
    for (int corner = 0; corner < N; ++corner) {
      if (cv[corner][3] < (Real)g.alpha_floor) {
        cv[corner][3] = Real(0);
        bits &= ~(8u << (4 * corner));
      }
    }
  }
  if constexpr (MODE == PGB_NEAREST) {
#pragma unroll
    for (int ch = 0; ch < 4; ++ch) v[ch] = cv[0][ch];
  } else {
    // blend x, then y, then z, as src/grid_functions.py:34-42
    if constexpr (sizeof(Real) == 4) {
      // Products of channel pairs, every operation rounded as below. The sums are scalar ones:
      // the assembler fuses a paired multiplication into a paired addition whatever their
      // rounding suffixes say, and a blend an ulp away turns up as 6e-4 of a gradient where
      // the beta term's 1 / (1 - alpha + eps) meets an opacity near 1. (Same time.)
      const F2 one = F2::of(1.f, 1.f);
      const F2 wx2 = F2::of(wx, wx), wy2 = F2::of(wy, wy), wz2 = F2::of(wz, wz);
      const F2 ux2 = sub2(one, wx2), uy2 = sub2(one, wy2), uz2 = sub2(one, wz2);
      const auto blend = [](F2 a, F2 w, F2 b, F2 u) {
        float p, q, r, s;
        mul2(a, w).get(p, q);
        mul2(b, u).get(r, s);
        return F2::of(radd(p, r), radd(q, s));
      };
#pragma unroll
      for (int p = 0; p < 4; p += 2) {
        F2 a4[4];
#pragma unroll
        for (int yz = 0; yz < 4; ++yz)
          a4[yz] = blend(F2::of(cv[yz][p], cv[yz][p + 1]), wx2,
                         F2::of(cv[4 + yz][p], cv[4 + yz][p + 1]), ux2);
        const F2 b0 = blend(a4[0], wy2, a4[2], uy2), b1 = blend(a4[1], wy2, a4[3], uy2);
        blend(b0, wz2, b1, uz2).get(v[p], v[p + 1]);
      }
    } else {
      const Real ux = rsub(Real(1), wx), uy = rsub(Real(1), wy), uz = rsub(Real(1), wz);
#pragma unroll
      for (int ch = 0; ch < 4; ++ch) {
        Real a4[4];
#pragma unroll
        for (int yz = 0; yz < 4; ++yz)
          a4[yz] = radd(rmul(cv[yz][ch], wx), rmul(cv[4 + yz][ch], ux));
        const Real b0 = radd(rmul(a4[0], wy), rmul(a4[2], uy));
        const Real b1 = radd(rmul(a4[1], wy), rmul(a4[3], uy));
        v[ch] = radd(rmul(b0, wz), rmul(b1, uz));
      }
    }
  }
  if (nan != 0u) {
#pragma unroll
    for (int ch = 0; ch < 4; ++ch)
      if ((nan >> ch) & 1u) v[ch] = (Real)__int_as_float(0x7fffffff);
  }
}

#ifndef PGB_SCATTER_INLINE
#define PGB_SCATTER_INLINE 1
#endif
#if PGB_SCATTER_INLINE
#define PGB_SCATTER_ATTR __device__ __forceinline__
#else
#define PGB_SCATTER_ATTR __device__ __noinline__
#endif

// Marks the gradient unit of cell c in the bitmap of units (mark_unit_of).
__device__ __forceinline__ void mark_unit(uint32_t* marks, uint64_t c) {
  const uint64_t u = mark_unit_of(c);
  atomicOr(marks + (u >> 5), 1u << ((uint32_t)u & 31u));
}

// Scatter dL/dvalue of one sample into the dense gradient (the autograd replay of the
// blend, the clamp mask and index_put accumulate). marks (optional): the unit of every
// written cell is marked.
//
// Which corners are written follows from the flags and the non-zero partials alone (a
// corner whose weight is 0 gets an update of zeros): one test per corner instead of a
// product and a comparison per channel.
template <typename Real, int MODE, int A>
PGB_SCATTER_ATTR void sample_scatter(const GridP<Real>& g, Real* grad, Real nx, Real ny,
                                     Real nz, const Real dv[4], uint32_t bits,
                                     uint32_t* marks = nullptr) {
  uint32_t live = 0u;  // channels with a non-zero partial
#pragma unroll
  for (int ch = 0; ch < 4; ++ch) live |= dv[ch] != Real(0) ? 1u << ch : 0u;
  if (MODE == PGB_NEAREST) {
    bits &= live;
    if (bits == 0u) return;
    uint64_t c;
    if (!nearest_cell<A>(g, nx, ny, nz, c)) return;
    Real gv[4];
#pragma unroll
    for (int ch = 0; ch < 4; ++ch) gv[ch] = ((bits >> ch) & 1u) ? dv[ch] : Real(0);
    grad_add(grad, c, gv);
    if (marks != nullptr) mark_unit(marks, c);
  } else {
    bits &= live * 0x11111111u;
    if (bits == 0u) return;
    Corners<Real> q;
    if (!trilinear_corners<A>(g, nx, ny, nz, q)) return;
    const CornerCells<A, Real> cells(g, q);
    const Real wx = q.w[0], wy = q.w[1], wz = q.w[2];
    const Real ux = rsub(Real(1), wx), uy = rsub(Real(1), wy), uz = rsub(Real(1), wz);
    // corner weights, corner order of src/grid_functions.py:16-24
    const Real wyz[4] = {wy * wz, wy * uz, uy * wz, uy * uz};
#pragma unroll
    for (int pair = 0; pair < 4; ++pair) {  // the ceil and the floor corner along z
      const uint32_t pb = (bits >> (8 * pair)) & 0xffu;
      if (pb == 0u) continue;
#pragma unroll
      for (int f = 0; f < 2; ++f) {
        const int corner = 2 * pair + f;
        const uint32_t cb = bits >> (4 * corner);
        if ((cb & 0xfu) == 0u) continue;
        const Real wc = ((corner & 4) ? ux : wx) * wyz[corner & 3];
        Real gv[4];
#pragma unroll
        for (int ch = 0; ch < 4; ++ch) gv[ch] = ((cb >> ch) & 1u) ? dv[ch] * wc : Real(0);
        grad_add(grad, cells(corner), gv);
      }
      if (marks != nullptr) {
        // the pair's two units mostly share a bitmap word: one OR then
        const uint64_t uc = mark_unit_of(cells(2 * pair)), uf = mark_unit_of(cells(2 * pair + 1));
        const uint32_t mc = (pb & 0x0fu) ? 1u << ((uint32_t)uc & 31u) : 0u;
        const uint32_t mf = (pb & 0xf0u) ? 1u << ((uint32_t)uf & 31u) : 0u;
        if ((uc >> 5) == (uf >> 5)) {
          atomicOr(marks + (uc >> 5), mc | mf);
        } else {
          if (mc) atomicOr(marks + (uc >> 5), mc);
          if (mf) atomicOr(marks + (uf >> 5), mf);
        }
      }
    }
  }
}

// sample_scatter for trilinear lookup with the updates of a warp merged per cell. For each
// corner, lanes whose update goes to the same cell as their lower neighbour's form a run
// (consecutive samples of a ray inside one cell, which is where a cell repeats: samples
// move monotonically along the ray); the run's partials are summed into its first lane
// by a segmented shuffle reduction and that lane issues the one atomic. A cell split
// over two runs gets two atomics, so the result is the same sum in another order. Every
// lane of the warp must call it; has = false marks a lane with nothing to add.
template <typename Real, int A>
__device__ __forceinline__ void warp_merged_scatter(const GridP<Real>& g, Real* grad, bool has,
                                                    Real nx, Real ny, Real nz, const Real dv[4],
                                                    uint32_t bits, int lane) {
  Corners<Real> q = {};
  if (has) has = trilinear_corners<A>(g, nx, ny, nz, q);
  const Real wx = q.w[0], wy = q.w[1], wz = q.w[2];
  const Real ux = Real(1) - wx, uy = Real(1) - wy, uz = Real(1) - wz;
  const Real wyz[4] = {wy * wz, wy * uz, uy * wz, uy * uz};
#pragma unroll 1
  for (int corner = 0; corner < 8; ++corner) {
    const uint32_t cb = has ? (bits >> (4 * corner)) & 0xfu : 0u;
    const Real wc = ((corner & 4) ? ux : wx) * wyz[corner & 3];
    Real gv[4];
    bool any = false;
#pragma unroll
    for (int ch = 0; ch < 4; ++ch) {
      gv[ch] = ((cb >> ch) & 1u) ? dv[ch] * wc : Real(0);
      any |= gv[ch] != Real(0);
    }
    if (!__any_sync(kFull, any)) continue;
    // a lane with nothing to add gets a key no other lane and no cell has
    const int ix = (corner & 4) ? q.f[0] : q.c[0];
    const int iy = (corner & 2) ? q.f[1] : q.c[1];
    const int iz = (corner & 1) ? q.f[2] : q.c[2];
    const uint64_t key = any ? cell_index(g, ix, iy, iz) : ~0ull - (uint64_t)lane;
    const uint64_t prev = __shfl_up_sync(kFull, key, 1);
    const bool head = lane == 0 || prev != key;
    const uint32_t heads = __ballot_sync(kFull, head);
    const uint32_t later = lane == kWarp - 1 ? 0u : heads & ~((2u << lane) - 1u);
    const int seg_end = later ? __ffs(later) - 2 : kWarp - 1;
#pragma unroll
    for (int d = 1; d < kWarp; d <<= 1) {
#pragma unroll
      for (int ch = 0; ch < 4; ++ch) {
        const Real y = __shfl_down_sync(kFull, gv[ch], d);
        if (lane + d <= seg_end) gv[ch] += y;
      }
    }
    if (head && any) grad_add(grad, key, gv);
  }
}

// Blocks of the render kernels (compile-time; the shipped values are the measured best on
// GB300). fp32 blocks share a queue of rays, so they are large: the fewer there are, the less
// the slowest one waits for. Nearest lookup runs one block of 32 warps per SM (64 registers;
// two of 16 warps took 76 us for 71 at 7500 rays x 600, 85 before the queue); trilinear
// lookup with 32-sample chunks two blocks of 12 warps for the gradient (80 registers; one of
// 24 warps the same within 2 %, six of 4 warps 345 us for 333) and two of 14 for a forward
// pass (72 registers). Longer trilinear chunks need 90 to 210 registers: 8 warps a block, two
// blocks of up to 256-sample chunks per SM (8192 rays x 256 with the beta term: 277 us with
// one, 185 with two). fp64 launches have a ray per warp, in blocks of 4 or 8 warps.
#ifndef PGB_RENDER_THREADS
#define PGB_RENDER_THREADS 256
#endif
#ifndef PGB_RENDER_THREADS_NEAREST
#define PGB_RENDER_THREADS_NEAREST 1024
#endif
#ifndef PGB_RENDER_THREADS_K1
#define PGB_RENDER_THREADS_K1 384
#endif
#ifndef PGB_RENDER_THREADS_FWD
#define PGB_RENDER_THREADS_FWD 448
#endif

// The per-warp shared-memory stage of the render and batched kernels: per chunk slot,
// for the last M chunks,
//   - the normalised coordinates (COORDS; otherwise the reverse pass recomputes them from
//     the ray: the stratification hash and the exact divisions),
//   - with M > 1, the clamped values and clamp-pass bits, so the reverse pass reads the
//     M - 1 chunks before the last from here instead of gathering them from the grid
//     again,
//   - with TS, the forward pass's transmittances, so the reverse pass skips their scan.
// Layout [slot][field][K][32]: each lane reads back only what it wrote, without bank
// conflicts.
template <typename Real, int K, int MSLOTS, bool COORDS = true, bool TS = false>
struct ChunkStage {
  static constexpr int M = MSLOTS;
  static constexpr bool kHasCoords = COORDS;
  static constexpr bool kHasTs = TS;  // the transmittance of every sample too
  static_assert((M & (M - 1)) == 0, "stage slots must be a power of two");
  static_assert(COORDS || M > 1, "a stage without coordinates holds values");
  static_assert(!TS || M > 1, "transmittances are held with the values");
  static constexpr int kCoordBytes = COORDS ? 3 * K * kWarp * (int)sizeof(Real) : 0;
  static constexpr int kVBytes = 4 * K * kWarp * (int)sizeof(Real);
  static constexpr int kBitsBytes = K * kWarp * 4;
  static constexpr int kTsBytes = TS ? K * kWarp * (int)sizeof(Real) : 0;
  static constexpr int kValBytes = M > 1 ? kVBytes + kBitsBytes + kTsBytes : 0;
  static constexpr int kSlotBytes = kCoordBytes + kValBytes;
  static constexpr int kBytesPerWarp = M * kSlotBytes;
  unsigned char* base;
  __device__ __forceinline__ ChunkStage(unsigned char* all, int warp)
      : base(all + (size_t)warp * kBytesPerWarp) {}
  __device__ __forceinline__ unsigned char* slot(int c) const { return base + (c & (M - 1)) * kSlotBytes; }
  // chunk c is still in the stage when the reverse pass reaches it (last = last chunk)
  __device__ __forceinline__ static bool holds(int c, int last) { return M > 1 && c > last - M; }
  __device__ __forceinline__ void put(int c, int k, int lane, Real x, Real y, Real z) {
    if constexpr (!COORDS) return;
    Real* n = reinterpret_cast<Real*>(slot(c));
    n[(0 * K + k) * kWarp + lane] = x;
    n[(1 * K + k) * kWarp + lane] = y;
    n[(2 * K + k) * kWarp + lane] = z;
  }
  __device__ __forceinline__ void get(int c, int k, int lane, Real& x, Real& y, Real& z) const {
    const Real* n = reinterpret_cast<const Real*>(slot(c));
    x = n[(0 * K + k) * kWarp + lane];
    y = n[(1 * K + k) * kWarp + lane];
    z = n[(2 * K + k) * kWarp + lane];
  }
  __device__ __forceinline__ void put_vals(int c, int k, int lane, const Real v[4], uint32_t bits) {
    if constexpr (M > 1) {
      Real* w = reinterpret_cast<Real*>(slot(c) + kCoordBytes);
#pragma unroll
      for (int ch = 0; ch < 4; ++ch) w[(ch * K + k) * kWarp + lane] = v[ch];
      reinterpret_cast<uint32_t*>(slot(c) + kCoordBytes + kVBytes)[k * kWarp + lane] = bits;
    }
  }
  __device__ __forceinline__ void get_vals(int c, int k, int lane, Real v[4], uint32_t& bits) const {
    if constexpr (M > 1) {
      const Real* w = reinterpret_cast<const Real*>(slot(c) + kCoordBytes);
#pragma unroll
      for (int ch = 0; ch < 4; ++ch) v[ch] = w[(ch * K + k) * kWarp + lane];
      bits = reinterpret_cast<const uint32_t*>(slot(c) + kCoordBytes + kVBytes)[k * kWarp + lane];
    }
  }
  __device__ __forceinline__ void put_t(int c, int k, int lane, Real t) {
    if constexpr (TS) reinterpret_cast<Real*>(slot(c) + kCoordBytes + kVBytes + kBitsBytes)[k * kWarp + lane] = t;
  }
  __device__ __forceinline__ Real get_t(int c, int k, int lane) const {
    if constexpr (TS)
      return reinterpret_cast<const Real*>(slot(c) + kCoordBytes + kVBytes + kBitsBytes)[k * kWarp + lane];
    return Real(0);
  }
};

#ifndef PGB_RENDER_GATHER_INLINE
#define PGB_RENDER_GATHER_INLINE 1
#endif
#if PGB_RENDER_GATHER_INLINE
#define PGB_RENDER_GATHER_ATTR __device__ __forceinline__
#else
#define PGB_RENDER_GATHER_ATTR __device__ __noinline__
#endif

// One sample of a ray: coordinates and value (zero outside the grid).
template <typename Real, typename Store, int MODE, int A, bool BITS>
PGB_RENDER_GATHER_ATTR void render_sample(const RenderArgs<Real>& a, const Ray<Real>& ray, int s,
                                          Real v[4], uint32_t& bits, Real& nx, Real& ny, Real& nz) {
  sample_coords<A>(a, ray, s, nx, ny, nz);
  sample_value<Real, Store, MODE, A, BITS>(a.g, nx, ny, nz, v, bits);
}

// Gathers chunk `c` (K slots) of the ray's samples from `first` to before `end` into
// registers (and its coordinates into the stage when the adjoint follows and the stage
// keeps coordinates).
template <typename Real, typename Store, int MODE, int K, int A, bool ADJ, typename Stage>
__device__ __forceinline__ void gather_chunk(const RenderArgs<Real>& a, const Ray<Real>& ray,
                                             int first, int end, int c, int lane, Real v[K][4],
                                             uint32_t bits[K], Stage& cs) {
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const int s = first + (c * K + k) * kWarp + lane;
    v[k][0] = v[k][1] = v[k][2] = v[k][3] = Real(0);
    bits[k] = 0u;
    if (s < end) {
      Real nx, ny, nz;
      render_sample<Real, Store, MODE, A, ADJ>(a, ray, s, v[k], bits[k], nx, ny, nz);
      if (ADJ) cs.put(c, k, lane, nx, ny, nz);
    }
  }
}

// Exclusive transmittance of every sample of a chunk from the chunk's starting T;
// returns T after the chunk.
#ifndef PGB_SLOT_SKIP
#define PGB_SLOT_SKIP 0  // 1: skip the scans of slots whose 32 samples all have alpha 0
#endif                   //    (exact; a vote per slot costs more than it saves here)
#ifndef PGB_REVERSE_LOOP
#define PGB_REVERSE_LOOP 1  // 1: one copy of the trilinear reverse-pass body in a slot loop
#endif                      // (the gather stays unrolled for its load parallelism):
                            // 0.158 -> 0.147 ms; 2: also for nearest; 0: unrolled
#ifndef PGB_SKIP_ZERO_DV
#define PGB_SKIP_ZERO_DV 1  // skip the scatter of samples whose four partials are all 0
#endif

template <typename Real, int K>
__device__ __forceinline__ Real scan_chunk(const Real v[K][4], Real T, int lane, Real Ts[K]) {
#pragma unroll
  for (int k = 0; k < K; ++k) {
    if (PGB_SLOT_SKIP && !__any_sync(kFull, v[k][3] != Real(0))) {
      Ts[k] = T;  // every factor (1 - alpha) is 1: the exact result of the scan
      continue;
    }
    const Real incl = warp_incl_prod(Real(1) - v[k][3], lane);
    Real excl = __shfl_up_sync(kFull, incl, 1);
    if (lane == 0) excl = Real(1);
    Ts[k] = T * excl;
    T *= __shfl_sync(kFull, incl, kWarp - 1);
  }
  return T;
}

// Error-free sum a + b = s + e (Knuth's TwoSum, six additions, no FMA). An infinite sum
// (an opaque sample: log(1 - 1) = -inf) carries no error term.
__device__ __forceinline__ void two_sum(float a, float b, float& s, float& e) {
  s = __fadd_rn(a, b);
  if (isinf(s)) {
    e = 0.0f;
    return;
  }
  const float bb = __fsub_rn(s, a);
  e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
}

// Compensated log-sum form of scan_chunk: T_s = exp(sum_{j<s} log(1 - alpha_j)), the sum
// carried as an unevaluated pair (L + C) across slots and chunks, each warp-scan step an
// error-free TwoSum whose error joins the compensation term (Kahan-Babuska style). Alpha
// must lie in [0, 1] (clipped cells): log1p(-alpha) is -inf at alpha = 1 and T is then 0.
template <int K>
__device__ __forceinline__ void scan_chunk_log(const float v[K][4], float& L, float& C, int lane,
                                               float Ts[K]) {
#pragma unroll
  for (int k = 0; k < K; ++k) {
    float a = log1pf(-v[k][3]);
    float c = 0.0f;
#pragma unroll
    for (int d = 1; d < kWarp; d <<= 1) {
      const float ya = __shfl_up_sync(kFull, a, d), yc = __shfl_up_sync(kFull, c, d);
      if (lane >= d) {
        float sum, err;
        two_sum(ya, a, sum, err);
        a = sum;
        c = __fadd_rn(__fadd_rn(c, yc), err);
      }
    }
    float ea = __shfl_up_sync(kFull, a, 1), ec = __shfl_up_sync(kFull, c, 1);
    if (lane == 0) ea = ec = 0.0f;
    float sum, err;
    two_sum(L, ea, sum, err);
    Ts[k] = isinf(sum) ? 0.0f : expf(__fadd_rn(sum, __fadd_rn(__fadd_rn(C, ec), err)));
    const float ta = __shfl_sync(kFull, a, kWarp - 1), tc = __shfl_sync(kFull, c, kWarp - 1);
    two_sum(L, ta, sum, err);
    L = sum;
    C = isinf(sum) ? 0.0f : __fadd_rn(__fadd_rn(C, tc), err);
  }
}

// v[i] for a runtime i in [0,4) without indexing a register array dynamically.
template <typename Real>
__device__ __forceinline__ Real pick4(const Real v[4], int i) {
  return i == 0 ? v[0] : (i == 1 ? v[1] : (i == 2 ? v[2] : v[3]));
}

// The render kernel's stage at 32-sample chunks: the values and clamp bits of the last
// PGB_RENDER_STAGE_CHUNKS chunks, without their coordinates (the reverse pass recomputes
// a sample's coordinates from its ray: cheaper than gathering a chunk from the grid
// again). 256^3, 8192 rays x 256 samples: 8 chunks without coordinates (5 KB per warp)
// 0.0928 ms per step; 4 chunks with them (4 KB) 0.1000 ms, without 0.0976 ms; 8 chunks
// with them (8 KB, 192 KB of shared memory per SM, leaving little L1) 0.175 ms.
#ifndef PGB_RENDER_STAGE_CHUNKS
#define PGB_RENDER_STAGE_CHUNKS 8
#endif
#ifndef PGB_RENDER_STAGE_COORDS
#define PGB_RENDER_STAGE_COORDS 0
#endif
// The staged chunks' transmittances as well (0: never, 1: always, 2: for the log-sum
// transmittance only). Recomputing them in the reverse pass is a warp scan; for the
// compensated log-sum it is a costly one. 512^3 log-sum, 65,536 rays x 512: 0.4567 ms
// staged against 0.4865 ms; 256^3 product: 0.0965 against 0.0934 ms.
#ifndef PGB_RENDER_STAGE_TS
#define PGB_RENDER_STAGE_TS 2
#endif
// At 64-sample chunks (nearest lookup), fp32, the last four, the same 5 KB per warp: the cells
// of a nearest step are hardly ever found in L1 again (3 % of sectors), so its space is better
// spent on the stage. 7500 rays x 600 with beta 124 -> 121 us, without 73 -> 70 us, 8192 x 256
// opaque 36 -> 35 us.
template <typename Real, int K, bool LOGT = false>
using RenderStage =
    ChunkStage<Real, K, (K == 1 ? PGB_RENDER_STAGE_CHUNKS : K == 2 && sizeof(Real) == 4 ? 4 : 1),
               (!(K == 2 && sizeof(Real) == 4) && (K != 1 || PGB_RENDER_STAGE_COORDS != 0)),
               (K == 1 && (PGB_RENDER_STAGE_TS == 1 || (PGB_RENDER_STAGE_TS == 2 && LOGT)))>;

// A forward launch has no reverse pass and no stage: its SM's shared memory is all L1 (256^3,
// 100,000 rays x 256 without order, trilinear opaque 166 -> 138 us, half transparent 609 -> 540;
// three 400 x 400 pictures 645 -> 631, half transparent 1631 -> 1506; nearest 84 -> 82).
template <typename Real, int K, int PHASE, bool LOGT>
constexpr int render_smem_bytes(int warps_per_block) {
  return PHASE == kForward ? 0 : RenderStage<Real, K, LOGT>::kBytesPerWarp * warps_per_block;
}

// the smallest block of an fp64 launch (it bounds the number of blocks per ray count)
constexpr int kRenderMinThreads64 = 128;

template <typename Real, int MODE, int K, int PHASE>
constexpr int render_threads() {
  return sizeof(Real) != 4 ? (MODE != PGB_NEAREST && K == 1 ? kRenderMinThreads64 : PGB_RENDER_THREADS)
         : MODE == PGB_NEAREST ? PGB_RENDER_THREADS_NEAREST
         : K != 1 ? PGB_RENDER_THREADS
         : PHASE == kForward ? PGB_RENDER_THREADS_FWD : PGB_RENDER_THREADS_K1;
}

template <typename Real, int MODE, int K, int PHASE>
constexpr int render_min_blocks() {
  if (sizeof(Real) != 4) return MODE == PGB_NEAREST ? 4 : (K == 1 ? 6 : 0);
  return MODE == PGB_NEAREST ? 1024 / PGB_RENDER_THREADS_NEAREST
         : K != 1 ? (K <= 8 ? 2 : 0)
         : PHASE == kForward ? 896 / PGB_RENDER_THREADS_FWD : 768 / PGB_RENDER_THREADS_K1;
}

// LOGT: transmittance as the compensated log-sum (scan_chunk_log, fp32 only) instead of
// the reference's product scan. A: the index arithmetic (Arith).
template <typename Real, typename Store, int MODE, int K, int PHASE, bool LOGT, int A>
__global__ void __launch_bounds__((render_threads<Real, MODE, K, PHASE>()),
                                  (render_min_blocks<Real, MODE, K, PHASE>()))
render_kernel(const RenderArgs<Real> a) {
  static_assert(!LOGT || sizeof(Real) == 4, "log-sum transmittance is an fp32 form");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr bool ADJ = PHASE != kForward;
  const int lane = threadIdx.x & (kWarp - 1);
  const int warps_per_block = blockDim.x >> 5;
  const int64_t gw = (int64_t)blockIdx.x * warps_per_block + (threadIdx.x >> 5);
  const int64_t nw = (int64_t)gridDim.x * warps_per_block;
  RenderStage<Real, K, LOGT> cs(smem_raw, threadIdx.x >> 5);
  // Launches over fp32 grids are one wave of blocks whose warps each take the block's next ray
  // when their last one ends (a counter in shared memory; block b has groups of rays b, b +
  // blocks, ..., so every block's rays come from all over the batch, and neighbouring rays of
  // a large one, a picture's, meet in one L1). With a ray per warp and 4 to 8 rays
  // per block a slot waited for its slowest ray: 13 of 24 resident warps were busy on
  // average. One training launch, before -> now: 256^3 trilinear, 8192 rays x 256, opaque
  // blobs 79 -> 68 us; half transparent, 7500 rays x 600: trilinear 356 -> 333, nearest 131 ->
  // 122 us; nearest, opaque 43 -> 36 us. A counter in global memory was slower (96 us for the
  // first): its answers queue behind the gradient's atomics, and fetched a ray ahead they
  // hand rays to warps that are still busy.
  constexpr bool QUEUE = sizeof(Real) == 4;
  constexpr bool SUMS = QUEUE && PHASE == kTrain;  // loss sums that no order of rays changes
  BinSum loss_bins, beta_bins;  // SUMS
  LossSum<Real> loss_lane;  // otherwise, lane 0: squared errors of the warp's rays
  LossSum<Real> beta_lane;  // per lane: beta terms of its samples (SUMS: of the current ray)
  const bool with_beta = PHASE == kTrain && a.use_beta;
  // Exact early stop. With alpha clamped to [0,1], T is exactly 0 only behind an opaque
  // sample z (alpha_z = 1) or after an underflow, and every later sample then has weight
  // 0 and colour and alpha gradients 0. One term still reads them: z's own alpha gradient
  // T_z (G_z - S_{z+1}), whose suffix S_{z+1} runs over the samples behind z up to the next
  // opaque one. So a ray stops after the chunk in which T reached 0 once z's alpha
  // gradient is masked by the clamp (stored alpha above 1) or a second opaque sample has
  // been gathered; an underflowed T drops terms below T's own magnitude (< 1e-38). The
  // beta term reads every sample's alpha, so it keeps them all.
  const bool stop_at_zero = a.g.clip && !with_beta;
  constexpr uint32_t kAlphaBits = MODE == PGB_NEAREST ? 0x8u : 0x88888888u;
  // beta_w / (R*S) * (1 + 2 eps): the numerator of 1/(alpha+eps) + 1/(1-alpha+eps)
  const Real beta_scale = a.beta_scale;
  const Real grad_scale = a.grad_scale;
  __shared__ double s_part[32];  // per-warp loss partials (training phase)
  __shared__ double s_part_beta[32];
  __shared__ unsigned s_done;    // warps of this block that finished (training phase)
  __shared__ unsigned long long s_bins[2][kWarp];  // SUMS: the block's sums
  __shared__ unsigned s_special[2];
  __shared__ unsigned s_taken;  // QUEUE: rays of this block that have a warp
  __shared__ unsigned s_cleared;  // SUMS: rounds of the clear that have a warp
  const bool clear_early = SUMS && a.clear_early;
  if (QUEUE || PHASE == kTrain) {
    if (threadIdx.x == 0) {
      s_done = 0u;
      s_taken = clear_early ? 0u : (unsigned)warps_per_block;
      s_cleared = 0u;
    }
    if (SUMS && threadIdx.x < 2 * kWarp) s_bins[threadIdx.x >> 5][lane] = 0ull;
    if (SUMS && threadIdx.x < 2) s_special[threadIdx.x] = 0u;
    __syncthreads();
  }
  const auto ray_of = [&](unsigned t) -> int64_t {  // the block's t-th ray
    const unsigned in_group = t & ((1u << a.group_log2) - 1u);
    return (((int64_t)(t >> a.group_log2) * gridDim.x + blockIdx.x) << a.group_log2) + in_group;
  };
  const auto next_ray = [&](int64_t r) -> int64_t {
    if (!QUEUE) return r + nw;
    unsigned taken = 0;
    if (lane == 0) taken = atomicAdd(&s_taken, 1u);
    return ray_of(__shfl_sync(kFull, taken, 0));
  };

  // A round of the clear of the other gradient buffer: 32 mark words from a second counter of the
  // block; false: none is left. On a stream of its own the clear took the SMs that the kernel's
  // blocks were waiting for, and two event waits a step: nearest steps of 3500 rays x 140..320
  // 46 -> 27 and 50 -> 40 us, 512^3 log-sum 378 -> 338 us. Warps take rounds when they have run out
  // of rays, while the block's last ones run; in long launches some also take them before their
  // first ray (clear_early). Of the 8192-ray trilinear step's 95 us (256^3) the clear's 50 MB of
  // zeros are about 15 and the marks 10.
  const auto clear_round = [&]() -> bool {
    const int64_t rounds = (a.clear_words + kWarp - 1) / kWarp;
    unsigned taken = 0;
    if (lane == 0) taken = atomicAdd(&s_cleared, 1u);
    const int64_t round = (int64_t)blockIdx.x + (int64_t)gridDim.x * __shfl_sync(kFull, taken, 0);
    if (round >= rounds) return false;
    clear_marked_warp(a.clear_grad, a.clear_total16, kMarkCellsLog2, a.clear_marks, a.clear_words, round,
                      rounds, lane);
    return true;
  };
  if (clear_early && (threadIdx.x & kWarp) != 0) {  // every other warp: three quarters of it
    const unsigned early = (unsigned)(a.clear_words / (kWarp * (int64_t)gridDim.x) * 3 / 4);
    const auto taken = [&]() -> unsigned {  // the same in every lane
      return __shfl_sync(kFull, lane == 0 ? *(volatile unsigned*)&s_cleared : 0u, 0);
    };
    while (taken() < early && clear_round()) {
    }
  }

  for (int64_t r = !QUEUE ? gw : clear_early ? next_ray(0) : ray_of(threadIdx.x >> 5); r < a.R; r = next_ray(r)) {
    Ray<Real> ray;
    load_ray(a, r, ray, PHASE == kTrain);
    int first, end;
    ray_span(a, ray, first, end);
    if (a.term_thr > 0.0f) {  // a threshold on T is looked at after every chunk, and samples
      // behind it have no beta term: chunks stay where they were
      first = with_beta ? 0 : first - first % (kWarp * K);
      end = with_beta ? a.S : end;
    }
    const int nchunks = (end - first + kWarp * K - 1) / (kWarp * K);
    if (SUMS) beta_lane = LossSum<Real>();
    if (with_beta && lane == 0 && end - first < a.S)  // the samples left out have alpha 0
      beta_lane.add((Real)(a.S - (end - first)) * a.beta_zero);

    Real v[K][4];
    uint32_t bits[K];
    Real Ts[K];
    Real acc[4] = {Real(0), Real(0), Real(0), Real(0)};
    Real T = Real(1);
    Real Tstart = Real(1);  // lane c: transmittance at the start of chunk c
    float LT = 0.0f, LC = 0.0f, LTstart = 0.0f, LCstart = 0.0f;  // LOGT: log T = LT + LC
    int last = -1;          // last composited chunk (-1: none, e.g. zero samples)
    int n_opaque = 0;       // opaque samples gathered so far (warp-uniform)
    bool first_needs = false;  // the first opaque sample's alpha gradient passes the clamp
    for (int c = 0; c < nchunks; ++c) {
      if (lane == c) {
        Tstart = T;
        LTstart = LT;
        LCstart = LC;
      }
      __syncwarp();
      gather_chunk<Real, Store, MODE, K, A, ADJ>(a, ray, first, end, c, lane, v, bits, cs);
      if (ADJ) {
#pragma unroll
        for (int k = 0; k < K; ++k) cs.put_vals(c, k, lane, v[k], bits[k]);
      }
      if constexpr (LOGT) {
        scan_chunk_log<K>(v, LT, LC, lane, Ts);
        T = isinf(LT) ? Real(0) : (Real)expf(LT + LC);
      } else {
        T = scan_chunk<Real, K>(v, T, lane, Ts);
      }
      if (ADJ) {
#pragma unroll
        for (int k = 0; k < K; ++k) cs.put_t(c, k, lane, Ts[k]);
      }
#pragma unroll
      for (int k = 0; k < K; ++k) {
        const Real w = v[k][3] * Ts[k];
        acc[0] += w * v[k][0];
        acc[1] += w * v[k][1];
        acc[2] += w * v[k][2];
        acc[3] += w;
      }
      if (with_beta) {  // per-chunk partial in Real, one fp64 add per chunk
        Real bsum = Real(0);
#pragma unroll
        for (int k = 0; k < K; ++k) {
          if (first + (c * K + k) * kWarp + lane < end) {
            const Real al = v[k][3], e = (Real)a.beta_eps;
            bsum += log(al + e) - log(Real(1) - al + e);
          }
        }
        beta_lane.add(bsum);
      }
      last = c;
      if (PHASE == kForward) {  // no gradient needs the samples behind T = 0
        if (stop_at_zero && T == Real(0)) break;
      } else if (stop_at_zero) {
#pragma unroll
        for (int k = 0; k < K; ++k) {
          const unsigned opq = __ballot_sync(kFull, Real(1) - v[k][3] == Real(0));
          if (opq != 0u) {
            const unsigned need =
                __ballot_sync(kFull, (bits[k] & kAlphaBits) != 0u && Ts[k] > Real(0));
            if (n_opaque == 0) first_needs = ((need >> (__ffs(opq) - 1)) & 1u) != 0u;
            n_opaque += __popc(opq);
          }
        }
        if (T == Real(0) && (!first_needs || n_opaque >= 2)) break;
      }
      if (a.term_thr > 0.0f && T < (Real)a.term_thr) break;
    }
    Real px[4];
#pragma unroll
    for (int ch = 0; ch < 4; ++ch) px[ch] = warp_sum(acc[ch]);
    if (a.use_bg) {
#pragma unroll
      for (int ch = 0; ch < 3; ++ch) px[ch] += (Real(1) - px[3]) * (Real)a.bg[ch];
    }

    if (PHASE == kForward) {
      if (lane < 4) a.rgba_out[4 * r + lane] = pick4(px, lane);
      continue;
    }

    Real gpx[4];
    if (PHASE == kBackward) {
#pragma unroll
      for (int ch = 0; ch < 4; ++ch) gpx[ch] = a.d_rgba[4 * r + ch];
    } else {
      // the ray's squared error in Real (4 terms), accumulated over rays in double
      Real sq = Real(0);
#pragma unroll
      for (int ch = 0; ch < 4; ++ch) {
        const Real diff = px[ch] - __shfl_sync(kFull, ray.tgt, ch);
        sq += diff * diff;
        gpx[ch] = grad_scale * diff;
      }
      if constexpr (SUMS) {
        loss_bins.add(sq, lane);
        if (with_beta) {
          const LossSum<Real> ray_beta = warp_sum(beta_lane);
          beta_bins.add(__shfl_sync(kFull, ray_beta.hi, 0), lane);
          beta_bins.add(__shfl_sync(kFull, ray_beta.lo, 0), lane);
        }
      } else {
        if (lane == 0) loss_lane.add(sq);
      }
      if (a.rgba_out != nullptr && lane < 4) a.rgba_out[4 * r + lane] = pick4(px, lane);
    }
    if (a.use_bg)  // d(rgb + (1 - A) bg)/dA = -bg
      gpx[3] -= gpx[0] * (Real)a.bg[0] + gpx[1] * (Real)a.bg[1] + gpx[2] * (Real)a.bg[2];

    // reverse pass over the chunks that were composited
    Real Snext_carry = Real(0);  // S at the first sample after the current slot
    for (int c = last; c >= 0; --c) {
      if (c != last) {
        __syncwarp();
        const bool staged = RenderStage<Real, K, LOGT>::holds(c, last);
        if (staged) {  // the chunk's values are still staged
#pragma unroll
          for (int k = 0; k < K; ++k) cs.get_vals(c, k, lane, v[k], bits[k]);
        } else {
          gather_chunk<Real, Store, MODE, K, A, true>(a, ray, first, end, c, lane, v, bits, cs);
        }
        if (RenderStage<Real, K, LOGT>::kHasTs && staged) {  // the forward pass's transmittances
#pragma unroll
          for (int k = 0; k < K; ++k) Ts[k] = cs.get_t(c, k, lane);
        } else if constexpr (LOGT) {
          float l = __shfl_sync(kFull, LTstart, c), lc = __shfl_sync(kFull, LCstart, c);
          scan_chunk_log<K>(v, l, lc, lane, Ts);
        } else {
          scan_chunk<Real, K>(v, __shfl_sync(kFull, Tstart, c), lane, Ts);
        }
      }
      __syncwarp();
      // trilinear: a loop (the 8-corner scatter body is large); nearest: unrolled
      constexpr int kRevUnroll =
          (PGB_REVERSE_LOOP == 2 || (PGB_REVERSE_LOOP == 1 && MODE == PGB_TRILINEAR)) ? 1 : K;
#pragma unroll kRevUnroll
      for (int k = K - 1; k >= 0; --k) {
        Real vk[4], tk;
        uint32_t bk;
#pragma unroll
        for (int kk = 0; kk < K; ++kk) {
          if (kk == k) {
            vk[0] = v[kk][0]; vk[1] = v[kk][1]; vk[2] = v[kk][2]; vk[3] = v[kk][3];
            bk = bits[kk];
            tk = Ts[kk];
          }
        }
        // a slot with alpha 0 and nothing to scatter leaves S unchanged (identity maps)
        if (PGB_SLOT_SKIP && !__any_sync(kFull, bk != 0u || vk[3] != Real(0))) continue;
        const Real al = vk[3];
        const Real G = gpx[0] * vk[0] + gpx[1] * vk[1] + gpx[2] * vk[2] + gpx[3];
        Real fa = G * al, fb = Real(1) - al;
        if constexpr (MODE == PGB_NEAREST && K == 2 && sizeof(Real) == 4) {
          // The first step's a + b * a2 with a = G * al has two fused forms, an ulp apart. Rays
          // of more than 128 samples without early stop take the form that the code for 256-sample
          // chunks has: a training run with the beta term, whose 1 / (1 - alpha + eps) turns an
          // ulp of an opacity near 1 into 6e-4 of the next step's gradient, keeps its bits
          // whether its chunks are picked, asked for at the same size, or of 256 samples.
          const Real a2 = __shfl_down_sync(kFull, fa, 1), b2 = __shfl_down_sync(kFull, fb, 1);
          const Real near = rfma(fb, a2, fa), far = rfma(G, al, rmul(fb, a2));
          if (lane < kWarp - 1) {
            fa = a.long_ray ? far : near;
            fb = fb * b2;
          }
          warp_suffix_affine(fa, fb, lane, 2);
        } else {
          warp_suffix_affine(fa, fb, lane);
        }
        const Real S_here = fa + fb * Snext_carry;          // S_s for this lane's sample
        Real S_after = __shfl_down_sync(kFull, S_here, 1);  // S_{s+1}
        if (lane == kWarp - 1) S_after = Snext_carry;
        Snext_carry = __shfl_sync(kFull, S_here, 0);
        if (bk != 0u) {
          const Real w = al * tk;
          Real dv[4];
          dv[0] = gpx[0] * w;
          dv[1] = gpx[1] * w;
          dv[2] = gpx[2] * w;
          dv[3] = tk * (G - S_after);
          if (with_beta) {  // d/dalpha of log(alpha + e) - log(1 - alpha + e), one division
            const Real e = (Real)a.beta_eps;
            dv[3] += beta_scale / ((al + e) * (Real(1) - al + e));
          }
          // behind an opaque sample (T = 0) every partial is 0 and no corner would be written
          if (PGB_SKIP_ZERO_DV &&
              !(dv[0] != Real(0) || dv[1] != Real(0) || dv[2] != Real(0) || dv[3] != Real(0)))
            continue;
          Real nx, ny, nz;
          if constexpr (RenderStage<Real, K, LOGT>::kHasCoords)
            cs.get(c, k, lane, nx, ny, nz);
          else
            sample_coords<A>(a, ray, first + (c * K + k) * kWarp + lane, nx, ny, nz);
          sample_scatter<Real, MODE, A>(a.g, a.grad, nx, ny, nz, dv, bk, a.grad_marks);
        }
      }
    }
  }

  if constexpr (SUMS) {
    if (a.clear_words > 0)
      while (clear_round()) {
      }
    // Warps add their bins up in shared memory and the block's last warp adds them to the
    // launch's, so that a block fences once, at its end (a fence at device scope also empties
    // the SM's L1: one per warp took the nearest step of 8192 rays from 44 to 66 us). The last
    // block takes the sums and leaves the state zero for the next launch.
    TrainState* st = a.state;
    if (loss_bins.bin != 0) atomicAdd(&s_bins[0][lane], (unsigned long long)loss_bins.bin);
    if (beta_bins.bin != 0) atomicAdd(&s_bins[1][lane], (unsigned long long)beta_bins.bin);
    if (lane == 0) {
      if (loss_bins.special) atomicOr(&s_special[0], loss_bins.special);
      if (beta_bins.special) atomicOr(&s_special[1], beta_bins.special);
    }
    __threadfence_block();
    __syncwarp();
    unsigned last = 0;
    if (lane == 0) last = atomicAdd(&s_done, 1u) == (unsigned)warps_per_block - 1u;
    if (!__shfl_sync(kFull, last, 0)) return;
    __threadfence_block();
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const unsigned long long bin = *(volatile unsigned long long*)&s_bins[i][lane];
      const unsigned special = *(volatile unsigned*)&s_special[i];
      if (bin != 0ull) atomicAdd(&st->bins[i][lane], bin);
      if (lane == 0 && special != 0u) atomicOr(&st->special[i], special);
    }
    __threadfence();
    __syncwarp();
    if (lane == 0) last = atomicAdd(&st->blocks_done, 1u) == gridDim.x - 1u;
    if (!__shfl_sync(kFull, last, 0)) return;
    __threadfence();
    BinSum sums[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      sums[i].bin = (long long)__ldcg(&st->bins[i][lane]);
      sums[i].special = __ldcg(&st->special[i]);
    }
    const double mse = sums[0].value(lane), beta = with_beta ? sums[1].value(lane) : 0.0;
    st->bins[0][lane] = 0ull;
    st->bins[1][lane] = 0ull;
    if (lane == 0) {
      a.loss_out[0] = (Real)(a.loss_w * mse * a.inv_count);
      if (with_beta) a.loss_out[1] = (Real)(a.beta_w * beta * a.inv_samples);
      st->blocks_done = 0u;
      st->special[0] = st->special[1] = 0u;
    }
  } else if (PHASE == kTrain) {
    // deterministic loss without a barrier: warps count themselves out in shared memory,
    // the block's last warp sums the block in warp order and takes one global ticket, and
    // the last block sums the blocks in block order
    const int wib = threadIdx.x >> 5;
    unsigned last_warp = 0;
    if (with_beta) beta_lane = warp_sum(beta_lane);
    if (lane == 0) {
      loss_lane.store_volatile(&s_part[wib]);
      beta_lane.store_volatile(&s_part_beta[wib]);
      __threadfence_block();
      last_warp = atomicAdd(&s_done, 1u) == (unsigned)warps_per_block - 1u;
    }
    last_warp = __shfl_sync(kFull, last_warp, 0);
    if (last_warp) {
      unsigned last_block = 0;
      if (lane == 0) {
        __threadfence_block();
        LossSum<Real> sum, bsum;
        for (int i = 0; i < warps_per_block; ++i) {
          sum.add(LossSum<Real>::load_volatile(&s_part[i]));
          bsum.add(LossSum<Real>::load_volatile(&s_part_beta[i]));
        }
        sum.store(a.partials + blockIdx.x);
        if (with_beta) bsum.store(a.partials_beta + blockIdx.x);
        __threadfence();
        last_block = atomicAdd(a.counter, 1u) == gridDim.x - 1u;
      }
      last_block = __shfl_sync(kFull, last_block, 0);
      if (last_block) {
        __threadfence();
        // block partials in block order, eight loads in flight per lane (L2 reads: the
        // partials were written by other blocks before their ticket)
        LossSum<Real> sum, bsum;
        for (unsigned i0 = lane; i0 < gridDim.x; i0 += 8 * kWarp) {
          LossSum<Real> p[8];
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            const unsigned i = i0 + u * kWarp;
            if (i < gridDim.x) p[u] = LossSum<Real>::load_cg(a.partials + i);
          }
#pragma unroll
          for (int u = 0; u < 8; ++u) sum.add(p[u]);
          if (with_beta) {
#pragma unroll
            for (int u = 0; u < 8; ++u) {
              const unsigned i = i0 + u * kWarp;
              if (i < gridDim.x) p[u] = LossSum<Real>::load_cg(a.partials_beta + i);
            }
#pragma unroll
            for (int u = 0; u < 8; ++u) bsum.add(p[u]);
          }
        }
        sum = warp_sum(sum);
        if (with_beta) bsum = warp_sum(bsum);
        if (lane == 0) {
          a.loss_out[0] = (Real)(a.loss_w * sum.value() * a.inv_count);
          if (with_beta) a.loss_out[1] = (Real)(a.beta_w * bsum.value() * a.inv_samples);
          *a.counter = 0u;
        }
      }
    }
  }
}

}  // namespace pgb
