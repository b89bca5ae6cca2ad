// FP64 3D type-2 / type-1 NUFFT with the exponential-of-semicircle kernel:
// the reference's own tolerance (eps = 1e-12 in double,
// spinifel/extern/nufft_ext.py:62, finufft_ext.py:70-94), which an FP32 grid
// cannot reach (its floor is about 1e-7).  Kernel widths 2..16.
//
// Same layout and conventions as the FP32 plan of nufft.cu, in double:
//   fine   : n1*n2*n3, the upsampled grid, and half, its half spectrum (D2Z);
//   re_pad : Re of the type-2 fine grid with a periodic halo of
//            p = ceil(w/2)+1 cells per side (no modulo in the inner loops);
//   im_pad : Im (only when requested);
//   acc_pad: padded accumulator of type-1 spreading, folded before the FFT.
// Points (radians) map to fine-grid coordinate t = x n / (2 pi), wrapped into
// [-n/2, n/2); the footprint is l0 .. l0+w-1 with l0 = ceil(t - w/2).
//
// GB300 runs FP64 at about 1/64 of its FP32 rate, so the FP64 kernels are
// bound by the FP64 pipe (W^3 FMAs per point); the grid (tens of MB) stays
// in L2 and is read through L1 without shared-memory staging.  Slices of panel
// detectors run over pairs of floats instead (k_slice_pairs).
#include <cufft.h>
#include <math.h>

#include <vector>

#include "common.cuh"
#include "es_params.cuh"
#include "fine_grid.cuh"

struct spf_nufft64_plan_s {
  int dev = 0;
  int m[3] = {0, 0, 0};
  int n[3] = {0, 0, 0};
  int np[3] = {0, 0, 0};
  int pad = 0;
  int w = 0;
  double beta = 0, sigma = 2.0, eps = 1e-12;
  double *inv_p[3] = {nullptr, nullptr, nullptr};
  double *fine = nullptr;       // n1*n2*n3
  double2 *half = nullptr;      // n1*n2*(n3/2+1)
  double *re_pad = nullptr;
  double *im_pad = nullptr;
  double *acc_pad = nullptr;
  // slicing by pairs of floats (NULL: in FP64): the padded grid over a power of
  // two as (high, low) pairs, that power, exp at the table's points
  float2 *pair_pad = nullptr;
  unsigned long long *peak = nullptr;  // bits of max |re_pad|
  float2 *exp_table = nullptr;
  cufftHandle fft = 0;
  bool fft_ok = false;
};

namespace spf {
namespace f64 {

struct Geom {
  int n1, n2, n3;
  int p1, p2, p3;
  int off1, off2, off3;
  double beta;
  double inv_half_w;
};

static Geom geom_of(const spf_nufft64_plan_s *P) {
  Geom g;
  g.n1 = P->n[0]; g.n2 = P->n[1]; g.n3 = P->n[2];
  g.p1 = P->np[0]; g.p2 = P->np[1]; g.p3 = P->np[2];
  g.off1 = P->n[0] / 2 + P->pad;
  g.off2 = P->n[1] / 2 + P->pad;
  g.off3 = P->n[2] / 2 + P->pad;
  g.beta = P->beta;
  g.inv_half_w = 2.0 / P->w;
  return g;
}

// Padded first index and the W kernel values along one axis for a point at
// x (radians) with grid scale s = n / (2 pi) (times the caller's coordinate
// scale); t is wrapped into [-n/2, n/2).
template <int W>
__device__ __forceinline__ int axis_setup(double x, double s, int n, int off, double beta,
                                          double inv_half_w, double *wt) {
  const double fn = (double)n;
  double t = __dmul_rn(x, s);
  t = __dsub_rn(t, __dmul_rn(fn, floor(__dadd_rn(__ddiv_rn(t, fn), 0.5))));
  const double l0 = ceil(__dsub_rn(t, 0.5 * W));
#pragma unroll
  for (int a = 0; a < W; ++a) {
    const double z = (l0 + (double)a - t) * inv_half_w;
    const double q = fmax(fma(-z, z, 1.0), 0.0);
    wt[a] = exp(beta * (sqrt(q) - 1.0));
  }
  return (int)l0 + off;
}

template <int W>
__device__ __forceinline__ double interp_point(const double *__restrict__ grid, const Geom &g,
                                               double x1, double s1, double x2, double s2,
                                               double x3, double s3) {
  double w1[W], w2[W], w3[W];
  const int i0 = axis_setup<W>(x1, s1, g.n1, g.off1, g.beta, g.inv_half_w, w1);
  const int j0 = axis_setup<W>(x2, s2, g.n2, g.off2, g.beta, g.inv_half_w, w2);
  const int k0 = axis_setup<W>(x3, s3, g.n3, g.off3, g.beta, g.inv_half_w, w3);
  double acc = 0.0;
#pragma unroll 1
  for (int a = 0; a < W; ++a) {
    double acc_a = 0.0;
    const double *plane = grid + ((size_t)(i0 + a) * g.p2 + j0) * g.p3 + k0;
#pragma unroll
    for (int b = 0; b < W; ++b) {
      const double *row = plane + (size_t)b * g.p3;
      double r = 0.0;
#pragma unroll
      for (int c = 0; c < W; ++c) r = fma(w3[c], __ldg(row + c), r);
      acc_a = fma(w2[b], r, acc_a);
    }
    acc = fma(w1[a], acc_a, acc);
  }
  return acc;
}

// Rotation of pixel position q by the inverse (transpose) of R(quat)
// (quat = [w,x,y,z]; spinifel/extern/nufft_ext.py:59-60 inverts the
// skopi quaternion2rot3d matrix), in double.
__device__ __forceinline__ void rotate_inv(const double *__restrict__ quat, double qx, double qy,
                                           double qz, double &h, double &k, double &l) {
  const double q0 = quat[0], q1 = quat[1], q2 = quat[2], q3 = quat[3];
  const double r00 = 1.0 - 2.0 * (q2 * q2 + q3 * q3), r01 = 2.0 * (q1 * q2 - q0 * q3),
               r02 = 2.0 * (q1 * q3 + q0 * q2);
  const double r10 = 2.0 * (q1 * q2 + q0 * q3), r11 = 1.0 - 2.0 * (q1 * q1 + q3 * q3),
               r12 = 2.0 * (q2 * q3 - q0 * q1);
  const double r20 = 2.0 * (q1 * q3 - q0 * q2), r21 = 2.0 * (q2 * q3 + q0 * q1),
               r22 = 1.0 - 2.0 * (q1 * q1 + q2 * q2);
  h = r00 * qx + r10 * qy + r20 * qz;
  k = r01 * qx + r11 * qy + r21 * qz;
  l = r02 * qx + r12 * qy + r22 * qz;
}

template <int W>
__global__ void __launch_bounds__(128)
    k_interp(const double *__restrict__ re_pad, const double *__restrict__ im_pad, Geom g,
             const double *__restrict__ x, const double *__restrict__ y,
             const double *__restrict__ z, int64_t npts, double *__restrict__ out_re,
             double *__restrict__ out_im) {
  const double sc1 = g.n1 * (0.5 / M_PI), sc2 = g.n2 * (0.5 / M_PI), sc3 = g.n3 * (0.5 / M_PI);
  for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < npts;
       j += (int64_t)gridDim.x * blockDim.x) {
    out_re[j] = interp_point<W>(re_pad, g, x[j], sc1, y[j], sc2, z[j], sc3);
    if (out_im) out_im[j] = interp_point<W>(im_pad, g, x[j], sc1, y[j], sc2, z[j], sc3);
  }
}

// 2^-(e + 1) for max |v| in [2^e, 2^(e + 1)), and whether pairs of floats can
// hold the grid (finite and not all below the normal doubles)
__device__ __forceinline__ bool pair_scale(unsigned long long peak, double &down, double &up) {
  const int e = (int)(peak >> 52);  // biased exponent
  if (e >= 2046 || e < 1) return false;
  down = __longlong_as_double((long long)(2045 - e) << 52);  // 2^(1022 - e)
  up = __longlong_as_double((long long)(e + 1) << 52);       // 2^(e - 1022)
  return e <= 2044;
}

// Slicing: point (o, p) = scale * R(q_o)^-1 ppr[:, p]; out[o * n_pix + p] = Re c.
template <int W>
__global__ void __launch_bounds__(128)
    k_slice(const double *__restrict__ re_pad, Geom g, const double *__restrict__ quats,
            const double *__restrict__ ppr, int64_t n_pix, double s1, double s2, double s3,
            double *__restrict__ out, const unsigned long long *__restrict__ peak) {
  double down, up;
  if (peak && pair_scale(*peak, down, up)) return;  // k_slice_pairs has it
  const int64_t o = blockIdx.x;
  const int64_t p = blockIdx.y * (int64_t)blockDim.x + threadIdx.x;
  if (p >= n_pix) return;
  double h, k, l;
  rotate_inv(quats + 4 * o, ppr[p], ppr[n_pix + p], ppr[2 * n_pix + p], h, k, l);
  out[o * n_pix + p] = interp_point<W>(re_pad, g, h, s1, k, s2, l, s3);
}

// ---------------------------------------------------------------------------
// Slicing with pairs of floats
//
// A warp's FP64 instruction holds its quarter of the SM for 64 clocks, so the
// W^3 FMAs and 3 W kernel values of a point (39 exponentials and roots at
// eps 1e-12, about as dear as 1,500 FMAs) take 2.66 ms for 409,600 points.
// The same sums over unevaluated pairs of floats (error-free products and
// sums: Dekker 1971, Knuth TAOCP 2, 4.2.2) take twelve FP32 instructions a
// term and are good to about 2^-46 of the terms' magnitudes: a pixel is at most
// 3.2e-14 of the largest value off the FP64 kernel's, where the interpolation of
// a kernel of W <= 13 is off by 5e-13 and more (against the direct sums, FP64 and
// pairs: 8.3778e-13 and 8.3786e-13 at 21^3, 2.3936e-12 and 2.3927e-12 at 41^3);
// wider kernels resolve less than that and stay in FP64.  409,600 points at 41^3
// take 0.85 ms (2.69 in FP64 throughout), 262,144 at 81^3 on 4 x 128 x 128
// pixels 0.54 (1.72).
//
// A CTA takes a 4 x 8 pixel patch of one panel at one orientation: three
// warps compute its grid coordinates in FP64 (one axis each), all eight the
// kernel values, then the box of the footprints is staged in shared memory
// and each warp sums every eighth of the W^2 footprint rows for the 32 pixels.
// The grid is scaled by a power of two to at most 1, so that the low halves
// stay in FP32's range.
// ---------------------------------------------------------------------------
constexpr int PAIR_MAX_W = 13;
constexpr int PAIR_PX = 4, PAIR_PY = 8, PAIR_PIX = 32, PAIR_WARPS = 8;
constexpr int PAIR_CELLS = 10240;    // 80 KB: two CTAs an SM
constexpr int EXP_PER_UNIT = 128;    // exp(-j / 128) in the table

struct Pair {
  float h, l;
};
__device__ __forceinline__ Pair two_sum(float a, float b) {
  const float s = __fadd_rn(a, b), t = __fsub_rn(s, a);
  return Pair{s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, t)), __fsub_rn(b, t))};
}
__device__ __forceinline__ Pair fast_two_sum(float a, float b) {  // |a| >= |b|
  const float s = __fadd_rn(a, b);
  return Pair{s, __fsub_rn(b, __fsub_rn(s, a))};
}
__device__ __forceinline__ Pair mul(Pair a, Pair b) {
  const float p = __fmul_rn(a.h, b.h);
  float e = __fmaf_rn(a.h, b.h, -p);
  e = __fmaf_rn(a.h, b.l, e);
  e = __fmaf_rn(a.l, b.h, e);
  return fast_two_sum(p, e);
}
__device__ __forceinline__ Pair add(Pair a, float b) {
  const Pair s = two_sum(a.h, b);
  return fast_two_sum(s.h, __fadd_rn(s.l, a.l));
}

// sum of products: h + l; the terms' errors collect in l (a term's own first:
// the large sum is rounded once a term)
__device__ __forceinline__ void accumulate(Pair &acc, float wh, float wl, float gh, float gl) {
  const float p = __fmul_rn(wh, gh);
  const float e = __fmaf_rn(wl, gh, __fmaf_rn(wh, gl, __fmaf_rn(wh, gh, -p)));
  const Pair s = two_sum(acc.h, p);
  acc.h = s.h;
  acc.l = __fadd_rn(acc.l, __fadd_rn(s.l, e));
}

// The kernel's constants: with u the distance in cells, z^2 = per_z2 u^2 and
// beta z^2 = -expo u^2.
struct PairKernel {
  Pair per_z2, expo;
};

// exp(beta (sqrt(1 - z^2) - 1)) at u = f + a, good to about 2^-46 (sums of the
// W values to 1e-14; the same operations replayed on the host, 4e5
// fractions, W = 7, 10, 13).  The exponent is taken as
// x = -beta z^2 / (1 + sqrt(1 - z^2)), which keeps its relative error where
// sqrt - 1 cancels, and exp(x) = T[j] exp(t), x = -j / 128 + t, with the Taylor
// polynomial of exp(t) - 1: for |t| <= 1/256 its cube is small enough to be
// rounded to FP32 (with 32 entries a unit that rounding alone was 2^-42.2).
__device__ __forceinline__ Pair es_pair(Pair f, int a, const PairKernel &k,
                                        const float2 *__restrict__ table, int table_last) {
  const Pair u1 = add(f, (float)a);
  const Pair u2 = mul(u1, u1);
  const Pair z2 = mul(u2, k.per_z2), num = mul(u2, k.expo);
  Pair q = two_sum(1.0f, -z2.h);
  q = fast_two_sum(q.h, __fsub_rn(q.l, z2.l));
  if (!(q.h > 0.0f)) q = Pair{0.0f, 0.0f};
  const float root = __fsqrt_rn(q.h);
  const float rest = __fadd_rn(__fmaf_rn(-root, root, q.h), q.l);
  Pair d = two_sum(1.0f, root);  // 1 + the root
  d = fast_two_sum(d.h, __fadd_rn(d.l, root > 0.0f ? __fdividef(0.5f * rest, root) : 0.0f));
  const float inv = __fdividef(1.0f, d.h);
  const float y = __fmul_rn(num.h, inv);
  const float left = __fadd_rn(__fmaf_rn(-y, d.h, num.h), __fmaf_rn(-y, d.l, num.l));
  const Pair x = fast_two_sum(y, __fmul_rn(left, inv));  // -beta .. 0
  const int j = min(max(__float2int_rn(-EXP_PER_UNIT * x.h), 0), table_last);
  const float2 T = __ldg(table + j);
  const Pair t = fast_two_sum(__fadd_rn(x.h, (float)j * (1.0f / EXP_PER_UNIT)), x.l);
  const float p = __fmul_rn(t.h, t.h);
  const float pe = __fmaf_rn(2.0f * t.h, t.l, __fmaf_rn(t.h, t.h, -p));
  const float cube = p * t.h * fmaf(t.h, fmaf(t.h, 1.0f / 120.0f, 1.0f / 24.0f), 1.0f / 6.0f);
  Pair u = two_sum(t.h, 0.5f * p);
  u = fast_two_sum(u.h, __fadd_rn(__fadd_rn(u.l, t.l), __fmaf_rn(0.5f, pe, cube)));
  const Pair Tu = mul(Pair{T.x, T.y}, u);
  const Pair w = two_sum(T.x, Tu.h);
  return fast_two_sum(w.h, __fadd_rn(w.l, __fadd_rn(T.y, Tu.l)));
}

__global__ void k_to_pairs(const double *__restrict__ v, int64_t n,
                           const unsigned long long *__restrict__ peak,
                           float2 *__restrict__ out) {
  double down, up;
  if (!pair_scale(*peak, down, up)) return;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const double x = v[i] * down;
    const float h = (float)x;
    out[i] = make_float2(h, (float)(x - (double)h));
  }
}

template <int W>
__global__ void __launch_bounds__(PAIR_WARPS * 32, 2)
    k_slice_pairs(const float2 *__restrict__ grid, const unsigned long long *__restrict__ peak,
                  Geom g, const double *__restrict__ quats, const double *__restrict__ ppr,
                  int n_panels, int nx, int ny, double s1, double s2, double s3, PairKernel kernel,
                  const float2 *__restrict__ exp_table, int table_last,
                  double *__restrict__ out) {
  extern __shared__ __align__(16) float2 box[];  // PAIR_CELLS
  __shared__ float2 wts[3 * W][PAIR_PIX];
  __shared__ double part[PAIR_WARPS][PAIR_PIX];
  __shared__ float2 frac[3][PAIR_PIX];
  __shared__ int first[3][PAIR_PIX], lo[3], hi[3];
  double down, up;
  if (!pair_scale(*peak, down, up)) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t o = blockIdx.x;
  const int patches_y = (ny + PAIR_PY - 1) / PAIR_PY, patches_x = (nx + PAIR_PX - 1) / PAIR_PX;
  const int panel = blockIdx.y / (patches_x * patches_y), rem = blockIdx.y % (patches_x * patches_y);
  // pixels past the panel's edge repeat its last row or column
  const int px = (rem / patches_y) * PAIR_PX + lane / PAIR_PY,
            py = (rem % patches_y) * PAIR_PY + lane % PAIR_PY;
  const bool valid = px < nx && py < ny;
  const int64_t n_pix = (int64_t)n_panels * nx * ny;
  const int64_t p = ((int64_t)panel * nx + min(px, nx - 1)) * ny + min(py, ny - 1);
  if (warp < 3) {
    double h, k, l;
    rotate_inv(quats + 4 * o, ppr[p], ppr[n_pix + p], ppr[2 * n_pix + p], h, k, l);
    const int n = warp == 0 ? g.n1 : warp == 1 ? g.n2 : g.n3;
    const int off = warp == 0 ? g.off1 : warp == 1 ? g.off2 : g.off3;
    const double x = warp == 0 ? h : warp == 1 ? k : l, s = warp == 0 ? s1 : warp == 1 ? s2 : s3;
    // the cell of axis_setup, operation by operation
    const double fn = (double)n;
    double t = __dmul_rn(x, s);
    t = __dsub_rn(t, __dmul_rn(fn, floor(__dadd_rn(__ddiv_rn(t, fn), 0.5))));
    const double l0 = ceil(__dsub_rn(t, 0.5 * W));
    const double f = __dsub_rn(l0, t);
    const float fh = (float)f;
    frac[warp][lane] = make_float2(fh, (float)(f - (double)fh));
    const int i0 = (int)l0 + off;
    first[warp][lane] = i0;
    const int a = __reduce_min_sync(0xffffffffu, i0), b = __reduce_max_sync(0xffffffffu, i0);
    if (lane == 0) {
      lo[warp] = a;
      hi[warp] = b + W;
    }
  }
  __syncthreads();
  // the box from an even cell on: rows of the padded grid (even length) and of
  // the box start on 16 bytes, and half a warp copies a row, 16 bytes a lane
  const int i0 = lo[0], j0 = lo[1], k0 = lo[2] & ~1;
  const int di = hi[0] - i0, dj = hi[1] - j0, dk = (hi[2] - k0 + 1) & ~1;
  const int sk = dk | 2, sj = dj | 1;  // strides that spread rows over the banks
  const bool staged = (int64_t)di * sj * sk <= PAIR_CELLS;
  if (staged) {
    constexpr int STEP = 2 * PAIR_WARPS;  // rows at a time
    int jj = 2 * warp + (lane >> 4), ii = 0;
    while (jj >= dj) {
      jj -= dj;
      ++ii;
    }
    const int c0 = 2 * (lane & 15);
    const float2 *src = grid + ((size_t)i0 * g.p2 + j0) * g.p3 + k0 + c0;
    const unsigned dst = (unsigned)__cvta_generic_to_shared(box + c0);
    while (ii < di) {
      const float2 *row = src + (ii * g.p2 + jj) * g.p3;
      const unsigned to = dst + (unsigned)((ii * sj + jj) * sk) * (unsigned)sizeof(float2);
      for (int c = c0; c < dk; c += 32)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                         to + (unsigned)((c - c0) * sizeof(float2))),
                     "l"(row + (c - c0))
                     : "memory");
      jj += STEP;
      while (jj >= dj) {
        jj -= dj;
        ++ii;
      }
    }
  }
  // the kernel values while the box is on its way (plain loads, a
  // warp a row, took most of the kernel: 1,297 us in all)
  for (int e = warp; e < 3 * W; e += PAIR_WARPS) {
    const float2 f = frac[e / W][lane];
    const Pair w = es_pair(Pair{f.x, f.y}, e % W, kernel, exp_table, table_last);
    wts[e][lane] = make_float2(w.h, w.l);
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  float2 w3[W];
#pragma unroll
  for (int c = 0; c < W; ++c) w3[c] = wts[2 * W + c][lane];
  const int li = first[0][lane], lj = first[1][lane], lk = first[2][lane];
  Pair sum{0.0f, 0.0f};
  auto rows = [&](auto cell) {
    for (int r = warp; r < W * W; r += PAIR_WARPS) {
      const int a = r / W, b = r - a * W;
      const auto row = cell(a, b);
      Pair acc{0.0f, 0.0f};
#pragma unroll
      for (int c = 0; c < W; ++c) {
        const float2 v = row(c);
        accumulate(acc, w3[c].x, w3[c].y, v.x, v.y);
      }
      const float2 u = wts[a][lane], v = wts[W + b][lane];
      const Pair w12 = mul(Pair{u.x, u.y}, Pair{v.x, v.y});
      const Pair n = fast_two_sum(acc.h, acc.l);
      accumulate(sum, w12.h, w12.l, n.h, n.l);
    }
  };
  if (staged) {
    const float2 *base = box + ((li - i0) * sj + (lj - j0)) * sk + (lk - k0);
    rows([&](int a, int b) {
      const float2 *row = base + (a * sj + b) * sk;
      return [row](int c) { return row[c]; };
    });
  } else {
    const float2 *base = grid + ((size_t)li * g.p2 + lj) * g.p3 + lk;
    rows([&](int a, int b) {
      const float2 *row = base + ((size_t)a * g.p2 + b) * g.p3;
      return [row](int c) { return __ldg(row + c); };
    });
  }
  part[warp][lane] = (double)sum.h + (double)sum.l;
  __syncthreads();
  if (warp != 0 || !valid) return;
  double v = part[0][lane];
  for (int q = 1; q < PAIR_WARPS; ++q) v += part[q][lane];
  out[o * n_pix + p] = v * up;
}

template <int W>
__global__ void __launch_bounds__(128)
    k_spread(double *__restrict__ acc_pad, Geom g, const double *__restrict__ x,
             const double *__restrict__ y, const double *__restrict__ z,
             const double *__restrict__ c, int64_t npts) {
  const double sc1 = g.n1 * (0.5 / M_PI), sc2 = g.n2 * (0.5 / M_PI), sc3 = g.n3 * (0.5 / M_PI);
  for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < npts;
       j += (int64_t)gridDim.x * blockDim.x) {
    double w1[W], w2[W], w3[W];
    const int i0 = axis_setup<W>(x[j], sc1, g.n1, g.off1, g.beta, g.inv_half_w, w1);
    const int j0 = axis_setup<W>(y[j], sc2, g.n2, g.off2, g.beta, g.inv_half_w, w2);
    const int k0 = axis_setup<W>(z[j], sc3, g.n3, g.off3, g.beta, g.inv_half_w, w3);
    const double cj = c[j];
#pragma unroll
    for (int q = 0; q < W; ++q) w3[q] *= cj;
#pragma unroll 1
    for (int a = 0; a < W; ++a) {
#pragma unroll 1
      for (int b = 0; b < W; ++b) {
        const double wab = w1[a] * w2[b];
        double *row = acc_pad + ((size_t)(i0 + a) * g.p2 + (j0 + b)) * g.p3 + k0;
#pragma unroll
        for (int q = 0; q < W; ++q) atomicAdd(row + q, wab * w3[q]);
      }
    }
  }
}

#define SPF_W64_DISPATCH(w, KERNEL_CALL)                           \
  switch (w) {                                                     \
    case 2: { constexpr int W = 2; KERNEL_CALL; break; }           \
    case 3: { constexpr int W = 3; KERNEL_CALL; break; }           \
    case 4: { constexpr int W = 4; KERNEL_CALL; break; }           \
    case 5: { constexpr int W = 5; KERNEL_CALL; break; }           \
    case 6: { constexpr int W = 6; KERNEL_CALL; break; }           \
    case 7: { constexpr int W = 7; KERNEL_CALL; break; }           \
    case 8: { constexpr int W = 8; KERNEL_CALL; break; }           \
    case 9: { constexpr int W = 9; KERNEL_CALL; break; }           \
    case 10: { constexpr int W = 10; KERNEL_CALL; break; }         \
    case 11: { constexpr int W = 11; KERNEL_CALL; break; }         \
    case 12: { constexpr int W = 12; KERNEL_CALL; break; }         \
    case 13: { constexpr int W = 13; KERNEL_CALL; break; }         \
    case 14: { constexpr int W = 14; KERNEL_CALL; break; }         \
    case 15: { constexpr int W = 15; KERNEL_CALL; break; }         \
    case 16: { constexpr int W = 16; KERNEL_CALL; break; }         \
    default: set_error("unsupported kernel width %d", w); return SPF_ERR_UNSUPPORTED; \
  }

static int check_plan(spf_nufft64_plan P, const char *what) {
  if (!P) {
    set_error("%s: plan is NULL", what);
    return SPF_ERR_ARG;
  }
  int dev = -1;
  cudaGetDevice(&dev);
  if (dev != P->dev) {
    set_error("%s: plan was made on device %d, current device is %d", what, P->dev, dev);
    return SPF_ERR_ARG;
  }
  return SPF_OK;
}

static GridDims grid_dims(const spf_nufft64_plan_s *P) {
  const Geom g = geom_of(P);
  return GridDims{g.n1, g.n2, g.n3, g.p1, g.p2, g.p3, g.off1, g.off2, g.off3};
}

// half spectrum (sign -1) of the fine grid
static int fft_exec(spf_nufft64_plan P, cudaStream_t s, const char *what) {
  if (cufftSetStream(P->fft, s) != CUFFT_SUCCESS) {
    set_error("%s: cufftSetStream failed", what);
    return SPF_ERR_CUDA;
  }
  cufftResult r = cufftExecD2Z(P->fft, reinterpret_cast<cufftDoubleReal *>(P->fine),
                               reinterpret_cast<cufftDoubleComplex *>(P->half));
  if (r != CUFFT_SUCCESS) {
    set_error("%s: cufftExecD2Z failed (%d)", what, (int)r);
    return SPF_ERR_CUDA;
  }
  count_launch();
  return SPF_OK;
}

// points per thread-block for the FP64 kernels, and the scale of the
// coordinate (radians) to the fine grid per axis
static void grid_scales(const spf_nufft64_plan_s *P, double scale, double *s) {
  for (int d = 0; d < 3; ++d) s[d] = scale * P->n[d] / (2.0 * M_PI);
}

}  // namespace f64
}  // namespace spf

using namespace spf;
using namespace spf::f64;

extern "C" {

static Pair pair_of(double v) {
  Pair p;
  p.h = (float)v;
  p.l = (float)(v - (double)p.h);
  return p;
}

// The float-pair grid, its peak and the table of exponentials in one
// allocation, made with the plan (setting a model then allocates nothing and
// can be captured).  Where there is no memory for it the plan does without, and
// slices in FP64.
static int alloc_pairs(spf_nufft64_plan P) {
  const size_t npad = (size_t)P->np[0] * P->np[1] * P->np[2];
  const int n = (int)ceil(EXP_PER_UNIT * P->beta) + 2;
  // exp(-j / 128) as a product of two (to 2^-52): an exponential for each of the
  // 3,900 takes the host longer than the allocation
  constexpr int step = 64;
  double part[step], whole = 1.0;
  for (int j = 0; j < step; ++j) part[j] = exp(-(double)j / EXP_PER_UNIT);
  std::vector<float2> t(n);
  for (int j = 0; j < n; ++j) {
    if (j % step == 0) whole = exp(-(double)j / EXP_PER_UNIT);
    const Pair p = pair_of(whole * part[j % step]);
    t[j] = make_float2(p.h, p.l);
  }
  if (cudaMalloc(&P->pair_pad, (npad + n + 1) * sizeof(float2)) != cudaSuccess) {
    cudaGetLastError();
    P->pair_pad = nullptr;
    return SPF_OK;
  }
  P->exp_table = P->pair_pad + npad;
  P->peak = reinterpret_cast<unsigned long long *>(P->exp_table + n);
  return check_cuda(cudaMemcpy(P->exp_table, t.data(), n * sizeof(float2), cudaMemcpyHostToDevice),
                    "plan64_create");
}

int spf_nufft64_plan_create(int m1, int m2, int m3, double eps, double upsampfac,
                            spf_nufft64_plan *out) {
  SPF_REQUIRE(out != nullptr, "spf_nufft64_plan_create: out is NULL");
  *out = nullptr;
  SPF_REQUIRE(m1 > 0 && m2 > 0 && m3 > 0 && m1 <= 2048 && m2 <= 2048 && m3 <= 2048,
              "spf_nufft64_plan_create: bad mode counts (%d, %d, %d)", m1, m2, m3);
  SPF_REQUIRE(eps >= 1e-15 && eps < 1, "spf_nufft64_plan_create: eps must be in [1e-15, 1)");
  const double sigma = upsampfac <= 0 ? 2.0 : upsampfac;
  SPF_REQUIRE(sigma >= 1.25 && sigma <= 4.0, "spf_nufft64_plan_create: upsampfac out of range");
  auto *P = new spf_nufft64_plan_s();
  cudaGetDevice(&P->dev);
  P->m[0] = m1; P->m[1] = m2; P->m[2] = m3;
  P->eps = eps;
  P->sigma = sigma;
  P->w = es_width_for(eps, sigma, 2, 16);
  P->beta = es_beta_for(P->w, sigma);
  P->pad = (P->w + 1) / 2 + 1;
  for (int d = 0; d < 3; ++d) {
    int want = (int)ceil(sigma * P->m[d]);
    if (want < 2 * P->w) want = 2 * P->w;
    P->n[d] = es_next_smooth_even(want);
    P->np[d] = P->n[d] + 2 * P->pad;
  }
  // rows of the float-pair grid start on 16-byte boundaries; the extra cell is
  // never inside a footprint
  P->np[2] = (P->np[2] + 1) & ~1;
  int st = SPF_OK;
  const size_t nfine = (size_t)P->n[0] * P->n[1] * P->n[2];
  const size_t npad = (size_t)P->np[0] * P->np[1] * P->np[2];
  for (int d = 0; d < 3 && st == SPF_OK; ++d) {
    auto v = es_inverse_kernel_ft(P->m[d], P->n[d], P->w, P->beta);
    st = check_cuda(cudaMalloc(&P->inv_p[d], v.size() * sizeof(double)), "plan64_create");
    if (st == SPF_OK)
      st = check_cuda(cudaMemcpy(P->inv_p[d], v.data(), v.size() * sizeof(double),
                                 cudaMemcpyHostToDevice), "plan64_create");
  }
  // one allocation: the real grid (an even number of values), then its half spectrum
  if (st == SPF_OK)
    st = check_cuda(cudaMalloc(&P->fine, nfine * sizeof(double) + (size_t)P->n[0] * P->n[1] *
                                             (P->n[2] / 2 + 1) * sizeof(double2)), "plan64_create");
  if (st == SPF_OK) P->half = reinterpret_cast<double2 *>(P->fine + nfine);
  if (st == SPF_OK) st = check_cuda(cudaMalloc(&P->re_pad, npad * sizeof(double)), "plan64_create");
  if (st == SPF_OK) {
    cufftResult r = cufftPlan3d(&P->fft, P->n[0], P->n[1], P->n[2], CUFFT_D2Z);
    if (r != CUFFT_SUCCESS) {
      set_error("plan64_create: cufftPlan3d(%d,%d,%d) failed (%d)", P->n[0], P->n[1], P->n[2],
                (int)r);
      st = r == CUFFT_ALLOC_FAILED ? SPF_ERR_OOM : SPF_ERR_CUDA;
    } else {
      P->fft_ok = true;
    }
  }
  if (st == SPF_OK && P->w <= PAIR_MAX_W) st = alloc_pairs(P);
  if (st != SPF_OK) {
    spf_nufft64_plan_destroy(P);
    return st;
  }
  *out = P;
  return SPF_OK;
}

int spf_nufft64_plan_destroy(spf_nufft64_plan P) {
  if (!P) return SPF_OK;
  int prev = -1;
  cudaGetDevice(&prev);
  if (prev != P->dev) cudaSetDevice(P->dev);
  for (int d = 0; d < 3; ++d) cudaFree(P->inv_p[d]);
  cudaFree(P->fine);
  cudaFree(P->re_pad);
  cudaFree(P->im_pad);
  cudaFree(P->acc_pad);
  cudaFree(P->pair_pad);
  if (P->fft_ok) cufftDestroy(P->fft);
  if (prev != P->dev && prev >= 0) cudaSetDevice(prev);
  delete P;
  return SPF_OK;
}

int spf_nufft64_plan_info(spf_nufft64_plan P, int *n_fine, int *width, double *beta,
                          int *n_padded) {
  SPF_REQUIRE(P != nullptr, "spf_nufft64_plan_info: plan is NULL");
  for (int d = 0; d < 3; ++d) {
    if (n_fine) n_fine[d] = P->n[d];
    if (n_padded) n_padded[d] = P->np[d];
  }
  if (width) *width = P->w;
  if (beta) *beta = P->beta;
  return SPF_OK;
}

// the float-pair copy of the padded grid, part of setting a model (so that a
// captured slicing reads the model set last)
static int make_pairs(spf_nufft64_plan P, cudaStream_t s) {
  const int64_t npad = (int64_t)P->np[0] * P->np[1] * P->np[2];
  k_to_pairs<<<grid_for(npad, 256, (int64_t)sm_count() * 16), 256, 0, s>>>(P->re_pad, npad, P->peak,
                                                                          P->pair_pad);
  return check_launch("k_to_pairs");
}

int spf_nufft64_t2_set_modes(spf_nufft64_plan P, const double *d_modes, const double *d_support,
                             int isign, int want_imag, void *stream) {
  SPF_TRY(check_plan(P, "spf_nufft64_t2_set_modes"));
  SPF_REQUIRE(d_modes != nullptr, "spf_nufft64_t2_set_modes: modes is NULL");
  SPF_REQUIRE(isign == 1 || isign == -1, "spf_nufft64_t2_set_modes: isign must be +-1");
  cudaStream_t s = as_stream(stream);
  const size_t npad = (size_t)P->np[0] * P->np[1] * P->np[2];
  if (want_imag && !P->im_pad)
    SPF_TRY(check_cuda(cudaMalloc(&P->im_pad, npad * sizeof(double)), "spf_nufft64_t2_set_modes"));
  const GridDims g = grid_dims(P);
  k_modes_to_grid<double><<<row_grid((int64_t)g.n1 * g.n2), row_block(), 0, s>>>(
      d_modes, d_support, P->m[0], P->m[1], P->m[2], g, P->inv_p[0], P->inv_p[1], P->inv_p[2],
      P->fine, P->peak);
  SPF_TRY(check_launch("k_modes_to_grid"));
  SPF_TRY(fft_exec(P, s, "spf_nufft64_t2_set_modes"));
  k_spectrum_to_padded<double><<<row_grid((int64_t)g.p1 * g.p2), row_block(), 0, s>>>(
      P->half, g, isign < 0 ? double(1) : double(-1), P->re_pad,
      want_imag ? P->im_pad : nullptr, nullptr, P->peak);
  SPF_TRY(check_launch("k_spectrum_to_padded"));
  return P->pair_pad ? make_pairs(P, s) : SPF_OK;
}

int spf_nufft64_t2_interp(spf_nufft64_plan P, const double *d_x, const double *d_y,
                          const double *d_z, int64_t npts, double *d_out_re, double *d_out_im,
                          void *stream) {
  SPF_TRY(check_plan(P, "spf_nufft64_t2_interp"));
  SPF_REQUIRE(npts >= 0, "spf_nufft64_t2_interp: npts < 0");
  if (npts == 0) return SPF_OK;
  SPF_REQUIRE(d_x && d_y && d_z && d_out_re, "spf_nufft64_t2_interp: NULL pointer");
  SPF_REQUIRE(!d_out_im || P->im_pad,
              "spf_nufft64_t2_interp: imaginary output needs set_modes(want_imag=1)");
  cudaStream_t s = as_stream(stream);
  const Geom g = geom_of(P);
  const int grid = grid_for(npts, 128, (int64_t)sm_count() * 32);
  SPF_W64_DISPATCH(P->w, (k_interp<W><<<grid, 128, 0, s>>>(P->re_pad, P->im_pad, g, d_x, d_y,
                                                              d_z, npts, d_out_re, d_out_im)));
  return check_launch("k_interp (f64)");
}

static int slice_f64(spf_nufft64_plan P, const double *d_quats, int64_t n_orient,
                     const double *d_ppr, int64_t n_pix, double scale, double *d_out,
                     const unsigned long long *peak, cudaStream_t s) {
  const Geom g = geom_of(P);
  double sc[3];
  grid_scales(P, scale, sc);
  const dim3 grid((unsigned)n_orient, (unsigned)((n_pix + 127) / 128));
  SPF_W64_DISPATCH(P->w, (k_slice<W><<<grid, 128, 0, s>>>(P->re_pad, g, d_quats, d_ppr, n_pix,
                                                             sc[0], sc[1], sc[2], d_out, peak)));
  return check_launch("k_slice (f64)");
}

int spf_slice_t2_f64(spf_nufft64_plan P, const double *d_quats, int64_t n_orient,
                     const double *d_ppr, int64_t n_pix, double scale, double *d_out,
                     void *stream) {
  SPF_TRY(check_plan(P, "spf_slice_t2_f64"));
  SPF_REQUIRE(n_orient >= 0 && n_pix >= 0, "spf_slice_t2_f64: negative size");
  if (n_orient == 0 || n_pix == 0) return SPF_OK;
  SPF_REQUIRE(d_quats && d_ppr && d_out, "spf_slice_t2_f64: NULL pointer");
  SPF_REQUIRE(n_orient < (1LL << 31) && n_pix <= 65535LL * 128, "spf_slice_t2_f64: size too large");
  return slice_f64(P, d_quats, n_orient, d_ppr, n_pix, scale, d_out, nullptr, as_stream(stream));
}

// Whether slices by pairs are the quicker ones.  A patch costs the same however few
// of its 32 pixels a panel has; the FP64 kernel's unit is 32 consecutive pixels.
// By width, a patch over a unit: 0.78-0.95 at W = 3, 0.62 at 4, 0.41 at 7, 0.33 at
// 10, 0.30 at 13 (in FP64 always at W = 2: 1.02-1.2).  Pairs / FP64, us: 1 x 4096 x 1
// pixels (8 patches a unit) 2,912 / 1,354 at W = 13 and 1,973 / 797 at 10;
// 1 x 4096 x 3 (2.7) 1,760 / 2,306 at 13, 807 / 748 at 7; 16 x 17 x 19 (1.5)
// 569 / 1,354 at 13, 196 / 216 at 4.
static bool pairs_pay(int w, int64_t patches, int64_t n_pix) {
  const int64_t units = (n_pix + PAIR_PIX - 1) / PAIR_PIX;
  return (0.12 + 2.3 / w) * (double)patches <= 0.95 * (double)units;
}

int spf_slice_t2_f64_det(spf_nufft64_plan P, const double *d_quats, int64_t n_orient,
                         const double *d_ppr, int n_panels, int nx, int ny, double scale,
                         double *d_out, void *stream) {
  SPF_TRY(check_plan(P, "spf_slice_t2_f64_det"));
  SPF_REQUIRE(n_orient >= 0 && n_panels >= 0 && nx >= 0 && ny >= 0,
              "spf_slice_t2_f64_det: negative size");
  if (n_orient == 0 || n_panels == 0 || nx == 0 || ny == 0) return SPF_OK;
  const int64_t patches =
      (int64_t)n_panels * ((nx + PAIR_PX - 1) / PAIR_PX) * ((ny + PAIR_PY - 1) / PAIR_PY);
  const int64_t n_pix = (int64_t)n_panels * nx * ny;
  if (!P->pair_pad || patches > 65535 || !pairs_pay(P->w, patches, n_pix))
    return spf_slice_t2_f64(P, d_quats, n_orient, d_ppr, n_pix, scale, d_out, stream);
  SPF_REQUIRE(d_quats && d_ppr && d_out, "spf_slice_t2_f64_det: NULL pointer");
  SPF_REQUIRE(n_orient < (1LL << 31) && n_pix <= 65535LL * 128,
              "spf_slice_t2_f64_det: size too large");
  cudaStream_t s = as_stream(stream);
  const Geom g = geom_of(P);
  double sc[3];
  grid_scales(P, scale, sc);
  const dim3 grid((unsigned)n_orient, (unsigned)patches);
  const int smem = PAIR_CELLS * (int)sizeof(float2);
  const double per_z2 = 4.0 / ((double)P->w * P->w);
  const PairKernel kernel{pair_of(per_z2), pair_of(-P->beta * per_z2)};
  const int last = (int)ceil(EXP_PER_UNIT * P->beta) + 1;
#define SPF_PAIR_CASE(w_)                                                                        \
  case w_:                                                                                       \
    cudaFuncSetAttribute(k_slice_pairs<w_>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);  \
    k_slice_pairs<w_><<<grid, PAIR_WARPS * 32, smem, s>>>(                                       \
        P->pair_pad, P->peak, g, d_quats, d_ppr, n_panels, nx, ny, sc[0], sc[1], sc[2], kernel,  \
        P->exp_table, last, d_out);                                                        \
    break;
  switch (P->w) {
    SPF_PAIR_CASE(2)
    SPF_PAIR_CASE(3)
    SPF_PAIR_CASE(4)
    SPF_PAIR_CASE(5)
    SPF_PAIR_CASE(6)
    SPF_PAIR_CASE(7)
    SPF_PAIR_CASE(8)
    SPF_PAIR_CASE(9)
    SPF_PAIR_CASE(10)
    SPF_PAIR_CASE(11)
    SPF_PAIR_CASE(12)
    SPF_PAIR_CASE(13)
    default: set_error("unsupported kernel width %d", P->w); return SPF_ERR_UNSUPPORTED;
  }
#undef SPF_PAIR_CASE
  SPF_TRY(check_launch("k_slice_pairs"));
  // a grid that pairs of floats cannot hold (NaN, infinity, nothing normal)
  return slice_f64(P, d_quats, n_orient, d_ppr, n_pix, scale, d_out, P->peak, s);
}

int spf_nufft64_t1_zero(spf_nufft64_plan P, void *stream) {
  SPF_TRY(check_plan(P, "spf_nufft64_t1_zero"));
  const size_t npad = (size_t)P->np[0] * P->np[1] * P->np[2];
  if (!P->acc_pad)
    SPF_TRY(check_cuda(cudaMalloc(&P->acc_pad, npad * sizeof(double)), "spf_nufft64_t1_zero"));
  return check_cuda(cudaMemsetAsync(P->acc_pad, 0, npad * sizeof(double), as_stream(stream)),
                    "spf_nufft64_t1_zero");
}

int spf_nufft64_t1_spread(spf_nufft64_plan P, const double *d_x, const double *d_y,
                          const double *d_z, const double *d_c, int64_t npts, void *stream) {
  SPF_TRY(check_plan(P, "spf_nufft64_t1_spread"));
  SPF_REQUIRE(P->acc_pad != nullptr, "spf_nufft64_t1_spread: call spf_nufft64_t1_zero first");
  SPF_REQUIRE(npts >= 0, "spf_nufft64_t1_spread: npts < 0");
  if (npts == 0) return SPF_OK;
  SPF_REQUIRE(d_x && d_y && d_z && d_c, "spf_nufft64_t1_spread: NULL pointer");
  cudaStream_t s = as_stream(stream);
  const Geom g = geom_of(P);
  const int grid = grid_for(npts, 128, (int64_t)sm_count() * 32);
  SPF_W64_DISPATCH(P->w, (k_spread<W><<<grid, 128, 0, s>>>(P->acc_pad, g, d_x, d_y, d_z, d_c,
                                                              npts)));
  return check_launch("k_spread (f64)");
}

int spf_nufft64_t1_finish(spf_nufft64_plan P, int isign, double *d_out_re, double *d_out_im,
                          void *stream) {
  SPF_TRY(check_plan(P, "spf_nufft64_t1_finish"));
  SPF_REQUIRE(P->acc_pad != nullptr, "spf_nufft64_t1_finish: call spf_nufft64_t1_zero first");
  SPF_REQUIRE(isign == 1 || isign == -1, "spf_nufft64_t1_finish: isign must be +-1");
  SPF_REQUIRE(d_out_re != nullptr, "spf_nufft64_t1_finish: out_re is NULL");
  cudaStream_t s = as_stream(stream);
  const GridDims g = grid_dims(P);
  k_fold_padded<double><<<row_grid((int64_t)g.n1 * g.n2), row_block(), 0, s>>>(P->acc_pad, g, P->fine);
  SPF_TRY(check_launch("k_fold_padded"));
  SPF_TRY(fft_exec(P, s, "spf_nufft64_t1_finish"));
  k_spectrum_to_modes<double><<<row_grid((int64_t)P->m[0] * P->m[1]), row_block(), 0, s>>>(
      P->half, P->m[0], P->m[1], P->m[2], g, P->inv_p[0], P->inv_p[1], P->inv_p[2],
      isign < 0 ? double(1) : double(-1), d_out_re, d_out_im);
  return check_launch("k_spectrum_to_modes");
}

}  // extern "C"
