// The regular-grid side of the NUFFT plans, FP32 and FP64: modes to the
// upsampled grid, its spectrum to the padded grid that type 2 reads, the
// accumulator of type 1 back onto the grid, and the spectrum to modes.
//
// Modes (type 2) and strengths (type 1) are real, so one real-to-complex
// transform does: half the spectrum is kept, half[a][b][c] for c <= n3 / 2, and
// F(-k) = conj F(k) gives the rest.  The transform, which is of the sign -1,
// costs less than a complex one (320^3: 420 us before, 275 now), and either
// sign's result is read from it (the sign +1 is the conjugate).
//
// Every kernel walks rows along the fastest axis, a warp a row, so that a row
// costs one division and its cells none; flat indices with 64-bit divisions a
// cell took 221 us to fold a 320^3 grid and 47 us to fill the padded 162^3,
// these take 65 and 17.
#pragma once
#include "common.cuh"

namespace spf {

template <class T>
struct Complex;
template <>
struct Complex<float> {
  using type = float2;
};
template <>
struct Complex<double> {
  using type = double2;
};

struct GridDims {
  int n1, n2, n3;        // upsampled grid
  int p1, p2, p3;        // padded grid
  int off1, off2, off3;  // n / 2 + pad
};

constexpr int ROWS_PER_CTA = 8;
inline dim3 row_block() { return dim3(32, ROWS_PER_CTA); }
inline unsigned row_grid(int64_t rows) {
  return (unsigned)((rows + ROWS_PER_CTA - 1) / ROWS_PER_CTA);
}

__device__ __forceinline__ int wrap(int i, int n) {
  i %= n;
  return i < 0 ? i + n : i;
}

// grid[k mod n] = f_k * support_k / (p1 p2 p3), zero elsewhere; and *peak = 0
template <class T>
__global__ void k_modes_to_grid(const T *__restrict__ f, const T *__restrict__ sup, int m1, int m2,
                                int m3, GridDims g, const T *__restrict__ ip1,
                                const T *__restrict__ ip2, const T *__restrict__ ip3,
                                T *__restrict__ grid, unsigned long long *__restrict__ peak) {
  if (peak && blockIdx.x == 0 && threadIdx.x == 0 && threadIdx.y == 0) *peak = 0;
  const int64_t row = (int64_t)blockIdx.x * ROWS_PER_CTA + threadIdx.y;
  if (row >= (int64_t)g.n1 * g.n2) return;
  const int fa = (int)(row / g.n2), fb = (int)(row % g.n2);
  // signed mode numbers; negative modes sit at the end of an axis
  const int ka = fa >= g.n1 - m1 / 2 ? fa - g.n1 : fa, kb = fb >= g.n2 - m2 / 2 ? fb - g.n2 : fb;
  const bool in = ka < m1 - m1 / 2 && kb < m2 - m2 / 2;
  const int a = ka + m1 / 2, b = kb + m2 / 2;
  const T *src = f + ((int64_t)a * m2 + b) * m3, *ssrc = sup + ((int64_t)a * m2 + b) * m3;
  const T p12 = in ? ip1[a] * ip2[b] : T(0);
  T *dst = grid + row * g.n3;
  for (int fc = threadIdx.x; fc < g.n3; fc += 32) {
    const int kc = fc >= g.n3 - m3 / 2 ? fc - g.n3 : fc;
    T v = T(0);
    if (in && kc < m3 - m3 / 2) {
      const int c = kc + m3 / 2;
      v = src[c];
      if (sup) v *= ssrc[c];
      v *= p12 * ip3[c];
    }
    dst[fc] = v;
  }
}

// re[i] = Re F[(i - off) mod n] for every padded cell, and where asked for
// im = im_sign Im F or the pairs (re, im); for doubles, in *peak the bits of
// max |re| (NaN above infinity above all values)
template <class T>
__global__ void k_spectrum_to_padded(const typename Complex<T>::type *__restrict__ half,
                                     GridDims g, T im_sign, T *__restrict__ re,
                                     T *__restrict__ im,
                                     typename Complex<T>::type *__restrict__ cx,
                                     unsigned long long *__restrict__ peak) {
  const int64_t row = (int64_t)blockIdx.x * ROWS_PER_CTA + threadIdx.y;
  if (row >= (int64_t)g.p1 * g.p2) return;
  unsigned long long top = 0;
  const int nh = g.n3 / 2 + 1;
  const int a = wrap((int)(row / g.p2) - g.off1, g.n1), b = wrap((int)(row % g.p2) - g.off2, g.n2);
  const auto *h = half + ((int64_t)a * g.n2 + b) * nh;
  const auto *hm =
      half + ((int64_t)(a ? g.n1 - a : 0) * g.n2 + (b ? g.n2 - b : 0)) * nh;  // at (-a, -b)
  for (int k = threadIdx.x; k < g.p3; k += 32) {
    int c = k - g.off3;
    while (c < 0) c += g.n3;
    while (c >= g.n3) c -= g.n3;
    const bool direct = c < nh;
    const auto v = direct ? h[c] : hm[g.n3 - c];
    re[row * g.p3 + k] = v.x;
    if constexpr (sizeof(T) == 8) {
      const unsigned long long b = (unsigned long long)__double_as_longlong(v.x) & ~(1ULL << 63);
      top = b > top ? b : top;
    }
    const T y = direct ? im_sign * v.y : -im_sign * v.y;
    if (im) im[row * g.p3 + k] = y;
    if (cx) {
      typename Complex<T>::type q;
      q.x = v.x;
      q.y = y;
      cx[row * g.p3 + k] = q;
    }
  }
  if constexpr (sizeof(T) == 8) {
    if (!peak) return;
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) {
      const unsigned long long u = __shfl_xor_sync(0xffffffffu, top, o);
      top = u > top ? u : top;
    }
    // most rows are below what others have put there
    if (threadIdx.x == 0 && top > *(volatile unsigned long long *)peak) atomicMax(peak, top);
  }
}

// grid[l] = sum of acc[i] over padded i == l + off (mod n)
template <class T>
__global__ void k_fold_padded(const T *__restrict__ acc, GridDims g, T *__restrict__ grid) {
  const int64_t row = (int64_t)blockIdx.x * ROWS_PER_CTA + threadIdx.y;
  if (row >= (int64_t)g.n1 * g.n2) return;
  const int i0 = wrap((int)(row / g.n2) + g.off1, g.n1), j0 = wrap((int)(row % g.n2) + g.off2, g.n2);
  T *dst = grid + row * g.n3;
  if (i0 + g.n1 >= g.p1 && j0 + g.n2 >= g.p2 && g.off3 + g.n3 >= g.p3 &&
      g.off3 <= g.n3) {
    // one row of the accumulator (all but the halo's): a cell is its cells k -
    // n3 and k = c + off3 (the conditions on n3, which every but the smallest
    // grid meets: k + n3 is past the row for all c, and k - 2 n3 before it),
    // four cells' loads in flight (98 us for 320^3 cells through the loops below)
    const T *r = acc + ((int64_t)i0 * g.p2 + j0) * g.p3;
#pragma unroll 4
    for (int c = threadIdx.x; c < g.n3; c += 32) {
      const int k = c + g.off3;
      T s = T(0);
      if (k >= g.n3) s += r[k - g.n3];
      if (k < g.p3) s += r[k];
      dst[c] = s;
    }
    return;
  }
  for (int c = threadIdx.x; c < g.n3; c += 32) {
    int k0 = c + g.off3;
    while (k0 >= g.n3) k0 -= g.n3;
    T s = T(0);
    for (int i = i0; i < g.p1; i += g.n1)
      for (int j = j0; j < g.p2; j += g.n2) {
        const T *r = acc + ((int64_t)i * g.p2 + j) * g.p3;
        for (int k = k0; k < g.p3; k += g.n3) s += r[k];
      }
    dst[c] = s;
  }
}

// modes[k] = F(k) / (p1 p2 p3), im_sign as above
template <class T>
__global__ void k_spectrum_to_modes(const typename Complex<T>::type *__restrict__ half, int m1,
                                    int m2, int m3, GridDims g, const T *__restrict__ ip1,
                                    const T *__restrict__ ip2, const T *__restrict__ ip3,
                                    T im_sign, T *__restrict__ out_re, T *__restrict__ out_im) {
  const int64_t row = (int64_t)blockIdx.x * ROWS_PER_CTA + threadIdx.y;
  if (row >= (int64_t)m1 * m2) return;
  const int nh = g.n3 / 2 + 1;
  const int a = (int)(row / m2), b = (int)(row % m2);
  const int fa = wrap(a - m1 / 2, g.n1), fb = wrap(b - m2 / 2, g.n2);
  const auto *h = half + ((int64_t)fa * g.n2 + fb) * nh;
  const auto *hm = half + ((int64_t)(fa ? g.n1 - fa : 0) * g.n2 + (fb ? g.n2 - fb : 0)) * nh;
  const T p12 = ip1[a] * ip2[b];
  for (int c = threadIdx.x; c < m3; c += 32) {
    const int kc = c - m3 / 2;
    const auto v = kc >= 0 ? h[kc] : hm[-kc];
    const T s = p12 * ip3[c];
    out_re[row * m3 + c] = v.x * s;
    if (out_im) out_im[row * m3 + c] = (kc >= 0 ? im_sign : -im_sign) * v.y * s;
  }
}

}  // namespace spf
