// FP64 argmin of the distances sum_p (x_p - s_p)^2 without computing all of
// them in FP64, which this chip runs at about 1/64 of its FP32 rate (2
// instructions a pixel and pair: 13.5 ms at best for 500 x 2,000 pairs of
// 4,096 pixels).
//
// An FP32 pass over converted rows gives v = s^2 - 2 x.s for every pair with a
// bound B on its error (below).  With m = min_r (v_r + B_r), a reference with
// v_r - B_r > m is further than the one at the minimum; the others, a handful
// a frame, get their distance in FP64 with the arithmetic of spf_dist_f64, one
// chain d = x_p - s_p, acc = fma(d, d, acc) over the pixels in order, so the
// answer is the full computation's, distance bits and ties (lower index)
// included.  A frame with more than half of the references left (equal
// references, values FP32 cannot tell apart, NaN or infinity) is computed
// against all of them.  500 x 2,000 pairs of 4,096 pixels: 35.9 ms with
// 128-pair FP64 tiles, 17.8 with 64-pair tiles, 0.46 here (FP32 pass 234 us,
// FP64 chains 171 us, their latency).
//
// The bound.  u = 2^-24; X, S the rows' norms.  Conversion moves an element by
// at most u of it (2^-126 below FP32's normal range); sums run in chains of
// 256 pixels that are added up, so a sum of K products is off by at most
// (256 + K/256) u of the sum of magnitudes, itself at most X S
// (Cauchy-Schwarz; Higham 2002, 3.1); the rounding of v adds 2 u.  Together
// c (S^2 + 2 X S) with c = 1.05 (256 + K/256 + 16) u, plus (K + 8) 2^-52 (X + S)^2
// for the FP64 chains' own rounding and K 1e-37 (1 + X + S) for underflow.
// Rows with NaN, infinity or elements of 2^50 and more have no bound and are
// never left out.
#include <math.h>

#include "common.cuh"
#include "match_tile.cuh"

namespace spf {
namespace m64 {

constexpr int SUM_STEPS = 16;  // k-steps a chain: 256 pixels

// converted rows, their norms (infinity: no bound), and the per-call counters
struct Work {
  float *x32, *r32;
  float *xn, *rn;
  float *v;       // [n_img][ldv]; later the listed pairs' FP64 distances
  int2 *pairs;    // (image, reference), at most ldv / 2 an image
  int *base, *cnt;  // an image's pairs; cnt < 0: all references
  int *total;
  double *part_d;   // [n_img][parts]: minima over blocks of references, for
  int64_t *part_r;  // frames without a list
  int64_t ldx, ldv, parts;
};

constexpr int ALL_REFS = 512;  // references a block of k_all

// Double to nearest float by integer operations (conversions run at the FP64
// rate); zero below the normal range.  bad: NaN, infinity or |d| >= 2^50.
__device__ __forceinline__ float narrow(double d, bool &bad) {
  const unsigned lo = (unsigned)__double2loint(d), hi = (unsigned)__double2hiint(d);
  const unsigned e = (hi >> 20) & 0x7ffu;
  bad |= e >= 1023u + 50u;
  if (e < 897u || e >= 1023u + 50u) return 0.0f;
  const unsigned bits = (((hi & 0x7fffffffu) << 3) | (lo >> 29)) - (896u << 23);
  return __uint_as_float((hi & 0x80000000u) | (bits + ((lo >> 28) & 1u)));
}

// one CTA a row
__global__ void __launch_bounds__(256)
    k_narrow_rows(const double *__restrict__ x, int64_t n_pix, float *__restrict__ out,
                  int64_t ld, float *__restrict__ norm) {
  __shared__ float part[8];
  const int64_t r = blockIdx.x;
  const double *p = x + r * n_pix;
  float *o = out + r * ld;
  float s = 0.0f;
  bool bad = false;
  constexpr int U = 8;
  for (int64_t k = threadIdx.x; k < n_pix; k += 256 * U) {
    double d[U];
#pragma unroll
    for (int u = 0; u < U; ++u) d[u] = k + 256 * u < n_pix ? __ldg(p + k + 256 * u) : 0.0;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const float f = narrow(d[u], bad);
      s = fmaf(f, f, s);
      if (k + 256 * u < n_pix) o[k + 256 * u] = f;
    }
  }
  for (int64_t k = n_pix + threadIdx.x; k < ld; k += 256) o[k] = 0.0f;
#pragma unroll
  for (int q = 16; q >= 1; q >>= 1) s += __shfl_xor_sync(0xffffffffu, s, q);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = s;
  const bool any = __syncthreads_or(bad);
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; ++w) s += part[w];
    norm[r] = any ? __int_as_float(0x7f800000) : sqrtf(s);
  }
}

// v[i][r] = S_r^2 - 2 x_i . s_r (-infinity for a reference without a bound)
template <class TL>
__global__ void __launch_bounds__(TL::THREADS)
    k_filter(Work w, int64_t n_img, int64_t n_ref, int64_t K, int group_m) {
  __shared__ __align__(16) float As[2][TB_K][TL::TM + 4];
  __shared__ __align__(16) float Bs[2][TB_K][TL::TN + 4];
  int64_t mt, nt;
  tile_coords((n_img + TL::TM - 1) / TL::TM, (n_ref + TL::TN - 1) / TL::TN, group_m, mt, nt);
  float acc[TL::RM][TL::RN];
  tile_sums<float, Mode::DOT, TL, SUM_STEPS>(w.x32, n_img, w.r32, n_ref, w.ldx, K, mt * TL::TM,
                                             nt * TL::TN, acc, As, Bs);
  const int tx = threadIdx.x % TL::NTX, ty = threadIdx.x / TL::NTX;
#pragma unroll
  for (int j = 0; j < TL::RN; ++j) {
    const int64_t r = nt * TL::TN + TL::col(tx, j);
    if (r >= n_ref) continue;
    const float sn = w.rn[r];
    const bool bound = sn < __int_as_float(0x7f800000);
#pragma unroll
    for (int i = 0; i < TL::RM; ++i) {
      const int64_t d = mt * TL::TM + TL::row(ty, i);
      if (d < n_img)
        w.v[d * w.ldv + r] = bound ? fmaf(-2.0f, acc[i][j], sn * sn) : -__int_as_float(0x7f800000);
    }
  }
}

// One CTA a frame: the references that can hold its minimum.
__global__ void __launch_bounds__(256) k_select(Work w, int64_t n_ref, int64_t K) {
  __shared__ float mins[8];
  __shared__ int count, at;
  const int64_t i = blockIdx.x;
  const float *v = w.v + i * w.ldv;
  const float X = w.xn[i];
  const float kf = (float)K;
  const float c = 1.05f * (256.0f + kf * (1.0f / 256.0f) + 16.0f) * 5.9604645e-8f;
  const float c64 = (kf + 8.0f) * 2.2204460e-16f, e0 = kf * 1e-37f;
  auto band = [&](float S) {
    const float t = X + S;
    return 1.0001f * (c * S * (S + 2.0f * X) + c64 * t * t + e0 * (1.0f + t));
  };
  float m = __int_as_float(0x7f800000);
  for (int64_t r = threadIdx.x; r < n_ref; r += 256) {
    const float S = w.rn[r];
    if (S < __int_as_float(0x7f800000)) m = fminf(m, v[r] + band(S));
  }
#pragma unroll
  for (int q = 16; q >= 1; q >>= 1) m = fminf(m, __shfl_xor_sync(0xffffffffu, m, q));
  if ((threadIdx.x & 31) == 0) mins[threadIdx.x >> 5] = m;
  if (threadIdx.x == 0) count = 0;
  __syncthreads();
  for (int q = 0; q < 8; ++q) m = fminf(m, mins[q]);
  m = fmaf(fabsf(m), 1e-6f, m);  // the rounding of v + B and v - B
  const bool all = !(X < __int_as_float(0x7f800000));
  auto keep = [&](int64_t r) {
    const float S = w.rn[r];
    return !(S < __int_as_float(0x7f800000)) || !(v[r] - band(S) > m);
  };
  int mine = 0;
  for (int64_t r = threadIdx.x; r < n_ref; r += 256) mine += keep(r);
  if (mine) atomicAdd(&count, mine);
  __syncthreads();
  const int cnt = count;
  const bool dense = all || cnt > (int)(w.ldv / 2);
  if (threadIdx.x == 0) {
    at = 0;
    if (!dense) at = atomicAdd(w.total, cnt);
    w.base[i] = at;
    w.cnt[i] = dense ? -1 : cnt;
  }
  __syncthreads();
  if (dense) return;
  for (int64_t r = threadIdx.x; r < n_ref; r += 256)
    if (keep(r)) w.pairs[atomicAdd(&at, 1)] = make_int2((int)i, (int)r);
}

// FP64 distances of the listed pairs.  A CTA takes 32 pairs at a time; warp 0
// runs the 32 chains, one a lane.  An FP64 instruction holds a warp's quarter
// of the SM for about 64 clocks whatever its lanes, so the chains are 64
// clocks a pixel and nothing but their FMA is left to warp 0: warps 1-3, on
// the other quarters, load the rows a chunk of 32 pixels ahead and subtract
// (500 pairs of 4,096 pixels: 171 us; 291 us with the subtraction in warp 0).
constexpr int CH_PIX = 32, CH_STRIDE = CH_PIX + 2, CH_THREADS = 128, CH_ROWS = 11;

__global__ void __launch_bounds__(CH_THREADS)
    k_pairs(Work w, const double *__restrict__ img, const double *__restrict__ ref, int64_t K) {
  __shared__ __align__(16) double diff[2][32][CH_STRIDE];
  __shared__ const double *rows[2][32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int total = *w.total;
  const int64_t nch = (K + CH_PIX - 1) / CH_PIX;
  double *dist = reinterpret_cast<double *>(w.v);
  for (int q0 = blockIdx.x * 32; q0 < total; q0 += gridDim.x * 32) {
    __syncthreads();  // the previous pairs are done with the rows and the chunks
    if (tid < 32) {
      const int2 pr = w.pairs[min(q0 + lane, total - 1)];
      rows[0][lane] = img + pr.x * K;
      rows[1][lane] = ref + pr.y * K;
    }
    __syncthreads();
    // warp 1 + m takes rows m, m + 3, ...; a pixel past the end subtracts to
    // zero, which leaves a chain as it is
    double x[CH_ROWS], s[CH_ROWS];
    auto load = [&](int64_t ch) {
      const int64_t k = ch * CH_PIX + lane;
#pragma unroll
      for (int u = 0; u < CH_ROWS; ++u) {
        const int r = warp - 1 + 3 * u;
        const bool in = r < 32 && k < K;
        x[u] = in ? __ldg(rows[0][r] + k) : 0.0;
        s[u] = in ? __ldg(rows[1][r] + k) : 0.0;
      }
    };
    auto subtract = [&](int64_t ch) {
#pragma unroll
      for (int u = 0; u < CH_ROWS; ++u) {
        const int r = warp - 1 + 3 * u;
        if (r < 32) diff[ch & 1][r][lane] = x[u] - s[u];
      }
    };
    if (warp > 0) {
      load(0);
      subtract(0);
      load(1);
    }
    double acc = 0.0;
    for (int64_t ch = 0; ch < nch; ++ch) {
      __syncthreads();  // chunk ch is there, and warp 0 is done with chunk ch - 1
      if (warp > 0) {
        subtract(ch + 1);
        load(ch + 2);
      } else {
        const double *d = diff[ch & 1][lane];
#pragma unroll
        for (int k = 0; k < CH_PIX; k += 2) {
          const double2 v = *reinterpret_cast<const double2 *>(d + k);
          acc = fma(v.x, v.x, acc);
          acc = fma(v.y, v.y, acc);
        }
      }
    }
    if (tid < 32 && q0 + lane < total) dist[q0 + lane] = acc;
  }
}

// the better of (d, r) and (od, o): smaller distance, then lower reference
__device__ __forceinline__ void fold(double &d, int64_t &r, double od, int64_t o) {
  if (o >= 0 && (r < 0 || od < d || (od == d && o < r))) {
    d = od;
    r = o;
  }
}

// minimum of (d, r) over a CTA of 128 threads, in thread 0
__device__ __forceinline__ void block_fold(double &d, int64_t &r) {
  __shared__ double sd[4];
  __shared__ int64_t sr[4];
#pragma unroll
  for (int o = 16; o >= 1; o >>= 1) {
    const double od = __shfl_xor_sync(0xffffffffu, d, o);
    const int64_t orr = __shfl_xor_sync(0xffffffffu, r, o);
    fold(d, r, od, orr);
  }
  if ((threadIdx.x & 31) == 0) {
    sd[threadIdx.x >> 5] = d;
    sr[threadIdx.x >> 5] = r;
  }
  __syncthreads();
  if (threadIdx.x == 0)
    for (int q = 1; q < 4; ++q) fold(d, r, sd[q], sr[q]);
}

// Frames without a list: the minimum over a block of ALL_REFS references.  A
// thread a pair, rows read through L1: with every frame dense no slower than the
// tiled distance block (500 x 2,000 x 4,096: 15.8 ms with the pass before, 17.9 the
// block; 1,000 x 3,000 x 1,024: 11.2 and 11.2; 5 x 2,000 x 4,096: 2.4 and 4.3).
__global__ void __launch_bounds__(128)
    k_all(Work w, const double *__restrict__ img, const double *__restrict__ ref, int64_t n_ref,
          int64_t K) {
  const int64_t i = blockIdx.x;
  if (w.cnt[i] >= 0) return;
  const double *x = img + i * K;
  for (int64_t blk = blockIdx.y; blk < w.parts; blk += gridDim.y) {
    const int64_t r0 = blk * ALL_REFS;
    double bd = INFINITY;
    int64_t br = -1;
    for (int64_t r = r0 + threadIdx.x; r < n_ref && r < r0 + ALL_REFS; r += 128) {
      const double *s = ref + r * K;
      double acc = 0.0;
      for (int64_t k = 0; k < K; ++k) {
        const double d = __ldg(x + k) - __ldg(s + k);
        acc = fma(d, d, acc);
      }
      if (acc < INFINITY) fold(bd, br, acc, r);
    }
    __syncthreads();  // thread 0 has read the block before's minima
    block_fold(bd, br);
    if (threadIdx.x == 0) {
      w.part_d[i * w.parts + blk] = bd;
      w.part_r[i * w.parts + blk] = br;
    }
  }
}

// One CTA a frame: the minimum of its pairs or blocks folded into the running
// best as k_argmin_rows_f64 does (strictly smaller distances only; NaN and
// infinity never chosen).
__global__ void __launch_bounds__(128)
    k_best(Work w, int64_t ref_offset, double *__restrict__ best_dist,
           int64_t *__restrict__ best_idx) {
  const int64_t i = blockIdx.x;
  const int cnt = w.cnt[i];
  double bd = INFINITY;
  int64_t br = -1;
  if (cnt >= 0) {
    const double *dist = reinterpret_cast<const double *>(w.v) + w.base[i];
    const int2 *pairs = w.pairs + w.base[i];
    for (int q = threadIdx.x; q < cnt; q += 128)
      if (dist[q] < INFINITY) fold(bd, br, dist[q], pairs[q].y);
  } else {
    for (int64_t q = threadIdx.x; q < w.parts; q += 128)
      fold(bd, br, w.part_d[i * w.parts + q], w.part_r[i * w.parts + q]);
  }
  block_fold(bd, br);
  if (threadIdx.x == 0 && br >= 0 && (best_idx[i] < 0 || bd < best_dist[i])) {
    best_dist[i] = bd;
    best_idx[i] = br + ref_offset;
  }
}

static int64_t up(int64_t v, int64_t a) { return (v + a - 1) / a * a; }

// carves the workspace; returns its size
static int64_t layout(Work &w, unsigned char *p, int64_t n_img, int64_t n_ref, int64_t n_pix) {
  w.ldx = up(n_pix, 4);
  w.ldv = up(n_ref, 2);
  w.parts = up(n_ref, ALL_REFS) / ALL_REFS;
  int64_t off = 0;
  auto take = [&](int64_t bytes) {
    unsigned char *at = p + off;
    off += up(bytes, 256);
    return at;
  };
  w.x32 = reinterpret_cast<float *>(take(n_img * w.ldx * 4));
  w.r32 = reinterpret_cast<float *>(take(n_ref * w.ldx * 4));
  w.v = reinterpret_cast<float *>(take(n_img * w.ldv * 4));
  w.pairs = reinterpret_cast<int2 *>(take(n_img * w.ldv * 4));
  w.xn = reinterpret_cast<float *>(take(n_img * 4));
  w.rn = reinterpret_cast<float *>(take(n_ref * 4));
  w.base = reinterpret_cast<int *>(take(n_img * 4));
  w.cnt = reinterpret_cast<int *>(take(n_img * 4));
  w.total = reinterpret_cast<int *>(take(4));
  w.part_d = reinterpret_cast<double *>(take(n_img * w.parts * 8));
  w.part_r = reinterpret_cast<int64_t *>(take(n_img * w.parts * 8));
  return off;
}

}  // namespace m64
}  // namespace spf

using namespace spf;
using namespace spf::m64;

extern "C" {

int64_t spf_argmin_f64_work_bytes(int64_t n_img, int64_t n_ref, int64_t n_pix) {
  if (n_img <= 0 || n_ref <= 0 || n_pix < 0) return 0;
  Work w;
  return layout(w, nullptr, n_img, n_ref, n_pix) + 256;
}

int spf_argmin_f64(const double *d_img, int64_t n_img, const double *d_ref, int64_t n_ref,
                   int64_t n_pix, int64_t ref_offset, void *d_work, int64_t work_bytes,
                   double *d_best_dist, int64_t *d_best_idx, void *stream) {
  SPF_REQUIRE(n_img >= 0 && n_ref >= 0 && n_pix >= 0 && ref_offset >= 0,
              "spf_argmin_f64: negative size");
  if (n_img == 0 || n_ref == 0) return SPF_OK;
  SPF_REQUIRE(d_img && d_ref && d_work && d_best_dist && d_best_idx,
              "spf_argmin_f64: NULL pointer");
  SPF_REQUIRE(n_img < (1LL << 31) && n_ref < (1LL << 31) && n_img * up(n_ref, 2) / 2 < (1LL << 31),
              "spf_argmin_f64: size too large");
  SPF_REQUIRE(work_bytes >= spf_argmin_f64_work_bytes(n_img, n_ref, n_pix),
              "spf_argmin_f64: workspace too small");
  Work w;
  layout(w, reinterpret_cast<unsigned char *>(up((int64_t)(uintptr_t)d_work, 256)), n_img, n_ref,
         n_pix);
  cudaStream_t s = as_stream(stream);
  SPF_TRY(check_cuda(cudaMemsetAsync(w.total, 0, sizeof(int), s), "spf_argmin_f64"));
  k_narrow_rows<<<(unsigned)n_img, 256, 0, s>>>(d_img, n_pix, w.x32, w.ldx, w.xn);
  SPF_TRY(check_launch("k_narrow_rows"));
  k_narrow_rows<<<(unsigned)n_ref, 256, 0, s>>>(d_ref, n_pix, w.r32, w.ldx, w.rn);
  SPF_TRY(check_launch("k_narrow_rows"));
  const int pairs = pick_tile(n_img, n_ref, 0.9, 0.6);
  const int64_t tiles = tile_count(n_img, n_ref, pairs);
  SPF_REQUIRE(tiles < (1LL << 31), "spf_argmin_f64: too many tiles");
  const int group_m = (int)tune_get(SPF_TUNE_FP32_GROUP_M, GROUP_M);
  SPF_TILE_DISPATCH(pairs, (k_filter<TL><<<(unsigned)tiles, TL::THREADS, 0, s>>>(
                               w, n_img, n_ref, n_pix, group_m)));
  SPF_TRY(check_launch("k_filter"));
  k_select<<<(unsigned)n_img, 256, 0, s>>>(w, n_ref, n_pix);
  SPF_TRY(check_launch("k_select"));
  k_pairs<<<(unsigned)(4 * sm_count()), CH_THREADS, 0, s>>>(w, d_img, d_ref, n_pix);
  SPF_TRY(check_launch("k_pairs"));
  k_all<<<dim3((unsigned)n_img, (unsigned)(w.parts < 65535 ? w.parts : 65535)), 128, 0, s>>>(w, d_img, d_ref, n_ref, n_pix);
  SPF_TRY(check_launch("k_all"));
  k_best<<<(unsigned)n_img, 128, 0, s>>>(w, ref_offset, d_best_dist, d_best_idx);
  return check_launch("k_best");
}

}  // extern "C"
