// Plain (SIMT) distance kernels: the drop-in for the reference's CUDA KNN
// module and the FP32 distance + argmin that SNM computes with cuBLAS + CUB.
//
// Both operands are row-major with the pixel axis contiguous ("K-major"):
// images [n_img][n_pix] and references [n_ref][n_pix].  A CTA computes a tile
// of (image, reference) pairs, each thread a register tile, K staged through
// shared memory in steps of 16 pixels with register double-buffering.  The
// tile order is grouped (8 image tiles per group) so that CTAs resident at
// the same time share image and reference rows in L2.
#include "common.cuh"
#include "match_tile.cuh"

namespace spf {

// out[d][r] = sum_{p < K} (data[d][p] - ref[r][p])^2
template <typename T, class TL>
__global__ void __launch_bounds__(TL::THREADS) k_knn_eudist(const T *__restrict__ ref,
                                                           const T *__restrict__ data,
                                                           int64_t n_ref, int64_t n_data,
                                                           int64_t ld, int64_t K,
                                                           T *__restrict__ out, int group_m) {
  constexpr int TB_M = TL::TM, TB_N = TL::TN, RM = TL::RM, RN = TL::RN;
  __shared__ __align__(16) T As[2][TB_K][TB_M + 4];
  __shared__ __align__(16) T Bs[2][TB_K][TB_N + 4];
  int64_t n_img_tiles = (n_data + TB_M - 1) / TB_M;
  int64_t n_ref_tiles = (n_ref + TB_N - 1) / TB_N;
  int64_t mt, nt;
  tile_coords(n_img_tiles, n_ref_tiles, group_m, mt, nt);
  T acc[RM][RN];
  tile_sums<T, Mode::DIFF, TL>(data, n_data, ref, n_ref, ld, K, mt * TB_M, nt * TB_N, acc,
                                   As, Bs);
  const int tx = threadIdx.x % TL::NTX;
  const int ty = threadIdx.x / TL::NTX;
#pragma unroll
  for (int i = 0; i < RM; ++i) {
    int64_t d = mt * TB_M + TL::row(ty, i);
    if (d >= n_data) continue;
#pragma unroll
    for (int j = 0; j < RN; ++j) {
      int64_t r = nt * TB_N + TL::col(tx, j);
      if (r < n_ref) out[d * n_ref + r] = acc[i][j];
    }
  }
}

// Running argmin of x2 + s2 - 2 x.s, packed (order key << 32 | index).
template <class TL>
__global__ void __launch_bounds__(TL::THREADS, TL::MINB) k_dist_argmin_f32(
    const float *__restrict__ img, const float *__restrict__ img_sq, int64_t n_img,
    const float *__restrict__ ref, const float *__restrict__ ref_sq, int64_t n_ref, int64_t K,
    int64_t ref_offset, unsigned long long *__restrict__ best, int group_m) {
  constexpr int TB_M = TL::TM, TB_N = TL::TN, RM = TL::RM, RN = TL::RN;
  __shared__ __align__(16) float As[2][TB_K][TB_M + 4];
  __shared__ __align__(16) float Bs[2][TB_K][TB_N + 4];
  int64_t n_img_tiles = (n_img + TB_M - 1) / TB_M;
  int64_t n_ref_tiles = (n_ref + TB_N - 1) / TB_N;
  int64_t mt, nt;
  tile_coords(n_img_tiles, n_ref_tiles, group_m, mt, nt);
  float acc[RM][RN];
  tile_sums<float, Mode::DOT, TL>(img, n_img, ref, n_ref, K, K, mt * TB_M, nt * TB_N, acc,
                                      As, Bs);
  const int tx = threadIdx.x % TL::NTX;
  const int ty = threadIdx.x / TL::NTX;
  float s2[RN];
  int64_t rr[RN];
#pragma unroll
  for (int j = 0; j < RN; ++j) {
    rr[j] = nt * TB_N + TL::col(tx, j);
    s2[j] = rr[j] < n_ref ? ref_sq[rr[j]] : 0.0f;
  }
#pragma unroll
  for (int i = 0; i < RM; ++i) {
    int64_t d = mt * TB_M + TL::row(ty, i);
    float x2 = d < n_img ? img_sq[d] : 0.0f;
    unsigned long long key = ~0ULL;
#pragma unroll
    for (int j = 0; j < RN; ++j) {
      if (rr[j] < n_ref) {
        float dist = __fsub_rn(__fadd_rn(x2, s2[j]), __fmul_rn(2.0f, acc[i][j]));
        unsigned long long k2 =
            ((unsigned long long)float_key(dist) << 32) | (unsigned long long)(rr[j] + ref_offset);
        key = k2 < key ? k2 : key;
      }
    }
    // the NTX threads with this ty hold the other columns of the row
#pragma unroll
    for (int o = TL::NTX / 2; o >= 1; o >>= 1) {
      unsigned long long other = __shfl_xor_sync(0xffffffffu, key, o, TL::NTX);
      key = other < key ? other : key;
    }
    if (tx == 0 && d < n_img && key != ~0ULL) atomicMin(best + d, key);
  }
}

__global__ void k_best_init(unsigned long long *best, int64_t n) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    best[i] = ~0ULL;
}

__global__ void k_best_unpack(const unsigned long long *__restrict__ best, int64_t n,
                              int32_t *__restrict__ idx, float *__restrict__ dist) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    unsigned long long b = best[i];
    if (idx) idx[i] = (b == ~0ULL) ? -1 : (int32_t)(b & 0xffffffffu);
    if (dist) dist[i] = key_float((uint32_t)(b >> 32));
  }
}

// FP64 running argmin over the rows of a distance block [n_img][n_ref]: one
// warp per image; the lowest column wins ties within the block, and the
// running best changes only on a strictly smaller distance (earlier blocks
// hold lower reference indices), as argmin over the whole row would.
__global__ void k_argmin_rows_f64(const double *__restrict__ dist, int64_t n_img, int64_t n_ref,
                                  int64_t ref_offset, double *__restrict__ best_dist,
                                  int64_t *__restrict__ best_idx) {
  const int lane = threadIdx.x & 31;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < n_img;
       i += nwarps) {
    const double *row = dist + i * n_ref;
    double bd = INFINITY;
    int64_t bi = -1;
    for (int64_t r = lane; r < n_ref; r += 32) {
      const double d = row[r];
      if (d < bd) {  // lanes walk their columns in increasing order
        bd = d;
        bi = r;
      }
    }
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) {
      const double od = __shfl_xor_sync(0xffffffffu, bd, o);
      const int64_t oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (oi >= 0 && (bi < 0 || od < bd || (od == bd && oi < bi))) {
        bd = od;
        bi = oi;
      }
    }
    if (lane == 0 && bi >= 0 && (best_idx[i] < 0 || bd < best_dist[i])) {
      best_dist[i] = bd;
      best_idx[i] = bi + ref_offset;
    }
  }
}

__global__ void k_best64_init(double *best_dist, int64_t *best_idx, int64_t n) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    best_dist[i] = INFINITY;
    best_idx[i] = -1;
  }
}

// Sum of squares per row, rounded to FP32, by one warp a row (W = 1) or one
// CTA of W warps.  Each thread keeps its sum as three unevaluated floats
// (error-free products and sums: Dekker 1971, Knuth TAOCP 2, 4.2.2), which loses
// less than FP64 does, and the parts are added in FP64.  FP64 in the loop (a
// conversion and an FMA an element) runs at this chip's FP64 rate: 8,000 rows
// of 16,384 pixels took 530 us, 113 us now.  A row whose sum overflows FP32 or
// is so small that squares are lost to underflow is summed in FP64.
template <int W>
__global__ void __launch_bounds__(256) k_row_sqnorm(const float *__restrict__ x, int64_t n_rows,
                                                    int64_t n_pix, float *__restrict__ out,
                                                    int vec) {
  __shared__ double part[8];
  constexpr int T = 32 * W, RPB = 8 / W;  // threads a row, rows a CTA
  const int t = threadIdx.x % T, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  auto row_sum = [&](double v) {  // over the row's threads, in every one of them
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (W > 1) {
      __syncthreads();
      if (lane == 0) part[warp] = v;
      __syncthreads();
      v = 0.0;
      for (int w = 0; w < W; ++w) v += part[w];
    }
    return v;
  };
  const int64_t step = (int64_t)gridDim.x * RPB;
  for (int64_t r = (int64_t)blockIdx.x * RPB + threadIdx.x / T; r < n_rows; r += step) {
    const float *p = x + r * n_pix;
    float s = 0.0f, c = 0.0f, l = 0.0f;  // the sum, its errors, their errors
    auto exact_add = [](float &to, float v) {  // returns what the rounding lost
      const float u = __fadd_rn(to, v), z = __fsub_rn(u, to);
      const float lost = __fadd_rn(__fsub_rn(to, __fsub_rn(u, z)), __fsub_rn(v, z));
      to = u;
      return lost;
    };
    auto add = [&](float v) {
      const float q = __fmul_rn(v, v), e = __fmaf_rn(v, v, -q);
      const float d = exact_add(s, q);
      l = __fadd_rn(l, exact_add(c, d));
      l = __fadd_rn(l, exact_add(c, e));
    };
    if (vec) {
      const float4 *p4 = reinterpret_cast<const float4 *>(p);
      const int64_t n4 = n_pix >> 2;
      constexpr int U = 4;
      for (int64_t k = t; k < n4; k += T * U) {
        float4 v[U];
#pragma unroll
        for (int u = 0; u < U; ++u)
          v[u] = k + u * T < n4 ? __ldg(p4 + k + u * T) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int u = 0; u < U; ++u) {
          add(v[u].x);
          add(v[u].y);
          add(v[u].z);
          add(v[u].w);
        }
      }
    } else {
      constexpr int U = 8;
      for (int64_t k = t; k < n_pix; k += T * U) {
        float v[U];
#pragma unroll
        for (int u = 0; u < U; ++u) v[u] = k + u * T < n_pix ? __ldg(p + k + u * T) : 0.0f;
#pragma unroll
        for (int u = 0; u < U; ++u) add(v[u]);
      }
    }
    double sum = row_sum((double)s + ((double)c + (double)l));
    if (!(sum > 1e-24 && sum < 3e38)) {  // the same for all threads of the row
      double d = 0.0;
      for (int64_t k = t; k < n_pix; k += T) d = fma((double)p[k], (double)p[k], d);
      sum = row_sum(d);
    }
    if (t == 0) out[r] = (float)sum;
  }
}

// uint16 counts -> f32 (+ bf16) (+ squared norm, 4-norm); one CTA of 256
// threads per frame (a warp per frame left 10,000 frames in just over one
// wave of resident warps, half the time spent in the tail).  Both norms are
// summed exactly in integers and rounded at the end: sum x^2 (at most
// 65535^2 * n_pix, far below 2^64) in one 64-bit sum, sum x^4 as the sums of
// its terms' low and high 32 bits.  (In FP64 the 4-norm's two operations a
// pixel ran at this chip's FP64 rate and bound the kernel: 991 us for 4,096
// frames of 65,536 pixels; 327 us now, 6.6 TB/s.)  Rows move as 16-byte vectors (8 counts) when
// aligned, four loads in flight per thread.
constexpr int INGEST_THREADS = 256;

__global__ void __launch_bounds__(INGEST_THREADS)
    k_ingest_u16(const uint16_t *__restrict__ in, int64_t n_img, int64_t n_pix,
                 float *__restrict__ f32, __nv_bfloat16 *__restrict__ bf, int64_t ld,
                 float *__restrict__ sq, float *__restrict__ n4, int vec) {
  constexpr int NW = INGEST_THREADS / 32;
  __shared__ unsigned long long sh2[NW], sh4l[NW], sh4h[NW];
  const int t = (int)threadIdx.x, lane = t & 31, wid = t >> 5;
  const bool want4 = n4 != nullptr;
  for (int64_t r = blockIdx.x; r < n_img; r += gridDim.x) {
    const uint16_t *p = in + r * n_pix;
    unsigned long long s2 = 0, s4l = 0, s4h = 0;
    auto add4 = [&](unsigned long long v) {
      s4l += (uint32_t)v;
      s4h += v >> 32;
    };
    auto sq32 = [](uint32_t v) { return (unsigned long long)v * v; };
    if (vec) {
      const uint4 *pv = reinterpret_cast<const uint4 *>(p);
      float4 *fv = reinterpret_cast<float4 *>(f32 + r * n_pix);
      uint4 *bv = bf ? reinterpret_cast<uint4 *>(bf + r * ld) : nullptr;
      const int64_t n8 = n_pix / 8;
      constexpr int U = 4;
      for (int64_t k0 = t; k0 < n8; k0 += INGEST_THREADS * U) {
        uint4 raw[U];
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (k0 + INGEST_THREADS * u < n8) raw[u] = __ldg(pv + k0 + INGEST_THREADS * u);
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int64_t k = k0 + INGEST_THREADS * u;
          if (k >= n8) break;
          const uint32_t w[4] = {raw[u].x, raw[u].y, raw[u].z, raw[u].w};
          float v[8];
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            // 2^23 + count, less 2^23: exact, and no integer conversion unit
            v[2 * q] = __uint_as_float(0x4b000000u | (w[q] & 0xffffu)) - 8388608.0f;
            v[2 * q + 1] = __uint_as_float(0x4b000000u | (w[q] >> 16)) - 8388608.0f;
          }
          if (((w[0] | w[1] | w[2] | w[3]) & 0xf000f000u) == 0) {
            // counts below 4,096: eight squares fit in 32 bits, eight fourth
            // powers in 64
            uint32_t a2 = 0;
            unsigned long long a4 = 0;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const uint32_t lo = w[q] & 0xffffu, hi = w[q] >> 16;
              const uint32_t l2 = lo * lo, h2 = hi * hi;
              a2 += l2 + h2;
              if (want4) a4 += sq32(l2) + sq32(h2);
            }
            s2 += a2;
            if (want4) add4(a4);
          } else {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const uint32_t lo = w[q] & 0xffffu, hi = w[q] >> 16;
              s2 += (unsigned long long)(lo * lo) + (unsigned long long)(hi * hi);
              if (want4) {
                add4(sq32(lo * lo));
                add4(sq32(hi * hi));
              }
            }
          }
          fv[2 * k] = make_float4(v[0], v[1], v[2], v[3]);
          fv[2 * k + 1] = make_float4(v[4], v[5], v[6], v[7]);
          if (bv) {
            uint4 o;
            uint32_t *ow = reinterpret_cast<uint32_t *>(&o);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * q], v[2 * q + 1]);
              ow[q] = *reinterpret_cast<uint32_t *>(&h);
            }
            bv[k] = o;
          }
        }
      }
    } else {
      for (int64_t k = t; k < n_pix; k += INGEST_THREADS) {
        const uint32_t c = p[k];
        const float v = (float)c;
        f32[r * n_pix + k] = v;
        if (bf) bf[r * ld + k] = __float2bfloat16_rn(v);
        s2 += (unsigned long long)(c * c);
        if (want4) add4(sq32(c * c));
      }
    }
    if (bf)
      for (int64_t k = n_pix + t; k < ld; k += INGEST_THREADS)
        bf[r * ld + k] = __float2bfloat16_rn(0.0f);
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) {
      s2 += __shfl_xor_sync(0xffffffffu, s2, o);
      if (want4) {
        s4l += __shfl_xor_sync(0xffffffffu, s4l, o);
        s4h += __shfl_xor_sync(0xffffffffu, s4h, o);
      }
    }
    if (lane == 0) {
      sh2[wid] = s2;
      sh4l[wid] = s4l;
      sh4h[wid] = s4h;
    }
    __syncthreads();
    if (t == 0) {
      unsigned long long a2 = 0, al = 0, ah = 0;
      for (int w = 0; w < NW; ++w) {
        a2 += sh2[w];
        al += sh4l[w];
        ah += sh4h[w];
      }
      if (sq) sq[r] = __ull2float_rn(a2);
      if (n4) n4[r] = (float)sqrt(fma((double)ah, 4294967296.0, (double)al));
    }
    __syncthreads();  // the partial sums are reused by the next frame
  }
}

// dst[i] = src[rows[i]] for rows of row_bytes bytes (16-byte chunks when aligned)
__global__ void k_gather_rows16(const uint4 *__restrict__ src, int64_t row_chunks,
                                const int64_t *__restrict__ rows, int64_t n,
                                uint4 *__restrict__ dst) {
  int64_t total = n * row_chunks;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total;
       e += (int64_t)gridDim.x * blockDim.x) {
    int64_t i = e / row_chunks, c = e % row_chunks;
    dst[e] = src[rows[i] * row_chunks + c];
  }
}

__global__ void k_gather_rows1(const unsigned char *__restrict__ src, int64_t row_bytes,
                               const int64_t *__restrict__ rows, int64_t n,
                               unsigned char *__restrict__ dst) {
  int64_t total = n * row_bytes;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total;
       e += (int64_t)gridDim.x * blockDim.x) {
    int64_t i = e / row_bytes, c = e % row_bytes;
    dst[e] = src[rows[i] * row_bytes + c];
  }
}

// dst[rows[i]] = src[i], rows of row_bytes bytes
__global__ void k_scatter_rows1(const unsigned char *__restrict__ src, int64_t row_bytes,
                                const int64_t *__restrict__ rows, int64_t n,
                                unsigned char *__restrict__ dst) {
  int64_t total = n * row_bytes;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total;
       e += (int64_t)gridDim.x * blockDim.x) {
    int64_t i = e / row_bytes, c = e % row_bytes;
    dst[rows[i] * row_bytes + c] = src[e];
  }
}

__global__ void k_f32_to_bf16(const float *__restrict__ src, int64_t n_rows, int64_t n_pix,
                              __nv_bfloat16 *__restrict__ dst, int64_t ld) {
  int64_t total = n_rows * ld;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total;
       i += (int64_t)gridDim.x * blockDim.x) {
    int64_t r = i / ld, p = i % ld;
    dst[i] = __float2bfloat16_rn(p < n_pix ? src[r * n_pix + p] : 0.0f);
  }
}

// k smallest of each row, ascending, ties to the lower index; warp per row.
template <typename T>
__global__ void k_topk(const T *__restrict__ dist, int64_t n_rows, int64_t n_cols, int k,
                       int32_t *__restrict__ out) {
  constexpr int KMAX = 32;
  int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  int lane = threadIdx.x & 31;
  int nwarps = (gridDim.x * blockDim.x) >> 5;
  for (int64_t r = warp; r < n_rows; r += nwarps) {
    T d[KMAX];
    int32_t ix[KMAX];
    int cnt = 0;
    const T *row = dist + r * n_cols;
    for (int64_t c = lane; c < n_cols; c += 32) {
      T v = row[c];
      int32_t ci = (int32_t)c;
      // columns arrive in increasing order per lane, so an equal value never
      // displaces an existing entry (lower index wins)
      if (cnt < k) {
        int pos = cnt++;
        while (pos > 0 && d[pos - 1] > v) {
          d[pos] = d[pos - 1];
          ix[pos] = ix[pos - 1];
          --pos;
        }
        d[pos] = v;
        ix[pos] = ci;
      } else if (v < d[k - 1]) {
        int pos = k - 1;
        while (pos > 0 && d[pos - 1] > v) {
          d[pos] = d[pos - 1];
          ix[pos] = ix[pos - 1];
          --pos;
        }
        d[pos] = v;
        ix[pos] = ci;
      }
    }
    int head = 0;
    for (int t = 0; t < k; ++t) {
      T hv = head < cnt ? d[head] : T(0);
      int32_t hi = head < cnt ? ix[head] : INT32_MAX;
      bool valid = head < cnt;
      // warp min by (valid, value, index)
      T bv = hv;
      int32_t bi = hi;
      bool bvalid = valid;
#pragma unroll
      for (int o = 16; o >= 1; o >>= 1) {
        T ov = __shfl_xor_sync(0xffffffffu, bv, o);
        int32_t oi = __shfl_xor_sync(0xffffffffu, bi, o);
        bool ovalid = __shfl_xor_sync(0xffffffffu, (int)bvalid, o);
        bool take = ovalid && (!bvalid || ov < bv || (ov == bv && oi < bi));
        if (take) {
          bv = ov;
          bi = oi;
          bvalid = true;
        }
      }
      if (valid && hi == bi) ++head;
      if (lane == 0) out[r * k + t] = bvalid ? bi : -1;
    }
  }
}

}  // namespace spf

using namespace spf;

template <typename T>
static int launch_eudist(const T *ref, const T *data, int64_t n_ref, int64_t n_data,
                         int64_t n_pix, int64_t K, T *out, void *stream, const char *name) {
  // FP64 tiles are all bound by the FP64 pipe and run at one rate: at the FP32
  // rates 64 x 20,000 pairs of 512 pixels took 64-pair tiles and 3.37 ms (32-pair
  // ones 2.81), 640 x 640 x 1,000 2.24 (1.70), 2,000 x 8,000 x 256 128-pair ones
  // and 15.7 (14.5)
  const bool fp64 = sizeof(T) == 8;
  const int pairs = pick_tile(n_data, n_ref, fp64 ? 1.0 : 0.9, fp64 ? 1.0 : 0.6);
  const int64_t tiles = tile_count(n_data, n_ref, pairs);
  SPF_REQUIRE(tiles < (1LL << 31), "%s: too many tiles", name);
  const int group_m = (int)tune_get(SPF_TUNE_FP32_GROUP_M, GROUP_M);
  SPF_TILE_DISPATCH(pairs, (k_knn_eudist<T, TL><<<(unsigned)tiles, TL::THREADS, 0,
                                                  as_stream(stream)>>>(
                               ref, data, n_ref, n_data, n_pix, K, out, group_m)));
  return check_launch(name);
}

template <typename T>
static int knn_eudist(const T *ref, const T *data, int64_t n_ref, int64_t n_data, int64_t n_pix,
                      T *out, void *stream, const char *name) {
  SPF_REQUIRE(n_ref >= 0 && n_data >= 0 && n_pix >= 0, "%s: negative size", name);
  if (n_ref == 0 || n_data == 0) return SPF_OK;
  SPF_REQUIRE(ref && data && out, "%s: NULL pointer", name);
  int64_t K = (n_pix / 16) * 16;  // the reference kernel drops the ragged tail
  return launch_eudist<T>(ref, data, n_ref, n_data, n_pix, K, out, stream, name);
}

template <typename T>
static int knn_topk(const T *dist, int64_t n_data, int64_t n_ref, int k, int32_t *idx,
                    void *stream, const char *name) {
  SPF_REQUIRE(n_data >= 0 && n_ref >= 0, "%s: negative size", name);
  SPF_REQUIRE(k >= 1 && k <= 32, "%s: k must be in [1, 32]", name);
  SPF_REQUIRE(k <= n_ref || n_data == 0, "%s: k > n_ref", name);
  if (n_data == 0) return SPF_OK;
  SPF_REQUIRE(dist && idx, "%s: NULL pointer", name);
  int blocks = grid_for(n_data * 32, 256, (int64_t)sm_count() * 32);
  k_topk<T><<<blocks, 256, 0, as_stream(stream)>>>(dist, n_data, n_ref, k, idx);
  return check_launch(name);
}

extern "C" {

int spf_knn_eudist_f32(const float *d_ref, const float *d_data, int64_t n_ref, int64_t n_data,
                       int64_t n_pix, float *d_out, void *stream) {
  return knn_eudist<float>(d_ref, d_data, n_ref, n_data, n_pix, d_out, stream,
                           "spf_knn_eudist_f32");
}

int spf_knn_eudist_f64(const double *d_ref, const double *d_data, int64_t n_ref, int64_t n_data,
                       int64_t n_pix, double *d_out, void *stream) {
  return knn_eudist<double>(d_ref, d_data, n_ref, n_data, n_pix, d_out, stream,
                            "spf_knn_eudist_f64");
}

int spf_knn_topk_f32(const float *d_dist, int64_t n_data, int64_t n_ref, int k, int32_t *d_idx,
                     void *stream) {
  return knn_topk<float>(d_dist, n_data, n_ref, k, d_idx, stream, "spf_knn_topk_f32");
}

int spf_knn_topk_f64(const double *d_dist, int64_t n_data, int64_t n_ref, int k, int32_t *d_idx,
                     void *stream) {
  return knn_topk<double>(d_dist, n_data, n_ref, k, d_idx, stream, "spf_knn_topk_f64");
}

int spf_row_sqnorm_f32(const float *d_x, int64_t n_rows, int64_t n_pix, float *d_out,
                       void *stream) {
  SPF_REQUIRE(n_rows >= 0 && n_pix >= 0, "spf_row_sqnorm_f32: negative size");
  if (n_rows == 0) return SPF_OK;
  SPF_REQUIRE(d_x && d_out, "spf_row_sqnorm_f32: NULL pointer");
  const int vec = n_pix % 4 == 0 && aligned(d_x, 16);
  cudaStream_t s = as_stream(stream);
  // a warp a row for rows too short to give a CTA's threads a few loads each
  if (n_pix <= 2048)
    k_row_sqnorm<1><<<grid_for(n_rows, 8, (int64_t)sm_count() * 32), 256, 0, s>>>(d_x, n_rows, n_pix,
                                                                             d_out, vec);
  else
    k_row_sqnorm<8><<<grid_for(n_rows, 1, (int64_t)sm_count() * 32), 256, 0, s>>>(d_x, n_rows, n_pix,
                                                                             d_out, vec);
  return check_launch("spf_row_sqnorm_f32");
}

int spf_frames_ingest_u16(const uint16_t *d_counts, int64_t n_img, int64_t n_pix, float *d_f32,
                          void *d_bf16, int64_t ld, float *d_sq, float *d_n4, void *stream) {
  SPF_REQUIRE(n_img >= 0 && n_pix >= 0, "spf_frames_ingest_u16: negative size");
  SPF_REQUIRE(!d_bf16 || ld >= n_pix, "spf_frames_ingest_u16: ld < n_pix");
  if (n_img == 0 || n_pix == 0) return SPF_OK;
  SPF_REQUIRE(d_counts && d_f32, "spf_frames_ingest_u16: NULL pointer");
  // one CTA per frame; frames beyond 2^24 are taken by a grid-stride loop
  const int blocks = (int)std::min<int64_t>(n_img, int64_t(1) << 24);
  const int vec = n_pix % 8 == 0 && aligned(d_counts, 16) && aligned(d_f32, 16) &&
                  (!d_bf16 || (aligned(d_bf16, 16) && ld % 8 == 0));
  k_ingest_u16<<<blocks, INGEST_THREADS, 0, as_stream(stream)>>>(
      d_counts, n_img, n_pix, d_f32, reinterpret_cast<__nv_bfloat16 *>(d_bf16), ld, d_sq, d_n4,
      vec);
  return check_launch("spf_frames_ingest_u16");
}

int spf_gather_rows(const void *d_src, int64_t n_src_rows, int64_t row_bytes,
                    const int64_t *d_rows, int64_t n, void *d_dst, void *stream) {
  SPF_REQUIRE(n >= 0 && row_bytes >= 0 && n_src_rows >= 0, "spf_gather_rows: negative size");
  if (n == 0 || row_bytes == 0) return SPF_OK;
  SPF_REQUIRE(d_src && d_rows && d_dst, "spf_gather_rows: NULL pointer");
  cudaStream_t s = as_stream(stream);
  if (row_bytes % 16 == 0 && aligned(d_src, 16) && aligned(d_dst, 16)) {
    int64_t chunks = row_bytes / 16;
    k_gather_rows16<<<grid_for(n * chunks, 256, (int64_t)sm_count() * 16), 256, 0, s>>>(
        reinterpret_cast<const uint4 *>(d_src), chunks, d_rows, n,
        reinterpret_cast<uint4 *>(d_dst));
  } else {
    k_gather_rows1<<<grid_for(n * row_bytes, 256, (int64_t)sm_count() * 16), 256, 0, s>>>(
        reinterpret_cast<const unsigned char *>(d_src), row_bytes, d_rows, n,
        reinterpret_cast<unsigned char *>(d_dst));
  }
  return check_launch("spf_gather_rows");
}

int spf_scatter_rows(const void *d_src, int64_t row_bytes, const int64_t *d_rows, int64_t n,
                     void *d_dst, int64_t n_dst_rows, void *stream) {
  SPF_REQUIRE(n >= 0 && row_bytes >= 0 && n_dst_rows >= 0, "spf_scatter_rows: negative size");
  if (n == 0 || row_bytes == 0) return SPF_OK;
  SPF_REQUIRE(d_src && d_rows && d_dst, "spf_scatter_rows: NULL pointer");
  k_scatter_rows1<<<grid_for(n * row_bytes, 256, (int64_t)sm_count() * 16), 256, 0,
                    as_stream(stream)>>>(reinterpret_cast<const unsigned char *>(d_src), row_bytes,
                                         d_rows, n, reinterpret_cast<unsigned char *>(d_dst));
  return check_launch("spf_scatter_rows");
}

int spf_f32_to_bf16(const float *d_src, int64_t n_rows, int64_t n_pix, void *d_dst, int64_t ld,
                    void *stream) {
  SPF_REQUIRE(n_rows >= 0 && n_pix >= 0 && ld >= n_pix, "spf_f32_to_bf16: bad sizes");
  if (n_rows == 0 || ld == 0) return SPF_OK;
  SPF_REQUIRE(d_src && d_dst, "spf_f32_to_bf16: NULL pointer");
  k_f32_to_bf16<<<grid_for(n_rows * ld, 256, (int64_t)sm_count() * 64), 256, 0,
                  as_stream(stream)>>>(d_src, n_rows, n_pix,
                                       reinterpret_cast<__nv_bfloat16 *>(d_dst), ld);
  return check_launch("spf_f32_to_bf16");
}

int spf_best_init(uint64_t *d_best, int64_t n_img, void *stream) {
  SPF_REQUIRE(n_img >= 0, "spf_best_init: negative size");
  if (n_img == 0) return SPF_OK;
  SPF_REQUIRE(d_best != nullptr, "spf_best_init: NULL pointer");
  k_best_init<<<grid_for(n_img, 256, 4096), 256, 0, as_stream(stream)>>>(
      reinterpret_cast<unsigned long long *>(d_best), n_img);
  return check_launch("spf_best_init");
}

int spf_dist_argmin_f32(const float *d_img, const float *d_img_sq, int64_t n_img,
                        const float *d_ref, const float *d_ref_sq, int64_t n_ref, int64_t n_pix,
                        int64_t ref_offset, uint64_t *d_best, void *stream) {
  SPF_REQUIRE(n_img >= 0 && n_ref >= 0 && n_pix >= 0 && ref_offset >= 0,
              "spf_dist_argmin_f32: negative size");
  if (n_img == 0 || n_ref == 0) return SPF_OK;
  SPF_REQUIRE(d_img && d_img_sq && d_ref && d_ref_sq && d_best,
              "spf_dist_argmin_f32: NULL pointer");
  SPF_REQUIRE(ref_offset + n_ref < (1LL << 32), "spf_dist_argmin_f32: index exceeds 32 bits");
  const int pairs = pick_tile(n_img, n_ref, 0.9, 0.6);
  const int64_t tiles = tile_count(n_img, n_ref, pairs);
  SPF_REQUIRE(tiles < (1LL << 31), "spf_dist_argmin_f32: too many tiles");
  SPF_TILE_DISPATCH(pairs, (k_dist_argmin_f32<TL><<<(unsigned)tiles, TL::THREADS, 0,
                                                    as_stream(stream)>>>(
                               d_img, d_img_sq, n_img, d_ref, d_ref_sq, n_ref, n_pix, ref_offset,
                               reinterpret_cast<unsigned long long *>(d_best),
                               (int)tune_get(SPF_TUNE_FP32_GROUP_M, GROUP_M))));
  return check_launch("spf_dist_argmin_f32");
}

int spf_best_unpack(const uint64_t *d_best, int64_t n_img, int32_t *d_idx, float *d_dist,
                    void *stream) {
  SPF_REQUIRE(n_img >= 0, "spf_best_unpack: negative size");
  if (n_img == 0) return SPF_OK;
  SPF_REQUIRE(d_best != nullptr, "spf_best_unpack: NULL pointer");
  k_best_unpack<<<grid_for(n_img, 256, 4096), 256, 0, as_stream(stream)>>>(
      reinterpret_cast<const unsigned long long *>(d_best), n_img, d_idx, d_dist);
  return check_launch("spf_best_unpack");
}

int spf_dist_argmin_fp32(const float *d_img, const float *d_img_sq, int64_t n_img,
                         const float *d_ref, const float *d_ref_sq, int64_t n_ref, int64_t n_pix,
                         uint64_t *d_best, int32_t *d_idx, float *d_dist, void *stream) {
  SPF_REQUIRE(n_img == 0 || (d_idx && d_dist), "spf_dist_argmin_fp32: NULL output");
  SPF_TRY(spf_best_init(d_best, n_img, stream));
  SPF_TRY(spf_dist_argmin_f32(d_img, d_img_sq, n_img, d_ref, d_ref_sq, n_ref, n_pix, 0, d_best,
                              stream));
  return spf_best_unpack(d_best, n_img, d_idx, d_dist, stream);
}

int spf_dist_f64(const double *d_ref, const double *d_data, int64_t n_ref, int64_t n_data,
                 int64_t n_pix, double *d_out, void *stream) {
  SPF_REQUIRE(n_ref >= 0 && n_data >= 0 && n_pix >= 0, "spf_dist_f64: negative size");
  if (n_ref == 0 || n_data == 0) return SPF_OK;
  SPF_REQUIRE(d_ref && d_data && d_out, "spf_dist_f64: NULL pointer");
  return launch_eudist<double>(d_ref, d_data, n_ref, n_data, n_pix, n_pix, d_out, stream,
                               "spf_dist_f64");
}

int spf_best64_init(double *d_best_dist, int64_t *d_best_idx, int64_t n_img, void *stream) {
  SPF_REQUIRE(n_img >= 0, "spf_best64_init: negative size");
  if (n_img == 0) return SPF_OK;
  SPF_REQUIRE(d_best_dist && d_best_idx, "spf_best64_init: NULL pointer");
  k_best64_init<<<grid_for(n_img, 256, 4096), 256, 0, as_stream(stream)>>>(d_best_dist,
                                                                           d_best_idx, n_img);
  return check_launch("spf_best64_init");
}

int spf_argmin_rows_f64(const double *d_dist, int64_t n_img, int64_t n_ref, int64_t ref_offset,
                        double *d_best_dist, int64_t *d_best_idx, void *stream) {
  SPF_REQUIRE(n_img >= 0 && n_ref >= 0 && ref_offset >= 0, "spf_argmin_rows_f64: negative size");
  if (n_img == 0 || n_ref == 0) return SPF_OK;
  SPF_REQUIRE(d_dist && d_best_dist && d_best_idx, "spf_argmin_rows_f64: NULL pointer");
  k_argmin_rows_f64<<<grid_for(n_img * 32, 256, (int64_t)sm_count() * 16), 256, 0,
                      as_stream(stream)>>>(d_dist, n_img, n_ref, ref_offset, d_best_dist,
                                           d_best_idx);
  return check_launch("spf_argmin_rows_f64");
}

}  // extern "C"
