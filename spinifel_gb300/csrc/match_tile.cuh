// Register-tiled sums over pixels of image x reference pairs (squared
// differences or products), shared by the FP32 and FP64 distance kernels, and
// the rule that picks a tile.
#pragma once
#include "common.cuh"

namespace spf {

constexpr int TB_K = 16;
constexpr int GROUP_M = 8;

enum class Mode { DIFF, DOT };

// TM x TN pairs by a CTA, RM x RN by a thread (rows in groups of four, so a
// warp's 16-byte shared reads are free of bank conflicts).  Every pair's sum
// is one chain over the pixels in order whatever the tile, so the tile never
// changes a bit of the result.
//
// PF k-steps of both operands are on their way in registers: a 32-pair tile
// has two warps, and with few of them on an SM nothing else hides a step's
// loads (32 x 8,000 pairs of 16,384 pixels: 623 us with one step, 525 with
// four).  MINB CTAs an SM are asked of the compiler for the 128-pair tile's
// argmin (54.0 TFLOP/s against 49.3 with one; its bound of 128 registers then
// spills 124 bytes a thread, which that rate includes).
template <int TM_, int TN_, int RM_, int RN_, int PF_>
struct Tile {
  static constexpr int TM = TM_, TN = TN_, RM = RM_, RN = RN_, PF = PF_;
  static constexpr int MINB = TM == 128 ? 2 : 1;
  static constexpr int NTX = TN / RN, THREADS = NTX * (TM / RM);
  static_assert((RM == 8 || RM == 4) && (RN == 8 || RN == 4) && NTX <= 32, "row groups of four");
  __device__ static __forceinline__ int row(int ty, int i) {
    return ty * 4 + (i & 3) + (TM / 2) * (i >> 2);
  }
  __device__ static __forceinline__ int col(int tx, int j) {
    return tx * 4 + (j & 3) + (TN / 2) * (j >> 2);
  }
};
using Tile128 = Tile<128, 128, 8, 8, 1>;  // 256 threads
using Tile64 = Tile<64, 64, 8, 4, 1>;     // 128 threads
using Tile32 = Tile<32, 32, 4, 4, 4>;     // 64 threads

template <typename T, int ROWS, int THREADS, bool VEC>
struct TileLoader {
  // ROWS x 16 k per tile, N groups of four per thread.  FP32 rows that are
  // 16-byte aligned move as float4 (group g of row r); others element by
  // element with 16 lanes along a row, so that a warp's load touches two
  // rows' 64 bytes and not eight rows four times over (333 x 1,999 pairs of
  // 5,550 pixels: 342 us against 455).
  static constexpr int N = ROWS * 4 / THREADS;
  static_assert(THREADS % 16 == 0, "whole rows of lanes");
  T v[N][4];
  __device__ __forceinline__ void load(const T *__restrict__ base, int64_t n_rows, int64_t ld,
                                       int64_t K, int64_t row0, int64_t k0) {
    const int tid = threadIdx.x;
    if constexpr (VEC) {
#pragma unroll
      for (int i = 0; i < N; ++i) {
        const int idx = tid + i * THREADS;
        const int64_t row = row0 + (idx >> 2);
        const int64_t k = k0 + (idx & 3) * 4;
        const T *p = base + row * ld + k;
        if (row < n_rows && k + 3 < K) {
          const float4 f = __ldg(reinterpret_cast<const float4 *>(p));
          v[i][0] = f.x; v[i][1] = f.y; v[i][2] = f.z; v[i][3] = f.w;
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j) v[i][j] = row < n_rows && k + j < K ? __ldg(p + j) : T(0);
        }
      }
    } else {
      const int64_t k = k0 + (tid & 15);
      const int rows = (int)(n_rows - row0 < ROWS ? n_rows - row0 : ROWS);
      const int r0 = k < K ? tid >> 4 : ROWS;  // past K: no row
      const T *p = base + (row0 + (tid >> 4)) * ld + k;
#pragma unroll
      for (int e = 0; e < 4 * N; ++e) {
        v[e >> 2][e & 3] = r0 + e * (THREADS / 16) < rows ? __ldg(p) : T(0);
        p += (THREADS / 16) * ld;
      }
    }
  }
  __device__ __forceinline__ void store(T (*s)[ROWS + 4]) {
    const int tid = threadIdx.x;
    if constexpr (VEC) {
#pragma unroll
      for (int i = 0; i < N; ++i) {
        const int idx = tid + i * THREADS;
        const int r = idx >> 2, kq = (idx & 3) * 4;
#pragma unroll
        for (int j = 0; j < 4; ++j) s[kq + j][r] = v[i][j];
      }
    } else {
#pragma unroll
      for (int e = 0; e < 4 * N; ++e)
        s[tid & 15][(tid >> 4) + e * (THREADS / 16)] = v[e >> 2][e & 3];
    }
  }
};

__device__ __forceinline__ void tile_coords(int64_t n_img_tiles, int64_t n_ref_tiles,
                                            int group_m, int64_t &mt, int64_t &nt) {
  int64_t bid = blockIdx.x;
  int64_t per_group = (int64_t)group_m * n_ref_tiles;
  int64_t group = bid / per_group;
  int64_t first_m = group * group_m;
  int64_t gm = n_img_tiles - first_m;
  if (gm > group_m) gm = group_m;
  int64_t in = bid % per_group;
  mt = first_m + in % gm;
  nt = in / gm;
}

// acc[i][j] accumulates for image row TL::row(ty, i) and reference row
// TL::col(tx, j) of the tile.
// SUM > 0: the chain is cut every SUM k-steps and the pieces are added up, for
// sums that need a small error bound and not one chain's bits.
template <typename T, Mode MODE, class TL, bool VEC, int SUM>
__device__ __forceinline__ void tile_mainloop(const T *__restrict__ A, int64_t n_a,
                                              const T *__restrict__ B, int64_t n_b, int64_t ld,
                                              int64_t K, int64_t a0, int64_t b0,
                                              T acc[TL::RM][TL::RN],
                                              T (*As)[TB_K][TL::TM + 4],
                                              T (*Bs)[TB_K][TL::TN + 4]) {
  constexpr int RM = TL::RM, RN = TL::RN;
  const int tx = threadIdx.x % TL::NTX;
  const int ty = threadIdx.x / TL::NTX;
#pragma unroll
  for (int i = 0; i < RM; ++i)
#pragma unroll
    for (int j = 0; j < RN; ++j) acc[i][j] = T(0);
  T tot[SUM ? RM : 1][SUM ? RN : 1];
  if constexpr (SUM > 0) {
#pragma unroll
    for (int i = 0; i < RM; ++i)
#pragma unroll
      for (int j = 0; j < RN; ++j) tot[i][j] = T(0);
  }
  // FP64 tiles are bound by the FP64 pipe; element loads need the registers
  constexpr int PF = sizeof(T) == 8 ? 1 : VEC ? TL::PF : TL::PF < 2 ? TL::PF : 2;
  TileLoader<T, TL::TM, TL::THREADS, VEC> la[PF];
  TileLoader<T, TL::TN, TL::THREADS, VEC> lb[PF];
  const int64_t ktiles = (K + TB_K - 1) / TB_K;
  if (ktiles == 0) return;
  // k-step t travels in slot t mod PF (a step past the end loads zeros)
#pragma unroll
  for (int p = 0; p < PF; ++p) {
    la[p].load(A, n_a, ld, K, a0, p * TB_K);
    lb[p].load(B, n_b, ld, K, b0, p * TB_K);
  }
  la[0].store(As[0]);
  lb[0].store(Bs[0]);
  la[0].load(A, n_a, ld, K, a0, PF * TB_K);
  lb[0].load(B, n_b, ld, K, b0, PF * TB_K);
  T fa[2][RM], fb[2][RN];
  auto frag = [&](int f, int cur, int k) {
#pragma unroll
    for (int i = 0; i < RM; ++i) fa[f][i] = As[cur][k][TL::row(ty, i)];
#pragma unroll
    for (int j = 0; j < RN; ++j) fb[f][j] = Bs[cur][k][TL::col(tx, j)];
  };
  __syncthreads();
  for (int64_t kt0 = 0; kt0 < ktiles; kt0 += PF) {
#pragma unroll
    for (int u = 0; u < PF; ++u) {
      const int64_t kt = kt0 + u;
      if (kt >= ktiles) break;
      const int cur = kt & 1;
      const int slot = (u + 1) % PF;  // of step kt + 1
      if (kt + 1 < ktiles) {
        la[slot].store(As[cur ^ 1]);
        lb[slot].store(Bs[cur ^ 1]);
        la[slot].load(A, n_a, ld, K, a0, (kt + 1 + PF) * TB_K);
        lb[slot].load(B, n_b, ld, K, b0, (kt + 1 + PF) * TB_K);
      }
      frag(0, cur, 0);
#pragma unroll
      for (int k = 0; k < TB_K; ++k) {
        // the next pixel's operands are read while this one's FMAs issue
        const int f = k & 1;
        if (k + 1 < TB_K) frag(f ^ 1, cur, k + 1);
        const T *a = fa[f], *b = fb[f];
        if constexpr (sizeof(T) == 4) {
          // two outputs per instruction (packed sub / fma, each lane the same
          // IEEE operation as below, so every output's chain is unchanged)
#pragma unroll
          for (int i = 0; i < RM; ++i)
#pragma unroll
            for (int j = 0; j < RN; j += 2) {
              const float2 ai = make_float2(a[i], a[i]), bj = make_float2(b[j], b[j + 1]);
              const float2 c = make_float2(acc[i][j], acc[i][j + 1]);
              float2 r;
              if constexpr (MODE == Mode::DIFF) {
                const float2 d = fsub2(ai, bj);
                r = ffma2(d, d, c);
              } else {
                r = ffma2(ai, bj, c);
              }
              acc[i][j] = r.x;
              acc[i][j + 1] = r.y;
            }
        } else {
#pragma unroll
          for (int i = 0; i < RM; ++i)
#pragma unroll
            for (int j = 0; j < RN; ++j) {
              if constexpr (MODE == Mode::DIFF) {
                T d = a[i] - b[j];
                acc[i][j] = fma(d, d, acc[i][j]);
              } else {
                acc[i][j] = fma(a[i], b[j], acc[i][j]);
              }
            }
        }
      }
      if constexpr (SUM > 0) {
        if (kt % SUM == SUM - 1 || kt + 1 == ktiles) {
#pragma unroll
          for (int i = 0; i < RM; ++i)
#pragma unroll
            for (int j = 0; j < RN; ++j) {
              tot[i][j] += acc[i][j];
              acc[i][j] = T(0);
            }
        }
      }
      __syncthreads();
    }
  }
  if constexpr (SUM > 0) {
#pragma unroll
    for (int i = 0; i < RM; ++i)
#pragma unroll
      for (int j = 0; j < RN; ++j) acc[i][j] = tot[i][j];
  }
}

template <typename T, Mode MODE, class TL, int SUM = 0>
__device__ __forceinline__ void tile_sums(const T *__restrict__ A, int64_t n_a,
                                          const T *__restrict__ B, int64_t n_b, int64_t ld,
                                          int64_t K, int64_t a0, int64_t b0,
                                          T acc[TL::RM][TL::RN], T (*As)[TB_K][TL::TM + 4],
                                          T (*Bs)[TB_K][TL::TN + 4]) {
  if (sizeof(T) == 4 && ld % 4 == 0 && aligned(A, 16) && aligned(B, 16))
    tile_mainloop<T, MODE, TL, sizeof(T) == 4, SUM>(A, n_a, B, n_b, ld, K, a0, b0, acc, As, Bs);
  else
    tile_mainloop<T, MODE, TL, false, SUM>(A, n_a, B, n_b, ld, K, a0, b0, acc, As, Bs);
}

// Tile of the distance kernels for n_a x n_b pairs: the one whose tiles the
// busiest SM finishes first, at the rates the tiles reach with a full chip
// (128: 54, 64: 47, 32: 30 TFLOP/s).  The 128-pair tile reads shared memory
// least per operation; with few tiles most of the chip would idle under it:
// 333 x 1,999 x 5,550 takes 608 us there and 342 us with 32-pair tiles,
// 500 x 2,000 x 4,096 takes 436 us and, with 64-pair tiles, 266 us (FP64,
// whose tiles have one rate: 35.9 and 17.8 ms); 1,500 x 8,000 x 8,192 takes
// 3.65 ms there, 4.2 ms with 64.
template <int PAIRS>
inline double tile_cost(int64_t n_a, int64_t n_b, double rate) {
  const int64_t t = ((n_a + PAIRS - 1) / PAIRS) * ((n_b + PAIRS - 1) / PAIRS);
  const int64_t sms = sm_count();
  return (double)((t + sms - 1) / sms) * PAIRS * PAIRS / rate;
}
inline int64_t tile_count(int64_t n_a, int64_t n_b, int pairs) {
  return ((n_a + pairs - 1) / pairs) * ((n_b + pairs - 1) / pairs);
}
// 128, 64 or 32
inline int pick_tile(int64_t n_a, int64_t n_b, double rate64, double rate32) {
  const double c128 = tile_cost<128>(n_a, n_b, 1.0), c64 = tile_cost<64>(n_a, n_b, rate64),
               c32 = tile_cost<32>(n_a, n_b, rate32);
  if (c128 <= c64 && c128 <= c32) return 128;
  return c64 <= c32 ? 64 : 32;
}

#define SPF_TILE_DISPATCH(pairs, KERNEL_CALL)                 \
  switch (pairs) {                                            \
    case 128: { using TL = Tile128; KERNEL_CALL; break; }     \
    case 64: { using TL = Tile64; KERNEL_CALL; break; }       \
    default: { using TL = Tile32; KERNEL_CALL; break; }       \
  }

}  // namespace spf
