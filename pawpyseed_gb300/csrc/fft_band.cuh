// The two passes of the band FFT (fft3d, linalg.c:14-45, batched over bands) for the grids that the
// register kernels (fft_fast.cuh) are not compiled for and whose lengths split into two groups
// (fft_two.cuh): every length up to 168 without prime factors above 13 but a few; and in the register
// kernels' order of operations for the lengths of fft_band_reg_order.
//
// Pass A, one CTA per (plane g1, band): the plane's coefficients into a shared tile, the occupied
// rows along the third axis, every column along the second, to H. H keeps the third axis in the order
// the tile has it (two_pos): lanes take neighbouring columns without padding or a table of positions
// (90^3, 90 x 91 values: three CTAs per SM against two with the padding of natural order, 2.23 ms
// against 2.73 for 1,024 bands). Pass B, one CTA per (plane j of
// the second axis, band): the first axis from H into a shared tile, then the plane's sphere points
// to the band's picked row. Rows and columns outside the plane-wave sphere are known to be zero
// and are neither read nor transformed.
#pragma once

#include "bf16split.cuh"
#include "fft_two.cuh"
#include "kernels.h"

#include <algorithm>
#include <initializer_list>

namespace pawpy {

namespace {

// shared memory of a CTA; pass A keeps its masks (m2, m3) in static shared memory beside the tile
constexpr size_t kBandSmemCap = 227 * 1024;
constexpr size_t kPlanesSmemCap = kBandSmemCap - 2 * kTwoMaxRadix * sizeof(uint32_t);

// Threads per CTA at most (chosen per launch, band_threads): with radices up to 10 the steps fit
// in 64 registers.
constexpr int max_threads(int radix) { return radix <= 10 ? 320 : 256; }
constexpr int min_ctas(int radix) { return radix <= 16 ? 3 : 2; }
constexpr int group_max(int a, int b) { return a > b ? a : b; }
template <typename L>
constexpr int len_group() {
  return group_max(L::a, L::b);
}

// row length of pass A's tile: odd (lanes along the rows hit distinct banks)
__host__ __device__ constexpr int planes_ld(int n3) { return n3 | 1; }

// Groups of a length in either order on the host: stage by stage (TwoRadix), or the register kernels'
// (RegLen).
struct BandLen {
  int a = 0, b = 0, ld = 0;
};
inline BandLen band_len(int n, int order) {
  if (order == 1) {
    const RegRadix z = make_reg(n);
    return {z.a, z.b, z.ld};
  }
  const TwoRadix t = make_two(n);
  return {t.a, t.b, two_tw_ld(t.b)};
}
inline int band_group(const BandLen &t) { return t.a > t.b ? t.a : t.b; }

// shared memory: the tile, its lengths' twiddles (16-byte aligned)
__host__ __device__ constexpr int even(int n) { return (n + 1) & ~1; }
inline size_t planes_bytes(const PlaneGeom &g, const BandLen &t2, const BandLen &t3) {
  return sizeof(float2) * (even(g.N2 * planes_ld(g.N3)) + t2.a * t2.ld + t3.a * t3.ld);
}
inline size_t xtile_bytes(const PlaneGeom &g, const BandLen &t1) {
  return sizeof(float2) * (even(g.N1 * g.N3) + t1.a * t1.ld) + sizeof(int) * (size_t)g.N1;
}

__device__ __forceinline__ int wrap_pos(int v, int N) {
  v %= N;
  return v < 0 ? v + N : v;
}

}  // namespace

// L2, L3: the lengths (TwoLen, RegLen); RMAX: the largest group
template <typename L2, typename L3, int RMAX>
__global__ void __launch_bounds__(max_threads(RMAX), min_ctas(RMAX))
    k_band_planes(const float2 *__restrict__ C, int Wpad, const int *__restrict__ pstart,
                  const unsigned short *__restrict__ ppos, PlaneGeom g, TwoRadix r2, TwoRadix r3,
                  const float2 *__restrict__ tw2g, const float2 *__restrict__ tw3g, float2 *__restrict__ H) {
  const L2 t2(r2);
  const L3 t3(r3);
  const int N2 = t2.n, N3 = t3.n, LD = planes_ld(N3);
  extern __shared__ __align__(16) unsigned char smraw[];
  float2 *tile = reinterpret_cast<float2 *>(smraw);
  float2 *tw2 = tile + even(N2 * LD), *tw3 = tw2 + t2.a * t2.tw_ld();
  __shared__ uint32_t m2[kTwoMaxRadix], m3[kTwoMaxRadix];  // occupied elements of each first-step item
  const int p = blockIdx.x, b = blockIdx.y, n2 = g.n2;
  const int s2 = wrap_pos(g.g2min, N2), s3 = wrap_pos(g.g3min, N3);
  auto row_of = [&](int r) { return s2 + r - (s2 + r >= N2 ? N2 : 0); };
  two_twiddles(t2.a * t2.tw_ld(), tw2g, tw2);
  two_twiddles(t3.a * t3.tw_ld(), tw3g, tw3);
  two_masks(t2, s2, n2, m2);
  two_masks(t3, s3, g.n3, m3);
  // the occupied rows whole (their columns outside the sphere stay zero)
  two_items(n2, LD, [&](int r, int c) { tile[row_of(r) * LD + c] = make_float2(0.f, 0.f); });
  __syncthreads();
  const int t0 = pstart[p], cnt = pstart[p + 1] - t0;
  const float2 *cb = C + (long long)b * Wpad + t0;
  for (int t = threadIdx.x; t < cnt; t += blockDim.x) tile[ppos[t0 + t]] = cb[t];
  __syncthreads();
  // third axis, the occupied rows; lanes along the rows (odd LD).
  // Columns outside the occupied range are zero and are not read.
  two_switch<two_fix_a<L3>(), RMAX>(t3.a, [&](auto RR) {
    constexpr int R = decltype(RR)::value;
    two_items(t3.b, n2, [&](int q, int r) {
      float2 *row = tile + row_of(r) * LD + q;
      const uint32_t m = m3[q];
      two_item<L3, R, true>([&](int i) { return (m >> i) & 1u ? row[i * t3.b] : make_float2(0.f, 0.f); },
                        [&](int k, float2 v) { row[k * t3.b] = v; }, nullptr);
    });
  });
  __syncthreads();
  two_switch<two_fix_b<L3>(), RMAX>(t3.b, [&](auto RR) {
    constexpr int R = decltype(RR)::value;
    two_items(t3.a, n2, [&](int q, int r) {
      float2 *row = tile + row_of(r) * LD + q * t3.b;
      two_item<L3, R, false>([&](int i) { return row[i]; }, [&](int k, float2 v) { row[k] = v; },
                         tw3 + q * t3.tw_ld());
    });
  });
  __syncthreads();
  // second axis, every column: lanes along the columns
  two_switch<two_fix_a<L2>(), RMAX>(t2.a, [&](auto RR) {
    constexpr int R = decltype(RR)::value;
    two_items(t2.b, N3, [&](int q, int z) {
      float2 *col = tile + q * LD + z;
      const int es = t2.b * LD;
      const uint32_t m = m2[q];
      two_item<L2, R, true>([&](int i) { return (m >> i) & 1u ? col[i * es] : make_float2(0.f, 0.f); },
                        [&](int k, float2 v) { col[k * es] = v; }, nullptr);
    });
  });
  __syncthreads();
  float2 *out = H + ((long long)b * g.n1 + p) * (N2 * N3);
  two_switch<two_fix_b<L2>(), RMAX>(t2.b, [&](auto RR) {
    constexpr int R = decltype(RR)::value;
    two_items(t2.a, N3, [&](int q, int z) {
      const float2 *col = tile + q * t2.b * LD + z;
      float2 *o = out + q * N3 + z;
      const int os = t2.a * N3;
      two_item<L2, R, false>([&](int i) { return col[i * LD]; }, [&](int k, float2 v) { o[k * os] = v; },
                         tw2 + q * t2.tw_ld());
    });
  });
}

// First-axis transform of plane j of one band (hb: its H rows) into the tile rows two_pos(x) (row
// length N3); the last step's values go through put(tile element, value).
template <int RMAX, typename L1, typename Put>
__device__ __forceinline__ void first_axis_tile(const float2 *__restrict__ hb, const PlaneGeom &g, const L1 &t1,
                                                int N3, const float2 *__restrict__ tw1g, float2 *tw1, float2 *tile,
                                                Put &&put) {
  // H offset of the plane of every first-axis index, -1 for the unoccupied ones
  int *xo = reinterpret_cast<int *>(tw1 + t1.a * t1.tw_ld());
  const int N1 = t1.n, s1 = wrap_pos(g.g1min, N1), pstride = g.N2 * N3;
  two_twiddles(t1.a * t1.tw_ld(), tw1g, tw1);
  for (int x = threadIdx.x; x < N1; x += blockDim.x) {
    const int d = x - s1 + (x < s1 ? N1 : 0);
    xo[x] = d < g.n1 ? d * pstride : -1;
  }
  __syncthreads();
  two_switch<two_fix_a<L1>(), RMAX>(t1.a, [&](auto RR) {
    constexpr int R = decltype(RR)::value;
    two_items(t1.b, N3, [&](int q, int z) {
      float2 *col = tile + q * N3 + z;
      const float2 *hz = hb + z;
      const int es = t1.b * N3, *xq = xo + q;
      two_item<L1, R, true>(
          [&](int i) {
            const int d = xq[i * t1.b];
            return d >= 0 ? hz[d] : make_float2(0.f, 0.f);
          },
          [&](int k, float2 v) { col[k * es] = v; }, nullptr);
    });
  });
  __syncthreads();
  two_switch<two_fix_b<L1>(), RMAX>(t1.b, [&](auto RR) {
    constexpr int R = decltype(RR)::value;
    two_items(t1.a, N3, [&](int q, int z) {
      float2 *col = tile + q * t1.b * N3 + z;
      two_item<L1, R, false>([&](int i) { return col[i * N3]; }, [&](int k, float2 v) { put(col + k * N3, v); },
                         tw1 + q * t1.tw_ld());
    });
  });
  __syncthreads();
}

// FORM 0: complex64 rows; 1: split rows; 2: split rows at Gamma (no phase: the tile is split once
// per grid point, (hi, lo) words in the value's place, and the pick copies words)
// F3 > 0: the third length, fixed
template <typename L1, int F3, int RMAX, int FORM>
__global__ void __launch_bounds__(max_threads(RMAX), min_ctas(RMAX))
    k_band_pick(const float2 *__restrict__ H, PlaneGeom g, TwoRadix r1, const float2 *__restrict__ tw1g,
                const int *__restrict__ plane_first, const uint2 *__restrict__ ent,
                const float2 *__restrict__ phase, float2 *__restrict__ X, long long xstride, long long lo_words) {
  const L1 t1(r1);
  const int N3 = F3 > 0 ? F3 : g.N3;
  extern __shared__ __align__(16) unsigned char smraw[];
  float2 *tile = reinterpret_cast<float2 *>(smraw), *tw1 = tile + even(t1.n * N3);
  const int b = blockIdx.x, j = blockIdx.y;
  const float2 *hb = H + ((long long)b * g.n1 * g.N2 + j) * N3;
  first_axis_tile<RMAX>(hb, g, t1, N3, tw1g, tw1, tile, [&](float2 *dst, float2 v) {
    if constexpr (FORM == 2) {
      uint32_t h, l;
      split_bf16x2(v, h, l);
      *reinterpret_cast<uint2 *>(dst) = make_uint2(h, l);
    } else {
      *dst = v;
    }
  });
  const int pf = plane_first[j], npj = plane_first[j + 1] - pf, nt = blockDim.x;
  constexpr int U = 8;
  const uint2 *en = ent + pf;
  const float2 *ph = phase ? phase + pf : nullptr;
  uint32_t *w0 = reinterpret_cast<uint32_t *>(X) + (long long)b * 16;
  float2 *x0 = X + (long long)b * xstride;
  for (int q0 = threadIdx.x; q0 < npj; q0 += nt * U) {
    uint2 e[U];
    float2 f[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int q = q0 + u * nt;
      if (q < npj) {
        e[u] = __ldg(en + q);
        if (FORM != 2 && ph) f[u] = __ldg(ph + q);
      }
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int q = q0 + u * nt;
      if (q < npj) {
        if constexpr (FORM == 2) {
          const uint2 v = reinterpret_cast<const uint2 *>(tile)[e[u].x];
          w0[e[u].y] = v.x;
          w0[e[u].y + lo_words] = v.y;
        } else {
          const float2 v = ph ? cmul(tile[e[u].x], f[u]) : tile[e[u].x];
          if constexpr (FORM == 1) {
            uint32_t h, l;
            split_bf16x2(v, h, l);
            w0[e[u].y] = h;
            w0[e[u].y + lo_words] = l;
          } else {
            x0[e[u].y] = v;
          }
        }
      }
    }
  }
}

// Pass B writing whole grids, band-tiled (grid_value_index).
template <typename L1, int F3, int RMAX>
__global__ void __launch_bounds__(max_threads(RMAX), min_ctas(RMAX))
    k_band_grid(const float2 *__restrict__ H, PlaneGeom g, TwoRadix r1, int a3, const float2 *__restrict__ tw1g,
                float2 *__restrict__ grid, int b0) {
  const L1 t1(r1);
  const int N1 = t1.n, N3 = F3 > 0 ? F3 : g.N3;
  extern __shared__ __align__(16) unsigned char smraw[];
  float2 *tile = reinterpret_cast<float2 *>(smraw), *tw1 = tile + even(N1 * N3);
  const int b = blockIdx.x, j = blockIdx.y, bb = b0 + b;
  const float2 *hb = H + ((long long)b * g.n1 * g.N2 + j) * N3;
  first_axis_tile<RMAX>(hb, g, t1, N3, tw1g, tw1, tile, [&](float2 *dst, float2 v) { *dst = v; });
  float2 *gb = grid + ((long long)(bb >> 4) * N1 * g.N2 * N3 + (long long)j * N3) * 16 + (bb & 15);
  const int b3 = N3 / a3;
  two_items(N1, N3, [&](int x, int p) {
    const int z = p / b3 + a3 * (p % b3);  // the third-axis index at position p
    gb[((long long)x * g.N2 * N3 + z) * 16] = tile[two_pos(t1, x, t1.b) * N3 + p];
  });
}

// ------------------------------------------------------------------ host side

namespace {

// Lengths (second, third) or (first, third) with kernels of their own (constant strides and groups);
// the cubic grids that the register kernels (fft_fast.cuh) do not cover.
#define PAWPY_BAND_PAIRS(X) \
  X(28, 28) X(30, 30) X(32, 32) X(40, 40) X(42, 42) X(54, 54) X(56, 56) X(70, 70) X(84, 84) X(100, 100) X(108, 108) \
  X(112, 112) X(120, 120)

// Threads of a CTA whose phases have the given numbers of equal items: the count that keeps the
// most threads of an SM busy, counting the idle ones of each phase's last round and the CTAs that
// fit an SM (registers, shared memory, 64 warps).
inline int group_regs(int radix) { return radix <= 10 ? 64 : radix <= 16 ? 80 : 128; }
inline int band_threads(int max_threads, int regs, size_t smem, std::initializer_list<int> items) {
  int best = 128;
  double top = 0;
  for (int t = 96; t <= max_threads; t += 32) {
    const int ctas = std::min({(int)(65536 / (regs * t)), (int)(227 * 1024 / (smem + 1024)), 2048 / t, 24});
    double rounds = 0, work = 0;
    for (int n : items) {
      rounds += ceil_div(n, t);
      work += (double)n / t;
    }
    const double busy = ctas * t * work / rounds;
    if (busy > top * 1.01) top = busy, best = t;
  }
  return best;
}

}  // namespace

}  // namespace pawpy
