// Complex overlap contraction on the CUDA cores (FP32), the "plain FP32 GPU
// form" of pseudoprojection (pseudoprojector.c:63-90) batched over every
// defect band: out[n][m] = sum_k conj(A[m][k]) B[n][k] per k-point, with the
// K range made of two segments (plane-wave coefficients, then the augmentation
// columns of the PAW terms), split over CTAs and reduced in a fixed order.
#include <cuda_runtime.h>

#include <type_traits>

#include "kernels.h"

namespace pawpy {

// One output tile per CTA (64 x 64: four warps; 32 x 32: two). A thread holds RM rows (basis bands) x RN
// columns (defect bands); its sums are packed FP32 pairs of two neighbouring rows, so that the four
// multiply-adds of a complex product of two rows are four FFMA2. Chunks of 16 k go from global memory
// through registers into planar shared tiles [k][row] of re and im, double-buffered; a thread's rows
// of one plane are 16-byte loads that the warp shares (one wavefront each).
//
// Bound: shared-memory reads beside the FP32 pipe. Per k a thread of the 64 x 64 tile issues 64 FFMA2 (128 of
// the pipe's cycles) and 6 shared loads; 168 registers leave three CTAs per SM. At 300 x 250 x 23,056 (22
// splits, 291 us, 47 TFLOP/s) the FMA pipe is 65% and the shared-memory path 77% busy, and the warps wait
// mostly for the loads (short scoreboard). The form with scalar multiply-adds and 4 x 4 sums per thread reached
// 32 TFLOP/s there (0.44 ms with its reduction, now 0.297). Every sum keeps its order: k ascending within a
// split, acc_r + a.y b.y + a.x b.x and acc_i - a.y b.x + a.x b.y.
namespace {

constexpr int BK = 16;

// WM x WN warps of 4 x 8 lanes, RM x RN outputs per thread
template <int RM, int RN, int WM, int WN>
struct F32Tile {
  static constexpr int M = WM * 4 * RM, N = WN * 8 * RN, NT = 32 * WM * WN;
};

}  // namespace

template <int RM, int RN, int WM, int WN>
__device__ __forceinline__ void zgemm_f32_tile(const GemmBatch &bt, int z, int sp, int M, int N, int splits,
                                               float2 *__restrict__ ws, int nz) {
  using T = F32Tile<RM, RN, WM, WN>;
  constexpr int TM = T::M, TN = T::N, NT = T::NT;
  __shared__ __align__(16) float As[2][2][BK][TM], Bs[2][2][BK][TN];
  const int m0 = blockIdx.x * TM, n0 = blockIdx.y * TN;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int mt = warp % WM * 4 * RM + (lane & 3) * RM, nt = warp / WM * 8 * RN + (lane >> 2) * RN;
  const int K1 = bt.K1, K12 = bt.K1 + bt.K2;
  const int chunks = (K12 + bt.K3) / BK;
  const int c0 = (int)((long long)chunks * sp / splits), c1 = (int)((long long)chunks * (sp + 1) / splits);
  // loader: lanes along the rows, each thread KA (KB) consecutive k of one row
  constexpr int KA = BK * TM / NT, KB = BK * TN / NT;
  const int ra = tid % TM, ka = tid / TM * KA, rb = tid % TN, kb = tid / TN * KB;
  float4 pa[KA / 2], pb[KB / 2];
  auto load = [&](int c) {
    auto rows = [&](const float2 *base, long long ld, int row, bool ok, float4 *dst, auto cnt) {
      const float4 *p = reinterpret_cast<const float4 *>(base + (long long)row * ld);
#pragma unroll
      for (int i = 0; i < decltype(cnt)::value; i++) dst[i] = ok ? __ldg(p + i) : make_float4(0.f, 0.f, 0.f, 0.f);
    };
    const int k = c * BK;
    const float2 *A, *B;
    long long lda, ldb;
    if (k < K1) {
      A = bt.A1 + k, B = bt.B1 + k, lda = bt.lda1, ldb = bt.ldb1;
    } else if (k < K12) {
      A = bt.A2 + (k - K1), B = bt.B2 + (k - K1), lda = bt.lda2, ldb = bt.ldb2;
    } else {
      A = bt.A3 + (k - K12), B = bt.B3 + (k - K12), lda = bt.lda3, ldb = bt.ldb3;
    }
    rows(A + ka, lda, m0 + ra, m0 + ra < M, pa, std::integral_constant<int, KA / 2>{});
    rows(B + kb, ldb, n0 + rb, n0 + rb < N, pb, std::integral_constant<int, KB / 2>{});
  };
  auto store = [&](int buf) {
#pragma unroll
    for (int i = 0; i < KA / 2; i++) {
      const int k = ka + 2 * i;
      As[buf][0][k][ra] = pa[i].x;
      As[buf][1][k][ra] = pa[i].y;
      As[buf][0][k + 1][ra] = pa[i].z;
      As[buf][1][k + 1][ra] = pa[i].w;
    }
#pragma unroll
    for (int i = 0; i < KB / 2; i++) {
      const int k = kb + 2 * i;
      Bs[buf][0][k][rb] = pb[i].x;
      Bs[buf][1][k][rb] = pb[i].y;
      Bs[buf][0][k + 1][rb] = pb[i].z;
      Bs[buf][1][k + 1][rb] = pb[i].w;
    }
  };
  float2 acc_r[RM / 2][RN], acc_i[RM / 2][RN];
#pragma unroll
  for (int i = 0; i < RM / 2; i++)
#pragma unroll
    for (int j = 0; j < RN; j++) acc_r[i][j] = acc_i[i][j] = make_float2(0.f, 0.f);
  if (c0 < c1) {
    load(c0);
    store(0);
    __syncthreads();
    for (int c = c0; c < c1; c++) {
      const int buf = (c - c0) & 1;
      const bool more = c + 1 < c1;
      if (more) load(c + 1);
#pragma unroll
      for (int kk = 0; kk < BK; kk++) {
        float2 a[2][RM / 2];
        float b[2][RN];
#pragma unroll
        for (int q = 0; q < 2; q++)
#pragma unroll
          for (int i = 0; i < RM; i += 4) {
            const float4 v = *reinterpret_cast<const float4 *>(&As[buf][q][kk][mt + i]);
            a[q][i / 2] = make_float2(v.x, v.y);
            a[q][i / 2 + 1] = make_float2(v.z, v.w);
          }
#pragma unroll
        for (int q = 0; q < 2; q++)
#pragma unroll
          for (int j = 0; j < RN; j += 4) {
            const float4 v = *reinterpret_cast<const float4 *>(&Bs[buf][q][kk][nt + j]);
            b[q][j] = v.x;
            b[q][j + 1] = v.y;
            b[q][j + 2] = v.z;
            b[q][j + 3] = v.w;
          }
#pragma unroll
        for (int j = 0; j < RN; j++) {
          const float2 bx = make_float2(b[0][j], b[0][j]), by = make_float2(b[1][j], b[1][j]),
                       nbx = make_float2(-b[0][j], -b[0][j]);
#pragma unroll
          for (int i = 0; i < RM / 2; i++) {
            // conj(a) b
            acc_r[i][j] = __ffma2_rn(a[0][i], bx, __ffma2_rn(a[1][i], by, acc_r[i][j]));
            acc_i[i][j] = __ffma2_rn(a[0][i], by, __ffma2_rn(a[1][i], nbx, acc_i[i][j]));
          }
        }
      }
      if (more) store(buf ^ 1);
      __syncthreads();
    }
  }
  float2 *out = splits == 1 ? bt.out : ws + ((long long)sp * nz + z) * (long long)N * M;
#pragma unroll
  for (int j = 0; j < RN; j++) {
    const int n = n0 + nt + j;
    if (n >= N) continue;
#pragma unroll
    for (int i = 0; i < RM / 2; i++) {
      const int m = m0 + mt + 2 * i;
      if (m < M) out[(long long)n * M + m] = make_float2(acc_r[i][j].x, acc_i[i][j].x);
      if (m + 1 < M) out[(long long)n * M + m + 1] = make_float2(acc_r[i][j].y, acc_i[i][j].y);
    }
  }
}

template <int RM, int RN, int WM, int WN>
__global__ void __launch_bounds__(32 * WM * WN) k_zgemm_f32(const GemmBatch *__restrict__ batches, int M, int N, int splits,
                                                  float2 *__restrict__ ws, int nz) {
  const int z = blockIdx.z / splits, sp = blockIdx.z % splits;
  const GemmBatch bt = batches[z];
  zgemm_f32_tile<RM, RN, WM, WN>(bt, z, sp, M, N, splits, ws, nz);
}

template <int RM, int RN, int WM, int WN>
__global__ void __launch_bounds__(32 * WM * WN) k_zgemm_f32_one(const GemmBatch bt, int M, int N, int splits,
                                                      float2 *__restrict__ ws) {
  zgemm_f32_tile<RM, RN, WM, WN>(bt, 0, blockIdx.z, M, N, splits, ws, 1);
}

// Sum of the splits' values of one output, in split order; SRU loads in flight (one at a time the loop
// waited for each: 64 splits of a 32 x 32 output took 55 us).
namespace {
constexpr int SRU = 16;
}
__device__ __forceinline__ float2 split_sum(const float2 *__restrict__ w, long long stride, int splits) {
  float2 s = make_float2(0.f, 0.f);
  for (int sp = 0; sp < splits; sp += SRU) {
    float2 v[SRU];
#pragma unroll
    for (int u = 0; u < SRU; u++)
      if (sp + u < splits) v[u] = __ldg(w + (sp + u) * stride);
#pragma unroll
    for (int u = 0; u < SRU; u++)
      if (sp + u < splits) {
        s.x += v[u].x;
        s.y += v[u].y;
      }
  }
  return s;
}

__global__ void k_split_reduce(const GemmBatch *__restrict__ batches, const float2 *__restrict__ ws, int M,
                               int N, int splits, int nz) {
  const int z = blockIdx.y;
  float2 *out = batches[z].out;
  long long MN = (long long)M * N;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < MN; e += (long long)gridDim.x * blockDim.x) {
    float2 s = make_float2(0.f, 0.f);
    for (int sp = 0; sp < splits; sp++) {
      float2 v = ws[((long long)sp * nz + z) * MN + e];
      s.x += v.x;
      s.y += v.y;
    }
    out[e] = s;
  }
}

__global__ void k_split_reduce_wide(const GemmBatch *__restrict__ batches, const float2 *__restrict__ ws, int M,
                                    int N, int splits, int nz) {
  const int z = blockIdx.y;
  const long long MN = (long long)M * N, e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (e < MN) batches[z].out[e] = split_sum(ws + (long long)z * MN + e, (long long)nz * MN, splits);
}

__global__ void k_split_reduce_one(float2 *__restrict__ out, const float2 *__restrict__ ws, int M, int N,
                                   int splits) {
  const long long MN = (long long)M * N, e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (e < MN) out[e] = split_sum(ws + e, MN, splits);
}

namespace {
// 32 x 32 tiles where 64 x 64 ones would be more than half padding
bool small_tiles(int M, int N) {
  return 2LL * ceil_div(M, 32) * ceil_div(N, 32) * 1024 <= (long long)ceil_div(M, 64) * ceil_div(N, 64) * 4096;
}
}  // namespace

void zgemm_f32_one(const GemmBatch &bt, int M, int N, int splits, float2 *ws, cudaStream_t s) {
  if (small_tiles(M, N))
    k_zgemm_f32_one<4, 4, 2, 1><<<dim3(ceil_div(M, 32), ceil_div(N, 32), splits), 64, 0, s>>>(bt, M, N, splits, ws);
  else
    k_zgemm_f32_one<8, 4, 2, 2><<<dim3(ceil_div(M, 64), ceil_div(N, 64), splits), 128, 0, s>>>(bt, M, N, splits, ws);
}
void split_reduce_one(float2 *out, const float2 *ws, int M, int N, int splits, cudaStream_t s) {
  k_split_reduce_one<<<ceil_div((long long)M * N, 128), 128, 0, s>>>(out, ws, M, N, splits);
}

void launch_zgemm_f32(const GemmBatch *batches_dev, int nz, int M, int N, int splits, float2 *workspace) {
  if (nz <= 0 || M <= 0 || N <= 0) return;
  if (splits < 1) splits = 1;
  if (small_tiles(M, N)) {
    dim3 grid(ceil_div(M, 32), ceil_div(N, 32), nz * splits);
    PAWPY_LAUNCH("gemm_f32", (k_zgemm_f32<4, 4, 2, 1><<<grid, 64, 0, stream()>>>(batches_dev, M, N, splits, workspace, nz)));
  } else {
    dim3 grid(ceil_div(M, 64), ceil_div(N, 64), nz * splits);
    PAWPY_LAUNCH("gemm_f32", (k_zgemm_f32<8, 4, 2, 2><<<grid, 128, 0, stream()>>>(batches_dev, M, N, splits, workspace, nz)));
  }
  if (splits > 1) {
    dim3 g2(ceil_div((long long)M * N, 128), nz);
    PAWPY_LAUNCH("gemm_reduce", k_split_reduce_wide<<<g2, 128, 0, stream()>>>(batches_dev, workspace, M, N, splits, nz));
  }
}

}  // namespace pawpy
