// All-electron wavefunctions on a real-space grid (the 'realspace' method and
// the AE densities of density.c:158-310):
//
//   psi(r) = V^-1/2 sum_G C_G exp(i G.r) exp(2 pi i k.r_frac)
//          + sum_sites sum_{n,l,m} <p_nlm|psi> (phi_nl - phit_nl)(|r - R|)/|r - R| Y_lm(r - R)
//            exp(2 pi i k.(R + T))
//
// at every grid point r within wave_grid[last] of a site R (T the lattice
// vector that wraps the box point onto the grid), as realspace_state
// (density.c:245-310) evaluates it. The sphere tables (points, values of
// (phi - phit)/r Y_lm, phases per k-point) are built once per wavefunction and
// grid, on the device in double precision; the grids of a batch of bands come
// from rs_fft.cu, then one pass takes each value times its Bloch factor, adds
// the sphere terms of its cell with the sites in order (the reference adds them
// from parallel threads, so its order is not fixed) and stores the state or
// sums its density.
#include <algorithm>
#include <cuda_runtime.h>

#include "kernels.h"

namespace pawpy {

namespace {

__device__ __forceinline__ void to_cart(const double *f, const double *L, double *o) {
  o[0] = f[0] * L[0] + f[1] * L[3] + f[2] * L[6];
  o[1] = f[0] * L[1] + f[1] * L[4] + f[2] * L[7];
  o[2] = f[0] * L[2] + f[1] * L[5] + f[2] * L[8];
}

// Box point q of slab jb of site s: grid indices (unwrapped) and the displacement
// r - R from the site (box around round(coord N), density.c:269-287); inside the sphere?
__device__ __forceinline__ bool ae_point(const SiteDesc &s, int jb, int q, const double *L, const int *N, int *ijk,
                                         double *path) {
  const int w2 = 2 * s.g[2] + 1;
  ijk[0] = q / w2 - s.g[0] + s.c[0];
  ijk[1] = jb - s.g[1] + s.c[1];
  ijk[2] = q % w2 - s.g[2] + s.c[2];
  const double fr[3] = {(double)ijk[0] / N[0] - s.coord[0], (double)ijk[1] / N[1] - s.coord[1],
                        (double)ijk[2] / N[2] - s.coord[2]};
  to_cart(fr, L, path);
  return sqrt(path[0] * path[0] + path[1] * path[1] + path[2] * path[2]) < s.R0;
}

}  // namespace

__global__ void k_ae_count(const SiteDesc *__restrict__ sites, const int2 *__restrict__ slabs,
                           const double *__restrict__ Lg, const int *__restrict__ Ng, int *__restrict__ counts) {
  __shared__ int total;
  const int2 sl = slabs[blockIdx.x];
  const SiteDesc s = sites[sl.x];
  double L[9];
  const int N[3] = {Ng[0], Ng[1], Ng[2]};
  for (int i = 0; i < 9; i++) L[i] = Lg[i];
  if (threadIdx.x == 0) total = 0;
  __syncthreads();
  const int n = (2 * s.g[0] + 1) * (2 * s.g[2] + 1);
  int c = 0;
  for (int q = threadIdx.x; q < n; q += blockDim.x) {
    int ijk[3];
    double path[3];
    if (ae_point(s, sl.y, q, L, N, ijk, path)) c++;
  }
  atomicAdd(&total, c);
  __syncthreads();
  if (threadIdx.x == 0) counts[blockIdx.x] = total;
}

// One CTA per segment (a non-empty slab): its inside points in (i, k) order, with
// cell = (ii N2 + jj) N3 + kk, the values (phi - phit)(r)/r Y_lm (wave_value2,
// utils.c:522-545: spline on the logarithmic grid, r below the first grid point
// divided by it) and, per k-point, exp(2 pi i k.(R + T)) (density.c:289-300).
__global__ void k_ae_fill(const SiteDesc *__restrict__ sites, const SegFill *__restrict__ segs,
                          const AeSpeciesDev *__restrict__ species, const double *__restrict__ Lg,
                          const int *__restrict__ Ng, const double *__restrict__ kfrac, int nkp, long long npts,
                          int *__restrict__ cell, float2 *__restrict__ val, float2 *__restrict__ phase, int *__restrict__ pt_site) {
  __shared__ int warp_cnt[32];
  __shared__ int base_s;
  const SegFill sg = segs[blockIdx.x];
  const SiteDesc s = sites[sg.site];
  const AeSpeciesDev &sp = species[s.species];
  double L[9];
  const int N[3] = {Ng[0], Ng[1], Ng[2]};
  for (int i = 0; i < 9; i++) L[i] = Lg[i];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  if (threadIdx.x == 0) base_s = 0;
  __syncthreads();
  const int n = (2 * s.g[0] + 1) * (2 * s.g[2] + 1);
  for (int start = 0; start < n; start += blockDim.x) {
    const int q = start + threadIdx.x;
    int ijk[3];
    double t[3];
    const bool in = q < n && ae_point(s, sg.jb, q, L, N, ijk, t);
    const unsigned m = __ballot_sync(0xffffffffu, in);
    if (lane == 0) warp_cnt[wid] = __popc(m);
    __syncthreads();
    int before = 0, chunk = 0;
    for (int w = 0; w < nw; w++) {
      if (w < wid) before += warp_cnt[w];
      chunk += warp_cnt[w];
    }
    const int pos = base_s + before + __popc(m & ((1u << lane) - 1u));
    if (in && pos < sg.npts) {
      int wrapped[3], shift[3];
      for (int a = 0; a < 3; a++) {
        wrapped[a] = ((ijk[a] % N[a]) + N[a]) % N[a];
        shift[a] = (wrapped[a] - ijk[a]) / N[a];  // the lattice vector T (integer division, exact)
      }
      const long long pt = sg.pt_off + pos;
      cell[pt] = (wrapped[0] * N[1] + wrapped[1]) * N[2] + wrapped[2];
      pt_site[pt] = sg.site;
      const double r = sqrt(t[0] * t[0] + t[1] * t[1] + t[2] * t[2]);
      // Y_lm of the displacement: cos(theta) = z / r, exp(i phi) = (x + i y) / rho (phi = 0 on
      // the polar axis and at r = 0), associated Legendre functions by recurrence
      double ct = 1.0, cp = 1.0, sn = 0.0;
      if (r != 0) {
        ct = t[2] / r;
        const double rho = sqrt(t[0] * t[0] + t[1] * t[1]);
        if (rho != 0 && r - fabs(t[2]) != 0) {
          cp = t[0] / rho;
          sn = t[1] / rho;
        }
      }
      const double st = sqrt(fmax(0.0, 1.0 - ct * ct));
      double P[4][4];
      P[0][0] = 1.0;
      for (int mm = 1; mm <= 3; mm++) P[mm][mm] = -(2 * mm - 1) * st * P[mm - 1][mm - 1];
      for (int mm = 0; mm < 3; mm++) P[mm + 1][mm] = (2 * mm + 1) * ct * P[mm][mm];
      P[2][0] = (3.0 * ct * P[1][0] - P[0][0]) / 2.0;
      P[3][0] = (5.0 * ct * P[2][0] - 2.0 * P[1][0]) / 3.0;
      P[3][1] = (5.0 * ct * P[2][1] - 3.0 * P[1][1]) / 2.0;
      double er[4] = {1.0, cp, 0, 0}, ei[4] = {0.0, sn, 0, 0};
      for (int mm = 2; mm <= 3; mm++) {
        er[mm] = er[mm - 1] * cp - ei[mm - 1] * sn;
        ei[mm] = er[mm - 1] * sn + ei[mm - 1] * cp;
      }
      // spline on the logarithmic grid x (wave_interpolate, utils.c:477-489)
      const double x0 = sp.x[0], xl = sp.x[sp.size - 1];
      int ind = 0;
      double rem = 0;
      if (r >= x0 && r <= xl) {
        ind = min((int)(log(r / x0) / sp.logstep), sp.size - 2);
        rem = r - sp.x[ind];
      }
      const double inv_r = 1.0 / (r < x0 ? x0 : r);
      double rad = 0.0;
      int last_f = -1;
      for (int lm = 0; lm < sp.total; lm++) {
        const int l = sp.lm_l[lm], mv = sp.lm_m[lm], fi = sp.lm_f[lm];
        if (fi != last_f) {
          const double *f = sp.f + (long long)fi * sp.size;
          const double *b = sp.spl + (long long)fi * 3 * sp.size;
          if (r > xl)
            rad = 0.0;
          else if (r < x0)
            rad = f[0];
          else
            rad = f[ind] + rem * (b[ind] + rem * (b[sp.size + ind] + rem * b[2 * sp.size + ind]));
          rad *= inv_r;
          last_f = fi;
        }
        const int am = mv < 0 ? -mv : mv;
        const double y = sp.lm_coef[lm] * P[l][am] * rad;
        const double cs = er[am], ss = mv < 0 ? -ei[am] : ei[am];
        val[sg.site_val + (long long)(sg.pt_off - sg.site_pt + pos) * ae_stride(sp.total) + lm] =
            make_float2((float)(y * cs), (float)(y * ss));
      }
      if (sp.total & 1)
        val[sg.site_val + (long long)(sg.pt_off - sg.site_pt + pos) * ae_stride(sp.total) + sp.total] =
            make_float2(0.f, 0.f);
      for (int kq = 0; kq < nkp; kq++) {
        const double *kf = kfrac + 3 * kq;
        double a = 0;
        for (int d = 0; d < 3; d++) a += kf[d] * (s.coord[d] + shift[d]);
        a = 2.0 * (a - rint(a));  // in units of pi, reduced to [-1, 1]
        double sv, cv;
        sincospi(a, &sv, &cv);
        phase[(long long)kq * npts + pt] = make_float2((float)cv, (float)sv);
      }
    }
    __syncthreads();
    if (threadIdx.x == 0) base_s += chunk;
    __syncthreads();
  }
}

void launch_ae_count(const SiteDesc *sites, const int2 *slabs, int nslabs, const double *lattice, const int *fftg,
                     int *counts) {
  if (nslabs <= 0) return;
  PAWPY_LAUNCH("ae_tables", k_ae_count<<<nslabs, 256, 0, stream()>>>(sites, slabs, lattice, fftg, counts));
}

void launch_ae_fill(const SiteDesc *sites, const SegFill *segs, int nseg, const AeSpeciesDev *species,
                    const double *lattice, const int *fftg, const double *kfrac, int nkp, long long npts, int *cell,
                    float2 *val, float2 *phase, int *pt_site) {
  if (nseg <= 0) return;
  PAWPY_LAUNCH("ae_tables", k_ae_fill<<<nseg, 128, 0, stream()>>>(sites, segs, species, lattice, fftg, kfrac, nkp,
                                                                   npts, cell, val, phase, pt_site));
}

// ---- the points of every cell, in point order (site order), as first[cell] .. first[cell + 1)

namespace {
constexpr int SCAN_T = 256, SCAN_V = 16, SCAN_TILE = SCAN_T * SCAN_V;
}

__global__ void k_cell_count(const int *__restrict__ cell, long long npts, int *__restrict__ cnt) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i < npts) atomicAdd(cnt + cell[i], 1);
}

// Exclusive sum over a tile of SCAN_TILE values, in place; the tile's total to sums[block].
__global__ void __launch_bounds__(SCAN_T) k_scan_tiles(int *__restrict__ v, long long n, int *__restrict__ sums) {
  __shared__ int warp_sum[SCAN_T / 32];
  const long long base = blockIdx.x * (long long)SCAN_TILE + threadIdx.x * SCAN_V;
  int x[SCAN_V], t = 0;
#pragma unroll
  for (int i = 0; i < SCAN_V; i++) {
    x[i] = base + i < n ? v[base + i] : 0;
    t += x[i];
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int inc = t;
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += y;
  }
  if (lane == 31) warp_sum[warp] = inc;
  __syncthreads();
  int before = inc - t;
  for (int w = 0; w < warp; w++) before += warp_sum[w];
#pragma unroll
  for (int i = 0; i < SCAN_V; i++) {
    if (base + i < n) v[base + i] = before;
    before += x[i];
  }
  if (threadIdx.x == SCAN_T - 1 && sums) sums[blockIdx.x] = before;
}

__global__ void k_scan_add(int *__restrict__ v, long long n, const int *__restrict__ sums) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i < n) v[i] += sums[i / SCAN_TILE];
}

__global__ void k_cell_fill(const int *__restrict__ cell, const int *__restrict__ pt_site, long long npts,
                            int *__restrict__ cursor, int2 *__restrict__ ent) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i < npts) ent[atomicAdd(cursor + cell[i], 1)] = make_int2((int)i, pt_site[i]);
}

// a cell's few entries into point order
__global__ void k_cell_sort(const int *__restrict__ first, long long ncell, int2 *__restrict__ ent) {
  const long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (c >= ncell) return;
  const int a = first[c], b = first[c + 1];
  for (int i = a + 1; i < b; i++) {
    const int2 e = ent[i];
    int j = i;
    while (j > a && ent[j - 1].x > e.x) {
      ent[j] = ent[j - 1];
      j--;
    }
    ent[j] = e;
  }
}

static void scan_exclusive(int *v, long long n) {
  const long long tiles = (n + SCAN_TILE - 1) / SCAN_TILE;
  DevBuf<int> sums(tiles);
  PAWPY_LAUNCH("ae_tables", k_scan_tiles<<<(unsigned)tiles, SCAN_T, 0, stream()>>>(v, n, sums.p));
  if (tiles > 1) {
    scan_exclusive(sums.p, tiles);
    PAWPY_LAUNCH("ae_tables", k_scan_add<<<ceil_div(n, 256), 256, 0, stream()>>>(v, n, sums.p));
  }
}

void launch_cell_entries(const int *cell, const int *pt_site, long long npts, long long ncell, int *first, int2 *ent) {
  PAWPY_CUDA(cudaMemsetAsync(first, 0, sizeof(int) * (size_t)(ncell + 1), stream()));
  if (npts <= 0) return;
  PAWPY_LAUNCH("ae_tables", k_cell_count<<<ceil_div(npts, 256), 256, 0, stream()>>>(cell, npts, first));
  scan_exclusive(first, ncell + 1);
  DevBuf<int> cursor(ncell);
  PAWPY_CUDA(cudaMemcpyAsync(cursor.p, first, sizeof(int) * (size_t)ncell, cudaMemcpyDeviceToDevice, stream()));
  PAWPY_LAUNCH("ae_tables", k_cell_fill<<<ceil_div(npts, 256), 256, 0, stream()>>>(cell, pt_site, npts, cursor.p, ent));
  PAWPY_LAUNCH("ae_tables", k_cell_sort<<<ceil_div(ncell, 256), 256, 0, stream()>>>(first, ncell, ent));
}

// grid[b][(g1 N2 + g2) N3 + g3] = C[b][t] at the wrapped plane-wave indices (grids zeroed
// before); grid (W / 256, nb)
__global__ void k_scatter_bands(const float2 *__restrict__ C, int Wpad, const int *__restrict__ g, int W, int N1,
                                int N2, int N3, float2 *__restrict__ grid) {
  const int b = blockIdx.y;
  const long long n3d = (long long)N1 * N2 * N3;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < W; t += gridDim.x * blockDim.x) {
    const int g1 = ((g[3 * t] % N1) + N1) % N1, g2 = ((g[3 * t + 1] % N2) + N2) % N2,
              g3 = ((g[3 * t + 2] % N3) + N3) % N3;
    grid[b * n3d + ((long long)g1 * N2 + g2) * N3 + g3] = C[(long long)b * Wpad + t];
  }
}

void launch_scatter_bands(const float2 *C, int Wpad, const int *gsorted, int W, int N1, int N2, int N3,
                          float2 *grid, int nb) {
  if (nb <= 0) return;
  PAWPY_CUDA(cudaMemsetAsync(grid, 0, sizeof(float2) * (size_t)nb * N1 * N2 * N3, stream()));
  if (W <= 0) return;
  dim3 g(ceil_div(W, 256), nb);
  PAWPY_LAUNCH("rs_fft", k_scatter_bands<<<g, 256, 0, stream()>>>(C, Wpad, gsorted, W, N1, N2, N3, grid));
}

// PT[tile][channel][NB/2] = (re b0, re b1, im b0, im b1) of the band pairs of the tile of NB bands (zero
// past nb)
__global__ void k_ae_transpose(const float2 *__restrict__ P, int Pstride, int nb, int NB, float4 *__restrict__ PT) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x, t = blockIdx.y;
  if (c >= Pstride) return;
  for (int i = 0; i < NB; i += 2) {
    const int b = t * NB + i;
    const float2 z = make_float2(0.f, 0.f);
    const float2 u = b < nb ? P[(long long)b * Pstride + c] : z, v = b + 1 < nb ? P[(long long)(b + 1) * Pstride + c] : z;
    PT[((long long)t * Pstride + c) * (NB / 2) + i / 2] = make_float4(u.x, v.x, u.y, v.y);
  }
}

// (c, s) = scale exp(2 pi i k.(i/N1, j/N2, k/N3)) of every cell as pairs of FP32 (hi, lo), 48 bits:
// (c hi, c lo, s hi, s lo); one CTA per row of the third axis
__global__ void k_bloch_table(int N1, int N2, int N3, int x0, double kx, double ky, double kz, double scale,
                              float4 *__restrict__ out) {
  const int ij = blockIdx.x, i = x0 + ij / N2, j = ij % N2;
  const double base = kx * i / N1 + ky * j / N2;
  for (int k = threadIdx.x; k < N3; k += blockDim.x) {
    double a = base + kz * k / N3;
    a = 2.0 * (a - rint(a));
    double sv, cv;
    sincospi(a, &sv, &cv);
    sv *= scale;
    cv *= scale;
    const float ch = (float)cv, sh = (float)sv;
    out[(long long)ij * N3 + k] = make_float4(ch, (float)(cv - ch), sh, (float)(sv - sh));
  }
}

// A sum in double-single form (48 bits): a += hi + lo
__device__ __forceinline__ void ds_add(float2 &a, float hi, float lo) {
  const float u = __fadd_rn(a.x, hi), v = __fsub_rn(u, a.x);
  const float e = __fadd_rn(__fsub_rn(a.x, __fsub_rn(u, v)), __fsub_rn(hi, v));
  a.x = u;
  a.y = __fadd_rn(a.y, __fadd_rn(e, lo));
}

// x c - y s with c and s as (hi, lo) pairs, rounded once to FP32 (but for about one value in 2^20
// that lies within 2^-44 of a rounding boundary); infinities and NaN as in the plain product, whose corrections
// are then not finite
__device__ __forceinline__ float ds_rot(float x, float y, float ch, float cl, float sh, float sl) {
  const float p = __fmul_rn(x, ch), q = __fmul_rn(y, sh);
  const float pe = __fmaf_rn(x, cl, __fmaf_rn(x, ch, -p)), qe = __fmaf_rn(y, sl, __fmaf_rn(y, sh, -q));
  const float d = __fsub_rn(p, q), v = __fsub_rn(d, p);
  const float e = __fsub_rn(__fsub_rn(p, __fsub_rn(d, v)), __fadd_rn(q, v));
  const float r = __fadd_rn(d, __fadd_rn(e, __fsub_rn(pe, qe)));
  return fabsf(r) < INFINITY ? r : d;
}

// psi of the band at place i of its tile, as k_ae_apply evaluates it (pt: the tile's coefficients)
__device__ __forceinline__ float2 ae_value(const AeSpread &c, const float4 *__restrict__ pt, int NP, int i,
                                           const float2 *__restrict__ ph, int cell, float2 u, float4 bl) {
  float ar = 0.f, ai = 0.f;
  const int e1 = c.first[cell + 1];
  for (int e = c.first[cell]; e < e1; e++) {
    const int2 en = c.ent[e];
    const AeSite si = c.sites[en.y];
    const float2 *v = c.val + si.val + (long long)(en.x - si.pt) * ae_stride(si.total);
    const float4 *pp = pt + (long long)si.pcol * NP + i / 2;
    float yr = 0.f, yi = 0.f;
#pragma unroll 1
    for (int q = 0; q < si.total; q++) {
      const float4 a = pp[q * NP];
      const float re = i & 1 ? a.y : a.x, im = i & 1 ? a.w : a.z;
      yr = __fadd_rn(yr, __fmaf_rn(re, v[q].x, __fmul_rn(im, -v[q].y)));
      yi = __fadd_rn(yi, __fmaf_rn(re, v[q].y, __fmul_rn(im, v[q].x)));
    }
    const float2 f = ph[en.x];
    ar = __fadd_rn(ar, __fmaf_rn(yr, f.x, __fmul_rn(yi, -f.y)));
    ai = __fadd_rn(ai, __fmaf_rn(yr, f.y, __fmul_rn(yi, f.x)));
  }
  return make_float2(__fadd_rn(ds_rot(u.x, u.y, bl.x, bl.y, bl.z, bl.w), ar),
                     __fadd_rn(ds_rot(u.y, -u.x, bl.x, bl.y, bl.z, bl.w), ai));
}

// The range in which squares and their products with the weights keep both halves of a double-single value:
// the low half of 2^-90 is a multiple of 2^-138 (denormals end at 2^-149), and 16 bands of 2^100 do not overflow.
constexpr float kDsMin = 0x1p-90f, kDsMax = 0x1p100f;

// psi_b(cell) = scale exp(2 pi i k.r) u_b(cell) + sum over the cell's entries of
//   phase sum_n val_n P_b,n, bands b < nb of the tiles of NB (blockIdx.y); one thread per cell of the slab
// [x0, x1) of the first axis (bloch: the factors by cell).
// MODE 0: rho[cell] += sum_b w_b |psi_b|^2; MODE 1: psi back into the grid; MODE 2: psi to out
// (complex128).
//
// A thread keeps NB bands' sums, so that a table value (8 bytes per point and channel, most of the
// traffic: 300 MB for 64 atoms on 120^3) is read once per NB bands; a point's channels are
// consecutive (two per 16-byte load), and the coefficients of a channel come as 16-byte broadcasts of
// two bands, whose real and imaginary parts are summed as packed FP32 pairs. A warp takes a brick of
// 2 x 4 x 4 cells: its cells lie in the same few spheres, so that the lanes run the same entries
// (32 cells of one row cross two or three sphere boundaries on that grid).
// FP64 runs at two operations per clock and SM here: the Bloch factor (once FP64 sine, cosine and
// product per band and cell, 20 ms of that workload) is a table of double-single factors, applied in
// double-single FP32; densities are summed in double-single over the tile's bands, then in FP64,
// within 1e-13 of the FP64 sum (cells whose squares FP32 pairs do not hold: in FP64).
template <int NB, int MODE>
__global__ void __launch_bounds__(128, NB == 16 ? 4 : 8)
    k_ae_apply(AeSpread c, const float4 *__restrict__ PT, int Pstride, int kq, const float4 *__restrict__ bloch,
               float2 scale, float2 *__restrict__ grid, long long stride, int nb, int x0, int x1, int N2, int N3,
               int ncell, const float2 *__restrict__ w, double *__restrict__ rho, double2 *__restrict__ out) {
  constexpr int NP = NB / 2;  // band pairs
  // brick of the warp: z fastest
  const int bz = (N3 + 3) / 4, by = (N2 + 3) / 4;
  const int brick = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  const int z = brick % bz * 4 + (lane & 3), y = brick / bz % by * 4 + (lane >> 2 & 3),
            x = x0 + brick / (bz * by) * 2 + (lane >> 4);
  if (x >= x1 || y >= N2 || z >= N3) return;
  const int cell = (x * N2 + y) * N3 + z;
  const int b0 = blockIdx.y * NB;
  const float4 *pt = PT + (long long)blockIdx.y * Pstride * NP;
  const float2 *ph = c.phase + (long long)kq * c.npts;
  float2 ar[NP], ai[NP];
#pragma unroll
  for (int i = 0; i < NP; i++) ar[i] = ai[i] = make_float2(0.f, 0.f);
  const int e1 = c.first[cell + 1];
  for (int e = c.first[cell]; e < e1; e++) {
    const int2 en = __ldg(c.ent + e);
    const AeSite si = c.sites[en.y];
    const float4 *v = reinterpret_cast<const float4 *>(c.val + si.val + (long long)(en.x - si.pt) * ae_stride(si.total));
    const float4 *pp = pt + (long long)si.pcol * NP;
    const float2 f = __ldg(ph + en.x);
    float2 yr[NP], yi[NP];
#pragma unroll
    for (int i = 0; i < NP; i++) yr[i] = yi[i] = make_float2(0.f, 0.f);
    // y += P val, each product as fma(P.x, v.x, -(P.y v.y)) and fma(P.x, v.y, P.y v.x)
    auto channel = [&](int q, float vx, float vy) {
      const float2 wx = make_float2(vx, vx), wy = make_float2(vy, vy), nwy = make_float2(-vy, -vy);
#pragma unroll
      for (int i = 0; i < NP; i++) {
        const float4 a = __ldg(pp + q * NP + i);
        const float2 re = make_float2(a.x, a.y), im = make_float2(a.z, a.w);
        yr[i] = __fadd2_rn(yr[i], __ffma2_rn(re, wx, __fmul2_rn(im, nwy)));
        yi[i] = __fadd2_rn(yi[i], __ffma2_rn(re, wy, __fmul2_rn(im, wx)));
      }
    };
    const int T = si.total;
    float4 u = __ldg(v);
    for (int q = 0; q < T; q += 2) {
      const float4 cur = u;
      if (q + 2 < T) u = __ldg(v + q / 2 + 1);
      channel(q, cur.x, cur.y);
      if (q + 1 < T) channel(q + 1, cur.z, cur.w);
    }
    const float2 fx = make_float2(f.x, f.x), fy = make_float2(f.y, f.y), nfy = make_float2(-f.y, -f.y);
#pragma unroll
    for (int i = 0; i < NP; i++) {
      ar[i] = __fadd2_rn(ar[i], __ffma2_rn(yr[i], fx, __fmul2_rn(yi[i], nfy)));
      ai[i] = __fadd2_rn(ai[i], __ffma2_rn(yr[i], fy, __fmul2_rn(yi[i], fx)));
    }
  }
  // (at Gamma the factor is the scale)
  const float4 bl = bloch ? bloch[cell] : make_float4(scale.x, scale.y, 0.f, 0.f);
  float2 acc = make_float2(0.f, 0.f);
  float least = kDsMax, most = kDsMin;
#pragma unroll
  for (int i = 0; i < NB; i++) {
    if (b0 + i >= nb) break;
    float2 *g = grid + (b0 + i) * stride + cell;
    const float2 u = *g;
    const float sr = i & 1 ? ar[i / 2].y : ar[i / 2].x, si = i & 1 ? ai[i / 2].y : ai[i / 2].x;
    const float2 psi = make_float2(__fadd_rn(ds_rot(u.x, u.y, bl.x, bl.y, bl.z, bl.w), sr),
                                   __fadd_rn(ds_rot(u.y, -u.x, bl.x, bl.y, bl.z, bl.w), si));
    if constexpr (MODE == 0) {
      const float2 wb = w[b0 + i];
      const float p = __fmul_rn(psi.x, psi.x), pe = __fmaf_rn(psi.x, psi.x, -p);
      const float r = __fmul_rn(psi.y, psi.y), re = __fmaf_rn(psi.y, psi.y, -r);
      float2 t = make_float2(p, __fadd_rn(pe, re));
      ds_add(t, r, 0.f);
      const float m = __fmul_rn(wb.x, t.x);
      const float me = __fadd_rn(__fmaf_rn(wb.x, t.x, -m), __fadd_rn(__fmul_rn(wb.x, t.y), __fmul_rn(wb.y, t.x)));
      ds_add(acc, m, me);
      least = fminf(least, fminf(t.x, m));
      most = fmaxf(most, fmaxf(t.x, m));
    } else if constexpr (MODE == 1) {
      *g = psi;
    } else {
      out[(long long)(b0 + i) * ncell + cell] = make_double2(psi.x, psi.y);
    }
  }
  if constexpr (MODE == 0) {
    if (least >= kDsMin && most <= kDsMax) {
      rho[cell] += (double)acc.x + (double)acc.y;
      return;
    }
    // a square that FP32 pairs do not hold (or an exact zero): the cell's sum again, in FP64
    double s = rho[cell];
#pragma unroll 1
    for (int i = 0; i < NB && b0 + i < nb; i++) {
      const float2 psi = ae_value(c, pt, NP, i, ph, cell, grid[(b0 + i) * stride + cell], bl);
      s += ((double)w[b0 + i].x + w[b0 + i].y) * ((double)psi.x * psi.x + (double)psi.y * psi.y);
    }
    rho[cell] = s;
  }
}

void launch_bloch_table(const int *N, const BlochSlab &slab, const double *kfrac, double scale, float4 *out) {
  PAWPY_LAUNCH("ae_apply", k_bloch_table<<<slab.nx * N[1], 128, 0, stream()>>>(N[0], N[1], N[2], slab.x0, kfrac[0],
                                                                             kfrac[1], kfrac[2], scale, out));
}

namespace {

template <int MODE>
void ae_apply(const AeSpread &c, const float2 *P, int Pstride, int kq, const BlochSlab &slab, double scale, float2 *grid,
              long long stride, int nb, const int *N, const float2 *w, double *rho, double2 *out) {
  if (nb <= 0 || slab.nx <= 0) return;
  // 16 bands per thread; narrower for a few bands
  const int NB = nb <= 2 ? 2 : nb <= 4 ? 4 : 16, tiles = ceil_div(nb, NB);
  DevBuf<float4> PT((size_t)tiles * std::max(1, Pstride) * NB / 2);
  if (Pstride > 0)
    PAWPY_LAUNCH("ae_apply", k_ae_transpose<<<dim3(ceil_div(Pstride, 128), tiles), 128, 0, stream()>>>(
                                 P, Pstride, nb, NB, PT.p));
  const float hi = (float)scale;
  const float2 sc = make_float2(hi, (float)(scale - hi));
  const long long bricks = (long long)ceil_div(slab.nx, 2) * ceil_div(N[1], 4) * ceil_div(N[2], 4);
  auto fn = NB == 2 ? k_ae_apply<2, MODE> : NB == 4 ? k_ae_apply<4, MODE> : k_ae_apply<16, MODE>;
  const float4 *bloch = slab.p ? slab.p - (long long)slab.x0 * N[1] * N[2] : nullptr;
  // the density sums over the tiles: one launch per tile (each adds to rho)
  const int per = MODE == 0 ? 1 : tiles;
  for (int t = 0; t < tiles; t += per) {
    const int b = t * NB, n = std::min(nb - b, per * NB);
    PAWPY_LAUNCH("ae_apply", fn<<<dim3(ceil_div(bricks, 4), per), 128, 0, stream()>>>(
                                 c, PT.p + (size_t)t * Pstride * NB / 2, Pstride, kq, bloch, sc, grid + b * stride,
                                 stride, n, slab.x0, slab.x0 + slab.nx, N[1], N[2], N[0] * N[1] * N[2],
                                 w ? w + b : nullptr, rho, out));
  }
}

}  // namespace

void launch_ae_density(const AeSpread &c, const float2 *P, int Pstride, int kq, const BlochSlab &slab, double scale,
                       float2 *grid, long long stride, int nb, const int *N, const float2 *w, double *rho) {
  ae_apply<0>(c, P, Pstride, kq, slab, scale, grid, stride, nb, N, w, rho, nullptr);
}
void launch_ae_store(const AeSpread &c, const float2 *P, int Pstride, int kq, const BlochSlab &slab, double scale,
                     float2 *grid, long long stride, int nb, const int *N) {
  ae_apply<1>(c, P, Pstride, kq, slab, scale, grid, stride, nb, N, nullptr, nullptr, nullptr);
}
void launch_ae_states(const AeSpread &c, const float2 *P, int Pstride, int kq, const BlochSlab &slab, double scale,
                      float2 *grid, long long stride, int nb, const int *N, double2 *out) {
  ae_apply<2>(c, P, Pstride, kq, slab, scale, grid, stride, nb, N, nullptr, nullptr, out);
}

// x[i] *= exp(-2 pi i k.(i/N1, j/N2, k/N3)) in double precision (remove_phase)
__global__ void k_remove_phase(double2 *__restrict__ x, int N1, int N2, int N3, double kx, double ky, double kz) {
  const int ij = blockIdx.x;
  const int i = ij / N2, j = ij % N2;
  double2 *row = x + (long long)ij * N3;
  const double base = kx * i / N1 + ky * j / N2;
  for (int k = threadIdx.x; k < N3; k += blockDim.x) {
    double a = base + kz * k / N3;
    a = 2.0 * (a - rint(a));
    double sv, cv;
    sincospi(a, &sv, &cv);
    const double2 v = row[k];
    row[k] = make_double2(v.x * cv + v.y * sv, v.y * cv - v.x * sv);
  }
}

void launch_remove_phase(double2 *x, int N1, int N2, int N3, const double *kfrac) {
  dim3 g(N1 * N2);
  PAWPY_LAUNCH("remove_phase", k_remove_phase<<<g, 128, 0, stream()>>>(x, N1, N2, N3, kfrac[0], kfrac[1], kfrac[2]));
}

}  // namespace pawpy
