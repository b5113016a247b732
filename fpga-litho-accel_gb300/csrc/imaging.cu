// FP32 imaging pipeline: mask -> spectrum window -> SOCS intensity band -> image.
//
// The reference computes (litho.cpp:1318-1451)
//   mskf  = fftshift(FFT2(ifftshift(pad(mask)))) / (Fx*Fy)          FT_r2c_padded
//   tmpImg = sum_k s_k |IFFT_N(embed(K_k * mskf_window))|^2          calcSOCS kernel loop
//   image = crop(roll(C2R_F(zero-pad(R2C_N(tmpImg)/N^2))))           FI + crop
// Only the (2Ny+1)x(2Nx+1) window of mskf around DC reaches the kernels, and the
// intensity is band-limited to |f| <= 2N, so this file computes exactly those
// pieces and nothing else:
//
//   win_fold_kernel: W[v][u] = 1/(FxFy) sum_{y,x} m[y][x] e^{-2 pi i (u x'/Fx + v y'/Fy)}
//                    (x' = x + (Fx-Lx)/2 - Fx/2), imaging_fold.cu.  HBM: one read of
//                    the mask.
//   socs_kernel    : per kernel k, embed K_k*W in an N x N grid, 2-D inverse FFT
//                    (warp-shuffle radix-2, fft_warp.cuh), accumulate s_k|E|^2 in
//                    registers; then a forward FFT of the intensity and the
//                    |f| <= 2N band S[fy][fx] / N^2 is written out.
//   fi_rows_kernel : T[fy][X] = sum_fx S[fy][fx] e^{+2 pi i fx x'/Fx}   (fy >= 0)
//   fi_fold_kernel : image[Y][X] = T0 + 2 sum_{fy>0} Re(e^{2 pi i fy y'/Fy} T[fy][X]),
//                    imaging_fold.cu.  HBM: one write of the image.
// With C2R's Hermitian completion and the two rolls of litho.cpp:934 and
// litho.cpp:700, that is exactly FI's zero-padded interpolation followed by
// crop2DCentered (litho.cpp:164-177, 997-1001).
#include "litho_internal.cuh"
#include "fft_warp.cuh"
#include "fft_lane8.cuh"
#include "tc_common.cuh"

#include <algorithm>

namespace litho {

// ---------------------------------------------------------------------------
// SOCS: K inverse FFTs on the N x N conv grid, intensity accumulation in
// registers, forward FFT of the intensity, band output.  socs_kernel<N> uses the
// warp-shuffle transforms of fft_warp.cuh and serves the 32 x 32 grid; the 64 and
// 128 grids have their own kernels on the lane-group transforms of fft_lane8.cuh.
// The groups' bands are stored last group first.  Kernels come by falling weight, and the
// interpolation rows add the bands in the stored order: the first group's, as large as all the
// others', is rounded once then, and not for each of them (calcSOCS of 512 x 512 with ten groups:
// 2.07e-7 from 64 bits in the mean of twelve masks, and 1.83e-7).
// ---------------------------------------------------------------------------
constexpr int SOCS_THREADS = 256;

template <int N>
__global__ void __launch_bounds__(SOCS_THREADS) socs_kernel(
    const float2* __restrict__ win_part, int nparts, const float* __restrict__ mskf_r,
    const float* __restrict__ mskf_i, int Fx, int Fy, int Nx, int Ny, const float2* __restrict__ krn,
    const float* __restrict__ scales, int nk, int kpg, float2* __restrict__ band_part,
    float* __restrict__ tmpImgp) {
  constexpr int J = N / 32, SG = N + 1, CPW = N / 8;
  const int KX = 2 * Nx + 1, KY = 2 * Ny + 1, KD = KX * KY;
  extern __shared__ __align__(16) float2 sg[];
  // only the KY embedded rows of the conv grid are ever non-zero, and the forward
  // pass keeps the rows fy <= 2Ny (= KY rows): a compact [KY][SG] grid
  float2* grid = sg;             // [KY][SG]
  float2* tw = grid + KY * SG;   // [N/2]
  float2* win = tw + N / 2;      // [KY][KX]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = blockIdx.x, img = blockIdx.y, ngroups = gridDim.x;
  early_next();

  for (int e = tid; e < N / 2; e += SOCS_THREADS) {
    float s, c;
    sincospif(2.0f * (float)e / (float)N, &s, &c);
    tw[e] = make_float2(c, -s);
  }
  early_wait(win_part);
  for (int idx = tid; idx < KD; idx += SOCS_THREADS) {
    const int ky = idx / KX, kx = idx - ky * KX;
    const int v = ky - Ny, u = kx - Nx;
    float2 w;
    if (mskf_r != nullptr) {
      const size_t off = (size_t)img * Fx * Fy + (size_t)(Fy / 2 + v) * Fx + (Fx / 2 + u);
      w = make_float2(mskf_r[off], mskf_i[off]);
    } else {
      const bool neg = u < 0;
      const int vv = neg ? -v : v, uu = neg ? -u : u;
      const float2* P = win_part + (size_t)img * nparts * KY * (Nx + 1) + (size_t)(vv + Ny) * (Nx + 1) + uu;
      const float2 t = sum_strided(P, (size_t)KY * (Nx + 1), nparts);
      w = make_float2(t.x, neg ? -t.y : t.y);
    }
    win[idx] = w;
  }
  __syncthreads();

  const int ex = (N - KX) / 2, ey = (N - KY) / 2;
  float acc[CPW][J];
#pragma unroll
  for (int m = 0; m < CPW; ++m)
#pragma unroll
    for (int j = 0; j < J; ++j) acc[m][j] = 0.f;

  const int k0 = g * kpg, k1 = min(nk, k0 + kpg);
  for (int k = k0; k < k1; ++k) {
    const float2* K = krn + (size_t)k * KD;
    const float lam = scales[k];
    for (int ky = warp; ky < KY; ky += 8) {
      float2 x[J];
#pragma unroll
      for (int j = 0; j < J; ++j) {
        const int kx = lane + 32 * j - ex;
        x[j] = (kx >= 0 && kx < KX) ? cmul(K[ky * KX + kx], win[ky * KX + kx]) : make_float2(0.f, 0.f);
      }
      warp_fft_dif<N, true>(x, tw, lane);
#pragma unroll
      for (int j = 0; j < J; ++j) grid[ky * SG + lane + 32 * j] = x[j];
    }
    __syncthreads();
#pragma unroll
    for (int m = 0; m < CPW; ++m) {
      const int c = warp + 8 * m;
      float2 x[J];
#pragma unroll
      for (int j = 0; j < J; ++j) {
        const int y = lane + 32 * j;  // rows outside the embedded band are zero
        x[j] = (unsigned)(y - ey) < (unsigned)KY ? grid[(y - ey) * SG + c] : make_float2(0.f, 0.f);
      }
      warp_fft_dif<N, true>(x, tw, lane);
#pragma unroll
      for (int j = 0; j < J; ++j) acc[m][j] = fmaf(lam, fmaf(x[j].x, x[j].x, x[j].y * x[j].y), acc[m][j]);
    }
    __syncthreads();
  }

  if (tmpImgp != nullptr) {
    // litho.cpp:934 myShift(tmpImg -> tmpImgp, fftshift); positions are bit-reversed
    float* T = tmpImgp + ((size_t)img * gridDim.x + g) * N * N;
#pragma unroll
    for (int m = 0; m < CPW; ++m) {
      const int xs = bitrev<N>(warp + 8 * m);
#pragma unroll
      for (int j = 0; j < J; ++j) {
        const int ys = bitrev<N>(lane + 32 * j);
        T[((ys + N / 2) & (N - 1)) * N + ((xs + N / 2) & (N - 1))] = acc[m][j];
      }
    }
  }

  // forward transform of the intensity: columns (DIT, bit-reversed in -> natural out)
#pragma unroll
  for (int m = 0; m < CPW; ++m) {
    const int c = warp + 8 * m;
    float2 x[J];
#pragma unroll
    for (int j = 0; j < J; ++j) x[j] = make_float2(acc[m][j], 0.f);
    warp_fft_dit<N, false>(x, tw, lane);
#pragma unroll
    for (int j = 0; j < J; ++j) {
      const int fy = lane + 32 * j;
      if (fy <= 2 * Ny) grid[fy * SG + c] = x[j];
    }
  }
  __syncthreads();
  const int BW = 4 * Nx + 1;
  const float inv = 1.0f / ((float)N * (float)N);
  float2* band = band_part + ((size_t)img * ngroups + (ngroups - 1 - g)) * KY * BW;
  for (int fy = warp; fy <= 2 * Ny; fy += 8) {
    float2 x[J];
#pragma unroll
    for (int j = 0; j < J; ++j) x[j] = grid[fy * SG + lane + 32 * j];
    warp_fft_dit<N, false>(x, tw, lane);
#pragma unroll
    for (int j = 0; j < J; ++j) {
      const int fx = lane + 32 * j;
      int d = 1 << 30;
      if (fx <= 2 * Nx) d = fx;
      else if (fx >= N - 2 * Nx) d = fx - N;
      if (d != (1 << 30)) band[fy * BW + d + 2 * Nx] = cscale(x[j], inv);
    }
  }
}

// SOCS on the 64 x 64 conv grid with the eight-lane 64-point FFTs of
// fft_lane8.cuh: four transforms per warp, natural order throughout.  Same
// arguments, grid and output as socs_kernel<64>.
//   rows     : row ky = 8 q + warp of the embedded kernel * window product
//              (q = lane group); 2Ny + 1 <= 31 rows is one round
//   columns  : column c = warp + 8 (q + 4 m), m = 0, 1; only the embedded rows
//              [ey, ey + 2Ny] are read (the others are zero), so the grid is
//              never cleared; |E|^2 accumulates in registers at (t + 8 k2, c)
//   intensity: forward column transforms of the real intensity, rows fy <= 2Ny
//              kept, then forward row transforms of those rows -> band
// |E|^2 does not depend on where the kernel sits in the grid (a shift is a
// unimodular phase on E); the embedding is the centred one of socs_kernel.
// ---------------------------------------------------------------------------
constexpr int S64_SG = 65;  // grid row stride (float2): columns of a warp's groups 16 banks apart

size_t socs64_smem_bytes(int KD) {
  return ((size_t)64 * S64_SG + 32 + (size_t)(SOCS_THREADS / 32) * 4 * L8_SCR + KD) * sizeof(float2);
}

__global__ void __launch_bounds__(SOCS_THREADS) socs64_kernel(
    const float2* __restrict__ win_part, int nparts, const float* __restrict__ mskf_r,
    const float* __restrict__ mskf_i, int Fx, int Fy, int Nx, int Ny, const float2* __restrict__ krn,
    const float* __restrict__ scales, int nk, int kpg, float2* __restrict__ band_part,
    float* __restrict__ tmpImgp) {
  constexpr int N = 64, SG = S64_SG, NW = SOCS_THREADS / 32;
  extern __shared__ __align__(16) float2 sg[];
  float2* grid = sg;                  // [N][SG]
  float2* tw = grid + N * SG;         // [N/2]
  float2* scr = tw + N / 2;           // [NW][4][L8_SCR]
  float2* win = scr + NW * 4 * L8_SCR;  // [KY][KX]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int q = lane >> 3, t = lane & 7;
  float2* my_scr = scr + (warp * 4 + q) * L8_SCR;
  const int g = blockIdx.x, img = blockIdx.y, ngroups = gridDim.x;
  early_next();
  const int KX = 2 * Nx + 1, KY = 2 * Ny + 1, KD = KX * KY;

  for (int e = tid; e < N / 2; e += SOCS_THREADS) {
    float s, c;
    sincospif(2.0f * (float)e / (float)N, &s, &c);
    tw[e] = make_float2(c, -s);
  }
  early_wait(win_part);
  for (int idx = tid; idx < KD; idx += SOCS_THREADS) {
    const int ky = idx / KX, kx = idx - ky * KX;
    const int v = ky - Ny, u = kx - Nx;
    float2 w;
    if (mskf_r != nullptr) {
      const size_t off = (size_t)img * Fx * Fy + (size_t)(Fy / 2 + v) * Fx + (Fx / 2 + u);
      w = make_float2(mskf_r[off], mskf_i[off]);
    } else {
      const bool neg = u < 0;
      const int vv = neg ? -v : v, uu = neg ? -u : u;
      const float2* P = win_part + (size_t)img * nparts * KY * (Nx + 1) + (size_t)(vv + Ny) * (Nx + 1) + uu;
      const float2 s = sum_strided(P, (size_t)KY * (Nx + 1), nparts);
      w = make_float2(s.x, neg ? -s.y : s.y);
    }
    win[idx] = w;
  }
  __syncthreads();
  float2 w64[8];
  lane8_twiddles(w64, tw, t);

  const int ex = (N - KX) / 2, ey = (N - KY) / 2;
  float acc[2][8];
#pragma unroll
  for (int m = 0; m < 2; ++m)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[m][j] = 0.f;

  const int k0 = g * kpg, k1 = min(nk, k0 + kpg);
  for (int k = k0; k < k1; ++k) {
    const float2* K = krn + (size_t)k * KD;
    const float lam = scales[k];
    {
      const int ky = 8 * q + warp;
      const bool act = ky < KY;
      float2 x[8];
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        const int kx = t + 8 * r - ex;
        x[r] = (act && kx >= 0 && kx < KX) ? cmul(K[ky * KX + kx], win[ky * KX + kx]) : make_float2(0.f, 0.f);
      }
      fft64_lane8<true>(x, w64, my_scr, t);
      if (act) {
#pragma unroll
        for (int j = 0; j < 8; ++j) grid[(ey + ky) * SG + t + 8 * j] = x[j];
      }
    }
    __syncthreads();
#pragma unroll
    for (int m = 0; m < 2; ++m) {
      const int c = warp + 8 * (q + 4 * m);
      float2 x[8];
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        const int y = t + 8 * r;
        x[r] = (unsigned)(y - ey) < (unsigned)KY ? grid[y * SG + c] : make_float2(0.f, 0.f);
      }
      fft64_lane8<true>(x, w64, my_scr, t);
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[m][j] = fmaf(lam, fmaf(x[j].x, x[j].x, x[j].y * x[j].y), acc[m][j]);
    }
    __syncthreads();
  }

  if (tmpImgp != nullptr) {
    // litho.cpp:934 myShift(tmpImg -> tmpImgp, fftshift)
    float* T = tmpImgp + ((size_t)img * gridDim.x + g) * N * N;
#pragma unroll
    for (int m = 0; m < 2; ++m) {
      const int c = warp + 8 * (q + 4 * m);
#pragma unroll
      for (int j = 0; j < 8; ++j) T[((t + 8 * j + N / 2) & (N - 1)) * N + ((c + N / 2) & (N - 1))] = acc[m][j];
    }
  }

  // forward transform of the intensity: columns, then the rows fy <= 2Ny
#pragma unroll
  for (int m = 0; m < 2; ++m) {
    const int c = warp + 8 * (q + 4 * m);
    float2 x[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) x[r] = make_float2(acc[m][r], 0.f);
    fft64_lane8<false>(x, w64, my_scr, t);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int fy = t + 8 * j;
      if (fy <= 2 * Ny) grid[fy * SG + c] = x[j];
    }
  }
  __syncthreads();
  const int BW = 4 * Nx + 1;
  const float inv = 1.0f / ((float)N * (float)N);
  float2* band = band_part + ((size_t)img * ngroups + (ngroups - 1 - g)) * KY * BW;
  {
    const int fy = 8 * q + warp;
    const bool act = fy <= 2 * Ny;
    float2 x[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) x[r] = act ? grid[fy * SG + t + 8 * r] : make_float2(0.f, 0.f);
    fft64_lane8<false>(x, w64, my_scr, t);
    if (act) {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int fx = t + 8 * j;
        int d = 1 << 30;
        if (fx <= 2 * Nx) d = fx;
        else if (fx >= N - 2 * Nx) d = fx - N;
        if (d != (1 << 30)) band[fy * BW + d + 2 * Nx] = cscale(x[j], inv);
      }
    }
  }
}

// SOCS on the 128 x 128 conv grid with the sixteen-lane 128-point FFTs of
// fft_lane8.cuh (two transforms per warp), 512 threads so that each lane keeps
// four columns' intensities in registers.  Same arguments, grid and output as
// socs_kernel<128>.  Lane (t, h, slot): t = lane & 7, h = (lane >> 3) & 1,
// slot = lane >> 4; transform slot sl = 16 slot + warp of a round (32 per round).
//   rows     : row ky = 32 r + sl of the embedded product, read at columns
//              t + 8i + 64h (inverse, DIF) and stored at columns 2t + h + 16i
//   columns  : column c = 32 m + sl, m = 0..3, read at rows t + 8i + 64h of the
//              compact grid (only the 2Ny + 1 embedded rows exist); |E|^2 lands
//              at rows 2t + h + 16i
//   intensity: forward column transforms (DIT) take that layout and give
//              fy = t + 8i + 64h, rows fy <= 2Ny kept; forward row transforms read
//              columns 2t + h + 16i and give fx = t + 8i + 64h -> band
// ---------------------------------------------------------------------------
constexpr int S128_SG = 129;       // compact grid row stride (float2)
constexpr int S128_THREADS = 512;

size_t socs128_smem_bytes(int KY, int KD) {
  return ((size_t)KY * S128_SG + 64 + 32 + (size_t)(S128_THREADS / 32) * 4 * L8_SCR + KD) * sizeof(float2);
}

__global__ void __launch_bounds__(S128_THREADS) socs128_kernel(
    const float2* __restrict__ win_part, int nparts, const float* __restrict__ mskf_r,
    const float* __restrict__ mskf_i, int Fx, int Fy, int Nx, int Ny, const float2* __restrict__ krn,
    const float* __restrict__ scales, int nk, int kpg, float2* __restrict__ band_part,
    float* __restrict__ tmpImgp) {
  constexpr int N = 128, SG = S128_SG, NW = S128_THREADS / 32;
  const int KX = 2 * Nx + 1, KY = 2 * Ny + 1, KD = KX * KY;
  extern __shared__ __align__(16) float2 sg[];
  float2* grid = sg;                     // [KY][SG]
  float2* tw128 = grid + KY * SG;        // [64]
  float2* tw64 = tw128 + 64;             // [32]
  float2* scr = tw64 + 32;               // [NW][4][L8_SCR]
  float2* win = scr + NW * 4 * L8_SCR;   // [KY][KX]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int t = lane & 7, h = (lane >> 3) & 1, sl = 16 * (lane >> 4) + warp;
  float2* my_scr = scr + (warp * 4 + (lane >> 3)) * L8_SCR;
  const int g = blockIdx.x, img = blockIdx.y, ngroups = gridDim.x;
  early_next();

  for (int e = tid; e < 64; e += S128_THREADS) {
    float sn, cs;
    sincospif((float)e / 64.0f, &sn, &cs);  // W128^e = exp(-2 pi i e / 128)
    tw128[e] = make_float2(cs, -sn);
    if (e < 32) {
      sincospif((float)e / 32.0f, &sn, &cs);
      tw64[e] = make_float2(cs, -sn);
    }
  }
  early_wait(win_part);
  for (int idx = tid; idx < KD; idx += S128_THREADS) {
    const int ky = idx / KX, kx = idx - ky * KX;
    const int v = ky - Ny, u = kx - Nx;
    float2 w;
    if (mskf_r != nullptr) {
      const size_t off = (size_t)img * Fx * Fy + (size_t)(Fy / 2 + v) * Fx + (Fx / 2 + u);
      w = make_float2(mskf_r[off], mskf_i[off]);
    } else {
      const bool neg = u < 0;
      const int vv = neg ? -v : v, uu = neg ? -u : u;
      const float2* P = win_part + (size_t)img * nparts * KY * (Nx + 1) + (size_t)(vv + Ny) * (Nx + 1) + uu;
      const float2 sm = sum_strided(P, (size_t)KY * (Nx + 1), nparts);
      w = make_float2(sm.x, neg ? -sm.y : sm.y);
    }
    win[idx] = w;
  }
  __syncthreads();
  float2 w64[8];
  lane8_twiddles(w64, tw64, t);

  const int ex = (N - KX) / 2, ey = (N - KY) / 2;
  float acc[4][8];
#pragma unroll
  for (int m = 0; m < 4; ++m)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[m][j] = 0.f;

  const int k0 = g * kpg, k1 = min(nk, k0 + kpg);
  for (int k = k0; k < k1; ++k) {
    const float2* K = krn + (size_t)k * KD;
    const float lam = scales[k];
    for (int r0 = 0; r0 < KY; r0 += 32) {  // uniform bound: every lane takes every round
      const int ky = r0 + sl;
      const bool act = ky < KY;
      float2 x[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int kx = t + 8 * i + 64 * h - ex;
        x[i] = (act && kx >= 0 && kx < KX) ? cmul(K[ky * KX + kx], win[ky * KX + kx]) : make_float2(0.f, 0.f);
      }
      fft128_inv_dif(x, w64, tw128, my_scr, t, h);
      if (act) {
#pragma unroll
        for (int i = 0; i < 8; ++i) grid[ky * SG + 2 * t + h + 16 * i] = x[i];
      }
    }
    __syncthreads();
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      const int c = 32 * m + sl;
      float2 x[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int y = t + 8 * i + 64 * h;
        x[i] = (unsigned)(y - ey) < (unsigned)KY ? grid[(y - ey) * SG + c] : make_float2(0.f, 0.f);
      }
      fft128_inv_dif(x, w64, tw128, my_scr, t, h);
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[m][i] = fmaf(lam, fmaf(x[i].x, x[i].x, x[i].y * x[i].y), acc[m][i]);
    }
    __syncthreads();
  }

  if (tmpImgp != nullptr) {
    // litho.cpp:934 myShift(tmpImg -> tmpImgp, fftshift)
    float* T = tmpImgp + ((size_t)img * gridDim.x + g) * N * N;
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      const int c = 32 * m + sl;
#pragma unroll
      for (int i = 0; i < 8; ++i)
        T[((2 * t + h + 16 * i + N / 2) & (N - 1)) * N + ((c + N / 2) & (N - 1))] = acc[m][i];
    }
  }

  // forward transform of the intensity: columns, then the rows fy <= 2Ny
#pragma unroll
  for (int m = 0; m < 4; ++m) {
    const int c = 32 * m + sl;
    float2 x[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) x[i] = make_float2(acc[m][i], 0.f);
    fft128_fwd_dit(x, w64, tw128, my_scr, t, h);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int fy = t + 8 * i + 64 * h;
      if (fy <= 2 * Ny) grid[fy * SG + c] = x[i];
    }
  }
  __syncthreads();
  const int BW = 4 * Nx + 1;
  const float inv = 1.0f / ((float)N * (float)N);
  float2* band = band_part + ((size_t)img * ngroups + (ngroups - 1 - g)) * KY * BW;
  for (int r0 = 0; r0 < KY; r0 += 32) {
    const int fy = r0 + sl;
    const bool act = fy <= 2 * Ny;
    float2 x[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) x[i] = act ? grid[fy * SG + 2 * t + h + 16 * i] : make_float2(0.f, 0.f);
    fft128_fwd_dit(x, w64, tw128, my_scr, t, h);
    if (act) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int fx = t + 8 * i + 64 * h;
        int d = 1 << 30;
        if (fx <= 2 * Nx) d = fx;
        else if (fx >= N - 2 * Nx) d = fx - N;
        if (d != (1 << 30)) band[fy * BW + d + 2 * Nx] = cscale(x[i], inv);
      }
    }
  }
}

// ---------------------------------------------------------------------------
// FI, step 1: T[fy][X] = sum_fx S[fy][fx] e^{+2 pi i fx x'/Fx} for fy = 0..2Ny
// (T[-fy] = conj(T[fy]) because the intensity is real), x' = X + (Fx-Lx)/2 - Fx/2.
// The band, summed over its kernel-group partials in a fixed order, sits in shared
// memory pre-combined as C[fy][d] = (Re(p+q), -Im(p-q), Im(p+q), Re(p-q)) for
// p = S[fy][d], q = S[fy][-d].  With t = e^{+2 pi i d x'/Fx},
//   T(x') = S0 + U + V,  T(-x') = S0 + U - V,
//   U = sum_{d>0} (p+q) Re t,  V = sum_{d>0} i (p-q) Im t,
// so one thread serves a column with x' < 0 and its mirror -x': its packed
// (f32x2) FMAs keep the cos and sin halves apart, and one broadcast shared load
// and two packed FMAs per (fy, d) give both columns.  The columns with x' < 0
// are X in [0, nb), nb = Fx/2 - (Fx-Lx)/2; the mirror of X is 2nb - X when that
// lies inside the image; the column x' = 0 (X = nb) is S0 + sum_{d>0} (p+q) and
// is summed by one warp of the first column block.  A CTA keeps its columns'
// twiddles in registers and walks the images blockIdx.y, blockIdx.y + gridDim.y, ...
// Two output layouts:
//   plain  tm[img][r][X]: r = 0 Re T0, 1..2Ny Re T, 2Ny+1..4Ny Im T (fi_fold_kernel)
//   K-major (tensor-core FI) t0[img][X] = Re T0 and hi/lo TF32 splits of
//          tm[img][X][KP]: r = fy-1 Re T, 2Ny+fy-1 Im T, zero to KP
// ---------------------------------------------------------------------------
constexpr int FR_THREADS = 256, FR_COLS = 128, FR_ROWS = 2 * FR_COLS + 1;  // column, mirror, x' = 0

template <int MAXD, bool KMAJ, int KPC, int PRE>
__global__ void __launch_bounds__(FR_THREADS) fi_rows_kernel(const float2* __restrict__ band_part, int ngroups,
                                                             const float2* __restrict__ twF, int Lx, int Fx,
                                                             int Nx, int Ny, int kp_rt, int batch,
                                                             float* __restrict__ tm, float* __restrict__ tmh,
                                                             float* __restrict__ tml, float* __restrict__ t0) {
  extern __shared__ __align__(16) float4 frs[];
  const int KP = KPC > 0 ? KPC : kp_rt;  // K-major row width (compile time where known)
  const int BH = 2 * Ny + 1, BW = 4 * Nx + 1, ND = 2 * Nx + 1;
  float4* sC = frs;                                       // [BH][MAXD]
  float* sO = reinterpret_cast<float*>(sC + BH * MAXD);  // K-major: [FR_ROWS][KP + 1]
  const int tid = threadIdx.x, xl = tid & (FR_COLS - 1), grp = tid / FR_COLS;
  const int nb = Fx / 2 - (Fx - Lx) / 2, M = 2 * nb;
  const int X0 = blockIdx.x * FR_COLS, X = X0 + xl, Xm = M - X;
  const bool live = X < nb, mlive = live && Xm < Lx;
  const bool xtra = blockIdx.x == 0 && nb < Lx;  // this block adds the column x' = 0
  early_next();
  float2 tw[MAXD];  // (the table is from before the window DFT, which no stage of its image precedes)
#pragma unroll
  for (int d = 1; d < MAXD; ++d)
    tw[d] = (d < ND && live) ? twF[(size_t)d * Lx + X] : make_float2(0.f, 0.f);
  early_wait(band_part);
  if (KMAJ)  // the K padding columns stay zero for every image
    for (int idx = tid; idx < FR_ROWS * (KP - 4 * Ny); idx += FR_THREADS) {
      const int c = idx / (KP - 4 * Ny), r = 4 * Ny + idx % (KP - 4 * Ny);
      sO[c * (KP + 1) + r] = 0.f;
    }
  const int fy0 = grp == 0 ? 0 : Ny + 1, fy1 = grp == 0 ? Ny + 1 : BH;
  const size_t pst = (size_t)BH * BW;
  // rows of this block in the K-major store: its columns X0.., their mirrors (ascending
  // X = Mlo + j for slots FR_COLS + nbase - 1 - j) and, in the first block, x' = 0
  const int nbase = max(0, min(FR_COLS, nb - X0));
  const int imin = max(0, M - X0 - Lx + 1);
  const int nmir = max(0, nbase - imin), Mlo = M - X0 - nbase + 1;
  const int nrows = nbase + nmir + (xtra ? 1 : 0);
  // the next image's band partials stream into shared memory (8-byte cp.async) while
  // this image is computed where two buffers fit (PRE = 2); with one (PRE = 1) this image's all
  // arrive together, and without (PRE = 0) they are summed from L2, eight loads in flight
  const int RAWN = ngroups * BH * BW;
  float2* raw = reinterpret_cast<float2*>(
      (reinterpret_cast<uintptr_t>(sO + (KMAJ ? FR_ROWS * (KP + 1) : 0)) + 15) & ~uintptr_t(15));
  auto fetch = [&](int im, float2* dst) {
    const float2* src = band_part + (size_t)im * RAWN;
    for (int e = tid; e < RAWN; e += FR_THREADS) {
      const unsigned da = (unsigned)__cvta_generic_to_shared(dst + e);
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(da), "l"(src + e) : "memory");
    }
  };
  if (PRE == 2) {
    if ((int)blockIdx.y < batch) fetch(blockIdx.y, raw);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  for (int img = blockIdx.y, k = 0; img < batch; img += gridDim.y, ++k) {
    if (PRE == 2) {
      if (img + (int)gridDim.y < batch) fetch(img + gridDim.y, raw + (size_t)((k + 1) & 1) * RAWN);
      asm volatile("cp.async.commit_group;" ::: "memory");
      asm volatile("cp.async.wait_group 1;" ::: "memory");  // this image's partials have landed
    }
    if (PRE == 1) {  // every thread is past the previous image's combine (the barrier behind it)
      fetch(img, raw);
      asm volatile("cp.async.wait_all;" ::: "memory");
    }
    __syncthreads();  // the previous image is out of sC and sO (and this one's partials are visible)
    const float2* B = PRE ? raw + (size_t)(PRE == 2 ? k & 1 : 0) * RAWN : band_part + (size_t)img * RAWN;
    for (int idx = tid; idx < BH * MAXD; idx += FR_THREADS) {
      const int fy = idx / MAXD, d = idx - fy * MAXD;  // MAXD: a compile-time divisor
      if (d >= ND) continue;
      const float2* S = B + fy * BW + 2 * Nx;
      float2 pv, qv;  // the kernel groups' partials in a fixed order
      if constexpr (PRE != 0) {
        pv = S[d];
        qv = S[-d];
        for (int gi = 1; gi < ngroups; ++gi) {
          const float2 a = S[gi * pst + d], b = S[gi * pst - d];
          pv.x += a.x;
          pv.y += a.y;
          qv.x += b.x;
          qv.y += b.y;
        }
      } else {
        pv = sum_strided(S + d, pst, ngroups);
        qv = d > 0 ? sum_strided(S - d, pst, ngroups) : pv;
      }
      if (d == 0) {
        sC[fy * MAXD] = make_float4(pv.x, pv.y, 0.f, 0.f);
      } else {
        sC[fy * MAXD + d] = make_float4(pv.x + qv.x, -(pv.y - qv.y), pv.y + qv.y, pv.x - qv.x);
      }
    }
    __syncthreads();
    float* out = KMAJ ? nullptr : tm + (size_t)img * (4 * Ny + 1) * Lx;
    for (int fy = fy0; fy < fy1; ++fy) {
      const float4* C = sC + fy * MAXD;
      // four independent FMA chains as two packed pairs: (ra, rb) += (c0, c1) * t and
      // (ia, ib) += (c2, c3) * t with t = (cos, sin) of the column, one f32x2 FMA each
      // (per component the same fmaf); without the term guard when 2Nx+1 is the table width
      float2 r = make_float2(C[0].x, 0.f), i2 = make_float2(C[0].y, 0.f);
      if (ND == MAXD) {
#pragma unroll
        for (int d = 1; d < MAXD; ++d) {
          const float4 a = C[d];
          r = __ffma2_rn(make_float2(a.x, a.y), tw[d], r);
          i2 = __ffma2_rn(make_float2(a.z, a.w), tw[d], i2);
        }
      } else {
#pragma unroll
        for (int d = 1; d < MAXD; ++d) {
          if (d < ND) {
            const float4 a = C[d];
            r = __ffma2_rn(make_float2(a.x, a.y), tw[d], r);
            i2 = __ffma2_rn(make_float2(a.z, a.w), tw[d], i2);
          }
        }
      }
      if (!live) continue;
      const float re = r.x + r.y, im = i2.x + i2.y, rem = r.x - r.y, imm = i2.x - i2.y;
      if (KMAJ) {
        if (fy == 0) {
          t0[(size_t)img * Lx + X] = re;
          if (mlive) t0[(size_t)img * Lx + Xm] = rem;
        } else {
          sO[xl * (KP + 1) + fy - 1] = re;
          sO[xl * (KP + 1) + 2 * Ny + fy - 1] = im;
          sO[(FR_COLS + xl) * (KP + 1) + fy - 1] = rem;  // unused when the mirror is outside
          sO[(FR_COLS + xl) * (KP + 1) + 2 * Ny + fy - 1] = imm;
        }
      } else if (fy == 0) {
        out[X] = re;
        if (mlive) out[Xm] = rem;
      } else {
        out[(size_t)fy * Lx + X] = re;
        out[(size_t)(2 * Ny + fy) * Lx + X] = im;
        if (mlive) {
          out[(size_t)fy * Lx + Xm] = rem;
          out[(size_t)(2 * Ny + fy) * Lx + Xm] = imm;
        }
      }
    }
    if (xtra && tid < 32) {  // the column x' = 0: S0 + sum_{d>0} (p + q), d in order
      for (int fy = tid; fy < BH; fy += 32) {
        const float4* C = sC + fy * MAXD;
        float re = C[0].x, im = C[0].y;
        for (int d = 1; d < ND; ++d) {
          re += C[d].x;
          im += C[d].z;
        }
        if (KMAJ) {
          if (fy == 0) {
            t0[(size_t)img * Lx + nb] = re;
          } else {
            sO[2 * FR_COLS * (KP + 1) + fy - 1] = re;
            sO[2 * FR_COLS * (KP + 1) + 2 * Ny + fy - 1] = im;
          }
        } else if (fy == 0) {
          out[nb] = re;
        } else {
          out[(size_t)fy * Lx + nb] = re;
          out[(size_t)(2 * Ny + fy) * Lx + nb] = im;
        }
      }
    }
    if (KMAJ) {
      __syncthreads();
      // each row is KP floats of [X][KP]: float4 stores, rows of one run contiguous
      const int q4 = KP / 4;
      for (int e = tid; e < nrows * q4; e += FR_THREADS) {
        const int s = e / q4, c = 4 * (e - s * q4);
        int srow, Xg;
        if (s < nbase) {
          srow = s;
          Xg = X0 + s;
        } else if (s < nbase + nmir) {
          const int j = s - nbase;
          srow = FR_COLS + nbase - 1 - j;
          Xg = Mlo + j;
        } else {
          srow = 2 * FR_COLS;
          Xg = nb;
        }
        const float* v = sO + srow * (KP + 1) + c;
        const float h0 = tc::tf32_round(v[0]), h1 = tc::tf32_round(v[1]), h2 = tc::tf32_round(v[2]),
                    h3 = tc::tf32_round(v[3]);
        const size_t o = ((size_t)img * Lx + Xg) * KP + c;
        *reinterpret_cast<float4*>(tmh + o) = make_float4(h0, h1, h2, h3);
        *reinterpret_cast<float4*>(tml + o) = make_float4(v[0] - h0, v[1] - h1, v[2] - h2, v[3] - h3);
      }
    }
  }
}

template <int MAXD, bool KMAJ, int KPC = 0>
static cudaError_t launch_fi_rows_t(cudaStream_t s, const ImgPlan& p, const float2* band_part, const float2* twF,
                                    int KP, float* tm, float* tmh, float* tml, float* t0) {
  const ImgGeom& g = p.g;
  // shared memory for the band partials: two buffers where they fit in 32 KB (the next image's
  // arrive meanwhile), one up to 110 KB (small batches have many kernel groups: one image of
  // 1024^2 with 24 of them took 23 us when they were summed from L2)
  const int rawn = p.ngroups * (2 * g.Ny + 1) * (4 * g.Nx + 1);
  const size_t raw = (size_t)rawn * sizeof(float2);
  const int pre = 2 * raw <= 32 * 1024 ? 2 : raw <= 110 * 1024 ? 1 : 0;
  const size_t smem = (size_t)(2 * g.Ny + 1) * MAXD * sizeof(float4) +
                      (KMAJ ? (size_t)FR_ROWS * (KP + 1) * sizeof(float) : 0) +
                      (pre ? pre * raw + 16 : 0);
  auto k = pre == 2 ? fi_rows_kernel<MAXD, KMAJ, KPC, 2> : pre == 1 ? fi_rows_kernel<MAXD, KMAJ, KPC, 1>
                                                                    : fi_rows_kernel<MAXD, KMAJ, KPC, 0>;
  cudaError_t e = allow_smem(k);
  if (e != cudaSuccess) return e;
  // column blocks over the x' < 0 half; as many image groups as keep every CTA resident
  // at once (a second partial wave would double the time of the CTAs in it), each CTA
  // walking its group's images with its twiddles kept in registers
  const int nb = g.Fx / 2 - (g.Fx - g.Lx) / 2;
  const int ncb = std::max(1, (nb + FR_COLS - 1) / FR_COLS);
  const int sms = p.sms > 0 ? p.sms : 148;
  int per_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, FR_THREADS, smem);
  if (e != cudaSuccess) return e;
  const int groups = std::max(1, std::min(p.batch, std::max(1, per_sm) * sms / ncb));
  return launch_early(p.early, k, dim3(ncb, groups), FR_THREADS, smem, s, band_part, p.ngroups, twF, g.Lx, g.Fx, g.Nx, g.Ny,
                      KP, p.batch, tm, tmh, tml, t0);
}

cudaError_t launch_fi_rows(cudaStream_t s, const ImgPlan& p, const float2* band_part, const float2* twF, int KP,
                           float* tm, float* tmh, float* tml, float* t0) {
  const int ND = 2 * p.g.Nx + 1;
  const bool km = tmh != nullptr;
  if (km) {  // Ny > 8: the K-major rows are 64 wide
    if (ND <= 5) return launch_fi_rows_t<5, true, 64>(s, p, band_part, twF, KP, tm, tmh, tml, t0);
    if (ND <= 9) return launch_fi_rows_t<9, true, 64>(s, p, band_part, twF, KP, tm, tmh, tml, t0);
    if (ND <= 17) return launch_fi_rows_t<17, true, 64>(s, p, band_part, twF, KP, tm, tmh, tml, t0);
    return launch_fi_rows_t<33, true, 64>(s, p, band_part, twF, KP, tm, tmh, tml, t0);
  }
  if (ND <= 5) return launch_fi_rows_t<5, false>(s, p, band_part, twF, KP, tm, tmh, tml, t0);
  if (ND <= 9) return launch_fi_rows_t<9, false>(s, p, band_part, twF, KP, tm, tmh, tml, t0);
  if (ND <= 17) return launch_fi_rows_t<17, false>(s, p, band_part, twF, KP, tm, tmh, tml, t0);
  return launch_fi_rows_t<33, false>(s, p, band_part, twF, KP, tm, tmh, tml, t0);
}

// twF[d][X] = e^{+2 pi i d x'/Fx}, d = 0..2Nx: the FI column twiddles
__global__ void twF_init_kernel(float2* __restrict__ tw, int Lx, int Fx, int ND) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x, d = blockIdx.y;
  if (x >= Lx || d >= ND) return;
  const long long xp = (long long)x + (Fx - Lx) / 2 - Fx / 2;
  float2 t;
  cis_round((long long)d * xp, Fx, &t.x, &t.y);
  tw[(size_t)d * Lx + x] = t;
}

// cached per (Lx, Fx, Nx) on the context
int fi_twiddles(litho_ctx* ctx, const ImgGeom& g, const float2** out) {
  auto key = std::make_tuple(g.Lx, g.Fx, g.Nx, -4000);
  auto it = ctx->twx_tables.find(key);
  if (it == ctx->twx_tables.end()) {
    const int ND = 2 * g.Nx + 1;
    DevBuf b;
    LITHO_RET(b.ensure(ctx, (size_t)ND * g.Lx * sizeof(float2)));
    StageScope sc(ctx, LITHO_STAGE_UPLOAD);
    twF_init_kernel<<<dim3((g.Lx + 127) / 128, ND), 128, 0, ctx->stream>>>(b.as<float2>(), g.Lx, g.Fx, ND);
    LITHO_CUDA_TRY(ctx, cudaGetLastError());
    it = ctx->twx_tables.emplace(key, b).first;
  }
  *out = it->second.as<float2>();
  return LITHO_OK;
}

// ---------------------------------------------------------------------------
// Full centred mask spectrum (litho_fft_mask): two passes of a block FFT over
// shared-memory rows, each pass writing its result transposed.
//   C[X] = sum_p a[p] e^{-2 pi i (X - F/2)(p - F/2)/F}
//        = (-1)^(X + F/2) * DFT((-1)^p a[p])[X]
// Up to three radix-2 stages at a time run in registers (the same butterflies and
// twiddles as one by one), the first of them straight from global memory, so that
// a row of 1024 crosses shared memory four times instead of eleven; and a CTA takes
// four rows instead of sixteen, which gives every SM work (64 CTAs for 1024 rows
// left most idle).  One 1024 x 1024 mask: 2 x 75 us -> 2 x 14.
// ---------------------------------------------------------------------------
constexpr int FM_THREADS = 256;

// place of element i of a row: consecutive ones, and ones F/16 or 8 apart, spread over the banks
__host__ __device__ __forceinline__ int fm_pad(int i) { return i + (i >> 3) + (i >> 6); }
__host__ __device__ __forceinline__ int fm_stride(int F) { return ((fm_pad(F - 1) + 16) & ~15) + 4; }

// stages h, 2 h, .. 2^(S-1) h on 2^S elements pos + m h of one group
template <int S>
__device__ __forceinline__ void fm_stages(float2 (&x)[8], const float2* tw, int logF, int lh, int pos) {
#pragma unroll
  for (int q = 0; q < S; ++q)
#pragma unroll
    for (int m = 0; m < (1 << S); ++m)
      if (!(m & (1 << q))) {
        const float2 w = tw[(pos + ((m & ((1 << q) - 1)) << lh)) << (logF - lh - q - 1)];
        const float2 t = cmul(w, x[m | (1 << q)]), a = x[m];
        x[m] = cadd(a, t);
        x[m | (1 << q)] = csub(a, t);
      }
}
template <int S>
__device__ __forceinline__ void fm_pass(float2* s, int SF, const float2* tw, int TR, int logF, int lh) {
  const int per = 1 << (logF - S);
  for (int idx = threadIdx.x; idx < TR * per; idx += FM_THREADS) {
    const int j = idx & (per - 1), pos = j & ((1 << lh) - 1);
    float2* row = s + (idx >> (logF - S)) * SF;
    const int base = ((j >> lh) << (lh + S)) + pos;
    float2 x[8];
#pragma unroll
    for (int m = 0; m < (1 << S); ++m) x[m] = row[fm_pad(base + (m << lh))];
    fm_stages<S>(x, tw, logF, lh, pos);
#pragma unroll
    for (int m = 0; m < (1 << S); ++m) row[fm_pad(base + (m << lh))] = x[m];
  }
}

// rows: `nrows` input rows of length `len` (real if in_i == nullptr), padded
// centred into F; output written transposed: out[X][row] (row stride ldo).
template <int S0>
__global__ void __launch_bounds__(FM_THREADS) fft_rows_centred_kernel(
    const float* __restrict__ in_r, const float* __restrict__ in_i, const float2* __restrict__ in_c,
    int nrows, int len, int logF, int TR, float scale, float2* __restrict__ out_c, float* __restrict__ out_r,
    float* __restrict__ out_i, int ldo) {
  extern __shared__ __align__(16) float2 fr[];
  const int F = 1 << logF, SF = fm_stride(F);
  float2* s = fr;                 // [TR][SF]
  float2* tw = fr + TR * SF;      // [F/2]
  const int tid = threadIdx.x;
  const int r0 = blockIdx.x * TR;
  const int off = (F - len) / 2;
  for (int e = tid; e < F / 2; e += FM_THREADS) {
    float sn, cs;
    sincospif(2.0f * (float)e / (float)F, &sn, &cs);
    tw[e] = make_float2(cs, -sn);
  }
  __syncthreads();
  // the first stages, on elements q + m F / 2^S0 (bit-reversed: adjacent), pre-multiplied by (-1)^p
  const int per = F >> S0;
  for (int idx = tid; idx < TR * per; idx += FM_THREADS) {
    const int r = idx >> (logF - S0), q = idx & (per - 1);
    const int row = r0 + r;
    float2 x[8];
#pragma unroll
    for (int m = 0; m < (1 << S0); ++m) {
      const int p = q + (int)(__brev((unsigned)m) >> (32 - S0)) * per, i = p - off;
      float2 v = make_float2(0.f, 0.f);
      if (row < nrows && i >= 0 && i < len) {
        const size_t o = (size_t)row * len + i;
        if (in_c) v = in_c[o];
        else v = make_float2(in_r[o], in_i ? in_i[o] : 0.f);
        if (p & 1) v = make_float2(-v.x, -v.y);
      }
      x[m] = v;
    }
    fm_stages<S0>(x, tw, logF, 0, 0);
    const int base = logF == S0 ? 0 : (int)(__brev((unsigned)q) >> (32 - (logF - S0))) << S0;
#pragma unroll
    for (int m = 0; m < (1 << S0); ++m) s[r * SF + fm_pad(base + m)] = x[m];
  }
  __syncthreads();
  for (int lh = S0; lh < logF;) {
    const int left = logF - lh;
    if (left == 3 || left > 4) {
      fm_pass<3>(s, SF, tw, TR, logF, lh);
      lh += 3;
    } else if (left >= 2) {
      fm_pass<2>(s, SF, tw, TR, logF, lh);
      lh += 2;
    } else {
      fm_pass<1>(s, SF, tw, TR, logF, lh);
      lh += 1;
    }
    __syncthreads();
  }
  // transposed write with (-1)^(X + F/2) and scale
  const float sgnF = ((F / 2) & 1) ? -1.f : 1.f;
  for (int idx = tid; idx < TR * F; idx += FM_THREADS) {
    const int X = idx / TR, r = idx - X * TR;
    const int row = r0 + r;
    if (row >= nrows) continue;
    float2 v = s[r * SF + fm_pad(X)];
    const float sg = ((X & 1) ? -sgnF : sgnF) * scale;
    v = make_float2(v.x * sg, v.y * sg);
    const size_t o = (size_t)X * ldo + row;
    if (out_c) out_c[o] = v;
    else {
      out_r[o] = v.x;
      out_i[o] = v.y;
    }
  }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
ImgPlan make_plan(const ImgGeom& g, int batch, int sm_count) {
  ImgPlan p;
  p.g = g;
  p.batch = batch;
  win_fold_plan(p, sm_count);
  // SOCS is latency-bound (warp-shuffle FFT chains), but every kernel group also
  // transforms its own partial intensity: ~2.5 CTAs (20 warps) per SM measured best
  // at 1024^2, K=24, 64 masks (4 kernels per CTA: 36.9 us; 3: 38.9; 8: 45.0)
  int ng = (5 * sm_count + 2 * batch - 1) / (2 * batch);
  ng = std::max(1, std::min(ng, g.nk));
  p.kpg = (g.nk + ng - 1) / ng;
  p.ngroups = (g.nk + p.kpg - 1) / p.kpg;
  p.sms = sm_count;
  return p;
}

// coefficient tables of the folded transforms, cached per (Ly, Fy, Ny) on the context
static int fold_table(litho_ctx* ctx, const ImgGeom& g, int kind, size_t floats,
                      cudaError_t (*init)(cudaStream_t, const ImgGeom&, float*), const float** out) {
  auto key = std::make_tuple(g.Ly, g.Fy, g.Ny, kind);
  auto it = ctx->twx_tables.find(key);
  if (it == ctx->twx_tables.end()) {
    DevBuf b;
    LITHO_RET(b.ensure(ctx, floats * sizeof(float)));
    StageScope sc(ctx, LITHO_STAGE_UPLOAD);
    LITHO_CUDA_TRY(ctx, init(ctx->stream, g, b.as<float>()));
    it = ctx->twx_tables.emplace(key, b).first;
  }
  *out = it->second.as<float>();
  return LITHO_OK;
}

int run_win_dft(litho_ctx* ctx, const WinPart* parts, int n, float2* win_part, int nparts, int precision, const int* form) {
  const ImgGeom& g0 = parts[0].plan.g;
  if (g0.Nx > 16 || g0.Ny > 16) {
    set_error(ctx, LITHO_ERR_UNSUPPORTED, "window DFT supports Nx, Ny <= 16 (got %d, %d)", g0.Nx, g0.Ny);
    return LITHO_ERR_UNSUPPORTED;
  }
  if (n < 1 || n > WIN_MAX_SIZES) {
    set_error(ctx, LITHO_ERR_ARG, "window DFT over %d mask sizes (1..%d)", n, WIN_MAX_SIZES);
    return LITHO_ERR_ARG;
  }
  const float* coef[WIN_MAX_SIZES];
  const float2* twF[WIN_MAX_SIZES];
  for (int i = 0; i < n; ++i) {
    const ImgGeom& g = parts[i].plan.g;
    if (g.Fx != g0.Fx || g.Fy != g0.Fy || g.Nx != g0.Nx || g.Ny != g0.Ny || parts[i].plan.nparts() > nparts) {
      set_error(ctx, LITHO_ERR_ARG, "window DFT mask sizes of one launch must share the period and the kernels");
      return LITHO_ERR_ARG;
    }
    LITHO_RET(fold_table(ctx, g, -6001, win_fold_coef_floats(g), win_fold_coefs, &coef[i]));
    LITHO_RET(fi_twiddles(ctx, g, &twF[i]));
  }
  int* err = nullptr;
  LITHO_RET(tc_err_flag_public(ctx, &err));
  StageScope sc(ctx, LITHO_STAGE_WIN_DFT);
  LITHO_CUDA_TRY(ctx, launch_win_fold(ctx->stream, parts, n, coef, twF, win_part, nparts,
                                      precision == LITHO_PREC_MIXED ? ctx->test_stall_chunk : -1, err, form));
  return LITHO_OK;
}

template <int N>
static int launch_socs_t(litho_ctx* ctx, const ImgPlan& p, const WindowSrc& w, const float2* krn,
                         const float* scales, float2* band_part, float* tmpImgp) {
  const ImgGeom& g = p.g;
  const int KD = (2 * g.Nx + 1) * (2 * g.Ny + 1);
  size_t smem;
  decltype(&socs64_kernel) k;
  if constexpr (N == 64) {
    smem = socs64_smem_bytes(KD);
    k = socs64_kernel;
  } else if constexpr (N == 128) {
    smem = socs128_smem_bytes(2 * g.Ny + 1, KD);
    k = socs128_kernel;
  } else {
    smem = ((size_t)(2 * g.Ny + 1) * (N + 1) + N / 2 + KD) * sizeof(float2);
    k = socs_kernel<N>;
  }
  LITHO_CUDA_TRY(ctx, allow_smem(k));
  dim3 grid(p.ngroups, p.batch);
  StageScope sc(ctx, LITHO_STAGE_SOCS);
  LITHO_CUDA_TRY(ctx, launch_early(p.early, k, grid, N == 128 ? S128_THREADS : SOCS_THREADS, smem, ctx->stream, w.part,
                                   w.nparts, w.mskf_r, w.mskf_i, w.Fx ? w.Fx : g.Fx, w.Fy ? w.Fy : g.Fy, g.Nx, g.Ny, krn,
                                   scales, g.nk, p.kpg, band_part, tmpImgp));
  return LITHO_OK;
}

// tmpImgp of one image: the groups' intensities added in order
__global__ void tmp_join_kernel(const float* __restrict__ part, int ngroups, int n, float* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float v = part[i];
#pragma unroll 8
  for (int g = 1; g < ngroups; ++g) v += part[(size_t)g * n + i];
  out[i] = v;
}

// tmpImgp: [image][group][convN][convN]
int run_socs(litho_ctx* ctx, const ImgPlan& p, const WindowSrc& w, const float2* krn, const float* scales,
             float2* band_part, float* tmpImgp) {
  switch (p.g.convN) {
    case 32: return launch_socs_t<32>(ctx, p, w, krn, scales, band_part, tmpImgp);
    case 64: return launch_socs_t<64>(ctx, p, w, krn, scales, band_part, tmpImgp);
    case 128: return launch_socs_t<128>(ctx, p, w, krn, scales, band_part, tmpImgp);
    default:
      set_error(ctx, LITHO_ERR_UNSUPPORTED, "conv grid %d not in {32, 64, 128}", p.g.convN);
      return LITHO_ERR_UNSUPPORTED;
  }
}

int run_tmp_join(litho_ctx* ctx, const float* part, int ngroups, int n, float* tmpImgp) {
  StageScope sc(ctx, LITHO_STAGE_SOCS);
  tmp_join_kernel<<<(n + 127) / 128, 128, 0, ctx->stream>>>(part, ngroups, n, tmpImgp);
  LITHO_CUDA_TRY(ctx, cudaGetLastError());
  return LITHO_OK;
}

int run_fi(litho_ctx* ctx, const ImgPlan& p, const float2* band_part, float* tm, float* images) {
  const ImgGeom& g = p.g;
  {
    const float2* twF = nullptr;
    LITHO_RET(fi_twiddles(ctx, g, &twF));
    StageScope sc(ctx, LITHO_STAGE_FI_PREP);
    LITHO_CUDA_TRY(ctx, launch_fi_rows(ctx->stream, p, band_part, twF, 0, tm, nullptr, nullptr, nullptr));
  }
  const float* coef = nullptr;
  LITHO_RET(fold_table(ctx, g, -5001, fi_fold_coef_floats(g), fi_fold_coefs, &coef));
  StageScope sc(ctx, LITHO_STAGE_FI_OUT);
  LITHO_CUDA_TRY(ctx, launch_fi_fold(ctx->stream, p, tm, coef, images));
  return LITHO_OK;
}

// rows per CTA: four (two of 8192, by their shared memory), or enough for every thread
static int fm_rows_per_cta(int F) { return F >= 8192 ? 16384 / F : std::max(4, std::min(32, 2048 / F)); }

static int run_fft_rows(litho_ctx* ctx, const float* in_r, const float2* in_c, int nrows, int len, int F, float scale,
                        float2* out_c, float* out_r, float* out_i, int ldo) {
  const int TR = fm_rows_per_cta(F), logF = 31 - __builtin_clz((unsigned)F);
  const size_t smem = ((size_t)TR * fm_stride(F) + F / 2) * sizeof(float2);
  auto k = logF >= 3 ? fft_rows_centred_kernel<3> : logF == 2 ? fft_rows_centred_kernel<2> : fft_rows_centred_kernel<1>;
  LITHO_CUDA_TRY(ctx, allow_smem(k));
  k<<<(nrows + TR - 1) / TR, FM_THREADS, smem, ctx->stream>>>(in_r, nullptr, in_c, nrows, len, logF, TR, scale, out_c,
                                                             out_r, out_i, ldo);
  LITHO_CUDA_TRY(ctx, cudaGetLastError());
  return LITHO_OK;
}

int run_fft_mask(litho_ctx* ctx, const float* mask, int Lx, int Ly, float* mskf_r, float* mskf_i) {
  const int Fx = next_pow2(Lx), Fy = next_pow2(Ly);
  LITHO_RET(ctx->stage_x.ensure(ctx, (size_t)Fx * Ly * sizeof(float2)));
  float2* tmp = ctx->stage_x.as<float2>();
  StageScope sc(ctx, LITHO_STAGE_FFT_MASK, 2);
  // mask rows -> tmp[X][y] (Fx x Ly complex)
  LITHO_RET(run_fft_rows(ctx, mask, nullptr, Ly, Lx, Fx, 1.0f, tmp, nullptr, nullptr, Ly));
  // tmp rows (one per X, length Ly) -> mskf[Y][X] / (Fx*Fy)
  return run_fft_rows(ctx, nullptr, tmp, Fx, Ly, Fy, 1.0f / ((float)Fx * (float)Fy), nullptr, mskf_r, mskf_i, Fx);
}

// ---------------------------------------------------------------------------
// Context-free launch of the FP32 pipeline for one image into caller-provided
// scratch (used by the allocation-free entry point in noalloc.cu).  Launches
// only; it allocates nothing and records nothing on a context.
// ---------------------------------------------------------------------------
// kernels interleaved; also, the flag of the window's bounded waits starts every call at zero
__global__ void pack_planes_kernel(const float* __restrict__ kr, const float* __restrict__ ki, int n,
                                   float2* __restrict__ out, int* __restrict__ err) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0) *err = 0;
  if (i < n) out[i] = make_float2(kr[i], ki[i]);
}

// the flag of the kernels' bounded waits; then kernels, scales, window partials, band partials,
// interpolation rows, and the three tables
size_t noctx_scratch_layout(const ImgPlan& p, size_t off[8]) {
  const ImgGeom& g = p.g;
  const int KD = (2 * g.Nx + 1) * (2 * g.Ny + 1), KY = 2 * g.Ny + 1;
  const size_t sz[8] = {(size_t)g.nk * KD * sizeof(float2),
                        (size_t)g.nk * sizeof(float),
                        (size_t)p.nparts() * KY * (g.Nx + 1) * sizeof(float2),
                        (size_t)p.ngroups * KY * (4 * g.Nx + 1) * sizeof(float2),
                        (size_t)(4 * g.Ny + 1) * g.Lx * sizeof(float),
                        (size_t)(2 * g.Nx + 1) * g.Lx * sizeof(float2),
                        win_fold_coef_floats(g) * sizeof(float),
                        fi_fold_coef_floats(g) * sizeof(float)};
  size_t o = 256;
  for (int i = 0; i < 8; ++i) {
    off[i] = o;
    o += (sz[i] + 255) & ~size_t(255);
  }
  return o;
}

template <int N>
static cudaError_t noctx_socs_t(cudaStream_t s, const ImgPlan& p, const float2* win_part, const float2* krn,
                                const float* scales, float2* band_part) {
  const ImgGeom& g = p.g;
  const int KD = (2 * g.Nx + 1) * (2 * g.Ny + 1);
  size_t smem;
  decltype(&socs64_kernel) k;
  if constexpr (N == 64) {
    smem = socs64_smem_bytes(KD);
    k = socs64_kernel;
  } else if constexpr (N == 128) {
    smem = socs128_smem_bytes(2 * g.Ny + 1, KD);
    k = socs128_kernel;
  } else {
    smem = ((size_t)(2 * g.Ny + 1) * (N + 1) + N / 2 + KD) * sizeof(float2);
    k = socs_kernel<N>;
  }
  cudaError_t e = allow_smem(k);
  if (e != cudaSuccess) return e;
  k<<<dim3(p.ngroups, p.batch), N == 128 ? S128_THREADS : SOCS_THREADS, smem, s>>>(win_part, p.nparts(), nullptr,
                                                                                 nullptr, g.Fx, g.Fy, g.Nx,
                                                          g.Ny, krn, scales, g.nk, p.kpg, band_part, nullptr);
  return cudaGetLastError();
}

cudaError_t image_pipeline_noctx(cudaStream_t s, const ImgPlan& p, const float* mask, const float* krn_r,
                                 const float* krn_i, const float* scales, char* scratch, float* image) {
  const ImgGeom& g = p.g;
  size_t off[8];
  noctx_scratch_layout(p, off);
  int* err = reinterpret_cast<int*>(scratch);
  float2* krn = reinterpret_cast<float2*>(scratch + off[0]);
  float* sc = reinterpret_cast<float*>(scratch + off[1]);
  float2* win_part = reinterpret_cast<float2*>(scratch + off[2]);
  float2* band_part = reinterpret_cast<float2*>(scratch + off[3]);
  float* tm = reinterpret_cast<float*>(scratch + off[4]);
  float2* twF = reinterpret_cast<float2*>(scratch + off[5]);
  float* wcoef = reinterpret_cast<float*>(scratch + off[6]);
  float* fcoef = reinterpret_cast<float*>(scratch + off[7]);
  const int KD = (2 * g.Nx + 1) * (2 * g.Ny + 1), ND = 2 * g.Nx + 1;
  cudaError_t e;
  pack_planes_kernel<<<(g.nk * KD + 255) / 256, 256, 0, s>>>(krn_r, krn_i, g.nk * KD, krn, err);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  if ((e = cudaMemcpyAsync(sc, scales, g.nk * sizeof(float), cudaMemcpyDeviceToDevice, s)) != cudaSuccess) return e;
  twF_init_kernel<<<dim3((g.Lx + 127) / 128, ND), 128, 0, s>>>(twF, g.Lx, g.Fx, ND);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  if ((e = win_fold_coefs(s, g, wcoef)) != cudaSuccess) return e;
  if ((e = fi_fold_coefs(s, g, fcoef)) != cudaSuccess) return e;
  const WinPart part{p, mask, 0};
  const float* wc = wcoef;
  const float2* wt = twF;
  if ((e = launch_win_fold(s, &part, 1, &wc, &wt, win_part, p.nparts(), -1, err, nullptr)) != cudaSuccess) return e;
  switch (g.convN) {
    case 32: e = noctx_socs_t<32>(s, p, win_part, krn, sc, band_part); break;
    case 64: e = noctx_socs_t<64>(s, p, win_part, krn, sc, band_part); break;
    default: e = noctx_socs_t<128>(s, p, win_part, krn, sc, band_part); break;
  }
  if (e != cudaSuccess) return e;
  if ((e = launch_fi_rows(s, p, band_part, twF, 0, tm, nullptr, nullptr, nullptr)) != cudaSuccess) return e;
  return launch_fi_fold(s, p, tm, fcoef, image);
}

int image_pipeline(litho_ctx* ctx, const ImgGeom& g, int batch, const float* masks, const litho_kernel_set* ks,
                   float* images, int precision) {
  const int KY = 2 * g.Ny + 1;
  const bool tc = precision == LITHO_PREC_MIXED && fi_tc_serves(g);
  const bool band = use_band_tcc(ctx, ks, batch);
  ImgPlan p = make_plan(g, batch, ctx->sm_count);
  const bool win_tc = precision == LITHO_PREC_MIXED && win_tc_serves(g, batch) &&
                      (reinterpret_cast<uintptr_t>(masks) & 15) == 0;
  if (win_tc) win_tc_plan(p);
  if (band) {
    p.ngroups = ks->band_nc;
    p.kpg = g.nk;
  }
  // The stages of a small call are a few microseconds each, and so is the gap between two launches: one
  // image of 256^2 took 20.6 us with the gaps and takes 14.4 without, one of 1024^2 31.9 and 24.7,
  // sixteen 54.8 and 51.3, and large batches the same with and without (the next stage's CTAs come in only
  // when the last of this one's has started)
  p.early = true;
  LITHO_RET(ctx->win_part.ensure(ctx, (size_t)batch * p.nparts() * KY * (g.Nx + 1) * sizeof(float2)));
  LITHO_RET(ctx->band_part.ensure(ctx, (size_t)batch * p.ngroups * KY * (4 * g.Nx + 1) * sizeof(float2)));
  if (band) LITHO_RET(ctx->band_w.ensure(ctx, band_wsum_bytes(g, batch)));
  if (!tc) LITHO_RET(ctx->tm.ensure(ctx, (size_t)batch * (4 * g.Ny + 1) * g.Lx * sizeof(float)));
  const WinPart part{p, masks, 0};
  if (win_tc) {
    const float2* twF = nullptr;  // the interpolation rows read it before they wait: made before this stage
    LITHO_RET(fi_twiddles(ctx, g, &twF));
    LITHO_RET(run_win_dft_tc(ctx, &part, 1, ctx->win_part.as<float2>(), p.nparts(), nullptr));
  } else {
    LITHO_RET(run_win_dft(ctx, &part, 1, ctx->win_part.as<float2>(), p.nparts(), precision, nullptr));
  }
  WindowSrc w;
  w.part = ctx->win_part.as<float2>();
  w.nparts = p.nparts();
  if (band) LITHO_RET(run_band_tcc(ctx, p, w, ks, ctx->band_w.as<float2>(), ctx->band_part.as<float2>()));
  else LITHO_RET(run_socs(ctx, p, w, ks->krn, ks->scales, ctx->band_part.as<float2>(), nullptr));
  if (tc) return run_fi_tc(ctx, p, ctx->band_part.as<float2>(), nullptr, images);
  return run_fi(ctx, p, ctx->band_part.as<float2>(), ctx->tm.as<float>(), images);
}

}  // namespace litho
