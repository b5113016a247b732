// SOCS kernel extraction (litho.cpp:579-645 calcKernels): the top-nk eigenpairs
// of the Hermitian TCC in FP64 on the GPU.  The reference calls LAPACK zheevr
// ('V', 'I', 'U'); this file computes the same eigenpairs with
//
//   1. hermitize_kernel     A = upper triangle of TCC mirrored (zheevr reads 'U' only)
//   2. Householder tridiagonalisation, one reflector per column k (the zhetd2
//      recurrence), two launches per column: symv_hh_kernel forms v, tau, beta
//      and x = tau*B*v; her2_kernel B -= v w^H + w v^H with w = x - tau/2 (x^H v) v
//      on the lower-triangle tiles, mirrored.  The off-diagonal comes out real.
//      Column k below the diagonal is read as the conjugate of row k (A stays
//      Hermitian in full), and v_k is packed contiguously for the back-transform.
//      Matrices whose rows fit the SMs' shared memory take one cooperative launch
//      instead (tridiag_kernel).
//      Both kernels are bound by the FP64 pipe (GB300: 2 DFMA/clk/SM), so the
//      arithmetic is written as FMA chains and the update touches each element
//      pair once.
//   3. multisect_kernel     the nk largest eigenvalues of the real tridiagonal T
//                           by Sturm counts taken from both ends of T, a cluster of
//                           CTAs per eigenvalue: each round evaluates up to 256
//                           points of the bracketing interval at once;
//   4. invvec_kernel        eigenvector j of T by inverse iteration on the
//                           pivoted tridiagonal LU of T - shift_j I (the dgttrf
//                           recurrence), one CTA per eigenvector with the LU in
//                           shared memory;
//      cluster_rr_kernel    inside each cluster of close eigenvalues (a symmetric
//                           source gives exact degenerate pairs) the vectors are
//                           orthonormalised (Cholesky QR, twice) and rotated by
//                           a Rayleigh-Ritz step on the cluster's subspace
//                           (Jacobi eigendecomposition of Z^T T Z);
//   5. backtransform_kernel y = H_0 H_1 ... H_{n-2} z;
//   6. output_kernel        scales[i] = lambda_i (descending) and
//                           krn[i][j] = y_i[n-1-j] (litho.cpp:626-634 reversal).
// No kernel waits on another; every step is a separate launch on the stream (tridiag_kernel's CTAs wait
// on one another inside their cooperative launch, each time with a limit).
#include "litho_internal.cuh"
#include "tc_common.cuh"

#include <cooperative_groups.h>

#include <algorithm>
#include <cfloat>
#include <cmath>
#include <vector>

namespace litho {

__device__ __forceinline__ double2 zmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 zconj(double2 a) { return make_double2(a.x, -a.y); }
// conj by flipping the sign bit on the integer pipe (the FP64 pipe is the scarce one)
__device__ __forceinline__ double2 zconj_bits(double2 a) {
  return make_double2(a.x, __longlong_as_double(__double_as_longlong(a.y) ^ (long long)0x8000000000000000ull));
}
// lower-triangle tile t = I (I + 1) / 2 + J -> (I, J), in FP32 plus integer fix-ups
__device__ __forceinline__ void tri_tile(int t, int& I, int& J) {
  I = (int)((sqrtf(8.0f * (float)t + 1.0f) - 1.0f) * 0.5f);
  while (I * (I + 1) / 2 > t) --I;
  while ((I + 1) * (I + 2) / 2 <= t) ++I;
  J = t - I * (I + 1) / 2;
}

template <int NT>
__device__ double block_sum(double v, double* red) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();
  if (lane == 0) red[w] = v;
  __syncthreads();
  double t = 0.0;
  if (threadIdx.x < NT / 32) t = red[threadIdx.x];
  if (w == 0) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (lane == 0) red[0] = t;
  }
  __syncthreads();
  const double r = red[0];
  __syncthreads();
  return r;
}

__global__ void hermitize_kernel(const double2* __restrict__ in, double2* __restrict__ A, int n) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x, i = blockIdx.y;
  if (i >= n || j >= n) return;
  double2 v;
  if (i < j) v = in[(size_t)i * n + j];
  else if (i > j) v = zconj(in[(size_t)j * n + i]);
  else v = make_double2(in[(size_t)i * n + i].x, 0.0);
  A[(size_t)i * n + j] = v;
}

// Step k of the reduction, fused: the reflector of column k and x = tau B v with
// B = A[k+1:, k+1:].  Column k below the diagonal is conj(row k right of it), read
// contiguously.  Every CTA derives the reflector's scalars (norm, beta, tau, scale)
// from row k by the same fixed-order reduction, so they agree bitwise, and CTA 0
// publishes v, tau, d[k], e[k] and the packed copy of v kept for the back-transform.
// With v = (1, scl conj(row_k[1:])), B v = B[:,0] + scl B[:,1:] conj(row_k[1:]), so a
// row needs only row k itself; one warp per row, FMA chains (4 per complex element).
// Each CTA also leaves the partial sum of conj(x_i) v_i over its rows: the rank-2
// update adds them up in a fixed order for its correction term.
__device__ __forceinline__ size_t vpack_off(int n, int k) { return (size_t)k * (n - 1) - (size_t)k * (k - 1) / 2; }

__global__ void __launch_bounds__(256) symv_hh_kernel(const double2* __restrict__ A, int n, int k,
                                                      double2* __restrict__ vbuf, double2* __restrict__ vpack,
                                                      double2* __restrict__ tau, double* __restrict__ d,
                                                      double* __restrict__ e, double2* __restrict__ xbuf,
                                                      double2* __restrict__ part) {
  __shared__ double red[32];
  __shared__ double2 sp[8];
  const int m = n - k - 1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const double2* rowk = A + (size_t)k * n + (k + 1);
  double s = 0.0;
  for (int i = 1 + threadIdx.x; i < m; i += 256) {
    const double2 x = rowk[i];
    s = fma(x.x, x.x, s);
    s = fma(x.y, x.y, s);
  }
  const double xnorm2 = block_sum<256>(s, red);
  __shared__ double2 s_t, s_scl;
  __shared__ double s_beta;
  if (threadIdx.x == 0) {  // the reflector's scalars (FP64 is scarce: one thread)
    const double2 alpha = zconj(rowk[0]);
    double2 tt = make_double2(0.0, 0.0);
    double beta = alpha.x;
    double2 sc = make_double2(0.0, 0.0);
    if (!(xnorm2 == 0.0 && alpha.y == 0.0)) {
      const double nrm = sqrt(alpha.x * alpha.x + alpha.y * alpha.y + xnorm2);
      beta = alpha.x >= 0.0 ? -nrm : nrm;
      tt = make_double2((beta - alpha.x) / beta, -alpha.y / beta);
      // scl = 1 / (alpha - beta)
      const double2 den = make_double2(alpha.x - beta, alpha.y);
      const double dd = den.x * den.x + den.y * den.y;
      sc = make_double2(den.x / dd, -den.y / dd);
    }
    s_t = tt;
    s_scl = sc;
    s_beta = beta;
  }
  __syncthreads();
  const double2 t = s_t, scl = s_scl;
  const double beta = s_beta;
  if (blockIdx.x == 0) {
    double2* vp = vpack + vpack_off(n, k);
    for (int i = threadIdx.x; i < m; i += 256) {
      const double2 v = i == 0 ? make_double2(1.0, 0.0) : zmul(zconj(rowk[i]), scl);
      vbuf[i] = v;
      vp[i] = v;
    }
    if (threadIdx.x == 0) {
      tau[k] = t;
      e[k] = beta;
      d[k] = A[(size_t)k * n + k].x;
    }
  }
  const int row = blockIdx.x * 8 + warp;
  double2 contrib = make_double2(0.0, 0.0);
  if (row < m) {
    const double2* Ar = A + (size_t)(k + 1 + row) * n + (k + 1);
    double re = 0.0, im = 0.0;
    for (int j = 1 + lane; j < m; j += 32) {
      const double2 a = Ar[j], r = rowk[j];  // a * conj(r)
      re = fma(a.x, r.x, re);
      re = fma(a.y, r.y, re);
      im = fma(a.y, r.x, im);
      im = fma(-a.x, r.y, im);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      re += __shfl_xor_sync(0xffffffffu, re, o);
      im += __shfl_xor_sync(0xffffffffu, im, o);
    }
    const double2 a0 = Ar[0];
    const double2 bv = make_double2(a0.x + (scl.x * re - scl.y * im), a0.y + (scl.x * im + scl.y * re));
    const double2 xr = zmul(t, bv);
    const double2 vr = row == 0 ? make_double2(1.0, 0.0) : zmul(zconj(rowk[row]), scl);
    contrib = zmul(zconj(xr), vr);
    if (lane == 0) xbuf[row] = xr;
  }
  if (lane == 0) sp[warp] = contrib;
  __syncthreads();
  if (threadIdx.x == 0) {
    double2 acc = sp[0];
    for (int w = 1; w < 8; ++w) acc = make_double2(acc.x + sp[w].x, acc.y + sp[w].y);
    part[blockIdx.x] = acc;
  }
}

// B -= v w^H + w v^H with w = x - tau/2 (x^H v) v, on the lower-triangle 32 x 32
// tiles (I >= J) only; x^H v is the fixed-order sum of the nparts partials of the
// product kernel, formed by every CTA.  An off-diagonal tile is computed once and
// written twice, as itself and as its conjugate transpose (staged in shared memory
// so both writes are coalesced); a diagonal tile writes its lower half and mirrors
// it into the upper.  That halves the FP64 work, and B stays exactly Hermitian,
// which the product kernel (full rows) relies on.  Each element is 8 FMAs.
// blockIdx.x enumerates the tiles row by row: t = I (I + 1) / 2 + J.
__global__ void __launch_bounds__(256) her2_kernel(double2* __restrict__ A, int n, int k,
                                                   const double2* __restrict__ vbuf, const double2* __restrict__ xbuf,
                                                   const double2* __restrict__ tau, const double2* __restrict__ part,
                                                   int nparts) {
  __shared__ double2 tile[32][33];
  __shared__ double2 s_c;
  __shared__ double2 s_v[2][32], s_w[2][32];  // [0]: the tile's columns, [1]: its rows
  const int m = n - k - 1;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  if (ty == 0) {
    double sr = 0.0, si = 0.0;
    for (int p = tx; p < nparts; p += 32) {
      sr += part[p].x;
      si += part[p].y;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      sr += __shfl_xor_sync(0xffffffffu, sr, o);
      si += __shfl_xor_sync(0xffffffffu, si, o);
    }
    if (tx == 0) {
      const double2 tk = tau[k];
      s_c = zmul(make_double2(-0.5 * tk.x, -0.5 * tk.y), make_double2(sr, si));
    }
  }
  __syncthreads();
  int I, J;
  tri_tile(blockIdx.x, I, J);
  if (threadIdx.x < 64) {  // w = x + c v for the tile's 32 columns and 32 rows, once
    const int side = threadIdx.x >> 5, q = (side ? I : J) * 32 + tx;
    double2 vq = make_double2(0.0, 0.0), wq = vq;
    if (q < m) {
      const double2 c = s_c;
      vq = vbuf[q];
      const double2 xq = xbuf[q];
      wq = make_double2(xq.x + (c.x * vq.x - c.y * vq.y), xq.y + (c.x * vq.y + c.y * vq.x));
    }
    s_v[side][tx] = vq;
    s_w[side][tx] = wq;
  }
  __syncthreads();
  const int j = J * 32 + tx;
  const double2 vj = s_v[0][tx], wj = s_w[0][tx];
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int i = I * 32 + ty + 8 * r;
    if (i < m && j < m) {
      const double2 vi = s_v[1][ty + 8 * r], wi = s_w[1][ty + 8 * r];
      double2* a = A + (size_t)(k + 1 + i) * n + (k + 1 + j);
      const double2 av = *a;
      // a - vi conj(wj) - wi conj(vj)
      double re = fma(-vi.x, wj.x, av.x);
      re = fma(-vi.y, wj.y, re);
      re = fma(-wi.x, vj.x, re);
      re = fma(-wi.y, vj.y, re);
      double im = fma(-vi.y, wj.x, av.y);
      im = fma(vi.x, wj.y, im);
      im = fma(-wi.y, vj.x, im);
      im = fma(wi.x, vj.y, im);
      const double2 nv = make_double2(re, im);
      if (I != J) *a = nv;
      tile[ty + 8 * r][tx] = nv;
    }
  }
  __syncthreads();
  if (I == J) {  // diagonal tile: lower half as computed, upper half mirrored
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int ii = ty + 8 * r, i = I * 32 + ii;
      if (i < m && j < m)
        A[(size_t)(k + 1 + i) * n + (k + 1 + j)] = ii >= tx ? tile[ii][tx] : zconj_bits(tile[tx][ii]);
    }
    return;
  }
  // mirror: A[J-tile row jj][I-tile col ii] = conj(tile[ii][jj])
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int jj = ty + 8 * r, ii = tx;
    const int row = J * 32 + jj, col = I * 32 + ii;
    if (row < m && col < m) A[(size_t)(k + 1 + row) * n + (k + 1 + col)] = zconj_bits(tile[ii][jj]);
  }
}

// ---------------------------------------------------------------------------
// The same reduction in one cooperative launch, for matrices whose rows fit the SMs' shared
// memory (n <= ~1200): CTA c keeps rows c, c + G, .. there in full for the whole reduction, and a
// column costs one grid barrier instead of two launches.  Per column k, with r the pivot row right
// of the diagonal (v = (1, scl conj(r[1:]))):
//   product   x_i = tau (B_i0 + scl sum_j B_ij conj(r_j)) for the CTA's rows, and its partial of
//             gamma = 2 Re(-tau/2 x^H v); the owner of row k + 1 has published that row as it is
//   barrier
//   update    B_ij -= v_i conj(x_j) + u_i conj(v_j),  u = x + gamma v,
//             which is v w^H + w v^H with w = x - tau/2 (x^H v) v; conj(v_j) = conj(scl) r_j, so
//             neither v nor w is formed but for the CTA's own rows.  Every CTA updates the next
//             pivot row for itself first (v_i = 1 there), so that its norm and scalars, formed by
//             the ninth warp meanwhile, need no exchange of their own.
// The FP64 units bound it: each quarter of an SM takes a warp's FP64 instruction every ~66 cycles,
// dependent or not and whatever its lanes do.  Large matrices spend them on 12 m^2 FMAs per column
// over all SMs (full rows: half of the update is done twice, which costs less than exchanging the
// halves would), small ones on the chain from the barrier to the next x; the barrier takes ~3,000
// cycles.  Measured, reduction: n = 289 6.0 -> 1.8 ms, n = 1089 31 -> 17.2 ms.  Polling values
// in place of a barrier was slower (n = 289: 9,000 cycles an exchange: 152 CTAs poll every value).
// ---------------------------------------------------------------------------
constexpr int TD_WARPS = 8, TD_THREADS = 32 * (TD_WARPS + 1);
constexpr int TD_MAX_ROWS = 16;
constexpr size_t TD_MAX_SMEM = 224 * 1024;

size_t tridiag_smem(int n, int G) {
  return ((size_t)((n + G - 1) / G) * n + 3 * (size_t)n) * sizeof(double2);
}

// Waits until *p has reached `target` (bounded: false after a second, with *err set).
__device__ __forceinline__ bool td_wait(const unsigned* p, unsigned target, int* err) {
  uint64_t t0 = 0;
  for (int spin = 0;; ++spin) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    if (v >= target) return true;
    if ((spin & 255) == 255) {
      const uint64_t t = tc::global_ns();
      if (t0 == 0) t0 = t;
      if (t - t0 > 1000000000ull || *reinterpret_cast<volatile int*>(err) != 0) {
        atomicExch(err, 1);
        return false;
      }
    }
  }
}
// grid barrier in two halves: arrive() after the CTA's writes, wait() for every CTA's arrival
__device__ __forceinline__ void td_arrive(unsigned* count) {
  __syncthreads();
  if (threadIdx.x == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(count) : "memory");
}
__device__ __forceinline__ bool td_arrived(const unsigned* count, unsigned target, int* err, int* s_ok) {
  if (threadIdx.x == 0) *s_ok = td_wait(count, target, err);
  __syncthreads();
  return *s_ok != 0;
}

// (re, im) summed over the warp: re in lanes 0-15, im in lanes 16-31
__device__ __forceinline__ double pair_sum(double re, double im, int lane) {
  const bool up = lane & 16;
  double v = (up ? im : re) + __shfl_xor_sync(0xffffffffu, up ? re : im, 16);
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// the same over each half of the warp by itself: re in the half's first eight lanes, im in its last
__device__ __forceinline__ double half_pair_sum(double re, double im, int lane) {
  const bool up = lane & 8;
  double v = (up ? im : re) + __shfl_xor_sync(0xffffffffu, up ? re : im, 8);
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// the reflector of a pivot row with pivot alpha = conj(first) and squared norm xn2 past it: the
// zlarfg scalars, the two reciprocals side by side in lanes 0 and 1 (whole warp)
struct TdScalars {
  double2 tau, scl;  // scl = 1 / (alpha - beta)
  double beta;
};
__device__ __forceinline__ TdScalars td_reflector(double2 first, double xn2, int lane) {
  const double2 alpha = zconj(first);
  const bool plain = xn2 == 0.0 && alpha.y == 0.0;
  const double nr = sqrt(fma(alpha.x, alpha.x, fma(alpha.y, alpha.y, xn2)));
  TdScalars r;
  r.beta = plain ? alpha.x : alpha.x >= 0.0 ? -nr : nr;
  const double dr = alpha.x - r.beta;
  const double inv = 1.0 / (lane == 0 ? r.beta : fma(dr, dr, alpha.y * alpha.y));
  const double ib = __shfl_sync(0xffffffffu, inv, 0), id = __shfl_sync(0xffffffffu, inv, 1);
  const double2 z = make_double2(0.0, 0.0);
  r.tau = plain ? z : make_double2(-dr * ib, -alpha.y * ib);
  r.scl = plain ? z : make_double2(dr * id, -alpha.y * id);
  return r;
}

// How many warps share a row, for rows of `steps` warp-widths: the FP64 unit of a quarter of an SM
// takes one warp instruction per ~66 cycles whatever else there is, so the load of the fullest
// quarter decides (per step and 5 for the reduction over the lanes).
__device__ __forceinline__ int td_split(int nact, int steps) {
  const int c1 = (nact + 3) / 4 * (12 * steps + 5), c2 = (nact + 1) / 2 * (6 * steps + 11),
            c4 = nact * (3 * steps + 14);
  return c1 <= c2 && c1 <= c4 ? 1 : c2 <= c4 ? 2 : 4;
}

__global__ void __launch_bounds__(TD_THREADS, 1) tridiag_kernel(const double2* __restrict__ A, int n,
                                                                double2* __restrict__ vpack, double2* __restrict__ tau,
                                                                double* __restrict__ d, double* __restrict__ e,
                                                                double* __restrict__ e2, double2* __restrict__ xg,
                                                                double2* __restrict__ rowbuf, double* __restrict__ part,
                                                                unsigned* count, int* err) {
  extern __shared__ __align__(16) double2 tds[];
  __shared__ double s_dot[TD_MAX_ROWS][4][2];  // per row and warp of the row: (re, im)
  __shared__ double2 s_x[TD_MAX_ROWS], s_v[TD_MAX_ROWS], s_us[TD_MAX_ROWS], s_us1;
  __shared__ TdScalars s_sc;
  __shared__ double2 s_ts;  // tau scl
  __shared__ int s_ok;
  const int c = blockIdx.x, G = gridDim.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int T = (n - c + G - 1) / G;  // rows c + G t, t < T
  double2* rows = tds;                                // [T][n]
  double2* xs = tds + (size_t)((n + G - 1) / G) * n;  // [n]
  double2* rs = xs + n;                               // [n] pivot row
  double2* rn = rs + n;                               // [n] next pivot row
  // the ninth warp: norm of pivot row k past its pivot and the reflector's scalars
  auto scalars = [&](int k, const double2* r) {
    double q = 0.0;
    for (int j = k + 2 + lane; j < n; j += 32) q = fma(r[j].x, r[j].x, fma(r[j].y, r[j].y, q));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) q += __shfl_xor_sync(0xffffffffu, q, o);
    const TdScalars t = td_reflector(r[k + 1], q, lane);
    const double2 ts = zmul(t.tau, t.scl);
    if (lane == 0) {
      s_sc = t;
      s_ts = ts;
      if (c == 0) {
        tau[k] = t.tau;
        e[k] = t.beta;
        e2[k] = t.beta * t.beta;
      }
    }
  };
  for (int t = 0; t < T; ++t)
    for (int j = tid; j < n; j += TD_THREADS) rows[(size_t)t * n + j] = A[(size_t)(c + G * t) * n + j];
  for (int j = tid; j < n; j += TD_THREADS) rs[j] = A[j];
  __syncthreads();
  if (warp == TD_WARPS) scalars(0, rs);
  if (c == 0 && tid == 0) d[0] = rs[0].x;
  for (int k = 0; k + 1 < n; ++k) {
    const int t0 = k < c ? 0 : (k - c) / G + 1, nact = T - t0;  // the CTA's rows past k
    const int wpr = td_split(nact, (n - k - 2 + 31) / 32), rstep = TD_WARPS / wpr, sub = warp & (wpr - 1);
    double2* xk = xg + (size_t)(k & 1) * n;
    double2* rowk = rowbuf + (size_t)(k & 1) * n;  // row k + 1
    double* pk = part + (size_t)(k & 1) * G;
    if (warp < TD_WARPS) {
      if (c == (k + 1) % G)
        for (int j = k + 1 + tid; j < n; j += 32 * TD_WARPS) __stcg(rowk + j, rows[(size_t)t0 * n + j]);
      for (int a = warp / wpr; a < nact; a += rstep) {
        const double2* row = rows + (size_t)(t0 + a) * n;
        double re = 0.0, im = 0.0;
        for (int j = k + 2 + 32 * sub + lane; j < n; j += 32 * wpr) {
          const double2 b = row[j], r = rs[j];  // b * conj(r)
          re = fma(b.x, r.x, re);
          re = fma(b.y, r.y, re);
          im = fma(b.y, r.x, im);
          im = fma(-b.x, r.y, im);
        }
        const double v = pair_sum(re, im, lane);
        if ((lane & 15) == 0) s_dot[a][sub][lane >> 4] = v;
      }
    }
    __syncthreads();  // products, and the scalars of the ninth warp
    if (warp == 0) {
      // lane a < 16: x of row a; lane 16 + a: its v and tau v (an FP64 instruction takes a warp's
      // time whatever its lanes do, so the two halves do different products at once)
      const int a = lane & 15, i = c + G * (t0 + a);
      const bool live = a < nact, hi = lane >= 16;
      double2 dt = make_double2(0.0, 0.0), p = dt, q = dt;
      if (live) {
        dt = make_double2(s_dot[a][0][0], s_dot[a][0][1]);
        for (int w = 1; w < wpr; ++w) {
          dt.x += s_dot[a][w][0];
          dt.y += s_dot[a][w][1];
        }
        p = hi ? (i == k + 1 ? make_double2(1.0, 0.0) : zconj(rs[i])) : s_sc.tau;
        q = hi ? (i == k + 1 ? make_double2(1.0, 0.0) : s_sc.scl) : rows[(size_t)(t0 + a) * n + k + 1];
      }
      const double2 z1 = zmul(p, q);                                // tau a0 | v
      const double2 z2 = zmul(hi ? s_sc.tau : s_ts, hi ? z1 : dt);  // tau scl dot | tau v
      const double2 x = make_double2(z1.x + z2.x, z1.y + z2.y);
      const double2 tv = make_double2(__shfl_down_sync(0xffffffffu, z2.x, 16), __shfl_down_sync(0xffffffffu, z2.y, 16));
      if (live && !hi) {
        __stcg(xk + i, x);
        s_x[a] = x;
      }
      double g = live && !hi ? -fma(x.x, tv.x, x.y * tv.y) : 0.0;  // -Re(tau conj(x) v)
      for (int o = nact <= 1 ? 0 : nact <= 2 ? 1 : nact <= 4 ? 2 : 8; o > 0; o >>= 1)
        g += __shfl_xor_sync(0xffffffffu, g, o);
      if (lane == 0) __stcg(pk + c, g);
      if (live && hi) {
        s_v[a] = z1;
        vpack[vpack_off(n, k) + i - (k + 1)] = z1;
      }
    }
    td_arrive(count);
    if (!td_arrived(count, (unsigned)G * (k + 1), err, &s_ok)) return;
    if (warp < TD_WARPS) {
      for (int j = k + 1 + tid; j < n; j += 32 * TD_WARPS) {
        xs[j] = __ldcg(xk + j);
        rn[j] = __ldcg(rowk + j);
      }
    } else {  // gamma, then u conj(scl) of the rows (lanes < 16) and of the next pivot row (lane 16)
      double g = 0.0;
      for (int p = lane; p < G; p += 160) {
        double v[5];
#pragma unroll
        for (int u = 0; u < 5; ++u) v[u] = p + 32 * u < G ? __ldcg(pk + p + 32 * u) : 0.0;
        g += ((v[0] + v[1]) + (v[2] + v[3])) + v[4];
      }
      const double2 x1 = __ldcg(xk + k + 1);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) g += __shfl_xor_sync(0xffffffffu, g, o);
      const bool mine = lane < nact, one = lane == 16;
      const double2 x = mine ? s_x[lane & 15] : x1, v = mine ? s_v[lane & 15] : make_double2(1.0, 0.0);
      const double2 u = make_double2(fma(g, v.x, x.x), fma(g, v.y, x.y)), us = zmul(u, zconj(s_sc.scl));
      if (mine) s_us[lane] = us;
      if (one) {
        s_us1 = us;
        if (c == 0) d[k + 1] = __ldcg(rowk + k + 1).x - x1.x - u.x;  // conj(v) = 1 there, and real
      }
    }
    __syncthreads();
    {  // the next pivot row
      const double2 us = s_us1;
      for (int j = k + 2 + tid; j < n; j += TD_THREADS) {
        const double2 b = rn[j], xj = xs[j], r = rs[j];
        double re = b.x - xj.x, im = b.y + xj.y;  // b - conj(xj) - us r
        re = fma(-us.x, r.x, re);
        re = fma(us.y, r.y, re);
        im = fma(-us.x, r.y, im);
        im = fma(-us.y, r.x, im);
        rn[j] = make_double2(re, im);
      }
    }
    __syncthreads();
    if (warp == TD_WARPS) {
      if (k + 2 < n) scalars(k + 1, rn);
    } else {
      for (int a = warp / wpr; a < nact; a += rstep) {
        if (c + G * (t0 + a) == k + 1) continue;
        double2* row = rows + (size_t)(t0 + a) * n;
        const double2 v = s_v[a], us = s_us[a];
        for (int j = k + 2 + 32 * sub + lane; j < n; j += 32 * wpr) {
          const double2 b = row[j], xj = xs[j], r = rs[j];
          // b - v conj(xj) - us r
          double re = fma(-v.x, xj.x, b.x);
          re = fma(-v.y, xj.y, re);
          re = fma(-us.x, r.x, re);
          re = fma(us.y, r.y, re);
          double im = fma(-v.y, xj.x, b.y);
          im = fma(v.x, xj.y, im);
          im = fma(-us.x, r.y, im);
          im = fma(-us.y, r.x, im);
          row[j] = make_double2(re, im);
        }
      }
      tc::named_bar(1, 32 * TD_WARPS);  // rows updated, before other warps take them
    }
    double2* t = rs;
    rs = rn;
    rn = t;
  }
}

__global__ void last_diag_kernel(const double2* __restrict__ A, int n, double* __restrict__ d) {
  if (threadIdx.x == 0) d[n - 1] = A[(size_t)(n - 1) * n + (n - 1)].x;
}

__global__ void square_kernel(const double* __restrict__ e, double* __restrict__ e2, int m) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < m) e2[i] = e[i] * e[i];
}

// Number of eigenvalues of T below x (Sylvester's law of inertia on the twisted factorisation
// of T - xI at row h): the negative pivots of the leading h rows, taken downwards, of the rows
// past h, taken upwards, and the sign of what both leave at row h.  The two halves are as long and
// independent, so two lanes share a point: lane l < 16 of a warp goes down, lane l + 16 up, and a
// count costs half the serial chain of the usual one-way recurrence.
//
// A half's pivots are the ratios q_i = p_i / p_{i-1} of its minors, p_i = (d_i - x) p_{i-1} -
// e_i^2 p_{i-2}, so a negative pivot is a sign change of p.  A row takes three FP64 instructions and
// nothing else on that pipe: a quarter of an SM issues one warp instruction per ~66 cycles, and a
// division is ten of them.  Signs, zeros and exponents are read as integers.  A minor that comes out
// zero is replaced by -pivmin p_{i-1} (the pivot -pivmin).  When a lane's |p_i| leaves
// [2^-256, 2^256), every lane of the warp brings its p_i towards 1 by a power of two of at most
// 2^+-256 (exact), p_{i-1} along with it: the lanes of a warp drift alike, so they go rarely together
// instead of often one by one.  p stays below 2^512, so a step cannot overflow.
__device__ __noinline__ double2 sturm_rescale(double pn, double p, double m, double pivmin) {
  if (pn == 0.0) pn = -pivmin * p;
  const int ex = (int)(((unsigned)__double2hiint(pn) >> 20) & 0x7FFu);
  const double f = __hiloint2double((1023 + max(-256, min(256, 1023 - ex))) << 20, 0);
  return make_double2(pn * f, m * f);
}

__device__ __forceinline__ int sturm_count_lt(const double* __restrict__ d, const double* __restrict__ e2, int n,
                                              double x, double pivmin, int lane) {
  const bool up = lane & 16;
  const int h = (n - 1) / 2, step = up ? -1 : 1;  // rows past h: h, or h + 1 where n is even
  const double* pd = up ? d + (n - 1) : d;        // the half's row i: pd[step i]
  const double* pe = up ? e2 + (n - 2) : e2;      // its coupling to the next row (the last one's: to row h)
  int c = 0;
  double p = 1.0, m = 0.0, a = *pd - x;  // p_{i-1}, e_{i-1}^2 p_{i-2}, d_i - x
  // a row ahead of their use: a load takes longer than a row leaves it
  double d1 = n > 1 ? pd[step] : 0.0, e1 = n > 1 ? *pe : 0.0;
  for (int i = 0; i < h; ++i) {
    const double dn = d1, en = e1;
    d1 = pd[step * (i + 2)];
    e1 = pe[step * (i + 1)];
    double pn = fma(a, p, -m);
    a = dn - x;
    m = en * p;  // these two don't wait for pn, so the pipe is never idle
    // outside [2^-256, 2^256), zero or subnormal
    const bool out = (((unsigned)__double2hiint(pn) >> 20) & 0x7FFu) - 767u >= 512u;
    if (__any_sync(0xffffffffu, out)) {
      const double2 r = sturm_rescale(pn, p, m, pivmin);
      pn = r.x;
      m = r.y;
    }
    c += (unsigned)(__double2hiint(pn) ^ __double2hiint(p)) >> 31;
    p = pn;
  }
  if (up && n - 1 - h > h) {
    double pn = fma(a, p, -m);
    m = e1 * p;
    if (pn == 0.0) pn = -pivmin * p;
    c += (unsigned)(__double2hiint(pn) ^ __double2hiint(p)) >> 31;
    p = pn;
  }
  // row h: (d_h - x) - e_{h-1}^2 / q_{h-1} - e_h^2 / q_{h+1}
  const double q = m / p;  // 0 for a half without rows
  const double qo = __shfl_xor_sync(0xffffffffu, q, 16);
  c += __shfl_xor_sync(0xffffffffu, c, 16);
  return c + (((d[h] - x) - (up ? qo : q)) - (up ? q : qo) < 0.0 ? 1 : 0);
}

// eigenvalue j (0 = largest) of T (diagonal d, off-diagonal e) by multisection: one cluster of C CTAs
// per eigenvalue; every round evaluates the Sturm count at 64 C interior points of the bracket
// [lo, hi], count(lo) <= m < count(hi) with m the ascending index, and keeps the sub-interval
// holding the crossing.  A count is a serial FP64 chain, the points of a round run side by side, one
// warp on each quarter of an SM (a second one there would wait for the first), so a round over four
// SMs gains log2(257) bits where bisection gains one.  The rounds stop when the bracket no longer
// shrinks in floating point.
// 24 eigenvalues, n = 289: 940 -> 202 us; n = 1089: 3,502 -> 708 us.
constexpr int MS_THREADS = 128, MS_POINTS = MS_THREADS / 2, MS_CMAX = 4;

__global__ void __launch_bounds__(MS_THREADS) multisect_kernel(const double* __restrict__ d,
                                                               const double* __restrict__ e,
                                                               const double* __restrict__ e2, int n,
                                                               double* __restrict__ evals) {
  namespace cg = cooperative_groups;
  __shared__ double sh[3][MS_THREADS / 32];
  __shared__ unsigned masks[2][MS_CMAX][MS_THREADS / 32];  // by parity of the round: 16 points a warp
  cg::cluster_group cl = cg::this_cluster();
  const int C = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  const int j = blockIdx.x / C, t = threadIdx.x, lane = t & 31, warp = t >> 5;
  double lo = 1e300, hi = -1e300, emax = 0.0;
  for (int i = t; i < n; i += MS_THREADS) {
    const double r = (i > 0 ? fabs(e[i - 1]) : 0.0) + (i < n - 1 ? fabs(e[i]) : 0.0);
    lo = fmin(lo, d[i] - r);
    hi = fmax(hi, d[i] + r);
    if (i < n - 1) emax = fmax(emax, e[i] * e[i]);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    emax = fmax(emax, __shfl_xor_sync(0xffffffffu, emax, o));
  }
  if (lane == 0) {
    sh[0][warp] = lo;
    sh[1][warp] = hi;
    sh[2][warp] = emax;
  }
  __syncthreads();
  for (int w = 0; w < MS_THREADS / 32; ++w) {
    lo = fmin(lo, sh[0][w]);
    hi = fmax(hi, sh[1][w]);
    emax = fmax(emax, sh[2][w]);
  }
  const double span = fmax(fabs(lo), fabs(hi));
  lo -= 2.0 * DBL_EPSILON * span + 1e-300;
  hi += 2.0 * DBL_EPSILON * span + 1e-300;
  const double pivmin = 1e-290 * fmax(1.0, emax);
  const int m = n - 1 - j;  // ascending index
  const int points = MS_POINTS * C;
  const int mine = rank * MS_POINTS + warp * 16 + (lane & 15);
  cl.sync();  // every CTA of the cluster runs before its shared memory is written
  for (int it = 0; it < 64; ++it) {
    // every thread evaluates the same expressions, so lo, hi stay identical in all
    const double mid = 0.5 * (lo + hi);
    if (!(mid > lo && mid < hi)) break;  // neighbours: no point between them
    const double w = (hi - lo) / (double)(points + 1);
    const double x = lo + w * (double)(mine + 1);
    const bool in = x > lo && x < hi;
    const bool above = sturm_count_lt(d, e2, n, in ? x : lo, pivmin, lane) > m && in;
    const unsigned up = __ballot_sync(0xffffffffu, above) & 0xffffu;
    if (lane < C) *cl.map_shared_rank(&masks[it & 1][rank][warp], lane) = up;
    cl.sync();  // the masks of every CTA; those of the round before last are no longer read
    // counts grow with the point index: the first point above m
    int f = points;
    for (int c = C - 1; c >= 0; --c)
      for (int ww = MS_THREADS / 32 - 1; ww >= 0; --ww) {
        const unsigned u = masks[it & 1][c][ww];
        if (u) f = c * MS_POINTS + 16 * ww + __ffs(u) - 1;
      }
    const double nlo = f == 0 ? lo : lo + w * (double)f;
    const double nhi = f == points ? hi : lo + w * (double)(f + 1);
    if (!(nhi - nlo < hi - lo)) break;  // no progress: the bracket is a few ulps wide
    lo = nlo;
    hi = nhi;
  }
  if (rank == 0 && t == 0) evals[j] = 0.5 * (lo + hi);
}

// Eigenvector j of T by inverse iteration, one CTA per eigenvector.  Inside a
// cluster of close eigenvalues the shifts are separated as dstein does, so each
// member starts from a distinct shift; the cluster's vectors are made orthonormal
// and rotated afterwards (cluster_rr_kernel).  Thread 0 runs the pivoted
// tridiagonal LU of T - shift I (the dgttrf recurrence) and the triangular solves,
// which are sequential by nature, on arrays in shared memory (or in this CTA's
// slice of global scratch when n is large); the CTA does what is not.
// Thread 0's chain bounds it: an FP64 instruction takes ~66 cycles and a division ten of them, so
// the LU's recurrence carries numerators over a common denominator (four instructions a row, the
// divisions follow side by side), the solves' rows carry one and two, and operands are loaded a
// row ahead.  24 vectors, n = 289: 477 -> 279 us; n = 1089: 1,757 -> 1,002 us.
constexpr int IV_THREADS = 128;
constexpr int IV_ITERS = 4;

__device__ __forceinline__ double iv_ortol(const double* d, const double* e, int n, double* red) {
  double t = 0.0;
  for (int i = threadIdx.x; i < n; i += IV_THREADS)
    t = fmax(t, fabs(d[i]) + (i > 0 ? fabs(e[i - 1]) : 0.0) + (i < n - 1 ? fabs(e[i]) : 0.0));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) t = fmax(t, __shfl_xor_sync(0xffffffffu, t, o));
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = t;
  __syncthreads();
  double r = 0.0;
  for (int w = 0; w < IV_THREADS / 32; ++w) r = fmax(r, red[w]);
  __syncthreads();
  return r;
}

// Shared-memory path: [dl, dd, du, du2, z] (5n doubles) + n pivot bytes.  Global
// path (large n): this CTA's slice of `scratch`, [dl, dd, du, du2, z, pivot] as 6n
// doubles; vectors j0 .. j0 + gridDim.x - 1.
template <bool SMEM>
__global__ void __launch_bounds__(IV_THREADS) invvec_kernel(const double* __restrict__ d,
                                                            const double* __restrict__ e, int n, int j0,
                                                            const double* __restrict__ evals, double* __restrict__ Z,
                                                            double* __restrict__ scratch) {
  extern __shared__ __align__(16) double ivs[];
  __shared__ double red[32];
  const int j = j0 + blockIdx.x;
  double* base = SMEM ? ivs : scratch + (size_t)blockIdx.x * 6 * n;
  double* dl = base;           // L multipliers
  double* dd = base + n;       // U diagonal, as its reciprocal
  double* du = base + 2 * n;   // U first super-diagonal, over the diagonal
  double* du2 = base + 3 * n;  // U second super-diagonal, over the diagonal
  double* z = base + 4 * n;
  unsigned char* pivb = reinterpret_cast<unsigned char*>(base + 5 * n);  // SMEM: bytes
  double* pivd = base + 5 * n;                                           // global: doubles
  const double tnorm = iv_ortol(d, e, n, red);
  const double ortol = 1e-3 * tnorm;
  const double eps = DBL_EPSILON;
  const double tiny = eps * fmax(tnorm, 1e-300);
  // the shift of member j: dstein's perturbation applied along its cluster
  double lam = evals[j];
  {
    int c0 = j;
    while (c0 > 0 && fabs(evals[c0 - 1] - evals[c0]) <= ortol) --c0;
    double prev = evals[c0];
    for (int i = c0 + 1; i <= j; ++i) {
      double li = evals[i];
      const double pert = 10.0 * eps * fmax(fabs(li), tnorm * 1e-3);
      if (prev - li < pert) li = prev - pert;
      prev = li;
    }
    lam = prev;
  }
  // deterministic start vector
  for (int i = threadIdx.x; i < n; i += IV_THREADS) {
    unsigned h = (unsigned)(i * 2654435761u) ^ (unsigned)((j + 1) * 40503u);
    h ^= h >> 13;
    h *= 0x5bd1e995u;
    h ^= h >> 15;
    z[i] = ((double)(h & 0xffffff) / 16777216.0) - 0.5;
  }
  if (threadIdx.x == 0) {
    // row i of U before its elimination: a / s on the diagonal, b / s past it
    double a = d[0] - lam, b = n > 1 ? e[0] : 0.0, s = 1.0;
    double l = b, dn = n > 1 ? d[1] : 0.0;  // e[i], d[i + 1]
    for (int i = 0; i < n - 1; ++i) {
      const double un = i < n - 2 ? e[i + 1] : 0.0, dnn = i < n - 2 ? d[i + 2] : 0.0;
      const double g = l * s;
      const long long ab = __double_as_longlong(a) & 0x7fffffffffffffffll,
                      gb = __double_as_longlong(g) & 0x7fffffffffffffffll;
      const bool sw = ab < gb;  // |a / s| < |e[i]|
      if (!sw && ab == 0) a = tiny * s;
      dd[i] = a;
      du[i] = b;
      dl[i] = s;
      if (SMEM) pivb[i] = sw ? 1 : 0;
      else pivd[i] = sw ? 1.0 : 0.0;
      // kept: (dn a - l b) / a, un a / a; exchanged: (b l - a dn) / (s l), -a un / (s l)
      const long long flip = sw ? (long long)0x8000000000000000ull : 0;
      const double na = fma(dn - lam, a, -(l * b)), nb = un * a;
      s = sw ? g : a;
      a = __longlong_as_double(__double_as_longlong(na) ^ flip);
      b = __longlong_as_double(__double_as_longlong(nb) ^ flip);
      const unsigned ex = ((unsigned)__double2hiint(s) >> 20) & 0x7FFu;
      if (ex - 767u >= 512u) {  // s outside [2^-256, 2^256): all three by a power of two (exact)
        const double f = ex >= 1279u ? 0x1p-256 : 0x1p256;
        a *= f;
        b *= f;
        s *= f;
      }
      l = un;
      dn = dnn;
    }
    dd[n - 1] = a;
    dl[n - 1] = s;
  }
  __syncthreads();
  // the multipliers; U's rows over their diagonal (clamped away from zero) and its reciprocal
  for (int i = threadIdx.x; i < n; i += IV_THREADS) {
    const double s = dl[i], a = dd[i], b = du[i];
    const bool sw = i < n - 1 && (SMEM ? pivb[i] != 0 : pivd[i] != 0.0);
    double v = a / s, f = 0.0, u = 0.0, u2 = 0.0;
    if (sw) {
      f = v / e[i];
      v = e[i];
      u = d[i + 1] - lam;
      u2 = i < n - 2 ? e[i + 1] : 0.0;
    } else {
      if (v == 0.0) v = tiny;
      if (i < n - 1) {
        f = e[i] / v;
        u = b / s;
      }
    }
    if (fabs(v) < tiny) v = v < 0.0 ? -tiny : tiny;
    const double r = 1.0 / v;
    dl[i] = f;
    dd[i] = r;
    du[i] = u * r;
    du2[i] = u2 * r;
  }
  __syncthreads();
  for (int it = 0; it < IV_ITERS; ++it) {
    if (threadIdx.x == 0) {  // L
      double cur = z[0], zn = z[min(1, n - 1)], f = dl[0];
      bool sw = n > 1 && (SMEM ? pivb[0] != 0 : pivd[0] != 0.0);
      for (int i = 0; i < n - 1; ++i) {
        const int i1 = min(i + 1, n - 2);
        const double zn2 = z[min(i + 2, n - 1)], f1 = dl[i1];
        const bool sw1 = SMEM ? pivb[i1] != 0 : pivd[i1] != 0.0;
        const double p = sw ? zn : cur, q = sw ? cur : zn;
        z[i] = p;
        cur = fma(-f, p, q);
        zn = zn2;
        f = f1;
        sw = sw1;
      }
      z[n - 1] = cur;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += IV_THREADS) z[i] *= dd[i];
    __syncthreads();
    if (threadIdx.x == 0) {  // U, rows over their diagonal
      double z1 = z[n - 1], z2 = 0.0;
      int i1 = max(n - 2, 0);
      double t = z[i1], u = du[i1], u2 = du2[i1];
      for (int i = n - 2; i >= 0; --i) {
        i1 = max(i - 1, 0);
        const double tn = z[i1], un = du[i1], u2n = du2[i1];
        const double v = fma(-u, z1, fma(-u2, z2, t));
        z[i] = v;
        z2 = z1;
        z1 = v;
        t = tn;
        u = un;
        u2 = u2n;
      }
    }
    __syncthreads();
    double sq = 0.0;
    for (int i = threadIdx.x; i < n; i += IV_THREADS) sq += z[i] * z[i];
    sq = block_sum<IV_THREADS>(sq, red);
    const double inv = sq > 0.0 ? 1.0 / sqrt(sq) : 0.0;
    for (int i = threadIdx.x; i < n; i += IV_THREADS) z[i] *= inv;
    __syncthreads();
  }
  for (int i = threadIdx.x; i < n; i += IV_THREADS) Z[(size_t)j * n + i] = z[i];
}

// Clusters of close eigenvalues (|lambda_{i-1} - lambda_i| <= 1e-3 ||T||, the
// inverse-iteration cluster rule; on a flat spectrum it chains many members): the
// members' vectors Z_c are orthonormalised by Cholesky QR applied twice (Gram matrix
// G = Z_c^T Z_c = L L^T, Z_c <- Z_c L^-T), then rotated by the eigenvectors of the
// Rayleigh quotient H = Z_c^T T Z_c (cyclic Jacobi), ordered by descending Ritz
// value, so each member is the eigenvector of its own eigenvalue, not a mixture.
// The Gram and Rayleigh matrices are formed with one warp per entry pair and every
// row update is one thread per vector component, so the work is parallel.  A cluster
// larger than RR_MAXC (the near-zero tail of a rank-deficient TCC), or one whose
// Gram matrix is not numerically positive definite, is orthonormalised by modified
// Gram-Schmidt (two passes) instead, without the rotation in the first case.
// One CTA per cluster: CTA j works only if a cluster starts at j.  Chains of divisions and roots bound
// it (some ten FP64 instructions of ~66 cycles each), so nothing but those is left to one thread: the
// factorisation with a thread per row and a rotation by two reciprocal roots, 24 vectors of the
// usual quasar source, took 287 -> 204 us at n = 289 and 221 -> 184 at n = 1089.
constexpr int RR_THREADS = 256, RR_MAXC = 48;

// y_i = (T z)_i for the symmetric tridiagonal T
__device__ __forceinline__ double tri_mul(const double* d, const double* e, const double* z, int n, int i) {
  double y = d[i] * z[i];
  if (i > 0) y += e[i - 1] * z[i - 1];
  if (i < n - 1) y += e[i] * z[i + 1];
  return y;
}

// S[a][b] = z_a . (T z_b) (withT) or z_a . z_b over the c x c lower triangle, mirrored;
// one warp per pair
__device__ void rr_pairs(const double* d, const double* e, const double* Zc, int n, int c, bool withT,
                         double (*S)[RR_MAXC + 1]) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int np = c * (c + 1) / 2;
  for (int p = warp; p < np; p += RR_THREADS / 32) {
    int a, b;
    tri_tile(p, a, b);
    const double* za = Zc + (size_t)a * n;
    const double* zb = Zc + (size_t)b * n;
    // four independent partial sums: four loads of each row in flight per lane
    double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
    int i = lane;
    if (withT) {
      for (; i + 96 < n; i += 128) {
        s0 += za[i] * tri_mul(d, e, zb, n, i);
        s1 += za[i + 32] * tri_mul(d, e, zb, n, i + 32);
        s2 += za[i + 64] * tri_mul(d, e, zb, n, i + 64);
        s3 += za[i + 96] * tri_mul(d, e, zb, n, i + 96);
      }
      for (; i < n; i += 32) s0 += za[i] * tri_mul(d, e, zb, n, i);
    } else {
      for (; i + 96 < n; i += 128) {
        s0 += za[i] * zb[i];
        s1 += za[i + 32] * zb[i + 32];
        s2 += za[i + 64] * zb[i + 64];
        s3 += za[i + 96] * zb[i + 96];
      }
      for (; i < n; i += 32) s0 += za[i] * zb[i];
    }
    double sd = (s0 + s1) + (s2 + s3);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sd += __shfl_xor_sync(0xffffffffu, sd, o);
    if (lane == 0) {
      S[a][b] = sd;
      S[b][a] = sd;
    }
  }
}

__global__ void __launch_bounds__(RR_THREADS) cluster_rr_kernel(const double* __restrict__ d,
                                                                const double* __restrict__ e, int n, int nk,
                                                                const double* __restrict__ evals,
                                                                double* __restrict__ Z) {
  __shared__ double red[32];
  __shared__ double H[RR_MAXC][RR_MAXC + 1];
  __shared__ double V[RR_MAXC][RR_MAXC + 1];
  __shared__ double s_inv[RR_MAXC], s_diag;
  __shared__ int s_order[RR_MAXC];
  double tn = 0.0;
  for (int i = threadIdx.x; i < n; i += RR_THREADS)
    tn = fmax(tn, fabs(d[i]) + (i > 0 ? fabs(e[i - 1]) : 0.0) + (i < n - 1 ? fabs(e[i]) : 0.0));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) tn = fmax(tn, __shfl_xor_sync(0xffffffffu, tn, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = tn;
  __syncthreads();
  double tnorm = 0.0;
  for (int w = 0; w < RR_THREADS / 32; ++w) tnorm = fmax(tnorm, red[w]);
  __syncthreads();
  const double ortol = 1e-3 * tnorm;
  const int c0 = blockIdx.x;
  if (c0 > 0 && fabs(evals[c0 - 1] - evals[c0]) <= ortol) return;  // not a cluster start
  int c1 = c0 + 1;
  while (c1 < nk && fabs(evals[c1 - 1] - evals[c1]) <= ortol) ++c1;
  const int c = c1 - c0;
  if (c < 2) return;
  double* Zc = Z + (size_t)c0 * n;
  bool ok = c <= RR_MAXC;
  // Cholesky QR, twice
  for (int pass = 0; ok && pass < 2; ++pass) {
    rr_pairs(d, e, Zc, n, c, false, H);
    __syncthreads();
    // H <- L (lower), in place, a column at a time with a thread per row; s_inv: 1 / L_aa
    ok = true;
    for (int a = 0; a < c && ok; ++a) {
      const int r = a + (int)threadIdx.x;
      double v = 0.0;
      if (r < c) {
        v = H[r][a];
        for (int b = 0; b < a; ++b) v = fma(-H[r][b], H[a][b], v);
        if (r == a) s_diag = v;
      }
      __syncthreads();
      const double diag = s_diag;
      ok = diag > 1e-24;
      if (ok && r < c) {
        const double root = sqrt(diag), inv = 1.0 / root;
        H[r][a] = r == a ? root : v * inv;
        if (r == a) s_inv[a] = inv;
      }
      __syncthreads();
    }
    if (!ok) break;
    // z_i <- L^-1 z_i for every component i (forward substitution)
    for (int i = threadIdx.x; i < n; i += RR_THREADS) {
      double y[RR_MAXC];
      for (int a = 0; a < c; ++a) {
        double v = Zc[(size_t)a * n + i];
        for (int b = 0; b < a; ++b) v -= H[a][b] * y[b];
        y[a] = v * s_inv[a];
      }
      for (int a = 0; a < c; ++a) Zc[(size_t)a * n + i] = y[a];
    }
    __syncthreads();
  }
  if (!ok) {  // modified Gram-Schmidt, two passes
    for (int pass = 0; pass < 2; ++pass)
      for (int a = 0; a < c; ++a) {
        double* za = Zc + (size_t)a * n;
        for (int b = 0; b < a; ++b) {
          const double* zb = Zc + (size_t)b * n;
          double sd = 0.0;
          for (int i = threadIdx.x; i < n; i += RR_THREADS) sd += zb[i] * za[i];
          sd = block_sum<RR_THREADS>(sd, red);
          for (int i = threadIdx.x; i < n; i += RR_THREADS) za[i] -= sd * zb[i];
          __syncthreads();
        }
        double sq = 0.0;
        for (int i = threadIdx.x; i < n; i += RR_THREADS) sq += za[i] * za[i];
        sq = block_sum<RR_THREADS>(sq, red);
        const double inv = sq > 0.0 ? 1.0 / sqrt(sq) : 0.0;
        for (int i = threadIdx.x; i < n; i += RR_THREADS) za[i] *= inv;
        __syncthreads();
      }
    if (c > RR_MAXC) return;
  }
  // Rayleigh-Ritz: H = Z_c^T T Z_c
  rr_pairs(d, e, Zc, n, c, true, H);
  for (int i = threadIdx.x; i < c * c; i += RR_THREADS) V[i / c][i % c] = (i / c == i % c) ? 1.0 : 0.0;
  __syncthreads();
  // cyclic Jacobi on the c x c symmetric H, V accumulating the rotations, in
  // round-robin order: a sweep is cp - 1 rounds (cp = c rounded up to even; index
  // c is a dummy when c is odd), each rotating cp/2 disjoint pairs (p, q) at once.
  // A pair's rotation is computed from the matrix before its round (the 2 x 2
  // block of (p, q) is touched by no other rotation of the round), then all
  // column rotations (H <- H J, V <- V J) and all row rotations (H <- J^T H)
  // are applied by the whole block.  Same rotation formulas as the serial
  // cyclic method; the circle method pairs every (p, q) once per sweep.
  {
    __shared__ double s_cs[RR_MAXC / 2], s_sn[RR_MAXC / 2];
    __shared__ int s_p[RR_MAXC / 2], s_q[RR_MAXC / 2];
    const int cp = c + (c & 1), np = cp / 2;
    for (int sweep = 0; sweep < 30; ++sweep) {
      double off = 0.0, dia = 0.0;
      for (int i = threadIdx.x; i < c * c; i += RR_THREADS) {
        const int x = i / c, y = i - x * c;
        const double v = H[x][y];
        if (x == y) dia = fma(v, v, dia);
        else if (x < y) off = fma(v, v, off);
      }
      off = block_sum<RR_THREADS>(off, red);
      dia = block_sum<RR_THREADS>(dia, red);
      if (off <= 1e-32 * dia) break;
      for (int r = 0; r < cp - 1; ++r) {
        if (threadIdx.x < np) {
          const int i = threadIdx.x, j = cp - 1 - i;
          const int a = i == 0 ? 0 : (i - 1 + r) % (cp - 1) + 1;
          const int b = (j - 1 + r) % (cp - 1) + 1;
          const int pp = min(a, b), qq = max(a, b);
          double cs = 1.0, sn = 0.0;
          if (qq < c) {
            const double apq = H[pp][qq];
            if (apq != 0.0) {
              const double h = H[qq][qq] - H[pp][pp], g2 = 2.0 * apq, rr = fma(h, h, g2 * g2);
              if (rr > 1e-280 && rr < 1e280) {
                // cos 2 phi = |h| / r, sin 2 phi = +-2 apq / r: two reciprocal roots instead of three
                // divisions and two roots in a chain
                const double ir = rsqrt(rr), c2 = fma(0.5 * fabs(h), ir, 0.5), rc = rsqrt(c2);
                cs = c2 * rc;
                sn = (h >= 0.0 ? 0.5 : -0.5) * g2 * ir * rc;
              } else {  // the squares leave the range
                const double theta = h / g2;
                const double t = (theta >= 0.0 ? 1.0 : -1.0) / (fabs(theta) + sqrt(theta * theta + 1.0));
                cs = 1.0 / sqrt(t * t + 1.0);
                sn = t * cs;
              }
            }
          }
          s_p[i] = pp;
          s_q[i] = qq;
          s_cs[i] = cs;
          s_sn[i] = sn;
        }
        __syncthreads();
        for (int w = threadIdx.x; w < np * c; w += RR_THREADS) {  // columns p, q of H and V
          const int i = w / c, k = w - i * c, pp = s_p[i], qq = s_q[i];
          if (qq < c) {
            const double cs = s_cs[i], sn = s_sn[i];
            const double hkp = H[k][pp], hkq = H[k][qq];
            H[k][pp] = cs * hkp - sn * hkq;
            H[k][qq] = sn * hkp + cs * hkq;
            const double vkp = V[k][pp], vkq = V[k][qq];
            V[k][pp] = cs * vkp - sn * vkq;
            V[k][qq] = sn * vkp + cs * vkq;
          }
        }
        __syncthreads();
        for (int w = threadIdx.x; w < np * c; w += RR_THREADS) {  // rows p, q of H
          const int i = w / c, k = w - i * c, pp = s_p[i], qq = s_q[i];
          if (qq < c) {
            const double cs = s_cs[i], sn = s_sn[i];
            const double hpk = H[pp][k], hqk = H[qq][k];
            H[pp][k] = cs * hpk - sn * hqk;
            H[qq][k] = sn * hpk + cs * hqk;
          }
        }
        __syncthreads();
      }
    }
  }
  if (threadIdx.x == 0) {  // descending Ritz values
    for (int a = 0; a < c; ++a) s_order[a] = a;
    for (int a = 1; a < c; ++a) {
      const int key = s_order[a];
      int b = a - 1;
      while (b >= 0 && H[s_order[b]][s_order[b]] < H[key][key]) {
        s_order[b + 1] = s_order[b];
        --b;
      }
      s_order[b + 1] = key;
    }
  }
  __syncthreads();
  // Z_c <- Z_c V (columns in descending Ritz order), one thread per component
  for (int i = threadIdx.x; i < n; i += RR_THREADS) {
    double x[RR_MAXC];
    for (int b = 0; b < c; ++b) x[b] = Zc[(size_t)b * n + i];
    for (int a = 0; a < c; ++a) {
      const int col = s_order[a];
      double acc = 0.0;
      for (int b = 0; b < c; ++b) acc += x[b] * V[b][col];
      Zc[(size_t)a * n + i] = acc;
    }
  }
}

// y_j = H_0 H_1 ... H_{n-2} z_j for every eigenvector j; H_k = I - tau_k v_k v_k^H acting on rows
// k+1..n-1, v_k packed contiguously in vpack.  The reflectors are taken WY_NB at a time in compact
// WY form: H_k0 ... H_{k0+nb-1} = I - V T V^H (V the block's reflectors as columns, T upper
// triangular: T_jj = tau_j, T[0:j, j] = -tau_j T[0:j, 0:j] (V[:, 0:j]^H v_j)), so a block costs one
// exchange (w = V^H y summed over the rows, u = T w, y -= V u) instead of one per reflector, for
// the same FP64 work.
constexpr int WY_NB = 16, WY_THREADS = 256, WY_CLUSTER = 4;

// T of every block (one cluster per block): the Gram products v_i^H v_j (i < j, over v_j's support)
// one warp per pair, the pairs shared out over the cluster; then the triangular recurrence, a column
// at a time over the rows and summands, in the first CTA.  FP64-bound: one CTA per block, with the
// recurrence on one thread, took 242 us at n = 289 and 340 at n = 1089; this takes 33 and 87.
__global__ void __launch_bounds__(WY_THREADS) wy_t_kernel(const double2* __restrict__ vpack,
                                                          const double2* __restrict__ tau, int n,
                                                          double2* __restrict__ Tg) {
  namespace cg = cooperative_groups;
  __shared__ double G[WY_NB][WY_NB][2];
  __shared__ double2 T[WY_NB][WY_NB + 1];
  cg::cluster_group cl = cg::this_cluster();
  const int C = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  const int b = blockIdx.x / C, k0 = b * WY_NB, nbb = min(WY_NB, n - 1 - k0);
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int np = nbb * (nbb - 1) / 2;
  cl.sync();  // every CTA of the cluster runs before its shared memory is written
  for (int p = warp * C + rank; p < np; p += WY_THREADS / 32 * C) {
    int j = 1;
    while ((j + 1) * j / 2 <= p) ++j;  // p = j (j - 1) / 2 + i, i < j
    const int i = p - j * (j - 1) / 2;
    const int ki = k0 + i, kj = k0 + j;
    const double2* vi = vpack + vpack_off(n, ki) - (ki + 1);  // v_i[r], r in [ki+1, n)
    const double2* vj = vpack + vpack_off(n, kj) - (kj + 1);
    double sr = 0.0, si = 0.0;  // conj(v_i) . v_j
#pragma unroll 4
    for (int r = kj + 1 + lane; r < n; r += 32) {
      const double2 a = vi[r], c = vj[r];
      sr = fma(a.x, c.x, fma(a.y, c.y, sr));
      si = fma(a.x, c.y, fma(-a.y, c.x, si));
    }
    const double v = pair_sum(sr, si, lane);
    if ((lane & 15) == 0) *cl.map_shared_rank(&G[i][j][lane >> 4], 0) = v;
  }
  cl.sync();
  if (rank != 0) return;
  const int ii = t >> 4, l = t & 15;
  T[ii][l] = ii == l && ii < nbb ? tau[k0 + ii] : make_double2(0.0, 0.0);
  __syncthreads();
  for (int jj = 1; jj < nbb; ++jj) {
    double2 z = make_double2(0.0, 0.0);
    if (ii <= l && l < jj) z = zmul(T[ii][l], make_double2(G[l][jj][0], G[l][jj][1]));
    const double s = half_pair_sum(z.x, z.y, lane);
    const double im = __shfl_down_sync(0xffffffffu, s, 8);
    const double2 tj = T[jj][jj];
    if (l == 0 && ii < jj) {
      const double2 v = zmul(tj, make_double2(s, im));
      T[ii][jj] = make_double2(-v.x, -v.y);
    }
    __syncthreads();
  }
  Tg[(size_t)b * WY_NB * WY_NB + t] = T[ii][l];
}

// One cluster of CTAs per vector; the rows go to the CTAs 32 at a time in turn, which spreads the
// shrinking support of the reflectors evenly, and stay in shared memory for the whole loop.  Per
// block: each warp forms two entries of w over the CTA's rows, the CTAs exchange the partial w
// through the cluster's shared memory (one cluster barrier; two buffers, by parity), every CTA forms u,
// and each warp updates 32 rows.  FP64-bound (a quarter of an SM issues one warp instruction per ~66
// cycles), so a vector takes as many SMs as there are for it; on one SM each, 24 vectors took 467 us
// at n = 289 and 2,674 at n = 1089, now 144 and 648.
constexpr int BK_CMAX = 8;

size_t backtransform_smem(int n, int C) {
  const int chunks = (n + 31) / 32;
  return (size_t)((chunks + C - 1) / C) * 32 * sizeof(double2);
}

__global__ void __launch_bounds__(WY_THREADS) backtransform_kernel(const double2* __restrict__ vpack, int n,
                                                                   const double2* __restrict__ Tg,
                                                                   const double* __restrict__ Z,
                                                                   double2* __restrict__ Y) {
  namespace cg = cooperative_groups;
  extern __shared__ __align__(16) double2 s_y[];          // [local chunk][32]
  __shared__ double s_part[2][BK_CMAX][2 * WY_NB];        // w of every CTA: re, im interleaved
  __shared__ double2 s_w[WY_NB], s_u[WY_NB];
  cg::cluster_group cl = cg::this_cluster();
  const int C = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  const int j = blockIdx.x / C, t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int chunks = (n + 31) / 32;
  const int mine = (chunks - rank + C - 1) / C;  // chunks rank, rank + C, ...
  for (int q = warp; q < mine; q += WY_THREADS / 32) {
    const int r = (rank + q * C) * 32 + lane;
    s_y[q * 32 + lane] = make_double2(r < n ? Z[(size_t)j * n + r] : 0.0, 0.0);
  }
  cl.sync();  // s_y; also, every CTA of the cluster runs before its shared memory is written
  const int nblk = (n - 1 + WY_NB - 1) / WY_NB;
  for (int b = nblk - 1; b >= 0; --b) {
    const int k0 = b * WY_NB, nbb = min(WY_NB, n - 1 - k0);
    // the first local chunk that reaches past row k0 (c = rank + q C with 32 c + 31 > k0)
    const int cf = (k0 + 1) / 32, q0 = max(0, (cf - rank + C - 1) / C);
    const double2 tv = Tg[(size_t)b * WY_NB * WY_NB + t];
    {
      const int i0 = 2 * warp, i1 = i0 + 1;
      // v_i[r] = vpack[base_i + r] for r in (k0 + i, n)
      const double2* v0 = vpack + ((long long)vpack_off(n, k0 + (i0 < nbb ? i0 : 0)) - (k0 + (i0 < nbb ? i0 : 0) + 1));
      const double2* v1 = vpack + ((long long)vpack_off(n, k0 + (i1 < nbb ? i1 : 0)) - (k0 + (i1 < nbb ? i1 : 0) + 1));
      const int f0 = i0 < nbb ? k0 + i0 : n, f1 = i1 < nbb ? k0 + i1 : n;
      double a0r = 0.0, a0i = 0.0, a1r = 0.0, a1i = 0.0;
#pragma unroll 3
      for (int q = q0; q < mine; ++q) {
        const int r = (rank + q * C) * 32 + lane;
        const double2 yy = s_y[q * 32 + lane];
        double2 p = make_double2(0.0, 0.0), s = p;
        if (r > f0 && r < n) p = v0[r];
        if (r > f1 && r < n) s = v1[r];
        a0r = fma(p.x, yy.x, fma(p.y, yy.y, a0r));  // conj(v) y
        a0i = fma(p.x, yy.y, fma(-p.y, yy.x, a0i));
        a1r = fma(s.x, yy.x, fma(s.y, yy.y, a1r));
        a1i = fma(s.x, yy.y, fma(-s.y, yy.x, a1i));
      }
      // reflector i0 in lanes 0-15, i1 in 16-31, then their re and im in halves of those
      const bool hi = lane & 16;
      const double kr = (hi ? a1r : a0r) + __shfl_xor_sync(0xffffffffu, hi ? a0r : a1r, 16);
      const double ki = (hi ? a1i : a0i) + __shfl_xor_sync(0xffffffffu, hi ? a0i : a1i, 16);
      const double v = half_pair_sum(kr, ki, lane);
      // every lane of a group of eight holds its sum: lane c of the group writes to CTA c
      const int c = lane & 7;
      if (c < C) *cl.map_shared_rank(&s_part[b & 1][rank][4 * warp + (lane >> 3)], c) = v;
    }
    cl.sync();  // the parts of this block; nobody still reads those of the block before last
    if (t < 2 * WY_NB) {
      double v = s_part[b & 1][0][t];
      for (int c = 1; c < C; ++c) v += s_part[b & 1][c][t];
      reinterpret_cast<double*>(s_w)[t] = v;
    }
    __syncthreads();
    {  // u = T w: row t / 16, summand t % 16 (T is zero below its diagonal and past nbb)
      const double2 z = zmul(tv, s_w[t & 15]);
      const double s = half_pair_sum(z.x, z.y, lane);
      if ((lane & 7) == 0) reinterpret_cast<double*>(s_u)[2 * (t >> 4) + ((lane >> 3) & 1)] = s;
    }
    __syncthreads();
    for (int q = q0 + warp; q < mine; q += WY_THREADS / 32) {  // y -= V u
      const int r = (rank + q * C) * 32 + lane;
      double2 yy = s_y[q * 32 + lane];
      const double2* v = vpack + ((long long)vpack_off(n, k0) - (k0 + 1)) + r;
#pragma unroll
      for (int i = 0; i < WY_NB; ++i) {
        if (i < nbb) {
          double2 vv = make_double2(0.0, 0.0);
          if (r > k0 + i && r < n) vv = *v;
          const double2 u = s_u[i];
          yy.x = fma(-u.x, vv.x, fma(u.y, vv.y, yy.x));
          yy.y = fma(-u.x, vv.y, fma(-u.y, vv.x, yy.y));
          v += n - 2 - (k0 + i);  // the next reflector starts one row later and is one shorter
        }
      }
      s_y[q * 32 + lane] = yy;
    }
    __syncthreads();
  }
  for (int q = warp; q < mine; q += WY_THREADS / 32) {
    const int r = (rank + q * C) * 32 + lane;
    if (r < n) Y[(size_t)j * n + r] = s_y[q * 32 + lane];
  }
}

__global__ void output_kernel(const double2* __restrict__ Y, const double* __restrict__ evals, int n, int nk,
                              float* __restrict__ kr, float* __restrict__ ki, float* __restrict__ sc,
                              double2* __restrict__ k64, double* __restrict__ s64) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x, i = blockIdx.y;
  if (i >= nk) return;
  if (j < n) {
    const double2 v = Y[(size_t)i * n + (n - 1 - j)];
    kr[(size_t)i * n + j] = (float)v.x;
    ki[(size_t)i * n + j] = (float)v.y;
    if (k64) k64[(size_t)i * n + j] = v;
  }
  if (j == 0) {
    sc[i] = (float)evals[i];
    if (s64) s64[i] = evals[i];
  }
}

// `groups` clusters of C CTAs each
template <typename... P, typename... A>
static cudaError_t launch_clusters(void (*k)(P...), int groups, int C, int threads, size_t smem, cudaStream_t stream,
                                   A... args) {
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = (unsigned)C;
  at.val.clusterDim.y = at.val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(groups * C));
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k, P(args)...);
}

}  // namespace litho

using namespace litho;

extern "C" int litho_calc_kernels(litho_ctx* ctx, const double* tcc, int tccSize, int nk, float* krn_r, float* krn_i,
                                  float* scales, double* krn64, double* scales64, int mem) {
  if (ctx == nullptr) return LITHO_ERR_ARG;
  LITHO_ARG_CHECK(ctx, tcc && krn_r && krn_i && scales, "null pointer");
  LITHO_ARG_CHECK(ctx, tccSize >= 1 && tccSize <= 8192, "tccSize %d outside [1, 8192]", tccSize);
  LITHO_ARG_CHECK(ctx, nk >= 1 && nk <= tccSize, "nk %d outside [1, tccSize=%d]", nk, tccSize);
  LITHO_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  const int n = tccSize;
  const size_t nn = (size_t)n * n;
  const void* dtcc = nullptr;
  LITHO_RET(stage_in(ctx, ctx->tcc_c, tcc, nn * sizeof(double2), mem, &dtcc));
  LITHO_RET(ctx->eig_v.ensure(ctx, nn * sizeof(double2)));
  // workspace: vbuf, xbuf, tau (n double2 each); packed reflectors (n(n-1)/2
  // double2); per-CTA partial dots ((n+7)/8 double2); d, e (n double); evals (nk);
  // Z (nk*n double); inverse-iteration scratch (large n only: IV_CHUNK * 6n double);
  // Y (nk*n double2)
  const size_t iv_smem = (size_t)5 * n * sizeof(double) + n;
  const bool iv_in_smem = iv_smem <= 200 * 1024;  // (the solver kernels' own static shared memory: under 8 KB)
  constexpr int IV_CHUNK = 64;
  const size_t iv_scratch = iv_in_smem ? 0 : (size_t)IV_CHUNK * 6 * n * sizeof(double);
  const size_t vpack_bytes = (size_t)n * (n - 1) / 2 * sizeof(double2) + sizeof(double2);
  const size_t part_bytes = (size_t)((n + 7) / 8) * sizeof(double2);
  const size_t td_part_bytes = (size_t)2 * ctx->sm_count * sizeof(double) + 64;  // partials by parity, barrier count
  const size_t wbytes = 3 * n * sizeof(double2) + vpack_bytes + part_bytes + 3 * n * sizeof(double) + nk * sizeof(double) +
                        (size_t)nk * n * sizeof(double) + iv_scratch + (size_t)nk * n * sizeof(double2) +
                        (size_t)((n + WY_NB - 1) / WY_NB + 1) * WY_NB * WY_NB * sizeof(double2) +
                        (size_t)4 * n * sizeof(double2) + td_part_bytes + 19 * 64;
  LITHO_RET(ctx->eig_work.ensure(ctx, wbytes));
  char* w = ctx->eig_work.as<char>();
  auto take = [&](size_t b) {
    char* p = w;
    w += (b + 63) & ~size_t(63);
    return p;
  };
  double2* vbuf = reinterpret_cast<double2*>(take(n * sizeof(double2)));
  double2* xbuf = reinterpret_cast<double2*>(take(n * sizeof(double2)));
  double2* tau = reinterpret_cast<double2*>(take(n * sizeof(double2)));
  double2* vpack = reinterpret_cast<double2*>(take(vpack_bytes));
  double2* part = reinterpret_cast<double2*>(take(part_bytes));
  double* d = reinterpret_cast<double*>(take(n * sizeof(double)));
  double* e = reinterpret_cast<double*>(take(n * sizeof(double)));
  double* e2 = reinterpret_cast<double*>(take(n * sizeof(double)));
  double* ev = reinterpret_cast<double*>(take(nk * sizeof(double)));
  double* Z = reinterpret_cast<double*>(take((size_t)nk * n * sizeof(double)));
  double* ivs = iv_in_smem ? nullptr : reinterpret_cast<double*>(take(iv_scratch));
  double2* Y = reinterpret_cast<double2*>(take((size_t)nk * n * sizeof(double2)));
  const int wy_blocks = n > 1 ? (n - 1 + WY_NB - 1) / WY_NB : 0;
  double2* Tg = reinterpret_cast<double2*>(take((size_t)(wy_blocks > 0 ? wy_blocks : 1) * WY_NB * WY_NB * sizeof(double2)));
  double2* td_vec = reinterpret_cast<double2*>(take((size_t)4 * n * sizeof(double2)));  // x and pivot rows, by parity
  double* td_part = reinterpret_cast<double*>(take(td_part_bytes));
  double2* A = ctx->eig_v.as<double2>();
  {
    // hermitize, reduction (one cooperative launch, or two per reflector, last diagonal and e^2),
    // multisection, inverse iteration (one launch, or one per chunk of IV_CHUNK vectors), cluster
    // Rayleigh-Ritz, WY factors, back-transform
    const int iv_launches = iv_in_smem ? 1 : (nk + IV_CHUNK - 1) / IV_CHUNK;
    const int G = std::min(n, ctx->sm_count);
    const size_t td_smem = tridiag_smem(n, G);
    const bool coop = n > 1 && td_smem <= TD_MAX_SMEM && (n + G - 1) / G <= TD_MAX_ROWS;
    StageScope sc(ctx, LITHO_STAGE_EIG, (coop ? 1 : 2 * n) + 4 + (wy_blocks > 0 ? 1 : 0) + iv_launches);
    hermitize_kernel<<<dim3((n + 127) / 128, n), 128, 0, ctx->stream>>>(static_cast<const double2*>(dtcc), A, n);
    LITHO_CUDA_TRY(ctx, cudaGetLastError());
    LITHO_CUDA_TRY(ctx, cudaMemsetAsync(e, 0, n * sizeof(double), ctx->stream));
    if (coop) {
      int* err = nullptr;
      LITHO_RET(tc_err_flag_public(ctx, &err));
      unsigned* count = reinterpret_cast<unsigned*>(td_part + 2 * G);
      LITHO_CUDA_TRY(ctx, cudaMemsetAsync(count, 0, sizeof(unsigned), ctx->stream));
      LITHO_CUDA_TRY(ctx, allow_smem(tridiag_kernel, SMEM_MOST - (int)TD_MAX_SMEM));
      const double2* Ac = A;
      double2 *xg = td_vec, *rowbuf = td_vec + 2 * (size_t)n;
      int nn_ = n;
      void* args[] = {&Ac, &nn_, &vpack, &tau, &d, &e, &e2, &xg, &rowbuf, &td_part, &count, &err};
      // cooperative: all CTAs are resident at once, as their waits on one another need
      LITHO_CUDA_TRY(ctx, cudaLaunchCooperativeKernel((const void*)tridiag_kernel, dim3(G), dim3(TD_THREADS), args,
                                                      td_smem, ctx->stream));
    } else {
      for (int k = 0; k + 1 < n; ++k) {
        const int m = n - k - 1;
        const int nb = (m + 7) / 8;
        symv_hh_kernel<<<nb, 256, 0, ctx->stream>>>(A, n, k, vbuf, vpack, tau, d, e, xbuf, part);
        const int nt = (m + 31) / 32;
        her2_kernel<<<nt * (nt + 1) / 2, 256, 0, ctx->stream>>>(A, n, k, vbuf, xbuf, tau, part, nb);
      }
      LITHO_CUDA_TRY(ctx, cudaGetLastError());
      last_diag_kernel<<<1, 32, 0, ctx->stream>>>(A, n, d);
      square_kernel<<<(n + 255) / 256, 256, 0, ctx->stream>>>(e, e2, n - 1);
    }
    // four SMs per eigenvalue while there are as many; further eigenvalues take one each
    LITHO_CUDA_TRY(ctx, launch_clusters(multisect_kernel, nk, nk * MS_CMAX <= ctx->sm_count ? MS_CMAX : 1, MS_THREADS, 0,
                                        ctx->stream, (const double*)d, (const double*)e, (const double*)e2, n, ev));
    if (iv_in_smem) {
      LITHO_CUDA_TRY(ctx, allow_smem(invvec_kernel<true>, 1024));
      invvec_kernel<true><<<nk, IV_THREADS, iv_smem, ctx->stream>>>(d, e, n, 0, ev, Z, nullptr);
    } else {
      for (int j0 = 0; j0 < nk; j0 += IV_CHUNK)
        invvec_kernel<false><<<std::min(IV_CHUNK, nk - j0), IV_THREADS, 0, ctx->stream>>>(d, e, n, j0, ev, Z, ivs);
    }
    cluster_rr_kernel<<<nk, RR_THREADS, 0, ctx->stream>>>(d, e, n, nk, ev, Z);
    const double2 *cvpack = vpack, *ctau = tau, *cTg = Tg;
    if (wy_blocks > 0)
      LITHO_CUDA_TRY(ctx, launch_clusters(wy_t_kernel, wy_blocks, WY_CLUSTER, WY_THREADS, 0, ctx->stream, cvpack, ctau, n, Tg));
    // as many SMs per vector as there are, up to the portable cluster size and the row chunks; a fifth
    // of the SMs is left, as clusters don't fill every GPC (24 vectors, n = 1089: 648 us on clusters
    // of five, 783 on six and 710 on four)
    const int bc = std::max(1, std::min({BK_CMAX, ctx->sm_count * 4 / 5 / nk, (n + 31) / 32}));
    const size_t bt_smem = backtransform_smem(n, bc);
    LITHO_CUDA_TRY(ctx, allow_smem(backtransform_kernel, 8 * 1024));
    LITHO_CUDA_TRY(ctx, launch_clusters(backtransform_kernel, nk, bc, WY_THREADS, bt_smem, ctx->stream, cvpack, n, cTg,
                                        (const double*)Z, Y));
    LITHO_CUDA_TRY(ctx, cudaGetLastError());
  }
  float *okr = krn_r, *oki = krn_i, *osc = scales;
  double *ok64 = krn64, *os64 = scales64;
  if (mem == LITHO_MEM_HOST) {
    LITHO_RET(ctx->eig_info.ensure(ctx, (size_t)nk * n * (2 * sizeof(float) + sizeof(double2)) +
                                            nk * (sizeof(float) + sizeof(double)) + 256));
    char* o = ctx->eig_info.as<char>();
    ok64 = reinterpret_cast<double*>(o);
    o += (size_t)nk * n * sizeof(double2);
    os64 = reinterpret_cast<double*>(o);
    o += nk * sizeof(double);
    okr = reinterpret_cast<float*>(o);
    o += (size_t)nk * n * sizeof(float);
    oki = reinterpret_cast<float*>(o);
    o += (size_t)nk * n * sizeof(float);
    osc = reinterpret_cast<float*>(o);
  }
  {
    StageScope sc(ctx, LITHO_STAGE_UPLOAD);
    output_kernel<<<dim3((n + 127) / 128, nk), 128, 0, ctx->stream>>>(Y, ev, n, nk, okr, oki, osc,
                                                                     reinterpret_cast<double2*>(ok64), os64);
    LITHO_CUDA_TRY(ctx, cudaGetLastError());
  }
  if (mem == LITHO_MEM_HOST) {
    LITHO_CUDA_TRY(ctx, cudaMemcpyAsync(krn_r, okr, (size_t)nk * n * sizeof(float), cudaMemcpyDeviceToHost, ctx->stream));
    LITHO_CUDA_TRY(ctx, cudaMemcpyAsync(krn_i, oki, (size_t)nk * n * sizeof(float), cudaMemcpyDeviceToHost, ctx->stream));
    LITHO_CUDA_TRY(ctx, cudaMemcpyAsync(scales, osc, nk * sizeof(float), cudaMemcpyDeviceToHost, ctx->stream));
    if (krn64)
      LITHO_CUDA_TRY(ctx, cudaMemcpyAsync(krn64, ok64, (size_t)nk * n * sizeof(double2), cudaMemcpyDeviceToHost, ctx->stream));
    if (scales64)
      LITHO_CUDA_TRY(ctx, cudaMemcpyAsync(scales64, os64, nk * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
    LITHO_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
    LITHO_RET(tc_check_flag(ctx));
    for (int i = 0; i < nk; ++i)
      if (!std::isfinite(scales[i])) {
        set_error(ctx, LITHO_ERR_NAN, "non-finite eigenvalue %d", i);
        return LITHO_ERR_NAN;
      }
  }
  return LITHO_OK;
}
