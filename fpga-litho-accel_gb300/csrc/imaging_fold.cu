// The two FP32 transforms of the plain imaging form, folded four rows at a time (fold.hpp).
//
//   win_fold_kernel  W[v][u] = 1/(FxFy) sum_{y,x} m[y][x] e^{-2 pi i (u x'/Fx + v y'/Fy)}:
//                    the row sums first (over y, per mask column), each base row's four mask
//                    rows folded by eight additions into the operands of the even/odd cos and
//                    sin sums; then the short column sums of a CTA's columns.
//   fi_fold_kernel   image[Y][X] = T0 + sum_r 2 Re(e^{2 pi i r y'/Fy} T_r[X]): the even/odd cos
//                    and sin sums of a base row give four image rows by eight additions.
//
// Every sum stays in FP32 on the CUDA cores.  Per pixel the window takes (2Ny+1)/4 FMAs and two
// additions and the image (4Ny+1)/4 and two, a quarter of the unfolded contractions (which were
// bound by the FP32 pipe and by shared-memory reads), so up to Ny = 8 the 4 bytes per pixel of
// HBM bound both: 1024 masks of 1024^2 (4 GiB each way) measured 1172 -> 639 us (6.7 TB/s) for the
// window and 1299 -> 639 us for the image, 40 grey masks of 777 x 913 (rows at any alignment)
// 90 -> 34 and 51 -> 30 us.  At Ny = 16 the FMAs bound the image (44 of 2048^2: 195 us, 3.8 TB/s).
// Scalar FMAs: packed (f32x2) ones gave no higher rate here and cost register moves.
#include "litho_internal.cuh"
#include "fold.hpp"
#include "tc_common.cuh"

#include <algorithm>

namespace litho {

// element offsets of a base row's four rows, -1 where a row is outside
__device__ __forceinline__ int4 fold_offsets(int b, int Lx, int Ly, int Fy) {
  int o[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const FoldRange fr = fold_range(k, Ly, Fy);
    o[k] = (unsigned)(b - fr.lo) < (unsigned)fr.n ? fold_y(b, k, Ly, Fy) * Lx : -1;
  }
  return make_int4(o[0], o[1], o[2], o[3]);
}

// ---------------------------------------------------------------------------
// window DFT
// ---------------------------------------------------------------------------
// Template support: 2NY+1 sums per column.  Four columns per lane, so that a coefficient read (a broadcast
// takes shared memory a wavefront per word) serves four: 68 accumulator registers at NY = 8, in two CTAs of
// eight warps per SM; 132 at NY = 16, in two of four warps with a deeper ring.  (Two columns per lane and eight
// warps above NY = 8: 16 masks of 1999 x 2001 254 us, now 227; 200 of 1280^2 1,050, now 957; 100 of
// 1100^2 487, now 438; 10 of 2048^2 147, now 130; one 55.7, now 60.)
constexpr int WF_CPL = 4;
constexpr int wf_stride(int NY) { return 2 * NY; }
constexpr int wf_warps(int NY) { return NY <= 8 ? 8 : 4; }
constexpr int wf_st(int NY) { return NY <= 8 ? 4 : 8; }  // ring stages: three, seven base rows (2 KB each) of every warp in flight
// base rows whose coefficients and row offsets are staged at a time
constexpr int wf_stage(int NY) { return (NY <= 8 ? 40 : 18) * 1024 / (wf_stride(NY) * 4 + 16) / 8 * 8; }

static int wf_ny(int Ny) { return Ny <= 2 ? 2 : Ny <= 4 ? 4 : Ny <= 8 ? 8 : Ny <= 12 ? 12 : Ny <= 16 ? 16 : -1; }

// coef[b][.]: cos(n t) for n = 1..NY, then sin(n t), t = 2 pi b/Fy; zero past Ny
__global__ void wf_coef_kernel(float* __restrict__ coef, int nb, int NY, int Ny, int Fy) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x, e = blockIdx.y, n = e % NY + 1;
  if (b >= nb) return;
  float c = 0.f, s = 0.f;
  if (n <= Ny) cis_round((long long)n * b, Fy, &c, &s);
  coef[(size_t)b * wf_stride(NY) + e] = e < NY ? c : s;
}

template <int NY>
struct WinFold {
  static constexpr int CPL = WF_CPL, COLS = 32 * CPL, KS = wf_stride(NY), NR = 2 * NY + 1;
  static constexpr int WARPS = wf_warps(NY), THREADS = 32 * WARPS, ST = wf_st(NY), AHEAD = (ST - 1) * WARPS;
  static constexpr int RB = COLS + 4;       // ring row (floats): the columns and one granule of misalignment
  static constexpr int RING = WARPS * ST * 4 * RB;
  static constexpr int RS = COLS + 4;       // row stride of the summed row sums (floats)
  static constexpr int TS = COLS + 2;       // row stride of the column twiddles (float2)
  static constexpr int ZERO = RB + 4;       // a row of zeros, padded to 16 bytes
  static constexpr int RED = WARPS * NR * COLS;  // floats of the warps' sums
  static constexpr int BARS = WARPS * ST * 2;  // floats of the ring's barriers
};

template <int NY>
static size_t win_fold_smem(int Nx, int rows) {
  using P = WinFold<NY>;
  const size_t tw = (size_t)(Nx + 1) * P::TS * 2;
  const int st = std::min(rows, wf_stage(NY));
  const size_t loop = (size_t)P::RING + (size_t)(st + P::AHEAD) * 4 + (size_t)st * P::KS;
  const size_t sums = (size_t)P::RED + (size_t)P::NR * P::RS;
  return (P::BARS + P::ZERO + tw + std::max(loop, sums)) * sizeof(float);
}

__device__ __forceinline__ void wf_copy_lane(float* dst, const void* src, bool ok) {  // 16 bytes, zeros where !ok
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(tc::smem_u32(dst)), "l"(src), "r"(ok ? 16 : 0)
               : "memory");
}
// bulk copy global -> shared (16-byte aligned, whole 16 bytes), counted on an mbarrier
__device__ __forceinline__ void wf_copy(float* dst, const void* src, int bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   tc::smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(tc::smem_u32(bar))
               : "memory");
}

// One CTA per (column block of 128 columns, share of the base rows, image).  Row sums
// C_n = sum_y m cos(2 pi n y'/Fy), S_n = sum_y m sin of every column: warp w takes the base rows
// b0 + w, b0 + w + WARPS, ..; their four mask rows stream through the warp's own ring (rows and columns
// outside the mask as zeros), a lane folds its CPL columns and adds them into its 2NY+1 sums with
// one broadcast load per four coefficients.  The warps' sums are then added in order and summed
// over the columns with the column twiddles.
// VEC (rows 16-byte aligned): every lane copies its own neighbouring columns with cp.async and
// reads them back.  Otherwise lanes 0-3 issue a bulk copy of one row each, the ring holds whole
// 16-byte granules and the lanes read their columns (lane + 32 i) past each row's misalignment;
// every wait is bounded: a warp whose copies do not land in a second issues no more, waits for what
// it has in flight, sets *err and makes its sums NaN, so that the images show it too; while *err is
// set, warps issue nothing and end the same way.  (Measured, window stage: 256 masks of 1024^2
// 186 us with cp.async, 222 with bulk copies (the same masks off by four bytes); 44 of 2048^2, Ny = 16, 167
// and 257; 40 ragged 913 x 777 masks, which have no aligned rows, 37.)
// The masks of up to WIN_MAX_SIZES sizes that share the period and the kernel support are one
// launch: its CTAs are the tiles of win_tiles.hpp (per size: image, column block, share of the
// base rows).  An image has nparts partials; those its size does not use are left zero.
struct WinSet {
  WinTiles T;
  int Lx[WIN_MAX_SIZES], Ly[WIN_MAX_SIZES];
  const float* masks[WIN_MAX_SIZES];
  const float* coef[WIN_MAX_SIZES];   // win_fold_coefs
  const float2* twF[WIN_MAX_SIZES];   // column twiddles (fi_twiddles)
  int rows;                           // most base rows of a tile
};

template <int NY, bool VEC, bool ASK>
__global__ void __launch_bounds__(32 * wf_warps(NY), 2) win_fold_kernel(const __grid_constant__ WinSet G, int Fx, int Fy, int Nx,
                                                                 int Ny, float2* __restrict__ win_part, int nparts,
                                                                 int stall, int* err, const int* __restrict__ form) {
  using P = WinFold<NY>;
  constexpr int CPL = P::CPL, COLS = P::COLS, KS = P::KS;
  extern __shared__ __align__(16) float sm[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  early_next();
  if constexpr (ASK) {  // launched early after win_dft_tc_kernel
    early_wait(form);
    if (*form == 0) return;  // the tensor cores have done these masks
  }
  uint64_t* bar = reinterpret_cast<uint64_t*>(sm) + warp * P::ST;
  float* zero = sm + P::BARS;
  float2* sTw = reinterpret_cast<float2*>(zero + P::ZERO);    // [Nx+1][TS]
  float* sK = zero + P::ZERO + 2 * (Nx + 1) * P::TS;          // ring, row offsets, coefficients; then the warps' sums
  int4* sOff = reinterpret_cast<int4*>(sK + P::RING);         // [rows + P::AHEAD]
  const int srows = min(G.rows, wf_stage(NY));
  float* sCoef = sK + P::RING + 4 * (srows + P::AHEAD);       // [rows][KS]
  float* ring = sK + warp * (P::ST * 4 * P::RB);
  int sz, img, cb, rs, b0, b1;
  win_tile(G.T, blockIdx.x, 1, sz, img, cb, rs, b0, b1);
  const int Lx = G.Lx[sz], Ly = G.Ly[sz];
  const float* coef = G.coef[sz];
  const float2* twF = G.twF[sz];
  const int X0 = cb * COLS, ncol = min(COLS, Lx - X0);
  const float* M = G.masks[sz] + (size_t)img * Lx * Ly + X0;
  const int base4 = (int)((reinterpret_cast<uintptr_t>(M) >> 2) & 3);  // misalignment of row 0 (floats)

  auto issue_vec = [&](int4 o4, int st) {  // the rows at offsets o4 (-1: none) into ring stage st
    const int off[4] = {o4.x, o4.y, o4.z, o4.w};
    float* dst = ring + st * (4 * P::RB) + CPL * lane;
    const bool in = CPL * lane < ncol;
    const float* base = M + (in ? CPL * lane : 0);
#pragma unroll
    for (int k = 0; k < 4; ++k)
      wf_copy_lane(dst + k * P::RB, base + (off[k] >= 0 ? off[k] : 0), off[k] >= 0 && in);
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  bool ok = VEC || __all_sync(0xffffffffu, *reinterpret_cast<volatile int*>(err) == 0);  // after a timeout, end quickly
  int flight = 0, unit = 0;  // stages issued and not waited for; stages issued
  auto issue = [&](int off, int st) {  // lanes 0-3: the row at offset off (-1: none) into ring stage st
    if (!ok || (stall >= 0 && unit >= stall)) return;  // (stall: the error-path test hook)
    ++flight;
    ++unit;
    if (lane >= 4) return;
    int bytes = off >= 0 ? 4 * ncol : 0;
    const float* row = M + off;
    if (bytes) {  // the granules the row touches
      const uintptr_t g = reinterpret_cast<uintptr_t>(row) & ~uintptr_t(15);
      bytes = (int)(((reinterpret_cast<uintptr_t>(row + ncol) + 15) & ~uintptr_t(15)) - g);
      row = reinterpret_cast<const float*>(g);
    }
    tc::mbar_arrive_expect_tx(&bar[st], bytes);
    if (bytes) wf_copy(ring + (st * 4 + lane) * P::RB, row, bytes, &bar[st]);
  };
  auto offset_of = [&](int b) {  // this lane's row of base row b
    int off = -1;
    if (lane < 4 && b < b1) {
      const FoldRange fr = fold_range(lane, Ly, Fy);
      if ((unsigned)(b - fr.lo) < (unsigned)fr.n) off = fold_y(b, lane, Ly, Fy) * Lx;
    }
    return off;
  };

  float c[NY + 1][CPL], s[NY][CPL];  // cos sums n = 0..NY, sin sums n = 1..NY
#pragma unroll
  for (int i = 0; i < CPL; ++i) {
#pragma unroll
    for (int n = 0; n <= NY; ++n) c[n][i] = 0.f;
#pragma unroll
    for (int n = 0; n < NY; ++n) s[n][i] = 0.f;
  }
  int b = b0 + warp;
  if constexpr (VEC) {
#pragma unroll
    for (int k = 0; k < P::ST - 1; ++k) {
      const int bk = b + k * P::WARPS;
      issue_vec(bk < b1 ? fold_offsets(bk, Lx, Ly, Fy) : make_int4(-1, -1, -1, -1), k);
    }
  } else {
    if (lane == 0) {
      for (int i = 0; i < P::ST; ++i) tc::mbar_init(&bar[i], 4);  // one arrival per row
      tc::fence_mbar_init();
    }
    __syncwarp();
#pragma unroll
    for (int k = 0; k < P::ST - 1; ++k) issue(offset_of(b + k * P::WARPS), k);
    for (int e = tid; e < P::ZERO; e += P::THREADS) zero[e] = 0.f;
  }
  for (int e = tid; e < (Nx + 1) * COLS; e += P::THREADS) {
    const int u = e / COLS, x = e - u * COLS;
    sTw[u * P::TS + x] = x < ncol ? __ldg(twF + (size_t)u * Lx + X0 + x) : make_float2(0.f, 0.f);
  }
  int st = 0;
  uint32_t ph = 0;
  for (int t0 = b0; t0 < b1; t0 += wf_stage(NY)) {  // one stage up to 2,000 rows at NY = 8
    const int t1 = min(b1, t0 + wf_stage(NY));
    if (t0 > b0) __syncthreads();
    const float4* src = reinterpret_cast<const float4*>(coef + (size_t)t0 * KS);
    for (int e = tid; e < (t1 - t0) * (KS / 4); e += P::THREADS) reinterpret_cast<float4*>(sCoef)[e] = __ldg(src + e);
    for (int e = tid; e < t1 - t0 + P::AHEAD; e += P::THREADS)
      sOff[e] = t0 + e < b1 ? fold_offsets(t0 + e, Lx, Ly, Fy) : make_int4(-1, -1, -1, -1);
    __syncthreads();
    for (; b < t1; b += P::WARPS) {
      float p[4][CPL];
      const float* src = ring + st * (4 * P::RB);
      if constexpr (VEC) {
        asm volatile("cp.async.wait_group %0;" ::"n"(P::ST - 2) : "memory");
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const float4 v = *reinterpret_cast<const float4*>(src + k * P::RB + 4 * lane);
          p[k][0] = v.x;
          p[k][1] = v.y;
          p[k][2] = v.z;
          p[k][3] = v.w;
        }
        issue_vec(sOff[b - t0 + P::AHEAD], st == 0 ? P::ST - 1 : st - 1);  // the previous row's slot
      } else {
        const int4 o4 = sOff[b - t0];
        const int off[4] = {o4.x, o4.y, o4.z, o4.w};
        if (ok) ok = __all_sync(0xffffffffu, tc::mbar_wait(&bar[st], ph));
        if (!ok) continue;
        --flight;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const float* q = off[k] >= 0 ? src + k * P::RB + ((base4 + off[k]) & 3) : zero;
#pragma unroll
          for (int i = 0; i < CPL; ++i) p[k][i] = q[lane + 32 * i];  // (past ncol: left in the ring, dropped below)
        }
        __syncwarp();  // the slot refilled below (the previous row's) has been read by every lane
        issue(lane < 4 ? reinterpret_cast<const int*>(sOff + (b - t0 + P::AHEAD))[lane] : -1,
              st == 0 ? P::ST - 1 : st - 1);
      }
      if (++st == P::ST) {
        st = 0;
        ph ^= 1;
      }
      float ce[CPL], co[CPL], se[CPL], so[CPL];  // operands of the even and odd cos sums and sin sums
#pragma unroll
      for (int i = 0; i < CPL; ++i) {
        const float a = p[0][i] + p[1][i], e = p[2][i] + p[3][i], d = p[0][i] - p[1][i], f = p[2][i] - p[3][i];
        ce[i] = a + e;
        co[i] = a - e;
        se[i] = d - f;
        so[i] = d + f;
        c[0][i] += ce[i];
      }
      const float4* k4 = reinterpret_cast<const float4*>(sCoef + (size_t)(b - t0) * KS);
#pragma unroll
      for (int q = 0; q < KS / 4; ++q) {
        const float4 kv = k4[q];
        const float kk[4] = {kv.x, kv.y, kv.z, kv.w};
#pragma unroll
        for (int h = 0; h < 4; ++h) {
          const int e = 4 * q + h;  // cos 1..NY, sin 1..NY
#pragma unroll
          for (int i = 0; i < CPL; ++i) {
            if (e < NY) c[e < NY ? e + 1 : 0][i] = fmaf(kk[h], (e & 1) ? ce[i] : co[i], c[e < NY ? e + 1 : 0][i]);
            else s[e < NY ? 0 : e - NY][i] = fmaf(kk[h], ((e - NY) & 1) ? se[i] : so[i], s[e < NY ? 0 : e - NY][i]);
          }
        }
      }
    }
  }
  // the ring's memory is reused: what was issued past the last row (nothing copied) completes too
  if constexpr (VEC) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
  } else {
    for (; flight > 0; --flight) {
      if (!__all_sync(0xffffffffu, tc::mbar_wait(&bar[st], ph, ok ? 1000u : 200u))) ok = false;
      if (++st == P::ST) {
        st = 0;
        ph ^= 1;
      }
    }
    if (!ok) {
      if (lane == 0) atomicExch(err, 1);
#pragma unroll
      for (int i = 0; i < CPL; ++i) c[0][i] = __int_as_float(0x7fffffff);  // W[0][.], and every image that it is in
    }
  }
  __syncthreads();  // ring, offsets and coefficients are read: their memory takes the warps' sums
  float* red = sK;                 // [warps][NR][COLS]
  float* sC = sK + P::RED;         // [NR][RS]: cos 0..NY, sin 1..NY
  {
    float* r = red + (size_t)warp * P::NR * COLS;
    auto put = [&](int n, const float(&v)[CPL]) {
      if constexpr (VEC) {
        reinterpret_cast<float4*>(r + n * COLS)[lane] = make_float4(v[0], v[1], v[2], v[3]);
      } else {
#pragma unroll
        for (int i = 0; i < CPL; ++i) r[n * COLS + lane + 32 * i] = lane + 32 * i < ncol ? v[i] : 0.f;
      }
    };
#pragma unroll
    for (int n = 0; n <= NY; ++n) put(n, c[n]);
#pragma unroll
    for (int n = 1; n <= NY; ++n) put(NY + n, s[n - 1]);
  }
  __syncthreads();
  for (int e = tid; e < P::NR * (COLS / 4); e += P::THREADS) {  // the warps' sums in order
    const int j = e / (COLS / 4), x = 4 * (e - j * (COLS / 4));
    float4 t = *reinterpret_cast<const float4*>(red + j * COLS + x);
#pragma unroll
    for (int w = 1; w < P::WARPS; ++w) {
      const float4 a = *reinterpret_cast<const float4*>(red + (size_t)w * P::NR * COLS + j * COLS + x);
      t.x += a.x;
      t.y += a.y;
      t.z += a.z;
      t.w += a.w;
    }
    *reinterpret_cast<float4*>(sC + j * P::RS + x) = t;
  }
  __syncthreads();
  // Column sums, with C, S the cos and sin row sums of v:
  //   W[v][u] = sum_x (C - iS)(cos - i sin),  W[-v][u] = sum_x (C + iS)(cos - i sin).
  // A thread takes v, three u and every Q-th four columns (neighbouring threads neighbouring
  // columns), so that a loaded C and S serve three u.
  constexpr int UT = 3;
  const int KY = 2 * Ny + 1, NU = Nx + 1, UG = (NU + UT - 1) / UT, NP = (Ny + 1) * UG;
  int Q = 8;
  while (Q > 1 && NP * Q > P::THREADS) Q >>= 1;
  const float scale = 1.0f / ((float)Fx * (float)Fy);
  float2* parts = win_part + (size_t)(G.T.img0[sz] + img) * nparts * KY * NU;
  const int used = G.T.rows[sz] * G.T.ncs[sz];
  if (cb == 0 && rs == 0)
    for (int e = tid; e < (nparts - used) * KY * NU; e += P::THREADS) parts[(size_t)used * KY * NU + e] = make_float2(0.f, 0.f);
  float2* out = parts + (size_t)(cb * G.T.ncs[sz] + rs) * KY * NU;
  for (int base = 0; base < NP * Q; base += P::THREADS) {  // uniform bound: whole warps shuffle
    const int t = base + tid, q = t % Q, pr = min(t / Q, NP - 1), v = pr / UG, u0 = (pr - v * UG) * UT;
    const float* C = sC + v * P::RS;
    const float* S = sC + (NY + v) * P::RS;  // v = 0: any row, times zero
    float A[UT], B[UT], D[UT], E[UT];
#pragma unroll
    for (int i = 0; i < UT; ++i) A[i] = B[i] = D[i] = E[i] = 0.f;
    for (int x = 4 * q; x < COLS; x += 4 * Q) {
      const float4 c4 = *reinterpret_cast<const float4*>(C + x);
      float4 s4 = *reinterpret_cast<const float4*>(S + x);
      if (v == 0) s4 = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int i = 0; i < UT; ++i) {
        const float4* T = reinterpret_cast<const float4*>(sTw + min(u0 + i, Nx) * P::TS + x);
        const float4 ta = T[0], tb = T[1];
        A[i] = fmaf(c4.w, tb.z, fmaf(c4.z, tb.x, fmaf(c4.y, ta.z, fmaf(c4.x, ta.x, A[i]))));
        B[i] = fmaf(c4.w, tb.w, fmaf(c4.z, tb.y, fmaf(c4.y, ta.w, fmaf(c4.x, ta.y, B[i]))));
        D[i] = fmaf(s4.w, tb.z, fmaf(s4.z, tb.x, fmaf(s4.y, ta.z, fmaf(s4.x, ta.x, D[i]))));
        E[i] = fmaf(s4.w, tb.w, fmaf(s4.z, tb.y, fmaf(s4.y, ta.w, fmaf(s4.x, ta.y, E[i]))));
      }
    }
    for (int o = Q / 2; o > 0; o >>= 1) {
#pragma unroll
      for (int i = 0; i < UT; ++i) {
        A[i] += __shfl_xor_sync(0xffffffffu, A[i], o);
        B[i] += __shfl_xor_sync(0xffffffffu, B[i], o);
        D[i] += __shfl_xor_sync(0xffffffffu, D[i], o);
        E[i] += __shfl_xor_sync(0xffffffffu, E[i], o);
      }
    }
    if (q == 0 && t < NP * Q) {
#pragma unroll
      for (int i = 0; i < UT; ++i) {
        if (u0 + i > Nx) continue;
        out[(Ny + v) * NU + u0 + i] = make_float2((A[i] - E[i]) * scale, -(B[i] + D[i]) * scale);
        if (v > 0) out[(Ny - v) * NU + u0 + i] = make_float2((A[i] + E[i]) * scale, (D[i] - B[i]) * scale);
      }
    }
  }
}

// Row splits of a launch of `units` x splits CTAs of `warps` warps, `slots` of them resident at
// once: the fewest row steps over all waves, a CTA costing its start and end in row steps besides
// its own.  A part-filled last wave costs as much as a full one, so small batches take what fits
// one wave (window of 16 masks of 1024^2: 21 us with the 256 CTAs of two splits, 31 us with 640).
static int fold_splits(long long units, int nb, int warps, int most, long long slots, int ends) {
  int best = 1;
  long long least = -1;
  for (int r : {1, 2, 3, 4, 5, 6, 8, 12, 16, 24, 32}) {
    if (r > most) break;
    const long long cost = (units * r + slots - 1) / slots * ((nb + warps * r - 1) / (warps * r) + ends);
    if (least < 0 || cost < least) {
      least = cost;
      best = r;
    }
  }
  return best;
}

// Row splits of the window DFTs of `tiles` column blocks in all, ncb to an image.  Each split is
// one more partial per column block for the next stage to add up, so at most 32 partials an image
// (or two splits): one mask of 1024^2 takes 22 us in the two stages with 32, 44 us with 256.
int win_fold_splits(const ImgGeom& g, int ncb, long long tiles, int sm_count) {
  const int nb = fold_nbase(g.Ly, g.Fy);
  const int warps = wf_warps(wf_ny(g.Ny)), most = std::max(1, std::min(nb / warps, std::max(2, 32 / ncb)));  // a base row per warp at least
  return fold_splits(tiles, nb, warps, most, 2LL * sm_count, g.Ny > 8 ? 24 : 8);
}

// column blocks and row splits of a window DFT
void win_fold_plan(ImgPlan& p, int sm_count) {
  const int cols = 32 * WF_CPL;
  p.rowBlocks = (p.g.Lx + cols - 1) / cols;
  p.colSplits = win_fold_splits(p.g, p.rowBlocks, (long long)p.rowBlocks * p.batch, sm_count);
}

size_t win_fold_coef_floats(const ImgGeom& g) { return (size_t)fold_nbase(g.Ly, g.Fy) * wf_stride(wf_ny(g.Ny)); }

cudaError_t win_fold_coefs(cudaStream_t s, const ImgGeom& g, float* coef) {
  const int nb = fold_nbase(g.Ly, g.Fy), NY = wf_ny(g.Ny);
  wf_coef_kernel<<<dim3((nb + 127) / 128, wf_stride(NY)), 128, 0, s>>>(coef, nb, NY, g.Ny, g.Fy);
  return cudaGetLastError();
}

template <int NY>
static cudaError_t launch_win_fold_t(cudaStream_t s, const WinSet& G, const ImgGeom& g, bool vec, float2* win_part,
                                     int nparts, int stall, int* err, const int* __restrict__ form) {
  const size_t smem = win_fold_smem<NY>(g.Nx, G.rows);
  const bool ask = vec && form != nullptr;  // (its own kernel: the test alone cost one image of 256^2 0.6 us)
  auto k = ask ? win_fold_kernel<NY, true, true> : vec ? win_fold_kernel<NY, true, false> : win_fold_kernel<NY, false, false>;
  const cudaError_t e = allow_smem(k);
  if (e != cudaSuccess) return e;
  const int tiles = G.T.tile0[G.T.n];
  if (ask)
    return launch_early(true, k, dim3((unsigned)tiles), WinFold<NY>::THREADS, smem, s, G, g.Fx, g.Fy, g.Nx, g.Ny, win_part,
                        nparts, stall, err, form);
  k<<<tiles, WinFold<NY>::THREADS, smem, s>>>(G, g.Fx, g.Fy, g.Nx, g.Ny, win_part, nparts, stall, err, nullptr);
  return cudaGetLastError();
}

// n <= WIN_MAX_SIZES mask sizes of one period and support, nparts partials per image; err: the
// timeout flag; stall >= 0: the error-path test hook; form: nullptr, or a device word that says whether
// the launch has masks to do (run_win_dft_tc; not asked with the hook, which stalls both kernels)
cudaError_t launch_win_fold(cudaStream_t s, const WinPart* parts, int n, const float* const* coef,
                            const float2* const* twF, float2* win_part, int nparts, int stall, int* err,
                            const int* __restrict__ form) {
  const ImgGeom& g0 = parts[0].plan.g;
  WinSet G = {};
  G.T.n = n;
  bool vec = stall < 0;
  for (int i = 0; i < n; ++i) {
    const ImgPlan& p = parts[i].plan;
    const int nb = fold_nbase(p.g.Ly, p.g.Fy);
    G.T.Lx[i] = nb;  // the extent that the splits share out: base rows
    G.T.rows[i] = p.rowBlocks;
    G.T.ncs[i] = p.colSplits;
    G.T.img0[i] = parts[i].img0;
    G.T.tile0[i + 1] = G.T.tile0[i] + p.rowBlocks * p.colSplits * p.batch;
    G.Lx[i] = p.g.Lx;
    G.Ly[i] = p.g.Ly;
    G.masks[i] = parts[i].masks;
    G.coef[i] = coef[i];
    G.twF[i] = twF[i];
    G.rows = std::max(G.rows, (nb + p.colSplits - 1) / p.colSplits);
    vec = vec && (p.g.Lx & 3) == 0 && (reinterpret_cast<uintptr_t>(parts[i].masks) & 15) == 0;
  }
  switch (wf_ny(g0.Ny)) {
    case 2: return launch_win_fold_t<2>(s, G, g0, vec, win_part, nparts, stall, err, form);
    case 4: return launch_win_fold_t<4>(s, G, g0, vec, win_part, nparts, stall, err, form);
    case 8: return launch_win_fold_t<8>(s, G, g0, vec, win_part, nparts, stall, err, form);
    case 12: return launch_win_fold_t<12>(s, G, g0, vec, win_part, nparts, stall, err, form);
    default: return launch_win_fold_t<16>(s, G, g0, vec, win_part, nparts, stall, err, form);
  }
}

// ---------------------------------------------------------------------------
// interpolation output
// ---------------------------------------------------------------------------
constexpr int FF_WARPS = 4, FF_THREADS = 32 * FF_WARPS;
constexpr int ff_cpl(int NY) { return NY <= 8 ? 4 : 2; }
constexpr int ff_stride(int NY) { return 4 * NY; }
constexpr int ff_stage(int NY) { return 44 * 1024 / (ff_stride(NY) * 4 + 16) / FF_WARPS * FF_WARPS; }

// coef[b][.]: 2cos(r t) for r = 1..2NY, then -2sin(r t), t = 2 pi b/Fy; zero past 2Ny
__global__ void ff_coef_kernel(float* __restrict__ coef, int nb, int NY, int Ny, int Fy) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x, e = blockIdx.y, r = e % (2 * NY) + 1;
  if (b >= nb) return;
  float c = 0.f, s = 0.f;
  if (r <= 2 * Ny) cis_round((long long)r * b, Fy, &c, &s);
  coef[(size_t)b * ff_stride(NY) + e] = e < 2 * NY ? 2.f * c : -2.f * s;
}

// One CTA per (column block, share of the base rows, image): its four warps take turns at the base
// rows, each lane with its columns of Tm in registers for all of them (CPL columns: 132 registers
// at NY = 8, so three CTAs of four warps per SM), so that a base row costs one broadcast load per
// four coefficients and the stores.  A tile of Tm in shared memory instead (4 x 4 outputs per
// thread) was bound by its reads.
template <int NY, bool VEC>
__global__ void __launch_bounds__(FF_THREADS, 3) fi_fold_kernel(const float* __restrict__ tm, int Lx, int Ly, int Fy,
                                                                int Ny, const float* __restrict__ coef, int nb,
                                                                float* __restrict__ images) {
  constexpr int CPL = ff_cpl(NY), COLS = 32 * CPL, KS = ff_stride(NY);
  extern __shared__ __align__(16) float sK[];  // [rows][KS] coefficients, then [rows] row offsets
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  early_wait(tm);
  early_wait(coef);
  const int X0 = blockIdx.x * COLS, img = blockIdx.z;
  const int b0 = (int)((long long)nb * blockIdx.y / gridDim.y), b1 = (int)((long long)nb * (blockIdx.y + 1) / gridDim.y);
  const int xl = VEC ? X0 + CPL * lane : X0 + lane;
  const float* T = tm + (size_t)img * (4 * Ny + 1) * Lx + xl;
  float tc[2 * NY + 1][CPL], ts[2 * NY][CPL];  // the lane's columns of Tm: cos rows 0..2NY, sin rows 1..2NY
  auto row = [&](int r, bool ok, float(&v)[CPL]) {
    const float* p = T + (size_t)(ok ? r : 0) * Lx;
    if constexpr (VEC && CPL == 4) {
      float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
      if (ok && xl < Lx) q = __ldg(reinterpret_cast<const float4*>(p));
      v[0] = q.x;
      v[1] = q.y;
      v[2] = q.z;
      v[3] = q.w;
    } else if constexpr (VEC) {
      float2 q = make_float2(0.f, 0.f);
      if (ok && xl < Lx) q = __ldg(reinterpret_cast<const float2*>(p));
      v[0] = q.x;
      v[1] = q.y;
    } else {
#pragma unroll
      for (int i = 0; i < CPL; ++i) v[i] = ok && xl + 32 * i < Lx ? __ldg(p + 32 * i) : 0.f;
    }
  };
#pragma unroll
  for (int r = 0; r <= 2 * NY; ++r) row(r, r <= 2 * Ny, tc[r]);
#pragma unroll
  for (int r = 1; r <= 2 * NY; ++r) row(2 * Ny + r, r <= 2 * Ny, ts[r - 1]);
  const int srows = min((nb + (int)gridDim.y - 1) / (int)gridDim.y, ff_stage(NY));
  int4* sOff = reinterpret_cast<int4*>(sK + srows * KS);
  float* O = images + (size_t)img * Lx * Ly + xl;
  for (int t0 = b0; t0 < b1; t0 += ff_stage(NY)) {  // one stage up to 1,200 rows at NY = 8
    const int t1 = min(b1, t0 + ff_stage(NY));
    if (t0 > b0) __syncthreads();
    const float4* src = reinterpret_cast<const float4*>(coef + (size_t)t0 * KS);
    for (int e = tid; e < (t1 - t0) * (KS / 4); e += FF_THREADS) reinterpret_cast<float4*>(sK)[e] = __ldg(src + e);
    for (int e = tid; e < t1 - t0; e += FF_THREADS) sOff[e] = fold_offsets(t0 + e, Lx, Ly, Fy);
    __syncthreads();
    for (int b = t0 + warp; b < t1; b += FF_WARPS) {
      const float4* k4 = reinterpret_cast<const float4*>(sK + (size_t)(b - t0) * KS);
      float ae[CPL], ao[CPL], be[CPL], bo[CPL];  // even and odd cos sums and sin sums
#pragma unroll
      for (int i = 0; i < CPL; ++i) {
        ae[i] = tc[0][i];
        ao[i] = be[i] = bo[i] = 0.f;
      }
#pragma unroll
      for (int q = 0; q < KS / 4; ++q) {
        const float4 kv = k4[q];
        const float kk[4] = {kv.x, kv.y, kv.z, kv.w};
#pragma unroll
        for (int h = 0; h < 4; ++h) {
          const int e = 4 * q + h;  // cos 1..2NY, sin 1..2NY
#pragma unroll
          for (int i = 0; i < CPL; ++i) {
            if (e < 2 * NY) {
              if (e & 1) ae[i] = fmaf(kk[h], tc[e < 2 * NY ? e + 1 : 0][i], ae[i]);
              else ao[i] = fmaf(kk[h], tc[e < 2 * NY ? e + 1 : 0][i], ao[i]);
            } else {
              if (e & 1) be[i] = fmaf(kk[h], ts[e < 2 * NY ? 0 : e - 2 * NY][i], be[i]);
              else bo[i] = fmaf(kk[h], ts[e < 2 * NY ? 0 : e - 2 * NY][i], bo[i]);
            }
          }
        }
      }
      float o[4][CPL];
#pragma unroll
      for (int i = 0; i < CPL; ++i) {
        const float u = ae[i] + ao[i], w = ae[i] - ao[i], s = be[i] + bo[i], t = be[i] - bo[i];
        o[0][i] = u + s;
        o[1][i] = u - s;
        o[2][i] = w - t;
        o[3][i] = w + t;
      }
      const int4 o4 = sOff[b - t0];
      const int off[4] = {o4.x, o4.y, o4.z, o4.w};
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        float* dst = O + off[k];
        if constexpr (VEC && CPL == 4) {
          if (off[k] >= 0 && xl < Lx) __stcs(reinterpret_cast<float4*>(dst), make_float4(o[k][0], o[k][1], o[k][2], o[k][3]));
        } else if constexpr (VEC) {
          if (off[k] >= 0 && xl < Lx) __stcs(reinterpret_cast<float2*>(dst), make_float2(o[k][0], o[k][1]));
        } else {
#pragma unroll
          for (int i = 0; i < CPL; ++i)
            if (off[k] >= 0 && xl + 32 * i < Lx) __stcs(dst + 32 * i, o[k][i]);
        }
      }
    }
  }
}

size_t fi_fold_coef_floats(const ImgGeom& g) { return (size_t)fold_nbase(g.Ly, g.Fy) * ff_stride(wf_ny(g.Ny)); }

cudaError_t fi_fold_coefs(cudaStream_t s, const ImgGeom& g, float* coef) {
  const int nb = fold_nbase(g.Ly, g.Fy), NY = wf_ny(g.Ny);
  ff_coef_kernel<<<dim3((nb + 127) / 128, ff_stride(NY)), 128, 0, s>>>(coef, nb, NY, g.Ny, g.Fy);
  return cudaGetLastError();
}

template <int NY>
static cudaError_t launch_fi_fold_t(cudaStream_t s, const ImgPlan& p, const float* tm, const float* coef,
                                    float* images) {
  const ImgGeom& g = p.g;
  const int nb = fold_nbase(g.Ly, g.Fy), cols = 32 * ff_cpl(NY), ncb = (g.Lx + cols - 1) / cols;
  const int R = fold_splits((long long)ncb * p.batch, nb, FF_WARPS, std::max(1, std::min(32, nb / FF_WARPS)),
                            3LL * (p.sms > 0 ? p.sms : 148), 7);
  const size_t smem = (size_t)std::min((nb + R - 1) / R, ff_stage(NY)) * (ff_stride(NY) * sizeof(float) + sizeof(int4));
  const bool vec = (g.Lx & 3) == 0 && ((reinterpret_cast<uintptr_t>(tm) | reinterpret_cast<uintptr_t>(images)) & 15) == 0;
  auto k = vec ? fi_fold_kernel<NY, true> : fi_fold_kernel<NY, false>;
  const cudaError_t e = allow_smem(k);
  if (e != cudaSuccess) return e;
  return launch_early(p.early, k, dim3(ncb, R, p.batch), FF_THREADS, smem, s, tm, g.Lx, g.Ly, g.Fy, g.Ny, coef, nb, images);
}

cudaError_t launch_fi_fold(cudaStream_t s, const ImgPlan& p, const float* tm, const float* coef, float* images) {
  switch (wf_ny(p.g.Ny)) {
    case 2: return launch_fi_fold_t<2>(s, p, tm, coef, images);
    case 4: return launch_fi_fold_t<4>(s, p, tm, coef, images);
    case 8: return launch_fi_fold_t<8>(s, p, tm, coef, images);
    case 12: return launch_fi_fold_t<12>(s, p, tm, coef, images);
    default: return launch_fi_fold_t<16>(s, p, tm, coef, images);
  }
}

}  // namespace litho
