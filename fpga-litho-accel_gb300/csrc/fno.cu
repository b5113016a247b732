// Fourier-neural-operator surrogate of the SOCS imaging map: forward, backward
// and Adam kernels, and the litho_surrogate_* C ABI.
//
// The reference has no surrogate (it images every mask with calcSOCS,
// litho.cpp:795-880); the network is the published FNO-2d (Li et al., ICLR
// 2021) with one input channel (the mask), width 32, 16 retained modes per
// axis, four Fourier layers and a 32->128->1 projection.
//
// Data layout (all per batch of B masks, L x L, channels-last):
//   z_l      bf16 [B][L][L][32]   pre-activation of Fourier layer l (v_{l+1} = GELU(z_l))
//   Xf / Xg  f32x2 [B][L][16][32] x-DFT of one row at kx = 0..15 (activations / gradients)
//   Gy / Gg  f32x2 [B][L][16][32] inverse y-DFT of the mixed modes, per row and kx
//   Vs_l     f32x2 [B][32][16][32] retained modes of v_l (kept for dR)
// A Fourier layer is two launches:
//   column kernel  (one CTA per kx and mask): y-DFT of Xf at the 32 kept ky,
//                  mode mixing by R (FP32 master weights), inverse y-DFT -> Gy
//   row kernel     (persistent over rows): z = W v + b + Re sum_kx Gy e^{i kx x}
//                  as two BF16 tensor-core GEMMs (K = 32 each), GELU, and the
//                  x-DFT of the result for the next layer as a third GEMM.
// The 1/L^2 and the factor 2 of the half spectrum are folded into the mixing
// (s_kx = c_kx / L^2), so the inverse evaluation E(U)(p) = sum Re(U phi_p) is
// the same sum in both directions; its adjoint is the forward partial DFT.
// Backward reuses the same pieces in reverse: the gradient of a layer input is
// W^T g_z + E(s conj(R)^T DFT(g_z)) and dR = s DFT(g_z) conj(V).
//
// GEMMs run on the tensor cores with mma.sync m16n8k16 BF16 (FP32 accumulate);
// weights stay in FP32 master copies and are rounded to BF16 in shared memory
// by every CTA.  The spectral intermediates stay FP32.

#include <cuda_bf16.h>

#include <cmath>
#include <cstring>
#include <random>
#include <vector>

#include "litho_internal.cuh"

using bf16 = __nv_bfloat16;

namespace litho {
namespace fno {

constexpr int C = LITHO_FNO_WIDTH;    // 32 channels
constexpr int M = LITHO_FNO_MODES;    // 16 retained kx (and 2 x 16 retained ky)
constexpr int J = 2 * M;              // 32 ky slots: ky = j (j < 16), L - 32 + j (j >= 16)
constexpr int H = LITHO_FNO_HIDDEN;   // 128 projection channels
constexpr int NL = LITHO_FNO_LAYERS;  // 4 Fourier layers
constexpr int THREADS = 256;
constexpr int SP = 40;                // padded bf16 row stride of the 32-wide shared tiles

// flat FP32 parameter vector (the oracle's layout)
struct Off {
  static constexpr size_t Pw = 0, Pb = C;
  static constexpr size_t W = 2 * C;                   // [NL][C o][C c]
  static constexpr size_t Wb = W + (size_t)NL * C * C; // [NL][C]
  static constexpr size_t R = Wb + (size_t)NL * C;     // [NL][J][M][C c][C o][2]
  static constexpr size_t RL = (size_t)J * M * C * C * 2;
  static constexpr size_t Q1 = R + NL * RL;            // [H][C]
  static constexpr size_t q1b = Q1 + (size_t)H * C;
  static constexpr size_t Q2 = q1b + H;
  static constexpr size_t q2b = Q2 + H;
  static constexpr size_t N = q2b + 1;
};

// dense (non-spectral) gradient slots written per CTA by the row kernels
struct Dn {
  static constexpr int Pw = 0, Pb = C, W = 2 * C, Wb = W + NL * C * C, Q1 = Wb + NL * C, q1b = Q1 + H * C,
                       Q2 = q1b + H, q2b = Q2 + H, N = q2b + 1;
};

__host__ __device__ inline size_t dense_to_param(int i) {
  if (i < Dn::Wb) return (size_t)i;  // Pw, Pb, W share their offsets
  if (i < Dn::Q1) return Off::Wb + (i - Dn::Wb);
  return Off::Q1 + (size_t)(i - Dn::Q1);  // Q1, q1b, Q2, q2b are contiguous in both
}

// ---------------------------------------------------------------------------
// small device helpers
// ---------------------------------------------------------------------------
__device__ __forceinline__ void mma16816(float* d, const uint32_t* a, uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};\n"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ float2 unpack2(uint32_t u) {
  __nv_bfloat162 v = *reinterpret_cast<__nv_bfloat162*>(&u);
  return __bfloat1622float2(v);
}
__device__ __forceinline__ uint32_t lds32(const bf16* p) { return *reinterpret_cast<const uint32_t*>(p); }
__device__ __forceinline__ uint32_t ldg32(const bf16* p) { return __ldg(reinterpret_cast<const unsigned int*>(p)); }

__device__ __forceinline__ float2 cmulf(float2 a, float2 b) {
  return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

// GELU in its tanh form (Hendrycks & Gimpel 2016): 0.5 x (1 + tanh(k0 (x + k1 x^3)))
constexpr float GK0 = 0.79788456080286536f, GK1 = 0.044715f;
__device__ __forceinline__ float tanh_hw(float x) {
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// Two values at once with the packed FP32 instructions (each half rounds as a scalar does): the row
// kernels run out of issue slots before they run out of arithmetic, and a GELU is seven FP32
// instructions and one of the special-function unit.
struct F2 {
  uint64_t v;
};
__device__ __forceinline__ F2 f2(float a, float b) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ F2 f2(float a) { return f2(a, a); }
__device__ __forceinline__ float2 f2_get(F2 a) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a.v));
  return r;
}
__device__ __forceinline__ F2 operator*(F2 a, F2 b) {
  F2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 operator+(F2 a, F2 b) {
  F2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}
__device__ __forceinline__ F2 tanh2(F2 a) {
  const float2 x = f2_get(a);
  return f2(tanh_hw(x.x), tanh_hw(x.y));
}
__device__ __forceinline__ F2 gelu2(F2 x) {
  const F2 t = tanh2(f2(GK0) * fma2(f2(GK1) * x, x * x, x));
  return (f2(0.5f) * x) * (f2(1.0f) + t);
}
__device__ __forceinline__ F2 gelu_grad2(F2 x) {
  const F2 x2 = x * x;
  const F2 t = tanh2(f2(GK0) * fma2(f2(GK1) * x, x2, x));
  const F2 h = f2(0.5f) * x, u = fma2(f2(-1.0f) * t, t, f2(1.0f));
  return fma2(h * u * f2(GK0), fma2(f2(3.0f * GK1), x2, f2(1.0f)), f2(0.5f) * (f2(1.0f) + t));
}
__device__ __forceinline__ uint32_t pack2(F2 a) {
  const float2 x = f2_get(a);
  return pack2(x.x, x.y);
}
__device__ __forceinline__ F2 unpack_f2(uint32_t u) {
  const float2 x = unpack2(u);
  return f2(x.x, x.y);
}
// A fragment (16 x 16, row major) of a C-layout accumulator pair (n tiles 2ks, 2ks+1)
__device__ __forceinline__ void acc_to_a(const float* c0, const float* c1, uint32_t* a) {
  a[0] = pack2(c0[0], c0[1]);
  a[1] = pack2(c0[2], c0[3]);
  a[2] = pack2(c1[0], c1[1]);
  a[3] = pack2(c1[2], c1[3]);
}

// ---------------------------------------------------------------------------
// tables: Ttab[px][2kx+ri] = (cos, -sin)(2 pi kx px / L); TT = transpose
// ---------------------------------------------------------------------------
__global__ void tables_kernel(int L, bf16* Ttab, bf16* TT, float2* twL) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < L * M) {
    const int px = i / M, kx = i % M;
    float s, c;
    sincospif(2.0f * (float)((kx * px) % L) / (float)L, &s, &c);
    Ttab[(size_t)px * J + 2 * kx] = __float2bfloat16(c);
    Ttab[(size_t)px * J + 2 * kx + 1] = __float2bfloat16(-s);
    TT[(size_t)(2 * kx) * L + px] = __float2bfloat16(c);
    TT[(size_t)(2 * kx + 1) * L + px] = __float2bfloat16(-s);
  }
  if (i < L) {
    float s, c;
    sincospif(2.0f * (float)i / (float)L, &s, &c);
    twL[i] = make_float2(c, s);  // e^{+2 pi i k / L}
  }
}

// ---------------------------------------------------------------------------
// x-DFT of four real rows at kx = 0..15 by one warp: lane -> kx = lane & 15, pixels of one parity
// (lane >> 4), then both parities together; every lane ends with its kx.  The latency of a twiddle
// gather and a pixel per step bound the form with a row a warp; four rows share the twiddle and take
// their pixels in one 16-byte read.  sM: the warp's [L] x 4 rows, sTw: e^{+2 pi i k / L}.
// 16,384 rows of 256: lift_dft 57 -> 28 us, band_rows 52 -> 21.
// ---------------------------------------------------------------------------
constexpr int DR = 4;
__device__ __forceinline__ void rows_dft(int L, const float* __restrict__ src, int nrows, float4* sM,
                                         const float2* sTw, float (&re)[DR], float (&im)[DR]) {
  const int lane = threadIdx.x & 31, kx = lane & 15, half = lane >> 4;
  float* m = reinterpret_cast<float*>(sM);
#pragma unroll
  for (int r = 0; r < DR; ++r)
    for (int px = lane; px < L; px += 32) m[DR * px + r] = r < nrows ? __ldg(src + (size_t)r * L + px) : 0.f;
  __syncwarp();
#pragma unroll
  for (int r = 0; r < DR; ++r) re[r] = im[r] = 0.f;
  int ang = kx * half;
#pragma unroll 4
  for (int px = half; px < L; px += 2) {
    const float2 w = sTw[ang];
    const float4 v = sM[px];
    ang = (ang + 2 * kx) & (L - 1);
    re[0] = fmaf(v.x, w.x, re[0]);
    im[0] = fmaf(-v.x, w.y, im[0]);
    re[1] = fmaf(v.y, w.x, re[1]);
    im[1] = fmaf(-v.y, w.y, im[1]);
    re[2] = fmaf(v.z, w.x, re[2]);
    im[2] = fmaf(-v.z, w.y, im[2]);
    re[3] = fmaf(v.w, w.x, re[3]);
    im[3] = fmaf(-v.w, w.y, im[3]);
  }
#pragma unroll
  for (int r = 0; r < DR; ++r) {
    re[r] += __shfl_xor_sync(0xffffffffu, re[r], 16);
    im[r] += __shfl_xor_sync(0xffffffffu, im[r], 16);
  }
}
__host__ __device__ inline size_t rows_dft_smem(int L) {
  return (size_t)L * sizeof(float2) + (size_t)(THREADS / 32) * L * DR * sizeof(float);
}

// lift + x-DFT of layer 0: v0 = Pw m + Pb, so X0[kx][c] = Pw[c] DFT(m)[kx] + Pb[c] L d(kx).
__global__ void __launch_bounds__(THREADS) lift_dft_kernel(int L, int rows, const float* __restrict__ theta,
                                                           const float* __restrict__ masks,
                                                           const float2* __restrict__ twL, float2* __restrict__ Xf,
                                                           float2* __restrict__ Mrow) {
  extern __shared__ __align__(16) unsigned char smraw[];
  early_next();
  float2* sTw = reinterpret_cast<float2*>(smraw);
  for (int i = threadIdx.x; i < L; i += THREADS) sTw[i] = twL[i];
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int row0 = (blockIdx.x * (THREADS / 32) + warp) * DR, n = min(DR, rows - row0);
  if (n <= 0) return;
  float re[DR], im[DR];
  rows_dft(L, masks + (size_t)row0 * L, n, reinterpret_cast<float4*>(sTw + L) + (size_t)warp * L, sTw, re, im);
  const float pw = theta[Off::Pw + lane], pb = theta[Off::Pb + lane];
#pragma unroll
  for (int r = 0; r < DR; ++r) {
    if (r >= n) break;
    if (Mrow && lane < 16) Mrow[(size_t)(row0 + r) * 16 + lane] = make_float2(re[r], im[r]);  // mask row DFT, kx < 16
    float2* out = Xf + (size_t)(row0 + r) * M * C;
#pragma unroll
    for (int k = 0; k < M; ++k) {
      const float mr = __shfl_sync(0xffffffffu, re[r], k), mi = __shfl_sync(0xffffffffu, im[r], k);
      out[k * C + lane] = make_float2(pw * mr + (k == 0 ? pb * (float)L : 0.f), pw * mi);
    }
  }
}

// ---------------------------------------------------------------------------
// column kernel: per (kx, group of G masks)
//   FWD: V = DFT_y(Xf) at kept ky; U = s R V; Gy = sum_j U e^{+i ky y}
//   BWD: gU = DFT_y(Xg); gV = s conj(R)^T gU; Gg = sum_j gV e^{+i ky y}
// Both y-transforms are real GEMMs on interleaved (re, im) operands, run on the
// tensor cores in TF32 (mma.sync m16n8k8, FP32 accumulate):
//   DFT_y : [2J x 2L] . [2L x C],  rows 2j+ro, K index 2y+ri
//   inverse: [2L x 2J] . [2J x C], rows 2y+ro, K index 2j+ri
// The mode weights R[.][kx] are read once per CTA for all G masks (FP32 mixing).
//
// What it must move is Xin once and Gout once (67 MB each at 64 masks of 256 x 256); the products
// themselves are short, so the operands' way to the registers decides.  The twiddles depend on
// neither kx nor the mask: column_tables_kernel lays them out once as the fragments a lane holds, one
// 16-byte load each (gathered from a cosine table they took four loads, four selects and four
// conversions).  The columns and the table stream through a ring, four steps ahead of their use (a CTA
// meets the table once, so that its loads are L2's).  A mask has 8 / G warps of its own, its mixed modes
// stay in their registers for all rows of the inverse.
// 64 masks: 142 -> 48 us a launch; 32 masks: forward 84 -> 31, backward 75 -> 35 (columns straight from global
// memory into fragments, a step ahead: 51, 31 and 36).  What is left is mostly the operands' shared-memory reads.
// ---------------------------------------------------------------------------
constexpr int COL_G = 4;
constexpr int COL_ST = 5;          // ring stages, eight rows of the columns each: four of them in flight
constexpr int CXP = 2 * C + 16;    // padded row of the ring (floats): the two rows of a fragment load miss each other's banks
constexpr int CP = C + 8;  // padded row of the modes in shared memory: fragment loads of two rows miss each other's banks

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}
__device__ __forceinline__ uint32_t tf32r(float x) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ void mma1688(float* d, const uint4& a, uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};\n"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b0), "r"(b1));
}

// A fragments of the two transforms, [row tile][k step][lane]: DFT_y 4 x L/4, inverse L/8 x 8
__global__ void column_tables_kernel(int L, const float2* __restrict__ twL, uint4* __restrict__ fd,
                                     uint4* __restrict__ fi) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= L * 32) return;
  const int lane = i & 31, g = lane >> 2, t = lane & 3, ro = g & 1, ri = t & 1;
  auto tw = [&](int ky, int y) { return twL[(ky * y) & (L - 1)]; };
  {
    const int mt = i / (8 * L), ks = i / 32 % (L / 4);
    const int j = 8 * mt + (g >> 1);  // rows g and g + 8 -> j and j + 4
    const int ky0 = j < M ? j : L - J + j, ky1 = (j + 4) < M ? j + 4 : L - J + j + 4;
    const int y0 = 4 * ks + (t >> 1), y1 = y0 + 2;
    // ro = 0: (cos, sin); ro = 1: (-sin, cos) over ri = 0, 1
    auto el = [&](float2 w) { return tf32r(ro == 0 ? (ri == 0 ? w.x : w.y) : (ri == 0 ? -w.y : w.x)); };
    fd[i] = make_uint4(el(tw(ky0, y0)), el(tw(ky1, y0)), el(tw(ky0, y1)), el(tw(ky1, y1)));
  }
  {
    const int mt = i / 256, ks = i / 32 % 8;
    const int y = 8 * mt + (g >> 1);  // rows g, g + 8 -> y, y + 4
    const int j0 = 4 * ks + (t >> 1), j1 = j0 + 2;
    const int ky0 = j0 < M ? j0 : L - J + j0, ky1 = j1 < M ? j1 : L - J + j1;
    // ro = 0: (cos, -sin); ro = 1: (sin, cos) over ri = 0, 1
    auto el = [&](float2 w) { return tf32r(ro == 0 ? (ri == 0 ? w.x : -w.y) : (ri == 0 ? w.y : w.x)); };
    fi[i] = make_uint4(el(tw(ky0, y)), el(tw(ky0, y + 4)), el(tw(ky1, y)), el(tw(ky1, y + 4)));
  }
}

template <bool BWD, int G>
__global__ void __launch_bounds__(THREADS, 2) column_kernel(int L, int B, const float* __restrict__ theta, int layer,
                                                            const float2* __restrict__ Xin, float2* __restrict__ Gout,
                                                            float2* __restrict__ modes_out,
                                                            const uint4* __restrict__ fd,
                                                            const uint4* __restrict__ fi) {
  extern __shared__ __align__(16) unsigned char smraw[];
  float2* sV = reinterpret_cast<float2*>(smraw);  // [G][J][CP]
  float2* sR = sV + G * J * CP;                   // the ring; then, BWD mixing, per-warp transposed R blocks
  constexpr int WPM = THREADS / 32 / G;           // warps of a mask
  constexpr int MT = G == 4 ? 2 : 1, NT = G == 1 ? 2 : 4;  // a warp's DFT_y tiles: MT x NT of 4 x 4
  const int kx = blockIdx.x, b0 = blockIdx.y * G, tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3, ri = t & 1;
  const int ng = min(G, B - b0);
  early_next();
  early_wait(Xin);
  const int gi = warp / WPM, sub = warp % WPM;
  {
    const int mt0 = G == 1 ? sub >> 1 : sub * MT, n0 = G == 1 ? 2 * (sub & 1) : 0;
    // steps of eight rows (two K steps) of every mask's column and the table's fragments for them, through
    // one ring of the CTA
    constexpr int XS = 8 * CXP;                       // floats of a mask's step
    constexpr int STEP = G * XS + 2 * 4 * 128;        // and the table's: [K step][row tile][lane] x 16 bytes
    float* ring = reinterpret_cast<float*>(sV + G * J * CP);
    const float2* x = Xin + ((size_t)b0 * L * M + kx) * C;
    const int N2 = L / 8;
    auto copy = [&](int k2) {
      if (k2 < N2) {
        float* st = ring + (k2 % COL_ST) * STEP;
        for (int i = tid; i < 128 * ng; i += THREADS) {  // 16-byte pieces: mask i / 128, its row i / 16 % 8
          const int m = i >> 7, r = (i >> 4) & 7, q = i & 15;
          cp_async16(smem_u32(st + m * XS + r * CXP + 4 * q), x + ((size_t)m * L + 8 * k2 + r) * M * C + 2 * q);
        }
        const int k = tid >> 7, m = (tid >> 5) & 3;
        cp_async16(smem_u32(st + G * XS + 4 * tid), fd + ((size_t)m * (L / 4) + 2 * k2 + k) * 32 + lane);
      }
      cp_async_commit();
    };
#pragma unroll
    for (int k2 = 0; k2 < COL_ST - 1; ++k2) copy(k2);
    float d[MT][NT][4] = {};
    for (int k2 = 0; k2 < N2; ++k2) {
      cp_async_wait<COL_ST - 2>();
      __syncthreads();  // the step is there; the one before is read
      copy(k2 + COL_ST - 1);
      const float* st = ring + (k2 % COL_ST) * STEP;
      // X[y][c].ri at y = 4 ks + t / 2 (+ 2), c = 8 n + g
      const float* b = st + gi * XS + (t >> 1) * CXP + 2 * (8 * n0 + g) + ri;
      const uint4* af = reinterpret_cast<const uint4*>(st + G * XS) + 32 * mt0 + lane;
      if (gi < ng) {
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          uint4 A[MT];
#pragma unroll
          for (int m = 0; m < MT; ++m) A[m] = af[128 * k + 32 * m];
#pragma unroll
          for (int n = 0; n < NT; ++n) {
            const uint32_t b0r = tf32r(b[4 * k * CXP + 16 * n]), b1r = tf32r(b[(4 * k + 2) * CXP + 16 * n]);
#pragma unroll
            for (int m = 0; m < MT; ++m) mma1688(d[m][n], A[m], b0r, b1r);
          }
        }
      }
    }
    // D rows m = 16 mt + g (+8) = 2j + ro, cols c
    if (gi < ng)
#pragma unroll
      for (int m = 0; m < MT; ++m) {
        const int j = 8 * (mt0 + m) + (g >> 1), ro = g & 1;
        float* v = reinterpret_cast<float*>(sV + ((size_t)gi * J + j) * CP) + ro;
#pragma unroll
        for (int n = 0; n < NT; ++n) {
          const int c = 8 * (n0 + n) + 2 * t;
          v[2 * c] = d[m][n][0];
          v[2 * c + 2] = d[m][n][1];
          v[4 * CP * 2 + 2 * c] = d[m][n][2];
          v[4 * CP * 2 + 2 * c + 2] = d[m][n][3];
        }
      }
  }
  __syncthreads();
  if (modes_out)
    for (int i = tid; i < ng * J * C; i += THREADS) {
      const int m = i / (J * C), j = (i / C) % J, c = i % C;
      modes_out[(((size_t)(b0 + m) * J + j) * M + kx) * C + c] = sV[((size_t)m * J + j) * CP + c];
    }
  // mixing: thread (lane = output channel, j = warp + 8 r) for every mask of the group
  const float s = (kx == 0 ? 1.0f : 2.0f) / ((float)L * (float)L);
  const float2* Rl = reinterpret_cast<const float2*>(theta + Off::R + (size_t)layer * Off::RL);
  float2 u[J / 8][G];
#pragma unroll
  for (int r = 0; r < J / 8; ++r)
#pragma unroll
    for (int gg = 0; gg < G; ++gg) u[r][gg] = make_float2(0.f, 0.f);
  float2* sRt = sR + (size_t)warp * C * (C + 1);  // BWD: this warp's block, transposed [o][c] (padded)
#pragma unroll
  for (int r = 0; r < J / 8; ++r) {
    const int j = warp + 8 * r;
    const float2* Rj = Rl + ((size_t)j * M + kx) * C * C;  // [c][o]
    if (BWD) {
      __syncwarp();
#pragma unroll 8
      for (int c = 0; c < C; ++c) sRt[lane * (C + 1) + c] = Rj[c * C + lane];
      __syncwarp();
    }
    // FWD: U[o] = s sum_c R[c][o] V[c]; BWD: gV[c] = s sum_o conj(R[c][o]) gU[o], lane = c
#pragma unroll 8
    for (int c = 0; c < C; c += 2) {
      const float2 ra = BWD ? sRt[c * (C + 1) + lane] : Rj[c * C + lane];
      const float2 rb = BWD ? sRt[(c + 1) * (C + 1) + lane] : Rj[(c + 1) * C + lane];
      const float iy = BWD ? -1.f : 1.f;
#pragma unroll
      for (int gg = 0; gg < G; ++gg) {
        const float4 v = *reinterpret_cast<const float4*>(sV + ((size_t)gg * J + j) * CP + c);
        u[r][gg].x = fmaf(ra.x, v.x, fmaf(-iy * ra.y, v.y, u[r][gg].x));
        u[r][gg].y = fmaf(ra.x, v.y, fmaf(iy * ra.y, v.x, u[r][gg].y));
        u[r][gg].x = fmaf(rb.x, v.z, fmaf(-iy * rb.y, v.w, u[r][gg].x));
        u[r][gg].y = fmaf(rb.x, v.w, fmaf(iy * rb.y, v.z, u[r][gg].y));
      }
    }
  }
  __syncthreads();  // every thread is done reading sV
#pragma unroll
  for (int r = 0; r < J / 8; ++r) {
    const int j = warp + 8 * r;
#pragma unroll
    for (int gg = 0; gg < G; ++gg)
      sV[((size_t)gg * J + j) * CP + lane] = make_float2(__uint_as_float(tf32r(s * u[r][gg].x)),
                                                         __uint_as_float(tf32r(s * u[r][gg].y)));
  }
  __syncthreads();
  if (gi >= ng) return;
  // inverse y as [2L x 2J] . [2J x C]: rows m = 2y + ro, K index 2j + ri; the mask's warps share
  // its L / 8 row tiles, all 4 n-tiles each.  K step ks covers j = 4 ks + t/2 (+2), ri = t & 1
  uint32_t bf[J / 4][4][2];
#pragma unroll
  for (int ks = 0; ks < J / 4; ++ks)
#pragma unroll
    for (int n = 0; n < 4; ++n)
#pragma unroll
      for (int h = 0; h < 2; ++h)
        bf[ks][n][h] = reinterpret_cast<const uint32_t*>(
            sV + ((size_t)gi * J + 4 * ks + (t >> 1) + 2 * h) * CP + 8 * n + g)[ri];
  const int ntile = (L / 8 - sub + WPM - 1) / WPM;
  uint4 A[2][4];  // half a tile's table fragments, and the next half's
  auto load_a = [&](uint4* q, int i, int h) {
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) q[ks] = __ldg(fi + (size_t)(sub + WPM * i) * 256 + 32 * (4 * h + ks) + lane);
  };
  load_a(A[0], 0, 0);
  for (int i = 0; i < ntile; ++i) {
    const int y = 8 * (sub + WPM * i) + (g >> 1), ro = g & 1;  // rows g, g + 8 -> y, y + 4
    float d[4][4] = {};
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      if (h == 0) load_a(A[1], i, 1);
      else if (i + 1 < ntile) load_a(A[0], i + 1, 0);
#pragma unroll
      for (int ks = 0; ks < 4; ++ks)
#pragma unroll
        for (int n = 0; n < 4; ++n) mma1688(d[n], A[h][ks], bf[4 * h + ks][n][0], bf[4 * h + ks][n][1]);
    }
    // lanes g (re) and g ^ 1 (im) hold channels c, c + 1 of one row: each takes one of the two whole
    float2* go = Gout + (((size_t)(b0 + gi) * L + y) * M + kx) * C + 2 * t + ro;
#pragma unroll
    for (int n = 0; n < 4; ++n) {
      const float p = __shfl_xor_sync(0xffffffffu, ro ? d[n][0] : d[n][1], 4);
      const float q = __shfl_xor_sync(0xffffffffu, ro ? d[n][2] : d[n][3], 4);
      go[8 * n] = ro ? make_float2(p, d[n][1]) : make_float2(d[n][0], p);
      go[(size_t)4 * M * C + 8 * n] = ro ? make_float2(q, d[n][3]) : make_float2(d[n][2], q);
    }
  }
}

size_t column_smem(int G, bool bwd) {
  const size_t rings = (size_t)COL_ST * (G * 8 * CXP + 1024) / 2, r = bwd ? (size_t)(THREADS / 32) * C * (C + 1) : 0;
  return ((size_t)G * J * CP + std::max(rings, r)) * sizeof(float2);
}

// ---------------------------------------------------------------------------
// shared-memory tiles of the row kernels: [px][32 channels] bf16, rows of 64 bytes whose four 16-byte
// chunks are permuted by (px / 2) & 3, so that the eight rows of a matrix load touch every bank once.
// A tile is both a row-major operand (ldmatrix) and a column-major one (ldmatrix.trans), and
// a row of it is 16 KB of global memory in one piece.
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t tile_off(int px, int chunk) {
  return (uint32_t)(px * 64 + ((chunk ^ ((px >> 1) & 3)) << 4));
}
__device__ __forceinline__ void ldsm4(uint32_t* r, uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}
__device__ __forceinline__ void ldsm4t(uint32_t* r, uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}
__device__ __forceinline__ void stsm4(uint32_t addr, uint32_t r0, uint32_t r1, uint32_t r2, uint32_t r3) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.shared.b16 [%0], {%1,%2,%3,%4};\n" ::"r"(addr), "r"(r0), "r"(r1),
               "r"(r2), "r"(r3)
               : "memory");
}
// A fragment of pixels 16 mt .. + 15, channels 16 ks .. + 15; also the place of a C-layout pair of n tiles
// 2 ks, 2 ks + 1 (stsm4) with the lane's row and chunk
__device__ __forceinline__ uint32_t tile_frag(int mt, int ks, int lane) {
  return tile_off(16 * mt + (lane & 15), 2 * ks + (lane >> 4));
}
// the 16 x 32 accumulator of pixels 16 mt .. + 15, rounded to bf16, into the tile
__device__ __forceinline__ void tile_put(uint32_t tile, int mt, int lane, const float (*v)[4]) {
#pragma unroll
  for (int ks = 0; ks < 2; ++ks)
    stsm4(tile + tile_frag(mt, ks, lane), pack2(v[2 * ks][0], v[2 * ks][1]), pack2(v[2 * ks][2], v[2 * ks][3]),
          pack2(v[2 * ks + 1][0], v[2 * ks + 1][1]), pack2(v[2 * ks + 1][2], v[2 * ks + 1][3]));
}
// pixels 16 mt .. + 15 of the tile to their kilobyte of global memory (the warp that wrote them)
__device__ __forceinline__ void tile_store(const unsigned char* tile, int mt, int lane, bf16* row) {
  __syncwarp();
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const int i = 32 * q + lane, px = 16 * mt + (i >> 2);
    *reinterpret_cast<uint4*>(row + (size_t)(16 * mt) * C + 8 * i) =
        *reinterpret_cast<const uint4*>(tile + tile_off(px, i & 3));
  }
}
// a row of [L][32] bf16 on its way into a tile
__device__ __forceinline__ void tile_load(uint32_t tile, const bf16* row, int L, int tid) {
  for (int i = tid; i < 4 * L; i += THREADS) cp_async16(tile + tile_off(i >> 2, i & 3), row + 8 * i);
}
// B fragments of a [n rows][32 k] bf16 table with rows of SP: b[ks][0..1] of the eight rows from n0
__device__ __forceinline__ void ldsm_b(uint32_t (*b)[2], uint32_t tab, int n0, int lane) {
  uint32_t r[4];
  ldsm4(r, tab + (uint32_t)((n0 + (lane & 7)) * SP + 8 * (lane >> 3)) * 2);
  b[0][0] = r[0];
  b[0][1] = r[1];
  b[1][0] = r[2];
  b[1][1] = r[3];
}
// the warp's 16 x 8 tile of X[kxri][c] = sum_px TT[kxri][px] v[px][c] (rows 16 (warp / 4), columns
// 8 (warp % 4)), to one row of Xf / Xg; T pixel tiles of 16
__device__ __forceinline__ void row_dft(uint32_t sTT, int LP, uint32_t tile, int T, int warp, int lane, float2* xrow) {
  const int mt2 = warp >> 2, nt = warp & 3, g = lane >> 2, t = lane & 3;
  float d[4] = {0.f, 0.f, 0.f, 0.f};
  const uint32_t ta = sTT + (uint32_t)((16 * mt2 + (lane & 15)) * LP + 8 * (lane >> 4)) * 2;
#pragma unroll 2
  for (int ks = 0; ks < T; ks += 2) {
    uint32_t b[4], a0[4], a1[4];
    ldsm4t(b, tile + tile_off(16 * ks + lane, nt));  // pixels 16 ks .. + 31
    ldsm4(a0, ta + 32 * ks);
    ldsm4(a1, ta + 32 * ks + 32);
    mma16816(d, a0, b[0], b[1]);
    mma16816(d, a1, b[2], b[3]);
  }
  // lanes g (re) and g ^ 1 (im) of rows kxri = 2 kx + ri: each takes one of the two channels whole
  const int ri = g & 1;
  const float p = __shfl_xor_sync(0xffffffffu, ri ? d[0] : d[1], 4);
  const float q = __shfl_xor_sync(0xffffffffu, ri ? d[2] : d[3], 4);
  float2* x = xrow + (8 * mt2 + (g >> 1)) * C + 8 * nt + 2 * t + ri;
  x[0] = ri ? make_float2(p, d[1]) : make_float2(d[0], p);
  x[4 * C] = ri ? make_float2(q, d[3]) : make_float2(d[2], q);
}

// ---------------------------------------------------------------------------
// forward row kernel (persistent over rows; the next row's inputs are
// on their way while the current row is computed)
//   v   = lift(mask) (layer 0) or act_in ? GELU(zin) : zin
//   z_l = W_l v + Wb_l + E(Gy row)
//   zout (optional) = act_out ? GELU(z_l) : z_l
//   !FINAL: Xf = x-DFT(GELU(z_l))        (input of the next column kernel)
//    FINAL: out = Q2 . GELU(Q1 z_3 + q1b) + q2b
// The inverse / forward DFT tables live in shared memory, W_l in registers.
//
// !FINAL moves 40 KB a row (16 KB in, 16 KB out, 4 KB of each spectrum) and is to be bound by
// that.  Activations pass through tiles in shared memory: whole 16-byte pieces on the global side
// (fragment-sized 4-byte accesses used half of each sector) and matrix loads and stores on the other,
// where one tile serves the store and, transposed, the x-DFT (it took 16 two-byte stores a lane
// and tile, and 40 scalar fragment loads).  What is left is the shared memory's bandwidth (70% busy),
// half of it the x-DFT's operands.  64 masks of 256 x 256: 220 -> 139 us a launch.
// Two CTAs per SM: a third took the registers of the two pixel tiles (172 us).
// FINAL's 128 GELUs a pixel bound it (one MUFU result takes a quarter of an SM 8 cycles a warp: 115 us):
// a warp takes both its pixel tiles through the projection together, so that they share its operands.
// 333 -> 267 us.
// ---------------------------------------------------------------------------
struct RowFwd {
  int L, rows, layer, act_in, act_out;
  const float* theta;
  const float* masks;
  const bf16* zin;
  const float2* Gy;
  bf16* zout;
  float2* Xf;
  float* out;
  const bf16* Ttab;
  const bf16* TT;
};

constexpr int MAXT = 2;  // m-tiles (16 pixels) per warp and row: L <= 256

struct FwdSmem {
  size_t sG, sW, sTT, sZ, sV, sQ1, sQ, total;
  __host__ __device__ static constexpr size_t up16(size_t x) { return (x + 15) & ~(size_t)15; }
  __host__ __device__ FwdSmem(int L, bool fin) {
    const size_t LP = (size_t)L + 8;
    size_t o = 0;
    sZ = o; o += 2 * (size_t)L * C * 2;  // two rows of zin, by parity
    sG = o; o += 2 * up16(C * SP * 2);   // two rows, by parity
    sW = o; o += up16(C * SP * 2);
    sTT = sV = sQ1 = sQ = 0;
    if (!fin) {
      sV = o; o += (size_t)L * C * 2;
      sTT = o; o += up16(J * LP * 2);
    } else {
      sQ1 = o; o += up16(H * SP * 2);
      sQ = o; o += up16(2 * H * sizeof(float));
    }
    total = o;
  }
};

enum { FWD_FIRST = 0, FWD_MID = 1, FWD_LAST = 2 };
constexpr int FWD_CTAS = 2;  // per SM

template <int KIND>
__global__ void __launch_bounds__(THREADS, FWD_CTAS) row_fwd_kernel(const RowFwd a) {
  constexpr bool FIRST = KIND == FWD_FIRST, FINAL = KIND == FWD_LAST;
  extern __shared__ __align__(16) unsigned char smraw[];
  const int L = a.L, LP = L + 8, l = FIRST ? 0 : FINAL ? NL - 1 : a.layer, T = L / 16;
  const FwdSmem S(L, FINAL);
  bf16* sG0 = reinterpret_cast<bf16*>(smraw + S.sG);   // [2][C c][SP]
  bf16* sW = reinterpret_cast<bf16*>(smraw + S.sW);    // [C o][SP]
  bf16* sTT = reinterpret_cast<bf16*>(smraw + S.sTT);  // [J][LP]: forward table
  bf16* sQ1 = reinterpret_cast<bf16*>(smraw + S.sQ1);  // [H][SP]
  float* sQ = reinterpret_cast<float*>(smraw + S.sQ);  // q1b[H], Q2[H] / 2
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const float* th = a.theta;
  for (int i = tid; i < C * C; i += THREADS) sW[(i / C) * SP + i % C] = __float2bfloat16(th[Off::W + l * C * C + i]);
  if (!FINAL)
    for (int i = tid; i < J * L / 2; i += THREADS) {
      const int k = i / (L / 2), px = 2 * (i % (L / 2));
      *reinterpret_cast<uint32_t*>(sTT + k * LP + px) = *reinterpret_cast<const uint32_t*>(a.TT + (size_t)k * L + px);
    }
  if (FINAL) {
    for (int i = tid; i < H * C; i += THREADS) sQ1[(i / C) * SP + i % C] = __float2bfloat16(th[Off::Q1 + i]);
    for (int i = tid; i < H; i += THREADS) {
      sQ[i] = th[Off::q1b + i];
      sQ[H + i] = 0.5f * th[Off::Q2 + i];
    }
  }
  // A fragments of the inverse table at the warp's pixels, the same for every row
  uint32_t AT[MAXT][2][4];
#pragma unroll
  for (int i = 0; i < MAXT; ++i)
    if (warp + 8 * i < T)
#pragma unroll
      for (int ks = 0; ks < 2; ++ks) {
        const bf16* ta = a.Ttab + (size_t)(16 * (warp + 8 * i) + g) * J + 16 * ks + 2 * t;
        AT[i][ks][0] = ldg32(ta);
        AT[i][ks][1] = ldg32(ta + 8 * J);
        AT[i][ks][2] = ldg32(ta + 8);
        AT[i][ks][3] = ldg32(ta + 8 * J + 8);
      }
  float bias[4][2], pw[2][4], pb[2][4];
#pragma unroll
  for (int n = 0; n < 4; ++n) {
    bias[n][0] = th[Off::Wb + l * C + 8 * n + 2 * t];
    bias[n][1] = th[Off::Wb + l * C + 8 * n + 2 * t + 1];
  }
  if (FIRST)
#pragma unroll
    for (int ks = 0; ks < 2; ++ks) {
      const int c0 = 16 * ks + 2 * t;
      pw[ks][0] = th[Off::Pw + c0];     pb[ks][0] = th[Off::Pb + c0];
      pw[ks][1] = th[Off::Pw + c0 + 1]; pb[ks][1] = th[Off::Pb + c0 + 1];
      pw[ks][2] = th[Off::Pw + c0 + 8]; pb[ks][2] = th[Off::Pb + c0 + 8];
      pw[ks][3] = th[Off::Pw + c0 + 9]; pb[ks][3] = th[Off::Pb + c0 + 9];
    }
  const float q2b = th[Off::q2b];

  // the next row's inputs: zin into the tile of its parity, the rest into registers
  early_next();
  const bf16* __restrict__ zin = a.zin;
  const float2* __restrict__ Gy = a.Gy;
  float mr[MAXT][2];
  float2 gr[2];
  auto load_row = [&](int row, int st) {
    if (FIRST) {
#pragma unroll
      for (int i = 0; i < MAXT; ++i) {
        const int mt = warp + 8 * i;
        if (mt < T) {
          mr[i][0] = __ldg(a.masks + (size_t)row * L + 16 * mt + g);
          mr[i][1] = __ldg(a.masks + (size_t)row * L + 16 * mt + g + 8);
        }
      }
    } else {
      tile_load(smem_u32(smraw + S.sZ) + st * L * C * 2, zin + (size_t)row * L * C, L, tid);
    }
    const float2* gp = Gy + (size_t)row * M * C;
    gr[0] = __ldg(gp + tid);
    gr[1] = __ldg(gp + tid + THREADS);
  };
  early_wait(zin);  // (the prologue reads parameters and tables alone)
  early_wait(Gy);
  if (blockIdx.x < a.rows) load_row(blockIdx.x, 0);
  cp_async_commit();

  int st = 0;
  for (int row = blockIdx.x; row < a.rows; row += gridDim.x, st ^= 1) {
    bf16* sG = sG0 + st * (FwdSmem::up16(C * SP * 2) / 2);
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int i = tid + THREADS * q, kx = i / C, c = i % C;
      *reinterpret_cast<uint32_t*>(sG + c * SP + 2 * kx) = pack2(gr[q].x, gr[q].y);
    }
    float mc[MAXT][2];
    if (FIRST)
#pragma unroll
      for (int i = 0; i < MAXT; ++i) {
        mc[i][0] = mr[i][0];
        mc[i][1] = mr[i][1];
      }
    cp_async_wait<0>();
    __syncthreads();  // this row's inputs; also, the other tile and sV are no longer read
    if (row + (int)gridDim.x < a.rows) load_row(row + gridDim.x, st ^ 1);
    cp_async_commit();
    unsigned char* sZ = smraw + S.sZ + (size_t)st * L * C * 2;
    const uint32_t tz = smem_u32(sZ), tv = smem_u32(smraw + S.sV);
    // z_l of the warp's pixel tiles in C layout, both at a time: they share the weights' and the
    // spectrum's fragments and hide each other's latency
    if (warp < T) {
      const bool two = warp + 8 < T;
      float acc[MAXT][4][4];
      {
        uint32_t A[MAXT][2][4];
#pragma unroll
        for (int i = 0; i < MAXT; ++i) {
          if (i == 1 && !two) break;
          if (FIRST) {
            const float m0 = mc[i][0], m1 = mc[i][1];
#pragma unroll
            for (int ks = 0; ks < 2; ++ks) {
              A[i][ks][0] = pack2(fmaf(pw[ks][0], m0, pb[ks][0]), fmaf(pw[ks][1], m0, pb[ks][1]));
              A[i][ks][1] = pack2(fmaf(pw[ks][0], m1, pb[ks][0]), fmaf(pw[ks][1], m1, pb[ks][1]));
              A[i][ks][2] = pack2(fmaf(pw[ks][2], m0, pb[ks][2]), fmaf(pw[ks][3], m0, pb[ks][3]));
              A[i][ks][3] = pack2(fmaf(pw[ks][2], m1, pb[ks][2]), fmaf(pw[ks][3], m1, pb[ks][3]));
            }
          } else {
#pragma unroll
            for (int ks = 0; ks < 2; ++ks) ldsm4(A[i][ks], tz + tile_frag(warp + 8 * i, ks, lane));
          }
        }
        if (!FIRST && a.act_in)
#pragma unroll
          for (int i = 0; i < MAXT; ++i) {
            if (i == 1 && !two) break;
#pragma unroll
            for (int e = 0; e < 8; ++e) A[i][e >> 2][e & 3] = pack2(gelu2(unpack_f2(A[i][e >> 2][e & 3])));
          }
#pragma unroll
        for (int n = 0; n < 4; ++n) {
          uint32_t bw[2][2], bg[2][2];
          ldsm_b(bw, smem_u32(sW), 8 * n, lane);
          ldsm_b(bg, smem_u32(sG), 8 * n, lane);
#pragma unroll
          for (int i = 0; i < MAXT; ++i) {
            acc[i][n][0] = bias[n][0]; acc[i][n][1] = bias[n][1];
            acc[i][n][2] = bias[n][0]; acc[i][n][3] = bias[n][1];
          }
#pragma unroll
          for (int ks = 0; ks < 2; ++ks)
#pragma unroll
            for (int i = 0; i < MAXT; ++i) {
              if (i == 1 && !two) break;
              mma16816(acc[i][n], A[i][ks], bw[ks][0], bw[ks][1]);
              mma16816(acc[i][n], AT[i][ks], bg[ks][0], bg[ks][1]);
            }
        }
      }
      if (a.zout && (FINAL || !a.act_out)) {  // z_l takes the place of the warp's own input
#pragma unroll
        for (int i = 0; i < MAXT; ++i) {
          if (i == 1 && !two) break;
          tile_put(tz, warp + 8 * i, lane, acc[i]);
          tile_store(sZ, warp + 8 * i, lane, a.zout + (size_t)row * L * C);
        }
      }
      if constexpr (!FINAL) {
#pragma unroll
        for (int i = 0; i < MAXT; ++i) {
          if (i == 1 && !two) break;
#pragma unroll
          for (int n = 0; n < 4; ++n)
#pragma unroll
            for (int e = 0; e < 4; e += 2) {
              const float2 v = f2_get(gelu2(f2(acc[i][n][e], acc[i][n][e + 1])));
              acc[i][n][e] = v.x;
              acc[i][n][e + 1] = v.y;
            }
        }
#pragma unroll
        for (int i = 0; i < MAXT; ++i) {
          if (i == 1 && !two) break;
          tile_put(tv, warp + 8 * i, lane, acc[i]);
          if (a.zout && a.act_out) tile_store(smraw + S.sV, warp + 8 * i, lane, a.zout + (size_t)row * L * C);
        }
      } else {
        uint32_t Az[MAXT][2][4];
#pragma unroll
        for (int i = 0; i < MAXT; ++i) {
          acc_to_a(acc[i][0], acc[i][1], Az[i][0]);
          acc_to_a(acc[i][2], acc[i][3], Az[i][1]);
        }
        F2 p[MAXT][2];
#pragma unroll
        for (int i = 0; i < MAXT; ++i) p[i][0] = p[i][1] = f2(0.f);
#pragma unroll 2
        for (int nh = 0; nh < H / 8; ++nh) {
          uint32_t bq[2][2];
          ldsm_b(bq, smem_u32(sQ1), 8 * nh, lane);
          const float2 b = *reinterpret_cast<const float2*>(sQ + 8 * nh + 2 * t);
          const float2 qs = *reinterpret_cast<const float2*>(sQ + H + 8 * nh + 2 * t);
          const F2 q = f2(qs.x, qs.y);
#pragma unroll
          for (int i = 0; i < MAXT; ++i) {
            if (i == 1 && !two) break;
            float hc[4] = {b.x, b.y, b.x, b.y};
            mma16816(hc, Az[i][0], bq[0][0], bq[0][1]);
            mma16816(hc, Az[i][1], bq[1][0], bq[1][1]);
            // q gelu(x) = (q/2) x + (q/2) x tanh(x (k0 + k0 k1 x^2))
#pragma unroll
            for (int r = 0; r < 2; ++r) {
              const F2 x = f2(hc[2 * r], hc[2 * r + 1]), hx = q * x;
              const F2 th_ = tanh2(x * fma2(f2(GK0 * GK1), x * x, f2(GK0)));
              p[i][r] = fma2(hx, th_, p[i][r] + hx);
            }
          }
        }
#pragma unroll
        for (int i = 0; i < MAXT; ++i) {
          if (i == 1 && !two) break;
          const float2 s0 = f2_get(p[i][0]), s1 = f2_get(p[i][1]);
          float p0 = s0.x + s0.y, p1 = s1.x + s1.y;
          p0 += __shfl_xor_sync(0xffffffffu, p0, 1);
          p0 += __shfl_xor_sync(0xffffffffu, p0, 2);
          p1 += __shfl_xor_sync(0xffffffffu, p1, 1);
          p1 += __shfl_xor_sync(0xffffffffu, p1, 2);
          if (t == 0) {
            float* o = a.out + (size_t)row * L + 16 * (warp + 8 * i) + g;
            o[0] = p0 + q2b;
            o[8] = p1 + q2b;
          }
        }
      }
    }
    if constexpr (!FINAL) {
      __syncthreads();
      row_dft(smem_u32(sTT), LP, tv, T, warp, lane, a.Xf + (size_t)row * M * C);
    }
  }
}

size_t row_fwd_smem(int L, bool final_) { return FwdSmem(L, final_).total; }

// ---------------------------------------------------------------------------
// loss: per mask e = ||out - y||, n = ||y||; loss_b = e / n, coef_b = 1 / (B e n).  The squares are
// summed in FP64, which bounds it (a quarter of an SM takes one such instruction per ~66 cycles), so a
// mask is shared by as many CTAs as there are SMs for it, and a second kernel adds their sums in
// order.  32 masks of 256 x 256: 99 us on a CTA each -> 29 + 4.
// ---------------------------------------------------------------------------
constexpr int LOSS_SHARES = 16;
__global__ void __launch_bounds__(THREADS) loss_part_kernel(int L, const float* __restrict__ out,
                                                            const float* __restrict__ tgt, double2* __restrict__ part) {
  early_next();
  early_wait(out);
  const size_t b = blockIdx.x / LOSS_SHARES, n = (size_t)L * L;
  const int sh = blockIdx.x % LOSS_SHARES;
  const float* o = out + b * n;
  const float* y = tgt + b * n;
  double se = 0.0, sy = 0.0;
#pragma unroll 4
  for (size_t i = sh * THREADS + threadIdx.x; i < n; i += LOSS_SHARES * THREADS) {
    const double t = (double)__ldg(y + i), d = (double)__ldg(o + i) - t;
    se = fma(d, d, se);
    sy = fma(t, t, sy);
  }
  __shared__ double2 r[THREADS / 32];
  for (int k = 16; k > 0; k >>= 1) {
    se += __shfl_xor_sync(0xffffffffu, se, k);
    sy += __shfl_xor_sync(0xffffffffu, sy, k);
  }
  if ((threadIdx.x & 31) == 0) r[threadIdx.x >> 5] = make_double2(se, sy);
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < THREADS / 32; ++w) {
      se += r[w].x;
      sy += r[w].y;
    }
    part[blockIdx.x] = make_double2(se, sy);
  }
}
__global__ void loss_kernel(int B, const double2* __restrict__ part, float* __restrict__ loss_b, float* __restrict__ coef) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  early_wait(part);
  if (b >= B) return;
  double a = 0.0, c = 0.0;
#pragma unroll
  for (int s = 0; s < LOSS_SHARES; ++s) {
    const double2 v = part[(size_t)b * LOSS_SHARES + s];
    a += v.x;
    c += v.y;
  }
  const double e = sqrt(a), nn = sqrt(c);
  loss_b[b] = nn > 0.0 ? (float)(e / nn) : 0.f;
  coef[b] = (e > 0.0 && nn > 0.0) ? (float)(1.0 / ((double)B * e * nn)) : 0.f;
}

// ---------------------------------------------------------------------------
// backward row kernel (persistent over rows; per-CTA weight-gradient partials)
//   HEAD_PROJ (layer 3): g_z3 from the projection (dQ1, dq1b, dQ2, dq2b)
//   HEAD_SPEC (layer l < 3): g_z_l = (gvpw_{l+1} + E(Gg_{l+1} row)) * GELU'(z_l)
//   HEAD_LIFT: g_v0 = gvpw_0 + E(Gg_0 row) -> dPw, dPb (no tail)
//   tail (PROJ, SPEC): dW_l += g_z^T v_l, dWb_l += sum g_z, Xg = x-DFT(g_z),
//                      gvpw_l = g_z W_l (bf16)
// ---------------------------------------------------------------------------
enum { HEAD_PROJ = 0, HEAD_SPEC = 1, HEAD_LIFT = 2 };

struct RowBwd {
  int L, rows, layer;
  const float* theta;
  const float* masks;
  const bf16* zl;     // z_l (PROJ: z_3 = v4; SPEC: z_l for GELU')
  const bf16* zlm1;   // z_{l-1} (v_l = GELU(z_{l-1})), unused for l == 0
  const bf16* gvin;   // gvpw_{l+1} (SPEC) / gvpw_0 (LIFT)
  const float2* Gg;   // Gg_{l+1} (SPEC) / Gg_0 (LIFT)
  const float* out;   // PROJ
  const float* tgt;   // PROJ
  const float* coef;  // PROJ [B]
  bf16* gvout;        // gvpw_l
  float2* Xg;         // x-DFT of g_z_l
  float* gpart;       // [gridDim.x][Dn::N]
  const bf16* Ttab;
  const bf16* TT;
};

// the two warps of a pair
__device__ __forceinline__ void pair_bar(int pair) { asm volatile("bar.sync %0, 64;" ::"r"(pair + 1) : "memory"); }
// sums over the rows g of a warp's fragments (lanes xor 4, 8, 16)
__device__ __forceinline__ float red_g(float v) {
  v += __shfl_xor_sync(0xffffffffu, v, 4);
  v += __shfl_xor_sync(0xffffffffu, v, 8);
  v += __shfl_xor_sync(0xffffffffu, v, 16);
  return v;
}
// the warp's 16 x 8 tile of dW[o][c] += sum_px gz[px][o] v[px][c] (rows 16 mt2, columns 8 nt)
__device__ __forceinline__ void row_dw(uint32_t tgz, uint32_t tv, int T, int mt2, int nt, int lane, float* dW) {
  // the transposed operand's matrices: (o 0-7, px 0-7), (o 8-15, px 0-7), (o 0-7, px 8-15), (o 8-15, px 8-15)
  const int px = (lane & 7) + 8 * (lane >> 4), ch = 2 * mt2 + ((lane >> 3) & 1);
#pragma unroll 2
  for (int ks = 0; ks < T; ks += 2) {
    uint32_t b[4], a0[4], a1[4];
    ldsm4t(b, tv + tile_off(16 * ks + lane, nt));
    ldsm4t(a0, tgz + tile_off(16 * ks + px, ch));
    ldsm4t(a1, tgz + tile_off(16 * ks + 16 + px, ch));
    mma16816(dW, a0, b[0], b[1]);
    mma16816(dW, a1, b[2], b[3]);
  }
}
__device__ __forceinline__ void put_dw(float* w, int mt2, int nt, int lane, const float* dW) {
  const int o = 16 * mt2 + (lane >> 2), c = 8 * nt + 2 * (lane & 3);
  w[o * C + c] = dW[0];
  w[o * C + c + 1] = dW[1];
  w[(o + 8) * C + c] = dW[2];
  w[(o + 8) * C + c + 1] = dW[3];
}
// v_l = lift(mask) of pixels 16 mt + g, + 8 at fragment ks
__device__ __forceinline__ void lift_frag(const float* pw, const float* pb, float m0, float m1, uint32_t* A) {
  A[0] = pack2(fmaf(pw[0], m0, pb[0]), fmaf(pw[1], m0, pb[1]));
  A[1] = pack2(fmaf(pw[0], m1, pb[0]), fmaf(pw[1], m1, pb[1]));
  A[2] = pack2(fmaf(pw[2], m0, pb[2]), fmaf(pw[3], m0, pb[3]));
  A[3] = pack2(fmaf(pw[2], m1, pb[2]), fmaf(pw[3], m1, pb[3]));
}
__device__ __forceinline__ void lift_coef(const float* th, int ks, int t, float* pw, float* pb) {
  const int c0 = 16 * ks + 2 * t;
  pw[0] = th[Off::Pw + c0];     pb[0] = th[Off::Pb + c0];
  pw[1] = th[Off::Pw + c0 + 1]; pb[1] = th[Off::Pb + c0 + 1];
  pw[2] = th[Off::Pw + c0 + 8]; pb[2] = th[Off::Pb + c0 + 8];
  pw[3] = th[Off::Pw + c0 + 9]; pb[3] = th[Off::Pb + c0 + 9];
}

struct BwdSmem {
  size_t sGv, sV, sZ, sWT, sG, sTT, sRed, total;
  __host__ __device__ static constexpr size_t up16(size_t x) { return (x + 15) & ~(size_t)15; }
  __host__ __device__ BwdSmem(int L, int head) {
    const size_t LP = (size_t)L + 8, tile = (size_t)L * C * 2;
    size_t o = 0;
    sGv = o; o += 2 * tile;  // gvin, by parity; g_z takes its place
    sV = sZ = sTT = sWT = 0;
    if (head == HEAD_SPEC) {
      sV = o; o += 2 * tile;  // z_{l-1}, by parity; v_l takes its place
      sZ = o; o += tile;      // z_l; gvpw_l takes its place
      sTT = o; o += up16(J * LP * 2);
      sWT = o; o += up16(C * SP * 2);
    }
    sG = o; o += 2 * up16(C * SP * 2);
    sRed = o; o += up16((size_t)(THREADS / 32) * 2 * C * sizeof(float));
    total = o;
  }
};

// HEAD_SPEC and HEAD_LIFT.  SPEC moves 72 KB a row and is to be bound by that: rows arrive by
// asynchronous copies (z_l, needed for one half of the work, while the other half runs; the rest a row
// ahead) in the tiles of the forward kernel, results take their operands' places, and the two
// contractions over the row (dW, Xg) read them transposed.  It took scalar loads of half-used sectors
// with nothing in flight but the current tile's, and two-byte transposing stores.
// 32 masks of 256 x 256: 220 -> 143 us a layer; LIFT 78 -> 40.
template <int HEAD>
__global__ void __launch_bounds__(THREADS, 2) row_bwd_kernel(const RowBwd a) {
  constexpr bool SPEC = HEAD == HEAD_SPEC;
  extern __shared__ __align__(16) unsigned char smraw[];
  const int L = a.L, LP = L + 8, l = a.layer, T = L / 16;
  const BwdSmem S(L, HEAD);
  const size_t tile = (size_t)L * C * 2;
  bf16* sWT = reinterpret_cast<bf16*>(smraw + S.sWT);  // [C c][SP]: W_l[o][c] at [c][o]
  bf16* sG0 = reinterpret_cast<bf16*>(smraw + S.sG);   // [2][C c][SP]
  bf16* sTT = reinterpret_cast<bf16*>(smraw + S.sTT);  // [J][LP]: forward table
  float* sRed = reinterpret_cast<float*>(smraw + S.sRed);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const float* th = a.theta;
  if (SPEC) {
    for (int i = tid; i < J * L / 2; i += THREADS) {
      const int k = i / (L / 2), px = 2 * (i % (L / 2));
      *reinterpret_cast<uint32_t*>(sTT + k * LP + px) = *reinterpret_cast<const uint32_t*>(a.TT + (size_t)k * L + px);
    }
    for (int i = tid; i < C * C; i += THREADS) {
      const int o = i / C, c = i % C;
      sWT[c * SP + o] = __float2bfloat16(th[Off::W + l * C * C + i]);
    }
  }
  uint32_t AT[MAXT][2][4];  // A fragments of the inverse table at the warp's pixels
#pragma unroll
  for (int i = 0; i < MAXT; ++i)
    if (warp + 8 * i < T)
#pragma unroll
      for (int ks = 0; ks < 2; ++ks) {
        const bf16* ta = a.Ttab + (size_t)(16 * (warp + 8 * i) + g) * J + 16 * ks + 2 * t;
        AT[i][ks][0] = ldg32(ta);
        AT[i][ks][1] = ldg32(ta + 8 * J);
        AT[i][ks][2] = ldg32(ta + 8);
        AT[i][ks][3] = ldg32(ta + 8 * J + 8);
      }
  // per-thread partial sums over rows g, g + 8 (columns 8n + 2t, + 1)
  float vb[4][2] = {};                 // dWb (SPEC) or dPb (LIFT)
  float vw[4][2] = {};                 // dPw (LIFT)
  float dW[4] = {0.f, 0.f, 0.f, 0.f};  // the warp's 16 x 8 tile of dW_l

  early_next();
  const bf16 *__restrict__ gvin = a.gvin, *__restrict__ zl = a.zl, *__restrict__ zlm1 = a.zlm1;
  const float2* __restrict__ Gg = a.Gg;
  float mr[MAXT][2];
  float2 gr[2];
  const bool masks = !SPEC || l == 0;
  auto load_row = [&](int row, int st) {  // all but z_l
    tile_load(smem_u32(smraw + S.sGv) + st * (uint32_t)tile, gvin + (size_t)row * L * C, L, tid);
    if (SPEC && l > 0) tile_load(smem_u32(smraw + S.sV) + st * (uint32_t)tile, zlm1 + (size_t)row * L * C, L, tid);
    if (masks)
#pragma unroll
      for (int i = 0; i < MAXT; ++i)
        if (warp + 8 * i < T) {
          mr[i][0] = __ldg(a.masks + (size_t)row * L + 16 * (warp + 8 * i) + g);
          mr[i][1] = __ldg(a.masks + (size_t)row * L + 16 * (warp + 8 * i) + g + 8);
        }
    const float2* gp = Gg + (size_t)row * M * C;
    gr[0] = __ldg(gp + tid);
    gr[1] = __ldg(gp + tid + THREADS);
  };
  auto load_z = [&](int row) {
    if (SPEC) tile_load(smem_u32(smraw + S.sZ), zl + (size_t)row * L * C, L, tid);
  };
  early_wait(gvin);  // (the prologue reads parameters and tables alone)
  early_wait(zl);
  early_wait(zlm1);
  early_wait(Gg);
  if (blockIdx.x < a.rows) {
    load_row(blockIdx.x, 0);
    load_z(blockIdx.x);
  }
  cp_async_commit();

  int st = 0;
  for (int row = blockIdx.x; row < a.rows; row += gridDim.x, st ^= 1) {
    const int next = row + gridDim.x;
    bf16* sG = sG0 + st * (BwdSmem::up16(C * SP * 2) / 2);
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int i = tid + THREADS * q, kx = i / C, c = i % C;
      *reinterpret_cast<uint32_t*>(sG + c * SP + 2 * kx) = pack2(gr[q].x, gr[q].y);
    }
    float mc[MAXT][2];
#pragma unroll
    for (int i = 0; i < MAXT; ++i) {
      mc[i][0] = mr[i][0];
      mc[i][1] = mr[i][1];
    }
    cp_async_wait<0>();
    __syncthreads();  // this row's inputs; the other parity's tiles are no longer read
    if (next < a.rows) load_row(next, st ^ 1);
    cp_async_commit();
    const uint32_t tgv = smem_u32(smraw + S.sGv) + st * (uint32_t)tile, tv = smem_u32(smraw + S.sV) + st * (uint32_t)tile,
                   tz = smem_u32(smraw + S.sZ);
#pragma unroll
    for (int i = 0; i < MAXT; ++i) {
      const int mt = warp + 8 * i;
      if (mt >= T) break;
      // g_v = gvin + E(G row)
      float gz[4][4];
#pragma unroll
      for (int ks = 0; ks < 2; ++ks) {
        uint32_t r[4];
        ldsm4(r, tgv + tile_frag(mt, ks, lane));
        const float2 f0 = unpack2(r[0]), f1 = unpack2(r[1]), f2_ = unpack2(r[2]), f3 = unpack2(r[3]);
        gz[2 * ks][0] = f0.x; gz[2 * ks][1] = f0.y; gz[2 * ks][2] = f1.x; gz[2 * ks][3] = f1.y;
        gz[2 * ks + 1][0] = f2_.x; gz[2 * ks + 1][1] = f2_.y; gz[2 * ks + 1][2] = f3.x; gz[2 * ks + 1][3] = f3.y;
      }
#pragma unroll
      for (int n = 0; n < 4; ++n) {
        uint32_t bg[2][2];
        ldsm_b(bg, smem_u32(sG), 8 * n, lane);
        mma16816(gz[n], AT[i][0], bg[0][0], bg[0][1]);
        mma16816(gz[n], AT[i][1], bg[1][0], bg[1][1]);
      }
      if (!SPEC) {
        const float m0 = mc[i][0], m1 = mc[i][1];
#pragma unroll
        for (int n = 0; n < 4; ++n) {
          vb[n][0] += gz[n][0] + gz[n][2];
          vb[n][1] += gz[n][1] + gz[n][3];
          vw[n][0] += gz[n][0] * m0 + gz[n][2] * m1;
          vw[n][1] += gz[n][1] * m0 + gz[n][3] * m1;
        }
        continue;
      }
      // g_z_l = g_v GELU'(z_l); v_l
#pragma unroll
      for (int ks = 0; ks < 2; ++ks) {
        uint32_t r[4];
        ldsm4(r, tz + tile_frag(mt, ks, lane));
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          float* z = &gz[2 * ks + (q >> 1)][2 * (q & 1)];
          const float2 v = f2_get(f2(z[0], z[1]) * gelu_grad2(unpack_f2(r[q])));
          z[0] = v.x;
          z[1] = v.y;
        }
        if (l == 0) {
          float pw[4], pb[4];
          lift_coef(th, ks, t, pw, pb);
          lift_frag(pw, pb, mc[i][0], mc[i][1], r);
        } else {
          ldsm4(r, tv + tile_frag(mt, ks, lane));
#pragma unroll
          for (int q = 0; q < 4; ++q) r[q] = pack2(gelu2(unpack_f2(r[q])));
        }
        stsm4(tv + tile_frag(mt, ks, lane), r[0], r[1], r[2], r[3]);
      }
#pragma unroll
      for (int n = 0; n < 4; ++n) {
        vb[n][0] += gz[n][0] + gz[n][2];
        vb[n][1] += gz[n][1] + gz[n][3];
      }
      tile_put(tgv, mt, lane, gz);
      // gvpw_l = g_z W_l: B[k = o][n = c] = W[o][c] = sWT[c][o]
      uint32_t AZ[2][4];
      acc_to_a(gz[0], gz[1], AZ[0]);
      acc_to_a(gz[2], gz[3], AZ[1]);
      float d[4][4] = {};
#pragma unroll
      for (int n = 0; n < 4; ++n) {
        uint32_t bw[2][2];
        ldsm_b(bw, smem_u32(sWT), 8 * n, lane);
        mma16816(d[n], AZ[0], bw[0][0], bw[0][1]);
        mma16816(d[n], AZ[1], bw[1][0], bw[1][1]);
      }
      tile_put(tz, mt, lane, d);
      tile_store(smraw + S.sZ, mt, lane, a.gvout + (size_t)row * L * C);
    }
    if (!SPEC) continue;
    __syncthreads();
    if (next < a.rows) load_z(next);
    cp_async_commit();
    row_dw(tgv, tv, T, warp >> 2, warp & 3, lane, dW);
    row_dft(smem_u32(sTT), LP, tgv, T, warp, lane, a.Xg + (size_t)row * M * C);
  }

  // ---- per-CTA partials; over the warps in a fixed order, so that the gradient repeats bit for bit ----
  float* gp = a.gpart + (size_t)blockIdx.x * Dn::N;
  cp_async_wait<0>();
  float* mine = sRed + warp * 2 * C;
#pragma unroll
  for (int n = 0; n < 4; ++n)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const float s0 = red_g(vb[n][e]), s1 = SPEC ? 0.f : red_g(vw[n][e]);
      if (g == 0) {
        mine[8 * n + 2 * t + e] = s0;
        mine[C + 8 * n + 2 * t + e] = s1;
      }
    }
  __syncthreads();
  for (int i = tid; i < (SPEC ? C : 2 * C); i += THREADS) {
    float s = 0.f;
    for (int w = 0; w < THREADS / 32; ++w) s += sRed[w * 2 * C + i];
    gp[SPEC ? Dn::Wb + l * C + i : i < C ? Dn::Pb + i : Dn::Pw + i - C] = s;
  }
  if (SPEC) put_dw(gp + Dn::W + l * C * C, warp >> 2, warp & 3, lane, dW);
}

// ---------------------------------------------------------------------------
// HEAD_PROJ: one CTA of sixteen warps per SM.  The hidden layer bounds it: 128 GELUs with their
// derivatives a pixel (about fifteen FP32 instructions each, taken two at a time).  Two warps share a
// pixel tile, one half of the hidden channels each, which halves the sums a thread keeps (dq1b, dQ2) and
// lets sixteen warps fit; they exchange halves of g_v4.  The hidden gradients stay in shared memory,
// row-major, and are read transposed for dQ1 after the row's one barrier, beside dW, Xg and gvpw.
// With eight warps, all hidden channels each and two-byte transposing stores: 740 us for 32 masks of
// 256 x 256; now 446.
// ---------------------------------------------------------------------------
constexpr int PROJ_THREADS = 512, PROJ_WARPS = PROJ_THREADS / 32;
constexpr int PROJ_RED = H + 2 * C;  // a warp's slots: dq1b, dQ2 of its half, dWb of its half, dq2b

struct ProjSmem {
  size_t sZ, sV, sGz, sGH, sX, sTT, sQ1, sWT, sq, total;
  __host__ __device__ static constexpr size_t up16(size_t x) { return (x + 15) & ~(size_t)15; }
  __host__ __device__ explicit ProjSmem(int L) {
    const size_t LP = (size_t)L + 8, tile = (size_t)L * C * 2;
    size_t o = 0;
    sZ = o; o += 2 * tile;            // z_3, by parity
    sV = o; o += 2 * tile;            // z_2, by parity; v_3 takes its place
    sGz = o; o += tile;               // g_z
    sX = o; o += PROJ_WARPS * 1024;   // a kilobyte a warp: halves of g_v4, then gvpw tiles
    sGH = o;                          // [L][H] hidden gradients; at the end, the warps' sums
    const size_t gh = (size_t)L * H * 2, red = PROJ_WARPS * PROJ_RED * sizeof(float);
    o += gh > red ? gh : red;
    sTT = o; o += up16(J * LP * 2);
    sQ1 = o; o += up16(H * SP * 2);
    sWT = o; o += up16(C * SP * 2);
    sq = o; o += 2 * H * sizeof(float);  // q1b, Q2
    total = o;
  }
};

__global__ void __launch_bounds__(PROJ_THREADS, 1) row_bwd_proj_kernel(const RowBwd a) {
  extern __shared__ __align__(16) unsigned char smraw[];
  const int L = a.L, LP = L + 8, l = NL - 1, T = L / 16;
  const ProjSmem S(L);
  const size_t tile = (size_t)L * C * 2;
  bf16* sTT = reinterpret_cast<bf16*>(smraw + S.sTT);
  bf16* sQ1 = reinterpret_cast<bf16*>(smraw + S.sQ1);  // [H][SP]
  bf16* sWT = reinterpret_cast<bf16*>(smraw + S.sWT);  // [C c][SP]: W[o][c] at [c][o]
  float* sq = reinterpret_cast<float*>(smraw + S.sq);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int hh = warp & 1, pair = warp >> 1;  // half of the hidden channels; tiles pair, pair + 8
  early_next();
  const float* th = a.theta;
  for (int i = tid; i < J * L / 2; i += PROJ_THREADS) {
    const int k = i / (L / 2), px = 2 * (i % (L / 2));
    *reinterpret_cast<uint32_t*>(sTT + k * LP + px) = *reinterpret_cast<const uint32_t*>(a.TT + (size_t)k * L + px);
  }
  for (int i = tid; i < C * C; i += PROJ_THREADS)
    sWT[(i % C) * SP + i / C] = __float2bfloat16(th[Off::W + l * C * C + i]);
  for (int i = tid; i < H * C; i += PROJ_THREADS) sQ1[(i / C) * SP + i % C] = __float2bfloat16(th[Off::Q1 + i]);
  for (int i = tid; i < H; i += PROJ_THREADS) {
    sq[i] = th[Off::q1b + i];
    sq[H + i] = th[Off::Q2 + i];
  }
  const uint32_t gh = smem_u32(smraw + S.sGH);
  auto gh_off = [](int px, int chunk) { return (uint32_t)(px * 2 * H + ((chunk ^ (px & 7)) << 4)); };

  F2 dq1b[8], dq2[8];  // over rows g, g + 8; channels 64 hh + 8 nh + 2 t, + 1
#pragma unroll
  for (int i = 0; i < 8; ++i) dq1b[i] = dq2[i] = f2(0.f);
  float vb[2][2] = {};                 // dWb, channels 16 hh + 8 n + 2 t, + 1
  float dq2b = 0.f;
  float dW[4] = {0.f, 0.f, 0.f, 0.f};  // warps 8-15: a 16 x 8 tile of dW_l
  float dQ1[2][4] = {};                // hidden rows 16 pair, columns 8 (2 hh), 8 (2 hh + 1)

  float po[MAXT][2], pt[MAXT][2];  // the next row's outputs and targets
  auto load_row = [&](int row, int st) {
    const uint32_t tz = smem_u32(smraw + S.sZ) + st * (uint32_t)tile, tv = smem_u32(smraw + S.sV) + st * (uint32_t)tile;
    for (int i = tid; i < 4 * L; i += PROJ_THREADS) {
      cp_async16(tz + tile_off(i >> 2, i & 3), a.zl + (size_t)row * L * C + 8 * i);
      cp_async16(tv + tile_off(i >> 2, i & 3), a.zlm1 + (size_t)row * L * C + 8 * i);
    }
#pragma unroll
    for (int i = 0; i < MAXT; ++i)
      if (pair + 8 * i < T) {
        const size_t p = (size_t)row * L + 16 * (pair + 8 * i) + g;
        po[i][0] = __ldg(a.out + p);
        po[i][1] = __ldg(a.out + p + 8);
        pt[i][0] = __ldg(a.tgt + p);
        pt[i][1] = __ldg(a.tgt + p + 8);
      }
  };
  if (blockIdx.x < a.rows) load_row(blockIdx.x, 0);
  cp_async_commit();

  int st = 0;
  for (int row = blockIdx.x; row < a.rows; row += gridDim.x, st ^= 1) {
    const float cf = __ldg(a.coef + row / L);
    float go[MAXT][2];
#pragma unroll
    for (int i = 0; i < MAXT; ++i) {
      go[i][0] = (po[i][0] - pt[i][0]) * cf;
      go[i][1] = (po[i][1] - pt[i][1]) * cf;
    }
    cp_async_wait<0>();
    __syncthreads();  // this row's inputs; the previous row is done with every tile
    if (row + (int)gridDim.x < a.rows) load_row(row + gridDim.x, st ^ 1);
    cp_async_commit();
    const uint32_t tz = smem_u32(smraw + S.sZ) + st * (uint32_t)tile, tv = smem_u32(smraw + S.sV) + st * (uint32_t)tile,
                   tg = smem_u32(smraw + S.sGz);
    float* xch = reinterpret_cast<float*>(smraw + S.sX);
#pragma unroll 1
    for (int i = 0; i < MAXT; ++i) {
      const int mt = pair + 8 * i;
      if (mt >= T) break;
      const float go0 = i ? go[1][0] : go[0][0], go1 = i ? go[1][1] : go[0][1];
      if (t == 0 && hh == 0) dq2b += go0 + go1;
      uint32_t A[2][4];
      ldsm4(A[0], tz + tile_frag(mt, 0, lane));
      ldsm4(A[1], tz + tile_frag(mt, 1, lane));
      float gz[4][4] = {};
#pragma unroll
      for (int kh = 0; kh < 4; ++kh) {  // hidden channels 64 hh + 16 kh .. + 15
        const int h0 = 64 * hh + 16 * kh;
        uint32_t AG[4];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          uint32_t bq[2][2];
          ldsm_b(bq, smem_u32(sQ1), h0 + 8 * u, lane);
          const float2 b = *reinterpret_cast<const float2*>(sq + h0 + 8 * u + 2 * t);
          const float2 qv = *reinterpret_cast<const float2*>(sq + H + h0 + 8 * u + 2 * t);
          float hc[4] = {b.x, b.y, b.x, b.y};
          mma16816(hc, A[0], bq[0][0], bq[0][1]);
          mma16816(hc, A[1], bq[1][0], bq[1][1]);
          const F2 q = f2(qv.x, qv.y);
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            // GELU and its derivative; gh = go Q2, ghp = gh GELU'(hpre)
            const F2 x = f2(hc[2 * r], hc[2 * r + 1]), x2 = x * x;
            const F2 tt = tanh2(x * fma2(f2(GK0 * GK1), x2, f2(GK0)));
            const F2 hx = f2(0.5f) * x, gr_ = f2(r ? go1 : go0);
            dq2[2 * kh + u] = fma2(gr_, fma2(hx, tt, hx), dq2[2 * kh + u]);
            const F2 d = fma2(hx * fma2(f2(-1.0f) * tt, tt, f2(1.0f)), fma2(f2(3.0f * GK0 * GK1), x2, f2(GK0)),
                              fma2(f2(0.5f), tt, f2(0.5f)));
            const F2 gp = (gr_ * q) * d;
            dq1b[2 * kh + u] = dq1b[2 * kh + u] + gp;
            AG[2 * u + r] = pack2(gp);
          }
        }
        stsm4(gh + gh_off(16 * mt + (lane & 15), h0 / 8 + (lane >> 4)), AG[0], AG[1], AG[2], AG[3]);
        // g_v4 += ghp Q1: B[k = h][n = c], the table read transposed
#pragma unroll
        for (int n2 = 0; n2 < 2; ++n2) {
          uint32_t bq[4];
          ldsm4t(bq, smem_u32(sQ1) + (uint32_t)((h0 + (lane & 15)) * SP + 8 * (2 * n2 + (lane >> 4))) * 2);
          mma16816(gz[2 * n2], AG, bq[0], bq[1]);
          mma16816(gz[2 * n2 + 1], AG, bq[2], bq[3]);
        }
      }
      // channels 16 (1 - hh) .. + 15 go to the other warp of the pair, 16 hh .. stay
      float* mine = xch + warp * 256 + lane * 8;
      const float* other = xch + (warp ^ 1) * 256 + lane * 8;
#pragma unroll
      for (int n = 0; n < 2; ++n)
        *reinterpret_cast<float4*>(mine + 4 * n) =
            hh ? make_float4(gz[n][0], gz[n][1], gz[n][2], gz[n][3])
               : make_float4(gz[2 + n][0], gz[2 + n][1], gz[2 + n][2], gz[2 + n][3]);
      // v_3, the same channels
      {
        uint32_t r[4];
        ldsm4(r, tv + tile_frag(mt, hh, lane));
#pragma unroll
        for (int q = 0; q < 4; ++q) r[q] = pack2(gelu2(unpack_f2(r[q])));
        stsm4(tv + tile_frag(mt, hh, lane), r[0], r[1], r[2], r[3]);
      }
      pair_bar(pair);
      float z[2][4];
#pragma unroll
      for (int n = 0; n < 2; ++n) {
        const float4 o = *reinterpret_cast<const float4*>(other + 4 * n);
        z[n][0] = (hh ? gz[2 + n][0] : gz[n][0]) + o.x;
        z[n][1] = (hh ? gz[2 + n][1] : gz[n][1]) + o.y;
        z[n][2] = (hh ? gz[2 + n][2] : gz[n][2]) + o.z;
        z[n][3] = (hh ? gz[2 + n][3] : gz[n][3]) + o.w;
        vb[n][0] += z[n][0] + z[n][2];
        vb[n][1] += z[n][1] + z[n][3];
      }
      stsm4(tg + tile_frag(mt, hh, lane), pack2(z[0][0], z[0][1]), pack2(z[0][2], z[0][3]), pack2(z[1][0], z[1][1]),
            pack2(z[1][2], z[1][3]));
      pair_bar(pair);  // the exchange is read before it is written again
    }
    __syncthreads();
    if (warp < T) {  // gvpw = g_z W of pixel tile `warp`
      uint32_t AZ[2][4];
      ldsm4(AZ[0], tg + tile_frag(warp, 0, lane));
      ldsm4(AZ[1], tg + tile_frag(warp, 1, lane));
      float d[4][4] = {};
#pragma unroll
      for (int n = 0; n < 4; ++n) {
        uint32_t bw[2][2];
        ldsm_b(bw, smem_u32(sWT), 8 * n, lane);
        mma16816(d[n], AZ[0], bw[0][0], bw[0][1]);
        mma16816(d[n], AZ[1], bw[1][0], bw[1][1]);
      }
      unsigned char* x = smraw + S.sX + warp * 1024;  // as a tile of its own
      tile_put(smem_u32(x), 0, lane, d);
      tile_store(x, 0, lane, a.gvout + ((size_t)row * L + 16 * warp) * C);
    }
    if (warp < 8) row_dft(smem_u32(sTT), LP, tg, T, warp, lane, a.Xg + (size_t)row * M * C);
    else row_dw(tg, tv, T, (warp - 8) >> 2, warp & 3, lane, dW);
    {  // dQ1: hidden rows 16 pair .. + 15 by channels 16 hh .. + 15
      const int px = (lane & 7) + 8 * (lane >> 4), ch = 2 * pair + ((lane >> 3) & 1);
#pragma unroll 4
      for (int ks = 0; ks < T; ++ks) {
        uint32_t A[4], b[4];
        ldsm4t(A, gh + gh_off(16 * ks + px, ch));
        ldsm4t(b, tz + tile_off(16 * ks + (lane & 15), 2 * hh + (lane >> 4)));
        mma16816(dQ1[0], A, b[0], b[1]);
        mma16816(dQ1[1], A, b[2], b[3]);
      }
    }
  }

  // ---- per-CTA partials; over the warps in a fixed order, so that the gradient repeats bit for bit ----
  float* gp = a.gpart + (size_t)blockIdx.x * Dn::N;
  cp_async_wait<0>();
  __syncthreads();
  float* sRed = reinterpret_cast<float*>(smraw + S.sGH);
  float* red = sRed + warp * PROJ_RED;
#pragma unroll
  for (int nh = 0; nh < 8; ++nh) {
    const float2 b = f2_get(dq1b[nh]), q = f2_get(dq2[nh]);
    const float s0 = red_g(b.x), s1 = red_g(b.y), s2 = red_g(q.x), s3 = red_g(q.y);
    if (g == 0) {
      red[8 * nh + 2 * t] = s0;
      red[8 * nh + 2 * t + 1] = s1;
      red[64 + 8 * nh + 2 * t] = s2;
      red[64 + 8 * nh + 2 * t + 1] = s3;
    }
  }
#pragma unroll
  for (int n = 0; n < 2; ++n)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const float s = red_g(vb[n][e]);
      if (g == 0) red[H + 8 * n + 2 * t + e] = s;
    }
  float sb = dq2b;
  for (int k = 16; k > 0; k >>= 1) sb += __shfl_xor_sync(0xffffffffu, sb, k);
  if (lane == 0) red[H + 16] = sb;
  __syncthreads();
  for (int i = tid; i < 2 * H + C + 1; i += PROJ_THREADS) {
    int w, slot, dst;  // first warp of the half, its slot, where it goes
    if (i < H) {
      w = i >= 64;
      slot = i & 63;
      dst = Dn::q1b + i;
    } else if (i < 2 * H) {
      w = i - H >= 64;
      slot = 64 + (i & 63);
      dst = Dn::Q2 + i - H;
    } else if (i < 2 * H + C) {
      w = i - 2 * H >= 16;
      slot = H + (i & 15);
      dst = Dn::Wb + l * C + i - 2 * H;
    } else {
      w = 0;
      slot = H + 16;
      dst = Dn::q2b;
    }
    float s = 0.f;
    for (; w < PROJ_WARPS; w += 2) s += sRed[w * PROJ_RED + slot];
    gp[dst] = s;
  }
  if (warp >= 8) put_dw(gp + Dn::W + l * C * C, (warp - 8) >> 2, warp & 3, lane, dW);
  {
    const int h = 16 * pair + g;
#pragma unroll
    for (int n = 0; n < 2; ++n) {
      float* w = gp + Dn::Q1 + h * C + 16 * hh + 8 * n + 2 * t;
      w[0] = dQ1[n][0];
      w[1] = dQ1[n][1];
      w[8 * C] = dQ1[n][2];
      w[8 * C + 1] = dQ1[n][3];
    }
  }
}

// dense partials -> gradient vector
__global__ void reduce_dense_kernel(const float* __restrict__ gpart, int nparts, float* __restrict__ grad) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= Dn::N) return;
  float s = 0.f;
  for (int p = 0; p < nparts; ++p) s += gpart[(size_t)p * Dn::N + i];
  grad[dense_to_param(i)] = s;
}

// dR[j][kx][c][o] = s_kx sum_b gU_b[j][kx][o] conj(V_b[j][kx][c]); one CTA per (j, kx), the operands of
// DR_MASKS masks at a time in shared memory (one mask between two barriers, its load exposed, took
// 20 us for 32 masks; now 8)
constexpr int DR_MASKS = 32;
__global__ void __launch_bounds__(THREADS) dR_kernel(int L, int B, int layer, const float2* __restrict__ gU,
                                                     const float2* __restrict__ V, float* __restrict__ grad) {
  const int jk = blockIdx.x, tid = threadIdx.x;  // jk = j * M + kx
  const int kx = jk % M, lane = tid & 31, warp = tid >> 5;
  __shared__ float2 su[DR_MASKS][C], sv[DR_MASKS][C];
  early_next();
  early_wait(gU);
  early_wait(V);
  float2 acc[4] = {};  // c = warp + 8 r, o = lane
  for (int b0 = 0; b0 < B; b0 += DR_MASKS) {
    const int nb = min(DR_MASKS, B - b0);
    __syncthreads();
#pragma unroll
    for (int q = 0; q < DR_MASKS / 8; ++q) {
      const int b = warp + 8 * q;
      if (b < nb) {
        const size_t i = ((size_t)(b0 + b) * J * M + jk) * C + lane;
        su[b][lane] = __ldg(gU + i);
        sv[b][lane] = __ldg(V + i);
      }
    }
    __syncthreads();
#pragma unroll 4
    for (int b = 0; b < nb; ++b) {
      const float2 u = su[b][lane];
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const float2 v = sv[b][warp + 8 * r];
        acc[r].x += u.x * v.x + u.y * v.y;
        acc[r].y += u.y * v.x - u.x * v.y;
      }
    }
  }
  const float s = (kx == 0 ? 1.0f : 2.0f) / ((float)L * (float)L);
  float2* out = reinterpret_cast<float2*>(grad + Off::R + (size_t)layer * Off::RL) + (size_t)jk * C * C;
#pragma unroll
  for (int r = 0; r < 4; ++r) out[tid + THREADS * r] = make_float2(s * acc[r].x, s * acc[r].y);
}

// Adam (torch semantics: L2 weight decay added to the gradient)
__global__ void adam_kernel(size_t n, float* __restrict__ p, const float* __restrict__ gr, float* __restrict__ m,
                            float* __restrict__ v, float lr, float b1, float b2, float eps, float wd, float bc1,
                            float bc2) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const float g = gr[i] + wd * p[i];
    const float mi = b1 * m[i] + (1.f - b1) * g;
    const float vi = b2 * v[i] + (1.f - b2) * g * g;
    m[i] = mi;
    v[i] = vi;
    p[i] -= lr * (mi / bc1) / (sqrtf(vi / bc2) + eps);
  }
}

// ---------------------------------------------------------------------------
// seeded rectangle masks (SplitMix64 counters); one CTA per mask
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint64_t splitmix(uint64_t x) {
  uint64_t z = x + 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

__global__ void rect_masks_kernel(uint64_t seed, long long first, int L, int nmin, int nmax, int wmin, int wmax,
                                  float* __restrict__ out) {
  __shared__ int4 rc[256];
  __shared__ int nr;
  const uint64_t i = (uint64_t)(first + blockIdx.x);
  const uint64_t base = seed * 0xD1B54A32D192ED03ull + i * 0x9E3779B97F4A7C15ull;
  if (threadIdx.x == 0) nr = nmin + (int)(splitmix(base) % (uint64_t)(nmax - nmin + 1));
  __syncthreads();
  const uint64_t span = (uint64_t)(wmax - wmin + 1);
  for (int r = threadIdx.x; r < nr; r += blockDim.x) {
    const int w = wmin + (int)(splitmix(base + 1 + 4 * r) % span);
    const int h = wmin + (int)(splitmix(base + 2 + 4 * r) % span);
    const int x0 = (int)(splitmix(base + 3 + 4 * r) % (uint64_t)(L - w + 1));
    const int y0 = (int)(splitmix(base + 4 + 4 * r) % (uint64_t)(L - h + 1));
    rc[r] = make_int4(x0, y0, x0 + w, y0 + h);
  }
  __syncthreads();
  float* m = out + (size_t)blockIdx.x * L * L;
  for (int p = threadIdx.x; p < L * L; p += blockDim.x) {
    const int y = p / L, x = p % L;
    float v = 0.f;
    for (int r = 0; r < nr; ++r) {
      const int4 q = rc[r];
      if (x >= q.x && x < q.z && y >= q.y && y < q.w) {
        v = 1.f;
        break;
      }
    }
    m[p] = v;
  }
}

// ---------------------------------------------------------------------------
// band projection of an image onto |kx| <= KB, |ky| <= KBy (the support of any
// SOCS image with kernels of half-width Nx = KB/2, Ny = KBy/2) and its
// out-of-band residual, the surrogate's error estimate.
// ---------------------------------------------------------------------------
// x-DFT of each row at kx = 0..KB (KB <= 15)
__global__ void __launch_bounds__(THREADS) band_rows_kernel(int L, int rows, int KB, const float* __restrict__ img,
                                                            const float2* __restrict__ twL, float2* __restrict__ Xb) {
  extern __shared__ __align__(16) unsigned char smraw[];
  early_next();
  float2* sTw = reinterpret_cast<float2*>(smraw);
  for (int i = threadIdx.x; i < L; i += THREADS) sTw[i] = twL[i];
  __syncthreads();
  early_wait(img);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int row0 = (blockIdx.x * (THREADS / 32) + warp) * DR, n = min(DR, rows - row0);
  if (n <= 0) return;
  float re[DR], im[DR];
  rows_dft(L, img + (size_t)row0 * L, n, reinterpret_cast<float4*>(sTw + L) + (size_t)warp * L, sTw, re, im);
#pragma unroll
  for (int r = 0; r < DR; ++r)
    if (r < n && lane <= KB && lane < 16) Xb[(size_t)(row0 + r) * 16 + lane] = make_float2(re[r], im[r]);
}

// C[ky + KBy][kx] = sum_y X[y][kx] e^{-i ky y} for kx <= KB, |ky| <= KBy (plain 2-D DFT).  One CTA
// per mask and ky: 16 kx by 16 shares of the rows, added in order (one thread per coefficient over
// all rows, one CTA per mask, took 85 us for 64 masks of 256 x 256; now 6).
__global__ void __launch_bounds__(THREADS) band_coef_kernel(int L, int KB, int KBy, const float2* __restrict__ Xb,
                                                            const float2* __restrict__ twL, float2* __restrict__ Cb) {
  __shared__ float2 part[THREADS / 16][16];
  early_next();
  early_wait(Xb);
  const int b = blockIdx.y, kyi = blockIdx.x, ky = kyi - KBy, kx = threadIdx.x & 15, sh = threadIdx.x >> 4;
  float re = 0.f, im = 0.f;
  if (kx <= KB) {
#pragma unroll 4
    for (int y = sh; y < L; y += THREADS / 16) {
      const float2 x = __ldg(Xb + ((size_t)b * L + y) * 16 + kx);
      const float2 w = __ldg(twL + (((ky + L) * y) & (L - 1)));  // e^{+i ky y}; use conj
      re = fmaf(x.x, w.x, fmaf(x.y, w.y, re));
      im = fmaf(x.y, w.x, fmaf(-x.x, w.y, im));
    }
  }
  part[sh][kx] = make_float2(re, im);
  __syncthreads();
  if (sh == 0 && kx <= KB) {
    for (int s = 1; s < THREADS / 16; ++s) {
      re += part[s][kx].x;
      im += part[s][kx].y;
    }
    Cb[((size_t)b * gridDim.x + kyi) * 16 + kx] = make_float2(re, im);
  }
}

// in-place synthesis of the band: img[y][x] = 1/L^2 sum_kx w_kx Re(G_y[kx] e^{i kx x}),
// G_y[kx] = sum_ky Cb[ky][kx] e^{i ky y}; per-row energies of the removed part and of the result.
// One warp per row, a lane per kx and then per pixel of each 32, so that nothing waits for another
// warp (a CTA per row, two barriers apart: 75 us for 16,384 rows of 256; now 18).
__global__ void __launch_bounds__(THREADS) band_synth_kernel(int L, int rows, int KB, int KBy,
                                                             const float2* __restrict__ Cb,
                                                             const float2* __restrict__ twL, float* __restrict__ img,
                                                             float* __restrict__ Eres, float* __restrict__ Enew) {
  __shared__ float2 sTw[256];
  constexpr int MAXI = 256 / 32;
  for (int i = threadIdx.x; i < L; i += THREADS) sTw[i] = twL[i];
  __syncthreads();
  early_next();
  early_wait(Cb);
  const int row = blockIdx.x * (THREADS / 32) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (row >= rows) return;
  const int b = row / L, y = row % L, nky = 2 * KBy + 1, kx = lane & 15;
  float* p = img + (size_t)row * L;
  float old[MAXI];
#pragma unroll
  for (int i = 0; i < MAXI; ++i) old[i] = 32 * i < L ? p[lane + 32 * i] : 0.f;
  float re = 0.f, im = 0.f;
  if (kx <= KB) {
    const float2* cb = Cb + (size_t)b * nky * 16 + kx;
#pragma unroll 4
    for (int kyi = 0; kyi < nky; ++kyi) {
      const float2 c = __ldg(cb + kyi * 16);
      const float2 w = sTw[((kyi - KBy + L) * y) & (L - 1)];
      re = fmaf(c.x, w.x, fmaf(-c.y, w.y, re));
      im = fmaf(c.x, w.y, fmaf(c.y, w.x, im));
    }
    const float sc = (kx == 0 ? 1.f : 2.f) / ((float)L * (float)L);
    re *= sc;
    im *= sc;
  }
  float v[MAXI] = {};
  for (int k = 0; k <= KB; ++k) {
    const float gx = __shfl_sync(0xffffffffu, re, k), gy = __shfl_sync(0xffffffffu, im, k);
#pragma unroll
    for (int i = 0; i < MAXI; ++i)
      if (32 * i < L) {
        const float2 w = sTw[(k * (lane + 32 * i)) & (L - 1)];
        v[i] = fmaf(gx, w.x, fmaf(-gy, w.y, v[i]));
      }
  }
  float er = 0.f, en = 0.f;
#pragma unroll
  for (int i = 0; i < MAXI; ++i)
    if (32 * i < L) {
      const float d = old[i] - v[i];
      er = fmaf(d, d, er);
      en = fmaf(v[i], v[i], en);
      p[lane + 32 * i] = v[i];
    }
#pragma unroll
  for (int k = 16; k > 0; k >>= 1) {
    er += __shfl_xor_sync(0xffffffffu, er, k);
    en += __shfl_xor_sync(0xffffffffu, en, k);
  }
  if (lane == 0) {
    Eres[row] = er;
    Enew[row] = en;
  }
}

// est[b] = alpha * sqrt(sum_rows Eres / sum_rows Enew)
__global__ void oob_est_kernel(int L, int B, const float* __restrict__ Eres, const float* __restrict__ Enew,
                               float alpha, float* __restrict__ est) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= B) return;
  double a = 0.0, c = 0.0;
  for (int y = 0; y < L; ++y) {
    a += Eres[(size_t)b * L + y];
    c += Enew[(size_t)b * L + y];
  }
  est[b] = c > 0.0 ? (float)(alpha * sqrt(a / c)) : INFINITY;
}

// Exact image coefficients at the five lowest frequencies q in {(0,0), (1,0), (0,1),
// (1,1), (-1,1)} (with their conjugates the 3 x 3 lowest block):
//   I(q) = 1/L^2 sum_k s_k sum_f B_k(f + q) conj(B_k(f)),  B_k(f) = krn_k(f) M(f),
// M the plain DFT of the mask on the (2Nx+1) x (2Ny+1) window (Cm holds u >= 0).
// est[b] = alpha * sqrt(sum_q w_q |I_net(q) - I(q)|^2 / L^2) / ||image||, w = 1 at DC, 2 else.
// One CTA per mask, one thread per q and kernel.
constexpr int LOWQ_THREADS = 5 * 64;
__global__ void __launch_bounds__(LOWQ_THREADS) lowq_est_kernel(int L, int Nx, int Ny, const float2* __restrict__ Cm,
                                                       const float2* __restrict__ Cb, const float2* __restrict__ krn,
                                                       const float* __restrict__ scales, int nk,
                                                       const float* __restrict__ Enew, float alpha,
                                                       float* __restrict__ est) {
  const int b = blockIdx.x, tid = threadIdx.x;
  const int KX = 2 * Nx + 1, KY = 2 * Ny + 1, KD = KX * KY;
  __shared__ float2 sM[33 * 33];
  __shared__ float2 part[5][64];
  __shared__ double en;
  early_wait(Cm);
  early_wait(Cb);
  early_wait(Enew);
  for (int i = tid; i < KD; i += blockDim.x) {
    const int v = i / KX - Ny, u = i % KX - Nx;
    float2 m;
    if (u >= 0) {
      m = Cm[((size_t)b * KY + (v + Ny)) * 16 + u];
    } else {
      const float2 c = Cm[((size_t)b * KY + (-v + Ny)) * 16 + (-u)];
      m = make_float2(c.x, -c.y);
    }
    sM[i] = m;
  }
  if (tid < 32) {
    double a = 0.0;
    for (int y = tid; y < L; y += 32) a += Enew[(size_t)b * L + y];
    for (int k = 16; k > 0; k >>= 1) a += __shfl_xor_sync(0xffffffffu, a, k);
    if (tid == 0) en = a;
  }
  __syncthreads();
  const int qx[5] = {0, 1, 0, 1, -1}, qy[5] = {0, 0, 1, 1, 1};
  for (int p = tid; p < 5 * 64; p += blockDim.x) {
    const int qi = p / 64, k = p % 64;
    float re = 0.f, im = 0.f;
    if (k < nk) {
      const float2* kk = krn + (size_t)k * KD;
      for (int i = 0; i < KD; ++i) {
        const int v = i / KX - Ny, u = i % KX - Nx;
        const int v2 = v + qy[qi], u2 = u + qx[qi];
        if (v2 < -Ny || v2 > Ny || u2 < -Nx || u2 > Nx) continue;
        const int j = (v2 + Ny) * KX + (u2 + Nx);
        const float2 a = cmulf(kk[j], sM[j]), c = cmulf(kk[i], sM[i]);
        re = fmaf(a.x, c.x, fmaf(a.y, c.y, re));   // a conj(c)
        im = fmaf(a.y, c.x, fmaf(-a.x, c.y, im));
      }
      re *= scales[k];
      im *= scales[k];
    }
    part[qi][k] = make_float2(re, im);
  }
  __syncthreads();
  if (tid < 32) {
    float d2 = 0.f;
    for (int qi = 0; qi < 5; ++qi) {
      float re = part[qi][tid].x + part[qi][tid + 32].x, im = part[qi][tid].y + part[qi][tid + 32].y;
      for (int k = 16; k > 0; k >>= 1) {
        re += __shfl_xor_sync(0xffffffffu, re, k);
        im += __shfl_xor_sync(0xffffffffu, im, k);
      }
      const float inv = 1.0f / ((float)L * (float)L);
      re *= inv;
      im *= inv;
      float2 net;
      const int KBy = 2 * Ny;
      if (qx[qi] >= 0) {
        net = Cb[((size_t)b * (2 * KBy + 1) + (qy[qi] + KBy)) * 16 + qx[qi]];
      } else {
        const float2 c = Cb[((size_t)b * (2 * KBy + 1) + (-qy[qi] + KBy)) * 16 + (-qx[qi])];
        net = make_float2(c.x, -c.y);
      }
      const float dr = net.x - re, di = net.y - im;
      d2 += (qi == 0 ? 1.f : 2.f) * (dr * dr + di * di);
    }
    if (tid == 0) {
      const double e = sqrt((double)d2) / (double)L;
      est[b] = en > 0.0 ? (float)(alpha * e / sqrt(en)) : INFINITY;
    }
  }
}

}  // namespace fno
}  // namespace litho

// ===========================================================================
// host side
// ===========================================================================
using namespace litho;
using namespace litho::fno;

struct litho_fno {
  litho_ctx* ctx = nullptr;
  int L = 0;
  int cap = 0;  // batch capacity of the workspaces
  long long step = 0;
  DevBuf theta, grad, adam_m, adam_v;
  DevBuf Ttab, TT, twL, colF, colI;  // tables; the column kernel's as fragments
  DevBuf z[NL];      // z_l (training keeps all; inference ping-pongs z[0], z[1])
  DevBuf Xf, Gy;     // per-row spectral intermediates (also Xg, Gg in backward)
  DevBuf Vs[NL], gU;
  DevBuf gv[2];      // gvpw ping-pong
  DevBuf out, lossb, lossp, coef, gpart;
  int bwd_grid = 0;
  // error estimate = alpha * ||out-of-band residual|| / ||band part||
  float est_alpha = 1.0f;
  DevBuf Xb, Eres, Enew, Cb, Mrow, Cm, est, stage_m, stage_i;
};

namespace {

int fwd_grid(litho_fno* f, int rows) { return std::max(1, std::min(rows, FWD_CTAS * f->ctx->sm_count)); }
int fno_grid(litho_fno* f, int rows) { return std::max(1, std::min(rows, 2 * f->ctx->sm_count)); }

// The column kernel over B masks, in groups of four, two or one: the more masks share the reading of
// R the better, while there are three CTAs for every two SMs (32 masks, us
// forward and backward: four a CTA, 128 CTAs, 47 and 46; two, 256, 31 and 36; one, 512, 46 and 56)
template <bool BWD>
int launch_column(litho_fno* f, int B, int layer, const float2* Xin, float2* Gout, float2* modes_out) {
  litho_ctx* ctx = f->ctx;
  auto go = [&](auto* k, int G) {
    const size_t smem = column_smem(G, BWD);
    cudaError_t e = allow_smem(k);
    if (e != cudaSuccess) return e;
    return launch_early(true, k, dim3(M, (B + G - 1) / G), THREADS, smem, ctx->stream, f->L, B, f->theta.as<float>(), layer,
                        Xin, Gout, modes_out, f->colF.as<uint4>(), f->colI.as<uint4>());
  };
  const int want = 3 * ctx->sm_count / 2;
  cudaError_t e;
  if (M * ((B + 3) / 4) >= want) e = go(column_kernel<BWD, 4>, 4);
  else if (M * ((B + 1) / 2) >= want) e = go(column_kernel<BWD, 2>, 2);
  else e = go(column_kernel<BWD, 1>, 1);
  LITHO_CUDA_TRY(ctx, e);
  return LITHO_OK;
}

int ensure_batch(litho_fno* f, int B, bool train) {
  litho_ctx* ctx = f->ctx;
  const size_t L = f->L;
  const size_t act = (size_t)B * L * L * C * sizeof(bf16);
  const size_t row = (size_t)B * L * M * C * sizeof(float2);
  for (int l = 0; l < (train ? NL : 2); ++l) LITHO_RET(f->z[l].ensure(ctx, act));
  LITHO_RET(f->Xf.ensure(ctx, row));
  LITHO_RET(f->Gy.ensure(ctx, row));
  LITHO_RET(f->out.ensure(ctx, (size_t)B * L * L * sizeof(float)));
  LITHO_RET(f->lossb.ensure(ctx, (size_t)B * sizeof(float)));
  LITHO_RET(f->coef.ensure(ctx, (size_t)B * sizeof(float)));
  if (train) {
    LITHO_RET(f->lossp.ensure(ctx, (size_t)B * LOSS_SHARES * sizeof(double2)));
    for (int l = 0; l < NL; ++l) LITHO_RET(f->Vs[l].ensure(ctx, (size_t)B * J * M * C * sizeof(float2)));
    LITHO_RET(f->gU.ensure(ctx, (size_t)B * J * M * C * sizeof(float2)));
    LITHO_RET(f->gv[0].ensure(ctx, act));
    LITHO_RET(f->gv[1].ensure(ctx, act));
    f->bwd_grid = fno_grid(f, (int)(B * L));
    LITHO_RET(f->gpart.ensure(ctx, (size_t)f->bwd_grid * Dn::N * sizeof(float)));
  }
  return LITHO_OK;
}

// CTAs of the kernels that take DR rows a warp
int dft_blocks(int rows) { return (rows + DR * THREADS / 32 - 1) / (DR * THREADS / 32); }

// masks in launches of at most 65,535, the limit of the grid's second dimension
int launch_band_coef(litho_fno* f, int KB, int KBy, int batch, const float2* X, float2* Cb) {
  litho_ctx* ctx = f->ctx;
  const int nky = 2 * KBy + 1;
  for (int b = 0; b < batch; b += 65535) {
    LITHO_CUDA_TRY(ctx, launch_early(true, band_coef_kernel, dim3(nky, std::min(65535, batch - b)), THREADS, 0, ctx->stream, f->L,
                                     KB, KBy, X + (size_t)b * f->L * 16, f->twL.as<float2>(), Cb + (size_t)b * nky * 16));
  }
  return LITHO_OK;
}

// forward pass over B masks; train keeps z_l and V_l for the backward pass.  From the second kernel on
// each is launched early, here and in the passes below: it loads its tables and weights while the one
// before it ends, and waits before it touches anything a pass writes (64 masks of 256 x 256, predict:
// 1,000 -> 959 us; 32, loss and gradients: 1,910 -> 1,847).
int forward(litho_fno* f, const float* masks, int B, bool train, float* images, float2* Mrow = nullptr) {
  litho_ctx* ctx = f->ctx;
  const int L = f->L, rows = B * L;
  const float* th = f->theta.as<float>();
  LITHO_CUDA_TRY(ctx, allow_smem(row_fwd_kernel<FWD_FIRST>));
  LITHO_CUDA_TRY(ctx, allow_smem(row_fwd_kernel<FWD_MID>));
  LITHO_CUDA_TRY(ctx, allow_smem(row_fwd_kernel<FWD_LAST>));
  StageScope sc(ctx, LITHO_STAGE_SURROGATE, 2 * NL + 1);
  lift_dft_kernel<<<dft_blocks(rows), THREADS, rows_dft_smem(L), ctx->stream>>>(L, rows, th, masks, f->twL.as<float2>(),
                                                                               f->Xf.as<float2>(), Mrow);
  const int grid = fwd_grid(f, rows);
  for (int l = 0; l < NL; ++l) {
    LITHO_RET(launch_column<false>(f, B, l, f->Xf.as<float2>(), f->Gy.as<float2>(),
                                   train ? f->Vs[l].as<float2>() : nullptr));
    RowFwd a;
    a.L = L; a.rows = rows; a.layer = l; a.theta = th; a.masks = masks;
    a.act_in = train ? 1 : 0;   // training keeps z_l, inference keeps GELU(z_l)
    a.act_out = train ? 0 : 1;
    a.zin = l == 0 ? nullptr : (train ? f->z[l - 1].as<bf16>() : f->z[(l - 1) & 1].as<bf16>());
    a.Gy = f->Gy.as<float2>();
    a.zout = train ? f->z[l].as<bf16>() : (l < NL - 1 ? f->z[l & 1].as<bf16>() : nullptr);
    a.Xf = f->Xf.as<float2>();
    a.out = images;
    a.Ttab = f->Ttab.as<bf16>(); a.TT = f->TT.as<bf16>();
    if (l == 0)
      LITHO_CUDA_TRY(ctx, launch_early(true, row_fwd_kernel<FWD_FIRST>, dim3(grid), THREADS, row_fwd_smem(L, false), ctx->stream, a));
    else if (l < NL - 1)
      LITHO_CUDA_TRY(ctx, launch_early(true, row_fwd_kernel<FWD_MID>, dim3(grid), THREADS, row_fwd_smem(L, false), ctx->stream, a));
    else
      LITHO_CUDA_TRY(ctx, launch_early(true, row_fwd_kernel<FWD_LAST>, dim3(grid), THREADS, row_fwd_smem(L, true), ctx->stream, a));
  }
  LITHO_CUDA_TRY(ctx, cudaGetLastError());
  return LITHO_OK;
}

cudaError_t launch_loss(litho_fno* f, const float* targets, int B) {
  cudaStream_t s = f->ctx->stream;
  const cudaError_t e = launch_early(true, loss_part_kernel, dim3((unsigned)B * LOSS_SHARES), THREADS, 0, s, f->L,
                                     f->out.as<float>(), targets, f->lossp.as<double2>());
  if (e != cudaSuccess) return e;
  return launch_early(true, loss_kernel, dim3((B + 31) / 32), 32, 0, s, B, f->lossp.as<double2>(), f->lossb.as<float>(),
                      f->coef.as<float>());
}

// loss (device, per mask) + gradient into f->grad
int backward(litho_fno* f, const float* masks, const float* targets, int B) {
  litho_ctx* ctx = f->ctx;
  const int L = f->L, rows = B * L, grid = f->bwd_grid;
  const float* th = f->theta.as<float>();
  const BwdSmem ss(L, HEAD_SPEC), sl(L, HEAD_LIFT);
  const ProjSmem sp(L);
  LITHO_CUDA_TRY(ctx, allow_smem(row_bwd_proj_kernel));
  LITHO_CUDA_TRY(ctx, allow_smem(row_bwd_kernel<HEAD_SPEC>));
  LITHO_CUDA_TRY(ctx, allow_smem(row_bwd_kernel<HEAD_LIFT>));
  StageScope sc(ctx, LITHO_STAGE_SURROGATE, 3 * NL + 4);
  LITHO_CUDA_TRY(ctx, launch_loss(f, targets, B));
  LITHO_CUDA_TRY(ctx, cudaMemsetAsync(f->gpart.p, 0, (size_t)grid * Dn::N * sizeof(float), ctx->stream));
  float2* Xg = f->Xf.as<float2>();
  float2* Gg = f->Gy.as<float2>();
  RowBwd a{};
  a.L = L; a.rows = rows; a.theta = th; a.masks = masks;
  a.out = f->out.as<float>(); a.tgt = targets; a.coef = f->coef.as<float>();
  a.Xg = Xg; a.Gg = Gg; a.gpart = f->gpart.as<float>();
  a.Ttab = f->Ttab.as<bf16>(); a.TT = f->TT.as<bf16>();
  int cur = 0;
  for (int l = NL - 1; l >= 0; --l) {
    a.layer = l;
    a.zl = f->z[l].as<bf16>();
    a.zlm1 = l > 0 ? f->z[l - 1].as<bf16>() : nullptr;
    a.gvin = f->gv[cur ^ 1].as<bf16>();
    a.gvout = f->gv[cur].as<bf16>();
    if (l == NL - 1)
      row_bwd_proj_kernel<<<std::min(rows, ctx->sm_count), PROJ_THREADS, sp.total, ctx->stream>>>(a);
    else
      LITHO_CUDA_TRY(ctx, launch_early(true, row_bwd_kernel<HEAD_SPEC>, dim3(grid), THREADS, ss.total, ctx->stream, a));
    LITHO_RET(launch_column<true>(f, B, l, Xg, Gg, f->gU.as<float2>()));
    LITHO_CUDA_TRY(ctx, launch_early(true, dR_kernel, dim3(J * M), THREADS, 0, ctx->stream, L, B, l, f->gU.as<float2>(),
                                     f->Vs[l].as<float2>(), f->grad.as<float>()));
    cur ^= 1;
  }
  a.layer = 0;
  a.gvin = f->gv[cur ^ 1].as<bf16>();
  LITHO_CUDA_TRY(ctx, launch_early(true, row_bwd_kernel<HEAD_LIFT>, dim3(grid), THREADS, sl.total, ctx->stream, a));
  reduce_dense_kernel<<<(Dn::N + 255) / 256, 256, 0, ctx->stream>>>(f->gpart.as<float>(), grid,
                                                                    f->grad.as<float>());
  LITHO_CUDA_TRY(ctx, cudaGetLastError());
  return LITHO_OK;
}

// band projection of `images` onto |kx| <= 2Nx, |ky| <= 2Ny (in place) -> f->Cb, f->Eres, f->Enew
int project(litho_fno* f, int Nx, int Ny, float* images, int batch) {
  litho_ctx* ctx = f->ctx;
  const int L = f->L, rows = batch * L, KB = 2 * Nx, KBy = 2 * Ny;
  LITHO_RET(f->Xb.ensure(ctx, (size_t)rows * 16 * sizeof(float2)));
  LITHO_RET(f->Eres.ensure(ctx, (size_t)rows * sizeof(float)));
  LITHO_RET(f->Enew.ensure(ctx, (size_t)rows * sizeof(float)));
  LITHO_RET(f->Cb.ensure(ctx, (size_t)batch * (2 * KBy + 1) * 16 * sizeof(float2)));
  StageScope sc(ctx, LITHO_STAGE_SURROGATE, 3);
  LITHO_CUDA_TRY(ctx, launch_early(true, band_rows_kernel, dim3(dft_blocks(rows)), THREADS, rows_dft_smem(L), ctx->stream, L,
                                   rows, KB, images, f->twL.as<float2>(), f->Xb.as<float2>()));
  LITHO_RET(launch_band_coef(f, KB, KBy, batch, f->Xb.as<float2>(), f->Cb.as<float2>()));
  LITHO_CUDA_TRY(ctx, launch_early(true, band_synth_kernel, dim3((rows + 7) / 8), THREADS, 0, ctx->stream, L, rows, KB, KBy,
                                   f->Cb.as<float2>(), f->twL.as<float2>(), images, f->Eres.as<float>(), f->Enew.as<float>()));
  LITHO_CUDA_TRY(ctx, cudaGetLastError());
  return LITHO_OK;
}

// network -> band projection -> exact low-frequency check (est on the device)
int predict(litho_fno* f, const litho_kernel_set* ks, const float* masks, int batch, float* images, float* est) {
  litho_ctx* ctx = f->ctx;
  const int L = f->L, rows = batch * L;
  LITHO_RET(ensure_batch(f, batch, false));
  LITHO_RET(f->Mrow.ensure(ctx, (size_t)rows * 16 * sizeof(float2)));
  LITHO_RET(f->Cm.ensure(ctx, (size_t)batch * (2 * ks->Ny + 1) * 16 * sizeof(float2)));
  LITHO_RET(forward(f, masks, batch, false, images, f->Mrow.as<float2>()));
  LITHO_RET(project(f, ks->Nx, ks->Ny, images, batch));
  StageScope sc(ctx, LITHO_STAGE_SURROGATE, 2);
  LITHO_RET(launch_band_coef(f, ks->Nx, ks->Ny, batch, f->Mrow.as<float2>(), f->Cm.as<float2>()));
  LITHO_CUDA_TRY(ctx, launch_early(true, lowq_est_kernel, dim3(batch), LOWQ_THREADS, 0, ctx->stream, L, ks->Nx, ks->Ny,
                                   f->Cm.as<float2>(), f->Cb.as<float2>(), ks->krn, ks->scales, ks->nk, f->Enew.as<float>(),
                                   f->est_alpha, est));
  LITHO_CUDA_TRY(ctx, cudaGetLastError());
  return LITHO_OK;
}

// Kaiming-uniform linear layers and FNO spectral weights (scale/(in*out) * U[0,1))
void init_params(std::vector<float>& p, unsigned long long seed) {
  std::mt19937_64 rng(seed);
  auto uni = [&](float lo, float hi) {
    return lo + (hi - lo) * (float)((rng() >> 11) * (1.0 / 9007199254740992.0));
  };
  p.assign(Off::N, 0.f);
  for (int i = 0; i < C; ++i) p[Off::Pw + i] = uni(-1.f, 1.f);
  for (int i = 0; i < C; ++i) p[Off::Pb + i] = uni(-1.f, 1.f);
  const float bw = 1.0f / std::sqrt((float)C);
  for (int l = 0; l < NL; ++l) {
    for (int i = 0; i < C * C; ++i) p[Off::W + (size_t)l * C * C + i] = uni(-bw, bw);
    for (int i = 0; i < C; ++i) p[Off::Wb + (size_t)l * C + i] = uni(-bw, bw);
  }
  const float sc = 1.0f / (float)(C * C);
  for (size_t i = 0; i < NL * Off::RL; ++i) p[Off::R + i] = sc * uni(0.f, 1.f);
  for (int i = 0; i < H * C; ++i) p[Off::Q1 + i] = uni(-bw, bw);
  for (int i = 0; i < H; ++i) p[Off::q1b + i] = uni(-bw, bw);
  const float bh = 1.0f / std::sqrt((float)H);
  for (int i = 0; i < H; ++i) p[Off::Q2 + i] = uni(-bh, bh);
  p[Off::q2b] = uni(-bh, bh);
}

}  // namespace

extern "C" {

long long litho_surrogate_num_params(void) { return (long long)Off::N; }

int litho_surrogate_create(litho_ctx* ctx, int L, unsigned long long seed, litho_fno** out) {
  if (ctx == nullptr || out == nullptr) return LITHO_ERR_ARG;
  *out = nullptr;
  LITHO_ARG_CHECK(ctx, L == 64 || L == 128 || L == 256, "surrogate grid L=%d must be 64, 128 or 256", L);
  LITHO_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  litho_fno* f = new litho_fno;
  f->ctx = ctx;
  f->L = L;
  int rc = LITHO_OK;
  do {
    const size_t pb = Off::N * sizeof(float);
    if ((rc = f->theta.ensure(ctx, pb)) || (rc = f->grad.ensure(ctx, pb)) || (rc = f->adam_m.ensure(ctx, pb)) ||
        (rc = f->adam_v.ensure(ctx, pb)))
      break;
    if ((rc = f->Ttab.ensure(ctx, (size_t)L * J * sizeof(bf16))) || (rc = f->TT.ensure(ctx, (size_t)L * J * sizeof(bf16))) ||
        (rc = f->twL.ensure(ctx, (size_t)L * sizeof(float2))) || (rc = f->colF.ensure(ctx, (size_t)L * 32 * sizeof(uint4))) ||
        (rc = f->colI.ensure(ctx, (size_t)L * 32 * sizeof(uint4))))
      break;
    std::vector<float> p;
    init_params(p, seed);
    if (cudaMemcpyAsync(f->theta.p, p.data(), pb, cudaMemcpyHostToDevice, ctx->stream) != cudaSuccess ||
        cudaMemsetAsync(f->adam_m.p, 0, pb, ctx->stream) != cudaSuccess ||
        cudaMemsetAsync(f->adam_v.p, 0, pb, ctx->stream) != cudaSuccess ||
        cudaMemsetAsync(f->grad.p, 0, pb, ctx->stream) != cudaSuccess) {
      set_error(ctx, LITHO_ERR_CUDA, "surrogate parameter upload failed");
      rc = LITHO_ERR_CUDA;
      break;
    }
    tables_kernel<<<(L * M + 255) / 256, 256, 0, ctx->stream>>>(L, f->Ttab.as<bf16>(), f->TT.as<bf16>(),
                                                               f->twL.as<float2>());
    column_tables_kernel<<<(L * 32 + 255) / 256, 256, 0, ctx->stream>>>(L, f->twL.as<float2>(), f->colF.as<uint4>(),
                                                                       f->colI.as<uint4>());
    if (cudaGetLastError() != cudaSuccess || cudaStreamSynchronize(ctx->stream) != cudaSuccess) {
      set_error(ctx, LITHO_ERR_CUDA, "surrogate table setup failed");
      rc = LITHO_ERR_CUDA;
    }
  } while (0);
  if (rc != LITHO_OK) {
    litho_surrogate_destroy(f);
    return rc;
  }
  *out = f;
  return LITHO_OK;
}

void litho_surrogate_destroy(litho_fno* f) {
  if (!f) return;
  DevBuf* bufs[] = {&f->theta, &f->grad, &f->adam_m, &f->adam_v, &f->Ttab, &f->TT, &f->twL, &f->colF, &f->colI, &f->Xf, &f->Gy,
                    &f->gU, &f->gv[0], &f->gv[1], &f->out, &f->lossb, &f->lossp, &f->coef, &f->gpart, &f->Xb, &f->Eres,
                    &f->Enew, &f->Cb, &f->Mrow, &f->Cm, &f->est, &f->stage_m, &f->stage_i};
  for (DevBuf* b : bufs) b->release();
  for (int l = 0; l < NL; ++l) {
    f->z[l].release();
    f->Vs[l].release();
  }
  delete f;
}

int litho_surrogate_get_params(litho_fno* f, float* host, long long n) {
  if (!f || !host) return LITHO_ERR_ARG;
  litho_ctx* ctx = f->ctx;
  LITHO_ARG_CHECK(ctx, n == (long long)Off::N, "expected %lld parameters", (long long)Off::N);
  LITHO_CUDA_TRY(ctx, cudaMemcpyAsync(host, f->theta.p, Off::N * sizeof(float), cudaMemcpyDeviceToHost, ctx->stream));
  LITHO_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
  return LITHO_OK;
}

int litho_surrogate_set_params(litho_fno* f, const float* host, long long n) {
  if (!f || !host) return LITHO_ERR_ARG;
  litho_ctx* ctx = f->ctx;
  LITHO_ARG_CHECK(ctx, n == (long long)Off::N, "expected %lld parameters", (long long)Off::N);
  const size_t pb = Off::N * sizeof(float);
  LITHO_CUDA_TRY(ctx, cudaMemcpyAsync(f->theta.p, host, pb, cudaMemcpyHostToDevice, ctx->stream));
  LITHO_CUDA_TRY(ctx, cudaMemsetAsync(f->adam_m.p, 0, pb, ctx->stream));
  LITHO_CUDA_TRY(ctx, cudaMemsetAsync(f->adam_v.p, 0, pb, ctx->stream));
  LITHO_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
  f->step = 0;
  return LITHO_OK;
}

int litho_surrogate_forward(litho_fno* f, const float* masks, int batch, float* images) {
  if (!f) return LITHO_ERR_ARG;
  litho_ctx* ctx = f->ctx;
  LITHO_ARG_CHECK(ctx, masks && images && batch >= 1, "bad argument");
  LITHO_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  LITHO_RET(ensure_batch(f, batch, false));
  return forward(f, masks, batch, false, images);
}

int litho_surrogate_loss_grad(litho_fno* f, const float* masks, const float* targets, int batch, float* loss,
                              float* grad_host) {
  if (!f || !masks || !targets || batch < 1) return LITHO_ERR_ARG;
  litho_ctx* ctx = f->ctx;
  LITHO_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  LITHO_RET(ensure_batch(f, batch, true));
  LITHO_RET(forward(f, masks, batch, true, f->out.as<float>()));
  LITHO_RET(backward(f, masks, targets, batch));
  if (loss) {
    std::vector<float> lb(batch);
    LITHO_CUDA_TRY(ctx, cudaMemcpyAsync(lb.data(), f->lossb.p, batch * sizeof(float), cudaMemcpyDeviceToHost, ctx->stream));
    LITHO_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
    double s = 0.0;
    for (float v : lb) s += v;
    *loss = (float)(s / batch);
  }
  if (grad_host) {
    LITHO_CUDA_TRY(ctx, cudaMemcpyAsync(grad_host, f->grad.p, Off::N * sizeof(float), cudaMemcpyDeviceToHost, ctx->stream));
    LITHO_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
  }
  return LITHO_OK;
}

int litho_surrogate_train_step(litho_fno* f, const float* masks, const float* targets, int batch, float lr,
                               float weight_decay, float* loss) {
  if (!f || !masks || !targets || batch < 1) return LITHO_ERR_ARG;
  litho_ctx* ctx = f->ctx;
  LITHO_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  LITHO_RET(ensure_batch(f, batch, true));
  LITHO_RET(forward(f, masks, batch, true, f->out.as<float>()));
  LITHO_RET(backward(f, masks, targets, batch));
  f->step += 1;
  const float b1 = 0.9f, b2 = 0.999f;
  const float bc1 = 1.f - (float)std::pow((double)b1, (double)f->step);
  const float bc2 = 1.f - (float)std::pow((double)b2, (double)f->step);
  {
    StageScope sc(ctx, LITHO_STAGE_SURROGATE);
    adam_kernel<<<4 * ctx->sm_count, 256, 0, ctx->stream>>>(Off::N, f->theta.as<float>(), f->grad.as<float>(),
                                                            f->adam_m.as<float>(), f->adam_v.as<float>(), lr, b1, b2,
                                                            1e-8f, weight_decay, bc1, bc2);
  }
  LITHO_CUDA_TRY(ctx, cudaGetLastError());
  if (loss) {
    std::vector<float> lb(batch);
    LITHO_CUDA_TRY(ctx, cudaMemcpyAsync(lb.data(), f->lossb.p, batch * sizeof(float), cudaMemcpyDeviceToHost, ctx->stream));
    LITHO_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
    double s = 0.0;
    for (float v : lb) s += v;
    *loss = (float)(s / batch);
  }
  return LITHO_OK;
}

int litho_rect_masks(litho_ctx* ctx, unsigned long long seed, long long first, int count, int L, int nmin, int nmax,
                     int wmin, int wmax, float* masks) {
  if (ctx == nullptr) return LITHO_ERR_ARG;
  LITHO_ARG_CHECK(ctx, masks && count >= 1 && L >= 1, "bad argument");
  LITHO_ARG_CHECK(ctx, nmin >= 0 && nmax >= nmin && nmax <= 256, "rectangle count range [%d, %d] (max 256)", nmin, nmax);
  LITHO_ARG_CHECK(ctx, wmin >= 1 && wmax >= wmin && wmax <= L, "rectangle side range [%d, %d] for L=%d", wmin, wmax, L);
  LITHO_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  rect_masks_kernel<<<count, 256, 0, ctx->stream>>>((uint64_t)seed, first, L, nmin, nmax, wmin, wmax, masks);
  LITHO_CUDA_TRY(ctx, cudaGetLastError());
  return LITHO_OK;
}

int litho_surrogate_set_alpha(litho_fno* f, float alpha) {
  if (!f) return LITHO_ERR_ARG;
  LITHO_ARG_CHECK(f->ctx, alpha > 0.f && std::isfinite(alpha), "alpha must be positive");
  f->est_alpha = alpha;
  return LITHO_OK;
}

float litho_surrogate_get_alpha(const litho_fno* f) { return f ? f->est_alpha : 0.f; }

int litho_surrogate_project(litho_fno* f, int Nx, int Ny, float* images, int batch, float* est) {
  if (!f) return LITHO_ERR_ARG;
  litho_ctx* ctx = f->ctx;
  const int L = f->L;
  LITHO_ARG_CHECK(ctx, images && est && batch >= 1, "bad argument");
  LITHO_ARG_CHECK(ctx, Nx >= 0 && Ny >= 0 && 2 * Nx <= 15 && 2 * Ny <= 15, "band half-widths Nx=%d Ny=%d unsupported (2 N <= 15)", Nx, Ny);
  LITHO_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  LITHO_RET(project(f, Nx, Ny, images, batch));
  StageScope sc(ctx, LITHO_STAGE_SURROGATE);
  oob_est_kernel<<<(batch + 127) / 128, 128, 0, ctx->stream>>>(L, batch, f->Eres.as<float>(), f->Enew.as<float>(),
                                                               f->est_alpha, est);
  LITHO_CUDA_TRY(ctx, cudaGetLastError());
  return LITHO_OK;
}

int litho_surrogate_predict(litho_fno* f, const litho_kernel_set* ks, const float* masks, int batch, float* images,
                            float* est) {
  if (!f) return LITHO_ERR_ARG;
  litho_ctx* ctx = f->ctx;
  LITHO_ARG_CHECK(ctx, ks && masks && images && est && batch >= 1, "bad argument");
  LITHO_ARG_CHECK(ctx, ks->ctx == ctx, "kernel set belongs to another context");
  LITHO_ARG_CHECK(ctx, 2 * ks->Nx <= 15 && 2 * ks->Ny <= 15 && ks->nk <= 64,
                  "estimator needs 2 Nx, 2 Ny <= 15 and nk <= 64 (Nx=%d Ny=%d nk=%d)", ks->Nx, ks->Ny, ks->nk);
  LITHO_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  return predict(f, ks, masks, batch, images, est);
}

int litho_surrogate_image(litho_fno* f, const litho_kernel_set* ks, const float* masks, int batch, float threshold,
                          float* images, float* est_host, int* used_socs) {
  if (!f) return LITHO_ERR_ARG;
  litho_ctx* ctx = f->ctx;
  const int L = f->L;
  LITHO_ARG_CHECK(ctx, ks && masks && images && batch >= 1, "bad argument");
  LITHO_ARG_CHECK(ctx, ks->ctx == ctx, "kernel set belongs to another context");
  LITHO_ARG_CHECK(ctx, 2 * ks->Nx <= 15 && 2 * ks->Ny <= 15 && ks->nk <= 64,
                  "estimator needs 2 Nx, 2 Ny <= 15 and nk <= 64 (Nx=%d Ny=%d nk=%d)", ks->Nx, ks->Ny, ks->nk);
  LITHO_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  LITHO_RET(f->est.ensure(ctx, (size_t)batch * sizeof(float)));
  LITHO_RET(predict(f, ks, masks, batch, images, f->est.as<float>()));
  std::vector<float> est(batch);
  LITHO_CUDA_TRY(ctx, cudaMemcpyAsync(est.data(), f->est.p, batch * sizeof(float), cudaMemcpyDeviceToHost, ctx->stream));
  LITHO_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
  std::vector<int> rej;
  for (int b = 0; b < batch; ++b) {
    const bool r = !(est[b] <= threshold);  // NaN rejects
    if (r) rej.push_back(b);
    if (used_socs) used_socs[b] = r ? 1 : 0;
    if (est_host) est_host[b] = est[b];
  }
  if (!rej.empty()) {
    const int n = (int)rej.size();
    const size_t img = (size_t)L * L * sizeof(float);
    LITHO_RET(f->stage_m.ensure(ctx, n * img));
    LITHO_RET(f->stage_i.ensure(ctx, n * img));
    for (int i = 0; i < n; ++i)
      LITHO_CUDA_TRY(ctx, cudaMemcpyAsync(f->stage_m.as<char>() + i * img, reinterpret_cast<const char*>(masks) + rej[i] * img,
                                          img, cudaMemcpyDeviceToDevice, ctx->stream));
    const ImgGeom g{L, L, L, L, ks->Nx, ks->Ny, ks->nk, default_conv_n(ks->Nx, ks->Ny)};
    LITHO_RET(image_pipeline(ctx, g, n, f->stage_m.as<float>(), ks, f->stage_i.as<float>(),
                             LITHO_PREC_FP32));
    for (int i = 0; i < n; ++i)
      LITHO_CUDA_TRY(ctx, cudaMemcpyAsync(reinterpret_cast<char*>(images) + rej[i] * img, f->stage_i.as<char>() + i * img,
                                          img, cudaMemcpyDeviceToDevice, ctx->stream));
  }
  return LITHO_OK;
}

}  // extern "C"
