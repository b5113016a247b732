// Internal declarations shared by the liblitho_gb300 translation units.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <cstdarg>
#include <cstdio>
#include <string>
#include <map>
#include <memory>
#include <tuple>
#include <vector>

#include "../../include/litho_gb300.h"
#include "win_tiles.hpp"

namespace litho {

// ---------------------------------------------------------------------------
// error plumbing
// ---------------------------------------------------------------------------
struct Status {
  int code = LITHO_OK;
  std::string msg;
};

void set_error(litho_ctx* ctx, int code, const char* fmt, ...);

#define LITHO_CUDA_TRY(ctx, call)                                                       \
  do {                                                                                  \
    cudaError_t e_ = (call);                                                            \
    if (e_ != cudaSuccess) {                                                            \
      ::litho::set_error((ctx), LITHO_ERR_CUDA, "%s failed: %s (%s:%d)", #call,          \
                         cudaGetErrorString(e_), __FILE__, __LINE__);                   \
      return LITHO_ERR_CUDA;                                                            \
    }                                                                                   \
  } while (0)

#define LITHO_ARG_CHECK(ctx, cond, ...)                                                 \
  do {                                                                                  \
    if (!(cond)) {                                                                      \
      ::litho::set_error((ctx), LITHO_ERR_ARG, __VA_ARGS__);                            \
      return LITHO_ERR_ARG;                                                             \
    }                                                                                   \
  } while (0)

#define LITHO_RET(expr)             \
  do {                              \
    int r_ = (expr);                \
    if (r_ != LITHO_OK) return r_;  \
  } while (0)

// ---------------------------------------------------------------------------
// grow-only device buffer owned by a context
// ---------------------------------------------------------------------------
struct DevBuf {
  void* p = nullptr;
  size_t bytes = 0;
  int ensure(litho_ctx* ctx, size_t need);
  void release();
  template <class T> T* as() const { return static_cast<T*>(p); }
};

// Sum of n float2 values p[0], p[stride], ... (partials written by an earlier
// kernel): eight independent loads in flight and a fixed summation order.
__device__ __forceinline__ float2 sum_strided(const float2* __restrict__ p, size_t stride, int n) {
  float2 a[8];
#pragma unroll
  for (int u = 0; u < 8; ++u) a[u] = make_float2(0.f, 0.f);
  int i = 0;
  for (; i + 8 <= n; i += 8) {
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const float2 t = __ldg(p + (size_t)(i + u) * stride);
      a[u].x += t.x;
      a[u].y += t.y;
    }
  }
#pragma unroll
  for (int u = 0; u < 7; ++u)
    if (i + u < n) {
      const float2 t = __ldg(p + (size_t)(i + u) * stride);
      a[u].x += t.x;
      a[u].y += t.y;
    }
  return make_float2(((a[0].x + a[1].x) + (a[2].x + a[3].x)) + ((a[4].x + a[5].x) + (a[6].x + a[7].x)),
                     ((a[0].y + a[1].y) + (a[2].y + a[3].y)) + ((a[4].y + a[5].y) + (a[6].y + a[7].y)));
}

// cos and sin of 2 pi m / F (F a power of two) for an exact integer m, rounded once
__device__ __forceinline__ void cis_round(long long m, int F, float* c, float* s) {
  double sd, cd;
  sincospi(2.0 * (double)(m & (long long)(F - 1)) / (double)F, &sd, &cd);
  *c = (float)cd;
  *s = (float)sd;
}

// Autotuned shape of the split-BF16 TCC GEMM for one (n, Kp): column tile width, K
// slice, schedule (gemm_schedule's sched) and every candidate's measured time.
struct TccTune {
  struct Cand {
    int bn, bk, sched;
    float ms;
  };
  int bn = 128, bk = 64, sched = 0;
  std::vector<Cand> cands;
};

inline int next_pow2(int x) {
  int p = 1;
  while (p < x) p <<= 1;
  return p;
}
inline bool is_pow2(int x) { return x > 0 && (x & (x - 1)) == 0; }

}  // namespace litho

// The context.  One stream, a set of grow-only workspaces and cached tables.
// device staging slots each way of the host-buffer imaging pipeline (6 measured
// no faster: chunked copies, not slot reuse, bound the pipeline)
constexpr int HB_SLOTS = 3;

struct litho_ctx {
  int device = 0;
  int sm_count = 0;
  cudaStream_t own_stream = nullptr;
  cudaStream_t stream = nullptr;
  std::string last_error;
  // imaging workspaces
  litho::DevBuf win_part, band_part, tm, stage_in, stage_out, stage_k, stage_s, stage_x, band_w;
  // how the SOCS band is formed for kernel sets that carry a TCC band table
  // (litho_ctx_set_band_method): LITHO_BAND_AUTO / _FFT / _TCC
  int band_method = 0;
  // mask bytes per chunk of the host-buffer path (litho_ctx_set_host_chunk); 0: default
  size_t host_chunk_bytes = 0;
  // twiddle and coefficient tables keyed by (L, F, N, kind)
  std::map<std::tuple<int, int, int, int>, litho::DevBuf> twx_tables;
  // TCC / eigensolver workspaces
  litho::DevBuf socs_tmp, tcc_a, tcc_b, tcc_c, tcc_pq, tcc_part, eig_w, eig_v, eig_work, eig_info;
  // mixed-precision (tensor-core) workspaces
  litho::DevBuf mx_b, mx_c, mx_d;
  // host-buffer batches: copy streams and per-slot events of the staging pipeline
  cudaStream_t copy_in = nullptr, copy_out = nullptr;
  cudaEvent_t ev_in[HB_SLOTS] = {}, ev_comp[HB_SLOTS] = {}, ev_out[HB_SLOTS] = {}, ev_start = nullptr;
  // per-stage timers
  bool timing = false;
  double stage_ms[LITHO_STAGE_COUNT] = {};
  long long stage_launches[LITHO_STAGE_COUNT] = {};
  struct Pending { int stage; cudaEvent_t a, b; };
  std::vector<Pending> pending;
  std::vector<cudaEvent_t> event_pool;
  // split-BF16 TCC GEMM: tuned shape per (n, Kp) and device schedule tables per
  // (n, K slices, BN, split)
  std::map<std::pair<int, int>, litho::TccTune> tcc_tune;
  std::map<std::tuple<int, int, int, int>, std::shared_ptr<void>> gemm_tables;
  int tcc_force_bn = 0, tcc_force_bk = 64, tcc_force_sched = 0;  // litho_tcc_gemm_shape: bn > 0 bypasses the tuner
  // error-path test hook (litho_ctx_set_test_stall): >= 0 stops the copies of a mixed call's
  // window DFT after that many steps of every warp (folded) or CTA (tensor cores); -1 = off
  int test_stall_chunk = -1;
};

struct litho_kernel_set {
  litho_ctx* ctx = nullptr;
  int nk = 0, Nx = 0, Ny = 0;
  float2* krn = nullptr;    // [nk][(2Ny+1)(2Nx+1)]
  float* scales = nullptr;  // [nk]
  // rank-K TCC over the window, T(p, q) = sum_k s_k K_k(p) conj(K_k(q)), laid out for
  // band_tcc_kernel in band_nc row chunks (band_tcc.cu); band_nc == 0: none
  float2* band_tab = nullptr;
  int band_nc = 0;
};

namespace litho {

// Brackets one stage's launches with CUDA events when timing is on and counts
// its kernel launches always.
struct StageScope {
  litho_ctx* ctx;
  int stage;
  cudaEvent_t b = nullptr;
  StageScope(litho_ctx* c, int s, int launches = 1);
  ~StageScope();
};

// ---------------------------------------------------------------------------
// imaging pipeline (imaging.cu)
// ---------------------------------------------------------------------------
struct ImgGeom {
  int Lx, Ly;   // physical size (image and mask)
  int Fx, Fy;   // padded FFT size (power of two >= L)
  int Nx, Ny;   // kernel half-support
  int nk;
  int convN;    // SOCS conv grid (power of two >= 4*max(N)+1)
};

// Launch plan for one batch of one size class.
struct ImgPlan {
  ImgGeom g;
  int batch = 1;
  int rowBlocks = 1, colSplits = 1;  // window DFT: column blocks, row splits -> nparts
  int kpg = 1, ngroups = 1;          // SOCS kernels per CTA -> ngroups
  int sms = 0;                       // SMs of the device (launch sizing)
  bool early = false;                // each stage's CTAs start while the stage before it runs (launch_early)
  int nparts() const { return rowBlocks * colSplits; }
};

// Programmatic dependent launch.  A kernel launched `early` may start once every CTA of the one before
// it on the stream has called early_next (or ended); what that one writes is there after early_wait,
// which comes before a kernel's first write and its first read of anything the launches of its call
// write.  early_wait hands back the pointers read from then on, so that no read moves before it.  Both
// are nothing in a launch without it.
__device__ __forceinline__ void early_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
template <typename T>
__device__ __forceinline__ void early_wait(const T* __restrict__& p) {
  unsigned long long v = reinterpret_cast<unsigned long long>(p);
  asm volatile("griddepcontrol.wait;" : "+l"(v)::"memory");
  p = reinterpret_cast<const T*>(v);
}
template <typename... P, typename... A>
cudaError_t launch_early(bool early, void (*k)(P...), dim3 grid, int threads, size_t smem, cudaStream_t s, A... args) {
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = &at;
  cfg.numAttrs = early ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, k, P(args)...);
}

// Lets a kernel ask for all the dynamic shared memory there is beside its own `fixed` bytes of static.
// The limit is an attribute of the kernel, which every thread of the process shares: set to what one
// launch needs, it would refuse the larger launch that another thread has between its own setting and
// its launch.
constexpr int SMEM_MOST = 227 * 1024;
template <typename... P>
cudaError_t allow_smem(void (*k)(P...), int fixed = 0) {
  return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_MOST - fixed);
}

ImgPlan make_plan(const ImgGeom& g, int batch, int sm_count);

// SOCS conv grid used by the imaging entry points: pow2 >= 4 max(Nx, Ny) + 1, at least 32.
int default_conv_n(int Nx, int Ny);

int calc_tcc_impl(litho_ctx* ctx, const float* src, int srcSize, float outerSigma, float wavelength, float NA,
                  float defocus, int Lx, int Ly, int Nx, int Ny, double* tcc, int tccPrecision, int mem, int sh_in,
                  int oSgm_in, float n_medium = 1.0f);

// Host input -> device staging buffer (device input passes through).
int stage_in(litho_ctx* ctx, DevBuf& buf, const void* src, size_t bytes, int mem, const void** dev);

// Window source for the SOCS stage.
struct WindowSrc {
  const float2* part = nullptr;  // [batch][nparts][2Ny+1][Nx+1] partial sums (fused path)
  int nparts = 0;
  const float* mskf_r = nullptr;  // or full spectrum planes [batch][Fy][Fx]
  const float* mskf_i = nullptr;
  int Fx = 0, Fy = 0;             // the planes' size: 0 the image's, or the window's own
};

// the folded FP32 transforms (imaging_fold.cu): plan fields of a plain window DFT, coefficient
// tables and launches
void win_fold_plan(ImgPlan& p, int sm_count);
int win_fold_splits(const ImgGeom& g, int ncb, long long tiles, int sm_count);
size_t win_fold_coef_floats(const ImgGeom& g);
cudaError_t win_fold_coefs(cudaStream_t s, const ImgGeom& g, float* coef);
// masks of one size for a window launch over several sizes (at most WIN_MAX_SIZES, win_tiles.hpp):
// its plan, its masks and its first image in the shared partial array
struct WinPart {
  ImgPlan plan;
  const float* masks;
  int img0;
};
cudaError_t launch_win_fold(cudaStream_t s, const WinPart* parts, int n, const float* const* coef,
                            const float2* const* twF, float2* win_part, int nparts, int stall, int* err,
                            const int* form);
size_t fi_fold_coef_floats(const ImgGeom& g);
cudaError_t fi_fold_coefs(cudaStream_t s, const ImgGeom& g, float* coef);
cudaError_t launch_fi_fold(cudaStream_t s, const ImgPlan& p, const float* tm, const float* coef, float* images);

// window DFT of up to WIN_MAX_SIZES mask sizes, nparts partials per image; precision: whether the
// error-path test hook acts; form: nullptr, or what run_win_dft_tc wrote just before
int run_win_dft(litho_ctx* ctx, const WinPart* parts, int n, float2* win_part, int nparts, int precision, const int* form);
int run_socs(litho_ctx* ctx, const ImgPlan& p, const WindowSrc& w, const float2* krn,
             const float* scales, float2* band_part, float* tmpImgp);
int run_tmp_join(litho_ctx* ctx, const float* part, int ngroups, int n, float* tmpImgp);
int run_fi(litho_ctx* ctx, const ImgPlan& p, const float2* band_part, float* tm, float* images);
// FI step 1 for both layouts (tmh == nullptr: plain tm; else K-major hi/lo + t0)
cudaError_t launch_fi_rows(cudaStream_t s, const ImgPlan& p, const float2* band_part, const float2* twF, int KP,
                           float* tm, float* tmh, float* tml, float* t0);
int fi_twiddles(litho_ctx* ctx, const ImgGeom& g, const float2** out);
int run_fft_mask(litho_ctx* ctx, const float* mask, int Lx, int Ly, float* mskf_r, float* mskf_i);
int upload_kernels(litho_ctx* ctx, const float* krn_r, const float* krn_i, const float* scales,
                   int nk, int kdim, int mem, float2* krn_dev, float* scales_dev);

// Full imaging pipeline on device pointers for one size class (window DFT ->
// SOCS -> FI), FP32 or mixed precision.
int image_pipeline(litho_ctx* ctx, const ImgGeom& g, int batch, const float* masks,
                   const litho_kernel_set* ks, float* images, int precision);

// the SOCS band as the bilinear form of the kernel set's rank-K TCC (band_tcc.cu)
int build_band_table(litho_ctx* ctx, litho_kernel_set* ks, cudaStream_t stream);
size_t band_wsum_bytes(const ImgGeom& g, int batch);
int run_band_tcc(litho_ctx* ctx, const ImgPlan& p, const WindowSrc& w, const litho_kernel_set* ks,
                 float2* wsum, float2* band_part);
// whether the TCC band may serve a kernel set under the context's band method
inline bool band_tcc_available(const litho_ctx* ctx, const litho_kernel_set* ks) {
  return ks->band_nc > 0 && ctx->band_method != LITHO_BAND_FFT;
}
// whether a batch of images takes the TCC band: LITHO_BAND_TCC wherever the table exists,
// LITHO_BAND_AUTO where the band cost model (band_sched.hpp) expects it to be faster
bool use_band_tcc(const litho_ctx* ctx, const litho_kernel_set* ks, int batch);

// mixed precision interpolation (imaging_tc.cu): whether it serves a geometry of the mixed form
// (elsewhere the folded FP32 kernel does), and its launches
bool fi_tc_serves(const ImgGeom& g);
bool win_tc_serves(const ImgGeom& g, int batch);
void win_tc_plan(ImgPlan& p);
int run_win_dft_tc(litho_ctx* ctx, const WinPart* parts, int n, float2* win_part, int nparts, int* form);
int run_fi_tc(litho_ctx* ctx, const ImgPlan& p, const float2* band_part, float* tmT, float* images);
struct FiTcBufs {
  float *tmh, *tml, *t0;
};
FiTcBufs fi_tc_bufs(float* base, const ImgGeom& g, int total, int first);
int run_fi_rows_tc(litho_ctx* ctx, const ImgPlan& p, const float2* band_part, const FiTcBufs& b);
int run_fi_out_tc(litho_ctx* ctx, const ImgPlan& p, const FiTcBufs& b, float* images);
size_t fi_tc_workspace_bytes(const ImgGeom& g, int batch);
int tc_check_flag(litho_ctx* ctx);
int tc_err_flag_public(litho_ctx* ctx, int** flag);  // the flag of the kernels' bounded waits, made on first use

}  // namespace litho
