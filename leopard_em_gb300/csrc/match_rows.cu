// Launchers: zero-padded projection rfft and the row c2r + statistics pass
// (image width W).
#include "match_kernels.cuh"
#include "match_launch.h"

namespace lgb {

// Spectrum rows of wc columns -> rows of wcp, zero filled: one warp per row (64-bit
// divisions per element held the flat form to 3.0 TB/s; this 7.4, partly L2, at 86k rows of 145).
__global__ void __launch_bounds__(256)
    repack_rows_kernel(const float2* __restrict__ src, long long rows, int wc, int wcp, float2* __restrict__ dst) {
  const long long row = blockIdx.x * 8LL + threadIdx.x / 32;
  if (row >= rows) return;
  const float2* s = src + row * wc;
  float2* d = dst + row * wcp;
  for (int k = threadIdx.x & 31; k < wcp; k += 256) {  // eight loads in flight
    float2 v[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) v[q] = k + 32 * q < wc ? __ldg(s + k + 32 * q) : make_float2(0.f, 0.f);
#pragma unroll
    for (int q = 0; q < 8; ++q)
      if (k + 32 * q < wcp) d[k + 32 * q] = v[q];
  }
}

int launch_repack_rows(const void* src, long long rows, int wc, int wcp, void* dst, cudaStream_t s) {
  repack_rows_kernel<<<(unsigned)((rows + 7) / 8), 256, 0, s>>>(static_cast<const float2*>(src), rows, wc, wcp,
                                                                static_cast<float2*>(dst));
  return cudaGetLastError() == cudaSuccess ? LGB_OK : LGB_ERR_CUDA;
}

// One warp per correlogram: the normalisation constants (edge mean e, scale
// s) from the h row moments, stored as a float2 over rowstats[c][0][0] (row
// 0's moments are not needed afterwards), so that every pad_rfft or column
// pass CTA reads them instead of reducing all rows again.  offset (or null)
// takes Re(I00 conj(P00)) scale, P00 = s (sum of the projection - e h^2).
// The FP64 pipe bounds it (a warp-wide add holds it for 32 cycles), so the
// warps are CTAs of their own, spread over the SMs: 300 correlograms
// 10.4 us in CTAs of eight warps, 7.3 in one each, 5.6 without the divisions.
__global__ void __launch_bounds__(32)
    norm_constants_kernel(double* __restrict__ rowstats, NormSizes sizes, const float2* __restrict__ dc, size_t dc_stride,
                          float scale, float* __restrict__ offset) {
  chain_wait();
  LGB_CHAIN_POINTER(rowstats);
  LGB_CHAIN_POINTER(dc);
  LGB_CHAIN_POINTER(offset);
  const int c = blockIdx.x, h = sizes.h;
  double* rs = rowstats + (size_t)c * h * 3;
  float e = 0.f, s = 0.f;
  const double sum = projection_norm_constants(rs, sizes, &e, &s);
  __syncwarp();
  if (threadIdx.x == 0) {
    *reinterpret_cast<float2*>(rs) = make_float2(e, s);
    if (offset) {  // (P00's imaginary part is 0: times it, so that an infinite bin still shows)
      const float2 I = dc[c * dc_stride];
      offset[c] = (float)(((double)I.x * ((double)s * (sum - (double)e * h * h)) + (double)I.y * 0.0) * (double)scale);
    }
  }
}

int launch_norm_constants(double* rowstats, int n_c, int h, int norm_h, int norm_w, cudaStream_t s, const float2* dc,
                          size_t dc_stride, float scale, float* offset) {
  return launch_chained(norm_constants_kernel, dim3(n_c), dim3(32), 0, s, rowstats, NormSizes(h, norm_h, norm_w), dc,
                        dc_stride, scale, offset);
}


// W/2 of the short rows, which the generic row pass takes
#define LGB_ROW_GENERIC_SIZES(X) X(24) X(32) X(40) X(64) X(128) X(144) X(288)

// W/2 values
#define LGB_ROW_SIZES(X) \
  X(24) X(32) X(40) X(64) X(128) X(144) X(256) X(288) X(512) X(1024) X(1440) X(1536) X(1920) X(2048) X(2880)

bool supported_row(int W) {
  if (W % 2) return false;
  switch (W / 2) {
#define X(n) case n:
    LGB_ROW_SIZES(X)
#undef X
    return true;
    default:
      return false;
  }
}

template <int WH>
static int pad_rfft_t(const float* proj, const double* rowstats, int h, int norm_h, int norm_w, int Wcp, int n_c,
                      void* A, cudaStream_t s, bool norm_ready) {
  constexpr int NT = FftThreads<WH>::value;
  // at least one full warp: the normalisation reduction shuffles across warp 0
  constexpr int ROWS0 = NT >= 128 ? 2 : (NT >= 32 ? 4 : (NT >= 16 ? 8 : 16));
  constexpr int ROWS1 = ROWS0 * NT >= 32 ? ROWS0 : (32 + NT - 1) / NT;
  // static shared memory (ROWS rows of the padded transform) stays under 40 KB
  constexpr int ROWS = ROWS1 * (IdxPad16::pad(WH) + 2) * 8 <= 40960 ? ROWS1 : 1;
  static_assert(ROWS * NT >= 32, "pad_rfft CTA must hold a full warp");
  const int ctas = (h + ROWS - 1) / ROWS;
  // precompute the constants when many CTAs share a correlogram (each would
  // otherwise reduce all h rows in FP64); a few CTAs do it themselves
  const int ready = norm_ready || ctas >= 16;
  if (ready && !norm_ready) {
    const int st = launch_norm_constants(const_cast<double*>(rowstats), n_c, h, norm_h, norm_w, s);
    if (st) return st;
  }
  dim3 grid(ctas, n_c);
  return launch_chained(pad_rfft_kernel<WH, ROWS>, grid, dim3(ROWS * NT), 0, s, proj, rowstats, h,
                        NormSizes(h, norm_h, norm_w), Wcp, ready, static_cast<float2*>(A));
}

template <int WH>
static int rowpass_t(const void* Y, int H, int y_rows, int Wcp, int n_c, int nb, int n_orient, int o0,
                     const int* o0_dev, float* mip, int* best, double* s1, double* s2, cudaStream_t s) {
  constexpr int NT = row_threads(WH);
  constexpr size_t SMEM = RowGeneric<WH>::SMEM;
  if (cudaFuncSetAttribute(rowpass_kernel<WH, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM) !=
      cudaSuccess)
    return LGB_ERR_CUDA;
  const float scale = 1.0f / ((float)H * (float)(2 * WH));
  return launch_chained(rowpass_kernel<WH, NT>, dim3(y_rows), dim3(NT), SMEM, s, static_cast<const float2*>(Y), y_rows,
                        Wcp, n_c, nb, n_orient, o0, o0_dev, scale, mip, best, s1, s2);
}

int launch_pad_rfft(int W, const float* proj, const double* rowstats, int h, int norm_h, int norm_w, int Wcp,
                    int n_c, void* A, cudaStream_t s, bool norm_ready) {
  if (W % 2 || norm_w > W || norm_w < h || norm_h < h) return LGB_ERR_UNSUPPORTED_SIZE;
  if (!supported_row(W)) return LGB_ERR_UNSUPPORTED_SIZE;
  if (h % 2) return LGB_ERR_UNSUPPORTED_SIZE;
  switch (W / 2) {
#define X(n)  \
  case n / 2: \
    return launch_pad_rfft_##n(proj, rowstats, h, norm_h, norm_w, Wcp, n_c, A, s, norm_ready);
    LGB_PAD_REG_SIZES(X)
#undef X
#define X(n) \
  case n:    \
    return pad_rfft_t<n>(proj, rowstats, h, norm_h, norm_w, Wcp, n_c, A, s, norm_ready);
    LGB_ROW_GENERIC_SIZES(X)
#undef X
    default:
      return LGB_ERR_UNSUPPORTED_SIZE;
  }
}

int launch_rowpass(int W, const void* Y, int H, int y_rows, int Wcp, int n_c, int nb, int n_orient, int o0,
                   const int* o0_dev, float* mip, int* best, double* s1, double* s2, cudaStream_t s) {
  if (W % 2 || y_rows < 1 || y_rows > H) return LGB_ERR_INVALID_ARGUMENT;
  switch (W / 2) {
#define X(n)        \
  case n / 2:       \
    return launch_rowpass_##n(Y, H, y_rows, Wcp, n_c, nb, n_orient, o0, o0_dev, mip, best, s1, s2, s);
    LGB_ROW_HALF_SIZES(X)
#undef X
#define X(n) \
  case n:    \
    return rowpass_t<n>(Y, H, y_rows, Wcp, n_c, nb, n_orient, o0, o0_dev, mip, best, s1, s2, s);
    LGB_ROW_GENERIC_SIZES(X)
#undef X
    default:
      return LGB_ERR_UNSUPPORTED_SIZE;
  }
}

}  // namespace lgb
