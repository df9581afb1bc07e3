// Launchers: Fourier slice, projection column/row passes (template size h).
#include "match_kernels.cuh"
#include "match_launch.h"

namespace lgb {

// ---------------------------------------------------------------------------
// Fourier-slice extraction with trilinear interpolation.
// Output slices[b][r][kx], r in fft order (the reference's ifftshift of the
// fftshifted slice), DC set to 0, multiplied by -1.
//
// What bounds it: the sectors that a warp's gathers touch.  A warp samples a
// patch of 8 columns x 4 rows: whatever the orientation, its points share
// volume rows, where 32 columns of one row, as before, lie in up to 32 of them.
// 300 slices of 256: 128 -> 118 us; 32 slices of 64 a batch: 10.3 -> 6.6,
// 5.0 with a thread for each FP64 sincos.  Loading the 16 B that hold both x
// neighbours where they are aligned: 130 us for the 300.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256)
    slice_kernel(const float2* __restrict__ vol, int d, const float* __restrict__ euler, int o0,
                 const int* __restrict__ o0_dev, const float* __restrict__ rotations, int tiles,
                 float2* __restrict__ slices) {
  chain_wait();
  LGB_CHAIN_POINTER(vol);
  LGB_CHAIN_POINTER(euler);
  LGB_CHAIN_POINTER(o0_dev);
  LGB_CHAIN_POINTER(rotations);
  LGB_CHAIN_POINTER(slices);
  const int b = blockIdx.y;
  __shared__ float R[9];
  __shared__ SinCos angle[3];
  if (rotations) {
    if (threadIdx.x < 9) R[threadIdx.x] = rotations[9 * (size_t)b + threadIdx.x];
  } else {
    if (threadIdx.x < 3) {
      const int o = o0 + (o0_dev ? *o0_dev : 0) + b;
      angle[threadIdx.x] = sincos_degrees(euler[3 * (size_t)o + threadIdx.x]);
    }
    __syncwarp();
    if (threadIdx.x == 0) rotmat_zyz(angle, R);
  }
  __syncthreads();
  const int wc = d / 2 + 1, half = d / 2;
  const float fd = (float)d;
  // warp -> patch: `tiles` patches cover a strip of four rows
  const int w = blockIdx.x * 8 + threadIdx.x / 32, lane = threadIdx.x & 31;
  const int strip = w / tiles;
  const int r = strip * 4 + lane / 8, kx = (w - strip * tiles) * 8 + lane % 8;
  if (r >= d || kx >= wc) return;
  const float fy = (float)(r < (d + 1) / 2 ? r : r - d) / fd;
  const float fx = (float)kx / fd;
  float X = R[0] * fx + R[1] * fy;
  float Y = R[3] * fx + R[4] * fy;
  float Z = R[6] * fx + R[7] * fy;
  const bool cj = X < 0.f;
  if (cj) { X = -X; Y = -Y; Z = -Z; }
  const float cz = Z * fd + (float)half, cy = Y * fd + (float)half, cx = X * fd;
  float2 val = make_float2(0.f, 0.f);
  if (cz >= 0.f && cz <= (float)(d - 1) && cy >= 0.f && cy <= (float)(d - 1) && cx >= 0.f && cx <= (float)(wc - 1)) {
    const int z0 = (int)floorf(cz), y0 = (int)floorf(cy), x0 = (int)floorf(cx);
    const float tz = cz - (float)z0, ty = cy - (float)y0, tx = cx - (float)x0;
    const int z1 = min(z0 + 1, d - 1), y1 = min(y0 + 1, d - 1), x1 = min(x0 + 1, wc - 1);
    const int zz[2] = {z0, z1}, yy[2] = {y0, y1}, xx[2] = {x0, x1};
    const float wz[2] = {1.f - tz, tz}, wy[2] = {1.f - ty, ty}, wx[2] = {1.f - tx, tx};
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
      for (int bb = 0; bb < 2; ++bb)
#pragma unroll
        for (int cc = 0; cc < 2; ++cc) {
          const float wt = wz[a] * wy[bb] * wx[cc];
          // d <= 512: the volume's elements count in 32 bits
          const float2 s = __ldg(vol + ((unsigned)(zz[a] * d + yy[bb]) * (unsigned)wc + (unsigned)xx[cc]));
          val.x = fmaf(s.x, wt, val.x);
          val.y = fmaf(s.y, wt, val.y);
        }
  }
  if (cj) val.y = -val.y;
  if (r == 0 && kx == 0) val = make_float2(0.f, 0.f);
  slices[((size_t)b * d + r) * wc + kx] = make_float2(-val.x, -val.y);
}


#define LGB_TEMPLATE_SIZES(X) X(16) X(32) X(48) X(64) X(96) X(128) X(192) X(256) X(288) X(384) X(512)

bool supported_template(int h) {
  switch (h) {
#define X(n) case n:
    LGB_TEMPLATE_SIZES(X)
#undef X
    return true;
    default:
      return false;
  }
}

int launch_slice(const void* vol, int d, const float* euler, int o0, const int* o0_dev, int nb,
                 const float* rotations, void* slices, cudaStream_t s) {
  const int tiles = (d / 2 + 1 + 7) / 8, patches = tiles * ((d + 3) / 4);
  dim3 grid((patches + 7) / 8, nb);
  return launch_chained(slice_kernel, grid, dim3(256), 0, s, static_cast<const float2*>(vol), d, euler, o0, o0_dev,
                        rotations, tiles, static_cast<float2*>(slices));
}

constexpr int kProjCols = 8;

// Splits of the template sizes for the two-pass kernels: d = R1 R2 of the column
// pass (R2 = A x B), d / 2 = R1 R2 of the row pass; 0: the generic kernel
// (d / 2 = 96 has no split whose rows are lane aligned).  Against three to
// five passes through shared memory, microseconds for 96 correlograms, columns
// and rows: 64 4.8 + 4.2 -> 3.3 + 4.2, 128 6.9 + 6.9 -> 5.2 + 5.6, 192 12.8 -> 8.3
// (columns), 288 32 + 40 -> 16 + 20, 384 38 + 54 -> 23 + 34, 512 59 + 70 -> 40 + 60;
// for two correlograms 288 7.5 + 7.4 -> 3.9 + 4.6.
template <int HT>
struct ProjSplit {
  static constexpr int COL1 = 0, COL2A = 0, COL2B = 0, ROW1 = 0, ROW2 = 0, ROWS = 8;
};
#define LGB_PROJ_SPLIT(n, c1, c2a, c2b, r1, r2, rows)                                                      \
  template <>                                                                                              \
  struct ProjSplit<n> {                                                                                    \
    static constexpr int COL1 = c1, COL2A = c2a, COL2B = c2b, ROW1 = r1, ROW2 = r2, ROWS = rows;           \
  };
LGB_PROJ_SPLIT(64, 8, 1, 8, 8, 4, 16)
LGB_PROJ_SPLIT(96, 12, 1, 8, 16, 3, 8)
LGB_PROJ_SPLIT(128, 16, 1, 8, 8, 8, 16)
LGB_PROJ_SPLIT(192, 16, 1, 12, 0, 0, 8)
LGB_PROJ_SPLIT(256, 16, 1, 16, 16, 8, 8)
LGB_PROJ_SPLIT(288, 16, 1, 18, 16, 9, 8)
LGB_PROJ_SPLIT(384, 16, 3, 8, 16, 12, 8)
LGB_PROJ_SPLIT(512, 16, 4, 8, 16, 16, 8)
#undef LGB_PROJ_SPLIT

template <int HT>
static int proj_col_t(const void* slices, const float* pf, int nb, int n_cd, int n_c, void* T, cudaStream_t s) {
  constexpr int WC = HT / 2 + 1;
  using PS = ProjSplit<HT>;
  if constexpr (PS::COL1 > 0) {
    using PC = ProjColPair<PS::COL1, PS::COL2A, PS::COL2B>;
    dim3 pgrid((WC + PC::G - 1) / PC::G, n_c);
    return launch_chained(proj_col_pair_kernel<PS::COL1, PS::COL2A, PS::COL2B>, pgrid, dim3(PC::G * PC::NT), 0, s,
                          static_cast<const float2*>(slices), pf, nb, n_cd, static_cast<float2*>(T));
  } else {
    dim3 grid((WC + kProjCols - 1) / kProjCols, n_c);
    return launch_chained(proj_col_kernel<HT, kProjCols>, grid, dim3(kProjCols * FftThreads<HT>::value), 0, s,
                          static_cast<const float2*>(slices), pf, nb, n_cd, static_cast<float2*>(T));
  }
}

template <int HT>
static int proj_row_t(const void* T, int n_c, float* proj, double* rowstats, cudaStream_t s) {
  using PS = ProjSplit<HT>;
  static_assert(HT % PS::ROWS == 0, "rows per CTA must divide the template size");
  dim3 grid(HT / PS::ROWS, n_c);
  if constexpr (PS::ROW1 > 0)
    return launch_chained(proj_row_pair_kernel<PS::ROW1, PS::ROW2, PS::ROWS>, grid, dim3(PS::ROWS * PS::ROW1), 0, s,
                          static_cast<const float2*>(T), proj, rowstats);
  else
    return launch_chained(proj_row_kernel<HT, PS::ROWS>, grid, dim3(PS::ROWS * FftThreads<HT / 2>::value), 0, s,
                          static_cast<const float2*>(T), proj, rowstats);
}

bool supported_proj_row_rfft(int h, int W) { return h == 256 && W == 288; }

int launch_proj_row_rfft(int h, int W, const void* T, int n_c, double* rowstats, int Wcp, void* A, cudaStream_t s) {
  if (!supported_proj_row_rfft(h, W) || Wcp < W / 2 + 1) return LGB_ERR_UNSUPPORTED_SIZE;
  // 8-row groups that share a CTA's roots: up to 8 of 32, as long as two rounds
  // of seven CTAs per SM are left
  constexpr int ROWS = 8;
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  int groups = 8;
  while (groups > 1 && (long long)n_c * (256 / (ROWS * groups)) < 14LL * sms) groups /= 2;
  return launch_chained(proj_row_rfft_kernel<ROWS>, dim3(256 / (ROWS * groups), n_c), dim3(ROWS * 16), 0, s,
                        static_cast<const float2*>(T), rowstats, Wcp, groups, static_cast<float2*>(A));
}

int launch_proj_col(int h, const void* slices, const float* pf, int nb, int n_cd, int n_c, void* T, cudaStream_t s) {
  switch (h) {
#define X(n) \
  case n:    \
    return proj_col_t<n>(slices, pf, nb, n_cd, n_c, T, s);
    LGB_TEMPLATE_SIZES(X)
#undef X
    default:
      return LGB_ERR_UNSUPPORTED_SIZE;
  }
}

int launch_proj_row(int h, const void* T, int n_c, float* proj, double* rowstats, cudaStream_t s) {
  switch (h) {
#define X(n) \
  case n:    \
    return proj_row_t<n>(T, n_c, proj, rowstats, s);
    LGB_TEMPLATE_SIZES(X)
#undef X
    default:
      return LGB_ERR_UNSUPPORTED_SIZE;
  }
}

}  // namespace lgb
