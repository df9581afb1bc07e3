// Kernels of the plain FP32 whole-orientation search.
//
// Per orientation batch (B orientations, C*D projective filters, n_c = C*D*B
// correlograms, c = (cs*D + df)*B + b):
//   slice_kernel      Fourier slice of the template at R(phi,theta,psi),
//                     rows un-shifted, DC zeroed, contrast flipped
//                     (cross_correlation.py:76-92)                     [B, d, d/2+1]
//   proj_col_kernel   x projective filter, inverse FFT along y          [n_c, d, d/2+1]
//   proj_row_kernel   c2r along x, 1/d^2, ifftshift, per-row moments    [n_c, d, d]
//   pad_rfft_kernel   edge-mean/variance normalisation (utils.py:106-188)
//                     and the zero-padded row rfft of length W          [n_c, d, Wcp]
//   column pass       per column: pruned FFT along y (length H), cross power
//                     image * conj(P) with P[0,0]=0, inverse FFT along y
//                     (colpass_reg_kernel and, for short columns,
//                     colpass_fused / _tab / _pair_kernel)             [n_c, H, Wcp]
//   row pass          per row: c2r of length W (1/(H W)) and the fused
//                     (rowpass_half_kernel, short rows rowpass_kernel)
//                     statistics update (utils.py:191-255): max over the
//                     batch, strict '>' MIP update, global index, FP64 sums
// Templates from 64 run their projection passes in two register passes
// (proj_col_pair_kernel, proj_row_pair_kernel).  Refinement crops (288^2, d = 256)
// take proj_row_rfft_kernel instead of the row pass and pad_rfft: the row c2r
// 16 x 8 and the padded rfft 9 x 16 in one kernel; the normalisation moves to
// the column pass (colpass_pair_kernel in match_fused.cuh).
#pragma once

#include "chain.cuh"
#include "fft.cuh"
#include "reg_dft.cuh"

namespace lgb {

constexpr int kColGroup = 4;  // columns per colpass CTA: 4 x 8 B = one 32 B sector per row

__host__ __device__ inline int pad4(int n) { return (n + 3) & ~3; }

// ---------------------------------------------------------------------------
// Sines and cosines of ZYZ Euler angles, FP64 -> R = Rz(phi) Ry(theta) Rz(psi).
// (FP64 sincos is a chain of a microsecond: callers give each angle a thread.)
// ---------------------------------------------------------------------------
struct SinCos {
  double s, c;
};
__device__ inline SinCos sincos_degrees(float a) {
  SinCos v;
  sincos((double)a * (3.14159265358979323846 / 180.0), &v.s, &v.c);
  return v;
}
template <class T>
__device__ inline void rotmat_zyz(const SinCos* e, T* R) {
  const double sp = e[0].s, cp = e[0].c, st = e[1].s, ct = e[1].c, ss = e[2].s, cs = e[2].c;
  R[0] = (T)(cp * ct * cs - sp * ss);
  R[1] = (T)(-cp * ct * ss - sp * cs);
  R[2] = (T)(cp * st);
  R[3] = (T)(sp * ct * cs + cp * ss);
  R[4] = (T)(-sp * ct * ss + cp * cs);
  R[5] = (T)(sp * st);
  R[6] = (T)(-st * cs);
  R[7] = (T)(st * ss);
  R[8] = (T)ct;
}

// ---------------------------------------------------------------------------
// proj_col: T[c][y][kx] = IFFT_y( slice_b[y][kx] * pf[cd][y][kx] )   (unscaled)
// ---------------------------------------------------------------------------
template <int HT, int COLS>
__global__ void __launch_bounds__(COLS* FftThreads<HT>::value)
    proj_col_kernel(const float2* __restrict__ slices, const float* __restrict__ pf, int nb, int n_cd,
                    float2* __restrict__ T) {
  constexpr int NT = FftThreads<HT>::value;
  constexpr int WC = HT / 2 + 1;
  constexpr int STRIDE = IdxPad16::pad(HT) + 2;
  __shared__ float2 buf[COLS * STRIDE];
  chain_wait();
  LGB_CHAIN_POINTER(slices);
  LGB_CHAIN_POINTER(pf);
  LGB_CHAIN_POINTER(T);
  // c = (p*n_cd + cd)*nb + b: slices are per (p, b), filters per (p, cd)
  const int c = blockIdx.y;
  const int pc = c / nb, b = c - (c / nb) * nb;
  const int p = pc / n_cd;
  const float2* sl = slices + ((size_t)p * nb + b) * HT * WC;
  const float* f = pf + (size_t)pc * HT * WC;
  const int kx0 = blockIdx.x * COLS;
  for (int e = threadIdx.x; e < HT * COLS; e += blockDim.x) {
    const int y = e / COLS, i = e % COLS, kx = kx0 + i;
    float2 v = make_float2(0.f, 0.f);
    if (kx < WC) {
      v = sl[y * WC + kx];
      const float w = f[y * WC + kx];
      v.x *= w;
      v.y *= w;
    }
    buf[i * STRIDE + IdxPad16::f(y)] = v;
  }
  __syncthreads();
  const int g = threadIdx.x / NT, t = threadIdx.x - (threadIdx.x / NT) * NT;
  block_fft<HT, NT, +1, IdxPad16>(buf + g * STRIDE, t);
  float2* out = T + (size_t)c * HT * WC;
  for (int e = threadIdx.x; e < HT * COLS; e += blockDim.x) {
    const int y = e / COLS, i = e % COLS, kx = kx0 + i;
    if (kx < WC) out[y * WC + kx] = buf[i * STRIDE + IdxPad16::f(y)];
  }
}

// proj_col for HT = R1*R2 (ProjSplit, match_proj.cu) in two register passes: radix R1
// over rows t + R2*q of slice x filter straight from global memory ->
// shared transpose M1[t][q] (odd stride R1+1; column stride 2 mod 16) ->
// radix R2 with twiddles w^(r*t), w = exp(+2 pi i / HT) -> rows t + R1*r of T.
// G columns per CTA (lane bits 0-2), one thread per butterfly.
// R2 = R2A R2B: above 18 points a composite transform in registers.
template <int R1, int R2A, int R2B>
struct ProjColPair {
  static constexpr int R2 = R2A * R2B, HT = R1 * R2;
  static constexpr int NT = R1 > R2 ? R1 : R2;
  static constexpr int G = 8;
  static constexpr int S1 = R1 + 1;
  static constexpr int CB = R2 * S1;
  static constexpr int STRIDE = CB + (18 - CB % 16) % 16;  // = 2 (mod 16)
  static constexpr int NROOT = (R1 - 1) * (R2 - 1) + 1;
};

template <int R1, int R2A, int R2B>
__global__ void __launch_bounds__(ProjColPair<R1, R2A, R2B>::G* ProjColPair<R1, R2A, R2B>::NT)
    proj_col_pair_kernel(const float2* __restrict__ slices, const float* __restrict__ pf, int nb, int n_cd,
                         float2* __restrict__ T) {
  using PC = ProjColPair<R1, R2A, R2B>;
  constexpr int R2 = PC::R2, HT = PC::HT, WC = HT / 2 + 1, G = PC::G, S1 = PC::S1;
  __shared__ float2 buf[G * PC::STRIDE];
  __shared__ float2 root[PC::NROOT];  // exp(+2 pi i m / HT)
  for (int m = threadIdx.x; m < PC::NROOT; m += blockDim.x) {
    float sn, cs;
    sincospif(2.0f * (float)m / (float)HT, &sn, &cs);
    root[m] = make_float2(cs, sn);
  }
  chain_wait();
  LGB_CHAIN_POINTER(slices);
  LGB_CHAIN_POINTER(pf);
  LGB_CHAIN_POINTER(T);
  // c = (p*n_cd + cd)*nb + b: slices are per (p, b), filters per (p, cd)
  const int c = blockIdx.y;
  const int pc = c / nb, b = c - (c / nb) * nb;
  const int p = pc / n_cd;
  const float2* sl = slices + ((size_t)p * nb + b) * HT * WC;
  const float* f = pf + (size_t)pc * HT * WC;
  const int g = threadIdx.x % G, t = threadIdx.x / G;
  const int kx = blockIdx.x * G + g;
  const bool col_ok = kx < WC;
  float2* x = buf + g * PC::STRIDE;
  if (t < R2) {
    float2 v[R1];
#pragma unroll
    for (int q = 0; q < R1; ++q) {
      const int y = t + q * R2;
      v[q] = make_float2(0.f, 0.f);
      if (col_ok) {
        const float2 s = __ldg(sl + (size_t)y * WC + kx);
        const float w = __ldg(f + (size_t)y * WC + kx);
        v[q] = make_float2(s.x * w, s.y * w);
      }
    }
    Dft<R1, +1>::run(v);
#pragma unroll
    for (int q = 0; q < R1; ++q) x[t * S1 + q] = v[q];
  }
  __syncthreads();
  if (t < R1) {
    float2 w[R2];
#pragma unroll
    for (int r = 0; r < R2; ++r) w[r] = cmul(x[r * S1 + t], root[r * t]);
    if constexpr (R2A == 1)
      Dft<R2, +1>::run(w);
    else
      DftNT<R2A, R2B, +1>::run(w);
    if (col_ok) {
      float2* out = T + (size_t)c * HT * WC + (size_t)t * WC + kx;
#pragma unroll
      for (int s = 0; s < R2; ++s) out[(size_t)(R2A == 1 ? s : DftNT<R2A, R2B, +1>::out(s)) * R1 * WC] = w[s];
    }
  }
}

// ---------------------------------------------------------------------------
// proj_row: c2r along x of each row of T[c] (length HT via an HT/2 complex
// inverse FFT), scale 1/HT^2, ifftshift both axes, and per-row moments
// rowstats[c][py] = (sum, sum of squares, edge sum) in FP64.
// Imaginary parts of the DC and Nyquist bins are ignored (c2r convention).
// ---------------------------------------------------------------------------
template <int HT, int ROWS>
__global__ void __launch_bounds__(ROWS* FftThreads<HT / 2>::value)
    proj_row_kernel(const float2* __restrict__ T, float* __restrict__ proj, double* __restrict__ rowstats) {
  constexpr int M = HT / 2;
  constexpr int WC = HT / 2 + 1;
  constexpr int NT = FftThreads<M>::value;
  constexpr int ZS = IdxPad16::pad(M) + 2;
  __shared__ float2 xin[ROWS][WC];
  __shared__ float2 z[ROWS][ZS];
  __shared__ float part[ROWS * NT][3];
  chain_wait();
  LGB_CHAIN_POINTER(T);
  LGB_CHAIN_POINTER(proj);
  LGB_CHAIN_POINTER(rowstats);
  const int c = blockIdx.y;
  const int g = threadIdx.x / NT, t = threadIdx.x - (threadIdx.x / NT) * NT;
  const int row0 = blockIdx.x * ROWS;
  const float2* src = T + ((size_t)c * HT + row0) * WC;
  for (int e = threadIdx.x; e < ROWS * WC; e += blockDim.x) xin[e / WC][e % WC] = src[e];
  __syncthreads();
  for (int k = t; k < M; k += NT) {
    float2 A = xin[g][k];
    float2 B = xin[g][M - k];
    if (k == 0) { A.y = 0.f; B.y = 0.f; }  // DC and Nyquist: real parts only
    B.y = -B.y;                            // conj
    const float2 xe = cadd(A, B);
    float s, co;
    sincospif(2.0f * (float)k / (float)HT, &s, &co);
    const float2 xo = cmul(csub(A, B), make_float2(co, s));
    z[g][IdxPad16::f(k)] = cadd(xe, mul_i<1>(xo));
  }
  __syncthreads();
  block_fft<M, NT, +1, IdxPad16>(z[g], t);
  const int y = row0 + g;
  const int py = (y + HT - HT / 2) % HT;
  const float scale = 1.0f / ((float)HT * (float)HT);
  const bool edge_row = (py == 0) || (py == HT - 1);
  // partial moments in FP32, per thread and then across the row's threads;
  // FP64 only for the stored row moments (FP64 arithmetic, conversions
  // included, runs at about one operation per SM per clock on this GPU); the
  // cross-row reduction is FP64
  float s1 = 0.f, s2 = 0.f, se = 0.f;
  float* prow = proj + ((size_t)c * HT + py) * HT;
  for (int m = t; m < M; m += NT) {
    const float2 v = z[g][IdxPad16::f(m)];
    const float a = v.x * scale, b = v.y * scale;
    const int px0 = (2 * m + HT - HT / 2) % HT, px1 = (2 * m + 1 + HT - HT / 2) % HT;
    prow[px0] = a;
    prow[px1] = b;
    s1 += a + b;
    s2 = fmaf(a, a, fmaf(b, b, s2));
    if (edge_row) {
      se += a + b;
    } else {
      if (px0 == 0 || px0 == HT - 1) se += a;
      if (px1 == 0 || px1 == HT - 1) se += b;
    }
  }
  part[threadIdx.x][0] = s1;
  part[threadIdx.x][1] = s2;
  part[threadIdx.x][2] = se;
  __syncthreads();
  if (t == 0) {
    float a = 0.f, b = 0.f, e = 0.f;
    for (int i = 0; i < NT; ++i) {
      a += part[g * NT + i][0];
      b += part[g * NT + i][1];
      e += part[g * NT + i][2];
    }
    double* rs = rowstats + ((size_t)c * HT + py) * 3;
    rs[0] = (double)a;
    rs[1] = (double)b;
    rs[2] = (double)e;
  }
}

// proj_row for HT/2 = R1*R2 (ProjSplit) in two register passes: the c2r
// pre-twiddle is applied while loading the radix-R1 inputs k = t + R2*q from
// the staged row; shared transpose M1[t][q]; radix R2 with twiddles w^(r*t)
// leaves pixel pairs m = t + R1*r in thread t.  Same outputs, ifftshift and
// moments as proj_row_kernel; R1 threads per row, ROWS rows per CTA.
template <int R1, int R2, int ROWS>
struct ProjRowPair {
  static constexpr int M = R1 * R2;
  static constexpr int NT = R1;
  static constexpr int S1 = R1 + 1;
  static constexpr int ZR = R2 * S1 + 1;
  static constexpr int NROOT = (R1 - 1) * (R2 - 1) + 1;
  static_assert(R1 >= R2, "second pass uses every thread of the row");
};

template <int R1, int R2, int ROWS>
__global__ void __launch_bounds__(ROWS* R1)
    proj_row_pair_kernel(const float2* __restrict__ T, float* __restrict__ proj, double* __restrict__ rowstats) {
  using PR = ProjRowPair<R1, R2, ROWS>;
  constexpr int M = PR::M, HT = 2 * M, WC = M + 1, NT = PR::NT, S1 = PR::S1;
  __shared__ float2 xin[ROWS][WC + 1];
  __shared__ float2 zb[ROWS][PR::ZR];
  __shared__ float2 pre[M];            // exp(+i pi k / M)
  __shared__ float2 root[PR::NROOT];   // exp(+2 pi i m / M)
  static_assert(32 % R1 == 0, "rows must be lane aligned for the shuffle reduction");
  for (int k = threadIdx.x; k < M; k += blockDim.x) {
    float sn, cs;
    sincospif((float)k / (float)M, &sn, &cs);
    pre[k] = make_float2(cs, sn);
  }
  for (int m = threadIdx.x; m < PR::NROOT; m += blockDim.x) {
    float sn, cs;
    sincospif(2.0f * (float)m / (float)M, &sn, &cs);
    root[m] = make_float2(cs, sn);
  }
  chain_wait();
  LGB_CHAIN_POINTER(T);
  LGB_CHAIN_POINTER(proj);
  LGB_CHAIN_POINTER(rowstats);
  const int c = blockIdx.y;
  const int g = threadIdx.x / NT, t = threadIdx.x - (threadIdx.x / NT) * NT;
  const int row0 = blockIdx.x * ROWS;
  const float2* src = T + ((size_t)c * HT + row0) * WC;
  for (int e = threadIdx.x; e < ROWS * WC; e += blockDim.x) xin[e / WC][e % WC] = src[e];
  __syncthreads();
  // ---- pass 1 (radix R1, stride 1) on the pre-twiddled z[k], k = t + R2*q
  if (t < R2) {
    float2 v[R1];
#pragma unroll
    for (int q = 0; q < R1; ++q) {
      const int k = t + q * R2;
      float2 A = xin[g][k];
      float2 B = xin[g][M - k];
      if (k == 0) { A.y = 0.f; B.y = 0.f; }  // DC and Nyquist: real parts only
      B.y = -B.y;                            // conj
      const float2 xo = cmul(csub(A, B), pre[k]);
      v[q] = cadd(cadd(A, B), mul_i<1>(xo));
    }
    Dft<R1, +1>::run(v);
#pragma unroll
    for (int q = 0; q < R1; ++q) zb[g][t * S1 + q] = v[q];
  }
  __syncthreads();
  // ---- pass 2 (radix R2, stride R1): w[r] = z[t + R1*r]
  float2 w[R2];
#pragma unroll
  for (int r = 0; r < R2; ++r) w[r] = cmul(zb[g][r * S1 + t], root[r * t]);
  Dft<R2, +1>::run(w);
  const int y = row0 + g;
  const int py = (y + HT - HT / 2) % HT;
  const float scale = 1.0f / ((float)HT * (float)HT);
  const bool edge_row = (py == 0) || (py == HT - 1);
  float s1 = 0.f, s2 = 0.f, se = 0.f;
  float* prow = proj + ((size_t)c * HT + py) * HT;
#pragma unroll
  for (int r = 0; r < R2; ++r) {
    const int m = t + r * R1;
    const float a = w[r].x * scale, b = w[r].y * scale;
    const int px0 = (2 * m + HT - HT / 2) % HT;  // even: px0 + 1 does not wrap
    *reinterpret_cast<float2*>(prow + px0) = make_float2(a, b);
    s1 += a + b;
    s2 = fmaf(a, a, fmaf(b, b, s2));
    if (edge_row) {
      se += a + b;
    } else {
      if (px0 == 0) se += a;
      if (px0 + 1 == HT - 1) se += b;
    }
  }
  // row reduction across the row's R1 lanes in FP32 (R1 divides 32, rows are
  // lane aligned); FP64 only for the stored row moments: this GPU's FP64 pipe
  // retires about one operation per SM per clock, conversions included
#pragma unroll
  for (int o = R1 / 2; o > 0; o >>= 1) {
    s1 += __shfl_xor_sync(0xffffffffu, s1, o);
    s2 += __shfl_xor_sync(0xffffffffu, s2, o);
    se += __shfl_xor_sync(0xffffffffu, se, o);
  }
  if (t == 0) {
    double* rs = rowstats + ((size_t)c * HT + py) * 3;
    rs[0] = (double)s1;
    rs[1] = (double)s2;
    rs[2] = (double)se;
  }
}

// proj_row and the zero-padded row rfft in one kernel, for d = 256 templates
// and rows of W = 288 (the refinement crops).  Per row y of T[c]: the 256-point
// c2r through 128 = 16 x 8 complex points, the row moments, the ifftshift (pixel
// pair m -> m' = (m + 64) mod 128), then the rfft of the un-normalised row zero
// padded to W through 144 = 16 x 9 points:
//   A[c][py][k] = sum_{px < d} p[py][px] exp(-2 pi i k px / W),  k <= W/2.
// The projection never goes to memory.  Its normalisation (p - e) s
// (utils.py:106-188) is affine, rfft((p - e) s) = s (A - e U) with
// U[k] = sum_{px < d} exp(-2 pi i k px / W), and is applied by the column pass.
//
// What bounds it: the shared-memory data path and the issue slots, 70 % each.
// The passes: radix 16 of the c2r (8 DFTs a row) -> shared transpose -> radix 8,
// whose thread t then holds the pixel pairs m' = t + 16 q that the rfft's radix-9
// DFT t takes (q = 8 is the zero padding), so that both run in registers -> shared
// transpose -> radix 16 (9 DFTs a row).  Both mirrored reads of the real
// transforms are shuffles between the threads t and -t of a row; roots that
// depend on the thread come from small tables (in registers they cost the
// seventh resident CTA or spill), the others are literals.
// The radix-16 passes have too few DFTs for four warps: warps 0 to 2 finish a row
// group (three rows each), warps 2 and 3 start the next one, two barriers a group.
// 38,304 correlograms: 6.35 ms in four passes with a transpose and a barrier
// between all of them, 5.73 now (five warps, one role each: 7.7).
template <int ROWS>
__global__ void __launch_bounds__(ROWS * 16, 7)
    proj_row_rfft_kernel(const float2* __restrict__ T, double* __restrict__ rowstats, int Wcp, int groups,
                         float2* __restrict__ A) {
  constexpr int HT = 256, M = 128, WC = M + 1, NT = 16, S1 = 17;
  constexpr int WH = 144;  // W / 2
  constexpr int C2 = 8;    // c2r: M = 16 x 8
  constexpr int R2 = 9;    // rfft: WH = 9 x 16
  static_assert(ROWS == 8, "three warps of three rows (the last of two), then two of four");
  // row strides of 8 and 9 (mod 16) float2: the radix-16 passes pack 8 and 9
  // DFTs a row densely onto the lanes without conflicts
  constexpr int SC = C2 * S1, SR = R2 * S1;  // 136 and 153
  static_assert(SC % 16 == 8 && SR % 16 == 9, "conflict-free row strides");
  __shared__ float2 zc[ROWS * SC];  // c2r transpose (8 x 17 a row)
  __shared__ float2 zr[ROWS * SR];  // rfft transpose (9 x 17)
  __shared__ float2 pre[M];         // exp(+i pi k / M)
  __shared__ float2 post[WH + 1];   // exp(-i pi k / WH)
  for (int k = threadIdx.x; k < M; k += blockDim.x) {
    float sn, cs;
    sincospif((float)k / (float)M, &sn, &cs);
    pre[k] = make_float2(cs, sn);
  }
  for (int k = threadIdx.x; k <= WH; k += blockDim.x) {
    float sn, cs;
    sincospif((float)k / (float)WH, &sn, &cs);
    post[k] = make_float2(cs, -sn);
  }
  __syncthreads();
  const int c = blockIdx.y;
  const int warp = threadIdx.x / 32, lane = threadIdx.x & 31;
  const int g = threadIdx.x / NT, t = threadIdx.x % NT;
  // roots of this thread's position: exp(+2 pi i r t / M) = +-pre[2 r t mod M] and
  // exp(-2 pi i r t / WH) = +-post[2 r t mod WH]
  __shared__ float2 rootc[C2 * NT];
  {
    const int m = 2 * (threadIdx.x / NT) * t;
    const float2 v = pre[m & (M - 1)];
    rootc[threadIdx.x] = m < M ? v : make_float2(-v.x, -v.y);
  }
  __shared__ float2 rootr[R2 * NT];
  for (int i = threadIdx.x; i < R2 * NT; i += ROWS * NT) {
    const int m = 2 * (i / NT) * (i % NT);
    const float2 v = post[m <= WH ? m : m - WH];
    rootr[i] = m <= WH ? v : make_float2(-v.x, -v.y);
  }
  const float2 prej = pre[lane % C2], postj = post[lane % R2];
  chain_wait();
  LGB_CHAIN_POINTER(T);
  LGB_CHAIN_POINTER(rowstats);
  LGB_CHAIN_POINTER(A);
  // ---- c2r pass 1 (radix 16) over k = tt + 8q of a group's rows: warps 2 and 3, four rows each
  auto start = [&](int grp) {
    const int tt = lane % C2;
    const int mirror = (lane & ~(C2 - 1)) | ((C2 - tt) & (C2 - 1));  // M - k = (8 - tt) + 8 (15 - q)
    const int gg = lane / C2 + 4 * (warp - 2);
    const float2* src = T + ((size_t)c * HT + (blockIdx.x * groups + grp) * ROWS + gg) * WC;
    float2 x[16], u[16];
#pragma unroll
    for (int q = 0; q < 16; ++q) x[q] = __ldg(src + tt + C2 * q);
    const float2 nyquist = tt == 0 ? __ldg(src + M) : make_float2(0.f, 0.f);
    static_for<16>([&](auto q_) {
      constexpr int q = decltype(q_)::value;
      float2 a = x[q], b;
      b.x = __shfl_sync(0xffffffffu, x[15 - q].x, mirror);
      b.y = __shfl_sync(0xffffffffu, x[15 - q].y, mirror);
      const float2 own = q ? x[(16 - q) % 16] : nyquist;
      if (tt == 0) b = own;
      if (q == 0 && tt == 0) a.y = b.y = 0.f;  // DC and Nyquist: real parts only
      b.y = -b.y;
      const float2 xo = mul_root<q, 32, +1>(cmul(csub(a, b), prej));
      u[q] = cadd(cadd(a, b), mul_i<1>(xo));
    });
    Dft<16, +1>::run(u);
#pragma unroll
    for (int q = 0; q < 16; ++q) zc[gg * SC + tt * S1 + q] = u[q];
  };
  if (warp >= 2) start(0);
#pragma unroll 1
  for (int grp = 0; grp < groups; ++grp) {
    const int row0 = (blockIdx.x * groups + grp) * ROWS;
    __syncthreads();  // this group's c2r rows are there, the last one's rfft rows are read
    // ---- c2r pass 2 (radix 8): pixel pairs m = t + 16 r, moments, and the rfft's
    // pass 1 (radix 9) over m' = t + 16 q, q = (r + 4) mod 8 (the ifftshift)
    {
      const int py = (row0 + g + HT - HT / 2) % HT;
      float2 w[C2], u[R2];
#pragma unroll
      for (int r = 0; r < C2; ++r) {
        w[r] = zc[g * SC + r * S1 + t];
        if (r) w[r] = cmul(w[r], rootc[r * NT + t]);
      }
      Dft<C2, +1>::run(w);
      const float scale = 1.0f / ((float)HT * (float)HT);
      const bool edge_row = (py == 0) || (py == HT - 1);
      float s1 = 0.f, s2 = 0.f, se = 0.f;
#pragma unroll
      for (int r = 0; r < C2; ++r) {
        const float a = w[r].x * scale, b = w[r].y * scale;
        const int q = (r + C2 / 2) % C2, mp = t + q * 16;  // px = 2 mp, 2 mp + 1
        u[q] = make_float2(a, b);
        s1 += a + b;
        s2 = fmaf(a, a, fmaf(b, b, s2));
        if (edge_row) {
          se += a + b;
        } else {
          if (mp == 0) se += a;
          if (mp == M - 1) se += b;
        }
      }
      u[R2 - 1] = make_float2(0.f, 0.f);
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) {
        s1 += __shfl_xor_sync(0xffffffffu, s1, o);
        s2 += __shfl_xor_sync(0xffffffffu, s2, o);
        se += __shfl_xor_sync(0xffffffffu, se, o);
      }
      if (t == 0) {
        double* rs = rowstats + ((size_t)c * HT + py) * 3;
        rs[0] = (double)s1;
        rs[1] = (double)s2;
        rs[2] = (double)se;
      }
      Dft<R2, -1>::run(u);
#pragma unroll
      for (int r = 0; r < R2; ++r) zr[g * SR + r * S1 + t] = r ? cmul(u[r], rootr[r * NT + t]) : u[r];
    }
    __syncthreads();
    if (warp < 3) {
      // ---- rfft pass 2 (radix 16): Z[b + 9 s], then the real post-process with
      // Z[WH - k] = Z[(9 - b) + 9 (15 - s)]
      const int b = lane % R2, own_row = 3 * warp + lane / R2;
      const bool act = lane < 3 * R2 && own_row < ROWS;
      const int row = act ? own_row : 0;
      float2 v[16];
#pragma unroll
      for (int q = 0; q < 16; ++q) v[q] = zr[row * SR + b * S1 + q];
      Dft<16, -1>::run(v);
      const int py = (row0 + row + HT - HT / 2) % HT;
      float2* out = A + ((size_t)c * HT + py) * Wcp + b;
      const int mirror = b ? lane - b + R2 - b : lane;
      static_for<16>([&](auto s_) {
        constexpr int s = decltype(s_)::value;
        float2 zm;
        zm.x = __shfl_sync(0xffffffffu, v[15 - s].x, mirror);
        zm.y = __shfl_sync(0xffffffffu, v[15 - s].y, mirror);
        if (b == 0) zm = v[(16 - s) % 16];
        zm.y = -zm.y;
        const float2 xe = cscale(cadd(v[s], zm), 0.5f);
        const float2 xo = mul_i<-1>(cscale(csub(v[s], zm), 0.5f));
        const float2 X = cadd(xe, mul_root<s, 32, -1>(cmul(xo, postj)));
        if (act) out[R2 * s] = X;
      });
      if (act && b == 0) out[WH] = make_float2(v[0].x - v[0].y, 0.f);
      if (act && WH + 1 + b < Wcp) out[WH + 1] = make_float2(0.f, 0.f);
    }
    if (warp >= 2 && grp + 1 < groups) start(grp + 1);
  }
}

// Factors of the normalisation that depend on sizes alone: the FP64 divisions
// and the square root of them were half of norm_constants_kernel's time.
struct NormSizes {
  int h;
  double inv_edge;   // 1 / (4 h - 4)
  double n;          // h^2
  double mean;       // rel^2 / n, rel = n / (H W)
  double border;     // (H - h) (W - h)
  double root;       // sqrt(H W)
  NormSizes(int h_, int H, int W)
      : h(h_), inv_edge(1.0 / (4.0 * h_ - 4.0)), n((double)h_ * h_), mean(n / ((double)H * W) / ((double)H * W)),
        border((double)(H - h_) * (double)(W - h_)), root(sqrt((double)H * (double)W)) {}
};

// Normalisation constants of utils.py:106-188 from the per-row moments:
// returns edge mean e and scale s such that normalised = (p - e) * s.
// Called by all 32 lanes of warp 0 (the launcher guarantees a full warp);
// lane 0 gets the constants and, returned, the projection's sum.
__device__ inline double projection_norm_constants(const double* rs, const NormSizes& ns, float* e_out, float* s_out) {
  // warp 0 reduces h rows
  double s1 = 0, s2 = 0, se = 0;
  const int lane = threadIdx.x & 31;
#pragma unroll 4
  for (int r = lane; r < ns.h; r += 32) {
    s1 += rs[3 * r];
    s2 += rs[3 * r + 1];
    se += rs[3 * r + 2];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    s1 += __shfl_down_sync(0xffffffffu, s1, o);
    s2 += __shfl_down_sync(0xffffffffu, s2, o);
    se += __shfl_down_sync(0xffffffffu, se, o);
  }
  if (lane == 0) {
    const double e = se * ns.inv_edge;
    const double S1 = s1 - ns.n * e;                     // sum of (p - e)
    const double S2 = s2 - 2.0 * e * s1 + ns.n * e * e;  // sum of (p - e)^2
    const double mean = S1 * ns.mean;
    double var = S2 - 2.0 * mean * S1 + ns.n * mean * mean;
    var += ns.border * mean * mean;
    if (var < 1e-8) var = 1e-8;
    *e_out = (float)e;
    *s_out = (float)(ns.root * rsqrt(var));
  }
  return s1;
}

// ---------------------------------------------------------------------------
// pad_rfft: A[c][y][k] = rfft_W( normalised projection row y, zero padded )
// for k = 0..W/2, zeros up to Wcp.  The normalisation is that of a
// norm_h x norm_w micrograph (W may exceed norm_w when the micrograph was
// zero padded to a supported FFT length).  Real FFT of length W = 2*WH through a
// WH-point complex FFT (first pass pruned to the h/2 non-zero inputs; templates
// are even).  The short rows: a CTA holds many and fills the shared tables of
// twiddles and post-twiddles once for them.
// ---------------------------------------------------------------------------
template <int WH, int ROWS>
__global__ void __launch_bounds__(ROWS* FftThreads<WH>::value)
    pad_rfft_kernel(const float* __restrict__ proj, const double* __restrict__ rowstats, int h, NormSizes sizes,
                    int Wcp, int norm_ready, float2* __restrict__ A) {
  constexpr int NT = FftThreads<WH>::value;
  constexpr int ZS = IdxPad16::pad(WH) + 2;
  __shared__ float2 z[ROWS][ZS];
  __shared__ float2 post[WH + 1];  // exp(-i pi k / WH)
  __shared__ float2 tab[FftTable<WH>::SIZE + 1];
  fill_fft_table<WH>(tab, threadIdx.x, blockDim.x);
  for (int k = threadIdx.x; k <= WH; k += blockDim.x) {
    float sn, cs;
    sincospif((float)k / (float)WH, &sn, &cs);
    post[k] = make_float2(cs, -sn);
  }
  const int c = blockIdx.y;
  chain_wait();
  LGB_CHAIN_POINTER(proj);
  LGB_CHAIN_POINTER(rowstats);
  LGB_CHAIN_POINTER(A);
  // norm_ready: constants (e, s) precomputed by norm_constants_kernel as a
  // float2 over rowstats[c][0][0]; otherwise warp 0 reduces the row moments here
  __shared__ float norm[2];
  if (norm_ready) {
    if (threadIdx.x == 0) {
      const float2 es = *reinterpret_cast<const float2*>(rowstats + (size_t)c * h * 3);
      norm[0] = es.x;
      norm[1] = es.y;
    }
  } else if (threadIdx.x < 32) {
    projection_norm_constants(rowstats + (size_t)c * h * 3, sizes, &norm[0], &norm[1]);
  }
  __syncthreads();
  const float e = norm[0], s = norm[1];
  const int g = threadIdx.x / NT, t = threadIdx.x - (threadIdx.x / NT) * NT;
  const int y = blockIdx.x * ROWS + g;
  const bool active = y < h;
  const int nz = h / 2;
  if (active) {
    const float* p = proj + ((size_t)c * h + y) * h;
    for (int m = t; m < nz; m += NT) z[g][IdxPad16::f(m)] = make_float2((p[2 * m] - e) * s, (p[2 * m + 1] - e) * s);
  }
  __syncthreads();
  block_fft_pruned_tab<WH, NT, -1, IdxPad16>(z[g], tab, t, nz);
  if (!active) return;
  float2* out = A + ((size_t)c * h + y) * Wcp;
  for (int k = t; k <= WH; k += NT) {
    const float2 Zk = z[g][IdxPad16::f(k == WH ? 0 : k)];
    const float2 Zm = cconj(z[g][IdxPad16::f(k == 0 ? 0 : WH - k)]);
    const float2 xe = cscale(cadd(Zk, Zm), 0.5f);
    const float2 xo = mul_i<-1>(cscale(csub(Zk, Zm), 0.5f));
    out[k] = cadd(xe, cmul(post[k], xo));
  }
  for (int k = WH + 1 + t; k < Wcp; k += NT) out[k] = make_float2(0.f, 0.f);
}


// ---------------------------------------------------------------------------
// rowpass: row y of every correlogram in the batch: c2r of length W = 2*WH
// (imaginary parts of DC / Nyquist ignored), scale 1/(H W) (passed in), then the fused
// statistics update of utils.py:191-255 (max over the batch in c order with
// strict '>', MIP update with strict '>', global index, FP64 sums).
// ---------------------------------------------------------------------------
constexpr int kRowThreads = 256;

template <int WH>
struct RowGeneric {
  static constexpr size_t SMEM = sizeof(float2) * ((size_t)WH + 4 + IdxPad16::pad(WH) + 2 + WH +
                                                   FftTable<WH>::SIZE + 1);
};

// Largest divisor of WH that is <= kRowThreads (threads of one rowpass CTA).
constexpr int row_threads(int wh, int cand = kRowThreads) {
  return cand <= 1 ? 1 : (wh % cand == 0 ? cand : row_threads(wh, cand - 1));
}

template <int WH, int NT>
__global__ void __launch_bounds__(NT, 2)
    rowpass_kernel(const float2* __restrict__ Y, int y_rows, int Wcp, int n_c, int nb, int n_orient, int o0,
                   const int* __restrict__ o0_dev, float scale, float* __restrict__ mip, int* __restrict__ best,
                   double* __restrict__ s1, double* __restrict__ s2) {
  static_assert(NT >= FftThreads<WH>::value, "row FFT needs more threads");
  static_assert(WH % NT == 0, "row length must be a multiple of the CTA size");
  constexpr int PIX = WH / NT;
  constexpr int ZS = IdxPad16::pad(WH) + 2;
  // dynamic shared memory (RowGeneric<WH>::SMEM): row, transform, c2r
  // pre-twiddles and FFT twiddle table (filled once, reused by every correlogram)
  extern __shared__ float2 rgsm[];
  float2* xr = rgsm;
  float2* z = xr + WH + 4;
  float2* pre = z + ZS;
  float2* tab = pre + WH;
  const int y = blockIdx.x;
  const int t = threadIdx.x;
  fill_fft_table<WH>(tab, t, NT);
  for (int k = t; k < WH; k += NT) {
    float sn, cs;
    sincospif((float)k / (float)WH, &sn, &cs);
    pre[k] = make_float2(cs, sn);
  }
  chain_wait();
  LGB_CHAIN_POINTER(Y);
  LGB_CHAIN_POINTER(o0_dev);
  LGB_CHAIN_POINTER(mip);
  LGB_CHAIN_POINTER(best);
  LGB_CHAIN_POINTER(s1);
  LGB_CHAIN_POINTER(s2);
  float bmax[2 * PIX], bs[2 * PIX], bss[2 * PIX];
  int barg[2 * PIX];
#pragma unroll
  for (int i = 0; i < 2 * PIX; ++i) {
    bmax[i] = -INFINITY;
    barg[i] = 0;
    bs[i] = 0.f;
    bss[i] = 0.f;
  }
  for (int c = 0; c < n_c; ++c) {
    const float2* row = Y + ((size_t)c * y_rows + y) * Wcp;
    for (int k = t; k <= WH; k += NT) xr[k] = row[k];
    __syncthreads();
    for (int k = t; k < WH; k += NT) {
      float2 A = xr[k];
      float2 B = xr[WH - k];
      if (k == 0) { A.y = 0.f; B.y = 0.f; }
      B.y = -B.y;
      const float2 xe = cadd(A, B);
      const float2 xo = cmul(csub(A, B), pre[k]);
      z[IdxPad16::f(k)] = cadd(xe, mul_i<1>(xo));
    }
    __syncthreads();
    block_fft_tab<WH, NT, +1, IdxPad16>(z, tab, t);
#pragma unroll
    for (int r = 0; r < PIX; ++r) {
      const float2 v = z[IdxPad16::f(t + r * NT)];
      const float a = v.x * scale, b = v.y * scale;
      if (a > bmax[2 * r]) { bmax[2 * r] = a; barg[2 * r] = c; }
      if (b > bmax[2 * r + 1]) { bmax[2 * r + 1] = b; barg[2 * r + 1] = c; }
      bs[2 * r] += a;
      bss[2 * r] = fmaf(a, a, bss[2 * r]);
      bs[2 * r + 1] += b;
      bss[2 * r + 1] = fmaf(b, b, bss[2 * r + 1]);
    }
    __syncthreads();
  }
  const size_t W = 2 * (size_t)WH;
  if (o0_dev) o0 += *o0_dev;
#pragma unroll
  for (int r = 0; r < PIX; ++r) {
    const size_t idx = (size_t)y * W + 2 * (size_t)(t + r * NT);
    float2 m = *reinterpret_cast<float2*>(mip + idx);
    int2 bi = *reinterpret_cast<int2*>(best + idx);
    double2 a = *reinterpret_cast<double2*>(s1 + idx);
    double2 q = *reinterpret_cast<double2*>(s2 + idx);
    if (bmax[2 * r] > m.x) {
      m.x = bmax[2 * r];
      const int cc = barg[2 * r];
      bi.x = (cc / nb) * n_orient + o0 + (cc - (cc / nb) * nb);
    }
    if (bmax[2 * r + 1] > m.y) {
      m.y = bmax[2 * r + 1];
      const int cc = barg[2 * r + 1];
      bi.y = (cc / nb) * n_orient + o0 + (cc - (cc / nb) * nb);
    }
    a.x += f2d_bits(bs[2 * r]);
    a.y += f2d_bits(bs[2 * r + 1]);
    q.x += f2d_bits(bss[2 * r]);
    q.y += f2d_bits(bss[2 * r + 1]);
    *reinterpret_cast<float2*>(mip + idx) = m;
    *reinterpret_cast<int2*>(best + idx) = bi;
    *reinterpret_cast<double2*>(s1 + idx) = a;
    *reinterpret_cast<double2*>(s2 + idx) = q;
  }
}

}  // namespace lgb
