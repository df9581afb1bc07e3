// Register-fused column passes of the plain FP32 search.
//
// colpass_fused_kernel<R>  (H = R^2 = 64, 256, one butterfly per thread per pass)
//   The forward FFT's last Stockham pass leaves element j + q*H/R of the
//   column in thread j, and the inverse FFT's first pass consumes exactly those
//   elements in the same thread: forward-last -> cross power -> inverse-first
//   run in registers.  The pruned forward first pass reads its (at most two)
//   non-zero inputs straight from global memory, the inverse last pass writes
//   its outputs straight to global memory, so each correlogram column costs
//   four shared-memory round trips instead of eight.  Twiddles come from a
//   per-CTA shared table (built once with sincospif).  Thread layout: lane
//   bits 0-1 select one of four adjacent columns, so each warp touches 8 rows
//   x 32 B: whole sectors.
#pragma once

#include "fft.cuh"
#include "match_kernels.cuh"

namespace lgb {

// L2 placement: measured, neither an evict_last policy on the image-spectrum
// loads nor streaming stores of the intermediate help -- both take L2 away
// from the correlogram rows that the row pass re-reads right after.

// exp(-2 pi i r / 16), r = 0..15 (roots for the sparse first pass; R | 16)
static __constant__ float2 kRootsFwd16[16] = {
    {1.0f, 0.0f},
    {0.92387953251128674f, -0.38268343236508977f},
    {0.70710678118654752f, -0.70710678118654752f},
    {0.38268343236508977f, -0.92387953251128674f},
    {0.0f, -1.0f},
    {-0.38268343236508977f, -0.92387953251128674f},
    {-0.70710678118654752f, -0.70710678118654752f},
    {-0.92387953251128674f, -0.38268343236508977f},
    {-1.0f, 0.0f},
    {-0.92387953251128674f, 0.38268343236508977f},
    {-0.70710678118654752f, 0.70710678118654752f},
    {-0.38268343236508977f, 0.92387953251128674f},
    {0.0f, 1.0f},
    {0.38268343236508977f, 0.92387953251128674f},
    {0.70710678118654752f, 0.70710678118654752f},
    {0.92387953251128674f, 0.38268343236508977f},
};

// Value of v that the compiler cannot treat as loop invariant: keeps per-row
// address arithmetic inside the loop instead of holding 16 hoisted addresses.
__device__ __forceinline__ int opaque(int v) {
  int r;
  asm volatile("mov.b32 %0, %1;" : "=r"(r) : "r"(v));
  return r;
}

// ---------------------------------------------------------------------------
// Fused column pass for H = R^2.
// ---------------------------------------------------------------------------
template <int R>
struct ColFused {
  using RL = Radices<R, R>;
  static constexpr int N = R * R;
  static constexpr int NB = R;                        // butterflies per pass = threads per column
  static constexpr int THREADS = kColGroup * NB;
  static constexpr int STRIDE = IdxPad16::pad(N) + 4; // column stride in shared memory (float2)
  static constexpr int TAB = TableSize<1, RL>::value; // twiddle entries of the second pass
  static constexpr size_t SMEM = sizeof(float2) * (size_t)(kColGroup * STRIDE + TAB);
};

template <int R>
__global__ void __launch_bounds__(ColFused<R>::THREADS, 1)
    colpass_fused_kernel(const float2* __restrict__ A, const float2* __restrict__ Ip, int ips, int h, int Wcp, int n_c,
                         int c_per_block, int c_per_image, int y_rows, float2* __restrict__ Y) {
  using CF = ColFused<R>;
  using RL = typename CF::RL;
  constexpr int N = CF::N, NB = CF::NB, STRIDE = CF::STRIDE;
  extern __shared__ float2 csm[];
  float2* tab = csm + kColGroup * STRIDE;
  FillTables<N, 1, RL>::run(tab, threadIdx.x, CF::THREADS);

  const int lane = threadIdx.x & 31;
  const int g = lane & 3;                             // column within the group
  const int j = (threadIdx.x >> 5) * 8 + (lane >> 2); // butterfly index
  float2* x = csm + g * STRIDE;
  const int kx = blockIdx.x * kColGroup + g;
  const int c_begin = blockIdx.y * c_per_block;
  const int c_end = min(n_c, c_begin + c_per_block);
  // first-pass sparse form: at most two non-zero inputs per butterfly when h <= 2*NB
  const bool sparse = h <= 2 * NB;
  chain_wait();
  LGB_CHAIN_POINTER(A);
  LGB_CHAIN_POINTER(Ip);
  LGB_CHAIN_POINTER(Y);
  __syncthreads();

  const int fj = IdxPad16::f(j);
  const int f1 = padded_first<R>(j);
  // sparse inputs of the first correlogram; later ones are prefetched one
  // correlogram ahead, while the current one is transformed
  float2 nx0 = make_float2(0.f, 0.f), nx1 = make_float2(0.f, 0.f);
  if (sparse && c_begin < c_end) {
    const float2* a = A + (size_t)c_begin * h * Wcp + kx;
    if (j < h) nx0 = __ldg(a + (size_t)j * Wcp);
    if (j + NB < h) nx1 = __ldg(a + (size_t)(j + NB) * Wcp);
  }
#pragma unroll 1
  for (int c = c_begin; c < c_end; ++c) {
    float2 v[R];
    const size_t ws = (size_t)opaque(Wcp);  // row stride, re-derived per correlogram
    const float2* a = A + (size_t)c * h * ws + kx;
    // ---- forward pass 1 (stride 1, inputs from global, rows >= h are zero)
    if (sparse) {
      const float2 x0 = nx0, x1 = nx1;
      if (c + 1 < c_end) {
        const float2* an = a + (size_t)h * ws;
        nx0 = j < h ? __ldg(an + (size_t)j * ws) : make_float2(0.f, 0.f);
        nx1 = j + NB < h ? __ldg(an + (size_t)(j + NB) * ws) : make_float2(0.f, 0.f);
      }
      // y[r] = x0 + x1 * exp(-2 pi i r / R)
      static_assert(16 % R == 0, "sparse first pass needs R | 16");
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = cadd(x0, cmul(x1, kRootsFwd16[r * (16 / R)]));
    } else {
      const float2* ar = a + (size_t)j * ws;
#pragma unroll
      for (int q = 0; q < R; ++q) {
        v[q] = j + q * NB < h ? __ldg(ar) : make_float2(0.f, 0.f);
        ar += NB * ws;
      }
      Dft<R, -1>::run(v);
    }
#pragma unroll
    for (int q = 0; q < R; ++q) x[f1 + q] = v[q];
    __syncthreads();
    // ---- forward pass 2 -> registers
#pragma unroll
    for (int q = 0; q < R; ++q) v[q] = x[padded_at<IdxPad16, NB>(fj, j, q)];
    twiddle_from_table<R, -1, R>(v, tab, j);
    Dft<R, -1>::run(v);
    // v[q] = P[row j + q*NB]; cross power with the image spectrum, P[0,0] = 0
    {
      const float2* ip = Ip + ((size_t)(c / c_per_image) * N + j) * ips + kx;
#pragma unroll
      for (int q = 0; q < R; ++q) {
        const float2 I = kx < ips ? __ldg(ip) : make_float2(0.f, 0.f);
        ip += (size_t)NB * ips;
        v[q] = (q == 0 && j == 0 && kx == 0) ? make_float2(0.f, 0.f) : cmulc(I, v[q]);
      }
    }
    // ---- inverse pass 1 in registers (stride 1, no twiddles)
    Dft<R, +1>::run(v);
    __syncthreads();  // everyone has read the forward pass 2 inputs
#pragma unroll
    for (int q = 0; q < R; ++q) x[f1 + q] = v[q];
    __syncthreads();
    // ---- inverse pass 2 -> global
#pragma unroll
    for (int q = 0; q < R; ++q) v[q] = x[padded_at<IdxPad16, NB>(fj, j, q)];
    twiddle_from_table<R, +1, R>(v, tab, j);
    Dft<R, +1>::run(v);
    float2* yo = Y + (size_t)c * y_rows * ws + (size_t)j * ws + kx;
#pragma unroll
    for (int q = 0; q < R; ++q) {
      if (j + q * NB < y_rows) *yo = v[q];
      yo += NB * ws;
    }
    __syncthreads();  // before the next correlogram's first-pass stores
  }
}

// ---------------------------------------------------------------------------
// Column pass for the short lengths without a uniform R^P plan: the generic
// Stockham schedule of Plan<HN> with the twiddles of every pass
// after the first read from one shared table (filled once per CTA) instead
// of sincospif per butterfly.  The forward first pass is pruned to the h
// non-zero inputs.  G columns per CTA.
// ---------------------------------------------------------------------------
template <int HN>
struct ColTab {
  using RL = typename Plan<HN>::type;
  static constexpr int NT = FftThreads<HN>::value;
  static constexpr int G = kColGroup;
  static constexpr int STRIDE = IdxPad16::pad(HN) + 4;
  static constexpr int TAB = TableSize<1, RL>::value;
  static constexpr size_t SMEM = sizeof(float2) * ((size_t)G * STRIDE + TAB);
};

template <int HN>
__global__ void __launch_bounds__(ColTab<HN>::G* ColTab<HN>::NT)
    colpass_tab_kernel(const float2* __restrict__ A, const float2* __restrict__ Ip, int ips, int h, int Wcp, int n_c,
                       int c_per_block, int c_per_image, int y_rows, float2* __restrict__ Y) {
  using CT = ColTab<HN>;
  using RL = typename CT::RL;
  constexpr int NT = CT::NT, G = CT::G, STRIDE = CT::STRIDE, NTH = G * NT;
  constexpr int R1 = Head<RL>::value;
  extern __shared__ float2 ctsm[];
  float2* tab = ctsm + G * STRIDE;
  FillTables<HN, 1, RL>::run(tab, threadIdx.x, NTH);
  const int kx0 = blockIdx.x * G;
  const int c_begin = blockIdx.y * c_per_block;
  const int c_end = min(n_c, c_begin + c_per_block);
  const int g = threadIdx.x / NT, t = threadIdx.x - (threadIdx.x / NT) * NT;
  float2* x = ctsm + g * STRIDE;
  chain_wait();
  LGB_CHAIN_POINTER(A);
  LGB_CHAIN_POINTER(Ip);
  LGB_CHAIN_POINTER(Y);
  __syncthreads();
#pragma unroll 1
  for (int c = c_begin; c < c_end; ++c) {
    const float2* a = A + (size_t)c * h * Wcp + kx0;
    for (int e = threadIdx.x; e < h * G; e += NTH) {
      const int y = e / G, i = e % G;
      // the last group may run past Wcp when G does not divide it
      ctsm[i * STRIDE + IdxPad16::f(y)] = kx0 + i < Wcp ? a[(size_t)y * Wcp + i] : make_float2(0.f, 0.f);
    }
    __syncthreads();
    // forward: pruned first pass (no twiddles), then the table passes
    stockham_pass<HN, R1, 1, NT, -1, IdxPad16, true>(x, t, h);
    TablePasses<HN, NT, -1, IdxPad16, R1, typename Tail<RL>::type>::run(x, tab, t);
    const float2* ipc = Ip + (size_t)(c / c_per_image) * HN * ips;
    for (int e = threadIdx.x; e < HN * G; e += NTH) {
      const int y = e / G, i = e % G;
      const float2 I = kx0 + i < ips ? __ldg(ipc + (size_t)y * ips + kx0 + i) : make_float2(0.f, 0.f);
      const int si = i * STRIDE + IdxPad16::f(y);
      float2 X = cmulc(I, ctsm[si]);
      if (y == 0 && kx0 + i == 0) X = make_float2(0.f, 0.f);
      ctsm[si] = X;
    }
    __syncthreads();
    TablePasses<HN, NT, +1, IdxPad16, 1, RL>::run(x, tab, t);
    float2* yo = Y + (size_t)c * y_rows * Wcp + kx0;
    for (int e = threadIdx.x; e < y_rows * G; e += NTH) {
      const int y = e / G, i = e % G;
      if (kx0 + i < Wcp) yo[(size_t)y * Wcp + i] = ctsm[i * STRIDE + IdxPad16::f(y)];
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// Column pass for H = R1*R2 (288 = 16*18) in two register passes per
// direction.  Forward (Stockham): radix R1 over rows b + R2*q (pruned to the h
// non-zero rows, read from global) -> shared transpose M1[b][q] -> radix R2
// with twiddles w^(r*b), which leaves P[b + R1*r] in thread b; the cross
// power and the inverse's first pass (radix R2, stride 1: the same elements)
// stay in registers -> shared transpose M2[b][r] -> inverse radix R1 with
// twiddles w^(-q*b) -> rows b + R2*q to global.  Two shared round trips per
// column and correlogram; twiddle roots exp(-2 pi i m / H) for m = r*b <=
// (R1-1)(R2-1) from one shared table.  Odd transpose row strides and a column
// stride of 2 (mod 16) float2 make both transposes conflict free for the
// lane layout (8 columns x consecutive butterflies).
// ---------------------------------------------------------------------------
template <int R1, int R2>
struct ColPair {
  static constexpr int N = R1 * R2;
  static constexpr int NT = R1 > R2 ? R1 : R2;  // threads per column
  static constexpr int G = 8;                   // columns per CTA: 64 B row segments
  static constexpr int THREADS = G * NT;
  static constexpr int S1 = R1 + 1, S2 = R2 + 1;  // transpose row strides
  static_assert(S1 % 2 == 1 && S2 % 2 == 1, "odd transpose strides");
  static constexpr int CB = R2 * S1 > R1 * S2 ? R2 * S1 : R1 * S2;
  static constexpr int STRIDE = CB + (18 - CB % 16) % 16;  // = 2 (mod 16)
  static constexpr int NROOT = (R1 - 1) * (R2 - 1) + 1;
  static constexpr size_t SMEM = sizeof(float2) * ((size_t)G * STRIDE + NROOT);
};

// QOUT: rows below QOUT R2 cover y_rows, the others' outputs are not computed (the
// issue slots bound this kernel; 38,304 correlograms of 33 rows: 6.54 -> 6.12 ms).
template <int R1, int R2, int QOUT>
__global__ void __launch_bounds__(ColPair<R1, R2>::THREADS, 4)
    colpass_pair_kernel(const float2* __restrict__ A, const float2* __restrict__ Ip, int ips, int h, int Wcp, int n_c,
                        int c_per_block, int c_per_image, int y_rows, float2* __restrict__ Y,
                        const float2* __restrict__ norm, int norm_stride, int norm_w) {
  using CP = ColPair<R1, R2>;
  constexpr int N = CP::N, G = CP::G, S1 = CP::S1, S2 = CP::S2;
  extern __shared__ float2 psm[];
  float2* root = psm + G * CP::STRIDE;  // root[m] = exp(-2 pi i m / N)
  for (int m = threadIdx.x; m < CP::NROOT; m += CP::THREADS) {
    float sn, cs;
    sincospif(2.0f * (float)m / (float)N, &sn, &cs);
    root[m] = make_float2(cs, -sn);
  }
  const int g = threadIdx.x % G, b = threadIdx.x / G;
  const int kx = blockIdx.x * G + g;
  const bool col_ok = kx < Wcp;  // the last group may run past Wcp
  float2* x = psm + g * CP::STRIDE;
  const int c_begin = blockIdx.y * c_per_block;
  const int c_end = min(n_c, c_begin + c_per_block);
  // deferred normalisation: rfft_W((p - e) s) = s (A - e U), U[k] = sum_{x<h} w^(k x)
  // = exp(-i pi k (h-1) / W) sin(pi k h / W) / sin(pi k / W), w = exp(-2 pi i / W)
  float2 U = make_float2(0.f, 0.f);
  if (norm && col_ok && kx <= norm_w / 2) {
    if (kx == 0) {
      U = make_float2((float)h, 0.f);
    } else {
      const int w2 = 2 * norm_w;
      float sa, ca, sn, cn, sd, cd;
      sincospif((float)((kx * (h - 1)) % w2) / (float)norm_w, &sa, &ca);
      sincospif((float)((kx * h) % w2) / (float)norm_w, &sn, &cn);
      sincospif((float)kx / (float)norm_w, &sd, &cd);
      const float mag = sn / sd;
      U = make_float2(ca * mag, -sa * mag);
    }
  }
  chain_wait();
  LGB_CHAIN_POINTER(A);
  LGB_CHAIN_POINTER(Ip);
  LGB_CHAIN_POINTER(Y);
  LGB_CHAIN_POINTER(norm);
  __syncthreads();
#pragma unroll 1
  for (int c = c_begin; c < c_end; ++c) {
    // ---- forward pass 1 (radix R1, stride 1): rows b + R2*q, rows >= h are zero
    if (b < R2) {
      float2 v[R1];
      const float2* a = A + ((size_t)c * h + b) * Wcp + kx;
#pragma unroll
      for (int q = 0; q < R1; ++q)
        v[q] = (col_ok && b + q * R2 < h) ? __ldg(a + (size_t)q * R2 * Wcp) : make_float2(0.f, 0.f);
      if (norm) {
        const float2 es = __ldg(norm + (size_t)c * norm_stride);
        const float2 eU = make_float2(es.x * U.x, es.x * U.y);
#pragma unroll
        for (int q = 0; q < R1; ++q)
          if (b + q * R2 < h) v[q] = make_float2(es.y * (v[q].x - eU.x), es.y * (v[q].y - eU.y));
      }
      Dft<R1, -1>::run(v);
#pragma unroll
      for (int q = 0; q < R1; ++q) x[b * S1 + q] = v[q];
    }
    __syncthreads();
    float2 w[R2];
    if (b < R1) {
      // ---- forward pass 2 (radix R2, stride R1): w[r] = P[row b + R1*r]
#pragma unroll
      for (int r = 0; r < R2; ++r) w[r] = cmul(x[r * S1 + b], root[r * b]);
      Dft<R2, -1>::run(w);
      // ---- cross power with the image spectrum, P[0,0] = 0
      const float2* ip = Ip + ((size_t)(c / c_per_image) * N + b) * ips + kx;
#pragma unroll
      for (int r = 0; r < R2; ++r) {
        const float2 I = kx < ips ? __ldg(ip + (size_t)r * R1 * ips) : make_float2(0.f, 0.f);
        w[r] = (r == 0 && b == 0 && kx == 0) ? make_float2(0.f, 0.f) : cmulc(I, w[r]);
      }
      // ---- inverse pass 1 (radix R2, stride 1) on the same elements
      Dft<R2, +1>::run(w);
    }
    __syncthreads();  // every read of M1 is done
    if (b < R1) {
#pragma unroll
      for (int r = 0; r < R2; ++r) x[b * S2 + r] = w[r];
    }
    __syncthreads();
    // ---- inverse pass 2 (radix R1, stride R2) -> rows b + R2*q
    if (b < R2) {
      float2 v[R1];
#pragma unroll
      for (int q = 0; q < R1; ++q) v[q] = cmulc(x[q * S2 + b], root[q * b]);
      Dft<R1, +1>::run(v);
      if (col_ok) {
        float2* yo = Y + ((size_t)c * y_rows + b) * Wcp + kx;
#pragma unroll
        for (int q = 0; q < QOUT; ++q)
          if (b + q * R2 < y_rows) yo[(size_t)q * R2 * Wcp] = v[q];
      }
    }
    __syncthreads();  // before the next correlogram's pass-1 stores
  }
}

}  // namespace lgb
