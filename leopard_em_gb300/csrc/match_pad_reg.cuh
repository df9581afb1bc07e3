// Zero-padded rfft of the normalised projection rows (W = 2 WH) for the longer
// rows: a WH-point complex transform in three passes of about 16 points a
// thread.  The first pass takes its inputs (zeros beyond the template) straight
// from the projection, normalised on the way; in the last pass a thread has the
// butterflies j and WH/R - j, whose outputs mirror each other, so that the real
// post-process X[k] = xe + t, X[WH - k] = conj(xe - t) runs in registers.
//
// What bounds it: the shared-memory data path.  Four or five radix-8 passes through
// shared memory and mirrored reads for the post-process took it to 71 % (and a
// CTA walked 32 rows even where few CTAs were left); three passes move half as
// much.  Microseconds a batch (with the constants), before -> now:
//   4096, 192 correlograms of 384: 560 -> 402    3840, 84 of 256: 223 -> 117
//   2048, 32 of 64: 30.7 -> 12.1, 4 of 64: 30.5 -> 6.2
//   512, 32 of 64: 7.2 -> 6.3, 8 of 64: 6.9 -> 5.0, 96 of 128: 16.8 -> 15.0
#pragma once

#include "match_kernels.cuh"
#include "reg_dft.cuh"

namespace lgb {

template <int WH_, int NT_, int ROWS_, class RL_>
struct PadReg {
  using RL = RL_;
  static constexpr int WH = WH_, NT = NT_, ROWS = ROWS_, THREADS = NT * ROWS;
  static constexpr int R1 = Head<RL>::value, RLAST = Last<RL>::value;
  static constexpr int NB1 = WH / R1, PER1 = (NB1 + NT - 1) / NT;
  static constexpr int NBL = WH / RLAST, UNITS = NBL / 2, PERU = (UNITS + NT - 1) / NT;
  static_assert(NBL % 2 == 0, "butterfly 0 is paired with NBL / 2");
  static constexpr int ZS = IdxPad16::pad(WH) + 2;
  static constexpr int TAB = TableSize<1, RL>::value;
  static constexpr size_t SMEM = sizeof(float2) * ((size_t)ROWS * ZS + TAB);
};

template <class C>
__global__ void __launch_bounds__(C::THREADS)
    pad_rfft_reg_kernel(const float* __restrict__ proj, const double* __restrict__ rowstats, int h, NormSizes sizes,
                        int Wcp, int norm_ready, int rows_per_cta, float2* __restrict__ A) {
  using RL = typename C::RL;
  constexpr int WH = C::WH, NT = C::NT, ROWS = C::ROWS, R1 = C::R1, R = C::RLAST, NB1 = C::NB1, NBL = C::NBL;
  extern __shared__ float2 pgsm[];
  __shared__ float norm[2];
  const int g = ROWS == 1 ? 0 : threadIdx.x / NT, t = ROWS == 1 ? threadIdx.x : threadIdx.x - g * NT;
  float2* z = pgsm + g * C::ZS;
  float2* tab = pgsm + ROWS * C::ZS;
  FillTables<WH, 1, RL>::run(tab, threadIdx.x, C::THREADS);
  const float2* tab_last = tab + TableSize<1, typename DropLast<RL>::type>::value;
  // post-process roots exp(-i pi k / WH) at k = j + q NBL: this one times exp(-i pi q / R)
  float2 post[C::PERU];
#pragma unroll
  for (int p = 0; p < C::PERU; ++p) {
    float sn, cs;
    sincospif((float)(t + p * NT) / (float)WH, &sn, &cs);
    post[p] = make_float2(cs, -sn);
  }
  chain_wait();
  LGB_CHAIN_POINTER(proj);
  LGB_CHAIN_POINTER(rowstats);
  LGB_CHAIN_POINTER(A);
  const int c = blockIdx.y;
  // the constants (e, s): precomputed over rowstats[c][0][0], or reduced here by warp 0
  if (norm_ready) {
    if (threadIdx.x < 2) norm[threadIdx.x] = reinterpret_cast<const float*>(rowstats + (size_t)c * h * 3)[threadIdx.x];
  } else if (threadIdx.x < 32) {
    projection_norm_constants(rowstats + (size_t)c * h * 3, sizes, &norm[0], &norm[1]);
  }
  __syncthreads();
  const float e = norm[0], s = norm[1];
  const int nz = h / 2;  // templates are even
  const int y_end = min(h, (int)(blockIdx.x + 1) * rows_per_cta);
#pragma unroll 1
  for (int y0 = blockIdx.x * rows_per_cta; y0 < y_end; y0 += ROWS) {
    const int y = y0 + g;
    const bool active = y < y_end;
    const float2* p = reinterpret_cast<const float2*>(proj + ((size_t)c * h + (active ? y : y0)) * h);
#pragma unroll
    for (int i = 0; i < C::PER1; ++i) {
      const int j = t + i * NT;
      if (NB1 % NT == 0 || j < NB1) {
        float2 u[R1];
#pragma unroll
        for (int q = 0; q < R1; ++q) {
          u[q] = make_float2(0.f, 0.f);
          if (j + q * NB1 < nz) {
            const float2 v = __ldg(p + j + q * NB1);
            u[q] = make_float2((v.x - e) * s, (v.y - e) * s);
          }
        }
        Dft<R1, -1>::run(u);
#pragma unroll
        for (int q = 0; q < R1; ++q) z[IdxPad16::f(j * R1 + q)] = u[q];
      }
    }
    __syncthreads();
    TablePasses<WH, NT, -1, IdxPad16, R1, typename Middle<RL>::type>::run(z, tab, t);
    float2* out = A + ((size_t)c * h + y) * Wcp;
#pragma unroll
    for (int i = 0; i < C::PERU; ++i) {
      const int j = t + i * NT;
      if (C::UNITS % NT == 0 || j < C::UNITS) {
        const int jm = j ? NBL - j : NBL / 2;
        float2 a[R], b[R];
        const int fa = IdxPad16::f(j), fb = IdxPad16::f(jm);
#pragma unroll
        for (int q = 0; q < R; ++q) {
          a[q] = z[padded_at<IdxPad16, NBL>(fa, j, q)];
          b[q] = z[padded_at<IdxPad16, NBL>(fb, jm, q)];
        }
        twiddle_from_table<R, -1, NBL>(a, tab_last, j);
        twiddle_from_table<R, -1, NBL>(b, tab_last, jm);
        Dft<R, -1>::run(a);
        Dft<R, -1>::run(b);
        if (active) {
          // X[k] and X[WH - k] from Z[k] and Z[WH - k], w = exp(-i pi k / WH)
          auto both = [&](float2 zk, float2 zm, float2 w, int k) {
            zm.y = -zm.y;
            const float2 xe = cscale(cadd(zk, zm), 0.5f), xo = mul_i<-1>(cscale(csub(zk, zm), 0.5f)), x = cmul(w, xo);
            out[k] = cadd(xe, x);
            out[WH - k] = cconj(csub(xe, x));
          };
          if (j) {
            static_for<R>([&](auto q_) {
              constexpr int q = decltype(q_)::value;
              both(a[q], b[R - 1 - q], mul_root<q, 2 * R, -1>(post[i]), j + q * NBL);
            });
          } else {  // butterflies 0 and NBL / 2 mirror themselves
            static_for<R / 2 + 1>([&](auto q_) {
              constexpr int q = decltype(q_)::value;
              both(a[q], a[(R - q) % R], mul_root<q, 2 * R, -1>(make_float2(1.f, 0.f)), q * NBL);
            });
            static_for<(R + 1) / 2>([&](auto q_) {
              constexpr int q = decltype(q_)::value;
              both(b[q], b[R - 1 - q], mul_root<2 * q + 1, 4 * R, -1>(make_float2(1.f, 0.f)), NBL / 2 + q * NBL);
            });
          }
        }
      }
    }
    if (active)
      for (int k = WH + 1 + t; k < Wcp; k += NT) out[k] = make_float2(0.f, 0.f);
    __syncthreads();  // z is read
  }
}

template <class C>
int pad_rfft_reg_t(const float* proj, const double* rowstats, int h, int norm_h, int norm_w, int Wcp, int n_c, void* A,
                   cudaStream_t s, bool norm_ready) {
  if (cudaFuncSetAttribute(pad_rfft_reg_kernel<C>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM) !=
      cudaSuccess)
    return LGB_ERR_CUDA;
  // rows that share a CTA's tables: up to 32, as long as six CTAs per SM are left
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  int per = 32;
  while (per > C::ROWS && (long long)((h + per - 1) / per) * n_c < 6LL * sms) per /= 2;
  const int ctas = (h + per - 1) / per;
  // the constants: a grid of one wave reduces the rows itself in each CTA (2 us of
  // FP64 latency, the extra kernel takes 3.5); more CTAs would queue for the FP64 pipe
  if (!norm_ready && (long long)ctas * n_c > 6LL * sms) {
    const int st = launch_norm_constants(const_cast<double*>(rowstats), n_c, h, norm_h, norm_w, s);
    if (st) return st;
    norm_ready = true;
  }
  return launch_chained(pad_rfft_reg_kernel<C>, dim3(ctas, n_c), dim3(C::THREADS), C::SMEM, s, proj, rowstats, h,
                        NormSizes(h, norm_h, norm_w), Wcp, (int)norm_ready, per,
                        static_cast<float2*>(A));
}

}  // namespace lgb
