// Row pass of the search: c2r of length W = 2 WH through a WH-point complex
// transform in three passes (the pre-twiddle X[k], conj X[WH-k] -> Z[k] applied
// while the first one loads the staged row), ROWS rows per CTA, and the fused
// statistics: maximum, its correlogram, sum and sum of squares of a thread's
// pixels stay in registers over the batch, and the maps are read and written
// once per batch.  A value is scaled before it enters them: the sum of squares
// then holds whatever the correlogram itself can hold (unscaled it overflowed
// H W times earlier), and values that tie once scaled tie within a batch as
// between two (4096 x 4096: 23.63 us a correlogram unscaled, 24.07 with two
// multiplications a pair, 23.66 with a packed one).  A CTA takes row after row: its roots are built once, and the
// next row's first data come in under the map update.  Rows are staged with
// cp.async (completion by wait_group, no spins).
//
// Why 16 points per thread in three passes: four passes of 8 (256 threads a
// row) moved 92 B of shared memory and issued 98 instructions a point, and both
// pipes were two thirds busy; three passes move 70 B and issue 77.  Fewer, fatter
// threads (128 of 168 registers, three CTAs per SM) still fill both to two
// thirds.  Measured, microseconds per correlogram before -> now (before: the
// four-pass form at 4096, 2048, 5760 and 512, a generic table kernel elsewhere):
//   4096 x 4096 29.0 -> 23.9 (48 in a batch), 34.9 -> 32.4 (12), 188 -> 194 (1)
//   2048 x 2048 8.5 -> 6.1 (48)    1024 x 1024 7.6 -> 1.7 (96)    512 x 512 1.21 -> 1.10 (32)
//   3840 x 3840 58 -> 25 (24)      3072 x 3072 53 -> 17 (24)      2880 x 2880 50 -> 16 (24)
//   5760 wide x 4096 71 -> 52 (24; 105 registers of statistics spill)
// Two correlograms in one full-length transform measured 25.4 at 4096 and would
// tie a correlogram's rounding to its partner; two passes of 64 points with the
// statistics in tensor memory measured 30.0.
#pragma once

#include "match_kernels.cuh"
#include "reg_dft.cuh"

namespace lgb {

// SPLIT > 1: a CTA has one row and shares its correlograms out to SPLIT groups
// of NT threads, whose statistics meet in shared memory.
template <int WH_, int NT_, int ROWS_, class RL_, int MINB_, int SPLIT_ = 1>
struct RowHalf {
  using RL = RL_;
  static constexpr int WH = WH_, NT = NT_, ROWS = ROWS_, MINB = MINB_, SPLIT = SPLIT_;
  static_assert(SPLIT == 1 || ROWS == 1, "one row per CTA where it is split");
  static constexpr int THREADS = NT * ROWS * SPLIT;
  static constexpr int R1 = Head<RL>::value, RLAST = Last<RL>::value;
  static constexpr int NB1 = WH / R1, PER1 = (NB1 + NT - 1) / NT;
  static constexpr int NBL = WH / RLAST, PERL = (NBL + NT - 1) / NT;
  static constexpr int PX = PERL * RLAST;                   // complex outputs (pixel pairs) per thread
  static constexpr int WCP = (WH + 1 + 3) / 4 * 4;          // row stride of Y
  static constexpr int ZS = (IdxPad16::pad(WH) + 2) / 2 * 2;
  static constexpr int TAB = TableSize<1, RL>::value;
  static constexpr size_t SMEM = sizeof(float2) * ((size_t)ROWS * SPLIT * (WCP + ZS) + TAB);
  // a group's statistics pass through its own rows, sums after maxima
  static_assert(SPLIT == 1 || 2 * (WCP + ZS) >= 4 * PX * NT, "room for the statistics");
};

template <class C>
__global__ void __launch_bounds__(C::THREADS, C::MINB)
    rowpass_half_kernel(const float2* __restrict__ Y, int y_rows, int n_c, int nb, int n_orient, int o0,
                        const int* __restrict__ o0_dev, float scale, float* __restrict__ mip, int* __restrict__ best,
                        double* __restrict__ s1, double* __restrict__ s2) {
  using RL = typename C::RL;
  constexpr int WH = C::WH, NT = C::NT, ROWS = C::ROWS, R1 = C::R1, RLAST = C::RLAST, NB1 = C::NB1, NBL = C::NBL,
                PERL = C::PERL, PER1 = C::PER1, PX = C::PX;
  extern __shared__ float2 rhsm[];
  constexpr int SPLIT = C::SPLIT, SLOTS = ROWS * SPLIT;
  const int slot = SLOTS == 1 ? 0 : threadIdx.x / NT, t = SLOTS == 1 ? threadIdx.x : threadIdx.x - slot * NT;
  const int g = SPLIT == 1 ? slot : 0, part = SPLIT == 1 ? 0 : slot;
  float2* xs = rhsm + slot * (C::WCP + C::ZS);
  float2* z = xs + C::WCP;
  float2* tab = rhsm + SLOTS * (C::WCP + C::ZS);
  // this group's correlograms
  const int per = SPLIT == 1 ? n_c : (n_c + SPLIT - 1) / SPLIT, c0 = SPLIT == 1 ? 0 : part * per;
  // row y of correlogram c -> xs, 16 bytes a copy
  auto stage = [&](int y, int c) {
    if (y < y_rows && (SPLIT == 1 || c < n_c)) {
      const float2* src = Y + ((size_t)c * y_rows + y) * C::WCP;
      for (int i = t; i < C::WCP / 2; i += NT) cp_async16(xs + 2 * i, src + 2 * i);
    }
    cp_async_commit();
  };
  FillTables<WH, 1, RL>::run(tab, threadIdx.x, C::THREADS);
  // c2r pre-twiddle exp(+i pi k / WH) at k = j + q NB1: exp(i pi j / WH), kept
  // in registers, times the constant exp(i pi q / R1)
  float2 prej[PER1];
#pragma unroll
  for (int p = 0; p < PER1; ++p) {
    float sn, cs;
    sincospif((float)(t + p * NT) / (float)WH, &sn, &cs);
    prej[p] = make_float2(cs, sn);
  }
  const float2* tab_last = tab + TableSize<1, typename DropLast<RL>::type>::value;
  chain_wait();
  LGB_CHAIN_POINTER(Y);
  LGB_CHAIN_POINTER(o0_dev);
  LGB_CHAIN_POINTER(mip);
  LGB_CHAIN_POINTER(best);
  LGB_CHAIN_POINTER(s1);
  LGB_CHAIN_POINTER(s2);
  stage(blockIdx.x * ROWS + g, c0);
  if (o0_dev) o0 += *o0_dev;
#pragma unroll 1
  for (int y0 = blockIdx.x * ROWS; y0 < y_rows; y0 += gridDim.x * ROWS) {
    const int y = y0 + g;
    float top[2 * PX], sm[2 * PX], sq[2 * PX];
    unsigned arg[PX];  // batch index of a pixel pair's maxima: low / high 16 bits
#pragma unroll
    for (int i = 0; i < 2 * PX; ++i) {
      top[i] = -INFINITY;
      sm[i] = sq[i] = 0.f;
    }
#pragma unroll
    for (int i = 0; i < PX; ++i) arg[i] = 0u;
#pragma unroll 1
    for (int c = c0; c < c0 + per; ++c) {
      cp_async_wait<0>();
      __syncthreads();
#pragma unroll
      for (int p = 0; p < PER1; ++p) {
        const int j = t + p * NT;
        if (NB1 % NT == 0 || j < NB1) {
          float2 u[R1];
          static_for<R1>([&](auto q_) {
            constexpr int q = decltype(q_)::value;
            const int k = j + q * NB1;
            float2 a = xs[k], b = xs[WH - k];
            if (q == 0 && j == 0) a.y = b.y = 0.f;  // DC and Nyquist: real parts only
            b.y = -b.y;
            const float2 xo = mul_root<q, 2 * R1, +1>(cmul(csub(a, b), prej[p]));
            u[q] = cadd(cadd(a, b), mul_i<1>(xo));
          });
          Dft<R1, +1>::run(u);
#pragma unroll
          for (int q = 0; q < R1; ++q) z[IdxPad16::f(j * R1 + q)] = u[q];
        }
      }
      __syncthreads();
      // the staged row is read: the next one comes in during the other passes
      if (c + 1 < c0 + per)
        stage(y, c + 1);
      else if (SPLIT == 1 && y0 + gridDim.x * ROWS < y_rows)
        stage(y + gridDim.x * ROWS, c0);
      TablePasses<WH, NT, +1, IdxPad16, R1, typename Middle<RL>::type>::run(z, tab, t);
#pragma unroll
      for (int p = 0; p < PERL; ++p) {
        const int j = t + p * NT;
        if ((NBL == PERL * NT || j < NBL) && (SPLIT == 1 || c < n_c)) {
          float2 v[RLAST];
          const int fj = IdxPad16::f(j);
#pragma unroll
          for (int q = 0; q < RLAST; ++q) v[q] = z[padded_at<IdxPad16, NBL>(fj, j, q)];
          twiddle_from_table<RLAST, +1, NBL>(v, tab_last, j);
          Dft<RLAST, +1>::run(v);
#pragma unroll
          for (int q = 0; q < RLAST; ++q) {
            const int k = p * RLAST + q;
            const float2 ab = cscale_packed(v[q], scale);
            const float a = ab.x, b = ab.y;
            if (a > top[2 * k]) {
              top[2 * k] = a;
              arg[k] = (arg[k] & 0xffff0000u) | (unsigned)c;
            }
            if (b > top[2 * k + 1]) {
              top[2 * k + 1] = b;
              arg[k] = (arg[k] & 0xffffu) | ((unsigned)c << 16);
            }
            sm[2 * k] += a;
            sq[2 * k] = fmaf(a, a, sq[2 * k]);
            sm[2 * k + 1] += b;
            sq[2 * k + 1] = fmaf(b, b, sq[2 * k + 1]);
          }
        }
      }
    }
    // ---- the groups' statistics, in the order of their correlograms (a tie goes to the first)
    if constexpr (SPLIT > 1) {
      float* mine = reinterpret_cast<float*>(xs);
      __syncthreads();
      if (part) {
#pragma unroll
        for (int i = 0; i < 2 * PX; ++i) mine[i * NT + t] = top[i];
#pragma unroll
        for (int i = 0; i < PX; ++i) mine[(2 * PX + i) * NT + t] = __uint_as_float(arg[i]);
      }
      __syncthreads();
      if (!part) {
#pragma unroll 1
        for (int o = 1; o < SPLIT; ++o) {
          const float* other = mine + o * 2 * (C::WCP + C::ZS);
#pragma unroll
          for (int i = 0; i < PX; ++i) {
            const float a = other[2 * i * NT + t], b = other[(2 * i + 1) * NT + t];
            const unsigned at = __float_as_uint(other[(2 * PX + i) * NT + t]);
            if (a > top[2 * i]) {
              top[2 * i] = a;
              arg[i] = (arg[i] & 0xffff0000u) | (at & 0xffffu);
            }
            if (b > top[2 * i + 1]) {
              top[2 * i + 1] = b;
              arg[i] = (arg[i] & 0xffffu) | (at & 0xffff0000u);
            }
          }
        }
      }
      __syncthreads();
      if (part) {
#pragma unroll
        for (int i = 0; i < 2 * PX; ++i) {
          mine[i * NT + t] = sm[i];
          mine[(2 * PX + i) * NT + t] = sq[i];
        }
      }
      __syncthreads();
      if (!part) {
#pragma unroll 1
        for (int o = 1; o < SPLIT; ++o) {
          const float* other = mine + o * 2 * (C::WCP + C::ZS);
#pragma unroll
          for (int i = 0; i < 2 * PX; ++i) {
            sm[i] += other[i * NT + t];
            sq[i] += other[(2 * PX + i) * NT + t];
          }
        }
      }
      if (y0 + gridDim.x < y_rows) {  // the next row's first data
        __syncthreads();
        stage(y + gridDim.x, c0);
      }
    }
    // ---- one read-modify-write of the maps
    if (y < y_rows && !part) {
#pragma unroll
      for (int p = 0; p < PERL; ++p) {
        const int j = t + p * NT;
        if (NBL == PERL * NT || j < NBL) {
          const size_t base = (size_t)y * (2 * WH) + 2 * j;
          float2 m[RLAST];
          int2 bi[RLAST];
          double2 d[RLAST];
#pragma unroll
          for (int q = 0; q < RLAST; ++q) {
            m[q] = *reinterpret_cast<const float2*>(mip + base + 2 * NBL * q);
            bi[q] = *reinterpret_cast<const int2*>(best + base + 2 * NBL * q);
            d[q] = *reinterpret_cast<const double2*>(s1 + base + 2 * NBL * q);
          }
#pragma unroll
          for (int q = 0; q < RLAST; ++q) {
            const int k = p * RLAST + q;
            const float a = top[2 * k], b = top[2 * k + 1];
            if (a > m[q].x) {
              m[q].x = a;
              const int cc = (int)(arg[k] & 0xffffu);
              bi[q].x = (cc / nb) * n_orient + o0 + (cc - (cc / nb) * nb);
            }
            if (b > m[q].y) {
              m[q].y = b;
              const int cc = (int)(arg[k] >> 16);
              bi[q].y = (cc / nb) * n_orient + o0 + (cc - (cc / nb) * nb);
            }
            d[q].x += f2d_bits(sm[2 * k]);
            d[q].y += f2d_bits(sm[2 * k + 1]);
            *reinterpret_cast<float2*>(mip + base + 2 * NBL * q) = m[q];
            *reinterpret_cast<int2*>(best + base + 2 * NBL * q) = bi[q];
            *reinterpret_cast<double2*>(s1 + base + 2 * NBL * q) = d[q];
          }
#pragma unroll
          for (int q = 0; q < RLAST; ++q) d[q] = *reinterpret_cast<const double2*>(s2 + base + 2 * NBL * q);
#pragma unroll
          for (int q = 0; q < RLAST; ++q) {
            const int k = p * RLAST + q;
            d[q].x += f2d_bits(sq[2 * k]);
            d[q].y += f2d_bits(sq[2 * k + 1]);
            *reinterpret_cast<double2*>(s2 + base + 2 * NBL * q) = d[q];
          }
        }
      }
    }
  }
}

template <class C>
int rowpass_half_launch(const void* Y, int H, int y_rows, int n_c, int nb, int n_orient, int o0, const int* o0_dev,
                        float* mip, int* best, double* s1, double* s2, int sms, cudaStream_t s) {
  if (cudaFuncSetAttribute(rowpass_half_kernel<C>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM) !=
          cudaSuccess ||
      cudaFuncSetAttribute(rowpass_half_kernel<C>, cudaFuncAttributePreferredSharedMemoryCarveout,
                           cudaSharedmemCarveoutMaxShared) != cudaSuccess)
    return LGB_ERR_CUDA;
  const float scale = 1.0f / ((float)H * (float)(2 * C::WH));
  const int groups = (y_rows + C::ROWS - 1) / C::ROWS, ctas = sms * C::MINB;
  return launch_chained(rowpass_half_kernel<C>, dim3(groups < ctas ? groups : ctas), dim3(C::THREADS), C::SMEM, s,
                        static_cast<const float2*>(Y), y_rows, n_c, nb, n_orient, o0, o0_dev, scale, mip, best, s1, s2);
}

// C, or the first of the SPLIT forms in Cs (most groups first) whose rows are
// all resident at once and whose groups have two correlograms or more (one each
// measured no better).
template <class C, class... Cs>
int rowpass_half_t(const void* Y, int H, int y_rows, int Wcp, int n_c, int nb, int n_orient, int o0,
                   const int* o0_dev, float* mip, int* best, double* s1, double* s2, cudaStream_t s) {
  if (Wcp != C::WCP) return LGB_ERR_INVALID_ARGUMENT;
  if (n_c > 0xffff) return LGB_ERR_INVALID_ARGUMENT;  // batch indices are kept in 16 bits
  int dev = 0, sms = 0, st = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const bool done = ((y_rows <= sms * Cs::MINB && n_c >= 2 * Cs::SPLIT &&
                      (st = rowpass_half_launch<Cs>(Y, H, y_rows, n_c, nb, n_orient, o0, o0_dev, mip, best, s1, s2, sms,
                                                    s),
                       true)) ||
                     ...);
  if (done) return st;
  return rowpass_half_launch<C>(Y, H, y_rows, n_c, nb, n_orient, o0, o0_dev, mip, best, s1, s2, sms, s);
}

}  // namespace lgb
