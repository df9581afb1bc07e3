// Column pass of the search in two register passes per direction (H = R1 R2,
// up to 80 points of a column in one thread).
//
// Forward: radix R1 over rows b + R2 q (rows >= h are zero) -> shared
// transpose M1[b][q] -> roots w^(r b) -> radix R2, which leaves P[b + R1 r] in
// thread b.  The cross power with the image spectrum and the inverse's radix
// R2 over the same elements stay in registers -> shared transpose M2[b][r] ->
// conjugate roots w^(q b) -> inverse radix R1 -> rows b + R2 q of Y.
//
// A CTA keeps its G columns for a range of correlograms, so their part of the
// image spectrum is read from memory once per CTA and held in tensor memory
// (2 R2 columns per thread); the kernel issues no MMA.
//
// Why two passes: with three radix-16 passes per direction (one 16-point
// butterfly per thread) a point crossed shared memory four times and read its
// roots there, 94 B in all, and the image spectrum came from L2 for every
// correlogram; load, exchange and arithmetic phases of the one resident CTA
// followed each other.  Now it is 48 B and no re-read.  What is left is the
// FP32 arithmetic (74 operations a point, half of the FMA pipe's time at 8
// warps) and fetching the unrolled code; spreading the stores of Y over the
// next correlogram, packed FP32 adds, one shared code path for both directions
// and strip layouts of Y all measured no better.
// Microseconds per correlogram, before -> now (before: three radix-16 passes
// at 4096, the generic table kernel at the other lengths):
//   4096 x 2049, h 384: 41.6 -> 31.6    3840 x 1921, h 256: 84 -> 33.5
//   3072 x 1441, h 256: 40 -> 21        2880 x 1441, h 256: 64 -> 23
//   2048 x 1025, h 256: 18.1 -> 8.5     1024 x 513, h 128: 5.2 -> 2.0
//   576 x 289, h 128: 2.4 -> 0.7        5760 x 2049, h 256: 177 -> 70
// 5760 rows take ten warps of 168 registers and 150 KB of code in the loop, more
// than the instruction caches hold.  Their split 80 x 72 (the larger radix where
// no image and roots are held) spills 460 bytes and measured 70 us, 72 x 80 85;
// 64 x 90 in eight warps of 255 registers 122 (260 KB of code), three columns a
// CTA 165 (24-byte row pieces), both directions in one code path 73.
// A batch of one correlogram runs the whole code once, cold: 5760 x 257 takes 74 us
// where the generic kernel's few instructions took 35 (two correlograms 74
// against 62), 4096 x 257 8 us more than the radix-16 passes.  The kernel may not
// depend on the batch, or a correlogram's bits would.
#pragma once

#include "reg_dft.cuh"
#include "match_kernels.cuh"
#include "tmem.cuh"

namespace lgb {

// TWO: w^(r b) as a product of w^(r0 b) and w^(L r1 b), r = r0 + L r1 (L = R1B
// and R2B), for the length whose whole table does not fit beside its columns.
template <int R1A_, int R1B_, int R2A_, int R2B_, int NT_, int G_, int MINB_, bool TWO_ = false>
struct ColReg {
  static constexpr int R1A = R1A_, R1B = R1B_, R2A = R2A_, R2B = R2B_;
  static constexpr int R1 = R1A * R1B, R2 = R2A * R2B, N = R1 * R2;
  static constexpr int NT = NT_, G = G_, MINB = MINB_;
  static constexpr bool TWO = TWO_;
  static constexpr int D1 = (R2 + NT - 1) / NT;  // radix-R1 transforms per thread
  static_assert(NT >= R1, "one radix-R2 transform per thread at most");
  static constexpr int THREADS = (G * NT + 31) / 32 * 32;
  // odd row strides and a column stride of 16 / G (mod 16) float2 keep both
  // transposes conflict free for G columns x consecutive b per half-warp
  static constexpr int S1 = R1 | 1, S2 = R2 | 1;
  static constexpr int CB = R2 * S1 > R1 * S2 ? R2 * S1 : R1 * S2;
  static constexpr int STRIDE = CB + ((16 / G) - CB % 16 + 16) % 16;
  // root table: [r][b], row stride TS; two-level: [r0 | R2B r1][b < R1], then [q0 | R1B q1][b < R2]
  static constexpr int TS = R1 | 1;
  static constexpr int TAB = TWO ? (R2A + R2B) * R1 + (R1A + R1B) * R2 : R2 * TS;
  static constexpr size_t SMEM = sizeof(float2) * ((size_t)G * STRIDE + TAB);
  static constexpr int CH = R2 % 16 == 0 ? 16 : (R2 % 4 == 0 && R2 % 8 ? 4 : 8);  // complex values per tensor-memory access
  static constexpr int SLOTS = (R2 + CH - 1) / CH * CH;
  static constexpr int WORDS = 2 * SLOTS;  // tensor-memory columns per thread
  static constexpr int WPQ = (THREADS / 32 + 3) / 4;         // warps that share a lane quarter
  static constexpr int COLS_USED = WORDS * WPQ;
  static constexpr int COLS = COLS_USED <= 32    ? 32
                              : COLS_USED <= 64  ? 64
                              : COLS_USED <= 128 ? 128
                              : COLS_USED <= 256 ? 256
                                                 : 512;
  static_assert(COLS_USED <= 512 && COLS * MINB <= 512, "tensor memory holds every resident CTA's image columns");
};

// v[r] *= w^(r b) (DIR = -1) or its conjugate, from a whole table's entries
// tab[r step] (L = 0) or from the two levels lo[r0 step], hi[r1 step].
template <int R, int DIR, int L>
__device__ __forceinline__ void apply_roots(float2* v, const float2* tab, int step) {
  if constexpr (L == 0) {
#pragma unroll
    for (int r = 1; r < R; ++r) {
      const float2 w = tab[r * step];
      v[r] = DIR < 0 ? cmul(v[r], w) : cmulc(v[r], w);
    }
  } else {
    float2 lo[L];
#pragma unroll
    for (int r = 1; r < L; ++r) {
      lo[r] = tab[r * step];
      v[r] = DIR < 0 ? cmul(v[r], lo[r]) : cmulc(v[r], lo[r]);
    }
#pragma unroll
    for (int r1 = 1; r1 < R / L; ++r1) {
      const float2 hi = tab[(L + r1) * step];
#pragma unroll
      for (int r0 = 0; r0 < L; ++r0) {
        const float2 w = r0 ? cmul(hi, lo[r0]) : hi;
        v[L * r1 + r0] = DIR < 0 ? cmul(v[L * r1 + r0], w) : cmulc(v[L * r1 + r0], w);
      }
    }
  }
}

template <class C, bool SPARSE>
__global__ void __launch_bounds__(C::THREADS, C::MINB)
    colpass_reg_kernel(const float2* __restrict__ A, const float2* __restrict__ Ip, int ips, int h, int Wcp, int n_c,
                       int c_per_block, int c_per_image, int y_rows, float2* __restrict__ Y) {
  constexpr int R1 = C::R1, R2 = C::R2, N = C::N, G = C::G, NT = C::NT, D1 = C::D1, S1 = C::S1, S2 = C::S2;
  constexpr int CH = C::CH, SLOTS = C::SLOTS;
  // no thread idles in a pass: its guards are constant, which spares the loads' zero fills
  constexpr bool FULL1 = D1 * NT == R2 && G * NT == C::THREADS, FULL2 = NT == R1 && G * NT == C::THREADS;
  extern __shared__ float2 crsm[];
  __shared__ unsigned tm_slot;
  const int warp = threadIdx.x / 32;
  const int g = threadIdx.x % G, t = threadIdx.x / G;
  float2* x = crsm + g * C::STRIDE;
  float2* tab = crsm + G * C::STRIDE;
  if (warp == 0) tmem_alloc(&tm_slot, C::COLS);
  const int kx = blockIdx.x * G + g;
  const bool col_ok = kx < Wcp;
  const bool act2 = FULL2 || t < R1;  // holds a radix-R2 transform
  const int c_begin = blockIdx.y * c_per_block;
  const int c_end = min(n_c, c_begin + c_per_block);
  // sparse inputs of the coming correlogram, read one correlogram ahead
  constexpr int NZ = SPARSE ? C::R1B : 1;
  float2 nx[D1][NZ];
  auto fetch = [&](int c) {
    const float2* a = A + (size_t)c * h * Wcp + kx;
#pragma unroll
    for (int i = 0; i < D1; ++i) {
      const int b = t + NT * i;
#pragma unroll
      for (int q = 0; q < NZ; ++q)
        nx[i][q] = (col_ok && (FULL1 || (t < NT && b < R2)) && b + R2 * q < h)
                       ? __ldg(a + (size_t)(b + R2 * q) * Wcp)
                       : make_float2(0.f, 0.f);
    }
  };
  if constexpr (C::TWO) {
    auto fill = [&](float2* dst, int low, int high, int nb) {  // rows 0..low-1: r, then low (row - low)
      for (int e = threadIdx.x; e < (low + high) * nb; e += C::THREADS) {
        const int row = e / nb, b = e - (e / nb) * nb, r = row < low ? row : low * (row - low);
        float sn, cs;
        sincospif(2.0f * (float)(r * b) / (float)N, &sn, &cs);
        dst[e] = make_float2(cs, -sn);
      }
    };
    fill(tab, C::R2B, C::R2A, R1);
    fill(tab + (C::R2A + C::R2B) * R1, C::R1B, C::R1A, R2);
  } else {
    for (int e = threadIdx.x; e < R2 * R1; e += C::THREADS) {
      const int r = e / R1, b = e - (e / R1) * R1;
      float sn, cs;
      sincospif(2.0f * (float)(r * b) / (float)N, &sn, &cs);
      tab[r * C::TS + b] = make_float2(cs, -sn);
    }
  }
  chain_wait();
  LGB_CHAIN_POINTER(A);
  LGB_CHAIN_POINTER(Ip);
  LGB_CHAIN_POINTER(Y);
  if (SPARSE && c_begin < c_end) fetch(c_begin);
  int image = c_begin / c_per_image;
  float2 first[SLOTS];
  {
    const float2* ip = Ip + (size_t)image * N * ips + kx;
#pragma unroll
    for (int s = 0; s < SLOTS; ++s) {
      const int row = t + R1 * DftNT<C::R2A, C::R2B, -1>::out(s);
      first[s] = (s < R2 && kx < ips && act2 && c_begin < c_end) ? __ldg(ip + (size_t)row * ips) : make_float2(0.f, 0.f);
    }
  }
  tmem_barrier();
  const unsigned tm_base = tm_slot;
  const unsigned tm = tm_base + ((unsigned)(warp % 4) << 21) + (unsigned)(warp / 4) * C::WORDS;
#pragma unroll
  for (int s0 = 0; s0 < R2; s0 += CH) tmem_put<CH>(tm + 2 * s0, first + s0);
  tmem_wait_st();
  using FO = DftNT<C::R1A, C::R1B, +1>;
  const unsigned y_off = (unsigned)(t * Wcp + kx) * 8u, y_step = (unsigned)(R2 * Wcp) * 8u,
                 y_nt = (unsigned)(NT * Wcp) * 8u;
#pragma unroll 1
  for (int c = c_begin; c < c_end; ++c) {
    // ---- this image's columns -> tensor memory, in the slot order of P
    if (c / c_per_image != image) {
      image = c / c_per_image;
      const float2* ip = Ip + (size_t)image * N * ips + kx;
#pragma unroll
      for (int s0 = 0; s0 < R2; s0 += CH) {
        float2 w[CH];
#pragma unroll
        for (int i = 0; i < CH; ++i) {
          const int row = t + R1 * DftNT<C::R2A, C::R2B, -1>::out(s0 + i);
          w[i] = (s0 + i < R2 && kx < ips && act2) ? __ldg(ip + (size_t)row * ips) : make_float2(0.f, 0.f);
        }
        tmem_put<CH>(tm + 2 * s0, w);
      }
      tmem_wait_st();
    }
    // ---- forward radix R1 -> M1
#pragma unroll
    for (int i = 0; i < D1; ++i) {
      const int b = t + NT * i;
      const bool act1 = FULL1 || (t < NT && b < R2);
      float2 u[R1];
      if constexpr (SPARSE) {
#pragma unroll
        for (int q = 0; q < C::R1B; ++q) u[q] = nx[i][q];
      } else {
        const float2* a = A + (size_t)c * h * Wcp + kx;
#pragma unroll
        for (int q = 0; q < R1; ++q)
          u[q] = (col_ok && act1 && b + R2 * q < h) ? __ldg(a + (size_t)(b + R2 * q) * Wcp) : make_float2(0.f, 0.f);
      }
      using F = DftNT<C::R1A, C::R1B, -1, SPARSE>;
      F::run(u);
      if (i == 0) __syncthreads();  // the last correlogram's M2 is read
      if (act1) {
#pragma unroll
        for (int s = 0; s < R1; ++s) x[b * S1 + F::out(s)] = u[s];
      }
    }
    if (SPARSE && c + 1 < c_end) fetch(c + 1);
    __syncthreads();
    // ---- forward radix R2: slot s holds P[t + R1 out(s)]
    {
      float2 v[R2];
      // (an idle thread reads row 0's entries and stores nothing)
      const int tt = act2 ? t : 0;
#pragma unroll
      for (int r = 0; r < R2; ++r) v[r] = x[r * S1 + tt];
      apply_roots<R2, -1, C::TWO ? C::R2B : 0>(v, tab + tt, C::TWO ? R1 : C::TS);
      DftNT<C::R2A, C::R2B, -1>::run(v);
      // ---- cross power, P[0,0] = 0
#pragma unroll
      for (int s0 = 0; s0 < R2; s0 += CH) {
        float2 w[CH];
        tmem_get<CH>(tm + 2 * s0, w);
#pragma unroll
        for (int i = 0; i < CH; ++i)
          if (s0 + i < R2) v[s0 + i] = cmulc(w[i], v[s0 + i]);
      }
      if (t == 0 && kx == 0) v[0] = make_float2(0.f, 0.f);
      // ---- inverse radix R2 on the same elements: output r in slot r
      DftTN<C::R2B, C::R2A, +1>::run(v);
      __syncthreads();  // M1 is read
      if (act2) {
#pragma unroll
        for (int r = 0; r < R2; ++r) x[t * S2 + r] = v[r];
      }
    }
    __syncthreads();
    // ---- inverse radix R1: rows b + R2 out(s)
#pragma unroll
    for (int i = 0; i < D1; ++i) {
      const int b = t + NT * i;
      const bool act1 = FULL1 || (t < NT && b < R2);
      float2 u[R1];
      const int bb = act1 ? b : 0;
#pragma unroll
      for (int q = 0; q < R1; ++q) u[q] = x[q * S2 + bb];
      if constexpr (C::TWO)
        apply_roots<R1, +1, C::R1B>(u, tab + (C::R2A + C::R2B) * R1 + bb, R2);
      else
        apply_roots<R1, +1, 0>(u, tab + bb * C::TS, 1);
      FO::run(u);
      if (col_ok && act1) {
        char* yc = reinterpret_cast<char*>(Y + (size_t)c * y_rows * Wcp);  // 32-bit offsets from here: H Wcp 8 B < 2^32
        const unsigned off = y_off + i * y_nt;
        if (y_rows == N) {
#pragma unroll
          for (int s = 0; s < R1; ++s) *reinterpret_cast<float2*>(yc + (off + y_step * FO::out(s))) = u[s];
        } else {
#pragma unroll
          for (int s = 0; s < R1; ++s)
            if (b + R2 * FO::out(s) < y_rows) *reinterpret_cast<float2*>(yc + (off + y_step * FO::out(s))) = u[s];
        }
      }
    }
  }
  tmem_barrier();
  if (warp == 0) tmem_dealloc(tm_base, C::COLS);
}

// Correlograms per CTA for `groups` column groups over `slots` resident CTAs:
// the split whose rounds are cheapest, a CTA costing its correlograms plus
// about one more for its roots and image columns (4096 rows, 48 correlograms:
// 48 / 24 / 12 per CTA measured 33.8 / 31.9 / 32.4 us per correlogram).  A
// caller's `waves` asks for about waves x the SM count CTAs instead.
inline int colpass_per_block(int groups, int n_c, int sms, int per_sm, int waves) {
  if (waves > 0) {
    int split = 1;
    while (split < n_c && (long long)groups * split < (long long)waves * sms) split *= 2;
    if (split > n_c) split = n_c;
    return (n_c + split - 1) / split;
  }
  const int slots = sms * per_sm;
  int best = n_c;
  long long best_cost = -1;
  for (int split = 1; split <= n_c && split <= 64; ++split) {
    const int per = (n_c + split - 1) / split;
    const long long rounds = ((long long)groups * ((n_c + per - 1) / per) + slots - 1) / slots;
    const long long cost = rounds * (per + 1);
    if (best_cost < 0 || cost < best_cost) {
      best_cost = cost;
      best = per;
    }
  }
  return best;
}

template <class C, bool SPARSE>
int colpass_reg_launch(const void* A, const void* Ip, int ips, int h, int Wcp, int n_c, int cpi, int y_rows, int waves, void* Y,
                       cudaStream_t s) {
  if (cudaFuncSetAttribute(colpass_reg_kernel<C, SPARSE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)C::SMEM) != cudaSuccess)
    return LGB_ERR_CUDA;
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int groups = (Wcp + C::G - 1) / C::G;
  const int per = colpass_per_block(groups, n_c, sms, C::MINB, waves);
  return launch_chained(colpass_reg_kernel<C, SPARSE>, dim3(groups, (n_c + per - 1) / per), dim3(C::THREADS), C::SMEM, s,
                        static_cast<const float2*>(A), static_cast<const float2*>(Ip), ips, h, Wcp, n_c, per, cpi,
                        y_rows, static_cast<float2*>(Y));
}

// The sparse form reads inputs q < R1B only: rows h <= R1B R2.  The first split
// in Cs (the fastest first) that covers h, else the dense form of the last one;
// templates have at most kMaxTemplate rows.
constexpr int kMaxTemplate = 512;
template <class C, class... Cs>
int colpass_reg_t(const void* A, const void* Ip, int ips, int h, int Wcp, int n_c, int cpi, int y_rows, int waves,
                  void* Y, cudaStream_t s) {
  if (h > kMaxTemplate) return LGB_ERR_UNSUPPORTED_SIZE;
  if constexpr (C::R1B * C::R2 < kMaxTemplate) {
    if (h > C::R1B * C::R2) {
      if constexpr (sizeof...(Cs) > 0)
        return colpass_reg_t<Cs...>(A, Ip, ips, h, Wcp, n_c, cpi, y_rows, waves, Y, s);
      else
        return colpass_reg_launch<C, false>(A, Ip, ips, h, Wcp, n_c, cpi, y_rows, waves, Y, s);
    }
  }
  return colpass_reg_launch<C, true>(A, Ip, ips, h, Wcp, n_c, cpi, y_rows, waves, Y, s);
}

}  // namespace lgb
