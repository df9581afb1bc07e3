// Composite DFTs held in one thread's registers (R = RA * RB up to 80) with
// compile-time roots, for the two-pass transforms of match_cols_reg.cuh and
// match_rows_half.cuh.
//
// A long transform in two register passes exchanges its data once through
// shared memory instead of two or three times; what bounds the passes is then
// the FP32 pipe instead of the shared-memory data path.  The roots inside a
// composite are literals of the code, so they cost neither registers nor
// loads.
#pragma once

#include <utility>

#include "fft.cuh"

namespace lgb {

// ---- compile-time roots ------------------------------------------------------
// exp(2 pi i k / n): the angle is reduced to one octant, where the Taylor
// series of sine and cosine converge to double precision.
constexpr double series_sin(double x) {
  double term = x, sum = x;
  for (int i = 1; i < 12; ++i) {
    term *= -x * x / ((2.0 * i) * (2.0 * i + 1.0));
    sum += term;
  }
  return sum;
}
constexpr double series_cos(double x) {
  double term = 1.0, sum = 1.0;
  for (int i = 1; i < 12; ++i) {
    term *= -x * x / ((2.0 * i - 1.0) * (2.0 * i));
    sum += term;
  }
  return sum;
}
constexpr double root_part(int k, int n, bool sine) {
  k = ((k % n) + n) % n;
  const int oct = (8 * k) / n;
  const double pi4 = 0.78539816339744830962;
  const double phi = pi4 * (double)(8 * k - oct * n) / (double)n;  // in [0, pi/4)
  const int quarter = (oct + 1) / 2;
  const double a = oct % 2 ? pi4 - phi : phi;
  const double c = series_cos(a), s = oct % 2 ? -series_sin(a) : series_sin(a);
  switch (quarter % 4) {
    case 0:
      return sine ? s : c;
    case 1:
      return sine ? c : -s;
    case 2:
      return sine ? -s : -c;
    default:
      return sine ? -c : s;
  }
}

template <int K, int N>
struct Root {
  static constexpr float c = (float)root_part(K, N, false);
  static constexpr float s = (float)root_part(K, N, true);
};

template <int... I, class F>
__device__ __forceinline__ void static_for_impl(std::integer_sequence<int, I...>, F&& f) {
  (f(std::integral_constant<int, I>{}), ...);
}
// f(integral_constant<0>) ... f(integral_constant<N-1>)
template <int N, class F>
__device__ __forceinline__ void static_for(F&& f) {
  static_for_impl(std::make_integer_sequence<int, N>{}, static_cast<F&&>(f));
}

// a * exp(DIR 2 pi i K / N)
template <int K, int N, int DIR>
__device__ __forceinline__ float2 mul_root(float2 a) {
  constexpr int k = ((K % N) + N) % N;
  if constexpr (k == 0) {
    return a;
  } else if constexpr (4 * k == N) {
    return mul_i<DIR>(a);
  } else if constexpr (2 * k == N) {
    return make_float2(-a.x, -a.y);
  } else if constexpr (4 * k == 3 * N) {
    return mul_i<-DIR>(a);
  } else {
    constexpr float c = Root<k, N>::c, s = DIR > 0 ? Root<k, N>::s : -Root<k, N>::s;
    return make_float2(fmaf(a.x, c, -a.y * s), fmaf(a.y, c, a.x * s));
  }
}

// Prime-factor (Good-Thomas) 3 x 5: input n = (5 n1 + 3 n2) mod 15, output
// k = (10 k1 + 6 k2) mod 15 (10 = 1 mod 3 and 0 mod 5, 6 = 0 mod 3 and 1 mod 5).
template <int DIR>
struct Dft<15, DIR> {
  static __device__ __forceinline__ void run(float2* v) {
    float2 u[3][5];
#pragma unroll
    for (int n1 = 0; n1 < 3; ++n1) {
#pragma unroll
      for (int n2 = 0; n2 < 5; ++n2) u[n1][n2] = v[(5 * n1 + 3 * n2) % 15];
      Dft<5, DIR>::run(u[n1]);
    }
#pragma unroll
    for (int k2 = 0; k2 < 5; ++k2) {
      float2 t[3] = {u[0][k2], u[1][k2], u[2][k2]};
      Dft<3, DIR>::run(t);
#pragma unroll
      for (int k1 = 0; k1 < 3; ++k1) v[(10 * k1 + 6 * k2) % 15] = t[k1];
    }
  }
};

// Prime-factor 2 x 5: input n = (5 n1 + 2 n2) mod 10, output k = (5 k1 + 6 k2) mod 10.
template <int DIR>
struct Dft<10, DIR> {
  static __device__ __forceinline__ void run(float2* v) {
    float2 a[5], b[5];
#pragma unroll
    for (int n2 = 0; n2 < 5; ++n2) {
      const float2 x0 = v[(2 * n2) % 10], x1 = v[(5 + 2 * n2) % 10];
      a[n2] = cadd(x0, x1);
      b[n2] = csub(x0, x1);
    }
    Dft<5, DIR>::run(a);
    Dft<5, DIR>::run(b);
#pragma unroll
    for (int k2 = 0; k2 < 5; ++k2) {
      v[(6 * k2) % 10] = a[k2];
      v[(5 + 6 * k2) % 10] = b[k2];
    }
  }
};

// Prime-factor 3 x 4: input n = (4 n1 + 3 n2) mod 12, output k = (4 k1 + 9 k2) mod 12.
template <int DIR>
struct Dft<12, DIR> {
  static __device__ __forceinline__ void run(float2* v) {
    float2 u[3][4];
#pragma unroll
    for (int n1 = 0; n1 < 3; ++n1) {
#pragma unroll
      for (int n2 = 0; n2 < 4; ++n2) u[n1][n2] = v[(4 * n1 + 3 * n2) % 12];
      Dft<4, DIR>::run(u[n1]);
    }
#pragma unroll
    for (int k2 = 0; k2 < 4; ++k2) {
      float2 t[3] = {u[0][k2], u[1][k2], u[2][k2]};
      Dft<3, DIR>::run(t);
#pragma unroll
      for (int k1 = 0; k1 < 3; ++k1) v[(4 * k1 + 9 * k2) % 12] = t[k1];
    }
  }
};

// ---- composite DFT of RA * RB points -----------------------------------------
// RA-point transforms over qa, roots w^(qb ra), RB-point transforms over qb;
// output r = ra + RA rb.  NT: input q = qa RB + qb in slot q, output r in slot
// ra RB + rb.  TN: input q in slot qb RA + qa, output r in slot r; it takes
// what an NT of RB * RA left behind.  SPARSE (NT): inputs q >= RB are zero and
// are not read; the RA-point transforms are then copies.
template <int RA, int RB, int DIR, bool SPARSE = false>
struct DftNT {
  static constexpr int R = RA * RB;
  // output index held by slot s
  __host__ __device__ static constexpr int out(int s) { return s / RB + RA * (s % RB); }
  static __device__ __forceinline__ void run(float2* v) {
    static_for<RB>([&](auto qb_) {
      constexpr int qb = decltype(qb_)::value;
      float2 t[RA];
      if constexpr (SPARSE) {
#pragma unroll
        for (int a = 0; a < RA; ++a) t[a] = v[qb];
      } else {
#pragma unroll
        for (int a = 0; a < RA; ++a) t[a] = v[a * RB + qb];
        Dft<RA, DIR>::run(t);
      }
      static_for<RA>([&](auto ra_) {
        constexpr int ra = decltype(ra_)::value;
        v[ra * RB + qb] = mul_root<qb * ra, R, DIR>(t[ra]);
      });
    });
    static_for<RA>([&](auto ra_) {
      constexpr int ra = decltype(ra_)::value;
      Dft<RB, DIR>::run(v + ra * RB);
    });
  }
};

template <int RA, int RB, int DIR>
struct DftTN {
  static constexpr int R = RA * RB;
  static __device__ __forceinline__ void run(float2* v) {
    static_for<RB>([&](auto qb_) {
      constexpr int qb = decltype(qb_)::value;
      Dft<RA, DIR>::run(v + qb * RA);
      static_for<RA>([&](auto ra_) {
        constexpr int ra = decltype(ra_)::value;
        v[qb * RA + ra] = mul_root<qb * ra, R, DIR>(v[qb * RA + ra]);
      });
    });
    static_for<RA>([&](auto ra_) {
      constexpr int ra = decltype(ra_)::value;
      float2 t[RB];
#pragma unroll
      for (int b = 0; b < RB; ++b) t[b] = v[b * RA + ra];
      Dft<RB, DIR>::run(t);
#pragma unroll
      for (int b = 0; b < RB; ++b) v[b * RA + ra] = t[b];
    });
  }
};

}  // namespace lgb
