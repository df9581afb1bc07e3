// Convolutions and linear layers of the proposal network on the tensor cores:
// each pass is a GEMM (for the 3x3 convolutions an implicit GEMM) run by the
// tcgen05 GEMM of tc_gemm.cuh (BF16 operands, FP32 accumulation in TMEM), with
// gather kernels that write the operands directly in the GEMM's blocked
// core-matrix layout and epilogues that scatter the accumulator to the
// network's NCHW / [N][features] tensors.
//
//   forward      y[p][co]   = sum_k  im2col(x)[p][k] * w[co][k]        k = ci*9 + tap
//   input grad   dx[q][ci]  = sum_k' col(g)[q][k'] * wT[ci][k']        k' = co*9 + tap
//   weight grad  dw[co][k]  = sum_p  im2col(x)[p][k] * g[p][co]        as [k][co], split over p, atomic adds
//
// p runs over output pixels (n, oy, ox), q over input pixels (n, iy, ix).  The
// linear layers run the same three products with x [N][In], w [Out][In], in
// transposed form (outputs as rows) so the epilogue's stores are coalesced.  The
// output gradient g (FP32) enters the tensor cores rounded to BF16, like the
// activations; accumulation stays FP32.  The bias gradient is one more column
// of the weight-gradient GEMM (a row of ones in its operand).  No reference
// counterpart (Leopard-EM has no learned component).
#include <cuda_bf16.h>

#include <type_traits>

#include "tc_gemm.cuh"

namespace lgb {

using bf16t = __nv_bfloat16;

struct ConvShape {
  int N, Cin, H, W, Cout, s, Ho, Wo;
  int P, Q, K, Kt;  // output pixels, input pixels, Cin*9, Cout*9 (P, Q < 2^23: checked by the entry points)
};

static ConvShape conv_shape(int N, int Cin, int H, int W, int Cout, int s) {
  ConvShape c{N, Cin, H, W, Cout, s, (H - 1) / s + 1, (W - 1) / s + 1, 0, 0, 0, 0};
  c.P = N * c.Ho * c.Wo;
  c.Q = N * H * W;
  c.K = Cin * 9;
  c.Kt = Cout * 9;
  return c;
}

__host__ __device__ constexpr int round_up(int a, int b) { return (a + b - 1) / b * b; }

// N tile (B rows per CTA) for a GEMM N extent: 32, 64 or 128 (TMEM columns are a power of two)
static int bn_for(int n) { return n <= 32 ? 32 : (n <= 64 ? 64 : 128); }

// ---- operand writers: 8 consecutive K elements (one 16-byte core-matrix row) per thread ----
__device__ __forceinline__ void store8(uint16_t* dst, const float* v) {
  uint4 u;
  uint16_t* h = reinterpret_cast<uint16_t*>(&u);
#pragma unroll
  for (int e = 0; e < 8; ++e) h[e] = __bfloat16_as_ushort(__float2bfloat16_rn(v[e]));
  *reinterpret_cast<uint4*>(dst) = u;
}

// Threads walk the operand in its memory order, one 16-byte unit (8 K values of
// one row) each, so the stores are fully coalesced: unit u of a blocked operand
// with TR-row tiles and KC chunks holds row r, K elements [k0, k0 + 8).
__device__ __forceinline__ void unit_rk(long long u, int TR, int KC, int& r, int& k0) {
  // (TR is a power of two, and operands have fewer than 2^32 groups of 64 units)
  const int r8 = (int)(u & 7), kg = (int)((u >> 3) & 7);
  const unsigned rest = (unsigned)(u >> 6), rg = rest & (unsigned)(TR / 8 - 1);
  const unsigned tc = rest >> (31 - __clz(TR / 8)), tile = tc / (unsigned)KC;
  r = (int)(tile * TR + rg * 8 + r8);
  k0 = (int)((tc - tile * KC) * kTcKC + kg * 8);
}

__device__ __forceinline__ void store8_bits(uint16_t* dst, const uint16_t* v) {
  uint4 u;
  uint16_t* h = reinterpret_cast<uint16_t*>(&u);
#pragma unroll
  for (int e = 0; e < 8; ++e) h[e] = v[e];
  *reinterpret_cast<uint4*>(dst) = u;
}

// What bounds the gathers is integer arithmetic (its pipe runs at half the FP32
// rate) unless positions are divided out once for many elements and the stride
// is a template argument; a run-time stride and per-element divisions cost 256
// samples of the network's step 1,648 us in gcol and 762 us in im2col, units of
// eight elements with stepped positions 580 and 390, this 193 and 185 (gcol of
// stride-2 layers again: gcol_pairs_kernel).
//
// A row's 72 consecutive K elements are the 9 taps of 8 channels: one thread
// takes them (nine 16-byte units), its taps at compile time, its position and
// the taps that fall inside found once.  A warp has 32 consecutive rows, so its
// sources are neighbours in the image and its stores whole 128-byte lines.
// pick(t, offset) gives tap t's offset in a channel plane, or false.
template <class T, class Pick>
__device__ __forceinline__ void gather_taps(long long e, int rows_pad, int TR, int k_pad, int channels, int plane_size,
                                            const T* __restrict__ src, Pick pick, uint16_t* __restrict__ out) {
  const int KC = k_pad / kTcKC, units = k_pad / 8;
  const int r = (int)(e % rows_pad), group = (int)(e / rows_pad);
  int off[9];
  unsigned in = 0;
  const size_t first = pick(r, off, in);  // channel 0 of the row's image
  const T* plane = src + first + (size_t)group * 8 * plane_size;
  uint16_t v[72];
#pragma unroll
  for (int ch = 0; ch < 8; ++ch) {
    const bool ok = group * 8 + ch < channels;
#pragma unroll
    for (int t = 0; t < 9; ++t) {
      if constexpr (sizeof(T) == 2) {
        v[ch * 9 + t] = (ok && (in >> t & 1u)) ? (uint16_t)plane[off[t]] : (uint16_t)0;
      } else {
        v[ch * 9 + t] = __bfloat16_as_ushort(__float2bfloat16_rn((ok && (in >> t & 1u)) ? plane[off[t]] : 0.f));
      }
    }
    plane += plane_size;
  }
  const int tile = r / TR, rl = r - tile * TR;
#pragma unroll
  for (int u = 0; u < 9; ++u) {
    const int ku = group * 9 + u;
    if (ku < units) {
      const size_t unit = ((size_t)tile * KC + ku / 8) * (TR * 8) + (rl / 8) * 64 + (ku % 8) * 8 + rl % 8;
      store8_bits(out + unit * 8, v + u * 8);
    }
  }
}
__host__ __device__ constexpr int tap_groups(int k_pad) { return (k_pad / 8 + 8) / 9; }

// A of the forward: im2col(x) [rows p][k = ci*9+tap], rows padded to TR, K
// padded to 64 (zeros).
template <int S>
__global__ void __launch_bounds__(256) im2col_kernel(ConvShape c, const uint16_t* __restrict__ x, int rows_pad,
                                                     int k_pad, int TR, uint16_t* __restrict__ out) {
  const long long n = (long long)rows_pad * tap_groups(k_pad);
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x)
    gather_taps(e, rows_pad, TR, k_pad, c.Cin, c.H * c.W, x,
                [&](int p, int* off, unsigned& in) -> size_t {
                  if (p >= c.P) return 0;
                  const unsigned img = (unsigned)p / (unsigned)(c.Ho * c.Wo), pix = p - img * (c.Ho * c.Wo);
                  const int oy = (int)(pix / (unsigned)c.Wo), ox = (int)pix - oy * c.Wo;
#pragma unroll
                  for (int t = 0; t < 9; ++t) {
                    const int iy = oy * S - 1 + t / 3, ix = ox * S - 1 + t % 3;
                    off[t] = iy * c.W + ix;
                    if (iy >= 0 && iy < c.H && ix >= 0 && ix < c.W) in |= 1u << t;
                  }
                  return (size_t)img * c.Cin * (c.H * c.W);
                },
                out);
}

// A of the weight gradient: rows k = ci*9+tap, K over output pixels p, plus row
// Cin*9 of ones, whose product with g is the bias gradient.
template <int S>
__global__ void im2col_t_kernel(ConvShape c, const uint16_t* __restrict__ x, int rows_pad, int k_pad, int TR,
                                uint16_t* __restrict__ out) {
  constexpr uint16_t kOne = 0x3f80;  // 1 in BF16
  const long long n8 = (long long)rows_pad * (k_pad / 8);
  const int KC = k_pad / kTcKC;
  const unsigned HoWo = c.Ho * c.Wo;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n8; e += (long long)gridDim.x * blockDim.x) {
    int k, p0;
    unit_rk(e, TR, KC, k, p0);
    uint16_t v[8];
    const int ci = k / 9, tap = k - (k / 9) * 9;
    const int dy = tap / 3 - 1, dx = tap % 3 - 1;
    const unsigned n = (unsigned)p0 / HoWo, pix = (unsigned)p0 - n * HoWo;
    int oy = (int)(pix / (unsigned)c.Wo), ox = (int)pix - oy * c.Wo;
    const uint16_t* plane = x + ((size_t)n * c.Cin + ci) * (c.H * c.W);
    if (c.Wo % 8 == 0 && k < c.K) {  // the eight pixels share an image row
      const int iy = oy * S + dy, ix = ox * S + dx;
      const bool row = p0 < c.P && iy >= 0 && iy < c.H;
      const uint16_t* src = plane + iy * c.W + ix;
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = (row && ix + i * S >= 0 && ix + i * S < c.W) ? src[i * S] : (uint16_t)0;
      store8_bits(out + e * 8, v);
      continue;
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int iy = oy * S + dy, ix = ox * S + dx;
      const bool in = p0 + i < c.P, ok = in && k < c.K && iy >= 0 && iy < c.H && ix >= 0 && ix < c.W;
      v[i] = ok ? plane[iy * c.W + ix] : (in && k == c.K ? kOne : (uint16_t)0);
      if (++ox == c.Wo) {
        ox = 0;
        if (++oy == c.Ho) {
          oy = 0;
          plane += (size_t)c.Cin * (c.H * c.W);
        }
      }
    }
    store8_bits(out + e * 8, v);
  }
}

// B of the forward: w[co][k] (bf16 [Cout][Cin*9])
__global__ void weights_kernel(int rows, int cols, const bf16t* __restrict__ w, int rows_pad, int k_pad, int TR,
                               uint16_t* __restrict__ out) {
  const long long n8 = (long long)rows_pad * (k_pad / 8);
  const int KC = k_pad / kTcKC;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n8; e += (long long)gridDim.x * blockDim.x) {
    int r, k0;
    unit_rk(e, TR, KC, r, k0);
    float v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
      v[i] = (r < rows && k0 + i < cols) ? __bfloat162float(w[(size_t)r * cols + k0 + i]) : 0.f;
    store8(out + e * 8, v);
  }
}

// B of the input gradient: wT[ci][co*9 + tap] = w[co][ci][tap]
__global__ void weights_t_kernel(ConvShape c, const bf16t* __restrict__ w, int rows_pad, int k_pad, int TR,
                                 uint16_t* __restrict__ out) {
  const long long n8 = (long long)rows_pad * (k_pad / 8);
  const int KC = k_pad / kTcKC;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n8; e += (long long)gridDim.x * blockDim.x) {
    int ci, k0;
    unit_rk(e, TR, KC, ci, k0);
    float v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int kt = k0 + i;
      v[i] = (ci < c.Cin && kt < c.Kt)
                 ? __bfloat162float(w[((size_t)(kt / 9) * c.Cin + ci) * 9 + kt % 9])
                 : 0.f;
    }
    store8(out + e * 8, v);
  }
}

// A of the input gradient: col(g)[q][co*9 + tap] = g[n][co][oy][ox] for the
// output pixel whose tap covers input pixel q (zero where none does)
template <int S>
__global__ void __launch_bounds__(256) gcol_kernel(ConvShape c, const float* __restrict__ g, int rows_pad, int k_pad,
                                                   uint16_t* __restrict__ out) {
  const long long n = (long long)rows_pad * tap_groups(k_pad);
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x)
    gather_taps(e, rows_pad, kTcM, k_pad, c.Cout, c.Ho * c.Wo, g,
                [&](int q, int* off, unsigned& in) -> size_t {
                  if (q >= c.Q) return 0;
                  const unsigned img = (unsigned)q / (unsigned)(c.H * c.W), pix = q - img * (c.H * c.W);
                  const int iy = (int)(pix / (unsigned)c.W), ix = (int)pix - iy * c.W;
#pragma unroll
                  for (int t = 0; t < 9; ++t) {
                    const int ty = iy + 1 - t / 3, tx = ix + 1 - t % 3;
                    const int oy = ty / S, ox = tx / S;  // used for ty, tx >= 0 only
                    off[t] = oy * c.Wo + ox;
                    if (ty >= 0 && tx >= 0 && oy * S == ty && ox * S == tx && oy < c.Ho && ox < c.Wo) in |= 1u << t;
                  }
                  return (size_t)img * c.Cout * (c.Ho * c.Wo);
                },
                out);
}

// The same operand of a stride-2 layer of even width, two neighbouring input
// pixels a thread: of their 18 taps 3 (even image row) or 6 (odd row) meet an
// output pixel, and which ones is known at compile time, where the general form
// tests and loads nine a pixel.  Their units are neighbours too: 32-byte stores.
// 256 samples: 134 -> 77 us for the layer of 32 x 32 inputs, 43 -> 25 and 12 -> 8 for the next.
__global__ void __launch_bounds__(256) gcol_pairs_kernel(ConvShape c, const float* __restrict__ g, int rows_pad,
                                                         int k_pad, uint16_t* __restrict__ out) {
  const int pairs = rows_pad / 2, KC = k_pad / kTcKC, units = k_pad / 8, plane_size = c.Ho * c.Wo;
  const long long n = (long long)pairs * tap_groups(k_pad);
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
    const int group = (int)(e / pairs), q = 2 * (int)(e - (long long)group * pairs);
    const unsigned img = (unsigned)q / (unsigned)(c.H * c.W), pix = q - img * (c.H * c.W);
    const int iy = (int)(pix / (unsigned)c.W), oy = iy / 2, ox = ((int)pix - iy * c.W) / 2;
    const bool in = q < c.Q, right = ox + 1 < c.Wo, odd = iy & 1, down = odd && oy + 1 < c.Ho;
    const float* src = g + ((size_t)img * c.Cout + group * 8) * plane_size + oy * c.Wo + ox;
    // g at (oy, ox), (oy, ox + 1) and, for odd rows, one row down
    uint16_t at[8][4];
#pragma unroll
    for (int ch = 0; ch < 8; ++ch) {
      const bool ok = in && group * 8 + ch < c.Cout;
      at[ch][0] = __bfloat16_as_ushort(__float2bfloat16_rn(ok ? src[0] : 0.f));
      at[ch][1] = __bfloat16_as_ushort(__float2bfloat16_rn(ok && right ? src[1] : 0.f));
      at[ch][2] = __bfloat16_as_ushort(__float2bfloat16_rn(ok && down ? src[c.Wo] : 0.f));
      at[ch][3] = __bfloat16_as_ushort(__float2bfloat16_rn(ok && down && right ? src[c.Wo + 1] : 0.f));
      src += plane_size;
    }
    const int tile = q / kTcM, rl = q - tile * kTcM;
    auto emit = [&](auto odd_row) {
#pragma unroll
      for (int u = 0; u < 9; ++u) {
        const int ku = group * 9 + u;
        unsigned w[8];  // the even pixel's eight K elements, then the odd pixel's
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const int k = u * 8 + i % 8, ch = k / 9, t = k % 9;
          int from;  // which of at[ch], -1: none
          if constexpr (decltype(odd_row)::value)
            from = i < 8 ? (t == 1 ? 2 : t == 7 ? 0 : -1) : (t == 0 ? 3 : t == 2 ? 2 : t == 6 ? 1 : t == 8 ? 0 : -1);
          else
            from = i < 8 ? (t == 4 ? 0 : -1) : (t == 3 ? 1 : t == 5 ? 0 : -1);
          const unsigned v = from < 0 ? 0u : at[ch][from];
          w[i / 2] = i % 2 ? w[i / 2] | v << 16 : v;
        }
        if (ku < units) {
          const size_t unit = ((size_t)tile * KC + ku / 8) * (kTcM * 8) + (rl / 8) * 64 + (ku % 8) * 8 + rl % 8;
          asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(out + unit * 8), "r"(w[0]),
                       "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7])
                       : "memory");
        }
      }
    };
    if (odd)
      emit(std::true_type{});
    else
      emit(std::false_type{});
  }
}

// B of the weight gradient: gT[co][p] = g[n][co][oy][ox]
__global__ void gT_kernel(ConvShape c, const float* __restrict__ g, int rows_pad, int k_pad, int TR,
                          uint16_t* __restrict__ out) {
  const long long n8 = (long long)rows_pad * (k_pad / 8);
  const int KC = k_pad / kTcKC;
  const unsigned HoWo = c.Ho * c.Wo;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n8; e += (long long)gridDim.x * blockDim.x) {
    int co, p0;
    unit_rk(e, TR, KC, co, p0);
    float v[8];
    const unsigned n = (unsigned)p0 / HoWo;
    unsigned pix = (unsigned)p0 - n * HoWo;
    const float* plane = g + ((size_t)n * c.Cout + co) * HoWo;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      v[i] = (co < c.Cout && p0 + i < c.P) ? plane[pix] : 0.f;
      if (++pix == HoWo) {
        pix = 0;
        plane += (size_t)c.Cout * HoWo;
      }
    }
    store8(out + e * 8, v);
  }
}

// Linear-layer operands: (r, k) = src[r*sr + k*sk] for r < R, k < Kv; row
// ones_row (if >= R) holds ones for k < Kv; zeros elsewhere.
__device__ __forceinline__ float to_f(bf16t v) { return __bfloat162float(v); }
__device__ __forceinline__ float to_f(float v) { return v; }

template <class T>
__global__ void pack_kernel(const T* __restrict__ src, long long sr, long long sk, int R, int Kv, int ones_row,
                            int rows_pad, int k_pad, int TR, uint16_t* __restrict__ out) {
  const long long n8 = (long long)rows_pad * (k_pad / 8);
  const int KC = k_pad / kTcKC;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n8; e += (long long)gridDim.x * blockDim.x) {
    int r, k0;
    unit_rk(e, TR, KC, r, k0);
    float v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int k = k0 + i;
      v[i] = k >= Kv ? 0.f : (r < R ? to_f(src[r * sr + k * sk]) : (r == ones_row ? 1.f : 0.f));
    }
    store8(out + e * 8, v);
  }
}

// ---- epilogues ----------------------------------------------------------------
struct EpiConvFwd {
  struct Params {
    bf16t* y;
    const float* bias;
    int Cout, HoWo, P, relu;
  };
  static __device__ __forceinline__ void apply(int row, int col0, const float* v, const Params& p) {
    if (row >= p.P) return;
    const int n = row / p.HoWo, pix = row % p.HoWo;
#pragma unroll
    for (int i = 0; i < 32; ++i) {
      const int co = col0 + i;
      if (co < p.Cout) {
        float a = v[i] + (p.bias ? p.bias[co] : 0.f);
        if (p.relu && a < 0.f) a = 0.f;
        p.y[((size_t)n * p.Cout + co) * p.HoWo + pix] = __float2bfloat16(a);
      }
    }
  }
};

struct EpiConvDx {
  struct Params {
    float* dx;
    int Cin, HW, Q;
  };
  static __device__ __forceinline__ void apply(int row, int col0, const float* v, const Params& p) {
    if (row >= p.Q) return;
    const int n = row / p.HW, pix = row % p.HW;
#pragma unroll
    for (int i = 0; i < 32; ++i)
      if (col0 + i < p.Cin) p.dx[((size_t)n * p.Cin + col0 + i) * p.HW + pix] = v[i];
  }
};

// rows: k = ci*9 + tap (row Cin*9: the bias), columns: co.  Adjacent threads
// add to adjacent words of dw.
struct EpiConvDw {
  struct Params {
    float* dw;
    float* db;  // optional
    int Cout, K;
  };
  static __device__ __forceinline__ void apply(int row, int col0, const float* v, const Params& p) {
    if (row > p.K || (row == p.K && !p.db)) return;
    float* dst = row < p.K ? p.dw + row : p.db;
    const int stride = row < p.K ? p.K : 1;
#pragma unroll
    for (int i = 0; i < 32; ++i)
      if (col0 + i < p.Cout) atomicAdd(dst + (size_t)(col0 + i) * stride, v[i]);
  }
};

// linear forward as y^T: rows o, columns n (adjacent threads write adjacent outputs)
struct EpiLinFwd {
  struct Params {
    bf16t* y;
    float* yf;
    const float* bias;
    int Out, N, relu;
  };
  static __device__ __forceinline__ void apply(int row, int col0, const float* v, const Params& p) {
    if (row >= p.Out) return;
    const float b = p.bias ? p.bias[row] : 0.f;
#pragma unroll
    for (int i = 0; i < 32; ++i) {
      const int n = col0 + i;
      if (n < p.N) {
        float a = v[i] + b;
        if (p.relu && a < 0.f) a = 0.f;
        if (p.y) p.y[(size_t)n * p.Out + row] = __float2bfloat16(a);
        if (p.yf) p.yf[(size_t)n * p.Out + row] = a;
      }
    }
  }
};

// linear input gradient as dx^T: rows i, columns n
struct EpiLinDx {
  struct Params {
    float* dx;
    int In, N;
  };
  static __device__ __forceinline__ void apply(int row, int col0, const float* v, const Params& p) {
    if (row >= p.In) return;
#pragma unroll
    for (int i = 0; i < 32; ++i)
      if (col0 + i < p.N) p.dx[(size_t)(col0 + i) * p.In + row] = v[i];
  }
};

template <class Epi, int BN, int ST>
static int launch_gemm(dim3 grid, const TcGemmArgs& g, const typename Epi::Params& ep, cudaStream_t s) {
  constexpr int SMEM = TcSmem<BN, false, ST>::BYTES;  // single BF16 term: no lo buffers
  if (cudaFuncSetAttribute(tc_gemm_kernel<Epi, BN, false, false, ST>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           SMEM) != cudaSuccess)
    return LGB_ERR_CUDA;
  tc_gemm_kernel<Epi, BN, false, false, ST><<<grid, kTcThreads, SMEM, s>>>(g, ep);
  return cudaGetLastError() == cudaSuccess ? LGB_OK : LGB_ERR_CUDA;
}

// Stages of K chunks.  Six (all that fit) where a grid has at most a CTA per SM
// and each chunk's latency shows: 18 chunks of 128 x 128 in 32 CTAs 22.8 -> 17.9
// us.  Larger grids share an SM: three stages leave room for two to three CTAs
// and suit four chunks or more (512 CTAs of 14 chunks 56 -> 41 us; four stages
// 57); with fewer, two stages and one CTA more are better (2,048 CTAs of two
// chunks 26 us, 31 with three stages).
template <class Epi, int BN>
static int run_gemm(int m_tiles, int n_tiles, int k_chunks, int splits, const uint16_t* a, const uint16_t* b,
                    int* status, const typename Epi::Params& ep, cudaStream_t s) {
  const int per = (k_chunks + splits - 1) / splits;
  const int z = (k_chunks + per - 1) / per;
  TcGemmArgs g{a, nullptr, b, nullptr, k_chunks, 1, status, splits > 1 ? per : 0};
  const dim3 grid(n_tiles, m_tiles, z);
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if ((long long)n_tiles * m_tiles * z <= sms) return launch_gemm<Epi, BN, 6>(grid, g, ep, s);
  if (per >= 4) return launch_gemm<Epi, BN, 3>(grid, g, ep, s);
  return launch_gemm<Epi, BN, 2>(grid, g, ep, s);
}

template <class Epi>
static int run_gemm_bn(int bn, int m_tiles, int n_tiles, int k_chunks, int splits, const uint16_t* a,
                       const uint16_t* b, int* status, const typename Epi::Params& ep, cudaStream_t s) {
  switch (bn) {
    case 32:
      return run_gemm<Epi, 32>(m_tiles, n_tiles, k_chunks, splits, a, b, status, ep, s);
    case 64:
      return run_gemm<Epi, 64>(m_tiles, n_tiles, k_chunks, splits, a, b, status, ep, s);
    default:
      return run_gemm<Epi, 128>(m_tiles, n_tiles, k_chunks, splits, a, b, status, ep, s);
  }
}

static int grid256(long long n) {
  long long g = (n + 255) / 256;
  if (g > 65535LL * 16) g = 65535LL * 16;
  return (int)(g < 1 ? 1 : g);
}

// Operand sizes (bytes) of each pass, 256-byte aligned.
struct ConvWs {
  size_t fwd_a, fwd_b, dx_a, dx_b, dw_a, dw_b, total_fwd, total_bwd;
};
static size_t al256(size_t n) { return (n + 255) & ~(size_t)255; }
static ConvWs conv_ws(const ConvShape& c) {
  ConvWs w{};
  const int bnf = bn_for(c.Cout), bnx = bn_for(c.Cin);
  w.fwd_a = al256((size_t)round_up(c.P, kTcM) * round_up(c.K, kTcKC) * 2);
  w.fwd_b = al256((size_t)round_up(c.Cout, bnf) * round_up(c.K, kTcKC) * 2);
  w.dx_a = al256((size_t)round_up(c.Q, kTcM) * round_up(c.Kt, kTcKC) * 2);
  w.dx_b = al256((size_t)round_up(c.Cin, bnx) * round_up(c.Kt, kTcKC) * 2);
  w.dw_a = al256((size_t)round_up(c.K + 1, kTcM) * round_up(c.P, kTcKC) * 2);
  w.dw_b = al256((size_t)round_up(c.Cout, bnf) * round_up(c.P, kTcKC) * 2);
  w.total_fwd = w.fwd_a + w.fwd_b;
  w.total_bwd = w.dx_a + w.dx_b > w.dw_a + w.dw_b ? w.dx_a + w.dx_b : w.dw_a + w.dw_b;
  return w;
}

struct LinWs {
  size_t fwd_a, fwd_b, dx_a, dx_b, dw_a, dw_b, total;
};
static LinWs lin_ws(int N, int In, int Out) {
  LinWs w{};
  const int bnN = bn_for(N), bnO = bn_for(Out);
  w.fwd_a = al256((size_t)round_up(Out, kTcM) * round_up(In, kTcKC) * 2);
  w.fwd_b = al256((size_t)round_up(N, bnN) * round_up(In, kTcKC) * 2);
  w.dx_a = al256((size_t)round_up(In, kTcM) * round_up(Out, kTcKC) * 2);
  w.dx_b = al256((size_t)round_up(N, bnN) * round_up(Out, kTcKC) * 2);
  w.dw_a = al256((size_t)round_up(In + 1, kTcM) * round_up(N, kTcKC) * 2);
  w.dw_b = al256((size_t)round_up(Out, bnO) * round_up(N, kTcKC) * 2);
  size_t t = w.fwd_a + w.fwd_b;
  if (w.dx_a + w.dx_b > t) t = w.dx_a + w.dx_b;
  if (w.dw_a + w.dw_b > t) t = w.dw_a + w.dw_b;
  w.total = t;
  return w;
}

static int sm_count() {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms > 0 ? sms : 1;
}

}  // namespace lgb

using namespace lgb;

extern "C" {

int lgb_nn_conv3x3_workspace_size(int N, int Cin, int H, int W, int Cout, int stride, size_t* bytes) {
  if (N < 1 || Cin < 1 || H < 1 || W < 1 || Cout < 1 || Cout > 128 || Cin > 128 || (stride != 1 && stride != 2) ||
      !bytes)
    return LGB_ERR_INVALID_ARGUMENT;
  const ConvShape c = conv_shape(N, Cin, H, W, Cout, stride);
  if ((long long)N * H * W > 65535LL * kTcM) return LGB_ERR_INVALID_ARGUMENT;  // M tiles on grid y
  const ConvWs w = conv_ws(c);
  *bytes = w.total_fwd > w.total_bwd ? w.total_fwd : w.total_bwd;
  return LGB_OK;
}

int lgb_nn_conv3x3_forward(int N, int Cin, int H, int W, int Cout, int stride, int relu, const void* x, const void* w,
                           const float* b, void* y, void* workspace, size_t workspace_bytes, int* device_status,
                           void* stream) {
  size_t need = 0;
  if (lgb_nn_conv3x3_workspace_size(N, Cin, H, W, Cout, stride, &need) != LGB_OK || !x || !w || !y || !workspace ||
      !device_status)
    return LGB_ERR_INVALID_ARGUMENT;
  if (workspace_bytes < need) return LGB_ERR_WORKSPACE_TOO_SMALL;
  if (reinterpret_cast<uintptr_t>(workspace) & 255) return LGB_ERR_INVALID_ARGUMENT;
  cudaStream_t s = (cudaStream_t)stream;
  const ConvShape c = conv_shape(N, Cin, H, W, Cout, stride);
  const ConvWs ws = conv_ws(c);
  uint16_t* a = static_cast<uint16_t*>(workspace);
  uint16_t* bm = reinterpret_cast<uint16_t*>(static_cast<char*>(workspace) + ws.fwd_a);
  const int bn = bn_for(Cout);
  const int kp = round_up(c.K, kTcKC), pp = round_up(c.P, kTcM), cp = round_up(Cout, bn);
  (stride == 1 ? im2col_kernel<1> : im2col_kernel<2>)<<<grid256((long long)pp * tap_groups(kp)), 256, 0, s>>>(
      c, static_cast<const uint16_t*>(x), pp, kp, kTcM, a);
  weights_kernel<<<grid256((long long)cp * kp / 8), 256, 0, s>>>(Cout, c.K, static_cast<const bf16t*>(w), cp, kp, bn,
                                                                 bm);
  if (cudaGetLastError() != cudaSuccess) return LGB_ERR_CUDA;
  EpiConvFwd::Params ep{static_cast<bf16t*>(y), b, Cout, c.Ho * c.Wo, c.P, relu};
  return run_gemm_bn<EpiConvFwd>(bn, pp / kTcM, cp / bn, kp / kTcKC, 1, a, bm, device_status, ep, s);
}

int lgb_nn_conv3x3_backward(int N, int Cin, int H, int W, int Cout, int stride, const void* x, const void* w,
                            const float* g, float* dx, float* dw, float* db, void* workspace, size_t workspace_bytes,
                            int* device_status, void* stream) {
  size_t need = 0;
  if (lgb_nn_conv3x3_workspace_size(N, Cin, H, W, Cout, stride, &need) != LGB_OK || !x || !w || !g || !dw ||
      !workspace || !device_status)
    return LGB_ERR_INVALID_ARGUMENT;
  if (workspace_bytes < need) return LGB_ERR_WORKSPACE_TOO_SMALL;
  if (reinterpret_cast<uintptr_t>(workspace) & 255) return LGB_ERR_INVALID_ARGUMENT;
  cudaStream_t s = (cudaStream_t)stream;
  const ConvShape c = conv_shape(N, Cin, H, W, Cout, stride);
  const ConvWs ws = conv_ws(c);
  char* base = static_cast<char*>(workspace);
  int st;
  if (dx) {  // input gradient
    uint16_t* a = reinterpret_cast<uint16_t*>(base);
    uint16_t* bm = reinterpret_cast<uint16_t*>(base + ws.dx_a);
    const int bn = bn_for(Cin);
    const int kp = round_up(c.Kt, kTcKC), qp = round_up(c.Q, kTcM), cp = round_up(Cin, bn);
    if (stride == 2 && W % 2 == 0)
      gcol_pairs_kernel<<<grid256((long long)qp / 2 * tap_groups(kp)), 256, 0, s>>>(c, g, qp, kp, a);
    else
      (stride == 1 ? gcol_kernel<1> : gcol_kernel<2>)<<<grid256((long long)qp * tap_groups(kp)), 256, 0, s>>>(c, g, qp,
                                                                                                              kp, a);
    weights_t_kernel<<<grid256((long long)cp * kp / 8), 256, 0, s>>>(c, static_cast<const bf16t*>(w), cp, kp, bn, bm);
    if (cudaGetLastError() != cudaSuccess) return LGB_ERR_CUDA;
    EpiConvDx::Params ep{dx, Cin, H * W, c.Q};
    if ((st = run_gemm_bn<EpiConvDx>(bn, qp / kTcM, cp / bn, kp / kTcKC, 1, a, bm, device_status, ep, s)))
      return st;
  }
  {  // weight and bias gradients: [Cin*9 + 1] x [Cout] over K = output pixels, split across CTAs
     // (atomic adds into zeroed dw, db)
    uint16_t* a = reinterpret_cast<uint16_t*>(base);
    uint16_t* bm = reinterpret_cast<uint16_t*>(base + ws.dw_a);
    const int bn = bn_for(Cout);
    const int pk = round_up(c.P, kTcKC), kr = round_up(c.K + 1, kTcM), cp = round_up(Cout, bn);
    (stride == 1 ? im2col_t_kernel<1> : im2col_t_kernel<2>)<<<grid256((long long)kr * pk / 8), 256, 0, s>>>(
        c, static_cast<const uint16_t*>(x), kr, pk, kTcM, a);
    gT_kernel<<<grid256((long long)cp * pk / 8), 256, 0, s>>>(c, g, cp, pk, bn, bm);
    if (cudaGetLastError() != cudaSuccess) return LGB_ERR_CUDA;
    if (cudaMemsetAsync(dw, 0, sizeof(float) * (size_t)Cout * c.K, s) != cudaSuccess) return LGB_ERR_CUDA;
    if (db && cudaMemsetAsync(db, 0, sizeof(float) * (size_t)Cout, s) != cudaSuccess) return LGB_ERR_CUDA;
    const int m_tiles = kr / kTcM, k_chunks = pk / kTcKC;
    int splits = (2 * sm_count() + m_tiles - 1) / m_tiles;
    if (splits > k_chunks) splits = k_chunks;
    EpiConvDw::Params ep{dw, db, Cout, c.K};
    if ((st = run_gemm_bn<EpiConvDw>(bn, m_tiles, cp / bn, k_chunks, splits, a, bm, device_status, ep, s))) return st;
  }
  return LGB_OK;
}

int lgb_nn_linear_workspace_size(int N, int In, int Out, size_t* bytes) {
  if (N < 1 || In < 1 || Out < 1 || !bytes || (long long)round_up(In + 1, kTcM) / kTcM > 65535 ||
      (long long)round_up(Out, kTcM) / kTcM > 65535)
    return LGB_ERR_INVALID_ARGUMENT;
  *bytes = lin_ws(N, In, Out).total;
  return LGB_OK;
}

int lgb_nn_linear_forward(int N, int In, int Out, int relu, const void* x, const void* w, const float* b, void* y_bf16,
                          float* y_f32, void* workspace, size_t workspace_bytes, int* device_status, void* stream) {
  size_t need = 0;
  if (lgb_nn_linear_workspace_size(N, In, Out, &need) != LGB_OK || !x || !w || (!y_bf16 && !y_f32) || !workspace ||
      !device_status)
    return LGB_ERR_INVALID_ARGUMENT;
  if (workspace_bytes < need) return LGB_ERR_WORKSPACE_TOO_SMALL;
  if (reinterpret_cast<uintptr_t>(workspace) & 255) return LGB_ERR_INVALID_ARGUMENT;
  cudaStream_t s = (cudaStream_t)stream;
  const LinWs ws = lin_ws(N, In, Out);
  uint16_t* a = static_cast<uint16_t*>(workspace);
  uint16_t* bm = reinterpret_cast<uint16_t*>(static_cast<char*>(workspace) + ws.fwd_a);
  const int bn = bn_for(N);
  const int kp = round_up(In, kTcKC), op = round_up(Out, kTcM), np = round_up(N, bn);
  pack_kernel<bf16t><<<grid256((long long)op * kp / 8), 256, 0, s>>>(static_cast<const bf16t*>(w), In, 1, Out, In, -1,
                                                                      op, kp, kTcM, a);
  pack_kernel<bf16t><<<grid256((long long)np * kp / 8), 256, 0, s>>>(static_cast<const bf16t*>(x), In, 1, N, In, -1,
                                                                      np, kp, bn, bm);
  if (cudaGetLastError() != cudaSuccess) return LGB_ERR_CUDA;
  EpiLinFwd::Params ep{static_cast<bf16t*>(y_bf16), y_f32, b, Out, N, relu};
  return run_gemm_bn<EpiLinFwd>(bn, op / kTcM, np / bn, kp / kTcKC, 1, a, bm, device_status, ep, s);
}

int lgb_nn_linear_backward(int N, int In, int Out, const void* x, const void* w, const float* g, float* dx, float* dw,
                           float* db, void* workspace, size_t workspace_bytes, int* device_status, void* stream) {
  size_t need = 0;
  if (lgb_nn_linear_workspace_size(N, In, Out, &need) != LGB_OK || !x || !w || !g || !dw || !workspace ||
      !device_status)
    return LGB_ERR_INVALID_ARGUMENT;
  if (workspace_bytes < need) return LGB_ERR_WORKSPACE_TOO_SMALL;
  if (reinterpret_cast<uintptr_t>(workspace) & 255) return LGB_ERR_INVALID_ARGUMENT;
  cudaStream_t s = (cudaStream_t)stream;
  const LinWs ws = lin_ws(N, In, Out);
  char* base = static_cast<char*>(workspace);
  int st;
  if (dx) {  // dx^T[i][n] = sum_o w[o][i] g[n][o]
    uint16_t* a = reinterpret_cast<uint16_t*>(base);
    uint16_t* bm = reinterpret_cast<uint16_t*>(base + ws.dx_a);
    const int bn = bn_for(N);
    const int kp = round_up(Out, kTcKC), ip = round_up(In, kTcM), np = round_up(N, bn);
    pack_kernel<bf16t><<<grid256((long long)ip * kp / 8), 256, 0, s>>>(static_cast<const bf16t*>(w), 1, In, In, Out,
                                                                        -1, ip, kp, kTcM, a);
    pack_kernel<float><<<grid256((long long)np * kp / 8), 256, 0, s>>>(g, Out, 1, N, Out, -1, np, kp, bn, bm);
    if (cudaGetLastError() != cudaSuccess) return LGB_ERR_CUDA;
    EpiLinDx::Params ep{dx, In, N};
    if ((st = run_gemm_bn<EpiLinDx>(bn, ip / kTcM, np / bn, kp / kTcKC, 1, a, bm, device_status, ep, s))) return st;
  }
  {  // [dw^T; db][i][o] = sum_n [x; 1][n][i] g[n][o], split over n with atomic adds
    uint16_t* a = reinterpret_cast<uint16_t*>(base);
    uint16_t* bm = reinterpret_cast<uint16_t*>(base + ws.dw_a);
    const int bn = bn_for(Out);
    const int kp = round_up(N, kTcKC), ip = round_up(In + 1, kTcM), op = round_up(Out, bn);
    pack_kernel<bf16t><<<grid256((long long)ip * kp / 8), 256, 0, s>>>(static_cast<const bf16t*>(x), 1, In, In, N, In,
                                                                        ip, kp, kTcM, a);
    pack_kernel<float><<<grid256((long long)op * kp / 8), 256, 0, s>>>(g, 1, Out, Out, N, -1, op, kp, bn, bm);
    if (cudaGetLastError() != cudaSuccess) return LGB_ERR_CUDA;
    if (cudaMemsetAsync(dw, 0, sizeof(float) * (size_t)Out * In, s) != cudaSuccess) return LGB_ERR_CUDA;
    if (db && cudaMemsetAsync(db, 0, sizeof(float) * (size_t)Out, s) != cudaSuccess) return LGB_ERR_CUDA;
    const int m_tiles = ip / kTcM, n_tiles = op / bn, k_chunks = kp / kTcKC;
    int splits = (2 * sm_count() + m_tiles * n_tiles - 1) / (m_tiles * n_tiles);
    if (splits > k_chunks) splits = k_chunks;
    EpiConvDw::Params ep{dw, db, Out, In};
    if ((st = run_gemm_bn<EpiConvDw>(bn, m_tiles, n_tiles, k_chunks, splits, a, bm, device_status, ep, s))) return st;
  }
  return LGB_OK;
}

}  // extern "C"
