// Lines of any even 2,3,5,7-smooth length up to 128 for the convolution's own
// kernels on grids whose sizes are not all 32, 64 or 128: Stockham passes in
// shared memory, a radix a pass, every butterfly of the block's lines shared
// out over its threads.  A plan (host) gives the radices of a length and
// the divisions by its pass lengths as multiplications.
//
// Forward e^(-2 pi i nk/K), inverse e^(+2 pi i nk/K), neither normalized, as
// nb_fft.cuh and cuFFT.
#pragma once
#include <cmath>

#include "nb_fft.cuh"

#define NB_FFT_ANY_MAX 128
#define NB_FFT_ANY_PASSES 5
#define NB_FFT_ANY_THREADS 512

// t / d for t below 2^16 and d from 2 to 2^16 by its reciprocal in 2^-32:
// ceil(2^32 / d) exceeds 2^32 / d by less than one, so the product's error
// stays below t / 2^32 of a unit, less than the 1/d to the next quotient.
struct NbFftDiv {
  unsigned d, m;
  __host__ void set(unsigned v) {
    d = v;
    m = v > 1 ? (unsigned)((0x100000000ull + v - 1) / v) : 0u;
  }
  __device__ __forceinline__ int div(int t) const { return d > 1 ? (int)__umulhi((unsigned)t, m) : t; }
};

// One dimension: pass s joins ns[s] values (the product of the radices before
// it) r[s] at a time.
struct NbFftDim {
  int K, passes;
  int r[NB_FFT_ANY_PASSES], step[NB_FFT_ANY_PASSES];  // radix; K / (ns r), the twiddles' step
  NbFftDiv nj[NB_FFT_ANY_PASSES], ns[NB_FFT_ANY_PASSES];  // K / r butterflies a line; ns
  NbFftDiv k;
};

// The plan of a length; false when it has other factors or is out of range.
inline bool nb_fft_any_plan(int K, NbFftDim &D) {
  D = NbFftDim{};
  if (K < 8 || K > NB_FFT_ANY_MAX || K % 2) return false;
  D.K = K;
  D.k.set((unsigned)K);
  int rest = K, ns = 1;
  while (rest > 1) {
    int r = 0;
    for (int c : {16, 8, 4, 7, 5, 3, 2})
      if (rest % c == 0) {
        r = c;
        break;
      }
    if (!r || D.passes == NB_FFT_ANY_PASSES) return false;
    const int s = D.passes++;
    D.r[s] = r;
    D.nj[s].set((unsigned)(K / r));
    D.ns[s].set((unsigned)ns);
    D.step[s] = K / (ns * r);
    ns *= r;
    rest /= r;
  }
  return true;
}

// An R-point DFT of registers, natural order, for R = 3, 5 and 7: the sums and
// differences of mirrored inputs, each output pair from one cosine and one
// sine sum.
template <int R, bool INV>
__device__ __forceinline__ void nb_fft_dft_odd(float2 (&v)[R]) {
  constexpr int M = (R - 1) / 2;
  // cos and sin of 2 pi k / R
  constexpr float c[3] = {R == 3 ? -0.5f : R == 5 ? 0.30901699437494742f : 0.62348980185873353f,
                          R == 5 ? -0.80901699437494742f : -0.22252093395631440f, -0.90096886790241913f};
  constexpr float s[3] = {R == 3 ? 0.86602540378443865f : R == 5 ? 0.95105651629515357f : 0.78183148246802981f,
                          R == 5 ? 0.58778525229247313f : 0.97492791218182361f, 0.43388373911755812f};
  float2 p[M], d[M];
#pragma unroll
  for (int j = 0; j < M; ++j) {
    p[j] = make_float2(v[j + 1].x + v[R - 1 - j].x, v[j + 1].y + v[R - 1 - j].y);
    d[j] = make_float2(v[j + 1].x - v[R - 1 - j].x, v[j + 1].y - v[R - 1 - j].y);
  }
  const float2 v0 = v[0];
  float2 sum = v0;
#pragma unroll
  for (int j = 0; j < M; ++j) {
    sum.x += p[j].x;
    sum.y += p[j].y;
  }
  v[0] = sum;
#pragma unroll
  for (int k = 1; k <= M; ++k) {
    float2 A = v0, B = make_float2(0.f, 0.f);
#pragma unroll
    for (int j = 1; j <= M; ++j) {
      const int e = (j * k) % R;  // the angle, mirrored past half a turn
      const float cj = c[(e <= M ? e : R - e) - 1];
      const float sj = e <= M ? s[e - 1] : -s[R - e - 1];
      A.x = fmaf(cj, p[j - 1].x, A.x);
      A.y = fmaf(cj, p[j - 1].y, A.y);
      B.x = fmaf(sj, d[j - 1].x, B.x);
      B.y = fmaf(sj, d[j - 1].y, B.y);
    }
    if (INV) B = make_float2(-B.x, -B.y);
    v[k] = make_float2(A.x + B.y, A.y - B.x);
    v[R - k] = make_float2(A.x - B.y, A.y + B.x);
  }
}

template <int R, bool INV>
__device__ __forceinline__ void nb_fft_any_dft(float2 (&v)[R]) {
  if constexpr (R == 2) {
    const float2 a = v[0], b = v[1];
    v[0] = make_float2(a.x + b.x, a.y + b.y);
    v[1] = make_float2(a.x - b.x, a.y - b.y);
  } else if constexpr (R == 4 || R == 8 || R == 16) {
    nb_fft_dft<R, INV>(v);
  } else {
    nb_fft_dft_odd<R, INV>(v);
  }
}

// Pass s of `lines` lines of `stride` values from a to b.
template <int R, bool INV>
__device__ __forceinline__ void nb_fft_any_pass(const float2 *a, float2 *b, int lines, int stride, const NbFftDim &D,
                                                int s, const float2 *tw) {
  const NbFftDiv nj = D.nj[s], nsd = D.ns[s];
  const int NJ = (int)nj.d, NS = (int)nsd.d, step = D.step[s];
  for (int t = threadIdx.x; t < lines * NJ; t += blockDim.x) {
    const int line = nj.div(t), j = t - line * NJ;
    const int q = nsd.div(j), k = j - q * NS;
    const float2 *in = a + line * stride + j;
    float2 v[R];
#pragma unroll
    for (int i = 0; i < R; ++i) v[i] = in[i * NJ];
#pragma unroll
    for (int i = 1; i < R; ++i) {
      float2 w = tw[i * k * step];
      if (INV) w.y = -w.y;
      v[i] = make_float2(v[i].x * w.x - v[i].y * w.y, v[i].x * w.y + v[i].y * w.x);
    }
    nb_fft_any_dft<R, INV>(v);
    float2 *out = b + line * stride + q * NS * R + k;
#pragma unroll
    for (int i = 0; i < R; ++i) out[i * NS] = v[i];
  }
}

// The transforms of `lines` lines in a, with b of the same size as the other
// side; a and b are swapped so that a holds the result.  Every thread of the
// block calls it; the lines are written and synchronized before, and after.
template <bool INV>
__device__ __forceinline__ void nb_fft_any_lines(float2 *&a, float2 *&b, int lines, int stride, const NbFftDim &D,
                                                 const float2 *tw) {
  for (int s = 0; s < D.passes; ++s) {
    switch (D.r[s]) {
      case 2: nb_fft_any_pass<2, INV>(a, b, lines, stride, D, s, tw); break;
      case 3: nb_fft_any_pass<3, INV>(a, b, lines, stride, D, s, tw); break;
      case 4: nb_fft_any_pass<4, INV>(a, b, lines, stride, D, s, tw); break;
      case 5: nb_fft_any_pass<5, INV>(a, b, lines, stride, D, s, tw); break;
      case 7: nb_fft_any_pass<7, INV>(a, b, lines, stride, D, s, tw); break;
      case 8: nb_fft_any_pass<8, INV>(a, b, lines, stride, D, s, tw); break;
      default: nb_fft_any_pass<16, INV>(a, b, lines, stride, D, s, tw); break;
    }
    __syncthreads();
    float2 *t = a;
    a = b;
    b = t;
  }
}
