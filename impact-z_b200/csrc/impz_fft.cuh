// impz_fft.cuh -- complex FFTs of 2^3 .. 2^13 points held in registers.
//
// A line of N points is shared by TPL = N/E threads; thread j holds the E
// elements j, j + TPL, j + 2 TPL, ... before and after the transform, in
// natural order (Stockham autosort: no bit reversal anywhere).  Every stage
// is a butterfly of radix E (the last one of whatever radix is left) on the
// thread's own registers; between stages the line is exchanged once through
// shared memory.  E is 16 points in FP32 (two stages up to 256 points, three
// up to 4096) and 8 in FP64, which keeps a thread near 64 registers of data
// and temporaries.  Against radix-2^3 groups run in shared memory this moves
// each point through shared memory once per 16-fold (8-fold) stage instead
// of twice per 8-fold one, and drops the index arithmetic of the
// bit-reversed order: the z convolution of 64x64x128 issued 19.8 M warp
// instructions in that form.
//
// Twiddles come from a table in the order the threads read them: stage with
// Ns points done holds exp(-2 pi i e m / (Ns R)), e = 1..R-1 by m = 0..Ns-1,
// from entry Ns - E on (the stages' sizes telescope, so a table has N - E
// entries).  They are rounded once from the exact angle, never products.  An
// FP32 table has what the rounding dropped from entry N on.
//
// Rounded constants are not harmless in FP32.  The butterflies use the same few
// in every line (cos pi/8 is 3e-8 short), and the first stage's meet the same
// stretches of a line each time: a gain that depends on the position.  The
// entries of the low harmonics turn +k and -k by different angles: a shift.
// Either gives a bunch a net force of its own field, the same in every bunch
// and every step: 9e-9 of the rms force along x and 6e-9 along y at 64x64x128,
// where radix-2 transforms had 4e-9 of random sign and their centroids came out
// five to ten times as close.  So the butterflies' constants have a second term
// (c_mulc), everywhere, and the twiddles too (FINE) in the transforms along x
// and y: net means below 1e-9, rms 2e-9 and 3e-9, the potential's error 1.10e-7
// -> 0.92e-7, the rms momenta over 20 steps of 4e6 particles 9.4e-8 -> 1.4e-8.
// Along z the net force was no worse than before, and second terms of its
// tables cost (64x64x512: 311 -> 335 us a step, 64x64x4096: 2.0 -> 4.1 ms).
#pragma once
#include <cuda_runtime.h>

namespace impz {

template <typename T> struct Cplx;
template <> struct Cplx<double> { typedef double2 type; };
template <> struct Cplx<float> { typedef float2 type; };

// log2 of the elements per thread
template <typename T>
struct FftLog2E { static constexpr int value = sizeof(T) == 4 ? 4 : 3; };

// multiply-add written out: the translation units of the field solve are
// compiled without contraction
__device__ __forceinline__ float fft_fma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fft_fma(double a, double b, double c) { return __fma_rn(a, b, c); }

template <typename C>
__device__ __forceinline__ C c_add(C a, C b) { C r; r.x = a.x + b.x; r.y = a.y + b.y; return r; }
template <typename C>
__device__ __forceinline__ C c_sub(C a, C b) { C r; r.x = a.x - b.x; r.y = a.y - b.y; return r; }
// a * w, w conjugated for the inverse transform (SIGN > 0)
template <int SIGN, typename C>
__device__ __forceinline__ C c_mulw(C a, C w) {
  C r;
  if (SIGN < 0) {
    r.x = fft_fma(a.x, w.x, -(a.y * w.y));
    r.y = fft_fma(a.x, w.y, a.y * w.x);
  } else {
    r.x = fft_fma(a.x, w.x, a.y * w.y);
    r.y = fft_fma(a.y, w.x, -(a.x * w.y));
  }
  return r;
}
// a * (w + l), conjugated likewise: l is what the rounding of w dropped
template <int SIGN, typename C>
__device__ __forceinline__ C c_mulw2(C a, C w, C l) {
  C r;
  if (SIGN < 0) {
    r.x = fft_fma(a.x, w.x, fft_fma(-a.y, w.y, fft_fma(a.x, l.x, -(a.y * l.y))));
    r.y = fft_fma(a.x, w.y, fft_fma(a.y, w.x, fft_fma(a.x, l.y, a.y * l.x)));
  } else {
    r.x = fft_fma(a.x, w.x, fft_fma(a.y, w.y, fft_fma(a.x, l.x, a.y * l.y)));
    r.y = fft_fma(a.y, w.x, fft_fma(-a.x, w.y, fft_fma(a.y, l.x, -(a.x * l.y))));
  }
  return r;
}
// a * (c + i s), a constant of the butterflies, with its second term in FP32
template <int SIGN, typename T, typename C>
__device__ __forceinline__ C c_mulc(C a, double c, double s) {
  C w, l;
  w.x = (T)c;
  w.y = (T)s;
  l.x = (T)(c - (double)w.x);
  l.y = (T)(s - (double)w.y);
  return sizeof(T) == 4 ? c_mulw2<SIGN>(a, w, l) : c_mulw<SIGN>(a, w);
}
// a * (SIGN i)
template <int SIGN, typename C>
__device__ __forceinline__ C c_muli(C a) {
  C r;
  r.x = SIGN < 0 ? a.y : -a.y;
  r.y = SIGN < 0 ? -a.x : a.x;
  return r;
}

// butterflies, natural order in and out; HALF: the upper half of the inputs
// is zero (a zero-padded line's first stage)
template <int SIGN, bool HALF, typename C>
__device__ __forceinline__ void dft4(C& a0, C& a1, C& a2, C& a3) {
  if (HALF) {
    const C u = a0, v = a1, iv = c_muli<SIGN>(a1);
    a0 = c_add(u, v); a1 = c_add(u, iv); a2 = c_sub(u, v); a3 = c_sub(u, iv);
  } else {
    const C t0 = c_add(a0, a2), t1 = c_sub(a0, a2), t2 = c_add(a1, a3);
    const C t3 = c_muli<SIGN>(c_sub(a1, a3));
    a0 = c_add(t0, t2); a1 = c_add(t1, t3); a2 = c_sub(t0, t2); a3 = c_sub(t1, t3);
  }
}

template <int R, int SIGN, bool HALF, typename T, typename C>
__device__ __forceinline__ void dft(C* v) {
  constexpr double h = 0.70710678118654752440;    // cos(pi/4)
  constexpr double c1 = 0.92387953251128675613;   // cos(pi/8)
  constexpr double s1 = 0.38268343236508977173;   // sin(pi/8)
  if (R == 2) {
    const C u = v[0], t = v[1];
    v[0] = c_add(u, t);
    v[1] = c_sub(u, t);
  } else if (R == 4) {
    dft4<SIGN, HALF>(v[0], v[1], v[2], v[3]);
  } else if (R == 8) {
    // even and odd inputs, then the radix-2 step
    dft4<SIGN, HALF>(v[0], v[2], v[4], v[6]);
    dft4<SIGN, HALF>(v[1], v[3], v[5], v[7]);
    const C o0 = v[1], o2 = c_muli<SIGN>(v[5]);
    const C o1 = c_mulc<SIGN, T>(v[3], h, -h);
    const C o3 = c_mulc<SIGN, T>(v[7], -h, -h);
    const C e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6];
    v[0] = c_add(e0, o0); v[4] = c_sub(e0, o0);
    v[1] = c_add(e1, o1); v[5] = c_sub(e1, o1);
    v[2] = c_add(e2, o2); v[6] = c_sub(e2, o2);
    v[3] = c_add(e3, o3); v[7] = c_sub(e3, o3);
  } else {  // 16 = 4 x 4
#pragma unroll
    for (int n = 0; n < 4; n++) dft4<SIGN, HALF>(v[n], v[n + 4], v[n + 8], v[n + 12]);
    // element (n, k) at v[n + 4 k] times w16^(n k)
    v[5] = c_mulc<SIGN, T>(v[5], c1, -s1);
    v[9] = c_mulc<SIGN, T>(v[9], h, -h);
    v[13] = c_mulc<SIGN, T>(v[13], s1, -c1);
    v[6] = c_mulc<SIGN, T>(v[6], h, -h);
    v[10] = c_muli<SIGN>(v[10]);
    v[14] = c_mulc<SIGN, T>(v[14], -h, -h);
    v[7] = c_mulc<SIGN, T>(v[7], s1, -c1);
    v[11] = c_mulc<SIGN, T>(v[11], -h, -h);
    v[15] = c_mulc<SIGN, T>(v[15], -c1, s1);
#pragma unroll
    for (int k = 0; k < 4; k++) dft4<SIGN, false>(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
    // X[k + 4 m] sits at v[4 k + m]: transpose
#pragma unroll
    for (int k = 0; k < 4; k++)
#pragma unroll
      for (int m = k + 1; m < 4; m++) {
        const C t = v[4 * k + m];
        v[4 * k + m] = v[4 * m + k];
        v[4 * m + k] = t;
      }
  }
}

// the exchange of a line among threads of one warp, or of the block
struct WarpSync { __device__ __forceinline__ void operator()() const { __syncwarp(); } };
struct BlockSync { __device__ __forceinline__ void operator()() const { __syncthreads(); } };

// FINE: the twiddles with their second terms (FP32)
template <typename T, int LOGN, bool FINE = false>
struct Fft {
  typedef typename Cplx<T>::type C;
  static constexpr int N = 1 << LOGN;
  static constexpr int LE = LOGN < FftLog2E<T>::value ? LOGN : FftLog2E<T>::value;
  static constexpr int E = 1 << LE;
  static constexpr int TPL = N / E;        // threads per line
  static constexpr int LEN = N + N / E;    // shared-memory slots of a line
  // one spare slot after every E elements: the first stage's threads write
  // E consecutive elements each
  static __device__ __forceinline__ int pad(int i) { return i + (i >> LE); }

  // the stage after 2^LNS points, on the registers the previous exchange filled
  template <int SIGN, bool HALF, int LNS, typename S>
  static __device__ __forceinline__ void stage(C (&v)[E], int j, C* ex, const C* __restrict__ tw,
                                               const S& sync) {
    constexpr int LR = LOGN - LNS < LE ? LOGN - LNS : LE;
    constexpr int R = 1 << LR, SUB = E / R, NS = 1 << LNS;
    constexpr bool last = LNS + LR == LOGN;
    if (LNS > 0) {
#pragma unroll
      for (int q = 0; q < SUB; q++) {
        const int m = (j + TPL * q) & (NS - 1);
#pragma unroll
        for (int e = 1; e < R; e++) {
          const int t = NS - E + (e - 1) * NS + m;
          C& a = v[q * R + e];
          a = FINE ? c_mulw2<SIGN>(a, tw[t], tw[N + t]) : c_mulw<SIGN>(a, tw[t]);
        }
      }
    }
#pragma unroll
    for (int q = 0; q < SUB; q++) dft<R, SIGN, HALF && LNS == 0, T>(v + q * R);
    if constexpr (last) {
      // sub-transform q's output k is element j + TPL (q + SUB k)
      if (SUB > 1) {
        C o[E];
#pragma unroll
        for (int e = 0; e < E; e++) o[e] = v[e];
#pragma unroll
        for (int q = 0; q < SUB; q++)
#pragma unroll
          for (int k = 0; k < R; k++) v[q + SUB * k] = o[q * R + k];
      }
    } else {
      const int b = ((j >> LNS) << (LNS + LR)) + (j & (NS - 1));
      sync();  // the previous readers of the buffer are done
#pragma unroll
      for (int k = 0; k < R; k++) ex[pad(b + k * NS)] = v[k];
      sync();
      constexpr int LR2 = LOGN - LNS - LR < LE ? LOGN - LNS - LR : LE;
      constexpr int R2 = 1 << LR2, SUB2 = E / R2;
#pragma unroll
      for (int q = 0; q < SUB2; q++)
#pragma unroll
        for (int e = 0; e < R2; e++) v[q * R2 + e] = ex[pad(j + TPL * q + TPL * SUB2 * e)];
      stage<SIGN, HALF, LNS + LR>(v, j, ex, tw, sync);
    }
  }

  // v[e] = x[j + TPL e] -> X[j + TPL e]; HALF: x is zero from N/2 on (the
  // upper half of v is not read)
  template <int SIGN, bool HALF, typename S>
  static __device__ __forceinline__ void run(C (&v)[E], int j, C* ex, const C* __restrict__ tw,
                                             const S& sync) {
    stage<SIGN, HALF, 0>(v, j, ex, tw, sync);
  }
};

}  // namespace impz
