// Launch wrappers of the open-boundary Poisson solve (impz_poisson.cuh) for
// one type, included by impz_poisson_f32.cu and impz_poisson_f64.cu.
// Compiled with --fmad=false: the Green-function corners and differences
// keep the reference's rounding; the FFT passes write their multiply-adds
// out (impz_fft.cuh).
#include "impz_launch.h"
#include "impz_poisson.cuh"

namespace impz {
namespace {

int ilog2(int n) {
  int l = 0;
  while ((1 << l) < n) l++;
  return l;
}

PoissonDims dims_of(int nx, int ny, int nz) {
  PoissonDims d;
  d.nx = nx; d.ny = ny; d.nz = nz;
  d.lx = ilog2(2 * nx); d.ly = ilog2(2 * ny); d.lz = ilog2(2 * nz);
  return d;
}

// The bunches of one launch: one by value, or nmem of one grid size in
// device memory.
struct Members {
  PoissonMember one;
  const PoissonMember* many;
  int nmem;
};

Members solo(const PoissonBuffers& b) {
  Members m;
  m.one = poisson_member(b);
  m.many = nullptr;
  m.nmem = 1;
  return m;
}

Members group(const PoissonMember* mem, int nmem) {
  Members m = {};
  m.many = mem;
  m.nmem = nmem;
  return m;
}

template <typename K>
cudaError_t allow_smem(K kernel, size_t bytes) {
  if (bytes <= 48 * 1024) return cudaSuccess;
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

// Calls f.template operator()<L>() for the L in [LO, HI] that equals l.
template <int LO, int HI, typename F>
cudaError_t with_log(int l, F&& f) {
  if constexpr (LO > HI) {
    return cudaErrorInvalidValue;
  } else {
    if (l == LO) return f.template operator()<LO>();
    return with_log<LO + 1, HI>(l, f);
  }
}

template <typename T>
struct XyFwd {
  const PoissonDims& d;
  const Members& m;
  cudaStream_t s;
  template <int LX>
  cudaError_t operator()() const {
    return with_log<3, 7>(d.ly, Ly<LX>{*this});
  }
  template <int LX>
  struct Ly {
    const XyFwd& o;
    template <int LY>
    cudaError_t operator()() const {
      typedef XyShape<T, LX, LY> X;
      const cudaError_t e = allow_smem(k_fft_xy_fwd<T, LX, LY>, X::smem);
      if (e != cudaSuccess) return e;
      return launch_pdl(k_fft_xy_fwd<T, LX, LY>, dim3(o.d.nz, o.m.nmem), dim3(X::NT), X::smem, o.s,
                        o.d, o.m.one, o.m.many);
    }
  };
};

template <typename T>
struct XyInv {
  const PoissonDims& d;
  const Members& m;
  cudaStream_t s;
  template <int LX>
  cudaError_t operator()() const {
    return with_log<3, 7>(d.ly, Ly<LX>{*this});
  }
  template <int LX>
  struct Ly {
    const XyInv& o;
    template <int LY>
    cudaError_t operator()() const {
      typedef XyShape<T, LX, LY> X;
      const cudaError_t e = allow_smem(k_fft_xy_inv<T, LX, LY>, X::smem);
      if (e != cudaSuccess) return e;
      return launch_pdl(k_fft_xy_inv<T, LX, LY>, dim3(o.d.nz, o.m.nmem), dim3(X::NT), X::smem, o.s,
                        o.d, o.m.one, o.m.many);
    }
  };
};

template <typename T>
struct GreenXy {
  const PoissonDims& d;
  const Members& m;
  cudaStream_t s;
  template <int LX>
  cudaError_t operator()() const {
    return with_log<3, 7>(d.ly, Ly<LX>{*this});
  }
  template <int LX>
  struct Ly {
    const GreenXy& o;
    template <int LY>
    cudaError_t operator()() const {
      typedef GreenShape<T, LX, LY> X;
      const cudaError_t e = allow_smem(k_green_xy<T, LX, LY>, X::smem);
      if (e != cudaSuccess) return e;
      k_green_xy<T, LX, LY><<<dim3(o.d.nz + 1, o.m.nmem), X::NT, X::smem, o.s>>>(o.d, o.m.one,
                                                                               o.m.many);
      return cudaGetLastError();
    }
  };
};

template <typename T>
struct ZConvolve {
  const PoissonDims& d;
  const Members& m;
  cudaStream_t s;
  template <int LZ>
  cudaError_t operator()() const {
    typedef ZConv<T, LZ> Q;
    const cudaError_t e = allow_smem(k_fft_z_conv<T, LZ>, Q::Z::smem);
    if (e != cudaSuccess) return e;
    const int groups = (d.ny * d.nx + d.ny) >> Q::lt;
    return launch_pdl(k_fft_z_conv<T, LZ>, dim3((groups + Q::GPB - 1) / Q::GPB, m.nmem),
                      dim3(Q::Z::NT), Q::Z::smem, s, d, m.one, m.many);
  }
};

template <typename T>
struct DctZ {
  const PoissonDims& d;
  const Members& m;
  cudaStream_t s;
  template <int LZ>
  cudaError_t operator()() const {
    typedef ZDct<T, LZ> Q;
    const cudaError_t e = allow_smem(k_dct_z<T, LZ>, Q::Z::smem);
    if (e != cudaSuccess) return e;
    const int pairs = ((d.nx + 1) * (d.ny + 1) + 1) / 2;
    const double scale = 1.0 / ((double)(2 * d.nx) * (double)(2 * d.ny) * (double)(2 * d.nz));
    k_dct_z<T, LZ><<<dim3((pairs + Q::PAR - 1) / Q::PAR, m.nmem), Q::NT, Q::Z::smem, s>>>(
        d, m.one, m.many, (T)scale);
    return cudaGetLastError();
  }
};

// The Green function: FP64 corners, then per z plane the FP64 8-corner
// difference (it cancels catastrophically, Field.f90:420-428) and the DCT-I
// along x and y in the convolution's type T (FP64 in the plain form, FP32 in
// the FP32-convolution form), then the DCT-I along z.
template <typename T>
cudaError_t green(const PoissonDims& d, const Members& m, cudaStream_t s) {
  const long long nc = (long long)(d.nx + 2) * (d.ny + 2) * (d.nz + 2);
  const long long cap = (148 * 16 + m.nmem - 1) / m.nmem;
  long long gb = (nc + 255) / 256;
  if (gb > cap) gb = cap;
  k_igf_corners<<<dim3((unsigned)gb, m.nmem), 256, 0, s>>>(d.nx, d.ny, d.nz, m.one, m.many);
  cudaError_t e = with_log<3, 7>(d.lx, GreenXy<T>{d, m, s});
  if (e != cudaSuccess) return e;
  return with_log<3, 13>(d.lz, DctZ<T>{d, m, s});
}

template <typename T>
cudaError_t conv_forward(const PoissonDims& d, const Members& m, cudaStream_t s) {
  return with_log<3, 7>(d.lx, XyFwd<T>{d, m, s});
}

// the z convolution (needs G-hat) and the inverse transform
template <typename T>
cudaError_t conv_rest(const PoissonDims& d, const Members& m, cudaStream_t s) {
  const cudaError_t e = with_log<3, 13>(d.lz, ZConvolve<T>{d, m, s});
  if (e != cudaSuccess) return e;
  return with_log<3, 7>(d.lx, XyInv<T>{d, m, s});
}

template <typename T>
cudaError_t efield(const PoissonDims& d, const Members& m, const double* wake,
                   unsigned long long* wake_line, cudaStream_t s) {
  const int blocks = (d.nx * d.ny * d.nz + 255) / 256;
  return launch_pdl(k_efield<T>, dim3(blocks, m.nmem), dim3(256), 0, s, d, m.one, m.many, wake,
                    wake_line);
}

// exp(-2 pi i k / 2^logn), logn >= 3: the angle is reduced to the first
// octant as an integer, so that it is rounded once, in extended precision,
// and the multiples of an eighth of a turn come out as they are.  An angle
// up to a full turn in FP64 put the entries several units in the last place
// off.
void unit_root(int logn, long long k, long double& re, long double& im) {
  const long long n = 1ll << logn, eighth = n >> 3;
  k &= n - 1;
  const long long octant = k / eighth, rest = k & (eighth - 1);
  const bool odd = octant & 1;  // counted back from the octant's end
  const long double a = 2.0L * 3.14159265358979323846264338327950288L *
                        (long double)(odd ? eighth - rest : rest) / (long double)n;
  const long double c = std::cos(a), s = std::sin(a);
  const long double x[4] = {c, s, -s, -c}, y[4] = {s, c, c, s};  // cos and sin, octants 0..3
  const int o = (int)octant & 3;
  re = octant < 4 ? x[o] : -x[o];
  im = octant < 4 ? -y[o] : y[o];
}

}  // namespace

// Twiddles of a transform of 2^logn points in the order the stages of
// impz_fft.cuh read them, and in FP32 what their rounding dropped from entry
// 2^logn on; returns the number of entries, the second terms not counted.
template <>
int fft_twiddles<IMPZ_POISSON_T>(int logn, void* out) {
  typedef Cplx<IMPZ_POISSON_T>::type C;
  C* t = (C*)out;
  const int le = logn < FftLog2E<IMPZ_POISSON_T>::value ? logn : FftLog2E<IMPZ_POISSON_T>::value;
  int n = 0;
  for (int lns = le; lns < logn;) {
    const int lr = logn - lns < le ? logn - lns : le;
    const int ns = 1 << lns, r = 1 << lr;
    for (int e = 1; e < r; e++)
      for (int m = 0; m < ns; m++, n++) {
        long double x, y;
        unit_root(lns + lr, (long long)e * m, x, y);
        t[n].x = (IMPZ_POISSON_T)x;
        t[n].y = (IMPZ_POISSON_T)y;
        if (sizeof(IMPZ_POISSON_T) == 4) {
          t[(1 << logn) + n].x = (IMPZ_POISSON_T)(x - (long double)t[n].x);
          t[(1 << logn) + n].y = (IMPZ_POISSON_T)(y - (long double)t[n].y);
        }
      }
    lns += lr;
  }
  return n;
}

template <>
cudaError_t launch_green<IMPZ_POISSON_T>(const PoissonBuffers& b, cudaStream_t s) {
  return green<IMPZ_POISSON_T>(dims_of(b.nx, b.ny, b.nz), solo(b), s);
}
template <>
cudaError_t launch_conv_forward<IMPZ_POISSON_T>(const PoissonBuffers& b, cudaStream_t s) {
  return conv_forward<IMPZ_POISSON_T>(dims_of(b.nx, b.ny, b.nz), solo(b), s);
}
template <>
cudaError_t launch_conv_rest<IMPZ_POISSON_T>(const PoissonBuffers& b, cudaStream_t s) {
  return conv_rest<IMPZ_POISSON_T>(dims_of(b.nx, b.ny, b.nz), solo(b), s);
}
template <>
cudaError_t launch_convolve<IMPZ_POISSON_T>(const PoissonBuffers& b, cudaStream_t s) {
  const cudaError_t e = launch_conv_forward<IMPZ_POISSON_T>(b, s);
  return e != cudaSuccess ? e : launch_conv_rest<IMPZ_POISSON_T>(b, s);
}
template <>
cudaError_t launch_efield<IMPZ_POISSON_T>(const PoissonBuffers& b, cudaStream_t s) {
  return efield<IMPZ_POISSON_T>(dims_of(b.nx, b.ny, b.nz), solo(b), b.wake, b.wake_line, s);
}
template <>
cudaError_t launch_green_group<IMPZ_POISSON_T>(int nx, int ny, int nz, const PoissonMember* mem,
                                               int nmem, cudaStream_t s) {
  return green<IMPZ_POISSON_T>(dims_of(nx, ny, nz), group(mem, nmem), s);
}
template <>
cudaError_t launch_conv_group_forward<IMPZ_POISSON_T>(int nx, int ny, int nz,
                                                      const PoissonMember* mem, int nmem,
                                                      cudaStream_t s) {
  return conv_forward<IMPZ_POISSON_T>(dims_of(nx, ny, nz), group(mem, nmem), s);
}
template <>
cudaError_t launch_conv_group_rest<IMPZ_POISSON_T>(int nx, int ny, int nz,
                                                   const PoissonMember* mem, int nmem,
                                                   cudaStream_t s) {
  return conv_rest<IMPZ_POISSON_T>(dims_of(nx, ny, nz), group(mem, nmem), s);
}
template <>
cudaError_t launch_efield_group<IMPZ_POISSON_T>(int nx, int ny, int nz, const PoissonMember* mem,
                                                int nmem, cudaStream_t s) {
  return efield<IMPZ_POISSON_T>(dims_of(nx, ny, nz), group(mem, nmem), nullptr, nullptr, s);
}

}  // namespace impz
