// impz_poisson.cuh -- open-boundary Poisson solve on the device.
//
// Restates openBC3D + greenf1tIntnew (src/Appl/Field.f90:239-519): Hockney's
// doubled-grid convolution phi = IFFT(FFT(rho_padded) * FFT(G_even)) with the
// integrated Green's function G, then kick1's finite-difference field
// (src/Appl/BeamBunch.f90:1784-2005).  Any correct FFT reproduces the
// reference's FFTPACK convolution to rounding, so the transforms here are the
// project's own register FFTs (impz_fft.cuh) laid out for the doubled grid:
//
//   xy-forward  one block per z plane: int64 charge -> real, R2C along x
//               (two real rows packed into one complex FFT of length 2Nx),
//               C2C along y (length 2Ny, upper half zero), spectrum plane out
//   z-convolve  a few lines per block: C2C along z (length 2Nz, upper half
//               zero), times the real even G-hat, inverse C2C, only the Nz
//               planes the crop needs are written back
//   xy-inverse  one block per z plane < Nz: inverse C2C along y, C2R along x,
//               potential plane out (only Nx x Ny of the doubled grid)
//
// After the x transform the kx = 0 and kx = Nx rows are real, so they travel
// through the y transform as one complex line: a plane has Nx lines, a power
// of two, and the pair is separated (joined) where the spectrum is stored
// (loaded).
//
// G is even in every direction, so its transform is real and is computed as
// three DCT-I passes over the octant (Nx+1)(Ny+1)(Nz+1) (two lines packed
// into one complex FFT: even real sequences have real transforms).  The
// 1/(n1 n2 n3) inverse normalisation of Field.f90:321-323 is folded into G-hat.
//
// Layouts in HBM.  The z convolution is the pass with the long lines, so the
// spectrum is stored for it: the lines are grouped, 2T to a group (T values
// of the line index q at ky and the same T at 2Ny - ky), and a group's
// points lie together, z by z, S[group][z][side][T]: a block reads and
// writes one contiguous piece, and the xy passes touch whole 32-byte sectors
// (T = 4 FP32 values, 2 or 4 FP64 ones; zt_log).  Line q = row * Nx + kx for kx < Nx, and
// Ny * Nx + row for kx = Nx, with row = ky (side 0) or 2Ny - ky (side 1; row
// 0 holds ky = 0 and ky = Ny).  G-hat holds T lines together in the same
// way, ((q / T) (Nz+1) + kz) T + q mod T with q = ky Nx + kx, then the kx =
// Nx lines, and the last line (ky = Ny, kx = Nx) alone.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "impz_common.h"
#include "impz_device.cuh"
#include "impz_fft.cuh"

namespace impz {

struct PoissonDims {
  int nx, ny, nz;
  int lx, ly, lz;  // log2 of the doubled lengths 2nx, 2ny, 2nz
};

// log2 of T, the lines of one side of a group, for z transforms of 2^lz
// points.  Never less than a 32-byte sector: with T = 1 for the long lines
// (as many as the z convolution works on at once) the xy passes moved 8 of
// every 32 bytes, and took 307 of 501 us at 64x64x2048.
template <typename T>
__host__ __device__ constexpr int zt_log(int lz) {
  return sizeof(T) == 4 ? 2 : lz <= 8 ? 2 : 1;
}

// element index of spectrum line (ky, kx) at plane z
__device__ __forceinline__ size_t spec_index(const PoissonDims& d, int lt, int ky, int kx, int z) {
  const int n2 = 2 * d.ny;
  const int side = ky >= d.ny ? 1 : 0;
  const int row = ky < d.ny ? ky : ky == d.ny ? 0 : n2 - ky;
  const int q = kx < d.nx ? row * d.nx + kx : d.ny * d.nx + row;
  return (((size_t)(q >> lt) * d.nz + z) << (lt + 1)) + (side << lt) + (q & ((1 << lt) - 1));
}

// first element and spacing along kz of line (ky, kx) of G-hat (ky <= ny, kx <= nx)
__device__ __forceinline__ size_t ghat_line(int nx, int ny, int nz, int lt, int ky, int kx,
                                            int& spacing) {
  const int q = kx < nx ? ky * nx + kx : (ny + 1) * nx + ky;
  spacing = (kx == nx && ky == ny) ? 1 : 1 << lt;
  return (((size_t)(q >> lt) * (nz + 1)) << lt) + (q & ((1 << lt) - 1));
}

__host__ __device__ constexpr int round_to(int v, int m) { return (v + m - 1) / m * m; }

// The xy kernels' shape: lines of the x transform (row pairs) and of the y
// transform, each rounded to whole warps (the spare lines are scratch), the
// pitches of their lines, and the block.  The pitches put the transposing
// reads between the two transforms on different banks: 2 mod 16 eight-byte
// slots (FP32), odd sixteen-byte slots (FP64).
template <typename T, int LX, int LY>
struct XyShape {
  typedef Fft<T, LX, sizeof(T) == 4> FX;
  typedef Fft<T, LY, sizeof(T) == 4> FY;
  typedef typename Cplx<T>::type C;
  static constexpr int nx = 1 << (LX - 1), ny = 1 << (LY - 1), hy = ny / 2;
  static constexpr int TA = round_to(hy * FX::TPL, 32), TB = round_to(nx * FY::TPL, 32);
  static constexpr int LA = TA / FX::TPL, LB = TB / FY::TPL;
  static constexpr int extra = sizeof(T) == 4 ? 2 : 1;
  static constexpr int XP = FX::LEN + extra, YP = FY::LEN + extra;
  static constexpr int NT = TA > TB ? TA : TB;
  // the x and y lines are never needed at the same time
  static constexpr size_t smem = sizeof(C) * (size_t)(LA * XP > LB * YP ? LA * XP : LB * YP);
};

// The bunch a block works for: the *_group launches give the members of a
// group of one grid size in device memory (blockIdx.y = member), a solo
// launch passes its own by value.  Copied, not referred to: a reference that
// may point to either was compiled into reads of the wrong one.
__device__ __forceinline__ PoissonMember member_of(const PoissonMember& one,
                                                   const PoissonMember* __restrict__ many) {
  PoissonMember m = one;
  if (many) m = many[blockIdx.y];
  return m;
}

// ---------------------------------------------------------------------
// xy-forward: one block per z plane.  Bound by latency (128 planes on 148
// SMs at 64x64x128): every thread holds its part of one line, so a plane
// takes two register transforms, three block barriers and one exchange of
// the plane in between.
template <typename T, int LX, int LY>
__device__ __forceinline__ void fft_xy_fwd_body(const PoissonDims& d, const PoissonMember& mm) {
  typedef XyShape<T, LX, LY> X;
  typedef typename X::FX FX;
  typedef typename X::FY FY;
  typedef typename Cplx<T>::type C;
  constexpr int nx = X::nx, ny = X::ny, hy = X::hy, n1 = 2 * nx, n2 = 2 * ny;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* sm = reinterpret_cast<C*>(smem_raw);
  const int tid = threadIdx.x, z = blockIdx.x;
  griddep_wait();
  const unsigned long long* rho = mm.rho + (size_t)nx * ny * z;
  if (tid < X::TA) {  // rows l and l + hy as one complex line
    const int l = tid / FX::TPL, j = tid % FX::TPL;
    C v[FX::E];
#pragma unroll
    for (int e = 0; e < FX::E / 2; e++) {
      const int x = j + FX::TPL * e;
      v[e].x = 0;
      v[e].y = 0;
      if (l < hy) {
        v[e].x = (T)((double)(long long)rho[l * nx + x] * mm.qscale);
        v[e].y = (T)((double)(long long)rho[(l + hy) * nx + x] * mm.qscale);
      }
    }
    C* L = sm + l * X::XP;
    FX::template run<-1, true>(v, j, L, (const C*)mm.twx, WarpSync());
    __syncwarp();
#pragma unroll
    for (int e = 0; e < FX::E; e++) L[FX::pad(j + FX::TPL * e)] = v[e];
  }
  __syncthreads();
  // unpack: row a = (Z(k)+conj(Z(n1-k)))/2, row b = (Z(k)-conj(Z(n1-k)))/(2i);
  // at kx = 0 both rows' kx = 0 and kx = nx values (real) as one complex line
  const int kx = tid / FY::TPL, j = tid % FY::TPL;
  C v[FY::E];
  if (tid < X::TB) {
#pragma unroll
    for (int e = 0; e < FY::E / 4; e++) {
      C a, b;
      a.x = a.y = b.x = b.y = 0;
      if (kx < nx) {
        const C* L = sm + (j + FY::TPL * e) * X::XP;
        const C zk = L[FX::pad(kx)];
        const C zm = L[FX::pad(kx ? n1 - kx : nx)];
        if (kx) {
          a.x = (T)0.5 * (zk.x + zm.x);
          a.y = (T)0.5 * (zk.y - zm.y);
          b.x = (T)0.5 * (zk.y + zm.y);
          b.y = (T)0.5 * (zm.x - zk.x);
        } else {
          a.x = zk.x; a.y = zm.x;
          b.x = zk.y; b.y = zm.y;
        }
      }
      v[e] = a;
      v[e + FY::E / 4] = b;
    }
  }
  __syncthreads();
  if (tid >= X::TB) return;
  C* L = sm + kx * X::YP;
  FY::template run<-1, true>(v, j, L, (const C*)mm.twy, WarpSync());
  C* S = (C*)mm.spec;
  const int lt = zt_log<T>(d.lz);
  if (kx > 0 && kx < nx) {
#pragma unroll
    for (int e = 0; e < FY::E; e++) S[spec_index(d, lt, j + FY::TPL * e, kx, z)] = v[e];
  }
  if (tid < 32) {  // the warp of the packed line: separate its two real rows
    __syncwarp();
    if (kx == 0) {
#pragma unroll
      for (int e = 0; e < FY::E; e++) L[FY::pad(j + FY::TPL * e)] = v[e];
    }
    __syncwarp();
    if (kx == 0) {
#pragma unroll
      for (int e = 0; e < FY::E; e++) {
        const int ky = j + FY::TPL * e;
        const C m = L[FY::pad((n2 - ky) & (n2 - 1))];
        C a, b;
        a.x = (T)0.5 * (v[e].x + m.x);
        a.y = (T)0.5 * (v[e].y - m.y);
        b.x = (T)0.5 * (v[e].y + m.y);
        b.y = (T)0.5 * (m.x - v[e].x);
        S[spec_index(d, lt, ky, 0, z)] = a;
        S[spec_index(d, lt, ky, nx, z)] = b;
      }
    }
  }
}

template <typename T, int LX, int LY>
__global__ void __launch_bounds__((XyShape<T, LX, LY>::NT))
    k_fft_xy_fwd(PoissonDims d, PoissonMember one, const PoissonMember* __restrict__ many) {
  fft_xy_fwd_body<T, LX, LY>(d, member_of(one, many));
}

// ---------------------------------------------------------------------
// xy-inverse: one block per z plane k < nz; phi out (nx, ny, nz) real.
template <typename T, int LX, int LY>
__device__ __forceinline__ void fft_xy_inv_body(const PoissonDims& d, const PoissonMember& mm) {
  typedef XyShape<T, LX, LY> X;
  typedef typename X::FX FX;
  typedef typename X::FY FY;
  typedef typename Cplx<T>::type C;
  constexpr int nx = X::nx, ny = X::ny, hy = X::hy, n1 = 2 * nx;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* sm = reinterpret_cast<C*>(smem_raw);
  const int tid = threadIdx.x, z = blockIdx.x;
  const int lt = zt_log<T>(d.lz);
  griddep_wait();
  if (tid < X::TB) {
    const int kx = tid / FY::TPL, j = tid % FY::TPL;
    const C* S = (const C*)mm.spec;
    C v[FY::E];
#pragma unroll
    for (int e = 0; e < FY::E; e++) {
      v[e].x = 0;
      v[e].y = 0;
      if (kx < nx) v[e] = S[spec_index(d, lt, j + FY::TPL * e, kx, z)];
      if (kx == 0) {  // the kx = 0 and kx = nx rows as one complex line
        const C b = S[spec_index(d, lt, j + FY::TPL * e, nx, z)];
        v[e].x = v[e].x - b.y;
        v[e].y = v[e].y + b.x;
      }
    }
    C* L = sm + kx * X::YP;
    FY::template run<1, false>(v, j, L, (const C*)mm.twy, WarpSync());
    __syncwarp();
#pragma unroll
    for (int e = 0; e < FY::E / 2; e++) L[FY::pad(j + FY::TPL * e)] = v[e];
  }
  __syncthreads();
  // C2R along x for row pairs (l, l + hy): Z(kx) = Xa(kx) + i Xb(kx), with
  // X(n1-kx) = conj(X(kx))
  const int l = tid / FX::TPL, j = tid % FX::TPL;
  C v[FX::E];
  if (tid < X::TA) {
#pragma unroll
    for (int e = 0; e < FX::E; e++) {
      const int kk = j + FX::TPL * e;
      v[e].x = 0;
      v[e].y = 0;
      if (l < hy) {
        const C* L = sm + ((kk == nx ? 0 : kk < nx ? kk : n1 - kk) * X::YP);
        C xa = L[FY::pad(l)], xb = L[FY::pad(l + hy)];
        if (kk == 0) { xa.y = 0; xb.y = 0; }
        if (kk == nx) { xa.x = xa.y; xb.x = xb.y; xa.y = 0; xb.y = 0; }
        if (kk > nx) { xa.y = -xa.y; xb.y = -xb.y; }
        v[e].x = xa.x - xb.y;
        v[e].y = xa.y + xb.x;
      }
    }
  }
  __syncthreads();
  if (tid >= X::TA) return;
  FX::template run<1, false>(v, j, sm + l * X::XP, (const C*)mm.twx, WarpSync());
  if (l >= hy) return;
  T* ph = (T*)mm.phi + (size_t)nx * ny * z;
#pragma unroll
  for (int e = 0; e < FX::E / 2; e++) {
    const int x = j + FX::TPL * e;
    ph[l * nx + x] = v[e].x;
    ph[(l + hy) * nx + x] = v[e].y;
  }
}

template <typename T, int LX, int LY>
__global__ void __launch_bounds__((XyShape<T, LX, LY>::NT))
    k_fft_xy_inv(PoissonDims d, PoissonMember one, const PoissonMember* __restrict__ many) {
  fft_xy_inv_body<T, LX, LY>(d, member_of(one, many));
}

// ---------------------------------------------------------------------
// The z kernels' shape.  PAR lines are in work at once, thread (j, line)
// with the lines fastest: the spectrum's group and the threads of a warp run
// along the same contiguous piece.  The pitch puts the lines of a half
// (quarter) warp on different banks.
template <typename T, int LZ, int PAR>
struct ZShape {
  typedef Fft<T, LZ> F;
  static constexpr int slots = 128 / (int)(2 * sizeof(T));  // of one shared-memory wavefront
  static constexpr int want = PAR < slots ? slots / PAR : 1;
  static constexpr int P0 = F::LEN;
  static constexpr int pitch = P0 + (want + slots - P0 % slots) % slots;
  static constexpr int NT = PAR * F::TPL;
  static constexpr size_t smem = sizeof(typename Cplx<T>::type) * (size_t)PAR * pitch;
};

// lines of the z convolution in work at once: a whole group, several groups
// where the lines are short, and a part of the group, round by round, where a
// block of 512 threads holds no more (the rounds share sectors that stay in
// L1 or L2)
template <typename T, int LZ>
struct ZConv {
  typedef Fft<T, LZ> F;
  static constexpr int lt = zt_log<T>(LZ), NL = 2 << lt;
  static constexpr int GPB = NL * F::TPL >= 128 ? 1 : 128 / (NL * F::TPL);  // groups per block
  static constexpr int PAR = NL * F::TPL <= 512 ? NL * GPB : F::TPL >= 512 ? 1 : 512 / F::TPL;
  static constexpr int ROUNDS = NL * GPB / PAR;
  typedef ZShape<T, LZ, PAR> Z;
};

template <typename T, int LZ>
__device__ __forceinline__ void fft_z_conv_body(const PoissonDims& d, const PoissonMember& mm) {
  typedef ZConv<T, LZ> Q;
  typedef typename Q::F F;
  typedef typename Cplx<T>::type C;
  constexpr int lt = Q::lt, NL = Q::NL, nz = F::N / 2;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* sm = reinterpret_cast<C*>(smem_raw);
  const int nx = d.nx, ny = d.ny;
  const int ngroups = (ny * nx + ny) >> lt;
  const int j = (int)threadIdx.x / Q::PAR, p = (int)threadIdx.x % Q::PAR;
  griddep_wait();
#pragma unroll 1
  for (int r = 0; r < Q::ROUNDS; r++) {
    const int slot = r * Q::PAR + p;  // of the block's NL * GPB lines
    const int g = blockIdx.x * Q::GPB + slot / NL, l = slot % NL;
    const bool live = g < ngroups;
    C* S = (C*)mm.spec + (size_t)(live ? g : 0) * nz * NL + l;
    // the line's place, and G-hat's line for it
    const int q = (g << lt) + (l & ((1 << lt) - 1));
    int row, kx;
    if (q < nx * ny) { row = q >> (d.lx - 1); kx = q & (nx - 1); }
    else { row = q - nx * ny; kx = nx; }
    const int kyp = (l >> lt) && row == 0 ? ny : row;
    int gs = 1;
    const T* G = (const T*)mm.ghat + (live ? ghat_line(nx, ny, nz, lt, kyp, kx, gs) : 0);
    C v[F::E];
    T gv[F::E];
#pragma unroll
    for (int e = 0; e < F::E / 2; e++) {
      const int z = j + F::TPL * e;
      v[e].x = 0;
      v[e].y = 0;
      if (live) v[e] = S[(size_t)z * NL];
    }
#pragma unroll
    for (int e = 0; e < F::E; e++) {
      const int kz = j + F::TPL * e;
      gv[e] = 0;
      if (live) gv[e] = __ldg(G + (size_t)(e < F::E / 2 ? kz : F::N - kz) * gs);
    }
    C* L = sm + p * Q::Z::pitch;
    F::template run<-1, true>(v, j, L, (const C*)mm.twz, BlockSync());
#pragma unroll
    for (int e = 0; e < F::E; e++) {
      v[e].x *= gv[e];
      v[e].y *= gv[e];
    }
    F::template run<1, false>(v, j, L, (const C*)mm.twz, BlockSync());
    if (live) {
#pragma unroll
      for (int e = 0; e < F::E / 2; e++) S[(size_t)(j + F::TPL * e) * NL] = v[e];
    }
  }
}

// The three passes of a step took 70 us at 64x64x128 in FP32 as radix-2^3
// groups in shared memory and take 36 so (FP64 97 and 56); at 64x64x2048,
// where the spectrum (136 MB) no longer fits L2, 1498 and 411 (35 and 394
// without the second terms of the constants and of the x and y twiddles).
template <typename T, int LZ>
__global__ void __launch_bounds__((ZConv<T, LZ>::Z::NT))
    k_fft_z_conv(PoissonDims d, PoissonMember one, const PoissonMember* __restrict__ many) {
  fft_z_conv_body<T, LZ>(d, member_of(one, many));
}

// ---------------------------------------------------------------------
// greenf1tIntnew corner antiderivative (Field.f90:392-418), FP64, at the
// (nx+2)(ny+2)(nz+2) corners v = (i-1)h - h/2.
__device__ __forceinline__ void igf_corners_body(int nx, int ny, int nz, const DevState* st,
                                                 double* F) {
  const int ax = nx + 2, ay = ny + 2, az = nz + 2;
  const long long total = (long long)ax * ay * az;
  const double hx = st->geom.h[0], hy = st->geom.h[1], hz = st->geom.h[2];
  const double hxyz = hx * hy * hz;
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < total;
       e += (long long)gridDim.x * blockDim.x) {
    const int i0 = (int)(e % ax);
    const int j0 = (int)((e / ax) % ay);
    const int k0 = (int)(e / ((long long)ax * ay));
    const double v1 = (double)i0 * hx - hx / 2;
    const double v2 = (double)j0 * hy - hy / 2;
    const double v3 = (double)k0 * hz - hz / 2;
    const double rr = sqrt(v1 * v1 + v2 * v2 + v3 * v3);
    const double aa = -(v3 * v3 * atan(v1 * v2 / (v3 * rr)) / 2);
    const double bb = -(v2 * v2 * atan(v1 * v3 / (v2 * rr)) / 2);
    const double cc = -(v1 * v1 * atan(v2 * v3 / (v1 * rr)) / 2);
    const double dd = v2 * v3 * log(v1 + rr);
    const double ee = v1 * v3 * log(v2 + rr);
    const double ff = v1 * v2 * log(v3 + rr);
    const double gg2 = aa + bb + cc + dd + ee + ff;
    F[e] = gg2 / hxyz;
  }
}

static __global__ void k_igf_corners(int nx, int ny, int nz, PoissonMember one,
                              const PoissonMember* __restrict__ many) {
  const PoissonMember m = member_of(one, many);
  igf_corners_body(nx, ny, nz, m.st, m.F);
}

// The Green octant one z plane per block: the 8-corner difference of plane
// k (Field.f90:420-428, FP64: it cancels catastrophically), rounded to the
// convolution's type T, then its DCT-I along x and along y in shared memory
// (rows, then columns, two lines per complex FFT of length 2n), written to
// plane k of G-hat; the z pass follows.  One pass over the corners and one
// write of the plane instead of a difference kernel and two strided DCT
// passes through global memory.
template <typename T, int LX, int LY>
struct GreenShape {
  typedef Fft<T, LX> FX;
  typedef Fft<T, LY> FY;
  typedef typename Cplx<T>::type C;
  static constexpr int nx = 1 << (LX - 1), ny = 1 << (LY - 1), gx = nx + 1, gy = ny + 1;
  static constexpr int npx = (gy + 1) / 2;  // row pairs (t, t + npx) for the x transform
  static constexpr int npy = (gx + 1) / 2;  // column pairs for the y transform
  static constexpr int TA = round_to(npx * FX::TPL, 32), TB = round_to(npy * FY::TPL, 32);
  static constexpr int LA = TA / FX::TPL, LB = TB / FY::TPL;
  static constexpr int NF = TA > TB ? TA : TB;
  static constexpr int NT = NF < 512 && gx * gy > 1024 ? 512 : NF;  // for the difference pass
  static constexpr size_t lines = LA * FX::LEN > LB * FY::LEN ? LA * FX::LEN : LB * FY::LEN;
  static constexpr size_t smem = sizeof(C) * lines + sizeof(T) * (size_t)gx * gy;
};

template <typename T, int LX, int LY>
__device__ __forceinline__ void green_xy_body(const PoissonDims& d, const PoissonMember& mm) {
  typedef GreenShape<T, LX, LY> X;
  typedef typename X::FX FX;
  typedef typename X::FY FY;
  typedef typename Cplx<T>::type C;
  constexpr int nx = X::nx, ny = X::ny, gx = X::gx, gy = X::gy, ax = nx + 2, ay = ny + 2;
  constexpr int npx = X::npx, npy = X::npy;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* sm = reinterpret_cast<C*>(smem_raw);
  T* P = reinterpret_cast<T*>(sm + X::lines);
  const int tid = threadIdx.x, k = blockIdx.x;
  const double* F0 = mm.F + (size_t)ax * ay * k;  // corner planes k and k + 1
  const double* F1 = F0 + (size_t)ax * ay;
#pragma unroll 4
  for (int e = tid; e < gx * gy; e += X::NT) {
    const int j = e / gx, i = e - j * gx;
#define IMPZ_F(p, a, b) __ldg(p + (a) + ax * (b))
    const double v = IMPZ_F(F1, i + 1, j + 1) - IMPZ_F(F1, i, j + 1) - IMPZ_F(F1, i + 1, j) +
                     IMPZ_F(F1, i, j) - IMPZ_F(F0, i + 1, j + 1) + IMPZ_F(F0, i, j + 1) +
                     IMPZ_F(F0, i + 1, j) - IMPZ_F(F0, i, j);
#undef IMPZ_F
    P[e] = (T)v;
  }
  __syncthreads();
  if (tid < X::TA) {  // along x: row t with row t + npx (real and imaginary parts)
    const int t = tid / FX::TPL, j = tid % FX::TPL;
    C v[FX::E];
#pragma unroll
    for (int e = 0; e < FX::E; e++) {
      const int m = j + FX::TPL * e, m1 = m <= nx ? m : 2 * nx - m;
      v[e].x = t < npx ? P[t * gx + m1] : (T)0;
      v[e].y = t + npx < gy ? P[(t + npx) * gx + m1] : (T)0;
    }
    FX::template run<-1, false>(v, j, sm + t * FX::LEN, (const C*)mm.twx, WarpSync());
#pragma unroll
    for (int e = 0; e < FX::E; e++) {
      const int m = j + FX::TPL * e;
      if (m > nx) continue;
      if (t < npx) P[t * gx + m] = v[e].x;
      if (t + npx < gy) P[(t + npx) * gx + m] = v[e].y;
    }
  }
  __syncthreads();
  if (tid >= X::TB) return;
  {  // along y: column t with column t + npy
    const int t = tid / FY::TPL, j = tid % FY::TPL;
    const int lt = zt_log<T>(d.lz);
    C v[FY::E];
#pragma unroll
    for (int e = 0; e < FY::E; e++) {
      const int m = j + FY::TPL * e, m1 = m <= ny ? m : 2 * ny - m;
      v[e].x = t < npy ? P[m1 * gx + t] : (T)0;
      v[e].y = t + npy < gx ? P[m1 * gx + t + npy] : (T)0;
    }
    FY::template run<-1, false>(v, j, sm + t * FY::LEN, (const C*)mm.twy, WarpSync());
    T* out = (T*)mm.ghat;
#pragma unroll
    for (int e = 0; e < FY::E; e++) {
      const int m = j + FY::TPL * e;
      if (m > ny) continue;
      int gs;
      if (t < npy) {
        const size_t b = ghat_line(nx, ny, d.nz, lt, m, t, gs);
        out[b + (size_t)k * gs] = v[e].x;
      }
      if (t + npy < gx) {
        const size_t b = ghat_line(nx, ny, d.nz, lt, m, t + npy, gs);
        out[b + (size_t)k * gs] = v[e].y;
      }
    }
  }
}

template <typename T, int LX, int LY>
__global__ void __launch_bounds__((GreenShape<T, LX, LY>::NT))
    k_green_xy(PoissonDims d, PoissonMember one, const PoissonMember* __restrict__ many) {
  green_xy_body<T, LX, LY>(d, member_of(one, many));
}

// DCT-I (transform of the even extension) along z of G-hat's lines, in
// place, times `scale`: lines 2p and 2p + 1 (neighbours in storage) as the
// real and imaginary parts of one complex FFT of length 2nz.
template <typename T, int LZ>
struct ZDct {
  typedef Fft<T, LZ> F;
  static constexpr int PAR = F::TPL >= 128 ? 1 : 128 / F::TPL > 16 ? 16 : 128 / F::TPL;
  typedef ZShape<T, LZ, PAR> Z;
  static constexpr int NT = round_to(Z::NT, 32);
};

template <typename T, int LZ>
__device__ __forceinline__ void dct_z_body(const PoissonDims& d, const PoissonMember& mm,
                                           T scale) {
  typedef ZDct<T, LZ> Q;
  typedef typename Q::F F;
  typedef typename Cplx<T>::type C;
  constexpr int lt = zt_log<T>(LZ), nz = F::N / 2;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* sm = reinterpret_cast<C*>(smem_raw);
  const int nlines = (d.nx + 1) * (d.ny + 1);
  const int j = (int)threadIdx.x / Q::PAR, p = (int)threadIdx.x % Q::PAR;
  const int qa = 2 * (blockIdx.x * Q::PAR + p), qb = qa + 1;
  const bool la = qa < nlines && j < F::TPL, lb = qb < nlines && j < F::TPL;
  const int sa = qa == nlines - 1 ? 1 : 1 << lt, sb = qb == nlines - 1 ? 1 : 1 << lt;
  T* A = (T*)mm.ghat + (la ? (((size_t)(qa >> lt) * (nz + 1)) << lt) + (qa & ((1 << lt) - 1)) : 0);
  T* B = (T*)mm.ghat + (lb ? (((size_t)(qb >> lt) * (nz + 1)) << lt) + (qb & ((1 << lt) - 1)) : 0);
  C v[F::E];
#pragma unroll
  for (int e = 0; e < F::E; e++) {
    const int m = j + F::TPL * e, m1 = m <= nz ? m : F::N - m;
    v[e].x = la ? A[(size_t)m1 * sa] : (T)0;
    v[e].y = lb ? B[(size_t)m1 * sb] : (T)0;
  }
  F::template run<-1, false>(v, j, sm + p * Q::Z::pitch, (const C*)mm.twz, BlockSync());
#pragma unroll
  for (int e = 0; e < F::E; e++) {
    const int m = j + F::TPL * e;
    if (m > nz) continue;
    if (la) A[(size_t)m * sa] = v[e].x * scale;
    if (lb) B[(size_t)m * sb] = v[e].y * scale;
  }
}

template <typename T, int LZ>
__global__ void __launch_bounds__((ZDct<T, LZ>::NT))
    k_dct_z(PoissonDims d, PoissonMember one, const PoissonMember* __restrict__ many, T scale) {
  dct_z_body<T, LZ>(d, member_of(one, many), scale);
}

// ---------------------------------------------------------------------
// kick1_BeamBunch finite differences (BeamBunch.f90:1784-2005), one rank,
// open BC: centred inside, one-sided on the faces.  Out: {Ex,Ey,Ez,0}.
// Also clears the charge grid (its last reader, the forward transform, is
// done) for the next deposit.  With a wake (read-in or CSR), adds its
// per-plane field wake = {dEx, dEy, dEz}[nz] to every node of the plane
// (kick1wake, BeamBunch.f90:5015-5033) and clears the wake's line sums.
// One node per thread, its place by shifts (the sides are powers of two; the
// 64-bit divisions of an earlier form kept the kernel at half of the issue
// rate), one 16-byte store (two in FP64).
__device__ __forceinline__ void store_field(float* E, int e, float x, float y, float z) {
  reinterpret_cast<float4*>(E)[e] = make_float4(x, y, z, 0.f);
}
__device__ __forceinline__ void store_field(double* E, int e, double x, double y, double z) {
  reinterpret_cast<double2*>(E)[2 * e] = make_double2(x, y);
  reinterpret_cast<double2*>(E)[2 * e + 1] = make_double2(z, 0.0);
}

template <typename T>
__global__ void __launch_bounds__(256)
    k_efield(PoissonDims d, PoissonMember one, const PoissonMember* __restrict__ many,
             const double* __restrict__ wake, unsigned long long* __restrict__ wake_line) {
  const PoissonMember mm = member_of(one, many);
  griddep_wait();
  const int nx = d.nx, ny = d.ny, nz = d.nz;
  const int e = blockIdx.x * 256 + threadIdx.x;
  if (wake_line)
    for (int t = e; t < 3 * nz; t += gridDim.x * 256) wake_line[t] = 0ull;
  if (e >= nx * ny * nz) return;
  const T* phi = (const T*)mm.phi;
  const T hxi = (T)mm.st->geom.hi[0], hyi = (T)mm.st->geom.hi[1], hzi = (T)mm.st->geom.hi[2];
  const T half = (T)0.5;
  const int i = e & (nx - 1), j = (e >> (d.lx - 1)) & (ny - 1), k = e >> (d.lx + d.ly - 2);
  const int sy = nx, sz = nx * ny;
  const T c = phi[e];
  const T xm = i > 0 ? phi[e - 1] : c, xp = i < nx - 1 ? phi[e + 1] : c;
  const T ym = j > 0 ? phi[e - sy] : c, yp = j < ny - 1 ? phi[e + sy] : c;
  const T zm = k > 0 ? phi[e - sz] : c, zp = k < nz - 1 ? phi[e + sz] : c;
  T ex = (i == 0 || i == nx - 1 ? hxi : half * hxi) * (xm - xp);
  T ey = (j == 0 || j == ny - 1 ? hyi : half * hyi) * (ym - yp);
  T ez = (k == 0 || k == nz - 1 ? hzi : half * hzi) * (zm - zp);
  if (wake) {
    ex = ex + (T)wake[k];
    ey = ey + (T)wake[nz + k];
    ez = ez + (T)wake[2 * nz + k];
  }
  mm.rho[e] = 0ull;  // the next deposit accumulates into a cleared charge grid
  store_field((T*)mm.efield, e, ex, ey, ez);
}

}  // namespace impz
