// impz_static.cu -- the charge deposit without any device allocation.
//
// Some callers may not allocate device memory while they run: a host code
// whose GPU memory is all handed out by its own pool or arena (it would be
// bypassed, and the allocation can fail in the middle of a run), or a timed
// loop that cannot take the device-wide synchronization cudaMalloc and
// cudaFree imply.  impz_deposit_static serves them: the caller passes the
// particles and the output grid in device memory it owns, and the only
// scratch, the int64 fixed-point accumulator of the deposit, is a fixed
// array in this library's device image (IMPZ_STATIC_MAX_CELLS nodes, 4 MiB),
// held by every GPU that loads the library until the process exits.
//
// The arithmetic is that of the bunch deposit (k_deposit): the z->t frame
// conversion and loss test of conv1st, the CIC cell and weights of
// deposit_BeamBunch, the same fixed-point quanta with the remainder on the
// largest corner, with the quantum chosen from this call's n; for a bunch
// created with the same n and the same geometry the grid equals
// impz_deposit's bit for bit.  Sums go straight to the accumulator with
// 64-bit atomics (integer adds: the result does not depend on their order).
//
// Compiled with --fmad=false like the other FP64 kernels.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <mutex>

#include "../../include/impz_b200.h"
#include "impz_host.h"
#include "impz_launch.h"

#define IMPZ_NS noalloc
#include "impz_particle.cuh"

namespace impz {
namespace noalloc {

// The deposit's accumulator, one int64 per grid node.  Every call on a device
// uses the same array, and it keeps the last call's sums: each call clears
// the nodes it uses before depositing.
static __device__ __align__(256) unsigned long long g_static_rho[IMPZ_STATIC_MAX_CELLS];

struct StaticDepositArgs {
  const double* col[6];  // x, px, y, py, ph, pt (Pts1 rows 1..6), device
  long long n;
  double gam, rad, xl, scale;
  int nx, ny, nz, fixbits;
  Geom g;
};

__global__ void k_static_clear(unsigned long long* acc, long long G) {
  griddep_launch();
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < G;
       i += (long long)gridDim.x * blockDim.x)
    acc[i] = 0ull;
}

// conv1st z->t frame and loss test, deposit_BeamBunch cell, weights and the
// int64 quanta of k_deposit; 64-bit global reductions per corner.  A
// particle outside the caller's box (far outside included: cell_inside does
// not overflow) is skipped, as deposit_BeamBunch skips it.
__global__ void __launch_bounds__(256) k_static_deposit(StaticDepositArgs a,
                                                        unsigned long long* acc) {
  const int nx = a.nx, ny = a.ny, nz = a.nz;
  const long long P = (long long)nx * ny;
  const double scale = ldexp(1.0, a.fixbits);
  const unsigned unit_lo = (unsigned)(1ull << a.fixbits);
  griddep_launch();
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < a.n;
       i += (long long)gridDim.x * blockDim.x) {
    Particle p;
    p.x = a.col[0][i]; p.px = a.col[1][i]; p.y = a.col[2][i];
    p.py = a.col[3][i]; p.ph = a.col[4][i]; p.pt = a.col[5][i];
    const TFrame t = to_tframe(p, a.gam, a.rad, a.xl);
    if (t.lost) continue;
    const Cell c = cic_cell(t.xt, t.yt, t.zt, a.g);
    if (!cell_inside(c, nx, ny, nz)) continue;
    unsigned long long qv[8];
    corner_sums(corner_quanta(c.ab, c.cd, c.ef, scale, unit_lo), qv);
    griddep_wait();  // the cells are cleared
    const long long cc = lin_cell(c, nx, ny);
    const long long node[8] = {cc, cc + nx, cc + nx + P, cc + P, cc + 1 + P, cc + 1 + nx + P,
                               cc + 1 + nx, cc + 1};
#pragma unroll
    for (int k = 0; k < 8; k++) atomicAdd(acc + node[k], qv[k]);
  }
  griddep_wait();  // in every thread, so that this grid cannot end before the clear
}

// chgdens = sum of quanta * weight * 2^-fixbits, as impz_deposit forms it
__global__ void k_static_finish(const unsigned long long* acc, long long G, double scale,
                                double* out) {
  griddep_wait();
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < G;
       i += (long long)gridDim.x * blockDim.x)
    out[i] = (double)(long long)acc[i] * scale;
}

// Device address of g_static_rho and the device's SM count, looked up once
// per device.  In host code the name g_static_rho is only a host-side
// stand-in for the symbol, so the kernels are always given this address,
// never the name.  The cached address belongs to the device's current
// context: a cudaDeviceReset would invalidate it, so the library must not be
// used across one.
constexpr int kMaxDevices = 64;
std::mutex g_addr_mu;
unsigned long long* g_addr[kMaxDevices] = {nullptr};
int g_sms[kMaxDevices] = {0};

int scratch_address(unsigned long long** out, int* sms) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return report_cuda_error(e, "impz_deposit_static: cudaGetDevice");
  if (dev < 0 || dev >= kMaxDevices) return IMPZ_ERR_UNSUPPORTED;
  std::lock_guard<std::mutex> g(g_addr_mu);
  if (!g_addr[dev]) {
    int n_sm = 0;
    e = cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return report_cuda_error(e, "impz_deposit_static: SM count");
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_static_rho);
    if (e != cudaSuccess) return report_cuda_error(e, "impz_deposit_static: cudaGetSymbolAddress");
    g_addr[dev] = (unsigned long long*)p;
    g_sms[dev] = n_sm > 0 ? n_sm : 1;
  }
  *out = g_addr[dev];
  *sms = g_sms[dev];
  return IMPZ_OK;
}

}  // namespace noalloc
}  // namespace impz

extern "C" int impz_deposit_static(const double* x, const double* px, const double* y,
                                   const double* py, const double* ph, const double* pt,
                                   long long n, double gam, double piperad, double piperad2,
                                   double freq, double weight, const double range[6], int nx,
                                   int ny, int nz, double* chgdens, void* stream) {
  using namespace impz;
  using namespace impz::noalloc;
  if (nx < 2 || ny < 2 || nz < 2 || n < 0 || !range || !chgdens || !(freq > 0)) return IMPZ_ERR_ARG;
  const long long G = (long long)nx * ny * nz;
  if (G > IMPZ_STATIC_MAX_CELLS) return IMPZ_ERR_LIMIT;
  if (n > 0 && (!x || !px || !y || !py || !ph || !pt)) return IMPZ_ERR_ARG;
  unsigned long long* acc = nullptr;
  int sms = 1;
  int r = scratch_address(&acc, &sms);
  if (r) return r;
  StaticDepositArgs a;
  const double* cols[6] = {x, px, y, py, ph, pt};
  for (int c = 0; c < 6; c++) a.col[c] = cols[c];
  a.n = n;
  a.gam = gam;
  a.rad = (piperad + piperad2) / 2;       // as impz_sc_prepare forms it
  a.xl = make_phys(freq).Scxl;
  a.nx = nx; a.ny = ny; a.nz = nz;
  int l = 0;
  while ((1ll << l) < n + 1) l++;
  a.fixbits = std::min(40, 62 - l);       // the bunch's rule, l = ceil(log2(n + 1))
  a.scale = weight * std::ldexp(1.0, -a.fixbits);
  // update_CompDom's mesh sizes for this box, as the device computes them
  const int mesh[3] = {nx, ny, nz};
  for (int k = 0; k < 3; k++) {
    a.g.ptrange[2 * k] = a.g.ptrange[2 * k + 1] = 0.0;
    a.g.range[2 * k] = range[2 * k];
    a.g.range[2 * k + 1] = range[2 * k + 1];
    a.g.h[k] = (range[2 * k + 1] - range[2 * k]) / (double)(mesh[k] - 1);
    a.g.hi[k] = 1.0 / a.g.h[k];
    if (!(a.g.h[k] > 0.0) || !std::isfinite(a.g.hi[k])) return IMPZ_ERR_ARG;
  }
  cudaStream_t s = (cudaStream_t)stream;
  const int gclear = (int)std::min<long long>((G + 255) / 256, (long long)sms * 8);
  // the deposit and the last kernel are scheduled while their predecessors
  // run: a small call is three launch latencies and little else (2e4 particles
  // on 32x32x64: 12.3 us a call without it, 9.6 with)
  k_static_clear<<<gclear, 256, 0, s>>>(acc, G);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess && n > 0) {
    const int gdep = (int)std::min<long long>((n + 255) / 256, (long long)sms * 16);
    e = launch_pdl(k_static_deposit, dim3(gdep), dim3(256), 0, s, a, acc);
  }
  if (e == cudaSuccess)
    e = launch_pdl(k_static_finish, dim3(gclear), dim3(256), 0, s, (const unsigned long long*)acc,
                   G, a.scale, chgdens);
  if (e != cudaSuccess) return report_cuda_error(e, "impz_deposit_static: launch");
  count_launches(n > 0 ? 3 : 2);
  return IMPZ_OK;
}
