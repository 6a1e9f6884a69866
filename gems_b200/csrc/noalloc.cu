// noalloc.cu -- SMA-TB forces for callers that cannot allocate device memory.
//
// Some callers of this library may not allocate: a host program that owns a
// fixed device-memory budget and hands the library only its own buffers, or
// one that evaluates forces inside a region where cudaMalloc / cudaFree are
// not allowed (they synchronise the whole device, and are refused while a
// stream is being captured into a CUDA graph).  For them this file provides
// gemsgpu_smatb_forces_noalloc: the SMA-TB density and force passes over
// caller-owned device buffers, with the only scratch (the per-atom density
// rho_i and 1/sqrt(rho_i) carried from the first pass to the second) in a
// fixed file-scope device array.  Nothing here allocates.
//
// The neighbourhood is all pairs within rce (minimum image on periodic
// dimensions), so no neighbour list -- and no list memory -- is needed; the
// result equals the list-based SMA-TB kernels' up to summation order.
#include <cuda_runtime.h>

#include <cmath>
#include <mutex>

#include "../../include/gemsgpu.h"
#include "common.cuh"
#include "fp64.cuh"

namespace {

constexpr int NA_MAX = GEMSGPU_NOALLOC_MAX_ATOMS;
constexpr int NA_BLOCK = 512;
constexpr int NA_UNR = 4;     // candidates per lane and step
constexpr int NA_TILE = 512;  // candidates staged at a time
constexpr int NA_MAXDEV = 64;

// rho_i in [0, NA_MAX), 1/sqrt(rho_i) in [NA_MAX, 2 NA_MAX): 256 KiB that
// every GPU which loads the library holds until the process exits.
static __device__ __align__(256) double g_noalloc_scratch[2 * NA_MAX];

// Device address of g_noalloc_scratch per device.  In host code the symbol
// is only a host-side stand-in, so its device address is looked up once per
// device (with that device current) and passed to the kernels.  The cached
// address belongs to the device's current context: after cudaDeviceReset
// (or anything else that destroys and re-creates the primary context) the
// module may load elsewhere, so a process that resets a device must not
// call gemsgpu_smatb_forces_noalloc on it again.
std::mutex g_na_mutex;
double* g_na_addr[NA_MAXDEV] = {nullptr};

cudaError_t scratch_address(double** out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= NA_MAXDEV) return cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> lk(g_na_mutex);
  if (!g_na_addr[dev]) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess) return e;
    g_na_addr[dev] = static_cast<double*>(p);
  }
  *out = g_na_addr[dev];
  return cudaSuccess;
}

struct NaBox {
  double L[3], invL[3];
  int pbc[3];
};

__device__ __forceinline__ void na_vd(const NaBox& B, const double* x, int i, int j, double& v0,
                                      double& v1, double& v2) {
  v0 = x[3 * j] - x[3 * i];
  v1 = x[3 * j + 1] - x[3 * i + 1];
  v2 = x[3 * j + 2] - x[3 * i + 2];
  if (B.pbc[0]) v0 = v0 - B.L[0] * round(v0 * B.invL[0]);
  if (B.pbc[1]) v1 = v1 - B.L[1] * round(v1 * B.invL[1]);
  if (B.pbc[2]) v2 = v2 - B.L[2] * round(v2 * B.invL[2]);
}

// An atom's record for the filter: its position relative to x0 (its periodic
// image nearest to x0) in single precision, and in w a bound in units of 2^-24
// on the components' rounding errors together (the box lengths' included).
__device__ __forceinline__ float4 na_record(const NaBox& B, const double* x, int j, double3 x0) {
  double d[3] = {x[3 * j] - x0.x, x[3 * j + 1] - x0.y, x[3 * j + 2] - x0.z};
  float w = 0.0f;
#pragma unroll
  for (int k = 0; k < 3; k++) {
    if (B.pbc[k]) {
      d[k] -= B.L[k] * round(d[k] * B.invL[k]);
      w += (float)B.L[k];
    }
    w += fabsf((float)d[k]);
  }
  return make_float4((float)d[0], (float)d[1], (float)d[2], w);
}

// Both passes over all pairs: the density pass (smatb_preinteraction,
// src/TB.F90:367-455) into the scratch, then the force pass (smatb_interact,
// :457-586) from it.
//
// All pairs are tested, but only about 40 of an atom's thousands of candidates
// lie within rce, so the test is done in FP32 on records staged in shared
// memory (a superset: rce plus a bound on the records' errors), 32 candidates
// per warp and step.  What passes is queued, and a full queue of 32 is
// evaluated by the whole warp in FP64 with the exact vector and the exact
// cut-off, so the FP64 arithmetic runs on full warps.  Two warps share an
// atom's candidates; sixteen warps share the staged tile.  Sums are combined
// in a fixed order.
//
// Bound by the filter's issue slots and its ballots' latency from some 3000
// atoms (16384: 777 us), by the launches' and the tiles' latency below (147:
// 10.5 us).  4000 atoms take 72 us.  The form before, one thread per atom with all
// pairs in FP64, took 2.69 ms: 32 blocks on 148 SMs, and every warp entered the
// FP64 branch for almost every candidate.  64 registers (two blocks per SM)
// against 107: 72 and 92 us.  Four atoms per warp pair, for fewer record
// loads: 94 us; 256 threads per block: 68 us, but 878 us at 16384 atoms.
template <bool FORCE>
__global__ void __launch_bounds__(NA_BLOCK, 2) k_na(const double* __restrict__ x, int n, NaBox B, gg::SmFP64 c,
                                                    double* __restrict__ scratch, double* __restrict__ force,
                                                    double* __restrict__ epot) {
  constexpr int NW = NA_BLOCK / 32, NV = FORCE ? 4 : 1;
  const unsigned FULL = 0xffffffffu;
  __shared__ float4 tile[NA_TILE];
  __shared__ int queue[NW][64];
  __shared__ double part[NW / 2][NV];
  const int warp = threadIdx.x >> 5, ln = threadIdx.x & 31, half = warp & 1;
  const unsigned lt = (1u << ln) - 1u;
  const int first = blockIdx.x * (NW / 2);
  const int i = first + (warp >> 1), ic = min(i, n - 1);
  const double3 x0 = make_double3(x[3 * first], x[3 * first + 1], x[3 * first + 2]);
  const float eps = 2.4e-7f;  // > 2^-22
  const float Lx = B.pbc[0] ? (float)B.L[0] : 3e38f, Ly = B.pbc[1] ? (float)B.L[1] : 3e38f,
              Lz = B.pbc[2] ? (float)B.L[2] : 3e38f;
  float4 ri = na_record(B, x, ic, x0);
  ri.w = fmaf(eps, ri.w, (float)c.rce * (1.0f + 1e-6f));
  const double ebi = FORCE ? scratch[NA_MAX + ic] : 0.0;
  int* const q = queue[warp];
  int cnt = 0;
  double sum[NV] = {};
  // the exact pair with the queue's entry of this lane
  auto eval = [&](bool on) {
    const int j = on ? q[ln] : ic;
    double v0, v1, v2, rinv;
    na_vd(B, x, ic, j, v0, v1, v2);
    const double n2 = v0 * v0 + v1 * v1 + v2 * v2;
    const double dr = gg::sqrt_pos(n2, rinv);
    const bool off = !on || dr > c.rce || n2 > 1e300;  // sqrt_pos has no infinities
    const double d = dr - c.rce, d2 = d * d, d3 = d2 * d;
    const double P = fma(fma(c.b1, d, c.b2), d, c.b3) * d3;
    const double e2 = gg::sm_exp(c, fma(c.kq, dr, c.q2));
    if constexpr (!FORCE) {
      const double banda = dr < c.rci ? c.eps2 * e2 : P * P;
      sum[0] += off ? 0.0 : banda;
    } else {
      const double ebs = ebi + scratch[NA_MAX + j];
      const double e1 = gg::sm_exp(c, fma(c.kp, dr, c.p));
      const double dPe = fma(fma(c.dp5, d, c.dp4), d, c.dp3) * d2;
      const double dRe = fma(fma(c.dr5, d, c.dr4), d, c.dr3) * d2;
      const bool inner = dr <= c.rci;
      const double factor = inner ? c.c1e * e1 - c.c2e * e2 * ebs : P * dPe * ebs - dRe;  // with ev_ui
      const double repul = inner ? c.A * e1 : fma(fma(c.r1, d, c.r2), d, c.r3) * d3;
      const double fr = factor * rinv;
      sum[0] -= off ? 0.0 : fr * v0;
      sum[1] -= off ? 0.0 : fr * v1;
      sum[2] -= off ? 0.0 : fr * v2;
      sum[3] += off ? 0.0 : repul;
    }
  };
  for (int t0 = 0; t0 < n; t0 += NA_TILE) {
    __syncthreads();
    for (int k = threadIdx.x; k < NA_TILE; k += NA_BLOCK)
      tile[k] = t0 + k < n ? na_record(B, x, t0 + k, x0) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    __syncthreads();
    const int nt = min(NA_TILE, n - t0), self = i - t0;
    // the halves of a pair take alternate runs of 32 NA_UNR candidates
    for (int k = 32 * NA_UNR * half; k < nt; k += 64 * NA_UNR) {
      bool in[NA_UNR];
      unsigned bal[NA_UNR], any = 0;
#pragma unroll
      for (int u = 0; u < NA_UNR; u++) {
        const int e = k + 32 * u + ln;
        const float4 a = tile[e];
        float dx = fabsf(a.x - ri.x), dy = fabsf(a.y - ri.y), dz = fabsf(a.z - ri.z);
        dx = fminf(dx, Lx - dx);  // the records' difference is within L: one image at most
        dy = fminf(dy, Ly - dy);
        dz = fminf(dz, Lz - dz);
        const float t = fmaf(eps, a.w, ri.w);
        // NaN passes: the exact test decides
        in[u] = !(fmaf(dz, dz, fmaf(dy, dy, dx * dx)) >= t * t) && e < nt && e != self;
        bal[u] = __ballot_sync(FULL, in[u]);
        any |= bal[u];
      }
      if (!any) continue;  // uniform
#pragma unroll
      for (int u = 0; u < NA_UNR; u++) {
        if (in[u]) q[cnt + __popc(bal[u] & lt)] = t0 + k + 32 * u + ln;
        cnt += __popc(bal[u]);
        if (cnt >= 32) {
          __syncwarp();
          eval(true);
          const int rest = q[32 + ln];
          __syncwarp();
          q[ln] = rest;
          cnt -= 32;
        }
      }
    }
  }
  __syncwarp();
  if (cnt) eval(ln < cnt);
#pragma unroll
  for (int k = 0; k < NV; k++)
    for (int o = 16; o; o >>= 1) sum[k] += __shfl_xor_sync(FULL, sum[k], o);
  if (half && ln == 0)
    for (int k = 0; k < NV; k++) part[warp >> 1][k] = sum[k];
  __syncthreads();
  if (half || ln || i >= n) return;
  for (int k = 0; k < NV; k++) sum[k] += part[warp >> 1][k];
  if constexpr (!FORCE) {
    scratch[i] = sum[0];  // every entry < n is written: no clearing
    scratch[NA_MAX + i] = 1.0 / sqrt(sum[0]);
  } else {
    force[3 * i] = sum[0];
    force[3 * i + 1] = sum[1];
    force[3 * i + 2] = sum[2];
    epot[i] = (sum[3] - sqrt(scratch[i])) * EV_UI;
  }
}

}  // namespace

extern "C" int gemsgpu_smatb_forces_noalloc(const double* d_pos, int n, int boxed, const double L[3],
                                            const int pbc[3], double A, double xi, double p, double q,
                                            double r0, double rci, double rce, double* d_force,
                                            double* d_epot, void* stream) {
  if (!d_pos || !d_force || !d_epot || n <= 0) return GEMSGPU_ERR_ARG;
  if (n > NA_MAX) return GEMSGPU_ERR_FULL;
  if (!(rce > rci) || !(r0 > 0.0)) return GEMSGPU_ERR_ARG;
  NaBox B{};
  for (int k = 0; k < 3; k++) {
    bool per = boxed && L && pbc && pbc[k];
    if (per && !(L[k] > 0.0)) return GEMSGPU_ERR_ARG;
    B.pbc[k] = per ? 1 : 0;
    B.L[k] = per ? L[k] : 0.0;
    B.invL[k] = per ? 1.0 / L[k] : 0.0;
  }
  // smatb_set tail coefficients (Logsdail et al. 2012)
  gg::PairP P{};
  const double dcut = rce - rci;
  const double ab = -1.0 / (dcut * dcut * dcut);
  double bb = -(q / r0) / (dcut * dcut);
  double cb = -((q / r0) * (q / r0)) / dcut;
  double aux = xi * std::exp(-q * (rci / r0 - 1.0));
  P.v[7] = aux * (12.0 * ab - 6.0 * bb + cb) / (2.0 * (dcut * dcut));
  P.v[8] = aux * (15.0 * ab - 7.0 * bb + cb) / dcut;
  P.v[9] = aux * (20.0 * ab - 8.0 * bb + cb) / 2.0;
  aux = A * std::exp(-p * (rci / r0 - 1.0));
  bb = -(p / r0) / (dcut * dcut);
  cb = -((p / r0) * (p / r0)) / dcut;
  P.v[10] = aux * (12.0 * ab - 6.0 * bb + cb) / (2.0 * (dcut * dcut));
  P.v[11] = aux * (15.0 * ab - 7.0 * bb + cb) / dcut;
  P.v[12] = aux * (20.0 * ab - 8.0 * bb + cb) / 2.0;
  P.v[0] = A; P.v[1] = xi; P.v[2] = p; P.v[3] = q; P.v[4] = r0; P.v[5] = rci; P.v[6] = rce;
  gg::SmFP64 c = gg::sm_load(P);
  double* scratch = nullptr;
  if (scratch_address(&scratch) != cudaSuccess) return GEMSGPU_ERR_CUDA;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const dim3 grid((n + NA_BLOCK / 64 - 1) / (NA_BLOCK / 64)), block(NA_BLOCK);
  // cudaLaunchKernel returns this launch's own status, so an error left
  // behind by the caller's earlier work is not reported as this call's
  void* args[] = {(void*)&d_pos, (void*)&n, (void*)&B, (void*)&c, (void*)&scratch, (void*)&d_force, (void*)&d_epot};
  for (const void* fn : {(const void*)k_na<false>, (const void*)k_na<true>})
    if (cudaLaunchKernel(fn, grid, block, args, 0, st) != cudaSuccess) return GEMSGPU_ERR_CUDA;
  return GEMSGPU_OK;
}
