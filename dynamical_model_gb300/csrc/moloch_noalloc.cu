// WAF advection of one field that allocates no device memory
// (moloch_gpu_wafone_noalloc in include/moloch_gb300.h).
//
// Who needs it: callers that own every byte of device memory themselves --
// a Fortran model whose arrays live in its own CUDA/OpenACC data regions, or
// a host framework running its own memory pool -- and therefore cannot let a
// library call cudaMalloc (which can synchronise the device, fragment or
// exceed the caller's pool, or fail in a process that has already reserved
// the GPU's memory).  They pass device pointers for the inputs and the
// output; the two work arrays of wafone (wz, p0) live in a fixed
// file-scope __device__ array instead of being allocated.
//
// The arithmetic is that of wafone (nompi/mod_moloch.F90:929-1311) with the
// metric factors computed inline from fmz, fmzf and the map factors; this
// file is compiled without multiply-add contraction, so its results are the
// same as the advection phase of the exact FP64 build.
#define MOLOCH_KNS knoalloc
#include <cstdio>
#include <mutex>

#include "../../include/moloch_gb300.h"
#include "moloch_kernels.cuh"

extern "C" void moloch_internal_set_error(const char* msg);

namespace moloch {
namespace knoalloc {

// Largest jx*iy*kz a call may pass: 2^21 points.  Scratch = wz + p0 =
// 2 * 2^21 doubles = 32 MiB.  The CUDA runtime reserves it on a device when
// it loads this file's device code there -- with lazy module loading (the
// default), during the first call on that device, which looks the array up
// -- and holds it until the process exits.
constexpr long long kMaxPoints = 1LL << 21;
static __device__ __align__(256) double g_scratch[2 * kMaxPoints];

struct NaArgs {
  double* pp;
  const double* s;
  const double* u;
  const double* v;
  const double* fmz;
  const double* fmzf;
  const double* mu;
  const double* mv;
  const double* mx;
  double* wz;
  double* p0;
  int nj, ni, kz;
  double dtrdx, dtrdy, dtrdz;
  int rotllr;
};

// What bounds these kernels: the FP64 pipe (two lanes an SM and clock, 16
// clocks a warp instruction), not the 9 words of traffic a point.  So every
// flux, every reciprocal of a metric and every 1 / m of the map factors is
// computed once and handed on -- down the march, through shared memory or
// over the levels of a thread -- and comparisons, selects and signs run on
// the integer pipe.  FP64 instructions a point, both fluxes and every metric
// factor taken at each point -> now: vertical 112 -> 87, meridional 103 -> 68,
// zonal 90 -> 51, at 81-87 % of the pipe; one call at 160 x 128 x 64 1060 ->
// 550 us, 64 x 48 x 30 226 -> 86 us, 200 x 190 x 20 574 -> 349 us, bit for bit
// the same results.

// horizontal flux (:1088-1104); dm, d0, dp: the differences x(i) - x(i-1) at
// the face before, this one and the next
__device__ __forceinline__ double na_hflux(double zamu, double dm, double d0, double dp, double m1, double x0) {
  const bool up = __double_as_longlong(zamu) > 0;
  return waf_flux_rn(up, zamu, up ? dm : dp, d0, m1, x0);
}
// flux through the lower face of x1 (:966-1012); d0, d1, d2: x(k) - x(k+1)
// above x1, below it and below x2
__device__ __forceinline__ double na_vflux(double s1, double zamu, double d0, double d1, double d2, double x1, double x2) {
  const long long z = __double_as_longlong(zamu);
  const bool up = z >= 0 || z == (long long)0x8000000000000000ULL;
  return half_of(s1) * waf_flux_rn(up, zamu, up ? d2 : d0, d1, x2, x1);
}

// Both vertical passes (:966-1072).  A warp holds 32 columns and up to
// kNaLevels levels of them, the warps of a block one after the other down the
// column, so that 1 / fmzf is taken once a face and the metric factors of the
// first pass stay in registers for the second; what the passes exchange goes
// through shared memory.  Four to eight levels a warp measure the same within
// 5 %; two take 12 % more (the first flux of a warp is taken twice).  Columns
// deeper than kNaWarps kNaLevels march with one thread each
// (k_na_vertical_deep), which takes every metric factor twice.
constexpr int kNaLevels = 6, kNaWarps = 12;
__global__ void __launch_bounds__(32 * kNaWarps) k_na_vertical(NaArgs a) {
  extern __shared__ double sx[];  // [kz][32]
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const size_t pl = (size_t)a.nj * a.ni, cc = (size_t)blockIdx.x * 32 + lane, c = cc < pl ? cc : pl - 1;
  const int kz = a.kz, lv = (kz + nw - 1) / nw, k0 = w * lv, k1 = min(k0 + lv, kz);
  for (int k = k0; k < k1; ++k) sx[k * 32 + lane] = a.pp[c + k * pl];
  __syncthreads();
  double zu[kNaLevels], zd[kNaLevels], dv[kNaLevels], xo[kNaLevels];
  auto X = [&](int k) { return sx[min(max(k, 0), kz - 1) * 32 + lane]; };
#pragma unroll 1
  for (int pass = 0; pass < 2; ++pass) {
    if (k0 < k1) {
      RcpRn r0;
      if (pass == 0) r0 = rcp_rn_of(a.fmzf[c + k0 * pl]);
      double x1 = X(k0), x2 = X(k0 + 1), d0 = X(k0 - 1) - x1, d1 = x1 - x2;
      double s0 = a.s[c + k0 * pl], w0 = 0.0;
      if (k0 > 0) w0 = na_vflux(s0, s0 * a.dtrdz, X(k0 - 2) - X(k0 - 1), d0, d1, X(k0 - 1), x1);
#pragma unroll
      for (int n = 0; n < kNaLevels; ++n) {
        const int k = k0 + n;
        if (k < k1) {
          const double s1 = a.s[c + (k + 1) * pl], x3 = X(k + 2), d2 = x2 - x3;
          const double w1 = k < kz - 1 ? na_vflux(s1, s1 * a.dtrdz, d0, d1, d2, x1, x2) : 0.0;
          if (pass == 0) {
            const double f = a.dtrdz * a.fmz[c + k * pl];
            const RcpRn r1 = rcp_rn_of(a.fmzf[c + (k + 1) * pl]);
            zu[n] = quot_rn(f, r0);
            zd[n] = quot_rn(f, r1);
            dv[n] = s0 * zu[n] - s1 * zd[n];
            r0 = r1;
          }
          xo[n] = ((x1 - w0 * zu[n]) + w1 * zd[n]) + dv[n] * x1;
          x1 = x2; x2 = x3; d0 = d1; d1 = d2; w0 = w1; s0 = s1;
        }
      }
    }
    __syncthreads();  // every warp has read what the others overwrite
#pragma unroll
    for (int n = 0; n < kNaLevels; ++n)
      if (k0 + n < k1) {
        if (pass == 0) sx[(k0 + n) * 32 + lane] = xo[n];
        else if (cc < pl) a.wz[c + (k0 + n) * pl] = xo[n];
      }
    __syncthreads();
  }
}

// one pass down a whole column (:966-1020 / :1022-1072)
__device__ void na_vpass(const double* src, double* dst, const NaArgs& a, size_t c) {
  const size_t pl = (size_t)a.nj * a.ni;
  const int kz = a.kz;
  double x1 = src[c], x2 = src[c + pl], d0 = 0.0, d1 = x1 - x2;
  double w0 = 0.0, s0 = a.s[c];
  RcpRn r0 = rcp_rn_of(a.fmzf[c]);
  for (int k = 0; k < kz; ++k) {
    const size_t o = c + k * pl;
    const double s1 = a.s[o + pl], x3 = src[c + min(k + 2, kz - 1) * pl], d2 = x2 - x3;
    const double w1 = k < kz - 1 ? na_vflux(s1, s1 * a.dtrdz, d0, d1, d2, x1, x2) : 0.0;
    const double f = a.dtrdz * a.fmz[o];
    const RcpRn r1 = rcp_rn_of(a.fmzf[o + pl]);
    const double zu = quot_rn(f, r0), zd = quot_rn(f, r1);
    dst[o] = ((x1 - w0 * zu) + w1 * zd) + (s0 * zu - s1 * zd) * x1;
    x1 = x2; x2 = x3; d0 = d1; d1 = d2; w0 = w1; s0 = s1; r0 = r1;
  }
}
__global__ void __launch_bounds__(128) k_na_vertical_deep(NaArgs a) {
  const size_t c = (size_t)blockIdx.x * 128 + threadIdx.x;
  if (c >= (size_t)a.nj * a.ni) return;
  na_vpass(a.pp, a.wz, a, c);
  na_vpass(a.wz, a.wz, a, c);
}

// Meridional flux + update (:1080-1131).  A thread marches kNaRows rows of
// one column: the flux, the reciprocal of fmz(i) + fmz(i+1) and 1 / mv of a
// face serve both its rows (four rows against 6, 8 and 16: 585, 591, 590 and
// 611 us a call at 160 x 128 x 64, 84, 82, 87 and 112 at 64 x 48 x 30; two or
// four levels a thread leave too few warps there, 108 and 157).
constexpr int kNaRows = 4;
__global__ void __launch_bounds__(128) k_na_meridional(NaArgs a) {
  const int nj = a.nj, ni = a.ni, strips = (ni + kNaRows - 1) / kNaRows;
  const int t = blockIdx.x * 128 + threadIdx.x;
  if (t >= nj * strips) return;
  const int jj = t % nj, i0 = (t / nj) * kNaRows, i1 = min(i0 + kNaRows, ni);
  const size_t pl = (size_t)nj * ni;
  const size_t ko = blockIdx.y * pl + jj;
  auto row = [&](int i) { return (size_t)nj * wrap2(i, ni); };
  auto face = [&](double v, double rm, double dm, double d0, double dp, double m1, double x0) {  // zpby
    const double vr = a.rotllr ? v : v * rm;
    const double fl = na_hflux(vr * a.dtrdy, dm, d0, dp, m1, x0);
    return a.rotllr ? half_of(v) * fl : (half_of(v) * rm) * fl;
  };
  double rms = inv_rn(a.mv[row(i0) + jj]);
  const double m2 = a.wz[ko + row(i0 - 2)], m1 = a.wz[ko + row(i0 - 1)];
  double x1 = a.wz[ko + row(i0)], x2 = a.wz[ko + row(i0 + 1)], d0 = x1 - m1, d1 = x2 - x1;
  double vs = a.v[ko + row(i0)], fc = a.fmz[ko + row(i0)];
  double zs = face(vs, rms, m1 - m2, d0, d1, m1, x1);
  RcpRn rs = rcp_rn_of(fc + a.fmz[ko + row(i0 - 1)]);
  const double dt2 = a.dtrdy * 2.0;  // (c m) 2 f rounds as ((2 c) m) f
#pragma unroll 1
  for (int i = i0; i < i1; ++i) {
    const size_t rc = row(i), rn = row(i + 1), rnn = row(i + 2);
    const double rmn = inv_rn(a.mv[rn + jj]), mxx = a.mx[rc + jj];
    const double hn = a.rotllr ? (dt2 * rmn) * mxx : mxx * mxx, hs = a.rotllr ? (dt2 * rms) * mxx : 0.0;
    const double x3 = a.wz[ko + rnn], vn = a.v[ko + rn], fn = a.fmz[ko + rn], pp = a.pp[ko + rc];
    const double d2 = x3 - x2, zn = face(vn, rmn, d0, d1, d2, x1, x2);
    const RcpRn r = rcp_rn_of(fc + fn);
    double p0;
    if (a.rotllr) {
      const double zrfmn = quot_rn(hn * fc, r), zrfms = quot_rn(hs * fc, rs);
      const double zdv = (vn * zrfmn - vs * zrfms) * pp;
      p0 = ((x1 + zs * zrfms) - zn * zrfmn) + zdv;
    } else {
      const double h = dt2 * fc;
      const double zrfmn = quot_rn(h, r), zrfms = quot_rn(h, rs);
      const double zdv = ((vn * rmn) * zrfmn - (vs * rms) * zrfms) * pp;
      p0 = x1 + hn * (((zs * zrfms) - zn * zrfmn) + zdv);
    }
    a.p0[ko + rc] = p0;
    x1 = x2; x2 = x3; d0 = d1; d1 = d2; fc = fn; vs = vn; zs = zn; rs = r;
    rms = rmn;
  }
}

// Zonal flux + update of pp (:1138-1187).  A thread takes one western face
// and one point of kNaZonK levels; faces go to the points through shared
// memory.  A block holds `rows` whole rows of nj points, or one segment of a
// row (one face more than points) where nj is above kNaSeg.
constexpr int kNaSeg = 256, kNaZonK = 2;
__global__ void __launch_bounds__(kNaSeg) k_na_zonal(NaArgs a, int rows, int len, int faces, int segs) {
  __shared__ double sz[kNaZonK][kNaSeg], sy[kNaZonK][kNaSeg], sb[kNaZonK][kNaSeg], sm[kNaSeg];
  __shared__ bool sk[kNaZonK][kNaSeg];
  const int nj = a.nj, ni = a.ni, t = threadIdx.x;
  const size_t pl = (size_t)nj * ni;
  const int r = t / faces, jf = t - r * faces;
  const int ii = (blockIdx.x / segs) * rows + r, j0 = (blockIdx.x % segs) * len;
  const int jp = j0 + jf;  // nj itself is the face 0 of the next image
  const bool face = r < rows && ii < ni && jp <= nj;
  const size_t row = (size_t)nj * ii;
  const int kk = blockIdx.y * kNaZonK, nk = min(kNaZonK, a.kz - kk);
  const int jc = wrap2(jp, nj), jm = wm1(jc, nj), jm2 = wm1(jm, nj), je = wp1(jc, nj);
  double x1[kNaZonK], fc[kNaZonK], uw[kNaZonK];
  if (face) {
    const double mu = a.mu[row + jc], m = a.rotllr ? mu : inv_rn(mu);
    sm[t] = m;
#pragma unroll
    for (int n = 0; n < kNaZonK; ++n) {
      const size_t o = (size_t)(kk + min(n, nk - 1)) * pl + row;
      const double u = a.u[o + jc], xw = a.p0[o + jm];
      x1[n] = a.p0[o + jc];
      fc[n] = a.fmz[o + jc];
      uw[n] = u;
      const double zamu = (u * m) * a.dtrdx;
      const bool up = __double_as_longlong(zamu) > 0;
      const double num = (up ? xw : a.p0[o + je]) - (up ? a.p0[o + jm2] : x1[n]);
      const double fl = waf_flux_rn(up, zamu, num, x1[n] - xw, xw, x1[n]);
      sz[n][t] = a.rotllr ? half_of(u) * fl : (half_of(u) * m) * fl;
      const RcpRn y = rcp_rn_of(fc[n] + a.fmz[o + jm]);
      sb[n][t] = y.b;
      sy[n][t] = y.y;
      sk[n][t] = y.ok;
    }
  }
  __syncthreads();
  if (!face || jf >= len || jp >= nj) return;
  const int e = (faces == nj && jf == nj - 1) ? t - jf : t + 1;  // the eastern face
  const double m = sm[t], me = sm[e], mx = a.mx[row + jc], dt2 = a.dtrdx * 2.0;
#pragma unroll
  for (int n = 0; n < kNaZonK; ++n) {
    if (n >= nk) break;
    const size_t o = (size_t)(kk + n) * pl + row;
    const double ue = a.u[o + je], pp = a.pp[o + jc];
    const RcpRn re = {sb[n][e], sy[n][e], sk[n][e]}, rw = {sb[n][t], sy[n][t], sk[n][t]};
    double out;
    if (a.rotllr) {
      const double h = (dt2 * m) * fc[n];
      const double zrfme = quot_rn(h, re), zrfmw = quot_rn(h, rw);
      const double zdv = (ue * zrfme - uw[n] * zrfmw) * pp;
      out = ((x1[n] + sz[n][t] * zrfmw) - sz[n][e] * zrfme) + zdv;
    } else {
      const double h = dt2 * fc[n];
      const double zrfme = quot_rn(h, re), zrfmw = quot_rn(h, rw);
      const double zdv = ((ue * me) * zrfme - (uw[n] * m) * zrfmw) * pp;
      out = x1[n] + (mx * mx) * (((sz[n][t] * zrfmw) - sz[n][e] * zrfme) + zdv);
    }
    a.pp[o + jc] = out;
  }
}

// device address of g_scratch, looked up once per device
constexpr int kMaxDevices = 64;
static double* g_scratch_ptr[kMaxDevices];
static std::mutex g_scratch_mu;

}  // namespace knoalloc
}  // namespace moloch

extern "C" int moloch_gpu_wafone_noalloc(double* pp, const double* s, const double* u, const double* v,
                                         const double* fmz, const double* fmzf, const double* msfu,
                                         const double* msfv, const double* msfx, int jx, int iy, int kz,
                                         double dta, double dx, double dzita, int rotllr, void* stream) {
  using namespace moloch::knoalloc;
  if (!pp || !s || !u || !v || !fmz || !fmzf || !msfu || !msfv || !msfx) {
    moloch_internal_set_error("wafone_noalloc: null pointer");
    return MOLOCH_ERR_ARG;
  }
  if (jx < 4 || iy < 4 || kz < 4) {
    moloch_internal_set_error("wafone_noalloc: jx, iy and kz must be >= 4");
    return MOLOCH_ERR_ARG;
  }
  if (kz > 65535) {  // the meridional kernel takes k as gridDim.y, the zonal one kz / 2
    moloch_internal_set_error("wafone_noalloc: kz must be <= 65535");
    return MOLOCH_ERR_ARG;
  }
  if ((long long)jx * iy * kz > kMaxPoints) {
    char buf[200];
    snprintf(buf, sizeof buf, "wafone_noalloc: jx*iy*kz = %lld exceeds the fixed scratch of %lld points",
             (long long)jx * iy * kz, kMaxPoints);
    moloch_internal_set_error(buf);
    return MOLOCH_ERR_ARG;
  }
  if (!(dta > 0) || !(dx > 0) || !(dzita > 0)) {
    moloch_internal_set_error("wafone_noalloc: dta, dx and dzita must be positive");
    return MOLOCH_ERR_ARG;
  }
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || dev < 0 || dev >= kMaxDevices) {
    moloch_internal_set_error("wafone_noalloc: no current CUDA device");
    return MOLOCH_ERR_CUDA;
  }
  double* scratch;
  {
    std::lock_guard<std::mutex> lk(g_scratch_mu);
    if (!g_scratch_ptr[dev]) {  // set-up on the first call on this device
      void* p = nullptr;
      e = cudaGetSymbolAddress(&p, g_scratch);
      if (e != cudaSuccess || !p) {
        moloch_internal_set_error(cudaGetErrorString(e));
        return MOLOCH_ERR_CUDA;
      }
      g_scratch_ptr[dev] = (double*)p;
    }
    scratch = g_scratch_ptr[dev];
  }
  NaArgs a;
  a.pp = pp; a.s = s; a.u = u; a.v = v; a.fmz = fmz; a.fmzf = fmzf;
  a.mu = msfu; a.mv = msfv; a.mx = msfx;
  const size_t n = (size_t)jx * iy * kz;
  a.wz = scratch;      // fully written by k_na_vertical before it is read
  a.p0 = scratch + n;  // fully written by k_na_meridional before it is read
  a.nj = jx; a.ni = iy; a.kz = kz;
  a.dtrdx = dta / dx;  // wafone :951-956
  a.dtrdy = dta / dx;
  a.dtrdz = 0.5 * (dta / dzita);
  a.rotllr = rotllr;
  cudaStream_t st = (cudaStream_t)stream;
  // each launch's own status: cudaGetLastError here would also return (and
  // clear) an error the caller left pending before this call
  void* args[] = {&a};
  const int pl = jx * iy;
  // fewest warps that hold the column, at most kNaLevels levels each
  const int nw = (kz + kNaLevels - 1) / kNaLevels;
  if (nw <= kNaWarps)
    e = cudaLaunchKernel((const void*)k_na_vertical, dim3((pl + 31) / 32), dim3(32 * nw), args, (size_t)kz * 32 * 8, st);
  else
    e = cudaLaunchKernel((const void*)k_na_vertical_deep, dim3((pl + 127) / 128), dim3(128), args, 0, st);
  const int strips = (iy + kNaRows - 1) / kNaRows;
  if (e == cudaSuccess)
    e = cudaLaunchKernel((const void*)k_na_meridional, dim3((jx * strips + 127) / 128, kz),
                         dim3(128), args, 0, st);
  int rows = 1, len = jx, faces = jx, segs = 1;
  if (jx > kNaSeg) {
    segs = (jx + kNaSeg - 2) / (kNaSeg - 1);
    len = (jx + segs - 1) / segs;
    faces = len + 1;
  } else {
    rows = kNaSeg / jx < iy ? kNaSeg / jx : iy;
  }
  void* zargs[] = {&a, &rows, &len, &faces, &segs};
  if (e == cudaSuccess)
    e = cudaLaunchKernel((const void*)k_na_zonal, dim3((iy + rows - 1) / rows * segs, (kz + kNaZonK - 1) / kNaZonK),
                         dim3((rows * faces + 31) / 32 * 32), zargs, 0, st);
  if (e != cudaSuccess) {
    moloch_internal_set_error(cudaGetErrorString(e));
    return MOLOCH_ERR_CUDA;
  }
  return MOLOCH_OK;
}
