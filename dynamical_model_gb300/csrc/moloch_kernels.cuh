// MOLOCH step kernels for sm_103a.  Included by one .cu file per arithmetic
// build (MOLOCH_KNS names the namespace): the exact FP64 build is compiled
// with --fmad=false so every expression keeps the reference's evaluation
// order; the fast build allows multiply-add contraction and also carries the
// FP32-storage instantiation.
//
// Kernel map (reference: nompi/mod_moloch.F90):
//   k_prediag          :289-323  p, qsat, tvirt, qwltot, qwitot, tetav
//   k_sound_div        :514-597  u/v halo + surface w + s (Eq. 10) + zdiv2 (Eq. 16)
//   k_sound_damp       :853-895 + :627-630  divdamp and the vertical s term
//   k_sound_column     :634-728  implicit w (Thomas; one thread per column, a block
//                      per 8 to 32 columns (_split, FP64), or staged by TMA (_tw, FP32)),
//                      Exner/theta update, nompi pai halo order, s completion (:843-849)
//   k_divdamp_quad, _strip  div and damp in one pass (FP32)
//   k_lap_filter       :423-440 divergence_filter (mo_divfilter)
//   k_pai_update       :716-728 (split form used when the filter is on)
//   k_sound_momentum   :730-837  Equations 17, 18
//   k_waf_vertical     :966-1073  both vertical WAF passes in registers, all 10 fields
//                      (_pair: two columns per thread, FP32),
//                      with (u,v,w) -> (ux,vx,wx) of :1327-1341, :1389-1417 formed on the fly
//   k_waf_horizontal   :1075-1187 meridional + zonal WAF of one level, p0 in shared memory
//                      (_hstrip: warp strips; _hpair: strips of two columns a lane, FP32)
//   k_stag_from_x      :1343-1387  (ux,vx,wx) -> (u,v,w)
//   k_filter_increment :442-481 + :333-353 filtpai / filttheta
//   k_postdiag         :355-391  tvirt, t, p, rho, ps, qsat
//   k_diag_*           :395-411  max/min of ps, u, v; NaN/Inf check; FP64 column sums
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <atomic>
#include <cstdint>
#include <type_traits>

#include "moloch_constants.h"
#include "moloch_device.h"
#include "moloch_view.h"

#ifndef MOLOCH_KNS
#error "MOLOCH_KNS must name the namespace of this kernel build"
#endif

namespace moloch {
namespace MOLOCH_KNS {

constexpr int kColBX = 32;  // column kernels: 32 j x 4 i threads
constexpr int kColBY = 4;
constexpr int kPtBX = 32;   // point kernels: 32 j x 8 i threads
constexpr int kPtBY = 8;

template <class T>
struct FieldPtrs {
  T* f[kNumAdvected];
};

// block-cooperative copy of a member's view into shared memory (batched kernels)
template <class V>
__device__ __forceinline__ void copy_view(V* dst, const V* __restrict__ src) {
  static_assert(sizeof(V) % 4 == 0, "view size");
  const int n = (int)(sizeof(V) / 4);
  const int nt = blockDim.x * blockDim.y;
  for (int q = threadIdx.x + blockDim.x * threadIdx.y; q < n; q += nt)
    reinterpret_cast<int*>(dst)[q] = reinterpret_cast<const int*>(src)[q];
}

// The contracting builds' FP64 arithmetic is written for few FP64 operations
// (MOLOCH_LEAN_FP64): GB300 has two FP64 lanes an SM and every FP64 kernel of
// the step is bound by them (82-85 % of the pipe busy at 10-25 % of DRAM), so
// each expression folds what is static into stored terms, divides through an
// FP32 estimate and leaves sign, order and scaling to the integer pipe.  The
// exact build keeps the reference's expressions, FP32 storage its own.
#if defined(MOLOCH_LEAN_FP64)
template <class T> constexpr bool kLean = sizeof(T) == 8;
#else
template <class T> constexpr bool kLean = false;
#endif

// ---- small device helpers ---------------------------------------------
__device__ __forceinline__ float fma_rn(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fma_rn(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float add_rn(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double add_rn(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float sub_rn(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ double sub_rn(double a, double b) { return __dsub_rn(a, b); }
// Point of a thread in the plane: tile (bx, by) of BX x BY points or, by < 0,
// the bx-th BX BY points of the plane in order.  FP64 kernels take the plane
// in order where whole warps a row leave a tenth of the lanes idle: they are
// bound by the FP64 pipe, whose 16 clocks a warp instruction do not shrink
// with idle lanes (a row of 100 columns is four warps instead of 3.1).  Per
// step, rows | in order: 100 x 100 x 30 vertical WAF 0.492 | 0.382 ms, momentum
// 0.499 | 0.407, divergence 0.284 | 0.249, damping 0.283 | 0.240; 203 x 157 x 45
// momentum 1.61 | 1.44.  Not worth it where rows fill (150 x 140 x 40, 6 % idle:
// divergence 0.466 | 0.488) or launches bound (24 x 20 x 12: 0.112 | 0.119).
template <int BX, int BY, class T>
__device__ __forceinline__ void point_at(const View<T>& d, const int bx, const int by, int& jj, int& ii) {
  if (sizeof(T) == 8 && by < 0) {
    const unsigned q = bx * (BX * BY) + threadIdx.y * BX + threadIdx.x;
    ii = q / (unsigned)d.nj;
    jj = q - ii * d.nj;
  } else {
    jj = bx * BX + threadIdx.x;
    ii = by * BY + threadIdx.y;
  }
}
template <class T>
__host__ __device__ __forceinline__ bool in_order(const View<T>& d) {
  const int padded = (d.nj + 31) / 32 * 32;
  return sizeof(T) == 8 && d.pl >= 4096 && 10 * padded >= 11 * d.nj;
}
template <class T>
__device__ __forceinline__ int tile_y(const View<T>& d) {
  return in_order(d) ? -1 : (int)blockIdx.y;
}

// Two FP32 values in one 64-bit register pair: sm_103a adds, multiplies and
// fuses both in one instruction, each rounded as alone.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float a, float b) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ f32x2 pack2(float2 a) { return pack2(a.x, a.y); }
__device__ __forceinline__ float2 unpack2(f32x2 a) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a));
  return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 sub2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ int wm1(int x, int n) { return x == 0 ? n - 1 : x - 1; }
__device__ __forceinline__ int wp1(int x, int n) { return x == n - 1 ? 0 : x + 1; }
__device__ __forceinline__ int wm2(int x, int n) { int y = x - 2; return y < 0 ? y + n : y; }
__device__ __forceinline__ int wp2(int x, int n) { int y = x + 2; return y >= n ? y - n : y; }

// a*b - c*d and a*b + c*d with the multiply-add contraction fixed in the builds
// that contract: left to the compiler either product may be fused, and which
// one it fuses depends on the code around the expression, so the same body in
// two kernels (k_sound_column and k_sound_column_tw; a batched kernel and
// the persistent ensemble kernel) could round differently.  The exact build
// contracts nothing.
__device__ __forceinline__ float prod_sub(float a, float b, float c, float d) { return __fmaf_rn(a, b, -__fmul_rn(c, d)); }
__device__ __forceinline__ float prod_add(float a, float b, float c, float d) { return __fmaf_rn(c, d, __fmul_rn(a, b)); }
#if defined(MOLOCH_LEAN_FP64)
__device__ __forceinline__ double prod_sub(double a, double b, double c, double d) { return __fma_rn(a, b, -__dmul_rn(c, d)); }
__device__ __forceinline__ double prod_add(double a, double b, double c, double d) { return __fma_rn(c, d, __dmul_rn(a, b)); }
#else
__device__ __forceinline__ double prod_sub(double a, double b, double c, double d) { return a * b - c * d; }
__device__ __forceinline__ double prod_add(double a, double b, double c, double d) { return a * b + c * d; }
#endif
// the fourth-order average of the staggering (:1327-1417) of the inner pair's
// sum and the outer pair's, likewise fixed in FP64
__device__ __forceinline__ float average4(float inner, float outer) { return 0.5625f * inner - 0.0625f * outer; }
__device__ __forceinline__ double average4(double inner, double outer) { return prod_sub(0.5625, inner, 0.0625, outer); }
__device__ __forceinline__ int wrapn(int x, int n) { int y = x % n; return y < 0 ? y + n : y; }
// periodic index for -n <= x < 2n (no integer division)
__device__ __forceinline__ int wrap2(int x, int n) { return x < 0 ? x + n : (x >= n ? x - n : x); }

__device__ __forceinline__ double dexp(double a) { return exp(a); }
__device__ __forceinline__ float dexp(float a) { return expf(a); }

// Quotient of the WAF limiter ratio.  FP64 builds: the IEEE quotient, as
// the reference.  FP32 storage: the fast approximate quotient (2 ulp); the
// ratio only selects and scales the limiter, and the FP32 error is measured
// against the FP64 step anyway.  Written as the product with the estimate of
// 1 / b: the bits of __fdividef for 1e-30 <= |b| <= 1e6 and any |a| <= 1e6
// (compared on 2^30 seeded pairs, subnormal a included) without the
// instructions that rescale other b.
__device__ __forceinline__ float qdiv(float a, float b) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(b));
  return a * r;
}

// Exact FP32 -> FP64 widening on the integer pipe.  GB300 executes F2F
// conversions on its FP64 pipe (1/64 of the FP32 rate); these few integer
// operations do not touch it.  Zeros, normal values of either sign,
// infinities and NaNs convert exactly; FP32 subnormals become zero of the
// same sign.
__device__ __forceinline__ double widen_f32(float x) {
  const unsigned b = __float_as_uint(x);
  const unsigned ex = b & 0x7f800000u, sg = b & 0x80000000u;
  unsigned hi = (((b & 0x7fffffffu) >> 3) + 0x38000000u) | sg;  // exponent rebiased by 1023 - 127
  unsigned lo = b << 29;
  if (ex == 0u) { hi = sg; lo = 0u; }
  if (ex == 0x7f800000u) hi |= 0x7ff00000u;
  return __hiloint2double((int)hi, (int)lo);
}

// FP64 -> FP32 by truncation on the integer pipe: sign and exponent exact,
// mantissa cut to 23 bits (relative error < 2^-23).  Magnitudes below the
// FP32 normal range become zero, above it infinity; NaNs stay NaN.
__device__ __forceinline__ float narrow_trunc(double x) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  const unsigned ax = hi & 0x7fffffffu;
  unsigned m = (__funnelshift_l(lo, hi, 3) - (896u << 23)) & 0x7fffffffu;  // exponent rebiased by 127 - 1023
  if (ax < 0x38100000u) m = 0u;
  if (ax >= 0x47f00000u) m = (ax > 0x7ff00000u || (ax == 0x7ff00000u && lo != 0u)) ? 0x7fc00000u : 0x7f800000u;
  return __uint_as_float(m | (hi & 0x80000000u));
}


// ---- FP64 quotients and roots written out --------------------------------
// FP32 estimate of 1 / b for |b| in the FP32 normal range (relative error
// below 2^-21.9: the estimate's ulp and b cut to 23 bits)
__device__ __forceinline__ double rcp_seed(double b) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(narrow_trunc(b)));
  return widen_f32(r);
}
// |b| where the estimates below hold (between 2^-100 and 2^100), tested on
// the high word; false for zeros, infinities and NaN
__device__ __forceinline__ bool mid_range(double b) {
  const unsigned h = (unsigned)__double2hiint(b) & 0x7fffffffu;
  return h - 0x39b00000u < 0x46300000u - 0x39b00000u;
}
// 1 / b to half an ulp times 1 + 2^-11.6 (the estimate's third-order step,
// rounded), and whether quot_rn may use it.
struct RcpRn {
  double b, y;
  bool ok;
};
__device__ __forceinline__ RcpRn rcp_rn_of(double b) {
  RcpRn r;
  r.b = b;
  r.ok = mid_range(b) && (__double2hiint(b) & 0xffe00) != 0xffe00;
  const double x = rcp_seed(b), e = __fma_rn(-b, x, 1.0);
  r.y = __fma_rn(x, __fma_rn(e, e, e), x);
  return r;
}
// a / b, correctly rounded, with Markstein's quotient correction (P.
// Markstein, "IA-64 and Elementary Functions", 2000): q = a y is within 1.5
// ulp, the first residual takes it to half an ulp (1 + 2^-49), and the second
// is exact, so that what is rounded last differs from a / b by at most
// 2^-107 b (1 + 2^-11.5) where a >= b (a and b scaled to [1, 2)).  A quotient
// of two doubles is no nearer than 2^-105 / b to the middle of two doubles:
// the rounding is right while b < 2 (1 - 2^-12.5).  a < b halves both.  Other
// b, and |a| outside 2^-800 .. 2^800 but 0, divide as IEEE.  A zero's first
// product has the quotient's sign; the residuals would turn -0 into +0.
// Eight FP64 operations with the reciprocal.  (Two corrections of a y from the
// estimate itself are five, but only within an ulp, and make NaN of infinite
// and overflowing quotients.)
__device__ __forceinline__ double quot_rn(double a, const RcpRn& r) {
  const unsigned h = (unsigned)__double2hiint(a) & 0x7fffffffu;
  const bool zero = (h | (unsigned)__double2loint(a)) == 0u;
  if (!(r.ok && (zero || h - 0x0df00000u < 0x71f00000u - 0x0df00000u))) return a / r.b;
  const double q0 = mul_rn(a, r.y);
  double q = __fma_rn(__fma_rn(-r.b, q0, a), r.y, q0);
  q = __fma_rn(__fma_rn(-r.b, q, a), r.y, q);
  return zero ? q0 : q;
}
// 1 / b, correctly rounded (the same with q = y)
__device__ __forceinline__ double inv_rn(double b) {
  const RcpRn r = rcp_rn_of(b);
  return r.ok ? __fma_rn(__fma_rn(-b, r.y, 1.0), r.y, r.y) : 1.0 / b;
}
// the column pivots' reciprocal in the contracting build.  Without inv_rn's last
// correction it is two operations shorter but rounds one reciprocal in some
// thousands the other way than 1 / b (column solve at 256 x 256 x 60 5.74 ms per
// step, 5.99 now; 100 x 100 x 30 0.754, 0.785).
__device__ __forceinline__ double pivot_rcp(double b) { return inv_rn(b); }
// pai^3.5 = pai^3 sqrt(pai), the root by the coupled iteration for g =
// sqrt(a), h = 1 / (2 sqrt(a)) (Goldschmidt's, as in Markstein's book) from an
// FP32 estimate.  The root, its square's residual times h, the cube and the
// product are each carried in two words (products by the fused residual, T. J.
// Dekker, Numer. Math. 18, 1971), whose neglected terms are below 2^-80 of the
// value: half an ulp, where three rounded products reach 2.5 and pow 1.2 ulp.
// 16 FP64 operations where pow takes about seventy (256 x 256 x 60: k_prediag
// 0.93 -> 0.42 ms, k_postdiag 1.14 -> 0.47 ms).
__device__ __forceinline__ double pow35(double a) {
  static_assert(kCpovr == 3.5, "cp / R");
  if (!mid_range(a) || __double2hiint(a) < 0) return pow(a, kCpovr);
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(narrow_trunc(a)));
  double g = mul_rn(a, widen_f32(r)), h = widen_f32(0.5f * r);
  const double e = fma_rn(-g, h, 0.5);
  g = fma_rn(g, e, g);
  h = fma_rn(h, e, h);
  const double gl = mul_rn(fma_rn(-g, g, a), h);  // sqrt(a) - g
  const double s = mul_rn(a, a), c = mul_rn(s, a);
  const double cl = fma_rn(fma_rn(a, a, -s), a, fma_rn(s, a, -c));  // a^3 - c
  const double p = mul_rn(c, g);
  return add_rn(p, fma_rn(c, gl, fma_rn(cl, g, fma_rn(c, g, -p))));
}
#if defined(MOLOCH_LEAN_FP64)
__device__ __forceinline__ double qdiv(double a, double b) { return quot_rn(a, rcp_rn_of(b)); }
__device__ __forceinline__ double pow_cpovr(double a) { return pow35(a); }
#else
__device__ __forceinline__ double qdiv(double a, double b) { return a / b; }
__device__ __forceinline__ double pow_cpovr(double a) { return pow(a, kCpovr); }
#endif
__device__ __forceinline__ float pow_cpovr(float a) { return powf(a, (float)kCpovr); }
// the quotients of the diagnostics: FP32 storage divides as IEEE
__device__ __forceinline__ double ddiv(double a, double b) { return qdiv(a, b); }
__device__ __forceinline__ float ddiv(float a, float b) { return a / b; }

// pfesat / pfwsat (:119-181)
template <class T>
__device__ __forceinline__ T pfwsat(T t, T p) {
  T tl = t - T(kTzero);
  if (tl > T(100)) tl = T(100);
  if (tl < T(-75)) tl = T(-75);
  T td = tl, esat;
  if (td >= T(0)) {
    esat = T(kEsA0) + td * (T(kEsA1) + td * (T(kEsA2) + td * (T(kEsA3) + td * (T(kEsA4) +
           td * (T(kEsA5) + td * (T(kEsA6) + td * (T(kEsA7) + td * T(kEsA8))))))));
  } else {
    esat = T(kEsC0) + td * (T(kEsC1) + td * (T(kEsC2) + td * (T(kEsC3) + td * (T(kEsC4) +
           td * (T(kEsC5) + td * (T(kEsC6) + td * (T(kEsC7) + td * T(kEsC8))))))));
  }
  T lim = T(0.15) * p;
  T es = esat < lim ? esat : lim;
  return T(kEp2) * ddiv(es, p - es);
}

// ---- pre-diagnostics (:289-323) ----------------------------------------
template <class T>
__device__ __forceinline__ void b_prediag(const View<T>& d, const int bx, const int by, const int bz, int filterpai, int filtertheta) {
  int jj, ii;
  point_at<kPtBX, kPtBY>(d, bx, by, jj, ii);
  if (jj >= d.nj || ii >= d.ni) return;
  size_t c = (size_t)jj + (size_t)d.nj * ii + (size_t)bz * d.pl;
  T pai = d.pai[c], t = d.t[c];
  T qv = d.q[0][c], qc = d.q[1][c], qi = d.q[2][c], qr = d.q[3][c], qs = d.q[4][c];
  T p = pow_cpovr(pai) * T(kP00);
  d.p[c] = p;
  d.qsat[c] = pfwsat(t, p);
  T tv = t * ((((T(1) + T(kEp1) * qv) - qc) - qi) - qr - qs);
  d.tvirt[c] = tv;
  d.qwltot[c] = qc + qr;
  d.qwitot[c] = qi + qs;
  T tet = ddiv(tv, pai);
  d.tetav[c] = tet;
  if (filterpai) d.pf[c] = pai;
  if (filtertheta) d.tf[c] = tet;
}

template <class T>
__global__ void __launch_bounds__(kPtBX* kPtBY) k_prediag(View<T> d, int filterpai, int filtertheta) {
  b_prediag<T>(d, blockIdx.x, tile_y(d), blockIdx.z, filterpai, filtertheta);
}

template <class T>
__global__ void __launch_bounds__(kPtBX* kPtBY)
    kb_prediag(const View<T>* __restrict__ views, const int4* __restrict__ tiles, int filterpai, int filtertheta) {
  __shared__ View<T> sv;
  const int4 t = tiles[blockIdx.x];
  copy_view(&sv, views + t.x);
  __syncthreads();
  b_prediag<T>(sv, t.y, t.z, t.w, filterpai, filtertheta);
}


// ---- sound: halo, surface w, s (Eq. 10), horizontal divergence (Eq. 16) ---
// One thread per point.  Boundary threads also store the pre-divdamp u/v
// edge values that the momentum step reads as the stale ud/vd halo ring
// (:730-735); the bottom level computes w(kz+1) and s(kz+1) (:536-549).
template <class T>
__device__ __forceinline__ void b_sound_div(const View<T>& d, const int bx, const int by, const int bz) {
  if (d.sur_skip && *d.sur_skip) return;  // the surrogate took this cycle
  int jj, ii;
  point_at<kPtBX, kPtBY>(d, bx, by, jj, ii);
  const int kk = bz;
  const int nj = d.nj, ni = d.ni, kz = d.kz;
  if (jj >= nj || ii >= ni) return;
  const size_t pl = d.pl;
  const int jp = wp1(jj, nj), ip = wp1(ii, ni);
  const T* __restrict__ u = d.ubuf[d.cur];
  const T* __restrict__ v = d.vbuf[d.cur];
  const size_t c = (size_t)jj + (size_t)nj * ii;
  const size_t ce = (size_t)jp + (size_t)nj * ii;  // (j+1, i)
  const size_t cn = (size_t)jj + (size_t)nj * ip;  // (j, i+1)
  const size_t o = (size_t)kk * pl;
  const T u0 = u[c + o], u1 = u[ce + o], v0 = v[c + o], v1 = v[cn + o];
  const T hx0 = d.hx[c], hx1 = d.hx[ce], hy0 = d.hy[c], hy1 = d.hy[cn];
  if constexpr (kLean<T>) {
    // the metric factors of Equation 16 are stored with rfw, rfs and fmx: 16
    // FP64 operations a point instead of 24 (256 x 256 x 60: 2.75 -> 1.83 ms
    // per step)
    if (kk > 0) {
      const T zh = fma_rn(add_rn(u0, u[c + o - pl]), hx0, mul_rn(add_rn(u1, u[ce + o - pl]), hx1)) ;
      const T zs = fma_rn(add_rn(v0, v[c + o - pl]), hy0, fma_rn(add_rn(v1, v[cn + o - pl]), hy1, zh));
      d.s[c + o] = mul_rn(zs, mul_rn(T(-0.25), d.gzitak[kk]));
    }
    const T du = fma_rn(u1, d.rfw[ce + o], -mul_rn(u0, d.rfw[c + o]));
    const T dv = fma_rn(v1, d.rfs[cn + o], -mul_rn(v0, d.rfs[c + o]));
    d.zdiv2a[c + o] = mul_rn(d.fmx[c + o], add_rn(du, dv));
  } else {
  if (kk > 0) {  // s(k), k = 2..kz  (:557-570)
    const T u0p = u[c + o - pl], u1p = u[ce + o - pl], v0p = v[c + o - pl], v1p = v[cn + o - pl];
    T zuh = prod_add(u0 + u0p, hx0, u1 + u1p, hx1);
    T zvh = prod_add(v0 + v0p, hy0, v1 + v1p, hy1);
    d.s[c + o] = -((T(0.25) * (zuh + zvh)) * d.gzitak[kk]);
  }
  const T dtrdx = d.dtrdx, dtrdy = d.dtrdy;
  const T f = d.fmz[c + o];
  const T zrfmzum = d.rfw[c + o], zrfmzup = d.rfw[ce + o];
  const T zrfmzvm = d.rfs[c + o], zrfmzvp = d.rfs[cn + o];
  const T rmv0 = d.rmv[c], rmv1 = d.rmv[cn];
  // zum = (dtrdx u0) zrfmzum etc.; zup - zum and zvp - zvm with the
  // contraction fixed
  if (d.rotllr) {
    const T du = prod_sub(dtrdx * u1, zrfmzup, dtrdx * u0, zrfmzum);
    const T dv = prod_sub((dtrdy * v1) * zrfmzvp, rmv1, (dtrdy * v0) * zrfmzvm, rmv0);
    d.zdiv2a[c + o] = (f * d.mx[c]) * (du + dv);
  } else {
    const T rmu0 = d.rmu[c], rmu1 = d.rmu[ce];
    const T du = prod_sub((dtrdx * u1) * rmu1, zrfmzup, (dtrdx * u0) * rmu0, zrfmzum);
    const T dv = prod_sub((dtrdy * v1) * rmv1, zrfmzvp, (dtrdy * v0) * rmv0, zrfmzvm);
    d.zdiv2a[c + o] = (d.mx2[c] * f) * (du + dv);
  }
  }
  if (jj == 0) d.eu_j[ii + (size_t)ni * kk] = u0;
  if (ii == ni - 1) d.eu_i[jj + (size_t)nj * kk] = u0;
  if (jj == nj - 1) d.ev_j[ii + (size_t)ni * kk] = v0;
  if (ii == 0) d.ev_i[jj + (size_t)nj * kk] = v0;
  if (kk == kz - 1) {  // surface w(kz+1), s(kz+1)
    T zuh = prod_add(u0, hx0, u1, hx1);
    T zvh = prod_add(v0, hy0, v1, hy1);
    T ws = T(0.5) * (zuh + zvh);
    d.w[c + (size_t)kz * pl] = ws;
    d.s[c + (size_t)kz * pl] = -ws;
  }
}

template <class T>
__global__ void __launch_bounds__(kPtBX* kPtBY) k_sound_div(View<T> d) {
  b_sound_div<T>(d, blockIdx.x, tile_y(d), blockIdx.z);
}

template <class T>
__global__ void __launch_bounds__(kPtBX* kPtBY)
    kb_sound_div(const View<T>* __restrict__ views, const int4* __restrict__ tiles) {
  __shared__ View<T> sv;
  const int4 t = tiles[blockIdx.x];
  copy_view(&sv, views + t.x);
  __syncthreads();
  b_sound_div<T>(sv, t.y, t.z, t.w);
}


// ---- sound: divdamp (:853-895) and the vertical s term (:627-630) -------
// zdiv2b of a point (kLean): zdiv2 + ddamp2 (0.125 sum - 0.5 zdiv2) + fmz
// dtrdz (s(k) - s(k+1)), 7 FP64 operations instead of 9 (k_sound_damp_km at
// 256 x 256 x 60: 1.70 -> 1.54 ms per step)
template <class T>
__device__ __forceinline__ T damp_lean(T ddamp2, T zc, T zw, T ze, T zs, T zn, T fzd, T s0, T s1) {
  const T sum = add_rn(add_rn(add_rn(zw, ze), zs), zn);
  const T zd = fma_rn(mul_rn(T(0.125), ddamp2), sum, mul_rn(fma_rn(T(-0.5), ddamp2, T(1)), zc));
  return fma_rn(fzd, sub_rn(s0, s1), zd);
}
// One thread per point: damps u and v in place (their halo edges already
// hold the pre-damping values) and writes the divergence the implicit
// solve starts from into zdiv2b.
template <class T>
__device__ __forceinline__ void b_sound_damp(const View<T>& d, const int bx, const int by, const int bz) {
  if (d.sur_skip && *d.sur_skip) return;  // the surrogate took this cycle
  int jj, ii;
  point_at<kPtBX, kPtBY>(d, bx, by, jj, ii);
  const int kk = bz;
  const int nj = d.nj, ni = d.ni;
  if (jj >= nj || ii >= ni) return;
  const size_t pl = d.pl;
  const size_t o = (size_t)kk * pl;
  const size_t c = (size_t)jj + (size_t)nj * ii;
  T* __restrict__ u = d.ubuf[d.cur];
  T* __restrict__ v = d.vbuf[d.cur];
  const T zc = d.zdiv2a[c + o];
  const T zw = d.zdiv2a[o + wm1(jj, nj) + (size_t)nj * ii];
  const T ze = d.zdiv2a[o + wp1(jj, nj) + (size_t)nj * ii];
  const T zs = d.zdiv2a[o + jj + (size_t)nj * wm1(ii, ni)];
  const T zn = d.zdiv2a[o + jj + (size_t)nj * wp1(ii, ni)];
  const T cd = d.cdamp[kk];
  u[c + o] = u[c + o] + ((cd * d.mu[c]) * (zc - zw));
  if (d.rotllr)
    v[c + o] = v[c + o] + cd * (zc - zs);
  else
    v[c + o] = v[c + o] + ((cd * d.mv[c]) * (zc - zs));
  if constexpr (kLean<T>) {
    d.zdiv2b[c + o] = damp_lean(d.ddamp2, zc, zw, ze, zs, zn, d.fzd[c + o], d.s[c + o], d.s[c + o + pl]);
    return;
  }
  const T p2d = prod_sub(T(0.125), ((zw + ze) + zs) + zn, T(0.5), zc);
  T zd = zc + d.ddamp2 * p2d;
  zd = zd + (d.fmz[c + o] * d.dtrdz) * (d.s[c + o] - d.s[c + o + pl]);
  d.zdiv2b[c + o] = zd;
}

template <class T>
__global__ void __launch_bounds__(kPtBX* kPtBY) k_sound_damp(View<T> d) {
  b_sound_damp<T>(d, blockIdx.x, tile_y(d), blockIdx.z);
}

template <class T>
__global__ void __launch_bounds__(kPtBX* kPtBY)
    kb_sound_damp(const View<T>* __restrict__ views, const int4* __restrict__ tiles) {
  __shared__ View<T> sv;
  const int4 t = tiles[blockIdx.x];
  copy_view(&sv, views + t.x);
  __syncthreads();
  b_sound_damp<T>(sv, t.y, t.z, t.w);
}


// Quotient of the Exner/theta update in FP32 storage: the reciprocal
// estimate q = a * rcp(b) with one residual correction q + (a - b q) rcp(b)
// (Markstein's quotient correction, P. Markstein, "IA-64 and Elementary
// Functions", 2000): within one ulp of the IEEE quotient for the normal,
// well-scaled values it sees here (b = 1 + 0.96 qv + 4.8 qc), with no slow
// path or branch.  FP64 keeps the IEEE quotient.
__device__ __forceinline__ float div_corr(float a, float b) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(b));
  const float q = a * r;
  return fmaf(fmaf(-b, q, a), r, q);
}
__device__ __forceinline__ double div_corr(double a, double b) { return a / b; }

// zrom1w of the implicit w with the latent-heat term of saturated rising
// air (:641-652).  FP32 storage: the term is evaluated on every level (fast
// divide) and selected, so the level loop has no data-dependent branch;
// FP64: the reference's branch and IEEE divide.
template <class T>
__device__ __forceinline__ T zrom1w_moist(T zrom1w, T qvk, T qsk, T qskm, T wk, T fz, T pkm, T tm, T ns1, T dts) {
  if constexpr (sizeof(T) == 4) {
    const T zqs = T(0.5) * (qsk + qskm);
    const T zdth = __fdividef((((((T(kEgrav) * wk) * ns1) * dts) * T(kWlhv)) * T(kWlhv)) * zqs,
                              (((T(kCpd) * pkm) * T(kRwat)) * tm) * tm);
    const T zl = zrom1w + zdth * fz;
    return (qvk > T(0.96) * qsk && wk > T(0.1)) ? zl : zrom1w;
  } else {
    if (qvk > T(0.96) * qsk && wk > T(0.1)) {
      const T zqs = T(0.5) * (qsk + qskm);
      const T zdth = ((((((T(kEgrav) * wk) * ns1) * dts) * T(kWlhv)) * T(kWlhv)) * zqs) /
                     ((((T(kCpd) * pkm) * T(kRwat)) * tm) * tm);
      zrom1w = zrom1w + zdth * fz;
    }
    return zrom1w;
  }
}

// ---- sound: implicit w (Thomas, :634-686) + Exner/theta (:690-728) -----
// One thread per column.  Down-sweep k = kz..2 with FP64 pivots in every
// mode, stash of the FP64 down-sweep values, then back-substitution fused
// with the Exner/theta/pai update of the level above it.
// defer_pai: leave zdiv2b final and pai to k_pai_update (divergence filter on).
// PD: levels loaded ahead of the level computed, in both sweeps (a register
// ring of PD level records): 1, and 2 on small FP32 grids (k_sound_column).  A
// ring of 3 levels at 4 blocks per SM (so that the back-substitution finds more
// of the down-sweep's levels in L2) measured 13 % slower at 512 x 512 x 60:
// fewer columns in flight cost more bandwidth than the extra L2 hits saved.
template <class T, int PD>
__device__ __forceinline__ void b_sound_column_std(const View<T>& d, const int jj, const int ii, int nsound, int last, int defer_pai) {
  const int nj = d.nj, ni = d.ni, kz = d.kz;
  if (jj >= nj || ii >= ni) return;
  const size_t pl = d.pl;
  const size_t c = (size_t)jj + (size_t)nj * ii;
  // one restrict-qualified pointer per array, offset to this column, so the
  // loads of the next level can be issued ahead of the current level's
  // stores and FP64 work
  T* __restrict__ W = d.w + c;
  const T* __restrict__ FMZF = d.fmzf + c;
  const T* __restrict__ QV = d.q[0] + c;
  const T* __restrict__ QC = d.q[1] + c;
  T* __restrict__ TET = d.tetav + c;
  T* __restrict__ PAI = d.pai + c;
  const T* __restrict__ QSAT = d.qsat + c;
  const T* __restrict__ TT = d.t + c;
  T* __restrict__ ZD = d.zdiv2b + c;
  const T* __restrict__ FMZ = d.fmz + c;
  const T* __restrict__ QWL = d.qwltot + c;
  const T* __restrict__ QWI = d.qwitot + c;
  T* __restrict__ S = d.s + c;
  T* __restrict__ DW = d.deltaw + c;
  const T* __restrict__ FF = d.ffilt;
  const T ns = T(nsound), ns1 = T(nsound - 1);
  const T zcs2 = d.zcs2, dts = d.dts, egdts = d.egdts, dtrdz = d.dtrdz;

  // (b) down-sweep k = kz .. 2, loads of the next level issued one level ahead.
  // The pivots (den, its reciprocal zrapp and the ratio wwkw) are FP64 in
  // every mode.  FP64 storage: the right-hand-side sweep and the stash are
  // FP64 too (the reference's arithmetic).  FP32 storage: the right-hand
  // side and the stash are FP32, which keeps the FP64 pipe -- 1/64 of the
  // FP32 rate on GB300 -- to the pivot recurrence.
  constexpr bool kF32 = sizeof(T) == 4;
  using ST = typename std::conditional<kF32, float, double>::type;  // stash / RHS type
  ST* __restrict__ WPs = reinterpret_cast<ST*>(d.wp) + c;
  ST* __restrict__ WWs = reinterpret_cast<ST*>(d.wwkw) + c;
  const T wsurf = W[(size_t)kz * pl];  // w(kz+1) from k_sound_div
  ST wkp1 = (ST)wsurf;
  double wwp1 = 0.0;  // wwkw(kz+1) = 0 (FP64 storage)
  double cwp1 = 1.0;  // 1 - wwkw(kz+1) (FP32 storage)
  // level kk of the down-sweep reads w, fmzf, qv, ffilt at kk and tetav,
  // pai, qsat, zdiv2b, fmz, t at kk-1 (carried as the next level's kk values)
  struct Dn { T wk, fz, qv, ff, tkm, pkm, qskm, zdkm, fkm, tm; };
  auto load_dn = [&](int kk, Dn& x) {
    const size_t on = (size_t)kk * pl, onm = on - pl;
    x.wk = W[on]; x.fz = FMZF[on]; x.qv = QV[on]; x.ff = FF[kk];
    x.tkm = TET[onm]; x.pkm = PAI[onm]; x.qskm = QSAT[onm]; x.zdkm = ZD[onm];
    x.fkm = FMZ[onm]; x.tm = TT[onm];
  };
  size_t o = (size_t)(kz - 1) * pl;
  T zd_k = ZD[o], tk = TET[o], pk = PAI[o], fk = FMZ[o], qsk = QSAT[o];
  Dn dring[PD];
#pragma unroll
  for (int u = 0; u < PD; ++u)
    if (kz - 1 - u >= 1) load_dn(kz - 1 - u, dring[u]);
  for (int base = kz - 1; base >= 1; base -= PD) {
#pragma unroll
  for (int u = 0; u < PD; ++u) {
    const int kk = base - u;
    if (kk < 1) break;
    o = (size_t)kk * pl;
    const Dn cur = dring[u];
    if (kk - PD >= 1) load_dn(kk - PD, dring[u]);
    const T wk = cur.wk, fz = cur.fz, qvk = cur.qv, ff = cur.ff, tkm = cur.tkm, pkm = cur.pkm;
    const T qskm = cur.qskm, zd_km = cur.zdkm, fkm = cur.fkm, tm = cur.tm;
    T zrom1w = ((T(0.5) * T(kCpd)) * fz) * (tkm + tk);
    zrom1w = zrom1w - (((((T(kCpd) * wk) * fz) * fz) * ns) * dtrdz) * (tkm - tk);
    zrom1w = zrom1w_moist(zrom1w, qvk, qsk, qskm, wk, fz, pkm, tm, ns1, dts);
    T zwexpl = (wk - (zrom1w * dtrdz) * (pkm - pk)) - egdts;
    zwexpl = zwexpl + ((T(kRdrcv) * zrom1w) * dtrdz) * prod_sub(pkm, zd_km, pk, zd_k);
    const T zu_t = ((zcs2 * fkm) * zrom1w) * pkm + ff;
    const T zd_t = ((zcs2 * fk) * zrom1w) * pk + ff;
    ST wpk;
    double wwk;
    if constexpr (kF32) {
      // The pivot recurrence in FP64, written for the complement
      // c = 1 - wwkw: den = (1 + zd c(k+1)) + zu, c(k) = (1 + zd c(k+1)) / den
      // -- the reference's den = ((1 + zd) + zu) - zd wwkw(k+1) and
      // wwkw(k) = zu / den without the cancellation of zd against
      // zd wwkw(k+1).  Four FP64 operations a level: the quotient starts
      // from the FP32 estimate q0 = tt r (r the FP32 estimate of 1/den) and
      // takes one correction, r times the FP64 residual tt - den q0
      // (relative error ~2e-13); the widenings and narrowings run on the
      // integer pipe.  The FP32 right-hand side and the stash use r itself.
      const double zu = widen_f32(zu_t), zdd = widen_f32(zd_t);
      const double tt = fma(zdd, cwp1, 1.0);
      const double den = tt + zu;
      float r;
      asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(narrow_trunc(den)));
      const double q0 = widen_f32(narrow_trunc(tt) * r);
      const double rem = fma(-den, q0, tt);
      cwp1 = q0 + widen_f32(r * narrow_trunc(rem));
      wwk = 0.0;
      wpk = r * (zwexpl + zd_t * wkp1);
      WWs[o] = r * zu_t;
    } else {
      const double zu = (double)zu_t;
      const double zdd = (double)zd_t;
      const double den = ((1.0 + zdd) + zu) - zdd * wwp1;
      const double zrapp = 1.0 / den;
      wwk = zrapp * zu;
      wpk = zrapp * ((double)zwexpl + zdd * wkp1);
      WWs[o] = (ST)wwk;
    }
    WPs[o] = wpk;
    wkp1 = wpk; wwp1 = wwk;
    zd_k = zd_km; tk = tkm; pk = pkm; fk = fkm; qsk = qskm;
  }
  }

  // (c) back-substitution (:681-686) fused with the Exner/theta update of
  // the level above (:690-728); w(1) = 0 always (init_moloch :260-262).
  // Level kk is solved while level kk-1 is finalized; loads run PD ahead.
  const T rdrcv = T(kRdrcv);
  ST wlo_d = 0;
  T wlo = T(0);
  // finalize inputs of level m
  struct Fin { T zd, fmz, qv, qc, tet, qwl, qwi, pai, s, fmzf; };
  auto load_fin = [&](int m) {
    const size_t q = (size_t)m * pl;
    Fin f;
    f.zd = ZD[q]; f.fmz = FMZ[q]; f.qv = QV[q]; f.qc = QC[q]; f.tet = TET[q];
    f.qwl = QWL[q]; f.qwi = QWI[q]; f.pai = PAI[q];
    f.s = last ? S[q] : T(0);
    f.fmzf = last ? FMZF[q] : T(0);
    return f;
  };
  auto finalize = [&](int m, const Fin& f, T wl, T wh) {
    const size_t q = (size_t)m * pl;
    T zd = f.zd;
    zd = zd + (dtrdz * f.fmz) * (wl - wh);
    zd = div_corr(zd * ((T(1) + T(0.86) * f.qv) + T(3.2) * f.qc), (T(1) + T(0.96) * f.qv) + T(4.8) * f.qc);
    TET[q] = f.tet * (T(1) + (rdrcv * zd) * (prod_add(T(0.25), f.qv, T(4.2), f.qwl) + T(2.1) * f.qwi));
    if (defer_pai) {
      ZD[q] = zd;
    } else {
      if (jj == nj - 1) d.ep_j[ii + (size_t)ni * m] = f.pai;
      if (ii == ni - 1) d.ep_i[jj + (size_t)nj * m] = f.pai;
      PAI[q] = f.pai * (T(1) - rdrcv * zd);
    }
    if (last) S[q] = m == 0 ? T(0) : (wl + f.s) * f.fmzf;  // complete Equation 10 (:843-849)
  };
  // record m = 1 .. kz: the stash and old w of level m (m < kz) and the
  // finalize inputs of level m-1
  struct Bk { ST wp, ww; T wold; Fin f; };
  auto load_bk = [&](int m, Bk& x) {
    x.f = load_fin(m - 1);
    if (m < kz) {
      const size_t q = (size_t)m * pl;
      x.wp = WPs[q]; x.ww = WWs[q]; x.wold = W[q];
    }
  };
  Bk bring[PD];
#pragma unroll
  for (int u = 0; u < PD; ++u)
    if (1 + u <= kz) load_bk(1 + u, bring[u]);
  for (int base = 1; base <= kz; base += PD) {
#pragma unroll
  for (int u = 0; u < PD; ++u) {
    const int kk = base + u;
    if (kk > kz) break;
    const Bk cur = bring[u];
    if (kk + PD <= kz) load_bk(kk + PD, bring[u]);
    if (kk < kz) {
      const size_t q = (size_t)kk * pl;
      wlo_d = cur.wp + cur.ww * wlo_d;
      const T wn = (T)wlo_d;
      DW[q] = (-cur.wold) + wn;
      W[q] = wn;
      finalize(kk - 1, cur.f, wlo, wn);
      wlo = wn;
    } else {
      finalize(kz - 1, cur.f, wlo, wsurf);
    }
  }
  }
  if (last) S[(size_t)kz * pl] = T(0);
}

// The same in the contracting FP64 build, in 39 FP64 operations a level
// (about 80 as above).  A = zrom1w dtrdz and B = rdrcv A scale the pressure
// and divergence differences, and zu, zd = B fzd(k-1) pai(k-1), B fzd(k)
// pai(k) with the level's products carried to the next.  The pivots run on
// the complement c = 1 - wwkw (den = (1 + zd c(k+1)) + zu), their reciprocal
// by pivot_rcp.  The moist factors of the Exner/theta update do not change
// within a sound() call: the first substep forms and stores them (mo1, mo2),
// the others read those two instead of qv, qc, qwltot, qwitot and divide no
// more.  The latent-heat branch compares w > 0.1 as integers (positive
// doubles order as their bits) before it forms anything.  It leaves out the
// ffilt(k) the other solves add to zu and zd, which is zero (View::ffilt).
// 256 x 256 x 60: 8.6 -> 6.0 ms per step.
template <int PD>
__device__ __forceinline__ void b_sound_column_lean(const View<double>& d, const int jj, const int ii, int nsound,
                                                    int last, int defer_pai) {
  const int nj = d.nj, ni = d.ni, kz = d.kz;
  if (jj >= nj || ii >= ni) return;
  const size_t pl = d.pl;
  const size_t c = (size_t)jj + (size_t)nj * ii;
  double* __restrict__ W = d.w + c;
  const double* __restrict__ FMZF = d.fmzf + c;
  const double* __restrict__ QV = d.q[0] + c;
  const double* __restrict__ QC = d.q[1] + c;
  double* __restrict__ TET = d.tetav + c;
  double* __restrict__ PAI = d.pai + c;
  const double* __restrict__ QSAT = d.qsat + c;
  const double* __restrict__ TT = d.t + c;
  double* __restrict__ ZD = d.zdiv2b + c;
  const double* __restrict__ FZD = d.fzd + c;
  const double* __restrict__ QWL = d.qwltot + c;
  const double* __restrict__ QWI = d.qwitot + c;
  double* __restrict__ MO1 = d.mo1 + c;
  double* __restrict__ MO2 = d.mo2 + c;
  double* __restrict__ S = d.s + c;
  double* __restrict__ DW = d.deltaw + c;
  double* __restrict__ WPs = d.wp + c;
  double* __restrict__ WWs = d.wwkw + c;
  const double dts = d.dts, egdts = d.egdts, dtrdz = d.dtrdz;
  const double c2 = 2.0 * (double)nsound * dtrdz;
  const bool first = nsound == 1;

  // down-sweep k = kz .. 2
  const double wsurf = W[(size_t)kz * pl];
  double wkp1 = wsurf, cwp1 = 1.0;
  struct Dn { double wk, fz, tkm, pkm, zdkm, fkm; };
  auto load_dn = [&](int kk, Dn& x) {
    const size_t on = (size_t)kk * pl, onm = on - pl;
    x.wk = W[on]; x.fz = FMZF[on];
    x.tkm = TET[onm]; x.pkm = PAI[onm]; x.zdkm = ZD[onm]; x.fkm = FZD[onm];
  };
  size_t o = (size_t)(kz - 1) * pl;
  double tk = TET[o], pk = PAI[o];
  double fp = mul_rn(FZD[o], pk), pz = mul_rn(pk, ZD[o]);
  Dn dring[PD];
#pragma unroll
  for (int u = 0; u < PD; ++u)
    if (kz - 1 - u >= 1) load_dn(kz - 1 - u, dring[u]);
  for (int base = kz - 1; base >= 1; base -= PD) {
#pragma unroll
  for (int u = 0; u < PD; ++u) {
    const int kk = base - u;
    if (kk < 1) break;
    o = (size_t)kk * pl;
    const Dn x = dring[u];
    if (kk - PD >= 1) load_dn(kk - PD, dring[u]);
    double zr = mul_rn(mul_rn(0.5 * kCpd, x.fz), fma_rn(-mul_rn(mul_rn(x.fz, x.wk), c2), sub_rn(x.tkm, tk), add_rn(x.tkm, tk)));
    if (__double_as_longlong(x.wk) > __double_as_longlong(0.1)) {  // latent heat of saturated rising air (:641-652)
      const double qsk = QSAT[o], qskm = QSAT[o - pl], tm = TT[o - pl];
      if (QV[o] > 0.96 * qsk) {
        const double zqs = 0.5 * (qsk + qskm);
        const double zdth = ((((((kEgrav * x.wk) * (double)(nsound - 1)) * dts) * kWlhv) * kWlhv) * zqs) /
                            ((((kCpd * x.pkm) * kRwat) * tm) * tm);
        zr = zr + zdth * x.fz;
      }
    }
    const double A = mul_rn(zr, dtrdz), B = mul_rn(kRdrcv, A);
    const double pzm = mul_rn(x.pkm, x.zdkm), fpm = mul_rn(x.fkm, x.pkm);
    const double ex = fma_rn(B, sub_rn(pzm, pz), sub_rn(fma_rn(-A, sub_rn(x.pkm, pk), x.wk), egdts));
    const double zu = mul_rn(B, fpm), zd = mul_rn(B, fp);
    const double tt = fma_rn(zd, cwp1, 1.0);
    const double r = pivot_rcp(add_rn(tt, zu));
    wkp1 = mul_rn(r, fma_rn(zd, wkp1, ex));
    cwp1 = mul_rn(r, tt);
    WPs[o] = wkp1;
    WWs[o] = mul_rn(r, zu);
    tk = x.tkm; pk = x.pkm; fp = fpm; pz = pzm;
  }
  }

  // back-substitution fused with the Exner/theta update of the level above
  struct Bk { double wp, ww, wold, zd, fz, tet, pai, m1, m2, s, fmzf; };
  auto load_bk = [&](int m, Bk& x) {  // level m (m < kz) of the stash and of w, level m-1 of the rest
    const size_t q = (size_t)(m - 1) * pl;
    x.zd = ZD[q]; x.fz = FZD[q]; x.tet = TET[q]; x.pai = PAI[q];
    if (first) {
      const double qv = QV[q], qc = QC[q];
      x.m1 = qdiv(fma(3.2, qc, fma(0.86, qv, 1.0)), fma(4.8, qc, fma(0.96, qv, 1.0)));
      x.m2 = fma(2.1, QWI[q], fma(4.2, QWL[q], 0.25 * qv));
    } else {
      x.m1 = MO1[q]; x.m2 = MO2[q];
    }
    x.s = last ? S[q] : 0.0;
    x.fmzf = last ? FMZF[q] : 0.0;
    if (m < kz) {
      x.wp = WPs[q + pl]; x.ww = WWs[q + pl]; x.wold = W[q + pl];
    }
  };
  double wl = 0.0;  // w(1) = 0 always (init_moloch :260-262)
  Bk bring[PD];
#pragma unroll
  for (int u = 0; u < PD; ++u)
    if (1 + u <= kz) load_bk(1 + u, bring[u]);
  for (int base = 1; base <= kz; base += PD) {
#pragma unroll
  for (int u = 0; u < PD; ++u) {
    const int kk = base + u;
    if (kk > kz) break;
    const Bk x = bring[u];
    if (kk + PD <= kz) load_bk(kk + PD, bring[u]);
    const size_t q = (size_t)(kk - 1) * pl;
    double wh = wsurf;
    if (kk < kz) {
      wh = fma_rn(x.ww, wl, x.wp);
      DW[q + pl] = sub_rn(wh, x.wold);
      W[q + pl] = wh;
    }
    const double zd = mul_rn(fma_rn(x.fz, sub_rn(wl, wh), x.zd), x.m1);
    const double r = mul_rn(kRdrcv, zd);
    TET[q] = mul_rn(x.tet, fma_rn(r, x.m2, 1.0));  // rounds as the reference's products do
    if (first) {
      MO1[q] = x.m1;
      MO2[q] = x.m2;
    }
    if (defer_pai) {
      ZD[q] = zd;
    } else {
      if (jj == nj - 1) d.ep_j[ii + (size_t)ni * (kk - 1)] = x.pai;
      if (ii == ni - 1) d.ep_i[jj + (size_t)nj * (kk - 1)] = x.pai;
      PAI[q] = mul_rn(x.pai, sub_rn(1.0, r));
    }
    if (last) S[q] = kk == 1 ? 0.0 : mul_rn(add_rn(wl, x.s), x.fmzf);  // complete Equation 10 (:843-849)
    wl = wh;
  }
  }
  if (last) S[(size_t)kz * pl] = 0.0;
}

template <class T, int PD>
__device__ __forceinline__ void b_sound_column(const View<T>& d, const int jj, const int ii, int nsound, int last,
                                               int defer_pai) {
  if (d.sur_skip && *d.sur_skip) return;  // the surrogate took this cycle
  if constexpr (kLean<T>) b_sound_column_lean<PD>(d, jj, ii, nsound, last, defer_pai);
  else b_sound_column_std<T, PD>(d, jj, ii, nsound, last, defer_pai);
}

// FP32: 9 blocks of 128 threads per SM (56 registers, 24 bytes spilled):
// 1.5 waves at 512 x 512 instead of 1.68 with 8 blocks (4.51 against
// 4.61 ms per step; 10 blocks, 48 registers, 4.84 ms)
//
// PD = 2, 4 blocks (118 registers): the FP32 kernel of domains whose columns
// (up to 4 x 128 x SMs) are all in flight at once either way, where a second
// level of loads in flight hides more than occupancy does: 28 against 35 us
// per launch at 100 x 100 x 30, 56 against 75 at 203 x 157 x 45, 64 against 80
// at 256 x 256 x 40; above, 188 against 172 at 384 x 384 x 60.  FP64 gains
// nothing from it (81 against 82 us at 100 x 100 x 30).  Where blocks of four
// rows are fewer than two an SM, blocks of one row spread the warps: exact
// FP64 at 100 x 100 x 30 115 -> 105 us.
template <class T, int PD>
__global__ void __launch_bounds__(kColBX* kColBY, sizeof(T) == 4 && PD == 1 ? 9 : 4)
    k_sound_column(View<T> d, int nsound, int last, int defer_pai) {
  b_sound_column<T, PD>(d, blockIdx.x * kColBX + threadIdx.x, blockIdx.y * blockDim.y + threadIdx.y, nsound, last,
                        defer_pai);
}

// FP64 on few columns: a block holds C columns (C neighbours of the plane,
// across row ends) and all their levels.  Its 256 threads form the
// right-hand sides and coefficients of all levels side by side, C of them run
// the recurrence down and the substitution up through shared memory, then all
// of them update Exner function, theta and pai.  Same expressions and bits as
// the march, where 10,000 columns are two warps an SM and each level's 39
// (exact: about 80) FP64 operations, 16 clocks each, wait for the one before.
// Here only the recurrence (11 and about 18) does, and neither wp nor wwkw leave
// the SM.  64 registers, so that four blocks an SM overlap their phases (142
// registers, one block: 76 us instead of 50 at 100 x 100 x 30, with a reciprocal
// of two operations less).
constexpr int kSplitThreads = 256;
constexpr size_t split_smem_bytes(int columns, int kz) { return (size_t)3 * kz * columns * sizeof(double); }
template <int C>
__global__ void __launch_bounds__(kSplitThreads, 4)
    k_sound_column_split(View<double> d, int nsound, int last, int defer_pai) {
  if (d.sur_skip && *d.sur_skip) return;  // the surrogate took this cycle
  extern __shared__ double split_smem[];
  constexpr int NG = kSplitThreads / C;
  const int kz = d.kz, nj = d.nj, ni = d.ni;
  const size_t pl = d.pl;
  double* const sx = split_smem;  // [level][column]: right-hand side, then wp, then w
  double* const su = sx + kz * C;  // zu, then wwkw
  double* const sd = su + kz * C;  // zd
  const int col = threadIdx.x % C, grp = threadIdx.x / C;
  const size_t cc = (size_t)blockIdx.x * C + col;
  const bool on = cc < pl;
  const size_t c = on ? cc : pl - 1;
  double* __restrict__ W = d.w + c;
  const double* __restrict__ FMZF = d.fmzf + c;
  const double* __restrict__ FMZ = d.fmz + c;
  const double* __restrict__ QV = d.q[0] + c;
  const double* __restrict__ QC = d.q[1] + c;
  double* __restrict__ TET = d.tetav + c;
  double* __restrict__ PAI = d.pai + c;
  const double* __restrict__ QSAT = d.qsat + c;
  const double* __restrict__ TT = d.t + c;
  double* __restrict__ ZD = d.zdiv2b + c;
  const double* __restrict__ QWL = d.qwltot + c;
  const double* __restrict__ QWI = d.qwitot + c;
  double* __restrict__ S = d.s + c;
  double* __restrict__ DW = d.deltaw + c;
  const double dts = d.dts, egdts = d.egdts, dtrdz = d.dtrdz, zcs2 = d.zcs2;
  const double ns = nsound, ns1 = nsound - 1;
  const double c2 = 2.0 * ns * dtrdz;
  const double* __restrict__ FZD = kLean<double> ? d.fzd + c : FMZ;
  const double wsurf = W[(size_t)kz * pl];

  // coefficients of levels kz .. 2
  for (int kk = 1 + grp; kk < kz; kk += NG) {
    const size_t o = (size_t)kk * pl, om = o - pl;
    const double wk = W[o], fz = FMZF[o], tk = TET[o], tkm = TET[om], pk = PAI[o], pkm = PAI[om];
    const double zk = ZD[o], zkm = ZD[om], fk = FZD[o], fkm = FZD[om];
    double ex, zu, zd;
    if constexpr (kLean<double>) {
      double zr = mul_rn(mul_rn(0.5 * kCpd, fz), fma_rn(-mul_rn(mul_rn(fz, wk), c2), sub_rn(tkm, tk), add_rn(tkm, tk)));
      if (__double_as_longlong(wk) > __double_as_longlong(0.1)) {  // latent heat of saturated rising air (:641-652)
        const double qsk = QSAT[o], qskm = QSAT[om], tm = TT[om];
        if (QV[o] > 0.96 * qsk) {
          const double zqs = 0.5 * (qsk + qskm);
          const double zdth = ((((((kEgrav * wk) * ns1) * dts) * kWlhv) * kWlhv) * zqs) /
                              ((((kCpd * pkm) * kRwat) * tm) * tm);
          zr = zr + zdth * fz;
        }
      }
      const double A = mul_rn(zr, dtrdz), B = mul_rn(kRdrcv, A);
      ex = fma_rn(B, sub_rn(mul_rn(pkm, zkm), mul_rn(pk, zk)), sub_rn(fma_rn(-A, sub_rn(pkm, pk), wk), egdts));
      zu = mul_rn(B, mul_rn(fkm, pkm));
      zd = mul_rn(B, mul_rn(fk, pk));
    } else {
      double zrom1w = ((0.5 * kCpd) * fz) * (tkm + tk);
      zrom1w = zrom1w - (((((kCpd * wk) * fz) * fz) * ns) * dtrdz) * (tkm - tk);
      zrom1w = zrom1w_moist(zrom1w, QV[o], QSAT[o], QSAT[om], wk, fz, pkm, TT[om], ns1, dts);
      ex = (wk - (zrom1w * dtrdz) * (pkm - pk)) - egdts;
      ex = ex + ((kRdrcv * zrom1w) * dtrdz) * prod_sub(pkm, zkm, pk, zk);
      zu = ((zcs2 * fkm) * zrom1w) * pkm + d.ffilt[kk];
      zd = ((zcs2 * fk) * zrom1w) * pk + d.ffilt[kk];
    }
    sx[kk * C + col] = ex;
    su[kk * C + col] = zu;
    sd[kk * C + col] = zd;
  }
  __syncthreads();
  if (threadIdx.x < C) {
    double wkp1 = wsurf, wwp1 = 0.0, cwp1 = 1.0;
    for (int kk = kz - 1; kk >= 1; --kk) {
      const double ex = sx[kk * C + col], zu = su[kk * C + col], zd = sd[kk * C + col];
      if constexpr (kLean<double>) {
        const double tt = fma_rn(zd, cwp1, 1.0), r = pivot_rcp(add_rn(tt, zu));
        wkp1 = mul_rn(r, fma_rn(zd, wkp1, ex));
        cwp1 = mul_rn(r, tt);
        wwp1 = mul_rn(r, zu);
      } else {
        const double den = ((1.0 + zd) + zu) - zd * wwp1;
        const double zrapp = 1.0 / den;
        wwp1 = zrapp * zu;
        wkp1 = zrapp * (ex + zd * wkp1);
      }
      sx[kk * C + col] = wkp1;
      su[kk * C + col] = wwp1;
    }
    double wl = 0.0;  // w(1) = 0 always (init_moloch :260-262)
    sx[col] = wl;
    for (int kk = 1; kk < kz; ++kk) {
      if constexpr (kLean<double>) wl = fma_rn(su[kk * C + col], wl, sx[kk * C + col]);
      else wl = sx[kk * C + col] + su[kk * C + col] * wl;
      sx[kk * C + col] = wl;
    }
  }
  __syncthreads();
  if (!on) return;
  // w, deltaw and the Exner/theta update (:690-728)
  const int jj = (int)(c % nj), ii = (int)(c / nj);
  for (int m = grp; m < kz; m += NG) {
    const size_t q = (size_t)m * pl;
    const double wl = sx[m * C + col], wh = m + 1 < kz ? sx[(m + 1) * C + col] : wsurf;
    if (m > 0) {
      DW[q] = kLean<double> ? sub_rn(wl, W[q]) : (-W[q]) + wl;
      W[q] = wl;
    }
    const double tet = TET[q], pai = PAI[q];
    double zd, r;
    if constexpr (kLean<double>) {
      double m1, m2;
      if (nsound == 1) {
        const double qv = QV[q], qc = QC[q];
        m1 = qdiv(fma(3.2, qc, fma(0.86, qv, 1.0)), fma(4.8, qc, fma(0.96, qv, 1.0)));
        m2 = fma(2.1, QWI[q], fma(4.2, QWL[q], 0.25 * qv));
        d.mo1[c + q] = m1;
        d.mo2[c + q] = m2;
      } else {
        m1 = d.mo1[c + q];
        m2 = d.mo2[c + q];
      }
      zd = mul_rn(fma_rn(FZD[q], sub_rn(wl, wh), ZD[q]), m1);
      r = mul_rn(kRdrcv, zd);
      TET[q] = mul_rn(tet, fma_rn(r, m2, 1.0));  // rounds as the reference's products do
    } else {
      const double qv = QV[q], qc = QC[q];
      zd = ZD[q] + (dtrdz * FMZ[q]) * (wl - wh);
      zd = div_corr(zd * ((1.0 + 0.86 * qv) + 3.2 * qc), (1.0 + 0.96 * qv) + 4.8 * qc);
      r = kRdrcv * zd;
      TET[q] = tet * (1.0 + r * (prod_add(0.25, qv, 4.2, QWL[q]) + 2.1 * QWI[q]));
    }
    if (defer_pai) {
      ZD[q] = zd;
    } else {
      if (jj == nj - 1) d.ep_j[ii + (size_t)ni * m] = pai;
      if (ii == ni - 1) d.ep_i[jj + (size_t)nj * m] = pai;
      PAI[q] = kLean<double> ? mul_rn(pai, sub_rn(1.0, r)) : pai * (1.0 - r);
    }
    if (last) {  // complete Equation 10 (:843-849)
      S[q] = m == 0 ? 0.0 : kLean<double> ? mul_rn(add_rn(wl, S[q]), FMZF[q]) : (wl + S[q]) * FMZF[q];
      if (m == kz - 1) S[q + pl] = 0.0;
    }
  }
}

template <class T>
__global__ void __launch_bounds__(kColBX* kColBY, sizeof(T) == 4 ? 8 : 4)
    kb_sound_column(const View<T>* __restrict__ views, const int4* __restrict__ tiles, int nsound, int last, int defer_pai) {
  __shared__ View<T> sv;
  const int4 t = tiles[blockIdx.x];
  copy_view(&sv, views + t.x);
  __syncthreads();
  b_sound_column<T, 1>(sv, t.y * kColBX + threadIdx.x, t.z * kColBY + threadIdx.y, nsound, last, defer_pai);
}



}  // namespace MOLOCH_KNS
}  // namespace moloch
#include "moloch_column_tm.cuh"
namespace moloch {
namespace MOLOCH_KNS {

// ---- 5-point Laplacian filter of one field, out of place ----------------
// out = a + coef(k) * (0.125*(aW+aE+aS+aN) - 0.5*a)   (:423-481)
// coef(k) = anu2 * xknu(k) when use_xknu, else the constant c0.
template <class T>
__device__ __forceinline__ void b_lap_filter(const View<T>& d, const int bx, const int by, const int bz) {
  if (d.sur_skip && *d.sur_skip) return;  // the surrogate took this cycle
  const T* __restrict__ a = d.zdiv2b;
  T* __restrict__ out = d.zdiv2a;

  int jj, ii;
  point_at<kPtBX, kPtBY>(d, bx, by, jj, ii);
  const int nj = d.nj, ni = d.ni;
  if (jj >= nj || ii >= ni) return;
  const size_t o = (size_t)bz * d.pl;
  const size_t c = jj + (size_t)nj * ii;
  T aw = a[o + wm1(jj, nj) + (size_t)nj * ii], ae = a[o + wp1(jj, nj) + (size_t)nj * ii];
  T as = a[o + jj + (size_t)nj * wm1(ii, ni)], an = a[o + jj + (size_t)nj * wp1(ii, ni)];
  T ac = a[o + c];
  T p2d = prod_sub(T(0.125), ((aw + ae) + as) + an, T(0.5), ac);
  const T coef = d.anu2 * d.xknu[bz];
  out[o + c] = ac + coef * p2d;
}

template <class T>
__global__ void __launch_bounds__(kPtBX* kPtBY) k_lap_filter(View<T> d) {
  b_lap_filter<T>(d, blockIdx.x, tile_y(d), blockIdx.z);
}

template <class T>
__global__ void __launch_bounds__(kPtBX* kPtBY)
    kb_lap_filter(const View<T>* __restrict__ views, const int4* __restrict__ tiles) {
  __shared__ View<T> sv;
  const int4 t = tiles[blockIdx.x];
  copy_view(&sv, views + t.x);
  __syncthreads();
  b_lap_filter<T>(sv, t.y, t.z, t.w);
}


// pai update with the nompi halo order (:716-728), split form
template <class T>
__device__ __forceinline__ void b_pai_update(const View<T>& d, const int bx, const int by, const int bz) {
  if (d.sur_skip && *d.sur_skip) return;  // the surrogate took this cycle
  const T* __restrict__ zd = d.zdiv2a;

  int jj, ii;
  point_at<kPtBX, kPtBY>(d, bx, by, jj, ii);
  const int nj = d.nj, ni = d.ni, kk = bz;
  if (jj >= nj || ii >= ni) return;
  const size_t c = jj + (size_t)nj * ii + (size_t)kk * d.pl;
  const T pold = d.pai[c];
  if (jj == nj - 1) d.ep_j[ii + (size_t)ni * kk] = pold;
  if (ii == ni - 1) d.ep_i[jj + (size_t)nj * kk] = pold;
  d.pai[c] = pold * (T(1) - T(kRdrcv) * zd[c]);
}

template <class T>
__global__ void __launch_bounds__(kPtBX* kPtBY) k_pai_update(View<T> d) {
  b_pai_update<T>(d, blockIdx.x, tile_y(d), blockIdx.z);
}

template <class T>
__global__ void __launch_bounds__(kPtBX* kPtBY)
    kb_pai_update(const View<T>* __restrict__ views, const int4* __restrict__ tiles) {
  __shared__ View<T> sv;
  const int4 t = tiles[blockIdx.x];
  copy_view(&sv, views + t.x);
  __syncthreads();
  b_pai_update<T>(sv, t.y, t.z, t.w);
}


// filtpai / filttheta on the step increment (:333-353, :442-481):
// x = a - ref; a = ((x + nupaitq * lap(x)) + ref), written to out
template <class T>
__device__ __forceinline__ void b_filter_increment(const View<T>& d, const int bx, const int by, const int bz, int which) {  const T* __restrict__ a = which ? d.tetav : d.pai;
  const T* __restrict__ ref = which ? d.tf : d.pf;
  T* __restrict__ out = d.fscr;

  int jj, ii;
  point_at<kPtBX, kPtBY>(d, bx, by, jj, ii);
  const int nj = d.nj, ni = d.ni;
  if (jj >= nj || ii >= ni) return;
  const size_t o = (size_t)bz * d.pl;
  auto X = [&](int j, int i) {
    size_t q = o + j + (size_t)nj * i;
    return a[q] - ref[q];
  };
  T xw = X(wm1(jj, nj), ii), xe = X(wp1(jj, nj), ii), xs = X(jj, wm1(ii, ni)), xn = X(jj, wp1(ii, ni));
  T xc = X(jj, ii);
  T p2d = prod_sub(T(0.125), ((xw + xe) + xs) + xn, T(0.5), xc);
  const size_t c = o + jj + (size_t)nj * ii;
  out[c] = (xc + T(kNupaitq) * p2d) + ref[c];
}

template <class T>
__global__ void __launch_bounds__(kPtBX* kPtBY) k_filter_increment(View<T> d, int which) {
  b_filter_increment<T>(d, blockIdx.x, tile_y(d), blockIdx.z, which);
}

template <class T>
__global__ void __launch_bounds__(kPtBX* kPtBY)
    kb_filter_increment(const View<T>* __restrict__ views, const int4* __restrict__ tiles, int which) {
  __shared__ View<T> sv;
  const int4 t = tiles[blockIdx.x];
  copy_view(&sv, views + t.x);
  __syncthreads();
  b_filter_increment<T>(sv, t.y, t.z, t.w, which);
}


// u plus and v minus the Coriolis term k sum of Equations 17 and 18.  FP32: as
// one multiply-add, or (rounded) with the product rounded first, as
// k_sound_momentum takes it; the rest of the equations rounds alike in all
// variants.  The quads and strips can do either (View::cor_rounded).
__device__ __forceinline__ float plus_cor(float u, float k, float sum, int rounded) {
  return rounded ? __fadd_rn(u, __fmul_rn(k, sum)) : __fmaf_rn(k, sum, u);
}
__device__ __forceinline__ double plus_cor(double u, double k, double sum, int) { return u + k * sum; }
template <class T>
__device__ __forceinline__ T minus_cor(T v, T k, T sum, int rounded) { return plus_cor(v, -k, sum, rounded); }

// ---- sound: momentum, Equations 17 and 18 (:737-837) --------------------
// One thread per point; reads u, v (current buffer, damped interior + the
// pre-damping edges) and writes the other buffer of the pair.
template <class T>
__device__ __forceinline__ void b_sound_momentum(const View<T>& d, const int bx, const int by, const int bz) {
  if (d.sur_skip && *d.sur_skip) return;  // the surrogate took this cycle
  int jj, ii;
  point_at<kPtBX, kPtBY>(d, bx, by, jj, ii);
  const int kk = bz;
  const int nj = d.nj, ni = d.ni;
  if (jj >= nj || ii >= ni) return;
  const size_t pl = d.pl;
  const int jm = wm1(jj, nj), jp = wp1(jj, nj), im = wm1(ii, ni), ip = wp1(ii, ni);
  const T* __restrict__ u = d.ubuf[d.cur];
  const T* __restrict__ v = d.vbuf[d.cur];
  T* __restrict__ uo = d.ubuf[d.cur ^ 1];
  T* __restrict__ vo = d.vbuf[d.cur ^ 1];
  const size_t c = (size_t)jj + (size_t)nj * ii;
  const size_t cw = (size_t)jm + (size_t)nj * ii, ce = (size_t)jp + (size_t)nj * ii;
  const size_t cs = (size_t)jj + (size_t)nj * im, cn = (size_t)jj + (size_t)nj * ip;
  const size_t cwn = (size_t)jm + (size_t)nj * ip, ces = (size_t)jp + (size_t)nj * im;
  const size_t o = (size_t)kk * pl, o1 = o + pl;
  const T dts = d.dts, egdts = d.egdts;
  const T dw_c = d.deltaw[c + o], dw_c1 = d.deltaw[c + o1];
  const T tc = d.tetav[c + o];
  const T pc = d.pai[c + o];
  const T gzh = d.gzitakh[kk];
  const T hcpd = T(0.5) * T(kCpd);
  // Equation 17
  {
    const T zcx = d.dtrdx * d.mu[c];
    const T zfz = egdts + T(0.25) * (((d.deltaw[cw + o] + d.deltaw[cw + o1]) + dw_c) + dw_c1);
    const T zrom1u = hcpd * (d.tetav[cw + o] + tc);
    const T vdc = v[c + o];
    const T vdw = jj == 0 ? d.ev_j[ii + (size_t)ni * kk] : v[cw + o];
    const T vdwn = jj == 0 ? d.ev_j[ip + (size_t)ni * kk] : (ii == ni - 1 ? d.ev_i[jm + (size_t)nj * kk] : v[cwn + o]);
    const T vdn = ii == ni - 1 ? d.ev_i[jj + (size_t)nj * kk] : v[cn + o];
    const T ucor = plus_cor(u[c + o], (d.coru[c] * dts) * T(0.25), ((vdc + vdw) + vdwn) + vdn, 1);
    const T paw = jj == 0 ? d.ep_j[ii + (size_t)ni * kk] : d.pai[cw + o];
    uo[c + o] = (ucor - (zfz * d.hx[c]) * gzh) - (zcx * zrom1u) * (pc - paw);
  }
  // Equation 18
  {
    const T zcy = d.rotllr ? d.dtrdy : d.dtrdy * d.mv[c];
    const T zfz = egdts + T(0.25) * (((d.deltaw[cs + o] + d.deltaw[cs + o1]) + dw_c) + dw_c1);
    const T zrom1v = hcpd * (d.tetav[cs + o] + tc);
    const T udc = u[c + o];
    const T uds = ii == 0 ? d.eu_i[jj + (size_t)nj * kk] : u[cs + o];
    const T ude = jj == nj - 1 ? d.eu_j[ii + (size_t)ni * kk] : u[ce + o];
    const T udes = jj == nj - 1 ? d.eu_j[im + (size_t)ni * kk] : (ii == 0 ? d.eu_i[jp + (size_t)nj * kk] : u[ces + o]);
    const T vcor = minus_cor(v[c + o], (d.corv[c] * dts) * T(0.25), ((udc + uds) + ude) + udes, 1);
    const T pas = ii == 0 ? d.ep_i[jj + (size_t)nj * kk] : d.pai[cs + o];
    vo[c + o] = (vcor - (zfz * d.hy[c]) * gzh) - (zcy * zrom1v) * (pc - pas);
  }
}

template <class T>
__global__ void __launch_bounds__(kPtBX* kPtBY) k_sound_momentum(View<T> d) {
  b_sound_momentum<T>(d, blockIdx.x, tile_y(d), blockIdx.z);
}

template <class T>
__global__ void __launch_bounds__(kPtBX* kPtBY)
    kb_sound_momentum(const View<T>* __restrict__ views, const int4* __restrict__ tiles) {
  __shared__ View<T> sv;
  const int4 t = tiles[blockIdx.x];
  copy_view(&sv, views + t.x);
  __syncthreads();
  b_sound_momentum<T>(sv, t.y, t.z, t.w);
}

// ---- k-marching variants of the point kernels of the sound loop ---------
// One thread per (j, i) and chunk of kKC levels; the inputs of level k+1
// are loaded into registers before level k is computed and stored, so each
// thread keeps a level of loads in flight (the one-level-per-thread
// versions above leave that to the warp scheduler and stall on latency).
// Same arithmetic, expression by expression.
template <class T>
__device__ __forceinline__ void b_sound_div_km(const View<T>& d, const int bx, const int by, const int bz) {
  if (d.sur_skip && *d.sur_skip) return;  // the surrogate took this cycle
  int jj, ii;
  point_at<kPtBX, kPtBY>(d, bx, by, jj, ii);
  const int nj = d.nj, ni = d.ni, kz = d.kz;
  if (jj >= nj || ii >= ni) return;
  const int k0 = bz * kKC, k1 = min(kz, k0 + kKC);
  const size_t pl = d.pl;
  const int jp = wp1(jj, nj), ip = wp1(ii, ni);
  const T* __restrict__ u = d.ubuf[d.cur];
  const T* __restrict__ v = d.vbuf[d.cur];
  const size_t c = (size_t)jj + (size_t)nj * ii;
  const size_t ce = (size_t)jp + (size_t)nj * ii;  // (j+1, i)
  const size_t cn = (size_t)jj + (size_t)nj * ip;  // (j, i+1)
  const T hx0 = d.hx[c], hx1 = d.hx[ce], hy0 = d.hy[c], hy1 = d.hy[cn];
  const T dtrdx = d.dtrdx, dtrdy = d.dtrdy;
  const T rmv0 = d.rmv[c], rmv1 = d.rmv[cn];
  const bool rot = d.rotllr;
  const T mxc = rot ? d.mx[c] : d.mx2[c];
  const T rmu0 = rot ? T(0) : d.rmu[c], rmu1 = rot ? T(0) : d.rmu[ce];
  T slope_p = T(0);  // u hx + v hy of level k-1 over the point's four faces (kLean)
  struct L { T u0, u1, v0, v1, f, rfw0, rfw1, rfs0, rfs1, gz; };
  auto load = [&](int k, L& x) {
    const size_t o = (size_t)k * pl;
    x.u0 = u[c + o]; x.u1 = u[ce + o]; x.v0 = v[c + o]; x.v1 = v[cn + o];
    x.f = kLean<T> ? d.fmx[c + o] : d.fmz[c + o];
    x.rfw0 = d.rfw[c + o]; x.rfw1 = d.rfw[ce + o]; x.rfs0 = d.rfs[c + o]; x.rfs1 = d.rfs[cn + o];
    x.gz = d.gzitak[k];
  };
  T u0p = T(0), u1p = T(0), v0p = T(0), v1p = T(0);  // level k-1
  if (k0 > 0) {
    const size_t q = (size_t)(k0 - 1) * pl;
    u0p = u[c + q]; u1p = u[ce + q]; v0p = v[c + q]; v1p = v[cn + q];
  }
  auto slope = [&](T a0, T a1, T b0, T b1) {
    return fma_rn(a0, hx0, fma_rn(a1, hx1, fma_rn(b0, hy0, mul_rn(b1, hy1))));
  };
  if constexpr (kLean<T>) slope_p = slope(u0p, u1p, v0p, v1p);
  L cur, nxt;
  load(k0, nxt);
  for (int kk = k0; kk < k1; ++kk) {
    cur = nxt;
    if (kk + 1 < k1) load(kk + 1, nxt);
    const size_t o = (size_t)kk * pl;
    const T u0 = cur.u0, u1 = cur.u1, v0 = cur.v0, v1 = cur.v1;
    if constexpr (kLean<T>) {
      // each level's slope term serves s(k) and s(k+1): 13 FP64 operations a
      // point (256 x 256 x 60: 2.81 -> 1.65 ms per step)
      const T sl = slope(u0, u1, v0, v1);
      if (kk > 0) d.s[c + o] = mul_rn(add_rn(sl, slope_p), mul_rn(T(-0.25), cur.gz));
      slope_p = sl;
      const T du = fma_rn(u1, cur.rfw1, -mul_rn(u0, cur.rfw0));
      const T dv = fma_rn(v1, cur.rfs1, -mul_rn(v0, cur.rfs0));
      d.zdiv2a[c + o] = mul_rn(cur.f, add_rn(du, dv));
    } else {
    if (kk > 0) {  // s(k), k = 2..kz  (:557-570)
      T zuh = prod_add(u0 + u0p, hx0, u1 + u1p, hx1);
      T zvh = prod_add(v0 + v0p, hy0, v1 + v1p, hy1);
      d.s[c + o] = -((T(0.25) * (zuh + zvh)) * cur.gz);
    }
    const T f = cur.f;
    if (rot) {
      const T du = prod_sub(dtrdx * u1, cur.rfw1, dtrdx * u0, cur.rfw0);
      const T dv = prod_sub((dtrdy * v1) * cur.rfs1, rmv1, (dtrdy * v0) * cur.rfs0, rmv0);
      d.zdiv2a[c + o] = (f * mxc) * (du + dv);
    } else {
      const T du = prod_sub((dtrdx * u1) * rmu1, cur.rfw1, (dtrdx * u0) * rmu0, cur.rfw0);
      const T dv = prod_sub((dtrdy * v1) * rmv1, cur.rfs1, (dtrdy * v0) * rmv0, cur.rfs0);
      d.zdiv2a[c + o] = (mxc * f) * (du + dv);
    }
    }
    if (jj == 0) d.eu_j[ii + (size_t)ni * kk] = u0;
    if (ii == ni - 1) d.eu_i[jj + (size_t)nj * kk] = u0;
    if (jj == nj - 1) d.ev_j[ii + (size_t)ni * kk] = v0;
    if (ii == 0) d.ev_i[jj + (size_t)nj * kk] = v0;
    if (kk == kz - 1) {  // surface w(kz+1), s(kz+1)
      T zuh = prod_add(u0, hx0, u1, hx1);
      T zvh = prod_add(v0, hy0, v1, hy1);
      T ws = T(0.5) * (zuh + zvh);
      d.w[c + (size_t)kz * pl] = ws;
      d.s[c + (size_t)kz * pl] = -ws;
    }
    u0p = u0; u1p = u1; v0p = v0; v1p = v1;
  }
}

template <class T>
__device__ __forceinline__ void b_sound_damp_km(const View<T>& d, const int bx, const int by, const int bz) {
  if (d.sur_skip && *d.sur_skip) return;  // the surrogate took this cycle
  int jj, ii;
  point_at<kPtBX, kPtBY>(d, bx, by, jj, ii);
  const int nj = d.nj, ni = d.ni;
  if (jj >= nj || ii >= ni) return;
  const int k0 = bz * kKC, k1 = min(d.kz, k0 + kKC);
  const size_t pl = d.pl;
  const size_t c = (size_t)jj + (size_t)nj * ii;
  const size_t cw = (size_t)wm1(jj, nj) + (size_t)nj * ii, ce = (size_t)wp1(jj, nj) + (size_t)nj * ii;
  const size_t cs = (size_t)jj + (size_t)nj * wm1(ii, ni), cn = (size_t)jj + (size_t)nj * wp1(ii, ni);
  T* __restrict__ u = d.ubuf[d.cur];
  T* __restrict__ v = d.vbuf[d.cur];
  const T muc = d.mu[c];
  const T mvc = d.rotllr ? T(0) : d.mv[c];
  const T ddamp2 = d.ddamp2, dtrdz = d.dtrdz;
  struct L { T zc, zw, ze, zs, zn, s1, uc, vc, fz, cd; };
  auto load = [&](int k, L& x) {
    const size_t o = (size_t)k * pl;
    x.zc = d.zdiv2a[c + o]; x.zw = d.zdiv2a[cw + o]; x.ze = d.zdiv2a[ce + o];
    x.zs = d.zdiv2a[cs + o]; x.zn = d.zdiv2a[cn + o];
    x.s1 = d.s[c + o + pl];
    x.uc = u[c + o]; x.vc = v[c + o];
    x.fz = kLean<T> ? d.fzd[c + o] : d.fmz[c + o];
    x.cd = d.cdamp[k];
  };
  T s_k = d.s[c + (size_t)k0 * pl];  // s(k); s(k+1) is carried to the next level
  L cur, nxt;
  load(k0, nxt);
  for (int kk = k0; kk < k1; ++kk) {
    cur = nxt;
    if (kk + 1 < k1) load(kk + 1, nxt);
    const size_t o = (size_t)kk * pl;
    const T zc = cur.zc, zw = cur.zw, ze = cur.ze, zs = cur.zs, zn = cur.zn, cd = cur.cd;
    u[c + o] = cur.uc + ((cd * muc) * (zc - zw));
    if (d.rotllr)
      v[c + o] = cur.vc + cd * (zc - zs);
    else
      v[c + o] = cur.vc + ((cd * mvc) * (zc - zs));
    if constexpr (kLean<T>) {
      d.zdiv2b[c + o] = damp_lean(ddamp2, zc, zw, ze, zs, zn, cur.fz, s_k, cur.s1);
      s_k = cur.s1;
      continue;
    }
    const T p2d = prod_sub(T(0.125), ((zw + ze) + zs) + zn, T(0.5), zc);
    T zd = zc + ddamp2 * p2d;
    zd = zd + (cur.fz * dtrdz) * (s_k - cur.s1);
    d.zdiv2b[c + o] = zd;
    s_k = cur.s1;
  }
}

template <class T>
__device__ __forceinline__ void b_sound_momentum_km(const View<T>& d, const int bx, const int by, const int bz) {
  if (d.sur_skip && *d.sur_skip) return;  // the surrogate took this cycle
  int jj, ii;
  point_at<kPtBX, kPtBY>(d, bx, by, jj, ii);
  const int nj = d.nj, ni = d.ni;
  if (jj >= nj || ii >= ni) return;
  const int k0 = bz * kKC, k1 = min(d.kz, k0 + kKC);
  const size_t pl = d.pl;
  const int jm = wm1(jj, nj), jp = wp1(jj, nj), im = wm1(ii, ni), ip = wp1(ii, ni);
  const T* __restrict__ u = d.ubuf[d.cur];
  const T* __restrict__ v = d.vbuf[d.cur];
  T* __restrict__ uo = d.ubuf[d.cur ^ 1];
  T* __restrict__ vo = d.vbuf[d.cur ^ 1];
  const size_t c = (size_t)jj + (size_t)nj * ii;
  const size_t cw = (size_t)jm + (size_t)nj * ii, ce = (size_t)jp + (size_t)nj * ii;
  const size_t cs = (size_t)jj + (size_t)nj * im, cn = (size_t)jj + (size_t)nj * ip;
  const size_t cwn = (size_t)jm + (size_t)nj * ip, ces = (size_t)jp + (size_t)nj * im;
  const T dts = d.dts, egdts = d.egdts;
  const T hcpd = T(0.5) * T(kCpd);
  const T zcx = d.dtrdx * d.mu[c];
  const T zcy = d.rotllr ? d.dtrdy : d.dtrdy * d.mv[c];
  const T corx = (d.coru[c] * dts) * T(0.25), cory = (d.corv[c] * dts) * T(0.25);
  const T hxc = d.hx[c], hyc = d.hy[c];
  const T zcxh = hcpd * zcx, zcyh = hcpd * zcy;
  struct L { T dwc1, dww1, dws1, tc, tw, ts, pc, pw, ps, uc, us, ue, ues, vc, vw, vwn, vn, gzh; };
  auto load = [&](int k, L& x) {
    const size_t o = (size_t)k * pl, o1 = o + pl;
    x.dwc1 = d.deltaw[c + o1]; x.dww1 = d.deltaw[cw + o1]; x.dws1 = d.deltaw[cs + o1];
    x.tc = d.tetav[c + o]; x.tw = d.tetav[cw + o]; x.ts = d.tetav[cs + o];
    x.pc = d.pai[c + o];
    x.pw = jj == 0 ? d.ep_j[ii + (size_t)ni * k] : d.pai[cw + o];
    x.ps = ii == 0 ? d.ep_i[jj + (size_t)nj * k] : d.pai[cs + o];
    x.vc = v[c + o];
    x.vw = jj == 0 ? d.ev_j[ii + (size_t)ni * k] : v[cw + o];
    x.vwn = jj == 0 ? d.ev_j[ip + (size_t)ni * k] : (ii == ni - 1 ? d.ev_i[jm + (size_t)nj * k] : v[cwn + o]);
    x.vn = ii == ni - 1 ? d.ev_i[jj + (size_t)nj * k] : v[cn + o];
    x.uc = u[c + o];
    x.us = ii == 0 ? d.eu_i[jj + (size_t)nj * k] : u[cs + o];
    x.ue = jj == nj - 1 ? d.eu_j[ii + (size_t)ni * k] : u[ce + o];
    x.ues = jj == nj - 1 ? d.eu_j[im + (size_t)ni * k] : (ii == 0 ? d.eu_i[jp + (size_t)nj * k] : u[ces + o]);
    x.gzh = d.gzitakh[k];
  };
  // deltaw at level k of (c, w, s); level k+1 is carried to the next level
  T dw_c = d.deltaw[c + (size_t)k0 * pl], dw_w = d.deltaw[cw + (size_t)k0 * pl];
  T dw_s = d.deltaw[cs + (size_t)k0 * pl];
  L cur, nxt;
  load(k0, nxt);
  for (int kk = k0; kk < k1; ++kk) {
    cur = nxt;
    if (kk + 1 < k1) load(kk + 1, nxt);
    const size_t o = (size_t)kk * pl;
    const T tc = cur.tc, pc = cur.pc, gzh = cur.gzh;
    if constexpr (kLean<T>) {
      // layer sums of deltaw and the metric products formed once: 27 FP64
      // operations a point instead of 32 (256 x 256 x 60: 3.97 -> 3.73 ms per
      // step)
      const T d2 = add_rn(dw_c, cur.dwc1);
      const T zu = fma_rn(T(0.25), add_rn(add_rn(dw_w, cur.dww1), d2), egdts);
      const T zv = fma_rn(T(0.25), add_rn(add_rn(dw_s, cur.dws1), d2), egdts);
      const T cu = add_rn(add_rn(cur.vc, cur.vw), add_rn(cur.vwn, cur.vn));
      const T cv = add_rn(add_rn(cur.uc, cur.us), add_rn(cur.ue, cur.ues));
      const T pu = mul_rn(add_rn(cur.tw, tc), zcxh), pv = mul_rn(add_rn(cur.ts, tc), zcyh);
      uo[c + o] = fma_rn(-pu, sub_rn(pc, cur.pw), fma_rn(-zu, mul_rn(hxc, gzh), fma_rn(corx, cu, cur.uc)));
      vo[c + o] = fma_rn(-pv, sub_rn(pc, cur.ps), fma_rn(-zv, mul_rn(hyc, gzh), fma_rn(-cory, cv, cur.vc)));
      dw_c = cur.dwc1; dw_w = cur.dww1; dw_s = cur.dws1;
      continue;
    }
    // Equation 17
    {
      const T zfz = egdts + T(0.25) * (((dw_w + cur.dww1) + dw_c) + cur.dwc1);
      const T zrom1u = hcpd * (cur.tw + tc);
      const T ucor = plus_cor(cur.uc, corx, ((cur.vc + cur.vw) + cur.vwn) + cur.vn, 0);
      uo[c + o] = (ucor - (zfz * hxc) * gzh) - (zcx * zrom1u) * (pc - cur.pw);
    }
    // Equation 18
    {
      const T zfz = egdts + T(0.25) * (((dw_s + cur.dws1) + dw_c) + cur.dwc1);
      const T zrom1v = hcpd * (cur.ts + tc);
      const T vcor = minus_cor(cur.vc, cory, ((cur.uc + cur.us) + cur.ue) + cur.ues, 0);
      vo[c + o] = (vcor - (zfz * hyc) * gzh) - (zcy * zrom1v) * (pc - cur.ps);
    }
    dw_c = cur.dwc1; dw_w = cur.dww1; dw_s = cur.dws1;
  }
}

#define MOLOCH_KM_KERNELS(NAME)                                                                      \
  template <class T>                                                                                 \
  __global__ void __launch_bounds__(kPtBX* kPtBY) k_##NAME##_km(View<T> d) {                          \
    b_##NAME##_km<T>(d, blockIdx.x, tile_y(d), blockIdx.z);                                         \
  }                                                                                                  \
  template <class T>                                                                                 \
  __global__ void __launch_bounds__(kPtBX* kPtBY)                                                    \
      kb_##NAME##_km(const View<T>* __restrict__ views, const int4* __restrict__ tiles) {            \
    __shared__ View<T> sv;                                                                           \
    const int4 t = tiles[blockIdx.x];                                                                \
    copy_view(&sv, views + t.x);                                                                     \
    __syncthreads();                                                                                 \
    b_##NAME##_km<T>(sv, t.y, t.z, t.w);                                                             \
  }
MOLOCH_KM_KERNELS(sound_div)
MOLOCH_KM_KERNELS(sound_damp)
MOLOCH_KM_KERNELS(sound_momentum)
#undef MOLOCH_KM_KERNELS


// ---- momentum as warp strips (:730-837) -------------------------------------
// asynchronous global -> shared copies (cp.async, one element per lane)
template <class T>
__device__ __forceinline__ void cp_async_elem(T* dst_smem, const T* src) {
  const uint32_t dst = static_cast<uint32_t>(__cvta_generic_to_shared(dst_smem));
  if constexpr (sizeof(T) == 4)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// One warp per strip of 30 output columns x R rows of one level, lanes on
// columns j0-1 .. j0+30.  West and east neighbours come from the lanes
// beside (shuffles), the row below and the row above (v at i+1) from a ring
// of kMomS row slots in shared memory: the six state arrays of a row (u, v,
// tetav, pai, deltaw at k and k+1) are copied there with cp.async
// kMomS - 3 rows ahead of the row computed, each lane copying and later
// reading only its own column, so the pipeline needs no warp barrier and
// holds no registers; the 2-D metric fields come one row ahead in
// registers.  The stale-halo reads of the reference (edge buffers at
// j = 1, j = nj, i = 1, i = ni) replace the neighbour values on those lanes
// and rows, as in k_sound_momentum.
constexpr int kMomS = 6;  // row slots: rows i-1, i, i+1 and three in flight
template <class T>
using MomSlots = T[kMomS][6][32];  // one warp's ring: [slot][array][lane]
template <class T>
using MomRing = MomSlots<T>[4];    // [warp] of a 128-thread block

// bx: block of nw strips, wid: this warp's strip in it, rg: its ring
template <class T>
__device__ __forceinline__ void b_momentum_strip(const View<T>& d, const int bx, const int k, const int R,
                                                 MomSlots<T>& rg, const int wid, const int nw) {
  if (d.sur_skip && *d.sur_skip) return;  // the surrogate took this cycle
  const int lane = threadIdx.x & 31;
  const int nj = d.nj, ni = d.ni, pl = d.pl;
  const int nsj = (nj + kMomJ - 1) / kMomJ, nsi = (ni + R - 1) / R;
  const int w = bx * nw + wid;
  if (w >= nsj * nsi) return;  // whole warp
  const int sj = w % nsj, si = w / nsj;
  const int jl = sj * kMomJ - 1 + lane;
  const int jj = wrapn(jl, nj);
  const bool out_lane = lane >= 1 && lane <= kMomJ && jl < nj;
  const int i_s = si * R, i_e = min(i_s + R, ni);
  const size_t o = (size_t)k * pl, o1 = o + pl;
  const T* __restrict__ u = d.ubuf[d.cur] + o;
  const T* __restrict__ v = d.vbuf[d.cur] + o;
  T* __restrict__ uo = d.ubuf[d.cur ^ 1] + o;
  T* __restrict__ vo = d.vbuf[d.cur ^ 1] + o;
  const T* __restrict__ tet = d.tetav + o;
  const T* __restrict__ pai = d.pai + o;
  const T* __restrict__ dw0 = d.deltaw + o;
  const T* __restrict__ dw1 = d.deltaw + o1;
  const T dts = d.dts, egdts = d.egdts, dtrdx = d.dtrdx, dtrdy = d.dtrdy;
  const T hcpd = T(0.5) * T(kCpd);
  const T gzh = d.gzitakh[k];
  const bool rot = d.rotllr;
  const int rounded = d.cor_rounded;
  const int jm = wm1(jj, nj), jp = wp1(jj, nj);
  // rows i_s-1 .. i_e stream through the slots in order; the slot indices
  // rotate by one per row
  auto nxt = [](int q) { return q + 1 == kMomS ? 0 : q + 1; };
  auto issue = [&](int r, int q) {  // copies of row r into slot q (nothing past i_e); one group either way
    if (r <= i_e) {
      const size_t c = (size_t)jj + (size_t)nj * wrap2(r, ni);
      T(*const sl)[32] = rg[q];
      cp_async_elem(&sl[0][lane], u + c);
      cp_async_elem(&sl[1][lane], v + c);
      cp_async_elem(&sl[2][lane], tet + c);
      cp_async_elem(&sl[3][lane], pai + c);
      cp_async_elem(&sl[4][lane], dw0 + c);
      cp_async_elem(&sl[5][lane], dw1 + c);
    }
    cp_async_commit();
  };
  // 2-D fields of a row, one row ahead in registers
  struct Row2 { T coru, corv, hx, hy, mu, mv; };
  auto load2 = [&](int i, Row2& x) {
    const size_t c = (size_t)jj + (size_t)nj * wrap2(i, ni);
    x.coru = d.coru[c]; x.corv = d.corv[c]; x.hx = d.hx[c]; x.hy = d.hy[c]; x.mu = d.mu[c];
    x.mv = rot ? T(0) : d.mv[c];
  };
  for (int r = i_s - 1, q = 0; r <= i_s + kMomS - 3; ++r, ++q) issue(r, q);
  Row2 c2, n2;
  load2(i_s, n2);
  // slots of rows i-1, i, i+1 and of the row issued next (i + kMomS - 2)
  int qb = 0, qc = 1, qn = 2, qi = kMomS - 1;
  // a strip that touches none of the domain edges (j = 1, nj; i = 1, ni)
  // never reads the stale-halo edge buffers: its rows run a copy of the
  // step without those tests
  const bool interior = sj != 0 && sj != nsj - 1 && i_s != 0 && i_e != ni;
  auto row = [&](const int i, auto edge) {
    constexpr bool EDGE = decltype(edge)::value;
    issue(i + kMomS - 2, qi);        // into the slot of row i-2
    cp_async_wait<kMomS - 3>();      // rows up to i+1 have landed
    c2 = n2;
    if (i + 1 < i_e) load2(i + 1, n2);
    const T(*const sb)[32] = rg[qb];
    const T(*const sc)[32] = rg[qc];
    const T(*const sn)[32] = rg[qn];
    const T cu = sc[0][lane], cv = sc[1][lane], ct = sc[2][lane], cp = sc[3][lane];
    const T cd0 = sc[4][lane], cd1 = sc[5][lane];
    const T us = sb[0][lane], ts = sb[2][lane], ps = sb[3][lane], ds0 = sb[4][lane], ds1 = sb[5][lane];
    const T vn = sn[1][lane];
    const int ii = i;
    // neighbours from the lanes beside
    const T ue = __shfl_down_sync(0xffffffffu, cu, 1);
    const T ues = __shfl_down_sync(0xffffffffu, us, 1);
    const T vw = __shfl_up_sync(0xffffffffu, cv, 1);
    const T vwn = __shfl_up_sync(0xffffffffu, vn, 1);
    const T tw = __shfl_up_sync(0xffffffffu, ct, 1);
    const T pw = __shfl_up_sync(0xffffffffu, cp, 1);
    const T dw0w = __shfl_up_sync(0xffffffffu, cd0, 1);
    const T dw1w = __shfl_up_sync(0xffffffffu, cd1, 1);
    if (out_lane) {
      const T dw_c = cd0, dw_c1 = cd1;
      const T tc = ct, pc = cp;
      // Equation 17
      {
        const T zcx = dtrdx * c2.mu;
        const T zfz = egdts + T(0.25) * (((dw0w + dw1w) + dw_c) + dw_c1);
        const T zrom1u = hcpd * (tw + tc);
        const T vdc = cv;
        T vdw = vw, vdwn = vwn, vdn = vn, paw = pw;
        if (EDGE) {
          const int ip = wp1(ii, ni);
          vdw = jj == 0 ? d.ev_j[ii + (size_t)ni * k] : vw;
          vdwn = jj == 0 ? d.ev_j[ip + (size_t)ni * k] : (ii == ni - 1 ? d.ev_i[jm + (size_t)nj * k] : vwn);
          vdn = ii == ni - 1 ? d.ev_i[jj + (size_t)nj * k] : vn;
          paw = jj == 0 ? d.ep_j[ii + (size_t)ni * k] : pw;
        }
        const T ucor = plus_cor(cu, (c2.coru * dts) * T(0.25), ((vdc + vdw) + vdwn) + vdn, rounded);
        uo[(size_t)jj + (size_t)nj * ii] = (ucor - (zfz * c2.hx) * gzh) - (zcx * zrom1u) * (pc - paw);
      }
      // Equation 18
      {
        const T zcy = rot ? dtrdy : dtrdy * c2.mv;
        const T zfz = egdts + T(0.25) * (((ds0 + ds1) + dw_c) + dw_c1);
        const T zrom1v = hcpd * (ts + tc);
        const T udc = cu;
        T uds = us, ude = ue, udes = ues, pas = ps;
        if (EDGE) {
          const int im = wm1(ii, ni);
          uds = ii == 0 ? d.eu_i[jj + (size_t)nj * k] : us;
          ude = jj == nj - 1 ? d.eu_j[ii + (size_t)ni * k] : ue;
          udes = jj == nj - 1 ? d.eu_j[im + (size_t)ni * k] : (ii == 0 ? d.eu_i[jp + (size_t)nj * k] : ues);
          pas = ii == 0 ? d.ep_i[jj + (size_t)nj * k] : ps;
        }
        const T vcor = minus_cor(cv, (c2.corv * dts) * T(0.25), ((udc + uds) + ude) + udes, rounded);
        vo[(size_t)jj + (size_t)nj * ii] = (vcor - (zfz * c2.hy) * gzh) - (zcy * zrom1v) * (pc - pas);
      }
    }
    qb = qc; qc = qn; qn = nxt(qn); qi = nxt(qi);
  };
  if (interior)
    for (int i = i_s; i < i_e; ++i) row(i, std::false_type());
  else
    for (int i = i_s; i < i_e; ++i) row(i, std::true_type());
  cp_async_wait<0>();  // no copy outlives the kernel
}

template <class T>
__global__ void __launch_bounds__(128, sizeof(T) == 4 ? 8 : 4) k_momentum_strip(View<T> d, int R) {
  __shared__ __align__(16) MomRing<T> ring;
  b_momentum_strip<T>(d, blockIdx.x, blockIdx.y, R, ring[threadIdx.x >> 5], threadIdx.x >> 5, 4);
}

template <class T>
__global__ void __launch_bounds__(128)
    kb_momentum_strip(const View<T>* __restrict__ views, const int4* __restrict__ tiles, int R) {
  __shared__ View<T> sv;
  __shared__ __align__(16) MomRing<T> ring;
  const int4 t = tiles[blockIdx.x];
  copy_view(&sv, views + t.x);
  __syncthreads();
  b_momentum_strip<T>(sv, t.y, t.z, R, ring[threadIdx.x >> 5], threadIdx.x >> 5, 4);
}

// ---- momentum as warp strips, two columns per lane (FP32, jx even) --------
// b_momentum_strip with each lane on a pair of adjacent columns: strip s
// computes columns 62 s - 1 .. 62 s + 60 (inside the domain), lane l holds
// columns 62 s - 2 + 2 l and the next one, so a warp covers 62 output
// columns with 64 loaded.  The six state arrays of a row arrive as one
// 8-byte cp.async copy per array and lane, the metric fields as 8-byte
// loads; a west or east neighbour is the lane's own other column or one
// shuffle of the lane beside (half the copies, shared loads, shuffles and
// address arithmetic per point of the one-column strips).  Pairs start at
// even columns, and with jx even a pair never straddles the periodic seam,
// so every copy and load is 8-byte aligned.  The same expressions in the
// same order as b_momentum_strip: the results are bit-identical.
constexpr int kMom2J = 62;
constexpr int kMom2S = 6;  // row slots: rows i-1, i, i+1 and three in flight
using Mom2Slots = float[kMom2S][6][64];  // one warp's ring: [slot][array][column]

__device__ __forceinline__ void cp_async_8(void* dst_smem, const void* src) {
  const uint32_t dst = static_cast<uint32_t>(__cvta_generic_to_shared(dst_smem));
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}

__device__ __forceinline__ void b_momentum_strip2(const View<float>& d, const int bx, const int k, const int R,
                                                  Mom2Slots& rg, const int wid, const int nw) {
  if (d.sur_skip && *d.sur_skip) return;  // the surrogate took this cycle
  const int lane = threadIdx.x & 31;
  const int nj = d.nj, ni = d.ni, pl = d.pl;
  const int nsj = (nj + 1 + kMom2J - 1) / kMom2J, nsi = (ni + R - 1) / R;
  const int w = bx * nw + wid;
  if (w >= nsj * nsi) return;  // whole warp
  const int sj = w % nsj, si = w / nsj;
  const int cl = kMom2J * sj - 2 + 2 * lane;  // first column of the pair, before wrapping
  const int ja = wrapn(cl, nj), jb = ja + 1;  // ja even, so jb < nj
  const bool out0 = lane >= 1 && cl >= 0 && cl < nj;
  const bool out1 = lane <= 30 && cl + 1 >= 0 && cl + 1 < nj;
  const int i_s = si * R, i_e = min(i_s + R, ni);
  const size_t o = (size_t)k * pl, o1 = o + pl;
  const float* __restrict__ u = d.ubuf[d.cur] + o;
  const float* __restrict__ v = d.vbuf[d.cur] + o;
  float* __restrict__ uo = d.ubuf[d.cur ^ 1] + o;
  float* __restrict__ vo = d.vbuf[d.cur ^ 1] + o;
  const float* __restrict__ tet = d.tetav + o;
  const float* __restrict__ pai = d.pai + o;
  const float* __restrict__ dw0 = d.deltaw + o;
  const float* __restrict__ dw1 = d.deltaw + o1;
  const float dts = d.dts, egdts = d.egdts, dtrdx = d.dtrdx, dtrdy = d.dtrdy;
  const float hcpd = 0.5f * float(kCpd);
  const float gzh = d.gzitakh[k];
  const bool rot = d.rotllr;
  const int rounded = d.cor_rounded;
  auto nxt = [](int q) { return q + 1 == kMom2S ? 0 : q + 1; };
  auto issue = [&](int r, int q) {  // copies of row r into slot q (nothing past i_e); one group either way
    if (r <= i_e) {
      const size_t c = (size_t)ja + (size_t)nj * wrap2(r, ni);
      float(*const sl)[64] = rg[q];
      cp_async_8(&sl[0][2 * lane], u + c);
      cp_async_8(&sl[1][2 * lane], v + c);
      cp_async_8(&sl[2][2 * lane], tet + c);
      cp_async_8(&sl[3][2 * lane], pai + c);
      cp_async_8(&sl[4][2 * lane], dw0 + c);
      cp_async_8(&sl[5][2 * lane], dw1 + c);
    }
    cp_async_commit();
  };
  struct Row2 { float2 coru, corv, hx, hy, mu, mv; };
  auto ld2 = [](const float* p) { return *reinterpret_cast<const float2*>(p); };
  auto load2 = [&](int i, Row2& x) {
    const size_t c = (size_t)ja + (size_t)nj * wrap2(i, ni);
    x.coru = ld2(d.coru + c); x.corv = ld2(d.corv + c); x.hx = ld2(d.hx + c); x.hy = ld2(d.hy + c);
    x.mu = ld2(d.mu + c);
    x.mv = rot ? make_float2(0.f, 0.f) : ld2(d.mv + c);
  };
  for (int r = i_s - 1, q = 0; r <= i_s + kMom2S - 3; ++r, ++q) issue(r, q);
  Row2 c2, n2;
  load2(i_s, n2);
  int qb = 0, qc = 1, qn = 2, qi = kMom2S - 1;
  const bool interior = sj != 0 && sj != nsj - 1 && i_s != 0 && i_e != ni;
  // one column: its values, its west / east neighbours and metric terms
  struct Col { float cu, cv, ct, cp, cd0, cd1, us, ts, ps, ds0, ds1, vn; };
  auto point = [&](const int jj, const int ii, const Col& x, const float vw, const float vwn, const float tw,
                   const float pw, const float dw0w, const float dw1w, const float ue, const float ues,
                   const float coru, const float corv, const float hx, const float hy, const float mu,
                   const float mv, auto edge, float& un, float& vnew) {
    constexpr bool EDGE = decltype(edge)::value;
    // Equation 17
    {
      const float zcx = dtrdx * mu;
      const float zfz = egdts + 0.25f * (((dw0w + dw1w) + x.cd0) + x.cd1);
      const float zrom1u = hcpd * (tw + x.ct);
      float vdw = vw, vdwn = vwn, vdn = x.vn, paw = pw;
      if (EDGE) {
        const int ip = wp1(ii, ni), jm = wm1(jj, nj);
        vdw = jj == 0 ? d.ev_j[ii + (size_t)ni * k] : vw;
        vdwn = jj == 0 ? d.ev_j[ip + (size_t)ni * k] : (ii == ni - 1 ? d.ev_i[jm + (size_t)nj * k] : vwn);
        vdn = ii == ni - 1 ? d.ev_i[jj + (size_t)nj * k] : x.vn;
        paw = jj == 0 ? d.ep_j[ii + (size_t)ni * k] : pw;
      }
      const float ucor = plus_cor(x.cu, (coru * dts) * 0.25f, ((x.cv + vdw) + vdwn) + vdn, rounded);
      un = (ucor - (zfz * hx) * gzh) - (zcx * zrom1u) * (x.cp - paw);
    }
    // Equation 18
    {
      const float zcy = rot ? dtrdy : dtrdy * mv;
      const float zfz = egdts + 0.25f * (((x.ds0 + x.ds1) + x.cd0) + x.cd1);
      const float zrom1v = hcpd * (x.ts + x.ct);
      float uds = x.us, ude = ue, udes = ues, pas = x.ps;
      if (EDGE) {
        const int im = wm1(ii, ni), jp = wp1(jj, nj);
        uds = ii == 0 ? d.eu_i[jj + (size_t)nj * k] : x.us;
        ude = jj == nj - 1 ? d.eu_j[ii + (size_t)ni * k] : ue;
        udes = jj == nj - 1 ? d.eu_j[im + (size_t)ni * k] : (ii == 0 ? d.eu_i[jp + (size_t)nj * k] : ues);
        pas = ii == 0 ? d.ep_i[jj + (size_t)nj * k] : x.ps;
      }
      const float vcor = minus_cor(x.cv, (corv * dts) * 0.25f, ((x.cu + uds) + ude) + udes, rounded);
      vnew = (vcor - (zfz * hy) * gzh) - (zcy * zrom1v) * (x.cp - pas);
    }
  };
  auto row = [&](const int i, auto edge) {
    issue(i + kMom2S - 2, qi);   // into the slot of row i-2
    cp_async_wait<kMom2S - 3>();  // rows up to i+1 have landed
    c2 = n2;
    if (i + 1 < i_e) load2(i + 1, n2);
    auto lds2 = [&](int q, int a) { return *reinterpret_cast<const float2*>(&rg[q][a][2 * lane]); };
    const float2 cu = lds2(qc, 0), cv = lds2(qc, 1), ct = lds2(qc, 2), cp = lds2(qc, 3);
    const float2 cd0 = lds2(qc, 4), cd1 = lds2(qc, 5);
    const float2 us = lds2(qb, 0), ts = lds2(qb, 2), ps = lds2(qb, 3), ds0 = lds2(qb, 4), ds1 = lds2(qb, 5);
    const float2 vn = lds2(qn, 1);
    // east neighbours of the second column: the next lane's first
    const float ue1 = __shfl_down_sync(0xffffffffu, cu.x, 1);
    const float ues1 = __shfl_down_sync(0xffffffffu, us.x, 1);
    // west neighbours of the first column: the previous lane's second
    const float vw0 = __shfl_up_sync(0xffffffffu, cv.y, 1);
    const float vwn0 = __shfl_up_sync(0xffffffffu, vn.y, 1);
    const float tw0 = __shfl_up_sync(0xffffffffu, ct.y, 1);
    const float pw0 = __shfl_up_sync(0xffffffffu, cp.y, 1);
    const float dw0w0 = __shfl_up_sync(0xffffffffu, cd0.y, 1);
    const float dw1w0 = __shfl_up_sync(0xffffffffu, cd1.y, 1);
    const Col xa{cu.x, cv.x, ct.x, cp.x, cd0.x, cd1.x, us.x, ts.x, ps.x, ds0.x, ds1.x, vn.x};
    const Col xb{cu.y, cv.y, ct.y, cp.y, cd0.y, cd1.y, us.y, ts.y, ps.y, ds0.y, ds1.y, vn.y};
    float ua = 0.f, va = 0.f, ub = 0.f, vb = 0.f;
    if (out0)
      point(ja, i, xa, vw0, vwn0, tw0, pw0, dw0w0, dw1w0, cu.y, us.y, c2.coru.x, c2.corv.x, c2.hx.x, c2.hy.x,
            c2.mu.x, c2.mv.x, edge, ua, va);
    if (out1)
      point(jb, i, xb, cv.x, vn.x, ct.x, cp.x, cd0.x, cd1.x, ue1, ues1, c2.coru.y, c2.corv.y, c2.hx.y, c2.hy.y,
            c2.mu.y, c2.mv.y, edge, ub, vb);
    const size_t c = (size_t)ja + (size_t)nj * i;
    if (out0 && out1) {
      *reinterpret_cast<float2*>(uo + c) = make_float2(ua, ub);
      *reinterpret_cast<float2*>(vo + c) = make_float2(va, vb);
    } else if (out0) {
      uo[c] = ua;
      vo[c] = va;
    } else if (out1) {
      uo[c + 1] = ub;
      vo[c + 1] = vb;
    }
    qb = qc; qc = qn; qn = nxt(qn); qi = nxt(qi);
  };
  if (interior)
    for (int i = i_s; i < i_e; ++i) row(i, std::false_type());
  else
    for (int i = i_s; i < i_e; ++i) row(i, std::true_type());
  cp_async_wait<0>();  // no copy outlives the kernel
}

__global__ void __launch_bounds__(128, 5) k_momentum_strip2(View<float> d, int R) {
  __shared__ __align__(16) Mom2Slots ring[4];
  b_momentum_strip2(d, blockIdx.x, blockIdx.y, R, ring[threadIdx.x >> 5], threadIdx.x >> 5, 4);
}

// ---- momentum with four columns per thread (FP32, jx a multiple of 4) -----
// One thread per quad of columns, row and level: every array of the stencil
// is read with 16-byte loads, all issued before the first use, the west and
// east neighbours come from the lanes beside (from memory on the warp's end
// lanes), and the stale-halo rows of the reference (:716-735) are read
// through the row pointers, so no column tests them.
__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void st4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
constexpr int kQuadY = 4;  // rows of a block of the quad kernels, one warp (128 columns) each

__global__ void __launch_bounds__(32 * kQuadY, 5) k_momentum_quad(const __grid_constant__ View<float> d) {
  if (d.sur_skip && *d.sur_skip) return;  // the surrogate took this cycle
  const int nj = d.nj, ni = d.ni, k = blockIdx.z;
  const unsigned pl = (unsigned)d.pl, o = (unsigned)k * pl;
  const int lane = threadIdx.x, ii = blockIdx.y * kQuadY + threadIdx.y;
  if (ii >= ni) return;  // whole warp
  const int jq = 4 * (blockIdx.x * 32 + lane);
  const bool in = jq < nj;
  const int j0 = in ? jq : 0;  // lanes past the row repeat its first quad
  const unsigned r = (unsigned)nj * ii, rs = (unsigned)nj * wm1(ii, ni), ej = (unsigned)ni * k, ei = (unsigned)nj * k;
  const float* __restrict__ u = d.ubuf[d.cur] + o + r;
  const float* __restrict__ v = d.vbuf[d.cur] + o + r;
  const float* __restrict__ t = d.tetav + o;
  const float* __restrict__ p = d.pai + o + r;
  const float* __restrict__ dw = d.deltaw + o;
  // rows i-1 and i+1 whose periodic image is the older halo value
  const float* __restrict__ us = ii == 0 ? d.eu_i + ei : u - nj;
  const float* __restrict__ ps = ii == 0 ? d.ep_i + ei : p - nj;
  const float* __restrict__ vn = ii == ni - 1 ? d.ev_i + ei : v + nj;
  const float4 U = ld4(u + j0), V = ld4(v + j0), T = ld4(t + r + j0), P = ld4(p + j0);
  const float4 D0 = ld4(dw + r + j0), D1 = ld4(dw + pl + r + j0);
  const float4 US = ld4(us + j0), VN = ld4(vn + j0), TS = ld4(t + rs + j0), PS = ld4(ps + j0);
  const float4 S0 = ld4(dw + rs + j0), S1 = ld4(dw + pl + rs + j0);
  const float4 CU = ld4(d.coru + r + j0), CV = ld4(d.corv + r + j0), HX = ld4(d.hx + r + j0), HY = ld4(d.hy + r + j0);
  const float4 MU = ld4(d.mu + r + j0);
  const bool rot = d.rotllr;
  const int rounded = d.cor_rounded;
  const float4 MV = rot ? make_float4(0.f, 0.f, 0.f, 0.f) : ld4(d.mv + r + j0);
  // column j0-1 of v, v(i+1), tetav, pai, deltaw and column j0+4 of u, u(i-1)
  float vw = 0.f, vnw = 0.f, tw = 0.f, pw = 0.f, dw0 = 0.f, dw1 = 0.f, ue = 0.f, use = 0.f;
  if (lane == 0) {
    if (j0 == 0) {
      vw = d.ev_j[ej + ii]; vnw = d.ev_j[ej + wp1(ii, ni)]; pw = d.ep_j[ej + ii];
    } else {
      vw = v[j0 - 1]; vnw = vn[j0 - 1]; pw = p[j0 - 1];
    }
    const unsigned jw = r + (j0 == 0 ? nj : j0) - 1;
    tw = t[jw]; dw0 = dw[jw]; dw1 = dw[pl + jw];
  }
  if (lane == 31 || j0 + 4 >= nj) {
    if (j0 + 4 >= nj) {
      ue = d.eu_j[ej + ii]; use = d.eu_j[ej + wm1(ii, ni)];
    } else {
      ue = u[j0 + 4]; use = us[j0 + 4];
    }
  }
  auto west = [&](float x, float own) {
    const float y = __shfl_up_sync(0xffffffffu, x, 1);
    return lane == 0 ? own : y;
  };
  auto east = [&](float x, float own) {
    const float y = __shfl_down_sync(0xffffffffu, x, 1);
    return lane == 31 || j0 + 4 >= nj ? own : y;
  };
  vw = west(V.w, vw); vnw = west(VN.w, vnw); tw = west(T.w, tw); pw = west(P.w, pw);
  dw0 = west(D0.w, dw0); dw1 = west(D1.w, dw1);
  ue = east(U.x, ue); use = east(US.x, use);
  const float dts = d.dts, egdts = d.egdts, dtrdx = d.dtrdx, dtrdy = d.dtrdy, hcpd = 0.5f * float(kCpd);
  const float gzh = d.gzitakh[k];
  auto eq17 = [&](float cu, float cv, float wv, float wvn, float cvn, float wt, float ct, float wp, float cp, float wd0,
                  float wd1, float cd0, float cd1, float coru, float hx, float mu) {
    const float zcx = dtrdx * mu;
    const float zfz = egdts + 0.25f * (((wd0 + wd1) + cd0) + cd1);
    const float zrom1u = hcpd * (wt + ct);
    const float ucor = plus_cor(cu, (coru * dts) * 0.25f, ((cv + wv) + wvn) + cvn, rounded);
    return (ucor - (zfz * hx) * gzh) - (zcx * zrom1u) * (cp - wp);
  };
  auto eq18 = [&](float cv, float cu, float su, float eu, float esu, float st, float ct, float sp, float cp, float sd0,
                  float sd1, float cd0, float cd1, float corv, float hy, float mv) {
    const float zcy = rot ? dtrdy : dtrdy * mv;
    const float zfz = egdts + 0.25f * (((sd0 + sd1) + cd0) + cd1);
    const float zrom1v = hcpd * (st + ct);
    const float vcor = minus_cor(cv, (corv * dts) * 0.25f, ((cu + su) + eu) + esu, rounded);
    return (vcor - (zfz * hy) * gzh) - (zcy * zrom1v) * (cp - sp);
  };
  if (!in) return;
  const unsigned c = o + r + j0;
  st4(d.ubuf[d.cur ^ 1] + c,
      make_float4(eq17(U.x, V.x, vw, vnw, VN.x, tw, T.x, pw, P.x, dw0, dw1, D0.x, D1.x, CU.x, HX.x, MU.x),
                  eq17(U.y, V.y, V.x, VN.x, VN.y, T.x, T.y, P.x, P.y, D0.x, D1.x, D0.y, D1.y, CU.y, HX.y, MU.y),
                  eq17(U.z, V.z, V.y, VN.y, VN.z, T.y, T.z, P.y, P.z, D0.y, D1.y, D0.z, D1.z, CU.z, HX.z, MU.z),
                  eq17(U.w, V.w, V.z, VN.z, VN.w, T.z, T.w, P.z, P.w, D0.z, D1.z, D0.w, D1.w, CU.w, HX.w, MU.w)));
  st4(d.vbuf[d.cur ^ 1] + c,
      make_float4(eq18(V.x, U.x, US.x, U.y, US.y, TS.x, T.x, PS.x, P.x, S0.x, S1.x, D0.x, D1.x, CV.x, HY.x, MV.x),
                  eq18(V.y, U.y, US.y, U.z, US.z, TS.y, T.y, PS.y, P.y, S0.y, S1.y, D0.y, D1.y, CV.y, HY.y, MV.y),
                  eq18(V.z, U.z, US.z, U.w, US.w, TS.z, T.z, PS.z, P.z, S0.z, S1.z, D0.z, D1.z, CV.z, HY.z, MV.z),
                  eq18(V.w, U.w, US.w, ue, use, TS.w, T.w, PS.w, P.w, S0.w, S1.w, D0.w, D1.w, CV.w, HY.w, MV.w)));
}

// ---- divergence + divdamp as warp strips (:514-597, :853-895, :627-630) ---
// The work of k_sound_div and k_sound_damp in one pass.  One warp per strip
// of kDDJ output columns x R rows of one level k, lanes on columns
// j0-1 .. j0+30.  For each row the lane's point gets s(k) and s(k+1)
// (Equation 10, or the surface values when k is the lowest level) and the
// horizontal divergence zdiv2a (Equation 16) from the pre-damping u, v of
// the current buffer: east neighbours from the lane beside (shuffles),
// north neighbours from the next row, whose v-part is loaded two rows
// ahead.  The damping of row i then takes zdiv2a of the lanes beside and of
// rows i-1, i+1 from registers.  Damped u, v go to the other buffer
// (ubuf[cur^1]) -- the caller flips cur -- so no strip ever reads a value
// another strip has damped; zdiv2a never goes to memory.  The boundary
// lanes and rows store the pre-damping edge values the momentum step reads
// as the stale ud/vd halo (:730-735), as k_sound_div does.
template <class T>
__device__ __forceinline__ void b_divdamp_strip(const View<T>& d, const int bx, const int k, const int R,
                                                const int wid, const int nw) {
  if (d.sur_skip && *d.sur_skip) return;  // the surrogate took this cycle
  const int lane = threadIdx.x & 31;
  const int nj = d.nj, ni = d.ni, kz = d.kz;
  const size_t pl = d.pl;
  const int nsj = (nj + kDDJ - 1) / kDDJ, nsi = (ni + R - 1) / R;
  const int w = bx * nw + wid;
  if (w >= nsj * nsi) return;  // whole warp
  const int sj = w % nsj, si = w / nsj;
  const int jl = sj * kDDJ - 1 + lane;
  const int jj = wrapn(jl, nj);
  const bool out_lane = lane >= 1 && lane <= kDDJ && jl < nj;
  const int i_s = si * R, i_e = min(i_s + R, ni);
  const size_t o = (size_t)k * pl;
  const bool has_up = k > 0, has_dn = k < kz - 1;  // levels k-1 and k+1 exist
  const T* __restrict__ u = d.ubuf[d.cur] + o;
  const T* __restrict__ v = d.vbuf[d.cur] + o;
  T* __restrict__ uo = d.ubuf[d.cur ^ 1] + o;
  T* __restrict__ vo = d.vbuf[d.cur ^ 1] + o;
  const T* __restrict__ rfw = d.rfw + o;
  const T* __restrict__ rfs = d.rfs + o;
  const T* __restrict__ fmz = d.fmz + o;
  const bool rot = d.rotllr;
  const T dtrdx = d.dtrdx, dtrdy = d.dtrdy, dtrdz = d.dtrdz, ddamp2 = d.ddamp2;
  const T cd = d.cdamp[k];
  const T gzk = has_up ? d.gzitak[k] : T(0), gzk1 = has_dn ? d.gzitak[k + 1] : T(0);
  // u-part and v-part of a row of this lane's column
  struct Ur { T uk, um, up, rfw, fmz, hx, mx, rmu, mu, mv, s0; };
  struct Vr { T vk, vm, vp, rfs, rmv, hy; };
  auto load_u = [&](int i, Ur& x) {
    const size_t c = (size_t)jj + (size_t)nj * wrap2(i, ni);
    x.uk = u[c];
    x.um = has_up ? u[c - pl] : T(0);
    x.up = has_dn ? u[c + pl] : T(0);
    x.rfw = rfw[c]; x.fmz = fmz[c]; x.hx = d.hx[c]; x.mu = d.mu[c];
    x.mx = rot ? d.mx[c] : d.mx2[c];
    x.rmu = rot ? T(0) : d.rmu[c];
    x.mv = rot ? T(0) : d.mv[c];
    x.s0 = has_up ? T(0) : d.s[c];  // s at the top level is never computed here
  };
  auto load_v = [&](int i, Vr& x) {
    const size_t c = (size_t)jj + (size_t)nj * wrap2(i, ni);
    x.vk = v[c];
    x.vm = has_up ? v[c - pl] : T(0);
    x.vp = has_dn ? v[c + pl] : T(0);
    x.rfs = rfs[c]; x.rmv = d.rmv[c]; x.hy = d.hy[c];
  };
  // zdiv2a, s(k), s(k+1) of a row from its u-part and the v-parts of the
  // row and the row after (expressions of k_sound_div)
  struct Zr { T z, sk, sk1, ws; };
  auto row_terms = [&](const Ur& a, const Vr& b, const Vr& bn) {
    const T uk_e = __shfl_down_sync(0xffffffffu, a.uk, 1);
    const T um_e = __shfl_down_sync(0xffffffffu, a.um, 1);
    const T up_e = __shfl_down_sync(0xffffffffu, a.up, 1);
    const T rfw_e = __shfl_down_sync(0xffffffffu, a.rfw, 1);
    const T hx_e = __shfl_down_sync(0xffffffffu, a.hx, 1);
    const T rmu_e = __shfl_down_sync(0xffffffffu, a.rmu, 1);
    Zr r;
    if (has_up) {
      const T zuh = prod_add(a.uk + a.um, a.hx, uk_e + um_e, hx_e);
      const T zvh = prod_add(b.vk + b.vm, b.hy, bn.vk + bn.vm, bn.hy);
      r.sk = -((T(0.25) * (zuh + zvh)) * gzk);
    } else {
      r.sk = a.s0;
    }
    if (has_dn) {
      const T zuh = prod_add(a.up + a.uk, a.hx, up_e + uk_e, hx_e);
      const T zvh = prod_add(b.vp + b.vk, b.hy, bn.vp + bn.vk, bn.hy);
      r.sk1 = -((T(0.25) * (zuh + zvh)) * gzk1);
      r.ws = T(0);
    } else {  // surface w(kz+1) and s(kz+1) (:536-549)
      const T zuh = prod_add(a.uk, a.hx, uk_e, hx_e);
      const T zvh = prod_add(b.vk, b.hy, bn.vk, bn.hy);
      r.ws = T(0.5) * (zuh + zvh);
      r.sk1 = -r.ws;
    }
    if (rot) {
      const T du = prod_sub(dtrdx * uk_e, rfw_e, dtrdx * a.uk, a.rfw);
      const T dv = prod_sub((dtrdy * bn.vk) * bn.rfs, bn.rmv, (dtrdy * b.vk) * b.rfs, b.rmv);
      r.z = (a.fmz * a.mx) * (du + dv);
    } else {
      const T du = prod_sub((dtrdx * uk_e) * rmu_e, rfw_e, (dtrdx * a.uk) * a.rmu, a.rfw);
      const T dv = prod_sub((dtrdy * bn.vk) * bn.rmv, bn.rfs, (dtrdy * b.vk) * b.rmv, b.rfs);
      r.z = (a.mx * a.fmz) * (du + dv);
    }
    return r;
  };
  // prologue: zdiv2a of row i_s-1, all terms of row i_s
  Ur ua, ub, un;
  Vr va, vb, vc, vn;
  load_u(i_s - 1, ua); load_v(i_s - 1, va); load_v(i_s, vb);
  load_u(i_s, ub); load_v(i_s + 1, vc);
  const T z_first = row_terms(ua, va, vb).z;
  T z_prev = z_first;
  Zr zcur = row_terms(ub, vb, vc);
  Ur ucur = ub;
  Vr vcur = vb;
  if (i_s + 1 <= i_e) { load_u(i_s + 1, un); load_v(i_s + 2, vn); }
  for (int i = i_s; i < i_e; ++i) {
    // in registers: z(i-1); row i (ucur, vcur, zcur); v-part of row i+1 (vc);
    // in flight: u-part of row i+1 (un), v-part of row i+2 (vn)
    const Ur unext = un;
    const Vr vnext = vn;
    if (i + 2 <= i_e) { load_u(i + 2, un); load_v(i + 3, vn); }
    const Zr znext = row_terms(unext, vc, vnext);  // row i+1
    const T zc = zcur.z;
    const T zw = __shfl_up_sync(0xffffffffu, zc, 1);
    const T ze = __shfl_down_sync(0xffffffffu, zc, 1);
    const T zs = z_prev, zn = znext.z;
    if (out_lane) {
      const int ii = i;
      const size_t c = (size_t)jj + (size_t)nj * ii;
      const T u0 = ucur.uk, v0 = vcur.vk;
      if (has_up) d.s[o + c] = zcur.sk;
      if (!has_dn) {
        d.w[c + (size_t)kz * pl] = zcur.ws;
        d.s[c + (size_t)kz * pl] = -zcur.ws;
      }
      if (jj == 0) d.eu_j[ii + (size_t)ni * k] = u0;
      if (ii == ni - 1) d.eu_i[jj + (size_t)nj * k] = u0;
      if (jj == nj - 1) d.ev_j[ii + (size_t)ni * k] = v0;
      if (ii == 0) d.ev_i[jj + (size_t)nj * k] = v0;
      uo[c] = u0 + ((cd * ucur.mu) * (zc - zw));
      if (rot)
        vo[c] = v0 + cd * (zc - zs);
      else
        vo[c] = v0 + ((cd * ucur.mv) * (zc - zs));
      const T p2d = prod_sub(T(0.125), ((zw + ze) + zs) + zn, T(0.5), zc);
      T zd = zc + ddamp2 * p2d;
      zd = zd + (ucur.fmz * dtrdz) * (zcur.sk - zcur.sk1);
      d.zdiv2b[o + c] = zd;
    }
    z_prev = zc;
    zcur = znext;
    ucur = unext;
    vcur = vc;
    vc = vnext;
  }
}

// (8 blocks per SM with 64 registers measured slower in the full step:
// 2.74 against 2.56 ms per step)
template <class T>
__global__ void __launch_bounds__(128) k_divdamp_strip(View<T> d, int R) {
  b_divdamp_strip<T>(d, blockIdx.x, blockIdx.y, R, threadIdx.x >> 5, 4);
}

template <class T>
__global__ void __launch_bounds__(128, sizeof(T) == 4 ? 8 : 3)
    kb_divdamp_strip(const View<T>* __restrict__ views, const int4* __restrict__ tiles, int R) {
  __shared__ View<T> sv;
  const int4 t = tiles[blockIdx.x];
  copy_view(&sv, views + t.x);
  __syncthreads();
  b_divdamp_strip<T>(sv, t.y, t.z, R, threadIdx.x >> 5, 4);
}

// The same strips over NL consecutive levels k0 .. k0+NL-1 per warp
// (kmarch bit 512, with 16).  The levels of a strip share each row's loads
// of u and v at the levels between them (NL+2 levels instead of 3 NL), its
// 2-D metric fields, the east shuffles of those values and the address
// arithmetic, and s(k) at each inner level is formed once instead of
// twice (as s(k+1) of the level above and s(k) of the level below: the
// same sums in the same order, so the same bits).  Per level the
// arithmetic is that of b_divdamp_strip.
template <class T, int NL>
__device__ __forceinline__ void b_divdamp_strip_nl(const View<T>& d, const int bx, const int kp, const int R,
                                                   const int wid, const int nw) {
  if (d.sur_skip && *d.sur_skip) return;  // the surrogate took this cycle
  const int lane = threadIdx.x & 31;
  const int nj = d.nj, ni = d.ni, kz = d.kz;
  const unsigned pl = (unsigned)d.pl;  // 32-bit element offsets: a field holds at most 2^31 points
  const int nsj = (nj + kDDJ - 1) / kDDJ, nsi = (ni + R - 1) / R;
  const int w = bx * nw + wid;
  if (w >= nsj * nsi) return;  // whole warp
  const int sj = w % nsj, si = w / nsj;
  const int jl = sj * kDDJ - 1 + lane;
  const int jj = wrapn(jl, nj);
  const bool out_lane = lane >= 1 && lane <= kDDJ && jl < nj;
  const int i_s = si * R, i_e = min(i_s + R, ni);
  const int k0 = kp * NL;
  const T* __restrict__ u = d.ubuf[d.cur];
  const T* __restrict__ v = d.vbuf[d.cur];
  T* __restrict__ uo = d.ubuf[d.cur ^ 1];
  T* __restrict__ vo = d.vbuf[d.cur ^ 1];
  const bool rot = d.rotllr;
  const T dtrdx = d.dtrdx, dtrdy = d.dtrdy, dtrdz = d.dtrdz, ddamp2 = d.ddamp2;
  // level k0-1+l, l = 0 .. NL+1, inside the domain; level k0+l, l < NL
  bool lin[NL + 2];
#pragma unroll
  for (int l = 0; l < NL + 2; ++l) lin[l] = k0 - 1 + l >= 0 && k0 - 1 + l < kz;
  T cd[NL], gz[NL + 1];
#pragma unroll
  for (int l = 0; l < NL; ++l) cd[l] = lin[l + 1] ? d.cdamp[k0 + l] : T(0);
#pragma unroll
  for (int l = 0; l <= NL; ++l) gz[l] = (k0 + l >= 1 && k0 + l <= kz - 1) ? d.gzitak[k0 + l] : T(0);
  // u-part and v-part of a row of this lane's column: u, v at the levels
  // k0-1 .. k0+NL, rfw, fmz, rfs at k0 .. k0+NL-1
  struct Ur { T u[NL + 2], rfw[NL], fmz[NL]; T hx, mx, rmu, mu, mv, s0; };
  struct Vr { T v[NL + 2], rfs[NL]; T rmv, hy; };
  auto load_u = [&](int i, Ur& x) {
    const unsigned c = (unsigned)jj + (unsigned)nj * (unsigned)wrap2(i, ni);
#pragma unroll
    for (int l = 0; l < NL + 2; ++l) x.u[l] = lin[l] ? u[c + (unsigned)(k0 - 1 + l) * pl] : T(0);
#pragma unroll
    for (int l = 0; l < NL; ++l) {
      x.rfw[l] = lin[l + 1] ? d.rfw[c + (unsigned)(k0 + l) * pl] : T(0);
      x.fmz[l] = lin[l + 1] ? d.fmz[c + (unsigned)(k0 + l) * pl] : T(0);
    }
    x.hx = d.hx[c]; x.mu = d.mu[c];
    x.mx = rot ? d.mx[c] : d.mx2[c];
    x.rmu = rot ? T(0) : d.rmu[c];
    x.mv = rot ? T(0) : d.mv[c];
    x.s0 = k0 == 0 ? d.s[c] : T(0);  // s at the top level is never computed here
  };
  auto load_v = [&](int i, Vr& x) {
    const unsigned c = (unsigned)jj + (unsigned)nj * (unsigned)wrap2(i, ni);
#pragma unroll
    for (int l = 0; l < NL + 2; ++l) x.v[l] = lin[l] ? v[c + (unsigned)(k0 - 1 + l) * pl] : T(0);
#pragma unroll
    for (int l = 0; l < NL; ++l) x.rfs[l] = lin[l + 1] ? d.rfs[c + (unsigned)(k0 + l) * pl] : T(0);
    x.rmv = d.rmv[c]; x.hy = d.hy[c];
  };
  // zdiv2a of the levels, s at k0 .. k0+NL (the surface value -ws at kz),
  // ws when the lowest level is kz-1 (expressions of k_sound_div)
  struct Zr { T z[NL], s[NL + 1], ws; };
  auto row_terms = [&](const Ur& a, const Vr& b, const Vr& bn) {
    T ue[NL + 2];
#pragma unroll
    for (int l = 0; l < NL + 2; ++l) ue[l] = __shfl_down_sync(0xffffffffu, a.u[l], 1);
    T rfw_e[NL];
#pragma unroll
    for (int l = 0; l < NL; ++l) rfw_e[l] = __shfl_down_sync(0xffffffffu, a.rfw[l], 1);
    const T hx_e = __shfl_down_sync(0xffffffffu, a.hx, 1);
    const T rmu_e = __shfl_down_sync(0xffffffffu, a.rmu, 1);
    Zr r;
    r.ws = T(0);
#pragma unroll
    for (int l = 0; l <= NL; ++l) {
      const int kk = k0 + l;  // s(kk) from the levels kk-1 (index l) and kk (index l+1)
      if (kk == 0) {
        r.s[l] = a.s0;
      } else if (kk <= kz - 1) {
        const T zuh = prod_add(a.u[l + 1] + a.u[l], a.hx, ue[l + 1] + ue[l], hx_e);
        const T zvh = prod_add(b.v[l + 1] + b.v[l], b.hy, bn.v[l + 1] + bn.v[l], bn.hy);
        r.s[l] = -((T(0.25) * (zuh + zvh)) * gz[l]);
      } else if (kk == kz) {  // surface w(kz+1) and s(kz+1) (:536-549)
        const T zuh = prod_add(a.u[l], a.hx, ue[l], hx_e);
        const T zvh = prod_add(b.v[l], b.hy, bn.v[l], bn.hy);
        r.ws = T(0.5) * (zuh + zvh);
        r.s[l] = -r.ws;
      } else {
        r.s[l] = T(0);
      }
    }
#pragma unroll
    for (int l = 0; l < NL; ++l) {
      const T uk = a.u[l + 1], uk_e = ue[l + 1];
      if (rot) {
        const T du = prod_sub(dtrdx * uk_e, rfw_e[l], dtrdx * uk, a.rfw[l]);
        const T dv = prod_sub((dtrdy * bn.v[l + 1]) * bn.rfs[l], bn.rmv, (dtrdy * b.v[l + 1]) * b.rfs[l], b.rmv);
        r.z[l] = (a.fmz[l] * a.mx) * (du + dv);
      } else {
        const T du = prod_sub((dtrdx * uk_e) * rmu_e, rfw_e[l], (dtrdx * uk) * a.rmu, a.rfw[l]);
        const T dv = prod_sub((dtrdy * bn.v[l + 1]) * bn.rmv, bn.rfs[l], (dtrdy * b.v[l + 1]) * b.rmv, b.rfs[l]);
        r.z[l] = (a.mx * a.fmz[l]) * (du + dv);
      }
    }
    return r;
  };
  // prologue: zdiv2a of row i_s-1, all terms of row i_s
  Ur ua, ub, un;
  Vr va, vb, vc, vn;
  load_u(i_s - 1, ua); load_v(i_s - 1, va); load_v(i_s, vb);
  load_u(i_s, ub); load_v(i_s + 1, vc);
  const Zr zfirst = row_terms(ua, va, vb);
  T z_prev[NL];
#pragma unroll
  for (int l = 0; l < NL; ++l) z_prev[l] = zfirst.z[l];
  Zr zcur = row_terms(ub, vb, vc);
  Ur ucur = ub;
  Vr vcur = vb;
  if (i_s + 1 <= i_e) { load_u(i_s + 1, un); load_v(i_s + 2, vn); }
  for (int i = i_s; i < i_e; ++i) {
    // in registers: z(i-1); row i (ucur, vcur, zcur); v-part of row i+1 (vc);
    // in flight: u-part of row i+1 (un), v-part of row i+2 (vn)
    const Ur unext = un;
    const Vr vnext = vn;
    if (i + 2 <= i_e) { load_u(i + 2, un); load_v(i + 3, vn); }
    const Zr znext = row_terms(unext, vc, vnext);  // row i+1
    const unsigned c = (unsigned)jj + (unsigned)nj * (unsigned)i;
#pragma unroll
    for (int l = 0; l < NL; ++l) {
      const int k = k0 + l;
      const T zc = zcur.z[l];
      const T zw = __shfl_up_sync(0xffffffffu, zc, 1);
      const T ze = __shfl_down_sync(0xffffffffu, zc, 1);
      const T zs = z_prev[l], zn = znext.z[l];
      if (out_lane && k < kz) {
        const unsigned o = (unsigned)k * pl;
        const T u0 = ucur.u[l + 1], v0 = vcur.v[l + 1];
        if (k > 0) d.s[o + c] = zcur.s[l];
        if (k == kz - 1) {
          d.w[c + (unsigned)kz * pl] = zcur.ws;
          d.s[c + (unsigned)kz * pl] = -zcur.ws;
        }
        if (jj == 0) d.eu_j[i + (size_t)ni * k] = u0;
        if (i == ni - 1) d.eu_i[jj + (size_t)nj * k] = u0;
        if (jj == nj - 1) d.ev_j[i + (size_t)ni * k] = v0;
        if (i == 0) d.ev_i[jj + (size_t)nj * k] = v0;
        uo[o + c] = u0 + ((cd[l] * ucur.mu) * (zc - zw));
        if (rot)
          vo[o + c] = v0 + cd[l] * (zc - zs);
        else
          vo[o + c] = v0 + ((cd[l] * ucur.mv) * (zc - zs));
        const T p2d = prod_sub(T(0.125), ((zw + ze) + zs) + zn, T(0.5), zc);
        T zd = zc + ddamp2 * p2d;
        zd = zd + (ucur.fmz[l] * dtrdz) * (zcur.s[l] - zcur.s[l + 1]);
        d.zdiv2b[o + c] = zd;
      }
      z_prev[l] = zc;
    }
    zcur = znext;
    ucur = unext;
    vcur = vc;
    vc = vnext;
  }
}

// 4 blocks per SM (FP32: 122 registers): 0.167 ms per launch at
// 512 x 512 x 60 against 0.171 for the one-level strips; 5 blocks (96
// registers, spills) 0.180
template <class T>
__global__ void __launch_bounds__(128, 4) k_divdamp_strip_nl(View<T> d, int R) {
  b_divdamp_strip_nl<T, kDDLevels>(d, blockIdx.x, blockIdx.y, R, threadIdx.x >> 5, 4);
}
template <class T>
__global__ void __launch_bounds__(128, 4)
    kb_divdamp_strip_nl(const View<T>* __restrict__ views, const int4* __restrict__ tiles, int R) {
  __shared__ View<T> sv;
  const int4 t = tiles[blockIdx.x];
  copy_view(&sv, views + t.x);
  __syncthreads();
  b_divdamp_strip_nl<T, kDDLevels>(sv, t.y, t.z, R, threadIdx.x >> 5, 4);
}

// ---- divergence + divdamp with four columns per thread (FP32) ------------
// A CTA an SM marches down the levels of tiles of 128 columns x kDQRows rows.
// A warp per row (and one for the row on either side) holds a quad of columns
// per lane, with u and v of the level and of the one below it in registers;
// each level reads u, v, the v of the row after, rfw, rfs and fmz once, copied
// kDQSlots - 1 levels ahead into a ring in shared memory (cp.async, each lane
// its own quads); s(k+1) is carried to the next level and the 2-D metric
// fields stay in registers.  The horizontal divergence of the rows goes
// through shared memory (two buffers, one barrier a level); one more warp
// forms it on the two columns beside the tile.  The tiles' levels, taken one
// after another, are cut into one equal share a CTA, so no last wave is left.
// Per level the arithmetic is that of b_divdamp_strip.  s is stored in the
// last substep only (LAST): no other reads it outside this kernel.
// The strips spend about 270 warp instructions on 32 points and issue in 60 %
// of their cycles; this about 110.  Per step at 512 x 512 x 60: 2.32 (strips
// over two levels) -> 1.73 ms; 10 rows 1.99, two CTAs of 5 rows 2.23; with the
// loads in registers instead of the ring 2.15; 1024 x 1024 x 60 9.13 -> 7.35,
// 256 x 256 x 40 0.59 -> 0.40.
constexpr int kDQRows = 13;
constexpr int kDQThreads = 32 * (kDQRows + 3);
constexpr int kDQSlots = 3;
struct DQSlot {
  float4 f[7][32];
  float e[2][32];  // rfw and u(k+1) of the column after the row's last
};
constexpr int kDQRing = (kDQRows + 2) * kDQSlots * (int)sizeof(DQSlot);
constexpr int kDQMaxKz = 512;  // levels whose gzitak and cdamp fit beside the ring
inline int dq_smem_bytes(int kz) { return kDQRing + 8 * kz; }
__device__ __forceinline__ void cp_async_16(void* dst_smem, const void* src) {
  const uint32_t dst = static_cast<uint32_t>(__cvta_generic_to_shared(dst_smem));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
template <bool ROT, int LAST>
__global__ void __launch_bounds__(kDQThreads, 1) k_divdamp_quad(const __grid_constant__ View<float> d) {
  if (d.sur_skip && *d.sur_skip) return;  // the surrogate took this cycle
  extern __shared__ __align__(16) unsigned char dq_smem[];
  // z of rows i0-1 .. i0+kDQRows, columns jb-4 .. jb+131 (of the outer quads only jb-1 and jb+128 are set)
  __shared__ __align__(16) float zs[2][kDQRows + 2][136];
  const int nj = d.nj, ni = d.ni, kz = d.kz;
  const unsigned pl = (unsigned)d.pl;
  const int lane = threadIdx.x, wr = threadIdx.y;
  const int ntj = (nj + 127) / 128;
  // gzitak(k+1), cdamp(k) behind the ring
  float* const s_gz = reinterpret_cast<float*>(dq_smem + kDQRing);
  float* const s_cd = s_gz + kz;
  for (int k = lane + 32 * wr; k < kz; k += kDQThreads) { s_gz[k] = d.gzitak[k + 1]; s_cd[k] = d.cdamp[k]; }
  const float* __restrict__ u = d.ubuf[d.cur];
  const float* __restrict__ v = d.vbuf[d.cur];
  const float dtrdx = d.dtrdx, dtrdy = d.dtrdy, dtrdz = d.dtrdz, ddamp2 = d.ddamp2;
  auto zdiv = [&](float ue, float u0, float vn, float v0, float rfwe, float rfw, float rfsn, float rfs, float rmue,
                  float rmu, float rmvn, float rmv, float fmz, float mx) {
    if (ROT) {
      const float du = prod_sub(dtrdx * ue, rfwe, dtrdx * u0, rfw);
      const float dv = prod_sub((dtrdy * vn) * rfsn, rmvn, (dtrdy * v0) * rfs, rmv);
      return (fmz * mx) * (du + dv);
    }
    const float du = prod_sub((dtrdx * ue) * rmue, rfwe, (dtrdx * u0) * rmu, rfw);
    const float dv = prod_sub((dtrdy * vn) * rmvn, rfsn, (dtrdy * v0) * rmv, rfs);
    return (mx * fmz) * (du + dv);
  };
  const long long total = (long long)ntj * ((ni + kDQRows - 1) / kDQRows) * kz;
  const long long last_step = total * (blockIdx.x + 1) / gridDim.x;
  for (long long at0 = total * blockIdx.x / gridDim.x; at0 < last_step;) {
    const int tile = (int)(at0 / kz), k0 = (int)(at0 % kz), k1 = (int)min((long long)kz, k0 + (last_step - at0));
    at0 += k1 - k0;
    const int jb = tile % ntj * 128, i0 = tile / ntj * kDQRows;
    const int rows = min(kDQRows, ni - i0);  // output rows
    __syncthreads();  // every warp is done with the last tile's z
    if (wr == kDQRows + 2) {
      // the columns beside the block: lane 2 r + side
      const int r = lane >> 1, side = lane & 1;
      const bool on = r <= rows + 1;
      const int jr = min(jb + 128, nj);
      const int j = on ? (side ? (jr == nj ? 0 : jr) : (jb == 0 ? nj - 1 : jb - 1)) : 0;
      const int i = on ? wrap2(i0 - 1 + r, ni) : 0;
      const unsigned c = (unsigned)j + (unsigned)nj * i, ce = (unsigned)wp1(j, nj) + (unsigned)nj * i;
      const unsigned cn = (unsigned)j + (unsigned)nj * wp1(i, ni);
      const float mx = ROT ? d.mx[c] : d.mx2[c], rmv = d.rmv[c], rmvn = d.rmv[cn];
      const float rmu = ROT ? 0.f : d.rmu[c], rmue = ROT ? 0.f : d.rmu[ce];
      const int at = side ? 4 + jr - jb : 3;
      struct E { float ue, u0, vn, v0, rfwe, rfw, rfsn, rfs, f; };
      auto load = [&](int k, E& e) {  // the next level's, while this one's wait at the barrier
        const unsigned o = (unsigned)k * pl;
        e.ue = u[o + ce]; e.u0 = u[o + c]; e.vn = v[o + cn]; e.v0 = v[o + c];
        e.rfwe = d.rfw[o + ce]; e.rfw = d.rfw[o + c]; e.rfsn = d.rfs[o + cn]; e.rfs = d.rfs[o + c]; e.f = d.fmz[o + c];
      };
      E e1, e2;
      load(k0, e1);
      if (k0 + 1 < k1) load(k0 + 1, e2);
      for (int k = k0; k < k1; ++k) {
        const E e = e1;
        e1 = e2;
        if (k + 2 < k1) load(k + 2, e2);
        if (on) zs[k & 1][r][at] = zdiv(e.ue, e.u0, e.vn, e.v0, e.rfwe, e.rfw, e.rfsn, e.rfs, rmue, rmu, rmvn, rmv, e.f, mx);
        __syncthreads();
      }
      continue;
    }
    // a row of quads; rows past the block's and lanes past the domain's edge only keep the barriers
    const bool on = wr <= rows + 1, out = wr >= 1 && wr <= rows;
    const int ii = on ? wrap2(i0 - 1 + wr, ni) : 0;
    const int jq = jb + 4 * lane;
    const bool in = jq < nj;
    const int j0 = in ? jq : 0;
    const bool endl = lane == 31 || jq + 4 >= nj;  // its east neighbours come from memory
    const unsigned c = (unsigned)j0 + (unsigned)nj * ii, cn = (unsigned)j0 + (unsigned)nj * wp1(ii, ni);
    const unsigned ce = (unsigned)(jq + 4 >= nj ? 0 : j0 + 4) + (unsigned)nj * ii;
    const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 HX = ld4(d.hx + c), HY = ld4(d.hy + c), HYN = ld4(d.hy + cn);
    const float4 MX = ROT ? ld4(d.mx + c) : ld4(d.mx2 + c), RMV = ld4(d.rmv + c), RMVN = ld4(d.rmv + cn);
    const float4 MU = ld4(d.mu + c), RMU = ROT ? z4 : ld4(d.rmu + c), MV = ROT ? z4 : ld4(d.mv + c);
    // the east neighbour of a lane's last column: the lane beside, or own (a
    // load issued together with the quads) at the end of the row
    auto east = [&](float x, float own) {
      const float y = __shfl_down_sync(0xffffffffu, x, 1);
      return endl ? own : y;
    };
    auto own = [&](const float* p, unsigned at) { return endl ? p[at] : 0.f; };
    const float hxe = east(HX.x, own(d.hx, ce)), rmue = ROT ? 0.f : east(RMU.x, own(d.rmu, ce));
    // slope sums of a level pair or of one level: -> s(k) and the surface w
    auto sval = [&](float a, float ae, float b, float bn, float hx, float hxe_, float hy, float hyn, float gz) {
      const float zuh = prod_add(a, hx, ae, hxe_);
      const float zvh = prod_add(b, hy, bn, hyn);
      return -((0.25f * (zuh + zvh)) * gz);
    };
    auto wval = [&](float a, float ae, float b, float bn, float hx, float hxe_, float hy, float hyn) {
      const float zuh = prod_add(a, hx, ae, hxe_);
      const float zvh = prod_add(b, hy, bn, hyn);
      return 0.5f * (zuh + zvh);
    };
    auto spair = [&](const float4& ua, float uae, const float4& ub, float ube, const float4& va, const float4& vna,
                     const float4& vb, const float4& vnb, float gz) {  // levels a (lower) and b (upper)
      return make_float4(
          sval(ua.x + ub.x, ua.y + ub.y, va.x + vb.x, vna.x + vnb.x, HX.x, HX.y, HY.x, HYN.x, gz),
          sval(ua.y + ub.y, ua.z + ub.z, va.y + vb.y, vna.y + vnb.y, HX.y, HX.z, HY.y, HYN.y, gz),
          sval(ua.z + ub.z, ua.w + ub.w, va.z + vb.z, vna.z + vnb.z, HX.z, HX.w, HY.z, HYN.z, gz),
          sval(ua.w + ub.w, uae + ube, va.w + vb.w, vna.w + vnb.w, HX.w, hxe, HY.w, HYN.w, gz));
    };
    unsigned o = (unsigned)k0 * pl;
    float4 U = ld4(u + o + c), V = ld4(v + o + c), VN = ld4(v + o + cn);
    float ue = own(u, o + ce);
    ue = east(U.x, ue);
    float4 S = z4;  // s(k)
    if (k0 == 0) {
      S = ld4(d.s + c);  // s at the top level is never computed here
    } else {
      const float4 um = ld4(u + o - pl + c), vm = ld4(v + o - pl + c), vnm = ld4(v + o - pl + cn);
      const float ume = east(um.x, own(u, o - pl + ce));
      S = spair(U, ue, um, ume, V, VN, vm, vnm, d.gzitak[k0]);
    }
    // ring of kDQSlots levels in shared memory, each lane copying and reading
    // its own quads: rfw, rfs, rfs(i+1), fmz at k and u, v, v(i+1) at k+1
    DQSlot* const ring = reinterpret_cast<DQSlot*>(dq_smem) + wr * kDQSlots;
    auto issue = [&](int k) {
      if (k < k1) {
        DQSlot& q = ring[(k - k0) % kDQSlots];
        const unsigned ok = (unsigned)k * pl;
        cp_async_16(&q.f[0][lane], d.rfw + ok + c); cp_async_16(&q.f[1][lane], d.rfs + ok + c);
        cp_async_16(&q.f[2][lane], d.rfs + ok + cn); cp_async_16(&q.f[3][lane], d.fmz + ok + c);
        if (endl) cp_async_elem(&q.e[0][lane], d.rfw + ok + ce);
        if (k < kz - 1) {
          cp_async_16(&q.f[4][lane], u + ok + pl + c); cp_async_16(&q.f[5][lane], v + ok + pl + c);
          cp_async_16(&q.f[6][lane], v + ok + pl + cn);
          if (endl) cp_async_elem(&q.e[1][lane], u + ok + pl + ce);
        }
      }
      cp_async_commit();
    };
  #pragma unroll
    for (int q = 0; q < kDQSlots - 1; ++q) issue(k0 + q);
    for (int k = k0; k < k1; ++k, o += pl) {
      issue(k + kDQSlots - 1);  // into the slot of level k-1
      cp_async_wait<kDQSlots - 1>();
      const DQSlot& sl = ring[(k - k0) % kDQSlots];
      const float4 RFW = sl.f[0][lane], RFS = sl.f[1][lane], RFSN = sl.f[2][lane], F = sl.f[3][lane];
      float4 U1 = z4, V1 = z4, VN1 = z4;
      if (k < kz - 1) { U1 = sl.f[4][lane]; V1 = sl.f[5][lane]; VN1 = sl.f[6][lane]; }
      const float rfwe = east(RFW.x, sl.e[0][lane]), u1e = east(U1.x, sl.e[1][lane]);
      float4 Z;
      Z.x = zdiv(U.y, U.x, VN.x, V.x, RFW.y, RFW.x, RFSN.x, RFS.x, RMU.y, RMU.x, RMVN.x, RMV.x, F.x, MX.x);
      Z.y = zdiv(U.z, U.y, VN.y, V.y, RFW.z, RFW.y, RFSN.y, RFS.y, RMU.z, RMU.y, RMVN.y, RMV.y, F.y, MX.y);
      Z.z = zdiv(U.w, U.z, VN.z, V.z, RFW.w, RFW.z, RFSN.z, RFS.z, RMU.w, RMU.z, RMVN.z, RMV.z, F.z, MX.z);
      Z.w = zdiv(ue, U.w, VN.w, V.w, rfwe, RFW.w, RFSN.w, RFS.w, rmue, RMU.w, RMVN.w, RMV.w, F.w, MX.w);
      float(*const zb)[136] = zs[k & 1];
      if (on && in) *reinterpret_cast<float4*>(&zb[wr][4 + 4 * lane]) = Z;
      float4 S1;  // s(k+1), or -w at the surface
      if (k < kz - 1)
        S1 = spair(U1, u1e, U, ue, V1, VN1, V, VN, s_gz[k]);
      else
        S1 = make_float4(wval(U.x, U.y, V.x, VN.x, HX.x, HX.y, HY.x, HYN.x), wval(U.y, U.z, V.y, VN.y, HX.y, HX.z, HY.y, HYN.y),
                         wval(U.z, U.w, V.z, VN.z, HX.z, HX.w, HY.z, HYN.z), wval(U.w, ue, V.w, VN.w, HX.w, hxe, HY.w, HYN.w));
      __syncthreads();
      if (out && in) {
        if (k == kz - 1) {
          st4(d.w + (unsigned)kz * pl + c, S1);
          S1 = make_float4(-S1.x, -S1.y, -S1.z, -S1.w);
        }
        const float4 ZS = ld4(&zb[wr - 1][4 + 4 * lane]), ZN = ld4(&zb[wr + 1][4 + 4 * lane]);
        const float zw = zb[wr][3 + 4 * lane], ze = zb[wr][8 + 4 * lane];
        const float cd = s_cd[k];
        if (LAST && k > 0) st4(d.s + o + c, S);
        if (j0 == 0) d.eu_j[ii + (unsigned)ni * k] = U.x;
        if (j0 + 4 == nj) d.ev_j[ii + (unsigned)ni * k] = V.w;
        if (ii == ni - 1) st4(d.eu_i + (unsigned)nj * k + j0, U);
        if (ii == 0) st4(d.ev_i + (unsigned)nj * k + j0, V);
        auto un = [&](float u0, float mu, float zc, float w) { return u0 + ((cd * mu) * (zc - w)); };
        auto vn = [&](float v0, float mv, float zc, float z0) { return ROT ? v0 + cd * (zc - z0) : v0 + ((cd * mv) * (zc - z0)); };
        auto zn = [&](float zc, float w, float e, float z0, float z1, float fz, float s0, float s1) {
          const float p2d = prod_sub(0.125f, ((w + e) + z0) + z1, 0.5f, zc);
          float zd = zc + ddamp2 * p2d;
          return zd + (fz * dtrdz) * (s0 - s1);
        };
        st4(d.ubuf[d.cur ^ 1] + o + c, make_float4(un(U.x, MU.x, Z.x, zw), un(U.y, MU.y, Z.y, Z.x), un(U.z, MU.z, Z.z, Z.y),
                                                   un(U.w, MU.w, Z.w, Z.z)));
        st4(d.vbuf[d.cur ^ 1] + o + c, make_float4(vn(V.x, MV.x, Z.x, ZS.x), vn(V.y, MV.y, Z.y, ZS.y),
                                                   vn(V.z, MV.z, Z.z, ZS.z), vn(V.w, MV.w, Z.w, ZS.w)));
        st4(d.zdiv2b + o + c, make_float4(zn(Z.x, zw, Z.y, ZS.x, ZN.x, F.x, S.x, S1.x), zn(Z.y, Z.x, Z.z, ZS.y, ZN.y, F.y, S.y, S1.y),
                                          zn(Z.z, Z.y, Z.w, ZS.z, ZN.z, F.z, S.z, S1.z), zn(Z.w, Z.z, ze, ZS.w, ZN.w, F.w, S.w, S1.w)));
      }
      U = U1; V = V1; VN = VN1; ue = u1e; S = S1;
    }
    cp_async_wait<0>();  // no copy outlives the tile
  }
}

// once a device: the attribute is a device's own
inline void dq_attributes() {
  static std::atomic<bool> done[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64 || done[dev].load(std::memory_order_acquire)) return;
  const int bytes = dq_smem_bytes(kDQMaxKz);
  cudaFuncSetAttribute(k_divdamp_quad<true, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  cudaFuncSetAttribute(k_divdamp_quad<true, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  cudaFuncSetAttribute(k_divdamp_quad<false, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  cudaFuncSetAttribute(k_divdamp_quad<false, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  done[dev].store(true, std::memory_order_release);
}

// ---- FP64 WAF value with the reference's rounding in fewer FP64 operations ----
// (the exact build and the one-field advection): quotients that round as IEEE
// (quot_rn), sign, order, halving and doubling by the bits.
// Bound by the FP64 pipe (16 clocks a warp instruction).  Exact build, 53 x 47 x
// 21, ms per step: vertical 0.464 -> 0.346, horizontal 0.479 -> 0.356, the same
// bits.
// x / 2 by the exponent
__device__ __forceinline__ double half_of(double x) {
  const unsigned e = ((unsigned)__double2hiint(x) >> 20) & 0x7ffu;
  if (e - 2u < 0x7ffu - 2u) return __hiloint2double(__double2hiint(x) - 0x100000, __double2loint(x));
  return 0.5 * x;
}

// superbee limiter max(0, min(2, max(r, min(2r, 1)))) (:994) by the bits of r:
// 0 below 0, 2r up to 1/2, 1 up to 1, r up to 2, then 2; 1 for NaN, as the
// comparisons of the expression fall
__device__ __forceinline__ double superbee_bits(double r) {
  const long long x = __double_as_longlong(r);
  const long long half = 0x3fe0000000000000LL, one = 0x3ff0000000000000LL, two = 0x4000000000000000LL;
  long long b = x < one ? one : x;
  if (x < half) b = x >= 0x0010000000000000LL ? x + 0x0010000000000000LL : x << 1;  // subnormal: twice by a shift
  if (x >= two) b = two;
  if (x < 0) b = 0;
  if ((x & 0x7fffffffffffffffLL) > 0x7ff0000000000000LL) b = one;
  return __longlong_as_double(b);
}
// sign(max(abs(z), minden), z) (:992) by the bits of z (NaN becomes minden)
__device__ __forceinline__ double safeden_bits(double z) {
  const unsigned long long lo = (unsigned long long)__double_as_longlong(kMinden), inf = 0x7ff0000000000000ULL;
  const unsigned long long x = (unsigned long long)__double_as_longlong(z);
  unsigned long long m = x & 0x7fffffffffffffffULL;
  if (m - lo > inf - lo) m = lo;
  return __longlong_as_double((long long)(m | (x & 0x8000000000000000ULL)));
}

// (1 + zphi) m1 + (1 - zphi) x0 of the flux between cells m1 and x0; up: the
// wind comes from m1's side, num the difference that side of it
__device__ __forceinline__ double waf_flux_rn(bool up, double zamu, double num, double den, double m1, double x0) {
  const double is = up ? 1.0 : -1.0;
  const double b = superbee_bits(quot_rn(num, rcp_rn_of(safeden_bits(den))));
  const double zphi = (is + zamu * b) - (up ? b : -b);
  return (1.0 + zphi) * m1 + (1.0 - zphi) * x0;
}
// ---- advection: vertical WAF, two passes at dt/2 (:966-1073) ------------
// wfw(k+1) of one pass from x(max(k-1,1)), x(k), x(k+1), x(min(k+2,kz))
template <class T>
__device__ __forceinline__ T waf_vflux(T s_k1, T dtrdz, T xm, T x0, T x1, T x2) {
  const T zamu = s_k1 * dtrdz;
  const long long z = __double_as_longlong(zamu);
  const bool pos = z >= 0 || z == (long long)0x8000000000000000ULL;  // zamu >= 0
  const T num = (pos ? x1 : xm) - (pos ? x2 : x0);  // k1 = k+1 or max(k-1, 1), k1p1 = min(k+2, kz) or k
  return half_of(s_k1) * waf_flux_rn(pos, zamu, num, x0 - x1, x1, x0);
}
// FP32 storage: the same flux, rearranged for fewer instructions (these
// kernels are bound by the ALU pipe, not HBM): superbee as
// max(sat(2r), min(r, 2)), phi = is + bb (zamu - is), and
// (1+phi) x1 + (1-phi) x0 = (x1 + x0) - phi (x0 - x1)
template <>
__device__ __forceinline__ float waf_vflux<float>(float s_k1, float dtrdz, float xm, float x0, float x1, float x2) {
  const float zamu = s_k1 * dtrdz;
  const bool pos = zamu >= 0.f;
  const float d = x0 - x1;
  const float den = copysignf(fmaxf(fabsf(d), (float)kMinden), d);
  const float r = qdiv(pos ? x1 - x2 : xm - x0, den);
  const float bb = fmaxf(__saturatef(2.f * r), fminf(r, 2.f));
  const float is = pos ? 1.f : -1.f;
  const float zphi = fmaf(bb, zamu - is, is);
  return (0.5f * s_k1) * fmaf(-zphi, d, x1 + x0);
}

// The contracting builds (MOLOCH_LEAN_FP64) evaluate the FP64 WAF value in
// flux form, without the slope ratio.  With d the difference across the face
// and num the upwind one, phi d = is d + (zamu - is) L where
//   L = superbee(num / d) d = sign(d) max(0, min(2 min(a, b), max(a, b))),
//   a = sign(d) num, b = |d|
// (the superbee limiter, P. K. Sweby, SIAM J. Numer. Anal. 21, 1984, times the
// denominator of its argument), so half the WAF value is
// x_upwind - 0.5 (zamu - is) L: no division, no guard against a small
// denominator (for |d| < kMinden the two forms differ by less than
// 4 kMinden), and with the velocity-only factors shared by a thread's fields
// two FP64 operations a face instead of about 25.  GB300 has two FP64 lanes
// an SM, and these kernels were bound by them (81-84 % busy, two thirds of
// the FP64 step); minimum, maximum, doubling and sign run on the integer
// pipe.  Where d is not finite the value is NaN, as in the quotient form.
// Per step at 256 x 256 x 60: vertical 14.9 -> 4.2 ms, horizontal 18.0 -> 4.9
// (tiles) or 4.2 ms (strips).  FP32 keeps the quotient form: its kernels wait
// on memory (1.69 -> 1.63 and 1.76 -> 1.70 ms per step at 512 x 512 x 60 with
// the flux form), and w, a small difference of large terms, moves by 1e-3 of
// itself with any change of an FP32 rounding.
__device__ __forceinline__ double limited(double num, double d) {
  typedef unsigned long long u64;
  const u64 top = 0x8000000000000000ull;
  const u64 db = (u64)__double_as_longlong(d), sg = db & top;
  const u64 b = db ^ sg, a = (u64)__double_as_longlong(num) ^ sg;
  const bool lt = a < b;  // non-negative doubles order as their bits; a < 0 is caught below
  const u64 mn = lt ? a : b, mx = lt ? b : a;
  const u64 two = mn >= (1ull << 52) ? mn + (1ull << 52) : mn;  // 2 mn (subnormals stay: below 2^-1022)
  u64 l = two < mx ? two : mx;
  if (a & top) l = 0ull;
  if (b >= 0x7ff0000000000000ull) l = 0x7ff8000000000000ull;  // NaN where d is not finite
  return __longlong_as_double((long long)(l ^ sg));
}
// Velocity-only terms of a face: whether the positive direction is upwind
// and 0.5 (zamu - is), zamu = vel dt
template <class T>
struct Face {
  bool pos;
  T hz;
};
template <class T>
__device__ __forceinline__ Face<T> face_of(bool pos, T vel, T dt) {
  return {pos, fma_rn(vel, mul_rn(T(0.5), dt), pos ? T(-0.5) : T(0.5))};
}
// half the WAF value at a face: d the difference across it (ahead minus
// behind, or either order as long as npos and nneg, the differences across
// the neighbouring faces behind and ahead, are in the same), xpos and xneg
// the values behind and ahead
template <class T>
__device__ __forceinline__ T waf_half(const Face<T>& f, T d, T npos, T nneg, T xpos, T xneg) {
  return fma_rn(-f.hz, limited(f.pos ? npos : nneg, d), f.pos ? xpos : xneg);
}
// new value of a cell: x + cb vb - ca va + (ca - cb) old, with vb, va half
// the WAF values of the faces behind and ahead and cb, ca their velocities
// times the metric terms
template <class T>
__device__ __forceinline__ T waf_update(T x, T cb, T vb, T ca, T va, T cdv, T old) {
  return fma_rn(cdv, old, fma_rn(-ca, va, fma_rn(cb, vb, x)));
}

// One thread per column and F fields (F = 1, 2, 5 or 10: the tuned
// View::vfields).  Both passes stream k in registers: pass 1 yields wz1(t)
// at step t, pass 2 consumes it two levels later, so the intermediate field
// never leaves the SM.  The fields of a thread share the loads of s, wafu,
// wafd and the velocity-only terms of the fluxes (Courant number, its sign,
// s/2, the metric term of the update), which the compiler computes once.
// The grid puts the field group fastest, so the groups of one column tile
// run together and share the s / metric loads through L2.
// G >= 0: the thread's field group holds some of fields 2, 3, 4 (ux, vx,
// wx), which are formed here from the staggered winds -- the fourth-order
// averages of :1327-1341 and :1389-1417, two-point at the bottom and top
// levels of wx -- and stored for the horizontal pass, which reads them.
// Each level is formed once, in order, with its store; the clamped repeats
// at the bottom reuse the last level.  G = -1: a group of read fields only.
template <class T, int F, int G>
__device__ __forceinline__ void b_waf_vertical_g(const View<T>& d, const int g, const int jj, const int ii) {
  const int nj = d.nj, ni = d.ni, kz = d.kz;
  // element offsets fit in 32 bits (a field holds at most 2^31 points)
  const unsigned pl = (unsigned)d.pl;
  const unsigned c = (unsigned)jj + (unsigned)nj * (unsigned)ii;
  const T* src[F];
  T* wz[F];
#pragma unroll
  for (int u = 0; u < F; ++u) {
    src[u] = d.fset[d.fcur][g * F + u];
    wz[u] = d.wz + (size_t)(g * F + u) * d.pl * kz;
  }
  const T* __restrict__ s = d.s;
  const T* __restrict__ wafu = d.wafu;
  const T* __restrict__ wafd = d.wafd;
  const T dtrdz = d.dtrdz_a;
  auto xval = [&](const int u, const int kk) -> T {
    const unsigned o = (unsigned)kk * pl;
    if constexpr (G < 0) {
      return src[u][c + o];
    } else {
      const int f = G * F + u;
      T x;
      if (f == 2) {
        const T* __restrict__ us = d.ubuf[d.cur] + (o + (unsigned)nj * ii);
        x = average4(us[wp1(jj, nj)] + us[jj], us[wp2(jj, nj)] + us[wm1(jj, nj)]);
      } else if (f == 3) {
        const T* __restrict__ vs = d.vbuf[d.cur] + (o + jj);
        x = average4(vs[(unsigned)nj * wp1(ii, ni)] + vs[(unsigned)nj * ii],
                     vs[(unsigned)nj * wp2(ii, ni)] + vs[(unsigned)nj * wm1(ii, ni)]);
      } else if (f == 4) {
        const T* __restrict__ w = d.w + c;
        if (kk == 0)
          x = T(0.5) * (w[pl] + w[0]);
        else if (kk == kz - 1)
          x = T(0.5) * (w[(unsigned)kz * pl] + w[(unsigned)(kz - 1) * pl]);
        else
          x = average4(w[(kk + 1) * pl] + w[kk * pl], w[(kk + 2) * pl] + w[(kk - 1) * pl]);
      } else {
        return src[u][c + o];
      }
      const_cast<T*>(src[u])[c + o] = x;
      return x;
    }
  };
  if constexpr (kLean<T>) {
    // Flux form: the windows hold the two values a face takes and the
    // differences across it and its neighbours, each formed once.  Pass 1 at
    // step t: xb, xc = x(t), x(t+1), dx, ex = x(t-1)-x(t), x(t)-x(t+1); pass 2
    // at m = t-2: y1, y2, y3 = wz1(m .. m+2), dy, ey likewise.
    T xb[F], xc[F], dx[F], ex[F], y1[F], y2[F], y3[F], dy[F], ey[F];
    T h1[F], h2[F];  // half WAF values of the faces above levels t and m
#pragma unroll
    for (int u = 0; u < F; ++u) {
      xb[u] = xval(u, 0); xc[u] = kz > 1 ? xval(u, 1) : xb[u];
      dx[u] = T(0); ex[u] = sub_rn(xb[u], xc[u]);
      y1[u] = T(0); y2[u] = T(0); y3[u] = T(0); dy[u] = T(0); ey[u] = T(0);
      h1[u] = T(0); h2[u] = T(0);
    }
    T sB = T(0), sC = s[c];                       // s(t-1), s(t)
    T uA = T(0), uB = T(0), dA = T(0), dB = T(0);  // s(k) wafu(k), s(k+1) wafd(k) at k = t-2, t-1
    auto step = [&](const int t, auto fast) {
      constexpr bool FAST = decltype(fast)::value;
      T uC = T(0), dC = T(0), sD = T(0);
      const int m = t - 2;
      if (FAST || t <= kz) {
        sD = s[c + (unsigned)t * pl];
        uC = mul_rn(sC, wafu[c + (unsigned)(t - 1) * pl]);
        dC = mul_rn(sD, wafd[c + (unsigned)(t - 1) * pl]);
      }
      const Face<T> f1 = face_of(sD >= T(0), sD, dtrdz), f2 = face_of(sB >= T(0), sB, dtrdz);
      const T v1 = sub_rn(uC, dC), v2 = sub_rn(uA, dA);
#pragma unroll
      for (int u = 0; u < F; ++u) {
        T w1 = y3[u];
        if (FAST || t <= kz) {
          const T xd = (FAST || t + 2 <= kz) ? xval(u, t + 1) : xc[u];  // x(min(t+2, kz))
          const T d3 = sub_rn(xc[u], xd);
          const T h = (FAST || t <= kz - 1) ? waf_half(f1, ex[u], d3, dx[u], xc[u], xb[u]) : T(0);
          w1 = waf_update(xb[u], dC, h, uC, h1[u], v1, xb[u]);
          dx[u] = ex[u]; ex[u] = d3; xb[u] = xc[u]; xc[u] = xd; h1[u] = h;
        }
        // wz1(t-1) - wz1(t); none at t = 1, and for t > kz wz1 stays at wz1(kz)
        const T e3 = (FAST || t > 1) ? sub_rn(y3[u], w1) : T(0);
        y1[u] = y2[u]; y2[u] = y3[u]; y3[u] = w1;
        if (FAST || m >= 1) {
          const T h = (FAST || m <= kz - 1) ? waf_half(f2, ey[u], e3, dy[u], y2[u], y1[u]) : T(0);
          wz[u][c + (unsigned)(m - 1) * pl] = waf_update(y1[u], dA, h, uA, h2[u], v2, y1[u]);
          h2[u] = h;
        }
        dy[u] = ey[u]; ey[u] = e3;
      }
      sB = sC; sC = sD;
      uA = uB; uB = uC; dA = dB; dB = dC;
    };
    const int tf = kz - 2 >= 4 ? kz - 2 : 3;  // last step of the fast range
    for (int t = 1; t <= 3; ++t) step(t, std::false_type());
    for (int t = 4; t <= tf; ++t) step(t, std::true_type());
    for (int t = tf + 1; t <= kz + 2; ++t) step(t, std::false_type());
    return;
  } else {
  T xa[F], xb[F], xc[F];               // pass-1 window x(t-1), x(t), x(t+1)
  T wfw1[F], wfw2[F];                  // wfw1(t), wfw2(m)
  T y0[F], y1[F], y2[F], y3[F];        // wz1(t-3 .. t)
#pragma unroll
  for (int u = 0; u < F; ++u) {
    xa[u] = xval(u, 0); xb[u] = xa[u]; xc[u] = kz > 1 ? xval(u, 1) : xa[u];
    wfw1[u] = T(0); wfw2[u] = T(0);
    y0[u] = T(0); y1[u] = T(0); y2[u] = T(0); y3[u] = T(0);
  }
  T sA = T(0), sB = T(0), sC = s[c], sD;    // s(t-2 .. t+1)
  T uA = T(0), uB = T(0), dA = T(0), dB = T(0);  // wafu/wafd at t-2, t-1
  // one step t of both passes; FAST: 4 <= t <= kz-2, where no boundary
  // case applies (t2 = t+2, both fluxes exist, ym = y0), so the tests drop
  auto step = [&](const int t, auto fast) {
    constexpr bool FAST = decltype(fast)::value;
    T uC = T(0), dC = T(0);
    sD = T(0);
    const int m = t - 2;
    if (FAST || t <= kz) {
      sD = s[c + (unsigned)t * pl];
      uC = wafu[c + (unsigned)(t - 1) * pl];
      dC = wafd[c + (unsigned)(t - 1) * pl];
    }
    const int t2 = FAST ? t + 2 : (t + 2 <= kz ? t + 2 : kz);
#pragma unroll
    for (int u = 0; u < F; ++u) {
      T w1 = y3[u];
      if (FAST || t <= kz) {
        const T xd = (FAST || t + 2 <= kz) ? xval(u, t2 - 1) : xc[u];  // x(min(t+2, kz))
        const T wfw1n = (FAST || t <= kz - 1) ? waf_vflux(sD, dtrdz, xa[u], xb[u], xc[u], xd) : T(0);
        w1 = ((xb[u] - wfw1[u] * uC) + wfw1n * dC) + (sC * uC - sD * dC) * xb[u];
        xa[u] = xb[u]; xb[u] = xc[u]; xc[u] = xd; wfw1[u] = wfw1n;
      }
      y0[u] = y1[u]; y1[u] = y2[u]; y2[u] = y3[u]; y3[u] = w1;  // for t > kz, wz1 stays clamped at wz1(kz)
      if (FAST || m >= 1) {
        const T ym = (!FAST && m == 1) ? y1[u] : y0[u];
        const T wfw2n = (FAST || m <= kz - 1) ? waf_vflux(sB, dtrdz, ym, y1[u], y2[u], y3[u]) : T(0);
        wz[u][c + (unsigned)(m - 1) * pl] = ((y1[u] - wfw2[u] * uA) + wfw2n * dA) + (sA * uA - sB * dA) * y1[u];
        wfw2[u] = wfw2n;
      }
    }
    sA = sB; sB = sC; sC = sD;
    uA = uB; uB = uC; dA = dB; dB = dC;
  };
  const int tf = kz - 2 >= 4 ? kz - 2 : 3;  // last step of the fast range
  for (int t = 1; t <= 3; ++t) step(t, std::false_type());
  for (int t = 4; t <= tf; ++t) step(t, std::true_type());
  for (int t = tf + 1; t <= kz + 2; ++t) step(t, std::false_type());
  }
}

template <class T, int F>
__device__ __forceinline__ void b_waf_vertical(const View<T>& d, const int bx, const int by, const int bz) {
  constexpr int NG = kNumAdvected / F;
  const int g = bx % NG;
  const int tj = bx / NG;
  int jj, ii;
  point_at<kColBX, kColBY>(d, tj, by, jj, ii);
  if (jj >= d.nj || ii >= d.ni) return;
  // the groups holding fields 2..4 (block-uniform branch)
  if constexpr (F == 1) {
    if (g == 2) b_waf_vertical_g<T, 1, 2>(d, g, jj, ii);
    else if (g == 3) b_waf_vertical_g<T, 1, 3>(d, g, jj, ii);
    else if (g == 4) b_waf_vertical_g<T, 1, 4>(d, g, jj, ii);
    else b_waf_vertical_g<T, 1, -1>(d, g, jj, ii);
  } else if constexpr (F == 2) {
    if (g == 1) b_waf_vertical_g<T, 2, 1>(d, g, jj, ii);
    else if (g == 2) b_waf_vertical_g<T, 2, 2>(d, g, jj, ii);
    else b_waf_vertical_g<T, 2, -1>(d, g, jj, ii);
  } else if constexpr (F == 5) {
    if (g == 0) b_waf_vertical_g<T, 5, 0>(d, g, jj, ii);
    else b_waf_vertical_g<T, 5, -1>(d, g, jj, ii);
  } else {
    b_waf_vertical_g<T, F, 0>(d, g, jj, ii);
  }
}

// FP32 with jx even: two columns (j, j+1) of one field per thread.  One column
// per thread (above) is bound by issue slots and by the latency of its loads
// (91 instructions a point, 63 % of the slots, 35 % of DRAM at 512 x 512 x 60).
// Here products, sums and fused operations take both columns in one
// instruction, the differences across a face serve three fluxes, the loop
// turns three levels so that its windows move by name, and what a level reads
// comes through shared memory two steps ahead.  ux, vx and wx are formed from
// staged winds: formed from plain loads their blocks took twice the time of
// the others and the kernel 1.27 ms.  Every rounding is that of the one-column
// form.  Per step, one column -> two: 1024 x 1024 x 60 6.63 -> 4.31 ms, 512 x
// 512 x 60 1.70 -> 1.11, 256 x 256 x 40 0.322 -> 0.228, 100 x 100 x 30 0.074 ->
// 0.060.  Six blocks an SM (80 registers, no spills): seven 1.16 ms at 512 x
// 512 x 60; five fields of the same columns per block, to share s, wafu and
// wafd in L1, 1.57 instead of 1.40 at that stage.
struct VFace2 {
  bool p0, p1;   // the positive direction is upwind
  f32x2 nis, zm, nh;  // -is, is - zamu, -0.5 s
};
__device__ __forceinline__ VFace2 vface2(f32x2 s, f32x2 dt) {
  VFace2 f;
  const f32x2 z = mul2(s, dt);
  const float2 zz = unpack2(z);
  f.p0 = zz.x >= 0.f;
  f.p1 = zz.y >= 0.f;
  f.nis = pack2(f.p0 ? -1.f : 1.f, f.p1 ? -1.f : 1.f);
  f.zm = sub2(pack2(f.p0 ? 1.f : -1.f, f.p1 ? 1.f : -1.f), z);
  f.nh = mul2(s, pack2(-0.5f, -0.5f));
  return f;
}
__device__ __forceinline__ float bb_of(float num, float d) {
  const float r = qdiv(num, copysignf(fmaxf(fabsf(d), (float)kMinden), d));
  return fmaxf(__saturatef(2.f * r), fminf(r, 2.f));
}
// minus the WAF flux: d, dm, dp the differences behind minus ahead at the
// face and its neighbours, x0 and x1 the values behind and ahead
__device__ __forceinline__ f32x2 nflux2(const VFace2& f, f32x2 dm, f32x2 d, f32x2 dp, f32x2 x0, f32x2 x1) {
  const float2 a = unpack2(dm), b = unpack2(d), c = unpack2(dp);
  const f32x2 bb = pack2(bb_of(f.p0 ? c.x : a.x, b.x), bb_of(f.p1 ? c.y : a.y, b.y));
  const f32x2 nphi = fma2(bb, f.zm, f.nis);
  return mul2(f.nh, fma2(nphi, d, add2(x1, x0)));
}
constexpr int kVPAhead = 2;                 // steps a level's values travel ahead
constexpr int kVPArrays = 7, kVPThreads = kColBX * kColBY;  // s, wafu, wafd and up to four of x
constexpr int kVPSmem = (kVPAhead + 1) * kVPArrays * kVPThreads * 8;
__device__ __forceinline__ void cp_async8(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
template <int G>
__device__ __forceinline__ void b_waf_vertical_pair(const View<float>& d, const int g, const int jj, const int ii, const unsigned mask) {
  const int nj = d.nj, ni = d.ni, kz = d.kz;
  const unsigned pl = (unsigned)d.pl;
  const unsigned c = (unsigned)jj + (unsigned)nj * (unsigned)ii;
  const float* src = d.fset[d.fcur][g];
  float* wz = d.wz + (size_t)g * d.pl * kz;
  const float* __restrict__ s = d.s;
  const float* __restrict__ wafu = d.wafu;
  const float* __restrict__ wafd = d.wafd;
  auto ld = [](const float* q) -> f32x2 { return pack2(*reinterpret_cast<const float2*>(q)); };
  auto st = [](float* q, f32x2 v) { *reinterpret_cast<float2*>(q) = unpack2(v); };
  const int jm1 = wm1(jj, nj), jp2 = wp2(jj, nj);
  // x(0), x(1)
  auto xval = [&](const int kk) -> f32x2 {
    const unsigned o = (unsigned)kk * pl;
    float2 x;
    if constexpr (G == 2) {
      const float* __restrict__ us = d.ubuf[d.cur] + (o + (unsigned)nj * ii);
      const float2 u = *reinterpret_cast<const float2*>(us + jj);
      const float um = us[jm1], u2 = us[jp2], u3 = us[jp2 + 1];
      x.x = 0.5625f * (u.y + u.x) - 0.0625f * (u2 + um);
      x.y = 0.5625f * (u2 + u.y) - 0.0625f * (u3 + u.x);
    } else if constexpr (G == 3) {
      const float* __restrict__ vs = d.vbuf[d.cur] + (o + jj);
      const float2 n1 = *reinterpret_cast<const float2*>(vs + (unsigned)nj * wp1(ii, ni));
      const float2 v0 = *reinterpret_cast<const float2*>(vs + (unsigned)nj * ii);
      const float2 n2 = *reinterpret_cast<const float2*>(vs + (unsigned)nj * wp2(ii, ni));
      const float2 m1 = *reinterpret_cast<const float2*>(vs + (unsigned)nj * wm1(ii, ni));
      x.x = 0.5625f * (n1.x + v0.x) - 0.0625f * (n2.x + m1.x);
      x.y = 0.5625f * (n1.y + v0.y) - 0.0625f * (n2.y + m1.y);
    } else if constexpr (G == 4) {
      const float* __restrict__ w = d.w + c;
      auto W = [&](int k) { return *reinterpret_cast<const float2*>(w + (unsigned)k * pl); };
      if (kk == 0) {
        const float2 a = W(1), b = W(0);
        x.x = 0.5f * (a.x + b.x);
        x.y = 0.5f * (a.y + b.y);
      } else {
        const float2 a = W(kk + 1), b = W(kk), e = W(kk + 2), f = W(kk - 1);
        x.x = 0.5625f * (a.x + b.x) - 0.0625f * (e.x + f.x);
        x.y = 0.5625f * (a.y + b.y) - 0.0625f * (e.y + f.y);
      }
    } else {
      return ld(src + c + o);
    }
    *reinterpret_cast<float2*>(const_cast<float*>(src) + c + o) = x;
    return pack2(x);
  };
  const f32x2 dt = pack2(d.dtrdz_a, d.dtrdz_a), zero = pack2(0.f, 0.f), neg = pack2(-1.f, -1.f);
  // What step t reads -- s(t), wafu(t-1), wafd(t-1) and what x(t+1) is made
  // of -- travels kVPAhead steps ahead through the thread's own slots of
  // shared memory.
  extern __shared__ float2 vp_ring[];
  float2* const slot0 = vp_ring + (threadIdx.y * kColBX + threadIdx.x);
  const float* const sp = s + c + pl;
  const float* const up = wafu + c;
  const float* const dp = wafd + c;
  const float* const xp = (G == 2 ? d.ubuf[d.cur] : G == 3 ? d.vbuf[d.cur] : G == 4 ? d.w + 2 * (size_t)pl : src) + c + 2 * (size_t)pl;
  const bool first = threadIdx.x == 0, last = threadIdx.x == kColBX - 1 || jj + 2 >= nj;
  const int em = jm1 - jj, e2 = jp2 - jj;
  const int r1 = nj * (wp1(ii, ni) - ii), r2 = nj * (wp2(ii, ni) - ii), rm = nj * (wm1(ii, ni) - ii);
  // step t's values into slot st; o = (t - 1) pl, ox the same or, where
  // x(t+1) is below the column, its last
  auto fetch = [&](const unsigned o, const unsigned ox, const int st) {
    float2* q = slot0 + st * (kVPArrays * kVPThreads);
    cp_async8(q, sp + o);
    cp_async8(q + kVPThreads, up + o);
    cp_async8(q + 2 * kVPThreads, dp + o);
    const float* x = xp + ox;
    cp_async8(q + 3 * kVPThreads, x);
    if constexpr (G == 2) {
      if (first) cp_async_elem(&q[4 * kVPThreads].x, x + em);
      if (last) cp_async8(q + 5 * kVPThreads, x + e2);
    }
    if constexpr (G == 3) {
      cp_async8(q + 4 * kVPThreads, x + r1);
      cp_async8(q + 5 * kVPThreads, x + r2);
      cp_async8(q + 6 * kVPThreads, x + rm);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  f32x2 wa = zero, wb = zero, wc = zero;  // w(t), w(t+1), w(t+2) (G == 4)
  if constexpr (G == 4) {
    wa = ld(d.w + c + pl);
    wb = ld(d.w + c + 2 * pl);
    wc = ld(d.w + c + 3 * pl);
  }
  // x(t+1) of step t from its slot
  auto xnext = [&](const int t, const float2* q, auto bottom) -> f32x2 {
    const f32x2 x0 = pack2(q[3 * kVPThreads]);
    if constexpr (G < 0) {
      return x0;
    } else {
      f32x2 hi, lo;  // the inner and the outer two points
      if constexpr (G == 2) {
        const float2 u = unpack2(x0);
        float um = __shfl_up_sync(mask, u.y, 1), u2 = __shfl_down_sync(mask, u.x, 1), u3 = __shfl_down_sync(mask, u.y, 1);
        if (first) um = q[4 * kVPThreads].x;
        if (last) {
          const float2 e = q[5 * kVPThreads];
          u2 = e.x;
          u3 = e.y;
        }
        hi = add2(pack2(u.y, u2), x0);
        lo = add2(pack2(u2, u3), pack2(um, u.x));
      } else if constexpr (G == 3) {
        hi = add2(pack2(q[4 * kVPThreads]), x0);
        lo = add2(pack2(q[5 * kVPThreads]), pack2(q[6 * kVPThreads]));
      } else {
        hi = add2(wc, wb);
        lo = add2(x0, wa);
        wa = wb; wb = wc; wc = x0;
      }
      const f32x2 x = (G == 4 && bottom(t)) ? mul2(pack2(0.5f, 0.5f), hi)
                                            : fma2(pack2(0.5625f, 0.5625f), hi, mul2(lo, pack2(-0.0625f, -0.0625f)));
      st(const_cast<float*>(src) + c + (unsigned)(t + 1) * pl, x);
      return x;
    }
  };
  auto fetch_at = [&](const int t, const int st) {
    fetch((unsigned)(min(t, kz) - 1) * pl, (unsigned)(min(t, G == 4 ? kz - 3 : kz - 2) - 1) * pl, st);
  };
#pragma unroll
  for (int n = 0; n < kVPAhead; ++n) fetch_at(1 + n, n);
  f32x2 xb = xval(0), xc = xval(1);
  f32x2 dx = zero, ex = sub2(xb, xc);           // x(t-1) - x(t), x(t) - x(t+1)
  f32x2 y1 = zero, y2 = zero, y3 = zero, dy = zero, ey = zero;  // wz1(m .. m+2) and their differences
  f32x2 h1 = zero, h2 = zero;                   // minus the fluxes above levels t and m
  f32x2 sB = zero, sC = ld(s + c);
  f32x2 uA = zero, uB = zero, dA = zero, dB = zero, vA = zero, vB = zero;
  // rd: the slot of step t, (t - 1) mod (kVPAhead + 1)
  // FAST: 4 <= t and t + kVPAhead <= kz - 3, where no test is needed
  auto step = [&](const int t, const int rd, auto fast) {
    constexpr bool FAST = decltype(fast)::value;
    const int m = t - 2;
    f32x2 uC = zero, dC = zero, vC = zero, sD = zero;
    f32x2 w1 = y3;
    if (FAST || t <= kz) {
      asm volatile("cp.async.wait_group %0;" ::"n"(kVPAhead - 1) : "memory");
      const float2* q = slot0 + rd * (kVPArrays * kVPThreads);
      sD = pack2(q[0]);
      uC = pack2(q[kVPThreads]);
      dC = mul2(pack2(q[2 * kVPThreads]), neg);
      const f32x2 xd = (FAST || t + 2 <= kz) ? xnext(t, q, [&](int t) { return !FAST && t == kz - 2; }) : xc;
      const int wr = rd == 0 ? kVPAhead : rd - 1;
      const unsigned o = (unsigned)(t + kVPAhead - 1) * pl;
      if constexpr (FAST) fetch(o, o, wr);
      else fetch_at(t + kVPAhead, wr);
      const f32x2 d3 = sub2(xc, xd);
      const f32x2 h = (FAST || t <= kz - 1) ? nflux2(vface2(sD, dt), dx, ex, d3, xb, xc) : zero;
      vC = fma2(sC, uC, mul2(sD, dC));
      w1 = fma2(vC, xb, fma2(h, dC, fma2(h1, uC, xb)));
      dx = ex; ex = d3; xb = xc; xc = xd; h1 = h;
    }
    const f32x2 e3 = (FAST || t > 1) ? sub2(y3, w1) : zero;
    y1 = y2; y2 = y3; y3 = w1;
    if (FAST || m >= 1) {
      const f32x2 h = (FAST || m <= kz - 1) ? nflux2(vface2(sB, dt), dy, ey, e3, y1, y2) : zero;
      st(wz + c + (unsigned)(m - 1) * pl, fma2(vA, y1, fma2(h, dA, fma2(h2, uA, y1))));
      h2 = h;
    }
    dy = ey; ey = e3;
    sB = sC; sC = sD;
    uA = uB; uB = uC; dA = dB; dB = dC; vA = vB; vB = vC;
  };
  constexpr int NS = kVPAhead + 1;
  int t = 1;
  for (; t <= 3; ++t) step(t, (t - 1) % NS, std::false_type());
  // NS steps at a time, so that the windows rotate by name
  for (; t + 2 * kVPAhead <= kz - 3; t += NS) {
#pragma unroll
    for (int n = 0; n < NS; ++n) step(t + n, (3 + n) % NS, std::true_type());
  }
  int r = (t - 1) % NS;
  for (; t <= kz + 2; ++t) {
    step(t, r, std::false_type());
    r = r == kVPAhead ? 0 : r + 1;
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
}
__global__ void __launch_bounds__(kColBX* kColBY, 6) k_waf_vertical_pair(View<float> d) {
  const int g = blockIdx.x % kNumAdvected;
  const int jj = ((blockIdx.x / kNumAdvected) * kColBX + threadIdx.x) * 2, ii = blockIdx.y * kColBY + threadIdx.y;
  if (ii >= d.ni) return;
  const unsigned mask = __ballot_sync(0xffffffffu, jj < d.nj);
  if (jj >= d.nj) return;
  if (g == 2) b_waf_vertical_pair<2>(d, g, jj, ii, mask);
  else if (g == 3) b_waf_vertical_pair<3>(d, g, jj, ii, mask);
  else if (g == 4) b_waf_vertical_pair<4>(d, g, jj, ii, mask);
  else b_waf_vertical_pair<-1>(d, g, jj, ii, mask);
}

// Blocks per SM by bulk type and fields per thread.  FP32, one field per
// thread: 12 (40 registers; with 32-bit element offsets about 50 bytes
// spilled, 128 with 64-bit ones): 1.69 ms per step at 512 x 512 x 60
// (1.88 with 64-bit offsets), against 1.75 at 13 to 16 blocks, 1.76 at 10
// (48 registers) and 2.00 at 9 (56 registers, no spills); the other
// variants keep the occupancy of their unconstrained register counts.
template <class T, int F>
constexpr int vert_min_blocks() {
  if (sizeof(T) == 4) return F == 1 ? 12 : F == 2 ? 9 : F == 5 ? 5 : 3;
  return F == 1 ? 6 : F == 2 ? 4 : F == 5 ? 2 : 1;
}

template <class T, int F>
__global__ void __launch_bounds__(kColBX* kColBY, vert_min_blocks<T, F>()) k_waf_vertical(View<T> d) {
  b_waf_vertical<T, F>(d, blockIdx.x, tile_y(d), blockIdx.z);
}

template <class T, int F>
__global__ void __launch_bounds__(kColBX* kColBY, vert_min_blocks<T, F>())
    kb_waf_vertical(const View<T>* __restrict__ views, const int4* __restrict__ tiles) {
  __shared__ View<T> sv;
  const int4 t = tiles[blockIdx.x];
  copy_view(&sv, views + t.x);
  __syncthreads();
  b_waf_vertical<T, F>(sv, t.y, t.z, t.w);
}

// ---- advection: meridional + zonal WAF (:1075-1187) ----------------------
// Block = 32 (j) x 8 (i) output points of kHzLevels consecutive levels, ten
// fields per level.  Per field: the wz tile with a 2-point halo in both
// directions and the pp tile go to shared memory; the meridional fluxes and
// p0 are formed for the 36-wide strip the zonal step needs, then the zonal
// fluxes and the new pp.  p0 never leaves the SM.  The next field's tiles
// travel in registers while the current one is computed.  The result goes to
// the other field buffer (dst): neighbouring blocks still read the old pp at
// their halo columns.  The wrapped (periodic) tile offsets are computed once
// per block and reused for every level and field; d.hz_levels (levels per
// block) is picked by the autotuner (moloch_gpu_autotune).

// WAF flux between cells m1 and x0 (limiter from m2, p1), the reference's
// expression (:1091-1106, :1148-1163)
template <class T>
__device__ __forceinline__ T waf_hflux(T zamu, T m2, T m1, T x0, T p1) {
  const bool pos = __double_as_longlong(zamu) > 0;
  const T num = (pos ? m1 : p1) - (pos ? m2 : x0);  // ih = i-1 or i+1, ihm1 = i-2 or i
  return waf_flux_rn(pos, zamu, num, x0 - m1, m1, x0);
}
// FP32 storage: rearranged as waf_vflux<float>
template <>
__device__ __forceinline__ float waf_hflux<float>(float zamu, float m2, float m1, float x0, float p1) {
  const bool pos = zamu > 0.f;
  const float d = x0 - m1;
  const float den = copysignf(fmaxf(fabsf(d), (float)kMinden), d);
  const float r = qdiv(pos ? m1 - m2 : p1 - x0, den);
  const float bb = fmaxf(__saturatef(2.f * r), fminf(r, 2.f));
  const float is = pos ? 1.f : -1.f;
  const float zphi = fmaf(bb, zamu - is, is);
  return fmaf(zphi, -d, m1 + x0);
}

template <class T>
__device__ __forceinline__ void b_waf_horizontal(const View<T>& d, const int bx, const int by, const int bz) {
  constexpr int TJ = 32, TI = 8, HJ = TJ + 4, HI = TI + 4;
  constexpr int NW = HI * HJ, NP = TI * HJ, NM = (TI + 1) * HJ, NZ = TI * (TJ + 1);
  // flat row-major tiles: a work item's linear number q is its own index
  __shared__ T sw[2][NW];  // wz, rows i0-2 .. i0+TI+1, cols j0-2 .. j0+TJ+1
  __shared__ T sp[2][NP];  // pp (old), rows i0 .., cols j0-2 ..
  __shared__ T smf[NM];    // meridional fluxes at rows i0 .. i0+TI
  __shared__ T sp0[NP];    // p0
  __shared__ T szf[NZ];    // zonal fluxes at cols j0 .. j0+TJ
  const int tx = threadIdx.x, ty = threadIdx.y, tid = tx + 32 * ty;
  const int nj = d.nj, ni = d.ni, kz = d.kz, pl = d.pl;
  const int j0 = bx * TJ, i0 = by * TI;
  const int k0 = bz * d.hz_levels;
  const int k1 = min(k0 + d.hz_levels, kz);
  const T* __restrict__ u = d.ubuf[d.cur];
  const T* __restrict__ v = d.vbuf[d.cur];
  const T dtrdx = d.dtrdx_a, dtrdy = d.dtrdy_a;
  const int rot = d.rotllr;

  // ---- per block: wrapped offsets (valid for every level) and map factors
  int woff[2], poff[2], pnoff[2], zoffg[2], zoff[2];
  T mrm[2], prs[2], prn[2], pmx[2], zm[2];
  for (int n = 0; n < 2; ++n) {
    const int q = tid + 256 * n;
    const int jq = wrapn(j0 - 2 + q % HJ, nj);
    woff[n] = q < NW ? jq + nj * wrapn(i0 - 2 + q / HJ, ni) : 0;
    const int iq = wrapn(i0 + q / HJ, ni);  // meridional flux rows and p0 rows
    poff[n] = q < NM ? jq + nj * iq : 0;
    pnoff[n] = q < NP ? jq + nj * wp1(iq, ni) : 0;
    const int r = q / (TJ + 1), x = q % (TJ + 1);
    zoff[n] = q < NZ ? r * HJ + x : 0;
    zoffg[n] = q < NZ ? wrapn(j0 + x, nj) + nj * wrapn(i0 + r, ni) : 0;
  }
  const int jo = j0 + tx, io = i0 + ty;
  const bool ook = jo < nj && io < ni;
  const int co = ook ? jo + nj * io : 0;
  const int coe = ook ? wp1(jo, nj) + nj * io : 0;
  const int op0 = ty * HJ + tx + 2, ozf = ty * (TJ + 1) + tx;

  // raw per-level inputs (velocities, metric factors), loaded one level ahead
  T rv[2], rwn[2], rws[2], rvn[2], ru[2], rwe = T(0), rww = T(0), ruw = T(0), rue = T(0);
  auto fetch_level = [&](int k) {
    const size_t ko = (size_t)k * pl;
    for (int n = 0; n < 2; ++n) {
      const int q = tid + 256 * n;
      rv[n] = q < NM ? v[ko + poff[n]] : T(0);
      rwn[n] = q < NP ? d.wafn[ko + poff[n]] : T(0);
      rws[n] = q < NP ? d.wafs[ko + poff[n]] : T(0);
      rvn[n] = q < NP ? v[ko + pnoff[n]] : T(0);
      ru[n] = q < NZ ? u[ko + zoffg[n]] : T(0);
    }
    rwe = d.wafe[ko + co]; rww = d.wafw[ko + co];
    ruw = u[ko + co]; rue = u[ko + coe];
  };
  T rw[2], rp[2];
  auto fetch = [&](int k, int f) {
    const T* __restrict__ wzf = d.wz + ((size_t)f * kz + k) * pl;
    const T* __restrict__ ppf = d.fset[d.fcur][f] + (size_t)k * pl;
    for (int n = 0; n < 2; ++n) {
      const int q = tid + 256 * n;
      rw[n] = q < NW ? wzf[woff[n]] : T(0);
      rp[n] = q < NP ? ppf[poff[n]] : T(0);
    }
  };
  auto stash = [&](int b) {
    for (int n = 0; n < 2; ++n) {
      const int q = tid + 256 * n;
      if (q < NW) sw[b][q] = rw[n];
      if (q < NP) sp[b][q] = rp[n];
    }
  };
  fetch_level(k0);
  fetch(k0, 0);
  for (int n = 0; n < 2; ++n) {
    const int q = tid + 256 * n;
    mrm[n] = q < NM ? d.rmv[poff[n]] : T(1);
    prs[n] = q < NP ? d.rmv[poff[n]] : T(1);
    prn[n] = q < NP ? d.rmv[pnoff[n]] : T(1);
    pmx[n] = q < NP ? d.mx2[poff[n]] : T(0);
    zm[n] = q < NZ ? (rot ? d.mu[zoffg[n]] : d.rmu[zoffg[n]]) : T(0);
  }
  const T ormw = d.rmu[co], orme = d.rmu[coe], omx = d.mx2[co];
  stash(0);
  __syncthreads();
  int b = 0;
  for (int k = k0; k < k1; ++k) {
    const size_t ko = (size_t)k * pl;
    T mz[2], mfac[2], pn[2], ps_[2], pdv[2], zz[2], zfac[2];
    Face<T> mf[2], zf[2];
    T oe = rwe, ow = rww, odv;
    if constexpr (kLean<T>) {
      // the faces' velocity terms; the cells' metric terms times the face
      // velocities (and the squared map factor, non-ROTLLR)
      for (int n = 0; n < 2; ++n) {
        const T vm = rot ? rv[n] : mul_rn(rv[n], mrm[n]);
        mf[n] = face_of(vm > T(0), vm, dtrdy);
        T cs = mul_rn(rot ? rv[n] : mul_rn(rv[n], prs[n]), rws[n]);
        T cn = mul_rn(rot ? rvn[n] : mul_rn(rvn[n], prn[n]), rwn[n]);
        if (!rot) { cs = mul_rn(cs, pmx[n]); cn = mul_rn(cn, pmx[n]); }
        ps_[n] = cs; pn[n] = cn; pdv[n] = sub_rn(cn, cs);
        const T um = mul_rn(ru[n], zm[n]);
        zf[n] = face_of(um > T(0), um, dtrdx);
      }
      ow = mul_rn(rot ? ruw : mul_rn(ruw, ormw), ow);
      oe = mul_rn(rot ? rue : mul_rn(rue, orme), oe);
      if (!rot) { ow = mul_rn(ow, omx); oe = mul_rn(oe, omx); }
      odv = sub_rn(oe, ow);
    } else {
    for (int n = 0; n < 2; ++n) {
      const T vv = rv[n];
      mz[n] = rot ? vv * dtrdy : (vv * mrm[n]) * dtrdy;
      mfac[n] = rot ? T(0.5) * vv : (T(0.5) * vv) * mrm[n];
      const T zrfmn = rwn[n], zrfms = rws[n], vs = rv[n], vn = rvn[n];
      pn[n] = zrfmn; ps_[n] = zrfms;
      pdv[n] = rot ? (vn * zrfmn - vs * zrfms) : ((vn * prn[n]) * zrfmn - (vs * prs[n]) * zrfms);
      const T uu = ru[n];
      zz[n] = (uu * zm[n]) * dtrdx;
      zfac[n] = rot ? T(0.5) * uu : (T(0.5) * uu) * zm[n];
    }
    odv = rot ? (rue * oe - ruw * ow) : ((rue * orme) * oe - (ruw * ormw) * ow);
    }
    for (int f = 0; f < kNumAdvected; ++f) {
      const T* __restrict__ W = sw[b];
      const T* __restrict__ P = sp[b];
      const bool next_field = f + 1 < kNumAdvected;
      const bool next_level = !next_field && k + 1 < k1;
      if (next_field) fetch(k, f + 1);
      if (next_level) {
        fetch(k + 1, 0);
        fetch_level(k + 1);
      }
      for (int n = 0; n < 2; ++n) {  // zpby between tile rows r+1 and r+2 (flat: q+HJ, q+2HJ)
        const int q = tid + 256 * n;
        if (q < NM) {
          if constexpr (kLean<T>) {
            const T m2 = W[q], m1 = W[q + HJ], x0 = W[q + 2 * HJ], p1 = W[q + 3 * HJ];
            const bool pos = mf[n].pos;
            const T num = sub_rn(pos ? m1 : p1, pos ? m2 : x0);
            smf[q] = waf_half(mf[n], sub_rn(x0, m1), num, num, m1, x0);
          } else {
            smf[q] = mfac[n] * waf_hflux(mz[n], W[q], W[q + HJ], W[q + 2 * HJ], W[q + 3 * HJ]);
          }
        }
      }
      __syncthreads();
      for (int n = 0; n < 2; ++n) {  // p0 (:1113-1131, :1222-1240)
        const int q = tid + 256 * n;
        if (q < NP) {
          const T wc = W[q + 2 * HJ];
          if constexpr (kLean<T>) {
            sp0[q] = waf_update(wc, ps_[n], smf[q], pn[n], smf[q + HJ], pdv[n], P[q]);
            continue;
          }
          const T zdv = pdv[n] * P[q];
          sp0[q] = rot ? ((wc + smf[q] * ps_[n]) - smf[q + HJ] * pn[n]) + zdv
                       : wc + pmx[n] * (((smf[q] * ps_[n]) - smf[q + HJ] * pn[n]) + zdv);
        }
      }
      __syncthreads();
      for (int n = 0; n < 2; ++n) {  // zpbw between sp0 cols x+1 and x+2
        const int q = tid + 256 * n;
        if (q < NZ) {
          const int z0 = zoff[n];
          if constexpr (kLean<T>) {
            const T m2 = sp0[z0], m1 = sp0[z0 + 1], x0 = sp0[z0 + 2], p1 = sp0[z0 + 3];
            const bool pos = zf[n].pos;
            const T num = sub_rn(pos ? m1 : p1, pos ? m2 : x0);
            szf[q] = waf_half(zf[n], sub_rn(x0, m1), num, num, m1, x0);
          } else {
            szf[q] = zfac[n] * waf_hflux(zz[n], sp0[z0], sp0[z0 + 1], sp0[z0 + 2], sp0[z0 + 3]);
          }
        }
      }
      __syncthreads();
      if (ook) {  // new pp (:1173-1187, :1283-1297)
        const T p0 = sp0[op0];
        T out;
        if constexpr (kLean<T>) {
          out = waf_update(p0, ow, szf[ozf], oe, szf[ozf + 1], odv, P[op0]);
        } else {
          const T zdv = odv * P[op0];
          out = rot ? ((p0 + szf[ozf] * ow) - szf[ozf + 1] * oe) + zdv
                    : p0 + omx * (((szf[ozf] * ow) - szf[ozf + 1] * oe) + zdv);
        }
        d.fset[d.fcur ^ 1][f][ko + co] = out;
      }
      if (next_field || next_level) stash(b ^ 1);  // the other buffer was last read two fields ago
      b ^= 1;
      __syncthreads();
    }
  }
}

template <class T>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 3 : 2) k_waf_horizontal(View<T> d) {
  b_waf_horizontal<T>(d, blockIdx.x, blockIdx.y, blockIdx.z);
}

template <class T>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 3 : 2)
    kb_waf_horizontal(const View<T>* __restrict__ views, const int4* __restrict__ tiles) {
  __shared__ View<T> sv;
  const int4 t = tiles[blockIdx.x];
  copy_view(&sv, views + t.x);
  __syncthreads();
  b_waf_horizontal<T>(sv, t.y, t.z, t.w);
}

// ---- advection: horizontal WAF as warp strips (:1075-1187) ---------------
// One warp per strip of 28 output columns x R rows of one level (R =
// d.hz_levels, 16..64), 32 lanes on columns j0-2 .. j0+29.  Each lane marches
// down its own column: the wz values of rows i-1 .. i+2 and the meridional
// flux of the face above the row stay in registers, p0 of the row is formed
// in the lane, and the zonal fluxes take their p0 neighbours from the lanes
// beside it (warp shuffles).  No shared memory and no barriers.  Fields are
// processed G at a time so the per-row velocities and metric factors are
// loaded once per group.  The result goes to the other field buffer.
constexpr int kStripJ = 28;
template <class T> struct StripG { static constexpr int G = 10; };
template <> struct StripG<double> { static constexpr int G = 5; };

template <class T>
__device__ __forceinline__ void b_waf_hstrip(const View<T>& d, const int bx, const int k) {
  constexpr int G = StripG<T>::G;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int nj = d.nj, ni = d.ni, pl = d.pl, kz = d.kz;
  const int R = d.hz_levels;
  const int nsj = (nj + kStripJ - 1) / kStripJ, nsi = (ni + R - 1) / R;
  const int w = bx * (blockDim.x >> 5) + wid;
  if (w >= nsj * nsi) return;  // whole warp
  const int sj = w % nsj, si = w / nsj;
  const int j0 = sj * kStripJ;
  const int jl = j0 - 2 + lane;  // this lane's column before wrapping
  const int j = wrapn(jl, nj);
  const bool out_lane = lane >= 2 && lane < 2 + kStripJ && jl < nj;
  const int i_s = si * R, i_e = min(i_s + R, ni);
  const T* __restrict__ u = d.ubuf[d.cur] + (size_t)k * pl;
  const T* __restrict__ v = d.vbuf[d.cur] + (size_t)k * pl;
  const T* __restrict__ wn_ = d.wafn + (size_t)k * pl;
  const T* __restrict__ ws_ = d.wafs + (size_t)k * pl;
  const T* __restrict__ we_ = d.wafe + (size_t)k * pl;
  const T* __restrict__ ww_ = d.wafw + (size_t)k * pl;
  const T dtrdx = d.dtrdx_a, dtrdy = d.dtrdy_a;
  const bool rot = d.rotllr;
  auto row = [&](int i) { return (size_t)j + (size_t)nj * wrap2(i, ni); };

  if constexpr (kLean<T>) {
    // Flux form.  Per field: w0, wp1 = wz(i), wz(i+1), da, db =
    // wz(i)-wz(i-1), wz(i+1)-wz(i), and half the WAF value of the face below
    // row i; the row's velocity and metric terms are shared by the fields.
    static_assert(kNumAdvected % G == 0, "fields per group");
    for (int g0 = 0; g0 < kNumAdvected; g0 += G) {
      const T* wz[G];
      const T* pp[G];
      T* out[G];
      T w0[G], w1[G], da[G], db[G], vs[G];
#pragma unroll
      for (int g = 0; g < G; ++g) {
        wz[g] = d.wz + ((size_t)(g0 + g) * kz + k) * pl;
        pp[g] = d.fset[d.fcur][g0 + g] + (size_t)k * pl;
        out[g] = d.fset[d.fcur ^ 1][g0 + g] + (size_t)k * pl;
      }
      T v_i;  // v at the face below row i (times 1 / msfv, non-ROTLLR)
      {
        const size_t r = row(i_s);
        v_i = rot ? v[r] : mul_rn(v[r], d.rmv[r]);
        const Face<T> f = face_of(v_i > T(0), v_i, dtrdy);
        const size_t r2 = row(i_s - 2), r1 = row(i_s - 1), rp = row(i_s + 1);
#pragma unroll
        for (int g = 0; g < G; ++g) {
          const T a = wz[g][r2], b = wz[g][r1], cc = wz[g][r], e = wz[g][rp];
          w0[g] = cc; w1[g] = e;
          da[g] = sub_rn(cc, b); db[g] = sub_rn(e, cc);
          vs[g] = waf_half(f, da[g], sub_rn(b, a), db[g], b, cc);
        }
      }
      // the loads of row i+1 are issued while row i is computed
      T n_wp2[G], n_pold[G];
      T n_vn, n_rmvn, n_pn, n_ps, n_uu, n_oe, n_ow, n_zm, n_mx2;
      auto fetch_row = [&](int i) {
        const size_t r = row(i), rn = row(i + 1), r2 = row(i + 2);
#pragma unroll
        for (int g = 0; g < G; ++g) {
          n_wp2[g] = wz[g][r2];
          n_pold[g] = pp[g][r];
        }
        n_vn = v[rn];
        n_rmvn = rot ? T(1) : d.rmv[rn];
        n_pn = wn_[r]; n_ps = ws_[r];
        n_uu = u[r];
        n_oe = we_[r]; n_ow = ww_[r];
        n_zm = rot ? d.mu[r] : d.rmu[r];
        n_mx2 = rot ? T(1) : d.mx2[r];
      };
      fetch_row(i_s);
      for (int i = i_s; i < i_e; ++i) {
        const size_t r = row(i);
        const T v_n = rot ? n_vn : mul_rn(n_vn, n_rmvn);
        const T um = mul_rn(n_uu, n_zm), uf = rot ? n_uu : um;
        const T ufe = __shfl_down_sync(0xffffffffu, uf, 1);  // u(j+1)
        T cs = mul_rn(v_i, n_ps), cn = mul_rn(v_n, n_pn), cw = mul_rn(uf, n_ow), ce = mul_rn(ufe, n_oe);
        if (!rot) { cs = mul_rn(cs, n_mx2); cn = mul_rn(cn, n_mx2); cw = mul_rn(cw, n_mx2); ce = mul_rn(ce, n_mx2); }
        const T pdv = sub_rn(cn, cs), odv = sub_rn(ce, cw);
        const Face<T> fm = face_of(v_n > T(0), v_n, dtrdy), fz = face_of(um > T(0), um, dtrdx);
        T wp2v[G], poldv[G];
#pragma unroll
        for (int g = 0; g < G; ++g) { wp2v[g] = n_wp2[g]; poldv[g] = n_pold[g]; }
        if (i + 1 < i_e) fetch_row(i + 1);
#pragma unroll
        for (int g = 0; g < G; ++g) {
          const T dn = sub_rn(wp2v[g], w1[g]);
          const T vn = waf_half(fm, db[g], da[g], dn, w0[g], w1[g]);  // face between rows i and i+1
          const T p0 = waf_update(w0[g], cs, vs[g], cn, vn, pdv, poldv[g]);
          w0[g] = w1[g]; w1[g] = wp2v[g]; da[g] = db[g]; db[g] = dn; vs[g] = vn;
          const T pm1 = __shfl_up_sync(0xffffffffu, p0, 1);
          const T dz = sub_rn(p0, pm1);  // across the face between j-1 and j
          const T dzm = __shfl_up_sync(0xffffffffu, dz, 1), dzp = __shfl_down_sync(0xffffffffu, dz, 1);
          const T vw = waf_half(fz, dz, dzm, dzp, pm1, p0);
          const T ve = __shfl_down_sync(0xffffffffu, vw, 1);  // face between j and j+1
          if (out_lane) out[g][r] = waf_update(p0, cw, vw, ce, ve, odv, poldv[g]);
        }
        v_i = v_n;
      }
    }
    return;
  } else {
  for (int g0 = 0; g0 < kNumAdvected; g0 += G) {
    const int ng = min(G, kNumAdvected - g0);
    const T* wz[G];
    const T* pp[G];
    T* out[G];
    T wm1_[G], w0_[G], wp1_[G], fl_[G];  // wz(i-1), wz(i), wz(i+1), flux of face i
#pragma unroll
    for (int g = 0; g < G; ++g) {
      if (g < ng) {
        wz[g] = d.wz + ((size_t)(g0 + g) * kz + k) * pl;
        pp[g] = d.fset[d.fcur][g0 + g] + (size_t)k * pl;
        out[g] = d.fset[d.fcur ^ 1][g0 + g] + (size_t)k * pl;
      }
    }
    // warm-up: the flux of face i_s (between rows i_s-1 and i_s)
    T v_i, rmv_i = T(1);
    {
      const size_t r = row(i_s);
      v_i = v[r];
      if (!rot) rmv_i = d.rmv[r];
      const T mz = rot ? v_i * dtrdy : (v_i * rmv_i) * dtrdy;
      const T mfac = rot ? T(0.5) * v_i : (T(0.5) * v_i) * rmv_i;
      const size_t r2 = row(i_s - 2), r1 = row(i_s - 1), rp = row(i_s + 1);
#pragma unroll
      for (int g = 0; g < G; ++g) {
        if (g < ng) {
          const T a = wz[g][r2], b = wz[g][r1], c = wz[g][r], e = wz[g][rp];
          fl_[g] = mfac * waf_hflux(mz, a, b, c, e);
          wm1_[g] = b; w0_[g] = c; wp1_[g] = e;
        }
      }
    }
    // the loads of row i+1 are issued while row i is computed
    T n_wp2[G], n_pold[G];
    T n_vn, n_rmvn, n_pn, n_ps, n_uu, n_oe, n_ow, n_zm, n_mx2;
    auto fetch_row = [&](int i) {
      const size_t r = row(i), rn = row(i + 1), r2 = row(i + 2);
#pragma unroll
      for (int g = 0; g < G; ++g) {
        if (g < ng) {
          n_wp2[g] = wz[g][r2];
          n_pold[g] = pp[g][r];
        }
      }
      n_vn = v[rn];
      n_rmvn = rot ? T(1) : d.rmv[rn];
      n_pn = wn_[r]; n_ps = ws_[r];
      n_uu = u[r];
      n_oe = we_[r]; n_ow = ww_[r];
      n_zm = rot ? d.mu[r] : d.rmu[r];
      n_mx2 = rot ? T(0) : d.mx2[r];
    };
    fetch_row(i_s);
    for (int i = i_s; i < i_e; ++i) {
      const size_t r = row(i);
      // per-row values shared by the fields of the group
      const T v_n = n_vn, rmv_n = n_rmvn, pn = n_pn, ps = n_ps, uu = n_uu, oe = n_oe, ow = n_ow;
      const T zm = n_zm, mx2 = n_mx2;
      T wp2v[G], poldv[G];
#pragma unroll
      for (int g = 0; g < G; ++g) { wp2v[g] = n_wp2[g]; poldv[g] = n_pold[g]; }
      if (i + 1 < i_e) fetch_row(i + 1);
      const T mz = rot ? v_n * dtrdy : (v_n * rmv_n) * dtrdy;
      const T mfac = rot ? T(0.5) * v_n : (T(0.5) * v_n) * rmv_n;
      const T pdv = rot ? (v_n * pn - v_i * ps) : ((v_n * rmv_n) * pn - (v_i * rmv_i) * ps);
      const T zz = (uu * zm) * dtrdx;
      const T zfac = rot ? T(0.5) * uu : (T(0.5) * uu) * zm;
      const T ue = __shfl_down_sync(0xffffffffu, uu, 1);  // u(j+1)
      const T zme = __shfl_down_sync(0xffffffffu, zm, 1);
      const T odv = rot ? (ue * oe - uu * ow) : ((ue * zme) * oe - (uu * zm) * ow);
#pragma unroll
      for (int g = 0; g < G; ++g) {
        if (g < ng) {
          const T wp2 = wp2v[g];
          const T fl_n = mfac * waf_hflux(mz, wm1_[g], w0_[g], wp1_[g], wp2);  // face i+1
          const T pold = poldv[g];
          const T zdv = pdv * pold;
          const T p0 = rot ? ((w0_[g] + fl_[g] * ps) - fl_n * pn) + zdv
                           : w0_[g] + mx2 * (((fl_[g] * ps) - fl_n * pn) + zdv);
          const T pm2 = __shfl_up_sync(0xffffffffu, p0, 2);
          const T pm1 = __shfl_up_sync(0xffffffffu, p0, 1);
          const T pp1 = __shfl_down_sync(0xffffffffu, p0, 1);
          const T zf = zfac * waf_hflux(zz, pm2, pm1, p0, pp1);  // face between j-1 and j
          const T zfe = __shfl_down_sync(0xffffffffu, zf, 1);    // face between j and j+1
          if (out_lane) {
            const T zdv2 = odv * pold;
            out[g][r] = rot ? ((p0 + zf * ow) - zfe * oe) + zdv2 : p0 + mx2 * (((zf * ow) - zfe * oe) + zdv2);
          }
          wm1_[g] = w0_[g]; w0_[g] = wp1_[g]; wp1_[g] = wp2; fl_[g] = fl_n;
        }
      }
      v_i = v_n; rmv_i = rmv_n;
    }
  }
  }
}

// FP32 with jx even: strips of 60 output columns, two (j, j+1) per lane.  The
// one-column strips are bound by issue slots (105 instructions a point, 77 %
// of the slots); here sums, products and fused operations take both columns
// in one instruction, of the four p0 neighbours and the next flux a pair needs
// four shuffles instead of eight, and 60 of 64 columns are output instead of
// 28 of 32.  Each warp takes five of the ten fields -- ten need 250 registers,
// 4.83 instead of 5.04 ms at 1024 x 1024 x 60 but 0.339 instead of 0.271 at 256
// x 256 x 40 -- the groups of a strip run together and share the rows of
// winds and metric terms in L2, and the next row travels through shared memory
// (in registers it spills: 5.39 ms).  Three blocks an SM (154 registers): four
// with 16 bytes spilled 5.68 ms.  Every rounding is that of the one-column
// form.  Per step, one column -> two: 1024 x 1024 x 60 6.08 -> 5.04 ms, 512 x
// 512 x 60 1.62 -> 1.35, 256 x 256 x 40 0.381 -> 0.271, 202 x 157 x 45 0.220 ->
// 0.159, 100 x 100 x 30 0.098 -> 0.060.
struct HFace2 {
  bool p0, p1;  // the positive direction is upwind
  f32x2 nis, zm;  // -is, is - zamu
};
__device__ __forceinline__ HFace2 hface2(f32x2 vel, f32x2 dt) {
  HFace2 f;
  const f32x2 z = mul2(vel, dt);
  const float2 zz = unpack2(z);
  f.p0 = zz.x > 0.f;
  f.p1 = zz.y > 0.f;
  f.nis = pack2(f.p0 ? -1.f : 1.f, f.p1 ? -1.f : 1.f);
  f.zm = sub2(pack2(f.p0 ? 1.f : -1.f, f.p1 ? 1.f : -1.f), z);
  return f;
}
// WAF value between m1 and x0, n0 and n1 the upwind differences, d = x0 - m1
__device__ __forceinline__ f32x2 hflux2(const HFace2& f, float n0, float n1, f32x2 d, f32x2 m1, f32x2 x0) {
  const float2 b = unpack2(d);
  const f32x2 bb = pack2(bb_of(n0, b.x), bb_of(n1, b.y));
  return fma2(fma2(bb, f.zm, f.nis), d, add2(m1, x0));
}
constexpr int kHPairJ = 60;
constexpr int kHPThreads = 128;  // 32 and 64 the same
constexpr int kHPG = 5, kHPAhead = 1, kHPArrays = 2 * kHPG + 9;  // fields per warp, rows ahead
constexpr int kHPSmem = (kHPAhead + 1) * kHPArrays * kHPThreads * 8;
// a b, a product that no sum may absorb (the assembler fuses mul.rn.f32x2
// with an add.rn.f32x2 that follows it)
__device__ __forceinline__ f32x2 product2(f32x2 a, f32x2 b) {
  const float2 x = unpack2(a), y = unpack2(b);
  return pack2(__fmul_rn(x.x, y.x), __fmul_rn(x.y, y.y));
}
template <bool ROT>
__device__ __forceinline__ void b_waf_hpair(const View<float>& d, const int bx, const int k, const int g0) {
  constexpr int G = kHPG;
  static_assert(kNumAdvected % G == 0, "fields per group");
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int nj = d.nj, ni = d.ni, kz = d.kz;
  const unsigned pl = (unsigned)d.pl;
  const int R = d.hz_levels;
  const int nsj = (nj + kHPairJ - 1) / kHPairJ, nsi = (ni + R - 1) / R;
  const int w = bx * (blockDim.x >> 5) + wid;
  if (w >= nsj * nsi) return;  // whole warp
  const int sj = w % nsj, si = w / nsj;
  const int jl = sj * kHPairJ - 2 + 2 * lane;  // this lane's first column before wrapping
  const int j = wrapn(jl, nj);
  const bool out_lane = lane >= 1 && lane < 31 && jl < nj;
  const int i_s = si * R, i_e = min(i_s + R, ni);
  auto ld = [](const float* q) -> f32x2 { return pack2(*reinterpret_cast<const float2*>(q)); };
  const float* __restrict__ u = d.ubuf[d.cur] + (size_t)k * pl;
  const float* __restrict__ v = d.vbuf[d.cur] + (size_t)k * pl;
  const float* __restrict__ wn_ = d.wafn + (size_t)k * pl;
  const float* __restrict__ ws_ = d.wafs + (size_t)k * pl;
  const float* __restrict__ we_ = d.wafe + (size_t)k * pl;
  const float* __restrict__ ww_ = d.wafw + (size_t)k * pl;
  const f32x2 dtx = pack2(d.dtrdx_a, d.dtrdx_a), dty = pack2(d.dtrdy_a, d.dtrdy_a);
  const f32x2 half = pack2(0.5f, 0.5f), neg = pack2(-1.f, -1.f);
  auto row = [&](int i) { return (unsigned)j + (unsigned)nj * (unsigned)wrap2(i, ni); };
  {
    const float* wz[G];
    const float* pp[G];
    float* out[G];
    f32x2 w0[G], w1[G], da[G], db[G], fl[G];  // wz(i), wz(i+1), their differences, the flux of face i
#pragma unroll
    for (int g = 0; g < G; ++g) {
      wz[g] = d.wz + ((size_t)(g0 + g) * kz + k) * pl;
      pp[g] = d.fset[d.fcur][g0 + g] + (size_t)k * pl;
      out[g] = d.fset[d.fcur ^ 1][g0 + g] + (size_t)k * pl;
    }
    auto mflux = [&](const HFace2& f, f32x2 dm, f32x2 d0, f32x2 dp, f32x2 m1, f32x2 x0) {
      const float2 a = unpack2(dm), c = unpack2(dp);
      return hflux2(f, f.p0 ? a.x : c.x, f.p1 ? a.y : c.y, d0, m1, x0);
    };
    f32x2 v_i;  // v at the face below row i (times 1 / msfv, non-ROTLLR)
    {
      const unsigned r = row(i_s), r2 = row(i_s - 2), r1 = row(i_s - 1), rp = row(i_s + 1);
      v_i = ld(v + r);
      const f32x2 rm = ROT ? neg : ld(d.rmv + r);
      const f32x2 fac = ROT ? mul2(half, v_i) : mul2(mul2(half, v_i), rm);
      if (!ROT) v_i = mul2(v_i, rm);
      const HFace2 f = hface2(v_i, dty);
#pragma unroll
      for (int g = 0; g < G; ++g) {
        const f32x2 a = ld(wz[g] + r2), b = ld(wz[g] + r1);
        w0[g] = ld(wz[g] + r);
        w1[g] = ld(wz[g] + rp);
        da[g] = sub2(w0[g], b);
        db[g] = sub2(w1[g], w0[g]);
        fl[g] = mul2(fac, mflux(f, sub2(b, a), da[g], db[g], b, w0[g]));
      }
    }
    // row i's values travel kHPAhead rows ahead through the thread's own
    // slots of shared memory
    extern __shared__ float2 hp_ring[];
    float2* const slot0 = hp_ring + threadIdx.x;
    auto fetch_row = [&](int i, int st) {
      if (i < i_e) {
        float2* q = slot0 + st * (kHPArrays * kHPThreads);
        const unsigned r = row(i), rn = row(i + 1), r2 = row(i + 2);
#pragma unroll
        for (int g = 0; g < G; ++g) {
          cp_async8(q + g * kHPThreads, wz[g] + r2);
          cp_async8(q + (G + g) * kHPThreads, pp[g] + r);
        }
        q += 2 * G * kHPThreads;
        cp_async8(q, v + rn);
        cp_async8(q + kHPThreads, wn_ + r);
        cp_async8(q + 2 * kHPThreads, ws_ + r);
        cp_async8(q + 3 * kHPThreads, u + r);
        cp_async8(q + 4 * kHPThreads, we_ + r);
        cp_async8(q + 5 * kHPThreads, ww_ + r);
        cp_async8(q + 6 * kHPThreads, (ROT ? d.mu : d.rmu) + r);
        if (!ROT) {
          cp_async8(q + 7 * kHPThreads, d.rmv + rn);
          cp_async8(q + 8 * kHPThreads, d.mx2 + r);
        }
      }
      cp_async_commit();
    };
#pragma unroll
    for (int n = 0; n < kHPAhead; ++n) fetch_row(i_s + n, n);
    int rd = 0;
#pragma unroll 1
    for (int i = i_s; i < i_e; ++i) {
      const unsigned r = row(i);
      cp_async_wait<kHPAhead - 1>();
      const float2* q = slot0 + rd * (kHPArrays * kHPThreads);
      const float2* qs = q + 2 * G * kHPThreads;
      const f32x2 vr = pack2(qs[0]), pn = pack2(qs[kHPThreads]), ps = pack2(qs[2 * kHPThreads]), uu = pack2(qs[3 * kHPThreads]), oe = pack2(qs[4 * kHPThreads]),
                  ow = pack2(qs[5 * kHPThreads]), zmf = pack2(qs[6 * kHPThreads]);
      const f32x2 rmv = ROT ? neg : pack2(qs[7 * kHPThreads]), mx2 = ROT ? neg : pack2(qs[8 * kHPThreads]);
      const f32x2 uz = mul2(uu, zmf);
      const f32x2 v_n = ROT ? vr : mul2(vr, rmv), uf = ROT ? uu : uz;
      const f32x2 mfac = ROT ? mul2(half, vr) : mul2(mul2(half, vr), rmv);
      const f32x2 zfac = ROT ? mul2(half, uu) : mul2(mul2(half, uu), zmf);
      const HFace2 fm = hface2(v_n, dty), fz = hface2(uz, dtx);
      const float2 ufx = unpack2(uf);
      const f32x2 ufe = pack2(ufx.y, __shfl_down_sync(0xffffffffu, ufx.x, 1));
      const f32x2 npn = mul2(pn, neg), noe = mul2(oe, neg);
      // a b - c d: the first product is fused, as in the one-column form
      const f32x2 pdv = fma2(v_n, pn, mul2(v_i, mul2(ps, neg)));
      const f32x2 odv = fma2(ufe, oe, mul2(uf, mul2(ow, neg)));
      f32x2 wp2[G], pold[G];
#pragma unroll
      for (int g = 0; g < G; ++g) { wp2[g] = pack2(q[g * kHPThreads]); pold[g] = pack2(q[(G + g) * kHPThreads]); }
      fetch_row(i + kHPAhead, rd == 0 ? kHPAhead : rd - 1);
#pragma unroll
      for (int g = 0; g < G; ++g) {
        const f32x2 dn = sub2(wp2[g], w1[g]);
        const f32x2 fn = mul2(mfac, mflux(fm, da[g], db[g], dn, w0[g], w1[g]));  // face i+1
        const f32x2 p0 = ROT ? fma2(pdv, pold[g], fma2(fn, npn, fma2(fl[g], ps, w0[g])))
                             : fma2(mx2, fma2(pdv, pold[g], fma2(fl[g], ps, mul2(fn, npn))), w0[g]);
        w0[g] = w1[g]; w1[g] = wp2[g]; da[g] = db[g]; db[g] = dn; fl[g] = fn;
        const float2 p = unpack2(p0);
        const float pm2 = __shfl_up_sync(0xffffffffu, p.x, 1), pm1 = __shfl_up_sync(0xffffffffu, p.y, 1);
        const float pp1 = __shfl_down_sync(0xffffffffu, p.x, 1);
        const f32x2 m1 = pack2(pm1, p.x), dz = sub2(p0, m1);
        const float2 z = unpack2(dz), e = unpack2(sub2(pack2(pm1, pp1), pack2(pm2, p.y)));
        const f32x2 zf = mul2(zfac, hflux2(fz, fz.p0 ? e.x : z.y, fz.p1 ? z.x : e.y, dz, m1, p0));  // western faces
        const float2 zz = unpack2(zf);
        const f32x2 zfe = pack2(zz.y, __shfl_down_sync(0xffffffffu, zz.x, 1));
        const f32x2 zdv = product2(odv, pold[g]);  // not fused, as in the one-column form
        const f32x2 o = ROT ? add2(zdv, fma2(zfe, noe, fma2(zf, ow, p0)))
                            : fma2(mx2, add2(zdv, fma2(zf, ow, mul2(zfe, noe))), p0);
        if (out_lane) *reinterpret_cast<float2*>(out[g] + r) = unpack2(o);
      }
      v_i = v_n;
      rd = rd == kHPAhead ? 0 : rd + 1;
    }
    cp_async_wait<0>();
  }
}
template <bool ROT>
__global__ void __launch_bounds__(kHPThreads, 384 / kHPThreads) k_waf_hpair(View<float> d) {
  constexpr int NG = kNumAdvected / kHPG;
  b_waf_hpair<ROT>(d, blockIdx.x / NG, blockIdx.y, (blockIdx.x % NG) * kHPG);
}

template <class T>
__global__ void __launch_bounds__(128) k_waf_hstrip(View<T> d) {
  b_waf_hstrip<T>(d, blockIdx.x, blockIdx.y);
}

template <class T>
__global__ void __launch_bounds__(128)
    kb_waf_hstrip(const View<T>* __restrict__ views, const int4* __restrict__ tiles) {
  __shared__ View<T> sv;
  const int4 t = tiles[blockIdx.x];
  copy_view(&sv, views + t.x);
  __syncthreads();
  b_waf_hstrip<T>(sv, t.y, t.z);
}


// ---- advection: cross points -> staggered (:1343-1387) ------------------
// Writes u, v into buffer 0 so every step replays the same pointers.
template <class T>
__device__ __forceinline__ void b_stag_from_x(const View<T>& d, const int bx, const int by, const int bz) {
  int jj, ii;
  point_at<kPtBX, kPtBY>(d, bx, by, jj, ii);
  const int nj = d.nj, ni = d.ni, kz = d.kz, kk = bz;
  if (jj >= nj || ii >= ni) return;
  // 32-bit element offsets: a field holds at most 2^31 points
  const unsigned pl = (unsigned)d.pl;
  const unsigned o = (unsigned)kk * pl;
  const unsigned c = (unsigned)jj + (unsigned)nj * (unsigned)ii;
  const unsigned rowj = (unsigned)nj * (unsigned)ii;
  const T* __restrict__ ux = d.ux;
  const T* __restrict__ vx = d.vx;
  d.ubuf[0][o + c] = average4(ux[o + c] + ux[o + rowj + wm1(jj, nj)],
                              ux[o + rowj + wp1(jj, nj)] + ux[o + rowj + wm2(jj, nj)]);
  d.vbuf[0][o + c] = average4(vx[o + c] + vx[o + jj + (unsigned)nj * wm1(ii, ni)],
                              vx[o + jj + (unsigned)nj * wp1(ii, ni)] + vx[o + jj + (unsigned)nj * wm2(ii, ni)]);
  // w(k), k = 2..kz (1-based) <- wx ; level index kk = k-1 in 1..kz-1
  if (kk >= 1) {
    const T* __restrict__ wx = d.wx;
    T wv;
    if (kk == 1)
      wv = T(0.5) * (wx[c + pl] + wx[c]);
    else if (kk == kz - 1)
      wv = T(0.5) * (wx[c + (unsigned)(kz - 1) * pl] + wx[c + (unsigned)(kz - 2) * pl]);
    else
      wv = average4(wx[c + kk * pl] + wx[c + (kk - 1) * pl], wx[c + (kk + 1) * pl] + wx[c + (kk - 2) * pl]);
    d.w[c + kk * pl] = wv;
  }
}

template <class T>
__global__ void __launch_bounds__(kPtBX* kPtBY) k_stag_from_x(View<T> d) {
  b_stag_from_x<T>(d, blockIdx.x, tile_y(d), blockIdx.z);
}

// The same for FP32 storage with jx a multiple of 4 (View::stag4): each
// thread takes four consecutive columns j0 .. j0+3 of one row and level,
// with 16-byte loads and stores -- ux of columns j0-4 .. j0+7 (periodic:
// the neighbouring quads wrap whole, since jx is a multiple of 4), vx of
// rows i-2 .. i+1 and wx of levels k-2 .. k+1 -- and the expressions of
// b_stag_from_x per column: 14 vector memory instructions per four points
// instead of 60 scalar ones.
__global__ void __launch_bounds__(kPtBX* kPtBY) k_stag_from_x4(View<float> d) {
  const int nj = d.nj, ni = d.ni, kz = d.kz, kk = blockIdx.z;
  const int nq = nj >> 2;
  const int qj = blockIdx.x * kPtBX + threadIdx.x, ii = blockIdx.y * kPtBY + threadIdx.y;
  if (qj >= nq || ii >= ni) return;
  const unsigned pl = (unsigned)d.pl, o = (unsigned)kk * pl;
  const int j0 = 4 * qj;
  const unsigned row = (unsigned)nj * (unsigned)ii;
  const unsigned c = (unsigned)j0 + row;
  auto ld4 = [](const float* p) { return *reinterpret_cast<const float4*>(p); };
  auto st4 = [](float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; };
  auto f = [](float a, float b, float cc, float dd) { return 0.5625f * (a + b) - 0.0625f * (cc + dd); };
  {  // u(j) <- ux(j-2 .. j+1)
    const float* ux = d.ux + o + row;
    const float4 A = ld4(ux + (j0 == 0 ? nj - 4 : j0 - 4)), B = ld4(ux + j0), C = ld4(ux + (j0 + 4 == nj ? 0 : j0 + 4));
    st4(d.ubuf[0] + o + c, make_float4(f(B.x, A.w, B.y, A.z), f(B.y, B.x, B.z, A.w), f(B.z, B.y, B.w, B.x),
                                       f(B.w, B.z, C.x, B.y)));
  }
  {  // v(i) <- vx(i-2 .. i+1)
    const float* vx = d.vx + o + j0;
    const float4 P = ld4(vx + row), M1 = ld4(vx + (unsigned)nj * wm1(ii, ni)), P1 = ld4(vx + (unsigned)nj * wp1(ii, ni)),
                 M2 = ld4(vx + (unsigned)nj * wm2(ii, ni));
    st4(d.vbuf[0] + o + c, make_float4(f(P.x, M1.x, P1.x, M2.x), f(P.y, M1.y, P1.y, M2.y), f(P.z, M1.z, P1.z, M2.z),
                                       f(P.w, M1.w, P1.w, M2.w)));
  }
  if (kk >= 1) {  // w(k), k = 2..kz (1-based) <- wx; level index kk = k-1 in 1..kz-1
    const float* wx = d.wx + c;
    float4 wv;
    if (kk == 1 || kk == kz - 1) {
      const float4 a = ld4(wx + (unsigned)kk * pl), b = ld4(wx + (unsigned)(kk - 1) * pl);
      wv = make_float4(0.5f * (a.x + b.x), 0.5f * (a.y + b.y), 0.5f * (a.z + b.z), 0.5f * (a.w + b.w));
    } else {
      const float4 a = ld4(wx + (unsigned)kk * pl), b = ld4(wx + (unsigned)(kk - 1) * pl);
      const float4 e = ld4(wx + (unsigned)(kk + 1) * pl), g = ld4(wx + (unsigned)(kk - 2) * pl);
      wv = make_float4(f(a.x, b.x, e.x, g.x), f(a.y, b.y, e.y, g.y), f(a.z, b.z, e.z, g.z), f(a.w, b.w, e.w, g.w));
    }
    st4(d.w + c + (unsigned)kk * pl, wv);
  }
}

template <class T>
__global__ void __launch_bounds__(kPtBX* kPtBY)
    kb_stag_from_x(const View<T>* __restrict__ views, const int4* __restrict__ tiles) {
  __shared__ View<T> sv;
  const int4 t = tiles[blockIdx.x];
  copy_view(&sv, views + t.x);
  __syncthreads();
  b_stag_from_x<T>(sv, t.y, t.z, t.w);
}


// ---- post-diagnostics (:355-391), one thread per point -------------------
// The threads of the lowest level also form the surface pressure, from tvirt
// of the two lowest levels.  One thread per column marched down the levels
// with one level of loads in flight: 100 x 100 x 30 FP32 33 -> 8 us, FP64 88 ->
// 46, 256 x 256 x 40 FP32 66 -> 31; 512 x 512 x 60 the same 0.145 ms.
template <class T>
__device__ __forceinline__ void b_postdiag(const View<T>& d, const int bx, const int by, const int bz) {
  int jj, ii;
  point_at<kPtBX, kPtBY>(d, bx, by, jj, ii);
  const int nj = d.nj, ni = d.ni, kz = d.kz;
  if (jj >= nj || ii >= ni) return;
  const size_t pl = d.pl;
  const size_t c = jj + (size_t)nj * ii;
  const size_t q = c + (size_t)bz * pl;
  const T pai = d.pai[q];
  const T tvk = mul_rn(d.tetav[q], pai);  // rounded products, also inside the lapse rate below
  d.tvirt[q] = tvk;
  const T qv = d.q[0][q], qc = d.q[1][q], qi = d.q[2][q], qr = d.q[3][q], qs = d.q[4][q];
  const T t = ddiv(tvk, (((T(1) + T(kEp1) * qv) - qc) - qi) - qr - qs);
  d.t[q] = t;
  const T p = pow_cpovr(pai) * T(kP00);
  d.p[q] = p;
  d.rho[q] = ddiv(p, T(kRgas) * t);
  d.qsat[q] = pfwsat(t, p);
  if (bz != kz - 1) return;
  const T tv_km1 = mul_rn(d.tetav[q - pl], d.pai[q - pl]);
  const T z = d.zeta[q], zm = d.zeta[q - pl];
  const T zdgz = z * T(kEgrav);
  T lrt = (tv_km1 - tvk) / (zm - z);
  lrt = T(0.65) * lrt - T(0.35) * T(kLrate);
  const T tv = tvk - (T(0.5) * z) * lrt;
  d.ps[c] = p * dexp(zdgz / (T(kRgas) * tv));
}

template <class T>
__global__ void __launch_bounds__(kPtBX* kPtBY) k_postdiag(View<T> d) {
  b_postdiag<T>(d, blockIdx.x, tile_y(d), blockIdx.z);
}

template <class T>
__global__ void __launch_bounds__(kPtBX* kPtBY)
    kb_postdiag(const View<T>* __restrict__ views, const int4* __restrict__ tiles) {
  __shared__ View<T> sv;
  const int4 t = tiles[blockIdx.x];
  copy_view(&sv, views + t.x);
  __syncthreads();
  b_postdiag<T>(sv, t.y, t.z, t.w);
}


// ---- diagnostics: max/min ps, u, v (:395-411) and FP64 column sums ------
// partial record per block: maxps minps maxu minu maxv minv mass energy nonfinite
constexpr int kDiagN = 9;
template <class T>
__global__ void __launch_bounds__(kColBX* kColBY) k_diag_partial(View<T> d) {
  __shared__ double sh[kDiagN][kColBX * kColBY];
  const int tid = threadIdx.x + kColBX * threadIdx.y;
  int jj = blockIdx.x * kColBX + threadIdx.x;
  int ii = blockIdx.y * kColBY + threadIdx.y;
  const int nj = d.nj, ni = d.ni, kz = d.kz;
  double r[kDiagN] = {-INFINITY, INFINITY, -INFINITY, INFINITY, -INFINITY, INFINITY, 0.0, 0.0, 0.0};
  if (jj < nj && ii < ni) {
    const size_t pl = d.pl;
    const size_t c = jj + (size_t)nj * ii;
    const double ps = (double)d.ps[c];
    if (!isfinite(ps)) r[8] = 1.0;
    else { r[0] = ps; r[1] = ps; }
    const T* __restrict__ u = d.ubuf[d.cur];
    const T* __restrict__ v = d.vbuf[d.cur];
    double mass = 0.0, en = 0.0;
    for (int kk = 0; kk < kz; ++kk) {
      const size_t q = c + (size_t)kk * pl;
      const double uu = (double)u[q], vv = (double)v[q];
      r[2] = fmax(r[2], uu); r[3] = fmin(r[3], uu);
      r[4] = fmax(r[4], vv); r[5] = fmin(r[5], vv);
      const double rdz = (double)d.rho[q] * (double)d.dz[q];
      const double wm = 0.5 * ((double)d.w[q] + (double)d.w[q + pl]);
      mass += rdz;
      en += rdz * (kCvd * (double)d.t[q] + kEgrav * (double)d.zeta[q] + 0.5 * (uu * uu + vv * vv + wm * wm));
    }
    r[6] = mass; r[7] = en;
  }
  for (int n = 0; n < kDiagN; ++n) sh[n][tid] = r[n];
  __syncthreads();
  for (int st = (kColBX * kColBY) / 2; st > 0; st >>= 1) {
    if (tid < st) {
      sh[0][tid] = fmax(sh[0][tid], sh[0][tid + st]); sh[1][tid] = fmin(sh[1][tid], sh[1][tid + st]);
      sh[2][tid] = fmax(sh[2][tid], sh[2][tid + st]); sh[3][tid] = fmin(sh[3][tid], sh[3][tid + st]);
      sh[4][tid] = fmax(sh[4][tid], sh[4][tid + st]); sh[5][tid] = fmin(sh[5][tid], sh[5][tid + st]);
      sh[6][tid] += sh[6][tid + st]; sh[7][tid] += sh[7][tid + st]; sh[8][tid] += sh[8][tid + st];
    }
    __syncthreads();
  }
  if (tid == 0) {
    const size_t b = blockIdx.x + (size_t)gridDim.x * blockIdx.y;
    for (int n = 0; n < kDiagN; ++n) d.dpart[b * kDiagN + n] = sh[n][0];
  }
}

__global__ void __launch_bounds__(256) k_diag_final(const double* __restrict__ part, int nparts, double* res) {
  __shared__ double sh[kDiagN][256];
  const int tid = threadIdx.x;
  double r[kDiagN] = {-INFINITY, INFINITY, -INFINITY, INFINITY, -INFINITY, INFINITY, 0.0, 0.0, 0.0};
  for (int b = tid; b < nparts; b += 256) {  // fixed assignment: deterministic sums
    const double* p = part + (size_t)b * kDiagN;
    r[0] = fmax(r[0], p[0]); r[1] = fmin(r[1], p[1]); r[2] = fmax(r[2], p[2]); r[3] = fmin(r[3], p[3]);
    r[4] = fmax(r[4], p[4]); r[5] = fmin(r[5], p[5]); r[6] += p[6]; r[7] += p[7]; r[8] += p[8];
  }
  for (int n = 0; n < kDiagN; ++n) sh[n][tid] = r[n];
  __syncthreads();
  for (int st = 128; st > 0; st >>= 1) {
    if (tid < st) {
      sh[0][tid] = fmax(sh[0][tid], sh[0][tid + st]); sh[1][tid] = fmin(sh[1][tid], sh[1][tid + st]);
      sh[2][tid] = fmax(sh[2][tid], sh[2][tid + st]); sh[3][tid] = fmin(sh[3][tid], sh[3][tid + st]);
      sh[4][tid] = fmax(sh[4][tid], sh[4][tid + st]); sh[5][tid] = fmin(sh[5][tid], sh[5][tid + st]);
      sh[6][tid] += sh[6][tid + st]; sh[7][tid] += sh[7][tid + st]; sh[8][tid] += sh[8][tid + st];
    }
    __syncthreads();
  }
  if (tid == 0)
    for (int n = 0; n < kDiagN; ++n) res[n] = sh[n][0];
}

// =========================================================================
// Launchers.  Each returns the number of kernels it started.
// =========================================================================
inline thread_local KernelTimer* g_timer = nullptr;
void set_timer(KernelTimer* t) { g_timer = t; }
#define MOLOCH_LAUNCH(KIND, STREAM, ...)                        \
  do {                                                          \
    if (g_timer) g_timer->mark((KIND), (STREAM), true);         \
    __VA_ARGS__;                                                \
    if (g_timer) g_timer->mark((KIND), (STREAM), false);        \
  } while (0)
template <class T>
inline FieldPtrs<T> field_set(const View<T>& d, int set) {
  FieldPtrs<T> fp;
  for (int n = 0; n < kNumAdvected; ++n) fp.f[n] = d.fset[set][n];
  return fp;
}

inline dim3 col_grid(int nj, int ni, int z = 1) {
  return dim3((nj + kColBX - 1) / kColBX, (ni + kColBY - 1) / kColBY, z);
}
template <class T>
dim3 pt_grid(const View<T>& d, int nz) {
  if (in_order(d)) return dim3((unsigned)((d.pl + kPtBX * kPtBY - 1) / (kPtBX * kPtBY)), 1, nz);
  return dim3((d.nj + kPtBX - 1) / kPtBX, (d.ni + kPtBY - 1) / kPtBY, nz);
}

template <class T>
int launch_prediag(const View<T>& d, cudaStream_t st, const PhaseFlags& fl) {
  MOLOCH_LAUNCH(KK_PREDIAG, st, k_prediag<T><<<pt_grid(d, d.kz), dim3(kPtBX, kPtBY), 0, st>>>(d, fl.filterpai, fl.filtertheta));
  return 1;
}

// the staged column kernel runs when asked for (kmarch bit 32) on an FP32
// domain whose tensor maps were built
template <class T>
inline bool column_tw_ok(const View<T>& d) {
  return sizeof(T) == 4 && (d.kmarch & 32) && d.cmaps != nullptr;
}
// the one-thread column solve (variants: k_sound_column)
template <class T>
void launch_sound_column(const View<T>& d, cudaStream_t st, int ns, int last, int defer_pai) {
  if constexpr (sizeof(T) == 8) {
    // FP64 columns split over a block (k_sound_column_split) while the march
    // leaves SMs idle.  us per launch, march | 32 columns a block | 8:
    //   lean   37 | 19 | 15 at 24 x 20 x 12, 57 | 26 | 24 at 53 x 47 x 21, 77 | 35 | 35
    //          at 64 x 64 x 30, 81 | 53 | 78 at 100 x 100 x 30, 170 | 154 | 273 at
    //          203 x 157 x 45, 304 | 269 | 458 at 199 x 200 x 60, 386 | 392 | 716 at
    //          256 x 256 x 60
    //   exact  47 | 23 | 16, 74 | 34 | 31, 104 | 46 | 47, 104 | 82 | 106; 170 | 178 |
    //          240 at 150 x 140 x 40
    // Deeper columns take fewer to a block (48 KB of shared memory), march | 16
    // columns a block | 8:
    //   lean   178 | 60 | 52 at 24 x 20 x 72, 181 | 66 | 64 at 53 x 47 x 72, 325 | 120 |
    //          111 at 54 x 55 x 128, 205 | 166 | 241 at 126 x 126 x 72, 362 | 289 | 422
    //          at 126 x 126 x 128, 286 | 305 | 434 at 160 x 160 x 96; 729 | - | 205 at
    //          53 x 47 x 256
    //   exact  243 | 76 | 62, 239 | 93 | 84, 419 | 167 | 147, 254 | 255 | 337, 445 | 445 |
    //          591, 463 | 509 | 678; 832 | - | 279
    const auto split = [&](auto k, int cols) {
      MOLOCH_LAUNCH(KK_SOUND_COLUMN, st,
                    k<<<((unsigned)d.pl + cols - 1) / cols, kSplitThreads, split_smem_bytes(cols, d.kz), st>>>(d, ns, last,
                                                                                                            defer_pai));
    };
    if (d.pl <= 3000 && d.kz <= 256) return split(k_sound_column_split<8>, 8);
    if (d.pl <= (kLean<T> ? 40000 : 16000) && d.kz <= 64) return split(k_sound_column_split<32>, 32);
    if (d.pl <= 16000 && d.kz <= 128) return split(k_sound_column_split<16>, 16);
  }
  const int bj = (d.nj + kColBX - 1) / kColBX;
  const int rows = bj * ((d.ni + kColBY - 1) / kColBY) < 2 * sm_count() ? 1 : kColBY;
  const dim3 cb(kColBX, rows), cg(bj, (d.ni + rows - 1) / rows);
  if constexpr (sizeof(T) == 4) {
    if (d.pl <= 4 * kColBX * kColBY * sm_count()) {
      MOLOCH_LAUNCH(KK_SOUND_COLUMN, st, k_sound_column<T, 2><<<cg, cb, 0, st>>>(d, ns, last, defer_pai));
      return;
    }
  }
  MOLOCH_LAUNCH(KK_SOUND_COLUMN, st, k_sound_column<T, 1><<<cg, cb, 0, st>>>(d, ns, last, defer_pai));
}

// persistent CTAs of the staged column solve over ntiles tiles
inline int column_tw_grid(int ntiles) {
  const int slots = TwCfg<0>::ctas * sm_count();
  return ntiles < slots ? ntiles : slots;
}
template <class T>
inline int column_tw_grid(const View<T>& d) {
  const int w = d.twide;
  return column_tw_grid(((d.nj + 32 * w - 1) / (32 * w)) * ((d.ni * w + kTwWarps - 1) / kTwWarps));
}

// one sound() call: nsound substeps; flips d.cur once per substep, twice
// with the fused divergence/damping kernel (kmarch bit 16)
template <class T>
int launch_sound(View<T>& d, cudaStream_t st, const PhaseFlags& fl) {
  int n = 0;
  const dim3 pb(kPtBX, kPtBY), pg = pt_grid(d, d.kz);
  const dim3 kg = pt_grid(d, (d.kz + kKC - 1) / kKC);  // k-marching: chunks of kKC levels
  for (int ns = 1; ns <= fl.nsound; ++ns) {
    const int last = ns == fl.nsound;
    // the fused strips recompute the divergence of a rim: bound by the FP64
    // pipe, the contracting FP64 build runs the two kernels instead (256 x
    // 256 x 60: 7.0 against 3.2 ms per step)
    bool fused = false;
    if constexpr (!kLean<T>) {
      if (d.kmarch & 16) {
        const int nstrips = ((d.nj + kDDJ - 1) / kDDJ) * ((d.ni + kDDR - 1) / kDDR);
        const dim3 g2((nstrips + 3) / 4, (d.kz + kDDLevels - 1) / kDDLevels);
        bool quads = false;
        if constexpr (sizeof(T) == 4) {
          if ((d.kmarch & 512) && d.nj % 4 == 0 && d.kz <= kDQMaxKz) {  // four columns per thread
            const int g4 = sm_count(), sm4 = dq_smem_bytes(d.kz);
            const dim3 b4(32, kDQRows + 3);
            dq_attributes();
            if (d.rotllr && last)
              MOLOCH_LAUNCH(KK_SOUND_DIVDAMP, st, k_divdamp_quad<true, 1><<<g4, b4, sm4, st>>>(d));
            else if (d.rotllr)
              MOLOCH_LAUNCH(KK_SOUND_DIVDAMP, st, k_divdamp_quad<true, 0><<<g4, b4, sm4, st>>>(d));
            else if (last)
              MOLOCH_LAUNCH(KK_SOUND_DIVDAMP, st, k_divdamp_quad<false, 1><<<g4, b4, sm4, st>>>(d));
            else
              MOLOCH_LAUNCH(KK_SOUND_DIVDAMP, st, k_divdamp_quad<false, 0><<<g4, b4, sm4, st>>>(d));
            quads = true;
          }
        }
        if (quads) {
        } else if (d.kmarch & 512)  // kDDLevels levels per warp
          MOLOCH_LAUNCH(KK_SOUND_DIVDAMP, st, k_divdamp_strip_nl<T><<<g2, 128, 0, st>>>(d, kDDR));
        else
          MOLOCH_LAUNCH(KK_SOUND_DIVDAMP, st, k_divdamp_strip<T><<<dim3((nstrips + 3) / 4, d.kz), 128, 0, st>>>(d, kDDR));
        d.cur ^= 1;  // the damped u, v are in the other buffer
        ++n;
        fused = true;
      }
    }
    if (!fused) {
      if (d.kmarch & 1)
        MOLOCH_LAUNCH(KK_SOUND_DIV, st, k_sound_div_km<T><<<kg, pb, 0, st>>>(d));
      else
        MOLOCH_LAUNCH(KK_SOUND_DIV, st, k_sound_div<T><<<pg, pb, 0, st>>>(d));
      if (d.kmarch & 2)
        MOLOCH_LAUNCH(KK_SOUND_DAMP, st, k_sound_damp_km<T><<<kg, pb, 0, st>>>(d));
      else
        MOLOCH_LAUNCH(KK_SOUND_DAMP, st, k_sound_damp<T><<<pg, pb, 0, st>>>(d));
      n += 2;
    }
    if (fl.divfilter) {
      launch_sound_column<T>(d, st, ns, last, 1);
      MOLOCH_LAUNCH(KK_LAP_FILTER, st, k_lap_filter<T><<<pg, pb, 0, st>>>(d));
      MOLOCH_LAUNCH(KK_PAI_UPDATE, st, k_pai_update<T><<<pg, pb, 0, st>>>(d));
      n += 3;
    } else {
      bool staged = false;
      if constexpr (sizeof(T) == 4) {
        if (column_tw_ok(d)) {
          const ColumnMaps& cm = static_cast<const ColumnMaps*>(d.cmaps)[d.fcur];
          const int grid = column_tw_grid(d);
          if (last)
            MOLOCH_LAUNCH(KK_SOUND_COLUMN_TW, st,
                          k_sound_column_tw<T, 1><<<grid, TwCfg<1>::threads, TwCfg<1>::smem, st>>>(d, cm, ns));
          else
            MOLOCH_LAUNCH(KK_SOUND_COLUMN_TW, st,
                          k_sound_column_tw<T, 0><<<grid, TwCfg<0>::threads, TwCfg<0>::smem, st>>>(d, cm, ns));
          staged = true;
        }
      }
      if (!staged) launch_sound_column<T>(d, st, ns, last, 0);
      ++n;
    }
    bool pairs = false;
    if constexpr (sizeof(T) == 4) {
      if ((d.kmarch & 8) && (d.kmarch & 64) && d.nj % 4 == 0) {  // four columns per thread
        const dim3 g4((d.nj / 4 + 31) / 32, (d.ni + kQuadY - 1) / kQuadY, d.kz);
        MOLOCH_LAUNCH(KK_SOUND_MOMENTUM, st, k_momentum_quad<<<g4, dim3(32, kQuadY), 0, st>>>(d));
        pairs = true;
      } else if ((d.kmarch & 8) && (d.kmarch & 64) && d.nj % 2 == 0) {  // two columns per lane
        const int nstrips = ((d.nj + 1 + kMom2J - 1) / kMom2J) * ((d.ni + d.srows - 1) / d.srows);
        MOLOCH_LAUNCH(KK_SOUND_MOMENTUM, st,
                      k_momentum_strip2<<<dim3((nstrips + 3) / 4, d.kz), 128, 0, st>>>(d, d.srows));
        pairs = true;
      }
    }
    if (pairs) {
    } else if (d.kmarch & 8) {
      const int nstrips = ((d.nj + kMomJ - 1) / kMomJ) * ((d.ni + d.srows - 1) / d.srows);
      MOLOCH_LAUNCH(KK_SOUND_MOMENTUM, st, k_momentum_strip<T><<<dim3((nstrips + 3) / 4, d.kz), 128, 0, st>>>(d, d.srows));
    } else if (d.kmarch & 4)
      MOLOCH_LAUNCH(KK_SOUND_MOMENTUM, st, k_sound_momentum_km<T><<<kg, pb, 0, st>>>(d));
    else
      MOLOCH_LAUNCH(KK_SOUND_MOMENTUM, st, k_sound_momentum<T><<<pg, pb, 0, st>>>(d));
    ++n;
    d.cur ^= 1;
  }
  return n;
}

// launch of the vertical WAF with the View's fields per thread
template <class T>
void launch_waf_vertical(const View<T>& d, cudaStream_t st) {
  const int ng = kNumAdvected / d.vfields;
  const dim3 vb(kColBX, kColBY);
  const dim3 vg = in_order(d) ? dim3((unsigned)((d.pl + kColBX * kColBY - 1) / (kColBX * kColBY)) * ng)
                              : dim3(((d.nj + kColBX - 1) / kColBX) * ng, (d.ni + kColBY - 1) / kColBY);
  // jx even: rows of column pairs (8-byte loads); faster at every size
  if constexpr (sizeof(T) == 4) {
    if (d.vfields == 1 && d.nj % 2 == 0) {
      const dim3 pg((d.nj + 2 * kColBX - 1) / (2 * kColBX) * kNumAdvected, vg.y);
      MOLOCH_LAUNCH(KK_WAF_VERTICAL, st, k_waf_vertical_pair<<<pg, vb, kVPSmem, st>>>(d));
      return;
    }
  }
  switch (d.vfields) {
    case 2: MOLOCH_LAUNCH(KK_WAF_VERTICAL, st, k_waf_vertical<T, 2><<<vg, vb, 0, st>>>(d)); break;
    case 5: MOLOCH_LAUNCH(KK_WAF_VERTICAL, st, k_waf_vertical<T, 5><<<vg, vb, 0, st>>>(d)); break;
    case 10: MOLOCH_LAUNCH(KK_WAF_VERTICAL, st, k_waf_vertical<T, 10><<<vg, vb, 0, st>>>(d)); break;
    default: MOLOCH_LAUNCH(KK_WAF_VERTICAL, st, k_waf_vertical<T, 1><<<vg, vb, 0, st>>>(d)); break;
  }
}

template <class T>
void blaunch_waf_vertical(const Batch<T>& b, const View<T>* views, cudaStream_t st) {
  const int n = b.ntiles[TK_VERTICAL];
  const int4* tl = b.tiles[TK_VERTICAL];
  const dim3 vb(kColBX, kColBY);
  switch (b.vfields) {
    case 2: MOLOCH_LAUNCH(KK_WAF_VERTICAL, st, kb_waf_vertical<T, 2><<<n, vb, 0, st>>>(views, tl)); break;
    case 5: MOLOCH_LAUNCH(KK_WAF_VERTICAL, st, kb_waf_vertical<T, 5><<<n, vb, 0, st>>>(views, tl)); break;
    case 10: MOLOCH_LAUNCH(KK_WAF_VERTICAL, st, kb_waf_vertical<T, 10><<<n, vb, 0, st>>>(views, tl)); break;
    default: MOLOCH_LAUNCH(KK_WAF_VERTICAL, st, kb_waf_vertical<T, 1><<<n, vb, 0, st>>>(views, tl)); break;
  }
}


// one advection() call; the advected fields move to the other buffer set
template <class T>
int launch_advection(View<T>& d, cudaStream_t st) {
  const dim3 pb(kPtBX, kPtBY), pg = pt_grid(d, d.kz);
  const dim3 hg((d.nj + 31) / 32, (d.ni + 7) / 8, (d.kz + d.hz_levels - 1) / d.hz_levels);
  launch_waf_vertical<T>(d, st);  // forms ux, vx, wx from u, v, w as well
  bool pairs = false;  // jx even: 8-byte loads of column pairs; faster at every size
  if constexpr (sizeof(T) == 4) {
    pairs = d.hz_levels >= 16 && d.nj % 2 == 0;
    if (pairs) {
      const int np = ((d.nj + kHPairJ - 1) / kHPairJ) * ((d.ni + d.hz_levels - 1) / d.hz_levels);
      const dim3 g((np + kHPThreads / 32 - 1) / (kHPThreads / 32) * (kNumAdvected / kHPG), d.kz);
      if (d.rotllr) MOLOCH_LAUNCH(KK_WAF_HORIZONTAL, st, k_waf_hpair<true><<<g, kHPThreads, kHPSmem, st>>>(d));
      else MOLOCH_LAUNCH(KK_WAF_HORIZONTAL, st, k_waf_hpair<false><<<g, kHPThreads, kHPSmem, st>>>(d));
    }
  }
  if (pairs) {
  } else if (d.hz_levels >= 16) {  // warp strips of hz_levels rows
    const int nstrips = ((d.nj + kStripJ - 1) / kStripJ) * ((d.ni + d.hz_levels - 1) / d.hz_levels);
    // one warp a block, which balances a few hundred strips over the SMs: FP64
    // at 100 x 100 x 30 0.547 (four) -> 0.430 ms per step; larger grids and FP32
    // the same
    MOLOCH_LAUNCH(KK_WAF_HORIZONTAL, st, k_waf_hstrip<T><<<dim3(nstrips, d.kz), 32, 0, st>>>(d));
  } else {
    MOLOCH_LAUNCH(KK_WAF_HORIZONTAL, st, k_waf_horizontal<T><<<hg, dim3(32, 8), 0, st>>>(d));
  }
  d.fcur ^= 1;
  d.bind_fields();
  bool vec = false;
  if constexpr (sizeof(T) == 4) {
    if (d.stag4 && d.nj % 4 == 0) {  // four columns per thread
      const dim3 g4((d.nj / 4 + kPtBX - 1) / kPtBX, (d.ni + kPtBY - 1) / kPtBY, d.kz);
      MOLOCH_LAUNCH(KK_STAG_FROM_X, st, k_stag_from_x4<<<g4, pb, 0, st>>>(d));
      vec = true;
    }
  }
  if (!vec) MOLOCH_LAUNCH(KK_STAG_FROM_X, st, k_stag_from_x<T><<<pg, pb, 0, st>>>(d));
  d.cur = 0;
  return 3;
}

template <class T>
int launch_postdiag(View<T>& d, cudaStream_t st, const PhaseFlags& fl, const T* zk, const T* zkm1) {
  int n = 0;
  const dim3 pb(kPtBX, kPtBY), pg = pt_grid(d, d.kz);
  const size_t bytes = sizeof(T) * (size_t)d.pl * d.kz;
  if (fl.filterpai) {
    MOLOCH_LAUNCH(KK_FILTER_INCREMENT, st, k_filter_increment<T><<<pg, pb, 0, st>>>(d, 0));
    cudaMemcpyAsync(d.pai, d.fscr, bytes, cudaMemcpyDeviceToDevice, st);
    ++n;
  }
  if (fl.filtertheta) {
    MOLOCH_LAUNCH(KK_FILTER_INCREMENT, st, k_filter_increment<T><<<pg, pb, 0, st>>>(d, 1));
    cudaMemcpyAsync(d.tetav, d.fscr, bytes, cudaMemcpyDeviceToDevice, st);
    ++n;
  }
  MOLOCH_LAUNCH(KK_POSTDIAG, st, k_postdiag<T><<<pg, pb, 0, st>>>(d));
  return n + 1;
}

template <class T>
int launch_diag(const View<T>& d, cudaStream_t st) {
  const dim3 g = col_grid(d.nj, d.ni);
  MOLOCH_LAUNCH(KK_DIAG, st, k_diag_partial<T><<<g, dim3(kColBX, kColBY), 0, st>>>(d));
  MOLOCH_LAUNCH(KK_DIAG, st, k_diag_final<<<1, 256, 0, st>>>(d.dpart, (int)(g.x * g.y), d.dres));
  return 2;
}

// ---- batched launchers (ensembles) --------------------------------------
// One launch per phase covers every member; cur / fcur track the u/v buffer
// and field-set parities exactly as the single-domain launchers do.
template <class T>
int blaunch_step(const Batch<T>& b, cudaStream_t st, const PhaseFlags& fl, int& cur, int& fcur) {
  int n = 0;
  const dim3 pb(kPtBX, kPtBY), cb(kColBX, kColBY), hb(32, 8);
  auto V = [&]() { return b.views[cur][fcur]; };
  const int4* PT = b.tiles[TK_POINT];
  const int4* CO = b.tiles[TK_COLUMN];
  const int4* HZ = b.tiles[TK_HORIZONTAL];
  const int4* KC = b.tiles[TK_CHUNK];
  const int nkc = b.ntiles[TK_CHUNK];
  const int npt = b.ntiles[TK_POINT], nco = b.ntiles[TK_COLUMN];
  const int nhz = b.ntiles[TK_HORIZONTAL];
  MOLOCH_LAUNCH(KK_PREDIAG, st, kb_prediag<T><<<npt, pb, 0, st>>>(V(), PT, fl.filterpai, fl.filtertheta));
  ++n;
  for (int a = 0; a < fl.nadv; ++a) {
    for (int ns = 1; ns <= fl.nsound; ++ns) {
      const int last = ns == fl.nsound;
      bool fused = false;
      if constexpr (!kLean<T>) {
        if (b.kmarch & 16) {
          if (b.kmarch & 512)  // two levels per warp
            MOLOCH_LAUNCH(KK_SOUND_DIVDAMP, st,
                          kb_divdamp_strip_nl<T><<<b.ntiles[TK_DSTRIP2], 128, 0, st>>>(V(), b.tiles[TK_DSTRIP2], kDDR));
          else
            MOLOCH_LAUNCH(KK_SOUND_DIVDAMP, st,
                          kb_divdamp_strip<T><<<b.ntiles[TK_DSTRIP], 128, 0, st>>>(V(), b.tiles[TK_DSTRIP], kDDR));
          cur ^= 1;  // the damped u, v are in the other buffer
          --n;
          fused = true;
        }
      }
      if (!fused) {
        if (b.kmarch & 1)
          MOLOCH_LAUNCH(KK_SOUND_DIV, st, kb_sound_div_km<T><<<nkc, pb, 0, st>>>(V(), KC));
        else
          MOLOCH_LAUNCH(KK_SOUND_DIV, st, kb_sound_div<T><<<npt, pb, 0, st>>>(V(), PT));
        if (b.kmarch & 2)
          MOLOCH_LAUNCH(KK_SOUND_DAMP, st, kb_sound_damp_km<T><<<nkc, pb, 0, st>>>(V(), KC));
        else
          MOLOCH_LAUNCH(KK_SOUND_DAMP, st, kb_sound_damp<T><<<npt, pb, 0, st>>>(V(), PT));
      }
      if (fl.divfilter) {
        MOLOCH_LAUNCH(KK_SOUND_COLUMN, st, kb_sound_column<T><<<nco, cb, 0, st>>>(V(), CO, ns, last, 1));
        MOLOCH_LAUNCH(KK_LAP_FILTER, st, kb_lap_filter<T><<<npt, pb, 0, st>>>(V(), PT));
        MOLOCH_LAUNCH(KK_PAI_UPDATE, st, kb_pai_update<T><<<npt, pb, 0, st>>>(V(), PT));
        n += 2;
      } else {
        bool staged = false;
        if constexpr (sizeof(T) == 4) {
          if ((b.kmarch & 32) && b.cmaps) {
            // the staged column solve over the tiles of the members with
            // tensor maps, the one-thread kernel over the others
            const int ntw = b.ntiles[TK_COLTW], nrest = b.ntiles[TK_COLREST];
            const ColumnMaps* cms = static_cast<const ColumnMaps*>(b.cmaps);
            if (ntw > 0) {
              const int grid = column_tw_grid(ntw);
              if (last)
                MOLOCH_LAUNCH(KK_SOUND_COLUMN, st,
                              kb_sound_column_tw<T, 1><<<grid, TwCfg<1>::threads, TwCfg<1>::smem, st>>>(
                                  V(), cms, b.tiles[TK_COLTW], ntw, fcur, ns, b.kerr, b.spin));
              else
                MOLOCH_LAUNCH(KK_SOUND_COLUMN, st,
                              kb_sound_column_tw<T, 0><<<grid, TwCfg<0>::threads, TwCfg<0>::smem, st>>>(
                                  V(), cms, b.tiles[TK_COLTW], ntw, fcur, ns, b.kerr, b.spin));
            }
            if (nrest > 0) {
              MOLOCH_LAUNCH(KK_SOUND_COLUMN, st,
                            kb_sound_column<T><<<nrest, cb, 0, st>>>(V(), b.tiles[TK_COLREST], ns, last, 0));
              if (ntw > 0) ++n;
            }
            staged = true;
          }
        }
        if (!staged) MOLOCH_LAUNCH(KK_SOUND_COLUMN, st, kb_sound_column<T><<<nco, cb, 0, st>>>(V(), CO, ns, last, 0));
      }
      if (b.kmarch & 8)
        MOLOCH_LAUNCH(KK_SOUND_MOMENTUM, st,
                      kb_momentum_strip<T><<<b.ntiles[TK_MSTRIP], 128, 0, st>>>(V(), b.tiles[TK_MSTRIP], b.mrows));
      else if (b.kmarch & 4)
        MOLOCH_LAUNCH(KK_SOUND_MOMENTUM, st, kb_sound_momentum_km<T><<<nkc, pb, 0, st>>>(V(), KC));
      else
        MOLOCH_LAUNCH(KK_SOUND_MOMENTUM, st, kb_sound_momentum<T><<<npt, pb, 0, st>>>(V(), PT));
      n += 4;
      cur ^= 1;
    }
    blaunch_waf_vertical<T>(b, V(), st);
    if (b.hstrip)
      MOLOCH_LAUNCH(KK_WAF_HORIZONTAL, st, kb_waf_hstrip<T><<<nhz, 128, 0, st>>>(V(), HZ));
    else
      MOLOCH_LAUNCH(KK_WAF_HORIZONTAL, st, kb_waf_horizontal<T><<<nhz, hb, 0, st>>>(V(), HZ));
    fcur ^= 1;
    MOLOCH_LAUNCH(KK_STAG_FROM_X, st, kb_stag_from_x<T><<<npt, pb, 0, st>>>(V(), PT));
    cur = 0;
    n += 3;
  }
  MOLOCH_LAUNCH(KK_POSTDIAG, st, kb_postdiag<T><<<npt, pb, 0, st>>>(V(), PT));
  return n + 1;
}

// the advection phase alone, for the ensemble autotuner
template <class T>
int blaunch_advection(const Batch<T>& b, cudaStream_t st, int& cur, int& fcur) {
  const dim3 pb(kPtBX, kPtBY), cb(kColBX, kColBY), hb(32, 8);
  blaunch_waf_vertical<T>(b, b.views[cur][fcur], st);
  if (b.hstrip)
    MOLOCH_LAUNCH(KK_WAF_HORIZONTAL, st, kb_waf_hstrip<T><<<b.ntiles[TK_HORIZONTAL], 128, 0, st>>>(b.views[cur][fcur], b.tiles[TK_HORIZONTAL]));
  else
    MOLOCH_LAUNCH(KK_WAF_HORIZONTAL, st, kb_waf_horizontal<T><<<b.ntiles[TK_HORIZONTAL], hb, 0, st>>>(b.views[cur][fcur], b.tiles[TK_HORIZONTAL]));
  fcur ^= 1;
  MOLOCH_LAUNCH(KK_STAG_FROM_X, st, kb_stag_from_x<T><<<b.ntiles[TK_POINT], pb, 0, st>>>(b.views[cur][fcur], b.tiles[TK_POINT]));
  cur = 0;
  return 3;
}

int diag_parts(int nj, int ni) {
  const dim3 g = col_grid(nj, ni);
  return (int)(g.x * g.y);
}

}  // namespace MOLOCH_KNS
}  // namespace moloch
