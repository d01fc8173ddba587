// Implicit w (Thomas, one thread per column) + Exner/theta/pai update of
// sound() for FP32 storage (nompi/mod_moloch.F90:634-728, :843-849), staged
// by TMA, with the column state the back-substitution needs kept on chip.
//
// The one-thread-per-column kernel (b_sound_column) reads the down-sweep's
// inputs, writes an FP32 stash of the recurrence, and in the
// back-substitution reads the stash and six of the inputs again; at
// 512 x 512 x 60 about 175 K columns are in flight, so level k is read again
// 2k+1 level steps later, long after L2 evicted it (1.49x the algorithmic
// DRAM bytes).  Here:
//   * persistent CTAs, two an SM, walk tiles of 256 columns (256 x 1 to
//     32 x 8), eight compute warps of 32 columns each, one thread per column;
//   * a producer warp stages chunks of kct levels of every input with 3-D
//     TMA boxes into a ring of shared-memory stages, running ahead through
//     the down-sweep chunks, the back-substitution chunks and the next
//     tile's chunks, so loads never wait on the recurrence;
//   * the recurrence's wp and ww of each level go into the thread's own TMEM
//     lane (2 words a level: warps w and w+4 share a lane quarter), which
//     stands in for registers that cannot be indexed by level;
//   * w, qv, tetav, pai, zdiv2b and fmz, which the back-substitution stages
//     again, are loaded with an L2 evict_last policy in the down-sweep (the
//     resident set of all CTAs is 304 x 256 columns x 60 levels x 24 B =
//     112 MB at most) and every other load and store with evict_first.
// The arithmetic per level is that of b_sound_column<float> (FP64 pivots in
// complement form, FP32 right-hand side and back-substitution).
//
// Waits are bounded by View::spin_cycles SM cycles; a wait that gives up
// sets *View::kerr, the CTA stops, waits (bounded) for its copies in
// flight, frees TMEM and returns.
#pragma once

#include "moloch_tc.cuh"

namespace moloch {
namespace MOLOCH_KNS {

constexpr int kTwMaxKz = 64;  // 2 words x kz TMEM columns per warp

// tensor maps of the staged arrays (tetav, pai, qv, qc depend on the
// advected-field buffer set, so the host keeps one set per parity)
enum ColMap { CM_W = 0, CM_FMZF, CM_QV, CM_TET, CM_PAI, CM_QSAT, CM_ZD, CM_FMZ, CM_T, CM_QC, CM_QWL, CM_QWI, CM_S,
              CM_COUNT };
struct ColumnMaps {
  CUtensorMap m[CM_COUNT];
};
// FP32 <-> FP64 conversions on the integer pipe for values known to lie in
// the FP32 normal range -- in the pivot recurrence zu, zd > 0, tt, den >= 1,
// q0 in (0, 1] -- giving the bits widen_f32 / narrow_trunc give there,
// without their zero, subnormal, infinity and NaN cases (which cost most of
// their operations, all on the recurrence's dependency chain).  The
// quotient's residual may be zero: narrow_residual flushes magnitudes below
// the FP32 normal range to zero.
__device__ __forceinline__ double widen_normal(float x) {
  const unsigned b = __float_as_uint(x);
  const unsigned hi = (((b & 0x7fffffffu) >> 3) + 0x38000000u) | (b & 0x80000000u);
  return __hiloint2double((int)hi, (int)(b << 29));
}
__device__ __forceinline__ float narrow_normal(double x) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  const unsigned m = (__funnelshift_l(lo, hi, 3) - (896u << 23)) & 0x7fffffffu;
  return __uint_as_float(m | (hi & 0x80000000u));
}
__device__ __forceinline__ float narrow_residual(double x) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  const unsigned m = (__funnelshift_l(lo, hi, 3) - (896u << 23)) & 0x7fffffffu;
  return __uint_as_float(((hi & 0x7fffffffu) < 0x38100000u ? 0u : m) | (hi & 0x80000000u));
}

__device__ __forceinline__ uint32_t fbits(float x) { return __float_as_uint(x); }
__device__ __forceinline__ float bitsf(uint32_t x) { return __uint_as_float(x); }

// Shape of the staged kernel.  Two CTAs an SM of eight compute warps each:
// the CTAs drift apart, so one's down-sweep (bound by the FP64 pipe) runs
// beside the other's back-substitution (bound by memory); one CTA of twelve
// warps swept in step.  A warp takes 32 columns; the warps of a CTA lie side
// by side along j as far as that wastes none of the tile (View::twide of
// them), because a 256-column row of a box is one 1 KB run of DRAM where a
// 32-column one is 128 B.  Per step at 512 x 512 x 60 (1024 x 1024 x 60): one
// CTA of twelve warps, 32 columns wide, 3.51 (12.50) ms; two of eight warps,
// 32 wide, 3.39 (12.85); 128 wide 3.26 (11.52); 256 wide 3.23 (11.27); four
// of four warps, 128 wide, 3.23 (11.60).  256 x 256 x 40: 1.01 -> 0.69.
template <int LAST>
struct TwCfg {
  static constexpr int warps = kTwWarps;               // compute warps of a CTA
  static constexpr int kct = 4;                        // levels per staged chunk
  static constexpr int ctas = 2;                       // CTAs per SM
  static constexpr int slots = LAST ? 11 : 9;          // arrays per stage (the last substep also completes s)
  static constexpr int slot_bytes = kct * warps * 32 * 4;
  static constexpr int stage_bytes = slots * slot_bytes;
  static constexpr int stages = (226 * 1024 / ctas - 2048) / stage_bytes;  // ring depth within 227 KB an SM
  static constexpr int smem = stages * stage_bytes + 128;
  static constexpr int threads = 32 * (warps + 1);
  static constexpr int bank = 2 * kTwMaxKz;            // TMEM columns per warp: 2 words a level
  static constexpr int tmem = warps / 4 * bank;        // TMEM columns of a CTA
  static_assert(warps % 4 == 0 && ctas * tmem <= 512, "TMEM holds 512 columns a lane");
};

// The arrays and scalars of the domain a column tile belongs to
template <class T>
struct TwDom {
  const T *zdiv2b, *fmz, *qsat, *ffilt;
  T *w, *deltaw, *tetav, *pai, *s, *ep_j, *ep_i;
  int nj, ni, kz;
  size_t pl;
  T zcs2, dts, egdts, dtrdz;
};
template <class T>
__device__ __forceinline__ TwDom<T> tw_dom(const View<T>& d) {
  TwDom<T> v;
  v.zdiv2b = d.zdiv2b; v.fmz = d.fmz; v.qsat = d.qsat; v.ffilt = d.ffilt;
  v.w = d.w; v.deltaw = d.deltaw; v.tetav = d.tetav; v.pai = d.pai; v.s = d.s; v.ep_j = d.ep_j; v.ep_i = d.ep_i;
  v.nj = d.nj; v.ni = d.ni; v.kz = d.kz; v.pl = d.pl;
  v.zcs2 = d.zcs2; v.dts = d.dts; v.egdts = d.egdts; v.dtrdz = d.dtrdz;
  return v;
}

// The body of k_sound_column_tw (one domain: BATCH false, the tiles of
// that domain computed from the tile number) and of kb_sound_column_tw
// (an ensemble: BATCH true, tile t is tiles[t] = {member, tile x, tile y},
// the member's view in views[member] and its tensor maps in
// cms[2 member + fcur]).  A CTA walks tiles blockIdx.x, + gridDim.x, ...;
// the producer and the compute warps count the same jobs (the chunks of
// each tile, which depend on the tile's kz).
template <class T, int LAST, bool BATCH>
__device__ __forceinline__ void column_tw_body(const View<T>* views, const ColumnMaps* cms, const int4* tiles,
                                               int ntiles_in, int fcur, int nsound, int* kerr, long long lim,
                                               int skip_job) {
  using C = TwCfg<LAST>;
  constexpr int KC = C::kct, NST = C::stages, SLOTF = C::slot_bytes / 4;
  constexpr bool last = LAST != 0;  // the last substep also completes s (Equation 10)
  static_assert(sizeof(T) == 4, "FP32 storage only");
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t full[NST], empty[NST];
  __shared__ uint32_t tmem_base;
  __shared__ int s_fail, s_consumed;
  __shared__ int s_last_job[NST];
  __shared__ float s_ff[kTwMaxKz];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 127) & ~(uintptr_t)127);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // one domain: tiles of nbx x nby
  const int wide1 = BATCH ? 1 : views[0].twide;
  const int nbx1 = BATCH ? 1 : (views[0].nj + 32 * wide1 - 1) / (32 * wide1);
  const int ntiles = BATCH ? ntiles_in : nbx1 * ((views[0].ni * wide1 + C::warps - 1) / C::warps);
  struct Tile { int m, x, y, wide; };  // first column and row, warps side by side
  auto tile_of = [&](int t) -> Tile {
    if constexpr (BATCH) {
      const int4 q = tiles[t];
      const int w = views[q.x].twide;
      return {q.x, q.y * 32 * w, q.z * (C::warps / w), w};
    } else {
      return {0, (t % nbx1) * 32 * wide1, (t / nbx1) * (C::warps / wide1), wide1};
    }
  };

  if (warp == 0) tc::tmem_alloc(&tmem_base, C::tmem);
  if (tid == 32 * C::warps) {
    for (int q = 0; q < NST; ++q) {
      tc::mbar_init(&full[q], 1);
      tc::mbar_init(&empty[q], C::warps);
      s_last_job[q] = -1;
    }
    s_fail = 0;
    s_consumed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if constexpr (!BATCH)
    for (int k = tid; k < views[0].kz; k += blockDim.x) s_ff[k] = views[0].ffilt[k];
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tbase = tmem_base;

  if (warp == C::warps) {
    // ---- producer: one thread issues every TMA box of this CTA's jobs
    if (lane == 0) {
      const uint64_t keep = tc::policy_evict_last(), once = tc::policy_evict_first();
      const uint32_t down_bytes = 9u * C::slot_bytes, up_bytes = (last ? 11u : 9u) * C::slot_bytes;
      int g = 0;
      bool stop = false;
      for (int t = (int)blockIdx.x; t < ntiles && !stop; t += (int)gridDim.x) {
        const Tile tl = tile_of(t);
        const int kz = views[tl.m].kz;
        const int nd = (kz - 1 + KC - 1) / KC, jpt = nd + (kz + KC - 1) / KC;
        const CUtensorMap* mp = (BATCH ? cms[2 * tl.m + fcur] : cms[0]).m;
        for (int c = 0; c < jpt; ++c, ++g) {
          const int q = g % NST;
          if (g >= NST && !tc::mbar_wait_cycles(&empty[q], ((g / NST) - 1) & 1, lim)) {
            s_fail = 1;
            stop = true;
            break;
          }
          if (*(volatile int*)&s_fail) {
            stop = true;
            break;
          }
          if (g == skip_job) continue;  // test hook: leave this job unissued
          uint8_t* stg = smem + q * C::stage_bytes;
          auto box = [&](int slot, int map, int z, uint64_t pol) {
            tc::tma_load_3d_hint(stg + slot * C::slot_bytes, &mp[map], tl.x, tl.y, z, &full[q], pol);
          };
          if (c < nd) {
            const int kk_lo = kz - 1 - c * KC - (KC - 1);
            tc::mbar_arrive_expect_tx(&full[q], down_bytes);
            // level kk of w, fmzf, qv and level kk-1 of the others share a
            // slot index; w, qv, tetav, pai, zdiv2b, fmz are read again by
            // the back-substitution and stay in L2
            box(0, CM_W, kk_lo, keep);
            box(1, CM_FMZF, kk_lo, once);
            box(2, CM_QV, kk_lo, keep);
            box(3, CM_TET, kk_lo - 1, keep);
            box(4, CM_PAI, kk_lo - 1, keep);
            box(5, CM_QSAT, kk_lo - 1, once);
            box(6, CM_ZD, kk_lo - 1, keep);
            box(7, CM_FMZ, kk_lo - 1, keep);
            box(8, CM_T, kk_lo - 1, once);
          } else {
            // levels m = m0 .. m0+KC-1 of the arrays of the update, level
            // m+1 of the old w
            const int m0 = (c - nd) * KC;
            tc::mbar_arrive_expect_tx(&full[q], up_bytes);
            box(0, CM_FMZ, m0, once);
            box(1, CM_QV, m0, once);
            box(2, CM_TET, m0, once);
            box(3, CM_PAI, m0, once);
            box(4, CM_QC, m0, once);
            box(5, CM_QWL, m0, once);
            box(6, CM_QWI, m0, once);
            box(7, CM_W, m0 + 1, once);
            box(8, CM_ZD, m0, once);
            if (last) {
              box(9, CM_S, m0, once);
              box(10, CM_FMZF, m0, once);
            }
          }
          s_last_job[q] = g;
        }
      }
    }
  } else {
    // ---- compute warps: warp w holds 32 columns of row y + w / wide of the
    // tile; its TMEM: lane quarter w % 4, columns 128 (w / 4) .., 2 per level
    const uint32_t trow = tbase + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)((warp >> 2) * C::bank);
    const uint64_t once = tc::policy_evict_first();
    const T ns = T(nsound), ns1 = T(nsound - 1);
    const T rdrcv = T(kRdrcv);
    int g = 0;  // job counter, in the producer's order
    bool fail = false;
    auto wait_full = [&](int job) -> const float* {
      const int q = job % NST;
      bool ok = tc::mbar_wait_cycles(&full[q], (job / NST) & 1, lim);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) {
        if (lane == 0) s_fail = 1;
        fail = true;
        return nullptr;
      }
      return reinterpret_cast<const float*>(smem + q * C::stage_bytes);
    };
    auto release = [&](int job) {
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&empty[job % NST]);
    };
    // slot a, level index q (0 .. KC-1) of this thread's column
    const int sl = warp * 32 + lane;
    auto S_ = [&](const float* st, int a, int q) { return st[a * SLOTF + q * (C::warps * 32) + sl]; };
    // the values a tile starts from: level kz-1 of zdiv2b, tetav, pai, fmz,
    // qsat and the surface w (columns outside the domain read column 0)
    struct Init { T zd, tk, pk, fk, qsk, wsurf; };
    auto load_init = [&](int t, Init& v) {
      const Tile tl = tile_of(t);
      const TwDom<T> dm = tw_dom(views[tl.m]);
      const int jj = tl.x + (warp & (tl.wide - 1)) * 32 + lane, ii = tl.y + warp / tl.wide;
      const size_t c = (jj < dm.nj && ii < dm.ni) ? (size_t)jj + (size_t)dm.nj * ii : 0;
      const size_t o = (size_t)(dm.kz - 1) * dm.pl;
      v.zd = dm.zdiv2b[c + o]; v.tk = dm.tetav[c + o]; v.pk = dm.pai[c + o]; v.fk = dm.fmz[c + o];
      v.qsk = dm.qsat[c + o]; v.wsurf = dm.w[c + (size_t)dm.kz * dm.pl];
    };
    Init nx{};
    if ((int)blockIdx.x < ntiles) load_init((int)blockIdx.x, nx);

    for (int t = (int)blockIdx.x; t < ntiles && !fail; t += (int)gridDim.x) {
      const Tile tl = tile_of(t);
      const TwDom<T> v = tw_dom(views[tl.m]);
      const int nj = v.nj, ni = v.ni, kz = v.kz;
      const size_t pl = v.pl;
      const T zcs2 = v.zcs2, dts = v.dts, egdts = v.egdts, dtrdz = v.dtrdz;
      const int nd = (kz - 1 + KC - 1) / KC;  // down-sweep chunks: kk = kz-1 .. 1
      const int nu = (kz + KC - 1) / KC;      // back-substitution chunks: kk = 1 .. kz
      const int nfull = (kz - 1) / KC;        // back-substitution chunks whose levels all lie below kz
      const int jj = tl.x + (warp & (tl.wide - 1)) * 32 + lane, ii = tl.y + warp / tl.wide;
      const bool own = jj < nj && ii < ni;
      const size_t c = own ? (size_t)jj + (size_t)nj * ii : 0;
      T zd_k = nx.zd, tk = nx.tk, pk = nx.pk, fk = nx.fk, qsk = nx.qsk;
      const T wsurf = nx.wsurf;
      float wkp1 = wsurf;
      double cwp1 = 1.0;  // 1 - wwkw(kz+1)
      auto ffilt = [&](int kk) -> T {
        if constexpr (BATCH) return v.ffilt[kk];
        else return s_ff[kk];
      };

      // one level kk of the down-sweep from slot index q; the record of
      // level kk (wp, ww) goes to rec[0..1]
      auto dn_level = [&](const float* st, const int q, const int kk, uint32_t* rec) {
        const T wk = S_(st, 0, q), fz = S_(st, 1, q), qvk = S_(st, 2, q), ff = ffilt(kk);
        const T tkm = S_(st, 3, q), pkm = S_(st, 4, q), qskm = S_(st, 5, q), zd_km = S_(st, 6, q);
        const T fkm = S_(st, 7, q), tm = S_(st, 8, q);
        T zrom1w = ((T(0.5) * T(kCpd)) * fz) * (tkm + tk);
        zrom1w = zrom1w - (((((T(kCpd) * wk) * fz) * fz) * ns) * dtrdz) * (tkm - tk);
        zrom1w = zrom1w_moist(zrom1w, qvk, qsk, qskm, wk, fz, pkm, tm, ns1, dts);
        T zwexpl = (wk - (zrom1w * dtrdz) * (pkm - pk)) - egdts;
        zwexpl = zwexpl + ((T(kRdrcv) * zrom1w) * dtrdz) * prod_sub(pkm, zd_km, pk, zd_k);
        const T zu_t = ((zcs2 * fkm) * zrom1w) * pkm + ff;
        const T zd_t = ((zcs2 * fk) * zrom1w) * pk + ff;
        const double zu = widen_normal(zu_t), zdd = widen_normal(zd_t);
        const double tt = fma(zdd, cwp1, 1.0);
        const double den = tt + zu;
        float r;
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(narrow_normal(den)));
        const double q0 = widen_normal(narrow_normal(tt) * r);
        const double rem = fma(-den, q0, tt);
        cwp1 = q0 + widen_normal(r * narrow_residual(rem));
        const float wpk = r * (zwexpl + zd_t * wkp1);
        rec[0] = fbits(wpk); rec[1] = fbits(r * zu_t);
        wkp1 = wpk;
        zd_k = zd_km; tk = tkm; pk = pkm; fk = fkm; qsk = qskm;
      };

      // (b) down-sweep k = kz .. 2 (reference order)
      for (int cc = 0; cc < nd; ++cc, ++g) {
        const float* st = wait_full(g);
        if (!st) break;
        const int kk_hi = kz - 1 - cc * KC, kk_lo = kk_hi - (KC - 1);
        if (kk_lo >= 1) {  // a whole chunk: one TMEM store of its 8 words
          uint32_t rec[2 * KC];
#pragma unroll
          for (int u = 0; u < KC; ++u) dn_level(st, KC - 1 - u, kk_hi - u, rec + 2 * (KC - 1 - u));
          tc::tmem_st8p(trow + (uint32_t)(2 * kk_lo), rec);
        } else {
          for (int kk = kk_hi; kk >= 1; --kk) {
            uint32_t rec[2];
            dn_level(st, kk - kk_lo, kk, rec);
            tc::tmem_st2(trow + (uint32_t)(2 * kk), rec[0], rec[1]);
          }
        }
        release(g);
      }
      if (fail) break;
      tc::tmem_wait_st();
      // the next tile's starting values, loaded while this one finishes
      if (t + (int)gridDim.x < ntiles) load_init(t + (int)gridDim.x, nx);

      // (c) back-substitution (:681-686) fused with the Exner/theta update
      // of the level above (:690-728); w(1) = 0 always (init_moloch :260-262).
      // Chunk cc holds levels kk = 4 cc + 1 .. 4 cc + 4; the records of a
      // whole chunk (all kk < kz) are 8 consecutive TMEM columns, loaded one
      // chunk ahead.
      float wlo_d = 0.f;
      T wlo = T(0);
      uint32_t cur[2 * KC], nxt[2 * KC];
      if (nfull > 0) tc::tmem_ld8p(trow + 2u, nxt);
      T* __restrict__ pw = v.w + c;
      T* __restrict__ pdw = v.deltaw + c;
      T* __restrict__ ptet = v.tetav + c;
      T* __restrict__ ppai = v.pai + c;
      T* __restrict__ psv = v.s + c;
      // level kk (record rec when kk < kz) and the update of level kk-1
      auto up_level = [&](const float* st, const int q, const int kk, const uint32_t* rec) {
        const int m = kk - 1;
        T wn;
        if (rec) {
          wlo_d = bitsf(rec[0]) + bitsf(rec[1]) * wlo_d;
          wn = (T)wlo_d;
          if (own) {
            const size_t qq = (size_t)kk * pl;
            tc::st_hint(pdw + qq, (-S_(st, 7, q)) + wn, once);
            tc::st_hint(pw + qq, wn, once);
          }
        } else {
          wn = wsurf;
        }
        const T ffmz = S_(st, 0, q), fqv = S_(st, 1, q), ftet = S_(st, 2, q), fpai = S_(st, 3, q);
        const T fqc = S_(st, 4, q), fqwl = S_(st, 5, q), fqwi = S_(st, 6, q);
        T zd = S_(st, 8, q);
        zd = zd + (dtrdz * ffmz) * (wlo - wn);
        zd = div_corr(zd * ((T(1) + T(0.86) * fqv) + T(3.2) * fqc), (T(1) + T(0.96) * fqv) + T(4.8) * fqc);
        if (own) {
          const size_t qm = (size_t)m * pl;
          tc::st_hint(ptet + qm,
                      ftet * (T(1) + (rdrcv * zd) * (prod_add(T(0.25), fqv, T(4.2), fqwl) + T(2.1) * fqwi)), once);
          if (jj == nj - 1) v.ep_j[ii + (size_t)ni * m] = fpai;
          if (ii == ni - 1) v.ep_i[jj + (size_t)nj * m] = fpai;
          tc::st_hint(ppai + qm, fpai * (T(1) - rdrcv * zd), once);
          if (last) tc::st_hint(psv + qm, m == 0 ? T(0) : (wlo + S_(st, 9, q)) * S_(st, 10, q), once);  // Eq. 10
        }
        wlo = wn;
      };
      for (int cc = 0; cc < nu; ++cc, ++g) {
        const float* st = wait_full(g);
        if (!st) break;
        const int kk0 = cc * KC + 1;
        if (cc < nfull) {
          tc::tmem_wait_ld8p(nxt);
#pragma unroll
          for (int e = 0; e < 2 * KC; ++e) cur[e] = nxt[e];
          if (cc + 1 < nfull) tc::tmem_ld8p(trow + (uint32_t)(2 * (kk0 + KC)), nxt);
#pragma unroll
          for (int u = 0; u < KC; ++u) up_level(st, u, kk0 + u, cur + 2 * u);
        } else {
          for (int kk = kk0; kk <= kz && kk < kk0 + KC; ++kk) {
            if (kk < kz) {
              uint32_t rec[2];
              tc::tmem_ld2(trow + (uint32_t)(2 * kk), rec);
              tc::tmem_wait_ld2(rec);
              up_level(st, kk - kk0, kk, rec);
            } else {
              up_level(st, kk - kk0, kk, nullptr);
            }
          }
        }
        release(g);
      }
      if (fail) break;
      if (last && own) v.s[c + (size_t)kz * pl] = T(0);
    }
    // no TMEM load or store of this thread may be in flight when TMEM is
    // freed (a wait that gave up can leave one of either)
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
    if (lane == 0 && warp == 0) s_consumed = g;  // first job warp 0 did not finish
  }
  tc::tc_fence_before();
  __syncthreads();
  if (tid == 32 * C::warps && s_fail) {
    // a wait gave up: flag it and let the copies still in flight land
    // before the CTA's shared memory is released (bounded)
    atomicExch(kerr, 1);
    for (int q = 0; q < NST; ++q) {
      const int j = s_last_job[q];
      if (j >= s_consumed) tc::mbar_wait_cycles(&full[q], (j / NST) & 1, lim);
    }
  }
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  if (warp == 0) tc::tmem_dealloc(tbase, C::tmem);
}

template <class T, int LAST>
__global__ void __launch_bounds__(TwCfg<LAST>::threads, TwCfg<LAST>::ctas)
    k_sound_column_tw(const __grid_constant__ View<T> d, const __grid_constant__ ColumnMaps maps, int nsound) {
  if (d.sur_skip && *d.sur_skip) return;  // the surrogate took this cycle
  column_tw_body<T, LAST, false>(&d, &maps, nullptr, 0, 0, nsound, d.kerr, d.spin_cycles, d.fault_skip_job);
}

// An ensemble's column tiles in one persistent launch: the tile table
// lists (member, tile x, tile y) heaviest member first; cms holds each
// member's tensor maps, whose boxes have its tiles' shape (View::twide), two
// buffer-set parities per member.  A wait that gives up sets *kerr (the ensemble's error word).
template <class T, int LAST>
__global__ void __launch_bounds__(TwCfg<LAST>::threads, TwCfg<LAST>::ctas)
    kb_sound_column_tw(const View<T>* __restrict__ views, const ColumnMaps* __restrict__ cms,
                       const int4* __restrict__ tiles, int ntiles, int fcur, int nsound, int* kerr, long long lim) {
  column_tw_body<T, LAST, true>(views, cms, tiles, ntiles, fcur, nsound, kerr, lim, -1);
}

}  // namespace MOLOCH_KNS
}  // namespace moloch
