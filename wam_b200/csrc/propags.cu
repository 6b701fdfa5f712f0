// PROPAGS stencil and CHECK_CFL coefficient extrema (compiled with
// -fmad=false so the coefficient arithmetic rounds like the reference).
#include "propags.cuh"
#include "kernels.hpp"

namespace wamgpu {

// One thread per (sea point i, frequency m) walking the directions: what the
// pair stencils below do not take (propags_pairs).
template <typename R, int VAR, bool RED, bool REFRD>
__device__ __forceinline__ void propags_point(const PropArgs<R>& A, const R* __restrict__ f1, int ld1,
                                              R* __restrict__ f3, int ld3, int i, int m) {
  using S = Site<R, VAR, RED, REFRD>;
  const S site(A, i, m);
  const int KL = A.KL, ML = A.ML;
  const size_t plane = (size_t)ld1 * KL;
  const R* fm = f1 + plane * m;
  auto F = [&](int p1, int k) -> R { return p1 == 0 ? R(0) : __ldg(&fm[(p1 - 1) + (size_t)ld1 * k]); };
  const bool theta = REFRD || S::SPH;
  R fkm = F(i + 1, KL - 1), fk = F(i + 1, 0);
  R* out = f3 + i + (size_t)ld3 * KL * m;
  typename S::Win W = site.window(0);
  for (int k = 0; k < KL; ++k) {
    const int kp = (k + 1 == KL) ? 0 : k + 1;
    const R fkp = F(i + 1, kp);
    const Coefs<R> c = site.coef_w(W);
    R v;
    if (!S::CUR) {
      const bool ic0 = W.cs >= R(0.), is0 = W.sn >= R(0.);
      v = c.sum * fk + c.lat11 * F(ic0 ? site.s0 : site.n0, k) + c.lon1 * F(is0 ? site.w0 : site.e0, k);
      if (theta) v = v + c.th1 * fkp + c.th2 * fkm;
      if (RED) v = v + c.lat12 * F(ic0 ? site.s1 : site.n1, k);
    } else {
      const int mm = (m == 0) ? 0 : m - 1, mp = (m == ML - 1) ? ML - 1 : m + 1;
      const R fmp = __ldg(&f1[i + (size_t)ld1 * k + plane * mp]), fmm = __ldg(&f1[i + (size_t)ld1 * k + plane * mm]);
      v = c.sum * fk + c.lat21 * F(site.n0, k) + c.lat11 * F(site.s0, k) + c.lon2 * F(site.e0, k) +
          c.lon1 * F(site.w0, k) + c.th1 * fkp + c.th2 * fkm + c.sg1 * fmp + c.sg2 * fmm;
      if (RED) v = v + c.lat22 * F(site.n1, k) + c.lat12 * F(site.s1, k);
    }
    out[(size_t)ld3 * k] = v;
    fkm = fk; fk = fkp;
    site.advance(W, k);
  }
}

template <typename R, int VAR, bool RED, bool REFRD>
__global__ void __launch_bounds__(128) propags_kernel(const __grid_constant__ PropArgs<R> A, const R* __restrict__ f1,
                                                      int ld1, R* __restrict__ f3, int ld3, int m0) {
  const int i = A.i0 + blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= A.i1) return;
  propags_point<R, VAR, RED, REFRD>(A, f1, ld1, f3, ld3, i, m0 + blockIdx.y);
}

// The stencil for the variants without currents, two frequencies m, m+1 of one
// sea point per thread (a sub-step of plane m reads plane m only).  Issue-bound
// work, so what the coefficients of Site::coef_w recompute is formed once, with
// the same operations and hence the same bits:
//   - the boundary term of directions k and k+1 (DTP of k) is also DTM of k+1:
//     its sums and products commute, so one value per direction serves both,
//     and its share of direction k+1 is multiplied by F(k) at once;
//   - products that depend on the point and the frequency alone (group velocity
//     sums of the neighbours, DRGM*CG) are formed before the loop;
//   - which neighbour is upwind changes with the signs of SIN and COS only: the
//     directions go in segments of constant signs (A.seg), the selection is made
//     per segment, and the loop inside has no branch, so that it unrolls with
//     the loads of three directions in flight;
//   - a land neighbour is read as the point itself and replaced by 0;
//   - row offsets are 32-bit and run along;
//   - CHECK_CFL's division by COUNTER runs as an exact scaled Markstein quotient.
// 105 -> 70 thread instructions per bin (32 of them FP32) on the shallow
// spherical grid with depth refraction.  A sub-step of 756k points, 36x30, takes
// 1.93 ms (3.4 TB/s of algorithmic traffic) against 2.69 before, with COUNTER = 2
// on 159k points 36x35 0.67 against 1.39, deep on 47k points 24x25 0.074 against
// 0.100.  The pairs of a block of points run next to each other (the blocks of a
// pair next to each other instead: 1.98 ms).
// Now bound by issue (78 % of the slots) and the latency of L2: three
// directions in flight are the most that 64 registers hold (unrolled by 1, 2 or
// 4 without the prefetch below: 4.1, 3.5 and 2.8 ms); the leaner deep stencil
// takes six.
// x / COUNTER, rounded as the division rounds it.
template <typename R> struct CounterDiv;
template <> struct CounterDiv<float> {
  float b, y;
  __device__ explicit CounterDiv(float rc) : b(rc), y(1.0f / rc) {}
  // scaled by 2^60, the residuals are exact for every coefficient (at most
  // COUNTER in size), and so is the way back above 2^-126
  __device__ float operator()(float x) const {
    const float a = x * 1152921504606846976.f;
    float q = a * y;
    q = __fmaf_rn(__fmaf_rn(-q, b, a), y, q);
    q = __fmaf_rn(__fmaf_rn(-q, b, a), y, q);
    return q * 8.67361737988403547e-19f;
  }
};
template <> struct CounterDiv<double> {
  double b;
  __device__ explicit CounterDiv(double rc) : b(rc) {}
  __device__ double operator()(double x) const { return x / b; }
};

// What one frequency of a point carries along the directions.
template <typename R> struct Line {
  R kS, kN, kW, kE;      // factors of the south, north, west and east boundary
  R drc, tsi;            // DRGM*CG, depth refraction factor
  R fk;                  // F(k)
  R mn;                  // negative part of DTM
  R up;                  // positive part of DTM (over COUNTER) times F(k-1)
  R th;                  // THDD(k)
};

template <typename R, int VAR, bool RED, bool REFRD, bool CNT>
__device__ __forceinline__ void propags_pair(const PropArgs<R>& A, const R* __restrict__ f1, int ld1, R* __restrict__ f3,
                                             int ld3, int i, int m, bool two) {
  using S = Site<R, VAR, RED, REFRD>;
  static_assert(!S::CUR, "the pair stencil is for the variants without currents");
  constexpr bool SH = S::SH, SPH = S::SPH, THETA = SPH || (SH && REFRD), TH = SH && REFRD;
  constexpr int UN = SH || CNT ? 3 : 6;  // directions whose loads are in flight
  const int KL = A.KL, mb = two ? m + 1 : m;
  const R one = R(1.), z = R(0.);
  unsigned iS, iN, iW, iE, iS2 = 0, iN2 = 0;  // neighbours' indices, the point's own for land
  bool lS, lN, lW, lE, lS2 = false, lN2 = false;
  R wl1 = one, wl2 = one, d0, ddphi = z, ddlam = z, gom[2] = {z, z};
  Line<R> L[2];
  {
    auto nb = [&](int p1, unsigned& idx, bool& land) { land = p1 == 0; idx = land ? (unsigned)i : (unsigned)(p1 - 1); };
    const S sa(A, i, m), sb(A, i, mb);
    nb(sa.s0, iS, lS); nb(sa.n0, iN, lN); nb(sa.w0, iW, lW); nb(sa.e0, iE, lE);
    if (RED) { nb(sa.s1, iS2, lS2); nb(sa.n1, iN2, lN2); wl1 = sa.wl1; wl2 = sa.wl2; }
    d0 = sa.d0;
    if (TH) { ddphi = sa.ddphi; ddlam = sa.ddlam; }
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const S& s = q ? sb : sa;
      Line<R>& l = L[q];
      gom[q] = s.gom;
      if (SH) {
        if (SPH && RED) {
          l.kS = s.cg + s.ps * (s.wl1 * s.cgS + (one - s.wl1) * s.cgS1);
          l.kN = s.cg + s.pn * (s.wl2 * s.cgN + (one - s.wl2) * s.cgN1);
        } else if (SPH) { l.kS = s.cg + s.ps * s.cgS; l.kN = s.cg + s.pn * s.cgN; }
        else { l.kS = s.cgS + s.cg; l.kN = s.cgN + s.cg; }
        l.kW = s.cgW + s.cg; l.kE = s.cgE + s.cg;
        l.drc = s.dr * s.cg; l.tsi = TH ? s.tsi : z;
      } else {
        l.kS = s.ps + one; l.kN = s.pn + one; l.kW = l.kE = one;
        l.drc = s.dr; l.tsi = z;
      }
    }
  }
  const CounterDiv<R> cd(CNT ? A.rcounter : one);
  const R* fp[2] = {f1 + (size_t)ld1 * KL * m, f1 + (size_t)ld1 * KL * mb};
  R* op[2] = {f3 + (size_t)ld3 * KL * m, f3 + (size_t)ld3 * KL * mb};
  const unsigned ui = (unsigned)i, st1 = (unsigned)ld1, st3 = (unsigned)ld3;
  // direction KL-1 to 0: the first DTM, F(KL-1), F(0)
  const R snl = A.sinth[KL - 1], csl = A.costh[KL - 1];
  R sn = A.sinth[0], cs = A.costh[0];
  const R sp0 = A.DELTH0 * (sn + snl);
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    Line<R>& l = L[q];
    const R fl = __ldg(fp[q] + st1 * (unsigned)(KL - 1) + ui);
    l.fk = __ldg(fp[q] + ui);
    R d = z;
    l.th = z;
    if (TH) {
      l.th = (sn * ddphi - cs * ddlam) * l.tsi;
      const R thm = (snl * ddphi - csl * ddlam) * l.tsi;
      d = SPH ? l.drc * sp0 + (l.th + thm) * A.DELTHR : (l.th + thm) * A.DELTHR;
    } else if (THETA) d = l.drc * sp0;
    l.mn = dmin(z, d);
    R th2 = dmax(z, d);
    if (SPH && !SH) th2 = gom[q] * th2;
    if (CNT) th2 = cd(th2);
    l.up = th2 * fl;
  }
  unsigned row = 0, orow = ui;  // row offsets of direction k
  int k = 0;
  for (int sgm = 0; k < KL; ++sgm) {
    const int kend = A.seg[sgm];
    const bool ic = cs >= z, is = sn >= z;
    const unsigned jlat = ic ? iS : iN, jlon = is ? iW : iE, jlat2 = RED ? (ic ? iS2 : iN2) : 0u;
    const bool landlat = ic ? lS : lN, landlon = is ? lW : lE, landlat2 = RED && (ic ? lS2 : lN2);
    const R wl = RED ? (ic ? wl1 : wl2) : one;
    R in_lat[2], out_lat[2], in_lon[2], out_lon[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      in_lat[q] = ic ? L[q].kS : L[q].kN; out_lat[q] = ic ? L[q].kN : L[q].kS;
      in_lon[q] = is ? L[q].kW : L[q].kE; out_lon[q] = is ? L[q].kE : L[q].kW;
    }
#pragma unroll UN
    for (; k < kend; ++k) {
      const bool wrap = k + 1 == KL;
      const int kp = wrap ? 0 : k + 1;
      const unsigned next = wrap ? 0u : row + st1;
      const R snp = A.sinth[kp], csp = A.costh[kp];
      R flat[2], flon[2], fkp[2], flat2[2] = {z, z};
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        fkp[q] = __ldg(fp[q] + (next + ui));
        flat[q] = __ldg(fp[q] + (row + jlat));
        flon[q] = __ldg(fp[q] + (row + jlon));
        if (RED) flat2[q] = __ldg(fp[q] + (row + jlat2));
        flat[q] = landlat ? z : flat[q];
        flon[q] = landlon ? z : flon[q];
        if (RED) flat2[q] = landlat2 ? z : flat2[q];
      }
      // direction-dependent terms common to both frequencies
      const R sda = dabs(sn), cda = dabs(cs * A.DELPH0);
      const R sp = SPH ? A.DELTH0 * (sn + snp) : z;
      const R grad = TH ? snp * ddphi - csp * ddlam : z;
      R dp_ = z, dpn_ = z, dle_ = z, dtc_ = z;  // deep spherical: without the frequency
      if (SPH && !SH) {
        dpn_ = cda * in_lat[0]; dle_ = sda * d0;
        dp_ = L[0].drc * sp;
        dtc_ = cda * out_lat[0] + dle_;
        dtc_ = dtc_ + dmax(z, dp_) - L[0].mn;
      }
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        Line<R>& l = L[q];
        R sum, lat, lat2 = z, lon, th1 = z, th2 = z, mn = z;
        if (SH) {
          lat = cda * in_lat[q];
          lon = sda * in_lon[q] * d0;
          const R ol = sda * out_lon[q] * d0;
          if (SPH) sum = (one - cda * out_lat[q]) - ol;
          else sum = (one - ol) - cda * out_lat[q];
          if (THETA) {
            R d;
            if (TH) {
              const R thp = grad * l.tsi;
              d = SPH ? l.drc * sp + (l.th + thp) * A.DELTHR : (l.th + thp) * A.DELTHR;
              l.th = thp;
            } else d = l.drc * sp;
            const R mx = dmax(z, d);
            mn = dmin(z, d);
            sum = sum - mx + l.mn;
            if (CNT) { const R qd = cd(d); th1 = -dmin(z, qd); th2 = dmax(z, qd); }
            else { th1 = -mn; th2 = mx; }
          }
        } else if (SPH) {
          const R g = gom[q];
          mn = dmin(z, dp_);
          lat = g * dpn_; lon = g * dle_;
          th1 = -(g * mn); th2 = g * dmax(z, dp_);
          sum = one - g * dtc_;
          if (CNT) { th1 = cd(th1); th2 = cd(th2); }
        } else {
          const R g = gom[q];
          lat = dabs(cs * A.DELPH0 * g); lon = dabs(sn * g) * d0;
          sum = one - lon - lat;
        }
        if (RED && SPH) { lat2 = lat * (one - wl); lat = lat * wl; }
        if (CNT) {
          lat = cd(lat); lon = cd(lon);
          if (RED) lat2 = cd(lat2);
          sum = one - cd(one - sum);
        }
        R v = sum * l.fk + lat * flat[q] + lon * flon[q];
        if (THETA) { v = v + th1 * fkp[q] + l.up; l.up = th2 * l.fk; }
        if (RED) v = v + lat2 * flat2[q];
        if (q == 0 || two) op[q][orow] = v;
        l.fk = fkp[q]; l.mn = mn;
      }
      row = next; orow += st3;
      sn = snp; cs = csp;
    }
  }
}

// What one frequency of a point carries with currents.
template <typename R> struct CurLine {
  R cg, cgS, cgN, cgW, cgE, cgS1, cgN1, tsi;
  R fk;  // F(k)
  R mn;  // negative part of DTM
  R up;  // positive part of DTM (over COUNTER) times F(k-1)
  R th;  // THDD(k)
};

// The stencil for the variants with currents, two frequencies m, m+1 of one sea
// point per thread.  Issue-bound like the one above, and by the same means: one
// boundary term serves direction k as DTP and k+1 as DTM; likewise one boundary
// term in frequency serves m as DOP and m+1 as DOM, so that two frequencies take
// three of them (from SIDC of m-1 .. m+2) instead of four; the direction's part
// of THDD and SIDC (products of SIN and COS with the current gradients) is formed
// once for both; F of one frequency is the other's neighbour in frequency; the
// quotients by 1.1 and by COUNTER are exact scaled Markstein quotients.  The
// expressions are those of Site::coef_w, so the results have the same bits.
// The frequency pairs of a block of points run next to each other, so that the
// planes m-1 and m+2, which other CTAs own, come from L2 on any grid.  A call on
// 47k points, 36x30, COUNTER = 1, with its copy of the spectrum: 578 us by the
// one-frequency kernel, 377 us.
template <typename R, int VAR, bool RED, bool CNT>
__device__ __forceinline__ void propags_pair_cur(const PropArgs<R>& A, const R* __restrict__ f1, int ld1,
                                                 R* __restrict__ f3, int ld3, int i, int m, bool two) {
  using S = Site<R, VAR, RED, false>;  // the refraction by currents knows no switch
  static_assert(S::CUR, "for the variants with currents");
  constexpr bool SH = S::SH, SPH = S::SPH;
  const int KL = A.KL, mb = min(m + 1, A.ML - 1), mlo = max(m - 1, 0), mhi = two ? min(m + 2, A.ML - 1) : mb;
  const R one = R(1.), z = R(0.);
  unsigned iS, iN, iW, iE, iS2 = 0, iN2 = 0;  // neighbours' indices, the point's own for land
  bool lS, lN, lW, lE, lS2 = false, lN2 = false;
  R wl1 = one, wl2 = one, d0, dr, ps, pn, ddphi = z, ddlam = z, duphi, dulam, dvphi, dvlam;
  R u0, uW, uE, v0, vS, vN, vS1 = z, vN1 = z;
  R scg[4], stt[4], stk[4], sdf[3];  // SIDC's factors of m-1 .. m+2, DELFR0/FR of the three boundaries
  CurLine<R> L[2];
  {
    auto nb = [&](int p1, unsigned& idx, bool& land) { land = p1 == 0; idx = land ? (unsigned)i : (unsigned)(p1 - 1); };
    const S sa(A, i, m), sb(A, i, mb);
    nb(sa.s0, iS, lS); nb(sa.n0, iN, lN); nb(sa.w0, iW, lW); nb(sa.e0, iE, lE);
    if (RED) { nb(sa.s1, iS2, lS2); nb(sa.n1, iN2, lN2); wl1 = sa.wl1; wl2 = sa.wl2; vS1 = sa.vS1; vN1 = sa.vN1; }
    d0 = sa.d0; dr = sa.dr; ps = sa.ps; pn = sa.pn;
    duphi = sa.duphi; dulam = sa.dulam; dvphi = sa.dvphi; dvlam = sa.dvlam;
    u0 = sa.u0; uW = sa.uW; uE = sa.uE; v0 = sa.v0; vS = sa.vS; vN = sa.vN;
    if (SH) {
      ddphi = sa.ddphi; ddlam = sa.ddlam;
      scg[0] = sa.cgM; stt[0] = sa.tempc * sa.tsiM; stk[0] = sa.tfkM;
      scg[1] = sa.cg; stt[1] = sa.tempc * sa.tsi; stk[1] = sa.tfk;
      scg[2] = sb.cg; stt[2] = sa.tempc * sb.tsi; stk[2] = sb.tfk;
      scg[3] = sb.cgP; stt[3] = sa.tempc * sb.tsiP; stk[3] = sb.tfkP;
      sdf[0] = sa.dfm; sdf[1] = sa.dfp; sdf[2] = sb.dfp;
    }
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const S& s = q ? sb : sa;
      CurLine<R>& l = L[q];
      if (SH) {
        l.cg = s.cg; l.cgS = s.cgS; l.cgN = s.cgN; l.cgW = s.cgW; l.cgE = s.cgE; l.tsi = s.tsi;
        l.cgS1 = s.cgS1; l.cgN1 = s.cgN1;
      } else {
        l.cg = l.cgS = l.cgN = l.cgW = l.cgE = l.cgS1 = l.cgN1 = s.gom; l.tsi = z;
      }
    }
  }
  const CounterDiv<R> cd(CNT ? A.rcounter : one), c11(R(1.1));
  const size_t plane = (size_t)ld1 * KL;
  const R* fp[2] = {f1 + plane * m, f1 + plane * mb};
  const R *flo = f1 + plane * mlo, *fhi = f1 + plane * mhi;
  R* op[2] = {f3 + (size_t)ld3 * KL * m, f3 + (size_t)ld3 * KL * mb};
  const unsigned ui = (unsigned)i, st1 = (unsigned)ld1, st3 = (unsigned)ld3;
  auto thdc = [&](R ss, R sc, R cc) { return ss * duphi + sc * dvphi - sc * dulam - cc * dvlam; };
  // boundary in direction between k and k+1 of a frequency: sines, THDD of both
  auto dbound = [&](const CurLine<R>& l, R sp, R spd, R t0, R tp) {
    if (!SPH) return (t0 + tp) * A.DELTHR;
    if (SH) return spd * l.cg + (t0 + tp) * A.DELTHR;
    return sp * l.cg * dr + (t0 + tp) * A.DELTHR;
  };
  R sn = A.sinth[0], cs = A.costh[0];
  R ss = sn * sn, sc = sn * cs, cc = cs * cs;
  {
    const R snl = A.sinth[KL - 1], csl = A.costh[KL - 1];
    const R sp = A.DELTH0 * (sn + snl), spd = sp * dr;
    const R t0 = thdc(ss, sc, cc), tl = thdc(snl * snl, snl * csl, csl * csl);
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      CurLine<R>& l = L[q];
      const R fl = __ldg(fp[q] + st1 * (unsigned)(KL - 1) + ui);
      l.fk = __ldg(fp[q] + ui);
      l.th = SH ? (sn * ddphi - cs * ddlam) * l.tsi + t0 : t0;
      const R thm = SH ? (snl * ddphi - csl * ddlam) * l.tsi + tl : tl;
      const R d = dbound(l, sp, spd, l.th, thm);
      l.mn = dmin(z, d);
      R th2 = dmax(z, d);
      if (CNT) th2 = cd(th2);
      l.up = th2 * fl;
    }
  }
  unsigned row = 0, orow = ui;
#pragma unroll 2
  for (int k = 0; k < KL; ++k) {
    const bool wrap = k + 1 == KL;
    const int kp = wrap ? 0 : k + 1;
    const unsigned next = wrap ? 0u : row + st1;
    R fS[2], fN[2], fW[2], fE[2], fkp[2], fS2[2] = {z, z}, fN2[2] = {z, z};
    const R fm1 = __ldg(flo + (row + ui)), fp2 = __ldg(fhi + (row + ui));
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      fkp[q] = __ldg(fp[q] + (next + ui));
      fN[q] = __ldg(fp[q] + (row + iN)); fS[q] = __ldg(fp[q] + (row + iS));
      fE[q] = __ldg(fp[q] + (row + iE)); fW[q] = __ldg(fp[q] + (row + iW));
      if (RED) { fN2[q] = __ldg(fp[q] + (row + iN2)); fS2[q] = __ldg(fp[q] + (row + iS2)); }
      fN[q] = lN ? z : fN[q]; fS[q] = lS ? z : fS[q]; fE[q] = lE ? z : fE[q]; fW[q] = lW ? z : fW[q];
      if (RED) { fN2[q] = lN2 ? z : fN2[q]; fS2[q] = lS2 ? z : fS2[q]; }
    }
    const R snp = A.sinth[kp], csp = A.costh[kp];
    // frequency shift: SIDC without the frequency, then the three boundaries
    const R b = -(sc * duphi) - cc * dvphi - ss * dulam - sc * dvlam;
    R g[3];
    if (SH) {
      R sv[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) sv[q] = (b * scg[q] + stt[q]) * stk[q];
#pragma unroll
      for (int q = 0; q < 3; ++q) g[q] = (sv[q] + sv[q + 1]) * sdf[q];
    } else {
      g[0] = g[1] = g[2] = b * A.DELFR0;
    }
    const R ssp = snp * snp, scp = snp * csp, ccp = csp * csp;
    const R tcp = thdc(ssp, scp, ccp), grad = SH ? snp * ddphi - csp * ddlam : z;
    const R sp = SPH ? A.DELTH0 * (sn + snp) : z, spd = SPH && SH ? sp * dr : z;
    R v[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      CurLine<R>& l = L[q];
      const R w1 = u0 + sn * l.cg, w2 = (v0 + cs * l.cg) * A.DELPH0;
      const R dlw = (w1 + (uW + sn * l.cgW)) * d0, dle = (w1 + (uE + sn * l.cgE)) * d0;
      R dtc = one - dmax(z, dle) + dmin(z, dlw);
      R lon1 = dmax(z, dlw), lon2 = -dmin(z, dle), lat11, lat12 = z, lat21, lat22 = z;
      auto wok2 = [&](R vv, R cgv) { return (vv + cs * cgv) * A.DELPH0; };
      if (!(SPH && RED)) {
        const R dps = SPH ? w2 + ps * wok2(vS, l.cgS) : w2 + wok2(vS, l.cgS);
        const R dpn = SPH ? w2 + pn * wok2(vN, l.cgN) : w2 + wok2(vN, l.cgN);
        dtc = dtc - dmax(z, dpn) + dmin(z, dps);
        lat11 = dmax(z, dps); lat21 = -dmin(z, dpn);
      } else {
        R dps, dps2, dpn, dpn2;
        if (SH) {
          dps = w2 + ps * (wl1 * wok2(vS, l.cgS) + (one - wl1) * wok2(vS1, l.cgS1));
          dps2 = dps * (one - wl1); dps = dps * wl1;
          dpn = w2 + pn * (wl2 * wok2(vN, l.cgN) + (one - wl2) * wok2(vN1, l.cgN1));
          dpn2 = dpn * (one - wl2); dpn = dpn * wl2;
        } else {
          dps = (w2 + wok2(vS, l.cgS) * ps) * wl1; dps2 = (w2 + wok2(vS1, l.cgS1) * ps) * (one - wl1);
          dpn = (w2 + wok2(vN, l.cgN) * pn) * wl2; dpn2 = (w2 + wok2(vN1, l.cgN1) * pn) * (one - wl2);
        }
        dtc = dtc - dmax(z, dpn) - dmax(z, dpn2) + dmin(z, dps) + dmin(z, dps2);
        lat11 = dmax(z, dps); lat12 = dmax(z, dps2); lat21 = -dmin(z, dpn); lat22 = -dmin(z, dpn2);
      }
      const R thp = SH ? grad * l.tsi + tcp : tcp;
      const R d = dbound(l, sp, spd, l.th, thp);
      const R mx = dmax(z, d), mn = dmin(z, d);
      dtc = dtc - mx + l.mn;
      R th1 = -mn, th2 = mx;
      R sg1 = c11(-dmin(z, g[q + 1])), sg2 = dmax(z, g[q]) * R(1.1);
      R sum = SH ? dtc - dmax(z, g[q + 1]) + dmin(z, g[q]) : dtc - dabs(g[0]);
      if (CNT) {
        lat11 = cd(lat11); lat21 = cd(lat21); lon1 = cd(lon1); lon2 = cd(lon2);
        if (RED) { lat12 = cd(lat12); lat22 = cd(lat22); }
        th1 = cd(th1); th2 = cd(th2); sg1 = cd(sg1); sg2 = cd(sg2);
        sum = one - cd(one - sum);
      }
      const R fmp = q ? fp2 : L[1].fk, fmm = q ? L[0].fk : fm1;
      v[q] = sum * l.fk + lat21 * fN[q] + lat11 * fS[q] + lon2 * fE[q] + lon1 * fW[q] + th1 * fkp[q] + l.up + sg1 * fmp +
             sg2 * fmm;
      if (RED) v[q] = v[q] + lat22 * fN2[q] + lat12 * fS2[q];
      l.up = th2 * l.fk;
      l.mn = mn; l.th = thp;
    }
    op[0][orow] = v[0];
    if (two) op[1][orow] = v[1];
    L[0].fk = fkp[0]; L[1].fk = fkp[1];
    row = next; orow += st3;
    sn = snp; cs = csp; ss = ssp; sc = scp; cc = ccp;
  }
}

// The rows of n points from i of both planes, all directions, on their way to
// L2: a thread per row, issued before the stencil's first load.  A thread keeps
// only the loads of three directions in flight, which covers the latency of L2
// but not that of DRAM.  Whole 16-byte granules: they hold valid data and so lie
// in mapped pages.
template <typename R>
__device__ __forceinline__ void prefetch_rows(const R* __restrict__ f1, int ld1, int KL, int i, int n, int m, bool two) {
  for (int t = threadIdx.x; t < (two ? 2 * KL : KL); t += blockDim.x) {
    const int q = t >= KL ? 1 : 0;
    const unsigned long long p = (unsigned long long)(f1 + (size_t)ld1 * ((size_t)KL * (m + q) + (t - q * KL)) + i);
    const unsigned long long b = p & ~15ull, e = (p + (unsigned long long)n * sizeof(R) + 15) & ~15ull;
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(b), "r"((unsigned)(e - b)) : "memory");
  }
}

// Frequencies m0 + 2*blockIdx.y and the next one (if below m0 + mcount).
template <typename R, int VAR, bool RED, bool REFRD, bool CNT>
__global__ void __launch_bounds__(128) propags_pair_kernel(const __grid_constant__ PropArgs<R> A, const R* __restrict__ f1,
                                                           int ld1, R* __restrict__ f3, int ld3, int m0, int mcount) {
  const int npair = (mcount + 1) / 2, x = blockIdx.x / npair, q = 2 * (blockIdx.x - x * npair);
  const int ib = A.i0 + x * blockDim.x, i = ib + threadIdx.x;
  prefetch_rows(f1, ld1, A.KL, ib, min((int)blockDim.x, A.i1 - ib), m0 + q, q + 1 < mcount);
  if (i >= A.i1) return;
  propags_pair<R, VAR, RED, REFRD, CNT>(A, f1, ld1, f3, ld3, i, m0 + q, q + 1 < mcount);
}

template <typename R, int VAR, bool RED, bool CNT>
__global__ void __launch_bounds__(128) propags_pair_cur_kernel(const __grid_constant__ PropArgs<R> A,
                                                               const R* __restrict__ f1, int ld1, R* __restrict__ f3,
                                                               int ld3, int m0, int mcount) {
  const int npair = (mcount + 1) / 2, x = blockIdx.x / npair, q = 2 * (blockIdx.x - x * npair);
  const int ib = A.i0 + x * blockDim.x, i = ib + threadIdx.x;
  prefetch_rows(f1, ld1, A.KL, ib, min((int)blockDim.x, A.i1 - ib), m0 + q, q + 1 < mcount);
  if (i >= A.i1) return;
  propags_pair_cur<R, VAR, RED, CNT>(A, f1, ld1, f3, ld3, i, m0 + q, q + 1 < mcount);
}

// Batched form: every member of an ensemble (one coefficient family) in one
// launch of BS-point CTAs.  CTA b belongs to member g with first[g] <= b <
// first[g + 1] and covers one frequency, or two of them where the pair stencil
// applies (PropMember::pair), of BS points of that member; the member's metadata block (direction tables included) is copied into shared
// memory first.
template <typename R, int VAR, bool RED, bool REFRD, int BS>
__global__ void __launch_bounds__(BS) propags_batch_kernel(const PropMember<R>* __restrict__ mem,
                                                           const int* __restrict__ first, int nmem) {
  __shared__ __align__(16) PropMember<R> sm;
  __shared__ int sg;
  if (threadIdx.x == 0) {
    int lo = 0, hi = nmem - 1;
    while (lo < hi) { int mid = (lo + hi + 1) >> 1; if (first[mid] <= (int)blockIdx.x) lo = mid; else hi = mid - 1; }
    sg = lo;
  }
  __syncthreads();
  const int g = sg;
  {
    const int nw = (int)(sizeof(PropMember<R>) / sizeof(int));
    const int* src = reinterpret_cast<const int*>(mem + g);
    int* dst = reinterpret_cast<int*>(&sm);
    for (int q = threadIdx.x; q < nw; q += BS) dst[q] = src[q];
  }
  __syncthreads();
  const int lb = (int)blockIdx.x - first[g], r = lb / sm.nbi;
  const int ib = sm.A.i0 + (lb - r * sm.nbi) * BS, i = ib + threadIdx.x;
  if (sm.pair) {
    const int m = 2 * r;
    const bool two = m + 1 < sm.A.ML;
    prefetch_rows(sm.src, sm.ld, sm.A.KL, ib, min(BS, sm.A.i1 - ib), m, two);
    if (i >= sm.A.i1) return;
    if constexpr (Site<R, VAR, RED, REFRD>::CUR) {
      if (sm.A.counter == 1) propags_pair_cur<R, VAR, RED, false>(sm.A, sm.src, sm.ld, sm.dst, sm.ld, i, m, two);
      else propags_pair_cur<R, VAR, RED, true>(sm.A, sm.src, sm.ld, sm.dst, sm.ld, i, m, two);
    } else {
      if (sm.A.counter == 1) propags_pair<R, VAR, RED, REFRD, false>(sm.A, sm.src, sm.ld, sm.dst, sm.ld, i, m, two);
      else propags_pair<R, VAR, RED, REFRD, true>(sm.A, sm.src, sm.ld, sm.dst, sm.ld, i, m, two);
    }
    return;
  }
  if (i >= sm.A.i1) return;
  propags_point<R, VAR, RED, REFRD>(sm.A, sm.src, sm.ld, sm.dst, sm.ld, i, r);
}

// Transpose of one sub-step, thread per (sea point i, frequency m): every
// term c * F_old(source) of the forward stencil becomes lam_old(source) +=
// c * lam_new(i, k, m).  The own point's direction neighbours (refraction)
// and the point itself are summed in registers first; spatial and frequency
// neighbours take atomic adds (lam_old zeroed by the caller).
template <typename R, int VAR, bool RED, bool REFRD>
__global__ void __launch_bounds__(128) propags_adj_kernel(const __grid_constant__ PropArgs<R> A,
                                                          const R* __restrict__ lnew, int ld1, R* lold, int ld3) {
  const int i = A.i0 + blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= A.i1) return;
  const int m = blockIdx.y;
  using S = Site<R, VAR, RED, REFRD>;
  const S site(A, i, m);
  const int KL = A.KL, ML = A.ML;
  const size_t plane = (size_t)ld3 * KL;
  const R* lm = lnew + (size_t)ld1 * KL * m;
  R* om = lold + plane * m;
  auto add = [&](int p1, int k, R v) { if (p1 != 0) atomicAdd(&om[(p1 - 1) + (size_t)ld3 * k], v); };
  const bool theta = REFRD || S::SPH;
  typename S::Win W = site.window(0);
  R carry0 = 0, first_th2 = 0, prev_own = 0;  // own-point sums waiting for the next direction
  for (int k = 0; k < KL; ++k) {
    const Coefs<R> c = site.coef_w(W);
    const R l = lm[i + (size_t)ld1 * k];
    R own = c.sum * l + carry0;  // + th1 of direction k-1 (carried)
    carry0 = 0;
    if (!S::CUR) {
      const bool ic0 = W.cs >= R(0.), is0 = W.sn >= R(0.);
      add(ic0 ? site.s0 : site.n0, k, c.lat11 * l);
      add(is0 ? site.w0 : site.e0, k, c.lon1 * l);
      if (RED) add(ic0 ? site.s1 : site.n1, k, c.lat12 * l);
    } else {
      add(site.n0, k, c.lat21 * l); add(site.s0, k, c.lat11 * l); add(site.e0, k, c.lon2 * l); add(site.w0, k, c.lon1 * l);
      if (RED) { add(site.n1, k, c.lat22 * l); add(site.s1, k, c.lat12 * l); }
      const int mm = (m == 0) ? 0 : m - 1, mp = (m == ML - 1) ? ML - 1 : m + 1;
      atomicAdd(&lold[i + (size_t)ld3 * k + plane * mp], c.sg1 * l);
      atomicAdd(&lold[i + (size_t)ld3 * k + plane * mm], c.sg2 * l);
    }
    if (theta || S::CUR) {
      // F_new(k) reads F_old(k+1) with th1 and F_old(k-1) with th2
      carry0 = c.th1 * l;                 // -> direction k+1
      if (k == 0) first_th2 = c.th2 * l;  // -> direction KL-1, added at the end
      else prev_own = prev_own + c.th2 * l;
    }
    if (k > 0) atomicAdd(&om[i + (size_t)ld3 * (k - 1)], prev_own);
    prev_own = own;
    site.advance(W, k);
  }
  // direction KL-1 gets its own sum and th2 of direction 0; direction 0 gets th1 of KL-1
  atomicAdd(&om[i + (size_t)ld3 * (KL - 1)], prev_own + first_th2);
  if (theta || S::CUR) atomicAdd(&om[i], carry0);
}

// Order-preserving float <-> int mapping for atomic max/min of extrema.
__device__ __forceinline__ int f2o(float f) { int i = __float_as_int(f); return i >= 0 ? i : i ^ 0x7fffffff; }
__device__ __forceinline__ long long d2o(double d) { long long i = __double_as_longlong(d); return i >= 0 ? i : i ^ 0x7fffffffffffffffLL; }

// ext[2*c] = max, ext[2*c+1] = min of coefficient class c (CflClass)
template <typename R, int VAR, bool RED, bool REFRD>
__global__ void __launch_bounds__(256) cfl_extrema_kernel(const __grid_constant__ PropArgs<R> A, long long* ext) {
  const int nown = A.i1 - A.i0;
  const size_t n = (size_t)nown * A.ML;
  R mx[CFL_NCLASS], mn[CFL_NCLASS];
  for (int c = 0; c < CFL_NCLASS; ++c) { mx[c] = R(-1e30); mn[c] = R(1e30); }
  for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < n; t += (size_t)gridDim.x * blockDim.x) {
    const int i = A.i0 + (int)(t % nown), m = (int)(t / nown);
    const Site<R, VAR, RED, REFRD> site(A, i, m);
    for (int k = 0; k < A.KL; ++k) {
      Coefs<R> c = site.coef(k);
      R v[CFL_NCLASS] = {c.lat11, c.lat21, c.lat12, c.lat22, c.lon1, c.lon2, c.th1, c.th2, c.sg1, c.sg2, c.sum};
      for (int q = 0; q < CFL_NCLASS; ++q) { mx[q] = dmax(mx[q], v[q]); mn[q] = dmin(mn[q], v[q]); }
    }
  }
  for (int q = 0; q < CFL_NCLASS; ++q) {
    mx[q] = warp_max(mx[q]);
    R x = mn[q];
    for (int o = 16; o > 0; o >>= 1) x = dmin(x, __shfl_xor_sync(0xffffffffu, x, o));
    mn[q] = x;
  }
  if ((threadIdx.x & 31) == 0)
    for (int q = 0; q < CFL_NCLASS; ++q) {
      long long a = sizeof(R) == 4 ? (long long)f2o((float)mx[q]) : d2o((double)mx[q]);
      long long b = sizeof(R) == 4 ? (long long)f2o((float)mn[q]) : d2o((double)mn[q]);
      atomicMax(&ext[2 * q], a);
      atomicMin(&ext[2 * q + 1], b);
    }
}

__global__ void cfl_init_kernel(long long* ext) {
  int q = threadIdx.x;
  if (q < CFL_NCLASS) { ext[2 * q] = LLONG_MIN; ext[2 * q + 1] = LLONG_MAX; }
}

// Compile-time dispatch over the ten reference variants (eight coefficient
// families x reduced grid x depth refraction).
template <typename R, template <typename, int, bool, bool> class K, typename... Args>
cudaError_t dispatch(const PropArgs<R>& A, Args&&... args) {
  const bool red = A.reduced != 0, rd = A.refr_d != 0;
#define VCASE(V)                                                             \
  case V:                                                                    \
    if (red) { if (rd) return K<R, V, true, true>::run(A, args...); return K<R, V, true, false>::run(A, args...); } \
    if (rd) return K<R, V, false, true>::run(A, args...);                    \
    return K<R, V, false, false>::run(A, args...);
  switch (A.variant) {
    VCASE(V_CART_DEEP) VCASE(V_CART_SHALLOW) VCASE(V_CART_DEEP_CUR) VCASE(V_CART_SHALLOW_CUR)
    VCASE(V_SPHER_DEEP) VCASE(V_SPHER_SHALLOW) VCASE(V_SPHER_DEEP_CURR) VCASE(V_SPHER_SHALLOW_CURR)
  }
#undef VCASE
  return cudaErrorInvalidValue;
}

// CTAs of pairs from which on two frequencies per thread are taken.  As long as the
// CTAs are all resident, a launch lasts as long as one thread's walk along the
// directions, which is shorter with one frequency (sub-step, pairs against one
// frequency, us; 36x30 shallow with depth refraction: 720 points, 90 CTAs, 14.5
// against 12.5; 2000 points, 240 CTAs, 14.7 against 14.6; 3000 points, 360 CTAs, 16.6
// against 17.5; 24x25 deep: 208 CTAs 11.4 against 10.5, 312 CTAs 12.5 both).  Not so
// where the walk itself gets shorter: COUNTER above 1 (15 CTAs, shallow 15.5 against
// 24.8, deep 11.9 against 16.8) and currents (15 CTAs, shallow 18.7 against 24.8;
// deep 13 CTAs 18.6 against 16.6, 39 CTAs 19.6 against 20.7).  In double precision
// the line is the same (3000 points, 360 CTAs, COUNTER 2 49 against 54, currents 64
// against 68; 720 points 43 against 39 and 35 against 33).
template <typename R, int V> unsigned pairs_from(int counter) {
  if (sizeof(R) == 8 || (!var_current(V) && counter == 1)) return 257;
  return var_current(V) && !var_shallow(V) ? 33 : 0;
}
template <typename R, int V, bool RED, bool RD> struct PropLaunch {
  static cudaError_t run(const PropArgs<R>& A, const R* f1, int ld1, R* f3, int ld3, int m0, int mcount, cudaStream_t s) {
    const unsigned n = (unsigned)((A.i1 - A.i0 + 127) / 128) * ((mcount + 1) / 2);
    if (propags_pairs(A, std::max(ld1, ld3)) && n >= pairs_from<R, V>(A.counter)) {
      if constexpr (var_current(V)) {
        if (A.counter == 1) propags_pair_cur_kernel<R, V, RED, false><<<n, 128, 0, s>>>(A, f1, ld1, f3, ld3, m0, mcount);
        else propags_pair_cur_kernel<R, V, RED, true><<<n, 128, 0, s>>>(A, f1, ld1, f3, ld3, m0, mcount);
      } else if (A.counter == 1) propags_pair_kernel<R, V, RED, RD, false><<<n, 128, 0, s>>>(A, f1, ld1, f3, ld3, m0, mcount);
      else propags_pair_kernel<R, V, RED, RD, true><<<n, 128, 0, s>>>(A, f1, ld1, f3, ld3, m0, mcount);
      return cudaGetLastError();
    }
    dim3 grid((A.i1 - A.i0 + 127) / 128, mcount);
    propags_kernel<R, V, RED, RD><<<grid, 128, 0, s>>>(A, f1, ld1, f3, ld3, m0);
    return cudaGetLastError();
  }
};
template <typename R, int V, bool RED, bool RD> struct CflLaunch {
  static cudaError_t run(const PropArgs<R>& A, long long* ext, int blocks, cudaStream_t s) {
    cfl_extrema_kernel<R, V, RED, RD><<<blocks, 256, 0, s>>>(A, ext);
    return cudaGetLastError();
  }
};

template <typename R, int V, bool RED, bool RD> struct PropBatchLaunch {
  static cudaError_t run(const PropArgs<R>&, const PropMember<R>* mem, const int* first, int nmem, int nblocks, int bs,
                         cudaStream_t s) {
    if (bs == 128) propags_batch_kernel<R, V, RED, RD, 128><<<nblocks, 128, 0, s>>>(mem, first, nmem);
    else if (bs == 256) propags_batch_kernel<R, V, RED, RD, 256><<<nblocks, 256, 0, s>>>(mem, first, nmem);
    else return cudaErrorInvalidValue;
    return cudaGetLastError();
  }
};

template <typename R>
cudaError_t launch_propags_batch(const PropArgs<R>& family, const PropMember<R>* mem, const int* first, int nmem,
                                 int nblocks, int bs, cudaStream_t s) {
  if (nblocks == 0) return cudaSuccess;
  return dispatch<R, PropBatchLaunch>(family, mem, first, nmem, nblocks, bs, s);
}

template <typename R, int V, bool RED, bool RD> struct PropAdjLaunch {
  static cudaError_t run(const PropArgs<R>& A, const R* ln, int ld1, R* lo, int ld3, cudaStream_t s) {
    dim3 grid((A.i1 - A.i0 + 127) / 128, A.ML);
    propags_adj_kernel<R, V, RED, RD><<<grid, 128, 0, s>>>(A, ln, ld1, lo, ld3);
    return cudaGetLastError();
  }
};

template <typename R>
cudaError_t launch_propags_adj(const PropArgs<R>& A, const R* lam_new, int ld1, R* lam_old, int ld3, cudaStream_t s) {
  if (A.i1 <= A.i0) return cudaSuccess;
  return dispatch<R, PropAdjLaunch>(A, lam_new, ld1, lam_old, ld3, s);
}

template <typename R>
cudaError_t launch_propags(const PropArgs<R>& A, const R* f1, int ld1, R* f3, int ld3, cudaStream_t s, int m0, int mcount) {
  if (mcount < 0) mcount = A.ML - m0;
  if (m0 < 0 || mcount < 0 || m0 + mcount > A.ML) return cudaErrorInvalidValue;
  if (A.i1 <= A.i0 || mcount == 0) return cudaSuccess;
  return dispatch<R, PropLaunch>(A, f1, ld1, f3, ld3, m0, mcount, s);
}

bool propags_planes_independent(int variant) {
  return variant != V_CART_DEEP_CUR && variant != V_CART_SHALLOW_CUR && variant != V_SPHER_DEEP_CURR &&
         variant != V_SPHER_SHALLOW_CURR;
}

bool propags_shallow(int variant) { return var_shallow(variant); }

template <typename R>
cudaError_t launch_cfl_extrema(const PropArgs<R>& A, long long* ext, int nsm, cudaStream_t s) {
  cfl_init_kernel<<<1, 32, 0, s>>>(ext);
  if (A.i1 <= A.i0) return cudaGetLastError();
  size_t n = (size_t)(A.i1 - A.i0) * A.ML;
  int blocks = (int)std::min<size_t>((n + 255) / 256, (size_t)nsm * 8);
  if (blocks < 1) blocks = 1;
  return dispatch<R, CflLaunch>(A, ext, blocks, s);
}

// Fixed F1 ping-pong spectrum of wamgpu_propags_dev_static: one per device,
// reserved when the module loads, never allocated or freed by the library.
static __device__ __align__(256) unsigned char g_static_prop_scratch[WAMGPU_STATIC_SCRATCH_BYTES];

// Device address of g_static_prop_scratch on the current device.
cudaError_t static_scratch_address(void** p) { return cudaGetSymbolAddress(p, g_static_prop_scratch); }

double cfl_decode(long long v, int precision) {
  if (precision == 4) {
    int i = (int)v;
    i = i >= 0 ? i : i ^ 0x7fffffff;
    float f; memcpy(&f, &i, 4); return f;
  }
  long long i = v >= 0 ? v : v ^ 0x7fffffffffffffffLL;
  double d; memcpy(&d, &i, 8); return d;
}

template cudaError_t launch_propags<float>(const PropArgs<float>&, const float*, int, float*, int, cudaStream_t, int, int);
template cudaError_t launch_propags<double>(const PropArgs<double>&, const double*, int, double*, int, cudaStream_t, int, int);
template cudaError_t launch_propags_batch<float>(const PropArgs<float>&, const PropMember<float>*, const int*, int, int,
                                                 int, cudaStream_t);
template cudaError_t launch_propags_batch<double>(const PropArgs<double>&, const PropMember<double>*, const int*, int,
                                                  int, int, cudaStream_t);
template cudaError_t launch_propags_adj<float>(const PropArgs<float>&, const float*, int, float*, int, cudaStream_t);
template cudaError_t launch_propags_adj<double>(const PropArgs<double>&, const double*, int, double*, int, cudaStream_t);
template cudaError_t launch_cfl_extrema<float>(const PropArgs<float>&, long long*, int, cudaStream_t);
template cudaError_t launch_cfl_extrema<double>(const PropArgs<double>&, long long*, int, cudaStream_t);

}  // namespace wamgpu
