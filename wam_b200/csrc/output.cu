// Integrated output parameters on the device: COMPUTE_OUTPUT_PARAMETER
// (myWAveModel/WAM wam_output_module.f90:481-640) for the parameters that
// are functions of one sea point's spectrum and fields, so that an output
// step reads NSEA x 40 values instead of downloading the spectrum.
//
// A CTA of six warps integrates 32 sea points, lane = point.  The spectrum
// FL3(IJ,K,M) has the sea point fastest, so a warp reads 128 contiguous bytes
// of every bin.  The warps take frequencies for the sums over directions and
// directions for the sums over frequencies, so that every sum is one thread's
// loop in the reference's order; the integrals are then dealt out to the warps.
// One thread per point, the direction sums in shared memory, had 18 warps on an
// SM wait for one chain of loads each.  84k points, 36x30, the parameters and
// the wind sea / swell split together: 1275 us then, 290 us now (reading the
// spectrum once from DRAM takes 56 us; each of the two calls has to).
//   - output_kernel (121 us) reads each bin once, six frequencies on their way
//     to shared memory while six are summed; reading the spectrum twice, the
//     second time along the frequencies, took 236 us, since eight CTAs on an SM
//     hold more than L2 does.
//   - swell_kernel (168 us) does read it twice: bound by issue (54 % of the
//     slots), and with the staging rows in shared memory too few warps fit
//     (248 us).
// The unit is compiled without FMA contraction, so the results are those of the
// reference's separate operations; only ATAN2 (current direction, mean
// direction) is the device library's.
//
// Routines (wam_interface_module.f90): TOTAL_ENERGY_B :1342-1410, FEMEAN
// :207-286, TM1_TM2_PERIODS_B :1152-1245, PEAK_PERIOD_B :741-813,
// MEAN_DIRECTION_B :412-533, MEANSQS :639-737, CHARNOCK_PAR :159-203; AIRSEA
// (wam_source_module.f90:868-971) when USTAR is zero everywhere.
#include <cfloat>
#include "kernels.hpp"
#include "devmath.cuh"

namespace wamgpu {

namespace {

constexpr int kOutWarps = 6;
static_assert(kOutWarps == 6, "the integrals are dealt out to six warps");

template <typename R> struct OutConst {
  static constexpr R DEG = R(180.) / Phys<R>::PI;
};

template <typename R> __device__ __forceinline__ R orient(R deg, int from) {
  return from ? deg : fmod(deg + R(180.), R(360.));
}

// Largest USTAR of the points (non-negative values, ordered as their bit patterns).
template <typename R>
__global__ void __launch_bounds__(256) ustar_max_kernel(const R* __restrict__ ustar, int n, unsigned long long* out) {
  unsigned long long best = 0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const double u = (double)ustar[i];
    if (u > 0) best = max(best, (unsigned long long)__double_as_longlong(u));
  }
  for (int o = 16; o > 0; o >>= 1) best = max(best, __shfl_xor_sync(0xffffffffu, best, o));
  if ((threadIdx.x & 31) == 0 && best) atomicMax(out, best);
}

// The integrals of one spectrum from its frequency sums Tm[m * 32] (directions
// summed in order) and direction sums Tk[k * 32] (DFIM-weighted, frequencies in
// order), in three independent parts for different warps.  TOTAL_ENERGY, FEMEAN
// and TM1_TM2_PERIODS: Hs, TM, TM1, TM2 to the rows p0.. (p0 + 2..4).
template <typename R, class Put>
__device__ __forceinline__ void energy_part(const OutArgs<R>& a, const R* Tm, const Put& put, int phs, int ptm) {
  const int ml = a.ML;
  const R tail = Tm[(ml - 1) * 32];
  R E = a.MO_TAIL * tail, FM = a.MM1_TAIL * tail, TM1 = a.MP1_TAIL * tail, TM2 = a.MP2_TAIL * tail;
  for (int m = 0; m < ml; ++m) {
    const R t = Tm[m * 32];
    E = E + t * a.DFIM[m];
    FM = FM + t * a.DFIMOFR[m];
    TM1 = TM1 + t * a.DFIM_FR[m];
    TM2 = TM2 + t * a.DFIM_FR2[m];
  }
  E = dmax(E, R(1.0E-12));
  FM = E / dmax(FM, R(1.0E-12));
  put(phs, R(4.) * sqrt(E));
  put(ptm, R(1.) / FM);
  put(ptm + 1, (E > R(1.0E-12)) ? E / TM1 : R(1.));
  put(ptm + 2, (E > R(1.0E-12)) ? sqrt(E / TM2) : R(1.));
}

// PEAK_PERIOD: the first maximum of the frequency spectrum.
template <typename R> __device__ __forceinline__ R peak_part(const OutArgs<R>& a, const R* Tm) {
  int ip = 0;
  R best = Tm[0];
  for (int m = 1; m < a.ML; ++m) {
    const R t = Tm[m * 32];
    if (t > best) { best = t; ip = m; }
  }
  return ip == 0 ? R(1.) : R(1.) / a.FR[ip];
}

// MEAN_DIRECTION: direction and spread to the rows pd, pd + 1.
template <typename R, class Put>
__device__ __forceinline__ void direction_part(const OutArgs<R>& a, const R* Tk, const Put& put, int pd) {
  using P_ = Phys<R>;
  const R DEG = OutConst<R>::DEG;
  R SI = 0, CI = 0, SP = 0;
  for (int k = 0; k < a.KL; ++k) {
    const R t = Tk[k * 32];
    SI = SI + a.SINTH[k] * t;
    CI = CI + a.COSTH[k] * t;
    SP = SP + t;
  }
  {
    const R ci = (CI == R(0.)) ? R(0.1E-30) : CI;
    R thq = atan2(SI, ci);
    if (thq < R(0.)) thq = thq + P_::ZPI;
    if (thq > P_::ZPI - R(0.001)) thq = R(0.);
    put(pd, orient(thq * DEG, a.from));
  }
  {
    const R lim = R(0.1E-15);
    const R ci = (dabs(CI) < lim) ? copysign(lim, CI) : CI;
    const R si = (dabs(SI) < lim) ? copysign(lim, SI) : SI;
    R sp = (dabs(SP) < lim) ? copysign(lim, SP) : SP;
    sp = R(2.) * (R(1.) - sqrt(si * si + ci * ci) / sp);
    sp = (sp <= R(0)) ? (sizeof(R) == 4 ? R(FLT_MIN) : R(DBL_MIN)) : sqrt(sp);  // TINY(1.)
    put(pd + 1, sp * DEG);
  }
}

template <typename R>
__global__ void __launch_bounds__(kOutWarps * 32) output_kernel(const __grid_constant__ OutArgs<R> a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int ij = min((int)blockIdx.x * 32 + lane, a.nsea - 1);
  const bool real = (int)blockIdx.x * 32 + lane < a.nsea;
  const int kl = a.KL, ml = a.ML;
  using P_ = Phys<R>;
  const R DEG = OutConst<R>::DEG;
  R* Tk = reinterpret_cast<R*>(smem_raw) + lane;  // [k * 32]: direction sums over frequency
  R* Tm = Tk + kl * 32;                           // [m * 32]: frequency spectrum (sum over directions)
  R* X = Tm + ml * 32;                            // twice six frequencies of the spectrum
  R* DF = X + 2 * kOutWarps * kl * 32 - lane;     // DFIM
  for (int m = threadIdx.x; m < ml; m += kOutWarps * 32) DF[m] = a.DFIM[m];
  __syncthreads();
  // six frequencies on their way while six are summed
  auto load = [&](int m0, int buf) {
    if (m0 + w < ml) {
      const R* fm = a.fl3 + ij + (size_t)a.ld * kl * (m0 + w);
      unsigned x = (unsigned)__cvta_generic_to_shared(X + (buf * kOutWarps + w) * kl * 32);
#pragma unroll 4
      for (int k = 0; k < kl; ++k, fm += a.ld, x += 32 * sizeof(R))
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(x), "l"(fm), "n"(sizeof(R)) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  load(0, 0);
  for (int m0 = 0, buf = 0; m0 < ml; m0 += kOutWarps, buf ^= 1) {
    load(m0 + kOutWarps, buf ^ 1);
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();
    const int nm = min(kOutWarps, ml - m0);
    const R* x = X + buf * kOutWarps * kl * 32;
    if (w < nm) {
      R s = R(0);
#pragma unroll 12
      for (int k = 0; k < kl; ++k) s = s + x[(w * kl + k) * 32];
      Tm[(m0 + w) * 32] = s;
    }
    for (int k = w; k < kl; k += kOutWarps) {
      R t = m0 == 0 ? R(0) : Tk[k * 32];
#pragma unroll
      for (int j = 0; j < kOutWarps; ++j)
        if (j < nm) t = t + x[(j * kl + k) * 32] * DF[m0 + j];
      Tk[k * 32] = t;
    }
    __syncthreads();
  }
  R* out = a.block + ij;
  auto put = [&](int p, R v) { if (real) out[(size_t)a.block_ld * (p - 1)] = v; };
  if (w == 0) {
    energy_part(a, Tm, put, 9, 11);
  } else if (w == 1) {
    put(10, peak_part(a, Tm));
  } else if (w == 2) {
    direction_part(a, Tk, put, 14);
  } else if (w == 3) {  // MEANSQS
    R SM = R(1.0E-33);  // MAX(CONST2*TEMP(ML), EPSMIN) with CONST2 = 0.*LOG(FC/FS) = 0
    const int jd = a.shallow ? a.indep[ij] - 1 : 0;
    for (int m = 0; m < ml; ++m) {
      const R t = Tm[m * 32];
      if (a.shallow) {
        const R tk = __ldg(&a.TFAK[jd + a.NDEPTH * m]);
        SM = SM + a.DFIM[m] * (tk * tk) * t;
      } else {
        SM = SM + a.MSSFD[m] * t;
      }
    }
    put(40, SM);
  } else if (w == 4) {
    R U10 = a.u10[ij], UDIR = a.udir[ij], TAUW = a.tauw[ij];
    R USTAR = a.ustar[ij], Z0 = a.z0[ij];
    if (a.ustar_max && *a.ustar_max == 0ull) {
      // IF (MAXVAL(USTAR(:)).EQ.0.) CALL AIRSEA (U10, TAUW, USTAR, Z0)
      adj::airsea<R, R>(a.A, U10, TAUW, USTAR, Z0);
      if (real) { a.ustar[ij] = USTAR; a.z0[ij] = Z0; }
    }
    put(1, U10);
    put(2, orient(DEG * UDIR, a.from));
    put(3, USTAR);
    const R TAU = USTAR * USTAR + R(0.0001);
    put(4, TAU / (U10 * U10 + R(0.01)));
    put(16, TAUW / (TAU * P_::ROAIR));
    put(5, P_::G * Z0 / dmax(USTAR * USTAR, R(1.0E-6)));
    put(32, Z0);
  } else {
    put(6, a.shallow ? a.depth[ij] : R(999.));
    const R cu = a.u ? a.u[ij] : R(0), cv = a.v ? a.v[ij] : R(0);
    put(7, sqrt(cu * cu + cv * cv));
    R cdir = orient(atan2(cu, cv) * DEG, a.from);
    if (cdir < R(0.)) cdir = cdir + R(360.);
    put(8, cdir);
    // parameters that are not computed stay 0
    for (int p = 17; p < 40; ++p)
      if (p != 32) put(p, R(0));
  }
}

// SWELL_SEPARATION (wam_swell_module.f90:106-350) without the partitioning
// (parameters 41-49).  A bin is swell where FRIC/C(M) * 1.2*USTAR*COS(TH(K)-UDIR)
// < 1, its swell value MAX(F, EPSMIN) there and 0 elsewhere, its wind-sea value
// F minus that.  The cosine is the correctly rounded single-precision value (the
// oracle forms it the same way, so both split every bin alike).  The frequency
// sums of both spectra still add their directions in order, the direction sums
// their frequencies in order.  Parameters 17-23 (wind sea) and 25-31 (swell):
// Hs, peak period, mean period, TM1, TM2, mean direction, spread.
template <typename R>
__global__ void __launch_bounds__(kOutWarps * 32) swell_kernel(const __grid_constant__ OutArgs<R> a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int ij = min((int)blockIdx.x * 32 + lane, a.nsea - 1);
  const bool real = (int)blockIdx.x * 32 + lane < a.nsea;
  const int kl = a.KL, ml = a.ML;
  R* Tk1 = reinterpret_cast<R*>(smem_raw) + lane;  // swell direction sums
  R* Tk4 = Tk1 + kl * 32;                          // wind-sea direction sums
  R* Tm1 = Tk4 + kl * 32;                          // swell frequency sums
  R* Tm4 = Tm1 + ml * 32;                          // wind-sea frequency sums
  R* FP = Tm4 + ml * 32;                           // 1.2*USTAR*COS(TH(K)-UDIR)
  R* CM = FP + kl * 32 - lane;                     // FRIC/C(M)
  const R FRIC = R(28.), EPSMIN = R(0.1E-32);
  const R us = a.ustar[ij], ud = a.udir[ij];
  for (int k = w; k < kl; k += kOutWarps) FP[k * 32] = R(1.2) * us * crcos(a.TH[k] - ud);
  R* DF = CM + ml;                                 // DFIM
  for (int m = threadIdx.x; m < ml; m += kOutWarps * 32) { CM[m] = FRIC / a.C[m]; DF[m] = a.DFIM[m]; }
  __syncthreads();
  const R* f = a.fl3 + ij;
  for (int m = w; m < ml; m += kOutWarps) {
    const R* fm = f + (size_t)a.ld * kl * m;
    const R cm = CM[m];
    R s1 = R(0), s4 = R(0);
#pragma unroll 12
    for (int k = 0; k < kl; ++k, fm += a.ld) {
      const R v = __ldg(fm);
      const R f1 = (cm * FP[k * 32] < R(1.0)) ? dmax(v, EPSMIN) : R(0.);
      s1 = s1 + f1;
      s4 = s4 + (v - f1);
    }
    Tm1[m * 32] = s1;
    Tm4[m * 32] = s4;
  }
  for (int k = w; k < kl; k += kOutWarps) {
    const R* fk = f + (size_t)a.ld * k;
    const size_t step = (size_t)a.ld * kl;
    const R flpp = FP[k * 32];
    R t1 = R(0), t4 = R(0);
#pragma unroll 10
    for (int m = 0; m < ml; ++m, fk += step) {
      const R v = __ldg(fk), df = DF[m];
      const R f1 = (CM[m] * flpp < R(1.0)) ? dmax(v, EPSMIN) : R(0.);
      t1 = t1 + f1 * df;
      t4 = t4 + (v - f1) * df;
    }
    Tk1[k * 32] = t1;
    Tk4[k * 32] = t4;
  }
  __syncthreads();
  R* out = a.block + ij;
  auto put = [&](int p, R v) { if (real) out[(size_t)a.block_ld * (p - 1)] = v; };
  // even warps the wind sea, odd ones the swell
  const bool swell = w & 1;
  const R* Tm = swell ? Tm1 : Tm4;
  const int p = swell ? 25 : 17;
  if (w < 2) energy_part(a, Tm, put, p, p + 2);
  else if (w < 4) put(p + 1, peak_part(a, Tm));
  else direction_part(a, swell ? Tk1 : Tk4, put, p + 5);
}

template <typename R> size_t output_smem(int KL, int ML) { return (size_t)(32 * ((1 + 2 * kOutWarps) * KL + ML) + ML) * sizeof(R); }
template <typename R> size_t swell_smem(int KL, int ML) { return (size_t)(32 * (3 * KL + 2 * ML) + 2 * ML) * sizeof(R); }

}  // namespace

template <typename R> cudaError_t launch_swell(const OutArgs<R>& a, cudaStream_t s) {
  if (a.nsea == 0) return cudaSuccess;
  const size_t smem = swell_smem<R>(a.KL, a.ML);
  if (smem > 48 * 1024) {  // the limit belongs to the current device
    cudaError_t e = cudaFuncSetAttribute(swell_kernel<R>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)swell_smem<R>(MAX_KL, MAX_ML));
    if (e != cudaSuccess) return e;
  }
  swell_kernel<R><<<(a.nsea + 31) / 32, kOutWarps * 32, smem, s>>>(a);
  return cudaGetLastError();
}
template cudaError_t launch_swell<float>(const OutArgs<float>&, cudaStream_t);
template cudaError_t launch_swell<double>(const OutArgs<double>&, cudaStream_t);

// PUT_ICE / PUT_DRY: rows of the listed sea points set to a value.  One
// thread per (row, listed point): the list is short and scattered, each
// thread writes one element.
template <typename R>
__global__ void __launch_bounds__(256) put_points_kernel(R* __restrict__ data, size_t ld, int nrows,
                                                         const int* __restrict__ points, int n, int lo, int hi, R value) {
  const size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (t >= (size_t)n * nrows) return;
  const int i = (int)(t % n), row = (int)(t / n);
  const int ij = points[i];  // 1-based sea point number
  if (ij < lo || ij > hi) return;
  data[(size_t)(ij - 1) + ld * row] = value;
}

template <typename R>
cudaError_t launch_put_points(R* data, size_t ld, int nrows, const int* points, int n, int lo, int hi, R value,
                              cudaStream_t s) {
  const size_t total = (size_t)n * nrows;
  if (total == 0) return cudaSuccess;
  put_points_kernel<R><<<(unsigned)((total + 255) / 256), 256, 0, s>>>(data, ld, nrows, points, n, lo, hi, value);
  return cudaGetLastError();
}
template cudaError_t launch_put_points<float>(float*, size_t, int, const int*, int, int, int, float, cudaStream_t);
template cudaError_t launch_put_points<double>(double*, size_t, int, const int*, int, int, int, double, cudaStream_t);

// WAM_WIND (wam_wind_module.f90:1063-1216): one input wind field to the sea
// points.  Bilinear interpolation with the tables of INTERPOLATION_TO_GRID
// (:1224-1377; a plain copy on the model's own grid, EQUAL_GRID), then speed
// and direction ATAN2(U,V) in [0, 2*pi), the friction-velocity (CODE_IN 1)
// or surface-stress (2) input turned into U10 through a Charnock drag, and
// U10 >= 2 m/s.  One thread per sea point; the unit rounds every operation
// separately, as the reference does.
template <typename R>
__global__ void __launch_bounds__(256) wind_kernel(const R* __restrict__ u_in, const R* __restrict__ v_in, int nx_in,
                                                   int n, const int* __restrict__ tab, const R* __restrict__ w, int equal,
                                                   int code_in, R* __restrict__ us, R* __restrict__ ds) {
  const int ij = blockIdx.x * blockDim.x + threadIdx.x;
  if (ij >= n) return;
  const int i1 = tab[ij] - 1, i2 = tab[ij + n] - 1, k1 = tab[ij + 2 * n] - 1, k2 = tab[ij + 3 * n] - 1;
  auto at = [&](const R* f, int i, int k) { return __ldg(&f[i + (size_t)nx_in * k]); };
  R uu, vv;
  if (equal) {
    uu = at(u_in, i1, k1);
    vv = at(v_in, i1, k1);
  } else {
    const R di = w[ij], dk = w[ij + n];
    uu = (at(u_in, i1, k1) * (R(1.) - di) + at(u_in, i2, k1) * di) * (R(1.) - dk) +
         (at(u_in, i1, k2) * (R(1.) - di) + at(u_in, i2, k2) * di) * dk;
    vv = (at(v_in, i1, k1) * (R(1.) - di) + at(v_in, i2, k1) * di) * (R(1.) - dk) +
         (at(v_in, i1, k2) * (R(1.) - di) + at(v_in, i2, k2) * di) * dk;
  }
  R s = sqrt(uu * uu + vv * vv);
  R d = (s != R(0.)) ? atan2(uu, vv) : R(0.);
  if (d < R(0.)) d = d + Phys<R>::ZPI;
  if (code_in == 1 || code_in == 2) {
    const R alphach = R(0.0185);
    const R ust = code_in == 1 ? dmax(R(0.01), s) : dmax(R(0.01), sqrt(s / Phys<R>::ROAIR));
    const R z0 = alphach / Phys<R>::G * (ust * ust);
    const R cd = Phys<R>::XKAPPA / log(R(10.) / z0);
    s = ust / cd;
  }
  us[ij] = dmax(s, R(2.0));
  ds[ij] = d;
}

template <typename R>
cudaError_t launch_wind(const R* u_in, const R* v_in, int nx_in, int n, const int* tab, const R* w, int equal,
                        int code_in, R* us, R* ds, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  wind_kernel<R><<<(n + 255) / 256, 256, 0, s>>>(u_in, v_in, nx_in, n, tab, w, equal, code_in, us, ds);
  return cudaGetLastError();
}
template cudaError_t launch_wind<float>(const float*, const float*, int, int, const int*, const float*, int, int, float*,
                                        float*, cudaStream_t);
template cudaError_t launch_wind<double>(const double*, const double*, int, int, const int*, const double*, int, int,
                                         double*, double*, cudaStream_t);

// Restart records: rows b0..b0+nb-1 of a sea-point-fastest device array
// gathered into REAL file order (file position p holds model point perm[p],
// 1-based; perm null = the identity) and scattered back.
template <typename R>
__global__ void __launch_bounds__(256) restart_gather_kernel(const R* __restrict__ src, size_t ld, int nsea,
                                                             const int* __restrict__ perm, int b0, int nb,
                                                             float* __restrict__ out) {
  const size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (t >= (size_t)nsea * nb) return;
  const int p = (int)(t % nsea), b = b0 + (int)(t / nsea);
  const int ij = perm ? perm[p] - 1 : p;
  out[t] = (float)src[ij + ld * b];
}
template <typename R>
__global__ void __launch_bounds__(256) restart_scatter_kernel(const float* __restrict__ in, int nsea,
                                                              const int* __restrict__ perm, int b0, int nb,
                                                              R* __restrict__ dst, size_t ld) {
  const size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (t >= (size_t)nsea * nb) return;
  const int p = (int)(t % nsea), b = b0 + (int)(t / nsea);
  const int ij = perm ? perm[p] - 1 : p;
  dst[ij + ld * b] = (R)in[t];
}
template <typename R>
cudaError_t launch_restart_gather(const R* src, size_t ld, int nsea, const int* perm, int b0, int nb, float* out,
                                  cudaStream_t s) {
  const size_t n = (size_t)nsea * nb;
  if (n == 0) return cudaSuccess;
  restart_gather_kernel<R><<<(unsigned)((n + 255) / 256), 256, 0, s>>>(src, ld, nsea, perm, b0, nb, out);
  return cudaGetLastError();
}
template <typename R>
cudaError_t launch_restart_scatter(const float* in, int nsea, const int* perm, int b0, int nb, R* dst, size_t ld,
                                   cudaStream_t s) {
  const size_t n = (size_t)nsea * nb;
  if (n == 0) return cudaSuccess;
  restart_scatter_kernel<R><<<(unsigned)((n + 255) / 256), 256, 0, s>>>(in, nsea, perm, b0, nb, dst, ld);
  return cudaGetLastError();
}
template cudaError_t launch_restart_gather<float>(const float*, size_t, int, const int*, int, int, float*, cudaStream_t);
template cudaError_t launch_restart_gather<double>(const double*, size_t, int, const int*, int, int, float*, cudaStream_t);
template cudaError_t launch_restart_scatter<float>(const float*, int, const int*, int, int, float*, size_t, cudaStream_t);
template cudaError_t launch_restart_scatter<double>(const float*, int, const int*, int, int, double*, size_t,
                                                    cudaStream_t);

template <typename R> cudaError_t launch_output(const OutArgs<R>& a, unsigned long long* ustar_max, cudaStream_t s) {
  if (a.nsea == 0) return cudaSuccess;
  OutArgs<R> b = a;
  b.ustar_max = nullptr;
  if (ustar_max) {
    cudaError_t e = cudaMemsetAsync(ustar_max, 0, sizeof(unsigned long long), s);
    if (e != cudaSuccess) return e;
    ustar_max_kernel<R><<<148, 256, 0, s>>>(a.ustar, a.nsea, ustar_max);
    b.ustar_max = ustar_max;
  }
  const size_t smem = output_smem<R>(a.KL, a.ML);
  if (smem > 48 * 1024) {  // the limit belongs to the current device
    cudaError_t e = cudaFuncSetAttribute(output_kernel<R>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)output_smem<R>(MAX_KL, MAX_ML));
    if (e != cudaSuccess) return e;
  }
  output_kernel<R><<<(a.nsea + 31) / 32, kOutWarps * 32, smem, s>>>(b);
  return cudaGetLastError();
}

template cudaError_t launch_output<float>(const OutArgs<float>&, unsigned long long*, cudaStream_t);
template cudaError_t launch_output<double>(const OutArgs<double>&, unsigned long long*, cudaStream_t);

}  // namespace wamgpu
