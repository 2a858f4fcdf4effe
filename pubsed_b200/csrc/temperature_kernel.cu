// temperature_kernel.cu -- the radiative-equilibrium gas temperature that
// ends transport::step (src/transport/solve_equilibrium.cpp:66-96, LTE).
//
// One CTA per zone runs temp_brent_method (:227-320) on rad_eq_function_LTE
// with solve_flag 0 (:113-170): the zone's emission
// sum_i 4 pi kappa_abs,i B_nu(T) dnu_i, with the absorption opacities of
// the last opacity build, minus its normalised absorbed-energy tally e_abs.
// Every thread of the CTA holds the same iterates; an evaluation is split
// over the threads by frequency bin and summed in a fixed tree, so the
// result is the same from run to run.  Compiled without FMA contraction like
// the rest.
//
// What bounds it: one FP64 exp and one FP64 division per bin and evaluation
// (20-40 evaluations).  One thread per zone, the bins in order, left the chip
// idle but for ceil(zones / 128) CTAs and waited on the chain exp -> divide ->
// add of every bin.  On B200: 256 zones x 4096 bins 74.4 ms -> 171 us, 97 x
// 1500 25.9 ms -> 74 us, 128 x 1024 17.6 ms -> 57 us (about 30 evaluations of
// a few hundred nanoseconds' chain each).
#include <cmath>
#include "sed_internal.h"

namespace sed {

namespace {

constexpr int TEMP_THREADS = 256;
// The T-independent factors of a bin, h nu / k and 4 pi kappa 2 h nu^3/c^2 dnu
// (16 B), are formed once and kept in shared memory up to this many bins
// (96 KB: two CTAs per SM); beyond it every evaluation forms them again.
constexpr int TEMP_SMEM_BINS = 6144;

template <typename OT>
__device__ __forceinline__ double2 bin_factors(const OT* __restrict__ row, const DevLoc& nu, int i)
{
  const double nc = loc_center(nu, i);
  const double b = 2.0 * nc * nc * nc * H_PLANCK / C_LIGHT / C_LIGHT;  // transport_opacity.cpp:322-326
  return make_double2(H_PLANCK * nc / K_BOLTZ, 4.0 * PI * (double)__ldg(&row[i].x) * b * loc_delta(nu, i));
}

// the zone's emission minus its absorption at temperature T, the same value
// in every thread.  The partial sums alternate between two buffers, so one
// barrier per evaluation is enough: a thread can only reach the second
// evaluation from here, which writes this buffer again, past a barrier every
// thread has arrived at after reading it.
template <typename OT>
__device__ double rad_eq_lte(const OT* __restrict__ row, const DevLoc& nu, const double2* __restrict__ s_fac,
                             bool cached, double e_abs, double T, double (*red)[TEMP_THREADS / 32], int& buf)
{
  if (nu.n == 1) return 4.0 * PI * (double)row[0].x * SB / PI * pow(T, 4) - e_abs;
  const double inv_T = 1.0 / T;
  double sum = 0;
  for (int i = threadIdx.x; i < nu.n; i += TEMP_THREADS) {
    const double2 f = cached ? s_fac[i] : bin_factors<OT>(row, nu, i);
    sum += f.y / (exp(f.x * inv_T) - 1);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  if ((threadIdx.x & 31) == 0) red[buf][threadIdx.x >> 5] = sum;
  __syncthreads();
  double E_emitted = 0.;
#pragma unroll
  for (int w = 0; w < TEMP_THREADS / 32; ++w) E_emitted += red[buf][w];
  buf ^= 1;
  return E_emitted - e_abs;
}

template <typename OT>
__global__ void __launch_bounds__(TEMP_THREADS) temperature_kernel(const TemperatureArgs A)
{
  extern __shared__ double2 s_fac[];
  __shared__ double red[2][TEMP_THREADS / 32];
  const int c = blockIdx.x;
  const bool lead = threadIdx.x == 0;
  if (A.set_Tgas_to_Trad) {
    if (lead) A.T[c] = pow(A.e_rad[c] / A_RAD, 0.25);
    return;
  }
  const OT* row = reinterpret_cast<const OT*>(A.opac) + (size_t)c * A.nu.n;
  const double e_abs = A.e_abs[c];
  const bool cached = A.nu.n <= TEMP_SMEM_BINS;
  // a thread reads back only the entries it writes here: no barrier
  if (cached && A.nu.n > 1)
    for (int i = threadIdx.x; i < A.nu.n; i += TEMP_THREADS) s_fac[i] = bin_factors<OT>(row, A.nu, i);
  int buf = 0;
  auto f = [&](double T) { return rad_eq_lte<OT>(row, A.nu, s_fac, cached, e_abs, T, red, buf); };
  const double brent_solve_tolerance = 1.0e-2;
  const int ITMAX = 100;
  const double EPS = 3.0e-8;
  double a = A.temp_min, b = A.temp_max, cc = b, d = 0, e = 0, min1, min2;
  double fa = f(a), fb = f(b);
  double fc, p, q, r, s, tol1, xm;
  fc = fb;
  for (int iter = 1; iter <= ITMAX; iter++) {
    if ((fb > 0.0 && fc > 0.0) || (fb < 0.0 && fc < 0.0)) { cc = a; fc = fa; e = d = b - a; }
    if (fabs(fc) < fabs(fb)) { a = b; b = cc; cc = a; fa = fb; fb = fc; fc = fa; }
    tol1 = 2.0 * EPS * fabs(b) + 0.5 * brent_solve_tolerance;
    xm = 0.5 * (cc - b);
    if (fabs(xm) <= tol1 || fb == 0.0) {
      if (lead) A.T[c] = b;
      return;
    }
    if (fabs(e) >= tol1 && fabs(fa) > fabs(fb)) {
      s = fb / fa;
      if (a == cc) { p = 2.0 * xm * s; q = 1.0 - s; }
      else {
        q = fa / fc;
        r = fb / fc;
        p = s * (2.0 * xm * q * (q - r) - (b - a) * (r - 1.0));
        q = (q - 1.0) * (r - 1.0) * (s - 1.0);
      }
      if (p > 0.0) q = -q;
      p = fabs(p);
      min1 = 3.0 * xm * q - fabs(tol1 * q);
      min2 = fabs(e * q);
      if (2.0 * p < (min1 < min2 ? min1 : min2)) { e = d; d = p / q; }
      else { d = xm; e = d; }
    } else { d = xm; e = d; }
    a = b;
    fa = fb;
    if (fabs(d) > tol1) b += d;
    else b += (xm >= 0.0 ? fabs(tol1) : -fabs(tol1));
    fb = f(b);
  }
  // the reference prints "Maximum number of iterations exceeded" and uses 0
  if (lead) {
    A.T[c] = 0.0;
    atomicAdd(A.n_unsolved, 1);
  }
}

template <typename OT>
int launch_t(const TemperatureArgs& a, cudaStream_t s)
{
  const size_t smem = (a.nu.n > 1 && a.nu.n <= TEMP_SMEM_BINS) ? (size_t)a.nu.n * sizeof(double2) : 0;
  if (smem > 48 * 1024 &&
      cudaFuncSetAttribute(temperature_kernel<OT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
          cudaSuccess)
    return -1;
  temperature_kernel<OT><<<a.nz, TEMP_THREADS, smem, s>>>(a);
  return 1;
}

}  // namespace

int launch_temperature(const TemperatureArgs& a, cudaStream_t s)
{
  if (a.nz <= 0) return 0;
  return a.precision ? launch_t<float2>(a, s) : launch_t<double2>(a, s);
}

}  // namespace sed
