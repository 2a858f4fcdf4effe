// temperature_kernel.cu -- the radiative-equilibrium gas temperature that
// ends transport::step (src/transport/solve_equilibrium.cpp:66-96, LTE).
//
// The lanes of a zone (a CTA, a warp or one thread: temperature_lanes) run
// temp_brent_method (:227-320) on rad_eq_function_LTE with solve_flag 0
// (:113-170): the zone's emission sum_i 4 pi kappa_abs,i B_nu(T) dnu_i, with
// the absorption opacities of the last opacity build, minus its normalised
// absorbed-energy tally e_abs.  Every lane holds the same iterates; an
// evaluation is split over the lanes by frequency bin and summed in a fixed
// tree, so the result is the same from run to run.  Compiled without FMA
// contraction like the rest.
//
// What bounds it: one FP64 exp and one FP64 division per bin and evaluation
// (20-40 evaluations), and the root search between evaluations, which every
// lane repeats.  One thread per zone waits on the chain exp -> divide -> add
// of every bin and leaves the chip idle but for ceil(zones / 128) CTAs: on
// B200, a CTA per zone against that, 256 zones x 4096 bins 74.4 ms -> 171 us,
// 97 x 1500 25.9 ms -> 74 us, 128 x 1024 17.6 ms -> 57 us (about 30 evaluations
// of a few hundred nanoseconds' chain each).  With few bins the search is what
// counts, and a CTA repeats it 256 times.
#include <cmath>
#include "sed_internal.h"

namespace sed {

namespace {

// Lanes that share a zone: a whole CTA of TEMP_THREADS, a warp, or one thread.
constexpr int TEMP_THREADS = 256;
constexpr int TEMP_BLOCK = 128;  // CTA size of the warp and thread forms
// The T-independent factors of a bin, h nu / k and 4 pi kappa 2 h nu^3/c^2 dnu
// (16 B), are formed once and kept in shared memory up to this many bins
// (96 KB: two CTAs per SM); beyond it, and where a thread holds the zone
// alone, every evaluation forms them again.
constexpr int TEMP_SMEM_BINS = 6144;

template <typename OT>
__device__ __forceinline__ double2 bin_factors(const OT* __restrict__ row, const DevLoc& nu, int i)
{
  const double nc = loc_center(nu, i);
  const double b = 2.0 * nc * nc * nc * H_PLANCK / C_LIGHT / C_LIGHT;  // transport_opacity.cpp:322-326
  return make_double2(H_PLANCK * nc / K_BOLTZ, 4.0 * PI * (double)__ldg(&row[i].x) * b * loc_delta(nu, i));
}

// the zone's emission minus its absorption at temperature T, the same value
// in every lane of the zone.  The CTA's partial sums alternate between two
// buffers, so one barrier per evaluation is enough: a thread can only reach the
// second evaluation from here, which writes this buffer again, past a barrier
// every thread has arrived at after reading it.
template <typename OT, int LANES>
__device__ double rad_eq_lte(const OT* __restrict__ row, const DevLoc& nu, const double2* __restrict__ s_fac,
                             bool cached, double e_abs, double T, double (*red)[TEMP_THREADS / 32], int& buf)
{
  if (nu.n == 1) return 4.0 * PI * (double)row[0].x * SB / PI * pow(T, 4) - e_abs;
  const double inv_T = 1.0 / T;
  double sum = 0;
  for (int i = threadIdx.x % LANES; i < nu.n; i += LANES) {
    const double2 f = (LANES > 1 && cached) ? s_fac[i] : bin_factors<OT>(row, nu, i);
    sum += f.y / (exp(f.x * inv_T) - 1);
  }
  if constexpr (LANES >= 32) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  }
  if constexpr (LANES > 32) {
    if ((threadIdx.x & 31) == 0) red[buf][threadIdx.x >> 5] = sum;
    __syncthreads();
    sum = 0.;
#pragma unroll
    for (int w = 0; w < LANES / 32; ++w) sum += red[buf][w];
    buf ^= 1;
  }
  return sum - e_abs;
}

template <typename OT, int LANES>
__global__ void __launch_bounds__(LANES > 32 ? LANES : TEMP_BLOCK) temperature_kernel(const TemperatureArgs A)
{
  extern __shared__ double2 s_all[];
  __shared__ double red[2][TEMP_THREADS / 32];
  const int c = (LANES > 32) ? (int)blockIdx.x : (int)(blockIdx.x * (TEMP_BLOCK / LANES) + threadIdx.x / LANES);
  if (c >= A.nz) return;  // whole warps of the warp form; the CTA form has a CTA per zone
  const bool lead = threadIdx.x % LANES == 0;
  if (A.set_Tgas_to_Trad) {
    if (lead) A.T[c] = pow(A.e_rad[c] / A_RAD, 0.25);
    return;
  }
  const OT* row = reinterpret_cast<const OT*>(A.opac) + (size_t)c * A.nu.n;
  const double e_abs = A.e_abs[c];
  const bool cached = LANES > 1 && A.nu.n > 1 && A.nu.n <= TEMP_SMEM_BINS;
  double2* s_fac = s_all;
  if constexpr (LANES == 32) s_fac += (threadIdx.x / 32) * A.nu.n;
  // a thread reads back only the entries it writes here: no barrier
  if (cached)
    for (int i = threadIdx.x % LANES; i < A.nu.n; i += LANES) s_fac[i] = bin_factors<OT>(row, A.nu, i);
  int buf = 0;
  auto f = [&](double T) { return rad_eq_lte<OT, LANES>(row, A.nu, s_fac, cached, e_abs, T, red, buf); };
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

template <typename OT, int LANES>
int launch_lanes(const TemperatureArgs& a, cudaStream_t s)
{
  constexpr int threads = LANES > 32 ? LANES : TEMP_BLOCK, zones = threads / LANES;
  const bool cached = LANES > 1 && a.nu.n > 1 && a.nu.n <= TEMP_SMEM_BINS;
  const size_t smem = cached ? (size_t)zones * a.nu.n * sizeof(double2) : 0;
  if (smem > 48 * 1024 &&
      cudaFuncSetAttribute(temperature_kernel<OT, LANES>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
          cudaSuccess)
    return -1;
  temperature_kernel<OT, LANES><<<(a.nz + zones - 1) / zones, threads, smem, s>>>(a);
  return 1;
}

// The lanes a zone takes.  sed_solve_temperature on B200 in ms, FP64 (FP32
// tables the same within 5 %), copies and launch included:
//      zones x bins   CTA    warp   thread
//    262 144 x 1      23.8    3.4    0.56     64 000 x 1     5.8   0.90  0.20
//    262 144 x 8      16.5    2.7    0.91     64 000 x 8     4.1   0.73  0.33
//    262 144 x 32     16.4    2.7    2.2      64 000 x 32    4.1   0.76  0.81
//    262 144 x 128    18.0    4.7    7.4      64 000 x 512   6.4   3.4
//      8 000 x 8       0.56   0.15   0.18      1 000 x 32    0.12  0.07  0.46
//      8 000 x 512     0.85   0.52             1 000 x 128   0.155 0.113
//      8 000 x 2048    1.84   6.1              1 000 x 512   0.18  0.20
//         64 x 8       0.08   0.07   0.17         64 x 128   0.08  0.11
// A thread, as soon as enough zones fill the chip with threads to cover its
// chain of bins; a warp up to where its share of the bins outweighs the idle
// warps of a CTA (more zones, more bins) and while its factors in shared memory
// (64 B a bin and CTA) leave room for other warps; a CTA beyond.
int temperature_lanes(int nz, int nn, bool to_trad, int num_sms)
{
  if (nn == 1 || to_trad) return 1;
  if (nn <= 32) return nz >= (int64_t)14 * num_sms * nn ? 1 : 32;
  return (nn <= 512 && nz >= (int64_t)num_sms * nn / 32) ? 32 : TEMP_THREADS;
}

template <typename OT>
int launch_t(const TemperatureArgs& a, int num_sms, cudaStream_t s)
{
  const int l = temperature_lanes(a.nz, a.nu.n, a.set_Tgas_to_Trad != 0, num_sms);
  return l == 1 ? launch_lanes<OT, 1>(a, s) : l == 32 ? launch_lanes<OT, 32>(a, s) : launch_lanes<OT, TEMP_THREADS>(a, s);
}

}  // namespace

int launch_temperature(const TemperatureArgs& a, int num_sms, cudaStream_t s)
{
  if (a.nz <= 0) return 0;
  return a.precision ? launch_t<float2>(a, num_sms, s) : launch_t<double2>(a, num_sms, s);
}

}  // namespace sed
