// opacity_kernel.cu -- per-zone opacity/emissivity build on the device
// (transport::set_opacity, src/transport/transport_opacity.cpp:21-260).
//
//   zone_state_warp_kernel
//                       one warp per zone (zone_state_kernel, one thread,
//                       for very long level lists and many zones of short ones): temperature clamp, mass
//                       fractions, then the LTE electron-density solve
//                       (GasState::solve_state / ne_brent_method,
//                       src/opacity/GasState.cpp:208-337) with
//                       AtomicSpecies::solve_lte (AtomicSpecies_state.cpp:56-123).
//                       Boltzmann factors depend on T only and are computed
//                       once per zone instead of once per Brent iteration
//                       (same values, same rounding).
//   zone_opacity_kernel one CTA per zone: electron scattering, free-free,
//                       bound-free, Sobolev line and fuzz-line expansion
//                       opacity per frequency bin in the reference's order
//                       (GasState::computeOpacity, GasState_opacities.cpp:11-136),
//                       then the opacity cap, Planck/Rosseland means,
//                       emissivity CDF (cdf_array::set_value prefix sum, in
//                       the reference's order for FP64 grids up to 65536
//                       zones), L_thermal, Fleck factor and
//                       the packed tables the packet kernel reads.  The
//                       zone's level populations are staged in shared memory
//                       with their reciprocals, so a line costs two
//                       shared-memory reads, one 16 B and one 16 B (8 B in
//                       FP32) global load and no division.  Line lists are
//                       sorted by (bin, atom) with a stable sort, so each bin
//                       is one contiguous run in the reference's list order.
//                       In the mixed-precision form the per-line Sobolev sums
//                       run in FP32 with Kahan compensation; everything else
//                       stays FP64.
//
// The host runs the kernels once per chunk of zones: per-zone inputs and
// outputs are passed offset to the chunk, and every scratch array
// (index * nzones + zone) is sized for one chunk, so a 128^3-zone grid with
// thousands of bins builds its tables through a bounded working set.
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <mutex>
#include <type_traits>
#include "../../include/sedona_gpu.h"
#include "sed_internal.h"

namespace sed {
namespace {

// ------------------------------------------------------------ LTE
// Per-zone scratch is stored level-major / ion-major (index * nz + zone) so
// neighbouring threads (zones) touch neighbouring addresses.

// AtomicSpecies::solve_lte for atom a at electron density ne; partition
// functions `part` (ion-major scratch) and Boltzmann factors are cached.
__device__ void solve_lte_atom(const OpacityArgs& A, int z, int a, double ne, double T, const double* boltz_e,
                               double* part, double* frac, double* lev, int write_lev, double* net)
{
  const int nz = A.nzones;
  const int i0 = A.ion_off[a], ni = A.ion_off[a + 1] - i0;
  const int l0 = A.lev_off[a], nl = A.lev_off[a + 1] - l0;
  const double lt = H_PLANCK * H_PLANCK / (2.0 * PI * MASS_E * K_BOLTZ * T);
  const double fac = 2 / ne / pow(lt, 1.5);
  frac[(size_t)i0 * nz + z] = 1.;
  for (int i = 1; i < ni; ++i) {
    const double chi = A.ion_chi[i0 + i - 1];
    double saha = exp(-1.0 * chi / K_EV / T);
    saha = saha * (part[(size_t)(i0 + i) * nz + z] / part[(size_t)(i0 + i - 1) * nz + z]) * fac;
    double fi = saha * frac[(size_t)(i0 + i - 1) * nz + z];
    if (ne < 1e-50) fi = 0;
    frac[(size_t)(i0 + i) * nz + z] = fi;
    double norm = 0;
    for (int j = 0; j <= i; j++) norm += frac[(size_t)(i0 + j) * nz + z];
    for (int j = 0; j <= i; j++) frac[(size_t)(i0 + j) * nz + z] = frac[(size_t)(i0 + j) * nz + z] / norm;
  }
  double x = 0;
  for (int i = 0; i < nl; ++i) {
    const int ion = A.lev_ion[l0 + i];
    const double Z = part[(size_t)(i0 + ion) * nz + z];
    const double f = frac[(size_t)(i0 + ion) * nz + z];
    double v = f * A.lev_g[l0 + i] * boltz_e[(size_t)(l0 + i) * nz + z] / Z;
    if (v < 1e-30) v = 1e-30;
    if (write_lev) lev[(size_t)(l0 + i) * nz + z] = v;
    x += v * A.lev_ion[l0 + i];
  }
  *net = x;
}

__device__ double charge_conservation(const OpacityArgs& A, int z, double ne, double T, double dens,
                                      const double* boltz_e, int write_lev)
{
  double f = 0;
  for (int a = 0; a < A.natoms; ++a) {
    double net;
    solve_lte_atom(A, z, a, ne, T, boltz_e, A.ion_part, A.ion_frac, A.lev_n, write_lev, &net);
    f += dens * A.mass_frac[(size_t)a * A.nzones + z] / (A.eA[a] * MASS_P) * net;
  }
  return f - ne;
}

// GasState::ne_brent_method (GasState.cpp:270-337) on f(ne), the charge
// conservation of one zone; *last = last point evaluated
template <class F>
__device__ double ne_brent(F& f, double x1, double x2, double tol, double* last, int* err)
{
  const int ITMAX = 100;
  const double EPS = 3.0e-8;
  double a = x1, b = x2, c = x2, d = 0, e = 0, min1, min2;
  double fa = f(a);
  double fb = f(b);
  *last = b;
  double fc, p, q, r, s, tol1, xm;
  if ((fa > 0.0 && fb > 0.0) || (fa < 0.0 && fb < 0.0)) *err = 1;
  fc = fb;
  for (int iter = 1; iter <= ITMAX; iter++) {
    if ((fb > 0.0 && fc > 0.0) || (fb < 0.0 && fc < 0.0)) { c = a; fc = fa; e = d = b - a; }
    if (fabs(fc) < fabs(fb)) { a = b; b = c; c = a; fa = fb; fb = fc; fc = fa; }
    tol1 = 2.0 * EPS * fabs(b) + 0.5 * tol;
    xm = 0.5 * (c - b);
    if (fabs(xm) <= tol1 || fb == 0.0) return b;
    if (fabs(e) >= tol1 && fabs(fa) > fabs(fb)) {
      s = fb / fa;
      if (a == c) { p = 2.0 * xm * s; q = 1.0 - s; }
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
    b += (fabs(d) > tol1) ? d : (xm >= 0.0 ? fabs(tol1) : -fabs(tol1));
    fb = f(b);
    *last = b;
  }
  *err = 2;
  return 0.0;
}

// a zone's clamped temperature, mass fractions (GasState::set_mass_fractions,
// GasState.cpp:137-156) and mean ion mass number
__device__ __forceinline__ double zone_temperature(const OpacityArgs& A, int z)
{
  double T = A.T[z];
  if (T < A.temp_min) T = A.temp_min;
  if (T > A.temp_max) T = A.temp_max;
  return T;
}

__device__ __forceinline__ double zone_mass_fractions(const OpacityArgs& A, int z, bool write)
{
  double norm = 0.0;
  for (int a = 0; a < A.nelem; ++a) norm += A.X[(size_t)z * A.nelem + a];
  double inv = 0.;
  for (int a = 0; a < A.nelem; ++a) {
    const double mf = A.X[(size_t)z * A.nelem + a] / norm;
    if (write) A.mass_frac[(size_t)a * A.nzones + z] = mf;
    inv += mf / A.eA[a];
  }
  return 1. / inv;
}

// One thread per zone: the form for level lists too long for the shared
// memory of zone_state_warp_kernel, and for many zones of short ones
// (zone_state_by_thread).
__global__ void zone_state_kernel(const OpacityArgs A, double* boltz_e)
{
  const int z = blockIdx.x * blockDim.x + threadIdx.x;
  const int nz = A.nzones;
  if (z >= nz) return;
  const double T = zone_temperature(A, z);
  A.temp_c[z] = T;
  const double dens = A.rho[z];
  const double mu_I = zone_mass_fractions(A, z, true);
  A.solve_err[z] = 0;
  if (A.grey[z] != 0 || A.natoms == 0) { A.n_elec[z] = 0; return; }
  for (int a = 0; a < A.natoms; ++a)
    A.n_dens[(size_t)a * nz + z] = dens * A.mass_frac[(size_t)a * nz + z] / (A.eA[a] * MASS_P);
  // Boltzmann factors exp(-E/kT) and partition functions: T only
  for (int a = 0; a < A.natoms; ++a) {
    const int i0 = A.ion_off[a], ni = A.ion_off[a + 1] - i0;
    const int l0 = A.lev_off[a], nl = A.lev_off[a + 1] - l0;
    for (int i = 0; i < ni; ++i) A.ion_part[(size_t)(i0 + i) * nz + z] = 0;
    for (int i = 0; i < nl; ++i) {
      const double eb = exp(-A.lev_E[l0 + i] / K_EV / T);
      boltz_e[(size_t)(l0 + i) * nz + z] = eb;
      const int ion = A.lev_ion[l0 + i];
      A.ion_part[(size_t)(i0 + ion) * nz + z] += A.lev_g[l0 + i] * eb;
    }
  }
  const double max_ne = 100 * dens / (mu_I * MASS_P);
  const double min_ne = 1e-10 * dens / (mu_I * MASS_P);
  double last = 0;
  int err = 0;
  auto f = [&](double ne) { return charge_conservation(A, z, ne, T, dens, boltz_e, 0); };
  const double ne = ne_brent(f, min_ne, max_ne, 1e-3, &last, &err);
  charge_conservation(A, z, last, T, dens, boltz_e, 1);  // populations of the last evaluation
  A.n_elec[z] = ne;
  A.solve_err[z] = err;
}

// One warp per zone, ZONE_WARPS neighbouring zones per CTA, the zone's LTE
// state in shared memory.  What bounds the solve is a chain: some 30 Brent
// evaluations, each a pass over the ion stages and the levels.  One thread per
// zone walked that chain alone, its state in global scratch: 2.2 ms for any
// 1D model (one or two CTAs at work).  Here the lanes share the levels, lane a
// the stages and the sum of atom a.
//
// The per-level terms, the stage recursion of each atom and every sum are the
// reference's, in its order, so the FP64 form's populations are the same to
// the bit.  With FP32 tables (FAST) an evaluation takes the mean charge of an
// atom from its stage fractions, sum_i i f_i, instead of summing v_l i over
// the levels: the level populations of a stage add up to f_i by construction,
// so the two differ by rounding, and by the floor of 1e-30 per level, which
// is below 1e-15 of any n_e inside the solver's bracket (n_e >= 1e-10 of the
// ions).  An evaluation is then a dozen operations per stage instead of two
// dozen per level.  On B200, against one thread per zone: 256 zones x 606
// levels 2.2 ms -> 63 us (FP64 132 us), 18 494 zones 3.8 ms -> 344 us, 64^3
// zones x 906 levels 18.7 -> 6.0 ms.
constexpr int ZONE_WARPS = 4;  // 4 zones x 8 B: the CTA's level-major results fill whole 32 B sectors

// doubles of shared memory per zone
__host__ __device__ inline size_t zone_state_doubles(bool fast, int na, int ni, int nl)
{
  return (size_t)(fast ? 1 : 2) * nl + 3 * (size_t)ni + 2 * (size_t)na;
}

// stage fractions of atom a at electron density ne (AtomicSpecies::solve_lte,
// AtomicSpecies_state.cpp:70-90): c[i] = exp(-chi/kT) part_i / part_(i-1)
__device__ __forceinline__ void stage_fractions(double* fr, const double* c, int ni, double ne, double fac)
{
  fr[0] = 1.;
  for (int i = 1; i < ni; ++i) {
    double fi = c[i] * fac * fr[i - 1];
    if (ne < 1e-50) fi = 0;
    fr[i] = fi;
    double norm = 0;
    for (int j = 0; j <= i; j++) norm += fr[j];
    for (int j = 0; j <= i; j++) fr[j] = fr[j] / norm;
  }
}

template <bool FAST>
__global__ void __launch_bounds__(32 * ZONE_WARPS) zone_state_warp_kernel(const OpacityArgs A)
{
  extern __shared__ double zsm[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nz = A.nzones, na = A.natoms, nI = A.n_ions_total, nL = A.n_lev_total;
  const int z0 = blockIdx.x * ZONE_WARPS, z = z0 + warp;
  // entries in use: a caller may give room for more than the lists hold
  const int nIu = (na > 0) ? min(nI, A.ion_off[na]) : 0, nLu = (na > 0) ? min(nL, A.lev_off[na]) : 0;
  const size_t per = zone_state_doubles(FAST, na, nI, nL);
  double* lev = zsm + warp * per;           // [nL] Boltzmann factors, then the populations (FAST); else the
  double* eb = FAST ? lev : lev + nL;       // terms of the sums, then the populations, beside the factors
  double* part = eb + nL;                   // [nI] partition functions
  double* frac = part + nI;                 // [nI] stage fractions
  double* coef = frac + nI;                 // [nI] exp(-chi/kT) part_i / part_(i-1)
  double* nd = coef + nI;                   // [na] atom densities
  double* net = nd + na;                    // [na] mean charges
  bool micro = false;
  if (z < nz) {
    const double T = zone_temperature(A, z);
    const double dens = A.rho[z];
    const double mu_I = zone_mass_fractions(A, z, lane == 0);
    micro = !(A.grey[z] != 0 || na == 0);
    if (lane == 0) {
      A.temp_c[z] = T;
      A.solve_err[z] = 0;
      if (!micro) A.n_elec[z] = 0;
    }
    if (micro) {
      __syncwarp();  // lane 0's mass fractions
      for (int a = lane; a < na; a += 32) nd[a] = dens * A.mass_frac[(size_t)a * nz + z] / (A.eA[a] * MASS_P);
      for (int l = lane; l < nLu; l += 32) eb[l] = exp(-A.lev_E[l] / K_EV / T);
      __syncwarp();
      for (int i = lane; i < nIu; i += 32) {  // a stage's levels in order, a lane per stage
        int a = 0;
        while (A.ion_off[a + 1] <= i) ++a;
        const int ion = i - A.ion_off[a], l1 = A.lev_off[a + 1];
        double sum = 0;
        for (int l = A.lev_off[a]; l < l1; ++l)
          if (A.lev_ion[l] == ion) sum += A.lev_g[l] * eb[l];
        part[i] = sum;
      }
      __syncwarp();
      for (int i = lane; i < nIu; i += 32) {
        int a = 0;
        while (A.ion_off[a + 1] <= i) ++a;
        if (i > A.ion_off[a]) coef[i] = exp(-1.0 * A.ion_chi[i - 1] / K_EV / T) * (part[i] / part[i - 1]);
      }
      __syncwarp();
      const double lt = H_PLANCK * H_PLANCK / (2.0 * PI * MASS_E * K_BOLTZ * T);
      const double lt15 = pow(lt, 1.5);
      // level populations at the current stage fractions, times the charge for the sum over levels
      auto levels = [&](bool charge) {
        for (int a = 0; a < na; ++a) {
          const int i0 = A.ion_off[a], l1 = A.lev_off[a + 1];
          for (int l = A.lev_off[a] + lane; l < l1; l += 32) {
            const int ion = A.lev_ion[l];
            double v = frac[i0 + ion] * A.lev_g[l] * eb[l] / part[i0 + ion];
            if (v < 1e-30) v = 1e-30;
            lev[l] = charge ? v * ion : v;
          }
        }
        __syncwarp();
      };
      auto stages = [&](double ne) {
        const double fac = 2 / ne / lt15;
        for (int a = lane; a < na; a += 32) {
          const int i0 = A.ion_off[a];
          stage_fractions(frac + i0, coef + i0, A.ion_off[a + 1] - i0, ne, fac);
        }
        __syncwarp();
      };
      auto f = [&](double ne) {
        if constexpr (FAST) {
          const double fac = 2 / ne / lt15;
          for (int a = lane; a < na; a += 32) {
            const int i0 = A.ion_off[a], ni = A.ion_off[a + 1] - i0;
            double u = 1., sum = 1., q = 0.;  // stage i to stage 0, their sum, the charge
            for (int i = 1; i < ni; ++i) {
              u = (ne < 1e-50) ? 0. : coef[i0 + i] * fac * u;
              sum += u;
              q += i * u;
              if (sum > 1e100) { const double r = 1. / sum; u *= r; q *= r; sum = 1.; }
            }
            net[a] = q / sum;
          }
        } else {
          stages(ne);
          levels(true);
          for (int a = lane; a < na; a += 32) {
            double x = 0;
            const int l1 = A.lev_off[a + 1];
            for (int l = A.lev_off[a]; l < l1; ++l) x += lev[l];
            net[a] = x;
          }
        }
        __syncwarp();
        double s = 0;
        for (int a = 0; a < na; ++a) s += nd[a] * net[a];
        __syncwarp();
        return s - ne;
      };
      const double max_ne = 100 * dens / (mu_I * MASS_P);
      const double min_ne = 1e-10 * dens / (mu_I * MASS_P);
      double last = 0;
      int err = 0;
      const double ne = ne_brent(f, min_ne, max_ne, 1e-3, &last, &err);
      stages(last);  // populations of the last evaluation
      levels(false);
      if (lane == 0) {
        A.n_elec[z] = ne;
        A.solve_err[z] = err;
      }
    }
  }
  // the CTA's results, the zones of a level next to each other
  __shared__ int s_micro[ZONE_WARPS];
  if (lane == 0) s_micro[warp] = micro;
  __syncthreads();
  auto put = [&](double* out, size_t off, int n) {
    for (int i = threadIdx.x; i < n * ZONE_WARPS; i += 32 * ZONE_WARPS) {
      const int q = i % ZONE_WARPS, k = i / ZONE_WARPS;
      if (s_micro[q]) out[(size_t)k * nz + z0 + q] = zsm[q * per + off + k];
    }
  };
  const size_t o = (FAST ? 1 : 2) * (size_t)nL;
  put(A.lev_n, 0, nLu);
  put(A.ion_part, o, nIu);
  put(A.ion_frac, o + nI, nIu);
  put(A.n_dens, o + 3 * (size_t)nI, na);
}

// Shared memory a CTA of zone_state_warp_kernel may take: level lists beyond
// it (about 3000 levels in FP64, 6000 with FP32 tables) take one thread per
// zone.
constexpr size_t ZONE_STATE_SMEM = 200 * 1024;
// Many zones fill the chip with a thread each, and a warp's 32 lanes then cost
// more than the shared state saves: with short level lists most of them have
// nothing to do in an evaluation, and in FP64 the lanes that sum an atom's
// levels leave the others idle.  sed_set_opacity on B200 (4 bins, so mostly this
// solve) in ms, a warp / a thread per zone:
//   levels (atoms)      11 (1)       102 (2)      156 (6)      906 (6)
//   FP64   4 096 zones  0.15 / 0.16  0.17 / 0.43  0.18 / 0.86  0.54 / 3.21
//         32 768        0.97 / 0.40  1.15 / 0.77  1.25 / 1.26  3.45 / 6.52
//        110 592        3.24 / 1.18  3.90 / 2.16  4.32 / 3.71  11.6 / 13.6
//        262 144        7.66 / 2.84  9.25 / 4.66  10.1 / 7.34  26.4 / 23.0
//   FP32  32 768        0.53 / 0.39  0.61 / 0.75  0.65 / 1.25  1.30 / 6.48
//        262 144        4.07 / 2.62  4.95 / 4.46  5.29 / 7.12  9.64 / 22.3
bool zone_state_by_thread(bool fast, int nz, int n_lev, int num_sms)
{
  if (nz < 128 * num_sms) return false;
  return fast ? n_lev <= 64 : nz >= (int64_t)210 * n_lev;
}

int launch_zone_state(const OpacityArgs& a, int num_sms, cudaStream_t s)
{
  const bool fast = a.precision != 0;
  const size_t smem = ZONE_WARPS * sizeof(double) * zone_state_doubles(fast, a.natoms, a.n_ions_total, a.n_lev_total);
  if (smem > ZONE_STATE_SMEM || zone_state_by_thread(fast, a.nzones, a.n_lev_total, num_sms)) {
    zone_state_kernel<<<(a.nzones + 127) / 128, 128, 0, s>>>(a, a.boltz);
    return 1;
  }
  auto k = fast ? zone_state_warp_kernel<true> : zone_state_warp_kernel<false>;
  if (smem > 48 * 1024 &&
      cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
    return -1;
  k<<<(a.nzones + ZONE_WARPS - 1) / ZONE_WARPS, 32 * ZONE_WARPS, smem, s>>>(a);
  return 1;
}

// ------------------------------------------------------------ per zone
// xy_array::value_at_with_zero_edges (src/utils/xy_array.cpp:42-104)
__device__ double photo_cs(const OpacityArgs& A, int lev, double zv)
{
  const int p0 = A.photo_off[lev], n = A.photo_off[lev + 1] - p0;
  const double* x = A.photo_E + p0;
  const double* y = A.photo_s + p0;
  if (n <= 0) return 0;
  if (zv < x[0]) return 0;
  if (zv > x[n - 1]) return 0;
  if (n == 1) return y[0];
  int ind;
  if (zv >= x[n - 1]) ind = n;
  else if (zv <= x[0]) ind = 0;
  else {
    int bl = 0, bu = n - 1;
    while (bu - bl > 1) { const int bm = (bu + bl) / 2; if (x[bm] <= zv) bl = bm; else bu = bm; }
    ind = bl;
  }
  int i1, i2;
  if (ind < n - 1) { i1 = ind; i2 = ind + 1; }
  else { i2 = ind < n ? ind : n - 1; i1 = i2 - 1; }
  const double slope = (y[i2] - y[i1]) / (x[i2] - x[i1]);
  return y[ind < n ? ind : n - 1] + slope * (zv - x[i1]);
}

// 1 - exp(-tau), the Sobolev escape factor of one line, as the reference
// writes it: for tau below ~1e-16 it is exactly 0 and for small tau it
// carries the cancellation of 1 - exp(-tau), which the FP64 tables reproduce.
__device__ __forceinline__ double sobolev_term(double tau) { return 1 - exp(-tau); }

// Two FP32 values in one 64-bit register pair and the instructions that work
// on both at once (PTX f32x2), each half rounded as the scalar one is.  The
// line sums are bound by issue slots (74-80 %), so two terms share the slots of
// their arithmetic: 64^3 cells x 1e5 level lines 55.4 -> 52.7 ms, 18 494 zones x
// 3e4 fuzz lines 2.03 -> 1.98 ms (the packed instructions hold the FP32 pipe
// for two slots, so only what the others wait for is won).
struct F2 {
  unsigned long long v;
  __device__ __forceinline__ F2() {}
  __device__ __forceinline__ F2(float lo, float hi) { asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi)); }
  __device__ __forceinline__ explicit F2(float both) : F2(both, both) {}
  __device__ __forceinline__ float2 get() const
  {
    float2 f;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
    return f;
  }
};
__device__ __forceinline__ F2 operator*(F2 a, F2 b)
{
  F2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 one_minus(F2 a)  // 1 - a, one rounding
{
  F2 r;
  const F2 m(-1.f), o(1.f);
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(m.v), "l"(o.v));
  return r;
}

// FP32 form of 1 - exp(-x) for x >= 0, two values, branch-free: below x = 0.1 the
// Taylor series to x^7 (truncation below x^8/8! < 3e-12 relative), above it
// 1 - __expf(-x), whose ~2^-22 relative error in exp(-x) stays below 3e-6
// relative in 1 - exp(-x) for x >= 0.1.  Neither has the cancellation of
// 1 - expf(-x) at small x.
__device__ __forceinline__ float2 one_minus_exp32(F2 x)
{
  F2 s = one_minus(x * F2(1.f / 7));
  s = one_minus(x * F2(1.f / 6) * s);
  s = one_minus(x * F2(0.2f) * s);
  s = one_minus(x * F2(0.25f) * s);
  s = one_minus(x * F2(1.f / 3) * s);
  s = one_minus(x * F2(0.5f) * s);
  const float2 p = (x * s).get(), v = x.get();
  const float ex = 1.f - __expf(-v.x), ey = 1.f - __expf(-v.y);
  return make_float2((v.x < 0.1f) ? p.x : ex, (v.y < 0.1f) ? p.y : ey);
}

// Level populations of one zone in the chunk scratch (level-major).
struct LevView {
  const double* p;
  int64_t stride;
  __device__ __forceinline__ double n(int l) const { return p[l * stride]; }
};

// Per-bin Sobolev sums of one line list (level-to-level lines, or fuzz lines
// when FUZZ) for a tile of ZT zones: S[z][bin] = sum of (1 - exp(-tau)) over
// the bin's lines, Se[z][bin] the same weighted by the line's atom epsilon
// when atoms differ in epsilon (AtomicSpecies_opacities.cpp:292-375,
// GasState_opacities.cpp:424-494).  The tile's level populations times the
// atom's number density, n_l n_atom, and their reciprocals (or the ion
// populations for fuzz lines) are staged in shared memory level-major, ZT
// zones contiguous; the ratio n_u g_l / (n_l g_u) is formed from them (the
// atom density cancels).  A warp takes one bin at a time (the warps of the
// gridDim.y CTAs of a tile deal the bins of `order`, which lists them by
// decreasing line count, among themselves): its lanes are ZT zones x 32/ZT line slots, slot s summing the
// bin's lines s, s + 32/ZT, ... (sorted by bin, atom), and the slots of a
// zone are then added in FP64 in a fixed butterfly order, so the sums are
// the same from run to run.  The FP64 form sums in FP64; the mixed form
// computes its terms in FP32 and sums them in FP32 with Kahan compensation
// (measured on the Type Ia and 3D builds: the same time and the same
// largest error against the FP64 oracle as FP64 sums of the FP32 terms,
// 1.6e-6 relative, which the FP32 tables' rounding sets).
// Level populations come from the LTE solve, floored at 1e-30, so they are
// normal FP32 numbers and the reference's n_l < DBL_MIN skip never applies
// to them; a NaN term is skipped as in the reference.
constexpr int LINE_SUM_WARPS = 8;  // line_sum_kernel runs 256 threads per CTA

template <bool MIXED, bool FUZZ, int ZT>
__global__ void __launch_bounds__(32 * LINE_SUM_WARPS) line_sum_kernel(const OpacityArgs A, double* S, double* Se)
{
  using V = typename std::conditional<MIXED, float, double>::type;
  extern __shared__ double lsm[];
  const int nn = A.n_nu, nz = A.nzones, na = A.natoms, tid = threadIdx.x, bd = blockDim.x;
  const int z0 = blockIdx.x * ZT;
  const int nzt = min(ZT, nz - z0);
  if (nzt <= 0) return;
  // shared: ndv[na][ZT], epsv[na], invT[ZT], pop[np][ZT], ipop[np][ZT] (V)
  const int np = FUZZ ? A.n_ions_total : A.n_lev_total;
  V* ndv = reinterpret_cast<V*>(lsm);
  V* epsv = ndv + na * ZT;
  V* invT = epsv + na;
  V* pop = invT + ZT;
  V* ipop = pop + (size_t)np * ZT;
  for (int i = tid; i < na * ZT; i += bd) {
    const int a = i / ZT, zi = i % ZT;
    ndv[i] = (zi < nzt) ? (V)A.n_dens[(size_t)a * nz + z0 + zi] : (V)0;
  }
  for (int a = tid; a < na; a += bd) epsv[a] = A.zero_eps_atom[a] ? (V)0 : (V)A.epsilon;
  for (int zi = tid; zi < ZT; zi += bd) invT[zi] = (zi < nzt) ? (V)(1.0 / A.temp_c[z0 + zi]) : (V)0;
  for (int i = tid; i < np * ZT; i += bd) {
    const int l = i / ZT, zi = i % ZT;
    double v = 0;
    if (zi < nzt) {
      if constexpr (FUZZ) {
        const int a = A.ion_atom[l];
        v = A.n_dens[(size_t)a * nz + z0 + zi] * A.ion_frac[(size_t)l * nz + z0 + zi] /
            A.ion_part[(size_t)l * nz + z0 + zi];
      } else {
        v = A.lev_n[(size_t)l * nz + z0 + zi] * A.n_dens[(size_t)A.lev_atom[l] * nz + z0 + zi];
      }
    }
    pop[i] = (V)v;
    if constexpr (!FUZZ) ipop[i] = (zi < nzt) ? (V)(1.0 / v) : (V)0;
  }
  __syncthreads();
  const bool want_e = !A.uniform_eps;
  const int32_t* seg = FUZZ ? A.fz_seg : A.ln_seg;
  const int32_t* order = FUZZ ? A.fz_order : A.ln_order;
  const double time = A.time;
  // a warp per bin: its 32 lanes are ZT zones x LS line slots; slot s takes
  // the bin's lines s, s + LS, ..., so the lanes of a warp run the same
  // number of lines (up to one) and read the same few line records.  The
  // warp stages the bin's records 32 at a time in its shared-memory buffer,
  // one coalesced load per lane, and the slots read them from there: one
  // memory round trip per 32 records instead of one per LS (48^3 level-line
  // build 61.2 -> 48.5 ms, Type Ia fuzz-line build 5.2 -> 5.0 ms).  The
  // line loop is unrolled by two (Type Ia 6.9 -> 5.4 ms before the staging).
  constexpr int LS = 32 / ZT;
  static_assert(32 % LS == 0, "a slot keeps its lines across the 32-record chunks");
  const int lane = tid & 31, warp = tid >> 5, nwarps = (bd >> 5) * gridDim.y;
  const int zi = lane % ZT, slot = lane / ZT;
  using CRec = typename std::conditional<MIXED, typename std::conditional<FUZZ, float4, float2>::type, double2>::type;
  __shared__ int4 s_ix[LINE_SUM_WARPS][32];
  __shared__ CRec s_cr[LINE_SUM_WARPS][32];
  __shared__ double s_h[(FUZZ && !MIXED) ? LINE_SUM_WARPS : 1][32];
  const int4* __restrict__ ix_g = FUZZ ? A.fz_ia : A.ln_lv;
  const CRec* __restrict__ cr_g;
  if constexpr (MIXED) {
    if constexpr (FUZZ) cr_g = A.fz_c32; else cr_g = A.ln_c32;
  } else {
    cr_g = FUZZ ? A.fz_c : A.ln_c;
  }
  for (int jj = warp * gridDim.y + blockIdx.y; jj < nn; jj += nwarps) {
    const int j = __ldg(order + jj);
    double acc = 0, acce = 0;
    float ks = 0.f, kc = 0.f, kse = 0.f, kce = 0.f;  // the mixed form's FP32 Kahan sums
    const int k0 = seg[j], k1 = seg[j + 1];
    for (int kb = k0; kb < k1; kb += 32) {
      const int nk = min(32, k1 - kb);
      __syncwarp();
      if (lane < nk) {
        s_ix[warp][lane] = __ldg(ix_g + kb + lane);
        CRec cr = __ldg(cr_g + kb + lane);
        if constexpr (MIXED) cr.x *= (float)time;  // once per record, not per term
        s_cr[warp][lane] = cr;
        if constexpr (FUZZ && !MIXED) s_h[warp][lane] = __ldg(A.fz_h + kb + lane);
      }
      __syncwarp();
      if constexpr (MIXED) {
        // a slot's lines two at a time through the f32x2 instructions, then
        // added one after the other by Kahan (compensated) summation: the
        // rounding error of each addition is carried into the next term
        auto add = [&](float term, int atom) {
          { const float y = term - kc; const float t = ks + y; kc = (t - ks) - y; ks = t; }
          if (want_e) {
            const float y = term * epsv[atom] - kce;
            const float t = kse + y;
            kce = (t - kse) - y;
            kse = t;
          }
        };
        for (int kk = slot; kk < nk; kk += 2 * LS) {
          const bool two = kk + LS < nk;
          const int k2 = two ? kk + LS : kk;
          const int4 i1 = s_ix[warp][kk], i2 = s_ix[warp][k2];
          const CRec c1 = s_cr[warp][kk], c2 = s_cr[warp][k2];
          float2 t;
          if constexpr (!FUZZ) {
            // tau = n_l n_atom sigma_tot f lambda t (1 - n_u g_l / (n_l g_u)), 0 past the laser limit
            const F2 pl(pop[(size_t)i1.x * ZT + zi], pop[(size_t)i2.x * ZT + zi]);    // n_l n_atom
            const F2 il(ipop[(size_t)i1.x * ZT + zi], ipop[(size_t)i2.x * ZT + zi]);  // 1 / (n_l n_atom)
            const F2 pu(pop[(size_t)i1.y * ZT + zi], pop[(size_t)i2.y * ZT + zi]);    // n_u n_atom
            const F2 r = pu * il * F2(c1.y, c2.y);
            const float2 rr = r.get(), tt = (pl * F2(c1.x, c2.x) * one_minus(r)).get();
            t = one_minus_exp32(F2((rr.x > 1.f) ? 0.f : tt.x, (rr.y > 1.f) ? 0.f : tt.y));
            t.x = (t.x == t.x) ? t.x : 0.f;
            t.y = (t.y == t.y) ? t.y : 0.f;
            add(t.x, i1.w);
            if (two) add(t.y, i2.w);
          } else {
            // n_l = n_ion exp(-E_l/kT) / Z_ion, tau = sigma_tot lambda n_l gf (1 - exp(-h nu/kT)) t
            const float iT = invT[zi];
            const F2 pi(pop[(size_t)i1.x * ZT + zi], pop[(size_t)i2.x * ZT + zi]);
            const float2 stim = one_minus_exp32(F2(c1.z, c2.z) * F2(iT));
            const F2 bz(__expf(-c1.y * iT), __expf(-c2.y * iT));
            t = one_minus_exp32(F2(c1.x, c2.x) * pi * bz * F2(stim.x, stim.y));
            add(t.x, i1.z);
            if (two) add(t.y, i2.z);
          }
        }
      } else {
#pragma unroll 2
        for (int kk = slot; kk < nk; kk += LS) {
          int atom;
          double term;
          if constexpr (!FUZZ) {
            const int4 lv = s_ix[warp][kk];
            atom = lv.w;
            const V pl = pop[(size_t)lv.x * ZT + zi];
            const V il = ipop[(size_t)lv.x * ZT + zi];
            const V pu = pop[(size_t)lv.y * ZT + zi];
            const CRec c = s_cr[warp][kk];
            double t = 0;
            if (!(pl < DBL_MIN)) {
              const double r = pu * il * c.y;
              const double tau = (r > 1) ? 0.0 : pl * c.x * time * (1 - r);
              t = sobolev_term(tau);
              if (isnan(t)) t = 0;
            }
            term = t;
          } else {
            const int4 ia = s_ix[warp][kk];
            atom = ia.z;
            const V pi = pop[(size_t)ia.x * ZT + zi];
            const CRec c = s_cr[warp][kk];
            const double h = s_h[warp][kk];
            if (zi < nzt) {
              const double temp = A.temp_c[z0 + zi];
              const double nl = pi * exp(-c.y / temp);
              const double stim_cor = (1 - exp(-h / temp));
              const double tau = c.x * nl * stim_cor * time;
              term = sobolev_term(tau);
            } else {
              term = 0;
            }
          }
          acc += term;
          if (want_e) acce += term * epsv[atom];
        }
      }
    }
    if constexpr (MIXED) { acc = (double)ks; acce = (double)kse; }
    // the LS slots of each zone, summed in a fixed butterfly order
#pragma unroll
    for (int off = ZT; off < 32; off <<= 1) {
      acc += __shfl_xor_sync(0xffffffffu, acc, off);
      acce += __shfl_xor_sync(0xffffffffu, acce, off);
    }
    if (slot == 0 && zi < nzt) {
      S[(size_t)(z0 + zi) * nn + j] = acc;
      if (want_e) Se[(size_t)(z0 + zi) * nn + j] = acce;
    }
  }
}

// Per-bin factors no zone changes, [BIN_TAB][n_nu], formed once per context
// by bin_table_kernel: with them a bin of a zone costs one or two exponentials
// and a handful of divisions instead of a pow() and a dozen divisions more.
enum BinTab { BT_NU, BT_B, BT_HNK, BT_NU4, BT_D, BT_FAC };

__global__ void bin_table_kernel(const DevLoc nu_grid, double* __restrict__ tab, double2* __restrict__ lr)
{
  const int nn = nu_grid.n;
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < nn; j += gridDim.x * blockDim.x) {
    const double nu = loc_center(nu_grid, j), d = loc_delta(nu_grid, j);
    lr[j] = make_double2(loc_left(nu_grid, j), nu_grid.right[j]);
    tab[BT_NU * nn + j] = nu;
    tab[BT_B * nn + j] = 2.0 * nu * nu * nu * H_PLANCK / C_LIGHT / C_LIGHT;  // B_nu (e^zeta - 1)
    tab[BT_HNK * nn + j] = H_PLANCK * nu / K_BOLTZ;                          // zeta T
    tab[BT_NU4 * nn + j] = pow(nu, 4);
    tab[BT_D * nn + j] = d;
    tab[BT_FAC * nn + j] = nu / d / C_LIGHT;  // times 1/t: the expansion opacity of one Sobolev term
  }
}

// the guide tables of zone_opacity_kernel, from CDF rows written otherwise
template <typename T>
__global__ void guide_kernel(const T* __restrict__ cdf, int64_t nz, int nn, uint16_t* __restrict__ guide, int G)
{
  const int64_t n = nz * (G + 1);
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const T* row = cdf + (size_t)(i / (G + 1)) * nn;
    const double t = (double)(i % (G + 1)) / (double)G;
    int lo = 0, hi = nn;
    while (lo < hi) {
      const int m = (lo + hi) >> 1;
      if ((double)row[m] <= t) lo = m + 1; else hi = m;
    }
    guide[i] = (uint16_t)lo;
  }
}

// the packed bins of zone_opacity_kernel, from tables written otherwise
__global__ void pack_bins_kernel(const float2* __restrict__ opac, const float* __restrict__ cdf, int64_t n, int nn,
                                 float4* __restrict__ out)
{
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const float2 o = opac[i];
    out[i] = make_float4(i % nn ? cdf[i - 1] : 0.f, cdf[i], o.x, o.y);
  }
}

// Opacity, scattering and emissivity of one bin of zone z (GasState::
// computeOpacity, GasState_opacities.cpp:11-136, with its terms in the
// reference's order: electron scattering, free-free, bound-free, Sobolev
// lines, fuzz lines).  The line terms arrive as the bin's Sobolev sums
// (ls, lse, fs, fse; the epsilon-weighted sums only when atoms differ in
// epsilon).  nu, the Planck function bb and ez = exp(h nu/kT) are shared with
// the caller; fac_t = nu / dnu / c / t.  MIXED: the free-free factors from bb,
// 1/ez and 1/nu^3 (the tables are FP32); else the reference's expressions.
// BF: with the bound-free term, whose loop over levels takes the registers of
// two more CTAs per SM (122 against 61).
template <bool MIXED, bool BF>
__device__ void bin_opacity(const OpacityArgs& A, int zc, double nu, double b_num, double bb, double ez, double zeta,
                            double fac_t, double temp, double grey, double ne, double es, double ff_fac,
                            const double* nd, const LevView& L, double ls, double lse, double fs, double fse,
                            double& ab_o, double& sc_o, double& em_o)
{
  double ab = 0, sc = 0, em = 0;
  if (grey != 0) {  // GasState_opacities.cpp:29-41
    const double gopac = A.rho[zc] * grey;
    ab = gopac * A.epsilon;
    sc = gopac * (1 - A.epsilon);
    em += bb * ab;
  } else if (A.natoms > 0) {
    if (A.use_es) {  // :49-58
      sc += es;
      ab += 1e-20 * A.epsilon * es;
    }
    if (A.use_ff) {  // GasState::free_free_opacity :152-183
      if constexpr (MIXED) {
        const double op = ff_fac / (nu * nu * nu) * (1 - 1.0 / ez);
        ab += op;
        em += op * bb;
      } else {
        const double ezeta = exp(-zeta);
        const double bf = b_num / (1.0 / ezeta - 1);
        const double op = ff_fac / nu / nu / nu * (1 - ezeta);
        ab += op;
        em += op * bf;
      }
    }
    if constexpr (BF) {  // GasState::bound_free_opacity + AtomicSpecies_opacities.cpp:58-151
      const double kt_ev = K_EV * temp;
      const double lam_t = sqrt(H_PLANCK * H_PLANCK / (2 * PI * MASS_E * K_BOLTZ * temp));
      const double E = H_PLANCK * nu * ERGS_TO_EV;
      const double emis_fac = 2. * H_PLANCK * nu * nu * nu / C_LIGHT / C_LIGHT;
      double so = 0, se = 0;
      for (int a = 0; a < A.natoms; ++a) {
        const int l0 = A.lev_off[a], nl = A.lev_off[a + 1] - l0;
        double ao = 0, ae = 0;
        for (int q = 0; q < nl; ++q) {
          const int ic = A.lev_ic[l0 + q];
          if (ic == -1) continue;
          const double Eion = A.lev_Eion[l0 + q];
          if (E < Eion) continue;
          const double nc = nd[a] * L.n(l0 + ic);
          const double gl_o_gc = (1.0 * A.lev_g[l0 + q]) / (1.0 * A.lev_g[l0 + ic]);
          const double ncp = nc * gl_o_gc / 2. * lam_t * lam_t * lam_t;
          const double zeta_net = (Eion - E) / kt_ev;
          const double ezeta_net = exp(zeta_net);
          const double sigma = photo_cs(A, l0 + q, E);
          double opac_fac = nd[a] * L.n(l0 + q) - ncp * ne * ezeta_net;
          if (opac_fac < 0) opac_fac = 0.;
          ao += sigma * opac_fac;
          ae += emis_fac * sigma * ncp * ezeta_net;
        }
        so += ao;
        se += ae;
      }
      ab += so;
      em += se * ne;
    }
    if (A.use_line) {  // GasState::line_expansion_opacity :424-454
      const double opac = ls * fac_t;
      const double aopac = (A.uniform_eps ? ls * A.epsilon : lse) * fac_t;
      ab += aopac;
      sc += opac - aopac;
      em += bb * aopac;
    }
    if (A.use_fuzz) {  // GasState::fuzz_expansion_opacity :464-494
      const double opac = fs * fac_t;
      const double aopac = (A.uniform_eps ? fs * A.epsilon : fse) * fac_t;
      ab += aopac;
      sc += opac - aopac;
      em += bb * aopac;
    }
  }
  ab_o = ab;
  sc_o = sc;
  em_o = em;
}

__device__ __forceinline__ double warp_sum_f64(double v)
{
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// One CTA per zone of the chunk, after line_sum_kernel: each thread builds
// bins j = tid, tid + THREADS, ... from the continuum terms and the bin's
// Sobolev sums (GasState::computeOpacity), caps them and accumulates the
// Planck/Rosseland partial sums (GasState_opacities.cpp:564-666); then the
// CTA forms the emissivity CDF, L_thermal and eps_imc
// (transport_opacity.cpp:152-252) and writes the packed tables the packet
// kernel reads.  The FP64 rows (abs, scat, emissivity) live in shared memory
// when they fit (A.smem_rows); otherwise abs and scat overwrite the line and
// fuzz sums of the zone in the chunk scratch (each bin is read, then written,
// by the same thread) and the emissivity row is scratch too.
//
// What bounds it: FP64 arithmetic per bin, then the serial parts of a row.
// The bin constants come from bin_table_kernel, the sums and the scan are
// warp shuffles, and the guide table is written bin by bin (below): 64^3 zones
// x 2048 bins, FP32 tables, 31.7 -> 11.6 ms (1.2 of it so that no sum of the
// scan falls; its traffic, 11.8 GB, is 1.8 ms of HBM), 18 494 zones 3.07 -> 1.02
// ms, with bound-free levels (128 zones x 2048 bins x 606 levels) 1.10 -> 0.48
// ms.
template <bool MIXED, int THREADS, bool BF>
__global__ void __launch_bounds__(THREADS, BF ? 1 : 1024 / THREADS) zone_opacity_kernel(const OpacityArgs A)
{
  constexpr int WARPS = THREADS / 32;
  extern __shared__ double dsm[];
  __shared__ double red[4][WARPS];
  __shared__ double zs[2];  // electron scattering, free-free factor
  const int z = blockIdx.x;
  if (z >= A.nzones) return;
  const int nn = A.n_nu, nz = A.nzones, na = A.natoms, tid = threadIdx.x, bd = THREADS;
  const int lane = tid & 31, warp = tid >> 5;
  const double temp = A.temp_c[z];
  const double grey = A.grey[z];
  const double ne = A.n_elec[z];
  const bool want_e = !A.uniform_eps;

  // shared layout: nd[na] rows[3 nn]
  double* nd = dsm;
  double* rows = nd + na;
  const size_t zo = (size_t)z * nn;
  const double* LS = A.abs64 + zo;
  const double* FS = A.scat64 + zo;
  const double* LSe = A.epsl64 + zo;
  const double* FSe = A.epsf64 + zo;
  double* R0 = A.smem_rows ? rows : A.abs64 + zo;
  double* R1 = A.smem_rows ? rows + nn : A.scat64 + zo;
  double* R2 = A.smem_rows ? rows + 2 * nn : A.emis64 + zo;
  const double* __restrict__ tab = A.bin_tab;

  const bool micro = (grey == 0 && na > 0);
  if (micro) {
    for (int a = tid; a < na; a += bd) nd[a] = A.n_dens[(size_t)a * nz + z];
    if (tid == 0) {
      zs[0] = THOMSON * ne;
      double ff = 0;
      if (A.use_ff) {  // GasState::free_free_opacity :152-183 (zone factor)
        const double dens = A.rho[z];
        for (int a = 0; a < na; ++a) {
          const int i0 = A.ion_off[a], ni = A.ion_off[a + 1] - i0;
          double zsq = 0;
          for (int q = 0; q < ni; q++) zsq += A.ion_frac[(size_t)(i0 + q) * nz + z] * q * q;
          const double n_ion = A.mass_frac[(size_t)a * nz + z] * dens / (A.eA[a] * MASS_P);
          ff += n_ion * zsq;
        }
        ff *= 3.7e8 * pow(temp, -0.5) * ne;
      }
      zs[1] = ff;
    }
  }
  __syncthreads();
  LevView L;
  L.p = A.lev_n + z;
  L.stride = nz;
  const double es = micro ? zs[0] : 0.0, ff_fac = micro ? zs[1] : 0.0;
  const bool lines = micro && A.use_line, fuzz = micro && A.use_fuzz;

  // bins, cap (transport_opacity.cpp:189-200) and mean-opacity partial sums
  const double max_ext = A.max_opacity * A.rho[z];
  const double inv_T = 1.0 / temp, inv_t = 1.0 / A.time;  // FP32 tables only
  double pm = 0, pn = 0, rm = 0, rn = 0;
  for (int j = tid; j < nn; j += bd) {
    const double nu = __ldg(tab + BT_NU * nn + j), b_num = __ldg(tab + BT_B * nn + j);
    const double hnk = __ldg(tab + BT_HNK * nn + j), nu4 = __ldg(tab + BT_NU4 * nn + j);
    const double d = __ldg(tab + BT_D * nn + j), fac = __ldg(tab + BT_FAC * nn + j);
    const double zeta = MIXED ? hnk * inv_T : hnk / temp;
    const double ez = exp(zeta);
    const double i1 = MIXED ? 1.0 / (ez - 1) : 0.0;
    const double bb = MIXED ? b_num * i1 : b_num / (ez - 1);
    double ab, sc, em;
    bin_opacity<MIXED, BF>(A, z, nu, b_num, bb, ez, zeta, MIXED ? fac * inv_t : fac / A.time, temp, grey, ne, es, ff_fac,
                       nd, L, lines ? LS[j] : 0.0, (lines && want_e) ? LSe[j] : 0.0, fuzz ? FS[j] : 0.0,
                       (fuzz && want_e) ? FSe[j] : 0.0, ab, sc, em);
    if (A.omit_scat) sc = 0;
    else if (sc > max_ext) sc = max_ext;
    if (ab > max_ext) ab = max_ext;
    R0[j] = ab;
    R1[j] = sc;
    R2[j] = em;
    double Bnu = bb;
    if (isnan(Bnu)) Bnu = 0;
    const double W = Bnu * d;
    pm += W * ab;
    pn += W;
    double dBdT = MIXED ? nu4 * ez * i1 * i1 : nu4 * ez / (ez - 1) / (ez - 1);
    if (isnan(dBdT)) dBdT = 0;
    const double Wr = dBdT * d;
    rm += Wr / (ab + sc);
    rn += Wr;
  }
  double* ab_r = R0;
  double* sc_r = R1;
  pm = warp_sum_f64(pm); pn = warp_sum_f64(pn); rm = warp_sum_f64(rm); rn = warp_sum_f64(rn);
  if (lane == 0) { red[0][warp] = pm; red[1][warp] = pn; red[2][warp] = rm; red[3][warp] = rn; }
  __syncthreads();
  double pm_tot = 0, pn_tot = 0, rm_tot = 0, rn_tot = 0;
  if (tid == 0)
    for (int w = 0; w < WARPS; ++w) {
      pm_tot += red[0][w]; pn_tot += red[1][w]; rm_tot += red[2][w]; rn_tot += red[3][w];
    }
  __syncthreads();

  // emissivity CDF: cdf_array::set_value prefix sum of emis*dnu (cdf_array.h:
  // 53-75) and L_thermal = 4 pi sum(emis*dnu).  FP64 tables of grids up to
  // 65536 zones: in the reference's order, so the CDF is the reference's sum
  // to the bit (and a bin's share of it, the difference of two neighbouring
  // values, too): the terms in parallel, the running sums by one thread, a
  // few microseconds per zone.  Otherwise (FP32 tables, or millions of zones
  // where a serial row per CTA would dominate the build) a blocked scan in a
  // fixed order: each warp scans a contiguous run of bins 32 at a time, the
  // run totals are added up in order, each run adds its offset; non-negative
  // terms, so every prefix is within a few ulp of the sequential sum and none is
  // below the one before it, and a NaN term propagates to the end as in the
  // sequential sum.
  double* em = R2;
  double Lth = 0;
  if (nn == 1) {
    if (tid == 0) {
      const double bb_int = SB * pow(A.T[z], 4) / PI;
      Lth += 4 * PI * ab_r[0] * bb_int;
      em[0] = 1;
    }
  } else if (!MIXED && A.seq_cdf) {
    for (int j = tid; j < nn; j += bd) em[j] = em[j] * __ldg(tab + BT_D * nn + j);
    __syncthreads();
    if (tid == 0) {
      double run = 0, L = 0;
      for (int j = 0; j < nn; ++j) {
        const double ednu = em[j];
        run = (j == 0) ? ednu : run + ednu;
        em[j] = run;
        L += 4 * PI * ednu;
      }
      Lth = L;
    }
  } else {
    const int per = ((nn + WARPS - 1) / WARPS + 31) & ~31;
    const int j0 = min(nn, warp * per), j1 = min(nn, j0 + per);
    double base = 0, Lp = 0;
    for (int jb = j0; jb < j1; jb += 32) {
      const int j = jb + lane;
      double v = (j < j1) ? em[j] * __ldg(tab + BT_D * nn + j) : 0.0;
      Lp += 4 * PI * v;
      const bool rises = __all_sync(0xffffffffu, !(v < 0));
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const double u = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += u;
      }
      // two lanes' sums round on their own: where the terms are small the later
      // one may come out an ulp below, so each takes the largest up to it
      if (rises) {
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const double u = __shfl_up_sync(0xffffffffu, v, o);
          if (lane >= o && u > v) v = u;
        }
      }
      v += base;
      if (j < j1) em[j] = v;
      base = __shfl_sync(0xffffffffu, v, 31);
    }
    Lp = warp_sum_f64(Lp);
    if (lane == 0) { red[0][warp] = base; red[1][warp] = Lp; }
    __syncthreads();
    double off = 0;
    for (int w = 0; w < warp; ++w) off += red[0][w];
    if (warp > 0)
      for (int j = j0 + lane; j < j1; j += 32) em[j] = off + em[j];
    if (tid == 0)
      for (int w = 0; w < WARPS; ++w) Lth += red[1][w];
  }
  __syncthreads();
  // cdf_array::normalize: NaN entries to 0, an all-zero row to a flat one
  for (int j = tid; j < nn; j += bd) if (isnan(em[j])) em[j] = 0;
  __syncthreads();
  const bool all_zero = (em[nn - 1] == 0);
  __syncthreads();
  if (all_zero) for (int j = tid; j < nn; j += bd) em[j] = 1.0;
  __syncthreads();
  if (tid == 0) {
    A.L_th[z] = Lth;
    if (nn == 1) {
      A.planck[z] = ab_r[0];
      A.ross[z] = ab_r[0] + sc_r[0];
    } else {
      A.planck[z] = pm_tot / pn_tot;
      A.ross[z] = rn_tot / rm_tot;
    }
    if (A.radiative_eq) A.eps_imc[z] = 1.;
    else {
      const double fleck_beta = 4.0 * A_RAD * pow(A.T[z], 4) / (A.e_gas[z] * A.rho[z]);
      const double tfac = C_LIGHT * A.planck[z] * A.dt;
      double f_imc = A.fleck_alpha * fleck_beta * tfac;
      if (A.fleck_alpha == 0) f_imc = 0.;
      A.eps_imc[z] = 1.0 / (1.0 + f_imc);
    }
  }
  const double N = em[nn - 1];
  __syncthreads();  // every thread has N before em[] is overwritten below
  // normalised CDF, packed tables and the coarse CDF index for the packet kernel
  for (int j = tid; j < nn; j += bd) {
    const size_t k = (size_t)z * nn + j;
    const double c = em[j] / N;
    if constexpr (MIXED) {
      reinterpret_cast<float2*>(A.opac_out)[k] = make_float2((float)ab_r[j], (float)sc_r[j]);
      reinterpret_cast<float*>(A.cdf_out)[k] = (float)c;
    } else {
      reinterpret_cast<double2*>(A.opac_out)[k] = make_double2(ab_r[j], sc_r[j]);
      reinterpret_cast<double*>(A.cdf_out)[k] = c;
    }
    if ((j % CDF_STRIDE) == CDF_STRIDE - 1 || j == nn - 1) {
      const size_t kc = (size_t)z * A.n_coarse + j / CDF_STRIDE;
      if constexpr (MIXED) reinterpret_cast<float*>(A.cdf_coarse_out)[kc] = (float)c;
      else reinterpret_cast<double*>(A.cdf_coarse_out)[kc] = c;
    }
    // the value the packet kernel compares against, as a double
    em[j] = MIXED ? (double)(float)c : c;
  }
  // guide table of the stored row: guide[k] = upper_bound(row, k / G).  In a
  // row that rises from 0 or more to 1 and holds no NaN, that is j for the k
  // with row[j-1] <= k/G < row[j] (G a power of two, so row * G is exact) and
  // nn from k = G on: each bin writes the entries it owns, G + 1 in all,
  // instead of a binary search of the row for every entry.  Any other row
  // (an overflowed or a falling one) is searched.
  __syncthreads();
  if constexpr (MIXED)
    if (A.bin4_out)
      for (int j = tid; j < nn; j += bd)
        A.bin4_out[(size_t)z * nn + j] =
            make_float4(j ? (float)em[j - 1] : 0.f, (float)em[j], (float)ab_r[j], (float)sc_r[j]);
  if (A.cdf_guide_out) {
    const int G = A.guide_n;
    uint16_t* gz = A.cdf_guide_out + (size_t)z * (G + 1);
    bool rises = true;
    for (int j = tid; j < nn; j += bd) rises = rises && ((j ? em[j - 1] : 0.0) <= em[j]) && em[j] <= 1.0;
    if (__syncthreads_and(rises && em[nn - 1] == 1.0)) {
      for (int j = tid; j < nn; j += bd) {
        const int k0 = j ? (int)ceil(em[j - 1] * (double)G) : 0, k1 = (int)ceil(em[j] * (double)G);
        for (int k = k0; k < k1; ++k) gz[k] = (uint16_t)j;
      }
      if (tid == 0) gz[G] = (uint16_t)nn;
    } else {
      for (int k = tid; k <= G; k += bd) {
        const double t = (double)k / (double)G;
        int lo = 0, hi = nn;
        while (lo < hi) {
          const int m = (lo + hi) >> 1;
          if (em[m] <= t) lo = m + 1; else hi = m;
        }
        gz[k] = (uint16_t)lo;
      }
    }
  }
}

// zone tiles of the line-sum kernel: 8 zones per CTA in FP32, 4 in FP64
constexpr int LINE_TILE_MIXED = 8;
constexpr int LINE_TILE_FP64 = 4;

// CTAs per tile: with few zones (a 1D model has 256, 32 tiles of 8) a CTA per
// tile left most SMs without work, so the bins of a tile are dealt over as
// many CTAs as bring the grid to LINE_SUM_CTAS_PER_SM per SM (the 2048 threads
// an SM holds), but at least one bin per warp.  A bin is summed by one warp in
// either case: the sums do not depend on the split.  On B200, FP32: 256 zones x
// 4096 bins x 5e5 lines 3.18 ms -> 344 us, 128 x 2048 x 1e5 725 -> 47 us, 97 x
// 1500 x 3e4 293 -> 21 us; 18 494 zones (2312 tiles, unsplit as before) 2.03 ms.
constexpr int LINE_SUM_CTAS_PER_SM = 8;

template <bool MIXED, bool FUZZ>
int launch_line_sums(const OpacityArgs& a, double* S, double* Se, int num_sms, cudaStream_t s)
{
  constexpr int ZT = MIXED ? LINE_TILE_MIXED : LINE_TILE_FP64;
  const size_t vs = MIXED ? sizeof(float) : sizeof(double);
  const size_t np = FUZZ ? (size_t)a.n_ions_total : (size_t)a.n_lev_total;
  const size_t smem = vs * ((size_t)a.natoms * ZT + a.natoms + ZT + 2 * np * ZT);
  auto k = line_sum_kernel<MIXED, FUZZ, ZT>;
  if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return -1;
  const int tiles = (a.nzones + ZT - 1) / ZT;
  const int bin_groups = (a.n_nu + LINE_SUM_WARPS - 1) / LINE_SUM_WARPS;
  const int want = (num_sms * LINE_SUM_CTAS_PER_SM + tiles - 1) / tiles;
  const dim3 grid((unsigned)tiles, (unsigned)std::min(std::min(want, bin_groups), 65535));
  k<<<grid, 32 * LINE_SUM_WARPS, smem, s>>>(a, S, Se);
  return 1;
}

}  // namespace

int launch_bin_table(const DevLoc& nu, double* tab, double2* lr, cudaStream_t s)
{
  bin_table_kernel<<<(nu.n + 127) / 128, 128, 0, s>>>(nu, tab, lr);
  return 1;
}

int launch_guide(int precision, const void* cdf, int64_t nz, int nn, uint16_t* guide, int G, int num_sms,
                 cudaStream_t s)
{
  const unsigned b = (unsigned)num_sms * 8;
  if (precision) guide_kernel<<<b, 256, 0, s>>>(static_cast<const float*>(cdf), nz, nn, guide, G);
  else guide_kernel<<<b, 256, 0, s>>>(static_cast<const double*>(cdf), nz, nn, guide, G);
  return 1;
}

int launch_pack_bins(const void* opac, const void* cdf, int64_t nz, int nn, float4* out, int num_sms, cudaStream_t s)
{
  pack_bins_kernel<<<num_sms * 8, 256, 0, s>>>(static_cast<const float2*>(opac), static_cast<const float*>(cdf),
                                               nz * nn, nn, out);
  return 1;
}

size_t opacity_smem_bytes(const OpacityArgs& a)
{
  size_t d = (size_t)a.natoms;
  if (a.smem_rows) d += 3 * (size_t)a.n_nu;
  return d * sizeof(double);
}

size_t line_sum_smem_bytes(int precision, int natoms, int n_pop)
{
  const int ZT = precision ? LINE_TILE_MIXED : LINE_TILE_FP64;
  const size_t vs = precision ? sizeof(float) : sizeof(double);
  return vs * ((size_t)natoms * ZT + natoms + ZT + 2 * (size_t)n_pop * ZT);
}

template <bool MIXED, int THREADS>
static int launch_zone_opacity(const OpacityArgs& a, cudaStream_t s)
{
  const size_t smem = opacity_smem_bytes(a);
  auto k = a.use_bf ? zone_opacity_kernel<MIXED, THREADS, true> : zone_opacity_kernel<MIXED, THREADS, false>;
  if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return -1;
  k<<<a.nzones, THREADS, smem, s>>>(a);
  return 1;
}

int launch_opacity(const OpacityArgs& a, int num_sms, cudaStream_t s)
{
  const int nz = a.nzones;
  int n = 0;
  if (launch_zone_state(a, num_sms, s) < 0) return -1;
  ++n;
  const bool micro = a.natoms > 0;
  int r = 0;
  if (micro && a.use_line)
    r = a.precision ? launch_line_sums<true, false>(a, a.abs64, a.epsl64, num_sms, s)
                    : launch_line_sums<false, false>(a, a.abs64, a.epsl64, num_sms, s);
  if (r < 0) return -1;
  n += r;
  r = 0;
  if (micro && a.use_fuzz)
    r = a.precision ? launch_line_sums<true, true>(a, a.scat64, a.epsf64, num_sms, s)
                    : launch_line_sums<false, true>(a, a.scat64, a.epsf64, num_sms, s);
  if (r < 0) return -1;
  n += r;
  // with at most two zones per SM a CTA's warps are all the SM has: 1024
  // threads share a zone's bins, unless the FP64 row's serial sums are what
  // the CTA waits for
  const bool wide = nz <= 2 * num_sms && a.n_nu > 256 && (a.precision || a.use_bf);
  r = a.precision ? (wide ? launch_zone_opacity<true, 1024>(a, s) : launch_zone_opacity<true, 256>(a, s))
                  : (wide ? launch_zone_opacity<false, 1024>(a, s) : launch_zone_opacity<false, 256>(a, s));
  if (r < 0) return -1;
  return n + 1;
}

}  // namespace sed

// ---------------------------------------------------------------------------
// LTE electron densities without any device allocation.
//
// Some callers cannot allocate device memory at the point where they need
// this result: a host code whose device memory is entirely handed out by its
// own pool allocator, or one that runs the solve inside a per-step loop where
// the implicit synchronisation of cudaMalloc/cudaFree is not acceptable.
// They own the inputs and the outputs.  The per-zone working set of the
// solve (mass fractions, number densities, clamped temperature, partition
// functions, ion fractions, level populations, Boltzmann factors) lives in
// the fixed array below, which is part of the library image: every GPU that
// loads the library holds it until the process exits.
namespace {
constexpr size_t NOALLOC_SCRATCH_DOUBLES = size_t(1) << 19;  // 4 MiB per device
__device__ __align__(256) double g_lte_scratch[NOALLOC_SCRATCH_DOUBLES];

constexpr int NOALLOC_MAX_DEVICES = 64;
std::mutex g_scratch_mutex;
double* g_scratch_addr[NOALLOC_MAX_DEVICES] = {};
}  // namespace

extern "C" int sed_lte_electron_density_noalloc(int32_t n_zones, const double* rho, const double* T_gas,
                                                const double* X, int32_t n_elems, const int32_t* elem_A,
                                                const sed_atomic_data* atoms_dev, int32_t n_ions_total,
                                                int32_t n_levels_total, double temp_min, double temp_max,
                                                double* n_elec, int32_t* solve_err, void* stream)
{
  using namespace sed;
  if (n_zones <= 0 || n_elems <= 0 || n_ions_total <= 0 || n_levels_total <= 0) return SED_ERR_ARG;
  if (!rho || !T_gas || !X || !elem_A || !atoms_dev || !n_elec || !solve_err) return SED_ERR_ARG;
  if (atoms_dev->n_atoms != n_elems || !atoms_dev->ion_off || !atoms_dev->ion_chi || !atoms_dev->lev_off ||
      !atoms_dev->lev_ion || !atoms_dev->lev_g || !atoms_dev->lev_E)
    return SED_ERR_ARG;
  const size_t nz = (size_t)n_zones, na = (size_t)n_elems;
  const size_t ni = (size_t)n_ions_total, nl = (size_t)n_levels_total;
  // doubles per zone, then zones: the limit is checked as a quotient so that
  // no product of the caller's counts can wrap around
  const size_t per_zone = 2 * na + 2 + 2 * ni + 2 * nl;
  if (per_zone > NOALLOC_SCRATCH_DOUBLES || nz > NOALLOC_SCRATCH_DOUBLES / per_zone)
    return SED_ERR_CAPACITY;  // limit stated in include/sedona_gpu.h

  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= NOALLOC_MAX_DEVICES) return SED_ERR_CUDA;
  double* base = nullptr;
  {
    // first call on this device: look up the array's device address with
    // this device current (the host-side symbol is only a stand-in)
    std::lock_guard<std::mutex> lock(g_scratch_mutex);
    if (!g_scratch_addr[dev]) {
      void* p = nullptr;
      if (cudaGetSymbolAddress(&p, g_lte_scratch) != cudaSuccess || !p) return SED_ERR_CUDA;
      g_scratch_addr[dev] = static_cast<double*>(p);
    }
    base = g_scratch_addr[dev];
  }
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  OpacityArgs A{};
  A.nzones = n_zones;
  A.nelem = n_elems;
  A.natoms = n_elems;
  A.temp_min = temp_min;
  A.temp_max = temp_max;
  A.rho = rho;
  A.T = T_gas;
  A.X = X;
  A.eA = elem_A;
  A.ion_off = atoms_dev->ion_off;
  A.ion_chi = atoms_dev->ion_chi;
  A.lev_off = atoms_dev->lev_off;
  A.lev_ion = atoms_dev->lev_ion;
  A.lev_g = atoms_dev->lev_g;
  A.lev_E = atoms_dev->lev_E;
  A.n_ions_total = n_ions_total;
  A.n_lev_total = n_levels_total;
  // carve the scratch array
  double* q = base;
  A.mass_frac = q;  q += na * nz;
  A.n_dens = q;     q += na * nz;
  A.temp_c = q;     q += nz;
  double* grey = q; q += nz;  // all zones take the microphysical path: zero grey opacity
  A.ion_part = q;   q += ni * nz;
  A.ion_frac = q;   q += ni * nz;
  A.lev_n = q;      q += nl * nz;
  A.boltz = q;      q += nl * nz;
  A.grey = grey;
  A.n_elec = n_elec;
  A.solve_err = solve_err;
  // the array keeps the previous call's contents; only the grey-opacity
  // column must start at zero (every other entry is written before it is read)
  if (cudaMemsetAsync(grey, 0, nz * sizeof(double), s) != cudaSuccess) return SED_ERR_CUDA;
  int num_sms = 0;
  if (cudaDeviceGetAttribute(&num_sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return SED_ERR_CUDA;
  if (launch_zone_state(A, num_sms, s) < 0) return SED_ERR_CUDA;
  return cudaGetLastError() == cudaSuccess ? SED_OK : SED_ERR_CUDA;
}
