// diff_kernel.cuh -- differentiable transport on FP32 tables (homologous 1D
// spheres and 3D Cartesian grids): MODE 1 the weighted forward, MODE 2 the
// adjoint replay of its escaped packets.  Included by transport_kernel.cu
// inside its anonymous namespace, after the shared helpers.
//
// Packets take the paths propagate_kernel's division-free form gives them in
// these modes, to the bit (a replay has to walk the forward's paths, and both
// what propagate_kernel walked): the same expressions, deviates and rounding.
// Like there, a step is bound by the chain of a packet's segments (the escaped
// eighth of the Type Ia packets holds 98 % of them).  What is shorter here:
// the zone's walls are held for the visit, the frequency bin comes from the
// FP32 index estimate alone where that is clear of a wall, the wall distances
// take branch-free square roots (sed_common.cuh), the blocks of a segment and
// of its scattering are formed together, a bin's band is a 32-bit division,
// and a segment's attenuation is its Taylor series where the absorption depth
// is below 1/64 (exp and expm1 beyond).  Sums that no path depends on (zone
// tallies, in the thread's shared-memory slots and 32 global copies) are
// ordered freely.  Type Ia, 1e6 packets: forward 117 -> 85 ms, replay 81 -> 72
// ms, and 56 ms in order of length (below).

// (1 - exp(-x)) / x for 0 <= x < 1/64: the series 1 - x/2 + x^2/6 - ... to
// x^7 (the next term is below 2^-63)
__device__ __forceinline__ double mean_attenuation(double x)
{
  double s = 1.0 / 40320;
  s = fma(-x, s, 1.0 / 5040);
  s = fma(-x, s, 1.0 / 720);
  s = fma(-x, s, 1.0 / 120);
  s = fma(-x, s, 1.0 / 24);
  s = fma(-x, s, 1.0 / 6);
  s = fma(-x, s, 0.5);
  return fma(-x, s, 1.0);
}

// The replay's queue: the escaped packets by decreasing segment count, which
// the forward recorded (buckets of 1/64 of a factor of two, any order within
// one).  The lanes of a warp then end their packets at nearly the same time;
// in queue order a warp waited for the longest of its 32, with ever fewer
// lanes at work (Type Ia, 1e6 packets, 1.3e5 of them escaped with 8 000 to
// 27 000 segments: replay 72.2 -> 55.7 ms).
__device__ __forceinline__ int replay_bucket(int32_t seg)
{
  const int b = (__float_as_int((float)max(seg, 1)) >> 17) - (127 << 6);
  return REPLAY_BUCKETS - 1 - min(max(b, 0), REPLAY_BUCKETS - 1);
}

__global__ void replay_count_kernel(const int32_t* __restrict__ esc_bin, const int32_t* __restrict__ esc_seg, int64_t n,
                                    int32_t* __restrict__ cursor)
{
  __shared__ int32_t s_n[REPLAY_BUCKETS];
  for (int i = threadIdx.x; i < REPLAY_BUCKETS; i += blockDim.x) s_n[i] = 0;
  __syncthreads();
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    if (esc_bin[i] >= 0) atomicAdd(s_n + replay_bucket(esc_seg[i]), 1);
  __syncthreads();
  for (int i = threadIdx.x; i < REPLAY_BUCKETS; i += blockDim.x)
    if (s_n[i]) atomicAdd(cursor + i, s_n[i]);
}

// counts -> first places (one CTA of 1024 threads, two buckets each); cursor[REPLAY_BUCKETS]: their sum
__global__ void replay_scan_kernel(int32_t* __restrict__ cursor)
{
  static_assert(REPLAY_BUCKETS == 2048, "two buckets per thread");
  __shared__ int32_t s[32];
  const int t = threadIdx.x, lane = t & 31;
  const int32_t a = cursor[2 * t], b = cursor[2 * t + 1];
  int32_t v = a + b;
  for (int o = 1; o < 32; o <<= 1) {
    const int32_t u = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += u;
  }
  if (lane == 31) s[t >> 5] = v;
  __syncthreads();
  int32_t base = 0;
  for (int w = 0; w < (t >> 5); ++w) base += s[w];
  cursor[2 * t] = base + v - a - b;
  cursor[2 * t + 1] = base + v - b;
  if (t == 1023) cursor[REPLAY_BUCKETS] = base + v;
}

__global__ void replay_place_kernel(const int32_t* __restrict__ esc_bin, const int32_t* __restrict__ esc_seg, int64_t n,
                                    int32_t* __restrict__ cursor, int32_t* __restrict__ order)
{
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    if (esc_bin[i] >= 0) order[atomicAdd(cursor + replay_bucket(esc_seg[i]), 1)] = (int32_t)i;
}

template <int GRID, int MODE, int THREADS, int MINB>
__global__ void __launch_bounds__(THREADS, MINB) propagate_diff_kernel(const StepArgs A, const GridDev G)
{
  __shared__ unsigned long long s_cnt[6];
  __shared__ double s_acc[MODE == 1 ? 5 : 1][THREADS];  // e_abs, fx, fy, fz, fr of the zone visit
  __shared__ unsigned long long s_pid[THREADS];
  const int tid = threadIdx.x;
  if (tid < 6) s_cnt[tid] = 0;
  if constexpr (MODE == 1)
    for (int k = 0; k < 5; ++k) s_acc[k][tid] = 0.0;
  __syncthreads();
  const int nz = G.nzones, nn = A.nu.n;
  const int nj = A.store_Jnu ? nn : 1;
  const int64_t rep_off = (A.n_rep > 0) ? (int64_t)(blockIdx.x % A.n_rep) * 5 * nz : -1;
  const float2* __restrict__ opac = reinterpret_cast<const float2*>(A.opac);
  const int32_t limit = A.max_segments > 0 ? A.max_segments : 10000000;
  const uint32_t K = ((A.core_radius == 0 ? 2u : 4u) + (A.core_freq > 0 ? 0u : 2u) + 1u + 3u) / 4u;
  const int64_t n_queue = (MODE == 2 && A.replay_order) ? __ldg(A.n_replay) : A.n_packets;
  const bool wide_band = (int64_t)nn * A.n_bands > 0xFFFFFFFFll;
  Pkt p;
  p.dvds = 0;
  uint64_t stream = 0;
  uint32_t n_blk = 0;
  int fate = ABSORBED;
  bool have = false, live = (tid & 31) < A.lanes;
  int32_t seg = 0, n_scat = 0;
  int acc = -1;           // zone of the visit
  double r_o = 0, r_in = 0;
  int ind_in = -1;
  double adj_w = 0, acc_g = 0;  // replay: the packet's weight, the sum of one (zone, band)
  int64_t adj_row = 0, acc_key = -1;
  auto block = [&](uint32_t n) { return philox_words(A, stream, n); };
  auto flush = [&](int z) {
    mixed::add_visit(A, nullptr, nz, rep_off, z, s_acc[0][tid], s_acc[MODE == 1 ? 1 : 0][tid],
                     s_acc[MODE == 1 ? 2 : 0][tid], s_acc[MODE == 1 ? 3 : 0][tid], s_acc[MODE == 1 ? 4 : 0][tid]);
    for (int k = 0; k < 5; ++k) s_acc[MODE == 1 ? k : 0][tid] = 0.0;
  };
  for (;;) {
    __syncwarp();  // the lanes of the warp meet every iteration (propagate_mixed_kernel)
    if (!__any_sync(0xffffffffu, live)) break;
    if (!live) continue;
    if (fate != MOVING) {
      if (have) {
        atomicAdd(s_cnt + 3, (unsigned long long)seg);
        atomicAdd(s_cnt + 4, (unsigned long long)n_scat);
        if constexpr (MODE == 2) {
          if (acc_key >= 0) atomicAdd(A.adj_out + acc_key, -adj_w * acc_g);
        } else {
          const unsigned long long pid = s_pid[tid];
          if (acc >= 0) flush(acc);
          if (fate == ESCAPED) {
            const double t_obs = p.t - (p.x[0] * p.D[0] + p.x[1] * p.D[1] + p.x[2] * p.D[2]) / C_LIGHT;
            A.esc_bin[pid] = (int32_t)spectrum_count(A, A.flux, A.click, t_obs, p.nu, p.e, p.D);
            A.esc_e[pid] = p.e;
            A.esc_seg[pid] = seg;
            p.t = t_obs;
            atomicAdd(s_cnt + 0, 1ULL);
          } else {
            A.esc_bin[pid] = -1;
            atomicAdd(s_cnt + (fate == ABSORBED ? 1 : 2), 1ULL);
          }
          if (A.rec_fate) {
            A.rec_fate[pid] = fate;
            A.rec_ind[pid] = p.ind;
            A.rec_draws[pid] = (int32_t)(n_blk - K);
            if (A.rec_type) A.rec_type[pid] = TYPE_PHOTON;
            double* s = A.rec_state + pid * 9;
            s[0] = p.x[0]; s[1] = p.x[1]; s[2] = p.x[2];
            s[3] = p.D[0]; s[4] = p.D[1]; s[5] = p.D[2];
            s[6] = p.t; s[7] = p.e; s[8] = p.nu;
          }
        }
        have = false;
      }
      unsigned long long pid = atomicAdd(A.counters + C_QUEUE, 1ULL);
      if (pid >= (unsigned long long)n_queue) { live = false; continue; }
      if (MODE == 2 && A.replay_order) pid = (unsigned long long)__ldg(A.replay_order + pid);
      s_pid[tid] = pid;
      if constexpr (MODE == 2) {
        // only packets that reached the spectrum carry a gradient
        const int32_t sb = A.esc_bin[pid];
        adj_w = 0;
        if (sb >= 0) adj_w = A.adj_jacobian ? A.esc_e[pid] : A.adj_g[sb] * A.esc_e[pid];
        if (adj_w == 0) continue;  // fate is not MOVING: pull the next packet
        adj_row = A.adj_jacobian ? (int64_t)sb * nz * A.n_bands : 0;
        acc_key = -1;
        acc_g = 0;
      }
      PacketRng er;
      er.init(A.seed, (uint64_t)A.first_pid + pid, A.step, 0);
      DrawWords d{er};
      emit_core<GRID>(A, G, p, d, A.core_radius, A.Ep, A.core_cdf, GridZoneOf<GRID>{G});
      stream = er.pid;
      n_blk = er.n;
      fate = MOVING;
      if (p.ind == -1) fate = ABSORBED;
      else if (p.ind == -2) fate = ESCAPED;
      seg = 0;
      n_scat = 0;
      acc = -1;
      have = true;
      if (fate != MOVING) continue;
    }
    // ------------------------------------------------------------- segment
    if (seg >= limit) { fate = STOPPED; atomicAdd(s_cnt + 5, 1ULL); continue; }
    ++seg;
    const int iz = p.ind;
    if (iz != acc) {
      if (MODE == 1 && acc >= 0) flush(acc);
      acc = iz;
      if constexpr (GRID == 0) {
        r_o = __ldg(G.r_out.right + iz);
        r_in = (iz != 0) ? __ldg(G.r_out.right + iz - 1) : G.r_out.min;
        ind_in = (iz != 0) ? iz - 1 : -1;
        if (A.core_radius >= r_in) { r_in = A.core_radius; ind_in = -1; }
      }
    }
    const uint4 blk = block(n_blk);
    const double rsq = fma(p.x[0], p.x[0], fma(p.x[1], p.x[1], p.x[2] * p.x[2]));
    const double xdotD = fma(p.D[0], p.x[0], fma(p.D[1], p.x[1], p.D[2] * p.x[2]));
    double d_bn;
    int new_ind;
    if constexpr (GRID == 0)
      new_ind = next_zone_rn(r_o, r_in, ind_in, (iz + 1 == nz) ? -2 : iz + 1, (iz == 0) && (r_in == 0), rsq, xdotD,
                             &d_bn);
    else new_ind = get_next_zone<GRID, true>(G, p.x, p.D, iz, A.core_radius, rsq, xdotD, &d_bn);
    const double dshift = dshift_fast(A, rsq, xdotD);
    const int i_nu = loc_within_mixed(A.nu, p.nu * dshift);
    const float2 ab = __ldg(opac + (size_t)iz * nn + i_nu);
    const int band = wide_band ? (int)(((int64_t)i_nu * A.n_bands) / nn)
                               : (int)(((uint32_t)i_nu * (uint32_t)A.n_bands) / (uint32_t)nn);
    double a_opac = (double)ab.x;
    const double s_opac = A.omit_scat ? 0.0 : (double)ab.y;
    if (A.abs_scale) a_opac *= __ldg(A.abs_scale + (size_t)iz * A.n_bands + band);
    double d_nu = (double)__fdividef((float)(loc_delta(A.nu, i_nu) * A.ct), (float)p.nu);
    if (d_nu < 0) d_nu = -1 * d_nu;
    if (d_nu < d_bn) { d_bn = d_nu; new_ind = iz; }
    const double tot_lab = s_opac * dshift;
    const double u = u01(blk.x, blk.y);
    const double tau_r = (double)((u < 0.5) ? -log1pf(-(float)u) : -logf((float)(1.0 - u)));
    double d_sc = (double)__fdividef((float)tau_r, (float)tot_lab);
    if (tot_lab == 0) d_sc = INFINITY;
    double d_tm = (A.tstop - p.t) * C_LIGHT;
    if (A.steady) d_tm = INFINITY;
    int event;
    double this_d;
    if ((d_sc < d_bn) && (d_sc < d_tm)) { event = 0; this_d = d_sc; }
    else if (d_bn < d_tm) { event = 1; this_d = d_bn; }
    else { event = 2; this_d = d_tm; }
    if constexpr (MODE == 1) {
      // absorption over the segment: the weight falls by exp(-tau_a); the
      // tallies use its segment average e (1 - exp(-tau_a)) / tau_a
      const double tau_a = a_opac * dshift * this_d;
      double mean, att;
      if (tau_a >= 0 && tau_a < 0.015625) {
        mean = mean_attenuation(tau_a);
        att = fma(-tau_a, mean, 1.0);
      } else {
        att = exp(-tau_a);
        mean = (tau_a > 0) ? -expm1(-tau_a) / tau_a : 1.0;
      }
      const double this_E = p.e * mean * this_d;
      const double ed = this_E * dshift;
      s_acc[0][tid] += ed * a_opac * dshift * __ldg(A.eps_imc + iz);
      atomicAdd(A.J + (size_t)iz * nj + (A.store_Jnu ? i_nu : 0), this_E);
      if (A.tally_forces) {
        const double w = ed * (a_opac + s_opac) * dshift;
        s_acc[1][tid] += w * p.D[0];
        s_acc[2][tid] += w * p.D[1];
        s_acc[3][tid] += w * p.D[2];
        s_acc[4][tid] += w * xdotD * rsqrt_nr(rsq);
      }
      p.e *= att;
    } else {
      const int64_t key = A.adj_density ? iz : adj_row + (int64_t)iz * A.n_bands + band;
      if (key != acc_key) {
        if (acc_key >= 0) atomicAdd(A.adj_out + acc_key, -adj_w * acc_g);
        acc_key = key;
        acc_g = 0;
      }
      if (A.adj_density) {
        // d / d ln rho of zone iz, opacity per mass held: the weight's log
        // falls by a dshift l, the sampled path's log-likelihood by
        // s dshift l per segment and rises by one per scattering
        acc_g += (a_opac + s_opac) * dshift * this_d;
        if (event == 0) acc_g -= 1.0;
      } else {
        acc_g += (double)ab.x * dshift * this_d;  // d(theta a0 dshift l) / d theta
      }
    }
    p.x[0] += this_d * p.D[0];
    p.x[1] += this_d * p.D[1];
    p.x[2] += this_d * p.D[2];
    constexpr double INV_C = 1.0 / C_LIGHT;
    p.t = p.t + this_d * INV_C;
    ++n_blk;
    if (event == 1) {
      if (new_ind == -1) {
        if (A.bound_in_reflect) { p.D[0] *= -1; p.D[1] *= -1; p.D[2] *= -1; }
        else { p.ind = new_ind; fate = ABSORBED; }
      } else if (new_ind == -2) {
        if (A.bound_out_reflect) { p.D[0] *= -1; p.D[1] *= -1; p.D[2] *= -1; }
        else { p.ind = new_ind; fate = ESCAPED; }
      } else {
        p.ind = new_ind;
      }
    } else if (event == 0) {
      ++n_scat;
      isotropic_scatter_fast(A, p, block(n_blk), 0);
      ++n_blk;
    } else {
      fate = STOPPED;
    }
  }
  __syncthreads();
  if (tid < 6) {
    constexpr int slot[6] = {C_ESCAPED, C_ABSORBED, C_STOPPED, C_SEGMENTS, C_SCATTERS, C_LIMIT};
    const unsigned long long v = s_cnt[tid];
    if (v) atomicAdd(A.counters + slot[tid], v);
  }
}
