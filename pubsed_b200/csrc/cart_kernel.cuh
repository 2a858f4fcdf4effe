// cart_kernel.cuh -- the mixed-form packet kernel on 3D Cartesian grids (FP32
// {abs, scat} tables and emissivity CDF, FP64 packet state).  Included by
// transport_kernel.cu inside its anonymous namespace, after the shared
// helpers.
//
// Packets have the histories propagate_kernel's division-free form gives them
// on these grids, to the bit: the same expressions, deviates (one Philox block
// per segment, one per interaction) and rounding.  A third of the segments end
// in an interaction, the others at cell walls and bin edges, and every new cell
// or bin is a gather from tables far beyond the L2: the kernel waits for DRAM
// latency, so what counts is how many warps wait at once and how little else
// each segment holds them for.  Here a lane carries its cell as three indices
// (no division of the zone index), takes the pushed walls from a table per
// axis, keeps the reciprocals of its direction, the visit's tallies and its
// start and end state in its own shared-memory slots, and finds its bin by the
// FP32 estimate; core packets are emitted ahead (emit_mixed_kernel) and escaped
// ones binned into the spectrum afterwards, so neither long stretch holds a
// warp for one of its lanes.

// EMIT = 0: a step of core packets alone, emitted ahead into em_state, where an
// escaped packet's {t_obs, e, nu, D} are left for count_escaped_kernel (its
// em_ind ESCAPED_SLOT); EMIT = 1: any step, packets emitted and counted here.
constexpr int32_t ESCAPED_SLOT = -3;

template <int EMIT, int THREADS, int MINB>
__global__ void __launch_bounds__(THREADS, MINB) propagate_cart_kernel(const StepArgs A, const GridDev G)
{
  __shared__ unsigned long long s_cnt[6];
  __shared__ double s_acc[5][THREADS];  // e_abs, fx, fy, fz, fr of the cell visit
  __shared__ double s_inv[3][THREADS];  // 1/D
  __shared__ unsigned long long s_pid[THREADS];
  __shared__ uint32_t s_k0[THREADS];
  __shared__ int s_scat[THREADS];
  const int tid = threadIdx.x;
  if (tid < 6) s_cnt[tid] = 0;
#pragma unroll
  for (int k = 0; k < 5; ++k) s_acc[k][tid] = 0.0;
  __syncthreads();
  const int nn = A.nu.n, nyz = G.ny * G.nz;
  const int64_t rep_off = (A.n_rep > 0) ? (int64_t)(blockIdx.x % A.n_rep) * 5 * G.nzones : -1;
  const int nj = A.store_Jnu ? nn : 1;
  double* __restrict__ J = tally_J(A, G.nzones, nj);
  const float2* __restrict__ opac = reinterpret_cast<const float2*>(A.opac);
  const int32_t limit = A.max_segments > 0 ? A.max_segments : 10000000;
  const uint32_t K = ((A.core_radius == 0 ? 2u : 4u) + (A.core_freq > 0 ? 0u : 2u) + 1u + 3u) / 4u;
  Pkt p;
  p.dvds = 0;
  uint64_t stream = 0;
  uint32_t n_blk = 0;
  int c0 = 0, c1 = 0, c2 = 0;  // the cell
  int fate = ABSORBED;
  bool have = false, live = (tid & 31) < A.lanes;
  int32_t seg = 0;
  int acc = -1;  // cell of the visit
  auto flush = [&](int z) {
    mixed::add_visit(A, nullptr, G.nzones, rep_off, z, s_acc[0][tid], s_acc[1][tid], s_acc[2][tid], s_acc[3][tid], s_acc[4][tid]);
#pragma unroll
    for (int k = 0; k < 5; ++k) s_acc[k][tid] = 0.0;
  };
  auto directions = [&]() {
#pragma unroll
    for (int a = 0; a < 3; ++a) s_inv[a][tid] = rcp_nr(p.D[a]);
  };
  for (;;) {
    __syncwarp();  // the lanes of the warp meet every iteration (propagate_mixed_kernel)
    if (!__any_sync(0xffffffffu, live)) break;
    if (!live) continue;
    if (fate != MOVING) {
      if (have) {
        if (acc >= 0) { flush(acc); acc = -1; }
        atomicAdd(s_cnt + 3, (unsigned long long)seg);
        atomicAdd(s_cnt + 4, (unsigned long long)s_scat[tid]);
        const unsigned long long pid = s_pid[tid];
        if (fate == ESCAPED) {
          const double t_obs = p.t - (p.x[0] * p.D[0] + p.x[1] * p.D[1] + p.x[2] * p.D[2]) / C_LIGHT;
          if constexpr (EMIT) {
            spectrum_count(A, A.flux, A.click, t_obs, p.nu, p.e, p.D);
          } else {
            double* s = A.em_state + pid;
            const int64_t n = A.em_n;
            s[0] = t_obs; s[n] = p.e; s[2 * n] = p.nu;
            s[3 * n] = p.D[0]; s[4 * n] = p.D[1]; s[5 * n] = p.D[2];
            A.em_ind[pid] = ESCAPED_SLOT;
          }
          p.t = t_obs;
          atomicAdd(s_cnt + 0, 1ULL);
        } else {
          atomicAdd(s_cnt + (fate == ABSORBED ? 1 : 2), 1ULL);
        }
        if (A.rec_fate) {
          A.rec_fate[pid] = fate;
          A.rec_ind[pid] = p.ind;
          A.rec_draws[pid] = (int32_t)(n_blk - s_k0[tid]);
          if (A.rec_type) A.rec_type[pid] = TYPE_PHOTON;
          double* s = A.rec_state + pid * 9;
          s[0] = p.x[0]; s[1] = p.x[1]; s[2] = p.x[2];
          s[3] = p.D[0]; s[4] = p.D[1]; s[5] = p.D[2];
          s[6] = p.t; s[7] = p.e; s[8] = p.nu;
        }
        have = false;
      }
      const unsigned long long pid = atomicAdd(A.counters + C_QUEUE, 1ULL);
      if (pid >= (unsigned long long)A.n_packets) { live = false; continue; }
      s_pid[tid] = pid;
      if constexpr (EMIT) {
        if (A.q_n != nullptr && (int64_t)pid >= A.n_core) {
          // a queued photon: census (stream position 0) or an optical photon
          // the gamma-ray kernel handed over at its stream position
          const int64_t k = (int64_t)pid - A.n_core;
          const uint32_t qn = A.q_n[k];
          if (qn == RADIO_NO_PHOTON) continue;
          const double* q = A.q_state + (size_t)k * 9;
          p.x[0] = q[0]; p.x[1] = q[1]; p.x[2] = q[2];
          p.D[0] = q[3]; p.D[1] = q[4]; p.D[2] = q[5];
          p.t = q[6]; p.e = q[7]; p.nu = q[8];
          p.ind = A.q_ind[k];
          stream = (uint64_t)(A.radio_first_pid + k);
          n_blk = qn;
          s_k0[tid] = 0;  // a radioactive packet records every deviate of its stream
        } else {
          PacketRng er;
          er.init(A.seed, (uint64_t)A.first_pid + pid, A.step, 0);
          DrawWords d{er};
          emit_core<1>(A, G, p, d, A.core_radius, A.Ep, A.core_cdf, GridZoneOf<1>{G});
          stream = er.pid;
          n_blk = er.n;
          s_k0[tid] = K;
        }
      } else {
        mixed::load_emitted(A, p, (int64_t)pid);
        stream = (uint64_t)A.first_pid + pid;
        n_blk = K;
        s_k0[tid] = K;
      }
      fate = MOVING;
      if (p.ind == -1) fate = ABSORBED;
      else if (p.ind == -2) fate = ESCAPED;
      seg = 0;
      s_scat[tid] = 0;
      have = true;
      if (fate != MOVING) continue;
      c0 = p.ind / nyz;
      c1 = (p.ind / G.nz) % G.ny;
      c2 = p.ind % G.nz;
      directions();
    }
    // ------------------------------------------------------------- segment
    if (seg >= limit) { fate = STOPPED; atomicAdd(s_cnt + 5, 1ULL); continue; }
    ++seg;
    const int iz = p.ind;
    if (iz != acc) {
      if (acc >= 0) flush(acc);
      acc = iz;
    }
    const double rsq = fma(p.x[0], p.x[0], fma(p.x[1], p.x[1], p.x[2] * p.x[2]));
    const double xdotD = fma(p.D[0], p.x[0], fma(p.D[1], p.x[1], p.D[2] * p.x[2]));
    const double dshift = dshift_fast(A, rsq, xdotD);
    const int i_nu = loc_within_mixed(A.nu, p.nu * dshift);
    const float2 ab = __ldg(opac + (size_t)iz * nn + i_nu);
    // the next cell (get_next_zone), while the opacities are on their way
    double len[3];
    {
      const int c[3] = {c0, c1, c2};
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const double* w = reinterpret_cast<const double*>(A.ax_push[a] + c[a]);
        const double bn = __ldg(w + (p.D[a] > 0 ? 1 : 0));
        len[a] = (p.D[a] != 0.0) ? (bn - p.x[a]) * s_inv[a][tid] : (double)INFINITY;
      }
    }
    int ax = 2;
    if ((len[0] < len[1]) && (len[0] < len[2])) ax = 0;
    else if (len[1] < len[2]) ax = 1;
    double d_bn = (ax == 0) ? len[0] : (ax == 1) ? len[1] : len[2];
    bool leaves = true;  // the segment ends at the cell's wall rather than the bin's
    double d_nu = (double)__fdividef((float)(loc_delta(A.nu, i_nu) * A.ct), (float)p.nu);
    if (d_nu < 0) d_nu = -1 * d_nu;
    if (d_nu < d_bn) { d_bn = d_nu; leaves = false; }
    const uint4 blk = philox_words(A, stream, n_blk);
    const double a_opac = (double)ab.x;
    const double s_opac = A.omit_scat ? 0.0 : (double)ab.y;
    const double op = a_opac + s_opac;
    const double tot_lab = op * dshift;
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
    // tallies (transport.cpp:361-392)
    const double this_E = p.e * this_d;
    atomicAdd(J + (size_t)iz * nj + (A.store_Jnu ? i_nu : 0), this_E);
    const double eps_imc = __ldg(A.eps_imc + iz);
    const double ed = this_E * dshift;
    s_acc[0][tid] += ed * dshift * a_opac * eps_imc;
    if (A.tally_forces) {
      const double w = ed * op * dshift;
      s_acc[1][tid] += w * p.D[0];
      s_acc[2][tid] += w * p.D[1];
      s_acc[3][tid] += w * p.D[2];
      s_acc[4][tid] += w * xdotD * rsqrt_nr(rsq);
    }
    // move
    p.x[0] += this_d * p.D[0];
    p.x[1] += this_d * p.D[1];
    p.x[2] += this_d * p.D[2];
    constexpr double INV_C = 1.0 / C_LIGHT;
    p.t = p.t + this_d * INV_C;
    ++n_blk;
    if (event == 1) {
      if (leaves) {
        const int step = ((ax == 0 ? p.D[0] : ax == 1 ? p.D[1] : p.D[2]) < 0) ? -1 : 1;
        const int to = (ax == 0 ? c0 : ax == 1 ? c1 : c2) + step;
        const int n = (ax == 0) ? G.nx : (ax == 1) ? G.ny : G.nz;
        if (to < 0 || to > n - 1) {
          if (A.bound_out_reflect) {
            p.D[0] *= -1; p.D[1] *= -1; p.D[2] *= -1;
            directions();
          } else {
            p.ind = -2;
            fate = ESCAPED;
          }
        } else {
          if (ax == 0) c0 = to;
          else if (ax == 1) c1 = to;
          else c2 = to;
          p.ind = c0 * nyz + c1 * G.nz + c2;
        }
      }
    } else if (event == 0) {
      // transport::do_scatter (scatter.cpp:12-70)
      s_scat[tid] += 1;
      int redist = 0;
      const double eps = absorbed_part_rn(a_opac, op);
      if (!(w01(blk.z) > eps)) {
        if ((w01(blk.w) > eps_imc) || A.radiative_eq) redist = 1;
        else fate = ABSORBED;
      }
      if (fate == MOVING) {
        isotropic_scatter_fast(A, p, philox_words(A, stream, n_blk), redist);
        ++n_blk;
        directions();
      }
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

// the spectrum of the packets propagate_cart_kernel<0> left as escaped
__global__ void __launch_bounds__(256) count_escaped_kernel(const StepArgs A)
{
  const int64_t n = A.em_n;
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x) {
    if (A.em_ind[q] != ESCAPED_SLOT) continue;
    const double* s = A.em_state + q;
    const double D[3] = {s[3 * n], s[4 * n], s[5 * n]};
    spectrum_count(A, A.flux, A.click, s[0], s[2 * n], s[n], D);
  }
}
