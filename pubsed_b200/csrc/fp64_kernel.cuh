// fp64_kernel.cuh -- the FP64 packet kernel on homologous grids (1D spheres,
// batches of them, 3D Cartesian).  Included by transport_kernel.cu inside its
// anonymous namespace, after the shared helpers.
//
// Every packet has the history propagate_kernel's FP64 form gives it, to the
// bit: the reference's expressions in the reference's order, its deviate
// layout (one 53-bit deviate per draw), IEEE-rounded operations.  What bounds
// the kernel is not the arithmetic's volume but its chain: a packet takes one
// segment after the other, and with CUDA's division and square root, whose
// special-case branches keep the compiler from overlapping one with the next,
// a segment alone took 5.2 us (some 30 divisions of 114 cycles, 7 Philox
// blocks of 150).  Here
//
//  * divisions and square roots are branch-free sequences with the same
//    results (sed_common.cuh), so independent ones overlap; those by c and by
//    the grid time, which never change, start from stored reciprocals;
//  * velocity and Lorentz factor are formed once per position, for the
//    interaction there and for the next segment's Doppler factor;
//  * the blocks of an interaction's deviates are formed together: draws 2k and
//    2k + 1 share a block, so an interaction takes three, not six;
//  * tallies, which no history depends on, use the cheaper forms (e_abs
//    without a / op, |x| from the reciprocal square root) and are summed per
//    zone visit in the thread's own shared-memory slots.

// velocity, |x|^2 and Lorentz factor at a position
struct Flow {
  double v[3], rsq, gamma;
};

__device__ __forceinline__ Flow flow_at(const StepArgs& A, const double* x)
{
  Flow f;
  f.rsq = (x[0] * x[0] + x[1] * x[1] + x[2] * x[2]);
#pragma unroll
  for (int k = 0; k < 3; ++k) f.v[k] = div_by(x[k], A.t_grid, A.inv_t, A.inv_t_lo);
  const double beta2 = div_c(div_c(f.v[0] * f.v[0] + f.v[1] * f.v[1] + f.v[2] * f.v[2]));
  f.gamma = rcp_sqrt_rn(1 - beta2);  // 1.0 / sqrt(1 - beta2)
  return f;
}

// get_next_zone (grid_1D_sphere.cpp:510-590) between the walls r_in, r_o
__device__ __forceinline__ int next_zone_rn(double r_o, double r_in, int ind_in, int ind_out, bool no_inner, double rsq,
                                            double xdotD, double* l)
{
  constexpr double tiny_offset = 1 + 1e-6;
  const double l_out = -1 * xdotD + sqrt_rn(xdotD * xdotD + r_o * r_o - rsq);
  const double rad = xdotD * xdotD + r_in * r_in - rsq;
  const double l_c = -1 * xdotD - sqrt_rn(rad);
  const double l_in = (no_inner || xdotD > 0 || rad < 0) ? -1.0 : l_c;
  const bool out = (l_out < l_in) || (l_in < 0);
  const int ind = out ? ind_out : ind_in;
  const double d = out ? l_out : l_in;
  *l = (ind < 0) ? d / tiny_offset : d * tiny_offset;
  return ind;
}

// grid_3D_cart::get_next_zone (grid_3D_cart.cpp:396-469)
__device__ __forceinline__ int next_cell_rn(const GridDev& G, const double* x, const double* D, int i, double* l)
{
  const int nyz = G.ny * G.nz;
  const int idx3[3] = {i / nyz, (i / G.nz) % G.ny, i % G.nz};
  const double tiny = 1e-10;
  double len[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const double lo = loc_left(G.ax[a], idx3[a]), hi = __ldg(G.ax[a].right + idx3[a]);
    const double dd = hi - lo;
    const double bn = (D[a] > 0) ? hi + dd * tiny : lo - dd * tiny;
    len[a] = div_rn(bn - x[a], D[a]);
    if (D[a] == 0) len[a] = (bn - x[a]) / D[a];
  }
  int d[3] = {0, 0, 0};
  if ((len[0] < len[1]) && (len[0] < len[2])) { d[0] = (D[0] < 0) ? -1 : 1; *l = len[0]; }
  else if (len[1] < len[2]) { d[1] = (D[1] < 0) ? -1 : 1; *l = len[1]; }
  else { d[2] = (D[2] < 0) ? -1 : 1; *l = len[2]; }
  const int nx_ = idx3[0] + d[0], ny_ = idx3[1] + d[1], nz_ = idx3[2] + d[2];
  if (nx_ < 0 || nx_ > G.nx - 1) return -2;
  if (ny_ < 0 || ny_ > G.ny - 1) return -2;
  if (nz_ < 0 || nz_ > G.nz - 1) return -2;
  return nx_ * nyz + ny_ * G.nz + nz_;
}

// the packet's deviate stream: draw n is half n & 1 of block n >> 1
// (PacketRng::next).  One model's key and step are the kernel's arguments.
template <int BATCH>
struct DrawStream {
  uint64_t pid;
  uint32_t n, key, step;
  __device__ __forceinline__ PhiloxOut block(const StepArgs& A, uint32_t ctr) const
  {
    return philox4x32_10(ctr, (uint32_t)pid, (uint32_t)(pid >> 32), BATCH ? step : A.step, BATCH ? key : A.seed, 0u);
  }
};

template <int GRID, int BATCH, int THREADS, int MINB>
__global__ void __launch_bounds__(THREADS, MINB) propagate_fp64_kernel(const StepArgs A, const GridDev G)
{
  extern __shared__ double s_tal[];  // [5][nz] when A.smem_zones
  __shared__ unsigned long long s_cnt[6];
  __shared__ double s_acc[5][THREADS];  // e_abs, fx, fy, fz, fr of the zone visit
  __shared__ unsigned long long s_pid[THREADS];
  __shared__ uint32_t s_k0[THREADS];
  __shared__ int s_m[BATCH ? THREADS : 1];
  __shared__ long long s_qn[BATCH ? THREADS : 1], s_qe[BATCH ? THREADS : 1];
  const int tid = threadIdx.x;
  if (tid < 6) s_cnt[tid] = 0;
  const int nz = G.nzones;
  const int nn = A.nu.n;
  const int nj = A.store_Jnu ? nn : 1;
  double* __restrict__ J = tally_J(A, G.nzones, nj);
  if (A.smem_zones)
    for (int i = tid; i < 5 * nz; i += THREADS) s_tal[i] = 0.0;
#pragma unroll
  for (int k = 0; k < 5; ++k) s_acc[k][tid] = 0.0;
  if constexpr (BATCH) { s_qn[tid] = 0; s_qe[tid] = 0; }
  __syncthreads();
  const int64_t rep_off = (!A.smem_zones && A.n_rep > 0) ? (int64_t)(blockIdx.x % A.n_rep) * 5 * nz : -1;
  const double2* __restrict__ opac = reinterpret_cast<const double2*>(A.opac);
  const int32_t limit = A.max_segments > 0 ? A.max_segments : 10000000;
  uint32_t step = A.step;
  if constexpr (BATCH) step = *A.step_dev;
  Pkt p;
  p.dvds = 0;
  DrawStream<BATCH> rng;
  Flow fl{};
  int fate = ABSORBED;  // no packet yet
  bool have = false, live = (tid & 31) < A.lanes;
  int32_t seg = 0, n_scat = 0;
  int acc = -1;  // zone of the visit summed in s_acc
  auto flush = [&](int z) {
    mixed::add_visit(A, s_tal, nz, rep_off, z, s_acc[0][tid], s_acc[1][tid], s_acc[2][tid], s_acc[3][tid],
                     s_acc[4][tid]);
#pragma unroll
    for (int k = 0; k < 5; ++k) s_acc[k][tid] = 0.0;
  };
  for (;;) {
    // the lanes of the warp meet every iteration (propagate_mixed_kernel)
    __syncwarp();
    if (!__any_sync(0xffffffffu, live)) break;
    if (!live) continue;
    if (fate != MOVING) {
      if (have) {
        if (acc >= 0) { flush(acc); acc = -1; }
        atomicAdd(s_cnt + 3, (unsigned long long)seg);
        atomicAdd(s_cnt + 4, (unsigned long long)n_scat);
        if (fate == ESCAPED) {
          const double t_obs = p.t - (p.x[0] * p.D[0] + p.x[1] * p.D[1] + p.x[2] * p.D[2]) / C_LIGHT;
          if constexpr (BATCH) {
            const int m = s_m[tid];
            const int64_t so = A.models[m].spec_off;
            spectrum_count(A, A.flux + so, A.click + so, t_obs, p.nu, p.e, p.D);
            atomicAdd(A.model_escaped + m, 1ULL);
          } else {
            spectrum_count(A, A.flux, A.click, t_obs, p.nu, p.e, p.D);
          }
          p.t = t_obs;
          atomicAdd(s_cnt + 0, 1ULL);
        } else if (fate == ABSORBED) {
          atomicAdd(s_cnt + 1, 1ULL);
        } else {
          atomicAdd(s_cnt + 2, 1ULL);
        }
        if (A.rec_fate) {
          const unsigned long long pid = s_pid[tid];
          A.rec_fate[pid] = fate;
          A.rec_ind[pid] = p.ind;
          A.rec_draws[pid] = (int32_t)(rng.n - s_k0[tid]);
          if (A.rec_type) A.rec_type[pid] = TYPE_PHOTON;
          double* s = A.rec_state + pid * 9;
          s[0] = p.x[0]; s[1] = p.x[1]; s[2] = p.x[2];
          s[3] = p.D[0]; s[4] = p.D[1]; s[5] = p.D[2];
          s[6] = p.t; s[7] = p.e; s[8] = p.nu;
        }
        have = false;
      }
      PacketRng er;  // emission draws one by one
      if constexpr (BATCH) {
        long long q_next = s_qn[tid], q_end = s_qe[tid];
        if (q_next >= q_end) {
          q_next = (long long)atomicAdd(A.counters + C_QUEUE, (unsigned long long)A.queue_chunk);
          q_end = q_next + A.queue_chunk;
          if (q_end > A.n_packets) q_end = A.n_packets;
          s_qe[tid] = q_end;
        }
        if (q_next >= A.n_packets) { live = false; continue; }
        s_qn[tid] = q_next + 1;
        s_pid[tid] = (unsigned long long)q_next;
        const int m = find_model(A.models, A.n_models, (int64_t)q_next);
        s_m[tid] = m;
        const BatchModel& M = A.models[m];
        er.init(M.seed, (uint64_t)(M.first_pid + ((int64_t)q_next - M.pkt_off)), step, 0);
        BatchZoneOf zf;
        zf.slice = G.r_out;
        zf.slice.n = M.n_zones;
        zf.slice.min = M.r_min;
        zf.slice.right = G.r_out.right + M.zone_off;
        zf.zone_off = M.zone_off;
        DrawNext d{er};
        emit_core<GRID>(A, G, p, d, M.core_radius, M.Ep, M.core_cdf, zf);
        s_k0[tid] = M.emit_draws;
      } else {
        const unsigned long long pid = atomicAdd(A.counters + C_QUEUE, 1ULL);
        if (pid >= (unsigned long long)A.n_packets) { live = false; continue; }
        s_pid[tid] = pid;
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
          er.init(A.seed, (uint64_t)(A.radio_first_pid + k), step, qn);
          s_k0[tid] = 0;  // a radioactive packet records every deviate of its stream
        } else {
          er.init(A.seed, (uint64_t)A.first_pid + pid, step, 0);
          DrawNext d{er};
          emit_core<GRID>(A, G, p, d, A.core_radius, A.Ep, A.core_cdf, GridZoneOf<GRID>{G});
          s_k0[tid] = er.n;
        }
      }
      rng.pid = er.pid;
      rng.n = er.n;
      rng.key = er.seed;
      rng.step = step;
      fate = MOVING;
      if (p.ind == -1) fate = ABSORBED;
      else if (p.ind == -2) fate = ESCAPED;
      seg = 0;
      n_scat = 0;
      have = true;
      if (fate != MOVING) continue;
      fl = flow_at(A, p.x);
    }
    // ------------------------------------------------------------- segment
    if (seg >= limit) { fate = STOPPED; atomicAdd(s_cnt + 5, 1ULL); continue; }
    ++seg;
    const int iz = p.ind;
    if (iz != acc) {
      if (acc >= 0) flush(acc);
      acc = iz;
    }
    // the depth's deviate; the other half of its block may be the next draw
    const uint32_t c0 = rng.n >> 1;
    const bool odd = rng.n & 1u;
    const PhiloxOut o0 = rng.block(A, c0);
    const double u_tau = odd ? u01(o0.w[2], o0.w[3]) : u01(o0.w[0], o0.w[1]);
    const double xdotD = (p.D[0] * p.x[0] + p.D[1] * p.x[1] + p.D[2] * p.x[2]);
    double d_bn;
    int new_ind;
    if constexpr (GRID == 1) {
      new_ind = next_cell_rn(G, p.x, p.D, iz, &d_bn);
    } else if constexpr (BATCH) {
      const int4 nb = __ldg(A.zone_nbr + iz);
      new_ind = next_zone_rn(__ldg(G.r_out.right + iz), __ldg(A.zone_rin + iz), nb.x, nb.y, nb.z != 0, fl.rsq, xdotD,
                             &d_bn);
    } else {
      double r_in = (iz != 0) ? __ldg(G.r_out.right + iz - 1) : G.r_out.min;
      int ind_in = (iz != 0) ? iz - 1 : -1;
      if (A.core_radius >= r_in) { r_in = A.core_radius; ind_in = -1; }
      new_ind = next_zone_rn(__ldg(G.r_out.right + iz), r_in, ind_in, (iz + 1 == nz) ? -2 : iz + 1,
                             (iz == 0) && (r_in == 0), fl.rsq, xdotD, &d_bn);
    }
    const double vdd = fl.v[0] * p.D[0] + fl.v[1] * p.D[1] + fl.v[2] * p.D[2];
    const double dshift = fl.gamma * (1 - div_c(vdd));
    // transport::get_opacity (transport_opacity.cpp:268-299)
    const int i_nu = loc_within_mixed(A.nu, p.nu * dshift);
    const double2 ab = __ldg(opac + (size_t)iz * nn + i_nu);
    const double a_opac = ab.x;
    const double s_opac = A.omit_scat ? 0.0 : ab.y;
    const double op = a_opac + s_opac;
    const double2 lr = __ldg(A.nu_lr + i_nu);
    double d_nu = div_by(div_rn(lr.y - lr.x, p.nu) * C_LIGHT, A.inv_t, A.inv_dvds, A.inv_dvds_lo);
    if (d_nu < 0) d_nu = -1 * d_nu;
    if (d_nu < d_bn) { d_bn = d_nu; new_ind = iz; }
    const double tot_lab = op * dshift;
    const double tau_r = -1.0 * log(1 - u_tau);
    const double d_sc = flight(tau_r, tot_lab);
    double d_tm = (A.tstop - p.t) * C_LIGHT;
    if (A.steady) d_tm = INFINITY;
    int event;
    double this_d;
    if ((d_sc < d_bn) && (d_sc < d_tm)) { event = 0; this_d = d_sc; }
    else if (d_bn < d_tm) { event = 1; this_d = d_bn; }
    else { event = 2; this_d = d_tm; }
    // tallies (transport.cpp:361-392)
    const double this_E = p.e * this_d;
    const double eps_imc = __ldg(A.eps_imc + iz);
    const double ed = this_E * dshift;
    atomicAdd(J + (size_t)iz * nj + (A.store_Jnu ? i_nu : 0), this_E);
    s_acc[0][tid] += ed * a_opac * dshift * eps_imc;
    if (A.tally_forces) {
      const double w = ed * op * dshift;
      s_acc[1][tid] += w * p.D[0];
      s_acc[2][tid] += w * p.D[1];
      s_acc[3][tid] += w * p.D[2];
      s_acc[4][tid] += w * xdotD * rsqrt_nr(fl.rsq);
    }
    // move
    p.x[0] += this_d * p.D[0];
    p.x[1] += this_d * p.D[1];
    p.x[2] += this_d * p.D[2];
    p.t = p.t + div_c(this_d);
    fl = flow_at(A, p.x);
    ++rng.n;
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
      // transport::do_scatter (scatter.cpp:12-70): draws n .. n + 6 from the
      // depth's block and the three after it
      ++n_scat;
      const double eps = absorbed_part_rn(a_opac, op);
      const PhiloxOut o1 = rng.block(A, c0 + 1), o2 = rng.block(A, c0 + 2);
      const double z1 = odd ? u01(o1.w[0], o1.w[1]) : u01(o0.w[2], o0.w[3]);
      ++rng.n;
      bool redist = false, absorb = !(z1 > eps);
      if (absorb) {
        const double z2 = odd ? u01(o1.w[2], o1.w[3]) : u01(o1.w[0], o1.w[1]);
        ++rng.n;
        if ((z2 > eps_imc) || A.radiative_eq) redist = true;
        else fate = ABSORBED;
      }
      if (fate == MOVING) {
        // transport::isotropic_scatter (scatter.cpp:303-351)
        const int j = (odd ? 1 : 0) + (absorb ? 1 : 0);
        const uint32_t m0 = (j == 0) ? o1.w[0] : (j == 1) ? o1.w[2] : o2.w[0];
        const uint32_t m1 = (j == 0) ? o1.w[1] : (j == 1) ? o1.w[3] : o2.w[1];
        const uint32_t f0 = (j == 0) ? o1.w[2] : (j == 1) ? o2.w[0] : o2.w[2];
        const uint32_t f1 = (j == 0) ? o1.w[3] : (j == 1) ? o2.w[1] : o2.w[3];
        rng.n += 2;
        // the emissivity CDF's guide entries are on their way while the
        // direction is formed; the row is searched between them at the end
        int lo = 0, hi = 0;
        double u_cdf = 0, pos = 0;
        if (redist) {
          const PhiloxOut o3 = rng.block(A, c0 + 3);
          u_cdf = odd ? u01(o3.w[0], o3.w[1]) : u01(o2.w[2], o2.w[3]);
          pos = odd ? u01(o3.w[2], o3.w[3]) : u01(o3.w[0], o3.w[1]);
          rng.n += 2;
          if (A.cdf_guide && nn > 1) {
            const uint16_t* g = A.cdf_guide + (size_t)p.ind * (A.guide_n + 1) + (int)(u_cdf * (double)A.guide_n);
            lo = __ldg(g);
            hi = __ldg(g + 1);
          }
        }
        const double vdotD = fl.v[0] * p.D[0] + fl.v[1] * p.D[1] + fl.v[2] * p.D[2];
        const double dshift_in = fl.gamma * (1 - div_c(vdotD));
        p.e = p.e * dshift_in;
        p.nu = p.nu * dshift_in;
        const double mu = 1 - 2.0 * u01(m0, m1);
        const double phi = 2.0 * PI * u01(f0, f1);
        const double smu = sqrt_rn(1 - mu * mu);
        double sn, cs;
        sincos(phi, &sn, &cs);
        const double Dn[3] = {smu * cs, smu * sn, mu};
        const double V[3] = {-fl.v[0], -fl.v[1], -fl.v[2]};
        const double vdp = (Dn[0] * V[0] + Dn[1] * V[1] + Dn[2] * V[2]);
        const double vd_out = fl.gamma * (1 - div_c(vdp));
        const double f = (1 - div_rn(div_c(fl.gamma * vdp), fl.gamma + 1));
        const double inv_vd = rcp_rn(vd_out);
#pragma unroll
        for (int k = 0; k < 3; ++k) p.D[k] = inv_vd * (Dn[k] - div_c(fl.gamma * V[k]) * f);
        const double norm = sqrt_rn(p.D[0] * p.D[0] + p.D[1] * p.D[1] + p.D[2] * p.D[2]);
        const double inv_norm = rcp_rn(norm);
#pragma unroll
        for (int k = 0; k < 3; ++k) p.D[k] = div_rn(p.D[k], norm, inv_norm);
        p.e = p.e * vd_out;
        if (redist) {  // transport::sample_photon_frequency (emission.cpp:27-46), locate_array::sample
          if (nn == 1) p.nu = 0;
          else {
            if (A.cdf_guide) {
              const double* row = reinterpret_cast<const double*>(A.cdf) + (size_t)p.ind * nn;
              while (lo < hi) {
                const int m = (lo + hi) >> 1;
                if (__ldg(row + m) <= u_cdf) lo = m + 1; else hi = m;
              }
              lo = min(lo, nn - 1);
            } else {
              lo = cdf_row_sample<double>(A, p.ind, u_cdf);
            }
            const double2 lr = __ldg(A.nu_lr + lo);
            p.nu = lr.x + (lr.y - lr.x) * pos;
          }
        }
        p.nu = p.nu * vd_out;
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
  if (A.smem_zones) {
    double* g[5] = {A.e_abs, A.fx, A.fy, A.fz, A.fr};
    for (int i = tid; i < 5 * nz; i += THREADS) {
      const double v = s_tal[i];
      if (v != 0.0 || isnan(v)) atomicAdd(g[i / nz] + (i % nz), v);
    }
  }
}
