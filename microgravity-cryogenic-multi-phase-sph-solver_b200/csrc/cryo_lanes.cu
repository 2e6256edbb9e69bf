// cryo_lanes.cu -- the neighbour passes of the rate evaluation for small tanks
// (exact arithmetic): PASS_LANES lanes share a particle.
//
// A thread that walks its particle's ~75 neighbours (cryo_physics.cu) is one
// chain of dependent loads and additions, 20 to 160 us long whatever the
// tank's size; a tank of some ten thousand particles leaves most of the chip
// idle meanwhile.  Here a round takes PASS_LANES neighbours side by side
// (NbrRounds), one per lane, and every sum then takes the lanes' terms one
// after another in lane order.  That is the order of the list, so each sum
// sees the additions of the one-thread pass and has its bits: a neighbour
// without a term adds a zero, which leaves a sum as it is (a sum starts at +0
// and can only return to zero as +0, so it is never -0).
//
// The fast arithmetic has no passes here: its sums are contracted with the
// products they add, term by term, in the one-thread order.
#include "cryo_kernels.cuh"

namespace cryo {
namespace lanes {

constexpr unsigned kAll = 0xffffffffu;
constexpr int L = PASS_LANES;

// compute_density_summation (SPH_kernels.cu:6-34) and the equation of state
// (navier_stokes.cu:5-14), as exact::k_density with fuse_eos.
__global__ void __launch_bounds__(kBlock) k_density(Params P, View V) {
  {
    const Range wr = wall_range(P, V);
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < wr.count; t += gridDim.x * blockDim.x) {
      const int i = particle_at(wr, t);
      reinterpret_cast<float*>(V.mrps + i)[3] = 1.0f / P.vol0;
      V.rmin[i] = P.support;
    }
  }
  const Range fr = fluid_range(P, V);
  const int sub = threadIdx.x % L;
  const int step = gridDim.x * (kBlock / L);
  for (int t0 = blockIdx.x * (kBlock / L) + (threadIdx.x & ~31) / L; t0 < fr.count; t0 += step) {
    const int t = t0 + (threadIdx.x & 31) / L;
    const bool live = t < fr.count;
    const int i = particle_at(fr, live ? t : t0);
    const float4 xpi = V.xp[i];
    const int ph = ph_of(xpi);
    const V3 xi = xyz(xpi);
    NbrRounds<L> nbrs(P, V, i, xi, sub, live);
    float s[1] = {0.0f}, r2min = P.support2;
    while (__any_sync(kAll, nbrs.more())) {
      float4 xj;
      const int j = nbrs.take(xj);
      float w[1] = {0.0f};
      if (j >= 0) {
        const float r2 = norm2(xi - xyz(xj));
        w[0] = kernel_W(P, sqrtf(r2));
        if (j != i && r2 < r2min) r2min = r2;
      }
      add_terms<L>(s, w);
    }
#pragma unroll
    for (int o = L / 2; o > 0; o >>= 1) {
      const float other = __shfl_xor_sync(kAll, r2min, o);
      if (other < r2min) r2min = other;
    }
    if (sub != 0 || !live) continue;
    const float sum = s[0];
    float* mr = reinterpret_cast<float*>(V.mrps + i);
    mr[3] = sum;
    V.rmin[i] = sqrtf(r2min);
    float rho = mr[1];
    if (P.density_mode == CRYO_DENSITY_SUMMATION) {
      rho = (ph == kLiquid ? V.vt[i].w : mr[0]) * sum;
      mr[1] = rho;
    }
    const float Ti = V.vT[i].w;
    mr[2] = eos_pressure(P, ph, rho, Ti);
    V.aux[i] = make_float4(mr[0] / rho, 1.0f / sum, sound_speed(P, ph, Ti), 0.0f);
  }
}

// compute_wall_boundary (navier_stokes.cu:16-69), as exact::k_wall.
__global__ void __launch_bounds__(kBlock) k_wall(Params P, View V) {
  const DynState* dyn = V.dyn;
  const Range rg = wall_range(P, V);
  const V3 g = v3(dyn->fr.gravity[0], dyn->fr.gravity[1], dyn->fr.gravity[2]);
  const int sub = threadIdx.x % L;
  const int step = gridDim.x * (kBlock / L);
  for (int t0 = blockIdx.x * (kBlock / L) + (threadIdx.x & ~31) / L; t0 < rg.count; t0 += step) {
    const int t = t0 + (threadIdx.x & 31) / L;
    const bool live = t < rg.count;
    const int i = particle_at(rg, live ? t : t0);
    const float4 xpi = V.xp[i];
    const V3 xi = xyz(xpi);
    NbrRounds<L> nbrs(P, V, i, xi, sub, live);
    // w, p w, g.r rho w per phase; rho w, v w
    float liq[3] = {0, 0, 0}, vap[3] = {0, 0, 0}, both[4] = {0, 0, 0, 0};
    while (__any_sync(kAll, nbrs.more())) {
      float4 xj;
      const int j = nbrs.take(xj);
      float tl[3] = {0, 0, 0}, tv[3] = {0, 0, 0}, tb[4] = {0, 0, 0, 0};
      const int phj = j >= 0 ? ph_of(xj) : kDead;
      if (is_fluid(phj)) {
        const V3 rwf = xi - xyz(xj);
        const float w = kernel_W(P, sqrtf(norm2(rwf)));
        const float4 mr = __ldg(V.mrps + j);
        const float t3[3] = {w, mr.z * w, dot(g, rwf) * mr.y * w};
        const bool v = phj == kVapor;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          tl[k] = v ? 0.0f : t3[k];
          tv[k] = v ? t3[k] : 0.0f;
        }
        const V3 vw = xyz(__ldg(V.vT + j)) * w;
        tb[0] = mr.y * w;
        tb[1] = vw.x;
        tb[2] = vw.y;
        tb[3] = vw.z;
      }
      add_terms<L>(liq, tl);
      if (__any_sync(kAll, phj == kVapor)) add_terms<L>(vap, tv);
      add_terms<L>(both, tb);
    }
    if (sub != 0 || !live) continue;
    const float sw[2] = {liq[0], vap[0]}, sp[2] = {liq[1], vap[1]}, sgr[2] = {liq[2], vap[2]};
    float pw[2];
    for (int k = 0; k < 2; ++k) {
      pw[k] = sw[k] > 0.0f ? (sp[k] + sgr[k]) / sw[k] : P.p_bg;
      if (P.clamp_neg && pw[k] < 0.0f) pw[k] = 0.0f;
    }
    if (!(sw[0] > 0.0f) && sw[1] > 0.0f) pw[0] = pw[1];
    if (!(sw[1] > 0.0f) && sw[0] > 0.0f) pw[1] = pw[0];
    float* mr = reinterpret_cast<float*>(V.mrps + i);
    mr[2] = pw[0];
    V.nrm[i].w = (sw[0] + sw[1]) > 0.0f ? sw[0] / (sw[0] + sw[1]) : 0.0f;
    const float swt = sw[0] + sw[1];
    V3 vw;
    if (swt > 0.0f) {
      mr[1] = both[0] / swt;
      vw = V3{both[1], both[2], both[3]} * (-1.0f / swt);
    } else {
      mr[1] = P.rho0[0];
      vw = V3{0, 0, 0};
    }
    V.vwp[i] = f4(vw, pw[1]);
    V.a4[i] = make_float4(0.0f, 0.0f, 0.0f, V.a4[i].w);
  }
}

// compute_interface_fields (surface_tension.cu:5-85), as exact::k_interface.
template <int TAPE>
__global__ void __launch_bounds__(INTERFACE_BLOCK) k_interface(Params P, View V, int sorted) {
  const Range rg = fluid_range(P, V);
  const bool write_ns = P.csf_active && !P.csf_smooth;
  const int sub = threadIdx.x % L;
  const int step = gridDim.x * (INTERFACE_BLOCK / L);
  for (int t0 = blockIdx.x * (INTERFACE_BLOCK / L) + (threadIdx.x & ~31) / L; t0 < rg.count; t0 += step) {
    const int t = t0 + (threadIdx.x & 31) / L;
    const bool live = t < rg.count;
    const int i = particle_at(rg, live ? t : t0);
    const float4 xpi = V.xp[i];
    const int ph = ph_of(xpi);
    const V3 xi = xyz(xpi);
    const float ci = ph == kLiquid ? 1.0f : 0.0f;
    // as in exact::k_interface: only walls count in a tank without vapour
    const bool walls_only = !TAPE && !P.has_vapor && P.st_model != CRYO_ST_AKINCI;
    // (and a particle with no wall and none of the other phase around it has only zeros to add)
    const bool alone = !TAPE && sorted && P.st_model != CRYO_ST_AKINCI &&
                       !(V.near_kinds[i] & (kNearWall | (ph == kVapor ? kNearLiquid : kNearVapor)));
    NbrRounds<L> nbrs(P, V, i, xi, sub, live && !alone);
    // the sums a round has no term for are left alone
    float sv[2] = {0, 0}, sw[8] = {0, 0, 0, 0, 0, 0, 0, 0}, sg[3] = {0, 0, 0}, sk[3] = {0, 0, 0};
    while (__any_sync(kAll, nbrs.more())) {
      float4 xj;
      const int j = nbrs.take(xj);
      const int phj = j >= 0 ? ph_of(xj) : kDead;
      float tv[2] = {0, 0}, tw[8] = {0, 0, 0, 0, 0, 0, 0, 0}, tg[3] = {0, 0, 0}, tk[3] = {0, 0, 0};
      bool coloured = false, cohesive = false;
      if (phj == kWall) {
        const V3 rij = xi - xyz(xj);
        const float r = sqrtf(norm2(rij));
        const float vw = P.vol0 * kernel_W(P, r);
        const float4 nj = __ldg(V.nrm + j);
        const V3 gw = kernel_gradW(P, rij, r);
        const V3 wn = xyz(nj) * vw, gp = gw * P.vol0;
        tw[0] = vw;
        tw[1] = (fl_of(xj) & kHeated) ? vw : 0.0f;
        tw[2] = wn.x; tw[3] = wn.y; tw[4] = wn.z;
        tw[5] = gp.x; tw[6] = gp.y; tw[7] = gp.z;
        if (P.wall_colour) {
          const V3 gc = gw * (P.vol0 * (nj.w - ci));
          tg[0] = gc.x; tg[1] = gc.y; tg[2] = gc.z;
          coloured = true;
        }
      } else if (j >= 0 && !walls_only) {
        const V3 rij = xi - xyz(xj);
        const float r = sqrtf(norm2(rij));
        const float Vj = __ldg(V.aux + j).x;  // m_j / rho_j
        tv[0] = Vj * kernel_W(P, r);
        if (phj != ph) tv[1] = tv[0];
        if (j != i && (phj != ph || P.st_model == CRYO_ST_AKINCI)) {
          const V3 gw = kernel_gradW(P, rij, r);
          const float cj = phj == kLiquid ? 1.0f : 0.0f;
          const V3 gc = gw * (Vj * (cj - ci));
          tg[0] = gc.x; tg[1] = gc.y; tg[2] = gc.z;
          coloured = true;
          if (phj == kLiquid) {
            const V3 k = gw * Vj;
            tk[0] = k.x; tk[1] = k.y; tk[2] = k.z;
            cohesive = true;
          }
        }
      }
      if (__any_sync(kAll, phj == kWall)) add_terms<L>(sw, tw);
      if (!walls_only) add_terms<L>(sv, tv);
      if (__any_sync(kAll, coloured)) add_terms<L>(sg, tg);
      if (P.st_model == CRYO_ST_AKINCI && __any_sync(kAll, cohesive)) add_terms<L>(sk, tk);
    }
    if (sub != 0 || !live) continue;
    const float s_all = sv[0], s_other = sv[1], ww = sw[0], hw = sw[1];
    const V3 wall_n{sw[2], sw[3], sw[4]}, gradphi{sw[5], sw[6], sw[7]}, akn{sk[0], sk[1], sk[2]};
    V3 gradc{sg[0], sg[1], sg[2]};
    if (TAPE) {
      const int tn = V.tape_n;
      V.tape[3 * tn + i] = f4(gradc, s_all);
      V.tape[4 * tn + i] = f4(wall_n, s_other);
      V.tape[5 * tn + i] = make_float4(ww, 0.0f, 0.0f, 0.0f);
    }
    const float alpha = s_all > 0.0f ? s_other / s_all : 0.0f;
    V.wall_w[i] = ww;
    V.heat_w[i] = hw;
    if (P.st_model == CRYO_ST_AKINCI) {
      V.nrm[i] = f4(ph == kLiquid ? akn * (-P.h) : V3{0, 0, 0}, alpha);
    } else {
      const float gmag = norm(gradc);
      V3 vwi{0, 0, 0};
      if (P.wetting_model != 0 && ww > 0.0f && gmag > P.normal_eps && norm2(wall_n) > 0.0f) {
        const V3 nw = normalized(wall_n);
        const V3 nh = gradc / gmag;
        const V3 tan_in = nh - nw * dot(nh, nw);
        const float tm = norm(tan_in);
        if (tm > 1e-6f) {
          const float cos_d = -dot(nh, nw);
          const float delta_w = 2.0f * norm(gradphi);
          const float coeff = 2.0f * P.sigma / (P.rho0[0] + P.rho0[1]);
          vwi = tan_in * (-(P.cos_theta - cos_d) * coeff * gmag * delta_w / tm);
        }
      }
      V.vwp[i] = f4(vwi, V.vwp[i].w);
      if (P.wetting_model != 1 && ww > 0.0f && gmag > P.normal_eps) {
        const V3 nw = normalized(wall_n);
        const V3 nh = gradc / gmag;
        V3 t = nh - nw * dot(nh, nw);
        const float tmag = norm(t);
        if (norm2(nw) > 0.0f && tmag > 1e-6f) {
          t = t / tmag;
          const V3 target = nw * (-P.cos_theta) + t * P.sin_theta;
          const float beta = clampf(ww / P.wall_adhesion_weight, 0.0f, 1.0f);
          const V3 blended = normalized(nh * (1.0f - beta) + target * beta);
          gradc = blended * gmag;
        }
      }
      V.nrm[i] = f4(gradc, alpha);
      if (write_ns) {
        const float gm = norm(gradc);
        const V3 ns = gm > P.normal_eps ? gradc / gm : V3{0, 0, 0};
        V.ns4[i] = f4(ns, V.ns4[i].w);
      }
    }
  }
}
template __global__ void k_interface<0>(Params, View, int);
template __global__ void k_interface<1>(Params, View, int);

// The fused force pass of exact::k_forces_t (cryo_physics.cu: what it covers
// and why it may be fused).  The pairs' terms go through shared memory, one row
// per term and component, a column per lane, and are added in list order, each
// sum by one lane: lanes 0-2 the force, acceleration and wall force of one
// axis, lanes 3-5 the transport, surface-tension and wall-moment sums of one
// axis, lanes 6 and 7 the scalar sums.  So a lane holds four sums where a
// thread of the one-thread pass holds 25, and the eight additions per round are
// spread over the lanes.  Measured: 159 -> 58 us on the heated 26k-particle
// cylinder, 158 -> 36 us on a 4k-particle box, 124 -> 29 us on a 27k-particle
// dam break; at 97k fluid particles it is slower (249 against 199 us: a pair
// costs 1.75 times the instructions), hence FORCES_LANES_MAX.
enum {  // rows
  kRowP = 0, kRowC = 3, kRowA = 6, kRowX = 9, kRowF = 12, kRowA1 = 15, kRowA2 = 18, kRowS = 21, kRowT = 24,
  kRowG = 27, kRowK = 30, kRowDiv = 33, kRowDiff = 34, kRowNum = 35, kRowDen = 36, kRowQ = 37, kRowZero = 38,
  kForceRows = 39,
  kRowStride = 36  // 32 lanes and a pad: eight lanes reading eight rows use all banks
};

template <int WHAT>
__global__ void __launch_bounds__(FORCES_LANED_BLOCK, 4) k_forces_t(Params P, View V) {
  static_assert(L == 8, "the rows hold eight columns per particle");
  constexpr int what = WHAT;
  constexpr int kWarps = FORCES_LANED_BLOCK / 32;
  __shared__ __align__(16) float shared_rows[kWarps][kForceRows * kRowStride];
  DynState* dyn = V.dyn;
  const bool thermal = (what & FORCE_THERMAL) && dyn->thermal_on;
  const float dt = dyn->dt;
  const V3 origin = v3(dyn->fr.frame_origin[0], dyn->fr.frame_origin[1], dyn->fr.frame_origin[2]);
  const float h = P.h;
  const float eta2 = 0.01f * h * h;
  const float r_guard = 0.6f * P.dx;
  const bool tvf_stress = P.tvf && P.tvf_stress;
  const float inv_gamma = 1.0f / P.tait_gamma;
  const float csf_coeff = 2.0f * P.sigma / (P.rho0[0] + P.rho0[1]);
  const bool iso_walls = P.wall_bc == CRYO_WALL_ISOTHERMAL;
  const int own_lo = dyn->own_lo, own_hi = dyn->own_hi, n_sorted = dyn->n_sorted;
  float vmax_l = 0.0f, amax_l = 0.0f, tv_l = 0.0f, sr_l = 0.0f, nut_l = 0.0f;

  // walls: zero outputs
  {
    const Range wr = wall_range(P, V);
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < wr.count; t += gridDim.x * blockDim.x) {
      const int i = particle_at(wr, t);
      V.ab4[i] = make_float4(0.0f, 0.0f, 0.0f, (what & FORCE_DRHO) ? 0.0f : V.ab4[i].w);
      V.a4[i] = make_float4(0.0f, 0.0f, 0.0f, thermal ? 0.0f : V.a4[i].w);
      V.fw[i] = make_float4(0, 0, 0, 0);
      V.mw[i] = make_float4(0, 0, 0, 0);
    }
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int sub = lane % L, lead = lane - sub;
  float* const rows = shared_rows[warp];
  auto put_row = [&](int r, float v) { rows[r * kRowStride + lane] = v; };
  auto put_rows = [&](int r, V3 v) {
    put_row(r, v.x);
    put_row(r + 1, v.y);
    put_row(r + 2, v.z);
  };
  // the eight values of this lane's particle in row r
  auto get_row = [&](int r, float (&v)[8]) {
    const float4 a = *reinterpret_cast<const float4*>(rows + r * kRowStride + lead);
    const float4 b = *reinterpret_cast<const float4*>(rows + r * kRowStride + lead + 4);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
  };
  put_row(kRowZero, 0.0f);
  constexpr bool do_D = (what & FORCE_DRHO) != 0;
  const Range fr = fluid_range(P, V);
  constexpr int kPer = 32 / L;  // particles per warp
  for (int t0 = (blockIdx.x * kWarps + warp) * kPer; t0 < fr.count; t0 += gridDim.x * kWarps * kPer) {
    const int t = t0 + lane / L;
    const bool live = t < fr.count;
    const int i = particle_at(fr, live ? t : t0);
    const float4 xpi = V.xp[i];
    const int ph = ph_of(xpi);
    const int pi_idx = phase_index(ph);
    const V3 xi = xyz(xpi);
    NbrRounds<L> nbrs(P, V, i, xi, sub, live);
    const float4 vTi = V.vT[i];
    const V3 vi = xyz(vTi);
    const float Ti = vTi.w;
    const float4 mri = V.mrps[i];
    const float mi = mri.x, rhoi = mri.y, pi = mri.z, sigmai = mri.w;
    const float alpha_i_pc = V.nrm[i].w;
    const float4 vti4 = V.vt[i];
    const float Vi = mi / rhoi;
    const float Vi2 = Vi * Vi;
    const float ci = sound_speed(P, ph, Ti);
    const float etai = P.mu[pi_idx] + (P.sps ? rhoi * V.nu_t[i] : 0.0f);
    const float alpha_i = ph == kVapor ? P.alpha_av_vap : P.alpha_av;
    // harmonic viscosity per neighbour phase (navier_stokes.cu:190-196)
    float eta_pair0 = 0.0f, eta_pair1 = 0.0f;
    if (!P.sps) {
      auto harmonic = [&](float etaj) {
        const float eta_sum = etai + etaj;
        return eta_sum > 0.0f ? 2.0f * etai * etaj / eta_sum : 0.0f;
      };
      eta_pair0 = harmonic(P.mu[0] + 0.0f);
      eta_pair1 = harmonic(P.mu[1] + 0.0f);
    }
    // transport (SPH_kernels.cu:61-74)
    const bool do_T = live && P.tvf && !(sigmai < P.tvf_sigma_min) && !(P.tvf_interface_only && !(alpha_i_pc > 0.0f));
    const bool any_T = __any_sync(kAll, do_T);
    const float VT_i = 1.0f / sigmai;
    const float VT_i2 = VT_i * VT_i;
    const V3 dvi = xyz(vti4) - vi;
    // CSF (surface_tension.cu:131-136)
    V3 ni{0, 0, 0};
    bool do_C = false;
    if (what & FORCE_CSF) {
      ni = xyz(V.ns4[i]);
      do_C = norm2(ni) > 0.25f;
    }
    const bool any_C = __any_sync(kAll, live && do_C);
    const float ciC = ph == kLiquid ? 1.0f : 0.0f;
    // Akinci
    const bool do_A = (what & FORCE_AKINCI) && ph == kLiquid;
    const float akc = P.support;
    const float psi = P.rho0[0] * P.vol0;
    // density rate
    const V3 veli = P.tvf ? xyz(vti4) : vi;
    // thermal: the harmonic conductivity per neighbour phase (phase_change.cu:57-61)
    const float ki = P.k[pi_idx];
    const float k_pair0 = 4.0f * ki * P.k[0] / (ki + P.k[0]);
    const float k_pair1 = 4.0f * ki * P.k[1] / (ki + P.k[1]);

    float s0 = 0.0f, s1 = 0.0f, s2 = 0.0f, s3 = 0.0f;  // the sums this lane keeps
    while (__any_sync(kAll, nbrs.more())) {
      float4 xj;
      const int j = nbrs.take(xj);
      const bool wall = j >= 0 && ph_of(xj) == kWall;  // i is fluid, so j != i
      const unsigned walls = __ballot_sync(kAll, wall);
      bool guard = false, warm = false;
      const V3 zero{0, 0, 0};  // a pair without a term adds a zero
      put_rows(kRowP, zero);
      put_rows(kRowC, zero);
      put_rows(kRowA, zero);
      if (tvf_stress) put_rows(kRowS, zero);
      if (walls) {
        put_rows(kRowA1, zero);
        put_rows(kRowA2, zero);
      }
      if (any_T) put_rows(kRowT, zero);
      if (any_C) {
        put_row(kRowNum, 0.0f);
        put_row(kRowDen, 0.0f);
        if (P.csf_balanced) put_rows(kRowG, zero);
      }
      if (what & FORCE_AKINCI) put_rows(kRowK, zero);
      if (do_D) {
        put_row(kRowDiv, 0.0f);
        put_row(kRowDiff, 0.0f);
      }
      if (thermal) put_row(kRowQ, 0.0f);
      if (j >= 0 && j != i) {
        const V3 rij = xi - xyz(xj);
        const float r2 = norm2(rij);
        const float r = sqrtf(r2);
        const float dW = kernel_dWdr(P, r);
        const bool separated = r > 1e-12f * h;
        const V3 gw = separated ? rij * (dW / r) : V3{0, 0, 0};  // == kernel_gradW
        if (wall) {
          const float4 mrj = __ldg(V.mrps + j);
          const float4 vwj = __ldg(V.vwp + j);
          if (do_T) {
            float rho_w;
            if (ph == kVapor) {
              rho_w = (vwj.w - (P.p_bg - P.vapor_K)) / (P.gas_R * Ti);
            } else {
              const float ratio = (mrj.z - P.p_bg) / P.tait_B + 1.0f;
              rho_w = P.rho0[0] * powf(ratio > 0.5f ? ratio : 0.5f, inv_gamma);
            }
            const float Vj = rho_w > 0.0f ? VT_i * rhoi / rho_w : VT_i;
            put_rows(kRowT, gw * (VT_i2 + Vj * Vj));
          }
          const float Vj = P.vol0;
          const float vsum = Vi2 + Vj * Vj;
          const float pw = ph == kVapor ? vwj.w : mrj.z;
          put_rows(kRowP, -(gw * (vsum * 0.5f * (pi + pw))));
          if (tvf_stress) put_rows(kRowS, vi * (0.5f * vsum * rhoi * dot(dvi, gw)));
          if (r < r_guard && separated) {
            guard = true;
            const float qg = 1.0f - r / r_guard;
            const V3 nn = rij / r;
            put_rows(kRowA1, nn * (4.0f * ci * ci * qg * qg / r_guard));
            const float vn = dot(vi, nn);
            if (vn < 0.0f && dt > 0.0f) put_rows(kRowA2, -(nn * (qg * vn / dt)));
          }
          if (P.no_slip) {
            const V3 vij = vi - xyz(vwj);
            if (separated) put_rows(kRowC, vij * (vsum * etai * dW / r));
            const float vr = dot(vij, rij);
            if (alpha_i > 0.0f && vr < 0.0f) {
              const float mu_ij = h * vr / (r2 + eta2);
              const float Pi = -alpha_i * ci * mu_ij / rhoi;
              put_rows(kRowA, -(gw * (rhoi * P.vol0 * Pi)));
            }
          }
          put_rows(kRowX, xyz(xj) - origin);
          if (do_A && r2 > 0.0f) put_rows(kRowK, -((rij / r) * (P.akinci_beta * psi * akinci_adhesion(r, akc))));
          if (do_D) put_row(kRowDiv, P.vol0 * dot(veli, gw));
          if (thermal && iso_walls) {
            const float Tw = __ldg(V.vT + j).w;
            if (Ti != Tw) {  // equal temperatures: a zero term
              const float kij = 2.0f * ki;
              const float rgw = r * dW;
              put_row(kRowQ, Vi * P.vol0 * kij * (Ti - Tw) * rgw / (r2 + eta2));
              warm = true;
            }
          }
        } else {
          const int phj = ph_of(xj);
          const float4 mrj = __ldg(V.mrps + j);
          const float4 vTj = __ldg(V.vT + j);
          const float4 axj = __ldg(V.aux + j);  // {m_j / rho_j, 1 / sigma_j, c_j}
          const float mj = mrj.x, rhoj = mrj.y;
          if (do_T) {
            const float Vj = axj.y;
            put_rows(kRowT, gw * (VT_i2 + Vj * Vj));
          }
          const float Vj = axj.x;
          const float vsum = Vi2 + Vj * Vj;
          const float pt = (rhoj * pi + rhoi * mrj.z) / (rhoi + rhoj);
          put_rows(kRowP, -(gw * (vsum * pt)));
          if (tvf_stress) {
            const V3 vj = xyz(vTj);
            const V3 Ag = vi * (rhoi * dot(dvi, gw)) + vj * (rhoj * dot(xyz(__ldg(V.vt + j)) - vj, gw));
            put_rows(kRowS, Ag * (0.5f * vsum));
          }
          const V3 vij = vi - xyz(vTj);
          if (P.sps) {
            const float etaj = P.mu[phase_index(phj)] + rhoj * V.nu_t[j];
            const float eta_sum = etai + etaj;
            if (eta_sum > 0.0f && separated) {
              const float eta_ij = 2.0f * etai * etaj / eta_sum;
              put_rows(kRowC, vij * (vsum * eta_ij * dW / r));
            }
          } else {
            const float eta_ij = phj == kVapor ? eta_pair1 : eta_pair0;
            if (eta_ij != 0.0f && separated) put_rows(kRowC, vij * (vsum * eta_ij * dW / r));
          }
          if (alpha_i > 0.0f && phj == ph) {
            const float vr = dot(vij, rij);
            if (vr < 0.0f) {
              const float cj = axj.z;
              const float mu_ij = h * vr / (r2 + eta2);
              const float Pi = -alpha_i * 0.5f * (ci + cj) * mu_ij / (0.5f * (rhoi + rhoj));
              put_rows(kRowA, -(gw * (mj * Pi)));
            }
          }
          if (do_C) {
            const V3 gwC = separated ? gw : rij * (dW / r);  // the same product where gw is not zeroed
            const V3 nj = xyz(__ldg(V.ns4 + j));
            if (norm2(nj) > 0.25f) {
              put_row(kRowNum, Vj * dot(ni - nj, gwC));
              put_row(kRowDen, Vj * r * (-dW));
            }
            if (P.csf_balanced) {
              const float cj = phj == kLiquid ? 1.0f : 0.0f;
              put_rows(kRowG, gwC * ((Vi * Vi + Vj * Vj) * (rhoj * ciC + rhoi * cj) / (rhoi + rhoj)));
            }
          }
          if (do_A && phj == kLiquid && r2 > 0.0f) {
            const V3 rhat = rij / r;
            const float K = 2.0f * P.rho0[0] / (rhoi + rhoj);
            const V3 f_coh = rhat * (-P.akinci_gamma * mi * mj * akinci_cohesion(r, akc));
            const V3 f_curv = (xyz(V.nrm[i]) - xyz(__ldg(V.nrm + j))) * (-P.akinci_gamma * mi);
            put_rows(kRowK, (f_coh + f_curv) * (K / mi));
          }
          if (do_D) {
            const V3 velj = P.tvf ? xyz(__ldg(V.vt + j)) : xyz(vTj);
            put_row(kRowDiv, Vj * dot(veli - velj, gw));
            if (phj == ph) put_row(kRowDiff, Vj * 2.0f * (rhoj - rhoi) * dot(-rij, gw) / (r2 + eta2));
          }
          // equal temperatures give a zero term that leaves q as it is
          if (thermal && Ti != vTj.w) {
            const float kij = phj == kVapor ? k_pair1 : k_pair0;
            const float rgw = r * dW;
            put_row(kRowQ, Vi * Vj * kij * (Ti - vTj.w) * rgw / (r2 + eta2));
            warm = true;
          }
        }
      }
      // every sum takes its eight terms in order
      const bool any_guard = walls && __any_sync(kAll, guard);
      const bool any_q = thermal && __any_sync(kAll, warm);
      __syncwarp();
      const int ax = sub < 3 ? sub : sub - 3;  // the axis of lanes 0-5
      const int r0 = sub < 3   ? kRowP + ax
                     : sub < 6 ? (any_T ? kRowT + ax : kRowZero)
                     : do_D    ? (sub == 6 ? kRowDiv : kRowDiff)
                               : kRowZero;
      const int r1 = sub < 3   ? kRowA + ax
                     : !any_C  ? kRowZero
                     : sub < 6 ? (P.csf_balanced ? kRowG + ax : kRowZero)
                               : (sub == 6 ? kRowNum : kRowDen);
      float p8[8], c8[8], a8[8], st8[8];
      get_row(r0, p8);
      get_row(sub < 3 ? kRowC + ax : kRowZero, c8);
      get_row(r1, a8);
      if (tvf_stress) get_row(sub < 3 ? kRowS + ax : kRowZero, st8);
      if (!walls) {
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          s0 += p8[u];
          if (tvf_stress) s0 += st8[u];
          s0 += c8[u];
          s1 += a8[u];
        }
      } else {
        float g1[8], g2[8];
        get_row(sub < 3 && any_guard ? kRowA1 + ax : kRowZero, g1);
        get_row(sub < 3 && any_guard ? kRowA2 + ax : kRowZero, g2);
        const unsigned mine = (walls >> lead) & 0xffu;
        float d8[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const float f_before = s0, a_before = s1;
          s0 += p8[u];
          if (tvf_stress) s0 += st8[u];
          s0 += c8[u];
          s1 += g1[u];
          s1 += g2[u];
          s1 += a8[u];
          // the wall's share (navier_stokes.cu:236-241): what this pair did to the running sums
          const float d = (s0 - f_before) + (s1 - a_before) * mi;
          d8[u] = (mine >> u) & 1u ? d : 0.0f;
          if (sub < 3) s2 += d8[u];
        }
        if (sub < 3) {
          float4* to = reinterpret_cast<float4*>(rows + (kRowF + ax) * kRowStride + lead);
          to[0] = make_float4(d8[0], d8[1], d8[2], d8[3]);
          to[1] = make_float4(d8[4], d8[5], d8[6], d8[7]);
        }
        __syncwarp();
        const int ay = ax == 2 ? 0 : ax + 1, az = ax == 0 ? 2 : ax - 1;  // the other two axes, in cross-product order
        float xy[8], xz[8], fy[8], fz[8];
        get_row(kRowX + (sub < 6 ? ay : 0), xy);
        get_row(kRowX + (sub < 6 ? az : 0), xz);
        get_row(kRowF + (sub < 6 ? ay : 0), fy);
        get_row(kRowF + (sub < 6 ? az : 0), fz);
        if (sub >= 3 && sub < 6) {
#pragma unroll
          for (int u = 0; u < 8; ++u)
            if ((mine >> u) & 1u) s2 += xy[u] * fz[u] - xz[u] * fy[u];
        }
      }
      if (what & FORCE_AKINCI) {
        float k8[8];
        get_row(sub >= 3 && sub < 6 ? kRowK + ax : kRowZero, k8);
#pragma unroll
        for (int u = 0; u < 8; ++u) s3 += k8[u];
      }
      if (any_q) {
        float q8[8];
        get_row(sub == 6 ? kRowQ : kRowZero, q8);
#pragma unroll
        for (int u = 0; u < 8; ++u) s3 += q8[u];
      }
      __syncwarp();  // the rows are free again
    }

    // the particle's sums, in its first lane
    auto from = [&](float v, int l) { return __shfl_sync(kAll, v, lead + l); };
    const V3 force{from(s0, 0), from(s0, 1), from(s0, 2)};
    const V3 acc_av{from(s1, 0), from(s1, 1), from(s1, 2)};
    const V3 fwall{from(s2, 0), from(s2, 1), from(s2, 2)};
    const V3 sumT{from(s0, 3), from(s0, 4), from(s0, 5)};
    const V3 G{from(s1, 3), from(s1, 4), from(s1, 5)};
    const V3 mwall{from(s2, 3), from(s2, 4), from(s2, 5)};
    const V3 accA = (what & FORCE_AKINCI) ? V3{from(s3, 3), from(s3, 4), from(s3, 5)} : V3{0, 0, 0};
    const float div = from(s0, 6), diff = from(s0, 7), num = from(s1, 6), den = from(s1, 7);
    float q = from(s3, 6);
    if (!live || sub != 0) continue;

    if constexpr ((WHAT & FORCE_TAPE) != 0) {
      const int tn = V.tape_n;
      V.tape[i] = f4(force, q);
      V.tape[tn + i] = f4(sumT, num);
      V.tape[2 * tn + i] = make_float4(den, 0.0f, 0.0f, 0.0f);
    }
    V3 ab{0, 0, 0};
    if (do_T) {
      const float mT_i = rhoi * VT_i;
      const float pb = P.tvf_factor * P.rho0[pi_idx] * ci * ci;
      ab = sumT * (-pb / mT_i);
    }
    V.ab4[i] = f4(ab, V.ab4[i].w);
    float4 a4 = V.a4[i];
    V3 acc = xyz(a4);
    if (what & FORCE_MOMENTUM) {
      const V3 grav = v3(dyn->fr.gravity[0], dyn->fr.gravity[1], dyn->fr.gravity[2]);
      acc = grav + force / mi + acc_av;
      if (dyn->fr.frame_rot) {
        const V3 omega = v3(dyn->fr.omega[0], dyn->fr.omega[1], dyn->fr.omega[2]);
        const V3 omega_dot = v3(dyn->fr.omega_dot[0], dyn->fr.omega_dot[1], dyn->fr.omega_dot[2]);
        const V3 rr = xi - origin;
        acc -= cross(omega_dot, rr) + cross(omega, cross(omega, rr)) + cross(omega, vi) * 2.0f;
      }
      V.fw[i] = f4(fwall, 0.0f);
      V.mw[i] = f4(mwall, 0.0f);
    }
    if (what & FORCE_CSF) {
      float4 ns4 = V.ns4[i];
      if (!do_C) {
        ns4.w = 0.0f;
      } else {
        const float kappa = den > 0.0f ? 3.0f * num / den : 0.0f;
        ns4.w = kappa;
        if (P.wetting_model != 0) acc += xyz(V.vwp[i]);
        if (P.csf_balanced) acc += G * (P.sigma * kappa / mi);
        else acc += xyz(V.nrm[i]) * (csf_coeff * kappa);
      }
      V.ns4[i] = ns4;
    }
    if (do_A) acc += accA;
    if (do_D) reinterpret_cast<float*>(V.ab4 + i)[3] = rhoi * div + P.delta_sph * h * P.c0 * diff;
    if (thermal) {
      q += P.heat_power * V.heat_w[i] * dyn->heat_inv_norm;
      a4.w = q / (mi * P.cp[pi_idx]);
    }
    V.a4[i] = f4(acc, a4.w);

    if ((what & FORCE_MAXIMA) && owned(own_lo, own_hi, n_sorted, i)) {
      vmax_l = fmaxf(vmax_l, norm(vi));
      const float rm = V.rmin[i];
      const float rr = rm > 0.05f * P.dx ? rm : 0.05f * P.dx;
      sr_l = fmaxf(sr_l, 0.5f * P.dx / rr);
      const float aa = norm(acc), bb = norm(ab);
      amax_l = fmaxf(amax_l, aa > bb ? aa : bb);
      if (ph == kVapor) tv_l = fmaxf(tv_l, Ti);
      if (P.sps) nut_l = fmaxf(nut_l, V.nu_t[i]);
    }
  }
  if (what & FORCE_MAXIMA) {
    vmax_l = warp_max(vmax_l);
    amax_l = warp_max(amax_l);
    tv_l = warp_max(tv_l);
    sr_l = warp_max(sr_l);
    nut_l = warp_max(nut_l);
    if ((threadIdx.x & 31) == 0) {
      atomic_max_pos(&dyn->v_max, vmax_l);
      atomic_max_pos(&dyn->a_max, amax_l);
      if (P.has_vapor) atomic_max_pos(&dyn->Tv_max, tv_l);
      atomic_max_pos(&dyn->spacing_ratio, sr_l);
      if (P.sps) atomic_max_pos(&dyn->nu_t_max, nut_l);
    }
  }
}


#define FORCES_INSTANCE(W) template __global__ void k_forces_t<W>(Params, View);
FORCES_INSTANCE(FORCE_BASE)
FORCES_INSTANCE(FORCE_BASE | FORCE_THERMAL)
FORCES_INSTANCE(FORCE_BASE | FORCE_DRHO)
FORCES_INSTANCE(FORCE_BASE | FORCE_DRHO | FORCE_THERMAL)
FORCES_INSTANCE(FORCE_BASE | FORCE_AKINCI)
FORCES_INSTANCE(FORCE_BASE | FORCE_AKINCI | FORCE_THERMAL)
FORCES_INSTANCE(FORCE_BASE | FORCE_AKINCI | FORCE_DRHO)
FORCES_INSTANCE(FORCE_BASE | FORCE_AKINCI | FORCE_DRHO | FORCE_THERMAL)
FORCES_INSTANCE(FORCE_BASE | FORCE_CSF)
FORCES_INSTANCE(FORCE_BASE | FORCE_CSF | FORCE_THERMAL)
FORCES_INSTANCE(FORCE_BASE | FORCE_CSF | FORCE_DRHO)
FORCES_INSTANCE(FORCE_BASE | FORCE_CSF | FORCE_DRHO | FORCE_THERMAL)
FORCES_INSTANCE(FORCE_BASE | FORCE_TAPE)
FORCES_INSTANCE(FORCE_BASE | FORCE_THERMAL | FORCE_TAPE)
FORCES_INSTANCE(FORCE_BASE | FORCE_CSF | FORCE_TAPE)
FORCES_INSTANCE(FORCE_BASE | FORCE_CSF | FORCE_THERMAL | FORCE_TAPE)

}  // namespace lanes
}  // namespace cryo
