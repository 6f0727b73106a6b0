// FP32-bulk / FP64-critical kernels of the reacting-RANS step.
//
// Same discretisation and step structure as the FP64 kernels (and the
// reference), with the precision split:
//   FP32: reconstruction and limiter, mixture thermodynamics at faces, AUSM+
//         and viscous fluxes, local time step, SST source, DPLUR flux-Jacobian
//         products, transport properties (mu, lambda, rho D, cp, gamma, a);
//   FP64: the state arrays and the conservative update accumulation, the
//         temperature Newton inversion (k_update), the finite-rate chemistry
//         with its equilibrium constants exp(-dG/RT) and reverse rates, the
//         point-implicit (EPI) Jacobian and its LU solve, the residual norms.
// Device arrays stay FP64 (one state for both paths); the FP32 kernels
// convert on load and round their results back on store.
#pragma once

#include "kernels_step.cuh"

namespace ostc {

// Float copies of the tables the FP32 kernels read.
struct MixParams {
  float mw[kMaxSpec], mw_inv[kMaxSpec], ru_mw[kMaxSpec], t_low[kMaxSpec], t_mid[kMaxSpec];
  float low[kMaxSpec * 7], high[kMaxSpec * 7];
  float lj_inv[kMaxSpec], vis_coeff[kMaxSpec];
  float wq[kMaxSpec * kMaxSpec], w8[kMaxSpec * kMaxSpec];
  float cfl, Pr, Prt, Sct, Sc;
};

static __constant__ MixParams cF;

inline MixParams make_mix_params(const DevParams &p) {
  MixParams f{};
  for (int i = 0; i < kMaxSpec; ++i) {
    f.mw[i] = static_cast<float>(p.mw[i]);
    f.mw_inv[i] = p.mw[i] != 0 ? static_cast<float>(1.0 / p.mw[i]) : 0.f;
    f.ru_mw[i] = static_cast<float>(p.ru_mw[i]);
    f.t_low[i] = static_cast<float>(p.t_low[i]);
    f.t_mid[i] = static_cast<float>(p.t_mid[i]);
    f.lj_inv[i] = static_cast<float>(p.lj_inv[i]);
    f.vis_coeff[i] = static_cast<float>(p.vis_coeff[i]);
  }
  for (int i = 0; i < kMaxSpec * 7; ++i) {
    f.low[i] = static_cast<float>(p.low[i]);
    f.high[i] = static_cast<float>(p.high[i]);
  }
  for (int i = 0; i < kMaxSpec * kMaxSpec; ++i) {
    f.wq[i] = static_cast<float>(p.wq[i]);
    f.w8[i] = static_cast<float>(p.w8[i]);
  }
  f.cfl = static_cast<float>(p.cfl);
  f.Pr = static_cast<float>(p.Pr);
  f.Prt = static_cast<float>(p.Prt);
  f.Sct = static_cast<float>(p.Sct);
  f.Sc = static_cast<float>(p.Sc);
  return f;
}

namespace fp32 {

// tanh of a non-negative argument from one hardware exponential:
// 1 - 2 / (e^{2x} + 1) (relative error near 1e-6; 1 where e^{2x} overflows).
// The SST blending functions F1, F2 take it.
__device__ __forceinline__ float tanh_pos(float x) { return 1.f - __fdividef(2.f, __expf(2.f * x) + 1.f); }

constexpr float kRu = 8314.462618f;

__device__ __forceinline__ float ldf(const double *p) { return static_cast<float>(__ldg(p)); }

__device__ __forceinline__ float minmod(float a, float b) {
  return 0.5f * ((a < 0 ? -1.f : 1.f) + (b < 0 ? -1.f : 1.f)) * fminf(fabsf(a), fabsf(b));
}

// NASA-7 polynomial coefficient q of species i (two ranges)
__device__ __forceinline__ float nasa(int i, int q, bool lowrange) {
  return lowrange ? cF.low[i * 7 + q] : cF.high[i * 7 + q];
}

// Species h_k and cp_k (J/kg, J/kg/K) at t; below T_low h is extrapolated
// linearly with cp frozen, as in the FP64 path.
template <int NS, bool WANT_H, bool WANT_CP>
__device__ __forceinline__ void thermo(float t, float *h, float *cp) {
  OSTC_UNROLL for (int i = 0; i < NS; ++i) {
    const bool below = t < cF.t_low[i];
    const float tt = below ? cF.t_low[i] : t;
    const bool lo = below || tt < cF.t_mid[i];
    const float c0 = nasa(i, 0, lo), c1 = nasa(i, 1, lo), c2 = nasa(i, 2, lo), c3 = nasa(i, 3, lo),
                c4 = nasa(i, 4, lo);
    const float c = c0 + tt * (c1 + tt * (c2 + tt * (c3 + tt * c4)));
    if constexpr (WANT_H) {
      float hh = tt * (c0 + tt * (0.5f * c1 + tt * (c2 * (1.f / 3.f) + tt * (0.25f * c3 + tt * (0.2f * c4))))) +
                 nasa(i, 5, lo);
      if (below) hh += c * (t - tt);
      h[i] = hh * cF.ru_mw[i];
    }
    if constexpr (WANT_CP) cp[i] = c * cF.ru_mw[i];
  }
}

// The FP32 copy of the operands of the flux passes and the sweeps
// (DevBlock::f32), written once per step by k_pack32 and, for the geometry,
// once per run by k_pack32_static.  Four components of a cell lie together
// (quads, one array of B.G.size float4 per quad), so that a stencil point is
// a few 16-byte loads: a face reads 74 of them instead of 348 4-byte ones, and
// those loads, with their address arithmetic, are what the passes waited for.
struct Quad {
  static constexpr int rho_vel = 0,    // rho, u, v, w
      p_t_turb = 1,                    // p, T, k, omega
      y0 = 2, y4 = 3,                  // Y_0..3, Y_4..7
      y8_mu = 4,                       // Y_8, mu, mu_t, lambda
      misc = 5,                        // lambda_t, a, gamma, (rho D)_8
      d0 = 6, d4 = 7,                  // (rho D)_0..3, _4..7
      n_dynamic = 8, metric = 8,       // metric + d: grad of coordinate d, and J, wall distance, 0
      count = 11;
};

// h_k and cp_k of species i at t (thermo<> for one species)
__device__ __forceinline__ void thermo_one(int i, float t, float &h, float &cp) {
  const bool below = t < cF.t_low[i];
  const float tt = below ? cF.t_low[i] : t;
  const bool lo = below || tt < cF.t_mid[i];
  const float c0 = nasa(i, 0, lo), c1 = nasa(i, 1, lo), c2 = nasa(i, 2, lo), c3 = nasa(i, 3, lo),
              c4 = nasa(i, 4, lo);
  const float c = c0 + tt * (c1 + tt * (c2 + tt * (c3 + tt * c4)));
  float hh = tt * (c0 + tt * (0.5f * c1 + tt * (c2 * (1.f / 3.f) + tt * (0.25f * c3 + tt * (0.2f * c4))))) +
             nasa(i, 5, lo);
  if (below) hh += c * (t - tt);
  h = hh * cF.ru_mw[i];
  cp = c * cF.ru_mw[i];
}

// ------------------------------------------------------------ inviscid face
// Left and right values at a face of a variable with these four stencil values.
__device__ __forceinline__ void reconstruct(int rec, float pm, float p0, float p1, float p2, float &l, float &r) {
  if (rec == 2 || rec == 3) {
    const float d_i = p0 - pm, d_i1 = p1 - p0, d_i2 = p2 - p1;
    const float ml = minmod(d_i, d_i1), mr = minmod(d_i1, d_i2);
    if (rec == 2) {  // kappa = 1/3: both slopes of a side are the same minmod
      l = p0 + 0.25f * ((2.f / 3.f) * ml + (4.f / 3.f) * ml);
      r = p1 - 0.25f * ((2.f / 3.f) * mr + (4.f / 3.f) * mr);
    } else {
      l = p0 + 0.5f * ml;
      r = p1 - 0.5f * mr;
    }
  } else {
    l = p0;
    r = p1;
  }
}

// AUSM+/MUSCL flux through the face between cells n and n + s of direction d
// (f: the quads), and the face's area vector k.
template <class C>
__device__ __forceinline__ void inviscid_face(const float4 *__restrict__ f, int64_t sz, int64_t n, int d, int64_t s,
                                              float *fc, float &k1, float &k2, float &k3) {
  constexpr int NV = C::nv, NS = C::ns;
  static_assert(C::mix != 0 && NS == 9 && C::turb, "the quads hold nine species and k, omega");
  float pl[NV + 2], pr[NV + 2];
  const int rec = cP.reconstruction;
  // the quad's x, y, z, w are flux variables lx, ly, lz, lw (-1: none)
  auto take = [&](int quad, int lx, int ly, int lz, int lw) {
    const float4 *q = f + quad * sz + n;
    const float4 c = __ldg(q), e = __ldg(q + s);
    float4 m = c, g = e;
    if (rec == 2 || rec == 3) {
      m = __ldg(q - s);
      g = __ldg(q + 2 * s);
    }
    if (lx >= 0) reconstruct(rec, m.x, c.x, e.x, g.x, pl[lx], pr[lx]);
    if (ly >= 0) reconstruct(rec, m.y, c.y, e.y, g.y, pl[ly], pr[ly]);
    if (lz >= 0) reconstruct(rec, m.z, c.z, e.z, g.z, pl[lz], pr[lz]);
    if (lw >= 0) reconstruct(rec, m.w, c.w, e.w, g.w, pl[lw], pr[lw]);
  };
  take(Quad::rho_vel, 0, 1, 2, 3);
  take(Quad::p_t_turb, 4, -1, 5 + NS, 6 + NS);
  take(Quad::y0, 5, 6, 7, 8);
  take(Quad::y4, 9, 10, 11, 12);
  take(Quad::y8_mu, 13, -1, -1, -1);
  float el = 0.5f * (pl[1] * pl[1] + pl[2] * pl[2] + pl[3] * pl[3]);
  float er = 0.5f * (pr[1] * pr[1] + pr[2] * pr[2] + pr[3] * pr[3]);
  float mwl = 0, mwr = 0;
  OSTC_UNROLL for (int l = 0; l < NS; ++l) {
    mwl += pl[5 + l] * cF.mw_inv[l];
    mwr += pr[5 + l] * cF.mw_inv[l];
  }
  const float tl = pl[4] / (pl[0] * kRu * mwl);
  const float tr = pr[4] / (pr[0] * kRu * mwr);
  float cpl = 0, cpr = 0, cvl = 0, cvr = 0;
  OSTC_UNROLL for (int l = 0; l < NS; ++l) {
    float hl, hr, cpl_l, cpr_l;
    thermo_one(l, tl, hl, cpl_l);
    thermo_one(l, tr, hr, cpr_l);
    cpl += cpl_l * pl[l + 5];
    cpr += cpr_l * pr[l + 5];
    cvl += pl[l + 5] * (cpl_l - cF.ru_mw[l]);
    cvr += pr[l + 5] * (cpr_l - cF.ru_mw[l]);
    el += hl * pl[l + 5];
    er += hr * pr[l + 5];
  }
  pl[NV] = pl[0] * el - pl[4];
  pr[NV] = pr[0] * er - pr[4];
  pl[NV + 1] = cpl / cvl;
  pr[NV + 1] = cpr / cvr;
  const float4 *xi = f + (Quad::metric + d) * sz + n, *jac = f + Quad::metric * sz + n;
  const float4 ml = __ldg(xi), mr = __ldg(xi + s);
  const float jl = __ldg(&jac->w), jr = __ldg(&(jac + s)->w);
  k1 = 0.5f * (jl * ml.x + jr * mr.x);
  k2 = 0.5f * (jl * ml.y + jr * mr.y);
  k3 = 0.5f * (jl * ml.z + jr * mr.z);
  const float gk = sqrtf(k1 * k1 + k2 * k2 + k3 * k3);
  const float inv_gk = 1.f / gk;
  const float ul = (k1 * pl[1] + k2 * pl[2] + k3 * pl[3]) * inv_gk;
  const float ur = (k1 * pr[1] + k2 * pr[2] + k3 * pr[3]) * inv_gk;
  const float p_l = pl[4], p_r = pr[4], rho_l = pl[0], rho_r = pr[0];
  const float c = 0.5f * (sqrtf(pl[NV + 1] * p_l / rho_l) + sqrtf(pr[NV + 1] * p_r / rho_r));
  const float inv_c = 1.f / c;
  const float mach_l = ul * inv_c, mach_r = ur * inv_c;
  float mlp, mrn, plp, prn;
  constexpr float alpha = 3.f / 16.f;
  if (fabsf(mach_l) > 1) {
    mlp = 0.5f * (mach_l + fabsf(mach_l));
    plp = mlp / mach_l;
  } else {
    const float a = (mach_l + 1) * (mach_l + 1) * 0.25f;
    const float b = (mach_l * mach_l - 1) * (mach_l * mach_l - 1);
    mlp = a + 0.125f * b;
    plp = a * (2 - mach_l) + alpha * mach_l * b;
  }
  if (fabsf(mach_r) > 1) {
    mrn = 0.5f * (mach_r - fabsf(mach_r));
    prn = mrn / mach_r;
  } else {
    const float a = (mach_r - 1) * (mach_r - 1) * 0.25f;
    const float b = (mach_r * mach_r - 1) * (mach_r * mach_r - 1);
    mrn = -a - 0.125f * b;
    prn = a * (2 + mach_r) - alpha * mach_r * b;
  }
  const float p_coeff = plp * p_l + prn * p_r;
  const float m_half = mlp + mrn;
  const float mach_pos = 0.5f * (m_half + fabsf(m_half));
  const float mach_neg = 0.5f * (m_half - fabsf(m_half));
  const float mass_flux_half = c * (rho_l * mach_pos + rho_r * mach_neg);
  const float coeff = mass_flux_half * gk;
  const bool up = mass_flux_half >= 0;
  // upwind state, selected per element so that pl / pr stay in registers
  auto q = [&](int l) { return up ? pl[l] : pr[l]; };
  fc[0] = coeff;
  fc[1] = coeff * q(1) + p_coeff * k1;
  fc[2] = coeff * q(2) + p_coeff * k2;
  fc[3] = coeff * q(3) + p_coeff * k3;
  fc[4] = coeff * (q(NV) + q(4)) / q(0);
  OSTC_UNROLL for (int l = 5; l < NV; ++l) fc[l] = coeff * q(l);
}

// ------------------------------------------------------------- viscous face
// A quad at both cells of a face and its three computational-space derivatives
// there (the normal one by the two-point difference, the others by the
// four-point average).
struct FaceQuad {
  float4 a, b, xi, eta, zeta;
};

__device__ __forceinline__ FaceQuad face_quad(const float4 *__restrict__ q, int64_t s, int d, int64_t sx, int64_t sxy) {
  FaceQuad r;
  r.a = __ldg(q);
  r.b = __ldg(q + s);
  const float4 normal = make_float4(r.b.x - r.a.x, r.b.y - r.a.y, r.b.z - r.a.z, r.b.w - r.a.w);
  auto across = [&](int64_t t) {
    const float4 ap = __ldg(q + t), am = __ldg(q - t), bp = __ldg(q + s + t), bm = __ldg(q + s - t);
    return make_float4(0.25f * (ap.x - am.x + bp.x - bm.x), 0.25f * (ap.y - am.y + bp.y - bm.y),
                       0.25f * (ap.z - am.z + bp.z - bm.z), 0.25f * (ap.w - am.w + bp.w - bm.w));
  };
  r.xi = d == 0 ? normal : across(1);
  r.eta = d == 1 ? normal : across(sx);
  r.zeta = d == 2 ? normal : across(sxy);
  return r;
}

// Adds the viscous flux through the face between n and n + s (area vector
// kx, ky, kz) to g.  The derivative of a scalar along k needs the three
// products k . grad(xi), k . grad(eta), k . grad(zeta) once per face and not the
// scalar's Cartesian gradient; the species fluxes sum up to their correction.
template <class C>
__device__ __forceinline__ void viscous_face_add(const float4 *__restrict__ f, int64_t sz, int64_t sx, int64_t sxy,
                                                 int64_t n, int d, int64_t s, float kx, float ky, float kz, float *g) {
  constexpr int NS = C::ns;
  const float4 *fn = f + n;
  auto both = [&](int quad) {
    const float4 a = __ldg(fn + quad * sz), b = __ldg(fn + quad * sz + s);
    return make_float4(0.5f * (a.x + b.x), 0.5f * (a.y + b.y), 0.5f * (a.z + b.z), 0.5f * (a.w + b.w));
  };
  const float4 mx = both(Quad::metric), me = both(Quad::metric + 1), mz = both(Quad::metric + 2);
  const float wall_dist = me.w;
  const float c_xi = kx * mx.x + ky * mx.y + kz * mx.z, c_eta = kx * me.x + ky * me.y + kz * me.z,
              c_zeta = kx * mz.x + ky * mz.y + kz * mz.z;
  // the mean of Y_8, mu, mu_t, lambda comes with Y_8's derivatives, at the end
  const float4 mu4 = both(Quad::y8_mu), misc = both(Quad::misc);
  const float mul = mu4.y, mut = mu4.z, conductivity = mu4.w + misc.x;
  const float viscosity = mul + mut;
  constexpr float third = 1.f / 3.f;
  float rhom, rho_a, rho_b;
  {
    const FaceQuad q = face_quad(fn + Quad::rho_vel * sz, s, d, sx, sxy);
    auto cart = [&](float a_xi, float a_eta, float a_zeta, float &ax, float &ay, float &az) {
      ax = a_xi * mx.x + a_eta * me.x + a_zeta * mz.x;
      ay = a_xi * mx.y + a_eta * me.y + a_zeta * mz.y;
      az = a_xi * mx.z + a_eta * me.z + a_zeta * mz.z;
    };
    float u_x, u_y, u_z, v_x, v_y, v_z, w_x, w_y, w_z;
    cart(q.xi.y, q.eta.y, q.zeta.y, u_x, u_y, u_z);
    cart(q.xi.z, q.eta.z, q.zeta.z, v_x, v_y, v_z);
    cart(q.xi.w, q.eta.w, q.zeta.w, w_x, w_y, w_z);
    const float4 ta = __ldg(fn + Quad::p_t_turb * sz), tb = __ldg(fn + Quad::p_t_turb * sz + s);
    const float tt = -third * (q.a.x * ta.z + q.b.x * tb.z);  // -2/3 rho k
    const float tau_xx = viscosity * (4 * u_x - 2 * v_y - 2 * w_z) * third + tt;
    const float tau_yy = viscosity * (4 * v_y - 2 * u_x - 2 * w_z) * third + tt;
    const float tau_zz = viscosity * (4 * w_z - 2 * u_x - 2 * v_y) * third + tt;
    const float tau_xy = viscosity * (u_y + v_x);
    const float tau_xz = viscosity * (u_z + w_x);
    const float tau_yz = viscosity * (v_z + w_y);
    const float f1 = kx * tau_xx + ky * tau_xy + kz * tau_xz, f2 = kx * tau_xy + ky * tau_yy + kz * tau_yz,
                f3 = kx * tau_xz + ky * tau_yz + kz * tau_zz;
    g[1] += f1;
    g[2] += f2;
    g[3] += f3;
    g[4] += 0.5f * (q.a.y + q.b.y) * f1 + 0.5f * (q.a.z + q.b.z) * f2 + 0.5f * (q.a.w + q.b.w) * f3;
    rho_a = q.a.x;
    rho_b = q.b.x;
    rhom = 0.5f * (rho_a + rho_b);
  }
  float tm;
  {
    const FaceQuad q = face_quad(fn + Quad::p_t_turb * sz, s, d, sx, sxy);
    tm = 0.5f * (q.a.y + q.b.y);
    g[4] += conductivity * (c_xi * q.xi.y + c_eta * q.eta.y + c_zeta * q.zeta.y);
    const float k_n = c_xi * q.xi.z + c_eta * q.eta.z + c_zeta * q.zeta.z;
    const float o_n = c_xi * q.xi.w + c_eta * q.eta.w + c_zeta * q.zeta.w;
    float f1 = 1;
    if (wall_dist > 1e-25f) {
      auto dx = [&](float a, float b, float c) { return a * mx.x + b * me.x + c * mz.x; };
      auto dy = [&](float a, float b, float c) { return a * mx.y + b * me.y + c * mz.y; };
      auto dz = [&](float a, float b, float c) { return a * mx.z + b * me.z + c * mz.z; };
      const float cross = dx(q.xi.z, q.eta.z, q.zeta.z) * dx(q.xi.w, q.eta.w, q.zeta.w) +
                          dy(q.xi.z, q.eta.z, q.zeta.z) * dy(q.xi.w, q.eta.w, q.zeta.w) +
                          dz(q.xi.z, q.eta.z, q.zeta.z) * dz(q.xi.w, q.eta.w, q.zeta.w);
      const float km = 0.5f * (q.a.z + q.b.z), omegam = 0.5f * (q.a.w + q.b.w);
      const float param1 = sqrtf(km) / (0.09f * omegam * wall_dist);
      const float d2 = wall_dist * wall_dist;
      const float param2 = 500 * mul / (rhom * d2 * omegam);
      constexpr float so2 = static_cast<float>(sst::sigma_omega2);
      const float CDkomega = fmaxf(1e-20f, 2 * rhom * so2 / omegam * cross);
      const float param3 = 4 * rhom * so2 * km / (CDkomega * d2);
      const float arg1 = fminf(fmaxf(param1, param2), param3);
      f1 = tanh_pos(arg1 * arg1 * arg1 * arg1);
    }
    const float sigma_k = static_cast<float>(sst::sigma_k2) + static_cast<float>(sst::delta_sigma_k) * f1;
    const float sigma_omega =
        static_cast<float>(sst::sigma_omega2) + static_cast<float>(sst::delta_sigma_omega) * f1;
    g[5 + NS] += (mul + mut * sigma_k) * k_n;
    g[6 + NS] += (mul + mut * sigma_omega) * o_n;
  }
  const float turb_d = mut / cF.Sct;
  float hflux = 0, total = 0;
  auto species = [&](int l, float dif, float xi, float eta, float zeta) {
    float h, cp_unused;
    thermo_one(l, tm, h, cp_unused);
    const float flux = (dif + turb_d) * (c_xi * xi + c_eta * eta + c_zeta * zeta);
    g[5 + l] += flux;
    hflux += h * flux;
    total += flux;
  };
  float4 y0, y4;
  float y8;
  {
    const float4 dif = both(Quad::d0);
    const FaceQuad q = face_quad(fn + Quad::y0 * sz, s, d, sx, sxy);
    species(0, dif.x, q.xi.x, q.eta.x, q.zeta.x);
    species(1, dif.y, q.xi.y, q.eta.y, q.zeta.y);
    species(2, dif.z, q.xi.z, q.eta.z, q.zeta.z);
    species(3, dif.w, q.xi.w, q.eta.w, q.zeta.w);
    y0 = make_float4(0.5f * (q.a.x + q.b.x), 0.5f * (q.a.y + q.b.y), 0.5f * (q.a.z + q.b.z), 0.5f * (q.a.w + q.b.w));
  }
  {
    const float4 dif = both(Quad::d4);
    const FaceQuad q = face_quad(fn + Quad::y4 * sz, s, d, sx, sxy);
    species(4, dif.x, q.xi.x, q.eta.x, q.zeta.x);
    species(5, dif.y, q.xi.y, q.eta.y, q.zeta.y);
    species(6, dif.z, q.xi.z, q.eta.z, q.zeta.z);
    species(7, dif.w, q.xi.w, q.eta.w, q.zeta.w);
    y4 = make_float4(0.5f * (q.a.x + q.b.x), 0.5f * (q.a.y + q.b.y), 0.5f * (q.a.z + q.b.z), 0.5f * (q.a.w + q.b.w));
  }
  {
    const FaceQuad q = face_quad(fn + Quad::y8_mu * sz, s, d, sx, sxy);
    species(8, misc.w, q.xi.x, q.eta.x, q.zeta.x);
    y8 = 0.5f * (q.a.x + q.b.x);
  }
  g[4] += hflux;
  g[5] -= y0.x * total;
  g[6] -= y0.y * total;
  g[7] -= y0.z * total;
  g[8] -= y0.w * total;
  g[9] -= y4.x * total;
  g[10] -= y4.y * total;
  g[11] -= y4.z * total;
  g[12] -= y4.w * total;
  g[13] -= y8 * total;
}

// ------------------------------------------------------------- SST source
template <class C>
__device__ __forceinline__ void sst_source(const DevBlock &B, int64_t n, double &src_k, double &src_w,
                                           double &mut_out, double &jk, double &jw) {
  constexpr int NS = C::ns;
  const int64_t sz = B.G.size, sx = B.G.sx, sxy = B.G.sxy;
  const double *m = B.metric;
  const float xi_x = ldf(m + n), xi_y = ldf(m + sz + n), xi_z = ldf(m + 2 * sz + n);
  const float eta_x = ldf(m + 3 * sz + n), eta_y = ldf(m + 4 * sz + n), eta_z = ldf(m + 5 * sz + n);
  const float zeta_x = ldf(m + 6 * sz + n), zeta_y = ldf(m + 7 * sz + n), zeta_z = ldf(m + 8 * sz + n);
  auto cgrad = [&](const double *a, float &gx, float &gy, float &gz) {
    const float a_xi = ldf(a + n + 1) - ldf(a + n - 1), a_eta = ldf(a + n + sx) - ldf(a + n - sx),
                a_zeta = ldf(a + n + sxy) - ldf(a + n - sxy);
    gx = 0.5f * (xi_x * a_xi + eta_x * a_eta + zeta_x * a_zeta);
    gy = 0.5f * (xi_y * a_xi + eta_y * a_eta + zeta_y * a_zeta);
    gz = 0.5f * (xi_z * a_xi + eta_z * a_eta + zeta_z * a_zeta);
  };
  float u_x, u_y, u_z, v_x, v_y, v_z, w_x, w_y, w_z, k_x, k_y, k_z, o_x, o_y, o_z;
  cgrad(B.bv + sz, u_x, u_y, u_z);
  cgrad(B.bv + 2 * sz, v_x, v_y, v_z);
  cgrad(B.bv + 3 * sz, w_x, w_y, w_z);
  const double *tk = B.sv + NS * sz, *tw = B.sv + (NS + 1) * sz;
  cgrad(tk, k_x, k_y, k_z);
  cgrad(tw, o_x, o_y, o_z);
  const float density = ldf(B.bv + n), omega = ldf(tw + n), tke = ldf(tk + n);
  constexpr float so2 = static_cast<float>(sst::sigma_omega2), a1 = static_cast<float>(sst::a_1);
  const float inter_var = 2 * density * so2 / omega * (k_x * o_x + k_y * o_y + k_z * o_z);
  const float rhoK = density * tke;
  const float vorticity =
      sqrtf((v_x - u_y) * (v_x - u_y) + (w_x - u_z) * (w_x - u_z) + (w_y - v_z) * (w_y - v_z));
  float f1 = 1, f2 = 1;
  const float dy = ldf(B.wall_dist + n);
  if (dy > 1e-25f) {
    const float param1 = sqrtf(tke) / (0.09f * omega * dy);
    const float d2 = dy * dy;
    const float param2 = 500 * ldf(B.mul + n) / (density * d2 * omega);
    const float arg2 = fmaxf(2 * param1, param2);
    f2 = tanh_pos(arg2 * arg2);
    const float CDkomega = fmaxf(1e-20f, inter_var);
    const float param3 = 4 * density * so2 * tke / (CDkomega * d2);
    const float arg1 = fminf(fmaxf(param1, param2), param3);
    f1 = tanh_pos(arg1 * arg1 * arg1 * arg1);
  }
  float mut = 0;
  if (const float den = fmaxf(a1 * omega, vorticity * f2); den > 1e-25f) mut = a1 * rhoK / den;
  mut_out = mut;
  const float beta = static_cast<float>(sst::beta_2) + static_cast<float>(sst::delta_beta) * f1;
  src_k = 0;
  src_w = 0;
  if (mut > 1e-25f) {
    const float divU = u_x + v_y + w_z;
    const float prod_k = mut * (2 * (u_x * u_x + v_y * v_y + w_z * w_z) - (2.f / 3.f) * divU * divU +
                                (u_y + v_x) * (u_y + v_x) + (u_z + w_x) * (u_z + w_x) + (v_z + w_y) * (v_z + w_y)) -
                         (2.f / 3.f) * rhoK * divU;
    const float diss_k = static_cast<float>(sst::beta_star) * rhoK * omega;
    const float jac = ldf(B.jac + n);
    src_k = jac * (prod_k - diss_k);
    const float gamma = static_cast<float>(sst::gamma2) + static_cast<float>(sst::delta_gamma) * f1;
    const float prod_omega = gamma * density / mut * prod_k + (1 - f1) * inter_var;
    const float diss_omega = beta * density * omega * omega;
    src_w = jac * (prod_omega - diss_omega);
  }
  jk = -2 * sst::beta_star * omega;
  jw = -2.0 * beta * omega;
}

}  // namespace fp32

// Finite-rate chemistry of one cell in FP64 (the FP64 path's code with each
// Arrhenius rate as one exponential):
// returns dq species = J omega and writes the EPI / DA Jacobian.  q1, q2:
// this thread's column of the CTA's shared rate arrays (stride kCta).
template <class C, class M>
__device__ __forceinline__ void chem_cell(const DevBlock &B, int64_t n, int64_t nz, double *q1, double *q2,
                                          double *dq_spec) {
  constexpr int NS = C::ns;
  const int64_t sz = B.G.size, sz0 = B.Z.size;
  double Y[NS], omega[NS], omega_d[NS];
  OSTC_UNROLL for (int l = 0; l < NS; ++l) Y[l] = ld(B.sv + l * sz + n);
  const double density = ld(B.bv + n), t = ld(B.bv + 5 * sz + n);
  const bool general = chemistry_of<NS, true, M>(density, t, Y, omega, omega_d, q1, q2, kCta);
  const double jac = ld(B.jac + n);
  OSTC_UNROLL for (int l = 0; l < NS; ++l) dq_spec[l] = jac * omega[l];
  const int method = cP.chem_src_method;
  if (method == 1) {
    // compute_chem_src_jacobian, row by row
    const int na = cP.na;
    // 1 / (rho Y_q) once per species (0 below the floor): products, not
    // NS^2 divisions, within an ulp of the FP64 path's quotients
    double inv_rho_y[NS];
    OSTC_UNROLL for (int q = 0; q < NS; ++q) inv_rho_y[q] = Y[q] > 1e-25 ? 1.0 / (density * Y[q]) : 0.0;
    // only the leading na x na block (the other rows and columns are zero)
    jacobian_rows<NS, M>(general, na, q1, q2, kCta, [&](int m, const double *zz) {
      OSTC_UNROLL for (int q = 0; q < NS; ++q) {
        if (q >= na) break;
        const double v = zz[q] * inv_rho_y[q];
        B.chem_jac[(m * na + q) * sz0 + nz] = cP.mw[m] * v * 1e+3;
      }
    });
  } else if (method == 2) {
    OSTC_UNROLL for (int l = 0; l < NS; ++l) {
      double v = 0;
      if (Y[l] > 1e-25) v = -omega_d[l] / (Y[l] * density);
      B.chem_jac[l * sz0 + nz] = v;
    }
  }
}

// dq = source terms: SST in FP32, finite-rate chemistry and its EPI Jacobian
// in FP64 (the same code as the FP64 path).  With the surrogate on
// (chem_quiet set) the chemistry of the cells it did not judge quiet runs in
// k_chem_list over a compacted list instead, with every lane of a warp busy;
// here those cells get zero species source, which k_chem_list overwrites.
template <class C, class M>
__global__ void __launch_bounds__(kCta, 4) k_source_mx(const DevBlock *__restrict__ blks, Tiles T) {
  constexpr int NS = C::ns, NV = C::nv;
  extern __shared__ double sq[];
  int b, i, j, k;
  if (!tile_cell<kTX, kTY, kTZ>(T, b, i, j, k, blks)) return;
  const DevBlock &B = blks[b];
  const int64_t n = B.G.at(i, j, k), nd = B.D.at(i, j, k), nz = B.Z.at(i, j, k);
  const int64_t szd = B.D.size, sz0 = B.Z.size;
  double dq[NV];
  OSTC_UNROLL for (int l = 0; l < NV; ++l) dq[l] = 0;
  if constexpr (C::turb) {
    double sk, sw, mut, jk, jw;
    fp32::sst_source<C>(B, n, sk, sw, mut, jk, jw);
    B.mut[n] = mut;
    dq[NS + 5] = sk;
    dq[NS + 6] = sw;
    if (cP.turb_implicit == 1) {
      B.turb_src_jac[nz] = jk;
      B.turb_src_jac[sz0 + nz] = jw;
    }
    B.turb_cond[n] = static_cast<float>(mut) * fp32::ldf(B.cp + n) / cF.Prt;
  }
  if constexpr (C::mix == 2) {
    if (B.chem_quiet) {
      if (B.chem_quiet[nz]) {
        // judged chemically quiet by the surrogate: its rate and no Jacobian
        // (the implicit stages treat the cell's species diagonally and never
        // read its chem_jac)
        const double jac = ld(B.jac + n);
        OSTC_UNROLL for (int l = 0; l < NS; ++l) dq[l + 5] = jac * B.chem_rate[l * sz0 + nz];
      }
    } else {
      const int tid = threadIdx.x + kTX * (threadIdx.y + kTY * threadIdx.z);
      chem_cell<C, M>(B, n, nz, sq + tid, sq + cP.nr * kCta + tid, dq + 5);
    }
  }
  OSTC_UNROLL for (int l = 0; l < NV; ++l) B.dq[l * szd + nd] = dq[l];
}

// The cells of block b the surrogate did not judge quiet, listed (any order).
template <class C>
__global__ void __launch_bounds__(256) k_chem_compact(const DevBlock *__restrict__ blks, int b, int *list,
                                                      int *count) {
  const DevBlock &B = blks[b];
  const int64_t cells = static_cast<int64_t>(B.mx) * B.my * B.mz;
  const int lane = threadIdx.x & 31;
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  for (int64_t base = static_cast<int64_t>(blockIdx.x) * blockDim.x; base < cells; base += stride) {
    const int64_t c = base + threadIdx.x;
    bool pick = false;
    if (c < cells) {
      const int i = static_cast<int>(c % B.mx), j = static_cast<int>((c / B.mx) % B.my),
                k = static_cast<int>(c / (static_cast<int64_t>(B.mx) * B.my));
      pick = B.chem_quiet[B.Z.at(i, j, k)] == 0;
    }
    const unsigned m = __ballot_sync(0xffffffffu, pick);
    int at = 0;
    if (lane == 0 && m) at = atomicAdd(count, __popc(m));
    at = __shfl_sync(0xffffffffu, at, 0);
    if (pick) list[at + __popc(m & ((1u << lane) - 1u))] = static_cast<int>(c);
  }
}

// Chemistry of the listed cells (k_chem_compact), one thread per entry, full
// warps; launched for the block's cell count, entries past the list return.
template <class C, class M>
__global__ void __launch_bounds__(kCta, 4) k_chem_list(const DevBlock *__restrict__ blks, int b,
                                                       const int *__restrict__ list, const int *count) {
  constexpr int NS = C::ns;
  extern __shared__ double sq[];
  const int q = blockIdx.x * kCta + threadIdx.x;
  if (q >= *count) return;
  const DevBlock &B = blks[b];
  const int64_t c = list[q];
  const int i = static_cast<int>(c % B.mx), j = static_cast<int>((c / B.mx) % B.my),
            k = static_cast<int>(c / (static_cast<int64_t>(B.mx) * B.my));
  const int64_t n = B.G.at(i, j, k), nz = B.Z.at(i, j, k), nd = B.D.at(i, j, k), szd = B.D.size;
  double dqs[NS];
  chem_cell<C, M>(B, n, nz, sq + threadIdx.x, sq + cP.nr * kCta + threadIdx.x, dqs);
  OSTC_UNROLL for (int l = 0; l < NS; ++l) B.dq[(5 + l) * szd + nd] = dqs[l];
}

// Local time step of cell (i, j, k) in FP32 (local_time_step,
// src/TimeAdvanceFunc.cuh:21-71); also stores the spectral radii the DPLUR
// sweeps use.
template <class C>
__device__ __forceinline__ void local_time_step_q(const DevBlock &B, const float4 *__restrict__ f, int i, int j, int k,
                                                  int64_t n, int64_t nd) {
  using Q = fp32::Quad;
  const int64_t szd = B.D.size, sz = B.G.size;
  const bool three_d = B.mz > 1;
  const float4 m1 = __ldg(f + Q::metric * sz + n), m2 = __ldg(f + (Q::metric + 1) * sz + n),
               m3 = __ldg(f + (Q::metric + 2) * sz + n), s = __ldg(f + Q::rho_vel * sz + n),
               misc = __ldg(f + Q::misc * sz + n), mu = __ldg(f + Q::y8_mu * sz + n);
  const float grad_xi = sqrtf(m1.x * m1.x + m1.y * m1.y + m1.z * m1.z);
  const float grad_eta = sqrtf(m2.x * m2.x + m2.y * m2.y + m2.z * m2.z);
  const float grad_zeta = sqrtf(m3.x * m3.x + m3.y * m3.y + m3.z * m3.z);
  const float a = misc.y;
  const float s0 = fabsf(s.y * m1.x + s.z * m1.y + s.w * m1.z) + a * grad_xi;
  const float s1 = fabsf(s.y * m2.x + s.z * m2.y + s.w * m2.z) + a * grad_eta;
  const float s2 = three_d ? fabsf(s.y * m3.x + s.z * m3.y + s.w * m3.z) + a * grad_zeta : 0.f;
  B.inv_spec[nd] = s0;
  B.inv_spec[szd + nd] = s1;
  B.inv_spec[2 * szd + nd] = s2;
  const float coeff_1 = fmaxf(misc.z, 4.f / 3.f) / s.x;
  const float coeff_2 = mu.y / cF.Pr + mu.z / cF.Prt;
  float srv = grad_xi * grad_xi + grad_eta * grad_eta;
  if (three_d) srv += grad_zeta * grad_zeta;
  srv *= coeff_1 * coeff_2;
  B.visc_spec[nd] = srv;
  B.dt_local[B.Z.at(i, j, k)] = cF.cfl / (s0 + s1 + s2 + srv);
}

// ----------------------------------------------------- direction passes
// The flux differences as three passes, one per direction d: every face
// along d is evaluated once, inviscid and viscous together, as
// G = F_viscous - F_inviscid, and each cell adds G(c + 1/2) - G(c - 1/2) to
// its FP64 dq.  A pass keeps one face's fluxes in registers and needs no
// shared memory or barrier, so its warps run independently and the SM keeps
// as many loads in flight as its register file allows; the price is dq read
// and written once per direction instead of once.  The x pass also stores
// the local time step.
//   x: a warp holds 32 consecutive faces of one row (i - 1/2 + lane) and
//      gives 31 cells their difference, the left face coming from the lane
//      below by a shuffle; a CTA covers 4 rows (j).
//   y, z: each thread marches over some cells along d, carrying the lower face
//      from one cell to the next; lanes run along i, the CTA's 4 warps over
//      the remaining index (k for y, j for z).
// The variants (flux_cut.hpp) differ in registers: 4, 6 and 8 CTAs per SM cap a thread
// at 128, 80 and 64 registers, with 60 to 132, 200 to 212 and 292 to 356 B of spill
// stores.  The loads in flight decide all the same: the three passes take 4.08, 3.52
// and 3.17 ms at 384x192x64, 1.02, 0.89 and 0.74 ms at 160x96x64 (one B200), and with a
// march of 16 instead of 8 at 8 CTAs 3.09 and 0.74 ms.

__device__ __forceinline__ void dir_tile(const Tiles &T, int &b, int &t0, int &t1, int &t2) {
  int t = tile_of(T, blockIdx.x, b);
  t0 = t % T.ntx[b];
  t /= T.ntx[b];
  t1 = t % T.nty[b];
  t2 = t / T.nty[b];
}

// G = F_viscous - F_inviscid at the face between linear index nl and nl + s,
// from the FP32 copy of the operands
template <class C>
__device__ __forceinline__ void face_g(const DevBlock &B, int64_t nl, int d, int64_t s, float *g) {
  constexpr int NV = C::nv;
  float kx, ky, kz;
  fp32::inviscid_face<C>(B.f32, B.G.size, nl, d, s, g, kx, ky, kz);
  OSTC_UNROLL for (int l = 0; l < NV; ++l) g[l] = -g[l];
  if (cP.viscous_order != 0)
    fp32::viscous_face_add<C>(B.f32, B.G.size, B.G.sx, B.G.sxy, nl, d, s, kx, ky, kz, g);
}

// The FP32 copy of the operands of the direction passes, over every point of
// layout G: the fields that change every step (after the source stage, which
// writes mu_t and lambda_t; blockIdx.y: block) ...
template <class C>
__global__ void __launch_bounds__(256) k_pack32(const DevBlock *__restrict__ blks) {
  using Q = fp32::Quad;
  const DevBlock &B = blks[blockIdx.y];
  const int64_t sz = B.G.size;
  float4 *f = B.f32;
  for (int64_t n = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; n < sz;
       n += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    // all loads, then all stores (a store would otherwise hold back the
    // loads after it: the compiler cannot rule out that they overlap)
    float v[4 * Q::n_dynamic];
    auto bv = [&](int l) { return fp32::ldf(B.bv + l * sz + n); };
    auto sv = [&](int l) { return fp32::ldf(B.sv + l * sz + n); };
    OSTC_UNROLL for (int l = 0; l < 4; ++l) {
      v[4 * Q::rho_vel + l] = bv(l);
      v[4 * Q::y0 + l] = sv(l);
      v[4 * Q::y4 + l] = sv(4 + l);
      v[4 * Q::d0 + l] = fp32::ldf(B.rho_d + l * sz + n);
      v[4 * Q::d4 + l] = fp32::ldf(B.rho_d + (4 + l) * sz + n);
    }
    v[4 * Q::p_t_turb] = bv(4);
    v[4 * Q::p_t_turb + 1] = bv(5);
    v[4 * Q::p_t_turb + 2] = sv(C::ns);
    v[4 * Q::p_t_turb + 3] = sv(C::ns + 1);
    v[4 * Q::y8_mu] = sv(8);
    v[4 * Q::y8_mu + 1] = fp32::ldf(B.mul + n);
    v[4 * Q::y8_mu + 2] = fp32::ldf(B.mut + n);
    v[4 * Q::y8_mu + 3] = fp32::ldf(B.cond + n);
    v[4 * Q::misc] = fp32::ldf(B.turb_cond + n);
    v[4 * Q::misc + 1] = fp32::ldf(B.acoustic + n);
    v[4 * Q::misc + 2] = fp32::ldf(B.gamma + n);
    v[4 * Q::misc + 3] = fp32::ldf(B.rho_d + 8 * sz + n);
    OSTC_UNROLL for (int q = 0; q < Q::n_dynamic; ++q)
      f[q * sz + n] = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
  }
}

// ... and the geometry, which changes only when the grid is set.
template <class C>
__global__ void __launch_bounds__(256) k_pack32_static(const DevBlock *__restrict__ blks, int b) {
  using Q = fp32::Quad;
  const DevBlock &B = blks[b];
  const int64_t sz = B.G.size;
  for (int64_t n = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; n < sz;
       n += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const float extra[3] = {static_cast<float>(B.jac[n]), B.wall_dist ? static_cast<float>(B.wall_dist[n]) : 0.f, 0.f};
    OSTC_UNROLL for (int d = 0; d < 3; ++d) {
      auto m = [&](int q) { return static_cast<float>(B.metric[(3 * d + q) * sz + n]); };
      B.f32[(Q::metric + d) * sz + n] = make_float4(m(0), m(1), m(2), extra[d]);
    }
  }
}

template <class C, int MINB>
__global__ void __launch_bounds__(kCta, MINB) k_flux_x(const DevBlock *__restrict__ blks, Tiles T) {
  constexpr int NV = C::nv;
  int b, t0, t1, t2;
  dir_tile(T, b, t0, t1, t2);
  const DevBlock &B = blks[b];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int j = t1 * kTY + warp, k = t2;
  if (j >= B.my) return;  // the whole warp
  const int f = t0 * kXSeg - 1 + lane;  // the face between cells f and f + 1
  const bool face = f < B.mx;
  float g[NV];
  if (face) {
    face_g<C>(B, B.G.at(f, j, k), 0, 1, g);
  } else {
    OSTC_UNROLL for (int l = 0; l < NV; ++l) g[l] = 0;
  }
  const bool cell = face && lane > 0;
  const int64_t szd = B.D.size;
  const int64_t nd = cell ? B.D.at(f, j, k) : 0;
  OSTC_UNROLL for (int l = 0; l < NV; ++l) {
    const float gm = __shfl_up_sync(0xffffffffu, g[l], 1);
    if (cell) B.dq[l * szd + nd] += static_cast<double>(g[l] - gm);
  }
  if (cell) local_time_step_q<C>(B, B.f32, f, j, k, B.G.at(f, j, k), nd);
}

template <class C, int D, int MINB>
__global__ void __launch_bounds__(kCta, MINB) k_flux_march(const DevBlock *__restrict__ blks, Tiles T, int march) {
  constexpr int NV = C::nv;
  static_assert(D == 1 || D == 2, "march passes run along y or z");
  int b, t0, t1, t2;
  dir_tile(T, b, t0, t1, t2);
  const DevBlock &B = blks[b];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int i = t0 * kTX + lane, o = t1 * kTY + warp;  // o: k for the y pass, j for the z pass
  if (i >= B.mx || o >= (D == 1 ? B.mz : B.my)) return;
  const int m = D == 1 ? B.my : B.mz;
  const int c0 = t2 * march, c1 = min(c0 + march, m);
  const int64_t s = D == 1 ? B.G.sx : B.G.sxy;
  const int64_t n0 = D == 1 ? B.G.at(i, c0, o) : B.G.at(i, o, c0);
  const int64_t sd = D == 1 ? B.D.sx : B.D.sxy;
  const int64_t nd0 = D == 1 ? B.D.at(i, c0, o) : B.D.at(i, o, c0);
  const int64_t szd = B.D.size;
  float gm[NV];
  face_g<C>(B, n0 - s, D, s, gm);  // face c0 - 1/2
#pragma unroll 1
  for (int c = c0; c < c1; ++c) {
    float g[NV];
    face_g<C>(B, n0 + (c - c0) * s, D, s, g);  // face c + 1/2
    const int64_t nd = nd0 + (c - c0) * sd;
    OSTC_UNROLL for (int l = 0; l < NV; ++l) {
      B.dq[l * szd + nd] += static_cast<double>(g[l] - gm[l]);
      gm[l] = g[l];
    }
  }
}

// The terms of a cell's flux-Jacobian product that no direction enters
// (compute_jacobian_times_dq, src/DPLURHPP.cuh:78-125), kept per cell so that a
// sweep does not sum over the species for each of the six neighbours that take
// them: once per step the total enthalpy h (beside the spectral radii, radii32)
// and the weights gamma R T / W_l - (gamma - 1) h_l of the species increments
// in the pressure term, and per sweep the pressure term itself, by the kernel
// that writes the increments.
template <class C>
__device__ __forceinline__ float pressure_term32(const DevBlock &B, int64_t n, int64_t nd, const float *d) {
  const int64_t szd = B.D.size;
  const float4 s = __ldg(B.f32 + fp32::Quad::rho_vel * B.G.size + n);
  const float gamma = __ldg(&(B.f32 + fp32::Quad::misc * B.G.size + n)->z);
  float p = (gamma - 1) * (0.5f * (s.y * s.y + s.z * s.z + s.w * s.w) * d[0] - s.y * d[1] - s.z * d[2] - s.w * d[3] + d[4]);
  OSTC_UNROLL for (int l = 0; l < C::ns; ++l) p += B.weight32[l * szd + nd] * d[5 + l];
  return p;
}

// increments of a cell in buffer q of the sweeps: four quads in the order of
// the flux variables
template <class C>
__device__ __forceinline__ void store_increments32(float4 *f, int64_t szd, int64_t nd, const float *d) {
  static_assert(C::nv == 16, "four quads");
  OSTC_UNROLL for (int q = 0; q < 4; ++q) f[q * szd + nd] = make_float4(d[4 * q], d[4 * q + 1], d[4 * q + 2], d[4 * q + 3]);
}
template <class C>
__device__ __forceinline__ void load_increments32(const float4 *__restrict__ f, int64_t szd, int64_t nd, float *d) {
  OSTC_UNROLL for (int q = 0; q < 4; ++q) {
    const float4 v = __ldg(f + q * szd + nd);
    d[4 * q] = v.x;
    d[4 * q + 1] = v.y;
    d[4 * q + 2] = v.z;
    d[4 * q + 3] = v.w;
  }
}

// of dq0, by k_sweep_terms
template <class C>
__device__ __forceinline__ void sweep_terms32(const DevBlock &B, int64_t n, int64_t nd) {
  constexpr int NS = C::ns, NV = C::nv;
  const int64_t sz = B.G.size, szd = B.D.size;
  const float4 s = __ldg(B.f32 + fp32::Quad::rho_vel * sz + n);
  const double t = ld(B.bv + 5 * sz + n), gamma = ld(B.gamma + n);
  float d[NV];
  load_increments32<C>(B.dqf[0], szd, nd, d);
  double hk[NS], h = 0.5 * (s.y * s.y + s.z * s.z + s.w * s.w);
  enthalpy<NS>(t, hk);
  const float g1 = static_cast<float>(gamma) - 1;
  float p = g1 * (0.5f * (s.y * s.y + s.z * s.z + s.w * s.w) * d[0] - s.y * d[1] - s.z * d[2] - s.w * d[3] + d[4]);
  float w[NS];
  OSTC_UNROLL for (int l = 0; l < NS; ++l) {
    h += ld(B.sv + l * sz + n) * hk[l];
    w[l] = static_cast<float>(gamma * t * cP.ru_mw[l] - (gamma - 1) * hk[l]);
    p += w[l] * d[5 + l];
  }
  const float4 radii = make_float4(static_cast<float>(ld(B.inv_spec + nd)), static_cast<float>(ld(B.inv_spec + szd + nd)),
                                   static_cast<float>(ld(B.inv_spec + 2 * szd + nd)), static_cast<float>(h));
  OSTC_UNROLL for (int l = 0; l < NS; ++l) B.weight32[l * szd + nd] = w[l];
  B.radii32[nd] = radii;
  B.terms32[nd] = p;
}

// EPI solve of a DPLUR sweep with the stored factors of the leading NA x NA
// block; the trailing species have the single pivot diag, so their solve is
// rhs / diag, the operation the full factors would do for them.
template <int NS, int NA>
__device__ __forceinline__ void epi_solve_block(const DevBlock &B, int64_t nz, int64_t sz0, double diag,
                                                double *rhs) {
  int piv[NA];
  OSTC_UNROLL for (int q = 0; q < NA; ++q) piv[q] = B.lu_piv[q * sz0 + nz];
  lu_solve_g<NA>(B.chem_jac + nz, sz0, piv, rhs);
  OSTC_UNROLL for (int l = NA; l < NS; ++l) rhs[l] /= diag;
}

// DPLUR sweep with FP32 flux-Jacobian products; the update of the point
// implicit blocks (EPI: stored LU factors) in FP64.  The increments are FP32
// arrays: reads dqf[in_sel] (neighbours) and dqf[0] (dq0), writes
// dqf[out_sel], or the FP64 dq when out_sel < 0 (the last sweep).
template <class C>
__global__ void __launch_bounds__(kCta, 4) k_sweep_mx(const DevBlock *__restrict__ blks, Tiles T, int in_sel,
                                                      int out_sel) {
  constexpr int NS = C::ns, NV = C::nv;
  int b, i, j, k;
  if (!tile_cell<kTX, kTY, kTZ>(T, b, i, j, k, blks)) return;
  const DevBlock &B = blks[b];
  using Q = fp32::Quad;
  const float4 *dqin = B.dqf[in_sel];
  const int64_t sz = B.G.size, szd = B.D.size, sz0 = B.Z.size;
  const int64_t n = B.G.at(i, j, k), nd = B.D.at(i, j, k), nz = B.Z.at(i, j, k);
  const int64_t sx = B.G.sx, sxy = B.G.sxy, dsx = B.D.sx, dsxy = B.D.sxy;
  const float4 *f = B.f32;
  float tot[NV];
  OSTC_UNROLL for (int l = 0; l < NV; ++l) tot[l] = 0;
#pragma unroll 1
  for (int q = 0; q < 6; ++q) {
    const int dir = q < 3 ? q : q - 3;
    const bool plus = q >= 3;
    const int id = dir == 0 ? i : (dir == 1 ? j : k);
    const int ext = dir == 0 ? B.mx : (dir == 1 ? B.my : B.mz);
    if (plus ? id == ext - 1 : id == 0) continue;
    const int64_t gs = dir == 0 ? 1 : (dir == 1 ? sx : sxy), ds = dir == 0 ? 1 : (dir == 1 ? dsx : dsxy);
    const int64_t on = plus ? n + gs : n - gs, od = plus ? nd + ds : nd - ds;
    // compute_jacobian_times_dq (src/DPLURHPP.cuh:78-125) at the neighbour,
    // its state from the step's FP32 copy (k_pack32; unchanged until the update)
    const float4 xi = __ldg(f + (Q::metric + dir) * sz + on), vel = __ldg(f + Q::rho_vel * sz + on);
    const float4 y0 = __ldg(f + Q::y0 * sz + on), y4 = __ldg(f + Q::y4 * sz + on);
    const float4 turb = __ldg(f + Q::p_t_turb * sz + on), radii = __ldg(B.radii32 + od);
    const float y8 = __ldg(&(f + Q::y8_mu * sz + on)->x);
    const float p = __ldg(B.terms32 + in_sel * szd + od), h = radii.w;
    float d[NV];
    load_increments32<C>(dqin, szd, od, d);
    const float sr = dir == 0 ? radii.x : (dir == 1 ? radii.y : radii.z);
    const float U = xi.x * vel.y + xi.y * vel.z + xi.z * vel.w;
    const float b1 = xi.x * d[1] + xi.y * d[2] + xi.z * d[3] - U * d[0];
    const float sg = plus ? -0.5f : 0.5f;
    const float lmd1 = sg * (U + (plus ? -sr : sr)), c1 = sg * b1, cp = sg * p;
    tot[0] += c1 + lmd1 * d[0];
    tot[1] += vel.y * c1 + xi.x * cp + lmd1 * d[1];
    tot[2] += vel.z * c1 + xi.y * cp + lmd1 * d[2];
    tot[3] += vel.w * c1 + xi.z * cp + lmd1 * d[3];
    tot[4] += h * c1 + U * cp + lmd1 * d[4];
    const float y[NV - 5] = {y0.x, y0.y, y0.z, y0.w, y4.x, y4.y, y4.z, y4.w, y8, turb.z, turb.w};
    OSTC_UNROLL for (int l = 0; l < C::nsc; ++l) tot[5 + l] += lmd1 * d[5 + l] + y[l] * c1;
  }
  const float4 rad = __ldg(B.radii32 + nd);
  float dq0[NV];
  load_increments32<C>(B.dqf[0], szd, nd, dq0);
  const double dt = B.dt_local[nz];
  const double diag =
      1 + dt * (static_cast<double>(rad.x) + static_cast<double>(rad.y) + static_cast<double>(rad.z));
  double out[NV];
  if constexpr (C::mix != 2) {
    OSTC_UNROLL for (int l = 0; l < 5 + NS; ++l) out[l] = static_cast<double>(dq0[l]) + dt * tot[l] / diag;
  } else {
    OSTC_UNROLL for (int l = 0; l < 5; ++l) out[l] = static_cast<double>(dq0[l]) + dt * tot[l] / diag;
    const int method = cP.chem_src_method;
    if (B.chem_quiet && B.chem_quiet[nz]) {
      // chemically quiet: the stored factors would be diag I
      OSTC_UNROLL for (int l = 0; l < NS; ++l) out[5 + l] = static_cast<double>(dq0[5 + l]) + dt * tot[5 + l] / diag;
    } else if (method == 1) {
      double rhs[NS];
      OSTC_UNROLL for (int l = 0; l < NS; ++l) rhs[l] = static_cast<double>(tot[5 + l]) * dt;
      if (cP.na == NS - 1)
        epi_solve_block<NS, NS - 1>(B, nz, sz0, diag, rhs);
      else
        epi_solve_block<NS, NS>(B, nz, sz0, diag, rhs);
      OSTC_UNROLL for (int l = 0; l < NS; ++l) out[5 + l] = static_cast<double>(dq0[5 + l]) + rhs[l];
    } else if (method == 2) {
      OSTC_UNROLL for (int l = 0; l < NS; ++l)
        out[5 + l] = static_cast<double>(dq0[5 + l]) + dt * tot[5 + l] / (diag - dt * B.chem_jac[l * sz0 + nz]);
    } else {
      OSTC_UNROLL for (int l = 0; l < NS; ++l) out[5 + l] = static_cast<double>(dq0[5 + l]) + dt * tot[5 + l] / diag;
    }
  }
  if constexpr (C::turb) {
    if (cP.turb_implicit == 1) {
      out[NS + 5] = static_cast<double>(dq0[NS + 5]) + dt * tot[5 + NS] / (diag - dt * B.turb_src_jac[nz]);
      out[NS + 6] = static_cast<double>(dq0[NS + 6]) + dt * tot[6 + NS] / (diag - dt * B.turb_src_jac[sz0 + nz]);
    } else {
      out[NS + 5] = static_cast<double>(dq0[NS + 5]) + dt * tot[5 + NS] / diag;
      out[NS + 6] = static_cast<double>(dq0[NS + 6]) + dt * tot[6 + NS] / diag;
    }
  }
  if (out_sel < 0) {
    OSTC_UNROLL for (int l = 0; l < NV; ++l) B.dq[l * szd + nd] = out[l];
  } else {
    float d[NV];
    OSTC_UNROLL for (int l = 0; l < NV; ++l) d[l] = static_cast<float>(out[l]);
    B.terms32[out_sel * szd + nd] = pressure_term32<C>(B, n, nd, d);
    store_increments32<C>(B.dqf[out_sel], szd, nd, d);
  }
}

// Thermodynamic and transport properties in FP32 (update_physical_properties).
template <class C>
__global__ void __launch_bounds__(kCta) k_props_mx(const DevBlock *__restrict__ blks, Tiles T,
                                                   unsigned int *bad_count) {
  if (blockIdx.x == 0 && threadIdx.x + threadIdx.y == 0) *bad_count = 0;
  constexpr int NS = C::ns;
  using fp32::ldf;
  int b, i, j, k;
  if (!tile_cell<kTX, kTY, kTZ>(T, b, i, j, k, blks)) return;
  const DevBlock &B = blks[b];
  const int64_t n = B.G.at(i, j, k), sz = B.G.size;
  const float t = ldf(B.bv + 5 * sz + n);
  if constexpr (C::mix != 0) {
    float cp[NS], Y[NS];
    const float vel = ldf(B.vel + n);  // read before the first store, which would hold it back
    fp32::thermo<NS, false, true>(t, nullptr, cp);
    float mw_inv = 0, cp_tot = 0, cv = 0;
    OSTC_UNROLL for (int l = 0; l < NS; ++l) {
      Y[l] = ldf(B.sv + l * sz + n);
      mw_inv += Y[l] * cF.mw_inv[l];
      cp_tot += Y[l] * cp[l];
      cv += Y[l] * (cp[l] - cF.ru_mw[l]);
    }
    const float gamma = __fdividef(cp_tot, cv);
    B.cp[n] = cp_tot;
    B.gamma[n] = gamma;
    const float a = sqrtf(gamma * fp32::kRu * t * mw_inv);
    B.acoustic[n] = a;
    const float mw = 1.f / mw_inv;
    float X[NS], vis[NS], rs[NS], sq[NS];  // sq = sqrt(mu_k), rs = 1 / sq
    const float st = sqrtf(t);
    OSTC_UNROLL for (int l = 0; l < NS; ++l) {
      X[l] = Y[l] * mw * cF.mw_inv[l];
      const float t_dl = t * cF.lj_inv[l];
      // the hardware-approximate power and quotients (errors of a few ulp)
      const float r = __fdividef(1.f, t_dl + 0.5f);
      const float ci = 1.147f * __powf(t_dl, -0.145f) + r * r;
      vis[l] = __fdividef(cF.vis_coeff[l] * st, ci);
      rs[l] = rsqrtf(vis[l]);
      sq[l] = vis[l] * rs[l];
    }
    float viscosity = 0, conductivity = 0;
    OSTC_UNROLL for (int m = 0; m < NS; ++m) {
      float vt = 0;
      OSTC_UNROLL for (int q = 0; q < NS; ++q) {
        float phi = 1.f;
        if (m != q) {  // Wilke's phi_mq with sqrt(mu_m / mu_q) as sqrt(mu_m) / sqrt(mu_q)
          const float num = 1 + sq[m] * rs[q] * cF.wq[m * NS + q];
          phi = num * num * cF.w8[m * NS + q];
        }
        vt += phi * X[q];
      }
      viscosity += __fdividef(vis[m] * X[m], vt);
      const float lambda = vis[m] * (cp[m] + 1.25f * cF.ru_mw[m]);
      conductivity += __fdividef(lambda * X[m], 1.065f * vt - 0.065f * X[m]);
    }
    B.mul[n] = viscosity;
    B.cond[n] = conductivity;
    OSTC_UNROLL for (int l = 0; l < NS; ++l) {
      const float dd = fabsf(X[l] - 1) < 1e-3f ? viscosity / cF.Sc : (1 - Y[l]) * viscosity / ((1 - X[l]) * cF.Sc);
      B.rho_d[l * sz + n] = dd;
    }
    B.mach[n] = vel / a;
  } else {
    const float a = sqrtf(1.4f * fp32::kRu / static_cast<float>(kDMwAir) * t);
    B.acoustic[n] = a;
    const float mul = 1.716e-5f * powf(t / 273.f, 1.5f) * (273.f + 111.f) / (t + 111.f);
    B.mul[n] = mul;
    B.cond[n] = mul * static_cast<float>(kDGammaAir * kDR_u / kDMwAir / (kDGammaAir - 1)) / cF.Pr;
    B.mach[n] = ldf(B.vel + n) / a;
  }
}

}  // namespace ostc
