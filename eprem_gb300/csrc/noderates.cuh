// noderates.cuh -- a node's focusing and change rates and sub-cycle counts,
// fixed for one updateEnergeticParticles call (AdiabaticFocusing
// src/energeticParticles.c:1582-1670, AdiabaticChange :861-950).
//
// The counts are ceil(dt / (0.9 d / vmax)) with vmax the largest face or cell
// speed of the node, formed with the reference's expressions without fused
// multiply-adds so that the integers match.  A maximum does not depend on the
// order, and only the cells near it need the exact expressions: the speeds are
// first taken in float, and those within 1e-4 of the float scale of the
// largest one are formed again in FP64 (a speed's float rounding is below
// 1e-6 of that scale).  One thread per node: FP64 runs at 1/64 of the float
// rate here, so a node's 2 M exact face speeds are what there is to save.
#pragma once
#include "common.cuh"

namespace eprem {
namespace rates {

__device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double sub(double a, double b) { return __dsub_rn(a, b); }

// Focusing cell velocity at mu (src/energeticParticles.c:1620-1627).
__device__ __forceinline__ double focus_vel(double mu, double a, double b) {
  return mul(mul(0.5, sub(1.0, mul(mu, mu))), add(a, mul(mu, b)));
}
__device__ __forceinline__ double focus_face(const RunView &r, int m, double a, double b) {
  return fabs(mul(0.5, add(focus_vel(r.mugrid[m], a, b), focus_vel(r.mugrid[m - 1], a, b))));
}
// Change velocity at mu (:873-890).
__device__ __forceinline__ double change_vel(double mu, double vi, double dupar, double dlnb,
                                             double dlnn, double cool) {
  const double mu2 = mul(mu, mu);
  const double b = add(mul(mu2, sub(dlnn, dlnb)), mul(mul(0.5, sub(1.0, mu2)), dlnb));
  return fabs(mul(cool, add(mul(mul(-mu, dupar), vi), b)));
}

// Whether float holds speeds of this scale with room on both sides.
__device__ __forceinline__ bool float_scale(double s) { return s > 1e-25 && s < 1e25; }

// Largest |face speed| over the faces for one a; NaN faces take no part, as the
// reference's fabs(v) > max passes over them.
__device__ __forceinline__ double focus_max(const RunView &r, double a, double b) {
  const double scale = fabs(a) + fabs(b);
  double best = 0.0;
  if (!float_scale(scale)) {
    for (int m = 1; m < r.M; m++) best = fmax(best, focus_face(r, m, a, b));
    return best;
  }
  const float af = (float)a, bf = (float)b;
  auto face = [&](int m) {
    const float u = r.mugrid32[m], v = r.mugrid32[m - 1];
    return fabsf((1.f - u * u) * (af + u * bf) + (1.f - v * v) * (af + v * bf));
  };
  float top = 0.f;
  for (int m = 1; m < r.M; m++) top = fmaxf(top, face(m));
  const float near = top - 1e-4f * (float)scale;
  for (int m = 1; m < r.M; m++)
    if (face(m) >= near) best = fmax(best, focus_face(r, m, a, b));
  return best;
}

// Largest |change speed| over mu at one energy's 1/v.
__device__ __forceinline__ double change_max(const RunView &r, double vi, double dupar,
                                             double dlnb, double dlnn, double cool) {
  const double scale = fabs(dupar) * vi + fabs(dlnn) + fabs(dlnb);
  double best = 0.0;
  if (!float_scale(scale)) {
    for (int m = 0; m < r.M; m++)
      best = fmax(best, change_vel(r.mugrid[m], vi, dupar, dlnb, dlnn, cool));
    return best;
  }
  const float d = (float)(dupar * vi), nb = (float)(dlnn - dlnb), hb = (float)(0.5 * dlnb);
  const float c = (float)fabs(cool);
  auto vel = [&](int m) {
    const float u = r.mugrid32[m], u2 = u * u;
    return fabsf(u2 * nb + (1.f - u2) * hb - u * d) * c;
  };
  float top = 0.f;
  for (int m = 0; m < r.M; m++) top = fmaxf(top, vel(m));
  const float near = top - 1e-4f * ((float)scale * c);
  for (int m = 0; m < r.M; m++)
    if (vel(m) >= near) best = fmax(best, change_vel(r.mugrid[m], vi, dupar, dlnb, dlnn, cool));
  return best;
}

struct NodeRates {
  double dupar, dlnb, dlnn;  // per unit time
  double b, dlnbds, cool;
  int ns_f, ns_c;            // sub-cycles (0 where nothing moves)
};

// Rates and counts of node g (k: its place on the stream; 0, the spawn node,
// takes no sub-cycles).  ds, bplus, bminus: updateStreamValues' results.
__device__ __forceinline__ NodeRates node_rates(const RunView &r, size_t g, int k, double ds,
                                                double bplus, double bminus) {
  NodeRates o{};
  const double dt = r.dt, full = r.dt_full;
  const bool ok = k != 0;
  o.dupar = node_field(r, EPREM_NODE_DUPAR)[g] / full;
  o.dlnb = node_field(r, EPREM_NODE_DLNB)[g] / full;
  o.dlnn = node_field(r, EPREM_NODE_DLNN)[g] / full;
  if (r.use_focus) {
    o.b = sub(mul(2.0, o.dlnn), mul(3.0, o.dlnb));
    o.dlnbds = (bplus == 0.0 || bminus == 0.0)
                   ? 0.0
                   : (log(bplus) - log(bminus)) / add(mul(2.0, ds), DBL_MIN);
    // the speed is linear in a, so its maximum over the energies lies on the
    // rows of the smallest and largest a
    double amin = DBL_MAX, amax = -DBL_MAX;
    auto exact = [&](int e) {
      const double a = sub(mul(-r.ec[e].vgrid, o.dlnbds), mul(r.ec[e].two_vi, o.dupar));
      amin = a < amin ? a : amin;
      amax = a > amax ? a : amax;
    };
    // (1 / v is largest at the first energy, v below 1)
    const double scale = fabs(o.dlnbds) + r.ec[0].two_vi * fabs(o.dupar);
    if (float_scale(scale)) {
      const float d = (float)o.dlnbds, u = 2.f * (float)o.dupar;
      auto rough = [&](int e) { return -r.ec[e].v32 * d - r.ec[e].vi32 * u; };
      float lo = FLT_MAX, hi = -FLT_MAX;
      for (int e = 0; e < r.E; e++) {
        lo = fminf(lo, rough(e));
        hi = fmaxf(hi, rough(e));
      }
      const float near = 1e-4f * (float)scale;
      for (int e = 0; e < r.E; e++)
        if (rough(e) <= lo + near || rough(e) >= hi - near) exact(e);
    } else {
      for (int e = 0; e < r.E; e++) exact(e);
    }
    double vmax = 0.0;
    if (amin <= amax) vmax = fmax(focus_max(r, amin, o.b), focus_max(r, amax, o.b));
    const double nsub = ceil(dt / (mul(0.9, r.dmu) / vmax));
    if (nsub <= (double)r.max_subcycles)
      o.ns_f = ok ? (int)nsub : 0;
    else if (ok)
      set_error(r, EPREM_GPU_ERR_SUBCYCLES, 2, (int)(g / r.N), k, -1, -1);
  }
  if (r.use_change) {
    o.cool = (o.dlnn < 0) ? 1.0 - r.damp_cooling : 1.0;
    // linear in 1/v, which is monotonic in energy: the first and last rows
    const double vmax =
        fmax(change_max(r, r.ec[0].vgrid_i, o.dupar, o.dlnb, o.dlnn, o.cool),
             change_max(r, r.ec[r.E - 1].vgrid_i, o.dupar, o.dlnb, o.dlnn, o.cool));
    const double nsub = ceil(dt / (mul(0.9, r.dlnp) / vmax));
    if (nsub <= (double)r.max_subcycles)
      o.ns_c = ok ? (int)nsub : 0;
    else if (ok)
      set_error(r, EPREM_GPU_ERR_SUBCYCLES, 3, (int)(g / r.N), k, -1, -1);
  }
  return o;
}

// The log statistics of a warp's nodes (every lane takes part; lanes without a
// node pass zeros): sub-cycle maxima and cell sub-cycles of all sub-steps.
__device__ __forceinline__ void count_nodes(const RunView &r, int ns_f, int ns_c) {
  constexpr unsigned FULL = 0xffffffffu;
  const unsigned long long cells = (unsigned long long)r.E * r.M * r.num_ep_steps;
  const int mf = __reduce_max_sync(FULL, ns_f), mc = __reduce_max_sync(FULL, ns_c);
  unsigned long long sf = ns_f, sc = ns_c;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    sf += __shfl_xor_sync(FULL, sf, o);
    sc += __shfl_xor_sync(FULL, sc, o);
  }
  if ((threadIdx.x & 31) == 0) {
    if (mf) atomicMax(&r.status->max_focus, mf);
    if (mc) atomicMax(&r.status->max_change, mc);
    if (sf) atomicAdd(&r.status->focus_cs, sf * cells);
    if (sc) atomicAdd(&r.status->change_cs, sc * cells);
  }
}

}  // namespace rates
}  // namespace eprem
