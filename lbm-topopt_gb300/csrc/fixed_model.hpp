// fixed_model.hpp -- the constants of a model's fixed-point collision
// (lbm_fixed.cuh), computed on the host once per handle.
#pragma once

#include <climits>
#include <cmath>

#include "../../include/lbmgpu.h"
#include "lbm_device.cuh"
#include "lbm_ops.h"

namespace lbm {

inline bool velocity_objective(const lbm_config& c) {
  return c.objective == LBM_OBJ_THROUGH_FLOW || c.objective == LBM_OBJ_OUTFLOW ||
         c.objective == LBM_OBJ_HEAT_FLUX;
}

// v * 2^bits as an even unsigned constant; clears ok where it does not fit.
inline unsigned long long fixed_constant(long double v, int bits, bool& ok) {
  const long double x = ldexpl(v, bits);
  if (!(x >= 0.L && x < 18446744073709551614.L)) {
    ok = false;
    return 0;
  }
  return (unsigned long long)(x / 2 + 0.5L) * 2;
}

// The constants of the model's collision in fixed point (lbm_fixed.cuh), with
// ok set where the model has such a form and its constants fit.
inline FixedModel fixed_model(const lbm_config& c) {
  FixedModel m = {};
  if (c.storage != LBM_STORE_FP64) return m;
  bool ok = true;
  const long double om = c.omega;
  if (c.lattice == LBM_D3Q19 && c.collision == LBM_MRT) {
    const long double s1 = c.mrt[0], s2 = c.mrt[1], s4 = c.mrt[2], s10 = c.mrt[3], s16 = c.mrt[4];
    const long double v[9] = {s1 / 63, s2 * 2 / 63, s4 / 12, om / 18, s10 / 36,
                              om / 6,  s10 / 12,    om / 2,  s16 / 4};
    for (int i = 0; i < 9; ++i) m.c[i] = fixed_constant(v[i], 64, ok);
    const double we3 = c.mrt[5] - 3., wej = c.mrt[6], wxx = c.mrt[7];
    m.wej = fixed_constant(fabsl((long double)wej) / 4, 62, ok);
    m.wxx = fixed_constant(fabsl((long double)wxx), 62, ok);
    m.we3c = fixed_constant(fabsl((long double)we3) / 4, 62, ok);
    m.wej_neg = wej < 0. ? -1 : 0;
    m.wxx_neg = wxx < 0. ? -1 : 0;
    m.we3_neg = we3 < 0. ? -1 : 0;
    m.we3 = we3 != 0. ? 1 : 0;
    // every rate at most 2 and the eps row's bound (1.44 + |wej|/4 j^2 +
    // |we - 3|/4 rho with j^2 < 1.2, rho < 2.4) below 4
    for (int i = 0; i < 5; ++i) ok = ok && c.mrt[i] >= 0. && c.mrt[i] <= 2.;
    ok = ok && fabs(wxx) <= 1. && 1.44 + 0.3 * fabs(wej) + 0.6 * fabs(we3) < 3.9;
  } else if (c.collision == LBM_BGK) {
    m.c[0] = fixed_constant(om / 2, 64, ok);
    m.c[1] = fixed_constant(om / 6, 64, ok);
  } else if (c.lattice == LBM_D2Q9 && c.collision == LBM_MRT) {
    const long double v[4] = {(long double)c.mrt[0] / 36, (long double)c.mrt[1] / 12,
                              (long double)c.mrt[2] / 6, om / 2};
    for (int i = 0; i < 4; ++i) m.c[i] = fixed_constant(v[i], 64, ok);
    for (int i = 0; i < 3; ++i) ok = ok && c.mrt[i] >= 0. && c.mrt[i] <= 2.;
  } else {
    ok = false;
  }
  // (9/2) nu omega^2 = (3/2) omega (1 - omega/2), at most 3/4
  m.cv = fixed_constant(1.5L * om * (1 - om / 2), 64, ok);
  const long double w = frexpl(fabsl((long double)c.obj_weight), &m.w_exp);
  bool weight = true;
  m.w = fixed_constant(w, 64, weight);
  m.w_neg = c.obj_weight < 0. ? -1 : 0;
  if (!weight) ok = ok && c.objective != LBM_OBJ_DISSIPATION;
  // The porosity plane holds imult in steps of 2^-64 (KParams::im), where imult
  // itself, one minus a quotient, is off by some 2^-55 of the scale.  With scales
  // below 2^-12 the steps are the larger (value of the dissipation in a flow
  // without stresses, u = 0.08, against extended precision: scale 2^-11 1.6e-22,
  // FP64 4.1e-22; 1e-4 2.9e-22 and 8.4e-23).
  if (c.objective == LBM_OBJ_DISSIPATION && c.interp_scale != 0. &&
      fabs(c.interp_scale) < 0x1p-11)
    ok = false;
  m.ok = ok ? 1 : 0;
  return m;
}

// Steps t whose state f_t keeps the FP64 operators, forward and reverse: a
// velocity objective of a flow that is still at rest is nothing but rounding, and
// the FP64 operators' rounding is the reference's.  The rule is one of the model
// and of t alone, so that a sweep gives the same bits however it is cut into
// calls.  1.1 times what sound (1/sqrt(3) cells a step) takes from the nearest
// boundary that drives the flow to the cells that the objective averages over, and
// 30 for the front to rise.  (A heat flux sums over its box, where only the warm
// part counts: to the middle.)  By then the objective, summed with a weight of
// one, is above 1e-7 on pumps of 60x60 to 420x420 cells and above 1e-6 soon
// after, where the roundings of one step add 3e-16 (201x201 MRT: sound takes 164
// steps; 1e-15 after 115, 1e-7 after 153, 1e-5 after 199; kept to 211).
// J, its steps and dJ/dgamma of sweeps that end 1 to 300 steps later are within 4e-11
// of FP64 throughout or of fixed point throughout (pumps of 60x60 to 420x420, BGK and
// MRT; heat fluxes of 64x32 to 300x129).
// A 201x201 MRT step costs 21 / 49 us forward / reverse with the FP64 operators and
// 5.0 / 8.1 in fixed point.
// INT_MAX where no boundary drives the flow, 0 for the other objectives.
inline int flow_start_up(const lbm_config& c) {
  ObjectiveInfo oi;
  if (!velocity_objective(c) || !objective_info(c.objective, &oi)) return 0;
  double best = -1.;
  for (int k = 0; k < c.nbc; ++k) {
    const lbm_bc& b = c.bc[k];
    const bool velocity = b.kind == LBM_BC_VELOCITY || b.kind == LBM_BC_VELOCITY_STANDARD;
    const bool pressure = b.kind == LBM_BC_PRESSURE || b.kind == LBM_BC_PRESSURE_STANDARD;
    const bool drives = (velocity && (b.value != 0. || b.profile == LBM_PROFILE_TABLE)) ||
                        (pressure && (b.value != 1. || b.amp != 0. || b.profile == LBM_PROFILE_TABLE ||
                                      b.time_law != LBM_TIME_OFFSET_SINE));
    if (!drives) continue;
    for (int side = 0; side < 2; ++side) {
      if (!(oi.uses & (side ? kUsesOut : kUsesIn))) continue;
      const int* o = side ? c.obj_out : c.obj_in;
      double d2 = 0.;
      for (int a = 0; a < 3; ++a) {
        const int lo = o[2 * a] - b.box[2 * a + 1], hi = b.box[2 * a] - o[2 * a + 1];
        double gap = lo > hi ? lo : hi;
        if (c.objective == LBM_OBJ_HEAT_FLUX) {
          const double mid = 0.5 * (o[2 * a] + o[2 * a + 1]);
          gap = fmax(mid - b.box[2 * a + 1], b.box[2 * a] - mid);
        }
        if (gap > 0.) d2 += gap * gap;
      }
      if (best < 0. || d2 < best) best = d2;
    }
  }
  return best < 0. ? INT_MAX : (int)(1.1 * sqrt(3. * best)) + 30;
}

}  // namespace lbm
