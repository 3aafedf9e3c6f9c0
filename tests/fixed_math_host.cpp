// Host build of the fixed-point collisions (lbm-topopt_gb300/csrc/lbm_fixed.cuh)
// and of the FP64 operators they stand in for, for tests without a GPU.
// Test infrastructure only.
#include <cmath>
#include <cstdio>
#include <cstring>
#define __device__
#define __host__
#define __forceinline__ inline
#define __noinline__
#define __global__
#define __launch_bounds__(...)
#include <cuda_fp16.h>
#include <cuda_runtime.h>
struct lbm_dim3_stub { unsigned x = 0, y = 0, z = 0; };
static lbm_dim3_stub threadIdx, blockIdx, blockDim, gridDim;
template <class T> T __shfl_down_sync(unsigned, T v, int) { return v; }
inline int __any_sync(unsigned, int v) { return v; }
inline void __syncthreads() {}
inline void __threadfence() {}
inline unsigned atomicAdd(unsigned* p, unsigned v) { unsigned o = *p; *p += v; return o; }
inline double atomicAdd(double* p, double v) { double o = *p; *p += v; return o; }
inline unsigned __umulhi(unsigned a, unsigned b) { return (unsigned)(((unsigned long long)a * b) >> 32); }
inline float __uint_as_float(unsigned u) { float f; memcpy(&f, &u, 4); return f; }
inline unsigned __float_as_uint(float f) { unsigned u; memcpy(&u, &f, 4); return u; }
#include "../lbm-topopt_gb300/csrc/lbm_fixed.cuh"
#include "../lbm-topopt_gb300/csrc/fixed_model.hpp"

using namespace lbm;

namespace {
KParams params(const lbm_config* c) {
  KParams p;
  memset(&p, 0, sizeof(p));
  ModelParams<double>& d = p.md;
  d.omega = c->omega;
  for (int i = 0; i < 8; ++i) d.mrt[i] = c->mrt[i];
  d.pbb_scale = c->interp_scale;
  d.pbb_q = c->interp_q;
  d.diff = c->diffusivity;
  d.ramp_q = c->ramp_q;
  d.ramp_ck = c->ramp_ck;
  d.heat_rate = c->heat_rate;
  d.heat_T = c->heat_T;
  p.fix = fixed_model(*c);
  return p;
}

template <int LAT, int COLL>
int forward(const lbm_config* c, int n, const double* f, const double* g, double* fixed,
            double* fp64) {
  const KParams p = params(c);
  constexpr int Q = Lattice<LAT>::Q;
  if (!p.fix.ok) return -1;
  int taken = 0;
  for (int i = 0; i < n; ++i) {
    const double imult = 0.5 * (p.md.pbb_scale * bp(g[i], p.md.pbb_q));
    double a[Q], rho, jx, jy, jz;
    memcpy(a, f + i * Q, sizeof(a));
    flow_collide<LAT, COLL>(a, imult, rho, jx, jy, jz, p);
    memcpy(fp64 + i * Q, a, sizeof(a));
    fx::Window w;
    fx::i64 x[Q];
    static_for<Q>([&](auto K) {
      constexpr int q = decltype(K)::value;
      x[q] = w.template load<LAT, q>(f[i * Q + q]);
    });
    if (w.template ok<LAT>(x)) {
      fx::collide<LAT, COLL>(x, fx::Factor((fx::u64)(imult * 18446744073709551616.)), p.fix, a);
      ++taken;
    }
    memcpy(fixed + i * Q, a, sizeof(a));
  }
  return taken;
}

// Transposes at states f and output adjoints lo: (fixed, dgf) and (fp64, dgd),
// dg by imult.
template <int LAT, int COLL>
int transpose(const lbm_config* c, int n, const double* f, const double* g, const double* lo,
              double* fixed, double* dgf, double* fp64, double* dgd) {
  const KParams p = params(c);
  constexpr int Q = Lattice<LAT>::Q;
  if (!p.fix.ok) return -1;
  int taken = 0;
  for (int i = 0; i < n; ++i) {
    const double imult = 0.5 * (p.md.pbb_scale * bp(g[i], p.md.pbb_q));
    double a[Q];
    memcpy(a, lo + i * Q, sizeof(a));
    dgd[i] = 0.;
    flow_reverse<LAT, COLL>(f + i * Q, a, imult, 1., dgd[i], p);
    memcpy(fp64 + i * Q, a, sizeof(a));
    dgf[i] = dgd[i];
    fx::Window w;
    fx::i64 x[Q];
    static_for<Q>([&](auto K) {
      constexpr int q = decltype(K)::value;
      x[q] = w.template load<LAT, q>(f[i * Q + q]);
    });
    fx::Block b;
    b.template measure<Q>(lo + i * Q);
    if (b.zero) {
      memset(a, 0, sizeof(a));
      dgf[i] = 0.;
      ++taken;
    } else if (w.template ok<LAT>(x) && b.ok) {
      memcpy(a, lo + i * Q, sizeof(a));
      dgf[i] = fx::reverse<LAT, COLL>(x, a, b, fx::Factor((fx::u64)(imult * 18446744073709551616.)),
                                       p.fix, fx::Source2());
      ++taken;
    }
    memcpy(fixed + i * Q, a, sizeof(a));
  }
  return taken;
}

#define BY_MODEL(fn, ...)                                                       \
  do {                                                                          \
    if (c->lattice == LBM_D3Q19 && c->collision == LBM_MRT)                     \
      return fn<LAT_D3Q19, LBM_MRT>(__VA_ARGS__);                               \
    if (c->lattice == LBM_D2Q9 && c->collision == LBM_BGK)                      \
      return fn<LAT_D2Q9, LBM_BGK>(__VA_ARGS__);                                \
    if (c->lattice == LBM_D2Q9 && c->collision == LBM_MRT)                      \
      return fn<LAT_D2Q9, LBM_MRT>(__VA_ARGS__);                                \
    if (c->lattice == LBM_D3Q19 && c->collision == LBM_BGK)                     \
      return fn<LAT_D3Q19, LBM_BGK>(__VA_ARGS__);                               \
    return -1;                                                                  \
  } while (0)
}  // namespace

extern "C" {
// One collision of n cells in fixed point and in FP64; returns the cells that
// the fixed-point form took (-1: the model has none).
int fixed_forward(const lbm_config* c, int n, const double* f, const double* g, double* fixed,
                  double* fp64) {
  BY_MODEL(forward, c, n, f, g, fixed, fp64);
}
int fixed_reverse(const lbm_config* c, int n, const double* f, const double* g, const double* lo,
                  double* fixed, double* dgf, double* fp64, double* dgd) {
  BY_MODEL(transpose, c, n, f, g, lo, fixed, dgf, fp64, dgd);
}

// Temperature collision of n cells: flow populations f (n x 9), temperatures t
// (n x 5) and adjoints l (n x 5), om_T per cell.  out, lout: (fixed, FP64 in the
// order of thermal_collide / thermal_reverse without heating), n x 5 each;
// misc: n x 3 of the fixed-point adjoint's dx, dy, sum6.
int fixed_thermal(int n, const double* f, const double* t, const double* l, const double* om,
                  double* out, double* out64, double* lout, double* lout64, double* misc) {
  constexpr double W5[5] = {1. / 3., 1. / 6., 1. / 6., 1. / 6., 1. / 6.};
  constexpr int EX5[5] = {0, 0, -1, 0, 1}, EY5[5] = {0, -1, 0, 1, 0};
  for (int i = 0; i < n; ++i) {
    fx::Window w;
    fx::i64 x[9];
    static_for<9>([&](auto K) {
      constexpr int q = decltype(K)::value;
      x[q] = w.load<LAT_D2Q9_D2Q5, q>(f[i * 9 + q]);
    });
    if (!w.ok<LAT_D2Q9_D2Q5>(x)) return i;
    const fx::Pairs2 u(x);
    fx::ThermalBlock b, a;
    b.measure<5>(t + 5 * i);
    a.measure<5>(l + 5 * i);
    const fx::u64 om6 = (fx::u64)(om[i] * 3074457345618258602.7);
    memcpy(out + 5 * i, t + 5 * i, 40);
    memcpy(lout + 5 * i, l + 5 * i, 40);
    if (!b.zero) fx::thermal_collide(fx::Thermal(t + 5 * i, b, u.jx, u.jy), b, om6, out + 5 * i);
    if (!a.zero) {
      const fx::ThermalAdjoint r = fx::thermal_reverse(lout + 5 * i, a, u.jx, u.jy, om6);
      misc[3 * i] = r.dx;
      misc[3 * i + 1] = r.dy;
      misc[3 * i + 2] = r.sum6;
    }
    double rho, ux, uy;
    macros_d2q9(f + 9 * i, rho, ux, uy);
    const double* g = t + 5 * i;
    const double T = g[0] + g[1] + g[2] + g[3] + g[4];
    double TR = 0.;
    for (int k = 0; k < 5; ++k) {
      const double sc = EX5[k] * ux + EY5[k] * uy, eq = W5[k] * T * (1. + 3. * sc);
      out64[5 * i + k] = g[k] * (1. - om[i]) + om[i] * eq;
      TR += om[i] * l[5 * i + k] * W5[k] * (1. + 3. * sc);
    }
    for (int k = 0; k < 5; ++k) lout64[5 * i + k] = (1. - om[i]) * l[5 * i + k] + TR;
  }
  return n;
}

// Dissipation of n cells: value, source (n x 9) and derivative by imult (over
// the weight), in fixed point and (value, source) by the objective functor;
// scaled: the cells whose source fitted the adjoint's units.
int fixed_dissipation(const lbm_config* c, int n, const double* f, const double* g, double* val,
                      double* src, double* dim, double* val64, double* src64, int* scaled) {
  KParams p = params(c);
  p.md.obj_weight = c->obj_weight;
  *scaled = 0;
  p.md.cv_diss = 4.5 * ((1. / c->omega - 0.5) / 3.) * c->omega * c->omega;
  for (int i = 0; i < n; ++i) {
    const double imult = 0.5 * (p.md.pbb_scale * bp(g[i], p.md.pbb_q));
    const fx::u64 im = (fx::u64)(imult * 18446744073709551616.);
    fx::Window w;
    fx::i64 x[9];
    static_for<9>([&](auto K) {
      constexpr int q = decltype(K)::value;
      x[q] = w.load<LAT_D2Q9, q>(f[i * 9 + q]);
    });
    if (!w.ok<LAT_D2Q9>(x)) return i;
    val[i] = c->obj_weight * fx::energy(fx::dissipation2(x, im, p.fix.cv));
    for (int k = 0; k < 9; ++k) src[9 * i + k] = src64[9 * i + k] = 0.;
    const fx::Dissipation2 d(x, fx::Factor(im), p.fix.cv);
    dim[i] = d.dim;
    // in the units of an adjoint of size 2^e (e from -40 to 20 over the cells)
    // where it fits there, else in FP64
    fx::Block b;
    const double size[1] = {ldexp(1.3, i % 61 - 40)};
    b.measure<1>(size);
    const fx::Source2 r = d.scaled(p.fix, b);
    if (r.on) {
      *scaled += 1;
      src[9 * i] = b.store(r.ev[0]);
      static_for<4>([&](auto D) {
        constexpr int k = decltype(D)::value + 1;
        const fx::i64 eg = e_dot<LAT_D2Q9, k>(r.gx, r.gy, (fx::i64)0);
        src[9 * i + k] = b.store(r.ev[k] + eg);
        src[9 * i + k + 4] = b.store(r.ev[k] - eg);
      });
    } else {
      // beside an adjoint of zero, as in units that take it
      fx::Block z;
      const double none[1] = {0.};
      z.measure<1>(none);
      z.at_most(d.scale_limit(p.fix));
      const fx::Source2 r0 = d.scaled(p.fix, z);
      if (!r0.on) return i;
      src[9 * i] = z.store(r0.ev[0]);
      static_for<4>([&](auto D) {
        constexpr int k = decltype(D)::value + 1;
        const fx::i64 eg = e_dot<LAT_D2Q9, k>(r0.gx, r0.gy, (fx::i64)0);
        src[9 * i + k] = z.store(r0.ev[k] + eg);
        src[9 * i + k + 4] = z.store(r0.ev[k] - eg);
      });
    }
    val64[i] = ObjDissipation::evaluate<LAT_D2Q9, false>(f + 9 * i, g[i], 0, 0, 0, p);
    double dg = 0.;
    ObjDissipation::source<LAT_D2Q9, false>(f + 9 * i, g[i], src64 + 9 * i, dg, 0, 0, 0, p);
  }
  return n;
}
}
