// Host build of a whole reverse step of a D2Q9 cell with the dissipation objective:
// source and transposed collision together, in fixed point as the step kernel
// combines them and by the FP64 operators.  Test infrastructure only.
#include "fixed_math_host.cpp"

namespace {
template <int COLL>
int step(const lbm_config* c, int n, const double* f, const double* g, const double* lo,
         double* fixed, double* dgf, double* fp64, double* dgd) {
  KParams p = params(c);
  p.md.obj_weight = c->obj_weight;
  p.md.cv_diss = 4.5 * ((1. / c->omega - 0.5) / 3.) * c->omega * c->omega;
  for (int i = 0; i < n; ++i) {
    const double imult = 0.5 * (p.md.pbb_scale * bp(g[i], p.md.pbb_q));
    const double dimult = 0.5 * (p.md.pbb_scale * bp_diff(g[i], p.md.pbb_q));
    double a[9];
    memcpy(a, lo + 9 * i, sizeof(a));
    dgd[i] = 0.;
    flow_reverse<LAT_D2Q9, COLL>(f + 9 * i, a, imult, dimult, dgd[i], p);
    ObjDissipation::source<LAT_D2Q9, false>(f + 9 * i, g[i], a, dgd[i], 0, 0, 0, p);
    memcpy(fp64 + 9 * i, a, sizeof(a));
    fx::Window w;
    fx::i64 x[9];
    static_for<9>([&](auto K) {
      constexpr int q = decltype(K)::value;
      x[q] = w.template load<LAT_D2Q9, q>(f[9 * i + q]);
    });
    if (!w.template ok<LAT_D2Q9>(x)) return i;
    const fx::Factor im((fx::u64)(imult * 18446744073709551616.));
    fx::Block b;
    b.template measure<9>(lo + 9 * i);
    const fx::Dissipation2 d(x, im, p.fix.cv);
    b.at_most(d.scale_limit(p.fix));
    memcpy(a, lo + 9 * i, sizeof(a));
    dgf[i] = dimult * fx::reverse<LAT_D2Q9, COLL>(x, a, b, im, p.fix, d.scaled(p.fix, b));
    dgf[i] += dimult * (p.md.obj_weight * d.dim);
    memcpy(fixed + 9 * i, a, sizeof(a));
  }
  return n;
}
}  // namespace

extern "C" int fixed_source_step(const lbm_config* c, int n, const double* f, const double* g,
                                 const double* lo, double* fixed, double* dgf, double* fp64,
                                 double* dgd) {
  return c->collision == LBM_MRT ? step<LBM_MRT>(c, n, f, g, lo, fixed, dgf, fp64, dgd)
                                 : step<LBM_BGK>(c, n, f, g, lo, fixed, dgf, fp64, dgd);
}
