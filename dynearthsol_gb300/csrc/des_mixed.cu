// des_mixed.cu -- kernels of the mixed-precision step (DES_PREC_MIXED).
//
// On GB300 an FP64 instruction issues at 1/64 of the FP32 rate, and the FP64
// step is FP64-pipe-bound (update_stress keeps the FP64 pipe ~86% busy).
// The mixed step keeps every state variable, every stress and strain
// increment and every nodal sum in FP64, and moves to FP32 the expensive
// work whose result is a coefficient or a small correction:
//
// * the viscosity (Arrhenius power law: pow, exp; the harmonic mean over
//   the element's materials), evaluated to ~2e-7 with FP32 transcendentals
//   on an exact exponent split (visc_mixed);
// * the Mohr-Coulomb yield test: the DEVIATORIC trial stress is
//   diagonalised in FP32 (branch-free cyclic Jacobi) to screen out the
//   elements that are elastic by a margin above the FP32 error bound; the
//   others -- everything at or beyond yield -- run the FP64 return map
//   (FP64 eigen-solve), so plastic flow is never computed in FP32.  In the
//   EVP rheology (k_update_stress_evp3) a cheaper screen on an upper bound
//   comes first, and the FP64 branches of a block are listed and run side
//   by side;
// * the shear strain rates, the spin and the heat stencil: sums of products
//   of shape function derivatives with nodal values whose sum over the
//   element vanishes, evaluated in FP32 on FP64 differences (v_i - v_0,
//   T_j - T_i); the Jaumann rotation increments.  The normal strain rates
//   are double-word (see k_strain_rate_mixed3).
// The elastic and Maxwell increments stay FP64: the quasi-static explicit
// scheme integrates their rounding without dissipating it (damping option 2
// only scales the force), and in FP32 they alone moved the stress by 4e-6
// (relative L2) after 2000 steps of the 998,400-tet workload.
// Element volumes and masses stay FP64; shape functions and forces are
// double-word (des_kernels.cu).
#include <algorithm>
#include <cfloat>

#include "des_kernels.cuh"
#include "des_rheology.cuh"
#include "des_mixed.cuh"
#include "des_dw.cuh"
#include "des_gather.cuh"
#include "des_mixed_elem.cuh"

namespace des {

constexpr int TPB_M = 256;

__device__ __forceinline__ float shp32_at(const KP &p, int k, int i, int e)
{
    return p.shpdw[((size_t)k * 4 + i) * p.ne + e].x;   // the pair's high part: the nearest float
}

// exp(x) for |x| < 690 as 2^k exp(r): any integer k near x / ln 2 keeps |r|
// small, so k is rounded in FP32; r = x - k ln 2 is one FP64 fma; 2^k goes
// into the exponent field of expf(r) (in [0.7, 1.5], so the result stays
// normal).  Within ~1.5e-7 of exp(x).
__device__ __forceinline__ double exp_mixed(double x)
{
    const double LN2 = 0.6931471805599453;
    const float kf = fminf(fmaxf(rintf(f32_of(x) * 1.44269504f), -1000.0f), 1000.0f);
    const float rr = f32_of(fma(-f64_of(kf), LN2, x));
    const double m = f64_of(expf(rr));
    return __hiloint2double(__double2hiint(m) + ((int)kf << 20), __double2loint(m));
}

// ln visc_m of material m from ln(edot_II) and 1/T, clamped exactly to
// [visc_min, visc_max] on ln visc, then exp_mixed (visc_mixed's terms)
__device__ __forceinline__ double visc_law_mixed(const KP &p, int m, double ln_ed, double r)
{
    const double lnv = fma(p.mat.visc_qnr[m], r, fma(p.mat.visc_pw[m], ln_ed, p.mat.visc_lnc[m]));
    // with clamps above 1 Pa s the comparisons are those of the bit patterns,
    // off the FP64 pipe: a negative lnv lies below every clamp, a NaN of
    // either sign counts as above (as the FP64 law at T = 0)
    const long long b = __double_as_longlong(lnv);
    const bool nan = (b & 0x7fffffffffffffffLL) > 0x7ff0000000000000LL;
    const bool low = p.mat.visc_ln_pos ? !nan && b <= __double_as_longlong(p.mat.visc_lnmin) : lnv <= p.mat.visc_lnmin;
    const bool high = p.mat.visc_ln_pos ? nan || b >= __double_as_longlong(p.mat.visc_lnmax) : !(lnv < p.mat.visc_lnmax);
    if (low) return p.mat.visc_min;
    if (high) return p.mat.visc_max;   // also T = 0 (1/T infinite), as the FP64 law
    return exp_mixed(lnv);
}

// visc_mixed over the element's markers.  One material present: its law
// (n / (n / visc) = visc).  Several: the harmonic mean.  Out of line: the
// registers of the blend stay out of the one-material kernels.
static __device__ __noinline__ double visc_blend_mixed(const KP &p, int e, double ln_ed, double r)
{
    int mone = -1, present = 0;
    for (int m = 0; m < p.mat.nmat; ++m)
        if (mcount(p, e, m)) {
            mone = m;
            ++present;
        }
    if (present == 1) return visc_law_mixed(p, mone, ln_ed, r);
    double result = 0;
    int n = 0;
    for (int m = 0; m < p.mat.nmat; ++m) {
        const int k = mcount(p, e, m);
        if (k == 0) continue;
        double lnv = fma(p.mat.visc_qnr[m], r, fma(p.mat.visc_pw[m], ln_ed, p.mat.visc_lnc[m]));
        lnv = fmin(fmax(lnv, p.mat.visc_lnmin - 50), p.mat.visc_lnmax + 50);
        result = fma((double)k, exp_mixed(-lnv), result);
        n += k;
    }
    return dmin_(dmax_(n / result, p.mat.visc_min), p.mat.visc_max);
}

// Arrhenius power-law viscosity (matprops.cxx:276-312), per material m
//   ln visc_m = ln(0.25e6 coef_m) + pw_m ln(edot_II) + Q_m / (n_m R T),
// with every term kept to ~1e-8 absolute at ~10 FP64 operations:
// ln(edot_II) = logf(mantissa) + exponent ln 2 (the FP32 log only sees
// [0.5, 1)); 1/T from an FP32 seed and one FP64 Newton step; exp by
// exp_mixed.  One material in the element: the clamps to [visc_min,
// visc_max] are exact on ln visc.  Several: the harmonic mean over the
// element's markers,
// n / sum_m k_m exp(-ln visc_m), over the materials it holds (each ln visc_m
// limited to 50 beyond the clamps, which moves no clamped mean), then the
// clamps.  The result is within ~2e-7 of the FP64 law.  Every FP64 <-> FP32
// conversion is f32_of / f64_of (integer instructions).
__device__ __forceinline__ double visc_mixed(const KP &p, int e, const double *edot, const float *t, double T)
{
    if (p.ef[DES_EF_LOG10_VISC]) return m_visc<3>(p, e, edot);
    const double LN2 = 0.6931471805599453;
    const float a = (t[0] + t[1] + t[2]) * (1.0f / 3.0f);
    const float j2 = 0.5f * ((t[0] - a) * (t[0] - a) + (t[1] - a) * (t[1] - a) + (t[2] - a) * (t[2] - a))
        + t[3] * t[3] + t[4] * t[4] + t[5] * t[5];
    const float ed = fmaxf(sqrtf(j2), 1e-30f);
    int ex;
    const float mant = frexpf(ed, &ex);
    const double ln_ed = fma(f64_of((float)ex), LN2, f64_of(logf(mant)));
    double r = f64_of(1.0f / f32_of(T));
    r = r * fma(-T, r, 2.0);
    if (p.mat.nmat == 1) return visc_law_mixed(p, 0, ln_ed, r);
    return visc_blend_mixed(p, e, ln_ed, r);
}

__device__ __forceinline__ double visc_mixed(const KP &p, int e, const double *edot, double T)
{
    float t[6];
#pragma unroll
    for (int i = 0; i < 6; ++i) t[i] = f32_of(edot[i]);
    return visc_mixed(p, e, edot, t, T);
}

// maxwell (rheology.cxx:118-134).  The relaxation coefficients come from
// FP32: tmp = dt G / (2 visc) and f2 - 1 = -tmp / (1 + tmp), each within
// ~2^-22 of itself (the viscosity they scale is good to ~2e-7), so f1 =
// 1 - tmp and f2 are one FP64 addition each instead of two FP64 Newton
// reciprocals.  The updates are fused multiply-adds, and the mean stress
// and K dv are added to the deviator in one step.  The divisions by 3 are
// div3, bit-identical.
struct MaxwellCoef {
    double f1, f2;
};

__device__ __forceinline__ MaxwellCoef maxwell_coef(double shearm, double viscosity, double dt)
{
    const float tf = (0.5f * f32_of(dt) * f32_of(shearm)) / f32_of(viscosity);
    return {1 - f64_of(tf), 1 + f64_of(-tf / (1.0f + tf))};
}

// the update on the old normal deviator x_i = s_i - s0 and y_i = 2G (de_i -
// tr(de)/3); s0k = s0 + K dv; s and de for the shear components
__device__ __forceinline__ void maxwell_mixed_xy(const MaxwellCoef &c, double g2, double s0k, const double *x,
                                                 const double *y, const double *s, const double *de, double *out)
{
#pragma unroll
    for (int i = 0; i < 3; ++i) out[i] = fma(fma(x[i], c.f1, y[i]), c.f2, s0k);
#pragma unroll
    for (int i = 3; i < 6; ++i) out[i] = fma(s[i], c.f1, g2 * de[i]) * c.f2;
}

__device__ __forceinline__ void maxwell_mixed(double bulkm, double shearm, double viscosity, double dt, double dv,
                                              const double *de, double *s)
{
    const double dev = div3(de[0] + de[1] + de[2]);
    const double s0 = div3(s[0] + s[1] + s[2]);
    const double g2 = 2 * shearm;
    double x[3], y[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        x[i] = s[i] - s0;
        y[i] = g2 * (de[i] - dev);
    }
    maxwell_mixed_xy(maxwell_coef(shearm, viscosity, dt), g2, s0 + bulkm * dv, x, y, s, de, s);
}

// elastic_ (rheology.cxx:13-40) with fused multiply-adds: 2G de_i + lambda tr(de)
// as one fma, each shear update as one fma (rounding an ulp from elastic_'s)
__device__ __forceinline__ void elastic_mixed(double bulkm, double shearm, const double *de, double *s)
{
    const double lambda = bulkm - 2. / 3 * shearm;
    const double ldev = lambda * (de[0] + de[1] + de[2]);
    const double g2 = 2 * shearm;
#pragma unroll
    for (int i = 0; i < 3; ++i) s[i] += fma(g2, de[i], ldev);
#pragma unroll
    for (int i = 3; i < 6; ++i) s[i] = fma(g2, de[i], s[i]);
}

// ------------------------------------------------------------------
// The mixed EVP branch in increment form.  Both candidates of the branch
// choice (rheology.cxx:594-634) are the old stress s plus an FP32 increment
// added in FP64:
//   Maxwell (rheology.cxx:118-134)  dv = c1 x + f2 y + K dv_vol   (normal),
//                                        c1 x + f2 y              (shear),
//   elastic trial (elastic_)        dp = y + K tr(de)             (normal),
//                                        y                        (shear),
// x the old deviator (s_i - s0 for the normal components, the old shear
// stress), y = 2G (de - tr(de)/3) (normal) and 2G de (shear) the trial's
// deviatoric increment, f2 = 1 / (1 + tmp), c1 = f1 f2 - 1 = -2 tmp f2
// with f1 = 1 - tmp and tmp = dt G / (2 visc): the Maxwell update
// (x f1 + y) f2 + s0 + K dv_vol less the old stress.  The increments are
// small against the stress (a few hundred Pa per step against ~1e8 Pa in
// the 998,400-tet workload), so their FP32 rounding (~2^-23 of themselves)
// moves the stress by ~1e-5 Pa per step, while the FP64 additions keep the
// state's own precision: 6 FP64 additions per candidate instead of the 16
// FP64 operations of the FP64-coefficient update.
// ------------------------------------------------------------------
// relative volume change vol / vol_old - 1 in FP32 from the FP64 difference
// (exact for volumes within a factor 2 of each other)
__device__ __forceinline__ float dvol_f(const KP &p, int e)
{
    const double vo = p.vol_old[e];
    return f32_of(p.vol[e] - vo) / f32_of(vo);
}

// The branch choice svII < spII of the mixed step, decided from FP32 values
// where an identity allows.  The comparison it stands for is the FP64 one of
// the FP64 candidates (those the branch forms where the screen is
// undecided): the elastic trial sp = elastic_mixed(s, de) and the Maxwell
// update sv = maxwell_mixed_xy(x, y) with f1 = 1 - tmp, f2 = 1 / (1 + tmp).
// Their exact deviators are q = x + y and f2 (q - tmp x), so
//   J2(sv) - J2(sp) = -f2^2 tmp Q,  Q = (2 + tmp) J(q) + 2 <q, x> - tmp J(x),
// J(v) = (v0^2 + v1^2 + v2^2) / 2 + v3^2 + v4^2 + v5^2, <,> its bilinear
// form: the Maxwell candidate wins exactly when Q > 0.  Q carries no
// cancellation (for a small increment q ~ x and Q ~ 4 J(q)), so its FP32
// value decides the comparison wherever f2^2 tmp |Q| clears the FP64
// comparison's own roundings, even in cold elements whose relaxation tmp
// (~1e-8 per step) lies below FP32's resolution of the stress.
//   Inputs: xf, yf, qf the FP32 forms of x, y, q (per component, xf within
// 2^-24 |xf| of x plus 2^-50 S for the FP64 mean; yf, formed from FP32
// strain increments, within 2^-22 (|yf| + Y) of the FP64 y, Y = 2G sum
// |de_i|; qf within the sum of both plus 2^-24 |qf|).  The bound on
// |Q_est - Q| sums, per component with weights 1 (normal) and 2 (shear),
// the first-order terms of those errors in J(q), <q, x> and J(x) with their
// squares, and 2^-20 of the absolute terms for Q's own FP32 evaluation.
// R bounds the FP64 side: two second_invariant2_ evaluations (each within
// 12 u J + 12.25 u S sqrt(J) + 37.5 u^2 S^2, j2_est3's analysis) and the
// candidates' roundings (2 u S per component), taken as 2^-45 J + 2^-45 S
// sqrt(J) + (2^-46 S)^2 with J ~ Jq (margins of 8 and more), and the FP32 rounding of f2 - 1 in maxwell_coef
// (2^-23 tmp relative, times J(q) + 2 tmp |<q, x>| + tmp^2 J(x), taken as
// 2^-20 tmp of the absolute terms).  Returns 1 (Maxwell), 0 (elasto-
// plastic: not svII < spII, ties included) or -1 (undecided, or tmp not
// positive, or a non-finite input).
__device__ __forceinline__ int evp_choice_f(const float *xf, const float *yf, const float *qf, float tf, float Y,
                                            float S)
{
    const float e64 = 0x1p-50f * S;
    float jq2 = 0.0f, jx2 = 0.0f, c2 = 0.0f, Aqx = 0.0f, Eqq = 0.0f, Eqx = 0.0f, Exx = 0.0f;
#pragma unroll
    for (int c = 0; c < 6; ++c) {
        const float wt = c < 3 ? 1.0f : 2.0f;
        const float aq = fabsf(qf[c]), ax = fabsf(xf[c]);
        jq2 += wt * qf[c] * qf[c];
        jx2 += wt * xf[c] * xf[c];
        c2 += wt * qf[c] * xf[c];
        Aqx += wt * aq * ax;
        const float ex = 0x1p-24f * ax + e64;
        const float eq = ex + 0x1p-22f * (fabsf(yf[c]) + Y) + 0x1p-24f * aq;
        Eqq += wt * eq * (2.0f * aq + eq);
        Eqx += wt * (eq * ax + ex * aq + eq * ex);
        Exx += wt * ex * (2.0f * ax + ex);
    }
    const float Q = 0.5f * (2.0f + tf) * jq2 + c2 - 0.5f * tf * jx2;
    const float absQ = (2.0f + tf) * jq2 + Aqx + tf * jx2;
    const float EQ = 0.5f * (2.0f + tf) * Eqq + Eqx + 0.5f * tf * Exx + 0x1p-20f * absQ;
    const float f2 = 1.0f / (1.0f + tf);
    const float G = f2 * f2 * tf;
    const float h = 0x1p-46f * S;
    const float R = 0x1p-46f * jq2 + 0x1p-46f * S * sqrtf(2.0f * jq2) + h * h + 0x1p-20f * tf * absQ + 0x1p-100f;
    if (!(tf > 0.0f)) return -1;
    if (G * (Q - EQ) > R) return 1;
    if (G * (Q + EQ) < -R) return 0;
    return -1;
}

// relative volume change (rheology.cxx:569,600: vol / vol_old - 1) as
// (vol - vol_old) (1 / vol_old): the difference is exact for volumes within a
// factor 2 of each other, and recip_newton's ~1e-14 relative error scales the
// ~1e-8 volume change, against the ~1e-16 absolute rounding of the quotient
// form; one FP64 division fewer
__device__ __forceinline__ double dvol_mixed(const KP &p, int e)
{
    const double vo = p.vol_old[e];
    return (p.vol[e] - vo) * recip_newton(vo);
}

// the anti-locking correction of the normal strain rates (rheology.cxx:527-534),
// as the FP64 step rounds it
__device__ __forceinline__ void correct_edot(double edv, double *edot)
{
    const double corr = div3(edv - (edot[0] + edot[1] + edot[2]));
#pragma unroll
    for (int i = 0; i < 3; ++i) edot[i] += corr;
}

// The element's strain rate before that correction.  ahead: the shear
// components come as the FP32 values that the look-ahead geometry pass formed.
__device__ __forceinline__ void load_srate(const KP &p, int e, bool ahead, double *edot)
{
    const size_t ne = p.ne;
#pragma unroll
    for (int c = 0; c < 3; ++c) edot[c] = p.srate[c * ne + e];
#pragma unroll
    for (int c = 3; c < 6; ++c) edot[c] = ahead ? f64_of(p.sh32[(c - 3) * ne + e]) : p.srate[c * ne + e];
}

// edvoldt (geometry.cxx:158-179) from the step's nodal dvoldt
__device__ __forceinline__ double elem_edv(const KP &p, int e)
{
    double dj = p.ntmp[conn_at(p, 0, e)];
#pragma unroll
    for (int i = 1; i < 4; ++i) dj += p.ntmp[conn_at(p, i, e)];
    return node_mean<4>(dj);
}

// the pressure change, and for the NMD gather its double-word product with
// the volume, formed once per element instead of per node
__device__ __forceinline__ void store_dp(const KP &p, int e, double dp, dw w, bool fused)
{
    p.dp[e] = dp;
    if (fused && p.pv) {
        const dw m = dw_mul(w, dw_split(p.vol[e]));
        p.pv[e] = make_float2(m.hi, m.lo);
    }
}

struct PlasticProps {
    double amc, anphi, anpsi, hardn, ten_max;
};

// The mixed EVP branch where the FP32 screens leave it to FP64: the FP64
// candidates -- the trial as the EP branch forms it (through the return map
// unless the yield screen passed it) and the Maxwell update with FP64 terms
// -- and, for an undecided choice (vless < 0), their FP64 comparison.  edot:
// the corrected strain rate, s: the old stress, m: the plastic properties
// (read unless elastic).  Out of line: the registers of the return map stay
// out of the common path.
static __device__ __noinline__ void evp_fp64_branch(const KP &p, int e, bool elastic, int vless, bool fused,
                                                    const double *edot, const double *s, double pls,
                                                    const PlasticProps &m)
{
    const size_t ne = p.ne;
    const double dt = p.clk->dt;
    const double bulkm = m_bulkm(p, e), shearm = m_shearm(p, e);
    double de[6], sp[6], sv[6];
#pragma unroll
    for (int c = 0; c < 6; ++c) {
        sp[c] = s[c];
        de[c] = edot[c] * dt;
    }
    const double old_s = s[0] + s[1] + s[2];
    elastic_mixed(bulkm, shearm, de, sp);
    double depls = 0;
    if (!elastic && mc_return_<3>(bulkm, shearm, m.amc, m.anphi, m.anpsi, m.hardn, m.ten_max, depls, sp))
        set_err(p, DES_DEV_QL_NOCONV);
    if (vless < 0) {
        const double s0 = div3(old_s), dev = div3((de[0] + de[1]) + de[2]);
        const double g2 = 2 * shearm;
        double x[3], y[3];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            x[i] = s[i] - s0;
            y[i] = g2 * (de[i] - dev);
        }
        const double visc = visc_mixed(p, e, edot, elem_avg_T<4>(p, e));
        maxwell_mixed_xy(maxwell_coef(shearm, visc, dt), g2, s0 + bulkm * dvol_mixed(p, e), x, y, s, de, sv);
        vless = second_invariant2_<3>(sv) < second_invariant2_<3>(sp);
    }
    double out[6];
#pragma unroll
    for (int i = 0; i < 6; ++i) {
        out[i] = vless ? sv[i] : sp[i];
        p.stress[i * ne + e] = out[i];
    }
    if (!vless) {
        p.pls[e] = pls + depls;
        p.dpls[e] = depls;
    }
    const double dp = (out[0] + out[1] + out[2]) - old_s;
    store_dp(p, e, dp, dw_split(dp), fused);
}

// what is left of an element after the FP32 screens: nothing, or its FP64
// branch with the screens' answers, or the screens again with the FP64
// material terms
enum EvpRest : int { EVP_DONE = 0, EVP_ELASTIC = 1, EVP_PLASTIC_BRANCH = 2, EVP_FP64 = 4, EVP_SCREEN = 8 };

// The EVP branch choice of an element from its FP32 strain increments def and
// relaxation tf, and its stress where the choice is the Maxwell branch: the
// old stress s plus an FP32 increment.
__device__ __forceinline__ int evp_screens(const KP &p, int e, const double *s, const float *def, float tf,
                                           float shearf, float kf, ScreenTerms mt, bool fused)
{
    const size_t ne = p.ne;
    const double s0 = div3(s[0] + s[1] + s[2]);
    const float g2f = 2.0f * shearf;
    const float trdef = (def[0] + def[1]) + def[2];
    const float devf = trdef * (1.0f / 3.0f);
    // x: the old deviator; y: the trial's deviatoric increment
    float xf[6], yf[6], qf[6];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        xf[i] = f32_of(s[i] - s0);
        yf[i] = g2f * (def[i] - devf);
        xf[i + 3] = f32_of(s[i + 3]);
        yf[i + 3] = g2f * def[i + 3];
    }
    const float dmp = kf * trdef;
#pragma unroll
    for (int c = 0; c < 6; ++c) qf[c] = xf[c] + yf[c];
    // the yield screen on the trial deviator qf: against the deviator of
    // the FP64 trial elastic_mixed(s, de) it is off by xf's and qf's
    // roundings and by yf's distance from the FP64 y (2^-22 of
    // Lx + Ly + Y per component, taken as 2^-21 in the 2-norm) and by
    // the FP64 roundings of the mean (22 u S, taken as 2^-44 S)
    const float s0f = f32_of(s0);
    float Y = 0.0f, Sdev = 0.0f;
#pragma unroll
    for (int i = 0; i < 3; ++i) Y += fabsf(def[i]);
    Y *= g2f;
#pragma unroll
    for (int c = 0; c < 6; ++c) Sdev += fabsf(xf[c]) + fabsf(yf[c]);
    Sdev += Y;
    const float S = fabsf(s0f) + Sdev + 2.0f * fabsf(kf) * (Y / fmaxf(g2f, 1e-30f));
    const int screen = yield_screen3_f(mt.af, mt.cf, mt.tf, s0f + dmp, fabsf(s0f) + fabsf(dmp), qf,
                                       0x1p-44f * S + 0x1p-21f * Sdev, mt.err);
    if (screen < 0) return EVP_SCREEN;
    if (screen == 0) return EVP_FP64;
    const int vless = evp_choice_f(xf, yf, qf, tf, Y, S);
    if (vless != 1) return EVP_FP64 | EVP_ELASTIC | (vless == 0 ? EVP_PLASTIC_BRANCH : 0);
    const float f2 = 1.0f / (1.0f + tf), c1 = -2.0f * tf * f2;
    const float dmv = kf * dvol_f(p, e);
    float dn = 0.0f;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const float d = fmaf(xf[i], c1, fmaf(yf[i], f2, dmv));
        p.stress[i * ne + e] = s[i] + f64_of(d);
        dn += d;
        p.stress[(i + 3) * ne + e] = s[i + 3] + f64_of(fmaf(xf[i + 3], c1, yf[i + 3] * f2));
    }
    const double dp = f64_of(dn);
    store_dp(p, e, dp, dw_split(dp), fused);
    return EVP_DONE;
}

// tmp = dt G / (2 visc), the Maxwell update's relaxation
__device__ __forceinline__ float relaxation_f(float dtf, float shearf, float viscf)
{
    return (0.5f * dtf * shearf) / viscf;
}

__device__ __forceinline__ void load_stress(const KP &p, int e, double *s)
{
#pragma unroll
    for (int c = 0; c < 6; ++c) s[c] = p.stress[c * (size_t)p.ne + e];
}

__device__ __forceinline__ ScreenTerms exact_terms(const PlasticProps &m)
{
    return {f32_of(m.anphi), f32_of(m.amc), f32_of(m.ten_max), 0.0f};
}

__device__ __forceinline__ int screened_choice(int rest) { return rest & EVP_PLASTIC_BRANCH ? 0 : -1; }

// what evp_screens left of element e; edot_done: p.srate holds the corrected
// strain rate
static __device__ __noinline__ void evp_rest(const KP &p, int e, int rest, bool fused, bool edot_done, bool ahead)
{
    double edot[6], s[6];
    load_srate(p, e, ahead && !edot_done, edot);
    if (!edot_done) correct_edot(elem_edv(p, e), edot);
    load_stress(p, e, s);
    const double pls = p.pls[e];
    PlasticProps m{};
    if (!(rest & EVP_ELASTIC)) m_plastic_props(p, e, pls, m.amc, m.anphi, m.anpsi, m.hardn, m.ten_max);
    if (rest & EVP_SCREEN) {
        const float dtf = f32_of(p.clk->dt), shearf = f32_of(m_shearm(p, e));
        float def[6];
#pragma unroll
        for (int c = 0; c < 6; ++c) def[c] = f32_of(edot[c]) * dtf;
        const float viscf = f32_of(visc_mixed(p, e, edot, elem_avg_T<4>(p, e)));
        rest = evp_screens(p, e, s, def, relaxation_f(dtf, shearf, viscf), shearf, f32_of(m_bulkm(p, e)),
                           exact_terms(m), fused);
        if (rest == EVP_DONE) return;
    }
    evp_fp64_branch(p, e, (rest & EVP_ELASTIC) != 0, screened_choice(rest), fused, edot, s, pls, m);
}

// update_stress (rheology.cxx:510-646), 3D, mixed precision, the EVP
// rheology.  Each thread updates its element's strain and, where the FP32
// screens decide it (nearly all elements of a mesh that does not yield), its
// stress by the Maxwell increments.  The others -- at or near the yield
// surface, or with nearly tied branches -- go to a list in shared memory,
// and once the block's common path is done its first threads run their FP64
// branch side by side: a return map's FP64 instructions (several hundred)
// then serve full warps instead of the few lanes of each warp that yield,
// and its registers stay out of the common path.  An element's result does
// not depend on its place in the list.  LIST false (a mesh of at most one
// wave, where the length of a thread's chain shows and registers do not): the
// thread forms the FP64 properties first and goes on to the FP64 branch with
// what it holds.
// outputs: write the strain rate and edvoldt, which only the end of a call
// shows (a chained step that another follows leaves them out).
// Bounds: the FP64 pipe (48 FP64-pipe instructions an element off the yield
// surface, 72% of its rate) and the issue of the FP32 work beside it.
// 998,400 tets: 177 us with the FP64 branches in place, 121 us with the list,
// 111 us with the shear strain rates as floats (ahead), the density's
// buoyancy formed where the forces are, and the quarterings, clamps and
// softening bounds taken as integer operations.
template <bool LIST>
__global__ void __launch_bounds__(LIST ? 128 : 64, LIST ? 8 : 4) k_update_stress_evp3(KP p, int fused, int outputs,
                                                                                       int ahead)
{
    __shared__ int list[128];
    __shared__ int listed;
    if (LIST) {
        if (threadIdx.x == 0) listed = 0;
        __syncthreads();
    }
    const int base = p.e_lo + (int)(blockIdx.x * blockDim.x), e = base + (int)threadIdx.x;
    const size_t ne = p.ne;
    if (e < p.e_hi) {
        const float dtf = f32_of(p.clk->dt);
        float def[6];
        double edot[6];
        float edf[6];   // the strain rate in FP32
        {   // FP32 strain increments; the strain accumulates them in FP64
            double edv;
            if (fused) {
                edv = elem_edv(p, e);
                if (outputs) p.edvoldt[e] = edv;
            } else {
                edv = p.edvoldt[e];
            }
            if (ahead) {   // f32_of(f64_of(x)) is x, a subnormal's a zero
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    edot[c] = p.srate[c * ne + e];
                    const float x = p.sh32[c * ne + e];
                    edf[3 + c] = fabsf(x) < FLT_MIN ? copysignf(0.0f, x) : x;
                    edot[3 + c] = f64_of(edf[3 + c]);
                }
            } else {
                load_srate(p, e, false, edot);
#pragma unroll
                for (int c = 3; c < 6; ++c) edf[c] = f32_of(edot[c]);
            }
            correct_edot(edv, edot);
#pragma unroll
            for (int c = 0; c < 3; ++c) edf[c] = f32_of(edot[c]);
#pragma unroll
            for (int c = 0; c < 6; ++c) {
                if (outputs) p.srate[c * ne + e] = edot[c];
                def[c] = edf[c] * dtf;
                p.strain[c * ne + e] += f64_of(def[c]);
            }
        }
        const double T = elem_avg_T<4>(p, e);
        const float shearf = f32_of(m_shearm(p, e));
        const float tf = relaxation_f(dtf, shearf, f32_of(visc_mixed(p, e, edot, edf, T)));
        if (fused && p.rho_e) p.rho_e[e] = m_rho_T(p, e, T);   // the step's: the temperature is final
        const double pls = p.pls[e];
        double s[6];
        load_stress(p, e, s);
        PlasticProps m;
        ScreenTerms mt;
        if (LIST) {
            mt = screen_terms(p, e, pls);
        } else {
            m_plastic_props(p, e, pls, m.amc, m.anphi, m.anpsi, m.hardn, m.ten_max);
            mt = exact_terms(m);
        }
        const int rest = evp_screens(p, e, s, def, tf, shearf, f32_of(m_bulkm(p, e)), mt, fused != 0);
        if (LIST) {
            if (rest) list[atomicAdd(&listed, 1)] = ((int)threadIdx.x << 4) | rest;
        } else if (rest) {
            evp_fp64_branch(p, e, (rest & EVP_ELASTIC) != 0, screened_choice(rest), fused != 0, edot, s, pls, m);
        }
    }
    if (!LIST) return;
    __syncthreads();
    const int n = listed;
    for (int k = threadIdx.x; k < n; k += blockDim.x)
        evp_rest(p, base + (list[k] >> 4), list[k] & 15, fused != 0, outputs || !fused, ahead != 0);
}

// the other rheologies
__global__ void __launch_bounds__(128, 6) k_update_stress_mixed3(KP p, int fused, int ahead)
{
    int e = p.e_lo + blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= p.e_hi) return;
    const size_t ne = p.ne;
    double edv;
    if (fused) {
        edv = elem_edv(p, e);
        p.edvoldt[e] = edv;
    } else {
        edv = p.edvoldt[e];
    }
    double s[6], es[6], edot[6], de[6];
    load_srate(p, e, ahead != 0, edot);
    correct_edot(edv, edot);
    const double dt = p.clk->dt;
#pragma unroll
    for (int c = 0; c < 6; ++c) {
        s[c] = p.stress[c * ne + e];
        de[c] = edot[c] * dt;
        es[c] = p.strain[c * ne + e] + de[c];
    }
    const double old_s = s[0] + s[1] + s[2];
    const int rt = p.mat.rheol_type;
    const double bulkm = m_bulkm(p, e), shearm = m_shearm(p, e);
    const double T = elem_avg_T<4>(p, e);
    unsigned bits = 0;
    if (rt == DES_RH_ELASTIC) {
        elastic_mixed(bulkm, shearm, de, s);
    } else if (rt == DES_RH_VISCOUS) {
        viscous_<3>(bulkm, visc_mixed(p, e, edot, T), es[0] + es[1] + es[2], edot, s);
    } else if (rt == DES_RH_MAXWELL) {
        maxwell_mixed(bulkm, shearm, visc_mixed(p, e, edot, T), dt, dvol_mixed(p, e), de, s);
    } else {   // EP
        double amc, anphi, anpsi, hardn, ten_max;
        const double pls = p.pls[e];
        m_plastic_props(p, e, pls, amc, anphi, anpsi, hardn, ten_max);
        elastic_mixed(bulkm, shearm, de, s);
        const double am = div3(s[0] + s[1] + s[2]);
        const double q[3] = {s[0] - am, s[1] - am, s[2] - am};
        double depls = 0;
        if (!clearly_elastic3_dev(amc, anphi, ten_max, am, q, s)
            && mc_return_<3>(bulkm, shearm, amc, anphi, anpsi, hardn, ten_max, depls, s))
            bits |= DES_DEV_QL_NOCONV;
        p.pls[e] = pls + depls;
        p.dpls[e] = depls;
    }
#pragma unroll
    for (int c = 0; c < 6; ++c) {
        p.stress[c * ne + e] = s[c];
        p.strain[c * ne + e] = es[c];
        p.srate[c * ne + e] = edot[c];
    }
    const double dp = (s[0] + s[1] + s[2]) - old_s;
    store_dp(p, e, dp, dw_split(dp), fused != 0);
    if (fused && p.rho_e) p.rho_e[e] = m_rho_T(p, e, T);
    if (bits) set_err(p, bits);
}

// strain rate (fields.cxx:166-232) of one element, loaded from memory and
// formed by strain_rate_mixed_vals (des_mixed_elem.cuh)
__device__ __forceinline__ void strain_rate_mixed_elem(const KP &p, int e, double *out)
{
    const size_t ne = p.ne;
    dw v[4][3];
    float2 h[3][3];   // dN_i/dx_k of slots 1..3 as double-word pairs
    load_elem_v_dw(p, e, v);
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int i = 1; i < 4; ++i) h[k][i - 1] = p.shpdw[((size_t)k * 4 + i) * ne + e];
    float shear[3];
    strain_rate_mixed_vals(v, h, out, shear);
#pragma unroll
    for (int c = 0; c < 3; ++c) out[3 + c] = f64_of(shear[c]);
#pragma unroll
    for (int c = 0; c < 6; ++c) p.srate[c * ne + e] = out[c];
}

__global__ void __launch_bounds__(TPB_M) k_strain_rate_mixed3(KP p)
{
    int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= p.ne) return;
    double sr[6];
    strain_rate_mixed_elem(p, e, sr);
}

// dvoldt (quantity 0) in FP64, the others in compensated FP32 sums
struct SumNode {
    using Term = double;   // the pairs travel as the FP64 value's two words
    struct State {
        double d = 0;
        dw_sum w;
    };
    static __device__ __forceinline__ Term pack(dw w)
    {
        return __hiloint2double(__float_as_int(w.hi), __float_as_int(w.lo));
    }
    static __device__ __forceinline__ void add(int c, State &s, Term t)
    {
        if (c == 0) s.d += t;
        else s.w.add(dw{__int_as_float(__double2hiint(t)), __int_as_float(__double2loint(t))});
    }
    static __device__ __forceinline__ double value(int c, const State &s) { return c == 0 ? s.d : s.w.value(); }
};

// des_update_temperature's heat sums (fields.cxx:99-146): the stencil on FP64
// temperature differences (sum_j D_ij = 0), FP32 products, a compensated FP32
// sum of the terms.  A walk reads its node's temperature once, a staged entry
// for itself.
struct SumF32 {
    using Term = float;
    using State = dw_sum;
    static __device__ __forceinline__ void add(int, State &s, Term t) { s.add(t); }
    static __device__ __forceinline__ double value(int, const State &s) { return s.value(); }
};

template <bool STAGED>
__global__ void __launch_bounds__(256) k_heat_gather_mixed3(KP p)
{
    const bool k_const = (p.mat.nmat == 1) && !p.ef[DES_EF_THERM_COND];
    double tdot;
    const int n = node_sums<SumF32, 1, 3, STAGED>(
        p.sup_off, 0, p.nn, 1,
        [&](int q, float *t, int node) {
            const int ent = p.sup_ent[q];
            const int e = ent >> 2, i = ent & 3;
            const double Tn = p.T[STAGED ? conn_at(p, i, e) : node];
            const float sxi = shp32_at(p, 0, i, e), syi = shp32_at(p, 1, i, e), szi = shp32_at(p, 2, i, e);
            float diffusion = 0.0f;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (j == i) continue;
                const float D = sxi * shp32_at(p, 0, j, e) + syi * shp32_at(p, 1, j, e) + szi * shp32_at(p, 2, j, e);
                diffusion += D * f32_of(p.T[conn_at(p, j, e)] - Tn);
            }
            const float volf = f32_of(p.vol[e]);
            const float kv = f32_of(k_const ? p.mat.therm_cond[0] : m_k(p, e)) * volf;
            const float rh = f32_of(m_hr_over_cp(p, e)) * volf;
            *t = kv * diffusion - rh;
        },
        FromZero<SumF32>(), &tdot);
    if (n >= 0) p.tdot[n] = tdot;
}

// ------------------------------------------------------------------
// Fused step: strain rate, heat, dvoldt and the temperature update as one
// element pass and one node pass.  The per-pair work of the node-centric
// gather above (k_heat_gather_mixed3: the stencil row of the node's slot,
// four temperature differences and their FP32 conversions, which issue on
// the FP64 pipe) is done once per element: the element pass stores the
// four FP32 heat terms of the element and its dvoldt term, and the node
// pass sums them over the support list in ascending element order.  Each
// term is the very value the gather forms for that (node, element) pair,
// and the sums run in the same order, so the result is bit-identical to
// k_strain_rate_mixed3 + k_heat_gather_mixed3 + k_dvoldt + k_temperature_update.
// ------------------------------------------------------------------
__global__ void __launch_bounds__(TPB_M) k_elem_pass_mixed3(KP p, int heat)
{
    int e = p.e_lo + blockIdx.x * blockDim.x + threadIdx.x;
    if (e == 0) {   // var.steps++; var.time += var.dt (dynearthsol.cxx:325-326)
        p.clk->steps += 1;
        p.clk->time += p.clk->dt;
    }
    if (e >= p.e_hi) return;
    double sr[6];
    strain_rate_mixed_elem(p, e, sr);
    float s32[3][4];
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int i = 0; i < 4; ++i) s32[k][i] = shp32_at(p, k, i, e);
    elem_terms_mixed(p, e, sr, p.vol[e], s32, heat);
}

// The node pass: heat and dvoldt sums, the temperature update.  MASS (a chained
// step): it also forms the previous step's compute_mass sums (volume_n, mass,
// tmass) from the element records that the look-ahead geometry pass wrote
// (KP::ndpk), as k_mass_sum forms them, and starts the step's clock, which the
// look-ahead pass could not: its last block forms dt.
// The heat terms go into a compensated FP32 sum (des_dw.cuh), as
// k_heat_gather_mixed3 sums them; the dvoldt terms into an FP64 one: they
// cancel between a node's elements, and the 2^-47 of a double-word split of
// each moved the volumetric rate enough to change the default damping's
// copysign at some nodes within ten steps.
template <bool MASS, bool STAGED>
__global__ void __launch_bounds__(192) k_node_pass_mixed3(KP p, int heat)
{
    if (MASS && blockIdx.x == 0 && threadIdx.x == 0) {   // dynearthsol.cxx:325-326
        p.clk->steps += 1;
        p.clk->time += p.clk->dt;
    }
    constexpr int NQ = MASS ? 5 : 2;
    const size_t ne = p.ne;
    const bool thermal = p.prm.has_thermal_diffusion;
    double sum[NQ] = {};   // dvoldt, tdot, volume_n, mass, tmass
    const int n = node_sums<SumNode, NQ, 3, STAGED>(
        p.sup_off, p.n_lo, p.n_hi, NQ,
        [&](int q, double *t) {
            const int ent = p.sup_ent[q];
            const int e = ent >> 2, i = ent & 3;
            if constexpr (MASS) {
                const double4 r = p.ndpk[e];   // qv, vol, me, tme
                t[0] = r.x;
                t[2] = SumNode::pack(dw_split(r.y));
                t[3] = SumNode::pack(dw_split(r.z));
                t[4] = thermal ? SumNode::pack(dw_split(r.w)) : 0.0;
            } else {
                t[0] = p.qv[e];
            }
            t[1] = heat ? SumNode::pack(dw{p.hc[(size_t)i * ne + e], 0.0f}) : 0.0;
        },
        FromZero<SumNode>(), sum);
    if (n < 0) return;
    double vol_n, tmass = 0;
    if constexpr (MASS) {
        vol_n = sum[2];
        tmass = thermal ? sum[4] : 0.0;
        p.vol_n[n] = vol_n;
        p.mass[n] = sum[3];
        p.tmass[n] = tmass;
    } else {
        vol_n = p.vol_n[n];
        if (heat) tmass = p.tmass[n];
    }
    p.ntmp[n] = sum[0] / vol_n;
    if (heat) {   // temperature update + Dirichlet BC (fields.cxx:151-162)
        const unsigned flag = p.bcflag[n];
        if (flag & BOUNDZ1) p.T[n] = p.prm.surface_temperature;
        else if ((flag & BOUNDZ0) && !p.prm.has_fixed_bottom_temperature) p.T[n] = p.prm.mantle_temperature;
        else p.T[n] -= sum[1] * p.clk->dt / tmass;
    }
}

int launch_update_stress_mixed(const KP &p, cudaStream_t s, bool fused, bool outputs, bool ahead)
{
    const int n = p.e_hi - p.e_lo, out = outputs || !fused;
    if (p.mat.rheol_type != DES_RH_EVP)
        DES_LAUNCH(k_update_stress_mixed3, n, s, p, (int)fused, (int)ahead);
    // The line is the one between blocks of 64 and of 128, whose registers the two
    // forms have.  100 steps, list / in place: 14,400 tets with a yielding band
    // 9.0 / 8.1 ms, 49,152 10.9 / 10.5, 105,600 14.8 / 15.7, 193,536 21.1 / 25.0,
    // 301,056 26.7 / 31.7; without yielding 4.7 / 4.6, 5.74 / 5.69, 9.0 / 9.6,
    // 14.4 / 14.7, 16.8 / 17.7: the list would already pay from ~80,000 on.
    else if (one_wave(n))
        DES_LAUNCH(k_update_stress_evp3<false>, n, s, p, (int)fused, out, (int)ahead);
    else
        DES_LAUNCH(k_update_stress_evp3<true>, n, s, p, (int)fused, out, (int)ahead);
    return 1;
}

int launch_strain_rate_mixed(const KP &p, cudaStream_t s)
{
    DES_LAUNCH(k_strain_rate_mixed3, p.ne, s, p);
    return 1;
}

int launch_heat_gather_mixed(const KP &p, cudaStream_t s)
{
    // a term here is an element's stencil row: a walk forms a node's 24 rows one
    // after the other, so that staging pays on larger meshes too.  20 loops of
    // the per-function entry points, staged / walk: 73,728 tets 3.38 / 3.87 ms,
    // 162,624 (30,375 nodes) 4.82 / 5.18, 282,240 (51,984) 6.62 / 6.77.  The
    // walk's time is the L1 and L2 hits of its rows: a warp to a block 221 us a
    // call at 998,400 tets, blocks of 64 248, 128 234, 192 229, 256 231.
    if (p.nn <= 152 * 256) k_heat_gather_mixed3<true><<<(p.nn + NPB - 1) / NPB, STAGED_THREADS, 0, s>>>(p);
    else k_heat_gather_mixed3<false><<<(p.nn + 31) / 32, 32, 0, s>>>(p);
    return 1;
}

int launch_elem_pass_mixed(const KP &p, cudaStream_t s, bool heat)
{
    DES_LAUNCH(k_elem_pass_mixed3, p.e_hi - p.e_lo, s, p, (int)heat);
    return 1;
}

int launch_node_pass_mixed(const KP &p, cudaStream_t s, bool heat, bool mass_sums)
{
    const int n = p.n_hi - p.n_lo;
    if (mass_sums) DES_NODES((k_node_pass_mixed3<true, STAGED>), n, s, p, (int)heat);
    else DES_NODES((k_node_pass_mixed3<false, STAGED>), n, s, p, (int)heat);
    return 1;
}

}  // namespace des
