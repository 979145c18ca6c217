// euler_kernels.cuh -- device code of the Eulerian grid hydrocode (the
// reference's hydrocodes/euler/hydro_cpu.cpp), shared by the two precision
// forms:
//   plain (FP64, euler.cu, compiled without fused multiply-adds): every
//     expression in the reference's operation order;
//   mixed (euler_mixed.cu): primitives, face fluxes, the right-hand side's
//     sources, the yield surface, damage growth and the CFL speed in FP32 (the
//     arithmetic of the reference's own GPU solver); the state and its
//     Runge-Kutta updates, the fluidization update and dt in FP64.
// The compute type R is the template parameter; the state is always FP64, the
// right-hand side stored in R.  Literals are written as R(...) so that an
// FP32 instantiation never promotes to FP64.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "fp64_int.cuh"

namespace deu {

// ---------------------------------------------------------------- arithmetic by compute type

// Divisions, square roots, comparisons and halvings in the compute type R: FP32
// as written; FP64 with the same IEEE results from the integer pipes
// (fp64_int.cuh), because the FP64 kernels here wait on the FP64 pipe and
// nothing else.  On the 96^3 impact (ncu) a face flux was 671 FP64
// instructions and is 157 with these, the EOS's shared subexpressions and one
// HLLC side per face; a face pass 1.14 -> 0.30 ms, a right-hand side 865 -> 194
// instructions and 1.46 -> 0.39 ms, the step 11.1 -> 3.0 ms, same bits.
template <class R>
struct DivBy;  // a divisor used more than once
template <>
struct DivBy<float> {
    float b;
};
template <>
struct DivBy<double> {
    fi::Divisor d;
};
FI_FN DivBy<float> div_by(float b) { return DivBy<float>{b}; }
FI_FN DivBy<double> div_by(double b) { return DivBy<double>{fi::divisor(b)}; }
FI_FN float dv(float a, const DivBy<float>& d) { return a / d.b; }
FI_FN double dv(double a, const DivBy<double>& d) { return fi::div(a, d.d); }
FI_FN float dv(float a, float b) { return a / b; }
FI_FN double dv(double a, double b) { return fi::div(a, b); }
static __device__ __forceinline__ float root(float x) { return sqrtf(x); }
static __device__ __forceinline__ double root(double x) { return fi::sqrt(x); }
FI_FN float half(float x) { return 0.5f * x; }
FI_FN double half(double x) { return fi::half(x); }
FI_FN bool lt(float a, float b) { return a < b; }
FI_FN bool lt(double a, double b) { return fi::lt(a, b); }
FI_FN bool ge(float a, float b) { return a >= b; }
FI_FN bool ge(double a, double b) { return fi::le(b, a); }
FI_FN bool lt0(float x) { return x < 0.0f; }
FI_FN bool lt0(double x) { return fi::lt0(x); }
FI_FN bool gt0(float x) { return x > 0.0f; }
FI_FN bool gt0(double x) { return fi::gt0(x); }
FI_FN bool ge0(float x) { return x >= 0.0f; }
FI_FN bool ge0(double x) { return fi::ge0(x); }
FI_FN bool le0(float x) { return x <= 0.0f; }
FI_FN bool le0(double x) { return fi::le0(x); }
// a + m / 2: the halving is exact, so one fused operation rounds as the two do
static __device__ __forceinline__ float add_half(float a, float m) { return a + 0.5f * m; }
static __device__ __forceinline__ double add_half(double a, double m) { return __fma_rn(0.5, m, a); }
// a b + c: fused in FP32 (explicit where the compiler's own choice of the fused
// product would depend on the code around it), the reference's two operations in FP64
static __device__ __forceinline__ float mad(float a, float b, float c) { return fmaf(a, b, c); }
static __device__ __forceinline__ double mad(double a, double b, double c) { return a * b + c; }
static __device__ __forceinline__ float sub_half(float a, float m) { return a - 0.5f * m; }
static __device__ __forceinline__ double sub_half(double a, double m) { return __fma_rn(-0.5, m, a); }

// ---------------------------------------------------------------- materials

template <class R>
struct MatT {
    int32_t ideal;
    R gamma, rho0, a, b, A, B, alpha, beta, u0, uiv, ucv, G, Y, Emod, wm, wk;
    // formed once on the host (mat_derive): quotients and divisors of the constants above
    R A_rho0, B2, iuv;
    DivBy<R> d_rho0, d_uv, d_Emod;
};
using Mat = MatT<double>;

template <class R>
inline void mat_derive(MatT<R>& m) {
    m.A_rho0 = m.A / m.rho0;
    m.B2 = R(2) * m.B;
    m.iuv = R(1) / (m.ucv - m.uiv);
    m.d_rho0 = div_by(m.rho0);
    m.d_uv = div_by(m.ucv - m.uiv);
    m.d_Emod = div_by(m.Emod);
}
inline MatT<float> mat_f32(const Mat& m) {
    MatT<float> f{m.ideal, float(m.gamma), float(m.rho0), float(m.a), float(m.b), float(m.A), float(m.B),
                  float(m.alpha), float(m.beta), float(m.u0), float(m.uiv), float(m.ucv), float(m.G), float(m.Y),
                  float(m.Emod), float(m.wm), float(m.wk)};
    mat_derive(f);
    return f;
}

// Settings + material + grid geometry, passed by value to every kernel.
struct P {
    Mat m;
    MatT<float> mf;  // the material rounded to FP32 once on the host (for the FP32 form)
    // settings the FP32 form reads, rounded to FP32 once on the host (ymi: y_m - y_i0)
    struct {
        float y_i0, mu_i, ymi, y_d0, mu_d, y_m, y_bingham, c_reg, eps_act, dx, invdx, rho_vac;
    } cf;
    double gz, tdec, eta_af, c_act, p_coh, p_act, rho_cfl, damp, rho_vac;
    double y_i0, mu_i, mu_d, y_d0, y_m, y_bingham, c_reg, af_sat;
    int32_t axisym, rock, af_reg, af_prel, af_seeddp;
    int32_t nx, ny, nz;
    int32_t flat;  // bit a: one cell along axis a, so its two face fluxes are equal and every
                   // difference along it is zero: no sweep (not the cylindrical r axis)
    int64_t n;
    double dx, invdx, id2;  // cell width, 1 / dx, 1 / dx^2
    DivBy<double> d_dx, d_3;  // divisors dx and 3
    double eps_act;  // weakest-flaw activation strain, formed on the host as in hydro_cpu.cpp:254
    // hydrostatic reference of set_ref (hydro_cpu.cpp:259-261), null when off:
    // the well-balanced z-sweep and gravity source and the void-cell reset
    const double* ref_r0;
    const double* ref_p0;
    const double* ref_pf;  // reference pressure at every z-face (zero internal energy, clamped at 0)
    const double* ref_dp;  // per cell p0(top face) - p0(bottom face) of the well-balanced gravity source
    double void_amb;  // VOID_AMB: void cells reset to this density instead of the reference's
    int32_t void_cons;  // VOID_CONS: the reset moves the excess mass to a neighbour first
    int32_t visc_imp;   // VISC_IMP: fluidization viscosity by the implicit solve, not in the Lop
};

// The material in the compute type R: FP64 as given, FP32 as rounded once on
// the host (the same values a per-thread conversion gives, without the
// per-thread conversions, which run on the FP64 pipe).
template <class R>
__device__ __forceinline__ MatT<R> mat_of(const P& p) {
    if constexpr (sizeof(R) == 4) return p.mf;
    else return p.m;
}

// A setting in the compute type R: FP64 as given, FP32 as rounded on the host.
#define EU_SETTING(R, name) (sizeof(R) == 4 ? R(p.cf.name) : R(p.name))

// x in the compute type R (FP64: x itself) and back to FP64.  The FP32 form
// converts on the integer pipes: its Runge-Kutta kernels wait on the FP64 pipe
// (a conversion takes an FP64 instruction's 64 cycles there).
template <class R>
__device__ __forceinline__ R narrow(double x) {
    if constexpr (sizeof(R) == 4) return fi::to_float(x);
    else return x;
}
__device__ __forceinline__ double widen(float y) { return fi::to_double(y); }
__device__ __forceinline__ double widen(double y) { return y; }

template <class R> __device__ __forceinline__ R dmax2(R a, R b) { return lt(a, b) ? b : a; }  // std::max
template <class R> __device__ __forceinline__ R dmin2(R a, R b) { return lt(b, a) ? b : a; }  // std::min

// The FP32 form's equation of state.

// Tillotson pressure, eos.hpp:52-63.
static __device__ float till(const MatT<float>& m, float rho, float u) {
    if (rho <= 0.0f) return 0.0f;
    float eta = rho / m.rho0, mu = eta - 1.0f;
    float w0 = u / (m.u0 * eta * eta) + 1.0f;
    float Pc = (m.a + m.b / w0) * rho * u + m.A * mu + m.B * mu * mu;
    if (rho >= m.rho0 || u <= m.uiv) return Pc;
    float z = m.rho0 / rho - 1.0f;
    float Pe = m.a * rho * u + (m.b * rho * u / w0 + m.A * mu * exp(-m.beta * z)) * exp(-m.alpha * z * z);
    if (u >= m.ucv) return Pe;
    return ((u - m.uiv) * Pe + (m.ucv - u) * Pc) / (m.ucv - m.uiv);
}

static __device__ __forceinline__ float pressure(const MatT<float>& m, float rho, float u) {  // eos.hpp:65-68
    if (m.ideal) return (m.gamma - 1.0f) * rho * u;
    return till(m, rho, u);
}

// Condensed-branch value and analytic derivatives, eos.hpp:72-79.
static __device__ void cond_d(const MatT<float>& m, float rho, float u, float& P, float& dPdr, float& dPdu) {
    float eta = rho / m.rho0, mu = eta - 1.0f;
    float w = 1.0f + u / (m.u0 * eta * eta), aob = m.a + m.b / w;
    P = aob * rho * u + m.A * mu + m.B * mu * mu;
    dPdu = aob * rho - m.b * rho * u / (w * w * m.u0 * eta * eta);
    float dwdr = -2.0f * u / (m.u0 * eta * eta * eta * m.rho0);
    dPdr = aob * u + rho * u * (-m.b / (w * w)) * dwdr + m.A / m.rho0 + 2.0f * m.B * mu / m.rho0;
}

// Expanded-branch value and analytic derivatives, eos.hpp:80-94.
static __device__ void expd_d(const MatT<float>& m, float rho, float u, float& P, float& dPdr, float& dPdu) {
    float eta = rho / m.rho0, mu = eta - 1.0f;
    float w = 1.0f + u / (m.u0 * eta * eta);
    float z = m.rho0 / rho - 1.0f, dzdr = -m.rho0 / (rho * rho);
    float E1 = exp(-m.alpha * z * z), E2 = exp(-m.beta * z);
    float G = m.b * rho * u / w + m.A * mu * E2;
    P = m.a * rho * u + G * E1;
    float dwdr = -2.0f * u / (m.u0 * eta * eta * eta * m.rho0);
    float dGu = m.b * rho / w - m.b * rho * u / (w * w * m.u0 * eta * eta);
    dPdu = m.a * rho + dGu * E1;
    float dbruw_dr = m.b * u / w + m.b * rho * u * (-1.0f / (w * w)) * dwdr;
    float dGr = dbruw_dr + m.A * E2 / m.rho0 + m.A * mu * (E2 * (-m.beta) * dzdr);
    float dE1dr = E1 * (-m.alpha * 2.0f * z) * dzdr;
    dPdr = m.a * u + dGr * E1 + G * dE1dr;
}

// Analytic sound speed, eos.hpp:95-113.
static __device__ float sound_speed(const MatT<float>& m, float rho, float u) {
    if (m.ideal) {
        float Pi = (m.gamma - 1.0f) * rho * u;
        return sqrt(dmax2(m.gamma * Pi / dmax2(rho, 1e-30f), 1e-12f));
    }
    if (rho <= 0.0f) return 1e-3f;
    float Pp, dPdr, dPdu;
    if (rho >= m.rho0 || u <= m.uiv) {
        cond_d(m, rho, u, Pp, dPdr, dPdu);
    } else if (u >= m.ucv) {
        expd_d(m, rho, u, Pp, dPdr, dPdu);
    } else {
        float Pc, dPcr, dPcu, Pe, dPer, dPeu;
        cond_d(m, rho, u, Pc, dPcr, dPcu);
        expd_d(m, rho, u, Pe, dPer, dPeu);
        float inv = 1.0f / (m.ucv - m.uiv);
        Pp = ((u - m.uiv) * Pe + (m.ucv - u) * Pc) * inv;
        dPdu = ((Pe + (u - m.uiv) * dPeu) + (-Pc + (m.ucv - u) * dPcu)) * inv;
        dPdr = ((u - m.uiv) * dPer + (m.ucv - u) * dPcr) * inv;
    }
    return sqrt(dmax2(dPdr + Pp / (rho * rho) * dPdu, 1e-6f));
}

// hydro_cpu.cpp:38: pressure clamped at 0 and the sound speed.
static __device__ __forceinline__ void eos_pc(const MatT<float>& m, float rho, float e, float& p, float& cs) {
    p = pressure(m, rho, e);
    if (p < 0.0f) p = 0.0f;
    cs = sound_speed(m, rho, e);
}

// The FP64 form's: the same expressions, each operation the reference's.

// Tillotson pressure, eos.hpp:52-63.
static __device__ double till(const MatT<double>& m, double rho, double u) {
    if (le0(rho)) return 0.0;
    double eta = dv(rho, m.d_rho0), mu = eta - 1.0;
    double w0 = dv(u, m.u0 * eta * eta) + 1.0;
    double Pc = (m.a + dv(m.b, w0)) * rho * u + m.A * mu + m.B * mu * mu;
    if (ge(rho, m.rho0) || ge(m.uiv, u)) return Pc;
    double z = dv(m.rho0, rho) - 1.0;
    double Pe = m.a * rho * u + (dv(m.b * rho * u, w0) + m.A * mu * exp(-m.beta * z)) * exp(-m.alpha * z * z);
    if (ge(u, m.ucv)) return Pe;
    return dv((u - m.uiv) * Pe + (m.ucv - u) * Pc, m.d_uv);
}

static __device__ __forceinline__ double pressure(const MatT<double>& m, double rho, double u) {  // eos.hpp:65-68
    if (m.ideal) return (m.gamma - 1.0) * rho * u;
    return till(m, rho, u);
}

// hydro_cpu.cpp:38: pressure clamped at 0 and the sound speed, in one pass:
// Tillotson pressure (eos.hpp:52-63), the condensed and expanded branches'
// values and analytic derivatives (72-94) and the sound speed (95-113) share
// their subexpressions, each formed by the reference's operations.
static __device__ void eos_pc(const MatT<double>& m, double rho, double u, double& p, double& cs) {
    if (m.ideal) {
        const double Pi = (m.gamma - 1.0) * rho * u;
        cs = root(dmax2(dv(m.gamma * Pi, dmax2(rho, 1e-30)), 1e-12));
        p = lt0(Pi) ? 0.0 : Pi;
        return;
    }
    if (le0(rho)) {
        p = 0.0;
        cs = 1e-3;
        return;
    }
    const double eta = dv(rho, m.d_rho0), mu = eta - 1.0;
    const double ue2 = m.u0 * eta * eta;
    const double w = dv(u, ue2) + 1.0, aob = m.a + dv(m.b, w), ar = aob * rho;
    const double Pc = ar * u + m.A * mu + m.B * mu * mu;
    const double bru = m.b * rho * u, ww = w * w;
    const double bt = dv(bru, ww * m.u0 * eta * eta);
    const double dwdr = dv(-2.0 * u, ue2 * eta * m.rho0);
    const double Cu = ar - bt;
    const double Cr = aob * u + rho * u * dv(-m.b, ww) * dwdr + m.A_rho0 + dv(m.B2 * mu, m.d_rho0);
    double P, Pp, dPdr, dPdu;  // P as eos.hpp:52-63 gives it, Pp as the sound speed's own value
    if (ge(rho, m.rho0) || ge(m.uiv, u)) {
        P = Pp = Pc;
        dPdr = Cr;
        dPdu = Cu;
    } else {
        const double z = dv(m.rho0, rho) - 1.0, dzdr = dv(-m.rho0, rho * rho);
        const double E1 = exp(-m.alpha * z * z), E2 = exp(-m.beta * z);
        const double G = dv(bru, w) + m.A * mu * E2;
        const double Pe = m.a * rho * u + G * E1;
        const double Eu = m.a * rho + (dv(m.b * rho, w) - bt) * E1;
        const double dbruw_dr = dv(m.b * u, w) + bru * dv(-1.0, ww) * dwdr;
        const double dGr = dbruw_dr + dv(m.A * E2, m.d_rho0) + m.A * mu * (E2 * (-m.beta) * dzdr);
        const double Er = m.a * u + dGr * E1 + G * (E1 * (-m.alpha * 2.0 * z) * dzdr);
        if (ge(u, m.ucv)) {
            P = Pp = Pe;
            dPdr = Er;
            dPdu = Eu;
        } else {
            const double x = (u - m.uiv) * Pe + (m.ucv - u) * Pc;
            P = dv(x, m.d_uv);
            Pp = x * m.iuv;
            dPdu = ((Pe + (u - m.uiv) * Eu) + (-Pc + (m.ucv - u) * Cu)) * m.iuv;
            dPdr = ((u - m.uiv) * Er + (m.ucv - u) * Cr) * m.iuv;
        }
    }
    cs = root(dmax2(dPdr + dv(Pp, rho * rho) * dPdu, 1e-6));
    p = lt0(P) ? 0.0 : P;
}

// ---------------------------------------------------------------- face flux

template <class R>
struct F5 {
    R r, mn, mt1, mt2, E;
};

template <class R>
__device__ __forceinline__ F5<R> flux_of(R r, R vn, R t1, R t2, R p, R E) {
    return F5<R>{r * vn, r * vn * vn + p, r * vn * t1, r * vn * t2, (E + p) * vn};
}

// FP32 fluxes.

// Exact rarefaction into vacuum sampled at the face, hydro_cpu.cpp:43-53.
static __device__ F5<float> vac_flux(const MatT<float>& m, float rM, float vnM, float t1M, float t2M, float eM, int side) {
    float pM, cM;
    eos_pc(m, rM, eM, pM, cM);
    float g = rM * cM * cM / dmax2(pM, 1e-30f);
    if (g < 1.01f) g = 1.01f;
    if (g > 1e5f) g = 1e5f;
    float s = (float)side, vn = s * vnM;
    if (vn - cM >= 0.0f) {
        float E = rM * eM + 0.5f * rM * (vnM * vnM + t1M * t1M + t2M * t2M);
        return F5<float>{rM * vnM, rM * vnM * vnM + pM, rM * vnM * t1M, rM * vnM * t2M, (E + pM) * vnM};
    }
    if (vn + 2.0f * cM / (g - 1.0f) <= 0.0f) return F5<float>{0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
    float u0 = 2.0f / (g + 1.0f) * (cM + 0.5f * (g - 1.0f) * vn), c0 = u0;
    float r0 = rM * pow(c0 / cM, 2.0f / (g - 1.0f)), p0 = pM * pow(r0 / rM, g), e0 = p0 / ((g - 1.0f) * r0),
      un0 = s * u0;
    float E0 = r0 * e0 + 0.5f * r0 * (un0 * un0 + t1M * t1M + t2M * t2M);
    return F5<float>{r0 * un0, r0 * un0 * un0 + p0, r0 * un0 * t1M, r0 * un0 * t2M, (E0 + p0) * un0};
}

static __device__ __forceinline__ F5<float> hllc_star(float r, float vn, float t1, float t2, float p, float E, float S, float Ss, F5<float> Fk) {
    float f = r * (S - vn) / (S - Ss);
    F5<float> Us{f, f * Ss, f * t1, f * t2, f * (E / r + (Ss - vn) * (Ss + p / (r * (S - vn))))};
    F5<float> U{r, r * vn, r * t1, r * t2, E};
    return F5<float>{Fk.r + S * (Us.r - U.r), Fk.mn + S * (Us.mn - U.mn), Fk.mt1 + S * (Us.mt1 - U.mt1),
                 Fk.mt2 + S * (Us.mt2 - U.mt2), Fk.E + S * (Us.E - U.E)};
}

// HLLC, hydro_cpu.cpp:54-74.
static __device__ F5<float> hllc(const MatT<float>& m, float rho_vac, float rL, float vnL, float t1L, float t2L, float eL, float rR, float vnR, float t1R, float t2R,
                      float eR) {
    if (rho_vac > 0.0f) {
        bool vL = rL < rho_vac, vR = rR < rho_vac;
        if (vL && vR) return F5<float>{0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
        if (vR) return vac_flux(m, rL, vnL, t1L, t2L, eL, +1);
        if (vL) return vac_flux(m, rR, vnR, t1R, t2R, eR, -1);
    }
    float pL, cL, pR, cR;
    eos_pc(m, rL, eL, pL, cL);
    eos_pc(m, rR, eR, pR, cR);
    float SL = dmin2(vnL - cL, vnR - cR), SR = dmax2(vnL + cL, vnR + cR);
    float Ss = (pR - pL + rL * vnL * (SL - vnL) - rR * vnR * (SR - vnR)) / (rL * (SL - vnL) - rR * (SR - vnR));
    float EL = rL * eL + 0.5f * rL * (vnL * vnL + t1L * t1L + t2L * t2L),
      ER = rR * eR + 0.5f * rR * (vnR * vnR + t1R * t1R + t2R * t2R);
    if (SL >= 0.0f) return flux_of(rL, vnL, t1L, t2L, pL, EL);
    if (SR <= 0.0f) return flux_of(rR, vnR, t1R, t2R, pR, ER);
    if (Ss >= 0.0f) return hllc_star(rL, vnL, t1L, t2L, pL, EL, SL, Ss, flux_of(rL, vnL, t1L, t2L, pL, EL));
    return hllc_star(rR, vnR, t1R, t2R, pR, ER, SR, Ss, flux_of(rR, vnR, t1R, t2R, pR, ER));
}

// HLLC with the face pressures given (the well-balanced z-sweep), hydro_cpu.cpp:75-88.
static __device__ F5<float> hllc_p(const MatT<float>& m, float rL, float vnL, float t1L, float t2L, float eL, float pL, float rR, float vnR, float t1R, float t2R, float eR,
                        float pR) {
    float cL = sound_speed(m, rL, eL), cR = sound_speed(m, rR, eR);
    if (pL < 0.0f) pL = 0.0f;
    if (pR < 0.0f) pR = 0.0f;
    float SL = dmin2(vnL - cL, vnR - cR), SR = dmax2(vnL + cL, vnR + cR);
    float Ss = (pR - pL + rL * vnL * (SL - vnL) - rR * vnR * (SR - vnR)) / (rL * (SL - vnL) - rR * (SR - vnR));
    float EL = rL * eL + 0.5f * rL * (vnL * vnL + t1L * t1L + t2L * t2L),
      ER = rR * eR + 0.5f * rR * (vnR * vnR + t1R * t1R + t2R * t2R);
    if (SL >= 0.0f) return flux_of(rL, vnL, t1L, t2L, pL, EL);
    if (SR <= 0.0f) return flux_of(rR, vnR, t1R, t2R, pR, ER);
    if (Ss >= 0.0f) return hllc_star(rL, vnL, t1L, t2L, pL, EL, SL, Ss, flux_of(rL, vnL, t1L, t2L, pL, EL));
    return hllc_star(rR, vnR, t1R, t2R, pR, ER, SR, Ss, flux_of(rR, vnR, t1R, t2R, pR, ER));
}

// FP64 fluxes.

// Exact rarefaction into vacuum sampled at the face, hydro_cpu.cpp:43-53.
static __device__ F5<double> vac_flux(const MatT<double>& m, double rM, double vnM, double t1M, double t2M, double eM, int side) {
    double pM, cM;
    eos_pc(m, rM, eM, pM, cM);
    double g = dv(rM * cM * cM, dmax2(pM, 1e-30));
    if (lt(g, 1.01)) g = 1.01;
    if (lt(1e5, g)) g = 1e5;
    double s = (double)side, vn = s * vnM;
    if (ge0(vn - cM)) {
        double E = rM * eM + 0.5 * rM * (vnM * vnM + t1M * t1M + t2M * t2M);
        return F5<double>{rM * vnM, rM * vnM * vnM + pM, rM * vnM * t1M, rM * vnM * t2M, (E + pM) * vnM};
    }
    if (le0(vn + dv(2.0 * cM, g - 1.0))) return F5<double>{0.0, 0.0, 0.0, 0.0, 0.0};
    double u0 = dv(2.0, g + 1.0) * (cM + 0.5 * (g - 1.0) * vn), c0 = u0;
    double r0 = rM * pow(dv(c0, cM), dv(2.0, g - 1.0)), p0 = pM * pow(dv(r0, rM), g), e0 = dv(p0, (g - 1.0) * r0),
      un0 = s * u0;
    double E0 = r0 * e0 + 0.5 * r0 * (un0 * un0 + t1M * t1M + t2M * t2M);
    return F5<double>{r0 * un0, r0 * un0 * un0 + p0, r0 * un0 * t1M, r0 * un0 * t2M, (E0 + p0) * un0};
}

// The HLLC flux of given face states, pressures and sound speeds,
// hydro_cpu.cpp:54-74 and 75-88.  The flux needs one side only -- which, the
// wave speeds say -- so the side is chosen first and its terms are formed once
// (warps with faces of both signs then do not run both).
static __device__ __forceinline__ F5<double> hllc_pc(double rL, double vnL, double t1L, double t2L, double eL, double pL, double cL, double rR, double vnR, double t1R, double t2R, double eR,
                                         double pR, double cR) {
    const double SL = dmin2(vnL - cL, vnR - cR), SR = dmax2(vnL + cL, vnR + cR);
    const double mL = rL * (SL - vnL), mR = rR * (SR - vnR);  // r (S - vn)
    const double Ss = dv(pR - pL + rL * vnL * (SL - vnL) - rR * vnR * (SR - vnR), mL - mR);
    const bool fromL = ge0(SL), fromR = le0(SR);
    const bool left = fromL || (!fromR && ge0(Ss));
    const double r = left ? rL : rR, vn = left ? vnL : vnR, t1 = left ? t1L : t1R, t2 = left ? t2L : t2R;
    const double e = left ? eL : eR, p = left ? pL : pR, S = left ? SL : SR, mS = left ? mL : mR;
    const double E = r * e + half(r) * (vn * vn + t1 * t1 + t2 * t2);
    F5<double> F = flux_of(r, vn, t1, t2, p, E);
    if (fromL || fromR) return F;
    const double f = dv(mS, S - Ss);
    const F5<double> Us{f, f * Ss, f * t1, f * t2, f * (dv(E, r) + (Ss - vn) * (Ss + dv(p, mS)))};
    return F5<double>{F.r + S * (Us.r - r), F.mn + S * (Us.mn - r * vn), F.mt1 + S * (Us.mt1 - r * t1),
                 F.mt2 + S * (Us.mt2 - r * t2), F.E + S * (Us.E - E)};
}

// HLLC, hydro_cpu.cpp:54-74.
static __device__ F5<double> hllc(const MatT<double>& m, double rho_vac, double rL, double vnL, double t1L, double t2L, double eL, double rR, double vnR, double t1R, double t2R,
                      double eR) {
    if (rho_vac > 0.0) {
        bool vL = lt(rL, rho_vac), vR = lt(rR, rho_vac);
        if (vL && vR) return F5<double>{0.0, 0.0, 0.0, 0.0, 0.0};
        if (vR) return vac_flux(m, rL, vnL, t1L, t2L, eL, +1);
        if (vL) return vac_flux(m, rR, vnR, t1R, t2R, eR, -1);
    }
    double pL, cL, pR, cR;
    eos_pc(m, rL, eL, pL, cL);
    eos_pc(m, rR, eR, pR, cR);
    return hllc_pc(rL, vnL, t1L, t2L, eL, pL, cL, rR, vnR, t1R, t2R, eR, pR, cR);
}

// HLLC with the face pressures given (the well-balanced z-sweep), hydro_cpu.cpp:75-88.
static __device__ F5<double> hllc_p(const MatT<double>& m, double rL, double vnL, double t1L, double t2L, double eL, double pL, double rR, double vnR, double t1R, double t2R, double eR,
                        double pR) {
    double q, cL, cR;
    eos_pc(m, rL, eL, q, cL);
    eos_pc(m, rR, eR, q, cR);
    if (lt0(pL)) pL = 0.0;
    if (lt0(pR)) pR = 0.0;
    return hllc_pc(rL, vnL, t1L, t2L, eL, pL, cL, rR, vnR, t1R, t2R, eR, pR, cR);
}

__device__ __forceinline__ float mm(float a, float b) {  // minmod, hydro_cpu.cpp:89
    return (a * b <= 0.0f) ? 0.0f : (fabsf(a) < fabsf(b) ? a : b);
}
__device__ __forceinline__ double mm(double a, double b) { return fi::minmod(a, b); }

// ---------------------------------------------------------------- state

enum { F_R, F_MU, F_MV, F_MW, F_E, F_SXX, F_SYY, F_SZZ, F_SXY, F_SXZ, F_SYZ, F_D, F_AF, F_RC, F_VIB, F_PMAX, NF };
// Runge-Kutta fields (hydro_cpu.cpp:413-417) and the right-hand side, same order.
enum { D_R, D_MU, D_MV, D_MW, D_E, D_SXX, D_SYY, D_SZZ, D_SXY, D_SXZ, D_SYZ, D_D, D_RC, D_VIB, ND };
__host__ __device__ constexpr int rk_field(int q) {  // r .. Syz, D keep their index; rc, vib follow af
    return q <= D_D ? q : (q == D_RC ? F_RC : F_VIB);
}
inline const char* const kFieldNames[NF] = {"r", "mu", "mv", "mw", "E", "Sxx", "Syy", "Szz",
                                      "Sxy", "Sxz", "Syz", "D", "af", "rc", "vib", "Pmax"};
inline const char* const kRhsNames[ND] = {"r", "mu", "mv", "mw", "E", "Sxx", "Syy", "Szz", "Sxy", "Sxz", "Syz", "D", "rc", "vib"};

// One state of the grid: the 16 fields (a predictor state aliases af and Pmax
// of the state it was formed from).
struct Fields {
    double* q[NF];
};
template <class R>
struct RhsT {  // the right-hand side in the Lop's compute type (FP32 form: FP32, summed there)
    R* q[ND];
};
template <class R>
struct PrimT {  // rho, vx, vy, vz, e, rc/rho in the Lop's compute type, and (with a
    R* w[7];    // reference state) the pressure deviation Pcell - REF_P0 formed in FP64
    // Sxx Syy Szz Sxy Sxz Syz D vib as the right-hand side reads them: in FP64
    // the state's own arrays; in FP32 copies converted once per Lop by k_prim
    // (the same values the conversion at every stencil read gave)
    R* sq[8];
    uint8_t* vd;  // FP32 form: near-void flag per cell (rho < RHO_CFL), formed in FP64
};
template <class R>
struct FacesT {  // per direction: mass, normal / tangential momentum, energy, tracer fluxes
    R* q[3][6];
};

// Device-resident step control (the drivers' loop of hydro_cpu.cpp:452).
struct Ctl {
    double dt, t, t_end, cfl;
    int64_t steps, max_steps;
    int32_t active;
    unsigned int done;  // blocks of the speed reduction that have finished
    double af_dec;  // exp(-dt / TDEC) of this step (fluidization decay)
    unsigned long long smax_bits;  // CFL speed of this step (positive doubles order as their bits)
    // implicit viscosity: grid barrier of its persistent launch, a wait that
    // ran out (error), conjugate-gradient iterations so far
    unsigned int bar_count;
    int32_t visc_err;  // bar_count and visc_err are cleared together before each launch
    unsigned int bar_gen;
    int32_t pad2;
    long long visc_iters;
};

static __device__ __forceinline__ int64_t gtid() { return (int64_t)blockIdx.x * blockDim.x + threadIdx.x; }

// hydro_cpu.cpp:94-95
static __device__ __forceinline__ double eint_of(double r, double mu, double mv, double mw, double E) {
    const DivBy<double> d = div_by(r);
    const double ke = dv(half(mu * mu + mv * mv + mw * mw), d);
    return dv(E - ke, d);
}
static __device__ __forceinline__ double pcell(const P& p, const Fields& s, int64_t c) {
    double pr, cs;
    const double r = s.q[F_R][c];
    eos_pc(p.m, r, eint_of(r, s.q[F_MU][c], s.q[F_MV][c], s.q[F_MW][c], s.q[F_E][c]), pr, cs);
    return pr;
}

// One cell's fields in registers.  The per-cell kernels load every field
// before they store one: the columns may alias as far as the compiler knows, so
// a store between two fields' loads makes the second wait for the first
// (256^3-class grids, FP32 form, 160^3: predictor with the primitives 0.53 ->
// 0.38 ms, corrector 0.53 -> 0.39 ms).
struct Cell {
    double q[NF];
};
template <class... Q>
static __device__ __forceinline__ void load_cell(Cell& x, const Fields& s, int64_t c, Q... q) {
    ((x.q[q] = s.q[q][c]), ...);
}
template <class... Q>
static __device__ __forceinline__ void store_cell(const Cell& x, const Fields& s, int64_t c, Q... q) {
    ((s.q[q][c] = x.q[q]), ...);
}
#define EU_HYDRO F_R, F_MU, F_MV, F_MW, F_E
#define EU_STRESS F_SXX, F_SYY, F_SZZ, F_SXY, F_SXZ, F_SYZ
#define EU_RK EU_HYDRO, EU_STRESS, F_D, F_RC, F_VIB

// Acoustic fluidization of one cell, hydro_cpu.cpp:390-410.
// dec = exp(-dt / TDEC), the same for every cell.
static __device__ __forceinline__ void update_af_cell(const P& p, Cell& x, double dec) {
    const double r = x.q[F_R], mu = x.q[F_MU], mv = x.q[F_MV], mw = x.q[F_MW];
    const double e = eint_of(r, mu, mv, mw, x.q[F_E]);
    double Pc, cs;  // Pcell and MAT.sound_speed of the cell
    eos_pc(p.m, r, e, Pc, cs);
    if (lt(x.q[F_PMAX], Pc)) {
        const double dP = Pc - x.q[F_PMAX];
        x.q[F_PMAX] = Pc;
        if (lt(p.p_act, dP)) {
            const double sp = p.af_seeddp ? dv(dP, dmax2(r, 1e-30) * dmax2(cs, 1e-30))
                                          : dv(root(mu * mu + mv * mv + mw * mw), dmax2(r, 1e-30));
            x.q[F_VIB] = dmax2(x.q[F_VIB], p.c_act * sp);
        }
    }
    const double v0 = x.q[F_VIB];
    x.q[F_VIB] = v0 * dec;
    const double pov = dmax2(Pc, p.p_coh);
    if (p.af_reg) {
        if (lt(dmax2(p.rho_cfl, 1e-12), r)) x.q[F_E] += 0.5 * r * (v0 * v0 - x.q[F_VIB] * x.q[F_VIB]);
        const double vcap = dv(p.af_sat * pov, dmax2(r, 1e-30) * dmax2(cs, 1e-30));
        if (lt(vcap, x.q[F_VIB])) x.q[F_VIB] = vcap;
    }
    const double pvib = r * cs * x.q[F_VIB];
    x.q[F_AF] = dv(pvib, pvib + pov);
}

// Specific internal energy for an EOS evaluated in R: FP64, the reference's
// two quotients (eint_of); FP32, one FP64 reciprocal of rho (E - ke cancels in
// kinetic-dominated cells, so the difference stays FP64), the result rounded
// to FP32 by the caller.
template <class R>
static __device__ __forceinline__ double eint_r(double r, double mu, double mv, double mw, double E) {
    if constexpr (sizeof(R) == 8) {
        return eint_of(r, mu, mv, mw, E);
    } else {
        const double inv = fi::div(1.0, r);
        return (E - 0.5 * (mu * mu + mv * mv + mw * mw) * inv) * inv;
    }
}

// Pcell (hydro_cpu.cpp:95) with the EOS evaluated in R: the clamped pressure.
template <class R>
static __device__ __forceinline__ R pcell_r(const P& p, const Cell& x) {
    const double r = x.q[F_R];
    R pr = pressure(mat_of<R>(p), narrow<R>(r),
                    narrow<R>(eint_r<R>(r, x.q[F_MU], x.q[F_MV], x.q[F_MW], x.q[F_E])));
    return lt0(pr) ? R(0) : pr;
}

// A cell's Pcell formed at most once per state and shared by the damage
// growth and the radial return that follow each other in a stage (damage
// growth changes only D, so both see the same pressure).
template <class R>
struct PcellOnce {
    bool have = false;
    R v = R(0);
    __device__ __forceinline__ R get(const P& p, const Cell& x) {
        if (!have) {
            v = pcell_r<R>(p, x);
            have = true;
        }
        return v;
    }
};

// Radial return of one cell, hydro_cpu.cpp:229-252 (s: the stress / energy /
// vibration state; af from the state the step started from).  The yield
// surface and the return factor are formed in R; the state stays FP64.
template <class R>
static __device__ __forceinline__ void vonmises_cell(const P& p, Cell& x, double af, bool reg, PcellOnce<R>& pc) {
    if (p.m.Y <= 0 && !p.rock) return;
    R Y;
    const double r = x.q[F_R];
    const R afc = narrow<R>(af);
    if (p.rock) {
        R Peff;
        if (p.af_prel && gt0(x.q[F_VIB])) {
            R p2, cs2;  // Pcell and the sound speed
            eos_pc(mat_of<R>(p), narrow<R>(r),
                   narrow<R>(eint_r<R>(r, x.q[F_MU], x.q[F_MV], x.q[F_MW], x.q[F_E])), p2, cs2);
            Peff = dmax2(dmax2(p2, R(0)) - narrow<R>(r) * cs2 * narrow<R>(x.q[F_VIB]), R(0));
        } else {
            Peff = dmax2(pc.get(p, x), R(0));
        }
        const R mu_i = EU_SETTING(R, mu_i);
        const R ymi = sizeof(R) == 4 ? R(p.cf.ymi) : R(p.y_m - p.y_i0);
        const R mP = mu_i * Peff;
        R Yi = EU_SETTING(R, y_i0) + dv(mP, R(1) + dv(mP, dmax2(ymi, R(1))));
        R Yd = dmin2(EU_SETTING(R, y_d0) + EU_SETTING(R, mu_d) * Peff, EU_SETTING(R, y_m));
        const R D = narrow<R>(x.q[F_D]);
        R Yb = (R(1) - D) * Yi + D * Yd;
        Y = p.af_prel ? Yb : Yb * (R(1) - afc);
        if (p.y_bingham > 0 && lt(R(1e-3), afc)) {
            R Yf = dmin2(EU_SETTING(R, y_bingham), Yb);
            if (lt(Y, Yf)) Y = Yf;
        }
    } else {
        Y = (R(1) - narrow<R>(x.q[F_D])) * (R(1) - afc) * mat_of<R>(p).Y;
    }
    const double sxx = x.q[F_SXX], syy = x.q[F_SYY], szz = x.q[F_SZZ], sxy = x.q[F_SXY],
                 sxz = x.q[F_SXZ], syz = x.q[F_SYZ];
    const R xx = narrow<R>(sxx), yy = narrow<R>(syy), zz = narrow<R>(szz), xy = narrow<R>(sxy),
            xz = narrow<R>(sxz), yz = narrow<R>(syz);
    R J2 = half(xx * xx + yy * yy + zz * zz) + xy * xy + xz * xz + yz * yz;
    R vm = root(R(3) * J2);
    if (lt(Y, vm)) {
        const double f = widen(gt0(vm) ? dv(Y, vm) : R(0));
        x.q[F_SXX] = sxx * f; x.q[F_SYY] = syy * f; x.q[F_SZZ] = szz * f;
        x.q[F_SXY] = sxy * f; x.q[F_SXZ] = sxz * f; x.q[F_SYZ] = syz * f;
        if (p.af_reg && reg && p.m.G > 0 && (p.rho_cfl <= 0 || lt(p.rho_cfl, r))) {
            R dW = dv(vm * vm - Y * Y, R(6) * mat_of<R>(p).G);
            const R vb = narrow<R>(x.q[F_VIB]);
            x.q[F_VIB] = widen(root(vb * vb + dv(R(2) * EU_SETTING(R, c_reg) * dW, narrow<R>(r))));
            x.q[F_E] -= widen(EU_SETTING(R, c_reg) * dW);
        }
    }
}

// Tensile damage growth of one cell, hydro_cpu.cpp:253-258 (threshold and
// growth formed in R).
template <class R>
static __device__ __forceinline__ void grow_damage_cell(const P& p, Cell& x, double dt, PcellOnce<R>& pc) {
    if (p.m.Emod <= 0 || p.m.wk <= 0) return;
    const double D = x.q[F_D];
    if (ge(D, 1.0)) return;
    const R Pp = pc.get(p, x);
    const R sigmax = dmax2(-Pp + narrow<R>(x.q[F_SXX]),
                           dmax2(-Pp + narrow<R>(x.q[F_SYY]), -Pp + narrow<R>(x.q[F_SZZ])));
    if (gt0(sigmax) && lt(EU_SETTING(R, eps_act), dv(sigmax, mat_of<R>(p).d_Emod))) {
        R cg = R(0.4) * root(dv(mat_of<R>(p).Emod, dmax2(narrow<R>(x.q[F_R]), R(1e-30)))),
          Rs = R(0.5) * EU_SETTING(R, dx);
        R d13 = pow(narrow<R>(D), R(1) / R(3)) + dv(cg, Rs) * narrow<R>(dt);
        x.q[F_D] = widen(dmin2(R(1), d13 * d13 * d13));
    }
}


// ---------------------------------------------------------------- kernels

// Is there a step to take (drivers' loop)?  Also clears the speed.
static __device__ __forceinline__ void next_step(Ctl* ctl) {
    ctl->active = (ctl->t < ctl->t_end && (ctl->max_steps < 0 || ctl->steps < ctl->max_steps)) ? 1 : 0;
    ctl->smax_bits = (unsigned long long)__double_as_longlong(1e-30);
}

// maxspeed (hydro_cpu.cpp:378-380): per-cell signal speed, block maximum, one
// atomic per block on the ordered bits.  The block that finishes last then
// forms the step (with_dt): dt = CFL dx / maxspeed, clipped at t_end
// (hydro_cpu.cpp:452), and the fluidization's decay over it.
template <class R>
static __global__ void __launch_bounds__(256) k_maxspeed(P p, Fields g, Ctl* ctl, int with_dt) {
    __shared__ double red[8];
    const int64_t c = gtid();
    double s = 1e-30;
    if (ctl->active && c < p.n) {
        const double r = g.q[F_R][c];
        if (!lt(r, p.rho_cfl)) {
            const double mu = g.q[F_MU][c], mv = g.q[F_MV][c], mw = g.q[F_MW][c];
            const R rr = narrow<R>(r);
            R pr, cs;
            eos_pc(mat_of<R>(p), rr, narrow<R>(eint_r<R>(r, mu, mv, mw, g.q[F_E][c])), pr, cs);
            const DivBy<R> d = div_by(rr);
            R cel = root(cs * cs + (p.m.G > 0 ? dv(R(4.0 / 3.0) * mat_of<R>(p).G, d) : R(0)));
            const R fu = narrow<R>(mu), fv = narrow<R>(mv), fw = narrow<R>(mw);
            R v = dv(root(fu * fu + fv * fv + fw * fw), d);
            s = dmax2(s, widen(v + cel));
        }
    }
    for (int o = 16; o > 0; o >>= 1) s = dmax2(s, __shfl_xor_sync(0xffffffffu, s, o));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x < 32) {
        s = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 1e-30;
        for (int o = 16; o > 0; o >>= 1) s = dmax2(s, __shfl_xor_sync(0xffffffffu, s, o));
        if (threadIdx.x == 0) {
            atomicMax(&ctl->smax_bits, (unsigned long long)__double_as_longlong(s));
            if (with_dt && ctl->active) {
                __threadfence();
                if (atomicAdd(&ctl->done, 1u) == gridDim.x - 1) {
                    ctl->done = 0;
                    __threadfence();
                    double dt = ctl->cfl * p.dx / __longlong_as_double((long long)atomicMax(&ctl->smax_bits, 0ull));
                    if (ctl->t + dt > ctl->t_end) dt = ctl->t_end - ctl->t;
                    ctl->dt = dt;
                    if (p.tdec > 0) ctl->af_dec = exp(-dt / p.tdec);
                }
            }
        }
    }
}

static __global__ void k_end(Ctl* ctl) {
    if (!ctl->active) return;
    ctl->t += ctl->dt;
    ctl->steps++;
    next_step(ctl);
}

// update_af as its own call (hydro_cpu.cpp:390-410).
static __global__ void k_update_af(P p, Fields g, const Ctl* ctl) {
    const int64_t c = gtid();
    if (c >= p.n || !ctl->active) return;
    Cell x;
    load_cell(x, g, c, EU_HYDRO, F_VIB, F_PMAX);
    const double pm = x.q[F_PMAX];
    update_af_cell(p, x, ctl->af_dec);
    store_cell(x, g, c, F_AF, F_VIB);
    if (lt(pm, x.q[F_PMAX])) store_cell(x, g, c, F_PMAX);
    if (p.af_reg) store_cell(x, g, c, F_E);
}

// Primitives of one state (hydro_cpu.cpp:101) and the tracer ratio rc/rho,
// formed in FP64 and stored in the Lop's compute type R.  FP64: the
// reference's quotients, one division each.  FP32: one FP64 reciprocal of
// rho, the velocities, kinetic energy and internal energy from it in FP64
// (E - ke cancels in kinetic-dominated cells), rounded to FP32; also the
// strength fields in FP32 and the near-void flags for the right-hand side.
template <class R>
static __device__ __forceinline__ void prim_cell(const P& p, const Cell& x, const PrimT<R>& W, int64_t c) {
    const double r = x.q[F_R], mu = x.q[F_MU], mv = x.q[F_MV], mw = x.q[F_MW];
    const double E = x.q[F_E], rc = x.q[F_RC];
    if constexpr (sizeof(R) == 4) {
        const double inv = fi::div(1.0, r), vx = mu * inv, vy = mv * inv, vz = mw * inv;
        const double e = (E - 0.5 * (mu * vx + mv * vy + mw * vz)) * inv;
        W.w[0][c] = narrow<R>(r);
        W.w[1][c] = narrow<R>(vx);
        W.w[2][c] = narrow<R>(vy);
        W.w[3][c] = narrow<R>(vz);
        W.w[4][c] = narrow<R>(e);
        W.w[5][c] = narrow<R>(rc * inv);
        if (p.ref_p0) {
            double pr = pressure(p.m, r, e);
            if (lt0(pr)) pr = 0;
            W.w[6][c] = narrow<R>(pr - p.ref_p0[c]);
        }
#pragma unroll
        for (int q = 0; q < 6; q++) W.sq[q][c] = narrow<R>(x.q[F_SXX + q]);
        W.sq[6][c] = narrow<R>(x.q[F_D]);
        W.sq[7][c] = narrow<R>(x.q[F_VIB]);
        W.vd[c] = (p.rho_cfl > 0 && lt(r, p.rho_cfl)) ? 1 : 0;
        return;
    }
    W.w[0][c] = R(r);
    const DivBy<double> d = div_by(r);  // one divisor for the cell's six quotients
    W.w[1][c] = R(dv(mu, d));
    W.w[2][c] = R(dv(mv, d));
    W.w[3][c] = R(dv(mw, d));
    const double e = dv(E - dv(half(mu * mu + mv * mv + mw * mw), d), d);
    W.w[4][c] = R(e);
    W.w[5][c] = R(dv(rc, d));
    if (p.ref_p0) {  // Pcell - REF_P0 (hydro_cpu.cpp:116)
        double pr = pressure(p.m, r, e);
        if (lt0(pr)) pr = 0;
        W.w[6][c] = R(pr - p.ref_p0[c]);
    }
}

// Primitives of the state a step starts from, after its update_af where the
// fluidization is on (hydro_cpu.cpp:412).
template <class R, bool AF>
static __global__ void k_prim(P p, Fields s, PrimT<R> W, const Ctl* ctl) {
    const int64_t c = gtid();
    if (c >= p.n || !ctl->active) return;
    Cell x;
    load_cell(x, s, c, EU_HYDRO, F_RC);
    if (sizeof(R) == 4) load_cell(x, s, c, EU_STRESS, F_D);
    if (sizeof(R) == 4 || AF) load_cell(x, s, c, F_VIB);
    if (AF) {
        load_cell(x, s, c, F_PMAX);
        const double pm = x.q[F_PMAX];
        update_af_cell(p, x, ctl->af_dec);
        store_cell(x, s, c, F_AF, F_VIB);
        if (lt(pm, x.q[F_PMAX])) store_cell(x, s, c, F_PMAX);
        if (p.af_reg) store_cell(x, s, c, F_E);
    }
    prim_cell<R>(p, x, W, c);
}

// Element i of a column of the compute type.  FP32: a 32-bit byte offset from
// the (uniform) base, so one offset serves every column at that cell and the
// address costs no 64-bit arithmetic (an FP32 column stays below 2^32 bytes:
// eu_create refuses larger grids, which no device memory holds).  Cell and face
// numbers are below 2^32 in both forms; 32-bit divisions find their indices.
__device__ __forceinline__ float at(const float* a, uint32_t i) {
    return *reinterpret_cast<const float*>(reinterpret_cast<const char*>(a) + i * 4u);
}
__device__ __forceinline__ double at(const double* a, uint32_t i) { return a[i]; }
__device__ __forceinline__ void put(float* a, uint32_t i, float x) {
    *reinterpret_cast<float*>(reinterpret_cast<char*>(a) + i * 4u) = x;
}
__device__ __forceinline__ void put(double* a, uint32_t i, double x) { a[i] = x; }

// Face geometry of direction DIR: number of faces and, for face id, the face
// position f along DIR and the cell of position p along DIR on its line.
template <int DIR>
struct FaceLine {
    uint32_t base, stride;  // cell(p) = base + p * stride
    int f, nL;
    __device__ __forceinline__ FaceLine(const P& p, uint32_t id) {
        if (DIR == 0) {
            const uint32_t plane = (uint32_t)p.ny * p.nz;
            f = (int)(id / plane);
            base = id - (uint32_t)f * plane;
            stride = plane;
            nL = p.nx;
        } else if (DIR == 1) {
            const uint32_t row = (uint32_t)(p.ny + 1) * p.nz;
            const uint32_t i = id / row, rem = id - i * row;
            f = (int)(rem / (uint32_t)p.nz);
            base = i * (uint32_t)p.ny * p.nz + (rem - (uint32_t)f * p.nz);
            stride = p.nz;
            nL = p.ny;
        } else {
            const uint32_t line = id / (uint32_t)(p.nz + 1);
            f = (int)(id - line * (uint32_t)(p.nz + 1));
            base = line * (uint32_t)p.nz;
            stride = 1;
            nL = p.nz;
        }
    }
    __device__ __forceinline__ uint32_t cell(int q) const { return base + (uint32_t)q * stride; }
};

template <int DIR>
__host__ __device__ __forceinline__ int64_t face_count(int nx, int ny, int nz) {
    return DIR == 0 ? (int64_t)(nx + 1) * ny * nz : (DIR == 1 ? (int64_t)nx * (ny + 1) * nz : (int64_t)nx * ny * (nz + 1));
}

// Face fluxes of direction DIR (hydro_cpu.cpp:109-121): MUSCL-minmod
// reconstruction of the primitives, floors, HLLC / vacuum flux, tracer flux
// upwinded by the mass flux.
template <int DIR, class R>
static __device__ __forceinline__ void face_one(const P& p, const PrimT<R>& W, const FacesT<R>& F, int64_t id0) {
    if (id0 >= face_count<DIR>(p.nx, p.ny, p.nz)) return;
    const uint32_t id = (uint32_t)id0;
    const FaceLine<DIR> ln(p, id);
    const int f = ln.f, nL = ln.nL;
    const int iL = max(0, f - 1), iR = min(nL - 1, f), iLL = max(0, f - 2), iRR = min(nL - 1, f + 1);
    const uint32_t cL = ln.cell(iL), cR = ln.cell(iR), cLL = ln.cell(iLL), cRR = ln.cell(iRR);
    R L[5], Rr[5];
#pragma unroll
    for (int q = 0; q < 5; q++) {
        const R* w = W.w[q];
        const R A = at(w, cL), B = at(w, cR), AA = at(w, cLL), BB = at(w, cRR);
        const R mid = B - A;
        L[q] = add_half(A, mm(A - AA, mid));
        Rr[q] = sub_half(B, mm(mid, BB - B));
        if (q == 0) {
            if (lt(L[0], R(1e-9))) L[0] = A;
            if (lt(Rr[0], R(1e-9))) Rr[0] = B;
        }
        if (q == 4) {
            if (lt0(L[4])) L[4] = A;
            if (lt0(Rr[4])) Rr[4] = B;
        }
    }
    constexpr int in = DIR == 0 ? 1 : (DIR == 1 ? 2 : 3), it1 = DIR == 0 ? 2 : 1, it2 = DIR == 2 ? 2 : 3;
    const MatT<R> m = mat_of<R>(p);
    F5<R> fl;
    if (DIR == 2 && p.ref_p0) {  // well-balanced: reconstruct the deviation from the reference (hydro_cpu.cpp:114-119)
        const R* dv = W.w[6];
        const R dLL = at(dv, cLL), dL = at(dv, cL), dR = at(dv, cR), dRR = at(dv, cRR);
        const R dLf = add_half(dL, mm(dL - dLL, dR - dL)), dRf = sub_half(dR, mm(dR - dL, dRR - dR));
        const double p0f = p.ref_pf[id];
        fl = hllc_p(m, L[0], L[in], L[it1], L[it2], L[4], R(p0f) + dLf, Rr[0], Rr[in], Rr[it1], Rr[it2], Rr[4],
                    R(p0f) + dRf);
    } else {
        fl = hllc(m, EU_SETTING(R, rho_vac), L[0], L[in], L[it1], L[it2], L[4], Rr[0], Rr[in], Rr[it1], Rr[it2], Rr[4]);
    }
    put(F.q[DIR][0], id, fl.r);
    put(F.q[DIR][1], id, fl.mn);
    put(F.q[DIR][2], id, fl.mt1);
    put(F.q[DIR][3], id, fl.mt2);
    put(F.q[DIR][4], id, fl.E);
    put(F.q[DIR][5], id, fl.r * (ge0(fl.r) ? at(W.w[5], cL) : at(W.w[5], cR)));
}

// One direction's face fluxes, or (small grids) every direction's in one
// launch: blocks below b1 take the x faces, below b2 the y faces, the rest the
// z faces.
template <int DIR, class R>
static __global__ void __launch_bounds__(256) k_face(P p, PrimT<R> W, FacesT<R> F, const Ctl* ctl) {
    if (ctl->active) face_one<DIR, R>(p, W, F, gtid());
}
template <class R>
static __global__ void __launch_bounds__(256) k_faces(P p, PrimT<R> W, FacesT<R> F, const Ctl* ctl, unsigned b1,
                                                      unsigned b2) {
    if (!ctl->active) return;
    const unsigned b = blockIdx.x;
    if (b < b1) face_one<0, R>(p, W, F, (int64_t)b * blockDim.x + threadIdx.x);
    else if (b < b2) face_one<1, R>(p, W, F, (int64_t)(b - b1) * blockDim.x + threadIdx.x);
    else face_one<2, R>(p, W, F, (int64_t)(b - b2) * blockDim.x + threadIdx.x);
}

// Right-hand side of one cell (hydro_cpu.cpp:98-214): the three directions'
// flux differences in the reference's order, gravity, strength sources.
// s: the state Lop reads; W: its primitives (k_prim), whose velocities mu/rho
// are the very quotients the reference forms for every neighbour it reads;
// af: the fluidization ratio.  Flux differences and strength sources are
// formed in R and added to the FP64 right-hand side (with R = double: every
// operation of the reference, in its order).
// One launch holds two parts (blockIdx.y): 0 the conserved fields (flux
// differences, gravity, div S, the explicit viscosity, div(S.v)), 1 the
// stress, damage and vibration rates.  They write different fields and share
// little; one kernel for both needed 168 registers in FP64 (13 % of the warps in
// flight) and spilled in FP32.  MINB resident blocks of 128 are asked of the
// compiler: the loads' latency bounds a large grid, so it takes many (FP32,
// 160^3 step: 3.18 / 2.99 / 2.89 / 2.93 ms at 8 / 10 / 12 / 14; FP64, 96^3 step:
// 3.18 / 3.04 / 3.00 ms at 4 / 6 / 8); a grid whose blocks are all resident
// anyway takes the registers (150 x 110 crater, FP64: 0.179 ms at 4, 0.181 at 8).
constexpr int kRhsMinbF32[2] = {8, 12}, kRhsMinbF64[2] = {4, 8};  // small grids, large grids
// The cell's neighbours, their near-void flags and the differences over them.
template <class R>
struct Stencil {
    const P& p;
    uint32_t xm, xp, ym, yp, zm, zp;
    bool hx, hy, hz;  // both neighbours exist: differences over two cells
    __device__ __forceinline__ Stencil(const P& p_, uint32_t c, int i, int j, int k, uint32_t plane) : p(p_) {
        xm = c - (i > 0 ? plane : 0u); xp = c + (i < p.nx - 1 ? plane : 0u);
        ym = c - (j > 0 ? (uint32_t)p.nz : 0u); yp = c + (j < p.ny - 1 ? (uint32_t)p.nz : 0u);
        zm = c - (k > 0 ? 1u : 0u); zp = c + (k < p.nz - 1 ? 1u : 0u);
        hx = i > 0 && i < p.nx - 1; hy = j > 0 && j < p.ny - 1; hz = k > 0 && k < p.nz - 1;
    }
    // x / dx, and the halved quotient across two cells (x / (2 dx), exactly)
    __device__ __forceinline__ R over_dx(R x) const {
        if constexpr (sizeof(R) == 4) return x / EU_SETTING(R, dx);
        else return dv(x, p.d_dx);
    }
    __device__ __forceinline__ R over(R x, bool two) const {
        if constexpr (sizeof(R) == 4) return x / ((two ? R(2) : R(1)) * EU_SETTING(R, dx));
        else return two ? half(dv(x, p.d_dx)) : dv(x, p.d_dx);
    }
};
template <class R>
static __device__ __forceinline__ bool is_void(const P& p, const Fields& s, const PrimT<R>& W, uint32_t q) {
    if constexpr (sizeof(R) == 4) return W.vd[q] != 0;  // k_prim's flags
    else return p.rho_cfl > 0 && lt(s.q[F_R][q], p.rho_cfl);
}

template <class R, int LARGE>
static __global__ void __launch_bounds__(128, sizeof(R) == 4 ? kRhsMinbF32[LARGE] : kRhsMinbF64[LARGE])
    k_rhs(P p, Fields s, PrimT<R> W, const double* af, FacesT<R> F, RhsT<R> d, const Ctl* ctl) {
    const int64_t c0 = gtid();
    if (c0 >= p.n || !ctl->active) return;
    const uint32_t c = (uint32_t)c0, plane = (uint32_t)p.ny * p.nz;
    const int i = (int)(c / plane);
    const uint32_t rem = c - (uint32_t)i * plane;
    const int j = (int)(rem / (uint32_t)p.nz), k = (int)(rem - (uint32_t)j * p.nz);
    const bool solid = p.m.G > 0 && !is_void<R>(p, s, W, c);
    const Stencil<R> st(p, c, i, j, k, plane);
    const uint32_t xm = st.xm, xp = st.xp, ym = st.ym, yp = st.yp, zm = st.zm, zp = st.zp;
    const bool hx = st.hx, hy = st.hy, hz = st.hz;
    const R* Vx = W.w[1];  // mu / rho of every cell
    const R* Vy = W.w[2];
    const R* Vz = W.w[3];
    const R* Sxx = W.sq[0];
    const R* Syy = W.sq[1];
    const R* Szz = W.sq[2];
    const R* Sxy = W.sq[3];
    const R* Sxz = W.sq[4];
    const R* Syz = W.sq[5];
    const bool ny1 = p.flat >> 1 & 1;  // no differences along y (its terms are zero)
    using A = R;
    if (blockIdx.y == 1) {  // strength sources of S, D and vib, hydro_cpu.cpp:145-213
        A dS[6] = {A(0), A(0), A(0), A(0), A(0), A(0)}, dD = A(0), dvib = A(0);
        if (solid) {
            const R G = mat_of<R>(p).G;
            const R vxc = at(Vx, c), vyc = at(Vy, c), vzc = at(Vz, c);
            const bool oxm = is_void<R>(p, s, W, xm), oxp = is_void<R>(p, s, W, xp), ozm = is_void<R>(p, s, W, zm),
                       ozp = is_void<R>(p, s, W, zp);
            auto grad = [&](const R* V, R vc, uint32_t q1, bool o1, uint32_t q0, bool o0, bool two) {
                return st.over((o1 ? vc : at(V, q1)) - (o0 ? vc : at(V, q0)), two);
            };
            const R Lxx = grad(Vx, vxc, xp, oxp, xm, oxm, hx), Lxz = grad(Vx, vxc, zp, ozp, zm, ozm, hz);
            const R Lyx = grad(Vy, vyc, xp, oxp, xm, oxm, hx), Lyz = grad(Vy, vyc, zp, ozp, zm, ozm, hz);
            const R Lzx = grad(Vz, vzc, xp, oxp, xm, oxm, hx), Lzz = grad(Vz, vzc, zp, ozp, zm, ozm, hz);
            R Lxy = R(0), Lyy = R(0), Lzy = R(0);
            if (!ny1) {
                const bool oym = is_void<R>(p, s, W, ym), oyp = is_void<R>(p, s, W, yp);
                Lxy = grad(Vx, vxc, yp, oyp, ym, oym, hy);
                Lyy = grad(Vy, vyc, yp, oyp, ym, oym, hy);
                Lzy = grad(Vz, vzc, yp, oyp, ym, oym, hy);
            }
            const R eyy = p.axisym ? dv(vxc, R((i + 0.5) * p.dx)) : Lyy;
            const R exx = Lxx, ezz = Lzz, exy = half(Lxy + Lyx), exz = half(Lxz + Lzx), eyz = half(Lyz + Lzy);
            R tr;
            if constexpr (sizeof(R) == 4) tr = (exx + eyy + ezz) / R(3);
            else tr = dv(exx + eyy + ezz, p.d_3);
            const R Wxy = half(Lxy - Lyx), Wxz = half(Lxz - Lzx), Wyz = half(Lyz - Lzy);
            const R sxx = at(Sxx, c), syy = at(Syy, c), szz = at(Szz, c), sxy = at(Sxy, c), sxz = at(Sxz, c), syz = at(Syz, c);
            R J00, J11, J22, J01, J02, J12;  // S.W - W.S, hydro_cpu.cpp:172-173
            if constexpr (sizeof(R) == 4) {
                const R Sm[3][3] = {{sxx, sxy, sxz}, {sxy, syy, syz}, {sxz, syz, szz}};
                const R Wm[3][3] = {{R(0), Wxy, Wxz}, {-Wxy, R(0), Wyz}, {-Wxz, -Wyz, R(0)}};
                auto J = [&](int aa, int bb) {
                    R t = R(0);
#pragma unroll
                    for (int cc = 0; cc < 3; cc++) t += Sm[aa][cc] * Wm[cc][bb] - Wm[aa][cc] * Sm[cc][bb];
                    return t;
                };
                J00 = J(0, 0); J11 = J(1, 1); J22 = J(2, 2);
                J01 = J(0, 1); J02 = J(0, 2); J12 = J(1, 2);
            } else {
                // without the products with W's zero diagonal; a diagonal entry's
                // paired products are equal, so each pair is one product doubled
                const R bxy = sxy * Wxy, bxz = sxz * Wxz, byz = syz * Wyz;
                J00 = R(-2) * (bxy + bxz); J11 = R(2) * (bxy - byz); J22 = R(2) * (bxz + byz);
                J01 = sxx * Wxy - Wxy * syy + (-(sxz * Wyz) - Wxz * syz);
                J02 = sxx * Wxz + (sxy * Wyz - Wxy * syz) - Wxz * szz;
                J12 = (sxy * Wxz + Wxy * sxz) + syy * Wyz - Wyz * szz;
            }
            const R u = vxc, v = vyc, w = vzc;
            const bool pu = gt0(u), pv = gt0(v), pw = gt0(w);
            // the upwind difference's cells; outside the grid the cell itself, so
            // the difference is zero there
            const uint32_t x1 = pu ? c : xp, x0 = pu ? xm : c, y1 = pv ? c : yp, y0 = pv ? ym : c;
            const uint32_t z1 = pw ? c : zp, z0 = pw ? zm : c;
            auto adv = [&](const R* S) {  // upwind v . grad S, hydro_cpu.cpp:175-178
                const R ay = ny1 ? R(0) : st.over_dx(at(S, y1) - at(S, y0));
                return mad(w, st.over_dx(at(S, z1) - at(S, z0)), mad(u, st.over_dx(at(S, x1) - at(S, x0)), v * ay));
            };
            dS[0] = R(2) * G * (exx - tr) + J00 - adv(Sxx);
            dS[1] = R(2) * G * (eyy - tr) + J11 - adv(Syy);
            dS[2] = R(2) * G * (ezz - tr) + J22 - adv(Szz);
            dS[3] = R(2) * G * exy + J01 - adv(Sxy);
            dS[4] = R(2) * G * exz + J02 - adv(Sxz);
            dS[5] = R(2) * G * eyz + J12 - adv(Syz);
            dD = -adv(W.sq[6]);
            dvib = -adv(W.sq[7]);
        }
#pragma unroll
        for (int q = 0; q < 6; q++) put(d.q[D_SXX + q], c, dS[q]);
        put(d.q[D_D], c, dD);
        put(d.q[D_VIB], c, dvib);
        return;
    }
    const double* r = s.q[F_R];
    const double* mw = s.q[F_MW];
    // Sums of the right-hand side: in the FP64 form the reference's additions; in
    // the FP32 form the terms are FP32 already and are summed in FP32 (in the
    // same order).
    A dr = A(0), dE = A(0), drc = A(0), dmu = A(0), dmv = A(0), dmw = A(0);
    // ---- hydro sweeps (hydro_cpu.cpp:122-133), x then y then z
    {
        const uint32_t lo[3] = {c, ((uint32_t)i * (p.ny + 1) + j) * p.nz + k, ((uint32_t)i * p.ny + j) * (p.nz + 1) + k};
        const uint32_t up[3] = {plane, (uint32_t)p.nz, 1u};
#pragma unroll
        for (int dir = 0; dir < 3; dir++) {
            if (p.flat >> dir & 1) continue;
            const uint32_t a = lo[dir], b = lo[dir] + up[dir];
            const R* const* Fq = F.q[dir];
            R vr, vE, vrc, dmn, dt1, dt2;
            if (dir == 0 && p.axisym) {
                const R w0 = R(i * p.dx), w1 = R((i + 1) * p.dx), inv = R(fi::div(1.0, ((i + 0.5) * p.dx) * p.dx));
                vr = -(w1 * at(Fq[0], b) - w0 * at(Fq[0], a)) * inv;
                vE = -(w1 * at(Fq[4], b) - w0 * at(Fq[4], a)) * inv;
                vrc = -(w1 * at(Fq[5], b) - w0 * at(Fq[5], a)) * inv;
                dmn = -(w1 * at(Fq[1], b) - w0 * at(Fq[1], a)) * inv;
                dt1 = -(w1 * at(Fq[2], b) - w0 * at(Fq[2], a)) * inv;
                dt2 = -(w1 * at(Fq[3], b) - w0 * at(Fq[3], a)) * inv;
                R pr, cs;
                eos_pc(mat_of<R>(p), at(W.w[0], c), at(W.w[4], c), pr, cs);  // Pcell: EOS at the cell's internal energy
                dmn += dv(pr, R((i + 0.5) * p.dx));
            } else {  // face weights 1 (exact products)
                const R inv = EU_SETTING(R, invdx);
                vr = -(at(Fq[0], b) - at(Fq[0], a)) * inv;
                vE = -(at(Fq[4], b) - at(Fq[4], a)) * inv;
                vrc = -(at(Fq[5], b) - at(Fq[5], a)) * inv;
                dmn = -(at(Fq[1], b) - at(Fq[1], a)) * inv;
                dt1 = -(at(Fq[2], b) - at(Fq[2], a)) * inv;
                dt2 = -(at(Fq[3], b) - at(Fq[3], a)) * inv;
            }
            dr += A(vr);
            dE += A(vE);
            drc += A(vrc);
            if (dir == 0) {
                dmu += A(dmn); dmv += A(dt1); dmw += A(dt2);
            } else if (dir == 1) {
                dmv += A(dmn); dmu += A(dt1); dmw += A(dt2);
            } else {
                dmw += A(dmn); dmu += A(dt1); dmv += A(dt2);
            }
        }
    }
    if (p.gz != 0.0) {
        if (!p.ref_r0) {  // plain gravity body force, hydro_cpu.cpp:137-138
            dmw += narrow<A>(-p.gz * r[c]);
            dE += narrow<A>(-p.gz * mw[c]);
        } else {  // well-balanced source against the reference, hydro_cpu.cpp:139-143
            const double* R0 = p.ref_r0;
            dmw += narrow<A>(-p.gz * (r[c] - R0[c]) + p.ref_dp[c] * p.invdx);  // ref_dp: k_ref_dp
            dE += narrow<A>(-p.gz * mw[c]);
        }
    }
    if (solid) {  // strength sources of the conserved fields
        const R rcyl = R((i + 0.5) * p.dx);
        const DivBy<R> d_rcyl = div_by(rcyl);
        // div S into momentum (central differences), hydro_cpu.cpp:183-186
        auto cd = [&](const R* S, uint32_t q1, uint32_t q0, bool two) { return st.over(at(S, q1) - at(S, q0), two); };
        const R dSxx_x = cd(Sxx, xp, xm, hx), dSxz_z = cd(Sxz, zp, zm, hz);
        const R dSxy_x = cd(Sxy, xp, xm, hx), dSyz_z = cd(Syz, zp, zm, hz);
        const R dSxz_x = cd(Sxz, xp, xm, hx), dSzz_z = cd(Szz, zp, zm, hz);
        R dSxy_y = R(0), dSyy_y = R(0), dSyz_y = R(0);
        if (!ny1) {
            dSxy_y = cd(Sxy, yp, ym, hy);
            dSyy_y = cd(Syy, yp, ym, hy);
            dSyz_y = cd(Syz, yp, ym, hy);
        }
        dmu += A(dSxx_x + dSxy_y + dSxz_z);
        dmv += A(dSxy_x + dSyy_y + dSyz_z);
        dmw += A(dSxz_x + dSyz_y + dSzz_z);
        if (p.axisym) {
            dmu += A(dv(at(Sxx, c) - at(Syy, c), d_rcyl));
            dmw += A(dv(at(Sxz, c), d_rcyl));
        }
        if (p.eta_af > 0 && !p.visc_imp && gt0(af[c])) {  // explicit fluidization viscosity, hydro_cpu.cpp:190-197
            const R eta = R(af[c] * p.eta_af), id2 = R(p.id2);
            auto lap = [&](const R* V) {
                return eta * (at(V, xp) + at(V, xm) + at(V, yp) + at(V, ym) + at(V, zp) + at(V, zm) - R(6) * at(V, c)) * id2;
            };
            dmu += A(lap(Vx));
            dmv += A(lap(Vy));
            dmw += A(lap(Vz));
            if (p.axisym) {
                const bool oxm = is_void<R>(p, s, W, xm), oxp = is_void<R>(p, s, W, xp);
                const R vxc = at(Vx, c), vzc = at(Vz, c);
                const R Lxx = st.over((oxp ? vxc : at(Vx, xp)) - (oxm ? vxc : at(Vx, xm)), hx);
                const R Lzx = st.over((oxp ? vzc : at(Vz, xp)) - (oxm ? vzc : at(Vz, xm)), hx);
                dmu += A(eta * (dv(Lxx, d_rcyl) - dv(vxc, rcyl * rcyl)));
                dmw += A(eta * dv(Lzx, d_rcyl));
            }
        }
        // div(S.v) into energy, hydro_cpu.cpp:198-203
        auto sv = [&](const R* a, const R* b, const R* e, uint32_t q) {
            return mad(at(e, q), at(Vz, q), mad(at(a, q), at(Vx, q), at(b, q) * at(Vy, q)));
        };
        const R ex = st.over(sv(Sxx, Sxy, Sxz, xp) - sv(Sxx, Sxy, Sxz, xm), hx);
        const R ey = ny1 ? R(0) : st.over(sv(Sxy, Syy, Syz, yp) - sv(Sxy, Syy, Syz, ym), hy);
        const R ez = st.over(sv(Sxz, Syz, Szz, zp) - sv(Sxz, Syz, Szz, zm), hz);
        dE += A(ex + ey + ez);
        if (p.axisym) dE += A(dv(sv(Sxx, Sxy, Sxz, c), d_rcyl));
    }
    put(d.q[D_R], c, dr);
    put(d.q[D_MU], c, dmu);
    put(d.q[D_MV], c, dmv);
    put(d.q[D_MW], c, dmw);
    put(d.q[D_E], c, dE);
    put(d.q[D_RC], c, drc);
}

// Near-void cell: momentum zeroed; with a reference state also reset to the
// reference (or ambient) density with no energy, stress or tracer,
// hydro_cpu.cpp:272-290 (not the conservative transfer).
static __device__ __forceinline__ void void_cell(const P& p, Cell& x, int64_t c) {
    if (!(p.rho_cfl > 0 && lt(x.q[F_R], p.rho_cfl))) return;
    if (p.void_cons && p.ref_r0) return;  // the serial conservative pass (k_void_cons) does it
    x.q[F_MU] = x.q[F_MV] = x.q[F_MW] = 0;
    if (p.ref_r0) {
        x.q[F_R] = (p.void_amb > 0 ? p.void_amb : p.ref_r0[c]);
        x.q[F_E] = 0;
        x.q[F_SXX] = x.q[F_SYY] = x.q[F_SZZ] = x.q[F_SXY] = x.q[F_SXZ] = x.q[F_SYZ] = 0;
        x.q[F_RC] = 0;
    }
}

// The conservative void reset (VOID_CONS, hydro_cpu.cpp:272-290): every
// near-void cell, in index order, zeroes its momentum, moves its excess over
// the ambient density to the densest face neighbour above RHO_CFL (candidates
// x-, x+, z-, z+, then y-, y+ when ny > 1; first of equals; volume-weighted in
// cylindrical geometry) and is reset.  The choice of neighbour depends on the
// transfers of the cells before it, so one thread walks the cells in order;
// the block loads each 1024-cell chunk's densities in parallel first.  A cell
// below RHO_CFL is never a transfer target (targets exceed RHO_CFL and only
// grow), so whether a cell is void and its own density are unchanged from the
// chunk's load until its turn.
static __global__ void __launch_bounds__(1024) k_void_cons(P p, Fields g, const Ctl* ctl) {
    if (!ctl->active) return;
    __shared__ double rs[1024];
    double* r = g.q[F_R];
    const int64_t plane = (int64_t)p.ny * p.nz;
    for (int64_t base = 0; base < p.n; base += 1024) {
        const int64_t c0 = base + threadIdx.x;
        rs[threadIdx.x] = c0 < p.n ? r[c0] : 1e300;
        __syncthreads();
        if (threadIdx.x == 0) {
            const int m = (int)(p.n - base < 1024 ? p.n - base : 1024);
            for (int t = 0; t < m; t++) {
                if (!(rs[t] < p.rho_cfl)) continue;
                const int64_t c = base + t;
                g.q[F_MU][c] = g.q[F_MV][c] = g.q[F_MW][c] = 0;
                const double amb = (p.void_amb > 0 ? p.void_amb : 0.27), exc = rs[t] - amb;
                if (exc > 0) {
                    const int i = (int)(c / plane), j = (int)((c / p.nz) % p.ny), k = (int)(c % p.nz);
                    int64_t nb = -1;
                    double rbest = p.rho_cfl;
                    const int cand[6][3] = {{i - 1, j, k}, {i + 1, j, k}, {i, j, k - 1},
                                            {i, j, k + 1}, {i, j - 1, k}, {i, j + 1, k}};
                    const int nc = p.ny > 1 ? 6 : 4;
                    for (int q = 0; q < nc; q++) {
                        const int ii = cand[q][0], jj = cand[q][1], kk = cand[q][2];
                        if (ii < 0 || ii >= p.nx || jj < 0 || jj >= p.ny || kk < 0 || kk >= p.nz) continue;
                        const int64_t cc = ((int64_t)ii * p.ny + jj) * p.nz + kk;
                        if (r[cc] > rbest) {
                            rbest = r[cc];
                            nb = cc;
                        }
                    }
                    if (nb >= 0) {
                        double w = 1.0;
                        if (p.axisym) {
                            const int inb = (int)(nb / plane);
                            w = (i + 0.5) / (inb + 0.5);
                        }
                        r[nb] += exc * w;
                    }
                }
                r[c] = (p.void_amb > 0 ? p.void_amb : p.ref_r0[c]);
                g.q[F_E][c] = 0;
                g.q[F_SXX][c] = g.q[F_SYY][c] = g.q[F_SZZ][c] = g.q[F_SXY][c] = g.q[F_SXZ][c] = g.q[F_SYZ][c] = 0;
                g.q[F_RC][c] = 0;
            }
        }
        __syncthreads();
    }
}

// The predictor's radial return when the conservative void pass runs between
// the update and the return.
template <class R>
static __global__ void k_yield_stage(P p, Fields g1, const double* af, PrimT<R> W, const Ctl* ctl) {
    const int64_t c = gtid();
    if (c >= p.n || !ctl->active) return;
    Cell x;
    load_cell(x, g1, c, EU_RK);
    PcellOnce<R> pc;
    vonmises_cell<R>(p, x, af[c], false, pc);
    store_cell(x, g1, c, EU_STRESS);
    prim_cell<R>(p, x, W, c);
}

// The reference state's pressure at every z-face (hydro_cpu.cpp:114-119,
// 139-143): p0 at the averaged reference densities of the two cells, zero
// internal energy, clamped at 0.  It depends only on the frozen reference and
// the material, so it is formed once per reference (and material) instead of
// in every Lop; k_ref_dp differences it over each cell for the well-balanced
// gravity source.
static __global__ void k_ref_pf(P p, const double* R0, double* pf) {
    const int64_t id = gtid();
    if (id >= (int64_t)p.nx * p.ny * (p.nz + 1)) return;
    const int64_t line = id / (p.nz + 1);
    const int f = (int)(id - line * (p.nz + 1));
    const int64_t base = line * p.nz;
    const int64_t cL = base + max(0, f - 1), cR = base + min(p.nz - 1, f);
    double p0 = pressure(p.m, 0.5 * (R0[cL] + R0[cR]), 0.0);
    if (p0 < 0) p0 = 0;
    pf[id] = p0;
}
static __global__ void k_ref_dp(P p, const double* pf, double* dp) {
    const int64_t c = gtid();
    if (c >= p.n) return;
    const int64_t f = c + c / p.nz;  // the cell's bottom z-face
    dp[c] = pf[f + 1] - pf[f];
}

// set_ref (hydro_cpu.cpp:259-261): density and pressure frozen as the reference.
static __global__ void k_set_ref(P p, Fields g, double* r0, double* p0) {
    const int64_t c = gtid();
    if (c >= p.n) return;
    r0[c] = g.q[F_R][c];
    p0[c] = pcell(p, g, c);
}

// Predictor (hydro_cpu.cpp:413-418): g1 = g + dt d, void-cell reset, radial
// return without regeneration.
// The predictor state's primitives, which the second Lop reads, are formed
// here from the values at hand (with the conservative void pass, after it).
template <class R>
static __global__ void k_predict(P p, Fields g, Fields g1, PrimT<R> W, RhsT<R> d, const Ctl* ctl) {
    const int64_t c = gtid();
    if (c >= p.n || !ctl->active) return;
    const double dt = ctl->dt, af = g.q[F_AF][c];
    Cell x;
    R dq[ND];
    load_cell(x, g, c, EU_RK);
#pragma unroll
    for (int q = 0; q < ND; q++) dq[q] = d.q[q][c];
#pragma unroll
    for (int q = 0; q < ND; q++) x.q[rk_field(q)] = x.q[rk_field(q)] + dt * widen(dq[q]);
    void_cell(p, x, c);
    if (!(p.void_cons && p.ref_r0)) {  // else after k_void_cons
        PcellOnce<R> pc;
        vonmises_cell<R>(p, x, af, false, pc);
        prim_cell<R>(p, x, W, c);
    }
    store_cell(x, g1, c, EU_RK);
}

// Corrector and the end of the step (hydro_cpu.cpp:419-424): trapezoidal
// average, damage growth, radial return, damping, void-cell reset.  With the
// implicit viscosity, which runs between the average and the rest, stage 1 is
// the average alone and stage 2 the rest; stage 0 is all of it.
template <class R>
static __global__ void k_correct(P p, Fields g, Fields g1, RhsT<R> d, const Ctl* ctl, int stage) {
    const int64_t c = gtid();
    if (c >= p.n || !ctl->active) return;
    const double dt = ctl->dt, af = g.q[F_AF][c];
    Cell x;
    load_cell(x, g, c, EU_RK);
    if (stage != 2) {
        Cell y;
        R dq[ND];
        load_cell(y, g1, c, EU_RK);
#pragma unroll
        for (int q = 0; q < ND; q++) dq[q] = d.q[q][c];
#pragma unroll
        for (int q = 0; q < ND; q++)
            x.q[rk_field(q)] = half(x.q[rk_field(q)] + y.q[rk_field(q)] + dt * widen(dq[q]));
    }
    if (stage != 1) {
        PcellOnce<R> pc;
        grow_damage_cell<R>(p, x, dt, pc);
        vonmises_cell<R>(p, x, af, true, pc);
        if (p.damp < 1.0) {
            x.q[F_MU] *= p.damp;
            x.q[F_MV] *= p.damp;
            x.q[F_MW] *= p.damp;
        }
        void_cell(p, x, c);
    }
    store_cell(x, g, c, EU_RK);
}

// Driver adjustments after each step (eu_set_driver), in this order:
//   pin:   the lowest `pin` z-layers return to the reference density at rest
//          with no energy (DRV_PIN_STRESS: and no deviatoric stress);
//   isp:   columns i >= isp relax toward the reference with weight
//          ((i - isp) / max(1, nx - 1 - isp))^2 (isp < 0: none);
//   DRV_VOID_AMBIENT: near-void cells (rho < RHO_CFL) become ambient gas
//          (0.27 kg/m^3) at rest with no energy and no stress;
//   DRV_TRACK_PMAX: Pmax = max(Pmax, Pcell) per cell.
// The crater mode's floor pin and radial sponge (hydro_cpu.cpp:634-637), the
// collapse demo's held floor (893-894), the Prater run's void cleanup
// (823-824) and the Pierazzo run's peak-pressure record (769).
enum { DRV_PIN_STRESS = 1, DRV_VOID_AMBIENT = 2, DRV_TRACK_PMAX = 4 };

static __global__ void k_driver(P p, Fields g, const Ctl* ctl, int pin, int isp, int flags) {
    const int64_t c = gtid();
    if (c >= p.n || !ctl->active) return;
    const int i = (int)(c / ((int64_t)p.ny * p.nz)), k = (int)(c % p.nz);
    if (k < pin) {
        g.q[F_R][c] = p.ref_r0[c];
        g.q[F_MU][c] = g.q[F_MV][c] = g.q[F_MW][c] = 0;
        g.q[F_E][c] = 0;
        if (flags & DRV_PIN_STRESS)
            g.q[F_SXX][c] = g.q[F_SYY][c] = g.q[F_SZZ][c] = g.q[F_SXY][c] = g.q[F_SXZ][c] = g.q[F_SYZ][c] = 0;
    }
    if (isp >= 0 && i >= isp) {
        const int span = p.nx - 1 - isp;
        const double xi = (double)(i - isp) / (span > 1 ? span : 1), sp = xi * xi;
        g.q[F_R][c] = (1 - sp) * g.q[F_R][c] + sp * p.ref_r0[c];
        g.q[F_MU][c] *= (1 - sp);
        g.q[F_MV][c] *= (1 - sp);
        g.q[F_MW][c] *= (1 - sp);
        g.q[F_E][c] *= (1 - sp);
    }
    if ((flags & DRV_VOID_AMBIENT) && g.q[F_R][c] < p.rho_cfl) {
        g.q[F_R][c] = 0.27;
        g.q[F_MU][c] = g.q[F_MV][c] = g.q[F_MW][c] = 0;
        g.q[F_E][c] = 0;
        g.q[F_SXX][c] = g.q[F_SYY][c] = g.q[F_SZZ][c] = g.q[F_SXY][c] = g.q[F_SXZ][c] = g.q[F_SYZ][c] = 0;
    }
    if (flags & DRV_TRACK_PMAX) {
        const double P = pcell(p, g, c);
        if (P > g.q[F_PMAX][c]) g.q[F_PMAX][c] = P;
    }
}

// Single operators for the C ABI's unit calls.
static __global__ void k_vonmises(P p, Fields g, int reg) {
    const int64_t c = gtid();
    PcellOnce<double> pc;
    if (c >= p.n) return;
    Cell x;
    load_cell(x, g, c, EU_RK);
    vonmises_cell<double>(p, x, g.q[F_AF][c], reg != 0, pc);
    store_cell(x, g, c, EU_STRESS, F_E, F_VIB);
}
static __global__ void k_grow_damage(P p, Fields g, double dt) {
    const int64_t c = gtid();
    PcellOnce<double> pc;
    if (c >= p.n) return;
    Cell x;
    load_cell(x, g, c, EU_RK);
    grow_damage_cell<double>(p, x, dt, pc);
    store_cell(x, g, c, F_D);
}
static __global__ void k_pressure(P p, Fields g, double* out) {
    const int64_t c = gtid();
    if (c < p.n) out[c] = pcell(p, g, c);
}

static __global__ void k_set_step(P p, Ctl* ctl, double dt) {  // a step at a host dt
    ctl->dt = dt;
    if (p.tdec > 0) ctl->af_dec = exp(-dt / p.tdec);
    ctl->active = 1;
}
static __global__ void k_set_run(Ctl* ctl, double cfl, double t_end, int64_t max_steps) {
    ctl->cfl = cfl;
    ctl->t_end = t_end;
    ctl->max_steps = max_steps < 0 ? -1 : ctl->steps + max_steps;
    next_step(ctl);
}
static __global__ void k_widen(const float* x, double* y, int64_t n) {
    const int64_t c = gtid();
    if (c < n) y[c] = (double)x[c];
}
static __global__ void k_set_time(Ctl* ctl, double t) { ctl->t = t; }
static __global__ void k_maxspeed_begin(Ctl* ctl) {
    ctl->active = 1;
    ctl->smax_bits = (unsigned long long)__double_as_longlong(1e-30);
}


// ---------------------------------------------------------------- Lop launcher

constexpr unsigned kOneLaunchBlocks = 152 * 6;

// One Lop (hydro_cpu.cpp:98-214) of state s in compute type R whose primitives
// are formed: the directions' face fluxes, then the right-hand side's two
// parts in one launch.  Returns the launches made.
template <class R>
inline int enqueue_lop_t(const P& p, const Fields& s, PrimT<R> W, const double* af, FacesT<R> F, RhsT<R> d,
                          const Ctl* ctl, cudaStream_t st) {
    auto blocks = [](int64_t count, int b) { return (unsigned)((count + b - 1) / b); };
    if constexpr (sizeof(R) == 8) {  // FP64: the right-hand side reads the state's own strength fields
#pragma unroll
        for (int q = 0; q < 6; q++) W.sq[q] = s.q[F_SXX + q];
        W.sq[6] = s.q[F_D];
        W.sq[7] = s.q[F_VIB];
        W.vd = nullptr;
    }
    const unsigned bx = p.flat & 1 ? 0 : blocks(face_count<0>(p.nx, p.ny, p.nz), 256);
    const unsigned by = p.flat & 2 ? 0 : blocks(face_count<1>(p.nx, p.ny, p.nz), 256);
    const unsigned bz = p.flat & 4 ? 0 : blocks(face_count<2>(p.nx, p.ny, p.nz), 256);
    // One launch while all its blocks are about resident at once (152 SMs);
    // beyond, a kernel per direction (FP32, 160^3: 0.46 ms, against 0.57 ms as one).
    if (bx + by + bz <= kOneLaunchBlocks) {
        if (bx + by + bz > 0) k_faces<R><<<bx + by + bz, 256, 0, st>>>(p, W, F, ctl, bx, bx + by);
    } else {
        if (bx) k_face<0, R><<<bx, 256, 0, st>>>(p, W, F, ctl);
        if (by) k_face<1, R><<<by, 256, 0, st>>>(p, W, F, ctl);
        if (bz) k_face<2, R><<<bz, 256, 0, st>>>(p, W, F, ctl);
    }
    const dim3 rb(blocks(p.n, 128), 2);
    if (2 * rb.x <= 152u * 8) k_rhs<R, 0><<<rb, 128, 0, st>>>(p, s, W, af, F, d, ctl);
    else k_rhs<R, 1><<<rb, 128, 0, st>>>(p, s, W, af, F, d, ctl);
    return 1 + (bx + by + bz == 0 ? 0 : bx + by + bz <= kOneLaunchBlocks ? 1 : (bx > 0) + (by > 0) + (bz > 0));
}
// The primitives of a state, after its update_af (af: 1).
template <class R>
inline void enqueue_prim_t(const P& p, const Fields& s, PrimT<R> W, const Ctl* ctl, cudaStream_t st, int af) {
    const unsigned nb = (unsigned)((p.n + 255) / 256);
    if (af) k_prim<R, true><<<nb, 256, 0, st>>>(p, s, W, ctl);
    else k_prim<R, false><<<nb, 256, 0, st>>>(p, s, W, ctl);
}

// The CFL speed reduction, the predictor and the corrector in compute type R.
template <class R>
inline void enqueue_maxspeed_t(const P& p, const Fields& g, Ctl* ctl, cudaStream_t st, int with_dt) {
    k_maxspeed<R><<<(unsigned)((p.n + 255) / 256), 256, 0, st>>>(p, g, ctl, with_dt);
}
template <class R>
inline void enqueue_predict_t(const P& p, const Fields& g, const Fields& g1, PrimT<R> W, RhsT<R> d, const Ctl* ctl,
                              cudaStream_t st) {
    k_predict<R><<<(unsigned)((p.n + 255) / 256), 256, 0, st>>>(p, g, g1, W, d, ctl);
    if (p.void_cons && p.ref_r0) {  // void_cells(g1) in order, then vonmises(g1, false)
        if (p.rho_cfl > 0) {
            k_void_cons<<<1, 1024, 0, st>>>(p, g1, ctl);
            k_yield_stage<R><<<(unsigned)((p.n + 255) / 256), 256, 0, st>>>(p, g1, g.q[F_AF], W, ctl);
        } else {
            enqueue_prim_t<R>(p, g1, W, ctl, st, 0);
        }
    }
}
template <class R>
inline void enqueue_correct_t(const P& p, const Fields& g, const Fields& g1, RhsT<R> d, const Ctl* ctl,
                              cudaStream_t st, int stage) {
    k_correct<R><<<(unsigned)((p.n + 255) / 256), 256, 0, st>>>(p, g, g1, d, ctl, stage);
    if (stage != 1 && p.void_cons && p.ref_r0 && p.rho_cfl > 0)
        k_void_cons<<<1, 1024, 0, st>>>(p, g, ctl);  // void_cells(g) last
}

// The FP32 instantiations live in euler_mixed.cu (compiled with fused
// multiply-adds); the FP64 ones in euler.cu (compiled without).
int enqueue_lop_f32(const P& p, const Fields& s, PrimT<float> W, const double* af, FacesT<float> F, RhsT<float> d,
                    const Ctl* ctl, cudaStream_t st);
void enqueue_prim_f32(const P& p, const Fields& s, PrimT<float> W, const Ctl* ctl, cudaStream_t st, int af);
void enqueue_maxspeed_f32(const P& p, const Fields& g, Ctl* ctl, cudaStream_t st, int with_dt);
void enqueue_predict_f32(const P& p, const Fields& g, const Fields& g1, PrimT<float> W, RhsT<float> d, const Ctl* ctl,
                         cudaStream_t st);
void enqueue_correct_f32(const P& p, const Fields& g, const Fields& g1, RhsT<float> d, const Ctl* ctl,
                         cudaStream_t st, int stage);

}  // namespace deu
