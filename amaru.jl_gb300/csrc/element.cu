// Element kernels of the mechanical hot path (FP64), sm_103a.
//
//  * stiffness_kernel   -- elem_stiffness (src/mech/elem/mech-solid.jl:124-166)
//  * gather_kernel      -- the duplicate summation of mount_K / sparse()
//                          (src/mech/mech-solver.jl:78-110), deterministic, no atomics
//  * internal_kernel    -- update_elem! + update_state!(mat, ...) (mech-solid.jl:243-279,
//                          src/mech/mat/{linear-elastic,von-mises,drucker-prager}.jl)
//  * node_gather_kernel -- the dFin[map] .+= dF accumulation (mech-solver.jl:124-144)
//  * load kernels       -- mech_boundary_forces / mech_solid_body_forces
//                          (src/mech/elem/distributed.jl:76-217)
//
// Every material of the path has a tangent of the form D = De(lambda, mu) - gamma m m^T
// (isotropic elastic part plus a symmetric rank-one plastic correction), so the
// element stiffness is assembled per node pair (a, b) as
//     K_ab = lambda T_ab + mu T_ab^T + mu tr(T_ab) I - P_ab,
//     T_ab = sum_ip w_ip g_a g_b^T,   P_ab = sum_ip w_ip gamma_ip (S g_a)(S g_b)^T,
// with g = dN/dX at the IP, w_ip = detJ * weight * thickness and S the symmetric
// tensor of m.  This is B^T D B written without the zeros of B.  Axisymmetric
// analyses (mech-solid.jl:94-102,143) add the hoop strain u_r / r (B row zz =
// N_a / r on the radial component, h_a below) and take the thickness 2 pi r at
// the IP, r = sum N_a x_a: the pair formula gains the terms of h_a h_b, h_a g_b
// and g_a h_b, and the plastic vectors S g_a the term m_zz h_a.
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <mutex>
#include <set>
#include <type_traits>
#include <vector>

#include "amr_internal.h"

#define SQ2 1.4142135623730951
#define ISQ2 0.70710678118654752

namespace {

struct GroupArgs {
    const double *tab;  // [nip][nen*dim] dNdR, [nip] w, [nip][nen] N
    int nip;
    int64_t first, count;
    const double *geo_g = nullptr, *geo_w = nullptr;  // 3-D geometry cache of the group (null: compute it)
};

struct ModelArgs {
    const double *coords;
    const int32_t *conn;
    const int64_t *conn_ptr;
    const int32_t *mat_type;
    const double *mat_par;
    const int64_t *ip_ptr;
    const int64_t *kel_ptr;
    const int64_t *fel_ptr;
    int64_t nip_total;
    int stressmodel;
    double thickness;
    // batched stages: elements of inactive parts are skipped, errors are recorded per part
    const int32_t *elem_part;
    const uint8_t *part_active;
    int32_t *part_err;
};

__device__ __forceinline__ bool elem_skipped(const ModelArgs &M, int64_t e) {
    return M.part_active && !M.part_active[M.elem_part[e]];
}

__device__ __forceinline__ void set_status(int32_t *st, int code, int64_t elem) {
    atomicCAS(&st[0], 0, code);
    atomicMin(&st[1], (int32_t)(elem < INT32_MAX ? elem : INT32_MAX));
}

// Lame constants of De (plane stress uses lambda* = E nu / (1 - nu^2))
__device__ __forceinline__ void lame(double E, double nu, bool ps, double &lam, double &mu) {
    mu = E / (2.0 * (1.0 + nu));
    lam = ps ? E * nu / (1.0 - nu * nu) : E * nu / ((1.0 + nu) * (1.0 - 2.0 * nu));
}

// y = De x (Mandel, 6 components); plane stress has a zero zz row/column
__device__ __forceinline__ void De_mul(double lam, double mu, bool ps, const double *x, double *y) {
    if (ps) {
        double t = lam * (x[0] + x[1]);
        y[0] = t + 2.0 * mu * x[0]; y[1] = t + 2.0 * mu * x[1]; y[2] = 0.0;
    } else {
        double t = lam * (x[0] + x[1] + x[2]);
        y[0] = t + 2.0 * mu * x[0]; y[1] = t + 2.0 * mu * x[1]; y[2] = t + 2.0 * mu * x[2];
    }
    y[3] = 2.0 * mu * x[3]; y[4] = 2.0 * mu * x[4]; y[5] = 2.0 * mu * x[5];
}

// J2 and dev in Mandel notation (src/tools/tensors.jl:4-27)
__device__ __forceinline__ double J2(const double *s) {
    double t23 = s[3] * ISQ2, t13 = s[4] * ISQ2, t12 = s[5] * ISQ2;
    double a = s[0] - s[1], b = s[1] - s[2], c = s[2] - s[0];
    return (a * a + b * b + c * c) / 6.0 + t23 * t23 + t13 * t13 + t12 * t12;
}
__device__ __forceinline__ void dev(const double *t, double *s) {
    double p = (t[0] + t[1] + t[2]) / 3.0;
    s[0] = t[0] - p; s[1] = t[1] - p; s[2] = t[2] - p; s[3] = t[3]; s[4] = t[4]; s[5] = t[5];
}
__device__ __forceinline__ double norm6(const double *v) {
    return sqrt(v[0] * v[0] + v[1] * v[1] + v[2] * v[2] + v[3] * v[3] + v[4] * v[4] + v[5] * v[5]);
}

// Rank-one plastic part of the tangent: D = De - gamma m m^T.  Returns gamma (0 if elastic).
__device__ double plastic_tangent(int mtype, const double *par, bool ps, const double *sig, double epa, double dl,
                                  double lam, double mu, double *m) {
    if (mtype == AMR_LINEAR_ELASTIC || dl == 0.0) return 0.0;
    if (mtype == AMR_VON_MISES) {
        double fy = par[2], H = par[3];
        double a[6];
        if (!ps) {  // von-mises.jl:112-126: a = sqrt(1.5) s/|s|, den = a.De.a + sqrt(1.5) H
            double s[6];
            dev(sig, s);
            double ns = norm6(s);
            for (int i = 0; i < 6; i++) a[i] = sqrt(1.5) * s[i] / ns;
            De_mul(lam, mu, false, a, m);
            double den = 0.0;
            for (int i = 0; i < 6; i++) den += a[i] * m[i];
            return 1.0 / (den + sqrt(1.5) * H);
        }
        // plane stress (von-mises.jl:187-198)
        a[0] = 2.0 / 3.0 * sig[0] - 1.0 / 3.0 * sig[1];
        a[1] = 2.0 / 3.0 * sig[1] - 1.0 / 3.0 * sig[0];
        a[2] = -1.0 / 3.0 * sig[0] - 1.0 / 3.0 * sig[1];
        a[3] = sig[3]; a[4] = sig[4]; a[5] = sig[5];
        double dfdep = -2.0 / 3.0 * H * (fy + H * epa);
        De_mul(lam, mu, true, a, m);
        double den = 0.0;
        for (int i = 0; i < 6; i++) den += a[i] * m[i];
        return 1.0 / (den - norm6(a) * dfdep);
    }
    // Drucker-Prager (drucker-prager.jl:86-109): D = De - (De Nu)(De V)^T / (V.De.Nu + H), Nu = V/|V|
    double alpha = par[2], H = par[4];
    double V[6];
    double nv;
    if (J2(sig) != 0.0) {
        double s[6];
        dev(sig, s);
        double ns = norm6(s);
        for (int i = 0; i < 6; i++) V[i] = (i < 3 ? alpha : 0.0) + (s[i] / ns) * ISQ2;
        nv = norm6(V);
    } else {
        for (int i = 0; i < 6; i++) V[i] = (i < 3) ? 1.0 / sqrt(3.0) : 0.0;
        nv = 1.0;
    }
    De_mul(lam, mu, ps, V, m);
    double VDV = 0.0;
    for (int i = 0; i < 6; i++) VDV += V[i] * m[i];
    return 1.0 / (VDV + nv * H);  // = 1 / (|V| (V.De.Nu + H))
}

// Plane-stress von Mises stress for a given dlambda (von-mises.jl:306-333)
__device__ void vm_ps_sigma(double E, double nu, double epa0, const double *str, double dl, double *sig, double *epa) {
    double G = E / (2 * (1 + nu));
    double den = E * E * dl * dl - 2 * E * nu * dl + 4 * E * dl - 3 * nu * nu + 3;
    double m11 = (2 * E * dl - E * nu * dl - 3 * nu * nu + 3) / den;
    double m12 = (E * dl - 2 * E * nu * dl) / den;
    double m66 = 1 / (2 * G * dl + 1);
    sig[0] = m11 * str[0] + m12 * str[1];
    sig[1] = m12 * str[0] + m11 * str[1];
    sig[2] = 0.0;
    sig[3] = m66 * str[3]; sig[4] = m66 * str[4]; sig[5] = m66 * str[5];
    double d[6] = {2.0 / 3.0 * sig[0] - 1.0 / 3.0 * sig[1], 2.0 / 3.0 * sig[1] - 1.0 / 3.0 * sig[0],
                   -1.0 / 3.0 * sig[0] - 1.0 / 3.0 * sig[1], sig[3], sig[4], sig[5]};
    *epa = epa0 + dl * norm6(d);
}
__device__ __forceinline__ double vm_ps_yield(double fy, double H, const double *sig, double epa) {
    double k = fy + H * epa;
    return J2(sig) - k * k / 3.0;
}

// Constitutive update of one IP: st0 (committed, 14 fields) -> st1 (trial), returns dsig.
// 0 on success, AMR_ERETMAP on failure.
__device__ int material_update(int mtype, const double *par, bool ps, const double *st0, double *st1, const double *de,
                               double *dsig) {
    double E = par[0], nu = par[1], lam, mu;
    lame(E, nu, ps, lam, mu);
    double sig0[6], str[6], t[6];
    for (int i = 0; i < 6; i++) sig0[i] = st0[i];
    De_mul(lam, mu, ps, de, t);
    for (int i = 0; i < 6; i++) str[i] = sig0[i] + t[i];
    double epa = st0[AMR_ST_EPA], dl = st0[AMR_ST_DL];
    double sig[6];
    if (mtype == AMR_LINEAR_ELASTIC) {
        for (int i = 0; i < 6; i++) sig[i] = str[i];
    } else if (mtype == AMR_VON_MISES && !ps) {  // von-mises.jl:128-157
        double fy = par[2], H = par[3];
        double j2 = J2(str);
        double ftr = sqrt(3.0 * j2) - fy - H * epa;
        if (ftr < 1e-8) {
            dl = 0.0;
            for (int i = 0; i < 6; i++) sig[i] = str[i];
        } else {
            double G = E / (2 * (1 + nu));
            dl = ftr / (3 * G + sqrt(1.5) * H);
            if (!(sqrt(j2) - dl * sqrt(3.0) * G >= 0.0)) return AMR_ERETMAP;
            double s[6];
            dev(str, s);
            double f = 1 - sqrt(3.0) * G * dl / sqrt(j2);
            for (int i = 0; i < 6; i++) s[i] *= f;
            double ns = norm6(s);
            for (int i = 0; i < 6; i++) sig[i] = str[i] - sqrt(6.0) * G * dl * s[i] / ns;
            epa += dl;
        }
    } else if (mtype == AMR_VON_MISES) {  // plane stress, bisection (von-mises.jl:200-303)
        double fy = par[2], H = par[3];
        double ftr = vm_ps_yield(fy, H, str, epa);
        if (ftr < 1e-8) {
            dl = 0.0;
            for (int i = 0; i < 6; i++) sig[i] = str[i];
        } else {
            double dfds[6] = {2.0 / 3.0 * str[0] - 1.0 / 3.0 * str[1], 2.0 / 3.0 * str[1] - 1.0 / 3.0 * str[0],
                              -1.0 / 3.0 * str[0] - 1.0 / 3.0 * str[1], str[3], str[4], str[5]};
            double Dd[6], dd[6];
            De_mul(lam, mu, true, dfds, Dd);
            for (int i = 0; i < 6; i++) dd[i] = str[i] - sig0[i];
            double dl0 = norm6(dd) / norm6(Dd);
            double a = 0.0, b = dl0, sg[6], ep, fa, fb, f = 0.0;
            vm_ps_sigma(E, nu, epa, str, a, sg, &ep);
            fa = vm_ps_yield(fy, H, sg, ep);
            vm_ps_sigma(E, nu, epa, str, b, sg, &ep);
            fb = vm_ps_yield(fy, H, sg, ep);
            if (fa * fb > 0) {
                bool found = false;
                double g = 1.0;
                for (int i = 1; i <= 50; i++) {
                    g *= 1.6;
                    b += dl0 * g;
                    vm_ps_sigma(E, nu, epa, str, b, sg, &ep);
                    fb = vm_ps_yield(fy, H, sg, ep);
                    if (fa * fb < 0.0) { found = true; break; }
                }
                if (!found) return AMR_ERETMAP;
            }
            double s0[6] = {0, 0, 0, 0, 0, 0};
            double tol = pow(10.0, -(10.0 - log10(fy)));
            bool done = false;
            for (int i = 1; i <= 50; i++) {
                dl = 0.5 * (a + b);
                vm_ps_sigma(E, nu, epa, str, dl, sg, &ep);
                f = vm_ps_yield(fy, H, sg, ep);
                if (fa * f < 0) b = dl;
                else { a = dl; fa = f; }
                double mx = 0.0;
                for (int k = 0; k < 6; k++) mx = fmax(mx, fabs(sg[k] - s0[k]));
                if (mx <= tol) { done = true; break; }
                for (int k = 0; k < 6; k++) s0[k] = sg[k];
            }
            if (!done) return AMR_ERETMAP;
            for (int i = 0; i < 6; i++) sig[i] = sg[i];
            epa = ep;
        }
    } else {  // Drucker-Prager (drucker-prager.jl:112-149)
        double alpha = par[2], kappa = par[3], H = par[4];
        double j1 = str[0] + str[1] + str[2];
        double j2 = J2(str);
        double ftr = alpha * j1 + sqrt(j2) - kappa - H * epa;
        if (ftr < 1.e-8) {
            dl = 0.0;
            for (int i = 0; i < 6; i++) sig[i] = str[i];
        } else {
            double K = E / (3.0 * (1.0 - 2.0 * nu)), G = E / (2.0 * (1.0 + nu));
            double n = 1.0 / sqrt(3.0 * alpha * alpha + 0.5);
            if (sqrt(j2) - dl * n * G > 0.0) {  // uses the committed dgamma, as the reference does
                dl = ftr / (9 * alpha * alpha * n * K + n * G + H);
                double jj1 = j1 - 9 * dl * alpha * n * K;
                double mm = 1.0 - dl * n * G / sqrt(j2);
                double d[6];
                dev(str, d);
                for (int i = 0; i < 6; i++) sig[i] = mm * d[i] + (i < 3 ? jj1 / 3.0 : 0.0);
            } else {
                dl = (alpha * j1 - kappa - H * epa) / (3 * sqrt(3.0) * alpha * K + H);
                double jj1 = j1 - 3 * sqrt(3.0) * dl * K;
                for (int i = 0; i < 6; i++) sig[i] = (i < 3 ? jj1 / 3.0 : 0.0);
            }
            epa += dl;
        }
    }
    for (int i = 0; i < 6; i++) {
        st1[i] = sig[i];
        st1[6 + i] = st0[6 + i] + de[i];
        dsig[i] = sig[i] - sig0[i];
    }
    st1[AMR_ST_EPA] = epa;
    st1[AMR_ST_DL] = dl;
    return 0;
}

// Geometry at one IP: g = dN/dX (nen x DIM) and detJ from coordinates C (nen x DIM)
template <int DIM>
__device__ __forceinline__ double ip_geometry(int nen, const double *dNdR, const double *C, double *g) {
    double J[DIM * DIM];
#pragma unroll
    for (int q = 0; q < DIM * DIM; q++) J[q] = 0.0;
    for (int i = 0; i < nen; i++)
#pragma unroll
        for (int a = 0; a < DIM; a++)
#pragma unroll
            for (int b = 0; b < DIM; b++) J[a * DIM + b] += C[i * DIM + a] * dNdR[i * DIM + b];
    double det, iJ[DIM * DIM];
    if (DIM == 2) {
        det = J[0] * J[3] - J[1] * J[2];
        double r = 1.0 / det;
        iJ[0] = J[3] * r; iJ[1] = -J[1] * r; iJ[2] = -J[2] * r; iJ[3] = J[0] * r;
    } else {
        double c0 = J[4] * J[8] - J[5] * J[7], c1 = J[5] * J[6] - J[3] * J[8], c2 = J[3] * J[7] - J[4] * J[6];
        det = J[0] * c0 + J[1] * c1 + J[2] * c2;
        double r = 1.0 / det;
        iJ[0] = c0 * r; iJ[1] = (J[2] * J[7] - J[1] * J[8]) * r; iJ[2] = (J[1] * J[5] - J[2] * J[4]) * r;
        iJ[3] = c1 * r; iJ[4] = (J[0] * J[8] - J[2] * J[6]) * r; iJ[5] = (J[2] * J[3] - J[0] * J[5]) * r;
        iJ[6] = c2 * r; iJ[7] = (J[1] * J[6] - J[0] * J[7]) * r; iJ[8] = (J[0] * J[4] - J[1] * J[3]) * r;
    }
    for (int i = 0; i < nen; i++)
#pragma unroll
        for (int b = 0; b < DIM; b++) {
            double s = 0.0;
#pragma unroll
            for (int a = 0; a < DIM; a++) s += dNdR[i * DIM + a] * iJ[a * DIM + b];
            g[i * DIM + b] = s;
        }
    return det;
}

// Pair sums of the 3-D stiffness in float-float arithmetic (a value is hi + lo, two FP32 numbers, about 48
// significant bits).  On this GPU the FP32 pipe issues some 70 times as many FMAs per clock as the FP64 pipe,
// which bounds the FP64 element kernels; a float-float FMA takes about 12 FP32 operations.  Terms are
// products of two FP64 inputs split as hi = fl32(x), lo = fl32(x - hi); the product's hi*hi part is
// exact (Dekker's two-product with an FMA), the cross terms are added in FP32, lo*lo (2^-48 relative) is
// dropped, and the sum keeps its rounding errors (Knuth's two-sum).  Relative error per pair sum about
// 1e-13 of its largest term (27 terms), for terms within the FP32 exponent range.
// Every operation is an explicit round-to-nearest intrinsic, so the compiler fuses none of them.
struct FF {
    float hi, lo;
};
// x split into hi + lo, the pair kept in the 8 bytes of a double (hi in the low word): the shared arrays of
// g and w g are rewritten in place and stay double arrays.  The split is done on the integer pipe from the
// bit pattern (conversions from FP64 take the FP64 pipe): hi = x with its 52-bit fraction cut to 23 bits,
// lo = the remaining 29 bits cut to a float's 24 significant bits, both with the sign of x, so that
// |x - hi - lo| < 2^-46 |x|.  Zeros give two zeros; subnormal, infinite or NaN x, |x| below 2^-78 (where lo
// could leave the normal float range) or above the float range fall back to conversions.
__device__ __forceinline__ double ff_split(double x) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(x);
    const unsigned sign = (unsigned)(b >> 32) & 0x80000000u;
    const int ex = (int)((b >> 52) & 0x7ff);
    if (ex == 0 && (b << 1) == 0) return __hiloint2double((int)sign, (int)sign);  // +-0
    const int e = ex - 1023;
    if (ex == 0 || ex == 0x7ff || e < -78 || e > 127) {  // (lo could leave the normal float range)
        const float h = __double2float_rn(x);
        const float l = __double2float_rn(x - (double)h);
        return __hiloint2double(__float_as_int(l), __float_as_int(h));
    }
    const unsigned long long mant = b & 0xFFFFFFFFFFFFFull;
    const unsigned hb = sign | ((unsigned)(e + 127) << 23) | (unsigned)(mant >> 29);
    const unsigned m29 = (unsigned)(mant & 0x1FFFFFFFull);
    unsigned lb = 0;
    if (m29 != 0) {
        const int p = 31 - __clz((int)m29);  // the leading one of the tail, bit 0..28
        const int le = e - 52 + p;
        if (le >= -126) {
            const unsigned frac = (p >= 23 ? (m29 >> (p - 23)) : (m29 << (23 - p))) & 0x7FFFFFu;
            lb = sign | ((unsigned)(le + 127) << 23) | frac;
        }
    }
    return __hiloint2double((int)lb, (int)hb);
}
__device__ __forceinline__ float2 ff_get(double packed) {
    return make_float2(__int_as_float(__double2loint(packed)), __int_as_float(__double2hiint(packed)));
}
// a b as a float-float pair (packed): the exact hi*hi product plus the cross terms, renormalised
__device__ __forceinline__ double ff_mul(float2 a, float2 b) {
    const float p = __fmul_rn(a.x, b.x);
    float e = __fmaf_rn(a.x, b.x, -p);
    e = __fmaf_rn(a.x, b.y, e);
    e = __fmaf_rn(a.y, b.x, e);
    const float h = __fadd_rn(p, e);
    const float l = __fsub_rn(e, __fsub_rn(h, p));
    return __hiloint2double(__float_as_int(l), __float_as_int(h));
}
// s += b (a float-float pair), by two-sum
__device__ __forceinline__ void ff_acc(float2 b, FF &s) {
    const float t = __fadd_rn(s.hi, b.x);
    const float bp = __fsub_rn(t, s.hi);
    const float err = __fadd_rn(__fsub_rn(s.hi, __fsub_rn(t, bp)), __fsub_rn(b.x, bp));
    s.lo = __fadd_rn(s.lo, __fadd_rn(err, b.y));
    s.hi = t;
}
// the pair renormalised (|lo| at most half an ulp of hi), as the next operation's input
__device__ __forceinline__ float2 ff_norm(FF s) {
    const float h = __fadd_rn(s.hi, s.lo);
    return make_float2(h, __fsub_rn(s.lo, __fsub_rn(h, s.hi)));
}
// a float widened to double on the integer pipe (exact); zeros, subnormals, infinities and NaN take the
// conversion instruction
__device__ __forceinline__ double f2d(float f) {
    const unsigned u = __float_as_uint(f), ex = (u >> 23) & 0xffu;
    if (ex == 0u || ex == 0xffu) return (double)f;
    return __hiloint2double((int)((u & 0x80000000u) | ((ex + 896u) << 20) | ((u & 0x7FFFFFu) >> 3)),
                            (int)((u & 0x7u) << 29));
}
__device__ __forceinline__ void ff_fma(float2 a, float2 b, FF &s) {
    const float p = __fmul_rn(a.x, b.x);
    float e = __fmaf_rn(a.x, b.x, -p);
    e = __fmaf_rn(a.x, b.y, e);
    e = __fmaf_rn(a.y, b.x, e);
    const float t = __fadd_rn(s.hi, p);
    const float bp = __fsub_rn(t, s.hi);
    const float err = __fadd_rn(__fsub_rn(s.hi, __fsub_rn(t, bp)), __fsub_rn(p, bp));
    s.lo = __fadd_rn(s.lo, __fadd_rn(err, e));
    s.hi = t;
}

// S(m) g : the symmetric tensor of Mandel vector m applied to g (= B_a^T m)
template <int DIM>
__device__ __forceinline__ void sym_apply(const double *m, const double *g, double *v) {
    if (DIM == 3) {
        v[0] = m[0] * g[0] + m[5] * ISQ2 * g[1] + m[4] * ISQ2 * g[2];
        v[1] = m[5] * ISQ2 * g[0] + m[1] * g[1] + m[3] * ISQ2 * g[2];
        v[2] = m[4] * ISQ2 * g[0] + m[3] * ISQ2 * g[1] + m[2] * g[2];
    } else {
        v[0] = m[0] * g[0] + m[5] * ISQ2 * g[1];
        v[1] = m[5] * ISQ2 * g[0] + m[1] * g[1];
    }
}

// The 3-D geometry cache of a group: thread per (element, IP), dN/dX and w = detJ * weight * thickness by
// ip_geometry, the same operations as the element kernels' own; *bad set where detJ <= 0 (the cache is then
// not used, and the element kernels report the element as before).
template <int NEN>
__global__ void geometry_kernel(ModelArgs M, GroupArgs G, double *geo_g, double *geo_w, int32_t *bad) {
    const int nip = G.nip;
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= G.count * nip) return;
    const int64_t el = t / nip;
    const int ip = (int)(t % nip);
    const int64_t e = G.first + el;
    double C[NEN * 3], g[NEN * 3];
    for (int q = 0; q < NEN * 3; q++) C[q] = M.coords[3 * (int64_t)M.conn[M.conn_ptr[e] + q / 3] + q % 3];
    const double det = ip_geometry<3>(NEN, G.tab + ip * NEN * 3, C, g);
    if (!(det > 0.0)) atomicExch(bad, 1);
    for (int q = 0; q < NEN * 3; q++) geo_g[(el * NEN * 3 + q) * nip + ip] = g[q];
    geo_w[el * nip + ip] = det * G.tab[nip * NEN * 3 + ip] * M.thickness;
}

// ---------------------------------------------------------------------------
// Stiffness: EPB elements per CTA.  Phase 1: thread per (element, IP) builds
// g, w and the plastic vectors in shared memory.  Phase 2: thread per
// (element, node pair a<=b) accumulates T_ab / P_ab over the IPs and writes
// the two element blocks (a,b), (b,a) to the staging array.
// ---------------------------------------------------------------------------
// CTAs per SM the stiffness kernel's registers allow: two, so one CTA's geometry phase (FP64 pipe)
// overlaps another's pair phase (FP32 pipe in 3-D)
template <int DIM, int NEN>
constexpr int stiff_min_blocks() { return 2; }

template <int DIM, int NEN>
__global__ void __launch_bounds__(256, stiff_min_blocks<DIM, NEN>()) stiffness_kernel(ModelArgs M, GroupArgs G, int epb, double *Kel,
                                                        const double *st, int32_t *status) {
    constexpr int NP = NEN * (NEN + 1) / 2;
    constexpr int BB = DIM * DIM;
    extern __shared__ double sm[];
    const int nip = G.nip;
    double *sC = sm;                              // epb x NEN*DIM
    double *sG = sC + epb * NEN * DIM;            // epb x nip x NEN*DIM
    double *sV = sG + epb * nip * NEN * DIM;      // epb x nip x NEN*DIM (plastic vectors)
    double *sW = sV + epb * nip * NEN * DIM;      // epb x nip
    double *sGam = sW + epb * nip;                // epb x nip
    double *sWG = sGam + epb * nip;               // epb x nip x NEN*DIM: w * g, the rounded products of phase 2
    double *sH = sWG + epb * nip * NEN * DIM;     // axisymmetric: epb x nip x NEN, h = N / r
    __shared__ int sPl[8];                        // per element: any plastic IP
    __shared__ double sLam[8], sMu[8];            // per element: Lame constants

    const int64_t e0 = G.first + (int64_t)blockIdx.x * epb;
    const int ne = (int)min((int64_t)epb, G.first + G.count - e0);
    const double *dNdR = G.tab;
    const double *wq = G.tab + nip * NEN * DIM;
    const double *Nt = wq + nip;
    const bool ps = (M.stressmodel == AMR_PLANESTRESS);
    const bool axi = DIM == 2 && M.stressmodel == AMR_AXISYMMETRIC;

    for (int t = threadIdx.x; t < ne * NEN * DIM; t += blockDim.x) {
        int el = t / (NEN * DIM), q = t % (NEN * DIM);
        int32_t node = M.conn[M.conn_ptr[e0 + el] + q / DIM];
        sC[t] = M.coords[3 * (int64_t)node + q % DIM];
    }
    if (threadIdx.x < epb) sPl[threadIdx.x] = 0;
    __syncthreads();

    if constexpr (DIM == 3) {
      if (G.geo_g) {
        // 3-D with the geometry cache: (b) thread per (element, IP): w and the material's tangent; (c) thread per
        // (element, node, IP): dN/dX from the cache, the plastic vector and the float-float splits
        double *sMv = sH;                    // epb x nip x 6: the plastic tangent's vector m
        const int64_t el0 = e0 - G.first;
        for (int t = threadIdx.x; t < ne * nip; t += blockDim.x) {
            const int el = t / nip, ip = t % nip;
            const int64_t e = e0 + el;
            const double w = G.geo_w[(el0 + el) * nip + ip];
            sW[el * nip + ip] = w;
            const double *par = M.mat_par + 8 * e;
            const int64_t gi = M.ip_ptr[e] + ip;
            double sig[6];
            for (int i = 0; i < 6; i++) sig[i] = st[i * M.nip_total + gi];
            double lam, mu, m[6];
            lame(par[0], par[1], ps, lam, mu);
            if (ip == 0) { sLam[el] = lam; sMu[el] = mu; }
            const double gam = plastic_tangent(M.mat_type[e], par, ps, sig, st[AMR_ST_EPA * M.nip_total + gi],
                                               st[AMR_ST_DL * M.nip_total + gi], lam, mu, m);
            sGam[el * nip + ip] = gam * w;
            if (gam != 0.0) {
                sPl[el] = 1;
                for (int i = 0; i < 6; i++) sMv[(el * nip + ip) * 6 + i] = m[i];
            }
        }
        __syncthreads();
        for (int t = threadIdx.x; t < ne * nip * NEN; t += blockDim.x) {
            const int el = t / (nip * NEN), r = t % (nip * NEN), i = r / nip, ip = r % nip;
            double g[DIM];
#pragma unroll
            for (int bb = 0; bb < DIM; bb++) g[bb] = G.geo_g[((el0 + el) * NEN * DIM + i * DIM + bb) * nip + ip];
            const int ipo = (el * nip + ip) * NEN * DIM + i * DIM;
            if (sGam[el * nip + ip] != 0.0) sym_apply<DIM>(sMv + (el * nip + ip) * 6, g, sV + ipo);
            const float2 wf = ff_get(ff_split(sW[el * nip + ip]));
#pragma unroll
            for (int bb = 0; bb < DIM; bb++) {
                const double gs = ff_split(g[bb]);
                sG[ipo + bb] = gs;
                sWG[ipo + bb] = ff_mul(wf, ff_get(gs));
            }
        }
      } else {
        // 3-D: the geometry spread over the CTA (the FP64 pipe is the bound, and a thread per IP left it to one
        // warp while the others waited at the barrier).  (a) thread per (element, IP, Jacobian entry)
        double *sJ = sH;                     // epb x nip x 9: J, then its inverse
        double *sMv = sJ + epb * nip * 9;    // epb x nip x 6: the plastic tangent's vector m
        for (int t = threadIdx.x; t < ne * nip * 9; t += blockDim.x) {
            const int el = t / (nip * 9), r = t % (nip * 9), ip = r / 9, a = (r % 9) / 3, bb = r % 3;
            const double *C = sC + el * NEN * DIM, *dN = dNdR + ip * NEN * DIM;
            double J = 0.0;
            for (int i = 0; i < NEN; i++) J = fma(C[i * DIM + a], dN[i * DIM + bb], J);
            sJ[(el * nip + ip) * 9 + r % 9] = J;
        }
        __syncthreads();
        // (b) thread per (element, IP): determinant, inverse, weight and the material's tangent
        for (int t = threadIdx.x; t < ne * nip; t += blockDim.x) {
            const int el = t / nip, ip = t % nip;
            const int64_t e = e0 + el;
            double *J = sJ + (el * nip + ip) * 9;
            const double c0 = J[4] * J[8] - J[5] * J[7], c1 = J[5] * J[6] - J[3] * J[8], c2 = J[3] * J[7] - J[4] * J[6];
            const double det = J[0] * c0 + J[1] * c1 + J[2] * c2;
            const double rd = 1.0 / det;
            double iJ[9];
            iJ[0] = c0 * rd; iJ[1] = (J[2] * J[7] - J[1] * J[8]) * rd; iJ[2] = (J[1] * J[5] - J[2] * J[4]) * rd;
            iJ[3] = c1 * rd; iJ[4] = (J[0] * J[8] - J[2] * J[6]) * rd; iJ[5] = (J[2] * J[3] - J[0] * J[5]) * rd;
            iJ[6] = c2 * rd; iJ[7] = (J[1] * J[6] - J[0] * J[7]) * rd; iJ[8] = (J[0] * J[4] - J[1] * J[3]) * rd;
#pragma unroll
            for (int q = 0; q < 9; q++) J[q] = iJ[q];
            if (!(det > 0.0)) set_status(status, AMR_ENEGJAC, e);
            const double w = det * wq[ip] * M.thickness;
            sW[el * nip + ip] = w;
            const double *par = M.mat_par + 8 * e;
            const int64_t gi = M.ip_ptr[e] + ip;
            double sig[6];
            for (int i = 0; i < 6; i++) sig[i] = st[i * M.nip_total + gi];
            double lam, mu, m[6];
            lame(par[0], par[1], ps, lam, mu);
            if (ip == 0) { sLam[el] = lam; sMu[el] = mu; }
            const double gam = plastic_tangent(M.mat_type[e], par, ps, sig, st[AMR_ST_EPA * M.nip_total + gi],
                                               st[AMR_ST_DL * M.nip_total + gi], lam, mu, m);
            sGam[el * nip + ip] = gam * w;
            if (gam != 0.0) {
                sPl[el] = 1;
                for (int i = 0; i < 6; i++) sMv[(el * nip + ip) * 6 + i] = m[i];
            }
        }
        __syncthreads();
        // (c) thread per (element, IP, node): g = dN/dX, the plastic vector S(m) g, and g and w g as float-float
        // pairs for the pair sums
        for (int t = threadIdx.x; t < ne * nip * NEN; t += blockDim.x) {
            const int el = t / (nip * NEN), r = t % (nip * NEN), ip = r / NEN, i = r % NEN;
            const double *iJ = sJ + (el * nip + ip) * 9, *dN = dNdR + ip * NEN * DIM + i * DIM;
            double g[DIM];
#pragma unroll
            for (int bb = 0; bb < DIM; bb++) {
                double sum = 0.0;
#pragma unroll
                for (int a = 0; a < DIM; a++) sum = fma(dN[a], iJ[a * DIM + bb], sum);
                g[bb] = sum;
            }
            const int ipo = (el * nip + ip) * NEN * DIM + i * DIM;
            if (sGam[el * nip + ip] != 0.0) sym_apply<DIM>(sMv + (el * nip + ip) * 6, g, sV + ipo);
            const float2 wf = ff_get(ff_split(sW[el * nip + ip]));
#pragma unroll
            for (int bb = 0; bb < DIM; bb++) {
                const double gs = ff_split(g[bb]);
                sG[ipo + bb] = gs;
                sWG[ipo + bb] = ff_mul(wf, ff_get(gs));
            }
        }
      }
    } else
    for (int t = threadIdx.x; t < ne * nip; t += blockDim.x) {
        int el = t / nip, ip = t % nip;
        int64_t e = e0 + el;
        double *g = sG + (el * nip + ip) * NEN * DIM;
        double det = ip_geometry<DIM>(NEN, dNdR + ip * NEN * DIM, sC + el * NEN * DIM, g);
        if (!(det > 0.0)) set_status(status, AMR_ENEGJAC, e);
        double th = M.thickness;
        if (axi) {
            const double *N = Nt + ip * NEN, *C = sC + el * NEN * DIM;
            double r = 0.0;
            for (int a = 0; a < NEN; a++) r += C[a * DIM] * N[a];
            th = 2 * M_PI * r;
            double *h = sH + (el * nip + ip) * NEN;
            for (int a = 0; a < NEN; a++) h[a] = N[a] / r;
        }
        double w = det * wq[ip] * th;
        sW[el * nip + ip] = w;
        {
            double *wg = sWG + (el * nip + ip) * NEN * DIM;
            for (int q = 0; q < NEN * DIM; q++) wg[q] = w * g[q];
        }
        const double *par = M.mat_par + 8 * e;
        int64_t gi = M.ip_ptr[e] + ip;
        double sig[6];
        for (int i = 0; i < 6; i++) sig[i] = st[i * M.nip_total + gi];
        double lam, mu, m[6];
        lame(par[0], par[1], ps, lam, mu);
        if (ip == 0) { sLam[el] = lam; sMu[el] = mu; }
        double gam = plastic_tangent(M.mat_type[e], par, ps, sig, st[AMR_ST_EPA * M.nip_total + gi],
                                     st[AMR_ST_DL * M.nip_total + gi], lam, mu, m);
        sGam[el * nip + ip] = gam * w;
        if (gam != 0.0) {
            sPl[el] = 1;
            double *v = sV + (el * nip + ip) * NEN * DIM;
            for (int a = 0; a < NEN; a++) sym_apply<DIM>(m, g + a * DIM, v + a * DIM);
            if (axi)
                for (int a = 0; a < NEN; a++) v[a * DIM] += m[2] * sH[(el * nip + ip) * NEN + a];
        }
    }
    __syncthreads();

    for (int t = threadIdx.x; t < ne * NP; t += blockDim.x) {
        int el = t / NP, p = t % NP;
        int a = 0, rem = p;
        while (rem >= NEN - a) { rem -= NEN - a; a++; }
        int b = a + rem;
        int64_t e = e0 + el;
        double T[BB], P[BB];
#pragma unroll
        for (int q = 0; q < BB; q++) { T[q] = 0.0; P[q] = 0.0; }
        const double *gbase = sG + el * nip * NEN * DIM;
        const double *wgbase = sWG + el * nip * NEN * DIM;
        FF tf[BB];  // 3-D: T_ab in float-float
        if (DIM == 3) {
#pragma unroll
            for (int q = 0; q < BB; q++) tf[q] = FF{0.0f, 0.0f};
            for (int ip = 0; ip < nip; ip++) {
                const double *wa = wgbase + ip * NEN * DIM + a * DIM;
                const double *gb = gbase + ip * NEN * DIM + b * DIM;
                float2 wv[DIM], gv[DIM];
#pragma unroll
                for (int i = 0; i < DIM; i++) { wv[i] = ff_get(wa[i]); gv[i] = ff_get(gb[i]); }
#pragma unroll
                for (int i = 0; i < DIM; i++)
#pragma unroll
                    for (int j = 0; j < DIM; j++) ff_fma(wv[i], gv[j], tf[i * DIM + j]);
            }
        } else {
            for (int ip = 0; ip < nip; ip++) {
                const double *wa = wgbase + ip * NEN * DIM + a * DIM;
                const double *gb = gbase + ip * NEN * DIM + b * DIM;
#pragma unroll
                for (int i = 0; i < DIM; i++)
#pragma unroll
                    for (int j = 0; j < DIM; j++) T[i * DIM + j] = fma(wa[i], gb[j], T[i * DIM + j]);
            }
        }
        if (sPl[el]) {
            const double *vbase = sV + el * nip * NEN * DIM;
            for (int ip = 0; ip < nip; ip++) {
                double gm = sGam[el * nip + ip];
                if (gm == 0.0) continue;
                const double *va = vbase + ip * NEN * DIM + a * DIM;
                const double *vb = vbase + ip * NEN * DIM + b * DIM;
#pragma unroll
                for (int i = 0; i < DIM; i++) {
                    double x = gm * va[i];
#pragma unroll
                    for (int j = 0; j < DIM; j++) P[i * DIM + j] = fma(x, vb[j], P[i * DIM + j]);
                }
            }
        }
        const double lam = sLam[el], mu = sMu[el];
        double K[BB];
        if (DIM == 3) {
            // lambda T + mu T' + mu tr(T) I in float-float too, each entry widened to FP64 once (one FP64 add), then
            // the plastic part in FP64
            float2 tn[BB];
#pragma unroll
            for (int q = 0; q < BB; q++) tn[q] = ff_norm(tf[q]);
            FF trs{tn[0].x, tn[0].y};
            ff_acc(tn[4], trs);
            ff_acc(tn[8], trs);
            const float2 trn = ff_norm(trs);
            const float2 lamf = ff_get(ff_split(lam)), muf = ff_get(ff_split(mu));
#pragma unroll
            for (int i = 0; i < DIM; i++)
#pragma unroll
                for (int j = 0; j < DIM; j++) {
                    FF kk{0.0f, 0.0f};
                    ff_fma(lamf, tn[i * DIM + j], kk);
                    ff_fma(muf, tn[j * DIM + i], kk);
                    if (i == j) ff_fma(muf, trn, kk);
                    K[i * DIM + j] = (f2d(kk.hi) + f2d(kk.lo)) - P[i * DIM + j];
                }
        } else {
            double tr = 0.0;
#pragma unroll
            for (int i = 0; i < DIM; i++) tr += T[i * DIM + i];
#pragma unroll
            for (int i = 0; i < DIM; i++)
#pragma unroll
                for (int j = 0; j < DIM; j++)
                    K[i * DIM + j] = lam * T[i * DIM + j] + mu * T[j * DIM + i] + (i == j ? mu * tr : 0.0) - P[i * DIM + j];
        }
        if (axi) {  // hoop terms: X1 = sum w h_a g_b, X2 = sum w g_a h_b, X3 = sum w h_a h_b
            double X1[2] = {0.0, 0.0}, X2[2] = {0.0, 0.0}, X3 = 0.0;
            for (int ip = 0; ip < nip; ip++) {
                const double *hh = sH + (el * nip + ip) * NEN;
                const double wha = sW[el * nip + ip] * hh[a], hb = hh[b];
                const double *wa = wgbase + ip * NEN * DIM + a * DIM;
                const double *gb = gbase + ip * NEN * DIM + b * DIM;
                X1[0] = fma(wha, gb[0], X1[0]); X1[1] = fma(wha, gb[1], X1[1]);
                X2[0] = fma(wa[0], hb, X2[0]); X2[1] = fma(wa[1], hb, X2[1]);
                X3 = fma(wha, hb, X3);
            }
            K[0] += lam * (X1[0] + X2[0] + X3) + 2.0 * mu * X3;
            K[1] += lam * X1[1];
            K[DIM] += lam * X2[1];
        }
        int64_t base = M.kel_ptr[e];
        double *o1 = Kel + (base + (int64_t)a * NEN + b) * BB;
#pragma unroll
        for (int q = 0; q < BB; q++) o1[q] = K[q];
        if (a != b) {
            double *o2 = Kel + (base + (int64_t)b * NEN + a) * BB;
#pragma unroll
            for (int i = 0; i < DIM; i++)
#pragma unroll
                for (int j = 0; j < DIM; j++) o2[j * DIM + i] = K[i * DIM + j];
        }
    }
}

// ---------------------------------------------------------------------------
// Reference-order stiffness: K_e = sum_ip coef * B^T (D B) evaluated exactly in
// the order of elem_stiffness (src/mech/elem/mech-solid.jl:142-158): J = C^T dN/dR,
// cofactor inverse, dN/dX, DB = D*B and K += coef*(B^T DB) with row-sequential
// sums, every product and sum rounded separately (no FMA contraction).  With
// the same dN/dR tables this reproduces the CPU restatement bit for bit, so the
// |K_ij| >= eps() decisions of entries that are zero only by cancellation come
// out as the reference's arithmetic makes them.  Used for the parity / export
// path; the fast kernel above serves the Newton loop.
// ---------------------------------------------------------------------------
#define RMUL __dmul_rn
#define RADD __dadd_rn
#define RSUB __dsub_rn
#define RDIV __ddiv_rn

// The nonzero rows of column (b, d) of B (setB, mech-solid.jl:82-121), ascending: kRefTerms of them, row(q) and value(q).
// g = dN/dX of node b, gs = g / sqrt(2) of the shear rows, hb = N_b / r, the hoop row of an axisymmetric analysis.
// Where a sum of the reference runs over all six rows, the products with B's zeros are left out: they add +-0 to
// sums that start at +0, which changes no bit of them.
constexpr int kRefTerms = 3;
template <int DIM>
__device__ __forceinline__ int ref_row(int q, int d) {
    if (DIM == 3) return q == 0 ? d : q == 1 ? (d == 0 ? 4 : 3) : (d == 2 ? 4 : 5);
    return q == 0 ? d : q == 1 ? 2 : 5;
}
template <int DIM>
__device__ __forceinline__ double ref_value(int q, int d, const double *g, const double *gs, double hb) {
    if (DIM == 3) return q == 0 ? g[d] : q == 1 ? gs[d == 2 ? 1 : 2] : gs[d == 0 ? 1 : 0];
    return q == 0 ? g[d] : q == 1 ? (d == 0 ? hb : 0.0) : gs[d == 0 ? 1 : 0];
}

// One element per CTA.  The geometry of all integration points first, a thread per entry: Jacobians, inverses (a division
// per thread), dN/dX and its shear form g / sqrt(2) (once, not at each use in a product), D; then D B for kRefChunk
// points at a time and the sums of B' (D B).  The FP64 pipe bounds it: 7 operations per entry and point, 0.3 ms for
// 4 901 HEX8 elements.  With a thread's serial geometry per point and B formed with its divisions inside the sums it
// took 4.1 ms there; now the whole assembly, gather and synchronisation included, takes 0.52 ms.
constexpr int kRefChunk = 8;
template <int DIM, int NEN>
__host__ __device__ constexpr int ref_doubles(int nip) {  // shared memory of the CTA, in doubles
    return NEN * DIM + nip * (2 * NEN * DIM + 36 + 2 * DIM * DIM + 1 + NEN) +
           (nip < kRefChunk ? nip : kRefChunk) * 6 * NEN * DIM;
}

template <int DIM, int NEN>
__global__ void __launch_bounds__(256) stiffness_ref_kernel(ModelArgs M, GroupArgs G, double *Kel, const double *st,
                                                            int32_t *status) {
    constexpr int ND = NEN * DIM, JJ = DIM * DIM;
    constexpr int NE = (ND * ND + 255) / 256;
    extern __shared__ double sm[];
    const int64_t e = G.first + blockIdx.x;
    const int nip = G.nip;
    double *sC = sm;                  // ND
    double *sG = sC + ND;             // nip x ND: dN/dX
    double *sS = sG + nip * ND;       // nip x ND: dN/dX / sqrt(2)
    double *sD = sS + nip * ND;       // nip x 36
    double *sJ = sD + nip * 36;       // nip x JJ
    double *sIJ = sJ + nip * JJ;      // nip x JJ
    double *sCoef = sIJ + nip * JJ;   // nip
    double *sH = sCoef + nip;         // nip x NEN
    double *sDB = sH + nip * NEN;     // chunk x 6 x ND
    const bool ps = (M.stressmodel == AMR_PLANESTRESS);
    const bool axi = DIM == 2 && M.stressmodel == AMR_AXISYMMETRIC;
    for (int t = threadIdx.x; t < ND; t += blockDim.x) {
        int32_t node = M.conn[M.conn_ptr[e] + t / DIM];
        sC[t] = M.coords[3 * (int64_t)node + t % DIM];
    }
    double acc[NE];
#pragma unroll
    for (int q = 0; q < NE; q++) acc[q] = 0.0;
    const double *par = M.mat_par + 8 * e;
    __syncthreads();
    for (int t = threadIdx.x; t < nip * JJ; t += blockDim.x) {  // J = C' dN/dR
        const int ip = t / JJ, a = t % JJ / DIM, b = t % DIM;
        const double *dNdR = G.tab + ip * ND;
        double s = 0.0;
        for (int i = 0; i < NEN; i++) s = RADD(s, RMUL(sC[i * DIM + a], dNdR[i * DIM + b]));
        sJ[t] = s;
    }
    __syncthreads();
    for (int t = threadIdx.x; t < nip * JJ; t += blockDim.x) {  // inv(J) by cofactors; the determinant by each thread
        const int ip = t / JJ, q = t % JJ;
        const double *J = sJ + ip * JJ;
        double det, num;
        if (DIM == 2) {
            det = RSUB(RMUL(J[0], J[3]), RMUL(J[1], J[2]));
            num = q == 0 ? J[3] : q == 1 ? -J[1] : q == 2 ? -J[2] : J[0];
        } else {
            const double c0 = RSUB(RMUL(J[4], J[8]), RMUL(J[5], J[7]));
            const double c1 = RSUB(RMUL(J[3], J[8]), RMUL(J[5], J[6]));
            const double c2 = RSUB(RMUL(J[3], J[7]), RMUL(J[4], J[6]));
            det = RADD(RSUB(RMUL(J[0], c0), RMUL(J[1], c1)), RMUL(J[2], c2));
            // entry (r, c) of the inverse: cofactor (c, r), as a difference of two products
            const int r = q / 3, c = q % 3;
            const int r1 = (c + 1) % 3, r2 = (c + 2) % 3, c1i = (r + 1) % 3, c2i = (r + 2) % 3;
            num = RSUB(RMUL(J[r1 * 3 + c1i], J[r2 * 3 + c2i]), RMUL(J[r1 * 3 + c2i], J[r2 * 3 + c1i]));
        }
        sIJ[t] = RDIV(num, det);
        if (q == 0) {
            if (!(det > 0.0)) set_status(status, AMR_ENEGJAC, e);
            double th = M.thickness;
            if (axi) {  // r = ip.coord.x, th = 2 pi r (mech-solid.jl:143), h = N / r
                const double *N = G.tab + nip * ND + nip + ip * NEN;
                double r = 0.0;
                for (int i = 0; i < NEN; i++) r = RADD(r, RMUL(sC[i * DIM], N[i]));
                th = RMUL(2 * M_PI, r);
                for (int i = 0; i < NEN; i++) sH[ip * NEN + i] = RDIV(N[i], r);
            } else {
                for (int i = 0; i < NEN; i++) sH[ip * NEN + i] = 0.0;
            }
            sCoef[ip] = RMUL(RMUL(det, G.tab[nip * ND + ip]), th);
        }
    }
    // D: calcDe (linear-elastic.jl:98-119), plastic part as De - gamma m m'; the last threads, which have least to do above
    for (int ip = blockDim.x - 1 - threadIdx.x; ip < nip; ip += blockDim.x) {
        double *D = sD + ip * 36;
        const double E = par[0], nu = par[1];
        for (int q = 0; q < 36; q++) D[q] = 0.0;
        if (ps) {
            double c = RDIV(E, RSUB(1.0, RMUL(nu, nu)));
            D[0] = c; D[1] = RMUL(c, nu); D[6] = RMUL(c, nu); D[7] = c;
            double sh = RMUL(c, RSUB(1.0, nu));
            D[21] = sh; D[28] = sh; D[35] = sh;
        } else {
            double c = RDIV(E, RMUL(RADD(1.0, nu), RSUB(1.0, RMUL(2.0, nu))));
            for (int i = 0; i < 3; i++)
                for (int j = 0; j < 3; j++) D[6 * i + j] = (i == j) ? RMUL(c, RSUB(1.0, nu)) : RMUL(c, nu);
            double sh = RMUL(c, RSUB(1.0, RMUL(2.0, nu)));
            D[21] = sh; D[28] = sh; D[35] = sh;
        }
        if (M.mat_type[e] != AMR_LINEAR_ELASTIC) {
            int64_t gi = M.ip_ptr[e] + ip;
            double sig[6], m[6], lam, mu;
            for (int i = 0; i < 6; i++) sig[i] = st[i * M.nip_total + gi];
            lame(E, nu, ps, lam, mu);
            double gam = plastic_tangent(M.mat_type[e], par, ps, sig, st[AMR_ST_EPA * M.nip_total + gi],
                                         st[AMR_ST_DL * M.nip_total + gi], lam, mu, m);
            if (gam != 0.0)
                for (int i = 0; i < 6; i++)
                    for (int j = 0; j < 6; j++) D[6 * i + j] -= gam * m[i] * m[j];
        }
    }
    __syncthreads();
    for (int t = threadIdx.x; t < nip * ND; t += blockDim.x) {  // dNdX = dNdR * inv(J)
        const int ip = t / ND, i = t % ND / DIM, b = t % DIM;
        const double *dNdR = G.tab + ip * ND, *iJ = sIJ + ip * JJ;
        double s = 0.0;
        for (int a = 0; a < DIM; a++) s = RADD(s, RMUL(dNdR[i * DIM + a], iJ[a * DIM + b]));
        sG[t] = s;
        sS[t] = RDIV(s, SQ2);
    }
    for (int ip0 = 0; ip0 < nip; ip0 += kRefChunk) {
        const int nc = min(kRefChunk, nip - ip0);
        __syncthreads();
        for (int t = threadIdx.x; t < nc * 6 * ND; t += blockDim.x) {  // DB = D * B
            const int ip = ip0 + t / (6 * ND), k = t / ND % 6, j = t % ND, b = j / DIM, d = j % DIM;
            const double *g = sG + ip * ND + b * DIM, *gs = sS + ip * ND + b * DIM, *D = sD + ip * 36 + 6 * k;
            const double hb = sH[ip * NEN + b];
            double s = 0.0;
#pragma unroll
            for (int q = 0; q < kRefTerms; q++)
                s = RADD(s, RMUL(D[ref_row<DIM>(q, d)], ref_value<DIM>(q, d, g, gs, hb)));
            sDB[t] = s;
        }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < NE; q++) {  // K += coef * B' * DB
            const int idx = threadIdx.x + q * 256;
            if (idx < ND * ND) {
                const int i = idx / ND, j = idx % ND, a = i / DIM, c = i % DIM;
                double v = acc[q];
                for (int l = 0; l < nc; l++) {
                    const int ip = ip0 + l;
                    const double *g = sG + ip * ND + a * DIM, *gs = sS + ip * ND + a * DIM, *DB = sDB + l * 6 * ND + j;
                    const double hb = DIM == 2 ? sH[ip * NEN + a] : 0.0;
                    double s = 0.0;
#pragma unroll
                    for (int u = 0; u < kRefTerms; u++) {
                        const double x = RMUL(ref_value<DIM>(u, c, g, gs, hb), DB[ref_row<DIM>(u, c) * ND]);
                        s = u == 0 ? x : RADD(s, x);
                    }
                    v = RADD(v, RMUL(sCoef[ip], s));
                }
                acc[q] = v;
            }
        }
    }
    const int64_t base = M.kel_ptr[e];
#pragma unroll
    for (int q = 0; q < NE; q++) {
        int idx = threadIdx.x + q * 256;
        if (idx < ND * ND) {
            int i = idx / ND, j = idx % ND;
            int a = i / DIM, c = i % DIM, b = j / DIM, d = j % DIM;
            Kel[(base + (int64_t)a * NEN + b) * DIM * DIM + c * DIM + d] = acc[q];
        }
    }
}

// ---------------------------------------------------------------------------
// Gather: warp per node row, lane per nonzero block.  Contributions are summed
// in element order skipping |Ke_ij| < eps() (the mount_K drop rule); the keep
// bits record which scalar entries the reference's sparse() would store.
// Also writes the Dirichlet-masked FP32 copy and the block-Jacobi inverses.
// ---------------------------------------------------------------------------
template <int B>
__device__ void invert_block(const double *A, double *X) {
    if (B == 2) {
        double d = A[0] * A[3] - A[1] * A[2];
        X[0] = A[3] / d; X[1] = -A[1] / d; X[2] = -A[2] / d; X[3] = A[0] / d;
    } else {
        double c0 = A[4] * A[8] - A[5] * A[7], c1 = A[5] * A[6] - A[3] * A[8], c2 = A[3] * A[7] - A[4] * A[6];
        double d = A[0] * c0 + A[1] * c1 + A[2] * c2;
        X[0] = c0 / d; X[1] = (A[2] * A[7] - A[1] * A[8]) / d; X[2] = (A[1] * A[5] - A[2] * A[4]) / d;
        X[3] = c1 / d; X[4] = (A[0] * A[8] - A[2] * A[6]) / d; X[5] = (A[2] * A[3] - A[0] * A[5]) / d;
        X[6] = c2 / d; X[7] = (A[1] * A[6] - A[0] * A[7]) / d; X[8] = (A[0] * A[4] - A[1] * A[3]) / d;
    }
}

// x rounded to the nearest float (ties to even), on the integer pipe from the bit pattern: bitwise the same
// as the conversion instruction, which takes the FP64 pipe on this GPU.  Zeros, subnormals, infinities, NaN and
// results outside the normal float range take the conversion instruction.
__device__ __forceinline__ float d2f_rn(double x) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(x);
    const unsigned sign = (unsigned)(b >> 32) & 0x80000000u;
    const int ex = (int)((b >> 52) & 0x7ff);
    const int e = ex - 1023;
    if (ex == 0 || ex == 0x7ff || e < -126 || e > 127) return __double2float_rn(x);
    const unsigned long long mant = b & 0xFFFFFFFFFFFFFull;
    const unsigned keep = (unsigned)(mant >> 29), rem = (unsigned)(mant & 0x1FFFFFFFull);
    const unsigned up = (rem > 0x10000000u || (rem == 0x10000000u && (keep & 1u))) ? 1u : 0u;
    const unsigned r = ((unsigned)(e + 127) << 23) + keep + up;  // a carry into the exponent is the right result
    if ((r >> 23) >= 255u) return __double2float_rn(x);          // rounds to infinity
    return __uint_as_float(sign | r);
}

// Block k (row n, column j) of K with values v: the Dirichlet-masked FP32 copy (unit diagonal at
// prescribed DOFs) and, on the diagonal, the block-Jacobi inverses.
template <int B>
__device__ __forceinline__ void finish_block(int64_t n, int64_t k, int32_t j, int64_t nblocks, const double *v,
                                             const uint8_t *fr, const uint8_t *free_mask, float *K32, float *Minv32,
                                             double *Minv64) {
    constexpr int BB = B * B;
    if (!K32 && !Minv32) return;
    uint8_t fc[B];
#pragma unroll
    for (int d = 0; d < B; d++) fc[d] = free_mask ? free_mask[(int64_t)j * B + d] : 1;
    double mk[BB];
#pragma unroll
    for (int c = 0; c < B; c++)
#pragma unroll
        for (int d = 0; d < B; d++) {
            double x = (fr[c] && fc[d]) ? v[c * B + d] : 0.0;
            if (j == n && c == d && !fr[c]) x = 1.0;
            mk[c * B + d] = x;
        }
    if (K32)
#pragma unroll
        for (int q = 0; q < BB; q++) K32[(int64_t)q * nblocks + k] = d2f_rn(mk[q]);
    if (j == n) {
        double X[BB];
        invert_block<B>(mk, X);
#pragma unroll
        for (int q = 0; q < BB; q++) {
            if (Minv32) Minv32[n * BB + q] = d2f_rn(X[q]);
            if (Minv64) Minv64[n * BB + q] = X[q];
        }
    }
}

// |x| < eps() and isnan(x) on the integer pipe, from the bit pattern (the FP64 pipe is the gather's
// bound on this GPU): the sign-cleared pattern of a double orders as its magnitude, NaNs above infinity
__device__ __forceinline__ bool below_eps(double x) {
    return (__double_as_longlong(x) & 0x7fffffffffffffffLL) < 0x3cb0000000000000LL;  // 2^-52
}
__device__ __forceinline__ bool is_nan_bits(double x) {
    return (__double_as_longlong(x) & 0x7fffffffffffffffLL) > 0x7ff0000000000000LL;
}

// A thread per block, the blocks taken in the order gorder, which groups them by their number of
// contributions: a warp's lanes then run equal contribution loops.  (A warp per node row with a lane per
// block left most lanes idle on the FP64 pipe, which bounds this kernel: the blocks of a HEX20 node row have
// 1 to 8 contributions each.)
template <int B>
__global__ void gather_kernel(int64_t nblocks, const int32_t *gorder, const int32_t *grow, const int32_t *bcol,
                                     const int64_t *contrib_ptr, const int64_t *contrib, const double *Kel,
                                     const uint8_t *free_mask, double *K64, int64_t stride, float *K32,
                                     uint16_t *keep, float *Minv32, double *Minv64, int32_t *status) {
    constexpr int BB = B * B;
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nblocks) return;
    const int64_t k = gorder[t];
    const int64_t n = grow[k];
    uint8_t fr[B];
#pragma unroll
    for (int c = 0; c < B; c++) fr[c] = free_mask ? free_mask[n * B + c] : 1;
    double v[BB];
#pragma unroll
    for (int q = 0; q < BB; q++) v[q] = 0.0;
    unsigned kb = 0;
    const int64_t c0 = contrib_ptr[k], c1 = contrib_ptr[k + 1];
    if (c0 < c1) {  // the first contribution is taken as it is: 0 + x = x, one FP64 add per entry saved
        const double *src = Kel + contrib[c0] * BB;
#pragma unroll
        for (int q = 0; q < BB; q++) {
            const double x = src[q];
            if (!below_eps(x)) { v[q] = x; kb |= 1u << q; }  // (-0 is below eps: v stays +0, as 0 + x leaves it)
        }
    }
    for (int64_t c = c0 + 1; c < c1; c++) {
        const double *src = Kel + contrib[c] * BB;
#pragma unroll
        for (int q = 0; q < BB; q++) {
            double x = src[q];
            if (!below_eps(x)) { v[q] += x; kb |= 1u << q; }  // NaN is pushed, as in mount_K
        }
    }
    const int32_t j = bcol[k];
    bool nan = false;
#pragma unroll
    for (int q = 0; q < BB; q++) {
        K64[(int64_t)q * stride + k] = v[q];
        nan |= is_nan_bits(v[q]);
    }
    if (nan) set_status(status, AMR_ENAN, -1);
    if (keep) keep[k] = (uint16_t)kb;
    finish_block<B>(n, k, j, stride, v, fr, free_mask, K32, Minv32, Minv64);
}

// K = a1 Ks + a2 K (the weighted tangent of the ME / BE / Ralston schemes, mech-solver.jl:280-288,
// K = a1*K + a2*K2 at :342-343): products and sum rounded separately, then the masked FP32 copy and
// block-Jacobi inverses of the result.
template <int B>
__global__ void combine_kernel(int64_t nnodes, int64_t nblocks, const int64_t *brow_ptr, const int32_t *bcol, double a1,
                               const double *Ks, double a2, const uint8_t *free_mask, double *K64, float *K32,
                               float *Minv32, double *Minv64, int32_t *status) {
    constexpr int BB = B * B;
    int lane = threadIdx.x & 31;
    int64_t n = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (n >= nnodes) return;
    uint8_t fr[B];
#pragma unroll
    for (int c = 0; c < B; c++) fr[c] = free_mask ? free_mask[n * B + c] : 1;
    for (int64_t k = brow_ptr[n] + lane; k < brow_ptr[n + 1]; k += 32) {
        double v[BB];
        bool nan = false;
#pragma unroll
        for (int q = 0; q < BB; q++) {
            const int64_t i = (int64_t)q * nblocks + k;
            v[q] = __dadd_rn(__dmul_rn(a1, Ks[i]), __dmul_rn(a2, K64[i]));
            K64[i] = v[q];
            nan |= isnan(v[q]);
        }
        if (nan) set_status(status, AMR_ENAN, -1);
        finish_block<B>(n, k, bcol[k], nblocks, v, fr, free_mask, K32, Minv32, Minv64);
    }
}

// Kp = K + s1 M + s2 (alpha M + beta K): the pseudo-stiffness of the dynamic Newton loop
// (src/mech/dyn-solver.jl:366-368, s1 = 4/dt^2, s2 = 2/dt), every product and sum rounded as the
// reference's sparse operations; K absent (Ks null) gives s1 M + s2 alpha M, the mass matrix itself with
// s1 = 1, s2 = 0.  Then the masked FP32 copy and block-Jacobi inverses of the result.
template <int B>
__global__ void dyn_combine_kernel(int64_t nnodes, int64_t nblocks, const int64_t *brow_ptr, const int32_t *bcol,
                                   const double *Ks, const double *M64, double s1, double s2, double alpha,
                                   double beta, const uint8_t *free_mask, double *K64, float *K32, float *Minv32,
                                   double *Minv64, int32_t *status) {
    constexpr int BB = B * B;
    int lane = threadIdx.x & 31;
    int64_t n = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (n >= nnodes) return;
    uint8_t fr[B];
#pragma unroll
    for (int c = 0; c < B; c++) fr[c] = free_mask ? free_mask[n * B + c] : 1;
    for (int64_t k = brow_ptr[n] + lane; k < brow_ptr[n + 1]; k += 32) {
        double v[BB];
        bool nan = false;
#pragma unroll
        for (int q = 0; q < BB; q++) {
            const int64_t i = (int64_t)q * nblocks + k;
            const double kk = Ks ? Ks[i] : 0.0, mm = M64[i];
            const double c = __dadd_rn(__dmul_rn(alpha, mm), __dmul_rn(beta, kk));
            v[q] = __dadd_rn(__dadd_rn(kk, __dmul_rn(s1, mm)), __dmul_rn(s2, c));
            K64[i] = v[q];
            nan |= isnan(v[q]);
        }
        if (nan) set_status(status, AMR_ENAN, -1);
        finish_block<B>(n, k, bcol[k], nblocks, v, fr, free_mask, K32, Minv32, Minv64);
    }
}

// ---------------------------------------------------------------------------
// Element mass: elem_mass (src/mech/elem/mech-solid.jl:169-205).  EPB elements per CTA.  Phase 1,
// thread per (element, IP): coef = rho detJ w th.  Phase 2, thread per (element, node pair a <= b):
// m_ab = sum over the IPs of (coef N_a) N_b, written as the blocks m_ab I at (a,b) and (b,a) of the
// staging array (N'N has no entry between different components).
// ---------------------------------------------------------------------------
template <int DIM, int NEN>
__global__ void __launch_bounds__(256) mass_kernel(ModelArgs M, GroupArgs G, int epb, const double *rho,
                                                   double *Kel, int32_t *status) {
    constexpr int NP = NEN * (NEN + 1) / 2;
    constexpr int BB = DIM * DIM;
    extern __shared__ double sm[];
    const int nip = G.nip;
    double *sC = sm;                    // epb x NEN*DIM
    double *sK = sC + epb * NEN * DIM;  // epb x nip
    const int64_t e0 = G.first + (int64_t)blockIdx.x * epb;
    const int ne = (int)min((int64_t)epb, G.first + G.count - e0);
    const double *dNdR = G.tab;
    const double *wq = G.tab + nip * NEN * DIM;
    const double *Nt = wq + nip;
    for (int t = threadIdx.x; t < ne * NEN * DIM; t += blockDim.x) {
        int el = t / (NEN * DIM), q = t % (NEN * DIM);
        int32_t node = M.conn[M.conn_ptr[e0 + el] + q / DIM];
        sC[t] = M.coords[3 * (int64_t)node + q % DIM];
    }
    __syncthreads();
    for (int t = threadIdx.x; t < ne * nip; t += blockDim.x) {
        const int el = t / nip, ip = t % nip;
        const int64_t e = e0 + el;
        const double *C = sC + el * NEN * DIM;
        const double *D = dNdR + ip * NEN * DIM;
        double J[DIM * DIM];
#pragma unroll
        for (int i = 0; i < DIM; i++)
#pragma unroll
            for (int j = 0; j < DIM; j++) {
                double s = 0.0;
                for (int a = 0; a < NEN; a++) s += C[a * DIM + i] * D[a * DIM + j];
                J[i * DIM + j] = s;
            }
        double det;
        if (DIM == 2) det = J[0] * J[3] - J[1] * J[2];
        else det = J[0] * (J[4] * J[8] - J[5] * J[7]) - J[1] * (J[3] * J[8] - J[5] * J[6]) +
                   J[2] * (J[3] * J[7] - J[4] * J[6]);
        if (!(det > 0.0)) set_status(status, AMR_ENEGJAC, e);
        double th = M.thickness;
        if (DIM == 2 && M.stressmodel == AMR_AXISYMMETRIC) {  // th = 2 pi r (mech-solid.jl:180)
            double r = 0.0;
            for (int a = 0; a < NEN; a++) r += C[a * DIM] * Nt[ip * NEN + a];
            th = 2 * M_PI * r;
        }
        sK[el * nip + ip] = rho[e] * det * wq[ip] * th;
    }
    __syncthreads();
    for (int t = threadIdx.x; t < ne * NP; t += blockDim.x) {
        const int el = t / NP, p = t % NP;
        int a = 0, rem = p;
        while (rem >= NEN - a) { rem -= NEN - a; a++; }
        const int b = a + rem;
        double mab = 0.0;
        for (int ip = 0; ip < nip; ip++) mab = fma(sK[el * nip + ip] * Nt[ip * NEN + a], Nt[ip * NEN + b], mab);
        const int64_t base = M.kel_ptr[e0 + el];
        double *o1 = Kel + (base + (int64_t)a * NEN + b) * BB;
        double *o2 = Kel + (base + (int64_t)b * NEN + a) * BB;
#pragma unroll
        for (int q = 0; q < BB; q++) {
            const double v = (q / DIM == q % DIM) ? mab : 0.0;
            o1[q] = v;
            o2[q] = v;
        }
    }
}

// ---------------------------------------------------------------------------
// Internal forces with the constitutive update: thread per (element, IP).
// ---------------------------------------------------------------------------
template <int DIM, int NEN>
__global__ void __launch_bounds__(256, 2) internal_kernel(ModelArgs M, GroupArgs G, int epb, const double *dU,
                                                       const double *stbk, double *st, double *Fel, int32_t *status) {
    extern __shared__ double sm[];
    const int nip = G.nip;
    double *sC = sm;                          // epb x NEN*DIM
    double *sU = sC + epb * NEN * DIM;        // epb x NEN*DIM
    double *sF = sU + epb * NEN * DIM;        // epb x nip x NEN*DIM
    const int64_t e0 = G.first + (int64_t)blockIdx.x * epb;
    const int ne = (int)min((int64_t)epb, G.first + G.count - e0);
    const double *dNdR = G.tab;
    const double *wq = G.tab + nip * NEN * DIM;
    const double *Nt = wq + nip;
    const bool ps = (M.stressmodel == AMR_PLANESTRESS);
    const bool axi = DIM == 2 && M.stressmodel == AMR_AXISYMMETRIC;
    for (int t = threadIdx.x; t < ne * NEN * DIM; t += blockDim.x) {
        int el = t / (NEN * DIM), q = t % (NEN * DIM);
        int64_t node = M.conn[M.conn_ptr[e0 + el] + q / DIM];
        sC[t] = M.coords[3 * node + q % DIM];
        sU[t] = dU[node * DIM + q % DIM];
    }
    __syncthreads();
    for (int t = threadIdx.x; t < ne * nip; t += blockDim.x) {
        int el = t / nip, ip = t % nip;
        int64_t e = e0 + el;
        if (elem_skipped(M, e)) continue;
        double g[NEN * DIM];
        const double det = ip_geometry<DIM>(NEN, dNdR + ip * NEN * DIM, sC + el * NEN * DIM, g);
        const double *u = sU + el * NEN * DIM;
        double de[6] = {0, 0, 0, 0, 0, 0};
        for (int a = 0; a < NEN; a++) {
            const double *ga = g + a * DIM;
            const double *ua = u + a * DIM;
            if (DIM == 3) {
                de[0] += ga[0] * ua[0];
                de[1] += ga[1] * ua[1];
                de[2] += ga[2] * ua[2];
                de[3] += (ga[2] * ua[1] + ga[1] * ua[2]) * ISQ2;
                de[4] += (ga[2] * ua[0] + ga[0] * ua[2]) * ISQ2;
                de[5] += (ga[1] * ua[0] + ga[0] * ua[1]) * ISQ2;
            } else {
                de[0] += ga[0] * ua[0];
                de[1] += ga[1] * ua[1];
                de[5] += (ga[1] * ua[0] + ga[0] * ua[1]) * ISQ2;
            }
        }
        double th = M.thickness, rr = 1.0;
        if (axi) {  // hoop strain u_r / r and th = 2 pi r (mech-solid.jl:94-102,260)
            const double *N = Nt + ip * NEN, *C = sC + el * NEN * DIM;
            double r = 0.0;
            for (int a = 0; a < NEN; a++) r += C[a * DIM] * N[a];
            rr = r;
            th = 2 * M_PI * r;
            for (int a = 0; a < NEN; a++) de[2] += N[a] / r * u[a * DIM];
        }
        int64_t gi = M.ip_ptr[e] + ip;
        double s0[AMR_NST], s1[AMR_NST], ds[6];
        for (int f = 0; f < AMR_NST; f++) s0[f] = stbk[f * M.nip_total + gi];
        int rc = material_update(M.mat_type[e], M.mat_par + 8 * e, ps, s0, s1, de, ds);
        if (rc) {
            if (M.part_err) atomicCAS(&M.part_err[M.elem_part[e]], 0, rc);
            else set_status(status, rc, e);
            for (int f = 0; f < AMR_NST; f++) s1[f] = s0[f];
            for (int i = 0; i < 6; i++) ds[i] = 0.0;
        }
        for (int f = 0; f < AMR_NST; f++) st[f * M.nip_total + gi] = s1[f];
        const double coef = det * wq[ip] * th;
        double *fo = sF + (el * nip + ip) * NEN * DIM;
        for (int a = 0; a < NEN; a++) {
            double v[DIM];
            sym_apply<DIM>(ds, g + a * DIM, v);
            if (axi) v[0] += ds[2] * (Nt[ip * NEN + a] / rr);
#pragma unroll
            for (int c = 0; c < DIM; c++) fo[a * DIM + c] = coef * v[c];
        }
    }
    __syncthreads();
    for (int t = threadIdx.x; t < ne * NEN * DIM; t += blockDim.x) {
        int el = t / (NEN * DIM), q = t % (NEN * DIM);
        if (elem_skipped(M, e0 + el)) continue;
        double s = 0.0;
        for (int ip = 0; ip < nip; ip++) s += sF[(el * nip + ip) * NEN * DIM + q];
        Fel[M.fel_ptr[e0 + el] + q] = s;
    }
}

// The same with the 3-D geometry cache, which is read where it is used: a thread per IP for the strains and the
// constitutive update, then a thread per force component, which sums B' (coef ds) over the IPs in their order.  dN/dX held
// in registers from one to the other (60 doubles for HEX20) spilled, and the IPs' forces passed through shared memory left
// two CTAs of half-idle threads on an SM.  FP64 bounds it (82 % of the pipe), so the factors 1 / sqrt(2) and coef are taken
// once per IP, not at each node: 31 x 13 x 13 HEX20, 141 500 IPs in von Mises flow, 251 us before and 176 now.
constexpr int kIntThreads = 64;
template <int NEN>
__global__ void __launch_bounds__(kIntThreads) internal_cached_kernel(ModelArgs M, GroupArgs G, int epb, const double *dU,
                                                                      const double *stbk, double *st, double *Fel,
                                                                      int32_t *status) {
    constexpr int ND = NEN * 3;
    extern __shared__ double sm[];
    const int nip = G.nip;
    double *sU = sm;              // epb x ND
    double *sM = sU + epb * ND;   // epb x nip x 7 (6 used: no bank conflicts): coef ds, the shear terms / sqrt(2)
    const int64_t e0 = G.first + (int64_t)blockIdx.x * epb, el0 = (int64_t)blockIdx.x * epb;
    const int ne = (int)min((int64_t)epb, G.count - el0);
    for (int t = threadIdx.x; t < ne * ND; t += kIntThreads) {
        const int el = t / ND, q = t % ND;
        sU[t] = dU[(int64_t)M.conn[M.conn_ptr[e0 + el] + q / 3] * 3 + q % 3];
    }
    __syncthreads();
    for (int t = threadIdx.x; t < ne * nip; t += kIntThreads) {
        const int el = t / nip, ip = t % nip;
        const int64_t e = e0 + el;
        if (elem_skipped(M, e)) continue;
        const double *geo = G.geo_g + (el0 + el) * ND * nip + ip, *u = sU + el * ND;
        const int64_t gi = M.ip_ptr[e] + ip;
        double s0[AMR_NST], s1[AMR_NST], ds[6];
        for (int f = 0; f < AMR_NST; f++) s0[f] = stbk[f * M.nip_total + gi];
        double de[6] = {0, 0, 0, 0, 0, 0};
#pragma unroll 5
        for (int a = 0; a < NEN; a++) {
            const double ga[3] = {geo[(3 * a) * nip], geo[(3 * a + 1) * nip], geo[(3 * a + 2) * nip]};
            const double *ua = u + a * 3;
            de[0] += ga[0] * ua[0];
            de[1] += ga[1] * ua[1];
            de[2] += ga[2] * ua[2];
            de[3] = fma(ga[2], ua[1], fma(ga[1], ua[2], de[3]));
            de[4] = fma(ga[2], ua[0], fma(ga[0], ua[2], de[4]));
            de[5] = fma(ga[1], ua[0], fma(ga[0], ua[1], de[5]));
        }
        for (int i = 3; i < 6; i++) de[i] *= ISQ2;
        int rc = material_update(M.mat_type[e], M.mat_par + 8 * e, M.stressmodel == AMR_PLANESTRESS, s0, s1, de, ds);
        if (rc) {
            if (M.part_err) atomicCAS(&M.part_err[M.elem_part[e]], 0, rc);
            else set_status(status, rc, e);
            for (int f = 0; f < AMR_NST; f++) s1[f] = s0[f];
            for (int i = 0; i < 6; i++) ds[i] = 0.0;
        }
        for (int f = 0; f < AMR_NST; f++) st[f * M.nip_total + gi] = s1[f];
        const double coef = G.geo_w[(el0 + el) * nip + ip], cs = coef * ISQ2;
#pragma unroll
        for (int i = 0; i < 6; i++) sM[t * 7 + i] = (i < 3 ? coef : cs) * ds[i];
    }
    __syncthreads();
    for (int t = threadIdx.x; t < ne * ND; t += kIntThreads) {
        const int el = t / ND, q = t % ND, c = q % 3;
        if (elem_skipped(M, e0 + el)) continue;
        // row c of the symmetric tensor, as places in (11, 22, 33, 23, 13, 12)
        const int r0 = c == 0 ? 0 : c == 1 ? 5 : 4, r1 = c == 0 ? 5 : c == 1 ? 1 : 3, r2 = c == 0 ? 4 : c == 1 ? 3 : 2;
        const double *g = G.geo_g + ((el0 + el) * ND + (q - c)) * nip, *m = sM + el * nip * 7;
        double s = 0.0;
#pragma unroll 4
        for (int ip = 0; ip < nip; ip++, m += 7) {
            s = fma(m[r2], g[2 * nip + ip], fma(m[r1], g[nip + ip], fma(m[r0], g[ip], s)));
        }
        Fel[M.fel_ptr[e0 + el] + q] = s;
    }
}

// dFin[node] = sum over incident (element, local) in element order
__global__ void node_gather_kernel(int64_t nnodes, int B, const int64_t *inc_ptr, const int64_t *inc,
                                   const int64_t *conn_ptr, const int64_t *fel_ptr, const double *Fel, double *out,
                                   int accumulate, int32_t *status, const int32_t *node_part,
                                   const uint8_t *part_active, int32_t *part_err) {
    int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nnodes * B) return;
    int64_t n = t / B;
    int c = (int)(t % B);
    double s = 0.0;
    for (int64_t q = inc_ptr[n]; q < inc_ptr[n + 1]; q++) {
        int64_t e = inc[q] >> 8;
        int a = (int)(inc[q] & 0xff);
        s += Fel[fel_ptr[e] + a * B + c];
    }
    if (isnan(s)) {
        if (part_err) {
            if (part_active[node_part[n]]) atomicCAS(&part_err[node_part[n]], 0, AMR_ENAN);
        } else {
            set_status(status, AMR_ENAN, -1);
        }
    }
    out[t] = accumulate ? out[t] + s : s;
}

// ---------------------------------------------------------------------------
// Distributed loads on facets / bodies: thread per item, staging per
// (item, local node, component); gathered per node in item order.
// tab: [nq][np*fd] dN/dR, [nq] w, [nq][np] N.
// ---------------------------------------------------------------------------
__global__ void load_kernel(int kind, int dir, int edge_key, int np, int fd, int nq, const double *tab,
                            const int64_t *items, int64_t nitems, const int32_t *conn, const int64_t *conn_ptr,
                            const int64_t *inv_perm, const double *coords, int ndim, int stressmodel,
                            double thickness, const double *cf, double t, double *Fst) {
    int64_t it = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (it >= nitems) return;
    double C[AMR_MAXN * 3];
    for (int a = 0; a < np; a++) {
        int64_t node;
        if (kind == AMR_LOAD_FACET) node = items[it * np + a];
        else node = conn[conn_ptr[inv_perm[items[it]]] + a];
        for (int k = 0; k < ndim; k++) C[a * ndim + k] = coords[3 * node + k];
    }
    double F[AMR_MAXN * 3];
    for (int q = 0; q < np * ndim; q++) F[q] = 0.0;
    const double *Dt = tab, *W = tab + nq * np * fd, *Nt = W + nq;
    for (int q = 0; q < nq; q++) {
        const double *D = Dt + q * np * fd;
        const double *N = Nt + q * np;
        double J[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0}, X[3] = {0, 0, 0};
        for (int a = 0; a < np; a++) {
            for (int k = 0; k < ndim; k++) {
                X[k] += C[a * ndim + k] * N[a];
                for (int l = 0; l < fd; l++) J[k * fd + l] += C[a * ndim + k] * D[a * fd + l];
            }
        }
        double val = cf[0] + cf[1] * X[0] + cf[2] * X[1] + (ndim == 3 ? cf[3] * X[2] : 0.0) + cf[4] * t;
        double Q[3] = {0, 0, 0};
        double jn;  // norm2(J) (src/tools/linalg.jl:50-72)
        if (fd == ndim) {
            jn = (ndim == 2) ? J[0] * J[3] - J[1] * J[2]
                             : J[0] * (J[4] * J[8] - J[5] * J[7]) - J[1] * (J[3] * J[8] - J[5] * J[6]) +
                                   J[2] * (J[3] * J[7] - J[4] * J[6]);
        } else if (fd == 1) {
            double s = 0.0;
            for (int k = 0; k < ndim; k++) s += J[k] * J[k];
            jn = sqrt(s);
        } else {  // 3 x 2
            double j1 = J[0] * J[3] - J[1] * J[2], j2 = J[0] * J[5] - J[1] * J[4], j3 = J[2] * J[5] - J[3] * J[4];
            jn = sqrt(j1 * j1 + j2 * j2 + j3 * j3);
        }
        if (dir < 3) {
            Q[dir] = val;
        } else {
            double nv[3];
            if (ndim == 2) { nv[0] = J[1]; nv[1] = -J[0]; nv[2] = 0.0; }
            else {
                nv[0] = J[2] * J[5] - J[4] * J[3];
                nv[1] = J[4] * J[1] - J[0] * J[5];
                nv[2] = J[0] * J[3] - J[2] * J[1];
            }
            double ln = sqrt(nv[0] * nv[0] + nv[1] * nv[1] + nv[2] * nv[2]);
            for (int k = 0; k < ndim; k++) Q[k] = val * nv[k] / ln;
        }
        double th = (kind == AMR_LOAD_FACET && edge_key) ? 1.0 : thickness;
        if (stressmodel == AMR_AXISYMMETRIC && !(kind == AMR_LOAD_FACET && edge_key)) th = 2 * M_PI * X[0];
        double coef = jn * W[q] * th;
        for (int a = 0; a < np; a++)
            for (int k = 0; k < ndim; k++) F[a * ndim + k] += coef * N[a] * Q[k];
    }
    for (int q = 0; q < np * ndim; q++) Fst[it * np * ndim + q] = F[q];
}

__global__ void load_gather_kernel(int64_t nnodes, int B, const int64_t *ptr, const int64_t *lst, int np,
                                   const double *Fst, double *F) {
    int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nnodes * B) return;
    int64_t n = t / B;
    int c = (int)(t % B);
    if (ptr[n] == ptr[n + 1]) return;
    double s = 0.0;
    for (int64_t q = ptr[n]; q < ptr[n + 1]; q++) s += Fst[(lst[q] / np * np + lst[q] % np) * B + c];
    F[t] += s;
}

inline unsigned nblk(int64_t n, int t) { return (unsigned)((n + t - 1) / t); }

ModelArgs margs(amr_model *m) {
    ModelArgs a;
    a.coords = m->coords; a.conn = m->conn; a.conn_ptr = m->conn_ptr; a.mat_type = m->mat_type;
    a.mat_par = m->mat_par; a.ip_ptr = m->ip_ptr; a.kel_ptr = m->kel_ptr; a.fel_ptr = m->fel_ptr;
    a.nip_total = m->nip_total; a.stressmodel = m->stressmodel; a.thickness = m->thickness;
    a.elem_part = m->bp_elem_part; a.part_active = m->bp_active; a.part_err = m->bp_err;
    return a;
}

template <int DIM, int NEN>
void launch_stiff(amr_model *m, const AmrGroup &g) {
    GroupArgs ga{g.tab, g.nip, g.first, g.count, m->geo_valid ? g.geo_g : nullptr, m->geo_valid ? g.geo_w : nullptr};
    int epb = g.epb;
    // coordinates, g, plastic vectors, w, gamma w, w g; then the axisymmetric N / r (2-D) or the Jacobians and
    // plastic tangent vectors (3-D)
    size_t smem = sizeof(double) * (size_t)epb * (NEN * DIM + 3 * g.nip * NEN * DIM + 2 * g.nip +
                                                 (m->stressmodel == AMR_AXISYMMETRIC ? g.nip * NEN : 0) +
                                                 (DIM == 3 ? 15 * g.nip : 0));
    constexpr int NP = NEN * (NEN + 1) / 2;
    int threads = epb * NP;
    threads = ((threads + 31) / 32) * 32;
    if (threads > 256) threads = 256;
    if (smem > 48 * 1024) AMR_CUDA(cudaFuncSetAttribute(stiffness_kernel<DIM, NEN>,
                                                        cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    unsigned grid = nblk(g.count, epb);
    stiffness_kernel<DIM, NEN><<<grid, threads, smem, m->stream>>>(margs(m), ga, epb, m->Kel, m->st, m->d_status);
    AMR_COUNT(1);
    AMR_CUDA(cudaGetLastError());
}

// allows a kernel the most dynamic shared memory that it is launched with, once per kernel and device: a launch that set
// its own size each time would race with other handles' threads
void allow_shared(const void *kernel, size_t bytes) {
    static std::mutex mu;
    static std::set<std::pair<const void *, int>> done;
    if (bytes <= 48 * 1024) return;
    int dev = 0;
    AMR_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lk(mu);
    if (!done.insert({kernel, dev}).second) return;
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) done.erase({kernel, dev});
    AMR_CUDA(e);
}

template <int DIM, int NEN>
void launch_stiff_ref(amr_model *m, const AmrGroup &g) {
    GroupArgs ga{g.tab, g.nip, g.first, g.count};
    const size_t smem = sizeof(double) * ref_doubles<DIM, NEN>(g.nip);
    allow_shared((const void *)stiffness_ref_kernel<DIM, NEN>, sizeof(double) * ref_doubles<DIM, NEN>(AMR_MAXIP));
    stiffness_ref_kernel<DIM, NEN><<<(unsigned)g.count, 256, smem, m->stream>>>(margs(m), ga, m->Kel, m->st, m->d_status);
    AMR_COUNT(1);
    AMR_CUDA(cudaGetLastError());
}

// elements per CTA of the internal-force kernel, with the 3-D geometry cache and without, and its shared memory
int internal_epb(int nen, int nip, bool cached) {
    (void)nen;
    return cached ? std::max(1, kIntThreads / nip) : nip >= 16 ? 4 : 16;
}
size_t internal_smem(int dim, int nen, int nip, bool cached, int epb) {
    return sizeof(double) * (size_t)epb * (cached ? nen * 3 + nip * 7 : 2 * nen * dim + nip * nen * dim);
}

template <int DIM, int NEN>
void launch_internal(amr_model *m, const AmrGroup &g, const double *dU) {
    GroupArgs ga{g.tab, g.nip, g.first, g.count, m->geo_valid ? g.geo_g : nullptr, m->geo_valid ? g.geo_w : nullptr};
    if constexpr (DIM == 3)
        if (ga.geo_g) {
            const int epb = g.epb_int > 0 ? g.epb_int : internal_epb(NEN, g.nip, true);
            const size_t smem = internal_smem(3, NEN, g.nip, true, epb);
            internal_cached_kernel<NEN><<<nblk(g.count, epb), kIntThreads, smem, m->stream>>>(
                margs(m), ga, epb, dU, m->stbk, m->st, m->Fel, m->d_status);
            AMR_COUNT(1);
            AMR_CUDA(cudaGetLastError());
            return;
        }
    int epb = g.epb_int > 0 ? g.epb_int : internal_epb(NEN, g.nip, false);
    size_t smem = internal_smem(DIM, NEN, g.nip, false, epb);
    int threads = std::max(epb * g.nip, epb * NEN * DIM);
    threads = ((threads + 31) / 32) * 32;
    if (threads > 256) threads = 256;
    if (smem > 48 * 1024) AMR_CUDA(cudaFuncSetAttribute(internal_kernel<DIM, NEN>,
                                                        cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    unsigned grid = nblk(g.count, epb);
    internal_kernel<DIM, NEN><<<grid, threads, smem, m->stream>>>(margs(m), ga, epb, dU, m->stbk, m->st, m->Fel,
                                                                  m->d_status);
    AMR_COUNT(1);
    AMR_CUDA(cudaGetLastError());
}

template <typename F3, typename F2>
void dispatch(amr_model *m, const AmrGroup &g, F3 f3, F2 f2) {
    switch (g.shape) {
    case AMR_HEX8: f3(std::integral_constant<int, 8>()); break;
    case AMR_HEX20: f3(std::integral_constant<int, 20>()); break;
    case AMR_TET4: f3(std::integral_constant<int, 4>()); break;
    case AMR_TET10: f3(std::integral_constant<int, 10>()); break;
    case AMR_TRI3: f2(std::integral_constant<int, 3>()); break;
    case AMR_TRI6: f2(std::integral_constant<int, 6>()); break;
    case AMR_QUAD4: f2(std::integral_constant<int, 4>()); break;
    case AMR_QUAD8: f2(std::integral_constant<int, 8>()); break;
    case AMR_QUAD9: f2(std::integral_constant<int, 9>()); break;
    default: throw AmrError(AMR_EUNSUPPORTED, "shape not supported on the GPU path");
    }
}

}  // namespace

int amr_check_status(amr_model *m) {
    AMR_CUDA(cudaMemcpyAsync(m->h_status, m->d_status, 2 * sizeof(int32_t), cudaMemcpyDeviceToHost, m->stream));
    AMR_CUDA(cudaStreamSynchronize(m->stream));
    int code = m->h_status[0];
    if (code) {
        int32_t reset[2] = {0, INT32_MAX};
        amr_h2d(m, m->d_status, reset, sizeof reset);
    }
    return code;
}

std::vector<int> amr_internal_candidates(int dim, int nen, int nip, bool cached) {
    std::vector<int> c{internal_epb(nen, nip, cached)};
    for (int e : {1, 2, 4, 8, 16})
        if (e != c[0] && internal_smem(dim, nen, nip, cached, e) <= (cached ? 48 : 200) * 1024) c.push_back(e);
    return c;
}

int amr_test_internal_candidates(int32_t dim, int32_t nen, int32_t nip, int32_t cached, int32_t *epb, int64_t *smem) {
    const std::vector<int> c = amr_internal_candidates(dim, nen, nip, cached != 0);
    for (size_t i = 0; i < c.size(); i++) {
        epb[i] = c[i];
        smem[i] = (int64_t)internal_smem(dim, nen, nip, cached != 0, c[i]);
    }
    return (int)c.size();
}

// Builds the 3-D groups' geometry caches once per model (the coordinates never change).  If an element is
// inverted the caches are dropped and the element kernels compute the geometry themselves, reporting the
// element at each call as they did without a cache.
void amr_ensure_geometry(amr_model *m) {
    if (m->geo_valid || m->ndim != 3) return;
    if (m->geo_tried) return;
    m->geo_tried = true;
    int32_t *bad = nullptr;
    amr_alloc(&bad, 1);
    AMR_CUDA(cudaMemsetAsync(bad, 0, sizeof(int32_t), m->stream));
    for (AmrGroup &g : m->groups) {
        amr_alloc(&g.geo_g, (size_t)std::max<int64_t>(g.count, 1) * g.nip * g.nen * 3);
        amr_alloc(&g.geo_w, (size_t)std::max<int64_t>(g.count, 1) * g.nip);
        GroupArgs ga{g.tab, g.nip, g.first, g.count};
        const unsigned grid = nblk(std::max<int64_t>(g.count * g.nip, 1), 128);
        dispatch(
            m, g,
            [&](auto n) {
                geometry_kernel<decltype(n)::value><<<grid, 128, 0, m->stream>>>(margs(m), ga, g.geo_g, g.geo_w, bad);
            },
            [&](auto) {});
        AMR_COUNT(1);
    }
    AMR_CUDA(cudaGetLastError());
    int32_t hb = 0;
    AMR_CUDA(cudaMemcpyAsync(&hb, bad, sizeof(int32_t), cudaMemcpyDeviceToHost, m->stream));
    AMR_CUDA(cudaStreamSynchronize(m->stream));
    amr_free(bad);
    if (hb) {
        for (AmrGroup &g : m->groups) {
            amr_free(g.geo_g); amr_free(g.geo_w);
            g.geo_g = g.geo_w = nullptr;
        }
        return;
    }
    m->geo_valid = true;
}

void amr_stiffness_elements(amr_model *m) {
    if (m->assembly_mode != AMR_ASSEMBLY_REFERENCE) amr_ensure_geometry(m);
    for (const AmrGroup &g : m->groups) {
        if (m->assembly_mode == AMR_ASSEMBLY_REFERENCE)
            dispatch(
                m, g, [&](auto n) { launch_stiff_ref<3, decltype(n)::value>(m, g); },
                [&](auto n) { launch_stiff_ref<2, decltype(n)::value>(m, g); });
        else
            dispatch(
                m, g, [&](auto n) { launch_stiff<3, decltype(n)::value>(m, g); },
                [&](auto n) { launch_stiff<2, decltype(n)::value>(m, g); });
    }
}

void amr_stiffness(amr_model *m) {
    amr_stiffness_elements(m);
    unsigned grid = nblk(m->nblocks, 256);
    if (m->B == 3) {
        gather_kernel<3><<<grid, 256, 0, m->stream>>>(m->nblocks, m->gorder, m->grow, m->bcol, m->contrib_ptr,
                                                             m->contrib, m->Kel, m->free_mask, m->K64, m->bstride,
                                                             m->K32, m->keep, m->Minv32, m->Minv64, m->d_status);
    } else {
        gather_kernel<2><<<grid, 256, 0, m->stream>>>(m->nblocks, m->gorder, m->grow, m->bcol, m->contrib_ptr,
                                                             m->contrib, m->Kel, m->free_mask, m->K64, m->bstride,
                                                             m->K32, m->keep, m->Minv32, m->Minv64, m->d_status);
    }
    AMR_COUNT(1);
    AMR_CUDA(cudaGetLastError());
    amr_amg_invalidate(m);
}

void amr_combine_K(amr_model *m, double a1, const double *Ks, double a2) {
    unsigned grid = nblk(m->nnodes * 32, 256);
    if (m->B == 3)
        combine_kernel<3><<<grid, 256, 0, m->stream>>>(m->nnodes, m->bstride, m->brow_ptr, m->bcol, a1, Ks, a2,
                                                       m->free_mask, m->K64, m->K32, m->Minv32, m->Minv64,
                                                       m->d_status);
    else
        combine_kernel<2><<<grid, 256, 0, m->stream>>>(m->nnodes, m->bstride, m->brow_ptr, m->bcol, a1, Ks, a2,
                                                       m->free_mask, m->K64, m->K32, m->Minv32, m->Minv64,
                                                       m->d_status);
    AMR_COUNT(1);
    AMR_CUDA(cudaGetLastError());
    amr_amg_invalidate(m);
}

void amr_mass(amr_model *m) {
    if (!m->rho) throw AmrError(AMR_EINVAL, "no density set (amr_set_density)");
    if (!m->M64) {
        amr_alloc(&m->M64, (size_t)m->bstride * m->BB);
        amr_alloc(&m->Mkeep, m->nblocks);
    }
    for (const AmrGroup &g : m->groups) {
        auto launch = [&](auto dim, auto nen) {
            constexpr int DIM = decltype(dim)::value, NEN = decltype(nen)::value;
            GroupArgs ga{g.tab, g.nip, g.first, g.count};
            const int epb = 4;
            const size_t smem = sizeof(double) * (size_t)epb * (NEN * DIM + g.nip);
            mass_kernel<DIM, NEN><<<nblk(g.count, epb), 256, smem, m->stream>>>(margs(m), ga, epb, m->rho, m->Kel,
                                                                                m->d_status);
            AMR_COUNT(1);
            AMR_CUDA(cudaGetLastError());
        };
        dispatch(
            m, g, [&](auto n) { launch(std::integral_constant<int, 3>(), n); },
            [&](auto n) { launch(std::integral_constant<int, 2>(), n); });
    }
    unsigned grid = nblk(m->nblocks, 256);
    if (m->B == 3)
        gather_kernel<3><<<grid, 256, 0, m->stream>>>(m->nblocks, m->gorder, m->grow, m->bcol, m->contrib_ptr,
                                                             m->contrib, m->Kel, m->free_mask, m->M64, m->bstride,
                                                             nullptr, m->Mkeep, nullptr, nullptr, m->d_status);
    else
        gather_kernel<2><<<grid, 256, 0, m->stream>>>(m->nblocks, m->gorder, m->grow, m->bcol, m->contrib_ptr,
                                                             m->contrib, m->Kel, m->free_mask, m->M64, m->bstride,
                                                             nullptr, m->Mkeep, nullptr, nullptr, m->d_status);
    AMR_COUNT(1);
    AMR_CUDA(cudaGetLastError());
}

void amr_dyn_combine(amr_model *m, const double *Ks, double s1, double s2, double alpha, double beta) {
    m->K_valid = false;  // K64 holds a combination from here on: K is mounted again before it is read as K
    unsigned grid = nblk(m->nnodes * 32, 256);
    if (m->B == 3)
        dyn_combine_kernel<3><<<grid, 256, 0, m->stream>>>(m->nnodes, m->bstride, m->brow_ptr, m->bcol, Ks, m->M64, s1,
                                                           s2, alpha, beta, m->free_mask, m->K64, m->K32, m->Minv32,
                                                           m->Minv64, m->d_status);
    else
        dyn_combine_kernel<2><<<grid, 256, 0, m->stream>>>(m->nnodes, m->bstride, m->brow_ptr, m->bcol, Ks, m->M64, s1,
                                                           s2, alpha, beta, m->free_mask, m->K64, m->K32, m->Minv32,
                                                           m->Minv64, m->d_status);
    AMR_COUNT(1);
    AMR_CUDA(cudaGetLastError());
    amr_amg_invalidate(m);
}

void amr_update_elements(amr_model *m, const double *dU_nm, double *dFin_nm) {
    amr_ensure_geometry(m);
    for (const AmrGroup &g : m->groups) {
        dispatch(
            m, g, [&](auto n) { launch_internal<3, decltype(n)::value>(m, g, dU_nm); },
            [&](auto n) { launch_internal<2, decltype(n)::value>(m, g, dU_nm); });
    }
    int64_t nt = m->nnodes * m->B;
    node_gather_kernel<<<nblk(nt, 256), 256, 0, m->stream>>>(m->nnodes, m->B, m->inc_ptr, m->inc, m->conn_ptr,
                                                             m->fel_ptr, m->Fel, dFin_nm, 0, m->d_status,
                                                             m->bp_node_part, m->bp_active, m->bp_err);
    AMR_COUNT(1);
    AMR_CUDA(cudaGetLastError());
}

void amr_loads(amr_model *m, const amr_load *loads, int nloads, double t, double *F_nm) {
    for (int l = 0; l < nloads; l++) {
        const amr_load &L = loads[l];
        if (L.nitems <= 0) continue;
        int np, fd, shape;
        std::vector<int64_t> nodes;  // per (item, local) node ids for the incidence
        if (L.kind == AMR_LOAD_FACET) {
            shape = L.facet_shape;
            np = amr::shape_npoints(shape);
            fd = amr::shape_ndim(shape);
            if (np <= 0) throw AmrError(AMR_EINVAL, "bad facet shape");
            nodes.assign(L.items, L.items + L.nitems * np);
        } else {
            int64_t e0 = L.items[0];
            if (e0 < 0 || e0 >= m->nelems) throw AmrError(AMR_EINVAL, "bad element id in body load");
            shape = m->h_shape[m->inv_perm[e0]];
            np = amr::shape_npoints(shape);
            fd = amr::shape_ndim(shape);
            nodes.resize(L.nitems * np);
            for (int64_t i = 0; i < L.nitems; i++) {
                int64_t e = L.items[i];
                if (e < 0 || e >= m->nelems) throw AmrError(AMR_EINVAL, "bad element id in body load");
                int64_t s = m->inv_perm[e];
                if (m->h_shape[s] != shape) throw AmrError(AMR_EUNSUPPORTED, "body load over mixed shapes");
                for (int a = 0; a < np; a++) nodes[i * np + a] = m->h_conn[m->h_conn_ptr[s] + a];
            }
        }
        if (L.dir < 0 || L.dir > 3 || (L.dir == 2 && m->ndim == 2)) throw AmrError(AMR_EINVAL, "bad load direction");
        if (L.kind == AMR_LOAD_FACET && L.edge_key && m->stressmodel == AMR_AXISYMMETRIC)  // distributed.jl:89
            throw AmrError(AMR_EINVAL, "mech_boundary_forces: edge boundary conditions are not applicable in a axisymmetric analysis");
        for (int64_t v : nodes)
            if (v < 0 || v >= m->nnodes) throw AmrError(AMR_EINVAL, "bad node id in load");
        // quadrature table of the facet / element default rule
        double R[64 * 3], w[64];
        int nq = amr::quadrature(shape, 0, R, w);
        std::vector<double> tab((size_t)nq * np * fd + nq + (size_t)nq * np);
        for (int q = 0; q < nq; q++) {
            amr::shape_deriv(shape, R + 3 * q, tab.data() + (size_t)q * np * fd);
            tab[(size_t)nq * np * fd + q] = w[q];
            amr::shape_func(shape, R + 3 * q, tab.data() + (size_t)nq * np * fd + nq + (size_t)q * np);
        }
        // host incidence node -> (item*np + local), in item order (counting sort)
        std::vector<int64_t> ptr(m->nnodes + 1, 0), lst(nodes.size());
        for (int64_t v : nodes) ptr[v + 1]++;
        for (int64_t i = 0; i < m->nnodes; i++) ptr[i + 1] += ptr[i];
        {
            std::vector<int64_t> pos(ptr.begin(), ptr.end() - 1);
            for (int64_t q = 0; q < (int64_t)nodes.size(); q++) lst[pos[nodes[q]]++] = q;
        }
        double *dtab, *dcf, *Fst;
        int64_t *ditems, *dptr, *dlst;
        amr_alloc(&dtab, tab.size());
        amr_alloc(&dcf, 5);
        amr_alloc(&Fst, (size_t)L.nitems * np * m->B);
        amr_alloc(&ditems, (size_t)L.nitems * (L.kind == AMR_LOAD_FACET ? np : 1));
        amr_alloc(&dptr, ptr.size());
        amr_alloc(&dlst, lst.size());
        cudaStream_t s = m->stream;
        AMR_CUDA(cudaMemcpyAsync(dtab, tab.data(), tab.size() * sizeof(double), cudaMemcpyHostToDevice, s));
        AMR_CUDA(cudaMemcpyAsync(dcf, L.coef, 5 * sizeof(double), cudaMemcpyHostToDevice, s));
        AMR_CUDA(cudaMemcpyAsync(ditems, L.items, (size_t)L.nitems * (L.kind == AMR_LOAD_FACET ? np : 1) * sizeof(int64_t),
                                 cudaMemcpyHostToDevice, s));
        AMR_CUDA(cudaMemcpyAsync(dptr, ptr.data(), ptr.size() * sizeof(int64_t), cudaMemcpyHostToDevice, s));
        AMR_CUDA(cudaMemcpyAsync(dlst, lst.data(), lst.size() * sizeof(int64_t), cudaMemcpyHostToDevice, s));
        int64_t *dinv = nullptr;
        if (L.kind == AMR_LOAD_BODY) {
            amr_alloc(&dinv, m->nelems);
            AMR_CUDA(cudaMemcpyAsync(dinv, m->inv_perm.data(), m->nelems * sizeof(int64_t), cudaMemcpyHostToDevice, s));
        }
        load_kernel<<<nblk(L.nitems, 128), 128, 0, s>>>(L.kind, L.dir, L.edge_key, np, fd, nq, dtab, ditems, L.nitems,
                                                        m->conn, m->conn_ptr, dinv, m->coords, m->ndim,
                                                        m->stressmodel, m->thickness, dcf, t, Fst);
        AMR_COUNT(1);
        int64_t nt = m->nnodes * m->B;
        load_gather_kernel<<<nblk(nt, 256), 256, 0, s>>>(m->nnodes, m->B, dptr, dlst, np, Fst, F_nm);
        AMR_COUNT(1);
        AMR_CUDA(cudaGetLastError());
        AMR_CUDA(cudaStreamSynchronize(s));
        amr_free(dtab); amr_free(dcf); amr_free(Fst); amr_free(ditems); amr_free(dptr); amr_free(dlst);
        amr_free(dinv);
    }
}
