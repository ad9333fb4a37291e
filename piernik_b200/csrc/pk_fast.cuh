// pk_fast.cuh -- the tolerance-mode arithmetic of the split sweep.
//
// The same algorithms as pk_device.cuh's utoq, riemann_hlld and
// riemann_hlld_u (interpolations.F90:69-106, hlld.F90:161-841) with the same
// branch structure, but rounding is not the reference's: the kernels that use
// these functions are compiled with multiply-add contraction (--fmad=true), and
// the solvers take the Fast arithmetic below: divisions by a common denominator
// become one reciprocal and products (1/rho in utoq; 1/(gamma-1) and 1/gamma
// from PhysParams, 1/ch from StepParams; 1/slsm, 1/srsm and 1/(add_dnsq) in the
// Riemann solver; the two Alfven divisions by sqrt(rho*) through the reciprocal
// square root), and the remaining quotients and reciprocals are the branch-free
// refinements below (rcp_nr, div_nr, rsqrt_nr).  Each replaced operation
// changes a result by a few units in the last place, so a time step agrees
// with the bit-exact path to ~1e-15 relative; the tests hold it to 1e-12 per
// step and 1e-9 after 100 steps.
#pragma once
#include <type_traits>

#include "pk_device.cuh"
#include "pk_quotient.cuh"

namespace pk {

// Reciprocal, quotient and reciprocal square root without the IEEE
// sequences' special-case branches: the hardware's approximate FP64
// reciprocal and reciprocal square root (PTX rcp.approx.ftz.f64,
// rsqrt.approx.ftz.f64, about 20 correct bits) refined by Newton-Raphson
// iterations (r' = r + r(1 - x r) and y' = y(3/2 - x y^2/2): each doubles the
// correct bits, two reach the double precision), the quotient finished with
// one residual correction (Markstein, IBM J. Res. Dev. 34 (1990) 111-119).
// Results are within about an ulp of the correctly rounded ones for normal
// finite operands, which is all the tolerance arithmetic asks; subnormal
// operands are flushed to zero by the seeds and are not expected in the
// states.  Square roots keep the IEEE operation: a Newton-refined root
// (tried) moved a three-fluid blast beyond the 1e-12 per-step bound.
PK_DEV double rcp_nr(double x)
{
    double r = rcp_seed(x);
    double e = fma(-x, r, 1.0);
    r = fma(r, e, r);
    e = fma(-x, r, 1.0);
    return fma(r, e, r);
}

PK_DEV double div_nr(double a, double b)
{
    const double r = rcp_nr(b);
    const double q = a * r;
    return fma(r, fma(-b, q, a), q);
}

PK_DEV double rsqrt_nr(double x)
{
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double hx = 0.5 * x;
    y = y * fma(-hx * y, y, 1.5);
    return y * fma(-hx * y, y, 1.5);
}


template <class PH>
PK_DEV void utoq_fast(const double (&u)[PH::NV], double (&q)[PH::NV], const PhysParams& pp)
{
#pragma unroll
    for (int f = 0; f < PH::NFL; ++f) {
        const int b = PH::beg(f);
        const double dn = u[b], mx = u[b + 1], my = u[b + 2], mz = u[b + 3];
        const double rdn = rcp_nr(dn);
        q[b] = dn;
        q[b + 1] = mx * rdn;
        q[b + 2] = my * rdn;
        q[b + 3] = mz * rdn;
        if (PH::has_en(f)) {
            const double ek = (0.5 * ((mx * mx + my * my) + mz * mz)) * rdn;
            double p = pp.gam_1[f] * (u[b + 4] - ek);
            if (PH::magn(f)) {
                const double bx = u[PH::IB], by = u[PH::IB + 1], bz = u[PH::IB + 2];
                p = p - (0.5 * pp.gam_1[f]) * ((bx * bx + by * by) + bz * bz);
            }
            q[b + 4] = p;
        }
    }
    if (PH::MHD) {
#pragma unroll
        for (int c = 0; c < 4; ++c) q[PH::IB + c] = u[PH::IB + c];
    }
}

// The solvers' tolerance-mode arithmetic (hlld_face, hllc_face): quotients by a
// shared denominator are products with its reciprocal, n / sqrt(x) is a product
// with the reciprocal square root, sqrt(x) = x * rsqrt(x).
struct Fast {
    static constexpr bool FAST = true;
    PK_DEV double div(double n, double d) { return div_nr(n, d); }
    PK_DEV double inv(double d) { return rcp_nr(d); }
    PK_DEV double quo(double n, double, double r) { return n * r; }
    PK_DEV double quoz(double n, double, double r) { return n * r; }
    PK_DEV double root(double x, double& y)
    {
        y = rsqrt_nr(x);
        return x * y;
    }
    PK_DEV double over_root(double n, double, double y) { return n * y; }
    template <int G>
    PK_DEV void settle(const double (&)[G], const double (&)[G], double (&)[G]) const
    {
    }
    PK_DEV bool ok() const { return true; }
};

// riemann_wrap / riemann_wrap_u (hlld.F90:62-155) for the right face of one
// cell of a tile in shared memory (planes of S doubles): its left state in q
// (KEEP) or at F[v * S], the right state at R[v * S].  The fluxes go to F[v * S]
// and, with KEEP, to q.  Each fluid's states are loaded just before its solve.
// rch: the correctly rounded 1/ch.  FAST: the tolerance-mode arithmetic; the
// GLM flux of psi multiplies by 1/ch instead of dividing.
template <class PH, int S, bool KEEP, bool FAST>
PK_DEV void riemann_cell(double (&q)[PH::NV], const double* R, double* F, double ch, double rch,
                         const PhysParams& pp)
{
    using Ar = std::conditional_t<FAST, Fast, Exact>;
    auto left = [&](int v) { return KEEP ? q[v] : F[v * S]; };
    auto put = [&](int v, double f) {
        F[v * S] = f;
        if (KEEP) q[v] = f;
    };
    double blv[3] = {0.0, 0.0, 0.0}, brv[3] = {0.0, 0.0, 0.0};
    if constexpr (PH::MHD) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            blv[c] = left(PH::IB + c);
            brv[c] = R[(PH::IB + c) * S];
        }
        const double bxl = blv[0], bxr = brv[0];
        const double psl = left(PH::IB + 3), psr = R[(PH::IB + 3) * S];
        double dps;
        if constexpr (FAST) {
            dps = (psr - psl) * rch;
        } else {
            Exact ar;
            ar.needd(ch);
            dps = ar.quoa(psr - psl, ch, rch, bxr + bxl);
            if (!ar.ok()) dps = divide_ieee(psr - psl, ch);
        }
        put(PH::IB + 3, ((ch * ch) * 0.5) * ((bxr + bxl) - dps));                // hlld.F90:229 (Dedner eq. 42)
        put(PH::IB, 0.5 * ((psr + psl) - ch * (bxr - bxl)));                     // :230
    }
#pragma unroll
    for (int f = 0; f < PH::NFL; ++f) {
        const int b = PH::beg(f);
        const int nc = PH::ncomp(PH::kind(f));
        double ul[5] = {0, 0, 0, 0, 0}, ur[5] = {0, 0, 0, 0, 0}, fv[5];
#pragma unroll
        for (int c = 0; c < 5; ++c)
            if (c < nc) {
                ul[c] = left(b + c);
                ur[c] = R[(b + c) * S];
            }
        Ar ar;
        if (PH::MHD) {
            double bL[3] = {0.0, 0.0, 0.0}, bR[3] = {0.0, 0.0, 0.0}, bf[2];
            if (PH::magn(f)) {
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    bL[c] = blv[c];
                    bR[c] = brv[c];
                }
            }
            hlld_face(ar, PH::has_en(f), pp.gam[f], pp.rgam_1[f], pp.rgam[f], ul, ur, bL, bR, fv, bf);
            if constexpr (!FAST)
                if (!ar.ok()) {
                    double x[16], o[7];
#pragma unroll
                    for (int c = 0; c < 5; ++c) {
                        x[c] = ul[c];
                        x[5 + c] = ur[c];
                        if (c < 3) {
                            x[10 + c] = bL[c];
                            x[13 + c] = bR[c];
                        }
                    }
                    hlld_ieee(PH::has_en(f), pp.gam[f], x, o);
#pragma unroll
                    for (int c = 0; c < 5; ++c) fv[c] = o[c];
                    bf[0] = o[5];
                    bf[1] = o[6];
                }
            if (PH::magn(f)) {
                put(PH::IB + 1, bf[0]);
                put(PH::IB + 2, bf[1]);
            }
        } else {
            hllc_face(ar, PH::has_en(f), pp.gam[f], pp.rgam_1[f], ul, ur, fv);
            if constexpr (!FAST)
                if (!ar.ok()) {
                    double x[10], o[5];
#pragma unroll
                    for (int c = 0; c < 5; ++c) {
                        x[c] = ul[c];
                        x[5 + c] = ur[c];
                    }
                    hllc_ieee(PH::has_en(f), pp.gam[f], x, o);
#pragma unroll
                    for (int c = 0; c < 5; ++c) fv[c] = o[c];
                }
        }
#pragma unroll
        for (int c = 0; c < 5; ++c)
            if (c < nc) put(b + c, fv[c]);
    }
}

}  // namespace pk
