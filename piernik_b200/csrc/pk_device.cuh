// pk_device.cuh -- per-cell and per-interface FP64 physics of the split sweep.
//
// Device restatement of PIERNIK's RIEMANN_SPLIT building blocks.  Every
// expression keeps the reference's evaluation order so that, compiled with
// --fmad=false (no contraction) and IEEE double division/sqrt, results are
// bit-identical to the Fortran (gfortran -O2, SSE2, no FMA) arithmetic:
//   utoq                 src/scheme/Riemann_Solver/interpolations.F90:69-106
//   limiters             src/scheme/Riemann_Solver/fluxlimiters.F90:109-216
//   linear               src/scheme/Riemann_Solver/interpolations.F90:170-204
//   riemann_hlld (+GLM)  src/scheme/Riemann_Solver/hlld.F90:161-609
//   riemann_hlld_u       src/scheme/Riemann_Solver/hlld.F90:615-841
//   internal_sources     src/fluids/sources.F90:151-244 (adds +0: -0.0 -> +0.0)
//   care_for_positives   src/fluids/sources.F90:299-433
//   ion_cs/neu_cs        src/fluids/ionized/initionized.F90:89-145,
//                        src/fluids/neutral/initneutral.F90:82-109
//
// A cell state is a register array in *swept* order: for each fluid
// [dn, m_n, m_t1, m_t2, (en)], then [B_n, B_t1, B_t2, psi] when magnetised,
// where (n, t1, t2) = (x,y,z), (y,x,z), (z,y,x) for sweeps along x, y, z
// (iarr_all_swp, fluids/fluidtypes.F90:318-320; iarr_mag_swp,
// fluids/fluidindex.F90:190-192).
#pragma once
#include <cmath>
#include <cstdint>
#include <cstring>

#define PK_DEV __device__ __forceinline__
#define PK_HD __host__ __device__ __forceinline__
// physics functions compile for the host too (unit tests of the adjoints)
#define PK_PHYS __host__ __device__ __forceinline__

namespace pk {

enum FluidKind { K_ION = 0, K_NEU = 1, K_DST = 2, K_NONE = 3 };
enum Limiter { L_VANLEER = 0, L_MINMOD = 1, L_MONCEN = 2, L_SUPERBEE = 3 };

// -------------------------------------------------------------------------
// Fortran intrinsics
// -------------------------------------------------------------------------

// SPACING(x) for real(8): 2**max(exponent(x)-53, -1022), TINY(x) at zero.
PK_PHYS unsigned long long f_bits(double x)
{
#ifdef __CUDA_ARCH__
    return (unsigned long long)__double_as_longlong(x);
#else
    unsigned long long b;
    memcpy(&b, &x, sizeof b);
    return b;
#endif
}
PK_PHYS double f_from_bits(unsigned long long b)
{
#ifdef __CUDA_ARCH__
    return __longlong_as_double((long long)b);
#else
    double x;
    memcpy(&x, &b, sizeof x);
    return x;
#endif
}
PK_PHYS double f_spacing(double x)
{
    const unsigned long long bits = f_bits(x);
    const int be = (int)((bits >> 52) & 0x7ffu);
    if (be == 0x7ff) return f_from_bits(0x7ff8000000000000ULL);
    if (be >= 53) return f_from_bits((unsigned long long)(be - 52) << 52);
    return 2.2250738585072014e-308;
}
PK_PHYS double f_sign1(double x) { return copysign(1.0, x); }
PK_PHYS double f_min(double a, double b) { return (b < a) ? b : a; }
PK_PHYS double f_max(double a, double b) { return (b > a) ? b : a; }

// -------------------------------------------------------------------------
// Compile-time description of the fluid set (flind order: ion, neu, dst)
// -------------------------------------------------------------------------

template <int K0, int K1, int K2, bool MAG>
struct Phys {
    PK_HD static constexpr int kind(int f) { return f == 0 ? K0 : (f == 1 ? K1 : K2); }
    static constexpr int NFL = (K0 != K_NONE) + (K1 != K_NONE) + (K2 != K_NONE);
    static constexpr bool MHD = MAG;
    PK_HD static constexpr int ncomp(int k) { return k == K_NONE ? 0 : (k == K_DST ? 4 : 5); }
    PK_HD static constexpr int beg(int f) { return f == 0 ? 0 : (f == 1 ? ncomp(K0) : ncomp(K0) + ncomp(K1)); }
    static constexpr int NVF = ncomp(K0) + ncomp(K1) + ncomp(K2);   // fluid components
    static constexpr int IB = NVF;                                 // first B component
    static constexpr int NV = NVF + (MAG ? 4 : 0);                 // with Bx,By,Bz,psi
    PK_HD static constexpr bool has_en(int f) { return kind(f) != K_DST; }
    PK_HD static constexpr bool magn(int f) { return MAG && kind(f) == K_ION; }
};

struct PhysParams {
    double gam[3];      // adiabatic index per fluid (dust: -1)
    double gam_1[3];    // gam - 1
    double rgam_1[3];   // 1 / (gam - 1), 1 / gam: the tolerance-mode kernels multiply by these
    double rgam[3];
    double smalld, smallei;
    int use_smalld, use_smallei, disallow_negatives;
    int lim, limb;      // flimiter, blimiter
    int weno3;          // interpol_str = 'weno3': WENO3 face states instead of limited linear ones
    double w_epsilon;   // WENO3 weight regulariser (global.F90:255)
};

// status bits written by kernels (never traps)
enum StatusBits : unsigned {
    ST_DN_NEGATIVE = 1u,   // dn_negative (sources.F90:349-350)
    ST_EI_NEGATIVE = 2u,   // ei_negative (sources.F90:422)
};

// The arithmetic of utoq and of the Riemann solves, passed as a policy (Ieee
// here; Exact, the kernels', in pk_quotient.cuh; Fast, the tolerance mode's, in
// pk_fast.cuh).  inv(d) is taken once per denominator and used by every
// quo(n, d, inv(d)); quoz is quo for numerators that are often exactly zero or
// fade towards it; quoa is quoz for a quotient that only enters sums with big,
// quob for one that is only compared with a and b; quoc divides by a constant d
// whose correctly rounded reciprocal y is known; root(x, aux) is sqrt(x), and
// over_root(n, root, aux) is n / that root.  settle ends a group of quotients taken
// with an A of its own.  ok() tells whether all quotients taken so far are the
// correctly rounded ones.
struct Ieee {
    static constexpr bool FAST = false;
    PK_PHYS double inv(double) { return 0.0; }
    PK_PHYS double quo(double n, double d, double) { return n / d; }
    PK_PHYS double quoz(double n, double d, double) { return n / d; }
    PK_PHYS double quoa(double n, double d, double, double) { return n / d; }
    PK_PHYS double quob(double n, double d, double, double, double) { return n / d; }
    PK_PHYS double quoc(double n, double d, double) { return n / d; }
    template <int G>
    PK_PHYS void settle(const double (&)[G], const double (&)[G], double (&)[G])
    {
    }
    PK_PHYS double root(double x, double&) { return sqrt(x); }
    PK_PHYS double over_root(double n, double root, double) { return n / root; }
    PK_PHYS bool ok() const { return true; }
};

// -------------------------------------------------------------------------
// utoq: conservative -> primitive, one cell (interpolations.F90:69-106)
// -------------------------------------------------------------------------
template <class PH, class A>
PK_PHYS void utoq(A& ar, const double (&u)[PH::NV], double (&q)[PH::NV], const PhysParams& pp)
{
#pragma unroll
    for (int f = 0; f < PH::NFL; ++f) {
        const int b = PH::beg(f);
        const double dn = u[b], mx = u[b + 1], my = u[b + 2], mz = u[b + 3], r = ar.inv(dn);
        const double n[4] = {mx, my, mz, PH::has_en(f) ? 0.5 * ((mx * mx + my * my) + mz * mz) : 0.0};
        const double d[4] = {dn, dn, dn, dn};
        double x[4] = {ar.quoz(mx, dn, r), ar.quoz(my, dn, r), ar.quoz(mz, dn, r), 0.0};
        if (PH::has_en(f)) x[3] = ar.quoa(n[3], dn, r, u[b + 4]);
        ar.settle(n, d, x);
        q[b] = dn;
        q[b + 1] = x[0];
        q[b + 2] = x[1];
        q[b + 3] = x[2];
        if (PH::has_en(f)) {
            const double ek = x[3];
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
        for (int c = 0; c < 4; ++c) q[PH::IB + c] = u[PH::IB + c];   // B and psi go to blimiter as they are
    }
}

template <class PH>
PK_PHYS void utoq(const double (&u)[PH::NV], double (&q)[PH::NV], const PhysParams& pp)
{
    Ieee ar;
    utoq<PH>(ar, u, q, pp);
}

// -------------------------------------------------------------------------
// Limited slopes.  Interior cell: dl = q(i)-q(i-1), dr = q(i+1)-q(i).
// Pencil end cells use the reference's one-sided rules (dl = dr, vanleer 0).
// -------------------------------------------------------------------------
PK_PHYS double slope_interior(int lim, double dl, double dr)
{
    if (lim == L_VANLEER) {                       // fluxlimiters.F90:122-133
        const double dcen = dl * dr;
        return (dcen > 0.0) ? (2.0 * dcen) / (dl + dr) : 0.0;
    }
    const double s = f_sign1(dl) + f_sign1(dr);
    if (lim == L_MINMOD) return (s * f_min(fabs(dl), fabs(dr))) * 0.5;                        // :158
    if (lim == L_MONCEN) return (s * f_min(f_min(2.0 * fabs(dl), 2.0 * fabs(dr)), 0.5 * fabs(dl + dr))) * 0.5;  // :185
    const double m = (fabs(dl) > fabs(dr)) ? f_min(fabs(dl), fabs(2.0 * dr)) : f_min(fabs(2.0 * dl), fabs(dr)); // :211-212
    return (s * 0.5) * m;
}

// half * f_limiter(q) of an interior cell for a limiter known at compile time
// (dq_interp = half * f_limiter(q), interpolations.F90:170-204; van Leer's is
// vanleer_half in pk_quotient.cuh).  Bit for bit
// 0.5 * slope_interior(LIM, dl, dr): the signs s of minmod, moncen and superbee
// are -2, 0 or 2, so ((s * m) * 0.5) * 0.5 rounds once, as (s / 4) * m does (for
// differences below 2^1022 and infinite ones; s = 0 keeps the +0, and the NaN of 0 * inf),
// and min(2a, 2b) = 2 min(a, b) exactly.
template <int LIM>
PK_PHYS double half_slope(double dl, double dr)
{
    static_assert(LIM != L_VANLEER, "van Leer's half slopes are taken in groups");
    const double adl = fabs(dl), adr = fabs(dr);
    double m;
    if (LIM == L_MINMOD) m = f_min(adl, adr);
    else if (LIM == L_MONCEN) m = f_min(2.0 * f_min(adl, adr), 0.5 * fabs(dl + dr));
    else m = (adl > adr) ? f_min(adl, 2.0 * adr) : f_min(2.0 * adl, adr);
    const unsigned long long bl = f_bits(dl), br = f_bits(dr);
    const double s = f_from_bits(((long long)(bl ^ br) < 0) ? 0ULL
                                                            : ((bl & 0x8000000000000000ULL) | 0x3fe0000000000000ULL));
    return s * m;
}

// WENO3 face states of cell c from q(c-1), q(c), q(c+1) (interpolations.F90:
// 210-337, Yamaleev & Carpenter 2009): ql = the left state of the right face,
// qr = the right state of the left face, in the reference's operation order.
// Six quotients a component by four denominators (tau / (weps + b) serves both
// faces): an arithmetic A of the policies above.
template <class A>
PK_PHYS void weno3_faces(A& ar, double qm, double qc, double qp, double weps, double& ql, double& qr)
{
    const double d0 = 2.0 / 3.0, d1 = 1.0 / 3.0;                              // Eq. 19 (twot, onet)
    const double b0 = (qp - qc) * (qp - qc);                                    // Eq. 20
    const double b1 = (qc - qm) * (qc - qm);
    const double tt = ((qp - 2.0 * qc) + qm);                                   // Eq. 22
    const double tau = tt * tt;
    const double e0 = weps + b0, e1 = weps + b1;
    const double t0 = ar.quoa(tau, e0, ar.inv(e0), 1.0), t1 = ar.quoa(tau, e1, ar.inv(e1), 1.0);
    double a0 = d0 * (1.0 + t0);                                                // Eq. 21
    double a1 = d1 * (1.0 + t1);
    double s = a0 + a1, r = ar.inv(s);
    double w0 = ar.quo(a0, s, r), w1 = ar.quo(a1, s, r);                        // Eq. 18
    double f0 = 0.5 * (qc + qp), f1 = 0.5 * (-qm + 3.0 * qc);                   // Eq. 15
    ql = w0 * f0 + w1 * f1;                                                     // Eq. 14
    a0 = d0 * (1.0 + t1);                                                       // the mirrored stencil
    a1 = d1 * (1.0 + t0);
    s = a0 + a1;
    r = ar.inv(s);
    w0 = ar.quo(a0, s, r);
    w1 = ar.quo(a1, s, r);
    f0 = 0.5 * (qc + qm);
    f1 = 0.5 * (-qp + 3.0 * qc);
    qr = w0 * f0 + w1 * f1;
}

// -------------------------------------------------------------------------
// Riemann solvers on one interface.  ql/qr: primitive swept states of one
// fluid; bl/br: swept B (zero for unmagnetised fluids); f: fluid fluxes;
// bf: transverse B fluxes.
// -------------------------------------------------------------------------

// transverse B flux of one side (b_cclf(ydim:zdim), hlld.F90:301,309)
PK_PHYS double side_bflux(const double* u, const double* b, int c)
{
    return (b[c] * u[1]) - (b[0] * u[1 + c]);
}

// HLLD flux of one interface (riemann_hlld, hlld.F90:161-609).  Everything up to
// the Alfven speeds is computed for both sides, whose chains of dependent
// quotients and roots overlap; then the side that the flux is taken from (both
// where sm = 0) is picked by selects, and its energy, its star energy and its
// flux are computed for that side only.
template <class A>
PK_PHYS void hlld_face(A& ar, bool has_energy, double gamma, double rgam_1, double rgam, const double (&ul)[5],
                       const double (&ur)[5], const double (&bl)[3], const double (&br)[3], double (&f)[5],
                       double (&bf)[2])
{
    const bool dust = gamma < 0.0;
    const double bbl = (bl[0] * bl[0] + bl[1] * bl[1]) + bl[2] * bl[2];
    const double bbr = (br[0] * br[0] + br[1] * br[1]) + br[2] * br[2];
    double prl = 0.0, prr = 0.0, c_fastm = 0.0;                                      // hlld.F90:245-249
    if (!dust) {
        prl = ul[4] + 0.5 * bbl;                                                      // :239-240, 258-259
        prr = ur[4] + 0.5 * bbr;
        const double gampr_l = gamma * ul[4];
        const double gampr_r = gamma * ur[4];
        const double al = gampr_l + bbl, ar_ = gampr_r + bbr;                        // :272-274
        const double nl = al + sqrt(al * al - ((4.0 * gampr_l) * (bl[0] * bl[0])));
        const double nr = ar_ + sqrt(ar_ * ar_ - ((4.0 * gampr_r) * (br[0] * br[0])));
        double cmax;
        if constexpr (A::FAST) {               // max(nl/rho_l, nr/rho_r) with one quotient (densities are positive)
            const bool lm = nl * ur[0] >= nr * ul[0];
            cmax = ar.div(lm ? nl : nr, lm ? ul[0] : ur[0]);
        } else {
            cmax = f_max(ar.quo(nl, ul[0], ar.inv(ul[0])), ar.quo(nr, ur[0], ar.inv(ur[0])));
        }
        c_fastm = sqrt(0.5 * cmax);
    }
    const double sl = f_min(ul[1], ur[1]) - c_fastm;                                // :291-292
    const double sr = f_max(ul[1], ur[1]) + c_fastm;

    // the flux of the picked side, from its energy on: fs alone (FAN 0, :312-319),
    // fs + s (u* - u) (FAN 1, Eq. 64), or ((fs + a u**) - (a - s) u*) - s u (FAN 2,
    // Eq. 65); add: the second of two sides whose mean is the flux
    double sm = 0.0, prt_star = 0.0, us0 = 0.0, vs[2] = {0.0, 0.0}, bs[2] = {0.0, 0.0}, a = 0.0, root = 0.0;
    double v2[2] = {0.0, 0.0}, b2[2] = {0.0, 0.0}, b2n = 0.0, rssm = 0.0;
    auto side = [&](bool left, int fan, bool add) {
        double u[5], b[3];
#pragma unroll
        for (int c = 0; c < 5; ++c) u[c] = left ? ul[c] : ur[c];
#pragma unroll
        for (int c = 0; c < 3; ++c) b[c] = left ? bl[c] : br[c];
        const double s = left ? sl : sr, pr = left ? prl : prr;
        double en = 1.7976931348623157e308;
        if (!dust) {                                                                 // :260-269
            double ei;
            if constexpr (A::FAST) ei = u[4] * rgam_1;
            else ei = ar.quoc(u[4], gamma - 1.0, rgam_1);
            en = (ei + ((0.5 * u[0]) * ((u[1] * u[1] + u[2] * u[2]) + u[3] * u[3]))) + (0.5 * (left ? bbl : bbr));
        }
        const double vb = (u[1] * b[0] + u[2] * b[1]) + u[3] * b[2];
        double us4 = 0.0, u24 = 0.0;
        if (fan && has_energy) {                                                     // :388-404
            const double vb_star = (sm * b[0] + vs[0] * bs[0]) + vs[1] * bs[1];
            us4 = ar.quo(((((s - u[1]) * en) - (pr * u[1])) + (prt_star * sm)) + (b[0] * (vb - vb_star)), s - sm, rssm);
            if (fan == 2) {                                                          // :474-489
                const double vb_2star = (sm * b2n + v2[0] * b2[0]) + v2[1] * b2[1];
                const double t = (((bl[0] >= 0.0) ? 1.0 : -1.0) * root) * (vb_star - vb_2star);
                u24 = left ? us4 - t : us4 + t;
            }
        }
        // side_flux (:296-309), the conserved state, u* and u**
        const double uc[7] = {u[0], u[0] * u[1], u[0] * u[2], u[0] * u[3], en, b[1], b[2]};
        const double fs[7] = {uc[1], ((u[0] * (u[1] * u[1])) + pr) - (b[0] * b[0]), (uc[2] * u[1]) - (b[0] * b[1]),
                              (uc[3] * u[1]) - (b[0] * b[2]), ((en + pr) * u[1]) - (b[0] * vb),
                              (b[1] * u[1]) - (b[0] * u[2]), (b[2] * u[1]) - (b[0] * u[3])};
        const double us[7] = {us0, us0 * sm, us0 * vs[0], us0 * vs[1], us4, bs[0], bs[1]};
        const double u2[7] = {us0, us0 * sm, us0 * v2[0], us0 * v2[1], u24, b2[0], b2[1]};
        const double ams = a - s;
#pragma unroll
        for (int c = 0; c < 7; ++c) {
            double o = fs[c];
            const double p = c < 5 ? f[c] : bf[c - 5];
            if (fan == 2) {
                o = ((fs[c] + a * u2[c]) - ams * us[c]) - s * uc[c];
                if (add) o = 0.5 * (p + o);                                          // :524-544
            } else if (fan == 1) {
                const double d = s * (us[c] - uc[c]);
                o = add ? 0.5 * ((p + fs[c]) + d) : fs[c] + d;                       // :583-599, summed left to right
            }
            if (c < 5) f[c] = o;
            else bf[c - 5] = o;
        }
    };

    if (sl >= 0.0 || sr <= 0.0) {                                                    // :312-319
        side(sl >= 0.0, 0, false);
        return;
    }
    const double slvxl = sl - ul[1], srvxr = sr - ur[1];                            // :323-330, 344-347
    const double dn_l = ul[0] * slvxl, dn_r = ur[0] * srvxr;
    {
        const double n = (dn_r * ur[1] - prr) - (dn_l * ul[1] - prl), d = dn_r - dn_l;
        if (fabs(d) < f_spacing(dn_r + dn_l)) {
            sm = (sl + sr) * 0.5;
        } else {
            if constexpr (A::FAST) sm = ar.div(n, d);
            else {
                A g;
                const double gn[1] = {n}, gd[1] = {d};
                double x[1] = {g.quoz(n, d, g.inv(d))};
                g.settle(gn, gd, x);
                sm = x[0];
            }
        }
    }
    const double slsm = sl - sm, srsm = sr - sm;                                    // :334-340
    const double b_lr = bl[0] * br[0];
    double b_lrgam;
    if constexpr (A::FAST) b_lrgam = b_lr * rgam;
    else b_lrgam = ar.quob(b_lr, gamma, rgam, ul[4], ur[4]);
    prt_star = 0.5 * ((prl + dn_l * (sm - ul[1])) + (prr + dn_r * (sm - ur[1])));
    // rho*, transverse B* (HLL fallback) and v* of both sides (:354-355, :362-382)
    const double rslsm = ar.inv(slsm), rsrsm = ar.inv(srsm);
    const double usl0 = ar.quo(dn_l, slsm, rslsm), usr0 = ar.quo(dn_r, srsm, rsrsm);
    double bsl[2], bsr[2], vsl[2], vsr[2];
    {
        const double cl = dn_l * slsm - b_lr, cr = dn_r * srsm - b_lr;
        const bool star_l = (fabs(cl) > f_spacing(b_lr)) && b_lrgam <= (has_energy ? ul[4] : 0.0);
        const bool star_r = (fabs(cr) > f_spacing(b_lr)) && b_lrgam <= (has_energy ? ur[4] : 0.0);
        const double tl = dn_l * slvxl - b_lr, tr = dn_r * srvxr - b_lr;
        double kl = 0.0, kr = 0.0;
        if constexpr (A::FAST) {
            const double ql = ar.div(tl, cl), qr = ar.div(tr, cr);
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                bsl[c] = bl[1 + c] * ql;
                bsr[c] = br[1 + c] * qr;
            }
        } else {
            A g;
            const double dl = star_l ? cl : 1.0, dr = star_r ? cr : 1.0;
            const double rl = g.inv(dl), rr = g.inv(dr);
            const double n[6] = {bl[1] * tl, bl[2] * tl, br[1] * tr, br[2] * tr, bl[0], br[0]};
            const double d[6] = {dl, dl, dr, dr, dn_l, dn_r};
            double x[6] = {g.quoz(n[0], dl, rl), g.quoz(n[1], dl, rl), g.quoz(n[2], dr, rr), g.quoz(n[3], dr, rr),
                           g.quoz(n[4], dn_l, g.inv(dn_l)), g.quoz(n[5], dn_r, g.inv(dn_r))};
            g.settle(n, d, x);
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                bsl[c] = x[c];
                bsr[c] = x[2 + c];
            }
            kl = x[4];
            kr = x[5];
        }
        if (!(star_l && star_r)) {
            const double d = sr - sl, r = ar.inv(d);
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const double h = ar.quoz((sr * br[1 + c] - sl * bl[1 + c]) - (side_bflux(ur, br, 1 + c) - side_bflux(ul, bl, 1 + c)), d, r);
                if (!star_l) bsl[c] = h;
                if (!star_r) bsr[c] = h;
            }
        }
        if constexpr (A::FAST) {
            kl = ar.div(bl[0], dn_l);
            kr = ar.div(br[0], dn_r);
        }
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            vsl[c] = ul[2 + c] + (kl * (bl[1 + c] - bsl[c]));
            vsr[c] = ur[2 + c] + (kr * (br[1 + c] - bsr[c]));
        }
    }
    bool left = sm > 0.0, both = !left && !(sm < 0.0), alfven = false;
    double rtl = 0.0, rtr = 0.0, alfven_l = 0.0, alfven_r = 0.0;
    if (fabs(bl[0]) > 0.0) {                                                         // :410-448
        double xl = 0.0, xr = 0.0;
        rtl = ar.root(usl0, xl);
        rtr = ar.root(usr0, xr);
        {
            A g;
            const double n[2] = {fabs(bl[0]), fabs(br[0])}, d[2] = {rtl, rtr};
            double x[2] = {g.over_root(n[0], rtl, xl), g.over_root(n[1], rtr, xr)};
            g.settle(n, d, x);
            alfven_l = sm - x[0];
            alfven_r = sm + x[1];
        }
        alfven = !(alfven_l > 0.0 || alfven_r < 0.0);
        if (!alfven) {
            left = alfven_l > 0.0;
            both = false;
        } else {                                                                     // :452-470
            const double b_sig = (bl[0] >= 0.0) ? 1.0 : -1.0;
            A g;
            const double d = rtl + rtr, r = g.inv(d), bsm = b_sig * (rtl * rtr);
            b2n = 0.5 * (bl[0] + br[0]);
            double n[4], x[4];
            const double ds[4] = {d, d, d, d};
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                n[c] = (rtl * vsl[c] + rtr * vsr[c]) + b_sig * (bsr[c] - bsl[c]);
                n[2 + c] = (rtl * bsr[c] + rtr * bsl[c]) + bsm * (vsr[c] - vsl[c]);
                x[c] = g.quoz(n[c], d, r);
                x[2 + c] = g.quoz(n[2 + c], d, r);
            }
            g.settle(n, ds, x);
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                v2[c] = x[c];
                b2[c] = x[2 + c];
            }
        }
    }
    auto pick = [&](bool l) {
        us0 = l ? usl0 : usr0;
        rssm = l ? rslsm : rsrsm;
        root = l ? rtl : rtr;
        a = l ? alfven_l : alfven_r;
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            vs[c] = l ? vsl[c] : vsr[c];
            bs[c] = l ? bsl[c] : bsr[c];
        }
    };
    left = left || both;
    pick(left);
    side(left, alfven ? 2 : 1, false);
    if (both) {                                                                      // sm = 0
        pick(false);
        side(false, alfven ? 2 : 1, true);
    }
}

// HLLC flux of one interface (riemann_hlld_u, hlld.F90:615-841): the side the flux
// is taken from picked by selects, both where sm = 0.
template <class A>
PK_PHYS void hllc_face(A& ar, bool has_energy, double gamma, double rgam_1, const double (&ul)[5],
                       const double (&ur)[5], double (&f)[5])
{
    const bool dust = gamma < 0.0;
    double prl = 0.0, prr = 0.0, c_fastm = 0.0;                                      // hlld.F90:673-677
    if (!dust) {                                                                     // :689-703
        prl = ul[4];
        prr = ur[4];
        const double gampr_l = gamma * ul[4];
        const double gampr_r = gamma * ur[4];
        double cmax;
        if constexpr (A::FAST) {
            const bool lm = gampr_l * ur[0] >= gampr_r * ul[0];
            cmax = ar.div(lm ? gampr_l : gampr_r, lm ? ul[0] : ur[0]);
        } else {
            cmax = f_max(ar.quo(gampr_l, ul[0], ar.inv(ul[0])), ar.quo(gampr_r, ur[0], ar.inv(ur[0])));
        }
        c_fastm = sqrt(cmax);
    }
    const double sl = f_min(ul[1], ur[1]) - c_fastm;                                // :719-720
    const double sr = f_max(ul[1], ur[1]) + c_fastm;
    const bool fan = !(sl >= 0.0 || sr <= 0.0);                                      // :738-743
    bool left = sl >= 0.0, both = false;
    double sm = 0.0, prt_star = 0.0;
    if (fan) {
        const double dn_l = ul[0] * (sl - ul[1]), dn_r = ur[0] * (sr - ur[1]);       // :747-764
        const double n = (dn_r * ur[1] - prr) - (dn_l * ul[1] - prl), d = dn_r - dn_l;
        if (fabs(d) < f_spacing(dn_r + dn_l)) {
            sm = (sl + sr) * 0.5;
        } else {
            if constexpr (A::FAST) sm = ar.div(n, d);
            else {
                A g;
                const double gn[1] = {n}, gd[1] = {d};
                double x[1] = {g.quoz(n, d, g.inv(d))};
                g.settle(gn, gd, x);
                sm = x[0];
            }
        }
        prt_star = 0.5 * ((prl + dn_l * (sm - ul[1])) + (prr + dn_r * (sm - ur[1])));
        left = !(sm < 0.0);
        both = left && !(sm > 0.0);
    }
    auto side = [&](bool l, bool add) {
        double u[5];
#pragma unroll
        for (int c = 0; c < 5; ++c) u[c] = l ? ul[c] : ur[c];
        const double s = l ? sl : sr, pr = l ? prl : prr;
        double en = 1.7976931348623157e308;
        if (!dust) {
            double ei;
            if constexpr (A::FAST) ei = u[4] * rgam_1;
            else ei = ar.quoc(u[4], gamma - 1.0, rgam_1);
            en = ei + ((0.5 * u[0]) * ((u[1] * u[1] + u[2] * u[2]) + u[3] * u[3]));
        }
        const double uc[5] = {u[0], u[0] * u[1], u[0] * u[2], u[0] * u[3], en};
        const double fs[5] = {uc[1], (u[0] * (u[1] * u[1])) + pr, uc[2] * u[1], uc[3] * u[1], (en + pr) * u[1]};   // :724-734
        if (!fan) {
#pragma unroll
            for (int c = 0; c < 5; ++c) f[c] = fs[c];
            return;
        }
        const double svx = s - u[1], ssm = s - sm, rssm = ar.inv(ssm);               // :771-796
        const double us0 = ar.quo(u[0] * svx, ssm, rssm);
        double us[5] = {us0, us0 * sm, us0 * u[2], us0 * u[3], 0.0};
        if (has_energy) us[4] = ar.quo(((svx * en) - (pr * u[1])) + (prt_star * sm), ssm, rssm);
#pragma unroll
        for (int c = 0; c < 5; ++c) {                                                // :798-829
            const double d = s * (us[c] - uc[c]);
            f[c] = add ? 0.5 * ((f[c] + fs[c]) + d) : fs[c] + d;
        }
    };
    side(left, false);
    if (both) side(false, true);
}

PK_PHYS void hlld_iface(bool has_energy, double gamma, const double* ul, const double* ur, const double* bl,
                       const double* br, double* f, double* bf)
{
    Ieee ar;
    const double l[5] = {ul[0], ul[1], ul[2], ul[3], has_energy ? ul[4] : 0.0};
    const double r[5] = {ur[0], ur[1], ur[2], ur[3], has_energy ? ur[4] : 0.0};
    const double x[3] = {bl[0], bl[1], bl[2]}, y[3] = {br[0], br[1], br[2]};
    double o[5] = {0.0, 0.0, 0.0, 0.0, 0.0}, ob[2] = {0.0, 0.0};
    hlld_face(ar, has_energy, gamma, 0.0, 0.0, l, r, x, y, o, ob);
    for (int c = 0; c < (has_energy ? 5 : 4); ++c) f[c] = o[c];
    bf[0] = ob[0];
    bf[1] = ob[1];
}

PK_PHYS void hllc_iface(bool has_energy, double gamma, const double* ul, const double* ur, double* f)
{
    Ieee ar;
    const double l[5] = {ul[0], ul[1], ul[2], ul[3], has_energy ? ul[4] : 0.0};
    const double r[5] = {ur[0], ur[1], ur[2], ur[3], has_energy ? ur[4] : 0.0};
    double o[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
    hllc_face(ar, has_energy, gamma, 0.0, l, r, o);
    for (int c = 0; c < (has_energy ? 5 : 4); ++c) f[c] = o[c];
}

// riemann_wrap / riemann_wrap_u (hlld.F90:62-155) for one interface of the
// whole state: fluid fluxes, then (MHD) fluxes of Bx, By, Bz, psi.
template <class PH>
PK_PHYS void riemann(const double (&ql)[PH::NV], const double (&qr)[PH::NV], double ch, const PhysParams& pp,
                    double (&fx)[PH::NV])
{
    if (PH::MHD) {
        const double bxl = ql[PH::IB], bxr = qr[PH::IB], psl = ql[PH::IB + 3], psr = qr[PH::IB + 3];
        fx[PH::IB + 3] = ((ch * ch) * 0.5) * ((bxr + bxl) - (psr - psl) / ch);       // hlld.F90:229 (Dedner eq. 42)
        fx[PH::IB] = 0.5 * ((psr + psl) - ch * (bxr - bxl));                          // :230
    }
#pragma unroll
    for (int f = 0; f < PH::NFL; ++f) {
        const int b = PH::beg(f);
        double fv[5];
        if (PH::MHD) {
            double blv[3] = {0.0, 0.0, 0.0}, brv[3] = {0.0, 0.0, 0.0}, bf[2];
            if (PH::magn(f)) {
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    blv[c] = ql[PH::IB + c];
                    brv[c] = qr[PH::IB + c];
                }
            }
            hlld_iface(PH::has_en(f), pp.gam[f], &ql[b], &qr[b], blv, brv, fv, bf);
            if (PH::magn(f)) {
                fx[PH::IB + 1] = bf[0];
                fx[PH::IB + 2] = bf[1];
            }
        } else {
            hllc_iface(PH::has_en(f), pp.gam[f], &ql[b], &qr[b], fv);
        }
#pragma unroll
        for (int c = 0; c < 5; ++c)
            if (c < PH::ncomp(PH::kind(f))) fx[b + c] = fv[c];
    }
}

// internal_sources (+0 added to every fluid component) and care_for_positives
// on one updated cell; B used for emag is the updated one (b1).  quotient(n, d, big):
// n / d, correctly rounded unless a positive energy big absorbs it.  (It does: the
// kinetic energy enters u - kin and, with the floored internal energy, e + kin.
// Where u > 0 and 2^62 kin < u, u - kin = u; for a magnetised fluid whose field
// energy cancels u the sum with that energy follows and absorbs it.)
struct IeeeQuotient {
    PK_PHYS double operator()(double n, double d, double) const { return n / d; }
};

template <class PH, class Quotient = IeeeQuotient>
PK_PHYS void sources_and_floors(double (&u)[PH::NV], const PhysParams& pp, unsigned& status,
                                const Quotient& quotient = Quotient())
{
#pragma unroll
    for (int c = 0; c < PH::NVF; ++c) u[c] = u[c] + 0.0;
#pragma unroll
    for (int f = 0; f < PH::NFL; ++f) {                                   // limit_minimal_density
        const int b = PH::beg(f);
        if (u[b] < 0.0) status |= ST_DN_NEGATIVE;
        if (pp.use_smalld) u[b] = f_max(u[b], pp.smalld);
    }
#pragma unroll
    for (int f = 0; f < PH::NFL; ++f) {                                   // limit_minimal_intener
        if (!PH::has_en(f)) continue;
        const int b = PH::beg(f);
        const double kin = quotient(0.5 * ((u[b + 1] * u[b + 1] + u[b + 2] * u[b + 2]) + u[b + 3] * u[b + 3]), u[b],
                                    u[b + 4] > 0.0 ? u[b + 4] : 0.0);
        double mag = 0.0, eint;
        if (PH::magn(f)) {
            const double bx = u[PH::IB], by = u[PH::IB + 1], bz = u[PH::IB + 2];
            mag = 0.5 * ((bx * bx + by * by) + bz * bz);
            eint = (u[b + 4] - kin) - mag;
        } else {
            eint = u[b + 4] - kin;
        }
        if (pp.disallow_negatives && eint < 0.0) status |= ST_EI_NEGATIVE;
        if (pp.use_smallei) eint = f_max(eint, pp.smallei);
        double e = eint + kin;
        if (PH::magn(f)) e = e + mag;
        u[b + 4] = e;
    }
}

// ---------------------------------------------------------------------------
// internal_sources + care_for_positives with a record of the floors taken
// ---------------------------------------------------------------------------
struct FloorRec {
    unsigned dn;   // bit f: the density floor of fluid f clipped
    unsigned en;   // bit f: the internal-energy floor of fluid f clipped
};

template <class PH, class Quotient = IeeeQuotient>
PK_PHYS void floors_rec(double (&u)[PH::NV], const PhysParams& pp, unsigned& status, FloorRec& rec,
                        const Quotient& quotient = Quotient())
{
    rec.dn = 0;
    rec.en = 0;
#pragma unroll
    for (int c = 0; c < PH::NVF; ++c) u[c] = u[c] + 0.0;
#pragma unroll
    for (int f = 0; f < PH::NFL; ++f) {
        const int b = PH::beg(f);
        if (u[b] < 0.0) status |= ST_DN_NEGATIVE;
        if (pp.use_smalld) {
            if (pp.smalld > u[b]) rec.dn |= 1u << f;
            u[b] = f_max(u[b], pp.smalld);
        }
    }
#pragma unroll
    for (int f = 0; f < PH::NFL; ++f) {
        if (!PH::has_en(f)) continue;
        const int b = PH::beg(f);
        const double kin = quotient(0.5 * ((u[b + 1] * u[b + 1] + u[b + 2] * u[b + 2]) + u[b + 3] * u[b + 3]), u[b],
                                    u[b + 4] > 0.0 ? u[b + 4] : 0.0);
        double mag = 0.0, eint;
        if (PH::magn(f)) {
            const double bx = u[PH::IB], by = u[PH::IB + 1], bz = u[PH::IB + 2];
            mag = 0.5 * ((bx * bx + by * by) + bz * bz);
            eint = (u[b + 4] - kin) - mag;
        } else {
            eint = u[b + 4] - kin;
        }
        if (pp.disallow_negatives && eint < 0.0) status |= ST_EI_NEGATIVE;
        if (pp.use_smallei) {
            if (pp.smallei > eint) rec.en |= 1u << f;
            eint = f_max(eint, pp.smallei);
        }
        double e = eint + kin;
        if (PH::magn(f)) e = e + mag;
        u[b + 4] = e;
    }
}

}  // namespace pk
