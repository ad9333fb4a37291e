// pk_quotient.cuh -- correctly rounded quotients without branches.
//
// The bit-exact kernels take about 28 quotients per cell and RK stage (MHD).  The
// compiler's division is a sequence with a conditional slow path: 19 issue
// slots, 126 cycles of latency, and because each one ends in a branch,
// independent divisions of a thread do not overlap (measured on B200: 34
// cycles per warp and division at four warps per scheduler, whether a thread
// has one or four independent ones in flight; a fused multiply-add takes 2).
// Exact computes the same bits from a reciprocal per denominator and three
// operations per quotient, straight-line, and records whether every operand
// was in the range where that is proven: numerators in [1e-231, 1e77] or zero,
// denominators in [5e-79, 7e75].  Others are divided in IEEE operations: a group of
// quotients at its end (settle), else the whole solve out of line (the callers'
// `if (!ar.ok())`).
// The small end is met in earnest: ahead of a blast in a medium at rest the
// velocities, Bz and psi fade through all exponents, and squares of them twice
// as fast.  While every such thread solved its face again in IEEE operations, a step
// of a 128^3 MHD blast took up to 4.0 ms (van Leer; 256^3 moncen 33) where IEEE
// divisions everywhere take 2.8 (26): up to half of the warps held one.  Hence
// settle, quoa and quob (quotients whose bits do not matter when they are that
// small) and the scaled mean: now at most 2.6 (23).  They cost 3 % where nothing
// fades: a step of the 256^3 MHD block 16.4 -> 16.9 ms, of a 16^3 one 9 %.
//
// Why the bits are the same (P. Markstein, "Computation of elementary functions
// on the IBM RISC System/6000 processor", IBM J. Res. Dev. 34 (1990) 111-119;
// ulp: unit in the last place of the result, d scaled into [1, 2)):
//  * y: the hardware's reciprocal approximation (about 20 bits) and three
//    Newton steps y + y (1 - d y).  After two of them y is less than an ulp off,
//    so the third's residual 1 - d y is exact and its result is the rounded 1/d:
//    with the one known exception of d = 2 - 2^-52 reached from below, which
//    rounding the second step upwards excludes.  So |y - 1/d| <= 2^-54.
//  * q = n y rounded, r = n - d q (exact by the fused operation, no underflow in
//    the checked range), result q + r y rounded once.  Before that rounding it
//    is off n/d by |r| |y - 1/d|.  (r is a multiple of the last places of d times
//    those of q, at least 2^-1073 where |n| >= 2^-968 and q is normal.)  A wrong rounding needs n/d closer than that to
//    the midpoint of two neighbours, but n/d stays at least 2^-53 / d ulp away
//    from every midpoint (n 2^k - d m is a nonzero integer in last places).
//    Where q is one of the two neighbours, |r| = d / 2 ulp there, and the error
//    stays below (d^2 / 4) 2^-53 / d ulp, less than the distance as d < 2.  Where
//    q is a neighbour's neighbour (n < d, n y off n/d by almost an ulp, 1 - 2^-52
//    at most since n <= 2 - 2^-51), n/d lies 2^-52 ulp beyond the midpoint and the
//    error is at most 1.5 2^-53 ulp.
//  * A zero numerator gives a zero; its sign is q's, which is put back.
// tests/test_gpu_quotient.py compares with CUDA's division over random and
// adversarial operands.  Measured with utoq and the Riemann solvers on it (one
// side's energy and flux, too): a step of the 256^3 MHD block 18.0 -> 16.6 ms, of
// a 64^3 Sedov blast 0.39 -> 0.26 ms, of a 149 x 93 x 70 open gas box 2.25 -> 1.31 ms,
// of the three-fluid refined blast 28.1 -> 23.3 ms.  (Picking the side before its
// star state, with fewer quotients and roots still, was slower: 18.4, 31.4 ms; its
// one chain of dependent operations leaves nothing to overlap.)
#pragma once
#include "pk_device.cuh"

namespace pk {

// the hardware's FP64 reciprocal approximation
PK_DEV double rcp_seed(double x)
{
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    return r;
}

static __device__ __noinline__ double divide_ieee(double n, double d) { return n / d; }

struct Exact {
    static constexpr bool FAST = false;
    // |n| in [2^-768, 2^256) and |d| in [2^-260, 2^252) keep every intermediate and
    // the quotient normal.  t = 2 x high word holds the exponent in its upper 11 bits:
    // a numerator outside its range sets the top bit of bad_n, a denominator one
    // of the two top bits of bad_d.
    unsigned bad_n = 0, bad_d = 0;
    static constexpr unsigned LOW_N = (1023u - 768u) << 21;            // twice(2^-768)
    PK_DEV static unsigned twice(double x) { return 2u * (unsigned)__double2hiint(x); }
    PK_DEV static unsigned high(double x) { return (unsigned)__double2hiint(x) & 0x7fffffffu; }
    PK_DEV bool ok() const { return (((bad_n >> 1) | bad_d) >> 30) == 0; }
    PK_DEV void need(double n) { bad_n |= twice(n) - LOW_N; }
    PK_DEV void needz(double n)             // the same, or zero
    {
        if (n != 0.0) need(n);
    }
    // the end of a group of G quotients x = n / d: the ones whose operands faded out of
    // the range are divided in IEEE operations here, so that the rest of the work
    // need not be done twice
    template <int G>
    PK_DEV void settle(const double (&n)[G], const double (&d)[G], double (&x)[G])
    {
        if (ok()) return;
#pragma unroll
        for (int k = 0; k < G; ++k) x[k] = divide_ieee(n[k], d[k]);
        bad_n = bad_d = 0;
    }
    PK_DEV void needd(double d) { bad_d |= twice(d) - ((1023u - 260u) << 21); }
    PK_DEV double inv(double d)
    {
        needd(d);
        return rounded_inverse(d);
    }
    PK_DEV static double rounded_inverse(double d)
    {
        const double m = fabs(d);
        double y = rcp_seed(m);
        y = fma(y, fma(-m, y, 1.0), y);
        y = __fma_ru(y, fma(-m, y, 1.0), y);
        return copysign(fma(y, fma(-m, y, 1.0), y), d);
    }
    PK_DEV static double quotient(double n, double d, double y, double& q)
    {
        q = n * y;
        return fma(fma(-d, q, n), y, q);
    }
    PK_DEV double quo(double n, double d, double y)
    {
        double q;
        need(n);
        return quotient(n, d, y, q);
    }
    PK_DEV static double signed_as(double x, double q)      // a zero quotient's sign is q's
    {
        return __hiloint2double((__double2hiint(x) & 0x7fffffff) | (__double2hiint(q) & 0x80000000), __double2loint(x));
    }
    PK_DEV double quoz(double n, double d, double y)
    {
        double q;
        const double x = quotient(n, d, y, q);
        needz(n);
        return signed_as(x, q);
    }
    // quoz of a quotient that only ever enters sums with `big`: where the numerator is
    // below 2^-768 it need not be right if big is at least 2^-440 (then it is less than
    // 2^-62 of big, and the rounded sum is big), so big must be in [2^-440, 2^584)
    PK_DEV double quoa(double n, double d, double y, double big)
    {
        double q;
        const double x = quotient(n, d, y, q);
        if (n != 0.0) bad_n |= twice(n) < LOW_N ? twice(big) - ((1023u - 440u) << 21) : twice(n) - LOW_N;
        return signed_as(x, q);
    }
    // a quotient that is only compared with a and b, by a constant d >= 1 whose rounded
    // reciprocal is y: below the range it need not be right where |a| and |b| are at
    // least 2^-750
    PK_DEV double quob(double n, double d, double y, double a, double b)
    {
        double q;
        needd(d);
        const double x = quotient(n, d, y, q);
        if (n != 0.0)
            bad_n |= twice(n) < LOW_N ? (twice(a) - ((1023u - 750u) << 21)) | (twice(b) - ((1023u - 750u) << 21))
                                      : twice(n) - LOW_N;
        return signed_as(x, q);
    }
    // van Leer's quotient 2 p / d of p = a b > 0 and d = a + b: taken as 2^401 p / 2^400 d,
    // which is the same quotient with its intermediates in range down to the
    // smallest products; needs d < 2^100 and a normal quotient; p = 0, d = 1 elsewhere
    PK_DEV double mean(double p, double d)
    {
        double q;
        const double n2 = p * 0x1p401, d2 = d * 0x1p400, x = quotient(n2, d2, rounded_inverse(d2), q);
        if (p != 0.0) {
            bad_n |= (twice(d) - ((1023u - 924u) << 21)) | (high(q) - (2u << 20));
        }
        return x;
    }
    PK_DEV double quoc(double n, double d, double y)
    {
        needd(d);
        return quoz(n, d, y);
    }
    PK_DEV double root(double x, double&) { return sqrt(x); }
    PK_DEV double over_root(double n, double root, double)
    {
        return quo(n, root, inv(root));
    }
};

// the IEEE versions for a thread whose operands left the range: out of line, so
// that their registers and code stay out of the kernels' way
// x: ul(5), ur(5), bl(3), br(3); f: fluid fluxes (5), transverse B fluxes (2)
static __device__ __noinline__ void hlld_ieee(bool has_energy, double gamma, const double* x, double* f)
{
    f[4] = 0.0;
    hlld_iface(has_energy, gamma, x, x + 5, x + 10, x + 13, f, f + 5);
}

static __device__ __noinline__ void hllc_ieee(bool has_energy, double gamma, const double* x, double* f)
{
    f[4] = 0.0;
    hllc_iface(has_energy, gamma, x, x + 5, f);
}

static __device__ __noinline__ void weno3_ieee(double qm, double qc, double qp, double weps, double* lr)
{
    Ieee ar;
    weno3_faces(ar, qm, qc, qp, weps, lr[0], lr[1]);
}

// Half slopes of van Leer's limiter (0.5 * slope_interior(L_VANLEER, ...): dl dr /
// (dl + dr) where dl dr > 0, else 0) of a group of G components: their quotients
// overlap, and a warp in a uniform region skips them together.  Zero at the
// pencil ends (on: not one).
// Against an IEEE division per component: unsplit step of a 128^3 MHD block
// 2.14 -> 2.01 ms, refined blast 23.3 -> 22.8; a 64^3 Sedov blast, at rest
// almost everywhere, 0.26 either way (without the joint skip 0.28).
// again(k, dl, dr) gives component k's differences once more, for the IEEE redo.
template <int G, class Again>
PK_DEV void vanleer_half(bool on, const double (&dl)[G], const double (&dr)[G], double (&h)[G], const Again& again)
{
    double n[G], d[G];
    bool any = false;
#pragma unroll
    for (int k = 0; k < G; ++k) {
        const double dcen = dl[k] * dr[k];
        const bool up = on && dcen > 0.0;
        n[k] = up ? dcen : 0.0;
        d[k] = up ? dl[k] + dr[k] : 1.0;
        h[k] = 0.0;
        any = any || up;
    }
    if (any) {
        Exact ar;
#pragma unroll
        for (int k = 0; k < G; ++k) h[k] = 0.5 * ar.mean(n[k], d[k]);
        if (!ar.ok()) {
#pragma unroll
            for (int k = 0; k < G; ++k) {
                double a, b;
                again(k, a, b);
                h[k] = a * b > 0.0 ? 0.5 * divide_ieee(2.0 * (a * b), a + b) : 0.0;
            }
        }
    }
}

// n / d, correctly rounded unless only sums with `big` follow that absorb it: the
// floors' quotient
struct ExactQuotient {
    PK_DEV double operator()(double n, double d, double big) const
    {
        Exact ar;
        const double x = ar.quoa(n, d, ar.inv(d), big);
        return ar.ok() ? x : divide_ieee(n, d);
    }
};

}  // namespace pk
