// fp64_cell.cuh -- the plain FP64 form of the column solve: arithmetic, gas
// optics, layer solution, clouds, preparation (the kernels: fp64.cuh).
//
// GB300 runs FP64 at 1/64 of its FP32 rate (two FP64 lanes per SM and
// cycle), so this form is bound by the FP64 pipe alone: an FP64 warp
// instruction holds it for 16 cycles, while integer, FP32 and memory
// instructions run beside it for next to nothing.  Everything here is
// written to issue few FP64 instructions per (g-point, layer) cell:
//
//   - no IEEE division or square root per cell: rcp64 / sqrt64 start from
//     the hardware's approximation and take one third-order step (3 and 5
//     FP64 instructions, error about an ulp) instead of a division sequence;
//   - explicit fma() (solve_fp64.cu is compiled without contraction, so its
//     kernels, which all inline these functions, round alike, bit for bit;
//     the derivatives' unit is not);
//   - what does not depend on the g-point is made once per (column, layer,
//     band): the species-ratio interpolation of taumol and the cloud and
//     aerosol optics (14 bands against 112 g-points);
//   - one gas-optics path for all bands (a warp's g-points span several);
//   - the nearest-entry index of the transmittance table comes from a pair
//     of FP32 numbers (tbl_index64), the FP64 quotient only when the pair
//     cannot decide; comparisons of positive numbers are integer ones;
//   - the layer solution has one reciprocal for reflectances and
//     transmittances, direct and diffuse (two_stream64);
//   - the vertical adding (rrtmg_sw_vrtqdr.f90:122-169) is solved as a
//     linear recurrence (up64 / down below): with the upward albedos known,
//     the diffuse flux below a layer follows from the fluxes above it through
//     the division that the up-sweep has done already.
//
// 172 FP64 instructions per cell with clouds and aerosol (without aerosol a dozen fewer
// in the layer solution alone: gamma3 = gamma4 = 1/2 and one alpha) where the
// reference's order of operations took about 570: 16 384 x 60 columns with
// clouds and aerosol 102.9 -> 36.3 ms, 4 096 x 60 with clouds 28.2 -> 8.4 ms,
// the FP64 pipe 84 % busy.  The layer solution is also written without the cancellation of
// thin layers: against a solve in 80-bit arithmetic the heating rates of
// 1 024 x 60 clear columns are 8.6e-11 off (2-norm), 1.04e-10 in the
// reference's order.  Cells near the two-stream resonance k mu0 = 1, where the
// reference divides rounding by a small number, keep its order (cell_ref64).
#pragma once

#include "kernel.cuh"

namespace rrsw {

// ------------------------------------------------------------ arithmetic
// 1/x for finite normal x with a normal reciprocal: the hardware's
// approximation r, e = 1 - x r (|e| < 2^-19), and one step of Householder's
// iteration of third order for r -> 1/x, r (1 + e + e^2) (A. S. Householder,
// The Numerical Treatment of a Single Nonlinear Equation, 1970); error below an ulp.
__device__ __forceinline__ double rcp64(double x) {
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    const double e = fma(-x, r, 1.0);
    return fma(r, fma(e, e, e), r);
}

// sqrt(x) for positive normal x: y ~ x^-1/2 from the hardware, e = 1 - x y^2, and
// the same iteration for y -> x^-1/2 times x: sqrt(x) = x y (1 + e/2 + 3 e^2 / 8),
// the binomial series of x y (1 - e)^-1/2; error below 1.1 ulp.
__device__ __forceinline__ double sqrt64(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double m = x * y;
    const double e = fma(-m, y, 1.0);
    return fma(m * e, fma(0.375, e, 0.5), m);
}

// a <= b, a < b for a, b >= 0, on the integer pipe
__device__ __forceinline__ bool le_pos(double a, double b) { return __double_as_longlong(a) <= __double_as_longlong(b); }
__device__ __forceinline__ bool lt_pos(double a, double b) { return __double_as_longlong(a) < __double_as_longlong(b); }

// A positive double in FP32's range as an FP32 pair hi + lo (46 bits), by
// bit operations: conversions run at the FP64 rate.
__device__ __forceinline__ void split32(double x, float& hi, float& lo) {
    const unsigned h = (unsigned)__double2hiint(x), l = (unsigned)__double2loint(x);
    const unsigned b = ((h - 0x38000000u) << 3) | (l >> 29);
    const unsigned e = b & 0x7f800000u;
    hi = __uint_as_float(b);
    lo = (__uint_as_float(e | ((l >> 6) & 0x7fffffu)) - __uint_as_float(e)) * 1.1920929e-07f;  // 2^-23
}

// x in FP32 (truncated; 0 below FP32's range), by bit operations
__device__ __forceinline__ float to32(double x) {
    const unsigned h = (unsigned)__double2hiint(x), l = (unsigned)__double2loint(x);
    const unsigned a = h & 0x7fffffffu;
    const unsigned b = a < 0x38100000u ? 0u : ((a - 0x38000000u) << 3) | (l >> 29);
    return __uint_as_float(b | (h & 0x80000000u));
}

// The reference's table index int(1e4 x / (bpade + x) + 0.5)
// (rrtmg_sw_reftra.f90:206-208) for 0.06 < x <= 500.  With i the FP32
// estimate, x (1e4 - i) - i bpade lies within half of bpade + x of zero
// exactly when i is the nearest entry; the difference is formed from FP32
// pairs (error below 1e-9 of bpade + x).  Within 2e-6 of an entry's edge
// the FP64 expression decides.
__device__ __forceinline__ int tbl_index64(double x) {
    float xh, xl;
    split32(x, xh, xl);
    const float bh = 3.5971222f;                               // 1 / 0.278 rounded to FP32 ..
    const float bl = (float)(1.0 / 0.278 - (double)3.5971222f);  // .. and the rest
    const float s = bh + xh;
    int i = (int)fmaf(10000.0f, __fdividef(xh, s), 0.5f);
    const float fi = (float)i, n = 10000.0f - fi;
    const float p = xh * n, q = fi * bh;
    const float d = (p - q) + ((fmaf(xh, n, -p) - fmaf(fi, bh, -q)) + (xl * n - fi * bl));
    const float over = fabsf(d) - 0.5f * s;
    if (fabsf(over) < 2.0e-6f * s) {
        i = (int)(10000.0 * (x / (cT.bpade + x)) + 0.5);
    } else if (over > 0.0f) {
        i += d > 0.0f ? 1 : -1;
    }
    return min(max(i, 0), NTBL);
}

// exp(-x) of the model for x >= 0 (x <= 500: beyond, the table holds its
// floor everywhere) and 1 - exp(-x), without cancellation where the
// quadratic stands for the table (rrtmg_sw_reftra.f90:203-209).
__device__ __forceinline__ double tbl_exp64(double x, const double* __restrict__ tab, double& om) {
    if (le_pos(x, 0.06)) {
        om = x * fma(-0.5, x, 1.0);
        return 1.0 - om;
    }
    const double e = ldt(tab, cT.exp_tbl + tbl_index64(x));
    om = 1.0 - e;
    return e;
}

__device__ __forceinline__ double clip500(double x) { return le_pos(x, 500.0) ? x : 500.0; }

// --------------------------------------------------------- prepared block
// One (column, layer) of the prepared block (doubles): setcoef's
// coefficients (F_*), the packed indices, per band the column amount that
// multiplies its k-table interpolation, per two-species band the fraction fs
// and the integer part js of the species ratio, the McICA thresholds.
enum { B_PK = NFR, B_COMB, B_FS = B_COMB + NBND, B_JS = B_FS + 8, B_TH, B_N = B_TH + 3 };
constexpr int B_STRIDE = (B_N + 1) & ~1;
// cloud optics of one (column, layer, band): delta-scaled depth, its
// scattering part, that times the asymmetry, its absorbing part, unscaled
// depth, error code
enum { CO_TAU, CO_S, CO_SG, CO_AB, CO_TAOR, CO_ERR, CO_N };
// aerosol of one (column, layer, band): depth, scattering, that times the
// asymmetry, absorption
enum { AO_TAU, AO_S, AO_SG, AO_AB, AO_N };

// level fields per (column, g-point, layer) and sky between the sweeps: the
// upward albedos (direct, diffuse) at the layer's top, the diffuse flux below
// the layer per direct and per diffuse flux above it, the direct
// transmittance.  The split kernels first keep the layer solution there:
// ref, refd, diffuse transmittance of the direct beam, trad, dbt.
enum { L_RUP, L_RUPD, L_ALPHA, L_BETA, L_DBT, L_SKY };
enum { L_REF = L_RUP, L_REFD = L_RUPD, L_TDIF = L_ALPHA, L_TRAD = L_BETA };
// idelm = 0 adds the unscaled direct transmittance of the total sky
__host__ __device__ inline int fields64(int idelm) { return 2 * L_SKY + (idelm == 0 ? 1 : 0); }

struct Slot64 {
    size_t blk, cld, aer, total;  // doubles; the level fields come first
};
__host__ __device__ inline Slot64 slot64(int L, int idelm, int nc, bool clouds, bool aerosol) {
    Slot64 s;
    size_t o = (size_t)L * fields64(idelm) * (size_t)(nc * NGPT);
    s.blk = o; o += (size_t)nc * L * B_STRIDE;
    s.cld = o; if (clouds) o += (size_t)nc * L * NBND * CO_N;
    s.aer = o; if (aerosol) o += (size_t)nc * L * NBND * AO_N;
    s.total = (o + 31) & ~(size_t)31;
    return s;
}

// Whether cloud optics are prepared per band (fused McICA, non-McICA path)
__host__ __device__ inline bool band_clouds(const SolveParams& P) { return (P.fused || P.nomcica) && P.icld >= 1; }

__device__ inline void fill_tm64(TmSmem* d) {
    for (int i = threadIdx.x; i < NBND * 2; i += blockDim.x) {
        TmSmem t;
        t.r = cT.tm[i / 2][i % 2];
        t.selfref = cT.b[i / 2].selfref;
        t.forref = cT.b[i / 2].forref;
        t.ng = cT.b[i / 2].ng;
        t.pad = cT.sslot[i / 2];
        d[i] = t;
    }
}

// ------------------------------------------------------------ gas optics
// One g-point of taumol16..29 (rrtmg_sw_taumol.f90:275-1785) through the band
// and region descriptors: `blk` is the (column, layer) block.
__device__ __forceinline__ void taumol64(const TmSmem& t, int ib, int ig, const double* blk,
                                         const double* __restrict__ tab, double& taug, double& taur) {
    const TmRegion& d = t.r;
    const int ng = t.ng, slot = t.pad;
    const int pk = *(const int*)(blk + B_PK);
    double tg = 0.0, fs = 0.0;
    int js = 0;
    if (d.kind == 1) {
        fs = blk[B_FS + slot];
        js = ((const unsigned char*)(blk + B_JS))[slot];
    }
    if (d.kind != 0) {
        const int jp = (pk & 0xff) - d.jo, jt = (pk >> 8) & 0xf, jt1 = (pk >> 12) & 0xf;
        const int nsp = d.nsp, two = d.kind == 1 ? ng : 0;  // one species: both ends of the ratio are the same entry
        const int i0 = d.ktab + ((jp * 5 + (jt - 1)) * nsp + js) * ng + ig - 1;
        const int i1 = d.ktab + (((jp + 1) * 5 + (jt1 - 1)) * nsp + js) * ng + ig - 1;
        const int dn = nsp * ng;
        const double a0 = ldt(tab, i0), a1 = ldt(tab, i0 + two), b0 = ldt(tab, i0 + dn), b1 = ldt(tab, i0 + dn + two);
        const double c0 = ldt(tab, i1), c1 = ldt(tab, i1 + two), e0 = ldt(tab, i1 + dn), e1 = ldt(tab, i1 + dn + two);
        double k = blk[F_FAC00] * fma(fs, a1 - a0, a0);
        k = fma(blk[F_FAC10], fma(fs, b1 - b0, b0), k);
        k = fma(blk[F_FAC01], fma(fs, c1 - c0, c0), k);
        k = fma(blk[F_FAC11], fma(fs, e1 - e0, e0), k);
        tg = blk[B_COMB + ib] * k;
    }
    if (d.cont >= 1) {
        const int indf = (pk >> 24) & 0xf;
        const double fa = ldt(tab, t.forref + (indf - 1) * ng + ig - 1), fb = ldt(tab, t.forref + indf * ng + ig - 1);
        double cont = blk[F_FORFAC] * fma(blk[F_FORFRAC], fb - fa, fa);
        if (d.cont == 1) {
            const int inds = (pk >> 16) & 0xff;
            const double sa = ldt(tab, t.selfref + (inds - 1) * ng + ig - 1);
            const double sb = ldt(tab, t.selfref + inds * ng + ig - 1);
            cont = fma(blk[F_SELFFAC], fma(blk[F_SELFFRAC], sb - sa, sa), cont);
        }
        tg = fma(blk[F_H2O], cont, tg);
    }
    if (d.minor == 9) tg = fma(4.35e-4 / 700.0, blk[F_O2], tg);
    else if (d.minor >= 0) tg = fma(blk[F_H2O + d.minor], ldt(tab, d.mtab + ig - 1), tg);
    double ra;
    if (d.rtype == 2) {
        const double r0 = ldt(tab, d.rtab + js * ng + ig - 1), r1 = ldt(tab, d.rtab + (js + 1) * ng + ig - 1);
        ra = fma(fs, r1 - r0, r0);
    } else {
        ra = ldt(tab, d.rtab + (d.rtype == 1 ? ig - 1 : 0));
    }
    taug = tg;
    taur = blk[F_MOL] * ra;
}

// ------------------------------------------------------------ two streams
// A layer's solution: reflectances, diffuse transmittance of the direct
// beam (ptra less the direct transmittance), of diffuse light, and the
// direct transmittance.
struct Rt64 {
    double ref, refd, tdif, trad, dbt;
};

struct Mu64 {
    double mu, rmu, mu34;  // mu0, its reciprocal, 3/4 mu0
};

// |1 - (k mu0)^2| / w below which a cell is computed in the reference's order:
// its numerators cancel there and divide their rounding (1e-16) by this
// number, so results agree with the reference's only operation by operation
// (a thin layer at 7e-7 moved a heating rate by 2e-7 K/day).  The scattered
// part carries a factor w; without it every absorbing cell of a column with
// mu0 near 1/2 (k = 2) would take that order, at four times the cost.
constexpr double RESONANCE64 = 2.0e-3;

// reftra_sw (rrtmg_sw_reftra.f90:151-326), kmodts = 2, from the layer's
// depth tau, its scattering part s, s times the asymmetry sg and its
// absorbing part ab (tau = s + ab).  With w = s/tau, wg = sg/tau,
// co = ab/tau: gamma1 - gamma2 = 2 co and gamma1 + gamma2 = 2 - w/2 - 3 wg/2,
// so k = sqrt(2 co (gamma1 + gamma2)).  The reference's numerators and its
// denominators zdenr and (1 - zbeta zem1^2) zrkg, all multiplied by
// zem1 = exp(-k tau), share B = k (1 + zem1^2) + gamma1 (1 - zem1^2):
// zdenr zem1 = (1 - (k mu0)^2) B.  near: the resonance is too close, the
// caller takes the reference's order.
template <bool G>  // G: the layer's asymmetry is not zero (aerosol or cloud)
__device__ __forceinline__ Rt64 two_stream64(double tau, double s, double sg, double ab, const Mu64& m,
                                             const double* __restrict__ tab, bool& near) {
    Rt64 o;
    const double rt = rcp64(tau);
    const double w = s * rt, co = ab * rt;
    double g = 0.0, wg = 0.0, g3, g4;
    double om2;
    const double e2 = tbl_exp64(clip500(tau * m.rmu), tab, om2);
    if constexpr (G) {
        wg = sg * rt;
        g = sg * rcp64(s);
        g3 = fma(-m.mu34, g, 0.5);
        g4 = 1.0 - g3;
    } else {
        g3 = g4 = 0.5;
    }
    // zwo >= 0.9999995 (reftra:183-188): decided in FP32 from the co-albedo,
    // 1 - zwo = co (1 - q^2) / (1 - co q^2) with q = g / (1 - g), and in FP64
    // in the reference's order where that is within 1 % of the switch
    bool cons;
    {
        const float cf = to32(co);
        float r = cf;
        bool sure = true;
        if constexpr (G) {
            const float gf = to32(g);
            const float q = gf / (1.0f - gf), q2 = q * q;
            const float den = 1.0f - cf * q2;
            r = cf * (1.0f - q2) / den;
            sure = fabsf(gf - 0.5f) > 0.01f && den > 0.01f;
        }
        cons = r <= 5.0e-7f;
        if (!sure || fabsf(r - 5.0e-7f) < 5.0e-9f) {
            double denom = 1.0, zwo = 0.0;
            if (g != 1.0) {
                const double q = g / (1.0 - g);
                denom = 1.0 - (1.0 - w) * (q * q);
            }
            if (w > 0.0 && denom != 0.0) zwo = w / denom;
            cons = zwo >= 0.9999995;
        }
    }
    o.dbt = e2;
    if (cons) {
        // conservative scattering (reftra:191-228)
        const double g1 = fma(-1.25, w, fma(-0.75, wg, 2.0));
        const double gt = g1 * tau;
        const double r1 = rcp64(1.0 + gt);
        o.ref = fma(-fma(g1, m.mu, -g3), om2, gt) * r1;
        o.refd = gt * r1;
        o.trad = 1.0 - o.refd;
        o.tdif = om2 - o.ref;
        if (__double_as_longlong(e2) == __double_as_longlong(1.0)) { o.ref = 0.0; o.refd = 0.0; o.trad = 1.0; o.tdif = 0.0; }
        return o;
    }
    // h: gamma1 - gamma2 with asymmetry, half of gamma1 + gamma2 without
    double h, g1, g2, k;
    if constexpr (G) {
        const double sum = fma(-0.5, w, fma(-1.5, wg, 2.0));
        h = co + co;
        g1 = fma(0.5, sum, co);
        g2 = fma(0.5, sum, -co);
        k = sqrt64(h * sum);
    } else {
        h = fma(-0.25, w, 1.0);
        g1 = h + co;
        g2 = h - co;
        k = sqrt64(4.0 * co * h);
    }
    const double kmu = k * m.mu;
    const double p1 = 1.0 + kmu, m1 = 1.0 - kmu;
    const double pp = p1 * m1;  // 1 - (k mu0)^2
    double om1;
    const double e1 = tbl_exp64(clip500(k * tau), tab, om1);
    const double oo = om1 * (1.0 + e1), k2 = k + k;  // oo = 1 - exp(-2 k tau)
    const double B = fma(g1 - k, oo, k2);
    const double pB = pp * B;  // zdenr zem1
    // (or |zdenr| <= 1e-8, where the reference replaces the solution)
    if (fabsf(to32(pp)) < (float)RESONANCE64 * to32(w) || lt_pos(fabs(pB), 1.1e-8)) near = true;
    const double r = rcp64(pB);
    const double rB = r * pp;        // 1 / B
    const double wr = w * r;
    // zr1 - zr2 ee - zr3 e1 e2 and zt3 e1 - e2 (zt1 - zt2 ee) with
    // zr1 = zr2 + zr3 and zt1 = zt2 + zt3: no cancellation in thin layers.
    // Without asymmetry gamma3 = gamma4 = 1/2, alpha1 = alpha2 = h.
    double r3, t3, r2o, t2o;  // zr3, zt3, zr2 oo, zt2 oo
    if constexpr (G) {
        const double a1 = fma(-h, g3, g1), a2 = fma(h, g3, g2);
        r3 = fma(-a2, m.mu, g3);
        t3 = fma(a1, m.mu, g4);
        r2o = p1 * fma(-k, g3, a2) * oo;
        t2o = m1 * fma(-k, g4, a1) * oo;
    } else {
        const double q = fma(-0.5, k, h) * oo;
        r3 = fma(-h, m.mu, 0.5);
        t3 = fma(h, m.mu, 0.5);
        r2o = p1 * q;
        t2o = m1 * q;
    }
    o.ref = wr * fma(k2 * r3, fma(e1, om2, om1), r2o);
    o.tdif = wr * fma(k2 * t3, om2 - om1, -e2 * t2o);
    o.refd = g2 * oo * rB;
    o.trad = k2 * e1 * rB;
    return o;
}

// ----------------------------------------------------------------- clouds
// Cloud optics of a layer in band ib (cldprmc_sw, rrtmg_sw_cldprmc.f90:53-349;
// with ttest >= 0 cldprop_sw's test) in the form two_stream64 takes.  The
// error code of an input out of range is returned in c[CO_ERR]: it counts
// only where a cloudy subcolumn meets it.  A radius that is no number counts as
// out of range: the preparation comes here for every layer that may be cloudy
// (with MT19937 for all), and some callers leave NaN where there is no cloud.
__device__ inline void cloud64(int ib, int inflag, int iceflag, int liqflag, double cldf, double ciwp, double clwp,
                               double rei, double rel, double fsfc, double tauc, double ssac, double asmc,
                               const double* __restrict__ tab, double ttest, double* c) {
    int err = 0;
    double taor = tauc, co = 1.0 - ssac;
    const double eps = 1.e-06, cldmin = 1.e-20;
    auto out = [&]() {
        const double sct = tauc * ssac;
        c[CO_TAU] = tauc;
        c[CO_S] = sct;
        c[CO_SG] = sct * asmc;
        c[CO_AB] = tauc * co;
        c[CO_TAOR] = taor;
        c[CO_ERR] = (double)err;
    };
    const double cwp = ciwp + clwp;
    if (!(cldf >= cldmin && (cwp >= cldmin || (ttest < 0.0 ? tauc : ttest) >= cldmin))) { out(); return; }
    if (inflag == 0) {
        const double f1 = 1.0 - fsfc, fs = 1.0 - fsfc * ssac, r = 1.0 / fs;
        co = (1.0 - ssac) * r;
        ssac = f1 * ssac * r;
        tauc = fs * tauc;
        asmc = (asmc - fsfc) / f1;
        out();
        return;
    }
    if (inflag != 2) { err = E_INFLAG1; out(); return; }
    double exti = 0.0, ssai = 0.0, gi = 0.0, fwi = 0.0, coi = 1.0, extl = 0.0, ssal = 0.0, gl = 0.0, fwl = 0.0, col = 1.0;
    auto lut = [&](int off, int n, int index, double f) {
        const double a = ldt(tab, off + ib * n + index - 1), b = ldt(tab, off + ib * n + index);
        return fma(f, b - a, a);
    };
    auto bad = [](double e, double s, double g) { return e < 0.0 || s > 1.0 || s < 0.0 || g > 1.0 || g < 0.0; };
    if (ciwp != 0.0 && iceflag == 1) {
        if (!(rei >= 13.0 && rei <= 130.0)) { err = E_ICERAD; out(); return; }
        const double w2 = ldt(tab, cT.wavenum2 + ib);
        const int icx = w2 > 1.43e04 ? 1 : w2 > 7.7e03 ? 2 : w2 > 5.3e03 ? 3 : w2 > 4.0e03 ? 4 : w2 >= 2.5e03 ? 5 : 0;
        exti = ldt(tab, cT.abari + icx - 1) + ldt(tab, cT.bbari + icx - 1) / rei;
        coi = fma(ldt(tab, cT.dbari + icx - 1), rei, ldt(tab, cT.cbari + icx - 1));
        ssai = 1.0 - ldt(tab, cT.cbari + icx - 1) - ldt(tab, cT.dbari + icx - 1) * rei;
        gi = fma(ldt(tab, cT.fbari + icx - 1), rei, ldt(tab, cT.ebari + icx - 1));
        if (gi >= 1.0) gi = 1.0 - eps;
        fwi = gi * gi;
        if (bad(exti, ssai, gi)) { err = E_ICEPROP; out(); return; }
    } else if (ciwp != 0.0 && iceflag == 2) {
        if (!(rei >= 5.0 && rei <= 131.0)) { err = E_ICERAD; out(); return; }
        const double factor = (rei - 2.0) / 3.0;
        int index = (int)factor;
        if (index == 43) index = 42;
        const double f = factor - (double)index;
        exti = lut(cT.extice2, 43, index, f);
        ssai = lut(cT.ssaice2, 43, index, f);
        coi = lut(cT.coice2, 43, index, f);
        gi = lut(cT.asyice2, 43, index, f);
        fwi = gi * gi;
        if (bad(exti, ssai, gi)) { err = E_ICEPROP; out(); return; }
    } else if (ciwp != 0.0 && iceflag == 3) {
        if (!(rei >= 5.0 && rei <= 140.0)) { err = E_ICEDGE; out(); return; }
        const double factor = (rei - 2.0) / 3.0;
        int index = (int)factor;
        if (index == 46) index = 45;
        const double f = factor - (double)index;
        exti = lut(cT.extice3, 46, index, f);
        ssai = lut(cT.ssaice3, 46, index, f);
        coi = lut(cT.coice3, 46, index, f);
        gi = lut(cT.asyice3, 46, index, f);
        const double fd = lut(cT.fdlice3, 46, index, f);
        if (fd < 0.0 || fd > 1.0) { err = E_ICEPROP; out(); return; }
        fwi = fd + 0.5 / ssai;
        if (fwi > gi) fwi = gi;
        if (bad(exti, ssai, gi)) { err = E_ICEPROP; out(); return; }
    }
    if (clwp != 0.0 && liqflag == 1) {
        if (!(rel >= 2.5 && rel <= 60.0)) { err = E_LIQRAD; out(); return; }
        int index = (int)(rel - 1.5);
        if (index == 0) index = 1;
        if (index == 58) index = 57;
        const double f = rel - 1.5 - (double)index;
        extl = lut(cT.extliq1, 58, index, f);
        ssal = lut(cT.ssaliq1, 58, index, f);
        col = lut(cT.coliq1, 58, index, f);
        if (f < 0.0 && ssal > 1.0) {
            ssal = ldt(tab, cT.ssaliq1 + ib * 58 + index - 1);
            col = ldt(tab, cT.coliq1 + ib * 58 + index - 1);
        }
        gl = lut(cT.asyliq1, 58, index, f);
        fwl = gl * gl;
        if (bad(extl, ssal, gl)) { err = E_LIQPROP; out(); return; }
    }
    // delta scaling (cldprmc:298-340): tau (1 - f ssa), scattering tau ssa
    // (1 - f), asymmetry (g - f) / (1 - f); so scattering times asymmetry is
    // tau ssa (g - f), and the absorption tau (1 - ssa) does not change
    const double tl = clwp * extl, ti = ciwp * exti;
    taor = tl + ti;
    const double td = fma(-fwl * ssal, tl, tl) + fma(-fwi * ssai, ti, ti);
    const double sl = tl * ssal, si = ti * ssai;
    double sc = (sl * (1.0 - fwl));
    double sic = si * (1.0 - fwi);
    if (sic == 0.0) sic = cldmin;
    sc += sic;
    const double gsum = sl * (gl - fwl) + (si * (1.0 - fwi) == 0.0 ? cldmin * ((gi - fwi) / (1.0 - fwi)) : si * (gi - fwi));
    c[CO_TAU] = td == 0.0 ? cldmin : td;
    c[CO_S] = sc;
    c[CO_SG] = gsum;
    c[CO_AB] = td == 0.0 ? 0.0 : tl * col + ti * coi;
    c[CO_TAOR] = taor;
    c[CO_ERR] = 0.0;
}

// ------------------------------------------------------------------ cells
// Which clouds a call has: none, prepared per band and switched by the
// McICA mask, the reference's subcolumn arrays, or the non-McICA path's
// layer clouds.
enum { CLD_NONE, CLD_MASK, CLD_ARRAYS, CLD_LAYER };
__host__ __device__ inline int cloud_mode(const SolveParams& P) {
    return P.icld < 1 ? CLD_NONE : P.nomcica ? CLD_LAYER : P.fused ? CLD_MASK : CLD_ARRAYS;
}

// One cell in the reference's order of operations.
static __device__ __noinline__ void cell_ref64(const SolveParams& P, const double* blk, bool low, int col, int g,
                                               int lay, int ib, int igb, bool cloudy, double cossza,
                                               const double* __restrict__ tab, Rt64& c, Rt64& t) {
    const Coef<double> C{blk, (const int*)(blk + B_PK), 1, low ? 1 : 0};
    CellIn<double> ci;
    taumol_g<double>(ib, igb, 1, C, tab, ci.taug, ci.taur);
    aerosol_in(P, col, lay, ib, tab, ci);
    cloud_in<double>(P, col, g, lay, ib, P.fused && P.icld >= 1, cloudy, nullptr, ci, tab);
    const CellOpt<double> o = cell_optics<double>(ci, 1, cossza, tab, tab, 0.0f);
    c.ref = o.rc.ref; c.refd = o.rc.refd; c.tdif = o.rc.tra - o.zdbtc; c.trad = o.rc.trad; c.dbt = o.zdbtc;
    t.ref = o.rt.ref; t.refd = o.rt.refd; t.tdif = o.rt.tra - o.zdbt; t.trad = o.rt.trad; t.dbt = o.zdbt;
}

// Layer optics of one (g-point, layer) cell (rrtmg_sw_spcvmc.f90:442-585):
// clear sky c and total sky t.  dbtn: idelm = 0's unscaled direct
// transmittance of the total sky.  `cld`, `aer`: the prepared optics of this
// (column, layer), [band][..].
__device__ __forceinline__ void cell64(const SolveParams& P, const TmSmem* sTm, const double* blk, const double* cld,
                                       const double* aer, bool low, int col, int g, int lay, int ib, int igb,
                                       int mode, bool mask, const Mu64& m, const double* __restrict__ tab, Rt64& c,
                                       Rt64& t, double& dbtn) {
    double taug, taur;
    taumol64(sTm[ib * 2 + (low ? 0 : 1)], ib, igb, blk, tab, taug, taur);
    double tau = taur + taug, s = taur, sg = 0.0, ab = taug;
    bool near = false;
    double tau0 = tau;
    if (P.iaer != 0) {
        const double* a = aer + ib * AO_N;
        tau0 = tau += a[AO_TAU];
        s += a[AO_S];
        sg = a[AO_SG];
        ab += a[AO_AB];
        // delta scaling (spcvmc:492-496): f = g^2 moves w f tau = sg^2 / s into the direct beam
        const double d = sg * sg * rcp64(s);
        tau -= d;
        s -= d;
        sg -= d;
        c = two_stream64<true>(tau, s, sg, ab, m, tab, near);
    } else {
        c = two_stream64<false>(tau, s, sg, ab, m, tab, near);
    }
    t = c;
    double om;
    if (P.idelm == 0) dbtn = tbl_exp64(clip500(tau0 * m.rmu), tab, om);
    bool cloudy = false;
    if (mode != CLD_NONE) {
        double loc[CO_N];
        const double* o = cld + ib * CO_N;
        double cf = 1.0;
        const size_t n = (size_t)P.ncol;
        if (mode == CLD_MASK) {
            cloudy = mask;
        } else if (mode == CLD_LAYER) {
            cf = P.cldfrac[(size_t)col + n * (size_t)(lay - 1)];
            cloudy = cf != 0.0;
        } else {
            const size_t kl = (size_t)col + n * (size_t)(lay - 1), kg = (size_t)g + NGPT * kl;
            cf = P.cldfmcl[kg];
            cloudy = cf != 0.0;
            if (cloudy) {
                cloud64(ib, P.inflag, P.iceflag, P.liqflag, cf, P.ciwpmcl[kg], P.clwpmcl[kg], P.reicmcl[kl],
                        P.relqmcl[kl], P.fsfcmcl[kg], P.taucmcl[kg], P.ssacmcl[kg], P.asmcmcl[kg], tab, -1.0, loc);
                o = loc;
            }
        }
        if (cloudy) {
            if (__double_as_longlong(o[CO_ERR]) != 0ll) set_error(P.err, (int)o[CO_ERR]);
            // total sky: clear + delta-scaled cloud (spcvmc:500-505); reftra
            // only where cldf > repclc (:427); mixed by cloud fraction (:546-549)
            const double to = tau + o[CO_TAU];
            if (cf > 1.e-12) {
                t = two_stream64<true>(to, s + o[CO_S], sg + o[CO_SG], ab + o[CO_AB], m, tab, near);
            } else {
                t.ref = 0.0; t.refd = 0.0; t.trad = 1.0;
                t.dbt = tbl_exp64(clip500(to * m.rmu), tab, om);
                t.tdif = 1.0 - t.dbt;
            }
            double bo = 0.0;
            if (P.idelm == 0) bo = tbl_exp64(clip500((tau0 + o[CO_TAOR]) * m.rmu), tab, om);
            if (cf != 1.0) {
                const double z = 1.0 - cf;
                t.ref = fma(cf, t.ref, z * c.ref);
                t.refd = fma(cf, t.refd, z * c.refd);
                t.tdif = fma(cf, t.tdif, z * c.tdif);
                t.trad = fma(cf, t.trad, z * c.trad);
                t.dbt = fma(cf, t.dbt, z * c.dbt);
                bo = fma(cf, bo, z * dbtn);
            }
            dbtn = bo;
        }
    }
    if (near) cell_ref64(P, blk, low, col, g, lay, ib, igb, cloudy, m.mu, tab, c, t);
}

// Upward adding through one layer (vrtqdr:122-140): on entry the albedos
// below it, on exit those at its top; alpha, beta: the diffuse flux below the
// layer per direct and diffuse flux above it.  (The flux up through the
// lower face is rup dbt dir + rupd dif, so dif = tdif dir + trad dif_above +
// refd (rup dbt dir + rupd dif), solved for dif.)
__device__ __forceinline__ void up64(const Rt64& r, double& rup, double& rupd, double& alpha, double& beta) {
    const double zr = rcp64(fma(-rupd, r.refd, 1.0));
    const double x = r.dbt * rup;
    beta = r.trad * zr;
    alpha = fma(r.refd, x, r.tdif) * zr;
    rup = fma(beta, fma(r.tdif, rupd, x), r.ref);
    rupd = fma(beta, r.trad * rupd, r.refd);
}

// ------------------------------------------------------------ preparation
// McICA thresholds of one (column, layer): those of 1 - cldf and of alpha as
// integers (kiss_threshold / mt_threshold), 1 - cldf itself.
enum { TH_KC, TH_KA, TH_OMCF, TH_N };
template <bool MT>
__device__ inline void thresholds64(const SolveParams& P, int pcol, int lay, double* th) {
    const bool real = pcol < P.ncol;
    const size_t kl = (size_t)pcol + (size_t)P.ncol * (size_t)(lay - 1);
    double cf = real ? P.cldfrac[kl] : 0.0;
    if (cf < 1.0e-20) cf = 0.0;
    const double omcf = DS(1.0, cf);
    const double al = P.icld >= 4 && real ? P.alpha[kl] : 0.0;
    long long kc, ka = 0;
    if constexpr (MT) {
        kc = mt_threshold(omcf);
        if (P.icld >= 4 && real) ka = mt_threshold(al);
    } else {
        kc = kiss_threshold(omcf);
        if (P.icld >= 4 && real) ka = kiss_threshold(al);
    }
    th[TH_KC] = __longlong_as_double(kc);
    th[TH_KA] = __longlong_as_double(ka);
    th[TH_OMCF] = omcf;
}

// KISS seeds of one column (mcica_subcol_gen_sw.f90:475-478)
__device__ inline void seeds64(const SolveParams& P, int pcol, uint32_t* seed) {
    const size_t n = (size_t)P.ncol;
    const double p1 = DM(P.play[pcol], 1.e2), p2 = DM(P.play[pcol + n], 1.e2);
    if (p1 < p2) set_error(P.err, E_KISSSEED);
    seed[0] = kiss_seed(p1);
    seed[1] = kiss_seed(p2);
    seed[2] = kiss_seed(DM(P.play[pcol + 2 * n], 1.e2));
    seed[3] = kiss_seed(DM(P.play[pcol + 3 * n], 1.e2));
}

// setcoef of one (column, layer) into its block; returns the packed indices
__device__ inline int setcoef64(const SolveParams& P, int pcol, int lay, double* blk, const double* __restrict__ tab) {
    double pdp;
    int* pk = (int*)(blk + B_PK);
    prep_layer<double>(P, pcol, lay, blk, pk, &pdp, 1, tab, nullptr, 0);
    if (P.nomcica && P.icld >= 1 && pcol < P.ncol) {
        // spcvrt_sw takes clear or overcast layers only (rrtmg_sw_rad.nomcica.f90:617-621)
        const double cf = P.cldfrac[(size_t)pcol + (size_t)P.ncol * (size_t)(lay - 1)];
        if (cf > 1.e-6 && cf < 1.0 - 1.e-6) set_error(P.err, E_PARTIAL);
    }
    return *pk;
}

// The band items of one (column, layer, band): the k-table's column amount
// and species ratio (e.g. rrtmg_sw_taumol.f90:309-324), cloud and aerosol
// optics.  cld / aer: this (column, layer)'s [band][..], or unused.
__device__ inline void prep_band64(const SolveParams& P, int pcol, int lay, int b, bool low, double* blk, double* cld,
                                   double* aer, int mode, bool always, const double* __restrict__ tab) {
    const int up = low ? 0 : 1;
    const TmRegion& d = cT.tm[b][up];
    if (d.kind == 1) {
        const double ca = blk[F_H2O + d.sa];
        const double comb = ca + cT.strrat64[b][up] * blk[F_H2O + d.sb];
        double p = ca / comb;
        if (p >= cT.oneminus) p = cT.oneminus;
        const double sm = (up ? 4.0 : 8.0) * p;
        const int js = (int)sm;
        blk[B_COMB + b] = comb;
        blk[B_FS + cT.sslot[b]] = sm - (double)js;
        ((unsigned char*)(blk + B_JS))[cT.sslot[b]] = (unsigned char)js;
    } else {
        blk[B_COMB + b] = d.kind == 2 ? blk[F_H2O + d.sa] * cT.fac64[b][up] : 0.0;
    }
    const size_t n = (size_t)P.ncol, kl = (size_t)pcol + n * (size_t)(lay - 1), kb = (size_t)b + 14 * kl;
    if (mode == CLD_MASK) {
        // a clear layer has no cloudy subcolumn (KISS draws stay below 1; an
        // MT draw can equal 1, so `always`)
        const double cf = P.cldfrac[kl];
        if (cf > 0.0 || always) {
            const bool in = P.tauc != nullptr;
            cloud64(b, P.inflag, P.iceflag, P.liqflag, 1.0, P.ciwp[kl], P.clwp[kl], P.rei[kl], P.rel[kl],
                    in ? P.fsfc[kb] : 0.0, in ? P.tauc[kb] : 0.0, in ? P.ssac[kb] : 1.0, in ? P.asmc[kb] : 0.0, tab,
                    -1.0, cld + b * CO_N);
        }
    } else if (mode == CLD_LAYER) {
        // cldprop_sw (rrtmg_sw_cldprop.f90:140-370)
        const double cf = P.cldfrac[kl];
        if (cf != 0.0) {
            const bool in = P.tauc != nullptr;
            double tot = 0.0;
            if (in)
                for (int i = 0; i < NBND; ++i) tot += P.tauc[(size_t)i + 14 * kl];
            const double cwp = P.ciwp[kl] + P.clwp[kl];
            const bool on = cf >= 1.e-20 && (cwp >= 1.e-20 || tot >= 1.e-20) && (P.inflag == 0 || P.inflag == 2);
            const double tin = in ? P.tauc[kb] : 0.0;
            double* c = cld + b * CO_N;
            if (on) {
                cloud64(b, P.inflag, P.iceflag, P.liqflag, cf, P.ciwp[kl], P.clwp[kl], P.rei[kl], P.rel[kl],
                        in ? P.fsfc[kb] : 0.0, tin, in ? P.ssac[kb] : 1.0, in ? P.asmc[kb] : 0.0, tab, tot, c);
            } else {
                c[CO_TAU] = c[CO_S] = c[CO_SG] = c[CO_AB] = c[CO_ERR] = 0.0;
                c[CO_TAOR] = tin;
            }
        }
    }
    if (P.iaer != 0) {
        double ta, oa, ga;
        aerosol(P, pcol, lay, b, tab, ta, oa, ga);
        double* a = aer + b * AO_N;
        const double sc = ta * oa;
        a[AO_TAU] = ta;
        a[AO_S] = sc;
        a[AO_SG] = sc * ga;
        a[AO_AB] = ta * (1.0 - oa);
    }
}

// Solar source of g-point igb of band ib at its reference layer (the
// laysolfr logic of taumol16..29, e.g. taumol.f90:364-378 and 495-517); blk0:
// the column's block of layer 1 (blocks `stride` apart); pk: its layers'
// packed indices.  For the adjoint also the reference layer and the source's
// derivative along the species ratio fs (0 where it is not interpolated).
__device__ inline double solar64(int ib, int igb, const double* blk0, int stride, const int* pk, int L, int laytrop,
                                 const SolveParams& P, const double* __restrict__ tab, int* lsol = nullptr,
                                 double* dfs = nullptr) {
    const int lref[14] = {18, 30, 6, 3, 3, 8, 2, 6, 1, 2, 0, 32, 42, 49};
    const int layreffr = lref[ib], band = ib + 16;
    auto jp = [&](int lay) { return pk[lay - 1] & 0xff; };
    const int lt = laytrop;
    int src = -1;
    if (band == 16 || band == 17 || band == 27 || band == 28 || band == 29) {
        int at = L, prev = jp(lt);
        for (int lay = lt + 1; lay <= L; ++lay) {
            const int cur = jp(lay);
            if (prev < layreffr && cur >= layreffr) at = lay;
            if (lay == at) src = lay;
            prev = cur;
        }
    } else if (band == 26) {
        src = lt;
    } else {
        int at = lt, cur = jp(1);
        for (int lay = 1; lay <= lt; ++lay) {
            const int nxt = lay + 1 <= L ? jp(lay + 1) : -1000;
            if (cur < layreffr && nxt >= layreffr) at = min(lay + 1, lt);
            if (lay == at) src = lay;
            cur = nxt;
        }
    }
    const BandOff& B = cT.b[ib];
    // the species interpolation of bands 17-19, 21, 22, 24, 28: their
    // source layer lies in the region whose ratio the block holds
    bool interp = false;
    double fs = 0.0;
    int js = 0;
    if (src >= 1 && cT.sslot[ib] >= 1) {
        const double* blk = blk0 + (size_t)(src - 1) * stride;
        fs = blk[B_FS + cT.sslot[ib]];
        js = ((const unsigned char*)(blk + B_JS))[cT.sslot[ib]];
        interp = true;
    }
    double slope = 0.0;
    auto val = [&](int off, double weight) -> double {
        const double a = ldt(tab, off + js * B.ng + igb - 1);
        if (!interp) return weight * a;
        const double b = ldt(tab, off + (js + 1) * B.ng + igb - 1);
        slope += weight * (b - a);
        return weight * (a + fs * (b - a));
    };
    double v;
    if (P.isolvar < 0)
        v = val(B.sfluxref, band == 27 ? 50.15 / 48.37 : 1.0);
    else
        v = val(B.facbrght, P.svar_f_bnd[ib]) + val(B.snsptdrk, P.svar_s_bnd[ib]) + val(B.irradnce, P.svar_i_bnd[ib]);
    if (lsol) *lsol = src;
    if (dfs) *dfs = slope;
    return v;
}

// Cloud mask of one subcolumn, bottom to top.  KISS with icld = 2 rescales
// its distribution in FP64 only where a layer has cloud: where the layer
// below is clear the rescaling multiplies by 1, and a clear layer is never
// cloudy (draws stay below 1).
template <bool MT>
struct Mask64 {
    McicaMask<MT> m;
    __device__ __forceinline__ bool step(int lay, const double* th) {
        if constexpr (!MT) {
            if (m.icld == 2) {
                const int32_t d = m.k.next_int();
                const double omcf = th[TH_OMCF];
                if (__double_as_longlong(omcf) == __double_as_longlong(1.0)) {
                    m.omcf_prev = 1.0;
                    m.cdf_prev = 0.0;
                    return false;
                }
                double cdf = kiss_real(d);
                if (lay >= 2) {
                    if (m.cdf_prev > m.omcf_prev) cdf = m.cdf_prev;
                    else cdf = __dmul_rn(cdf, m.omcf_prev);
                }
                m.cdf_prev = cdf;
                m.omcf_prev = omcf;
                return cdf >= omcf;
            }
        }
        return m.step(lay, __double_as_longlong(th[TH_KC]), __double_as_longlong(th[TH_KA]), th[TH_OMCF]);
    }
};

}  // namespace rrsw
