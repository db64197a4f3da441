// fp64.cuh -- the plain FP64 form of the column solve.
//
// GB300 runs FP64 at 1/64 of its FP32 rate (two FP64 lanes per SM and
// cycle), so this form is bound by the FP64 pipe alone: an FP64 warp
// instruction holds it for 16 cycles, while integer, FP32 and memory
// instructions run beside it for next to nothing.  Everything here is
// written to issue few FP64 instructions per (g-point, layer) cell:
//
//   - no IEEE division or square root per cell: rcp64 / sqrt64 start from
//     the hardware's approximation and take one third-order step (3 and 5
//     FP64 instructions, within an ulp) instead of a division sequence;
//   - explicit fma() (the unit is compiled without contraction, so every
//     kernel that inlines these functions rounds alike, bit for bit);
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
// About 170 FP64 instructions per cell (with aerosol) where the reference's
// order of operations took about 570: 16 384 x 60 columns with clouds and
// aerosol 102.9 -> 37.6 ms, 1 024 x 60 clear 7.04 -> 2.34 ms, the FP64 pipe 84 %
// busy.  The layer solution is also written without the cancellation of
// thin layers: against a solve in 80-bit arithmetic the heating rates of
// 1 024 x 60 clear columns are 8.6e-11 off (2-norm), 1.04e-10 in the
// reference's order.  Cells near the two-stream resonance k mu0 = 1, where the
// reference divides rounding by a small number, keep its order (cell_ref64).
#pragma once

#include "kernel.cuh"

namespace rrsw {

// ------------------------------------------------------------ arithmetic
// 1/x for finite normal x: the hardware's approximation r (relative error e,
// |e| < 2^-19) and one third-order step r (1 + e + e^2), error below an ulp.
__device__ __forceinline__ double rcp64(double x) {
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    const double e = fma(-x, r, 1.0);
    return fma(r, fma(e, e, e), r);
}

// sqrt(x) for positive normal x: y ~ x^-1/2 from the hardware, e = 1 - x y^2,
// sqrt(x) = x y (1 + e/2 + 3 e^2 / 8), error below an ulp.
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

// g-point sums kept per level: fu, fd, cu, cd, and the direct total flux when
// an output needs it; with the extra outputs fd and the direct flux are
// also summed over the UV (bands 25-28) and the other bands.
constexpr int KLEV64 = 4;
__host__ __device__ constexpr int klev64(int nc) { return nc > 2 ? KLEV64 / 2 : KLEV64; }
__host__ __device__ inline int num_q64(const SolveParams& P) { return P.extra || P.bands ? 5 : 4; }
__host__ __device__ inline int num_sum64(const SolveParams& P) { return P.extra ? 9 : num_q64(P); }

struct Smem64 {
    size_t tm, xs, seed, misc, jp, red, flux, total;
};
__host__ __device__ inline Smem64 smem64(const SolveParams& P, int nc) {
    Smem64 m;
    size_t o = 0;
    m.tm = o;   o = align16(o + NBND * 2 * sizeof(TmSmem));
    m.xs = o;   if (P.fused && P.icld >= 1) o = align16(o + NGPT * 32 * sizeof(uint32_t));
    m.seed = o; o = align16(o + nc * 4 * sizeof(uint32_t));
    m.misc = o; o = align16(o + nc * sizeof(int));
    m.jp = o;   o = align16(o + (size_t)nc * P.nlay * sizeof(int));
    m.red = o;  o = align16(o + (size_t)klev64(nc) * num_q64(P) * nc * NGPT * sizeof(double));
    m.flux = o; o = align16(o + (size_t)nc * num_sum64(P) * (P.nlay + 1) * sizeof(double));
    m.total = o;
    return m;
}

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
    const double sum = fma(-0.5, w, fma(-1.5, wg, 2.0));  // gamma1 + gamma2
    const double g1 = fma(0.5, sum, co);
    const double g2 = fma(0.5, sum, -co);
    const double co2 = co + co;
    const double k = sqrt64(co2 * sum);
    const double a1 = fma(g2, g3, g1 * g4);
    const double a2 = fma(g1, g3, g2 * g4);
    const double kmu = k * m.mu;
    const double p1 = 1.0 + kmu, m1 = 1.0 - kmu;
    const double pp = p1 * m1;  // 1 - (k mu0)^2
    double om1;
    const double e1 = tbl_exp64(clip500(k * tau), tab, om1);
    const double ee = e1 * e1, oo = om1 * (1.0 + e1);  // exp(-2 k tau) and 1 less it
    const double B = fma(g1, oo, fma(k, ee, k));
    const double pB = pp * B;  // zdenr zem1
    // (or |zdenr| <= 1e-8, where the reference replaces the solution)
    if (lt_pos(fabs(pp), RESONANCE64 * w) || lt_pos(fabs(pB), 1.1e-8)) near = true;
    const double r = rcp64(pB);
    const double rB = r * pp;        // 1 / B
    const double k2 = k + k;
    const double r2 = p1 * fma(-k, g3, a2), r3 = k2 * fma(-a2, m.mu, g3);
    const double t2 = m1 * fma(-k, g4, a1), t3 = k2 * fma(a1, m.mu, g4);
    const double wr = w * r;
    // zr1 - zr2 ee - zr3 e1 e2 and zt3 e1 - e2 (zt1 - zt2 ee) with
    // zr1 = zr2 + zr3 and zt1 = zt2 + zt3: no cancellation in thin layers
    o.ref = wr * fma(r2, oo, r3 * fma(e1, om2, om1));
    o.tdif = wr * fma(t3, om2 - om1, -e2 * (t2 * oo));
    o.refd = g2 * oo * rB;
    o.trad = k2 * e1 * rB;
    return o;
}

// ----------------------------------------------------------------- clouds
// Cloud optics of a layer in band ib (cldprmc_sw, rrtmg_sw_cldprmc.f90:53-349;
// with ttest >= 0 cldprop_sw's test) in the form two_stream64 takes.  The
// error code of an input out of range is returned in c[CO_ERR]: it counts
// only where a cloudy subcolumn meets it.
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
        if (rei < 13.0 || rei > 130.0) { err = E_ICERAD; out(); return; }
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
        if (rei < 5.0 || rei > 131.0) { err = E_ICERAD; out(); return; }
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
        if (rei < 5.0 || rei > 140.0) { err = E_ICEDGE; out(); return; }
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
        if (rel < 2.5 || rel > 60.0) { err = E_LIQRAD; out(); return; }
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
// the column's block of layer 1; pk: its layers' packed indices.
__device__ inline double solar64(int ib, int igb, const double* blk0, const int* pk, int L, int laytrop,
                                 const SolveParams& P, const double* __restrict__ tab) {
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
        const double* blk = blk0 + (size_t)(src - 1) * B_STRIDE;
        fs = blk[B_FS + cT.sslot[ib]];
        js = ((const unsigned char*)(blk + B_JS))[cT.sslot[ib]];
        interp = true;
    }
    auto val = [&](int off) -> double {
        const double a = ldt(tab, off + js * B.ng + igb - 1);
        if (!interp) return a;
        const double b = ldt(tab, off + (js + 1) * B.ng + igb - 1);
        return a + fs * (b - a);
    };
    if (P.isolvar < 0) {
        const double sf = val(B.sfluxref);
        return band == 27 ? (50.15 / 48.37) * sf : sf;
    }
    return P.svar_f_bnd[ib] * val(B.facbrght) + P.svar_s_bnd[ib] * val(B.snsptdrk) + P.svar_i_bnd[ib] * val(B.irradnce);
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

// ---------------------------------------------------------- sums, outputs
// The g-point sums of nlev buffered levels (fixed order: four runs of 28
// g-points, then the runs); red [level][q][NT], flux [column][sum][L + 1].
// qd: the buffered direct flux's place.  With nsum > qd + 1 the last four sums
// are the UV (bands 25-28) and other bands' parts of q 1 and of the direct flux.
// NTH: the CTA's threads (whole warps).
__device__ __forceinline__ void sum_levels64(const SolveParams& P, const double* red, double* flux, int NC, int NT,
                                             int NTH, int nq, int nsum, int qd, int jk, int nlev) {
    const int L = P.nlay, tid = threadIdx.x;
    const int items = NC * nsum * nlev;
    for (int base = 0; base < items * 4; base += NTH) {
        const int t = base + tid, item = t >> 2, part = t & 3;
        double v = 0.0;
        int c2 = 0, qi = 0, s = 0;
        if (item < items) {
            c2 = item / (nsum * nlev);
            qi = (item / nlev) % nsum;
            s = item % nlev;
            // past the direct flux: UV fd, UV direct, other fd, other direct
            const int x = qi - qd - 1;
            const int q = x < 0 ? qi : (x & 1) ? qd : 1;
            const double* src = red + ((size_t)s * nq + q) * NT + c2 * NGPT + part * 28;
            if (x < 0) {
#pragma unroll 4
                for (int j = 0; j < 28; ++j) v += src[j];
            } else {
                const int u0 = cT.b[9].g0 - part * 28, u1 = cT.b[13].g0 - part * 28;
                for (int j = 0; j < 28; ++j)
                    if ((j >= u0 && j < u1) == (x < 2)) v += src[j];
            }
        }
        warp_sum4(v);
        if (item < items && part == 0) flux[((size_t)c2 * nsum + qi) * (L + 1) + (L + 1 - (jk - (nlev - 1) + s))] = v;
    }
}

// Per-band sums of one buffered quantity into an output array (spcvmc:619-630 per band)
__device__ __forceinline__ void band_levels64(const SolveParams& P, const double* red, int NC, int NT, int NTH, int nq,
                                              int q, double* out, int group, int nmapped, int jk, int nlev) {
    if (!out) return;
    const int L = P.nlay;
    for (int t = threadIdx.x; t < NC * NBND * nlev; t += NTH) {
        const int s = t % nlev, b = (t / nlev) % NBND, c2 = t / (nlev * NBND);
        const int ocol = pair_col(P, group, c2, nmapped, NC);
        if (ocol >= P.ncol) continue;
        const double* src = red + ((size_t)s * nq + q) * NT + c2 * NGPT + cT.b[b].g0;
        double v = 0.0;
        for (int j = 0; j < cT.b[b].ng; ++j) v += src[j];
        const int l = L + 1 - (jk - (nlev - 1) + s);  // level index, 0 = surface
        out[(size_t)ocol + (size_t)P.ncol * ((size_t)l + (size_t)(L + 1) * b)] = v;
    }
}

// Outputs of one sky (rrtmg_sw_rad.f90:805-836) from the level sums of NC
// columns; qu: the sums' up flux (down: qu + 1), qd: the direct flux (with the
// UV and other parts behind it) when extra.
__device__ __forceinline__ void write_sky64(const SolveParams& P, const double* flux, int NC, int NTH, int nsum,
                                            int qu, int qd, bool extra, int group, int nmapped, double* up,
                                            double* dn, double* hr) {
    const int L = P.nlay;
    const size_t n = (size_t)P.ncol;
    for (int it = threadIdx.x; it < NC * (L + 1); it += NTH) {
        const int c2 = it / (L + 1), l = it % (L + 1);
        const int ocol = pair_col(P, group, c2, nmapped, NC);
        if (ocol >= P.ncol) continue;
        const double* F = flux + (size_t)c2 * nsum * (L + 1);
        const size_t o = (size_t)ocol + n * (size_t)l;
        const double fu = F[qu * (L + 1) + l], fd = F[(qu + 1) * (L + 1) + l];
        up[o] = fu;
        dn[o] = fd;
        if (l < L) {
            double h = 0.0;
            if (l < L - 1) {
                const double z = cT.heatfac / DS(P.plev[o], P.plev[o + n]);
                const double fu1 = F[qu * (L + 1) + l + 1], fd1 = F[(qu + 1) * (L + 1) + l + 1];
                h = DM(DS(DS(fd1, fu1), DS(fd, fu)), z);
            }
            hr[o] = h;
        }
        if (extra) {
            const double* D = F + qd * (L + 1) + l;
            const double dir = D[0], uvd = D[L + 1], uvr = D[2 * (L + 1)], nid = D[3 * (L + 1)], nir = D[4 * (L + 1)];
            const double vals[8] = {dir, DS(fd, dir), uvd, nid, uvr, DS(uvd, uvr), nir, DS(nid, nir)};
            for (int x = 0; x < 8; ++x)
                if (P.xout[x]) P.xout[x][o] = vals[x];
        }
    }
}

// ------------------------------------------------------------ fused solve
struct View64 {
    const TmSmem* tm;
    uint32_t* xs;
    uint32_t* seed;
    int* misc;
    int* jp;  // [nc][L] setcoef's packed indices
    double* red;
    double* flux;
};

__device__ inline View64 view64(unsigned char* raw, const SolveParams& P, int nc) {
    const Smem64 M = smem64(P, nc);
    View64 v;
    v.tm = (const TmSmem*)(raw + M.tm);
    v.xs = (uint32_t*)(raw + M.xs);
    v.seed = (uint32_t*)(raw + M.seed);
    v.misc = (int*)(raw + M.misc);
    v.jp = (int*)(raw + M.jp);
    v.red = (double*)(raw + M.red);
    v.flux = (double*)(raw + M.flux);
    return v;
}

// One group of NC columns, NC x 112 threads: preparation, cells and up-sweep
// bottom to top, down-sweep with the level sums, outputs.  `slot`: the CTA's
// scratch (slot64).
template <bool MT, int NC>
__device__ __forceinline__ void solve_group64(const SolveParams& P, int group, const View64& V, const KissJump& J,
                                              double* slot, const double* __restrict__ tab) {
    constexpr int NT = NC * NGPT;
    const int L = P.nlay, tid = threadIdx.x;
    const int cc = tid / NGPT, g = tid % NGPT;
    const int ib = cT.ngb[g], igb = cT.gib[g];
    const int mode = cloud_mode(P);
    const int nmapped = P.colmap ? *P.mapcount : 0;
    const int NF = fields64(P.idelm);
    const Slot64 S = slot64(L, P.idelm, NC, band_clouds(P), P.iaer != 0);
    double* blk0 = slot + S.blk;
    double* cld0 = slot + S.cld;
    double* aer0 = slot + S.aer;
    __syncthreads();  // the previous group is finished
    if (tid < NC) V.misc[tid] = 0;
    __syncthreads();
    for (int it = tid; it < NC * L; it += NT) {
        const int c2 = it / L, lay = it % L + 1;
        const int pcol = pair_col(P, group, c2, nmapped, NC);
        double* blk = blk0 + (size_t)it * B_STRIDE;
        const int pk = setcoef64(P, pcol, lay, blk, tab);
        V.jp[it] = pk;
        if ((pk >> 30) & 1) atomicAdd(V.misc + c2, 1);
        if (mode == CLD_MASK) {
            thresholds64<MT>(P, pcol, lay, blk + B_TH);
            if (!MT && lay == 1 && pcol < P.ncol) seeds64(P, pcol, V.seed + c2 * 4);
        }
    }
    __syncthreads();
    for (int it = tid; it < NC * L * NBND; it += NT) {
        const int b = it % NBND, cl = it / NBND, c2 = cl / L, lay = cl % L + 1;
        const int pcol = pair_col(P, group, c2, nmapped, NC);
        if (pcol < P.ncol)
            prep_band64(P, pcol, lay, b, lay <= V.misc[c2], blk0 + (size_t)cl * B_STRIDE,
                        cld0 + (size_t)cl * NBND * CO_N, aer0 + (size_t)cl * NBND * AO_N, mode, MT, tab);
    }
    __syncthreads();
    const int col = pair_col(P, group, cc, nmapped, NC);
    const int laytrop = V.misc[cc];
    bool active = col < P.ncol;
    if (active && (laytrop < 1 || laytrop >= L)) {
        set_error(P.err, E_LAYTROP);
        active = false;
    }
    double zinc = 0.0, albp = 0.0, albd = 0.0;
    double* sv0 = slot + tid;
    const double* blkc = blk0 + (size_t)cc * L * B_STRIDE;
    if (active) {
        Mu64 m;
        m.mu = P.coszen[col];
        if (m.mu < 1.e-10) m.mu = 1.e-10;
        m.rmu = 1.0 / m.mu;
        m.mu34 = 0.75 * m.mu;
        const bool nir = ib <= 8 || ib == 13;
        albp = nir ? P.aldir[col] : P.asdir[col];
        albd = nir ? P.aldif[col] : P.asdif[col];
        // zincflx = adjflux * ssi * prmu0 (spcvmc:349-356)
        zinc = P.adjflux[ib] * solar64(ib, igb, blkc, V.jp + cc * L, L, laytrop, P, tab) * m.mu;
        Mask64<MT> mc;
        if (mode == CLD_MASK)
            mc.m.start(kiss_start(V.seed + cc * 4, J, V.xs + g * 32), P.icld,
                       MT ? P.mt + mt_offset(P.icld, g, col, P.ncol, L) : nullptr);
        double rc = albp, rcd = albd, rt = albp, rtd = albd;
#pragma unroll 1
        for (int lay = 1; lay <= L; ++lay) {
            const double* blk = blkc + (size_t)(lay - 1) * B_STRIDE;
            const bool mask = mode == CLD_MASK && mc.step(lay, blk + B_TH);
            Rt64 c, t;
            double dbtn = 1.0, alpha, beta;
            cell64(P, V.tm, blk, cld0 + (size_t)(cc * L + lay - 1) * NBND * CO_N,
                   aer0 + (size_t)(cc * L + lay - 1) * NBND * AO_N, lay <= laytrop, col, g, lay, ib, igb, mode, mask,
                   m, tab, c, t, dbtn);
            double* sv = sv0 + (size_t)(L - lay) * NF * NT;
            up64(c, rc, rcd, alpha, beta);
            sv[L_RUP * NT] = rc;
            sv[L_RUPD * NT] = rcd;
            sv[L_ALPHA * NT] = alpha;
            sv[L_BETA * NT] = beta;
            sv[L_DBT * NT] = c.dbt;
            if (mode != CLD_NONE) {
                up64(t, rt, rtd, alpha, beta);
                sv[(L_SKY + L_RUP) * NT] = rt;
                sv[(L_SKY + L_RUPD) * NT] = rtd;
                sv[(L_SKY + L_ALPHA) * NT] = alpha;
                sv[(L_SKY + L_BETA) * NT] = beta;
                sv[(L_SKY + L_DBT) * NT] = t.dbt;
            }
            if (P.idelm == 0) sv[2 * L_SKY * NT] = dbtn;
        }
    }
    // down-sweep: direct and diffuse flux, weighted with the incident flux
    const int nq = num_q64(P), nsum = num_sum64(P);
    constexpr int KL = klev64(NC);
    double dc = zinc, fc = 0.0, dt = zinc, ft = 0.0, dn = zinc;
    const bool tot = mode != CLD_NONE;
    for (int jk = 1; jk <= L + 1; ++jk) {
        double cu = 0.0, cd = 0.0, fu = 0.0, fd = 0.0, dir = 0.0;
        if (active) {
            if (jk <= L) {
                const double* sv = sv0 + (size_t)(jk - 1) * NF * NT;
                if (jk < L) {
                    const double* nx = sv + (size_t)NF * NT;
#pragma unroll
                    for (int f = 0; f < 2 * L_SKY; ++f) asm volatile("prefetch.global.L1 [%0];" ::"l"(nx + f * NT));
                }
                cu = fma(sv[L_RUP * NT], dc, sv[L_RUPD * NT] * fc);
                cd = dc + fc;
                fc = fma(sv[L_ALPHA * NT], dc, sv[L_BETA * NT] * fc);
                dc *= sv[L_DBT * NT];
                if (tot) {
                    dir = dt;
                    fu = fma(sv[(L_SKY + L_RUP) * NT], dt, sv[(L_SKY + L_RUPD) * NT] * ft);
                    fd = dt + ft;
                    ft = fma(sv[(L_SKY + L_ALPHA) * NT], dt, sv[(L_SKY + L_BETA) * NT] * ft);
                    dt *= sv[(L_SKY + L_DBT) * NT];
                } else {
                    dir = dt;
                    dt = dc;
                }
                if (P.idelm == 0) {
                    dir = dn;
                    dn *= sv[2 * L_SKY * NT];
                }
            } else {
                cu = fma(albp, dc, albd * fc);
                cd = dc + fc;
                fu = fma(albp, dt, albd * ft);
                fd = dt + ft;
                dir = P.idelm == 0 ? dn : dt;
            }
            if (!tot) {
                fu = cu;
                fd = cd;
            }
        }
        const int s = (jk - 1) % KL;
        double* red = V.red + (size_t)s * nq * NT + tid;
        red[0] = fu;
        red[NT] = fd;
        red[2 * NT] = cu;
        red[3 * NT] = cd;
        if (nq > 4) red[4 * NT] = dir;
        if (s == KL - 1 || jk == L + 1) {
            __syncthreads();
            sum_levels64(P, V.red, V.flux, NC, NT, NT, nq, nsum, 4, jk, s + 1);
            if (P.bands) {
                const int qs[5] = {0, 1, 4, 2, 3};  // fu, fd, direct, cu, cd
                for (int k = 0; k < 5; ++k)
                    band_levels64(P, V.red, NC, NT, NT, nq, qs[k], P.bout[k], group, nmapped, jk, s + 1);
            }
            __syncthreads();
        }
    }
    write_sky64(P, V.flux, NC, NT, nsum, 0, 4, P.extra != 0, group, nmapped, P.swuflx, P.swdflx, P.swhr);
    write_sky64(P, V.flux, NC, NT, nsum, 2, 4, false, group, nmapped, P.swuflxc, P.swdflxc, P.swhrc);
}

template <bool MT>
__global__ void __launch_bounds__(CTA_THREADS, 2)
k_solve64(const SolveParams P, const double* __restrict__ tab) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const View64 V = view64(smem_raw, P, COLS_PER_CTA);
    fill_tm64((TmSmem*)V.tm);
    KissJump J{1u, 0u, 1u, 1u};
    if (!MT) J = kiss_setup(P, V.xs, threadIdx.x % NGPT);  // once per launch
    double* slot = (double*)P.scratch + (size_t)blockIdx.x * P.slot_elems;
    for (int pair = blockIdx.x; pair < P.npairs; pair += gridDim.x)
        solve_group64<MT, COLS_PER_CTA>(P, pair, V, J, slot, tab);
}

// The batch kernel (kernel.cuh, k_solve_batch) of this form.
template <int NC>
__global__ void __launch_bounds__(NC * NGPT, 4 / NC)
k_solve64_batch(const SolveParams* __restrict__ Pb, int ninst, const int* __restrict__ counts,
                const double* __restrict__ tab) {
    constexpr int NT = NC * NGPT;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int s_pref[MAX_BATCH + 1];
    __shared__ __align__(16) SolveParams sP;
    fill_tm64((TmSmem*)smem_raw);  // offset 0 in every instance's layout
    if (threadIdx.x == 0) {
        s_pref[0] = 0;
        for (int i = 0; i < ninst; ++i) s_pref[i + 1] = s_pref[i] + (counts[i] + NC - 1) / NC;
    }
    __syncthreads();
    const int total = s_pref[ninst];
    int cur = -1;
    View64 V{};
    KissJump J{1u, 0u, 1u, 1u};
    for (int item = blockIdx.x; item < total; item += gridDim.x) {
        int lo = 0, hi = ninst;
        while (hi - lo > 1) {
            const int mid = (lo + hi) / 2;
            if (s_pref[mid] <= item) lo = mid;
            else hi = mid;
        }
        if (lo != cur) {
            __syncthreads();  // the previous instance's shared data is no longer read
            {
                const int* src = (const int*)(Pb + lo);
                int* dst = (int*)&sP;
                for (int w = threadIdx.x; w < (int)(sizeof(SolveParams) / sizeof(int)); w += NT) dst[w] = src[w];
            }
            __syncthreads();
            V = view64(smem_raw, sP, NC);
            J = kiss_setup(sP, V.xs, threadIdx.x % NGPT);
            cur = lo;
        }
        double* slot = (double*)sP.scratch + (size_t)blockIdx.x * sP.slot_elems;
        solve_group64<false, NC>(sP, item - s_pref[lo], V, J, slot, tab);
    }
}

// ----------------------------------------------------------- split solve
// A call with few columns leaves most SMs idle when a CTA takes a column pair
// (one pair: 0.62 ms on one SM), though its cells are independent of each
// other: k_cells64 spreads them over (pair, block of layers) CTAs, and
// k_sweep64 then runs each (column, sky)'s sweeps, sums and outputs.  Both
// use the fused kernel's functions and summation order, so the results are
// the same bit for bit.  Scratch: one slot64 per pair.
constexpr int SPLIT_THREADS = CTA_THREADS + 32;  // the pair's subcolumns and one warp that prepares its layers
constexpr int SPLIT_MAXLB = 16;                  // layers per CTA

struct SplitSmem64 {
    size_t tm, th, seed, misc, total;
};
__host__ __device__ inline SplitSmem64 split_smem64(const SolveParams& P) {
    SplitSmem64 m;
    size_t o = 0;
    m.tm = o;   o = align16(o + NBND * 2 * sizeof(TmSmem));
    m.th = o;   if (cloud_mode(P) == CLD_MASK) o = align16(o + (size_t)COLS_PER_CTA * P.nlay * TH_N * sizeof(double));
    m.seed = o; o = align16(o + COLS_PER_CTA * 4 * sizeof(uint32_t));
    m.misc = o; o = align16(o + COLS_PER_CTA * sizeof(int));
    m.total = o;
    return m;
}

// State of a KISS stream n draws after its seeds, for one subcolumn: the
// shift register by the matrices of n's bits (the fused kernel's per-launch
// matrix costs more than one pair saves).
__device__ inline Kiss kiss_at(const uint32_t* seed, uint64_t n) {
    const KissJump J = kiss_jump_consts(n);
    Kiss k;
    k.s1 = J.A * seed[0] + J.C;
    uint32_t y = seed[1];
    for (int b = 0; b < 32 && (n >> b); ++b) {
        if (!((n >> b) & 1)) continue;
        uint32_t r = 0;
#pragma unroll 8
        for (int i = 0; i < 32; ++i) r ^= (0u - (y >> i & 1u)) & cT.xs_jump[b][i];
        y = r;
    }
    k.s2 = y;
    k.s3 = (uint32_t)mulmod(J.a3n, seed[2], KISS_M3);
    k.s4 = (uint32_t)mulmod(J.a4n, seed[3], KISS_M4);
    return k;
}

// Layers lay0 + 1 .. lay0 + lb of pair blockIdx.x, lay0 = blockIdx.y lb: the
// layer solutions of both skies into the pair's slot.  While seven warps walk
// the McICA masks up to their layers, the eighth prepares the layers.
template <bool MT>
__global__ void __launch_bounds__(SPLIT_THREADS, 2)
k_cells64(const SolveParams P, int lb, const double* __restrict__ tab) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr int NT = CTA_THREADS;
    const SplitSmem64 M = split_smem64(P);
    TmSmem* sTm = (TmSmem*)(smem_raw + M.tm);
    double* th = (double*)(smem_raw + M.th);
    uint32_t* seed = (uint32_t*)(smem_raw + M.seed);
    int* misc = (int*)(smem_raw + M.misc);
    const int L = P.nlay, tid = threadIdx.x, pair = blockIdx.x;
    const int mode = cloud_mode(P);
    const int lay0 = blockIdx.y * lb, lay1 = min(L, lay0 + lb), nl = lay1 - lay0;
    const Slot64 S = slot64(L, P.idelm, COLS_PER_CTA, band_clouds(P), P.iaer != 0);
    double* slot = (double*)P.scratch + (size_t)pair * P.slot_elems;
    double* blk0 = slot + S.blk;
    double* cld0 = slot + S.cld;
    double* aer0 = slot + S.aer;
    fill_tm64(sTm);
    if (tid < COLS_PER_CTA) misc[tid] = 0;
    __syncthreads();
    for (int it = tid; it < COLS_PER_CTA * L; it += SPLIT_THREADS) {
        const int c2 = it / L, lay = it % L + 1, pcol = COLS_PER_CTA * pair + c2;
        if (pcol >= P.ncol) continue;
        // laytrop counts every layer below ~100 hPa (rrtmg_sw_setcoef.f90:207, as prep_layer)
        if (log(P.play[(size_t)pcol + (size_t)P.ncol * (size_t)(lay - 1)]) > 4.56) atomicAdd(misc + c2, 1);
        if (mode == CLD_MASK) {
            if (lay <= lay1) thresholds64<MT>(P, pcol, lay, th + (size_t)it * TH_N);
            if (!MT && lay == 1) seeds64(P, pcol, seed + c2 * 4);
        }
    }
    __syncthreads();
    const int cc = tid / NGPT, g = tid % NGPT;  // (the preparing warp: cc = 2)
    const int col = COLS_PER_CTA * pair + cc;
    unsigned bits = 0u;  // cloudy layers of the block
    bool active = false;
    if (tid < NT) {
        const int laytrop = misc[cc];
        active = col < P.ncol;
        if (active && (laytrop < 1 || laytrop >= L)) {
            set_error(P.err, E_LAYTROP);
            active = false;
        }
        if (active && mode == CLD_MASK) {
            Mask64<MT> mc;
            Kiss k0{1u, 1u, 1u, 1u};
            if constexpr (!MT) k0 = kiss_at(seed + cc * 4, kiss_offset(P.icld, g, L, P.permuteseed));
            mc.m.start(k0, P.icld, MT ? P.mt + mt_offset(P.icld, g, col, P.ncol, L) : nullptr);
            const double* t = th + (size_t)cc * L * TH_N;
            for (int lay = 1; lay <= lay1; ++lay, t += TH_N) {
                const bool cloudy = mc.step(lay, t);
                if (lay > lay0 && cloudy) bits |= 1u << (lay - lay0 - 1);
            }
        }
    } else {
        for (int it = tid - NT; it < COLS_PER_CTA * nl; it += 32) {
            const int c2 = it / nl, lay = lay0 + it % nl + 1;
            setcoef64(P, COLS_PER_CTA * pair + c2, lay, blk0 + (size_t)(c2 * L + lay - 1) * B_STRIDE, tab);
        }
    }
    __syncthreads();
    for (int it = tid; it < COLS_PER_CTA * nl * NBND; it += SPLIT_THREADS) {
        const int b = it % NBND, cl = it / NBND, c2 = cl / nl, lay = lay0 + cl % nl + 1;
        const int pcol = COLS_PER_CTA * pair + c2;
        const size_t i = (size_t)(c2 * L + lay - 1);
        if (pcol < P.ncol)
            prep_band64(P, pcol, lay, b, lay <= misc[c2], blk0 + i * B_STRIDE, cld0 + i * NBND * CO_N,
                        aer0 + i * NBND * AO_N, mode, MT, tab);
    }
    __syncthreads();
    if (!active) return;
    Mu64 m;
    m.mu = P.coszen[col];
    if (m.mu < 1.e-10) m.mu = 1.e-10;
    m.rmu = 1.0 / m.mu;
    m.mu34 = 0.75 * m.mu;
    const int ib = cT.ngb[g], igb = cT.gib[g];
    const int NF = fields64(P.idelm), laytrop = misc[cc];
#pragma unroll 1
    for (int lay = lay0 + 1; lay <= lay1; ++lay) {
        const size_t i = (size_t)(cc * L + lay - 1);
        Rt64 c, t;
        double dbtn = 1.0;
        cell64(P, sTm, blk0 + i * B_STRIDE, cld0 + i * NBND * CO_N, aer0 + i * NBND * AO_N, lay <= laytrop, col, g, lay,
               ib, igb, mode, (bits >> (lay - lay0 - 1)) & 1u, m, tab, c, t, dbtn);
        double* sv = slot + tid + (size_t)(L - lay) * NF * NT;
        sv[L_REF * NT] = c.ref;
        sv[L_REFD * NT] = c.refd;
        sv[L_TDIF * NT] = c.tdif;
        sv[L_TRAD * NT] = c.trad;
        sv[L_DBT * NT] = c.dbt;
        if (mode != CLD_NONE) {
            sv[(L_SKY + L_REF) * NT] = t.ref;
            sv[(L_SKY + L_REFD) * NT] = t.refd;
            sv[(L_SKY + L_TDIF) * NT] = t.tdif;
            sv[(L_SKY + L_TRAD) * NT] = t.trad;
            sv[(L_SKY + L_DBT) * NT] = t.dbt;
        }
        if (P.idelm == 0) sv[2 * L_SKY * NT] = dbtn;
    }
}

constexpr int SWEEP_THREADS = 128;  // one column's 112 g-points, whole warps
constexpr int SWEEP_KLEV = 16;      // levels per round of sums

struct SweepSmem64 {
    size_t pk, misc, red, flux, total;
};
__host__ __device__ inline SweepSmem64 sweep_smem64(const SolveParams& P) {
    SweepSmem64 m;
    size_t o = 0;
    m.pk = o;   o = align16(o + (size_t)P.nlay * sizeof(int));
    m.misc = o; o = align16(o + sizeof(int));
    m.red = o;  o = align16(o + (size_t)SWEEP_KLEV * 3 * NGPT * sizeof(double));
    m.flux = o; o = align16(o + (size_t)7 * (P.nlay + 1) * sizeof(double));
    m.total = o;
    return m;
}

// Sweeps of column blockIdx.x, sky blockIdx.y (0 clear, 1 total; a clear call
// has one sky and writes both skies' outputs), g-point sums and outputs.
__global__ void __launch_bounds__(SWEEP_THREADS)
k_sweep64(const SolveParams P, const double* __restrict__ tab) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr int NT = CTA_THREADS;
    const SweepSmem64 M = sweep_smem64(P);
    int* pk = (int*)(smem_raw + M.pk);
    int* misc = (int*)(smem_raw + M.misc);
    double* red0 = (double*)(smem_raw + M.red);
    double* flux = (double*)(smem_raw + M.flux);
    const int L = P.nlay, tid = threadIdx.x, col = blockIdx.x, cc = col % COLS_PER_CTA;
    const int mode = cloud_mode(P), NF = fields64(P.idelm);
    const int sky = blockIdx.y;
    const bool total = mode == CLD_NONE || sky == 1;  // writes the total sky's outputs
    const Slot64 S = slot64(L, P.idelm, COLS_PER_CTA, band_clouds(P), P.iaer != 0);
    double* slot = (double*)P.scratch + (size_t)(col / COLS_PER_CTA) * P.slot_elems;
    const double* blkc = slot + S.blk + (size_t)cc * L * B_STRIDE;
    if (tid == 0) *misc = 0;
    __syncthreads();
    for (int l = tid; l < L; l += SWEEP_THREADS) {
        const int w = *(const int*)(blkc + (size_t)l * B_STRIDE + B_PK);
        pk[l] = w;
        if ((w >> 30) & 1) atomicAdd(misc, 1);
    }
    __syncthreads();
    const int laytrop = *misc;
    const int g = min(tid, NGPT - 1), ib = cT.ngb[g], igb = cT.gib[g];
    const bool active = tid < NGPT && laytrop >= 1 && laytrop < L;
    double* sv0 = slot + cc * NGPT + g + (size_t)sky * L_SKY * NT;
    double zinc = 0.0, albp = 0.0, albd = 0.0;
    if (active) {
        double mu = P.coszen[col];
        if (mu < 1.e-10) mu = 1.e-10;
        const bool nir = ib <= 8 || ib == 13;
        albp = nir ? P.aldir[col] : P.asdir[col];
        albd = nir ? P.aldif[col] : P.asdif[col];
        zinc = P.adjflux[ib] * solar64(ib, igb, blkc, pk, L, laytrop, P, tab) * mu;
        double ru = albp, rud = albd;
        // the fields of the next two layers are loaded while one is swept
        // (the stores would hold the loads back)
        auto load = [&](int lay) {
            const double* sv = sv0 + (size_t)(L - lay) * NF * NT;
            Rt64 r;
            r.ref = sv[L_REF * NT];
            r.refd = sv[L_REFD * NT];
            r.tdif = sv[L_TDIF * NT];
            r.trad = sv[L_TRAD * NT];
            r.dbt = sv[L_DBT * NT];
            return r;
        };
        Rt64 n1 = load(1), n2 = load(min(2, L));
        for (int lay = 1; lay <= L; ++lay) {
            double* sv = sv0 + (size_t)(L - lay) * NF * NT;
            const Rt64 r = n1;
            n1 = n2;
            n2 = load(min(lay + 2, L));
            double alpha, beta;
            up64(r, ru, rud, alpha, beta);
            sv[L_RUP * NT] = ru;
            sv[L_RUPD * NT] = rud;
            sv[L_ALPHA * NT] = alpha;
            sv[L_BETA * NT] = beta;
        }
    }
    const bool need_dir = total && (P.extra || P.bands);
    const int nq = need_dir ? 3 : 2, nsum = total && P.extra ? 7 : nq;
    double d = zinc, f = 0.0, dn = zinc;
    const double* svn = slot + cc * NGPT + g + (size_t)2 * L_SKY * NT;  // idelm = 0: unscaled direct transmittance
    for (int j0 = 1; j0 <= L + 1; j0 += SWEEP_KLEV) {
        const int nlev = min(SWEEP_KLEV, L + 2 - j0);
#pragma unroll 4
        for (int s = 0; s < nlev; ++s) {
            const int jk = j0 + s;
            const size_t o = (size_t)(jk - 1) * NF * NT;
            double u = 0.0, dd = 0.0, dir = 0.0;
            if (active) {
                dd = d + f;
                dir = P.idelm == 0 ? dn : d;
                if (jk <= L) {
                    const double* sv = sv0 + o;
                    u = fma(sv[L_RUP * NT], d, sv[L_RUPD * NT] * f);
                    f = fma(sv[L_ALPHA * NT], d, sv[L_BETA * NT] * f);
                    d *= sv[L_DBT * NT];
                    if (P.idelm == 0) dn *= svn[o];
                } else {
                    u = fma(albp, d, albd * f);
                }
            }
            if (tid < NGPT) {
                double* red = red0 + (size_t)s * nq * NGPT + tid;
                red[0] = u;
                red[NGPT] = dd;
                if (need_dir) red[2 * NGPT] = dir;
            }
        }
        __syncthreads();
        const int jk = j0 + nlev - 1;
        sum_levels64(P, red0, flux, 1, NGPT, SWEEP_THREADS, nq, nsum, 2, jk, nlev);
        if (P.bands) {
            double* const* bo = P.bout;
            if (total) {
                for (int k = 0; k < 3; ++k)
                    band_levels64(P, red0, 1, NGPT, SWEEP_THREADS, nq, k, bo[k], col, 0, jk, nlev);
            }
            if (sky == 0) {
                for (int k = 0; k < 2; ++k)
                    band_levels64(P, red0, 1, NGPT, SWEEP_THREADS, nq, k, bo[3 + k], col, 0, jk, nlev);
            }
        }
        __syncthreads();
    }
    if (total)
        write_sky64(P, flux, 1, SWEEP_THREADS, nsum, 0, 2, P.extra != 0, col, 0, P.swuflx, P.swdflx, P.swhr);
    if (sky == 0)
        write_sky64(P, flux, 1, SWEEP_THREADS, nsum, 0, 2, false, col, 0, P.swuflxc, P.swdflxc, P.swhrc);
}

}  // namespace rrsw
