// ad.cuh -- tangent-linear and adjoint of the column solve (FP64).
//
// Objective per column, total sky (rrtmg_sw_rad.f90:822-836):
//   J = w_toa_up * swuflx(top) + w_sfc_net * (swdflx(sfc) - swuflx(sfc))
//     + w_hr_sum * sum over layers 1..nlay-1 of swhr,
// differentiated with respect to tlay, h2ovmr, o3vmr, the McICA cloud
// water paths clwp, ciwp (masks frozen: they depend on cldfrac and the seeds
// only) and the four surface albedos.
//
// The model differentiated is the reference's with exp(-x) in place of the
// nearest-entry transmittance table and of its quadratic below od_lo
// (rrtmg_sw_reftra.f90:203-209, spcvmc:558-585): the table makes the
// reference piecewise constant in every optical depth, so its derivative is
// zero almost everywhere.  The value J returned is that of the smooth model,
// which is what finite differences of this entry point check.
//
// k_adjoint (one thread per (column, g-point), two passes over the layers):
//   bottom to top  the cell's gas optics with their derivatives along the
//            layer's tlay, h2ovmr, o3vmr; its layer solution; the up-sweep;
//            and the adjoint of the down-sweep: with the form of up64 the
//            down-sweep is linear in (direct, diffuse) flux, and the adjoint
//            of a level's two fluxes needs only what the up-sweep has made
//            below it.  At the top it is J per unit of incident flux.
//   top to bottom  the fluxes, the adjoint of the up-sweep, then that of the
//            layer solution down to its three optical inputs (scattering,
//            scattering times asymmetry, absorption) and, through the stored
//            derivatives, to the layer's inputs, summed over g-points (the
//            queued cells below by atomics, in no fixed order: gradients
//            differ in their last bits from run to run).
// Like the FP64 solve it is bound by the FP64 pipe.
//
// Where the reference's own derivative is dominated by rounding (NOISE_AD
// below), a cell's local Jacobian is formed instead in forward mode with the
// reference's order of operations (five outputs along three to five directions
// as duals, about 2 000 FP64 instructions): the second pass queues those cells
// and the CTA then takes them 32 to a warp.  Formed for every cell, as the
// tangent does: 4 096 x 60 columns with clouds 160 ms; now 34.6 ms (91 ms with
// each warp forming them on the spot, of its 32 lanes those that need it).
//
// k_tangent runs the forward model with every cell's Jacobian in duals
// contracted with the direction, an independent check of the adjoint; J itself
// comes from k_adjoint's first pass in both entry points, for the tangent in an
// instance that forms nothing else and runs beside k_tangent.
#pragma once

#include "fp64_cell.cuh"

namespace rrsw {

// ============================================================= Jacobians
// ---------------------------------------------------------------- duals
template <int N>
struct Dual {
    double v;
    double d[N];
    __host__ __device__ Dual() : v(0.0) {
        for (int i = 0; i < N; ++i) d[i] = 0.0;
    }
    __host__ __device__ Dual(double x) : v(x) {
        for (int i = 0; i < N; ++i) d[i] = 0.0;
    }
    __host__ __device__ explicit operator int() const { return (int)v; }
};
template <int N>
struct TabOf<Dual<N>> { typedef double type; };

#define DUAL_BIN(OP, VAL, DER)                                                                   \
    template <int N>                                                                             \
    __device__ inline Dual<N> operator OP(const Dual<N>& a, const Dual<N>& b) {                  \
        Dual<N> r;                                                                               \
        r.v = VAL;                                                                               \
        for (int i = 0; i < N; ++i) r.d[i] = DER;                                                \
        return r;                                                                                \
    }                                                                                            \
    template <int N>                                                                             \
    __device__ inline Dual<N> operator OP(const Dual<N>& a, double bv) { return a OP Dual<N>(bv); } \
    template <int N>                                                                             \
    __device__ inline Dual<N> operator OP(double av, const Dual<N>& b) { return Dual<N>(av) OP b; }
DUAL_BIN(+, a.v + b.v, a.d[i] + b.d[i])
DUAL_BIN(-, a.v - b.v, a.d[i] - b.d[i])
DUAL_BIN(*, a.v * b.v, a.d[i] * b.v + a.v * b.d[i])
DUAL_BIN(/, a.v / b.v, (a.d[i] - (a.v / b.v) * b.d[i]) / b.v)
#undef DUAL_BIN

template <int N>
__device__ inline Dual<N> operator-(const Dual<N>& a) {
    Dual<N> r;
    r.v = -a.v;
    for (int i = 0; i < N; ++i) r.d[i] = -a.d[i];
    return r;
}
template <int N>
__device__ inline Dual<N>& operator+=(Dual<N>& a, const Dual<N>& b) { a = a + b; return a; }
template <int N>
__device__ inline Dual<N>& operator-=(Dual<N>& a, const Dual<N>& b) { a = a - b; return a; }
template <int N>
__device__ inline Dual<N>& operator*=(Dual<N>& a, const Dual<N>& b) { a = a * b; return a; }

#define DUAL_CMP(OP)                                                                                    \
    template <int N>                                                                                    \
    __device__ inline bool operator OP(const Dual<N>& a, const Dual<N>& b) { return a.v OP b.v; }       \
    template <int N>                                                                                    \
    __device__ inline bool operator OP(const Dual<N>& a, double b) { return a.v OP b; }                 \
    template <int N>                                                                                    \
    __device__ inline bool operator OP(double a, const Dual<N>& b) { return a OP b.v; }
DUAL_CMP(<)
DUAL_CMP(<=)
DUAL_CMP(>)
DUAL_CMP(>=)
DUAL_CMP(==)
DUAL_CMP(!=)
#undef DUAL_CMP

template <int N>
__device__ inline Dual<N> sqrt(const Dual<N>& a) {
    Dual<N> r;
    r.v = ::sqrt(a.v);
    for (int i = 0; i < N; ++i) r.d[i] = a.d[i] / (2.0 * r.v);
    return r;
}
template <int N>
__device__ inline Dual<N> exp(const Dual<N>& a) {
    Dual<N> r;
    r.v = ::exp(a.v);
    for (int i = 0; i < N; ++i) r.d[i] = r.v * a.d[i];
    return r;
}
template <int N>
__device__ inline Dual<N> log(const Dual<N>& a) {
    Dual<N> r;
    r.v = ::log(a.v);
    for (int i = 0; i < N; ++i) r.d[i] = a.d[i] / a.v;
    return r;
}
template <int N>
__device__ inline Dual<N> fmin(const Dual<N>& a, double b) { return a.v <= b ? a : Dual<N>(b); }

template <> __device__ inline Dual<3> c_oneminus<Dual<3>>() { return Dual<3>(cT.oneminus); }
template <> __device__ inline Dual<5> c_oneminus<Dual<5>>() { return Dual<5>(cT.oneminus); }
template <> __device__ inline Dual<3> c_bpade<Dual<3>>() { return Dual<3>(cT.bpade); }
template <> __device__ inline Dual<5> c_bpade<Dual<5>>() { return Dual<5>(cT.bpade); }

// Dual<5> holding the value and derivatives of a Dual<3> in its first slots
__device__ inline Dual<5> widen(const Dual<3>& a) {
    Dual<5> r(a.v);
    r.d[0] = a.d[0]; r.d[1] = a.d[1]; r.d[2] = a.d[2];
    return r;
}

// ------------------------------------------------- setcoef with derivatives
// inatm_sw (rrtmg_sw_rad.f90:1527-1586) and setcoef_sw
// (rrtmg_sw_setcoef.f90:158-301) for one (column, layer) with derivatives
// with respect to (tlay, h2ovmr, o3vmr) of that layer; the indices are those
// of the values.  Writes the NFR coefficients (Dual<3>, [NFR] with stride L
// starting at cf) and the packed indices; returns the layer's pressure
// thickness.
__device__ inline double prep_layer_dual(const SolveParams& P, int col, int lay, Dual<3>* cf, int L, int* pk,
                                         const double* __restrict__ tab64) {
    typedef Dual<3> D;
    const int i = lay - 1;
    const size_t n = (size_t)P.ncol;
    const size_t k = (size_t)col + n * (size_t)i;
    const double p = P.play[k];
    D t(P.tlay[k]);
    t.d[0] = 1.0;
    D h2o(P.h2ovmr[k]);
    h2o.d[1] = 1.0;
    D o3(P.o3vmr[k]);
    o3.d[2] = 1.0;
    const double pzb = P.plev[k], pzt = P.plev[k + n];
    const double amd = 28.9660, amw = 18.0160, avogad = 6.02214199e+23, grav = 9.8066;
    const D amm = (1.0 - h2o) * amd + h2o * amw;
    const D coldry = ((pzb - pzt) * 1.e3 * avogad) / ((1.e2 * grav) * amm * (1.0 + h2o));
    const D w0 = coldry * h2o, w2 = coldry * o3;
    const D w1 = coldry * P.co2vmr[k], w5 = coldry * P.ch4vmr[k], w6 = coldry * P.o2vmr[k];
    const double pdp = pzb - pzt;
    const double stpfac = 296.0 / 1013.0;
    const double plog = ::log(p);
    int jp = (int)(36.0 - 5.0 * (plog + 0.04));
    jp = jp < 1 ? 1 : (jp > 58 ? 58 : jp);
    const double fp = 5.0 * (ldt(tab64, cT.preflog + jp - 1) - plog);
    const double tr0 = ldt(tab64, cT.tref + jp - 1), tr1 = ldt(tab64, cT.tref + jp);
    int jt = (int)(3.0 + (t.v - tr0) / 15.0);
    jt = jt < 1 ? 1 : (jt > 4 ? 4 : jt);
    const D ft = (t - tr0) / 15.0 - (double)(jt - 3);
    int jt1 = (int)(3.0 + (t.v - tr1) / 15.0);
    jt1 = jt1 < 1 ? 1 : (jt1 > 4 ? 4 : jt1);
    const D ft1 = (t - tr1) / 15.0 - (double)(jt1 - 3);
    const D water = w0 / coldry;
    const D scalefac = (p * stpfac) / t;
    D forfac, forfrac, selffac, selffrac;
    int indfor, indself, low;
    if (plog > 4.56) {
        low = 1;
        forfac = scalefac / (1.0 + water);
        D factor = (332.0 - t) / 36.0;
        indfor = (int)factor;
        indfor = indfor < 1 ? 1 : (indfor > 2 ? 2 : indfor);
        forfrac = factor - (double)indfor;
        selffac = water * forfac;
        factor = (t - 188.0) / 7.2;
        indself = (int)factor - 7;
        indself = indself < 1 ? 1 : (indself > 9 ? 9 : indself);
        selffrac = factor - (double)(indself + 7);
    } else {
        low = 0;
        forfac = scalefac / (1.0 + water);
        const D factor = (t - 188.0) / 36.0;
        indfor = 3;
        forfrac = factor - 1.0;
        selffac = D(0.0);
        selffrac = D(0.0);
        indself = 0;
    }
    const D colh2o = 1.e-20 * w0;
    D colco2 = 1.e-20 * w1, colo3 = 1.e-20 * w2, colch4 = 1.e-20 * w5, colo2 = 1.e-20 * w6;
    const D colmol = 1.e-20 * coldry + colh2o;
    if (colco2 == 0.0) colco2 = 1.e-32 * coldry;
    if (colch4 == 0.0) colch4 = 1.e-32 * coldry;
    if (colo2 == 0.0) colo2 = 1.e-32 * coldry;
    const double compfp = 1.0 - fp;
    cf[F_FAC10 * L + i] = compfp * ft;
    cf[F_FAC00 * L + i] = compfp * (1.0 - ft);
    cf[F_FAC11 * L + i] = fp * ft1;
    cf[F_FAC01 * L + i] = fp * (1.0 - ft1);
    cf[F_H2O * L + i] = colh2o;
    cf[F_CO2 * L + i] = colco2;
    cf[F_O3 * L + i] = colo3;
    cf[F_CH4 * L + i] = colch4;
    cf[F_O2 * L + i] = colo2;
    cf[F_MOL * L + i] = colmol;
    cf[F_SELFFAC * L + i] = selffac;
    cf[F_SELFFRAC * L + i] = selffrac;
    cf[F_FORFAC * L + i] = forfac;
    cf[F_FORFRAC * L + i] = forfrac;
    cf[F_PDP * L + i] = D(pdp);
    pk[i] = jp | (jt << 8) | (jt1 << 12) | (indself << 16) | (indfor << 24) | (low << 30);
    return pdp;
}

// --------------------------------------------------- smooth two-stream
// reftra_sw (rrtmg_sw_reftra.f90:151-326), kmodts = 2, with exp(-x) for
// every transmittance; T is double or a dual.
template <typename T>
struct RTs { T ref, refd, tra, trad, x, e2; };  // x = tau/mu0, e2 = exp(-x) for x <= 500

template <typename T>
__device__ inline RTs<T> reftra_sm(T zto1, T zw, T zg, double prmuz) {
    RTs<T> o;
    const double zwcrit = 0.9999995, eps = 1.e-08;
    const T zg3 = 3.0 * zg;
    const T zgamma1 = (8.0 - zw * (5.0 + zg3)) * 0.25;
    const T zgamma2 = 3.0 * (zw * (1.0 - zg)) * 0.25;
    const T zgamma3 = (2.0 - zg3 * prmuz) * 0.25;
    const T zgamma4 = 1.0 - zgamma3;
    o.x = zto1 / prmuz;
    T zwo(0.0), denom(1.0);
    if (zg != 1.0) {
        const T q = zg / (1.0 - zg);
        denom = 1.0 - (1.0 - zw) * (q * q);
    }
    if (zw > 0.0 && denom != 0.0) zwo = zw / denom;
    if (zwo >= zwcrit) {
        const T za1 = zgamma1 * prmuz - zgamma3;
        const T zgt = zgamma1 * zto1;
        const T ze2 = exp(-fmin(o.x, 500.0));
        o.e2 = ze2;
        o.ref = (zgt - za1 * (1.0 - ze2)) / (1.0 + zgt);
        o.tra = 1.0 - o.ref;
        o.refd = zgt / (1.0 + zgt);
        o.trad = 1.0 - o.refd;
        if (ze2 == 1.0) { o.ref = T(0.0); o.tra = T(1.0); o.refd = T(0.0); o.trad = T(1.0); }
        return o;
    }
    const T za1 = zgamma1 * zgamma4 + zgamma2 * zgamma3;
    const T za2 = zgamma1 * zgamma3 + zgamma2 * zgamma4;
    const T zrk = sqrt(zgamma1 * zgamma1 - zgamma2 * zgamma2);
    const T zrp = zrk * prmuz;
    const T zrp1 = 1.0 + zrp, zrm1 = 1.0 - zrp;
    const T zrk2 = 2.0 * zrk;
    const T zrpp = 1.0 - zrp * zrp;
    const T zrkg = zrk + zgamma1;
    const T zr1 = zrm1 * (za2 + zrk * zgamma3);
    const T zr2 = zrp1 * (za2 - zrk * zgamma3);
    const T zr3 = zrk2 * (zgamma3 - za2 * prmuz);
    const T zr4 = zrpp * zrkg;
    const T zr5 = zrpp * (zrk - zgamma1);
    const T zt1 = zrp1 * (za1 + zrk * zgamma4);
    const T zt2 = zrm1 * (za1 - zrk * zgamma4);
    const T zt3 = zrk2 * (zgamma4 + za1 * prmuz);
    const T zbeta = (zgamma1 - zrk) / zrkg;
    const T zem1 = exp(-fmin(zrk * zto1, 500.0));
    const T zep1 = 1.0 / zem1;
    const T zem2 = exp(-fmin(o.x, 500.0));
    o.e2 = zem2;
    const T zep2 = 1.0 / zem2;
    const T zdenr = zr4 * zep1 + zr5 * zem1;
    if (zdenr >= -eps && zdenr <= eps) {
        o.ref = T(eps);
        o.tra = zem2;
    } else {
        o.ref = zw * (zr1 * zep1 - zr2 * zem1 - zr3 * zem2) / zdenr;
        o.tra = zem2 - zem2 * zw * (zt1 * zep1 - zt2 * zem1 - zt3 * zep2) / zdenr;
    }
    const T zemm = zem1 * zem1;
    const T zdend = 1.0 / ((1.0 - zbeta * zemm) * zrkg);
    o.refd = zgamma2 * (1.0 - zemm) * zdend;
    o.trad = zrk2 * zem1 * zdend;
    return o;
}

// Total-sky optics of one cell for the objective (spcvmc:442-549 with the
// McICA cloud fraction 0 or 1): out[0..4] = pref, prefd, ptra, ptrad, zdbt.
// Without aerosol the clear sky's asymmetry is zero and its delta scaling the
// identity, value and derivatives; without its divisions, and with one
// exp(-tau/mu0) instead of two, a tangent-linear call of 8 192 x 60 columns
// takes 300 ms with clouds and 210 clear instead of 347 and 246.
template <typename T>
__device__ inline void cell_total(const CellIn<T>& ci, bool aer, double prmu0, T out[5]) {
    T ztauc = ci.taur + ci.taug, zomcc, zgcc(0.0);
    if (aer) {
        ztauc = ztauc + ci.rta;
        zomcc = ci.taur * 1.0 + ci.rta * ci.roa;
        zgcc = ci.rga * ci.roa * ci.rta / zomcc;
        zomcc = zomcc / ztauc;
        const T zf = zgcc * zgcc;
        const T zwf = zomcc * zf;
        ztauc = (1.0 - zwf) * ztauc;
        zomcc = (zomcc - zwf) / (1.0 - zwf);
        zgcc = (zgcc - zf) / (1.0 - zf);
    } else {
        zomcc = ci.taur / ztauc;
    }
    T tau = ztauc, om = zomcc, g = zgcc;
    if (ci.cloudy) {
        const T ztauo = ztauc + ci.tc;
        T zomco = ztauc * zomcc + ci.tc * ci.oc;
        const T zgco = (ci.tc * ci.oc * ci.gc + ztauc * zomcc * zgcc) / zomco;
        zomco = zomco / ztauo;
        tau = ztauo;
        om = zomco;
        g = zgco;
    }
    const RTs<T> r = reftra_sm(tau, om, g, prmu0);
    out[0] = r.ref;
    out[1] = r.refd;
    out[2] = r.tra;
    out[3] = r.trad;
    out[4] = r.x <= 500.0 ? r.e2 : exp(-r.x);
}

// Optics of one cell with derivatives (pass 1 and the recomputing reverse
// pass).  Gas optics and aerosol depend on (tlay, h2ovmr, o3vmr) only, so
// they run in Dual<3> for every cell; a cloudy cell widens them to Dual<5>
// over (tlay, h2ovmr, o3vmr, clwp, ciwp) for cldprmc and the two-stream
// solution, a clear cell finishes in Dual<3> and is widened with zero
// water-path derivatives.  Each variant is compiled once (not inlined at
// its call sites): the kernel's instruction footprint, not its arithmetic,
// was what its warps waited on most.
__device__ __noinline__ void ad_cell_clear(const CellIn<Dual<3>>& ci, bool aer, double cossza, Dual<5> out[5]) {
    Dual<3> o[5];
    cell_total(ci, aer, cossza, o);
    for (int k = 0; k < 5; ++k) out[k] = widen(o[k]);
}

__device__ __noinline__ void ad_cell_cloudy(const SolveParams& P, const CellIn<Dual<3>>& c3, int col, int lay, int ib,
                                            const double* cld, int L, double cossza,
                                            const double* __restrict__ tab64, Dual<5> out[5]) {
    typedef Dual<5> D;
    CellIn<D> ci;
    ci.taug = widen(c3.taug);
    ci.taur = widen(c3.taur);
    ci.rta = widen(c3.rta); ci.roa = widen(c3.roa); ci.rga = widen(c3.rga); ci.rcoa = widen(c3.rcoa);
    ci.cloudy = true;
    ci.cldf = D(1.0);
    D ciwp(cld[0 * L + lay - 1]), clwp(cld[1 * L + lay - 1]);
    clwp.d[3] = 1.0;
    ciwp.d[4] = 1.0;
    const D rei(cld[2 * L + lay - 1]), rel(cld[3 * L + lay - 1]);
    D tc(0.0), oc(1.0), gc(0.0), fsfc(0.0), taor(0.0), coc(0.0);
    if (P.tauc) {
        const size_t kb = (size_t)ib + 14 * ((size_t)col + (size_t)P.ncol * (size_t)(lay - 1));
        tc = D(P.tauc[kb]); oc = D(P.ssac[kb]); gc = D(P.asmc[kb]); fsfc = D(P.fsfc[kb]);
    }
    cldprmc_g<D>(ib, P.inflag, P.iceflag, P.liqflag, D(1.0), ciwp, clwp, rei, rel, fsfc, tc, oc, gc, taor, coc,
                 tab64, P.err);
    ci.tc = tc; ci.oc = oc; ci.gc = gc; ci.coc = coc; ci.taor = taor;
    cell_total(ci, P.iaer != 0, cossza, out);
}

__device__ __noinline__ void ad_cell(const SolveParams& P, const Dual<3>* coef3, const int* pk, int L, int laytrop,
                                     int col, int lay, int ib, int igb, bool cloudy, const double* cld,
                                     double cossza, const double* __restrict__ tab64, Dual<5> out[5]) {
    typedef Dual<3> D;
    D cf[NFR];
    for (int f = 0; f < NFR; ++f) cf[f] = coef3[f * L + lay - 1];
    const Coef<D> CN{cf, pk + lay - 1, 1, lay <= laytrop ? 1 : 0};
    CellIn<D> ci;
    taumol_g<D>(ib, igb, 1, CN, tab64, ci.taug, ci.taur);
    aerosol_in<D>(P, col, lay, ib, tab64, ci);
    ci.cloudy = false;
    ci.cldf = D(0.0);
    ci.tc = D(0.0); ci.oc = D(1.0); ci.gc = D(0.0); ci.coc = D(0.0); ci.taor = D(0.0);
    if (cloudy) ad_cell_cloudy(P, ci, col, lay, ib, cld, L, cossza, tab64, out);
    else ad_cell_clear(ci, P.iaer != 0, cossza, out);
}

// ================================================================ tangent
// ------------------------------------------------------- tangent kernel
// per-level scratch fields of one thread
enum { T_REF, T_REFD, T_TRA, T_TRAD, T_DBT, T_RUP, T_RUPD, T_N };

// scratch elements (doubles) per CTA slot: values and tangents, then the
// layers' coefficients
__host__ __device__ inline size_t tl_slot_elems(int L) {
    return (size_t)(L + 1) * 2 * T_N * CTA_THREADS + (size_t)COLS_PER_CTA * NFR * L * 4;
}

struct TlSmem {
    size_t pk, hc, misc, th, cld, seed, xs, jsum, total;
};
__host__ __device__ inline TlSmem tl_smem_layout(int L) {
    TlSmem m;
    size_t o = 0;
    m.pk = o;   o = align16(o + COLS_PER_CTA * L * sizeof(int));
    m.hc = o;   o = align16(o + COLS_PER_CTA * L * sizeof(double));
    m.misc = o; o = align16(o + 8 * sizeof(int));
    m.th = o;   o = align16(o + (size_t)COLS_PER_CTA * L * TH_N * sizeof(double));
    m.cld = o;  o = align16(o + (size_t)COLS_PER_CTA * 4 * L * sizeof(double));
    m.seed = o; o = align16(o + COLS_PER_CTA * 4 * sizeof(uint32_t));
    m.xs = o;   o = align16(o + NGPT * 32 * sizeof(uint32_t));
    m.jsum = o; o = align16(o + COLS_PER_CTA * sizeof(double));
    m.total = o;
    return m;
}

__device__ inline Dual<1> dual1(double v, double d) {
    Dual<1> r(v);
    r.d[0] = d;
    return r;
}

__global__ void __launch_bounds__(CTA_THREADS, 3)
k_tangent(const SolveParams P, const AdParams A, const double* __restrict__ tab64) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int L = P.nlay;
    const TlSmem M = tl_smem_layout(L);
    int* sPk = (int*)(smem_raw + M.pk);
    double* sHc = (double*)(smem_raw + M.hc);
    int* sMisc = (int*)(smem_raw + M.misc);
    double* sTh = (double*)(smem_raw + M.th);
    double* sCld = (double*)(smem_raw + M.cld);
    uint32_t* sSeed = (uint32_t*)(smem_raw + M.seed);
    uint32_t* sXs = (uint32_t*)(smem_raw + M.xs);
    double* sJ = (double*)(smem_raw + M.jsum);

    const int tid = threadIdx.x;
    const int cc = thread_col_ad(tid), g = thread_g_ad(tid);
    const int ib = cT.ngb[g], igb = cT.gib[g];
    const bool nir = ib <= 8 || ib == 13;
    const bool fused = P.fused && P.icld >= 1;
    double* slot = (double*)P.scratch + (size_t)blockIdx.x * P.slot_elems;
    Dual<3>* coef3 = (Dual<3>*)(slot + (size_t)(L + 1) * 2 * T_N * CTA_THREADS);
    const size_t n = (size_t)P.ncol;
    const KissJump J = kiss_setup(P, sXs, g);

    for (int pair = blockIdx.x; pair < P.npairs; pair += gridDim.x) {
        __syncthreads();
        if (tid < COLS_PER_CTA) sJ[tid] = 0.0;
        if (tid < COLS_PER_CTA) sMisc[tid] = 0;
        __syncthreads();
        for (int it = tid; it < COLS_PER_CTA * L; it += CTA_THREADS) {
            const int c2 = it / L, lay = it % L + 1;
            const int pcol = COLS_PER_CTA * pair + c2;
            const bool real = pcol < P.ncol;
            const size_t kl = (size_t)pcol + n * (size_t)(lay - 1);
            double pdp = 1.0;
            if (real) {
                pdp = prep_layer_dual(P, pcol, lay, coef3 + c2 * NFR * L, L, sPk + c2 * L, tab64);
                atomicAdd(sMisc + c2, (sPk[c2 * L + lay - 1] >> 30) & 1);
            } else {
                for (int f = 0; f < NFR; ++f) coef3[c2 * NFR * L + f * L + lay - 1] = Dual<3>(0.0);
                sPk[c2 * L + lay - 1] = 1 | (1 << 8) | (1 << 12) | (1 << 16) | (1 << 24);
            }
            sHc[c2 * L + lay - 1] = cT.heatfac / pdp;
            double* cd = sCld + c2 * 4 * L;
            cd[0 * L + lay - 1] = real && P.icld >= 1 ? P.ciwp[kl] : 0.0;
            cd[1 * L + lay - 1] = real && P.icld >= 1 ? P.clwp[kl] : 0.0;
            cd[2 * L + lay - 1] = real && P.icld >= 1 ? P.rei[kl] : 0.0;
            cd[3 * L + lay - 1] = real && P.icld >= 1 ? P.rel[kl] : 0.0;
            if (fused) {
                thresholds64<false>(P, pcol, lay, sTh + (size_t)it * TH_N);
                if (lay == 1 && real) seeds64(P, pcol, sSeed + c2 * 4);
            }
        }
        __syncthreads();
        const int col = COLS_PER_CTA * pair + cc;
        const int laytrop = sMisc[cc];
        bool active = col < P.ncol;
        if (active && (laytrop < 1 || laytrop >= L)) {
            set_error(P.err, E_LAYTROP);
            active = false;
        }
        auto at = [&](int jk, int fld) -> double& {  // level jk (1 = top .. L+1 = surface); tangents T_N behind
            return slot[((size_t)(jk - 1) * 2 * T_N + fld) * CTA_THREADS + tid];
        };
        const double* hc = sHc + cc * L;
        // objective seeds of level m (0 = surface .. L = top), without zinc
        auto seeds = [&](int m, double& sU, double& sD) {
            double an = 0.0;  // dJ/d net(m) through the heating-rate sum (layers 0 .. L-2)
            if (m >= 1 && m - 1 <= L - 2) an += A.w_hr * hc[m - 1];
            if (m <= L - 2) an -= A.w_hr * hc[m];
            sD = an + (m == 0 ? A.w_net : 0.0);
            sU = -an + (m == L ? A.w_toa : 0.0) - (m == 0 ? A.w_net : 0.0);
        };
        if (active) {
            double cossza = P.coszen[col];
            if (cossza < 1.e-10) cossza = 1.e-10;
            const double* a0 = A.dira[nir ? 2 : 0];
            const double* a1 = A.dira[nir ? 3 : 1];
            const Dual<1> albp = dual1(nir ? P.aldir[col] : P.asdir[col], a0 ? a0[col] : 0.0);
            const Dual<1> albd = dual1(nir ? P.aldif[col] : P.asdif[col], a1 ? a1[col] : 0.0);
            auto dirv = [&](int d, int lay) -> double {
                return A.dir[d] ? A.dir[d][(size_t)col + n * (size_t)(lay - 1)] : 0.0;
            };
            const Dual<3>* cf3 = coef3 + cc * NFR * L;
            const int* pk = sPk + cc * L;
            const Coef<Dual<3>> C3{cf3, pk, L, laytrop};
            const Dual<3> z3 = Dual<3>(P.adjflux[ib]) * solar_source<Dual<3>>(ib, igb, C3, P, tab64) * cossza;
            const int lsol = solar_layer(ib, C3);
            Dual<1> zinc(z3.v);
            if (lsol >= 1)
                for (int d = 0; d < 3; ++d) zinc.d[0] += z3.d[d] * dirv(d, lsol);
            Mask64<false> mc;
            if (fused) mc.m.start(kiss_start(sSeed + cc * 4, J, sXs + g * 32), P.icld);
            // pass 1: cells and up-sweep (vrtqdr:131-140), bottom -> top
            Dual<1> rup_b = albp, rupd_b = albd;
            for (int lay = 1; lay <= L; ++lay) {
                const int jk = L + 1 - lay;
                const bool cloudy = fused && mc.step(lay, sTh + (size_t)(cc * L + lay - 1) * TH_N);
                Dual<5> jac[5];
                ad_cell(P, cf3, pk, L, laytrop, col, lay, ib, igb, cloudy, sCld + cc * 4 * L, cossza, tab64, jac);
                double dv[5];
                for (int d = 0; d < 5; ++d) dv[d] = dirv(d, lay);
                Dual<1> o[5];
                for (int k = 0; k < 5; ++k) {
                    o[k].v = jac[k].v;
                    for (int d = 0; d < 5; ++d) o[k].d[0] += jac[k].d[d] * dv[d];
                }
                const Dual<1> zr = 1.0 / (1.0 - rupd_b * o[1]);
                const Dual<1> E = (o[2] - o[4]) * rupd_b + o[4] * rup_b;
                rup_b = o[0] + o[3] * E * zr;
                rupd_b = o[1] + o[3] * o[3] * rupd_b * zr;
                const Dual<1> w[T_N] = {o[0], o[1], o[2], o[3], o[4], rup_b, rupd_b};
                for (int k = 0; k < T_N; ++k) {
                    at(jk, k) = w[k].v;
                    at(jk, T_N + k) = w[k].d[0];
                }
            }
            // pass 2: down-sweep and level fluxes (vrtqdr:144-169), top -> bottom
            Dual<1> phi, tdbt(1.0), tdn(1.0), rdnd(0.0);
            for (int jk = 1; jk <= L + 1; ++jk) {
                const bool sfc = jk == L + 1;
                const Dual<1> rup = sfc ? albp : dual1(at(jk, T_RUP), at(jk, T_N + T_RUP));
                const Dual<1> rupd = sfc ? albd : dual1(at(jk, T_RUPD), at(jk, T_N + T_RUPD));
                const Dual<1> zr = 1.0 / (1.0 - rdnd * rupd);
                const Dual<1> D = tdn - tdbt;
                const Dual<1> fu = (tdbt * rup + D * rupd) * zr;
                const Dual<1> fd = tdbt + (D + tdbt * rup * rdnd) * zr;
                double sU, sD;
                seeds(L + 1 - jk, sU, sD);
                phi += sU * fu + sD * fd;
                if (!sfc) {
                    Dual<1> o[5];
                    for (int k = 0; k < 5; ++k) o[k] = dual1(at(jk, k), at(jk, T_N + k));
                    const Dual<1> z2 = 1.0 / (1.0 - o[1] * rdnd);
                    tdn = tdbt * o[2] + o[3] * (D + tdbt * o[0] * rdnd) * z2;
                    rdnd = o[1] + o[3] * o[3] * rdnd * z2;
                    tdbt = o[4] * tdbt;
                }
            }
            atomicAdd(&sJ[cc], (zinc * phi).d[0]);
        }
        __syncthreads();
        if (tid < COLS_PER_CTA) {
            const int ocol = COLS_PER_CTA * pair + tid;
            if (ocol < P.ncol) {
                if (A.dJ) A.dJ[ocol] = sJ[tid];
            }
        }
    }
}

// ================================================================ adjoint
// 1024 entries of 2^(-j/1024) and, exactly rounded, of 1 less it, at cT.exp2
// of the FP64 tables: exp(-x) for 0 <= x <= 500 with n = rint(1024 x / ln 2),
// exp(-x) = 2^(-n/1024) (1 + q), q = expm1(r), r = n ln 2 / 1024 - x, |r| <
// 3.4e-4 (table-driven, Tang 1989), and om = 1 - exp(-x) without cancellation.
// exp(-x) is within 2 ulp, om within 4.
constexpr int EXP2_N = 1024;
__device__ __forceinline__ void expm64(double x, const double* __restrict__ tab, double& e, double& om) {
    const double magic = 6755399441055744.0;  // 1.5 * 2^52
    const double t = fma(x, 1477.3197218702985, magic);  // 1024 / ln 2
    const double nd = t - magic;
    const int n = __double2loint(t), j = n & (EXP2_N - 1), m = n >> 10;
    double r = fma(nd, 6.769015435155716e-04, -x);       // ln 2 / 1024, rounded ..
    r = fma(nd, 2.264694154146777e-20, r);              // .. and the rest
    const double p = fma(fma(r, 1.0 / 24.0, 1.0 / 6.0), r, 0.5);
    const double q = fma(r * r, p, r);
    const double T0 = ldt(tab, cT.exp2 + 2 * j);
    const double T = __hiloint2double(__double2hiint(T0) - (m << 20), __double2loint(T0));
    e = fma(T, q, T);
    om = m == 0 ? fma(-T, q, ldt(tab, cT.exp2 + 2 * j + 1)) : 1.0 - e;
}

// sqrt64 with the reciprocal root: x^1/2 and x^-1/2 for positive normal x, both
// with an error below 1.1 ulp.
__device__ __forceinline__ void root64(double x, double& k, double& rk) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double m = x * y, e = fma(-m, y, 1.0), p = e * fma(0.375, e, 0.5);
    k = fma(m, p, m);
    rk = fma(y, p, y);
}

// The prepared block's derivative fields, behind fp64_cell.cuh's B_*: of the
// interpolation factors along tlay (fac10 = -fac00 and fac11 = -fac01), 1/tlay,
// d ln(column amount)/d h2ovmr, d colh2o and d colmol / d h2ovmr, d colo3 /
// d o3vmr, d forfac and d selffac / d h2ovmr, d forfrac / d tlay; per band
// the column amount's and per two-species band the ratio's along h2ovmr;
// along o3vmr those of bands 27 and 28.
enum { D_T0 = B_STRIDE, D_T1, D_IT, D_LH, D_HW, D_MOLH, D_O3O, D_FOH, D_SEH, D_FFT, D_COMBH, D_FSH = D_COMBH + NBND,
       D_COMBO = D_FSH + 8, D_FSO = D_COMBO + 2, D_END };
constexpr int D_STRIDE = (D_END + 1) & ~1;
// cloud optics' derivatives along clwp and ciwp: scattering, that times the
// asymmetry, absorption
enum { CJ_SL, CJ_GL, CJ_AL, CJ_SI, CJ_GI, CJ_AI, CJ_N };

// Stored per (layer, g-point): the up-sweep (albedos at the layer's top,
// alpha, beta, 1/(1 - rupd refd)), the layer solution, the adjoints of the
// direct and diffuse flux below the layer, the optical inputs with the aerosol's
// forward fraction (+ 2 if cloudy), the gas depth's derivatives along tlay,
// h2ovmr, o3vmr, the Rayleigh depth's along h2ovmr; with store = 1 also the
// solution's intermediates (1/tau, k, 1/k, exp(-k tau) and 1 less it, 1 -
// exp(-tau/mu0), 1/(zdenr zem1)), which store = 0 makes again.
enum { A_RUP, A_RUPD, A_ALPHA, A_BETA, A_ZR, A_REFD, A_TDIF, A_TRAD, A_DBT, A_ADIR, A_ADIF, A_S, A_SG, A_AB, A_FF,
       A_GT, A_GH, A_GO, A_RH, A_NREC, A_RT = A_NREC, A_K, A_RK, A_E1, A_OM1, A_OM2, A_R, A_NSTORE };
// AD_J in store's place: the pass that only forms J keeps nothing
constexpr int AD_J = -1;
__host__ __device__ inline int ad_fields(int store) { return store == AD_J ? 0 : store ? A_NSTORE : A_NREC; }

struct AdSlot {
    size_t blk, cld, cj, aer, coef3, wat, queue, total;  // doubles; the stored fields come first
};
__host__ __device__ inline AdSlot ad_slot(int L, int store, int nc) {
    AdSlot s;
    size_t o = (size_t)L * ad_fields(store) * (size_t)(nc * NGPT);
    s.blk = o; o += (size_t)nc * L * D_STRIDE;
    s.cld = o; o += (size_t)nc * L * NBND * CO_N;
    s.cj = o;  if (store != AD_J) o += (size_t)nc * L * NBND * CJ_N;
    s.aer = o; o += (size_t)nc * L * NBND * AO_N;
    s.coef3 = o; o += (size_t)nc * L * NFR * 4;  // setcoef in duals
    s.wat = o; o += (size_t)nc * L * 4;          // ciwp, clwp, rei, rel
    s.queue = o; if (store != AD_J) o += ((size_t)nc * NGPT * L + 1) / 2;  // cells for ad_cell (int each)
    s.total = (o + 31) & ~(size_t)31;
    return s;
}

constexpr int AD_KLEV = 4;  // layers per round of gradient sums
struct AdSmem {
    size_t tm, xs, seed, misc, jp, seeds, grad, red, total;
};
__host__ __device__ inline AdSmem ad_smem(int L, int nc, bool value) {
    AdSmem m;
    size_t o = 0;
    m.tm = o;    o = align16(o + NBND * 2 * sizeof(TmSmem));
    m.xs = o;    o = align16(o + NGPT * 32 * sizeof(uint32_t));
    m.seed = o;  o = align16(o + nc * 4 * sizeof(uint32_t));
    m.misc = o;  o = align16(o + (nc + 1) * sizeof(int));  // laytrop per column, queue length
    m.jp = o;    o = align16(o + (size_t)nc * L * sizeof(int));
    m.seeds = o; o = align16(o + (size_t)nc * (L + 1) * 2 * sizeof(double));
    m.grad = o;  if (!value) o = align16(o + (size_t)nc * L * 5 * sizeof(double));
    m.red = o;   o = align16(o + (size_t)(value ? 3 : AD_KLEV * 5) * nc * NGPT * sizeof(double));
    m.total = o;
    return m;
}

// Derivative fields of one (column, layer) whose coefficients setcoef64 has
// written (inatm_sw's amounts, rrtmg_sw_rad.f90:1527-1586, and
// rrtmg_sw_setcoef.f90:158-301, differentiated).
__device__ inline void prep_deriv(const SolveParams& P, int pcol, int lay, int pk, double* blk) {
    const size_t k = (size_t)pcol + (size_t)P.ncol * (size_t)(lay - 1);
    const double amd = 28.9660, amw = 18.0160;
    const double t = P.tlay[k], h = P.h2ovmr[k];
    const double amm = (1.0 - h) * amd + h * amw;
    const double lh = -((amw - amd) / amm + 1.0 / (1.0 + h));
    const double ch = blk[F_H2O], cd = blk[F_MOL] - ch;  // 1e-20 coldry
    const double ff = blk[F_FORFAC];
    const bool low = (pk >> 30) & 1;
    blk[D_T0] = (blk[F_FAC00] + blk[F_FAC10]) / 15.0;
    blk[D_T1] = (blk[F_FAC01] + blk[F_FAC11]) / 15.0;
    blk[D_IT] = 1.0 / t;
    blk[D_LH] = lh;
    blk[D_HW] = cd + ch * lh;
    blk[D_MOLH] = cd * lh + blk[D_HW];
    blk[D_O3O] = cd;
    blk[D_FOH] = -ff / (1.0 + h);
    blk[D_SEH] = low ? ff + h * blk[D_FOH] : 0.0;
    blk[D_FFT] = (low ? -1.0 : 1.0) / 36.0;
}

// .. and of one band of it, after prep_band64
__device__ inline void prep_band_deriv(const SolveParams& P, int pcol, int lay, int b, bool low, double* blk,
                                       double* cj, int mode, const double* __restrict__ tab) {
    const int up = low ? 0 : 1, slot = cT.sslot[b];
    const TmRegion& d = cT.tm[b][up];
    const double comb = blk[B_COMB + b], lh = blk[D_LH];
    double ch = 0.0, fh = 0.0, co = 0.0, fo = 0.0;
    if (d.kind == 1) {
        const double mult = up ? 4.0 : 8.0;
        const double ca = blk[F_H2O + d.sa], p = ca / comb;
        const double ca_h = d.sa == 0 ? blk[D_HW] : ca * lh;
        ch = ca_h + (comb - ca) * lh;
        const bool clamped = p >= cT.oneminus;
        fh = clamped ? 0.0 : mult * (ca_h - p * ch) / comb;
        if (d.sa == 2) {
            co = blk[D_O3O];
            fo = clamped ? 0.0 : mult * co * (1.0 - p) / comb;
        }
    } else if (d.kind == 2) {
        const double fac = cT.fac64[b][up];
        ch = d.sa == 0 ? blk[D_HW] * fac : comb * lh;
        if (d.sa == 2) co = blk[D_O3O] * fac;
    }
    blk[D_COMBH + b] = ch;
    if (slot >= 0) blk[D_FSH + slot] = fh;
    if (b == 11) blk[D_COMBO] = co;
    if (b == 12) {
        blk[D_COMBO + 1] = co;
        blk[D_FSO] = fo;
    }
    if (mode == CLD_MASK) {
        const size_t kl = (size_t)pcol + (size_t)P.ncol * (size_t)(lay - 1);
        if (P.cldfrac[kl] > 0.0) {
            // the optics are sums of a liquid and an ice part, each its
            // optics per unit of water path times the path (fixed when
            // inflgsw = 0, zero where a part has no path or no
            // parametrisation: cloud64 then puts its floor of 1e-20 there)
            const double wl = P.clwp[kl], wi = P.ciwp[kl];
            double* o = cj + b * CJ_N;
            for (int k = 0; k < CJ_N; ++k) o[k] = 0.0;
            const bool on = P.inflag == 2 &&
                            (wl + wi >= 1.e-20 || (P.tauc && P.tauc[(size_t)b + 14 * kl] >= 1.e-20));
            double c[CO_N];
            if (on && wl != 0.0) {
                cloud64(b, P.inflag, P.iceflag, P.liqflag, 1.0, 0.0, 1.0, P.rei[kl], P.rel[kl], 0.0, 0.0, 1.0, 0.0, tab,
                        -1.0, c);
                if (c[CO_TAU] > 1.e-20) {
                    o[CJ_SL] = c[CO_S];
                    o[CJ_GL] = c[CO_SG];
                    o[CJ_AL] = c[CO_AB];
                }
            }
            if (on && wi != 0.0) {
                cloud64(b, P.inflag, P.iceflag, P.liqflag, 1.0, 1.0, 0.0, P.rei[kl], P.rel[kl], 0.0, 0.0, 1.0, 0.0, tab,
                        -1.0, c);
                if (c[CO_TAU] > 1.e-20) {
                    o[CJ_SI] = c[CO_S];
                    o[CJ_GI] = c[CO_SG];
                    o[CJ_AI] = c[CO_AB];
                }
            }
        }
    }
}

// taumol64 with the gas depth's derivatives along tlay, h2ovmr, o3vmr and the
// Rayleigh depth's along h2ovmr.
struct Gas {
    double taug, taur, gt, gh, go, rh;
};
__device__ __forceinline__ Gas taumol_deriv(const TmSmem& t, int ib, int ig, const double* blk,
                                            const double* __restrict__ tab) {
    Gas G{0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    const TmRegion& d = t.r;
    const int ng = t.ng, slot = t.pad;
    const int pk = *(const int*)(blk + B_PK);
    double fs = 0.0, fsh = 0.0;
    int js = 0;
    if (d.kind == 1) {
        fs = blk[B_FS + slot];
        fsh = blk[D_FSH + slot];
        js = ((const unsigned char*)(blk + B_JS))[slot];
    }
    if (d.kind != 0) {
        const int jp = (pk & 0xff) - d.jo, jt = (pk >> 8) & 0xf, jt1 = (pk >> 12) & 0xf;
        const int nsp = d.nsp, two = d.kind == 1 ? ng : 0;
        const int i0 = d.ktab + ((jp * 5 + (jt - 1)) * nsp + js) * ng + ig - 1;
        const int i1 = d.ktab + (((jp + 1) * 5 + (jt1 - 1)) * nsp + js) * ng + ig - 1;
        const int dn = nsp * ng;
        const double a0 = ldt(tab, i0), b0 = ldt(tab, i0 + dn), c0 = ldt(tab, i1), e0 = ldt(tab, i1 + dn);
        const double ad = ldt(tab, i0 + two) - a0, bd = ldt(tab, i0 + dn + two) - b0;
        const double cd = ldt(tab, i1 + two) - c0, ed = ldt(tab, i1 + dn + two) - e0;
        const double p0 = fma(fs, ad, a0), p1 = fma(fs, bd, b0), p2 = fma(fs, cd, c0), p3 = fma(fs, ed, e0);
        const double f00 = blk[F_FAC00], f10 = blk[F_FAC10], f01 = blk[F_FAC01], f11 = blk[F_FAC11];
        const double k = fma(f11, p3, fma(f01, p2, fma(f10, p1, f00 * p0)));
        const double kt = fma(blk[D_T1], p3 - p2, blk[D_T0] * (p1 - p0));
        const double kf = fma(f11, ed, fma(f01, cd, fma(f10, bd, f00 * ad)));
        const double comb = blk[B_COMB + ib], ckf = comb * kf;
        G.taug = comb * k;
        G.gt = comb * kt;
        G.gh = fma(blk[D_COMBH + ib], k, ckf * fsh);
        if (ib == 11) G.go = blk[D_COMBO] * k;
        else if (ib == 12) G.go = fma(blk[D_COMBO + 1], k, ckf * blk[D_FSO]);
    }
    const double h2o = blk[F_H2O], lh = blk[D_LH];
    if (d.cont >= 1) {
        const int indf = (pk >> 24) & 0xf;
        const double fa = ldt(tab, t.forref + (indf - 1) * ng + ig - 1);
        const double fd = ldt(tab, t.forref + indf * ng + ig - 1) - fa;
        const double fp = fma(blk[F_FORFRAC], fd, fa), ff = blk[F_FORFAC];
        double c = ff * fp, ct = ff * blk[D_FFT] * fd, ch = blk[D_FOH] * fp;
        if (d.cont == 1) {
            const int inds = (pk >> 16) & 0xff;
            const double sa = ldt(tab, t.selfref + (inds - 1) * ng + ig - 1);
            const double sd = ldt(tab, t.selfref + inds * ng + ig - 1) - sa;
            const double sp = fma(blk[F_SELFFRAC], sd, sa), sf = blk[F_SELFFAC];
            c = fma(sf, sp, c);
            ct = fma(sf * (1.0 / 7.2), sd, ct);
            ch = fma(blk[D_SEH], sp, ch);
        }
        ct = fma(-blk[D_IT], c, ct);  // forfac and selffac go as 1/tlay
        G.taug = fma(h2o, c, G.taug);
        G.gt = fma(h2o, ct, G.gt);
        G.gh = fma(blk[D_HW], c, fma(h2o, ch, G.gh));
    }
    if (d.minor >= 0) {
        const double v = d.minor == 9 ? 4.35e-4 / 700.0 : ldt(tab, d.mtab + ig - 1);
        const double x = blk[F_H2O + (d.minor == 9 ? 4 : d.minor)];
        G.taug = fma(v, x, G.taug);
        G.gh = fma(v, d.minor == 0 ? blk[D_HW] : x * lh, G.gh);
        if (d.minor == 2) G.go = fma(v, blk[D_O3O], G.go);
    }
    const double mol = blk[F_MOL];
    if (d.rtype == 2) {
        const double r0 = ldt(tab, d.rtab + js * ng + ig - 1), rd = ldt(tab, d.rtab + (js + 1) * ng + ig - 1) - r0;
        const double ra = fma(fs, rd, r0);
        G.taur = mol * ra;
        G.rh = fma(blk[D_MOLH], ra, mol * rd * fsh);
    } else {
        const double ra = ldt(tab, d.rtab + (d.rtype == 1 ? ig - 1 : 0));
        G.taur = mol * ra;
        G.rh = blk[D_MOLH] * ra;
    }
    return G;
}

// The smooth layer solution (two_stream64's form with exp(-x)) from the
// layer's scattering s, s times asymmetry sg and absorption ab: what its
// adjoint needs again.  k = 0 marks conservative scattering; r = 0 the
// reference's replacement of the solution where |zdenr| <= 1e-8.
struct Sol {
    double rt, k, rk, e1, om1, e2, om2, r;
    bool noisy, near;
};
// .. and what follows from those with few operations
struct Mid {
    double w, co, wg, g, h, g1, g2, g3, g4, a1, a2, p1, m1, Y1, Y2, r2, t2, k2, r3, t3, oo, B, N, M, om12, dom, eoo;
};

// |1 - (k mu0)^2| k below which a cell's Jacobian is formed in forward mode in
// the reference's order of operations (ad_cell).  The reference's derivative
// divides rounding by that number and by k, so that the values it gives there
// hold only operation by operation: a gradient of the heating-rate sum moved
// by up to 1e-3 of its largest entry where one of 60 layers sat at 1e-6.  The
// derivative along ozone (bands 24, 25, 27, 28) is the most sensitive.  About a
// tenth of the cells; elsewhere both ways agree to 2e-10 of the gradients'
// 2-norm (30 to 137 layers; with 0.06 / 0.01 to 6e-10, with every cell analytic
// to 4e-6).
constexpr double NOISE_O3 = 0.1, NOISE_AD = 0.03;

template <bool G>
__device__ __forceinline__ Mid sol_mid(const Sol& o, double s, double sg, double ab, const Mu64& m) {
    Mid x;
    x.w = s * o.rt;
    x.co = ab * o.rt;
    x.wg = G ? sg * o.rt : 0.0;
    x.g = G ? sg * rcp64(s) : 0.0;
    const double t4 = G ? fma(-3.0, x.wg, 4.0 - x.w) : 4.0 - x.w;  // 2 (gamma1 + gamma2)
    x.h = 0.25 * t4;
    x.g1 = x.h + x.co;
    x.g2 = x.h - x.co;
    const double v = G ? m.mu34 * x.g : 0.0;
    x.g3 = 0.5 - v;
    x.g4 = 0.5 + v;
    const double u = G ? 2.0 * x.co * v : 0.0;
    x.a1 = x.h + u;
    x.a2 = x.h - u;
    const double km = o.k * m.mu;
    x.p1 = 1.0 + km;
    x.m1 = 1.0 - km;
    x.Y2 = fma(-o.k, x.g3, x.a2);
    x.Y1 = fma(-o.k, x.g4, x.a1);
    x.r2 = x.p1 * x.Y2;
    x.t2 = x.m1 * x.Y1;
    x.k2 = o.k + o.k;
    x.r3 = x.k2 * fma(-x.a2, m.mu, x.g3);
    x.t3 = x.k2 * fma(x.a1, m.mu, x.g4);
    x.oo = fma(o.om1, o.e1, o.om1);
    x.B = fma(x.g1 - o.k, x.oo, x.k2);
    x.om12 = fma(o.e1, o.om2, o.om1);
    x.dom = o.om2 - o.om1;
    x.eoo = o.e2 * x.oo;
    x.N = fma(x.r2, x.oo, x.r3 * x.om12);
    x.M = fma(x.t3, x.dom, -x.t2 * x.eoo);
    return x;
}

// Whether the reference takes the conservative branch (reftra:183-188)
__device__ __forceinline__ bool conservative(double w, double co, double g) {
    double denom = 1.0, zwo = 0.0;
    const float r = to32(co);
    if (g == 0.0) return r < 4.9e-7f || (r < 5.1e-7f && w >= 0.9999995);
    if (g != 1.0) {
        const double q = g * rcp64(1.0 - g);
        denom = 1.0 - (1.0 - w) * (q * q);
    }
    if (w > 0.0 && denom != 0.0) zwo = w / denom;
    return zwo >= 0.9999995;
}

// The solution and its intermediates.  Not inlined: both passes run the same
// code, so that recomputed intermediates equal the stored ones.
template <bool G>
__device__ __noinline__ void sol_forward(double s, double sg, double ab, const Mu64& m, double noise,
                                         const double* __restrict__ tab, Sol& o, Rt64& out) {
    const double tau = s + ab;
    o.rt = rcp64(tau);
    expm64(clip500(tau * m.rmu), tab, o.e2, o.om2);
    const double w = s * o.rt, co = ab * o.rt, wg = G ? sg * o.rt : 0.0;
    const double g = G ? sg * rcp64(s) : 0.0;
    o.k = o.rk = o.r = 0.0;
    o.noisy = o.near = false;
    o.e1 = 1.0;
    o.om1 = 0.0;
    if (conservative(w, co, g)) {
        const double g1 = fma(-1.25, w, fma(-0.75, wg, 2.0)), g3 = fma(-m.mu34, g, 0.5);
        const double gt = g1 * tau, r1 = rcp64(1.0 + gt);
        out.ref = fma(-fma(g1, m.mu, -g3), o.om2, gt) * r1;
        out.refd = gt * r1;
        out.trad = 1.0 - out.refd;
        out.tdif = o.om2 - out.ref;
        out.dbt = o.e2;
        return;
    }
    root64(co * (G ? fma(-3.0, wg, 4.0 - w) : 4.0 - w), o.k, o.rk);
    expm64(clip500(o.k * tau), tab, o.e1, o.om1);
    const Mid x = sol_mid<G>(o, s, sg, ab, m);
    const double pp = x.p1 * x.m1, pB = pp * x.B;
    o.noisy = lt_pos(fabs(pp) * o.k, noise);
    o.near = lt_pos(fabs(pp), RESONANCE64 * w);
    double rB;
    if (fabs(pB) > 1.e-8 * o.e1) {
        o.r = rcp64(pB);
        rB = o.r * pp;
    } else {
        rB = rcp64(x.B);
    }
    const double wr = x.w * o.r;
    out.ref = o.r != 0.0 ? wr * x.N : 1.e-8;
    out.tdif = wr * x.M;
    out.refd = x.g2 * x.oo * rB;
    out.trad = x.k2 * o.e1 * rB;
    out.dbt = o.e2;
}

// Adjoint of the solution: from those of ref, refd, tdif, trad, dbt (b) to
// those of s, sg, ab.
template <bool G>
__device__ __forceinline__ void sol_adjoint(const Sol& o, double s, double sg, double ab, const Mu64& m, const Rt64& b,
                                            double& sb, double& sgb, double& abb) {
    double wb, cob = 0.0, wgb, gb, taub;
    const double tau = s + ab;
    const double w = s * o.rt, co = ab * o.rt, wg = G ? sg * o.rt : 0.0;
    double rs = 0.0, g = 0.0;
    if constexpr (G) {
        rs = rcp64(s);
        g = sg * rs;
    }
    if (o.k == 0.0) {
        const double g1 = fma(-1.25, w, fma(-0.75, wg, 2.0)), g3 = fma(-m.mu34, g, 0.5);
        const double gt = g1 * tau, r1 = rcp64(1.0 + gt), za = fma(g1, m.mu, -g3);
        const double refb = b.ref - b.tdif, refdb = b.refd - b.trad;
        const double ref = fma(-za, o.om2, gt) * r1, refd = gt * r1;
        const double nb = refb * r1;
        const double gtb = nb + refdb * r1 - (refb * ref + refdb * refd) * r1;
        const double om2b = b.tdif - nb * za, zab = -nb * o.om2;
        const double g1b = fma(zab, m.mu, gtb * tau);
        const double x2b = (om2b - b.dbt) * o.e2;
        taub = fma(gtb, g1, x2b * m.rmu);
        wb = -1.25 * g1b;
        wgb = -0.75 * g1b;
        gb = m.mu34 * zab;  // g3 = 1/2 - 3 mu0 g / 4, za = .. - g3
    } else {
        const Mid x = sol_mid<G>(o, s, sg, ab, m);
        const double pp = x.p1 * x.m1;
        double rB, ppb = 0.0, Q = 0.0, Nb = 0.0, Mb = 0.0;
        wb = 0.0;
        if (o.r != 0.0) {
            rB = o.r * pp;
            const double wr = w * o.r, S = fma(b.ref, x.N, b.tdif * x.M);
            Nb = b.ref * wr;
            Mb = b.tdif * wr;
            wb = S * o.r;
            Q = wb * w;
            ppb = -Q * (o.r * x.B);
        } else {
            rB = rcp64(x.B);
        }
        const double dB = b.refd * rB, eB = b.trad * rB;
        const double refd = x.g2 * x.oo * rB, trad = x.k2 * o.e1 * rB;
        const double Bb = -(Q + fma(b.refd, refd, b.trad * trad)) * rB;
        double g2b = dB * x.oo, oob = dB * x.g2;
        double kb = 2.0 * eB * o.e1, e1b = eB * x.k2;
        // N = r2 oo + r3 om12, M = t3 dom - t2 e2 oo
        const double r2b = Nb * x.oo, r3b = Nb * x.om12, om12b = Nb * x.r3;
        const double t3b = Mb * x.dom, domb = Mb * x.t3, meo = Mb * x.oo;
        const double t2b = -meo * o.e2;
        double e2b = fma(-meo, x.t2, b.dbt);
        oob = fma(Nb, x.r2, fma(-Mb * o.e2, x.t2, oob));
        double om1b = om12b - domb;
        const double om2b = fma(om12b, o.e1, domb);
        e1b = fma(om12b, o.om2, e1b);
        // B = 2 k + (g1 - k) oo
        oob = fma(Bb, x.g1 - o.k, oob);
        kb = fma(Bb, 2.0 - x.oo, kb);
        const double g1b = Bb * x.oo;
        // oo = om1 (1 + e1); exp(-x)
        om1b = fma(oob, 1.0 + o.e1, om1b);
        e1b = fma(oob, o.om1, e1b);
        const double x1b = (om1b - e1b) * o.e1, x2b = (om2b - e2b) * o.e2;
        // r2 = p1 Y2, t2 = m1 Y1, r3 = 2 k (g3 - a2 mu), t3 = 2 k (g4 + a1 mu), pp = p1 m1
        const double Y2b = r2b * x.p1, Y1b = t2b * x.m1;
        const double p1b = fma(ppb, x.m1, r2b * x.Y2), m1b = fma(ppb, x.p1, t2b * x.Y1);
        const double z3b = r3b * x.k2, z4b = t3b * x.k2;
        kb = fma(fma(r3b, x.r3, t3b * x.t3), o.rk, kb);
        kb = fma(-Y2b, x.g3, fma(-Y1b, x.g4, kb));
        kb = fma(m.mu, p1b - m1b, kb);
        const double a2b = fma(-z3b, m.mu, Y2b), a1b = fma(z4b, m.mu, Y1b);
        double hb = a1b + a2b + g1b + g2b;
        cob = g1b - g2b;
        gb = 0.0;
        if constexpr (G) {
            const double da = 2.0 * (a1b - a2b), v = m.mu34 * g;
            cob = fma(da, v, cob);
            const double vb = fma(da, co, (z4b - Y1b * o.k) - (z3b - Y2b * o.k));
            gb = vb * m.mu34;
        }
        kb = fma(x1b, tau, kb);
        taub = fma(x1b, o.k, x2b * m.rmu);
        const double Xb = 0.5 * kb * o.rk;  // k^2 = co t4
        const double t4 = 4.0 * x.h;
        cob = fma(Xb, t4, cob);
        const double t4b = fma(Xb, co, 0.25 * hb);
        wb -= t4b;
        wgb = -3.0 * t4b;
    }
    double z = fma(wb, w, cob * co);
    if constexpr (G) z = fma(wgb, wg, z);
    taub = fma(-o.rt, z, taub);
    sb = fma(wb, o.rt, taub);
    abb = fma(cob, o.rt, taub);
    sgb = 0.0;
    if constexpr (G) {
        const double gs = gb * rs;
        sgb = fma(wgb, o.rt, gs);
        sb = fma(-gs, g, sb);
    }
}

// VALUE: J alone, for the tangent (no derivatives, nothing stored), by the same
// functions in the same order, so that J is the adjoint's bit for bit.  160
// FP64 instructions per cell, a tenth of k_tangent's: 2 048 x 60 columns 7 ms.
template <int NC, bool VALUE>
__global__ void __launch_bounds__(NC * NGPT, 4 / NC)
k_adjoint(const SolveParams P, const AdParams A, const double* __restrict__ tab) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr int NT = NC * NGPT;
    const int L = P.nlay, tid = threadIdx.x;
    const AdSmem M = ad_smem(L, NC, VALUE);
    const int store = VALUE ? AD_J : A.store;
    TmSmem* sTm = (TmSmem*)(smem_raw + M.tm);
    uint32_t* sXs = (uint32_t*)(smem_raw + M.xs);
    uint32_t* sSeed = (uint32_t*)(smem_raw + M.seed);
    int* sLt = (int*)(smem_raw + M.misc);
    int* sPk = (int*)(smem_raw + M.jp);
    double* sSeeds = (double*)(smem_raw + M.seeds);
    double* sRed = (double*)(smem_raw + M.red);
    double* sGrad = (double*)(smem_raw + M.grad);  // [NC][L][5]
    const int cc = tid / NGPT, g = tid % NGPT, ib = cT.ngb[g], igb = cT.gib[g];
    const bool nir = ib <= 8 || ib == 13;
    const double noise = ib == 8 || ib == 9 || ib == 11 || ib == 12 ? NOISE_O3 : NOISE_AD;
    const int mode = cloud_mode(P), NF = ad_fields(store);
    const AdSlot S = ad_slot(L, store, NC);
    double* slot = (double*)P.scratch + (size_t)blockIdx.x * P.slot_elems;
    double *blk0 = slot + S.blk, *cld0 = slot + S.cld, *cj0 = slot + S.cj, *aer0 = slot + S.aer, *wat0 = slot + S.wat;
    Dual<3>* coef30 = (Dual<3>*)(slot + S.coef3);
    int* queue = (int*)(slot + S.queue);
    const size_t n = (size_t)P.ncol;
    fill_tm64(sTm);
    const KissJump J = kiss_setup(P, sXs, g);
    const int groups = (P.ncol + NC - 1) / NC;
    for (int grp = blockIdx.x; grp < groups; grp += gridDim.x) {
        __syncthreads();
        if (tid <= NC) sLt[tid] = 0;
        __syncthreads();
        for (int it = tid; it < NC * L; it += NT) {
            const int c2 = it / L, lay = it % L + 1, pcol = NC * grp + c2;
            double* blk = blk0 + (size_t)it * D_STRIDE;
            const int pk = setcoef64(P, pcol, lay, blk, tab);
            sPk[it] = pk;
            if (pcol >= P.ncol) continue;
            if constexpr (!VALUE) prep_deriv(P, pcol, lay, pk, blk);
            prep_layer_dual(P, pcol, lay, coef30 + (size_t)c2 * NFR * L, L, sPk + c2 * L, tab);
            if (mode == CLD_MASK) {
                const size_t kl = (size_t)pcol + n * (size_t)(lay - 1);
                double* wt = wat0 + (size_t)c2 * 4 * L + lay - 1;
                wt[0 * L] = P.ciwp[kl];
                wt[1 * L] = P.clwp[kl];
                wt[2 * L] = P.rei[kl];
                wt[3 * L] = P.rel[kl];
            }
            if ((pk >> 30) & 1) atomicAdd(sLt + c2, 1);
            if (mode == CLD_MASK) {
                thresholds64<false>(P, pcol, lay, blk + B_TH);
                if (lay == 1) seeds64(P, pcol, sSeed + c2 * 4);
            }
        }
        // objective seeds of each level (0 = surface .. L = top), without the incident flux
        for (int it = tid; it < NC * (L + 1); it += NT) {
            const int c2 = it / (L + 1), l = it % (L + 1), pcol = NC * grp + c2;
            if (pcol >= P.ncol) continue;
            const double* pl = P.plev + pcol;
            double an = 0.0;  // dJ/d net(l) through the heating-rate sum (layers 0 .. L-2)
            if (l >= 1 && l - 1 <= L - 2) an += A.w_hr * cT.heatfac / (pl[n * (l - 1)] - pl[n * l]);
            if (l <= L - 2) an -= A.w_hr * cT.heatfac / (pl[n * l] - pl[n * (l + 1)]);
            sSeeds[2 * it] = -an + (l == L ? A.w_toa : 0.0) - (l == 0 ? A.w_net : 0.0);  // up
            sSeeds[2 * it + 1] = an + (l == 0 ? A.w_net : 0.0);                          // down
        }
        __syncthreads();
        for (int it = tid; it < NC * L * NBND; it += NT) {
            const int b = it % NBND, cl = it / NBND, c2 = cl / L, lay = cl % L + 1, pcol = NC * grp + c2;
            if (pcol >= P.ncol) continue;
            double* blk = blk0 + (size_t)cl * D_STRIDE;
            const bool low = lay <= sLt[c2];
            prep_band64(P, pcol, lay, b, low, blk, cld0 + (size_t)cl * NBND * CO_N, aer0 + (size_t)cl * NBND * AO_N,
                        mode, false, tab);
            if constexpr (!VALUE)
                prep_band_deriv(P, pcol, lay, b, low, blk, cj0 + (size_t)cl * NBND * CJ_N, mode, tab);
        }
        __syncthreads();
        const int col = NC * grp + cc, laytrop = sLt[cc];
        bool active = col < P.ncol;
        if (active && (laytrop < 1 || laytrop >= L)) {
            set_error(P.err, E_LAYTROP);
            active = false;
        }
        const double* blkc = blk0 + (size_t)cc * L * D_STRIDE;
        const double* seeds = sSeeds + (size_t)cc * (L + 1) * 2;
        double* sv0 = slot + tid;
        Mu64 m{1.0, 1.0, 0.75};
        double zinc = 0.0, zh = 0.0, zo = 0.0, albp = 0.0, albd = 0.0, phi = 0.0;
        int lsol = -1;
        if (active) {
            m.mu = P.coszen[col];
            if (m.mu < 1.e-10) m.mu = 1.e-10;
            m.rmu = 1.0 / m.mu;
            m.mu34 = 0.75 * m.mu;
            albp = nir ? P.aldir[col] : P.asdir[col];
            albd = nir ? P.aldif[col] : P.asdif[col];
            double zf = 0.0;
            zinc = solar64(ib, igb, blkc, D_STRIDE, sPk + cc * L, L, laytrop, P, tab, &lsol, &zf);
            const double am = P.adjflux[ib] * m.mu;
            zinc *= am;
            if (!VALUE && lsol >= 1 && cT.sslot[ib] >= 1) {
                const double* b = blkc + (size_t)(lsol - 1) * D_STRIDE;
                zh = am * zf * b[D_FSH + cT.sslot[ib]];
                zo = ib == 12 ? am * zf * b[D_FSO] : 0.0;
            } else {
                lsol = -1;
            }
            Mask64<false> mc;
            if (mode == CLD_MASK) mc.m.start(kiss_start(sSeed + cc * 4, J, sXs + g * 32), P.icld);
            // ---------------- bottom -> top
            double ru = albp, rud = albd;
            double ad = fma(seeds[0], albp, seeds[1]), af = fma(seeds[0], albd, seeds[1]);
#pragma unroll 1
            for (int lay = 1; lay <= L; ++lay) {
                const size_t cl = (size_t)(cc * L + lay - 1);
                const double* blk = blk0 + cl * D_STRIDE;
                const bool cloudy = mode == CLD_MASK && mc.step(lay, blk + B_TH);
                const TmSmem& tm = sTm[ib * 2 + (lay <= laytrop ? 0 : 1)];
                Gas G;
                if constexpr (VALUE) taumol64(tm, ib, igb, blk, tab, G.taug, G.taur);
                else G = taumol_deriv(tm, ib, igb, blk, tab);
                double s = G.taur, sg = 0.0, ab = G.taug, ff = 0.0;
                if (P.iaer != 0) {
                    const double* a = aer0 + cl * NBND * AO_N + ib * AO_N;
                    s += a[AO_S];
                    sg = a[AO_SG];
                    ab += a[AO_AB];
                    const double g0 = sg * rcp64(s), d = sg * g0;
                    ff = g0 * g0;
                    s -= d;
                    sg -= d;
                }
                Sol o;
                Rt64 r;
                if (cloudy) {
                    const double* c = cld0 + cl * NBND * CO_N + ib * CO_N;
                    if (__double_as_longlong(c[CO_ERR]) != 0ll) set_error(P.err, (int)c[CO_ERR]);
                    s += c[CO_S];
                    sg += c[CO_SG];
                    ab += c[CO_AB];
                }
                if (cloudy || P.iaer != 0) sol_forward<true>(s, sg, ab, m, noise, tab, o, r);
                else sol_forward<false>(s, sg, ab, m, noise, tab, o, r);
                if (o.near) {
                    // at the resonance the solution too keeps the reference's order of operations
                    Dual<5> jac[5];
                    ad_cell(P, coef30 + (size_t)cc * NFR * L, sPk + cc * L, L, laytrop, col, lay, ib, igb, cloudy,
                            wat0 + (size_t)cc * 4 * L, m.mu, tab, jac);
                    r.ref = jac[0].v;
                    r.refd = jac[1].v;
                    r.tdif = jac[2].v - jac[4].v;
                    r.trad = jac[3].v;
                    r.dbt = jac[4].v;
                }
                double* sv = sv0 + (size_t)(lay - 1) * NF * NT;
                if constexpr (!VALUE) {
                    sv[A_ADIR * NT] = ad;
                    sv[A_ADIF * NT] = af;
                }
                // up64, keeping its reciprocal
                const double zr = rcp64(fma(-rud, r.refd, 1.0)), x = r.dbt * ru;
                const double beta = r.trad * zr, alpha = fma(r.refd, x, r.tdif) * zr;
                ru = fma(beta, fma(r.tdif, rud, x), r.ref);
                rud = fma(beta, r.trad * rud, r.refd);
                // the fluxes at the layer's top: their part of J below, then this level's
                const double sU = seeds[2 * lay], sD = seeds[2 * lay + 1];
                ad = fma(af, alpha, fma(ad, r.dbt, fma(sU, ru, sD)));
                af = fma(af, beta, fma(sU, rud, sD));
                if constexpr (!VALUE) {
                    sv[A_RUP * NT] = ru;
                    sv[A_RUPD * NT] = rud;
                    sv[A_ALPHA * NT] = alpha;
                    sv[A_BETA * NT] = beta;
                    sv[A_ZR * NT] = zr;
                    sv[A_REFD * NT] = r.refd;
                    sv[A_TDIF * NT] = r.tdif;
                    sv[A_TRAD * NT] = r.trad;
                    sv[A_DBT * NT] = r.dbt;
                    sv[A_S * NT] = s;
                    sv[A_SG * NT] = sg;
                    sv[A_AB * NT] = ab;
                    sv[A_FF * NT] = ff + (cloudy ? 2.0 : 0.0) + (o.noisy ? 4.0 : 0.0);
                    sv[A_GT * NT] = G.gt;
                    sv[A_GH * NT] = G.gh;
                    sv[A_GO * NT] = G.go;
                    sv[A_RH * NT] = G.rh;
                    if (A.store) {
                        sv[A_RT * NT] = o.rt;
                        sv[A_K * NT] = o.k;
                        sv[A_RK * NT] = o.rk;
                        sv[A_E1 * NT] = o.e1;
                        sv[A_OM1 * NT] = o.om1;
                        sv[A_OM2 * NT] = o.om2;
                        sv[A_R * NT] = o.r;
                    }
                }
            }
            phi = ad;
        }
        // ---------------- top -> bottom
        double dir = zinc, dif = 0.0, cu = 0.0, cud = 0.0;
        for (int lay = VALUE ? 0 : L; lay >= 1; --lay) {
            double q[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
            if (active) {
                const size_t cl = (size_t)(cc * L + lay - 1);
                const double* sv = sv0 + (size_t)(lay - 1) * NF * NT;
                const double rub = lay > 1 ? sv[(A_RUP - NF) * NT] : albp, rudb = lay > 1 ? sv[(A_RUPD - NF) * NT] : albd;
                const double refd = sv[A_REFD * NT], tdif = sv[A_TDIF * NT], trad = sv[A_TRAD * NT], dbt = sv[A_DBT * NT];
                const double alpha = sv[A_ALPHA * NT], beta = sv[A_BETA * NT], zr = sv[A_ZR * NT];
                const double adb = sv[A_ADIR * NT], afb = sv[A_ADIF * NT];
                if (lay > 1) {
#pragma unroll
                    for (int f = 0; f < A_NREC; ++f) asm volatile("prefetch.global.L1 [%0];" ::"l"(sv + (f - NF) * NT));
                }
                const double sU = seeds[2 * lay];
                // adjoints of the albedos at the layer's top, of alpha and beta
                const double rb = fma(sU, dir, cu), rdb = fma(sU, dif, cud);
                const double alb = afb * dir;
                double beb = afb * dif;
                const double x = dbt * rub, E = fma(tdif, rudb, x), tr = trad * rudb;
                beb = fma(rb, E, fma(rdb, tr, beb));
                const double Eb = rb * beta, az = alb * zr, rbeta = rdb * beta;
                const double xb = fma(az, refd, Eb);
                const double z2 = zr * fma(alb, alpha, beb * beta);
                Rt64 b;
                b.ref = rb;
                b.tdif = fma(Eb, rudb, az);
                b.trad = fma(rbeta, rudb, beb * zr);
                b.refd = fma(az, x, fma(z2, rudb, rdb));
                b.dbt = fma(xb, rub, adb * dir);
                cu = xb * dbt;
                cud = fma(Eb, tdif, fma(rbeta, trad, z2 * refd));
                const double dif1 = fma(alpha, dir, beta * dif);
                dir *= dbt;
                dif = dif1;
                // the layer solution's adjoint
                const double s = sv[A_S * NT], sg = sv[A_SG * NT], ab = sv[A_AB * NT];
                double ffc = sv[A_FF * NT];
                const bool noisy = le_pos(4.0, ffc);
                if (noisy) ffc -= 4.0;
                const bool cloudy = le_pos(2.0, ffc);
                if (noisy) {
                    // left for the dense pass below: the adjoints of ref, refd, tra, trad, dbt
                    double* w = sv0 + (size_t)(lay - 1) * NF * NT;
                    w[(A_ALPHA + 0) * NT] = b.ref;
                    w[(A_ALPHA + 1) * NT] = b.refd;
                    w[(A_ALPHA + 2) * NT] = b.tdif;
                    w[(A_ALPHA + 3) * NT] = b.trad;
                    w[(A_ALPHA + 4) * NT] = b.dbt - b.tdif;
                    const unsigned mask = __activemask();
                    const int lane = tid & 31, lead = __ffs(mask) - 1;
                    int base = 0;
                    if (lane == lead) base = atomicAdd(sLt + NC, __popc(mask));
                    base = __shfl_sync(mask, base, lead);
                    queue[base + __popc(mask & ((1u << lane) - 1u))] = (lay << 10) | (tid << 1) | (cloudy ? 1 : 0);
                } else {
                    Sol o;
                    Rt64 unused;
                    double sb, sgb, abb;
                    if (A.store) {
                        o.rt = sv[A_RT * NT];
                        o.k = sv[A_K * NT];
                        o.rk = sv[A_RK * NT];
                        o.e1 = sv[A_E1 * NT];
                        o.om1 = sv[A_OM1 * NT];
                        o.om2 = sv[A_OM2 * NT];
                        o.r = sv[A_R * NT];
                        o.e2 = dbt;
                    }
                    if (cloudy || P.iaer != 0) {
                        if (!A.store) sol_forward<true>(s, sg, ab, m, noise, tab, o, unused);
                        sol_adjoint<true>(o, s, sg, ab, m, b, sb, sgb, abb);
                    } else {
                        if (!A.store) sol_forward<false>(s, sg, ab, m, noise, tab, o, unused);
                        sol_adjoint<false>(o, s, sg, ab, m, b, sb, sgb, abb);
                    }
                    double taurb = sb;
                    if (P.iaer != 0) {
                        // the aerosol's delta scaling moves ff of a change of Rayleigh depth
                        const double ff = cloudy ? ffc - 2.0 : ffc;
                        taurb = fma(ff, sb + sgb, sb);
                    }
                    q[0] = abb * sv[A_GT * NT];
                    q[1] = fma(abb, sv[A_GH * NT], taurb * sv[A_RH * NT]);
                    q[2] = abb * sv[A_GO * NT];
                    if (cloudy) {
                        const double* c = cj0 + cl * NBND * CJ_N + ib * CJ_N;
                        q[3] = fma(sb, c[CJ_SL], fma(sgb, c[CJ_GL], abb * c[CJ_AL]));
                        q[4] = fma(sb, c[CJ_SI], fma(sgb, c[CJ_GI], abb * c[CJ_AI]));
                    }
                }
                if (lay == lsol) {
                    // the solar source's interpolation in this layer's species ratio
                    q[1] = fma(phi, zh, q[1]);
                    q[2] = fma(phi, zo, q[2]);
                }
            }
            const int nd = mode == CLD_MASK ? 5 : 3;
            const int r = (L - lay) % AD_KLEV;
            for (int k = 0; k < nd; ++k) sRed[(r * 5 + k) * NT + tid] = q[k];
            if (r == AD_KLEV - 1 || lay == 1) {
                __syncthreads();
                // sums over g-points: four runs of 28, then the runs
                const int items = NC * nd * (r + 1);
                for (int base = 0; base < items * 4; base += NT) {
                    const int t = base + tid, item = t >> 2, part = t & 3;
                    double v = 0.0;
                    const int c2 = item % NC, d = (item / NC) % nd, rr = item / (NC * nd);
                    if (item < items) {
                        const double* src = sRed + (rr * 5 + d) * NT + c2 * NGPT + part * 28;
#pragma unroll 4
                        for (int j = 0; j < 28; ++j) v += src[j];
                    }
                    warp_sum4(v);
                    if (item < items && part == 0) sGrad[((size_t)c2 * L + lay + r - rr - 1) * 5 + d] = v;
                }
                __syncthreads();
            }
        }
        // the cells left to ad_cell, one per thread: its Jacobian contracted
        // (order of the sums over a layer's cells not fixed)
        {
            const int nq = VALUE ? 0 : sLt[NC];
            for (int i = tid; i < nq; i += NT) {
                const int e = queue[i], t = (e >> 1) & 511, lay = e >> 10, c2 = t / NGPT, gg = t % NGPT;
                const double* w = slot + (size_t)(lay - 1) * NF * NT + t;
                const int pcol = NC * grp + c2;
                double cz = P.coszen[pcol];
                if (cz < 1.e-10) cz = 1.e-10;
                Dual<5> jac[5];
                ad_cell(P, coef30 + (size_t)c2 * NFR * L, sPk + c2 * L, L, sLt[c2], pcol, lay, cT.ngb[gg], cT.gib[gg],
                        e & 1, wat0 + (size_t)c2 * 4 * L, cz, tab, jac);
                const int nd = mode == CLD_MASK ? 5 : 3;
                for (int d = 0; d < nd; ++d) {
                    double v = 0.0;
#pragma unroll
                    for (int k = 0; k < 5; ++k) v += w[(A_ALPHA + k) * NT] * jac[k].d[d];
                    if (v != 0.0) atomicAdd(&sGrad[((size_t)c2 * L + lay - 1) * 5 + d], v);
                }
            }
        }
        __syncthreads();
        for (int it = tid; it < NC * L; it += NT) {
            const int ocol = NC * grp + it / L;
            if (ocol >= P.ncol) continue;
            for (int d = 0; d < 5 && !VALUE; ++d)
                if (A.g[d])
                    A.g[d][(size_t)ocol + n * (size_t)(it % L)] =
                        d < 3 || mode == CLD_MASK ? sGrad[(size_t)it * 5 + d] : 0.0;
        }
        // surface albedos and J
        sRed[0 * NT + tid] = fma(seeds[0], dir, cu);
        sRed[1 * NT + tid] = fma(seeds[0], dif, cud);
        sRed[2 * NT + tid] = zinc * phi;
        if (!active) sRed[tid] = sRed[NT + tid] = sRed[2 * NT + tid] = 0.0;
        __syncthreads();
        for (int base = 0; base < NC * 5 * 4; base += NT) {
            const int t = base + tid, item = t >> 2, part = t & 3, c2 = item / 5, a = item % 5;
            double v = 0.0;
            if (item < NC * 5) {
                // asdir, asdif (other bands), aldir, aldif (near infrared), J
                const double* src = sRed + (a == 4 ? 2 : a & 1) * NT + c2 * NGPT;
                for (int j = part * 28; j < part * 28 + 28; ++j) {
                    const int b = cT.ngb[j];
                    if (a == 4 || (b <= 8 || b == 13) == (a >= 2)) v += src[j];
                }
            }
            warp_sum4(v);
            const int ocol = NC * grp + c2;
            if (item < NC * 5 && part == 0 && ocol < P.ncol) {
                if (a == 4) {
                    if (A.J) A.J[ocol] = v;
                } else if (!VALUE && A.ga[a]) {
                    A.ga[a][ocol] = v;
                }
            }
        }
    }
}

}  // namespace rrsw
