// fp64.cuh -- the plain FP64 form's solve kernels: the fused kernel (a CTA per
// column group, persistent), its batch variant, and the split kernels of
// small calls (fp64_cell.cuh holds what a cell computes).
#pragma once

#include "fp64_cell.cuh"

namespace rrsw {

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
        zinc = P.adjflux[ib] * solar64(ib, igb, blkc, B_STRIDE, V.jp + cc * L, L, laytrop, P, tab) * m.mu;
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
    return kiss_start(seed, kiss_jump_consts(n), xorshift_at(n, seed[1]));
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
// err_host: where one thread leaves the error word, which only k_cells64
// writes; a copy of its own would cost a small call a few microseconds.
__global__ void __launch_bounds__(SWEEP_THREADS)
k_sweep64(const SolveParams P, const double* __restrict__ tab, int* err_host) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    if (err_host && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) *(volatile int*)err_host = *P.err;
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
        zinc = P.adjflux[ib] * solar64(ib, igb, blkc, B_STRIDE, pk, L, laytrop, P, tab) * mu;
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
