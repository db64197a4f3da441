// solve_ad.cu -- tangent-linear and adjoint of the FP64 column solve (see ad.cuh).
#include "ad.cuh"
#include "launch.h"

namespace rrsw {

// every translation unit has its own copy of the constant tables
cudaError_t upload_tables_ad(const DevTables& t) { return cudaMemcpyToSymbol(cT, &t, sizeof(DevTables)); }

// CTAs of a persistent launch over the call's column pairs
template <typename K>
static int resident_grid(K kern, size_t smem, int npairs, int num_sms) {
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, CTA_THREADS, smem);
    if (per_sm < 1) per_sm = 1;
    int grid = num_sms * per_sm;
    if (grid > npairs) grid = npairs;
    return grid < 1 ? 1 : grid;
}

AdPlan plan_adjoint(const SolveParams& P, int tl, int store, int num_sms) {
    AdPlan a;
    const auto kern = tl ? k_adjoint<COLS_PER_CTA, true> : k_adjoint<COLS_PER_CTA, false>;
    a.smem = ad_smem(P.nlay, COLS_PER_CTA, tl != 0).total;
    a.slot_elems = ad_slot(P.nlay, tl ? AD_J : store, COLS_PER_CTA).total;
    a.grid = resident_grid(kern, a.smem, P.npairs, num_sms);
    a.scratch = (size_t)a.grid * a.slot_elems * sizeof(double);
    if (tl) {
        a.tl_smem = tl_smem_layout(P.nlay).total;
        a.tl_slot_elems = tl_slot_elems(P.nlay);
        a.tl_grid = resident_grid(k_tangent, a.tl_smem, P.npairs, num_sms);
        a.tl_scratch = a.scratch;
        a.scratch += (size_t)a.tl_grid * a.tl_slot_elems * sizeof(double);
    }
    return a;
}

cudaError_t launch_adjoint(SolveParams P, const AdParams& A, const double* tab64, const AdPlan& a, cudaStream_t s) {
    P.slot_elems = a.slot_elems;
    if (A.tl) k_adjoint<COLS_PER_CTA, true><<<a.grid, CTA_THREADS, a.smem, s>>>(P, A, tab64);
    else k_adjoint<COLS_PER_CTA, false><<<a.grid, CTA_THREADS, a.smem, s>>>(P, A, tab64);
    return cudaGetLastError();
}

cudaError_t launch_tangent(SolveParams P, const AdParams& A, const double* tab64, const AdPlan& a, cudaStream_t s) {
    P.scratch = (char*)P.scratch + a.tl_scratch;
    P.slot_elems = a.tl_slot_elems;
    k_tangent<<<a.tl_grid, CTA_THREADS, a.tl_smem, s>>>(P, A, tab64);
    return cudaGetLastError();
}

}  // namespace rrsw
