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
    a.smem = ad_smem(P.nlay, COLS_PER_CTA).total;
    a.slot_elems = ad_slot(P.nlay, store, COLS_PER_CTA).total;
    a.grid = resident_grid(k_adjoint<COLS_PER_CTA>, a.smem, P.npairs, num_sms);
    a.scratch = (size_t)a.grid * a.slot_elems * sizeof(double);
    if (tl) {
        a.tl_smem = tl_smem_layout(P.nlay).total;
        a.tl_slot_elems = tl_slot_elems(P.nlay);
        a.tl_grid = resident_grid(k_tangent, a.tl_smem, P.npairs, num_sms);
        const size_t need = (size_t)a.tl_grid * a.tl_slot_elems * sizeof(double);
        if (need > a.scratch) a.scratch = need;
    }
    return a;
}

cudaError_t launch_adjoint(SolveParams P, const AdParams& A, const double* tab64, const AdPlan& a, cudaStream_t s) {
    if (A.tl) {
        P.slot_elems = a.tl_slot_elems;
        k_tangent<<<a.tl_grid, CTA_THREADS, a.tl_smem, s>>>(P, A, tab64);
    }
    P.slot_elems = a.slot_elems;
    k_adjoint<COLS_PER_CTA><<<a.grid, CTA_THREADS, a.smem, s>>>(P, A, tab64);
    return cudaGetLastError();
}

}  // namespace rrsw
