// newton_step.cu -- one quasi-Newton step (NewtonSteps.py:217-246) as one call.
//
// The step's kernels are the ones of the separate entry points, in the same
// order; this only issues them from native code and hands the step's three
// scalars to the host.  Issued one by one through the Python binding, the
// fourteen launches and copies of a step took longer than a small problem's
// kernels run (L=48, q=4, 2^14 sequences: 207 us a step, 95 us of it kernels).
#include "common.cuh"

namespace mi3 {

// {sum w, sum w^2, min(0, dE), status} straight into pinned host memory: one
// launch instead of three copies.
__global__ void k_newton_report(const double *__restrict__ wstats64, const float *__restrict__ minout,
                                const int32_t *__restrict__ status, double *host_out) {
    host_out[0] = wstats64[0];
    host_out[1] = wstats64[1];
    host_out[2] = (double)*minout;
    host_out[3] = (double)*status;
}

}  // namespace mi3

using namespace mi3;

extern "C" int mi3_newton_step(const mi3_newton_args *a, float ref_E, void *stream) {
    if (!a) return fail(MI3_ERR_ARG, "mi3_newton_step: null pointer");
    if (!a->host_out || !a->event || !a->status || !a->weight_stats64)
        return fail(MI3_ERR_ARG, "mi3_newton_step: null pointer");
    if (a->reg < 0 || a->reg > 2) return fail(MI3_ERR_ARG, "mi3_newton_step: reg must be 0, 1 or 2");
    int rc = mi3_update_j(a->bi_target, a->bi, a->gamma, a->pc, a->dJ, a->dJ, a->L, a->q, stream);
    if (rc == MI3_OK && a->reg == 1) rc = mi3_reg_l1z(a->bi, a->gamma, a->pc, a->lJ, a->J, a->dJ, a->L, a->q, stream);
    if (rc == MI3_OK && a->reg == 2) rc = mi3_reg_l2z(a->bi, a->gamma, a->pc, a->lJ, a->J, a->dJ, a->L, a->q, stream);
    if (rc == MI3_OK)
        rc = mi3_energies(a->dJ, a->seqmem, a->buflen, a->nseq, a->energies, a->L, a->q, a->ws_energies,
                          a->ws_energies_bytes, stream);
    if (rc == MI3_OK)
        rc = mi3_weights_fused(ref_E, a->energies, a->weights, a->nseq, a->minout, a->weight_stats, a->weight_stats64,
                               a->ws_reduce, a->ws_reduce_bytes, stream);
    if (rc != MI3_OK) return rc;
    k_newton_report<<<1, 1, 0, as_stream(stream)>>>(a->weight_stats64, a->minout, a->status, a->host_out);
    if (cudaEventRecord(reinterpret_cast<cudaEvent_t>(a->event), as_stream(stream)) != cudaSuccess)
        return check_launch("mi3_newton_step: event");
    rc = mi3_weighted_marg(a->weights, a->seqmem, a->buflen, a->nseq, a->bi, a->L, a->q, nullptr, a->ws_wmarg,
                           a->ws_wmarg_bytes, stream);
    if (rc == MI3_OK) rc = mi3_renormalize_bimarg(a->bi, a->L, a->q, stream);
    return rc;
}
