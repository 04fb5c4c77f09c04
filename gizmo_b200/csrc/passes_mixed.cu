// gizmo_b200/csrc/passes_mixed.cu -- mixed form: FP32 force pair arithmetic,
// FP64 positions / membership / density and gradient sums / accumulation (see
// passes.cuh). Built with the approximate FP32 division and square root; the
// pairs whose FP32 branch decisions are too close to call are evaluated again
// by force_refine in passes_fp64.cu.
#include "passes.cuh"

namespace gz {

void force_mixed(const PassParams &p, const Particles &ps, const int *targets, int n_targets, Csr rows,
                 DevStatus *st, void *rec, void *flux, bool all, const RefineQueue &q, const RefineQueue &dq,
                 double *sums, const EventPair *ev, cudaStream_t s)
{
    launch_force<float>(p, ps, targets, n_targets, rows, st, rec, flux, all, q, dq, sums, ev, s);
}

}  // namespace gz
