// euler_mixed.cu -- the mixed form's kernels of the Eulerian grid hydrocode:
// primitives, face fluxes, right-hand-side sources, the yield surface, damage
// growth and the CFL speed in FP32 (the arithmetic of the reference's own GPU
// solver), compiled with fused multiply-adds; the FP64 state updates and the
// step control are shared with the FP64 form (euler.cu).
#include "euler_kernels.cuh"

namespace deu {

int enqueue_lop_f32(const P& p, const Fields& s, PrimT<float> W, const double* af, FacesT<float> F, RhsT<float> d,
                    const Ctl* ctl, cudaStream_t st) {
    return enqueue_lop_t<float>(p, s, W, af, F, d, ctl, st);
}

void enqueue_prim_f32(const P& p, const Fields& s, PrimT<float> W, const Ctl* ctl, cudaStream_t st, int af) {
    enqueue_prim_t<float>(p, s, W, ctl, st, af);
}

void enqueue_maxspeed_f32(const P& p, const Fields& g, Ctl* ctl, cudaStream_t st, int with_dt) {
    enqueue_maxspeed_t<float>(p, g, ctl, st, with_dt);
}

void enqueue_predict_f32(const P& p, const Fields& g, const Fields& g1, PrimT<float> W, RhsT<float> d, const Ctl* ctl,
                         cudaStream_t st) {
    enqueue_predict_t<float>(p, g, g1, W, d, ctl, st);
}

void enqueue_correct_f32(const P& p, const Fields& g, const Fields& g1, RhsT<float> d, const Ctl* ctl,
                         cudaStream_t st, int stage) {
    enqueue_correct_t<float>(p, g, g1, d, ctl, st, stage);
}

}  // namespace deu
