// engine_size.cu -- the step kernels of one grid size in one precision: compiled for
// each with NS2D_ENGINE_N and NS2D_ENGINE_REAL (Makefile).
#include "engine.cuh"

namespace ns2d {

template <typename Real, int N>
const EngineOps<Real>* engine_ops_of() {
    using E = Launch<Real, N>;
    static const EngineOps<Real> o{E::S::TC, E::S::TC_STAGE, E::setup, E::col, E::row, E::col_inv, E::fwd, E::row_c2r};
    return &o;
}
template const EngineOps<NS2D_ENGINE_REAL>* engine_ops_of<NS2D_ENGINE_REAL, NS2D_ENGINE_N>();

}  // namespace ns2d
