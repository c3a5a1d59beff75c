// engine_f32.cu -- the step kernels of every grid size in single precision.
#include "engine.cuh"

namespace ns2d {

template <>
const EngineOps<float>* engine_ops<float>(int n) {
    const EngineOps<float>* ops = nullptr;
    with_size<float>(n, [&](auto L) {
        using E = decltype(L);
        static const EngineOps<float> o{E::S::TC, E::S::TC_STAGE, E::setup, E::col, E::row, E::col_inv, E::fwd, E::row_c2r};
        ops = &o;
    });
    return ops;
}

}  // namespace ns2d
