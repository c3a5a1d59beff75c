// engine_f64.cu -- the step kernels of every grid size in double precision.
#include "engine.cuh"

namespace ns2d {

template <>
const EngineOps<double>* engine_ops<double>(int n) {
    const EngineOps<double>* ops = nullptr;
    with_size<double>(n, [&](auto L) {
        using E = decltype(L);
        static const EngineOps<double> o{E::S::TC, E::S::TC_STAGE, E::setup, E::col, E::row, E::col_inv, E::fwd, E::row_c2r};
        ops = &o;
    });
    return ops;
}

}  // namespace ns2d
