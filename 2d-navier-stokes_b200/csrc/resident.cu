// resident.cu -- instantiations of the resident small-grid kernel.
#include "resident.h"

namespace ns2d {
namespace {

template <typename Real, typename F>
bool with_resident_size(int n, F&& f) {
    switch (n) {
        case 16: f(ResLaunch<Real, 16>{}); return true;
        case 32: f(ResLaunch<Real, 32>{}); return true;
        case 64: f(ResLaunch<Real, 64>{}); return true;
        case 128: f(ResLaunch<Real, 128>{}); return true;
        default: return false;
    }
}

}  // namespace

bool resident_setup(int n, bool fp32) {
    bool ok = false;
    if (fp32) with_resident_size<float>(n, [&](auto L) { ok = decltype(L)::setup(); });
    else with_resident_size<double>(n, [&](auto L) { ok = decltype(L)::setup(); });
    return ok;
}

template <typename Real>
cudaError_t resident_launch(int n, int scheme, const ResArgs<Real>& a, cudaStream_t s) {
    cudaError_t e = cudaErrorInvalidValue;
    with_resident_size<Real>(n, [&](auto L) { e = decltype(L)::launch(scheme, a, s); });
    return e;
}
template cudaError_t resident_launch<float>(int, int, const ResArgs<float>&, cudaStream_t);
template cudaError_t resident_launch<double>(int, int, const ResArgs<double>&, cudaStream_t);

}  // namespace ns2d
