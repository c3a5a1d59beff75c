// diag.cuh -- ComputeSystemMeasurables (Solver/src/sys_msr.c:32-373) as one
// pass over the half spectrum: 13 totals reduced in FP64 (per-thread sums,
// warp and block trees, one atomic per block and total) and 8 spectra binned
// by round(|k|) in shared memory.  Raw sums are scaled on the host by the
// reference's constants (4 pi^2 and 0.5/(Nx Ny)^2).  Bound by FP64 arithmetic and
// the shared-memory atomics of the spectra (eight sums per mode): see the loop.
#pragma once
#include "kernels.cuh"

namespace ns2d {

enum { DG_E = 0, DG_Z, DG_P, DG_FORC, DG_DIV, DG_EDISS, DG_ZDISS, DG_DE, DG_EFLUX, DG_EDSB, DG_DZ, DG_ZFLUX, DG_ZDSB, DG_N };

template <typename Real>
struct DiagArgs {
    using C = typename Cx<Real>::T;
    const C* state;
    const C* rhs;    // RHS of the state minus forcing (flux terms), may be null
    int ldc, nx, ny, nyf;
    LinOp lin;       // pre_fac branch (sys_msr.c:166-181)
    int enst_quirk;  // weight-2 enstrophy dissipation without pre_fac (sys_msr.c:225)
    int force_i, force_j;
    double fre, fim;
    int has_force;
    const C* ffield;  // forcing of listed modes ([nx][ldc]), may be null
    int n_spect;
    double* out;     // [DG_N] raw totals, then 8 * n_spect raw spectra (zeroed by the host)
};

constexpr int kDiagThreads = 512;
inline size_t diag_smem(int n_spect) { return sizeof(double) * (8 * (size_t)n_spect + DG_N * (kDiagThreads / 32)); }

template <typename Real>
__global__ void __launch_bounds__(kDiagThreads) diag_kernel(DiagArgs<Real> a) {
    using C = typename Cx<Real>::T;
    extern __shared__ double dsm[];  // diag_smem(n_spect): 8 * n_spect spectra, then the warps' totals
    const int ns = a.n_spect;
    double* hist = dsm;
    double* wpart = dsm + 8 * ns;
    for (int q = threadIdx.x; q < 8 * ns; q += blockDim.x) hist[q] = 0.0;
    __syncthreads();
    double acc[DG_N];
#pragma unroll
    for (int k = 0; k < DG_N; ++k) acc[k] = 0.0;
    const long long n = (long long)a.nx * a.nyf;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (long long q0 = blockIdx.x * (long long)blockDim.x; q0 < n; q0 += (long long)gridDim.x * blockDim.x) {
        const long long q = q0 + threadIdx.x;
        const bool in = q < n;
        const int i = in ? (int)(q / a.nyf) : 0, j = in ? (int)(q % a.nyf) : 0;
        const int kx = (i <= a.nx / 2) ? i : i - a.nx;
        const int ky = j;
        C wc = cmake<C>(0, 0), r = wc;
        if (in) {
            wc = a.state[(size_t)i * a.ldc + j];
            if (a.rhs) r = a.rhs[(size_t)i * a.ldc + j];
        }
        const double wr = (double)wc.x, wi = (double)wc.y;
        const double k_sqr = (double)(kx * kx + ky * ky);
        const double pre_fac = lin_bracket(a.lin, k_sqr);
        // A mode that is exactly zero (the 2/3 rule leaves most of them so) adds
        // zeros everywhere; not one whose factors are not finite.
        const bool on = in && !(kx == 0 && ky == 0) &&
                        !(wr == 0.0 && wi == 0.0 && isfinite(pre_fac) && isfinite((double)r.x) && isfinite((double)r.y));
        if (!__any_sync(0xffffffffu, on)) continue;
        double s[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) s[k] = 0.0;
        int bin = -1;
        if (on) {
            const double inv = 1.0 / k_sqr;
            const double w2 = wr * wr + wi * wi;
            // u_z = i ky w / k^2, v_z = -i kx w / k^2, div = i (kx u_z + ky v_z)
            const double ur = -((double)ky * wi) * inv, ui = ((double)ky * wr) * inv;
            const double vr = ((double)kx * wi) * inv, vi = -((double)kx * wr) * inv;
            const double dre = (double)kx * ur + (double)ky * vr, dim = (double)kx * ui + (double)ky * vi;
            const double div2 = dre * dre + dim * dim;
            const double uv2 = ur * ur + ui * ui + vr * vr + vi * vi;
            double deriv = 0.0;
            if (a.rhs) {
                // the flux terms ignore forcing (sys_msr.c:127-132)
                if (a.has_force && i == a.force_i && j == a.force_j) {
                    r.x = (Real)((double)r.x - a.fre);
                    r.y = (Real)((double)r.y - a.fim);
                }
                if (a.ffield) {
                    const C f = a.ffield[(size_t)i * a.ldc + j];
                    r.x = (Real)((double)r.x - (double)f.x);
                    r.y = (Real)((double)r.y - (double)f.y);
                }
                // creal(w conj(r) + conj(w) r) = 2 Re(w conj r)
                deriv = (wr * (double)r.x + wi * (double)r.y) + ((double)r.x * wr + (double)r.y * wi);
            }
            const double diss = pre_fac * w2;
            const double wgt = (j == 0 || j == a.nyf - 1) ? 1.0 : 2.0;
            s[0] = wgt * w2 * inv;                // enrg
            s[1] = wgt * w2;                      // enst
            s[2] = wgt * (deriv + diss);          // d_enst_dt
            s[3] = wgt * deriv;                   // enst_flux
            s[4] = wgt * diss;                    // enst_diss
            s[5] = s[2] * inv;                    // d_enrg_dt
            s[6] = s[3] * inv;                    // enrg_flux
            s[7] = s[4] * inv;                    // enrg_diss
            acc[DG_E] += s[0];
            acc[DG_Z] += s[1];
            acc[DG_DIV] += wgt * div2;
            acc[DG_P] += wgt * k_sqr * w2;
            acc[DG_EDISS] += wgt * pre_fac * uv2;
            acc[DG_ZDISS] += (wgt == 2.0 && a.enst_quirk) ? 2.0 * w2 : s[4];
            if (k_sqr >= 0.0 && k_sqr < 4096.0) {
                acc[DG_DE] += s[5];
                acc[DG_EDSB] += s[7];
                acc[DG_EFLUX] += s[6];
                acc[DG_DZ] += s[2];
                acc[DG_ZDSB] += s[4];
                acc[DG_ZFLUX] += s[3];
            }
            if (a.has_force && i == a.force_i && j == a.force_j) {
                // cabs(forcing * w_hat[forced])  (sys_msr.c:135-139)
                const double pr = a.fre * wr - a.fim * wi, pi = a.fre * wi + a.fim * wr;
                acc[DG_FORC] += sqrt(pr * pr + pi * pi);
            }
            if (a.ffield) {
                const C f = a.ffield[(size_t)i * a.ldc + j];
                const double fr = (double)f.x, fi = (double)f.y;
                const double pr = fr * wr - fi * wi, pi = fr * wi + fi * wr;
                acc[DG_FORC] += sqrt(pr * pr + pi * pi);
            }
            const int b = (int)round(sqrt(k_sqr));
            if (b < ns) bin = b;
        }
        // Neighbouring lanes (consecutive ky of a row) mostly share a bin: each run
        // of equal bins is summed by shuffles first and added to shared memory once,
        // where 32 lanes on a few addresses would take turns.
        const int prev = __shfl_up_sync(0xffffffffu, bin, 1);
        const unsigned heads = __ballot_sync(0xffffffffu, lane == 0 || bin != prev);
        const int run = __popc(heads & (0xffffffffu >> (31 - lane)));
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const bool same = __shfl_down_sync(0xffffffffu, run, o) == run && lane + o < 32;
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const double v = __shfl_down_sync(0xffffffffu, s[k], o);
                if (same) s[k] += v;
            }
        }
        if (((heads >> lane) & 1u) && bin >= 0) {
#pragma unroll
            for (int k = 0; k < 8; ++k) atomicAdd(&hist[k * ns + bin], s[k]);
        }
    }
#pragma unroll
    for (int k = 0; k < DG_N; ++k) {
        double v = acc[k];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0) wpart[k * (kDiagThreads / 32) + warp] = v;
    }
    __syncthreads();
    if (threadIdx.x < DG_N) {
        double v = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) v += wpart[threadIdx.x * (kDiagThreads / 32) + w];
        atomicAdd(&a.out[threadIdx.x], v);
    }
    for (int q = threadIdx.x; q < 8 * ns; q += blockDim.x)
        if (hist[q] != 0.0) atomicAdd(&a.out[DG_N + q], hist[q]);
}

}  // namespace ns2d
