// adjoint.cuh -- discrete adjoint of the nonlinear term and of an RK4CN step.
//
// State x: the Hermitian half spectrum.  Inner product
//   <a, b>_W = sum_j c_j Re(conj(a_j) b_j),  c_j = 1 on ky = 0 and ky = N/2, 2 else,
// under which the unnormalised c2r (C) and r2c (R) are exact transposes.  With
// multipliers m_u = i ky/k^2, m_v = -i kx/k^2, m_x = i kx, m_y = i ky, dealias
// factor D and s = 1/(Nx Ny), the forward RHS is
//   F(X) = s^2 D R( C(m_u X) C(m_x X) + C(m_v X) C(m_y X) )
// and its adjoint at X applied to kappa is
//   F'(X)^T kappa = conj(m_u) R(wx mu) + conj(m_v) R(wy mu) + conj(m_x) R(u mu) + conj(m_y) R(v mu),
//   mu = C(s^2 D kappa),
// with u, v, wx, wy = C(m_u X), C(m_v X), C(m_x X), C(m_y X) the real fields of
// the forward stage, captured while the forward step is recomputed.
//
// Passes per adjoint stage (mirroring the forward step):
//   adj row pass  (y): mu = c2r(mu_x); products wx mu, wy mu, u mu, v mu, packed as
//                      Q = (wx + i wy) mu and R = (u + i v) mu; two forward y-FFTs;
//                      Q(ky) and conj Q(-ky) at ky >= 0 are P0 +- i P1 of the real
//                      products' half spectra (R: P2 +- i P3) and go out as they are.
//   adj col pass  (x): four forward x-FFTs of those, L = sum conj(m) P (the
//                      adjoint of this stage's input); lambda_x += L; the
//                      previous stage's kappa = b B lambda' + a dt L; then
//                      s^2 D kappa -> inverse x-FFT -> mu_x for the next row pass
//                      (columns that D empties are neither formed nor read).
#pragma once
#include "kernels.cuh"

namespace ns2d {

enum AdjMode : int { ADJ_START = 0, ADJ_MID = 1, ADJ_END = 2 };

template <typename Real>
struct AdjColArgs {
    using C = typename Cx<Real>::T;
    const C* P0;          // x-space spectra of the row pass (MID, END): Q(ky), conj Q(-ky),
    const C* P1;          // R(ky), conj R(-ky)
    const C* P2;
    const C* P3;
    C* lam_x;             // adjoint of the step input (accumulated), [kx][ldc]
    const C* lam_p;       // adjoint of the step output lambda'
    const double2* cn;    // ((2-D)/(2+D), 2dt/(2+D)) per mode
    C* mu;                // x-space mu_x for the next row pass (START, MID)
    const C* tw;
    int ldc, nyf;
    Real norm2;
    int kmax_sqr, dealias, houli_int, kolm;
    int kc;               // columns ky >= kc are emptied by D
    double b_next;        // weight of lambda' in the next kappa: b_{s-1} (MID) or b_4 (START)
    double adt;           // a_{s-1} dt (MID)
};

// Dealias factor of the forward RHS at (kx, ky) (solver.c:1039-1099).
template <typename Real>
__device__ __forceinline__ Real dealias_factor(int kx, int ky, int N, int kmax_sqr, int dealias, int houli_int,
                                               int kolm) {
    if (kx == 0 && ky == 0) return (Real)0;
    if (dealias == 0) {
        const double k2 = (double)kx * kx + (double)ky * ky;
        return (k2 >= (double)kmax_sqr || (kolm && kx == 0)) ? (Real)0 : (Real)1;
    }
    return houli_filter<Real>(kx, ky, N, N, houli_int);
}

// Exchange buffer of one group's transforms, synchronised with the group's own
// named barrier.
template <int N, int TC, typename C>
struct IlvGroupPolicy {
    C* sm;
    int c, bar;
    static constexpr int STRIDE = SmemLayout<N, TC>::ELEMS;
    __device__ __forceinline__ C& at(int b, int e) const { return sm[b * STRIDE + SmemLayout<N, TC>::slot(e, c)]; }
    __device__ __forceinline__ void sync() const {
        asm volatile("bar.sync %0, %1;\n" ::"r"(bar), "n"(Plan<N>::T * TC) : "memory");
    }
};

// Thread groups of the adjoint column pass: two, each transforming one of the two
// pairs of spectra, where a thread holds few enough elements for it (at 512^2
// FP64 17 us with one group); one group takes the pairs in turn otherwise.
template <int N>
constexpr int adj_groups() { return N / Plan<N>::T <= 8 ? 2 : 1; }

template <typename Real, int N, int TC>
struct AdjColSmem {
    using C = typename Cx<Real>::T;
    static constexpr int G = adj_groups<N>();
    static constexpr int FFT = SmemLayout<N, TC>::ELEMS;
    static constexpr size_t bytes() { return sizeof(C) * (size_t)(2 * G * FFT + G * N * TC); }
};

template <typename Real, int N, int TC, int MODE>
__global__ void __launch_bounds__(Plan<N>::T * TC * adj_groups<N>()) adj_col_kernel(AdjColArgs<Real> a) {
    using C = typename Cx<Real>::T;
    using P = Plan<N>;
    using SM = AdjColSmem<Real, N, TC>;
    constexpr int T = P::T;
    constexpr int E = N / T;
    constexpr int G = SM::G;
    constexpr int EG = E / G;  // elements of the epilogue per thread
    extern __shared__ __align__(16) unsigned char smraw[];
    C* sm = reinterpret_cast<C*>(smraw);
    C* Lbuf = sm + 2 * G * SM::FFT;  // [G][N][TC]: the groups' parts of L, then s^2 D kappa in the first
    const int g = threadIdx.x / (T * TC);
    const int c = threadIdx.x % TC;
    const int t = (threadIdx.x % (T * TC)) / TC;
    const int ky = blockIdx.x * TC + c;
    const bool valid = ky < a.nyf;
    const int kyc = valid ? ky : 0;
    const int ldc = a.ldc;
    const auto seed = twiddle_seeds<N>(a.tw, t);
    const IlvGroupPolicy<N, TC, C> pol{sm + 2 * g * SM::FFT, c, 1 + g};
    const Real tr = (Real)t, kyr = (Real)ky;

    // Operands of the epilogue: on their way under the transforms where a thread
    // holds few elements; with sixteen (1024 and 2048) they would spill there, 600
    // bytes a thread in FP64, and are read after (a reverse step at 1024^2 FP64 414 us
    // against 440, at 2048^2 1,782 against 1,930).
    constexpr bool AHEAD = EG <= 8;
    C lx[EG], lp[MODE == ADJ_END ? 1 : EG];
    double2 f[MODE == ADJ_END ? 1 : EG];
    const auto operands = [&] {
#pragma unroll
        for (int m = 0; m < EG; ++m) {
            const size_t q = (size_t)(t + T * (m + g * EG)) * ldc + kyc;
            if constexpr (MODE != ADJ_START) lx[m] = a.lam_x[q];
            if constexpr (MODE != ADJ_END) {
                lp[m] = a.lam_p[q];
                f[m] = a.cn[q];
            }
        }
    };
    if constexpr (AHEAD) operands();
    if constexpr (MODE != ADJ_START) {
        const C* const Ps[4] = {a.P0, a.P1, a.P2, a.P3};
#pragma unroll 1
        for (int pair = g; pair < 2; pair += G) {
            C v[2][E];
#pragma unroll
            for (int m = 0; m < E; ++m) {
                const size_t q = (size_t)(t + T * m) * ldc + kyc;
                v[0][m] = Ps[2 * pair][q];
                v[1][m] = Ps[2 * pair + 1][q];
            }
            fft_batched<N, -1, 2>(v, pol, seed, t);
            // The four terms conj(m) P, of Q+- = P0 +- i P1 and R+- = P2 +- i P3:
            //   pair 0: (kx (Q+ - Q-) - i ky (Q+ + Q-)) / (2 k^2)
            //   pair 1: (-i kx (R+ + R-) - ky (R+ - R-)) / 2
            // The factors with 1/k^2 are formed in FP64 and rounded once.
#pragma unroll
            for (int m = 0; m < E; ++m) {
                const Real kx = kx_of<Real, N, T>(m, t, tr);
                const C d = csub(v[0][m], v[1][m]), e = cadd(v[0][m], v[1][m]);
                C L;
                if (m == 0 && t == 0 && ky == 0) {
                    L = cmake<C>(0, 0);
                } else if (pair == 0) {
                    const double kd = (double)kx, h = 0.5 * inv_k2<double>(kd * kd + (double)ky * (double)ky);
                    const Real sx = (Real)(kd * h), sy = (Real)((double)ky * h);
                    L = cmake<C>(sx * d.x + sy * e.y, sx * d.y - sy * e.x);
                } else {
                    const Real sx = (Real)0.5 * kx, sy = (Real)0.5 * kyr;
                    L = cmake<C>(sx * e.y - sy * d.x, -(sx * e.x) - sy * d.y);
                }
                C* const to = Lbuf + (G > 1 ? g * N * TC : 0) + (t + T * m) * TC + c;
                if (G == 1 && pair > 0) L = cadd(*to, L);
                *to = L;
            }
        }
        if constexpr (G > 1) __syncthreads();
    }
    if constexpr (!AHEAD) operands();
#pragma unroll
    for (int m = 0; m < EG; ++m) {
        const int i = t + T * (m + g * EG);
        const size_t q = (size_t)i * ldc + ky;
        C L = cmake<C>(0, 0);
        if constexpr (MODE != ADJ_START) {
            L = Lbuf[i * TC + c];
            if constexpr (G > 1) L = cadd(L, Lbuf[N * TC + i * TC + c]);
        }
        if constexpr (MODE == ADJ_END) {
            if (valid) a.lam_x[q] = cadd(lx[m], L);
        } else {
            // lambda_x, then kappa of the next (earlier) stage and the source of mu
            C kappa = cscale(lp[m], (Real)(a.b_next * f[m].y));
            if constexpr (MODE == ADJ_MID) {
                if (valid) a.lam_x[q] = cadd(lx[m], L);
                kappa = cadd(kappa, cscale(L, (Real)a.adt));
            } else {
                if (valid) a.lam_x[q] = cscale(lp[m], (Real)f[m].x);  // lambda_x = A lambda'
            }
            const int kx = (i <= N / 2) ? i : i - N;
            const Real d = dealias_factor<Real>(kx, ky, N, a.kmax_sqr, a.dealias, a.houli_int, a.kolm);
            Lbuf[i * TC + c] = cscale(kappa, a.norm2 * d);
        }
    }
    if constexpr (MODE != ADJ_END) {
        if (blockIdx.x * TC >= a.kc) return;  // mu is zero here, and not read
        __syncthreads();
        if (g > 0) return;
        C v[1][E];
#pragma unroll
        for (int m = 0; m < E; ++m) v[0][m] = Lbuf[(t + T * m) * TC + c];
        fft_batched<N, +1, 1>(v, pol, seed, t);
        if (valid) {
#pragma unroll
            for (int m = 0; m < E; ++m) a.mu[(size_t)(t + T * m) * ldc + ky] = v[0][m];
        }
    }
}

template <typename Real>
struct AdjRowArgs {
    using C = typename Cx<Real>::T;
    const C* mu;          // x-space mu_x [x][ldc]
    const C* cap_uv;      // captured real fields of the forward stage: (u, v) and
    const C* cap_w;       // (w_x, w_y) as complex pairs, [x][y]
    C* P0;                // outputs at ky >= 0: Q(ky), conj Q(-ky), R(ky), conj R(-ky)
    C* P1;
    C* P2;
    C* P3;
    const C* tw;
    int ldc;
    int kc;               // mu_x is zero (and not stored) from ky = kc on
};

// Adjoint row pass: one team of T threads per row x, TC = 2 PAIRS rows per block.
template <typename Real, int N, int PAIRS>
__global__ void __launch_bounds__(Plan<N>::T * 2 * PAIRS) adj_row_kernel(AdjRowArgs<Real> a) {
    using C = typename Cx<Real>::T;
    using P = Plan<N>;
    constexpr int T = P::T;
    constexpr int E = N / T;
    constexpr int TC = 2 * PAIRS;
    using RS = RowSmem<Real, N, TC>;
    extern __shared__ __align__(16) unsigned char smraw[];
    const int g = threadIdx.x / T;
    const int t = threadIdx.x % T;
    const int x = blockIdx.x * TC + g;
    C* region = reinterpret_cast<C*>(smraw) + (size_t)g * RS::TEAM;
    const auto seed = twiddle_seeds<N, row_extra(N)>(a.tw, t);
    const TeamPolicy<N, C> pol{region, 1 + g};
    // mu = c2r(mu_x) along y: Hermitian extension, real parts at ky = 0 and N/2
    C z[1][E];
    {
        const C* __restrict__ M = a.mu + (size_t)x * a.ldc;
#pragma unroll
        for (int m = 0; m < E; ++m) {
            const int y = t + T * m;
            const int yy = (y <= N / 2) ? y : N - y;
            const C p = yy < a.kc ? M[yy] : cmake<C>(0, 0);
            if (y == 0 || y == N / 2) z[0][m] = cmake<C>(p.x, 0);
            else if (y < N / 2) z[0][m] = p;
            else z[0][m] = cconj(p);
        }
    }
    fft_batched<N, +1, 1>(z, pol, seed, t);
    // products with the captured fields, packed two per complex transform
    C q[2][E];
    {
        const C* __restrict__ cu = a.cap_uv + (size_t)x * N;
        const C* __restrict__ cw = a.cap_w + (size_t)x * N;
#pragma unroll
        for (int m = 0; m < E; ++m) {
            const int y = t + T * m;
            const Real mu = z[0][m].x;
            const C uv = cu[y], wxy = cw[y];
            q[0][m] = cmake<C>(wxy.x * mu, wxy.y * mu);
            q[1][m] = cmake<C>(uv.x * mu, uv.y * mu);
        }
    }
    fft_batched<N, -1, 2>(q, pol, seed, t);
    C* outs[4] = {a.P0, a.P1, a.P2, a.P3};
#pragma unroll
    for (int b = 0; b < 2; ++b) {
        C* __restrict__ op = outs[2 * b] + (size_t)x * a.ldc;
        C* __restrict__ on = outs[2 * b + 1] + (size_t)x * a.ldc;
#pragma unroll
        for (int m = 0; m < E; ++m) {
            const int k = t + T * m;
            if (k <= N / 2) op[k] = q[b][m];
            if (k == 0 || k >= N / 2) on[k == 0 ? 0 : N - k] = cconj(q[b][m]);
        }
    }
}

// Objective and its W-gradient at the final state: enstrophy
// Z = cZ sum_j c_j |w_j|^2 -> 2 cZ w; palinstrophy P = cZ sum_j c_j k^2 |w_j|^2
// -> 2 cZ k^2 w (cZ = 4 pi^2 0.5/(Nx Ny)^2, mean mode excluded;
// sys_msr.c:190-227, 356-363).  One FP64 partial sum per block (fixed grid, so
// the host's ordered sum of the partials is deterministic).
template <typename Real>
__global__ void __launch_bounds__(256) adj_objective_kernel(const typename Cx<Real>::T* state,
                                                            typename Cx<Real>::T* lam, int nx, int nyf, int ldc,
                                                            double cz, int palin, double* partials) {
    const long long n = (long long)nx * nyf;
    double acc = 0.0;
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x) {
        const int i = (int)(q / nyf), ky = (int)(q % nyf);
        const int kx = (i <= nx / 2) ? i : i - nx;
        const size_t o = (size_t)i * ldc + ky;
        double f = palin ? (double)(kx * kx + ky * ky) : 1.0;
        if (kx == 0 && ky == 0) f = 0.0;
        const auto w = state[o];
        const double w2 = (double)w.x * (double)w.x + (double)w.y * (double)w.y;
        acc += ((ky == 0 || ky == nyf - 1) ? 1.0 : 2.0) * f * w2;
        if (lam) lam[o] = cscale(w, (Real)(2.0 * cz * f));
    }
    __shared__ double red[8];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double tot = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) tot += red[w];
        partials[blockIdx.x] = cz * tot;
    }
}

// <a, b>_W = sum_j c_j Re(conj(a_j) b_j) over the half spectrum, FP64 partials per block.
template <typename Real>
__global__ void __launch_bounds__(256) adj_wdot_kernel(const typename Cx<Real>::T* a, const typename Cx<Real>::T* b,
                                                       int nx, int nyf, int ldc, double* partials) {
    const long long n = (long long)nx * nyf;
    double acc = 0.0;
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x) {
        const int i = (int)(q / nyf), ky = (int)(q % nyf);
        const size_t o = (size_t)i * ldc + ky;
        const auto x = a[o], y = b[o];
        acc += ((ky == 0 || ky == nyf - 1) ? 1.0 : 2.0) * ((double)x.x * (double)y.x + (double)x.y * (double)y.y);
    }
    __shared__ double red[8];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double tot = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) tot += red[w];
        partials[blockIdx.x] = tot;
    }
}

}  // namespace ns2d
