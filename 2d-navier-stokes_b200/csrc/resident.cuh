// resident.cuh -- whole time steps of a small grid (N <= 128) in one launch.
//
// At these sizes a step of the nine pass launches is bound by latency: each
// launch runs on a handful of SMs and costs a kernel boundary, several dependent
// L2 round trips and a few hundred cycles of transform (45 us a step at 64^2
// FP64, of which the arithmetic is under 1 us of the chip).  Here one
// thread-block cluster holds the whole field in the shared memory of its blocks
// for any number of steps: block r owns the ky columns r, r + CL, ... of the
// spectral arrays (state, accumulator, stage input, update factors) and the x
// rows [r N/CL, (r+1) N/CL).  The two transposes of an evaluation are stores to
// the other blocks' shared memory (distributed shared memory), and the only
// synchronisation between blocks is the cluster's hardware barrier, twice per
// evaluation:
//
//   columns: four derived spectra of the stage input per column, one inverse
//            x-FFT per (column, field) unit; results to the row owners
//   -- cluster barrier --
//   rows:    one inverse y-FFT per (row, Z1 or Z2) unit, the product of a row
//            formed by the two teams of its units through warp shuffles, one
//            packed forward y-FFT per row pair; results to the column owners
//   -- cluster barrier --
//   columns: forward x-FFT, dealiasing, forcing, conjugacy, stage combine or
//            update, all on the block's own columns
//
// What bounds it is the chain of latencies: at 64^2 FP64 an evaluation takes 7,000 to
// 8,000 cycles, of which the two cluster barriers 1,300-2,200 (a barrier of up to
// 8 blocks costs 500-860 cycles, of 16 about 900), the four transforms on the
// path about 800 each, and the rest loads, twiddles and the remote stores; at
// 128^2 FP64 arithmetic and remote-store issue add to it.  Measured per step
// (RK4CN, 2/3, FP64 / FP32, us): 16^2 28.8 / 28.8 -> 6.5 / 5.3, 32^2 39.0 / 34.9 ->
// 9.9 / 8.0, 64^2 45.3 / 41.1 -> 13.8 / 10.2, 128^2 53.4 / 44.6 -> 20.6 / 17.2 against
// the pass launches replayed from a graph; explicit RK4 at 64^2 154 -> 13.6 (its
// passes never settled on a graph).
//
// Columns that the 2/3 rule empties (ky >= kc, k2 >= kmax_sqr for every kx) hold
// zeros in every evaluation, and in the state too unless the caller put
// something there, so they are left out of the transforms when the state holds
// nothing in them (checked when it is loaded) and no forced mode lies there.
#pragma once
#include "kernels.cuh"

namespace ns2d {

// One kernel per scheme: the code of a step streams through the instruction
// caches with few warps to hide a miss, so each holds only what it runs.
enum ResScheme : int { RES_CN = 0, RES_EXPLICIT = 1, RES_AB4 = 2, RES_RHS = 3 };

template <typename Real>
struct ResArgs {
    using C = typename Cx<Real>::T;
    const C* src;          // RES_RHS: the evaluation's input
    const double2* src64;  // where the input or state comes from instead, in the caller's layout [N][nyf] ...
    double2* out64;        // ... and where the RHS or the new state also goes; both or neither for steps
    C* state;              // w_hat
    C* rhs;                // RES_RHS: the RHS; RES_CN: stage 1's RHS of every step (AB4 start-up), may be null
    C* h[4];               // AB4: RHS of steps n-3, n-2, n-1, and the one to be written
    const C* tw;
    const C* force_field;  // forcing added to every mode, may be null
    const double2* cn;     // Crank-Nicolson factors (RES_CN, RES_AB4 of the Navier-Stokes system)
    int ldc, nyf;
    int kmax_sqr, kc;      // 2/3 rule: kept modes k2 < kmax_sqr, all in columns ky < kc
    int dealias, houli_int, kolm;
    int has_force, force_i, force_j;
    C force_val;
    int wide;              // transform every column whatever the state holds
    int conj_quirk;        // RES_RHS: whether the state's column 0 is rewritten
    int lin_stage;         // as ColArgs
    int phase_only;
    int euler;             // RES_AB4: explicit update
    int nsteps;
    Real norm2;
    double dt, inv_nxny;
    LinOp lin;
    int* status;           // as ColArgs; a set word ends the launch before its first step.  RES_RHS: null
};

// Cluster and block shapes.  CL blocks of NT threads; a unit is one transform by
// a team of Plan<N>::T threads.  Measured per FP64 step (us): 16^2 1 x 128 7.8,
// 2 x 64 8.7, 4 x 32 7.9; 32^2 8 x 64 10.2, 4 x 128 10.9, 2 x 256 13.1, 1 x 512 16.5;
// 64^2 8 x 128 14.6, 8 x 256 15.6, 4 x 256 18.1 (16 x 64: 13.5, but 11.0 against
// 10.8 in FP32 and twice the SMs); 128^2 16 x 256 21.6, 16 x 128 22.4, 16 x 512 24.4
// (8 blocks do not hold an FP64 field).
template <int N>
struct ResShape;
template <> struct ResShape<16>  { static constexpr int CL = 1,  NT = 128; };
template <> struct ResShape<32>  { static constexpr int CL = 8,  NT = 64; };
template <> struct ResShape<64>  { static constexpr int CL = 8,  NT = 128; };
template <> struct ResShape<128> { static constexpr int CL = 16, NT = 256; };

template <typename Real, int N>
struct ResLayout {
    using C = typename Cx<Real>::T;
    using S = ResShape<N>;
    static constexpr int T = Plan<N>::T;
    static constexpr int TEAMS = S::NT / T;
    static constexpr int RPC = N / S::CL;                      // rows per block
    static constexpr int NYF = N / 2 + 1;
    static constexpr int SLOTS = (NYF + S::CL - 1) / S::CL;    // columns per block
    static constexpr int KS = 4 * RPC + 1;                     // x-space elements per ky, odd: no bank conflicts over ky
    static_assert(RPC % 2 == 0 && T <= 16 && S::NT % 32 == 0, "row pairs and paired teams in a warp");
    // element offsets
    static constexpr int F = 0;                                // [NYF][KS]: [field][local row]
    static constexpr int NL = F + NYF * KS;                    // [SLOTS][N] product spectrum n(x, ky)
    static constexpr int W = NL + SLOTS * N;                   // [SLOTS][N] state
    static constexpr int ACC = W + SLOTS * N;
    static constexpr int X = ACC + SLOTS * N;                  // stage input
    static constexpr int REG = X + SLOTS * N;                  // team exchange regions
    static constexpr int END = (REG + TEAMS * TeamLayout<N>::ROWS + 1) & ~1;  // 16-byte boundary
    // then [SLOTS][N] double2 update factors, [SLOTS][N] reals of dealiasing
    // factors and of 1/k^2, and [RPC][N] reals of the rows' products
    static constexpr size_t bytes() {
        return sizeof(C) * (size_t)END + sizeof(double2) * (size_t)SLOTS * N + sizeof(Real) * (size_t)(2 * SLOTS + RPC) * N;
    }
};

__device__ __forceinline__ unsigned cluster_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(r));
    return r;
}
template <int CL>
__device__ __forceinline__ void cluster_sync() {
    if constexpr (CL == 1) {
        __syncthreads();
    } else {
        asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
    }
}
// Address of this block's shared-memory location `local` in block `rank`.
__device__ __forceinline__ unsigned cluster_addr(unsigned local, unsigned rank) {
    unsigned a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(a) : "r"(local), "r"(rank));
    return a;
}
__device__ __forceinline__ void cluster_store(unsigned addr, double2 v) {
    asm volatile("st.shared::cluster.v2.f64 [%0], {%1, %2};\n" ::"r"(addr), "d"(v.x), "d"(v.y) : "memory");
}
__device__ __forceinline__ void cluster_store(unsigned addr, float2 v) {
    asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};\n" ::"r"(addr), "f"(v.x), "f"(v.y) : "memory");
}
__device__ __forceinline__ void cluster_store(unsigned addr, int v) {
    asm volatile("st.shared::cluster.s32 [%0], %1;\n" ::"r"(addr), "r"(v) : "memory");
}

// GEN: listed-mode forcing and the phase-only model compiled in.
template <typename Real, int N, int SCHEME, bool GEN>
__global__ void __launch_bounds__(ResShape<N>::NT) resident_kernel(const __grid_constant__ ResArgs<Real> a) {
    using C = typename Cx<Real>::T;
    using L = ResLayout<Real, N>;
    constexpr int CL = ResShape<N>::CL;
    constexpr int NT = ResShape<N>::NT;
    constexpr int T = L::T;
    constexpr int E = N / T;
    constexpr int RPC = L::RPC;
    extern __shared__ __align__(16) unsigned char smraw[];
    C* const sm = reinterpret_cast<C*>(smraw);
    C* const sF = sm + L::F;
    C* const sN = sm + L::NL;
    C* const sW = sm + L::W;
    C* const sA = sm + L::ACC;
    C* const sX = sm + L::X;
    double2* const sCn = reinterpret_cast<double2*>(sm + L::END);
    Real* const sD = reinterpret_cast<Real*>(sCn + L::SLOTS * N);
    Real* const sI = sD + L::SLOTS * N;
    Real* const sP = sI + L::SLOTS * N;
    __shared__ int s_wide[CL], s_stop[CL];
    const int rank = CL == 1 ? 0 : (int)cluster_rank();
    const int t = threadIdx.x % T;
    const int team = threadIdx.x / T;
    const int warp_team = (threadIdx.x & ~31) / T;  // first team of this warp
    const auto seed = twiddle_seeds<N>(a.tw, t);
    const TeamPolicy<N, C> pol{sm + L::REG + team * TeamLayout<N>::ROWS, 0};
    constexpr bool rhs_only = SCHEME == RES_RHS;
    constexpr bool ab4 = SCHEME == RES_AB4;
    constexpr int nstage = ab4 || rhs_only ? 1 : 4;

    // Load the block's columns.  A set status word (an earlier step's failed
    // SystemCheck) ends the launch, as it does every pass launch; it is read
    // before the cluster's first barrier, so every block sees the same value.
    const int status0 = !rhs_only && a.status ? *(volatile const int*)a.status : 0;
    if (threadIdx.x < CL) s_stop[threadIdx.x] = 0;
    bool wide = a.wide != 0;
    for (int q = threadIdx.x; q < L::SLOTS * N; q += NT) {
        const int ky = rank + CL * (q / N), i = q % N;
        C w = cmake<C>(0, 0);
        double2 f = make_double2(0.0, 0.0);
        Real d = 0, inv = 0;
        if (ky < a.nyf) {
            const size_t g = (size_t)i * a.ldc + ky;
            const int kx = (i <= N / 2) ? i : i - N;
            const int k2 = kx * kx + ky * ky;
            if (a.src64) {
                const double2 d64 = a.src64[(size_t)i * a.nyf + ky];
                w = cmake<C>((Real)d64.x, (Real)d64.y);
            } else {
                w = rhs_only ? a.src[g] : a.state[g];
            }
            if (k2 != 0) inv = inv_k2<Real>((Real)k2);
            if constexpr (SCHEME == RES_EXPLICIT) {
                if (a.lin_stage && k2 != 0) {
                    const double br = lin_bracket(a.lin, (double)k2);
                    f.x = a.lin_stage == 1 ? a.dt * br : br;
                }
            } else if constexpr (!rhs_only) {
                if (a.cn) f = a.cn[g];
            }
            if (a.dealias == 0) d = (k2 >= a.kmax_sqr || (a.kolm && kx == 0)) ? (Real)0 : (Real)1;
            else d = houli_filter<Real>(kx, ky, N, N, a.houli_int);
            if (ky >= a.kc) {
                wide |= w.x != (Real)0 || w.y != (Real)0 || !isfinite(f.x) || !isfinite(f.y);
                if constexpr (ab4) {
                    for (int r = 0; r < 3; ++r) wide |= a.h[r][g].x != (Real)0 || a.h[r][g].y != (Real)0;
                }
            }
        }
        sW[q] = w;
        sX[q] = w;
        sA[q] = cmake<C>(0, 0);
        sN[q] = cmake<C>(0, 0);
        sCn[q] = f;
        sD[q] = d;
        sI[q] = inv;
    }
    wide = __syncthreads_or(wide);
    cluster_sync<CL>();  // every block runs and has cleared its flags
    // The state goes back to where the step's result is expected (and over any
    // earlier content of the columns left out below).
    auto put_state = [&](int n) {
        for (int q = threadIdx.x; q < n * N; q += NT) {
            const int ky = rank + CL * (q / N), i = q % N;
            if (ky >= a.nyf) continue;
            const C w = sW[q];
            a.state[(size_t)i * a.ldc + ky] = w;
            if (a.out64) a.out64[(size_t)i * a.nyf + ky] = make_double2((double)w.x, (double)w.y);
        }
    };
    if constexpr (!rhs_only) {
        if (status0) {
            if (a.src64) put_state(L::SLOTS);
            return;
        }
    }
    if (threadIdx.x < CL) cluster_store(cluster_addr(smem_addr(&s_wide[rank]), threadIdx.x), wide ? 1 : 0);
    cluster_sync<CL>();
    wide = false;
#pragma unroll
    for (int r = 0; r < CL; ++r) wide |= s_wide[r] != 0;
    const int kx_cols = wide ? a.nyf : a.kc;                 // columns the transforms cover
    const int nl_cols = a.dealias == 0 ? a.kc : a.nyf;       // columns of the product that survive dealiasing
    const int slots = (kx_cols - rank + CL - 1) / CL;        // this block's columns among them (>= 0)

    // results that every later reader expects in the columns left out
    C* const fill = ab4 ? a.h[3] : a.rhs;
    if (fill) {
        for (int q = slots * N + threadIdx.x; q < L::SLOTS * N; q += NT) {
            const int ky = rank + CL * (q / N), i = q % N;
            if (ky < a.nyf) fill[(size_t)i * a.ldc + ky] = cmake<C>(0, 0);
        }
    }
    if constexpr (rhs_only) {
        for (int q = slots * N + threadIdx.x; a.out64 && q < L::SLOTS * N; q += NT) {
            const int ky = rank + CL * (q / N), i = q % N;
            if (ky < a.nyf) a.out64[(size_t)i * a.nyf + ky] = make_double2(0.0, 0.0);
        }
    }
    const C* h0 = a.h[0];
    const C* h1 = a.h[1];
    const C* h2 = a.h[2];
    C* h3 = a.h[3];
    int done = 0;
    bool stop = false;
    for (int step = 0; step < a.nsteps && !stop; ++step) {
        for (int s = 1; s <= nstage; ++s) {
            // --- columns: derived spectra and inverse x-FFTs
            for (int u0 = 0; u0 + warp_team < 4 * slots; u0 += L::TEAMS) {
                const int u = u0 + team;
                const bool on = u < 4 * slots;
                const int slot = on ? u >> 2 : 0, f = u & 3;
                const int ky = rank + CL * slot;
                // the field's derived spectrum (derived_pair): f & 1 the conj(q) ones,
                // f >= 2 those of X rather than X/k^2, turned by i.  Selects and exact
                // signs instead of branches: a warp's teams hold different fields
                // (an evaluation at 64^2 FP64 9,240 cycles with branches, 8,040 without).
                const Real tr = (Real)t;
                const Real kys = (f & 1) ? -(Real)ky : (Real)ky;
                const bool turn = f >= 2;
                const Real sx = f == 0 ? (Real)1 : (Real)-1, sy = f == 1 ? (Real)-1 : (Real)1;
                C v[1][E];
                Real sc[E];
#pragma unroll
                for (int m = 0; m < E; ++m) {
                    v[0][m] = sX[slot * N + t + T * m];
                    sc[m] = sI[slot * N + t + T * m];
                }
#pragma unroll
                for (int m = 0; m < E; ++m) {
                    const Real kx = kx_of<Real, N, T>(m, t, tr);
                    const Real s1 = turn ? (Real)1 : sc[m];
                    const C X = cmake<C>(mul_rn(s1, v[0][m].x), mul_rn(s1, v[0][m].y));
                    const C d = cmake<C>(fma_rn(kx, X.x, -mul_rn(kys, X.y)), fma_rn(kx, X.y, mul_rn(kys, X.x)));
                    v[0][m] = cmake<C>(mul_rn(sx, turn ? d.y : d.x), mul_rn(sy, turn ? d.x : d.y));
                }
                if (t == 0 && ky == 0) v[0][0] = cmake<C>(0, 0);
                fft_batched<N, +1, 1>(v, pol, seed, t);
                if (on) {
                    const unsigned base = smem_addr(sF + (size_t)ky * L::KS + f * RPC);
#pragma unroll
                    for (int m = 0; m < E; ++m) {
                        const int x = t + T * m;
                        const unsigned local = base + (unsigned)sizeof(C) * (x % RPC);
                        if constexpr (CL == 1) sF[(size_t)ky * L::KS + f * RPC + x] = v[0][m];
                        else cluster_store(cluster_addr(local, x / RPC), v[0][m]);
                    }
                }
            }
            cluster_sync<CL>();
            if (s == 1 && step > 0) {
#pragma unroll
                for (int r = 0; r < CL; ++r) stop |= s_stop[r] != 0;
                if (stop) break;  // the same in every block
            }
            // --- rows: inverse y-FFTs of Z1 = U + iV and Z2 = WX + iWY (fields as the passes')
            for (int u0 = 0; u0 + warp_team < 2 * RPC; u0 += L::TEAMS) {
                const int u = u0 + team;
                const bool on = u < 2 * RPC;
                const int g = on ? u >> 1 : 0, b = u & 1;
                C v[1][E];
#pragma unroll
                for (int m = 0; m < E; ++m) {
                    const int y = t + T * m;
                    const int yy = (y <= N / 2) ? y : N - y;
                    const C* const plus = sF + (size_t)yy * L::KS + (2 * b) * RPC + g;
                    C p = cmake<C>(0, 0);
                    if (yy < kx_cols) {
                        p = y <= N / 2 ? plus[0] : cconj(plus[RPC]);
                        if (y == 0 || y == N / 2) {
                            const C q = plus[RPC];
                            p = cmake<C>((Real)0.5 * (p.x + q.x), (Real)0.5 * (p.y - q.y));
                        }
                    }
                    v[0][m] = p;
                }
                fft_batched<N, +1, 1>(v, pol, seed, t);
                // n = u w_x + v w_y: the row's two teams (neighbours in the warp)
                // exchange halves, team 0 forms the first half of the elements
#pragma unroll
                for (int m = 0; m < E / 2; ++m) {
                    const C mine = b == 0 ? v[0][m] : v[0][m + E / 2];
                    const C give = b == 0 ? v[0][m + E / 2] : v[0][m];
                    const Real ox = __shfl_xor_sync(0xffffffffu, give.x, T);
                    const Real oy = __shfl_xor_sync(0xffffffffu, give.y, T);
                    const C uv = b == 0 ? mine : cmake<C>(ox, oy);
                    const C wg = b == 0 ? cmake<C>(ox, oy) : mine;
                    if (on) sP[g * N + t + T * (m + b * (E / 2))] = fma_rn(uv.x, wg.x, mul_rn(uv.y, wg.y));
                }
            }
            __syncthreads();
            // --- rows: packed forward y-FFT of each row pair, split into two half spectra
            for (int u0 = 0; u0 + warp_team < RPC / 2; u0 += L::TEAMS) {
                const int u = u0 + team;
                const bool on = u < RPC / 2;
                const int p = on ? u : 0;
                C z[1][E];
#pragma unroll
                for (int m = 0; m < E; ++m) {
                    const int y = t + T * m;
                    z[0][m] = cmake<C>(sP[(2 * p) * N + y], sP[(2 * p + 1) * N + y]);
                }
                fft_batched<N, -1, 1>(z, pol, seed, t);
#pragma unroll
                for (int m = 0; m < E; ++m) pol.sm[TeamLayout<N>::template slot<C>(t + T * m)] = z[0][m];
                pol.sync();
                if (on) {
#pragma unroll
                    for (int m = 0; m < E; ++m) {
                        const int k = t + T * m;
                        if (k < nl_cols) {  // k <= N/2
                            const C zk = pol.sm[TeamLayout<N>::template slot<C>(k)];
                            const C zm = pol.sm[TeamLayout<N>::template slot<C>((N - k) & (N - 1))];
                            const C ra = cmake<C>((Real)0.5 * (zk.x + zm.x), (Real)0.5 * (zk.y - zm.y));
                            const C rb = cmake<C>((Real)0.5 * (zk.y + zm.y), (Real)0.5 * (zm.x - zk.x));
                            const int at = (k / CL) * N + rank * RPC + 2 * p;
                            if constexpr (CL == 1) {
                                sN[at] = ra;
                                sN[at + 1] = rb;
                            } else {
                                const unsigned to = cluster_addr(smem_addr(sN + at), k % CL);
                                cluster_store(to, ra);
                                cluster_store(to + (unsigned)sizeof(C), rb);
                            }
                        }
                    }
                }
                pol.sync();  // the region is reused by this team's next transform
            }
            cluster_sync<CL>();
            // --- columns: forward x-FFT and the evaluation's epilogue
            double bsum = 0.0;
            bool bad = false;
            const bool last = s == nstage;
            const Real bc = (Real)(SCHEME == RES_EXPLICIT ? (s == 1 || last ? 1.0 : 2.0)
                                                          : (s == 1 || last ? 1.0 / 6.0 : 1.0 / 3.0));
            const Real adt = (Real)(a.dt * (s < 3 ? 0.5 : 1.0));
            for (int u0 = 0; u0 + warp_team < slots; u0 += L::TEAMS) {
                const int u = u0 + team;
                const bool on = u < slots;
                const int slot = on ? u : 0;
                const int ky = rank + CL * slot;
                const bool conj = ky == 0 && (a.conj_quirk || (!rhs_only && s == 1));
                C v[1][E];
#pragma unroll
                for (int m = 0; m < E; ++m) v[0][m] = sN[slot * N + t + T * m];
                C p0[ab4 ? E : 1], p1[ab4 ? E : 1], p2[ab4 ? E : 1];
                if constexpr (ab4) {
#pragma unroll
                    for (int m = 0; m < E; ++m) {
                        const size_t g = (size_t)(t + T * m) * a.ldc + ky;
                        p0[m] = h0[g];
                        p1[m] = h1[g];
                        p2[m] = h2[g];
                    }
                }
                fft_batched<N, -1, 1>(v, pol, seed, t);
                // ForceConjugacy side effect on the state (solver.c:1031, 2096-2103),
                // from the evaluation's input, which is replaced below
                if (conj && on) {
#pragma unroll
                    for (int m = E / 2; m < E; ++m) {
                        const int i = t + T * m;
                        if (i > N / 2) {
                            const C w = cconj(sX[N - i]);
                            if constexpr (rhs_only) a.state[(size_t)i * a.ldc] = w;
                            else sW[i] = w;
                        }
                    }
                }
                pol.sync();
                if (!on) continue;
                // All operands are read before any result is written: the loops
                // below are then straight-line code whose latencies overlap.
                const int q0 = slot * N + t;
                const size_t g0 = (size_t)t * a.ldc + ky;
                Real d[E];
#pragma unroll
                for (int m = 0; m < E; ++m) d[m] = sD[q0 + T * m];
                const bool mean0 = t == 0 && ky == 0;
#pragma unroll
                for (int m = 0; m < E; ++m) {
                    // normalisation and zero mean (solver.c:998-1013), dealiasing
                    // (solver.c:1039-1099; 2/3 mask or Hou-Li factor)
                    C r = cscale(v[0][m], a.norm2);
                    if (m == 0 && mean0) r = cmake<C>(0, 0);
                    if (a.dealias != 0) r = cscale(r, d[m]);
                    else if (d[m] == (Real)0) r = cmake<C>(0, 0);
                    v[0][m] = r;
                }
                // forcing (solver.c:1022-1027)
                if (a.has_force && ky == a.force_j) {
#pragma unroll
                    for (int m = 0; m < E; ++m)
                        if (t + T * m == a.force_i) v[0][m] = cadd(v[0][m], a.force_val);
                }
                if constexpr (GEN) {
                    if (a.force_field) {
#pragma unroll
                        for (int m = 0; m < E; ++m) v[0][m] = cadd(v[0][m], a.force_field[g0 + (size_t)(T * m) * a.ldc]);
                    }
                }
                C* const store = rhs_only ? a.rhs : ab4 ? h3 : (SCHEME == RES_CN && s == 1) ? a.rhs : nullptr;
                if (store) {
#pragma unroll
                    for (int m = 0; m < E; ++m) store[g0 + (size_t)(T * m) * a.ldc] = v[0][m];
                }
                if constexpr (rhs_only) {
                    if (a.out64) {
#pragma unroll
                        for (int m = 0; m < E; ++m)
                            a.out64[(size_t)(t + T * m) * a.nyf + ky] = make_double2((double)v[0][m].x, (double)v[0][m].y);
                    }
                }
                if constexpr (!rhs_only) {
                    C w[E];
#pragma unroll
                    for (int m = 0; m < E; ++m) w[m] = sW[q0 + T * m];
                    // linear term of explicit RK4 stages (solver.c:664-684)
                    if constexpr (SCHEME == RES_EXPLICIT) {
                        if (a.lin_stage) {
#pragma unroll
                            for (int m = 0; m < E; ++m) {
                                const C xs = s == 1 ? w[m] : sX[q0 + T * m];
                                const Real br = (Real)sCn[q0 + T * m].x;
                                const C r = a.lin_stage == 1 ? cadd(v[0][m], cscale(xs, br)) : csub(v[0][m], cscale(xs, br));
                                if (!(m == 0 && mean0)) v[0][m] = r;
                            }
                        }
                    }
                    C acc[ab4 ? 1 : E];
                    if constexpr (!ab4) {
#pragma unroll
                        for (int m = 0; m < E; ++m)
                            acc[m] = s == 1 ? cscale(v[0][m], bc) : cadd(sA[q0 + T * m], cscale(v[0][m], bc));
                    }
                    if (!last) {
                        if constexpr (!ab4) {
#pragma unroll
                            for (int m = 0; m < E; ++m) {
                                sA[q0 + T * m] = acc[m];
                                sX[q0 + T * m] = cadd(w[m], cscale(v[0][m], adt));
                            }
                        }
                    } else {
#pragma unroll
                        for (int m = 0; m < E; ++m) {
                            C tot;
                            if constexpr (ab4) {
                                // AB4 (solver.c:303-331): 55/24 N_n - 59/24 N_n-1 + 37/24 N_n-2 - 3/8 N_n-3
                                const Real dt = a.euler ? (Real)a.dt : (Real)1;
                                tot = cadd(cadd(cadd(cscale(v[0][m], dt * (Real)(55.0 / 24.0)), cscale(p2[m], dt * (Real)(-59.0 / 24.0))),
                                                cscale(p1[m], dt * (Real)(37.0 / 24.0))),
                                           cscale(p0[m], dt * (Real)(-3.0 / 8.0)));
                            } else {
                                tot = acc[m];
                            }
                            C wn;
                            if (SCHEME == RES_EXPLICIT) {
                                wn = cadd(w[m], cscale(tot, (Real)(a.dt / 6.0)));
                            } else if (ab4 && a.euler) {
                                wn = cadd(w[m], tot);
                            } else {
                                // Crank-Nicolson factors (solver.c:853)
                                const double2 f = sCn[q0 + T * m];
                                wn = cn_update<C>(w[m], tot, (Real)f.x, (Real)f.y);
                            }
                            if (m == 0 && mean0) wn = cmake<C>(0, 0);
                            if constexpr (GEN) {
                                if (a.phase_only && !(m == 0 && mean0)) {
                                    // amplitude reset of the phase-only model (solver.c:822-824, 855-857)
                                    const double an = hypot((double)wn.x, (double)wn.y);
                                    if (an > 0.0) {
                                        const double sc = hypot((double)w[m].x, (double)w[m].y) / an;
                                        wn = cmake<C>((Real)((double)wn.x * sc), (Real)((double)wn.y * sc));
                                    }
                                }
                            }
                            w[m] = wn;
                        }
                        double mag = 0.0;
#pragma unroll
                        for (int m = 0; m < E; ++m) {
                            sW[q0 + T * m] = w[m];
                            sX[q0 + T * m] = w[m];
                            const double one = fabs((double)w[m].x) + fabs((double)w[m].y);
                            bad |= !isfinite(one);
                            mag += one;
                        }
                        bsum += (ky == 0 || 2 * ky == N) ? mag : 2.0 * mag;
                    }
                }
            }
            if (!rhs_only && last) {
                // SystemCheck (solver.c:2301-2326), as the final column pass: status bit 1 for
                // a non-finite state, bit 2 when this block's share of the bound
                // sum|w_hat|/(Nx Ny) is large enough for the whole to reach 1e100
                // (each warp tests an equal share of the block's).
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) bsum += __shfl_xor_sync(0xffffffffu, bsum, o);
                const bool anybad = __any_sync(0xffffffffu, bad);
                const bool big = !(bsum * a.inv_nxny < 1e100 / (double)(CL * (NT / 32)));
                if ((threadIdx.x & 31) == 0 && (anybad || big)) {
                    atomicOr(a.status, (anybad ? 1 : 0) | (big ? 2 : 0));
                    for (int r = 0; r < CL; ++r) cluster_store(cluster_addr(smem_addr(&s_stop[rank]), r), 1);
                }
                ++done;
                if (ab4) {
                    C* const oldest = const_cast<C*>(h0);
                    h0 = h1;
                    h1 = h2;
                    h2 = h3;
                    h3 = oldest;
                }
            }
            __syncthreads();  // the stage input is complete before the next derived spectra
        }
    }
    if constexpr (!rhs_only) {
        put_state(a.src64 ? L::SLOTS : slots);
        if (a.status && rank == 0 && threadIdx.x == 0) atomicAdd(a.status + 1, done);
    }
    cluster_sync<CL>();  // no block leaves while another may still store into its shared memory
}

// Sets the kernels' limits on the current device; false when the device cannot
// run the cluster (the pass kernels then serve these sizes too).
template <typename Real, int N>
struct ResLaunch {
    static constexpr int CL = ResShape<N>::CL;
    static constexpr size_t smem() { return ResLayout<Real, N>::bytes(); }

    static void config(cudaLaunchConfig_t& cfg, cudaLaunchAttribute& at) {
        cfg.gridDim = dim3(CL);
        cfg.blockDim = dim3(ResShape<N>::NT);
        cfg.dynamicSmemBytes = smem();
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = CL;
        at.val.clusterDim.y = at.val.clusterDim.z = 1;
        cfg.attrs = &at;
        cfg.numAttrs = 1;
    }
    template <int SCHEME, bool GEN>
    static bool setup_one() {
        const void* f = (const void*)resident_kernel<Real, N, SCHEME, GEN>;
        if (cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem()) != cudaSuccess ||
            (CL > 8 && cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)) {
            cudaGetLastError();
            return false;
        }
        cudaLaunchConfig_t cfg{};
        cudaLaunchAttribute at{};
        config(cfg, at);
        int clusters = 0;
        if (cudaOccupancyMaxActiveClusters(&clusters, f, &cfg) != cudaSuccess) {
            cudaGetLastError();
            return false;
        }
        return clusters >= 1;
    }
    static bool setup() {
        return setup_one<RES_CN, false>() && setup_one<RES_CN, true>() && setup_one<RES_EXPLICIT, false>() &&
               setup_one<RES_EXPLICIT, true>() && setup_one<RES_AB4, false>() && setup_one<RES_AB4, true>() &&
               setup_one<RES_RHS, false>() && setup_one<RES_RHS, true>();
    }
    template <int SCHEME>
    static cudaError_t launch_one(const ResArgs<Real>& a, cudaStream_t s) {
        cudaLaunchConfig_t cfg{};
        cudaLaunchAttribute at{};
        config(cfg, at);
        cfg.stream = s;
        if (a.force_field || a.phase_only) return cudaLaunchKernelEx(&cfg, resident_kernel<Real, N, SCHEME, true>, a);
        return cudaLaunchKernelEx(&cfg, resident_kernel<Real, N, SCHEME, false>, a);
    }
    static cudaError_t launch(int scheme, const ResArgs<Real>& a, cudaStream_t s) {
        switch (scheme) {
            case RES_CN: return launch_one<RES_CN>(a, s);
            case RES_EXPLICIT: return launch_one<RES_EXPLICIT>(a, s);
            case RES_AB4: return launch_one<RES_AB4>(a, s);
            default: return launch_one<RES_RHS>(a, s);
        }
    }
};

}  // namespace ns2d
