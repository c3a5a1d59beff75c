// engine.cuh -- per-grid-size launch tables for the step kernels.
#pragma once
#include <cuda_runtime.h>

#include "aux_kernels.cuh"

namespace ns2d {

// Column-tile width (ky columns per block) and row pairs per block.  Column
// accesses fetch TC * 16 B per row in FP64, so wider tiles use each row's lines
// better, while narrower ones spread a pass over more SMs.  With the emptied
// columns left out a pass at 256 has 86 columns and at 512 171: two to a block
// there (a step at 512^2 FP64 57.4 us against 68.2 with four; one: 57.5; at 256^2
// 43.2 against 47.2 with four), four at 1024 (three: 153.6 us against 144.2, the
// six warps weigh on the four schedulers as eight do and the 48-byte rows break
// sectors; two: 141.8, but 4 us more for the final pass).
template <typename Real, int N>
struct Shape {
    static constexpr int T = Plan<N>::T;
    static constexpr int TC_RAW = 128 / T < 2 ? 2 : 128 / T;
    static constexpr int TC = (N == 16) ? 8 : (N == 1024) ? 4 : (N == 256) ? 2 : TC_RAW;
    // The common step's stage pass, which moves everything by TMA, two columns per
    // block at 1024 in FP64: two blocks share an SM and overlap their phases (22.5 us
    // a launch against 24.0).  Passes that read per-thread arrays keep four (AB4 step
    // 47 us, 53 with two; 32-byte rows are two to a line), and so does FP32 (17.7
    // against 19.1: 16-byte rows).
    static constexpr int TC_STAGE = (N == 1024 && sizeof(Real) == 8) ? 2 : TC;
    static_assert(TC % TC_STAGE == 0, "ColArgs::kdead");
    static constexpr int PAIRS_RAW = (N == 256) ? 1 : (128 / T) / 2 < 1 ? 1 : (128 / T) / 2;
    static constexpr int PAIRS = PAIRS_RAW > N / 2 ? N / 2 : PAIRS_RAW;
};

template <typename Real, int N>
struct Launch {
    using C = typename Cx<Real>::T;
    using S = Shape<Real, N>;
    static constexpr int SIZE = N;
    static constexpr size_t col_smem() { return ColSmem<Real, N, S::TC>::bytes(); }
    static constexpr size_t col_tma_smem() { return ColSmem<Real, N, S::TC>::bytes_tma() + 1024; }
    static constexpr size_t stage_tma_smem() { return ColSmem<Real, N, S::TC_STAGE>::bytes_tma() + 1024; }
    static constexpr size_t row_smem() { return RowSmem<Real, N, 2 * S::PAIRS>::bytes(); }
    static constexpr size_t inv_smem() { return sizeof(C) * SmemLayout<N, S::TC>::ELEMS; }
    static constexpr size_t c2r_smem() {
        size_t a = sizeof(C) * SmemLayout<N, 2 * S::PAIRS>::ELEMS;
        size_t b = sizeof(Real) * N * 2 * S::PAIRS;
        return a > b ? a : b;
    }

    template <int MODE, int SCH, typename F>
    static void set_col(const F& set) {
        set((const void*)col_kernel<Real, N, S::TC, MODE, SCH>, col_smem());
        set((const void*)col_tma_kernel<Real, N, S::TC, MODE, SCH>, col_tma_smem());
    }
    // A pass's launch; programmatic dependent launch where the passes use it and are
    // queued one by one (256^2: a step of changing dt 81 -> 71 us, a Dormand-Prince
    // step 155 -> 134).  Not into a graph, whose own edges are faster (512^2 FP64 57
    // us a step, 73 with programmatic ones).
    template <typename... P, typename... A>
    static void launch(void (*f)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, const A&... args) {
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = grid;
        cfg.blockDim = block;
        cfg.dynamicSmemBytes = smem;
        cfg.stream = s;
        cudaLaunchAttribute at{};
        at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at.val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = &at;
        cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
        if (pass_pdl(N) && cudaStreamIsCapturing(s, &cap) == cudaSuccess && cap == cudaStreamCaptureStatusNone)
            cfg.numAttrs = 1;
        cudaLaunchKernelEx(&cfg, f, args...);  // a failure is left for cudaGetLastError
    }
    static cudaError_t setup() {
        cudaError_t e = cudaSuccess;
        auto set = [&](const void* f, size_t bytes) {
            if (e == cudaSuccess)
                e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
        };
        set_col<COL_P1, SCH_CNX>(set);
        set_col<COL_RHS, SCH_CNX>(set);
        set_col<COL_STAGE, SCH_CNX>(set);
        set_col<COL_STAGE, SCH_EX>(set);
        set_col<COL_STAGE, SCH_DP>(set);
        set_col<COL_FINAL, SCH_CNX>(set);
        set_col<COL_FINAL, SCH_EX>(set);
        set_col<COL_FINAL, SCH_AB4>(set);
        set_col<COL_NEXT, SCH_CNX>(set);
        set_col<COL_NEXT, SCH_EX>(set);
        set_col<COL_NEXT, SCH_AB4>(set);
        set((const void*)col_tma_kernel<Real, N, S::TC_STAGE, COL_STAGE, SCH_CN>, stage_tma_smem());
        set((const void*)col_tma_kernel<Real, N, S::TC, COL_FINAL, SCH_CN>, col_tma_smem());
        set((const void*)col_tma_kernel<Real, N, S::TC, COL_NEXT, SCH_CN>, col_tma_smem());
        set((const void*)row_kernel<Real, N, S::PAIRS>, row_smem());
        set((const void*)col_inv_kernel<Real, N, S::TC>, inv_smem());
        set((const void*)row_c2r_kernel<Real, N, S::PAIRS, R2_MAXABS>, c2r_smem());
        set((const void*)row_c2r_kernel<Real, N, S::PAIRS, R2_CFL>, c2r_smem());
        set((const void*)row_c2r_kernel<Real, N, S::PAIRS, R2_STORE>, c2r_smem());
        set((const void*)fwd_kernel<Real, N, S::TC, FWD_ROWS>, inv_smem());
        set((const void*)fwd_kernel<Real, N, S::TC, FWD_COLS>, inv_smem());
        return e;
    }

    template <int MODE, int SCH>
    static void col_one(const ColArgs<Real>& a, cudaStream_t s, const ColMaps* maps, const ColMaps* stage_maps) {
        dim3 grid((a.nyf + S::TC - 1) / S::TC), block(S::T * S::TC);
        if (maps && col_tma_ok(a)) {
            if constexpr (SCH == SCH_CNX && (MODE == COL_STAGE || MODE == COL_FINAL || MODE == COL_NEXT)) {
                if (MODE == COL_STAGE && a.dealias == 0 && !a.rhs_store && stage_maps) {
                    dim3 sgrid((a.nyf + S::TC_STAGE - 1) / S::TC_STAGE), sblock(S::T * S::TC_STAGE);
                    launch(col_tma_kernel<Real, N, S::TC_STAGE, MODE, SCH_CN>, sgrid, sblock, stage_tma_smem(), s, a, *stage_maps);
                    return;
                }
                if (MODE != COL_STAGE && a.dealias == 0 && !a.rhs_store) {
                    launch(col_tma_kernel<Real, N, S::TC, MODE, SCH_CN>, grid, block, col_tma_smem(), s, a, *maps);
                    return;
                }
            }
            launch(col_tma_kernel<Real, N, S::TC, MODE, SCH>, grid, block, col_tma_smem(), s, a, *maps);
        } else {
            launch(col_kernel<Real, N, S::TC, MODE, SCH>, grid, block, col_smem(), s, a);
        }
    }
    // scheme: SCH_CN, SCH_EX, SCH_AB4 or SCH_DP (stage and final passes); maps: tensor maps
    // of the arrays the pass reads and writes (null: per-thread copies), stage_maps
    // the same for the stage pass's tiles.
    static void col(int mode, int scheme, const ColArgs<Real>& a, cudaStream_t s, const ColMaps* maps, const ColMaps* stage_maps) {
        switch (mode) {
            case COL_P1: col_one<COL_P1, SCH_CNX>(a, s, maps, stage_maps); break;
            case COL_RHS: col_one<COL_RHS, SCH_CNX>(a, s, maps, stage_maps); break;
            case COL_STAGE:
                if (scheme == SCH_EX) col_one<COL_STAGE, SCH_EX>(a, s, maps, stage_maps);
                else if (scheme == SCH_DP) col_one<COL_STAGE, SCH_DP>(a, s, maps, stage_maps);
                else col_one<COL_STAGE, SCH_CNX>(a, s, maps, stage_maps);
                break;
            case COL_NEXT:
                if (scheme == SCH_EX) col_one<COL_NEXT, SCH_EX>(a, s, maps, stage_maps);
                else if (scheme == SCH_AB4) col_one<COL_NEXT, SCH_AB4>(a, s, maps, stage_maps);
                else col_one<COL_NEXT, SCH_CNX>(a, s, maps, stage_maps);
                break;
            default:
                if (scheme == SCH_EX) col_one<COL_FINAL, SCH_EX>(a, s, maps, stage_maps);
                else if (scheme == SCH_AB4) col_one<COL_FINAL, SCH_AB4>(a, s, maps, stage_maps);
                else col_one<COL_FINAL, SCH_CNX>(a, s, maps, stage_maps);
                break;
        }
    }
    static void row(const RowArgs<Real>& a, cudaStream_t s) {
        dim3 grid(N / (2 * S::PAIRS)), block(S::T * 2 * S::PAIRS);
        launch(row_kernel<Real, N, S::PAIRS>, grid, block, row_smem(), s, a);
    }
    static void col_inv(const InvArgs<Real>& a, cudaStream_t s) {
        dim3 grid((a.nyf + S::TC - 1) / S::TC), block(S::T * S::TC);
        col_inv_kernel<Real, N, S::TC><<<grid, block, inv_smem(), s>>>(a);
    }
    // Forward transform passes (set-up only): rows of a real [N][N] field, then columns.
    static void fwd(int pass, const double* real_in, const C* in, C* out, int nlines, int ldc, const C* tw,
                    cudaStream_t s) {
        dim3 grid((nlines + S::TC - 1) / S::TC), block(S::T * S::TC);
        if (pass == FWD_ROWS)
            fwd_kernel<Real, N, S::TC, FWD_ROWS><<<grid, block, inv_smem(), s>>>(real_in, in, out, nlines, ldc, tw);
        else
            fwd_kernel<Real, N, S::TC, FWD_COLS><<<grid, block, inv_smem(), s>>>(real_in, in, out, nlines, ldc, tw);
    }
    static void row_c2r(int op, const RowC2RArgs<Real>& a, cudaStream_t s) {
        dim3 grid(N / (2 * S::PAIRS)), block(S::T * 2 * S::PAIRS);
        switch (op) {
            case R2_MAXABS: row_c2r_kernel<Real, N, S::PAIRS, R2_MAXABS><<<grid, block, c2r_smem(), s>>>(a); break;
            case R2_CFL: row_c2r_kernel<Real, N, S::PAIRS, R2_CFL><<<grid, block, c2r_smem(), s>>>(a); break;
            default: row_c2r_kernel<Real, N, S::PAIRS, R2_STORE><<<grid, block, c2r_smem(), s>>>(a); break;
        }
    }
};

// Runtime dispatch over the supported sizes.
template <typename Real, typename F>
inline bool with_size(int n, F&& f) {
    switch (n) {
        case 16: f(Launch<Real, 16>{}); return true;
        case 32: f(Launch<Real, 32>{}); return true;
        case 64: f(Launch<Real, 64>{}); return true;
        case 128: f(Launch<Real, 128>{}); return true;
        case 256: f(Launch<Real, 256>{}); return true;
        case 512: f(Launch<Real, 512>{}); return true;
        case 1024: f(Launch<Real, 1024>{}); return true;
        case 2048: f(Launch<Real, 2048>{}); return true;
        default: return false;
    }
}

// The launch functions of one grid size in one precision.  Each size and precision
// is a module of its own (engine_size.cu): the first handle of a program loads the
// kernels of its size and no others.
template <typename Real>
struct EngineOps {
    int tc, tc_stage;  // column-tile widths: of the passes, of the common step's stage pass
    cudaError_t (*setup)();
    void (*col)(int mode, int scheme, const ColArgs<Real>& a, cudaStream_t s, const ColMaps* maps, const ColMaps* stage_maps);
    void (*row)(const RowArgs<Real>& a, cudaStream_t s);
    void (*col_inv)(const InvArgs<Real>& a, cudaStream_t s);
    void (*fwd)(int pass, const double* real_in, const typename Cx<Real>::T* in, typename Cx<Real>::T* out, int nlines,
                int ldc, const typename Cx<Real>::T* tw, cudaStream_t s);
    void (*row_c2r)(int op, const RowC2RArgs<Real>& a, cudaStream_t s);
};
template <typename Real, int N>
const EngineOps<Real>* engine_ops_of();
// Null for a size that has none.
template <typename Real>
inline const EngineOps<Real>* engine_ops(int n) {
    const EngineOps<Real>* ops = nullptr;
    with_size<Real>(n, [&](auto L) { ops = engine_ops_of<Real, decltype(L)::SIZE>(); });
    return ops;
}

}  // namespace ns2d
