// Instantiates the half-line stage kernel for one Nq (compiled once per Nq = 4..8 with
// -DRB_LINE_NQ=<nq>); pipelined_inst.cu routes to these entry points.
#include "line_kernel.cuh"

#ifndef RB_LINE_NQ
#error "RB_LINE_NQ must be defined"
#endif

#define RB_LCAT2(a, b) a##b
#define RB_LCAT(a, b) RB_LCAT2(a, b)

namespace rb200 {

namespace {

template <int COMBO, typename T, bool BATCH, bool STG>
cudaError_t launch_m(const PipeArgs& a, const PipeBatch& b, int grid, cudaStream_t s, int* blocks_per_sm) {
    constexpr int Q = RB_LINE_NQ;
    auto kern = pipelined_stage_kernel<COMBO, T, BATCH, Q, STG>;
    constexpr size_t smem = sizeof(line::Smem<T, Q>);
    static std::atomic<uint64_t> configured{0};
    cudaError_t err = ensure_smem_limit(kern, (int)smem, configured);
    if (err != cudaSuccess) return err;
    if (blocks_per_sm)  // occupancy query only
        return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, kern, line::Shape<Q>::TH, smem);
    // a tick's first stage follows host-written chunk tables: plain order; its others read what
    // that stage has read, and wait for the stage before them like a single state's
    if (!BATCH || b.stage > 0) return launch_pdl(kern, grid, line::Shape<Q>::TH, smem, s, a, b);
    kern<<<grid, line::Shape<Q>::TH, smem, s>>>(a, b);
    return cudaGetLastError();
}

template <int COMBO, typename T, bool BATCH>
cudaError_t launch_l(const PipeArgs& a, const PipeBatch& b, int grid, cudaStream_t s, int* bps) {
    if (bps || a.mode >= MODE_STAGE) return launch_m<COMBO, T, BATCH, true>(a, b, grid, s, bps);
    if constexpr (sizeof(T) == 8 && !BATCH) return launch_m<COMBO, T, BATCH, false>(a, b, grid, s, bps);
    return cudaErrorInvalidValue;
}

template <typename T>
cudaError_t launch_t(int combo, bool batch, const PipeArgs& a, const PipeBatch& b, int grid, cudaStream_t s, int* bps) {
    if (batch) {
        if constexpr (RB_LINE_NQ % 2 == 0) {
            if (combo == EUL_KG) return launch_l<EUL_KG, T, true>(a, b, grid, s, bps);
        }
        return cudaErrorInvalidValue;
    }
    switch (combo) {
        case EUL_KG: return launch_l<EUL_KG, T, false>(a, b, grid, s, bps);
        case EUL_EC: return launch_l<EUL_EC, T, false>(a, b, grid, s, bps);
        case EUL_WEAK:  // one kernel; the tables tell the two forms apart
        case EUL_FDC: return launch_l<EUL_WEAK, T, false>(a, b, grid, s, bps);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace

// blocks_per_sm != nullptr: occupancy query, nothing is launched.
cudaError_t RB_LCAT(launch_line_q, RB_LINE_NQ)(int combo, int fp32, bool batch, const PipeArgs& a, const PipeBatch& b,
                                               int grid, cudaStream_t s, int* blocks_per_sm) {
    return fp32 ? launch_t<float>(combo, batch, a, b, grid, s, blocks_per_sm)
                : launch_t<double>(combo, batch, a, b, grid, s, blocks_per_sm);
}

}  // namespace rb200
