// Instantiations and launch helpers of the pipelined 3-D stage kernels: Euler on bricks (the
// half-line kernel of line_inst.cu), weak-form advection on bricks and curved grids; one
// state (the DGSEM handle) or the chunks of a serving class (BATCH).
#include "pipelined_adv.cuh"
#include "pipelined_curved.cuh"
#include "pipelined_kernel.cuh"

namespace rb200 {

#define RB_LINE_DECL(Q)                                                                                            \
    cudaError_t launch_line_q##Q(int combo, int fp32, bool batch, const PipeArgs& a, const PipeBatch& b, int grid, \
                                 cudaStream_t s, int* blocks_per_sm);
RB_LINE_DECL(4) RB_LINE_DECL(5) RB_LINE_DECL(6) RB_LINE_DECL(7) RB_LINE_DECL(8)

// The Euler law: the half-line kernel (line_inst.cu).
static cudaError_t launch_line(int nq, int combo, int fp32, bool batch, const PipeArgs& a, const PipeBatch& b, int grid,
                               cudaStream_t s, int* bps) {
    switch (nq) {
        case 4: return launch_line_q4(combo, fp32, batch, a, b, grid, s, bps);
        case 5: return launch_line_q5(combo, fp32, batch, a, b, grid, s, bps);
        case 6: return launch_line_q6(combo, fp32, batch, a, b, grid, s, bps);
        case 7: return launch_line_q7(combo, fp32, batch, a, b, grid, s, bps);
        case 8: return launch_line_q8(combo, fp32, batch, a, b, grid, s, bps);
        default: return cudaErrorInvalidValue;
    }
}

// The advection law: one field, pipea::npt<Q>() nodes a thread.
template <typename T, bool BATCH, int Q>
static cudaError_t launch_a(const PipeArgs& a, const PipeBatch& b, int grid, cudaStream_t s) {
    auto kern = pipelined_adv_kernel<T, BATCH, Q>;
    static std::atomic<uint64_t> configured{0};
    cudaError_t err = ensure_smem_limit(kern, (int)sizeof(pipea::Smem<T, Q>), configured);
    if (err != cudaSuccess) return err;
    // (a serving tick's first stage follows host-written chunk tables: plain order)
    if (!BATCH || b.stage > 0)
        return launch_pdl(kern, grid, Q * Q * Q / pipea::npt<Q>(), sizeof(pipea::Smem<T, Q>), s, a, b);
    kern<<<grid, Q * Q * Q / pipea::npt<Q>(), sizeof(pipea::Smem<T, Q>), s>>>(a, b);
    return cudaGetLastError();
}

template <typename T, bool BATCH>
static cudaError_t launch_adv(int nq, const PipeArgs& a, const PipeBatch& b, int grid, cudaStream_t s) {
    switch (nq) {
        case 4: return launch_a<T, BATCH, 4>(a, b, grid, s);
        case 6: return launch_a<T, BATCH, 6>(a, b, grid, s);
        case 8: return launch_a<T, BATCH, 8>(a, b, grid, s);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_pipelined(int nq, int combo, int fp32, const PipeArgs& a, int grid, cudaStream_t s) {
    const PipeBatch none{};
    if (combo != ADV_WEAK) return launch_line(nq, combo, fp32, false, a, none, grid, s, nullptr);
    return fp32 ? launch_adv<float, false>(nq, a, none, grid, s) : launch_adv<double, false>(nq, a, none, grid, s);
}

cudaError_t launch_pipelined_batch(int nq, int combo, int fp32, const PipeArgs& a, const PipeBatch& b, int grid,
                                   cudaStream_t s) {
    if (combo != ADV_WEAK) return launch_line(nq, combo, fp32, true, a, b, grid, s, nullptr);
    return fp32 ? launch_adv<float, true>(nq, a, b, grid, s) : launch_adv<double, true>(nq, a, b, grid, s);
}

template <typename T, bool BATCH, int Q>
static int occupancy_a() {
    auto kern = pipelined_adv_kernel<T, BATCH, Q>;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(pipea::Smem<T, Q>)) !=
        cudaSuccess)
        return 0;
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, Q * Q * Q / pipea::npt<Q>(), sizeof(pipea::Smem<T, Q>)) !=
        cudaSuccess)
        return 0;
    return n;
}

template <typename T, bool BATCH>
static int occupancy_adv(int nq) {
    switch (nq) {
        case 4: return occupancy_a<T, BATCH, 4>();
        case 6: return occupancy_a<T, BATCH, 6>();
        case 8: return occupancy_a<T, BATCH, 8>();
        default: return 0;
    }
}

static int occupancy_line(int nq, int combo, int fp32, bool batch) {
    int n = 0;
    return launch_line(nq, combo, fp32, batch, PipeArgs{}, PipeBatch{}, 0, nullptr, &n) == cudaSuccess ? n : 0;
}

int pipelined_blocks_per_sm(int nq, int combo, int fp32) {
    if (combo != ADV_WEAK) return occupancy_line(nq, combo, fp32, false);
    return fp32 ? occupancy_adv<float, false>(nq) : occupancy_adv<double, false>(nq);
}

int pipelined_batch_blocks_per_sm(int nq, int combo, int fp32) {
    if (combo != ADV_WEAK) return occupancy_line(nq, combo, fp32, true);
    return fp32 ? occupancy_adv<float, true>(nq) : occupancy_adv<double, true>(nq);
}

// The curved-grid kernel (Kennedy-Gruber).  blocks_per_sm != nullptr: occupancy query only.
template <typename T>
static cudaError_t launch_c(const PipeCurvedArgs& a, int grid, cudaStream_t s, int* blocks_per_sm) {
    auto kern = pipelined_curved_kernel<T>;
    constexpr size_t smem = sizeof(pipec::Smem<T>);
    static std::atomic<uint64_t> configured{0};
    cudaError_t err = ensure_smem_limit(kern, (int)smem, configured);
    if (err != cudaSuccess) return err;
    if (blocks_per_sm) return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, kern, pipec::NT, smem);
    return launch_pdl(kern, grid, pipec::NT, smem, s, a);
}

cudaError_t launch_pipelined_curved(int fp32, const PipeCurvedArgs& a, int grid, cudaStream_t s) {
    return fp32 ? launch_c<float>(a, grid, s, nullptr) : launch_c<double>(a, grid, s, nullptr);
}

int pipelined_curved_blocks_per_sm(int fp32) {
    int n = 0;
    const PipeCurvedArgs none{};
    return (fp32 ? launch_c<float>(none, 0, nullptr, &n) : launch_c<double>(none, 0, nullptr, &n)) == cudaSuccess ? n : 0;
}

}  // namespace rb200
