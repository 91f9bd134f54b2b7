// What the pipelined 3-D stage kernels share: their arguments and tables, the sequence of
// elements of a CTA (one state, or the chunks of a serving class), bulk copies, and bounded
// waits.  Every wait on an mbarrier is bounded: after kWaitLimit polls the CTA records
// RB200 status TIMEOUT in *A.status and returns.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <cmath>

#include "rb200_internal.h"
#include "stage_kernel.cuh"  // cp.async helpers, log_mean, Mode

namespace rb200 {

struct PipeArgs {
    const double* q_in;
    double* q_out;
    void* dq;
    const double* elem_geo;  // (4, E)
    const int32_t* nbr;      // (6, E); -2 marks a mortar face of an adapted grid
    const double* ncflux;    // mortar face fluxes ((6, E) faces x (Ns, Nfp)), or null
    int32_t* status;         // device status word (0 = ok)
    int64_t E;        // elements e_begin..E-1 are computed (one state)
    int64_t e_begin;
    int32_t mode;
    int32_t surface_rusanov;
    double rka, rkb_dt;
    double S[64];    // the volume term's table, entry a*Nq + id: see pipe_tables
    double w[8];
    double winv[8];  // 1 / w
    double adv[3];   // advection velocity (advection law only)
    double gas[3];   // gamma, gamma - 1, 1 / (2 (gamma - 1)) (Euler)
    float gasf[3];
    float Sf[64];    // (float)S, for FP32 arithmetic on table entries at fixed indices
};

// Fills the constants and tables of `p` from gamma, D[i + nq*j] = l_j'(r_i) and the weights w:
// * advection: D[a,id] w_a / w_id;
// * Euler flux differencing (KG, EC): D[a,id] w_a - D[id,a] w_id, which is skew;
// * Euler weak form: D[a,id] w_a;
// * Euler central flux differencing: half the skew table, and on the diagonal half its column
//   sums (the node's own flux in sum_a (F_a + F_id) / 2 Q[a,id]).
// Returns whether the half-line kernel's reading of the Euler tables holds: w even and the
// table odd under reflection of the line, to 8 roundings (every Lobatto line's are).
inline bool pipe_tables(PipeArgs& p, int combo, int nq, double gamma, const double* D, const double* w) {
    p.gas[0] = gamma, p.gas[1] = gamma - 1.0, p.gas[2] = 1.0 / (2.0 * (gamma - 1.0));
    for (int i = 0; i < 3; ++i) p.gasf[i] = (float)p.gas[i];
    for (int i = 0; i < nq; ++i) {
        p.w[i] = w[i];
        p.winv[i] = 1.0 / w[i];
    }
    for (int a = 0; a < nq; ++a)
        for (int id = 0; id < nq; ++id) {
            double& s = p.S[a * nq + id];
            if (combo == ADV_WEAK) s = D[a + nq * id] * (w[a] / w[id]);
            else if (combo == EUL_WEAK) s = D[a + nq * id] * w[a];
            else s = D[a + nq * id] * w[a] - D[id + nq * a] * w[id];
        }
    if (combo == EUL_FDC) {
        for (int id = 0; id < nq; ++id) {
            double sum = 0.0;
            for (int a = 0; a < nq; ++a) sum += p.S[a * nq + id];
            for (int a = 0; a < nq; ++a)
                if (a != id) p.S[a * nq + id] *= 0.5;
            p.S[id * nq + id] = 0.5 * sum;
        }
    }
    double big = 0.0;
    for (int i = 0; i < nq * nq; ++i) big = std::max(big, std::fabs(p.S[i]));
    for (int i = 0; i < nq * nq; ++i) p.Sf[i] = (float)p.S[i];
    bool odd = true;
    const double tol = 8 * 2.220446049250313e-16;
    for (int a = 0; a < nq; ++a) {
        odd = odd && std::fabs(w[a] - w[nq - 1 - a]) <= tol * std::fabs(w[a]);
        for (int id = 0; id < nq; ++id)
            odd = odd && std::fabs(p.S[a * nq + id] + p.S[(nq - 1 - a) * nq + nq - 1 - id]) <= tol * big;
    }
    return odd;
}

// Whether D is odd under reflection of the line, to 8 roundings (every Lobatto line's is).
inline bool pipe_odd_derivative(int nq, const double* D) {
    double big = 0.0;
    for (int i = 0; i < nq * nq; ++i) big = std::max(big, std::fabs(D[i]));
    bool odd = true;
    for (int i = 0; i < nq * nq; ++i) odd = odd && std::fabs(D[i] + D[nq * nq - 1 - i]) <= 8 * 2.220446049250313e-16 * big;
    return odd;
}

// Serving loop: the elements of a launch are the chunks of a class's running solves
// instead of the strided elements of one state (SolveDesc, Chunk: rb200_internal.h).
struct PipeBatch {
    const SolveDesc* solves;
    const Chunk* chunks;
    const int32_t* nchunks;  // chunk slots in use (device)
    const int64_t* tick;     // class tick counter (device)
    int32_t stage;           // 0..4: selects the ping-pong buffer with the tick
    double rkb;              // LSRK b coefficient of the stage (times each solve's dt)
};

// One element as the kernel sees it: its state's buffers and its index there.
struct ElemRef {
    const double* q;     // q_in of the element's state (neighbours are in the same state)
    double* q_out;
    void* dq;
    const double* geo;   // elem_geo of the state
    const int32_t* nbr;  // neighbour table of the state
    int64_t e;           // element index in its state; -1: none (end of the CTA's work)
    double rkb_dt;
};

namespace pipe {

constexpr int NS = 5, NAUX = 6;                    // fields and partner values of a node (Euler)
constexpr int PAD(int n) { return n + (n >> 3); }  // one slot of padding every 8 nodes

// Sizes of an element with Q nodes per direction (Q even: an element's state is then a
// whole number of 16-byte units, as the bulk copies need).
template <int Q>
struct Geo {
    static_assert(Q % 2 == 0 && Q >= 4 && Q <= 8, "Nq = 4, 6 or 8");
    static constexpr int NQ = Q, NP = Q * Q * Q, NFP = Q * Q, NSLOT = 6 * Q * Q, NPP = PAD(Q * Q * Q);
};
constexpr long kWaitLimit = 1L << 26;

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    return done != 0;
}

__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
            smem_addr(dst)),
        "l"(src), "r"(bytes), "r"(smem_addr(bar))
        : "memory");
}

__device__ __forceinline__ void cp_async8(void* dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async4(void* dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void fence_mbar_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }

// Partner values of a node, 6 a node: three 16-byte loads in FP64, a 16-byte and an 8-byte one
// in FP32 (i16, i8: the node's slots).
template <typename T, int N16, int N8>
struct Partners;
template <int N16, int N8>
struct Partners<double, N16, N8> {
    double2 v[3][N16];
    __device__ __forceinline__ void put(int i16, int, const double (&o)[6]) {
#pragma unroll
        for (int c = 0; c < 3; ++c) v[c][i16] = make_double2(o[2 * c], o[2 * c + 1]);
    }
    __device__ __forceinline__ void get(int i16, int, double (&o)[6]) const {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const double2 x = v[c][i16];
            o[2 * c] = x.x;
            o[2 * c + 1] = x.y;
        }
    }
};
template <int N16, int N8>
struct Partners<float, N16, N8> {
    float4 a[N16];
    float2 b[N8];
    __device__ __forceinline__ void put(int i16, int i8, const float (&o)[6]) {
        a[i16] = make_float4(o[0], o[1], o[2], o[3]);
        b[i8] = make_float2(o[4], o[5]);
    }
    __device__ __forceinline__ void get(int i16, int i8, float (&o)[6]) const {
        const float4 x = a[i16];
        const float2 y = b[i8];
        o[0] = x.x, o[1] = x.y, o[2] = x.z, o[3] = x.w, o[4] = y.x, o[5] = y.y;
    }
};

__device__ __forceinline__ bool bounded_wait(uint64_t* bar, uint32_t parity) {
    long it = 0;
    while (!mbar_try_wait(bar, parity)) {
        if (++it > kWaitLimit) return false;
    }
    return true;
}

// 0-based volume node of face slot `slot` (faces x-, x+, y-, y+, z-, z+; Q*Q slots each)
// and the node of the opposite face with the same in-face index.
template <int Q = 8>
__device__ __forceinline__ void slot_nodes(int slot, int& vn, int& opp) {
    const int f = slot / (Q * Q), jf = slot % (Q * Q);
    const int dir = f >> 1, side = f & 1;
    const int j1 = jf % Q, j2 = jf / Q, c = side ? Q - 1 : 0;
    if (dir == 0) {
        vn = c + Q * (j1 + Q * j2);
        opp = (Q - 1 - c) + Q * (j1 + Q * j2);
    } else if (dir == 1) {
        vn = j1 + Q * (c + Q * j2);
        opp = j1 + Q * ((Q - 1 - c) + Q * j2);
    } else {
        vn = j1 + Q * (j2 + Q * c);
        opp = j1 + Q * (j2 + Q * (Q - 1 - c));
    }
}

// The CTA's sequence of elements, advanced by thread 0 one element ahead of the work.
// One state: elements blockIdx.x + k*gridDim.x.  Serving batch: the elements of chunks
// blockIdx.x + k*gridDim.x, in order.
template <bool BATCH>
struct Cursor {
    int64_t e = 0;  // one state: element; batch: index within the chunk
    int ci = 0;     // batch: chunk slot
    int nch = 0;    // batch: chunk slots in use

    __device__ bool start(const PipeArgs& A, const PipeBatch& B) {
        if constexpr (!BATCH) {
            e = A.e_begin + blockIdx.x;
            return e < A.E;
        } else {
            nch = *B.nchunks;
            ci = blockIdx.x;
            e = 0;
            return skip_empty(B);
        }
    }
    __device__ bool advance(const PipeArgs& A, const PipeBatch& B) {
        if constexpr (!BATCH) {
            e += gridDim.x;
            return e < A.E;
        } else {
            if (++e < B.chunks[ci].count) return true;
            ci += gridDim.x;
            e = 0;
            return skip_empty(B);
        }
    }
    __device__ bool skip_empty(const PipeBatch& B) {
        while (ci < nch && (B.chunks[ci].solve < 0 || B.chunks[ci].count <= 0)) ci += gridDim.x;
        return ci < nch;
    }
    __device__ void resolve(const PipeArgs& A, const PipeBatch& B, ElemRef& r) const {
        if constexpr (!BATCH) {
            r = ElemRef{A.q_in, A.q_out, A.dq, A.elem_geo, A.nbr, e, A.rkb_dt};
        } else {
            const Chunk c = B.chunks[ci];
            const SolveDesc& sd = B.solves[c.solve];
            const int par = (int)((*B.tick - sd.start_tick + B.stage) & 1);
            r = ElemRef{sd.q[par], sd.q[par ^ 1], sd.dq, sd.elem_geo, sd.nbr, c.first + e, B.rkb * sd.dt};
        }
    }
};

// Threads 0..9: one value each of the geometry (4) and neighbour ids (6) of element r
// into a shared slot (cp.async).
__device__ __forceinline__ void fetch_part(const ElemRef& r, int t, double (&geo)[4], int32_t (&nb)[8]) {
    if (t < 4) cp_async8(&geo[t], r.geo + 4 * r.e + t);
    else cp_async4(&nb[t - 4], r.nbr + 6 * r.e + (t - 4));
}

}  // namespace pipe

}  // namespace rb200
