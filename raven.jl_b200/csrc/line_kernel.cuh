// Persistent LSRK stage kernel of the Euler law for 3-D hexahedra on unwarped bricks, Nq =
// 4..8: flux differencing (Kennedy-Gruber, entropy conservative, central) and the weak form.
//
// The volume term works on half lines.  In each direction the Nq^2 lines of an element are
// shared by 2 Nq^2 threads: a thread owns the H0 = ceil(Nq/2) nodes from one end of a line to
// its middle, counted from that end (the table of a Lobatto line is odd under reflection, so
// both halves use the same entries at fixed indices: kernel parameters, no loads).  It holds
// its nodes' values and sums in registers, takes the pairs among them once for both nodes
// (the table Q[a][i] = D[a,i] w_a - D[i,a] w_i is skew: S[a][i] = Q[a][i] / w_i of
// esvolumeterm_dir!, src/balancelaws/dgsem.jl:576-600, times drdx), and meets the other
// half's nodes one by one.  The thread's first node is the line's face node, so it adds the
// face flux of that node itself (surfaceterm!, dgsem.jl:733-784) from the neighbour's trace,
// which it loads into registers before its pairs: there is no face buffer and no face phase.
// Sums pass from one direction's threads to the next's through shared memory.
//
// The kernels before it gave each node its full lines of partners: 3.4 K shared-memory load
// wavefronts an element (Nq = 8; FP32 2.8 K) and 11.9 K warp instructions (13.5 K); here 2.3 K (1.4 K)
// and 9.7 K (9.3 K).
//
// What bounds it (Nq = 8): an element takes an SM 3.3 us in FP64 and 2.15 us in FP32 bulk (6.4 K and
// 4.2 K cycles), from 16^3 elements to 32^3.  No unit is full (FP64: the FP64 pipe 47 %, issue 39 %, the
// L1 data pipe 54 %; FP32: issue 59 %): with 8 or 12 warps an SM the latencies of shared memory, the
// FP64 pipe and the two barriers are not covered.  The FP64 pipe alone would
// take 2.9 K cycles, HBM 3.5 K (152 B/node).
// Measured on B200, one LSRK(5,4) step, the kernels before -> this one: Kennedy-Gruber Nq = 8, 32^3,
// over three states in turn FP64 4667 -> 4060 us, FP32 bulk 3562 -> 2740 (on one state again and again
// 3.52-3.70 ms and 2.35-2.41); Nq = 6, 24^3 864 -> 712 and 690 -> 538; Nq = 4, 30^3 449 -> 368 and 411 ->
// 274; entropy conservative Nq = 5, 18^3 FP64 914 -> 379 and weak form Nq = 7, 15^3 FP64 1135 -> 330
// (both from the generic kernel).
// Tried and slower, in us a step at Nq = 8, 32^3 FP64 on one state, against 3712 then: one state
// buffer with the old state read again at the end (3 CTAs an SM at 168 registers, spills: 4107-4800);
// the traces one element ahead (3800); the register added at the end from a buffer of its own
// (4317).  A fifth warp that only fetches would leave 168 registers at 2 CTAs: not tried.
//
// Nq = 8: z, then y, then x lines.  A warp owns two z planes in the y and x phases and when it
// builds the partner values, so those hand-overs need no CTA barrier; two barriers an element.
// The x half lines are four consecutive nodes: the last phase writes the state and the
// register 32 bytes a lane.  Other Nq: x, y, then z lines, coalesced along x.
//
// The element's state arrives by one bulk copy (even Nq) issued one element ahead, its
// register by another into the buffer of the sums, which then start from it; odd Nq, whose
// elements are not whole 16-byte units, fetch the state by cp.async, each thread the values it
// reads first, and read the register at the end.  Every mbarrier wait is bounded: on expiry
// the CTA records RB200 status TIMEOUT and returns.
#pragma once

#include <type_traits>

#include "pipelined_kernel.cuh"

namespace rb200 {

namespace line {

template <int Q>
struct Shape {
    static_assert(Q >= 4 && Q <= 8, "Nq = 4..8");
    static constexpr int NP = Q * Q * Q, NFP = Q * Q, H0 = (Q + 1) / 2;
    static constexpr int NT = 2 * Q * Q;             // threads with work
    static constexpr int TH = (NT + 31) / 32 * 32;   // threads of a CTA
    static constexpr bool BULK = Q % 2 == 0;
    // Slots of the partner values (in 16-byte units; FP32 has a second array of 8-byte units), laid
    // out so that a quarter-warp's 16-byte, or a half-warp's 8-byte, accesses of every
    // direction fall into distinct banks at Nq = 8: the upper half of an x line is stored in
    // the order of its thread (from the far end), x lines are padded by one slot, and the
    // 8-byte array keeps the lower and upper halves in two blocks half a bank row apart, each
    // group of four in one of four orders.  Without it 0.8 K of the 3.3 K
    // shared-memory wavefronts of an element are conflicts.
    // Nq = 4: padded every 16 nodes; the others need nothing.
    static constexpr int PAD16 = Q == 8 ? NP / 8 : Q == 4 ? NP / 16 : 0, PAD8 = Q == 8 ? 8 : PAD16;
    __host__ __device__ static constexpr int slot16(int n) {
        if (Q == 8) return 9 * (n >> 3) + ((n & 7) < 4 ? (n & 7) : 11 - (n & 7));
        return Q == 4 ? n + (n >> 4) : n;
    }
    __host__ __device__ static constexpr int slot8(int n) {
        if (Q == 8) return 4 * (n >> 3) + (((n & 7) < 4 ? (n & 7) : (7 - (n & 7)) ^ 2) ^ ((n >> 5) & 1)) + ((n & 7) < 4 ? 0 : 264);
        return slot16(n);
    }
    // Slots of the sums (Nq = 8): FP64 exchanges pairs of nodes on every other two x lines, so
    // that the x threads' 16-byte loads at a 32-byte stride fall into distinct banks; FP32
    // exchanges pairs of x lines in every other z plane, for the y threads of a warp's two
    // planes.  Both only move a node within the nodes of one z-phase warp (see there).
    template <typename T>
    __device__ static __forceinline__ int sum_slot(int n) {
        if constexpr (Q != 8) return n;
        else if constexpr (sizeof(T) == 8) return n ^ (((n >> 4) & 1) << 1);
        else return n ^ (((n >> 6) & 1) << 4);
    }
};

template <typename T, int Q>
struct Smem {
    using S = Shape<Q>;
    __align__(16) double q[2][pipe::NS][S::NP];  // state of the current / next element
    pipe::Partners<T, S::NP + S::PAD16, S::NP + S::PAD8> aux;  // per-node partner values
    __align__(16) T acc[pipe::NS][S::NP];        // the register (even Nq), then the sums of the directions done
    double geo[2][4];                            // elem_geo of the current / next element
    int32_t nb[2][8];                            // neighbours of the current / next element
    ElemRef ref[2];                              // the current / next element
    uint64_t bar[2];                             // the state's copies
    uint64_t bar_dq;                             // the register's copy
};

// CTAs per SM the registers are sized for, FP64 and FP32.  A thread holds its half line, its sums
// and three traces: 254 registers in FP64 at Nq = 8, 168 in FP32; one CTA more an SM spills and
// is slower (Nq = 8 FP64 3 CTAs 1108 against 955 us at 20^3, FP32 4 CTAs 693 against 622; Nq = 6,
// 24^3: 5 and 7 CTAs 752 and 603 against 712 and 538).
#ifndef RB200_LINE_MIN8
#define RB200_LINE_MIN8 2, 3
#endif
#ifndef RB200_LINE_MIN7
#define RB200_LINE_MIN7 3, 4
#endif
#ifndef RB200_LINE_MIN6
#define RB200_LINE_MIN6 4, 6
#endif
#ifndef RB200_LINE_MIN5
#define RB200_LINE_MIN5 6, 8
#endif
#ifndef RB200_LINE_MIN4
#define RB200_LINE_MIN4 12, 16
#endif
template <typename T, int Q>
constexpr int min_ctas() {
    constexpr int m[5][2] = {{RB200_LINE_MIN4}, {RB200_LINE_MIN5}, {RB200_LINE_MIN6}, {RB200_LINE_MIN7}, {RB200_LINE_MIN8}};
    return m[Q - 4][sizeof(T) == 4];
}

// 4 consecutive values, 32 bytes at once where the address allows it (`wide`).  The load is not
// volatile, so that the compiler may place it where registers allow: where it must stay behind
// a wait of the kernel, `p` comes from after().
__device__ __forceinline__ size_t after(size_t x) {
    asm volatile("mov.u64 %0, %0;" : "+l"(x)::"memory");
    return x;
}
__device__ __forceinline__ void load4(const double* p, bool wide, double (&v)[4]) {
    if (wide) {
        asm("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(v[0]), "=d"(v[1]), "=d"(v[2]), "=d"(v[3]) : "l"(p));
    } else {
        const double2 a = *reinterpret_cast<const double2*>(p), b = *reinterpret_cast<const double2*>(p + 2);
        v[0] = a.x, v[1] = a.y, v[2] = b.x, v[3] = b.y;
    }
}
__device__ __forceinline__ void store4(double* p, bool wide, const double (&v)[4]) {
    if (wide) {
        asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(v[0]), "d"(v[1]), "d"(v[2]), "d"(v[3]) : "memory");
    } else {
        *reinterpret_cast<double2*>(p) = make_double2(v[0], v[1]);
        *reinterpret_cast<double2*>(p + 2) = make_double2(v[2], v[3]);
    }
}

__device__ __forceinline__ int thread_index() {
    int t;
    asm volatile("mov.u32 %0, %%tid.x;" : "=r"(t));
    return t;
}

// gamma, gamma - 1 and 1 / (2 (gamma - 1)) (kernel parameters: no registers)
template <typename T>
__device__ __forceinline__ T gas(const PipeArgs& A, int i) {
    if constexpr (sizeof(T) == 8) return A.gas[i];
    else return A.gasf[i];
}

// The half line of thread t in direction DIR: the line's first node, its index on a face and
// which half.
template <int Q, int DIR>
struct HalfLine {
    int half, base, jf;
    __device__ __forceinline__ explicit HalfLine(int t) {
        if constexpr (DIR == 0) {
            half = t & 1;
            jf = t >> 1;
            base = Q * jf;
        } else if constexpr (DIR == 1) {
            const int i = t % Q, k = t / (2 * Q);
            half = (t / Q) & 1;
            jf = i + Q * k;
            base = i + Q * Q * k;
        } else {
            half = t >= Q * Q;
            jf = t - half * Q * Q;
            base = jf;
        }
    }
};

// Entry of the kernel's tables in type T (a kernel parameter at a fixed index)
template <typename T>
__device__ __forceinline__ T tab(const PipeArgs& A, int i) {
    if constexpr (sizeof(T) == 8) return A.S[i];
    else return A.Sf[i];
}

}  // namespace line

// COMBO: EUL_KG, EUL_EC, or EUL_WEAK for both forms that are linear in the physical flux (the
// weak form and central flux differencing, whose tables differ).  STG: the stage modes; else
// the tendency modes (FP64 only).  A kernel with both would spill some 200 bytes a thread.
template <int COMBO, typename T, bool BATCH, int Q, bool STG>
__global__ void __launch_bounds__(line::Shape<Q>::TH, (line::min_ctas<T, Q>()))
    pipelined_stage_kernel(const __grid_constant__ PipeArgs A, const __grid_constant__ PipeBatch B) {
    using namespace pipe;
    using LS = line::Shape<Q>;
    constexpr int NP = LS::NP, NFP = LS::NFP, H0 = LS::H0, NT = LS::NT, TH = LS::TH;
    constexpr bool WP = Q == 8;  // a warp owns two z planes in the x and y phases
    constexpr int NH = (NP + NT - 1) / NT;
    extern __shared__ __align__(128) unsigned char pipe_smem_raw[];
    line::Smem<T, Q>& sm = *reinterpret_cast<line::Smem<T, Q>*>(pipe_smem_raw);
    const int t = threadIdx.x;
    // the threads that issue the copies of the state and of the register
    constexpr int kStateThread = 32 * (TH > 32), kRegisterThread = 32 * (TH / 32 - 1);
    const bool work = TH == NT || t < NT;
    static_assert(STG || (sizeof(T) == 8 && !BATCH), "tendencies: one state, FP64");
    // whether the register is read: not by a stage with rka = 0, nor by a tendency that sets it
    const bool reads_dq = A.mode == MODE_STAGE || A.mode == MODE_TENDENCY_INC;
    // the nodes whose partner values this thread builds (Nq = 8: of its warp's planes)
    auto p0_node = [&](int h) { return WP ? (t & 31) + 32 * h + 128 * (t >> 5) : t + NT * h; };
    auto sync_plane = [&]() {
        if constexpr (WP) __syncwarp();
        else __syncthreads();
    };
    // a CTA barrier; records that a wait ran out
    auto give_up = [&](bool late) {
        if (!__syncthreads_or(late)) return false;
        if (t == 0) atomicExch(A.status, kStatusTimeout);
        return true;
    };
    auto pressure = [&](const T rinv, const T m0, const T m1, const T m2, const T E) {
        return line::gas<T>(A, 1) * (E - (m0 * m0 + m1 * m1 + m2 * m2) * (T(0.5) * rinv));
    };
    // the state of element r: a bulk copy by thread 0, or each thread its own values
    auto fetch_state = [&](const double* q, int64_t e, int b) {
        const double* src = q + (size_t)e * NS * NP;
        if constexpr (LS::BULK) {
            if (t == kStateThread) {
                mbar_expect_tx(&sm.bar[b], NS * NP * sizeof(double));
                bulk_g2s(&sm.q[b][0][0], src, NS * NP * sizeof(double), &sm.bar[b]);
            }
        } else if (work) {
#pragma unroll
            for (int h = 0; h < NH; ++h) {
                const int n = p0_node(h);
                if (NP % NT == 0 || n < NP) {
#pragma unroll
                    for (int s = 0; s < NS; ++s) cp_async8(&sm.q[b][s][n], src + s * NP + n);
                }
            }
        }
    };

    Cursor<BATCH> cur;  // meaningful in threads 0..9 and kStateThread
    if (LS::BULK && t == 0) {
        mbar_init(&sm.bar[0], 1);
        mbar_init(&sm.bar[1], 1);
        mbar_init(&sm.bar_dq, 1);
        fence_mbar_init();
    }
    if (t < 10 || t == kStateThread) {
        ElemRef r{};
        r.e = -1;
        if (cur.start(A, B)) cur.resolve(A, B, r);
        if (t == kStateThread) sm.ref[0] = r;
        if (t < 10 && r.e >= 0) fetch_part(r, t, sm.geo[0], sm.nb[0]);  // geometry: written by no kernel
    }
    // the previous kernel of the stream (the last stage, or this stage's mortar fluxes)
    // has completed before any state, register or mortar flux is read or written
    grid_dependency_wait();
    cp_async_commit();
    cp_async_wait_all();
    __syncthreads();
    if (sm.ref[0].e >= 0) fetch_state(sm.ref[0].q, sm.ref[0].e, 0);
    // The neighbours' traces at the thread's face nodes (or their mortar fluxes), all three
    // directions' loaded into registers before the first pairs, so that the later ones need not
    // wait for their own
    double tr[3][NS];
    bool mortar[3];
    auto trace = [&](auto dirc, const double* q, int64_t e, int b) {
        constexpr int DIR = decltype(dirc)::value;
        constexpr int STR = DIR == 0 ? 1 : DIR == 1 ? Q : Q * Q;
        const line::HalfLine<Q, DIR> L(line::thread_index());
        const int f = 2 * DIR + L.half, nbf = sm.nb[b][f];
        // q+ on a boundary face is q- (balancelaw.jl:77)
        const int own_end = L.base + (L.half ? (Q - 1) * STR : 0), far_end = L.base + (L.half ? 0 : (Q - 1) * STR);
        const double* qn = q + (nbf >= 0 ? (size_t)nbf * NS * NP + far_end : (size_t)e * NS * NP + own_end);
        int sn = NP;
        mortar[DIR] = nbf == -2;
        if (mortar[DIR]) {
            qn = A.ncflux + (((size_t)e * 6 + f) * NS) * NFP + L.jf;
            sn = NFP;
        }
#pragma unroll
        for (int s = 0; s < NS; ++s) tr[DIR][s] = qn[s * sn];
    };
    using I0 = std::integral_constant<int, 0>;
    using I1 = std::integral_constant<int, 1>;
    using I2 = std::integral_constant<int, 2>;
    uint32_t phase_q = 0, phase_dq = 0;
    int es = (int)A.e_begin + blockIdx.x;  // one state: the current element, kept in a register
    for (int buf = 0;; buf ^= 1, es += gridDim.x) {
        const int e = BATCH ? (int)sm.ref[buf].e : (es < (int)A.E ? es : -1);
        if (e < 0) break;
        // ---- this element's state
        bool late = false;
        if constexpr (LS::BULK) {
            late = !bounded_wait(&sm.bar[buf], phase_q);
            phase_q ^= buf;
        }
        cp_async_commit();
        cp_async_wait_all();  // own copies: the geometry and neighbours (threads 0..9), odd Nq the state
        sync_plane();         // the last phase of the previous element has read its partner values
        if (work && !late) {
#pragma unroll
            for (int h = 0; h < NH; ++h) {
                const int n = p0_node(h);
                if (NP % NT != 0 && n >= NP) continue;
                const T rho = (T)sm.q[buf][0][n];
                const T rinv = rcp_inner(rho);
                const T m0 = (T)sm.q[buf][1][n], m1 = (T)sm.q[buf][2][n], m2 = (T)sm.q[buf][3][n];
                const T u0 = m0 * rinv, u1 = m1 * rinv, u2 = m2 * rinv;
                const T rhoe = (T)sm.q[buf][4][n];
                const T p = pressure(rinv, m0, m1, m2, rhoe);
                T o[NAUX];
                if constexpr (COMBO == EUL_KG) {  // halves of rho, u, e, p
                    o[0] = rho * T(0.5);
                    o[1] = u0 * T(0.5);
                    o[2] = u1 * T(0.5);
                    o[3] = u2 * T(0.5);
                    o[4] = rhoe * rinv * T(0.5);
                    o[5] = p * T(0.5);
                } else if constexpr (COMBO == EUL_EC) {  // rho, u, b = rho/(2p), |u|^2
                    o[0] = rho;
                    o[1] = u0;
                    o[2] = u1;
                    o[3] = u2;
                    o[4] = T(0.5) * rho * rcp(p);
                    o[5] = u0 * u0 + u1 * u1 + u2 * u2;
                } else {  // rho, u, E, p
                    o[0] = rho;
                    o[1] = u0;
                    o[2] = u1;
                    o[3] = u2;
                    o[4] = rhoe;
                    o[5] = p;
                }
                sm.aux.put(LS::slot16(n), LS::slot8(n), o);
            }
        }
        if (give_up(late)) return;  // #1: partner values ready; the previous element's buffers are free
        // the next element's geometry, neighbours and state (bulk copy), and this element's register,
        // each by a warp of its own (as far as there are): one warp's issue of all three would
        // hold up the others at #2
        if (t < 10 || t == kStateThread) {
            ElemRef rn{};
            rn.e = -1;
            if (cur.advance(A, B)) cur.resolve(A, B, rn);
            if (t == kStateThread) {
                sm.ref[buf ^ 1] = rn;
                if (LS::BULK && rn.e >= 0) {
                    fence_proxy_async();
                    fetch_state(rn.q, rn.e, buf ^ 1);
                }
            }
            if (t < 10 && rn.e >= 0) fetch_part(rn, t, sm.geo[buf ^ 1], sm.nb[buf ^ 1]);
        }
        if (LS::BULK && reads_dq && t == kRegisterThread) {  // into the buffer of the sums
            const void* dq = BATCH ? sm.ref[buf].dq : A.dq;
            fence_proxy_async();
            mbar_expect_tx(&sm.bar_dq, NS * NP * sizeof(T));
            bulk_g2s(&sm.acc[0][0], static_cast<const T*>(dq) + (size_t)e * NS * NP, NS * NP * sizeof(T), &sm.bar_dq);
        }
        if constexpr (!LS::BULK) {
            static_assert(!BATCH || LS::BULK, "serving classes: even Nq");
            if (es + (int)gridDim.x < (int)A.E) fetch_state(A.q_in, es + gridDim.x, buf ^ 1);
        }
        // the element's state buffers (one state: the kernel parameters)
        const double* const qin_e = BATCH ? sm.ref[buf].q : A.q_in;
        void* const dq_e = BATCH ? sm.ref[buf].dq : A.dq;
        double* const qout_e = BATCH ? sm.ref[buf].q_out : A.q_out;
        const double rkb_dt = BATCH ? sm.ref[buf].rkb_dt : A.rkb_dt;
        const size_t g0 = (size_t)e * NS * NP;

        auto add_register = [&](const T v, const T old) {  // rka dq + sums (stages) or dq + sums
            if constexpr (STG) return fma((T)A.rka, old, v);
            else return old + v;
        };
        // One direction: DIR, and POS 0 (writes its sums), 1 (adds to them), 2 (adds and
        // finishes the element).
        auto direction = [&](auto dirc, auto posc) {
            constexpr int DIR = decltype(dirc)::value, POS = decltype(posc)::value;
            constexpr int STR = DIR == 0 ? 1 : DIR == 1 ? Q : Q * Q;
            const line::HalfLine<Q, DIR> L(line::thread_index());
            const int half = L.half, base = L.base;
            const int end = base + (half ? (Q - 1) * STR : 0), step = half ? -STR : STR;
            // the partner values of the line's node a, counted from the thread's end: slots
            // linear in a within each half of the line
            constexpr int S16 = Q == 8 && DIR == 0 ? 1 : LS::slot16(STR), S8 = Q == 8 && DIR > 0 ? STR / 2 : LS::slot8(STR);
            const int mid = end + (half ? -H0 : H0) * STR;
            const int own16 = LS::slot16(end), own8 = LS::slot8(end), far16 = LS::slot16(mid), far8 = LS::slot8(mid);
            auto values = [&](const int a, T (&v)[NAUX]) {
                const int d = a < H0 ? a : a - H0;
                if constexpr (Q == 8 && DIR == 0)
                    sm.aux.get(a < H0 ? own16 + d : far16 - d, a < H0 ? own8 ^ d : far8 ^ d, v);
                else
                    sm.aux.get((a < H0 ? own16 : far16) + (half ? -S16 : S16) * d,
                               (a < H0 ? own8 : far8) + (half ? -S8 : S8) * d, v);
            };
            T scale[H0];  // metric and mass, formed in FP64 and rounded once
#pragma unroll
            for (int m = 0; m < H0; ++m) scale[m] = (T)(sm.geo[buf][DIR] * A.winv[m]);
            // ---- volume term
            T acc[H0][NS], o[H0][NAUX];
#pragma unroll
            for (int m = 0; m < H0; ++m)
#pragma unroll
                for (int s = 0; s < NS; ++s) acc[m][s] = T(0);
            if constexpr (COMBO == EUL_WEAK) {
                // acc_m = sum_a Q[a][m] F_a, F the physical flux along the line (euler.jl:50-61)
#pragma unroll
                for (int a = 0; a < Q; ++a) {
                    T p[NAUX];
                    values(a, p);
                    if (a == 0) {
#pragma unroll
                        for (int c = 0; c < NAUX; ++c) o[0][c] = p[c];
                    }
                    const T ud = p[1 + DIR], mn = p[0] * ud;
                    T F[NS] = {mn, mn * p[1], mn * p[2], mn * p[3], ud * (p[4] + p[5])};
                    F[1 + DIR] += p[5];
#pragma unroll
                    for (int m = 0; m < H0; ++m)
#pragma unroll
                        for (int s = 0; s < NS; ++s) acc[m][s] = fma(F[s], line::tab<T>(A, a * Q + m), acc[m][s]);
                }
            } else if constexpr (COMBO == EUL_KG) {
                // the own-node parts of the momentum and energy averages are factored out of the
                // sums: sum F (o_k + p_k) = o_k sum F + sum F p_k, F = rho_avg u_avg Q
#pragma unroll
                for (int m = 0; m < H0; ++m) values(m, o[m]);
#pragma unroll
                for (int m = 0; m < H0; ++m)
#pragma unroll
                    for (int n = m + 1; n < H0; ++n) {  // pairs of own nodes, once for both
                        const T q = line::tab<T>(A, n * Q + m);
                        const T un = (o[m][1 + DIR] + o[n][1 + DIR]) * q;
                        const T f1 = (o[m][0] + o[n][0]) * un, pb = o[m][5] + o[n][5];
                        acc[m][0] += f1;
                        acc[n][0] -= f1;
#pragma unroll
                        for (int c = 1; c < NS; ++c) {
                            acc[m][c] = fma(f1, o[n][c], acc[m][c]);
                            acc[n][c] = fma(-f1, o[m][c], acc[n][c]);
                        }
                        acc[m][1 + DIR] = fma(pb, q, acc[m][1 + DIR]);
                        acc[n][1 + DIR] = fma(-pb, q, acc[n][1 + DIR]);
                        acc[m][4] = fma(un, pb, acc[m][4]);
                        acc[n][4] = fma(-un, pb, acc[n][4]);
                    }
#pragma unroll
                for (int a = H0; a < Q; ++a) {  // the other half's nodes
                    T p[NAUX];
                    values(a, p);
#pragma unroll
                    for (int m = 0; m < H0; ++m) {
                        const T q = line::tab<T>(A, a * Q + m);
                        const T un = (o[m][1 + DIR] + p[1 + DIR]) * q;
                        const T f1 = (o[m][0] + p[0]) * un, pb = o[m][5] + p[5];
                        acc[m][0] += f1;
#pragma unroll
                        for (int c = 1; c < NS; ++c) acc[m][c] = fma(f1, p[c], acc[m][c]);
                        acc[m][1 + DIR] = fma(pb, q, acc[m][1 + DIR]);
                        acc[m][4] = fma(un, pb, acc[m][4]);
                    }
                }
#pragma unroll
                for (int m = 0; m < H0; ++m)
#pragma unroll
                    for (int c = 1; c < NS; ++c) acc[m][c] = fma(o[m][c], acc[m][0], acc[m][c]);
            } else {  // EUL_EC
                // the two-point flux of nodes x and y along the line, times q; `far`: the pair is
                // beyond the power series of the logarithmic means
                bool far = false;
                auto two_point = [&](const T (&x)[NAUX], const T (&y)[NAUX], const T q, T (&F)[NS], auto exact) {
                    const T ua0 = (x[1] + y[1]) * T(0.5), ua1 = (x[2] + y[2]) * T(0.5), ua2 = (x[3] + y[3]) * T(0.5);
                    const T rs = x[0] + y[0], bs = x[4] + y[4];
                    constexpr bool kExact = decltype(exact)::value;
                    const T ir = newton_rcp<kExact>(rs), ib = newton_rcp<kExact>(bs);
                    T rlog, iblog;
                    if constexpr (kExact) {
                        rlog = log_mean(x[0], y[0], ir);
                        iblog = inverse_log_mean(x[4], y[4], ib);
                    } else {
                        const T fr = (x[0] - y[0]) * ir, fb = (x[4] - y[4]) * ib, ur = fr * fr, ub = fb * fb;
                        rlog = (T(0.5) * rs) * log_mean_inverse_series(ur);
                        iblog = (T(2) * ib) * log_mean_series(ub);
                        far |= !(ur < T(0.01)) | !(ub < T(0.01));
                    }
                    const T pt = (T(0.5) * rs) * ib;  // rho_avg / (2 b_avg)
                    const T un = (DIR == 0 ? ua0 : DIR == 1 ? ua1 : ua2) * q;
                    const T h = line::gas<T>(A, 2) * iblog - T(0.25) * (x[5] + y[5]) + (ua0 * ua0 + ua1 * ua1 + ua2 * ua2);
                    F[0] = rlog * un;
                    F[1] = F[0] * ua0;
                    F[2] = F[0] * ua1;
                    F[3] = F[0] * ua2;
                    F[1 + DIR] = fma(pt, q, F[1 + DIR]);
                    F[4] = un * fma(h, rlog, pt);
                };
#pragma unroll
                for (int m = 0; m < H0; ++m) values(m, o[m]);
#pragma unroll
                for (int m = 0; m < H0; ++m)
#pragma unroll
                    for (int n = m + 1; n < H0; ++n) {
                        T F[NS];
                        two_point(o[m], o[n], line::tab<T>(A, n * Q + m), F, std::false_type{});
#pragma unroll
                        for (int s = 0; s < NS; ++s) {
                            acc[m][s] += F[s];
                            acc[n][s] -= F[s];
                        }
                    }
#pragma unroll
                for (int a = H0; a < Q; ++a) {
                    T p[NAUX];
                    values(a, p);
#pragma unroll
                    for (int m = 0; m < H0; ++m) {
                        T F[NS];
                        two_point(o[m], p, line::tab<T>(A, a * Q + m), F, std::false_type{});
#pragma unroll
                        for (int s = 0; s < NS; ++s) acc[m][s] += F[s];
                    }
                }
                if (far) {  // a strong jump on this line: its sums again, with the logarithms
#pragma unroll
                    for (int m = 0; m < H0; ++m) {
#pragma unroll
                        for (int s = 0; s < NS; ++s) acc[m][s] = T(0);
#pragma unroll 1
                        for (int a = 0; a < Q; ++a) {
                            if (a == m) continue;
                            T p[NAUX], F[NS];
                            values(a, p);
                            two_point(o[m], p, line::tab<T>(A, a * Q + m), F, std::true_type{});
#pragma unroll
                            for (int s = 0; s < NS; ++s) acc[m][s] += F[s];
                        }
                    }
                }
            }
            // reflection, metric and mass: the half counted from the far end has the sign turned
#pragma unroll
            for (int m = 0; m < H0; ++m) {
                const T scm = half ? -scale[m] : scale[m];
#pragma unroll
                for (int s = 0; s < NS; ++s) acc[m][s] *= scm;
            }
            // ---- face term at the thread's first node: (wsJ nf) MJI with wsJ MJI = |drdx| / w_0
            {
                const T fsc = fabs(scale[0]);
                const T sn = half ? T(1) : T(-1);
                // q- is the state itself, and its velocity and pressure are what the element across
                // the face takes from it: both compute the same flux, and equal states (q+ is q- on
                // a boundary face) have no jump
                T qm[NS], um[3], pm;
#pragma unroll
                for (int s = 1; s < NS; ++s)
                    qm[s] = s == 4 && COMBO == EUL_WEAK ? o[0][4] : (T)sm.q[buf][s][end];
                const T rm = qm[0] = COMBO == EUL_KG ? T(2) * o[0][0] : o[0][0], rmi = rcp_inner(rm);
#pragma unroll
                for (int d = 0; d < 3; ++d) um[d] = COMBO == EUL_KG ? T(2) * o[0][1 + d] : o[0][1 + d];
                if constexpr (COMBO == EUL_KG) pm = T(2) * o[0][5];
                else if constexpr (COMBO == EUL_WEAK) pm = o[0][5];
                else pm = pressure(rmi, qm[1], qm[2], qm[3], qm[4]);
                const T rp = (T)tr[DIR][0], Ep = (T)tr[DIR][4], rinv = rcp_inner(rp);
                T mp[3], up[3];
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    mp[d] = (T)tr[DIR][1 + d];
                    up[d] = mp[d] * rinv;
                }
                const T pp = pressure(rinv, mp[0], mp[1], mp[2], Ep);
                const T unm = um[DIR] * sn, unp = up[DIR] * sn, mnm = qm[1 + DIR] * sn, mnp = mp[DIR] * sn;
                // the larger wave speed |u.n| + sqrt(gamma p / rho) (euler.jl:62-68)
                const T wm = fabs(unm) + root(line::gas<T>(A, 0) * pm * rmi), wp = fabs(unp) + root(line::gas<T>(A, 0) * pp * rinv);
                const T mx = A.surface_rusanov ? fmax(wm, wp) : T(0);
                // normal fluxes of both sides (euler.jl:50-60 with n = sn e_dir), field by field
#pragma unroll
                for (int s = 0; s < NS; ++s) {
                    T fm, fp, dq;
                    if (s == 0) {
                        fm = mnm;
                        fp = mnp;
                        dq = rp - rm;
                    } else if (s == 4) {
                        fm = unm * (qm[4] + pm);
                        fp = unp * (Ep + pp);
                        dq = Ep - qm[4];
                    } else {
                        fm = mnm * um[s - 1] + (DIR == s - 1 ? pm * sn : T(0));
                        fp = mnp * up[s - 1] + (DIR == s - 1 ? pp * sn : T(0));
                        dq = mp[s - 1] - qm[s];
                    }
                    const T nf = (fm + fp) * T(0.5) - (mx * dq) * T(0.5);
                    acc[0][s] -= (mortar[DIR] ? (T)tr[DIR][s] : nf) * fsc;
                }
            }
            // ---- hand the sums over, or finish
            auto owned = [&](int m) { return Q % 2 == 0 || m < H0 - 1 || half == 0; };  // odd Nq: the middle once
            if constexpr (POS == 0 && LS::BULK) {
                if (reads_dq) {  // with the register, which has arrived in their place
                    late = !bounded_wait(&sm.bar_dq, phase_dq);
                    phase_dq ^= 1;
                }
            }
            if constexpr (POS == 0) {
                // the register lies in node order, the sums in slot order: the nodes m of a warp
                // fill the same set of slots, so it reads them all before it writes any
                const bool add = LS::BULK && reads_dq;
#pragma unroll
                for (int m = 0; m < H0; ++m) {
                    const int n = end + step * m;
                    if (add) {
#pragma unroll
                        for (int s = 0; s < NS; ++s) acc[m][s] = add_register(acc[m][s], sm.acc[s][n]);
                    }
                    if constexpr (WP) __syncwarp();
                    if (!owned(m)) continue;
#pragma unroll
                    for (int s = 0; s < NS; ++s) sm.acc[s][LS::template sum_slot<T>(n)] = acc[m][s];
                }
            } else if constexpr (POS == 1) {
#pragma unroll
                for (int m = 0; m < H0; ++m) {
                    if (!owned(m)) continue;
                    const int n = LS::template sum_slot<T>(end + step * m);
#pragma unroll
                    for (int s = 0; s < NS; ++s) sm.acc[s][n] += acc[m][s];
                }
            } else if constexpr (Q == 8) {
                const int n0 = base + 4 * half;
                const size_t g = g0 + n0;
                const bool wide = (((uintptr_t)dq_e | (STG ? (uintptr_t)qout_e : 0)) & 31) == 0;
#pragma unroll
                for (int s = 0; s < NS; ++s) {
                    T v[4];
                    if constexpr (sizeof(T) == 8) {
                        const double2 a = *reinterpret_cast<const double2*>(&sm.acc[s][LS::template sum_slot<T>(n0)]);
                        const double2 b = *reinterpret_cast<const double2*>(&sm.acc[s][LS::template sum_slot<T>(n0 + 2)]);
                        v[0] = a.x, v[1] = a.y, v[2] = b.x, v[3] = b.y;
                    } else {
                        const float4 a = *reinterpret_cast<const float4*>(&sm.acc[s][LS::template sum_slot<T>(n0)]);
                        v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w;
                    }
#pragma unroll
                    for (int m = 0; m < 4; ++m) v[m] += half ? acc[3 - m][s] : acc[m][s];
                    if constexpr (sizeof(T) == 4)
                        *reinterpret_cast<float4*>(static_cast<float*>(dq_e) + g + s * NP) = make_float4(v[0], v[1], v[2], v[3]);
                    else
                        line::store4(static_cast<double*>(dq_e) + g + s * NP, wide, v);
                    if constexpr (STG) {
                        // every other four threads read their second pair first: distinct banks
                        const int first = (t >> 1) & 2;
                        const double2 x = *reinterpret_cast<const double2*>(&sm.q[buf][s][n0 + first]);
                        const double2 y = *reinterpret_cast<const double2*>(&sm.q[buf][s][n0 + 2 - first]);
                        const double2 a = first ? y : x, b = first ? x : y;
                        const double out[4] = {a.x + rkb_dt * (double)v[0], a.y + rkb_dt * (double)v[1],
                                               b.x + rkb_dt * (double)v[2], b.y + rkb_dt * (double)v[3]};
                        line::store4(qout_e + g + s * NP, wide, out);
                    }
                }
            } else {
                T old[H0][NS];
                if constexpr (!LS::BULK) {
#pragma unroll
                    for (int m = 0; m < H0; ++m)
#pragma unroll
                        for (int s = 0; s < NS; ++s)
                            old[m][s] = reads_dq ? static_cast<const T*>(dq_e)[g0 + s * NP + end + step * m] : T(0);
                }
#pragma unroll
                for (int m = 0; m < H0; ++m) {
                    if (!owned(m)) continue;
                    const int n = end + step * m;
#pragma unroll
                    for (int s = 0; s < NS; ++s) {
                        const size_t g = g0 + s * NP + n;
                        T v = sm.acc[s][n] + acc[m][s];
                        if constexpr (!LS::BULK) v = add_register(v, old[m][s]);
                        static_cast<T*>(dq_e)[g] = v;
                        if constexpr (STG) qout_e[g] = sm.q[buf][s][n] + rkb_dt * (double)v;
                    }
                }
            }
        };
        auto drain = [&]() {  // the next element's copy, before leaving early
            if (LS::BULK && sm.ref[buf ^ 1].e >= 0) bounded_wait(&sm.bar[buf ^ 1], phase_q);
        };
        if (work) {
            trace(I0{}, qin_e, e, buf);
            trace(I1{}, qin_e, e, buf);
            trace(I2{}, qin_e, e, buf);
        }
        if constexpr (WP) {
            direction(I2{}, I0{});
            if (give_up(late)) return drain();  // #2: the z sums of the warp's planes
            direction(I1{}, I1{});
            __syncwarp();
            direction(I0{}, I2{});
        } else {
            if (work) direction(I0{}, I0{});
            if (give_up(late)) return drain();
            if (work) direction(I1{}, I1{});
            __syncthreads();
            if (work) direction(I2{}, I2{});
        }
    }
}

}  // namespace rb200
