// Persistent LSRK stage kernel of the Euler law on curved 3-D grids with Nq = 8, Kennedy-Gruber
// flux differencing, FP64 or FP32 bulk (stage modes).
//
// The half-line design of line_kernel.cuh: 128 threads share an element, in each direction a
// thread owns the four nodes from one end of a line to its middle, takes the pairs among them
// once for both nodes, meets the other half's nodes one by one, and adds the face flux of its
// first node, which is the line's end.  z, then y, then x lines; sums pass between the
// directions through shared memory.  What a curved grid adds:
// * a pair's flux is contracted with G = D[a,i] l_g[a] - D[i,a] l_g[i] (esvolumeterm_dir!,
//   src/balancelaws/dgsem.jl:576-600; l_g = wJ dRdX[dir,:], the rows of vgeo), which is skew in
//   (a, i), and odd under reflection of the line like D;
// * each direction needs only its own three rows, so the rows arrive by one bulk copy a
//   direction (12 KB), into buffers that are free again when their direction is done: z's one
//   element ahead, y's and x's (with MJI) while z's pairs run.  They stay FP64 in shared memory,
//   FP32 bulk converts them as it reads;
// * the face normal and wsJ are loaded with the neighbour's trace, 32 bytes a thread.
//
// What bounds it: HBM (256 B/node in FP64, 220 in FP32 bulk: 6.0 and 5.1 K cycles an element and
// SM at the measured peak) and, in FP64, the FP64 pipe (4.5 K).  The kernels before this one (256
// threads, each node its full lines of partners with their metric rows) took 16.5 and 12.2 K, and
// this one 12.2 and 8.4 K: B200, one LSRK(5,4) step, FP64 13^3 635 -> 475 us, FP32 bulk 16^3 883 ->
// 606.  Two CTAs of 128 threads share an SM (255 registers a thread in FP64; shared memory 110
// and 85 KB a CTA): 8 warps do not cover the latencies between the two barriers.
//
// Every mbarrier wait is bounded: on expiry the CTA records RB200 status TIMEOUT and returns.
#pragma once

#include "line_kernel.cuh"

namespace rb200 {

struct PipeCurvedArgs {
    const double* q_in;
    double* q_out;
    void* dq;                // LSRK register, float* in FP32 bulk
    const double* vgeo;      // (512, 11, E): wJ dRdX[dir][d] (dir-major), MJI, MJ
    const double* sgeo;      // (4, 384, E): n, wsJ per face node
    const int32_t* nbr;      // (6, E)
    int32_t* status;
    int64_t E;               // elements e_begin..E-1 are computed
    int64_t e_begin;
    int32_t mode;            // MODE_STAGE or MODE_STAGE_FIRST
    int32_t surface_rusanov;
    double rka, rkb_dt;
    double gas[3];           // gamma, gamma - 1
    float gasf[3];
    double D[64];            // D[i + 8 j] = l_j'(r_i), odd under reflection of the line
    float Df[64];
};

namespace pipec {

constexpr int Q = 8, NP = 512, NFP = 64, NT = 128;
using LS = line::Shape<Q>;

template <typename T>
struct Smem {
    __align__(16) double q[pipe::NS][NP];   // state of the element, then (after #1) of the next one
    __align__(16) double geo[10][NP];       // rows l_g[dir][d] of the element, and MJI
    pipe::Partners<T, NP + LS::PAD16, NP + LS::PAD8> aux;
    __align__(16) T acc[pipe::NS][NP];      // sums of the directions done
    int32_t nb[2][8];                       // neighbours of the current / next element
    uint64_t bar_q, bar_geo[3];
};

// D[i, j] as a kernel parameter in type T
template <typename T>
__device__ __forceinline__ T dpar(const PipeCurvedArgs& A, int i, int j) {
    if constexpr (sizeof(T) == 8) return A.D[i + 8 * j];
    else return A.Df[i + 8 * j];
}
template <typename T>
__device__ __forceinline__ T gas(const PipeCurvedArgs& A, int i) {
    if constexpr (sizeof(T) == 8) return A.gas[i];
    else return A.gasf[i];
}

}  // namespace pipec

template <typename T>
__global__ void __launch_bounds__(pipec::NT, 2) pipelined_curved_kernel(const __grid_constant__ PipeCurvedArgs A) {
    using namespace pipe;
    using pipec::LS;
    constexpr int Q = pipec::Q, NP = pipec::NP, NFP = pipec::NFP, H0 = 4;
    extern __shared__ __align__(128) unsigned char pipe_smem_raw[];
    pipec::Smem<T>& sm = *reinterpret_cast<pipec::Smem<T>*>(pipe_smem_raw);
    const int t = threadIdx.x;
    const bool reads_dq = A.mode == MODE_STAGE;
    const int E = (int)A.E;
    // the rows of direction dir (x: with MJI) of element e into their place
    auto fetch_rows = [&](int dir, int64_t e) {
        const double* src = A.vgeo + (size_t)e * 11 * NP;
        constexpr uint32_t bytes = 3 * NP * sizeof(double);
        mbar_expect_tx(&sm.bar_geo[dir], bytes + (dir == 0 ? NP * sizeof(double) : 0));
        bulk_g2s(&sm.geo[3 * dir][0], src + 3 * dir * NP, bytes, &sm.bar_geo[dir]);
        if (dir == 0) bulk_g2s(&sm.geo[9][0], src + 9 * NP, NP * sizeof(double), &sm.bar_geo[0]);
    };
    auto fetch_state = [&](int64_t e) {
        mbar_expect_tx(&sm.bar_q, NS * NP * sizeof(double));
        bulk_g2s(&sm.q[0][0], A.q_in + (size_t)e * NS * NP, NS * NP * sizeof(double), &sm.bar_q);
    };

    int e = (int)A.e_begin + blockIdx.x;
    if (t == 0) {
        mbar_init(&sm.bar_q, 1);
#pragma unroll
        for (int d = 0; d < 3; ++d) mbar_init(&sm.bar_geo[d], 1);
        fence_mbar_init();
        if (e < E) fetch_rows(2, e);  // geometry: written by no kernel
    }
    if (t < 6 && e < E) cp_async4(&sm.nb[0][t], A.nbr + (size_t)6 * e + t);
    grid_dependency_wait();  // the previous kernel of the stream is complete
    if (t == 0 && e < E) fetch_state(e);
    cp_async_commit();
    cp_async_wait_all();
    __syncthreads();

    uint32_t ph = 0;     // parity of every copy: one of each an element
    bool late = false;   // a wait of this thread ran out
    for (int buf = 0; e < E; buf ^= 1, e += gridDim.x, ph ^= 1) {
        const int en = e + (int)gridDim.x;
        late |= !bounded_wait(&sm.bar_q, ph);
        cp_async_wait_all();
        __syncwarp();  // the x phase of the previous element has read its planes' partner values
        // ---- per-node partner values of the warp's two z planes: halves of rho, u, e, p
#pragma unroll
        for (int h = 0; h < 4; ++h) {
            const int n = (t & 31) + 32 * h + 128 * (t >> 5);
            const T rho = (T)sm.q[0][n], rinv = rcp_inner(rho);
            const T m0 = (T)sm.q[1][n], m1 = (T)sm.q[2][n], m2 = (T)sm.q[3][n], rhoe = (T)sm.q[4][n];
            const T u0 = m0 * rinv, u1 = m1 * rinv, u2 = m2 * rinv;
            const T p = pipec::gas<T>(A, 1) * (rhoe - (m0 * m0 + m1 * m1 + m2 * m2) * (T(0.5) * rinv));
            const T o[NAUX] = {rho * T(0.5), u0 * T(0.5), u1 * T(0.5), u2 * T(0.5), rhoe * rinv * T(0.5), p * T(0.5)};
            sm.aux.put(LS::slot16(n), LS::slot8(n), o);
        }
        if (__syncthreads_or(late)) {  // #1: partner values ready; the state's and the rows' buffers are free
            if (t == 0) {
                atomicExch(A.status, kStatusTimeout);
                bounded_wait(&sm.bar_geo[2], ph);
            }
            return;
        }
        if (t == 32) {
            fence_proxy_async();
            fetch_rows(1, e);
            fetch_rows(0, e);
        }
        if (t == 64 && en < E) {
            fence_proxy_async();
            fetch_state(en);
        }
        if (t == 96 && reads_dq)  // the register, read at the element's end, into the L2 cache
            asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(static_cast<const T*>(A.dq) + (size_t)e * NS * NP),
                         "n"(NS * NP * (int)sizeof(T))
                         : "memory");
        if (t < 6 && en < E) cp_async4(&sm.nb[buf ^ 1][t], A.nbr + (size_t)6 * en + t);
        cp_async_commit();
        const size_t g0 = (size_t)e * NS * NP;

        // One direction: DIR, and POS 0 (writes its sums), 1 (adds to them), 2 (finishes)
        auto direction = [&](auto dirc, auto posc) {
            constexpr int DIR = decltype(dirc)::value, POS = decltype(posc)::value;
            constexpr int STR = DIR == 0 ? 1 : DIR == 1 ? Q : Q * Q;
            const line::HalfLine<Q, DIR> L(line::thread_index());
            const int half = L.half, base = L.base;
            const int end = base + (half ? (Q - 1) * STR : 0), step = half ? -STR : STR;
            // ---- the neighbour's trace (q+ = q- on a boundary face, balancelaw.jl:77) and the face
            // geometry at the thread's face node, before the pairs
            const int f = 2 * DIR + half, nbf = sm.nb[buf][f];
            double tr[NS], sg[4];
            {
                const double* qn = A.q_in + (nbf >= 0 ? (size_t)nbf * NS * NP + base + (half ? 0 : (Q - 1) * STR) : g0 + end);
#pragma unroll
                for (int s = 0; s < NS; ++s) tr[s] = qn[s * NP];
                line::load4(A.sgeo + (((size_t)e * 6 + f) * NFP + L.jf) * 4, true, sg);
            }
            // ---- the line's rows, counted from the thread's end
            late |= !bounded_wait(&sm.bar_geo[DIR], ph);
            const double* const row = &sm.geo[3 * DIR][0];
            T lo[H0][3], lf[H0][3];  // own nodes, the other half's
            if constexpr (DIR == 0) {  // 4 consecutive nodes each
#pragma unroll
                for (int d = 0; d < 3; ++d)
#pragma unroll
                    for (int far = 0; far < 2; ++far) {
                        const double* r = row + d * NP + base + 4 * (far ? 1 - half : half);
                        const double2 a = *reinterpret_cast<const double2*>(r), b = *reinterpret_cast<const double2*>(r + 2);
                        const T v[4] = {(T)a.x, (T)a.y, (T)b.x, (T)b.y};
#pragma unroll
                        for (int m = 0; m < H0; ++m) (far ? lf : lo)[m][d] = half ? v[3 - m] : v[m];
                    }
            } else {
#pragma unroll
                for (int m = 0; m < H0; ++m)
#pragma unroll
                    for (int d = 0; d < 3; ++d) lo[m][d] = (T)row[d * NP + end + step * m];
            }
            // ---- the partner values of the line's node a: see line_kernel.cuh
            constexpr int S16 = DIR == 0 ? 1 : LS::slot16(STR), S8 = DIR > 0 ? STR / 2 : 1;
            const int mid = end + (half ? -H0 : H0) * STR;
            const int own16 = LS::slot16(end), own8 = LS::slot8(end), far16 = LS::slot16(mid), far8 = LS::slot8(mid);
            auto values = [&](const int a, T (&v)[NAUX]) {
                const int d = a < H0 ? a : a - H0;
                if constexpr (DIR == 0)
                    sm.aux.get(a < H0 ? own16 + d : far16 - d, a < H0 ? own8 ^ d : far8 ^ d, v);
                else
                    sm.aux.get((a < H0 ? own16 : far16) + (half ? -S16 : S16) * d,
                               (a < H0 ? own8 : far8) + (half ? -S8 : S8) * d, v);
            };
            T acc[H0][NS], o[H0][NAUX];
#pragma unroll
            for (int m = 0; m < H0; ++m) {
                values(m, o[m]);
#pragma unroll
                for (int s = 0; s < NS; ++s) acc[m][s] = T(0);
            }
#pragma unroll
            for (int m = 0; m < H0; ++m)
#pragma unroll
                for (int n = m + 1; n < H0; ++n) {  // pairs of own nodes, once for both
                    T G[3], un = T(0);
#pragma unroll
                    for (int d = 0; d < 3; ++d) {
                        G[d] = fma(pipec::dpar<T>(A, n, m), lo[n][d], -(pipec::dpar<T>(A, m, n) * lo[m][d]));
                        un = fma(o[m][1 + d] + o[n][1 + d], G[d], un);
                    }
                    const T f1 = (o[m][0] + o[n][0]) * un, pb = o[m][5] + o[n][5];
                    acc[m][0] += f1;
                    acc[n][0] -= f1;
#pragma unroll
                    for (int c = 1; c < NS; ++c) {
                        acc[m][c] = fma(f1, o[n][c], acc[m][c]);
                        acc[n][c] = fma(-f1, o[m][c], acc[n][c]);
                    }
#pragma unroll
                    for (int d = 0; d < 3; ++d) {
                        acc[m][1 + d] = fma(pb, G[d], acc[m][1 + d]);
                        acc[n][1 + d] = fma(-pb, G[d], acc[n][1 + d]);
                    }
                    acc[m][4] = fma(un, pb, acc[m][4]);
                    acc[n][4] = fma(-un, pb, acc[n][4]);
                }
#pragma unroll
            for (int a = H0; a < Q; ++a) {  // the other half's nodes
                T p[NAUX], lp[3];
                values(a, p);
#pragma unroll
                for (int d = 0; d < 3; ++d) lp[d] = DIR == 0 ? lf[a - H0][d] : (T)row[d * NP + end + step * a];
#pragma unroll
                for (int m = 0; m < H0; ++m) {
                    T G[3], un = T(0);
#pragma unroll
                    for (int d = 0; d < 3; ++d) {
                        G[d] = fma(pipec::dpar<T>(A, a, m), lp[d], -(pipec::dpar<T>(A, m, a) * lo[m][d]));
                        un = fma(o[m][1 + d] + p[1 + d], G[d], un);
                    }
                    const T f1 = (o[m][0] + p[0]) * un, pb = o[m][5] + p[5];
                    acc[m][0] += f1;
#pragma unroll
                    for (int c = 1; c < NS; ++c) acc[m][c] = fma(f1, p[c], acc[m][c]);
#pragma unroll
                    for (int d = 0; d < 3; ++d) acc[m][1 + d] = fma(pb, G[d], acc[m][1 + d]);
                    acc[m][4] = fma(un, pb, acc[m][4]);
                }
            }
            // the own-node parts of the averages, and the reflection of the far half
#pragma unroll
            for (int m = 0; m < H0; ++m) {
#pragma unroll
                for (int c = 1; c < NS; ++c) acc[m][c] = fma(o[m][c], acc[m][0], acc[m][c]);
#pragma unroll
                for (int s = 0; s < NS; ++s) acc[m][s] = half ? -acc[m][s] : acc[m][s];
            }
            // ---- face term at the thread's first node: wsJ nf (MJI follows at the end)
            {
                const T nv[3] = {(T)sg[0], (T)sg[1], (T)sg[2]}, wsJ = (T)sg[3];
                const T rm = T(2) * o[0][0], pm = T(2) * o[0][5], Em = rm * (T(2) * o[0][4]);
                const T rp = (T)tr[0], Ep = (T)tr[4], rinv = rcp_inner(rp);
                T um[3], mp[3], up[3], unm = T(0), unp = T(0);
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    um[d] = T(2) * o[0][1 + d];
                    mp[d] = (T)tr[1 + d];
                    up[d] = mp[d] * rinv;
                    unm = fma(um[d], nv[d], unm);
                    unp = fma(up[d], nv[d], unp);
                }
                const T pp = pipec::gas<T>(A, 1) * (Ep - (mp[0] * mp[0] + mp[1] * mp[1] + mp[2] * mp[2]) * (T(0.5) * rinv));
                // the larger wave speed |u.n| + sqrt(gamma p / rho) (euler.jl:62-68)
                const T wm = fabs(unm) + root(pipec::gas<T>(A, 0) * pm * rcp_inner(rm));
                const T wp = fabs(unp) + root(pipec::gas<T>(A, 0) * pp * rinv);
                // (q+ is q- on a boundary face: no jump, whatever the primitives' rounding)
                const T mx = A.surface_rusanov && nbf >= 0 ? fmax(wm, wp) : T(0);
                const T mnm = rm * unm, mnp = rp * unp;
#pragma unroll
                for (int s = 0; s < NS; ++s) {
                    T fm, fp, dq;
                    if (s == 0) {
                        fm = mnm;
                        fp = mnp;
                        dq = rp - rm;
                    } else if (s == 4) {
                        fm = unm * (Em + pm);
                        fp = unp * (Ep + pp);
                        dq = Ep - Em;
                    } else {
                        fm = mnm * um[s - 1] + pm * nv[s - 1];
                        fp = mnp * up[s - 1] + pp * nv[s - 1];
                        dq = mp[s - 1] - rm * um[s - 1];
                    }
                    acc[0][s] -= wsJ * ((fm + fp) * T(0.5) - (mx * dq) * T(0.5));
                }
            }
            // ---- hand the sums over, or finish: dq = rka dq + MJI sums; q_out = q + rkb dt dq
            if constexpr (POS < 2) {
#pragma unroll
                for (int m = 0; m < H0; ++m) {
                    const int n = LS::template sum_slot<T>(end + step * m);
#pragma unroll
                    for (int s = 0; s < NS; ++s) {
                        if constexpr (POS == 0) sm.acc[s][n] = acc[m][s];
                        else sm.acc[s][n] += acc[m][s];
                    }
                }
            } else {
                const int n0 = base + 4 * half;
                const size_t g = line::after(g0 + n0);
                const bool wide = (((uintptr_t)A.q_in | (uintptr_t)A.q_out | (sizeof(T) == 8 ? (uintptr_t)A.dq : 0)) & 31) == 0;
                T mji[4];
                {
                    const double2 a = *reinterpret_cast<const double2*>(&sm.geo[9][n0]);
                    const double2 b = *reinterpret_cast<const double2*>(&sm.geo[9][n0 + 2]);
                    mji[0] = (T)a.x, mji[1] = (T)a.y, mji[2] = (T)b.x, mji[3] = (T)b.y;
                }
                double qold[NS][4];  // all loads before the stores, which might alias them
                T old[NS][4];
#pragma unroll
                for (int s = 0; s < NS; ++s) {
                    line::load4(A.q_in + g + s * NP, wide, qold[s]);
#pragma unroll
                    for (int m = 0; m < 4; ++m) old[s][m] = T(0);
                    if (reads_dq) {
                        if constexpr (sizeof(T) == 8) {
                            line::load4(static_cast<const double*>(A.dq) + g + s * NP, wide, old[s]);
                        } else {
                            const float4 v = *reinterpret_cast<const float4*>(static_cast<const float*>(A.dq) + g + s * NP);
                            old[s][0] = v.x, old[s][1] = v.y, old[s][2] = v.z, old[s][3] = v.w;
                        }
                    }
                }
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
                    double out[4];
#pragma unroll
                    for (int m = 0; m < 4; ++m) {
                        v[m] += half ? acc[3 - m][s] : acc[m][s];
                        v[m] = fma((T)A.rka, old[s][m], v[m] * mji[m]);
                        out[m] = qold[s][m] + A.rkb_dt * (double)v[m];
                    }
                    if constexpr (sizeof(T) == 4)
                        *reinterpret_cast<float4*>(static_cast<float*>(A.dq) + g + s * NP) = make_float4(v[0], v[1], v[2], v[3]);
                    else
                        line::store4(static_cast<double*>(A.dq) + g + s * NP, wide, v);
                    line::store4(A.q_out + g + s * NP, wide, out);
                }
            }
        };
        using I0 = std::integral_constant<int, 0>;
        using I1 = std::integral_constant<int, 1>;
        using I2 = std::integral_constant<int, 2>;
        direction(I2{}, I0{});
        __syncthreads();  // #2: the z sums of the warp's planes; the z rows are free
        if (t == 96 && en < E) {
            fence_proxy_async();
            fetch_rows(2, en);
        }
        direction(I1{}, I1{});
        __syncwarp();
        direction(I0{}, I2{});
    }
    if (late) atomicExch(A.status, kStatusTimeout);  // the last element's rows
}

}  // namespace rb200
