/*
 * tg_ewald_node.cuh -- the node-sink Ewald kernels (gravity_CC_ewald,
 * src/gravity.cpp:680-731; gravity_CP_ewald, :733-785) as balanced work
 * units.  Included by tg_gravity.cu after k_node.
 *
 * Each node's CC_E list is cut into chunks of EN_KCC source nodes and its
 * CP_E list into chunks of EN_KCP source leaves.  One warp evaluates one
 * chunk, lanes over the chunk's sources (CP_E: over the particles of its
 * leaves as one range): a source's green_ewald per lane, in FP32 from the
 * expansion table (tg_ewald_table.cuh), in FP64 from the sums, where a chunk
 * of fewer than EWALD_WARP_LIST sources is evaluated one source at a time by
 * the whole warp (green_ewald_warp).  The warp's FP64 sum of the 35 expansion
 * terms goes to the chunk's slot of a scratch array, and k_node_ewald_reduce
 * adds a node's chunk sums, in chunk order, to its Lloc.
 */
#pragma once

constexpr int EN_KCC = 128; /* CC_E source nodes per chunk (4 per lane) */
constexpr int EN_KCP = 4;   /* CP_E source leaves per chunk */
#ifndef EN_MINB
#define EN_MINB 4 /* resident 128-thread blocks per SM the FP32 kernel is compiled for (3: 126, 4: 125 ms at 256^3) */
#endif
#ifndef EN_MINB_D
#define EN_MINB_D 2 /* and the FP64 kernel */
#endif

__global__ void k_node_ewald_count(int64_t nn, const int32_t *__restrict__ pb, const int32_t *__restrict__ pe,
                                   ListView LV, int32_t *__restrict__ cnt) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i > nn) return;
    if (i == nn || pe[i] == pb[i]) {
        cnt[i] = 0;
        return;
    }
    const int32_t ncc = LV.len[TG_CC_E][i], ncp = LV.len[TG_CP_E][i];
    cnt[i] = (ncc + EN_KCC - 1) / EN_KCC + (ncp + EN_KCP - 1) / EN_KCP;
}

/* the node of chunk c: largest i with off[i] <= c */
__device__ __forceinline__ int64_t en_node(const int32_t *__restrict__ off, int64_t nn, int32_t c) {
    int64_t lo = 0, hi = nn - 1;
    while (lo < hi) {
        const int64_t mid = (lo + hi + 1) >> 1;
        if (off[mid] <= c) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

template <class T>
__global__ void __launch_bounds__(128, sizeof(T) == 4 ? EN_MINB : EN_MINB_D)
    k_node_ewald(GParams P, int64_t nn, int32_t nchunks, const int32_t *__restrict__ off,
                 const int32_t *__restrict__ pb, const int32_t *__restrict__ pe, const MSrc *__restrict__ ms,
                 const int4 *__restrict__ pos, ListView LV, EwaldTables E, double *__restrict__ part) {
    const int lane = threadIdx.x & 31;
    const int32_t c = (int32_t)(((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    if (c >= nchunks) return;
    const int64_t i = en_node(off, nn, c);
    const int32_t k = c - off[i];
    const int32_t X[3] = {ms[i].x[0], ms[i].x[1], ms[i].x[2]};
    /* each lane's expansion sums (odd stride LP: no bank conflicts).  FP64
     * keeps them here throughout, which leaves the registers to green_ewald;
     * FP32, in registers until the end */
    constexpr int WARP_FLOATS = sizeof(T) == 4 ? 32 * ET_STRIDE : 32 * LP; /* FP32: a warp's table rows before that */
    __shared__ __align__(16) T s_buf[4 * WARP_FLOATS];
    T *const sL = s_buf + (threadIdx.x >> 5) * WARP_FLOATS;
    T *const sl = sL + lane * LP;
    T Lreg[sizeof(T) == 4 ? LP : 1];
    T *const L = sizeof(T) == 4 ? Lreg : sl;
#pragma unroll
    for (int q = 0; q < LP; q++) L[q] = T(0);
    const int32_t ncc = LV.len[TG_CC_E][i];
    const int32_t kcc = (ncc + EN_KCC - 1) / EN_KCC;
    if (k < kcc) {
        const int32_t *lst = LV.pool[TG_CC_E] + LV.off[TG_CC_E][i];
        const int32_t e0 = k * EN_KCC, e1 = min(ncc, e0 + EN_KCC);
        if constexpr (sizeof(T) == 4) {
            for (int32_t j0 = e0; j0 < e1; j0 += 32) {
                const MSrc &s = ms[lst[min(j0 + lane, e1 - 1)]];
                float dX[3], o[3], D[LP], M[MP];
                uint32_t sg[3];
#pragma unroll
                for (int d = 0; d < 3; d++) dX[d] = sep<float>(X[d], s.x[d], true);
                et_stage(E.tab, et_locate(dX, o, sg), min(32, e1 - j0), sL);
                if (j0 + lane >= e1) continue;
                et_eval(reinterpret_cast<const float4 *>(sL + lane * ET_STRIDE), dX, o, sg, D);
#pragma unroll
                for (int q = 0; q < MP; q++) M[q] = s.m[q];
                contract_M2L<float, float>(L, M, D);
            }
        } else if (e1 - e0 >= EWALD_WARP_LIST) {
            for (int32_t j = e0 + lane; j < e1; j += 32) {
                const MSrc &s = ms[lst[j]];
                T dX[3], D[LP], M[MP];
#pragma unroll
                for (int d = 0; d < 3; d++) dX[d] = sep<T>(X[d], s.x[d], true);
                green_ewald_any<T>(E, dX, D);
#pragma unroll
                for (int q = 0; q < MP; q++) M[q] = T(s.m[q]);
                contract_M2L<T, T>(L, M, D);
            }
        } else {
            for (int32_t j = e0; j < e1; j++) {
                const MSrc &s = ms[lst[j]];
                T dX[3], D[LP], M[MP];
#pragma unroll
                for (int d = 0; d < 3; d++) dX[d] = sep<T>(X[d], s.x[d], true);
                if (!(dX[0] * dX[0] + dX[1] * dX[1] + dX[2] * dX[2] > T(1.0e-12))) {
                    /* the node itself: green_ewald(0) = phi0 only (tigergrav/green.hpp:279) */
                    if (lane == 0) L[E0()] += T(s.m[0]) * T(EWALD_PHI0);
                    continue;
                }
#pragma unroll
                for (int q = 0; q < MP; q++) M[q] = T(s.m[q]);
                green_ewald_warp(E, dX, D, lane);
                contract_M2L<T, T>(L, M, D);
            }
        }
    } else {
        const int32_t ncp = LV.len[TG_CP_E][i];
        const int32_t *lst = LV.pool[TG_CP_E] + LV.off[TG_CP_E][i];
        const int32_t e0 = (k - kcc) * EN_KCP, e1 = min(ncp, e0 + EN_KCP);
        const T m = T(P.m_d);
        /* the chunk's particles as one range, lanes over it: the first EN_KCP lanes hold the leaves */
        int32_t sb = 0, incl = 0;
        if (lane < e1 - e0) {
            const int32_t src = lst[e0 + lane];
            sb = pb[src];
            incl = pe[src] - sb;
        }
#pragma unroll
        for (int o = 1; o < EN_KCP; o <<= 1) {
            const int32_t v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
        }
        const int32_t total = __shfl_sync(0xffffffffu, incl, EN_KCP - 1);
        const int32_t sb0 = __shfl_sync(0xffffffffu, sb, 0);
        for (int32_t q0 = 0; q0 < total; q0 += 32) {
            const int32_t q = q0 + lane;
            int32_t at = 0, lo = 0; /* this lane's particle */
#pragma unroll
            for (int u = 0; u < EN_KCP; u++) {
                const int32_t hi = __shfl_sync(0xffffffffu, incl, u), b = __shfl_sync(0xffffffffu, sb, u);
                if (q >= lo && q < hi) at = b + q - lo;
                lo = hi;
            }
            const int4 y = pos[q < total ? at : sb0];
            const int32_t yy[3] = {y.x, y.y, y.z};
            T dX[3], D[LP];
#pragma unroll
            for (int d = 0; d < 3; d++) dX[d] = sep<T>(X[d], yy[d], true);
            if constexpr (sizeof(T) == 4) {
                float o[3];
                uint32_t sg[3];
                et_stage(E.tab, et_locate(dX, o, sg), min(32, total - q0), sL);
                if (q < total) {
                    et_eval(reinterpret_cast<const float4 *>(sL + lane * ET_STRIDE), dX, o, sg, D);
                    contract_P2L<T, T>(L, m, D);
                }
            } else if (q < total) {
                green_ewald_any<T>(E, dX, D);
                contract_P2L<T, T>(L, m, D);
            }
        }
    }
    /* the warp's sum in FP64, a lane per term */
    if constexpr (sizeof(T) == 4) {
        __syncwarp(); /* the last rows are read */
#pragma unroll
        for (int q = 0; q < LP; q++) sl[q] = L[q];
    }
    __syncwarp();
    const T *w = sL;
    for (int q = lane; q < LP; q += 32) {
        double v = 0.0;
#pragma unroll 8
        for (int l = 0; l < 32; l++) v += (double)w[l * LP + q];
        part[(int64_t)c * LP + q] = v;
    }
}

/* Lloc += the node's chunk sums, in chunk order: one thread per (node, term) */
__global__ void k_node_ewald_reduce(int64_t nn, const int32_t *__restrict__ off, const double *__restrict__ part,
                                    double *__restrict__ Lloc) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nn * LP) return;
    const int64_t i = t / LP;
    const int q = (int)(t - i * LP);
    if (off[i + 1] == off[i]) return;
    double v = 0.0;
    for (int32_t c = off[i]; c < off[i + 1]; c++) v += part[(int64_t)c * LP + q];
    Lloc[i * LP + q] += v;
}
