/*
 * tg_ewald_leaf.cuh -- the leaf-sink Ewald kernels (gravity_PC_ewald,
 * src/gravity.cpp:616-678; gravity_PP_ewald, :491-614) as balanced work
 * units.  Included by tg_gravity.cu.
 *
 * The Ewald lists of a leaf are very uneven: large leaves in voids fail the
 * Ewald self test and interact with every leaf within (r_a + r_b)/theta, so
 * at theta = 0.2 on a clustered box 1% of the leaves hold half the PP_Ewald
 * pairs (up to 9e6 for one leaf); and a box of a few thousand particles has
 * fewer leaves than the GPU has SMs, each with every other leaf in its list.
 * So each leaf's PP_E list is cut into chunks of ew_kpp source leaves and its
 * PC_E list into chunks of EW_KPC source nodes; one 64-thread block (a thread
 * per sink) evaluates one chunk and writes its sinks' partial sums to its own
 * slot of a scratch array; k_ewald_reduce then adds a leaf's chunk sums in
 * chunk order to the leaf's FP64 accumulators.  The result does not depend on
 * scheduling.  Chunks are numbered PP_E first, then PC_E: off[0, nleaves] is
 * the scan of the leaves' PP_E chunk counts, off[nleaves + 1, 2 nleaves + 1]
 * that of their PC_E counts continued.
 *
 * A PP_E chunk's slots take 2 KB and its source sums 9 KB in FP32 and 20 KB in
 * FP64 (the Jacobian's 18 and 40 KB), and where every pair is an Ewald pair the
 * chunks grow with the square of the leaves.  So the leaves run in batches whose
 * chunks fit the scratch (EW_SCRATCH), each reduced before the next (leaf_batches), and where
 * the source leaves' own sums do not fit it, they are made for a range of vectors
 * at a time (k_ewald_tsum).  Neither changes the order of any sum.
 */
#pragma once

constexpr int EW_KPP_MAX = 32;
/* PP_E source leaves per chunk: 24 chunks of a list, of 4 to 32 leaves (at most
 * 32 * 64 * 64 pairs), so that small trees fill the GPU.  Leaf Ewald and L2P in ms
 * with 16 chunks of 8 leaves on / with 24 of 4 on (theta 0.7, leaf 64): 4096 uniform
 * 0.40 / 0.31, 20000 0.77 / 0.72, 32768 0.92 / 0.84, 50000 0.61 / 0.53, 1e5 and more,
 * and theta 0.25 to 0.5, the same.  By the list alone, so the order of the sums does
 * not depend on which leaves are active. */
__host__ __device__ __forceinline__ int32_t ew_kpp(int32_t len) {
    const int32_t k = (len + 23) / 24;
    return k < 4 ? 4 : (k > EW_KPP_MAX ? EW_KPP_MAX : k);
}
constexpr int EW_KPC = 64; /* PC_E source nodes per chunk */

/* leaves [l0, l1) with their PP_E chunks [a0, a0 + na) and PC_E chunks [c0, c0 + nc),
 * whose slots follow each other in that order */
struct EwBatch {
    int32_t l0, l1, a0, na, c0, nc;
};

/* one warp per leaf: chunk counts (zeros at li = nleaves, so that the scan ends
 * in the totals); with slot, marks the source leaves of the PP_E lists */
__global__ void k_ewald_count(const int32_t *__restrict__ leaves, int32_t nleaves, ListView LV,
                              int32_t *__restrict__ cnt, int32_t *__restrict__ slot) {
    const int32_t li = (int32_t)(((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    const int lane = threadIdx.x & 31;
    if (li > nleaves) return;
    int32_t npp = 0, npc = 0;
    if (li < nleaves) {
        const int32_t leaf = leaves[li];
        npp = LV.len[TG_PP_E][leaf], npc = LV.len[TG_PC_E][leaf];
        if (slot) {
            const int32_t *lst = LV.pool[TG_PP_E] + LV.off[TG_PP_E][leaf];
            for (int32_t e = lane; e < npp; e += 32) slot[lst[e]] = 0;
        }
    }
    if (lane == 0) {
        cnt[li] = (npp + ew_kpp(npp) - 1) / ew_kpp(npp);
        cnt[nleaves + 1 + li] = (npc + EW_KPC - 1) / EW_KPC;
    }
}

/* a slot for every marked source leaf (slot: 0 marked, -1 not), in no particular order */
__global__ void k_ewald_slots(int64_t nn, int32_t *__restrict__ slot, int32_t *__restrict__ src,
                              int32_t *__restrict__ count) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const bool m = i < nn && slot[i] == 0;
    const uint32_t b = __ballot_sync(0xffffffffu, m);
    if (!b) return;
    const int lane = threadIdx.x & 31;
    int32_t at = 0;
    if (lane == __ffs(b) - 1) at = atomicAdd(count, __popc(b));
    at = __shfl_sync(0xffffffffu, at, __ffs(b) - 1);
    if (m) {
        const int32_t k = at + __popc(b & ((1u << lane) - 1u));
        slot[i] = k;
        src[k] = (int32_t)i;
    }
}

/* the leaf of chunk c: largest li with off[li] <= c */
__device__ __forceinline__ int32_t ew_leaf(const int32_t *__restrict__ off, int32_t nleaves, int64_t c) {
    int32_t lo = 0, hi = nleaves - 1;
    while (lo < hi) {
        const int32_t mid = (lo + hi + 1) >> 1;
        if ((int64_t)off[mid] <= c) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

/* the source sums of a chunk (rows of sf, one per source leaf, holding vectors [t0, t1)) into its row of tpart */
template <class S>
__device__ __forceinline__ void ew_tsum(const int32_t *s_row, int n, int t0, int t1, int tid, const S *__restrict__ sf,
                                        double m, S *__restrict__ out) {
    for (int t = t0 + tid; t < t1; t += 64) {
        S a{};
#pragma unroll 8
        for (int u = 0; u < n; u++) sep_madd(a, m, sf[(int64_t)s_row[u] * (t1 - t0) + t - t0]);
        out[t] = a;
    }
}
/* the same in a launch of its own, for the chunks from `first` on, rows of N vectors */
template <class S>
__global__ void __launch_bounds__(64) k_ewald_tsum(int N, double m, const int32_t *__restrict__ leaves,
                                                   int32_t nleaves, int32_t first, const int32_t *__restrict__ off,
                                                   ListView LV, const int32_t *__restrict__ slot, int t0, int t1,
                                                   const S *__restrict__ sf, S *__restrict__ tpart) {
    __shared__ int32_t s_row[EW_KPP_MAX];
    const int tid = threadIdx.x;
    const int64_t c = (int64_t)first + blockIdx.x;
    const int32_t li = ew_leaf(off, nleaves, c), k = (int32_t)(c - off[li]);
    const int32_t leaf = leaves[li];
    const int32_t *lst = LV.pool[TG_PP_E] + LV.off[TG_PP_E][leaf];
    const int32_t len = LV.len[TG_PP_E][leaf], kpp = ew_kpp(len), e0 = k * kpp, e1 = min(len, e0 + kpp);
    if (tid < e1 - e0) s_row[tid] = slot[lst[e0 + tid]];
    __syncthreads();
    ew_tsum<S>(s_row, e1 - e0, t0, t1, tid, sf, m, tpart + (int64_t)blockIdx.x * N);
}

/* one chunk of a PP_E list: entries [k ew_kpp, ...) of its leaf.  The
 * real-space part per pair and, with sf (all vectors), the chunk's reciprocal
 * source sums (tpart).  Block b takes chunk first + b, its slot is b.
 *
 * What bounds it: latency of the image and polynomial chains at 16 blocks per SM in
 * FP32 (64 registers, issue 66 to 78 %, FP64 pipe 27 to 34 %): 64^3 clustered, theta 0.25,
 * 9.4e10 pairs/s (8.8e10 with every pair's images folded by itself).  Measured and
 * not kept: 12 or 14 blocks, the polynomials in even and odd halves, the erfc of
 * 7.1.26 (0.69 ms for 0.62 at 32768 uniform). */
template <class T>
__global__ void __launch_bounds__(64, sizeof(T) == 4 ? 16 : 12)
    k_ewald_pp(GParams P, const int32_t *__restrict__ leaves, int32_t nleaves, int32_t first,
               const int32_t *__restrict__ off, const int32_t *__restrict__ pb, const int32_t *__restrict__ pe,
               const int4 *__restrict__ pos, ListView LV, EwaldTables E, SepNear K, double *__restrict__ part,
               const int32_t *__restrict__ slot, const double2 *__restrict__ sf, double2 *__restrict__ tpart) {
    __shared__ int4 sy[64];
    __shared__ int32_t s_row[EW_KPP_MAX];
    const int tid = threadIdx.x;
    const int64_t c = (int64_t)first + blockIdx.x;
    const int32_t li = ew_leaf(off, nleaves, c), k = (int32_t)(c - off[li]);
    const int32_t leaf = leaves[li];
    const int32_t b = pb[leaf], cnt = pe[leaf] - b;
    const bool active = tid < cnt;
    const int4 xi = pos[b + (active ? tid : 0)];
    SepPairs<T> s;
    s.init();
    const int32_t *lst = LV.pool[TG_PP_E] + LV.off[TG_PP_E][leaf];
    const int32_t len = LV.len[TG_PP_E][leaf], kpp = ew_kpp(len), e0 = k * kpp, e1 = min(len, e0 + kpp);
    if (tid < e1 - e0) s_row[tid] = slot[lst[e0 + tid]];
    for (int32_t e = e0; e < e1; e++) {
        const int32_t src = lst[e];
        const int32_t sb = pb[src], sn = pe[src] - sb; /* leaf_max <= 64: one stage */
        __syncthreads();
        if (tid < sn) sy[tid] = pos[sb + tid];
        __syncthreads();
        if (tid < ((cnt + 31) & ~31)) /* a warp without sinks only stages */
            for (int32_t q = 0; q < sn;) {
                const int32_t q1 = min(sn, q + SEP_FOLD);
                for (; q < q1; q++) s.add(E, K, P.m_d, xi, sy[q]);
                s.fold();
            }
    }
    if (active)
        for (int q = 0; q < 4; q++) part[4 * ((int64_t)blockIdx.x * 64 + tid) + q] = s.get(q, P.m_d);
    /* this chunk's reciprocal source sums, a thread per vector (s_row: written before the loop's barriers) */
    if (sf) ew_tsum<double2>(s_row, e1 - e0, 0, Sep<T>::N, tid, sf, P.m_d, tpart + (int64_t)blockIdx.x * Sep<T>::N);
}

/* one chunk of a PC_E list: block b takes chunk first + b (offp: the PC_E part of the scan), its slot is slot0 + b */
template <class T>
__global__ void __launch_bounds__(64, sizeof(T) == 4 ? 8 : 6)
    k_ewald_pc(const int32_t *__restrict__ leaves, int32_t nleaves, int32_t first, int32_t slot0,
               const int32_t *__restrict__ offp,
               const int32_t *__restrict__ pb, const int32_t *__restrict__ pe, const MSrc *__restrict__ ms,
               const int4 *__restrict__ pos, ListView LV, EwaldTables E, double *__restrict__ part) {
    const int tid = threadIdx.x;
    const int64_t c = (int64_t)first + blockIdx.x;
    const int32_t li = ew_leaf(offp, nleaves, c), k = (int32_t)(c - offp[li]);
    const int32_t leaf = leaves[li];
    const int32_t b = pb[leaf], cnt = pe[leaf] - b;
    if (tid >= cnt) return;
    const int4 xi4 = pos[b + tid];
    const int32_t xi[3] = {xi4.x, xi4.y, xi4.z};
    Acc<T> aphi, ag[3];
    aphi.init(0.0);
    for (int d = 0; d < 3; d++) ag[d].init(0.0);
    const int32_t *lst = LV.pool[TG_PC_E] + LV.off[TG_PC_E][leaf];
    const int32_t e0 = k * EW_KPC, e1 = min(LV.len[TG_PC_E][leaf], e0 + EW_KPC);
    for (int32_t e = e0; e < e1; e++) {
        const MSrc &s = ms[lst[e]];
        T dX[3], D[LP], M[MP];
#pragma unroll
        for (int d = 0; d < 3; d++) dX[d] = sep<T>(xi[d], s.x[d], true);
        green_ewald_any<T>(E, dX, D);
#pragma unroll
        for (int q = 0; q < MP; q++) M[q] = T(s.m[q]);
        T ph, g[3];
        contract_M2P<T>(ph, g, M, D);
        aphi.add(ph);
        for (int d = 0; d < 3; d++) ag[d].add(g[d]);
    }
    double *o = part + 4 * ((int64_t)(slot0 + blockIdx.x) * 64 + tid);
    o[0] = aphi.get();
    for (int d = 0; d < 3; d++) o[1 + d] = ag[d].get();
}

/* Add each leaf's chunk sums, in chunk order, to its FP64 accumulators, and
 * the reciprocal part from the PP_E chunks' source sums (in chunk
 * order).  One block per leaf of the batch; the four groups of 64 threads take a
 * quarter of the vectors each. */
template <class T>
__global__ void __launch_bounds__(256) k_ewald_reduce(EwBatch B, const int32_t *__restrict__ leaves, int32_t nleaves,
                                                      const int32_t *__restrict__ off, const int32_t *__restrict__ pb,
                                                      const int32_t *__restrict__ pe, const double *__restrict__ part,
                                                      double *__restrict__ acc, const double2 *__restrict__ tpart,
                                                      const int4 *__restrict__ pos, EwaldTables E) {
    __shared__ SepTrig<T> trig;
    __shared__ double2 sT[Sep<T>::N];
    __shared__ double sv[4][64][4];
    const int32_t li = B.l0 + blockIdx.x;
    const int tid = threadIdx.x, t = tid & 63, grp = tid >> 6;
    const int32_t *offp = off + nleaves + 1;
    const int32_t a0 = off[li] - B.a0, a1 = off[li + 1] - B.a0; /* the leaf's slots */
    const int32_t p0 = offp[li] - B.c0 + B.na, p1 = offp[li + 1] - B.c0 + B.na;
    if (a1 == a0 && p1 == p0) return; /* block-uniform */
    const int32_t leaf = leaves[li];
    const int32_t b = pb[leaf], cnt = pe[leaf] - b;
    double v[4] = {0.0, 0.0, 0.0, 0.0};
    if (a1 > a0) { /* block-uniform */
        for (int i = tid; i < Sep<T>::N; i += 256) {
            double sx = 0.0, sy = 0.0;
            for (int64_t c = a0; c < a1; c++) {
                const double2 f = tpart[c * Sep<T>::N + i];
                sx += f.x;
                sy += f.y;
            }
            const double w = sizeof(T) == 4 ? __ldg(&E.sep_w[i]) : 1.0; /* FP32: the weight here */
            sT[i] = make_double2(w * sx, w * sy);
        }
        sep_trig<T>(trig, pos + b, cnt);
        __syncthreads();
        if (t < cnt) sep_eval<T>(E, trig, sT, grp, t, pos + b, v[0], v + 1);
    }
#pragma unroll
    for (int q = 0; q < 4; q++) sv[grp][t][q] = v[q];
    __syncthreads();
    if (t >= cnt || grp != 0) return;
    double *o = acc + 4 * (int64_t)(b + t);
    double w[4] = {0.0, 0.0, 0.0, 0.0};
    for (int64_t c = a0; c < a1; c++)
#pragma unroll
        for (int q = 0; q < 4; q++) w[q] += part[4 * (c * 64 + t) + q];
    for (int64_t c = p0; c < p1; c++)
#pragma unroll
        for (int q = 0; q < 4; q++) w[q] += part[4 * (c * 64 + t) + q];
#pragma unroll
    for (int q = 0; q < 4; q++) o[q] += w[q] + ((sv[0][t][q] + sv[1][t][q]) + (sv[2][t][q] + sv[3][t][q]));
}
