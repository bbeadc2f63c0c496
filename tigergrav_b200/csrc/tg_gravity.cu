/*
 * tg_gravity.cu -- the interaction kernels of kick_fmm (src/tree.cpp:400-631)
 * and the eight kernel-level seams of tigergrav/gravity.hpp:39-46.
 *
 *   k_node   one warp per node, lanes over sources: CC/CP direct; lane
 *            sums are reduced in FP64 -> Lloc (35 doubles)
 *   k_node_ewald (tg_ewald_node.cuh)  CC/CP Ewald in balanced chunks, one
 *            warp per chunk, one source's whole green_ewald per lane
 *            (walking only the lattice images inside the real-space cut);
 *            chunk sums added to Lloc in order
 *   k_l2l    one thread per node of a level, top-down:
 *            L = (L_parent << (x - x_parent)) + Lloc          (FP64)
 *   k_leaf   one block per leaf, one thread per sink particle: L2P, then
 *            PC_direct, PP_direct (source leaves staged in shared memory),
 *            PC_ewald, PP_ewald; -phi_self once (src/gravity.cpp:295).
 *            The FP32 path with leaf_max <= 64 runs it without PP_direct
 *            (into an FP64 buffer) and then pp_direct (tg_pp2.cuh), which adds
 *            PP_direct and phi_self and writes the float4 result.
 *
 * Precision: T = float (FP32 path: FP32 arithmetic, per-tile FP32 partial
 * sums folded into Kahan-compensated accumulators) or T = double (the plain
 * FP64 port).  Expansions L are FP64 in both.
 */
#include <memory>
#include <mutex>
#include <new>

#include "tg_solver.cuh"

namespace tg {

struct GParams {
    float m_f;
    double m_d;
    double h;
    float H, halfH, Hinv, H3inv, H2;
    double phi_self; /* -315/128 m / h */
    int ewald;
};

static GParams make_gparams(const tg_params &p) {
    GParams g;
    g.m_f = (float)p.m;
    g.m_d = p.m;
    g.h = p.soft_len;
    g.H = (float)p.soft_len;
    g.halfH = (float)(0.5 * p.soft_len);
    g.Hinv = (float)(1.0 / p.soft_len);
    g.H3inv = (float)(1.0 / p.soft_len / p.soft_len / p.soft_len);
    g.H2 = (float)(p.soft_len * p.soft_len);
    g.phi_self = (-315.0 / 128.0) * p.m / p.soft_len;
    g.ewald = p.ewald ? 1 : 0;
    return g;
}

/* ---- accumulators ---- */
template <class T> struct Acc;
template <> struct Acc<float> {
    KahanF k;
    __device__ __forceinline__ void init(double v) { k.s = (float)v; k.c = 0.0f; }
    __device__ __forceinline__ void add(float v) { k.add(v); }
    __device__ __forceinline__ double get() const { return (double)k.s - (double)k.c; }
};
template <> struct Acc<double> {
    double s;
    __device__ __forceinline__ void init(double v) { s = v; }
    __device__ __forceinline__ void add(double v) { s += v; }
    __device__ __forceinline__ double get() const { return s; }
};

/* ---- PP direct pair (src/gravity.cpp:214-287), GADGET spline softening.
 * Returns f (force factor, g -= dX * m * f) and p (phi -= m * p). */
template <class T>
__device__ __forceinline__ void pp_direct_pair(const GParams &P, const T *dX, T &f, T &p) {
    const T r2 = dX[0] * dX[0] + dX[1] * dX[1] + dX[2] * dX[2];
    if (r2 > T(P.h * P.h)) {
        const T rinv = t_rsqrt(r2);
        p = rinv;
        f = rinv * rinv * rinv;
        return;
    }
    const T H = T(P.h), halfH = T(0.5 * P.h), Hinv = T(1.0 / P.h), H3inv = T(1.0 / P.h / P.h / P.h);
    const T r = t_sqrt(r2);
    const T rinv = T(1) / (r > halfH ? r : halfH);
    const T rinv3 = rinv * rinv * rinv;
    const T sw1 = r > H ? T(1) : T(0);
    const T sw3 = r < halfH ? T(1) : T(0);
    const T sw2 = T(1) - sw1 - sw3;
    T roh = r * Hinv;
    roh = roh < T(1) ? roh : T(1);
    const T roh2 = roh * roh;
    const T roh3 = roh2 * roh;
    T f2 = T(-32.0 / 3.0);
    f2 = fma(f2, roh, T(192.0 / 5.0));
    f2 = fma(f2, roh, T(-48.0));
    f2 = fma(f2, roh, T(64.0 / 3.0));
    f2 = fma(f2, roh3, T(-1.0 / 15.0));
    f2 *= rinv3;
    T f3 = T(32.0);
    f3 = fma(f3, roh, T(-192.0 / 5.0));
    f3 = fma(f3, roh2, T(32.0 / 3.0));
    f3 *= H3inv;
    f = sw1 * rinv3 + sw2 * f2 + sw3 * f3;
    T p2 = T(32.0 / 15.0);
    p2 = fma(p2, roh, T(-48.0 / 5.0));
    p2 = fma(p2, roh, T(16.0));
    p2 = fma(p2, roh, T(-32.0 / 3.0));
    p2 = fma(p2, roh2, T(16.0 / 5.0));
    p2 = fma(p2, roh, T(-1.0 / 15.0));
    p2 *= rinv;
    T p3 = T(-32.0 / 5.0);
    p3 = fma(p3, roh, T(48.0 / 5.0));
    p3 = fma(p3, roh2, T(-16.0 / 3.0));
    p3 = fma(p3, roh2, T(14.0 / 5.0));
    p3 *= Hinv;
    p = sw1 * rinv + sw2 * p2 + sw3 * p3;
}

/* Nearest image (n = 0) of the real-space sum together with the removal of
 * the direct 1/r that the Ewald kernels perform (src/gravity.cpp:594-600):
 *   -erfc(alpha r)/r + 1/r = erf(alpha r)/r
 *   force factor (1 - erfc(alpha r) - (2 alpha r/sqrt(pi)) e^{-alpha^2 r^2}) / r^3
 * written without the cancellation of the two large 1/r terms (alpha: the
 * Ewald split, 2 in the reference).  With x = alpha r,
 * F(x) = erf(x) - (2x/sqrt(pi)) e^{-x^2} = (2/sqrt(pi)) sum_{k>=1} (-1)^{k+1} 2k x^{2k+1} / (k! (2k+1))
 * (Taylor series of erf and of x e^{-x^2}), used below x = 0.5. */
template <class T>
__device__ __forceinline__ void ewald_nearest(T alpha, T r, T rinv, T &p0, T &f0) {
    const T x = alpha * r;
    const T erfx = erf(x);
    p0 = erfx * rinv;
    if (x < T(0.5)) {
        const T y = x * x;
        T s = T(0);
        if constexpr (sizeof(T) == 8) { /* FP32 ends at y^7 */
            s = T(1.0 / 41731200.0);
            s = fma(s, y, T(-1.0 / 3810240.0));
            s = fma(s, y, T(1.0 / 383040.0));
        }
        s = fma(s, y, T(-1.0 / 42840.0));
        s = fma(s, y, T(1.0 / 5400.0));
        s = fma(s, y, T(-1.0 / 780.0));
        s = fma(s, y, T(1.0 / 132.0));
        s = fma(s, y, T(-1.0 / 27.0));
        s = fma(s, y, T(1.0 / 7.0));
        s = fma(s, y, T(-0.4));
        s = fma(s, y, T(2.0 / 3.0));
        f0 = T(1.1283791670955126) * (alpha * alpha * alpha) * s; /* F / r^3 = alpha^3 F / x^3 */
    } else {
        const T F = erfx - T(1.1283791670955126) * x * exp(-x * x);
        f0 = F * rinv * rinv * rinv;
    }
}

/* ---- PP Ewald pair (src/gravity.cpp:533-603): phi and g of the periodic
 * correction per unit mass.  The n = 0 image is taken by ewald_nearest. */
template <class T>
__device__ __forceinline__ void pp_ewald_pair(const EwaldTables &E, const T *dX0, T &phi, T *g) {
    const T r2 = dX0[0] * dX0[0] + dX0[1] * dX0[1] + dX0[2] * dX0[2];
    if (!(r2 > T(1.0e-12))) { /* r <= rcut: phi0, no force */
        phi = T(EWALD_PHI0);
        g[0] = g[1] = g[2] = T(0);
        return;
    }
    T ph = T(0), gx = T(0), gy = T(0), gz = T(0);
    ewald_images<T>(dX0, [&](const T *d, T rr2, bool origin) {
        if (origin) return;
        const T dx = d[0], dy = d[1], dz = d[2];
        const T rinv = t_rsqrt(rr2);
        const T r = rr2 * rinv;
        T expfac;
        const T erfc = t_erfcexp(T(2) * r, &expfac);
        const T d0 = -erfc * rinv;
        const T expfactor = T(2.2567583341910252) * r * expfac;
        const T d1 = (expfactor + erfc) * rinv * rinv * rinv;
        ph += d0;
        gx -= dx * d1;
        gy -= dy * d1;
        gz -= dz * d1;
    }, ewald_rcut2_pp<T>());
    for (int t = 0; t < NFOUR_HALF; t++) {
        const float4 h = __ldg(&E.four[t]);
        const T hdotdx = dX0[0] * T(h.x) + dX0[1] * T(h.y) + dX0[2] * T(h.z);
        T s, c;
        t_sincos2pi(hdotdx, &s, &c);
        T H0, Hx, Hy, Hz;
        if (sizeof(T) == 4) {
            const float4 q = __ldg(&E.Pf[t]);
            H0 = T(q.x), Hx = T(q.y), Hy = T(q.z), Hz = T(q.w);
        } else {
            const double2 q0 = __ldg(&E.Pd[2 * t]), q1 = __ldg(&E.Pd[2 * t + 1]);
            H0 = T(q0.x), Hx = T(q0.y), Hy = T(q1.x), Hz = T(q1.y);
        }
        ph += H0 * c;
        gx -= Hx * s;
        gy -= Hy * s;
        gz -= Hz * s;
    }
    const T rinv = t_rsqrt(r2);
    T p0, f0;
    ewald_nearest<T>(T(2), r2 * rinv, rinv, p0, f0);
    phi = ph + (T(0.78539816339744831) + p0);
    g[0] = gx + dX0[0] * f0;
    g[1] = gy + dX0[1] * f0;
    g[2] = gz + dX0[2] * f0;
}

/* full green_ewald(dX) evaluated by one thread (tigergrav/green.hpp:189-286) */
template <class T>
__device__ __forceinline__ void green_ewald_full(const EwaldTables &E, const T *X, T *D) {
#pragma unroll
    for (int k = 0; k < LP; k++) D[k] = T(0);
    const T r2 = X[0] * X[0] + X[1] * X[1] + X[2] * X[2];
    if (!(r2 > T(1.0e-12))) {
        D[0] = T(EWALD_PHI0);
        return;
    }
    EwaldMom<T> mom;
    mom.init();
    if constexpr (sizeof(T) == 4) {
        /* FP32: the n = 0 image carries the removal of the direct 1/r */
        ewald_images<T>(X, [&](const T *d, T rr2, bool origin) {
            if (origin) ewald_origin_add(D, mom, d, rr2);
            else ewald_real_image<T>(D, mom, d, rr2);
        });
    } else {
        ewald_images<T>(X, [&](const T *d, T rr2, bool) { ewald_real_image<T>(D, mom, d, rr2); });
    }
    ewald_mom_finish<T>(D, mom);
    for (int t = 0; t < NFOUR_HALF; t++) {
        const T *H = (sizeof(T) == 4) ? (const T *)(E.Hf + HS * t) : (const T *)(E.Hd + HS * t);
        ewald_four_term<T>(D, X, __ldg(&E.four[t]), H);
    }
    if constexpr (sizeof(T) == 4) D[E0()] += T(0.78539816339744831); /* pi/4 (tigergrav/green.hpp:270) */
    else ewald_finish<T, T>(D, X);
}

/* FP64: green_ewald(dX) split over a warp: this lane's share of the real-space
 * candidates and of the reciprocal terms, plus, on lane 0, the final assembly.
 * The sum of the 32 partial results is green_ewald; the M2L contractions are linear,
 * so each lane contracts its own part.  X must not be 0 (the caller handles
 * r <= 1e-6). */
__device__ __forceinline__ void green_ewald_warp(const EwaldTables &E, const double *X, double *D, int lane) {
#pragma unroll
    for (int k = 0; k < LP; k++) D[k] = 0.0;
    EwaldMom<double> mom;
    mom.init();
    for (int t = lane; t < NREAL; t += 32) {
        const float4 n = __ldg(&E.real[t]);
        const double dx[3] = {X[0] - n.x, X[1] - n.y, X[2] - n.z};
        const double r2 = dx[0] * dx[0] + dx[1] * dx[1] + dx[2] * dx[2];
        if (r2 < ewald_rcut2<double>()) ewald_real_image<double>(D, mom, dx, r2);
    }
    ewald_mom_finish<double>(D, mom);
    for (int t = lane; t < NFOUR_HALF; t += 32) ewald_four_term<double>(D, X, __ldg(&E.four[t]), E.Hd + HS * t);
    if (lane == 0) ewald_finish<double, double>(D, X);
}

/* FP64: CC Ewald lists shorter than this are evaluated one source at a time by
 * the whole warp (green_ewald_warp); longer ones one source per lane */
constexpr int EWALD_WARP_LIST = 12;

struct ListView {
    int32_t *pool[NLIST];
    int64_t *off[NLIST];
    int32_t *len[NLIST];
};

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

/* ---- node kernel: CC / CP direct -> Lloc ---- */
template <class T>
__global__ void __launch_bounds__(128) k_node(GParams P, int64_t nn, const int32_t *__restrict__ pb,
                                              const int32_t *__restrict__ pe, const MSrc *__restrict__ ms,
                                              const int4 *__restrict__ pos, ListView LV, double *__restrict__ Lloc) {
    const int lane = threadIdx.x & 31;
    const int64_t warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < nn; i += warps) {
        if (pe[i] == pb[i]) continue;
        const int32_t X[3] = {ms[i].x[0], ms[i].x[1], ms[i].x[2]};
        const bool per = P.ewald != 0;
        T L[LP];
#pragma unroll
        for (int k = 0; k < LP; k++) L[k] = T(0);
        /* CC direct (src/gravity.cpp:368-426) */
        {
            const int32_t *lst = LV.pool[TG_CC_D] + LV.off[TG_CC_D][i];
            const int32_t len = LV.len[TG_CC_D][i];
            for (int32_t j = lane; j < len; j += 32) {
                const MSrc &s = ms[lst[j]];
                T dX[3], D[LP], M[MP];
#pragma unroll
                for (int d = 0; d < 3; d++) dX[d] = sep<T>(X[d], s.x[d], per);
#pragma unroll
                for (int q = 0; q < MP; q++) M[q] = T(s.m[q]);
                green_direct<T>(dX, D);
                contract_M2L<T, T>(L, M, D);
            }
        }
        /* CP direct (src/gravity.cpp:428-486) */
        {
            const int32_t *lst = LV.pool[TG_CP_D] + LV.off[TG_CP_D][i];
            const int32_t len = LV.len[TG_CP_D][i];
            const T m = T(P.m_d);
            for (int32_t c = 0; c < len; c++) {
                const int32_t src = lst[c];
                for (int32_t q = pb[src] + lane; q < pe[src]; q += 32) {
                    const int4 y = pos[q];
                    const int32_t yy[3] = {y.x, y.y, y.z};
                    T dX[3], D[LP];
#pragma unroll
                    for (int d = 0; d < 3; d++) dX[d] = sep<T>(X[d], yy[d], per);
                    green_direct<T>(dX, D);
                    contract_P2L<T, T>(L, m, D);
                }
            }
        }
#pragma unroll
        for (int k = 0; k < LP; k++) {
            const double v = warp_sum((double)L[k]);
            if (lane == 0) Lloc[35 * i + k] = v;
        }
    }
}

#include "tg_ewald_table.cuh"
#include "tg_ewald_node.cuh"

/* ---- L2L, one level ---- */
__global__ void k_l2l(int64_t first, int64_t count, const int32_t *__restrict__ pb, const int32_t *__restrict__ pe,
                      const int32_t *__restrict__ parent, const MSrc *__restrict__ ms, const double *__restrict__ Lloc,
                      double *__restrict__ Lout) {
    const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= count) return;
    const int64_t i = first + k;
    if (pe[i] == pb[i]) return;
    double L[LP];
    double Lcom[3] = {0.5, 0.5, 0.5};
    const int32_t p = parent[i];
    if (p >= 0) {
#pragma unroll
        for (int q = 0; q < LP; q++) L[q] = Lout[35 * (int64_t)p + q];
        for (int d = 0; d < 3; d++) Lcom[d] = pos2d(ms[p].x[d]);
    } else {
#pragma unroll
        for (int q = 0; q < LP; q++) L[q] = 0.0;
    }
    double dx[3];
    for (int d = 0; d < 3; d++) dx[d] = __dadd_rn(pos2d(ms[i].x[d]), -Lcom[d]);
    L2L(L, dx);
#pragma unroll
    for (int q = 0; q < LP; q++) Lout[35 * i + q] = L[q] + Lloc[35 * i + q];
}

/* ---- leaf kernel ---- */
template <class T, int BLOCK, bool PP = true, bool EW = true>
__global__ void __launch_bounds__(BLOCK) k_leaf(GParams P, const int32_t *__restrict__ leaves, int32_t nleaves,
                                                const int32_t *__restrict__ pb, const int32_t *__restrict__ pe,
                                                const MSrc *__restrict__ ms, const int4 *__restrict__ pos, ListView LV,
                                                EwaldTables E, const double *__restrict__ Lnode,
                                                float4 *__restrict__ acc_f, double *__restrict__ acc_d) {
    __shared__ int4 sy[BLOCK];
    __shared__ double sL[LP];
    const int tid = threadIdx.x;
    for (int32_t li = blockIdx.x; li < nleaves; li += gridDim.x) {
        const int32_t leaf = leaves[li];
        const int32_t b = pb[leaf], cnt = pe[leaf] - b;
        const bool active = tid < cnt;
        const int4 xi4 = pos[b + (active ? tid : 0)];
        const int32_t xi[3] = {xi4.x, xi4.y, xi4.z};
        const bool per = P.ewald != 0;
        __syncthreads();
        if (tid < LP) sL[tid] = Lnode[35 * (int64_t)leaf + tid];
        __syncthreads();
        /* L2P (tigergrav/expansion.hpp:235-269; dX through float, src/tree.cpp:607) */
        Acc<T> aphi, ag[3];
        {
            double dx[3], ph, g[3];
            for (int d = 0; d < 3; d++)
                dx[d] = (double)__double2float_rn(__dadd_rn(pos2d(xi[d]), -pos2d(ms[leaf].x[d])));
            L2P<double>(sL, dx, ph, g);
            aphi.init(ph);
            for (int d = 0; d < 3; d++) ag[d].init(g[d]);
        }
        /* PC direct (src/gravity.cpp:302-366) */
        {
            const int32_t *lst = LV.pool[TG_PC_D] + LV.off[TG_PC_D][leaf];
            const int32_t len = LV.len[TG_PC_D][leaf];
            for (int32_t j = 0; j < len; j++) {
                const MSrc &s = ms[lst[j]];
                T dX[3], D[LP], M[MP];
#pragma unroll
                for (int d = 0; d < 3; d++) dX[d] = sep<T>(xi[d], s.x[d], per);
#pragma unroll
                for (int q = 0; q < MP; q++) M[q] = T(s.m[q]);
                green_direct<T>(dX, D);
                T ph, g[3];
                contract_M2P<T>(ph, g, M, D);
                aphi.add(ph);
                for (int d = 0; d < 3; d++) ag[d].add(g[d]);
            }
        }
        /* PP direct (src/gravity.cpp:171-300) */
        if (PP) {
            const int32_t *lst = LV.pool[TG_PP_D] + LV.off[TG_PP_D][leaf];
            const int32_t len = LV.len[TG_PP_D][leaf];
            const T m = T(P.m_d);
            for (int32_t c = 0; c < len; c++) {
                const int32_t src = lst[c];
                const int32_t sb = pb[src], sn = pe[src] - sb;
                for (int32_t base = 0; base < sn; base += BLOCK) {
                    const int32_t nt = min(BLOCK, sn - base);
                    __syncthreads();
                    if (tid < nt) sy[tid] = pos[sb + base + tid];
                    __syncthreads();
                    /* plain sums over groups of 8 pairs, folded into the compensated totals */
                    for (int32_t q0 = 0; q0 < nt; q0 += 8) {
                        T tp = T(0), tg0 = T(0), tg1 = T(0), tg2 = T(0);
                        const int32_t q1 = min(nt, q0 + 8);
                        for (int32_t q = q0; q < q1; q++) {
                            const int4 y = sy[q];
                            T dX[3] = {sep<T>(xi[0], y.x, per), sep<T>(xi[1], y.y, per), sep<T>(xi[2], y.z, per)};
                            T f, p;
                            pp_direct_pair<T>(P, dX, f, p);
                            tp += p;
                            tg0 += dX[0] * f;
                            tg1 += dX[1] * f;
                            tg2 += dX[2] * f;
                        }
                        aphi.add(-m * tp);
                        ag[0].add(-m * tg0);
                        ag[1].add(-m * tg1);
                        ag[2].add(-m * tg2);
                    }
                }
            }
        }
        if (EW && per) {
            /* PC Ewald (src/gravity.cpp:616-678) */
            const int32_t *lst = LV.pool[TG_PC_E] + LV.off[TG_PC_E][leaf];
            const int32_t len = LV.len[TG_PC_E][leaf];
            for (int32_t j = 0; j < len; j++) {
                const MSrc &s = ms[lst[j]];
                T dX[3], D[LP], M[MP];
#pragma unroll
                for (int d = 0; d < 3; d++) dX[d] = sep<T>(xi[d], s.x[d], true);
#pragma unroll
                for (int q = 0; q < MP; q++) M[q] = T(s.m[q]);
                green_ewald_full<T>(E, dX, D);
                T ph, g[3];
                contract_M2P<T>(ph, g, M, D);
                aphi.add(ph);
                for (int d = 0; d < 3; d++) ag[d].add(g[d]);
            }
            /* PP Ewald (src/gravity.cpp:491-614) */
            const int32_t *lpp = LV.pool[TG_PP_E] + LV.off[TG_PP_E][leaf];
            const int32_t npp = LV.len[TG_PP_E][leaf];
            const T m = T(P.m_d);
            for (int32_t c = 0; c < npp; c++) {
                const int32_t src = lpp[c];
                const int32_t sb = pb[src], sn = pe[src] - sb;
                for (int32_t base = 0; base < sn; base += BLOCK) {
                    const int32_t nt = min(BLOCK, sn - base);
                    __syncthreads();
                    if (tid < nt) sy[tid] = pos[sb + base + tid];
                    __syncthreads();
                    for (int32_t q = 0; q < nt; q++) {
                        const int4 y = sy[q];
                        T dX[3] = {wrap_sep_t<T>(xi[0], y.x), wrap_sep_t<T>(xi[1], y.y), wrap_sep_t<T>(xi[2], y.z)};
                        T ph, g[3];
                        pp_ewald_pair<T>(E, dX, ph, g);
                        aphi.add(m * ph);
                        for (int d = 0; d < 3; d++) ag[d].add(m * g[d]);
                    }
                }
            }
        }
        if (active) {
            const double phi = aphi.get() - (PP ? P.phi_self : 0.0);
            if (acc_f) acc_f[b + tid] = make_float4((float)phi, (float)ag[0].get(), (float)ag[1].get(), (float)ag[2].get());
            if (acc_d) {
                acc_d[4 * (int64_t)(b + tid) + 0] = phi;
                for (int d = 0; d < 3; d++) acc_d[4 * (int64_t)(b + tid) + 1 + d] = ag[d].get();
            }
        }
    }
}

/* offset of Y from Xr: int32 wrap (periodic) or plain difference (free space);
 * mag accumulates the largest magnitude, saturated at 2^31 (a free-space
 * offset that does not fit an int32 reads as 2^31) */
__device__ __forceinline__ int32_t rel_off(int32_t Y, int32_t Xr, bool per, uint32_t &mag) {
    if (per) {
        const int32_t a = (int32_t)((uint32_t)Y - (uint32_t)Xr);
        mag = max(mag, a < 0 ? 0u - (uint32_t)a : (uint32_t)a);
        return a;
    }
    const long long a = (long long)Y - (long long)Xr;
    const unsigned long long aa = (unsigned long long)(a < 0 ? -a : a);
    mag = max(mag, aa >= (1ull << 31) ? (1u << 31) : (uint32_t)aa);
    return (int32_t)a;
}

#include "tg_pp.cuh"
#include "tg_pp2.cuh"
#include "tg_ewald_sep.cuh"
#include "tg_ewald_leaf.cuh"

/* ---------------- kernel-level seams ---------------- */

/* PP seams: one block per sink group.  A pass takes up to SEAM_T sinks, ns of
 * them, in C = SEAM_T / ns copies (thread t: sink t % ns, copy t / ns); the
 * sources are staged SEAM_T at a time and copy p takes every C-th of a stage.
 * All sums are FP64, the copies added in order; in FP32 the pair's factors are
 * converted and multiplied by the separation's exact value, so a direct pair takes
 * two conversions.  4096 groups of 64 sinks and 2048 sources, direct: 2.13 ms with a
 * thread per sink, sources read from global memory and four float-to-double
 * conversions per pair, 1.38 ms now (compensated FP32 sums: 1.68). */
constexpr int SEAM_T = 128;
template <class T, bool EWALD>
__global__ void __launch_bounds__(SEAM_T) k_seam_pp(GParams P, int do_phi, int64_t ngroups,
                                                    const int64_t *__restrict__ sink_off,
                                                    const int32_t *__restrict__ sink_x,
                                                    const int64_t *__restrict__ src_off,
                                                    const int32_t *__restrict__ src_x, EwaldTables E,
                                                    double *__restrict__ f) {
    __shared__ int32_t sy[SEAM_T][3];
    __shared__ double red[SEAM_T][4];
    const int t = threadIdx.x;
    const bool per = P.ewald != 0;
    for (int64_t g = blockIdx.x; g < ngroups; g += gridDim.x) {
        const int64_t i1 = sink_off[g + 1], j0 = src_off[g], j1 = src_off[g + 1];
        for (int64_t i0 = sink_off[g]; i0 < i1; i0 += SEAM_T) {
            const int ns = (int)min((int64_t)SEAM_T, i1 - i0);
            const int C = SEAM_T / ns, phase = t / ns;
            const int64_t i = i0 + t % ns;
            const int32_t xi[3] = {sink_x[3 * i], sink_x[3 * i + 1], sink_x[3 * i + 2]};
            double o[4] = {0.0, 0.0, 0.0, 0.0};
            for (int64_t jb = j0; jb < j1; jb += SEAM_T) {
                const int nt = (int)min((int64_t)SEAM_T, j1 - jb);
                __syncthreads();
                for (int q = t; q < 3 * nt; q += SEAM_T) (&sy[0][0])[q] = src_x[3 * jb + q];
                __syncthreads();
                if (phase < C)
                    for (int q = phase; q < nt; q += C) {
                        const int32_t *y = sy[q];
                        if (EWALD) {
                            const T dX[3] = {wrap_sep_t<T>(xi[0], y[0]), wrap_sep_t<T>(xi[1], y[1]),
                                             wrap_sep_t<T>(xi[2], y[2])};
                            T p, g3[3];
                            pp_ewald_pair<T>(E, dX, p, g3);
                            o[0] += (double)p;
#pragma unroll
                            for (int d = 0; d < 3; d++) o[1 + d] += (double)g3[d];
                        } else {
                            const T dX[3] = {sep<T>(xi[0], y[0], per), sep<T>(xi[1], y[1], per),
                                             sep<T>(xi[2], y[2], per)};
                            T fk, p;
                            pp_direct_pair<T>(P, dX, fk, p);
                            o[0] -= (double)p;
#pragma unroll
                            for (int d = 0; d < 3; d++) {
                                const double x = sizeof(T) == 8 ? (double)dX[d]
                                                 : per ? i2d((int32_t)((uint32_t)xi[d] - (uint32_t)y[d]))
                                                       : i2d(xi[d]) - i2d(y[d]);
                                o[1 + d] = fma(-x, (double)fk, o[1 + d]);
                            }
                        }
                    }
            }
#pragma unroll
            for (int d = 0; d < 4; d++) red[t][d] = o[d];
            __syncthreads();
            if (t < ns) {
                double v[4] = {0.0, 0.0, 0.0, 0.0};
                for (int p = 0; p < C; p++)
#pragma unroll
                    for (int d = 0; d < 4; d++) v[d] += red[t + p * ns][d];
                if (EWALD || do_phi) f[4 * i] += P.m_d * v[0] - (EWALD ? 0.0 : P.phi_self);
                else f[4 * i] -= P.phi_self;
#pragma unroll
                for (int d = 0; d < 3; d++)
                    f[4 * i + 1 + d] += P.m_d * (EWALD || sizeof(T) == 8 ? v[1 + d] : v[1 + d] * POS_INV);
            }
            __syncthreads(); /* red is rewritten next */
        }
    }
}

template <class T>
__global__ void k_seam_pc(GParams P, int kind_ewald, int64_t ngroups, const int64_t *__restrict__ sink_off,
                          const int32_t *__restrict__ sink_x, const int64_t *__restrict__ src_off,
                          const float *__restrict__ src_m, const int32_t *__restrict__ src_x, EwaldTables E,
                          double *__restrict__ f) {
    const bool per = kind_ewald || P.ewald != 0;
    for (int64_t g = blockIdx.x; g < ngroups; g += gridDim.x) {
        for (int64_t i = sink_off[g] + threadIdx.x; i < sink_off[g + 1]; i += blockDim.x) {
            const int32_t xi[3] = {sink_x[3 * i], sink_x[3 * i + 1], sink_x[3 * i + 2]};
            double ph = 0, gg[3] = {0, 0, 0};
            for (int64_t j = src_off[g]; j < src_off[g + 1]; j++) {
                T dX[3], D[LP], M[MP];
                for (int d = 0; d < 3; d++) dX[d] = sep<T>(xi[d], src_x[3 * j + d], per);
                for (int q = 0; q < MP; q++) M[q] = T(src_m[MP * j + q]);
                if (kind_ewald) green_ewald_full<T>(E, dX, D);
                else green_direct<T>(dX, D);
                T p, g3[3];
                contract_M2P<T>(p, g3, M, D);
                ph += (double)p;
                for (int d = 0; d < 3; d++) gg[d] += (double)g3[d];
            }
            f[4 * i] += ph;
            for (int d = 0; d < 3; d++) f[4 * i + 1 + d] += gg[d];
        }
    }
}

/* CC/CP seams: one warp per group, lanes over sources */
template <class T>
__global__ void k_seam_node(GParams P, int kind_ewald, int is_cc, int64_t ngroups, const int32_t *__restrict__ sink_x,
                            const int64_t *__restrict__ src_off, const float *__restrict__ src_m,
                            const int32_t *__restrict__ src_x, EwaldTables E, double *__restrict__ Lout) {
    const int lane = threadIdx.x & 31;
    const int64_t warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const bool per = kind_ewald || P.ewald != 0;
    for (int64_t g = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; g < ngroups; g += warps) {
        const int32_t X[3] = {sink_x[3 * g], sink_x[3 * g + 1], sink_x[3 * g + 2]};
        T L[LP];
        for (int k = 0; k < LP; k++) L[k] = T(0);
        const int64_t b = src_off[g], e = src_off[g + 1];
        for (int64_t j = b + lane; j < e; j += 32) {
            T dX[3], D[LP];
            for (int d = 0; d < 3; d++) dX[d] = sep<T>(X[d], src_x[3 * j + d], per);
            if (kind_ewald) green_ewald_full<T>(E, dX, D);
            else green_direct<T>(dX, D);
            if (is_cc) {
                T M[MP];
                for (int q = 0; q < MP; q++) M[q] = T(src_m[MP * j + q]);
                contract_M2L<T, T>(L, M, D);
            } else {
                contract_P2L<T, T>(L, T(P.m_d), D);
            }
        }
        for (int k = 0; k < LP; k++) {
            const double v = warp_sum((double)L[k]);
            if (lane == 0) Lout[35 * g + k] += v;
        }
    }
}

static EwaldTables tables(Solver &S) {
    return EwaldTables{S.ew_real.p,  S.ew_four.p, S.ew_Hf.p,  S.ew_Hd.p,  S.ew_Pf.p, S.ew_Pd.p,
                       S.ew_sep_h.p, S.ew_sep_run.p, S.ew_sep_nrun, S.ew_sep_w.p, S.ew_sep_k, S.ew_sep_r0, S.ew_sep_r2, S.ew_tab};
}

static ListView listview(Solver &S) {
    ListView LV;
    for (int k = 0; k < NLIST; k++) {
        LV.pool[k] = S.pool[k].p;
        LV.off[k] = S.loff[k].p;
        LV.len[k] = S.llen[k].p;
    }
    return LV;
}

/* the node Ewald lists (CC_E, CP_E) of every node, in balanced chunks, added
 * to Lloc */
static int node_ewald(Solver &S, const GParams &P, const ListView &LV, const EwaldTables &E, bool f64,
                      cudaStream_t st) {
    const int64_t nn = S.nnodes;
    TG_TRY(ensure(S.ew_cnt, (size_t)nn + 1));
    TG_TRY(ensure(S.ew_off, (size_t)nn + 1));
    k_node_ewald_count<<<(int)((nn + 1 + 127) / 128), 128, 0, st>>>(nn, S.nd_pb.p, S.nd_pe.p, LV, S.ew_cnt.p);
    TG_TRY(launched(S));
    size_t stmp = 0;
    TG_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, stmp, S.ew_cnt.p, S.ew_off.p, (int)(nn + 1), st));
    TG_TRY(ensure(S.cub_tmp, stmp));
    TG_CUDA(cub::DeviceScan::ExclusiveSum(S.cub_tmp.p, stmp, S.ew_cnt.p, S.ew_off.p, (int)(nn + 1), st));
    int32_t total = 0;
    TG_TRY(read_small(S, st, &total, S.ew_off.p + nn, sizeof(int32_t)));
    if (total <= 0) return TG_OK;
    TG_TRY(ensure(S.ew_part, (size_t)total * LP));
    const int g = (int)(((int64_t)total * 32 + 127) / 128);
    if (f64)
        k_node_ewald<double><<<g, 128, 0, st>>>(P, nn, total, S.ew_off.p, S.nd_pb.p, S.nd_pe.p, S.nd_ms.p, S.pos.p, LV,
                                                E, S.ew_part.p);
    else
        k_node_ewald<float><<<g, 128, 0, st>>>(P, nn, total, S.ew_off.p, S.nd_pb.p, S.nd_pe.p, S.nd_ms.p, S.pos.p, LV,
                                               E, S.ew_part.p);
    TG_TRY(launched(S));
    k_node_ewald_reduce<<<(int)((nn * LP + 255) / 256), 256, 0, st>>>(nn, S.ew_off.p, S.ew_part.p, S.nd_Lloc.p);
    TG_TRY(launched(S));
    return TG_OK;
}

/* leaves of the tree (the empty ones too) */
static int64_t tree_leaves(const Solver &S) {
    int64_t n = 0;
    for (int64_t l : S.level_leaves) n += l;
    return n;
}

/* The leaf Ewald lists cut into chunks (tg_ewald_leaf.cuh): their offsets in
 * ew_off, the PP_E source leaves in ew_src with their rows in ew_slot, and the
 * numbers of PP_E chunks, of all chunks and of source leaves. */
static int leaf_chunks(Solver &S, const ListView &LV, int32_t &npp, int32_t &total, int32_t &nsrc, cudaStream_t st) {
    const int32_t nleaves = (int32_t)S.st.leaves;
    const int64_t nn = S.nnodes;
    const size_t nc = 2 * ((size_t)nleaves + 1);
    TG_TRY(ensure(S.ew_cnt, nc));
    TG_TRY(ensure(S.ew_off, nc + 1));
    TG_TRY(ensure(S.ew_slot, (size_t)nn));
    TG_TRY(ensure(S.ew_src, (size_t)nn));
    int32_t *slot = S.ew_slot.p, *nsrc_d = S.ew_off.p + nc; /* the source count sits behind the scan: one readback */
    TG_CUDA(cudaMemsetAsync(slot, 0xff, sizeof(int32_t) * nn, st));
    TG_CUDA(cudaMemsetAsync(nsrc_d, 0, sizeof(int32_t), st));
    k_ewald_count<<<(int)(((int64_t)(nleaves + 1) * 32 + 127) / 128), 128, 0, st>>>(S.idx.p, nleaves, LV, S.ew_cnt.p,
                                                                                  slot);
    TG_TRY(launched(S));
    k_ewald_slots<<<(int)((nn + 255) / 256), 256, 0, st>>>(nn, slot, S.ew_src.p, nsrc_d);
    TG_TRY(launched(S));
    size_t stmp = 0;
    TG_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, stmp, S.ew_cnt.p, S.ew_off.p, (int)nc, st));
    TG_TRY(ensure(S.cub_tmp, stmp));
    TG_CUDA(cub::DeviceScan::ExclusiveSum(S.cub_tmp.p, stmp, S.ew_cnt.p, S.ew_off.p, (int)nc, st));
    /* off[nleaves]: PP_E chunks; off[nc - 1]: all chunks; then the PP_E source leaves */
    TG_CUDA(cudaMemcpyAsync(S.h_small + 2048, S.ew_off.p + nleaves, sizeof(int32_t), cudaMemcpyDeviceToHost, st));
    TG_CUDA(cudaMemcpyAsync(S.h_small + 2052, S.ew_off.p + nc - 1, 2 * sizeof(int32_t), cudaMemcpyDeviceToHost, st));
    TG_CUDA(cudaStreamSynchronize(st));
    int32_t tot[3];
    std::memcpy(tot, S.h_small + 2048, sizeof(tot));
    npp = tot[0], total = tot[1], nsrc = tot[2];
    S.ew_max_npp = std::max(S.ew_max_npp, npp);
    S.ew_max_nsrc = std::max(S.ew_max_nsrc, nsrc);
    return TG_OK;
}

/* The leaves in batches whose chunks fit the scratch: pp and pc bytes per PP_E and
 * PC_E chunk.  All of them in one where they fit, else from the chunk offsets. */
static int leaf_batches(Solver &S, int32_t npp, int32_t total, size_t pp, size_t pc, std::vector<EwBatch> &out,
                        cudaStream_t st) {
    const int32_t nleaves = (int32_t)S.st.leaves;
    out.clear();
    if ((size_t)npp * pp + (size_t)(total - npp) * pc <= S.ew_scratch()) {
        out.push_back({0, nleaves, 0, npp, npp, total - npp});
        return TG_OK;
    }
    const size_t noff = 2 * ((size_t)nleaves + 1);
    std::unique_ptr<int32_t[]> off(new (std::nothrow) int32_t[noff]);
    if (!off) return TG_ERR_NOMEM;
    TG_CUDA(cudaMemcpyAsync(off.get(), S.ew_off.p, noff * sizeof(int32_t), cudaMemcpyDeviceToHost, st));
    TG_CUDA(cudaStreamSynchronize(st));
    const int32_t *offp = off.get() + nleaves + 1;
    for (int32_t l0 = 0, l1; l0 < nleaves; l0 = l1) {
        for (l1 = l0 + 1; l1 < nleaves; l1++) /* at least one leaf */
            if ((size_t)(off[l1 + 1] - off[l0]) * pp + (size_t)(offp[l1 + 1] - offp[l0]) * pc > S.ew_scratch()) break;
        out.push_back({l0, l1, off[l0], off[l1] - off[l0], offp[l0], offp[l1] - offp[l0]});
    }
    return TG_OK;
}
/* vectors whose source sums (nsrc rows, `bytes` each) are held at a time, of N */
static int ew_vectors(const Solver &S, int32_t nsrc, size_t bytes, int N) {
    const size_t n = S.ew_scratch() / (std::max(nsrc, 1) * bytes);
    return n >= (size_t)N ? N : std::max(1, (int)n);
}

/* the leaf Ewald lists (PP_E, PC_E) of every leaf, in balanced chunks, added
 * to the FP64 accumulators accd (leaf_max <= 64) */
template <class T>
static int leaf_ewald(Solver &S, const GParams &P, const ListView &LV, const EwaldTables &E, cudaStream_t st) {
    constexpr int N = Sep<T>::N;
    const int32_t nleaves = (int32_t)S.st.leaves;
    int32_t npp = 0, total = 0, nsrc = 0;
    TG_TRY(leaf_chunks(S, LV, npp, total, nsrc, st));
    if (total <= 0) return TG_OK;
    std::vector<EwBatch> batches;
    TG_TRY(leaf_batches(S, npp, total, (256 * sizeof(double)) + N * sizeof(double2), 256 * sizeof(double), batches, st));
    size_t slots = 0, sums = 0;
    for (const EwBatch &B : batches) {
        slots = std::max(slots, (size_t)B.na + B.nc);
        sums = std::max(sums, (size_t)B.na);
    }
    const int nv = ew_vectors(S, nsrc, sizeof(double2), N);
    TG_TRY(ensure(S.ew_part, slots * 64 * 4));
    if (npp > 0) {
        TG_TRY(ensure(S.ew_sf, (size_t)nsrc * nv * sizeof(double2)));
        TG_TRY(ensure(S.ew_tpart, sums * N * sizeof(double2)));
    }
    double2 *sf = reinterpret_cast<double2 *>(S.ew_sf.p), *tpart = reinterpret_cast<double2 *>(S.ew_tpart.p);
    const int32_t *offp = S.ew_off.p + nleaves + 1;
    if (npp > 0 && nv == N) {
        k_ewald_sf<T><<<nsrc, 128, 0, st>>>(S.ew_src.p, S.nd_pb.p, S.nd_pe.p, S.pos.p, E, 0, N, sf);
        TG_TRY(launched(S));
    }
    for (const EwBatch &B : batches) {
        if (B.na > 0) {
            k_ewald_pp<T><<<B.na, 64, 0, st>>>(P, S.idx.p, nleaves, B.a0, S.ew_off.p, S.nd_pb.p, S.nd_pe.p, S.pos.p,
                                               LV, E, S.ew_near, S.ew_part.p, S.ew_slot.p, nv == N ? sf : nullptr, tpart);
            TG_TRY(launched(S));
        }
        for (int t0 = 0; B.na > 0 && nv < N && t0 < N; t0 += nv) {
            const int t1 = std::min(N, t0 + nv);
            k_ewald_sf<T><<<nsrc, 128, 0, st>>>(S.ew_src.p, S.nd_pb.p, S.nd_pe.p, S.pos.p, E, t0, t1, sf);
            TG_TRY(launched(S));
            k_ewald_tsum<double2><<<B.na, 64, 0, st>>>(N, P.m_d, S.idx.p, nleaves, B.a0, S.ew_off.p, LV, S.ew_slot.p,
                                                       t0, t1, sf, tpart);
            TG_TRY(launched(S));
        }
        if (B.nc > 0) {
            k_ewald_pc<T><<<B.nc, 64, 0, st>>>(S.idx.p, nleaves, B.c0, B.na, offp, S.nd_pb.p, S.nd_pe.p, S.nd_ms.p,
                                               S.pos.p, LV, E, S.ew_part.p);
            TG_TRY(launched(S));
        }
        k_ewald_reduce<T><<<B.l1 - B.l0, 256, 0, st>>>(B, S.idx.p, nleaves, S.ew_off.p, S.nd_pb.p, S.nd_pe.p, S.ew_part.p,
                                                       S.accd.p, tpart, S.pos.p, E);
        TG_TRY(launched(S));
    }
    return TG_OK;
}

/* the node stage: CC/CP (direct, then Ewald) into Lloc, then L2L top-down into nd_L */
static int node_stage(Solver &S, const GParams &P, const ListView &LV, const EwaldTables &E, cudaStream_t st) {
    const int64_t nn = S.nnodes;
    const bool f64 = S.prm.precision == TG_PREC_F64;
    TG_TRY(ensure(S.nd_Lloc, 35 * nn));
    TG_TRY(ensure(S.nd_L, 35 * nn));
    {
        const int TPB = 128;
        const int64_t want = (nn * 32 + TPB - 1) / TPB;
        const int g = (int)(want < 65535 * 8 ? want : 65535 * 8);
        if (f64)
            k_node<double><<<g, TPB, 0, st>>>(P, nn, S.nd_pb.p, S.nd_pe.p, S.nd_ms.p, S.pos.p, LV, S.nd_Lloc.p);
        else
            k_node<float><<<g, TPB, 0, st>>>(P, nn, S.nd_pb.p, S.nd_pe.p, S.nd_ms.p, S.pos.p, LV, S.nd_Lloc.p);
        TG_TRY(launched(S));
    }
    if (S.prm.ewald) TG_TRY(node_ewald(S, P, LV, E, f64, st));
    for (int L = 0; L <= S.depth; L++) {
        const int64_t first = S.level_off[L], count = S.level_off[L + 1] - S.level_off[L];
        if (count <= 0) continue;
        const int g = (int)((count + 127) / 128);
        k_l2l<<<g, 128, 0, st>>>(first, count, S.nd_pb.p, S.nd_pe.p, S.nd_parent.p, S.nd_ms.p, S.nd_Lloc.p, S.nd_L.p);
        TG_TRY(launched(S));
    }
    return TG_OK;
}

/* PP direct of the FP32 path (leaf_max <= 64): far + PP_direct - phi_self into acc.
 * A list holds about 17 / theta^3 source leaves (leaves within (r_a + r_b) / theta,
 * at most all of them).
 *
 * From PPB_LONG on k_pp_long (whole leaves per warp) is the faster one of the two.
 * ms with k_pp_short / k_pp_long by that length:
 *   128^3 clustered, leaf 64   50: 4.08 / 4.57   266: 20.8 / 23.1   397: 29.4 / 32.2
 *                             630: 40.4 / 40.4   967: 55.3 / 52.5  2125: 107 / 98
 *   101^3 clustered, leaf 32  397: 7.56 / 8.74   864: 13.0 / 13.1  1597: 21.3 / 20.4
 *   101^3 uniform, leaf 48    266: 7.89 / 8.85   630: 16.9 / 18.2  1230: 27.1 / 25.7
 *   64^3 clustered, leaf 64   397: 4.18 / 4.48   774: 6.81 / 6.47
 *   64^3 clustered, leaf 16   397: 1.60 / 1.73   774: 2.67 / 2.70  1597: 4.99 / 4.71
 *   64^3 halos (free), leaf 32  266: 1.65 / 1.78  630: 2.84 / 2.93  1088: 4.06 / 3.94
 * and 256^3, leaf 48, 2480: 731 / 662 (703 in quarters).
 *
 * A list of at least 1 / PPB_WIDE of the tree's leaves reaches half a box, where
 * k_pp_short takes whole stages pair by pair; below PPB_LONG k_pp_long in quarters
 * of leaves takes those.  ms with k_pp_short / k_pp_long in quarters by the share:
 *   leaf 64, uniform   0.54: 0.165 / 0.052 (4096)     0.17: 0.581 / 0.108 (14000)
 *     0.13: 2.43 / 2.23 (1e5)  0.10: 0.325 / 0.087 (20000)  0.07: 0.122 / 0.124 (32768)
 *     0.06: 2.44 / 2.48 (2e5)  0.05: 0.208 / 0.220 (50000)  0.03: 1.26 / 1.27 (2e5)
 *   leaf 32, clustered 0.22: 0.458 / 0.112  0.09: 0.243 / 0.220  0.05: 0.302 / 0.312
 *   leaf 16, uniform   0.13: 0.400 / 0.151  0.07: 0.063 / 0.040  0.05: 0.218 / 0.243
 *   leaf 32, halos (free)  0.12: 0.355 / 0.083  0.06: 0.435 / 0.112  0.05: 1.32 / 0.79
 *                          0.03: 0.189 / 0.196
 *
 * Fewer leaves than one wave of blocks: the lists are cut into shares so that the
 * wave is full (4096 uniform: 0.79 ms without).  The choices depend on the tree alone,
 * not on which leaves are active, so a rung step's forces equal a full solve's bit
 * for bit. */
constexpr int PPB_LONG = 800, PPB_WIDE = 20;
static int pp_direct(Solver &S, const GParams &P, const ListView &LV, cudaStream_t st) {
    const int64_t n = S.n, nn = S.nnodes;
    const int32_t nleaves = (int32_t)S.st.leaves;
    TG_TRY(ensure(S.pp_rec, 2 * (size_t)nn));
    PPRec *rec = reinterpret_cast<PPRec *>(S.pp_rec.p);
    k_pp_records<<<(int)((nn + 255) / 256), 256, 0, st>>>(nn, S.nd_pb.p, S.nd_pe.p, S.nd_child0.p, S.nd_aabb.p, rec);
    TG_TRY(launched(S));
    const int64_t tree = tree_leaves(S);
    const double list = std::min(17.0 / (S.prm.theta * S.prm.theta * S.prm.theta), (double)tree);
    const bool whole = list >= PPB_LONG, quarter = !whole && list * PPB_WIDE >= (double)tree, longl = whole || quarter;
    const int wave = S.num_sms * (longl ? PPL_MINB : PPS_MINB);
    const int shares = tree >= wave ? 1 : (int)std::min<int64_t>((wave + tree - 1) / tree, PPB_SHARES);
    double *part = nullptr;
    if (shares > 1) {
        TG_TRY(ensure(S.pp_part, (size_t)shares * 4 * n));
        part = S.pp_part.p;
    }
    const dim3 g(nleaves, shares);
    if (quarter)
        k_pp_long<true><<<g, PPB_T, 0, st>>>(P, S.idx.p, S.nd_pb.p, S.nd_pe.p, S.nd_ms.p, rec, S.pos.p, LV, S.accd.p,
                                             S.acc.p, part, n);
    else if (longl)
        k_pp_long<false><<<g, PPB_T, 0, st>>>(P, S.idx.p, S.nd_pb.p, S.nd_pe.p, S.nd_ms.p, rec, S.pos.p, LV, S.accd.p,
                                              S.acc.p, part, n);
    else
        k_pp_short<<<g, PPB_T, 0, st>>>(P, S.idx.p, S.nd_pb.p, S.nd_pe.p, S.nd_ms.p, rec, S.pos.p, LV, S.accd.p,
                                        S.acc.p, part, n);
    TG_TRY(launched(S));
    if (shares > 1) {
        k_pp_reduce<<<nleaves, 64, 0, st>>>(P, S.idx.p, S.nd_pb.p, S.nd_pe.p, S.accd.p, part, shares, n, S.acc.p);
        TG_TRY(launched(S));
    }
    return TG_OK;
}

int gravity_forces(Solver &S, cudaStream_t st) {
    if (!S.have_lists) return TG_ERR_STATE;
    TG_TRY(ewald_tables(S, st));
    const int64_t n = S.n;
    const GParams P = make_gparams(S.prm);
    const EwaldTables E = tables(S);
    const ListView LV = listview(S);
    const bool f64 = S.prm.precision == TG_PREC_F64;
    const bool split_pp = !f64 && S.prm.leaf_max <= 64;
    if (f64 || split_pp) TG_TRY(ensure(S.accd, 4 * n));
    if (!f64) TG_TRY(ensure(S.acc, n));
    S.pp_timed = false;
    if (S.have_events) TG_CUDA(cudaEventRecord(S.ev[3], st));
    TG_TRY(node_stage(S, P, LV, E, st));
    if (S.have_events) TG_CUDA(cudaEventRecord(S.ev[4], st));
    const int32_t nleaves = (int32_t)S.st.leaves;
    if (nleaves > 0) {
        const int g = nleaves;
        if (S.prm.leaf_max <= 64) {
            /* L2P, PC direct (and for FP64 PP direct) per leaf; the Ewald lists as balanced chunks */
            if (f64)
                k_leaf<double, 64, true, false><<<g, 64, 0, st>>>(P, S.idx.p, nleaves, S.nd_pb.p, S.nd_pe.p, S.nd_ms.p,
                                                                  S.pos.p, LV, E, S.nd_L.p, nullptr, S.accd.p);
            else
                k_leaf<float, 64, false, false><<<g, 64, 0, st>>>(P, S.idx.p, nleaves, S.nd_pb.p, S.nd_pe.p,
                                                                  S.nd_ms.p, S.pos.p, LV, E, S.nd_L.p, nullptr,
                                                                  S.accd.p);
            TG_TRY(launched(S));
            if (S.prm.ewald) TG_TRY(f64 ? leaf_ewald<double>(S, P, LV, E, st) : leaf_ewald<float>(S, P, LV, E, st));
            if (!f64) {
                if (S.have_events) {
                    TG_CUDA(cudaEventRecord(S.ev[6], st));
                    S.pp_timed = true;
                }
                TG_TRY(pp_direct(S, P, LV, st));
            }
        } else {
            if (f64)
                k_leaf<double, 128><<<g, 128, 0, st>>>(P, S.idx.p, nleaves, S.nd_pb.p, S.nd_pe.p, S.nd_ms.p, S.pos.p, LV,
                                                       E, S.nd_L.p, nullptr, S.accd.p);
            else
                k_leaf<float, 128><<<g, 128, 0, st>>>(P, S.idx.p, nleaves, S.nd_pb.p, S.nd_pe.p, S.nd_ms.p, S.pos.p, LV,
                                                      E, S.nd_L.p, S.acc.p, nullptr);
            TG_TRY(launched(S));
        }
    }
    if (S.have_events) TG_CUDA(cudaEventRecord(S.ev[5], st));
    S.have_forces = true;
    return TG_OK;
}

/* seam drivers */
int seam_pp(Solver *Sopt, const tg_params &prm, int ewald_kind, int do_phi, int64_t ngroups, const int64_t *sink_off,
            const int32_t *sink_x, const int64_t *src_off, const int32_t *src_x, double *f, const EwaldTables &E,
            cudaStream_t st) {
    const GParams P = make_gparams(prm);
    const int g = (int)(ngroups < 65535 ? ngroups : 65535);
    if (g <= 0) return TG_OK;
    if (prm.precision == TG_PREC_F64) {
        if (ewald_kind)
            k_seam_pp<double, true><<<g, SEAM_T, 0, st>>>(P, do_phi, ngroups, sink_off, sink_x, src_off, src_x, E, f);
        else
            k_seam_pp<double, false><<<g, SEAM_T, 0, st>>>(P, do_phi, ngroups, sink_off, sink_x, src_off, src_x, E, f);
    } else {
        if (ewald_kind)
            k_seam_pp<float, true><<<g, SEAM_T, 0, st>>>(P, do_phi, ngroups, sink_off, sink_x, src_off, src_x, E, f);
        else
            k_seam_pp<float, false><<<g, SEAM_T, 0, st>>>(P, do_phi, ngroups, sink_off, sink_x, src_off, src_x, E, f);
    }
    TG_CUDA(cudaGetLastError());
    (void)Sopt;
    return TG_OK;
}

int seam_pc(const tg_params &prm, int ewald_kind, int64_t ngroups, const int64_t *sink_off, const int32_t *sink_x,
            const int64_t *src_off, const float *src_m, const int32_t *src_x, double *f, const EwaldTables &E,
            cudaStream_t st) {
    const GParams P = make_gparams(prm);
    const int g = (int)(ngroups < 65535 ? ngroups : 65535);
    if (g <= 0) return TG_OK;
    if (prm.precision == TG_PREC_F64)
        k_seam_pc<double><<<g, 128, 0, st>>>(P, ewald_kind, ngroups, sink_off, sink_x, src_off, src_m, src_x, E, f);
    else
        k_seam_pc<float><<<g, 128, 0, st>>>(P, ewald_kind, ngroups, sink_off, sink_x, src_off, src_m, src_x, E, f);
    TG_CUDA(cudaGetLastError());
    return TG_OK;
}

int seam_node(const tg_params &prm, int ewald_kind, int is_cc, int64_t ngroups, const int32_t *sink_x,
              const int64_t *src_off, const float *src_m, const int32_t *src_x, double *L, const EwaldTables &E,
              cudaStream_t st) {
    const GParams P = make_gparams(prm);
    const int64_t want = (ngroups * 32 + 127) / 128;
    const int g = (int)(want < 65535 ? want : 65535);
    if (g <= 0) return TG_OK;
    if (prm.precision == TG_PREC_F64)
        k_seam_node<double><<<g, 128, 0, st>>>(P, ewald_kind, is_cc, ngroups, sink_x, src_off, src_m, src_x, E, L);
    else
        k_seam_node<float><<<g, 128, 0, st>>>(P, ewald_kind, is_cc, ngroups, sink_x, src_off, src_m, src_x, E, L);
    TG_CUDA(cudaGetLastError());
    return TG_OK;
}

EwaldTables solver_tables(Solver &S) { return tables(S); }

} // namespace tg
