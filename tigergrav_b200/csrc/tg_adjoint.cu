/*
 * tg_adjoint.cu -- reverse-mode differentiation of the kick-drift-kick
 * leapfrog (part_vect_kick / part_vect_drift, src/part_vect.cpp:341-436,
 * 493-540, driven as in src/main.cpp:258-273) through the tree forces.
 *
 * Forward (forward_steps): K leapfrog steps; the particle state (positions
 * and velocities, caller order) is checkpointed before the first step and
 * after every step.
 *
 * Backward (backward_steps): with J(x) = dg/dx the Jacobian of the
 * accelerations and (lx, lv) the adjoints of (x, v) at the end,
 *     lx += dt/2 G J(x_K) lv
 *     for s = K-1 .. 0:   lv += dt lx;   lx += c_s G J(x_s) lv
 * with c_s = dt for s > 0 (the half kicks of steps s-1 and s share x_s) and
 * dt/2 for s = 0.  J is symmetric, so J^T lv = J lv.  Each J(x_s) lv
 * rebuilds the tree, multipoles, lists and local expansions at the
 * checkpoint x_s (recomputation instead of storing them) and then runs
 * k_tidal_leaf, which contracts with the upstream gradient u = lv:
 *   far field   the tidal tensor of the leaf's local expansion L at the
 *               particle (L2P differentiated once more), times u_i;
 *   PC (direct and Ewald)  the tidal tensor of each source multipole
 *               (monopole and quadrupole terms of M2P differentiated) times u_i;
 *   PP (direct and Ewald)  each pair's Hessian times (u_i - u_j): the exact
 *               derivative of the pair force with respect to both particles.
 * Not differentiated: how a source node's multipoles and a sink node's
 * local expansion move with the positions of the particles inside the
 * source node (the far field's source side) and the octupole term of the
 * PC tidal tensor.  For upstream gradients that do not vary smoothly across
 * the box these are small against the terms kept; the finite-difference
 * tests measure the result.
 */
#include "tg_solver.cuh"

namespace tg {

/* dg/d(dX) of the local expansion at dX (L2P's force differentiated once
 * more), as 6 values in I2 order */
__device__ __forceinline__ void L2T(const double *L, const double *dX, double *T6) {
#pragma unroll
    for (int a = 0; a < 3; a++)
#pragma unroll
        for (int e = a; e < 3; e++) {
            double v = L[E2(a, e)];
#pragma unroll
            for (int c = 0; c < 3; c++) {
                v += L[E3(a, e, c)] * dX[c];
#pragma unroll
                for (int d = c; d < 3; d++) v += L[E4(a, e, c, d)] * dX[c] * dX[d] * factor<double>(E2(c, d));
            }
            T6[I2(a, e)] = -v;
        }
}

/* dg/dx_sink of M2P (contract_M2P) for the monopole and quadrupole terms */
template <class T>
__device__ __forceinline__ void M2T(const T *M, const T *D, T *T6) {
#pragma unroll
    for (int a = 0; a < 3; a++)
#pragma unroll
        for (int e = a; e < 3; e++) {
            T v = M[0] * D[E2(a, e)];
#pragma unroll
            for (int b = 0; b < 3; b++)
#pragma unroll
                for (int c = b; c < 3; c++) v += M[M2(c, b)] * D[E4(a, b, c, e)] * factor<T>(E2(c, b));
            T6[I2(a, e)] = -v;
        }
}

/* Hessian part of the softened pair force g -= m dX f(r) (pp_direct_pair):
 * d(dX f)/d(dX) = f I + dX dX^T f'(r)/r; returns f and f'(r)/r */
template <class T>
__device__ __forceinline__ void pp_pair_deriv(const GParams &P, T r2, T &f, T &fpr) {
    const T h = T(P.h);
    if (r2 > h * h) {
        const T rinv = t_rsqrt(r2);
        const T rinv2 = rinv * rinv;
        f = rinv2 * rinv;
        fpr = T(-3) * f * rinv2;
        return;
    }
    const T r = t_sqrt(r2);
    const T u = r / h;
    const T hinv = T(1) / h;
    if (r < T(0.5) * h) {
        /* f3 = (32 u^3 - 192/5 u^2 + 32/3) / h^3 */
        f = ((T(32) * u - T(192.0 / 5.0)) * u * u + T(32.0 / 3.0)) * hinv * hinv * hinv;
        fpr = (T(96) * u - T(384.0 / 5.0)) * hinv * hinv * hinv * hinv * hinv;
        return;
    }
    /* f2 = P(u) / r^3, P = -32/3 u^6 + 192/5 u^5 - 48 u^4 + 64/3 u^3 - 1/15 */
    const T u3 = u * u * u;
    const T Pu = ((((T(-32.0 / 3.0) * u + T(192.0 / 5.0)) * u - T(48)) * u + T(64.0 / 3.0)) * u3) - T(1.0 / 15.0);
    const T dPu = (((T(-64) * u + T(192)) * u - T(192)) * u + T(64)) * u * u;
    const T rinv = T(1) / r;
    const T rinv3 = rinv * rinv * rinv;
    f = Pu * rinv3;
    fpr = (dPu * hinv * rinv - T(3) * Pu * rinv * rinv) * rinv3;
}

template <class T>
__device__ __forceinline__ void sym_mul_add(const T *T6, const T *u, Acc<T> *o) {
    o[0].add(T6[I2(0, 0)] * u[0] + T6[I2(0, 1)] * u[1] + T6[I2(0, 2)] * u[2]);
    o[1].add(T6[I2(0, 1)] * u[0] + T6[I2(1, 1)] * u[1] + T6[I2(1, 2)] * u[2]);
    o[2].add(T6[I2(0, 2)] * u[0] + T6[I2(1, 2)] * u[1] + T6[I2(2, 2)] * u[2]);
}

/* sums of u over tiles of USUM_TILE particles (sorted order), one warp each */
constexpr int USUM_TILE = 256;
__global__ void k_tile_usum(int64_t n, const double *__restrict__ u, double *__restrict__ tile) {
    const int lane = threadIdx.x & 31;
    const int64_t k = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (k * USUM_TILE >= n) return;
    double s[3] = {0.0, 0.0, 0.0};
    const int64_t e = min(n, (k + 1) * USUM_TILE);
    for (int64_t q = k * USUM_TILE + lane; q < e; q += 32)
        for (int d = 0; d < 3; d++) s[d] += u[3 * q + d];
    for (int d = 0; d < 3; d++) {
        const double v = warp_sum(s[d]);
        if (lane == 0) tile[3 * k + d] = v;
    }
}
/* U_B = sum over the node's particles of m u_j (the mass-weighted upstream
 * gradient, i.e. M_B times the first-order shift of its centre of mass):
 * one warp per node, u in sorted order; whole tiles from their sums (without
 * them the root's warp walked all particles: 0.68 ms at 64^3) */
__global__ void k_node_usum(int64_t nn, double m, const int32_t *__restrict__ pb, const int32_t *__restrict__ pe,
                            const double *__restrict__ u, const double *__restrict__ tile, double *__restrict__ U) {
    const int lane = threadIdx.x & 31;
    const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (i >= nn) return;
    double s[3] = {0.0, 0.0, 0.0};
    const int64_t b = pb[i], e = pe[i];
    const int64_t k0 = (b + USUM_TILE - 1) / USUM_TILE, k1 = e / USUM_TILE; /* the whole tiles [k0, k1) */
    const int64_t b1 = k0 < k1 ? k0 * USUM_TILE : e, e0 = k0 < k1 ? k1 * USUM_TILE : e;
    for (int64_t q = b + lane; q < b1; q += 32)
        for (int d = 0; d < 3; d++) s[d] += u[3 * q + d];
    for (int64_t k = k0 + lane; k < k1; k += 32)
        for (int d = 0; d < 3; d++) s[d] += tile[3 * k + d];
    for (int64_t q = e0 + lane; q < e; q += 32)
        for (int d = 0; d < 3; d++) s[d] += u[3 * q + d];
    for (int d = 0; d < 3; d++) {
        const double v = warp_sum(s[d]);
        if (lane == 0) U[3 * i + d] = m * v;
    }
}

/* The source side of the node stage: a source of mass M at X whose particles
 * move by u shifts its centre by U/M, which changes the acceleration it causes
 * at the sink by D2(X_sink - X) U (monopole order).  V_A sums this over the
 * CC and CP lists of node A (direct and Ewald), evaluated at A's centre.
 * One warp per node, lanes over sources. */
template <class T>
__global__ void __launch_bounds__(128) k_vfield_node(GParams P, int64_t nn, const int32_t *__restrict__ pb,
                                                     const int32_t *__restrict__ pe, const MSrc *__restrict__ ms,
                                                     const int4 *__restrict__ pos, ListView LV, EwaldTables E,
                                                     const double *__restrict__ U, const double *__restrict__ us,
                                                     double *__restrict__ V) {
    const int lane = threadIdx.x & 31;
    const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (i >= nn) return;
    double acc[3] = {0.0, 0.0, 0.0};
    if (pe[i] > pb[i]) {
        const int32_t X[3] = {ms[i].x[0], ms[i].x[1], ms[i].x[2]};
        const bool per = P.ewald != 0;
        for (int ew = 0; ew < (per ? 2 : 1); ew++) {
            const int kcc = ew ? TG_CC_E : TG_CC_D, kcp = ew ? TG_CP_E : TG_CP_D;
            const int32_t *lcc = LV.pool[kcc] + LV.off[kcc][i];
            const int32_t ncc = LV.len[kcc][i];
            for (int32_t j = lane; j < ncc; j += 32) {
                const int32_t src = lcc[j];
                T dX[3], D[LP];
                for (int d = 0; d < 3; d++) dX[d] = sep<T>(X[d], ms[src].x[d], ew ? true : per);
                if (ew) green_ewald_any<T>(E, dX, D);
                else green_direct<T>(dX, D);
                const double Ub[3] = {U[3 * (int64_t)src], U[3 * (int64_t)src + 1], U[3 * (int64_t)src + 2]};
                for (int a = 0; a < 3; a++)
                    acc[a] += (double)D[E2(a, 0)] * Ub[0] + (double)D[E2(a, 1)] * Ub[1] + (double)D[E2(a, 2)] * Ub[2];
            }
            const int32_t *lcp = LV.pool[kcp] + LV.off[kcp][i];
            const int32_t ncp = LV.len[kcp][i];
            for (int32_t c = 0; c < ncp; c++) {
                const int32_t src = lcp[c];
                for (int32_t q = pb[src] + lane; q < pe[src]; q += 32) {
                    const int4 y = pos[q];
                    const int32_t yy[3] = {y.x, y.y, y.z};
                    T dX[3], D[LP];
                    for (int d = 0; d < 3; d++) dX[d] = sep<T>(X[d], yy[d], ew ? true : per);
                    if (ew) green_ewald_any<T>(E, dX, D);
                    else green_direct<T>(dX, D);
                    for (int a = 0; a < 3; a++)
                        acc[a] += P.m_d * ((double)D[E2(a, 0)] * us[3 * (int64_t)q] +
                                           (double)D[E2(a, 1)] * us[3 * (int64_t)q + 1] +
                                           (double)D[E2(a, 2)] * us[3 * (int64_t)q + 2]);
                }
            }
        }
    }
    for (int a = 0; a < 3; a++) {
        const double v = warp_sum(acc[a]);
        if (lane == 0) V[3 * i + a] = v;
    }
}

/* Vtot = V + Vtot(parent), one level, top-down */
__global__ void k_vfield_down(int64_t first, int64_t count, const int32_t *__restrict__ parent,
                              const double *__restrict__ V, double *__restrict__ Vtot) {
    const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= count) return;
    const int64_t i = first + k;
    const int32_t p = parent[i];
    for (int d = 0; d < 3; d++) Vtot[3 * i + d] = V[3 * i + d] + (p >= 0 ? Vtot[3 * (int64_t)p + d] : 0.0);
}

/* out_i = (J u)_i for the sinks of each leaf; u and out in sorted order
 * (3 doubles per particle).  One block per leaf, one thread per sink.  PP: with
 * the pair lists (leaf_max > 64; else k_tidal_pp and k_tidal_ewald_pp). */
template <class T, int BLOCK, bool PP>
__global__ void __launch_bounds__(BLOCK) k_tidal_leaf(GParams P, const int32_t *__restrict__ leaves, int32_t nleaves,
                                                      const int32_t *__restrict__ pb, const int32_t *__restrict__ pe,
                                                      const MSrc *__restrict__ ms, const int4 *__restrict__ pos,
                                                      ListView LV, EwaldTables E, const double *__restrict__ Lnode,
                                                      const double *__restrict__ U, const double *__restrict__ Vtot,
                                                      const double *__restrict__ u, double *__restrict__ out) {
    __shared__ int4 sy[BLOCK];
    __shared__ T su[BLOCK][3];
    __shared__ double sL[LP];
    const int tid = threadIdx.x;
    const bool per = P.ewald != 0;
    for (int32_t li = blockIdx.x; li < nleaves; li += gridDim.x) {
        const int32_t leaf = leaves[li];
        const int32_t b = pb[leaf], cnt = pe[leaf] - b;
        const bool active = tid < cnt;
        const int32_t i = b + (active ? tid : 0);
        const int4 xi4 = pos[i];
        const int32_t xi[3] = {xi4.x, xi4.y, xi4.z};
        const T ui[3] = {T(u[3 * (int64_t)i]), T(u[3 * (int64_t)i + 1]), T(u[3 * (int64_t)i + 2])};
        __syncthreads();
        if (tid < LP) sL[tid] = Lnode[35 * (int64_t)leaf + tid];
        __syncthreads();
        Acc<T> o[3];
        for (int d = 0; d < 3; d++) o[d].init(0.0);
        {
            /* far field: tidal tensor of L (dX through float as in L2P) */
            double dx[3], T6[6];
            for (int d = 0; d < 3; d++)
                dx[d] = (double)__double2float_rn(__dadd_rn(pos2d(xi[d]), -pos2d(ms[leaf].x[d])));
            L2T(sL, dx, T6);
            const double ud[3] = {(double)ui[0], (double)ui[1], (double)ui[2]};
            for (int a = 0; a < 3; a++)
                o[a].add(T(T6[I2(a, 0)] * ud[0] + T6[I2(a, 1)] * ud[1] + T6[I2(a, 2)] * ud[2] +
                           Vtot[3 * (int64_t)leaf + a]));
        }
        /* PC direct and Ewald: sink-side tidal tensors */
        for (int ew = 0; ew < (per ? 2 : 1); ew++) {
            const int kind = ew ? TG_PC_E : TG_PC_D;
            const int32_t *lst = LV.pool[kind] + LV.off[kind][leaf];
            const int32_t len = LV.len[kind][leaf];
            for (int32_t j = 0; j < len; j++) {
                const MSrc &s = ms[lst[j]];
                T dX[3], D[LP], M[MP], T6[6];
#pragma unroll
                for (int d = 0; d < 3; d++) dX[d] = sep<T>(xi[d], s.x[d], ew ? true : per);
#pragma unroll
                for (int q = 0; q < MP; q++) M[q] = T(s.m[q]);
                if (ew) green_ewald_any<T>(E, dX, D);
                else green_direct<T>(dX, D);
                M2T<T>(M, D, T6);
                sym_mul_add<T>(T6, ui, o);
                /* source side: the source's centre moves by U/M (monopole order) */
                const T Ub[3] = {T(U[3 * (int64_t)lst[j]]), T(U[3 * (int64_t)lst[j] + 1]), T(U[3 * (int64_t)lst[j] + 2])};
                for (int a = 0; a < 3; a++) o[a].add(D[E2(a, 0)] * Ub[0] + D[E2(a, 1)] * Ub[1] + D[E2(a, 2)] * Ub[2]);
            }
        }
        /* PP direct and Ewald: pair Hessians times (u_i - u_j) */
        const T m = T(P.m_d);
        for (int ew = 0; ew < (!PP ? 0 : (per ? 2 : 1)); ew++) {
            const int kind = ew ? TG_PP_E : TG_PP_D;
            const int32_t *lst = LV.pool[kind] + LV.off[kind][leaf];
            const int32_t len = LV.len[kind][leaf];
            for (int32_t c = 0; c < len; c++) {
                const int32_t src = lst[c];
                const int32_t sb = pb[src], sn = pe[src] - sb;
                for (int32_t base = 0; base < sn; base += BLOCK) {
                    const int32_t nt = min(BLOCK, sn - base);
                    __syncthreads();
                    if (tid < nt) {
                        const int64_t q = sb + base + tid;
                        sy[tid] = pos[q];
                        for (int d = 0; d < 3; d++) su[tid][d] = T(u[3 * q + d]);
                    }
                    __syncthreads();
                    for (int32_t q = 0; q < nt; q++) {
                        const int4 y = sy[q];
                        const T du[3] = {ui[0] - su[q][0], ui[1] - su[q][1], ui[2] - su[q][2]};
                        if (!ew) {
                            const T dX[3] = {sep<T>(xi[0], y.x, per), sep<T>(xi[1], y.y, per),
                                             sep<T>(xi[2], y.z, per)};
                            const T r2 = dX[0] * dX[0] + dX[1] * dX[1] + dX[2] * dX[2];
                            T f, fpr;
                            pp_pair_deriv<T>(P, r2, f, fpr);
                            const T s = (dX[0] * du[0] + dX[1] * du[1] + dX[2] * du[2]) * fpr;
                            for (int d = 0; d < 3; d++) o[d].add(-m * (f * du[d] + dX[d] * s));
                        } else {
                            T dX[3] = {wrap_sep_t<T>(xi[0], y.x), wrap_sep_t<T>(xi[1], y.y), wrap_sep_t<T>(xi[2], y.z)};
                            if (!(dX[0] * dX[0] + dX[1] * dX[1] + dX[2] * dX[2] > T(1.0e-12))) continue;
                            T D[LP];
                            green_ewald_any<T>(E, dX, D);
                            for (int a = 0; a < 3; a++)
                                o[a].add(-m * (D[E2(a, 0)] * du[0] + D[E2(a, 1)] * du[1] + D[E2(a, 2)] * du[2]));
                        }
                    }
                }
            }
        }
        if (active)
            for (int d = 0; d < 3; d++) out[3 * (int64_t)i + d] = o[d].get();
    }
}

/*
 * PP direct: out_i += -sum_j m H(x_i - x_j) (u_i - u_j), H the Hessian of the
 * softened pair force (pp_pair_deriv).  One block per leaf of at most 64 sinks,
 * C = 128 / ns copies of them (copy p takes every C-th source of a stage), every
 * pair folded into the compensated totals, copies added in FP64 in order.  In
 * k_tidal_leaf, at the registers of the PC tensors, this was 2.2 of 5 ms of a 64^3
 * Jacobian product.  Plain sums over 8 pairs before each fold take 0.2 ms less of the
 * 15.8 ms of two steps forward and back there, and lose terms that are 2^-24 of
 * another in their group.
 */
template <class T>
__global__ void __launch_bounds__(128) k_tidal_pp(GParams P, const int32_t *__restrict__ leaves,
                                                  const int32_t *__restrict__ pb, const int32_t *__restrict__ pe,
                                                  const int4 *__restrict__ pos, ListView LV,
                                                  const double *__restrict__ u, double *__restrict__ out) {
    __shared__ int4 sy[128];
    __shared__ __align__(4 * sizeof(T)) T su[128][4]; /* x, y, z: one load */
    __shared__ double red[128][3];
    const int t = threadIdx.x;
    const bool per = P.ewald != 0;
    const int32_t leaf = leaves[blockIdx.x];
    const int32_t b = pb[leaf], ns = pe[leaf] - b;
    if (ns <= 0) return;
    const int C = 128 / ns, phase = t / ns;
    const int64_t i = b + t % ns;
    const int4 xi = pos[i];
    const T ui[3] = {T(u[3 * i]), T(u[3 * i + 1]), T(u[3 * i + 2])};
    const T m = T(P.m_d);
    Acc<T> o[3];
    for (int d = 0; d < 3; d++) o[d].init(0.0);
    const int32_t *lst = LV.pool[TG_PP_D] + LV.off[TG_PP_D][leaf];
    const int32_t len = LV.len[TG_PP_D][leaf];
    int32_t c = 0, done = 0; /* the next source: leaf c of the list, its particle `done` */
    for (;;) {
        /* stage up to 128 particles of consecutive source leaves */
        int32_t nt = 0;
        __syncthreads();
        while (c < len && nt < 128) {
            const int32_t sb = pb[lst[c]], sn = pe[lst[c]] - sb, k = min(sn - done, 128 - nt);
            if (t >= nt && t < nt + k) {
                const int64_t q = sb + done + t - nt;
                sy[t] = pos[q];
                for (int d = 0; d < 3; d++) su[t][d] = T(u[3 * q + d]);
            }
            nt += k;
            done += k;
            if (done == sn) {
                c++;
                done = 0;
            }
        }
        if (nt == 0) break;
        __syncthreads();
        if (phase >= C) continue;
#pragma unroll 4
        for (int32_t q = phase; q < nt; q += C) {
            const int4 y = sy[q];
            T du[3];
            if constexpr (sizeof(T) == 4) {
                const float4 uj = *reinterpret_cast<const float4 *>(su[q]);
                du[0] = ui[0] - uj.x, du[1] = ui[1] - uj.y, du[2] = ui[2] - uj.z;
            } else {
                for (int d = 0; d < 3; d++) du[d] = ui[d] - su[q][d];
            }
            const T dX[3] = {sep<T>(xi.x, y.x, per), sep<T>(xi.y, y.y, per), sep<T>(xi.z, y.z, per)};
            const T r2 = dX[0] * dX[0] + dX[1] * dX[1] + dX[2] * dX[2];
            T f, fpr;
            pp_pair_deriv<T>(P, r2, f, fpr);
            const T w = (dX[0] * du[0] + dX[1] * du[1] + dX[2] * du[2]) * fpr;
            for (int d = 0; d < 3; d++) o[d].add(-m * (f * du[d] + dX[d] * w));
        }
    }
    for (int d = 0; d < 3; d++) red[t][d] = phase < C ? o[d].get() : 0.0;
    __syncthreads();
    if (t < ns)
        for (int d = 0; d < 3; d++) {
            double v = 0.0;
            for (int p = 0; p < C; p++) v += red[t + p * ns][d];
            out[3 * i + d] += v;
        }
}

/*
 * PP Ewald: sum_j m D2(x_i - x_j) (u_i - u_j) with the split of
 * tg_ewald_sep.cuh.  The reciprocal part of D2 is sum_h 4 pi w_h h h^T
 * cos(th_i - th_j), so a source leaf gives per h the sums of (cos, sin) th_j and
 * of (h.u_j)(cos, sin) th_j; the real-space part is the Hessians of the nearest
 * image and its neighbours towards the near corner.  The whole green_ewald
 * per pair took 0.9 of a 64^3 Jacobian product (12e6 pairs).
 *
 * The reciprocal sums are FP64 in both paths: a sink takes (h.u_i) times one pair of
 * sums less the other, and with FP32 sums a common part of u, which every
 * u_i - u_j is free of, would leave its rounding.  In the FP32 path the nearest image
 * is FP64 too, as in the force (sep_near), for the same cancellation, at alpha^3.
 */
struct Sep4 {
    double c, s, uc, us;
};
__device__ __forceinline__ void sep_madd(Sep4 &a, double m, const Sep4 &f) {
    a.c = fma(m, f.c, a.c);
    a.s = fma(m, f.s, a.s);
    a.uc = fma(m, f.uc, a.uc);
    a.us = fma(m, f.us, a.us);
}

template <class T>
__global__ void __launch_bounds__(128) k_tidal_sf(const int32_t *__restrict__ src, const int32_t *__restrict__ pb,
                                                  const int32_t *__restrict__ pe, const int4 *__restrict__ pos,
                                                  const double *__restrict__ u, EwaldTables E, int t0, int t1,
                                                  Sep4 *__restrict__ sf) {
    __shared__ SepTrig<T> trig;
    const int32_t node = src[blockIdx.x];
    const int32_t b = pb[node], n = pe[node] - b;
    sep_trig<T>(trig, pos + b, n);
    Sep4 *const row = sf + (int64_t)blockIdx.x * (t1 - t0) - t0;
    if constexpr (sizeof(T) == 4) { /* a thread per run, as k_ewald_sf */
        for (int r = threadIdx.x; r < E.sep_nrun; r += 128) {
            const int4 run = __ldg(&E.sep_run[r]);
            const int t = run.w >> 8, len = run.w & 255;
            if (t >= t1 || t + len <= t0) continue;
            Sep4 a[SEP_RUN] = {};
            for (int32_t j = 0; j < n; j++) {
                double2 e = trig.first(j, run);
                const double2 z = trig.step(j);
                const double *uj = u + 3 * (int64_t)(b + j);
                double hu = run.x * uj[0] + run.y * uj[1] + run.z * uj[2];
#pragma unroll
                for (int k = 0; k < SEP_RUN; k++) {
                    a[k].c += e.x;
                    a[k].s += e.y;
                    a[k].uc = fma(hu, e.x, a[k].uc);
                    a[k].us = fma(hu, e.y, a[k].us);
                    hu += uj[2];
                    e = trig.mul(e, z);
                }
            }
#pragma unroll
            for (int k = 0; k < SEP_RUN; k++)
                if (k < len && t + k >= t0 && t + k < t1) row[t + k] = a[k];
        }
    } else {
        for (int t = t0 + threadIdx.x; t < t1; t += 128) {
            const int4 h = __ldg(&E.sep_h[t]);
            Sep4 a{};
            for (int32_t j = 0; j < n; j++) {
                const double2 q = trig.at(j, pos + b, h);
                const double *uj = u + 3 * (int64_t)(b + j);
                const double hu = h.x * uj[0] + h.y * uj[1] + h.z * uj[2];
                a.c += q.x;
                a.s += q.y;
                a.uc = fma(hu, q.x, a.uc);
                a.us = fma(hu, q.y, a.us);
            }
            row[t] = a;
        }
    }
}

/* r += (d1 + d2 x x^T) du for one image at displacement x */
template <class T>
__device__ __forceinline__ void tidal_image(const SepNear &K, T x0, T x1, T x2, T r2, const T *du, T *r) {
    const T alpha = T(Sep<T>::ALPHA);
    const T rinv = t_rsqrt(r2), r2inv = rinv * rinv, rr = r2 * rinv;
    T e;
    const T ec = sep_erfc(K, r2, rinv, e);
    const T ce = T(Sep<T>::ALPHA * 1.1283791670955126) * e; /* 2 alpha / sqrt(pi) e^(-alpha^2 r^2) */
    const T d1 = fma(ce, rr, ec) * rinv * r2inv;
    const T d2 = -fma(T(3), d1, T(2) * alpha * alpha * ce) * r2inv;
    const T s = (x0 * du[0] + x1 * du[1] + x2 * du[2]) * d2;
    r[0] = fma(x0, s, fma(d1, du[0], r[0]));
    r[1] = fma(x1, s, fma(d1, du[1], r[1]));
    r[2] = fma(x2, s, fma(d1, du[2], r[2]));
}

/* the mirror images of a pair at x: r += D2 du */
template <class T>
__device__ __forceinline__ void tidal_images(const SepNear &K, const T *x, const T *du, T *r) {
    T c[3], u[3], v[3];
#pragma unroll
    for (int d = 0; d < 3; d++) {
        c[d] = x[d] - copysign(T(1), x[d]);
        u[d] = x[d] * x[d];
        v[d] = c[d] * c[d];
    }
#pragma unroll
    for (int k = 1; k < 8; k++) {
        const T s = (k & 1 ? v[0] : u[0]) + (k & 2 ? v[1] : u[1]) + (k & 4 ? v[2] : u[2]);
        if (s < T(1)) tidal_image<T>(K, k & 1 ? c[0] : x[0], k & 2 ? c[1] : x[1], k & 4 ? c[2] : x[2], s, du, r);
    }
}

/* the sums of one sink over the real-space parts D2(x) (u_i - u_j) of its pairs,
 * times -m; a pair with r <= 1e-6 has none, and takes back what the leaf sums add */
template <class T> struct TidalPairs;
template <> struct TidalPairs<double> {
    double o[3], ui[3];
    __device__ __forceinline__ void init(const double *u) {
        for (int d = 0; d < 3; d++) o[d] = 0.0, ui[d] = u[d];
    }
    __device__ __forceinline__ void add(const EwaldTables &E, const SepNear &K, double m, int4 xi, int4 yj, const double *uj) {
        const double x[3] = {wrap_sep_d(xi.x, yj.x), wrap_sep_d(xi.y, yj.y), wrap_sep_d(xi.z, yj.z)};
        const double du[3] = {ui[0] - uj[0], ui[1] - uj[1], ui[2] - uj[2]};
        const double r2 = x[0] * x[0] + x[1] * x[1] + x[2] * x[2];
        if (!(r2 > 1.0e-12)) {
            for (int d = 0; d < 3; d++) o[d] += -m * (-E.sep_r2 * du[d]);
            return;
        }
        double q[3] = {0.0, 0.0, 0.0};
        tidal_images<double>(K, x, du, q);
        /* nearest image with the direct 1/r removed: d1 = -f0, d2 = (3 f0 - 2 alpha^2 c e) / r^2, or the
         * derivative of f0's series (ewald_nearest) for alpha r < 1/2, where the two cancel */
        const double alpha = Sep<double>::ALPHA;
        const double rinv = t_rsqrt(r2), rr = r2 * rinv, y = alpha * alpha * r2;
        double p0, f0, d2;
        ewald_nearest<double>(alpha, rr, rinv, p0, f0);
        if (y < 0.25) {
            double s = 10.0 / 41731200.0;
            s = fma(s, y, -9.0 / 3810240.0);
            s = fma(s, y, 8.0 / 383040.0);
            s = fma(s, y, -7.0 / 42840.0);
            s = fma(s, y, 6.0 / 5400.0);
            s = fma(s, y, -5.0 / 780.0);
            s = fma(s, y, 4.0 / 132.0);
            s = fma(s, y, -3.0 / 27.0);
            s = fma(s, y, 2.0 / 7.0);
            s = fma(s, y, -0.4);
            d2 = -2.0 * 1.1283791670955126 * (alpha * alpha * alpha * alpha * alpha) * s;
        } else {
            const double ce = Sep<double>::ALPHA * 1.1283791670955126 * exp(-y);
            d2 = (3.0 * f0 - 2.0 * alpha * alpha * ce) * rinv * rinv;
        }
        const double s = (x[0] * du[0] + x[1] * du[1] + x[2] * du[2]) * d2;
#pragma unroll
        for (int d = 0; d < 3; d++) o[d] += -m * (q[d] + x[d] * s - f0 * du[d]);
    }
    __device__ __forceinline__ void fold() {}
    __device__ __forceinline__ double get(int d, double) const { return o[d]; }
};
/* FP32: the nearest image in FP64, d1 = -f0 and d2 = -2 df0/dr^2; the mirror images
 * in FP32, summed as in SepPairs */
template <> struct TidalPairs<float> {
    double o[3], ui[3];
    float a[3];
    Acc<float> i[3];
    __device__ __forceinline__ void init(const double *u) {
#pragma unroll
        for (int d = 0; d < 3; d++) {
            o[d] = 0.0, ui[d] = u[d], a[d] = 0.0f;
            i[d].init(0.0);
        }
    }
    __device__ __forceinline__ void fold() {
#pragma unroll
        for (int d = 0; d < 3; d++) {
            i[d].add(a[d]);
            a[d] = 0.0f;
        }
    }
    __device__ __forceinline__ void add(const EwaldTables &E, const SepNear &K, double, int4 xi, int4 yj, const double *uj) {
        const int32_t n[3] = {(int32_t)((uint32_t)xi.x - (uint32_t)yj.x), (int32_t)((uint32_t)xi.y - (uint32_t)yj.y),
                              (int32_t)((uint32_t)xi.z - (uint32_t)yj.z)};
        float x[3], w[3];
        double X[3], du[3];
#pragma unroll
        for (int d = 0; d < 3; d++) {
            x[d] = __int2float_rn(n[d]) * 2.3283064365386963e-10f;
            X[d] = i2d(n[d]);
            du[d] = ui[d] - uj[d];
            w[d] = (float)du[d];
        }
        if (!(x[0] * x[0] + x[1] * x[1] + x[2] * x[2] > 1.0e-12f)) {
            for (int d = 0; d < 3; d++) o[d] -= E.sep_r2 * du[d];
            return;
        }
        tidal_images<float>(K, x, w, a);
        const double t = fma(fma(X[0], X[0], fma(X[1], X[1], X[2] * X[2])), 8.0 / 3.0 * POS_INV * POS_INV, -1.0);
        double f = K.f[SEP_DF], df = 0.0; /* f0 and its derivative by t */
#pragma unroll
        for (int k = SEP_DF - 1; k >= 0; k--) {
            df = fma(df, t, f);
            f = fma(f, t, K.f[k]);
        }
        const double s = fma(X[0], du[0], fma(X[1], du[1], X[2] * du[2])) * (-16.0 / 3.0 * POS_INV * POS_INV * df);
#pragma unroll
        for (int d = 0; d < 3; d++) o[d] += fma(X[d], s, -f * du[d]);
    }
    __device__ __forceinline__ double get(int d, double m) const { return -m * (o[d] + i[d].get()); }
};

/* one chunk of a PP_E list (as k_ewald_pp): the real-space part per pair into
 * part (3 per sink) and, with sf, the reciprocal source sums into tpart */
template <class T>
__global__ void __launch_bounds__(64) k_tidal_ewald_pp(GParams P, const int32_t *__restrict__ leaves, int32_t nleaves,
                                                       int32_t first, const int32_t *__restrict__ off, const int32_t *__restrict__ pb,
                                                       const int32_t *__restrict__ pe, const int4 *__restrict__ pos,
                                                       ListView LV, EwaldTables E, SepNear K, const double *__restrict__ u,
                                                       double *__restrict__ part, const int32_t *__restrict__ slot,
                                                       const Sep4 *__restrict__ sf, Sep4 *__restrict__ tpart) {
    __shared__ int4 sy[64];
    __shared__ double su[64][3];
    __shared__ int32_t s_row[EW_KPP_MAX];
    const int tid = threadIdx.x;
    const int64_t c = (int64_t)first + blockIdx.x;
    const int32_t li = ew_leaf(off, nleaves, c), k = (int32_t)(c - off[li]);
    const int32_t leaf = leaves[li];
    const int32_t b = pb[leaf], cnt = pe[leaf] - b;
    const int64_t i = b + (tid < cnt ? tid : 0);
    const int4 xi = pos[i];
    TidalPairs<T> o;
    o.init(u + 3 * i);
    const int32_t *lst = LV.pool[TG_PP_E] + LV.off[TG_PP_E][leaf];
    const int32_t len = LV.len[TG_PP_E][leaf], kpp = ew_kpp(len), e0 = k * kpp, e1 = min(len, e0 + kpp);
    if (tid < e1 - e0) s_row[tid] = slot[lst[e0 + tid]];
    for (int32_t e = e0; e < e1; e++) {
        const int32_t src = lst[e];
        const int32_t sb = pb[src], sn = pe[src] - sb; /* leaf_max <= 64: one stage */
        __syncthreads();
        if (tid < sn) {
            const int64_t q = sb + tid;
            sy[tid] = pos[q];
            for (int d = 0; d < 3; d++) su[tid][d] = u[3 * q + d];
        }
        __syncthreads();
        if (tid < ((cnt + 31) & ~31))
            for (int32_t q = 0; q < sn;) {
                const int32_t q1 = min(sn, q + SEP_FOLD);
                for (; q < q1; q++) o.add(E, K, P.m_d, xi, sy[q], su[q]);
                o.fold();
            }
    }
    if (tid < cnt)
        for (int d = 0; d < 3; d++) part[3 * ((int64_t)blockIdx.x * 64 + tid) + d] = o.get(d, P.m_d);
    if (sf) ew_tsum<Sep4>(s_row, e1 - e0, 0, Sep<T>::N, tid, sf, P.m_d, tpart + (int64_t)blockIdx.x * Sep<T>::N);
}

/* out += the chunk sums of each leaf, in chunk order, and the reciprocal part
 * -sum_h 4 pi w_h h ((h.u_i) cos(th_i - th_j) - (h.u_j) cos(th_i - th_j)) from
 * the chunks' source sums.  One block per leaf of the batch, four threads per sink. */
template <class T>
__global__ void __launch_bounds__(256) k_tidal_ewald_reduce(EwBatch B, const int32_t *__restrict__ leaves,
                                                            const int32_t *__restrict__ off,
                                                            const int32_t *__restrict__ pb, const int32_t *__restrict__ pe,
                                                            const int4 *__restrict__ pos, EwaldTables E,
                                                            const double *__restrict__ u, const double *__restrict__ part,
                                                            const Sep4 *__restrict__ tpart, double *__restrict__ out) {
    constexpr int TILE = sizeof(T) == 4 ? Sep<float>::N : 384; /* vectors whose sums are held at a time */
    __shared__ SepTrig<T> trig;
    __shared__ double4 sT[TILE];
    __shared__ double sv[4][64][3];
    const int32_t li = B.l0 + blockIdx.x;
    const int tid = threadIdx.x, t = tid & 63, grp = tid >> 6;
    const int32_t a0 = off[li] - B.a0, a1 = off[li + 1] - B.a0;
    if (a1 == a0) return; /* block-uniform */
    const int32_t leaf = leaves[li];
    const int32_t b = pb[leaf], cnt = pe[leaf] - b;
    const int64_t i = b + (t < cnt ? t : 0);
    const double ui[3] = {u[3 * i], u[3 * i + 1], u[3 * i + 2]};
    sep_trig<T>(trig, pos + b, cnt);
    double v[3] = {0.0, 0.0, 0.0};
    for (int t0 = 0; t0 < Sep<T>::N; t0 += TILE) {
        const int nt = min(TILE, Sep<T>::N - t0);
        __syncthreads();
        for (int q = tid; q < nt; q += 256) {
            double4 s = make_double4(0.0, 0.0, 0.0, 0.0);
            for (int64_t c = a0; c < a1; c++) {
                const Sep4 f = tpart[c * Sep<T>::N + t0 + q];
                s.x += f.c;
                s.y += f.s;
                s.z += f.uc;
                s.w += f.us;
            }
            sT[q] = s;
        }
        __syncthreads();
        if (t >= cnt) continue;
        if constexpr (sizeof(T) == 4) {
            const double2 z = trig.step(t);
            for (int r = grp; r < E.sep_nrun; r += 4) {
                const int4 run = __ldg(&E.sep_run[r]);
                const int q0 = run.w >> 8, len = run.w & 255;
                double2 e = trig.first(t, run);
                double hu = run.x * ui[0] + run.y * ui[1] + run.z * ui[2], h = run.z, sum = 0.0;
                for (int k = 0; k < len; k++) {
                    const double4 s = sT[q0 + k];
                    const double f = __ldg(&E.sep_w[q0 + k]) * (hu * (e.x * s.x + e.y * s.y) - (e.x * s.z + e.y * s.w));
                    sum += f;
                    v[2] = fma(f, h, v[2]);
                    h += 1.0;
                    hu += ui[2];
                    e = trig.mul(e, z);
                }
                v[0] = fma(sum, (double)run.x, v[0]);
                v[1] = fma(sum, (double)run.y, v[1]);
            }
        } else {
            for (int q = grp; q < nt; q += 4) {
                const int4 h = __ldg(&E.sep_h[t0 + q]);
                const double2 cs = trig.at(t, pos + b, h);
                const double4 s = sT[q];
                const double hu = h.x * ui[0] + h.y * ui[1] + h.z * ui[2];
                const double C = cs.x, Sn = cs.y;
                const double f = __ldg(&E.sep_w[t0 + q]) * (hu * (C * s.x + Sn * s.y) - (C * s.z + Sn * s.w));
                v[0] += f * h.x;
                v[1] += f * h.y;
                v[2] += f * h.z;
            }
        }
    }
    for (int d = 0; d < 3; d++) sv[grp][t][d] = v[d];
    __syncthreads();
    if (t >= cnt || grp != 0) return;
    for (int d = 0; d < 3; d++) {
        double w = 0.0;
        for (int64_t c = a0; c < a1; c++) w += part[3 * (c * 64 + t) + d];
        const double rec = (sv[0][t][d] + sv[1][t][d]) + (sv[2][t][d] + sv[3][t][d]);
        out[3 * i + d] += w - 12.566370614359172 * rec; /* 4 pi */
    }
}

/* bytes of a PP_E chunk of a Jacobian product */
constexpr size_t tidal_chunk_bytes(int N) { return 64 * 3 * sizeof(double) + N * sizeof(Sep4); }

/* the PP_E lists' part of J u, added to tid_o (leaf_max <= 64) */
template <class T>
static int tidal_ewald(Solver &S, const GParams &P, const ListView &LV, const EwaldTables &E, cudaStream_t st) {
    const int32_t nleaves = (int32_t)S.st.leaves;
    int32_t npp = 0, total = 0, nsrc = 0;
    TG_TRY(leaf_chunks(S, LV, npp, total, nsrc, st));
    if (npp <= 0) return TG_OK;
    constexpr int N = Sep<T>::N;
    std::vector<EwBatch> batches;
    TG_TRY(leaf_batches(S, npp, npp, tidal_chunk_bytes(N), 0, batches, st));
    size_t slots = 0;
    for (const EwBatch &B : batches) slots = std::max(slots, (size_t)B.na);
    const int nv = ew_vectors(S, nsrc, sizeof(Sep4), N);
    TG_TRY(ensure(S.ew_part, slots * 64 * 3));
    TG_TRY(ensure(S.ew_sf, (size_t)nsrc * nv * sizeof(Sep4)));
    TG_TRY(ensure(S.ew_tpart, slots * N * sizeof(Sep4)));
    Sep4 *sf = reinterpret_cast<Sep4 *>(S.ew_sf.p), *tpart = reinterpret_cast<Sep4 *>(S.ew_tpart.p);
    if (nv == N) {
        k_tidal_sf<T><<<nsrc, 128, 0, st>>>(S.ew_src.p, S.nd_pb.p, S.nd_pe.p, S.pos.p, S.tid_u.p, E, 0, N, sf);
        TG_TRY(launched(S));
    }
    for (const EwBatch &B : batches) {
        if (B.na == 0) continue;
        k_tidal_ewald_pp<T><<<B.na, 64, 0, st>>>(P, S.idx.p, nleaves, B.a0, S.ew_off.p, S.nd_pb.p, S.nd_pe.p, S.pos.p,
                                                 LV, E, S.ew_near, S.tid_u.p, S.ew_part.p, S.ew_slot.p, nv == N ? sf : nullptr, tpart);
        TG_TRY(launched(S));
        for (int t0 = 0; nv < N && t0 < N; t0 += nv) {
            const int t1 = std::min(N, t0 + nv);
            k_tidal_sf<T><<<nsrc, 128, 0, st>>>(S.ew_src.p, S.nd_pb.p, S.nd_pe.p, S.pos.p, S.tid_u.p, E, t0, t1, sf);
            TG_TRY(launched(S));
            k_ewald_tsum<Sep4><<<B.na, 64, 0, st>>>(N, P.m_d, S.idx.p, nleaves, B.a0, S.ew_off.p, LV, S.ew_slot.p, t0,
                                                    t1, sf, tpart);
            TG_TRY(launched(S));
        }
        k_tidal_ewald_reduce<T><<<B.l1 - B.l0, 256, 0, st>>>(B, S.idx.p, S.ew_off.p, S.nd_pb.p, S.nd_pe.p, S.pos.p, E,
                                                             S.tid_u.p, S.ew_part.p, tpart, S.tid_o.p);
        TG_TRY(launched(S));
    }
    return TG_OK;
}

/* u_sorted[i] = u[caller index of i] */
__global__ void k_gather3(int64_t n, const int4 *__restrict__ pos, const double *__restrict__ u,
                          double *__restrict__ us) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int64_t w = pos[i].w;
    for (int d = 0; d < 3; d++) us[3 * i + d] = u[3 * w + d];
}

/* y[caller index of i] += c * x_sorted[i] */
__global__ void k_scatter_axpy3(int64_t n, const int4 *__restrict__ pos, double c, const double *__restrict__ xs,
                                double *__restrict__ y) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int64_t w = pos[i].w;
    for (int d = 0; d < 3; d++) y[3 * w + d] += c * xs[3 * i + d];
}

/* y += c * x (n x 3, caller order) */
__global__ void k_axpy3(int64_t n, double c, const double *__restrict__ x, double *__restrict__ y) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= 3 * n) return;
    y[i] += c * x[i];
}

/* The buffers and kernels of tidal_apply, taken ahead of the first backward pass: an
 * allocation waits for the device, and took 0.2 to 0.7 s on some machines.  The Ewald
 * scratch is sized by the largest lists of the solver's force evaluations, which are
 * those of the checkpoints. */
int tidal_reserve(Solver &S) {
    const bool f64 = S.prm.precision == TG_PREC_F64, small = S.prm.leaf_max <= 64;
    TG_TRY(ensure(S.adj_x, 3 * S.n));
    TG_TRY(ensure(S.adj_v, 3 * S.n));
    TG_TRY(ensure(S.tid_u, 3 * S.n));
    TG_TRY(ensure(S.tid_o, 3 * S.n));
    TG_TRY(ensure(S.tid_U, 3 * S.nnodes));
    TG_TRY(ensure(S.tid_V, 6 * S.nnodes));
    TG_TRY(ensure(S.tid_tile, 3 * ((S.n + USUM_TILE - 1) / USUM_TILE)));
    if (S.ew_max_npp > 0) { /* as tidal_ewald */
        const int N = f64 ? Sep<double>::N : Sep<float>::N;
        const size_t slots = std::min<size_t>(S.ew_max_npp, S.ew_scratch() / tidal_chunk_bytes(N) + 1);
        TG_TRY(ensure(S.ew_part, slots * 64 * 3));
        TG_TRY(ensure(S.ew_tpart, slots * N * sizeof(Sep4)));
        TG_TRY(ensure(S.ew_sf, (size_t)S.ew_max_nsrc * ew_vectors(S, S.ew_max_nsrc, sizeof(Sep4), N) * sizeof(Sep4)));
    }
    const void *leaf = small ? (f64 ? (const void *)k_tidal_leaf<double, 64, false> : (const void *)k_tidal_leaf<float, 64, false>)
                             : (f64 ? (const void *)k_tidal_leaf<double, 128, true> : (const void *)k_tidal_leaf<float, 128, true>);
    const void *k[] = {leaf,
                       f64 ? (const void *)k_vfield_node<double> : (const void *)k_vfield_node<float>,
                       f64 ? (const void *)k_tidal_pp<double> : (const void *)k_tidal_pp<float>,
                       f64 ? (const void *)k_tidal_sf<double> : (const void *)k_tidal_sf<float>,
                       f64 ? (const void *)k_tidal_ewald_pp<double> : (const void *)k_tidal_ewald_pp<float>,
                       f64 ? (const void *)k_tidal_ewald_reduce<double> : (const void *)k_tidal_ewald_reduce<float>,
                       (const void *)k_gather3, (const void *)k_tile_usum, (const void *)k_node_usum,
                       (const void *)k_vfield_down, (const void *)k_scatter_axpy3, (const void *)k_axpy3};
    cudaFuncAttributes a;
    for (const void *f : k) TG_CUDA(cudaFuncGetAttributes(&a, f)); /* loads the kernel's code */
    return TG_OK;
}

/* acc += c J u (u, acc: n x 3 doubles in caller order, device) for the
 * particles and lists currently in S; runs the node stage for the local
 * expansions first */
int tidal_apply(Solver &S, const double *u, double *acc, double c, cudaStream_t st) {
    if (!S.have_lists) return TG_ERR_STATE;
    TG_TRY(ewald_tables(S, st));
    const int64_t n = S.n;
    const GParams P = make_gparams(S.prm);
    const EwaldTables E = tables(S);
    const ListView LV = listview(S);
    TG_TRY(node_stage(S, P, LV, E, st));
    TG_TRY(ensure(S.tid_u, 3 * n));
    TG_TRY(ensure(S.tid_o, 3 * n));
    const int64_t nn = S.nnodes;
    TG_TRY(ensure(S.tid_U, 3 * nn));
    TG_TRY(ensure(S.tid_V, 6 * nn));
    const int gn = (int)((n + 255) / 256);
    k_gather3<<<gn, 256, 0, st>>>(n, S.pos.p, u, S.tid_u.p);
    TG_TRY(launched(S));
    const bool f64n = S.prm.precision == TG_PREC_F64;
    const int gw = (int)((nn * 32 + 127) / 128);
    const int64_t ntile = (n + USUM_TILE - 1) / USUM_TILE;
    TG_TRY(ensure(S.tid_tile, 3 * ntile));
    k_tile_usum<<<(int)((ntile * 32 + 127) / 128), 128, 0, st>>>(n, S.tid_u.p, S.tid_tile.p);
    TG_TRY(launched(S));
    k_node_usum<<<gw, 128, 0, st>>>(nn, S.prm.m, S.nd_pb.p, S.nd_pe.p, S.tid_u.p, S.tid_tile.p, S.tid_U.p);
    TG_TRY(launched(S));
    double *V = S.tid_V.p, *Vtot = S.tid_V.p + 3 * nn;
    if (f64n)
        k_vfield_node<double><<<gw, 128, 0, st>>>(P, nn, S.nd_pb.p, S.nd_pe.p, S.nd_ms.p, S.pos.p, LV, E, S.tid_U.p,
                                                  S.tid_u.p, V);
    else
        k_vfield_node<float><<<gw, 128, 0, st>>>(P, nn, S.nd_pb.p, S.nd_pe.p, S.nd_ms.p, S.pos.p, LV, E, S.tid_U.p,
                                                 S.tid_u.p, V);
    TG_TRY(launched(S));
    for (int L = 0; L <= S.depth; L++) {
        const int64_t first = S.level_off[L], count = S.level_off[L + 1] - S.level_off[L];
        if (count <= 0) continue;
        k_vfield_down<<<(int)((count + 127) / 128), 128, 0, st>>>(first, count, S.nd_parent.p, V, Vtot);
        TG_TRY(launched(S));
    }
    const int32_t nleaves = (int32_t)S.st.leaves;
    if (nleaves > 0) {
        const bool f64 = S.prm.precision == TG_PREC_F64;
        if (S.prm.leaf_max <= 64) {
            if (f64)
                k_tidal_leaf<double, 64, false><<<nleaves, 64, 0, st>>>(P, S.idx.p, nleaves, S.nd_pb.p, S.nd_pe.p, S.nd_ms.p,
                                                                 S.pos.p, LV, E, S.nd_L.p, S.tid_U.p, Vtot, S.tid_u.p, S.tid_o.p);
            else
                k_tidal_leaf<float, 64, false><<<nleaves, 64, 0, st>>>(P, S.idx.p, nleaves, S.nd_pb.p, S.nd_pe.p, S.nd_ms.p,
                                                                S.pos.p, LV, E, S.nd_L.p, S.tid_U.p, Vtot, S.tid_u.p, S.tid_o.p);
        } else {
            if (f64)
                k_tidal_leaf<double, 128, true><<<nleaves, 128, 0, st>>>(P, S.idx.p, nleaves, S.nd_pb.p, S.nd_pe.p,
                                                                   S.nd_ms.p, S.pos.p, LV, E, S.nd_L.p, S.tid_U.p,
                                                                   Vtot, S.tid_u.p, S.tid_o.p);
            else
                k_tidal_leaf<float, 128, true><<<nleaves, 128, 0, st>>>(P, S.idx.p, nleaves, S.nd_pb.p, S.nd_pe.p,
                                                                  S.nd_ms.p, S.pos.p, LV, E, S.nd_L.p, S.tid_U.p,
                                                                  Vtot, S.tid_u.p, S.tid_o.p);
        }
        TG_TRY(launched(S));
        if (S.prm.leaf_max <= 64) {
            if (f64)
                k_tidal_pp<double><<<nleaves, 128, 0, st>>>(P, S.idx.p, S.nd_pb.p, S.nd_pe.p, S.pos.p, LV, S.tid_u.p,
                                                            S.tid_o.p);
            else
                k_tidal_pp<float><<<nleaves, 128, 0, st>>>(P, S.idx.p, S.nd_pb.p, S.nd_pe.p, S.pos.p, LV, S.tid_u.p,
                                                           S.tid_o.p);
            TG_TRY(launched(S));
        }
        if (S.prm.ewald && S.prm.leaf_max <= 64)
            TG_TRY(f64 ? tidal_ewald<double>(S, P, LV, E, st) : tidal_ewald<float>(S, P, LV, E, st));
    }
    k_scatter_axpy3<<<gn, 256, 0, st>>>(n, S.pos.p, c, S.tid_o.p, acc);
    TG_TRY(launched(S));
    return TG_OK;
}

} // namespace tg
