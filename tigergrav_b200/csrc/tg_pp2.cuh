/*
 * tg_pp2.cuh -- PP direct (gravity_PP_direct, src/gravity.cpp:171-300) for the
 * FP32 path, leaf_max <= 64.  Included by tg_gravity.cu after tg_pp.cuh.
 *
 * One block of four warps per sink leaf and share of its source list stages
 * source leaves in shared memory and runs them against the leaf's sinks, in one
 * of two kernels: k_pp_short shares each stage among the warps, k_pp_long gives
 * every warp its own source leaves (the rule is at pp_direct, tg_gravity.cu).
 *
 * Positions are staged in units of 2^-32 of the box (exact powers of two are
 * put back at the end), so staging is a subtraction and a conversion.  Three
 * kinds of source leaves, told apart per leaf from the particle bounding boxes
 * (nearest image):
 *   near  -- a gap to the sink leaf's box below max(2 (its diagonal + 2), h):
 *            split into a multiple of 2^16 and a remainder, both exact in FP32,
 *            so that dX = (hi_i - hi_j) + (lo_i - lo_j) is the reference's
 *            correctly rounded FP32 separation (src/gravity.cpp:223), bit for
 *            bit; softened pairs corrected to the reference's spline.
 *   far   -- every pair at least max(2 |a_i|, h) apart (a_i: the sink's offset
 *            from its leaf centre): offsets from the sink leaf centre rounded
 *            to FP32 once, dX = a_i - b_j in one subtraction.  Its error is at
 *            most 2^-24 (|a_i| + |b_j| + |dX|) <= 1.5 2^-23 |dX| (3 ulp of dX;
 *            the reference's conversion gives 0.5 ulp), and no pair is
 *            softened, so neither the clamp nor the spline check is needed.
 *   wrap  -- offsets that may exceed the int32 range of the two forms (sources
 *            about half a box from the sink leaf, in small boxes at small
 *            theta): per pair from the raw positions with the reference's wrap.
 * The far form costs one packed FP32x2 addition per axis for two pairs where
 * the split form costs three, and reads four sources per 16-byte load; at the
 * 256^3 clustered workload nearly all PP pairs are far.  Sums accumulate in
 * FP32 over groups of 16 interactions (near) or 32 (far), folded into
 * Kahan-compensated totals.
 */
#pragma once

constexpr int PPB_T = 128;     /* threads per block */
constexpr int PPB_W = PPB_T / 32;
constexpr int PPB_SHARES = 16; /* shares of a list, at most */

__device__ __forceinline__ uint32_t lanemask_lt_pp() {
    uint32_t r;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(r));
    return r;
}

/* a source leaf as the selection reads it: one 32-byte sector */
struct __align__(32) PPRec {
    int4 a; /* first particle, particles, box centre x, y (fixed point) */
    int4 b; /* box centre z, half widths x, y, z (float bits, fixed-point units, rounded up) */
};

__global__ void k_pp_records(int64_t nn, const int32_t *__restrict__ pb, const int32_t *__restrict__ pe,
                             const int32_t *__restrict__ child0, const int32_t *__restrict__ aabb,
                             PPRec *__restrict__ rec) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nn || child0[i] >= 0) return; /* only leaves are read */
    const int32_t n = pe[i] - pb[i];
    int32_t c[3] = {0, 0, 0};
    float h[3] = {0.0f, 0.0f, 0.0f};
    if (n > 0)
        for (int d = 0; d < 3; d++) {
            const uint32_t w = (uint32_t)aabb[6 * i + 3 + d] - (uint32_t)aabb[6 * i + d];
            c[d] = (int32_t)((uint32_t)aabb[6 * i + d] + (w >> 1));
            h[d] = __uint2float_ru((w >> 1) + 1u);
        }
    PPRec r;
    r.a = make_int4(pb[i], n, c[0], c[1]);
    r.b = make_int4(c[2], __float_as_int(h[0]), __float_as_int(h[1]), __float_as_int(h[2]));
    rec[i] = r;
}

/* what the selection of a sink leaf's sources needs of the sink leaf */
struct PPSel {
    int32_t c[3];      /* box centre, fixed point */
    int32_t x[3];      /* the leaf centre that offsets are taken from */
    float h[3];        /* half widths, fixed-point units */
    float gmin2, lim;  /* the far criterion, squared; the largest |source centre - x| + half width of near and far */
};
__device__ __forceinline__ PPSel ppb_sel(const GParams &P, const PPRec &me, const int32_t *Xr, uint32_t amag) {
    PPSel S;
    S.x[0] = Xr[0], S.x[1] = Xr[1], S.x[2] = Xr[2];
    S.c[0] = me.a.z, S.c[1] = me.a.w, S.c[2] = me.b.x;
    S.h[0] = __int_as_float(me.b.y), S.h[1] = __int_as_float(me.b.z), S.h[2] = __int_as_float(me.b.w);
    /* a source leaf is far when its box is at least max(2 (diagonal + 2), h + 2) away */
    const float diag = 2.000002f * sqrtf(S.h[0] * S.h[0] + S.h[1] * S.h[1] + S.h[2] * S.h[2]);
    const float gmin = fmaxf(2.0f * (diag + 4.0f), (float)(P.h * 4294967296.0) * 1.000001f + 4.0f);
    S.gmin2 = gmin * gmin;
    S.lim = 2147480000.0f - (float)amag * 1.000001f; /* |a_i - b_j| < 2^31 on each axis */
    return S;
}

/* whether a source leaf is far: FP32, rounded so that the gap is never overestimated */
__device__ __forceinline__ bool ppb_is_far(const PPSel &S, int4 ra, int4 rb, bool per) {
    const int32_t rc[3] = {ra.z, ra.w, rb.x};
    const int32_t rh[3] = {rb.y, rb.z, rb.w};
    float g2 = 0.0f;
#pragma unroll
    for (int d = 0; d < 3; d++) {
        float s;
        if (per) s = fabsf(__int2float_rn((int32_t)((uint32_t)S.c[d] - (uint32_t)rc[d])));
        else s = fabsf(__ll2float_rn((long long)S.c[d] - rc[d]));
        const float g = fmaxf(0.0f, s * 0.999999f - (S.h[d] + __int_as_float(rh[d])) * 1.000001f - 4.0f);
        g2 = fmaf(g, g, g2);
    }
    return g2 * 0.999999f >= S.gmin2;
}
/* the kind of a source leaf: 0 near, 1 far, 2 wrap (the offset never underestimated) */
__device__ __forceinline__ int ppb_kind(const PPSel &S, int4 ra, int4 rb, bool per) {
    const int32_t rc[3] = {ra.z, ra.w, rb.x};
    const int32_t rh[3] = {rb.y, rb.z, rb.w};
    float ext = 0.0f;
#pragma unroll
    for (int d = 0; d < 3; d++) {
        float o;
        if (per) o = fabsf(__int2float_rn((int32_t)((uint32_t)S.x[d] - (uint32_t)rc[d])));
        else o = fabsf(__ll2float_rn((long long)S.x[d] - rc[d]));
        ext = fmaxf(ext, o * 1.000001f + __int_as_float(rh[d]));
    }
    if (ext >= S.lim) return 2;
    return ppb_is_far(S, ra, rb, per) ? 1 : 0;
}

/* blockIdx.y's share [l0, l1) of a list */
__device__ __forceinline__ void ppb_share(int32_t len, int32_t &l0, int32_t &l1) {
    l0 = (int32_t)((int64_t)len * blockIdx.y / gridDim.y);
    l1 = (int32_t)((int64_t)len * (blockIdx.y + 1) / gridDim.y);
}
/* h^2 in units of 2^-64 */
__device__ __forceinline__ float ppb_h2(const GParams &P) { return (float)(P.h * P.h) * 1.8446744073709552e19f; }

/* particle y into slot q of a stage (near: SrcPair hx.x hx.y hy.x ... lz.y; far:
 * FarQuad x[4] y[4] z[4], its offset from Xr negated, within the int32 range;
 * wrap: as it is) */
__device__ __forceinline__ void ppb_put(float *sf, int q, int4 y, const int32_t *Xr, int pass) {
    if (pass == 2) {
        reinterpret_cast<int4 *>(sf)[q] = y;
        return;
    }
    const int32_t a0 = (int32_t)((uint32_t)Xr[0] - (uint32_t)y.x);
    const int32_t a1 = (int32_t)((uint32_t)Xr[1] - (uint32_t)y.y);
    const int32_t a2 = (int32_t)((uint32_t)Xr[2] - (uint32_t)y.z);
    if (pass == 0) {
        float *e = sf + (q >> 1) * 12 + (q & 1);
        pp_split(a0, e[0], e[6]);
        pp_split(a1, e[2], e[8]);
        pp_split(a2, e[4], e[10]);
    } else {
        float *e = sf + (q >> 2) * 12 + (q & 3);
        e[0] = __int2float_rn(a0);
        e[4] = __int2float_rn(a1);
        e[8] = __int2float_rn(a2);
    }
}
/* pad a stage of `used` sources to a whole pair (near) or quad (far), i = 0..2:
 * a source at 1e30 gives exactly zero terms */
__device__ __forceinline__ void ppb_pad(float *sf, int used, int i, int pass) {
    if (pass == 0 && i == 0 && (used & 1)) {
        float *e = sf + (used >> 1) * 12 + 1;
        e[0] = -1.0e30f;
        e[2] = e[4] = e[6] = e[8] = e[10] = 0.0f;
    }
    if (pass == 1 && used + i < ((used + 3) & ~3)) {
        float *e = sf + ((used + i) >> 2) * 12 + ((used + i) & 3);
        e[0] = -1.0e30f;
        e[4] = e[8] = 0.0f;
    }
}

/* four staged sources in the far form: negated FP32 offsets, one 16-byte
 * load per axis for four interactions */
struct __align__(16) FarQuad {
    float4 x, y, z;
};

/* two far sources (packed): 2 interactions, no softening possible */
__device__ __forceinline__ void ppb_far2(const float2 &ax, const float2 &ay, const float2 &az, float2 sx, float2 sy,
                                         float2 sz, PPAcc &a) {
    const float2 dx = __fadd2_rn(ax, sx), dy = __fadd2_rn(ay, sy), dz = __fadd2_rn(az, sz);
    const float2 r2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __fmul2_rn(dz, dz)));
    const float2 rinv = make_float2(rsqrt_ftz(r2.x), rsqrt_ftz(r2.y));
    const float2 f = __fmul2_rn(__fmul2_rn(rinv, rinv), rinv);
    a.tp = __fadd2_rn(a.tp, rinv);
    a.t0 = __ffma2_rn(dx, f, a.t0);
    a.t1 = __ffma2_rn(dy, f, a.t1);
    a.t2 = __ffma2_rn(dz, f, a.t2);
}
__device__ __forceinline__ void ppb_far4(const float2 &ax, const float2 &ay, const float2 &az, const FarQuad &s,
                                         PPAcc &a) {
    const float4 x = s.x, y = s.y, z = s.z;
    ppb_far2(ax, ay, az, make_float2(x.x, x.y), make_float2(y.x, y.y), make_float2(z.x, z.y), a);
    ppb_far2(ax, ay, az, make_float2(x.z, x.w), make_float2(y.z, y.w), make_float2(z.z, z.w), a);
}

/* near source pairs [q, q + n) with r^2 <= h^2: the reference's softened
 * kernel (box units) in place of the clamped 1/r terms */
__device__ __noinline__ void ppb_soft_fix(const GParams &P, float h2, const SrcPair *sy, int q, int n, const SinkHL &A,
                                          PPAcc &a) {
    const float u = 2.3283064365386963e-10f; /* 2^-32 */
    const float hinv = rsqrt_ftz(h2);
    const float hinv3 = hinv * hinv * hinv;
    for (int e = 2 * q; e < 2 * (q + n); e++) {
        float2 dx, dy, dz;
        pp_sep2(A, sy[e >> 1], dx, dy, dz);
        const bool o = e & 1;
        const float x = o ? dx.y : dx.x, y = o ? dy.y : dy.x, z = o ? dz.y : dz.x;
        const float r2 = fmaf(x, x, fmaf(y, y, z * z));
        if (r2 <= h2) {
            const float d[3] = {x * u, y * u, z * u};
            float f, p;
            pp_direct_pair<float>(P, d, f, p);
            f *= u * u * u;
            a.tp.x += p * u - hinv;
            a.t0.x = fmaf(x, f - hinv3, a.t0.x);
            a.t1.x = fmaf(y, f - hinv3, a.t1.x);
            a.t2.x = fmaf(z, f - hinv3, a.t2.x);
        }
    }
}

/* a sink against the far quads [q, q1) of a stage */
__device__ __forceinline__ void ppb_far_run(const FarQuad *st, int q, int q1, const float2 &ax, const float2 &ay,
                                            const float2 &az, PPAcc &a) {
    for (; q + 8 <= q1; q += 8) {
#pragma unroll
        for (int u = 0; u < 8; u++) ppb_far4(ax, ay, az, st[q + u], a);
        a.fold();
    }
    if (q < q1) {
        for (; q < q1; q++) ppb_far4(ax, ay, az, st[q], a);
        a.fold();
    }
}
/* a sink against the near pairs [q, q1) of a stage */
__device__ __forceinline__ void ppb_near_run(const GParams &P, float h2, const SrcPair *sp, int q, int q1,
                                             const SinkHL &A, PPAcc &a) {
    for (; q + 8 <= q1; q += 8) {
        float rmin = 3.0e38f;
#pragma unroll
        for (int u = 0; u < 8; u++) pp_pair2(A, sp[q + u], h2, rmin, a);
        if (rmin <= h2) ppb_soft_fix(P, h2, sp, q, 8, A, a);
        a.fold();
    }
    if (q < q1) {
        float rmin = 3.0e38f;
        for (int u = q; u < q1; u++) pp_pair2(A, sp[u], h2, rmin, a);
        if (rmin <= h2) ppb_soft_fix(P, h2, sp, q, q1 - q, A, a);
        a.fold();
    }
}
/* a sink against the wrap particles [q, q1) of a stage: the arithmetic of the near
 * form with the separation converted from the wrapped difference, every pair folded */
__device__ __forceinline__ void ppb_wrap_run(const GParams &P, float h2, const int4 *st, int q, int q1, int4 x,
                                             bool per, PPAcc &a) {
    const float u = 2.3283064365386963e-10f; /* 2^-32 */
    for (; q < q1; q++) {
        const int4 y = st[q];
        float d[3];
        if (per) {
            d[0] = __int2float_rn((int32_t)((uint32_t)x.x - (uint32_t)y.x));
            d[1] = __int2float_rn((int32_t)((uint32_t)x.y - (uint32_t)y.y));
            d[2] = __int2float_rn((int32_t)((uint32_t)x.z - (uint32_t)y.z));
        } else {
            d[0] = __ll2float_rn((long long)x.x - y.x);
            d[1] = __ll2float_rn((long long)x.y - y.y);
            d[2] = __ll2float_rn((long long)x.z - y.z);
        }
        const float r2 = fmaf(d[0], d[0], fmaf(d[1], d[1], d[2] * d[2]));
        float p = rsqrt_ftz(fmaxf(r2, h2)), f = p * p * p;
        if (r2 <= h2) { /* softened, in box units */
            const float b[3] = {d[0] * u, d[1] * u, d[2] * u};
            pp_direct_pair<float>(P, b, f, p);
            p *= u;
            f *= u * u * u;
        }
        a.tp.x = p;
        a.t0.x = d[0] * f;
        a.t1.x = d[1] * f;
        a.t2.x = d[2] * f;
        a.fold();
    }
}

/* the sums v of sink i (2^-32 units) to the result, or to this share's slot */
__device__ __forceinline__ void ppb_out(const GParams &P, double *v, int64_t i, const double *__restrict__ far,
                                        float4 *__restrict__ acc, double *__restrict__ part, int64_t n) {
    v[0] *= -P.m_d * 4294967296.0; /* 1/r times 2^32, dX/r^3 times 2^64 */
#pragma unroll
    for (int q = 1; q < 4; q++) v[q] *= -P.m_d * 18446744073709551616.0;
    if (part) {
        double *o = part + 4 * ((int64_t)blockIdx.y * n + i);
#pragma unroll
        for (int q = 0; q < 4; q++) o[q] = v[q];
    } else {
        const double *fr = far + 4 * i;
        acc[i] = make_float4((float)(fr[0] + v[0] - P.phi_self), (float)(fr[1] + v[1]), (float)(fr[2] + v[2]),
                             (float)(fr[3] + v[3]));
    }
}

/* far: the FP64 sums (phi, g) of L2P, PC and the Ewald kernels from
 * k_leaf<float, 64, false>.  With part == nullptr (gridDim.y == 1) acc receives
 * far + PP_direct - phi_self; else block (leaf, s) writes the sums over the
 * s-th of gridDim.y shares of the list to part[s][sink] and k_pp_reduce adds
 * them.  Launch of both kernels: blocks of PPB_T threads, grid = (nleaves, shares). */

/* ---- short lists: the block's warps share each stage ---- */

constexpr int PPS_STAGE = 512; /* staged source particles per pass */
constexpr int PPS_META = 64;   /* staged source leaves per pass, at most */
constexpr int PPS_MINB = 10;

/* a stage with offsets beyond the range of the near and far forms: this copy's
 * share, per pair from the raw positions */
__device__ __noinline__ void pps_wrap_stage(const GParams &P, const int32_t *m_start, const int32_t *m_pb, int nmeta,
                                            const int4 *pos, int phase, int C, int4 x, bool per, PPAcc &a) {
    const float u = 2.3283064365386963e-10f; /* 2^-32 */
    for (int k = 0; k < nmeta; k++) {
        for (int32_t q = m_start[k]; q < m_start[k + 1]; q++) {
            if (q % C != phase) continue;
            const int4 y = pos[m_pb[k] + (q - m_start[k])];
            const float d[3] = {sep<float>(x.x, y.x, per), sep<float>(x.y, y.y, per), sep<float>(x.z, y.z, per)};
            float f, p;
            pp_direct_pair<float>(P, d, f, p);
            f *= u * u; /* box units to 2^-32 units: p 2^-32, f dX 2^-64 */
            a.tp.x = p * u;
            a.t0.x = d[0] * f;
            a.t1.x = d[1] * f;
            a.t2.x = d[2] * f;
            a.fold();
        }
    }
}

/*
 * One block per sink leaf and share of its list.  A leaf of ns sinks runs
 * C = PPB_T / ns copies of them (thread t: sink t % ns, copy t / ns), copy p
 * takes the p-th of C contiguous shares of each stage, and the copies are added
 * in a fixed order.  Warp 0 picks whole source leaves, one warp copies a leaf,
 * all warps read the stage: with a few dozen leaves in a list this splits them
 * evenly, where whole leaves per warp leave the block waiting for its slowest
 * warp.  48 registers and 10 blocks per SM (a third pass for wrap leaves, as
 * k_pp_long has it, costs spills: 4.8 ms for 4.1 at 128^3 theta 0.7).
 */
__global__ void __launch_bounds__(PPB_T, PPS_MINB)
    k_pp_short(GParams P, const int32_t *__restrict__ leaves, const int32_t *__restrict__ pb,
               const int32_t *__restrict__ pe, const MSrc *__restrict__ ms, const PPRec *__restrict__ rec,
               const int4 *__restrict__ pos, ListView LV, const double *__restrict__ far, float4 *__restrict__ acc,
               double *__restrict__ part, int64_t n) {
    __shared__ __align__(16) SrcPair stage[PPS_STAGE / 2]; /* the far form (FarQuad) uses the first half */
    __shared__ int32_t m_start[PPS_META + 1], m_pb[PPS_META];
    __shared__ int32_t s_nmeta, s_used, s_cursor;
    __shared__ uint32_t s_amag, s_bmag;
    __shared__ double red[PPB_T][4];
    const int t = threadIdx.x, lane = t & 31;
    const bool per = P.ewald != 0;
    const float h2 = ppb_h2(P);
    const int32_t leaf = leaves[blockIdx.x];
    const int32_t b = pb[leaf], ns = pe[leaf] - b;
    if (ns <= 0) return;
    const int C = PPB_T / ns;
    const int sidx = t % ns, phase = t / ns;
    const bool active = phase < C;
    const int32_t Xr[3] = {ms[leaf].x[0], ms[leaf].x[1], ms[leaf].x[2]};
    const int4 xi = pos[b + sidx];
    SinkHL A;
    float2 ax, ay, az;
    uint32_t amag = 0;
    {
        float h, l;
        int32_t o = rel_off(xi.x, Xr[0], per, amag);
        pp_split(o, h, l);
        A.hx = f2(h), A.lx = f2(l), ax = f2(__int2float_rn(o));
        o = rel_off(xi.y, Xr[1], per, amag);
        pp_split(o, h, l);
        A.hy = f2(h), A.ly = f2(l), ay = f2(__int2float_rn(o));
        o = rel_off(xi.z, Xr[2], per, amag);
        pp_split(o, h, l);
        A.hz = f2(h), A.lz = f2(l), az = f2(__int2float_rn(o));
    }
    if (t == 0) s_amag = 0u;
    __syncthreads();
    atomicMax(&s_amag, amag);
    PPAcc a;
    a.load(make_float4(0.0f, 0.0f, 0.0f, 0.0f), make_float4(0.0f, 0.0f, 0.0f, 0.0f));
    int32_t l0, l1;
    ppb_share(LV.len[TG_PP_D][leaf], l0, l1);
    const int32_t *lst = LV.pool[TG_PP_D] + LV.off[TG_PP_D][leaf];
    float *sf = reinterpret_cast<float *>(stage);
    for (int pass = 0; pass < 2; pass++) { /* 0: near leaves (split form), 1: far leaves */
        if (t == 0) s_cursor = l0;
        __syncthreads();
        for (;;) {
            /* warp 0 picks the next whole source leaves of this kind that fit */
            if (t < 32) {
                const PPSel S = ppb_sel(P, rec[leaf], Xr, 0u);
                int nmeta = 0, used = 0, cur = s_cursor;
                while (cur < l1 && nmeta + 32 <= PPS_META) {
                    const int e = cur + lane;
                    int sn = 0, sb = 0;
                    if (e < l1) {
                        const PPRec &r = rec[lst[e]];
                        const int4 ra = r.a, rb = r.b;
                        sb = ra.x;
                        sn = ra.y;
                        if (ppb_is_far(S, ra, rb, per) != (pass == 1)) sn = 0;
                    }
                    int inc = sn;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const int v = __shfl_up_sync(0xffffffffu, inc, o);
                        if (lane >= o) inc += v;
                    }
                    const int navail = min(32, l1 - cur);
                    const int take = min(__popc(__ballot_sync(0xffffffffu, used + inc <= PPS_STAGE)), navail);
                    const bool take_me = lane < take && sn > 0;
                    const uint32_t rm = __ballot_sync(0xffffffffu, take_me);
                    if (take_me) {
                        const int k = nmeta + __popc(rm & lanemask_lt_pp());
                        m_start[k] = used + inc - sn;
                        m_pb[k] = sb;
                    }
                    nmeta += __popc(rm);
                    if (take > 0) used += __shfl_sync(0xffffffffu, inc, take - 1);
                    cur += take;
                    if (take < navail) break; /* the stage is full */
                }
                if (lane == 0) {
                    s_nmeta = nmeta;
                    s_used = used;
                    s_cursor = cur;
                    m_start[nmeta] = used;
                    s_bmag = 0u;
                }
            }
            __syncthreads();
            const int used = s_used, nmeta = s_nmeta;
            if (used == 0) break; /* the list is exhausted for this kind */
            /* warp w copies the source leaves w, w + 4, ...: its lanes take
             * consecutive particles of one leaf (coalesced loads) */
            uint32_t bmag = 0;
            for (int k = t >> 5; k < nmeta; k += PPB_W)
                for (int q = m_start[k] + lane; q < m_start[k + 1]; q += 32) {
                    const int4 y = pos[m_pb[k] + (q - m_start[k])];
                    rel_off(y.x, Xr[0], per, bmag);
                    rel_off(y.y, Xr[1], per, bmag);
                    rel_off(y.z, Xr[2], per, bmag);
                    ppb_put(sf, q, y, Xr, pass);
                }
            if (t < 3) ppb_pad(sf, used, t, pass);
            bmag = __reduce_max_sync(0xffffffffu, bmag);
            if (lane == 0) atomicMax(&s_bmag, bmag);
            __syncthreads();
            const int nq = pass == 0 ? (used + 1) >> 1 : (used + 3) >> 2; /* pairs (near) or quads (far) */
            /* both forms give the int32-wrapped (nearest image) separation
             * when every |a_i - b_j| < 2^31 */
            const bool fits = (unsigned long long)s_amag + s_bmag < (1ull << 31);
            if (active) {
                /* copy `phase` takes the contiguous source pairs or quads [q0, q1) */
                const int q0 = nq * phase / C, q1 = nq * (phase + 1) / C;
                if (pass == 0 && fits) ppb_near_run(P, h2, stage, q0, q1, A, a);
                else if (pass == 1 && fits) ppb_far_run(reinterpret_cast<const FarQuad *>(stage), q0, q1, ax, ay, az, a);
                else pps_wrap_stage(P, m_start, m_pb, nmeta, pos, phase, C, xi, per, a);
            }
            __syncthreads(); /* the stage is rewritten next */
        }
    }
    float4 s, c;
    a.store(s, c);
    red[t][0] = (double)s.x - (double)c.x;
    red[t][1] = (double)s.y - (double)c.y;
    red[t][2] = (double)s.z - (double)c.z;
    red[t][3] = (double)s.w - (double)c.w;
    __syncthreads();
    if (t < ns) {
        double v[4] = {0.0, 0.0, 0.0, 0.0};
        for (int p = 0; p < C; p++)
#pragma unroll
            for (int q = 0; q < 4; q++) v[q] += red[t + p * ns][q];
        ppb_out(P, v, b + t, far, acc, part, n);
    }
}

/* ---- long lists: every warp its own source leaves ---- */

#ifndef PPL_STAGE
#define PPL_STAGE 256          /* a warp's staged far particles; half as many near ones */
#endif
constexpr int PPL_META = 32;   /* a warp's staged source leaves, at most */
constexpr int PPL_PARTS = 3;   /* parts of at most 64 sinks */
#ifndef PPL_MINB
#define PPL_MINB 7
#endif

/* size of the next part of `left` sinks: 32, 16 or 8 fill the lanes, the rest as
 * it is where that wastes few (26 = 16 + 10, 43 = 32 + 8 + 3, 58 = 32 + 16 + 10) */
__host__ __device__ __forceinline__ int ppl_part(int left) {
    if (left >= 32) return 32;
    if (left > 16 && left < 27) return 16;
    if (left == 11 || left == 12) return 8;
    return left;
}

/*
 * Each warp takes every fourth source leaf of the list (QUARTER: a quarter of
 * every leaf), stages whole leaves (up to PPL_STAGE particles) in its own area
 * and runs them against all sinks, so no warp waits for another until the end.
 * The sinks are cut into parts of at most 32 (ppl_part): a part of p sinks runs
 * on p lanes times 32 / p copies, which share the stage.  24 to 64 sinks keep 97%
 * of the lanes busy (a lane per sink and copy over the whole block keeps 86%),
 * and the lanes of a full part read the same staged source (one shared-memory
 * wavefront instead of 2.8).  Each lane's compensated totals wait in shared
 * memory between stages and are added in FP64 in a fixed order at the end.
 *
 * What bounds it: instruction issue.  A far interaction is 12 packed operations
 * and 2 rsqrt for two pairs.  256^3 theta 0.19: 654 ms against 731 ms of
 * k_pp_short (7 blocks per SM; 8: 658, 9 spill: 704; warps sharing one stage of
 * 1024 behind block barriers: 680; two sinks per thread: 844).
 */
template <bool QUARTER>
__global__ void __launch_bounds__(PPB_T, PPL_MINB)
    k_pp_long(GParams P, const int32_t *__restrict__ leaves, const int32_t *__restrict__ pb,
              const int32_t *__restrict__ pe, const MSrc *__restrict__ ms, const PPRec *__restrict__ rec,
              const int4 *__restrict__ pos, ListView LV, const double *__restrict__ far, float4 *__restrict__ acc,
              double *__restrict__ part, int64_t n) {
    __shared__ __align__(16) FarQuad s_stage[PPB_W][PPL_STAGE / 4]; /* near: PPL_STAGE / 4 SrcPairs, as large */
    __shared__ float4 kst[PPL_PARTS][2][PPB_T]; /* each lane's compensated sums, and their errors */
    __shared__ int4 s_off[64];                  /* the sinks' offsets from the leaf centre */
    __shared__ int32_t s_lane[PPL_PARTS][32];   /* per part and lane: sink | copy << 8, or -1 */
    __shared__ int4 s_part[PPL_PARTS];          /* first sink, sinks, copies, 16-bit reciprocal of the copies */
    __shared__ int32_t s_nparts;
    __shared__ int2 s_meta[PPB_W][PPL_META];    /* a staged leaf's first slot and first particle */
    __shared__ uint32_t s_amag;
    __shared__ PPSel s_sel;
    static_assert(sizeof(SrcPair) == sizeof(FarQuad), "one stage for both forms");
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    const bool per = P.ewald != 0;
    const float h2 = ppb_h2(P);
    const int32_t leaf = leaves[blockIdx.x];
    const int32_t b = pb[leaf], ns = pe[leaf] - b;
    if (ns <= 0) return;
    const int32_t Xr[3] = {ms[leaf].x[0], ms[leaf].x[1], ms[leaf].x[2]};
    if (t == 0) s_amag = 0u;
    if (w < PPL_PARTS) { /* warp w: part w */
        int s0 = 0, p = ppl_part(ns), k = 0;
        while (k < w && s0 + p < ns) {
            s0 += p;
            p = ppl_part(ns - s0);
            k++;
        }
        if (k == w) {
            const int nsub = 32 / p, sub = lane / p;
            s_lane[w][lane] = sub < nsub ? (s0 + lane - sub * p) | sub << 8 : -1;
            s_part[w] = make_int4(s0, p, nsub, 65536 / nsub + 1);
            if (s0 + p == ns) s_nparts = w + 1;
        }
    }
    __syncthreads();
    if (t < ns) {
        const int4 x = pos[b + t];
        uint32_t mag = 0;
        s_off[t] = make_int4(rel_off(x.x, Xr[0], per, mag), rel_off(x.y, Xr[1], per, mag), rel_off(x.z, Xr[2], per, mag), 0);
        atomicMax(&s_amag, mag);
    }
#pragma unroll
    for (int k = 0; k < PPL_PARTS; k++) kst[k][0][t] = kst[k][1][t] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    __syncthreads();
    if (t == 0) s_sel = ppb_sel(P, rec[leaf], Xr, s_amag);
    __syncthreads();
    /* this block's share of the list; warp w takes the entries l0 + w, l0 + w + 4, ... of it */
    int32_t l0, l1;
    ppb_share(LV.len[TG_PP_D][leaf], l0, l1);
    constexpr int step = QUARTER ? 1 : PPB_W;
    constexpr int group = QUARTER ? 8 : 32; /* lanes per leaf while staging */
    const int32_t *lst = LV.pool[TG_PP_D] + LV.off[TG_PP_D][leaf] + l0 + (QUARTER ? 0 : w);
    const int32_t nv = QUARTER ? l1 - l0 : (l1 - l0 - w + PPB_W - 1) / PPB_W;
    FarQuad *const stage = s_stage[w];
    float *const sf = reinterpret_cast<float *>(stage);
    const SrcPair *const sp = reinterpret_cast<const SrcPair *>(stage);
    int2 *const meta = s_meta[w];
    bool wrap = false;
    for (int pass = 0; pass < 3; pass++) { /* near, far, wrap */
        if (pass == 2 && !__any_sync(0xffffffffu, wrap)) break; /* the near pass saw none */
        const int room = pass == 1 ? PPL_STAGE : PPL_STAGE / 2;
        int cur = 0;        /* entries read */
        int sn = 0, sb = 0; /* this lane's leaf of the batch read last: particles (0: none left), first particle */
        for (;;) {
            /* the next whole source leaves of this kind that fit */
            int nmeta = 0, used = 0;
            for (;;) {
                if (!__any_sync(0xffffffffu, sn > 0)) {
                    if (cur >= nv) break;
                    if (cur + lane < nv) {
                        const PPSel S = s_sel;
                        const PPRec &r = rec[lst[step * (cur + lane)]];
                        const int4 ra = r.a, rb = r.b;
                        const int kind = ppb_kind(S, ra, rb, per);
                        wrap |= kind == 2;
                        const int q0 = QUARTER ? ra.y * w >> 2 : 0, q1 = QUARTER ? ra.y * (w + 1) >> 2 : ra.y;
                        sb = ra.x + q0;
                        sn = kind == pass ? q1 - q0 : 0;
                    }
                    cur += 32;
                    continue;
                }
                int inc = sn;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int v = __shfl_up_sync(0xffffffffu, inc, o);
                    if (lane >= o) inc += v;
                }
                const uint32_t pend = __ballot_sync(0xffffffffu, sn > 0);
                const int k = nmeta + __popc(pend & lanemask_lt_pp());
                const bool take = sn > 0 && used + inc <= room && k < PPL_META; /* a prefix of the pending lanes */
                if (take) meta[k] = make_int2(used + inc - sn, sb);
                const uint32_t tm = __ballot_sync(0xffffffffu, take);
                if (take) sn = 0;
                nmeta += __popc(tm);
                if (tm) used += __shfl_sync(0xffffffffu, inc, 31 - __clz(tm));
                if (tm != pend) break; /* the stage is full */
            }
            if (used == 0) break; /* the list is exhausted for this kind */
            __syncwarp();
            for (int k = lane / group; k < nmeta; k += 32 / group) {
                /* a group of lanes takes consecutive particles of one leaf (coalesced loads) */
                const int2 me = meta[k];
                const int q1 = k + 1 < nmeta ? meta[k + 1].x : used;
                const int4 *src = pos + me.y - me.x;
                for (int q = me.x + lane % group; q < q1; q += group) ppb_put(sf, q, src[q], Xr, pass);
            }
            if (lane < 3) ppb_pad(sf, used, lane, pass);
            __syncwarp();
            /* the stage's source pairs, quads or particles against every part of the sinks */
            const int nq = pass == 0 ? (used + 1) >> 1 : (pass == 1 ? (used + 3) >> 2 : used);
            for (int k = 0; k < s_nparts; k++) {
                const int me = s_lane[k][lane];
                if (me < 0) continue;
                const int sub = me >> 8, nsub = s_part[k].z, inv = s_part[k].w;
                const int4 o = s_off[me & 255];
                PPAcc a;
                a.load(kst[k][0][t], kst[k][1][t]);
                /* copy sub of nsub: from floor(nq sub / nsub) on, by a 16-bit reciprocal */
                int q = nq * sub * inv >> 16;
                const int q1 = sub + 1 == nsub ? nq : nq * (sub + 1) * inv >> 16;
                if (pass == 1) {
                    ppb_far_run(stage, q, q1, f2(__int2float_rn(o.x)), f2(__int2float_rn(o.y)),
                                f2(__int2float_rn(o.z)), a);
                } else if (pass == 0) {
                    SinkHL A;
                    float h, l;
                    pp_split(o.x, h, l);
                    A.hx = f2(h), A.lx = f2(l);
                    pp_split(o.y, h, l);
                    A.hy = f2(h), A.ly = f2(l);
                    pp_split(o.z, h, l);
                    A.hz = f2(h), A.lz = f2(l);
                    ppb_near_run(P, h2, sp, q, q1, A, a);
                } else {
                    ppb_wrap_run(P, h2, reinterpret_cast<const int4 *>(stage), q, q1, pos[b + (me & 255)], per, a);
                }
                a.store(kst[k][0][t], kst[k][1][t]);
            }
            __syncwarp(); /* the stage is rewritten next */
        }
    }
    /* totals in FP64, in place: the copies of a part within each warp by
     * halving, then the warps in order */
    for (int k = 0; k < s_nparts; k++) {
        double2 *const d0 = reinterpret_cast<double2 *>(kst[k][0]), *const d1 = reinterpret_cast<double2 *>(kst[k][1]);
        const float4 s = kst[k][0][t], c = kst[k][1][t];
        d0[t] = make_double2((double)s.x - (double)c.x, (double)s.y - (double)c.y);
        d1[t] = make_double2((double)s.z - (double)c.z, (double)s.w - (double)c.w);
        const int me = s_lane[k][lane], p = s_part[k].y, nsub = s_part[k].z;
        for (int h = 16; h >= 1; h >>= 1) {
            __syncwarp();
            if (me >= 0 && (me >> 8) < h && (me >> 8) + h < nsub) {
                d0[t].x += d0[t + h * p].x;
                d0[t].y += d0[t + h * p].y;
                d1[t].x += d1[t + h * p].x;
                d1[t].y += d1[t + h * p].y;
            }
        }
    }
    __syncthreads();
    if (t < ns) {
        int k = 0;
        while (k + 1 < s_nparts && t >= s_part[k + 1].x) k++;
        double v[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
        for (int u = 0; u < PPB_T; u += 32) {
            const double2 p = reinterpret_cast<const double2 *>(kst[k][0])[u + t - s_part[k].x];
            const double2 q = reinterpret_cast<const double2 *>(kst[k][1])[u + t - s_part[k].x];
            v[0] += p.x;
            v[1] += p.y;
            v[2] += q.x;
            v[3] += q.y;
        }
        ppb_out(P, v, b + t, far, acc, part, n);
    }
}

/* the shares of the lists, in order: one thread per sink of the leaves */
__global__ void __launch_bounds__(64) k_pp_reduce(GParams P, const int32_t *__restrict__ leaves,
                                                  const int32_t *__restrict__ pb, const int32_t *__restrict__ pe,
                                                  const double *__restrict__ far, const double *__restrict__ part,
                                                  int shares, int64_t n, float4 *__restrict__ acc) {
    const int32_t leaf = leaves[blockIdx.x];
    const int64_t i = (int64_t)pb[leaf] + threadIdx.x;
    if (i >= pe[leaf]) return;
    const double *fr = far + 4 * i;
    double v[4] = {0.0, 0.0, 0.0, 0.0};
    for (int s = 0; s < shares; s++)
#pragma unroll
        for (int q = 0; q < 4; q++) v[q] += part[4 * ((int64_t)s * n + i) + q];
    acc[i] = make_float4((float)(fr[0] + v[0] - P.phi_self), (float)(fr[1] + v[1]), (float)(fr[2] + v[2]),
                         (float)(fr[3] + v[3]));
}
