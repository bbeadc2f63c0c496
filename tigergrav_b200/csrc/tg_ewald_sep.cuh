/*
 * tg_ewald_sep.cuh -- the particle-particle Ewald correction
 * (gravity_PP_ewald, src/gravity.cpp:491-614) split so that a pair costs few
 * images.  Included by tg_gravity.cu.
 *
 * The Ewald sum holds for every split alpha between real and reciprocal space
 * (the reference's kernels take alpha = 2).  The reciprocal part factorises
 * over a sink leaf, so its terms cost next to nothing per pair:
 *     sum_j m H(h) trig(2 pi h.(x_i - x_j)) = H(h) (trig of th_i) x (sums of
 *     cos th_j, sin th_j over the sources),   th = 2 pi h.x,
 * with the source sums taken once per source leaf (k_ewald_sf), added per
 * chunk of a sink's list, and the terms evaluated once per sink particle.  A
 * larger alpha therefore moves work to where it is shared.  In FP32, alpha = 4.5:
 *   - real-space images beyond r = 1 add at most 8e-9 to the force factor
 *     (as images beyond r = 2 do at alpha = 2), and inside r < 1 of a separation
 *     |x_d| <= 1/2 lie at most the nearest image and its 7 mirror neighbours
 *     towards the near corner of the box, ~4 of them on average (~34 at
 *     alpha = 2): no lists of images, no search;
 *   - |h|^2 <= 41 leaves a force tail of 1e-8: 570 vectors (half space) for 61.
 * In FP64, alpha = 5.2: images beyond r = 1 add 1.1e-11 to the force factor, and
 * |h|^2 <= 70 leaves a force tail of 9e-12 (the 61 vectors at alpha = 2 leave
 * 6e-11), for ~4 images instead of ~200.
 *
 * The nearest image and the reciprocal part grow with alpha^2 (8.7 at most in the
 * force of a unit mass for 1.7; their derivatives with alpha^3) and cancel to the
 * periodic correction's ~1, so FP32 rounding of either would show 5 (11) times as
 * much as at alpha = 2.  Both are FP64 in the FP32 path: the nearest image as two
 * polynomials in r^2 of the exact separation (SepNear), phases and source sums from
 * FP64 powers of e^(2 pi i x_d) (SepTrig); only the mirror images, at most 0.13
 * each, are FP32, their erfc from a polynomial good to 2e-9 (SepNear; a third of the
 * cost of erfc and expf, and two instructions fewer than the reference's 7.1.26 form,
 * whose 1.5e-7 showed: force 1.1e-7 over the cube).  Measured error of a pair against FP64, rms over |x_d| < 1/2, 1/4,
 * 1/10, 1/20, with the FP32 output's own rounding:
 *   force     4.6e-8, 2.5e-8, 1.6e-8, 2.1e-8
 *     the FP32 sums at alpha = 2: 5.4e-7, 5.2e-7, 1.7e-7, 2.0e-7
 *     FP32 throughout at alpha = 4.2: 9.4e-7, 2.1e-6, 1.3e-6, 3.6e-7
 *   Jacobian product (of ~10)  5.0e-7, 4.7e-7, 8.6e-7, 7.6e-7
 *     the FP32 sums at alpha = 2: 5.8e-6, 4.2e-6, 3.8e-6, 3.4e-6
 *     FP32 throughout at alpha = 4.2: 2.2e-5, 5.3e-5, 4.8e-5, 1.5e-5
 *
 * The nearest image stays combined with the removal of the direct 1/r
 * (ewald_nearest in FP64), and an interaction with r <= 1e-6 is phi0 alone, as the
 * reference has it (tigergrav/green.hpp:270-273): its reciprocal terms, which
 * the leaf sums include, are subtracted by that pair.
 *
 * Phases are exact: h.x mod 1 is an integer sum of the fixed-point coordinates
 * modulo 2^32 (plus 1/2 per odd h component for the 0.5 offset), or a product of
 * powers of the exact coordinates' phases.
 */
#pragma once

/* (cos, sin) of 2 pi h.x for the up to 64 particles of a leaf, held by a block.
 * FP32 solvers: from the powers 0..HMAX of e^(2 pi i x_d); a run of up to SEP_RUN
 * vectors along z takes three of them and then one multiplication by e^(2 pi i x_z)
 * each (three powers read per vector made shared memory the limit: source and sink
 * sums of 64^3, 423 vectors, 0.18 and 0.41 ms).  The odd row length keeps both lanes
 * over particles and lanes over runs free of bank conflicts.  FP64 solvers (powers
 * to 8: too much shared memory) from the phase. */
template <class T> struct SepTrig;
template <> struct SepTrig<float> {
    static constexpr int K = Sep<float>::HMAX + 1;
    double2 w[64][(3 * K) | 1];
    /* axis d of particle j */
    __device__ __forceinline__ void fill(int j, int d, int4 p) {
        const int32_t x = d == 0 ? p.x : (d == 1 ? p.y : p.z);
        double2 *q = w[j] + d * K, e, a = make_double2(1.0, 0.0);
        sincospi((double)x * 4.656612873077392578125e-10 + 1.0, &e.y, &e.x); /* 2 (x 2^-32 + 1/2) */
        q[0] = a;
#pragma unroll
        for (int k = 1; k < K; k++) {
            a = mul(a, e);
            q[k] = a;
        }
    }
    static __device__ __forceinline__ double2 mul(double2 a, double2 b) {
        return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
    }
    /* the first vector of a run (hx >= 0), and the step to the next */
    __device__ __forceinline__ double2 first(int j, int4 run) const {
        const double2 a = w[j][run.x];
        double2 b = w[j][K + abs(run.y)], c = w[j][2 * K + abs(run.z)];
        if (run.y < 0) b.y = -b.y;
        if (run.z < 0) c.y = -c.y;
        return mul(mul(a, b), c);
    }
    __device__ __forceinline__ double2 step(int j) const { return w[j][2 * K + 1]; }
};
template <> struct SepTrig<double> {
    __device__ __forceinline__ void fill(int, int, int4) {}
    /* pos: the leaf's particles */
    static __device__ __forceinline__ double2 at(int j, const int4 *pos, int4 h) {
        const int4 p = __ldg(&pos[j]);
        uint32_t u = (uint32_t)h.x * (uint32_t)p.x + (uint32_t)h.y * (uint32_t)p.y + (uint32_t)h.z * (uint32_t)p.z;
        u += (uint32_t)(h.x + h.y + h.z) << 31; /* the offset 0.5 of every coordinate */
        double2 cs;
        sincospi((double)(int32_t)u * 4.656612873077392578125e-10, &cs.y, &cs.x); /* 2 x 2^-32 */
        return cs;
    }
};
/* all threads: the particles pos[0, cnt) into trig */
template <class T>
__device__ __forceinline__ void sep_trig(SepTrig<T> &trig, const int4 *__restrict__ pos, int cnt) {
    if constexpr (sizeof(T) == 4) {
        for (int q = threadIdx.x; q < 3 * cnt; q += blockDim.x) trig.fill(q / 3, q % 3, pos[q / 3]);
        __syncthreads();
    }
}

/* source sums: a += m f */
__device__ __forceinline__ void sep_madd(double2 &a, double m, const double2 &f) {
    a.x = fma(m, f.x, a.x);
    a.y = fma(m, f.y, a.y);
}

/* One block per source leaf of some PP_E list: the sums of (cos, sin) over its
 * particles for the vectors [t0, t1), a thread per run (FP32) or vector */
template <class T>
__global__ void __launch_bounds__(128) k_ewald_sf(const int32_t *__restrict__ src, const int32_t *__restrict__ pb,
                                                  const int32_t *__restrict__ pe, const int4 *__restrict__ pos,
                                                  EwaldTables E, int t0, int t1, double2 *__restrict__ sf) {
    __shared__ SepTrig<T> trig;
    const int32_t node = src[blockIdx.x];
    const int32_t b = pb[node], n = pe[node] - b;
    double2 *const row = sf + (int64_t)blockIdx.x * (t1 - t0) - t0;
    sep_trig<T>(trig, pos + b, n);
    if constexpr (sizeof(T) == 4) {
        for (int r = threadIdx.x; r < E.sep_nrun; r += 128) {
            const int4 run = __ldg(&E.sep_run[r]);
            const int t = run.w >> 8, len = run.w & 255;
            if (t >= t1 || t + len <= t0) continue;
            double2 a[SEP_RUN] = {};
            for (int32_t j = 0; j < n; j++) {
                double2 e = trig.first(j, run);
                const double2 z = trig.step(j);
#pragma unroll
                for (int k = 0; k < SEP_RUN; k++) {
                    a[k].x += e.x;
                    a[k].y += e.y;
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
            double2 a = make_double2(0.0, 0.0);
            for (int32_t j = 0; j < n; j++) {
                const double2 q = trig.at(j, pos + b, h);
                a.x += q.x;
                a.y += q.y;
            }
            row[t] = a;
        }
    }
}

/* erfc(alpha r) and e^(-alpha^2 r^2) of a mirror image, 1/2 <= r < 1 */
__device__ __forceinline__ float sep_erfc(const SepNear &K, float r2, float rinv, float &e) {
    e = ex2_ftz(r2 * (float)(-Sep<float>::ALPHA * Sep<float>::ALPHA * 1.4426950408889634));
    const float w = fmaf(2.0f, rinv, -3.0f);
    float p = K.q[SEP_DQ];
#pragma unroll
    for (int k = SEP_DQ - 1; k >= 0; k--) p = fmaf(p, w, K.q[k]);
    return p * e;
}
__device__ __forceinline__ double sep_erfc(const SepNear &, double r2, double rinv, double &e) {
    return t_erfcexp(Sep<double>::ALPHA * (r2 * rinv), &e);
}
/* one image at the displacement d (r2 = |d|^2 < 1): -erfc(alpha r)/r and its force */
template <class T>
__device__ __forceinline__ void sep_image(const SepNear &K, T d0, T d1, T d2, T r2, T &ph, T &gx, T &gy, T &gz) {
    const T rinv = t_rsqrt(r2);
    const T r = r2 * rinv;
    T expfac;
    const T erfc = sep_erfc(K, r2, rinv, expfac);
    const T expfactor = T(Sep<T>::ALPHA * 1.1283791670955126) * r * expfac; /* 2 alpha / sqrt(pi) */
    const T f = (expfactor + erfc) * rinv * rinv * rinv;
    ph -= erfc * rinv;
    gx = fma(-d0, f, gx);
    gy = fma(-d1, f, gy);
    gz = fma(-d2, f, gz);
}

/* the mirror images inside r < 1 of a pair at x, u = x^2 per axis, added to ph and g */
template <class T>
__device__ __forceinline__ void sep_images(const SepNear &K, T x0, T x1, T x2, T u0, T u1, T u2, T &ph, T &gx, T &gy,
                                           T &gz) {
    const T c0 = x0 - copysign(T(1), x0), c1 = x1 - copysign(T(1), x1), c2 = x2 - copysign(T(1), x2);
    const T v0 = c0 * c0, v1 = c1 * c1, v2 = c2 * c2;
    T q;
    q = v0 + u1 + u2;
    if (q < T(1)) sep_image<T>(K, c0, x1, x2, q, ph, gx, gy, gz);
    q = u0 + v1 + u2;
    if (q < T(1)) sep_image<T>(K, x0, c1, x2, q, ph, gx, gy, gz);
    q = u0 + u1 + v2;
    if (q < T(1)) sep_image<T>(K, x0, x1, c2, q, ph, gx, gy, gz);
    q = v0 + v1 + u2;
    if (q < T(1)) sep_image<T>(K, c0, c1, x2, q, ph, gx, gy, gz);
    q = v0 + u1 + v2;
    if (q < T(1)) sep_image<T>(K, c0, x1, c2, q, ph, gx, gy, gz);
    q = u0 + v1 + v2;
    if (q < T(1)) sep_image<T>(K, x0, c1, c2, q, ph, gx, gy, gz);
    q = v0 + v1 + v2;
    if (q < T(1)) sep_image<T>(K, c0, c1, c2, q, ph, gx, gy, gz);
}

/* the sums of one sink over the real-space parts of its PP_E pairs, times m */
template <class T> struct SepPairs;
template <> struct SepPairs<double> {
    double s[4];
    __device__ __forceinline__ void init() { s[0] = s[1] = s[2] = s[3] = 0.0; }
    __device__ __forceinline__ void add(const EwaldTables &E, const SepNear &K, double m, int4 xi, int4 y) {
        const double x[3] = {wrap_sep_d(xi.x, y.x), wrap_sep_d(xi.y, y.y), wrap_sep_d(xi.z, y.z)};
        const double u0 = x[0] * x[0], u1 = x[1] * x[1], u2 = x[2] * x[2], r2 = u0 + u1 + u2;
        if (!(r2 > 1.0e-12)) { /* phi0 alone: take back the reciprocal terms, R0 + R2 r^2 / 2 */
            s[0] += m * ((double)EWALD_PHI0 - E.sep_r0);
            for (int d = 0; d < 3; d++) s[1 + d] += m * (E.sep_r2 * x[d]);
            return;
        }
        double ph = 0.0, gx = 0.0, gy = 0.0, gz = 0.0;
        sep_images<double>(K, x[0], x[1], x[2], u0, u1, u2, ph, gx, gy, gz);
        const double rinv = t_rsqrt(r2);
        double p0, f0;
        ewald_nearest<double>(Sep<double>::ALPHA, r2 * rinv, rinv, p0, f0);
        s[0] += m * (ph + (E.sep_k + p0)); /* sep_k = pi / alpha^2 */
        s[1] += m * fma(x[0], f0, gx);
        s[2] += m * fma(x[1], f0, gy);
        s[3] += m * fma(x[2], f0, gz);
    }
    __device__ __forceinline__ void fold() {}
    __device__ __forceinline__ double get(int q, double) const { return s[q]; }
};
/* FP32: the nearest image in FP64 (plain sums, the force in units of 2^-32), the
 * mirror images in FP32: plain sums over the pairs between two folds (SEP_FOLD,
 * with at most 0.13 per image a rounding of 2e-8, below a pair's own), then
 * compensated ones */
template <> struct SepPairs<float> {
    double s[4];
    float a[4];
    Acc<float> i[4];
    __device__ __forceinline__ void init() {
#pragma unroll
        for (int q = 0; q < 4; q++) {
            s[q] = 0.0;
            a[q] = 0.0f;
            i[q].init(0.0);
        }
    }
    __device__ __forceinline__ void fold() {
#pragma unroll
        for (int q = 0; q < 4; q++) {
            i[q].add(a[q]);
            a[q] = 0.0f;
        }
    }
    __device__ __forceinline__ void add(const EwaldTables &E, const SepNear &K, double, int4 xi, int4 y) {
        const int32_t d0 = (int32_t)((uint32_t)xi.x - (uint32_t)y.x), d1 = (int32_t)((uint32_t)xi.y - (uint32_t)y.y),
                      d2 = (int32_t)((uint32_t)xi.z - (uint32_t)y.z);
        const float w = 2.3283064365386963e-10f; /* 2^-32 */
        const float x0 = __int2float_rn(d0) * w, x1 = __int2float_rn(d1) * w, x2 = __int2float_rn(d2) * w;
        const float u0 = x0 * x0, u1 = x1 * x1, u2 = x2 * x2;
        const double X0 = i2d(d0), X1 = i2d(d1), X2 = i2d(d2);
        if (!(u0 + u1 + u2 > 1.0e-12f)) { /* phi0 alone, as above */
            s[0] += (double)EWALD_PHI0 - E.sep_r0;
            s[1] = fma(E.sep_r2, X0, s[1]);
            s[2] = fma(E.sep_r2, X1, s[2]);
            s[3] = fma(E.sep_r2, X2, s[3]);
            return;
        }
        sep_images<float>(K, x0, x1, x2, u0, u1, u2, a[0], a[1], a[2], a[3]);
        /* t = 8/3 r^2 - 1, r^2 in units of 2^-64 */
        const double t = fma(fma(X0, X0, fma(X1, X1, X2 * X2)), 8.0 / 3.0 * POS_INV * POS_INV, -1.0);
        double p = K.p[SEP_DP], f = K.f[SEP_DF];
#pragma unroll
        for (int k = SEP_DF - 1; k >= 0; k--) f = fma(f, t, K.f[k]);
#pragma unroll
        for (int k = SEP_DP - 1; k >= 0; k--) p = fma(p, t, K.p[k]);
        s[0] += p;
        s[1] = fma(X0, f, s[1]);
        s[2] = fma(X1, f, s[2]);
        s[3] = fma(X2, f, s[3]);
    }
    __device__ __forceinline__ double get(int q, double m) const {
        return m * ((q == 0 ? s[0] : s[q] * POS_INV) + i[q].get());
    }
};

/* The reciprocal part at sink particle j of a leaf (pos) from the leaf's sums src[h] =
 * (sum m cos th_j, sum m sin th_j) (FP32: times w_h), share grp of 4: with
 * w_h = 2 exp(-pi^2 h^2 / alpha^2) / h^2 (both of +-h),
 *   phi -= sum w_h / pi cos(th_i - th_j),  g -= sum 2 w_h h sin(th_i - th_j). */
template <class T>
__device__ __forceinline__ void sep_eval(const EwaldTables &E, const SepTrig<T> &trig, const double2 *src, int grp, int j,
                                         const int4 *pos, double &phi, double *g) {
    double ph = 0.0, gx = 0.0, gy = 0.0, gz = 0.0;
    if constexpr (sizeof(T) == 4) {
        const double2 z = trig.step(j);
        for (int r = grp; r < E.sep_nrun; r += 4) {
            const int4 run = __ldg(&E.sep_run[r]);
            const int t = run.w >> 8, len = run.w & 255;
            double2 e = trig.first(j, run);
            double s = 0.0, h = run.z;
            for (int k = 0; k < len; k++) {
                const double2 A = src[t + k];
                ph = fma(e.x, A.x, fma(e.y, A.y, ph));
                const double f = e.y * A.x - e.x * A.y;
                s += f;
                gz = fma(f, h, gz);
                h += 1.0;
                e = trig.mul(e, z);
            }
            gx = fma(s, (double)run.x, gx);
            gy = fma(s, (double)run.y, gy);
        }
    } else {
        for (int t = grp; t < Sep<T>::N; t += 4) {
            const int4 h = __ldg(&E.sep_h[t]);
            const double w = __ldg(&E.sep_w[t]);
            const double2 cs = trig.at(j, pos, h), A = src[t];
            ph += w * (cs.x * A.x + cs.y * A.y);
            const double f = w * (cs.y * A.x - cs.x * A.y);
            gx += f * h.x;
            gy += f * h.y;
            gz += f * h.z;
        }
    }
    phi -= ph * 0.31830988618379067;
    g[0] -= 2.0 * gx;
    g[1] -= 2.0 * gy;
    g[2] -= 2.0 * gz;
}
