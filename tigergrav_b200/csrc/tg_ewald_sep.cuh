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
 * larger alpha therefore moves work to where it is shared.  In FP32, alpha = 4.2:
 *   - real-space images beyond r = 1 add at most 1e-7 to the force factor
 *     (as images beyond r = 2 do at alpha = 2), and inside r < 1 of a separation
 *     |x_d| <= 1/2 lie at most the nearest image and its 7 mirror neighbours
 *     towards the near corner of the box, ~4 of them on average (~34 at
 *     alpha = 2): no lists of images, no search;
 *   - |h|^2 <= 30 leaves a force tail of 4e-8: 369 vectors (half space) for 61.
 * In FP64, alpha = 5.2: images beyond r = 1 add 1.1e-11 to the force factor, and
 * |h|^2 <= 70 leaves a force tail of 9e-12 (the 61 vectors at alpha = 2 leave
 * 6e-11), for ~4 images instead of ~200.
 * The nearest image stays combined with the removal of the direct 1/r
 * (ewald_nearest), and an interaction with r <= 1e-6 is phi0 alone, as the
 * reference has it (tigergrav/green.hpp:270-273): its reciprocal terms, which
 * the leaf sums include, are subtracted by that pair.
 *
 * Phases are exact: h.x mod 1 is an integer sum of the fixed-point coordinates
 * modulo 2^32 (plus 1/2 per odd h component for the 0.5 offset).
 */
#pragma once

/* (cos, sin) of 2 pi h.x for fixed-point x */
template <class T>
__device__ __forceinline__ typename Sep<T>::T2 sep_cs(int32_t x0, int32_t x1, int32_t x2, int4 h) {
    uint32_t u = (uint32_t)h.x * (uint32_t)x0 + (uint32_t)h.y * (uint32_t)x1 + (uint32_t)h.z * (uint32_t)x2;
    u += (uint32_t)(h.x + h.y + h.z) << 31; /* the offset 0.5 of every coordinate */
    const T r = T((int32_t)u) * T(4.656612873077392578125e-10); /* 2 x 2^-32 */
    typename Sep<T>::T2 cs;
    if constexpr (sizeof(T) == 4) sincospif(r, &cs.y, &cs.x);
    else sincospi(r, &cs.y, &cs.x);
    return cs;
}

/* source sums: zero, and a += m f */
template <class S> __device__ __forceinline__ S sep_zero();
template <> __device__ __forceinline__ float2 sep_zero<float2>() { return make_float2(0.0f, 0.0f); }
template <> __device__ __forceinline__ double2 sep_zero<double2>() { return make_double2(0.0, 0.0); }
template <class T, class S> __device__ __forceinline__ void sep_madd(S &a, T m, const S &f) {
    a.x = fma(m, f.x, a.x);
    a.y = fma(m, f.y, a.y);
}

/* One block per source leaf of some PP_E list: the sums of (cos, sin) over its
 * particles, a thread per vector of [t0, t1) */
template <class T>
__global__ void __launch_bounds__(128) k_ewald_sf(const int32_t *__restrict__ src, const int32_t *__restrict__ pb,
                                                  const int32_t *__restrict__ pe, const int4 *__restrict__ pos,
                                                  EwaldTables E, int t0, int t1,
                                                  typename Sep<T>::T2 *__restrict__ sf) {
    const int32_t node = src[blockIdx.x];
    const int32_t b = pb[node], e = pe[node];
    for (int t = t0 + threadIdx.x; t < t1; t += 128) {
        const int4 h = __ldg(&E.sep_h[t]);
        typename Sep<T>::T2 a;
        a.x = a.y = T(0);
        for (int32_t j = b; j < e; j++) {
            const int4 p = __ldg(&pos[j]);
            const typename Sep<T>::T2 q = sep_cs<T>(p.x, p.y, p.z, h);
            a.x += q.x;
            a.y += q.y;
        }
        sf[(int64_t)blockIdx.x * (t1 - t0) + t - t0] = a;
    }
}

/* one image at the displacement d (r2 = |d|^2 < 1): -erfc(alpha r)/r and its force */
template <class T>
__device__ __forceinline__ void sep_image(T d0, T d1, T d2, T r2, T &ph, T &gx, T &gy, T &gz) {
    const T rinv = t_rsqrt(r2);
    const T r = r2 * rinv;
    T expfac;
    const T erfc = t_erfcexp(T(Sep<T>::ALPHA) * r, &expfac);
    const T expfactor = T(Sep<T>::ALPHA * 1.1283791670955126) * r * expfac; /* 2 alpha / sqrt(pi) */
    const T f = (expfactor + erfc) * rinv * rinv * rinv;
    ph -= erfc * rinv;
    gx = fma(-d0, f, gx);
    gy = fma(-d1, f, gy);
    gz = fma(-d2, f, gz);
}

/* The real-space part of one PP_E pair at the nearest-image separation x. */
template <class T>
__device__ __forceinline__ void pp_ewald_pair_sep(const EwaldTables &E, const T *x, T &phi, T *g) {
    const T a0 = fabs(x[0]), a1 = fabs(x[1]), a2 = fabs(x[2]);
    const T u0 = a0 * a0, u1 = a1 * a1, u2 = a2 * a2;
    const T r2 = u0 + u1 + u2;
    if (!(r2 > T(1.0e-12))) { /* phi0 alone: take back the reciprocal terms, R0 + R2 r^2 / 2 */
        phi = T((double)EWALD_PHI0 - E.sep_r0);
        for (int d = 0; d < 3; d++) g[d] = T(E.sep_r2) * x[d];
        return;
    }
    const T b0 = T(1) - a0, b1 = T(1) - a1, b2 = T(1) - a2;
    const T v0 = b0 * b0, v1 = b1 * b1, v2 = b2 * b2;
    T ph = T(0), gx = T(0), gy = T(0), gz = T(0); /* in the octant of |x| */
    T q;
    q = v0 + u1 + u2;
    if (q < T(1)) sep_image<T>(-b0, a1, a2, q, ph, gx, gy, gz);
    q = u0 + v1 + u2;
    if (q < T(1)) sep_image<T>(a0, -b1, a2, q, ph, gx, gy, gz);
    q = u0 + u1 + v2;
    if (q < T(1)) sep_image<T>(a0, a1, -b2, q, ph, gx, gy, gz);
    q = v0 + v1 + u2;
    if (q < T(1)) sep_image<T>(-b0, -b1, a2, q, ph, gx, gy, gz);
    q = v0 + u1 + v2;
    if (q < T(1)) sep_image<T>(-b0, a1, -b2, q, ph, gx, gy, gz);
    q = u0 + v1 + v2;
    if (q < T(1)) sep_image<T>(a0, -b1, -b2, q, ph, gx, gy, gz);
    q = v0 + v1 + v2;
    if (q < T(1)) sep_image<T>(-b0, -b1, -b2, q, ph, gx, gy, gz);
    const T rinv = t_rsqrt(r2);
    T p0, f0;
    ewald_nearest<T>(T(Sep<T>::ALPHA), r2 * rinv, rinv, p0, f0);
    phi = ph + (T(E.sep_k) + p0); /* pi / alpha^2 */
    g[0] = fma(x[0], f0, copysign(T(1), x[0]) * gx);
    g[1] = fma(x[1], f0, copysign(T(1), x[1]) * gy);
    g[2] = fma(x[2], f0, copysign(T(1), x[2]) * gz);
}

/* The reciprocal part at one sink particle from its leaf's sums src[h] =
 * (sum m cos th_j, sum m sin th_j), vectors t0, t0 + stride, ...: with
 * w_h = 2 exp(-pi^2 h^2 / alpha^2) / h^2 (both of +-h),
 *   phi -= sum w_h / pi cos(th_i - th_j),  g -= sum 2 w_h h sin(th_i - th_j). */
template <class T>
__device__ __forceinline__ void sep_eval(const EwaldTables &E, const double2 *src, int t0, int stride, int4 p, double &phi,
                                         double *g) {
    double ph = 0.0, gx = 0.0, gy = 0.0, gz = 0.0;
    for (int t = t0; t < Sep<T>::N; t += stride) {
        const int4 h = __ldg(&E.sep_h[t]);
        const double w = __ldg(&E.sep_w[t]);
        const typename Sep<T>::T2 cs = sep_cs<T>(p.x, p.y, p.z, h);
        const double C = cs.x, S = cs.y;
        const double2 A = src[t];
        ph += w * (C * A.x + S * A.y);
        const double f = w * (S * A.x - C * A.y);
        gx += f * h.x;
        gy += f * h.y;
        gz += f * h.z;
    }
    phi -= ph * 0.31830988618379067;
    g[0] -= 2.0 * gx;
    g[1] -= 2.0 * gy;
    g[2] -= 2.0 * gz;
}
