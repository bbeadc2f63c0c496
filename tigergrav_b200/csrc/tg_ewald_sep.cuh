/*
 * tg_ewald_sep.cuh -- the particle-particle Ewald correction of the FP32 path
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
 * larger alpha therefore moves work to where it is shared.  At alpha = 4.2
 *   - real-space images beyond r = 1 add at most 1e-7 to the force factor
 *     (as images beyond r = 2 do at alpha = 2), and inside r < 1 of a separation
 *     |x_d| <= 1/2 lie at most the nearest image and its 7 mirror neighbours
 *     towards the near corner of the box, ~4 of them on average (~34 at
 *     alpha = 2): no lists of images, no search;
 *   - |h|^2 <= 30 leaves a force tail of 4e-8: 369 vectors (half space) for 61.
 * The nearest image stays combined with the removal of the direct 1/r
 * (ewald_nearest), and an interaction with r <= 1e-6 is phi0 alone, as the
 * reference has it (tigergrav/green.hpp:270-273): its reciprocal terms, which
 * the leaf sums include, are subtracted by that pair.
 *
 * Phases are exact: h.x mod 1 is an integer sum of the fixed-point coordinates
 * modulo 2^32 (plus 1/2 per odd h component for the 0.5 offset).
 */
#pragma once

constexpr float SEP_ALPHA = (float)SEP_ALPHA_D;

/* (cos, sin) of 2 pi h.x for fixed-point x */
__device__ __forceinline__ float2 sep_cs(int32_t x0, int32_t x1, int32_t x2, int4 h) {
    uint32_t u = (uint32_t)h.x * (uint32_t)x0 + (uint32_t)h.y * (uint32_t)x1 + (uint32_t)h.z * (uint32_t)x2;
    u += (uint32_t)(h.x + h.y + h.z) << 31; /* the offset 0.5 of every coordinate */
    float s, c;
    sincospif((float)(int32_t)u * 4.656612873077393e-10f, &s, &c); /* 2 x 2^-32 */
    return make_float2(c, s);
}

/* One block per source leaf of some PP_E list: the sums of (cos, sin) over its
 * particles, a thread per vector */
__global__ void __launch_bounds__(128) k_ewald_sf(const int32_t *__restrict__ src, const int32_t *__restrict__ pb,
                                                  const int32_t *__restrict__ pe, const int4 *__restrict__ pos,
                                                  EwaldTables E, float2 *__restrict__ sf) {
    const int32_t node = src[blockIdx.x];
    const int32_t b = pb[node], e = pe[node];
    for (int t = threadIdx.x; t < NSEP; t += 128) {
        const int4 h = __ldg(&E.sep_h[t]);
        float c = 0.0f, s = 0.0f;
        for (int32_t j = b; j < e; j++) {
            const int4 p = __ldg(&pos[j]);
            const float2 q = sep_cs(p.x, p.y, p.z, h);
            c += q.x;
            s += q.y;
        }
        sf[(int64_t)blockIdx.x * NSEP + t] = make_float2(c, s);
    }
}

/* one image at the displacement d (r2 = |d|^2 < 1): -erfc(alpha r)/r and its force */
__device__ __forceinline__ void sep_image(float d0, float d1, float d2, float r2, float &ph, float &gx, float &gy,
                                          float &gz) {
    const float rinv = rsqrt_ftz(r2);
    const float r = r2 * rinv;
    float expfac;
    const float erfc = t_erfcexp(SEP_ALPHA * r, &expfac);
    const float expfactor = (SEP_ALPHA * 1.1283791670955126f) * r * expfac; /* 2 alpha / sqrt(pi) */
    const float f = (expfactor + erfc) * rinv * rinv * rinv;
    ph -= erfc * rinv;
    gx = fmaf(-d0, f, gx);
    gy = fmaf(-d1, f, gy);
    gz = fmaf(-d2, f, gz);
}

/* The real-space part of one PP_E pair at the nearest-image separation x. */
__device__ __forceinline__ void pp_ewald_pair_sep(const EwaldTables &E, const float *x, float &phi, float *g) {
    const float a0 = fabsf(x[0]), a1 = fabsf(x[1]), a2 = fabsf(x[2]);
    const float u0 = a0 * a0, u1 = a1 * a1, u2 = a2 * a2;
    const float r2 = u0 + u1 + u2;
    if (!(r2 > 1.0e-12f)) { /* phi0 alone: take back the reciprocal terms, R0 + R2 r^2 / 2 */
        phi = EWALD_PHI0 - E.sep_r0;
        for (int d = 0; d < 3; d++) g[d] = E.sep_r2 * x[d];
        return;
    }
    const float b0 = 1.0f - a0, b1 = 1.0f - a1, b2 = 1.0f - a2;
    const float v0 = b0 * b0, v1 = b1 * b1, v2 = b2 * b2;
    float ph = 0.0f, gx = 0.0f, gy = 0.0f, gz = 0.0f; /* in the octant of |x| */
    float q;
    q = v0 + u1 + u2;
    if (q < 1.0f) sep_image(-b0, a1, a2, q, ph, gx, gy, gz);
    q = u0 + v1 + u2;
    if (q < 1.0f) sep_image(a0, -b1, a2, q, ph, gx, gy, gz);
    q = u0 + u1 + v2;
    if (q < 1.0f) sep_image(a0, a1, -b2, q, ph, gx, gy, gz);
    q = v0 + v1 + u2;
    if (q < 1.0f) sep_image(-b0, -b1, a2, q, ph, gx, gy, gz);
    q = v0 + u1 + v2;
    if (q < 1.0f) sep_image(-b0, a1, -b2, q, ph, gx, gy, gz);
    q = u0 + v1 + v2;
    if (q < 1.0f) sep_image(a0, -b1, -b2, q, ph, gx, gy, gz);
    q = v0 + v1 + v2;
    if (q < 1.0f) sep_image(-b0, -b1, -b2, q, ph, gx, gy, gz);
    const float rinv = rsqrt_ftz(r2);
    float p0, f0;
    ewald_nearest<float>(SEP_ALPHA, r2 * rinv, rinv, p0, f0);
    phi = ph + (E.sep_k + p0); /* pi / alpha^2 */
    g[0] = fmaf(x[0], f0, copysignf(1.0f, x[0]) * gx);
    g[1] = fmaf(x[1], f0, copysignf(1.0f, x[1]) * gy);
    g[2] = fmaf(x[2], f0, copysignf(1.0f, x[2]) * gz);
}

/* The reciprocal part at one sink particle from its leaf's sums T[h] =
 * (sum m cos th_j, sum m sin th_j), vectors t0, t0 + stride, ...: with
 * w_h = 2 exp(-pi^2 h^2 / alpha^2) / h^2 (both of +-h),
 *   phi -= sum w_h / pi cos(th_i - th_j),  g -= sum 2 w_h h sin(th_i - th_j). */
__device__ __forceinline__ void sep_eval(const EwaldTables &E, const double2 *T, int t0, int stride, int4 p, double &phi,
                                         double *g) {
    double ph = 0.0, gx = 0.0, gy = 0.0, gz = 0.0;
    for (int t = t0; t < NSEP; t += stride) {
        const int4 h = __ldg(&E.sep_h[t]);
        const double w = __ldg(&E.sep_w[t]);
        const float2 cs = sep_cs(p.x, p.y, p.z, h);
        const double C = cs.x, S = cs.y;
        const double2 A = T[t];
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
