/*
 * tg_ewald_table.cuh -- green_ewald (tigergrav/green.hpp:189-286) of the FP32
 * path from local expansions.  Included by tg_gravity.cu.
 *
 * psi(X) = green_ewald's D0, the periodic Green's function with the direct
 * 1/r of the nearest image taken out, is analytic on the minimum-image cube
 * [-1/2, 1/2]^3 (its nearest singularity is another image, at least 1/2 away)
 * and obeys Laplace psi = -4 pi there (the neutralising background).  So one
 * table of Taylor expansions to order ET_P about the centres of ET_N^3 cells
 * of the octant [0, 1/2]^3 gives every derivative tensor that the contractions
 * need: an evaluation shifts its cell's expansion by X - centre.  Mirror
 * symmetry gives the other octants (a component changes sign with each axis
 * that it has an odd power of).
 *
 * By Laplace's equation the coefficients t_ijk = D_ijk / (i! j! k!) with k >= 2
 * follow from those with k = 0 and 1, so a cell's row holds (ET_P + 1)^2 = 64
 * floats: 256 bytes, aligned.
 *
 * Cost: 16 16-byte loads and ~510 FP32 instructions per evaluation, against
 * ~39 image evaluations (185 operations and three transcendentals each) and 61
 * reciprocal terms (80 operations each) of the sums themselves.
 *
 * Error against FP64 of D0 (less ET_OFFSET) to D4, rms over 65536 points of the cube:
 * 1.6e-7, 6.7e-8, 3.6e-7, 1.1e-6, 2.3e-5 (values 2.4, 1.0, 3.9, 12, 63); the FP32 sums
 * 3.5e-7, 3.0e-7, 1.0e-6, 5.3e-6, 6.3e-5.  Near the cube's faces D4 has 4.5e-5 / 8.1e-5,
 * at the cells' corners, where an order-7 expansion leaves most, 1.1e-4 / 6.5e-5; every
 * other order is below the sums there too.
 *
 * The table is generated in FP64 from those sums (the reference's images and 61
 * reciprocal vectors), with the exact erfc.  One part of the FP32 sums is kept
 * on purpose: they lie ET_OFFSET below the FP64 value on average over the cube
 * (the reference's FP32 erfc, Abramowitz & Stegun 7.1.26,
 * tigergrav/simd.hpp:676-692, is off by -5.4e-7, and rounding gives part of it
 * back), so every potential, and E_pot, would move against the kernels that
 * evaluate the sums; each cell's constant carries that mean.
 */
#pragma once

constexpr int ET_N = 48;  /* cells per axis of the octant [0, 1/2]^3: 28 MB, kept in L2 */
constexpr int ET_P = 7;   /* expansion order */
constexpr int ET_ROW = (ET_P + 1) * (ET_P + 1);
constexpr int ET_A = (ET_P + 1) * (ET_P + 2) / 2; /* coefficients with k = 0; those with k = 1 follow */
constexpr double ET_OFFSET = -3.4e-7; /* mean of (FP32 sums - FP64) of D0 over the cube, one number for all X (-5.2e-7 for |X_d| < 1/4) */
constexpr double ET_LAPLACE = -12.566370614359172; /* -4 pi */
static_assert(ET_ROW == 64 && ET_A == 36, "row layout");

/* slot of x^i y^j in a plane of constant k, by order i + j */
__host__ __device__ constexpr int et_ij(int i, int j) { return (i + j) * (i + j + 1) / 2 + j; }

/* ---- generation: one block of 64 threads per cell with ix >= iy, a thread per
 * coefficient (psi is symmetric in x and y: the mirrored cell holds the same
 * coefficients with i and j exchanged).  2.2 ms of FP64 in all. ---- */

/* slot of (j, n >= j) among the pairs of 0..ET_P */
__device__ __forceinline__ int et_jn(int j, int n) { return j * (ET_P + 1) - j * (j - 1) / 2 + n - j; }

constexpr int ET_IMG = 96;        /* images within ET_CUT2 of a point of the octant: at most 94 */
constexpr double ET_CUT2 = 7.29;  /* r < 2.7: the images beyond add 1e-12 to D0 and 1e-7 of D4's rms */

/* the centre of cell q along one axis, the same FP32 value in generation and evaluation */
__device__ __forceinline__ float et_centre(int q) { return __fmul_rn((float)q + 0.5f, 0.5f / ET_N); }

__global__ void __launch_bounds__(64) k_ewald_table(const float4 *__restrict__ real, const float4 *__restrict__ four,
                                                    float *__restrict__ table) {
    __shared__ double sxp[ET_IMG][ET_P + 1], sw[ET_IMG][ET_A], sz[ET_IMG];
    __shared__ double hp[7][ET_P + 1], hc[NFOUR_HALF], hs[NFOUR_HALF];
    __shared__ int s_img[ET_IMG], s_w[2];
    const int tid = threadIdx.x, lane = tid & 31, wp = tid >> 5;
    const int iz = blockIdx.x, iy = blockIdx.y, ix = blockIdx.z;
    if (ix < iy) return; /* block-uniform */
    const double X[3] = {(double)et_centre(ix), (double)et_centre(iy), (double)et_centre(iz)};
    const double alpha = 2.0, pi = 3.141592653589793, cexp = 2.0 * alpha / 1.7724538509055159; /* 2 alpha / sqrt(pi) */
    const double ch[4] = {1.0, 0.5, 0.125, 1.0 / 48.0}; /* 1 / (p! 2^p) */
    const double rfact[ET_P + 1] = {1.0, 1.0, 1.0 / 2, 1.0 / 6, 1.0 / 24, 1.0 / 120, 1.0 / 720, 1.0 / 5040};
    /* the images inside the cut, in table order */
    int nimg = 0;
    for (int b = 0; b < NREAL; b += 64) {
        bool in = false;
        if (b + tid < NREAL) {
            const float4 n = real[b + tid];
            const double dx = X[0] - n.x, dy = X[1] - n.y, dz = X[2] - n.z;
            in = dx * dx + dy * dy + dz * dz < ET_CUT2;
        }
        const uint32_t m = __ballot_sync(0xffffffffu, in);
        if (lane == 0) s_w[wp] = __popc(m);
        __syncthreads();
        const int k = nimg + (wp ? s_w[0] : 0) + __popc(m & ((1u << lane) - 1u));
        if (in && k < ET_IMG) s_img[k] = b + tid;
        nimg += s_w[0] + s_w[1];
        __syncthreads();
    }
    nimg = min(nimg, ET_IMG);
    /* radial derivatives d_n = ((1/r) d/dr)^n of -erfc(2r)/r, or of erf(2r)/r at n = 0, and powers over factorials */
    for (int q = tid; q < nimg; q += 64) {
        const float4 n = real[s_img[q]];
        const double dx = X[0] - n.x, dy = X[1] - n.y, dz = X[2] - n.z;
        const double r2 = dx * dx + dy * dy + dz * dz;
        const double r = sqrt(r2), e2 = exp(-alpha * alpha * r2);
        sz[q] = dz;
        double px = 1.0, py = 1.0, yp[ET_P + 1], rd[ET_P + 1];
#pragma unroll
        for (int e = 0; e <= ET_P; e++) {
            sxp[q][e] = px * rfact[e];
            yp[e] = py * rfact[e];
            px *= dx;
            py *= dy;
        }
        if (n.w == 0.0f) {
            /* erf(alpha r)/r = cexp F_0(T), d_n = cexp (-2 alpha^2)^n F_n(T), T = alpha^2 r^2, with
             * F_n(T) = int_0^1 t^2n e^(-T t^2) dt: F_P from its series, the others by downward recursion */
            const double T = alpha * alpha * r2;
            double term = 1.0 / (2 * ET_P + 1), F = term;
            for (int m = 1; m < 40; m++) {
                term *= 2.0 * T / (2 * ET_P + 2 * m + 1);
                F += term;
            }
            F *= e2;
            double w = cexp;
#pragma unroll
            for (int m = 0; m < ET_P; m++) w *= -2.0 * alpha * alpha;
#pragma unroll
            for (int m = ET_P; m >= 0; m--) {
                rd[m] = w * F;
                w /= -2.0 * alpha * alpha;
                if (m > 0) F = (2.0 * T * F + e2) / (2 * m - 1);
            }
        } else {
            /* g_0 = erfc(alpha r)/r, r^2 g_(n+1) = -(2n+1) g_n - (-2 alpha^2)^n cexp e^(-alpha^2 r^2) */
            double g = erfc(alpha * r) / r, w = cexp * e2;
            const double r2inv = 1.0 / r2;
#pragma unroll
            for (int m = 0; m <= ET_P; m++) {
                rd[m] = -g;
                g = -((2 * m + 1) * g + w) * r2inv;
                w *= -2.0 * alpha * alpha;
            }
        }
        /* the y part: sum_s y^(j-2s)/(j-2s)! d_(n-s) / (s! 2^s) */
#pragma unroll
        for (int j = 0; j <= ET_P; j++)
#pragma unroll
            for (int n = j; n <= ET_P; n++) {
                double u = 0.0;
#pragma unroll
                for (int s = 0; 2 * s <= j; s++) u += ch[s] * yp[j - 2 * s] * rd[n - s];
                sw[q][et_jn(j, n)] = u;
            }
    }
    /* reciprocal vectors (one of each pair +-h): -(2/pi) c_h (cos, sin)(2 pi h.X), and (2 pi h)^e / e! */
    if (tid < NFOUR_HALF) {
        const float4 h = four[tid];
        const double h2 = (double)h.x * h.x + (double)h.y * h.y + (double)h.z * h.z;
        double sn, cs;
        sincospi(2.0 * (h.x * X[0] + h.y * X[1] + h.z * X[2]), &sn, &cs);
        const double w = -(2.0 / pi) * exp(-pi * pi * h2 / 4.0) / h2;
        hc[tid] = w * cs;
        hs[tid] = w * sn;
    }
    if (tid < 7) {
        double p = 1.0;
        for (int e = 0; e <= ET_P; e++) {
            hp[tid][e] = p * rfact[e];
            p *= 2.0 * pi * (tid - 3);
        }
    }
    __syncthreads();
    /* this thread's coefficient t_ijk = D_ijk / (i! j! k!): k = 0 for tid < ET_A, else k = 1 */
    const int kz = tid < ET_A ? 0 : 1;
    int i = 0, j = kz ? tid - ET_A : tid;
    for (int s = 0; j > s; s++) {
        j -= s + 1;
        i = s + 1;
    }
    i -= j; /* i held the order */
    double t = 0.0;
    for (int q = 0; q < nimg; q++) {
        /* D_ij0 / (i! j!) = sum_{p,s} x^(i-2p)/(i-2p)! y^(j-2s)/(j-2s)! d_(i+j-p-s) / (p! 2^p s! 2^s);
         * one more radial derivative times z for k = 1 */
        double v = 0.0;
        for (int p = 0; 2 * p <= i; p++) v += ch[p] * sxp[q][i - 2 * p] * sw[q][et_jn(j, i + j - p + kz)];
        t += kz ? v * sz[q] : v;
    }
    const int n = i + j + kz; /* cos differentiated n times: cos, -sin, -cos, sin */
    double rec = 0.0;
    for (int q = 0; q < NFOUR_HALF; q++) {
        const float4 h = four[q];
        double w = hp[(int)h.x + 3][i] * hp[(int)h.y + 3][j];
        if (kz) w *= hp[(int)h.z + 3][1];
        rec += w * ((n & 1) ? hs[q] : hc[q]);
    }
    t += ((n & 3) == 1 || (n & 3) == 2) ? -rec : rec;
    if (tid == 0) t += 0.78539816339744831 + ET_OFFSET; /* pi/4 (tigergrav/green.hpp:270) */
    table[(((int64_t)ix * ET_N + iy) * ET_N + iz) * ET_ROW + tid] = (float)t;
    table[(((int64_t)iy * ET_N + ix) * ET_N + iz) * ET_ROW + (kz ? ET_A : 0) + et_ij(j, i)] = (float)t;
}

/* ---- evaluation ---- */

/* T_k+2 from T_k by Laplace's equation: order N plane to order N - 2 */
template <int N, int K>
__device__ __forceinline__ void et_lift(const float *lo, float *hi) {
    constexpr float w = -1.0f / (float)((K + 2) * (K + 1));
#pragma unroll
    for (int s = 0; s <= N - 2; s++)
#pragma unroll
        for (int j = 0; j <= s; j++) {
            const int i = s - j;
            hi[et_ij(i, j)] = fmaf(w * (float)((i + 2) * (i + 1)), lo[et_ij(i + 2, j)],
                                   w * (float)((j + 2) * (j + 1)) * lo[et_ij(i, j + 2)]);
        }
}
/* A += wA T, B += wB T over a plane of order N */
template <int N>
__device__ __forceinline__ void et_add(float *A, float wA, float *B, float wB, const float *T) {
#pragma unroll
    for (int q = 0; q < (N + 1) * (N + 2) / 2; q++) {
        A[q] = fmaf(wA, T[q], A[q]);
        B[q] = fmaf(wB, T[q], B[q]);
    }
}
/* shift a plane of order N by (x, y): the coefficients of order <= M about the new centre */
template <int N, int M>
__device__ __forceinline__ void et_shift_xy(float *A, float x, float y) {
#pragma unroll
    for (int j = 0; j <= N; j++) /* along x: synthetic division, for powers of x up to M */
#pragma unroll
        for (int p = 0; p <= cmin(M, N - j); p++)
#pragma unroll
            for (int i = N - j - 1; i >= p; i--) A[et_ij(i, j)] = fmaf(x, A[et_ij(i + 1, j)], A[et_ij(i, j)]);
#pragma unroll
    for (int i = 0; i <= M; i++) /* along y */
#pragma unroll
        for (int p = 0; p <= M - i; p++)
#pragma unroll
            for (int j = N - i - 1; j >= p; j--) A[et_ij(i, j)] = fmaf(y, A[et_ij(i, j + 1)], A[et_ij(i, j)]);
}

/* flip the sign of v by the sign bit sg */
__device__ __forceinline__ float et_sgn(float v, uint32_t sg) { return __uint_as_float(__float_as_uint(v) ^ sg); }

/* one axis: cell index, offset from its centre (of |X|), and X's sign bit */
__device__ __forceinline__ int et_axis(float X, float &o, uint32_t &sg) {
    const float a = fabsf(X);
    sg = __float_as_uint(X) & 0x80000000u;
    const int q = min((int)(a * (2.0f * ET_N)), ET_N - 1);
    o = a - et_centre(q);
    return q;
}

/* the cell of X, X's offset from its centre in the octant of |X|, and X's signs */
__device__ __forceinline__ int et_locate(const float *X, float *o, uint32_t *sg) {
    int cell = 0;
#pragma unroll
    for (int d = 0; d < 3; d++) cell = cell * ET_N + et_axis(X[d], o[d], sg[d]);
    return cell;
}

/* green_ewald(X) for |X_d| <= 1/2 (tigergrav/green.hpp:189-286) from the row of
 * X's cell; r <= 1e-6 gives phi0 alone as there */
__device__ __forceinline__ void et_eval(const float4 *row, const float *X, const float *o, const uint32_t *sg, float *D) {
    float R[ET_ROW];
#pragma unroll
    for (int q = 0; q < ET_ROW / 4; q++) {
        const float4 v = row[q];
        R[4 * q] = v.x, R[4 * q + 1] = v.y, R[4 * q + 2] = v.z, R[4 * q + 3] = v.w;
    }
    float *A = R, *B = R + ET_A;
    const float z = o[2], z2 = z * z, z3 = z2 * z, z4 = z2 * z2, z5 = z4 * z, z6 = z4 * z2, z7 = z4 * z3;
    {
        /* shift along z: planes k >= 2 by Laplace's equation, added to the planes k = 0 and 1 */
        float T2[21], T3[15], T4[10], T5[6], T6[3], T7[1];
        et_lift<7, 0>(A, T2);
        T2[0] += (float)(0.5 * ET_LAPLACE); /* the background: t_002 = (-4 pi - 2 t_200 - 2 t_020) / 2 */
        et_lift<6, 1>(B, T3);
#pragma unroll
        for (int q = 0; q < 28; q++) A[q] = fmaf(z, B[q], A[q]);
        et_add<5>(A, z2, B, 2.0f * z, T2);
        et_add<4>(A, z3, B, 3.0f * z2, T3);
        et_lift<5, 2>(T2, T4);
        et_add<3>(A, z4, B, 4.0f * z3, T4);
        et_lift<4, 3>(T3, T5);
        et_add<2>(A, z5, B, 5.0f * z4, T5);
        et_lift<3, 4>(T4, T6);
        et_add<1>(A, z6, B, 6.0f * z5, T6);
        et_lift<2, 5>(T5, T7);
        et_add<0>(A, z7, B, 7.0f * z6, T7);
    }
    et_shift_xy<7, 4>(A, o[0], o[1]);
    et_shift_xy<6, 3>(B, o[0], o[1]);
    const uint32_t sx = sg[0], sy = sg[1], sz = sg[2];
    const float r2 = X[0] * X[0] + X[1] * X[1] + X[2] * X[2];
    D[E0()] = A[0];
    D[E1(0)] = et_sgn(A[et_ij(1, 0)], sx);
    D[E1(1)] = et_sgn(A[et_ij(0, 1)], sy);
    D[E1(2)] = et_sgn(B[0], sz);
    const float xx = 2.0f * A[et_ij(2, 0)], yy = 2.0f * A[et_ij(0, 2)];
    D[E2(0, 0)] = xx;
    D[E2(1, 1)] = yy;
    D[E2(2, 2)] = (float)ET_LAPLACE - xx - yy;
    D[E2(0, 1)] = et_sgn(A[et_ij(1, 1)], sx ^ sy);
    D[E2(0, 2)] = et_sgn(B[et_ij(1, 0)], sx ^ sz);
    D[E2(1, 2)] = et_sgn(B[et_ij(0, 1)], sy ^ sz);
    const float xxx = 6.0f * A[et_ij(3, 0)], xxy = 2.0f * A[et_ij(2, 1)], xyy = 2.0f * A[et_ij(1, 2)],
                yyy = 6.0f * A[et_ij(0, 3)];
    const float xxz = 2.0f * B[et_ij(2, 0)], xyz = B[et_ij(1, 1)], yyz = 2.0f * B[et_ij(0, 2)];
    D[E3(0, 0, 0)] = et_sgn(xxx, sx);
    D[E3(0, 0, 1)] = et_sgn(xxy, sy);
    D[E3(0, 1, 1)] = et_sgn(xyy, sx);
    D[E3(1, 1, 1)] = et_sgn(yyy, sy);
    D[E3(0, 0, 2)] = et_sgn(xxz, sz);
    D[E3(0, 1, 2)] = et_sgn(xyz, sx ^ sy ^ sz);
    D[E3(1, 1, 2)] = et_sgn(yyz, sz);
    D[E3(0, 2, 2)] = et_sgn(-xxx - xyy, sx);
    D[E3(1, 2, 2)] = et_sgn(-xxy - yyy, sy);
    D[E3(2, 2, 2)] = et_sgn(-xxz - yyz, sz);
    const float x4 = 24.0f * A[et_ij(4, 0)], x3y = 6.0f * A[et_ij(3, 1)], x2y2 = 4.0f * A[et_ij(2, 2)],
                xy3 = 6.0f * A[et_ij(1, 3)], y4 = 24.0f * A[et_ij(0, 4)];
    const float x3z = 6.0f * B[et_ij(3, 0)], x2yz = 2.0f * B[et_ij(2, 1)], xy2z = 2.0f * B[et_ij(1, 2)],
                y3z = 6.0f * B[et_ij(0, 3)];
    D[E4(0, 0, 0, 0)] = x4;
    D[E4(0, 0, 0, 1)] = et_sgn(x3y, sx ^ sy);
    D[E4(0, 0, 1, 1)] = x2y2;
    D[E4(0, 1, 1, 1)] = et_sgn(xy3, sx ^ sy);
    D[E4(1, 1, 1, 1)] = y4;
    D[E4(0, 0, 0, 2)] = et_sgn(x3z, sx ^ sz);
    D[E4(0, 0, 1, 2)] = et_sgn(x2yz, sy ^ sz);
    D[E4(0, 1, 1, 2)] = et_sgn(xy2z, sx ^ sz);
    D[E4(1, 1, 1, 2)] = et_sgn(y3z, sy ^ sz);
    const float xxzz = -x4 - x2y2, yyzz = -x2y2 - y4;
    D[E4(0, 0, 2, 2)] = xxzz;
    D[E4(0, 1, 2, 2)] = et_sgn(-x3y - xy3, sx ^ sy);
    D[E4(1, 1, 2, 2)] = yyzz;
    D[E4(0, 2, 2, 2)] = et_sgn(-x3z - xy2z, sx ^ sz);
    D[E4(1, 2, 2, 2)] = et_sgn(-x2yz - y3z, sy ^ sz);
    D[E4(2, 2, 2, 2)] = -xxzz - yyzz;
    if (!(r2 > 1.0e-12f)) {
        D[E0()] = EWALD_PHI0;
#pragma unroll
        for (int q = 1; q < LP; q++) D[q] = 0.0f;
    }
}

__device__ __forceinline__ void green_ewald_table(const float *__restrict__ table, const float *X, float *D) {
    float o[3];
    uint32_t sg[3];
    const int cell = et_locate(X, o, sg);
    et_eval(reinterpret_cast<const float4 *>(table + (int64_t)cell * ET_ROW), X, o, sg, D);
}

/* The rows of a warp's cells into shared memory, row k at buf + k ET_STRIDE, for
 * the first n lanes; all lanes call it.  Half a warp copies a row, 256
 * consecutive bytes, where a lane reading its own row touches another cache line
 * than every other lane with each load; those wavefronts bounded the node Ewald
 * kernel (node phase at 128^3 theta 0.2: 63.7 -> 47.7 ms, 256^3 theta 0.19: 148 ->
 * 125 ms; the 80-byte multipoles staged the same way as well: 144 ms).  The stride
 * keeps the lanes' 16-byte reads free of bank conflicts. */
constexpr int ET_STRIDE = ET_ROW + 4;
__device__ __forceinline__ void et_stage(const float *__restrict__ table, int cell, int n, float *buf) {
    const int lane = threadIdx.x & 31, h = lane >> 4, q = lane & 15;
    __syncwarp(); /* the rows of the last call are read */
#pragma unroll 8
    for (int k = 0; k < n; k += 2) {
        const int c = __shfl_sync(0xffffffffu, cell, (k + h) & 31);
        if (k + h < n) {
            const uint32_t dst = (uint32_t)__cvta_generic_to_shared(buf + (k + h) * ET_STRIDE + 4 * q);
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(table + (int64_t)c * ET_ROW + 4 * q)
                         : "memory");
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncwarp();
}

/* green_ewald of the solver's kernels: FP32 from the table, FP64 from the sums */
template <class T> __device__ __forceinline__ void green_ewald_any(const EwaldTables &E, const T *X, T *D);
template <> __device__ __forceinline__ void green_ewald_any<float>(const EwaldTables &E, const float *X, float *D) {
    green_ewald_table(E.tab, X, D);
}
template <> __device__ __forceinline__ void green_ewald_any<double>(const EwaldTables &E, const double *X, double *D) {
    green_ewald_full<double>(E, X, D);
}

/* ---- the table of a device: made by the first solver that needs it, shared, freed with the last ---- */
struct EwTabDev {
    float *p = nullptr;
    int refs = 0;
};
static std::mutex g_ewtab_mtx;
static EwTabDev g_ewtab[64];

size_t ewald_table_bytes() { return sizeof(float) * (size_t)ET_N * ET_N * ET_N * ET_ROW; }

int ewald_table_acquire(int dev, const float4 *real, const float4 *four, const float **tab, cudaStream_t st) {
    if (dev < 0 || dev >= 64) return TG_ERR_ARG;
    std::lock_guard<std::mutex> lk(g_ewtab_mtx);
    EwTabDev &t = g_ewtab[dev];
    if (!t.p) {
        float *p = nullptr;
        if (cudaMalloc(&p, ewald_table_bytes()) != cudaSuccess) {
            cudaGetLastError();
            return TG_ERR_NOMEM;
        }
        k_ewald_table<<<dim3(ET_N, ET_N, ET_N), 64, 0, st>>>(real, four, p);
        /* complete before any other stream or thread may read it */
        cudaError_t e = cudaGetLastError();
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        if (e != cudaSuccess) {
            cudaFree(p);
            set_last_cuda_error(e, "k_ewald_table", __FILE__, __LINE__);
            return TG_ERR_CUDA;
        }
        t.p = p;
        g_dev_bytes += (long long)ewald_table_bytes();
    }
    t.refs++;
    *tab = t.p;
    return TG_OK;
}

/* the caller has waited for its device: no kernel reads the table any more */
void ewald_table_release(int dev) {
    std::lock_guard<std::mutex> lk(g_ewtab_mtx);
    EwTabDev &t = g_ewtab[dev];
    if (--t.refs > 0) return;
    cudaFree(t.p);
    t.p = nullptr;
    g_dev_bytes -= (long long)ewald_table_bytes();
}
