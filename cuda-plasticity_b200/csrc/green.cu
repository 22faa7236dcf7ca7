// K-space pass of the stress pipeline (see stress.cu): the transforms along axis 0 with the contraction between.
#include "col_pass.cuh"

namespace cdd {

// ------------------------------------------------------------------------------------------
// Fused k-space pass along axis 0: forward FFT of the 9 components, Green contraction to the 6
// stress components (scaled by 1 / cells), inverse FFT of the 6. In place on the spectrum.
// ------------------------------------------------------------------------------------------
// Complex value times a real scalar (plus a complex value): one packed instruction in FP32.
template <typename V, typename T> __device__ __forceinline__ V csc(V a, T s) { a.x *= s; a.y *= s; return a; }
template <typename V, typename T> __device__ __forceinline__ V cfma(V a, T s, V c) {
    V r; r.x = a.x * s + c.x; r.y = a.y * s + c.y; return r;
}
template <> __device__ __forceinline__ float2 csc<float2, float>(float2 a, float s) {
    return __fmul2_rn(a, make_float2(s, s));
}
template <> __device__ __forceinline__ float2 cfma<float2, float>(float2 a, float s, float2 c) {
    return __ffma2_rn(a, make_float2(s, s), c);
}

template <typename T, typename V>
__device__ __forceinline__ void green_point(const V* b, V* out, T kx, T ky, T kz, bool kzero,
                                            T lam, T mu, T A, T B, T scale, bool drop_k0, V* phi_out) {
    const T k[3] = {kx, ky, kz};
    const T ksq = kx * kx + ky * ky + kz * kz;
    const T ikse = (T)1 / (ksq + (T)ME);
    const T ikqe = (T)1 / (ksq * ksq + (T)ME);
    V s1 = vadd(vadd(b[0], b[4]), b[8]);
    V p[3], q[3];
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        p[j] = cfma(b[6 + j], k[2], cfma(b[3 + j], k[1], csc(b[j], k[0])));
        q[j] = cfma(b[3 * j + 2], k[2], cfma(b[3 * j + 1], k[1], csc(b[3 * j], k[0])));
    }
    const V r = cfma(q[2], k[2], cfma(q[1], k[1], csc(q[0], k[0])));
    const V cc = vsub(csc(s1, A * ikse), csc(r, B * ikqe));
    const T mask = kzero ? (T)0 : (T)1;
    if (phi_out) {
        // phi = s1 / kSq - r / kSqSq: g_j depends on nu only through k_j (dA s1 / kSq - dB r / kSqSq)
        // with dA = dB, so d sigma / d nu at this k point is a multiple of phi (minus the lambda term)
        *phi_out = csc(vsub(csc(s1, ikse), csc(r, ikqe)), mask);
    }
    V g[3];
#pragma unroll
    for (int j = 0; j < 3; ++j) g[j] = csc(cfma(vadd(p[j], q[j]), ikse, csc(cc, k[j])), mask);
    const V tr = vsub(cfma(g[2], k[2], cfma(g[1], k[1], csc(g[0], k[0]))), s1);
    const int ia[6] = {0, 0, 0, 1, 1, 2};
    const int ja[6] = {0, 1, 2, 1, 2, 2};
#pragma unroll
    for (int o = 0; o < 6; ++o) {
        const int i = ia[o], j = ja[o];
        V v = csc(vsub(vsub(cfma(g[i], k[j], csc(g[j], k[i])), b[3 * i + j]), b[3 * j + i]), mu);
        if (i == j) v = cfma(tr, lam, v);
        v = csc(v, scale);
        if (drop_k0 && kzero) { v.x = 0; v.y = 0; }
        out[o] = v;
    }
}

// Transpose of green_point (a real linear map from 9 to 6 complex components per k point):
// cotangents of the 6 stress components in, cotangents of the 9 beta components out. Each line
// reverses one line of green_point.
template <typename T, typename V>
__device__ __forceinline__ void green_point_adj(const V* sb, V* bb, T kx, T ky, T kz, bool kzero,
                                                T lam, T mu, T A, T B, T scale) {
    const T k[3] = {kx, ky, kz};
    const T ksq = kx * kx + ky * ky + kz * kz;
    const T ikse = (T)1 / (ksq + (T)ME);
    const T ikqe = (T)1 / (ksq * ksq + (T)ME);
    const T mask = kzero ? (T)0 : (T)1;
    const int ia[6] = {0, 0, 0, 1, 1, 2};
    const int ja[6] = {0, 1, 2, 1, 2, 2};
    V gb[3], trb;
#pragma unroll
    for (int j = 0; j < 3; ++j) { gb[j].x = 0; gb[j].y = 0; }
    trb.x = 0; trb.y = 0;
#pragma unroll
    for (int c = 0; c < 9; ++c) { bb[c].x = 0; bb[c].y = 0; }
#pragma unroll
    for (int o = 0; o < 6; ++o) {
        const int i = ia[o], j = ja[o];
        V v = vscale(sb[o], scale);
        gb[j].x += mu * k[i] * v.x; gb[j].y += mu * k[i] * v.y;
        gb[i].x += mu * k[j] * v.x; gb[i].y += mu * k[j] * v.y;
        bb[3 * i + j].x -= mu * v.x; bb[3 * i + j].y -= mu * v.y;
        bb[3 * j + i].x -= mu * v.x; bb[3 * j + i].y -= mu * v.y;
        if (i == j) { trb.x += lam * v.x; trb.y += lam * v.y; }
    }
    V s1b;
    s1b.x = -trb.x; s1b.y = -trb.y;
#pragma unroll
    for (int i = 0; i < 3; ++i) { gb[i].x += k[i] * trb.x; gb[i].y += k[i] * trb.y; }
    V ccb, pb[3], qb[3];
    ccb.x = mask * (k[0] * gb[0].x + k[1] * gb[1].x + k[2] * gb[2].x);
    ccb.y = mask * (k[0] * gb[0].y + k[1] * gb[1].y + k[2] * gb[2].y);
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        pb[j].x = mask * ikse * gb[j].x; pb[j].y = mask * ikse * gb[j].y;
        qb[j] = pb[j];
    }
    s1b.x += A * ikse * ccb.x; s1b.y += A * ikse * ccb.y;
    V rb;
    rb.x = -B * ikqe * ccb.x; rb.y = -B * ikqe * ccb.y;
#pragma unroll
    for (int m = 0; m < 3; ++m) { qb[m].x += k[m] * rb.x; qb[m].y += k[m] * rb.y; }
#pragma unroll
    for (int j = 0; j < 3; ++j)
#pragma unroll
        for (int n = 0; n < 3; ++n) {
            bb[3 * j + n].x += qb[j].x * k[n]; bb[3 * j + n].y += qb[j].y * k[n];   // q_j = b_jn k_n
            bb[3 * n + j].x += k[n] * pb[j].x; bb[3 * n + j].y += k[n] * pb[j].y;   // p_j = k_m b_mj
        }
#pragma unroll
    for (int m = 0; m < 3; ++m) { bb[4 * m].x += s1b.x; bb[4 * m].y += s1b.y; }
}

// d sigma / d nu at fixed mu of green_point: A = nu/(1-nu), B = 1/(1-nu) and lam = 2 mu nu/(1-2nu)
// give dA = dB = 1/(1-nu)^2 and dlam = 2 mu/(1-2nu)^2.
template <typename T, typename V>
__device__ __forceinline__ void green_point_dnu(const V* b, V* out, T kx, T ky, T kz, bool kzero,
                                                T lam, T mu, T A, T B, T scale, T nu) {
    const T k[3] = {kx, ky, kz};
    const T ksq = kx * kx + ky * ky + kz * kz;
    const T ikse = (T)1 / (ksq + (T)ME);
    const T ikqe = (T)1 / (ksq * ksq + (T)ME);
    const T dA = (T)1 / ((1 - nu) * (1 - nu)), dB = dA;
    const T dlam = (T)2 * mu / ((1 - 2 * nu) * (1 - 2 * nu));
    V s1 = vadd(vadd(b[0], b[4]), b[8]);
    V p[3], q[3];
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        p[j].x = k[0] * b[j].x + k[1] * b[3 + j].x + k[2] * b[6 + j].x;
        p[j].y = k[0] * b[j].y + k[1] * b[3 + j].y + k[2] * b[6 + j].y;
        q[j].x = b[3 * j].x * k[0] + b[3 * j + 1].x * k[1] + b[3 * j + 2].x * k[2];
        q[j].y = b[3 * j].y * k[0] + b[3 * j + 1].y * k[1] + b[3 * j + 2].y * k[2];
    }
    V r;
    r.x = k[0] * q[0].x + k[1] * q[1].x + k[2] * q[2].x;
    r.y = k[0] * q[0].y + k[1] * q[1].y + k[2] * q[2].y;
    const T mask = kzero ? (T)0 : (T)1;
    V cc, dcc;
    cc.x = A * s1.x * ikse - B * r.x * ikqe;
    cc.y = A * s1.y * ikse - B * r.y * ikqe;
    dcc.x = dA * s1.x * ikse - dB * r.x * ikqe;
    dcc.y = dA * s1.y * ikse - dB * r.y * ikqe;
    V g[3], dg[3];
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        g[j].x = mask * (k[j] * cc.x + (p[j].x + q[j].x) * ikse);
        g[j].y = mask * (k[j] * cc.y + (p[j].y + q[j].y) * ikse);
        dg[j].x = mask * k[j] * dcc.x;
        dg[j].y = mask * k[j] * dcc.y;
    }
    V tr, dtr;
    tr.x = k[0] * g[0].x + k[1] * g[1].x + k[2] * g[2].x - s1.x;
    tr.y = k[0] * g[0].y + k[1] * g[1].y + k[2] * g[2].y - s1.y;
    dtr.x = k[0] * dg[0].x + k[1] * dg[1].x + k[2] * dg[2].x;
    dtr.y = k[0] * dg[0].y + k[1] * dg[1].y + k[2] * dg[2].y;
    const int ia[6] = {0, 0, 0, 1, 1, 2};
    const int ja[6] = {0, 1, 2, 1, 2, 2};
#pragma unroll
    for (int o = 0; o < 6; ++o) {
        const int i = ia[o], j = ja[o];
        V v;
        v.x = mu * (k[i] * dg[j].x + k[j] * dg[i].x);
        v.y = mu * (k[i] * dg[j].y + k[j] * dg[i].y);
        if (i == j) {
            v.x += dlam * tr.x + lam * dtr.x;
            v.y += dlam * tr.y + lam * dtr.y;
        }
        out[o] = vscale(v, scale);
    }
}

// ---- k-space observables (PlasticityState.py) ----
// One k point of an observable, scaled by 1 / cells for the inverse transform:
//  3: beta^E before the real-space -beta^P term (CalculateBetaElastic L357-390):
//     kmask sum_mn T_ijmn b_mn = kmask k_i g_j with g as in green_point and, b entering through
//     its symmetric part, p = q = sym(b) k;
//  4: its antisymmetric part (k_i g_j - k_j g_i) / 2 for (xy, xz, yz) (CalculateRotationField
//     L435-446);
//  5: the Rodrigues vector from beta^P (CalculateRotationRodrigues L447-475, source 'betaP'):
//     kmask sum_jst k_j (e_ijt k_s + e_ijs k_t) b_st / (2 kSq) = kmask (k x q)_i / kSq;
//  6: the Nye density rho_ai = -e_akl d_k b_li by Fourier derivatives (CalculateRhoFourier
//     L264-304): rho_xi = i (kz b_yi - ky b_zi), rho_yi = i (kx b_zi - kz b_xi),
//     rho_zi = i (ky b_xi - kx b_yi) (kz = 0 in 2-D), no mask;
//  8: the Rodrigues vector from the Nye density b = rho (CalculateRotationRodrigues L472-494, source
//     'rho'): kmask sum_mn D_imn b_mn, D_imn = i (2 k_n d_im - k_m d_in - k_i d_mn) / (2 kSq)
//     + i k_i k_n k_m / (2 kSqSq), i.e. i [(2 q_i - p_i - k_i s) / kSq + k_i r / kSqSq] / 2 with
//     q = b k, p = b^T k, s = tr b, r = k . b k.
// Inputs: 6 symmetric components xx xy xz yy yz zz (3-5) or all 9 (6, 8). The k values are those of
// the table the launch passes (the wrapped identity or, for 'sinK', the sine tables).
template <typename T, typename V, int GMODE>
__device__ __forceinline__ void obs_point(const V* b, V* o, T kx, T ky, T kz, bool kzero, T A, T B, T scale) {
    const T k[3] = {kx, ky, kz};
    if constexpr (GMODE == 8) {
        const T ksq = kx * kx + ky * ky + kz * kz;
        const T ikse = (T)1 / (ksq + (T)ME);
        const T ikqe = (T)1 / (ksq * ksq + (T)ME);
        const T f = (kzero ? (T)0 : (T)1) * (T)0.5 * scale;
        V q[3], p[3];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            q[i].x = b[3 * i].x * k[0] + b[3 * i + 1].x * k[1] + b[3 * i + 2].x * k[2];
            q[i].y = b[3 * i].y * k[0] + b[3 * i + 1].y * k[1] + b[3 * i + 2].y * k[2];
            p[i].x = k[0] * b[i].x + k[1] * b[3 + i].x + k[2] * b[6 + i].x;
            p[i].y = k[0] * b[i].y + k[1] * b[3 + i].y + k[2] * b[6 + i].y;
        }
        const V s1 = vadd(vadd(b[0], b[4]), b[8]);
        V r;
        r.x = k[0] * q[0].x + k[1] * q[1].x + k[2] * q[2].x;
        r.y = k[0] * q[0].y + k[1] * q[1].y + k[2] * q[2].y;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            V t;   // (2 q_i - p_i - k_i s) / kSq + k_i r / kSqSq, then times i f
            t.x = ((T)2 * q[i].x - p[i].x - k[i] * s1.x) * ikse + k[i] * r.x * ikqe;
            t.y = ((T)2 * q[i].y - p[i].y - k[i] * s1.y) * ikse + k[i] * r.y * ikqe;
            o[i].x = -t.y * f;
            o[i].y = t.x * f;
        }
        return;
    } else if constexpr (GMODE == 6) {
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const V bx = b[i], by = b[3 + i], bz = b[6 + i];
            V u[3];
            u[0].x = kz * by.x - ky * bz.x; u[0].y = kz * by.y - ky * bz.y;
            u[1].x = kx * bz.x - kz * bx.x; u[1].y = kx * bz.y - kz * bx.y;
            u[2].x = ky * bx.x - kx * by.x; u[2].y = ky * bx.y - kx * by.y;
#pragma unroll
            for (int a = 0; a < 3; ++a) {   // multiply by i
                o[3 * a + i].x = -u[a].y * scale;
                o[3 * a + i].y = u[a].x * scale;
            }
        }
        return;
    } else {
        const V b9[9] = {b[0], b[1], b[2], b[1], b[3], b[4], b[2], b[4], b[5]};
        const T ksq = kx * kx + ky * ky + kz * kz;
        const T ikse = (T)1 / (ksq + (T)ME);
        const T mask = kzero ? (T)0 : (T)1;
        V q[3];
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            q[j].x = b9[3 * j].x * k[0] + b9[3 * j + 1].x * k[1] + b9[3 * j + 2].x * k[2];
            q[j].y = b9[3 * j].y * k[0] + b9[3 * j + 1].y * k[1] + b9[3 * j + 2].y * k[2];
        }
        if constexpr (GMODE == 5) {
            const T f = mask * ikse * scale;
            o[0].x = f * (k[1] * q[2].x - k[2] * q[1].x); o[0].y = f * (k[1] * q[2].y - k[2] * q[1].y);
            o[1].x = f * (k[2] * q[0].x - k[0] * q[2].x); o[1].y = f * (k[2] * q[0].y - k[0] * q[2].y);
            o[2].x = f * (k[0] * q[1].x - k[1] * q[0].x); o[2].y = f * (k[0] * q[1].y - k[1] * q[0].y);
            return;
        } else {
            const T ikqe = (T)1 / (ksq * ksq + (T)ME);
            V s1 = vadd(vadd(b9[0], b9[4]), b9[8]);
            V r;
            r.x = k[0] * q[0].x + k[1] * q[1].x + k[2] * q[2].x;
            r.y = k[0] * q[0].y + k[1] * q[1].y + k[2] * q[2].y;
            V cc;
            cc.x = A * s1.x * ikse - B * r.x * ikqe;
            cc.y = A * s1.y * ikse - B * r.y * ikqe;
            V g[3];
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                g[j].x = mask * scale * (k[j] * cc.x + (q[j].x + q[j].x) * ikse);
                g[j].y = mask * scale * (k[j] * cc.y + (q[j].y + q[j].y) * ikse);
            }
            if constexpr (GMODE == 3) {
#pragma unroll
                for (int i = 0; i < 3; ++i)
#pragma unroll
                    for (int j = 0; j < 3; ++j) { o[3 * i + j].x = k[i] * g[j].x; o[3 * i + j].y = k[i] * g[j].y; }
            } else {
                const int ia[3] = {0, 0, 1}, ja[3] = {1, 2, 2};
                const T hf = (T)0.5;
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    const int i = ia[c], j = ja[c];
                    o[c].x = hf * (k[i] * g[j].x - k[j] * g[i].x);
                    o[c].y = hf * (k[i] * g[j].y - k[j] * g[i].y);
                }
            }
        }
    }
}

// The contraction of one k-space pass at every k point of the block's tile: component slots cs apart, k point
// (e, w) at (e << lgw) + w, in place. GMODE: the stress (0), its adjoint (1), its nu derivative (2), the
// observables (3-6, 8), the vacancy diffusion (7).
// phi (optional, one complex value per k point, laid out like one spectrum component with the
// instance base spoff / 9): GMODE 0 writes phi of the input; GMODE 1 reads the phi of the state
// whose stress the cotangent belongs to and adds to pacc its share of the Parseval sum
// sum_k w_k Re(conj(sigbar_hat) . (2 mu k k + lam kSq I) phi) / cells (w_k = 1 on the first and
// the Nyquist half-axis column, 2 elsewhere): the A/B part of <sigbar, (d sigma / d nu) beta>
// per unit dA.
template <typename T, bool MEAN64, int GMODE>
__device__ __forceinline__ void contract_tile(const InstDev& I, typename VecOf<T>::type* s, int cs, int lgw, int col0,
                                              int wv, int i1, long long estride, const T* __restrict__ ktab,
                                              typename VecOf<T>::type* __restrict__ phib, T vdt, double& pacc,
                                              int tid, int nt) {
    typedef typename VecOf<T>::type V;
    constexpr int NIN = green_nin(GMODE), NOUT = green_nout(GMODE);
    const int N = I.n0, W = 1 << lgw;
    // vacancy diffusion factor exp(-gamma dt kSq) (VacancyDynamics.DiffusionEvolution L41-61), dt of
    // the step just taken
    const T vg = (GMODE == 7) ? (T)(-I.vac_gamma) : (T)0;
    const T lam = (T)I.lamb, mu = (T)I.mu;
    const T A = (T)(I.lamb / (I.lamb + 2.0 * I.mu));
    const T B = (T)(2.0 * (I.lamb + I.mu) / (I.lamb + 2.0 * I.mu));
    const T scale = (T)I.inv_cells;
#pragma unroll 1
    for (int i = tid; i < N * W; i += nt) {
        const int e = i >> lgw, w = i & (W - 1);
        const int kh = col0 + w;
        if (w >= wv) continue;
        T kx, ky, kz;
        bool kzero;
        if (I.nd == 3) {
            kx = ktab[I.koff0 + e];
            ky = ktab[I.koff1 + i1];
            kz = ktab[I.koffh + kh];
            kzero = (e == 0 && i1 == 0 && kh == 0);
        } else {
            kx = ktab[I.koff0 + e];
            ky = ktab[I.koffh + kh];
            kz = (T)0;
            kzero = (e == 0 && kh == 0);
        }
        V b[NIN], o[NOUT];
#pragma unroll
        for (int c = 0; c < NIN; ++c) b[c] = s[c * cs + i];
        if constexpr (GMODE == 7) {
            const T ksq = kx * kx + ky * ky + kz * kz;
            const T f = exp(ksq * vg * vdt) * scale;
            o[0].x = b[0].x * f;
            o[0].y = b[0].y * f;
        } else if constexpr (GMODE >= 3) {
            obs_point<T, V, GMODE>(b, o, kx, ky, kz, kzero, A, B, scale);
        } else if constexpr (GMODE == 0) {
            // the symmetric 3 x 3 matrix of the six components (row-major, b9[3i + j])
            const V b9[9] = {b[0], b[1], b[2], b[1], b[3], b[4], b[2], b[4], b[5]};
            V ph;
            green_point<T, V>(b9, o, kx, ky, kz, kzero, lam, mu, A, B, scale, MEAN64, phib ? &ph : nullptr);
            if (phib) phib[e * estride + w] = ph;
        } else if constexpr (GMODE == 1) {
            if (phib) {
                const V ph = phib[e * estride + w];
                const double k3[3] = {(double)kx, (double)ky, (double)kz};
                const double ksq = k3[0] * k3[0] + k3[1] * k3[1] + k3[2] * k3[2];
                const int ia[6] = {0, 0, 0, 1, 1, 2}, ja[6] = {0, 1, 2, 1, 2, 2};
                double acc = 0.0;
#pragma unroll
                for (int c = 0; c < 6; ++c) {
                    double cf = 2.0 * (double)I.mu * k3[ia[c]] * k3[ja[c]];
                    if (ia[c] == ja[c]) cf += I.lamb * ksq;
                    acc += cf * ((double)b[c].x * (double)ph.x + (double)b[c].y * (double)ph.y);
                }
                const bool edge = (kh == 0) || (2 * kh == I.nl);
                pacc += (edge ? 1.0 : 2.0) * acc;
            }
            V bb[9];
            green_point_adj<T, V>(b, bb, kx, ky, kz, kzero, lam, mu, A, B, scale);
            // cotangent of beta_ij (= of beta_ji) through s_ij = (beta_ij + beta_ji) / 2
            const T hf = (T)0.5;
            o[0] = bb[0];
            o[1].x = hf * (bb[1].x + bb[3].x); o[1].y = hf * (bb[1].y + bb[3].y);
            o[2].x = hf * (bb[2].x + bb[6].x); o[2].y = hf * (bb[2].y + bb[6].y);
            o[3] = bb[4];
            o[4].x = hf * (bb[5].x + bb[7].x); o[4].y = hf * (bb[5].y + bb[7].y);
            o[5] = bb[8];
        } else {
            const V b9[9] = {b[0], b[1], b[2], b[1], b[3], b[4], b[2], b[4], b[5]};
            green_point_dnu<T, V>(b9, o, kx, ky, kz, kzero, lam, mu, A, B, scale, (T)I.nu);
        }
#pragma unroll
        for (int c = 0; c < NOUT; ++c) s[c * cs + i] = o[c];
    }
}

// Lines without a two-pass form (4, 8, 16, 512 and some others, plans tuned to radix 4): through the stage
// engine, three components at a time (one by one for the single-component mode) against three scratch slots
// after the component slots; when the stage count is odd the result is copied back.
template <typename V, bool INV, int K>
__device__ __forceinline__ void fft_slots(V* s, int n, V* scratch, int lgw, int cs, const LinePlan& lp,
                                          const V* __restrict__ tws, int tid, int nt) {
#pragma unroll 1
    for (int c = 0; c < n; c += K) {
        V* a = s + c * cs;
        ColLayout<K> lay{lgw, cs};
        V* r = fft_lines<V, INV>(a, scratch, lay, lp, tws, tid, nt, lp.twst[0]);
        if (r != a) {
            for (int i = tid; i < K * cs; i += nt) a[i] = r[i];
            __syncthreads();
        }
    }
}

// FP32 stress solves: FP64 mean of each of the six components from the row sums, for the C2R pass's mean stress.
// The launch's first 6 n_inst blocks, one per instance and component, form them beside the k-space work (a
// kernel of its own took 5 to 18 us per solve). Fixed order: deterministic.
struct MeanArgs {
    int blocks;              // 6 n_inst, or 0
    const double* rowsum;
    double* mean9;           // 9 per instance
};
__device__ __noinline__ void mean_block(const InstDev& I, int ii, int c, const MeanArgs& a, double* red) {
    const int tid = threadIdx.x, nt = blockDim.x;
    pdl_wait();
    const double* rs = a.rowsum + I.rsoff + (long long)c * I.rows;
    // eight independent accumulators per thread keep several loads in flight
    double acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    int r = tid;
    for (; r + 7 * nt < I.rows; r += 8 * nt)
#pragma unroll
        for (int q = 0; q < 8; ++q) acc[q] += rs[r + q * nt];
    for (; r < I.rows; r += nt) acc[0] += rs[r];
    double v = ((acc[0] + acc[1]) + (acc[2] + acc[3])) + ((acc[4] + acc[5]) + (acc[6] + acc[7]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((tid & 31) == 0) red[tid >> 5] = v;
    __syncthreads();
    if (tid == 0) {
        double sum = 0.0;
        for (int w = 0; w < (nt >> 5); ++w) sum += red[w];
        a.mean9[9 * ii + c] = sum * I.inv_cells;
    }
}

// Fused k-space pass along axis 0: forward FFT of the input components, contraction (scaled by 1 / cells),
// inverse FFT of the outputs, in place on the spectrum. A block owns W = 2^lgw spectrum columns (32 bytes) of row
// i1 (3-D) of one instance and all their components.
// In two passes per direction every phase runs in place in one set of component slots:
//   pass A global -> slots, pass B in place (its outputs m + A r are the positions it read), contraction,
//   inverse pass A in place (j + B q, natural order in; output m stays at j + B m), inverse pass B from
//   the B consecutive values at m B -> global.
// No static shared memory: the slots and twiddle rows of some lengths fill an SM's share to within 300 bytes (three
// blocks of 256 points at radix 8, two of 288 points with 12 slots; a 320-byte array made the latter's passes take 468
// us instead of 332).
// Four block barriers, no scratch slots and one butterfly per thread and pass at 256 (12 lines FP64, 24 FP32,
// on 192 threads). Bound by the latency of its phases and, at FP64, the FP64 pipe.
// TIER 0: every instance's passes are one stage each; 1: of at most 16 values; 2: all two-pass forms; 3: as 1, for plans
// with long lines of the stage engine (green_engine): FP64 on 256 threads instead of 192 (their slots leave an SM one or
// two blocks), and 512-point lines leave by their last stage (288 points, 288x64x256 FP64: 484 -> 438 us; 512 points,
// 512x128x128: FP64 964 -> 786, FP32 441 -> 390).
template <typename T, int TIER>
__global__ void __launch_bounds__(sizeof(T) == 4 || TIER == 3 ? 256 : 192, (TIER >= 2 && sizeof(T) == 8) ? 2 : 3)
k_green(const InstDev* __restrict__ insts, int n_inst, const int* __restrict__ pre, int gmode, int mean64, MeanArgs mean,
        typename VecOf<T>::type* spec, const typename VecOf<T>::type* __restrict__ tw,
        const T* __restrict__ ktab, typename VecOf<T>::type* phi, double* part,
        const InstClock* clk) {
    typedef typename VecOf<T>::type V;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    V* s = reinterpret_cast<V*>(smem_raw);
    if ((int)blockIdx.x < mean.blocks) {
        mean_block(insts[blockIdx.x / 6], blockIdx.x / 6, blockIdx.x % 6, mean, reinterpret_cast<double*>(smem_raw));
        return;
    }
    const int blk = blockIdx.x - mean.blocks;
    const int ii = find_instance(pre, n_inst, blk);
    const InstDev& I = insts[ii];
    if (gmode == 7 && !I.vacancy) {
        pdl_wait();
        return;
    }
    const int lb = blk - pre[ii];
    const PassTile& tl = I.tile[PASS_GREEN];
    const int lgw = tl.lgw, ta_n = tl.tiles_a;
    const int i1 = lb / ta_n;          // 0 in 2-D
    const int ta = lb - i1 * ta_n;
    const int W = 1 << lgw;
    const int N = I.n0, nhp = I.nhp, nh = I.nh;
    const int col0 = ta * W;
    const int wv = min(W, nh - col0);
    const int tid = threadIdx.x, nt = blockDim.x;
    const int cs = N * W + W;          // component slot in shared memory
    const long long estride = (I.nd == 3) ? (long long)I.n1 * nhp : (long long)nhp;
    const long long cstride = (long long)N * estride;
    V* base = spec + I.spoff + (I.nd == 3 ? (long long)i1 * nhp : 0) + col0;
    const int nin = green_nin(gmode), nout = green_nout(gmode), slots = nin > nout ? nin : nout;
    const LinePlan& lp = I.lp_first;
    const bool two = TIER == 0 || lp.pa != 0;
    constexpr int PT = TIER == 3 ? 1 : TIER;   // the two-pass forms compiled in
    V* scratch = s + slots * cs;
    V* tws = s + (((two ? slots : slots + 3) * cs + 1) & ~1);   // twiddle rows after the slots
    stage_tw_to_smem(lp, tw, tws, tid, nt);
    pdl_wait();
    const Cols<V> glob{base, cstride, wv}, slot{s, cs, W};
    if (two) {
        __syncthreads();
        col_pass_a<V, false, PT>(glob, estride, lp.B * estride, slot, (long long)lp.A << lgw, W, nin << lgw, lgw, lp, tws,
                                   tid, nt);
        col_pass_b<V, false, PT>(slot, W, (long long)lp.A << lgw, slot, W, (long long)lp.A << lgw, nin << lgw, lgw, lp, tws,
                                   tid, nt);
    } else if constexpr (TIER != 0) {
        if (W * (int)sizeof(V) >= 16) {
#pragma unroll 1
            for (int c = 0; c < nin; ++c) tile_async_load(s + c * cs, base + c * cstride, estride, N, lgw, wv, tid, nt);
        } else {
            // 8-byte columns (W = 1, FP32)
#pragma unroll 1
            for (int c = 0; c < nin; ++c) {
#pragma unroll 8
                for (int i = tid; i < N; i += nt) s[c * cs + i] = base[c * cstride + i * estride];
            }
        }
        cp_async_wait_all();
        __syncthreads();
        if (nin == 1) fft_slots<V, false, 1>(s, nin, scratch, lgw, cs, lp, tws, tid, nt);
        else fft_slots<V, false, 3>(s, nin, scratch, lgw, cs, lp, tws, tid, nt);
    }
    double pacc = 0.0;
    {
        V* phib = phi ? phi + I.spoff / 9 + (I.nd == 3 ? (long long)i1 * nhp : 0) + col0 : nullptr;
        const T vdt = (gmode == 7) ? (T)clk[ii].dt : (T)0;
#define CDD_CONTRACT(M64, G) contract_tile<T, M64, G>(I, s, cs, lgw, col0, wv, i1, estride, ktab, phib, vdt, pacc, tid, nt)
        if (gmode == 0) {
            if (mean64) CDD_CONTRACT(true, 0);
            else CDD_CONTRACT(false, 0);
        } else if (gmode == 1) {
            CDD_CONTRACT(false, 1);
        } else if constexpr (TIER != 0) {
            switch (gmode) {
                case 2: CDD_CONTRACT(false, 2); break;
                case 3: CDD_CONTRACT(false, 3); break;
                case 4: CDD_CONTRACT(false, 4); break;
                case 5: CDD_CONTRACT(false, 5); break;
                case 6: CDD_CONTRACT(false, 6); break;
                case 7: CDD_CONTRACT(false, 7); break;
                default: CDD_CONTRACT(false, 8); break;
            }
        }
#undef CDD_CONTRACT
    }
    if (gmode == 1 && part) {
        // fixed-order block reduction (deterministic), in the bytes that this mode's launch adds (launch_green)
        double* red = reinterpret_cast<double*>(tws + ((lp.twspan + 1) & ~1));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) pacc += __shfl_xor_sync(0xffffffffu, pacc, o);
        if ((tid & 31) == 0) red[tid >> 5] = pacc;
        __syncthreads();
        if (tid == 0) {
            double sum = 0.0;
            for (int w = 0; w < nt / 32; ++w) sum += red[w];
            part[blk] = sum * I.inv_cells;
        }
    }
    __syncthreads();
    if (two) {
        col_pass_a<V, true, PT>(slot, W, (long long)lp.B << lgw, slot, W, (long long)lp.B << lgw, nout << lgw, lgw, lp, tws,
                                  tid, nt);
        col_pass_b<V, true, PT>(slot, (long long)lp.B << lgw, W, glob, estride, lp.A * estride, nout << lgw, lgw, lp, tws,
                                  tid, nt);
    } else if constexpr (TIER != 0) {
        if constexpr (TIER == 3) {
            if (nout > 1 && line_512(lp)) {
                // 512 points: the last stage writes global memory (an odd stage count would end in the scratch slots)
                const SColT<V, 3> x{scratch, lgw, cs};
#pragma unroll 1
                for (int c = 0; c < nout; c += 3) {
                    const SColT<V, 3> slots3{s + c * cs, lgw, cs};
                    const GColT<V, 3> out{base + c * cstride, estride, cstride, lgw, wv};
                    fft_io_c<V, true, 3, SColT<V, 3>, GColT<V, 3>, 1, 16, 8, 4>(slots3, x, slots3, out, lgw, lp, tws, tid, nt,
                                                                               lp.twst[0], 0);
                }
                return;
            }
        }
        if (nout == 1) fft_slots<V, true, 1>(s, nout, scratch, lgw, cs, lp, tws, tid, nt);
        else fft_slots<V, true, 3>(s, nout, scratch, lgw, cs, lp, tws, tid, nt);
        if (W * (int)sizeof(V) >= 16) {
#pragma unroll 1
            for (int c = 0; c < nout; ++c) tile_store(base + c * cstride, s + c * cs, estride, N, lgw, wv, tid, nt);
        } else {
#pragma unroll 1
            for (int c = 0; c < nout; ++c) {
#pragma unroll 4
                for (int i = tid; i < N; i += nt) base[c * cstride + i * estride] = s[c * cs + i];
            }
        }
    }
}

template <typename T>
static void green_t(const PlanCore& P, const LaunchShape& L, int gmode, bool mean64, const void* ktab, void* phi, double* part,
                    cudaStream_t st) {
    typedef typename VecOf<T>::type V;
    const int tier = green_tier3(P) ? 3 : (P.green_lean && gmode <= 1) ? 0 : (P.big_green ? 2 : 1);
    const size_t smem = L.smem + (gmode == 1 ? 96 : 0);   // the block sums of the adjoint mode
    const MeanArgs mean{mean64 ? 6 * P.n_inst : 0, P.d_rowsum, P.d_sbar};
#define CDD_LAUNCH_G(TIER)                                                                                               \
    launch_pdl(k_green<T, TIER>, L.blocks + mean.blocks, L.threads, smem, st, P.d_inst, P.n_inst, L.d_pre, gmode, mean64, \
               mean, (V*)P.d_spec, (const V*)P.d_tw, (const T*)ktab, (V*)phi, part, P.d_clock)
    if (tier == 0) CDD_LAUNCH_G(0);
    else if (tier == 1) CDD_LAUNCH_G(1);
    else if (tier == 2) CDD_LAUNCH_G(2);
    else CDD_LAUNCH_G(3);
#undef CDD_LAUNCH_G
}

void launch_green(const PlanCore& P, const LaunchShape& L, int gmode, bool mean64, const void* ktab, void* phi, double* part,
                  cudaStream_t st) {
    if (P.precision == CDD_F32) green_t<float>(P, L, gmode, mean64, ktab, phi, part, st);
    else green_t<double>(P, L, gmode, mean64, ktab, phi, part, st);
}

// Columns per tile: 32-byte row segments; 64-byte ones (half the line lookups in L1 per byte; stress solve at
// 128^3 FP64 379 -> 357 us, 100 x 200 x 250 FP32 721 -> 701 us) where the six slots stay under 50 KB, so that as
// many blocks fit an SM, and the grid still has four blocks per SM (64^3 FP32 prefers 32 bytes, 64 us against 66).
int green_cols(const InstDev& I, int sms, size_t velt) {
    int W = (int)(32 / velt);
    while (W > 1 && (size_t)9 * (I.n0 * W + W) * velt > 100 * 1024) W >>= 1;
    const int wide = (int)(64 / velt), rows = (I.nd == 3) ? I.n1 : 1;
    if ((size_t)6 * (I.n0 + 1) * 64 <= 50 * 1024 && rows * ((I.nh + wide - 1) / wide) >= 4 * sms) W = wide;
    return W;
}
// Threads: FP32 tiles of long lines (three blocks per SM) run on 256 (256^3 stress solve 1196 us against 1259 on
// 192), others on 192 (64^3 64 us against 79). TIER 3 runs on 256.
int green_threads(const InstDev& I, size_t velt) { return velt == 8 && I.n0 >= 192 ? 256 : 192; }

size_t green_smem_bytes(const InstDev& I, int W, int slots, size_t velt) {
    const size_t n = (size_t)(I.lp_first.pa ? slots : slots + 3) * ((size_t)I.n0 * W + W);
    return ((n + 1) & ~(size_t)1) * velt + (size_t)I.lp_first.twspan * velt;
}
bool green_plan_lean(const LinePlan& lp) { return pass_lean(lp); }

template <typename T>
static cudaError_t green_attr(size_t smem) {
    cudaError_t e;
    if ((e = set_dyn_smem_limit(k_green<T, 0>, smem))) return e;
    if ((e = set_dyn_smem_limit(k_green<T, 1>, smem))) return e;
    if ((e = set_dyn_smem_limit(k_green<T, 3>, smem))) return e;
    return set_dyn_smem_limit(k_green<T, 2>, smem);
}
cudaError_t green_set_attributes(int precision, size_t smem) {
    return precision == CDD_F32 ? green_attr<float>(smem) : green_attr<double>(smem);
}

}  // namespace cdd
