// Vector-Jacobian product of the central-upwind flux L(beta) = flux(beta, sigma(beta) + load)
// (the forward is stencil.cu): given the cotangent gbar of rhs, produce the cotangent of beta.
//
// Phase A (one thread per cell) recomputes the cell's forward quantities -- the 54 limited
// one-sided derivatives U with the limiter selection of each, the per-axis velocity vectors A,
// |rho|^2 terms P and C, the corner velocities, the directional speeds with the corners that
// attain them, the corner weights and the contractions Q -- and then runs every step backwards,
// producing the cotangents Ubar of the 54 derivatives and sigbar of the total stress at the cell
// (6 symmetric components; its diagonal sums are the applied-load cotangent).
// Phase B gathers beta's cotangent from Ubar: the limiter minmod(a, c) returns a, c or 0, so each
// one-sided derivative is a fixed linear combination of u_{-2} .. u_{+2} once the selection is
// known (2 bits per derivative, recorded in phase A).
// The stress cotangent is mapped back through the transposed Green's function by the host
// (launch_stress_adjoint) and added in phase B.
#include "cdd_internal.cuh"

namespace cdd {

namespace {

// Offsets of the neighbours at distance 1 and 2 along one axis (a component has fewer than 2^31 cells).
struct Nbr {
    int p1, p2, m1, m2;
};

__device__ __forceinline__ Nbr make_nbr(int i, int n, int stride) {
    int ip1 = (i + 1 == n) ? 0 : i + 1;
    int ip2 = (ip1 + 1 == n) ? 0 : ip1 + 1;
    int im1 = (i == 0) ? n - 1 : i - 1;
    int im2 = (im1 == 0) ? n - 1 : im1 - 1;
    Nbr r;
    r.p1 = (ip1 - i) * stride;
    r.p2 = (ip2 - i) * stride;
    r.m1 = (im1 - i) * stride;
    r.m2 = (im2 - i) * stride;
    return r;
}

// Grid coordinates of cell cl of a 3-D (n0, n1, n2) or 2-D (n0, n1) grid; cells < 2^31, so the
// divisions are 32-bit.
__device__ __forceinline__ void cell_coords(long long cl, int nd, int n1, int n2, int& i0, int& i1, int& i2) {
    const unsigned c = (unsigned)cl;
    const unsigned nx = (unsigned)(nd == 3 ? n2 : n1);
    const unsigned r = c / nx;
    i2 = (int)(c - r * nx);
    if (nd == 3) {
        i0 = (int)(r / (unsigned)n1);
        i1 = (int)(r - (unsigned)i0 * (unsigned)n1);
    } else {
        i0 = (int)r;
        i1 = i2;
    }
}

__device__ __forceinline__ float inv_sqrt_a(float x) { return rsqrtf(x); }
__device__ __forceinline__ double inv_sqrt_a(double x) { return 1.0 / sqrt(x); }

// minmod of two values and which one it returned (1: a, 2: c, 0: neither)
template <typename T>
__device__ __forceinline__ T mm_sel(T a, T c, int& sel) {
    const bool same = (a > (T)0 && c > (T)0) || (a < (T)0 && c < (T)0);
    const bool pa = fabs(a) <= fabs(c);
    sel = same ? (pa ? 1 : 2) : 0;
    return same ? (pa ? a : c) : (T)0;
}

// The limiter arguments in the reference's difference order. The FP32 forward stencil forms e0 and
// em2 in a packed form that can differ from these in the last bit, so in an exact tie between two
// limiter arguments the FP32 reverse may take the other branch (the FP32 gradient is checked
// against the FP64 one, whose forward and reverse use the same differences).
template <typename T>
__device__ __forceinline__ void derivs_sel(const T* __restrict__ p, const Nbr& nb, T ih, T& up, T& um,
                                           int& sp, int& sm) {
    const T u0 = p[0], um2 = p[nb.m2], um1 = p[nb.m1], up1 = p[nb.p1], up2 = p[nb.p2];
    const T dm2 = um1 - um2, dm1 = u0 - um1, d0 = up1 - u0, d1 = up2 - up1;
    const T e0 = d1 - d0, em1 = d0 - dm1, em2 = dm1 - dm2;
    const T dd0 = mm_sel(e0, em1, sp);
    const T ddm = mm_sel(em1, em2, sm);
    up = (d0 - (T)0.5 * dd0) * ih;
    um = (dm1 + (T)0.5 * ddm) * ih;
}

template <typename T>
__device__ __forceinline__ double bsum(double v, double* red) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) red[warp] = v;
    __syncthreads();
    double r = red[0];
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w) r += red[w];
    return r;
}

constexpr int VJP_THREADS = 128;
template <typename T> constexpr size_t vjp_smem() { return (size_t)54 * VJP_THREADS * sizeof(T); }   // derivatives
constexpr int VJP_PARTS = 5;     // per-block partials: <sigbar, sigma>, tr tr, diag sigbar (3)

// Keeps the compiler from carrying values of the shared slots across (it would hold all 54 in registers again).
__device__ __forceinline__ void vjp_phase() { asm volatile("" ::: "memory"); }

template <typename T, int ND>
__device__ __forceinline__ void vjp_cell(const InstDev& I, long long cl, bool valid, const T* __restrict__ beta,
                                         const T* __restrict__ sig, const T* __restrict__ gbar, double tload,
                                         T* __restrict__ ubar, uint32_t* __restrict__ flags,
                                         T* __restrict__ sigbar, double* lsum, T* us) {
    const long long cells = I.cells;
    Nbr nb[ND];
    {
        int i0, i1, i2;
        cell_coords(cl, ND, I.n1, I.n2, i0, i1, i2);
        if (ND == 3) {
            nb[0] = make_nbr(i0, I.n0, I.n1 * I.n2);
            nb[1] = make_nbr(i1, I.n1, I.n2);
            nb[ND - 1] = make_nbr(i2, I.n2, 1);
        } else {
            nb[0] = make_nbr(i0, I.n0, I.n1);
            nb[ND - 1] = make_nbr(i1, I.n1, 1);
        }
    }
    const T ih = (T)I.inv_h;
    const T* u = beta + I.foff + cl;

    // ---------------- forward recomputation ----------------
    // the 54 derivatives live in this thread's shared-memory slots (U): in registers, beside their cotangents,
    // they left 8 warps per SM (FP32) or spilled 2 KB per thread (FP64)
    auto U = [us](int d, int s, int c) -> T { return us[((2 * d + s) * 9 + c) * VJP_THREADS]; };
    uint32_t fw[4] = {0u, 0u, 0u, 0u};
#pragma unroll
    for (int c = 0; c < 9; ++c)
#pragma unroll
        for (int d = 0; d < ND; ++d) {
            int sp, sm;
            T up, um;
            derivs_sel(u + (long long)c * cells, nb[d], ih, up, um, sp, sm);
            us[(2 * d * 9 + c) * VJP_THREADS] = up;
            us[((2 * d + 1) * 9 + c) * VJP_THREADS] = um;
            const int slot = c * 3 + d;
            fw[slot >> 3] |= (uint32_t)(sp | (sm << 2)) << (4 * (slot & 7));
        }
    vjp_phase();
    double add[3] = {0.0, 0.0, 0.0};
    if (I.has_load) {
        double eps[3];
        for (int i = 0; i < 3; ++i) eps[i] = I.load_init[i] + I.load_rate[i] * (tload - I.load_t0);
        double tr = eps[0] + eps[1] + eps[2];
        for (int i = 0; i < 3; ++i) add[i] = I.load_lamb * tr + 2.0 * I.load_mu * eps[i];
    }
    const T* sp6 = sig + I.soff + cl;
    T S[3][3];
    T s6[6];
    {
#pragma unroll
        for (int c = 0; c < 6; ++c) s6[c] = sp6[c * cells];
        S[0][0] = (T)((double)s6[0] + add[0]);
        S[1][1] = (T)((double)s6[3] + add[1]);
        S[2][2] = (T)((double)s6[5] + add[2]);
        S[0][1] = S[1][0] = s6[1];
        S[0][2] = S[2][0] = s6[2];
        S[1][2] = S[2][1] = s6[4];
    }
    const bool lam_on = (I.Lambda != 0.0);
    const T Lam = (T)I.Lambda;
    const T str = lam_on ? (S[0][0] + S[1][1] + S[2][2]) / (T)3 * Lam : (T)0;
    T A[ND][2][3], trU[ND][2], P[ND][2];
    constexpr int NP = (ND == 3) ? 3 : 1;
    const int pd[3] = {0, 1, 2}, pe[3] = {1, 2, 0};   // pair p couples axes (pd[p], pe[p])
    T Cp[NP][2][2];
#pragma unroll
    for (int d = 0; d < ND; ++d)
#pragma unroll
        for (int s = 0; s < 2; ++s) {
            T sd = 0, pq = 0, tu = 0;
#pragma unroll
            for (int l = 0; l < 3; ++l) {
                T a = 0;
#pragma unroll
                for (int n = 0; n < 3; ++n) {
                    const T v = U(d, s, 3 * l + n);
                    a += v * S[d][n];
                    sd += v * S[l][n];
                    if (l != d) pq += v * v;
                }
                A[d][s][l] = a;
                tu += U(d, s, 4 * l);
            }
            A[d][s][d] -= sd;
            trU[d][s] = tu;
            P[d][s] = pq;
            if (lam_on) {
                A[d][s][d] += str * tu;
#pragma unroll
                for (int l = 0; l < 3; ++l) A[d][s][l] -= str * U(d, s, 3 * l + d);
            }
        }
#pragma unroll
    for (int p = 0; p < NP; ++p)
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
            for (int b = 0; b < 2; ++b) {
                T acc = 0;
#pragma unroll
                for (int j = 0; j < 3; ++j) acc += U(pd[p], a, 3 * pe[p] + j) * U(pe[p] % ND, b, 3 * pd[p] + j);
                Cp[p][a][b] = acc;
            }
    constexpr int NC = 1 << ND;
    T V[NC][3], rr[NC];
    int sg[NC][3];
#pragma unroll
    for (int c = 0; c < NC; ++c) {
        sg[c][0] = (c >> (ND - 1)) & 1;
        sg[c][1] = (c >> (ND - 2)) & 1;
        sg[c][2] = (ND == 3) ? (c & 1) : 0;
        T rho2 = (T)ME;
#pragma unroll
        for (int d = 0; d < ND; ++d) rho2 += P[d][sg[c][d]];
#pragma unroll
        for (int p = 0; p < NP; ++p) rho2 -= (T)2 * Cp[p][sg[c][pd[p]]][sg[c][pe[p] % ND]];
        rr[c] = inv_sqrt_a(rho2);
#pragma unroll
        for (int l = 0; l < 3; ++l) {
            T a = 0;
#pragma unroll
            for (int d = 0; d < ND; ++d) a += A[d][sg[c][d]][l];
            V[c][l] = a * rr[c];
        }
    }
    T pp[ND], pm[ND], tot[ND];
    int cmx[ND], cmn[ND];
#pragma unroll
    for (int d = 0; d < ND; ++d) {
        T mx = 0, mn = 0;
        cmx[d] = -1;
        cmn[d] = -1;
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            if (V[c][d] > mx) { mx = V[c][d]; cmx[d] = c; }
            if (V[c][d] < mn) { mn = V[c][d]; cmn[d] = c; }
        }
        pp[d] = mx;
        pm[d] = -mn;
        tot[d] = pp[d] + pm[d] + (T)ME;
    }
    T w[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) {
        T ww = 1;
#pragma unroll
        for (int d = 0; d < ND; ++d) ww *= (sg[c][d] == 0) ? pm[d] : pp[d];
        w[c] = ww;
    }
    T Q[ND][2][3];
#pragma unroll
    for (int d = 0; d < ND; ++d)
#pragma unroll
        for (int s = 0; s < 2; ++s)
#pragma unroll
            for (int l = 0; l < 3; ++l) Q[d][s][l] = 0;
#pragma unroll
    for (int c = 0; c < NC; ++c)
#pragma unroll
        for (int l = 0; l < 3; ++l)
#pragma unroll
            for (int d = 0; d < ND; ++d) Q[d][sg[c][d]][l] += w[c] * V[c][l];
    T prod = 1;
#pragma unroll
    for (int d = 0; d < ND; ++d) prod *= tot[d];
    // FP32: a cell without gradients has prod = ME^3, below the FP32 range; there hs = 0, and the
    // smallest normal value keeps every term finite (the forward normalises its weights instead)
    if (sizeof(T) == 4 && !(prod >= (T)1.17549435e-38f)) prod = (T)1.17549435e-38f;
    const T inv_abc = (T)1 / prod;
    T coef[ND];
#pragma unroll
    for (int d = 0; d < ND; ++d) coef[d] = pm[d] * pp[d] / tot[d];
    vjp_phase();
    // ---------------- reverse ----------------
    // rhs_ij = -hs_ij inv_abc + sum_d (U+ - U-)_ij coef_d  [- J inv_abc on the diagonal]. First the cotangents
    // of Q, coef and inv_abc, then those of the corners, A, P and C; the 54 derivatives' cotangents are formed last,
    // each from these in one go, and stored at once.
    T gb[9];
    const T* gp = gbar + I.foff + cl;
#pragma unroll
    for (int c = 0; c < 9; ++c) gb[c] = (valid && gbar) ? gp[c * cells] : (T)0;
    T Qb[ND][2][3], coefb[ND];
#pragma unroll
    for (int d = 0; d < ND; ++d) {
        coefb[d] = 0;
#pragma unroll
        for (int s = 0; s < 2; ++s)
#pragma unroll
            for (int l = 0; l < 3; ++l) Qb[d][s][l] = 0;
    }
    T inv_abc_b = 0;
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            const int c = 3 * i + j;
            const T vb = gb[c];
            const T hb = -vb * inv_abc;
            T h = 0;   // hs_ij
#pragma unroll
            for (int d = 0; d < ND; ++d) {
                const T u0 = U(d, 0, c), u1 = U(d, 1, c);
                h += Q[d][0][d] * u0 + Q[d][1][d] * u1;
                coefb[d] += vb * (u0 - u1);
                Qb[d][0][d] += hb * u0;
                Qb[d][1][d] += hb * u1;
            }
            if (i < ND) {
#pragma unroll
                for (int s = 0; s < 2; ++s)
#pragma unroll
                    for (int l = 0; l < 3; ++l) {
                        const T v = U(i % ND, s, 3 * l + j);
                        h -= Q[i % ND][s][l] * v;
                        Qb[i % ND][s][l] -= hb * v;
                    }
            }
            inv_abc_b -= vb * h;
        }
    const T gdiag = gb[0] + gb[4] + gb[8];
    const T Jpb = lam_on ? (-inv_abc * gdiag) * (-Lam / (T)3) : (T)0;
    if (lam_on) {
        T Jp = 0;   // J = -Lambda / 3 Jp
#pragma unroll
        for (int d = 0; d < ND; ++d)
#pragma unroll
            for (int s = 0; s < 2; ++s) {
                const T tu = U(d, s, 0) + U(d, s, 4) + U(d, s, 8);
                Jp += Q[d][s][d] * tu;
                Qb[d][s][d] += Jpb * tu;
#pragma unroll
                for (int l = 0; l < 3; ++l) {
                    const T v = U(d, s, 3 * l + d);
                    Jp -= Q[d][s][l] * v;
                    Qb[d][s][l] -= Jpb * v;
                }
            }
        inv_abc_b -= -Lam / (T)3 * Jp * gdiag;
    }
    vjp_phase();
    T ppb[ND], pmb[ND], totb[ND];
#pragma unroll
    for (int d = 0; d < ND; ++d) {
        pmb[d] = coefb[d] * pp[d] / tot[d];
        ppb[d] = coefb[d] * pm[d] / tot[d];
        totb[d] = -coefb[d] * coef[d] / tot[d] - inv_abc_b * inv_abc / tot[d];
    }
    auto weight = [&](int c, int skip) {   // product of a corner's weights but axis `skip`
        T ww = 1;
#pragma unroll
        for (int d = 0; d < ND; ++d)
            if (d != skip) ww *= (sg[c][d] == 0) ? pm[d] : pp[d];
        return ww;
    };
    auto qsum = [&](int c, int l) {   // cotangent of w_c V_cl
        T q = 0;
#pragma unroll
        for (int d = 0; d < ND; ++d) q += Qb[d][sg[c][d]][l];
        return q;
    };
#pragma unroll
    for (int c = 0; c < NC; ++c) {
        T wb = 0;
#pragma unroll
        for (int l = 0; l < 3; ++l) wb += qsum(c, l) * V[c][l];
#pragma unroll
        for (int d = 0; d < ND; ++d) {
            if (sg[c][d] == 0) pmb[d] += wb * weight(c, d);
            else ppb[d] += wb * weight(c, d);
        }
    }
#pragma unroll
    for (int d = 0; d < ND; ++d) {
        ppb[d] += totb[d];
        pmb[d] += totb[d];
    }
    T Ab[ND][2][3], Pb[ND][2], Cpb[NP][2][2];
#pragma unroll
    for (int d = 0; d < ND; ++d)
#pragma unroll
        for (int s = 0; s < 2; ++s) {
            Pb[d][s] = 0;
#pragma unroll
            for (int l = 0; l < 3; ++l) Ab[d][s][l] = 0;
        }
#pragma unroll
    for (int p = 0; p < NP; ++p)
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
            for (int b = 0; b < 2; ++b) Cpb[p][a][b] = 0;
#pragma unroll
    for (int c = 0; c < NC; ++c) {
        const T wc = weight(c, -1);
        T rb = 0;   // V_c . its cotangent
#pragma unroll
        for (int l = 0; l < 3; ++l) {
            T vb = qsum(c, l) * wc;
            if (l < ND) {
                if (c == cmx[l % ND]) vb += ppb[l % ND];
                if (c == cmn[l % ND]) vb -= pmb[l % ND];
            }
            rb += vb * V[c][l];
            const T asb = vb * rr[c];
#pragma unroll
            for (int d = 0; d < ND; ++d) Ab[d][sg[c][d]][l] += asb;
        }
        const T rho2b = (T)-0.5 * rb * (rr[c] * rr[c]);
#pragma unroll
        for (int d = 0; d < ND; ++d) Pb[d][sg[c][d]] += rho2b;
#pragma unroll
        for (int p = 0; p < NP; ++p) Cpb[p][sg[c][pd[p]]][sg[c][pe[p] % ND]] -= (T)2 * rho2b;
    }
    vjp_phase();
    T Sb[3][3];
#pragma unroll
    for (int m = 0; m < 3; ++m)
#pragma unroll
        for (int n = 0; n < 3; ++n) Sb[m][n] = 0;
    T strb = 0;
    T* ub = ubar ? ubar + 54 * I.coff + cl : nullptr;
#pragma unroll
    for (int d = 0; d < ND; ++d)
#pragma unroll
        for (int s = 0; s < 2; ++s) {
            const T sdb = -Ab[d][s][d];
            const T ghd = (s == 0 ? coef[d] : -coef[d]) - inv_abc * Q[d][s][d];
            T trub = 0;
            if (lam_on) {
                trub = Jpb * Q[d][s][d] + Ab[d][s][d] * str;
                strb += Ab[d][s][d] * (U(d, s, 0) + U(d, s, 4) + U(d, s, 8));
            }
#pragma unroll
            for (int l = 0; l < 3; ++l)
#pragma unroll
                for (int n = 0; n < 3; ++n) {
                    const T v = U(d, s, 3 * l + n);
                    T a = gb[3 * l + n] * ghd + gb[3 * d + n] * (inv_abc * Q[d][s][l]);
                    if (l != d) a += (T)2 * v * Pb[d][s];
                    if (l != d && l < ND) {   // C: the pair of axes d and l
                        const int p = (ND == 3) ? ((l == (d + 1) % 3) ? d : l) : 0;
#pragma unroll
                        for (int b = 0; b < 2; ++b)
                            a += (pd[p] == d ? Cpb[p][s][b] : Cpb[p][b][s]) * U(l % ND, b, 3 * d + n);
                    }
                    a += Ab[d][s][l] * S[d][n] + sdb * S[l][n];
                    Sb[d][n] += Ab[d][s][l] * v;
                    Sb[l][n] += sdb * v;
                    if (lam_on) {
                        if (n == d) {
                            a -= Jpb * Q[d][s][l] + Ab[d][s][l] * str;
                            strb -= Ab[d][s][l] * v;
                        }
                        if (l == n) a += trub;
                    }
                    if (ub && valid) ub[(long long)((2 * d + s) * 9 + 3 * l + n) * cells] = a;
                }
        }
    if (lam_on) {
#pragma unroll
        for (int i = 0; i < 3; ++i) Sb[i][i] += strb * Lam / (T)3;
    }
    if (!valid) return;
    if (sigbar) {
        T* sb = sigbar + I.soff + cl;
        sb[0] = Sb[0][0];
        sb[cells] = Sb[0][1] + Sb[1][0];
        sb[2 * cells] = Sb[0][2] + Sb[2][0];
        sb[3 * cells] = Sb[1][1];
        sb[4 * cells] = Sb[1][2] + Sb[2][1];
        sb[5 * cells] = Sb[2][2];
        // parameter partials: <sigbar, sigma_int> (mu), tr sigbar tr sigma_int (nu through lambda),
        // and the diagonal of sigbar (the applied load)
        const double sb6[6] = {(double)Sb[0][0], (double)(Sb[0][1] + Sb[1][0]), (double)(Sb[0][2] + Sb[2][0]),
                               (double)Sb[1][1], (double)(Sb[1][2] + Sb[2][1]), (double)Sb[2][2]};
        double dot = 0.0;
#pragma unroll
        for (int c = 0; c < 6; ++c) dot += sb6[c] * (double)s6[c];
        lsum[0] += dot;
        lsum[1] += (sb6[0] + sb6[3] + sb6[5]) * ((double)s6[0] + (double)s6[3] + (double)s6[5]);
        lsum[2] += sb6[0];
        lsum[3] += sb6[3];
        lsum[4] += sb6[5];
    }
    // Word 3 holds the selections of slots 24..26 in bits 0..11; bits 12..31 record the corners
    // that attain the directional max / min speeds (index + 1, 0 = the zero entry), base 9.
    {
        uint32_t code = 0u, scale = 1u;
#pragma unroll
        for (int d = 0; d < ND; ++d) {
            code += (uint32_t)(cmx[d] + 1) * scale;
            scale *= 9u;
            code += (uint32_t)(cmn[d] + 1) * scale;
            scale *= 9u;
        }
        fw[3] |= code << 12;
    }
    uint32_t* fl = flags + 4 * I.coff + cl;
#pragma unroll
    for (int q = 0; q < 4; ++q) fl[(long long)q * cells] = fw[q];
}

// Bound by instruction issue (FP32: 5600 warp instructions per 32 cells, 55% of the slots, with instruction-cache
// misses of its 90 KB of code as the largest stall). Four FP32 blocks per SM (128 registers) instead of two,
// two FP64 ones with 0.4 KB of spills instead of 2 KB; the reverse of one step at 64^3 FP32 583 -> 525 us (with
// k_param_reduce), 32^3 FP64 223 -> 181. Three FP32 blocks without spills: 250 us per VJP against 213.
template <typename T>
__global__ void __launch_bounds__(VJP_THREADS, sizeof(T) == 4 ? 4 : 2) k_vjp_cells(const InstDev* __restrict__ insts, int n_inst,
                                                           const int* __restrict__ pre,
                                                           const T* beta, const T* sig,
                                                           const T* gbar, double t,
                                                           T* ubar, uint32_t* flags,
                                                           T* sigbar, double* bload) {
    __shared__ double red[VJP_THREADS / 32];
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T* us = reinterpret_cast<T*>(smem_raw) + threadIdx.x;
    const int ii = find_instance(pre, n_inst, blockIdx.x);
    const InstDev& I = insts[ii];
    const long long cell = (long long)(blockIdx.x - pre[ii]) * VJP_THREADS + threadIdx.x;
    const bool valid = cell < I.cells;
    pdl_wait();
    double lsum[VJP_PARTS] = {0.0, 0.0, 0.0, 0.0, 0.0};
    if (I.nd == 3)
        vjp_cell<T, 3>(I, valid ? cell : 0, valid, beta, sig, gbar, t, ubar, flags, sigbar, lsum, us);
    else
        vjp_cell<T, 2>(I, valid ? cell : 0, valid, beta, sig, gbar, t, ubar, flags, sigbar, lsum, us);
    if (!sigbar) return;
#pragma unroll
    for (int i = 0; i < VJP_PARTS; ++i) {
        double s = bsum<T>(lsum[i], red);
        if (threadIdx.x == 0) bload[VJP_PARTS * blockIdx.x + i] = s;
    }
}

// out = c (L^T g) + a1 x1 + a2 x2 + a3 x3 (absent x terms skipped), L^T g = ih * gather + addend.
template <typename T>
struct Axpy {
    T c;
    const T* x[3];
    T a[3];
};

template <typename T, int ND>
__device__ __forceinline__ void gather_cell(const InstDev& I, long long y, const T* __restrict__ ubar,
                                            const uint32_t* __restrict__ flags, const T* __restrict__ addend,
                                            const Axpy<T>& ax, T* out) {
    const long long cells = I.cells;
    Nbr nb[ND];
    {
        int i0, i1, i2;
        cell_coords(y, ND, I.n1, I.n2, i0, i1, i2);
        if (ND == 3) {
            nb[0] = make_nbr(i0, I.n0, I.n1 * I.n2);
            nb[1] = make_nbr(i1, I.n1, I.n2);
            nb[ND - 1] = make_nbr(i2, I.n2, 1);
        } else {
            nb[0] = make_nbr(i0, I.n0, I.n1);
            nb[ND - 1] = make_nbr(i1, I.n1, 1);
        }
    }
    const T ih = (T)I.inv_h;
    const T* ub = ubar + 54 * I.coff + y;
    const uint32_t* fl = flags + 4 * I.coff + y;
    // Along one axis u+_x = (d_x - (e_x+1 or e_x or 0) / 2) / h and u-_x = (d_x-1 + (e_x or e_x-1 or 0) / 2) / h with the
    // differences d_x = u_x+1 - u_x, e_x = u_x+1 - 2 u_x + u_x-1 and the recorded selections, so with the cotangents
    // P of u+ and M of u-
    //   D_x = P_x + M_x+1,  E_x = (M_x [1] + M_x+1 [2] - P_x-1 [1] - P_x [2]) / 2   ([k]: selection k at that cell)
    // and the value's cotangent is D_y-1 - D_y + E_y-1 - 2 E_y + E_y+1: 8 loads and about 45 instructions per component
    // and axis. (The five cells' coefficients formed one by one took twice the instructions.)
    T acc[9];
#pragma unroll
    for (int c = 0; c < 9; ++c) acc[c] = 0;
#pragma unroll
    for (int d = 0; d < ND; ++d) {
        const int off[5] = {nb[d].m2, nb[d].m1, 0, nb[d].p1, nb[d].p2};   // cells y-2 .. y+2
        uint32_t fw[5][4];
#pragma unroll
        for (int k = 0; k < 5; ++k)
#pragma unroll
            for (int w = 0; w < 4; ++w) fw[k][w] = (fl + (long long)w * cells)[off[k]];
#pragma unroll
        for (int c = 0; c < 9; ++c) {
            const T* up = ub + (long long)(2 * d * 9 + c) * cells;
            const T* um = up + 9 * cells;
            const int slot = c * 3 + d, w = slot >> 3, bit = 4 * (slot & 7);
            T P[5], M[5];   // P at y-2 .. y+1, M at y-1 .. y+2
#pragma unroll
            for (int k = 0; k < 4; ++k) P[k] = up[off[k]];
#pragma unroll
            for (int k = 1; k < 5; ++k) M[k] = um[off[k]];
            auto p = [&](int k, int sel) { return (fw[k][w] >> (bit + sel - 1)) & 1u ? P[k] : (T)0; };
            auto m = [&](int k, int sel) { return (fw[k][w] >> (bit + sel + 1)) & 1u ? M[k] : (T)0; };
            const T em = (m(1, 1) + m(2, 2)) - (p(0, 1) + p(1, 2));   // 2 E_y-1, 2 E_y, 2 E_y+1
            const T e0 = (m(2, 1) + m(3, 2)) - (p(1, 1) + p(2, 2));
            const T ep = (m(3, 1) + m(4, 2)) - (p(2, 1) + p(3, 2));
            acc[c] += ((P[1] + M[2]) - (P[2] + M[3])) + ((T)0.5 * (em + ep) - e0);
        }
    }
#pragma unroll
    for (int c = 0; c < 9; ++c) {
        const long long o = I.foff + (long long)c * cells + y;
        T v = acc[c] * ih;
        if (addend) v += addend[o];
        v *= ax.c;
#pragma unroll
        for (int k = 0; k < 3; ++k)
            if (ax.x[k]) v += ax.a[k] * ax.x[k][o];
        acc[c] = v;
    }
    // all loads before the first store: out may be an x term (same element), and no load can pass a store
#pragma unroll
    for (int c = 0; c < 9; ++c) out[I.foff + (long long)c * cells + y] = acc[c];
}

template <typename T>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 4 : 2) k_vjp_gather(const InstDev* __restrict__ insts, int n_inst,
                                                    const int* __restrict__ pre, const T* ubar,
                                                    const uint32_t* flags,
                                                    const T* addend, const Axpy<T> ax,
                                                    T* out) {   // out may alias an x term (same element)
    const int ii = find_instance(pre, n_inst, blockIdx.x);
    const InstDev& I = insts[ii];
    const long long y = (long long)(blockIdx.x - pre[ii]) * blockDim.x + threadIdx.x;
    pdl_wait();
    if (y >= I.cells) return;
    if (I.nd == 3) gather_cell<T, 3>(I, y, ubar, flags, addend, ax, out);
    else gather_cell<T, 2>(I, y, ubar, flags, addend, ax, out);
}

// Per-instance sums of the block partials of the load cotangent, added to the caller's array.
__global__ void __launch_bounds__(256) k_vjp_load_reduce(const int* __restrict__ pre, const double* bload,
                                                         double* out) {
    __shared__ double red[8];
    const int ii = blockIdx.x;
    pdl_wait();
    for (int i = 0; i < 3; ++i) {
        double acc = 0.0;
        for (int b = pre[ii] + threadIdx.x; b < pre[ii + 1]; b += blockDim.x) acc += bload[VJP_PARTS * b + 2 + i];
        acc = bsum<double>(acc, red);
        if (threadIdx.x == 0) out[3 * ii + i] += acc;
    }
}

// Parameter cotangents of one stage, scaled by the stage weight c and added to pbar (CDD_PBAR
// doubles per instance): [0] <sigbar, sigma_int>, [1] tr sigbar . tr sigma_int, [2] the k-space
// sum of the nu derivative per unit dA (from the green-block partials), [3..5] the diagonal of
// sigbar (load), [6..8] the same times (t - load_t0).
// One block per instance and sum (blockIdx.y; one block for all six took 14 us at 64^3).
__global__ void __launch_bounds__(256) k_param_reduce(const InstDev* __restrict__ insts,
                                                      const int* __restrict__ pre_v, const double* bpart,
                                                      const int* __restrict__ pre_g, const double* gpart,
                                                      double c, double t, double* pbar) {
    __shared__ double red[8];
    const int ii = blockIdx.x, i = blockIdx.y;
    const bool k = i == VJP_PARTS;   // the k-space sum
    const int* pre = k ? pre_g : pre_v;
    const int b0 = pre[ii], b1 = pre[ii + 1];
    pdl_wait();
    const double* src = k ? gpart : bpart + i;
    const int stride = k ? 1 : VJP_PARTS;
    double acc = 0.0;
    if (src) {
#pragma unroll 4
        for (int b = b0 + threadIdx.x; b < b1; b += 256) acc += src[(long long)stride * b];
    }
    const double v = bsum<double>(acc, red);
    if (threadIdx.x == 0) {
        double* o = pbar + CDD_PBAR * ii;
        if (k) o[2] += c * v;
        else if (i < 2) o[i] += c * v;
        else {
            o[1 + i] += c * v;
            o[4 + i] += c * (t - insts[ii].load_t0) * v;
        }
    }
}

}  // namespace

cudaError_t adjoint_set_attributes(int precision) {
    return precision == CDD_F32 ? set_dyn_smem_limit(k_vjp_cells<float>, SIZE_MAX) : set_dyn_smem_limit(k_vjp_cells<double>, SIZE_MAX);
}

cudaError_t launch_flux_branches(const PlanCore& P, const void* beta, double t, uint32_t* flags, cudaStream_t st) {
    const LaunchShape& V = P.vjp;
    cudaError_t e;
    if ((e = launch_stress(P, beta, P.d_sigma, st))) return e;
    if (P.precision == CDD_F32)
        launch_pdl(k_vjp_cells<float>, V.blocks, VJP_THREADS, vjp_smem<float>(), st, P.d_inst, P.n_inst, V.d_pre, (const float*)beta,
                                                            (const float*)P.d_sigma, nullptr, t, nullptr, flags,
                                                            nullptr, P.d_bload);
    else
        launch_pdl(k_vjp_cells<double>, V.blocks, VJP_THREADS, vjp_smem<double>(), st, P.d_inst, P.n_inst, V.d_pre, (const double*)beta,
                                                             (const double*)P.d_sigma, nullptr, t, nullptr, flags,
                                                             nullptr, P.d_bload);
    return cudaGetLastError();
}

cudaError_t launch_vjp_stage(const PlanCore& P, const void* v, const void* sig_v, const void* phi_v, double t,
                             const void* gbar, double c, const void* const x[3], const double a[3], void* out,
                             double* pbar, cudaStream_t st) {
    const LaunchShape& V = P.vjp;
    const LaunchShape& G = P.obs;
    cudaError_t e;
    const bool f32 = (P.precision == CDD_F32);
    if (f32)
        launch_pdl(k_vjp_cells<float>, V.blocks, VJP_THREADS, vjp_smem<float>(), st, P.d_inst, P.n_inst, V.d_pre, (const float*)v,
                                                            (const float*)sig_v, (const float*)gbar, t,
                                                            (float*)P.d_ubar, P.d_flags, (float*)P.d_sb6, P.d_bload);
    else
        launch_pdl(k_vjp_cells<double>, V.blocks, VJP_THREADS, vjp_smem<double>(), st, P.d_inst, P.n_inst, V.d_pre, (const double*)v,
                                                             (const double*)sig_v, (const double*)gbar, t,
                                                             (double*)P.d_ubar, P.d_flags, (double*)P.d_sb6,
                                                             P.d_bload);
    if ((e = cudaGetLastError())) return e;
    if ((e = launch_stress_adjoint(P, P.d_sb6, P.d_adj9, st, pbar ? phi_v : nullptr, pbar ? P.d_gpart : nullptr)))
        return e;
    if (pbar) {
        launch_pdl(k_param_reduce, dim3(P.n_inst, VJP_PARTS + 1), 256, 0, st, P.d_inst, V.d_pre, P.d_bload, P.pass[PASS_GREEN].d_pre,
                                                 phi_v ? P.d_gpart : nullptr, c, t, pbar);
        if ((e = cudaGetLastError())) return e;
    }
    if (f32) {
        Axpy<float> ax{(float)c, {(const float*)x[0], (const float*)x[1], (const float*)x[2]},
                       {(float)a[0], (float)a[1], (float)a[2]}};
        launch_pdl(k_vjp_gather<float>, G.blocks, 256, 0, st, P.d_inst, P.n_inst, G.d_pre, (const float*)P.d_ubar, P.d_flags,
                                                     (const float*)P.d_adj9, ax, (float*)out);
    } else {
        Axpy<double> ax{c, {(const double*)x[0], (const double*)x[1], (const double*)x[2]}, {a[0], a[1], a[2]}};
        launch_pdl(k_vjp_gather<double>, G.blocks, 256, 0, st, P.d_inst, P.n_inst, G.d_pre, (const double*)P.d_ubar,
                                                      P.d_flags, (const double*)P.d_adj9, ax, (double*)out);
    }
    return cudaGetLastError();
}

cudaError_t launch_flux_vjp(const PlanCore& P, const void* beta, double t, const void* gbar, void* sigbar,
                            void* betabar, double* load_bar, cudaStream_t st) {
    const LaunchShape& V = P.vjp;
    const LaunchShape& G = P.obs;
    cudaError_t e;
    if ((e = launch_stress(P, beta, P.d_sigma, st))) return e;
    if (P.precision == CDD_F32) {
        launch_pdl(k_vjp_cells<float>, V.blocks, VJP_THREADS, vjp_smem<float>(), st, P.d_inst, P.n_inst, V.d_pre, (const float*)beta,
                                                            (const float*)P.d_sigma, (const float*)gbar, t,
                                                            (float*)P.d_ubar, P.d_flags, (float*)sigbar, P.d_bload);
    } else {
        launch_pdl(k_vjp_cells<double>, V.blocks, VJP_THREADS, vjp_smem<double>(), st, P.d_inst, P.n_inst, V.d_pre, (const double*)beta,
                                                             (const double*)P.d_sigma, (const double*)gbar, t,
                                                             (double*)P.d_ubar, P.d_flags, (double*)sigbar,
                                                             P.d_bload);
    }
    if ((e = cudaGetLastError())) return e;
    if (load_bar) launch_pdl(k_vjp_load_reduce, P.n_inst, 256, 0, st, V.d_pre, P.d_bload, load_bar);
    if ((e = launch_stress_adjoint(P, sigbar, P.d_adj9, st))) return e;
    if (P.precision == CDD_F32) {
        const Axpy<float> ax{1.f, {nullptr, nullptr, nullptr}, {0.f, 0.f, 0.f}};
        launch_pdl(k_vjp_gather<float>, G.blocks, 256, 0, st, P.d_inst, P.n_inst, G.d_pre, (const float*)P.d_ubar, P.d_flags,
                                                     (const float*)P.d_adj9, ax, (float*)betabar);
    } else {
        const Axpy<double> ax{1.0, {nullptr, nullptr, nullptr}, {0.0, 0.0, 0.0}};
        launch_pdl(k_vjp_gather<double>, G.blocks, 256, 0, st, P.d_inst, P.n_inst, G.d_pre, (const double*)P.d_ubar,
                                                      P.d_flags, (const double*)P.d_adj9, ax, (double*)betabar);
    }
    return cudaGetLastError();
}

}  // namespace cdd
