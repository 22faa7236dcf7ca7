// Central-upwind Hamilton-Jacobi flux of the plastic distortion and the TVD-RK3 stage update,
// one thread per cell, plus the per-instance CFL time step.
//
// Reference semantics (Plasticity/FieldDynamics/CentralUpwindHJ3D.py L11-34, L99-271 and
// Plasticity/FieldDynamics/CentralUpwindHJBetaPDynamics3D.py L34-221):
//  * limited one-sided derivatives along each axis (FindDerivatives, theta = 1, Dx = 1/shape[-1]):
//      d_i = u_{i+1} - u_i, D1_i = (d_{i+1} - d_i)/h^2, D2_i = (d_{i+1} - d_{i-1})/(2 h^2),
//      dd_i = minmod(D1_i, D2_i, D1_{i-1}),
//      u+ = d_0/h - h dd_0 / 2,  u- = d_{-1}/h + h dd_{-1} / 2;
//  * at each of the 2^nd corners s (a choice of u+ or u- per axis) the dislocation velocity
//      V_l = [sum_n sum_d (u_d)_ln sigma_dn - sum_mn (u_l)_mn sigma_mn (+ Lambda terms)] / |rho|,
//      |rho|^2 = ME + sum_d |u_d|^2 - sum_d sum_j (u_d)_dj^2 - 2 sum_{d<e} sum_j (u_d)_ej (u_e)_dj,
//    and the Hamiltonian H_ij = sum_d V_d (u_d)_ij - sum_l V_l (u_i)_lj (+ Lambda trace term);
//  * directional speeds a+ = max(0, V_x over corners), a- = |min(0, V_x over corners)|, ...,
//    a_tot = a+ + a- + ME; rhs = -sum_s w_s H_s / (a_tot b_tot c_tot)
//    + sum_d (u_d+ - u_d-) a_d- a_d+ / a_d,tot, with w_s the product over axes of a_d- for a '+'
//    choice and a_d+ for a '-' choice; CFL speed = a_tot + b_tot + c_tot.
//
// Evaluation. V is linear in each axis' derivative tensor, so per axis and sign the kernel forms
// the 3-vector A[d][s] once; V at a corner is the sum of three of them over |rho|. |rho|^2 splits
// into per-axis terms P[d][s] and pair terms C_de[s_d][s_e]. The corner-weighted sum of H
// contracts to 6 scalars G[d][s] and 18 scalars Q[i][s][l] (sums of w V over the corners with a
// given sign on one axis). No per-corner H or derivative tensor is formed. The derivatives are
// computed once and stay in registers: pass 1 accumulates A, P, C from them, pass 2 forms rhs.
#include <cudaTypedefs.h>

#include "cdd_internal.cuh"
#include "fp64_math.cuh"

namespace cdd {

// The limiter of FindDerivatives is MinMod3(D1_i, D2_i, D1_{i-1}) (NumericalMethods.py L367-378)
// with D2_i = (D1_i + D1_{i-1}) / 2: the middle argument is the mean of the outer two. It has the
// sign of both when they agree and its magnitude is never below the smaller of theirs (also after
// rounding: fl(a + c) / 2 >= min(a, c) for a, c > 0), so the 3-way minmod equals the 2-way one:
// min(|a|, |c|) with their common sign, 0 when the signs differ or one is zero. That is the median
// of (a, c, 0), which FP32 forms with min / max operations (minmod_pair); FP64, which has none, folds
// the 0 into the factor 1/2 of the derivative (limited_f64).

// 1/sqrt and division of the FP32 form: the hardware approximations (<= 2 ulp).
__device__ __forceinline__ float inv_sqrt(float x) { return rsqrtf(x); }
__device__ __forceinline__ float fdiv(float a, float b) { return __fdividef(a, b); }

// Shared-memory tiles of the 2.5-D march: a block owns TXS x TYS cells of a plane (last axis x
// contiguous) and walks along axis 0 (3-D). Each staged plane holds all 9 components of a box of
// RY rows (2-row halo in y) by RX columns starting OX cells left of the tile: RX/OX keep the box's
// x origin on a 16-byte boundary (TMA), i.e. 40/4 for FP32 and 36/2 for FP64.
constexpr int TXS = 32;
template <typename T> struct TileGeom;
template <> struct TileGeom<float> { static constexpr int RX = 40, OX = 4, NS = 6, TY = 8; };
template <> struct TileGeom<double> { static constexpr int RX = 36, OX = 2, NS = 5, TY = 4; };
template <typename T> __host__ __device__ constexpr int tile_ry() { return TileGeom<T>::TY + 4; }
template <typename T> __host__ __device__ constexpr int st_threads() { return TXS * TileGeom<T>::TY; }
constexpr int ST_BLOCKS = 2;   // per SM
template <typename T> __host__ __device__ constexpr int tile_pp() { return tile_ry<T>() * TileGeom<T>::RX; }   // per component

// What a block keeps of beta_s. FP32 3-D: a ring of plane boxes. FP64 3-D: the box of the current plane only, and
// for each thread the five values z-2 .. z+2 of its own column (`column`), which it copies and reads back itself:
// a block starts after one box instead of five (FP64 flux at one plane per block, 128^3: 532 -> 361 us, 64^3 60 ->
// 54 us). Its 73 KB would let three blocks run, but at the 168 registers that leaves each thread the spills
// cost more than the warps give (256^3 2.65 ms against 1.65; 160-thread blocks at 200 registers 2.50).
template <typename T, int ND> __host__ __device__ constexpr bool own_columns() { return sizeof(T) == 8 && ND == 3; }
template <typename T, int ND>
struct TileView {
    static constexpr int RX = TileGeom<T>::RX, PP = tile_pp<T>();
    static constexpr bool OWN = own_columns<T, ND>();
    const T* sm;       // shared memory base
    const T* column;   // this thread's column slots (own_columns)
    int so[5];         // element offsets of the planes z-2 .. z+2 (3-D), in sm or column; so[2] = current plane
    int idx;           // in-plane offset of this thread's cell (halo included)
    __device__ __forceinline__ T center(int c) const {
        return OWN ? column[so[2] + c * st_threads<T>()] : sm[so[2] + c * PP + idx];
    }
    __device__ __forceinline__ void load5(int c, int d, T* v) const {
        if (ND == 3 && d == 0) {
#pragma unroll
            for (int q = 0; q < 5; ++q) v[q] = OWN ? column[so[q] + c * st_threads<T>()] : sm[so[q] + c * PP + idx];
        } else {
            const int st = (d == ND - 1) ? 1 : RX;
            const T* p = sm + (OWN ? 0 : so[2]) + c * PP + idx;
            v[0] = p[-2 * st]; v[1] = p[-st]; v[2] = p[0]; v[3] = p[st]; v[4] = p[2 * st];
        }
    }
};

// ---- TMA and mbarrier primitives (inline PTX, sm_100a) ----
__device__ __forceinline__ uint32_t smem_addr(const void* p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_mbar_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void fence_proxy_async() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ bool mbar_test(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// Bounded wait: gives up after ~2^22 polls (well above any TMA latency) and reports false.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) {
    for (int i = 0; i < (1 << 22); ++i) {
        if (mbar_test(bar, parity)) return true;
        if (i > 64) __nanosleep(64);
    }
    return false;
}
__device__ __forceinline__ void tma_load_5d(void* dst, const CUtensorMap* map, uint64_t* bar, int x, int y,
                                            int z, int c, int n) {
    asm volatile(
        "cp.async.bulk.tensor.5d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%2, %3, %4, %5, %6}], [%7];" ::"r"(smem_addr(dst)),
        "l"(map), "r"(x), "r"(y), "r"(z), "r"(c), "r"(n), "r"(smem_addr(bar))
        : "memory");
}

// One element (4 or 8 bytes) global -> shared without a register round trip; each thread waits for
// its own copies only (cp.async.wait_all), so no block barrier is needed when a thread reads back
// what it copied.
__device__ __forceinline__ void cp_async_elem(float* dst, const float* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_elem(double* dst, const double* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_own() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }
// Hint: bring the 128-byte line at p into L2 (no register result, no completion to wait for).
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];\n" ::"l"(p)); }

// u+ and u- from the five values u_{-2} .. u_{+2} along one axis. The limiter arguments D1, D2
// of FindDerivatives all carry 1/h^2; minmod is positively homogeneous, so the kernel limits the
// undivided second differences and applies 1/h once: u+ = (d_0 - mm/2) / h, u- = (d_-1 + mm_-1/2) / h.
// The two limiters of one axis share their middle argument em1: minmod(a, em1) is the median of
// (a, em1, 0), i.e. a clamped to [min(em1, 0), max(em1, 0)], so FP32 forms those bounds once.
__device__ __forceinline__ void minmod_pair(float e0, float em1, float em2, float& dd0, float& ddm) {
    const float lo = fminf(em1, 0.0f), hi = fmaxf(em1, 0.0f);
    dd0 = fminf(fmaxf(e0, lo), hi);
    ddm = fminf(fmaxf(em2, lo), hi);
}

// ---- FP32 flux with paired arithmetic ----
// Every quantity of the central-upwind flux that comes in a forward / backward pair (one-sided
// derivatives u+ / u-, the A, S_d, P, trace and Q sums, the final per-axis coefficients) is kept
// as one float2 (x: forward, y: backward) and updated with the packed FP32 instructions
// (__ffma2_rn, __fadd2_rn, __fmul2_rn: two lanes per instruction, each rounded as the scalar
// operation). The corners pair up along the last axis: corners 2m and 2m + 1 differ only in
// its sign. Same formulas as the scalar path; the rhs sums are regrouped per one-sided
// derivative: rhs_ij = sum_d [(c_d - Q+_dd) (u+_d)_ij + (-c_d - Q-_dd) (u-_d)_ij]
//                      + [i < ND] sum_{s,l} Q^s_il (u^s_i)_lj,
// with c_d = a+_d a-_d / tot_d, i.e. -H / (a_tot b_tot c_tot) + the viscous term of the scalar form.
__device__ __forceinline__ float2 f2(float a, float b) { return make_float2(a, b); }
// The differences in packed form around the centre c = u_0: P = (u_1, u_-1) - (c, c) = (d0, -dm1),
// Q = (u_2, u_-2) - (c, c), and the limiter's outer arguments (e0, em2) = Q - 2 P in one packed
// multiply-add (e0 = d1 - d0 and em2 = dm1 - dm2 up to rounding); the middle one em1 = d0 - dm1 =
// P.x + P.y and the one-sided derivatives (d0 - dd0 / 2, dm1 + ddm / 2) / h are formed as the
// scalar form does.
__device__ __forceinline__ float2 derivs5_f2(const float* v, float ih) {
    const float2 c2 = f2(v[2], v[2]);
    const float2 m1 = f2(-1.0f, -1.0f);
    const float2 P = __ffma2_rn(c2, m1, f2(v[3], v[1]));
    const float2 Q = __ffma2_rn(c2, m1, f2(v[4], v[0]));
    const float2 E = __ffma2_rn(P, f2(-2.0f, -2.0f), Q);
    float dd0, ddm;
    minmod_pair(E.x, P.x + P.y, E.y, dd0, ddm);
    return __fmul2_rn(__ffma2_rn(f2(dd0, ddm), f2(-0.5f, -0.5f), P), f2(ih, -ih));
}
__device__ __forceinline__ float lane(const float2& v, int s) { return s ? v.y : v.x; }
// Maximum / minimum that return NaN when either argument is NaN (fmaxf / fminf drop it).
__device__ __forceinline__ float fmax_nan(float a, float b) {
    float d;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(d) : "f"(a), "f"(b));
    return d;
}
__device__ __forceinline__ float fmin_nan(float a, float b) {
    float d;
    asm("min.NaN.f32 %0, %1, %2;" : "=f"(d) : "f"(a), "f"(b));
    return d;
}
// The same over three arguments in one instruction (three-input min / max, sm_100).
__device__ __forceinline__ float fmax3_nan(float a, float b, float c) {
    float d;
    asm("max.NaN.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
__device__ __forceinline__ float fmin3_nan(float a, float b, float c) {
    float d;
    asm("min.NaN.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

template <int ND, bool GLIDE>
__device__ __forceinline__ void flux_f32(const TileView<float, ND>& tv, float ih, const float (&S)[3][3],
                                         bool lam_on, bool glide, float Lambda, float (&rhs)[9], float& spd) {
    constexpr int NC = 1 << ND;
    constexpr int NP = (ND == 3) ? 3 : 1;
    const float2 z2 = f2(0.0f, 0.0f);
    float2 U[ND][9];   // (u+_d, u-_d) of component c = 3 l + j (row l, column j)
#pragma unroll
    for (int c = 0; c < 9; ++c)
#pragma unroll
        for (int d = 0; d < ND; ++d) {
            float v5[5];
            tv.load5(c, d, v5);
            U[d][c] = derivs5_f2(v5, ih);
        }
    const float str = lam_on ? (S[0][0] + S[1][1] + S[2][2]) / 3.0f * Lambda : 0.0f;

    // pass 1: A_d l = sum_j (u_d)_lj S_dj, S_d = sum_{l,j} (u_d)_lj S_lj, P_d = sum_{l != d, j} (u_d)_lj^2,
    // tr(u_d), C_de[s_d][s_e] = sum_j (u_d)_ej (u_e)_dj
    float2 A[ND][3], Sd[ND], Pq[ND], trU[ND];
    float Cp[NP][2][2];
#pragma unroll
    for (int d = 0; d < ND; ++d) {
        Sd[d] = z2; Pq[d] = z2; trU[d] = z2;
#pragma unroll
        for (int l = 0; l < 3; ++l) A[d][l] = z2;
    }
#pragma unroll
    for (int p = 0; p < NP; ++p)
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
            for (int b = 0; b < 2; ++b) Cp[p][a][b] = 0.0f;
#pragma unroll
    for (int j = 0; j < 3; ++j) {
#pragma unroll
        for (int d = 0; d < ND; ++d) {
            const float2 sdj = f2(S[d][j], S[d][j]);
#pragma unroll
            for (int l = 0; l < 3; ++l) {
                const float2 u = U[d][3 * l + j];
                A[d][l] = __ffma2_rn(u, sdj, A[d][l]);
                Sd[d] = __ffma2_rn(u, f2(S[l][j], S[l][j]), Sd[d]);
                if (l != d) Pq[d] = __ffma2_rn(u, u, Pq[d]);
            }
            if (lam_on || glide) trU[d] = __fadd2_rn(trU[d], U[d][4 * j]);
            if (lam_on && j == d) {
#pragma unroll
                for (int l = 0; l < 3; ++l) A[d][l] = __ffma2_rn(f2(-str, -str), U[d][3 * l + j], A[d][l]);
            }
        }
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
            for (int b = 0; b < 2; ++b) {
                Cp[0][a][b] += lane(U[0][3 + j], a) * lane(U[1 % ND][j], b);
                if (ND == 3) {
                    Cp[1 % NP][a][b] += lane(U[1 % ND][6 + j], a) * lane(U[2 % ND][3 + j], b);
                    Cp[2 % NP][a][b] += lane(U[2 % ND][j], a) * lane(U[0][6 + j], b);
                }
            }
    }
#pragma unroll
    for (int d = 0; d < ND; ++d) {
        A[d][d] = __fadd2_rn(A[d][d], f2(-Sd[d].x, -Sd[d].y));
        if (lam_on) A[d][d] = __ffma2_rn(f2(str, str), trU[d], A[d][d]);
    }

    // corners: V = (A_x[sx] + A_y[sy] (+ A_z[sz])) / |rho|, paired along the last axis
    float2 V[NC / 2][3];
    if constexpr (ND == 3 && !GLIDE) {
        // pair m = 2 sx + sy, lanes sz = 0, 1: the x and y parts of |rho|^2 and of A are common to
        // the pair, the z parts come as pairs
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            const int sx = m >> 1, sy = m & 1;
            const float cr = (float)ME + lane(Pq[0], sx) + lane(Pq[1 % ND], sy) - 2.0f * Cp[0][sx][sy];
            const float2 cz = f2(Cp[1 % NP][sy][0] + Cp[2 % NP][0][sx], Cp[1 % NP][sy][1] + Cp[2 % NP][1][sx]);
            const float2 r2 = __ffma2_rn(cz, f2(-2.0f, -2.0f), __fadd2_rn(f2(cr, cr), Pq[2 % ND]));
            const float2 inv2 = f2(inv_sqrt(r2.x), inv_sqrt(r2.y));
#pragma unroll
            for (int l = 0; l < 3; ++l) {
                const float ca = lane(A[0][l], sx) + lane(A[1 % ND][l], sy);
                V[m][l] = __fmul2_rn(__fadd2_rn(f2(ca, ca), A[2 % ND][l]), inv2);
            }
        }
    } else {
#pragma unroll
    for (int m = 0; m < NC / 2; ++m) {
        float av[2][3], inv[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int c = 2 * m + h;
            const int sx = (c >> (ND - 1)) & 1, sy = (c >> (ND - 2)) & 1;
            const int sz = (ND == 3) ? (c & 1) : 0;
            float rho2;
            if (ND == 3)
                rho2 = (float)ME + lane(Pq[0], sx) + lane(Pq[1 % ND], sy) + lane(Pq[2 % ND], sz)
                       - 2.0f * (Cp[0][sx][sy] + Cp[1 % NP][sy][sz] + Cp[2 % NP][sz][sx]);
            else
                rho2 = (float)ME + lane(Pq[0], sx) + lane(Pq[1 % ND], sy) - 2.0f * Cp[0][sx][sy];
            inv[h] = inv_sqrt(rho2);
#pragma unroll
            for (int l = 0; l < 3; ++l) {
                float a = lane(A[0][l], sx) + lane(A[1 % ND][l], sy);
                if (ND == 3) a += lane(A[2 % ND][l], sz);
                av[h][l] = a;
            }
            if (GLIDE && glide) {
                // glide-only projection (CentralUpwindHJBetaPGlideOnlyDynamics.py L152-201, 2-D L96-129):
                // g_d = tr(u_d) - sum_e (u_e)_{d e}, v += g (ME + v.g) / (ME + g.g), then v / |rho|
                const int sgc[3] = {sx, sy, sz};
                float gv[3];
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    float Dd = 0.0f;
#pragma unroll
                    for (int e = 0; e < ND; ++e) Dd += lane(U[e][3 * d + e], sgc[e]);
                    const float tr = (d < ND) ? lane(trU[d % ND], sgc[d]) : 0.0f;
                    gv[d] = tr - Dd;
                }
                const float rr = (float)ME + gv[0] * gv[0] + gv[1] * gv[1] + gv[2] * gv[2];
                const float rv = (float)ME + av[h][0] * gv[0] + av[h][1] * gv[1] + av[h][2] * gv[2];
                const float f = fdiv(rv, rr);
#pragma unroll
                for (int l = 0; l < 3; ++l) av[h][l] += gv[l] * f;
            }
        }
#pragma unroll
        for (int l = 0; l < 3; ++l) V[m][l] = __fmul2_rn(f2(av[0][l], av[1][l]), f2(inv[0], inv[1]));
    }
    }
    // one-sided speeds a+_d = max(0, max V_d), a-_d = -min(0, min V_d); weights normalised by
    // tot_d = a+_d + a-_d + ME first (the product of the three totals can underflow FP32). The
    // maxima and minima propagate NaN, so that a NaN anywhere in V reaches the CFL speed.
    float pp[ND], pm[ND], wm[ND], wp[ND];
    spd = 0.0f;
#pragma unroll
    for (int d = 0; d < ND; ++d) {
        float mx = 0.0f, mn = 0.0f;
        if constexpr (ND == 3) {
            // the 8 corners and 0 in four three-input operations each way
            mx = fmax3_nan(fmax3_nan(V[0][d].x, V[0][d].y, V[1][d].x), fmax3_nan(V[1][d].y, V[2][d].x, V[2][d].y),
                           fmax3_nan(V[3][d].x, V[3][d].y, 0.0f));
            mn = fmin3_nan(fmin3_nan(V[0][d].x, V[0][d].y, V[1][d].x), fmin3_nan(V[1][d].y, V[2][d].x, V[2][d].y),
                           fmin3_nan(V[3][d].x, V[3][d].y, 0.0f));
        } else {
#pragma unroll
            for (int m = 0; m < NC / 2; ++m) {
                mx = fmax_nan(mx, fmax_nan(V[m][d].x, V[m][d].y));
                mn = fmin_nan(mn, fmin_nan(V[m][d].x, V[m][d].y));
            }
        }
        pp[d] = mx;
        pm[d] = -mn;
        const float tot = pp[d] + pm[d] + (float)ME;
        spd += tot;
        const float it = fdiv(1.0f, tot);
        wm[d] = pm[d] * it;
        wp[d] = pp[d] * it;
    }

    // Q^s_dl = sum over corners with s_d = s of w_c V_cl (w_c: product of the weights a-_d / tot_d
    // or a+_d / tot_d of the corner's signs)
    float2 Q[ND][3];
#pragma unroll
    for (int d = 0; d < ND; ++d)
#pragma unroll
        for (int l = 0; l < 3; ++l) Q[d][l] = z2;
    if constexpr (ND == 3) {
        // pair m = 2 sx + sy; T_m = w V over its two corners (lanes: sz). Q_z = sum_m T_m lane-wise,
        // Q_x = lane sums of (T_0 + T_1, T_2 + T_3), Q_y = lane sums of (T_0 + T_2, T_1 + T_3)
        float2 w2[4];
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            const float wb = ((m >> 1) ? wp[0] : wm[0]) * ((m & 1) ? wp[1] : wm[1]);
            w2[m] = f2(wb * wm[2], wb * wp[2]);
        }
#pragma unroll
        for (int l = 0; l < 3; ++l) {
            float2 T4[4];
#pragma unroll
            for (int m = 0; m < 4; ++m) T4[m] = __fmul2_rn(w2[m], V[m][l]);
            const float2 a01 = __fadd2_rn(T4[0], T4[1]), a23 = __fadd2_rn(T4[2], T4[3]);
            const float2 b02 = __fadd2_rn(T4[0], T4[2]), b13 = __fadd2_rn(T4[1], T4[3]);
            Q[0][l] = f2(a01.x + a01.y, a23.x + a23.y);
            Q[1 % ND][l] = f2(b02.x + b02.y, b13.x + b13.y);
            Q[2 % ND][l] = __fadd2_rn(a01, a23);
        }
    } else {
#pragma unroll
        for (int m = 0; m < NC / 2; ++m) {
            const int c = 2 * m;
            int sg[2];
            sg[0] = (c >> (ND - 1)) & 1;
            sg[1] = (ND == 3) ? ((c >> 1) & 1) : 0;
            float wb = 1.0f;
#pragma unroll
            for (int d = 0; d < ND - 1; ++d) wb *= (sg[d] == 0) ? wm[d] : wp[d];
            const float2 w2 = f2(wb * wm[ND - 1], wb * wp[ND - 1]);
#pragma unroll
            for (int l = 0; l < 3; ++l) {
                const float2 wv = __fmul2_rn(w2, V[m][l]);
                const float sum = wv.x + wv.y;
#pragma unroll
                for (int d = 0; d < ND - 1; ++d) {
                    if (sg[d] == 0) Q[d][l].x += sum;
                    else Q[d][l].y += sum;
                }
                Q[ND - 1][l] = __fadd2_rn(Q[ND - 1][l], wv);
            }
        }
    }

    // pass 2: rhs
    float2 G[ND];
#pragma unroll
    for (int d = 0; d < ND; ++d) {
        const float coef = pm[d] * wp[d];
        const float2 qdd = (d == 0) ? Q[d][0] : ((d == 1) ? Q[d][1] : Q[d][2]);
        G[d] = f2(coef - qdd.x, -coef - qdd.y);
    }
    float2 Jp2 = z2;   // Lambda trace term, J = -Lambda/3 (Jp2.x + Jp2.y)
    if (lam_on) {
#pragma unroll
        for (int d = 0; d < ND; ++d) {
            const float2 qdd = (d == 0) ? Q[d][0] : ((d == 1) ? Q[d][1] : Q[d][2]);
            Jp2 = __ffma2_rn(qdd, trU[d], Jp2);
        }
    }
#pragma unroll
    for (int j = 0; j < 3; ++j) {
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            float2 acc = __fmul2_rn(G[0], U[0][3 * i + j]);
#pragma unroll
            for (int d = 1; d < ND; ++d) acc = __ffma2_rn(G[d], U[d][3 * i + j], acc);
            if (i < ND) {
#pragma unroll
                for (int l = 0; l < 3; ++l) acc = __ffma2_rn(Q[i % ND][l], U[i % ND][3 * l + j], acc);
            }
            rhs[3 * i + j] = acc.x + acc.y;
        }
        if (lam_on && j < ND) {
#pragma unroll
            for (int l = 0; l < 3; ++l)
                Jp2 = __ffma2_rn(f2(-Q[j % ND][l].x, -Q[j % ND][l].y), U[j % ND][3 * l + j], Jp2);
        }
    }
    if (lam_on) {
        // the trace term enters H_ii, so rhs_ii gets -J / (a_tot b_tot c_tot) (weights normalised)
        const float J = -Lambda / 3.0f * (Jp2.x + Jp2.y);
        rhs[0] -= J;
        rhs[4] -= J;
        rhs[8] -= J;
    }
}

// ---- FP64 flux ----
// The scalar counterpart of flux_f32, with the same regrouping of the rhs per one-sided derivative.
// The derivatives are undivided (times Dx): the velocities are ratios of two forms of the same degree in
// them, so only the ME terms take Dx^2 and the rhs the one factor 1 / Dx.
// Bound by the FP64 pipe (64 lanes per SM and clock: about 930 of its instructions per cell, 0.9 ms at 256^3) and
// by 8 resident warps per SM to hide its latency. All 54 derivatives stay in registers (246, no spills), formed
// once: forming them again for the rhs, with the five-compare minmod, 8 square roots and 8 + 4 divisions
// of the form before it, took 4272 us per 256^3 flux, this 2704 us; with the plane copies under the cell's own
// work (march) and 20 planes per block, 1796 us; with own columns and Newton's rsqrt and reciprocal, 1649 us; with the
// values of NaN, zero and infinite arguments (limited_f64, fp64_math.cuh), 1693 us.
// d + h minmod(e, m) for h = -1/2 or 1/2: the factor is 0 unless the signs of e and m agree (an integer test), and
// times the smaller magnitude otherwise, so the FP64 pipe sees one compare and one multiply-add. A NaN in e (two cells
// away) leaves d, as minmod's 0 does: only the cells whose d or m is NaN become NaN. (A result of arithmetic is a quiet
// NaN: adding its quiet bit to the upper word carries into the sign bit, and for no other value. This test costs 2% of
// a 256^3 flux, 1658 -> 1694 us; forming the rare cells with a NaN again at the end of the march cost as much.)
__device__ __forceinline__ double limited_f64(double d, double e, double m, double h) {
    const double v = fabs(e) < fabs(m) ? e : m;
    const int he = __double2hiint(e);
    const bool same = ((he ^ __double2hiint(m)) | (he ^ (int)((unsigned)he + 0x00080000u))) >= 0;
    return fma(__hiloint2double(same ? __double2hiint(h) : 0, 0), v, d);
}
// (u+, u-) times Dx from u_{-2} .. u_{+2}.
__device__ __forceinline__ void derivs5_f64(const double* v, double& up, double& um) {
    const double dm2 = v[1] - v[0], dm1 = v[2] - v[1], d0 = v[3] - v[2], d1 = v[4] - v[3];
    const double e0 = d1 - d0, em1 = d0 - dm1, em2 = dm1 - dm2;
    up = limited_f64(d0, e0, em1, -0.5);
    um = limited_f64(dm1, em2, em1, 0.5);
}

// meh: ME Dx^2. ring_read(): called once the thread has read all it needs of the ring but its cell's own
// values; false (a plane did not arrive) ends the cell. Returns false then.
template <int ND, bool GLIDE, class F>
__device__ __forceinline__ bool flux_f64(const TileView<double, ND>& tv, double ih, double meh, const double (&S)[3][3],
                                         bool lam_on, bool glide, double Lambda, double (&rhs)[9], double& spd,
                                         const F& ring_read) {
    constexpr int NC = 1 << ND;
    constexpr int NP = (ND == 3) ? 3 : 1;
    double U[ND][2][9];   // u+_d, u-_d of component c = 3 l + j, times Dx
    const double str = lam_on ? (S[0][0] + S[1][1] + S[2][2]) / 3.0 * Lambda : 0.0;

    // A_d l = sum_j (u_d)_lj S_dj (the d-th less sum_{l,j} (u_d)_lj S_lj), P_d = sum_{l != d, j} (u_d)_lj^2, one
    // axis after the other as its derivatives are formed
    double A[ND][2][3], Pq[ND][2], Cp[NP][2][2];
#pragma unroll
    for (int d = 0; d < ND; ++d) {
#pragma unroll
        for (int s = 0; s < 2; ++s) {
            Pq[d][s] = 0.0;
#pragma unroll
            for (int l = 0; l < 3; ++l) A[d][s][l] = 0.0;
        }
#pragma unroll
        for (int c = 0; c < 9; ++c) {
            const int l = c / 3, j = c - 3 * l;
            double v5[5];
            tv.load5(c, d, v5);
            derivs5_f64(v5, U[d][0][c], U[d][1][c]);
#pragma unroll
            for (int s = 0; s < 2; ++s) {
                const double u = U[d][s][c];
                A[d][s][l] = fma(u, S[d][j], A[d][s][l]);
                A[d][s][d] = fma(-u, S[l][j], A[d][s][d]);
                if (l != d) Pq[d][s] = fma(u, u, Pq[d][s]);
            }
        }
        if (lam_on) {
#pragma unroll
            for (int s = 0; s < 2; ++s) {
                A[d][s][d] = fma(str, U[d][s][0] + U[d][s][4] + U[d][s][8], A[d][s][d]);
#pragma unroll
                for (int l = 0; l < 3; ++l) A[d][s][l] = fma(-str, U[d][s][3 * l + d], A[d][s][l]);
            }
        }
    }
    if (!ring_read()) return false;
    // pair terms C_de[s_d][s_e] = sum_j (u_d)_ej (u_e)_dj
#pragma unroll
    for (int p = 0; p < NP; ++p)
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
            for (int b = 0; b < 2; ++b) {
                const int d = p, e = (p + 1) % 3;
                double t = 0.0;
#pragma unroll
                for (int j = 0; j < 3; ++j) t = fma(U[d % ND][a][3 * e + j], U[e % ND][b][3 * d + j], t);
                Cp[p][a][b] = t;
            }

    // corners: V = (A_x[sx] + A_y[sy] (+ A_z[sz])) / |rho|
    double V[NC][3];
#pragma unroll
    for (int c = 0; c < NC; ++c) {
        const int sx = (c >> (ND - 1)) & 1, sy = (c >> (ND - 2)) & 1;
        const int sz = (ND == 3) ? (c & 1) : 0;
        double r2 = fma(-2.0, Cp[0][sx][sy], meh + Pq[0][sx] + Pq[1][sy]);
        if (ND == 3) r2 = fma(-2.0, Cp[1 % NP][sy][sz] + Cp[2 % NP][sz][sx], r2 + Pq[2 % ND][sz]);
        const double inv = rsqrt_f64(r2);
        double av[3];
#pragma unroll
        for (int l = 0; l < 3; ++l) {
            av[l] = A[0][sx][l] + A[1][sy][l];
            if (ND == 3) av[l] += A[2 % ND][sz][l];
        }
        if (GLIDE && glide) {
            // glide-only projection (CentralUpwindHJBetaPGlideOnlyDynamics.py L152-201, 2-D L96-129):
            // g_d = tr(u_d) - sum_e (u_e)_{d e}, v += g (ME + v.g) / (ME + g.g), then v / |rho|
            const int sgc[3] = {sx, sy, sz};
            double gv[3];
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                double Dd = 0.0;
#pragma unroll
                for (int e = 0; e < ND; ++e) Dd += U[e][sgc[e]][3 * d + e];
                const double tr = (d < ND) ? U[d % ND][sgc[d]][0] + U[d % ND][sgc[d]][4] + U[d % ND][sgc[d]][8] : 0.0;
                gv[d] = tr - Dd;
            }
            const double rr = meh + gv[0] * gv[0] + gv[1] * gv[1] + gv[2] * gv[2];
            const double rv = meh + av[0] * gv[0] + av[1] * gv[1] + av[2] * gv[2];
            const double f = rv / rr;
#pragma unroll
            for (int l = 0; l < 3; ++l) av[l] = fma(gv[l], f, av[l]);
        }
#pragma unroll
        for (int l = 0; l < 3; ++l) V[c][l] = av[l] * inv;
    }
    // one-sided speeds a+_d = max(0, max V_d), a-_d = -min(0, min V_d); each axis' weights are divided by its
    // total a+_d + a-_d + ME. A NaN in V is dropped by the compares and carried to the speed by vsum.
    double pp[ND], pm[ND], wm[ND], wp[ND];
    double vsum = 0.0;
    spd = 0.0;
#pragma unroll
    for (int d = 0; d < ND; ++d) {
        double mx = 0.0, mn = 0.0, sum = 0.0;
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            mx = V[c][d] > mx ? V[c][d] : mx;
            mn = V[c][d] < mn ? V[c][d] : mn;
            sum += V[c][d];
        }
        vsum += sum;
        pp[d] = mx;
        pm[d] = -mn;
        const double tot = pp[d] + pm[d] + ME;
        spd += tot;
        const double it = rcp_f64(tot);
        wm[d] = pm[d] * it;
        wp[d] = pp[d] * it;
    }
    if (vsum != vsum) spd = vsum;

    // Q^s_dl = sum over corners with s_d = s of w_c V_cl
    double Q[ND][2][3];
    {
        double w[NC];
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            w[c] = ((c >> (ND - 1)) & 1) ? wp[0] : wm[0];
#pragma unroll
            for (int d = 1; d < ND; ++d) w[c] *= ((c >> (ND - 1 - d)) & 1) ? wp[d] : wm[d];
        }
#pragma unroll
        for (int l = 0; l < 3; ++l) {
            double T[NC];
#pragma unroll
            for (int c = 0; c < NC; ++c) T[c] = w[c] * V[c][l];
            if constexpr (ND == 3) {
                const double y0 = T[0] + T[1], y1 = T[2] + T[3], y2 = T[4] + T[5], y3 = T[6] + T[7];   // by (sx, sy)
                Q[0][0][l] = y0 + y1;
                Q[0][1][l] = y2 + y3;
                Q[1][0][l] = y0 + y2;
                Q[1][1][l] = y1 + y3;
                Q[2 % ND][0][l] = (T[0] + T[2]) + (T[4] + T[6]);
                Q[2 % ND][1][l] = (T[1] + T[3]) + (T[5] + T[7]);
            } else {
                Q[0][0][l] = T[0] + T[1];
                Q[0][1][l] = T[2 % NC] + T[3 % NC];
                Q[1][0][l] = T[0] + T[2 % NC];
                Q[1][1][l] = T[1] + T[3 % NC];
            }
        }
    }

    // rhs_ij = sum_d [(c_d - Q+_dd) (u+_d)_ij + (-c_d - Q-_dd) (u-_d)_ij] + [i < ND] sum_{s,l} Q^s_il (u^s_i)_lj,
    // c_d = a+_d a-_d / tot_d
    double G[ND][2];
#pragma unroll
    for (int d = 0; d < ND; ++d) {
        G[d][0] = fma(pm[d], wp[d], -Q[d][0][d]);
        G[d][1] = -fma(pm[d], wp[d], Q[d][1][d]);
    }
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            double acc = 0.0;
#pragma unroll
            for (int d = 0; d < ND; ++d)
#pragma unroll
                for (int s = 0; s < 2; ++s) acc = fma(G[d][s], U[d][s][3 * i + j], acc);
            if (i < ND) {
#pragma unroll
                for (int s = 0; s < 2; ++s)
#pragma unroll
                    for (int l = 0; l < 3; ++l) acc = fma(Q[i % ND][s][l], U[i % ND][s][3 * l + j], acc);
            }
            rhs[3 * i + j] = acc * ih;
        }
    if (lam_on) {
        // the Lambda trace term enters H_ii: rhs_ii -= J, J = -Lambda/3 sum_{d,s} [Q^s_dd tr(u_d) - sum_l Q^s_dl (u_d)_ld]
        double Jp = 0.0;
#pragma unroll
        for (int d = 0; d < ND; ++d)
#pragma unroll
            for (int s = 0; s < 2; ++s) {
                Jp = fma(Q[d][s][d], U[d][s][0] + U[d][s][4] + U[d][s][8], Jp);
#pragma unroll
                for (int l = 0; l < 3; ++l) Jp = fma(-Q[d][s][l], U[d][s][3 * l + d], Jp);
            }
        const double J = -Lambda / 3.0 * Jp * ih;
        rhs[0] -= J;
        rhs[4] -= J;
        rhs[8] -= J;
    }
    return true;
}

template <typename T>
__device__ __forceinline__ T block_reduce_max(T v, T* red) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) red[warp] = v;
    __syncthreads();
    T r = red[0];
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w) r = fmax(r, red[w]);
    return r;
}

__device__ __forceinline__ double block_reduce_sum(double v, double* red) {
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

__device__ __forceinline__ void applied_load(const InstDev& I, double t, double* add) {
    if (!I.has_load) { add[0] = add[1] = add[2] = 0.0; return; }
    double eps[3];
    for (int i = 0; i < 3; ++i) eps[i] = I.load_init[i] + I.load_rate[i] * (t - I.load_t0);
    double tr = eps[0] + eps[1] + eps[2];
    for (int i = 0; i < 3; ++i) add[i] = I.load_lamb * tr + 2.0 * I.load_mu * eps[i];
}

// Per block constants of one stage: the applied-load stress (FP64) and, for the stage updates,
// dt and whether the instance is still active.
struct StageConst {
    double ld[3];
    double dt;
    double meh;   // ME Dx^2 (FP64)
    bool active;
};

template <int MODE>
__device__ __forceinline__ StageConst stage_const(const InstDev& I, const InstClock& ck, double t_flux) {
    StageConst k;
    // load time: the step-start time in all three stages (FieldMover.py L62, L123, L133); stage 1
    // runs before its last block advances t (step_dt), stages 2 and 3 after it (t_stage holds the start).
    const double tload = (MODE == M_FLUX) ? t_flux : ((MODE == M_STAGE1) ? ck.t : ck.t_stage);
    applied_load(I, tload, k.ld);
    k.dt = ck.dt;
    k.meh = ME * I.h * I.h;
    k.active = ck.active != 0;
    return k;
}

// Per-thread pointers to the current cell (component 0; components are `cells` apart) and the
// instance scalars the cell update needs, formed once per block before the march: the march only
// advances the pointers by one plane, and nothing per cell re-reads the instance table (global
// stores through `out` would otherwise force those reloads).
template <typename T> struct CellCtx {
    const T* sig;   // internal stress (6 components)
    const T* bn;    // beta_n of the stage updates
    T* out;         // rhs (flux, stage 1) or the updated state (stages 2, 3)
    T* spd;         // CFL speed (flux mode, optional)
    long long cells;
    T ih;           // 1 / Dx
    bool has_load, lam_on, glide;
};

// CFL speed maximum of a thread's stage-1 cells; NaN and Inf map to +Inf. (A maximum of floats is exact.)
__device__ __forceinline__ void speed_max(float& m, float s) {
    if (!(s <= 3.402823466e38f)) s = __int_as_float(0x7f800000);
    m = fmaxf(m, s);
}
__device__ __forceinline__ void speed_max(double& m, double s) {
    if (!(s <= 1.0e300)) s = __longlong_as_double(0x7ff0000000000000LL);
    m = fmax(m, s);
}

// ssm: this thread's 6 shared-memory stress slots (component c at ssm[c * ST_THREADS]), filled by
// asynchronous copies issued one cell earlier; sig_next: the stress of the thread's cell in the
// next plane (its copies are issued as soon as this cell's values are read), or null; vmax: the thread's
// speed maximum (stage 1); kc: the block's constants, in shared memory; early() is called once the
// stress slots are free (FP32), ring_read() as in flux_f64 (FP64).
template <typename T, int ND, int MODE, int VAR, class FE, class FR>
__device__ __forceinline__ void stencil_cell(const InstDev& I, const CellCtx<T>& cx, bool valid,
                                             const TileView<T, ND>& tv, const StageConst& kc,
                                             T& vmax,
                                             const T* __restrict__ sig0, const T* __restrict__ vac,
                                             T* ssm, const T* sig_next, const FE& early, const FR& ring_read) {
    // compile-time variant: bit 0 carries the glide-only projection, bit 1 the vacancy term
    constexpr bool GLIDE = (VAR & 1) != 0;
    constexpr bool VAC = (VAR & 2) != 0;
    const T ih = cx.ih;
    const long long cells = cx.cells;
    // beta_n of the stage update is loaded after the flux (no registers to hold it across; FP32
    // requested its rows into L2 one plane ahead)
    constexpr bool UPD = (MODE == M_STAGE2 || MODE == M_STAGE3);
    const double* ld = kc.ld;
    // total stress at the cell: internal + applied load (FP64), symmetric
    T S[3][3];
    {
        T s6[6];
        cp_async_wait_own();
#pragma unroll
        for (int c = 0; c < 6; ++c) s6[c] = ssm[c * st_threads<T>()];
        if (sig_next) {
#pragma unroll
            for (int c = 0; c < 6; ++c) cp_async_elem(ssm + c * st_threads<T>(), sig_next + c * cells);
            cp_async_commit();
        }
        early();
        S[0][0] = (T)((double)s6[0] + ld[0]);
        S[1][1] = (T)((double)s6[3] + ld[1]);
        S[2][2] = (T)((double)s6[5] + ld[2]);
        if (!cx.has_load) { S[0][0] = s6[0]; S[1][1] = s6[3]; S[2][2] = s6[5]; }
        S[0][1] = S[1][0] = s6[1];
        S[0][2] = S[2][0] = s6[2];
        S[1][2] = S[2][1] = s6[4];
        if (VAC && vac && I.vacancy) {   // BetaP_VacancyDynamics.GetSigma (VacancyDynamics.py L23-29): sigma_ii -= alpha c
            // the cell's concentration, addressed on use from the kernel arguments (the stress
            // pointer's offset is the cell index) so that nothing stays live across the march
            const long long cl = cx.sig - (sig0 + I.soff);
            const T ac = (T)I.vac_alpha * vac[I.foff / 9 + cl];
            S[0][0] -= ac;
            S[1][1] -= ac;
            S[2][2] -= ac;
        }
    }
    T rhs[9];
    T spd;
    if constexpr (sizeof(T) == 4) {
        flux_f32<ND, GLIDE>(tv, ih, S, cx.lam_on, GLIDE && cx.glide, (float)I.Lambda, rhs, spd);
    } else {
        if (!flux_f64<ND, GLIDE>(tv, ih, kc.meh, S, cx.lam_on, GLIDE && cx.glide, I.Lambda, rhs, spd, ring_read)) return;
    }

    // ---------------- outputs ----------------
    if (MODE == M_FLUX) {
        if (valid) {
            T* o = cx.out;
#pragma unroll
            for (int c = 0; c < 9; ++c) o[c * cells] = rhs[c];
            if (cx.spd) *cx.spd = spd;
        }
    } else if (MODE == M_STAGE1) {
        if (valid) {
            T* o = cx.out;
#pragma unroll
            for (int c = 0; c < 9; ++c) o[c * cells] = rhs[c];
            speed_max(vmax, spd);
        }
    } else if constexpr (UPD) {
        if (valid && kc.active) {
            const T dt = (T)kc.dt;
            T* o = cx.out;
            T vn[9];
            const T* un = cx.bn;
#pragma unroll
            for (int c = 0; c < 9; ++c) vn[c] = un[c * cells];
#pragma unroll
            for (int c = 0; c < 9; ++c) {
                T vs = tv.center(c);
                T L = dt * rhs[c];
                T r;
                if (MODE == M_STAGE2) r = (T)0.75 * vn[c] + (T)0.25 * vs + (T)0.25 * L;
                else r = (T)(1.0 / 3.0) * vn[c] + (T)(2.0 / 3.0) * vs + (T)(2.0 / 3.0) * L;
                o[c * cells] = r;
            }
        }
    }
}

// Per-instance time step: dt = cfl / (max(shape) * max speed), clamped to t_end (FieldMover.py L94-111), by the
// block of the instance that finishes stage 1 last: every block writes its maximum and counts itself in
// done[ii]. (A kernel of its own took 8 us of a step.) A non-finite maximum (also of a block whose planes did not
// arrive) raises ST_NONFINITE and skips the step. The maximum is exact in any order.
struct DtArgs {
    const int* pre;      // prefix sums of the stencil blocks
    double* bmax;        // per-block speed maxima
    unsigned* done;      // per-instance count of finished blocks (0 between launches)
    int fixed;           // step of dt_fixed
    double dt_fixed;
};
__device__ __noinline__ void step_dt(const InstDev& I, int ii, double m, const DtArgs& a, InstClock* clk, int* status,
                                     double* red) {
    __shared__ int last;
    const int b0 = a.pre[ii], b1 = a.pre[ii + 1];
    if (threadIdx.x == 0) {
        a.bmax[blockIdx.x] = m;
        __threadfence();
        last = atomicAdd(a.done + ii, 1u) == (unsigned)(b1 - b0 - 1);
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    m = 0.0;
#pragma unroll 4
    for (int b = b0 + threadIdx.x; b < b1; b += blockDim.x) m = fmax(m, __ldcg(a.bmax + b));
    m = block_reduce_max(m, red);
    if (threadIdx.x != 0) return;
    InstClock c = clk[ii];
    c.vmax = m;
    c.t_stage = c.t;
    const bool finite = (m <= 1.0e300);
    if (!a.fixed && !finite) atomicOr(status, (int)ST_NONFINITE);
    const bool act = (c.t < c.t_end) && (a.fixed || finite);
    double dt;
    if (a.fixed) dt = a.dt_fixed;
    else dt = act ? I.cfl / (I.nmax * m) : 0.0;
    if (!a.fixed && I.dt_max > 0.0 && dt > I.dt_max) dt = I.dt_max;   // dtBound (FieldMover.py L359-360)
    if (act && c.t + dt > c.t_end) dt = c.t_end - c.t;
    if (!act) dt = 0.0;
    c.dt = dt;
    c.active = act ? 1 : 0;
    if (act) { c.t = c.t + dt; c.steps += 1; }
    clk[ii] = c;
    a.done[ii] = 0;
}

// The plane box of a stencil tile: RX x RY cells from (x0 - OX, y0 - 2) of the instance's field
// (component c at src + c * cells), wrapped periodically.
// Kept in shared memory, like StageConst, so that nothing of it stays in registers across the march.
template <typename T> struct BoxGeomT {
    const T* src;
    long long cells;
    int x0, y0, nX, nY, nZ, zr;   // zr: the grid plane of relative index 0
    int chunk;                    // elements per copy
    __device__ __forceinline__ int plane_of(int pr) const {
        int z = zr + pr;
        while (z < 0) z += nZ;
        while (z >= nZ) z -= nZ;
        return z;
    }
};
// CH consecutive elements global -> shared (4 to 16 bytes), asynchronously.
template <int BYTES> __device__ __forceinline__ void cp_async_chunk(void* dst, const void* src) {
    if constexpr (BYTES == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(smem_addr(dst)), "l"(src) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(smem_addr(dst)), "l"(src), "n"(BYTES) : "memory");
}
// Box of plane zp by asynchronous copies of CH elements, all in flight at once; the block's threads walk
// the box's rows (component, y) with a fixed column each. CH divides nX, x0 and OX, so a chunk never
// crosses the periodic boundary. The caller commits the group.
template <typename T, int CH>
__device__ __forceinline__ void box_async_ch(T* dst, const BoxGeomT<T>& g, int zp) {
    constexpr int RX = TileGeom<T>::RX, OX = TileGeom<T>::OX, RY = tile_ry<T>();
    constexpr int CPR = RX / CH, RS = st_threads<T>() / CPR;   // chunks per row, rows per sweep
    const int r0 = threadIdx.x / CPR, col = (threadIdx.x - r0 * CPR) * CH;
    if (r0 >= RS) return;
    int xx = g.x0 - OX + col;
    while (xx < 0) xx += g.nX;
    while (xx >= g.nX) xx -= g.nX;
    const T* sp = g.src + (long long)zp * g.nY * g.nX + xx;
#pragma unroll 1
    for (int r = r0; r < 9 * RY; r += RS) {
        const int c = r / RY, iy = r - c * RY;
        int yy = g.y0 - 2 + iy;
        while (yy < 0) yy += g.nY;
        while (yy >= g.nY) yy -= g.nY;
        cp_async_chunk<CH * (int)sizeof(T)>(dst + r * RX + col, sp + c * g.cells + yy * g.nX);
    }
}
// The widest chunk that the row length and the field's address allow (grids are even, tiles start at
// multiples of 4 or at nX - 32): 16 bytes, 8 bytes (FP32 rows of 4 k + 2 values), one value.
template <typename T> __device__ __forceinline__ int box_chunk(const T* src, int nX) {
    const uintptr_t a = (uintptr_t)src | (uintptr_t)nX * sizeof(T);
    return (a & 15) == 0 ? 16 / (int)sizeof(T) : ((a & 7) == 0 ? 8 / (int)sizeof(T) : 1);
}
template <typename T>
__device__ __forceinline__ void box_async(T* dst, const BoxGeomT<T>& g, int zp) {
    const int chunk = g.chunk;
    if (chunk == 16 / (int)sizeof(T)) box_async_ch<T, 16 / (int)sizeof(T)>(dst, g, zp);
    else if (sizeof(T) == 4 && chunk == 2) box_async_ch<T, 2>(dst, g, zp);
    else box_async_ch<T, 1>(dst, g, zp);
}

// One block: a TXS x TYS tile of planes [z0, z0 + zc) (3-D) or of the single plane (2-D).
// The 3-D ring holds planes z-2 .. z+2 of all 9 components of beta_s (NS slots). A tile whose box lies
// inside the grid stages a plane by one 5-D bulk-tensor copy from the tensor map of its instance's run of
// same-shape instances (I.tma_slot >= 0); the others, and those without a map, by asynchronous 16-byte (or
// narrower) copies with wrapped addresses (box_async). (A TMA copy of an edge tile would need its
// out-of-grid cells patched once it has landed, by loads whose latency nothing hides: 30% of the FP64 flux
// at 128^3, where half of the tiles are at an edge.)
// FP32 (6 box slots) requests plane z+3 as cell z starts. FP64 (one box, own columns) requests the box of plane
// z+1 and the columns' plane z+3 once the whole block has formed its derivatives, so the copies run under the
// corner and rhs work of the same cell; that barrier also collects the verdict of the bounded waits.
template <typename T, int ND, int MODE, int VAR>
__device__ __forceinline__ void march(const InstDev& I, int ii, int lb, T* sm, double* red, uint64_t* bars,
                                      const StencilMapSet& maps,
                                      const T* bs, const T* bn, T* out,
                                      const T* sig, T* speed_out,
                                      InstClock* clk, double t_flux, const DtArgs& dta,
                                      int* status, const T* vac) {
    constexpr int RX = TileGeom<T>::RX, OX = TileGeom<T>::OX, PP = tile_pp<T>();
    constexpr int TYS = TileGeom<T>::TY, RY = tile_ry<T>(), ST_THREADS = st_threads<T>();
    constexpr bool OWN = own_columns<T, ND>();
    constexpr int NB = (ND == 3 && !OWN) ? TileGeom<T>::NS : 1;      // plane boxes
    constexpr int NS = OWN ? TileGeom<T>::NS : NB;                   // slots of the five planes z-2 .. z+2
    constexpr int SP = OWN ? 9 * ST_THREADS : 9 * PP;                // elements per slot
    constexpr uint32_t PLANE_BYTES = 9u * PP * sizeof(T);
    const int nZ = (ND == 3) ? I.n0 : 1;
    const int nY = (ND == 3) ? I.n1 : I.n0;
    const int nX = (ND == 3) ? I.n2 : I.n1;
    const int tXn = (nX + TXS - 1) / TXS, tYn = (nY + TYS - 1) / TYS;
    int b = lb;
    const int bx = b % tXn; b /= tXn;
    const int by = b % tYn; b /= tYn;
    const int z0 = b * I.st_zc;
    const int z1 = min(z0 + I.st_zc, nZ);
    const int tid = threadIdx.x, tx = tid % TXS, ty = tid / TXS;
    // the tile's own cells start at (x0n, y0n); a last, partial tile is shifted back inside the
    // grid (it recomputes cells of its neighbour without storing them), so that its box leaves the
    // grid by the halo only (x0 stays a multiple of 4 when nX is: the TMA origin x0 - OX is aligned)
    const int x0n = bx * TXS, y0n = by * TYS;
    const int x0 = (x0n + TXS > nX && nX >= TXS) ? nX - TXS : x0n;
    const int y0 = (y0n + TYS > nY && nY >= TYS) ? nY - TYS : y0n;
    const int x = x0 + tx, y = y0 + ty;
    const bool vxy = (x < nX) && (y < nY);
    const bool own = vxy && x >= x0n && y >= y0n;
    const long long cells = I.cells;
    const long long plane = (long long)nY * nX;
    const T* src = bs + I.foff;
    const bool edge = (x0 - OX < 0) || (x0 - OX + RX > nX) || (y0 - 2 < 0) || (y0 - 2 + RY > nY);
    const bool use_tma = maps.enabled && (I.tma_slot >= 0) && !edge;

    __shared__ StageConst kc;   // read per cell from shared memory (keeps registers free)
    __shared__ BoxGeomT<T> bg;
    if (use_tma && tid == 0) {
#pragma unroll 1
        for (int s = 0; s < NB; ++s) mbar_init(&bars[s], 1);
        fence_mbar_init();
    }
    pdl_wait();
    if (tid == 0) {
        kc = stage_const<MODE>(I, clk[ii], t_flux);
        bg = {src, cells, x0, y0, nX, nY, nZ, ND == 3 ? z0 - 2 : 0, box_chunk<T>(src, nX)};
    }
    __syncthreads();
    // Box n: the plane with relative index n (= z - (z0 - 2)), or with own columns the n-th cell's (relative
    // index n + 2); it lives in box slot n % NB.
    constexpr int REL = OWN ? 2 : 0;
    auto issue = [&](int n) {   // TMA, one thread
        const int slot = n % NB;
        mbar_expect_tx(&bars[slot], PLANE_BYTES);
        tma_load_5d(sm + slot * 9 * PP, &maps.m[I.tma_slot], &bars[slot], bg.x0 - OX, bg.y0 - 2,
                    bg.plane_of(n + REL), 0, I.tma_sub);
    };
    auto stage = [&](int n) {   // asynchronous copies, all threads
        box_async<T>(sm + (n % NB) * 9 * PP, bg, bg.plane_of(n + REL));
        cp_async_commit();
    };
    auto landed = [&](int n) { return mbar_wait(&bars[n % NB], (uint32_t)((n / NB) & 1)); };
    // own columns: the thread's nine values of the next plane (relative index 0, 1, ...), to the next slot
    T* column = sm + NB * 9 * PP + tid;
    const T* col_src = nullptr;
    int col_z = 0, col_slot = 0;
    if constexpr (OWN) {
        col_z = bg.plane_of(0);
        col_src = bg.src + (long long)col_z * plane + (vxy ? y * nX + x : 0);
    }
    auto column_async = [&]() {
        T* d = column + col_slot;
#pragma unroll
        for (int c = 0; c < 9; ++c) cp_async_elem(d + c * ST_THREADS, col_src + c * cells);
        cp_async_commit();
        col_slot = (col_slot + SP == NS * SP) ? 0 : col_slot + SP;
        col_src += plane;
        if (++col_z == nZ) {
            col_z = 0;
            col_src -= cells;
        }
    };

    constexpr int NPL = (ND == 3 && !OWN) ? 5 : 1;   // first boxes: planes z0-2 .. z0+2, or the current plane
    int issued = -1;   // last box handed to TMA
    int ok = 1;        // block-uniform: every plane waited for has arrived
    if (use_tma) {
        if (tid == 0)
            for (int n = 0; n < NPL; ++n) issue(n);
        issued = NPL - 1;
    } else {
#pragma unroll 1
        for (int n = 0; n < NPL; ++n) stage(n);
    }
    if constexpr (OWN) {
#pragma unroll 1
        for (int q = 0; q < 5; ++q) column_async();
    }
    T vmax = 0;
    T* ssm = sm + NB * 9 * PP + (OWN ? NS * SP : 0) + tid;
    // this thread's cell in plane z0 (cell (z0, 0, 0) for threads outside the grid: in-bounds
    // loads, no stores)
    CellCtx<T> cx;
    {
        const long long cl0 = vxy ? ((long long)z0 * nY + y) * nX + x : (long long)z0 * plane;
        cx.sig = sig + I.soff + cl0;
        cx.bn = bn ? bn + I.foff + cl0 : nullptr;   // stage updates only
        cx.out = out + I.foff + cl0;
        cx.spd = speed_out ? speed_out + I.coff + cl0 : nullptr;
        cx.cells = cells;
        cx.ih = (T)I.inv_h;
        cx.has_load = I.has_load != 0;
        cx.lam_on = (I.Lambda != 0.0);
        cx.glide = (I.glide != 0);
    }
    TileView<T, ND> tv;
    tv.sm = sm;
    tv.column = column;
    tv.idx = (ty + 2) * RX + tx + OX;
    // the stress of the thread's cell, one plane ahead, in its shared-memory slots after the planes
#pragma unroll
    for (int c = 0; c < 6; ++c) cp_async_elem(ssm + c * ST_THREADS, cx.sig + c * cells);
    cp_async_commit();
    // the first planes: the barrier makes the staged copies visible
    if (!use_tma) cp_async_wait_own();
    __syncthreads();
    bool got = true;   // this thread saw every plane of the coming cell arrive
    if (use_tma) {
#pragma unroll 1
        for (int n = 0; n < NPL; ++n) got &= landed(n);
    }
    // FP32 stage updates read beta_n of their cell after the flux (no registers to hold it across): its rows
    // of the next plane are requested into L2 a plane ahead, one 128-byte row of 32 cells per thread for
    // the first 9 TYS threads of tiles inside the grid
    const bool ahead = nX >= TXS && nY >= TYS && tid < 9 * TYS;
#pragma unroll 1
    for (int z = z0, k = 0; z < z1; ++z, ++k) {
        const bool more = (z + 1 < z1);
        // collects the waits' verdict; every thread has read the planes it needs
        auto verdict = [&]() {
            if (__syncthreads_or(!got)) {
                ok = 0;
                if (tid == 0) atomicOr(status, (int)ST_TIMEOUT);
            }
            return ok != 0;
        };
        const int next = OWN ? k + 1 : k + 5;   // box to request
        auto request = [&]() {
            if (use_tma) {
                if (tid == 0) {
                    fence_proxy_async();
                    issue(next);
                }
                issued = next;
            } else {
                stage(next);
            }
        };
        if (!OWN && use_tma && !verdict()) break;
        if (ND == 3 && !OWN && use_tma && more) request();
        if (ND == 3) {
            // ring planes z-2 .. z+2 live in slots (k + q) mod NS, rotated by one plane per step
            if (k == 0) {
#pragma unroll
                for (int q = 0; q < 5; ++q) tv.so[q] = q * SP;
            } else {
#pragma unroll
                for (int q = 0; q < 4; ++q) tv.so[q] = tv.so[q + 1];
                tv.so[4] = (tv.so[3] + SP == NS * SP) ? 0 : tv.so[3] + SP;
            }
        } else {
            tv.so[2] = 0;
        }
        if constexpr (sizeof(T) == 4 && (MODE == M_STAGE2 || MODE == M_STAGE3)) {
            if (ahead && more) {
                const int c = tid / TYS, r = tid - c * TYS;
                prefetch_l2(cx.bn + c * cells + plane + (long long)(r - ty) * nX - tx);
            }
        }
        auto early = [&]() {   // FP32: the staged copies of plane k + 5, after the stress copies' wait
            if (ND == 3 && !OWN && !use_tma && more) stage(next);
        };
        auto ring_read = [&]() {   // FP64
            if (!OWN) return true;
            if (more) column_async();   // plane z + 3, into the slot of z - 2 that this thread has read
            if (use_tma) {
                if (!verdict()) return false;
            } else if (more) {
                __syncthreads();
            }
            if (more) request();
            return true;
        };
        stencil_cell<T, ND, MODE, VAR>(I, cx, own, tv, kc, vmax, sig, vac, ssm,
                                       more ? cx.sig + plane : nullptr, early, ring_read);
        if (!ok) break;
        cx.sig += plane;
        if (cx.bn) cx.bn += plane;
        cx.out += plane;
        if (cx.spd) cx.spd += plane;
        if (ND == 3 && more) {
            if (use_tma) {
                got = landed(next);
            } else {
                cp_async_wait_own();
                __syncthreads();
            }
        }
    }
    cp_async_wait_own();   // no copy in flight past here
    // a copy did not land in time: let every copy this block issued finish (bounded)
    if (!ok)
        for (int n = max(0, issued - NB + 1); n <= issued; ++n) landed(n);
    if (MODE == M_STAGE1) {
        const double m = ok ? block_reduce_max((double)vmax, red) : __longlong_as_double(0x7ff0000000000000LL);
        step_dt(I, ii, m, dta, clk, status, red);
    }
}

template <typename T, int MODE, int VAR>
__global__ void __launch_bounds__(st_threads<T>(), ST_BLOCKS)
k_stencil(const InstDev* __restrict__ insts, int n_inst, const int* __restrict__ pre,
          const T* bs, const T* bn, T* out, const T* sig,
          T* speed_out, InstClock* clk, double t_flux, const DtArgs dta, int* status,
          const T* vac, const __grid_constant__ StencilMapSet maps) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    T* sm = reinterpret_cast<T*>(smem_raw);
    __shared__ double red[st_threads<T>() / 32];
    __shared__ __align__(8) uint64_t bars[6];
    const int ii = find_instance(pre, n_inst, blockIdx.x);
    const InstDev& I = insts[ii];
    const int lb = blockIdx.x - pre[ii];
    if (I.nd == 3)
        march<T, 3, MODE, VAR>(I, ii, lb, sm, red, bars, maps, bs, bn, out, sig, speed_out, clk, t_flux, dta, status,
                          vac);
    else
        march<T, 2, MODE, VAR>(I, ii, lb, sm, red, bars, maps, bs, bn, out, sig, speed_out, clk, t_flux, dta, status,
                          vac);
}

// F0 = u + dt * rhs, in place on the rhs buffer, for active instances (one fused multiply-add per
// value). Instances with the fused plane passes form F0 in their forward pass instead.
template <typename T>
__global__ void __launch_bounds__(256) k_axpy_f0(const InstDev* __restrict__ insts, int n_inst,
                                                 const int* __restrict__ pre, const T* u,
                                                 T* f0, const InstClock* clk) {
    const int ii = find_instance(pre, n_inst, blockIdx.x);
    const InstDev& I = insts[ii];
    pdl_wait();
    if (!clk[ii].active || I.plane) return;
    const T dt = (T)clk[ii].dt;
    const long long n = 9 * I.cells;
    const long long b0 = (long long)(blockIdx.x - pre[ii]) * blockDim.x * 4;   // 4 elements per thread
    const T* uu = u + I.foff;
    T* ff = f0 + I.foff;
    if (blockDim.x == 256 && b0 + 1024 <= n && ((((uintptr_t)uu) | ((uintptr_t)ff)) & 15) == 0) {
        // 16-byte vectors: one float4 (FP32) or two double2 (FP64) per thread
        if constexpr (sizeof(T) == 4) {
            const long long i = b0 + 4 * threadIdx.x;
            const float4 a = *reinterpret_cast<const float4*>(uu + i);
            float4 r = *reinterpret_cast<const float4*>(ff + i);
            r.x = __fmaf_rn(dt, r.x, a.x);
            r.y = __fmaf_rn(dt, r.y, a.y);
            r.z = __fmaf_rn(dt, r.z, a.z);
            r.w = __fmaf_rn(dt, r.w, a.w);
            *reinterpret_cast<float4*>(ff + i) = r;
        } else {
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const long long i = b0 + 512 * k + 2 * threadIdx.x;
                const double2 a = *reinterpret_cast<const double2*>(uu + i);
                double2 r = *reinterpret_cast<const double2*>(ff + i);
                r.x = __fma_rn(dt, r.x, a.x);
                r.y = __fma_rn(dt, r.y, a.y);
                *reinterpret_cast<double2*>(ff + i) = r;
            }
        }
        return;
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        long long i = b0 + threadIdx.x + (long long)k * blockDim.x;
        if (i < n) ff[i] = fma(dt, ff[i], uu[i]);
    }
}

// Vacancy coupling, one thread per cell of the vacancy instances (OperatorSplittingTVDRK_FieldMover,
// FieldMover.py L339-380): tr(beta^P) at the step start (prevTrBetaP), and after the step
// c += vac_beta (TrBetaP - prevTrBetaP) for the instances whose step was applied; traces summed
// xx + yy, then zz, as the reference does.
template <typename T>
__global__ void __launch_bounds__(256) k_vac_trace(const InstDev* __restrict__ insts, int n_inst,
                                                   const int* __restrict__ pre, const T* beta,
                                                   T* tr) {
    const int ii = find_instance(pre, n_inst, blockIdx.x);
    const InstDev& I = insts[ii];
    pdl_wait();
    if (!I.vacancy) return;
    const long long cell = (long long)(blockIdx.x - pre[ii]) * blockDim.x + threadIdx.x;
    if (cell >= I.cells) return;
    const T* b = beta + I.foff + cell;
    tr[I.foff / 9 + cell] = (b[0] + b[4 * I.cells]) + b[8 * I.cells];
}

template <typename T>
__global__ void __launch_bounds__(256) k_vac_update(const InstDev* __restrict__ insts, int n_inst,
                                                    const int* __restrict__ pre, const T* beta,
                                                    const T* tr, T* c,
                                                    const InstClock* clk) {
    const int ii = find_instance(pre, n_inst, blockIdx.x);
    const InstDev& I = insts[ii];
    pdl_wait();
    if (!I.vacancy || !clk[ii].active) return;
    const long long cell = (long long)(blockIdx.x - pre[ii]) * blockDim.x + threadIdx.x;
    if (cell >= I.cells) return;
    const T* b = beta + I.foff + cell;
    const T trn = (b[0] + b[4 * I.cells]) + b[8 * I.cells];
    T& cv = c[I.foff / 9 + cell];
    cv = cv + (T)I.vac_beta * (trn - tr[I.foff / 9 + cell]);
}

// Energy and mean b_zz partials of a state whose internal stress is in sig (observables).
template <typename T>
__global__ void __launch_bounds__(256) k_observe(const InstDev* __restrict__ insts, int n_inst,
                                                        const int* __restrict__ pre,
                                                        const T* beta,
                                                        const T* sig,
                                                        double* bsum) {
    __shared__ double red[8];
    const int ii = find_instance(pre, n_inst, blockIdx.x);
    const InstDev& I = insts[ii];
    const long long cell = (long long)(blockIdx.x - pre[ii]) * blockDim.x + threadIdx.x;
    pdl_wait();
    double e = 0.0, z = 0.0;
    if (cell < I.cells) {
        const T* sp = sig + I.soff + cell;
        const long long cells = I.cells;
        double s0 = (double)sp[0], s1 = (double)sp[cells], s2 = (double)sp[2 * cells];
        double s3 = (double)sp[3 * cells], s4 = (double)sp[4 * cells], s5 = (double)sp[5 * cells];
        double sq = s0 * s0 + s3 * s3 + s5 * s5 + 2.0 * (s1 * s1 + s2 * s2 + s4 * s4);
        double tr = s0 + s3 + s5;
        e = (sq - I.nu / (1.0 + I.nu) * tr * tr) / (4.0 * I.mu);
        z = (double)beta[I.foff + 8 * cells + cell];
    }
    double es = block_reduce_sum(e, red);
    double zs = block_reduce_sum(z, red);
    if (threadIdx.x == 0) { bsum[2 * blockIdx.x] = es; bsum[2 * blockIdx.x + 1] = zs; }
}

__global__ void __launch_bounds__(256) k_obs_reduce(const InstDev* __restrict__ insts,
                                                    const int* __restrict__ pre,
                                                    const double* bsum,
                                                    double* obs) {
    __shared__ double red[8];
    const int ii = blockIdx.x;
    pdl_wait();
    double es = 0.0, zs = 0.0;
#pragma unroll 8
    for (int b = pre[ii] + threadIdx.x; b < pre[ii + 1]; b += blockDim.x) {
        es += bsum[2 * b];
        zs += bsum[2 * b + 1];
    }
    es = block_reduce_sum(es, red);
    zs = block_reduce_sum(zs, red);
    if (threadIdx.x == 0) {
        obs[2 * ii] = es;
        obs[2 * ii + 1] = zs * insts[ii].inv_cells;
    }
}

// ------------------------------------------------------------------------------------------
template <typename T>
static void stencil_dispatch(const PlanCore& P, int mode, const void* bs, const void* bn, void* out,
                             void* speed, double t, const StencilMapSet& maps, cudaStream_t st, int fixed, double dt_fixed) {
    const LaunchShape& L = P.stencil;
    const DtArgs dta{L.d_pre, P.d_bmax, P.d_done, fixed, dt_fixed};
    const T* b = (const T*)bs;
    const T* n = (const T*)bn;
    T* o = (T*)out;
    const T* s = (const T*)P.d_sigma;
    // the variant carries the glide-only projection (bit 0) and the vacancy term (bit 1) only when
    // the plan has such instances
    const int var = (P.any_glide ? 1 : 0) | (P.any_vac ? 2 : 0);
#define CDD_LAUNCH_V(M, V, SP)                                                                           \
    launch_pdl(k_stencil<T, M, V>, L.blocks, st_threads<T>(), L.smem, st, P.d_inst, P.n_inst, L.d_pre, b, n, o, s, SP,     \
                                                             P.d_clock, t, dta, P.d_status,    \
                                                             (const T*)P.d_vac, maps)
#define CDD_LAUNCH_ST(M, SP)                                  \
    switch (var) {                                            \
        case 0: CDD_LAUNCH_V(M, 0, SP); break;                \
        case 1: CDD_LAUNCH_V(M, 1, SP); break;                \
        case 2: CDD_LAUNCH_V(M, 2, SP); break;                \
        default: CDD_LAUNCH_V(M, 3, SP); break;               \
    }
    switch (mode) {
        case M_FLUX: CDD_LAUNCH_ST(M_FLUX, (T*)speed); break;
        case M_STAGE1: CDD_LAUNCH_ST(M_STAGE1, nullptr); break;
        case M_STAGE2: CDD_LAUNCH_ST(M_STAGE2, nullptr); break;
        default: CDD_LAUNCH_ST(M_STAGE3, nullptr); break;
    }
#undef CDD_LAUNCH_V
#undef CDD_LAUNCH_ST
}

template <typename T>
static cudaError_t vac_pre_t(const PlanCore& P, const void* beta, cudaStream_t st) {
    const LaunchShape& L = P.obs;
    launch_pdl(k_vac_trace<T>, L.blocks, L.threads, 0, st, P.d_inst, P.n_inst, L.d_pre, (const T*)beta, (T*)P.d_vtr);
    return cudaGetLastError();
}

cudaError_t launch_vacancy_pre(const PlanCore& P, const void* beta, cudaStream_t st) {
    return P.precision == CDD_F32 ? vac_pre_t<float>(P, beta, st) : vac_pre_t<double>(P, beta, st);
}

template <typename T>
static cudaError_t vac_post_t(const PlanCore& P, const void* beta, cudaStream_t st) {
    const LaunchShape& L = P.obs;
    launch_pdl(k_vac_update<T>, L.blocks, L.threads, 0, st, P.d_inst, P.n_inst, L.d_pre, (const T*)beta,
                                                    (const T*)P.d_vtr, (T*)P.d_vac, P.d_clock);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    return launch_vacancy_diffusion(P, st);
}

cudaError_t launch_vacancy_post(const PlanCore& P, const void* beta, cudaStream_t st) {
    return P.precision == CDD_F32 ? vac_post_t<float>(P, beta, st) : vac_post_t<double>(P, beta, st);
}

cudaError_t launch_stencil(const PlanCore& P, int mode, const void* bs, const void* bn, void* out,
                           void* speed, double t_flux, const StencilMapSet& maps, cudaStream_t st, int fixed,
                           double dt_fixed) {
    if (P.precision == CDD_F32) stencil_dispatch<float>(P, mode, bs, bn, out, speed, t_flux, maps, st, fixed, dt_fixed);
    else stencil_dispatch<double>(P, mode, bs, bn, out, speed, t_flux, maps, st, fixed, dt_fixed);
    return cudaGetLastError();
}

bool stencil_tma_eligible(const InstDev& I, int precision) {
    const int RX = precision == CDD_F32 ? TileGeom<float>::RX : TileGeom<double>::RX;
    const int RY = precision == CDD_F32 ? tile_ry<float>() : tile_ry<double>();
    const int nX = (I.nd == 3) ? I.n2 : I.n1, nY = (I.nd == 3) ? I.n1 : I.n0;
    if (nX < RX || nY < RY) return false;
    if (precision == CDD_F32 && nX % 4) return false;   // 16-byte row strides
    if (precision != CDD_F32 && nX % 2) return false;
    return true;
}

static PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    static bool tried = false;
    if (!tried) {
        tried = true;
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (PFN_cuTensorMapEncodeTiled_v12000)p;
    }
    return fn;
}

// 5-D map per run of consecutive same-shape instances: (x = last axis, y, z = axis 0 (3-D), component,
// instance of the run); box = one staged plane of all 9 components of one instance, RX x RY cells;
// no copy leaves the grid (tiles whose box does are staged by the threads: march).
bool encode_stencil_maps(const PlanCore& P, const InstDev* insts, const void* base, StencilMapSet& maps) {
    maps.enabled = 0;
    PFN_cuTensorMapEncodeTiled_v12000 enc = tensor_map_encoder();
    if (!enc || !base) return false;
    const bool f32 = (P.precision == CDD_F32);
    const size_t elt = f32 ? sizeof(float) : sizeof(double);
    const cuuint32_t RX = f32 ? TileGeom<float>::RX : TileGeom<double>::RX;
    const cuuint32_t RY = f32 ? tile_ry<float>() : tile_ry<double>();
    bool any = false;
    for (int i = 0; i < P.n_inst; ++i) {
        const InstDev& I = insts[i];
        if (I.tma_slot < 0 || I.tma_sub != 0) continue;
        int run = 1;
        while (i + run < P.n_inst && insts[i + run].tma_slot == I.tma_slot) ++run;
        const char* addr = (const char*)base + (size_t)I.foff * elt;
        if (((uintptr_t)addr) % 16) return false;
        // 2-D: (x = axis 1, y = axis 0, z of size 1)
        const cuuint64_t nX = (I.nd == 3) ? I.n2 : I.n1, nY = (I.nd == 3) ? I.n1 : I.n0;
        const cuuint64_t nZ = (I.nd == 3) ? I.n0 : 1;
        cuuint64_t dims[5] = {nX, nY, nZ, 9, (cuuint64_t)run};
        cuuint64_t strides[4] = {nX * elt, nX * nY * elt, (cuuint64_t)I.cells * elt, (cuuint64_t)9 * I.cells * elt};
        cuuint32_t box[5] = {RX, (cuuint32_t)RY, 1, 9, 1};
        cuuint32_t estr[5] = {1, 1, 1, 1, 1};
        CUresult r = enc(&maps.m[I.tma_slot], f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_FLOAT64,
                         5, (void*)addr, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                         CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS) return false;
        any = true;
    }
    maps.enabled = any ? 1 : 0;
    return any;
}

// Start every instance's clock at t with no end time (fixed-dt steps at a caller-given time).
__global__ void k_set_clock(InstClock* clk, int n_inst, double t) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    pdl_wait();
    if (i < n_inst) {
        clk[i].t = t;
        clk[i].t_end = 1.0e300;
    }
}

cudaError_t launch_set_clock(const PlanCore& P, double t, cudaStream_t st) {
    launch_pdl(k_set_clock, (P.n_inst + 127) / 128, 128, 0, st, P.d_clock, P.n_inst, t);
    return cudaGetLastError();
}

cudaError_t launch_axpy_f0(const PlanCore& P, const void* u, void* rhs_f0, cudaStream_t st) {
    const LaunchShape& L = P.cellwise;
    if (P.precision == CDD_F32)
        launch_pdl(k_axpy_f0<float>, L.blocks, 256, 0, st, P.d_inst, P.n_inst, L.d_pre, (const float*)u,
                                                   (float*)rhs_f0, P.d_clock);
    else
        launch_pdl(k_axpy_f0<double>, L.blocks, 256, 0, st, P.d_inst, P.n_inst, L.d_pre, (const double*)u,
                                                    (double*)rhs_f0, P.d_clock);
    return cudaGetLastError();
}

cudaError_t launch_observe(const PlanCore& P, const void* beta, cudaStream_t st) {
    const LaunchShape& L = P.obs;
    if (P.precision == CDD_F32)
        launch_pdl(k_observe<float>, L.blocks, 256, 0, st, P.d_inst, P.n_inst, L.d_pre, (const float*)beta,
                                                         (const float*)P.d_sigma, P.d_bsum);
    else
        launch_pdl(k_observe<double>, L.blocks, 256, 0, st, P.d_inst, P.n_inst, L.d_pre, (const double*)beta,
                                                          (const double*)P.d_sigma, P.d_bsum);
    launch_pdl(k_obs_reduce, P.n_inst, 256, 0, st, P.d_inst, P.obs.d_pre, P.d_bsum, P.d_obs);
    return cudaGetLastError();
}

template <typename T>
static cudaError_t st_attr(size_t smem) {
    cudaError_t e;
#define CDD_ATTR_V(V)                                                                   \
    if ((e = set_dyn_smem_limit(k_stencil<T, M_FLUX, V>, smem))) return e;              \
    if ((e = set_dyn_smem_limit(k_stencil<T, M_STAGE1, V>, smem))) return e;            \
    if ((e = set_dyn_smem_limit(k_stencil<T, M_STAGE2, V>, smem))) return e;            \
    if ((e = set_dyn_smem_limit(k_stencil<T, M_STAGE3, V>, smem))) return e;
    CDD_ATTR_V(0)
    CDD_ATTR_V(1)
    CDD_ATTR_V(2)
    CDD_ATTR_V(3)
#undef CDD_ATTR_V
    return cudaSuccess;
}

cudaError_t stencil_set_attributes(int precision, size_t smem) {
    return precision == CDD_F32 ? st_attr<float>(smem) : st_attr<double>(smem);
}

// The plane boxes and columns plus the 6 stress slots of every thread.
size_t stencil_smem_bytes(int precision, bool any3d) {
    if (precision == CDD_F32)
        return ((size_t)(any3d ? TileGeom<float>::NS : 1) * 9 * tile_pp<float>() + 6 * st_threads<float>()) * sizeof(float);
    return ((size_t)9 * tile_pp<double>() + ((any3d ? TileGeom<double>::NS * 9 : 0) + 6) * st_threads<double>()) * sizeof(double);
}

static int stencil_tiles(const InstDev& I, int precision) {
    const int nY = (I.nd == 3) ? I.n1 : I.n0;
    const int nX = (I.nd == 3) ? I.n2 : I.n1;
    const int TYS = precision == CDD_F32 ? TileGeom<float>::TY : TileGeom<double>::TY;
    return ((nX + TXS - 1) / TXS) * ((nY + TYS - 1) / TYS);
}

// Planes per block (one value for all 3-D instances of a plan). A block costs its planes and about c0 planes'
// time for its start (flux form at 256^3, planes per block 1 / 2 / 4 / 8 / 24: FP64 2565 / 2107 / 1837 / 1712 /
// 1649 us, FP32 1589 / 1180 / 982 / 894 / 851 us); two blocks per SM run at once, and a block alone on its SM takes
// about 0.7 of the time (128 blocks of 4, 8 and 16 planes against 256: FP32 0.72, 0.68, 0.65, FP64 0.83, 0.82,
// 0.81). Many short blocks pay c0 often, few long ones leave SMs idle (small grids) or a tail (a share of a block,
// chosen with c0, not measured by itself): the estimate is minimised. At least 8 planes per block whatever the grid,
// the rule before, gave one 32^3 FP64 flux 32 blocks and 50 us, against 25 us at one plane per block.
int stencil_default_planes(const InstDev* insts, int n, int precision, int sms) {
    const double c0 = precision == CDD_F32 ? 0.9 : 0.55, tail = precision == CDD_F32 ? 0.2 : 0.4;
    const int resident = ST_BLOCKS * sms;
    int best = 1;
    double best_cost = 1e300;
    for (int z = 1; z <= 64; ++z) {
        double sum = 0.0, longest = 0.0, blocks = 0.0;
        for (int i = 0; i < n; ++i) {
            const int nZ = (insts[i].nd == 3) ? insts[i].n0 : 1, len = (nZ + (nZ + z - 1) / z - 1) / ((nZ + z - 1) / z);
            const double b = (double)stencil_tiles(insts[i], precision) * ((nZ + len - 1) / len);
            blocks += b;
            sum += b * c0 + (double)stencil_tiles(insts[i], precision) * nZ;
            if (len + c0 > longest) longest = len + c0;
        }
        const double cost = blocks <= sms ? 0.7 * longest : (blocks <= resident ? longest : sum / resident + tail * longest);
        if (cost <= best_cost) { best_cost = cost; best = z; }
    }
    return best;
}

// Blocks of the stencil: (x, y) tiles times chunks of `planes` planes along axis 0.
void stencil_geometry(InstDev& I, int precision, int planes) {
    const int nZ = (I.nd == 3) ? I.n0 : 1;
    int chunks = 1;
    if (I.nd == 3) {
        chunks = (nZ + planes - 1) / planes;
        if (chunks > nZ) chunks = nZ;
        if (chunks < 1) chunks = 1;
    }
    I.st_zc = (nZ + chunks - 1) / chunks;
    chunks = (nZ + I.st_zc - 1) / I.st_zc;
    I.stencil_blocks = stencil_tiles(I, precision) * chunks;
}

}  // namespace cdd
