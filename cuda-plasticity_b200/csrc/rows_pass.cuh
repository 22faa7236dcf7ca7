// Row passes of the stress pipeline: the transforms along the contiguous axis, device code shared by the R2C
// and C2R kernels (r2c.cu, c2r.cu) and the fused plane passes (stress.cu).
#pragma once
#include "cdd_internal.cuh"

namespace cdd {

constexpr int ROW_THREADS = 256;

__host__ __device__ inline int rows_ld(int n) { return n + (n >> 4) + 1; }

// Four consecutive reals: one 16-byte access for float, two for double (16-byte aligned).
__device__ __forceinline__ void load4(const float* p, float* v) {
    float4 q = *reinterpret_cast<const float4*>(p);
    v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
}
__device__ __forceinline__ void load4(const double* p, double* v) {
    double2 a = reinterpret_cast<const double2*>(p)[0], b = reinterpret_cast<const double2*>(p)[1];
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}
__device__ __forceinline__ void store4(float* p, const float* v) {
    *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
}
__device__ __forceinline__ void store4(double* p, const double* v) {
    reinterpret_cast<double2*>(p)[0] = make_double2(v[0], v[1]);
    reinterpret_cast<double2*>(p)[1] = make_double2(v[2], v[3]);
}

// Symmetric component o = (SYM_I[o], SYM_J[o]): xx xy xz yy yz zz.
static __device__ __constant__ int SYM_I[6] = {0, 0, 0, 1, 1, 2};
static __device__ __constant__ int SYM_J[6] = {0, 1, 2, 1, 2, 2};

// Mean stress -lam tr<s> d_ij - 2 mu <s>_ij of symmetric component o, from the means m of the six
// components of s = sym(beta) (= -lam tr<b> d - mu (<b> + <b>^T)).
__device__ __forceinline__ double mean_stress(const InstDev& I, const double* m, int o) {
    double v = -2.0 * I.mu * m[o];
    if (o == 0 || o == 3 || o == 5) v -= I.lamb * (m[0] + m[3] + m[5]);
    return v;
}

// The stress depends on beta only through its symmetric part s = (beta + beta^T) / 2 (every term of
// the Green contraction and of sigma is symmetric in beta), so the transforms carry 6 components.
// Source rows of the R2C input, row ra = component o * rows + r:
//   RS_STRESS: row ra of a 6-component stress-layout array (p == q);
//   RS_SYM:    rows of beta_ij and beta_ji (p == q on the diagonal), 6 components;
//   RS_FULL:   row ra of a 9-component field (p == q), all 9 components.
// The value is (p + q) / 2, exact when p == q.
//   RS_VAC:    row ra of the vacancy concentrations (one component; vacancy instances only).
enum RowSource { RS_STRESS = 1, RS_SYM = 2, RS_FULL = 3, RS_VAC = 4 };

template <typename T>
__device__ __forceinline__ void src_rows(const InstDev& I, const T* base, int mode, long long ra, const T*& p,
                                         const T*& q) {
    if (mode == RS_STRESS) {
        p = q = base + I.soff + ra * I.nl;
        return;
    }
    if (mode == RS_FULL) {
        p = q = base + I.foff + ra * I.nl;
        return;
    }
    if (mode == RS_VAC) {
        p = q = base + I.foff / 9 + ra * I.nl;
        return;
    }
    const int o = fdiv_q(I.fd_rows, (int)ra);
    const long long r = ra - (long long)o * I.rows;
    const int i = SYM_I[o], j = SYM_J[o];
    p = base + I.foff + (long long)(3 * i + j) * I.cells + r * I.nl;
    q = base + I.foff + (long long)(3 * j + i) * I.cells + r * I.nl;
}

// ------------------------------------------------------------------------------------------
// Row passes of two-stage FFT plans (length N = R0 R1) with the first and the last stage in
// registers: the first stage's butterflies read their inputs straight from the rows, and the last
// stage's outputs go straight to the rows, so a tile passes through shared memory once, between
// the stages. R2C: the last stage's butterfly j of a line (R0 of them, consecutive lanes of one
// warp) holds X[j + R0 r]; the partner X[N - k] of k = j + R0 r sits in lane R0 - j at register
// R1 - 1 - r (in its own register R1 - r for j = 0), so one shuffle per r brings it, and the two
// half spectra of the line's rows are formed and stored from registers. The FP64 row sums of the
// FP32 form are summed from the first stage's inputs and reduced over the line's R1 lanes.
// Requires R0 dividing 32, R1 a power of two <= 32 and both stages' butterfly counts multiples of
// 32 (the block size is too): each warp takes part in a loop trip whole, as the shuffles need
// (rows_io_plan).
// ------------------------------------------------------------------------------------------
// The half spectra of pair p's two rows go to dst + 2 (p - p0) dld and one row (dld) further:
// the plan's spectrum (p0 = 0, dld = nhp) or a block's shared tile (the plane passes).
// F0 (the second RK3 stage's stress): the rows are formed as F0 = u + dt rhs from the rows of u and
// of rhs (held in f0w, the buffer rt points into) and written back over rhs, so the stage input is
// made in the same sweep that transforms it.
template <typename T> __device__ __forceinline__ T fma_t(T a, T b, T c);
template <> __device__ __forceinline__ float fma_t<float>(float a, float b, float c) { return __fmaf_rn(a, b, c); }
template <> __device__ __forceinline__ double fma_t<double>(double a, double b, double c) { return __fma_rn(a, b, c); }

template <typename T, bool F0>
__device__ __forceinline__ T row_value(const T* __restrict__ beta, T* f0w, const T* __restrict__ u, T dt,
                                       const RowPtr& e, int i) {
    if constexpr (F0) {
        const T xp = fma_t(dt, f0w[e.p + i], u[e.p + i]);
        f0w[e.p + i] = xp;
        T xq = xp;
        if (e.q != e.p) {
            xq = fma_t(dt, f0w[e.q + i], u[e.q + i]);
            f0w[e.q + i] = xq;
        }
        return (T)0.5 * (xp + xq);
    } else {
        return (T)0.5 * (beta[e.p + i] + beta[e.q + i]);
    }
}

// Where the row pass puts the two half spectra a (row 2q) and b (row 2q + 1) at bin k of the q-th
// line pair of the block (q = p - p0): rows of dst, dld apart.
template <typename V> struct RowSink {
    V* dst;
    int dld;
    __device__ __forceinline__ void operator()(long long q, int k, const V& a, const V& b, bool hasb) const {
        V* da = dst + 2 * q * dld;
        da[k] = a;
        if (hasb) da[dld + k] = b;
    }
};

template <typename T, bool MEAN64, int R0, int R1, bool F0, class Sink>
__device__ __forceinline__ void r2c_rows_io(const InstDev& I, int lb, int P, int ld, const RowPtr* __restrict__ rt,
                                            const T* __restrict__ beta, typename VecOf<T>::type* s,
                                            const typename VecOf<T>::type* __restrict__ tw1,
                                            const Sink& out, double* __restrict__ rowsum,
                                            long long nrows, long long npairs, int tid, int nt,
                                            long long p0, T* f0w = nullptr, const T* u = nullptr, T dt = 0) {
    typedef typename VecOf<T>::type V;
    // stage 0 (span 1): butterfly (l, j) takes elements j + R1 r of pair line l
#pragma unroll 1
    for (int g = tid; g < P * R1; g += nt) {
        const int l = g / R1, j = g - l * R1;
        const RowPtr ea = rt[2 * l], eb = rt[2 * l + 1];
        V v[R0];
        double sa = 0.0, sb = 0.0;
        // rows that are their own partners (diagonal components, stress rows) are read once: 0.5 (x + x) = x
        if (!F0 && ea.q == ea.p && eb.q == eb.p) {
#pragma unroll
            for (int r = 0; r < R0; ++r) {
                const int i = j + R1 * r;
                v[r].x = ea.p >= 0 ? beta[ea.p + i] : (T)0;
                v[r].y = eb.p >= 0 ? beta[eb.p + i] : (T)0;
            }
        } else {
#pragma unroll
            for (int r = 0; r < R0; ++r) {
                const int i = j + R1 * r;
                T a = 0, b = 0;
                if (ea.p >= 0) a = row_value<T, F0>(beta, f0w, u, dt, ea, i);
                if (eb.p >= 0) b = row_value<T, F0>(beta, f0w, u, dt, eb, i);
                v[r].x = a;
                v[r].y = b;
            }
        }
        if (MEAN64) {
#pragma unroll
            for (int r = 0; r < R0; ++r) { sa += (double)v[r].x; sb += (double)v[r].y; }
        }
        if (MEAN64) {
#pragma unroll
            for (int o = R1 / 2; o > 0; o >>= 1) {
                sa += __shfl_xor_sync(0xffffffffu, sa, o);
                sb += __shfl_xor_sync(0xffffffffu, sb, o);
            }
            const long long row = 2LL * ((long long)lb * P + l);
            if (j == 0 && row < nrows) rowsum[I.rsoff + row] = sa;
            if (j == 0 && row + 1 < nrows) rowsum[I.rsoff + row + 1] = sb;
        }
        dft<R0, V, false>(v);
        V* d = s + l * ld + row_pad(j * R0);   // outputs j R0 + r: inside one 16-element pad period
#pragma unroll
        for (int r = 0; r < R0; ++r) d[r] = v[r];
    }
    __syncthreads();
    // stage 1 (span R0): butterfly (l, j) takes elements j + R0 r, twiddle row j; outputs X[j + R0 r]
    const int nh = I.nh;
#pragma unroll 1
    for (int g = tid; g < P * R0; g += nt) {
        const int l = g / R0, j = g - l * R0;
        V w[R1], v[R1];
        load_tw_row<R1>(tw1 + j * tw_pitch(R1, sizeof(V)), w);
        const V* sl = s + l * ld + row_pad(j);
#pragma unroll
        for (int r = 0; r < R1; ++r) {
            const V x = sl[r * R0 + ((r * R0) >> 4)];
            v[r] = (r == 0) ? x : vmul(x, w[r]);
        }
        dft<R1, V, false>(v);
        const int lane = tid & 31;
        const int partner = lane - j + (R0 - j) % R0;
        const long long p = (long long)lb * P + l;
        const bool valid = p < npairs;
        const bool hasb = 2 * p + 1 < nrows;
#pragma unroll
        for (int r = 0; r < R1; ++r) {
            V zs;
            zs.x = __shfl_sync(0xffffffffu, v[R1 - 1 - r].x, partner);
            zs.y = __shfl_sync(0xffffffffu, v[R1 - 1 - r].y, partner);
            const V zm = (j == 0) ? v[(R1 - r) % R1] : zs;
            const V zk = v[r];
            const int k = j + R0 * r;
            if (valid && k < nh) {
                V a, b;
                a.x = (T)0.5 * (zk.x + zm.x);
                a.y = (T)0.5 * (zk.y - zm.y);
                b.x = (T)0.5 * (zk.y + zm.y);
                b.y = (T)-0.5 * (zk.x - zm.x);
                out(p - p0, k, a, b, hasb);
            }
        }
    }
}

// The same for the other two-pass plans (see pass_stages): pass A straight from the rows to the line buffer
// (group j of A values at j (A + 1)), pass B in place, then the half spectra from the buffer. `lines` is the
// number of groups (pass A) or group elements (pass B) per line.
template <typename T, bool MEAN64, int... Rs>
__device__ __forceinline__ void r2c_pass_a(const LinePlan& lp, int P, const RowPtr* __restrict__ rt, const T* __restrict__ beta,
                                           typename VecOf<T>::type* s, double* part,
                                           const typename VecOf<T>::type* __restrict__ tws, int tid, int nt) {
    typedef typename VecOf<T>::type V;
    constexpr int A = RadixProd<Rs...>::v;
    const int B = lp.B;
#pragma unroll 1
    for (int g = tid; g < P * B; g += nt) {
        const int l = g / B, j = g - l * B;
        const RowPtr ea = rt[2 * l], eb = rt[2 * l + 1];
        V v[A];
        double sa = 0.0, sb = 0.0;
        if (ea.q == ea.p && eb.q == eb.p) {
#pragma unroll
            for (int q = 0; q < A; ++q) {
                const int i = j + B * q;
                v[q].x = ea.p >= 0 ? beta[ea.p + i] : (T)0;
                v[q].y = eb.p >= 0 ? beta[eb.p + i] : (T)0;
            }
        } else {
#pragma unroll
            for (int q = 0; q < A; ++q) {
                const int i = j + B * q;
                T a = 0, b = 0;
                if (ea.p >= 0) a = (T)0.5 * (beta[ea.p + i] + beta[ea.q + i]);
                if (eb.p >= 0) b = (T)0.5 * (beta[eb.p + i] + beta[eb.q + i]);
                v[q].x = a;
                v[q].y = b;
            }
        }
        if (MEAN64) {
#pragma unroll
            for (int q = 0; q < A; ++q) { sa += (double)v[q].x; sb += (double)v[q].y; }
        }
        if (MEAN64) {
            part[2 * g] = sa;
            part[2 * g + 1] = sb;
        }
        pass_stages<V, false, true, Rs...>(v, lp, tws, 0, 0, 1);
        V* d = s + g * (A + 1);
#pragma unroll
        for (int q = 0; q < A; ++q) d[PassOut<Rs...>::of(q)] = v[q];
    }
    __syncthreads();
}
template <typename V, bool INV, int... Rs>
__device__ __forceinline__ void rows_pass_b(const LinePlan& lp, int P, V* s, const V* __restrict__ tws, int tid, int nt) {
    constexpr int B = RadixProd<Rs...>::v;
    const int A = lp.A;
#pragma unroll 1
    for (int g = tid; g < P * A; g += nt) {
        const int l = g / A, m = g - l * A;
        V* p = s + l * B * (A + 1) + m;
        V v[B];
#pragma unroll
        for (int q = 0; q < B; ++q) v[q] = p[q * (A + 1)];
        pass_stages<V, INV, false, Rs...>(v, lp, tws, lp.sa, m, A);
#pragma unroll
        for (int q = 0; q < B; ++q) p[PassOut<Rs...>::of(q) * (A + 1)] = v[q];
    }
    __syncthreads();
}
template <typename T, bool MEAN64, bool BIG, class Sink>
__device__ __forceinline__ void r2c_two_pass(const InstDev& I, int lb, int P, const RowPtr* __restrict__ rt,
                                             const T* __restrict__ beta, typename VecOf<T>::type* s,
                                             const typename VecOf<T>::type* __restrict__ tws, const Sink& out,
                                             double* __restrict__ rowsum, long long nrows, long long npairs, int tid, int nt) {
    typedef typename VecOf<T>::type V;
    const LinePlan& lp = I.lp_last;
    const int A = lp.A, B = lp.B, N = I.nl, nh = I.nh;
    double* part = MEAN64 ? reinterpret_cast<double*>(s + ((P * B * (A + 1) + 1) & ~1)) : nullptr;
    switch (lp.pa) {
#define CDD_CASE(C, ...) case C: r2c_pass_a<T, MEAN64, __VA_ARGS__>(lp, P, rt, beta, s, part, tws, tid, nt); break;
        CDD_PASS_A_SMALL(CDD_CASE)
        default:
            if constexpr (BIG) {
                switch (lp.pa) { CDD_PASS_A_BIG(CDD_CASE) }
            }
#undef CDD_CASE
    }
    if (MEAN64) {
        for (int r = tid; r < 2 * P; r += nt) {   // row r: its B partial sums in order
            const long long row = 2LL * lb * P + r;
            double acc = 0.0;
            for (int j = 0; j < B; ++j) acc += part[2 * ((r >> 1) * B + j) + (r & 1)];
            if (row < nrows) rowsum[I.rsoff + row] = acc;
        }
    }
    switch (lp.pb) {
#define CDD_CASE(C, ...) case C: rows_pass_b<V, false, __VA_ARGS__>(lp, P, s, tws, tid, nt); break;
        CDD_PASS_B_SMALL(CDD_CASE)
        default:
            if constexpr (BIG) {
                switch (lp.pb) { CDD_PASS_B_BIG(CDD_CASE) }
            }
#undef CDD_CASE
    }
    const FDiv& fa = lp.ns[lp.sa];   // division by A
#pragma unroll 2
    for (int i = tid; i < P * nh; i += nt) {
        const int pl = fdiv_q(I.fd_nh, i), k = i - pl * nh;
        const long long p = (long long)lb * P + pl;
        if (p >= npairs) continue;
        const V* sl = s + pl * B * (A + 1);
        const int km = (k == 0) ? 0 : N - k;
        const V zk = sl[k + fdiv_q(fa, k)], zm = sl[km + fdiv_q(fa, km)];   // k = r A + m at r (A + 1) + m
        V a, b;
        a.x = (T)0.5 * (zk.x + zm.x);
        a.y = (T)0.5 * (zk.y - zm.y);
        b.x = (T)0.5 * (zk.y + zm.y);
        b.y = (T)-0.5 * (zk.x - zm.x);
        out(p, k, a, b, 2 * p + 1 < nrows);
    }
}

// The two-stage plans the row passes run with register-resident first and last stages (the plans
// rows_io_plan accepts).
#define CDD_ROWIO_SEQS(X) X(16, 16) X(16, 8) X(16, 4) X(8, 4)

// ------------------------------------------------------------------------------------------
// C2R along the contiguous axis of 6 components (pairs of half spectra), row ra = o * rows + r:
//   RD_STRESS:    to row ra of a 6-component stress-layout array (+ the FP64 mean stress of FP32
//                 plans);
//   RD_SYM_FIELD: to rows (i, j) and (j, i) of a 9-component field (the cotangent of beta from
//                 that of its symmetric part: d/d beta_ij = d/d beta_ji = the symmetric entry).
// The imaginary parts of the k = 0 and Nyquist bins are dropped (numpy irfft semantics).
// ------------------------------------------------------------------------------------------
//   RD_FIELD9 / RD_FIELD3: row ra of a packed 9- / 3-component array (instance offsets foff and
//                 foff / 3), with an optional epilogue (RowEpilogue).
//   RD_VAC:       row ra of the vacancy concentrations (vacancy instances whose step was applied).
enum RowDest { RD_STRESS = 0, RD_SYM_FIELD = 1, RD_FIELD9 = 2, RD_FIELD3 = 3, RD_VAC = 4 };

// Real-space terms the observables subtract from the inverse transform of output component c:
// out_c -= coef (beta[EPI_P[c]] - beta[EPI_Q[c]]) (EPI_Q < 0: no second term). beta^E: -beta^P;
// rotation (xy, xz, yz) and Rodrigues vector (x, y, z): minus the antisymmetric part of beta^P
// (PlasticityState.py L357-390, L435-446, L447-475).
enum RowEpilogue { EPI_NONE = 0, EPI_BETA_E = 1, EPI_ROTATION = 2, EPI_RODRIGUES = 3 };
static __device__ __constant__ int EPI_P[4][9] = {{-1, -1, -1, -1, -1, -1, -1, -1, -1},
                                           {0, 1, 2, 3, 4, 5, 6, 7, 8},
                                           {1, 2, 5, -1, -1, -1, -1, -1, -1},
                                           {5, 6, 1, -1, -1, -1, -1, -1, -1}};
static __device__ __constant__ int EPI_Q[4][9] = {{-1, -1, -1, -1, -1, -1, -1, -1, -1},
                                           {-1, -1, -1, -1, -1, -1, -1, -1, -1},
                                           {3, 6, 7, -1, -1, -1, -1, -1, -1},
                                           {7, 2, 3, -1, -1, -1, -1, -1, -1}};
static __device__ __constant__ double EPI_COEF[4] = {0.0, 1.0, 0.5, 0.5};

template <typename T>
__device__ __forceinline__ void dst_rows(const InstDev& I, T* base, int mode, long long ra, T*& p, T*& q) {
    if (mode == RD_STRESS) {
        p = q = base + I.soff + ra * I.nl;
        return;
    }
    if (mode == RD_FIELD9 || mode == RD_FIELD3 || mode == RD_VAC) {
        p = q = base + (mode == RD_FIELD9 ? I.foff : (mode == RD_FIELD3 ? I.foff / 3 : I.foff / 9)) + ra * I.nl;
        return;
    }
    const int o = fdiv_q(I.fd_rows, (int)ra);
    const long long r = ra - (long long)o * I.rows;
    const int i = SYM_I[o], j = SYM_J[o];
    p = base + I.foff + (long long)(3 * i + j) * I.cells + r * I.nl;
    q = base + I.foff + (long long)(3 * j + i) * I.cells + r * I.nl;
}

// out -= coef (beta[e.p + idx ..] - beta[e.q + idx ..]) for four (epilogue4) or one value.
template <typename T>
__device__ __forceinline__ void epilogue4(const T* beta, const RowPtr& e, T coef, int idx, T* v) {
    T a[4], b[4] = {0, 0, 0, 0};
    load4(beta + e.p + idx, a);
    if (e.q >= 0) load4(beta + e.q + idx, b);
#pragma unroll
    for (int q = 0; q < 4; ++q) v[q] -= coef * (a[q] - b[q]);
}
template <typename T>
__device__ __forceinline__ T epilogue1(const T* beta, const RowPtr& e, T coef, int idx, T v) {
    const T b = e.q >= 0 ? beta[e.q + idx] : (T)0;
    return v - coef * (beta[e.p + idx] - b);
}

// C2R counterpart: the first stage forms z[i] = A[i] + i B[i] of a pair line straight from the
// half spectra of its two rows (z[N - i] from conjugates), the last stage writes the real rows
// (plus the FP64 mean stress or the real-space epilogue) straight to global memory.
template <typename T, bool MEAN64, int R0, int R1>
__device__ __forceinline__ void c2r_rows_io(const InstDev& I, int lb, int P, int ld, const RowPtr* __restrict__ rt,
                                            const RowPtr* __restrict__ re, const double* __restrict__ rmean,
                                            const typename VecOf<T>::type* __restrict__ src,
                                            typename VecOf<T>::type* s,
                                            const typename VecOf<T>::type* __restrict__ tw1, T* __restrict__ out,
                                            const T* __restrict__ beta, int epi, long long nrows, long long npairs,
                                            int tid, int nt, long long p0, int sld) {
    typedef typename VecOf<T>::type V;
    constexpr int N = R0 * R1;
#pragma unroll 1
    for (int g = tid; g < P * R1; g += nt) {
        const int l = g / R1, j = g - l * R1;
        const long long p = (long long)lb * P + l;
        const V* sa = (p < npairs) ? src + 2 * (p - p0) * sld : nullptr;
        const V* sb = (p < npairs && 2 * p + 1 < nrows) ? sa + sld : nullptr;
        V v[R0];
#pragma unroll
        for (int r = 0; r < R0; ++r) {
            const int i = j + R1 * r;
            const int m = (2 * i <= N) ? i : N - i;
            V A, B;
            A.x = A.y = B.x = B.y = 0;
            if (sa) A = sa[m];
            if (sb) B = sb[m];
            V z;
            if (i == 0 || 2 * i == N) { z.x = A.x; z.y = B.x; }
            else if (2 * i < N) { z.x = A.x - B.y; z.y = A.y + B.x; }
            else { z.x = A.x + B.y; z.y = B.x - A.y; }
            v[r] = z;
        }
        dft<R0, V, true>(v);
        V* d = s + l * ld + row_pad(j * R0);
#pragma unroll
        for (int r = 0; r < R0; ++r) d[r] = v[r];
    }
    __syncthreads();
#pragma unroll 1
    for (int g = tid; g < P * R0; g += nt) {
        const int l = g / R0, j = g - l * R0;
        V w[R1], v[R1];
        load_tw_row<R1>(tw1 + j * tw_pitch(R1, sizeof(V)), w);
        const V* sl = s + l * ld + row_pad(j);
#pragma unroll
        for (int r = 0; r < R1; ++r) {
            const V x = sl[r * R0 + ((r * R0) >> 4)];
            v[r] = (r == 0) ? x : vmulc(x, w[r]);
        }
        dft<R1, V, true>(v);
        const RowPtr ea = rt[2 * l], eb = rt[2 * l + 1];
        if (ea.p < 0) continue;
        const RowPtr xa = re[2 * l], xb = re[2 * l + 1];
        const T ma = (T)rmean[2 * l], mb = (T)rmean[2 * l + 1];
        if (epi != EPI_NONE) {
            // all loads before the first store: none can pass a store to another pointer (64 x 1024 x 64 FP64
            // rotation: 160 us a pass value by value, 125 this way)
#pragma unroll
            for (int r = 0; r < R1; ++r) {
                v[r].x = epilogue1(beta, xa, ma, j + R0 * r, v[r].x);
                if (eb.p >= 0) v[r].y = epilogue1(beta, xb, mb, j + R0 * r, v[r].y);
            }
        }
#pragma unroll
        for (int r = 0; r < R1; ++r) {
            const int k = j + R0 * r;
            T va = v[r].x, vb = v[r].y;
            if (MEAN64) { va += ma; vb += mb; }
            out[ea.p + k] = va;
            if (ea.q != ea.p) out[ea.q + k] = va;
            if (eb.p >= 0) {
                out[eb.p + k] = vb;
                if (eb.q != eb.p) out[eb.q + k] = vb;
            }
        }
    }
}

// The other two-pass plans: pass A forms the pair line from the half spectra; pass B runs in place (rows_pass_b)
// and the rows leave the buffer in 16-byte stores (stores straight from pass B, A values in a row, measured
// slower for 48 and 96).
template <typename T, int... Rs>
__device__ __forceinline__ void c2r_pass_a(const LinePlan& lp, int lb, int P, const typename VecOf<T>::type* __restrict__ src,
                                           int sld, typename VecOf<T>::type* s,
                                           const typename VecOf<T>::type* __restrict__ tws, long long nrows, long long npairs,
                                           int tid, int nt) {
    typedef typename VecOf<T>::type V;
    constexpr int A = RadixProd<Rs...>::v;
    const int B = lp.B, N = lp.n;
#pragma unroll 1
    for (int g = tid; g < P * B; g += nt) {
        const int l = g / B, j = g - l * B;
        const long long p = (long long)lb * P + l;
        const V* sa = (p < npairs) ? src + 2 * p * sld : nullptr;
        const V* sb = (p < npairs && 2 * p + 1 < nrows) ? sa + sld : nullptr;
        V v[A];
#pragma unroll
        for (int q = 0; q < A; ++q) {
            const int i = j + B * q;
            const int m = (2 * i <= N) ? i : N - i;
            V x, y, z;
            x.x = x.y = y.x = y.y = 0;
            if (sa) x = sa[m];
            if (sb) y = sb[m];
            if (i == 0 || 2 * i == N) { z.x = x.x; z.y = y.x; }
            else if (2 * i < N) { z.x = x.x - y.y; z.y = x.y + y.x; }
            else { z.x = x.x + y.y; z.y = y.x - x.y; }
            v[q] = z;
        }
        pass_stages<V, true, true, Rs...>(v, lp, tws, 0, 0, 1);
        V* d = s + g * (A + 1);
#pragma unroll
        for (int q = 0; q < A; ++q) d[PassOut<Rs...>::of(q)] = v[q];
    }
    __syncthreads();
}
}  // namespace cdd
