// Column passes: the transforms along axis 1 (fft_mid.cu) and axis 0 (green.cu) of the half spectra.
#pragma once
#include "cdd_internal.cuh"

namespace cdd {

// The tile's column lines, element i of line (c, w) at base[c cstride + i stride + w] (shared: stride 2^lgw):
// one pass (see pass_stages) of all `lines` = components << lgw lines, J butterflies each, butterfly j's
// elements q at in0(j) + q istep, its outputs m at out0(j) + m ostep. Columns w >= wv of a global tile read
// as zero and are not written. Consecutive threads walk the columns, then the components, so that
// neighbours read whole row segments and the slots (cs an odd number of rows apart) spread over the banks.
template <typename V> struct Cols {
    V* base;
    long long cstride;
    int wv;
};
template <typename V, bool INV, bool FIRST, int... Rs>
__device__ __forceinline__ void col_pass(const Cols<V>& in, long long in_j, long long in_q, const Cols<V>& out, long long out_j,
                                         long long out_m, int lines, int lgw, int J, const LinePlan& lp,
                                         const V* __restrict__ tws, int tid, int nt) {
    constexpr int R = RadixProd<Rs...>::v;
    const int W = 1 << lgw;
#pragma unroll 1
    for (int g = tid; g < lines * J; g += nt) {
        const int j = g / lines, l = g - j * lines;
        const int c = l >> lgw, w = l & (W - 1);
        const V* p = in.base + c * in.cstride + j * in_j + w;
        const bool vi = w < in.wv;
        V v[R];
#pragma unroll
        for (int q = 0; q < R; ++q) {
            V z;
            z.x = 0;
            z.y = 0;
            v[q] = vi ? p[q * in_q] : z;
        }
        pass_stages<V, INV, FIRST, Rs...>(v, lp, tws, FIRST ? 0 : lp.sa, FIRST ? 0 : j, FIRST ? 1 : lp.A);
        V* d = out.base + c * out.cstride + j * out_j + w;
        if (w < out.wv) {
#pragma unroll
            for (int q = 0; q < R; ++q) d[PassOut<Rs...>::of(q) * out_m] = v[q];
        }
    }
    __syncthreads();
}
// Pass A / pass B of lp. TIER 0: plans whose passes are one stage each (16, 8 | 16, 8, 4) only; 1: passes of
// at most 16 values; 2: all of them.
template <typename V, bool INV, int TIER>
__device__ __forceinline__ void col_pass_a(const Cols<V>& in, long long in_j, long long in_q, const Cols<V>& out, long long out_j,
                                           long long out_m, int lines, int lgw, const LinePlan& lp,
                                           const V* __restrict__ tws, int tid, int nt) {
#define CDD_RUN(...) col_pass<V, INV, true, __VA_ARGS__>(in, in_j, in_q, out, out_j, out_m, lines, lgw, lp.B, lp, tws, tid, nt)
    if constexpr (TIER == 0) {
        if (lp.A == 16) CDD_RUN(16);
        else CDD_RUN(8);
    } else {
        switch (lp.pa) {
#define CDD_CASE(C, ...) case C: CDD_RUN(__VA_ARGS__); break;
            CDD_PASS_A_SMALL(CDD_CASE)
            default:
                if constexpr (TIER == 2) {
                    switch (lp.pa) { CDD_PASS_A_BIG(CDD_CASE) }
                }
        }
    }
#undef CDD_RUN
}
template <typename V, bool INV, int TIER>
__device__ __forceinline__ void col_pass_b(const Cols<V>& in, long long in_j, long long in_q, const Cols<V>& out, long long out_j,
                                           long long out_m, int lines, int lgw, const LinePlan& lp,
                                           const V* __restrict__ tws, int tid, int nt) {
#define CDD_RUN(...) col_pass<V, INV, false, __VA_ARGS__>(in, in_j, in_q, out, out_j, out_m, lines, lgw, lp.A, lp, tws, tid, nt)
    if constexpr (TIER == 0) {
        if (lp.B == 16) CDD_RUN(16);
        else if (lp.B == 8) CDD_RUN(8);
        else CDD_RUN(4);
    } else {
        switch (lp.pb) {
            CDD_PASS_B_SMALL(CDD_CASE)
            default:
                if constexpr (TIER == 2) {
                    switch (lp.pb) { CDD_PASS_B_BIG(CDD_CASE) }
                }
#undef CDD_CASE
        }
    }
#undef CDD_RUN
}
// Whether TIER 0 runs lp.
inline bool pass_lean(const LinePlan& lp) {
    return lp.pa && lp.sa == 1 && lp.nst == 2 && (lp.A == 16 || lp.A == 8) && (lp.B == 16 || lp.B == 8 || lp.B == 4);
}

}  // namespace cdd
