// C2R row pass of the stress pipeline (see stress.cu).
#include "rows_pass.cuh"

namespace cdd {

template <typename T, bool MEAN64, int TIER>
__global__ void __launch_bounds__(row_threads_max(sizeof(T)), TIER == 2 ? 3 : 4)
k_c2r_rows(const InstDev* __restrict__ insts, int n_inst,
                                                  const int* __restrict__ pre,
                                                  const typename VecOf<T>::type* spec,
                                                  T* out,
                                                  const typename VecOf<T>::type* __restrict__ tw,
                                                  const double* sbar, int mode, int ncomp,
                                                  const T* beta, int epi,
                                                  const InstClock* clk) {
    typedef typename VecOf<T>::type V;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    V* s = reinterpret_cast<V*>(smem_raw);
    const int ii = find_instance(pre, n_inst, blockIdx.x);
    const InstDev& I = insts[ii];
    const int lb = blockIdx.x - pre[ii];
    const int N = I.nl, P = I.tile[PASS_C2R].lines, ld = rows_ld(N), nh = I.nh;
    const long long nrows = (long long)ncomp * I.rows;
    // a launch sized for more components than this pass carries, or other instances' diffusion
    if (2LL * lb * P >= nrows || (mode == RD_VAC && !I.vacancy)) {
        pdl_wait();
        return;
    }
    const long long npairs = (nrows + 1) / 2;
    const int tid = threadIdx.x, nt = blockDim.x;
    const V* src = spec + I.spoff;
    const bool io = rows_io_plan(I.lp_last, P);
    V* tws = s + ((rows_elems(I.lp_last, P, sizeof(V)) + 1) & ~1);
    stage_tw_to_smem(I.lp_last, tw, tws, tid, nt);
    pdl_wait();
    if (mode == RD_VAC && !clk[ii].active) return;
    // row table: the destination rows of each of the block's 2P rows and their FP64 mean stress
    RowPtr* rt = rows_table(tws, I.lp_last.twspan);
    RowPtr* re = rt + 2 * P;                                        // epilogue source rows
    double* rmean = reinterpret_cast<double*>(re + 2 * P);          // mean stress or epilogue coefficient
    for (int r = tid; r < 2 * P; r += nt) {
        const long long ra = 2LL * lb * P + r;
        RowPtr e, ep;
        e.p = e.q = -1;
        ep.p = ep.q = -1;
        double m = 0.0;
        if (ra < nrows) {
            T *pd, *qd;
            dst_rows(I, out, mode, ra, pd, qd);
            e.p = pd - out;
            e.q = qd - out;
            if (MEAN64) m = mean_stress(I, sbar + 9 * ii, fdiv_q(I.fd_rows, (int)ra));
            if (epi != EPI_NONE) {
                const int o = fdiv_q(I.fd_rows, (int)ra);
                const long long rr = ra - (long long)o * I.rows;
                const int cp = EPI_P[epi][o], cq = EPI_Q[epi][o];
                ep.p = I.foff + (long long)cp * I.cells + rr * I.nl;
                ep.q = cq >= 0 ? I.foff + (long long)cq * I.cells + rr * I.nl : -1;
                m = EPI_COEF[epi];
            }
        }
        rt[r] = e;
        re[r] = ep;
        rmean[r] = m;
    }
    {
        const LinePlan& lq = I.lp_last;
        const V* tw1 = tws + (lq.twst[1] - lq.twst[0]);
#define CDD_C2R_IO(A, B)                                                                                      \
        if (io && lq.radix[0] == A && lq.radix[1] == B) {                                                     \
            c2r_rows_io<T, MEAN64, A, B>(I, lb, P, ld, rt, re, rmean, src, s, tw1, out, beta, epi, nrows, npairs, \
                                          tid, nt, 0, I.nhp);                                                 \
            return;                                                                                           \
        }
        CDD_ROWIO_SEQS(CDD_C2R_IO)
#undef CDD_C2R_IO
    }
    if constexpr (TIER == 0) return;   // every instance took one of the forms above
    else {
    const LinePlan& lp = I.lp_last;
    const bool two = lp.pa != 0;
    if (two) {
        __syncthreads();
        switch (lp.pa) {
#define CDD_CASE(C, ...) case C: c2r_pass_a<T, __VA_ARGS__>(lp, lb, P, src, I.nhp, s, tws, nrows, npairs, tid, nt); break;
            CDD_PASS_A_SMALL(CDD_CASE)
            default:
                if constexpr (TIER == 2) {
                    switch (lp.pa) { CDD_PASS_A_BIG(CDD_CASE) }
                }
#undef CDD_CASE
        }
        switch (lp.pb) {
#define CDD_CASE(C, ...) case C: rows_pass_b<V, true, __VA_ARGS__>(lp, P, s, tws, tid, nt); break;
            CDD_PASS_B_SMALL(CDD_CASE)
            default:
                if constexpr (TIER == 2) {
                    switch (lp.pb) { CDD_PASS_B_BIG(CDD_CASE) }
                }
#undef CDD_CASE
        }
    } else {
#pragma unroll 4
    for (int i = tid; i < P * nh; i += nt) {
        int pl = fdiv_q(I.fd_nh, i), k = i - pl * nh;
        long long p = (long long)lb * P + pl;
        V A, B;
        A.x = A.y = B.x = B.y = 0;
        if (p < npairs) {
            long long ra = 2 * p;
            A = src[ra * I.nhp + k];
            if (ra + 1 < nrows) B = src[(ra + 1) * I.nhp + k];
        }
        V z;
        if (k == 0 || 2 * k == N) {
            z.x = A.x; z.y = B.x;
            s[pl * ld + row_pad(k)] = z;
        } else {
            z.x = A.x - B.y; z.y = A.y + B.x;
            s[pl * ld + row_pad(k)] = z;
            z.x = A.x + B.y; z.y = B.x - A.y;
            s[pl * ld + row_pad(N - k)] = z;
        }
    }
    __syncthreads();
    RowLayout lay{P, ld};
    s = fft_lines<V, true>(s, s + P * ld, lay, lp, tws, tid, nt, lp.twst[0]);
    }
    // element idx of line pl: two-pass lines are groups of A + 1
    const FDiv& fa = lp.ns[lp.sa];
    const int pitch = two ? lp.B * (lp.A + 1) : ld;
    const bool groups4 = !two || (lp.A & 3) == 0;   // four consecutive elements stay in one group (and pad period)
    auto at = [&](int idx) { return two ? idx + fdiv_q(fa, idx) : row_pad(idx); };
    const bool vec = ((N & 3) == 0) && ((((uintptr_t)(out + I.soff)) & 15) == 0) &&
                     ((((uintptr_t)(out + I.foff)) & 15) == 0) && ((((uintptr_t)(out + I.foff / 3)) & 15) == 0) &&
                     ((((uintptr_t)(out + I.foff / 9)) & 15) == 0) &&
                     (epi == EPI_NONE || ((((uintptr_t)(beta + I.foff)) & 15) == 0)) && ((I.cells & 3) == 0);
    if (vec) {
#pragma unroll 2
        for (int i4 = tid; i4 < (P * N) >> 2; i4 += nt) {
            const int i = i4 << 2;
            const int pl = fdiv_q(I.fd_nl, i), idx = i - pl * N;
            const RowPtr ea = rt[2 * pl], eb = rt[2 * pl + 1];
            if (ea.p < 0) continue;
            T va[4], vb[4];
            const V* sr = s + pl * pitch;
            const int o = at(idx);
#pragma unroll
            for (int q = 0; q < 4; ++q) { V z = sr[groups4 ? o + q : at(idx + q)]; va[q] = z.x; vb[q] = z.y; }
            if (MEAN64) {
                const T ma = (T)rmean[2 * pl], mb = (T)rmean[2 * pl + 1];
#pragma unroll
                for (int q = 0; q < 4; ++q) { va[q] += ma; vb[q] += mb; }
            }
            if (epi != EPI_NONE) {
                epilogue4(beta, re[2 * pl], (T)rmean[2 * pl], idx, va);
                if (eb.p >= 0) epilogue4(beta, re[2 * pl + 1], (T)rmean[2 * pl + 1], idx, vb);
            }
            store4(out + ea.p + idx, va);
            if (ea.q != ea.p) store4(out + ea.q + idx, va);
            if (eb.p >= 0) {
                store4(out + eb.p + idx, vb);
                if (eb.q != eb.p) store4(out + eb.q + idx, vb);
            }
        }
    } else {
        for (int i = tid; i < P * N; i += nt) {
            const int pl = fdiv_q(I.fd_nl, i), idx = i - pl * N;
            const RowPtr ea = rt[2 * pl], eb = rt[2 * pl + 1];
            if (ea.p < 0) continue;
            V z = s[pl * pitch + at(idx)];
            T va = z.x, vb = z.y;
            if (MEAN64) {
                va += (T)rmean[2 * pl];
                vb += (T)rmean[2 * pl + 1];
            }
            if (epi != EPI_NONE) {
                va = epilogue1(beta, re[2 * pl], (T)rmean[2 * pl], idx, va);
                if (eb.p >= 0) vb = epilogue1(beta, re[2 * pl + 1], (T)rmean[2 * pl + 1], idx, vb);
            }
            out[ea.p + idx] = va;
            if (ea.q != ea.p) out[ea.q + idx] = va;
            if (eb.p >= 0) {
                out[eb.p + idx] = vb;
                if (eb.q != eb.p) out[eb.q + idx] = vb;
            }
        }
    }
    }
}

template <typename T, bool MEAN64>
static void c2r_t(const PlanCore& P, const LaunchShape& L, void* out, int mode, int ncomp, const void* beta, int epi, cudaStream_t st) {
    typedef typename VecOf<T>::type V;
#define CDD_LAUNCH_R(TIER) launch_pdl(k_c2r_rows<T, MEAN64, TIER>, L.blocks, L.threads, L.smem, st, P.d_inst, P.n_inst, L.d_pre, (const V*)P.d_spec, (T*)out, \
        (const V*)P.d_tw, P.d_sbar, mode, ncomp, (const T*)beta, epi, P.d_clock)
    if (P.rows_tier == 0) CDD_LAUNCH_R(0);
    else if (P.rows_tier == 1) CDD_LAUNCH_R(1);
    else CDD_LAUNCH_R(2);
#undef CDD_LAUNCH_R
}

void launch_c2r(const PlanCore& P, const LaunchShape& L, void* out, bool mean64, int mode, int ncomp, const void* beta, int epi,
                cudaStream_t st) {
    if (P.precision != CDD_F32) c2r_t<double, false>(P, L, out, mode, ncomp, beta, epi, st);
    else if (mean64) c2r_t<float, true>(P, L, out, mode, ncomp, beta, epi, st);
    else c2r_t<float, false>(P, L, out, mode, ncomp, beta, epi, st);
}

template <typename T, bool MEAN64>
static cudaError_t c2r_attr(size_t smem) {
    cudaError_t e;
    if ((e = set_dyn_smem_limit(k_c2r_rows<T, MEAN64, 0>, smem))) return e;
    if ((e = set_dyn_smem_limit(k_c2r_rows<T, MEAN64, 1>, smem))) return e;
    return set_dyn_smem_limit(k_c2r_rows<T, MEAN64, 2>, smem);
}
cudaError_t c2r_set_attributes(int precision, size_t smem) {
    if (precision != CDD_F32) return c2r_attr<double, false>(smem);
    const cudaError_t e = c2r_attr<float, false>(smem);
    return e ? e : c2r_attr<float, true>(smem);
}

}  // namespace cdd
