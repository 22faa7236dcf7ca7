// R2C row pass of the stress pipeline (see stress.cu).
#include "rows_pass.cuh"

namespace cdd {

// ------------------------------------------------------------------------------------------
// R2C along the contiguous axis of the 6 input components (see RowSource): pairs of real rows
// (a + i b) per complex FFT. FP32 plans also record FP64 sums of the rows (the k = 0 mode).
// ------------------------------------------------------------------------------------------
template <typename T, bool MEAN64, int TIER>
__global__ void __launch_bounds__(row_threads_max(sizeof(T)), TIER == 2 ? 3 : 4)
k_r2c_rows(const InstDev* __restrict__ insts, int n_inst,
                                                  const int* __restrict__ pre,
                                                  const T* beta,
                                                  typename VecOf<T>::type* spec,
                                                  const typename VecOf<T>::type* __restrict__ tw,
                                                  double* rowsum, int mode, int ncomp) {
    typedef typename VecOf<T>::type V;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    V* s = reinterpret_cast<V*>(smem_raw);
    const int ii = find_instance(pre, n_inst, blockIdx.x);
    const InstDev& I = insts[ii];
    const int lb = blockIdx.x - pre[ii];
    const int N = I.nl, P = I.tile[PASS_R2C].lines, ld = rows_ld(N);
    const long long nrows = (long long)ncomp * I.rows;
    // a launch sized for more components than this pass carries, or other instances' diffusion
    if (2LL * lb * P >= nrows || (mode == RS_VAC && !I.vacancy)) {
        pdl_wait();
        return;
    }
    const long long npairs = (nrows + 1) / 2;
    const int tid = threadIdx.x, nt = blockDim.x;
    const T half = (T)0.5;

    // row table: the two source rows of each of the block's 2P rows (-1: past the last row)
    const bool io = rows_io_plan(I.lp_last, P);
    V* tws = s + ((rows_elems(I.lp_last, P, sizeof(V)) + 1) & ~1);   // twiddle rows, 16-byte aligned after the buffers
    RowPtr* rt = rows_table(tws, I.lp_last.twspan);
    for (int r = tid; r < 2 * P; r += nt) {
        const long long ra = 2LL * lb * P + r;
        RowPtr e;
        e.p = e.q = -1;
        if (ra < nrows) {
            const T *pa, *qa;
            src_rows(I, beta, mode, ra, pa, qa);
            e.p = pa - beta;
            e.q = qa - beta;
        }
        rt[r] = e;
    }
    stage_tw_to_smem(I.lp_last, tw, tws, tid, nt);
    pdl_wait();
    __syncthreads();
    {
        const LinePlan& lq = I.lp_last;
        const V* tw1 = tws + (lq.twst[1] - lq.twst[0]);
#define CDD_R2C_IO(A, B)                                                                                      \
        if (io && lq.radix[0] == A && lq.radix[1] == B) {                                                     \
            r2c_rows_io<T, MEAN64, A, B, false>(I, lb, P, ld, rt, beta, s, tw1, RowSink<V>{spec + I.spoff, I.nhp}, \
                                                 rowsum, nrows, npairs, tid, nt, 0);                          \
            return;                                                                                           \
        }
        CDD_ROWIO_SEQS(CDD_R2C_IO)
#undef CDD_R2C_IO
    }
    if constexpr (TIER == 0) return;   // every instance took one of the forms above
    else {
    if (I.lp_last.pa) {
        r2c_two_pass<T, MEAN64, TIER == 2>(I, lb, P, rt, beta, s, tws, RowSink<V>{spec + I.spoff, I.nhp}, rowsum, nrows, npairs, tid, nt);
        return;
    }
    const bool vec = ((N & 3) == 0) && ((((uintptr_t)(beta + I.foff)) & 15) == 0) &&
                     ((((uintptr_t)(beta + I.soff)) & 15) == 0) && ((((uintptr_t)(beta + I.foff / 9)) & 15) == 0) &&
                     ((I.cells & 3) == 0);
    if (vec) {
#pragma unroll 2
        for (int i4 = tid; i4 < (P * N) >> 2; i4 += nt) {
            const int i = i4 << 2;
            const int pl = fdiv_q(I.fd_nl, i), idx = i - pl * N;
            const RowPtr ea = rt[2 * pl], eb = rt[2 * pl + 1];
            T a[4] = {0, 0, 0, 0}, b[4] = {0, 0, 0, 0};
            if (ea.p >= 0) {
                T x[4], y[4];
                load4(beta + ea.p + idx, x);
                load4(beta + ea.q + idx, y);
#pragma unroll
                for (int q = 0; q < 4; ++q) a[q] = half * (x[q] + y[q]);
            }
            if (eb.p >= 0) {
                T x[4], y[4];
                load4(beta + eb.p + idx, x);
                load4(beta + eb.q + idx, y);
#pragma unroll
                for (int q = 0; q < 4; ++q) b[q] = half * (x[q] + y[q]);
            }
            V* d = s + pl * ld + row_pad(idx);
#pragma unroll
            for (int q = 0; q < 4; ++q) { V z; z.x = a[q]; z.y = b[q]; d[q] = z; }
        }
    } else {
#pragma unroll 2
        for (int i = tid; i < P * N; i += nt) {
            const int pl = fdiv_q(I.fd_nl, i), idx = i - pl * N;
            const RowPtr ea = rt[2 * pl], eb = rt[2 * pl + 1];
            V z; z.x = 0; z.y = 0;
            if (ea.p >= 0) z.x = half * (beta[ea.p + idx] + beta[ea.q + idx]);
            if (eb.p >= 0) z.y = half * (beta[eb.p + idx] + beta[eb.q + idx]);
            s[pl * ld + row_pad(idx)] = z;
        }
    }
    __syncthreads();
    if (MEAN64) {
        const int lane = tid & 31, warp = tid >> 5, nw = nt >> 5;
        for (int r = warp; r < 2 * P; r += nw) {
            int pl = r >> 1;
            long long row = ((long long)lb * P + pl) * 2 + (r & 1);
            double acc = 0.0;
            for (int idx = lane; idx < N; idx += 32) {
                V z = s[pl * ld + row_pad(idx)];
                acc += (double)((r & 1) ? z.y : z.x);
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
            if (lane == 0 && row < nrows) rowsum[I.rsoff + row] = acc;
        }
    }
    RowLayout lay{P, ld};
    s = fft_lines<V, false>(s, s + P * ld, lay, I.lp_last, tws, tid, nt, I.lp_last.twst[0]);
    const int nh = I.nh;
    V* dst = spec + I.spoff;
    for (int i = tid; i < P * nh; i += nt) {
        int pl = fdiv_q(I.fd_nh, i), k = i - pl * nh;
        long long p = (long long)lb * P + pl;
        if (p >= npairs) continue;
        V zk = s[pl * ld + row_pad(k)];
        int km = (k == 0) ? 0 : N - k;
        V zm = s[pl * ld + row_pad(km)];
        V a, b;
        a.x = (T)0.5 * (zk.x + zm.x);
        a.y = (T)0.5 * (zk.y - zm.y);
        b.x = (T)0.5 * (zk.y + zm.y);
        b.y = (T)-0.5 * (zk.x - zm.x);
        long long ra = 2 * p;
        dst[ra * I.nhp + k] = a;
        if (ra + 1 < nrows) dst[(ra + 1) * I.nhp + k] = b;
    }
    }
}

template <typename T, bool MEAN64>
static void r2c_t(const PlanCore& P, const LaunchShape& L, const void* in, double* rowsum, int mode, int ncomp, cudaStream_t st) {
    typedef typename VecOf<T>::type V;
#define CDD_LAUNCH_R(TIER) launch_pdl(k_r2c_rows<T, MEAN64, TIER>, L.blocks, L.threads, L.smem, st, P.d_inst, P.n_inst, L.d_pre, (const T*)in, (V*)P.d_spec, \
        (const V*)P.d_tw, rowsum, mode, ncomp)
    if (P.rows_tier == 0) CDD_LAUNCH_R(0);
    else if (P.rows_tier == 1) CDD_LAUNCH_R(1);
    else CDD_LAUNCH_R(2);
#undef CDD_LAUNCH_R
}

void launch_r2c(const PlanCore& P, const LaunchShape& L, const void* in, double* rowsum, int mode, int ncomp, cudaStream_t st) {
    if (P.precision != CDD_F32) r2c_t<double, false>(P, L, in, nullptr, mode, ncomp, st);
    else if (rowsum) r2c_t<float, true>(P, L, in, rowsum, mode, ncomp, st);
    else r2c_t<float, false>(P, L, in, nullptr, mode, ncomp, st);
}

template <typename T, bool MEAN64>
static cudaError_t r2c_attr(size_t smem) {
    cudaError_t e;
    if ((e = set_dyn_smem_limit(k_r2c_rows<T, MEAN64, 0>, smem))) return e;
    if ((e = set_dyn_smem_limit(k_r2c_rows<T, MEAN64, 1>, smem))) return e;
    return set_dyn_smem_limit(k_r2c_rows<T, MEAN64, 2>, smem);
}
cudaError_t r2c_set_attributes(int precision, size_t smem) {
    if (precision != CDD_F32) return r2c_attr<double, false>(smem);
    const cudaError_t e = r2c_attr<float, false>(smem);
    return e ? e : r2c_attr<float, true>(smem);
}

}  // namespace cdd
