// Axis-1 pass of the stress pipeline (see stress.cu).
#include "col_pass.cuh"

namespace cdd {

// ------------------------------------------------------------------------------------------
// Complex FFT along axis 1 of a 3-D spectrum, in place, for `ncomp` components.
// Block = (component, i0, column tile of W).
// ------------------------------------------------------------------------------------------
// One column tile: W = 2^lgw columns of N = n1 elements from base (row pitch nhp), wv of them valid.
// The kernel calls it with lgw as a literal for the usual tile widths, so that every shared-memory
// offset of the stages folds to a constant.
template <typename T, bool INV, int TIER>
__device__ __forceinline__ void fft_mid_tile(const InstDev& I, typename VecOf<T>::type* s,
                                             typename VecOf<T>::type* base,
                                             const typename VecOf<T>::type* __restrict__ tws, int lgw, int wv,
                                             int tid, int nt) {
    typedef typename VecOf<T>::type V;
    const int W = 1 << lgw;
    const int N = I.n1, nhp = I.nhp;
    if (line_plan_io(I.lp_mid)) {
        // both stages' other ends in global memory, one shared tile
        const GColT<V, 1> g{base, nhp, 0, lgw, wv};
        const SColT<V, 1> x{s, lgw, 0};
        fft_io<V, INV, 1>(g, x, g, lgw, I.lp_mid, tws, tid, nt, I.lp_mid.twst[0]);
        return;
    }
    if (I.lp_mid.pa) {
        // two passes through one shared tile
        const LinePlan& lp = I.lp_mid;
        __syncthreads();
        const Cols<V> g{base, 0, wv}, t{s, 0, W};
        col_pass_a<V, INV, TIER == 1 ? 1 : 2>(g, nhp, (long long)lp.B * nhp, t, (long long)lp.A << lgw, W, W, lgw, lp, tws, tid, nt);
        col_pass_b<V, INV, TIER == 1 ? 1 : 2>(t, W, (long long)lp.A << lgw, g, nhp, (long long)lp.A * nhp, W, lgw, lp, tws, tid, nt);
        return;
    }
    if (W * (int)sizeof(V) >= 16) {
        tile_async_load(s, base, nhp, N, lgw, wv, tid, nt);
    } else {
#pragma unroll 8
        for (int i = tid; i < N * W; i += nt) {
            const int e = i >> lgw, w = i & (W - 1);
            V z; z.x = 0; z.y = 0;
            if (w < wv) z = base[(long long)e * nhp + w];
            s[i] = z;
        }
    }
    cp_async_wait_all();
    __syncthreads();
    ColLayout<1> lay{lgw, 0};
    s = fft_lines<V, INV>(s, s + N * W, lay, I.lp_mid, tws, tid, nt, I.lp_mid.twst[0]);
    if (W * (int)sizeof(V) >= 16) {
        tile_store(base, s, nhp, N, lgw, wv, tid, nt);
    } else {
#pragma unroll 4
        for (int i = tid; i < N * W; i += nt) {
            const int e = i >> lgw, w = i & (W - 1);
            if (w < wv) base[(long long)e * nhp + w] = s[i];
        }
    }
}

// TIER 1: two-pass forms of at most 16 values a pass; 2: all of them; 3 (FP64): the same on 256 threads instead of 128,
// for plans with long axis-1 lines of the runtime stage engine (mid_engine), whose tiles of two buffers leave room for few blocks (288
// points, 64x288x256: 198 -> 178 us a pass; the compile-time stages of 512 points prefer 128: 270 us against 279).
template <typename T, bool INV, int TIER>
__global__ void __launch_bounds__(mid_threads(sizeof(T), TIER == 3), TIER == 1 ? 4 : (TIER == 2 ? 3 : 2))
k_fft_mid(const InstDev* __restrict__ insts, int n_inst,
                                                 const int* __restrict__ pre,
                                                 typename VecOf<T>::type* spec,
                                                 const typename VecOf<T>::type* __restrict__ tw,
                                                 int pass, int ncomp, int vac_only) {
    typedef typename VecOf<T>::type V;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    V* s = reinterpret_cast<V*>(smem_raw);
    const int ii = find_instance(pre, n_inst, blockIdx.x);
    const InstDev& I = insts[ii];
    int lb = blockIdx.x - pre[ii];
    const PassTile& tl = I.tile[pass];
    const int W = tl.lines, lgw = tl.lgw, ta_n = tl.tiles_a;
    const int ta = lb % ta_n; lb /= ta_n;
    const int i0 = lb % I.n0;
    const int c = lb / I.n0;
    const int N = I.n1, nhp = I.nhp, nh = I.nh;
    const int col0 = ta * W;
    const int wv = min(W, nh - col0);
    const int tid = threadIdx.x, nt = blockDim.x;
    V* tws = s + mid_buffers(I.lp_mid) * N * W;   // twiddle rows after the tile buffers
    stage_tw_to_smem(I.lp_mid, tw, tws, tid, nt);
    pdl_wait();
    if (c >= ncomp) return;   // launch sized for more components than this pass carries
    if (vac_only && !I.vacancy) return;
    V* base = spec + I.spoff + ((long long)c * I.n0 + i0) * (long long)N * nhp + col0;
    if (lgw == 4) fft_mid_tile<T, INV, TIER>(I, s, base, tws, 4, wv, tid, nt);
    else if (lgw == 3) fft_mid_tile<T, INV, TIER>(I, s, base, tws, 3, wv, tid, nt);
    else fft_mid_tile<T, INV, TIER>(I, s, base, tws, lgw, wv, tid, nt);
}

template <typename T, bool INV>
static void mid_t(const PlanCore& P, const LaunchShape& L, int ncomp, int vac_only, cudaStream_t st) {
    typedef typename VecOf<T>::type V;
    const int pass = INV ? PASS_MID_I : PASS_MID_F;
#define CDD_LAUNCH_M(TIER) launch_pdl(k_fft_mid<T, INV, TIER>, L.blocks, L.threads, L.smem, st, P.d_inst, P.n_inst, L.d_pre, \
        (V*)P.d_spec, (const V*)P.d_tw, pass, ncomp, vac_only)
    if constexpr (sizeof(T) == 8) {
        if (P.engine_mid) {
            CDD_LAUNCH_M(3);
            return;
        }
    }
    if (P.big_mid) CDD_LAUNCH_M(2);
    else CDD_LAUNCH_M(1);
#undef CDD_LAUNCH_M
}

void launch_mid(const PlanCore& P, const LaunchShape& L, bool inv, int ncomp, int vac_only, cudaStream_t st) {
    if (L.blocks <= 0) return;
    if (P.precision == CDD_F32) {
        if (inv) mid_t<float, true>(P, L, ncomp, vac_only, st);
        else mid_t<float, false>(P, L, ncomp, vac_only, st);
    } else {
        if (inv) mid_t<double, true>(P, L, ncomp, vac_only, st);
        else mid_t<double, false>(P, L, ncomp, vac_only, st);
    }
}

template <typename T>
static cudaError_t mid_attr(size_t smem) {
    cudaError_t e;
#define CDD_ATTR_M(TIER)                                                               \
    if ((e = set_dyn_smem_limit(k_fft_mid<T, true, TIER>, smem))) return e;            \
    if ((e = set_dyn_smem_limit(k_fft_mid<T, false, TIER>, smem))) return e;
    CDD_ATTR_M(1)
    CDD_ATTR_M(2)
    if constexpr (sizeof(T) == 8) { CDD_ATTR_M(3) }
#undef CDD_ATTR_M
    return cudaSuccess;
}
cudaError_t mid_set_attributes(int precision, size_t smem) {
    return precision == CDD_F32 ? mid_attr<float>(smem) : mid_attr<double>(smem);
}

}  // namespace cdd
