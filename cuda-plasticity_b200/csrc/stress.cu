// Internal stress sigma(beta^P) on the device: a batched real-to-complex / complex-to-real FFT
// pipeline with the isotropic Green's-function contraction fused into the k-space pass.
//
// Mathematics (PlasticityState.CalculateSigma(source='betaE') + CalculateBetaElastic,
// Plasticity/PlasticityStates/PlasticityState.py L85-127, L357-390):
//   betaE^(k)_ij = kmask * sum_mn T_ijmn(k) betaP^(k)_mn - betaP^(k)_ij,
//   T_ijmn = A k_i k_j d_mn / kSq + k_i (k_m d_jn + k_n d_jm) / kSq - B k_i k_j k_m k_n / kSqSq,
//   A = lam / (lam + 2 mu), B = 2 (lam + mu) / (lam + 2 mu), kSq += ME, kSqSq += ME,
//   sigma_ij = lam tr(betaE) d_ij + mu (betaE_ij + betaE_ji).
// Contracting T with betaP gives, per k point,
//   sum_mn T_ijmn b_mn = k_i g_j,  g_j = k_j (A s / kSq - B r / kSqSq) + (p_j + q_j) / kSq,
//   s = tr b, p_j = sum_m k_m b_mj, q_j = sum_n b_jn k_n, r = sum_m k_m q_m,
// so the six stress components are formed directly in k space and only six inverse transforms
// are needed. The k tables are the reference's (FourierSpaceTools.py L5-59), built on the host.
//
// 3-D pipeline (grid n0 x n1 x n2, last axis contiguous, spectrum rows of nhp complex):
//   R2C rows (axis 2, two real rows per complex FFT)  -> forward FFT along axis 1
//   -> [forward FFT along axis 0, Green contraction, inverse FFT along axis 0] in one kernel
//   -> inverse FFT along axis 1 -> C2R rows (axis 2).
// 2-D: R2C rows (axis 1) -> fused Green pass along axis 0 -> C2R rows.
//
// FP32 plans keep the k = 0 mode in FP64: the R2C pass records FP64 row sums of beta, the k-space pass's first
// blocks form their means, and the C2R pass adds the mean stress -lam tr<b> d - mu (<b> + <b>^T) after the FP32
// transforms (which carry a zero k = 0 mode).
#include "rows_pass.cuh"

#include <cooperative_groups.h>
namespace cg = cooperative_groups;

namespace cdd {

// ------------------------------------------------------------------------------------------
// Plane passes (3-D FP32 instances that plane_eligible accepts): the transforms along the
// contiguous axis and along axis 1 of one z-plane of one component in one kernel each way, so the
// spectrum crosses HBM once between them instead of twice. One cluster of PLANE_C blocks per
// (component o, plane z); block r owns rows [r Rc, (r+1) Rc) of the plane (Rc = n1 / PLANE_C) and
// spectrum columns [r W, (r+1) W) (W = nl / (2 PLANE_C)). Data moves between the blocks of a
// cluster by stores into the owner's shared memory (distributed shared memory), which do not stall
// the storing thread:
//   forward: block r runs the R2C of its rows (two real rows per complex FFT, as k_r2c_rows); the
//     last FFT stage stores each half-spectrum bin straight into the shared column tile S_col of
//     the block that owns its column; after a cluster barrier every block transforms its W columns
//     along axis 1 and writes them to the plan's spectrum, which the k-space pass (k_green) reads
//     as before;
//   inverse: block r runs the inverse axis-1 transform of its W columns, the first stage reading
//     them from the spectrum and the last stage storing each value into the shared row tile S_own
//     of the block that owns its row; after a cluster barrier every block runs the C2R of its rows
//     (plus the FP64 mean stress) into sigma.
// Every kernel starts with a cluster barrier, so no block stores into a block that has not started.
// Columns 0 and nl/2 of a row's half spectrum are real (the R2C split makes their imaginary parts
// exactly zero), so block 0 carries them as one complex column X0 + i X_{nl/2}; its axis-1
// transform F = F0 + i FN is split again by Hermitian symmetry, F0(ky) = (F(ky) + conj F(-ky)) / 2,
// FN(ky) = (F(ky) - conj F(-ky)) / (2i). The inverse packs the Hermitian parts H(G)(ky) =
// (G(ky) + conj G(-ky)) / 2 of the two columns as H(G0) + i H(GN): the inverse transform of H(G) is
// the real part of that of G, which is what the C2R keeps of those bins (numpy's irfft semantics;
// the k tables' positive Nyquist values make the k-space operator's output not exactly Hermitian
// on the axis-1 Nyquist line). That keeps W columns per block, a power of two. Same codelets,
// twiddles and row tables as the separate passes; results agree with them to rounding.
// Shared memory (V = complex): forward: the row pass's line buffer (P x rows_ld(nl); then the
// axis-1 scratch tile, n1 x W) and S_col (n1 x W); inverse: S_own (Rc x ldo) and a buffer of
// max(n1 x W, P x rows_ld(nl)) (the axis-1 scratch tile, then the C2R line buffer); both: the row
// twiddles and the row tables.
// ------------------------------------------------------------------------------------------
constexpr int PLANE_C = PLANE_CLUSTER;

struct PlaneGeom {
    int Rc, P, W, lgw, ldo, ld;
    size_t a, b, tw, tab, total;   // region sizes in bytes (16-byte multiples) and the sum
};

__host__ __device__ inline PlaneGeom plane_geom(const InstDev& I, size_t velt) {
    PlaneGeom g;
    g.Rc = I.n1 / PLANE_C;
    g.P = g.Rc / 2;
    g.W = (I.nl / 2) / PLANE_C;
    g.lgw = 0;
    while ((1 << g.lgw) < g.W) ++g.lgw;
    g.ldo = (I.nh + 1) & ~1;   // even: 16-byte aligned FP32 rows
    g.ld = rows_ld(I.nl);
    auto r16 = [](size_t v) { return (v + 15) & ~(size_t)15; };
    const size_t colt = (size_t)I.n1 * g.W * velt;
    const size_t own = (size_t)g.Rc * g.ldo * velt, line = (size_t)g.P * g.ld * velt;
    // region a: forward line buffer / axis-1 scratch, inverse S_own; region b: forward S_col,
    // inverse axis-1 scratch / C2R line buffer
    const size_t fa = line > colt ? line : colt, ia = own;
    const size_t fb = colt, ib = line > colt ? line : colt;
    g.a = r16(fa > ia ? fa : ia);
    g.b = r16(fb > ib ? fb : ib);
    g.tw = r16((size_t)I.lp_last.twspan * velt);
    g.tab = r16(rows_table_bytes(g.P));
    g.total = g.a + g.b + g.tw + g.tab;
    return g;
}

// Whether instance I runs its stress transforms through the plane passes (FP32 plans): n1 and nl
// powers of two with Rc = n1 / PLANE_C an even number of rows, at least two columns per block, the
// register-resident two-stage row codelets (rows_io_plan) and a two-stage compile-time axis-1 plan.
bool plane_eligible(const InstDev& I, int precision, size_t smem_limit) {
    if (precision != CDD_F32 || I.nd != 3) return false;
    auto pow2 = [](int v) { return v > 0 && (v & (v - 1)) == 0; };
    if (!pow2(I.n1) || !pow2(I.nl)) return false;
    if (I.n1 % (2 * PLANE_C) != 0 || (I.nl / 2) % (2 * PLANE_C) != 0) return false;
    const PlaneGeom g = plane_geom(I, sizeof(float2));
    if (!rows_io_plan(I.lp_last, g.P)) return false;
    if (!line_plan_io(I.lp_mid)) return false;
    return g.total + 1024 <= smem_limit;
}

size_t plane_smem_bytes(const InstDev& I) { return plane_geom(I, sizeof(float2)).total; }

// Forward: bin k of rows y0 + 2q and y0 + 2q + 1 of the plane goes to the column tile S_col of the
// block owning column k (element (y, w) at (y << lgw) + w); bins 0 and nl/2 (real) to the real and
// imaginary parts of block 0's column 0.
template <typename V> struct PlaneColSink {
    V* s_col;   // this block's S_col (the same offset in every block of the cluster)
    int y0, lgw, half;
    __device__ __forceinline__ void operator()(long long q, int k, const V& a, const V& b, bool) const {
        cg::cluster_group cl = cg::this_cluster();
        const int y = y0 + 2 * (int)q;
        if (k == 0 || k == half) {
            V* d = cl.map_shared_rank(s_col, 0);
            if (k == 0) {
                d[y << lgw].x = a.x;
                d[(y + 1) << lgw].x = b.x;
            } else {
                d[y << lgw].y = a.x;
                d[(y + 1) << lgw].y = b.x;
            }
        } else {
            const int w = k & ((1 << lgw) - 1);
            V* d = cl.map_shared_rank(s_col, k >> lgw);
            d[(y << lgw) + w] = a;
            d[((y + 1) << lgw) + w] = b;
        }
    }
};

// Inverse, first axis-1 stage: element ky of column w of this block read from the spectrum; block
// 0's column 0 is H(G0) + i H(GN) of spectrum columns 0 and nl/2.
template <typename V> struct PlaneSpecIn {
    const V* src;   // the plane's first spectrum row, at this block's first column
    long long nhp;
    int n1, half;
    bool packed;    // block 0: column 0 carries bins 0 and nl/2
    struct Walk {
        const V* p;       // element i0 of the column
        const V* base;    // row 0 of the plane at column 0 (packed column)
        long long stride, nhp;
        int i0, step, n1, half;
        bool packed;
        __device__ __forceinline__ V ld(int r) const {
            if (!packed) return p[r * stride];
            typedef decltype(V().x) T;
            const int ky = i0 + r * step, km = ky == 0 ? 0 : n1 - ky;
            const V* sr = base + (long long)ky * nhp;
            const V* sm = base + (long long)km * nhp;
            const V f0 = sr[0], f0m = sm[0], fn = sr[half], fnm = sm[half];
            const T ax = (T)0.5 * (f0.x + f0m.x), ay = (T)0.5 * (f0.y - f0m.y);
            const T bx = (T)0.5 * (fn.x + fnm.x), by = (T)0.5 * (fn.y - fnm.y);
            V v;
            v.x = ax - by;
            v.y = ay + bx;
            return v;
        }
    };
    __device__ __forceinline__ Walk walk(int l, int i0, int step) const {
        return {src + (long long)i0 * nhp + l, src, (long long)step * nhp, nhp, i0, step, n1, half, packed && l == 0};
    }
};

// Inverse, last axis-1 stage: element y of column w stored into the row tile S_own of the block
// owning row y (row ly at ly * ldo); block 0's column 0 is unpacked into bins 0 and nl/2 (real).
template <typename V> struct PlaneRowOut {
    V* s_own;
    int col0, lrc, ldo, half;
    bool packed;
    struct Walk {
        V* s_own;
        int i0, step, kx, lrc, ldo, half;
        bool packed;
        __device__ __forceinline__ void st(int r, V v) const {
            cg::cluster_group cl = cg::this_cluster();
            const int y = i0 + r * step;
            const int q = y >> lrc, ly = y & ((1 << lrc) - 1);
            V* d = cl.map_shared_rank(s_own, q) + ly * ldo;
            if (packed) {
                V a, b;
                a.x = v.x; a.y = 0;
                b.x = v.y; b.y = 0;
                d[0] = a;
                d[half] = b;
            } else {
                d[kx] = v;
            }
        }
    };
    __device__ __forceinline__ Walk walk(int l, int i0, int step) const {
        return {s_own, i0, step, col0 + l, lrc, ldo, half, packed && l == 0};
    }
};

// F0: beta holds the stage-1 rhs; the kernel forms F0 = u + dt rhs row by row (dt from the
// instance's clock), writes it back over rhs and transforms it (see r2c_rows_io).
template <typename T, bool F0>
__global__ void __cluster_dims__(PLANE_C, 1, 1) __launch_bounds__(ROW_THREADS, 3)
k_plane_fwd(const InstDev* __restrict__ insts, int n_inst, const int* __restrict__ pre, const T* beta,
            typename VecOf<T>::type* spec, const typename VecOf<T>::type* __restrict__ tw,
            double* rowsum, T* f0w, const T* u, const InstClock* clk) {
    typedef typename VecOf<T>::type V;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    cg::cluster_group cl = cg::this_cluster();
    pdl_wait();
    cl.sync();   // every block of the cluster runs before any stores into another
    const int ii = find_instance(pre, n_inst, blockIdx.x);
    const InstDev& I = insts[ii];
    const int lb = blockIdx.x - pre[ii];
    const int rank = (int)cl.block_rank();
    const int q = lb / PLANE_C;              // o * n0 + z
    const int o = q / I.n0, z = q - o * I.n0;
    const PlaneGeom g = plane_geom(I, sizeof(V));
    const int N = I.nl, n1 = I.n1, W = g.W, lgw = g.lgw, P = g.P;
    V* s_line = reinterpret_cast<V*>(smem_raw);            // line buffer, then the axis-1 scratch tile
    V* s_col = reinterpret_cast<V*>(smem_raw + g.a);
    V* tws = reinterpret_cast<V*>(smem_raw + g.a + g.b);
    RowPtr* rt = reinterpret_cast<RowPtr*>(smem_raw + g.a + g.b + g.tw);
    const int tid = threadIdx.x, nt = blockDim.x;
    const long long nrows = 6LL * I.rows, npairs = nrows / 2;
    const long long plane_row = (long long)o * I.rows + (long long)z * n1;   // first row of the plane
    const long long row0 = plane_row + (long long)rank * g.Rc;
    const long long p0 = row0 / 2;
    const int lbv = (int)(p0 / P);           // the row pass's block index of these rows
    for (int r = tid; r < 2 * P; r += nt) {
        const T *pa, *qa;
        src_rows(I, beta, RS_SYM, row0 + r, pa, qa);
        RowPtr e;
        e.p = pa - beta;
        e.q = qa - beta;
        rt[r] = e;
    }
    stage_tw_to_smem(I.lp_last, tw, tws, tid, nt);
    __syncthreads();
    {
        const LinePlan& lq = I.lp_last;
        const V* tw1 = tws + (lq.twst[1] - lq.twst[0]);
        constexpr bool MEAN64 = sizeof(T) == 4;
        const T dt = F0 ? (T)clk[ii].dt : (T)0;
        const PlaneColSink<V> sink{s_col, rank * g.Rc, lgw, N / 2};
#define CDD_PLANE_R2C(A, B)                                                                                 \
        r2c_rows_io<T, MEAN64, A, B, F0>(I, lbv, P, g.ld, rt, beta, s_line, tw1, sink, rowsum, nrows, npairs, \
                                         tid, nt, p0, f0w, u, dt)
        if (lq.radix[0] == 16 && lq.radix[1] == 16) CDD_PLANE_R2C(16, 16);
        else if (lq.radix[0] == 16 && lq.radix[1] == 8) CDD_PLANE_R2C(16, 8);
        else if (lq.radix[0] == 16 && lq.radix[1] == 4) CDD_PLANE_R2C(16, 4);
        else CDD_PLANE_R2C(8, 4);
#undef CDD_PLANE_R2C
    }
    cl.sync();   // every half-spectrum bin of the plane is in its owner's S_col
    SColT<V, 1> col{s_col, lgw, 0}, scr{s_line, lgw, 0};
    fft_io<V, false, 1>(col, scr, col, lgw, I.lp_mid, tw, tid, nt, 0);
    V* dst = spec + I.spoff + plane_row * I.nhp;
    for (int e = tid; e < n1 * W; e += nt) {
        const int ky = e >> lgw, w = e & (W - 1);
        const V v = s_col[e];
        V* d = dst + (long long)ky * I.nhp;
        if (rank == 0 && w == 0) {
            const int km = (ky == 0) ? 0 : n1 - ky;
            const V zm = s_col[km << lgw];
            V a, b;
            a.x = (T)0.5 * (v.x + zm.x);
            a.y = (T)0.5 * (v.y - zm.y);
            b.x = (T)0.5 * (v.y + zm.y);
            b.y = (T)-0.5 * (v.x - zm.x);
            d[0] = a;
            d[N / 2] = b;
        } else {
            d[rank * W + w] = v;
        }
    }
}

template <typename T>
__global__ void __cluster_dims__(PLANE_C, 1, 1) __launch_bounds__(ROW_THREADS, 3)
k_plane_inv(const InstDev* __restrict__ insts, int n_inst, const int* __restrict__ pre,
            const typename VecOf<T>::type* spec, T* out,
            const typename VecOf<T>::type* __restrict__ tw, const double* sbar) {
    typedef typename VecOf<T>::type V;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    cg::cluster_group cl = cg::this_cluster();
    pdl_wait();
    cl.sync();   // every block of the cluster runs before any stores into another
    const int ii = find_instance(pre, n_inst, blockIdx.x);
    const InstDev& I = insts[ii];
    const int lb = blockIdx.x - pre[ii];
    const int rank = (int)cl.block_rank();
    const int q = lb / PLANE_C;
    const int o = q / I.n0, z = q - o * I.n0;
    const PlaneGeom g = plane_geom(I, sizeof(V));
    const int N = I.nl, n1 = I.n1, lgw = g.lgw, ldo = g.ldo, P = g.P;
    V* s_own = reinterpret_cast<V*>(smem_raw);
    V* s_buf = reinterpret_cast<V*>(smem_raw + g.a);      // axis-1 scratch tile, then the C2R line buffer
    V* tws = reinterpret_cast<V*>(smem_raw + g.a + g.b);
    RowPtr* rt = reinterpret_cast<RowPtr*>(smem_raw + g.a + g.b + g.tw);
    RowPtr* re = rt + 2 * P;
    double* rmean = reinterpret_cast<double*>(re + 2 * P);
    const int tid = threadIdx.x, nt = blockDim.x;
    const long long nrows = 6LL * I.rows, npairs = nrows / 2;
    const long long plane_row = (long long)o * I.rows + (long long)z * n1;
    const long long row0 = plane_row + (long long)rank * g.Rc;
    const long long p0 = row0 / 2;
    const int lbv = (int)(p0 / P);
    constexpr bool MEAN64 = sizeof(T) == 4;
    for (int r = tid; r < 2 * P; r += nt) {
        T *pd, *qd;
        dst_rows(I, out, RD_STRESS, row0 + r, pd, qd);
        RowPtr e, ep;
        e.p = pd - out;
        e.q = qd - out;
        ep.p = ep.q = -1;
        rt[r] = e;
        re[r] = ep;
        rmean[r] = MEAN64 ? mean_stress(I, sbar + 9 * ii, o) : 0.0;
    }
    stage_tw_to_smem(I.lp_last, tw, tws, tid, nt);
    {
        const PlaneSpecIn<V> in{spec + I.spoff + plane_row * I.nhp + rank * g.W, I.nhp, n1, N / 2, rank == 0};
        const PlaneRowOut<V> rows{s_own, rank * g.W, 31 - __clz(g.Rc), ldo, N / 2, rank == 0};
        SColT<V, 1> scr{s_buf, lgw, 0};
        fft_io<V, true, 1>(in, scr, rows, lgw, I.lp_mid, tw, tid, nt, 0);
    }
    cl.sync();   // every row of every block's S_own is complete; no block reads the scratch tiles
    {
        const LinePlan& lq = I.lp_last;
        const V* tw1 = tws + (lq.twst[1] - lq.twst[0]);
#define CDD_PLANE_C2R(A, B)                                                                                   \
        c2r_rows_io<T, MEAN64, A, B>(I, lbv, P, g.ld, rt, re, rmean, s_own, s_buf, tw1, out, nullptr, EPI_NONE, \
                                     nrows, npairs, tid, nt, p0, ldo)
        if (lq.radix[0] == 16 && lq.radix[1] == 16) CDD_PLANE_C2R(16, 16);
        else if (lq.radix[0] == 16 && lq.radix[1] == 8) CDD_PLANE_C2R(16, 8);
        else if (lq.radix[0] == 16 && lq.radix[1] == 4) CDD_PLANE_C2R(16, 4);
        else CDD_PLANE_C2R(8, 4);
#undef CDD_PLANE_C2R
    }
}

// ------------------------------------------------------------------------------------------
// Host launch sequence
// ------------------------------------------------------------------------------------------
// u != null: beta holds the stage-1 rhs and the stress is that of F0 = u + dt rhs, formed in place
// first: by the plane instances' forward pass while it transforms the rows (fused), by the axpy
// kernel for the others (it skips the plane instances). A fused F0 in the separate row pass was
// measured slower: its write-back of F0 orders each row load after the previous store.
static cudaError_t run_stress(const PlanCore& P, const void* beta, void* sigma, void* phi, cudaStream_t st,
                              const void* u = nullptr) {
    const bool f32 = (P.precision == CDD_F32);
    float2* spec = (float2*)P.d_spec;             // FP32 plane passes
    const float2* tw = (const float2*)P.d_tw;
    // instances with the fused plane passes (FP32 only) skip the separate row and axis-1 passes
    const bool plane = f32 && P.plane.blocks > 0;
    const LaunchShape* LR = plane ? P.rest : P.pass;
    if (u && LR[PASS_R2C].blocks > 0) {   // the other instances form F0 with the axpy kernel first
        cudaError_t e = launch_axpy_f0(P, u, const_cast<void*>(beta), st);
        if (e != cudaSuccess) return e;
    }
    if (plane && u)
        launch_pdl(k_plane_fwd<float, true>, P.plane.blocks, P.plane.threads, P.plane.smem, st, 
            P.d_inst, P.n_inst, P.plane.d_pre, (const float*)beta, spec, tw, P.d_rowsum, (float*)beta, (const float*)u,
            P.d_clock);
    else if (plane)
        launch_pdl(k_plane_fwd<float, false>, P.plane.blocks, P.plane.threads, P.plane.smem, st, 
            P.d_inst, P.n_inst, P.plane.d_pre, (const float*)beta, spec, tw, P.d_rowsum, nullptr, nullptr, nullptr);
    if (LR[PASS_R2C].blocks > 0) launch_r2c(P, LR[PASS_R2C], beta, f32 ? P.d_rowsum : nullptr, RS_SYM, 6, st);
    launch_mid(P, LR[PASS_MID_F], false, 6, 0, st);
    launch_green(P, P.pass[PASS_GREEN], 0, f32, P.d_k, phi, nullptr, st);
    launch_mid(P, LR[PASS_MID_I], true, 6, 0, st);
    if (plane)
        launch_pdl(k_plane_inv<float>, P.plane.blocks, P.plane.threads, P.plane.smem, st, 
            P.d_inst, P.n_inst, P.plane.d_pre, spec, (float*)sigma, tw, P.d_sbar);
    if (LR[PASS_C2R].blocks > 0) launch_c2r(P, LR[PASS_C2R], sigma, f32, RD_STRESS, 6, nullptr, EPI_NONE, st);
    return cudaGetLastError();
}

// Adjoint (gmode 1: stress cotangent, 6 components in stress layout -> beta cotangent, written to all
// 9 components of a field) and the nu-derivative of the stress (gmode 2: beta -> 6 components).
// Both keep the k = 0 mode in the transforms (no FP64 mean path).
static cudaError_t run_stress_variant(const PlanCore& P, int gmode, const void* in, void* out, const void* phi, double* part,
                                      cudaStream_t st) {
    const LaunchShape* L = P.pass;
    launch_r2c(P, L[PASS_R2C], in, nullptr, gmode == 1 ? RS_STRESS : RS_SYM, 6, st);
    launch_mid(P, L[PASS_MID_F], false, 6, 0, st);
    launch_green(P, L[PASS_GREEN], gmode, false, P.d_k, const_cast<void*>(phi), part, st);
    launch_mid(P, L[PASS_MID_I], true, 6, 0, st);
    launch_c2r(P, L[PASS_C2R], out, false, gmode == 1 ? RD_SYM_FIELD : RD_STRESS, 6, nullptr, EPI_NONE, st);
    return cudaGetLastError();
}

cudaError_t launch_stress_adjoint(const PlanCore& P, const void* sigbar6, void* betabar9, cudaStream_t st,
                                  const void* phi, double* part) {
    return run_stress_variant(P, 1, sigbar6, betabar9, phi, part, st);
}

cudaError_t launch_stress_dnu(const PlanCore& P, const void* beta, void* out6, cudaStream_t st) {
    return run_stress_variant(P, 2, beta, out6, nullptr, nullptr, st);
}

// Vacancy diffusion: the concentrations of the vacancy instances (one component) forward, times
// exp(-gamma dt kSq) in the axis-0 pass, inverse, written back for the instances whose step was
// applied. The stress passes' launch shapes carry it (blocks past one component exit).
cudaError_t launch_vacancy_diffusion(const PlanCore& P, cudaStream_t st) {
    const LaunchShape* L = P.pass;
    launch_r2c(P, L[PASS_R2C], P.d_vac, nullptr, RS_VAC, 1, st);
    launch_mid(P, L[PASS_MID_F], false, 1, 1, st);
    launch_green(P, L[PASS_GREEN], 7, false, P.d_k, nullptr, nullptr, st);
    launch_mid(P, L[PASS_MID_I], true, 1, 1, st);
    launch_c2r(P, L[PASS_C2R], P.d_vac, false, RD_VAC, 1, nullptr, EPI_NONE, st);
    return cudaGetLastError();
}

// k-space observables: forward transforms of sym(beta) (6 components, the stress passes' launch
// shapes) or of all 9 components (the 9-component shapes), the observable's k-space operator in the
// fused axis-0 pass, inverse transforms of its 9 or 3 components with the real-space epilogue.
// No FP64 mean path: every operator's k = 0 mode is zero (kmask, or a factor k).
cudaError_t launch_observable(const PlanCore& P, int kind, const void* beta, void* out, cudaStream_t st,
                              bool sin_k) {
    int gmode, epi;
    switch (kind) {
        case CDD_OBS_BETA_ELASTIC: gmode = 3; epi = EPI_BETA_E; break;
        case CDD_OBS_ROTATION: gmode = 4; epi = EPI_ROTATION; break;
        case CDD_OBS_RODRIGUES: gmode = 5; epi = EPI_RODRIGUES; break;
        case CDD_OBS_RHO: gmode = 6; epi = EPI_NONE; break;
        case CDD_OBS_RODRIGUES_RHO: gmode = 8; epi = EPI_NONE; break;
        default: return cudaErrorInvalidValue;
    }
    const int nin = green_nin(gmode), nout = green_nout(gmode);
    const LaunchShape* LI = (nin == 9) ? P.pass9 : P.pass;
    const LaunchShape* LO = (nout == 9) ? P.pass9 : P.pass;
    const size_t elt = P.precision == CDD_F32 ? sizeof(float) : sizeof(double);
    launch_r2c(P, LI[PASS_R2C], beta, nullptr, nin == 9 ? RS_FULL : RS_SYM, nin, st);
    launch_mid(P, LI[PASS_MID_F], false, nin, 0, st);
    launch_green(P, P.pass9[PASS_GREEN], gmode, false, (const char*)P.d_k + (sin_k ? P.ksin_off * elt : 0), nullptr, nullptr, st);
    launch_mid(P, LO[PASS_MID_I], true, nout, 0, st);
    launch_c2r(P, LO[PASS_C2R], out, false, nout == 9 ? RD_FIELD9 : RD_FIELD3, nout, beta, epi, st);
    return cudaGetLastError();
}

cudaError_t launch_stress(const PlanCore& P, const void* beta, void* sigma, cudaStream_t st, void* phi) {
    return run_stress(P, beta, sigma, phi, st);
}

cudaError_t launch_stress_f0(const PlanCore& P, const void* u, void* rhs_f0, void* sigma, cudaStream_t st,
                             void* phi) {
    return run_stress(P, rhs_f0, sigma, phi, st, u);
}

cudaError_t stress_set_attributes(int precision, size_t smem) {
    cudaError_t e;
    if (precision == CDD_F32) {
        if ((e = set_dyn_smem_limit(k_plane_fwd<float, false>, smem))) return e;
        if ((e = set_dyn_smem_limit(k_plane_fwd<float, true>, smem))) return e;
        if ((e = set_dyn_smem_limit(k_plane_inv<float>, smem))) return e;
    }
    if ((e = r2c_set_attributes(precision, smem))) return e;
    if ((e = c2r_set_attributes(precision, smem))) return e;
    if ((e = mid_set_attributes(precision, smem))) return e;
    return green_set_attributes(precision, smem);
}

}  // namespace cdd
