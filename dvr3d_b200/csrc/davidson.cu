// davidson.cu -- block-Davidson for a few lowest levels of the assembled contracted
// Hamiltonian, preconditioned by its channel blocks (optionally with the learned correction),
// judged by FP64 residuals; and the trainer of the learned correction.
//
// The reference diagonalises the final Hamiltonian completely (diag3d -> dsyev,
// :2661-2764) even when NEVAL is small. For a few levels no factorisation is needed:
//   basis V (orthonormal, m <= 3 b columns), HV = H3 V (DMMA GEMM with the assembled H3)
//   -> Rayleigh-Ritz (G = V^T HV, shared-memory eigensolver) -> Ritz pairs, FP64 residuals
//   -> converged when every wanted pair satisfies rho^2 / gap <= tol
//   -> corrections t = P(r, theta) from the channel blocks (learned_precond.cuh)
//   -> classical Gram-Schmidt against V twice, Cholesky-QR twice, appended; thick restart
//      to the 2 b leading Ritz vectors when the basis is full.
// In training mode the solver records (residual, theta, basis) snapshots of the wanted pairs;
// after convergence the ideal corrections e = (x_final - x) outside the basis of that moment
// are formed and the network is fitted to them on the device (Adam, full batch).
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <numeric>
#include <string>
#include <vector>

#include "chol.cuh"
#include "common.cuh"
#include "eig_batched.cuh"
#include "gemm64.cuh"
#include "learned_precond.cuh"
#include "pipeline.cuh"
#include "tc_gemm.cuh"

#define CK(x)                                          \
    do {                                               \
        cudaError_t e_ = (x);                          \
        if (e_ != cudaSuccess) throw CudaFail{e_, #x}; \
    } while (0)

namespace dvr3d {

namespace {

constexpr int kBatchedRR = 160;  // Rayleigh-Ritz matrices up to this order go to the batched eigensolver


// R[:, j] = HX[:, j] - w_j X[:, j], rn[j] = ||R[:, j]||; one CTA per column
__global__ void residual_kernel(const double *X, const double *HX, long long ld, const double *w, int N, double *R,
                                double *rn) {
    const int j = blockIdx.x;
    const double wj = w[j];
    double s = 0.0;
    for (int i = threadIdx.x; i < N; i += blockDim.x) {
        const double r = HX[(size_t)j * ld + i] - wj * X[(size_t)j * ld + i];
        R[(size_t)j * ld + i] = r;
        s += r * r;
    }
    __shared__ double red[32];
    s = block_sum(s, red);
    if (threadIdx.x == 0) rn[j] = sqrt(s);
}

// E[:, j] = sign(xf_j . xs_j) xf_j - xs_j; one CTA per column
__global__ void ideal_correction_kernel(const double *XF, const double *XS, long long ld, int N, double *E) {
    const int j = blockIdx.x;
    const double *xf = XF + (size_t)j * ld, *xs = XS + (size_t)j * ld;
    double s = 0.0;
    for (int i = threadIdx.x; i < N; i += blockDim.x) s += xf[i] * xs[i];
    __shared__ double red[32];
    s = block_sum(s, red);
    const double sg = (s < 0.0) ? -1.0 : 1.0;
    for (int i = threadIdx.x; i < N; i += blockDim.x) E[(size_t)j * ld + i] = sg * xf[i] - xs[i];
}

// Column norms of T (one CTA per column); columns whose norm is below rel * max(norm_ref)
// are replaced by a deterministic pseudo-random vector, the others scaled to unit norm.
__global__ void colnorm_kernel(const double *T, long long ld, int N, double *nrm) {
    const int j = blockIdx.x;
    double s = 0.0;
    for (int i = threadIdx.x; i < N; i += blockDim.x) s += T[(size_t)j * ld + i] * T[(size_t)j * ld + i];
    __shared__ double red[32];
    s = block_sum(s, red);
    if (threadIdx.x == 0) nrm[j] = sqrt(s);
}

__global__ void normalize_or_refill_kernel(double *T, long long ld, int N, const double *nrm, const double *ref,
                                           double rel, unsigned seed) {
    const int j = blockIdx.x;
    const double nj = nrm[j], thr = rel * ref[j];
    const bool refill = !(nj > thr) || !isfinite(nj);
    const double inv = refill ? 0.0 : 1.0 / nj;
    for (int i = threadIdx.x; i < N; i += blockDim.x) {
        double v = T[(size_t)j * ld + i] * inv;
        if (refill) {
            unsigned x = (unsigned)i * 2654435761u ^ (seed + 7919u * (unsigned)j);
            x ^= x >> 16;
            x *= 0x7feb352dU;
            x ^= x >> 15;
            x *= 0x846ca68bU;
            x ^= x >> 16;
            v = ((double)(x & 0xffffff) / 8388608.0 - 1.0) / sqrt((double)N);
        }
        T[(size_t)j * ld + i] = v;
    }
}

// V[:, j] = channel mode j of the start block, embedded (zero outside its channel)
__global__ void embed_modes_kernel(ChanPrec cp, const int *mode_ch, const int *mode_q, double *V, long long ld,
                                   int N) {
    const int j = blockIdx.x;
    const int c = mode_ch[j], q = mode_q[j], n = cp.n[c], off = cp.off[c];
    double *v = V + (size_t)j * ld;
    for (int i = threadIdx.x; i < N; i += blockDim.x) v[i] = 0.0;
    __syncthreads();
    const double *Q = cp.Q + cp.qoff[c] + (size_t)q * n;
    for (int p = threadIdx.x; p < n; p += blockDim.x) v[cp.idx[off + p]] = Q[p];
}

inline unsigned nb256(long long n) { return (unsigned)((n + 255) / 256); }
inline long long rup(long long x, long long m) { return (x + m - 1) / m * m; }

void copy_cols(double *dst, long long ldd, const double *src, long long lds, int N, int ncol, cudaStream_t st) {
    if (ncol <= 0) return;
    CK(cudaMemcpy2DAsync(dst, ldd * sizeof(double), src, lds * sizeof(double), (size_t)N * sizeof(double), ncol,
                         cudaMemcpyDeviceToDevice, st));
}

int split_for(int M, int N, int K, int target) {
    const int tiles = ((M + 63) / 64) * ((N + 63) / 64);
    const int s = std::max(1, std::min({(target + tiles - 1) / tiles, 64, (K + 15) / 16}));
    return (s > 8 && tiles * 8 >= 296) ? 8 : s;
}

void gemm_split(GemmOp g, int target, double *work, cudaStream_t st) {
    if (target > 1) {
        g.splitk = split_for(g.M, g.N, g.K, target);
        g.work = work;
    }
    CK(launch_gemm(g, st));
}

void lp_init_weights(std::vector<double> &w) {
    // deterministic small initial weights (fan-in scaled), zero output layer
    w.assign(kLpParams, 0.0);
    unsigned long long s = 0x243f6a8885a308d3ull;
    auto u = [&]() {
        s = s * 6364136223846793005ull + 1442695040888963407ull;
        return (double)(s >> 11) / 9007199254740992.0 * 2.0 - 1.0;
    };
    for (int p = 0; p < kLpHidden * kLpFeat; ++p) w[p] = u() / std::sqrt((double)kLpFeat);
    const int o2 = kLpHidden * kLpFeat + kLpHidden;
    for (int p = 0; p < kLpHidden * kLpHidden; ++p) w[o2 + p] = u() / std::sqrt((double)kLpHidden);
}

}  // namespace

// ---------------------------------------------------------------- training loss / gradient
double lp_train_loss(dvr3d_ctx *ctx, const double *w, double *grad) {
    auto &S = ctx->lp_set;
    if (!S.valid) throw HostError{DVR3D_ERR_ARG, "no recorded training pairs (solve with learned_precond = 2 first)"};
    cudaStream_t st = ctx->stream;
    const int N = S.N, P = S.npair, nw = S.nwant;
    const long long ld = S.ld;
    auto A = [&](const std::string &nm, size_t n) { return ctx->arena.get_t<double>(nm, n); };
    const double *R = A("lp_R", ld * P), *E = A("lp_E", ld * P), *th = A("lp_theta", P);
    double *T = A("lp_T", ld * P), *PT = A("lp_PT", ld * P), *G = A("lp_G", ld * P);
    double *zraw = A("lp_zraw", (size_t)N * P), *delta = A("lp_delta", (size_t)N * P);
    const size_t msnap = (size_t)*std::max_element(S.snap_m.begin(), S.snap_m.end());
    double *proj = A("lp_proj", msnap * nw);
    double *sums = A("lp_sums", 3 * (size_t)P), *coef = A("lp_coef", 2 * (size_t)P), *loss = A("lp_loss", 8);
    double *work = A("lp_gwork", std::max({lp_grad_work_doubles(), (size_t)64 * msnap * nw, (size_t)1 << 22}));
    CK(launch_chan_apply(S.cp, w, R, ld, th, P, T, ld, zraw, st));
    copy_cols(PT, ld, T, ld, N, P, st);
    for (size_t s = 0; s < S.snap_m.size(); ++s) {
        const int m = S.snap_m[s];
        const double *V = A("lp_V" + std::to_string(s), ld * m);
        GemmOp c;  // proj = V^T T_s ; PT_s -= V proj
        c.M = m;
        c.N = nw;
        c.K = N;
        c.A = V;
        c.lda = ld;
        c.ta = true;
        c.B = T + (size_t)s * nw * ld;
        c.ldb = ld;
        c.C = proj;
        c.ldc = m;
        gemm_split(c, 600, work, st);
        GemmOp u;
        u.M = N;
        u.N = nw;
        u.K = m;
        u.alpha = -1.0;
        u.beta = 1.0;
        u.A = V;
        u.lda = ld;
        u.B = proj;
        u.ldb = m;
        u.C = PT + (size_t)s * nw * ld;
        u.ldc = ld;
        gemm_split(u, 0, work, st);
    }
    CK(launch_lp_pair_terms(T, PT, E, ld, N, P, sums, coef, loss, st));
    if (grad) {
        CK(launch_lp_dldt(E, PT, ld, N, P, coef, G, st));
        CK(launch_chan_back(S.cp, G, ld, zraw, P, delta, st));
        CK(lp_mlp_grad(S.cp.modes, w, th, P, delta, grad, work, st));
    }
    double lh = 0.0;
    CK(cudaMemcpyAsync(&lh, loss, sizeof(double), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    return lh;
}

// ---------------------------------------------------------------- Davidson
bool davidson_solve(dvr3d_ctx *ctx, const H3Op &op, const Contracted &C, const dvr3d_options &opt, int nwant,
                    int mode, double *lp_w, double *wv_dev, std::vector<double> &rn_host, double *evec_dev,
                    DavidsonStats &stats) {
    cudaStream_t st = ctx->stream;
    const int N = C.N;
    const bool split = (op.H3 == nullptr);
    if (split ? (!op.hi || !op.lo) : (op.ldh & 1)) return false;
    int bs = nwant <= kDavidsonMaxLevels ? std::min(kDavidsonMaxBlock, nwant + std::max(8, nwant / 2))
                                         : nwant + std::max(16, nwant / 4);
    bs += (bs & 1);
    const int keep = 2 * bs, mmax = 3 * bs;
    if (mmax >= N) return false;
    const bool big_rr = mmax > kBatchedRR;  // Rayleigh-Ritz on the dense eigensolver
    const double tolE = (opt.tol_cm > 0.0 ? opt.tol_cm : 1.0e-4) / 2.19474624e5;
    const int max_iter = opt.max_iter > 0 ? opt.max_iter : 300;
    const long long ld = rup(N, 8);
    auto A = [&](const std::string &nm, size_t n) { return ctx->arena.get_t<double>(nm, n); };
    double *V = A("dv_V", ld * mmax), *HV = A("dv_HV", ld * mmax);
    double *V2 = A("dv_V2", ld * keep), *HV2 = A("dv_HV2", ld * keep);
    double *X = A("dv_X", ld * bs), *HX = A("dv_HX", ld * bs), *R = A("dv_R", ld * bs), *Tc = A("dv_T", ld * bs);
    const long long ldg_max = big_rr ? rup(mmax, 8) : mmax;
    double *G = A("dv_G", (size_t)ldg_max * mmax), *Y = A("dv_Y", (size_t)mmax * mmax), *th = A("dv_th", mmax);
    double *rn = A("dv_rn", bs), *proj = A("dv_proj", (size_t)mmax * bs);
    double *Gb = A("dv_Gb", 64 * 64), *Gi = A("dv_Gi", 64 * 64);
    double *cn0 = A("dv_cn0", bs), *cn1 = A("dv_cn1", bs), *ones = A("dv_ones", bs);
    {
        std::vector<double> o(bs, 1.0);
        CK(cudaMemcpyAsync(ones, o.data(), sizeof(double) * bs, cudaMemcpyHostToDevice, st));
        CK(cudaStreamSynchronize(st));
    }
    // partial sums of the split products: H3 V and the projections by any block of columns, V^T HV
    // at any basis size (below about 2300 rows H3 V splits more than sixteen ways)
    size_t wk = 0;
    std::vector<int> widths{bs};  // a split depends on the width only through its 64-column tiles
    for (int c = 64; c < bs; c += 64) widths.push_back(c);
    for (int c : widths) wk = std::max(wk, gemm_splitk_work(N, c, split_for(N, c, N, 600)));
    for (int q = 1; q <= mmax; ++q) {
        wk = std::max(wk, gemm_splitk_work(q, q, split_for(q, q, N, 600)));
        for (int c : widths) wk = std::max(wk, gemm_splitk_work(q, c, split_for(q, c, N, 600)));
    }
    wk = std::max(wk, gemm_splitk_work(64, 64, 64));  // Cholesky-QR of 64 columns
    double *work = A("dv_work", wk);
    int *err = ctx->arena.get_t<int>("dv_err", 3);
    CK(cudaMemsetAsync(err, 0, 3 * sizeof(int), st));
    // Rayleigh-Ritz eigensolver of the small path: the batched solver's kernels on one block
    // (descriptor: n, selected count, zld as ints; aoff, voff, zoff as zeros)
    int *rr_int = ctx->arena.get_t<int>("dv_rri", 4);
    long long *rr_zero = ctx->arena.get_t<long long>("dv_rrz", 1);
    double *rr_a = big_rr ? nullptr : A("dv_rra", (size_t)mmax * mmax);
    double *rr_d = A("dv_rrd", mmax), *rr_e = A("dv_rre", mmax), *rr_tau = A("dv_rrt", mmax);
    CK(cudaMemsetAsync(rr_zero, 0, sizeof(long long), st));
    // BF16 slices of the vectors multiplied on the tensor cores (split form)
    const long long ldvb = rup(N, 8);
    __nv_bfloat16 *vb_hi = nullptr, *vb_lo = nullptr;
    if (split) {
        vb_hi = ctx->arena.get_t<__nv_bfloat16>("dv_vbh", (size_t)ldvb * mmax);
        vb_lo = ctx->arena.get_t<__nv_bfloat16>("dv_vbl", (size_t)ldvb * mmax);
    }
    // channel blocks; the start block is the bs lowest channel modes (approximate
    // eigenvectors of H3 in which the coupling between channels is left out)
    ChanPrec cp;
    std::vector<double> lam;
    std::vector<int> mch;
    channel_setup(ctx, op, C, cp, &lam, &mch);
    {
        std::vector<int> order(N);
        std::iota(order.begin(), order.end(), 0);
        std::partial_sort(order.begin(), order.begin() + bs, order.end(),
                          [&](int a, int b) { return lam[a] < lam[b]; });
        std::vector<int> mc(bs), mq(bs);
        for (int j = 0; j < bs; ++j) {
            const int m0 = order[j], c = mch[m0];
            int first = m0;
            while (first > 0 && mch[first - 1] == c) --first;
            mc[j] = c;
            mq[j] = m0 - first;
        }
        int *dmc = ctx->arena.get_t<int>("dv_mc", bs), *dmq = ctx->arena.get_t<int>("dv_mq", bs);
        CK(cudaMemcpyAsync(dmc, mc.data(), sizeof(int) * bs, cudaMemcpyHostToDevice, st));
        CK(cudaMemcpyAsync(dmq, mq.data(), sizeof(int) * bs, cudaMemcpyHostToDevice, st));
        note_h2d(2 * sizeof(int) * bs);
        CK(cudaMemsetAsync(V, 0, sizeof(double) * ld * bs, st));
        DVR3D_COUNT_LAUNCH(1);
        embed_modes_kernel<<<bs, 256, 0, st>>>(cp, dmc, dmq, V, ld, N);
        CK(cudaGetLastError());
        CK(cudaStreamSynchronize(st));
    }
    // Rayleigh-Ritz eigensolve of G (m x m, ldg): eigenvalues w (ascending), eigenvectors Z
    // (ld m; at least the `keep` lowest)
    auto rr_eig = [&](double *Gm, long long ldg, int m, double *w, double *Z) {
        if (big_rr) {
            dense_lowest(ctx, Gm, ldg, m, std::min(m, keep), true, w, Z, m, "dvrr_", false, nullptr);
            return;
        }
        // tridiagonalisation, all m eigenvalues by bisection, the keep lowest eigenvectors by
        // inverse iteration and a blocked back-transformation (eig_batched.cuh)
        const int nsel = std::min(m, keep);
        const int hi[3] = {m, nsel, m};
        CK(cudaMemcpyAsync(rr_int, hi, sizeof(hi), cudaMemcpyHostToDevice, st));
        CK(cudaMemcpy2DAsync(rr_a, sizeof(double) * m, Gm, sizeof(double) * ldg, sizeof(double) * m, m,
                             cudaMemcpyDeviceToDevice, st));
        BatchDesc bd{1, rr_int, rr_zero, rr_zero};
        launch_symmetrize_lower(bd, rr_a, m, st);
        launch_tridiag_batched(bd, rr_a, rr_d, rr_e, rr_tau, m, st);
        launch_eigvals_batched(bd, rr_d, rr_e, w, rr_int + 3, 0, 0.0, st);
        launch_eigvecs_batched(bd, rr_a, rr_d, rr_e, rr_tau, w, rr_int + 1, rr_zero, rr_int + 2, Z, m, err, st);
        CK(cudaGetLastError());
    };
    // HV[:, c0:c0+nc] = H3 V[:, c0:c0+nc]: BF16x3 tensor-core GEMM (split form, phase 1), the
    // matrix-free FP64 operator (split form, residual correction), or the FP64 DMMA GEMM
    int phase = split ? 1 : 2;
    auto hv_product = [&](int c0, int nc) {
        if (nc <= 0) return;
        if (split && phase == 1) {
            CK(launch_split_bf16(V + (size_t)c0 * ld, ld, nc, N, vb_hi, vb_lo, ldvb, st));
            TcGemm g;
            g.M = N;
            g.N = nc;
            g.K = N;
            g.nslice = 2;
            g.A_hi = op.hi;
            g.A_lo = op.lo;
            g.lda = op.ld;
            g.B_hi = vb_hi;
            g.B_lo = vb_lo;
            g.ldb = ldvb;
            g.C = HV + (size_t)c0 * ld;
            g.cm = 1;
            g.cn = ld;
            g.err = err + 2;
            CK(launch_tc_gemm(g, st));
            stats.low_matvecs += nc;
        } else if (split) {
            apply_h3_fp64(ctx, C, V + (size_t)c0 * ld, ld, nc, HV + (size_t)c0 * ld, ld);
        } else {
            GemmOp hv;
            hv.M = N;
            hv.N = nc;
            hv.K = N;
            hv.A = op.H3;
            hv.lda = op.ldh;
            hv.B = V + (size_t)c0 * ld;
            hv.ldb = ld;
            hv.C = HV + (size_t)c0 * ld;
            hv.ldc = ld;
            gemm_split(hv, 600, work, st);
        }
        stats.matvecs += nc;
    };
    // orthonormalise Tb (N x nb, nb <= 64) in place: Cholesky-QR twice
    auto cholqr = [&](double *Tb, int nb) {
        for (int pass = 0; pass < 2; ++pass) {
            GemmOp q;
            q.M = nb;
            q.N = nb;
            q.K = N;
            q.A = Tb;
            q.lda = ld;
            q.ta = true;
            q.B = Tb;
            q.ldb = ld;
            q.C = Gb;
            q.ldc = nb;
            gemm_split(q, 256, work, st);
            CK(launch_chol_small(Gb, nb, Gi, 1.0e-24, err + 1, st));
            GemmOp s2;
            s2.M = N;
            s2.N = nb;
            s2.K = nb;
            s2.A = Tb;
            s2.lda = ld;
            s2.B = Gi;
            s2.ldb = 64;
            s2.tb = true;
            s2.C = Tb;
            s2.ldc = ld;
            gemm_split(s2, 0, work, st);
        }
    };
    // Tb -= W (W^T Tb), twice (W: N x nw orthonormal columns)
    auto project_out = [&](const double *W, int nw, double *Tb, int nb) {
        for (int pass = 0; pass < 2; ++pass) {
            GemmOp c;
            c.M = nw;
            c.N = nb;
            c.K = N;
            c.A = W;
            c.lda = ld;
            c.ta = true;
            c.B = Tb;
            c.ldb = ld;
            c.C = proj;
            c.ldc = nw;
            gemm_split(c, 600, work, st);
            GemmOp u;
            u.M = N;
            u.N = nb;
            u.K = nw;
            u.alpha = -1.0;
            u.beta = 1.0;
            u.A = W;
            u.lda = ld;
            u.B = proj;
            u.ldb = nw;
            u.C = Tb;
            u.ldc = ld;
            gemm_split(u, 0, work, st);
        }
    };
    const int max_snaps = 16;
    const char *trace_env = std::getenv("DVR3D_DAV_TRACE");
    const bool trace = trace_env && trace_env[0] == '1';
    std::vector<int> snap_m;
    std::vector<double> snap_theta;
    if (mode == 2) ctx->lp_set.valid = false;
    int m = bs, nnew = bs;
    std::vector<double> thh(mmax), rnh(bs);
    bool done = false;
    double rprev = HUGE_VAL;
    int it = 0;
    for (; it < max_iter; ++it) {
        hv_product(m - nnew, nnew);
        const long long ldg = big_rr ? rup(m, 8) : m;
        GemmOp g;  // G = V^T HV
        g.M = m;
        g.N = m;
        g.K = N;
        g.A = V;
        g.lda = ld;
        g.ta = true;
        g.B = HV;
        g.ldb = ld;
        g.C = G;
        g.ldc = ldg;
        gemm_split(g, 600, work, st);
        rr_eig(G, ldg, m, th, Y);
        GemmOp x;  // X = V Y[:, :bs], HX = HV Y[:, :bs]
        x.M = N;
        x.N = bs;
        x.K = m;
        x.A = V;
        x.lda = ld;
        x.B = Y;
        x.ldb = m;
        x.C = X;
        x.ldc = ld;
        gemm_split(x, 0, work, st);
        x.A = HV;
        x.C = HX;
        gemm_split(x, 0, work, st);
        DVR3D_COUNT_LAUNCH(1);
        residual_kernel<<<bs, 256, 0, st>>>(X, HX, ld, th, N, R, rn);
        CK(cudaGetLastError());
        const int nth = big_rr ? std::min(m, keep) : m;
        int herr[3] = {0, 0, 0};
        CK(cudaMemcpyAsync(thh.data(), th, sizeof(double) * nth, cudaMemcpyDeviceToHost, st));
        CK(cudaMemcpyAsync(rnh.data(), rn, sizeof(double) * bs, cudaMemcpyDeviceToHost, st));
        CK(cudaMemcpyAsync(herr, err, sizeof(herr), cudaMemcpyDeviceToHost, st));
        CK(cudaStreamSynchronize(st));
        note_d2h(sizeof(double) * (nth + bs) + sizeof(herr));
        if (herr[0] != 0 || herr[2] != 0) break;  // Rayleigh-Ritz inverse iteration failed its growth
                                                    // test, or a tensor-core pipeline wait timed
                                                    // out: give up (the caller falls back)
        int nconv = 0;
        double rmax = 0.0;
        for (int j = 0; j < nwant; ++j) {
            double gap = thh[j + 1] - thh[j];
            if (j > 0) gap = std::min(gap, thh[j] - thh[j - 1]);
            const double bound = rnh[j] * rnh[j] / std::max(gap, rnh[j]);
            if (bound <= tolE && std::isfinite(bound)) ++nconv;
            rmax = std::max(rmax, rnh[j]);
        }
        if (trace)
            std::fprintf(stderr, "davidson it %d phase %d m %d converged %d/%d max residual %.3e theta0 %.10f\n", it,
                         phase, m, nconv, nwant, rmax, thh[0]);
        if (phase == 1) {
            ++stats.low_iterations;
            if (nconv == nwant || !(rmax < 0.7 * rprev) || it + 1 >= max_iter / 2) {
                // residual correction: the whole basis multiplied by the FP64 operator; the
                // next pass redoes the Rayleigh-Ritz step with these products
                phase = 2;
                hv_product(0, m);
                nnew = 0;
                continue;
            }
            rprev = rmax;
        } else if (nconv == nwant) {
            done = true;
            break;
        }
        if (mode == 2 && (int)snap_m.size() < max_snaps) {
            const int s = (int)snap_m.size();
            copy_cols(A("lp_X" + std::to_string(s), ld * nwant), ld, X, ld, N, nwant, st);
            copy_cols(A("lp_Rs" + std::to_string(s), ld * nwant), ld, R, ld, N, nwant, st);
            copy_cols(A("lp_V" + std::to_string(s), ld * m), ld, V, ld, N, m, st);
            snap_m.push_back(m);
            snap_theta.insert(snap_theta.end(), thh.begin(), thh.begin() + nwant);
        }
        if (m + bs > mmax) {  // thick restart to the leading Ritz vectors
            GemmOp r;
            r.M = N;
            r.N = keep;
            r.K = m;
            r.A = V;
            r.lda = ld;
            r.B = Y;
            r.ldb = m;
            r.C = V2;
            r.ldc = ld;
            gemm_split(r, 0, work, st);
            r.A = HV;
            r.C = HV2;
            gemm_split(r, 0, work, st);
            copy_cols(V, ld, V2, ld, N, keep, st);
            copy_cols(HV, ld, HV2, ld, N, keep, st);
            m = keep;
        }
        CK(launch_chan_apply(cp, mode == 1 ? lp_w : nullptr, R, ld, th, bs, Tc, ld, nullptr, st));
        // unit columns (corrections of converged pairs are tiny); refill any zero column
        DVR3D_COUNT_LAUNCH(2);
        colnorm_kernel<<<bs, 256, 0, st>>>(Tc, ld, N, cn0);
        normalize_or_refill_kernel<<<bs, 256, 0, st>>>(Tc, ld, N, cn0, ones, 1.0e-300, 17u * it + 1u);
        for (int sweep = 0; sweep < 2; ++sweep) {
            project_out(V, m, Tc, bs);
            // a correction (nearly) inside span(V) would make the block singular: replace it
            // by a random direction and orthogonalise once more
            DVR3D_COUNT_LAUNCH(2);
            colnorm_kernel<<<bs, 256, 0, st>>>(Tc, ld, N, cn1);
            normalize_or_refill_kernel<<<bs, 256, 0, st>>>(Tc, ld, N, cn1, ones, 1.0e-8, 31u * it + 5u + sweep);
        }
        // orthonormal block, 64 columns at a time
        for (int c0 = 0; c0 < bs; c0 += 64) {
            const int nb = std::min(64, bs - c0);
            if (c0 > 0) project_out(Tc, c0, Tc + (size_t)c0 * ld, nb);
            cholqr(Tc + (size_t)c0 * ld, nb);
        }
        int qe = 0;
        CK(cudaMemcpyAsync(&qe, err + 1, sizeof(int), cudaMemcpyDeviceToHost, st));
        CK(cudaStreamSynchronize(st));
        if (qe != 0) break;  // corrections became dependent: give up (the caller falls back)
        copy_cols(V + (size_t)m * ld, ld, Tc, ld, N, bs, st);
        m += bs;
        nnew = bs;
    }
    stats.iterations = it;
    if (!done) return false;
    rn_host.assign(rnh.begin(), rnh.begin() + nwant);
    stats.max_resid = *std::max_element(rn_host.begin(), rn_host.end());
    CK(cudaMemcpyAsync(wv_dev, th, sizeof(double) * nwant, cudaMemcpyDeviceToDevice, st));
    if (evec_dev) copy_cols(evec_dev, N, X, ld, N, nwant, st);
    if (mode == 2 && !snap_m.empty()) {
        // training pairs: e = (x_final - x) outside the basis of the snapshot
        const int P = (int)snap_m.size() * nwant;
        double *RP = A("lp_R", ld * P), *EP = A("lp_E", ld * P), *TP = A("lp_theta", P);
        double *pj = A("lp_proj", (size_t)*std::max_element(snap_m.begin(), snap_m.end()) * nwant);
        for (size_t s = 0; s < snap_m.size(); ++s) {
            const std::string k = std::to_string(s);
            const double *Xs = A("lp_X" + k, ld * nwant), *Vs = A("lp_V" + k, ld * snap_m[s]);
            double *Eq = EP + (size_t)s * nwant * ld;
            DVR3D_COUNT_LAUNCH(1);
            ideal_correction_kernel<<<nwant, 256, 0, st>>>(X, Xs, ld, N, Eq);
            GemmOp c;
            c.M = snap_m[s];
            c.N = nwant;
            c.K = N;
            c.A = Vs;
            c.lda = ld;
            c.ta = true;
            c.B = Eq;
            c.ldb = ld;
            c.C = pj;
            c.ldc = snap_m[s];
            gemm_split(c, 600, work, st);
            GemmOp u;
            u.M = N;
            u.N = nwant;
            u.K = snap_m[s];
            u.alpha = -1.0;
            u.beta = 1.0;
            u.A = Vs;
            u.lda = ld;
            u.B = pj;
            u.ldb = snap_m[s];
            u.C = Eq;
            u.ldc = ld;
            gemm_split(u, 0, work, st);
            copy_cols(RP + (size_t)s * nwant * ld, ld, A("lp_Rs" + k, ld * nwant), ld, N, nwant, st);
        }
        CK(cudaMemcpyAsync(TP, snap_theta.data(), sizeof(double) * P, cudaMemcpyHostToDevice, st));
        CK(cudaStreamSynchronize(st));
        note_h2d(sizeof(double) * P);
        auto &S = ctx->lp_set;
        S.valid = true;
        S.N = N;
        S.nwant = nwant;
        S.npair = P;
        S.ld = ld;
        S.snap_m = snap_m;
        S.cp = cp;
        // fit: Adam, full batch, from the initial weights (zero output layer = exact channel inverse)
        std::vector<double> w0;
        lp_init_weights(w0);
        CK(cudaMemcpyAsync(lp_w, w0.data(), sizeof(double) * kLpParams, cudaMemcpyHostToDevice, st));
        double *grad = A("lp_grad", kLpParams), *mom = A("lp_mom", kLpParams), *vel = A("lp_vel", kLpParams);
        CK(cudaMemsetAsync(mom, 0, sizeof(double) * kLpParams, st));
        CK(cudaMemsetAsync(vel, 0, sizeof(double) * kLpParams, st));
        const int steps = 200;
        for (int s = 1; s <= steps; ++s) {
            const double l = lp_train_loss(ctx, lp_w, grad);
            if (s == 1) stats.loss_first = l;
            CK(lp_adam_step(lp_w, grad, mom, vel, s, 3.0e-3, st));
        }
        stats.loss_last = lp_train_loss(ctx, lp_w, nullptr);
        stats.pairs = P;
        stats.trained = true;
    }
    CK(cudaStreamSynchronize(st));
    return true;
}

}  // namespace dvr3d
