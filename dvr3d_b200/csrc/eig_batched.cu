// eig_batched.cu -- batched FP64 symmetric eigensolver kernels: one or two CTAs a block in the
// reduction, up to eight for the eigenvalues and sixteen for the inverse iteration.
// See eig_batched.cuh for the role of each stage and the reference routines replaced.
#include <cooperative_groups.h>

#include <algorithm>
#include <cfloat>
#include <cmath>

#include "common.cuh"
#include "dmma.cuh"
#include "eig_batched.cuh"
#include "tridiag_dev.cuh"

namespace dvr3d {

namespace {

// ------------------------------------------------------------------ tridiagonalisation
// Lower Householder reduction as dsytd2('L'): for k = 0..n-3 the reflector H_k = I - tau_k v v^T,
// v = (0..0, 1, v_{k+2..n-1}), annihilates A[k+2:, k]. Columns are formed in panels of eight from the
// panel-start matrix (the dlatrd scheme: A v needs one read of the trailing matrix and no write; the
// matrix itself is updated once a panel, a rank-16 DMMA product over both triangles, subtracted from it
// as a whole: accumulators that start from the matrix round at its magnitude sixteen times, which
// doubled the vectors' errors, 9.8e-14 against 4.4e-14 rms for orders 160 to 459). A column k is a
// chain, kept short: the product with the trailing matrix and the panel's dot products use the
// column x itself and run beside its norm (v = e_{k+1} + sc x), every thread forms the reflector's
// scalars, and three block barriers and one exchange are left. A cluster of C CTAs shares a block:
// each takes every C-th column of the product and writes its partial sums to all; the vectors are
// replicated; the block stays in L2.
// Bound by that read (about 20 bytes a cycle and SM from L2) and, for small blocks, by the chain. 64
// blocks of order 465: 10.8 -> 5.1 ms against one CTA a block that read and wrote the trailing matrix
// for every column; 80 of order 300: 3.6 -> 2.4, 500 of order 300: 15.4 -> 9.5, 20 of order 1000:
// 90 -> 40 ms. Two CTAs a block (8.3 -> 5.1 ms for the 64) lose once they share an SM's L2 port.
constexpr int kTriNb = 8;
constexpr int kTriSmem = 152;
constexpr int kTriParts = 4;  // partial sums a row: C CTAs x 4 / C column subsets

template <int C>
__global__ void __launch_bounds__(1024) tridiag_kernel(BatchDesc bd, double *A, double *dg, double *eo, double *tauo, int ns) {
    namespace cg = cooperative_groups;
    const int b = blockIdx.x / C, rank = blockIdx.x % C;
    const int n = bd.n[b];
    double *ag = A + bd.aoff[b];
    double *d = dg + bd.voff[b], *e = eo + bd.voff[b], *tau = tauo + bd.voff[b];
    extern __shared__ double sm[];
    double *V = sm, *W = V + kTriNb * ns, *xs = W + kTriNb * ns, *sp0 = xs + ns;
    __shared__ double part[32], part2[32], zs[2 * kTriNb];
    if constexpr (C > 1) cg::this_cluster().barrier_arrive();
    const int T = blockDim.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = T >> 5;
    auto get = [&](int r, int c) { return __ldcg(ag + (unsigned)(c * n + r)); };
    auto exchange = [&]() {
        if constexpr (C > 1) cg::this_cluster().sync();
        else __syncthreads();
    };
    if (tid < 32) part[tid] = part2[tid] = 0.0;
    __syncthreads();
    const int row = tid;  // the row of this thread in the vector steps
    double acol = (row < n) ? get(row, 0) : 0.0, x = 0.0;
    if constexpr (C > 1) cg::this_cluster().barrier_wait();  // the others are there: partial sums go into them
    for (int k = 0; k + 2 < n; ++k) {
        const int i = k % kTriNb;
        if (i == 0 && k > 0) {
            // ---- A -= V W^T + W V^T on rows and columns k.. (16 rows x 16 columns a task)
            const int m = n - k, rt = (m + 15) / 16, ct = (m + 15) / 16, g = lane >> 2, t = lane & 3;
            for (int q = rank * nw + warp; q < rt * ct; q += C * nw) {
                const int r0 = k + (q % rt) * 16, c0 = k + (q / rt) * 16;
                double af[8];
#pragma unroll
                for (int h = 0; h < 8; ++h) af[h] = ((h >> 2) ? W : V)[(t + 4 * ((h >> 1) & 1)) * ns + r0 + g + 8 * (h & 1)];
                double old[2][4];
#pragma unroll
                for (int y = 0; y < 2; ++y)
#pragma unroll
                    for (int h = 0; h < 4; ++h) {
                        const int r = r0 + g + 8 * (h >> 1), c = c0 + 8 * y + 2 * t + (h & 1);
                        old[y][h] = (r < n && c < n) ? get(r, c) : 0.0;
                    }
#pragma unroll
                for (int y = 0; y < 2; ++y) {
                    double bf[4], acc[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
                    for (int h = 0; h < 4; ++h) bf[h] = ((h >> 1) ? V : W)[(t + 4 * (h & 1)) * ns + c0 + 8 * y + g];
                    dmma16(acc, af, bf);
#pragma unroll
                    for (int h = 0; h < 4; ++h) {
                        const int r = r0 + g + 8 * (h >> 1), c = c0 + 8 * y + 2 * t + (h & 1);
                        if (r < n && c < n) ag[(size_t)c * n + r] = old[y][h] - acc[h];
                    }
                }
            }
            exchange();
            acol = (row >= k && row < n) ? get(row, k) : 0.0;
        }
        // ---- the column, and its norm below the subdiagonal
        double ss = 0.0;
        const bool live = row > k && row < n;
        if (row >= k && row < n) {
            double v = acol;
            for (int t = 0; t < i; ++t) v -= V[t * ns + row] * W[t * ns + k] + W[t * ns + row] * V[t * ns + k];
            x = v;
            xs[row] = v;
            if (row == k && rank == 0) d[k] = v;
            if (row >= k + 2) ss = v * v;
        }
        ss = warp_sum(ss);
        if (lane == 0) part[warp] = ss;
        __syncthreads();
        // ---- A x (columns k+2..) in partial sums, and the panel's dot products with x
        double *sp = sp0 + (k & 1) * kTriParts * ns;  // the other CTAs may still read the last column's
        const int c0 = (k + 1) >> 5, nch = ((n - 1) >> 5) - c0 + 1;
        const int sub_n = max(1, min(kTriParts / C, nw / nch));
        const int sub = warp / nch;
        const double a1 = live ? get(row, k + 1) : 0.0;
        if (sub < sub_n) {
            const int g = rank * sub_n + sub, G = C * sub_n;  // this warp's columns: k + 2 + g mod G
            for (int ch = c0 + warp % nch; ch <= ((n - 1) >> 5); ch += (nch > nw) ? nw : nch) {
                const int r = 32 * ch + lane;
                const bool in = r > k && r < n;
                const int rc = in ? r : n - 1;
                double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
                int j = k + 2 + g;
                const double *col = ag + (unsigned)(j * n + rc);
                const unsigned st = (unsigned)(G * n);
                for (; j + 7 * G < n; j += 8 * G, col += 8 * st) {
                    double y[8];
#pragma unroll
                    for (int h = 0; h < 8; ++h) y[h] = __ldcg(col + h * st);
#pragma unroll
                    for (int h = 0; h < 8; h += 4) {
                        s0 = fma(y[h], xs[j + h * G], s0);
                        s1 = fma(y[h + 1], xs[j + (h + 1) * G], s1);
                        s2 = fma(y[h + 2], xs[j + (h + 2) * G], s2);
                        s3 = fma(y[h + 3], xs[j + (h + 3) * G], s3);
                    }
                }
                if (j < n) {  // the last columns, loads first
                    double y[7];
#pragma unroll
                    for (int h = 0; h < 7; ++h) y[h] = (j + h * G < n) ? __ldcg(col + h * st) : 0.0;
#pragma unroll
                    for (int h = 0; h < 7; ++h) s0 = fma(y[h], (j + h * G < n) ? xs[j + h * G] : 0.0, s0);
                }
                if (in) {
                    const double s = (s0 + s1) + (s2 + s3);
                    double *mine = sp + g * ns + r;
                    *mine = s;
                    if constexpr (C > 1) {
#pragma unroll
                        for (int q = 1; q < C; ++q) *cg::this_cluster().map_shared_rank(mine, (rank + q) % C) = s;
                    }
                }
            }
        }
        for (int t = warp; t < 2 * i; t += nw) {
            const double *col = (t < i) ? V + t * ns : W + (t - i) * ns;
            double s = 0.0;
            for (int r = k + 2 + lane; r < n; r += 32) s = fma(col[r], xs[r], s);
            s = warp_sum(s);
            if (lane == 0) zs[t] = s;
        }
        const double sig = warp_sum(part[lane]);
        const double alpha = xs[k + 1];
        double tk = 0.0, beta = alpha, sc = 0.0;
        if (sig != 0.0) {
            beta = -copysign(sqrt(alpha * alpha + sig), alpha);
            sc = 1.0 / (alpha - beta);
            tk = (beta - alpha) / beta;
        }
        exchange();
        // ---- q = A v on the current matrix, p.v, w = tau q - (tau^2 / 2)(q.v) v
        double qv = 0.0, v2 = 0.0;
        if (live) {
            double s = 0.0;
            for (int q = 0; q < C * sub_n; ++q) s += sp[q * ns + row];
            s = fma(sc, s, a1);
            for (int t = 0; t < i; ++t)
                s -= V[t * ns + row] * fma(sc, zs[i + t], W[t * ns + k + 1]) + W[t * ns + row] * fma(sc, zs[t], V[t * ns + k + 1]);
            v2 = (row == k + 1) ? 1.0 : sc * x;
            qv = s;
        }
        const double ps = warp_sum(qv * v2);
        if (lane == 0) part2[warp] = ps;
        __syncthreads();
        const double al = -0.5 * tk * tk * warp_sum(part2[lane]);
        if (live) {
            V[i * ns + row] = v2;
            W[i * ns + row] = fma(al, v2, tk * qv);
            if (rank == 0 && row > k + 1) ag[(size_t)k * n + row] = v2;  // reflector kept below the subdiagonal
        }
        acol = a1;
        if (tid == 0 && rank == 0) {
            e[k] = beta;
            tau[k] = tk;
        }
        __syncthreads();
    }
    // trailing 2 x 2 block: the last panel's columns are still pending
    if (tid == 0 && rank == 0) {
        const int cnt = (n > 2) ? (n - 3) % kTriNb + 1 : 0;
        auto cur = [&](int r, int c) {
            double v = get(r, c);
            for (int t = 0; t < cnt; ++t) v -= V[t * ns + r] * W[t * ns + c] + W[t * ns + r] * V[t * ns + c];
            return v;
        };
        if (n >= 2) {
            d[n - 2] = cur(n - 2, n - 2);
            e[n - 2] = cur(n - 1, n - 2);
            tau[n - 2] = 0.0;
        }
        d[n - 1] = cur(n - 1, n - 1);
        e[n - 1] = 0.0;
        tau[n - 1] = 0.0;
    }
    if constexpr (C > 1) cg::this_cluster().sync();
}

// Blocks that fit in shared memory: unblocked, the rank-2 update of the previous column fused with
// the product A x in one pass over shared memory. The same short chain a column: products with x
// beside its norm, three reductions, four barriers. One block of order 144: 0.64 -> 0.34 ms (the
// kernel above takes 0.59), 3200 of order 40: 0.31 -> 0.23, 500 of order 64: 0.20 -> 0.16 ms. The
// panel scheme loses here, its dot products cost more than the writes they save; at order 153 the
// block no longer fits beside its vectors.
__global__ void __launch_bounds__(512) tridiag_small_kernel(BatchDesc bd, double *A, double *dg, double *eo,
                                                            double *tauo) {
    const int b = blockIdx.x;
    const int n = bd.n[b];
    double *ag = A + bd.aoff[b];
    double *d = dg + bd.voff[b], *e = eo + bd.voff[b], *tau = tauo + bd.voff[b];
    extern __shared__ __align__(16) double sm[];
    double2 *xv = reinterpret_cast<double2 *>(sm);  // the column x; the previous reflector v
    double *ws = sm + 2 * n, *sp = ws + n, *as = sp + kTriParts * n;
    __shared__ double part[16], part2[16], s_alpha;
    const int T = blockDim.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = T >> 5, row = tid;
    for (int q = tid; q < n * n; q += T) as[q] = ag[q];
    for (int q = tid; q < n; q += T) {
        xv[q] = make_double2(0.0, 0.0);
        ws[q] = 0.0;
    }
    if (tid < 16) part[tid] = part2[tid] = 0.0;
    __syncthreads();
    double acol = (row < n) ? as[row] : 0.0, vp = 0.0, wp = 0.0;
    for (int k = 0; k + 2 < n; ++k) {
        const bool live = row > k && row < n;
        double x = 0.0, ss = 0.0;
        if (row >= k && row < n) {
            x = acol - (vp * ws[k] + wp * xv[k].y);
            if (row == k) d[k] = x;
            else if (row == k + 1) s_alpha = x;
            else ss = x * x;
            xv[row].x = (row >= k + 2) ? x : 0.0;
        }
        ss = warp_sum(ss);
        if (lane == 0) part[warp] = ss;
        __syncthreads();
        const int c0 = (k + 1) >> 5, nch = ((n - 1) >> 5) - c0 + 1;
        const int sub_n = max(1, min(kTriParts, nw / nch)), sub = warp / nch;
        if (sub < sub_n) {
            const int r = 32 * (c0 + warp % nch) + lane;
            if (r > k && r < n) {
                const double vr = xv[r].y, wr = ws[r];
                double s0 = 0.0, s1 = 0.0;
                int j = k + 1 + sub;
                double *col = as + (size_t)j * n + r;
                const int st = sub_n * n;
                for (; j + 3 * sub_n < n; j += 4 * sub_n, col += 4 * st) {
                    double a0 = col[0], a1 = col[st], a2 = col[2 * st], a3 = col[3 * st];
                    const double2 q0 = xv[j], q1 = xv[j + sub_n], q2 = xv[j + 2 * sub_n], q3 = xv[j + 3 * sub_n];
                    a0 -= vr * ws[j] + wr * q0.y;
                    a1 -= vr * ws[j + sub_n] + wr * q1.y;
                    a2 -= vr * ws[j + 2 * sub_n] + wr * q2.y;
                    a3 -= vr * ws[j + 3 * sub_n] + wr * q3.y;
                    col[0] = a0;
                    col[st] = a1;
                    col[2 * st] = a2;
                    col[3 * st] = a3;
                    s0 = fma(a0, q0.x, fma(a1, q1.x, s0));
                    s1 = fma(a2, q2.x, fma(a3, q3.x, s1));
                }
                for (; j < n; j += sub_n, col += st) {
                    const double2 q0 = xv[j];
                    const double a0 = col[0] - (vr * ws[j] + wr * q0.y);
                    col[0] = a0;
                    s0 = fma(a0, q0.x, s0);
                }
                sp[sub * n + r] = s0 + s1;
            }
        }
        const double sig = warp_sum(lane < 16 ? part[lane] : 0.0);
        const double alpha = s_alpha;
        double tk = 0.0, beta = alpha, sc = 0.0;
        if (sig != 0.0) {
            beta = -copysign(sqrt(alpha * alpha + sig), alpha);
            sc = 1.0 / (alpha - beta);
            tk = (beta - alpha) / beta;
        }
        __syncthreads();
        double qv = 0.0, v2 = 0.0;
        if (live) {
            acol = as[(size_t)(k + 1) * n + row];
            double s = 0.0;
            for (int q = 0; q < sub_n; ++q) s += sp[q * n + row];
            qv = fma(sc, s, acol);
            v2 = (row == k + 1) ? 1.0 : sc * x;
        }
        const double ps = warp_sum(qv * v2);
        if (lane == 0) part2[warp] = ps;
        __syncthreads();
        const double al = -0.5 * tk * tk * warp_sum(lane < 16 ? part2[lane] : 0.0);
        vp = v2;
        wp = fma(al, v2, tk * qv);
        if (live) {
            xv[row].y = vp;
            ws[row] = wp;
            if (row > k + 1) ag[(size_t)k * n + row] = v2;  // reflector kept below the subdiagonal
        }
        if (tid == 0) {
            e[k] = beta;
            tau[k] = tk;
        }
        __syncthreads();
    }
    if (tid == 0) {  // trailing 2 x 2 block: the last column is still pending
        auto cur = [&](int r, int c) { return as[(size_t)c * n + r] - (xv[r].y * ws[c] + ws[r] * xv[c].y); };
        if (n >= 2) {
            d[n - 2] = cur(n - 2, n - 2);
            e[n - 2] = cur(n - 1, n - 2);
            tau[n - 2] = 0.0;
        }
        d[n - 1] = cur(n - 1, n - 1);
        e[n - 1] = 0.0;
        tau[n - 1] = 0.0;
    }
}

// ------------------------------------------------------------------ eigenvalues
constexpr int kEvThreads = 512;

// Sturm-count multisection (by minors, or by quotients: tridiag_dev.cuh). Every CTA first counts at
// 512 equidistant points, which brackets each eigenvalue to 1/513 of the Gershgorin interval in one
// pass; then groups of L lanes narrow one eigenvalue each, L + 1 times a pass, L the largest power of
// two that keeps the CTA's threads busy.
// gridDim.y CTAs share a block's eigenvalues. Bound by the FP64 issue of the counts (three
// operations a row): 64 blocks of order 465, 62 eigenvalues each: 0.21 ms (one thread an eigenvalue
// with a division a row: 2.2 ms).
__global__ void __launch_bounds__(kEvThreads) eigvals_kernel(BatchDesc bd, const double *dg, const double *eo, double *wo,
                                                             int *cnt, int mode, double cut) {
    const int b = blockIdx.x;
    if (b >= bd.nblk) return;
    const int n = bd.n[b];
    const double *d = dg + bd.voff[b], *e = eo + bd.voff[b];
    double *w = wo + bd.voff[b];
    extern __shared__ double sm[];
    double *sd = sm, *ne2 = sm + n;
    __shared__ double s_min[kEvThreads], s_max[kEvThreads];
    __shared__ int s_cnt[kEvThreads];
    __shared__ int s_count;
    const int tid = threadIdx.x, lane = tid & 31;
    double lo = DBL_MAX, hi = -DBL_MAX;
    for (int i = tid; i < n; i += blockDim.x) {
        const double di = d[i];
        const double em = (i > 0) ? fabs(e[i - 1]) : 0.0, ep = (i < n - 1) ? fabs(e[i]) : 0.0;
        lo = fmin(lo, di - em - ep);
        hi = fmax(hi, di + em + ep);
    }
    s_min[tid] = lo;
    s_max[tid] = hi;
    __syncthreads();
    for (int s = blockDim.x / 2; s > 0; s >>= 1) {
        if (tid < s) {
            s_min[tid] = fmin(s_min[tid], s_min[tid + s]);
            s_max[tid] = fmax(s_max[tid], s_max[tid + s]);
        }
        __syncthreads();
    }
    // the matrix and its bounds in units of 1 / scale
    const double tnorm = fmax(fabs(s_min[0]), fabs(s_max[0]));
    double scale = sturm_scale(tnorm), piv = DBL_MIN;
    bool small = false;
    for (int i = tid; i < n; i += blockDim.x) {
        sd[i] = d[i] * scale;
        if (i < n - 1) {
            const double es = e[i] * scale;
            ne2[i] = -es * es;
            small |= !(es * es >= kSturmLeast);
        }
    }
    const bool quotients = __syncthreads_or(small);
    if (quotients) {
        scale = sturm_scale_quotients(tnorm);
        for (int i = tid; i < n; i += blockDim.x) {
            sd[i] = d[i] * scale;
            if (i < n - 1) {
                const double es = e[i] * scale;
                ne2[i] = es * es;
            }
        }
        __syncthreads();
        double most = 1.0;
        for (int i = 0; i < n - 1; ++i) most = fmax(most, ne2[i]);
        piv = DBL_MIN * most;
    }
    auto count = [&](double x) { return quotients ? sturm_quotients(sd, ne2, n, x, 1.0, piv) : sturm_count(sd, ne2, n, x); };
    const double unit = 1.0 / scale, margin = 2.0 * DBL_EPSILON * (tnorm * scale) * n + 2.0 * piv;
    const double glo = s_min[0] * scale - margin, ghi = s_max[0] * scale + margin;
    const double h = (ghi - glo) / (double)(kEvThreads + 1);
    s_cnt[tid] = count(glo + h * (double)(tid + 1));
    if (mode != 0 && tid == 0) {
        double x = cut;
        if (mode == 2) x = nextafter(cut, DBL_MAX);  // count of eigenvalues <= cut
        x *= scale;
        s_count = (x <= glo) ? 0 : (x >= ghi ? n : count(x));
    }
    __syncthreads();
    const int m = (mode != 0) ? s_count : n;
    const int P = gridDim.y, jb = (int)((long long)m * blockIdx.y / P), je = (int)((long long)m * (blockIdx.y + 1) / P);
    if (tid == 0 && blockIdx.y == 0) cnt[b] = m;
    int L = 1;
    while (L < 32 && (je - jb) * L * 2 <= kEvThreads) L *= 2;
    const int per = kEvThreads / L, sub = tid % L, g0 = lane - sub;  // eigenvalues at a time; lane in the group; its first
    const unsigned gmask = (L == 32 ? 0xffffffffu : ((1u << L) - 1u)) << g0;
    for (int j0 = jb; j0 < je; j0 += per) {
        const int j = j0 + tid / L;
        const bool mine = j < je;
        double a = glo, z = ghi;
        if (mine) {  // first point with more than j eigenvalues below it
            int p = 0, q = kEvThreads;
            while (p < q) {
                const int mid = (p + q) >> 1;
                if (s_cnt[mid] > j) q = mid;
                else p = mid + 1;
            }
            if (p > 0) a = glo + h * (double)p;
            if (p < kEvThreads) z = glo + h * (double)(p + 1);
        }
        bool run = mine;
        for (int pass = 0; pass < 200; ++pass) {
            if (run && z - a <= 2.0 * DBL_EPSILON * fmax(fabs(a), fabs(z))) run = false;
            if (!__any_sync(0xffffffffu, run)) break;
            const double x = (L == 1) ? 0.5 * (a + z) : a + (z - a) * ((double)(sub + 1) / (double)(L + 1));
            const bool above = count(x) > j;
            const unsigned bal = __ballot_sync(0xffffffffu, above) & gmask;
            const int f = bal ? __ffs(bal) - 1 - g0 : L;  // first lane above
            const double xl = __shfl_sync(0xffffffffu, x, g0 + (f > 0 ? f - 1 : 0));
            const double xh = __shfl_sync(0xffffffffu, x, g0 + (f < L ? f : L - 1));
            const double na = (f == 0) ? a : xl, nz = (f == L) ? z : xh;
            if (run) {
                if (!(nz - na < z - a)) run = false;  // interval at rounding level
                a = na;
                z = nz;
            }
        }
        if (mine && sub == 0) w[j] = 0.5 * (a + z) * unit;
    }
}

// ------------------------------------------------------------------ inverse iteration
// The first vector that failed its growth test since the last clear: {failed, block, eigenvalue
// index, block order}, for the host's error message.
__device__ int g_invit_fail[4];

// Eigenvectors of the tridiagonal matrices for the selected eigenvalues, as dstein: LU factors of
// T - lambda I with partial pivoting, four solves, modified Gram-Schmidt inside clusters of
// eigenvalues closer than 1e-6 ||T||. One warp per cluster with the factors and the iterate in its
// slice of shared memory; lane 0 runs the recurrences eight rows at a time, operands first, so that
// a row costs its dependent operations only. gridDim.y CTAs share a block's clusters. Bound by that
// chain: 3960 vectors of 64 blocks of order 465 take 1.0 ms.
__global__ void invit_batched_kernel(BatchDesc bd, const double *dg, const double *eo, const double *wo, const int *sel,
                                     const long long *zoff, const int *zld, double *Z, int *err) {
    const int b = blockIdx.x, part = blockIdx.y, nparts = gridDim.y;
    if (b >= bd.nblk) return;
    const int n = bd.n[b];
    const int m = sel[b];
    if (m <= 0) return;
    const double *w = wo + bd.voff[b];
    double *z = Z + zoff[b];
    const int ldz = zld[b];
    extern __shared__ double sm[];
    __shared__ int cstart[1026];
    __shared__ int s_ncl;
    __shared__ double red[32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarp = blockDim.x >> 5;
    const int np = (n + 8) & ~7;  // the eight-row loops run into the padding
    double *d = sm, *e = sm + np;
    double on = 0.0;
    for (int i = tid; i < np; i += blockDim.x) {
        const double di = (i < n) ? dg[bd.voff[b] + i] : 0.0, ei = (i < n - 1) ? eo[bd.voff[b] + i] : 0.0;
        const double em = (i > 0 && i < n) ? fabs(eo[bd.voff[b] + i - 1]) : 0.0;
        d[i] = di;
        e[i] = ei;
        on = fmax(on, fabs(di) + em + fabs(ei));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) on = fmax(on, __shfl_xor_sync(0xffffffffu, on, o));
    if (lane == 0) red[warp] = on;
    __syncthreads();
    on = red[0];
    for (int q = 1; q < nwarp; ++q) on = fmax(on, red[q]);
    const double onenrm = fmax(on, DBL_MIN);
    if (warp == 0) {  // cluster starts
        const double ortol = 1.0e-6 * onenrm;
        int nc = 0;
        for (int j0 = 0; j0 < m; j0 += 32) {
            const int j = j0 + lane;
            const bool st = j < m && (j == 0 || w[j] - w[j - 1] > ortol);
            const unsigned bal = __ballot_sync(0xffffffffu, st);
            if (st) cstart[nc + __popc(bal & ((1u << lane) - 1u))] = j;
            nc += __popc(bal);
        }
        if (lane == 0) {
            cstart[nc] = m;
            s_ncl = nc;
        }
    }
    __syncthreads();
    const size_t slice = (size_t)5 * np + np / 8;  // doubles per warp
    double *D = sm + 2 * np + warp * slice, *E1 = D + np, *E2 = E1 + np, *Lm = E2 + np, *x = Lm + np;
    unsigned char *P = reinterpret_cast<unsigned char *>(x + np);
    const double eps = DBL_EPSILON, tiny = eps * onenrm, pertol = 10.0 * eps * onenrm;
    const double grow_lim = invit_growth_limit(n);
    for (int c = part + nparts * warp; c < s_ncl; c += nparts * nwarp) {
        const int j0 = cstart[c], j1 = cstart[c + 1];
        double lamprev = 0.0;
        for (int j = j0; j < j1; ++j) {
            double lam = w[j];
            if (j > j0 && lam - lamprev < pertol) lam = lamprev + pertol;
            lamprev = lam;
            if (lane == 0) {
                double av = d[0] - lam, bv = e[0];
                for (int i = 0; i < n - 1; i += 8) {
                    double cc[9], an[8];
#pragma unroll
                    for (int u = 0; u < 8; ++u) {
                        cc[u] = e[i + u];
                        an[u] = d[min(i + u + 1, np - 1)] - lam;
                    }
                    cc[8] = e[min(i + 8, np - 1)];
#pragma unroll
                    for (int u = 0; u < 8; ++u) {
                        if (i + u < n - 1) {
                            const bool keep = fabs(av) >= fabs(cc[u]);
                            if (keep && av == 0.0) av = tiny;
                            const double piv = keep ? av : cc[u], mlt = (keep ? cc[u] : av) / piv;
                            const double bn = (i + u + 2 < n) ? cc[u + 1] : 0.0;
                            P[i + u] = keep ? 0 : 1;
                            Lm[i + u] = mlt;
                            D[i + u] = piv;
                            E1[i + u] = keep ? bv : an[u];
                            E2[i + u] = keep ? 0.0 : bn;
                            av = keep ? an[u] - mlt * bv : bv - mlt * an[u];
                            bv = keep ? bn : -mlt * bn;
                        }
                    }
                }
                if (fabs(av) < tiny) av = (av < 0.0) ? -tiny : tiny;
                D[n - 1] = av;
                // no superdiagonals in the last row of U; the back substitution reads them
                // (times zero), so stale shared memory must not leave a NaN there
                E1[n - 1] = 0.0;
                E2[n - 1] = 0.0;
            }
            __syncwarp();
            for (int i = lane; i < n - 1; i += 32)
                if (fabs(D[i]) < tiny) D[i] = (D[i] < 0.0) ? -tiny : tiny;
            __syncwarp();
            // the solves below multiply by the pivots' reciprocals (one division per pivot
            // here instead of one per pivot and iteration on the sequential path)
            const double dlast = D[n - 1];
            __syncwarp();
            for (int i = lane; i < n; i += 32) D[i] = 1.0 / D[i];
            for (int i = lane; i < n; i += 32) {
                const unsigned h = hash32((unsigned)(i * 2654435761u) ^ (unsigned)(j * 40503u + 17u));
                x[i] = ((double)(h & 0xffffff) / 8388608.0) - 1.0;
            }
            __syncwarp();
            int grown = 0;
            for (int it = 0; it < kInvitPasses; ++it) {
                double s1 = 0.0;
                for (int i = lane; i < n; i += 32) s1 += fabs(x[i]);
                s1 = warp_sum(s1);
                const double sc = (double)n * onenrm * fmax(eps, fabs(dlast)) / fmax(s1, DBL_MIN);
                for (int i = lane; i < n; i += 32) x[i] *= sc;
                __syncwarp();
                if (lane == 0) {
                    double y = x[0];
                    for (int i = 0; i < n - 1; i += 8) {
                        double xn[8], l[8];
                        const unsigned long long pm = *reinterpret_cast<const unsigned long long *>(P + i);
#pragma unroll
                        for (int u = 0; u < 8; ++u) {
                            xn[u] = x[min(i + u + 1, np - 1)];
                            l[u] = Lm[i + u];
                        }
#pragma unroll
                        for (int u = 0; u < 8; ++u) {
                            if (i + u < n - 1) {
                                const bool sw = (pm >> (8 * u)) & 1ull;
                                const double yi = sw ? xn[u] : y, yn = sw ? y : xn[u];
                                x[i + u] = yi;
                                y = yn - l[u] * yi;
                            }
                        }
                    }
                    x[n - 1] = y;
                    double x1 = 0.0, x2 = 0.0;
                    for (int i = ((n - 1) / 8) * 8; i >= 0; i -= 8) {
                        double xx[8], r1[8], r2[8], dd[8];
#pragma unroll
                        for (int u = 0; u < 8; ++u) {
                            xx[u] = x[i + u];
                            r1[u] = E1[i + u];
                            r2[u] = E2[i + u];
                            dd[u] = D[i + u];
                        }
#pragma unroll
                        for (int u = 7; u >= 0; --u) {
                            if (i + u < n) {
                                const double xi = (xx[u] - r2[u] * x2 - r1[u] * x1) * dd[u];
                                x[i + u] = xi;
                                x2 = x1;
                                x1 = xi;
                            }
                        }
                    }
                }
                __syncwarp();
                for (int jj = j0; jj < j; ++jj) {
                    const double *zc = z + (size_t)jj * ldz;
                    double dot = 0.0;
                    for (int i = lane; i < n; i += 32) dot += x[i] * zc[i];
                    dot = warp_sum(dot);
                    for (int i = lane; i < n; i += 32) x[i] -= dot * zc[i];
                }
                double nrm = 0.0, xinf = 0.0;
                for (int i = lane; i < n; i += 32) {
                    nrm += x[i] * x[i];
                    xinf = fmax(xinf, fabs(x[i]));
                }
                nrm = sqrt(warp_sum(nrm));
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) xinf = fmax(xinf, __shfl_xor_sync(0xffffffffu, xinf, o));
                grown += (xinf >= grow_lim);
                const double inv = (nrm > 0.0) ? 1.0 / nrm : 0.0;
                for (int i = lane; i < n; i += 32) x[i] *= inv;
                __syncwarp();
            }
            if (grown < kInvitGrowPasses && lane == 0 && err) {
                *err = kDevNoConv;
                if (atomicCAS(&g_invit_fail[0], 0, 1) == 0) {
                    g_invit_fail[1] = b;
                    g_invit_fail[2] = j;
                    g_invit_fail[3] = n;
                }
            }
            // sign convention: the first largest component positive
            double big = 0.0;
            int bi = n;
            for (int i = lane; i < n; i += 32)
                if (fabs(x[i]) > fabs(big)) {
                    big = x[i];
                    bi = i;
                }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const double ob = __shfl_xor_sync(0xffffffffu, big, o);
                const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
                if (fabs(ob) > fabs(big) || (fabs(ob) == fabs(big) && oi < bi)) {
                    big = ob;
                    bi = oi;
                }
            }
            const double sg = (big < 0.0) ? -1.0 : 1.0;
            double *zc = z + (size_t)j * ldz;
            for (int i = lane; i < n; i += 32) zc[i] = sg * x[i];
            __syncwarp();
        }
    }
}

// ------------------------------------------------------------------ back-transformation
// z <- H_0 H_1 ... H_{n-3} z by panels of 32 reflectors in compact WY form, I - V T V^T, on the FP64
// tensor path. V is read from the block itself (unit diagonal implied), T is kept in the block's
// upper triangle, which the reduction has left unused: panel p0's T(r, c), r <= c, at row p0 + r of
// column p0 + c + 1. 3960 vectors of 64 blocks of order 465: 0.05 + 0.38 ms; with inverse iteration
// 5.4 -> 1.45 ms against one kernel that walked a column per thread through panels of 16.
constexpr int kBtP = 32;

// V(i, c) of panel p0: rows i of the block
__device__ __forceinline__ double bt_v(const double *a, int n, int p0, int nbk, int i, int c) {
    const int top = p0 + c + 1;
    if (c >= nbk || i >= n || i < top) return 0.0;
    return (i == top) ? 1.0 : a[(size_t)(p0 + c) * n + i];
}

// T of every panel: the Gram matrix V^T V over four warps, then dlarft (forward, columnwise).
__global__ void __launch_bounds__(128) bt_factor_kernel(BatchDesc bd, double *A, const double *tauo, const int *sel) {
    const int b = blockIdx.y, p0 = blockIdx.x * kBtP;
    const int n = bd.n[b], nbk = min(kBtP, n - 2 - p0);
    if (nbk <= 0 || sel[b] <= 0) return;
    double *a = A + bd.aoff[b];
    const double *tau = tauo + bd.voff[b] + p0;
    __shared__ double G[4][32 * 33];
    __shared__ double T[32][33];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, r = lane >> 2, c = lane & 3;
    double acc[2][4][4];
#pragma unroll
    for (int x = 0; x < 2; ++x)
#pragma unroll
        for (int y = 0; y < 4; ++y)
#pragma unroll
            for (int h = 0; h < 4; ++h) acc[x][y][h] = 0.0;
    for (int k0 = p0 + 1 + 16 * warp; k0 < n; k0 += 64) {
        double af[2][8], bf[4][4];
#pragma unroll
        for (int x = 0; x < 2; ++x)
#pragma unroll
            for (int i = 0; i < 8; ++i) af[x][i] = bt_v(a, n, p0, nbk, k0 + c + 4 * (i >> 1), x * 16 + r + 8 * (i & 1));
#pragma unroll
        for (int y = 0; y < 4; ++y)
#pragma unroll
            for (int i = 0; i < 4; ++i) bf[y][i] = af[y >> 1][2 * i + (y & 1)];  // the same elements
#pragma unroll
        for (int x = 0; x < 2; ++x)
#pragma unroll
            for (int y = 0; y < 4; ++y) dmma16(acc[x][y], af[x], bf[y]);
    }
#pragma unroll
    for (int x = 0; x < 2; ++x)
#pragma unroll
        for (int y = 0; y < 4; ++y)
#pragma unroll
            for (int h = 0; h < 4; ++h) G[warp][(y * 8 + c * 2 + (h & 1)) * 33 + x * 16 + r + 8 * (h >> 1)] = acc[x][y][h];
    for (int q = tid; q < 32 * 33; q += 128) (&T[0][0])[q] = 0.0;
    __syncthreads();
    for (int q = tid; q < 1024; q += 128) {
        const int k = (q >> 5) * 33 + (q & 31);
        G[0][k] = (G[0][k] + G[1][k]) + (G[2][k] + G[3][k]);
    }
    __syncthreads();
    if (warp == 0) {
        for (int i = 0; i < nbk; ++i) {  // T(0:i, i) = -tau_i T(0:i, 0:i) V^T v_i
            const double ti = tau[i];
            double s0 = 0.0, s1 = 0.0;
            for (int k = 0; k < i; k += 2) {
                s0 = fma(T[lane][k], G[0][i * 33 + k], s0);
                if (k + 1 < i) s1 = fma(T[lane][k + 1], G[0][i * 33 + k + 1], s1);
            }
            T[lane][i] = (lane < i) ? -ti * (s0 + s1) : (lane == i ? ti : 0.0);
            __syncwarp();
        }
    }
    __syncthreads();
    for (int q = tid; q < 1024; q += 128) {
        const int i = q >> 5, k = q & 31;  // T(k, i)
        if (k <= i && i < nbk) a[(size_t)(p0 + i + 1) * n + p0 + k] = T[k][i];
    }
}

// NC columns of Z a CTA, kept in shared memory ([column][row], stride 4 mod 16) through all panels:
// W = V^T Z (rows split over the eight warps), W2 = T W, Z -= V W2 (the products summed first: Z is
// rounded once a panel, not once a reflector).
template <int NC>
__global__ void __launch_bounds__(256) bt_apply_kernel(BatchDesc bd, const double *A, const int *sel, const long long *zoff,
                                                       const int *zld, double *Z, int zs) {
    const int b = blockIdx.y, c0 = blockIdx.x * NC;
    const int n = bd.n[b], m = sel[b];
    if (c0 >= m || n < 3) return;
    constexpr int NT = NC / 8;
    const double *a = A + bd.aoff[b];
    double *z = Z + zoff[b] + (size_t)c0 * zld[b];
    const int ldz = zld[b], nc = min(NC, m - c0);
    extern __shared__ double sm[];
    double *zt = sm, *red = sm + (size_t)NC * zs, *W = red + 8 * NC * 33, *W2 = W + NC * 36;  // W: [column][k]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, r = lane >> 2, c = lane & 3;
    for (int k = 0; k < NC; ++k)
        for (int i = tid; i < zs; i += 256) zt[(size_t)k * zs + i] = (k < nc && i < n) ? z[(size_t)k * ldz + i] : 0.0;
    __syncthreads();
    for (int p0 = ((n - 3) / kBtP) * kBtP; p0 >= 0; p0 -= kBtP) {
        const int nbk = min(kBtP, n - 2 - p0);
        {
            double acc[2][NT][4];
#pragma unroll
            for (int x = 0; x < 2; ++x)
#pragma unroll
                for (int y = 0; y < NT; ++y)
#pragma unroll
                    for (int h = 0; h < 4; ++h) acc[x][y][h] = 0.0;
            for (int k0 = p0 + 1 + 16 * warp; k0 < n; k0 += 128) {
                double af[2][8], bf[NT][4];
#pragma unroll
                for (int x = 0; x < 2; ++x)
#pragma unroll
                    for (int i = 0; i < 8; ++i) af[x][i] = bt_v(a, n, p0, nbk, k0 + c + 4 * (i >> 1), x * 16 + r + 8 * (i & 1));
#pragma unroll
                for (int y = 0; y < NT; ++y)
#pragma unroll
                    for (int i = 0; i < 4; ++i) bf[y][i] = zt[(size_t)(y * 8 + r) * zs + k0 + c + 4 * i];
#pragma unroll
                for (int x = 0; x < 2; ++x)
#pragma unroll
                    for (int y = 0; y < NT; ++y) dmma16(acc[x][y], af[x], bf[y]);
            }
            double *mine = red + (size_t)warp * NC * 33;
#pragma unroll
            for (int x = 0; x < 2; ++x)
#pragma unroll
                for (int y = 0; y < NT; ++y)
#pragma unroll
                    for (int h = 0; h < 4; ++h) mine[(y * 8 + c * 2 + (h & 1)) * 33 + x * 16 + r + 8 * (h >> 1)] = acc[x][y][h];
        }
        __syncthreads();
        for (int q = tid; q < NC * 32; q += 256) {
            const int col = q >> 5, k = q & 31;
            double s = 0.0;
#pragma unroll
            for (int u = 0; u < 8; ++u) s += red[(size_t)u * NC * 33 + col * 33 + k];
            W[col * 36 + k] = s;
        }
        __syncthreads();
        if (warp < 2 * NT) {  // W2 = T W: 16 rows, 8 columns a warp
            const int m0 = (warp & 1) * 16, n0 = (warp >> 1) * 8;
            double acc[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
            for (int k0 = 0; k0 < 32; k0 += 16) {
                double af[8], bf[4];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int row = m0 + r + 8 * (i & 1), k = k0 + c + 4 * (i >> 1);
                    af[i] = (row <= k && k < nbk) ? a[(size_t)(p0 + k + 1) * n + p0 + row] : 0.0;
                }
#pragma unroll
                for (int i = 0; i < 4; ++i) bf[i] = W[(n0 + r) * 36 + k0 + c + 4 * i];
                dmma16(acc, af, bf);
            }
#pragma unroll
            for (int h = 0; h < 4; ++h) W2[(n0 + c * 2 + (h & 1)) * 36 + m0 + r + 8 * (h >> 1)] = -acc[h];
        }
        __syncthreads();
        for (int i0 = p0 + 1 + 16 * warp; i0 < n; i0 += 128) {
            double acc[NT][4];
#pragma unroll
            for (int y = 0; y < NT; ++y)
#pragma unroll
                for (int h = 0; h < 4; ++h) acc[y][h] = 0.0;
#pragma unroll
            for (int k0 = 0; k0 < 32; k0 += 16) {
                double af[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) af[i] = bt_v(a, n, p0, nbk, i0 + r + 8 * (i & 1), k0 + c + 4 * (i >> 1));
#pragma unroll
                for (int y = 0; y < NT; ++y) {
                    double bf[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) bf[i] = W2[(y * 8 + r) * 36 + k0 + c + 4 * i];
                    dmma16(acc[y], af, bf);
                }
            }
#pragma unroll
            for (int y = 0; y < NT; ++y)
#pragma unroll
                for (int h = 0; h < 4; ++h) zt[(size_t)(y * 8 + c * 2 + (h & 1)) * zs + i0 + r + 8 * (h >> 1)] += acc[y][h];
        }
        __syncthreads();
    }
    for (int k = 0; k < nc; ++k)
        for (int i = tid; i < n; i += 256) z[(size_t)k * ldz + i] = zt[(size_t)k * zs + i];
}

__global__ void symmetrize_lower_kernel(BatchDesc bd, double *A) {
    const int b = blockIdx.y;
    const int n = bd.n[b];
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (long long)n * n) return;
    const int i = (int)(idx % n), j = (int)(idx / n);
    if (j > i) A[bd.aoff[b] + idx] = A[bd.aoff[b] + (long long)i * n + j];
}

}  // namespace

void launch_symmetrize_lower(const BatchDesc &bd, double *A, int nmax, cudaStream_t st) {
    dim3 grid((unsigned)(((long long)nmax * nmax + 255) / 256), bd.nblk);
    DVR3D_COUNT_LAUNCH(1);
    symmetrize_lower_kernel<<<grid, 256, 0, st>>>(bd, A);
}

namespace {
int sm_count() {
    int dev = 0, nsm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    return std::max(nsm, 1);
}
}  // namespace

namespace {
template <int C>
void launch_tridiag(const BatchDesc &bd, double *A, double *d, double *e, double *tau, int nmax, cudaStream_t st) {
    const int ns = (nmax + 32) / 8 * 8;  // the update's tiles run past the end
    const size_t smem = (size_t)(2 * kTriNb + 1 + 2 * kTriParts) * ns * sizeof(double);
    int dev = 0;
    cudaGetDevice(&dev);
    static bool attr[kMaxAttrDevices] = {};
    if (dev < 0 || dev >= kMaxAttrDevices || !attr[dev]) {
        cudaFuncSetAttribute(tridiag_kernel<C>, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024);
        if (dev >= 0 && dev < kMaxAttrDevices) attr[dev] = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(bd.nblk * C);
    cfg.blockDim = dim3(1024);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = C;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, tridiag_kernel<C>, bd, A, d, e, tau, ns);
}
}  // namespace

void launch_tridiag_batched(const BatchDesc &bd, double *A, double *d, double *e, double *tau,
                            int nmax, cudaStream_t st) {
    if (bd.nblk <= 0) return;
    DVR3D_COUNT_LAUNCH(1);
    if (nmax <= kTriSmem) {
        int dev = 0;
        cudaGetDevice(&dev);
        static bool attr[kMaxAttrDevices] = {};
        if (dev < 0 || dev >= kMaxAttrDevices || !attr[dev]) {
            cudaFuncSetAttribute(tridiag_small_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024);
            if (dev >= 0 && dev < kMaxAttrDevices) attr[dev] = true;
        }
        // three column subsets a row chunk while the blocks are few
        const int rows = (nmax + 31) / 32;
        const int warps = std::max(2, std::min(16, bd.nblk > 4 * sm_count() ? rows : 3 * rows));
        const size_t smem = ((size_t)nmax * nmax + (3 + kTriParts) * (size_t)nmax) * sizeof(double);
        tridiag_small_kernel<<<bd.nblk, 32 * warps, smem, st>>>(bd, A, d, e, tau);
    } else if (2 * bd.nblk <= sm_count()) {  // two CTAs a block while they find an SM each
        launch_tridiag<2>(bd, A, d, e, tau, nmax, st);
    } else {
        launch_tridiag<1>(bd, A, d, e, tau, nmax, st);
    }
}

void launch_eigvals_batched(const BatchDesc &bd, const double *d, const double *e, double *w,
                            int *cnt, int mode, double cut, cudaStream_t st) {
    if (bd.nblk <= 0) return;
    // few blocks: several CTAs a block, each with its share of the eigenvalues
    const int parts = std::max(1, std::min(8, sm_count() / bd.nblk));
    // dynamic shared memory: d and -e^2 of the largest block (caller guarantees <= 1024)
    DVR3D_COUNT_LAUNCH(1);
    eigvals_kernel<<<dim3(bd.nblk, parts), kEvThreads, 2 * 1024 * sizeof(double), st>>>(bd, d, e, w, cnt, mode, cut);
}

void launch_eigvecs_batched(const BatchDesc &bd, double *A, const double *d, const double *e, const double *tau,
                            const double *w, const int *sel, const long long *zoff, const int *zld, double *Z, int nmax,
                            int *err, cudaStream_t st) {
    if (bd.nblk <= 0) return;
    constexpr size_t cap = 200 * 1024;
    const int np = (nmax + 8) & ~7;
    int nwarp = 8;
    auto invit_smem = [&](int k) { return ((size_t)2 * np + (size_t)k * (5 * np + np / 8)) * sizeof(double); };
    while (nwarp > 1 && invit_smem(nwarp) > cap) --nwarp;
    // 32 columns of Z a CTA where they fit (orders up to 527), else 16
    auto bt_smem = [&](int nc, int zs) { return ((size_t)nc * zs + 8 * nc * 33 + 2 * nc * 36) * sizeof(double); };
    const int zs = (nmax + 32) / 16 * 16 + 4;  // 16-row tiles run past the end
    const bool wide = bt_smem(32, zs) <= cap + 24 * 1024;
    int dev = 0;
    cudaGetDevice(&dev);
    // the shared-memory limit is a per-device attribute of the kernels
    static bool attr[kMaxAttrDevices] = {};
    if (dev < 0 || dev >= kMaxAttrDevices || !attr[dev]) {
        cudaFuncSetAttribute(invit_batched_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cap);
        cudaFuncSetAttribute(bt_apply_kernel<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cap + 24 * 1024);
        cudaFuncSetAttribute(bt_apply_kernel<16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cap + 24 * 1024);
        if (dev >= 0 && dev < kMaxAttrDevices) attr[dev] = true;
    }
    // fewer blocks than SMs: several CTAs per block (their clusters split between them)
    const int parts = std::max(1, std::min(16, sm_count() / bd.nblk));
    DVR3D_COUNT_LAUNCH(1);
    invit_batched_kernel<<<dim3(bd.nblk, parts), 32 * nwarp, invit_smem(nwarp), st>>>(bd, d, e, w, sel, zoff, zld, Z, err);
    if (nmax < 3) return;
    DVR3D_COUNT_LAUNCH(2);
    for (int b0 = 0; b0 < bd.nblk; b0 += 65535) {  // blocks per launch: gridDim.y
        BatchDesc q = bd;
        q.nblk = std::min(65535, bd.nblk - b0);
        q.n += b0;
        q.aoff += b0;
        q.voff += b0;
        bt_factor_kernel<<<dim3((nmax - 2 + kBtP - 1) / kBtP, q.nblk), 128, 0, st>>>(q, A, tau, sel + b0);
        if (wide)
            bt_apply_kernel<32><<<dim3((nmax + 31) / 32, q.nblk), 256, bt_smem(32, zs), st>>>(q, A, sel + b0, zoff + b0,
                                                                                           zld + b0, Z, zs);
        else
            bt_apply_kernel<16><<<dim3((nmax + 15) / 16, q.nblk), 256, bt_smem(16, zs), st>>>(q, A, sel + b0, zoff + b0,
                                                                                           zld + b0, Z, zs);
    }
}

void invit_fail_clear(cudaStream_t st) {
    void *p = nullptr;
    if (cudaGetSymbolAddress(&p, g_invit_fail) == cudaSuccess) cudaMemsetAsync(p, 0, sizeof(int) * 4, st);
}

void invit_fail_info(cudaStream_t st, int out[4]) {
    void *p = nullptr;
    out[0] = out[1] = out[2] = out[3] = 0;
    if (cudaGetSymbolAddress(&p, g_invit_fail) == cudaSuccess) {
        cudaMemcpyAsync(out, p, sizeof(int) * 4, cudaMemcpyDeviceToHost, st);
        cudaStreamSynchronize(st);
    }
}

}  // namespace dvr3d
