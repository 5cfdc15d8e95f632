// band_reduce.cu -- dense symmetric matrix -> band of half-bandwidth 32, the first stage of the
// two-stage reduction to tridiagonal form (the second is the bulge chase of band_eig.cu).
//
// The one-stage reduction reads the whole trailing matrix once per column; here it is read and
// updated once per 32 columns, by matrix-matrix products. Panel j0 (32 columns):
//   panel_qr_kernel  QR of the rows below the panel's diagonal block: V (unit lower trapezoidal),
//                    T with Q = I - V T V^T; R and the diagonal block go to the band;
//   symm_kernel      X = A2 V, A2 = A[j0+32:, j0+32:] (lower triangle stored);
//   vtx_kernel       S = V^T X, M = -T^T S T / 2;
//   w_kernel         W = X T + V M, and the next panel's columns of A2 - V W^T - W V^T;
//   syr2k_kernel     the rest of A2 <- A2 - V W^T - W V^T (lower triangle).
// 4/3 n^3 flop, nearly all in symm and syr2k on the FP64 tensor path (DMMA m16n8k16). The next panel
// needs only what w_kernel makes, so it runs beside syr2k, on 16 of the SMs. At n = 12202 the
// reduction to the band takes 125 ms (symm 54, syr2k with the panels beside it 66, vtx 6, w 4) and the
// chase 49, against 950 ms in one stage; one after the other, with a cluster barrier in every column
// of a panel, the two stages took 240.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cmath>

#include "band_reduce.cuh"
#include "cluster_dev.cuh"
#include "common.cuh"
#include "dmma.cuh"
#include "gemm64.cuh"

namespace dvr3d {

namespace {

namespace cg = cooperative_groups;

constexpr int kB = kBandMaxBw;      // panel width = half-bandwidth
constexpr int kCl = 16;             // CTAs of the panel's cluster
constexpr int kPanelWarps = 15;     // working warps per CTA (one more forms T)
constexpr int kPanelSmem = 24;      // 32 x 32 blocks a CTA holds in shared memory beside them
constexpr unsigned kFull = 0xffffffffu;

__device__ __forceinline__ void cp16(void *smem, const void *gmem, int bytes) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(bytes));
}

// ------------------------------------------------------------------ panel QR
struct PanelArgs {
    const double *P;    // the panel's rows j0.. (diagonal block first), 32 columns
    long long ldp;
    int R, nr;          // rows below the diagonal block; reflectors, min(32, R - 1)
    double *V;          // out: V, columns 0..31 and again 64..95
    long long ldv;
    double *Vk;         // out: V once more (for the back-transformation), or null
    long long ldk;
    double *T;          // out: 32 x 32, column-major, upper triangular
    double *C;          // the band
    int j0, n;
    int nsm;            // blocks of a CTA in shared memory, the rest in `spill` (L2)
    double *spill;
    int *err;           // set when a wait runs out
    unsigned long long limit;
};

struct PanelShared {
    double wpart[kPanelWarps][32];   // per warp: x^T a_c over its rows
    double prow[32];                 // pivot row (first CTA)
    double cpart[2][kCl][32];        // per CTA, written by every CTA of the cluster
    double ppart[2][32];
    double w[32], z[32];
    double T[32][33];
    double sc, beta;
    unsigned long long full[2];      // mbarriers: cpart and ppart are complete
};
constexpr unsigned kPanelBytes = (kCl + 1) * 32 * sizeof(double);  // what a column brings to each CTA
constexpr unsigned long long kPanelPolls = 1ull << 26;  // of a wait, about a second
constexpr int kBarPart = 1, kBarRow = 2;  // the warps' sums are there; the rank-1 update is known

// One thread-block cluster factors the panel. Each warp keeps one 32 x 32 block of it in registers
// (lane = (row mod 4, column mod 8): 8 x 4 elements) and, beyond 7680 rows, further blocks in
// shared memory (beyond 19968 in L2). Per column one all-reduce of x^T [a_0 .. a_31] over the cluster, x the column
// below its pivot, gives the norm, the row vector of the rank-1 update and the column of V^T V
// that T needs. A control warp does all of the exchange: it adds up the warps' sums, stores them into
// every CTA of the cluster (st.async: the mbarrier there counts the bytes, so nothing waits for the
// stores to return and no cluster barrier follows), adds up what has come in and forms the scalars;
// the others meet it at two named barriers a column, and T's column follows off the path.
// Latency bound: 1.6 us a column; 59 us a panel on average from 3960 rows down (81 with a cluster
// barrier a column and the exchange on a working warp).
__global__ void __launch_bounds__((kPanelWarps + 1) * 32, 1) panel_qr_kernel(PanelArgs p) {
    extern __shared__ __align__(16) double psm[];
    PanelShared &S = *reinterpret_cast<PanelShared *>(psm);
    double *blocks = psm + (sizeof(PanelShared) + 15) / 16 * 2;
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = (int)cluster.block_rank();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int NW = (int)(blockDim.x >> 5) - 1, nthr = (int)blockDim.x;
    const bool worker = warp < NW;
    const int rl = lane & 3, cl = lane >> 2;
    const int nblk = (p.R + 31) / 32;
    const int b0 = warp * kCl + rank;  // block of layer l: (l NW + warp) 16 + rank
    int layers = 0;
    if (worker)
        for (int b = b0; b < nblk; b += NW * kCl) ++layers;
    const bool top = worker && b0 == 0;  // holds the pivot rows
    // blocks of layers 1..: in shared memory, then in global memory; f(block, its row block index)
    auto beyond = [&](auto &&f) {
        for (int l = 1; l < layers; ++l) {
            const int q = (l - 1) * NW + warp, b = b0 + l * NW * kCl;
            if (q < p.nsm) f(blocks + (size_t)q * 1024, b);
            else f(p.spill + ((size_t)(q - p.nsm) * kCl + rank) * 1024, b);
        }
    };
    double a[8][4];
    auto fetch = [&](int b, int kk, int nt) {
        const int r = 32 * b + 4 * kk + rl;
        return (r < p.R) ? __ldcg(p.P + (size_t)(8 * nt + cl) * p.ldp + 32 + r) : 0.0;
    };
#pragma unroll
    for (int kk = 0; kk < 8; ++kk)
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) a[kk][nt] = (layers > 0) ? fetch(b0, kk, nt) : 0.0;
    beyond([&](double *B, int b) {
#pragma unroll
        for (int kk = 0; kk < 8; ++kk)
#pragma unroll
            for (int nt = 0; nt < 4; ++nt) B[(kk * 4 + nt) * 32 + lane] = fetch(b, kk, nt);
    });
    if (rank == 0) {  // the diagonal block
        for (int q = tid; q < 32 * 32; q += blockDim.x) {
            const int r = q & 31, c = q >> 5;
            if (r < c || p.j0 + r >= p.n) continue;
            const double v = __ldcg(p.P + (size_t)c * p.ldp + r);
            p.C[(size_t)(p.j0 + c) * kBandLd + r - c] = v;
        }
    }
    for (int q = tid; q < 32 * 33; q += blockDim.x) (&S.T[0][0])[q] = 0.0;
    const unsigned full0 = smem_u32(&S.full[0]);
    if (tid == 0) {
        for (int q = 0; q < 2; ++q) {
            mbar_init(full0 + 8 * q, 1);
            mbar_expect(full0 + 8 * q, kPanelBytes);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    cluster.sync();
    // the control warp: lane = (half of the cluster, pair of columns)
    const int hc = (lane >> 4) * (kCl / 2), cp2 = 2 * (lane & 15);
    bool patient = true;  // until a wait has ended without its data; the rest then runs without waits
    auto exchange = [&](int i) {
        const int par = i & 1;
        bar_sync(kBarPart, nthr);
        double s0 = 0.0, s1 = 0.0, t0 = 0.0, t1 = 0.0;
        int g = 0;
        for (; g + 1 < NW; g += 2) {
            const double2 p0 = *reinterpret_cast<const double2 *>(&S.wpart[g][cp2]);
            const double2 p1 = *reinterpret_cast<const double2 *>(&S.wpart[g + 1][cp2]);
            s0 += p0.x;
            t0 += p0.y;
            s1 += p1.x;
            t1 += p1.y;
        }
        if (g < NW) {
            const double2 p0 = *reinterpret_cast<const double2 *>(&S.wpart[g][cp2]);
            s0 += p0.x;
            t0 += p0.y;
        }
        s0 += s1;
        t0 += t1;
        const unsigned mine = smem_u32(&S.cpart[par][rank][cp2]), bar = full0 + 8 * par;
#pragma unroll
        for (int u = 0; u < kCl / 2; ++u) st_async2(map_rank(mine, hc + u), s0, t0, map_rank(bar, hc + u));
        if (rank == 0) {
            const double2 pv = *reinterpret_cast<const double2 *>(&S.prow[cp2]);
            const unsigned piv = smem_u32(&S.ppart[par][cp2]);
#pragma unroll
            for (int u = 0; u < kCl / 2; ++u) st_async2(map_rank(piv, hc + u), pv.x, pv.y, map_rank(bar, hc + u));
        }
        // Past the limit the error is recorded; the wait itself goes on to the default limit, so that
        // stores of this column do not arrive in a CTA that has left.
        unsigned long long spins = 0;
        while (patient && !mbar_test_cta(bar, (i >> 1) & 1)) {
            if (++spins == p.limit) atomicExch(p.err, (int)kDevBarrierTimeout);
            if (spins > p.limit && spins > kPanelPolls) patient = false;
        }
        __syncwarp();
        // for column i + 2, which nobody sends before our i + 1
        if (lane == 0 && patient) mbar_expect(bar, kPanelBytes);
        double q0 = 0.0, q1 = 0.0;
#pragma unroll
        for (int u = 0; u < kCl; u += 2) {
            q0 += S.cpart[par][u][lane];
            q1 += S.cpart[par][u + 1][lane];
        }
        const double q = q0 + q1, pc = S.ppart[par][lane];
        const double alpha = __shfl_sync(kFull, pc, i), sig = __shfl_sync(kFull, q, i);
        double tau = 0.0, beta = alpha, sc = 0.0;
        if (sig != 0.0) {
            beta = -copysign(sqrt(alpha * alpha + sig), alpha);
            sc = 1.0 / (alpha - beta);
            tau = (beta - alpha) / beta;
        }
        const double vq = fma(sc, q, pc);  // a_c^T v (c > i), V_c^T v (c < i)
        S.w[lane] = (lane > i) ? tau * vq : 0.0;
        if (lane == 0) {
            S.sc = sc;
            S.beta = beta;
        }
        bar_arrive(kBarRow, nthr);
        if (rank == kCl - 1) {
            // T[0:i, i] = -tau T[0:i, 0:i] z, T[i][i] = tau (dlarft, forward, columnwise)
            S.z[lane] = (lane < i) ? vq : 0.0;
            __syncwarp();
            double r0 = 0.0, r1 = 0.0;
            for (int c = 0; c < i; c += 2) {
                r0 = fma(S.T[lane][c], S.z[c], r0);
                r1 = fma(S.T[lane][c + 1], S.z[c + 1], r1);  // z[i] = 0
            }
            S.T[lane][i] = (lane < i) ? -tau * (r0 + r1) : (lane == i ? tau : 0.0);
            __syncwarp();
        }
    };
    if (!worker)
        for (int i = 0; i < p.nr; ++i) exchange(i);
#pragma unroll
    for (int ph = 0; ph < 4; ++ph) {
        if (!worker) break;
        for (int ii = 0; ii < 8; ++ii) {
            const int i = 8 * ph + ii;
            if (i >= p.nr) break;
            const int src = ii * 4 + rl;
            double x[8];
            double q4[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
            for (int kk = 0; kk < 8; ++kk) {
                x[kk] = __shfl_sync(kFull, a[kk][ph], src);
                if (top && 4 * kk + rl <= i) x[kk] = 0.0;
            }
#pragma unroll
            for (int kk = 0; kk < 8; ++kk)
#pragma unroll
                for (int nt = 0; nt < 4; ++nt) q4[nt] = fma(x[kk], a[kk][nt], q4[nt]);
            beyond([&](const double *B, int) {
#pragma unroll
                for (int kk = 0; kk < 8; ++kk) {
                    const double xs = B[(kk * 4 + ph) * 32 + src];
#pragma unroll
                    for (int nt = 0; nt < 4; ++nt) q4[nt] = fma(xs, B[(kk * 4 + nt) * 32 + lane], q4[nt]);
                }
            });
            // sums over the four row lanes: lane rl ends with column 8 rl + cl
            const bool hi = rl & 2, od = rl & 1;
            double u0 = hi ? q4[0] : q4[2], u1 = hi ? q4[1] : q4[3];
            u0 = __shfl_xor_sync(kFull, u0, 2);
            u1 = __shfl_xor_sync(kFull, u1, 2);
            const double v0 = (hi ? q4[2] : q4[0]) + u0, v1 = (hi ? q4[3] : q4[1]) + u1;
            const double s = (od ? v1 : v0) + __shfl_xor_sync(kFull, od ? v0 : v1, 1);
            S.wpart[warp][8 * rl + cl] = s;
            if (top && rl == (i & 3)) {
#pragma unroll
                for (int nt = 0; nt < 4; ++nt) S.prow[8 * nt + cl] = (ii >> 2) ? a[2 * ph + 1][nt] : a[2 * ph][nt];
            }
            bar_arrive(kBarPart, nthr);
            bar_sync(kBarRow, nthr);
            const double sc = S.sc;
            double wn[4];
#pragma unroll
            for (int nt = ph; nt < 4; ++nt) wn[nt] = S.w[8 * nt + cl];
#pragma unroll
            for (int kk = 0; kk < 8; ++kk) {
                const double v = sc * x[kk];
                if (top && 4 * kk + rl <= i) {
                    if (4 * kk + rl == i) {  // the pivot row
#pragma unroll
                        for (int nt = ph; nt < 4; ++nt) a[kk][nt] -= wn[nt];
                        if (cl == ii) a[kk][ph] = S.beta;
                    }
                } else {
#pragma unroll
                    for (int nt = ph; nt < 4; ++nt) a[kk][nt] = fma(-v, wn[nt], a[kk][nt]);
                    if (cl == ii) a[kk][ph] = v;
                }
            }
            beyond([&](double *B, int) {
#pragma unroll
                for (int kk = 0; kk < 8; ++kk) {
                    const double v = sc * B[(kk * 4 + ph) * 32 + src];
                    __syncwarp();
#pragma unroll
                    for (int nt = ph; nt < 4; ++nt) {
                        double *e = B + (kk * 4 + nt) * 32 + lane;
                        *e = (nt == ph && cl == ii) ? v : fma(-v, wn[nt], *e);
                    }
                }
                __syncwarp();
            });
        }
    }
    __syncthreads();
    auto put = [&](int b, int kk, int nt, double v) {
        const int r = 32 * b + 4 * kk + rl, c = 8 * nt + cl;
        if (r >= p.R) return;
        double o = v;
        if (b == 0 && r <= c) {  // R
            const int i = p.j0 + 32 + r, j = p.j0 + c;
            p.C[(size_t)j * kBandLd + i - j] = v;
            o = (r == c) ? 1.0 : 0.0;
        }
        if (c >= p.nr) o = 0.0;
        p.V[(size_t)c * p.ldv + r] = o;
        p.V[(size_t)(c + 64) * p.ldv + r] = o;
        if (p.Vk) p.Vk[(size_t)c * p.ldk + r] = o;
    };
    if (layers > 0) {
#pragma unroll
        for (int kk = 0; kk < 8; ++kk)
#pragma unroll
            for (int nt = 0; nt < 4; ++nt) put(b0, kk, nt, a[kk][nt]);
    }
    beyond([&](const double *B, int b) {
#pragma unroll
        for (int kk = 0; kk < 8; ++kk)
#pragma unroll
            for (int nt = 0; nt < 4; ++nt) put(b, kk, nt, B[(kk * 4 + nt) * 32 + lane]);
    });
    if (rank == kCl - 1)
        for (int q = tid; q < 32 * 32; q += blockDim.x) p.T[q] = S.T[q & 31][q >> 5];
    cluster.sync();
}

// ------------------------------------------------------------------ X = A2 V
constexpr int kBM = 64, kBK = 16, kThr = 128, kStages = 4, kSymmPerSm = 4;
constexpr int kSM = kBM + 4;         // column stride of the update's tiles
constexpr int kATile = kBM * kBK;    // [row][k] or [k][row], unpadded: pairs of doubles change places
constexpr int kBTile = kB * kBK;     // within a row by swz(pair, row), which spreads the fragments' reads
__device__ __forceinline__ int swz(int pair, int row) { return (pair ^ ((row & 3) << 1)) << 1; }
constexpr size_t kSymmSmem = (size_t)kStages * (kATile + kBTile) * sizeof(double);
constexpr int kSymmMost = 1024;  // CTAs
// CTAs of X = A2 V: kSymmPerSm an SM, but at least four k tiles each (28 steps from 900 rows down take
// 0.35 ms; with eight k tiles 0.43)
inline int symm_ctas(int R, int nsm) {
    const long long units = (long long)((R + kBM - 1) / kBM) * ((R + kBK - 1) / kBK);
    return (int)std::max(1ll, std::min((long long)std::min(kSymmMost, kSymmPerSm * nsm), units / 4));
}

// X (R x 32) = A2 V, A2 symmetric with its lower triangle stored: a 64-row tile takes k tiles left
// of its diagonal block as stored, those right of it transposed (from the rows below), and the
// diagonal block element by element. A2 is read twice (2/3 n^3 flop over n^3 / 12 bytes).
// All CTAs get the same number of k tiles, counted through tile after tile: a CTA ends one row tile
// and begins another, and whoever is last at a tile adds up its parts, in their order (a split of
// every tile into S equal parts, in a cluster, leaves SMs idle unless tiles x S happens to fill them:
// 48 -> 40 ms for the first 150 steps at n = 12241, 19.7 -> 23.8 TF/s for the first one). Four CTAs an
// SM by their four stages of unpadded tiles; three with padded ones: 43 ms.
__global__ void __launch_bounds__(kThr, kSymmPerSm) symm_kernel(const double *A2, long long lda, int R, const double *V, long long ldv,
                                                    double *X, long long ldx, double *part, int *count) {
    extern __shared__ __align__(16) double sm[];
    __shared__ int s_old;
    const int ntk = (R + kBK - 1) / kBK, G = gridDim.x;
    const long long units = (long long)((R + kBM - 1) / kBM) * ntk;
    long long u = units * blockIdx.x / G;
    const long long u1 = units * (blockIdx.x + 1) / G;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wm = (warp >> 1) * 32, wn = (warp & 1) * 16;
    const int r = lane >> 2, c = lane & 3;
    while (u < u1) {
        const int tile = (int)(u / ntk), i0 = tile * kBM, t0 = (int)(u - (long long)tile * ntk);
        const int t1 = (int)min((long long)ntk, t0 + (u1 - u));
        double acc[2][2][4];
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
            for (int b = 0; b < 2; ++b)
#pragma unroll
                for (int h = 0; h < 4; ++h) acc[a][b][h] = 0.0;
        auto load = [&](int kt) {
            double *As = sm + (kt - t0) % kStages * (kATile + kBTile), *Bs = As + kATile;
            const int k0 = kt * kBK, kmax = R - k0;
#pragma unroll
            for (int q = 0; q < 2; ++q) {  // V rows k0.., 32 columns, k-contiguous
                const int e = tid + q * kThr, j = e >> 3, k = (e & 7) * 2;
                const int valid = min(max(kmax - k, 0), 2);
                cp16(Bs + j * kBK + swz(k >> 1, j), valid ? V + (size_t)j * ldv + k0 + k : V, valid * 8);
            }
            if (k0 + kBK <= i0) {  // as stored: [k][row]
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int e = tid + q * kThr, k = e >> 5, i = (e & 31) * 2;
                    const int valid = min(max(R - i0 - i, 0), 2);
                    cp16(As + k * kBM + swz(i >> 1, k), valid ? A2 + (size_t)(k0 + k) * lda + i0 + i : A2, valid * 8);
                }
            } else if (k0 >= i0 + kBM) {  // transposed: [row][k]
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int e = tid + q * kThr, i = e >> 3, k = (e & 7) * 2;
                    const int valid = (i0 + i < R) ? min(max(kmax - k, 0), 2) : 0;
                    cp16(As + i * kBK + swz(k >> 1, i), valid ? A2 + (size_t)(i0 + i) * lda + k0 + k : A2, valid * 8);
                }
            } else {
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    const int e = tid + q * kThr, k = e >> 6, i = e & 63;
                    const int gi = i0 + i, gk = k0 + k;
                    As[k * kBM + swz(i >> 1, k) + (i & 1)] = (gi < R && gk < R) ? A2[(size_t)min(gi, gk) * lda + max(gi, gk)] : 0.0;
                }
            }
        };
#pragma unroll
        for (int q = 0; q < kStages - 1; ++q) {
            if (t0 + q < t1) load(t0 + q);
            asm volatile("cp.async.commit_group;\n" ::);
        }
        for (int kt = t0; kt < t1; ++kt) {
            asm volatile("cp.async.wait_group %0;\n" ::"n"(kStages - 2));
            __syncthreads();
            if (kt + kStages - 1 < t1) load(kt + kStages - 1);
            asm volatile("cp.async.commit_group;\n" ::);
            const double *As = sm + (kt - t0) % kStages * (kATile + kBTile), *Bs = As + kATile;
            const bool tr = kt * kBK >= i0 + kBM;
            double af[2][8], bf[2][4];
            if (tr) {
#pragma unroll
                for (int a = 0; a < 2; ++a)
#pragma unroll
                    for (int i = 0; i < 8; ++i)
                        af[a][i] = As[(wm + a * 16 + r + 8 * (i & 1)) * kBK + swz((c >> 1) + 2 * (i >> 1), r) + (c & 1)];
            } else {
#pragma unroll
                for (int a = 0; a < 2; ++a)
#pragma unroll
                    for (int i = 0; i < 8; ++i)
                        af[a][i] = As[(c + 4 * (i >> 1)) * kBM + swz(((wm + r) >> 1) + a * 8 + 4 * (i & 1), c) + (r & 1)];
            }
#pragma unroll
            for (int b = 0; b < 2; ++b)
#pragma unroll
                for (int i = 0; i < 4; ++i) bf[b][i] = Bs[(wn + b * 8 + r) * kBK + swz((c >> 1) + 2 * i, r) + (c & 1)];
#pragma unroll
            for (int a = 0; a < 2; ++a)
#pragma unroll
                for (int b = 0; b < 2; ++b) dmma16(acc[a][b], af[a], bf[b]);
        }
        asm volatile("cp.async.wait_group 0;\n" ::);
        __syncthreads();
        const bool whole = t0 == 0 && t1 == ntk;
        // a CTA has at most one part that begins its tile (the CTA's last) and one that does not
        double *out = part + ((size_t)blockIdx.x * 2 + (t0 == 0)) * (kBM * kB);
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
            for (int b = 0; b < 2; ++b)
#pragma unroll
                for (int h = 0; h < 4; ++h) {
                    const int i = wm + a * 16 + r + 8 * (h >> 1), j = wn + b * 8 + c * 2 + (h & 1);
                    if (!whole) __stcg(out + j * kBM + i, acc[a][b][h]);
                    else if (i0 + i < R) X[(size_t)j * ldx + i0 + i] = acc[a][b][h];
                }
        if (!whole) {
            // the CTAs of this tile's first and last unit
            const long long f = (long long)tile * ntk;
            const int qa = (int)(((f + 1) * G - 1) / units), qb = (int)(((f + ntk) * G - 1) / units);
            __threadfence();
            __syncthreads();
            if (tid == 0) s_old = atomicAdd(count + tile, 1);
            __syncthreads();
            if (s_old == qb - qa) {
                __threadfence();
                double2 sum[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) sum[e] = make_double2(0.0, 0.0);
                for (int q = qa; q <= qb; ++q) {
                    const double2 *src = reinterpret_cast<const double2 *>(part + ((size_t)q * 2 + (q == qa)) * (kBM * kB));
#pragma unroll
                    for (int e = 0; e < 8; ++e) {
                        const double2 v = __ldcg(src + tid + e * kThr);
                        sum[e].x += v.x;
                        sum[e].y += v.y;
                    }
                }
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    const int o = 2 * (tid + e * kThr), i = i0 + o % kBM;
                    double *x = X + (size_t)(o / kBM) * ldx + i;
                    if (i < R) x[0] = sum[e].x;
                    if (i + 1 < R) x[1] = sum[e].y;
                }
                if (tid == 0) count[tile] = 0;
            }
        }
        u += t1 - t0;
        __syncthreads();  // the operand buffers and s_old are free
    }
}

// ------------------------------------------------------------------ S = V^T X, M = -T^T S T / 2
// One cluster; every warp takes k steps of 16 rows, operands straight from L2 as fragments. Bound by
// latency: the warps' sums are added in two rounds and go to the first CTA in one store each, so that
// what follows the loads is two block barriers and one of the cluster: 10.5 us a launch on average
// from 900 rows down (13.7 with eight rounds and the first CTA reading the others' sums).
constexpr int kVS = 32 * 33;  // a 32 x 32 tile, column-major, 33 a column
constexpr size_t kVtxSmem = (size_t)(kCl + 4) * kVS * sizeof(double);
__global__ void __launch_bounds__(256) vtx_kernel(const double *V, long long ldv, const double *X, long long ldx, int R,
                                                  const double *T, double *M) {
    extern __shared__ __align__(16) double sm[];
    double *recv = sm, *loc = sm + kCl * kVS;  // every CTA's sum (first CTA); of this one's warps
    __shared__ double Ts[kVS], Y[kVS];
    cg::cluster_group cluster = cg::this_cluster();
    cluster.barrier_arrive();  // the first CTA is there before anything is stored into it
    const int rank = (int)cluster.block_rank();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, r = lane >> 2, c = lane & 3;
    for (int q = tid; q < 1024; q += 256) Ts[(q >> 5) * 33 + (q & 31)] = T[q];
    double acc[2][4][4];
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b)
#pragma unroll
            for (int h = 0; h < 4; ++h) acc[a][b][h] = 0.0;
    const int ks = (R + 15) / 16;
    for (int k = rank * 8 + warp; k < ks; k += kCl * 8) {
        const int k0 = k * 16;
        double af[2][8], bf[4][4];
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int kk = k0 + c + 4 * (i >> 1);
                af[a][i] = (kk < R) ? V[(size_t)(a * 16 + r + 8 * (i & 1)) * ldv + kk] : 0.0;
            }
#pragma unroll
        for (int b = 0; b < 4; ++b)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int kk = k0 + c + 4 * i;
                bf[b][i] = (kk < R) ? X[(size_t)(b * 8 + r) * ldx + kk] : 0.0;
            }
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
            for (int b = 0; b < 4; ++b) dmma16(acc[a][b], af[a], bf[b]);
    }
#pragma unroll
    for (int round = 0; round < 2; ++round) {  // warps 4..7 store, 0..3 add theirs
        if ((warp < 4) == (round == 1)) {
            double *l = loc + (warp & 3) * kVS;
#pragma unroll
            for (int a = 0; a < 2; ++a)
#pragma unroll
                for (int b = 0; b < 4; ++b)
#pragma unroll
                    for (int h = 0; h < 4; ++h) {
                        const int e = (b * 8 + c * 2 + (h & 1)) * 33 + a * 16 + r + 8 * (h >> 1);
                        l[e] = round ? l[e] + acc[a][b][h] : acc[a][b][h];
                    }
        }
        __syncthreads();
    }
    cluster.barrier_wait();
    for (int q = tid; q < 1024; q += 256) {
        const int e = (q >> 5) * 33 + (q & 31);
        *cluster.map_shared_rank(recv + rank * kVS + e, 0) = (loc[e] + loc[kVS + e]) + (loc[2 * kVS + e] + loc[3 * kVS + e]);
    }
    cluster.sync();
    if (rank == 0) {
        for (int q = tid; q < 1024; q += 256) {
            const int e = (q >> 5) * 33 + (q & 31);
            double s = 0.0;
#pragma unroll
            for (int u = 0; u < kCl; ++u) s += recv[u * kVS + e];
            Y[e] = s;  // S
        }
        __syncthreads();
        // warp: rows 16 (warp / 4), columns 8 (warp % 4); first S T, then T^T (S T)
        const int m0 = (warp >> 2) * 16, n0 = (warp & 3) * 8;
        double g[4] = {0.0, 0.0, 0.0, 0.0}, h4[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
        for (int k0 = 0; k0 < 32; k0 += 16) {
            double af[8], bf[4];
#pragma unroll
            for (int i = 0; i < 8; ++i) af[i] = Y[(k0 + c + 4 * (i >> 1)) * 33 + m0 + r + 8 * (i & 1)];
#pragma unroll
            for (int i = 0; i < 4; ++i) bf[i] = Ts[(n0 + r) * 33 + k0 + c + 4 * i];
            dmma16(g, af, bf);
        }
        __syncthreads();
#pragma unroll
        for (int h = 0; h < 4; ++h) Y[(n0 + c * 2 + (h & 1)) * 33 + m0 + r + 8 * (h >> 1)] = g[h];
        __syncthreads();
#pragma unroll
        for (int k0 = 0; k0 < 32; k0 += 16) {
            double af[8], bf[4];
#pragma unroll
            for (int i = 0; i < 8; ++i) af[i] = Ts[(m0 + r + 8 * (i & 1)) * 33 + k0 + c + 4 * (i >> 1)];
#pragma unroll
            for (int i = 0; i < 4; ++i) bf[i] = Y[(n0 + r) * 33 + k0 + c + 4 * i];
            dmma16(h4, af, bf);
        }
#pragma unroll
        for (int h = 0; h < 4; ++h) M[(n0 + c * 2 + (h & 1)) * 32 + m0 + r + 8 * (h >> 1)] = -0.5 * h4[h];
    }
}

// ------------------------------------------------------------------ W and the next panel
constexpr int kWS = kBM + 4;  // column stride of the 64-row tiles
constexpr int kPS = 36;       // column stride of the 32-row ones
constexpr size_t kWSmem = (size_t)(3 * 32 * kWS + 5 * 32 * kPS) * sizeof(double);

// 64 rows a CTA: W = X T + V M (also for the first 32 rows, which every CTA needs), then the
// next panel P = A2[:, 0:32] - V W_p^T - W V_p^T, W_p and V_p their first 32 rows. Bound by the
// latency of its loads, which therefore all leave at once: 7.6 us a launch on average from 3968 rows
// down (24 with loads of 8 bytes a few at a time).
__global__ void __launch_bounds__(kThr) w_kernel(double *VWV, long long ldv, const double *X, long long ldx, const double *T,
                                                 const double *M, int R, const double *A2, long long lda, double *P,
                                                 long long ldp) {
    extern __shared__ __align__(16) double sm[];
    double *Xs = sm, *Vs = Xs + 32 * kWS, *Ws = Vs + 32 * kWS;  // [column][row], 64 rows
    double *Xp = Ws + 32 * kWS, *Vp = Xp + 32 * kPS, *Wp = Vp + 32 * kPS, *Tm = Wp + 32 * kPS, *Mm = Tm + 32 * kPS;
    const int i0 = blockIdx.x * kBM;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, r = lane >> 2, c = lane & 3;
    // everything is asked for before anything is waited for
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const int e = tid + q * kThr, j = e >> 5, i = (e & 31) * 2, valid = min(max(R - i0 - i, 0), 2);
        cp16(Xs + j * kWS + i, valid ? X + (size_t)j * ldx + i0 + i : X, valid * 8);
        cp16(Vs + j * kWS + i, valid ? VWV + (size_t)j * ldv + i0 + i : VWV, valid * 8);
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int e = tid + q * kThr, j = e >> 4, i = (e & 15) * 2, valid = min(max(R - i, 0), 2);
        cp16(Xp + j * kPS + i, valid ? X + (size_t)j * ldx + i : X, valid * 8);
        cp16(Vp + j * kPS + i, valid ? VWV + (size_t)j * ldv + i : VWV, valid * 8);
        cp16(Tm + j * kPS + i, T + 32 * j + i, 16);
        cp16(Mm + j * kPS + i, M + 32 * j + i, 16);
    }
    asm volatile("cp.async.commit_group;\n" ::);
    double old[4][4];
#pragma unroll
    for (int b = 0; b < 4; ++b)
#pragma unroll
        for (int h = 0; h < 4; ++h) {
            const int i = i0 + warp * 16 + r + 8 * (h >> 1), j = b * 8 + c * 2 + (h & 1);
            old[b][h] = (i < R && i >= j) ? A2[(size_t)j * lda + i] : 0.0;
        }
    asm volatile("cp.async.wait_group 0;\n" ::);
    __syncthreads();
    // acc (16 rows m0.. of [column][row] tiles with stride s, nt column tiles from n0) += Lh Rh,
    // Lh(m, k) = L[k s + m], Rh(k, n) = B[n kPS + k] (bt: B[k kPS + n])
    auto mul = [&](double (*acc)[4], int nt, const double *L, int s, int m0, const double *B, int n0, bool bt) {
#pragma unroll
        for (int k0 = 0; k0 < 32; k0 += 16) {
            double af[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) af[i] = L[(k0 + c + 4 * (i >> 1)) * s + m0 + r + 8 * (i & 1)];
            for (int b = 0; b < nt; ++b) {
                double bf[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int k = k0 + c + 4 * i, n = n0 + b * 8 + r;
                    bf[i] = bt ? B[k * kPS + n] : B[n * kPS + k];
                }
                dmma16(acc[b], af, bf);
            }
        }
    };
    {
        double acc[4][4] = {}, accp[2][4] = {};
        mul(acc, 4, Xs, kWS, warp * 16, Tm, 0, false);
        mul(acc, 4, Vs, kWS, warp * 16, Mm, 0, false);
        const int mp = (warp >> 1) * 16, np = (warp & 1) * 16;
        mul(accp, 2, Xp, kPS, mp, Tm, np, false);
        mul(accp, 2, Vp, kPS, mp, Mm, np, false);
#pragma unroll
        for (int b = 0; b < 4; ++b)
#pragma unroll
            for (int h = 0; h < 4; ++h) Ws[(b * 8 + c * 2 + (h & 1)) * kWS + warp * 16 + r + 8 * (h >> 1)] = acc[b][h];
#pragma unroll
        for (int b = 0; b < 2; ++b)
#pragma unroll
            for (int h = 0; h < 4; ++h) Wp[(np + b * 8 + c * 2 + (h & 1)) * kPS + mp + r + 8 * (h >> 1)] = accp[b][h];
    }
    __syncthreads();
    for (int q = tid; q < 32 * 64; q += kThr) {
        const int j = q >> 6, i = q & 63;
        if (i0 + i < R) VWV[(size_t)(32 + j) * ldv + i0 + i] = Ws[j * kWS + i];
    }
    double acc[4][4] = {};
    mul(acc, 4, Vs, kWS, warp * 16, Wp, 0, true);  // (V W_p^T)(m, n) = sum_k V(m, k) W_p(n, k), W_p[k kPS + n]
    mul(acc, 4, Ws, kWS, warp * 16, Vp, 0, true);
#pragma unroll
    for (int b = 0; b < 4; ++b)
#pragma unroll
        for (int h = 0; h < 4; ++h) {
            const int i = i0 + warp * 16 + r + 8 * (h >> 1), j = b * 8 + c * 2 + (h & 1);
            if (i < R && i >= j) P[(size_t)j * ldp + i] = old[b][h] - acc[b][h];
        }
}

// ------------------------------------------------------------------ A -= V W^T + W V^T
constexpr size_t kSyrSmem = (size_t)3 * 64 * kSM * sizeof(double);
constexpr int kSyrThr = 256;

// One 64 x 64 tile of the lower triangle, K = 64: [V W] against [W V], which the buffer V W V
// holds side by side. The tile of A comes into shared memory behind the operands and the products'
// sum is subtracted from it once: accumulators that start from -A round at its magnitude 64 times
// (levels of order 3984: 2.1e-16 hartree rms against 1.1e-16), and no faster (128 -> 125 ms for the
// reduction at n = 12202). Eight warps of 32 x 16 (four of 32 x 32 left fewer in flight: 48.7 -> 47.1
// ms for the first 150 steps at n = 12241): 20 TF/s, against 6.2 for the one-stage path's update.
__global__ void __launch_bounds__(kSyrThr, 2) syr2k_band_kernel(double *A, long long lda, int R, const double *VWV, long long ldv) {
    extern __shared__ __align__(16) double sm[];
    double *Xs = sm, *Ys = sm + 64 * kSM, *As = Ys + 64 * kSM;
    const long long t = blockIdx.x;
    int ti = (int)((sqrt(8.0 * (double)t + 1.0) - 1.0) * 0.5);
    while ((long long)ti * (ti + 1) / 2 > t) --ti;
    while ((long long)(ti + 1) * (ti + 2) / 2 <= t) ++ti;
    const int i0 = ti * 64, j0 = (int)(t - (long long)ti * (ti + 1) / 2) * 64;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, r = lane >> 2, c = lane & 3;
    const int wm = (warp >> 2) * 32, wn = (warp & 3) * 16;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const int e = tid + q * kSyrThr, k = e >> 5, i = (e & 31) * 2;
        const int vi = min(max(R - i0 - i, 0), 2), vj = min(max(R - j0 - i, 0), 2);
        cp16(Xs + k * kSM + i, vi ? VWV + (size_t)k * ldv + i0 + i : VWV, vi * 8);
        cp16(Ys + k * kSM + i, vj ? VWV + (size_t)(32 + k) * ldv + j0 + i : VWV, vj * 8);
    }
    asm volatile("cp.async.commit_group;\n" ::);
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const int e = tid + q * kSyrThr, j = e >> 5, i = (e & 31) * 2;
        const int valid = (j0 + j < R) ? min(max(R - i0 - i, 0), 2) : 0;
        cp16(As + j * kSM + i, valid ? A + (size_t)(j0 + j) * lda + i0 + i : A, valid * 8);
    }
    asm volatile("cp.async.commit_group;\n" ::);
    double acc[2][2][4];
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int b = 0; b < 2; ++b)
#pragma unroll
            for (int h = 0; h < 4; ++h) acc[a][b][h] = 0.0;
    asm volatile("cp.async.wait_group 1;\n" ::);
    __syncthreads();
#pragma unroll
    for (int k0 = 0; k0 < 64; k0 += 16) {
        double af[2][8], bf[2][4];
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
            for (int i = 0; i < 8; ++i) af[a][i] = Xs[(k0 + c + 4 * (i >> 1)) * kSM + wm + a * 16 + r + 8 * (i & 1)];
#pragma unroll
        for (int b = 0; b < 2; ++b)
#pragma unroll
            for (int i = 0; i < 4; ++i) bf[b][i] = Ys[(k0 + c + 4 * i) * kSM + wn + b * 8 + r];
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
            for (int b = 0; b < 2; ++b) dmma16(acc[a][b], af[a], bf[b]);
    }
    asm volatile("cp.async.wait_group 0;\n" ::);
    __syncthreads();
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int b = 0; b < 2; ++b)
#pragma unroll
            for (int h = 0; h < 4; ++h) {
                const int i = wm + a * 16 + r + 8 * (h >> 1), j = wn + b * 8 + c * 2 + (h & 1);
                if (i0 + i < R && j0 + j <= i0 + i) A[(size_t)(j0 + j) * lda + i0 + i] = As[j * kSM + i] - acc[a][b][h];
            }
}

// the last columns of the matrix (nothing below them to eliminate), as a panel
__global__ void copy_panel_kernel(const double *A, long long lda, int rows, int cols, double *P, long long ldp) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long long)rows * kB) return;
    const int j = (int)(t / rows), i = (int)(t % rows);
    P[(size_t)j * ldp + i] = (j < cols && i >= j) ? A[(size_t)j * lda + i] : 0.0;
}

inline long long rup(long long x, long long m) { return (x + m - 1) / m * m; }

struct PanelPlan {
    int warps, extra, nsm;  // working warps; blocks of a CTA beyond registers; those in shared memory
    size_t smem;
    explicit PanelPlan(int R) {
        const int k = std::max(1, ((R + 31) / 32 + kCl - 1) / kCl);  // blocks of a CTA
        warps = std::min(kPanelWarps, k);
        extra = ((k + warps - 1) / warps - 1) * warps;
        nsm = std::min(extra, kPanelSmem);
        smem = (sizeof(PanelShared) + 15) / 16 * 16 + (size_t)nsm * 1024 * sizeof(double);
    }
    size_t spill_doubles() const { return (size_t)(extra - nsm) * kCl * 1024; }
};

struct ClusterLaunch {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    ClusterLaunch(dim3 grid, int threads, size_t smem, int cx, int cy, cudaStream_t st) {
        cfg.gridDim = grid;
        cfg.blockDim = dim3(threads);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = st;
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = cx;
        attr[0].val.clusterDim.y = cy;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
    }
};

cudaError_t set_attributes() {
    cudaError_t e;
    const int most = (int)PanelPlan(1 << 20).smem;
    if ((e = cudaFuncSetAttribute(panel_qr_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1)) != cudaSuccess) return e;
    if ((e = cudaFuncSetAttribute(vtx_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1)) != cudaSuccess) return e;
    if ((e = cudaFuncSetAttribute(panel_qr_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, most)) != cudaSuccess) return e;
    if ((e = cudaFuncSetAttribute(symm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSymmSmem)) != cudaSuccess) return e;
    if ((e = cudaFuncSetAttribute(vtx_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kVtxSmem)) != cudaSuccess) return e;
    if ((e = cudaFuncSetAttribute(w_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kWSmem)) != cudaSuccess) return e;
    return cudaFuncSetAttribute(syr2k_band_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSyrSmem);
}

// Per device: 0 not looked at yet, 1 attributes set and a cluster of kCl CTAs fits, 2 it does not.
std::atomic<int> g_state[kMaxAttrDevices];

}  // namespace

bool band_reduce_available() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxAttrDevices) return false;
    int s = g_state[dev].load(std::memory_order_acquire);
    if (s == 0) {
        bool ok = set_attributes() == cudaSuccess;
        if (ok) {
            ClusterLaunch l(dim3(kCl), (kPanelWarps + 1) * 32, PanelPlan(1 << 20).smem, kCl, 1, nullptr);
            int n = 0;
            ok = cudaOccupancyMaxActiveClusters(&n, panel_qr_kernel, &l.cfg) == cudaSuccess && n > 0;
        }
        if (!ok) cudaGetLastError();
        s = ok ? 1 : 2;
        g_state[dev].store(s, std::memory_order_release);
    }
    return s == 1;
}

static size_t symm_count_doubles(int n) { return (size_t)rup((n + kBM - 1) / kBM, 4) / 2; }

size_t band_reduce_work_doubles(int n) {
    const size_t ld = (size_t)rup(n, 8);
    // V W V twice, X, P, M, the counters and parts of symm_kernel, the panel's blocks in L2
    return ld * (2 * 96 + 32 + 32) + 1024 + symm_count_doubles(n) + (size_t)symm_ctas(n, kSymmMost) * 2 * kBM * kB +
           PanelPlan(n).spill_doubles();
}

cudaError_t launch_band_reduce(const BandReduce &b, cudaStream_t st) {
    const int n = b.n;
    const long long ld = rup(n, 8);
    double *X = b.work + 2 * 96 * ld, *P = X + 32 * ld, *M = P + 32 * ld;
    int *count = reinterpret_cast<int *>(M + 1024);
    double *part = M + 1024 + symm_count_doubles(n), *spill = part + (size_t)symm_ctas(n, kSymmMost) * 2 * kBM * kB;
    if (!band_reduce_available()) return cudaErrorNotSupported;
    cudaError_t e;
    if ((e = cudaMemsetAsync(count, 0, symm_count_doubles(n) * sizeof(double), st)) != cudaSuccess) return e;
    if ((e = cudaMemsetAsync(b.C, 0, band_storage_doubles(n) * sizeof(double), st)) != cudaSuccess) return e;
    int dev = 0, nsm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    // The panel needs only what w_kernel has made of its columns, so panel j + 1 runs beside the
    // update of step j, which goes to the side stream; V W V alternates between two buffers. Whichever
    // way this function is left, `st` waits for the side stream.
    struct Join {
        const BandReduce &b;
        cudaStream_t st;
        bool open = false;
        cudaError_t close() {
            if (!open) return cudaSuccess;
            open = false;
            const cudaError_t e = cudaEventRecord(b.done, b.side);
            return e == cudaSuccess ? cudaStreamWaitEvent(st, b.done, 0) : e;
        }
        ~Join() { close(); }
    } update{b, st};
    DVR3D_COUNT_LAUNCH(1);
    copy_panel_kernel<<<(unsigned)(((long long)n * kB + 255) / 256), 256, 0, st>>>(b.A, b.lda, n, std::min(kB, n), P, ld);
    for (int j0 = 0; j0 < n; j0 += kB) {
        const int R = std::max(0, n - j0 - kB);
        double *VWV = b.work + (j0 / kB & 1) * 96 * ld;
        PanelArgs pa{};
        pa.P = P;
        pa.ldp = ld;
        pa.R = R;
        pa.nr = std::max(0, std::min(kB, R - 1));
        pa.V = VWV;
        pa.ldv = ld;
        pa.Vk = b.keep ? b.A + (size_t)j0 * b.lda + j0 + kB : nullptr;
        pa.ldk = b.lda;
        pa.T = b.T + (size_t)(j0 / kB) * 1024;
        pa.C = b.C;
        pa.j0 = j0;
        pa.n = n;
        const PanelPlan pp(R);
        pa.nsm = pp.nsm;
        pa.spill = spill;
        pa.err = b.err;
        pa.limit = b.wait_limit ? b.wait_limit : kPanelPolls;
        {
            ClusterLaunch l(dim3(kCl), (pp.warps + 1) * 32, pp.smem, kCl, 1, st);
            DVR3D_COUNT_LAUNCH(1);
            if ((e = cudaLaunchKernelEx(&l.cfg, panel_qr_kernel, pa)) != cudaSuccess) return e;
        }
        if (R == 0) break;
        if ((e = update.close()) != cudaSuccess) return e;
        double *A2 = b.A + (size_t)(j0 + kB) * b.lda + j0 + kB;
        if (pa.nr == 0) {  // one row left: it lies in the band
            DVR3D_COUNT_LAUNCH(1);
            copy_panel_kernel<<<1, 32, 0, st>>>(A2, b.lda, R, R, P, ld);
            if ((e = cudaGetLastError()) != cudaSuccess) return e;
            continue;
        }
        const int tiles = (R + kBM - 1) / kBM;
        DVR3D_COUNT_LAUNCH(1);
        symm_kernel<<<symm_ctas(R, nsm), kThr, kSymmSmem, st>>>(A2, b.lda, R, VWV, ld, X, ld, part, count);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
        {
            ClusterLaunch l(dim3(kCl), 256, kVtxSmem, kCl, 1, st);
            DVR3D_COUNT_LAUNCH(1);
            if ((e = cudaLaunchKernelEx(&l.cfg, vtx_kernel, (const double *)VWV, ld, (const double *)X, ld, R,
                                        (const double *)pa.T, M)) != cudaSuccess)
                return e;
        }
        DVR3D_COUNT_LAUNCH(1);
        w_kernel<<<tiles, kThr, kWSmem, st>>>(VWV, ld, X, ld, pa.T, M, R, A2, b.lda, P, ld);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
        const int R2 = R - kB;
        if (R2 > 0) {
            const long long nt = (R2 + 63) / 64;
            if ((e = cudaEventRecord(b.ready, st)) != cudaSuccess || (e = cudaStreamWaitEvent(b.side, b.ready, 0)) != cudaSuccess)
                return e;
            update.open = true;
            DVR3D_COUNT_LAUNCH(1);
            syr2k_band_kernel<<<(unsigned)(nt * (nt + 1) / 2), kSyrThr, kSyrSmem, b.side>>>(A2 + (size_t)kB * b.lda + kB, b.lda, R2,
                                                                                      VWV + kB, ld);
            if ((e = cudaGetLastError()) != cudaSuccess) return e;
        }
    }
    return update.close();
}

size_t band_reduce_back_doubles(int nev) { return (size_t)2 * kB * nev + gemm_splitk_work(kB, nev, 64); }

cudaError_t launch_band_reduce_back(const BandReduce &b, double *Z, long long ldz, int nev, double *work, cudaStream_t st) {
    if (nev <= 0) return cudaSuccess;
    if (ldz & 1) return cudaErrorInvalidValue;
    double *Y = work, *Y2 = Y + (size_t)kB * nev, *sk = Y2 + (size_t)kB * nev;
    for (int q = band_reduce_panels(b.n) - 1; q >= 0; --q) {
        const int j0 = q * kB, R = b.n - j0 - kB;
        if (R < 2) continue;
        const double *V = b.A + (size_t)j0 * b.lda + j0 + kB;
        GemmOp g;  // Y = V^T Z
        g.M = kB;
        g.N = nev;
        g.K = R;
        g.A = V;
        g.lda = b.lda;
        g.ta = true;
        g.B = Z + j0 + kB;
        g.ldb = ldz;
        g.C = Y;
        g.ldc = kB;
        const int tiles = (nev + 63) / 64;
        g.splitk = std::max(1, std::min(64, std::min((600 + tiles - 1) / tiles, (R + 15) / 16)));
        g.work = sk;
        cudaError_t e = launch_gemm(g, st);
        if (e != cudaSuccess) return e;
        GemmOp t;  // Y2 = T Y
        t.M = kB;
        t.N = nev;
        t.K = kB;
        t.A = b.T + (size_t)q * 1024;
        t.lda = kB;
        t.B = Y;
        t.ldb = kB;
        t.C = Y2;
        t.ldc = kB;
        if ((e = launch_gemm(t, st)) != cudaSuccess) return e;
        GemmOp u;  // Z -= V Y2
        u.M = R;
        u.N = nev;
        u.K = kB;
        u.alpha = -1.0;
        u.beta = 1.0;
        u.A = V;
        u.lda = b.lda;
        u.B = Y2;
        u.ldb = kB;
        u.C = Z + j0 + kB;
        u.ldc = ldz;
        if ((e = launch_gemm(u, st)) != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace dvr3d
