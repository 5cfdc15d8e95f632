// band_eig.cu -- symmetric band matrix -> tridiagonal by bulge chasing, and the
// back-transformation of eigenvectors, for the projected matrix of the block Krylov solve.
//
// The block Lanczos recurrence makes T = Q^T M Q block tridiagonal: with full
// reorthogonalisation the entries more than one block (b) away from the diagonal are
// rounding-level reorthogonalisation coefficients, so T is a band matrix of half-bandwidth
// b. Instead of the dense one-stage reduction (O(m^2) grid-synchronised column steps) the
// band is chased to tridiagonal form (Schwarz / Lang successive bulge chasing, the
// "band to tridiagonal" stage of two-stage reductions):
//   sweep j, task 0: reflector H_0 annihilating A[j+2 : j+b+1, j]; H_0 applied from both
//                    sides to the diagonal block D_0 (rows/cols R_0 = [j+1, j+b]) and from
//                    the right to the block below it, O_1 = A[R_1, R_0] (which fills: the
//                    bulge);
//   task s >= 1:     H_s annihilates the first column of the bulge O_s below its first
//                    entry, is applied from the left to the rest of O_s, from both sides to
//                    D_s and from the right to O_{s+1}; the remainder of the bulge is
//                    eliminated by later sweeps.
// One CTA owns a whole sweep, keeping O_{s+1} between its tasks. Sweep j+1 may start task s once
// sweep j has written the beta of its task s + 2 (the only entry the two share), published
// through per-sweep progress counters with release / acquire ordering and bounded waits.
// Back-transformation: Q = prod over sweeps (in order) of prod over tasks of H; the
// reflectors of one sweep act on disjoint rows, so a CTA holding a slab of eigenvector
// columns in shared memory applies sweep after sweep (last first), its warps taking the
// tasks of a sweep in parallel.
#include <algorithm>

#include "band_eig.cuh"
#include "common.cuh"

namespace dvr3d {

namespace {

constexpr int kBW = kBandMaxBw;
constexpr int kTS = kBW + 1;            // shared-memory row stride of a block
constexpr int kBlk = kBW * kTS;         // doubles of one 32 x 32 block in shared memory
constexpr unsigned long long kSpinLimit = 1ull << 24;
constexpr unsigned kFull = 0xffffffffu;

__device__ __forceinline__ unsigned ld_acquire_u32(const unsigned *p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void st_release_u32(unsigned *p, unsigned v) {
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

__host__ __device__ __forceinline__ int band_ntask(int n, int b, int j) { return (n - 2 - j) / b + 1; }

__global__ void band_prepare_kernel(double *A, long long lda, int n, int b, unsigned long long *maxbits2) {
    // column j per block-row of threads; rows i > j
    double dropped = 0.0, inside = 0.0;
    const long long tot = (long long)n * n;
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < tot; t += (long long)gridDim.x * blockDim.x) {
        const int j = (int)(t / n), i = (int)(t % n);
        if (i < j) continue;
        double *p = A + (size_t)j * lda + i;
        const double a = fabs(*p);
        if (i - j <= b) inside = fmax(inside, a);
        else {
            dropped = fmax(dropped, a);
            if (i - j <= 2 * b) *p = 0.0;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        dropped = fmax(dropped, __shfl_xor_sync(kFull, dropped, o));
        inside = fmax(inside, __shfl_xor_sync(kFull, inside, o));
    }
    if ((threadIdx.x & 31) == 0) {
        atomicMax(maxbits2, (unsigned long long)__double_as_longlong(dropped));
        atomicMax(maxbits2 + 1, (unsigned long long)__double_as_longlong(inside));
    }
}

// Reflector of a task from its column x (x_0 = alpha, sig = sum of the other squares):
// H = I - tau v v^T, v = (1, sc x_1, sc x_2, ...), H x = beta e_0.
__device__ __forceinline__ void house_scalars(double alpha, double sig, double &tau, double &beta, double &sc) {
    tau = 0.0;
    beta = alpha;
    sc = 0.0;
    if (sig != 0.0) {
        beta = -copysign(sqrt(alpha * alpha + sig), alpha);
        sc = 1.0 / (alpha - beta);
        tau = (beta - alpha) / beta;
    }
}

// One CTA per sweep in flight. The band lives in compact storage (kBandLd doubles a column, both
// triangles within b of the diagonal, bulge space below): element (i, j) at C[j (kBandLd - 1) + i +
// kBW], so a column window is contiguous, nothing is clamped at the matrix end (zero padding) and
// the whole band stays in L2.
// The chase is a dependency chain, so everything is arranged around its length. Task s needs the
// column x that task s - 1 leaves in the bulge; all matrix-vector products of the task are formed
// with x itself (O x, D x, O^T x) beside the norm of x, and the reflector's three scalars are
// computed by every warp for itself, so one barrier (X) a task is all that stands between x and
// the next x. 18 warps:
//   L D (4)  wait for the previous sweep's flag, load task s+1's D and O into registers, then into
//            the raw buffer that task s-1 has left (barrier E);
//   O (4)    O_{s+1} <- O_{s+1} H: eight rows a warp, four lanes a row; the first column is the
//            next x, written first with its partial norms; the whole block goes to shared memory;
//   D (4)    D_s <- H D_s H, kept as a full symmetric block, to global memory;
//   L (4)    O_s <- H O_s (the bulge), to global memory, its first row mirrored above the diagonal;
//   P1       the reflector for the back-transformation, beta;
//   P2       publishes: flag f = reflector f-1 known (beta written) and tasks < f-1 complete
//            (counters in shared memory), the release off the chain.
// Sweep j+1 runs task s once sweep j's flag reaches s + 3: its blocks were completed by task s+1
// and the one entry that task s+2 changes is its beta. Sweeps follow one another at
// (task time) + (flag, fence and load latency): 2656 columns of half-bandwidth 32 (the projected
// matrix of 500 levels) take 17.7 ms, against 27.8 ms for five warps with the reflector broadcast
// through a second barrier and the blocks at the matrix's own stride; 12202 columns 119 ms. Of a
// task's 3400 cycles the D warps need 3000; fence, flag and loads take 1000 + 1900 + 1500.
constexpr int kChaseThreads = 18 * 32;
constexpr int kBarX = 1, kBarE = 3, kBarD = 5;

__device__ __forceinline__ void bar_sync(int id, int count) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(count) : "memory"); }
__device__ __forceinline__ void bar_arrive(int id, int count) { asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(count) : "memory"); }

struct ChaseSmem {
    double raw[2][2][kBlk];  // [buffer][D, O_{s+1}] as loaded
    double bulge[2][kBlk];   // O_s after the right-hand update
    double x[2][kBW];        // the task's column
    double part[2][4];       // its sum of squares without x_0, eight rows each
    double ya[kBW], p2[4];   // D x and x^T D x (without x_0)
    volatile int done[8];    // tasks completed by each of the D and L warps
    volatile int refl;       // reflectors known
    volatile int abort;
};

__global__ void __launch_bounds__(kChaseThreads, 1) band_chase_kernel(BandTri t) {
    extern __shared__ __align__(16) unsigned char chase_sm[];
    ChaseSmem &S = *reinterpret_cast<ChaseSmem *>(chase_sm);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, role = warp >> 2, w = warp & 3;
    const int n = t.n, b = t.b;
    constexpr long long ld = kBandLd - 1;
    constexpr int nX = 17 * 32, nE = 12 * 32;  // X: all but P2; E: O, D and the loaders
    const unsigned long long spin_limit = t.wait_limit ? t.wait_limit : kSpinLimit;
    double *A = t.C + kBW;
    if (tid == 0) S.abort = 0;
    int q = 0;  // tasks of this CTA so far: the parity of buffers and barriers
    for (int j = blockIdx.x; j <= n - 3; j += gridDim.x) {
        const int nt = band_ntask(n, b, j);
        const int ntp = (j > 0) ? band_ntask(n, b, j - 1) : 0;
        if (tid < 8) S.done[tid] = 0;
        if (tid == 8) S.refl = 0;
        __syncthreads();
        if (S.abort) return;
        if (role == 0) {
            // ---- loaders: columns 8w .. 8w+7, lane = row
            unsigned seen = (j > 0) ? 0u : 0xffffffffu;
            for (int s = 0; s < nt; ++s) {
                const int pb = (q + s) & 1;
                const unsigned need = (unsigned)min(s + 3, ntp + 1);
                if (seen < need && !S.abort) {
                    unsigned f = 0;
                    int ok = 1;
                    if (lane == 0) {
                        unsigned long long spins = 0;
                        while ((f = ld_acquire_u32(t.progress + j - 1)) < need) {
                            if (++spins > spin_limit) {
                                atomicExch(t.err, (int)kDevBarrierTimeout);
                                ok = 0;
                                break;
                            }
                            if ((spins & 255ull) == 0 && *(volatile int *)t.err != 0) {
                                ok = 0;
                                break;
                            }
                        }
                        if (!ok) S.abort = 1;  // this sweep runs on without waits; all leave at its end
                    }
                    seen = __shfl_sync(kFull, f, 0);
                }
                __syncwarp();
                const int r0 = j + 1 + s * b, L = min(b, n - r0), r1 = r0 + b, L1 = min(b, n - r1);
                double dv[8], ov[8], xv = 0.0;
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const int c = 8 * w + k;
                    const double *col = A + (long long)(r0 + c) * ld;
                    dv[k] = (c < L && lane < L) ? __ldcg(col + r0 + lane) : 0.0;
                    ov[k] = (c < L && lane < L1) ? __ldcg(col + r1 + lane) : 0.0;
                }
                if (s == 0 && lane < 8 && 8 * w + lane < L) xv = __ldcg(A + (long long)j * ld + r0 + 8 * w + lane);
                if (q + s >= 2) bar_sync(kBarE + pb, nE);
                double *D = S.raw[pb][0], *O = S.raw[pb][1];
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    D[lane * kTS + 8 * w + k] = dv[k];
                    O[lane * kTS + 8 * w + k] = ov[k];
                }
                if (s == 0) {
                    if (lane < 8) S.x[pb][8 * w + lane] = xv;
                    double sq = (w == 0 && lane == 0) ? 0.0 : xv * xv;
                    sq += __shfl_xor_sync(kFull, sq, 4);
                    sq += __shfl_xor_sync(kFull, sq, 2);
                    sq += __shfl_xor_sync(kFull, sq, 1);
                    if (lane == 0) S.part[pb][w] = sq;
                }
                bar_arrive(kBarX + pb, nX);
            }
        } else if (warp < 17) {
            const int rr = lane & 7, cg = lane >> 3, r = 8 * w + rr;
            for (int s = 0; s < nt; ++s) {
                const int pb = (q + s) & 1;
                const int r0 = j + 1 + s * b, L = min(b, n - r0);
                bar_sync(kBarX + pb, nX);
                const double *x = S.x[pb];
                const double alpha = x[0], sig = (S.part[pb][0] + S.part[pb][1]) + (S.part[pb][2] + S.part[pb][3]);
                if (role == 1) {
                    // ---- O_{s+1} <- O_{s+1} H
                    const double *R = S.raw[pb][1] + r * kTS;
                    double o[8], xc[8], a0 = 0.0, a1 = 0.0;
                    const double o0 = R[0];
#pragma unroll
                    for (int k = 0; k < 8; ++k) {
                        o[k] = R[8 * cg + k];
                        xc[k] = (k == 0 && cg == 0) ? 0.0 : x[8 * cg + k];
                    }
#pragma unroll
                    for (int k = 0; k < 8; k += 2) {
                        a0 = fma(o[k], xc[k], a0);
                        a1 = fma(o[k + 1], xc[k + 1], a1);
                    }
                    double a = a0 + a1;
                    a += __shfl_xor_sync(kFull, a, 8);
                    a += __shfl_xor_sync(kFull, a, 16);
                    double tau, beta, sc;
                    house_scalars(alpha, sig, tau, beta, sc);
                    const double tu = tau * fma(sc, a, o0);
                    const double xn = o0 - tu;
                    if (cg == 0) S.x[pb ^ 1][r] = xn;
                    double sq = (r == 0) ? 0.0 : xn * xn;
                    sq += __shfl_xor_sync(kFull, sq, 4);
                    sq += __shfl_xor_sync(kFull, sq, 2);
                    sq += __shfl_xor_sync(kFull, sq, 1);
                    if (lane == 0) S.part[pb ^ 1][w] = sq;
                    double *B = S.bulge[pb ^ 1] + r * kTS + 8 * cg;
                    const double tus = tu * sc;
#pragma unroll
                    for (int k = 0; k < 8; ++k) B[k] = (k == 0 && cg == 0) ? xn : fma(-tus, xc[k], o[k]);
                    bar_arrive(kBarE + pb, nE);
                } else if (role == 2) {
                    // ---- D_s <- H D_s H
                    const double *R = S.raw[pb][0];
                    double d[8], xc[8], a0 = 0.0, a1 = 0.0;
                    const double xr = (r == 0) ? 0.0 : x[r], d0 = R[r * kTS], d00 = R[0];
#pragma unroll
                    for (int k = 0; k < 8; ++k) {
                        d[k] = R[r * kTS + 8 * cg + k];
                        xc[k] = (k == 0 && cg == 0) ? 0.0 : x[8 * cg + k];
                    }
#pragma unroll
                    for (int k = 0; k < 8; k += 2) {
                        a0 = fma(d[k], xc[k], a0);
                        a1 = fma(d[k + 1], xc[k + 1], a1);
                    }
                    double a = a0 + a1;
                    a += __shfl_xor_sync(kFull, a, 8);
                    a += __shfl_xor_sync(kFull, a, 16);
                    if (cg == 0) S.ya[r] = a;
                    double p = xr * a;
                    p += __shfl_xor_sync(kFull, p, 4);
                    p += __shfl_xor_sync(kFull, p, 2);
                    p += __shfl_xor_sync(kFull, p, 1);
                    if (lane == 0) S.p2[w] = p;
                    bar_sync(kBarD, 4 * 32);
                    double tau, beta, sc;
                    house_scalars(alpha, sig, tau, beta, sc);
                    const double p2 = (S.p2[0] + S.p2[1]) + (S.p2[2] + S.p2[3]);
                    // v^T D v with v = e_0 + sc x
                    const double K = fma(sc, fma(sc, p2, 2.0 * S.ya[0]), d00);
                    const double hk = 0.5 * tau * tau * K;
                    const double vr = (r == 0) ? 1.0 : sc * xr;
                    const double wr = fma(-hk, vr, tau * fma(sc, a, d0));
                    double *dst = A + (long long)(r0 + 8 * cg) * ld + r0 + r;
#pragma unroll
                    for (int k = 0; k < 8; ++k) {
                        const double vc = (k == 0 && cg == 0) ? 1.0 : sc * xc[k];
                        const double wc = fma(-hk, vc, tau * fma(sc, S.ya[8 * cg + k], R[(8 * cg + k) * kTS]));
                        // the same rounding for (r, c) and (c, r): the block stays symmetric
                        const double g = __dadd_rn(__dmul_rn(vr, wc), __dmul_rn(wr, vc));
                        if (r < L && 8 * cg + k < L) dst[(long long)k * ld] = d[k] - g;
                    }
                    bar_arrive(kBarE + pb, nE);
                    __syncwarp();
                    if (lane == 0) {
                        __threadfence_block();
                        S.done[w] = s + 1;
                    }
                } else if (role == 3) {
                    // ---- O_s <- H O_s: columns 8w .. 8w+7, four lanes a column
                    if (s > 0) {
                        const int c = 8 * w + (lane >> 2), rg = lane & 3;
                        const double *B = S.bulge[pb] + c;
                        double o[8], xk[8], z0 = 0.0, z1 = 0.0;
                        const double o0 = B[0];
#pragma unroll
                        for (int k = 0; k < 8; ++k) {
                            o[k] = B[(rg + 4 * k) * kTS];
                            xk[k] = (k == 0 && rg == 0) ? 0.0 : x[rg + 4 * k];
                        }
#pragma unroll
                        for (int k = 0; k < 8; k += 2) {
                            z0 = fma(o[k], xk[k], z0);
                            z1 = fma(o[k + 1], xk[k + 1], z1);
                        }
                        double z = z0 + z1;
                        z += __shfl_xor_sync(kFull, z, 1);
                        z += __shfl_xor_sync(kFull, z, 2);
                        double tau, beta, sc;
                        house_scalars(alpha, sig, tau, beta, sc);
                        const double tz = tau * fma(sc, z, o0);
                        const double tzs = tz * sc;
                        if (c < b) {
                            double *dst = A + (long long)(r0 - b + c) * ld + r0;
#pragma unroll
                            for (int k = 0; k < 8; ++k) {
                                const int row = rg + 4 * k;
                                double v = (row == 0) ? o[k] - tz : fma(-tzs, xk[k], o[k]);
                                if (c == 0) v = (row == 0) ? beta : 0.0;
                                if (row < L) dst[row] = v;
                                if (row == 0) A[(long long)r0 * ld + (r0 - b + c)] = v;
                            }
                        }
                        __syncwarp();
                    }
                    if (lane == 0) {
                        __threadfence_block();
                        S.done[4 + w] = s + 1;
                    }
                } else {
                    // ---- P1: the reflector and beta
                    double tau, beta, sc;
                    house_scalars(alpha, sig, tau, beta, sc);
                    if (s == 0) {
                        if (lane < L) A[(long long)j * ld + r0 + lane] = (lane == 0) ? beta : 0.0;
                    } else if (lane == 0) {
                        A[(long long)(r0 - b) * ld + r0] = beta;
                    }
                    __syncwarp();
                    if (lane == 0) {
                        __threadfence_block();
                        S.refl = s + 1;
                    }
                    if (t.vs) {
                        t.vs[((size_t)j * t.ntmax + s) * kBW + lane] = (lane == 0) ? 1.0 : sc * x[lane];
                        if (lane == 0) t.taus[(size_t)j * t.ntmax + s] = tau;
                    }
                }
            }
        } else {
            // ---- P2: publication
            int pub = 0;
            while (pub <= nt) {
                int v = (lane < 8) ? S.done[lane] : 0x7fffffff;
                v = __reduce_min_sync(kFull, v);
                const int refl = S.refl;
                const int f = __shfl_sync(kFull, (v >= nt) ? nt + 1 : min(refl, v + 1), 0);
                if (f > pub) {
                    pub = f;
                    if (lane == 0) {
                        __threadfence_block();  // the counters' values before the release, which covers their writers' stores
                        st_release_u32(t.progress + j, (unsigned)f);
                    }
                }
            }
        }
        q += nt;
        __syncthreads();
    }
}

// The band of a symmetric matrix (lower triangle read) into the chase's compact storage: both
// triangles within b of the diagonal, zeros elsewhere, kBW zero columns at the end.
__global__ void band_compact_kernel(const double *A, long long lda, int n, int b, double *C) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long long)(n + kBW) * kBandLd) return;
    const int j = (int)(t / kBandLd), i = j + (int)(t % kBandLd) - kBW;
    const int lo = min(i, j), hi = max(i, j);
    C[t] = (lo >= 0 && hi < n && hi - lo <= b) ? A[(size_t)lo * lda + hi] : 0.0;
}

__global__ void band_diag_kernel(const double *C, int n, double *d, double *e) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    d[i] = C[(size_t)i * kBandLd + kBW];
    e[i] = (i + 1 < n) ? C[(size_t)i * kBandLd + kBW + 1] : 0.0;
}

// Back-transformation, COLS eigenvector columns per CTA held in shared memory (column c at
// zs + c ldzs, ldzs = 1 mod 16 so the lanes' rows and columns spread over the banks).
// Sweeps are applied last first; the tasks of one sweep act on disjoint rows and are split
// over the 8 warps (task w + 8 k of a chunk of kChunkTasks). In a warp, lane (rg, c) takes
// column c and rows COLS rg .. COLS rg + COLS - 1 of the reflector's window: COLS products,
// a shuffle sum over the 32 / COLS row groups, COLS updates. The reflectors of the next
// chunk are copied into shared memory (cp.async) while the current chunk is applied.
constexpr int kChunkTasks = 96;

__device__ __forceinline__ void cp_async8(double *dst, const double *src) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(src) : "memory");
}

template <int COLS>
__global__ void __launch_bounds__(256) band_bt_kernel(BandTri t, double *Z, long long ldz, int nev, int ldzs) {
    extern __shared__ double sm[];
    double *zs = sm;
    double *vb = sm + (size_t)COLS * ldzs;       // [2][kChunkTasks][kBW]
    double *tb = vb + 2 * kChunkTasks * kBW;     // [2][kChunkTasks]
    const int n = t.n, b = t.b;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int cc = lane % COLS, rg = lane / COLS;
    const int c0 = blockIdx.x * COLS;
    const int ncol = min(COLS, nev - c0);
    for (int q = tid; q < COLS * n; q += blockDim.x) {
        const int c = q / n, r = q - c * n;
        zs[(size_t)c * ldzs + r] = (c < ncol) ? Z[(size_t)(c0 + c) * ldz + r] : 0.0;
    }
    auto stage = [&](int j, int base, int buf) {
        const int cnt = min(kChunkTasks, band_ntask(n, b, j) - base);
        const double *vsrc = t.vs + ((size_t)j * t.ntmax + base) * kBW;
        double *vd = vb + (size_t)buf * kChunkTasks * kBW;
        for (int q = tid; q < cnt * kBW; q += blockDim.x) cp_async8(vd + q, vsrc + q);
        const double *tsrc = t.taus + (size_t)j * t.ntmax + base;
        double *td = tb + buf * kChunkTasks;
        for (int q = tid; q < cnt; q += blockDim.x) cp_async8(td + q, tsrc + q);
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    int j = n - 3, base = 0, buf = 0;
    if (j >= 0) stage(j, base, buf);
    while (j >= 0) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();  // chunk (j, base) staged; the previous chunk's updates are done
        const int cj = j, cbase = base, cbuf = buf;
        base += kChunkTasks;
        if (base >= band_ntask(n, b, j)) {
            --j;
            base = 0;
        }
        buf ^= 1;
        if (j >= 0) stage(j, base, buf);
        const double *vd = vb + (size_t)cbuf * kChunkTasks * kBW;
        const double *td = tb + cbuf * kChunkTasks;
        const int nt = band_ntask(n, b, cj);
        for (int s = cbase + warp; s < nt && s < cbase + kChunkTasks; s += 8) {
            const double tau = td[s - cbase];
            if (tau == 0.0) continue;
            const int r0 = cj + 1 + s * b;
            const double *v = vd + (size_t)(s - cbase) * kBW + rg * COLS;
            double vv[COLS], zz[COLS];
            double part = 0.0;
#pragma unroll
            for (int i = 0; i < COLS; ++i) {
                const int r = min(r0 + rg * COLS + i, n - 1);
                vv[i] = v[i];
                zz[i] = zs[(size_t)cc * ldzs + r];
                part += vv[i] * zz[i];
            }
#pragma unroll
            for (int o = COLS; o < 32; o <<= 1) part += __shfl_xor_sync(kFull, part, o);
            const double f = tau * part;
#pragma unroll
            for (int i = 0; i < COLS; ++i) {
                const int r = r0 + rg * COLS + i;
                if (vv[i] != 0.0 && r < n) zs[(size_t)cc * ldzs + r] = zz[i] - f * vv[i];
            }
        }
    }
    __syncthreads();
    for (int q = tid; q < COLS * n; q += blockDim.x) {
        const int c = q / n, r = q - c * n;
        if (c < ncol) Z[(size_t)(c0 + c) * ldz + r] = zs[(size_t)c * ldzs + r];
    }
}

template <int COLS>
cudaError_t launch_bt(const BandTri &t, double *Z, long long ldz, int nev, int ldzs, size_t smem, cudaStream_t st) {
    cudaError_t e = cudaFuncSetAttribute(band_bt_kernel<COLS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    DVR3D_COUNT_LAUNCH(1);
    band_bt_kernel<COLS><<<(unsigned)((nev + COLS - 1) / COLS), 256, smem, st>>>(t, Z, ldz, nev, ldzs);
    return cudaGetLastError();
}

}  // namespace

size_t band_reflector_doubles(int n, int b) {
    const size_t nt = (size_t)((n - 2) / std::max(b, 1) + 1);
    return (size_t)std::max(n - 2, 1) * nt * kBW;
}

size_t band_tau_doubles(int n, int b) {
    const size_t nt = (size_t)((n - 2) / std::max(b, 1) + 1);
    return (size_t)std::max(n - 2, 1) * nt;
}

cudaError_t launch_band_prepare(double *A, long long lda, int n, int b, unsigned long long *maxbits2,
                                cudaStream_t st) {
    cudaError_t e = cudaMemsetAsync(maxbits2, 0, 2 * sizeof(unsigned long long), st);
    if (e != cudaSuccess) return e;
    DVR3D_COUNT_LAUNCH(1);
    band_prepare_kernel<<<592, 256, 0, st>>>(A, lda, n, b, maxbits2);
    return cudaGetLastError();
}

size_t band_compact_doubles(int n) { return (size_t)(n + kBW) * kBandLd; }

cudaError_t launch_band_compact(const double *A, long long lda, int n, int b, double *C, cudaStream_t st) {
    const long long tot = (long long)(n + kBW) * kBandLd;
    DVR3D_COUNT_LAUNCH(1);
    band_compact_kernel<<<(unsigned)((tot + 255) / 256), 256, 0, st>>>(A, lda, n, b, C);
    return cudaGetLastError();
}

cudaError_t launch_band_chase(BandTri &t, cudaStream_t st) {
    if (t.b < 1 || t.b > kBW || t.n < 3) return cudaErrorInvalidValue;
    t.ntmax = band_ntask(t.n, t.b, 0);
    cudaError_t e = cudaMemsetAsync(t.progress, 0, sizeof(unsigned) * t.n, st);
    if (e != cudaSuccess) return e;
    const size_t smem = sizeof(ChaseSmem);
    e = cudaFuncSetAttribute(band_chase_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    // one CTA per sweep in flight: sweeps follow at least three tasks apart and a CTA is busy
    // for ntask tasks, so ntask / 2 plus slack keeps every sweep's successor supplied
    int grid = std::min(t.n - 2, std::max(8, t.ntmax / 2 + 8));
    int dev = 0, nsm = 0, per = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, band_chase_kernel, kChaseThreads, smem);
    grid = std::max(1, std::min(grid, nsm * std::max(per, 1)));
    void *args[] = {&t};
    DVR3D_COUNT_LAUNCH(1);
    e = cudaLaunchCooperativeKernel((void *)band_chase_kernel, dim3(grid), dim3(kChaseThreads), args, smem, st);
    if (e != cudaSuccess) return e;
    DVR3D_COUNT_LAUNCH(1);
    band_diag_kernel<<<(t.n + 255) / 256, 256, 0, st>>>(t.C, t.n, t.d, t.e);
    return cudaGetLastError();
}

cudaError_t launch_band_backtransform(const BandTri &t, double *Z, long long ldz, int nev, cudaStream_t st) {
    if (nev <= 0 || t.n < 3) return cudaSuccess;
    int optin = 0, dev = 0, nsm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    const int ldzs = (t.n + 15) / 16 * 16 + 1;
    const size_t fixed = (size_t)2 * kChunkTasks * (kBW + 1) * sizeof(double);
    auto need = [&](int cols) { return fixed + (size_t)cols * ldzs * sizeof(double); };
    // widest slab that fits, but no wider than keeps every SM busy
    int cols = 8;
    while (cols > 1 && (need(cols) > (size_t)optin || (nev + cols - 1) / cols < nsm)) cols /= 2;
    if (need(cols) > (size_t)optin) return cudaErrorInvalidValue;
    switch (cols) {
        case 8: return launch_bt<8>(t, Z, ldz, nev, ldzs, need(8), st);
        case 4: return launch_bt<4>(t, Z, ldz, nev, ldzs, need(4), st);
        case 2: return launch_bt<2>(t, Z, ldz, nev, ldzs, need(2), st);
        default: return launch_bt<1>(t, Z, ldz, nev, ldzs, need(1), st);
    }
}

}  // namespace dvr3d
