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
// sweep j has formed the beta of its task s + 2 (the only entry the two share).
// Back-transformation: Q = prod over sweeps (in order) of prod over tasks of H; the
// reflectors of one sweep act on disjoint rows, so a CTA holding a slab of eigenvector
// columns in shared memory applies sweep after sweep (last first), its warps taking the
// tasks of a sweep in parallel.
#include <cooperative_groups.h>

#include <algorithm>

#include "band_eig.cuh"
#include "cluster_dev.cuh"
#include "common.cuh"

namespace dvr3d {

namespace {

constexpr int kBW = kBandMaxBw;
constexpr int kTS = kBW + 1;            // shared-memory row stride of a block
constexpr int kBlk = kBW * kTS;         // doubles of one 32 x 32 block in shared memory
constexpr int kSlotDoubles = 2 * kBlk + 2;  // doubles of a slot of the chase
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

// One CTA per sweep in flight, sixteen consecutive sweeps a thread-block cluster. The chase is a
// dependency chain: task s of sweep j+1 needs what tasks s, s+1 of sweep j leave and the beta of its
// task s+2, so sweeps follow one another at about two task times plus one hand-off, and everything is
// arranged around these. A sweep's results are put together in slots, one a task, already shifted to
// the next sweep's window: D(r,c) = D_s(r+1,c+1), its last row and column the first row of O_{s+1}
// and D_{s+1}(0,0); O(r,c) = O_{s+1}(r+1,c+1), its last column D_{s+1}(r+1,0) and, apart from the
// block, the beta of task s+2. A slot is complete, and leaves, when task s+2 begins; parts that a
// sweep's last tasks do not have are zeros. Inside a cluster it goes to the next CTA's ring of slots
// in one bulk copy that an mbarrier counts (no flag, no trip through L2), with credits for the slots
// coming back. The last CTA of a cluster copies its slots to global memory behind a flag, where the
// first CTA of the next one fetches them; one buffer serves all, since a slot is written only after
// every earlier sweep has used it. The band itself enters as the slots of sweep 0.
// A task needs the column x that the task before left in the bulge; all its products are formed with
// x itself (O x, D x, O^T x) while one warp forms the reflector's scalars from its norm, so the
// barriers X (x is known) and Y (the scalars are) are all that a task waits for. 16 warps:
//   LD (1)   first CTA: waits for the flag, fetches slots into the ring; others: returns the ring's
//            credits;
//   ST (1)   sends the slots (fences and remote arrivals take longer than the scalars);
//   P1 (1)   the scalars; the betas; e, the reflector for the back-transformation;
//   O (4)    O_{s+1} <- O_{s+1} H: eight rows a warp, four lanes a row; the first column is the next
//            x, written first with its partial norms; the whole block goes to shared memory;
//   D (4)    D_s <- H D_s H, kept as a full symmetric block;
//   L (4)    O_s <- H O_s (the bulge).
// Half-bandwidth 32: 2656 columns (the projected matrix of 500 levels) 27.8 -> 9.7 ms, 913 columns 3.2
// ms, 12202 columns 119 (before slots, every sweep through L2) -> 49 ms. A task takes 1.15 us, of it
// 0.32 the scalars and 0.6 the D warps' chain through shared memory; sweeps follow at 3.5 us, 6.6
// across clusters. Seven clusters of sixteen fit a B200 (fifteen of eight: 50 ms, more hand-offs
// through L2).
constexpr int kChaseThreads = 16 * 32;
constexpr int kChaseCluster = 16;
constexpr int kRing = 5;
constexpr int kBarX = 1, kBarD = 3, kBarY = 4;  // kBarY + role: the scalars reach each group by itself

// Bulk copies of `bytes` (a multiple of 16): to another CTA's shared memory, from and to global memory.
__device__ __forceinline__ void bulk_to_cta(unsigned dst, unsigned src, unsigned bytes, unsigned bar) {
    asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "r"(src),
                 "r"(bytes), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void bulk_load(unsigned dst, const void *src, unsigned bytes, unsigned bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src),
                 "r"(bytes), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void bulk_store_wait(void *dst, unsigned src, unsigned bytes) {
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(src), "r"(bytes) : "memory");
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
    asm volatile("cp.async.bulk.wait_group 0;\n\tfence.proxy.async;" ::: "memory");
}
__device__ __forceinline__ void fence_async() { asm volatile("fence.proxy.async;" ::: "memory"); }

__device__ __forceinline__ void load8(double (&v)[8], const double *p) {  // 16-byte aligned
#pragma unroll
    for (int k = 0; k < 8; k += 2) {
        const double2 q = *reinterpret_cast<const double2 *>(p + k);
        v[k] = q.x;
        v[k + 1] = q.y;
    }
}

struct alignas(16) ChaseSlot {
    double d[kBlk], o[kBlk];  // [column][row]
    double beta, pad;         // last element of o
};
static_assert(sizeof(ChaseSlot) == kSlotDoubles * sizeof(double) && sizeof(ChaseSlot) % 16 == 0, "slots are copied in bulk");

struct alignas(128) ChaseSmem {
    ChaseSlot raw[kRing];      // the sweep's input
    ChaseSlot stage[kRing];    // the next sweep's, until they are complete
    double bulge[2][kBlk];     // O_s after the right-hand update, [column][row]
    alignas(16) double x[2][kBW];  // the task's column
    double xin[kBW];           // the sweep's first column
    double xout[kBW];          // the next sweep's
    double part[2][4];         // the column's sum of squares without x_0, eight rows each
    double scal[2][4];         // the reflector: tau, beta, sc
    alignas(16) double ya[kBW];
    double p2[4];              // D x and x^T D x (without x_0)
    unsigned long long full[kRing], fullx;  // slots of the ring and xin filled
    unsigned long long own[kRing];          // first CTA: slots of its ring free again
    unsigned long long credit[kRing];       // staged slots free again, here and at the next CTA
    volatile int tasks, refl;               // tasks begun; reflectors known, their betas staged
    volatile int abort;
    int slots_in, firsts_in;                // slots and first columns sent to this CTA in all
};

__global__ void __launch_bounds__(kChaseThreads, 1) band_chase_kernel(BandTri t) {
    extern __shared__ __align__(128) unsigned char chase_sm[];
    ChaseSmem &S = *reinterpret_cast<ChaseSmem *>(chase_sm);
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, role = warp >> 2, w = warp & 3;
    const int n = t.n, b = t.b;
    const int K = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
    const bool first = rank == 0, last = rank == K - 1;
    constexpr int nX = 13 * 32;  // O, D, L and P1
    constexpr unsigned slot_bytes = sizeof(ChaseSlot), block_bytes = 2 * kBlk * 8;
    const unsigned x_bytes = 8u * (unsigned)b;
    const unsigned long long flag_limit = t.wait_limit ? t.wait_limit : kSpinLimit;
    const unsigned long long smem_limit = t.wait_limit ? t.wait_limit : 4 * kSpinLimit;
    ChaseSlot *G = reinterpret_cast<ChaseSlot *>(t.slots);  // [0]: first column, [1 + s]: slot s
    for (int q = tid; q < (int)(2 * kRing * sizeof(ChaseSlot) / 8); q += kChaseThreads) reinterpret_cast<double *>(S.raw)[q] = 0.0;
    if (tid < kBW) S.xin[tid] = S.xout[tid] = 0.0;
    if (tid == 0) {
        S.abort = S.slots_in = S.firsts_in = 0;
        for (int q = 0; q < kRing; ++q) {
            mbar_init(smem_u32(&S.full[q]), 1);
            mbar_init(smem_u32(&S.own[q]), 1);
            mbar_init(smem_u32(&S.credit[q]), 1);
        }
        mbar_init(smem_u32(&S.fullx), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        if (!first) {
            for (int q = 0; q < kRing; ++q) mbar_expect(smem_u32(&S.full[q]), block_bytes + 8);
            mbar_expect(smem_u32(&S.fullx), x_bytes);
        }
    }
    cluster.sync();
    // bounded wait for a phase of one of this CTA's barriers; when it runs out the CTA runs on
    // without waits to the end of its sweep, and leaves
    auto wait = [&](unsigned long long *bar, unsigned parity) {
        const unsigned a = smem_u32(bar);
        unsigned long long spins = 0;
        while (!mbar_test(a, parity)) {
            if (S.abort) return;
            ++spins;
            if ((spins & 1023ull) == 0 && *(volatile int *)t.err != 0) S.abort = 1;
            if (spins > smem_limit) {
                atomicExch(t.err, (int)kDevBarrierTimeout);
                S.abort = 1;
            }
        }
    };
    // the same address in the next and the previous CTA of the cluster
    const unsigned noff = map_rank(smem_u32(&S), (unsigned)(last ? rank : rank + 1)) - smem_u32(&S);
    const unsigned poff = map_rank(smem_u32(&S), (unsigned)(first ? rank : rank - 1)) - smem_u32(&S);
    auto rem = [&](const void *p) { return smem_u32(p) + noff; };
    int q = 0;       // tasks of this CTA so far: the parity of buffers and barriers
    int in0 = 0;     // slots of this CTA's ring consumed by earlier sweeps
    int out0 = 0;    // slots sent by earlier sweeps
    int sweeps = 0;  // sweeps so far
    int blocks = 0, betas = 0, firsts = 0;  // sent to the next CTA by this thread
    int expected = 1;                       // first columns that this thread has told fullx to expect
    for (int j = (int)(blockIdx.x / K) * K + rank; j <= n - 3; j += gridDim.x, ++sweeps) {
        const int nt = band_ntask(n, b, j);
        const int ntp = (j > 0) ? band_ntask(n, b, j - 1) : 0;
        const bool send = j + 1 <= n - 3, near = send && !last, far = send && last;  // next CTA; global memory
        if (tid == 0) S.refl = S.tasks = 0;
        __syncthreads();
        const int gave_up = S.abort;
        __syncthreads();
        if (gave_up) break;
        // last CTA: slot s to global memory (s < 0: the first column), then its flag and credit
        auto copy_out = [&](int s) {
            if (s < 0) {
                for (int c = 0; c < b; ++c) G->d[c] = S.xout[c];
            } else {
                const int u = (out0 + s) % kRing;
                fence_async();
                bulk_store_wait(G + 1 + s, smem_u32(&S.stage[u]), slot_bytes);
                mbar_arrive(smem_u32(&S.credit[u]));
            }
            st_release_u32(t.progress + j, (unsigned)(s + 2));
        };
        auto give_back = [&](int m) {
            const int u = m % kRing;
            mbar_expect(smem_u32(&S.full[u]), block_bytes + 8);
            mbar_arrive_remote(smem_u32(&S.credit[u]) + poff);
        };
        if (role == 0 && w == 0) {
            if (first && lane == 0) {
                // ---- LD
                unsigned seen = (j > 0) ? 0u : 0xffffffffu;
                for (int s = -1; s < nt; ++s) {
                    unsigned long long spins = 0;
                    while (seen < (unsigned)(s + 2) && !S.abort) {
                        seen = ld_acquire_u32(t.progress + j - 1);
                        if (++spins > flag_limit) {
                            atomicExch(t.err, (int)kDevBarrierTimeout);
                            S.abort = 1;
                        }
                        if ((spins & 255ull) == 0 && *(volatile int *)t.err != 0) S.abort = 1;
                    }
                    if (s < 0) {
                        for (int c = 0; c < b; ++c) S.xin[c] = __ldcg(&G->d[c]);
                        mbar_arrive(smem_u32(&S.fullx));
                    } else {
                        const int m = in0 + s, sl = m % kRing;
                        wait(&S.own[sl], ((m / kRing) & 1) ^ 1);
                        if (!S.abort) {
                            mbar_expect(smem_u32(&S.full[sl]), slot_bytes);
                            fence_async();
                            bulk_load(smem_u32(&S.raw[sl]), G + 1 + s, slot_bytes, smem_u32(&S.full[sl]));
                            S.slots_in = m + 1;
                        }
                    }
                }
            } else if (!first && lane == 0) {
                // credits: slot s is read when task s + 1 begins, or the sweep ends; one more slot
                // where the sweep before had one task more
                for (int s = -1; s + 1 < nt && !S.abort; ++s) {
                    while (S.tasks < s + 2 && !S.abort) {}
                    if (S.abort) break;
                    if (s < 0) {  // the first column, for the next sweep
                        mbar_expect(smem_u32(&S.fullx), x_bytes);
                        ++expected;
                    } else {
                        give_back(in0 + s);
                    }
                }
            }
        } else if (role == 0 && w == 1) {
            if (near && lane == 0) {
                // ---- ST: slot s is complete when task s + 2 begins (its beta goes by itself)
                for (int s = 0; s + 2 < nt && !S.abort; ++s) {
                    while (S.tasks < s + 3 && !S.abort) {}
                    if (S.abort) break;
                    const int u = (out0 + s) % kRing;
                    fence_async();
                    bulk_to_cta(rem(&S.raw[u]), smem_u32(&S.stage[u]), block_bytes, rem(&S.full[u]));
                    blocks = out0 + s + 1;
                }
            } else if (far && lane == 0) {
                // the first column is known with task 1's beta, slot s with task s + 2's
                for (int s = -1; s + 2 < nt && !S.abort; ++s) {
                    while (S.refl < s + 3 && !S.abort) {}
                    __threadfence_block();
                    if (!S.abort) copy_out(s);
                }
            }
        } else if (role > 0 || w == 2) {
            const int rr = lane & 7, cg8 = lane >> 3, r = 8 * w + rr;
            // D: where this thread's elements go in a slot, and which of its columns do
            const int off = (8 * cg8 - 1) * kTS + r - 1, ecol = (b - 1) * kTS + (r == 0 ? b - 1 : kBlk + r - 1);
            unsigned cols = 0;
#pragma unroll
            for (int k = 0; k < 8; ++k)
                if (r >= 1 && r < b && 8 * cg8 + k >= 1 && 8 * cg8 + k < b) cols |= 1u << k;
            if (role == 1) {  // the first column
                wait(&S.fullx, sweeps & 1);
                double xv = (cg8 == 0) ? S.xin[r] : 0.0;
                if (cg8 == 0) S.x[q & 1][r] = xv;
                double sq = (r == 0) ? 0.0 : xv * xv;
                sq += __shfl_xor_sync(kFull, sq, 4);
                sq += __shfl_xor_sync(kFull, sq, 2);
                sq += __shfl_xor_sync(kFull, sq, 1);
                if (lane == 0) S.part[q & 1][w] = sq;
            }
            for (int s = 0; s < nt; ++s) {
                const int pb = (q + s) & 1, m = in0 + s, sl = m % kRing;
                // this task's staged slot and the two before it
                const int o = out0 + s, so = o % kRing, so1 = (o + kRing - 1) % kRing, so2 = (o + kRing - 2) % kRing;
                const bool end = s + 1 == nt, snd = send && !S.abort;
                bar_sync(kBarX + pb, nX);
                const double *x = S.x[pb];
                if (role == 1) {
                    // ---- O_{s+1} <- O_{s+1} H
                    double xc[8];
                    load8(xc, x + 8 * cg8);
                    if (cg8 == 0) xc[0] = 0.0;
                    wait(&S.full[sl], (m / kRing) & 1);
                    const double *R = S.raw[sl].o + r;
                    double o8[8], a0 = 0.0, a1 = 0.0;
                    const double o0 = R[0];
#pragma unroll
                    for (int k = 0; k < 8; ++k) o8[k] = R[(8 * cg8 + k) * kTS];
                    if (r == b - 1 && cg8 == (b - 1) / 8) {
                        const double bt = S.raw[sl].beta;
#pragma unroll
                        for (int k = 0; k < 8; ++k)
                            if (k == (b - 1) % 8) o8[k] = bt;
                    }
#pragma unroll
                    for (int k = 0; k < 8; k += 2) {
                        a0 = fma(o8[k], xc[k], a0);
                        a1 = fma(o8[k + 1], xc[k + 1], a1);
                    }
                    double a = a0 + a1;
                    a += __shfl_xor_sync(kFull, a, 8);
                    a += __shfl_xor_sync(kFull, a, 16);
                    bar_sync(kBarY + role, 5 * 32);
                    const double tau = S.scal[pb][0], sc = S.scal[pb][2];
                    const double tu = tau * fma(sc, a, o0);
                    const double xn = o0 - tu;
                    if (cg8 == 0) S.x[pb ^ 1][r] = xn;
                    double sq = (r == 0) ? 0.0 : xn * xn;
                    sq += __shfl_xor_sync(kFull, sq, 4);
                    sq += __shfl_xor_sync(kFull, sq, 2);
                    sq += __shfl_xor_sync(kFull, sq, 1);
                    if (lane == 0) S.part[pb ^ 1][w] = sq;
                    double *B = S.bulge[pb ^ 1] + 8 * cg8 * kTS + r;
                    const double tus = tu * sc;
#pragma unroll
                    for (int k = 0; k < 8; ++k) B[k * kTS] = (k == 0 && cg8 == 0) ? xn : fma(-tus, xc[k], o8[k]);
                } else if (role == 2) {
                    // ---- D_s <- H D_s H
                    double d[8], xc[8], a0 = 0.0, a1 = 0.0;
                    load8(xc, x + 8 * cg8);
                    if (cg8 == 0) xc[0] = 0.0;
                    const double xr = (r == 0) ? 0.0 : x[r];
                    wait(&S.full[sl], (m / kRing) & 1);
                    const double *R = S.raw[sl].d;
                    const double d0 = R[r], d00 = R[0];
#pragma unroll
                    for (int k = 0; k < 8; ++k) d[k] = R[(8 * cg8 + k) * kTS + r];
#pragma unroll
                    for (int k = 0; k < 8; k += 2) {
                        a0 = fma(d[k], xc[k], a0);
                        a1 = fma(d[k + 1], xc[k + 1], a1);
                    }
                    double a = a0 + a1;
                    a += __shfl_xor_sync(kFull, a, 8);
                    a += __shfl_xor_sync(kFull, a, 16);
                    if (cg8 == 0) S.ya[r] = a;
                    double p = xr * a;
                    p += __shfl_xor_sync(kFull, p, 4);
                    p += __shfl_xor_sync(kFull, p, 2);
                    p += __shfl_xor_sync(kFull, p, 1);
                    if (lane == 0) S.p2[w] = p;
                    if (snd) wait(&S.credit[so], ((o / kRing) & 1) ^ 1);
                    bar_sync(kBarD, 4 * 32);
                    double ys[8], dc[8];
                    load8(ys, S.ya + 8 * cg8);
                    load8(dc, R + 8 * cg8);  // the first column
                    const double p2 = (S.p2[0] + S.p2[1]) + (S.p2[2] + S.p2[3]), ya0 = S.ya[0];
                    bar_sync(kBarY + role, 5 * 32);
                    const double tau = S.scal[pb][0], sc = S.scal[pb][2];
                    // v^T D v with v = e_0 + sc x
                    const double Kq = fma(sc, fma(sc, p2, 2.0 * ya0), d00);
                    const double hk = 0.5 * tau * tau * Kq;
                    const double vr = (r == 0) ? 1.0 : sc * xr;
                    const double wr = fma(-hk, vr, tau * fma(sc, a, d0));
#pragma unroll
                    for (int k = 0; k < 8; ++k) {
                        const double vc = (k == 0 && cg8 == 0) ? 1.0 : sc * xc[k];
                        const double wc = fma(-hk, vc, tau * fma(sc, ys[k], dc[k]));
                        // the same rounding for (r, c) and (c, r): the block stays symmetric
                        d[k] -= __dadd_rn(__dmul_rn(vr, wc), __dmul_rn(wr, vc));
                    }
                    if (s == 0 && cg8 == 0) {
                        if (r == 0) t.d[j + 1] = d[0];
                        if (j == n - 3 && r == 1) {
                            t.e[n - 2] = d[0];
                            t.d[n - 1] = d[1];
                            t.e[n - 1] = 0.0;
                        }
                    }
                    if (snd) {
                        double *T = S.stage[so].d, *Tc = T + off;
#pragma unroll
                        for (int k = 0; k < 8; ++k)
                            if (cols & (1u << k)) Tc[k * kTS] = d[k];
                        if (cg8 == 0 && r < b) {  // the first column
                            if (s > 0) S.stage[so1].d[ecol] = d[0];
                            else if (r >= 1) S.xout[r - 1] = d[0];
                            if (end) T[ecol] = 0.0;  // task s + 1 has none
                        }
                    }
                } else if (role == 3) {
                    // ---- O_s <- H O_s: columns 8w .. 8w+7, four lanes a column
                    const int c = 8 * w + rr;
                    const double *B = S.bulge[pb] + c * kTS + 8 * cg8;
                    double o8[8], xk[8], z0 = 0.0, z1 = 0.0;
                    const double o0 = S.bulge[pb][c * kTS];
                    load8(xk, x + 8 * cg8);
                    if (cg8 == 0) xk[0] = 0.0;
#pragma unroll
                    for (int k = 0; k < 8; ++k) o8[k] = B[k];
#pragma unroll
                    for (int k = 0; k < 8; k += 2) {
                        z0 = fma(o8[k], xk[k], z0);
                        z1 = fma(o8[k + 1], xk[k + 1], z1);
                    }
                    double z = z0 + z1;
                    z += __shfl_xor_sync(kFull, z, 8);
                    z += __shfl_xor_sync(kFull, z, 16);
                    bar_sync(kBarY + role, 5 * 32);
                    const double tau = S.scal[pb][0], sc = S.scal[pb][2];
                    const double tz = tau * fma(sc, z, o0);
                    const double tzs = tz * sc;
                    auto put = [&](ChaseSlot &T, bool zero) {
                        if (c < 1 || c >= b) return;
                        double *od = T.o + (c - 1) * kTS + 8 * cg8 - 1;
#pragma unroll
                        for (int k = 0; k < 8; ++k) {
                            const double v = zero ? 0.0 : fma(-tzs, xk[k], o8[k]);
                            if (k > 0 || cg8 > 0) {
                                if (8 * cg8 + k < b) od[k] = v;
                            } else {  // the first row
                                T.d[(c - 1) * kTS + b - 1] = T.d[(b - 1) * kTS + c - 1] = zero ? 0.0 : o8[0] - tz;
                            }
                        }
                    };
                    if (snd && s > 0) put(S.stage[so1], false);
                    if (snd && end) {  // zeros for O_{s+1}, which task s + 1 does not finish
                        wait(&S.credit[so], ((o / kRing) & 1) ^ 1);
                        put(S.stage[so], true);
                    }
                } else {
                    // ---- P1
                    if (lane == 0) S.tasks = s + 1;
                    const double alpha = x[0], sig = (S.part[pb][0] + S.part[pb][1]) + (S.part[pb][2] + S.part[pb][3]);
                    double tau, beta, sc;
                    house_scalars(alpha, sig, tau, beta, sc);
                    if (lane == 0) {
                        S.scal[pb][0] = tau;
                        S.scal[pb][1] = beta;
                        S.scal[pb][2] = sc;
                    }
                    __syncwarp();
#pragma unroll
                    for (int g = 1; g <= 3; ++g) bar_arrive(kBarY + g, 5 * 32);
                    if (near && s == 1 && __all_sync(kFull, !S.abort)) {  // all of it or nothing
                        if (lane < b) st_async(rem(&S.xin[lane]), (lane == b - 1) ? beta : S.xout[lane], rem(&S.fullx));
                        ++firsts;
                    }
                    if (near && s >= 2 && lane == 0 && !S.abort) {
                        st_async(rem(&S.raw[so2].beta), beta, rem(&S.full[so2]));
                        betas = o - 1;
                    }
                    if (far && lane == 0) {
                        if (s == 1) S.xout[b - 1] = beta;
                        if (s >= 2) S.stage[so2].beta = beta;
                        __threadfence_block();
                        S.refl = s + 1;
                    }
                    // the slot that the task before has read is free
                    if (first && lane == 0 && s > 0 && !S.abort) mbar_arrive(smem_u32(&S.own[(m - 1) % kRing]));
                    if (s == 0 && lane == 0) {
                        t.e[j] = beta;
                        if (j == 0) t.d[0] = G->beta;
                    }
                    if (t.vs) {
                        t.vs[((size_t)j * t.ntmax + s) * kBW + lane] = (lane == 0) ? 1.0 : sc * x[lane];
                        if (lane == 0) t.taus[(size_t)j * t.ntmax + s] = tau;
                    }
                }
            }
        }
        __syncthreads();
        // the last two slots (and the first column of a sweep of one task); the betas of tasks nt and
        // nt + 1 are zero
        if (near && warp == 2 && __all_sync(kFull, !S.abort)) {
            if (nt == 1) {
                if (lane < b) st_async(rem(&S.xin[lane]), (lane == b - 1) ? 0.0 : S.xout[lane], rem(&S.fullx));
                ++firsts;
            }
            if (lane == 0) {
                fence_async();
                for (int s = max(0, nt - 2); s < nt; ++s) {
                    const int u = (out0 + s) % kRing;
                    bulk_to_cta(rem(&S.raw[u]), smem_u32(&S.stage[u]), block_bytes, rem(&S.full[u]));
                    st_async(rem(&S.raw[u].beta), 0.0, rem(&S.full[u]));
                }
                blocks = betas = out0 + nt;
            }
        }
        if (far && warp == 1 && lane == 0 && !S.abort) {
            if (nt == 1) {
                S.xout[b - 1] = 0.0;
                copy_out(-1);
            }
            for (int s = max(0, nt - 2); s < nt; ++s) {
                S.stage[(out0 + s) % kRing].beta = 0.0;
                copy_out(s);
            }
        }
        // credits for the last slot, and for the one that the sweep before had more
        if (warp == 2 && lane == 0 && !S.abort) {
            if (first) mbar_arrive(smem_u32(&S.own[(in0 + nt - 1) % kRing]));
            else
                for (int s = nt - 1; s < ntp; ++s) {
                    const int m = in0 + s;
                    if (s >= nt) wait(&S.full[m % kRing], (m / kRing) & 1);
                    if (S.abort) break;
                    give_back(m);
                }
        }
        q += nt;
        in0 += first ? nt : ntp;
        if (send) out0 += nt;
    }
    // Nobody leaves with a copy into its shared memory on the way, given up or not: a sender makes whole
    // what it has begun (a slot of which only the block or only the beta has gone: the receiver has
    // given its credit, so it expects the other part too) and says how much that was; then the
    // receiver waits for the last phases of these barriers, whether or not it has read the slots.
    if (warp == 1 && lane == 0) S.tasks = blocks;
    __syncthreads();
    if (warp == 2 && lane == 0 && !last) {
        blocks = max(blocks, S.tasks);
        const int whole = max(blocks, betas);
        fence_async();
        for (int m = min(blocks, betas); m < whole; ++m) {
            const int u = m % kRing;
            if (m >= blocks) bulk_to_cta(rem(&S.raw[u]), smem_u32(&S.stage[u]), block_bytes, rem(&S.full[u]));
            else st_async(rem(&S.raw[u].beta), 0.0, rem(&S.full[u]));
        }
        *cluster.map_shared_rank(&S.slots_in, rank + 1) = whole;
        *cluster.map_shared_rank(&S.firsts_in, rank + 1) = firsts;
    }
    cluster.sync();
    if (tid == 0) {
        auto arrived = [&](unsigned long long *bar, unsigned phase) {
            for (unsigned long long spins = 0; spins < 4 * kSpinLimit && !mbar_test(smem_u32(bar), phase & 1); ++spins) {}
        };
        const int slots = S.slots_in;
        for (int m = max(0, slots - kRing); m < slots; ++m) arrived(&S.full[m % kRing], m / kRing);
        if (S.firsts_in > expected) mbar_expect(smem_u32(&S.fullx), x_bytes);  // gave up before it came to that
        if (S.firsts_in > 0) arrived(&S.fullx, S.firsts_in - 1);
    }
    cluster.sync();
}

// The band of a symmetric matrix (lower triangle read, element (i, j) at A[j lda + i]) as the slots
// of the first sweep.
__global__ void band_slots_kernel(const double *A, long long lda, int n, int b, int nt, double *slots) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long long)(nt + 1) * kSlotDoubles) return;
    const int s = (int)(t / kSlotDoubles) - 1, e = (int)(t % kSlotDoubles);
    int i = -1, j = -1;
    if (s < 0) {  // the first column, and the first diagonal element
        if (e < b) i = 1 + e, j = 0;
        else if (e == 2 * kBlk) i = j = 0;
    } else {
        const int r0 = 1 + s * b, c = (e % kBlk) / kTS, r = (e % kBlk) % kTS;
        if (e < kBlk) i = r0 + r, j = r0 + c;
        else if (e < 2 * kBlk) i = r0 + b + r, j = r0 + c;
        if (e < 2 * kBlk && (r >= b || c >= b)) i = -1;
        if (e >= kBlk && r == b - 1) i = -1;
        if (e == 2 * kBlk) i = r0 + 2 * b - 1, j = r0 + b - 1;
    }
    double v = 0.0;
    if (i >= 0 && i < n && j < n) {
        const int lo = min(i, j), hi = max(i, j);
        if (hi - lo <= b) v = A[(size_t)lo * lda + hi];
    }
    slots[t] = v;
}

// Back-transformation, COLS eigenvector columns per CTA held in shared memory (column c at
// zs + c ldzs, ldzs = 1 mod 16 so the lanes' rows and columns spread over the banks).
// Sweeps are applied last first; the tasks of one sweep act on disjoint rows and are split
// over the warps (task w + kBtWarps k of a chunk of kChunkTasks). In a warp, lane (rg, c) takes
// column c and rows COLS rg .. COLS rg + COLS - 1 of the reflector's window: COLS products,
// a shuffle sum over the 32 / COLS row groups, COLS updates. The reflectors of the next
// chunk are copied into shared memory (cp.async) while the current chunk is applied.
// A task is a chain of loads, products, shuffles and stores (some 250 cycles), and a sweep a few of
// them and a barrier; so a warp takes several tasks at once, loads first.
// 330 vectors of order 1600 take 1.75 ms, 532 of order 2656 3.9 (2.1 and 5.1 with two columns a CTA
// and a task at a time).
constexpr int kChunkTasks = 96;
constexpr int kBtWarps = 8;

__device__ __forceinline__ void cp_async8(double *dst, const double *src) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(src) : "memory");
}

template <int COLS>
__global__ void __launch_bounds__(32 * kBtWarps) band_bt_kernel(BandTri t, double *Z, long long ldz, int nev, int ldzs) {
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
        constexpr int U = COLS < 8 ? 3 : 2;  // tasks at once; kBtWarps U divides kChunkTasks
        const int send = min(nt, cbase + kChunkTasks);
        for (int s0 = cbase + warp; s0 < send; s0 += kBtWarps * U) {
            double tau[U], vv[U][COLS], zz[U][COLS], part[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int s = s0 + kBtWarps * u, r0 = cj + 1 + s * b + rg * COLS;
                tau[u] = (s < send) ? td[s - cbase] : 0.0;
                const double *v = vd + (size_t)(s - cbase) * kBW + rg * COLS;
                part[u] = 0.0;
#pragma unroll
                for (int i = 0; i < COLS; ++i) {
                    vv[u][i] = (tau[u] != 0.0) ? v[i] : 0.0;
                    zz[u][i] = zs[(size_t)cc * ldzs + min(r0 + i, n - 1)];
                    part[u] += vv[u][i] * zz[u][i];
                }
            }
#pragma unroll
            for (int o = COLS; o < 32; o <<= 1)
#pragma unroll
                for (int u = 0; u < U; ++u) part[u] += __shfl_xor_sync(kFull, part[u], o);
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int r0 = cj + 1 + (s0 + kBtWarps * u) * b + rg * COLS;
                const double f = tau[u] * part[u];
#pragma unroll
                for (int i = 0; i < COLS; ++i)
                    if (vv[u][i] != 0.0 && r0 + i < n) zs[(size_t)cc * ldzs + r0 + i] = zz[u][i] - f * vv[u][i];
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
    band_bt_kernel<COLS><<<(unsigned)((nev + COLS - 1) / COLS), 32 * kBtWarps, smem, st>>>(t, Z, ldz, nev, ldzs);
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

size_t band_slot_doubles(int n, int b) { return (size_t)(band_ntask(n, b, 0) + 1) * kSlotDoubles; }

cudaError_t launch_band_slots(const double *A, long long lda, int n, int b, double *slots, cudaStream_t st) {
    const long long tot = (long long)band_slot_doubles(n, b);
    DVR3D_COUNT_LAUNCH(1);
    band_slots_kernel<<<(unsigned)((tot + 255) / 256), 256, 0, st>>>(A, lda, n, b, band_ntask(n, b, 0), slots);
    return cudaGetLastError();
}

cudaError_t launch_band_chase(BandTri &t, cudaStream_t st) {
    if (t.b < 2 || t.b > kBW || t.n < 3) return cudaErrorInvalidValue;
    t.ntmax = band_ntask(t.n, t.b, 0);
    cudaError_t e = cudaMemsetAsync(t.progress, 0, sizeof(unsigned) * t.n, st);
    if (e != cudaSuccess) return e;
    const int smem = (int)sizeof(ChaseSmem);
    if ((e = cudaFuncSetAttribute(band_chase_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem)) != cudaSuccess) return e;
    if ((e = cudaFuncSetAttribute(band_chase_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1)) != cudaSuccess) return e;
    // sweeps follow at least two tasks apart and a CTA is busy for ntask tasks, so ntask / 2 plus
    // slack keeps every sweep's successor supplied; clusters wait for one another, so no more than
    // the device holds at a time (a cooperative launch)
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeCooperative;
    attr[1].val.cooperative = 1;
    cfg.blockDim = dim3(kChaseThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = attr;
    for (int K = kChaseCluster; K >= 1; K /= 2) {
        attr[0].val.clusterDim.x = K;
        cfg.gridDim = dim3(K);
        cfg.numAttrs = 1;
        int most = 0;
        if (cudaOccupancyMaxActiveClusters(&most, band_chase_kernel, &cfg) != cudaSuccess || most < 1) {
            cudaGetLastError();
            continue;
        }
        const int want = (std::min(t.n - 2, std::max(8, t.ntmax / 2 + 8)) + K - 1) / K;
        cfg.gridDim = dim3(K * std::max(1, std::min(want, most)));
        cfg.numAttrs = 2;
        DVR3D_COUNT_LAUNCH(1);
        return cudaLaunchKernelEx(&cfg, band_chase_kernel, t);
    }
    return cudaErrorNotSupported;
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
    // The kernel is bound by shared memory: a reflector costs a slab of 1, 2, 4, 8 columns some 16, 20,
    // 30, 52 passes over it (loads, stores, shuffles), slabs on one SM add up. The width with the
    // fewest passes on the fullest SM: 330 columns in slabs of 4, on 83 SMs (order 1600, a reflector at
    // a time: 1.9 ms; in slabs of 2, two on some SMs, 2.1), 100 columns one each.
    static const int pass[4] = {16, 20, 30, 52};
    int cols = 0, best = 0;
    for (int q = 0; q < 4; ++q) {
        const int c = 1 << q, slabs = (nev + c - 1) / c, cost = (slabs + nsm - 1) / nsm * pass[q];
        if (need(c) <= (size_t)optin && (cols == 0 || cost < best)) {
            cols = c;
            best = cost;
        }
    }
    if (cols == 0) return cudaErrorInvalidValue;
    switch (cols) {
        case 8: return launch_bt<8>(t, Z, ldz, nev, ldzs, need(8), st);
        case 4: return launch_bt<4>(t, Z, ldz, nev, ldzs, need(4), st);
        case 2: return launch_bt<2>(t, Z, ldz, nev, ldzs, need(2), st);
        default: return launch_bt<1>(t, Z, ldz, nev, ldzs, need(1), st);
    }
}

}  // namespace dvr3d
