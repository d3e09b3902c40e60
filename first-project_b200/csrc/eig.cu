// FP64 blocked two-sided Jacobi eigensolver for the symmetric I_n x I_n
// unfolding Grams of HOSVD/HOOI (replaces cusolverDnSsyevdx at
// src/tucker_hosvd.cu:43-61).
//
// The matrix is cut into blocks of BS rows/columns.  One sweep visits every
// pair of blocks once in round-robin order; in each round the nb/2 disjoint
// pairs are processed in parallel:
//   1. each pair (I, J) diagonalises its 2BS x 2BS principal submatrix in
//      shared memory (inner cyclic Jacobi), giving an orthogonal Q_IJ;
//   2. every 2BS x 2BS block between two pairs:  A_kl <- Q_k^T A_kl Q_l, and
//      V[:, l] <- V[:, l] Q_l.
// One cooperative launch runs all sweeps; the phases are separated by a grid
// barrier whose spin is bounded (an expired wait sets an error flag and every
// CTA returns).  Convergence: off(A) <= tol^2 * ||A||_F^2, tested at the start
// of each sweep from per-CTA partial sums reduced in a fixed order.
#include <vector>
#include <algorithm>

#include "jacobi.cuh"
#include "kernels.cuh"

namespace cud {

namespace {

constexpr int BS = 16;          // block size
constexpr int M2 = 2 * BS;      // pair submatrix size
constexpr int NT = 256;
constexpr long kSpinLimit = 1L << 24;
// Relative off-norm at which a pair block counts as diagonal, and the least
// one that the whole matrix is held to.  The inner one is the smaller: blocks
// that all just met the same bound would sum to it, and with anything left
// between them the outer test could not pass any more.
constexpr double kInnerTol = 2e-15 * M2, kOuterTol = 4e-15 * M2;

struct EigArgs {
    double *A;          // n x n, destroyed
    double *V;          // n x n, eigenvectors (unsorted)
    double *Q;          // npairs x M2 x M2
    double *part;       // gridDim partial sums (2 per CTA)
    unsigned *bar;      // [count, generation]
    int *status;        // [error, sweeps]
    int n, nb, max_sweeps;
    double tol;
};

__device__ bool grid_barrier(const EigArgs &a) {
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        volatile unsigned *gen = a.bar + 1;
        unsigned g = *gen;
        __threadfence();
        unsigned arrived = atomicAdd(a.bar, 1u);
        if (arrived == gridDim.x - 1) {
            atomicExch(a.bar, 0u);
            __threadfence();
            atomicAdd(a.bar + 1, 1u);
        } else {
            long it = 0;
            while (*gen == g) {
                if (++it > kSpinLimit) { atomicExch(a.status, 1); break; }
                __nanosleep(20);
            }
        }
        __threadfence();
        s_ok = (*(volatile int *)a.status == 0);
    }
    __syncthreads();
    return s_ok;
}

__device__ __forceinline__ void pair_blocks(int k, int round, int nb, int &I, int &J) {
    int a = (k == 0) ? 0 : 1 + (k - 1 + round) % (nb - 1);
    int b = 1 + (nb - 2 - k + round) % (nb - 1);
    I = min(a, b);
    J = max(a, b);
}

__device__ __forceinline__ int pair_index(int I, int J, int jj) {
    return (jj < BS) ? I * BS + jj : J * BS + (jj - BS);
}

constexpr int LD = M2 + 1;  // column stride of the shared-memory blocks (33: column walks hit distinct banks)

// off^2 and total^2 of the M2 x M2 block S, the same on every thread, in a
// fixed order.
__device__ __forceinline__ void block_off(const double *S, double *red, double &off, double &tot) {
    off = 0.0;
    tot = 0.0;
#pragma unroll
    for (int i = 0; i < M2 * M2 / NT; i++) {
        const int e = threadIdx.x + NT * i, r = e % M2, c = e / M2;
        const double v = S[r + LD * c] * S[r + LD * c];
        tot += v;
        if (r != c) off += v;
    }
    for (int o = 16; o > 0; o >>= 1) {
        off += __shfl_xor_sync(0xffffffffu, off, o);
        tot += __shfl_xor_sync(0xffffffffu, tot, o);
    }
    __syncthreads();  // red's readers of the call before
    if ((threadIdx.x & 31) == 0) {
        red[threadIdx.x >> 5] = off;
        red[NT / 32 + (threadIdx.x >> 5)] = tot;
    }
    __syncthreads();
    off = tot = 0.0;
    for (int w = 0; w < NT / 32; w++) {
        off += red[w];
        tot += red[NT / 32 + w];
    }
}

// Cyclic Jacobi on S0 (M2 x M2, shared, column stride LD), accumulating Q.
// Bound: a serial chain, (M2 - 1) rounds a sweep, each a rotation's
// parameters, the update and the hand-over to the next round.  Thread (k, l)
// owns the 2 x 2 cells of row pair k and column pair l for the round and
// applies both rotations to them in registers, and every warp forms all 16
// rotations itself (lane k the one of pair k, the column pairs' by shuffle),
// so a round has one barrier: S alternates between two buffers, since other
// warps still read the pivots.  B200, the three FP64 Grams of a 96 x 80 x 72
// HOSVD: 35.7 ms with three barriers a round and the angles in FP64, 8.0 ms
// now (about 840 clocks a round; phase 2 and the grid barriers are a sixth).
__device__ void inner_jacobi(double *S0, double *S1, double *Q, double *red, double tol) {
    constexpr int H = M2 / 2;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int k = lane & (H - 1), l = warp * 2 + (lane >> 4);
    static_assert(H == 16 && NT == H * H, "one thread per pair of pairs");
    for (int e = threadIdx.x; e < M2 * M2; e += NT) Q[(e % M2) + LD * (e / M2)] = (e % M2 == e / M2) ? 1.0 : 0.0;
    double *S = S0, *T = S1;
    // Round robin: pair 0 keeps index 0, every other index steps through
    // 1 .. M2 - 1 by one a round; M2 - 1 rounds bring it back.
    int ka = k, kb = M2 - 1 - k, la = l, lb = M2 - 1 - l;
    auto step = [](int &x) { x = (x == M2 - 1) ? 1 : x + 1; };
    for (int sweep = 0; sweep < 12; sweep++) {
        double off, tot;
        block_off(S, red, off, tot);
        if (!(off > tol * tol * tot) || !(tot > 0.0)) break;
        for (int round = 0; round < M2 - 1; round++) {
            const int p = min(ka, kb), q = max(ka, kb), pl = min(la, lb), ql = max(la, lb);
            double c, s;
            const double app = S[p + LD * p], aqq = S[q + LD * q], apq = S[p + LD * q];
            const double pp = S[p + LD * pl], qp = S[q + LD * pl], pq = S[p + LD * ql], qq = S[q + LD * ql];
            const double v0 = Q[k + LD * pl], w0 = Q[k + LD * ql], v1 = Q[k + H + LD * pl], w1 = Q[k + H + LD * ql];
            jacobi_rotation(app, aqq, apq, c, s);
            const double cl = __shfl_sync(0xffffffffu, c, l), sl = __shfl_sync(0xffffffffu, s, l);
            const double rp = c * pp - s * qp, sp = s * pp + c * qp;  // rows p, q at column pl
            const double rq = c * pq - s * qq, sq = s * pq + c * qq;  // and at column ql
            T[p + LD * pl] = cl * rp - sl * rq;
            T[q + LD * pl] = cl * sp - sl * sq;
            T[p + LD * ql] = sl * rp + cl * rq;
            T[q + LD * ql] = sl * sp + cl * sq;
            Q[k + LD * pl] = cl * v0 - sl * w0;
            Q[k + LD * ql] = sl * v0 + cl * w0;
            Q[k + H + LD * pl] = cl * v1 - sl * w1;
            Q[k + H + LD * ql] = sl * v1 + cl * w1;
            if (k) step(ka);
            step(kb);
            if (l) step(la);
            step(lb);
            __syncthreads();
            double *x = S;
            S = T;
            T = x;
        }
    }
    __syncthreads();
}

// Y (M2 x M2) = A B (or A^T B), all in shared memory with column stride LD:
// thread t forms rows (t % 32) of the columns 4 (t / 32) .. + 3.
template <bool kTransA>
__device__ __forceinline__ void block_mul(const double *A, const double *B, double (&y)[4]) {
    const int r = threadIdx.x & 31, c0 = (threadIdx.x >> 5) * 4;
#pragma unroll
    for (int j = 0; j < 4; j++) y[j] = 0.0;
#pragma unroll 8
    for (int i = 0; i < M2; i++) {
        const double a = kTransA ? A[i + LD * r] : A[r + LD * i];
#pragma unroll
        for (int j = 0; j < 4; j++) y[j] = fma(a, B[i + LD * (c0 + j)], y[j]);
    }
}

__global__ void __launch_bounds__(NT) k_block_jacobi(EigArgs a) {
    extern __shared__ __align__(16) double smem_d[];
    double *S = smem_d, *S2 = S + LD * M2, *Qk = S2 + LD * M2, *Ql = Qk + LD * M2;
    __shared__ double red[2 * (NT / 32)];
    const int n = a.n, nb = a.nb, npairs = nb / 2;
    const long nn = (long)n * n;
    const int rblocks = (n + M2 - 1) / M2;  // 32-row blocks of V

    // V = I
    for (long e = blockIdx.x * (long)NT + threadIdx.x; e < nn; e += (long)gridDim.x * NT)
        a.V[e] = (e % n == e / n) ? 1.0 : 0.0;
    if (!grid_barrier(a)) return;

    int sweep = 0;
    for (;; sweep++) {
        // convergence test: per-CTA partials, reduced in fixed order by all
        double off = 0.0, tot = 0.0;
        for (long e = blockIdx.x * (long)NT + threadIdx.x; e < nn; e += (long)gridDim.x * NT) {
            double v = a.A[e] * a.A[e];
            tot += v;
            if (e % n != e / n) off += v;
        }
        for (int o = 16; o > 0; o >>= 1) {
            off += __shfl_xor_sync(0xffffffffu, off, o);
            tot += __shfl_xor_sync(0xffffffffu, tot, o);
        }
        if ((threadIdx.x & 31) == 0) {
            red[threadIdx.x >> 5] = off;
            red[NT / 32 + (threadIdx.x >> 5)] = tot;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            double o2 = 0.0, t2 = 0.0;
            for (int w = 0; w < NT / 32; w++) { o2 += red[w]; t2 += red[NT / 32 + w]; }
            a.part[2 * blockIdx.x] = o2;
            a.part[2 * blockIdx.x + 1] = t2;
        }
        if (!grid_barrier(a)) return;
        // every warp sums all partials the same way: lane-strided, then a
        // fixed shuffle tree
        double offs = 0.0, tots = 0.0;
        for (int b = threadIdx.x & 31; b < (int)gridDim.x; b += 32) {
            offs += ((volatile double *)a.part)[2 * b];
            tots += ((volatile double *)a.part)[2 * b + 1];
        }
        for (int o = 16; o > 0; o >>= 1) {
            offs += __shfl_xor_sync(0xffffffffu, offs, o);
            tots += __shfl_xor_sync(0xffffffffu, tots, o);
        }
        if (!(offs > a.tol * a.tol * tots) || tots == 0.0) break;
        if (sweep >= a.max_sweeps) {
            if (blockIdx.x == 0 && threadIdx.x == 0) a.status[0] = 2;
            break;
        }

        for (int round = 0; round < nb - 1; round++) {
            // phase 1: diagonalise each pair's 2BS x 2BS block.  (The first
            // round's barrier also separates the reads of `part` above from
            // the next sweep's writes.)
            for (int k = blockIdx.x; k < npairs; k += gridDim.x) {
                int I, J;
                pair_blocks(k, round, nb, I, J);
                for (int e = threadIdx.x; e < M2 * M2; e += NT) {
                    int ii = e % M2, jj = e / M2;
                    int gi = pair_index(I, J, ii), gj = pair_index(I, J, jj);
                    S[ii + LD * jj] = (gi < n && gj < n) ? a.A[gi + (long)n * gj] : 0.0;
                }
                __syncthreads();
                inner_jacobi(S, S2, Qk, red, kInnerTol);
                double *Qg = a.Q + (long)k * M2 * M2;
                for (int e = threadIdx.x; e < M2 * M2; e += NT) Qg[e] = Qk[(e % M2) + LD * (e / M2)];
                __syncthreads();
            }
            if (!grid_barrier(a)) return;
            // phase 2: A_kl <- Q_k^T A_kl Q_l for every pair of pairs, and
            // V_il <- V_il Q_l for every 32-row block of V; each task owns
            // its block, so rows and columns need no barrier between them
            const int ntask = (npairs + rblocks) * npairs;
            for (int task = blockIdx.x; task < ntask; task += gridDim.x) {
                const int l = task % npairs, k = task / npairs;
                const bool isA = k < npairs;
                int I, J, IK = 0, JK = 0;
                pair_blocks(l, round, nb, I, J);
                if (isA) pair_blocks(k, round, nb, IK, JK);
                double *Mx = isA ? a.A : a.V;
                __syncthreads();
                for (int e = threadIdx.x; e < M2 * M2; e += NT) {
                    const int r = e % M2, c = e / M2;
                    const int gr = isA ? pair_index(IK, JK, r) : (k - npairs) * M2 + r, gc = pair_index(I, J, c);
                    S[r + LD * c] = (gr < n && gc < n) ? Mx[gr + (long)n * gc] : 0.0;
                    Ql[r + LD * c] = __ldcg(a.Q + (long)l * M2 * M2 + e);
                    if (isA) Qk[r + LD * c] = __ldcg(a.Q + (long)k * M2 * M2 + e);
                }
                __syncthreads();
                const int r = threadIdx.x & 31, c0 = (threadIdx.x >> 5) * 4;
                double y[4];
                block_mul<false>(S, Ql, y);
                if (isA) {
#pragma unroll
                    for (int j = 0; j < 4; j++) S2[r + LD * (c0 + j)] = y[j];
                    __syncthreads();
                    block_mul<true>(Qk, S2, y);
                }
                const int gr = isA ? pair_index(IK, JK, r) : (k - npairs) * M2 + r;
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const int gc = pair_index(I, J, c0 + j);
                    if (gr < n && gc < n) Mx[gr + (long)n * gc] = y[j];
                }
            }
            if (!grid_barrier(a)) return;
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) a.status[1] = sweep;
}

// A key that orders doubles totally: -0 equals +0, every NaN is the largest.
__device__ __forceinline__ unsigned long long sort_key(double v) {
    if (v != v) return ~0ull;
    const unsigned long long b = (unsigned long long)__double_as_longlong(v + 0.0);
    return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}

// W ascending, and perm[position] = column of V: a thread per eigenvalue
// counts those before it (equal ones in index order, as a stable sort).  One
// thread's insertion sort, a dependent global load a step, took 150 us at
// n = 96 and its square beyond.
__global__ void __launch_bounds__(128) k_sort_eig(const double *__restrict__ A, int n, double *__restrict__ W,
                                                  int *__restrict__ perm) {
    __shared__ unsigned long long key[128];
    const int i = blockIdx.x * 128 + threadIdx.x;
    const double v = (i < n) ? A[i + (long)n * i] : 0.0;
    const unsigned long long mine = sort_key(v);
    int rank = 0;
    for (int j0 = 0; j0 < n; j0 += 128) {
        const int j = j0 + threadIdx.x;
        __syncthreads();
        if (j < n) key[threadIdx.x] = sort_key(A[j + (long)n * j]);
        __syncthreads();
        const int m = min(128, n - j0);
        for (int t = 0; t < m; t++) rank += (key[t] < mine) || (key[t] == mine && j0 + t < i);
    }
    if (i < n) {
        W[rank] = v;
        perm[rank] = i;
    }
}

__global__ void k_permute_cols(const double *__restrict__ Vin, const int *__restrict__ perm, int n,
                               double *__restrict__ Vout) {
    long nn = (long)n * n;
    for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < nn; e += (long)gridDim.x * blockDim.x) {
        long r = e % n, c = e / n;
        Vout[e] = Vin[r + (long)n * perm[c]];
    }
}

constexpr size_t kEigSmem = sizeof(double) * 4 * LD * M2;  // 33 KB

}  // namespace

int syev_jacobi(double *A, long n, double *W, double *V, int max_sweeps, cudaStream_t s) {
    if (n <= 0) return CUD_OK;
    if (n > 32768) return CUD_ERR_UNSUPPORTED;
    int nb = (int)((n + BS - 1) / BS);
    if (nb < 2) nb = 2;
    if (nb & 1) nb++;
    int npairs = nb / 2;
    int dev = 0, occ = 0;
    CUD_CHECK(cudaGetDevice(&dev));
    CUD_CHECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_block_jacobi, NT, kEigSmem));
    int sms = 0;
    CUD_CHECK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    // a CTA per phase-2 task, at most one wave: a grid barrier over few CTAs
    // is the cheaper one where the matrix is small
    const long tasks = (long)(npairs + (n + M2 - 1) / M2) * npairs;
    int grid = (int)std::max(1L, std::min((long)occ * sms, std::max((long)npairs, tasks)));
    size_t bytes_Q = sizeof(double) * (size_t)npairs * M2 * M2;
    size_t bytes_V = sizeof(double) * (size_t)n * n;
    size_t off_part = bytes_Q;
    size_t off_bar = off_part + sizeof(double) * 2 * grid;
    size_t off_st = off_bar + 64;
    size_t off_Vt = (off_st + 64 + 255) & ~size_t(255);
    size_t off_perm = off_Vt + bytes_V;
    int st;
    char *w = (char *)scratch(kSlotEig, off_perm + sizeof(int) * n + 64, &st);
    if (!w) return st;
    EigArgs a;
    a.A = A;
    a.V = (double *)(w + off_Vt);
    a.Q = (double *)w;
    a.part = (double *)(w + off_part);
    a.bar = (unsigned *)(w + off_bar);
    a.status = (int *)(w + off_st);
    a.n = (int)n;
    a.nb = nb;
    a.max_sweeps = max_sweeps > 0 ? max_sweeps : 40;
    // off(A) can only be driven to the rounding floor of the rotations,
    // about n * eps relative to ||A||_F, and no lower than the pair blocks'
    // own stop (kOuterTol): with a tighter outer test a
    // clustered spectrum (a near low-rank Gram) never met it
    a.tol = std::max(4.0 * 2.22e-16 * (double)std::max(16L, n), kOuterTol);
    CUD_CHECK(cudaMemsetAsync(w + off_bar, 0, 128, s));
    void *args[] = {&a};
    CUD_CHECK(cudaLaunchCooperativeKernel((void *)k_block_jacobi, grid, NT, args, kEigSmem, s));
    CUD_CHECK_LAUNCH("syev_jacobi");
    int *perm = (int *)(w + off_perm);
    k_sort_eig<<<(unsigned)((n + 127) / 128), 128, 0, s>>>(A, (int)n, W, perm);
    k_permute_cols<<<blocks_for(n * n, 256), 256, 0, s>>>(a.V, perm, (int)n, V);
    CUD_CHECK_LAUNCH("syev_jacobi sort");
    int hst[2] = {0, 0};
    CUD_CHECK(cudaMemcpyAsync(hst, a.status, sizeof(hst), cudaMemcpyDeviceToHost, s));
    CUD_CHECK(cudaStreamSynchronize(s));
    if (hst[0] == 1) return CUD_ERR_DEVICE_TIMEOUT;
    if (hst[0] == 2) return CUD_ERR_NOT_CONVERGED;
    return CUD_OK;
}

}  // namespace cud

extern "C" int cud_syev_jacobi(double *A, long n, double *W, double *V, int max_sweeps, void *stream) {
    if (n < 0 || (n > 0 && (!A || !W || !V))) return cud::set_status(CUD_ERR_INVALID_ARGUMENT);
    return cud::set_status(cud::syev_jacobi(A, n, W, V, max_sweeps, cud::as_stream(stream)));
}
