// Leading eigenvectors of a symmetric positive semi-definite FP64 matrix by
// subspace iteration, for the Tucker factors (the r_n leading eigenvectors
// of an I_n x I_n unfolding Gram; the reference asks cuSOLVER's syevdx for
// them, src/tucker_hosvd.cu:38-56).
//
//   V <- orth(G V)   (CholQR, applied twice for orthogonality),
//
// from a seeded Gaussian start, until the subspace stops moving
// (r - ||V_old^T V_new||_F^2 = sum of squared sines of the principal angles
// below a tolerance), then Rayleigh-Ritz: the r x r matrix V^T G V is
// diagonalised by Jacobi in shared memory and its eigenvectors rotate V.
// The iteration converges at the rate lambda_{r+1} / lambda_r, i.e. in a few
// steps when the Gram has a gap after its r-th eigenvalue (a low-rank-plus-
// noise tensor); callers fall back to the full Jacobi eigensolver when it
// does not converge.
#include <cooperative_groups.h>

#include <atomic>
#include <mutex>

#include "jacobi.cuh"
#include "kernels.cuh"

namespace cud {

namespace cg = cooperative_groups;

namespace {

constexpr int SI_RMAX = 64;

// C (8 x 8) += A (8 x 4) B (4 x 8) in FP64.
__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(c[0]), "+d"(c[1])
                 : "d"(a), "d"(b));
}

__device__ __forceinline__ unsigned long long si_mix(unsigned long long z) {
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ULL;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebULL;
    return z ^ (z >> 31);
}

// Entry e of the start block: i.i.d. standard normal (Box-Muller over a
// counter hash).
__device__ __forceinline__ double si_start(long e) {
    const double u1 = 1.0 - (double)(si_mix(2 * e + 0x51) >> 11) * (1.0 / 9007199254740992.0);
    const double u2 = (double)(si_mix(2 * e + 0x52) >> 11) * (1.0 / 9007199254740992.0);
    return sqrt(-2.0 * log(u1)) * cospi(2.0 * u2);
}

// V (n x r) = the start block.
__global__ void k_si_init(double *V, long n, int r) {
    const long total = n * r;
    for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < total; e += (long)gridDim.x * blockDim.x)
        V[e] = si_start(e);
}

// V (n x r) = the given FP32 start block.
__global__ void k_si_init_from(const float *__restrict__ U0, double *V, long n, int r) {
    const long total = n * r;
    for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < total; e += (long)gridDim.x * blockDim.x)
        V[e] = (double)U0[e];
}

// Y (n x r) = G (n x n) V (n x r), column-major.
__global__ void __launch_bounds__(256) k_si_apply(const double *__restrict__ G, const double *__restrict__ V,
                                                  long n, int r, double *__restrict__ Y) {
    const long total = n * r;
    for (long e = blockIdx.x * 256L + threadIdx.x; e < total; e += (long)gridDim.x * 256L) {
        const long i = e % n, c = e / n;
        double s = 0.0;
        for (long k = 0; k < n; k++) s = fma(G[i + n * k], V[k + n * c], s);
        Y[e] = s;
    }
}

// In place Y <- Y L^-T with L L^T = Y^T Y (Cholesky QR), one CTA.  Sets
// *fail when Y^T Y is not numerically positive definite.
__global__ void __launch_bounds__(256) k_si_cholqr(double *Y, long n, int r, int *fail) {
    __shared__ double C[SI_RMAX * SI_RMAX];
    __shared__ int bad;
    for (int e = threadIdx.x; e < r * r; e += blockDim.x) {
        const int a = e % r, b = e / r;
        double s = 0.0;
        if (a >= b)
            for (long i = 0; i < n; i++) s = fma(Y[i + n * a], Y[i + n * b], s);
        C[e] = s;
    }
    if (threadIdx.x == 0) bad = 0;
    __syncthreads();
    // Cholesky (lower, column by column), small: one column per step
    for (int j = 0; j < r; j++) {
        if (threadIdx.x == 0) {
            double d = C[j + r * j];
            for (int k = 0; k < j; k++) d -= C[j + r * k] * C[j + r * k];
            if (!(d > 0.0) || !isfinite(d)) { bad = 1; d = 1.0; }
            C[j + r * j] = sqrt(d);
        }
        __syncthreads();
        for (int i = j + 1 + threadIdx.x; i < r; i += blockDim.x) {
            double s = C[i + r * j];
            for (int k = 0; k < j; k++) s -= C[i + r * k] * C[j + r * k];
            C[i + r * j] = s / C[j + r * j];
        }
        __syncthreads();
    }
    if (bad) {
        if (threadIdx.x == 0) *fail = 1;
        return;
    }
    // rows of Y: y_i <- L^-1 y_i (forward substitution), i.e. Y <- Y L^-T
    for (long i = threadIdx.x; i < n; i += blockDim.x) {
        double z[SI_RMAX];
        for (int a = 0; a < r; a++) {
            double s = Y[i + n * a];
            for (int k = 0; k < a; k++) s -= C[a + r * k] * z[k];
            z[a] = s / C[a + r * a];
        }
        for (int a = 0; a < r; a++) Y[i + n * a] = z[a];
    }
}

// out = r - ||A^T B||_F^2 (A, B n x r orthonormal), one CTA.
__global__ void __launch_bounds__(256) k_si_gap(const double *A, const double *B, long n, int r, double *out) {
    __shared__ double red[256];
    double acc = 0.0;
    for (int e = threadIdx.x; e < r * r; e += blockDim.x) {
        const int a = e % r, b = e / r;
        double s = 0.0;
        for (long i = 0; i < n; i++) s = fma(A[i + n * a], B[i + n * b], s);
        acc += s * s;
    }
    red[threadIdx.x] = acc;
    __syncthreads();
    for (int w = 128; w > 0; w >>= 1) {
        if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) out[0] = (double)r - red[0];
}

// Rayleigh-Ritz: H = V^T Y (Y = G V), Jacobi on H in shared memory, then
// U[:, j] = V w_j for the eigenvalues in ascending order (FP32 out).  One CTA.
__global__ void __launch_bounds__(256) k_si_ritz(const double *V, const double *Y, long n, int r, float *U,
                                                 double *W) {
    __shared__ double H[SI_RMAX * SI_RMAX];  // W (r x r rotations) lives in global scratch
    __shared__ double cs[SI_RMAX / 2], sn[SI_RMAX / 2];
    __shared__ int pp[SI_RMAX / 2], qq[SI_RMAX / 2], ord[SI_RMAX];
    __shared__ double off_s;
    for (int e = threadIdx.x; e < r * r; e += blockDim.x) {
        const int a = e % r, b = e / r;
        double s = 0.0;
        for (long i = 0; i < n; i++) s = fma(V[i + n * a], Y[i + n * b], s);
        H[e] = s;
        W[e] = (a == b) ? 1.0 : 0.0;
    }
    __syncthreads();
    for (int e = threadIdx.x; e < r * r; e += blockDim.x) {  // symmetrise
        const int a = e % r, b = e / r;
        if (a < b) {
            const double m = 0.5 * (H[a + r * b] + H[b + r * a]);
            H[a + r * b] = m;
            H[b + r * a] = m;
        }
    }
    __syncthreads();
    const int m = (r + 1) & ~1;
    // stop at a relative off-diagonal norm of 1e-13: rounding alone keeps it
    // near r * eps, so a test at eps itself would run every sweep
    for (int sweep = 0; sweep < 40; sweep++) {
        if (threadIdx.x == 0) {
            double off = 0.0, tot = 0.0;
            for (int e = 0; e < r * r; e++) {
                tot += H[e] * H[e];
                if (e % r != e / r) off += H[e] * H[e];
            }
            off_s = (off <= 1e-26 * tot) ? -1.0 : off;
        }
        __syncthreads();
        if (off_s < 0) break;
        for (int round = 0; round < m - 1; round++) {
            if (threadIdx.x < m / 2) {
                const int k = threadIdx.x;
                int a = (k == 0) ? m - 1 : (round + k) % (m - 1);
                int b = (k == 0) ? round % (m - 1) : (round + m - 1 - k) % (m - 1);
                const int p = min(a, b), q = max(a, b);
                double c = 1.0, s = 0.0;
                if (q < r && H[p + r * q] != 0.0) {
                    const double theta = (H[q + r * q] - H[p + r * p]) / (2.0 * H[p + r * q]);
                    const double t = (theta >= 0 ? 1.0 : -1.0) / (fabs(theta) + sqrt(theta * theta + 1.0));
                    c = 1.0 / sqrt(t * t + 1.0);
                    s = t * c;
                }
                cs[k] = c; sn[k] = s; pp[k] = p; qq[k] = q;
            }
            __syncthreads();
            for (int e = threadIdx.x; e < (m / 2) * r; e += blockDim.x) {
                const int k = e / r, col = e % r, p = pp[k], q = qq[k];
                if (q >= r) continue;
                const double hp = H[p + r * col], hq = H[q + r * col];
                H[p + r * col] = cs[k] * hp - sn[k] * hq;
                H[q + r * col] = sn[k] * hp + cs[k] * hq;
            }
            __syncthreads();
            for (int e = threadIdx.x; e < (m / 2) * r; e += blockDim.x) {
                const int k = e / r, row = e % r, p = pp[k], q = qq[k];
                if (q >= r) continue;
                const double hp = H[row + r * p], hq = H[row + r * q];
                H[row + r * p] = cs[k] * hp - sn[k] * hq;
                H[row + r * q] = sn[k] * hp + cs[k] * hq;
                const double wp = W[row + r * p], wq = W[row + r * q];
                W[row + r * p] = cs[k] * wp - sn[k] * wq;
                W[row + r * q] = sn[k] * wp + cs[k] * wq;
            }
            __syncthreads();
        }
    }
    if (threadIdx.x == 0) {  // ascending eigenvalues
        for (int j = 0; j < r; j++) ord[j] = j;
        for (int a = 1; a < r; a++)
            for (int b = a; b > 0 && H[ord[b] + r * ord[b]] < H[ord[b - 1] + r * ord[b - 1]]; b--) {
                const int t = ord[b]; ord[b] = ord[b - 1]; ord[b - 1] = t;
            }
    }
    __syncthreads();
    for (long e = threadIdx.x; e < n * r; e += blockDim.x) {
        const long i = e % n;
        const int j = (int)(e / n), c = ord[j];
        double s = 0.0;
        for (int a = 0; a < r; a++) s = fma(V[i + n * a], W[a + r * c], s);
        U[e] = (float)s;
    }
}

// ---------------------------------------------------------------- fast path
// r <= 32 and n <= 2048, where the iteration does not fit in one launch
// (k_si_run_cl).  One step is two launches of the product G V
// (k_si_apply_cols; the k range split in slices whose partial products are
// kept apart) and one launch of a cluster of CL_N CTAs that owns the n x r
// iterate by row blocks (k_si_orth_cl): the partial products summed in
// slice order, two CholQR passes, and the subspace gap against the previous
// iterate.  Each r x r Gram or cross product is the sum of the CTAs' row-
// block contributions, read through distributed shared memory and added in
// rank order; every CTA forms the same sum, so the small factorisations run
// redundantly in each CTA with identical results and need no broadcast.
// The Rayleigh-Ritz step (k_si_ritz_cl) has the same shape.  The r x r
// work -- the factorisation with its triangular inverse, the Jacobi sweeps
// -- keeps the matrix cells in registers across all threads and takes a
// fixed number of block barriers per step; the n x r work -- partial sums,
// row-block Grams, Y L^-T, V W -- is spread over the rows.
constexpr int SI_FR = 32;
constexpr int CL_N = 8;    // CTAs per cluster
constexpr int CL_T = 256;  // threads per CTA
constexpr int CL_RS = 33;  // row stride (doubles) of the row-major blocks in shared memory
constexpr size_t CL_SMEM_MAX = 200 * 1024;

// Dynamic shared memory of the cluster kernels (offsets in doubles): two
// row blocks (nl x 32, zero beyond column r), the two r x r buffers the
// peers read, the tile partials, two 32 x 32 matrices.
struct ClLayout {
    int nl;  // rows per CTA
    size_t ya, yb, red, gp, C, T, total;
};
__host__ __device__ inline ClLayout cl_layout(long n) {
    ClLayout L;
    L.nl = (int)((n + CL_N - 1) / CL_N);
    const size_t blk = (size_t)L.nl * CL_RS;
    L.ya = 0;
    L.yb = L.ya + blk;
    L.red = L.yb + blk;
    L.gp = L.red + 2 * 32 * 32;
    L.C = L.gp + (size_t)CL_T * 16;
    L.T = L.C + 32 * CL_RS;
    L.total = L.T + 32 * CL_RS;
    return L;
}

// dst (nl x 32 row-major) = rows i0 .. i0 + nl - 1 of the sum of the nks
// column-major n x r slices of src, summed in slice order; columns r..31 zero.
__device__ void cl_load_rows(const double *__restrict__ src, int nks, long n, int r, long i0, int nl, double *dst) {
    const long nr = n * r;
#pragma unroll 4
    for (int e = threadIdx.x; e < nl * 32; e += CL_T) {
        const int a = e / nl, i = e - a * nl;
        double t = 0.0;
        if (a < r) {
            const double *p = src + (i0 + i) + n * a;
            for (int y = 0; y < nks; y++) t += p[(long)y * nr];
        }
        dst[i * CL_RS + a] = t;
    }
}

// Tile (ta, tb) of nt x nt (nt <= 4), or of its lower triangle in row order
// when sym; without divisions, which a chain this short would feel.
__device__ __forceinline__ void cl_tile(int tile, int nt, bool sym, int &ta, int &tb) {
    if (sym) {
        ta = (tile >= 1) + (tile >= 3) + (tile >= 6);
        tb = tile - (ta * (ta + 1) >> 1);
    } else {
        ta = nt == 3 ? tile * 11 >> 5 : tile >> (nt >> 1);
        tb = tile - ta * nt;
    }
}

// out (32 x 32 row-major) = this CTA's rows' part of A^T B (lower triangle
// when sym, with the diagonal tiles whole): 8 x 8 tiles by FP64 matrix
// instructions, the rows in 8, 2 or 1 groups for r <= 8, 16 or 32, whose
// partials are added in group order.  gp: 1024 doubles.  Ends on a block
// barrier.  (4 x 4 tiles a thread by FMAs took 2400 clocks for 32 rows and
// r = 16, most of them bank conflicts between the partials; this takes 730.)
__device__ void cl_cross(const double *A, const double *B, int nl, int r, bool sym, double *gp, double *out) {
    constexpr int NW = CL_T / 32;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int nt = (r + 7) >> 3;
    const int ntiles = sym ? nt * (nt + 1) >> 1 : nt * nt;
    const int lg = nt == 1 ? 3 : nt == 2 ? 1 : 0, nk = (nl + 3) >> 2;
    for (int it = w; it < ntiles << lg; it += NW) {
        int g = 0, tile = it, ta, tb;
        if (nt == 1) {
            g = it;
            tile = 0;
        } else if (it >= ntiles) {
            g = 1;
            tile = it - ntiles;
        }
        cl_tile(tile, nt, sym, ta, tb);
        double acc[2] = {0.0, 0.0};
        const int k0 = g * nk >> lg, k1 = (g + 1) * nk >> lg;
        int i = 4 * k0 + (lane & 3);
        const double *pa = A + i * CL_RS + 8 * ta + (lane >> 2), *pb = B + i * CL_RS + 8 * tb + (lane >> 2);
#pragma unroll 4
        for (int k = k0; k < k1; k++) {
            const bool in = i < nl;
            dmma(acc, in ? *pa : 0.0, in ? *pb : 0.0);
            i += 4;
            pa += 4 * CL_RS;
            pb += 4 * CL_RS;
        }
        double *o = gp + it * 64 + (lane >> 2) * 8 + 2 * (lane & 3);
        o[0] = acc[0];
        o[1] = acc[1];
    }
    __syncthreads();
    for (int e = threadIdx.x; e < ntiles * 64; e += CL_T) {
        const int tile = e >> 6, u = (e >> 3) & 7, v = e & 7;
        int ta, tb;
        cl_tile(tile, nt, sym, ta, tb);
        double t = 0.0;
        for (int g = 0; g < 1 << lg; g++) t += gp[(g * ntiles + tile) * 64 + 8 * u + v];
        out[(8 * ta + u) * 32 + 8 * tb + v] = t;
    }
    __syncthreads();
}

// dst (32 x CL_RS) = sum over the cluster's CTAs, in rank order, of their
// buffer `red` (entries a, b < r, a >= b when sym; zero elsewhere).  The
// caller has synchronised the cluster after the buffers were written.
__device__ void cl_sum(cg::cluster_group &cl, double *red, int r, bool sym, double *dst) {
    const int b = threadIdx.x & 31, w = threadIdx.x >> 5;
    const double *peer[CL_N];
#pragma unroll
    for (int q = 0; q < CL_N; q++) peer[q] = cl.map_shared_rank(red, q) + threadIdx.x;
#pragma unroll
    for (int u = 0; u < 32 * 32 / CL_T; u++) {
        const int a = w + (CL_T / 32) * u;
        double v[CL_N], t = 0.0;
        if (a < r && b < r && (!sym || a >= b)) {  // the loads go out together
#pragma unroll
            for (int q = 0; q < CL_N; q++) v[q] = peer[q][CL_T * u];
#pragma unroll
            for (int q = 0; q < CL_N; q++) t += v[q];
        }
        dst[a * CL_RS + b] = t;
    }
    __syncthreads();
}

// CholQR's r x r factor work: C (lower triangle valid, in shared memory) =
// L D L^T with unit L, and R = L^-1, by eliminating the rows of [C | I] in
// place: at step k column k of C is done and its place takes column k of R,
// so a row i > k loses the same multiple of row k in every column.  Then
// T = (L D^1/2)^-1 = D^-1/2 R (XL x XL, zero outside the lower r x r
// triangle).  XL lanes to a row, NQ rows a thread (rows i = i0 + 8q): a step
// reads row k, published in shared memory (double-buffered) with the pivot
// in it, takes a_ik from lane k and ends on one barrier of the warps that
// work.  A serial chain of the pivot's reciprocal, a product and an FMA, and
// the issue slots of its warps: for r <= 16 four warps of two 16-lane rows
// each.  16 steps took 16 000 clocks when C and R were two cases of a
// branch, 3900 now.  Returns on every thread whether every pivot was positive
// and finite.
template <int XL>
__device__ __forceinline__ bool cl_chol_steps(const double *C, double *T, int r, double *pub, double *dsh) {
    constexpr int NQ = XL / 8, NTH = 8 * XL;  // 8 rows at a time
    const int x = threadIdx.x % XL, i0 = threadIdx.x / XL, src = threadIdx.x & 31 & ~(XL - 1);
    double v[NQ];
#pragma unroll
    for (int q = 0; q < NQ; q++) {
        const int i = i0 + 8 * q;
        v[q] = (i < r && x < r) ? C[max(i, x) * CL_RS + min(i, x)] : 0.0;
    }
    if (i0 == 0) pub[x] = v[0];
    asm volatile("bar.sync 1, %0;" ::"n"(NTH) : "memory");
    bool ok = true;
    for (int k = 0; k < r; k++) {
        const double *row = pub + 32 * (k & 1);
        double *nrow = pub + 32 * ((k + 1) & 1);
        const double akk = row[k];
        double rx = row[x];
        // 1 / a_kk = y (1 + f): the 20-bit estimate and a third-order Newton
        // step, which the products with y do not wait for; the division where
        // the estimate would flush or underflow
        double y = rcp_approx(akk), f;
        if ((unsigned)__double2hiint(akk) - 0x00100000u < 0x7e000000u) {
            const double e = fma(-akk, y, 1.0);
            f = fma(e, e, e);
        } else {
            const bool good = akk > 0.0 && isfinite(akk);
            ok = ok && good;
            y = good ? 1.0 / akk : 0.0;
            f = 0.0;
        }
        if (threadIdx.x == 0) dsh[k] = akk;
        rx = (x == k ? 1.0 : rx) * y;
#pragma unroll
        for (int q = 0; q < NQ; q++) {
            const int i = i0 + 8 * q;
            const double aik = __shfl_sync(0xffffffffu, v[q], src + k);
            const double g = aik * rx;
            const double t = fma(-g, f, fma(-aik, rx, x == k ? 0.0 : v[q]));
            v[q] = i > k ? t : v[q];
            if (i == k + 1) nrow[x] = t;
        }
        asm volatile("bar.sync 1, %0;" ::"n"(NTH) : "memory");
    }
    if (threadIdx.x < 32) dsh[threadIdx.x] = threadIdx.x < r ? 1.0 / sqrt(dsh[threadIdx.x]) : 0.0;
    asm volatile("bar.sync 1, %0;" ::"n"(NTH) : "memory");
#pragma unroll
    for (int q = 0; q < NQ; q++) {
        const int i = i0 + 8 * q;
        T[i * CL_RS + x] = (i < r && x <= i) ? (x == i ? 1.0 : v[q]) * dsh[i] : 0.0;
    }
    return ok;
}

__device__ __forceinline__ bool cl_chol_inv(const double *C, double *T, int r, double *pub, double *dsh) {
    __shared__ int s_ok;
    if (r > 16) {
        const bool ok = cl_chol_steps<32>(C, T, r, pub, dsh);
        if (threadIdx.x == 0) s_ok = ok;
    } else if (threadIdx.x < 128) {
        const bool ok = cl_chol_steps<16>(C, T, r, pub, dsh);
        if (threadIdx.x == 0) s_ok = ok;
    }
    __syncthreads();
    return s_ok;
}

// dst[i][a] = sum_k M[a][k] src[i][k] over the nl rows (M r x r, row stride
// CL_RS, zero up to the next multiple of 8, as src's columns are), 8 x 8 tiles by FP64
// matrix instructions; dst's columns up to the next multiple of 8 are zero.
__device__ void cl_transform(const double *src, const double *M, int nl, int r, double *dst) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int nt = (r + 7) >> 3, nk = (r + 3) >> 2;
    for (int m = w; m < (nl + 7) >> 3; m += CL_T / 32) {
        const int i = 8 * m + (lane >> 2);
        const double *ps = src + i * CL_RS + (lane & 3), *pm = M + (lane >> 2) * CL_RS + (lane & 3);
        double acc[4][2] = {};
#pragma unroll
        for (int k = 0; k < 8; k++) {
            if (k >= nk) break;
            const double a = i < nl ? ps[4 * k] : 0.0;
#pragma unroll
            for (int j = 0; j < 4; j++)
                if (j < nt) dmma(acc[j], a, pm[8 * j * CL_RS + 4 * k]);
        }
        if (i < nl)
#pragma unroll
            for (int j = 0; j < 4; j++)
                if (j < nt) {
                    double *d = dst + i * CL_RS + 8 * j + 2 * (lane & 3);
                    d[0] = acc[j][0];
                    d[1] = acc[j][1];
                }
    }
}

// Cyclic Jacobi on all threads (round-robin pairs, h = m / 2 disjoint
// rotations a round) on the symmetric part of H0 (r x r, row stride CL_RS,
// zero beyond r), the rotations accumulated in W.  A round is a serial chain
// of angles, update and one barrier: every warp forms the rotations itself
// (lane k that of pair k) and a thread applies those of a pair of pairs to
// their 2 x 2 cell of H, from one buffer into the other, or a pair's to one
// row of W.  An odd r's dummy is a zero row, which no rotation touches.
// The entries are read before the angles are formed, and warps without an
// item form none (the angles' approximations share one unit).
// Stops at a relative off-diagonal norm of 1e-13 (rounding alone keeps it
// near r * eps, so a test at eps itself would run every sweep).  On return
// ord is the eigenvalue order, ascending.  Ends on a block barrier.
template <int NI>
__device__ __forceinline__ void cl_jacobi(double *H0, double *H1, double *W, int r, int *ord, double *wred) {
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int h = (r + 1) / 2, m = 2 * h;
    for (int e = tid; e < 32 * 32; e += CL_T) {
        const int i = e >> 5, j = e & 31;
        H1[i * CL_RS + j] = 0.5 * (H0[i * CL_RS + j] + H0[j * CL_RS + i]);
        W[i * CL_RS + j] = (i == j && i < r) ? 1.0 : 0.0;
    }
    // this thread's items: cells (k, l) of H first, then (pair k, row l) of W
    // (NI of them: h (h + m) <= NI CL_T)
    int ik[NI], il[NI];
    bool cell[NI], has[NI];
#pragma unroll
    for (int u = 0; u < NI; u++) {
        const int e = tid + CL_T * u, f = e - h * h;
        cell[u] = f < 0;
        has[u] = f < h * m;
        ik[u] = cell[u] ? e / h : f % h;
        il[u] = cell[u] ? e % h : has[u] ? f / h : 0;
    }
    const bool busy = __any_sync(0xffffffffu, has[0]);  // a warp without items only waits
    __syncthreads();
    double *cur = H1, *nxt = H0;
    for (int sweep = 0; sweep < 40; sweep++) {
        double off = 0.0, tot = 0.0;
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const double v = cur[(w + 8 * q) * CL_RS + lane];
            tot = fma(v, v, tot);
            if (w + 8 * q != lane) off = fma(v, v, off);
        }
        for (int o = 16; o > 0; o >>= 1) {
            off += __shfl_xor_sync(0xffffffffu, off, o);
            tot += __shfl_xor_sync(0xffffffffu, tot, o);
        }
        if (lane == 0) {
            wred[w] = off;
            wred[8 + w] = tot;
        }
        __syncthreads();
        double o2 = 0.0, t2 = 0.0;
        for (int v = 0; v < CL_T / 32; v++) {  // same order on every thread
            o2 += wred[v];
            t2 += wred[8 + v];
        }
        if (o2 <= 1e-26 * t2) break;  // (a round's barrier comes before wred's next write)
        for (int round = 0; round < m - 1; round++) {
            if (busy) {
                // pair k of the round: (m - 1, round) or (round + k, round - k) mod m - 1
                int a = round + lane, b = round - lane;
                if (a >= m - 1) a -= m - 1;
                if (b < 0) b += m - 1;
                if (lane == 0) a = m - 1;
                const int p = min(a, b) * CL_RS, q = max(a, b) * CL_RS;
                const int pc = min(a, b), qc = max(a, b), pq = pc | qc << 8;
                const bool pair = lane < h;
                const double app = pair ? cur[p + pc] : 1.0, aqq = pair ? cur[q + qc] : 1.0,
                             apq = pair ? cur[p + qc] : 0.0;
                int cq[NI];
                double *d0[NI], *d1[NI], x[NI], y[NI], z[NI], t[NI];
#pragma unroll
                for (int u = 0; u < NI; u++) {  // the items' entries, ahead of the angles
                    const int k = __shfl_sync(0xffffffffu, pq, ik[u]);
                    const int l = __shfl_sync(0xffffffffu, pq, cell[u] ? il[u] : 0);
                    const int pk = k & 255, qk = k >> 8, pl = l & 255, ql = l >> 8;
                    const bool in_w = has[u] && !cell[u];
                    d0[u] = in_w ? W + il[u] * CL_RS + pk : cur + pk * CL_RS + pl;
                    d1[u] = in_w ? W + il[u] * CL_RS + qk : cur + qk * CL_RS + pl;
                    cq[u] = ql - pl;
                    x[u] = *d0[u];
                    y[u] = *d1[u];
                    z[u] = cell[u] ? d0[u][cq[u]] : 0.0;
                    t[u] = cell[u] ? d1[u][cq[u]] : 0.0;
                }
                double c, s;
                jacobi_rotation<false>(app, aqq, apq, c, s);
#pragma unroll
                for (int u = 0; u < NI; u++) {
                    const double ck = __shfl_sync(0xffffffffu, c, ik[u]), sk = __shfl_sync(0xffffffffu, s, ik[u]);
                    const double cl = __shfl_sync(0xffffffffu, c, cell[u] ? il[u] : 0),
                                 sl = __shfl_sync(0xffffffffu, s, cell[u] ? il[u] : 0);
                    const double x1 = ck * x[u] - sk * y[u], y1 = sk * x[u] + ck * y[u];
                    if (cell[u]) {
                        const double z1 = ck * z[u] - sk * t[u], t1 = sk * z[u] + ck * t[u];
                        double *n0 = d0[u] + (nxt - cur), *n1 = d1[u] + (nxt - cur);
                        n0[0] = cl * x1 - sl * z1;
                        n0[cq[u]] = sl * x1 + cl * z1;
                        n1[0] = cl * y1 - sl * t1;
                        n1[cq[u]] = sl * y1 + cl * t1;
                    } else if (has[u]) {
                        *d0[u] = x1;
                        *d1[u] = y1;
                    }
                }
            }
            __syncthreads();
            double *t = cur;
            cur = nxt;
            nxt = t;
        }
    }
    if (tid < 32) {  // ascending order by rank (ties by index); a
                     // non-permutation (NaN eigenvalues) falls back
                     // to the identity order
        int rk = 0;
        if (lane < r) {
            const double d = cur[lane * CL_RS + lane];
            for (int b = 0; b < r; b++) {
                const double e = cur[b * CL_RS + b];
                rk += (e < d) || (e == d && b < lane);
            }
        }
        const unsigned bits = __reduce_or_sync(0xffffffffu, lane < r ? 1u << rk : 0u);
        const unsigned want = (r == 32) ? 0xffffffffu : ((1u << r) - 1u);
        if (lane < r) ord[bits == want ? rk : lane] = lane;
    }
    __syncthreads();
}

// Two CholQR passes on the cluster's row blocks, ya -> yb -> ya; false, in
// every CTA, when a Gram is not numerically positive definite.
__device__ __forceinline__ bool cl_orth(cg::cluster_group &cl, double *ya, double *yb, int nl, int r, double *red,
                                        double *gp, double *C, double *T, double *pub, double *dsh) {
    for (int pass = 0; pass < 2; pass++) {
        double *src = pass ? yb : ya, *dst = pass ? ya : yb, *rb = red + pass * 32 * 32;
        cl_cross(src, src, nl, r, true, gp, rb);
        cl.sync();
        cl_sum(cl, rb, r, true, C);
        if (!cl_chol_inv(C, T, r, pub, dsh)) return false;
        cl_transform(src, T, nl, r, dst);
        __syncthreads();
    }
    return true;
}

// r - ||C||_F^2 (32 x 32, row stride CL_RS), on every thread.
__device__ __forceinline__ double cl_gap(const double *C, int r, double *wred) {
    double t = 0.0;
    for (int e = threadIdx.x; e < 32 * 32; e += CL_T) {
        const double v = C[(e >> 5) * CL_RS + (e & 31)];
        t = fma(v, v, t);
    }
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if ((threadIdx.x & 31) == 0) wred[threadIdx.x >> 5] = t;
    __syncthreads();
    double g = 0.0;
    for (int w = 0; w < CL_T / 32; w++) g += wred[w];
    __syncthreads();
    return (double)r - g;
}

// V w_ord[j], ascending: the columns of W in M[j][a] = W[a][ord[j]], then
// dst = src M^T, and this CTA's rows of U.
__device__ __forceinline__ void cl_ritz_out(const double *src, const double *W, const int *ord, double *M, double *dst,
                                            int nl, int r, long i0, long n, float *__restrict__ U) {
    for (int e = threadIdx.x; e < 32 * 32; e += CL_T) {
        const int j = e >> 5, a = e & 31;
        M[j * CL_RS + a] = (j < r && a < r) ? W[a * CL_RS + ord[j]] : 0.0;
    }
    __syncthreads();
    cl_transform(src, M, nl, r, dst);
    __syncthreads();
    for (int e = threadIdx.x; e < nl * r; e += CL_T) {
        const int j = e / nl, i = e - j * nl;
        U[(i0 + i) + n * j] = (float)dst[i * CL_RS + j];
    }
}

// Y (n x r) = orth(sum of the nks partial slices) by two CholQR passes;
// with Vold, also scal[0] = r - ||Vold^T Y||_F^2.  *fail = 1 (and Y not
// written) when a Gram is not numerically positive definite.
//
// With st (a step of the iteration), the convergence test runs here, so
// the host can queue several steps and read the state once: st[0] done
// (later launches return at once), st[1] the steps still to run after the
// gap first fell below the tolerance, plus one (0: not yet), st[2] steps
// taken, st[3] the step whose iterate is final.  The state is read on entry
// by every CTA and written by CTA 0 only after the cluster's last barrier,
// so all CTAs of a launch see the same value.
__global__ void __cluster_dims__(CL_N, 1, 1) __launch_bounds__(CL_T)
    k_si_orth_cl(const double *__restrict__ part, int nks, const double *__restrict__ Vold, long n, int r,
                 double *__restrict__ Y, double *scal, int *fail, int *st) {
    if (st && st[0]) return;
    cg::cluster_group cl = cg::this_cluster();
    extern __shared__ double smc[];
    __shared__ double pub[128], dsh[32], wred[CL_T / 32];
    const ClLayout L = cl_layout(n);
    const int rank = (int)cl.block_rank();
    const long i0 = (long)rank * L.nl;
    const int nl = (int)max(0L, min((long)L.nl, n - i0));
    double *ya = smc + L.ya, *yb = smc + L.yb, *red = smc + L.red, *gp = smc + L.gp, *C = smc + L.C,
           *T = smc + L.T;
    cl_load_rows(part, nks, n, r, i0, nl, ya);
    __syncthreads();
    if (!cl_orth(cl, ya, yb, nl, r, red, gp, C, T, pub, dsh)) {  // the same verdict in every CTA
        cl.sync();                                                  // peers may still read this CTA's buffers
        if (rank == 0 && threadIdx.x == 0) {
            *fail = 1;
            if (st) st[0] = 1;
        }
        return;
    }
    if (Vold) {
        cl_load_rows(Vold, 1, n, r, i0, nl, yb);
        __syncthreads();
        cl_cross(yb, ya, nl, r, false, gp, red);  // buffer 0: its readers all passed the last cluster barrier
        cl.sync();
        if (rank == 0) {
            cl_sum(cl, red, r, false, C);
            const double g = cl_gap(C, r, wred);
            if (threadIdx.x == 0) scal[0] = g;
        }
    }
    for (int e = threadIdx.x; e < nl * r; e += CL_T) {
        const int a = e / nl, i = e - a * nl;
        Y[(i0 + i) + n * a] = ya[i * CL_RS + a];
    }
    cl.sync();  // keep this CTA's buffers alive until every peer has read them
    if (st && rank == 0 && threadIdx.x == 0) {
        // one more step after the gap first falls below the tolerance
        const int step = st[2] + 1;
        int extra = st[1] - 1;
        if (extra < 0 && scal[0] < 1e-13 * (double)r) extra = 1;
        if (extra >= 0 && extra-- == 0) {
            st[0] = 1;
            st[3] = step;
        }
        st[1] = extra + 1;
        st[2] = step;
    }
}

// Rayleigh-Ritz: H = V^T (G V) (G V = the sum of the partial slices),
// Jacobi on H, U[:, j] = V w_ord[j] with the eigenvalues ascending.
__global__ void __cluster_dims__(CL_N, 1, 1) __launch_bounds__(CL_T)
    k_si_ritz_cl(const double *__restrict__ part, int nks, const double *__restrict__ V, long n, int r,
                 float *__restrict__ U) {
    cg::cluster_group cl = cg::this_cluster();
    extern __shared__ double smc[];
    __shared__ double wred[16];
    __shared__ int ord[32];
    const ClLayout L = cl_layout(n);
    const int rank = (int)cl.block_rank();
    const long i0 = (long)rank * L.nl;
    const int nl = (int)max(0L, min((long)L.nl, n - i0));
    double *ya = smc + L.ya, *yb = smc + L.yb, *red = smc + L.red, *gp = smc + L.gp, *H = smc + L.C,
           *W = smc + L.T;
    cl_load_rows(part, nks, n, r, i0, nl, ya);
    cl_load_rows(V, 1, n, r, i0, nl, yb);
    __syncthreads();
    cl_cross(yb, ya, nl, r, false, gp, red);
    cl.sync();
    cl_sum(cl, red, r, false, H);
    cl_jacobi<3>(H, gp, W, r, ord, wred);
    cl_ritz_out(yb, W, ord, gp + 32 * CL_RS, ya, nl, r, i0, n, U);
    cl.sync();  // keep this CTA's buffers alive until every peer has read them
}

// ------------------------------------------------- the iteration in one launch
// Where an eighth of G fits in a CTA's shared memory beside two copies of V,
// one cluster keeps G there (its rows, as the iterate's) and runs the whole
// iteration: start block, steps, Rayleigh-Ritz.  The n x r products are FP64
// matrix instructions on shared memory; each CTA sends its rows of the
// result to its peers' copies (distributed shared memory), so a step waits
// on four cluster barriers.  Bound by the serial chain of the r x r work
// between them.  B200, each of the three modes of a 256^3 rank-16 HOSVD:
// 260 us of kernels, and the gaps between 11 launches, with a launch per
// product and per orthonormalisation; 105 us here (the whole call 1333 us,
// now 782).

// Dynamic shared memory (offsets in doubles): G's rows (padded to eights, row
// stride ldg), the two copies of V (row-major, row stride ldv; the second
// also holds the tile partials of the r x r work, which needs it between two
// products only), then as ClLayout.  ldg and ldv are 4 mod 8, so that the
// fragments' four rows or columns fall in different banks.
struct RunLayout {
    int nl, nlp, kp, ldg, ldv;
    size_t va, vb, ya, yb, red, C, T, total;
};
__host__ __device__ inline RunLayout run_layout(long n, int nt) {
    RunLayout L;
    L.nl = (int)((n + CL_N - 1) / CL_N);
    L.nlp = (L.nl + 7) / 8 * 8;
    L.kp = (int)((n + 7) / 8 * 8);
    L.ldg = L.kp + 4;
    L.ldv = 8 * nt + 4;
    const size_t v = (size_t)L.kp * L.ldv, gp = (size_t)CL_T * 16;
    L.va = (size_t)L.nlp * L.ldg;
    L.vb = L.va + v;
    L.ya = L.vb + (v > gp ? v : gp);
    L.yb = L.ya + (size_t)L.nl * CL_RS;
    L.red = (L.yb + (size_t)L.nl * CL_RS + 1) / 2 * 2;
    L.C = L.red + 2 * 32 * 32;
    L.T = L.C + 32 * CL_RS;
    L.total = L.T + 32 * CL_RS;
    return L;
}
constexpr size_t RUN_SMEM_MAX = 224 * 1024;

// out (nl x r, row stride CL_RS) = this CTA's rows of G V.  A warp takes 8
// rows and a share of k, with two accumulator sets for the matrix
// instructions' latency; the shares are added in order.  part: 32 x 64
// doubles.  Ends on a block barrier.
template <int NT>
__device__ __forceinline__ void run_apply(const RunLayout &L, const double *G, const double *V, double *part,
                                          double *out) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int mt = L.nlp / 8, ks = max(1, (CL_T / 32) / mt), nk = L.kp / 4;
    for (int it = w; it < mt * ks; it += CL_T / 32) {
        const int m = it % mt, s = it / mt;
        const int k0 = s * nk / ks, k1 = (s + 1) * nk / ks;
        double acc[2][NT][2];
#pragma unroll
        for (int j = 0; j < NT; j++) acc[0][j][0] = acc[0][j][1] = acc[1][j][0] = acc[1][j][1] = 0.0;
        const double *g = G + (8 * m + (lane >> 2)) * L.ldg + (lane & 3) + 4 * k0;
        const double *v = V + ((lane & 3) + 4 * k0) * L.ldv + (lane >> 2);
        const int step = 4 * L.ldv;
        int k = k0;
#pragma unroll 4
        for (; k + 1 < k1; k += 2) {
#pragma unroll
            for (int u = 0; u < 2; u++) {
                const double a = *g;
#pragma unroll
                for (int j = 0; j < NT; j++) dmma(acc[u][j], a, v[8 * j]);
                g += 4;
                v += step;
            }
        }
        if (k < k1) {
            const double a = *g;
#pragma unroll
            for (int j = 0; j < NT; j++) dmma(acc[0][j], a, v[8 * j]);
        }
#pragma unroll
        for (int j = 0; j < NT; j++)
#pragma unroll
            for (int x = 0; x < 2; x++)
                part[((s * mt + m) * 8 + (lane >> 2)) * (8 * NT) + 8 * j + 2 * (lane & 3) + x] =
                    acc[0][j][x] + acc[1][j][x];
    }
    __syncthreads();
    for (int e = threadIdx.x; e < L.nl * 8 * NT; e += CL_T) {
        const int i = e / (8 * NT), c = e % (8 * NT);
        double t = 0.0;
        for (int s = 0; s < ks; s++) t += part[(s * mt * 8 + i) * (8 * NT) + c];
        out[i * CL_RS + c] = t;
    }
    __syncthreads();
}

// Every CTA's copy V (rows i0 .. i0 + nl - 1) = src.  The caller synchronises
// the cluster.
template <int NT>
__device__ __forceinline__ void run_send(cg::cluster_group &cl, const RunLayout &L, const double *src, int nl, long i0,
                                         double *V) {
    for (int e = threadIdx.x; e < nl * 4 * NT; e += CL_T) {
        const int i = e / (4 * NT), c = e % (4 * NT);
        const double2 v = make_double2(src[i * CL_RS + 2 * c], src[i * CL_RS + 2 * c + 1]);
        double *d = V + (i0 + i) * L.ldv + 2 * c;
#pragma unroll
        for (int q = 0; q < CL_N; q++) *reinterpret_cast<double2 *>(cl.map_shared_rank(d, q)) = v;
    }
}

// state (pinned host memory): 1 converged, 2 not within max_iters, 3 a rank-
// deficient iterate; U is written in the first case only.  products: G V or
// G^2 V a step, and two or one more steps once the tolerance is met -- the steps
// of the path that had the call before this kernel (see top_eigvecs_run), so
// that the vectors keep their signs, which are the iterate's.
template <int NT>
__global__ void __cluster_dims__(CL_N, 1, 1) __launch_bounds__(CL_T)
    k_si_run_cl(const double *__restrict__ Gm, long n, int r, const float *U0, float *U, int max_iters, int products,
                volatile int *state) {
    cg::cluster_group cl = cg::this_cluster();
    extern __shared__ __align__(16) double smc[];
    __shared__ double pub[128], dsh[32], wred[16];
    __shared__ int ord[32];
    const RunLayout L = run_layout(n, NT);
    const int rank = (int)cl.block_rank();
    const long i0 = (long)rank * L.nl;
    const int nl = (int)max(0L, min((long)L.nl, n - i0));
    double *G = smc, *va = smc + L.va, *vb = smc + L.vb, *gp = vb, *ya = smc + L.ya, *yb = smc + L.yb,
           *red = smc + L.red, *C = smc + L.C, *T = smc + L.T;
    // G's rows are on their way while the start block is orthonormalised
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int i = lane; i < L.nlp; i += 32)
#pragma unroll 4
        for (int k = w; k < L.kp; k += CL_T / 32) {
            double *d = G + i * L.ldg + k;
            if (i < nl && k < n)
                asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(d)),
                             "l"(Gm + (i0 + i) + n * k)
                             : "memory");
            else
                *d = 0.0;
        }
    asm volatile("cp.async.commit_group;" ::: "memory");
    for (int e = threadIdx.x; e < (L.kp - (int)n) * L.ldv; e += CL_T) va[n * L.ldv + e] = 0.0;
    for (int i = lane; i < L.nl; i += 32)
        for (int a = w; a < CL_RS; a += CL_T / 32) {
            const long x = (i0 + i) + n * a;
            ya[i * CL_RS + a] = (i < nl && a < r) ? (U0 ? (double)U0[x] : si_start(x)) : 0.0;
            yb[i * CL_RS + a] = 0.0;
        }
    __syncthreads();
    int verdict = 0;  // the same in every CTA
    if (!cl_orth(cl, ya, yb, nl, r, red, gp, C, T, pub, dsh)) verdict = 3;
    run_send<NT>(cl, L, ya, nl, i0, va);
    asm volatile("cp.async.wait_all;" ::: "memory");
    cl.sync();
    int extra = -1;  // steps still to run after the tolerance is met
    for (int step = 0; verdict == 0; step++) {
        if (step == max_iters) {
            verdict = 2;
            break;
        }
        if (products == 2) {
            // two products per orthonormalisation (G^2 V): the columns' condition
            // grows by (lambda_1 / lambda_r)^2 per step, well inside CholQR2's range
            run_apply<NT>(L, G, va, C, yb);
            for (int e = threadIdx.x; e < (L.kp - (int)n) * L.ldv; e += CL_T) vb[n * L.ldv + e] = 0.0;
            run_send<NT>(cl, L, yb, nl, i0, vb);
            cl.sync();
            run_apply<NT>(L, G, vb, C, ya);
        } else {
            run_apply<NT>(L, G, va, C, ya);
            cl.sync();  // the gap's buffer has been read by every peer
        }
        if (!cl_orth(cl, ya, yb, nl, r, red, gp, C, T, pub, dsh)) {
            verdict = 3;
            break;
        }
        // the gap r - ||Vold^T V||^2, and V to the peers under the same barrier
        for (int e = threadIdx.x; e < nl * 32; e += CL_T) {
            const int i = e >> 5, a = e & 31;
            yb[i * CL_RS + a] = (a < r) ? va[(i0 + i) * L.ldv + a] : 0.0;
        }
        __syncthreads();
        cl_cross(yb, ya, nl, r, false, gp, red);
        run_send<NT>(cl, L, ya, nl, i0, va);
        cl.sync();
        cl_sum(cl, red, r, false, C);
        const double gap = cl_gap(C, r, wred);
        // one more step (two of one product) after the gap first falls below the
        // tolerance
        if (extra < 0 && gap < 1e-13 * (double)r) extra = 3 - products;
        if (extra >= 0 && extra-- == 0) verdict = 1;
    }
    if (verdict == 1) {
        // Rayleigh-Ritz on H = V^T (G V).  The second of the two buffers the
        // peers read: the first may still be read for the gap.
        run_apply<NT>(L, G, va, C, yb);
        cl_cross(ya, yb, nl, r, false, gp, red + 32 * 32);
        cl.sync();
        cl_sum(cl, red + 32 * 32, r, false, C);
        cl_jacobi<NT <= 2 ? 1 : NT - 1>(C, gp, T, r, ord, wred);
        cl_ritz_out(ya, T, ord, gp + 32 * CL_RS, yb, nl, r, i0, n, U);
    }
    if (rank == 0 && threadIdx.x == 0) *state = verdict;
    cl.sync();  // keep this CTA's buffers alive until every peer has read them
}

// part[y] (n x r) = G[:, slice y] V[slice y, :] for the k slices of kchunk
// rows (V given as the sum of nin n x r slices, summed in slice order).  A
// CTA takes 32 rows of G (one per lane) and one k slice; warp w forms
// columns 4w .. 4w+3, so each output has one owner and no cross-warp sum.
constexpr int AP_KB = 64;  // rows of V staged per pass
__global__ void __launch_bounds__(256) k_si_apply_cols(const double *__restrict__ G, const double *__restrict__ V,
                                                       int nin, long n, int r, long kchunk,
                                                       double *__restrict__ part, const int *st) {
    if (st && st[0]) return;  // the iteration has converged (k_si_orth_cl)
    __shared__ double sv[AP_KB][SI_FR + 1];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const long i = blockIdx.x * 32L + lane;
    const long k0 = blockIdx.y * kchunk, k1 = min(n, k0 + kchunk);
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    for (long kb = k0; kb < k1; kb += AP_KB) {
        const int nk = (int)min((long)AP_KB, k1 - kb);
        __syncthreads();
        for (int e = threadIdx.x; e < AP_KB * SI_FR; e += 256) {
            const int kk = e % AP_KB, c = e / AP_KB;
            double v = 0.0;
            if (kk < nk && c < r)
                for (int y = 0; y < nin; y++) v += V[(long)y * n * r + (kb + kk) + n * c];
            sv[kk][c] = v;
        }
        __syncthreads();
        if (i < n && 4 * w < r) {
            const double *g = G + i + n * kb;
#pragma unroll 16
            for (int kk = 0; kk < nk; kk++) {
                const double gv = g[n * kk];
#pragma unroll
                for (int u = 0; u < 4; u++) acc[u] = fma(gv, sv[kk][4 * w + u], acc[u]);
            }
        }
    }
    if (i < n)
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int c = 4 * w + u;
            if (c < r) part[(long)blockIdx.y * n * r + i + n * c] = acc[u];
        }
}

// After each batch of steps in the loop graph: whether its WHILE node runs
// another batch -- the host loop's rule (stop once the iteration has
// converged or failed, or max_iters steps have run; every step of a batch
// that has not converged runs, so st[2] counts the steps queued).
__global__ void k_si_loop_cond(cudaGraphConditionalHandle h, const int *fail, const int *st, int max_iters) {
    if (threadIdx.x != 0) return;
    const bool more = *fail == 0 && st[0] == 0 && st[2] < max_iters;
    cudaGraphSetConditional(h, more ? 1u : 0u);
}

constexpr int SI_BATCH = 4;  // steps queued between two reads of the state

// One batch of SI_BATCH fast-path steps from V = buffer 0 (ws), as the host
// loop queues it; SI_BATCH is even, so the batch ends with V in buffer 0
// again and every batch is the same launch sequence.
struct SiSteps {
    const double *G;
    long n;
    int r, nks;
    long kchunk;
    dim3 ga;
    size_t smem;
    double *ws, *part, *part2, *scal;
    int *fail, *st;
    void enqueue(int steps, cudaStream_t s) const {
        const long nr = n * (long)r;
        double *V = ws, *Y = ws + nr;
        for (int b = 0; b < steps; b++) {
            // two products per orthonormalisation (G^2 V): the columns' condition
            // grows by (lambda_1 / lambda_r)^2 per step, well inside CholQR2's range
            k_si_apply_cols<<<ga, 256, 0, s>>>(G, V, 1, n, r, kchunk, part2, st);
            k_si_apply_cols<<<ga, 256, 0, s>>>(G, part2, nks, n, r, kchunk, part, st);
            k_si_orth_cl<<<CL_N, CL_T, smem, s>>>(part, nks, V, n, r, Y, scal, fail, st);
            std::swap(V, Y);
        }
    }
};

// Loop graphs of the fast path, one per (device, G, n, r, ws, nks,
// max_iters): a WHILE node whose body is one batch and k_si_loop_cond, so a
// call reads the state once instead of once per batch.  The key holds the
// exact pointers the captured launches use.  A few entries (the Tucker
// drivers call with one Gram and one workspace per plan), never replaced,
// since another thread may be launching one: once all are taken, new keys
// keep the host loop.
struct SiGraph {
    int dev = -1;
    const double *G = nullptr, *ws = nullptr;
    long n = 0;
    int r = 0, nks = 0, max_iters = 0;
    cudaGraphExec_t ex = nullptr;
};
constexpr int SI_GRAPHS = 8;
std::mutex g_si_mu;
SiGraph g_si[SI_GRAPHS];
int g_si_used = 0;
bool g_si_refused[64] = {};  // per device: the driver refused a loop graph once; keep the host loop

// Capture the loop graph on a private stream (capturing records the
// launches without running them); null when the driver refuses any step,
// and the caller keeps the host loop.
cudaGraphExec_t si_build_loop(const SiSteps &k, int max_iters) {
    cudaStream_t cs = nullptr;
    if (cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking) != cudaSuccess) {
        (void)cudaGetLastError();
        return nullptr;
    }
    cudaGraph_t g = nullptr;
    cudaGraphExec_t ex = nullptr;
    bool ok = cudaGraphCreate(&g, 0) == cudaSuccess;
    cudaGraphConditionalHandle h = 0;
    cudaGraph_t body = nullptr;
    if (ok) ok = cudaGraphConditionalHandleCreate(&h, g, 1, cudaGraphCondAssignDefault) == cudaSuccess;
    if (ok) {
        cudaGraphNodeParams np = {};
        np.type = cudaGraphNodeTypeConditional;
        np.conditional.handle = h;
        np.conditional.type = cudaGraphCondTypeWhile;
        np.conditional.size = 1;
        cudaGraphNode_t node;
        ok = cudaGraphAddNode(&node, g, nullptr, 0, &np) == cudaSuccess;
        if (ok) body = np.conditional.phGraph_out[0];
    }
    if (ok) ok = cudaStreamBeginCaptureToGraph(cs, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal) ==
                 cudaSuccess;
    if (ok) {
        k.enqueue(SI_BATCH, cs);
        k_si_loop_cond<<<1, 32, 0, cs>>>(h, k.fail, k.st, max_iters);
        const bool launched = cudaGetLastError() == cudaSuccess;
        cudaGraph_t captured = nullptr;
        ok = cudaStreamEndCapture(cs, &captured) == cudaSuccess && launched;
    }
    if (ok) ok = cudaGraphInstantiate(&ex, g, 0) == cudaSuccess;
    (void)cudaGetLastError();
    if (!ok && ex) {
        cudaGraphExecDestroy(ex);
        ex = nullptr;
    }
    if (g) cudaGraphDestroy(g);  // the executable graph keeps what it needs
    cudaStreamDestroy(cs);
    return ex;
}

cudaGraphExec_t si_loop_graph(int dev, const SiSteps &k, int max_iters) {
    std::lock_guard<std::mutex> lk(g_si_mu);
    for (const SiGraph &e : g_si)
        if (e.ex && e.dev == dev && e.G == k.G && e.ws == k.ws && e.n == k.n && e.r == k.r && e.nks == k.nks &&
            e.max_iters == max_iters)
            return e.ex;
    if (g_si_used == SI_GRAPHS || g_si_refused[dev]) return nullptr;
    cudaGraphExec_t ex = si_build_loop(k, max_iters);
    if (!ex) {
        g_si_refused[dev] = true;
        return nullptr;
    }
    SiGraph &slot = g_si[g_si_used++];
    slot.dev = dev; slot.G = k.G; slot.ws = k.ws; slot.n = k.n; slot.r = k.r; slot.nks = k.nks;
    slot.max_iters = max_iters;
    slot.ex = ex;
    return ex;
}

}  // namespace

size_t subspace_ws_doubles(long n, long r) { return 3 * (size_t)n * r + 8; }  // V, Y, W (r*r <= n*r), scalars

// The whole iteration in one launch of a cluster (k_si_run_cl).
// CUD_ERR_UNSUPPORTED when its shared memory or the cluster does not fit.
// Steps of two products where ws_doubles would hold top_eigvecs_fast's partial
// products (it needs no workspace itself), of one where the general loop below
// would run.
template <int NT>
static int top_eigvecs_run(const double *G, long n, long r, float *U, size_t ws_doubles, int max_iters,
                           cudaStream_t s, const float *U0) {
    const size_t smem = run_layout(n, NT).total * sizeof(double);
    if (smem > RUN_SMEM_MAX) return CUD_ERR_UNSUPPORTED;
    int dev = 0;
    CUD_CHECK(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return CUD_ERR_UNSUPPORTED;
    static std::atomic<int> ready[64];  // 0 unknown, 1 usable, 2 not; zero-initialised
    if (!ready[dev]) {
        CUD_CHECK(cudaFuncSetAttribute(k_si_run_cl<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)RUN_SMEM_MAX));
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(CL_N);
        cfg.blockDim = dim3(CL_T);
        cfg.dynamicSmemBytes = RUN_SMEM_MAX;
        int nc = 0;
        const cudaError_t e = cudaOccupancyMaxActiveClusters(&nc, k_si_run_cl<NT>, &cfg);
        ready[dev] = (e == cudaSuccess && nc > 0) ? 1 : 2;
        (void)cudaGetLastError();
    }
    if (ready[dev] != 1) return CUD_ERR_UNSUPPORTED;
    double *h = pinned_scalars();
    if (!h) return CUD_ERR_NO_MEMORY;
    volatile int *state = reinterpret_cast<volatile int *>(h);
    *state = 0;
    const int products = ws_doubles >= 4 * (size_t)n * r + 8 ? 2 : 1;
    k_si_run_cl<NT><<<CL_N, CL_T, smem, s>>>(G, n, (int)r, U0, U, max_iters, products, state);
    CUD_CHECK_LAUNCH("subspace iteration");
    CUD_CHECK(cudaStreamSynchronize(s));
    return *state == 1 ? CUD_OK : CUD_ERR_NOT_CONVERGED;
}

// Fast path (r <= 32, n <= 2048): ws holds V, Y (n x r each) and two sets
// of nks partial products, nks as many as ws_doubles allows (at most 8).
// Each step forms G^2 V (two split products), then orthonormalises and
// measures the subspace change.
static int top_eigvecs_fast(const double *G, long n, long r, float *U, double *ws, size_t ws_doubles,
                            int max_iters, cudaStream_t s, const float *U0) {
    const long nr = n * r;
    const long room = ((long)ws_doubles - 2 * nr - 8) / (2 * nr);
    const int nks = (int)std::max(0L, std::min(8L, room));
    if (nks < 1) return CUD_ERR_UNSUPPORTED;
    const size_t smem = cl_layout(n).total * sizeof(double);
    int dev = 0;
    CUD_CHECK(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return CUD_ERR_UNSUPPORTED;
    {
        // once per device: the shared-memory opt-in, and whether a cluster
        // of this size can be resident at all
        static std::atomic<int> ready[64];  // 0 unknown, 1 usable, 2 not; zero-initialised
        if (!ready[dev]) {
            CUD_CHECK(cudaFuncSetAttribute(k_si_orth_cl, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)CL_SMEM_MAX));
            CUD_CHECK(cudaFuncSetAttribute(k_si_ritz_cl, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)CL_SMEM_MAX));
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(CL_N);
            cfg.blockDim = dim3(CL_T);
            cfg.dynamicSmemBytes = CL_SMEM_MAX;
            int nc = 0;
            const cudaError_t e1 = cudaOccupancyMaxActiveClusters(&nc, k_si_orth_cl, &cfg);
            int nc2 = 0;
            const cudaError_t e2 = cudaOccupancyMaxActiveClusters(&nc2, k_si_ritz_cl, &cfg);
            ready[dev] = (e1 == cudaSuccess && e2 == cudaSuccess && nc > 0 && nc2 > 0) ? 1 : 2;
            (void)cudaGetLastError();
        }
        if (ready[dev] != 1) return CUD_ERR_UNSUPPORTED;
    }
    double *V = ws, *Y = ws + nr, *part = ws + 2 * nr, *part2 = ws + (2 + nks) * nr,
           *scal = ws + (2 + 2 * nks) * nr;
    int *fail = reinterpret_cast<int *>(scal + 2);
    int *st = reinterpret_cast<int *>(scal + 3);  // 4 ints: done, extra + 1, steps, final step
    double *h = pinned_scalars();
    if (!h) return CUD_ERR_NO_MEMORY;
    const long kchunk = (n + nks - 1) / nks;
    const dim3 ga((unsigned)((n + 31) / 32), (unsigned)nks);
    const unsigned gi = (unsigned)std::min<long>((nr + 255) / 256, 4L * kNumSMs);
    CUD_CHECK(cudaMemsetAsync(fail, 0, 3 * sizeof(double), s));  // fail and the state
    if (U0) k_si_init_from<<<gi, 256, 0, s>>>(U0, Y, n, (int)r);
    else k_si_init<<<gi, 256, 0, s>>>(Y, n, (int)r);
    k_si_orth_cl<<<CL_N, CL_T, smem, s>>>(Y, 1, nullptr, n, (int)r, V, scal, fail, nullptr);
    CUD_CHECK_LAUNCH("subspace init");
    // Steps are queued SI_BATCH at a time and the launches after convergence
    // return at once.  Step j (from 1) writes buffer j % 2 (buffer 0 = the
    // initial V).  When max_iters is a whole number of batches, the batches
    // run in the loop graph and the state is read once; otherwise the host
    // reads it after every batch.
    const SiSteps k{G, n, (int)r, nks, kchunk, ga, smem, ws, part, part2, scal, fail, st};
    const cudaGraphExec_t loop = (max_iters % SI_BATCH == 0) ? si_loop_graph(dev, k, max_iters) : nullptr;
    for (int queued = 0; queued < max_iters;) {
        if (loop) {
            CUD_CHECK(cudaGraphLaunch(loop, s));
            queued = max_iters;
        } else {
            const int nb = std::min(SI_BATCH, max_iters - queued);
            k.enqueue(nb, s);
            CUD_CHECK_LAUNCH("subspace steps");
            queued += nb;
        }
        CUD_CHECK(cudaMemcpyAsync(h, scal + 2, 3 * sizeof(double), cudaMemcpyDeviceToHost, s));
        CUD_CHECK(cudaStreamSynchronize(s));
        const int *hs = reinterpret_cast<const int *>(h);  // fail, pad, done, extra + 1, steps, final
        if (hs[0]) return CUD_ERR_NOT_CONVERGED;          // rank-deficient iterate
        if (hs[2]) {
            const double *Vf = ws + ((hs[5] % 2) ? nr : 0);
            k_si_apply_cols<<<ga, 256, 0, s>>>(G, Vf, 1, n, (int)r, kchunk, part, nullptr);
            k_si_ritz_cl<<<CL_N, CL_T, smem, s>>>(part, nks, Vf, n, (int)r, U);
            CUD_CHECK_LAUNCH("subspace ritz");
            return CUD_OK;
        }
    }
    return CUD_ERR_NOT_CONVERGED;
}

static int subspace_run(const double *G, long n, long r, float *U, double *ws, size_t ws_doubles, int max_iters,
                        cudaStream_t s, const float *U0) {
    if (r <= SI_FR) {
        const int st = r <= 8    ? top_eigvecs_run<1>(G, n, r, U, ws_doubles, max_iters, s, U0)
                       : r <= 16 ? top_eigvecs_run<2>(G, n, r, U, ws_doubles, max_iters, s, U0)
                       : r <= 24 ? top_eigvecs_run<3>(G, n, r, U, ws_doubles, max_iters, s, U0)
                                 : top_eigvecs_run<4>(G, n, r, U, ws_doubles, max_iters, s, U0);
        if (st != CUD_ERR_UNSUPPORTED) return st;
    }
    if (r <= SI_FR && n <= 2048 && cl_layout(n).total * sizeof(double) <= CL_SMEM_MAX) {
        const int st = top_eigvecs_fast(G, n, r, U, ws, ws_doubles, max_iters, s, U0);
        if (st != CUD_ERR_UNSUPPORTED) return st;
    }
    double *V = ws, *Y = ws + n * r, *Wr = ws + 2 * n * r, *scal = ws + 3 * n * r;
    int *fail = reinterpret_cast<int *>(scal + 2);
    double *h = pinned_scalars();
    if (!h) return CUD_ERR_NO_MEMORY;
    const unsigned gb = (unsigned)std::min<long>((n * r + 255) / 256, 4L * kNumSMs);
    CUD_CHECK(cudaMemsetAsync(fail, 0, sizeof(int), s));
    if (U0) k_si_init_from<<<gb, 256, 0, s>>>(U0, V, n, (int)r);
    else k_si_init<<<gb, 256, 0, s>>>(V, n, (int)r);
    k_si_cholqr<<<1, 256, 0, s>>>(V, n, (int)r, fail);
    k_si_cholqr<<<1, 256, 0, s>>>(V, n, (int)r, fail);
    CUD_CHECK_LAUNCH("subspace init");
    int extra = -1;  // iterations still to run after the tolerance is met
    for (int it = 0; it < max_iters; it++) {
        k_si_apply<<<gb, 256, 0, s>>>(G, V, n, (int)r, Y);
        k_si_cholqr<<<1, 256, 0, s>>>(Y, n, (int)r, fail);
        k_si_cholqr<<<1, 256, 0, s>>>(Y, n, (int)r, fail);
        k_si_gap<<<1, 256, 0, s>>>(V, Y, n, (int)r, scal);
        CUD_CHECK_LAUNCH("subspace step");
        std::swap(V, Y);
        CUD_CHECK(cudaMemcpyAsync(h, scal, 3 * sizeof(double), cudaMemcpyDeviceToHost, s));
        CUD_CHECK(cudaStreamSynchronize(s));
        if (reinterpret_cast<int *>(h + 2)[0]) return CUD_ERR_NOT_CONVERGED;  // rank-deficient iterate
        if (extra < 0 && h[0] < 1e-13 * (double)r) extra = 2;
        if (extra >= 0 && extra-- == 0) {
            k_si_apply<<<gb, 256, 0, s>>>(G, V, n, (int)r, Y);
            k_si_ritz<<<1, 256, 0, s>>>(V, Y, n, (int)r, U, Wr);
            CUD_CHECK_LAUNCH("subspace ritz");
            return CUD_OK;
        }
    }
    return CUD_ERR_NOT_CONVERGED;
}

int top_eigvecs_subspace(const double *G, long n, long r, float *U, double *ws, size_t ws_doubles, int max_iters,
                         cudaStream_t s, const float *U0) {
    if (r <= 0 || r > SI_RMAX || r > n) return CUD_ERR_UNSUPPORTED;
    if (U0) {
        // U is written only on success: a failed warm start (a rank-
        // deficient start block) retries from the random block
        const int st = subspace_run(G, n, r, U, ws, ws_doubles, max_iters, s, U0);
        if (st != CUD_ERR_NOT_CONVERGED) return st;
    }
    return subspace_run(G, n, r, U, ws, ws_doubles, max_iters, s, nullptr);
}

}  // namespace cud

extern "C" int cud_syev_top(const double *G, long n, long r, float *U, const float *U0, int max_iters,
                            void *stream) {
    if (n <= 0 || r <= 0 || r > n || !G || !U || max_iters <= 0) return cud::set_status(CUD_ERR_INVALID_ARGUMENT);
    // room for the fast path's eight k slices of partial products
    const size_t wsd = std::max(cud::subspace_ws_doubles(n, r), (size_t)18 * (size_t)n * (size_t)r + 8);
    int st;
    double *ws = static_cast<double *>(cud::scratch(cud::kSlotEig, wsd * sizeof(double), &st));
    if (!ws) return cud::set_status(st);
    return cud::set_status(cud::top_eigvecs_subspace(G, n, r, U, ws, wsd, max_iters, cud::as_stream(stream), U0));
}
