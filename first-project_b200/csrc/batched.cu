// Batched CP-ALS: thousands of small, independent 3rd-order tensors of uneven
// shape and rank, one persistent kernel launch per ALS sweep for the whole
// batch (sized for 4096 tensors with dims in [16, 96] and ranks in [4, 16]).
//
// CTAs -- clusters of 2 to 8 of them where the tensors are too few to fill the
// GPU -- pull tensors from a work queue (largest first) and run one full sweep
// of that tensor, everything on-chip except X:
//   * the three factor matrices live in shared memory (<= 96 x 16 each,
//     row-major with the ranks padded to 16 with zeros);
//   * each MTTKRP streams X by cp.async through a ring per warp, the lanes
//     along the tensor's contiguous index i (one coalesced 128-byte request
//     per warp and copy), and contracts it against factor rows broadcast from
//     shared memory in packed FP32 FMAs (the ranks are too small for tensor
//     cores to pay); mode 1 keeps each lane's own row of M, modes 2 and 3
//     sum the lanes' terms by a recursive-halving shuffle (mttkrp_lanes);
//   * the R x R normal equations (Hadamard of the FP64 Grams) are inverted
//     by Gauss-Jordan (FP64, a cell per thread), with a tiny diagonal shift
//     retried when a pivot is not positive;
//   * the fit comes from ||X||^2 - 2 <M_3, C> + sum prod G (FP64), per
//     tensor; a tensor whose fit changed by less than `tol` is marked
//     converged and skipped by later sweeps.
// The host captures `sweeps_per_graph` sweeps (queue reset + kernel) in one
// CUDA graph and replays it until every tensor has converged or hit the
// sweep limit.  The CTAs a tensor and per SM come from a rule on the number of
// tensors (default_cfg), or from a small autotuner (cud_cp_batched_tune) that
// times two sweeps per candidate on the batch itself and caches the winner per
// batch shape class.
#include <cooperative_groups.h>

#include <atomic>
#include <map>
#include <mutex>
#include <vector>
#include <algorithm>

#include "kernels.cuh"
#include "tc_ptx.cuh"

namespace cg = cooperative_groups;

namespace cud {

namespace {

constexpr int BMAXD = 96;    // largest mode size handled (smem sizing)
constexpr int BMAXR = 16;    // largest rank handled
constexpr int RS = BMAXR;    // row stride of factors and results in shared memory (ranks padded)
constexpr int NORM_PARTS = 8;  // CTAs that share a tensor's norm

struct TensorMeta {
    long xoff;          // offset of X (elements) in the packed tensor buffer
    long uoff[3];       // offsets of the factors in the packed factor buffer
    int dims[3];
    int R;
    int done;
    int sweeps;
    double fit, fit_prev;
    double target;      // stop once fit >= target (<= 0: no target)
};

// What a tensor keeps on the device alone between sweeps.
struct TensorState {
    double normp[NORM_PARTS];    // ||X||^2 by parts of the tensor
    double G[3][BMAXR * BMAXR];  // factor Grams (FP64)
};

struct BatchArgs {
    TensorMeta *meta;
    TensorState *state;
    const int *order;   // processing order (largest first)
    int ntensors;
    const float *X;
    float *U;
    unsigned *queue;    // work counter, zero at kernel start
    int *ndone;         // tensors marked converged so far
    int *error;         // set by a wait that ran out
    int max_sweeps;
    double tol;
    int *fallbacks;
};

// Shared memory of a CTA of NW warps: the factors and the MTTKRP result
// row-major (rank contiguous, ranks padded to RS), and the partial results of
// the (at most three) 32-row chunks of modes 2 and 3.
constexpr int MAXCHUNK = (BMAXD + 31) / 32;
// Outer and inner indices of X per group of the MTTKRP, and groups in flight.
constexpr int NO = 4, UN = 4, RING = 4;

template <int NW, int CL>
struct BatchSmem {
    float F[3][BMAXD * RS];                     // rows to a multiple of 4, the last ones zero
    union {
        struct {
            float M[BMAXD * RS];                // this CTA's rows
            float Mg[CL > 1 ? BMAXD * RS : 4];  // the whole result, gathered from the cluster
        };
        float mail[CL > 1 ? NW : 1][BMAXR][32]; // mode 0, before the gather: the sums from the CTA before
    };
    float Mp[MAXCHUNK][BMAXD * RS];
    double G[3][BMAXR * BMAXR];                 // factor Grams (R x R, column-major)
    double V[BMAXR * BMAXR];                    // inverse of the normal matrix, row-major with stride RS
    double row[2][BMAXR], col[2][BMAXR], inv[2];
    double red[2 * NW];
    double diag[BMAXR];
    int tensor;
    float ring[NW][RING][NO * UN * 32];         // X on its way: each lane its own values
    uint64_t mail_full[NW];
};

static_assert(2 * (sizeof(BatchSmem<6, 8>) + 1024) <= 228 * 1024, "two CTAs an SM");

template <int NT, class Smem>
__device__ void load_factors(Smem &sm, const BatchArgs &a, const TensorMeta &t, const TensorState &g) {
    for (int m = 0; m < 3; m++) {
        const float *src = a.U + t.uoff[m];
        const int I = t.dims[m];
        for (int e = threadIdx.x; e < (I + 3) / 4 * 4 * RS; e += NT) {
            const int i = e / RS, r = e - i * RS;
            sm.F[m][e] = (r < t.R && i < I) ? src[i + I * r] : 0.f;
        }
        for (int e = threadIdx.x; e < t.R * t.R; e += NT) sm.G[m][e] = g.G[m][e];
    }
}

typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 dup2(float x) {
    f32x2 v;
    asm("mov.b64 %0, {%1, %1};" : "=l"(v) : "f"(x));
    return v;
}
__device__ __forceinline__ void fma2(f32x2 &c, f32x2 a, f32x2 b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b));
}
__device__ __forceinline__ f32x2 pack2(float x, float y) {
    f32x2 v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(x), "f"(y));
    return v;
}
__device__ __forceinline__ float2 unpack2(f32x2 v) {
    float2 f;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
    return f;
}
// D (8 x 8) += A (8 x 4) B (4 x 8) in FP64: lane l holds A[l / 4][l % 4],
// B[l % 4][l / 4] and D[l / 4][2 (l % 4)], D[l / 4][2 (l % 4) + 1].
__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(c[0]), "+d"(c[1])
                 : "d"(a), "d"(b));
}

// Sum of v[0..RP) over the warp's 32 lanes by recursive halving (levels
// with shuffle offsets 16, 8, ... each keep half of the values a lane
// holds); afterwards lane l holds the total of rank l >> (5 - L).  RP is 4,
// 8 or 16.  Every lane of the warp must call it.
template <int RP>
__device__ __forceinline__ float lane_sum(float (&v)[RP], int lane) {
    constexpr int L = (RP == 16) ? 4 : (RP == 8) ? 3 : 2;
#pragma unroll
    for (int l = 0; l < L; l++) {
        const int off = 16 >> l;
        const int n = RP >> (l + 1);
        const bool up = (lane & off) != 0;
#pragma unroll
        for (int j = 0; j < n; j++) {
            const float send = up ? v[j] : v[j + n];
            const float keep = up ? v[j + n] : v[j];
            v[j] = keep + __shfl_xor_sync(0xffffffffu, send, off);
        }
    }
    float s = v[0];
#pragma unroll
    for (int off = 16 >> L; off >= 1; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
    return s;
}

// sm.M (row-major, RS) = this CTA's share of the MTTKRP of mode `mode`,
// factors in shared memory.  The lanes of a warp run along i, the tensor's
// contiguous index (32 rows per warp, ceil(I / 32) warps per row chunk), so
// every load of X is one coalesced 128-byte request and goes straight into
// registers; the cluster's CTAs, and the warps of a chunk within a CTA, split
// the outer index:
//   mode 0: M[i, :] = sum_k C[k, :] * sum_j X[i, j, k] B[j, :]
//           (outer k, inner j; the lane's own row, no cross-lane sum)
//   mode 1: M[j, :] = sum_i A[i, :] * sum_k X[i, j, k] C[k, :]
//   mode 2: M[k, :] = sum_i A[i, :] * sum_j X[i, j, k] B[j, :]
//           (outer j or k; the lanes' terms summed by lane_sum)
// X comes NO outer and UN inner indices at a time (zeros past the ends), by
// cp.async into a ring that only the copying lane reads: RING - 1 groups in
// flight without registers.  (Loaded to registers, the warps waited for DRAM
// most of the time: long scoreboard 4.2 stalls an issue.)  In mode 0 a warp's
// rows are summed over its range of k in k's order whatever the cluster: the
// CTAs take the range's groups of NO in turn and hand the sums on through
// distributed shared memory, so results do not depend on the launch shape.  Each broadcast factor row (RP registers, which cost the SM's shared
// memory a clock each) feeds NO RP multiply-adds (NO RP / 4 clocks), so NO =
// 4 balances the two; they are packed pairs of ranks (fma.rn.f32x2).  With
// NO = 2 the kernel was bound by the factor rows' loads.  Partials of the
// warps (mode 0: per outer range; modes 1, 2: per row chunk) are combined in
// a fixed order.  RP = the rank rounded up to 4, 8 or 16; the padding ranks
// of the factors are zero.
template <int RP, int NW, int CL>
__device__ void mttkrp_lanes(BatchSmem<NW, CL> &sm, cg::cluster_group &cl, const BatchArgs &a, const TensorMeta &t,
                             int mode, int rank, uint32_t &mails) {
    constexpr int H = RP / 2;
    const int I = t.dims[0], J = t.dims[1], K = t.dims[2];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int LI = (I + 31) >> 5;
    const int NG = NW / LI;
    const int ic = warp % LI, g = warp / LI;
    const int i = ic * 32 + lane;
    const bool valid = i < I;
    const int IJ = I * J;
    const int O = (mode == 1) ? J : K;        // outer index
    const int Nn = (mode == 1) ? K : J;       // inner index
    const int so = (mode == 1) ? I : IJ;      // X strides of the outer and inner index
    const int sn = (mode == 1) ? IJ : I;
    const float *Vf = (mode == 1) ? sm.F[2] : sm.F[1];  // the inner index's factor rows
    // this warp's outer range: of the CTA's share, or (mode 0) of the whole,
    // in groups of NO of which every CL-th is this CTA's
    const bool turns = CL > 1 && mode == 0;
    const int c0 = turns ? 0 : O * rank / CL, c1 = turns ? O : O * (rank + 1) / CL;
    const int begin = (g < NG) ? c0 + (c1 - c0) * g / NG : c1;
    const int o0 = begin + (turns ? rank * NO : 0);
    const int o1 = (g < NG) ? c0 + (c1 - c0) * (g + 1) / NG : c1;
    const int ostep = turns ? CL * NO : NO;
    f32x2 acc[H];
#pragma unroll
    for (int r = 0; r < H; r++) acc[r] = 0;
    // the copies run RING - 1 groups ahead: position (po, pn)
    int po = o0, pn = 0, fill = 0, slot = 0;
    const float *px = a.X + t.xoff + (valid ? i : 0) + (long)so * o0;
    const uint32_t ring = smem_u32(&sm.ring[warp][0][lane]);
    const int size = valid ? 4 : 0;  // lanes past I copy zeros (and read nothing)
    auto copy = [&]() {
        if (po < o1) {
            const uint32_t d = ring + (uint32_t)fill * (NO * UN * 128u);
            const int lo = o1 - po, ln = Nn - pn;
            const float *pk = px;
            if (lo >= NO && ln >= UN) {
#pragma unroll
                for (int k = 0; k < UN; k++, pk += sn) {
                    const float *pu = pk;
#pragma unroll
                    for (int u = 0; u < NO; u++, pu += so)
                        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d + (k * NO + u) * 128u),
                                     "l"(pu), "r"(size));
                }
            } else {
#pragma unroll
                for (int k = 0; k < UN; k++)
#pragma unroll
                    for (int u = 0; u < NO; u++) {
                        const bool ok = u < lo && k < ln;
                        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d + (k * NO + u) * 128u),
                                     "l"(ok ? pk + (u * so + k * sn) : a.X), "r"(ok ? size : 0));
                    }
            }
            pn += UN;
            px += UN * sn;
            if (pn >= Nn) {
                px += ostep * so - pn * sn;
                pn = 0;
                po += ostep;
            }
        }
        asm volatile("cp.async.commit_group;");
        fill = fill + 1 == RING ? 0 : fill + 1;
    };
#pragma unroll 1
    for (int k = 0; k < RING - 1; k++) copy();
    for (int o = o0; o < o1; o += ostep) {
        f32x2 tt[NO][H];
#pragma unroll
        for (int u = 0; u < NO; u++)
#pragma unroll
            for (int r = 0; r < H; r++) tt[u][r] = 0;
#pragma unroll 1
        for (int n = 0; n < Nn; n += UN) {
            copy();  // into the slot read a group ago
            asm volatile("cp.async.wait_group %0;" ::"n"(RING - 1) : "memory");
            const float *xs = &sm.ring[warp][slot][lane];
            slot = slot + 1 == RING ? 0 : slot + 1;
            float x[UN][NO];
#pragma unroll
            for (int k = 0; k < UN; k++)
#pragma unroll
                for (int u = 0; u < NO; u++) x[k][u] = xs[(k * NO + u) * 32];
#pragma unroll
            for (int k = 0; k < UN; k++) {
                const ulonglong2 *vr = reinterpret_cast<const ulonglong2 *>(Vf + (n + k) * RS);
                f32x2 xx[NO];
#pragma unroll
                for (int u = 0; u < NO; u++) xx[u] = dup2(x[k][u]);
#pragma unroll
                for (int r = 0; r < H; r += 2) {
                    const ulonglong2 v = vr[r / 2];
#pragma unroll
                    for (int u = 0; u < NO; u++) {
                        fma2(tt[u][r], xx[u], v.x);
                        fma2(tt[u][r + 1], xx[u], v.y);
                    }
                }
            }
        }
        if (mode == 0) {
            if (turns && o > begin) {
                // the sums so far, from the CTA that had the group before
                if (!ptx::mbar_wait_cluster(&sm.mail_full[warp], mails & 1)) *a.error = 1;
                mails++;
#pragma unroll
                for (int r = 0; r < H; r++) acc[r] = pack2(sm.mail[warp][2 * r][lane], sm.mail[warp][2 * r + 1][lane]);
            }
#pragma unroll
            for (int u = 0; u < NO; u++) {
                if (o + u >= o1) continue;  // warp-uniform
                const ulonglong2 *c = reinterpret_cast<const ulonglong2 *>(sm.F[2] + (o + u) * RS);
#pragma unroll
                for (int r = 0; r < H; r += 2) {
                    const ulonglong2 w = c[r / 2];
                    fma2(acc[r], tt[u][r], w.x);
                    fma2(acc[r + 1], tt[u][r + 1], w.y);
                }
            }
            if (turns && o + NO < o1) {
                const int next = rank + 1 == CL ? 0 : rank + 1;
                float *to = cl.map_shared_rank(&sm.mail[warp][0][lane], next);
#pragma unroll
                for (int r = 0; r < H; r++) {
                    const float2 v = unpack2(acc[r]);
                    to[64 * r] = v.x;
                    to[64 * r + 32] = v.y;
                }
                ptx::fence_cluster();  // every lane's writes, before lane 0's arrive
                __syncwarp();
                if (lane == 0) ptx::mbar_arrive_cluster(&sm.mail_full[warp], next);
            }
        } else {
            // the lane's terms A[i, :] * t, summed over the lanes (rows i)
            const float *ar = sm.F[0] + (valid ? i : 0) * RS;
#pragma unroll
            for (int u = 0; u < NO; u++) {
                if (o + u >= o1) continue;  // warp-uniform
                float f[RP];
#pragma unroll
                for (int r = 0; r < RP; r += 2) {
                    const float2 v = unpack2(tt[u][r / 2]);
                    f[r] = v.x * ar[r];
                    f[r + 1] = v.y * ar[r + 1];
                }
                const float s = lane_sum<RP>(f, lane);
                constexpr int SH = (RP == 16) ? 1 : (RP == 8) ? 2 : 3;
                if ((lane & ((1 << SH) - 1)) == 0) sm.Mp[ic][(o + u) * RS + (lane >> SH)] = s;
            }
        }
    }
    if (turns) {
        // the range's last CTA (the first, if the range is empty) leaves the
        // sums with every CTA: rows of group g at g LI 32
        const int groups = (o1 - begin + NO - 1) / NO;
        if (g < NG && rank == (groups > 0 ? (groups - 1) % CL : 0)) {
            for (int c = 0; c < CL; c++) {
                float4 *to = reinterpret_cast<float4 *>(cl.map_shared_rank(&sm.Mp[0][0], c) + ((g * LI + ic) * 32 + lane) * RS);
#pragma unroll
                for (int r = 0; r < RP; r += 4) {
                    const float2 p = unpack2(acc[r / 2]), q = unpack2(acc[r / 2 + 1]);
                    to[r / 4] = make_float4(p.x, p.y, q.x, q.y);
                }
            }
        }
        return;
    }
    if (mode == 0) {
        // the groups' rows added into M in group order, one group per
        // barrier (deterministic, one buffer)
        for (int gg = 0; gg < NG; gg++) {
            if (g == gg && valid) {
                float4 *m = reinterpret_cast<float4 *>(&sm.M[i * RS]);
#pragma unroll
                for (int r = 0; r < RP; r += 4) {
                    const float2 p = unpack2(acc[r / 2]), q = unpack2(acc[r / 2 + 1]);
                    float4 v = make_float4(p.x, p.y, q.x, q.y);
                    if (gg) {
                        const float4 w = m[r / 4];
                        v.x += w.x; v.y += w.y; v.z += w.z; v.w += w.w;
                    }
                    m[r / 4] = v;
                }
            }
            __syncthreads();
        }
        return;
    }
    __syncthreads();
    for (int e = c0 * RS + threadIdx.x; e < c1 * RS; e += NW * 32) {
        if ((e & (RS - 1)) >= RP) continue;  // padding ranks: never read
        float v = 0.f;
        for (int p = 0; p < LI; p++) v += sm.Mp[p][e];
        sm.M[e] = v;
    }
    __syncthreads();
}

// The whole M, from the cluster's CTAs, into sm.Mg: mode 0 adds the groups'
// sums, which every CTA holds, in group order; the others take each row from
// its CTA.
template <int NW, int CL>
__device__ void gather(BatchSmem<NW, CL> &sm, cg::cluster_group &cl, const TensorMeta &t, int mode) {
    const int Q = t.dims[mode], LI = (t.dims[0] + 31) >> 5, NG = NW / LI;
    static_assert(NW * 32 * RS <= MAXCHUNK * BMAXD * RS, "the groups' sums fit Mp");
    for (int e = threadIdx.x; e < Q * (RS / 4); e += NW * 32) {
        const int q = e / (RS / 4);
        float4 v;
        if (mode == 0) {
            const float4 *p = reinterpret_cast<const float4 *>(&sm.Mp[0][0]);
            v = p[e];
            for (int g = 1; g < NG; g++) {
                const float4 w = p[e + g * LI * 32 * (RS / 4)];
                v.x += w.x; v.y += w.y; v.z += w.z; v.w += w.w;
            }
        } else {
            int c = 0;  // rows Q c / CL .. are CTA c's
            while (q >= Q * (c + 1) / CL) c++;
            v = reinterpret_cast<const float4 *>(cl.map_shared_rank(sm.M, c))[e];
        }
        reinterpret_cast<float4 *>(sm.Mg)[e] = v;
    }
}

// sm.V = the inverse of the Hadamard of the Grams other than `mode`
// (Gauss-Jordan, FP64): a cell per thread in registers, the pivot's row and
// column published to double-buffered shared memory, one barrier a pivot; the
// next pivot's owner takes its reciprocal.  Rows and columns past R are zero.
// True when both attempts met a non-positive pivot (V is then not an inverse
// and the caller keeps the old factor).
template <int NW, int CL>
__device__ bool normal_inverse_small(BatchSmem<NW, CL> &sm, int R, int mode, int *fallbacks) {
    constexpr int NT = NW * 32, EP = (BMAXR * BMAXR + NT - 1) / NT;
    for (int attempt = 0; attempt < 2; attempt++) {
        double v[EP];
        if (threadIdx.x < R) {
            double d = 1.0;
            for (int m = 0; m < 3; m++)
                if (m != mode) d *= sm.G[m][threadIdx.x * (R + 1)];
            sm.diag[threadIdx.x] = d;
        }
        __syncthreads();
        double maxdiag = 0.0;
        for (int j = 0; j < R; j++) maxdiag = fmax(maxdiag, fabs(sm.diag[j]));
        auto publish = [&](int k) {  // row, column and reciprocal of pivot k
#pragma unroll
            for (int q = 0; q < EP; q++) {
                const int e = threadIdx.x + NT * q, i = e & (BMAXR - 1), j = e >> 4;
                if (EP * NT > BMAXR * BMAXR && e >= BMAXR * BMAXR) continue;
                if (i == k) sm.row[k & 1][j] = v[q];
                if (j == k) sm.col[k & 1][i] = v[q];
                if (i == k && j == k) sm.inv[k & 1] = 1.0 / v[q];
            }
        };
#pragma unroll
        for (int q = 0; q < EP; q++) {
            const int e = threadIdx.x + NT * q, i = e & (BMAXR - 1), j = e >> 4;
            v[q] = 0.0;
            if (i < R && j < R) {
                double x = 1.0;
                for (int m = 0; m < 3; m++)
                    if (m != mode) x *= sm.G[m][i + R * j];
                if (attempt == 1 && i == j) x += 1e-10 * maxdiag + 1e-300;
                v[q] = x;
            }
        }
        bool fail = false;
        publish(0);
        for (int k = 0; k < R; k++) {
            __syncthreads();
            const double *row = sm.row[k & 1], *col = sm.col[k & 1];
            const double piv = row[k], inv = sm.inv[k & 1];
            if (!(piv > 1e-14 * maxdiag) || !isfinite(piv)) {
                fail = true;  // the same on every thread
                break;
            }
#pragma unroll
            for (int q = 0; q < EP; q++) {
                const int e = threadIdx.x + NT * q, i = e & (BMAXR - 1), j = e >> 4;
                if (EP * NT > BMAXR * BMAXR && e >= BMAXR * BMAXR) continue;
                const double rk = (j == k ? 1.0 : row[j]) * inv;
                const double old = (j == k) ? 0.0 : v[q];
                v[q] = (i == k) ? rk : old - col[i] * rk;
            }
            if (k + 1 < R) publish(k + 1);
        }
        if (!fail) {
#pragma unroll
            for (int q = 0; q < EP; q++) {
                const int e = threadIdx.x + NT * q, i = e & (BMAXR - 1), j = e >> 4;
                if (EP * NT > BMAXR * BMAXR && e >= BMAXR * BMAXR) continue;
                sm.V[i * RS + j] = v[q];
            }
            __syncthreads();
            return false;
        }
        __syncthreads();
        if (threadIdx.x == 0 && attempt == 0 && fallbacks) atomicAdd(fallbacks, 1);
    }
    return true;
}

// Sum over the CTA in a fixed order, the same on every thread; `red` holds a
// slot per warp.
template <int NW>
__device__ double block_sum(double v, double *red) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    v = 0.0;
    for (int w = 0; w < NW; w++) v += red[w];
    return v;
}

// One ALS sweep of every tensor not yet converged: clusters of CL CTAs of NW
// warps pull tensors from the queue.  The CTAs of a cluster share a tensor's
// MTTKRPs (outer index ranges), gather the result through distributed shared
// memory and then run the R x R side and the factor update redundantly, so
// each holds all factors.  The update U = M V^-1 and the Gram U^T U run on
// the FP64 matrix instruction.
// Six warps a CTA: one, two or three 32-row chunks divide them, so none idles.
template <int NW, int CL>
__global__ void __launch_bounds__(NW * 32, 2) k_batch_sweep(BatchArgs a) {
    constexpr int NT = NW * 32;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    BatchSmem<NW, CL> &sm = *reinterpret_cast<BatchSmem<NW, CL> *>(smem_raw);
    cg::cluster_group cl = cg::this_cluster();
    const int rank = CL > 1 ? (int)cl.block_rank() : 0;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint32_t mails = 0;  // mails that this warp has waited for
    if (CL > 1 && threadIdx.x < NW) {
        ptx::mbar_init(&sm.mail_full[threadIdx.x], 1);
        ptx::fence_mbar_init();
    }
    // every CTA of the cluster runs, and its barriers are set up, before a peer
    // writes to its shared memory
    if (CL > 1) cl.sync();
    for (;;) {
        if (rank == 0 && threadIdx.x == 0) {
            const unsigned w = atomicAdd(a.queue, 1u);
            const int ti = (w < (unsigned)a.ntensors) ? a.order[w] : -1;
            if (CL > 1) {
                for (int c = 0; c < CL; c++) *cl.map_shared_rank(&sm.tensor, c) = ti;
            } else {
                sm.tensor = ti;
            }
        }
        if (CL > 1) cl.sync();
        else __syncthreads();
        const int ti = sm.tensor;
        if (CL > 1) cl.sync();  // everyone has read it (and is still there) before it is written again
        else __syncthreads();
        if (ti < 0) return;
        TensorMeta &t = a.meta[ti];
        if (t.done) continue;
        const int R = t.R;
        TensorState &ts = a.state[ti];
        load_factors<NT>(sm, a, t, ts);
        __syncthreads();
        double inner = 0.0;
        for (int mode = 0; mode < 3; mode++) {
            if (R <= 4) mttkrp_lanes<4, NW, CL>(sm, cl, a, t, mode, rank, mails);
            else if (R <= 8) mttkrp_lanes<8, NW, CL>(sm, cl, a, t, mode, rank, mails);
            else mttkrp_lanes<16, NW, CL>(sm, cl, a, t, mode, rank, mails);
            const float *M = sm.M;
            if (CL > 1) {
                cl.sync();  // every CTA's M is written
                gather(sm, cl, t, mode);
                M = sm.Mg;
                cl.sync();  // and read, before the next mode's
            }
            const bool keep = normal_inverse_small(sm, R, mode, rank == 0 ? a.fallbacks : nullptr);
            // U = M V^-1, 8 rows a warp at a time, into shared (row-major)
            // and, a CTA's share of the rows, global (column-major) memory;
            // singular twice: the old factor is kept
            const int Q = t.dims[mode];
            float *Ug = a.U + t.uoff[mode], *F = sm.F[mode];
            double part = 0.0;
            for (int q0 = 8 * warp; q0 < Q; q0 += 8 * NW) {
                const int q = q0 + (lane >> 2);
                double c[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
                if (!keep) {
#pragma unroll
                    for (int k = 0; k < BMAXR; k += 4) {
                        const int r = k + (lane & 3);
                        const double m = (q < Q && r < R) ? (double)M[q * RS + r] : 0.0;
#pragma unroll
                        for (int h = 0; h < 2; h++) dmma(c[h], m, sm.V[r * RS + 8 * h + (lane >> 2)]);
                    }
                }
#pragma unroll
                for (int h = 0; h < 2; h++)
#pragma unroll
                    for (int j = 0; j < 2; j++) {
                        const int col = 8 * h + 2 * (lane & 3) + j;
                        if (q >= Q || col >= R) continue;
                        float u = F[q * RS + col];
                        if (!keep) {
                            u = (float)c[h][j];
                            F[q * RS + col] = u;
                            if (CL == 1 || (q0 >> 3) % CL == rank) Ug[q + Q * col] = u;
                        }
                        if (mode == 2) part += (double)M[q * RS + col] * (double)u;
                    }
            }
            __syncthreads();
            // Gram of the new factor: a warp per 8 x 8 tile, the rows in
            // order (as one chain of fused multiply-adds)
            for (int tile = warp; tile < 4; tile += NW) {
                const int p0 = 8 * (tile & 1), q0 = 8 * (tile >> 1);
                double c[2] = {0.0, 0.0};
#pragma unroll 4
                for (int i0 = 0; i0 < Q; i0 += 4) {
                    const int i = i0 + (lane & 3);
                    const double f = i < Q ? (double)F[i * RS + p0 + (lane >> 2)] : 0.0;
                    const double h = i < Q ? (double)F[i * RS + q0 + (lane >> 2)] : 0.0;
                    dmma(c, f, h);
                }
#pragma unroll
                for (int j = 0; j < 2; j++) {
                    const int p = p0 + (lane >> 2), q = q0 + 2 * (lane & 3) + j;
                    if (p < R && q < R) sm.G[mode][p + R * q] = c[j];
                }
            }
            if (mode == 2) inner = block_sum<NW>(part, sm.red);
            __syncthreads();
        }
        double hat = 0.0;
        for (int e = threadIdx.x; e < R * R; e += NT) hat += sm.G[0][e] * sm.G[1][e] * sm.G[2][e];
        hat = block_sum<NW>(hat, sm.red + NW);
        if (rank == 0) {
            for (int m = 0; m < 3; m++)
                for (int e = threadIdx.x; e < R * R; e += NT) ts.G[m][e] = sm.G[m][e];
        }
        if (rank == 0 && threadIdx.x == 0) {
            double normx2 = 0.0;
            for (int k = 0; k < NORM_PARTS; k++) normx2 += ts.normp[k];
            const double res2 = normx2 - 2.0 * inner + hat;
            const double fit = 1.0 - sqrt(res2 > 0.0 ? res2 : 0.0) / sqrt(normx2);
            t.fit_prev = t.fit;
            t.fit = fit;
            t.sweeps += 1;
            if ((a.tol > 0 && t.sweeps >= 2 && fabs(t.fit - t.fit_prev) < a.tol) || t.sweeps >= a.max_sweeps ||
                (t.target > 0.0 && t.fit >= t.target)) {
                t.done = 1;
                atomicAdd(a.ndone, 1);
            }
        }
        __syncthreads();
    }
}

// Per-tensor ||X||^2 (NORM_PARTS CTAs a tensor, a part of X each) and the
// initial Grams (the first of them).
__global__ void __launch_bounds__(256) k_batch_setup(TensorMeta *meta, TensorState *state, int ntensors,
                                                     const float *X, const float *U) {
    __shared__ double red[8];
    for (int b = blockIdx.x; b < ntensors * NORM_PARTS; b += gridDim.x) {
        const int ti = b / NORM_PARTS, part = b % NORM_PARTS;
        TensorMeta &t = meta[ti];
        TensorState &ts = state[ti];
        const int n = t.dims[0] * t.dims[1] * t.dims[2];
        const int e1 = (int)((long)n * (part + 1) / NORM_PARTS);
        const float *x = X + t.xoff;
        double s0 = 0.0;
#pragma unroll 8
        for (int e = (int)((long)n * part / NORM_PARTS) + threadIdx.x; e < e1; e += 256) {
            const double v = __ldg(x + e);
            s0 = fma(v, v, s0);
        }
        const double tot = block_sum<8>(s0, red);
        if (threadIdx.x == 0) ts.normp[part] = tot;
        __syncthreads();
        if (part) continue;
        if (threadIdx.x == 0) {
            t.fit = 0.0;
            t.fit_prev = 0.0;
            t.sweeps = 0;
            t.done = 0;
        }
        const int R = t.R;
        for (int m = 0; m < 3; m++) {
            const float *F = U + t.uoff[m];
            const int I = t.dims[m];
            for (int e = threadIdx.x; e < R * R; e += 256) {
                const int p = e % R, q = e / R;
                double g = 0.0;
#pragma unroll 8
                for (int i = 0; i < I; i++) g = fma((double)F[i + I * p], (double)F[i + I * q], g);
                ts.G[m][e] = g;
            }
        }
    }
}

struct BatchState {
    TensorMeta *meta = nullptr;
    int *order = nullptr;
    unsigned *queue = nullptr;
    int *fallbacks = nullptr;
};

template <int NW, int CL>
int launch_sweep(const BatchArgs &a, int ctas_per_sm, cudaStream_t s) {
    static std::atomic<bool> attr[64];  // per device; zero-initialised
    using Smem = BatchSmem<NW, CL>;
    int dev = 0;
    CUD_CHECK(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64 || !attr[dev].load(std::memory_order_acquire)) {
        CUD_CHECK(cudaFuncSetAttribute(k_batch_sweep<NW, CL>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)sizeof(Smem)));
        // the whole unified L1 as shared memory: the CTAs per SM the tuner
        // asks for are then limited by shared memory, not by the carveout
        CUD_CHECK(cudaFuncSetAttribute(k_batch_sweep<NW, CL>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                       (int)cudaSharedmemCarveoutMaxShared));
        if (dev >= 0 && dev < 64) attr[dev].store(true, std::memory_order_release);
    }
    CUD_CHECK(cudaMemsetAsync(a.queue, 0, sizeof(unsigned), s));
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = CL;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg{};
    // no more clusters than tensors
    cfg.gridDim = dim3((unsigned)(std::min((long)kNumSMs * ctas_per_sm / CL, (long)a.ntensors) * CL));
    cfg.blockDim = dim3(NW * 32);
    cfg.dynamicSmemBytes = sizeof(Smem);
    cfg.stream = s;
    cfg.attrs = at;
    cfg.numAttrs = CL > 1 ? 1 : 0;
    CUD_CHECK(cudaLaunchKernelEx(&cfg, k_batch_sweep<NW, CL>, a));
    CUD_CHECK_LAUNCH("batched sweep");
    return CUD_OK;
}

// Launch shape: threads per CTA (warps x 32), CTAs per SM, CTAs per tensor.
struct BatchCfg {
    int threads, ctas, cluster;
};

int launch_cfg(const BatchArgs &a, const BatchCfg &c, cudaStream_t s) {
    if (c.cluster == 8) return launch_sweep<6, 8>(a, c.ctas, s);
    if (c.cluster == 4) return launch_sweep<6, 4>(a, c.ctas, s);
    if (c.cluster == 2) return launch_sweep<6, 2>(a, c.ctas, s);
    return launch_sweep<6, 1>(a, c.ctas, s);
}

// The launch shape of a batch that was not tuned: as many CTAs a tensor as
// the SMs are short of tensors (a CTA alone takes most of a millisecond for a
// sweep of the largest).  B200, ms a sweep with setup, dims 16 to 96, ranks 4
// to 16, clusters of 1 / 2 / 4 / 8: 64 tensors 0.52 / 0.31 / 0.24 / 0.23;
// 148: 0.51 / 0.41 / 0.31 / 0.45; 256: 0.87 / 0.49 / 0.48 / 0.72; 512: 1.13 /
// 0.86 / 1.06 / 1.55; 1024: 1.59 / 1.63 / 2.00 / -; 2048: 2.90 / 3.19 / 3.93.
// (Six warps a CTA of 2 x 8 register tiles without clusters: 0.92 ms at 64,
// 1.28 at 256, 2.0 at 1024, 3.2 at 2048.)
// Tensors of up to 40000 elements have too little to share: their sweeps are
// barriers, which a cluster's make longer (B200, ms for 20 sweeps, clusters of 1 /
// 2 / 4 / 8: 60 tensors of dims 10 to 20 0.98 / 1.07 / 1.15 / 1.64, 200 1.19 / 1.76 /
// 2.32 / 4.24; dims 16 to 32, 100 tensors 1.42 / 1.41 / 2.06 / 3.17, 300 1.86 / 2.76 /
// 4.28 / 7.75; dims 24 to 48, 100 tensors 2.93 / 2.55 / 2.74 / 4.33).
BatchCfg default_cfg(int n, const int *dims) {
    int largest = 0;
    for (int t = 0; t < n; t++) largest = std::max(largest, dims[3 * t] * dims[3 * t + 1] * dims[3 * t + 2]);
    if (largest <= 40000) return {192, 2, 1};
    if (n <= kNumSMs / 2) return {192, 2, 8};
    if (n <= 2 * kNumSMs) return {192, 2, 4};
    if (n <= 6 * kNumSMs) return {192, 2, 2};
    return {192, 2, 1};
}

// Autotuner cache: shape class -> launch shape
std::mutex g_tune_mu;
std::map<long, BatchCfg> g_tune;

long shape_class(int n, const int *dims, const int *ranks) {
    // bucket the mean element count and mean rank; plus the batch size order
    double e = 0.0, r = 0.0;
    for (int t = 0; t < n; t++) {
        e += (double)dims[3 * t] * dims[3 * t + 1] * dims[3 * t + 2];
        r += ranks[t];
    }
    e /= std::max(1, n);
    r /= std::max(1, n);
    long eb = (long)log2(std::max(1.0, e)), rb = (long)r / 4, nb = (long)log2(std::max(1, n));
    return eb * 10000 + rb * 100 + nb;
}

}  // namespace

}  // namespace cud

using namespace cud;

namespace {

int batched_impl(int ntensors, const long *dims, const long *ranks, const float *X, const long *x_offsets, float *U,
                 const long *u_offsets, const cud_cp_options *opt_in, const double *targets, double *fits,
                 int *sweeps, int *kernel_launches, void *stream) {
    if (ntensors <= 0 || !dims || !ranks || !X || !x_offsets || !U || !u_offsets)
        return set_status(CUD_ERR_INVALID_ARGUMENT);
    cud_cp_options opt;
    cud_cp_default_options(&opt);
    if (opt_in) opt = *opt_in;
    if (opt.max_sweeps < 1) return set_status(CUD_ERR_INVALID_ARGUMENT);
    cudaStream_t s = as_stream(stream);
    // the tensors' descriptions and the processing order, uploaded as one
    // block: [meta][order]; the device's own state follows it in the scratch
    const size_t mbytes = (sizeof(TensorMeta) * ntensors + sizeof(int) * ntensors + 255) & ~size_t(255);
    std::vector<double> host((mbytes + 7) / 8);
    TensorMeta *hm = reinterpret_cast<TensorMeta *>(host.data());
    int *order = reinterpret_cast<int *>(hm + ntensors);
    std::vector<int> hd(3 * ntensors), hr(ntensors);
    std::vector<std::pair<double, int>> work(ntensors);
    for (int t = 0; t < ntensors; t++) {
        TensorMeta &m = hm[t];
        memset(&m, 0, sizeof(TensorMeta));
        for (int k = 0; k < 3; k++) {
            if (dims[3 * t + k] < 1 || dims[3 * t + k] > BMAXD) return set_status(CUD_ERR_UNSUPPORTED);
            m.dims[k] = (int)dims[3 * t + k];
            m.uoff[k] = u_offsets[3 * t + k];
            hd[3 * t + k] = m.dims[k];
        }
        if (ranks[t] < 1 || ranks[t] > BMAXR) return set_status(CUD_ERR_UNSUPPORTED);
        m.R = (int)ranks[t];
        hr[t] = m.R;
        m.xoff = x_offsets[t];
        m.target = targets ? targets[t] : 0.0;
        work[t] = {-(double)m.dims[0] * m.dims[1] * m.dims[2] * m.R, t};
    }
    std::sort(work.begin(), work.end());
    for (int t = 0; t < ntensors; t++) order[t] = work[t].second;

    int st;
    char *w = (char *)scratch(kSlotTmp1, mbytes + 256 + sizeof(TensorState) * ntensors, &st);
    if (!w) return set_status(st);
    BatchArgs a;
    a.meta = reinterpret_cast<TensorMeta *>(w);
    a.order = reinterpret_cast<int *>(a.meta + ntensors);
    a.queue = reinterpret_cast<unsigned *>(w + mbytes);
    a.fallbacks = reinterpret_cast<int *>(a.queue + 16);
    a.ndone = reinterpret_cast<int *>(a.queue + 32);
    a.error = a.ndone + 1;
    a.state = reinterpret_cast<TensorState *>(w + mbytes + 256);
    a.ntensors = ntensors;
    a.X = X;
    a.U = U;
    a.max_sweeps = opt.max_sweeps;
    a.tol = opt.tol;
    CUD_CHECK(cudaMemcpyAsync(w, hm, mbytes, cudaMemcpyHostToDevice, s));
    CUD_CHECK(cudaMemsetAsync(a.queue, 0, 256, s));
    k_batch_setup<<<std::min((long)ntensors * NORM_PARTS, kNumSMs * 64L), 256, 0, s>>>(a.meta, a.state, ntensors, X, U);
    CUD_CHECK_LAUNCH("batched setup");

    // launch shape: the autotuner's (CTAs a tensor), where this class was tuned
    long key = shape_class(ntensors, hd.data(), hr.data());
    BatchCfg cfg = default_cfg(ntensors, hd.data());
    {
        std::lock_guard<std::mutex> lk(g_tune_mu);
        auto it = g_tune.find(key);
        if (it != g_tune.end()) cfg = it->second;
    }
    // sweeps: graph of `per` sweeps replayed; the done-count read back between
    const int per = std::max(1, std::min(opt.check_every > 1 ? opt.check_every : 5, opt.max_sweeps));
    // a graph that would be replayed once is not built (capture, instantiation
    // and a stream of its own took 0.4 ms of a call)
    const bool use_graph = opt.use_graph && opt.max_sweeps > per;
    cudaStream_t cs = s;
    bool own = false;
    if (use_graph && (s == nullptr || s == cudaStreamLegacy || s == cudaStreamPerThread)) {
        CUD_CHECK(cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking));
        own = true;
        CUD_CHECK(cudaStreamSynchronize(s));
    }
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    st = CUD_OK;
    if (use_graph) {
        if (cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal) != cudaSuccess) st = CUD_ERR_CUDA;
        for (int i = 0; i < per && st == CUD_OK; i++) st = launch_cfg(a, cfg, cs);
        cudaError_t e = cudaStreamEndCapture(cs, &graph);
        if (st == CUD_OK && e != cudaSuccess) st = cuda_status(e, "batched capture");
        if (st == CUD_OK) {
            e = cudaGraphInstantiate(&exec, graph, 0);
            if (e != cudaSuccess) st = cuda_status(e, "batched instantiate");
        }
    }
    int launched = 0, done_sweeps = 0;
    double *hs = pinned_scalars();  // slot 63: the converged count
    int *ndone_h = hs ? reinterpret_cast<int *>(hs + 63) : nullptr;
    while (st == CUD_OK && done_sweeps < opt.max_sweeps) {
        if (exec) {
            if (cudaGraphLaunch(exec, cs) != cudaSuccess) { st = CUD_ERR_CUDA; break; }
        } else {
            for (int i = 0; i < per && st == CUD_OK; i++) st = launch_cfg(a, cfg, cs);
        }
        launched += per;
        done_sweeps += per;
        // convergence check: the count of converged tensors, and the error flag
        if (!ndone_h || cudaMemcpyAsync(ndone_h, a.ndone, 2 * sizeof(int), cudaMemcpyDeviceToHost, cs) != cudaSuccess ||
            cudaStreamSynchronize(cs) != cudaSuccess) { st = CUD_ERR_CUDA; break; }
        if (ndone_h[1]) { st = CUD_ERR_DEVICE_TIMEOUT; break; }
        if (ndone_h[0] >= ntensors) break;
    }
    if (exec) cudaGraphExecDestroy(exec);
    if (graph) cudaGraphDestroy(graph);
    std::vector<TensorMeta> out;
    if (st == CUD_OK && (fits || sweeps)) {
        out.resize(ntensors);
        if (cudaMemcpyAsync(out.data(), a.meta, sizeof(TensorMeta) * ntensors, cudaMemcpyDeviceToHost, cs) != cudaSuccess ||
            cudaStreamSynchronize(cs) != cudaSuccess)
            st = CUD_ERR_CUDA;
    }
    if (st == CUD_OK) {
        for (int t = 0; t < ntensors; t++) {
            if (fits) fits[t] = out[t].fit;
            if (sweeps) sweeps[t] = out[t].sweeps;
        }
        if (kernel_launches) *kernel_launches = launched;
    }
    if (own) {
        cudaStreamSynchronize(cs);
        cudaStreamDestroy(cs);
    }
    return set_status(st);
}

}  // namespace

extern "C" int cud_cp_als_batched(int ntensors, const long *dims, const long *ranks, const float *X,
                                  const long *x_offsets, float *U, const long *u_offsets,
                                  const cud_cp_options *opt_in, double *fits, int *sweeps,
                                  int *kernel_launches, void *stream) {
    return batched_impl(ntensors, dims, ranks, X, x_offsets, U, u_offsets, opt_in, nullptr, fits, sweeps,
                        kernel_launches, stream);
}

extern "C" int cud_cp_als_batched_target(int ntensors, const long *dims, const long *ranks, const float *X,
                                         const long *x_offsets, float *U, const long *u_offsets,
                                         const cud_cp_options *opt_in, const double *target_fits, double *fits,
                                         int *sweeps, int *kernel_launches, void *stream) {
    return batched_impl(ntensors, dims, ranks, X, x_offsets, U, u_offsets, opt_in, target_fits, fits, sweeps,
                        kernel_launches, stream);
}

extern "C" int cud_cp_batched_tune(int ntensors, const long *dims, const long *ranks, const float *X,
                                   const long *x_offsets, float *U_scratch, const long *u_offsets,
                                   int *threads, int *ctas_per_sm, void *stream) {
    if (ntensors <= 0 || !dims || !ranks) return set_status(CUD_ERR_INVALID_ARGUMENT);
    std::vector<int> hd(3 * ntensors), hr(ntensors);
    for (int t = 0; t < ntensors; t++) {
        for (int k = 0; k < 3; k++) hd[3 * t + k] = (int)dims[3 * t + k];
        hr[t] = (int)ranks[t];
    }
    long key = shape_class(ntensors, hd.data(), hr.data());
    // (threads, CTAs per SM, CTAs a tensor): two CTAs of 168 registers a thread
    // and ~100 KB of shared memory fill an SM, so the first two, which the
    // caller is told, are the same throughout
    const std::vector<BatchCfg> cand = {{192, 2, 1}, {192, 2, 2}, {192, 2, 4}, {192, 2, 8}};
    BatchCfg bestc = cand[0];
    cudaStream_t s = as_stream(stream);
    cudaEvent_t e0, e1;
    CUD_CHECK(cudaEventCreate(&e0));
    CUD_CHECK(cudaEventCreate(&e1));
    // an untimed round (first launches load each width's kernel), then two
    // timed rounds in turn; a candidate's time is its best of the two (one
    // timing a candidate picked a slower shape on some runs)
    std::vector<float> best_ms(cand.size(), 1e30f);
    for (int round = 0; round < 3; round++) {
        for (size_t ci = 0; ci < cand.size(); ci++) {
            {
                std::lock_guard<std::mutex> lk(g_tune_mu);
                g_tune[key] = cand[ci];
            }
            cud_cp_options opt;
            cud_cp_default_options(&opt);
            opt.max_sweeps = round == 0 ? 1 : 2;
            opt.tol = 0.0;
            opt.use_graph = 0;
            opt.check_every = opt.max_sweeps;
            cudaEventRecord(e0, s);
            int st = cud_cp_als_batched(ntensors, dims, ranks, X, x_offsets, U_scratch, u_offsets, &opt,
                                        nullptr, nullptr, nullptr, stream);
            cudaEventRecord(e1, s);
            cudaEventSynchronize(e1);
            if (st) { cudaEventDestroy(e0); cudaEventDestroy(e1); return set_status(st); }
            float ms = 0.f;
            cudaEventElapsedTime(&ms, e0, e1);
            if (round > 0 && ms < best_ms[ci]) best_ms[ci] = ms;
        }
    }
    float best = 1e30f;
    for (size_t ci = 0; ci < cand.size(); ci++)
        if (best_ms[ci] < best) {
            best = best_ms[ci];
            bestc = cand[ci];
        }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    {
        std::lock_guard<std::mutex> lk(g_tune_mu);
        g_tune[key] = bestc;
    }
    if (threads) *threads = bestc.threads;
    if (ctas_per_sm) *ctas_per_sm = bestc.ctas;
    return set_status(CUD_OK);
}
