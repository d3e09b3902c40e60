// MTTKRP of small tensors in one launch (plain FP32, CUD_PREC_FP32 and
// CUD_PREC_DEFAULT), any order, extents and alignment:
//     M[q, r] = sum_kappa X(q, kappa) KR(kappa, r).
//
// Bound: latency.  The kernels for large tensors pay for a wave of set-up
// (TMEM, rings, a pack or a cleared flag before, a split reduce behind): 48 x
// 40 x 36 at R = 8 took three launches and 13 us of GPU time a mode for 70
// thousand multiply-adds.  Here a cluster of up to 8 CTAs owns 4 rows q x 8
// ranks: a thread takes every (CTAs x 256)-th kappa, forms its 8 Khatri-Rao
// values from the factors (lanes along kappa: the fastest factor's reads are
// coalesced) and adds 4 x 8 products; the 32 sums are halved across a warp's
// lanes to one a lane, added over the warps, then over the cluster through
// distributed shared memory, in a fixed order -- no partials in memory, no
// second kernel.
#include <cooperative_groups.h>

#include "kernels.cuh"
#include "tc_ptx.cuh"

namespace cg = cooperative_groups;

namespace cud {

namespace {

constexpr int ST = 256, SQ = 4, SR = 8;

struct SmallArgs {
    const float *X;
    unsigned P, Q, K;  // K: contraction length
    int R, nf, vec;    // vec: 16-byte loads of X (mode 0)
    const float *U[kMaxOrder];
    unsigned rows[kMaxOrder];
    unsigned qtiles;
    float *out;
};

// kQ 0: mode 0 (q contiguous, kappa = s); 1: the others (kappa = p + P s).
template <int kQ>
__global__ void __launch_bounds__(ST) k_mttkrp_small(const __grid_constant__ SmallArgs a) {
    __shared__ float red[ST / 32][32];
    __shared__ double sums[32];
    cg::cluster_group cl = cg::this_cluster();
    const unsigned rank = cl.block_rank(), ncta = cl.num_blocks();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned tile = blockIdx.x / ncta;
    const unsigned q0 = tile * SQ;
    const int r0 = blockIdx.y * SR;
    // launched programmatically: nothing is read before the kernel ahead is done
    ptx::griddep_wait();
    ptx::griddep_launch();
    float acc[SQ * SR];
#pragma unroll
    for (int i = 0; i < SQ * SR; i++) acc[i] = 0.f;
#pragma unroll 2
    for (unsigned k = rank * ST + threadIdx.x; k < a.K; k += ncta * ST) {
        float x[SQ];
        if (kQ == 0) {
            const float *p = a.X + q0 + (size_t)a.Q * k;
            if (a.vec) {
                const float4 v = __ldg(reinterpret_cast<const float4 *>(p));
                x[0] = v.x; x[1] = v.y; x[2] = v.z; x[3] = v.w;
            } else {
#pragma unroll
                for (int i = 0; i < SQ; i++) x[i] = __ldg(p + min((unsigned)i, a.Q - 1 - q0));
            }
        } else {
            const unsigned s = k / a.P;
            const float *p = a.X + (k - s * a.P) + (size_t)a.P * (q0 + (size_t)a.Q * s);
#pragma unroll
            for (int i = 0; i < SQ; i++) x[i] = __ldg(p + (size_t)a.P * min((unsigned)i, a.Q - 1 - q0));
        }
        float v[SR];
        unsigned lin = k;
        for (int f = 0; f < a.nf; f++) {
            const unsigned rows = a.rows[f], next = f + 1 < a.nf ? lin / rows : 0;
            const float *u = a.U[f] + (lin - next * rows);
            lin = next;
#pragma unroll
            for (int j = 0; j < SR; j++) {
                const float w = __ldg(u + (size_t)min(r0 + j, a.R - 1) * rows);
                v[j] = f == 0 ? w : v[j] * w;
            }
        }
#pragma unroll
        for (int i = 0; i < SQ; i++)
#pragma unroll
            for (int j = 0; j < SR; j++) acc[i * SR + j] = fmaf(x[i], v[j], acc[i * SR + j]);
    }
    // recursive halving: lane l ends with the warp's sum of value l
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int j = 0; j < o; j++) {
            const float send = up ? acc[j] : acc[j + o], keep = up ? acc[j + o] : acc[j];
            acc[j] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
    red[warp][lane] = acc[0];
    __syncthreads();
    if (warp == 0) {
        double s = 0.0;
#pragma unroll
        for (int w = 0; w < ST / 32; w++) s += (double)red[w][lane];
        sums[lane] = s;
    }
    if (ncta > 1) cl.sync();
    else __syncthreads();
    if (rank == 0 && warp == 0) {
        double s = 0.0;
        for (unsigned c = 0; c < ncta; c++) s += *cl.map_shared_rank(&sums[lane], c);
        const unsigned q = q0 + lane / SR;
        const int r = r0 + lane % SR;
        if (q < a.Q && r < a.R) a.out[q + (size_t)a.Q * r] = (float)s;
    }
    if (ncta > 1) cl.sync();  // the sums are read before their CTA leaves
}

}  // namespace

// Where one launch beats two or three (B200, us a mode through the Python
// mirror, this kernel / the FFMA kernel and its reduce / tensor cores): 48 x 40
// x 36 R = 8 10.5 / 13.2 / 15.3, 64^3 R = 32 10.7 / 13.5 / 15.9, 24 x 48 x 512
// R = 16 10.5 / 13.3 / 24; 96^3 R = 16 (1.4e7) 13.8 / 13.7 / 16.3, R = 32 21.0 /
// 13.6 / 16.3; a long contraction over few rows, 20 x 20 x 2000 R = 8, 14.8 /
// 13.5 / 21.2.
bool mttkrp_small_applies(int order, const long *dims, int mode, long R) {
    double work = (double)R, K = 1.0;
    for (int m = 0; m < order; m++) {
        work *= (double)dims[m];
        if (m != mode) K *= (double)dims[m];
    }
    // A CTA computes whole tiles of 4 rows x 8 ranks, and all of its 256 threads
    // sum them, however short the contraction (us, this kernel / the one that
    // had the call before it: 10 x 1000 x 1000 R = 1 mode 2 44 / 33, 2 x 6 x 5000 R = 64
    // mode 2, 10000 tiles over K = 12, 53 / 8, 9 x 5 x 2291 R = 33 mode 2, 2865 tiles, 18 /
    // 8; 12 x 18 x 932 R = 34 mode 2, 1165 tiles, 9.5 / 9.8).
    const double tiles = (double)((dims[mode] + SQ - 1) / SQ) * (double)((R + SR - 1) / SR);
    return R <= 64 && work <= 1e7 && K <= 16384.0 && tiles <= 8.0 * kNumSMs && tiles * (SQ * SR) * K <= 2e7;
}

int mttkrp_small(const float *X, int order, const long *dims, const float *const *U, int mode, long R, float *out,
                 cudaStream_t s) {
    const ModeView v = mode_view(order, dims, mode);
    SmallArgs a;
    a.X = X;
    a.P = (unsigned)v.P;
    a.Q = (unsigned)v.Q;
    a.K = (unsigned)(v.P * v.S);
    a.R = (int)R;
    a.vec = mode == 0 && v.Q % 4 == 0 && (reinterpret_cast<uintptr_t>(X) & 15) == 0;
    a.nf = 0;
    for (int m = 0; m < order; m++) {
        if (m == mode) continue;
        a.U[a.nf] = U[m];
        a.rows[a.nf++] = (unsigned)dims[m];
    }
    a.qtiles = (a.Q + SQ - 1) / SQ;
    a.out = out;
    const unsigned rtiles = (unsigned)((R + SR - 1) / SR);
    // CTAs a cluster: while they fill two waves of the SMs and have a kappa a
    // thread
    unsigned cl = 1;
    while (cl < 8 && (long)a.qtiles * rtiles * cl * 2 <= 4L * kNumSMs && a.K >= cl * 2 * ST) cl *= 2;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = cl;
    at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(a.qtiles * cl, rtiles);
    cfg.blockDim = dim3(ST);
    cfg.stream = s;
    cfg.attrs = at;
    cfg.numAttrs = cl > 1 ? 2 : 1;
    const int pk = prof_begin(s);
    if (mode == 0) CUD_CHECK(cudaLaunchKernelEx(&cfg, k_mttkrp_small<0>, a));
    else CUD_CHECK(cudaLaunchKernelEx(&cfg, k_mttkrp_small<1>, a));
    prof_end(pk, s);
    CUD_CHECK_LAUNCH("mttkrp_small");
    return CUD_OK;
}

}  // namespace cud
