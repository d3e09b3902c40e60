// MTTKRP on FP64 data (the FP64 CP-ALS), any order and extents, in the
// tensor's native layout, with no Khatri-Rao matrix:
//     M[q, r] = sum_kappa X(q, kappa) KR(kappa, r),
// kappa = s where P = 1 (mode 0; q contiguous in memory), kappa = p + P s for
// the other modes (p contiguous).
//
// Bound: HBM up to rank ~20 (2 R flops for 8 bytes against 37 TFLOP/s and
// 6.5 TB/s), FP64 arithmetic above.  The multiply-adds are the FP64 matrix
// instruction (mma.m8n8k4, fused multiply-adds as on the FP64 lanes and at
// their rate): with 32 x 8 NT outputs a warp it needs 4 + NT loads of one
// double a lane for 4 NT instructions, where scalar FMAs would be bound by
// the shared memory that feeds them (128 bytes a clock and SM).
//   * A CTA (4 warps) owns 128 rows q x 8 NT ranks and a range of stages of
//     up to 16 kappa that never leave a row block of the fastest factor U0:
//     U0's rows are copied as they are and a lane scales the ranks it reads by
//     the block's constant row (the product of the other factors' rows), kept
//     in registers.
//   * X and U0 arrive by cp.async in a three-deep ring: 16-byte copies of X
//     where its contiguous extent is even and X 16-byte aligned, else 8-byte
//     ones.  The rings' row strides put a fragment's 16 lanes of a wavefront
//     on distinct banks.
// Partials [split][r][q] are summed in a fixed order by k_sum_splits_f64.
// B200, 160 x 144 x 120 R = 16, three modes: 299 -> 42 us (64 x 64
// tiles of scalar FMAs with the Khatri-Rao rows formed per element before).
#include <atomic>
#include <type_traits>

#include "kernels.cuh"
#include "tc_ptx.cuh"

namespace cud {

namespace {

constexpr int DQ = 128, DK = 16, DT = 128, DST = 3;
constexpr int LDQ = DQ + 4;  // [kappa][q] tile: 4 kappas x 4 rows on distinct banks
constexpr int LDK = DK + 4;  // [q][kappa] tile: the same

struct F64Args {
    const double *X;
    long P, Q, S;
    int R;
    int nf;             // factors of the KR rows, fastest first
    const double *U[kMaxOrder];
    long rows[kMaxOrder];
    long bsteps;        // stages per row block of U0
    long pblocks;       // row blocks in P (modes other than 0)
    long qtiles;
    long steps, chunk;  // total stages, stages per split
    double *part;       // [split][R][Q]
};

template <int kBytes>
__device__ __forceinline__ void copy_async(uint32_t dst, const double *src) {
    if constexpr (kBytes == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src));
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src));
}
__device__ __forceinline__ void zero8(uint32_t dst) { asm volatile("st.shared.f64 [%0], %1;" ::"r"(dst), "d"(0.0)); }

__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(c[0]), "+d"(c[1])
                 : "d"(a), "d"(b));
}

template <int kQ, int NT>
struct DTile {
    static constexpr int AF = kQ == 0 ? DK * LDQ : DQ * LDK;  // doubles of an X tile
    static constexpr int LDB = 8 * NT + 4;
    static constexpr int BF = DK * LDB;
    static constexpr int MINB = NT <= 4 ? 3 : 2;
    static constexpr size_t kSmem = 8 * (size_t)DST * (AF + BF);
};

// kQ 0: q contiguous in memory (mode 0), tile [kappa][q]; 1: the contraction
// index, tile [q][kappa].  kVec: 16-byte copies of X.  kAny: factors of 2^30
// elements and more (64-bit indices).
template <int kQ, bool kVec, bool kAny, int NT>
__global__ void __launch_bounds__(DT, DTile<kQ, NT>::MINB) k_mttkrp_f64(const __grid_constant__ F64Args a) {
    using T = DTile<kQ, NT>;
    using I = std::conditional_t<kAny, unsigned long long, unsigned>;  // factor indices
    constexpr int AF = T::AF, BF = T::BF, MT = 4;
    extern __shared__ __align__(16) double dsm[];
    double *Xring = dsm, *Bring = dsm + DST * AF;

    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const long q0 = (blockIdx.x % a.qtiles) * DQ;
    const long z = blockIdx.x / a.qtiles;
    const int r0 = blockIdx.y * (8 * NT);
    const long sbeg = z * a.chunk;
    const long send = min(a.steps, sbeg + a.chunk);
    if (sbeg >= send) return;  // (no such CTA in the plan's grid)
    const int nst = (int)(send - sbeg);
    const long rows0 = a.rows[0];
    const I bsteps = (I)a.bsteps;
    const int tail = (int)(rows0 - (a.bsteps - 1) * DK);  // kappas of a block's last stage

    // ---- copies.  The stage that is copied next: block lb, step lj in it.
    const I lb = (I)sbeg / bsteps;
    I lj = (I)sbeg - lb * bsteps;
    long lp = 0;  // kQ 1: position in the contiguous extent P
    const double *src;
    // each thread copies at kappa = ck (mode 0: + i STEP) and row cq (else: + i STEP)
    constexpr int W = kVec ? 2 : 1;         // doubles per copy
    constexpr int NC = DQ * DK / W / DT;    // copies per thread and stage
    const int cq = kQ == 0 ? W * t % DQ : W * t / DK;
    const int ck = kQ == 0 ? W * t / DQ : W * t % DK;
    constexpr int STEP = kQ == 0 ? W * DT / DQ : W * DT / DK;
    if (kQ == 0) {
        src = a.X + q0 + cq + a.Q * ((long)lb * rows0 + (long)lj * DK + ck);
    } else {
        const I pb = (I)a.pblocks, s = lb / pb;  // blocks per s
        lp = (long)(lb - s * pb) * rows0 + (long)lj * DK;
        src = a.X + lp + ck + a.P * (q0 + cq + a.Q * (long)s);
    }
    const long cstride = STEP * (kQ == 0 ? a.Q : a.P);
    // copies of this thread inside the tensor (mode 0: all or none); the
    // tile's other rows q keep what the memory holds and are not written out
    const long qleft = a.Q - q0 - cq;
    const int nrow = qleft <= 0 ? 0 : kQ == 0 ? NC : (int)min((long)NC, (qleft + STEP - 1) / STEP);
    const uint32_t xdst = smem_u32(Xring) + 8u * (kQ == 0 ? ck * LDQ + cq : cq * LDK + ck);
    constexpr uint32_t dstride = 8u * STEP * (kQ == 0 ? LDQ : LDK);
    // U0: 16 lanes = rows (those past the block's end are left as they are),
    // half-warps take the ranks in turn; ranks past R
    // repeat rank R - 1 (their results are not written)
    const int bk = t % DK, bc = t / DK;
    const uint32_t bdst = smem_u32(Bring) + 8u * (bk * T::LDB + bc);
    auto load = [&](int slot) {
        const int kc = lj == bsteps - 1 ? tail : DK;
        const double *p = src;
        const uint32_t d = xdst + (uint32_t)slot * (8u * AF);
        const int nr = kQ == 0 ? (nrow == 0 ? 0 : max(0, (kc - ck + STEP - 1) / STEP)) : ck < kc ? nrow : 0;
        if (nr == NC) {
#pragma unroll
            for (int i = 0; i < NC; i++, p += cstride) copy_async<8 * W>(d + dstride * i, p);
        } else {
#pragma unroll 2
            for (int i = 0; i < nr; i++, p += cstride) copy_async<8 * W>(d + dstride * i, p);
            // past the block's end: zeros (kappas are multiplied 4 at a time)
            const int zf = kQ == 0 ? max(0, (kc - ck + STEP - 1) / STEP) : ck < kc ? NC : 0;
#pragma unroll 2
            for (int i = zf; i < NC; i++) {
                zero8(d + dstride * i);
                if (kVec) zero8(d + dstride * i + 8);
            }
        }
        const uint32_t bd = bdst + (uint32_t)slot * (8u * BF);
        const I row = lj * DK + bk;
#pragma unroll
        for (int i = 0; i < NT; i++) {
            const I r = (I)min(r0 + bc + 8 * i, a.R - 1);
            if (bk < kc) copy_async<8>(bd + 64u * i, a.U[0] + (row + r * (I)rows0));
        }
        // the next stage
        lj++;
        src += kQ == 0 ? a.Q * kc : (long)kc;
        if (kQ != 0) {
            lp += kc;
            if (lp == a.P) {
                lp = 0;
                src += a.P * a.Q - a.P;
            }
        }
        if (lj == bsteps) lj = 0;
    };

    // ---- the constant row of the block that is multiplied, at this lane's
    // rank of each 8-rank group
    double cc[NT];
    auto const_row = [&](I block) {
#pragma unroll
        for (int j = 0; j < NT; j++) cc[j] = 1.0;
        I lin = block;
        for (int f = 1; f < a.nf; f++) {
            const I rows = (I)a.rows[f], next = lin / rows, d = lin - next * rows;
            lin = next;
#pragma unroll
            for (int j = 0; j < NT; j++)
                cc[j] *= __ldg(a.U[f] + (d + (I)min(r0 + 8 * j + (lane >> 2), a.R - 1) * rows));
        }
    };

    double acc[MT][NT][2];
#pragma unroll
    for (int i = 0; i < MT; i++)
#pragma unroll
        for (int j = 0; j < NT; j++) acc[i][j][0] = acc[i][j][1] = 0.0;

    // ---- the stages; the copies' lead-in is the loop's first rounds
    I cb = lb, cj = lj;  // block and step of the stage that is multiplied
    int slot = 0, fill = 0;
#pragma unroll 1
    for (int i = -(DST - 1); i < nst; i++) {
        if (i >= 0) {
            // this thread's copies of the stage have landed; after the barrier
            // everyone's have, and the slot read a stage ago is free
            asm volatile("cp.async.wait_group %0;" ::"n"(DST - 2));
            __syncthreads();
        }
        if (i + DST - 1 < nst) load(fill);
        asm volatile("cp.async.commit_group;");
        fill = fill + 1 == DST ? 0 : fill + 1;
        if (i < 0) continue;
        if (i == 0 || cj == 0) const_row(cb);
        const int kc = cj == bsteps - 1 ? tail : DK;
        // fragments: A row lane / 4, kappa lane % 4; B kappa lane % 4, rank lane / 4
        const int fr = 32 * warp + (lane >> 2), fk = lane & 3;
        const double *A = Xring + slot * AF + (kQ == 0 ? fk * LDQ + fr : fr * LDK + fk);
        const double *B = Bring + slot * BF + fk * T::LDB + (lane >> 2);
        // `in`: this lane's kappa is in the block.  Past its end X is zero, and
        // the Khatri-Rao value is too, not a product that an infinite constant
        // row would turn into NaN.  (B200, 253 x 211 x 187 R = 20: 29 / 34 / 38 us
        // a mode without this, 29 / 36 / 40 with it.)
        auto step = [&](int k, bool in) {
            double x[MT], y[NT];
#pragma unroll
            for (int m = 0; m < MT; m++) x[m] = A[kQ == 0 ? k * LDQ + 8 * m : 8 * m * LDK + k];
#pragma unroll
            for (int j = 0; j < NT; j++) y[j] = in ? B[k * T::LDB + 8 * j] * cc[j] : 0.0;
#pragma unroll
            for (int m = 0; m < MT; m++)
#pragma unroll
                for (int j = 0; j < NT; j++) dmma(acc[m][j], x[m], y[j]);
        };
        if (kc == DK) {
#pragma unroll
            for (int k = 0; k < DK; k += 4) step(k, true);
        } else {
            int k = 0;
#pragma unroll 1
            for (; k + 4 <= kc; k += 4) step(k, true);
            if (k < kc) step(k, k + fk < kc);
        }
        slot = slot + 1 == DST ? 0 : slot + 1;
        if (++cj == bsteps) {
            cj = 0;
            cb++;
        }
    }
    asm volatile("cp.async.wait_group 0;");

    double *P = a.part + z * (long)a.R * a.Q;
#pragma unroll
    for (int m = 0; m < MT; m++) {
        const long q = q0 + 32 * warp + 8 * m + (lane >> 2);
        if (q >= a.Q) continue;
#pragma unroll
        for (int j = 0; j < NT; j++)
#pragma unroll
            for (int c = 0; c < 2; c++) {
                const int r = r0 + 8 * j + 2 * (lane & 3) + c;
                if (r < a.R) P[q + a.Q * r] = acc[m][j][c];
            }
    }
    ptx::griddep_launch();
}

// out[e] = sum_z part[z][e]: a CTA owns sum_width(ZL) consecutive outputs, ZL
// lanes each over the splits, then a fixed order (two levels for 32 lanes).
template <int ZL>
__global__ void __launch_bounds__(sum_width(ZL) * ZL) k_sum_splits_f64(const double *__restrict__ part, int splits, long n,
                                                            double *__restrict__ out) {
    constexpr int OW = sum_width(ZL);
    __shared__ double red[ZL][OW];
    const int o = threadIdx.x % OW, zl = threadIdx.x / OW;
    const long e = blockIdx.x * (long)OW + o;
    ptx::griddep_wait();  // the partials
    double sum = 0.0;
    if (e < n) {
#pragma unroll 8
        for (int z = zl; z < splits; z += ZL) sum += __ldcs(part + (long)z * n + e);
    }
    red[zl][o] = sum;
    __syncthreads();
    constexpr int G = ZL > 8 ? 4 : 1;  // second-level sums
    if (zl < G) {
#pragma unroll
        for (int k = zl + G; k < ZL; k += G) sum += red[k][o];
        if (G > 1) red[zl][o] = sum;
    }
    if (G > 1) __syncthreads();
    if (zl == 0 && e < n) {
#pragma unroll
        for (int k = 1; k < G; k++) sum += red[k][o];
        out[e] = sum;
    }
}

struct F64Plan {
    int NT;
    bool any;  // factors beyond 32-bit indices
    long bsteps, qtiles, rtiles, steps, chunk, splits;
};

// Ranks per CTA at most 64, evenly over the rank tiles, in groups of 8; splits
// for one wave of the resident CTAs.
F64Plan f64_plan(int order, const long *dims, int mode, long R) {
    const ModeView v = mode_view(order, dims, mode);
    F64Plan p;
    int oth[kMaxOrder];
    const long rows0 = other_modes(order, dims, mode, oth) ? dims[oth[0]] : 1, blocks = v.P * v.S / rows0;
    p.bsteps = (rows0 + DK - 1) / DK;
    p.steps = blocks * p.bsteps;
    p.any = blocks > 0x3fffffffL || p.steps > 0x7fffffffL;
    for (int m = 0; m < order; m++) p.any = p.any || R * dims[m] > 0x3fffffffL;
    p.rtiles = (R + 63) / 64;
    const int rc = (int)((R + p.rtiles - 1) / p.rtiles);
    p.NT = p.any ? 8 : (rc + 7) / 8;
    if (p.NT == 5 || p.NT == 7) p.NT++;
    p.qtiles = (v.Q + DQ - 1) / DQ;
    const long want = std::max(1L, (p.NT <= 4 ? 3L : 2L) * kNumSMs / (p.qtiles * p.rtiles));
    p.splits = std::min(want, p.steps);
    p.chunk = (p.steps + p.splits - 1) / p.splits;
    p.splits = (p.steps + p.chunk - 1) / p.chunk;
    return p;
}

template <int kQ, bool kVec, bool kAny, int NT>
int launch(const F64Args &a, dim3 grid, cudaStream_t s) {
    static std::atomic<bool> attr[64];  // per device; zero-initialised
    constexpr size_t smem = DTile<kQ, NT>::kSmem;
    int dev = 0;
    CUD_CHECK(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64 || !attr[dev].load(std::memory_order_acquire)) {
        CUD_CHECK(cudaFuncSetAttribute(k_mttkrp_f64<kQ, kVec, kAny, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)smem));
        if (dev >= 0 && dev < 64) attr[dev].store(true, std::memory_order_release);
    }
    k_mttkrp_f64<kQ, kVec, kAny, NT><<<grid, DT, smem, s>>>(a);
    CUD_CHECK_LAUNCH("mttkrp_f64");
    return CUD_OK;
}

template <int kQ, bool kVec>
int launch_nt(const F64Plan &p, const F64Args &a, dim3 grid, cudaStream_t s) {
    switch (p.NT) {
        case 1: return launch<kQ, kVec, false, 1>(a, grid, s);
        case 2: return launch<kQ, kVec, false, 2>(a, grid, s);
        case 3: return launch<kQ, kVec, false, 3>(a, grid, s);
        case 4: return launch<kQ, kVec, false, 4>(a, grid, s);
        case 6: return launch<kQ, kVec, false, 6>(a, grid, s);
        default: return launch<kQ, kVec, false, 8>(a, grid, s);
    }
}

}  // namespace

size_t mttkrp_f64_ws_bytes(int order, const long *dims, int mode, long R) {
    return sizeof(double) * (size_t)f64_plan(order, dims, mode, R).splits * R * dims[mode];
}

int mttkrp_f64(const double *X, int order, const long *dims, const double *const *U, int mode, long R, double *out,
               void *ws, cudaStream_t s) {
    if (!ws) return CUD_ERR_INVALID_ARGUMENT;
    const ModeView v = mode_view(order, dims, mode);
    const F64Plan p = f64_plan(order, dims, mode, R);
    if (p.rtiles > 65535 || p.qtiles * p.splits > 0x7fffffffL) return CUD_ERR_UNSUPPORTED;
    F64Args a;
    a.X = X;
    a.P = v.P; a.Q = v.Q; a.S = v.S;
    a.R = (int)R;
    int oth[kMaxOrder];
    a.nf = other_modes(order, dims, mode, oth);
    for (int f = 0; f < a.nf; f++) {
        a.U[f] = U[oth[f]];
        a.rows[f] = dims[oth[f]];
    }
    a.bsteps = p.bsteps;
    const bool qfast = v.P == 1;  // q is contiguous in memory
    a.pblocks = qfast ? 1 : v.P / a.rows[0];
    a.qtiles = p.qtiles;
    a.steps = p.steps;
    a.chunk = p.chunk;
    a.part = static_cast<double *>(ws);
    const dim3 grid((unsigned)(p.qtiles * p.splits), (unsigned)p.rtiles);
    // 16-byte copies: whole ones along q, or of a row block of U0 (a pair that
    // crossed its end would multiply the next block's value by zero)
    const bool vec = (qfast ? v.Q : a.rows[0]) % 2 == 0 && (reinterpret_cast<uintptr_t>(X) & 15) == 0;
    const int pk = prof_begin(s);
    int st;
    if (p.any) st = qfast ? launch<0, false, true, 8>(a, grid, s) : launch<1, false, true, 8>(a, grid, s);
    else if (qfast) st = vec ? launch_nt<0, true>(p, a, grid, s) : launch_nt<0, false>(p, a, grid, s);
    else st = vec ? launch_nt<1, true>(p, a, grid, s) : launch_nt<1, false>(p, a, grid, s);
    prof_end(pk, s);
    if (st) return st;
    const long n = R * v.Q;
    const int lanes = sum_lanes((int)p.splits, n), ow = sum_width(lanes);
    PdlLaunch l((unsigned)((n + ow - 1) / ow), ow * lanes, 0, s);
    CUD_CHECK(cudaLaunchKernelEx(
        &l.cfg, lanes == 32 ? k_sum_splits_f64<32> : lanes == 8 ? k_sum_splits_f64<8> : k_sum_splits_f64<1>,
        (const double *)a.part, (int)p.splits, n, out));
    CUD_CHECK_LAUNCH("mttkrp_f64 reduce");
    return CUD_OK;
}

}  // namespace cud
