// MTTKRP on the FFMA pipe in FP32: the plain FP32 path, and the path of every
// shape, alignment or rank that the tensor-core kernels do not take (with the
// operands rounded first for FP16 and BF16).  Any order, any extents.
//
// Around mode n the tensor is a (P, Q, S) array and
//     M[q, r] = sum_kappa X(q, kappa) KR(kappa, r),
// kappa = s where P = 1 (mode 0; q contiguous in memory), kappa = p + P s for the
// other modes (p contiguous), KR(kappa, r) the product of the other factors' rows at
// kappa's digits.  X is read in its native layout, the Khatri-Rao rows are
// formed per stage in shared memory, nothing is materialised.
//
// Bound: FP32 FMA above rank ~18 (2 R flops for 4 bytes: 74 TFLOP/s against
// 6.5 TB/s), below it HBM.  What keeps an FFMA kernel from either is the
// shared memory that feeds it (a warp's load takes a clock of the SM per
// register filled, broadcast or not: 8 x 8 outputs a lane need 16 clocks of
// loads for 16 of multiply-adds) and the instructions beside the
// multiply-adds, so:
//   * a CTA (4 warps, two or three CTAs an SM) owns 128 rows q x NR TR ranks (at most
//     64) and a range of stages of up to 32 kappa; a lane accumulates TQ x TR
//     outputs, 16 x 8 where the rank allows (24 clocks of loads for 32),
//     TR = ceil(R / NR), so that odd ranks cost little padding;
//   * the warps split a stage's contraction (WK ways) before the rows, so
//     the lanes keep their tile at any Q; their accumulators are added in
//     shared memory, in warp order, at the end;
//   * a stage never leaves a row block of the fastest factor U0, so its
//     Khatri-Rao rows are U0's rows times one constant row c (the product of
//     the other factors' rows): U0's rows are copied to shared memory as they
//     are, and a lane scales the ranks it reads by its c, kept in registers
//     and renewed once a block.  Forming the rows per element (digits,
//     gathers, products, stores) took as many issue slots as the
//     multiply-adds;
//   * the multiply-adds are packed pairs (fma.rn.f32x2: the roundings of fmaf
//     at half the issue slots), along q for mode 0 and along r for the others,
//     whose X values lie along kappa in shared memory;
//   * X and U0 arrive by cp.async, two or three stages ahead: 16-byte copies
//     of X where its contiguous extent allows, else 4-byte copies (any extent
//     and alignment).
// B200, the kernel alone (events): 256^3 R = 32 37-39 us a mode (47-49 with
// 8 x 4 outputs a lane and a shared Khatri-Rao tile), 512^3 R = 64 381-424 us
// (45-40 TFLOP/s; 432-455), 512^3 R = 16 twice as fast; the ragged
// 253 x 211 x 187 R = 20 23-29 us (81-173 with 64 x 64 tiles of scalar loads).
// What is left: half of the FMA rate, at 8 to 12 warps an SM.
// Partials [split][r][q] are summed in FP64 by sum_splits.
#include <atomic>
#include <type_traits>

#include "kernels.cuh"
#include "tc_ptx.cuh"

namespace cud {

namespace {

constexpr int FQ = 128, FK = 32, FT = 128, NW = FT / 32;
constexpr int LDK = FK + 4;  // row stride of a [q][kappa] tile: 8 rows' 16-byte reads on distinct banks

struct FfmaArgs {
    const float *X;
    long P, Q, S;
    int R;
    int round;          // 0: operands as given; 1: X and the KR rows to FP16; 2: to BF16
    int nf;             // factors of the KR rows, fastest first
    const float *U[kMaxOrder];
    long rows[kMaxOrder];
    long bsteps;        // stages per row block of U0
    long pblocks;       // row blocks in P (modes other than 0)
    long qtiles;
    long steps, chunk;  // total stages, stages per split
    float *part;        // [split][R][Q]
};

__device__ __forceinline__ float round_to(float v, int mode) {
    if (mode == 1) return __half2float(__float2half_rn(v));
    if (mode == 2) return __bfloat162float(__float2bfloat16_rn(v));
    return v;
}

__device__ __forceinline__ void copy4(uint32_t dst, const float *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src));
}
__device__ __forceinline__ void copy16(uint32_t dst, const float *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src));
}

typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 dup2(float x) {
    f32x2 v;
    asm("mov.b64 %0, {%1, %1};" : "=l"(v) : "f"(x));
    return v;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 v;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(a), "l"(b));
    return v;
}
__device__ __forceinline__ f32x2 pack2(float x, float y) {
    f32x2 v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(x), "f"(y));
    return v;
}
__device__ __forceinline__ void fma2(f32x2 &c, f32x2 a, f32x2 b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b));
}
__device__ __forceinline__ float2 unpack2(f32x2 v) {
    float2 f;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
    return f;
}

// Tile of NR rank lanes: rows per lane, rows and contraction share per warp.
template <int kQ, int NR, int TR>
struct Tile {
    static constexpr int AF = kQ != 1 ? FK * FQ : FQ * LDK;  // floats of an X tile: [kappa][q] or [q][kappa]
    static constexpr int QL = 32 / NR;
    static constexpr int TQ = NR == 1 ? 4 : NR == 2 ? 8 : 16;
    static constexpr int WQ = QL * TQ;       // rows per warp: 128, or 64 with 8 rank lanes
    static constexpr int WM = FQ / WQ;
    static constexpr int WK = NW / WM;       // warps that share a stage's contraction
    // resident CTAs per SM and ring depth: three where 168 registers hold the
    // accumulators (more warps to hide latencies), else two
    static constexpr int MINB = TQ * TR <= 96 ? 3 : 2;
    static constexpr int NST = MINB == 3 ? 3 : 4;
    static constexpr int TP = (TR + 3) / 4;  // 4-rank groups per lane
    static constexpr int NG = NR * TP;       // 4-rank groups of a B row: [group of a lane][lane][4]
    static constexpr int LDB = NG * 4 + 4;   // B row stride: a copy's 32 rows on 8 bank groups
    static constexpr int BF = FK * LDB;
    static constexpr int BR = NR * TR;       // ranks per CTA
    static constexpr int LDQ = FQ + 8;       // row stride of the warps' sums: 4 rank lanes on distinct banks
    static constexpr size_t kRing = (size_t)NST * (AF + BF), kRed = (size_t)WK * BR * LDQ;
    static constexpr size_t kSmem = 4 * (kRing > kRed ? kRing : kRed);
};

// kQ 0: q contiguous in memory (mode 0); 1 and 2: the contraction index.  0
// and 2 keep a [kappa][q] tile, 1 a [q][kappa] one: 4-byte copies transpose
// as they land (2; the tile's columns swizzled so that a copy's 32 kappas
// fall on 16 banks: bits 2-4 by kappa's, bit 1 by kappa's bit 1), 16-byte
// ones cannot (1).  kVec: 16-byte copies of X.  kAny: operand rounding, or
// factors of 2^30 elements and more (64-bit indices; 4-byte copies).
template <int kQ, bool kVec, bool kAny, int NR, int TR>
__global__ void __launch_bounds__(FT, Tile<kQ, NR, TR>::MINB) k_mttkrp_ffma(const __grid_constant__ FfmaArgs a) {
    using T = Tile<kQ, NR, TR>;
    using I = std::conditional_t<kAny, unsigned long long, unsigned>;  // factor indices
    constexpr int AF = T::AF, BF = T::BF, NST = T::NST;
    extern __shared__ __align__(16) float smem[];
    float *Xring = smem, *Bring = smem + NST * AF;

    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int ql = lane / NR, rl = lane % NR;
    const int wm = warp % T::WM, wk = warp / T::WM;
    const long q0 = (blockIdx.x % a.qtiles) * FQ;
    const long z = blockIdx.x / a.qtiles;
    const int r0 = blockIdx.y * T::BR;
    const long sbeg = z * a.chunk;
    const long send = min(a.steps, sbeg + a.chunk);
    if (sbeg >= send) return;  // (no such CTA in the plan's grid)
    const int nst = (int)(send - sbeg);
    const long rows0 = a.rows[0];
    const int tail = (int)(rows0 - (a.bsteps - 1) * FK);  // kappas of a block's last stage

    // ---- copies.  The stage that is copied next: block lb, step lj in it.
    const I bsteps = (I)a.bsteps;
    I lb = (I)sbeg / bsteps;
    I lj = (I)sbeg - lb * bsteps;
    long lp = 0;  // kQ 1: position in the contiguous extent P
    const float *src;
    // X: each thread copies at kappa = ck (mode 0: + i STEP) and row cq (else: + i STEP)
    constexpr int NC = kVec ? 8 : 32;
    static_assert(kQ == 0 || kVec == (kQ == 1), "");
    const int cq = kQ == 0 ? (kVec ? 4 * lane : t % FQ) : (kVec ? t >> 3 : warp);
    const int ck = kQ == 0 ? (kVec ? warp : t / FQ) : (kVec ? 4 * (t & 7) : lane);
    constexpr int STEP = kQ == 0 ? (kVec ? NW : FT / FQ) : (kVec ? FT / 8 : NW);
    {
        if (kQ == 0) {
            src = a.X + q0 + cq + a.Q * ((long)lb * rows0 + (long)lj * FK + ck);
        } else {
            const I pb = (I)a.pblocks, s = lb / pb;  // blocks per s
            lp = (long)(lb - s * pb) * rows0 + (long)lj * FK;
            src = a.X + lp + ck + a.P * (q0 + cq + a.Q * (long)s);
        }
    }
    const long cstride = STEP * (kQ == 0 ? a.Q : a.P);
    // copies of this thread inside the tensor (mode 0: all or none); the
    // tile's other rows q keep what the memory holds and are not written out
    const long qleft = a.Q - q0 - cq;
    const int nrow = qleft <= 0 ? 0 : kQ == 0 ? NC : (int)min((long)NC, (qleft + STEP - 1) / STEP);
    const uint32_t xdst = smem_u32(Xring) + 4u * (kQ == 0 ? ck * FQ + cq : kQ == 1 ? cq * LDK + ck : ck * FQ);
    constexpr uint32_t dstride = 4u * STEP * (kQ == 0 ? FQ : LDK);
    const int swk = (ck & 28) | (ck & 2);
    // byte offset of copy i in its tile, from xdst
    auto place = [&](int i) { return kQ == 2 ? 4u * (uint32_t)((cq + STEP * i) ^ swk) : dstride * i; };
    // U0: lane = row, the warps take the ranks in turn; ranks past R repeat
    // rank R - 1 (their results are not written)
    constexpr int NB0 = (T::BR + NW - 1) / NW;
    const uint32_t bdst = smem_u32(Bring) + 4u * lane * T::LDB;
    auto load = [&](int slot) {
        const int kc = lj == bsteps - 1 ? tail : FK;
        const float *p = src;
        const uint32_t d = xdst + (uint32_t)slot * (4u * AF);
        // this thread's copies in the stage
        const int nr = kQ == 0 ? (nrow == 0 ? 0 : (kc - ck + STEP - 1) / STEP) : ck < kc ? nrow : 0;
        if (nr == NC) {
#pragma unroll
            for (int i = 0; i < NC; i++, p += cstride) {
                if constexpr (kVec) copy16(d + place(i), p);
                else copy4(d + place(i), p);
            }
        } else {
#pragma unroll 4
            for (int i = 0; i < nr; i++, p += cstride) {
                if constexpr (kVec) copy16(d + place(i), p);
                else copy4(d + place(i), p);
            }
        }
        const uint32_t bd = bdst + (uint32_t)slot * (4u * BF);
        const I row = lj * FK + lane;
#pragma unroll
        for (int i = 0; i < NB0; i++) {
            const int c = warp + NW * i;  // rank of the CTA's BR
            if (T::BR % NW != 0 && c >= T::BR) continue;
            const int j = c % TR, l = c / TR;  // rank j of lane l
            const uint32_t o = bd + 4u * ((j / 4) * (NR * 4) + l * 4 + (j & 3));
            const I r = (I)min(r0 + c, a.R - 1);
            if (lane < kc) copy4(o, a.U[0] + (row + r * (I)rows0));
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
    // Rounds this thread's copies of X in ring slot `slot` (rows past Q:
    // whatever is there).
    auto round_own = [&](int slot) {
        float *x = Xring + slot * AF + (kQ == 0 ? ck * FQ + cq : ck * FQ);
#pragma unroll 4
        for (int i = 0; i < NC; i++) x[place(i) / 4] = round_to(x[place(i) / 4], a.round);
    };

    // ---- the constant row of the block that is multiplied: this lane's
    // ranks (zero past TR)
    constexpr int H = T::TP * 2;
    f32x2 cc[H];
    auto const_row = [&](I block) {
        float c[2 * H];
#pragma unroll
        for (int j = 0; j < 2 * H; j++) c[j] = 1.f;
        I lin = block;
        for (int f = 1; f < a.nf; f++) {
            const I rows = (I)a.rows[f], next = lin / rows, d = lin - next * rows;
            lin = next;
#pragma unroll
            for (int j = 0; j < TR; j++) c[j] *= __ldg(a.U[f] + (d + (I)min(r0 + rl * TR + j, a.R - 1) * rows));
        }
#pragma unroll
        for (int j = 0; j < H; j++) cc[j] = pack2(c[2 * j], c[2 * j + 1]);
    };
    // B row k's values for this lane, scaled
    auto load_y = [&](const float *B, int k, f32x2 (&y)[H]) {
#pragma unroll
        for (int g = 0; g < T::TP; g++) {
            const ulonglong2 w = *reinterpret_cast<const ulonglong2 *>(B + k * T::LDB + 4 * g * NR);
            y[2 * g] = w.x;
            y[2 * g + 1] = w.y;
        }
#pragma unroll
        for (int j = 0; j < (TR + 1) / 2; j++) {
            y[j] = mul2(y[j], cc[j]);
            if (kAny) {
                const float2 v = unpack2(y[j]);
                y[j] = pack2(round_to(v.x, a.round), round_to(v.y, a.round));
            }
        }
    };

    // accumulators: pairs of rows (mode 0) or of ranks, with the last of an
    // odd number of ranks on its own
    constexpr int NA = kQ != 1 ? T::TQ / 2 : T::TQ, NB = kQ != 1 ? TR : TR / 2;
    constexpr bool kOdd = kQ == 1 && (TR & 1);
    f32x2 acc[NA][NB];
    float last[kOdd ? T::TQ : 1];
#pragma unroll
    for (int i = 0; i < NA; i++)
#pragma unroll
        for (int j = 0; j < NB; j++) acc[i][j] = 0;
#pragma unroll
    for (int i = 0; i < (kOdd ? T::TQ : 1); i++) last[i] = 0.f;
    // tile row i of this lane
    auto qrow = [&](int i) {
        return wm * T::WQ + (kQ != 1 ? 4 * ql + T::QL * 4 * (i >> 2) + (i & 3) : ql + T::QL * i);
    };

    // ---- the stages.  The copies' lead-in is the loop's first NST - 1
    // rounds (one copy of the code: a CTA runs a few to a few dozen stages,
    // and instruction fetches of code that runs once show).
    I cb = lb, cj = lj;  // block and step of the stage that is multiplied
    int slot = 0, fill = 0;
#pragma unroll 1
    for (int i = -(NST - 1); i < nst; i++) {
        if (i >= 0) {
            // this thread's copies of the stage have landed; after the barrier
            // everyone's have, and the slots read a stage ago are free
            asm volatile("cp.async.wait_group %0;" ::"n"(NST - 2));
            if (kAny && a.round) round_own(slot);
            __syncthreads();
        }
        if (i + NST - 1 < nst) load(fill);
        asm volatile("cp.async.commit_group;");
        fill = fill + 1 == NST ? 0 : fill + 1;
        if (i < 0) continue;
        if (i == 0 || cj == 0) const_row(cb);
        const int kc = cj == bsteps - 1 ? tail : FK;
        if constexpr (kQ != 1) {
            // the warp's kappas: its groups of 4, wk, wk + WK, ..
            const float *A = Xring + slot * AF;
            const float *B = Bring + slot * BF + 4 * rl;
            auto step = [&](const float *Ak, const int (&xo)[T::TQ / 4], const float *Bk, int u) {
                f32x2 yp[H];
                load_y(Bk, u, yp);
                ulonglong2 x[T::TQ / 4];
#pragma unroll
                for (int j = 0; j < T::TQ / 4; j++) {
                    x[j] = *reinterpret_cast<const ulonglong2 *>(Ak + u * FQ + xo[j]);
                    if (kQ == 2 && (u & 2)) {
                        const f32x2 w = x[j].x;
                        x[j].x = x[j].y;
                        x[j].y = w;
                    }
                }
#pragma unroll
                for (int c = 0; c < TR; c++) {
                    const float2 v = unpack2(yp[c / 2]);
                    const f32x2 yy = dup2((c & 1) ? v.y : v.x);
#pragma unroll
                    for (int j = 0; j < T::TQ / 4; j++) {
                        fma2(acc[2 * j][c], x[j].x, yy);
                        fma2(acc[2 * j + 1][c], x[j].y, yy);
                    }
                }
            };
#pragma unroll 1
            for (int k = 4 * wk; k < kc; k += 4 * T::WK) {
                const float *Ak = A + k * FQ, *Bk = B + k * T::LDB;
                int xo[T::TQ / 4];
#pragma unroll
                for (int j = 0; j < T::TQ / 4; j++) xo[j] = qrow(4 * j) ^ (kQ == 2 ? (k & 28) : 0);
                if (k + 4 <= kc) {
#pragma unroll
                    for (int u = 0; u < 4; u++) step(Ak, xo, Bk, u);
                } else {
#pragma unroll
                    for (int u = 0; u < 3; u++)
                        if (k + u < kc) step(Ak, xo, Bk, u);
                }
            }
        } else {
            // the warp's groups of 4 kappas: wk, wk + WK, .. (kc is a multiple of 4
            // here: whole 16-byte copies of a row block)
            const float *A = Xring + slot * AF + qrow(0) * LDK + 4 * wk;
            const float *B = Bring + slot * BF + 4 * rl + 4 * wk * T::LDB;
#pragma unroll 1
            for (int k = 0; k + 4 * wk < kc; k += 4 * T::WK) {
                f32x2 y[4][H];
#pragma unroll
                for (int u = 0; u < 4; u++) load_y(B, k + u, y[u]);
#pragma unroll
                for (int j = 0; j < T::TQ; j++) {
                    const float4 x = *reinterpret_cast<const float4 *>(A + T::QL * j * LDK + k);
                    const float xs[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
                    for (int u = 0; u < 4; u++) {
                        const f32x2 xx = dup2(xs[u]);
#pragma unroll
                        for (int c = 0; c < NB; c++) fma2(acc[j][c], xx, y[u][c]);
                        if constexpr (kOdd) last[j] = fmaf(xs[u], unpack2(y[u][NB]).x, last[j]);
                    }
                }
            }
        }
        slot = slot + 1 == NST ? 0 : slot + 1;
        if (++cj == bsteps) {
            cj = 0;
            cb++;
        }
    }
    asm volatile("cp.async.wait_group 0;");
    __syncthreads();

    // the warps' contraction shares, added in warp order
    constexpr int LDQ = T::LDQ;
    float *red = smem;  // [WK][BR][LDQ]
    float *mine = red + ((size_t)wk * T::BR + rl) * LDQ + qrow(0);  // rank c of lane l: row c NR + l
    if constexpr (kQ != 1) {
#pragma unroll
        for (int j = 0; j < T::TQ / 4; j++)
#pragma unroll
            for (int c = 0; c < TR; c++) {
                const float2 u = unpack2(acc[2 * j][c]), v = unpack2(acc[2 * j + 1][c]);
                *reinterpret_cast<float4 *>(mine + c * NR * LDQ + T::QL * 4 * j) = make_float4(u.x, u.y, v.x, v.y);
            }
    } else {
#pragma unroll
        for (int j = 0; j < T::TQ; j++) {
#pragma unroll
            for (int c = 0; c < NB; c++) {
                const float2 v = unpack2(acc[j][c]);
                mine[2 * c * NR * LDQ + T::QL * j] = v.x;
                mine[(2 * c + 1) * NR * LDQ + T::QL * j] = v.y;
            }
            if constexpr (kOdd) mine[(TR - 1) * NR * LDQ + T::QL * j] = last[j];
        }
    }
    __syncthreads();
    float *P = a.part + z * (long)a.R * a.Q;
    const int qt = t;
    static_assert(FT == FQ, "a thread per row");
    const long q = q0 + qt;
    if (q < a.Q) {
#pragma unroll 4
        for (int i = 0; i < T::BR; i++) {
            const int r = r0 + (i % NR) * TR + i / NR;
            float s = red[(size_t)i * LDQ + qt];
#pragma unroll
            for (int w = 1; w < T::WK; w++) s += red[((size_t)w * T::BR + i) * LDQ + qt];
            if (r < a.R) P[q + a.Q * r] = s;
        }
    }
    ptx::griddep_launch();
}

struct FfmaPlan {
    int NR, TR;
    bool any;  // operand rounding, or factors beyond 32-bit indices
    long bsteps, qtiles, rtiles, steps, chunk, splits;
};

// Ranks per CTA at most 64, evenly over the rank tiles; the fewest rank lanes
// that hold them 8 to a lane; splits for one wave of the resident CTAs.
FfmaPlan ffma_plan(int order, const long *dims, int mode, long R, int round) {
    const ModeView v = mode_view(order, dims, mode);
    FfmaPlan p;
    int oth[kMaxOrder];
    const long rows0 = other_modes(order, dims, mode, oth) ? dims[oth[0]] : 1, blocks = v.P * v.S / rows0;
    p.any = round != 0 || blocks > 0x3fffffffL || blocks * ((rows0 + FK - 1) / FK) > 0x7fffffffL;
    for (int m = 0; m < order; m++) p.any = p.any || R * dims[m] > 0x3fffffffL;
    p.rtiles = (R + 63) / 64;
    const int rc = (int)((R + p.rtiles - 1) / p.rtiles);  // 8 to a lane with kAny
    p.NR = rc <= 8 ? 1 : rc <= 16 ? 2 : rc <= 32 ? 4 : 8;
    p.TR = p.any ? 8 : std::max(4, (rc + p.NR - 1) / p.NR);
    p.qtiles = (v.Q + FQ - 1) / FQ;
    p.bsteps = (rows0 + FK - 1) / FK;
    p.steps = blocks * p.bsteps;
    const int tq = p.NR == 1 ? 4 : p.NR == 2 ? 8 : 16;
    const long want = std::max(1L, (tq * p.TR <= 96 ? 3L : 2L) * kNumSMs / (p.qtiles * p.rtiles));
    p.splits = std::min(want, p.steps);
    p.chunk = (p.steps + p.splits - 1) / p.splits;
    p.splits = (p.steps + p.chunk - 1) / p.chunk;
    return p;
}

template <int kQ, bool kVec, bool kAny, int NR, int TR>
int launch(const FfmaArgs &a, dim3 grid, cudaStream_t s) {
    static std::atomic<bool> attr[64];  // per device; zero-initialised
    constexpr size_t smem = Tile<kQ, NR, TR>::kSmem;
    int dev = 0;
    CUD_CHECK(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64 || !attr[dev].load(std::memory_order_acquire)) {
        CUD_CHECK(cudaFuncSetAttribute(k_mttkrp_ffma<kQ, kVec, kAny, NR, TR>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)smem));
        if (dev >= 0 && dev < 64) attr[dev].store(true, std::memory_order_release);
    }
    k_mttkrp_ffma<kQ, kVec, kAny, NR, TR><<<grid, FT, smem, s>>>(a);
    CUD_CHECK_LAUNCH("mttkrp_ffma");
    return CUD_OK;
}

template <int kQ, bool kVec, bool kAny, int NR>
int launch_tr(int TR, const FfmaArgs &a, dim3 grid, cudaStream_t s) {
    if constexpr (kAny) {
        return launch<kQ, kVec, true, NR, 8>(a, grid, s);
    } else {
        switch (TR) {
            case 4: if constexpr (NR == 1) return launch<kQ, kVec, false, NR, 4>(a, grid, s); else break;
            case 5: return launch<kQ, kVec, false, NR, 5>(a, grid, s);
            case 6: return launch<kQ, kVec, false, NR, 6>(a, grid, s);
            case 7: return launch<kQ, kVec, false, NR, 7>(a, grid, s);
            case 8: return launch<kQ, kVec, false, NR, 8>(a, grid, s);
        }
        return CUD_ERR_INVALID_ARGUMENT;  // (the plan gives no other)
    }
}

template <int kQ, bool kVec, bool kAny>
int launch_nr(const FfmaPlan &p, const FfmaArgs &a, dim3 grid, cudaStream_t s) {
    return p.NR == 1 ? launch_tr<kQ, kVec, kAny, 1>(p.TR, a, grid, s)
         : p.NR == 2 ? launch_tr<kQ, kVec, kAny, 2>(p.TR, a, grid, s)
         : p.NR == 4 ? launch_tr<kQ, kVec, kAny, 4>(p.TR, a, grid, s)
                     : launch_tr<kQ, kVec, kAny, 8>(p.TR, a, grid, s);
}

}  // namespace

// Microseconds that a CTA's stages take on B200, launches aside: fitted to 1048
// timed modes whose fastest factor has 2 to 24 rows (ranks 1 to 64, orders 2 to
// 5).  A stage of few kappas costs its barrier, the constant row's gathers and
// its copies (by the rank lanes, a third of it again for a full tile of rows
// q, and with 64-bit digits by their number), whatever its depth; the 64-rank
// tile's final sum takes 5 us.
double mttkrp_ffma_us(int order, const long *dims, int mode, long R, int round) {
    static const double kStage[4] = {0.9, 1.5, 1.3, 1.4}, kAnyStage[4] = {2.0, 2.2, 2.3, 2.7};
    static const double kDepth[4] = {0.0, 0.7, 0.7, 0.8}, kEnd[4] = {1.0, 1.1, 0.7, 4.7};
    const FfmaPlan p = ffma_plan(order, dims, mode, R, round);
    const int i = p.NR == 1 ? 0 : p.NR == 2 ? 1 : p.NR == 4 ? 2 : 3;
    const int tq = p.NR == 1 ? 4 : p.NR == 2 ? 8 : 16;
    const long ctas = p.qtiles * p.rtiles * p.splits, wave = (tq * p.TR <= 96 ? 3L : 2L) * kNumSMs;
    int oth[kMaxOrder];
    const int nf = other_modes(order, dims, mode, oth);
    const long rows0 = nf ? dims[oth[0]] : 1;
    // (the 64-rank tile's figure is for two CTAs an SM; narrower ones run three)
    const double crowd = i == 3 && tq * p.TR <= 96 ? 1.5 : 1.0;
    const double stage = (p.any ? kAnyStage : kStage)[i] * crowd + 0.6 * std::min(dims[mode], (long)FQ) / FQ +
                         kDepth[i] * std::min(rows0, (long)FK) / FK + (p.any ? 0.3 * std::max(0, nf - 3) : 0.0);
    return (kEnd[i] + stage * p.chunk) * ((ctas + wave - 1) / wave);
}

size_t mttkrp_ffma_ws_bytes(int order, const long *dims, int mode, long R, int round) {
    return sizeof(float) * (size_t)ffma_plan(order, dims, mode, R, round).splits * R * dims[mode];
}

int mttkrp_ffma(const float *X, int order, const long *dims, const float *const *U, int mode, long R, float *out,
                int round, void *ws, cudaStream_t s) {
    if (!ws) return CUD_ERR_INVALID_ARGUMENT;
    const ModeView v = mode_view(order, dims, mode);
    const FfmaPlan p = ffma_plan(order, dims, mode, R, round);
    if (p.rtiles > 65535 || p.qtiles * p.splits > 0x7fffffffL) return CUD_ERR_UNSUPPORTED;
    FfmaArgs a;
    a.X = X;
    a.P = v.P; a.Q = v.Q; a.S = v.S;
    a.R = (int)R;
    a.round = round;
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
    a.part = static_cast<float *>(ws);
    const dim3 grid((unsigned)(p.qtiles * p.splits), (unsigned)p.rtiles);
    const int pk = prof_begin(s);
    // 16-byte copies: along q whole ones; along kappa also whole ones of a row
    // block of U0 (a group of 4 that crossed its end would multiply the next
    // block's values, which may be infinite, by zeros)
    const bool vec = (qfast ? v.Q : a.rows[0]) % 4 == 0 && (reinterpret_cast<uintptr_t>(X) & 15) == 0;
    const bool any = p.any;
    const int st = qfast ? (any ? launch_nr<0, false, true>(p, a, grid, s)
                                : vec ? launch_nr<0, true, false>(p, a, grid, s) : launch_nr<0, false, false>(p, a, grid, s))
                             : (any ? launch_nr<2, false, true>(p, a, grid, s)
                                : vec ? launch_nr<1, true, false>(p, a, grid, s) : launch_nr<2, false, false>(p, a, grid, s));
    prof_end(pk, s);
    if (st) return st;
    return sum_splits(a.part, (int)p.splits, v.Q, R, 0, nullptr, out, s);
}

}  // namespace cud
