// FP32 GEMM on the FFMA pipe over strided operands: mode products, unfolding
// Grams and reconstructions of column-major tensors, without copies.  The
// operand with more rows ("long") is cut into 128-row tiles, the other one
// ("short") into tiles of up to 64 columns:
//     C(row, n) = sum_{kin, kout} L(row, kin, kout) W(kin, kout, n).
//
// Bound: FP32 FMA for 16 columns and more (a TTM with J = 32 reads 4 bytes
// for 64 flops), HBM below.  The tile is the FP32 MTTKRP's: 16 x 8 outputs a
// lane where the columns allow, packed FMAs, the warps of a CTA splitting a
// 32-deep stage of the contraction first, cp.async three stages ahead -- 16
// bytes at a time where the long operand is contiguous along the rows or
// along k and aligned, else 4 bytes, with any strides, transposed as they
// land.  Rows may run over two levels (a mode product's (p, s)), so a batch
// of thin matrices fills whole tiles.
// B200, mode products of 256 x 240 x 224 with J = 32, three modes:
// 234 -> 121 us; unfolding Grams of 256^3 401-964 -> 242-249 us a mode.
#include <atomic>

#include "kernels.cuh"

namespace cud {

namespace {

constexpr int FQ = 128, FK = 32, FT = 128, NW = FT / 32;
constexpr int LDK = FK + 4;  // row stride of a [row][k] tile: 8 rows' 16-byte reads on distinct banks

struct RowGemm {
    long rows, rin;              // row = i + rin o
    long N, Kin, Kout;
    const float *L;
    long l_r, l_ro, l_k, l_ko;   // strides of i, o, kin, kout
    const float *W;
    long w_n, w_k, w_ko;
    float *C;                    // the result, or the partials [split]
    long c_r, c_ro, c_n, c_z;
    long bsteps, steps, chunk;   // stages per kout, in all, per split
    long rtiles;
};

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
__device__ __forceinline__ void fma2(f32x2 &c, f32x2 a, f32x2 b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b));
}
__device__ __forceinline__ float2 unpack2(f32x2 v) {
    float2 f;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
    return f;
}

// Tile of NR column lanes: rows per lane, rows and contraction share per warp.
template <int kQ, int NR, int TR>
struct Tile {
    static constexpr int AF = kQ != 1 ? FK * FQ : FQ * LDK;  // floats of a long tile: [k][row] or [row][k]
    static constexpr int QL = 32 / NR;
    static constexpr int TQ = NR == 1 ? 4 : NR == 2 ? 8 : 16;
    static constexpr int WQ = QL * TQ;       // rows per warp: 128, or 64 with 8 column lanes
    static constexpr int WM = FQ / WQ;
    static constexpr int WK = NW / WM;       // warps that share a stage's contraction
    static constexpr int MINB = TQ * TR <= 96 ? 3 : 2;
    static constexpr int NST = MINB == 3 ? 3 : 4;
    static constexpr int TP = (TR + 3) / 4;  // 4-column groups per lane
    static constexpr int NG = NR * TP;       // groups of a short row: [group of a lane][lane][4]
    static constexpr int LDB = NG * 4 + 4;
    static constexpr int BF = FK * LDB;
    static constexpr int BR = NR * TR;       // columns per CTA
    static constexpr int LDQ = FQ + 8;       // row stride of the warps' sums
    static constexpr size_t kRing = (size_t)NST * (AF + BF), kRed = (size_t)WK * BR * LDQ;
    static constexpr size_t kSmem = 4 * (kRing > kRed ? kRing : kRed);
};

// The long operand: kQ 0 contiguous along the rows, tile [k][row]; 1
// contiguous along k, tile [row][k] (16-byte copies); 2 any strides, tile
// [k][row], transposed by 4-byte copies (columns swizzled: bits 2-4 by k's,
// bit 1 by k's bit 1).  kVec: 16-byte copies.
template <int kQ, bool kVec, int NR, int TR>
__global__ void __launch_bounds__(FT, Tile<kQ, NR, TR>::MINB) k_gemm_ffma(const __grid_constant__ RowGemm a) {
    using T = Tile<kQ, NR, TR>;
    constexpr int AF = T::AF, BF = T::BF, NST = T::NST;
    extern __shared__ __align__(16) float smem[];
    float *Xring = smem, *Bring = smem + NST * AF;

    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int ql = lane / NR, rl = lane % NR;
    const int wm = warp % T::WM, wk = warp / T::WM;
    const long n0 = (blockIdx.x % a.rtiles) * T::BR;
    const long q0 = (blockIdx.x / a.rtiles) * FQ;
    const long z = blockIdx.y;
    const long sbeg = z * a.chunk;
    const long send = min(a.steps, sbeg + a.chunk);
    const int nst = (int)max(0L, send - sbeg);
    const int tail = (int)(a.Kin - (a.bsteps - 1) * FK);  // k's of a kout's last stage
    const int ncol = (int)min((long)T::BR, a.N - n0);

    // ---- copies.  The stage that is copied next: step lj of its kout.
    const long lb = sbeg / a.bsteps;
    long lj = sbeg - lb * a.bsteps;
    // long operand: each thread copies at k = ck (kQ 0: + i STEP) and row cq (else: + i STEP)
    static_assert(kQ == 0 || kVec == (kQ == 1), "");
    constexpr int NC = kVec ? 8 : 32;
    const int cq = kQ == 0 ? (kVec ? 4 * lane : t % FQ) : (kVec ? t >> 3 : warp);
    const int ck = kQ == 0 ? (kVec ? warp : t / FQ) : (kVec ? 4 * (t & 7) : lane);
    constexpr int STEP = kQ == 0 ? (kVec ? NW : FT / FQ) : (kVec ? FT / 8 : NW);
    const float *src = a.L + lb * a.l_ko + (lj * FK + ck) * a.l_k;
    if (kQ == 0) {
        const long row = min(q0 + cq, a.rows - 1), o = a.rin < a.rows ? row / a.rin : 0;
        src += (row - o * a.rin) * a.l_r + o * a.l_ro;
    } else {
        src += (q0 + cq) * a.l_r;
    }
    const long cstride = STEP * (kQ == 0 ? a.l_k : a.l_r);
    const long lwrap = a.l_ko - a.Kin * a.l_k;
    // copies of this thread inside the operand (kQ 0: all or none); the
    // tile's other rows keep what the memory holds and are not written out
    const long qleft = a.rows - q0 - cq;
    const int nrow = qleft <= 0 ? 0 : kQ == 0 ? NC : (int)min((long)NC, (qleft + STEP - 1) / STEP);
    const uint32_t xdst = smem_u32(Xring) + 4u * (kQ == 0 ? ck * FQ + cq : kQ == 1 ? cq * LDK + ck : ck * FQ);
    constexpr uint32_t dstride = 4u * STEP * (kQ == 0 ? FQ : LDK);
    const int swk = (ck & 28) | (ck & 2);
    // byte offset of copy i in its tile, from xdst
    auto place = [&](int i) { return kQ == 2 ? 4u * (uint32_t)((cq + STEP * i) ^ swk) : dstride * i; };
    // short operand: along its columns where they are contiguous, else along
    // k; columns past N repeat the last (their results are not written)
    const bool wn = a.w_n == 1;
    constexpr int NB0 = (T::BR * FK + FT - 1) / FT;
    const float *wsrc = a.W + n0 * a.w_n + lb * a.w_ko + lj * FK * a.w_k;
    const long wwrap = a.w_ko - a.Kin * a.w_k;
    const uint32_t bdst = smem_u32(Bring);
    auto load = [&](int slot) {
        const int kc = lj == a.bsteps - 1 ? tail : FK;
        const float *p = src;
        const uint32_t d = xdst + (uint32_t)slot * (4u * AF);
        const int nr = kQ == 0 ? (nrow == 0 ? 0 : max(0, (kc - ck + STEP - 1) / STEP)) : ck < kc ? nrow : 0;
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
#pragma unroll 4
        for (int i = 0; i < NB0; i++) {
            const int e = t + FT * i;
            const int k = wn ? e / T::BR : e & (FK - 1), c = wn ? e % T::BR : e / FK;
            if (T::BR * FK % FT != 0 && e >= T::BR * FK) continue;
            const int j = c % TR, l = c / TR;  // column j of lane l
            const uint32_t o = bd + 4u * (k * T::LDB + (j / 4) * (NR * 4) + l * 4 + (j & 3));
            if (k < kc) copy4(o, wsrc + k * a.w_k + min(c, ncol - 1) * a.w_n);
        }
        // the next stage
        src += kc * a.l_k;
        wsrc += kc * a.w_k;
        if (++lj == a.bsteps) {
            lj = 0;
            src += lwrap;
            wsrc += wwrap;
        }
    };

    constexpr int H = T::TP * 2;
    auto load_y = [&](const float *B, int k, f32x2 (&y)[H]) {
#pragma unroll
        for (int g = 0; g < T::TP; g++) {
            const ulonglong2 w = *reinterpret_cast<const ulonglong2 *>(B + k * T::LDB + 4 * g * NR);
            y[2 * g] = w.x;
            y[2 * g + 1] = w.y;
        }
    };
    // accumulators: pairs of rows or (kQ 1) of columns, with the last of an
    // odd number of columns on its own
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

    // ---- the stages; the copies' lead-in is the loop's first rounds
    long cj = lj;  // step of the stage that is multiplied
    int slot = 0, fill = 0;
#pragma unroll 1
    for (int i = -(NST - 1); i < nst; i++) {
        if (i >= 0) {
            // this thread's copies of the stage have landed; after the barrier
            // everyone's have, and the slot read a stage ago is free
            asm volatile("cp.async.wait_group %0;" ::"n"(NST - 2));
            __syncthreads();
        }
        if (i + NST - 1 < nst) load(fill);
        asm volatile("cp.async.commit_group;");
        fill = fill + 1 == NST ? 0 : fill + 1;
        if (i < 0) continue;
        const int kc = cj == a.bsteps - 1 ? tail : FK;
        if constexpr (kQ != 1) {
            // the warp's k: its groups of 4, wk, wk + WK, ..
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
            // the warp's groups of 4 k: wk, wk + WK, .. (kc is a multiple of 4
            // here, as Kin is)
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
        if (++cj == a.bsteps) cj = 0;
    }
    asm volatile("cp.async.wait_group 0;");
    __syncthreads();

    // the warps' contraction shares, added in warp order
    constexpr int LDQ = T::LDQ;
    float *red = smem;  // [WK][BR][LDQ]
    float *mine = red + ((size_t)wk * T::BR + rl) * LDQ + qrow(0);  // column c of lane l: row c NR + l
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
    float *C = a.C + z * a.c_z;
    auto value = [&](int q, int c) {  // column c of the CTA's: row (c % TR) NR + c / TR of the sums
        const int i = (c % TR) * NR + c / TR;
        float s = red[(size_t)i * LDQ + q];
#pragma unroll
        for (int w = 1; w < T::WK; w++) s += red[((size_t)w * T::BR + i) * LDQ + q];
        return s;
    };
    if (a.c_n == 1) {  // columns contiguous
#pragma unroll 4
        for (int e = t; e < FQ * T::BR; e += FT) {
            const int q = e / T::BR, c = e % T::BR;
            const long row = q0 + q;
            if (row >= a.rows || c >= ncol) continue;
            const long o = a.rin < a.rows ? row / a.rin : 0;
            C[(row - o * a.rin) * a.c_r + o * a.c_ro + n0 + c] = value(q, c);
        }
    } else {
        const long row = q0 + t;
        static_assert(FT == FQ, "a thread per row");
        if (row < a.rows) {
            const long o = a.rin < a.rows ? row / a.rin : 0;
            float *c0 = C + (row - o * a.rin) * a.c_r + o * a.c_ro + n0 * a.c_n;
#pragma unroll 4
            for (int c = 0; c < T::BR; c++)
                if (c < ncol) c0[c * a.c_n] = value(t, c);
        }
    }
}

// C(m, n) = the sum over the splits of the dense M x N partials, in
// FP64 and a fixed order: a CTA owns 256 / ZL consecutive outputs, ZL lanes each.
template <int ZL>
__global__ void __launch_bounds__(256) k_gemm_sum(const float *__restrict__ part, int splits, long M, long N, void *C,
                                                  long c_m, long c_n, int f64) {
    constexpr int OW = 256 / ZL;
    __shared__ double red[ZL][OW];
    const int o = threadIdx.x % OW, zl = threadIdx.x / OW;
    const long e = blockIdx.x * (long)OW + o, n = M * N;
    double sum = 0.0;
    if (e < n) {
#pragma unroll 8
        for (int z = zl; z < splits; z += ZL) sum += (double)part[(long)z * n + e];
    }
    red[zl][o] = sum;
    __syncthreads();
    if (zl == 0 && e < n) {
        for (int k = 1; k < ZL; k++) sum += red[k][o];
        const long j = e / M, i = e - j * M, off = i * c_m + j * c_n;
        if (f64) static_cast<double *>(C)[off] = sum;
        else static_cast<float *>(C)[off] = (float)sum;
    }
}

template <int kQ, bool kVec, int NR, int TR>
int launch(const RowGemm &a, dim3 grid, cudaStream_t s) {
    static std::atomic<bool> attr[64];  // per device; zero-initialised
    constexpr size_t smem = Tile<kQ, NR, TR>::kSmem;
    int dev = 0;
    CUD_CHECK(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64 || !attr[dev].load(std::memory_order_acquire)) {
        CUD_CHECK(cudaFuncSetAttribute(k_gemm_ffma<kQ, kVec, NR, TR>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)smem));
        if (dev >= 0 && dev < 64) attr[dev].store(true, std::memory_order_release);
    }
    k_gemm_ffma<kQ, kVec, NR, TR><<<grid, FT, smem, s>>>(a);
    CUD_CHECK_LAUNCH("gemm_ffma");
    return CUD_OK;
}

template <int kQ, bool kVec, int NR>
int launch_tr(int TR, const RowGemm &a, dim3 grid, cudaStream_t s) {
    if constexpr (NR == 1)
        if (TR <= 4) return launch<kQ, kVec, NR, 4>(a, grid, s);
    return TR <= 6 ? launch<kQ, kVec, NR, 6>(a, grid, s) : launch<kQ, kVec, NR, 8>(a, grid, s);
}

template <int kQ, bool kVec>
int launch_nr(int NR, int TR, const RowGemm &a, dim3 grid, cudaStream_t s) {
    return NR == 1 ? launch_tr<kQ, kVec, 1>(TR, a, grid, s) : NR == 2 ? launch_tr<kQ, kVec, 2>(TR, a, grid, s)
         : NR == 4 ? launch_tr<kQ, kVec, 4>(TR, a, grid, s) : launch_tr<kQ, kVec, 8>(TR, a, grid, s);
}

}  // namespace

int gemm_ffma(const GemmDesc &d, cudaStream_t s) {
    if (d.M <= 0 || d.N <= 0 || d.batch <= 0 || d.Kin <= 0 || d.Kout <= 0 || d.alpha != 1.f || d.beta != 0.f)
        return CUD_ERR_UNSUPPORTED;
    // a batch becomes a second level of rows: one B, and rows that are
    // contiguous on the inner level
    if (d.batch > 1 && (d.b_b != 0 || d.out_f64 || d.a_m != 1)) return CUD_ERR_UNSUPPORTED;
    RowGemm g;
    const bool la = d.batch > 1 || d.M >= d.N;  // the long operand is A
    g.Kin = d.Kin;
    g.Kout = d.Kout;
    if (la) {
        g.rows = d.M * d.batch; g.rin = d.M; g.N = d.N;
        g.L = d.A; g.l_r = d.a_m; g.l_ro = d.a_b; g.l_k = d.a_kin; g.l_ko = d.a_kout;
        g.W = d.B; g.w_n = d.b_n; g.w_k = d.b_kin; g.w_ko = d.b_kout;
        g.c_r = d.c_m; g.c_ro = d.c_b; g.c_n = d.c_n;
    } else {
        g.rows = d.N; g.rin = d.N; g.N = d.M;
        g.L = d.B; g.l_r = d.b_n; g.l_ro = 0; g.l_k = d.b_kin; g.l_ko = d.b_kout;
        g.W = d.A; g.w_n = d.a_m; g.w_k = d.a_kin; g.w_ko = d.a_kout;
        g.c_r = d.c_n; g.c_ro = 0; g.c_n = d.c_m;
    }
    if (g.Kout == 1) g.l_ko = g.w_ko = 0;
    g.bsteps = (g.Kin + FK - 1) / FK;
    g.steps = g.Kout * g.bsteps;
    // columns per CTA at most 64, evenly over the tiles; the fewest column
    // lanes that hold them 8 to a lane
    g.rtiles = (g.N + 63) / 64;
    const int rc = (int)((g.N + g.rtiles - 1) / g.rtiles);
    const int NR = rc <= 8 ? 1 : rc <= 16 ? 2 : rc <= 32 ? 4 : 8;
    int TR = (rc + NR - 1) / NR;
    TR = NR == 1 && TR <= 4 ? 4 : TR <= 6 ? 6 : 8;
    g.rtiles = (g.N + NR * TR - 1) / (NR * TR);
    const long tiles = (g.rows + FQ - 1) / FQ * g.rtiles;
    if (tiles > 0x7fffffffL) return CUD_ERR_UNSUPPORTED;
    // Short contractions are bound by the outputs, where the 64 x 64 tile's
    // plain stores win (B200, gencp at 256^3: R = 32 82 against 74 us, R = 96
    // 155 against 156, R = 128 191 against 199; with row-contiguous outputs
    // K = 64, J = 256 31 against 47).
    const long K = g.Kin * g.Kout;
    // (A 4096 x 4096 Gram over K = 64, whose partials pass through memory: 498
    // against 250 us.)
    if (K < (d.out_f64 ? 512 : g.c_n == 1 ? 96 : 64)) return CUD_ERR_UNSUPPORTED;
    // A stage does not leave its kout: with a short inner contraction the flat
    // 16-deep slices of the 64 x 64 tile are the faster ones (B200, Gram of mode 1,
    // us: 2 x 300 x 1000 117 against 50, 5 x 300 x 1000 136 against 116, 7 x 200 x 999 81
    // against 121).
    if (g.Kout > 1 && g.Kin < 6) return CUD_ERR_UNSUPPORTED;
    // splits of the contraction for one wave of the resident CTAs, at least
    // four stages each
    long splits = d.splits;
    if (splits <= 0) {
        const int tq = NR == 1 ? 4 : NR == 2 ? 8 : 16;
        const long want = std::max(1L, (tq * TR <= 96 ? 3L : 2L) * kNumSMs / tiles);
        splits = d.batch > 1 ? 1 : std::max(1L, std::min(std::min(want, (g.steps + 3) / 4), 256L));
    }
    const bool few = tiles * splits < kNumSMs;
    if (d.splits <= 0 && splits > 1) {
        // a few CTAs more than SMs double the time: fewer, longer ones then
        // (B200, Grams of 100^3 by mode, us: 158 and 200 CTAs 28.0 / 25.9 / 26.9, 126 and
        // 134 with longer ranges 23.2 / 22.6 / 22.3)
        const long even = kNumSMs / tiles, longer = even > 0 ? (g.steps + even - 1) / even : 0;
        const long turns = (tiles * splits + kNumSMs - 1) / kNumSMs;
        if (even > 0 && even < splits && longer < (g.steps + splits - 1) / splits * turns) splits = even;
    }
    g.chunk = (g.steps + splits - 1) / splits;
    splits = (g.steps + g.chunk - 1) / g.chunk;
    if (g.chunk > 0x7fffffffL || splits > 65535) return CUD_ERR_UNSUPPORTED;
    // A lone CTA an SM hides little of its latencies: with fewer CTAs than SMs
    // the 64 x 64 tile, whose CTAs are more and wider, is the faster one above
    // 32 columns (B200, TTM of 256 x 256 x 16, mode 0, 32 tiles: J = 64 27
    // against 23 us, J = 32 17 against 23).
    if (few && NR == 8) return CUD_ERR_UNSUPPORTED;
    // (70^3, 39 tiles over K = 70: J = 32 8.2 against 7.3.)
    if (tiles * splits < kNumSMs / 3 && NR == 4 && K < 96) return CUD_ERR_UNSUPPORTED;
    // Above 32 columns the two tiles multiply at the same rate, and the 64 x 64
    // one spreads over the SMs more evenly; this one gains by rows that fill whole
    // tiles over a batch and by a long operand that lies along k.  In us per
    // wave of the SMs, fitted to mode products over K = 64 to 1000 (B200, this tile
    // / 64 x 64: 1000 x 1000 x 20 mode 1 J = 64 139 / 119, 500 x 64 x 80 mode 1 J = 64 24 / 19,
    // 200^3 mode 2 J = 64 51 / 45; mode 1 J = 64 52 / 54, J = 200 146 / 184, mode 0 J = 64
    // 50 / 60, 31 x 77 x 500 mode 1 J = 128 19 / 29).
    if (NR == 8 && !d.out_f64) {
        const double turns = (double)((tiles * splits + kNumSMs - 1) / kNumSMs);
        const double mine = 1.0 + (TR == 8 ? 1.0 : 0.9) * (2.5 + 0.07 * K) * turns;
        const double old = (double)((d.M + 63) / 64 * ((d.N + 63) / 64) * d.batch) / (2.0 * kNumSMs);
        const double other = (g.l_r == 1 ? 1.0 : 1.22) * (2.0 + 0.045 * K + (1.5 + 0.07 * K) * old);
        if (mine > other) return CUD_ERR_UNSUPPORTED;
    }
    const bool part = d.out_f64 || splits > 1;
    g.C = static_cast<float *>(d.C);
    g.c_z = 0;
    if (part) {
        if (d.batch > 1) return CUD_ERR_UNSUPPORTED;
        int st;
        g.C = (float *)scratch(kSlotTmp2, sizeof(float) * (size_t)splits * d.M * d.N, &st);
        if (!g.C) return st;
        g.c_z = d.M * d.N;
        g.c_r = la ? 1 : d.M;
        g.c_n = la ? d.M : 1;
    }
    auto mult4 = [](long a, long b, long c) { return a % 4 == 0 && b % 4 == 0 && c % 4 == 0; };
    const bool aligned = (reinterpret_cast<uintptr_t>(g.L) & 15) == 0;
    const dim3 grid((unsigned)tiles, (unsigned)splits);
    int st;
    if (g.l_r == 1) {
        const bool vec = aligned && g.rin % 4 == 0 && mult4(g.l_k, g.l_ko, g.l_ro);
        st = vec ? launch_nr<0, true>(NR, TR, g, grid, s) : launch_nr<0, false>(NR, TR, g, grid, s);
    } else if (g.l_k == 1 && aligned && g.Kin % 4 == 0 && mult4(g.l_r, g.l_ko, 0)) {
        st = launch_nr<1, true>(NR, TR, g, grid, s);
    } else {
        st = launch_nr<2, false>(NR, TR, g, grid, s);
    }
    if (st) return st;
    if (part) {
        const long n = d.M * d.N;
        if (sum_lanes((int)splits, n) > 1)
            k_gemm_sum<8><<<(unsigned)((n + 31) / 32), 256, 0, s>>>(g.C, (int)splits, d.M, d.N, d.C, d.c_m, d.c_n,
                                                                    d.out_f64);
        else
            k_gemm_sum<1><<<(unsigned)((n + 255) / 256), 256, 0, s>>>(g.C, (int)splits, d.M, d.N, d.C, d.c_m, d.c_n,
                                                                      d.out_f64);
        CUD_CHECK_LAUNCH("gemm_ffma reduce");
    }
    return CUD_OK;
}

}  // namespace cud
