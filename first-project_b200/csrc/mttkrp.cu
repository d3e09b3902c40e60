// MTTKRP dispatch and the public MTTKRP entry points.
//
// CUD_PREC_FP32 runs a CUDA-core kernel; every other precision runs the
// tcgen05 tensor-core kernel where it applies (shape, alignment, rank) and
// otherwise the CUDA-core kernel with the same operand rounding
// (BF16X3/DEFAULT fall back to plain FP32, which is at least as accurate).
// DEFAULT takes plain FP32 unless the tensor cores are clearly the faster.
// The CUDA-core kernel of the entry points is mttkrp_ffma.cu's, or
// mttkrp_simt.cu's where the fastest factor has few rows; a CP-ALS plan's
// sweeps keep mttkrp_simt.cu's throughout (see there).
#include "kernels.cuh"
#include "tc_ptx.cuh"

namespace cud {

namespace {

// A CTA owns OW (32, or 256 for one lane each) consecutive slots of a partial
// (coalesced reads), each summed by ZL lanes over the splits z = lane, lane + ZL, .. and then in a fixed
// two-level order.  Bound: the latency of the chain of L2 reads, so the lanes
// are as many as the splits can feed.
template <int ZL>
__global__ void __launch_bounds__(sum_width(ZL) * ZL) k_sum_splits(const float *__restrict__ part, int splits, long Q, long R,
                                                        long Rp, const int *__restrict__ error,
                                                        float *__restrict__ out) {
    constexpr int OW = sum_width(ZL);
    __shared__ double red[ZL][OW];
    const int o = threadIdx.x % OW, zl = threadIdx.x / OW;
    const long e = blockIdx.x * (long)OW + o;
    const long n = Q * (Rp ? Rp : R);
    ptx::griddep_wait();  // the partials
    double sum = 0.0;
    if (e < n) {
#pragma unroll 8
        for (int z = zl; z < splits; z += ZL) sum += (double)__ldcs(part + (long)z * n + e);
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
        // a CTA whose bounded wait expired left its partial incomplete: the
        // output becomes NaN so the failure cannot pass for a result
        if (error && *error) sum = __longlong_as_double(0x7ff8000000000000LL);
        if (Rp) {
            const long q = e / Rp, r = e - q * Rp;
            if (r < R) out[q + Q * r] = (float)sum;
        } else {
            out[e] = (float)sum;
        }
    }
}
int round_mode(int precision) {
    return precision == CUD_PREC_FP16 ? 1 : precision == CUD_PREC_BF16 ? 2 : 0;
}
}  // namespace

int sum_splits(const float *part, int splits, long Q, long R, long Rp, const int *error, float *out, cudaStream_t s) {
    const long n = Q * (Rp ? Rp : R);
    const int lanes = sum_lanes(splits, n), ow = sum_width(lanes);
    PdlLaunch l((unsigned)((n + ow - 1) / ow), ow * lanes, 0, s);
    CUD_CHECK(cudaLaunchKernelEx(&l.cfg, lanes == 32 ? k_sum_splits<32> : lanes == 8 ? k_sum_splits<8> : k_sum_splits<1>,
                                 part, splits, Q, R, Rp, error, out));
    CUD_CHECK_LAUNCH("mttkrp reduce");
    return CUD_OK;
}

namespace {

// Small tensors run in plain FP32, which is what CUD_PREC_FP32 asks for and
// at least as accurate as what CUD_PREC_DEFAULT promises.
bool small_path(int order, const long *dims, int mode, long R, int precision) {
    return (precision == CUD_PREC_FP32 || precision == CUD_PREC_DEFAULT) && mttkrp_small_applies(order, dims, mode, R);
}

// A stage of k_mttkrp_ffma ends with a row block of the fastest factor, so with
// few rows there it is shallow, and k_mttkrp_simt's flat steps can be the faster
// ones: by the two kernels' estimates (B200, us, FFMA / flat steps: BF16 2 x 2 x
// 1000 x 1000 R = 8 mode 1 5700 / 1236, 5 x 700 x 700 R = 32 mode 1 58 / 37, 17 x 301 x
// 301 R = 64 28.8 / 30.7; FP32 2 x 4 x 301 x 101 R = 64 mode 0 188 / 102, mode 1 169 /
// 476, 7 x 301 x 301 R = 64 18.4 / 18.7).
bool simt_faster(int order, const long *dims, int mode, long R, int round) {
    int oth[kMaxOrder];
    const long rows0 = other_modes(order, dims, mode, oth) ? dims[oth[0]] : 1;
    return rows0 < 32 && mttkrp_ffma_us(order, dims, mode, R, round) > mttkrp_simt_us(order, dims, mode, R, round);
}
double cuda_core_us(int order, const long *dims, int mode, long R, int round) {
    return simt_faster(order, dims, mode, R, round) ? mttkrp_simt_us(order, dims, mode, R, round)
                                                    : mttkrp_ffma_us(order, dims, mode, R, round);
}

// CUD_PREC_DEFAULT: the tensor cores (BF16x3) where they are clearly the faster
// ones, else plain FP32, which is the more accurate one.  Where the packed-B
// kernel runs, FP32 up to 6.5e7 multiply-adds, and up to 8e7 counting whole tiles of 128
// rows, which both kernels compute (6e7 for 13 to 24 ranks and above 64, whose FP32
// tiles are the less efficient ones); of a mode of up to 16 rows only the whole
// tiles count, since FP32 can take twice as long there (B200, us a mode, tensor
// cores / FP32: 160^3 R = 12 (7.9e7 whole) 14.3 / 13.7, 128^3 R = 32 (6.7e7) 12.1 / 11.3,
// R = 48 (1.0e8) 13.5 / 15.1, 256^3 R = 4 (6.7e7) 20.8 / 14.7; 256 x 4 x 256 mode 1
// R = 8 (6.7e7 whole) 15.4 / 12.3, R = 32 (2.7e8) 18.4 / 21.3, R = 64 16.2 / 34.9, 512 x 64 x 8
// mode 2 R = 64 12.3 / 22.9; between, 32^4 R = 17 12.1 / 14.2).  Where the Khatri-Rao
// rows are built per stage the tensor cores are the slower ones (200^3 R = 16
// 52 / 22, R = 64 105 / 48, 500^3 R = 32 704 / 248, 100^4 R = 16 512 / 164), but for a
// fastest factor of few rows, where the estimates decide (3 x 256 x 256 x 32 R = 16
// mode 2 42 / 72, 2 x 2 x 1000 x 1000 R = 8 mode 3 23 / 61).
bool default_fp32(int order, const long *dims, int mode, long R, int precision) {
    if (precision != CUD_PREC_DEFAULT) return false;
    size_t b = 0;
    if (mttkrp_tc_query(order, dims, mode, R, precision, &b) != CUD_OK) return true;
    if (mttkrp_tc_packed(order, dims, mode, R, precision)) {
        double work = (double)R;
        for (int m = 0; m < order; m++) work *= (double)dims[m];
        const double whole = work / (double)dims[mode] * (double)((dims[mode] + 127) / 128 * 128);
        return whole <= ((R > 12 && R <= 24) || R > 64 ? 6e7 : 8e7) || (dims[mode] > 16 && work <= 6.5e7);
    }
    int oth[kMaxOrder];
    const long rows0 = other_modes(order, dims, mode, oth) ? dims[oth[0]] : 1;
    return rows0 >= 24 || cuda_core_us(order, dims, mode, R, 0) <= mttkrp_tc_us(order, dims, mode, R, precision);
}

}  // namespace

// Sized for both paths, so a call may fall back (e.g. a misaligned X) with
// the same workspace.
size_t mttkrp_ws_bytes(int order, const long *dims, int mode, long R, int precision) {
    const int round = round_mode(precision);
    size_t b = simt_faster(order, dims, mode, R, round) ? mttkrp_simt_ws_bytes(order, dims, mode, R, round)
                                                        : mttkrp_ffma_ws_bytes(order, dims, mode, R, round);
    size_t t = 0;
    if (precision != CUD_PREC_FP32 && mttkrp_tc_query(order, dims, mode, R, precision, &t) == CUD_OK)
        b = std::max(b, t);
    return b;
}

int mttkrp_run(const float *X, int order, const long *dims, const float *const *U, int mode, long R,
               float *out, int precision, void *ws, cudaStream_t s) {
    if (small_path(order, dims, mode, R, precision)) return mttkrp_small(X, order, dims, U, mode, R, out, s);
    if (precision != CUD_PREC_FP32 && !default_fp32(order, dims, mode, R, precision)) {
        size_t b = 0;
        if (mttkrp_tc_query(order, dims, mode, R, precision, &b) == CUD_OK) {
            int st = mttkrp_tc(X, order, dims, U, mode, R, out, precision, ws, s);
            if (st != CUD_ERR_UNSUPPORTED) return st;
        }
    }
    const int round = round_mode(precision);
    return simt_faster(order, dims, mode, R, round) ? mttkrp_simt_rounded(X, order, dims, U, mode, R, out, round, ws, s)
                                                    : mttkrp_ffma(X, order, dims, U, mode, R, out, round, ws, s);
}

size_t mttkrp_sweep_ws_bytes(int order, const long *dims, int mode, long R, int precision) {
    size_t b = mttkrp_simt_ws_bytes(order, dims, mode, R, round_mode(precision));
    size_t t = 0;
    if (precision != CUD_PREC_FP32 && mttkrp_tc_query(order, dims, mode, R, precision, &t) == CUD_OK)
        b = std::max(b, t);
    return b;
}

int mttkrp_sweep_run(const float *X, int order, const long *dims, const float *const *U, int mode, long R,
                     float *out, int precision, void *ws, cudaStream_t s, MttkrpParts *parts) {
    if (precision != CUD_PREC_FP32) {
        size_t b = 0;
        if (mttkrp_tc_query(order, dims, mode, R, precision, &b) == CUD_OK) {
            int st = mttkrp_tc(X, order, dims, U, mode, R, out, precision, ws, s, parts);
            if (st != CUD_ERR_UNSUPPORTED) return st;
        }
    }
    int st = mttkrp_simt_rounded(X, order, dims, U, mode, R, out, round_mode(precision), ws, s);
    if (st == CUD_OK && parts) *parts = MttkrpParts{out, 0, 1, dims[mode], 1, nullptr};
    return st;
}

}  // namespace cud

using namespace cud;

extern "C" int cud_mttkrp(const float *X, int order, const long *dims, const float *const *U,
                          int mode, long R, float *out, int precision, void *stream) {
    if (order < 2 || order > kMaxOrder || !dims || mode < 0 || mode >= order || R <= 0 || !X ||
        !U || !out || precision < 0 || precision > CUD_PREC_DEFAULT)
        return set_status(CUD_ERR_INVALID_ARGUMENT);
    for (int m = 0; m < order; m++) {
        if (dims[m] <= 0) return set_status(CUD_ERR_INVALID_ARGUMENT);
        if (m != mode && !U[m]) return set_status(CUD_ERR_INVALID_ARGUMENT);
    }
    int st;
    void *ws = scratch(kSlotMttkrp, mttkrp_ws_bytes(order, dims, mode, R, precision), &st);
    if (!ws) return set_status(st);
    return set_status(mttkrp_run(X, order, dims, U, mode, R, out, precision, ws, as_stream(stream)));
}

extern "C" int cud_mttkrp_path(int order, const long *dims, int mode, long R, int precision) {
    if (order < 2 || order > kMaxOrder || !dims || mode < 0 || mode >= order || R <= 0) return 0;
    if (precision == CUD_PREC_FP32) return 0;
    for (int m = 0; m < order; m++)
        if (dims[m] <= 0) return 0;
    if (small_path(order, dims, mode, R, precision) || default_fp32(order, dims, mode, R, precision)) return 0;
    size_t b = 0;
    return mttkrp_tc_query(order, dims, mode, R, precision, &b) == CUD_OK ? 1 : 0;
}

extern "C" int cud_mttkrp_legacy(const float *X, const float *left, const float *right, float *XU,
                                 long flag, long m, long n, long k, long r, int precision,
                                 void *stream) {
    if (flag < 1 || flag > 3) return set_status(CUD_ERR_INVALID_ARGUMENT);
    long dims[3] = {m, n, k};
    const float *U[3] = {nullptr, nullptr, nullptr};
    // src/mttkrp.cu:12,32,55: the KR row is right[x] * left[y], right fastest
    if (flag == 1) { U[1] = right; U[2] = left; }
    else if (flag == 2) { U[0] = right; U[2] = left; }
    else { U[0] = right; U[1] = left; }
    return cud_mttkrp(X, 3, dims, U, (int)flag - 1, r, XU, precision, stream);
}
