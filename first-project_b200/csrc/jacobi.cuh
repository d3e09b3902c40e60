// The rotation of the FP64 Jacobi kernels (eig.cu, subspace.cu).
#pragma once

namespace cud {

// The rotation that annihilates the pair's off-diagonal apq.  The angle is
// formed in FP32 -- it leaves about 1e-7 of apq behind, which the next visit
// takes, so the convergence stays quadratic -- while c = (1 + t^2)^-1/2 (an
// FP32 estimate y, then one third-order Newton step on 1 - w y^2 in FP64) and
// s = t c are a rotation to FP64 rounding.  The FP64 division and square
// roots of an exact angle were most of a round's serial chain.  No rotation
// where |apq| <= 1e-17 sqrt|app aqq| (kSkip; otherwise where apq is next to
// zero or the angle is).
__device__ __forceinline__ double rcp_approx(double x) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    return y;
}
template <bool kSkip = true>
__device__ __forceinline__ void jacobi_rotation(double app, double aqq, double apq, double &c, double &s) {
    const double inv = rcp_approx(apq);
    // (apq / app) (apq / aqq) against 1e-34; a zero diagonal gives infinity
    const double ratio = kSkip ? fabs((apq * rcp_approx(app)) * (apq * rcp_approx(aqq))) : 1.0;
    const float th = 0.5f * (float)((aqq - app) * inv);
    float root, t;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(root) : "f"(fmaf(th, th, 1.f)));
    // |theta| beyond FP32's square: t < 3e-20, no rotation
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(t) : "f"(fabsf(th) + root));
    t = copysignf(t, th);
    const bool go = fabs(apq) > 1e-300 && ratio > 1e-34 && t == t;
    t = go ? t : 0.f;
    float y32;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y32) : "f"(fmaf(t, t, 1.f)));
    const double td = (double)t, y = (double)y32;
    const double ty = td * y;                             // exact: 24 x 24 bits
    const double r = fma(-ty, ty, fma(-y, y, 1.0));       // 1 - (1 + t^2) y^2
    const double g = fma(0.375, r, 0.5);
    c = fma(y * r, g, y);
    s = fma(ty * r, g, ty);
}

}  // namespace cud
