// arap_device.cuh -- device helpers shared by the single-pose and batched
// kernels: precision traits and the 3x3 rotation fit of the local step
// (inc/deform/arap.h:376-382).
#pragma once

#include <cuda_runtime.h>

#include "arap_kernels.h"

namespace arapgpu {
namespace dev {

template <typename T> __device__ __forceinline__ T tsqrt(T x);
template <> __device__ __forceinline__ float tsqrt(float x) { return sqrtf(x); }
template <> __device__ __forceinline__ double tsqrt(double x) { return sqrt(x); }

template <typename T> struct Eps;
template <> struct Eps<float> { static constexpr float v = 1.1920929e-07f; };
template <> struct Eps<double> { static constexpr double v = 2.220446049250313e-16; };

// Conversions on the integer pipe: an FP64 conversion instruction takes an FP64
// issue slot (about 64 clocks per warp and scheduler on this GPU).
// x 2^(1023 - e) in FP32, truncated (e: a biased FP64 exponent; the result must
// stay below 2^127; below 2^-126 it is 0)
__device__ __forceinline__ float to_float_scaled(double x, int e) {
    const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
    const int fe = (int)((hi >> 20) & 0x7ffu) - e + 127;
    const unsigned bits = ((unsigned)fe << 23) | ((hi & 0xfffffu) << 3) | (lo >> 29);
    return __uint_as_float((hi & 0x80000000u) | (fe > 0 ? bits : 0u));
}
// a finite x in FP64, denormals as 0
__device__ __forceinline__ double to_double_finite(float x) {
    const unsigned b = __float_as_uint(x), ex = (b >> 23) & 0xffu;
    const unsigned hi = (b & 0x80000000u) | (ex ? ((ex + 896u) << 20) | ((b >> 3) & 0xfffffu) : 0u);
    return __hiloint2double((int)hi, ex ? (int)(b << 29) : 0);
}
// (double)x. No branch to the conversion instruction: predicated off, it still
// holds the pipe (256 poses of 10,242 vertices 15.8 -> 16.6 ms with one).
__device__ __forceinline__ double to_double(float x) {
    const unsigned b = __float_as_uint(x), a = b & 0x7fffffffu;
    const bool small = a < 0x00800000u;  // denormals: normalised first
    const unsigned t = small ? __float_as_uint(fabsf(x) * 0x1p64f) : a;
    // exponent 255, infinities and NaN, becomes 2047
    const unsigned bias = small ? 832u << 20 : a >= 0x7f800000u ? 1792u << 20 : 896u << 20;
    const unsigned hi = (b & 0x80000000u) | (t ? (t >> 3) + bias : 0u);
    return __hiloint2double((int)hi, (int)(t << 29));
}

// (float)x, rounded to nearest even; outside FP32's normal range the
// conversion instruction
__device__ __forceinline__ float to_float_rn(double x) {
    unsigned long long b = (unsigned long long)__double_as_longlong(x);
    b += 0x0fffffffull + ((b >> 29) & 1ull);
    const unsigned hi = (unsigned)(b >> 32), lo = (unsigned)b;
    const int fe = (int)((hi >> 20) & 0x7ffu) - 896;
    if (fe <= 0 || fe >= 255) return (float)x;
    return __uint_as_float((hi & 0x80000000u) | ((unsigned)fe << 23) | ((hi & 0xfffffu) << 3) | (lo >> 29));
}

// A double as hi + mid + low in FP32: its leading 24 bits, the next 23 and the
// last 6. The difference of two is (hi - hi') + (mid - mid') + (low - low')
// with the rounding of the first difference (two-sum; none where the exponents
// agree) and of the first sum carried along, so that only the last addition
// rounds: the rounded FP64 difference, however short the edge, without an FP64
// instruction. 14 additions a component; the 5 of the plain sums rounded twice
// where exponents differ, 1.2e-7 instead of 6e-8.
// A magnitude below 2^-76 other than zero or from 2^128 on, and what is not
// finite, is NaN, and so is a covariance with it, which rotation_fp64 then
// forms in FP64.
struct Split {
    float hi, mid, low;
    __device__ __forceinline__ explicit Split(double x) {
        const unsigned h = (unsigned)__double2hiint(x), l = (unsigned)__double2loint(x), a = h & 0x7fffffffu;
        const unsigned q = a - (896u << 20);  // FP32's exponent and the fraction's upper 20 bits
        const unsigned f = (h & 0x80000000u) | (q << 3) | (l >> 29);
        const bool in = q - (51u << 20) < 204u << 20;
        hi = __uint_as_float(in ? f : (a | l) ? 0x7fffffffu : 0u);
        // bits as the fraction of a float of the right exponent, less its leading one (of zero: none)
        const unsigned e1 = (f & 0xff800000u) - (23u << 23), e2 = e1 - (23u << 23);
        mid = __uint_as_float(e1 | ((l >> 6) & 0x7fffffu)) - __uint_as_float(e1);
        low = __uint_as_float(e2 | ((l << 17) & 0x7e0000u)) - __uint_as_float(e2);
    }
    __device__ __forceinline__ float operator-(const Split &o) const {
        const float d = hi - o.hi, r = d - hi;
        const float s = (mid - o.mid) + ((hi - (d - r)) - (o.hi + r));
        const float t = d + s;
        return t + ((s - (t - d)) + (low - o.low));
    }
};

// Cosine and sine of the plane rotation that makes columns of squared norms a
// and b and inner product g orthogonal; false where they are already, to
// working precision. t = tan of the angle, the root of t^2 + 2 zeta t - 1 = 0
// of smaller magnitude, zeta = (b - a) / 2g.
__device__ __forceinline__ bool jacobi_angle(double a, double b, double g, double &c, double &sn) {
    if (fabs(g) <= Eps<double>::v * sqrt(a * b)) return false;
    const double zeta = (b - a) / (2.0 * g), az = fabs(zeta);
    const double r = az > 1.0 ? az * sqrt(1.0 + 1.0 / (az * az)) : sqrt(1.0 + az * az);
    const double t = (zeta < 0.0 ? -1.0 : 1.0) / (az + r);
    c = 1.0 / sqrt(1.0 + t * t);
    sn = c * t;
    return true;
}
// FP32: t = 2g / (d + sign(d) sqrt(d^2 + 4 g^2)), d = b - a. Any t gives a
// rotation; only c and sn = c t must be those of one angle to FP32 rounding,
// so t takes the approximate reciprocal and root, and c a Newton step after
// its approximate root. The columns are scaled to at most unit norm
// (rotation_from_cov), so nothing overflows; where d^2 + 4 g^2 underflows the
// columns are below FP32 resolution of the largest.
__device__ __forceinline__ bool jacobi_angle(float a, float b, float g, float &c, float &sn) {
    const float d = b - a, h = 2.f * g, q = fmaf(d, d, h * h);
    if (g * g <= Eps<float>::v * Eps<float>::v * (a * b) || !(q > 1e-37f)) return false;
    const float den = fabsf(d) + q * rsqrtf(q);
    const float t = copysignf(__fdividef(fabsf(h), den), d < 0.f ? -g : g);
    const float u = fmaf(t, t, 1.f), c0 = rsqrtf(u);
    c = c0 * fmaf(-0.5f * u * c0, c0, 1.5f);
    sn = c * t;
    return true;
}

// One-sided (Hestenes) Jacobi on a 3x3 matrix (Golub & Van Loan, Sec. 8.6.3;
// Demmel & Veselic 1992): plane rotations from the right orthogonalise the
// columns of B = S J1 J2 ..., V accumulates the rotations. On exit the columns
// of B are sigma_i u_i and those of V the right singular vectors. Working on S
// itself, not on S^T S, keeps the small singular directions accurate in FP32
// (the one-rings stretched close to rank one in the first iterations of a
// large handle move).
template <typename T>
__device__ __forceinline__ void hestenes3(T B[3][3], T V[3][3]) {
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) V[i][j] = (i == j) ? (T)1 : (T)0;
    const int sweeps = sizeof(T) == 4 ? 8 : 12;
    for (int sw = 0; sw < sweeps; ++sw) {
        bool rotated = false;
#pragma unroll
        for (int pq = 0; pq < 3; ++pq) {
            const int p = pq == 2 ? 1 : 0;
            const int q = pq == 0 ? 1 : 2;
            const T a = B[0][p] * B[0][p] + B[1][p] * B[1][p] + B[2][p] * B[2][p];
            const T b = B[0][q] * B[0][q] + B[1][q] * B[1][q] + B[2][q] * B[2][q];
            const T g = B[0][p] * B[0][q] + B[1][p] * B[1][q] + B[2][p] * B[2][q];
            T c, sn;
            if (!jacobi_angle(a, b, g, c, sn)) continue;  // columns orthogonal to working precision
            rotated = true;
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                const T bp = B[i][p], bq = B[i][q];
                B[i][p] = c * bp - sn * bq;
                B[i][q] = sn * bp + c * bq;
                const T vp = V[i][p], vq = V[i][q];
                V[i][p] = c * vp - sn * vq;
                V[i][q] = sn * vp + c * vq;
            }
        }
        if (!rotated) break;
    }
}

// Best rotation R = V diag(1,1,det(V U^T)) U^T for cov = U S V^T (arap.h:376-382),
// from the one-sided Jacobi SVD of cov: the right singular vectors v1, v2 of
// the two largest singular values and v3 = v1 x v2 (proper), the left ones
// u1 = b1/|b1|, u2 = Gram-Schmidt(b2) and u3 = u1 x u2 (proper). With both
// factors proper the sign of det(V U^T) lands on the smallest singular value,
// as the reference's reflection fix puts it.
// spread (optional): (sigma_2 + sigma_3) / sigma_1 of cov, which bounds how
// well R is determined by it (the polar factor's condition number is about
// its inverse); 0 for a zero covariance.
template <typename T>
__device__ __forceinline__ void rotation_from_cov(const T S_in[3][3], T R[3][3], T *spread = nullptr) {
    if (spread) *spread = (T)0;
    T f2 = (T)0;
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) f2 += S_in[i][j] * S_in[i][j];
    if (!(f2 > (T)0)) {
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int j = 0; j < 3; ++j) R[i][j] = (i == j) ? (T)1 : (T)0;
        return;
    }
    const T sc = (T)1 / tsqrt(f2);
    T B[3][3];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) B[i][j] = S_in[i][j] * sc;
    T Vm[3][3];
    hestenes3(B, Vm);
    // singular values (column norms of B), ordered descending
    T nrm[3];
#pragma unroll
    for (int j = 0; j < 3; ++j) nrm[j] = B[0][j] * B[0][j] + B[1][j] * B[1][j] + B[2][j] * B[2][j];
    // indices of the largest and second largest (ties keep the lower index)
    const int o0 = (nrm[1] > nrm[0]) ? ((nrm[2] > nrm[1]) ? 2 : 1) : ((nrm[2] > nrm[0]) ? 2 : 0);
    const int lo = o0 == 0 ? 1 : 0, hi = o0 == 2 ? 1 : 2;  // the other two, lo < hi
    const T nlo = lo == 0 ? nrm[0] : nrm[1], nhi = hi == 1 ? nrm[1] : nrm[2];
    const int o1 = (nhi > nlo) ? hi : lo;
    if (spread) {
        const T n0 = o0 == 0 ? nrm[0] : (o0 == 1 ? nrm[1] : nrm[2]);
        *spread = (tsqrt(nlo) + tsqrt(nhi)) / tsqrt(n0);
    }
    T v1[3], v2[3], v3[3];
    T u1[3], u2[3], u3[3];
    // columns picked by selects, not by indexing with o0/o1 (keeps every
    // array in registers)
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        v1[i] = o0 == 0 ? Vm[i][0] : (o0 == 1 ? Vm[i][1] : Vm[i][2]);
        v2[i] = o1 == 0 ? Vm[i][0] : (o1 == 1 ? Vm[i][1] : Vm[i][2]);
        u1[i] = o0 == 0 ? B[i][0] : (o0 == 1 ? B[i][1] : B[i][2]);
        u2[i] = o1 == 0 ? B[i][0] : (o1 == 1 ? B[i][1] : B[i][2]);
    }
    v3[0] = v1[1] * v2[2] - v1[2] * v2[1];
    v3[1] = v1[2] * v2[0] - v1[0] * v2[2];
    v3[2] = v1[0] * v2[1] - v1[1] * v2[0];
    const T n1 = tsqrt(u1[0] * u1[0] + u1[1] * u1[1] + u1[2] * u1[2]);
#pragma unroll
    for (int i = 0; i < 3; ++i) u1[i] /= n1;
    const T dp = u1[0] * u2[0] + u1[1] * u2[1] + u1[2] * u2[2];
#pragma unroll
    for (int i = 0; i < 3; ++i) u2[i] -= dp * u1[i];
    T n2 = tsqrt(u2[0] * u2[0] + u2[1] * u2[1] + u2[2] * u2[2]);
    if (!(n2 > (T)64 * Eps<T>::v * n1)) {
        // rank one: any unit vector orthogonal to u1
        const T a0 = fabs(u1[0]), a1 = fabs(u1[1]), a2 = fabs(u1[2]);
        const int mi = (a1 < a0) ? ((a2 < a1) ? 2 : 1) : ((a2 < a0) ? 2 : 0);
        const T d2 = mi == 0 ? u1[0] : (mi == 1 ? u1[1] : u1[2]);
#pragma unroll
        for (int i = 0; i < 3; ++i) u2[i] = (i == mi ? (T)1 : (T)0) - d2 * u1[i];
        n2 = tsqrt(u2[0] * u2[0] + u2[1] * u2[1] + u2[2] * u2[2]);
    }
#pragma unroll
    for (int i = 0; i < 3; ++i) u2[i] /= n2;
    u3[0] = u1[1] * u2[2] - u1[2] * u2[1];
    u3[1] = u1[2] * u2[0] - u1[0] * u2[2];
    u3[2] = u1[0] * u2[1] - u1[1] * u2[0];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) R[i][j] = v1[i] * u1[j] + v2[i] * u2[j] + v3[i] * u3[j];
}


// The mixed form's rotation fit runs in FP32. Where the one-ring's covariance
// is close to rank one ((sigma_2 + sigma_3) / sigma_1 below this bound, which
// happens where a large handle move stretches a one-ring in the first
// iterations), the FP32 rounding of the covariance is amplified by about the
// inverse of that ratio, so the fit is redone in FP64 from the FP64 rest and
// current positions: the FP64 arithmetic goes only where the stability needs
// it (a fraction of a percent of the vertices).
constexpr float kPolarFallback = 0.1f;

// The rotation of rotation_from_cov by Newton's method in FP32 from a nearby
// one, the vertex's rotation of the iteration before (the identity at first),
// in place. R of rotation_from_cov maximises tr(R S) over proper rotations.
// With R = R0 exp([w]x) the gradient at w = 0 is g, the axial vector of the
// skew part of Q = (S R0)^T, and the Hessian -H, H = tr(Q) I - sym(Q); the step
// w = H^-1 g is applied through the Cayley map, which keeps R orthogonal, and
// an error e becomes about e^2. About 130 FP32 instructions a step, one to
// three steps in most iterations, against some 1,500 of the Jacobi fit
// (256 poses of 10,242 vertices: local step 185 -> 154 us). The step after
// which the last one's remainder is below FP32 resolution orthonormalises R to
// first order and ends. A point with g = 0 and a positive definite H is the
// maximum (tr(R S) has no other local maximum on the proper rotations). False,
// and R undefined, where five steps do not end, or H is not safely positive
// definite: det(H) / tr(H)^3 above kWarmDet bounds (sigma_2 + sigma_3) / sigma_1
// from below by kPolarFallback (with x = (sigma_2 +- sigma_3) / sigma_1 it is at
// most x (1 + x/2)^2 / (2 + 2x)^3, 0.01035 at x = 0.1), so that what needs the
// FP64 fallback goes to the Jacobi fit, which tells.
constexpr float kWarmDet = 0.0104f;
__device__ __forceinline__ bool rotation_warm(const float S_in[3][3], float R[3][3]) {
    float f2 = 0.f;
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) f2 += S_in[i][j] * S_in[i][j];
    if (!(f2 > 1e-30f && f2 < 1e30f)) return false;
    const float sc = rsqrtf(f2);
    float S[3][3];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) S[i][j] = S_in[i][j] * sc;
#pragma unroll 1
    for (int it = 0; it < 5; ++it) {
        float Q[3][3];  // (S R)^T
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int b = 0; b < 3; ++b) Q[a][b] = S[b][0] * R[0][a] + S[b][1] * R[1][a] + S[b][2] * R[2][a];
        const float g0 = Q[2][1] - Q[1][2], g1 = Q[0][2] - Q[2][0], g2 = Q[1][0] - Q[0][1];
        const float h00 = Q[1][1] + Q[2][2], h11 = Q[0][0] + Q[2][2], h22 = Q[0][0] + Q[1][1];
        const float h01 = -0.5f * (Q[0][1] + Q[1][0]), h02 = -0.5f * (Q[0][2] + Q[2][0]),
                    h12 = -0.5f * (Q[1][2] + Q[2][1]);
        const float c00 = h11 * h22 - h12 * h12, c01 = h02 * h12 - h01 * h22, c02 = h01 * h12 - h02 * h11;
        const float c11 = h00 * h22 - h02 * h02, c12 = h01 * h02 - h00 * h12, c22 = h00 * h11 - h01 * h01;
        const float det = h00 * c00 + h01 * c01 + h02 * c02, tr = h00 + h11 + h22;
        if (!(h00 > 0.f && c22 > 0.f && det > kWarmDet * tr * tr * tr)) return false;
        // a = w / 2, w = H^-1 g; C(w) - I = f ([a]x + [a]x^2)
        const float id = __fdividef(0.5f, det);
        const float a0 = id * (c00 * g0 + c01 * g1 + c02 * g2), a1 = id * (c01 * g0 + c11 * g1 + c12 * g2),
                    a2 = id * (c02 * g0 + c12 * g1 + c22 * g2);
        const float n2 = a0 * a0 + a1 * a1 + a2 * a2, f = __fdividef(2.f, 1.f + n2);
        float K[3][3] = {{-f * (a1 * a1 + a2 * a2), f * (a0 * a1 - a2), f * (a0 * a2 + a1)},
                         {f * (a0 * a1 + a2), -f * (a0 * a0 + a2 * a2), f * (a1 * a2 - a0)},
                         {f * (a0 * a2 - a1), f * (a1 * a2 + a0), -f * (a0 * a0 + a1 * a1)}};
        const bool last = n2 < 4e-9f;
        if (last) {  // less half of R^T R - I
#pragma unroll
            for (int a = 0; a < 3; ++a)
#pragma unroll
                for (int b = a; b < 3; ++b) {
                    float x = a == b ? -1.f : 0.f;
#pragma unroll
                    for (int k = 0; k < 3; ++k) x = fmaf(R[k][a], R[k][b], x);
                    K[a][b] -= 0.5f * x;
                    if (a != b) K[b][a] -= 0.5f * x;
                }
        }
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const float r0 = R[a][0], r1 = R[a][1], r2 = R[a][2];
#pragma unroll
            for (int b = 0; b < 3; ++b) R[a][b] += r0 * K[0][b] + r1 * K[1][b] + r2 * K[2][b];
        }
        if (last) return true;
    }
    return false;
}

// FP64 rotation from an FP32 fit Rf by iterative refinement: FP64 only where
// the digits are made. With R = R0 exp([w]x) the objective's gradient g (the
// axial vector of the skew part of (S R)^T) and R's deviation from
// orthogonality E = R^T R - I are residuals, small numbers that FP64 products
// leave exact to FP64 rounding: 36 FP64 instructions a step. What is made of
// them needs only a few digits, so the Hessian H = tr(Q) I - sym(Q),
// w = H^-1 g, the Cayley map of w and the correction
//     dR = R ((I - E/2 + 3 E^2/8) C(w) - I)
// are formed in FP32 (H and R at Rf), and R + dR costs 9 more. A step leaves
// about |dR| (1e-6 / conditioning): with det(H) / tr(H)^3 above kNewtonDet
// (0.037 at equal singular values, 0.010 at (sigma_2 + sigma_3) / sigma_1 = 0.1
// without a reflection) 1e-6 -> 1e-11 -> below FP64 rounding in two steps, the
// first of which is all a result of FP32 needs. Below, steps go on until they
// are that small. FP64 Newton steps (S R, adjugate, Cayley map and products in
// FP64) take about 400 FP64 instructions for the same rotation, the FP64 Jacobi
// fit some thousands: the one-rings stretched by a handle's move made the first
// iterations' local step 62 to 67 us on the 61,600-vertex bar against 25 later,
// FP64 form.
// S's largest entry has the biased exponent e, Sf is S at that scale. False,
// and R undefined, below kRefineDet or where eight steps do not end.
// FULL false (the mixed form's refit, whose result is rounded to FP32) ends at
// |w / 2| of 1e-8, or after a first step within 1e-5, and goes down to
// kRefineDetFit, (sigma_2 +- sigma_3) / sigma_1 of about 8e-5: there H's FP32
// rounding is a hundredth of its small eigenvalue, so a step still leaves a
// hundredth, and errors stay below 3e-11 (random covariances of any smaller
// singular values). With the Jacobi fit from kRefineDet down the first local
// step of the twisted bar took 130 us more (set-up and one iteration 2,755 us,
// 2,603 so). An Rf that is no fit of Sf is refused by its gradient, 1e-6 of |S|
// for one made in FP32: the identity that stands for the rotation of an FP32
// covariance whose squares underflow can be anywhere.
constexpr float kNewtonDet = 4e-3f, kRefineDet = 6e-4f, kRefineDetFit = 1e-5f, kRefineSeed = 1e-10f;
constexpr int kRefineSteps = 8;

// What the steps share: Q = (S R)^T at Rf, adj(H), 1 / det(H)
struct RefineFrame {
    float Q[3][3], c00, c01, c02, c11, c12, c22, id;
    bool plain;  // a fixed number of steps suffices
    __device__ __forceinline__ bool init(const float Sf[3][3], const float Rf[3][3], float least) {
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int b = 0; b < 3; ++b) Q[a][b] = Sf[b][0] * Rf[0][a] + Sf[b][1] * Rf[1][a] + Sf[b][2] * Rf[2][a];
        const float h00 = Q[1][1] + Q[2][2], h11 = Q[0][0] + Q[2][2], h22 = Q[0][0] + Q[1][1];
        const float h01 = -0.5f * (Q[0][1] + Q[1][0]), h02 = -0.5f * (Q[0][2] + Q[2][0]),
                    h12 = -0.5f * (Q[1][2] + Q[2][1]);
        c00 = h11 * h22 - h12 * h12, c01 = h02 * h12 - h01 * h22, c02 = h01 * h12 - h02 * h11;
        c11 = h00 * h22 - h02 * h02, c12 = h01 * h02 - h00 * h12, c22 = h00 * h11 - h01 * h01;
        const float det = h00 * c00 + h01 * c01 + h02 * c02, tr = fabsf(h00) + fabsf(h11) + fabsf(h22);
        if (!(h00 > 0.f && c22 > 0.f && det > least * tr * tr * tr)) return false;
        plain = det > kNewtonDet * tr * tr * tr;
        id = 1.f / det;
        return true;
    }
    // the correction to R from g and E; returns |w / 2|^2
    __device__ __forceinline__ float correction(const float Rf[3][3], const float E[3][3], float g0, float g1, float g2,
                                                float dR[3][3]) const {
        // the gradient at the orthonormalised R (I - E/2): Q loses E Q / 2
        float M[3][3];
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int b = 0; b < 3; ++b) M[a][b] = E[a][0] * Q[0][b] + E[a][1] * Q[1][b] + E[a][2] * Q[2][b];
        const float f0 = (g0 - 0.5f * (M[2][1] - M[1][2])) * id, f1 = (g1 - 0.5f * (M[0][2] - M[2][0])) * id,
                    f2 = (g2 - 0.5f * (M[1][0] - M[0][1])) * id;
        // a = w / 2, w = H^-1 g; C(w) - I = f ([a]x + [a]x^2)
        const float a0 = 0.5f * (c00 * f0 + c01 * f1 + c02 * f2), a1 = 0.5f * (c01 * f0 + c11 * f1 + c12 * f2),
                    a2 = 0.5f * (c02 * f0 + c12 * f1 + c22 * f2);
        const float n2 = a0 * a0 + a1 * a1 + a2 * a2, f = 2.f / (1.f + n2);
        const float K[3][3] = {{-f * (a1 * a1 + a2 * a2), f * (a0 * a1 - a2), f * (a0 * a2 + a1)},
                               {f * (a0 * a1 + a2), -f * (a0 * a0 + a2 * a2), f * (a1 * a2 - a0)},
                               {f * (a0 * a2 - a1), f * (a1 * a2 + a0), -f * (a0 * a0 + a1 * a1)}};
        float D[3][3];  // -E/2 + 3 E^2/8, then the correction's factor
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int b = 0; b < 3; ++b)
                D[a][b] = -0.5f * E[a][b] + 0.375f * (E[a][0] * E[0][b] + E[a][1] * E[1][b] + E[a][2] * E[2][b]);
        float N[3][3];
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int b = 0; b < 3; ++b)
                N[a][b] = K[a][b] + D[a][b] + (D[a][0] * K[0][b] + D[a][1] * K[1][b] + D[a][2] * K[2][b]);
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int b = 0; b < 3; ++b) dR[a][b] = Rf[a][0] * N[0][b] + Rf[a][1] * N[1][b] + Rf[a][2] * N[2][b];
        return n2;
    }
    template <bool FULL> __device__ __forceinline__ bool done(int it, float n2) const {
        if (FULL) return plain ? it == 1 : n2 < 2.5e-27f;
        return n2 < (plain && it == 0 ? 1e-10f : 1e-16f);
    }
};

template <bool FULL>
__device__ __forceinline__ bool rotation_refine(const double S[3][3], int e, const float Sf[3][3],
                                                const float Rf[3][3], double R[3][3]) {
    RefineFrame fr;
    if (!fr.init(Sf, Rf, FULL ? kRefineDet : kRefineDetFit)) return false;
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int b = 0; b < 3; ++b) R[a][b] = to_double_finite(Rf[a][b]);
#pragma unroll 1
    for (int it = 0; it < kRefineSteps; ++it) {
        double g0 = 0.0, g1 = 0.0, g2 = 0.0;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            g0 += S[1][k] * R[k][2];
            g1 += S[2][k] * R[k][0];
            g2 += S[0][k] * R[k][1];
            g0 -= S[2][k] * R[k][1];
            g1 -= S[0][k] * R[k][2];
            g2 -= S[1][k] * R[k][0];
        }
        float E[3][3], dR[3][3];
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int b = a; b < 3; ++b) {
                double x = a == b ? -1.0 : 0.0;
#pragma unroll
                for (int k = 0; k < 3; ++k) x += R[k][a] * R[k][b];
                E[a][b] = E[b][a] = to_float_scaled(x, 1023);
            }
        const float f0 = to_float_scaled(g0, e), f1 = to_float_scaled(g1, e), f2 = to_float_scaled(g2, e);
        if (!FULL && it == 0 && !(f0 * f0 + f1 * f1 + f2 * f2 < kRefineSeed)) return false;
        const float n2 = fr.correction(Rf, E, f0, f1, f2, dR);
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int b = 0; b < 3; ++b) R[a][b] += to_double_finite(dR[a][b]);
        if (fr.done<FULL>(it, n2)) return true;
    }
    return false;
}

// Exponent and FP32 form of S for rotation_refine; false where the gradient's
// FP32 exponents would leave their range
__device__ __forceinline__ bool refine_scale(const double S[3][3], int &e, float Sf[3][3]) {
    e = 0;
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int b = 0; b < 3; ++b) e = max(e, (__double2hiint(S[a][b]) >> 20) & 0x7ff);
    if (!(e > 60 && e < 0x7f0)) return false;
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int b = 0; b < 3; ++b) Sf[a][b] = to_float_scaled(S[a][b], e);
    return true;
}

// FP64 covariance of vertex i's one-ring (estimateRotations, arap.h:358-374)
// and its rotation refined from the FP32 fit Rm (in place), from the rest
// positions p, current positions pc (element k of vertex k's pose at
// k * stride + off) and the FP64 weights: by rotation_refine, below its range
// by the FP64 Jacobi fit. There the FP32 fit is no seed for Newton's method:
// its error is FP32 rounding over (sigma_2 +- sigma_3) / sigma_1, and one step
// from it was off by half a turn below 1e-5 (one-rings with cap triangles).
// A Jacobi fit is one warp's chain of FP64 instructions: the iteration of a
// 900-vertex sheet with caps of a height of 1e-5 takes 73 us, 42 with caps of
// 1e-4, which the refinement takes.
__device__ __forceinline__ void rotation_fp64(int i, int e0, int e1, const int32_t *__restrict__ dcol,
                                              const double *__restrict__ w64, const Vec4<double> *__restrict__ p,
                                              const Vec4<double> *__restrict__ pc, int64_t stride, int64_t off,
                                              float Rm[3][3]) {
    const Vec4<double> pi = p[i], ci = pc[(int64_t)i * stride + off];
    double S[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
    for (int e = e0; e < e1; ++e) {
        const int j = dcol[e];
        const double wj = w64[e];
        const Vec4<double> pj = p[j], cj = pc[(int64_t)j * stride + off];
        const double ex = wj * (pi.x - pj.x), ey = wj * (pi.y - pj.y), ez = wj * (pi.z - pj.z);
        const double fx = ci.x - cj.x, fy = ci.y - cj.y, fz = ci.z - cj.z;
        S[0][0] += ex * fx; S[0][1] += ex * fy; S[0][2] += ex * fz;
        S[1][0] += ey * fx; S[1][1] += ey * fy; S[1][2] += ey * fz;
        S[2][0] += ez * fx; S[2][1] += ez * fy; S[2][2] += ez * fz;
    }
    double R[3][3];
    int ex;
    float Sf[3][3];
    if (!(refine_scale(S, ex, Sf) && rotation_refine<false>(S, ex, Sf, Rm, R))) rotation_from_cov<double>(S, R);
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int b = 0; b < 3; ++b) Rm[a][b] = to_float_rn(R[a][b]);
}

// Rotation fit of the FP64 form, from the FP32 fit (R: the rotation of the
// iteration before). Covariances closer to rank one than the refinement takes,
// or whose H is close to singular (a reflection with close small singular
// values), take the FP64 one-sided Jacobi fit.
__device__ __forceinline__ void rotation_fit_fp64(const double S[3][3], double R[3][3]) {
    int e;
    float Sf[3][3];
    if (refine_scale(S, e, Sf)) {
        float Rf[3][3];
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int b = 0; b < 3; ++b) Rf[a][b] = to_float_scaled(R[a][b], 1023);
        if (!rotation_warm(Sf, Rf)) rotation_from_cov<float>(Sf, Rf);
        if (rotation_refine<true>(S, e, Sf, Rf, R)) return;
    }
    rotation_from_cov<double>(S, R);
}

// The same by four lanes of a warp: lane l < 3 has row l of S and gets column l
// of R (lane 3 goes along with lane 0); R holds the rotation before on every
// lane. Column l's lane makes component l of g, E(l, l), E(l, l + 1) and its
// column's corrections: 15 FP64 instructions a step instead of 45, for small
// meshes, whose warps leave the FP64 pipes idle while each waits for its own
// chain.
__device__ __forceinline__ void rotation_fit_fp64_quad(const double row[3], int lane, const float Rb[3][3],
                                                       double col[3]) {
    const int q0 = lane & ~3, l = lane & 3, c = l == 3 ? 0 : l, c1 = c == 2 ? 0 : c + 1, c2 = c == 0 ? 2 : c - 1;
    const unsigned mask = 0xfu << q0;
    int e = 0;
#pragma unroll
    for (int k = 0; k < 3; ++k) e = max(e, (__double2hiint(row[k]) >> 20) & 0x7ff);
    e = max(e, __shfl_xor_sync(mask, e, 1));
    e = max(e, __shfl_xor_sync(mask, e, 2));
    if (e > 60 && e < 0x7f0) {  // as refine_scale
        float Sf[3][3], Rf[3][3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const float x = to_float_scaled(row[k], e);
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                Sf[a][k] = __shfl_sync(mask, x, q0 + a);
                Rf[a][k] = Rb[a][k];
            }
        }
        if (!rotation_warm(Sf, Rf)) rotation_from_cov<float>(Sf, Rf);
        RefineFrame fr;
        if (fr.init(Sf, Rf, kRefineDet)) {
            double Sa[3], Sb[3], C0[3], C1[3], C2[3];
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                Sa[k] = __shfl_sync(mask, row[k], q0 + c1);
                Sb[k] = __shfl_sync(mask, row[k], q0 + c2);
                C0[k] = to_double_finite(c == 0 ? Rf[k][0] : c == 1 ? Rf[k][1] : Rf[k][2]);
                C1[k] = to_double_finite(c == 0 ? Rf[k][1] : c == 1 ? Rf[k][2] : Rf[k][0]);
                C2[k] = to_double_finite(c == 0 ? Rf[k][2] : c == 1 ? Rf[k][0] : Rf[k][1]);
            }
#pragma unroll 1
            for (int it = 0; it < kRefineSteps; ++it) {
                double g = 0.0, x0 = -1.0, x1 = 0.0;
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    g += Sa[k] * C2[k];
                    x0 += C0[k] * C0[k];
                    g -= Sb[k] * C1[k];
                    x1 += C0[k] * C1[k];
                }
                const float gf = to_float_scaled(g, e), f0 = to_float_scaled(x0, 1023), f1 = to_float_scaled(x1, 1023);
                float E[3][3], dR[3][3], gs[3];
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                    gs[a] = __shfl_sync(mask, gf, q0 + a);
                    E[a][a] = __shfl_sync(mask, f0, q0 + a);
                    const int b = a == 2 ? 0 : a + 1;
                    E[a][b] = E[b][a] = __shfl_sync(mask, f1, q0 + a);
                }
                const float n2 = fr.correction(Rf, E, gs[0], gs[1], gs[2], dR);
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    C0[k] += to_double_finite(c == 0 ? dR[k][0] : c == 1 ? dR[k][1] : dR[k][2]);
                    C1[k] = __shfl_sync(mask, C0[k], q0 + c1);
                    C2[k] = __shfl_sync(mask, C0[k], q0 + c2);
                }
                if (fr.done<true>(it, n2)) {
#pragma unroll
                    for (int k = 0; k < 3; ++k) col[k] = C0[k];
                    return;
                }
            }
        }
    }
    double S[3][3], R[3][3];
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int a = 0; a < 3; ++a) S[a][k] = __shfl_sync(mask, row[k], q0 + a);
    rotation_from_cov<double>(S, R);
#pragma unroll
    for (int k = 0; k < 3; ++k) col[k] = c == 0 ? R[k][0] : c == 1 ? R[k][1] : R[k][2];
}

}  // namespace dev
}  // namespace arapgpu
