// The local step's 3x3 rotation fits (csrc/arap_device.cuh) on the host, against
// the rotation a covariance was built from: S = U diag(1, s2, s3) V^T has the
// best rotation V diag(1, 1, det(U V^T)) U^T, for s2 from order one down to
// 1e-7, s3 half of it or close to it, both signs of the determinant, and S of
// order one or so small that its squares are zero in FP32.
//
// Tolerance: S's rounding and the fit's own turn R by some multiple of the
// precision over the smallest eigenvalue of the objective's Hessian,
// s2 - s3 with a reflection (64 roundings here); a result in FP32 is rounded
// once more.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <random>

#include "device_on_host.h"

#include "arap_device.cuh"

using namespace arapgpu;

namespace {

std::mt19937_64 rng(7);

void random_rotation(long double R[3][3]) {
    std::normal_distribution<double> n;
    long double q[4], s = 0;
    for (auto &x : q) {
        x = n(rng);
        s += x * x;
    }
    s = std::sqrt(s);
    for (auto &x : q) x /= s;
    const long double w = q[0], x = q[1], y = q[2], z = q[3];
    const long double M[3][3] = {{1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y)},
                                 {2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x)},
                                 {2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)}};
    std::memcpy(R, M, sizeof M);
}

// S = U diag(sig) V^T and its rotation V diag(1, 1, sign) U^T
void covariance(const long double sig[3], bool reflect, double S[3][3], long double R[3][3]) {
    long double U[3][3], V[3][3];
    random_rotation(U);
    random_rotation(V);
    for (int a = 0; a < 3; ++a)
        for (int b = 0; b < 3; ++b) {
            long double s = 0, r = 0;
            for (int k = 0; k < 3; ++k) {
                s += U[a][k] * sig[k] * V[b][k] * (k == 2 && reflect ? -1 : 1);
                r += V[a][k] * U[b][k];
            }
            S[a][b] = (double)s;
            R[a][b] = r;
        }
}

// The mixed form's fit of a vertex whose one-ring has the covariance S: rest
// edges the axes, current edges S's rows.
void mixed_fit(const double S[3][3], float R[3][3]) {
    const int32_t dcol[3] = {1, 2, 3};
    const double w64[3] = {1.0, 1.0, 1.0};
    Vec4<double> p[4] = {}, pc[4] = {};
    float Sf[3][3];
    for (int k = 0; k < 3; ++k) {
        double *e = &p[k + 1].x, *f = &pc[k + 1].x;
        e[k] = -1.0;
        for (int c = 0; c < 3; ++c) {
            f[c] = -S[k][c];
            Sf[k][c] = (float)S[k][c];
        }
    }
    for (int a = 0; a < 3; ++a)
        for (int b = 0; b < 3; ++b) R[a][b] = a == b;
    if (dev::rotation_warm(Sf, R)) return;
    float spread;
    dev::rotation_from_cov<float>(Sf, R, &spread);
    if (!(spread >= dev::kPolarFallback)) dev::rotation_fp64(0, 0, 3, dcol, w64, p, pc, 1, 0, R);
}

template <typename T> double distance(const T R[3][3], const long double ref[3][3]) {
    double e = 0.0;
    for (int a = 0; a < 3; ++a)
        for (int b = 0; b < 3; ++b) {
            const double d = std::fabs((double)((long double)R[a][b] - ref[a][b]));
            e = d <= 1e30 ? std::max(e, d) : 1e30;  // NaN counts as far
        }
    return e;
}

}  // namespace

int main() {
    bool ok = true;
    for (int k = 0; k <= 7; ++k)
        for (const long double near : {0.5L, 0.999L})
            for (const bool reflect : {false, true})
                for (const double scale : {1.0, 1e-24}) {
                    const long double s2 = k ? std::pow(10.0L, -k) / 2 : 0.5L, s3 = s2 * near,
                                      gap = reflect ? s2 - s3 : s2 + s3;
                    const double tol64 = 64 * 0x1p-52 / (double)gap + 8 * 0x1p-52;
                    // the mixed form's fit is redone in FP64 below kPolarFallback and
                    // where FP32 shows no covariance, else the FP32 covariance's rounding stands
                    const bool redone = s2 + s3 < 0.1L || scale < 1.0;
                    const double tol32 = redone ? tol64 + 0x1p-24 : 64 * 0x1p-23 / (double)gap;
                    double worst64 = 0.0, worst32 = 0.0;
                    for (int t = 0; t < 2000; ++t) {
                        const long double sig[3] = {scale, scale * s2, scale * s3};
                        double S[3][3], D[3][3];
                        long double ref[3][3];
                        covariance(sig, reflect, S, ref);
                        for (int a = 0; a < 3; ++a)
                            for (int b = 0; b < 3; ++b) D[a][b] = a == b;
                        dev::rotation_fit_fp64(S, D);
                        worst64 = std::max(worst64, distance(D, ref));
                        float F[3][3];
                        mixed_fit(S, F);
                        worst32 = std::max(worst32, distance(F, ref));
                    }
                    const bool good = worst64 <= tol64 && worst32 <= tol32;
                    ok = ok && good;
                    std::printf("s2 %.0e s3 %.3f s2 %s scale %.0e: fp64 %.1e (%.1e), mixed %.1e (%.1e)%s\n", (double)s2,
                                (double)near, reflect ? "-" : "+", scale, worst64, tol64, worst32, tol32,
                                good ? "" : "  FAILED");
                }
    std::printf(ok ? "ok\n" : "failed\n");
    return ok ? 0 : 1;
}
