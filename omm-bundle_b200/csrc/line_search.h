// The CG step's quartic line search, shared by the host driver and the coefficients' kernel.
#pragma once

#include <cmath>

namespace ommgpu {

// Quartic line search (omm_quartic.F90:60-153), on the host and, for small problems, on the device.
__host__ __device__ inline void solve_quartic(const double c[5], double* x_min, bool* fail) {
    const double Pi = 3.141592653589793238462643383279502884197;
    *fail = false;
    double a = 3.0 * c[3] / (4.0 * c[4]);
    double b = 2.0 * c[2] / (4.0 * c[4]);
    if ((fabs(b) >= 1.0e11) || (fabs(c[4]) <= 1.0e-11)) {
        *x_min = -0.5 * c[1] / c[2];
        return;
    }
    double d = c[1] / (4.0 * c[4]);
    double Q = (a * a - 3.0 * b) / 9.0;
    double R = (2.0 * a * a * a - 9.0 * a * b + 27.0 * d) / 54.0;
    if (R * R < Q * Q * Q) {
        double theta = acos(R / sqrt(Q * Q * Q));
        double t[3], z[3];
        t[0] = -2.0 * sqrt(Q) * cos(theta / 3.0) - a / 3.0;
        t[1] = -2.0 * sqrt(Q) * cos((theta + 2.0 * Pi) / 3.0) - a / 3.0;
        t[2] = -2.0 * sqrt(Q) * cos((theta - 2.0 * Pi) / 3.0) - a / 3.0;
        for (int i = 0; i < 3; ++i) {
            double tt = t[i];
            z[i] = c[4] * (tt * tt) * (tt * tt) + c[3] * tt * tt * tt + c[2] * tt * tt + c[1] * tt + c[0];
        }
        if (c[4] > 0.0) {
            int o[3];
            if (z[0] >= z[1] && z[0] >= z[2]) { o[0] = 0; o[1] = 1; o[2] = 2; }
            else if (z[1] > z[2]) { o[0] = 1; o[1] = 2; o[2] = 0; }
            else { o[0] = 2; o[1] = 0; o[2] = 1; }
            if ((0.0 <= t[o[0]]) && (t[o[1]] <= t[o[0]])) *x_min = t[o[1]];
            else *x_min = t[o[2]];
        } else {
            if (z[0] <= z[1] && z[0] <= z[2]) *x_min = t[0];
            else if (z[1] < z[2]) *x_min = t[1];
            else *x_min = t[2];
        }
    } else {
        double S = -(R >= 0.0 ? 1.0 : -1.0) * pow(fabs(R) + sqrt(R * R - Q * Q * Q), 1.0 / 3.0);
        double U = (S == 0.0) ? 0.0 : Q / S;
        *x_min = (S + U) - (a / 3.0);
        if (c[4] < 0.0) *fail = true;
    }
}

// The energy along the direction at x (omm.F90:470)
__host__ __device__ inline double quartic_energy(const double c[5], double x) {
    return c[4] * (x * x) * (x * x) + c[3] * x * x * x + c[2] * x * x + c[1] * x + c[0];
}

}  // namespace ommgpu
