// phi.cuh — the standard normal distribution function in FP64 from a table of Taylor polynomials:
// ten fused multiply-adds where the library's erfc takes some fifty operations, on a device that
// issues FP64 at 1/64 of the FP32 rate.
//
// Phi(x) about x0 = k / 8: Phi(x0) + phi(x0) sum_n (-1)^(n-1) He_(n-1)(x0) h^n / n!, |h| <= 1/16,
// He the Hermite polynomials. Ten coefficients leave less than 2.3e-16 anywhere (and a relative
// 3e-10 at x = -8.2); beyond +-69/8 Phi is 0 or 1 to 1e-17.
#pragma once

#include <cuda_runtime.h>

namespace thoth {

constexpr int PHI_NODES = 139, PHI_COEF = 10, PHI_MID = 69;

// the table [PHI_NODES][PHI_COEF] (host)
void phi_coefficients(double* out);

// tab: 16-byte aligned, in shared or global memory
__device__ __forceinline__ double phi_table(const double* tab, double x)
{
    const double u = fmin(fmax(x, -8.625), 8.625);
    const int k = __double2int_rn(u * 8.0);
    const double h = fma((double)k, -0.125, u); // exact
    const double2* c = reinterpret_cast<const double2*>(tab + (k + PHI_MID) * PHI_COEF);
    double2 a = c[4];
    double p = fma(a.y, h, a.x);
#pragma unroll
    for (int i = 3; i >= 0; --i) {
        a = c[i];
        p = fma(fma(p, h, a.y), h, a.x);
    }
    return x == x ? p : x;
}

} // namespace thoth
