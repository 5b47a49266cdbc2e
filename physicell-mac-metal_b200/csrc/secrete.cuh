// secrete.cuh — one cell's secretion / uptake, shared by the kernels that
// apply it.
#pragma once

#include "pcg_kernels.cuh"

namespace pcg {

// One cell's processSecretion on one substrate (cell_phenotype.cpp:526-564):
// rho += c0; rho = (rho + c1) / c2; clamp at 0; FP32 store.  A term the
// instance never has (flags) is exactly +0 and is added as the constant.
__device__ __forceinline__ float secrete_terms(float rho32, double c0, double c1, double c2)
{
    double rho = static_cast<double>(rho32);
    rho = __dadd_rn(rho, c0);
    rho = __dadd_rn(rho, c1);
    rho = __ddiv_rn(rho, c2);
    if (rho < 0.0) rho = 0.0;
    return __double2float_rn(rho);
}

// The quotient a / b rounded as IEEE division rounds it, from y = RN(1 / b),
// without a call or a branch, so that several run side by side (the
// compiler's division is a subroutine of 128 cycles that does not overlap
// another): two residual corrections of a y give RN(a / b)
// (P. Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", 1990) while nothing over- or underflows: 'ok' is
// cleared when a (other than +0) or b leaves the range where that is certain.
__device__ __forceinline__ double quotient(double a, double b, double y, bool& ok)
{
    const uint32_t ea = static_cast<uint32_t>(__double2hiint(a)) & 0x7ff00000u;
    const uint32_t eb = static_cast<uint32_t>(__double2hiint(b)) & 0x7ff00000u;
    const bool a_fine = ea - (523u << 20) <= (1000u << 20) || __double_as_longlong(a) == 0;   // 2^-500 .. 2^500
    const bool b_fine = eb - (767u << 20) <= (512u << 20);                                    // 2^-256 .. 2^256
    ok = ok && a_fine && b_fine;
    double q = __dmul_rn(a, y);
#pragma unroll
    for (int i = 0; i < 2; ++i) q = __fma_rn(__fma_rn(-b, q, a), y, q);
    return q;
}

// RN(1 / b) by Newton iterations from the hardware's approximate reciprocal
// (20 bits, 40, then the full width, then the last place), for b in
// quotient()'s range.
__device__ __forceinline__ double reciprocal(double b)
{
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
#pragma unroll
    for (int i = 0; i < 3; ++i) y = __fma_rn(y, __fma_rn(-b, y, 1.0), y);
    return y;
}

// Uptake alone (both other terms +0) of one cell on N substrates of a voxel,
// side by side; rho + 0 + 0 is rho + 0.
template <int N>
__device__ __forceinline__ void take_up(float (&rho)[N], const double (&c2)[N])
{
    float v[N];
    bool ok = true;
#pragma unroll
    for (int u = 0; u < N; ++u) {
        double q = quotient(__dadd_rn(static_cast<double>(rho[u]), 0.0), c2[u], reciprocal(c2[u]), ok);
        if (q < 0.0) q = 0.0;
        v[u] = __double2float_rn(q);
    }
    if (!ok) {
#pragma unroll
        for (int u = 0; u < N; ++u) v[u] = secrete_terms(rho[u], 0.0, 0.0, c2[u]);
    }
#pragma unroll
    for (int u = 0; u < N; ++u) rho[u] = v[u];
}

// One cell on each of B voxels, side by side (y = RN(1 / c2)); a lane whose
// operands leave quotient()'s range takes the plain division.
template <int B>
__device__ __forceinline__ void secrete_side_by_side(float (&rho)[B], const double (&c0)[B], const double (&c1)[B],
                                                     const double (&c2)[B], const double (&y)[B], const bool (&act)[B])
{
    float v[B];
    bool ok = true;
#pragma unroll
    for (int b = 0; b < B; ++b) {
        const double a = __dadd_rn(__dadd_rn(static_cast<double>(rho[b]), c0[b]), c1[b]);
        double q = quotient(a, c2[b], y[b], ok);
        if (q < 0.0) q = 0.0;
        v[b] = __double2float_rn(q);
    }
    if (!ok) {
#pragma unroll
        for (int b = 0; b < B; ++b) v[b] = secrete_terms(rho[b], c0[b], c1[b], c2[b]);
    }
#pragma unroll
    for (int b = 0; b < B; ++b) rho[b] = act[b] ? v[b] : rho[b];
}

__device__ __forceinline__ float secrete_cell(float rho32, const double* __restrict__ cs, uint64_t o, uint64_t cap,
                                              uint32_t f)
{
    return secrete_terms(rho32, (f & 1u) ? cs[o] : 0.0, (f & 2u) ? cs[cap + o] : 0.0, cs[2 * cap + o]);
}

}  // namespace pcg
