// Device-side building blocks shared by all EU3D kernels: the HBM layout of
// the flowfield, the mechanism tables in constant memory and the NASA-9
// thermodynamic polynomials.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "../../include/eu3d_quirks.h"

namespace eu3d {

constexpr int NS = 9;        // species of the H2_JA919 mechanism
constexpr int NR = 19;       // reactions
constexpr int NV = NS + 4;   // conserved variables: NS partial densities, 3 momenta, total energy
constexpr int NPRIM = 7 + NS;  // primitive fields read by the flux sweeps
// primitive field order
constexpr int PD = 0, PU = 1, PV = 2, PW = 3, PP = 4, PH = 5, PG = 6, PY = 7;

constexpr double R_GAS = 8.31434;   // include/Reaction.hpp:269
constexpr double RU_CAL = 1.987;    // include/Reaction.hpp:270
constexpr double P0 = 101325.0;     // include/Reaction.hpp:271

// Ghost-padded structured grid in structure-of-arrays form: x fastest, each
// row padded to a multiple of 32 elements so that rows start 128-byte (FP32)
// or 256-byte (FP64) aligned, fields `fs` elements apart.
struct Layout {
    int ni, nj, nk, bc;
    int NI, NJ, NK;
    int px;        // row pitch in elements
    long long fs;  // field stride in elements
    __host__ __device__ long long at(int i, int j, int k) const { return ((long long)k * NJ + j) * px + i; }
    __host__ __device__ long long interior_cells() const { return (long long)ni * nj * nk; }
};

// Mechanism and thermo tables (constant memory, broadcast to all lanes).
struct MechConst {
    double c[2][9][NS];  // NASA-9 coefficients [range][a1..a7,b1,b2][species]
    double mw[NS], ri[NS];
    double imw[NS];      // 1 / mw
    double af[NR], bf[NR], eaf[NR];
    double sf[NS][NR], sb[NS][NR], tb[NS][NR];
    double nu[NS][NR];   // sb - sf
    double xr[NR];       // sum over species of (sb - sf)
    double p0xr[NR];     // pow(P0 * 1e-6, xr), evaluated on the host
    int has_tb[NR];      // reaction has third-body efficiencies
};

// defined once: every kernel lives in the single translation unit eu3d_gpu.cu
__constant__ MechConst cM;

struct Status {
    unsigned long long nonfinite;
    unsigned long long newton_capped;
    unsigned long long substeps;
    int nchem_max;
    int substep_capped;
    unsigned long long sur_cells;
    unsigned long long sur_fallback;
    unsigned long long audit_cells;        // surrogate cells also run through the integrator
    unsigned long long audit_max_dT_bits;  // largest |T_surrogate - T_integrator| (double bits)
    unsigned long long sur_reject[4];      // rejections: envelope, network output, energy residual, decode
    unsigned long long wait_timeouts;      // kernels that gave up a bounded wait (shared-memory ring, TMA)
    unsigned long long sur_frozen;         // cells the frozen-chemistry gate left out of the network
    unsigned long long frozen_audit_cells; // of those, cells also run through the integrator
    unsigned long long frozen_audit_max_dT_bits;  // largest |T_integrator - T| over them (double bits)
    unsigned long long drain_timeouts;     // a bounded wait for copies in flight after a timeout ran out too
};

// FP64 quotients and square roots without the compiler's out-of-line paths:
// the hardware's approximation, with e its residual three terms of the series of
// (1 - e)^-1 or (1 - e)^-1/2 (what is left is of order e^3), and Markstein's
// final correction by the exact remainder (P. Markstein, IBM J. Res. Dev. 34,
// 1990).  They round as IEEE division and square root do for
//     div_by, div_rn   2^-968 <= |a|, 2^-1000 <= |b| <= 2^1000, a normal quotient; or a = 0
//     rcp_rn           2^-1000 <= x <= 2^1000
//     sqrt_rn          2^-960 <= x, or 0
// but for one kind of quotient.  The correction's error is the remainder's share
// of the reciprocal's error, half an ulp and 2^-7 of an ulp more where 1/b is next
// to a midpoint (rcp_1ulp may then be the other neighbour); with b in [1, 2) it
// stays below the least distance of a quotient of doubles from a midpoint, 2^-106
// / b, while b (1 + 2^-7) < 2.  For b above 1.984 a quotient at that distance may
// come out as its other neighbour.  (Two more operations for an exactly rounded
// reciprocal would settle these, one pair of operands in 2^60 or fewer: FP64 flux of
// 160^3 0.84 ms against 0.78, one-step IMEX of 1.3 M cells 331 us against 309.)
// A test holds all this to IEEE's bits: random operands, significands next to all
// ones, quotients next to a midpoint, the ends of the ranges.  Below the
// numerators' bound the remainder is inexact and the last bit may differ; zero,
// infinite or NaN divisors and quotients past the range give NaN.
__device__ __forceinline__ double rcp_approx(double x)
{
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    return y;
}
__device__ __forceinline__ double rsqrt_approx(double x)
{
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    return y;
}
// 1/x within an ulp
__device__ __forceinline__ double rcp_1ulp(double x)
{
    const double y = rcp_approx(x), e = __fma_rn(-x, y, 1.0);
    return __fma_rn(y, __fma_rn(e, e, e), y);
}
// a/b from r = rcp_1ulp(b)
__device__ __forceinline__ double div_by(double a, double b, double r)
{
    const double q = __dmul_rn(a, r);
    return __fma_rn(__fma_rn(-b, q, a), r, q);
}
__device__ __forceinline__ double div_rn(double a, double b) { return div_by(a, b, rcp_1ulp(b)); }
// 1/x, x > 0.  The correction starts from an estimate rounded up: from below, that
// of an all-ones divisor ends in a tie that rounds the wrong way.
__device__ __forceinline__ double rcp_rn(double x)
{
    const double y0 = rcp_approx(x), e = __fma_rn(-x, y0, 1.0);
    const double y = __fma_ru(y0, __fma_rn(e, e, e), y0);
    return __fma_rn(__fma_rn(-x, y, 1.0), y, y);
}
__device__ __forceinline__ double sqrt_rn(double x)
{
    const double y0 = rsqrt_approx(x);
    const double e = __fma_rn(-__dmul_rn(x, y0), y0, 1.0);
    const double y = __fma_rn(__dmul_rn(y0, e), __fma_rn(e, 0.375, 0.5), y0);
    const double g = __dmul_rn(x, y);
    return x == 0.0 ? x : __fma_rn(__fma_rn(-g, g, x), __dmul_rn(0.5, y), g);
}

// Powers of T shared by every species' polynomial at one temperature.
struct TPow {
    double T, lnT, tm1, tm2, t2, t3, t4, t5;
    int hi;  // 1 when T >= 1000 K (high-range table)
    int rb;  // table the integration constants b1, b2 come from
};

// q: the handle's EU3D_Q_* set (the b1/b2 defect selects rb)
__device__ __forceinline__ TPow tpow(double T, unsigned q)
{
    TPow p;
    p.T = T;
    p.lnT = log(T);
    p.tm1 = 1.0 / T;
    p.tm2 = p.tm1 * p.tm1;
    p.t2 = T * T;
    p.t3 = p.t2 * T;
    p.t4 = p.t2 * p.t2;
    p.t5 = p.t4 * T;
    p.hi = !(T < 1000.0);
    p.rb = (q & EU3D_Q_THERMO_B12_LOW) ? 0 : p.hi;
    return p;
}

// Cp/R, Reaction::GetCpi bracket (src/Reaction.cpp:893-904)
__device__ __forceinline__ double cp_r(int s, const TPow &p)
{
    const int r = p.hi;
    return cM.c[r][0][s] * p.tm2 + cM.c[r][1][s] * p.tm1 + cM.c[r][2][s] + cM.c[r][3][s] * p.T +
           cM.c[r][4][s] * p.t2 + cM.c[r][5][s] * p.t3 + cM.c[r][6][s] * p.t4;
}

// H/R, Reaction::GetHi bracket (src/Reaction.cpp:916-926); the b1 quirk
// takes the integration constant from the low range above 1000 K.
__device__ __forceinline__ double h_r(int s, const TPow &p)
{
    const int r = p.hi, rb = p.rb;
    return -cM.c[r][0][s] * p.tm1 + cM.c[r][1][s] * p.lnT + cM.c[r][2][s] * p.T + cM.c[r][3][s] * p.t2 * 0.5 +
           cM.c[r][4][s] * p.t3 * (1.0 / 3.0) + cM.c[r][5][s] * p.t4 * 0.25 + cM.c[r][6][s] * p.t5 * 0.2 +
           cM.c[rb][7][s];
}

// S/R, Reaction::GetSi bracket (src/Reaction.cpp:938-948)
__device__ __forceinline__ double s_r(int s, const TPow &p)
{
    const int r = p.hi, rb = p.rb;
    return -cM.c[r][0][s] * p.tm2 * 0.5 - cM.c[r][1][s] * p.tm1 + cM.c[r][2][s] * p.lnT + cM.c[r][3][s] * p.T +
           cM.c[r][4][s] * p.t2 * 0.5 + cM.c[r][5][s] * p.t3 * (1.0 / 3.0) + cM.c[r][6][s] * p.t4 * 0.25 +
           cM.c[rb][8][s];
}

template <class P>
struct PrimPtr {
    P *p;           // NPRIM fields
    long long fs;
    __device__ __forceinline__ P &operator()(int f, long long c) const { return p[f * fs + c]; }
};

}  // namespace eu3d
