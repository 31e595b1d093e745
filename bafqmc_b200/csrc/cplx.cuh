// Complex FP64 helpers and CTA-level reductions for the BAFQMC sweep kernels.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#define DEVI __device__ __forceinline__

typedef double2 cplx;

DEVI cplx cmk(double r, double i) { return make_double2(r, i); }
DEVI cplx cadd(cplx a, cplx b) { return cmk(a.x + b.x, a.y + b.y); }
DEVI cplx csub(cplx a, cplx b) { return cmk(a.x - b.x, a.y - b.y); }
DEVI cplx cmul(cplx a, cplx b) { return cmk(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }
// a * conj(b)
DEVI cplx cmulcj(cplx a, cplx b) { return cmk(a.x * b.x + a.y * b.y, a.y * b.x - a.x * b.y); }
DEVI cplx cconj(cplx a) { return cmk(a.x, -a.y); }
DEVI cplx cscale(cplx a, double s) { return cmk(a.x * s, a.y * s); }
// acc + a*b
DEVI cplx cfma(cplx a, cplx b, cplx acc) {
    acc.x = fma(a.x, b.x, acc.x);
    acc.x = fma(-a.y, b.y, acc.x);
    acc.y = fma(a.x, b.y, acc.y);
    acc.y = fma(a.y, b.x, acc.y);
    return acc;
}
// acc + conj(a)*b
DEVI cplx cfmacj(cplx a, cplx b, cplx acc) {
    acc.x = fma(a.x, b.x, acc.x);
    acc.x = fma(a.y, b.y, acc.x);
    acc.y = fma(a.x, b.y, acc.y);
    acc.y = fma(-a.y, b.x, acc.y);
    return acc;
}
DEVI double cabs2(cplx a) { return a.x * a.x + a.y * a.y; }
DEVI double cabsv(cplx a) { return hypot(a.x, a.y); }
// Smith's algorithm for a / b.
DEVI cplx cdiv(cplx a, cplx b) {
    if (fabs(b.x) >= fabs(b.y)) {
        double r = b.y / b.x, den = b.x + b.y * r;
        return cmk((a.x + a.y * r) / den, (a.y - a.x * r) / den);
    } else {
        double r = b.x / b.y, den = b.y + b.x * r;
        return cmk((a.x * r + a.y) / den, (a.y * r - a.x) / den);
    }
}
// 1 / x for the serial chains: the approximate reciprocal (measured within 1e-6) and
// one step of Householder's method of cubic order, y (1 + e + e^2) with e = 1 - x y
// (within 1.01 ulp of 1.0 / x over 2^-100 .. 2^100, measured).  No branch: the
// compiler's division ends a basic block, and nothing is scheduled across it.
// x = 0 and infinite x give NaN.
DEVI double rcp_fast(double x) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x, y, 1.0);
    return fma(y, fma(e, e, e), y);
}
// 1 / sqrt(x) likewise: the approximation and the same method's cubic step
// y (1 + e / 2 + 3 e^2 / 8), e = 1 - x y^2, for normal x > 0 (within 1.27 * 2^-53 relative
// of the exact value over 2^-200 .. 2^200, measured; the reciprocal within 1.01 * 2^-53).
DEVI double rsqrt_fast(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x * y, y, 1.0);
    return fma(y, e * fma(0.375, e, 0.5), y);
}
// exp(z) for complex z
DEVI cplx cexpz(cplx z) {
    double s, c;
    sincos(z.y, &s, &c);
    double e = exp(z.x);
    return cmk(e * c, e * s);
}

// A value that every lane of the warp holds, in a form the compiler takes as uniform.
// Shuffles and mma under a branch or in a loop whose condition it cannot prove uniform
// (a value from memory, threadIdx.x >> 5, a call's argument) are each preceded by a
// warp synchronisation.
DEVI int uni(int v) { return __shfl_sync(0xffffffffu, v, 0); }
DEVI int warp_index() { return uni((int)threadIdx.x >> 5); }

// e / n by one multiplication, for loops over matrix elements (an integer division by a
// runtime n costs about 40 instructions): q = umulhi(e, m), m = floor((2^32 - 1) / n) + 1,
// exact for e n < 2^32 and n > 1 (and for e = 0).
DEVI uint32_t div_magic(int n) { return 0xffffffffu / (uint32_t)n + 1u; }
DEVI int div_by(int e, uint32_t m) { return (int)__umulhi((uint32_t)e, m); }

DEVI double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// dst[k] += sum over the warp of v[k], k < 16, without a barrier: each exchange halves the
// values a lane still holds (16 shuffles of a double against 80 for 16 separate sums).
// dst belongs to the warp.
DEVI void warp_add16(double (&v)[16], double* dst) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int h = 8; h > 0; h >>= 1) {   // partner 2h lanes away
        const bool up = (lane & (2 * h)) != 0;
#pragma unroll
        for (int k = 0; k < h; ++k) {
            const double send = up ? v[k] : v[k + h], keep = up ? v[k + h] : v[k];
            v[k] = keep + __shfl_xor_sync(0xffffffffu, send, 2 * h);
        }
    }
    v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
    if (!(lane & 1)) dst[lane >> 1] += v[0];
}

// Block-wide sum of NV values; result valid in every thread. scratch holds
// NV * (blockDim.x/32) doubles. Contains two __syncthreads.
template <int NV>
DEVI void block_sum(double (&v)[NV], double* scratch) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
    for (int k = 0; k < NV; ++k) v[k] = warp_sum(v[k]);
    if (lane == 0) {
#pragma unroll
        for (int k = 0; k < NV; ++k) scratch[k * nw + wid] = v[k];
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        double s = 0.0;
        for (int w = 0; w < nw; ++w) s += scratch[k * nw + w];
        v[k] = s;
    }
    __syncthreads();
}
