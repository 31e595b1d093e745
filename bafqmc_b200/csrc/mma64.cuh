// FP64 matrix products on the tensor pipe (mma.sync m8n8k4 f64; tcgen05 has no
// FP64 kind) for the classes whose operands a CTA reads in place.
//
// One mma does 256 FMAs from one double of A, one of B and two of C per lane, so
// a product needs an eighth of the instructions and about a third of the
// shared-memory loads of per-thread register tiles.  On B200 the pipe takes one
// m8n8k4 per 16 cycles and scheduler (64 FMA/clk/SM, the DFMA rate), with 26
// cycles of latency against 4 x 8.5 for the same four dependent DFMAs: three
// accumulators a warp and two warps a scheduler fill it.  The slice products of
// one sweep against register tiles of DFMAs, M cycles per chain: 64 sites,
// L = 40 (operand R in L2) 10.1 -> 4.3; 6x6 Nambu block, L = 40 14.4 -> 5.4;
// 36 sites, L = 160, two CTAs on the SM 6.6 -> 5.2; 16 sites, L = 80 1.03 -> 0.64.
#pragma once
#include "cplx.cuh"

DEVI void mma_f64(double& c0, double& c1, double a, double b) {
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
        : "+d"(c0), "+d"(c1)
        : "d"(a), "d"(b));
}

// Strided operand view: element (r, c) = p[r*sr + c*sc], optionally conjugated.
// A transposed view swaps the strides.  p may point to shared or global memory.
struct MatOp {
    const cplx* p;
    int sr, sc;
    int cj;
    DEVI cplx at(int r, int c) const {
        cplx v = p[(long)r * sr + (long)c * sc];
        return cj ? cconj(v) : v;
    }
};
DEVI MatOp op_n(const cplx* p, int ld) { return MatOp{p, ld, 1, 0}; }
DEVI MatOp op_c(const cplx* p, int ld) { return MatOp{p, 1, ld, 1}; }   // conjugate transpose

enum { TRI_NONE = 0, TRI_A_UPPER = 1, TRI_B_LOWER_FROM_C = 2 };

// Pointers of the classes whose matrices are all in shared memory: the products
// below then compile to ld.shared instead of generic loads.
template <bool SH>
DEVI void assume_shared(const void* p) {
    if constexpr (SH) __builtin_assume(__isShared(p));
}

// C = A B (n x n, C row-major with leading dimension ld, may alias A or B: results
// wait in registers across a barrier).  A warp owns groups of RT x CT tiles of
// 8 x 8 real elements and walks them in RND rounds (RND * warps >= groups).
//   PROD_CC    complex x complex.  Real columns of C are interleaved (re, im of a
//              complex column), and four complex k give two mma steps: the real
//              parts of A against (Re B, Im B), the imaginary parts against
//              (-Im B, Re B); one 16-byte load per lane and operand feeds both.
//   PROD_REAL_R  complex A x real B (doubles, leading dimension ld): real rows of
//              C are interleaved, one mma per four k.
//   PROD_REAL_L  real A x complex B, interleaved columns.
// tri: TRI_A_UPPER takes A(r, k) = 0 for k < r (ZTRMM 'L','U','N'),
// TRI_B_LOWER_FROM_C B(k, c) = 0 for k < c (ZTRMM 'R','U','C'); the k range that a
// tile does not need is skipped.
enum { PROD_CC = 0, PROD_REAL_R = 1, PROD_REAL_L = 2 };

template <int RT, int CT, int RND, int KIND, bool SH>
DEVI void prod_mma(int n, int ld, cplx* C, MatOp A, MatOp B, const double* R, int tri) {
    constexpr int RSH = KIND == PROD_REAL_R ? 2 : 3;   // log2 of the matrix rows of a tile
    constexpr int CSH = KIND == PROD_REAL_R ? 3 : 2;   // log2 of the matrix columns of a tile
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int l4 = lane & 3, part = (lane >> 2) & 1;
    const int nrt = (n + (1 << RSH) - 1) >> RSH, nct = (n + (1 << CSH) - 1) >> CSH;
    const int gr = (nrt + RT - 1) / RT, gc = (nct + CT - 1) / CT, ng = gr * gc;
    assume_shared<SH>(C);
    if (KIND != PROD_REAL_L) assume_shared<SH>(A.p);
    if (KIND != PROD_REAL_R) assume_shared<SH>(B.p);
    if (KIND != PROD_CC) assume_shared<SH>(R);
    double acc[RND][RT][CT][2];
#pragma unroll
    for (int q = 0; q < RND; ++q) {
        const int g = warp + q * nw;
#pragma unroll
        for (int i = 0; i < RT; ++i)
#pragma unroll
            for (int j = 0; j < CT; ++j) acc[q][i][j][0] = acc[q][i][j][1] = 0.0;
        if (g >= ng) continue;
        const int rt0 = (g / gc) * RT, ct0 = (g % gc) * CT;
        int row[RT], col[CT];
#pragma unroll
        for (int i = 0; i < RT; ++i)
            row[i] = min(((rt0 + i) << RSH) + (KIND == PROD_REAL_R ? lane >> 3 : lane >> 2), n - 1);
#pragma unroll
        for (int j = 0; j < CT; ++j)
            col[j] = min(((ct0 + j) << CSH) + (KIND == PROD_REAL_R ? lane >> 2 : lane >> 3), n - 1);
        int k0 = 0;
        if (KIND == PROD_CC && tri == TRI_A_UPPER) k0 = (rt0 << RSH) & ~3;
        if (KIND == PROD_CC && tri == TRI_B_LOWER_FROM_C) k0 = (ct0 << CSH) & ~3;
#pragma unroll 2
        for (; k0 < n; k0 += 4) {
            const int k = k0 + l4, kk = min(k, n - 1);
            if constexpr (KIND == PROD_CC) {
                cplx a[RT], b[CT];
#pragma unroll
                for (int i = 0; i < RT; ++i) {
                    a[i] = A.p[row[i] * A.sr + kk * A.sc];
                    if (k >= n || (tri == TRI_A_UPPER && k < row[i])) a[i] = cmk(0.0, 0.0);
                    if (A.cj) a[i].y = -a[i].y;
                }
#pragma unroll
                for (int j = 0; j < CT; ++j) {
                    b[j] = B.p[kk * B.sr + col[j] * B.sc];
                    if (tri == TRI_B_LOWER_FROM_C && k < col[j]) b[j] = cmk(0.0, 0.0);
                    if (B.cj) b[j].y = -b[j].y;
                    // this lane's real column: the real part (part 0) or the imaginary part of the complex one
                    b[j] = part ? cmk(b[j].y, b[j].x) : cmk(b[j].x, -b[j].y);
                }
#pragma unroll
                for (int i = 0; i < RT; ++i)
#pragma unroll
                    for (int j = 0; j < CT; ++j) mma_f64(acc[q][i][j][0], acc[q][i][j][1], a[i].x, b[j].x);
#pragma unroll
                for (int i = 0; i < RT; ++i)
#pragma unroll
                    for (int j = 0; j < CT; ++j) mma_f64(acc[q][i][j][0], acc[q][i][j][1], a[i].y, b[j].y);
            } else {
                double a[RT], b[CT];
#pragma unroll
                for (int i = 0; i < RT; ++i) {
                    a[i] = KIND == PROD_REAL_R ? reinterpret_cast<const double*>(A.p)[2 * (row[i] * ld + kk) + part]
                                               : R[row[i] * ld + kk];
                    if (k >= n) a[i] = 0.0;
                }
#pragma unroll
                for (int j = 0; j < CT; ++j)
                    b[j] = KIND == PROD_REAL_R ? R[kk * ld + col[j]]
                                               : reinterpret_cast<const double*>(B.p)[2 * (kk * ld + col[j]) + part];
#pragma unroll
                for (int i = 0; i < RT; ++i)
#pragma unroll
                    for (int j = 0; j < CT; ++j) mma_f64(acc[q][i][j][0], acc[q][i][j][1], a[i], b[j]);
            }
        }
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < RND; ++q) {
        const int g = warp + q * nw;
        if (g >= ng) continue;
        const int rt0 = (g / gc) * RT, ct0 = (g % gc) * CT;
#pragma unroll
        for (int i = 0; i < RT; ++i)
#pragma unroll
            for (int j = 0; j < CT; ++j) {
                const double v0 = acc[q][i][j][0], v1 = acc[q][i][j][1];
                if constexpr (KIND == PROD_REAL_R) {
                    // lanes of the two parts of a row trade one value, so that each stores a whole element
                    const double o = __shfl_xor_sync(0xffffffffu, part ? v0 : v1, 4);
                    const int r = ((rt0 + i) << 2) + (lane >> 3), c = ((ct0 + j) << 3) + 2 * l4 + part;
                    if (r < n && c < n) C[r * ld + c] = part ? cmk(o, v1) : cmk(v0, o);
                } else {
                    const int r = ((rt0 + i) << 3) + (lane >> 2), c = ((ct0 + j) << 2) + l4;
                    if (r < n && c < n) C[r * ld + c] = cmk(v0, v1);
                }
            }
    }
    __syncthreads();
}
