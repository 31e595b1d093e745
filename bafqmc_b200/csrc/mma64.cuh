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
// L = 40 (operand R in L2) 10.1 -> 4.2; 6x6 Nambu block, L = 40 14.4 -> 6.2;
// 36 sites, L = 160, two CTAs on the SM 6.6 -> 5.2; 16 sites, L = 80 1.03 -> 0.7.
#pragma once
#include <type_traits>

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

DEVI MatOp op_h(MatOp m) { return MatOp{m.p, m.sc, m.sr, m.cj ? 0 : 1}; }                 // of a view

enum { TRI_NONE = 0, TRI_A_UPPER = 1, TRI_B_LOWER_FROM_C = 2 };

// Pointers of the classes whose matrices are all in shared memory: the products
// below then compile to ld.shared instead of generic loads.
template <bool SH>
DEVI void assume_shared(const void* p) {
    if constexpr (SH) __builtin_assume(__isShared(p));
}

// Which matrix rows and columns a tile's eight take.  Matrices have an odd leading
// dimension (in 16-byte elements), so that pairing index i with i + 4 puts the two rows
// of a quarter-warp's 16-byte accesses 64 bytes apart modulo 128: fragments of either
// operand, transposed or not, and the stores of C fall in distinct banks.  Real operands
// (8 bytes) have a leading dimension of 4 or 12 modulo 16 and plain order.
DEVI int tile_at(int t, int i) { return 8 * t + (i >> 1) + 4 * (i & 1); }
// leading dimension (doubles) of the real e^{-+dtau K} of a class
__host__ __device__ constexpr int real_ld(int nmax) { return (nmax + 3) / 8 * 8 + 4; }
__host__ __device__ constexpr int mma_tiles(int n) { return ((n + 7) / 8) * ((n + 7) / 8); }

// C = A B (n x n, C row-major with leading dimension ld, may alias A or B: results
// wait in registers across a barrier).  Tiles of C are 8 x 8 complex elements, real and
// imaginary parts in accumulators of their own, so that one 16-byte load of a complex
// operand's element feeds two mma per tile (four if both are complex).  Shared memory
// moves 128 bytes a cycle: a step of four k then costs 6 (real kinds) or 8 cycles of it
// against 8 or 16 of the tensor pipe; with the parts as rows or columns of real tiles,
// an 8-byte load each, the loads took longer than the mma.  A warp takes tiles
// warp, warp + warps, ... (RND of them at most), NB at a time.
//   PROD_CC      complex A x complex B
//   PROD_REAL_R  complex x real (X <- X R, R of leading dimension ldr)
//   PROD_REAL_L  real x complex (X <- R X)
// The real kinds may take a second matrix X2 <- X2 R or R X2 in the same call (its tiles
// follow).  tri: TRI_A_UPPER takes A(r, k) = 0 for k < r (ZTRMM 'L','U','N'),
// TRI_B_LOWER_FROM_C B(k, c) = 0 for k < c (ZTRMM 'R','U','C'); the k range that no tile
// of a batch needs is skipped.
enum { PROD_CC = 0, PROD_REAL_R = 1, PROD_REAL_L = 2 };

template <int RND, int NB, int KIND, bool SH>
DEVI void prod_mma(int n, int ld, cplx* C, MatOp A, MatOp B, const double* R, int ldr, int tri, cplx* X2 = nullptr) {
    static_assert(RND % NB == 0, "whole batches");
    n = uni(n);
    tri = uni(tri);
    const int lane = threadIdx.x & 31, warp = warp_index(), nw = blockDim.x >> 5;
    const int l4 = lane & 3, l8 = lane >> 2;
    const int n8 = (n + 7) >> 3, nt1 = n8 * n8;
    const uint32_t m8 = div_magic(n8);
    const int nt = KIND != PROD_CC && uni(X2 != nullptr) ? 2 * nt1 : nt1;
    assume_shared<SH>(C);
    if (KIND == PROD_CC) assume_shared<SH>(A.p);
    if (KIND == PROD_CC) assume_shared<SH>(B.p);
    if (KIND != PROD_CC) assume_shared<SH>(R);
    const int xoff = KIND != PROD_CC ? (int)(X2 - C) : 0;   // the second matrix from the first (both in one space)
    double re[RND][2], im[RND][2];
#pragma unroll
    for (int q = 0; q < RND; ++q) re[q][0] = re[q][1] = im[q][0] = im[q][1] = 0.0;
    // matrix row and column of this lane's fragments in tile t, clamped
    const auto place = [&](int t, int& off, int& rt, int& ct) {
        off = 0;
        if (KIND != PROD_CC && t >= nt1) {
            t -= nt1;
            off = xoff;
        }
        rt = n8 == 1 ? 0 : div_by(t, m8);
        ct = t - rt * n8;
    };
#pragma unroll
    for (int q0 = 0; q0 < RND; q0 += NB) {
        if (warp + q0 * nw >= nt) break;
        const cplx *ap[NB], *bp[NB];   // this lane's elements at k = l4 (the real operand's as ra, rb)
        const double *ra[NB], *rb[NB];
        int row[NB], col[NB], k0 = 0;
#pragma unroll
        for (int q = 0; q < NB; ++q) {
            int off, rt, ct;
            place(min(warp + (q0 + q) * nw, nt - 1), off, rt, ct);
            row[q] = min(KIND == PROD_REAL_L ? 8 * rt + l8 : tile_at(rt, l8), n - 1);
            col[q] = min(KIND == PROD_REAL_R ? 8 * ct + l8 : tile_at(ct, l8), n - 1);
            if (KIND == PROD_CC) {
                ap[q] = A.p + row[q] * A.sr;
                bp[q] = B.p + col[q] * B.sc;
                const int kt = tri == TRI_A_UPPER ? 8 * rt : (tri == TRI_B_LOWER_FROM_C ? 8 * ct : 0);
                k0 = q == 0 ? kt : min(k0, kt);
            } else if (KIND == PROD_REAL_R) {
                ap[q] = C + off + row[q] * ld;
                rb[q] = R + col[q];
            } else {
                ra[q] = R + row[q] * ldr;
                bp[q] = C + off + col[q];
            }
        }
        const int da = KIND == PROD_CC ? A.sc : 1, db = KIND == PROD_CC ? B.sr : (KIND == PROD_REAL_R ? ldr : ld);
#pragma unroll
        for (int q = 0; q < NB; ++q) {
            if (KIND != PROD_REAL_L) ap[q] += (k0 + l4) * da;
            else ra[q] += (k0 + l4) * da;
            if (KIND != PROD_REAL_R) bp[q] += (k0 + l4) * db;
            else rb[q] += (k0 + l4) * db;
        }
        const double sa = KIND == PROD_CC && A.cj ? -1.0 : 1.0, sb = KIND == PROD_CC && B.cj ? -1.0 : 1.0;
        // one step of four k on the elements under the pointers; LAST: k past n is clamped and zero in A
        const auto step = [&](int k, auto last) {
            constexpr bool LAST = decltype(last)::value;
            const int back = LAST ? max(k - (n - 1), 0) : 0;   // how far this lane's k is past the end
            [[maybe_unused]] cplx ua[NB], ub[NB];
            [[maybe_unused]] double va[NB], vb[NB];
#pragma unroll
            for (int q = 0; q < NB; ++q) {
                if constexpr (KIND == PROD_REAL_L) {
                    va[q] = ra[q][-back * da];
                    if (LAST && back) va[q] = 0.0;
                } else {
                    ua[q] = ap[q][-back * da];
                    const bool z = (LAST && back) || (KIND == PROD_CC && tri == TRI_A_UPPER && k < row[q]);
                    ua[q] = cmk(z ? 0.0 : ua[q].x, z ? 0.0 : ua[q].y);
                    if (KIND == PROD_CC) ua[q].y *= sa;
                }
                if constexpr (KIND == PROD_REAL_R) {
                    vb[q] = rb[q][-back * db];
                } else {
                    ub[q] = bp[q][-back * db];
                    if (KIND == PROD_CC) {
                        const bool z = tri == TRI_B_LOWER_FROM_C && k < col[q];
                        ub[q] = cmk(z ? 0.0 : ub[q].x, z ? 0.0 : sb * ub[q].y);
                    }
                }
            }
#pragma unroll
            for (int q = 0; q < NB; ++q) {
                const int s = q0 + q;
                if constexpr (KIND == PROD_CC) {
                    mma_f64(re[s][0], re[s][1], ua[q].x, ub[q].x);
                    mma_f64(im[s][0], im[s][1], ua[q].x, ub[q].y);
                } else if constexpr (KIND == PROD_REAL_R) {
                    mma_f64(re[s][0], re[s][1], ua[q].x, vb[q]);
                    mma_f64(im[s][0], im[s][1], ua[q].y, vb[q]);
                } else {
                    mma_f64(re[s][0], re[s][1], va[q], ub[q].x);
                    mma_f64(im[s][0], im[s][1], va[q], ub[q].y);
                }
            }
            if constexpr (KIND == PROD_CC) {
#pragma unroll
                for (int q = 0; q < NB; ++q) {
                    mma_f64(re[q0 + q][0], re[q0 + q][1], -ua[q].y, ub[q].y);
                    mma_f64(im[q0 + q][0], im[q0 + q][1], ua[q].y, ub[q].x);
                }
            }
#pragma unroll
            for (int q = 0; q < NB; ++q) {
                if (KIND != PROD_REAL_L) ap[q] += 4 * da;
                else ra[q] += 4 * da;
                if (KIND != PROD_REAL_R) bp[q] += 4 * db;
                else rb[q] += 4 * db;
            }
        };
#pragma unroll 2
        for (; k0 + 4 <= n; k0 += 4) step(k0 + l4, std::false_type{});
        if (k0 < n) step(k0 + l4, std::true_type{});
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < RND; ++q) {
        const int t = warp + q * nw;
        if (t >= nt) break;
        int off, rt, ct;
        place(t, off, rt, ct);
        const int r = KIND == PROD_REAL_L ? 8 * rt + l8 : tile_at(rt, l8);
        cplx* D = C + off + r * ld;
        if constexpr (KIND == PROD_REAL_R) {
            // plain columns 2 l4 and 2 l4 + 1: the rows of odd l8 store the second one first, in other banks
            const int o = l8 & 1, c = 8 * ct + 2 * l4;
            const cplx v0 = cmk(re[q][0], im[q][0]), v1 = cmk(re[q][1], im[q][1]);
            const cplx w0 = cmk(o ? v1.x : v0.x, o ? v1.y : v0.y), w1 = cmk(o ? v0.x : v1.x, o ? v0.y : v1.y);
            if (r < n && c + o < n) D[c + o] = w0;
            if (r < n && c + 1 - o < n) D[c + 1 - o] = w1;
        } else {
            const int c = 8 * ct + l4;
            if (r < n && c < n) D[c] = cmk(re[q][0], im[q][0]);
            if (r < n && c + 4 < n) D[c + 4] = cmk(re[q][1], im[q][1]);
        }
    }
    __syncthreads();
}
