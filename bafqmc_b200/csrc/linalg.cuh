// CTA-level dense complex FP64 linear algebra on matrices resident in shared
// memory (row-major n x n with leading dimension ld; the sweep kernels use an
// odd ld so that a column walk touches every shared-memory bank group).  Every routine is called by all
// threads of the block and returns with the block synchronised.
//
// These restate the LAPACK/BLAS operations the reference sweep calls
// (src/number_conserving/src/stabilization.f90:41-190 and
// src/common/mymats.f90:20-29): ZGEMM, ZTRMM, ZGEQP3 (unblocked ZLAQP2 path,
// which LAPACK takes for the matrix sizes here), ZUNGQR, ZUNMQR, ZTRSM,
// ZLAPMR/ZLAPMT.  They are written for the sweep's sizes (n <= 64): one CTA
// owns one matrix.  The reflector and triangular-solve sequences run on 8-lane
// segments that each keep their columns (or rows) of the operand in registers
// for the whole sequence and reduce with shuffles, so no step needs a block
// barrier; divisions are replaced by precomputed reciprocals.
#pragma once
#include "mma64.cuh"

// Factorisation routines are kept out of line: they run once per wrap, and
// inlining them into the sweep kernel costs registers on the per-slice path.
#define COLD static __device__ __noinline__

// C = A * B for n x n operands (C may alias A or B), the complex product of
// prod_mma out of line.  tri as there.
template <int RND, int NB, bool SH>
COLD void gemm_rs(int n, int ld, cplx* C, MatOp A, MatOp B, int tri = TRI_NONE) {
    prod_mma<RND, NB, PROD_CC, SH>(n, ld, C, A, B, nullptr, 0, tri);
}

// The slice propagators e^{-+dtau K} are real (real hopping, chemical
// potential and pairing amplitude), so the per-slice products X <- X R or R X (and
// X2 alike) are complex x real.  Real operands are stored as doubles with leading
// dimension ldr (real_ld of the class).
template <int RND, int NB, bool RIGHT_REAL, bool SH>
COLD void gemm_smem_real(int n, int ld, int ldr, cplx* X, const double* R, cplx* X2 = nullptr) {
    prod_mma<RND, NB, RIGHT_REAL ? PROD_REAL_R : PROD_REAL_L, SH>(n, ld, X, MatOp{}, MatOp{}, R, ldr, TRI_NONE, X2);
}

// dst = op(src) elementwise copy for an n x n matrix (dst must not alias src
// unless op is the identity view).
COLD void copy_op(int n, int ld, cplx* dst, MatOp src) {
    const uint32_t dm = div_magic(n);
    for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
        const int r = div_by(e, dm), c = e - r * n;
        dst[r * ld + c] = src.at(r, c);
    }
    __syncthreads();
}

// In-place conjugate transpose via register staging; MAXE >= ceil(n*n/blockDim).
template <int MAXE>
COLD void conj_transpose_inplace(int n, int ld, cplx* A) {
    const uint32_t dm = div_magic(n);
    cplx v[MAXE];
#pragma unroll
    for (int k = 0; k < MAXE; ++k) {
        const int e = threadIdx.x + k * blockDim.x;
        if (e < n * n) {
            const int r = div_by(e, dm), c = e - r * n;
            v[k] = cconj(A[c * ld + r]);
        }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < MAXE; ++k) {
        const int e = threadIdx.x + k * blockDim.x;
        if (e < n * n) {
            const int r = div_by(e, dm), c = e - r * n;
            A[r * ld + c] = v[k];
        }
    }
    __syncthreads();
}

// Segmented (8-lane) reductions used by the column-parallel reflector passes.
// The mask covers only the calling thread's aligned 8-lane segment, so the
// segments of one warp may run different trip counts.
DEVI unsigned seg8_mask() { return 0xffu << (threadIdx.x & 24); }
DEVI double seg8_sum(double v) {
    const unsigned m = seg8_mask();
    v += __shfl_xor_sync(m, v, 4);
    v += __shfl_xor_sync(m, v, 2);
    v += __shfl_xor_sync(m, v, 1);
    return v;
}
DEVI double seg8_max(double v) {
    const unsigned m = seg8_mask();
    v = fmax(v, __shfl_xor_sync(m, v, 4));
    v = fmax(v, __shfl_xor_sync(m, v, 2));
    v = fmax(v, __shfl_xor_sync(m, v, 1));
    return v;
}

// Overflow-safe 2-norm of column j, rows [r0, n), computed by one 8-lane segment.
DEVI double seg8_colnorm(int n, int ld, const cplx* A, int j, int r0, int lane8) {
    double m = 0.0;
    for (int r = r0 + lane8; r < n; r += 8) m = fmax(m, fmax(fabs(A[r * ld + j].x), fabs(A[r * ld + j].y)));
    m = seg8_max(m);
    if (m == 0.0) return 0.0;
    double s = 0.0;
    for (int r = r0 + lane8; r < n; r += 8) {
        double a = A[r * ld + j].x / m, b = A[r * ld + j].y / m;
        s += a * a + b * b;
    }
    s = seg8_sum(s);
    return m * sqrt(s);
}

// Sum of squares of column j, rows r0..n-1, by one 8-lane segment.
DEVI double seg8_sumsq_col(int n, int ld, const cplx* A, int j, int r0, int lane8) {
    double ss = 0.0;
    for (int r = r0 + lane8; r < n; r += 8) {
        const cplx a = A[r * ld + j];
        ss = fma(a.x, a.x, fma(a.y, a.y, ss));
    }
    return seg8_sum(ss);
}

DEVI bool sumsq_unsafe(double ss) { return !(ss <= 1.0e300) || (ss != 0.0 && ss < 1.0e-290); }

// 2-norm of column j rows r0..n-1 (one segment); scaled only when the plain sum
// of squares would over- or underflow.
DEVI double seg8_norm(int n, int ld, const cplx* A, int j, int r0, int lane8) {
    const double ss = seg8_sumsq_col(n, ld, A, j, r0, lane8);
    if (!sumsq_unsafe(ss)) return sqrt(ss);
    return seg8_colnorm(n, ld, A, j, r0, lane8);
}

// Shared scratch for the factorisations (lives in shared memory, size ~ 6n).
struct QRScratch {
    cplx* tau;      // n
    int* piv;       // n   (0-based: (A P)[:, j] = A[:, piv[j]])
    int* ipiv;      // n   inverse permutation
    double* vn1;    // n
    double* vn2;    // n
    double* d;      // n   |R_ii|
    cplx* bcast;    // 4   broadcast slots
    int* ibcast;    // 4
    // qr_columns only, in buffers of the local update
    cplx* vb;         // n   the pivot column
    cplx* scl;        // n   1 / d of the reflectors
    long long* keys;  // n   remaining norms of the columns as ordered integers
    double* bet;      // n   signed diagonal of R
    int* ex;          // n   scale exponents of the columns
};

// Scale 2^e of a column by its largest entry, as an exponent: 0 for a zero or non-finite column.
DEVI int scale_exponent(double m) {
    const int e = (int)((__double_as_longlong(m) >> 52) & 0x7ff);
    return (e == 0 || e == 0x7ff) ? 0 : e - 1022;
}

// Pivoted QR of A (n x n): (A P) = Q R with ZGEQP3's pivot rule (the column of largest
// remaining norm), then the reference's QDRP_decompose post-step (stabilization.f90:41-67):
// d[i] = |R_ii| and row i of the upper triangle divided by d[i], piv and ipiv.
// AUG: also out <- Q^H in for the n x n view `in` (the identity if in.p is null), carried
// along with the columns of A, so that no pass over the reflectors follows; A's strict
// lower triangle is then not written.  Otherwise A holds the Householder vectors (unit
// leading entry implicit) below R, and s.tau their factors, for form_q and apply_*.
//
// LPC lanes own a column for the whole factorisation, RPL of its rows each in registers
// (RPL * LPC >= n), with the same lanes for a column of `in`; pivoting is by bookkeeping,
// no column moves, and a column is written once, at its place.  Per step the warps that
// own columns (a named barrier, the others wait at the end) choose the pivot from the
// keys in shared memory (redux on their bits), its owner copies it to shared memory, and
// every group forms the reflector for itself: its norm is the sum of squares of the
// column that the previous step's update left (every step computes the remaining norms
// exactly, so ZLAQP2's downdating and its recomputation test are not needed), and the
// product of the unscaled reflector with a column is under way while sqrt and 1/x are.
// Columns are scaled by powers of two on entry (exact, and reflectors act on rows), so
// that no sum of squares over- or underflows whatever D has grown to.
// Rows leave the registers from the top, a block of LPC at a time, so that no step masks
// them; a branch or a select per row cost more than the arithmetic (3500 cycles a step).
// Bound: the chain and the issue of a step on the warps that own columns, 1860 cycles at
// n = 36 with the second matrix (1460 without, 1075 at n = 16); 139 K -> 67 K cycles for the
// factorisation.  The version before kept the matrix in shared memory, reduced over eight
// lanes, downdated the norms and applied the reflectors in a pass of its own: a wrap of a
// 36-site chain took 560 K cycles with that one and takes 270 K.
// The per-thread state of the factorisation: its rows of the column of A and of `in`.
template <int RPL, bool AUG>
struct QrCol {
    cplx a[RPL], c[AUG ? RPL : 1];
    double n2;
    int ex;
    bool live;
};

// The LPC steps of row block kb, with K register rows left (those past n hold zeros).
template <int LPC, int RPL, int K, bool AUG>
DEVI void qr_block(int n, int ld, int kb, int nthr, cplx* A, const QRScratch& s, QrCol<RPL, AUG>& q, cplx* o, int osr,
                   int ocj) {
    constexpr long long kOff = (long long)0x8000000000000000ull;
    const int tid = threadIdx.x, lane = tid & 31, lc = tid % LPC, j = tid / LPC, lj = min(lane, n - 1);
    const bool first = lc == 0 && j < n;
    const auto group_sum = [&](double v) {
#pragma unroll
        for (int d = LPC / 2; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
        return v;
    };
#pragma unroll 1
    for (int li = 0; li < LPC; ++li) {
        const int i = kb * LPC + li, src = (lane & ~(LPC - 1)) + li;
        if (i >= n) break;
        asm volatile("bar.sync 1, %0;" ::"r"(nthr) : "memory");
        // pivot: the largest key, the lowest column of equal ones (every warp for itself)
        long long key = s.keys[lj];
        int bj = lj;
#pragma unroll
        for (int w = 32; w < LPC * RPL; w += 32) {
            const int jq = min(lane + w, n - 1);
            const long long k2 = s.keys[jq];
            bj = k2 > key ? jq : bj;
            key = k2 > key ? k2 : key;
        }
        const int hi = (int)(key >> 32), mh = __reduce_max_sync(0xffffffffu, hi);
        const unsigned lo = hi == mh ? (unsigned)key : 0u, ml = __reduce_max_sync(0xffffffffu, lo);
        const int p = (int)__reduce_min_sync(0xffffffffu, hi == mh && lo == ml ? (unsigned)bj : 0x7fffffffu);
        const bool own = q.live && j == p;
        q.live = q.live && !own;
        const double pn = s.vn1[p];
        if (own) {
#pragma unroll
            for (int k = 0; k < K; ++k) s.vb[lc + LPC * k] = q.a[k];
        }
        // row i leaves the registers
        const cplx ai = cmk(__shfl_sync(0xffffffffu, q.a[0].x, src), __shfl_sync(0xffffffffu, q.a[0].y, src));
        cplx ci = cmk(0.0, 0.0);
        if constexpr (AUG) ci = cmk(__shfl_sync(0xffffffffu, q.c[0].x, src), __shfl_sync(0xffffffffu, q.c[0].y, src));
        const bool at = lc == li;
        q.a[0] = cmk(at ? 0.0 : q.a[0].x, at ? 0.0 : q.a[0].y);
        if constexpr (AUG) q.c[0] = cmk(at ? 0.0 : q.c[0].x, at ? 0.0 : q.c[0].y);
        asm volatile("bar.sync 1, %0;" ::"r"(nthr) : "memory");
        const cplx alpha = s.vb[li];
        // S = sum over rows below i of conj(x) a, in two chains each
        constexpr bool KEEP = K * (AUG ? 3 : 2) <= 20;   // else read again below: the registers are full
        cplx x[KEEP ? K : 1], sa[2], sc[2];
        sa[0] = sa[1] = sc[0] = sc[1] = cmk(0.0, 0.0);
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const cplx xk = s.vb[lc + LPC * k];
            if constexpr (KEEP) x[k] = xk;
            sa[k & 1] = cfmacj(xk, q.a[k], sa[k & 1]);
            if constexpr (AUG) sc[k & 1] = cfmacj(xk, q.c[k], sc[k & 1]);
        }
        // beta = b = -sign(Re alpha) |column|, d = alpha - b, tau = (b - alpha) / b = -d / b (ZLARFG);
        // the unscaled reflector (d, x) takes conj(tau) / |d|^2 = -conj(d) / (b |d|^2)
        const bool zero = !(pn > 1.0e-300);
        const double y = rsqrt_fast(zero ? 1.0 : pn), nrm = pn * y;
        const double b = alpha.x >= 0.0 ? -nrm : nrm;
        const cplx d = cmk(alpha.x - b, alpha.y);
        const double d2 = fma(d.x, d.x, d.y * d.y);
        const double t0 = rcp_fast(b * d2), t = zero ? 0.0 : t0;
        const cplx tq = cmk(d.x * t, -d.y * t);   // minus the factor
        const cplx wa = cfmacj(d, ai, cmk(group_sum(sa[0].x + sa[1].x), group_sum(sa[0].y + sa[1].y)));
        const cplx f = cmul(tq, wa);
        const cplx fa = cmk(q.live ? f.x : 0.0, q.live ? f.y : 0.0);
        cplx fc = cmk(0.0, 0.0);
        if constexpr (AUG)
            fc = cmul(tq, cfmacj(d, ci, cmk(group_sum(sc[0].x + sc[1].x), group_sum(sc[0].y + sc[1].y))));
        double n2[2] = {0.0, 0.0};
        if constexpr (!KEEP) asm volatile("" ::: "memory");   // so that the second reading is one
#pragma unroll
        for (int k = 0; k < K; ++k) {
            cplx xk = x[0];
            if constexpr (KEEP) xk = x[k];
            else xk = s.vb[lc + LPC * k];
            if (k == 0) xk = cmk(at ? 0.0 : xk.x, at ? 0.0 : xk.y);
            q.a[k] = cfma(xk, fa, q.a[k]);
            if constexpr (AUG) q.c[k] = cfma(xk, fc, q.c[k]);
            n2[k & 1] = fma(q.a[k].x, q.a[k].x, fma(q.a[k].y, q.a[k].y, n2[k & 1]));
        }
        q.n2 = group_sum(n2[0] + n2[1]);
        // vb is rewritten after the next barrier only, vn1 and the keys before it
        if (first) {
            const long long kk = (__double_as_longlong(q.n2) >> 2) + ((long long)q.ex << 51);
            s.keys[j] = q.live ? (q.n2 == 0.0 ? kOff + 1 : kk) : kOff;
            s.vn1[j] = q.n2;
            if (q.live) A[i * ld + j] = cfma(d, fa, ai);   // R(i, j), at the column's first place
            if constexpr (AUG) {
                const cplx v = cfma(d, fc, ci);
                o[i * osr] = cmk(v.x, ocj ? -v.y : v.y);
            }
        }
        if (own) {
            if constexpr (!AUG) {
#pragma unroll
                for (int k = 0; k < K; ++k) {
                    const int r = kb * LPC + lc + LPC * k;
                    if (r > i && r < n) A[r * ld + j] = q.a[k];   // below the column's R
                }
            }
            if (lc == 0) {
                const double id2 = zero ? 0.0 : 1.0 / d2;
                s.piv[i] = j;
                s.ipiv[j] = i;
                s.tau[i] = zero ? cmk(0.0, 0.0) : cmk(-d.x * (b * y * y), -d.y * (b * y * y));   // 1 / b = b / |b|^2
                s.bet[i] = zero ? 0.0 : b;
                s.vn2[i] = zero ? __longlong_as_double(0x7ff0000000000000LL) : y;   // 1 / |beta|
                s.scl[i] = cmk(d.x * id2, -d.y * id2);                              // 1 / d
            }
        }
    }
#pragma unroll
    for (int k = 0; k + 1 < K; ++k) {   // the block's rows are done
        q.a[k] = q.a[k + 1];
        if constexpr (AUG) q.c[k] = q.c[k + 1];
    }
    q.a[K - 1] = cmk(0.0, 0.0);
    if constexpr (AUG) q.c[K - 1] = cmk(0.0, 0.0);
}

template <int LPC, int RPL, bool AUG>
COLD void qr_columns(int n, int ld, cplx* A, QRScratch s, MatOp in, MatOp out) {
    n = uni(n);
    const int tid = threadIdx.x, lc = tid % LPC, j = tid / LPC;
    const int nthr = (n * LPC + 31) & ~31;
    if (uni(tid) < nthr) {
        const bool col = j < n;
        const int jc = min(j, n - 1);
        cplx* const o = const_cast<cplx*>(out.p) + jc * out.sc;
        QrCol<RPL, AUG> q;
        double m = 0.0;
#pragma unroll
        for (int k = 0; k < RPL; ++k) {
            const int r = lc + LPC * k, rc = min(r, n - 1);
            const cplx v = A[rc * ld + jc];
            const bool ok = col && r < n;
            q.a[k] = cmk(ok ? v.x : 0.0, ok ? v.y : 0.0);
            m = fmax(m, fmax(fabs(q.a[k].x), fabs(q.a[k].y)));
            if constexpr (AUG) {
                cplx w = cmk(r == j ? 1.0 : 0.0, 0.0);
                if (in.p) {
                    w = in.p[rc * in.sr + jc * in.sc];
                    if (in.cj) w.y = -w.y;
                }
                q.c[k] = cmk(ok ? w.x : 0.0, ok ? w.y : 0.0);
            }
        }
#pragma unroll
        for (int d = LPC / 2; d > 0; d >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, d));
        q.ex = scale_exponent(m);
        const double down = scalbn(1.0, -q.ex);
        q.n2 = 0.0;
#pragma unroll
        for (int k = 0; k < RPL; ++k) {
            q.a[k] = cmk(q.a[k].x * down, q.a[k].y * down);
            q.n2 = fma(q.a[k].x, q.a[k].x, fma(q.a[k].y, q.a[k].y, q.n2));
        }
#pragma unroll
        for (int d = LPC / 2; d > 0; d >>= 1) q.n2 += __shfl_xor_sync(0xffffffffu, q.n2, d);
        q.live = col;
        if (lc == 0 && col) {
            s.keys[j] = q.n2 == 0.0 ? (long long)0x8000000000000001ull : (__double_as_longlong(q.n2) >> 2) + ((long long)q.ex << 51);
            s.vn1[j] = q.n2;
            s.ex[j] = q.ex;
        }
        // row blocks in three stretches, each with the register rows that its first block needs
        constexpr int K2 = (2 * RPL + 2) / 3, K3 = (RPL + 2) / 3;
        const int nb = (n + LPC - 1) / LPC;
        int kb = 0;
        for (; nb - kb > K2; ++kb) qr_block<LPC, RPL, RPL, AUG>(n, ld, kb, nthr, A, s, q, o, out.sr, out.cj);
        for (; nb - kb > K3; ++kb) qr_block<LPC, RPL, K2, AUG>(n, ld, kb, nthr, A, s, q, o, out.sr, out.cj);
        for (; kb < nb; ++kb) qr_block<LPC, RPL, K3, AUG>(n, ld, kb, nthr, A, s, q, o, out.sr, out.cj);
        asm volatile("bar.sync 1, %0;" ::"r"(nthr) : "memory");
        // columns to their places, in pivot order: rows of R divided by |beta| (and scaled back),
        // the reflector below divided by its leading entry
        const int i = s.ipiv[jc];
        const cplx scl = s.scl[i];
        cplx w[RPL];
#pragma unroll
        for (int k = 0; k < RPL; ++k) {
            const int r = min(lc + LPC * k, n - 1), e = q.ex - s.ex[s.piv[r]];
            const cplx v = A[r * ld + jc];
            const double f = s.vn2[r];
            w[k] = r == i ? cmk(s.bet[i] * f, 0.0) : cmk(scalbn(v.x * f, e), scalbn(v.y * f, e));
            if (!AUG && r > i) w[k] = cmul(v, scl);
        }
        asm volatile("bar.sync 1, %0;" ::"r"(nthr) : "memory");
#pragma unroll
        for (int k = 0; k < RPL; ++k) {
            const int r = lc + LPC * k;
            if (col && r < n && (!AUG || r <= i)) A[r * ld + i] = w[k];
        }
    }
    __syncthreads();
    for (int i = tid; i < n; i += blockDim.x) s.d[i] = scalbn(fabs(s.bet[i]), s.ex[s.piv[i]]);
    __syncthreads();
}

// C <- Q^H C (ZUNMQR 'L','C'): each segment holds its columns in registers.
template <int R8, int CPS>
COLD void apply_qh_left(int n, int ld, const cplx* F, const cplx* tau, cplx* C) {
    const int tid = threadIdx.x, lane8 = tid & 7, seg = tid >> 3, nseg = blockDim.x >> 3;
    cplx c[CPS][R8];
#pragma unroll
    for (int q = 0; q < CPS; ++q)
#pragma unroll
        for (int k = 0; k < R8; ++k) {
            const int j = seg + q * nseg, r = lane8 + 8 * k;
            c[q][k] = (j < n && r < n) ? C[r * ld + j] : cmk(0.0, 0.0);
        }
    for (int i = 0; i < n; ++i) {
        const cplx ct = cconj(tau[i]);
        cplx v[R8];
#pragma unroll
        for (int k = 0; k < R8; ++k) {
            const int r = lane8 + 8 * k;
            v[k] = (r == i) ? cmk(1.0, 0.0) : ((r > i && r < n) ? F[r * ld + i] : cmk(0.0, 0.0));
        }
#pragma unroll
        for (int q = 0; q < CPS; ++q) {
            cplx w = cmk(0.0, 0.0);
#pragma unroll
            for (int k = 0; k < R8; ++k) w = cfmacj(v[k], c[q][k], w);
            w.x = seg8_sum(w.x);
            w.y = seg8_sum(w.y);
            const cplx f = cmul(ct, w);
#pragma unroll
            for (int k = 0; k < R8; ++k) c[q][k] = csub(c[q][k], cmul(v[k], f));
        }
    }
#pragma unroll
    for (int q = 0; q < CPS; ++q)
#pragma unroll
        for (int k = 0; k < R8; ++k) {
            const int j = seg + q * nseg, r = lane8 + 8 * k;
            if (j < n && r < n) C[r * ld + j] = c[q][k];
        }
    __syncthreads();
}

// C <- C Q (ZUNMQR 'R','N'): each segment holds its rows in registers.
template <int R8, int CPS>
COLD void apply_q_right(int n, int ld, const cplx* F, const cplx* tau, cplx* C) {
    const int tid = threadIdx.x, lane8 = tid & 7, seg = tid >> 3, nseg = blockDim.x >> 3;
    cplx c[CPS][R8];   // c[q][k] = C[row seg+q*nseg][col lane8+8k]
#pragma unroll
    for (int q = 0; q < CPS; ++q)
#pragma unroll
        for (int k = 0; k < R8; ++k) {
            const int r = seg + q * nseg, col = lane8 + 8 * k;
            c[q][k] = (r < n && col < n) ? C[r * ld + col] : cmk(0.0, 0.0);
        }
    for (int i = 0; i < n; ++i) {
        const cplx t = tau[i];
        cplx v[R8];
#pragma unroll
        for (int k = 0; k < R8; ++k) {
            const int col = lane8 + 8 * k;
            v[k] = (col == i) ? cmk(1.0, 0.0) : ((col > i && col < n) ? F[col * ld + i] : cmk(0.0, 0.0));
        }
#pragma unroll
        for (int q = 0; q < CPS; ++q) {
            cplx w = cmk(0.0, 0.0);
#pragma unroll
            for (int k = 0; k < R8; ++k) w = cfma(c[q][k], v[k], w);
            w.x = seg8_sum(w.x);
            w.y = seg8_sum(w.y);
            const cplx f = cmul(t, w);
#pragma unroll
            for (int k = 0; k < R8; ++k) c[q][k] = csub(c[q][k], cmulcj(f, v[k]));
        }
    }
#pragma unroll
    for (int q = 0; q < CPS; ++q)
#pragma unroll
        for (int k = 0; k < R8; ++k) {
            const int r = seg + q * nseg, col = lane8 + 8 * k;
            if (r < n && col < n) C[r * ld + col] = c[q][k];
        }
    __syncthreads();
}

// Q = H_0 ... H_{n-1} (ZUNGQR), or Q^H with conjT, written to Q (no alias with F).
template <int R8, int CPS>
COLD void form_q(int n, int ld, const cplx* F, const cplx* tau, cplx* Q, bool conjT) {
    const int tid = threadIdx.x, lane8 = tid & 7, seg = tid >> 3, nseg = blockDim.x >> 3;
    cplx c[CPS][R8];
#pragma unroll
    for (int q = 0; q < CPS; ++q)
#pragma unroll
        for (int k = 0; k < R8; ++k) {
            const int j = seg + q * nseg, r = lane8 + 8 * k;
            c[q][k] = cmk((r == j) ? 1.0 : 0.0, 0.0);
        }
    for (int i = n - 1; i >= 0; --i) {
        const cplx t = tau[i];
        cplx v[R8];
#pragma unroll
        for (int k = 0; k < R8; ++k) {
            const int r = lane8 + 8 * k;
            v[k] = (r == i) ? cmk(1.0, 0.0) : ((r > i && r < n) ? F[r * ld + i] : cmk(0.0, 0.0));
        }
#pragma unroll
        for (int q = 0; q < CPS; ++q) {
            const int j = seg + q * nseg;
            if (j < i) continue;   // columns left of i are untouched by H_i (ZUNG2R), uniform per segment
            cplx w = cmk(0.0, 0.0);
#pragma unroll
            for (int k = 0; k < R8; ++k) w = cfmacj(v[k], c[q][k], w);
            w.x = seg8_sum(w.x);
            w.y = seg8_sum(w.y);
            const cplx f = cmul(t, w);
#pragma unroll
            for (int k = 0; k < R8; ++k) c[q][k] = csub(c[q][k], cmul(v[k], f));
        }
    }
#pragma unroll
    for (int q = 0; q < CPS; ++q)
#pragma unroll
        for (int k = 0; k < R8; ++k) {
            const int j = seg + q * nseg, r = lane8 + 8 * k;
            if (j < n && r < n) {
                if (conjT) Q[j * ld + r] = cconj(c[q][k]);
                else Q[r * ld + j] = c[q][k];
            }
        }
    __syncthreads();
}

// Inverses of the diagonal of the upper triangle of F into rinv (n complex),
// and of the positive vector d into dinv (n reals), for the triangular solves.
COLD void diag_inverse(int n, int ld, const cplx* F, const double* d, cplx* rinv, double* dinv) {
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const cplx a = F[i * ld + i];
        const double id2 = 1.0 / (a.x * a.x + a.y * a.y);
        rinv[i] = cmk(a.x * id2, -a.y * id2);
        dinv[i] = 1.0 / d[i];
    }
    __syncthreads();
}

// C <- R^{-1} diag(rs) C (ZTRSM 'L','U','N','N' after scaling row r of C by
// rs[r]); rinv from diag_inverse.  Each segment holds its columns in
// registers; row i's value comes from lane i%8 by shuffle.
template <int R8, int CPS>
COLD void trsm_left_upper(int n, int ld, const cplx* F, const cplx* rinv, const double* rs, cplx* C) {
    const int tid = threadIdx.x, lane8 = tid & 7, seg = tid >> 3, nseg = blockDim.x >> 3;
    const unsigned m = seg8_mask();
    const int base = tid & 24;
    cplx c[CPS][R8];
#pragma unroll
    for (int q = 0; q < CPS; ++q)
#pragma unroll
        for (int k = 0; k < R8; ++k) {
            const int j = seg + q * nseg, r = lane8 + 8 * k;
            if (j < n && r < n) {
                const cplx x = C[r * ld + j];
                const double f = rs[r];
                c[q][k] = cmk(x.x * f, x.y * f);
            } else {
                c[q][k] = cmk(0.0, 0.0);
            }
        }
#pragma unroll
    for (int kk = R8 - 1; kk >= 0; --kk) {
        for (int l = 7; l >= 0; --l) {
            const int i = 8 * kk + l;
            if (i >= n) continue;   // uniform
            const cplx ri = rinv[i];
            cplx fcol[R8];
#pragma unroll
            for (int k = 0; k < R8; ++k) {
                const int r = lane8 + 8 * k;
                fcol[k] = (r < i) ? F[r * ld + i] : cmk(0.0, 0.0);
            }
#pragma unroll
            for (int q = 0; q < CPS; ++q) {
                cplx x;
                x.x = __shfl_sync(m, c[q][kk].x, base + l);
                x.y = __shfl_sync(m, c[q][kk].y, base + l);
                x = cmul(x, ri);
                if (lane8 == l) c[q][kk] = x;
#pragma unroll
                for (int k = 0; k < R8; ++k) c[q][k] = csub(c[q][k], cmul(fcol[k], x));   // fcol = 0 for rows >= i
            }
        }
    }
#pragma unroll
    for (int q = 0; q < CPS; ++q)
#pragma unroll
        for (int k = 0; k < R8; ++k) {
            const int j = seg + q * nseg, r = lane8 + 8 * k;
            if (j < n && r < n) C[r * ld + j] = c[q][k];
        }
    __syncthreads();
}

// C <- C diag(cs) R^{-H} (ZTRSM 'R','U','C','N' after scaling column c of C by
// cs[c]): X R^H = C diag(cs) solved for columns n-1..0.  Each segment holds
// its rows in registers; column c's value comes from lane c%8.
template <int R8, int CPS>
COLD void trsm_right_upperH(int n, int ld, const cplx* F, const cplx* rinv, const double* cs, cplx* C) {
    const int tid = threadIdx.x, lane8 = tid & 7, seg = tid >> 3, nseg = blockDim.x >> 3;
    const unsigned m = seg8_mask();
    const int base = tid & 24;
    cplx c[CPS][R8];   // c[q][k] = C[row seg+q*nseg][col lane8+8k]
#pragma unroll
    for (int q = 0; q < CPS; ++q)
#pragma unroll
        for (int k = 0; k < R8; ++k) {
            const int r = seg + q * nseg, col = lane8 + 8 * k;
            if (r < n && col < n) {
                const cplx x = C[r * ld + col];
                const double f = cs[col];
                c[q][k] = cmk(x.x * f, x.y * f);
            } else {
                c[q][k] = cmk(0.0, 0.0);
            }
        }
#pragma unroll
    for (int kk = R8 - 1; kk >= 0; --kk) {
        for (int l = 7; l >= 0; --l) {
            const int cc = 8 * kk + l;
            if (cc >= n) continue;
            const cplx ri = cconj(rinv[cc]);   // 1 / conj(R_cc)
            cplx frow[R8];                      // R[k][cc] for k < cc
#pragma unroll
            for (int k = 0; k < R8; ++k) {
                const int col = lane8 + 8 * k;
                frow[k] = (col < cc) ? F[col * ld + cc] : cmk(0.0, 0.0);
            }
#pragma unroll
            for (int q = 0; q < CPS; ++q) {
                cplx x;
                x.x = __shfl_sync(m, c[q][kk].x, base + l);
                x.y = __shfl_sync(m, c[q][kk].y, base + l);
                x = cmul(x, ri);
                if (lane8 == l) c[q][kk] = x;
#pragma unroll
                for (int k = 0; k < R8; ++k) c[q][k] = csub(c[q][k], cmulcj(x, frow[k]));
            }
        }
    }
#pragma unroll
    for (int q = 0; q < CPS; ++q)
#pragma unroll
        for (int k = 0; k < R8; ++k) {
            const int r = seg + q * nseg, col = lane8 + 8 * k;
            if (r < n && col < n) C[r * ld + col] = c[q][k];
        }
    __syncthreads();
}

// Row permutation in place.  forward: out[k][:] = in[piv[k]][:] (ZLAPMR .true.,
// i.e. P^T X); backward: out[piv[k]][:] = in[k][:] (ZLAPMR .false., i.e. P X).
template <int MAXE>
COLD void permute_rows(int n, int ld, cplx* C, const int* piv, const int* ipiv, bool forward) {
    const uint32_t dm = div_magic(n);
    cplx v[MAXE];
#pragma unroll
    for (int k = 0; k < MAXE; ++k) {
        const int e = threadIdx.x + k * blockDim.x;
        if (e < n * n) {
            const int r = div_by(e, dm), c = e - r * n;
            v[k] = C[(forward ? piv[r] : ipiv[r]) * ld + c];
        }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < MAXE; ++k) {
        const int e = threadIdx.x + k * blockDim.x;
        if (e < n * n) {
            const int r = div_by(e, dm), c = e - r * n;
            C[r * ld + c] = v[k];
        }
    }
    __syncthreads();
}

// Column permutation in place.  forward: out[:, k] = in[:, piv[k]] (ZLAPMT
// .true., X P); backward: out[:, piv[k]] = in[:, k] (ZLAPMT .false., X P^T).
template <int MAXE>
COLD void permute_cols(int n, int ld, cplx* C, const int* piv, const int* ipiv, bool forward) {
    const uint32_t dm = div_magic(n);
    cplx v[MAXE];
#pragma unroll
    for (int k = 0; k < MAXE; ++k) {
        const int e = threadIdx.x + k * blockDim.x;
        if (e < n * n) {
            const int r = div_by(e, dm), c = e - r * n;
            v[k] = C[r * ld + (forward ? piv[c] : ipiv[c])];
        }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < MAXE; ++k) {
        const int e = threadIdx.x + k * blockDim.x;
        if (e < n * n) {
            const int r = div_by(e, dm), c = e - r * n;
            C[r * ld + c] = v[k];
        }
    }
    __syncthreads();
}
