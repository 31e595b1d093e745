// CTA-level dense complex FP64 linear algebra on matrices resident in shared
// memory (row-major n x n with leading dimension ld; the sweep kernels use an
// odd ld so that a column walk touches every shared-memory bank group).  Every routine is called by all
// threads of the block and returns with the block synchronised.
//
// These restate the LAPACK/BLAS operations the reference sweep calls
// (src/number_conserving/src/stabilization.f90:41-190 and
// src/common/mymats.f90:20-29): ZGEMM, ZTRMM, ZGEQP3 (its pivoting, with exact
// remaining norms in place of ZLAQP2's downdated ones), ZUNGQR, ZUNMQR, ZTRSM,
// ZLAPMR/ZLAPMT.  They are written for the sweep's sizes (n <= 72): one CTA
// owns one matrix.  The factorisation and the reflector and triangular-solve
// sequences keep the columns of their operand in registers and reduce with
// shuffles; their dependent chains take reciprocals instead of divisions.
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

DEVI bool sumsq_unsafe(double ss) { return !(ss <= 1.0e300) || (ss != 0.0 && ss < 1.0e-290); }

// Shared scratch for the factorisations (lives in shared memory, size ~ 6n).
struct QRScratch {
    cplx* tau;      // n
    int* piv;       // n   (0-based: (A P)[:, j] = A[:, piv[j]])
    int* ipiv;      // n   inverse permutation
    double* vn1;    // n
    double* vn2;    // n
    double* d;      // n   |R_ii|
    // qr_columns only, in buffers of the local update
    cplx* vb;         // n   the pivot column
    cplx* scl;        // n   1 / d of the reflectors
    long long* keys;  // n   remaining norms of the columns as ordered integers
    double* bet;      // n   signed diagonal of R
    int* ex;          // n   scale exponents of the columns
};

// Scale 2^e of a column by its largest entry, as an exponent: that entry to 2^kQrTop (less for one
// below 2^-680, as 2^-e has to be finite); 0 for a non-finite column.  The largest power that occurs is
// the cube of a column's norm, b d2 in qr_block, below 2^(3 kQrTop + 14) for 72 rows and above 2^-1000
// for a square norm above kQrZero: a column is taken as zero once its remaining norm is 2^-653 of its
// largest entry.
constexpr int kQrTop = 320;
constexpr double kQrZero = 0x1p-666;
DEVI int scale_exponent(double m) {
    const int e = (int)((__double_as_longlong(m) >> 52) & 0x7ff);
    return e == 0x7ff ? 0 : max(e - 1022 - kQrTop, -1000);
}

// Pivoted QR of A (n x n): (A P) = Q R with ZGEQP3's pivot rule (the column of largest
// remaining norm), then the reference's QDRP_decompose post-step (stabilization.f90:41-67):
// d[i] = |R_ii| and row i of the upper triangle divided by d[i], piv and ipiv.
// AUG: also out <- Q^H in for the n x n view `in` (the identity if in.p is null), carried
// along with the columns of A, so that no pass over the reflectors follows; A's strict
// lower triangle is then not written.  Otherwise A holds the Householder vectors (unit
// leading entry implicit) below R, and s.tau their factors, for seq_apply.
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
// Columns are scaled by powers of two on entry (exact, and reflectors act on rows), whatever
// D has grown to, so that no sum of squares or product of norms over- or underflows until a
// remaining norm is 2^-653 of its column's largest entry (scale_exponent).
// Rows leave the registers from the top, a block of LPC at a time, so that no step masks
// them; a branch or a select per row cost more than the arithmetic (3500 cycles a step).
// Bound: the chain and the issue of a step on the warps that own columns, 1930 cycles at
// n = 36 with the second matrix (1475 without, 1100 at n = 16; 3720 at n = 72, where the
// registers spill); 131 K -> 69 K cycles for the factorisation.  The version before kept the matrix in shared memory, reduced over eight
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
        const bool zero = !(pn > kQrZero);
        const double y = rsqrt_fast(zero ? 1.0 : pn), nr = pn * y;
        const double nrm = fma(0.5 * y, fma(-nr, nr, pn), nr);   // a Newton (Heron) step: rounded as sqrt is
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
                // 1 / b anew: y has twice its error against b, b y y three times, and a tau and a row factor
                // that far from the reflector applied above cost a 72 x 72 Q 1.3 times the error
                // (orthogonality 9.4e-15 against 7.2e-15 here, LAPACK's 6.6e-15; G of 6x6 Nambu chains
                // 2.2e-13 against 1.7e-13)
                const double id2 = zero ? 0.0 : 1.0 / d2, ib = rcp_fast(b);
                s.piv[i] = j;
                s.ipiv[j] = i;
                s.tau[i] = zero ? cmk(0.0, 0.0) : cmk(-d.x * ib, -d.y * ib);
                s.bet[i] = zero ? 0.0 : b;
                s.vn2[i] = zero ? __longlong_as_double(0x7ff0000000000000LL) : fabs(ib);   // 1 / |beta|
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

// The reflector and triangular-solve sequences.  Eight lanes own a column of the operand, RPL of
// its rows each in registers (RPL * 8 >= n) for CPT columns at once, and walk it block by block of
// eight steps; a block's columns of F are staged in shared memory (vs: 8 x vld) by the whole CTA
// with their zeros (and the reflector's unit entry) in place, while the next block's are on their
// way in registers, so that no step waits for L2 or masks a row.  Rows that are done leave the
// registers a block at a time, the step count of a block growing or shrinking in three stretches.
// Bound: reading the staged block (two 16-byte loads of shared memory per row block and step) and
// the FP64 issue of the updates.  The versions before read F from global memory step by step:
// 144 x 144 2.3 M (reflectors) and 1.2 M cycles (solve) against 1.4 M and 0.6 M; wraps of 7x9
// chains 31.7 -> 24.3 M cycles a sweep.
//
// Element (row r, step i) of what is staged for block b.
//   SEQ_QH    v_i(r): 0 above i, 1 at i, F(r, i) below;  rows 8b..n-1, steps upwards
//   SEQ_SOLVE R(r, i) above i, else 0;                   rows 0..8b+7, steps downwards
enum { SEQ_QH = 0, SEQ_SOLVE = 1 };
constexpr int kSeqPf = 3;   // prefetched elements per thread
// A staged column has 8 RPL rows; SEQ_SOLVE also reads (into registers that are never used) the
// rows before the first that the last stretch reaches.  Odd, so that the eight columns of a row
// are stored to eight banks.
template <int RPL> constexpr int kSeqPad = 8 * ((RPL + 2) / 3);
template <int RPL> constexpr int kSeqLd = 8 * RPL + kSeqPad<RPL> + 1;
template <int RPL> constexpr int kSeqElems = 8 * kSeqLd<RPL> + kSeqPad<RPL>;

template <int KIND>
DEVI cplx seq_element(int n, int ld, const cplx* F, int b, int e) {
    const int kk = e & 7, r = (KIND == SEQ_QH ? 8 * b : 0) + (e >> 3), i = 8 * b + kk;
    const cplx f = F[min(r, n - 1) * ld + min(i, n - 1)];
    const bool use = i < n && r < n && (KIND == SEQ_QH ? r > i : r < i);
    return cmk(use ? f.x : (KIND == SEQ_QH && r == i ? 1.0 : 0.0), use ? f.y : 0.0);
}

// One block on the K register rows in reach: c[.][k] is row 8b + 8k + lc (SEQ_QH) or
// 8b - 8k + lc (SEQ_SOLVE); then row block b leaves c[.][0].
template <int KIND, int RPL, int K, int CPT>
DEVI void seq_block(int n, int b, const cplx* vs, int vld, const cplx* coef, cplx (&c)[CPT][RPL]) {
    const int lane = threadIdx.x & 31, lc = lane & 7;
#pragma unroll 1
    for (int q = 0; q < 8; ++q) {
        const int kk = KIND == SEQ_QH ? q : 7 - q, i = 8 * b + kk;
        if (i >= n) continue;
        const cplx* v = vs + kk * vld + (KIND == SEQ_QH ? lc : 8 * b + lc);   // rows 8k on: + 8k, or - 8k
        const cplx t = coef[i];
#pragma unroll
        for (int m = 0; m < CPT; ++m) {
            cplx f;
            if constexpr (KIND == SEQ_QH) {
                cplx w[2] = {cmk(0.0, 0.0), cmk(0.0, 0.0)};
#pragma unroll
                for (int k = 0; k < K; ++k) w[k & 1] = cfmacj(v[8 * k], c[m][k], w[k & 1]);
                cplx s = cadd(w[0], w[1]);
#pragma unroll
                for (int d = 4; d > 0; d >>= 1) {
                    s.x += __shfl_xor_sync(0xffffffffu, s.x, d);
                    s.y += __shfl_xor_sync(0xffffffffu, s.y, d);
                }
                f = cmul(cmk(-t.x, t.y), s);   // -conj(tau) v^H c
            } else {
                const int src = (lane & 24) + kk;
                cplx x = cmk(__shfl_sync(0xffffffffu, c[m][0].x, src), __shfl_sync(0xffffffffu, c[m][0].y, src));
                x = cmul(x, t);
                c[m][0] = cmk(lc == kk ? x.x : c[m][0].x, lc == kk ? x.y : c[m][0].y);
                f = cmk(-x.x, -x.y);
            }
#pragma unroll
            for (int k = 0; k < K; ++k) c[m][k] = cfma(v[KIND == SEQ_QH ? 8 * k : -8 * k], f, c[m][k]);
        }
    }
}

// SEQ_QH:    out <- Q^H in, F and coef = tau from qr_columns or qrp_big (the identity if in.p is null)
// SEQ_SOLVE: out <- P R^{-1} diag(rs) in, coef = 1 / R_ii, row k of the solution to row piv[k]
// in and out are n x n views (conjugated views serve the products and solves from the right);
// they may be the same matrix.
template <int KIND, int RPL, int CPT>
COLD void seq_apply(int n, int ld, const cplx* F, const cplx* coef, const double* rs, const int* piv, MatOp in, MatOp out,
                    cplx* buf) {
    n = uni(n);
    const int vld = kSeqLd<RPL>;
    cplx* const vs = buf + kSeqPad<RPL>;
    const int tid = threadIdx.x, T = blockDim.x, lc = tid & 7, ng = T >> 3;
    const int nb = (n + 7) >> 3;
    constexpr int K2 = (2 * RPL + 2) / 3, K3 = (RPL + 2) / 3;
    cplx* const o = const_cast<cplx*>(out.p);
    for (int j0 = 0; j0 < n; j0 += ng * CPT) {
        const int j = j0 + (tid >> 3);
        cplx c[CPT][RPL];
#pragma unroll
        for (int m = 0; m < CPT; ++m)
#pragma unroll
            for (int k = 0; k < RPL; ++k) {
                const int r = 8 * (KIND == SEQ_QH ? k : nb - 1 - k) + lc, jm = j + m * ng;
                const int rc = max(min(r, n - 1), 0), jc = min(jm, n - 1);
                cplx w = cmk(r == jm ? 1.0 : 0.0, 0.0);
                if (in.p) {
                    w = in.p[rc * in.sr + jc * in.sc];
                    if (in.cj) w.y = -w.y;
                }
                const double f = KIND == SEQ_SOLVE ? rs[rc] : 1.0;
                const bool ok = r >= 0 && r < n && jm < n;
                c[m][k] = cmk(ok ? w.x * f : 0.0, ok ? w.y * f : 0.0);
            }
        cplx pf[kSeqPf];
        int b = KIND == SEQ_QH ? 0 : nb - 1;
        const int step = KIND == SEQ_QH ? 1 : -1;
#pragma unroll
        for (int q = 0; q < kSeqPf; ++q) pf[q] = seq_element<KIND>(n, ld, F, b, tid + q * T);
        for (int left = nb; left > 0; --left, b += step) {
            // SEQ_QH reads all the register rows in reach (zeros past n, as 0 x anything finite is needed)
            const int rows = KIND == SEQ_QH ? 8 * (left > K2 ? RPL : (left > K3 ? K2 : K3)) : 8 * (b + 1);
            __syncthreads();   // the staged block is free
#pragma unroll
            for (int q = 0; q < kSeqPf; ++q) {
                const int e = tid + q * T;
                if (e < 8 * rows) vs[(e & 7) * vld + (e >> 3)] = pf[q];
            }
            for (int e = tid + kSeqPf * T; e < 8 * rows; e += T) vs[(e & 7) * vld + (e >> 3)] = seq_element<KIND>(n, ld, F, b, e);
            __syncthreads();
            const int bn = max(min(b + step, nb - 1), 0);
#pragma unroll
            for (int q = 0; q < kSeqPf; ++q) pf[q] = seq_element<KIND>(n, ld, F, bn, tid + q * T);
            if (uni(j) < n) {   // any column of the warp
                if (left > K2) seq_block<KIND, RPL, RPL, CPT>(n, b, vs, vld, coef, c);
                else if (left > K3) seq_block<KIND, RPL, K2, CPT>(n, b, vs, vld, coef, c);
                else seq_block<KIND, RPL, K3, CPT>(n, b, vs, vld, coef, c);
            }
#pragma unroll
            for (int m = 0; m < CPT; ++m) {
                const int r = 8 * b + lc, jm = j + m * ng;
                if (r < n && jm < n) {
                    const int ro = KIND == SEQ_SOLVE ? piv[r] : r;
                    o[ro * out.sr + jm * out.sc] = out.cj ? cconj(c[m][0]) : c[m][0];
                }
#pragma unroll
                for (int k = 0; k + 1 < RPL; ++k) c[m][k] = c[m][k + 1];
                c[m][RPL - 1] = cmk(0.0, 0.0);
            }
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
