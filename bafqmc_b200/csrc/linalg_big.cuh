// Dense complex FP64 linear algebra for the largest size class (n up to 144),
// whose matrices live in a per-chain region of global memory because neither
// the shared memory of one SM (227 KB) nor its register file holds the five
// n x n complex matrices a chain works on.  While a chain runs, its region
// stays in L2.
//
// Same operations and conventions as linalg.cuh (ZGEMM/ZTRMM, ZGEQP3 in the ZLAQP2
// form with the QDRP_decompose post-step; row-major with leading dimension ld; called
// by all threads of the block, returning with the block synchronised).  In the QR one
// warp takes a column: lane l holds rows l, l+32, ... (RW >= ceil(n/32) of them), and
// reductions are warp shuffles.  Products are out of place through a scratch matrix S.
#pragma once
#include "linalg.cuh"

DEVI double warp_max(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// The factorisation works on a column-major copy: element (r, j) at A[j * ld + r], so that a
// warp's walk of a column is contiguous.
// Overflow-safe 2-norm of column j, rows [r0, n), by one warp.
DEVI double warp_colnorm(int n, int ld, const cplx* A, int j, int r0) {
    const int lane = threadIdx.x & 31;
    double m = 0.0;
    for (int r = r0 + lane; r < n; r += 32) m = fmax(m, fmax(fabs(A[j * ld + r].x), fabs(A[j * ld + r].y)));
    m = warp_max(m);
    if (m == 0.0) return 0.0;
    double s = 0.0;
    for (int r = r0 + lane; r < n; r += 32) {
        const double a = A[j * ld + r].x / m, b = A[j * ld + r].y / m;
        s += a * a + b * b;
    }
    return m * sqrt(warp_sum(s));
}

DEVI double warp_norm(int n, int ld, const cplx* A, int j, int r0) {
    const int lane = threadIdx.x & 31;
    double ss = 0.0;
    for (int r = r0 + lane; r < n; r += 32) {
        const cplx a = A[j * ld + r];
        ss = fma(a.x, a.x, fma(a.y, a.y, ss));
    }
    ss = warp_sum(ss);
    if (!sumsq_unsafe(ss)) return sqrt(ss);
    return warp_colnorm(n, ld, A, j, r0);
}

// C = A B (n x n <= 144, C apart from the operands) on the FP64 tensor pipe, operands in
// global memory (L2): k is staged in chunks of 16 through shared memory (`stage`, two
// buffers, cp.async), for column panels of 64.  KIND as in prod_mma: PROD_CC, or one real
// operand R (leading dimension ldr, even, rows 16-byte aligned) on the left (R X, X = B) or
// on the right, taken as C^T = R^T X^T (B = X^T): the complex operand, a chain's own, is
// then read once and R, which the point's chains share, once per panel.  The matrices of 148
// chains in flight are more than L2 holds.
// Each operand is staged in the order it is stored in (rows or columns contiguous), with
// an odd leading dimension in shared memory, and taken with the fragment maps of
// mma64.cuh.  A warp owns one column tile of a panel and up to nine row tiles, so a step of
// four k reads 10 fragments for 18 (real) or 36 mma: 38 of 72, or 40 of 144, cycles of
// shared memory.  tri as there (zeros are filled in when a chunk is staged).
// The mma bound of a complex x real product at n = 144 is 93 K cycles; it takes 160 K by
// itself and 270 K inside the sweep kernel, where the accumulators share the registers with
// the callers' state (per-thread tiles reading L2 took 500 K; 256 threads of twice the
// registers, or panels of 40 columns with six row tiles a warp, were no faster).
constexpr int kBigK = 16, kBigCols = 64, kBigRows = 144;
constexpr int kBigLa = kBigK + 1, kBigLb = kBigCols + 1, kBigLra = kBigK + 4, kBigLrt = kBigRows + 4;
constexpr size_t kBigABytes = sizeof(cplx) * kBigRows * kBigLa, kBigBBytes = sizeof(cplx) * kBigCols * kBigLa;
constexpr size_t kBigStage = 2 * (kBigABytes + kBigBBytes);

DEVI void cp16(void* dst, const void* src, int bytes) {   // the rest of the 16 bytes as zeros
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
                 "r"(bytes)
                 : "memory");
}

// one staged chunk into the accumulators of the warp's CNT row tiles (from rt0) and column tile ct
template <int KIND, int CNT>
DEVI void big_chunk(double (&re)[9][2], double (&im)[9][2], const unsigned char* sa, const unsigned char* sb, int rt0, int nrt,
                    int ct, int ars, int aks, int bcs, int bks, double ca, double cb) {
    const int lane = threadIdx.x & 31, l4 = lane & 3, l8 = lane >> 2;
    const cplx* A = reinterpret_cast<const cplx*>(sa);
    const cplx* B = reinterpret_cast<const cplx*>(sb);
    const double* Ra = reinterpret_cast<const double*>(sa);
#pragma unroll
    for (int k4 = 0; k4 < kBigK; k4 += 4) {
        const int k = k4 + l4;
        cplx b = B[tile_at(ct, l8) * bcs + k * bks];
        if (KIND == PROD_CC) b.y *= cb;
#pragma unroll
        for (int i = 0; i < CNT; ++i) {
            const int rt = min(rt0 + i, nrt - 1);
            if constexpr (KIND != PROD_CC) {
                const double ra = KIND == PROD_REAL_L ? Ra[(8 * rt + l8) * kBigLra + k] : Ra[k * kBigLrt + 8 * rt + l8];
                mma_f64(re[i][0], re[i][1], ra, b.x);
                mma_f64(im[i][0], im[i][1], ra, b.y);
            } else {
                cplx a = A[tile_at(rt, l8) * ars + k * aks];
                a.y *= ca;
                mma_f64(re[i][0], re[i][1], a.x, b.x);
                mma_f64(im[i][0], im[i][1], a.x, b.y);
                mma_f64(re[i][0], re[i][1], -a.y, b.y);
                mma_f64(im[i][0], im[i][1], a.y, b.x);
            }
        }
    }
}

template <int KIND>
COLD void gemm_big(int n, int ldc, cplx* C, MatOp A, MatOp B, const double* R, int ldr, int tri, unsigned char* stage) {
    n = uni(n);
    tri = uni(tri);
    const int tid = threadIdx.x, T = blockDim.x, lane = tid & 31, warp = warp_index(), nw = T >> 5;
    const int l4 = lane & 3, l8 = lane >> 2;
    const int n8 = (n + 7) >> 3, npan = (n8 + 7) >> 3, nk = (n + kBigK - 1) / kBigK, items = npan * nk;
    const bool arow = A.sc == 1, brow = B.sc == 1;   // stored with k (A) or columns (B) contiguous
    const int ars = arow ? kBigLa : 1, aks = arow ? 1 : kBigRows + 1;
    const int bcs = brow ? 1 : kBigLa, bks = brow ? kBigLb : 1;
    const double ca = A.cj ? -1.0 : 1.0, cb = B.cj ? -1.0 : 1.0;
    const auto fill = [&](int it) {
        if (it < items) {
            const int pan = it / nk, k0 = (it - pan * nk) * kBigK, c0 = pan * kBigCols;
            unsigned char* da = stage + (it & 1) * (kBigABytes + kBigBBytes);
            unsigned char* db = da + kBigABytes;
            if constexpr (KIND == PROD_REAL_L) {
                for (int e = tid; e < kBigRows * (kBigK / 2); e += T) {
                    const int r = e / (kBigK / 2), k = k0 + 2 * (e % (kBigK / 2));
                    const int ok = r < n ? min(max(n - k, 0), 2) : 0;
                    cp16(da + 8 * (r * kBigLra + k - k0), R + (ok ? r * ldr + k : 0), 8 * ok);
                }
            } else if constexpr (KIND == PROD_REAL_R) {   // R^T: rows contiguous
                for (int e = tid; e < kBigK * (kBigRows / 2); e += T) {
                    const int kk = e / (kBigRows / 2), r = 2 * (e % (kBigRows / 2)), k = k0 + kk;
                    const int ok = k < n ? min(max(n - r, 0), 2) : 0;
                    cp16(da + 8 * (kk * kBigLrt + r), R + (ok ? k * ldr + r : 0), 8 * ok);
                }
            } else if (arow) {
                for (int e = tid; e < kBigRows * kBigK; e += T) {
                    const int r = e / kBigK, kk = e % kBigK, k = k0 + kk;
                    const bool ok = r < n && k < n && !(tri == TRI_A_UPPER && k < r);
                    cp16(da + 16 * (r * kBigLa + kk), A.p + (ok ? r * A.sr + k : 0), ok ? 16 : 0);
                }
            } else {
                for (int e = tid; e < kBigRows * kBigK; e += T) {
                    const int kk = e / kBigRows, r = e % kBigRows, k = k0 + kk;
                    const bool ok = r < n && k < n;
                    cp16(da + 16 * (kk * (kBigRows + 1) + r), A.p + (ok ? r + k * A.sc : 0), ok ? 16 : 0);
                }
            }
            if (brow) {
                for (int e = tid; e < kBigK * kBigCols; e += T) {
                    const int kk = e / kBigCols, cc = e % kBigCols, k = k0 + kk, c = c0 + cc;
                    const bool ok = k < n && c < n;
                    cp16(db + 16 * (kk * kBigLb + cc), B.p + (ok ? k * B.sr + c : 0), ok ? 16 : 0);
                }
            } else {
                for (int e = tid; e < kBigCols * kBigK; e += T) {
                    const int cc = e / kBigK, kk = e % kBigK, k = k0 + kk, c = c0 + cc;
                    const bool ok = k < n && c < n && !(tri == TRI_B_LOWER_FROM_C && k < c);
                    cp16(db + 16 * (cc * kBigLa + kk), B.p + (ok ? k + c * B.sc : 0), ok ? 16 : 0);
                }
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    __syncthreads();   // the staging buffers are free
    fill(0);
    double re[9][2], im[9][2];
    for (int it = 0; it < items; ++it) {
        const int pan = it / nk, kc = it - pan * nk;
        const int pc = min(n8 - 8 * pan, 8), rs = nw / pc, rps = (n8 + rs - 1) / rs;
        const int ct = warp % pc, rg = warp / pc, rt0 = rg * rps;
        const bool on = rg < rs && rt0 < n8;
        if (kc == 0) {
#pragma unroll
            for (int i = 0; i < 9; ++i) re[i][0] = re[i][1] = im[i][0] = im[i][1] = 0.0;
        }
        fill(it + 1);
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();
        const unsigned char* sa = stage + (it & 1) * (kBigABytes + kBigBBytes);
        const unsigned char* sb = sa + kBigABytes;
        const int nrt = min(n8, rt0 + rps);
        if (on) {
            if (rps > 6) big_chunk<KIND, 9>(re, im, sa, sb, rt0, nrt, ct, ars, aks, bcs, bks, ca, cb);
            else if (rps > 3) big_chunk<KIND, 6>(re, im, sa, sb, rt0, nrt, ct, ars, aks, bcs, bks, ca, cb);
            else big_chunk<KIND, 3>(re, im, sa, sb, rt0, nrt, ct, ars, aks, bcs, bks, ca, cb);
        }
        __syncthreads();   // the chunk's buffer is filled again by the next turn
        if (kc == nk - 1 && on) {
#pragma unroll
            for (int i = 0; i < 9; ++i) {
                const int rt = rt0 + i;
                const int r = KIND == PROD_CC ? tile_at(rt, l8) : 8 * rt + l8, c = pan * kBigCols + 8 * ct + l4;
                const int rs1 = KIND == PROD_REAL_R ? 1 : ldc, cs1 = KIND == PROD_REAL_R ? ldc : 1;   // transposed back
                if (rt < nrt && r < n && c < n) C[r * rs1 + c * cs1] = cmk(re[i][0], im[i][0]);
                if (rt < nrt && r < n && c + 4 < n) C[r * rs1 + (c + 4) * cs1] = cmk(re[i][1], im[i][1]);
            }
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
}

COLD void copy_mat(int n, int ld, cplx* dst, const cplx* src) {
    const uint32_t dm = div_magic(n);
    for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
        const int r = div_by(e, dm), c = e - r * n;
        dst[r * ld + c] = src[r * ld + c];
    }
    __syncthreads();
}

// A <- A^H through S.
COLD void conj_transpose_big(int n, int ld, cplx* A, cplx* S) {
    copy_op(n, ld, S, op_c(A, ld));
    copy_mat(n, ld, A, S);
}

// ZGEQP3 (ZLAQP2 recurrence) + QDRP_decompose post-step.
// Per column: every warp finds the pivot and forms the reflector from the
// pivot column (barrier); the warps update the trailing columns one by one,
// column pvt from the old column i, with ZLAQP2's norm downdate (barrier);
// column i takes the reflector and beta, rows above i of columns i and pvt are
// swapped (barrier).  A is column-major, as above.
template <int RW>
COLD void qrp_big(int n, int ld, cplx* A, QRScratch s) {
#define QA(r, c) A[(c) * ld + (r)]
    const int tid = threadIdx.x, lane = tid & 31, wp = tid >> 5, nw = blockDim.x >> 5;
    const double tol3z = 1.0536712127723509e-08;   // sqrt(2^-53), LAPACK's sqrt(dlamch('E'))
    for (int j = wp; j < n; j += nw) {
        const double v = warp_norm(n, ld, A, j, 0);
        if (lane == 0) {
            s.vn1[j] = v;
            s.vn2[j] = v;
            s.piv[j] = j;
        }
    }
    __syncthreads();
    for (int i = 0; i < n; ++i) {
        double best = -1.0;
        int bi = n;
        for (int j = i + lane; j < n; j += 32) {
            const double v = s.vn1[j];
            if (v > best) {
                best = v;
                bi = j;
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const double ob = __shfl_xor_sync(0xffffffffu, best, o);
            const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
            if (ob > best || (ob == best && oi < bi)) {
                best = ob;
                bi = oi;
            }
        }
        const int pvt = (bi < n) ? bi : i;
        cplx v[RW];
        double ss = 0.0;
#pragma unroll
        for (int k = 0; k < RW; ++k) {
            const int r = lane + 32 * k;
            v[k] = (r < n && r > i) ? QA(r, pvt) : cmk(0.0, 0.0);
            ss = fma(v[k].x, v[k].x, fma(v[k].y, v[k].y, ss));
        }
        ss = warp_sum(ss);
        const cplx alpha = QA(i, pvt);
        double xn = sqrt(ss);
        if (sumsq_unsafe(ss)) xn = warp_colnorm(n, ld, A, pvt, i + 1);
        cplx tau = cmk(0.0, 0.0), beta = alpha, scl = cmk(0.0, 0.0);
        if (!(xn == 0.0 && alpha.y == 0.0)) {
            const double nrm = sqrt(alpha.x * alpha.x + alpha.y * alpha.y + xn * xn);
            const double b = (alpha.x >= 0.0) ? -nrm : nrm;
            const double ib = 1.0 / b;
            tau = cmk((b - alpha.x) * ib, -alpha.y * ib);
            const cplx d = cmk(alpha.x - b, alpha.y);
            const double id2 = 1.0 / (d.x * d.x + d.y * d.y);
            scl = cmk(d.x * id2, -d.y * id2);
            beta = cmk(b, 0.0);
        }
#pragma unroll
        for (int k = 0; k < RW; ++k) {
            const int r = lane + 32 * k;
            v[k] = (r == i) ? cmk(1.0, 0.0) : cmul(scl, v[k]);
        }
        __syncthreads();
        // trailing columns; logical column pvt holds the old column i
        const cplx ctau = cconj(tau);
        for (int j = i + 1 + wp; j < n; j += nw) {
            const int src = (j == pvt) ? i : j;
            cplx a[RW];
#pragma unroll
            for (int k = 0; k < RW; ++k) {
                const int r = lane + 32 * k;
                a[k] = (r < n && r >= i) ? QA(r, src) : cmk(0.0, 0.0);
            }
            const double t1 = s.vn1[src], t2 = s.vn2[src];
            cplx w = cmk(0.0, 0.0);
#pragma unroll
            for (int k = 0; k < RW; ++k) w = cfmacj(v[k], a[k], w);
            w.x = warp_sum(w.x);
            w.y = warp_sum(w.y);
            const cplx f = cmul(ctau, w);
            double ai2 = 0.0, rest = 0.0;
#pragma unroll
            for (int k = 0; k < RW; ++k) {
                const int r = lane + 32 * k;
                a[k] = csub(a[k], cmul(v[k], f));
                const double m2 = a[k].x * a[k].x + a[k].y * a[k].y;
                if (r == i) ai2 = m2;
                if (r > i && r < n) rest += m2;
                if (r < n && r >= i) QA(r, j) = a[k];
            }
            ai2 = warp_sum(ai2);
            rest = warp_sum(rest);
            double nv1 = t1, nv2 = t2;
            if (t1 != 0.0) {
                bool recompute;
                if (t1 < 1.0e150 && t2 < 1.0e150) {
                    const double rem = fmax(t1 * t1 - ai2, 0.0);
                    recompute = rem <= tol3z * t2 * t2;
                    nv1 = sqrt(rem);
                } else {
                    const double tt = sqrt(ai2) / t1;
                    const double temp = fmax(1.0 - tt * tt, 0.0);
                    const double qq = t1 / t2;
                    recompute = !(temp * qq * qq > tol3z);
                    nv1 = t1 * sqrt(temp);
                }
                if (recompute) {
                    if (sumsq_unsafe(rest)) {
                        __syncwarp();
                        nv1 = (i + 1 < n) ? warp_colnorm(n, ld, A, j, i + 1) : 0.0;
                    } else {
                        nv1 = sqrt(rest);
                    }
                    nv2 = nv1;
                }
            }
            __syncwarp();
            if (lane == 0) {
                s.vn1[j] = nv1;
                s.vn2[j] = nv2;
            }
        }
        __syncthreads();
        if (wp == 0) {
#pragma unroll
            for (int k = 0; k < RW; ++k) {
                const int r = lane + 32 * k;
                if (r < n && r > i) QA(r, i) = v[k];
            }
            if (lane == 0) {
                QA(i, i) = beta;
                s.tau[i] = tau;
            }
        }
        if (pvt != i && tid < i) {
            const cplx ui = QA(tid, i), up = QA(tid, pvt);
            QA(tid, i) = up;
            QA(tid, pvt) = ui;
        }
        if (tid == 0 && pvt != i) {
            const int t = s.piv[pvt];
            s.piv[pvt] = s.piv[i];
            s.piv[i] = t;
        }
        __syncthreads();
    }
    for (int i = tid; i < n; i += blockDim.x) {
        const cplx a = QA(i, i);
        const double d = hypot(a.x, a.y);
        s.d[i] = d;
        s.vn1[i] = 1.0 / d;
    }
    __syncthreads();
    const uint32_t dm = div_magic(n);
    for (int e = tid; e < n * n; e += blockDim.x) {
        const int c = div_by(e, dm), r = e - c * n;   // consecutive threads walk the storage order
        if (c >= r) {
            const double x = s.vn1[r];
            const cplx a = QA(r, c);
            QA(r, c) = cmk(a.x * x, a.y * x);
        }
    }
    for (int k = tid; k < n; k += blockDim.x) s.ipiv[s.piv[k]] = k;
    __syncthreads();
#undef QA
}
