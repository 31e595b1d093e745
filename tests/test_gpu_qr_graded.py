"""The register-held pivoted QR of linalg.cuh on matrices whose remaining column norms fall far below the
columns' largest entries, and on columns of very different scale, against determinants and dense products.

Rows are graded by powers of two in decreasing order, columns scaled by powers of two, so that the matrix is
exact and ln|det| is that of the ungraded random matrix B plus the exponents.  Tolerance: with column pivoting
and rows in decreasing order Householder QR is backward stable row by row, each row to a few n 2^-53 of its own
largest entry (64 n 2^-53 is allowed), and with columns of any scale column by column, which moves ln|det| by at
most n cond(B) of that (with both the pivoting follows the columns, and ln|det| is not compared); Q and the
product of the factors are normwise accurate, 64 n 2^-53 per element of a unit vector and of a column's norm."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "bafqmc_b200", "csrc")
PROGRAM = r"""
#include "linalg.cuh"
extern __shared__ __align__(16) unsigned char sm[];
// A <- its factorisation, Qh <- Q^H, d and piv, all row-major n x n
template <int LPC, int RPL, bool AUG, int SR, int SC, int NMAX, int TH>
__global__ void __launch_bounds__(TH) factor(int n, cplx* gA, cplx* gQ, double* gd, int* gp) {
    constexpr int LD = NMAX | 1;
    cplx *A = (cplx*)sm, *Q = A + NMAX * LD, *v = Q + NMAX * LD;
    QRScratch s;
    s.tau = v, v += NMAX;
    s.vb = v, v += NMAX + 1;
    s.scl = v, v += NMAX + 1;
    s.keys = (long long*)v, v += NMAX;
    s.bet = (double*)v, v += NMAX;
    s.ex = (int*)v, v += NMAX;
    s.vn1 = (double*)v, v += NMAX;
    s.vn2 = (double*)v, v += NMAX;
    s.d = (double*)v, v += NMAX;
    s.piv = (int*)v, v += NMAX;
    s.ipiv = (int*)v, v += NMAX;
    for (int e = threadIdx.x; e < n * n; e += blockDim.x) A[e / n * LD + e % n] = gA[e];
    __syncthreads();
    if (AUG) {
        qr_columns<LPC, RPL, true>(n, LD, A, s, MatOp{}, op_n(Q, LD));
    } else {
        qr_columns<LPC, RPL, false>(n, LD, A, s, MatOp{}, MatOp{});
        seq_apply<SEQ_QH, SR, SC>(n, LD, A, s.tau, nullptr, nullptr, MatOp{}, op_n(Q, LD), v);
    }
    for (int e = threadIdx.x; e < n * n; e += blockDim.x) gA[e] = A[e / n * LD + e % n], gQ[e] = Q[e / n * LD + e % n];
    for (int e = threadIdx.x; e < n; e += blockDim.x) gd[e] = s.d[e], gp[e] = s.piv[e];
}
template <int LPC, int RPL, bool AUG, int SR, int SC, int NMAX, int TH>
int go(int n, double* A, double* Q, double* d, int* p) {
    auto f = factor<LPC, RPL, AUG, SR, SC, NMAX, TH>;
    const int bytes = (2 * NMAX * (NMAX | 1) + 11 * NMAX + 2 + kSeqElems<SR>) * 16, m = n * n * 16;
    cplx *gA, *gQ;
    double* gd;
    int* gp;
    if (n > NMAX || cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess) return 1;
    if (cudaMalloc(&gA, m) || cudaMalloc(&gQ, m) || cudaMalloc(&gd, n * 8) || cudaMalloc(&gp, n * 4)) return 2;
    if (cudaMemcpy(gA, A, m, cudaMemcpyHostToDevice)) return 3;
    f<<<1, TH, bytes>>>(n, gA, gQ, gd, gp);
    if (cudaMemcpy(A, gA, m, cudaMemcpyDeviceToHost) || cudaMemcpy(Q, gQ, m, cudaMemcpyDeviceToHost) ||
        cudaMemcpy(d, gd, n * 8, cudaMemcpyDeviceToHost) || cudaMemcpy(p, gp, n * 4, cudaMemcpyDeviceToHost))
        return 4;
    cudaFree(gA), cudaFree(gQ), cudaFree(gd), cudaFree(gp);
    return 0;
}
extern "C" int run(int nmax, int n, double* A, double* Q, double* d, int* p) {
    if (nmax == 16) return go<4, 4, true, 2, 1, 16, 128>(n, A, Q, d, p);
    if (nmax == 36) return go<4, 9, true, 5, 2, 36, 256>(n, A, Q, d, p);
    return go<4, 18, false, 9, 2, 72, 512>(n, A, Q, d, p);
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    d = tmp_path_factory.mktemp("qr")
    (d / "q.cu").write_text(PROGRAM)
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O3", "-Xcompiler", "-fPIC", "-shared",
                    "-I", CSRC, "-o", str(d / "q.so"), str(d / "q.cu")], check=True, timeout=600)
    return C.CDLL(str(d / "q.so"))


@pytest.mark.parametrize("nmax,n", [(16, 1), (16, 9), (16, 16), (36, 17), (36, 36), (72, 37), (72, 63), (72, 72)])
@pytest.mark.parametrize("rows,cols", [(0, 0), (400, 0), (600, 0), (0, 900), (300, 300), (400, -400)])
def test_graded_matrix(lib, nmax, n, rows, cols):
    """Rows from 2^0 down to 2^-rows; columns by 2^(-cols/2 .. cols/2), rising or falling."""
    rng = np.random.default_rng(1000 * n + rows)
    B = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    k = np.arange(n) / max(n - 1, 1)
    er, ec = np.rint(-rows * k).astype(int), np.rint(cols * (k - 0.5)).astype(int)
    e = er[:, None] + ec[None, :]
    A = np.ldexp(B.real, e) + 1j * np.ldexp(B.imag, e)
    F, Q = A.copy(), np.zeros((n, n), dtype=np.complex128)
    d, piv = np.zeros(n), np.zeros(n, dtype=np.int32)
    p = lambda a: a.ctypes.data_as(C.c_void_p)
    assert lib.run(nmax, n, p(F), p(Q), p(d), p(piv)) == 0
    assert sorted(piv) == list(range(n))
    R = np.triu(F)
    assert np.all(np.isfinite(d)) and np.all(np.isfinite(R)) and np.all(np.isfinite(Q)) and np.all(d > 0)
    tol = 64 * n * 2.0 ** -53
    assert np.max(np.abs(Q @ Q.conj().T - np.eye(n))) <= tol
    np.testing.assert_allclose(np.abs(np.diag(R)), 1.0, rtol=0, atol=tol)
    if rows == 0 or cols == 0:   # ln|det|
        want = np.linalg.slogdet(B)[1] + np.log(2.0) * (er.sum() + ec.sum())
        assert abs(np.log(d).sum() - want) <= tol * n * np.linalg.cond(B)
    # the product, column by column, each in its own scale
    for j in range(n):
        c = piv[j]
        dr = d * R[:, j]   # d R is at most the column's norm
        got = Q.conj().T @ (np.ldexp(dr.real, -ec[c]) + 1j * np.ldexp(dr.imag, -ec[c]))
        col = np.ldexp(A[:, c].real, -ec[c]) + 1j * np.ldexp(A[:, c].imag, -ec[c])
        assert np.max(np.abs(got - col)) <= tol * np.linalg.norm(col)


@pytest.mark.parametrize("nmax,n", [(16, 16), (36, 36), (72, 36), (72, 72)])
def test_factors_as_exact_as_lapacks(lib, nmax, n):
    """Orthogonality of Q and the residual of the product, as means over matrices U D like those of a wrap, at most
    1.25 times LAPACK's on the same ones: both round the same sums, and a reflector's two scalars to a unit more here."""
    import scipy.linalg as sl
    ld, err = np.clongdouble, np.zeros((2, 2))
    p = lambda a: a.ctypes.data_as(C.c_void_p)
    for seed in range(20):
        rng = np.random.default_rng(seed)
        A = np.linalg.qr(rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)))[0] * np.exp(-rng.uniform(0, 20, n))
        F, Q, d, piv = A.copy(), np.zeros((n, n), dtype=np.complex128), np.zeros(n), np.zeros(n, dtype=np.int32)
        assert lib.run(nmax, n, p(F), p(Q), p(d), p(piv)) == 0
        lq, lr, lp = sl.qr(A, pivoting=True)
        for k, (q, r, pv) in enumerate(((Q.conj().T, np.triu(F) * d[:, None], piv), (lq, lr, lp))):
            q = q.astype(ld)
            err[k] += (np.linalg.norm((q.conj().T @ q - np.eye(n)).astype(complex)),
                       np.linalg.norm(((q @ r.astype(ld) - A[:, pv]) / np.linalg.norm(A[:, pv], axis=0)).astype(complex)))
    assert np.all(err[0] <= 1.25 * err[1]), err / 20
