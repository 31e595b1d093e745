// Sweep kernels for the BAFQMC number-conserving and Nambu pairing solvers on
// sm_100a.
//
// One CTA = one Markov chain.  sweep_kernel runs one full sweep (left then
// right traversal of imaginary time, local_sweep.f90:96-134 with is_beta
// = .true.) including every local update, slice propagation, stabilisation
// and equal-time measurement of that chain.  pre_kernel builds the right UDV
// slots and G(beta) (local_sweep.f90:80-94); warmup_kernel is the prior-only
// warm-up (local_sweep.f90:64-78).  Both sweep kernels are instantiated per
// shared-memory size class and per sector (PAIR: Nambu chains).
#include "sweep.cuh"
#include "kernels.h"
#include "linalg_big.cuh"
#include "tc.cuh"

namespace bq {

__constant__ uint32_t c_apow[kMaxPow];   // a^k mod 2^31 for k = 0 .. kMaxPow-1

template <int NMAX> struct Cfg;
// LPC lanes per column and RPL rows per lane for the pivoted QR, AUG: the second matrix
// is carried along (both columns fit the registers); SR rows per lane and SC columns per
// eight lanes for the reflector and solve sequences.
// MQ tiles per warp, MB at a time, for the complex products and MP for the real ones
// (mma64.cuh).
// LD: leading dimension of the shared-memory matrices, odd so that a column
// walk over 16-byte elements touches all eight bank groups.  MINB: CTAs per SM for the register
// budget.  GW: the two workspaces live in HBM (after the chain's arena) and
// only G and U in shared memory.  GG: G and U in HBM as well, products staged through shared
// memory, slice products also on the tensor cores (tc.cuh).
template <> struct Cfg<16> {
    static constexpr int THREADS = 128, MAXE = 2, KB = 8, LD = 17, MINB = 4;
    static constexpr bool GW = false, GG = false;
    static constexpr int MQ = 1, MB = 1, MP = 2;
    static constexpr bool AUG = true;
    static constexpr int LPC = 4, RPL = 4, SR = 2, SC = 1;
};
// N <= 36: two CTAs per SM, all four matrices in shared memory.
template <> struct Cfg<36> {
    static constexpr int THREADS = 256, MAXE = 6, KB = 8, LD = 37, MINB = 2;
    static constexpr bool GW = false, GG = false;
    static constexpr int MQ = 4, MB = 2, MP = 8;
    static constexpr bool AUG = true;
    static constexpr int LPC = 4, RPL = 9, SR = 5, SC = 2;
};
// N <= 72: G and U in shared memory, the workspaces in HBM (one CTA per SM)
template <> struct Cfg<72> {
    static constexpr int THREADS = 512, MAXE = 11, KB = 8, LD = 73, MINB = 1;
    static constexpr bool GW = true, GG = false;
    static constexpr int MQ = 6, MB = 2, MP = 6;
    static constexpr bool AUG = false;
    static constexpr int LPC = 4, RPL = 18, SR = 9, SC = 2;
};
// N <= 144 (up to the 12x12 lattice, number-conserving): G, U, both
// workspaces and a product scratch in HBM after the chain's arena (L2-resident
// while the chain runs), one CTA of 512 threads per SM.  Neither shared memory
// nor the register file holds these n x n matrices, so products stage panels
// out of place and the QR runs on a column-major copy, one warp per column with RW
// rows per lane (linalg_big.cuh).
static_assert(kTcPer * 512 >= 144 * kTcKC, "tensor-core staging: elements per thread must cover a chunk");
template <> struct Cfg<144> {
    static constexpr int THREADS = 512, MAXE = 41, KB = 8, LD = 145, MINB = 1;
    static constexpr bool GW = true, GG = true;
    static constexpr bool AUG = false;
    static constexpr int RW = 5, SR = 18, SC = 1;
};
template <int NMAX>
constexpr bool mma_fits() {   // the CTA's warps hold every tile of a product
    using C = Cfg<NMAX>;
    if constexpr (C::GG) return true;
    else return C::MQ * (C::THREADS / 32) >= mma_tiles(NMAX) && C::MP * (C::THREADS / 32) >= mma_tiles(NMAX);
}
template <int NMAX>
constexpr bool qr_fits() {
    using C = Cfg<NMAX>;
    if constexpr (C::GG) return C::RW * 32 >= NMAX && C::THREADS >= NMAX && C::GW;
    else return C::LPC * C::RPL >= NMAX && ((NMAX * C::LPC + 31) / 32) * 32 <= C::THREADS;
}
template <int NMAX>
constexpr bool cfg_ok() {
    using C = Cfg<NMAX>;
    return mma_fits<NMAX>() && qr_fits<NMAX>() && C::MAXE * C::THREADS >= NMAX * NMAX && C::SR * 8 >= NMAX &&
           kSeqElems<C::SR> <= 2 * C::KB * (NMAX + 1) &&
           (C::LD & 1) == 1 && C::LD >= NMAX;
}
static_assert(cfg_ok<16>() && cfg_ok<36>() && cfg_ok<72>() && cfg_ok<144>(),
              "class tiles and register layouts must cover NMAX");

// Dynamic shared memory of the sweep kernels.  Every buffer sits at a
// compile-time offset, so device code addresses it without holding pointers.
extern __shared__ __align__(16) unsigned char bq_smem[];

template <int NMAX>
struct Smem {
    static constexpr int kRed = 32 * (Cfg<NMAX>::THREADS / 32);
    static constexpr size_t MM = sizeof(cplx) * NMAX * Cfg<NMAX>::LD, VC = sizeof(cplx) * NMAX, VD = sizeof(double) * NMAX;
    static constexpr bool GW = Cfg<NMAX>::GW;   // workspaces in HBM
    static constexpr bool GG = Cfg<NMAX>::GG;   // G and U in HBM as well
    static constexpr size_t oG = 0, oU = MM, oW1 = 2 * MM, oW2 = 3 * MM;
    static constexpr int KB = Cfg<NMAX>::KB;
    // block vectors X and Y, at an odd stride: the mma fragments over slots and rows fall in distinct banks (mma64.cuh)
    static constexpr int VS = NMAX + 1;
    static constexpr size_t BV = sizeof(cplx) * VS * KB, BB = sizeof(cplx) * KB * KB;
    static constexpr size_t oTau = (GG ? 0 : (GW ? 2 : 4)) * MM, oCol = oTau + VC, oRow = oCol + BV;
    static constexpr size_t oXb = oRow + BV, oYb = oXb + BB, oSnap = oYb + BB, oFld = oSnap + BB, oDelta = oFld + VC;
    static constexpr size_t oDelta2 = oDelta + VC;
    static constexpr size_t oEao = oDelta2 + VC, oEan = oEao + VC, oEbo = oEan + VC, oEbn = oEbo + VC;
    static constexpr size_t oPh = oEbn + VC, oCoef = oPh + VC;
    static constexpr size_t oP = oCoef + 2 * KB * sizeof(cplx);
    static constexpr size_t oRg = oP + ((sizeof(PointDev) + 15) / 16) * 16;
    static constexpr size_t oU2 = oRg + VD, oPhin = oU2 + VD, oVn1 = oPhin + VD, oVn2 = oVn1 + VD, oD = oVn2 + VD;
    static constexpr size_t oRed = oD + VD, oObs = oRed + sizeof(double) * kRed;
    static constexpr size_t oPiv = oObs + sizeof(double) * (kObsScalars + NMAX);
    static constexpr size_t oIpiv = oPiv + sizeof(int) * NMAX, oAccf = oIpiv + sizeof(int) * NMAX;
    static constexpr size_t oSeed = oAccf + sizeof(int) * NMAX;
    static constexpr size_t oSxy = oSeed + 16;   // site coordinates x | y << 16
    static constexpr size_t oCnt = oSxy + ((sizeof(int) * NMAX + 15) / 16) * 16;   // nacc[2], nc[2], nobs of the sweep
    // tensor-core staging (classes with Cfg::GG): A hi | A lo | B hi | B lo, then
    // the MMA barrier, the tensor-memory base, the barrier parity and the on flag
    static constexpr size_t oMs = oCnt + 48;   // per warp, 16 sums over the sweep's measurements
    static constexpr size_t oEnd = oMs + 16 * sizeof(double) * (Cfg<NMAX>::THREADS / 32);
    static constexpr size_t oTc = ((oEnd + 127) / 128) * 128;
    static constexpr size_t oTcBar = oTc + 2 * kTcABytes + 2 * kTcBBytes;
    static constexpr size_t bytes() { return GG ? oTcBar + 32 : oEnd; }

    template <class T>
    static DEVI T* at(size_t off) { return reinterpret_cast<T*>(bq_smem + off); }
    DEVI cplx* G() const { return at<cplx>(oG); }
    DEVI cplx* U() const { return at<cplx>(oU); }
    DEVI cplx* W1() const { return at<cplx>(oW1); }   // shared-memory workspaces (N <= 36 classes)
    DEVI cplx* W2() const { return at<cplx>(oW2); }
    DEVI cplx* tau() const { return at<cplx>(oTau); }
    DEVI cplx* col(int m) const { return at<cplx>(oCol) + m * VS; }   // X of slot m of a block
    DEVI cplx* row(int m) const { return at<cplx>(oRow) + m * VS; }   // Y of slot m
    DEVI cplx* xb() const { return at<cplx>(oXb); }   // X and Y of a block on its own slots, [m][slot]
    DEVI cplx* yb() const { return at<cplx>(oYb); }
    DEVI double* fld() const { return at<double>(oFld); }   // fields of the slice under update, [site][channel]
    DEVI cplx* snap() const { return at<cplx>(oSnap); }   // submatrix of G at the start of the next block
    DEVI cplx* delta() const { return at<cplx>(oDelta); }
    DEVI cplx* delta2() const { return at<cplx>(oDelta2); }   // Nambu: Delta of the c^dagger index
    DEVI cplx* eao() const { return at<cplx>(oEao); }
    DEVI cplx* ean() const { return at<cplx>(oEan); }
    DEVI cplx* ebo() const { return at<cplx>(oEbo); }
    DEVI cplx* ebn() const { return at<cplx>(oEbn); }
    DEVI cplx* ph() const { return at<cplx>(oPh); }
    DEVI cplx* coef() const { return at<cplx>(oCoef); }
    DEVI PointDev* P() const { return at<PointDev>(oP); }
    DEVI double* rg() const { return at<double>(oRg); }
    DEVI double* u2() const { return at<double>(oU2); }
    DEVI double* phin() const { return at<double>(oPhin); }
    DEVI double* vn1() const { return at<double>(oVn1); }
    DEVI double* vn2() const { return at<double>(oVn2); }
    DEVI double* d() const { return at<double>(oD); }
    DEVI double* red() const { return at<double>(oRed); }
    DEVI double* obs() const { return at<double>(oObs); }
    DEVI int* piv() const { return at<int>(oPiv); }
    DEVI int* ipiv() const { return at<int>(oIpiv); }
    DEVI int* accf() const { return at<int>(oAccf); }
    DEVI uint32_t* seed() const { return at<uint32_t>(oSeed); }
    DEVI int* sxy() const { return at<int>(oSxy); }
    DEVI long long* cnt() const { return at<long long>(oCnt); }
    DEVI double* msum() const { return at<double>(oMs); }
    DEVI unsigned char* stage() const { return at<unsigned char>(oTc); }   // of the FP64 products
    DEVI uint64_t* tc_mbar() const { return at<uint64_t>(oTcBar); }
    DEVI uint32_t* tc_slot() const { return at<uint32_t>(oTcBar + 8); }
    DEVI uint32_t* tc_phase() const { return at<uint32_t>(oTcBar + 12); }
    DEVI int* tc_on() const { return at<int>(oTcBar + 16); }
    DEVI uint32_t* tc_pending() const { return at<uint32_t>(oTcBar + 20); }   // 2 + parity of a group left in flight
    DEVI int* tc_test() const { return at<int>(oTcBar + 24); }                // the wait-test mode of the products
    DEVI TcBufs tcb() const {
        return TcBufs{at<uint32_t>(oTc), at<uint32_t>(oTc + kTcABytes), at<uint32_t>(oTc + 2 * kTcABytes),
                      at<uint32_t>(oTc + 2 * kTcABytes + kTcBBytes), tc_mbar(), *tc_slot()};
    }
    DEVI QRScratch qr() const { return QRScratch{tau(), piv(), ipiv(), vn1(), vn2(), d(), col(0), col(1),
                         reinterpret_cast<long long*>(col(2)), reinterpret_cast<double*>(col(3)), reinterpret_cast<int*>(col(4))}; }
};

// green_from_M keeps n complex reciprocals in vn1 | vn2
static_assert(Smem<16>::oVn1 % 16 == 0 && Smem<36>::oVn1 % 16 == 0 && Smem<72>::oVn1 % 16 == 0 &&
                  Smem<144>::oVn1 % 16 == 0 &&
                  Smem<16>::oVn2 == Smem<16>::oVn1 + 8 * 16 && Smem<36>::oVn2 == Smem<36>::oVn1 + 8 * 36 &&
                  Smem<72>::oVn2 == Smem<72>::oVn1 + 8 * 72 && Smem<144>::oVn2 == Smem<144>::oVn1 + 8 * 144,
              "vn1 | vn2 must hold NMAX aligned complex values");
template <int NMAX>
constexpr bool smem_fits() { return Cfg<NMAX>::MINB * (Smem<NMAX>::bytes() + 1024) <= 228 * 1024; }
static_assert(smem_fits<16>() && smem_fits<36>() && smem_fits<72>() && smem_fits<144>(),
              "shared memory per SM for MINB CTAs");

// Per-chain view: the chain's arena base and fields in registers, the point
// parameters in shared memory.
template <int NMAX>
struct Ctx {
    Smem<NMAX> s;
    cplx* abase;
    double* phi;
    ChainScalars* sc;
    cplx* wg;   // HBM region after the arena: W1, W2 (N > 36), then G, U and a product scratch (N > 72)
    int n;
    DEVI const PointDev& P() const { return *s.P(); }
    DEVI Arena A() const { return make_arena(abase, n); }
    DEVI cplx* W1() const {
        if constexpr (Smem<NMAX>::GW) return wg;
        else return s.W1();
    }
    DEVI cplx* W2() const {
        if constexpr (Smem<NMAX>::GW) return wg + NMAX * Cfg<NMAX>::LD;
        else return s.W2();
    }
    // e^{-dtau K} and e^{+dtau K}, real, with leading dimension ldr: in the workspaces, or where
    // those are in HBM the point's own copy, which every chain of the point shares in L2
    DEVI int ldr() const {
        if constexpr (Smem<NMAX>::GW) return P().ldr;
        else return real_ld(NMAX);
    }
    DEVI const double* RP() const {
        if constexpr (Smem<NMAX>::GW) return P().realP;
        else return reinterpret_cast<const double*>(s.W1());
    }
    DEVI const double* RM() const {
        if constexpr (Smem<NMAX>::GW) return P().realM;
        else return reinterpret_cast<const double*>(s.W2());
    }
    DEVI cplx* G() const {
        if constexpr (Smem<NMAX>::GG) return wg + 2 * NMAX * Cfg<NMAX>::LD;
        else return s.G();
    }
    DEVI cplx* U() const {
        if constexpr (Smem<NMAX>::GG) return wg + 3 * NMAX * Cfg<NMAX>::LD;
        else return s.U();
    }
    DEVI cplx* S() const { return wg + 4 * NMAX * Cfg<NMAX>::LD; }   // product scratch (HBM-resident classes)
};

static_assert(kBigStage <= 2 * kTcABytes + 2 * kTcBBytes, "the staging buffers of both kinds of product share one region");

// ---------------------------------------------------------------------------
// Linear algebra per size class: the register-resident 8-lane-segment
// routines of linalg.cuh for the shared-memory classes, the warp-per-column
// routines of linalg_big.cuh (out of place through x.S()) for the HBM class.
template <int NMAX>
DEVI void gemm_any(Ctx<NMAX>& x, cplx* C, MatOp A, MatOp B, int tri = TRI_NONE) {
    using C_ = Cfg<NMAX>;
    if constexpr (C_::GG) {
        const bool alias = C == A.p || C == B.p;   // the product is out of place
        gemm_big<PROD_CC>(x.n, C_::LD, alias ? x.S() : C, A, B, nullptr, 0, tri, x.s.stage());
        if (alias) copy_mat(x.n, C_::LD, C, x.S());
    } else {
        gemm_rs<C_::MQ, C_::MB, !C_::GW>(x.n, C_::LD, C, A, B, tri);
    }
}
// Y <- X R (RIGHT_REAL) or R X with Y apart from X (HBM-resident classes)
template <int NMAX, bool RIGHT_REAL>
DEVI void gemm_real_out(Ctx<NMAX>& x, cplx* Y, const cplx* X, const double* R) {
    constexpr int LD = Cfg<NMAX>::LD;
    gemm_big<RIGHT_REAL ? PROD_REAL_R : PROD_REAL_L>(x.n, LD, Y, MatOp{}, RIGHT_REAL ? MatOp{X, 1, LD, 0} : op_n(X, LD), R,
                                                     x.ldr(), TRI_NONE, x.s.stage());
}
// X <- X R (RIGHT_REAL) or R X, and X2 alike if given
template <int NMAX, bool RIGHT_REAL>
DEVI void gemm_real_any(Ctx<NMAX>& x, cplx* X, const double* R, cplx* X2 = nullptr) {
    using C_ = Cfg<NMAX>;
    if constexpr (C_::GG) {
        gemm_real_out<NMAX, RIGHT_REAL>(x, x.S(), X, R);
        copy_mat(x.n, C_::LD, X, x.S());
        if (X2) gemm_real_any<NMAX, RIGHT_REAL>(x, X2, R);
    } else {
        // both in one call if the CTA's warps hold both results (they wait in registers)
        const bool two = X2 && 2 * mma_tiles(x.n) > C_::MP * (C_::THREADS / 32);
        gemm_smem_real<C_::MP, 2, RIGHT_REAL, !C_::GW>(x.n, C_::LD, x.ldr(), X, R, two ? nullptr : X2);
        if (two) gemm_smem_real<C_::MP, 2, RIGHT_REAL, !C_::GW>(x.n, C_::LD, x.ldr(), X2, R, nullptr);
    }
}
template <int NMAX>
DEVI void qrp_any(Ctx<NMAX>& x, cplx* A) {
    using C_ = Cfg<NMAX>;
    if constexpr (C_::GG) {
        // factorised in a column-major copy in S
        const int n = x.n;
        const uint32_t dm = div_magic(n);
        cplx* S = x.S();
        for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
            const int r = div_by(e, dm), c = e - r * n;
            S[c * C_::LD + r] = A[r * C_::LD + c];
        }
        __syncthreads();
        qrp_big<C_::RW>(n, C_::LD, S, x.s.qr());
        for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
            const int r = div_by(e, dm), c = e - r * n;
            A[r * C_::LD + c] = S[c * C_::LD + r];
        }
        __syncthreads();
    } else {
        qr_columns<C_::LPC, C_::RPL, false>(x.n, C_::LD, A, x.s.qr(), MatOp{}, MatOp{});
    }
}
// The pivoted QR of A, and out <- Q^H in (the identity if in.p is null): carried along in the
// classes with Cfg::AUG, from A's reflectors in the others.
template <int NMAX>
DEVI void qr_any(Ctx<NMAX>& x, cplx* A, MatOp in, MatOp out) {
    using C_ = Cfg<NMAX>;
    if constexpr (C_::AUG) {
        qr_columns<C_::LPC, C_::RPL, true>(x.n, C_::LD, A, x.s.qr(), in, out);
    } else {
        qrp_any(x, A);
        seq_apply<SEQ_QH, C_::SR, C_::SC>(x.n, C_::LD, A, x.s.tau(), nullptr, nullptr, in, out, x.s.col(0));
    }
}
// out <- P R^{-1} D^{-1} in for the factorisation in F (ZTRSM after the scaling, ZLAPMR)
template <int NMAX>
DEVI void solve_any(Ctx<NMAX>& x, const cplx* F, MatOp in, MatOp out) {
    using C_ = Cfg<NMAX>;
    cplx* rinv = reinterpret_cast<cplx*>(x.s.vn1());   // vn1 | vn2, n complex
    diag_inverse(x.n, C_::LD, F, x.s.d(), rinv, x.s.u2());
    seq_apply<SEQ_SOLVE, C_::SR, C_::SC>(x.n, C_::LD, F, rinv, x.s.u2(), x.s.piv(), in, out, x.s.col(0));
}
template <int NMAX>
DEVI void conj_transpose_any(Ctx<NMAX>& x, cplx* A) {
    using C_ = Cfg<NMAX>;
    if constexpr (C_::GG) conj_transpose_big(x.n, C_::LD, A, x.S());
    else conj_transpose_inplace<C_::MAXE>(x.n, C_::LD, A);
}

// One slice product in place: X <- X R (RIGHT) or X <- R X, R = e^{-+dtau K}
// real.  With the mixed-precision option on, classes with tensor-core staging
// run it as tc_product; a product that did not complete within its wait bound
// leaves X unchanged, flags the chain (status bit 2) and the kernel continues
// in FP64 (the tensor cores stay off for the rest of the launch, so the MMA
// barrier's parity bookkeeping is not used again).
template <int NMAX, bool RIGHT>
DEVI void slice_mult(Ctx<NMAX>& x, cplx* X, const double* R) {
    if constexpr (Cfg<NMAX>::GG) {
        if (*x.s.tc_on()) {
            if (tc_product(x.n, Cfg<NMAX>::LD, X, R, x.ldr(), RIGHT, x.s.tcb(), x.s.tc_phase(), *x.s.tc_test() != 0,
                           x.s.tc_pending()))
                return;
            if (threadIdx.x == 0) {
                *x.s.tc_on() = 0;
                x.sc->status |= 4;
            }
            __syncthreads();
        }
    }
    gemm_real_any<NMAX, RIGHT>(x, X, R);
}

// Tensor memory and the MMA barrier of a CTA that runs mixed-precision products
// (one CTA per SM in the classes with Cfg::GG): allocated after set-up, freed at exit.
template <int NMAX>
DEVI void tc_begin(Ctx<NMAX>& x, const KernelArgs& ka) {
    if constexpr (Cfg<NMAX>::GG) {
        if (threadIdx.x == 0) {
            *x.s.tc_on() = ka.mixed ? 1 : 0;
            *x.s.tc_phase() = 0;
            *x.s.tc_pending() = 0;
            *x.s.tc_test() = ka.mixed == 2 ? 1 : 0;
        }
        if (ka.mixed) {
            if (threadIdx.x < 32) tmem_alloc(smem_u32(x.s.tc_slot()), kTcCols);
            if (threadIdx.x == 0) mbar_init(smem_u32(x.s.tc_mbar()), 1);
            tc_fence_before();
        }
        __syncthreads();
        if (ka.mixed) tc_fence_after();
    }
}
// The tensor memory is released only after every MMA group the CTA issued has
// completed: a group that a product gave up on gets one more bounded wait here;
// if it still has not arrived the chain's status gets bit 3.
template <int NMAX>
DEVI void tc_end(Ctx<NMAX>& x, const KernelArgs& ka) {
    if constexpr (Cfg<NMAX>::GG) {
        if (ka.mixed) {
            tc_fence_before();
            __syncthreads();
            const uint32_t pend = *x.s.tc_pending();
            if (pend) {
                const bool done = mbar_wait(smem_u32(x.s.tc_mbar()), pend - 2u);
                if (threadIdx.x == 0 && !done) x.sc->status |= 8;
                __syncthreads();
            }
            tc_fence_after();
            if (threadIdx.x < 32) tmem_dealloc(*x.s.tc_slot(), kTcCols);
        }
    }
}

// ---------------------------------------------------------------------------
// small CTA helpers
DEVI void gcopy(cplx* dst, const cplx* src, int count) {
    for (int e = threadIdx.x; e < count; e += blockDim.x) dst[e] = src[e];
}
// identity in an n x n matrix with leading dimension ld
DEVI void set_identity(int n, int ld, cplx* A) {
    const uint32_t dm = div_magic(n);
    for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
        const int r = div_by(e, dm), c = e - r * n;
        A[r * ld + c] = cmk(r == c ? 1.0 : 0.0, 0.0);
    }
}
// dense n x n (global) <-> shared n x n with leading dimension ld
DEVI void sload(int n, int ld, cplx* dst, const cplx* src) {
    const uint32_t dm = div_magic(n);
    for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
        const int r = div_by(e, dm), c = e - r * n;
        dst[r * ld + c] = src[e];
    }
}
DEVI void sstore(int n, int ld, cplx* dst, const cplx* src) {
    const uint32_t dm = div_magic(n);
    for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
        const int r = div_by(e, dm), c = e - r * n;
        dst[e] = src[r * ld + c];
    }
}
DEVI void scopy(int n, int ld, cplx* dst, const cplx* src) {
    const uint32_t dm = div_magic(n);
    for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
        const int r = div_by(e, dm), c = e - r * n;
        dst[r * ld + c] = src[r * ld + c];
    }
}

// e^{-dtau K} (real) into W1 and e^{+dtau K} into W2 as doubles with the
// matrices' leading dimension.
DEVI void sload_real(int n, int ld, double* dst, const cplx* src) {
    const uint32_t dm = div_magic(n);
    for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
        const int r = div_by(e, dm), c = e - r * n;
        dst[r * ld + c] = src[e].x;
    }
}
template <int NMAX>
DEVI void load_expT(Ctx<NMAX>& x) {
    if constexpr (!Cfg<NMAX>::GW) {
        sload_real(x.n, x.ldr(), reinterpret_cast<double*>(x.W1()), x.P().expP);
        sload_real(x.n, x.ldr(), reinterpret_cast<double*>(x.W2()), x.P().expM);
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// local update of one channel over all sites of one slice, fused with the
// V-wrap of G (LocalU_prop_L / LocalU_prop_R, localU.f90:79-113, and
// LocalU_metro, localU.f90:31-77).
//
// Sites are strictly sequential.  The terms are the reference's updates; only the
// order of the additions changes.

// e^{+alpha phi} and e^{-alpha phi} for the HS coupling alpha = ar + i ai of one
// channel, which the reference makes purely real (U2) or purely imaginary (U1)
// (operator_Hubbard.f90:36-43): a real alpha needs only exp, an imaginary one
// one sincos with e^{-i theta} = conj(e^{i theta}).
DEVI void hs_factors(double ar, double ai, double p, cplx& ep, cplx& em) {
    if (ai == 0.0) {
        ep = cmk(exp(ar * p), 0.0);
        em = cmk(exp(-(ar * p)), 0.0);
    } else if (ar == 0.0) {
        double sn, cs;
        sincos(ai * p, &sn, &cs);
        ep = cmk(cs, sn);
        em = cmk(cs, -sn);
    } else {
        ep = cexpz(cmk(ar * p, ai * p));
        em = cexpz(cmk(-(ar * p), -(ai * p)));
    }
}
// e_new / e_old for those factors: a real quotient, or e_new conj(e_old) on the unit circle.
DEVI cplx ratio_unit(double ar, double ai, cplx en, cplx eo) {
    if (ai == 0.0) return cmk(en.x / eo.x, 0.0);
    if (ar == 0.0) return cmulcj(en, eo);
    return cdiv(en, eo);
}

// prop_channel visits the sites of a channel in blocks of KB slots, one slot per
// site of a number-conserving chain and two (b_i, c^dagger_i) per site of a
// Nambu chain.  Per block:
//  1. lead_block: one warp makes the block's Metropolis decisions in visiting
//     order on the block's kb x kb submatrix of G, held in registers, applying
//     each accepted term to the submatrix (no barrier per site);
//  2. block_vectors: the full update vectors of the block from the recorded
//     coefficients and block values;
//  3. rank_tiles: G += sum_m X_m Y_m^T on every element.
// Number-conserving (localU.f90:56-71, ZGERU): the rank-1 term of site i is
// G <- G + coef G(:,i) (e_i - G(i,:))^T.  Nambu (src/pairing/src/localU.f90:33-149
// on the {b, c^dagger} block): the reference forms the 4x4 P = I + Delta (I -
// G[isec,isec]) over the sectors of the site, takes ratio_det = det(P)^(-1/2), and
// on acceptance G -= G[:,isec] P^{-1} Delta (I[isec,:] - G[isec,:]).  P splits into
// the 2x2 block P1 on s = (i, Ns+i) and its complex conjugate, so det(P) = |det P1|^2
// (real and positive: the phase that PhaseCounter records is zero), and the block's
// term is the rank-2 G1 -= G1[:,s] P1^{-1} D1 (I[s,:] - G1[s,:]).
// For any diagonal E both satisfy F_i(E G E^-1) = E F_i(G) E^-1, and the ratio is
// that of G (a Nambu P1 becomes E P1 E^-1), so the wraps of the sites (row i by
// e^{a phi_i}, column i by e^{-a phi_i} before the decision in the right traversal,
// with the old field; row i by e^{-a phi_i} and column i by e^{a phi_i} after it in
// the left traversal, with the final field) commute with the updates and are
// applied once, as one diagonal similarity, in the last block's rank pass.
//
// Eight slots a block: what a block costs besides its decisions (two barriers, the
// vectors, the pass's loads and stores of G) is paid per eight slots, and the
// decisions (a chain of shuffle, ratio, reciprocal and update per site) run beside
// the pass, which takes the FP64 tensor pipe.  Bound: the decisions (about 300 cycles
// a site on their own) and the vectors (1.3 K cycles a block).  Against blocks of four
// with a DFMA pass (number-conserving) and one barrier per site with every thread
// keeping its elements (Nambu), M cycles of updates per sweep of a chain: 6x6 Nambu
// block, L = 40, one CTA per SM 89 -> 13.4; 4x4 Nambu, two CTAs 12.8 -> 5.7; 8x8,
// L = 40 24.0 -> 9.6; 12x12, L = 50 181 -> 137; 6x6, L = 160, two CTAs 26.2 -> 25.6.
static_assert(Cfg<16>::KB == 8 && Cfg<36>::KB == 8 && Cfg<72>::KB == 8 && Cfg<144>::KB == 8,
              "the lead warp holds the block's 8 x 8 submatrix, two rows per lane");

// matrix index of slot k of the block that starts at the k0-th visited site
template <bool LEFT, bool PAIR>
DEVI int slot_index(int ns, int k0, int k) {
    const int m = k0 + (PAIR ? k >> 1 : k);
    return (LEFT ? ns - 1 - m : m) + (PAIR && (k & 1) ? ns : 0);
}

// the channel's deferred wrap: factor of row r and of column c
template <int NMAX, bool LEFT, bool PAIR>
DEVI cplx wrap_row(const Ctx<NMAX>& x, int r, bool flip) {
    const auto& s = x.s;
    const bool cd = PAIR && r >= x.P().Ns;
    const int i = cd ? r - x.P().Ns : r;
    const bool up = (cd && flip) != !LEFT;   // e^{+alpha phi} rather than e^{-alpha phi}
    if constexpr (LEFT) return s.accf()[i] ? (up ? s.ean()[i] : s.ebn()[i]) : (up ? s.eao()[i] : s.ebo()[i]);
    else return up ? s.eao()[i] : s.ebo()[i];
}
template <int NMAX, bool LEFT, bool PAIR>
DEVI cplx wrap_col(const Ctx<NMAX>& x, int c, bool flip) {
    const auto& s = x.s;
    const bool cd = PAIR && c >= x.P().Ns;
    const int i = cd ? c - x.P().Ns : c;
    const bool up = (cd && flip) != LEFT;
    if constexpr (LEFT) return s.accf()[i] ? (up ? s.ean()[i] : s.ebn()[i]) : (up ? s.eao()[i] : s.ebo()[i]);
    else return up ? s.eao()[i] : s.ebo()[i];
}

// the submatrix at block start k0 into snap(); the lead warp reads it back after
// the barrier, when the rank pass may already be writing G
template <int NMAX, bool LEFT, bool PAIR>
DEVI void block_snapshot(const Ctx<NMAX>& x, const cplx* G, int k0, int kb) {
    constexpr int KB = Cfg<NMAX>::KB, LD = Cfg<NMAX>::LD;
    const int lane = threadIdx.x & 31, ns = x.P().Ns;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int a = (lane >> 3) + 4 * h, b = lane & 7;
        cplx v = cmk(0.0, 0.0);
        if (a < kb && b < kb) v = G[slot_index<LEFT, PAIR>(ns, k0, a) * LD + slot_index<LEFT, PAIR>(ns, k0, b)];
        x.s.snap()[a * KB + b] = v;
    }
}

DEVI cplx shfl_c(cplx v, int src) {
    return cmk(__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src));
}

// Step 1, by the lead warp (warp 0 of the CTA).  Lane l holds the elements
// (l / 8, l % 8) and (l / 8 + 4, l % 8) of the block's submatrix: the snapshot plus
// the previous block's kbp terms (to rounding the G that the pass writes there).
// The decisions run in visiting order, every lane computing the same ratio from the
// elements it receives by shuffle.  Records per slot m: the coefficients (coef()),
// X_m on the later block slots (xb, [m][a], a > m) and Y_m on them (yb, [m][b], b > m),
// where X_m = coef G_{m-1}(:, i_m) and Y_m = e_{i_m} - G_{m-1}(i_m, :)^T (Nambu: the
// two columns of -G[:,s] P1^{-1} D1 and the two rows of I[s,:] - G[s,:]).  Nothing
// later reads the submatrix or the records at slots up to m, so every lane updates
// and stores without a condition (lanes of one address hold one value): a divergent
// branch costs about what the arithmetic of a site does.  A rejected site has zero coefficients, so its update adds exact zeros.  The accept
// test r_g |ratio_det|^2 > u is taken as r_g > u |det|^2, which needs no division.
// Returns the accepted count.
template <int NMAX, bool LEFT, bool PAIR>
COLD long long lead_block(Ctx<NMAX> x, int k0, int kb, int kbp) {
    constexpr int KB = Cfg<NMAX>::KB;
    const auto& s = x.s;
    const int lane = threadIdx.x & 31, ns = uni(x.P().Ns);
    const int b = lane & 7, a0 = lane >> 3;
    k0 = uni(k0);
    kb = uni(kb);
    kbp = uni(kbp);
    cplx *xb = s.xb(), *yb = s.yb();
    cplx g[2];
    const int ib = slot_index<LEFT, PAIR>(ns, k0, min(b, kb - 1));
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int a = a0 + 4 * h;
        g[h] = s.snap()[a * KB + b];
        const int ia = slot_index<LEFT, PAIR>(ns, k0, min(a, kb - 1));
        if (kbp > 0) {   // all KB slots: block_vectors zeroes those that a short block does not have
            cplx t = cmk(0.0, 0.0);   // two chains: slots 0..3 onto g, 4..7 onto t
#pragma unroll
            for (int m = 0; m < KB / 2; ++m) {
                g[h] = cfma(s.col(m)[ia], s.row(m)[ib], g[h]);
                t = cfma(s.col(m + KB / 2)[ia], s.row(m + KB / 2)[ib], t);
            }
            g[h] = cadd(g[h], t);
        }
    }
    long long nacc = 0;
    if constexpr (!PAIR) {
        int i = slot_index<LEFT, PAIR>(ns, k0, 0);
        cplx d = s.delta()[i];
        double rg = s.rg()[i], u = s.u2()[i];
#pragma unroll
        for (int m = 0; m < KB; ++m) {
            if (m >= kb) break;
            const int src = (m & 3) << 3, hm = m >> 2;
            const cplx gmm = shfl_c(g[hm], src | m);
            const cplx gmb = shfl_c(g[hm], src | b);
            cplx gam[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) gam[h] = shfl_c(g[h], (lane & 24) | m);
            // w = 1 + Delta (1 - G_ii), coef = -Delta / w on acceptance (localU.f90:56-71)
            const cplx w = cmk(1.0 + (d.x * (1.0 - gmm.x) + d.y * gmm.y), d.y * (1.0 - gmm.x) - d.x * gmm.y);
            const double w2 = w.x * w.x + w.y * w.y;
            const bool accept = rg > u * w2;
            const double inv = rcp_fast(w2);
            const cplx t = cmulcj(d, w);   // Delta * conj(w)
            const cplx coef = cmk(accept ? -t.x * inv : 0.0, accept ? -t.y * inv : 0.0);
            const int ni = slot_index<LEFT, PAIR>(ns, k0, min(m + 1, kb - 1));
            d = s.delta()[ni];   // the next site's proposal, before this site's stores
            rg = s.rg()[ni];
            u = s.u2()[ni];
            const cplx yv = cmk(-gmb.x, -gmb.y);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const cplx xv = cmul(coef, gam[h]);
                g[h] = cfma(xv, yv, g[h]);
                xb[m * KB + a0 + 4 * h] = xv;
            }
            yb[m * KB + b] = yv;
            s.accf()[i] = accept ? 1 : 0;
            s.coef()[m] = coef;
            nacc += accept ? 1 : 0;
            i = ni;
        }
    } else {
#pragma unroll 1
        for (int m = 0; 2 * m < kb; ++m) {
            const int i = slot_index<LEFT, PAIR>(ns, k0, 2 * m);
            const cplx d0 = s.delta()[i], d1 = s.delta2()[i];
            const double rg = s.rg()[i], u = s.u2()[i];
            const int p = 2 * m, q = p + 1, sp = (p & 3) << 3, sq = (q & 3) << 3;
            const cplx gm = p < 4 ? g[0] : g[1];
            const cplx gaa = shfl_c(gm, sp | p), gab = shfl_c(gm, sp | q);
            const cplx gba = shfl_c(gm, sq | p), gbb = shfl_c(gm, sq | q);
            const cplx gpb = shfl_c(gm, sp | b), gqb = shfl_c(gm, sq | b);
            cplx gap[2], gaq[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                gap[h] = shfl_c(g[h], (lane & 24) | p);
                gaq[h] = shfl_c(g[h], (lane & 24) | q);
            }
            // P1 = I + D1 (I - G1[s,s]);  accept if |rg rc| > u |det P1|
            const cplx p00 = cadd(cmk(1.0, 0.0), cmul(d0, cmk(1.0 - gaa.x, -gaa.y)));
            const cplx p01 = cmul(d0, cmk(-gab.x, -gab.y));
            const cplx p10 = cmul(d1, cmk(-gba.x, -gba.y));
            const cplx p11 = cadd(cmk(1.0, 0.0), cmul(d1, cmk(1.0 - gbb.x, -gbb.y)));
            const cplx det = csub(cmul(p00, p11), cmul(p01, p10));
            const double det2 = det.x * det.x + det.y * det.y;
            const bool accept = rg > u * sqrt(det2);
            const double rr = rcp_fast(det2), inv = accept ? rr : 0.0;
            // -M, M = P1^{-1} D1, P1^{-1} = adj(P1) conj(det) / |det|^2
            const cplx id = cmk(-det.x * inv, det.y * inv);
            const cplx e0 = cmul(id, d0), e1 = cmul(id, d1);
            const cplx m00 = cmul(p11, e0), m01 = cmul(cmk(-p01.x, -p01.y), e1);
            const cplx m10 = cmul(cmk(-p10.x, -p10.y), e0), m11 = cmul(p00, e1);
            const cplx yp = cmk(-gpb.x, -gpb.y), yq = cmk(-gqb.x, -gqb.y);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int a = a0 + 4 * h;
                const cplx xp = cfma(gaq[h], m10, cmul(gap[h], m00)), xq = cfma(gaq[h], m11, cmul(gap[h], m01));
                g[h] = cfma(xq, yq, cfma(xp, yp, g[h]));
                xb[p * KB + a] = xp;
                xb[q * KB + a] = xq;
            }
            yb[p * KB + b] = yp;
            yb[q * KB + b] = yq;
            s.accf()[i] = accept ? 1 : 0;
            s.coef()[4 * m] = m00;
            s.coef()[4 * m + 1] = m01;
            s.coef()[4 * m + 2] = m10;
            s.coef()[4 * m + 3] = m11;
            nacc += accept ? 1 : 0;
        }
    }
    return nacc;
}

// Step 2.  The update vectors on every row and column, from the block's starting G:
// g_k(r) = G(r, i_k) + sum_{j<k} X_j(r) Y_j(i_k) gives X_k into col(k), and
// G(i_k, c) + sum_{j<k} X_j(i_k) Y_j(c) gives Y_k into row(k) (j over the slots of
// earlier sites).  Whole warps build the X rows, the next ones the Y columns.
template <int NMAX, bool LEFT, bool PAIR>
DEVI void block_vectors(const Ctx<NMAX>& x, const cplx* G, int n, int k0, int kb) {
    constexpr int KB = Cfg<NMAX>::KB, LD = Cfg<NMAX>::LD, W = PAIR ? 2 : 1;
    const auto& s = x.s;
    const cplx *xb = s.xb(), *yb = s.yb();
    const int ns = x.P().Ns;
    const int n32 = (n + 31) & ~31;
    kb = uni(kb);
    for (int t = threadIdx.x; t < 2 * n32; t += blockDim.x) {
        const bool isx = uni(t) < n32;
        const int v = isx ? t : t - n32;
        const int vc = min(v, n - 1);
        const cplx* other = isx ? yb : xb;   // the other vector's values at the block's slots
        cplx acc[KB];
        // the block's rows or columns of G first: their loads overlap
#pragma unroll
        for (int k = 0; k < KB; ++k) {
            const int ik = slot_index<LEFT, PAIR>(ns, k0, min(k, kb - 1));
            acc[k] = G[isx ? vc * LD + ik : ik * LD + vc];
        }
        // a finished slot is added to all later ones at once (independent chains); slots from kb
        // on take part with what the records hold and are stored as zeros
#pragma unroll
        for (int k = 0; k < KB; k += W) {
            // X_k = coef g_k, or Y_k = e - g_k: one form for both, as a branch here would keep the
            // loads of the later slots behind it
            if constexpr (PAIR) {
                const cplx* m = s.coef() + 2 * k;
                const cplx ga = acc[k], gb = acc[k + 1];
                const cplx xa = cfma(gb, m[2], cmul(ga, m[0])), xb_ = cfma(gb, m[3], cmul(ga, m[1]));
                const double ea = v == slot_index<LEFT, PAIR>(ns, k0, k) ? 1.0 : 0.0;
                const double eb = v == slot_index<LEFT, PAIR>(ns, k0, k + 1) ? 1.0 : 0.0;
                acc[k] = cmk(isx ? xa.x : ea - ga.x, isx ? xa.y : -ga.y);
                acc[k + 1] = cmk(isx ? xb_.x : eb - gb.x, isx ? xb_.y : -gb.y);
            } else {
                const cplx c = s.coef()[k], xk = cmul(c, acc[k]);
                const double e = v == slot_index<LEFT, PAIR>(ns, k0, k) ? 1.0 : 0.0;
                acc[k] = cmk(isx ? xk.x : e - acc[k].x, isx ? xk.y : -acc[k].y);
            }
#pragma unroll
            for (int j = k; j < k + W; ++j)
#pragma unroll
                for (int l = k + W; l < KB; ++l) acc[l] = cfma(acc[j], other[j * KB + l], acc[l]);
        }
        cplx* dst = isx ? s.col(0) : s.row(0);
#pragma unroll
        for (int k = 0; k < KB; ++k) {
            const cplx w = cmk(k < kb ? acc[k].x : 0.0, k < kb ? acc[k].y : 0.0);
            if (v < n) dst[k * Smem<NMAX>::VS + v] = w;
        }
    }
}

// Step 3 on the FP64 tensor pipe: tiles of
// 8 x 8 complex elements as in prod_mma, four mma per four slots, NB tiles of a warp in
// flight; warp w of nw (the lead's scheduler excluded) takes contiguous tiles.  WRAP (the
// channel's last block): the deferred wrap.  coef() is not read (the lead warp is already
// writing the next block's).
template <int NMAX, bool LEFT, bool PAIR, bool WRAP>
DEVI void rank_tiles(const Ctx<NMAX>& x, cplx* G, int n, int w, int nw, bool flip) {
    constexpr int LD = Cfg<NMAX>::LD, KB = Cfg<NMAX>::KB;
    constexpr int NB = Cfg<NMAX>::GG ? 4 : 2;   // G in L2: more loads in flight (12x12 updates 139 -> 137 M cycles)
    const auto& s = x.s;
    n = uni(n);
    w = uni(w);
    const int lane = threadIdx.x & 31, l4 = lane & 3, l8 = lane >> 2;
    const int n8 = (n + 7) >> 3, tiles = n8 * n8;
    const int t1 = (w + 1) * tiles / nw;
    int t0 = w * tiles / nw, rt = t0 / n8, ct = t0 - rt * n8;
    for (; t0 < t1; t0 += NB) {
        double re[NB][2], im[NB][2];
        cplx a[NB][KB / 4], b[NB][KB / 4];
        int r[NB], c[NB];
#pragma unroll
        for (int q = 0; q < NB; ++q) {
            const int ra = min(tile_at(rt, l8), n - 1), cb = min(tile_at(ct, l8), n - 1);
            r[q] = t0 + q < t1 ? tile_at(rt, l8) : n;
            c[q] = 8 * ct + l4;
            const cplx g0 = G[ra * LD + min(c[q], n - 1)], g1 = G[ra * LD + min(c[q] + 4, n - 1)];
            re[q][0] = g0.x;
            re[q][1] = g1.x;
            im[q][0] = g0.y;
            im[q][1] = g1.y;
#pragma unroll
            for (int k = 0; k < KB / 4; ++k) {
                a[q][k] = s.col(4 * k + l4)[ra];   // slots from kb on hold zeros
                b[q][k] = s.row(4 * k + l4)[cb];
            }
            const bool next = ++ct == n8;
            ct = next ? 0 : ct;
            rt = min(rt + (next ? 1 : 0), n8 - 1);
        }
#pragma unroll
        for (int k = 0; k < KB / 4; ++k) {
#pragma unroll
            for (int q = 0; q < NB; ++q) {
                mma_f64(re[q][0], re[q][1], a[q][k].x, b[q][k].x);
                mma_f64(im[q][0], im[q][1], a[q][k].x, b[q][k].y);
            }
#pragma unroll
            for (int q = 0; q < NB; ++q) {
                mma_f64(re[q][0], re[q][1], -a[q][k].y, b[q][k].y);
                mma_f64(im[q][0], im[q][1], a[q][k].y, b[q][k].x);
            }
        }
#pragma unroll
        for (int q = 0; q < NB; ++q) {
            cplx g0 = cmk(re[q][0], im[q][0]), g1 = cmk(re[q][1], im[q][1]);
            if constexpr (WRAP) {
                const cplx f = wrap_row<NMAX, LEFT, PAIR>(x, min(r[q], n - 1), flip);
                g0 = cmul(cmul(g0, f), wrap_col<NMAX, LEFT, PAIR>(x, min(c[q], n - 1), flip));
                g1 = cmul(cmul(g1, f), wrap_col<NMAX, LEFT, PAIR>(x, min(c[q] + 4, n - 1), flip));
            }
            if (r[q] < n && c[q] < n) G[r[q] * LD + c[q]] = g0;
            if (r[q] < n && c[q] + 4 < n) G[r[q] * LD + c[q] + 4] = g1;
        }
    }
}

// Start the copy of a slice's fields (both channels) into shared memory: issued before the
// products or the measurement that precede the slice's updates, which hide its latency.
// A site's two values go in one 16-byte copy where the fields start on 16 bytes (every handle's
// do), in two of eight where a caller's buffer (bafqmc_sweep_noalloc) is aligned to a double only:
// eight bytes a copy for all took a 3x3 chain's sweep from 0.950 to 0.964 ms, the two forms from
// 0.958 to 0.962.
template <int NMAX>
DEVI void stage_fields(const Ctx<NMAX>& x, int slice) {
    const int ns = x.P().Ns;
    const double* src = x.phi + (long)slice * ns * 2;
    const uint32_t dst = (uint32_t)__cvta_generic_to_shared(x.s.fld());
    if (((uintptr_t)x.phi & 15) == 0) {   // then every slice is: it has an even number of doubles
        for (int i = threadIdx.x; i < ns; i += blockDim.x)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(dst + 16 * i), "l"(src + 2 * i) : "memory");
    } else {
        for (int i = threadIdx.x; i < 2 * ns; i += blockDim.x)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst + 8 * i), "l"(src + i) : "memory");
    }
}

template <int NMAX, bool LEFT, bool PAIR>
COLD void prop_channel(Ctx<NMAX> x, int ch, int slice) {
    constexpr int KB = Cfg<NMAX>::KB, LD = Cfg<NMAX>::LD, W = PAIR ? 2 : 1, SB = KB / W;   // SB sites a block
    auto& s = x.s;
    const int n = uni(x.n), ns = uni(x.P().Ns), tid = threadIdx.x;
    const double ar = x.P().alpha_re[ch], ai = x.P().alpha_im[ch];
    const double shift = fabs(x.P().shiftLoc);
    const bool flip = PAIR && x.P().flip[ch] != 0;
    const uint32_t s0 = *s.seed();
    double* phis = x.phi + (long)slice * ns * 2;
    cplx* G = x.G();

    // the slice's fields were started on their way by stage_fields
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    // per-site proposals (Nambu: opU_get_delta, src/pairing/src/operator_Hubbard.f90:100-137);
    // draw order follows the visiting order of the sites
    for (int i = tid; i < ns; i += blockDim.x) {
        const int m = LEFT ? (ns - 1 - i) : i;
        const double xflip = lcg_u(lcg_mul(c_apow[2 * m + 1], s0));
        const double rnd = lcg_u(lcg_mul(c_apow[2 * m + 2], s0));
        const double po = s.fld()[i * 2 + ch];
        const double xdif = (xflip - 0.5) * shift;
        const double pn = po + xdif;
        const double go = exp(-0.5 * po * po), gn = exp(-0.5 * pn * pn);
        cplx eo, en, ebo, ebn;
        hs_factors(ar, ai, po, eo, ebo);
        hs_factors(ar, ai, pn, en, ebn);
        s.eao()[i] = eo;
        s.ean()[i] = en;
        s.ebo()[i] = ebo;
        s.ebn()[i] = ebn;
        if constexpr (PAIR) {
            cplx ep, em;
            hs_factors(ar, ai, pn - po, ep, em);
            const cplx dp = csub(ep, cmk(1.0, 0.0));
            s.delta()[i] = dp;                                        // b_i: e^{+alpha dphi} - 1 in both channels
            s.delta2()[i] = flip ? csub(em, cmk(1.0, 0.0)) : dp;      // c^dagger_i
            // |ratio_gaussian * ratio_constant|; ratio_constant = e^{alpha(phi_old - phi_new)} for U2
            const double rc = ch == 1 ? (ai == 0.0 ? fabs(eo.x / en.x) : cabsv(cdiv(eo, en))) : 1.0;
            s.rg()[i] = (gn / go) * rc;
        } else {
            s.delta()[i] = csub(ratio_unit(ar, ai, en, eo), cmk(1.0, 0.0));
            s.rg()[i] = gn / go;
        }
        s.u2()[i] = rnd;
        s.phin()[i] = pn;
        s.accf()[i] = 0;
    }
    __syncthreads();

    // Blocks of SB sites in visiting order.  The lead warp (warp 0) decides
    // block b + 1 while the other warps run block b's rank pass: it
    // copies block b + 1's submatrix during block b's vector step (G is not
    // written then) and adds block b's terms itself.  The last block's pass applies
    // the channel's deferred wrap.
    constexpr int NT = Cfg<NMAX>::THREADS;
    const bool lead = tid == 0;
    const int warp = warp_index();
    const bool lwarp = warp == 0;
    // The lead's chain of dependent FP64 operations waits behind every mma (16 cycles) that
    // another warp has on its scheduler (warp index modulo 4), so the pass leaves the lead's
    // scheduler alone.  Every CTA of an SM decides on warp 0: their leads share one scheduler,
    // which no pass uses.  Leads spread over the schedulers wait for the other CTAs' mma: a 6x6
    // sweep of two chains an SM 25.7 ms with the pass on two schedulers only, 24.3 on three,
    // 24.1 here; 4x4 chains, 14 an SM, 20.4 against 18.3 ms.
    const int rw = (warp & 3) ? (warp >> 2) * 3 + (warp & 3) - 1 : -1;
    constexpr int NRW = NT / 32 * 3 / 4;
    long long nacc = 0;   // accepted proposals, counted by the lead
    if (lwarp) {
        const int kb = W * min(SB, ns);
        block_snapshot<NMAX, LEFT, PAIR>(x, G, 0, kb);
        __syncwarp();
        const long long c = lead_block<NMAX, LEFT, PAIR>(x, 0, kb, 0);
        if (lead) nacc += c;
    }
    __syncthreads();
    for (int k0 = 0; k0 < ns; k0 += SB) {
        const int kb = W * min(SB, ns - k0), k1 = k0 + SB, kb1 = W * min(SB, ns - k1);
        const bool more = k1 < ns;
        block_vectors<NMAX, LEFT, PAIR>(x, G, n, k0, kb);
        if (lwarp && more) block_snapshot<NMAX, LEFT, PAIR>(x, G, k1, kb1);
        __syncthreads();
        if (lwarp) {
            if (more) {
                const long long c = lead_block<NMAX, LEFT, PAIR>(x, k1, kb1, kb);
                if (lead) nacc += c;
            }
        } else if (more) {
            if (rw >= 0) rank_tiles<NMAX, LEFT, PAIR, false>(x, G, n, rw, NRW, flip);
        } else if (rw >= 0) {
            rank_tiles<NMAX, LEFT, PAIR, true>(x, G, n, rw, NRW, flip);
        }
        __syncthreads();
    }
    // accepted fields, counters, seed, and the U factor wrap with the final fields
    for (int i = tid; i < ns; i += blockDim.x)
        if (s.accf()[i]) phis[i * 2 + ch] = s.phin()[i];   // the other channel's staged values stay as they are
    if (lead) {   // AccCounter%count, kept in shared memory
        s.cnt()[ch] += nacc;
        s.cnt()[2 + ch] += ns;
        *s.seed() = lcg_mul(c_apow[2 * ns], s0);
    }
    {   // U_L columns (left) or U_R rows (right)
        constexpr int MAXE = Cfg<NMAX>::MAXE, T = Cfg<NMAX>::THREADS;
        const uint32_t dm = div_magic(n);
        cplx* U = x.U();
#pragma unroll 3
        for (int k = 0; k < MAXE; ++k) {
            const int e = min(tid + k * T, n * n - 1);   // the last threads repeat the last element without storing it
            const int r = div_by(e, dm), c = e - r * n;
            const int idx = LEFT ? c : r;
            const bool cd = PAIR && idx >= ns;
            const int site = cd ? idx - ns : idx;
            const bool acc = s.accf()[site] != 0;
            const cplx* f = cd && flip ? (acc ? s.ebn() : s.ebo()) : (acc ? s.ean() : s.eao());
            const cplx v = cmul(U[r * LD + c], f[site]);
            if (tid + k * T < n * n) U[r * LD + c] = v;
        }
    }
    __syncthreads();
}

// ---------------------------------------------------------------------------
// propT_L / propT_R (multiply.f90:72-86): G <- e^{+dK} G e^{-dK}, U_L <- U_L e^{-dK}
// for the left traversal; G <- e^{-dK} G e^{+dK}, U_R <- e^{-dK} U_R for the
// right.  e^{-dtau K} is in W1, e^{+dtau K} in W2.
template <int NMAX, bool LEFT>
COLD void slice_products(Ctx<NMAX> x) {
    auto& s = x.s;
    const int n = x.n;
    const double *P = x.RP(), *M = x.RM();   // e^{-dtau K}, e^{+dtau K}
    // G and U take the same first factor: one call for both where the products run in place
    if constexpr (Cfg<NMAX>::GG) {
        if (*s.tc_on()) {
            slice_mult<NMAX, LEFT>(x, x.G(), P);
            slice_mult<NMAX, !LEFT>(x, x.G(), M);
            slice_mult<NMAX, LEFT>(x, x.U(), P);
        } else {   // G through the scratch matrix and back: no copy
            gemm_real_out<NMAX, LEFT>(x, x.S(), x.G(), P);
            gemm_real_out<NMAX, !LEFT>(x, x.G(), x.S(), M);
            gemm_real_any<NMAX, LEFT>(x, x.U(), P);
        }
    } else {
        gemm_real_any<NMAX, LEFT>(x, x.G(), P, x.U());
        gemm_real_any<NMAX, !LEFT>(x, x.G(), M);
    }
}

// ---------------------------------------------------------------------------
// equal-time estimators (Obs_equal_calc, obser_equal.f90:95-198).  The c
// flavour's Green's function is the complex conjugate of the b flavour's
// (obser_equal.f90:112-113), so every c-flavour sum is the conjugate of the
// b-flavour sum and is not recomputed.  The K-point phase depends only on the
// displacement r = i - j, so it comes from an Lq-entry table in shared memory.
template <int NMAX>
COLD void measure(Ctx<NMAX> x) {
    constexpr int LD = Cfg<NMAX>::LD;
    auto& s = x.s;
    const PointDev& P = x.P();
    const int n = x.n, tid = threadIdx.x, lx = P.Lx, ly = P.Ly;
    const cplx* G = x.G();
    const cplx* ph = s.ph();
    const bool hasK = P.hasK;
    // v: 0 sum Re(t_up), 1 sum |Gc|^2, 2-3 sf_K, 4-5 dw_K, 6-7 sum t_up, 8-9 sum du_i conj(du_j),
    //    10 kinetic, 11 sum Re du, 12 sum |du|^2, 13 sum Re du^2
    double v[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) v[k] = 0.0;
    const int* sxy = s.sxy();
    const int T = blockDim.x;
    // a = Grup(i,j), gc = Grupc(i,j) = G(j,i) - delta_ij, du the diagonal of G - 1
    auto add = [&](int i, int j, cplx a, cplx gc, cplx dui, cplx duj) {
        const cplx tup = cadd(cmul(dui, duj), cmul(gc, a));   // b-flavour density correlator
        const cplx tud = cmulcj(dui, duj);                     // du_i * dd_j
        v[0] += tup.x;
        v[1] += gc.x * gc.x + gc.y * gc.y;
        v[6] += tup.x;
        v[7] += tup.y;
        v[8] += tud.x;
        v[9] += tud.y;
        if (hasK) {
            const int pi = sxy[i], pj = sxy[j];
            int dx = (pi & 0xffff) - (pj & 0xffff), dy = (pi >> 16) - (pj >> 16);
            dx += (dx < 0) ? lx : 0;
            dy += (dy < 0) ? ly : 0;
            const cplx p = ph[dy * lx + dx];
            const double sfr = 2.0 * gc.x;                     // Grupc + Grdoc
            const double dwr = 2.0 * tup.x + 2.0 * tud.x;      // t_up + t_do + du_i dd_j + dd_i du_j
            v[2] += p.x * sfr;
            v[3] += p.y * sfr;
            v[4] += p.x * dwr;
            v[5] += p.y * dwr;
        }
    };
    if constexpr (Cfg<NMAX>::GG) {
        // G in L2: a warp takes 8 x 4 elements, so that both orders read whole sectors (8 rows of
        // 64 bytes and 4 rows of 128; a warp along a row reads its mirror from 32 lines), and the
        // diagonal comes from shared memory: 12x12, L = 50 12.4 -> 5.9 M cycles a sweep.  Elements past
        // the edge add zeros.
        cplx* dg = s.delta();   // rewritten by the next channel's proposals
        for (int i = tid; i < n; i += T) dg[i] = cmk(G[i * LD + i].x - 1.0, G[i * LD + i].y);
        __syncthreads();
        const int lane = tid & 31, nt = (n + 3) >> 2, tiles = ((n + 7) >> 3) * nt;
        const uint32_t dt = div_magic(nt);
#pragma unroll 2
        for (int t = tid >> 5; t < tiles; t += T >> 5) {
            const int rt = div_by(t, dt);
            const int i0 = 8 * rt + (lane >> 2), j0 = 4 * (t - rt * nt) + (lane & 3);
            const int i = min(i0, n - 1), j = min(j0, n - 1);
            const bool in = i0 < n && j0 < n;
            const cplx z = cmk(0.0, 0.0), a = G[i * LD + j];
            cplx gc = G[j * LD + i];
            gc.x -= i == j ? 1.0 : 0.0;
            add(i, j, in ? a : z, in ? gc : z, in ? dg[i] : z, in ? dg[j] : z);
        }
    } else {
        const uint32_t dm = div_magic(n);
        for (int e = tid; e < n * n; e += T) {
            const int i = div_by(e, dm), j = e - i * n;
            const cplx a = G[i * LD + j];
            cplx gc = G[j * LD + i];
            if (i == j) gc.x -= 1.0;
            add(i, j, a, gc, cmk(G[i * LD + i].x - 1.0, G[i * LD + i].y), cmk(G[j * LD + j].x - 1.0, G[j * LD + j].y));
        }
    }
    for (int e = tid; e < 3 * n; e += blockDim.x) {   // bonds (x+1,y), (x,y+1), (x-1,y+1) (lattice.f90:98-111)
        const int i = e / 3, nb = e - (e / 3) * 3;
        const int ix = sxy[i] & 0xffff, iy = sxy[i] >> 16;
        const int jx = (nb == 0) ? (ix + 1) % lx : (nb == 1 ? ix : (ix + lx - 1) % lx);
        const int jy = (nb == 0) ? iy : (iy + 1) % ly;
        const int jj = jy * lx + jx;
        cplx gij = G[jj * LD + i], gji = G[i * LD + jj];   // Grupc(i,jj), Grupc(jj,i)
        if (i == jj) { gij.x -= 1.0; gji.x -= 1.0; }
        v[10] += 2.0 * (gij.x + gji.x);
    }
    for (int i = tid; i < n; i += blockDim.x) {
        const cplx du = cmk(G[i * LD + i].x - 1.0, G[i * LD + i].y);
        v[11] += du.x;
        v[12] += du.x * du.x + du.y * du.y;
        v[13] += du.x * du.x - du.y * du.y;
        s.obs()[O_SITE + i] += 2.0 * du.x;
    }
    warp_add16(v, s.msum() + 16 * (tid >> 5));
    if (tid == 0) s.cnt()[4] += 1;
}

// The sweep's sums over all measurements (every record below is linear in them) into the
// bin record's scalars.
template <int NMAX>
DEVI void measure_finish(Ctx<NMAX>& x) {
    auto& s = x.s;
    const PointDev& P = x.P();
    const double lq = (double)P.Lq, lq2 = lq * lq;
    __syncthreads();
    if (threadIdx.x == 0) {
        double v[14];
        for (int k = 0; k < 14; ++k) {
            v[k] = 0.0;
            for (int w = 0; w < Cfg<NMAX>::THREADS / 32; ++w) v[k] += s.msum()[16 * w + k];
        }
        double* o = s.obs();
        const double onsite = 2.0 * v[13] + v[11];          // sum Re(2 du^2 + du)
        const double dbl = v[12] / lq;                       // doubleOcc sample
        const double kin = P.RT * v[10] / lq;
        const double inter = (P.U1 + P.U2) * (2.0 * onsite) / lq + 2.0 * (P.U2 - P.U1) * dbl;
        o[O_DENSITY_UP] += v[11] / lq;
        o[O_DENSITY_DO] += v[11] / lq;
        o[O_DENSITY_TOTAL] += 2.0 * v[11] / lq;
        o[O_KINETIC] += kin;
        o[O_DOUBLEOCC] += dbl;
        o[O_SQUAREOCC] += 2.0 * v[13] / lq;
        o[O_NUM_UP] += v[11];
        o[O_NUM_DO] += v[11];
        o[O_NUMSQUARE_UP] += v[0];
        o[O_NUMSQUARE_DO] += v[0];
        o[O_ONSITE_N2_UP] += onsite;
        o[O_ONSITE_N2_DO] += onsite;
        o[O_INTERACTION] += inter;
        o[O_ENERGY] += kin + inter;
        o[O_PSF_GAMMA] += v[1] / lq2;
        o[O_SF_K] += v[2] / lq2;
        o[O_SF_K + 1] += v[3] / lq2;
        o[O_DW_K] += v[4] / lq2;
        o[O_DW_K + 1] += v[5] / lq2;
        o[O_DEN_UPUP] += v[6] / lq;
        o[O_DEN_UPUP + 1] += v[7] / lq;
        o[O_DEN_DODO] += v[6] / lq;
        o[O_DEN_DODO + 1] -= v[7] / lq;
        o[O_DEN_UPDO] += v[8] / lq;
        o[O_DEN_UPDO + 1] += v[9] / lq;
    }
    __syncthreads();
}

// ---------------------------------------------------------------------------
// Nambu equal-time estimators (Obs_equal_calc, src/pairing/src/obser_equal.f90:112-271)
// from the {b, c^dagger} block.  With A = G1[b,b], B = G1[b,c^dagger],
// C = G1[c^dagger,b], D = G1[c^dagger,c^dagger], the reference's sixteen
// sub-blocks are A, -B, conj(A), -conj(B), conj(C), -conj(D), C, -D and zeros:
// n_b(i) = -conj(D_ii), n_c(i) = -D_ii, and every c-flavour sum is the complex
// conjugate of the b-flavour sum.  Pair terms:
//   Dbb(i,j) = n_b(i) n_b(j) - conj(D_ij) A_ij,  Dbc(i,j) = n_b(i) n_c(j) - conj(C_ij) B_ij,
//   Dcc = conj(Dbb), Dcb = conj(Dbc).
template <int NMAX>
COLD void measure_pair(Ctx<NMAX> x) {
    constexpr int LD = Cfg<NMAX>::LD;
    auto& s = x.s;
    const PointDev& P = x.P();
    const int n = x.n, ns = P.Ns, tid = threadIdx.x, lx = P.Lx, ly = P.Ly;
    const double lq2 = (double)P.Lq * (double)P.Lq;
    const cplx* G = x.G();
    const cplx* ph = s.ph();
    const bool hasK = P.hasK;
    // v: 0-1 sum Dbb, 2-3 sum Dbc, 4 sum |D_ij|^2, 5-6 sf_K, 7-8 dw_K, 9 kinetic bonds,
    //    10 sum Re n_b, 11 sum Re Dbc(i,i), 12 sum Re n_b^2, 13 sum Re Dbb(i,i),
    //    14 sum Re(C_ii - B_ii)
    double v[16], tr[4] = {0.0, 0.0, 0.0, 0.0};   // tr: traces of B and C, warp 0
#pragma unroll
    for (int k = 0; k < 16; ++k) v[k] = 0.0;
    const int* sxy = s.sxy();
    const int T = blockDim.x;
    const uint32_t dm = div_magic(ns);
    for (int e = tid; e < ns * ns; e += T) {
        const int i = div_by(e, dm), j = e - i * ns;
        const cplx A = G[i * LD + j], B = G[i * LD + ns + j], C = G[(ns + i) * LD + j], D = G[(ns + i) * LD + ns + j];
        const cplx di = G[(ns + i) * LD + ns + i], dj = G[(ns + j) * LD + ns + j];
        const cplx nbi = cmk(-di.x, di.y), nbj = cmk(-dj.x, dj.y), ncj = cmk(-dj.x, -dj.y);
        const cplx dbb = csub(cmul(nbi, nbj), cmul(cconj(D), A));
        const cplx dbc = csub(cmul(nbi, ncj), cmul(cconj(C), B));
        v[0] += dbb.x;
        v[1] += dbb.y;
        v[2] += dbc.x;
        v[3] += dbc.y;
        v[4] += D.x * D.x + D.y * D.y;
        if (hasK) {
            const int pi = sxy[i], pj = sxy[j];
            int dx = (pi & 0xffff) - (pj & 0xffff), dy = (pi >> 16) - (pj >> 16);
            dx += (dx < 0) ? lx : 0;
            dy += (dy < 0) ? ly : 0;
            const cplx p = ph[dy * lx + dx];
            const double sfr = -2.0 * D.x;                 // G_bdag_b + G_cdag_c
            const double dwr = 2.0 * (dbb.x + dbc.x);      // Dbb + Dcc + Dbc + Dcb
            v[5] += p.x * sfr;
            v[6] += p.y * sfr;
            v[7] += p.x * dwr;
            v[8] += p.y * dwr;
        }
    }
    for (int e = tid; e < 3 * ns; e += blockDim.x) {   // bonds (x+1,y), (x,y+1), (x-1,y+1)
        const int i = e / 3, nb = e - (e / 3) * 3;
        const int ix = sxy[i] & 0xffff, iy = sxy[i] >> 16;
        const int jx = (nb == 0) ? (ix + 1) % lx : (nb == 1 ? ix : (ix + lx - 1) % lx);
        const int jy = (nb == 0) ? iy : (iy + 1) % ly;
        const int jj = jy * lx + jx;
        v[9] += -2.0 * (G[(ns + i) * LD + ns + jj].x + G[(ns + jj) * LD + ns + i].x);
    }
    for (int i = tid; i < ns; i += blockDim.x) {
        const cplx A = G[i * LD + i], B = G[i * LD + ns + i], C = G[(ns + i) * LD + i], D = G[(ns + i) * LD + ns + i];
        const cplx nb = cmk(-D.x, D.y);
        const double nbnc = D.x * D.x + D.y * D.y;          // n_b n_c = |D_ii|^2
        const cplx cb = cmul(cconj(C), B);
        const cplx dbb = cadd(cmul(nb, nb), cmul(nb, A));
        v[10] += nb.x;
        v[11] += nbnc - cb.x;
        v[12] += nb.x * nb.x - nb.y * nb.y;
        v[13] += dbb.x;
        v[14] += C.x - B.x;
        s.obs()[O_SITE + i] += 2.0 * nb.x;
    }
    // psf_Gamma takes the product of this slice's traces: warp 0 forms them
    if (tid < 32) {
        for (int i = tid; i < ns; i += 32) {
            const cplx B = G[i * LD + ns + i], C = G[(ns + i) * LD + i];
            tr[0] += B.x;
            tr[1] += B.y;
            tr[2] += C.x;
            tr[3] += C.y;
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) tr[k] = warp_sum(tr[k]);
        if (tid == 0) {   // (-conj(tr C tr B) + sum |D_ij|^2) / Lq^2, the sum at the end of the sweep
            s.obs()[O_PSF_GAMMA] -= (tr[2] * tr[0] - tr[3] * tr[1]) / lq2;
            s.obs()[O_PSF_GAMMA + 1] += (tr[2] * tr[1] + tr[3] * tr[0]) / lq2;
            s.cnt()[4] += 1;
        }
    }
    warp_add16(v, s.msum() + 16 * (tid >> 5));
}

template <int NMAX>
DEVI void measure_pair_finish(Ctx<NMAX>& x) {
    auto& s = x.s;
    const PointDev& P = x.P();
    const double lq = (double)P.Lq, lq2 = lq * lq, dns = (double)P.Ns;
    __syncthreads();
    if (threadIdx.x == 0) {
        double v[15];
        for (int k = 0; k < 15; ++k) {
            v[k] = 0.0;
            for (int w = 0; w < Cfg<NMAX>::THREADS / 32; ++w) v[k] += s.msum()[16 * w + k];
        }
        double* o = s.obs();
        const double dens = 2.0 * v[10] / dns;
        const double dbl = v[11] / dns;
        const double pair = v[14] / dns;
        const double kin = P.RT * v[9] / dns;
        const double inter = (P.U1 + P.U2) * (2.0 * v[13]) / dns + 2.0 * (P.U2 - P.U1) * dbl;
        const double epair = P.Delta * pair;
        const double chem = -P.mu * dens;
        const double energy = kin + inter + epair;
        o[O_DENSITY_UP] += v[10] / dns;
        o[O_DENSITY_DO] += v[10] / dns;
        o[O_DENSITY] += dens;
        o[O_DENSITY_TOTAL] += dens;
        o[O_NUM_UP] += v[10];
        o[O_NUM_DO] += v[10];
        o[O_DOUBLEOCC] += dbl;
        o[O_SQUAREOCC] += 2.0 * v[12] / dns;
        o[O_LOCAL_NUMSQUARE] += 2.0 * v[13] / dns;
        o[O_PAIR_EQUAL] += pair;
        o[O_NUMSQUARE_UP] += v[0];
        o[O_NUMSQUARE_DO] += v[0];
        o[O_ONSITE_N2_UP] += v[13];
        o[O_ONSITE_N2_DO] += v[13];
        o[O_KINETIC] += kin;
        o[O_INTERACTION] += inter;
        o[O_PAIRING_ENERGY] += epair;
        o[O_CHEMICAL_ENERGY] += chem;
        o[O_ENERGY] += energy;
        o[O_GRAND_ENERGY] += energy + chem;
        o[O_SF_K] += v[5] / lq2;
        o[O_SF_K + 1] += v[6] / lq2;
        o[O_DW_K] += v[7] / lq2;
        o[O_DW_K + 1] += v[8] / lq2;
        o[O_PSF_GAMMA] += v[4] / lq2;
        o[O_DEN_UPUP] += v[0] / lq;
        o[O_DEN_UPUP + 1] += v[1] / lq;
        o[O_DEN_DODO] += v[0] / lq;
        o[O_DEN_DODO + 1] -= v[1] / lq;
        o[O_DEN_UPDO] += v[2] / lq;
        o[O_DEN_UPDO + 1] += v[3] / lq;
    }
    __syncthreads();
}

// ---------------------------------------------------------------------------
// stabilisation (stabilization.f90:69-190)

// stab_UR: (U_R D_R) P = Q R;  D_R <- |diag R|;  V_R <- R P^T V_R;  U_R <- Q.
// U_R is x.U(); on exit the new V_R is in x.W2() and in A.VRc, D_R in A.DRc.
template <int NMAX>
COLD void stab_UR(Ctx<NMAX> x) {
    constexpr int LD = Cfg<NMAX>::LD;
    auto& s = x.s;
    const int n = x.n;
    const uint32_t dm = div_magic(n);
    for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
        const int r = div_by(e, dm), c = e - r * n;
        x.W1()[r * LD + c] = cmul(x.U()[r * LD + c], x.A().DRc[c]);
    }
    __syncthreads();
    qr_any(x, x.W1(), MatOp{}, op_c(x.U(), LD));   // U_R <- Q where Q^H is carried along
    for (int i = threadIdx.x; i < n; i += blockDim.x) x.A().DRc[i] = cmk(s.d()[i], 0.0);
    for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
        const int r = div_by(e, dm), c = e - r * n;
        x.W2()[r * LD + c] = x.A().VRc[s.piv()[r] * n + c];
    }
    __syncthreads();
    gemm_any(x, x.W2(), op_n(x.W1(), LD), op_n(x.W2(), LD), TRI_A_UPPER);
    sstore(n, LD, x.A().VRc, x.W2());
    __syncthreads();
}

// stab_UL: (U_L^H D_L) P = Q R;  D_L <- |diag R|;  V_L <- V_L P R^H;  U_L <- Q^H.
template <int NMAX>
COLD void stab_UL(Ctx<NMAX> x) {
    constexpr int LD = Cfg<NMAX>::LD;
    auto& s = x.s;
    const int n = x.n;
    const uint32_t dm = div_magic(n);
    for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
        const int r = div_by(e, dm), c = e - r * n;
        x.W1()[r * LD + c] = cmul(cconj(x.U()[c * LD + r]), x.A().DLc[c]);
    }
    __syncthreads();
    qr_any(x, x.W1(), MatOp{}, op_n(x.U(), LD));   // U_L <- Q^H
    for (int i = threadIdx.x; i < n; i += blockDim.x) x.A().DLc[i] = cmk(s.d()[i], 0.0);
    for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
        const int r = div_by(e, dm), c = e - r * n;
        x.W2()[r * LD + c] = x.A().VLc[r * n + s.piv()[c]];
    }
    __syncthreads();
    gemm_any(x, x.W2(), op_n(x.W2(), LD), op_c(x.W1(), LD), TRI_B_LOWER_FROM_C);
    sstore(n, LD, x.A().VLc, x.W2());
    __syncthreads();
}

// M = U_R^H U_L^H - D_R V_R V_L D_L is in W2 (W1 free); finish stab_green:
// factor M (or M^H for nt > L/2) and write G = (I - B)^{-1} into W2.  The
// D^{-1} scaling before ZTRSM is applied as the solve loads its operand; the
// reciprocals of R's diagonal and of D live in the QR norm vectors (free once
// the factorisation is done) and in u2.
//
// right_local: the right side (U_R) is in shared memory and U_L in HBM
// (stab_green_right_local); otherwise the left side is local and U_R in HBM.
// The HBM factor of the final product is staged into W2 (free after the
// triangular solve) so that every product runs on shared memory.
template <int NMAX>
COLD void green_from_M(Ctx<NMAX> x, int nt, bool right_local, bool want_logdet) {
    constexpr int LD = Cfg<NMAX>::LD;
    auto& s = x.s;
    const int n = x.n, L = x.P().L;
    const MatOp Uloc = op_c(x.U(), LD);
    const MatOp URh = right_local ? Uloc : op_c(x.A().URc, n);
    const MatOp ULh = right_local ? op_c(x.A().ULc, n) : Uloc;
    if (nt > L / 2) conj_transpose_any(x, x.W2());
    // W1 <- Q^H U_R^H, or U_L^H Q = (Q^H (U_L^H)^H)^H
    const bool left = nt < L / 2 + 1;
    qr_any(x, x.W2(), left ? URh : op_h(ULh), left ? op_n(x.W1(), LD) : op_c(x.W1(), LD));
    if (left) {
        solve_any(x, x.W2(), op_n(x.W1(), LD), op_n(x.W1(), LD));
        if (right_local) {   // U_L^H from HBM, staged
            sload(n, LD, x.W2(), x.A().ULc);
            __syncthreads();
            gemm_any(x, x.W2(), op_c(x.W2(), LD), op_n(x.W1(), LD));
        } else {
            gemm_any(x, x.W2(), Uloc, op_n(x.W1(), LD));
        }
    } else {
        solve_any(x, x.W2(), op_c(x.W1(), LD), op_c(x.W1(), LD));   // from the right: of the conjugate transpose
        if (right_local) {
            gemm_any(x, x.W2(), op_n(x.W1(), LD), Uloc);
        } else {             // U_R^H from HBM, staged
            sload(n, LD, x.W2(), x.A().URc);
            __syncthreads();
            gemm_any(x, x.W2(), op_n(x.W1(), LD), op_c(x.W2(), LD));
        }
    }
    if (want_logdet) {
        double v[1] = {0.0};
        for (int i = threadIdx.x; i < n; i += blockDim.x) v[0] += log(s.d()[i]);
        block_sum<1>(v, s.red());
        if (threadIdx.x == 0) x.sc->logdetM = v[0];
    }
}

// M = invULUR - D_R (V_R V_L) D_L with V_R V_L already in W1 and invULUR in W2.
template <int NMAX>
DEVI void form_M(Ctx<NMAX>& x) {
    constexpr int LD = Cfg<NMAX>::LD;
    auto& s = x.s;
    const int n = x.n;
    const uint32_t dm = div_magic(n);
    for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
        const int r = div_by(e, dm), c = e - r * n;
        const cplx t = cmul(x.A().DLc[c], x.W1()[r * LD + c]);
        x.W2()[r * LD + c] = csub(x.W2()[r * LD + c], cmul(x.A().DRc[r], t));
    }
    __syncthreads();
}

// compare_mat + G <- G_new (stabilization.f90:256-266, 339-344)
template <int NMAX>
DEVI void drift_and_replace(Ctx<NMAX>& x) {
    auto& s = x.s;
    const int n = x.n;
    const uint32_t dm = div_magic(n);
    double v[1] = {0.0};
    constexpr int LD = Cfg<NMAX>::LD;
    for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
        const int r = div_by(e, dm), c = e - r * n;
        v[0] += cabsv(csub(x.W2()[r * LD + c], x.G()[r * LD + c]));
    }
    block_sum<1>(v, s.red());
    if (threadIdx.x == 0) {
        const double dif = v[0];
        if (dif > x.sc->xmax) x.sc->xmax = dif;
        x.sc->xmean += dif;
        if (!(dif == dif) || dif > 1.0e300) x.sc->status |= 1;
    }
    scopy(n, LD, x.G(), x.W2());
    __syncthreads();
}

// stab_green with the right side factored in shared memory (U = U_R, W2 = V_R)
// and the left side in HBM (A.ULc, A.VLc, A.DLc).
template <int NMAX>
COLD void stab_green_right_local(Ctx<NMAX> x, int nt, bool want_logdet) {
    constexpr int LD = Cfg<NMAX>::LD;
    auto& s = x.s;
    const int n = x.n;
    // HBM operands are staged into the workspace the product overwrites (the
    // products stage their results in registers, so C may alias an operand);
    // V_R in W2 is no longer needed after the first product (VRc holds it).
    sload(n, LD, x.W1(), x.A().VLc);
    __syncthreads();
    gemm_any(x, x.W1(), op_n(x.W2(), LD), op_n(x.W1(), LD));   // V_R V_L
    sload(n, LD, x.W2(), x.A().ULc);
    __syncthreads();
    gemm_any(x, x.W2(), op_c(x.U(), LD), op_c(x.W2(), LD));    // U_R^H U_L^H
    form_M(x);
    green_from_M(x, nt, true, want_logdet);
}

// stab_green with the left side in shared memory (U = U_L, W2 = V_L) and the
// right side in HBM.
template <int NMAX>
COLD void stab_green_left_local(Ctx<NMAX> x, int nt) {
    constexpr int LD = Cfg<NMAX>::LD;
    auto& s = x.s;
    const int n = x.n;
    sload(n, LD, x.W1(), x.A().VRc);
    __syncthreads();
    gemm_any(x, x.W1(), op_n(x.W1(), LD), op_n(x.W2(), LD));   // V_R V_L
    sload(n, LD, x.W2(), x.A().URc);
    __syncthreads();
    gemm_any(x, x.W2(), op_c(x.W2(), LD), op_c(x.U(), LD));    // U_R^H U_L^H
    form_M(x);
    green_from_M(x, nt, false, false);
}

// Wrap_L (stabilization.f90:301-331)
template <int NMAX>
COLD void wrap_L(Ctx<NMAX> x, int nt) {
    auto& s = x.s;
    const int n = x.n, st = nt / x.P().Nwrap;
    gcopy(x.A().URc, x.A().URs(st), n * n);
    gcopy(x.A().VRc, x.A().VRs(st), n * n);
    gcopy(x.A().DRc, x.A().DRs(st), n);
    __syncthreads();
    if (nt != x.P().L) {
        stab_UL(x);
        stab_green_left_local(x, nt);
        drift_and_replace(x);
    }
    sstore(n, Cfg<NMAX>::LD, x.A().ULs(st), x.U());
    gcopy(x.A().VLs(st), x.A().VLc, n * n);
    gcopy(x.A().DLs(st), x.A().DLc, n);
    __syncthreads();
    load_expT(x);
}

// Wrap_R (stabilization.f90:333-366)
template <int NMAX>
COLD void wrap_R(Ctx<NMAX> x, int nt) {
    auto& s = x.s;
    const int n = x.n, st = nt / x.P().Nwrap;
    gcopy(x.A().ULc, x.A().ULs(st), n * n);
    gcopy(x.A().VLc, x.A().VLs(st), n * n);
    gcopy(x.A().DLc, x.A().DLs(st), n);
    __syncthreads();
    if (nt != 0) {
        stab_UR(x);
        stab_green_right_local(x, nt, nt == x.P().L);
        drift_and_replace(x);
    }
    sstore(n, Cfg<NMAX>::LD, x.A().URs(st), x.U());
    gcopy(x.A().VRs(st), x.A().VRc, n * n);
    gcopy(x.A().DRs(st), x.A().DRc, n);
    __syncthreads();
    load_expT(x);
}

// ---------------------------------------------------------------------------
template <int NMAX>
DEVI bool setup_ctx(Ctx<NMAX>& x, const KernelArgs& ka, int chain) {
    const ChainDev cd = ka.chains[chain];
    if (threadIdx.x == 0) {
        *x.s.P() = ka.pts[cd.point];
    }
    __syncthreads();
    x.n = x.P().N;
    if (x.P().hasK)
        for (int r = threadIdx.x; r < x.P().Lq && r < NMAX; r += blockDim.x) x.s.ph()[r] = x.P().phaseR[r];
    for (int i = threadIdx.x; i < x.P().Lq && i < NMAX; i += blockDim.x) {
        const int lx = x.P().Lx;
        x.s.sxy()[i] = (i % lx) | ((i / lx) << 16);
    }
    x.abase = ka.arena + cd.arena_off;
    x.wg = x.abase + arena_base(x.n, x.P().Nst);
    x.phi = ka.phi + cd.phi_off;
    x.sc = ka.sc + chain;
    return x.n <= NMAX;
}

template <int NMAX>
DEVI void load_obs(Ctx<NMAX>& x) {
    for (int k = threadIdx.x; k < kObsScalars + NMAX; k += blockDim.x) x.s.obs()[k] = 0.0;
    for (int k = threadIdx.x; k < 16 * (Cfg<NMAX>::THREADS / 32); k += blockDim.x) x.s.msum()[k] = 0.0;
}
template <int NMAX>
DEVI void flush_obs(Ctx<NMAX>& x, double* gobs) {
    for (int k = threadIdx.x; k < kObsScalars + x.P().Lq; k += blockDim.x) gobs[k] += x.s.obs()[k];
}

template <int NMAX, bool PAIR, bool LEFT>
DEVI void prop_any(Ctx<NMAX>& x, int ch, int slice) {
    prop_channel<NMAX, LEFT, PAIR>(x, ch, slice);
}
template <int NMAX, bool PAIR>
DEVI void measure_any(Ctx<NMAX>& x) {
    if constexpr (PAIR) measure_pair<NMAX>(x);
    else measure<NMAX>(x);
}

// one sweep: Local_sweep_L then Local_sweep_R (local_sweep.f90:96-134)
template <int NMAX, bool PAIR>
__global__ void __launch_bounds__(Cfg<NMAX>::THREADS, Cfg<NMAX>::MINB) sweep_kernel(KernelArgs ka, const int* idx, int count) {
    if ((int)blockIdx.x >= count) return;
    const int chain = idx[blockIdx.x];
    Ctx<NMAX> x;
    if (!setup_ctx(x, ka, chain)) return;
    if (x.sc->status & 1) return;   // quarantined: non-finite G, skipped until its state is set again
    tc_begin(x, ka);
    auto& s = x.s;
    const int n = x.n, L = x.P().L;
    const bool tm = ka.timers && threadIdx.x == 0;
    long long tk = tm ? clock64() : 0;
#define lap(ph)                                      \
    do {                                             \
        if (tm) {                                    \
            const long long t_ = clock64();          \
            x.sc->cyc[ph] += t_ - tk;                \
            tk = t_;                                 \
        }                                            \
    } while (0)
    if (threadIdx.x == 0) {
        *s.seed() = x.sc->seed;
        for (int k = 0; k < 5; ++k) s.cnt()[k] = 0;
    }
    load_obs(x);
    sload(n, Cfg<NMAX>::LD, x.G(), x.A().G);
    sload(n, Cfg<NMAX>::LD, x.U(), x.A().ULc);
    __syncthreads();
    load_expT(x);
    lap(3);
    // ---- left traversal (skipped by a right-only launch, which continues from
    // the G, U_L and counters a left-only launch left in the arena)
    if (ka.traverse != 2) {
        for (int nt = L; nt >= 1; --nt) {
            if (nt % x.P().Nwrap == 0) {
                wrap_L(x, nt);
                lap(3);
            }
            stage_fields(x, nt - 1);
            measure_any<NMAX, PAIR>(x);
            lap(2);
            slice_products<NMAX, true>(x);
            lap(1);
            if (x.P().active[1]) prop_any<NMAX, PAIR, true>(x, 1, nt - 1);
            if (x.P().active[0]) prop_any<NMAX, PAIR, true>(x, 0, nt - 1);
            lap(0);
        }
        wrap_L(x, 0);
        sstore(n, Cfg<NMAX>::LD, x.A().ULc, x.U());
        __syncthreads();
    }
    // ---- right traversal
    if (ka.traverse != 1) {
    sload(n, Cfg<NMAX>::LD, x.U(), x.A().URc);
    __syncthreads();
    wrap_R(x, 0);
    lap(3);
    stage_fields(x, 0);
    for (int nt = 1; nt <= L; ++nt) {
        if (x.P().active[0]) prop_any<NMAX, PAIR, false>(x, 0, nt - 1);
        if (x.P().active[1]) prop_any<NMAX, PAIR, false>(x, 1, nt - 1);
        lap(0);
        if (nt < L) stage_fields(x, nt);
        slice_products<NMAX, false>(x);
        lap(1);
        if (nt % x.P().Nwrap == 0) {
            wrap_R(x, nt);
            lap(3);
        }
        measure_any<NMAX, PAIR>(x);
        lap(2);
    }
    sstore(n, Cfg<NMAX>::LD, x.A().URc, x.U());
    }
    sstore(n, Cfg<NMAX>::LD, x.A().G, x.G());
    if constexpr (PAIR) measure_pair_finish(x);
    else measure_finish(x);
    flush_obs(x, ka.obs + (long)chain * ka.obs_stride);
    if (threadIdx.x == 0) {
        x.sc->seed = *s.seed();
        x.sc->nacc[0] += s.cnt()[0];
        x.sc->nacc[1] += s.cnt()[1];
        x.sc->nc[0] += s.cnt()[2];
        x.sc->nc[1] += s.cnt()[3];
        x.sc->nobs += s.cnt()[4];
    }
    lap(3);
#undef lap
    tc_end(x, ka);
}

// Local_sweep_pre (local_sweep.f90:80-94) with Prop_make's identities
// (process_matrix.f90:37-47).  propU_pre scales the rows of U_R by the HS
// factors (multiply.f90:7-16); for a Nambu chain row Ns+i (c^dagger_i) takes
// e^{-alpha phi} in the U2 channel (src/pairing/src/operator_Hubbard.f90:155-166).
template <int NMAX, bool PAIR>
__global__ void __launch_bounds__(Cfg<NMAX>::THREADS, Cfg<NMAX>::MINB) pre_kernel(KernelArgs ka, const int* idx, int count) {
    constexpr int LD = Cfg<NMAX>::LD;
    if ((int)blockIdx.x >= count) return;
    const int chain = idx[blockIdx.x];
    Ctx<NMAX> x;
    if (!setup_ctx(x, ka, chain)) return;
    tc_begin(x, ka);
    auto& s = x.s;
    const int n = x.n, L = x.P().L;
    const uint32_t dm = div_magic(n);
    set_identity(n, LD, x.U());
    set_identity(n, LD, x.G());
    set_identity(n, n, x.A().VRc);
    set_identity(n, n, x.A().ULc);
    set_identity(n, n, x.A().VLc);
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        x.A().DRc[i] = cmk(1.0, 0.0);
        x.A().DLc[i] = cmk(1.0, 0.0);
    }
    __syncthreads();
    sstore(n, LD, x.A().URs(0), x.U());
    gcopy(x.A().VRs(0), x.A().VRc, n * n);
    gcopy(x.A().DRs(0), x.A().DRc, n);
    if constexpr (!Cfg<NMAX>::GW) sload_real(n, x.ldr(), reinterpret_cast<double*>(x.W1()), x.P().expP);
    __syncthreads();
    const int ns = x.P().Ns;
    for (int nt = 1; nt <= L; ++nt) {
        const double* ph = x.phi + (long)(nt - 1) * ns * 2;
        for (int ch = 0; ch < 2; ++ch) {
            if (!x.P().active[ch]) continue;
            const double ar = x.P().alpha_re[ch], ai = x.P().alpha_im[ch];
            const bool flip = x.P().flip[ch] != 0;
            for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
                const int r = div_by(e, dm), c = e - r * n;
                const int site = (PAIR && r >= ns) ? r - ns : r;
                const double p = ph[site * 2 + ch];
                const bool neg = PAIR && r >= ns && flip;
                const cplx f = neg ? cexpz(cmk(-(ar * p), -(ai * p))) : cexpz(cmk(ar * p, ai * p));
                x.U()[r * LD + c] = cmul(f, x.U()[r * LD + c]);
            }
            __syncthreads();
        }
        slice_mult<NMAX, false>(x, x.U(), x.RP());
        if (nt % x.P().Nwrap == 0) {
            const int st = nt / x.P().Nwrap;
            stab_UR(x);
            sstore(n, LD, x.A().URs(st), x.U());
            gcopy(x.A().VRs(st), x.A().VRc, n * n);
            gcopy(x.A().DRs(st), x.A().DRc, n);
            __syncthreads();
            if (nt == L) {
                stab_green_right_local(x, nt, true);
                scopy(n, LD, x.G(), x.W2());
                __syncthreads();
            }
            if constexpr (!Cfg<NMAX>::GW) {
                sload_real(n, x.ldr(), reinterpret_cast<double*>(x.W1()), x.P().expP);
                __syncthreads();
            }
        }
    }
    sstore(n, LD, x.A().URc, x.U());
    sstore(n, LD, x.A().G, x.G());
    // a chain whose G(beta) is not finite (overflowing fields) is quarantined
    {
        double v[1] = {0.0};
        for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
            const cplx g = x.A().G[e];
            if (!isfinite(g.x) || !isfinite(g.y)) v[0] += 1.0;
        }
        block_sum<1>(v, x.s.red());
        if (threadIdx.x == 0 && v[0] > 0.0) x.sc->status |= 1;
    }
    tc_end(x, ka);
}

// LocalU_prop_therm / LocalU_metro_therm over the whole field, nwarm sweeps
// (localU.f90:115-156, local_sweep.f90:64-78).  Each field value sees only its
// own proposals, so fields are updated in parallel; the draw index of a
// proposal is its position in the reference's sequential order.
__global__ void warmup_kernel(KernelArgs ka, int nwarm) {
    const int chain = blockIdx.x;
    if (chain >= ka.nchains) return;
    const ChainDev cd = ka.chains[chain];
    const PointDev P = ka.pts[cd.point];
    ChainScalars* sc = ka.sc + chain;
    double* phi = ka.phi + cd.phi_off;
    __shared__ double red[2 * 32];
    __shared__ int chs[2];
    __shared__ int nact;
    if (threadIdx.x == 0) {
        int a = 0;
        for (int ch = 0; ch < 2; ++ch)
            if (P.active[ch]) chs[a++] = ch;
        nact = a;
    }
    __syncthreads();
    const int A = nact, n = P.Ns, L = P.L;
    const uint32_t s0 = sc->seed;
    const unsigned long long per_sweep = (unsigned long long)L * A * n;
    const uint32_t step = lcg_pow(2ull * per_sweep);
    const double shift = fabs(P.shiftLoc);
    double cnt[2] = {0.0, 0.0};
    for (long long m = threadIdx.x; m < (long long)per_sweep; m += blockDim.x) {
        const int i = (int)(m % n);
        const int chpos = (int)((m / n) % A);
        const int nt = (int)(m / ((long long)n * A));
        const int ch = chs[chpos];
        double p = phi[((long)nt * n + i) * 2 + ch];
        uint32_t d1 = lcg_mul(lcg_pow(2ull * m + 1ull), s0);
        for (int w = 0; w < nwarm; ++w) {
            const uint32_t d2 = lcg_mul(kLcgA, d1);
            const double xflip = lcg_u(d1), rnd = lcg_u(d2);
            const double pn = p + (xflip - 0.5) * shift;
            const double ratio = exp(-0.5 * pn * pn) / exp(-0.5 * p * p);
            if (ratio > rnd) {
                p = pn;
                cnt[chpos] += 1.0;
            }
            d1 = lcg_mul(step, d1);
        }
        phi[((long)nt * n + i) * 2 + ch] = p;
    }
    double v[2] = {cnt[0], cnt[1]};
    block_sum<2>(v, red);
    if (threadIdx.x == 0) {
        for (int k = 0; k < A; ++k) sc->therm_acc_sum[chs[k]] += v[k] / ((double)L * n);
        sc->seed = lcg_mul(lcg_pow(2ull * per_sweep * (unsigned long long)nwarm), s0);
    }
}

// Start of a bin: Local_sweep_reset (local_sweep.f90:54-62).
__global__ void bin_reset_kernel(KernelArgs ka) {
    const int chain = blockIdx.x;
    if (chain >= ka.nchains) return;
    double* o = ka.obs + (long)chain * ka.obs_stride;
    for (int k = threadIdx.x; k < ka.obs_stride; k += blockDim.x) o[k] = 0.0;
    if (threadIdx.x == 0) {
        ChainScalars* sc = ka.sc + chain;
        sc->nc[0] = sc->nc[1] = 0;
        sc->nacc[0] = sc->nacc[1] = 0;
        sc->nobs = 0;
    }
}

// End of a bin: Obs_equal_ave and AccCounter%ratio (obser_equal.f90:66-93,
// operator_Hubbard.f90:124-129).
__global__ void bin_finish_kernel(KernelArgs ka) {
    const int chain = blockIdx.x;
    if (chain >= ka.nchains) return;
    ChainScalars* sc = ka.sc + chain;
    const int lq = ka.pts[ka.chains[chain].point].Lq;
    const double z = 1.0 / (double)sc->nobs;
    double* o = ka.obs + (long)chain * ka.obs_stride;
    for (int k = threadIdx.x; k < kObsScalars + lq; k += blockDim.x) o[k] *= z;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int ch = 0; ch < 2; ++ch) {
            if (sc->nc[ch] > 0) sc->acc_sum[ch] += (double)sc->nacc[ch] / (double)sc->nc[ch];
            sc->prop_tot[ch] += (double)sc->nc[ch];
            sc->acc_tot[ch] += (double)sc->nacc[ch];
        }
    }
}

// Chain average per point (m_process_obs_equal, fourier_trans.f90:350-457):
// out[p][k] = sum over the chains of point p of obs[chain][k] / (chains of p),
// over the chains that are not quarantined (NaN if none is left).
__global__ void point_average_kernel(KernelArgs ka, const int* point_chain_start, const int* point_chain_list,
                                     double* out) {
    const int p = blockIdx.x;
    const int b = point_chain_start[p], e = point_chain_start[p + 1];
    for (int k = threadIdx.x; k < ka.obs_stride; k += blockDim.x) {
        double s = 0.0;
        int m = 0;
        for (int c = b; c < e; ++c) {
            const int ch = point_chain_list[c];
            if (ka.sc[ch].status & 1) continue;   // quarantined chains leave the average
            s += ka.obs[(long)ch * ka.obs_stride + k];
            ++m;
        }
        out[(long)p * ka.obs_stride + k] = m > 0 ? s / (double)m : __longlong_as_double(0x7ff8000000000000LL);
    }
}

// Block statistics of the per-bin point averages: cur += pout (bins summed in
// order); when a block completes, blk = cur / block_size and cur restarts.
__global__ void stats_add_kernel(const double* pout, double* cur, double* blk, int n, int finish, int block_size) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        const double v = cur[k] + pout[k];
        if (finish) {
            blk[k] = v / (double)block_size;
            cur[k] = 0.0;
        } else {
            cur[k] = v;
        }
    }
}
// mean and standard error over nb block means, each element summed over the
// blocks in order: mean = sum / nb, sem = sqrt(sum (m - mean)^2 / (nb - 1) / nb)
__global__ void stats_final_kernel(const double* blk, int nb, int n, double* mean, double* sem) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        double s = 0.0;
        for (int b = 0; b < nb; ++b) s += blk[(long)b * n + k];
        const double m = s / (double)nb;
        double v = 0.0;
        for (int b = 0; b < nb; ++b) {   // square rounded, then added (no fused multiply-add)
            const double d = blk[(long)b * n + k] - m;
            v = __dadd_rn(v, __dmul_rn(d, d));
        }
        mean[k] = m;
        sem[k] = nb > 1 ? sqrt(v / (double)(nb - 1) / (double)nb) : __longlong_as_double(0x7ff8000000000000LL);
    }
}

// Global shift move: the shift part of Global_flip (global_update.f90:193-208),
// under this model's weight.  Per chain, two draws of the chain's LCG give a
// uniform shift X_ns = (u - 1/2) |shift_ns| of every field of auxiliary channel
// ns; the shifted field goes to the proposal state kp (same layout).
__global__ void global_propose_kernel(KernelArgs ka, KernelArgs kp, double shift0, double shift1) {
    const int chain = blockIdx.x;
    if (chain >= ka.nchains) return;
    const ChainDev cd = ka.chains[chain];
    const PointDev& P = ka.pts[cd.point];
    ChainScalars* sc = ka.sc + chain;
    if (sc->status & 1) return;   // quarantined
    __shared__ double X[2];
    if (threadIdx.x == 0) {
        uint32_t seed = sc->seed;
        const double amp[2] = {fabs(shift0), fabs(shift1)};
        for (int ns = 0; ns < 2; ++ns) {
            seed = lcg_mul(kLcgA, seed);
            X[ns] = (lcg_u(seed) - 0.5) * amp[ns];
        }
        sc->seed = seed;
        kp.sc[chain].status = 0;
    }
    __syncthreads();
    const long long tot = (long long)P.L * P.Ns * 2;
    const double* phi = ka.phi + cd.phi_off;
    double* phi2 = kp.phi + cd.phi_off;
    for (long long k = threadIdx.x; k < tot; k += blockDim.x) phi2[k] = phi[k] + X[k & 1];
}

// Exact Metropolis-Hastings decision of a global move (global_update.f90:237-249:
// accept if w'/w >= u, u the chain's next draw), with log w = -sum phi^2 / 2
// - f log|det(I - B(beta,0))| from the two states' last factorisations at
// tau = beta: f = 2 for a number-conserving chain (flavours b and c = conj(b)),
// f = 1 for a Nambu chain (the 4Ns determinant to the power -1/2 is the
// squared modulus of its {b, c^dagger} block's, to the power -1/2).
// hastings (optional) adds log q(phi|phi') - log q(phi'|phi) of a
// non-symmetric proposal; a non-finite exponent rejects.  An accepted chain
// takes the proposal's fields and UDV arena.
__global__ void global_accept_kernel(KernelArgs ka, KernelArgs kp, const double* fn, const double* fn2,
                                     const double* hastings, int* accepted) {
    const int chain = blockIdx.x;
    if (chain >= ka.nchains) return;
    const ChainDev cd = ka.chains[chain];
    const PointDev& P = ka.pts[cd.point];
    ChainScalars* sc = ka.sc + chain;
    __shared__ int acc;
    if (threadIdx.x == 0) {
        acc = 0;
        if (!(sc->status & 1)) {
            const double f = P.pairing ? 1.0 : 2.0;
            const double lw = fn[chain] - f * sc->logdetM;
            const double lw2 = fn2[chain] - f * kp.sc[chain].logdetM;
            const double x = lw2 - lw + (hastings ? hastings[chain] : 0.0);
            const uint32_t seed = lcg_mul(kLcgA, sc->seed);
            sc->seed = seed;
            acc = !(kp.sc[chain].status & 1) && !isnan(x) && x < INFINITY && exp(x) >= lcg_u(seed);
            sc->glb_prop += 1.0;
            if (acc) {
                sc->glb_acc += 1.0;
                sc->logdetM = kp.sc[chain].logdetM;
            }
        }
        if (accepted) accepted[chain] = acc;
    }
    __syncthreads();
    if (!acc) return;
    const long long na = arena_base(P.N, P.Nst), nphi = (long long)P.L * P.Ns * 2;
    const double2* a2 = kp.arena + cd.arena_off;
    double2* a = ka.arena + cd.arena_off;
    for (long long k = threadIdx.x; k < na; k += blockDim.x) a[k] = a2[k];
    const double* p2 = kp.phi + cd.phi_off;
    double* p = ka.phi + cd.phi_off;
    for (long long k = threadIdx.x; k < nphi; k += blockDim.x) p[k] = p2[k];
}

// bad[chain] = 1 if any field value of the chain is NaN or infinite
__global__ void field_check_kernel(KernelArgs ka, int* bad) {
    const int chain = blockIdx.x;
    if (chain >= ka.nchains) return;
    const ChainDev cd = ka.chains[chain];
    const PointDev& P = ka.pts[cd.point];
    const double* phi = ka.phi + cd.phi_off;
    const long long tot = (long long)P.L * P.Ns * 2;
    int any = 0;
    for (long long k = threadIdx.x; k < tot; k += blockDim.x) any |= !isfinite(phi[k]);
    any = __syncthreads_or(any);
    if (threadIdx.x == 0) bad[chain] = any;
}

// -0.5 * sum(phi^2) per chain (AuxConf_log_weight, fields.f90:29-33)
__global__ void field_norm_kernel(KernelArgs ka, double* out) {
    const int chain = blockIdx.x;
    if (chain >= ka.nchains) return;
    const ChainDev cd = ka.chains[chain];
    const PointDev P = ka.pts[cd.point];
    __shared__ double red[32];
    const double* phi = ka.phi + cd.phi_off;
    double v[1] = {0.0};
    const long long tot = (long long)P.L * P.Ns * 2;
    for (long long k = threadIdx.x; k < tot; k += blockDim.x) v[0] += phi[k] * phi[k];
    block_sum<1>(v, red);
    if (threadIdx.x == 0) out[chain] = -0.5 * v[0];
}

// ---------------------------------------------------------------------------
// Time-displaced Green's functions (Dyn_reset + Dyn_sweep_R, dynamics.f90:38-58;
// propgrU_R / propgrT_R, multiply.f90:48-97; Wrap_tau and stab_green_big,
// stabilization.f90:192-254, 368-404) of a number-conserving chain with
// N <= 72, run between its left and right traversals (Local_sweep_R's toggle,
// local_sweep.f90:119-123).  From G(0,0) and the left factors the left
// traversal stored, G(tau,0) = B(tau,0) G, G(0,tau) = -(I - G) B(tau,0)^-1 and
// G(tau,tau) = B(tau,0) G B(tau,0)^-1 are propagated slice by slice, and every
// Nwrap slices recomputed from the stabilised factors as blocks of
//   diag(V_R^-1, U_L^H) [[(V_R V_L)^-1, -D_L], [-D_R, (U_L U_R)^H]]^-1 diag(V_L^-1, U_R^H),
// the inverse of [[I, -B(beta,tau)], [-B(tau,0), I]]; the L1 distance between
// the propagated and the recomputed matrices is the drift Wrap_tau records.
// Two departures from the reference, both deliberate: the U2 operator uses the
// U2 field (dynamics.f90:52 passes the U1 field), and the 2N x 2N matrix has
// the bosonic -D_L (stabilization.f90:206-209 has +D_L, whose inverse is the
// fermionic (I + B)^-1 in its G(0,0) block).  The chain's own state is not
// touched: the pass works on copies in its own region of global memory, with
// the routines of the N <= 144 class (2N <= 144 rows).
namespace taud {
// The pass of an N <= 36 chain runs in the N <= 72 class's context (2N <= 72;
// G and U in shared memory, register-resident factorisations), that of a
// 36 < N <= 72 chain in the N <= 144 class's.  Matrices of the region have the
// class's leading dimension.
template <int NMAX> constexpr int LD = Cfg<NMAX>::LD;
template <int NMAX> constexpr long long MAT = (long long)NMAX * Cfg<NMAX>::LD;   // complex values per slot
// slots of a CTA's region; 0..4 are the class context's W1, W2 (and, N <= 144, G, U, S)
// (G holds G(0,0) of the pass, U the propagated right factor U_R)
enum { GT0 = 5, G0T = 6, GTT = 7, VR = 8, BIG = 9, X = 10, VRI = 11, VLI = 12, UL = 13, VEC = 14, EP = 15, EM = 16, SLOTS = 17 };
constexpr long long REGION = SLOTS * MAT<144>;   // the larger class's region serves both
template <int NMAX> DEVI cplx* slot(const Ctx<NMAX>& x, int k) { return x.wg + k * MAT<NMAX>; }
}  // namespace taud

long long tau_region_elems() { return taud::REGION; }

// C <- A^-1 C for the x.n x x.n matrix A, which is destroyed: pivoted QR,
// Q^H C, R^-1 D^-1, the row permutation back.
template <int NMAX>
COLD void tau_solve(Ctx<NMAX>& x, cplx* A, cplx* C) {
    constexpr int LD = taud::LD<NMAX>;
    qr_any(x, A, op_n(C, LD), op_n(C, LD));
    solve_any(x, A, op_n(C, LD), op_n(C, LD));
}

template <int NMAX>
DEVI void tau_copy(int n, cplx* dst, const cplx* src) {   // both with the class's leading dimension
    const uint32_t dm = div_magic(n);
    for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
        const int r = div_by(e, dm), c = e - r * n;
        dst[r * taud::LD<NMAX> + c] = src[r * taud::LD<NMAX> + c];
    }
    __syncthreads();
}

// L1 distance of two n x n matrices (compare_mat, stabilization.f90:256-266),
// valid in thread 0
template <int NMAX>
DEVI double tau_l1(Ctx<NMAX>& x, int n, const cplx* a, const cplx* b) {
    const uint32_t dm = div_magic(n);
    double v[1] = {0.0};
    for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
        const int r = div_by(e, dm), c = e - r * n;
        const cplx d = csub(a[r * taud::LD<NMAX> + c], b[r * taud::LD<NMAX> + c]);
        v[0] += sqrt(d.x * d.x + d.y * d.y);
    }
    block_sum<1>(v, x.s.red());
    return v[0];
}

// slice nt (1-based, propgrU_R then propgrT_R, multiply.f90:48-97 of both
// solvers): the HS factors of both channels, then e^{-dtau K} from the left and
// e^{+dtau K} from the right (real, in the EP and EM slots)
template <int NMAX>
COLD void tau_slice(Ctx<NMAX>& x, int nt) {
    constexpr int LD = taud::LD<NMAX>;
    const int n = x.n;
    const uint32_t dm = div_magic(n);
    const PointDev& P = x.P();
    cplx *T0 = taud::slot(x, taud::GT0), *T1 = taud::slot(x, taud::G0T), *T2 = taud::slot(x, taud::GTT);
    cplx* U = x.U();
    cplx *ep = x.s.ean(), *em = x.s.ebn();
    for (int ch = 0; ch < 2; ++ch) {
        if (!P.active[ch]) continue;
        // row i's factor e^{+-alpha phi}; on a Nambu chain's {b, c^dagger} block
        // row Ns + i (c^dagger_i) takes site i's field, with the inverse factor in
        // a flipped channel (src/pairing/src/operator_Hubbard.f90:139-199)
        for (int i = threadIdx.x; i < n; i += blockDim.x) {
            const bool cd = i >= P.Ns;
            const int site = cd ? i - P.Ns : i;
            cplx a, b;
            hs_factors(P.alpha_re[ch], P.alpha_im[ch], x.phi[((long)(nt - 1) * P.Ns + site) * 2 + ch], a, b);
            const bool inv = cd && P.flip[ch];
            ep[i] = inv ? b : a;
            em[i] = inv ? a : b;
        }
        __syncthreads();
        for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
            const int r = div_by(e, dm), c = e - r * n;
            T0[r * LD + c] = cmul(ep[r], T0[r * LD + c]);
            T1[r * LD + c] = cmul(T1[r * LD + c], em[c]);
            T2[r * LD + c] = cmul(cmul(ep[r], T2[r * LD + c]), em[c]);
            U[r * LD + c] = cmul(ep[r], U[r * LD + c]);
        }
        __syncthreads();
    }
    const double *kp = reinterpret_cast<const double*>(taud::slot(x, taud::EP)),
                 *km = reinterpret_cast<const double*>(taud::slot(x, taud::EM));
    gemm_real_any<NMAX, false>(x, T0, kp, T2);
    gemm_real_any<NMAX, true>(x, T1, km, T2);
    gemm_real_any<NMAX, false>(x, U, kp);
}

// Wrap_tau at slice nt (stabilization.f90:368-404): stab_UR of the propagated
// right factors, the 2N x 2N inverse, the drifts of G(0,tau), G(tau,0),
// G(tau,tau) against the propagated ones (thread 0 accumulates them in dr:
// max[3], sum[3], non-finite count), then the replacement.
template <int NMAX>
COLD void tau_wrap(Ctx<NMAX>& x, const Arena& A, int nt, double* dr) {
    using namespace taud;
    constexpr int LD = taud::LD<NMAX>;
    const int n = x.n, st = nt / x.P().Nwrap;
    cplx *W1 = x.W1(), *W2 = x.W2(), *U = x.U();
    cplx *M = slot(x, BIG), *Xi = slot(x, X), *VRi = slot(x, VRI), *VLi = slot(x, VLI), *ULs = slot(x, UL);
    stab_UR(x);                      // U = U_R, A.DRc = D_R, A.VRc and W2 = V_R
    tau_copy<NMAX>(n, M, W2);
    set_identity(n, LD, VRi);
    __syncthreads();
    tau_solve(x, M, VRi);            // V_R^-1
    sload(n, LD, M, A.VLs(st));
    set_identity(n, LD, VLi);
    __syncthreads();
    tau_solve(x, M, VLi);            // V_L^-1
    sload(n, LD, ULs, A.ULs(st));
    for (int e = threadIdx.x; e < 4 * n * n; e += blockDim.x) {
        const int r = e / (2 * n), c = e - r * (2 * n);
        M[r * LD + c] = cmk(0.0, 0.0);
    }
    __syncthreads();
    gemm_any(x, M, op_n(VLi, LD), op_n(VRi, LD));               // (V_R V_L)^-1
    gemm_any(x, M + n * LD + n, op_c(U, LD), op_c(ULs, LD));    // (U_L U_R)^H
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const cplx dl = A.DLs(st)[i], drv = A.DRc[i];
        M[i * LD + n + i] = cmk(-dl.x, -dl.y);
        M[(n + i) * LD + i] = cmk(-drv.x, -drv.y);
    }
    x.n = 2 * n;
    set_identity(2 * n, LD, Xi);
    __syncthreads();
    tau_solve(x, M, Xi);
    x.n = n;
    // G(0,0) = V_R^-1 X00 V_L^-1
    gemm_any(x, W1, op_n(VRi, LD), op_n(Xi, LD));
    gemm_any(x, x.G(), op_n(W1, LD), op_n(VLi, LD));
    // index 0: G(0,tau) = V_R^-1 X01 U_R^H; 1: G(tau,0) = U_L^H X10 V_L^-1; 2: G(tau,tau) = U_L^H X11 U_R^H
    cplx* dst[3] = {slot(x, G0T), slot(x, GT0), slot(x, GTT)};
    const MatOp left[3] = {op_n(VRi, LD), op_c(ULs, LD), op_c(ULs, LD)};
    const cplx* blk[3] = {Xi + n, Xi + n * LD, Xi + n * LD + n};
    const MatOp right[3] = {op_c(U, LD), op_n(VLi, LD), op_c(U, LD)};
    for (int k = 0; k < 3; ++k) {
        gemm_any(x, W1, left[k], op_n(blk[k], LD));
        gemm_any(x, W2, op_n(W1, LD), right[k]);
        const double dif = tau_l1(x, n, W2, dst[k]);
        if (threadIdx.x == 0) {
            if (dif == dif && dif <= 1.0e300) {
                if (dif > dr[k]) dr[k] = dif;
                dr[3 + k] += dif;
            } else {
                dr[6] += 1.0;
            }
        }
        tau_copy<NMAX>(n, dst[k], W2);
    }
}

// Dyn_reset + Dyn_sweep_R of one chain (dynamics.f90:37-57): copies of G and of
// the right factors, L slices, a wrap every Nwrap slices; the arena's D_R and
// V_R (which stab_UR updates) are put back at the end.
template <int NMAX>
COLD void tau_pass(Ctx<NMAX>& x, const KernelArgs& ka, int chain) {
    using namespace taud;
    constexpr int LD = taud::LD<NMAX>;
    const int n = x.n, L = x.P().L;
    const uint32_t dm = div_magic(n);
    const Arena A = x.A();
    cplx *G = x.G(), *T0 = slot(x, GT0), *T1 = slot(x, G0T), *T2 = slot(x, GTT);
    cplx *sv = slot(x, VEC), *svr = slot(x, VR);
    gcopy(sv, A.DRc, n);
    gcopy(svr, A.VRc, n * n);
    sload_real(n, x.ldr(), reinterpret_cast<double*>(slot(x, EP)), x.P().expP);
    sload_real(n, x.ldr(), reinterpret_cast<double*>(slot(x, EM)), x.P().expM);
    sload(n, LD, G, A.G);
    sload(n, LD, x.U(), A.URc);
    __syncthreads();
    for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
        const int r = div_by(e, dm), c = e - r * n;
        const cplx g = G[r * LD + c];
        T0[r * LD + c] = g;
        T2[r * LD + c] = g;
        T1[r * LD + c] = cmk(g.x - (r == c ? 1.0 : 0.0), g.y);   // -(I - G)
    }
    __syncthreads();
    double dr[7] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    for (int nt = 1; nt <= L; ++nt) {
        tau_slice(x, nt);
        if (nt % x.P().Nwrap == 0) tau_wrap(x, A, nt, dr);
        if (nt == ka.tau_probe_nt && ka.tau_probe) {
            cplx* pr = ka.tau_probe + (long long)chain * kTauProbeElems;
            const cplx* src[4] = {G, T1, T0, T2};   // G(0,0), G(0,tau), G(tau,0), G(tau,tau)
            for (int k = 0; k < 4; ++k) sstore(n, LD, pr + (long long)k * n * n, src[k]);
        }
    }
    gcopy(A.DRc, sv, n);
    gcopy(A.VRc, svr, n * n);
    if (threadIdx.x == 0) {
        double* o = ka.tau_stats + (long long)chain * kTauStats;
        for (int k = 0; k < 3; ++k) {
            o[k] = fmax(o[k], dr[k]);
            o[3 + k] += dr[3 + k];
        }
        o[6] += 1.0;
        o[7] += dr[6];
    }
    __syncthreads();
}

// One CTA per SM walks its share of the listed chains; its matrix region of
// tau_region_elems() complex values is indexed by blockIdx.x.  The N <= 72
// class's kernel takes the chains with N <= 36, the N <= 144 class's those
// with 36 < N <= kTauMaxN.
template <int NMAX>
__global__ void __launch_bounds__(Cfg<NMAX>::THREADS, 1) tau_kernel(KernelArgs ka, const int* idx, int count) {
    for (int k = blockIdx.x; k < count; k += gridDim.x) {
        const int chain = idx[k];
        Ctx<NMAX> x;
        const bool ok = setup_ctx(x, ka, chain) && 2 * x.n <= NMAX && (NMAX == 72 || 2 * x.n > 72) &&
                        x.n <= kTauMaxN && !(x.sc->status & 1);
        if (ok) {
            x.wg = ka.tau_ws + (long long)blockIdx.x * taud::REGION;
            tau_pass(x, ka, chain);
        }
        __syncthreads();
    }
}

template <int NMAX>
static cudaError_t launch_tau_cls(const KernelArgs& ka, const int* idx, int count, int grid, cudaStream_t st) {
    const size_t sm = Smem<NMAX>::bytes();
    const cudaError_t e = cudaFuncSetAttribute(tau_kernel<NMAX>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (e != cudaSuccess) return e;
    tau_kernel<NMAX><<<grid < count ? grid : count, Cfg<NMAX>::THREADS, sm, st>>>(ka, idx, count);
    return cudaGetLastError();
}
cudaError_t launch_tau(const KernelArgs& ka, const int* idx, int count, int grid, cudaStream_t st) {
    if (count <= 0) return cudaSuccess;
    const cudaError_t e = launch_tau_cls<72>(ka, idx, count, grid, st);
    return e != cudaSuccess ? e : launch_tau_cls<144>(ka, idx, count, grid, st);
}

// ---------------------------------------------------------------------------
template <int NMAX, bool PAIR>
static cudaError_t launch_cls(int which, const KernelArgs& ka, const int* idx, int count, cudaStream_t st) {
    if (count <= 0) return cudaSuccess;
    const size_t sm = Smem<NMAX>::bytes();
    cudaError_t e;
    if (which == 0) {
        e = cudaFuncSetAttribute(sweep_kernel<NMAX, PAIR>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
        if (e != cudaSuccess) return e;
        sweep_kernel<NMAX, PAIR><<<count, Cfg<NMAX>::THREADS, sm, st>>>(ka, idx, count);
    } else {
        e = cudaFuncSetAttribute(pre_kernel<NMAX, PAIR>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
        if (e != cudaSuccess) return e;
        pre_kernel<NMAX, PAIR><<<count, Cfg<NMAX>::THREADS, sm, st>>>(ka, idx, count);
    }
    return cudaGetLastError();
}

// class index: size class (NMAX 16 / 36 / 72) + 3 * Nambu sector; 6 = NMAX 144, number-conserving
static cudaError_t launch_any(int which, int cls, const KernelArgs& ka, const int* idx, int count, cudaStream_t st) {
    switch (cls) {
        case 0: return launch_cls<16, false>(which, ka, idx, count, st);
        case 1: return launch_cls<36, false>(which, ka, idx, count, st);
        case 2: return launch_cls<72, false>(which, ka, idx, count, st);
        case 3: return launch_cls<16, true>(which, ka, idx, count, st);
        case 4: return launch_cls<36, true>(which, ka, idx, count, st);
        case 5: return launch_cls<72, true>(which, ka, idx, count, st);
        case 6: return launch_cls<144, false>(which, ka, idx, count, st);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t upload_pow_table(const uint32_t* tab, int count) {
    if (count > kMaxPow) return cudaErrorInvalidValue;
    return cudaMemcpyToSymbol(c_apow, tab, sizeof(uint32_t) * count);
}

cudaError_t launch_sweep(int cls, const KernelArgs& ka, const int* idx, int count, cudaStream_t st) {
    return launch_any(0, cls, ka, idx, count, st);
}
cudaError_t launch_pre(int cls, const KernelArgs& ka, const int* idx, int count, cudaStream_t st) {
    return launch_any(1, cls, ka, idx, count, st);
}
cudaError_t launch_warmup(const KernelArgs& ka, int nwarm, cudaStream_t st) {
    warmup_kernel<<<ka.nchains, 256, 0, st>>>(ka, nwarm);
    return cudaGetLastError();
}
cudaError_t launch_bin_reset(const KernelArgs& ka, cudaStream_t st) {
    bin_reset_kernel<<<ka.nchains, 64, 0, st>>>(ka);
    return cudaGetLastError();
}
cudaError_t launch_bin_finish(const KernelArgs& ka, cudaStream_t st) {
    bin_finish_kernel<<<ka.nchains, 64, 0, st>>>(ka);
    return cudaGetLastError();
}
cudaError_t launch_point_average(const KernelArgs& ka, int npts, const int* start, const int* list, double* out,
                                 cudaStream_t st) {
    point_average_kernel<<<npts, 64, 0, st>>>(ka, start, list, out);
    return cudaGetLastError();
}
cudaError_t launch_stats_add(const double* pout, double* cur, double* blk, int n, int finish, int block_size,
                             cudaStream_t st) {
    stats_add_kernel<<<(n + 255) / 256, 256, 0, st>>>(pout, cur, blk, n, finish, block_size);
    return cudaGetLastError();
}
cudaError_t launch_stats_final(const double* blk, int nb, int n, double* mean, double* sem, cudaStream_t st) {
    stats_final_kernel<<<(n + 255) / 256, 256, 0, st>>>(blk, nb, n, mean, sem);
    return cudaGetLastError();
}
cudaError_t launch_global_propose(const KernelArgs& ka, const KernelArgs& kp, const double* shift, cudaStream_t st) {
    global_propose_kernel<<<ka.nchains, 256, 0, st>>>(ka, kp, shift[0], shift[1]);
    return cudaGetLastError();
}
cudaError_t launch_global_accept(const KernelArgs& ka, const KernelArgs& kp, const double* fn, const double* fn2,
                                 const double* hastings, int* accepted, cudaStream_t st) {
    global_accept_kernel<<<ka.nchains, 256, 0, st>>>(ka, kp, fn, fn2, hastings, accepted);
    return cudaGetLastError();
}
cudaError_t launch_field_check(const KernelArgs& ka, int* bad, cudaStream_t st) {
    field_check_kernel<<<ka.nchains, 256, 0, st>>>(ka, bad);
    return cudaGetLastError();
}
cudaError_t launch_field_norm(const KernelArgs& ka, double* out, cudaStream_t st) {
    field_norm_kernel<<<ka.nchains, 256, 0, st>>>(ka, out);
    return cudaGetLastError();
}
long long class_work_elems(int cls) {
    if (cls == 6) return 5LL * 144 * Cfg<144>::LD;   // W1, W2, G, U, product scratch
    const int sz = cls % 3;
    auto w = [](int nmax, int ld, bool gw) { return gw ? 2LL * nmax * ld : 0LL; };
    return sz == 0 ? w(16, Cfg<16>::LD, Cfg<16>::GW)
                   : (sz == 1 ? w(36, Cfg<36>::LD, Cfg<36>::GW) : w(72, Cfg<72>::LD, Cfg<72>::GW));
}
bool class_hbm_work(int cls) { return cls == 6 || cls % 3 == 2; }
int point_real_ld(int n) { return real_ld(n); }
size_t smem_bytes(int cls) {
    if (cls == 6) return Smem<144>::bytes();
    const int sz = cls % 3;
    return sz == 0 ? Smem<16>::bytes() : (sz == 1 ? Smem<36>::bytes() : Smem<72>::bytes());
}
int class_nmax(int cls) {
    if (cls == 6) return 144;
    const int sz = cls % 3;
    return sz == 0 ? 16 : (sz == 1 ? 36 : 72);
}
int class_of(int n, int pairing) {
    for (int c = 0; c < 3; ++c)
        if (n <= class_nmax(c)) return c + (pairing ? 3 : 0);
    if (!pairing && n <= 144) return 6;
    return -1;
}

}  // namespace bq
