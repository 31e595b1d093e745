// Weight gradient of a 3x3x3 layer on the tensor cores:
//   dW[k][o][i] = sum_p g[p][o] x[nbr(p, k)][i],   db[o] = sum_p g[p][o],
// a product of M = output channels by N = input channels over K = the points of the
// batch, for each of the 27 taps, in bf16 with float32 accumulation.
//
// A plane (8 channels) is a column of 16-byte rows, one per time slice, so a run of
// slices of one plane is a K x 8 block with the channels contiguous: ldmatrix.trans
// gives the fragments of both operands from it, and a time offset of the tap is a row
// offset.  A block takes one spatial offset (b, c), stages 32 slices of g and 34 of x
// of a (chain, site) pair per step (cp.async, four stages) and accumulates its three
// time taps from the same rows: 12 m16n8k16 per five ldmatrix.x4 of a warp.  K is split
// over blocks so that a float32 accumulator takes at most 640 points before it is added
// to the result in global memory (the batch has 10^5 to 10^6): the tensor cores truncate
// where they add, and 2560 points left 3e-6 of the gradient, 640 less than 1e-6 (and are
// no slower: 3.54 against 3.71 ms for the whole call, on one host).
//
// Bound: issue and latency of 16 warps an SM (registers allow two blocks): issue slots 44%,
// shared-memory wavefronts 44%, tensor pipe 35% of their peaks.  64 -> 64 channels, 64
// configurations of 6x6 x 160: 0.44 ms a layer, 81 GFLOP, 0.11 of the measured bf16 peak; the
// CUDA-core products of one tap per block that it replaces (27 reads of g and x, scalar
// shared-memory operands) took 39 of the 42 ms of the whole gradient, which is 3.5 to 3.7 ms
// now, by the host that converts the configurations.  tcgen05 has not been tried: it takes these
// operands as tiles with K along the rows.
#pragma once
#include <climits>

#include <cuda_bf16.h>

#include "net.h"
#include "sweep.cuh"

namespace bq {

constexpr int kWgThreads = 256, kWgRows = 32, kWgStages = 4, kWgPoints = 640;

struct WgradMmaArgs {
    NetShape s;
    const __nv_bfloat16* x;   // layer input, PI planes
    const __nv_bfloat16* g;   // gradient of the layer's pre-activation, PO planes
    int cin, cout;
    float* dw;                // [27][cout][cin]
    float* db;                // [cout]
    long long items;          // runs of 32 slices of the batch's (chain, site) pairs
    int per;                  // runs per block
};

// How the batch is split over blocks: a pair's slices are runs of kWgRows (the last one short), and a block
// takes `per` runs in sequence, whole pairs of at most kWgPoints points in all where a pair has fewer than
// that, kWgPoints points of a longer one.  The chunks go on the grid's x, whose limit (2^31 - 1) a batch that
// fits the memory does not reach.
struct WgradSplit {
    long long items, chunks;
    int per;
};
inline WgradSplit wgrad_split(int L, long long pairs) {
    WgradSplit w;
    const int runs = (L + kWgRows - 1) / kWgRows;
    w.items = pairs * runs;
    w.per = L < kWgPoints ? kWgPoints / L * runs : kWgPoints / kWgRows;
    w.chunks = (w.items + w.per - 1) / w.per;
    return w;
}

template <int PO, int PI>
struct WgradCfg {
    // warps along M x along N, and m16 x n8 tiles of a warp
    static constexpr int WM = PO == 8 && PI == 8 ? 2 : 1, WN = PO == 8 && PI == 8 ? 2 : 1;
    static constexpr int NM = PO / 2 / WM, NN = PI / WN;
    static_assert(NM * NN == kWgThreads / 32, "one tile group per warp");
    static constexpr int kRowsX = kWgRows + 2;
    static constexpr int kStage = (PO * kWgRows + PI * kRowsX) * 16;   // bytes
};

DEVI void wg_cp16(uint32_t dst, const void* src, bool ok) {   // zeros if !ok
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(ok ? 16 : 0) : "memory");
}
DEVI void wg_ldsm4(uint32_t a, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(a)
                 : "memory");
}
DEVI void wg_ldsm2(uint32_t a, uint32_t& r0, uint32_t& r1) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0, %1}, [%2];" : "=r"(r0), "=r"(r1) : "r"(a) : "memory");
}
DEVI void wg_mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// grid 9 chunks: the nine spatial offsets of a chunk run side by side and share its rows in L2
template <int PO, int PI>
__global__ void __launch_bounds__(kWgThreads, 2) wgrad_mma_kernel(WgradMmaArgs a) {
    using C = WgradCfg<PO, PI>;
    __shared__ __align__(128) unsigned char sm[kWgStages * C::kStage];
    const NetShape& s = a.s;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int off = blockIdx.x % 9, ob = off / 3 - 1, oc = off % 3 - 1;
    const int ntc = (s.L + kWgRows - 1) / kWgRows;
    const long long i0 = (long long)(blockIdx.x / 9) * a.per;
    const int items = (int)min((long long)a.per, a.items - i0);
    const int p0 = (int)(i0 / ntc), r0 = (int)(i0 - (long long)p0 * ntc);
    const uint32_t base = (uint32_t)__cvta_generic_to_shared(sm);
    const long long prow = s.L + 2;   // rows of a plane

    // stage item it (run r0 + it from the first of pair p0) into slot it % kWgStages
    const auto fill = [&](int it) {
        if (it < items) {
            const int pr = (r0 + it) / ntc, t0 = (r0 + it - pr * ntc) * kWgRows, p = p0 + pr;
            const int b = p / s.Ns, site = p - b * s.Ns, y = site / s.Lx, xx = site - y * s.Lx;
            const int yn = y + ob + (y + ob < 0 ? s.Ly : 0) - (y + ob >= s.Ly ? s.Ly : 0);
            const int xn = xx + oc + (xx + oc < 0 ? s.Lx : 0) - (xx + oc >= s.Lx ? s.Lx : 0);
            const __nv_bfloat16* gp = a.g + (long long)p * PO * prow * 8;
            const __nv_bfloat16* xp = a.x + ((long long)b * s.Ns + yn * s.Lx + xn) * PI * prow * 8;
            const uint32_t dst = base + (it % kWgStages) * C::kStage;
            for (int e = tid; e < PO * kWgRows; e += kWgThreads) {
                const int q = e / kWgRows, r = e % kWgRows, t = t0 + r;   // row t + 1; slices past the end as zeros
                wg_cp16(dst + e * 16, gp + (q * prow + min(t + 1, s.L)) * 8, t < s.L);
            }
            for (int e = tid; e < PI * C::kRowsX; e += kWgThreads) {
                const int q = e / C::kRowsX, r = e % C::kRowsX, tp = t0 + r;
                wg_cp16(dst + PO * kWgRows * 16 + e * 16, xp + (q * prow + min(tp, s.L + 1)) * 8, tp <= s.L + 1);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    float acc[3][C::WM][C::WN][4];
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int i = 0; i < C::WM; ++i)
#pragma unroll
            for (int j = 0; j < C::WN; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[k][i][j][e] = 0.f;
    float bsum = 0.f;
    const int wm = warp % C::NM, wn = warp / C::NM;
    const int mat = lane >> 3, r8 = lane & 7;
#pragma unroll
    for (int k = 0; k < kWgStages - 1; ++k) fill(k);
    for (int it = 0; it < items; ++it) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kWgStages - 2) : "memory");
        __syncthreads();   // item it is in place, and every warp is done with the slot that fill() takes next
        fill(it + kWgStages - 1);
        const uint32_t sg = base + (it % kWgStages) * C::kStage, sx = sg + PO * kWgRows * 16;
#pragma unroll
        for (int k0 = 0; k0 < kWgRows; k0 += 16) {
            uint32_t af[C::WM][4];
#pragma unroll
            for (int i = 0; i < C::WM; ++i) {
                const int plane = 2 * (wm * C::WM + i) + (mat & 1), row = k0 + (mat >> 1) * 8 + r8;
                wg_ldsm4(sg + (plane * kWgRows + row) * 16, af[i]);
            }
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                if constexpr (C::WN == 2) {
                    uint32_t bf[4];
                    const int plane = wn * 2 + (mat >> 1), row = k0 + (mat & 1) * 8 + r8 + k;
                    wg_ldsm4(sx + (plane * C::kRowsX + row) * 16, bf);
#pragma unroll
                    for (int i = 0; i < C::WM; ++i) {
                        wg_mma(acc[k][i][0], af[i], bf[0], bf[1]);
                        wg_mma(acc[k][i][1], af[i], bf[2], bf[3]);
                    }
                } else {
                    uint32_t b0, b1;
                    const int row = k0 + (mat & 1) * 8 + r8 + k;
                    wg_ldsm2(sx + (wn * C::kRowsX + row) * 16, b0, b1);
#pragma unroll
                    for (int i = 0; i < C::WM; ++i) wg_mma(acc[k][i][0], af[i], b0, b1);
                }
            }
        }
        if (off == 4) {   // the bias gradient, once per pair: thread (channel, row group)
            constexpr int CH = PO * 8, GR = kWgThreads / CH, RG = kWgRows / GR;
            const int o = tid % CH, rg = tid / CH;
            const __nv_bfloat16* gs =
                reinterpret_cast<const __nv_bfloat16*>(sm + (it % kWgStages) * C::kStage) + (o >> 3) * kWgRows * 8 + (o & 7);
#pragma unroll
            for (int r = 0; r < RG; ++r) bsum += __bfloat162float(gs[(rg * RG + r) * 8]);
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    // fragment element (row lane / 4 (+ 8), columns 2 (lane % 4), + 1)
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int i = 0; i < C::WM; ++i)
#pragma unroll
            for (int j = 0; j < C::WN; ++j)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int o = (wm * C::WM + i) * 16 + h * 8 + (lane >> 2), in = (wn * C::WN + j) * 8 + 2 * (lane & 3);
                    if (o < a.cout && in + 1 < a.cin) {
                        float* d = a.dw + ((long long)(3 * off + k) * a.cout + o) * a.cin + in;
                        asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(d), "f"(acc[k][i][j][2 * h]),
                                     "f"(acc[k][i][j][2 * h + 1])
                                     : "memory");
                    }
                }
    if (off == 4 && tid % (PO * 8) < a.cout) atomicAdd(a.db + tid % (PO * 8), bsum);
}

// whether the layer's weight gradient runs here (64 channels on the wide sides)
inline bool wgrad_mma_applies(const NetShape& s, int l) {
    const int po = s.pout[l], pi = s.pin[l];
    return (po == 8 && (pi == 8 || pi == 2)) || (po == 2 && pi == 8);
}

inline cudaError_t launch_wgrad_mma(const NetShape& s, int l, int chains, const __nv_bfloat16* x, const __nv_bfloat16* g,
                                    float* dw, float* db, cudaStream_t st) {
    WgradMmaArgs a{};
    a.s = s;
    a.x = x;
    a.g = g;
    a.cin = s.cin[l];
    a.cout = s.cout[l];
    a.dw = dw;
    a.db = db;
    const WgradSplit w = wgrad_split(s.L, (long long)chains * s.Ns);
    a.items = w.items;
    a.per = w.per;
    if (w.chunks > INT_MAX / 9) return cudaErrorInvalidValue;
    const unsigned grid = 9u * (unsigned)w.chunks;
    if (s.pout[l] == 8 && s.pin[l] == 8) wgrad_mma_kernel<8, 8><<<grid, kWgThreads, 0, st>>>(a);
    else if (s.pout[l] == 8) wgrad_mma_kernel<8, 2><<<grid, kWgThreads, 0, st>>>(a);
    else wgrad_mma_kernel<2, 8><<<grid, kWgThreads, 0, st>>>(a);
    return cudaGetLastError();
}

}  // namespace bq
