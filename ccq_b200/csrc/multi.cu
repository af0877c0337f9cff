// Many small contractions in one launch.
//
// A CC sweep is a few hundred contractions of which most take less time than a kernel launch: per launch the
// front end needs 1.2-2.4 us and a dependent kernel another 4-6 us of table loads, operand loads and epilogue,
// whatever the size.  The runtime therefore collects all small contractions whose inputs are ready at the same
// time and runs them as one grid: one block per item, an item being one output tile and one K range of one
// contraction (MultiItem, built once on the host with the tile's offset-table positions in it).
//
// An item is bound by latency, so it is laid out for the shortest chain: item -> offset tables -> operands ->
// DMMA -> output, with no dependent load beyond those.  Direct items load their operands straight from L2 to the
// m16n8k8 fragments (a fragment load touches whole 32-byte sectors in either orientation).  With more than two K slabs
// the four warps take them in turn (a chain of DMMAs on one scheduler takes 64 clocks each) and add up through shared
// memory; with one or two, each warp has its own rows.  Where a contraction's 64 x 64 tiles fill most of the chip they
// are used instead (gett_multi64_kernel).  Items of one output add with reductions (the output starts at zero or
// holds earlier terms), so a contraction's K ranges and the terms of one sum need no order among themselves; an item that
// overwrites is the only one of its output tile.
//
// One B200, a pass of six iterations, one launch per contraction -> shared launches: CCSD of 8 orbitals 1.98 ->
// 1.08 ms (138 -> 28 launches per sweep), 20 orbitals 2.33 -> 1.34 ms, eight CCSD systems of 16 to 30 orbitals at
// once 18.7 -> 6.5 ms, CCSDT of 13 orbitals 4.91 -> 1.88 ms (537 -> 56 launches), of 24 orbitals 9.50 -> 6.89 ms, left
// CCSD and CR-CC(2,3) of 32 orbitals 25.5 -> 13.2 ms.
#include "gett_tile.cuh"

namespace ccqb {

namespace {

constexpr int MT_THREADS = 128;

template <int MI, int NI>
struct Slab {
    double a[MI][4], b[NI][2];
};

template <int MI, int NI>
__device__ __forceinline__ void load_slab(Slab<MI, NI> &f, const MultiItem &it, const int (&ra)[MI][2],
                                          const int (&rb)[NI], const int *sa, const int *sb, int s, int tig) {
    int ka[2], kb[2];
    bool in[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const int k = s * 8 + tig + 4 * q;
        in[q] = k < it.k;
        ka[q] = sa[k];
        kb[q] = sb[k];
    }
#pragma unroll
    for (int mi = 0; mi < MI; ++mi)
#pragma unroll
        for (int q = 0; q < 4; ++q)
            f.a[mi][q] = in[q >> 1] ? it.A[(long long)ra[mi][q & 1] + ka[q >> 1]] : 0.0;
#pragma unroll
    for (int ni = 0; ni < NI; ++ni)
#pragma unroll
        for (int q = 0; q < 2; ++q) f.b[ni][q] = in[q] ? it.B[(long long)rb[ni] + kb[q]] : 0.0;
}

template <int MI, int NI>
__device__ __forceinline__ void mma_slab(double (&acc)[MI][NI][4], const Slab<MI, NI> &f) {
#pragma unroll
    for (int mi = 0; mi < MI; ++mi)
#pragma unroll
        for (int ni = 0; ni < NI; ++ni) dmma_16x8x8(acc[mi][ni], f.a[mi], f.b[ni]);
}

__device__ __forceinline__ void put(double *p, double v, bool add) {
    if (add)
        atomicAdd(p, v);
    else
        *p = v;
}

template <int MI, int NI>
__device__ __forceinline__ void multi_tile(const MultiItem &it, double *red, int *sa, int *sb) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int gid = lane >> 2, tig = lane & 3;
    const int nsl = (it.k + 7) >> 3;
    const bool ks = it.flags & MI_KSPLIT, add = it.flags & MI_ADD;
    for (int i = tid; i < nsl * 8; i += MT_THREADS) {
        const bool in = i < it.k;
        sa[i] = in ? __ldg(it.ak + i) : 0;
        sb[i] = in ? __ldg(it.bk + i) : 0;
    }
    // rows and columns past the tile read the tile's first one and are not written
    const int wm = ks ? 0 : warp * MI * 16;
    int ra[MI][2], rb[NI];
#pragma unroll
    for (int mi = 0; mi < MI; ++mi)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int m = wm + mi * 16 + gid + 8 * h;
            ra[mi][h] = __ldg(it.am + (m < it.m ? m : 0));
        }
#pragma unroll
    for (int ni = 0; ni < NI; ++ni) {
        const int n = ni * 8 + gid;
        rb[ni] = __ldg(it.bn + (n < it.n ? n : 0));
    }
    double acc[MI][NI][4];
#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int j = 0; j < NI; ++j)
#pragma unroll
            for (int q = 0; q < 4; ++q) acc[i][j][q] = 0.0;
    gdc_wait();   // the tables above are constant; operands and output may be the previous kernel's
    __syncthreads();
    if (wm < it.m) {
        const int step = ks ? 4 : 1;
        int s = ks ? warp : 0;
        for (; s < nsl; s += step) {
            Slab<MI, NI> f;
            load_slab<MI, NI>(f, it, ra, rb, sa, sb, s, tig);
            mma_slab<MI, NI>(acc, f);
        }
    }
    if (!ks) {
        if (wm >= it.m) return;
#pragma unroll
        for (int mi = 0; mi < MI; ++mi)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int m = wm + mi * 16 + gid + 8 * h;
                if (m >= it.m) continue;
                double *row = it.C + __ldg(it.cm + m);
#pragma unroll
                for (int ni = 0; ni < NI; ++ni)
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        const int n = ni * 8 + 2 * tig + j;
                        if (n < it.n) put(row + __ldg(it.cn + n), it.alpha * acc[mi][ni][2 * h + j], add);
                    }
            }
        return;
    }
    constexpr int RED_LD = NI * 8 + 2;   // fragment pairs stay 16-byte aligned
    // partial tiles of the four warps, added up in a fixed order and written along C's contiguous mode
#pragma unroll
    for (int mi = 0; mi < MI; ++mi)
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int ni = 0; ni < NI; ++ni)
                *reinterpret_cast<double2 *>(
                    &red[(warp * MI * 16 + mi * 16 + gid + 8 * h) * RED_LD + ni * 8 + 2 * tig]) =
                    make_double2(acc[mi][ni][2 * h], acc[mi][ni][2 * h + 1]);
    __syncthreads();
    constexpr int TM = MI * 16, TN = NI * 8;
    const bool nfast = it.flags & MI_NFAST;
#pragma unroll
    for (int e = tid; e < TM * TN; e += MT_THREADS) {
        const int m = nfast ? e / TN : e % TM, n = nfast ? e % TN : e / TM;
        if (m >= it.m || n >= it.n) continue;
        double v = 0.0;
#pragma unroll
        for (int w = 0; w < 4; ++w) v += red[(w * TM + m) * RED_LD + n];
        put(it.C + __ldg(it.cm + m) + __ldg(it.cn + n), it.alpha * v, add);
    }
}

// 64 x 64 tile: the operands of every K slab staged in shared memory, each warp a 32 x 32 quarter.  A 32 x 32 tile
// reads its operands from L2 at 32 bytes per clock and SM for every DMMA the pipe can take, about all that L2
// delivers; this one needs half of that.
template <bool AK, bool BK>
__device__ __forceinline__ void multi_tile64(const MultiItem &it, double *sm) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int gid = lane >> 2, tig = lane & 3, wm = (warp >> 1) * 32, wn = (warp & 1) * 32;
    double acc[2][4][4];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int q = 0; q < 4; ++q) acc[i][j][q] = 0.0;
    gett_mainloop<AK, BK, 2>(acc, sm, sm + 2 * TILE, it.A, it.B, it.am, it.ak, it.bn, it.bk, it.m, it.n, 0, 0, 0, it.k,
                             tid, wm, wn, gid, tig, (it.flags & MI_VA) != 0, (it.flags & MI_VB) != 0);
    const bool add = it.flags & MI_ADD;
    int cn[4][2];
#pragma unroll
    for (int ni = 0; ni < 4; ++ni)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int n = wn + ni * 8 + 2 * tig + j;
            cn[ni][j] = n < it.n ? __ldg(it.cn + n) : -1;
        }
#pragma unroll
    for (int mi = 0; mi < 2; ++mi)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int m = wm + mi * 16 + gid + 8 * h;
            if (m >= it.m) continue;
            double *row = it.C + __ldg(it.cm + m);
#pragma unroll
            for (int ni = 0; ni < 4; ++ni)
#pragma unroll
                for (int j = 0; j < 2; ++j)
                    if (cn[ni][j] >= 0) put(row + cn[ni][j], it.alpha * acc[mi][ni][2 * h + j], add);
        }
}

// partial tiles of four warps: 16 x 16, 32 x 8, 32 x 16 or 16 x 32, rows padded by two
constexpr int RED = 4 * 32 * 18;

// Direct and one-column items, copies: bound by latency, so registers and shared memory are held down to seven
// blocks per SM instead of loading ahead within a warp (six iterations of CCSDT at 24 orbitals 6.7 ms; with the next
// slab loaded ahead at 128 registers and four blocks 7.3 ms).
__global__ void __launch_bounds__(MT_THREADS, 7) gett_multi_kernel(const MultiItem *__restrict__ items) {
    __shared__ __align__(16) double sm[RED];
    __shared__ int sa[MULTI_K], sb[MULTI_K];
    gdc_launch();
    const MultiItem it = items[blockIdx.x];
    switch (it.flags >> MI_SHAPE) {
        case 0: multi_tile<1, 2>(it, sm, sa, sb); break;
        case 1: multi_tile<2, 1>(it, sm, sa, sb); break;
        case 2: multi_tile<2, 2>(it, sm, sa, sb); break;
        case 3: multi_tile<1, 4>(it, sm, sa, sb); break;
        case MS_VEC: {
            // one column, a few k: one thread per row, no tile
            constexpr int R = MULTI_VEC_ROWS / MT_THREADS;
            int ra[R];
            double v[R];
#pragma unroll
            for (int u = 0; u < R; ++u) {
                const int m = threadIdx.x + u * MT_THREADS;
                ra[u] = m < it.m ? __ldg(it.am + m) : -1;
                v[u] = 0.0;
            }
            const int rb = __ldg(it.bn);
            gdc_wait();
            // all rows' loads before the first store, which an ordinary load may not pass (row by row, and value by
            // value in the copies below: CCSD at 33 orbitals 1.52 against 1.46 ms, CCSDT at 24 orbitals 6.02 / 5.87 ms)
            for (int k = 0; k < it.k; ++k) {
                const int ka = __ldg(it.ak + k);
                const double b = it.B[(long long)rb + __ldg(it.bk + k)];
#pragma unroll
                for (int u = 0; u < R; ++u)
                    if (ra[u] >= 0) v[u] += it.A[(long long)ra[u] + ka] * b;
            }
#pragma unroll
            for (int u = 0; u < R; ++u) {
                const int m = threadIdx.x + u * MT_THREADS;
                if (ra[u] >= 0) put(it.C + __ldg(it.cm + m) + __ldg(it.cn), it.alpha * v[u], it.flags & MI_ADD);
            }
            break;
        }
        default: {
            // copy (A to C) or zero (A null) of m values; the loads first, as above
            constexpr int R = MULTI_COPY / MT_THREADS;
            double v[R];
            gdc_wait();
#pragma unroll
            for (int u = 0; u < R; ++u) {
                const int i = threadIdx.x + u * MT_THREADS;
                v[u] = it.A && i < it.m ? it.A[i] : 0.0;
            }
#pragma unroll
            for (int u = 0; u < R; ++u) {
                const int i = threadIdx.x + u * MT_THREADS;
                if (i < it.m) it.C[i] = v[u];
            }
        }
    }
}

__global__ void __launch_bounds__(MT_THREADS, 4) gett_multi64_kernel(const MultiItem *__restrict__ items) {
    __shared__ __align__(16) double sm[4 * TILE];   // two stages of both operands
    gdc_launch();
    const MultiItem it = items[blockIdx.x];
    gdc_wait();
    switch ((it.flags >> MI_SHAPE) - MS_64) {
        case 0: multi_tile64<false, false>(it, sm); break;
        case 1: multi_tile64<false, true>(it, sm); break;
        case 2: multi_tile64<true, false>(it, sm); break;
        default: multi_tile64<true, true>(it, sm); break;
    }
}

}  // namespace

void launch_gett_multi(const MultiItem *items, int n, bool tiles64, cudaStream_t s) {
    if (n <= 0) return;
    if (tiles64)
        launch_after(n <= kEarlyBlocks, gett_multi64_kernel, n, MT_THREADS, 0, s, items);
    else
        launch_after(n <= kEarlyBlocks, gett_multi_kernel, n, MT_THREADS, 0, s, items);
}

cudaError_t preload_multi() {
    cudaFuncAttributes fa;
    const cudaError_t e = cudaFuncGetAttributes(&fa, gett_multi_kernel);
    return e == cudaSuccess ? cudaFuncGetAttributes(&fa, gett_multi64_kernel) : e;
}

}  // namespace ccqb
