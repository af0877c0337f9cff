// Device code shared by the FP64 GETT kernels: cp.async, the m16n8k8 DMMA and the K loop of a 64 x 64 output tile.
#pragma once
#include "kernels.cuh"

namespace ccqb {

constexpr int BM = 64, BN = 64, BKT = 16, PADS = 4;
// Shared-memory operand tiles: m-major operands are stored [k][m] (row stride MS),
// k-major ones [m][k] (row stride KS), so that each can be filled with 16-byte
// copies along its contiguous mode; both strides keep the fragment reads of a
// half-warp on 16 distinct banks.
constexpr int MS = BM + PADS;   // 68
constexpr int KS = BKT + 4;     // 20
constexpr int TILE = BM * KS;   // doubles per tile buffer (>= BKT * MS)
static_assert(BKT * MS <= TILE, "tile buffer");
template <bool KMAJ>
__device__ __forceinline__ int tix(int k, int m) { return KMAJ ? m * KS + k : k * MS + m; }

__device__ __forceinline__ void cp_async8(void *smem, const void *gmem, bool pred) {
    unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
    int sz = pred ? 8 : 0;
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(s), "l"(gmem), "r"(sz));
}
__device__ __forceinline__ void cp_async16(void *smem, const void *gmem, bool pred) {
    unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
    int sz = pred ? 16 : 0;
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(sz));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

// m16n8k8 (sm_90 and later): a = {(g, t), (g + 8, t), (g, t + 4), (g + 8, t + 4)}, b = {(t, g), (t + 4, g)}
// for lane group g and thread-in-group t, as (row, k) and (k, column)
__device__ __forceinline__ void dmma_16x8x8(double (&c)[4], const double (&a)[4], const double (&b)[2]) {
    asm volatile(
        "mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
        : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b[0]), "d"(b[1]));
}

// Loads one BKT x BM tile of a GETT operand into shared memory (layout tix).
// kmajor: consecutive threads walk k (operand stride-1 along its k modes),
// else they walk m.  vec: the walked mode pairs up contiguous, 16-byte aligned
// elements, copied 16 bytes at a time.  Out-of-range elements are zero-filled.
template <bool KMAJOR>
__device__ __forceinline__ void load_tile(double *S, const double *base, const int *offm_reg, const int *offk, int m0,
                                          int M, int k0, int kend, int tid, bool vec) {
    if (KMAJOR && vec) {
        int kk = 2 * (tid & 7);
        int mrow = tid >> 3;
        int k = k0 + kk;
        bool kin = k < kend;
        int ok = kin ? __ldg(offk + k) : 0;
#pragma unroll
        for (int p = 0; p < 4; ++p) {
            int m = mrow + 16 * p;
            bool in = kin && (m0 + m < M);
            const double *src = in ? base + (long long)offm_reg[p] + ok : base;
            cp_async16(&S[tix<true>(kk, m)], src, in);
        }
    } else if (KMAJOR) {
        int kk = tid & 15;
        int mrow = tid >> 4;
        int k = k0 + kk;
        bool kin = k < kend;
        int ok = kin ? __ldg(offk + k) : 0;
#pragma unroll
        for (int p = 0; p < 8; ++p) {
            int m = mrow + 8 * p;
            bool in = kin && (m0 + m < M);
            const double *src = in ? base + (long long)offm_reg[p] + ok : base;
            cp_async8(&S[tix<true>(kk, m)], src, in);
        }
    } else if (vec) {
        // pairs (m, m+1) are contiguous and 16-byte aligned: half the copies
        int m = 2 * (tid & 31);
        int krow = tid >> 5;
        bool min_ = (m0 + m) < M;
#pragma unroll
        for (int p = 0; p < 4; ++p) {
            int kk = krow + 4 * p;
            int k = k0 + kk;
            bool in = min_ && k < kend;
            const double *src = in ? base + (long long)offm_reg[0] + __ldg(offk + k) : base;
            cp_async16(&S[tix<false>(kk, m)], src, in);
        }
    } else {
        int m = tid & 63;
        int krow = tid >> 6;
        bool min_ = (m0 + m) < M;
#pragma unroll
        for (int p = 0; p < 8; ++p) {
            int kk = krow + 2 * p;
            int k = k0 + kk;
            bool in = min_ && k < kend;
            const double *src = in ? base + (long long)offm_reg[0] + __ldg(offk + k) : base;
            cp_async8(&S[tix<false>(kk, m)], src, in);
        }
    }
}

// The MMAs of one staged BKT-deep K tile into a warp's 32 x 32 accumulator block.
template <bool AK, bool BKM>
__device__ __forceinline__ void mma_stage(double (&acc)[2][4][4], const double *As, const double *Bs, int wm, int wn,
                                          int gid, int tig, int nk) {
#pragma unroll
    for (int kk = 0; kk < BKT; kk += 8) {
        if (kk >= nk) break;   // the rest of the tile is the zero fill past the K range
        double a[2][4], b[4][2];
#pragma unroll
        for (int mi = 0; mi < 2; ++mi)
#pragma unroll
            for (int q = 0; q < 4; ++q)
                a[mi][q] = As[tix<AK>(kk + tig + 4 * (q >> 1), wm + mi * 16 + gid + 8 * (q & 1))];
#pragma unroll
        for (int ni = 0; ni < 4; ++ni)
#pragma unroll
            for (int q = 0; q < 2; ++q) b[ni][q] = Bs[tix<BKM>(kk + tig + 4 * q, wn + ni * 8 + gid)];
#pragma unroll
        for (int mi = 0; mi < 2; ++mi)
#pragma unroll
            for (int ni = 0; ni < 4; ++ni) dmma_16x8x8(acc[mi][ni], a[mi], b[ni]);
    }
}

// K loop of one contraction term over [kbeg, kend): NST-stage cp.async pipeline
// (As and Bs hold NST tiles each; one commit group per K tile, empty past the end).
template <bool AK, bool BKM, int NST>
__device__ __forceinline__ void gett_mainloop(double (&acc)[2][4][4], double *As, double *Bs, const double *A,
                                              const double *B,
                                              const int *offA_m, const int *offA_k, const int *offB_n,
                                              const int *offB_k, int M, int N, int m0, int n0, int kbeg, int kend,
                                              int tid, int wm, int wn, int gid, int tig, bool va, bool vb) {
    int offa[8], offb[8];
    if (AK) {
#pragma unroll
        for (int p = 0; p < 8; ++p) {
            int m = m0 + (va ? (tid >> 3) + 16 * p : (tid >> 4) + 8 * p);
            offa[p] = (m < M && (!va || p < 4)) ? __ldg(offA_m + m) : 0;
        }
    } else {
        int m = m0 + (va ? 2 * (tid & 31) : (tid & 63));
        offa[0] = m < M ? __ldg(offA_m + m) : 0;
    }
    if (BKM) {
#pragma unroll
        for (int p = 0; p < 8; ++p) {
            int n = n0 + (vb ? (tid >> 3) + 16 * p : (tid >> 4) + 8 * p);
            offb[p] = (n < N && (!vb || p < 4)) ? __ldg(offB_n + n) : 0;
        }
    } else {
        int n = n0 + (vb ? 2 * (tid & 31) : (tid & 63));
        offb[0] = n < N ? __ldg(offB_n + n) : 0;
    }
    const int ntiles = kend > kbeg ? (kend - kbeg + BKT - 1) / BKT : 0;
#pragma unroll
    for (int q = 0; q < NST - 1; ++q) {
        if (q < ntiles) {
            load_tile<AK>(As + q * TILE, A, offa, offA_k, m0, M, kbeg + q * BKT, kend, tid, va);
            load_tile<BKM>(Bs + q * TILE, B, offb, offB_k, n0, N, kbeg + q * BKT, kend, tid, vb);
        }
        cp_async_commit();
    }
    for (int t = 0; t < ntiles; ++t) {
        const int st = t % NST;
        // refill the stage computed in the previous step (released by its trailing barrier)
        const int tn = t + NST - 1;
        if (tn < ntiles) {
            const int sn = tn % NST;
            load_tile<AK>(As + sn * TILE, A, offa, offA_k, m0, M, kbeg + tn * BKT, kend, tid, va);
            load_tile<BKM>(Bs + sn * TILE, B, offb, offB_k, n0, N, kbeg + tn * BKT, kend, tid, vb);
        }
        cp_async_commit();
        cp_async_wait<NST - 1>();   // tile t has landed
        __syncthreads();
        mma_stage<AK, BKM>(acc, As + st * TILE, Bs + st * TILE, wm, wn, gid, tig, kend - (kbeg + t * BKT));
        __syncthreads();
    }
}

}  // namespace ccqb
