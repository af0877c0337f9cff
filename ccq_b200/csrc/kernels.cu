// Device kernels of libccq_b200; see kernels.cuh for the role of each.
#include "kernels.cuh"
#include "gett_tile.cuh"

#include <algorithm>
#include <mutex>

namespace ccqb {

// ---------------------------------------------------------------------------
// GETT, FP64 on the DMMA tensor pipe
// ---------------------------------------------------------------------------
// One 64 x 64 output tile (bx, by) of a GETT, K slice bz; split: several K slices add into C.
template <bool AK, bool BKM, bool GROUPED, int NST>
__device__ __forceinline__ void gett_f64_tile(const GettArgs &g, int bx, int by, int bz, bool split) {
    extern __shared__ __align__(16) double smem[];
    double *As = smem;
    double *Bs = smem + NST * TILE;
    const int tid = threadIdx.x;
    const int lane = tid & 31, warp = tid >> 5;
    const int wm = (warp >> 1) * 32, wn = (warp & 1) * 32;
    const int gid = lane >> 2, tig = lane & 3;
    const int m0 = bx * BM, n0 = by * BN;

    double acc[2][4][4];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int q = 0; q < 4; ++q) acc[i][j][q] = 0.0;

    double alpha = g.alpha;
    if (GROUPED) {
        // grouped: sum_s alpha_s A_s B_s^T, rescaling the running sum between terms
        for (int sgi = 0; sgi < g.nseg; ++sgi) {
            const GettSeg sg = g.segs[sgi];
            if (sgi > 0) {
                double r = g.segs[sgi - 1].alpha / sg.alpha;
#pragma unroll
                for (int i = 0; i < 2; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j)
#pragma unroll
                        for (int q = 0; q < 4; ++q) acc[i][j][q] *= r;
            }
            gett_mainloop<AK, BKM, NST>(acc, As, Bs, sg.A, sg.B, sg.offA_m, sg.offA_k, sg.offB_n, sg.offB_k, g.M, g.N, m0,
                                   n0, 0, sg.K, tid, wm, wn, gid, tig, g.vec_a != 0, g.vec_b != 0);
            alpha = sg.alpha;
        }
    } else {
        const int kbeg = bz * g.kchunk;
        const int kend = min(g.K, kbeg + g.kchunk);
        gett_mainloop<AK, BKM, NST>(acc, As, Bs, g.A, g.B, g.offA_m, g.offA_k, g.offB_n, g.offB_k, g.M, g.N, m0, n0, kbeg,
                               kend, tid, wm, wn, gid, tig, g.vec_a != 0, g.vec_b != 0);
    }

    // epilogue: stage the tile in shared memory, then write along the output's
    // contiguous mode (g.c_nfast) so that stores and the beta read coalesce
    // C tile layout: rows along the output's contiguous mode, so that the write-out reads rows.  [m][n]
    // with row stride CSN = BN + 8 when n is the fast mode (the fragments' (j = 0, 1) pairs are stored as
    // one 16-byte access, conflict-free per 8 lanes), else [n][m] with stride CSM = BM + 2 (scalar stores,
    // conflict-free per half-warp)
    constexpr int CSN = BN + 8, CSM = BM + 2;
    constexpr int CS_ELEMS = BM * CSN > BN * CSM ? BM * CSN : BN * CSM;
    static_assert(CS_ELEMS * 2 + BM + BN <= 8 * TILE, "C tile and output tables must fit in two stages");
    static_assert(CSN % 2 == 0 && CSM % 2 == 0, "16-byte aligned rows");
    double *Cs = smem;
    const bool nf = g.c_nfast != 0;
    auto cs = [&](int ml, int nl) -> double & { return nf ? Cs[ml * CSN + nl] : Cs[nl * CSM + ml]; };
    // the tile's output offsets, staged once (-1: outside C)
    int *ocm = reinterpret_cast<int *>(smem + CS_ELEMS);
    int *ocn = ocm + BM;
    if (tid < BM) ocm[tid] = m0 + tid < g.M ? __ldg(g.offC_m + m0 + tid) : -1;
    else if (tid < BM + BN) ocn[tid - BM] = n0 + tid - BM < g.N ? __ldg(g.offC_n + n0 + tid - BM) : -1;
    if (nf) {
#pragma unroll
        for (int mi = 0; mi < 2; ++mi)
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int ni = 0; ni < 4; ++ni)
                    *reinterpret_cast<double2 *>(&Cs[(wm + mi * 16 + gid + 8 * h) * CSN + wn + ni * 8 + 2 * tig]) =
                        make_double2(alpha * acc[mi][ni][2 * h], alpha * acc[mi][ni][2 * h + 1]);
    } else {
#pragma unroll
        for (int mi = 0; mi < 2; ++mi)
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int ni = 0; ni < 4; ++ni)
#pragma unroll
                    for (int j = 0; j < 2; ++j)
                        Cs[(wn + ni * 8 + 2 * tig + j) * CSM + wm + mi * 16 + gid + 8 * h] = alpha * acc[mi][ni][2 * h + j];
    }
    __syncthreads();
    // split-K slices and beta = 1 updates add into C with fire-and-forget reductions
    // (one add per element and slice: the same rounding as a read-add-write, with no
    // dependent read in the epilogue)
    const bool atomic = split || g.beta;
    if (g.vec_c && !atomic) {
        // output pairs along the fast mode are contiguous and 16-byte aligned
        const int fast = 2 * (tid & 31), slow0 = tid >> 5;
#pragma unroll 4
        for (int p0 = 0; p0 < 16; p0 += 4) {
            double2 *cp[4];
            double2 cv[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                int slow = slow0 + 4 * (p0 + u);
                int ml = g.c_nfast ? slow : fast;
                int nl = g.c_nfast ? fast : slow;
                const int om = ocm[ml], on = ocn[nl];
                cp[u] = (om >= 0 && on >= 0) ? reinterpret_cast<double2 *>(g.C + (long long)om + on) : nullptr;
                // the pair is contiguous in the tile's row as well
                cv[u] = *reinterpret_cast<const double2 *>(&cs(ml, nl));
            }
            double2 old[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) old[u] = (cp[u] && g.beta) ? *cp[u] : make_double2(0.0, 0.0);
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (cp[u]) *cp[u] = make_double2(old[u].x + cv[u].x, old[u].y + cv[u].y);
        }
        return;
    }
    const int fast = tid & 63, slow0 = tid >> 6;
    // all of this thread's output reads are issued before any write (memory-level
    // parallelism for the beta = 1 updates of large intermediates)
#pragma unroll 8
    for (int p0 = 0; p0 < 32; p0 += 8) {
        double *cp[8];
        double cv[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            int slow = slow0 + 2 * (p0 + u);
            int ml = g.c_nfast ? slow : fast;
            int nl = g.c_nfast ? fast : slow;
            const int om = ocm[ml], on = ocn[nl];
            cp[u] = (om >= 0 && on >= 0) ? g.C + (long long)om + on : nullptr;
            cv[u] = cs(ml, nl);
        }
        if (atomic) {
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if (cp[u]) atomicAdd(cp[u], cv[u]);
        } else {
            double old[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) old[u] = (cp[u] && g.beta) ? *cp[u] : 0.0;
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if (cp[u]) *cp[u] = old[u] + cv[u];
        }
    }
}

template <bool AK, bool BKM, bool GROUPED, int NST>
__global__ void __launch_bounds__(128) gett_f64_kernel(GettArgs g) {
    gett_f64_tile<AK, BKM, GROUPED, NST>(g, blockIdx.x, blockIdx.y, blockIdx.z, gridDim.z > 1);
}

// Many GETTs of the same operand orientation in one launch (one per context of a batch of
// independent solves): block b runs tile b - tstart[i] of GETT i, where tstart[i] <= b < tstart[i + 1]
// (64 x 64 tiles, the whole K range, no split-K).  GETT i is skipped when active[owner[i]] is zero.
template <bool AK, bool BKM, int NST>
__global__ void __launch_bounds__(128) gett_f64_batched_kernel(const GettArgs *__restrict__ args,
                                                               const int *__restrict__ tstart, int n,
                                                               const int *__restrict__ owner,
                                                               const int *__restrict__ active) {
    const int b = blockIdx.x;
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (__ldg(tstart + mid) <= b) lo = mid;
        else hi = mid - 1;
    }
    if (!__ldg(active + __ldg(owner + lo))) return;
    const GettArgs &g = args[lo];
    const int t = b - __ldg(tstart + lo);
    const int tm = (g.M + BM - 1) / BM, tn = (g.N + BN - 1) / BN;
    if (g.nseg > 0) {
        gett_f64_tile<AK, BKM, true, NST>(g, t % tm, (t / tm) % tn, 0, false);
    } else {
        // split-K slices (kchunk of the context's own launch) add into C, zeroed beforehand
        const int nz = (g.K + g.kchunk - 1) / g.kchunk;
        gett_f64_tile<AK, BKM, false, NST>(g, t % tm, (t / tm) % tn, t / (tm * tn), nz > 1);
    }
}

// the output views of many GETTs set to zero (before their split-K slices add into them)
__global__ void zero_views_batched_kernel(const GettArgs *__restrict__ args, int n, const int *__restrict__ owner,
                                          const int *__restrict__ active) {
    for (int i = blockIdx.y; i < n; i += gridDim.y) {
        if (!__ldg(active + __ldg(owner + i))) continue;
        const GettArgs &g = args[i];
        const long long total = (long long)g.M * g.N;
        for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
             e += (long long)gridDim.x * blockDim.x) {
            const int m = (int)(e / g.N), nn = (int)(e % g.N);
            g.C[(long long)__ldg(g.offC_m + m) + __ldg(g.offC_n + nn)] = 0.0;
        }
    }
}

void launch_zero_views_batched(const GettArgs *args, int n, const int *owner, const int *active, cudaStream_t s) {
    if (n <= 0) return;
    dim3 grid(64, (unsigned)std::min(n, 65535));
    zero_views_batched_kernel<<<grid, 256, 0, s>>>(args, n, owner, active);
}

void launch_gett_f64_batched(const GettArgs *args, const int *tstart, int n, int tiles, const int *owner,
                             const int *active, int a_kmajor, int b_kmajor, cudaStream_t s) {
    if (n <= 0 || tiles <= 0) return;
    constexpr size_t sm = sizeof(double) * 2 * 2 * TILE;
    if (a_kmajor && b_kmajor)
        gett_f64_batched_kernel<true, true, 2><<<tiles, 128, sm, s>>>(args, tstart, n, owner, active);
    else if (a_kmajor)
        gett_f64_batched_kernel<true, false, 2><<<tiles, 128, sm, s>>>(args, tstart, n, owner, active);
    else if (b_kmajor)
        gett_f64_batched_kernel<false, true, 2><<<tiles, 128, sm, s>>>(args, tstart, n, owner, active);
    else
        gett_f64_batched_kernel<false, false, 2><<<tiles, 128, sm, s>>>(args, tstart, n, owner, active);
}

// dynamic shared memory of gett_f64_kernel: the operand stages
template <bool G, int NST>
constexpr size_t gett_smem() { return sizeof(double) * 2 * NST * TILE; }

template <bool G, int NST>
void launch_gett_v(const GettArgs &a, int a_kmajor, int b_kmajor, dim3 grid, cudaStream_t s) {
    constexpr size_t sm = gett_smem<G, NST>();
    if (a_kmajor && b_kmajor)
        gett_f64_kernel<true, true, G, NST><<<grid, 128, sm, s>>>(a);
    else if (a_kmajor)
        gett_f64_kernel<true, false, G, NST><<<grid, 128, sm, s>>>(a);
    else if (b_kmajor)
        gett_f64_kernel<false, true, G, NST><<<grid, 128, sm, s>>>(a);
    else
        gett_f64_kernel<false, false, G, NST><<<grid, 128, sm, s>>>(a);
}

template <bool G, int NST>
cudaError_t gett_attr() {
    constexpr int sm = (int)gett_smem<G, NST>();
    constexpr auto at = cudaFuncAttributeMaxDynamicSharedMemorySize;
    cudaError_t e = cudaFuncSetAttribute(gett_f64_kernel<true, true, G, NST>, at, sm);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(gett_f64_kernel<true, false, G, NST>, at, sm);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(gett_f64_kernel<false, true, G, NST>, at, sm);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(gett_f64_kernel<false, false, G, NST>, at, sm);
    return e;
}

// ---------------------------------------------------------------------------
// Skinny GETT: one side of C has at most 32 entries.  The 64 x 64 tiles above
// would pad such a contraction to up to 64x its DMMA work; here a BMS x 128
// tile (BMS = 16 or 32) streams the long operand through a 4-stage cp.async
// ring, so these mostly memory-bound launches run near the HBM roof.  When N
// is the short side the kernel runs the transposed problem C^T = B A^T
// (operands, tables and the output's fast mode exchanged): its rows are always
// the short side.  All offset tables a tile uses (its rows, columns, output
// rows and columns, and the K slice's k offsets) are staged in shared memory
// once, so no copy or store waits on a dependent global read.
// ---------------------------------------------------------------------------
constexpr int SBN = 128, SBK = 16, SST = 4;
constexpr int SKS = SBK + 4;   // [row][k] stride of k-major tiles
constexpr int SBNS = SBN + 4;  // [k][n] stride of the long operand's n-major tile
constexpr int SKT = 512;       // k offsets staged per K slice (longer slices read them from global memory)
template <int BMS>
struct Skinny {
    static constexpr int AMS = BMS + 4;  // [k][m] stride of the short operand's m-major tile
    static constexpr int ATILE = SBK * AMS > BMS * SKS ? SBK * AMS : BMS * SKS;
    static constexpr int BTILE = SBK * SBNS > SBN * SKS ? SBK * SBNS : SBN * SKS;
    static constexpr int STAGE = ATILE + BTILE;
    // dynamic shared memory: offset tables (ints), then the stage ring; a launch
    // sizes the ring to the K slabs it has (small-K launches keep several CTAs
    // per SM), but never below the staged C tile
    static constexpr int OFFB = (2 * (BMS + SBN) + 2 * SKT) * 4;
    static constexpr int CS_STAGES = (BMS * (SBN + 1) + STAGE - 1) / STAGE;
    static constexpr int SMEM = OFFB + SST * STAGE * 8;
    static int smem(int stages) { return OFFB + stages * STAGE * 8; }
    static_assert(CS_STAGES <= SST, "C tile must fit in the stage ring");
    static_assert(OFFB % 16 == 0 && ATILE % 2 == 0 && STAGE % 2 == 0, "16-byte aligned tiles");
    template <bool KM>
    static __device__ __forceinline__ int ai(int k, int m) { return KM ? m * SKS + k : k * AMS + m; }
    template <bool KM>
    static __device__ __forceinline__ int bi(int k, int n) { return KM ? n * SKS + k : k * SBNS + n; }
};

// One contraction term in the launched orientation (A short, B long).
struct SkTerm {
    const double *A, *B;
    const int *am, *ak, *bn, *bk;
};

// Offset tables of the current tile and K slice in shared memory.  ka / kb are
// indexed by k - kb0 (the staged slice, kb0 = its first k) or point at the
// global tables (kb0 = 0) when the slice is longer than SKT.
struct SkTabs {
    int *a, *b, *cm, *cn, *ska, *skb;
    const int *ka, *kb;
    int kb0;
};

// Loads the k-slab [k0, k0 + SBK) of both operands into one ring stage.
// Out-of-range elements are zero-filled.
template <int BMS, bool AK, bool BKM>
__device__ __forceinline__ void skinny_load(double *st, const SkTerm &p, const SkTabs &t, int M, int N, int m0, int n0,
                                            int k0, int kend, int tid, bool vb) {
    using T = Skinny<BMS>;
    double *As = st, *Bs = st + T::ATILE;
    if (AK) {
        const int kk = tid & 15, k = k0 + kk;
        const bool kin = k < kend;
        const int ok = kin ? t.ka[k - t.kb0] : 0;
#pragma unroll
        for (int q = 0; q < BMS / 8; ++q) {
            const int m = (tid >> 4) + 8 * q;
            const bool in = kin && m0 + m < M;
            cp_async8(&As[T::template ai<true>(kk, m)], in ? p.A + (long long)t.a[m] + ok : p.A, in);
        }
    } else {
        constexpr int R = 128 / BMS;  // k rows per pass
        const int m = tid % BMS;
        const bool min_ = m0 + m < M;
        const long long om = t.a[m];
#pragma unroll
        for (int q = 0; q < SBK / R; ++q) {
            const int kk = tid / BMS + R * q, k = k0 + kk;
            const bool in = min_ && k < kend;
            cp_async8(&As[T::template ai<false>(kk, m)], in ? p.A + om + t.ka[k - t.kb0] : p.A, in);
        }
    }
    if (BKM && vb) {
        // k pairs are contiguous and 16-byte aligned
        const int kk = 2 * (tid & 7), k = k0 + kk;
        const bool kin = k < kend;
        const int ok = kin ? t.kb[k - t.kb0] : 0;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int n = (tid >> 3) + 16 * q;
            const bool in = kin && n0 + n < N;
            cp_async16(&Bs[T::template bi<true>(kk, n)], in ? p.B + (long long)t.b[n] + ok : p.B, in);
        }
    } else if (BKM) {
        const int kk = tid & 15, k = k0 + kk;
        const bool kin = k < kend;
        const int ok = kin ? t.kb[k - t.kb0] : 0;
#pragma unroll
        for (int q = 0; q < 16; ++q) {
            const int n = (tid >> 4) + 8 * q;
            const bool in = kin && n0 + n < N;
            cp_async8(&Bs[T::template bi<true>(kk, n)], in ? p.B + (long long)t.b[n] + ok : p.B, in);
        }
    } else if (vb) {
        // n pairs are contiguous and 16-byte aligned
        const int n = 2 * (tid & 63);
        const bool nin = n0 + n < N;
        const long long on = t.b[n];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int kk = (tid >> 6) + 2 * q, k = k0 + kk;
            const bool in = nin && k < kend;
            cp_async16(&Bs[T::template bi<false>(kk, n)], in ? p.B + on + t.kb[k - t.kb0] : p.B, in);
        }
    } else {
        const int n = tid;
        const bool nin = n0 + n < N;
        const long long on = t.b[n];
#pragma unroll
        for (int q = 0; q < 16; ++q) {
            const int k = k0 + q;
            const bool in = nin && k < kend;
            cp_async8(&Bs[T::template bi<false>(q, n)], in ? p.B + on + t.kb[k - t.kb0] : p.B, in);
        }
    }
}

// K loop of one term over [kbeg, kend): ST-stage ring, one barrier per slab
// (the slab loaded at step t overwrites the stage computed at step t - 1).
template <int BMS, bool AK, bool BKM, int ST>
__device__ __forceinline__ void skinny_mainloop(double (&acc)[BMS / 16][4][4], double *sm, SkTabs &t,
                                                const SkTerm &p, int M, int N, int m0, int n0, int kbeg, int kend,
                                                int tid, int wn, int gid, int tig, bool vb) {
    using T = Skinny<BMS>;
    __syncthreads();  // earlier users of the tables and of the ring are done
    for (int i = tid; i < BMS; i += 128) t.a[i] = m0 + i < M ? __ldg(p.am + m0 + i) : 0;
    for (int i = tid; i < SBN; i += 128) t.b[i] = n0 + i < N ? __ldg(p.bn + n0 + i) : 0;
    const int klen = kend - kbeg;
    if (klen <= SKT) {
        for (int i = tid; i < klen; i += 128) {
            t.ska[i] = __ldg(p.ak + kbeg + i);
            t.skb[i] = __ldg(p.bk + kbeg + i);
        }
        t.ka = t.ska;
        t.kb = t.skb;
        t.kb0 = kbeg;
    } else {
        t.ka = p.ak;
        t.kb = p.bk;
        t.kb0 = 0;
    }
    __syncthreads();
    const int nt = kend > kbeg ? (kend - kbeg + SBK - 1) / SBK : 0;
#pragma unroll
    for (int s = 0; s < ST - 1; ++s) {
        if (s < nt) skinny_load<BMS, AK, BKM>(sm + s * T::STAGE, p, t, M, N, m0, n0, kbeg + s * SBK, kend, tid, vb);
        cp_async_commit();
    }
    for (int it = 0; it < nt; ++it) {
        cp_async_wait<ST - 2>();
        __syncthreads();
        const int tn = it + ST - 1;
        if (tn < nt)
            skinny_load<BMS, AK, BKM>(sm + (tn % ST) * T::STAGE, p, t, M, N, m0, n0, kbeg + tn * SBK, kend, tid, vb);
        cp_async_commit();
        const double *As = sm + (it % ST) * T::STAGE, *Bs = As + T::ATILE;
        const int nk = kend - (kbeg + it * SBK);   // past it the slab holds the zero fill
#pragma unroll
        for (int kk = 0; kk < SBK; kk += 8) {
            if (kk >= nk) break;
            double a[BMS / 16][4], b[4][2];
#pragma unroll
            for (int mi = 0; mi < BMS / 16; ++mi)
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    a[mi][q] = As[T::template ai<AK>(kk + tig + 4 * (q >> 1), mi * 16 + gid + 8 * (q & 1))];
#pragma unroll
            for (int ni = 0; ni < 4; ++ni)
#pragma unroll
                for (int q = 0; q < 2; ++q) b[ni][q] = Bs[T::template bi<BKM>(kk + tig + 4 * q, wn + ni * 8 + gid)];
#pragma unroll
            for (int mi = 0; mi < BMS / 16; ++mi)
#pragma unroll
                for (int ni = 0; ni < 4; ++ni) dmma_16x8x8(acc[mi][ni], a[mi], b[ni]);
        }
    }
    cp_async_wait<0>();
    __syncthreads();
}

template <int BMS, bool AK, bool BKM, bool GROUPED, int ST>
__global__ void __launch_bounds__(128) gett_f64_skinny_kernel(GettArgs g) {
    using T = Skinny<BMS>;
    extern __shared__ __align__(16) unsigned char smraw[];
    SkTabs t;
    t.a = reinterpret_cast<int *>(smraw);
    t.b = t.a + BMS;
    t.cm = t.b + SBN;
    t.cn = t.cm + BMS;
    t.ska = t.cn + SBN;
    t.skb = t.ska + SKT;
    double *sm = reinterpret_cast<double *>(smraw + T::OFFB);
    const bool sw = g.N < g.M;  // transposed launch: N is the short side
    const int M = sw ? g.N : g.M, N = sw ? g.M : g.N;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int gid = lane >> 2, tig = lane & 3, wn = warp * 32;
    const int n0 = blockIdx.x * SBN, m0 = blockIdx.y * BMS;
    const bool vb = (sw ? g.vec_a : g.vec_b) != 0;
    // output offsets in the launched orientation (read after the mainloop's barriers)
    {
        const int *offm = sw ? g.offC_n : g.offC_m, *offn = sw ? g.offC_m : g.offC_n;
        for (int i = tid; i < BMS; i += 128) t.cm[i] = m0 + i < M ? __ldg(offm + m0 + i) : 0;
        for (int i = tid; i < SBN; i += 128) t.cn[i] = n0 + i < N ? __ldg(offn + n0 + i) : 0;
    }

    double acc[BMS / 16][4][4];
#pragma unroll
    for (int i = 0; i < BMS / 16; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int q = 0; q < 4; ++q) acc[i][j][q] = 0.0;

    double alpha = g.alpha;
    if (GROUPED) {
        for (int sgi = 0; sgi < g.nseg; ++sgi) {
            const GettSeg sg = g.segs[sgi];
            if (sgi > 0) {
                const double r = g.segs[sgi - 1].alpha / sg.alpha;
#pragma unroll
                for (int i = 0; i < BMS / 16; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j)
#pragma unroll
                        for (int q = 0; q < 4; ++q) acc[i][j][q] *= r;
            }
            const SkTerm p = sw ? SkTerm{sg.B, sg.A, sg.offB_n, sg.offB_k, sg.offA_m, sg.offA_k}
                                : SkTerm{sg.A, sg.B, sg.offA_m, sg.offA_k, sg.offB_n, sg.offB_k};
            skinny_mainloop<BMS, AK, BKM, ST>(acc, sm, t, p, M, N, m0, n0, 0, sg.K, tid, wn, gid, tig, vb);
            alpha = sg.alpha;
        }
    } else {
        const SkTerm p = sw ? SkTerm{g.B, g.A, g.offB_n, g.offB_k, g.offA_m, g.offA_k}
                            : SkTerm{g.A, g.B, g.offA_m, g.offA_k, g.offB_n, g.offB_k};
        const int kbeg = blockIdx.z * g.kchunk;
        const int kend = min(g.K, kbeg + g.kchunk);
        skinny_mainloop<BMS, AK, BKM, ST>(acc, sm, t, p, M, N, m0, n0, kbeg, kend, tid, wn, gid, tig, vb);
    }

    // epilogue: stage the tile, then write along the output's contiguous mode
    double (*Cs)[SBN + 1] = reinterpret_cast<double (*)[SBN + 1]>(sm);
#pragma unroll
    for (int mi = 0; mi < BMS / 16; ++mi)
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int ni = 0; ni < 4; ++ni)
#pragma unroll
                for (int j = 0; j < 2; ++j)
                    Cs[mi * 16 + gid + 8 * h][wn + ni * 8 + 2 * tig + j] = alpha * acc[mi][ni][2 * h + j];
    __syncthreads();
    // split-K slices and beta = 1 updates add into C with fire-and-forget reductions
    // (one add per element and slice: the same rounding as a read-add-write, with no
    // dependent read in the epilogue)
    const bool atomic = gridDim.z > 1 || g.beta;
    const bool nfast = sw ? !g.c_nfast : g.c_nfast;
    constexpr int R = 128 / BMS;
    // nfast: a thread owns column n = tid and walks the BMS rows; else BMS
    // consecutive threads cover the rows of one column, R columns per pass
    const int fl = nfast ? tid : tid % BMS;
    const int sl0 = nfast ? 0 : tid / BMS;
    const int sstep = nfast ? 1 : R;
    const int nsl = nfast ? BMS : SBN / R;
    const bool fin = nfast ? n0 + fl < N : m0 + fl < M;
    const long long ofix = nfast ? t.cn[fl] : t.cm[fl];
    for (int s0 = 0; s0 < nsl; s0 += 8) {
        double *cp[8];
        double cv[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int sl = sl0 + sstep * (s0 + u);
            const int ml = nfast ? sl : fl, nl = nfast ? fl : sl;
            const bool in = fin && m0 + ml < M && n0 + nl < N;
            cp[u] = in ? g.C + ofix + (nfast ? t.cm[ml] : t.cn[nl]) : nullptr;
            cv[u] = Cs[ml][nl];
        }
        if (atomic) {
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if (cp[u]) atomicAdd(cp[u], cv[u]);
        } else {
            double old[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) old[u] = (cp[u] && g.beta) ? *cp[u] : 0.0;
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if (cp[u]) *cp[u] = old[u] + cv[u];
        }
    }
}

template <int BMS, bool G, int ST>
void launch_skinny_v(const GettArgs &a, int ak, int bk, dim3 grid, cudaStream_t s) {
    // ring stages: every K slab of a slice when they fit below ST (all loaded
    // in the prologue), else the full ring; grouped launches take the full ring
    int stages = ST;
    if (!G) {
        const int nt = (std::min(a.K, a.kchunk) + SBK - 1) / SBK;
        if (nt < ST) stages = std::max(nt, Skinny<BMS>::CS_STAGES);
    }
    stages = std::max(stages, Skinny<BMS>::CS_STAGES);
    const int sm = Skinny<BMS>::smem(stages);
    if (ak && bk)
        gett_f64_skinny_kernel<BMS, true, true, G, ST><<<grid, 128, sm, s>>>(a);
    else if (ak)
        gett_f64_skinny_kernel<BMS, true, false, G, ST><<<grid, 128, sm, s>>>(a);
    else if (bk)
        gett_f64_skinny_kernel<BMS, false, true, G, ST><<<grid, 128, sm, s>>>(a);
    else
        gett_f64_skinny_kernel<BMS, false, false, G, ST><<<grid, 128, sm, s>>>(a);
}

template <int BMS, bool G, int ST>
cudaError_t skinny_attr() {
    const int sm = Skinny<BMS>::smem(std::max(ST, Skinny<BMS>::CS_STAGES));
    constexpr auto at = cudaFuncAttributeMaxDynamicSharedMemorySize;
    cudaError_t e = cudaFuncSetAttribute(gett_f64_skinny_kernel<BMS, true, true, G, ST>, at, sm);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(gett_f64_skinny_kernel<BMS, true, false, G, ST>, at, sm);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(gett_f64_skinny_kernel<BMS, false, true, G, ST>, at, sm);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(gett_f64_skinny_kernel<BMS, false, false, G, ST>, at, sm);
    return e;
}

// The shared-memory limits set by cudaFuncSetAttribute belong to the current
// device, so they are set once per device (the first GETT launch or context
// creation on each device), not once per process.
constexpr int kPrepDevices = 64;

cudaError_t gett_f64_prepare() {
    static std::once_flag once[kPrepDevices];
    static cudaError_t err[kPrepDevices];
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= kPrepDevices) return cudaErrorInvalidDevice;
    std::call_once(once[dev], [dev] {
        cudaError_t r = skinny_attr<16, false, SST>();
        if (r == cudaSuccess) r = skinny_attr<16, true, SST>();
        if (r == cudaSuccess) r = skinny_attr<32, false, SST>();
        if (r == cudaSuccess) r = skinny_attr<32, true, SST>();
        if (r == cudaSuccess) r = skinny_attr<16, false, 2>();
        if (r == cudaSuccess) r = skinny_attr<16, true, 2>();
        if (r == cudaSuccess) r = skinny_attr<32, false, 2>();
        if (r == cudaSuccess) r = skinny_attr<32, true, 2>();
        if (r == cudaSuccess) r = gett_attr<false, 3>();
        if (r == cudaSuccess) r = gett_attr<true, 3>();
        err[dev] = r;
    });
    return err[dev];
}

// ---------------------------------------------------------------------------
// Small-K GETT on the FP64 FMA pipe: for K of a few dozen the contraction is
// bound by writing C (16-268 MB intermediates at 40 orbitals), not by the
// products, and B200's FP64 FMA rate equals its DMMA rate.  One thread owns one
// index f of the output's contiguous side ("F side": n when c_nfast, else m)
// and BS indices of the other side, so every store of a warp covers 32
// consecutive outputs; the F operand streams straight into registers, the S
// operand is staged per K chunk in shared memory (scaled by alpha) and read by
// broadcast.  Grouped launches loop over their segments.
// ---------------------------------------------------------------------------
constexpr int QT = 256, QKC = 16;

template <int BS, bool GROUPED>
__global__ void __launch_bounds__(QT, 2) gett_f64_smallk_kernel(GettArgs g, int fside, int skm) {
    __shared__ __align__(16) double Ss[QKC][BS];
    __shared__ int soffc[BS];
    const int tid = threadIdx.x;
    const int Fsz = fside ? g.N : g.M, Ssz = fside ? g.M : g.N;
    const int f = blockIdx.x * QT + tid;
    const int s0 = blockIdx.y * BS;
    const bool fin = f < Fsz;
    const int *offcs = fside ? g.offC_m : g.offC_n;
    if (tid < BS) soffc[tid] = s0 + tid < Ssz ? __ldg(offcs + s0 + tid) : 0;
    double acc[BS];
#pragma unroll
    for (int q = 0; q < BS; ++q) acc[q] = 0.0;
    const int nseg = GROUPED ? g.nseg : 1;
    for (int sg = 0; sg < nseg; ++sg) {
        const double *A = g.A, *B = g.B;
        const int *oam = g.offA_m, *oak = g.offA_k, *obn = g.offB_n, *obk = g.offB_k;
        int K = g.K;
        double alpha = g.alpha;
        if (GROUPED) {
            const GettSeg &q = g.segs[sg];
            A = q.A;
            B = q.B;
            oam = q.offA_m;
            oak = q.offA_k;
            obn = q.offB_n;
            obk = q.offB_k;
            K = q.K;
            alpha = q.alpha;
        }
        const double *F = fside ? B : A, *S = fside ? A : B;
        const int *ofi = fside ? obn : oam, *ofk = fside ? obk : oak;
        const int *osi = fside ? oam : obn, *osk = fside ? oak : obk;
        const long long fb = fin ? (long long)__ldg(ofi + f) : 0;
        for (int k0 = 0; k0 < K; k0 += QKC) {
            const int kc = min(QKC, K - k0);
            double fv[QKC];
#pragma unroll
            for (int k = 0; k < QKC; ++k) fv[k] = (fin && k < kc) ? __ldg(F + fb + __ldg(ofk + k0 + k)) : 0.0;
            __syncthreads();  // the previous chunk's reads of Ss (and soffc) are done
            for (int i = tid; i < QKC * BS; i += QT) {
                const int k = skm ? i % QKC : i / BS;
                const int q = skm ? i / QKC : i % BS;
                double v = 0.0;
                if (k < kc && s0 + q < Ssz) v = alpha * __ldg(S + (long long)__ldg(osi + s0 + q) + __ldg(osk + k0 + k));
                Ss[k][q] = v;
            }
            __syncthreads();
#pragma unroll
            for (int k = 0; k < QKC; ++k) {
                if (k < kc) {
                    const double a = fv[k];
#pragma unroll
                    for (int q = 0; q < BS; q += 2) {
                        const double2 b = *reinterpret_cast<const double2 *>(&Ss[k][q]);
                        acc[q] += a * b.x;
                        acc[q + 1] += a * b.y;
                    }
                }
            }
        }
    }
    if (!fin) return;
    double *cf = g.C + __ldg((fside ? g.offC_n : g.offC_m) + f);
    // beta = 1 updates add with reductions (concurrent writers of one intermediate)
#pragma unroll
    for (int q = 0; q < BS; ++q) {
        if (s0 + q < Ssz) {
            if (g.beta)
                atomicAdd(cf + soffc[q], acc[q]);
            else
                cf[soffc[q]] = acc[q];
        }
    }
}

template <int BS>
void launch_smallk_bs(const GettArgs &a, int fside, int skm, dim3 grid, cudaStream_t s) {
    if (a.segs)
        gett_f64_smallk_kernel<BS, true><<<grid, QT, 0, s>>>(a, fside, skm);
    else
        gett_f64_smallk_kernel<BS, false><<<grid, QT, 0, s>>>(a, fside, skm);
}

// false when the shape does not fit the launch (the caller takes the DMMA path)
bool launch_smallk(const GettArgs &a, int a_kmajor, int b_kmajor, cudaStream_t s) {
    const int fside = a.c_nfast ? 1 : 0;
    const long long Fsz = fside ? a.N : a.M, Ssz = fside ? a.M : a.N;
    const int bs = Ssz <= 8 ? 8 : Ssz <= 16 ? 16 : 32;
    const long long gy = (Ssz + bs - 1) / bs, gx = (Fsz + QT - 1) / QT;
    if (gy > 65535 || gx > 0x7fffffffLL) return false;
    const int skm = fside ? a_kmajor : b_kmajor;
    dim3 grid((unsigned)gx, (unsigned)gy, 1);
    if (bs == 8)
        launch_smallk_bs<8>(a, fside, skm, grid, s);
    else if (bs == 16)
        launch_smallk_bs<16>(a, fside, skm, grid, s);
    else
        launch_smallk_bs<32>(a, fside, skm, grid, s);
    return true;
}

// ---------------------------------------------------------------------------
// Small-K GETT with register-direct operands: each warp owns a 32 x 32 block of a 64 x 64 tile and loads
// its m16n8k8 fragments straight from global memory through the offset tables (the operands of small-K
// contractions are small and stay in L2), so there is no shared-memory staging and no barrier; the
// accumulators are written from registers (8 consecutive outputs per lane group, 16-byte pairs where the
// output pairs up along n).  Whole K per launch, every warp independent; grouped launches loop over their
// segments, rescaling the running sum by alpha_{s-1} / alpha_s.
// ---------------------------------------------------------------------------
template <bool GROUPED>
__global__ void __launch_bounds__(128) gett_f64_direct_kernel(GettArgs g) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int gid = lane >> 2, tig = lane & 3;
    const int m0 = blockIdx.x * BM + (warp >> 1) * 32, n0 = blockIdx.y * BN + (warp & 1) * 32;
    if (m0 >= g.M || n0 >= g.N) return;   // the warp's block lies outside C (warp-uniform)
    double acc[2][4][4];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int q = 0; q < 4; ++q) acc[i][j][q] = 0.0;
    double alpha = g.alpha;
    const int nseg = GROUPED ? g.nseg : 1;
    for (int sgi = 0; sgi < nseg; ++sgi) {
        const double *A = g.A, *B = g.B;
        const int *oam = g.offA_m, *oak = g.offA_k, *obn = g.offB_n, *obk = g.offB_k;
        int K = g.K;
        double sa = g.alpha;
        if (GROUPED) {
            const GettSeg sg = g.segs[sgi];
            A = sg.A;
            B = sg.B;
            oam = sg.offA_m;
            oak = sg.offA_k;
            obn = sg.offB_n;
            obk = sg.offB_k;
            K = sg.K;
            sa = sg.alpha;
            if (sgi > 0 && sa != alpha) {
                const double r = alpha / sa;
#pragma unroll
                for (int i = 0; i < 2; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j)
#pragma unroll
                        for (int q = 0; q < 4; ++q) acc[i][j][q] *= r;
            }
            alpha = sa;
        }
        // A rows m0 + mi*16 + gid + 8h and B columns n0 + ni*8 + gid of this thread's fragments
        int ra[2][2], rb[4];
        bool ia[2][2], ib[4];
#pragma unroll
        for (int mi = 0; mi < 2; ++mi)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int m = m0 + mi * 16 + gid + 8 * h;
                ia[mi][h] = m < g.M;
                ra[mi][h] = ia[mi][h] ? __ldg(oam + m) : 0;
            }
#pragma unroll
        for (int ni = 0; ni < 4; ++ni) {
            const int n = n0 + ni * 8 + gid;
            ib[ni] = n < g.N;
            rb[ni] = ib[ni] ? __ldg(obn + n) : 0;
        }
        for (int k0 = 0; k0 < K; k0 += 8) {
            int ka[2], kb[2];
            bool ik[2];
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const int kk = k0 + tig + 4 * q;
                ik[q] = kk < K;
                ka[q] = ik[q] ? __ldg(oak + kk) : 0;
                kb[q] = ik[q] ? __ldg(obk + kk) : 0;
            }
            double a[2][4], b[4][2];
#pragma unroll
            for (int mi = 0; mi < 2; ++mi)
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int h = q & 1, kq = q >> 1;
                    a[mi][q] = (ia[mi][h] && ik[kq]) ? __ldg(A + (long long)ra[mi][h] + ka[kq]) : 0.0;
                }
#pragma unroll
            for (int ni = 0; ni < 4; ++ni)
#pragma unroll
                for (int q = 0; q < 2; ++q) b[ni][q] = (ib[ni] && ik[q]) ? __ldg(B + (long long)rb[ni] + kb[q]) : 0.0;
#pragma unroll
            for (int mi = 0; mi < 2; ++mi)
#pragma unroll
                for (int ni = 0; ni < 4; ++ni) dmma_16x8x8(acc[mi][ni], a[mi], b[ni]);
        }
    }
    // outputs (m0 + mi*16 + gid + 8h, n0 + ni*8 + 2 tig + j) = acc[mi][ni][2h + j]
    int om[2][2], on[4][2];
#pragma unroll
    for (int mi = 0; mi < 2; ++mi)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int m = m0 + mi * 16 + gid + 8 * h;
            om[mi][h] = m < g.M ? __ldg(g.offC_m + m) : -1;
        }
#pragma unroll
    for (int ni = 0; ni < 4; ++ni)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int n = n0 + ni * 8 + 2 * tig + j;
            on[ni][j] = n < g.N ? __ldg(g.offC_n + n) : -1;
        }
    const bool pairs = !g.beta && g.vec_c && g.c_nfast;
#pragma unroll
    for (int mi = 0; mi < 2; ++mi)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            if (om[mi][h] < 0) continue;
            double *crow = g.C + om[mi][h];
#pragma unroll
            for (int ni = 0; ni < 4; ++ni) {
                const double v0 = alpha * acc[mi][ni][2 * h], v1 = alpha * acc[mi][ni][2 * h + 1];
                if (pairs && on[ni][1] >= 0) {
                    *reinterpret_cast<double2 *>(crow + on[ni][0]) = make_double2(v0, v1);
                } else if (g.beta) {
                    if (on[ni][0] >= 0) atomicAdd(crow + on[ni][0], v0);
                    if (on[ni][1] >= 0) atomicAdd(crow + on[ni][1], v1);
                } else {
                    if (on[ni][0] >= 0) crow[on[ni][0]] = v0;
                    if (on[ni][1] >= 0) crow[on[ni][1]] = v1;
                }
            }
        }
}

int gett_f64_family(long long M, long long N) {
    if (M <= 32 && M <= N) return 1;
    if (N <= 32 && N < M) return 2;
    return 0;
}

int gett_f64_kchunk(long long M, long long N, long long K) {
    if (M <= 0 || N <= 0 || K <= 0) return 16;  // nothing is launched
    long long splits = 1;
    if (gett_f64_family(M, N)) {
        // stream the long operand with about two resident waves of CTAs
        long long shrt = std::min(M, N), lng = std::max(M, N);
        long long tiles = ((lng + SBN - 1) / SBN) * ((shrt + (shrt <= 16 ? 15 : 31)) / (shrt <= 16 ? 16 : 32));
        if (tiles < 592 && K >= 64) splits = std::min<long long>(std::min<long long>((592 + tiles - 1) / tiles, (K + 63) / 64), 256);
    } else {
        long long tiles = ((M + BM - 1) / BM) * ((N + BN - 1) / BN);
        if (tiles < 296 && K >= 128) splits = std::min<long long>(std::min<long long>((296 + tiles - 1) / tiles, (K + 31) / 32), 128);
    }
    if (splits < 1) splits = 1;
    long long chunk = (K + splits - 1) / splits;
    chunk = (chunk + 15) / 16 * 16;
    return (int)std::max<long long>(chunk, 16);
}

void launch_gett_f64(const GettArgs &a, int a_kmajor, int b_kmajor, cudaStream_t s) {
    if (a.tile == 3 && launch_smallk(a, a_kmajor, b_kmajor, s)) return;
    if (a.tile == 6) {
        // register-direct small-K kernel: the whole K range in one pass (no split-K slices)
        dim3 grid((a.M + BM - 1) / BM, (a.N + BN - 1) / BN, 1);
        if (a.segs)
            gett_f64_direct_kernel<true><<<grid, 128, 0, s>>>(a);
        else
            gett_f64_direct_kernel<false><<<grid, 128, 0, s>>>(a);
        return;
    }
    const int zsplit = a.segs ? 1 : std::max(1, (a.K + a.kchunk - 1) / a.kchunk);
    int fam = gett_f64_family(a.M, a.N);
    if (a.tile == 1 || a.tile == 4) fam = 0;
    else if ((a.tile == 2 || a.tile == 5) && std::min(a.M, a.N) <= 32) fam = a.M <= a.N ? 1 : 2;
    if (fam) {
        gett_f64_prepare();
        const int shrt = std::min(a.M, a.N), lng = std::max(a.M, a.N);
        const int ak = fam == 2 ? b_kmajor : a_kmajor, bk = fam == 2 ? a_kmajor : b_kmajor;
        const bool two = a.tile == 5;   // 2-stage ring: half the shared memory, more CTAs per SM
        if (shrt <= 16) {
            dim3 grid((lng + SBN - 1) / SBN, (shrt + 15) / 16, zsplit);
            if (two)
                a.segs ? launch_skinny_v<16, true, 2>(a, ak, bk, grid, s) : launch_skinny_v<16, false, 2>(a, ak, bk, grid, s);
            else
                a.segs ? launch_skinny_v<16, true, SST>(a, ak, bk, grid, s)
                       : launch_skinny_v<16, false, SST>(a, ak, bk, grid, s);
        } else {
            dim3 grid((lng + SBN - 1) / SBN, (shrt + 31) / 32, zsplit);
            if (two)
                a.segs ? launch_skinny_v<32, true, 2>(a, ak, bk, grid, s) : launch_skinny_v<32, false, 2>(a, ak, bk, grid, s);
            else
                a.segs ? launch_skinny_v<32, true, SST>(a, ak, bk, grid, s)
                       : launch_skinny_v<32, false, SST>(a, ak, bk, grid, s);
        }
        return;
    }
    dim3 grid((a.M + BM - 1) / BM, (a.N + BN - 1) / BN, zsplit);
    if (a.tile == 4) {
        gett_f64_prepare();
        a.segs ? launch_gett_v<true, 3>(a, a_kmajor, b_kmajor, grid, s)
               : launch_gett_v<false, 3>(a, a_kmajor, b_kmajor, grid, s);
    } else {
        a.segs ? launch_gett_v<true, 2>(a, a_kmajor, b_kmajor, grid, s)
               : launch_gett_v<false, 2>(a, a_kmajor, b_kmajor, grid, s);
    }
}

__global__ void zero_view_kernel(double *C, const int *offm, const int *offn, int M, int N) {
    long long total = (long long)M * N;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        int m = (int)(i / N), n = (int)(i % N);
        C[(long long)offm[m] + offn[n]] = 0.0;
    }
}

void launch_zero_view(double *C, const int *offm, const int *offn, int M, int N, cudaStream_t s) {
    long long total = (long long)M * N;
    int blocks = (int)((total + 255) / 256);
    if (blocks > 148 * 16) blocks = 148 * 16;
    if (blocks < 1) blocks = 1;
    zero_view_kernel<<<blocks, 256, 0, s>>>(C, offm, offn, M, N);
}

// ---------------------------------------------------------------------------
// assemble: residual gather + Jacobi + antisymmetric fill
// ---------------------------------------------------------------------------
// Term descriptor as staged in shared memory: pm has bit j*RK+k set when Z
// axes j < k belong to one antisymmetric group (sorted-with-sign reads);
// tst are the strides per target axis (used when pm == 0), zs per Z axis.
template <int RK>
struct SmTerm {
    const double *p;
    double coef;
    unsigned long long pm;
    int zs[RK];
    int tst[RK];
    unsigned char src[RK];
};

template <int RK>
__device__ __forceinline__ int pick(const int (&v)[RK], int i) {
    int r = 0;
#pragma unroll
    for (int e = 0; e < RK; ++e)
        if (e == i) r = v[e];
    return r;
}

// Each thread gathers EPT canonical elements, EPT * blockDim.x consecutive
// elements per block and step: every term descriptor read from shared memory
// serves EPT elements, and their loads are independent.
constexpr int ASM_EPT = 2;

template <int RK, typename Off>
__device__ __forceinline__ void canonical_element(const AsmArgs &a, Off lin, int (&x)[RK]) {
    int cq[RK];
    Off r = lin;
#pragma unroll
    for (int q = RK - 1; q >= 0; --q) {
        cq[q] = 0;
        if (q < a.nruns) {
            cq[q] = (int)(r % a.run_count[q]);
            r /= a.run_count[q];
        }
    }
#pragma unroll
    for (int q = 0; q < RK; ++q) {
        if (q < a.nruns) {
            const unsigned char *tup = a.combos + a.run_off[q] + cq[q] * a.run_len[q];
#pragma unroll
            for (int d = 0; d < RK; ++d) {
                int l = d - a.run_axis0[q];
                if (l >= 0 && l < a.run_len[q]) x[d] = tup[l];
            }
        }
    }
}

// Term descriptors [t0, t0 + nt) of an assemble into shared memory.
template <int RK>
__device__ __forceinline__ void stage_terms(const AsmArgs &a, SmTerm<RK> *st, int t0, int nt) {
    for (int t = threadIdx.x; t < nt; t += blockDim.x) {
        const AsmTerm &g = a.terms[t0 + t];
        SmTerm<RK> q;
        q.p = g.p;
        q.coef = g.coef;
        unsigned long long pm = 0;
        for (int gi = 0; gi < g.ng; ++gi)
            for (int u = 0; u < g.glen[gi]; ++u)
                for (int v = u + 1; v < g.glen[gi]; ++v) {
                    int j = g.gpos[gi][u], k = g.gpos[gi][v];
                    if (j > k) {
                        int tmp = j;
                        j = k;
                        k = tmp;
                    }
                    pm |= 1ull << (j * RK + k);
                }
        q.pm = pm;
#pragma unroll
        for (int d = 0; d < RK; ++d) {
            q.zs[d] = g.zstride[d];
            q.src[d] = (unsigned char)g.src[d];
            q.tst[d] = 0;
        }
#pragma unroll
        for (int j = 0; j < RK; ++j) q.tst[g.src[j]] += g.zstride[j];
        st[t] = q;
    }
}

// The term's value at element x, a view read sorted with sign.
template <int RK, typename Off>
__device__ __forceinline__ double sorted_term(const SmTerm<RK> &q, const int (&x)[RK]) {
    double sg = q.coef;
    int y[RK];
#pragma unroll
    for (int j = 0; j < RK; ++j) y[j] = pick<RK>(x, q.src[j]);
    // selection sort within groups: one sign flip per exchange
#pragma unroll
    for (int j = 0; j < RK; ++j)
#pragma unroll
        for (int k = j + 1; k < RK; ++k)
            if ((q.pm >> (j * RK + k)) & 1ull) {
                if (y[j] > y[k]) {
                    const int tmp = y[j];
                    y[j] = y[k];
                    y[k] = tmp;
                    sg = -sg;
                } else if (y[j] == y[k]) {
                    sg = 0.0;
                }
            }
    if (sg == 0.0) return 0.0;
    Off off = 0;
#pragma unroll
    for (int j = 0; j < RK; ++j) off += (Off)q.zs[j] * y[j];
    return sg * q.p[off];
}

// Off: index type of every offset (int when AsmArgs::off32 says they all fit)
// The canonical elements [base0, total) of one assemble, blockDim.x * ASM_EPT of them per step.
constexpr int ASM_PMAX = 64;   // orbit permutations whose write strides are staged in shared memory

template <int RK, typename Off, int CH>
__device__ __forceinline__ void assemble_body(const AsmArgs &a, SmTerm<RK> (&st)[CH], long long base0,
                                              long long step) {
    const int nch = (a.nterms + CH - 1) / CH;
    double nacc = 0.0;
    // write strides of every orbit permutation P: copy P of element x sits at sum_j pst[P][j] x[j]
    // (pst[P][P[d]] = tstride[d]), so a copy's offset takes RK multiply-adds and no index selects
    __shared__ int pst[ASM_PMAX * RK];
    const bool staged = a.nperm <= ASM_PMAX;
    if (staged) {
        for (int i = threadIdx.x; i < a.nperm * RK; i += blockDim.x) {
            const int pidx = i / RK, d = i - pidx * RK;
            pst[pidx * RK + a.perm[i]] = a.tstride[d];
        }
        __syncthreads();
    }
    for (long long base = base0; base < a.total; base += step) {
        int x[ASM_EPT][RK];
        bool act[ASM_EPT];    // an element of the block
        bool need[ASM_EPT];   // ... whose residual is gathered (inside the active space when one is set)
        double R[ASM_EPT];
#pragma unroll
        for (int e = 0; e < ASM_EPT; ++e) {
            const long long lin = base + e * (long long)blockDim.x + threadIdx.x;
            act[e] = lin < a.total;
            R[e] = 0.0;
#pragma unroll
            for (int d = 0; d < RK; ++d) x[e][d] = 0;
            if (act[e]) canonical_element<RK, Off>(a, (Off)lin, x[e]);
            need[e] = act[e];
            if (a.act && act[e]) {
                // CCSDt: at least one active occupied and one active virtual index
                bool occ = false, vir = false;
#pragma unroll
                for (int d = 0; d < RK; ++d) {
                    if (d < RK / 2)
                        occ = occ || x[e][d] >= a.act_occ_lo;
                    else
                        vir = vir || x[e][d] < a.act_vir_hi[a.spin[d]];
                }
                need[e] = occ && vir;
            }
        }
        for (int c = 0; c < nch; ++c) {
            __syncthreads();
            const int nt = min(CH, a.nterms - c * CH);
            stage_terms<RK>(a, st, c * CH, nt);
            __syncthreads();
            // plain views first (a branch-free loop, so the loads of several terms are in flight
            // together), then the views read sorted with sign
            const int np = min(max(a.nplain - c * CH, 0), nt);
#pragma unroll 4
            for (int t = 0; t < np; ++t) {
                const SmTerm<RK> &q = st[t];
                const double *p = q.p;
                double v[ASM_EPT];
#pragma unroll
                for (int e = 0; e < ASM_EPT; ++e) {
                    Off off = 0;
#pragma unroll
                    for (int d = 0; d < RK; ++d) off += (Off)q.tst[d] * x[e][d];
                    v[e] = need[e] ? p[off] : 0.0;
                }
#pragma unroll
                for (int e = 0; e < ASM_EPT; ++e) R[e] += q.coef * v[e];
            }
#pragma unroll 2
            for (int t = np; t < nt; ++t) {
#pragma unroll
                for (int e = 0; e < ASM_EPT; ++e)
                    if (need[e]) R[e] += sorted_term<RK, Off>(st[t], x[e]);
            }
        }
#pragma unroll
        for (int e = 0; e < ASM_EPT; ++e) {
            if (!act[e]) continue;
            Off toff = 0;
#pragma unroll
            for (int d = 0; d < RK; ++d) toff += (Off)a.tstride[d] * x[e][d];
            double tnew;
            if (a.mode != 1) {
                double D = a.shift;
                if (a.mode == 2) {
                    D -= *a.ecor;
                    nacc += a.nperm * R[e] * R[e];
                }
#pragma unroll
                for (int d = 0; d < RK; ++d) {
                    if (d < RK / 2)
                        D -= a.fdiag[a.spin[d]][x[e][d]];
                    else
                        D += a.fdiag[a.spin[d]][a.nocc[a.spin[d]] + x[e][d]];
                }
                tnew = a.T[toff] - R[e] / D;
                // triples outside the active space stay zero
                if (!need[e]) tnew = 0.0;
            } else {
                tnew = R[e];
            }
            if (staged) {
                for (int pidx = 0; pidx < a.nperm; ++pidx) {
                    Off o = 0;
#pragma unroll
                    for (int j = 0; j < RK; ++j) o += (Off)pst[pidx * RK + j] * x[e][j];
                    a.T[o] = a.psign[pidx] * tnew;
                }
            } else {
                for (int pidx = 0; pidx < a.nperm; ++pidx) {
                    const signed char *P = a.perm + pidx * RK;
                    Off o = 0;
#pragma unroll
                    for (int d = 0; d < RK; ++d) o += (Off)a.tstride[d] * pick<RK>(x[e], P[d]);
                    a.T[o] = a.psign[pidx] * tnew;
                }
            }
        }
    }
    if (a.mode == 2) {
        for (int o = 16; o > 0; o >>= 1) nacc += __shfl_down_sync(0xffffffffu, nacc, o);
        if ((threadIdx.x & 31) == 0 && nacc != 0.0) atomicAdd(a.norm, nacc);
    }
}

template <int RK, typename Off>
__global__ void __launch_bounds__(256, 4) assemble_kernel(AsmArgs a) {
    constexpr int CH = 128;
    __shared__ SmTerm<RK> st[CH];
    gdc_launch();
    gdc_wait();
    assemble_body<RK, Off, CH>(a, st, (long long)blockIdx.x * blockDim.x * ASM_EPT,
                               (long long)gridDim.x * blockDim.x * ASM_EPT);
}

// Few canonical elements, many terms or images (the T4 blocks of small systems: 210 elements, 826 terms, 576
// images): G neighbouring lanes share an element, taking its terms and then its images in turn.  With a thread per
// element such a block is one serial chain of loads and scattered stores on a few SMs (T4A of 14 orbitals 373 us, its
// copy T4E 203 us, T3A of 24 orbitals 41 us of an eager sweep).  A pass of six iterations: CCSDT 13 orbitals 1.60 -> 1.48
// ms, 24 orbitals 6.65 -> 6.53 ms, CCSDTQ 14 orbitals 45.2 -> 42.9 ms.
template <int RK, typename Off, int G>
__global__ void __launch_bounds__(256) assemble_group_kernel(AsmArgs a) {
    constexpr int CH = 128;
    __shared__ SmTerm<RK> st[CH];
    gdc_launch();
    gdc_wait();
    const int lane = threadIdx.x % G;
    const long long lin = blockIdx.x * (long long)(blockDim.x / G) + threadIdx.x / G;
    const bool act = lin < a.total;
    int x[RK];
#pragma unroll
    for (int d = 0; d < RK; ++d) x[d] = 0;
    if (act) canonical_element<RK, Off>(a, (Off)lin, x);
    bool need = act;
    if (a.act && act) {
        // CCSDt: at least one active occupied and one active virtual index
        bool occ = false, vir = false;
#pragma unroll
        for (int d = 0; d < RK; ++d) {
            if (d < RK / 2)
                occ = occ || x[d] >= a.act_occ_lo;
            else
                vir = vir || x[d] < a.act_vir_hi[a.spin[d]];
        }
        need = occ && vir;
    }
    double R = 0.0;
    for (int t0 = 0; t0 < a.nterms; t0 += CH) {
        __syncthreads();
        const int nt = min(CH, a.nterms - t0);
        stage_terms<RK>(a, st, t0, nt);
        __syncthreads();
        if (!need) continue;
        const int np = min(max(a.nplain - t0, 0), nt);
#pragma unroll 4
        for (int t = lane; t < np; t += G) {
            Off off = 0;
#pragma unroll
            for (int d = 0; d < RK; ++d) off += (Off)st[t].tst[d] * x[d];
            R += st[t].coef * st[t].p[off];
        }
#pragma unroll 2
        for (int t = np + lane; t < nt; t += G) R += sorted_term<RK, Off>(st[t], x);
    }
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) R += __shfl_xor_sync(0xffffffffu, R, o);
    Off toff = 0;
#pragma unroll
    for (int d = 0; d < RK; ++d) toff += (Off)a.tstride[d] * x[d];
    const double told = act && a.mode != 1 ? a.T[toff] : 0.0;
    __syncwarp();   // every lane of the group has read T before an image overwrites it
    if (act) {
        double tnew = R;
        if (a.mode != 1) {
            double D = a.shift;
            if (a.mode == 2) D -= *a.ecor;
#pragma unroll
            for (int d = 0; d < RK; ++d) {
                if (d < RK / 2)
                    D -= a.fdiag[a.spin[d]][x[d]];
                else
                    D += a.fdiag[a.spin[d]][a.nocc[a.spin[d]] + x[d]];
            }
            tnew = told - R / D;
            if (!need) tnew = 0.0;   // triples outside the active space stay zero
        }
        for (int pidx = lane; pidx < a.nperm; pidx += G) {
            const signed char *P = a.perm + pidx * RK;
            Off o = 0;
#pragma unroll
            for (int d = 0; d < RK; ++d) o += (Off)a.tstride[d] * pick<RK>(x, __ldg(P + d));
            a.T[o] = a.psign[pidx] * tnew;
        }
    }
    if (a.mode == 2) {
        double nacc = (act && lane == 0) ? a.nperm * R * R : 0.0;
        for (int o = 16; o > 0; o >>= 1) nacc += __shfl_down_sync(0xffffffffu, nacc, o);
        if ((threadIdx.x & 31) == 0 && nacc != 0.0) atomicAdd(a.norm, nacc);
    }
}

// Lanes per element of an assemble: enough that the elements fill the chip's threads once (148 SMs of 2048), where an
// element has that much to share.
int assemble_lanes(const AsmArgs &a) {
    const int work = a.nterms + a.nperm;
    if (a.total * 32 <= 148 * 2048 && work >= 64) return 32;
    if (a.total * 8 <= 148 * 2048 && work >= 16) return 8;
    return 1;
}

// Many assembles of the same rank in one launch (one per context of a batch of independent
// solves): block b handles the chunk b - cstart[i] (256 * ASM_EPT canonical elements) of assemble
// i, where cstart[i] <= b < cstart[i + 1]; assemble i is skipped when active[owner[i]] is zero.
template <int RK>
__global__ void __launch_bounds__(256, 4) assemble_batched_kernel(const AsmArgs *__restrict__ args,
                                                                  const long long *__restrict__ cstart, int n,
                                                                  const int *__restrict__ owner,
                                                                  const int *__restrict__ active) {
    constexpr int CH = 128;
    __shared__ SmTerm<RK> st[CH];
    const long long b = blockIdx.x;
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (__ldg(cstart + mid) <= b) lo = mid;
        else hi = mid - 1;
    }
    if (!__ldg(active + __ldg(owner + lo))) return;
    const AsmArgs &a = args[lo];
    const long long base = (b - __ldg(cstart + lo)) * blockDim.x * ASM_EPT;
    const long long step = a.total + 1;   // one chunk per block
    if (a.off32) assemble_body<RK, int, CH>(a, st, base, step);
    else assemble_body<RK, long long, CH>(a, st, base, step);
}

void launch_assemble_batched(const AsmArgs *args, const long long *cstart, int n, long long chunks, int rank,
                             const int *owner, const int *active, cudaStream_t s) {
    if (n <= 0 || chunks <= 0) return;
    switch (rank) {
        case 2: assemble_batched_kernel<2><<<(unsigned)chunks, 256, 0, s>>>(args, cstart, n, owner, active); break;
        case 4: assemble_batched_kernel<4><<<(unsigned)chunks, 256, 0, s>>>(args, cstart, n, owner, active); break;
        case 6: assemble_batched_kernel<6><<<(unsigned)chunks, 256, 0, s>>>(args, cstart, n, owner, active); break;
        case 8: assemble_batched_kernel<8><<<(unsigned)chunks, 256, 0, s>>>(args, cstart, n, owner, active); break;
        default: break;
    }
}

// Buffer copies (n doubles, src -> dst) and zeroing (src null) of many contexts in one launch;
// entry i belongs to context owner[i] and is skipped when active[owner[i]] is zero.
__global__ void copy_batched_kernel(const BatchCopy *__restrict__ cp, int n, const int *__restrict__ owner,
                                    const int *__restrict__ active) {
    for (int i = blockIdx.y; i < n; i += gridDim.y) {
        if (!__ldg(active + __ldg(owner + i))) continue;
        const BatchCopy c = cp[i];
        for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < c.n;
             e += (long long)gridDim.x * blockDim.x)
            c.dst[e] = c.src ? __ldg(c.src + e) : 0.0;
    }
}

void launch_copy_batched(const BatchCopy *cp, int n, const int *owner, const int *active, cudaStream_t s) {
    if (n <= 0) return;
    dim3 grid(64, (unsigned)std::min(n, 65535));
    copy_batched_kernel<<<grid, 256, 0, s>>>(cp, n, owner, active);
}

void launch_assemble(const AsmArgs &a, cudaStream_t s) {
    if (const int g = a.off32 ? assemble_lanes(a) : 1; g > 1 && a.total > 0) {
        const long long nb = (a.total * g + 255) / 256;
        auto go = [&](auto kernel) { launch_after(nb <= kEarlyBlocks, kernel, (unsigned)nb, 256, 0, s, a); };
        switch (a.rank) {
            case 2: go(g == 8 ? assemble_group_kernel<2, int, 8> : assemble_group_kernel<2, int, 32>); break;
            case 4: go(g == 8 ? assemble_group_kernel<4, int, 8> : assemble_group_kernel<4, int, 32>); break;
            case 6: go(g == 8 ? assemble_group_kernel<6, int, 8> : assemble_group_kernel<6, int, 32>); break;
            case 8: go(g == 8 ? assemble_group_kernel<8, int, 8> : assemble_group_kernel<8, int, 32>); break;
            default: break;
        }
        return;
    }
    long long blocks = (a.total + 256 * ASM_EPT - 1) / (256 * ASM_EPT);
    if (blocks > 148 * 32) blocks = 148 * 32;
    if (blocks < 1) blocks = 1;
    auto go = [&](auto kernel) { launch_after(blocks <= kEarlyBlocks, kernel, (unsigned)blocks, 256, 0, s, a); };
    if (a.off32) {
        switch (a.rank) {
            case 2: go(assemble_kernel<2, int>); break;
            case 4: go(assemble_kernel<4, int>); break;
            case 6: go(assemble_kernel<6, int>); break;
            case 8: go(assemble_kernel<8, int>); break;
            default: break;
        }
        return;
    }
    switch (a.rank) {
        case 2: go(assemble_kernel<2, long long>); break;
        case 4: go(assemble_kernel<4, long long>); break;
        case 6: go(assemble_kernel<6, long long>); break;
        case 8: go(assemble_kernel<8, long long>); break;
        default: break;
    }
}

// out[p][q][r][s] = f[p + n (q + n (r + n s))]: column-major (Fortran) n^4 array to
// C order; writes coalesce, reads gather
__global__ void f2c4_kernel(const double *__restrict__ f, double *__restrict__ out, long long n) {
    const long long total = n * n * n * n;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        const long long s = i % n, r = (i / n) % n, q = (i / (n * n)) % n, p = i / (n * n * n);
        out[i] = __ldg(f + p + n * (q + n * (r + n * s)));
    }
}

void launch_f2c4(const double *f, double *out, long long n, cudaStream_t s) {
    const long long total = n * n * n * n;
    long long blocks = (total + 255) / 256;
    if (blocks > 148 * 16) blocks = 148 * 16;
    if (blocks < 1) blocks = 1;
    f2c4_kernel<<<(int)blocks, 256, 0, s>>>(f, out, n);
}

__global__ void fill_kernel(double *p, double v, long long n) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        p[i] = v;
}

void launch_fill(double *p, double v, long long n, cudaStream_t s) {
    long long blocks = (n + 255) / 256;
    if (blocks > 148 * 16) blocks = 148 * 16;
    if (blocks < 1) blocks = 1;
    fill_kernel<<<(int)blocks, 256, 0, s>>>(p, v, n);
}

// ---------------------------------------------------------------------------
// DIIS on the HBM ring (src/diis.F90)
// ---------------------------------------------------------------------------
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// The step that follows every sweep, one pass: the new vector into its ring slot (cur; in place when src == cur), the
// squared distance from the previous slot (prev null: from zero) and, from the block that finishes last, the results of the
// iteration straight into the host's pinned slots.  Bound by HBM for the large vectors (24 bytes per element; the copy
// and the sum apart took 32: 0.34 -> 0.27 ms for the 67.3 M elements of 40 orbitals) and by launches for the small ones:
// copy, memset, sum and two result copies were 25 us of a 150 us iteration.
__global__ void __launch_bounds__(256) ring_step_kernel(const double *__restrict__ src, double *cur,
                                                        const double *__restrict__ prev, long long n,
                                                        double *partial, unsigned *count,
                                                        const double *__restrict__ energy, double *host) {
    double acc = 0.0;
    const long long step = (long long)gridDim.x * blockDim.x;
    const bool copy = src != cur;
    long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    for (; i + 3 * step < n; i += 4 * step) {
        double v[4], p[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            v[u] = src[i + u * step];
            p[u] = prev ? prev[i + u * step] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            if (copy) cur[i + u * step] = v[u];
            const double d = p[u] - v[u];
            acc += d * d;
        }
    }
    for (; i < n; i += step) {
        const double v = src[i], d = (prev ? prev[i] : 0.0) - v;
        if (copy) cur[i] = v;
        acc += d * d;
    }
    acc = warp_sum(acc);
    __shared__ double sh[32];
    __shared__ bool last;
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x < 32) {
        double v = threadIdx.x < (blockDim.x >> 5) ? sh[threadIdx.x] : 0.0;
        v = warp_sum(v);
        if (threadIdx.x == 0) {
            partial[blockIdx.x] = v;
            __threadfence();
            last = atomicAdd(count, 1u) == gridDim.x - 1;
        }
    }
    __syncthreads();
    if (!last) return;
    // the blocks' sums in their order: the result does not depend on which block is last
    __threadfence();
    acc = 0.0;
    for (int b = threadIdx.x; b < (int)gridDim.x; b += blockDim.x) acc += __ldcg(partial + b);
    acc = warp_sum(acc);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double v = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) v += sh[w];
        host[0] = *energy;
        host[1] = v;
        *count = 0;   // for the next launch
    }
}

void launch_ring_step(const double *src, double *cur, const double *prev, long long n, double *partial, unsigned *count,
                      const double *energy, double *host, cudaStream_t s) {
    const long long blocks = std::max(1LL, std::min<long long>((n + 1023) / 1024, RING_BLOCKS));
    ring_step_kernel<<<(int)blocks, 256, 0, s>>>(src, cur, prev, n, partial, count, energy, host);
}

// Bordered DIIS system of construct_b_mat (diis.F90:159-242, the corner is -1
// as in the reference) solved by LU with partial pivoting like dgesv, by one warp: lane j holds column j in shared
// memory (lane ds + 1 the right-hand side), the multipliers of a column are formed side by side.
__device__ void diis_solve_warp(const double *gram, int ds, double *coef, int *info, int *host_info) {
    __shared__ double B[13][15];
    const int lane = threadIdx.x & 31, n = ds + 1;
    for (int x = lane; x < n * (n + 1); x += 32) {
        const int i = x / (n + 1), j = x % (n + 1);
        double v;
        if (j == n) v = i == ds ? -1.0 : 0.0;
        else if (i == ds || j == ds) v = -1.0;
        else v = __ldcg(gram + (i <= j ? i * ds + j : j * ds + i));
        B[i][j] = v;
    }
    __syncwarp();
    int inf = 0;
    for (int k = 0; k < n; ++k) {
        int p = k;
        double best = fabs(B[k][k]);
        for (int i = k + 1; i < n; ++i)
            if (fabs(B[i][k]) > best) {
                best = fabs(B[i][k]);
                p = i;
            }
        if (best == 0.0) {
            inf = k + 1;
            break;
        }
        __syncwarp();
        if (p != k && lane <= n) {
            const double t = B[k][lane];
            B[k][lane] = B[p][lane];
            B[p][lane] = t;
        }
        __syncwarp();
        const double f = (lane > k && lane < n) ? B[lane][k] / B[k][k] : 0.0;
        const double bk = lane <= n ? B[k][lane] : 0.0;
        __syncwarp();
        for (int i = k + 1; i < n; ++i) {
            const double fi = __shfl_sync(0xffffffffu, f, i);
            if (lane >= k && lane <= n) B[i][lane] -= fi * bk;
        }
        __syncwarp();
    }
    if (lane == 0) {
        if (!inf) {
            double c[13];
            for (int i = n - 1; i >= 0; --i) {
                double s = B[i][n];
                for (int j = i + 1; j < n; ++j) s -= B[i][j] * c[j];
                c[i] = s / B[i][i];
            }
            for (int i = 0; i < n; ++i) coef[i] = c[i];
        }
        *info = inf;
        *host_info = inf;
    }
}

template <int DS>
__global__ void gram_kernel(const double *ring, long long stride, long long n, double *gram, unsigned *count,
                            double *coef, int *info, int *host_info) {
    double acc[DS][DS];
#pragma unroll
    for (int i = 0; i < DS; ++i)
#pragma unroll
        for (int j = 0; j < DS; ++j) acc[i][j] = 0.0;
    for (long long x = blockIdx.x * (long long)blockDim.x + threadIdx.x; x < n; x += (long long)gridDim.x * blockDim.x) {
        double v[DS + 1];
#pragma unroll
        for (int i = 0; i <= DS; ++i) v[i] = ring[i * stride + x];
        double d[DS];
#pragma unroll
        for (int i = 0; i < DS; ++i) d[i] = v[i + 1] - v[i];
#pragma unroll
        for (int i = 0; i < DS; ++i)
#pragma unroll
            for (int j = i; j < DS; ++j) acc[i][j] += d[i] * d[j];
    }
    __shared__ double sh[32];
#pragma unroll
    for (int i = 0; i < DS; ++i)
#pragma unroll
        for (int j = i; j < DS; ++j) {
            double v = warp_sum(acc[i][j]);
            __syncthreads();
            if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
            __syncthreads();
            if (threadIdx.x < 32) {
                double w = threadIdx.x < (blockDim.x >> 5) ? sh[threadIdx.x] : 0.0;
                w = warp_sum(w);
                if (threadIdx.x == 0) atomicAdd(&gram[i * DS + j], w);
            }
        }
    // the block that finishes last solves the bordered system and leaves the matrix at zero for the next step
    __shared__ bool last;
    if (threadIdx.x == 0) {
        __threadfence();
        last = atomicAdd(count, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    if (threadIdx.x < 32) {
        diis_solve_warp(gram, DS, coef, info, host_info);
        __syncwarp();
        for (int x = threadIdx.x; x < DS * DS; x += 32) gram[x] = 0.0;
        if (threadIdx.x == 0) *count = 0;
    }
}

void launch_diis_gram(const double *ring, long long stride, int ds, long long n, double *gram, unsigned *count,
                      double *coef, int *info, int *host_info, cudaStream_t s) {
    long long blocks = (n + 255) / 256;
    if (blocks > 148 * 4) blocks = 148 * 4;
    if (blocks < 1) blocks = 1;
    switch (ds) {
#define CASE(D) \
    case D: gram_kernel<D><<<(int)blocks, 256, 0, s>>>(ring, stride, n, gram, count, coef, info, host_info); break;
        CASE(1) CASE(2) CASE(3) CASE(4) CASE(5) CASE(6) CASE(7) CASE(8) CASE(9) CASE(10) CASE(11) CASE(12)
#undef CASE
        default: break;
    }
}

__global__ void diis_extrap_kernel(const double *ring, long long stride, int ds, long long n, const double *coef,
                                   double *t) {
    for (long long x = blockIdx.x * (long long)blockDim.x + threadIdx.x; x < n; x += (long long)gridDim.x * blockDim.x) {
        double acc = 0.0;
        for (int i = 0; i < ds; ++i) acc += coef[i] * ring[i * stride + x];
        t[x] = acc;
    }
}

void launch_diis_extrap(const double *ring, long long stride, int ds, long long n, const double *coef, double *t,
                        cudaStream_t s) {
    long long blocks = (n + 255) / 256;
    if (blocks > 148 * 16) blocks = 148 * 16;
    if (blocks < 1) blocks = 1;
    diis_extrap_kernel<<<(int)blocks, 256, 0, s>>>(ring, stride, ds, n, coef, t);
}

// With lazy module loading a kernel's code is loaded at its first launch; a
// first launch in the middle of a solve (the first DIIS step) was measured to
// stall for ~0.7 s after other libraries had loaded theirs.  Touching every
// function of the iteration here loads them when the context is created.
cudaError_t preload_kernels(int ds) {
    cudaFuncAttributes fa;
    cudaError_t e = cudaSuccess;
    auto touch = [&](const void *f) {
        if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, f);
    };
    switch (ds) {
#define CASE(D) \
    case D: touch((const void *)gram_kernel<D>); break;
        CASE(1) CASE(2) CASE(3) CASE(4) CASE(5) CASE(6) CASE(7) CASE(8) CASE(9) CASE(10) CASE(11) CASE(12)
#undef CASE
        default: break;
    }
    touch((const void *)zero_view_kernel);
    touch((const void *)f2c4_kernel);
    touch((const void *)fill_kernel);
    touch((const void *)ring_step_kernel);
    touch((const void *)diis_extrap_kernel);
    touch((const void *)assemble_group_kernel<2, int, 8>);
    touch((const void *)assemble_group_kernel<4, int, 8>);
    touch((const void *)assemble_group_kernel<6, int, 8>);
    touch((const void *)assemble_group_kernel<8, int, 8>);
    touch((const void *)assemble_group_kernel<2, int, 32>);
    touch((const void *)assemble_group_kernel<4, int, 32>);
    touch((const void *)assemble_group_kernel<6, int, 32>);
    touch((const void *)assemble_group_kernel<8, int, 32>);
    touch((const void *)assemble_kernel<2, int>);
    touch((const void *)assemble_kernel<4, int>);
    touch((const void *)assemble_kernel<6, int>);
    touch((const void *)assemble_kernel<8, int>);
    touch((const void *)assemble_kernel<2, long long>);
    touch((const void *)assemble_kernel<4, long long>);
    touch((const void *)assemble_kernel<6, long long>);
    touch((const void *)assemble_kernel<8, long long>);
    return e;
}

}  // namespace ccqb
