// T1 dressing of one two-electron block, exp(-T1) v exp(T1) (the shifted integrals that the reference's
// t*_update routines rebuild term by term, src/cc/t2A_update.f90), in two passes over the block:
//   bra:  u[pq] = v[pq] - [q vir] sum_j t2[j,q] v[pj];   V[pq] = u[pq] - [p vir] sum_i t1[i,p] u[iq]
//   ket:  M[r.] += sum_e t1[r,e] M[e.] for occupied r;   M[.s] += sum_f t2[s,f] M[.f] for occupied s
// As a copy and four contractions in place, each of the five launches reads and writes the whole n^4 block (or the
// slice it changes) and waits for the one before: at n = 48, 9 occupied, 17 us for the copy and 21-29 us for each
// transform, 117 us in all, for three blocks at the head of a sweep (and again before T1B of an open shell, and before T3
// of CCSDT).  Two passes read and write the block once each: 65 us.
// One B200, six CCSD iterations: 48 orbitals 4.43 -> 3.62 ms, 32 active orbitals (open shell) 2.00 -> 1.63 ms.  Blocks
// below 8 MiB (n < 32) keep the separate transforms: there these share launches with the other small contractions,
// and the three launches per block cost what they save or more (24 orbitals 6.89 against 6.90 ms, 13 orbitals 1.88
// against 2.13 ms).
#include <algorithm>

#include "gett_tile.cuh"

namespace ccqb {

namespace {

// Bra pass over the rows p in [pa, pb): first the occupied rows (no sum over i), then the virtual ones, whose sum over
// i reads the finished occupied rows.  A warp takes 16 rows, eight consecutive (r, s) columns and a share of the q; the
// warps of a block take neighbouring columns, so that a block reads and writes 256 consecutive bytes of every (p, q).
// The operands v[p, j, c] stay in registers for the q loop; what changes with q (16 rows of v, the occupied rows of u)
// comes through a ring of BRA_ST stages of each warp's own (cp.async, no block barrier).  The sum over j runs on the
// FMA pipe with t2[j, q] by broadcast (as many terms as there are occupied orbitals, up to the template's OMAX), the
// sum over i on the DMMA pipe.  PAIR: n is even, two columns are one 16-byte access.
constexpr int BRA_W = 4, BRA_ST = 4;
constexpr int ULD = 12;   // row stride of the u stage: conflict-free fragment reads

// doubles of one stage: 16 rows of v, then KT * 8 rows of u
__host__ __device__ constexpr int bra_stage(int omax, bool vir) { return 16 * 8 + (vir ? (omax + 7) / 8 * 8 * ULD : 0); }

template <bool PAIR>
__device__ __forceinline__ void load2(double (&v)[2], const double *p, bool in0, bool in1) {
    if (PAIR) {
        const double2 x = in0 ? __ldg(reinterpret_cast<const double2 *>(p)) : make_double2(0.0, 0.0);
        v[0] = x.x;
        v[1] = x.y;
    } else {
        v[0] = in0 ? __ldg(p) : 0.0;
        v[1] = in1 ? __ldg(p + 1) : 0.0;
    }
}

template <int OMAX, bool VIR, bool PAIR>
__global__ void __launch_bounds__(BRA_W * 32) dress_bra_kernel(DressArgs d, int tiles, int shares) {
    extern __shared__ __align__(16) double sm[];
    constexpr int KT = (OMAX + 7) / 8, STAGE = bra_stage(OMAX, VIR), EL = PAIR ? 2 : 1;
    const int n = d.n, o1 = d.o1, o2 = d.o2;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, gid = lane >> 2, tig = lane & 3;
    int b = blockIdx.x;
    const int share = b % shares;
    b /= shares;
    const int pa = VIR ? o1 : 0, pb = VIR ? n : o1, p0 = pa + (b % tiles) * 16;
    const long long n2 = (long long)n * n, c0 = ((long long)(b / tiles) * BRA_W + warp) * 8;
    const int qa = n * share / shares, nq = n * (share + 1) / shares - qa;
    double *ring = sm + warp * BRA_ST * STAGE;
    double *t2 = sm + BRA_W * BRA_ST * STAGE;   // [q - qa][OMAX], zero for occupied q and past o2
    const int cn = (int)min(8LL, n2 - c0);
    auto fetch = [&](int q) {
        if (q < nq && cn > 0) {
            double *st = ring + (q % BRA_ST) * STAGE;
            const long long at = (long long)(qa + q) * n2 + c0;
#pragma unroll
            for (int x = lane; x < 16 * 8 / EL; x += 32) {
                const int r = x / (8 / EL), c = x % (8 / EL) * EL;
                const bool in = p0 + r < pb && c < cn;
                const double *src = in ? d.v0 + (long long)(p0 + r) * n * n2 + at + c : d.v0;
                if (PAIR)
                    cp_async16(st + r * 8 + c, src, in);
                else
                    cp_async8(st + r * 8 + c, src, in);
            }
            if (VIR) {
#pragma unroll
                for (int x = lane; x < KT * 8 * 8 / EL; x += 32) {
                    const int i = x / (8 / EL), c = x % (8 / EL) * EL;
                    const bool in = i < o1 && c < cn;
                    const double *src = in ? d.v + (long long)i * n * n2 + at + c : d.v;
                    if (PAIR)
                        cp_async16(st + 128 + i * ULD + c, src, in);
                    else
                        cp_async8(st + 128 + i * ULD + c, src, in);
                }
            }
        }
        cp_async_commit();
    };
#pragma unroll
    for (int q = 0; q < BRA_ST - 1; ++q) fetch(q);
    for (int x = tid; x < nq * OMAX; x += BRA_W * 32) {
        const int q = qa + x / OMAX, j = x % OMAX;
        t2[x] = (q >= o2 && j < o2) ? __ldg(d.t2 + (long long)j * (n - o2) + q - o2) : 0.0;
    }
    // this lane's rows p = p0 + gid + 8 h and columns c = 2 tig + e
    double vj[OMAX][2][2], ta[KT][4];
    double *dst[2];
    bool in[2][2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int p = p0 + gid + 8 * h;
        const long long at = (long long)(p < pb ? p : pa) * n * n2 + c0 + 2 * tig;
        in[h][0] = p < pb && 2 * tig < cn;
        in[h][1] = p < pb && 2 * tig + 1 < cn;
        dst[h] = d.v + at + qa * n2;
#pragma unroll
        for (int j = 0; j < OMAX; ++j)
            load2<PAIR>(vj[j][h], d.v0 + at + j * n2, j < o2 && in[h][0], j < o2 && in[h][1]);
    }
    if (VIR) {
#pragma unroll
        for (int k = 0; k < KT; ++k)
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                const int p = p0 + gid + 8 * (x & 1), i = k * 8 + tig + 4 * (x >> 1);
                ta[k][x] = (p < n && i < o1) ? -__ldg(d.t1 + (long long)i * (n - o1) + p - o1) : 0.0;
            }
    }
    __syncthreads();
    for (int q = 0; q < nq; ++q) {
        cp_async_wait<BRA_ST - 2>();
        __syncwarp();   // stage q has landed, and every lane is done with the one that is filled next
        fetch(q + BRA_ST - 1);
        const double *st = ring + (q % BRA_ST) * STAGE;
        double acc[4];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const double2 x = *reinterpret_cast<const double2 *>(&st[(gid + 8 * h) * 8 + 2 * tig]);
            acc[2 * h] = x.x;
            acc[2 * h + 1] = x.y;
        }
#pragma unroll
        for (int j = 0; j < OMAX; j += 2) {
            const double2 t = *reinterpret_cast<const double2 *>(&t2[q * OMAX + j]);
#pragma unroll
            for (int x = 0; x < 4; ++x) acc[x] -= t.x * vj[j][x >> 1][x & 1];
#pragma unroll
            for (int x = 0; x < 4; ++x) acc[x] -= t.y * vj[j + 1][x >> 1][x & 1];
        }
        if (VIR) {
#pragma unroll
            for (int k = 0; k < KT; ++k) {
                double bu[2];
#pragma unroll
                for (int x = 0; x < 2; ++x) bu[x] = st[128 + (k * 8 + tig + 4 * x) * ULD + gid];
                dmma_16x8x8(acc, ta[k], bu);
            }
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            if (PAIR) {
                if (in[h][0]) *reinterpret_cast<double2 *>(dst[h]) = make_double2(acc[2 * h], acc[2 * h + 1]);
            } else {
                if (in[h][0]) dst[h][0] = acc[2 * h];
                if (in[h][1]) dst[h][1] = acc[2 * h + 1];
            }
            dst[h] += n2;
        }
    }
}

// Ket pass, in place: one (p, q) matrix M[r][s] (contiguous) at a time per block, staged in shared memory with the next
// one on its way (cp.async, 16 bytes where n is even).  The occupied rows are updated in place there, then the
// occupied columns of all rows are formed; only those rows and columns are written back.  Row strides of 4 mod 16
// doubles keep every fragment read conflict-free.  NT tiles of eight occupied orbitals.
constexpr int KET_W = 4;

__host__ __device__ constexpr int ket_ld(int x) { return (x + 15) / 16 * 16 + 4; }

template <int NT>
__global__ void __launch_bounds__(KET_W * 32) dress_ket_kernel(DressArgs d) {
    extern __shared__ __align__(16) double sm[];
    const int n = d.n, o1 = d.o1, o2 = d.o2, v1 = n - o1, v2 = n - o2;
    const int lt1 = ket_ld(v1), lt2 = ket_ld(v2), lm = ket_ld(n), mat = (n + 8) * lm;
    double *t1 = sm, *t2 = t1 + NT * 8 * lt1, *m = t2 + NT * 8 * lt2;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, gid = lane >> 2, tig = lane & 3;
    const long long total = (long long)n * n;
    auto load = [&](long long pq, double *buf) {
        if (pq < total) {
            const double *M = d.v + pq * total;
            if (n & 1) {
                for (int x = tid; x < n * n; x += KET_W * 32) {
                    const int r = x / n;
                    cp_async8(buf + r * lm + x - r * n, M + x, true);
                }
            } else {
                const int n2 = n >> 1;
                for (int x = tid; x < n * n2; x += KET_W * 32) {
                    const int r = x / n2;
                    cp_async16(buf + r * lm + 2 * (x - r * n2), M + 2 * x, true);
                }
            }
        }
        cp_async_commit();
    };
    load(blockIdx.x, m);
    for (int x = tid; x < NT * 8 * lt1; x += KET_W * 32) {
        const int r = x / lt1, e = x - r * lt1;
        t1[x] = (r < o1 && e < v1) ? __ldg(d.t1 + (long long)r * v1 + e) : 0.0;
    }
    for (int x = tid; x < NT * 8 * lt2; x += KET_W * 32) {
        const int s = x / lt2, f = x - s * lt2;
        t2[x] = (s < o2 && f < v2) ? __ldg(d.t2 + (long long)s * v2 + f) : 0.0;
    }
    int st = 0;
    for (long long pq = blockIdx.x; pq < total; pq += gridDim.x, st ^= 1) {
        load(pq + gridDim.x, m + (st ^ 1) * mat);
        cp_async_wait<1>();
        __syncthreads();
        double *S = m + st * mat, *M = d.v + pq * total;
        // occupied rows: D[s][r] = M[r][s] + sum_e M[e][s] t1[r][e]
        for (int s0 = warp * 16; s0 < n; s0 += KET_W * 16) {
            double acc[NT][4];
#pragma unroll
            for (int t = 0; t < NT; ++t)
#pragma unroll
                for (int x = 0; x < 4; ++x) {
                    const int s = s0 + gid + 8 * (x >> 1), r = t * 8 + 2 * tig + (x & 1);
                    acc[t][x] = (s < n && r < o1) ? S[r * lm + s] : 0.0;
                }
            const int sa = min(s0 + gid, n - 1), sb = min(s0 + gid + 8, n - 1);
#pragma unroll 2
            for (int k = 0; k < v1; k += 8) {
                double a[4];
#pragma unroll
                for (int x = 0; x < 4; ++x) {
                    const int e = k + tig + 4 * (x >> 1);
                    a[x] = e < v1 ? S[(o1 + e) * lm + ((x & 1) ? sb : sa)] : 0.0;
                }
#pragma unroll
                for (int t = 0; t < NT; ++t) {
                    double b[2];
#pragma unroll
                    for (int x = 0; x < 2; ++x) b[x] = t1[(t * 8 + gid) * lt1 + k + tig + 4 * x];
                    dmma_16x8x8(acc[t], a, b);
                }
            }
#pragma unroll
            for (int t = 0; t < NT; ++t)
#pragma unroll
                for (int x = 0; x < 4; ++x) {
                    const int s = s0 + gid + 8 * (x >> 1), r = t * 8 + 2 * tig + (x & 1);
                    if (s < n && r < o1) {
                        S[r * lm + s] = acc[t][x];
                        if (s >= o2) M[r * n + s] = acc[t][x];
                    }
                }
        }
        __syncthreads();
        // occupied columns: D[r][s] = M[r][s] + sum_f M[r][f] t2[s][f]
        for (int r0 = warp * 16; r0 < n; r0 += KET_W * 16) {
            const int ra = min(r0 + gid, n - 1), rb = min(r0 + gid + 8, n - 1);
            double acc[NT][4];
#pragma unroll
            for (int t = 0; t < NT; ++t)
#pragma unroll
                for (int x = 0; x < 4; ++x) {
                    const int s = t * 8 + 2 * tig + (x & 1);
                    acc[t][x] = s < o2 ? S[((x >> 1) ? rb : ra) * lm + s] : 0.0;
                }
#pragma unroll 2
            for (int k = 0; k < v2; k += 8) {
                double a[4];
#pragma unroll
                for (int x = 0; x < 4; ++x) {
                    const int f = k + tig + 4 * (x >> 1);
                    a[x] = f < v2 ? S[((x & 1) ? rb : ra) * lm + o2 + f] : 0.0;
                }
#pragma unroll
                for (int t = 0; t < NT; ++t) {
                    double b[2];
#pragma unroll
                    for (int x = 0; x < 2; ++x) b[x] = t2[(t * 8 + gid) * lt2 + k + tig + 4 * x];
                    dmma_16x8x8(acc[t], a, b);
                }
            }
#pragma unroll
            for (int t = 0; t < NT; ++t)
#pragma unroll
                for (int x = 0; x < 4; ++x) {
                    const int r = r0 + gid + 8 * (x >> 1), s = t * 8 + 2 * tig + (x & 1);
                    if (r < n && s < o2) M[r * n + s] = acc[t][x];
                }
        }
        __syncthreads();   // the buffer is free for the matrix after the next one
    }
}

// occupied orbitals held in registers by the bra pass (its template argument)
int bra_omax(const DressArgs &d) {
    const int o = std::max(d.o1, d.o2);
    return o <= 4 ? 4 : o <= 6 ? 6 : o <= 8 ? 8 : o <= 10 ? 10 : o <= 12 ? 12 : o <= 16 ? 16 : 24;
}

size_t bra_smem(const DressArgs &d, bool vir) {
    return sizeof(double) * ((size_t)BRA_W * BRA_ST * bra_stage(bra_omax(d), vir) + (size_t)d.n * bra_omax(d));
}

int occ_tiles(const DressArgs &d) { return (std::max(d.o1, d.o2) + 7) / 8; }

size_t ket_smem(const DressArgs &d) {
    return sizeof(double) * (8 * occ_tiles(d) * (size_t)(ket_ld(d.n - d.o1) + ket_ld(d.n - d.o2)) +
                             2 * (size_t)(d.n + 8) * ket_ld(d.n));
}

constexpr size_t kSmemMax = 200 << 10;

template <int OMAX, bool PAIR>
void launch_bra_p(const DressArgs &d, cudaStream_t s) {
    const long long cols = ((long long)d.n * d.n + 8 * BRA_W - 1) / (8 * BRA_W);
    const int to = (d.o1 + 15) / 16, tv = (d.n - d.o1 + 15) / 16;
    // shares of q: one wave of four blocks per SM, and at least eight q each (the operands that a warp holds in
    // registers are loaded once per share)
    auto shares = [&](int tiles) {
        return (int)std::max<long long>(1, std::min<long long>(d.n / 8, 148 * 4 / (cols * tiles)));
    };
    dress_bra_kernel<OMAX, false, PAIR>
        <<<(unsigned)(cols * to * shares(to)), BRA_W * 32, bra_smem(d, false), s>>>(d, to, shares(to));
    dress_bra_kernel<OMAX, true, PAIR>
        <<<(unsigned)(cols * tv * shares(tv)), BRA_W * 32, bra_smem(d, true), s>>>(d, tv, shares(tv));
}

template <int OMAX>
void launch_bra(const DressArgs &d, cudaStream_t s) {
    if (d.n % 2)
        launch_bra_p<OMAX, false>(d, s);
    else
        launch_bra_p<OMAX, true>(d, s);
}

template <int OMAX>
cudaError_t bra_attr() {
    constexpr auto at = cudaFuncAttributeMaxDynamicSharedMemorySize;
    cudaError_t e = cudaFuncSetAttribute(dress_bra_kernel<OMAX, false, false>, at, (int)kSmemMax);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(dress_bra_kernel<OMAX, false, true>, at, (int)kSmemMax);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(dress_bra_kernel<OMAX, true, false>, at, (int)kSmemMax);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(dress_bra_kernel<OMAX, true, true>, at, (int)kSmemMax);
    return e;
}

template <int NT>
void launch_ket(const DressArgs &d, cudaStream_t s) {
    const size_t sm = ket_smem(d);
    const long long per_sm = std::max<long long>(1, std::min<long long>(8, (220 << 10) / (long long)(sm + 1024)));
    const long long g = std::min<long long>((long long)d.n * d.n, 148 * per_sm);
    dress_ket_kernel<NT><<<(unsigned)g, KET_W * 32, sm, s>>>(d);
}

}  // namespace

bool dress_fits(const DressArgs &d) {
    return (long long)d.n * d.n * d.n * d.n * 8 >= (8LL << 20) && std::max(d.o1, d.o2) <= 24 &&
           bra_smem(d, true) <= kSmemMax && ket_smem(d) <= kSmemMax;
}

cudaError_t dress_prepare() {
    constexpr auto at = cudaFuncAttributeMaxDynamicSharedMemorySize;
    cudaError_t e = cudaFuncSetAttribute(dress_ket_kernel<1>, at, (int)kSmemMax);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(dress_ket_kernel<2>, at, (int)kSmemMax);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(dress_ket_kernel<3>, at, (int)kSmemMax);
    if (e == cudaSuccess) e = bra_attr<4>();
    if (e == cudaSuccess) e = bra_attr<6>();
    if (e == cudaSuccess) e = bra_attr<8>();
    if (e == cudaSuccess) e = bra_attr<10>();
    if (e == cudaSuccess) e = bra_attr<12>();
    if (e == cudaSuccess) e = bra_attr<16>();
    if (e == cudaSuccess) e = bra_attr<24>();
    return e;
}

int launch_dress(const DressArgs &d, cudaStream_t s) {
    switch (bra_omax(d)) {
        case 4: launch_bra<4>(d, s); break;
        case 6: launch_bra<6>(d, s); break;
        case 8: launch_bra<8>(d, s); break;
        case 10: launch_bra<10>(d, s); break;
        case 12: launch_bra<12>(d, s); break;
        case 16: launch_bra<16>(d, s); break;
        default: launch_bra<24>(d, s);
    }
    switch (occ_tiles(d)) {
        case 1: launch_ket<1>(d, s); break;
        case 2: launch_ket<2>(d, s); break;
        default: launch_ket<3>(d, s);
    }
    return 3;
}

}  // namespace ccqb
