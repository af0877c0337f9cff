// Device kernels of libccq_b200 (sm_100a).
//
//  gett_f64     : GEMM over strided/permuted tensor views (GETT) in FP64 on the
//                 DMMA tensor pipe (mma.sync m16n8k8 f64).  Operand addresses
//                 come from per-mode offset tables, so a permuted slice of a
//                 resident tensor is read in place: this fuses the reference's
//                 reorder_shift / reorder_stripe + egemm + sum_stripe triple
//                 (src/cc/reorder_stripe.f90, src/dgemm.f90) into one kernel.
//  assemble     : residual gather of a spin block from permuted views, Jacobi
//                 step and antisymmetric fill (src/cc/t*_update.f90 tails).
//  diis_*       : ring residuum, B matrix, bordered solve and extrapolation
//                 (src/diis.F90).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace ccqb {

// message returned by ccq_b200_last_error() on this thread
void set_last_error(const char *msg);

// Programmatic dependent launch.  A kernel launched with launch_after may start while the kernel before it on the same
// stream is still running; everything it reads or writes that another kernel touches comes after gdc_wait, which
// every thread of it executes, and is read with ordinary loads: __ldg promises data that is read-only while the kernel
// lives (the compiler may move such a load ahead of the wait), which holds for tables and items only.  gdc_launch lets
// the next such kernel start.  A sweep of a small system is a chain of
// about 25 dependent launches; starting each one (its item and tables loaded) before the last has drained took six
// iterations of CCSD at 8 orbitals from 0.95 to 0.86 ms, at 20 from 1.23 to 1.14, CCSDT at 13 from 1.74 to 1.61.
__device__ __forceinline__ void gdc_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void gdc_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
template <typename... P, typename... A>
inline void launch_after(bool early, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = early ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}
// Grids above this start only when the kernel before has ended: waiting blocks would hold the SMs against other streams.
// (Limit 0 / 296 / 600 / none: CCSD at 8 orbitals 0.97 / 0.86 / 0.86 / 0.86 ms, at 33 1.52 / 1.47 / 1.46 / 1.51.)
constexpr long long kEarlyBlocks = 148 * 2;

constexpr int MAXR = 8;        // max tensor rank (T4 blocks)
constexpr int MAX_TERMS = 65536; // max views gathered by one assemble

// One (A, B, K, alpha) term of a grouped GETT: several contractions that add
// into the same output view run as one launch, so the output is read and
// written once instead of once per contraction.
struct GettSeg {
    const double *A, *B;
    const int *offA_m, *offA_k, *offB_n, *offB_k;
    int K;
    double alpha;
};

struct GettArgs {
    const double *A;
    const double *B;
    double *C;
    const int *offA_m, *offA_k, *offB_n, *offB_k, *offC_m, *offC_n;
    int M, N, K;
    double alpha;
    int beta;       // 0: overwrite, 1: accumulate
    int kchunk;     // K range handled by one blockIdx.z (split-K, atomic epilogue)
    int c_nfast;    // 1: output contiguous along n (write-out walks n), 0: along m
    // 16-byte paths, set by the host only where the tables pair up contiguous,
    // 16-byte aligned elements: vec_a / vec_b for m- (n-) major operand loads,
    // vec_c for the output write-out along its fast mode
    int vec_a, vec_b, vec_c;
    const GettSeg *segs;  // grouped launch: nseg terms (A, B, tables, K, alpha above unused)
    int nseg;
    int tile;       // 0: tile family by shape (gett_f64_family); 1: 64 x 64 tiles; 2: skinny tiles;
                    // 3: small-K FMA kernel (whole K per launch, kchunk ignored);
                    // 4: 64 x 64 tiles with a 3-stage operand pipeline;
                    // 5: skinny tiles with a 2-stage ring (more CTAs per SM);
                    // 6: register-direct small-K kernel (whole K per launch, kchunk ignored)
};

constexpr int MAXG = 4;  // antisymmetric axis groups per source view

// One permuted view read by the assemble step.  Axis j of the source holds
// target axis src[j]; groups list source axes stored only for increasing
// indices (the source is antisymmetric in them), read sorted with sign.
struct AsmTerm {
    const double *p;
    double coef;
    int zstride[MAXR];
    signed char src[MAXR];
    signed char gpos[MAXG][MAXR];
    signed char glen[MAXG];
    signed char ng;
    signed char rank;
};

struct AsmArgs {
    double *T;
    int rank;                 // 2 * level
    int level;
    int dims[MAXR];
    int tstride[MAXR];
    int spin[MAXR];           // 0 alpha, 1 beta per axis
    int runstart[MAXR];       // 1 if this axis starts a same-spin run within its half
    const double *fdiag[2];   // denominator diagonals (active range): Fock, or Hbar for mode 2
    int nocc[2];
    double shift;
    int mode;                 // 0 jacobi, 1 copy, 2 left jacobi (shift - *ecor, sum of R^2 into *norm)
    const double *ecor;       // mode 2: correlation energy subtracted from the denominators
    double *norm;             // mode 2: accumulates nperm * R^2 (every stored element's LH^2)
    int nterms;
    const AsmTerm *terms;
    int nperm;                // orbit permutations of a canonical element
    const signed char *perm;  // nperm x rank axis maps
    const signed char *psign; // nperm signs
    long long total;          // number of canonical elements
    // canonical elements are enumerated run by run (a run = same-spin axes of one
    // half); run r covers axes [run_axis0[r], run_axis0[r] + run_len[r]) and has
    // run_count[r] increasing tuples stored at combos + run_off[r]
    int nruns;
    int run_axis0[MAXR], run_len[MAXR], run_count[MAXR], run_off[MAXR];
    const unsigned char *combos;
    int off32;                // every offset (terms, T, canonical index) fits in 32 bits
    int nplain;               // terms [0, nplain) read plain views (no sorted groups); the rest sorted
    // active-space triples (mode 0 only): an element is kept when at least one occupied index is
    // >= act_occ_lo and at least one virtual index is < act_vir_hi[spin]; the others are set to zero
    int act;
    int act_occ_lo;
    int act_vir_hi[2];
};

// FP64 GETT.  Tile family by output shape: 0 = 64 x 64 tiles; 1 = skinny rows
// (M <= 32), 2 = skinny columns (N <= 32, run transposed).  kchunk is the K
// range of one split-K slice that launch_gett_f64 expects in GettArgs::kchunk
// (more than one slice adds into C atomically, so C must start at zero).
int gett_f64_family(long long M, long long N);
int gett_f64_kchunk(long long M, long long N, long long K);
// Sets the shared-memory limits of the skinny kernels; call once before the
// first launch (outside stream capture).
cudaError_t gett_f64_prepare();
// Loads the code of the iteration's kernels now (lazy module loading would
// load each at its first launch, possibly in the middle of a solve).
cudaError_t preload_kernels(int diis_space);
void launch_gett_f64(const GettArgs &a, int a_kmajor, int b_kmajor, cudaStream_t s);
void launch_zero_view(double *C, const int *offm, const int *offn, int M, int N, cudaStream_t s);
void launch_assemble(const AsmArgs &a, cudaStream_t s);

// One block of a launch over many small contractions (multi.cu): an output tile and a K range of one of them,
// C[cm[i] + cn[j]] (+)= alpha sum_k A[am[i] + ak[k]] B[bn[j] + bk[k]] for i < m, j < n, k < K.
constexpr int MULTI_K = 256;   // longest K range of an item
constexpr int MI_ADD = 1, MI_KSPLIT = 2, MI_NFAST = 4;   // add into C; warps split K; C contiguous along j
constexpr int MI_VA = 8, MI_VB = 16;                     // 16-byte operand loads (as GettArgs::vec_a, vec_b)
constexpr int MI_SHAPE = 8;    // flags >> MI_SHAPE: tile shape, below
// 0..3: one warp's tile is 16 x 16, 32 x 8, 32 x 16, 16 x 32; 4..7: 64 x 64 of a block (+2: A k-major, +1: B
// k-major); 8: one column (n = 1) and a few k; 9: copy or zero
constexpr int MS_64 = 4, MS_VEC = 8, MS_COPY = 9;
constexpr int MULTI_VEC_ROWS = 512, MULTI_VEC_K = 16, MULTI_COPY = 1024;   // rows and k of 8; values of 9
inline void multi_shape(int shape, int &rows, int &cols) {
    rows = shape == MS_VEC ? MULTI_VEC_ROWS : shape >= MS_64 ? 64 : shape == 0 || shape == 3 ? 16 : 32;
    cols = shape == MS_VEC ? 1 : shape >= MS_64 ? 64 : shape == 1 ? 8 : shape == 3 ? 32 : 16;
}
struct __align__(16) MultiItem {
    const double *A, *B;
    double *C;
    const int *am, *bn, *ak, *bk, *cm, *cn;
    double alpha;
    int m, n, k, flags;
};
void launch_gett_multi(const MultiItem *items, int n, bool tiles64, cudaStream_t s);   // items of one kind
cudaError_t preload_multi();

// T1 dressing of one two-electron block v0[p][q][r][s] (n^4) into v (dress.cu): t1 [o1][n - o1] belongs to the
// first and third index, t2 [o2][n - o2] to the second and fourth.  dress_fits: the block is
// large enough to gain and the kernels' registers and shared memory hold its occupied orbitals.
struct DressArgs {
    const double *v0, *t1, *t2;
    double *v;
    int n, o1, o2;
};
bool dress_fits(const DressArgs &d);
cudaError_t dress_prepare();   // shared-memory limits on the current device
int launch_dress(const DressArgs &d, cudaStream_t s);   // returns the number of launches

// Batched launches over the contexts of many independent solves (one plan operation of every
// context at once).  owner[i] is the context of entry i; entries of contexts with active[owner[i]]
// zero do nothing.  GETTs: 64 x 64 tiles, split into K slices of the entry's kchunk (slices add into
// C atomically: zero it first), tstart[i] = first tile of entry i (tiles = all tiles); assembles: cstart[i] = first chunk of ASM_CHUNK canonical elements of entry i.
struct BatchCopy {
    double *dst;
    const double *src;   // null: zero dst
    long long n;
};
constexpr int ASM_CHUNK = 512;   // canonical elements per block of a batched assemble (256 threads x 2)
void launch_gett_f64_batched(const GettArgs *args, const int *tstart, int n, int tiles, const int *owner,
                             const int *active, int a_kmajor, int b_kmajor, cudaStream_t s);
void launch_assemble_batched(const AsmArgs *args, const long long *cstart, int n, long long chunks, int rank,
                             const int *owner, const int *active, cudaStream_t s);
void launch_copy_batched(const BatchCopy *cp, int n, const int *owner, const int *active, cudaStream_t s);
// zero the output views of the entries (before split-K slices add into them)
void launch_zero_views_batched(const GettArgs *args, int n, const int *owner, const int *active, cudaStream_t s);
void launch_fill(double *p, double v, long long n, cudaStream_t s);
void launch_f2c4(const double *f, double *out, long long n, cudaStream_t s);
// The new vector src into its ring slot cur, |prev - src|^2, and {*energy, that} into host[0..1] (pinned, mapped).
// partial: RING_BLOCKS doubles; count: zero before the first launch, and again after each.
constexpr int RING_BLOCKS = 148 * 8;
void launch_ring_step(const double *src, double *cur, const double *prev, long long n, double *partial, unsigned *count,
                      const double *energy, double *host, cudaStream_t s);

// ccq's compressed CCSDt T3 (get_t_sizes_act): geometry of its ten sub-blocks inside the full T3
// blocks of a T vector, and the gather / scatter between the two (csrc/ccsdt_layout.cu)
struct T3ActGeom {
    long long t12 = 0;              // T1 + T2 elements (the same in both layouts)
    long long sub_off[11] = {};     // sub-block offsets within the compressed T3 part
    int block[10] = {};             // 0..3: T3A..T3D
    int lo[10][6] = {}, n[10][6] = {};   // sub-range start (0-based in the full block's axis) and extent
    long long full_off[4] = {};     // T3A..T3D offsets in the full T vector
    int fn[4][6] = {};              // full block extents (Fortran axis order)
    long long n_act = 0;            // compressed T3 elements
    long long t3_begin = 0, t3_end = 0;   // T3 range of the full T vector
};
void t3act_geometry(long long froz, long long occ_a, long long occ_b, long long orbs, long long act_occ_b,
                    long long act_unocc_a, T3ActGeom &g);
void launch_t3act_gather(const T3ActGeom &g, const double *tvec, double *cvec, cudaStream_t s);
void launch_t3act_scatter(const T3ActGeom &g, const double *cvec, double *tvec, cudaStream_t s);
// B matrix of the ring's differences and the bordered solve: coef[ds + 1], info (also to the pinned host_info).
// gram (ds^2) and count are zero before the first launch, and again after each.
void launch_diis_gram(const double *ring, long long stride, int ds, long long n, double *gram, unsigned *count,
                      double *coef, int *info, int *host_info, cudaStream_t s);
void launch_diis_extrap(const double *ring, long long stride, int ds, long long n, const double *coef, double *t,
                        cudaStream_t s);

}  // namespace ccqb
