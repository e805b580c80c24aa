// Grouped gather/scatter GEMM on the SIMT pipes.
//
// Every dense translation of the FMM is one of these: for each group g
// (one translation operator A_g) and each pair p of the group,
// D[:, out(p), r] (op)= op(A_g) * B[:, in(p), r] for every right-hand side r.
// Groups are: one per level for the check-to-equivalent products (the
// reference's mat_vec(check_to_equiv, .), cpp/fmm.cpp:195,245,324,376,406),
// one per (level, octant) for M2M / L2L, one per distinct M2L translation
// (level pair + integer offset), and the compressions of the SVD-compressed
// M2L (rectangular operators).  Cell buffers are laid out [cell][rhs][len],
// so a column is len contiguous values: B columns have length k, D columns
// length m.
//
// FP32 (grouped_gemm_kernel): CTA of 256 threads, tile BM x 64 (BM = 128 or
// 64: the choice that pads m the least), each thread an (BM / 16) x 4 block of
// outputs; launches of few tiles: small_gemm_kernel.  FP64: dgemm_warp_kernel,
// tiles of one warp.  A launch with too
// few tiles to fill the GPU splits K over blockIdx.z (partial products added
// atomically).  K runs in steps of
// BK through two shared-memory buffers: the next step's global loads are in
// registers while the current step is multiplied, so one barrier per step
// and the load latency overlaps the FMAs.  Shared tiles are stored k-major
// (m / n contiguous, rows padded by 4 to spread the transposing stores over
// the banks) and read as 16-byte vectors.
#pragma once
#include <cuda_runtime.h>

namespace tbem {

constexpr int GM_BN = 64, GM_THREADS = 256;

// GEMM_ADD needs groups that write every output at most once (else the sum is
// a race): sets that add several products into one output run through a
// SlotPlan (plan.h) or atomically.
enum GemmMode { GEMM_STORE = 0, GEMM_ADD = 1, GEMM_ATOMIC = 2 };

template <typename T>
struct GemmArgs {
    const T* const* A;      // per group, row-major, rows of length lda
    const long* g_pair0;    // per group: first pair
    const int* g_npairs;    // per group: number of pairs
    const int* tile_group;  // per N-tile: group
    const int* tile_col0;   // per N-tile: first logical column within the group
    const int* in_cell;     // per pair
    const int* out_cell;    // per pair
    const T* B;
    T* D;
    int m;      // rows of op(A) = D column length
    int k;      // columns of op(A) = B column length
    int lda;    // row length of the stored A (k, or m when trans)
    int nrhs;
    int trans;  // op(A) = A^T
    int mode;
    int kchunk;  // split K: CTA z covers [z * kchunk, (z + 1) * kchunk) (multiple of BK)
};

template <typename T>
__device__ __forceinline__ void atomic_add_t(T* p, T v);
template <>
__device__ __forceinline__ void atomic_add_t<double>(double* p, double v) { atomicAdd(p, v); }
template <>
__device__ __forceinline__ void atomic_add_t<float>(float* p, float v) { atomicAdd(p, v); }

constexpr int GM_BK = 16;  // K step

// One output tile (column tile `tile`, row tile `mtile`, K split `kz`) of a
// grouped GEMM (the body of grouped_gemm_kernel).
template <int BM>
__device__ __forceinline__ void gemm_tile(const GemmArgs<float>& a, int tile, int mtile, int kz)
{
    using T = float;
    constexpr int BN = GM_BN, BK = GM_BK;
    constexpr int TM = BM / 16, TN = BN / 16;  // outputs per thread (rows x columns)
    constexpr int PA = BM + 4, PB = BN + 4;     // padded row lengths of the shared tiles
    constexpr int NA = BM * BK / GM_THREADS;    // A elements loaded per thread per step
    constexpr int NB = BN * BK / GM_THREADS;    // B elements loaded per thread per step
    static_assert(NA >= 1 && NB >= 1, "tile too small for the CTA");
    __shared__ __align__(16) T As[2][BK][PA];
    __shared__ __align__(16) T Bs[2][BK][PB];

    const int g = a.tile_group[tile];
    const int col0 = a.tile_col0[tile];
    const int m0 = mtile * BM;
    if (m0 >= a.m) return;
    const T* __restrict__ A = a.A[g];
    const long pair0 = a.g_pair0[g];
    const int ncols = a.g_npairs[g] * a.nrhs;
    const int M = a.m, K = a.k, lda = a.lda;
    const long ldb = (long)a.nrhs * K;  // cell stride in B
    const long ldd = (long)a.nrhs * M;  // cell stride in D
    const int tid = threadIdx.x;
    const int tx = tid % 16, ty = tid / 16;

    // B: this thread's gathered columns (fixed for the whole K loop).  Element
    // e = tid + i * 256 of a step is column e / BK, depth e % BK.
    const T* bcol[NB];
    int bk[NB], bj[NB];
#pragma unroll
    for (int i = 0; i < NB; i++) {
        const int e = tid + i * GM_THREADS;
        bj[i] = e / BK;
        bk[i] = e % BK;
        const int c = col0 + bj[i];
        bcol[i] = nullptr;
        if (c < ncols) {
            const int p = c / a.nrhs, r = c % a.nrhs;
            bcol[i] = a.B + (long)a.in_cell[pair0 + p] * ldb + (long)r * K;
        }
    }
    // A: element e of a step is (row e / BK, depth e % BK) without transpose
    // (k contiguous in memory), (depth e / BM, row e % BM) with it
    int am[NA], ak[NA];
#pragma unroll
    for (int i = 0; i < NA; i++) {
        const int e = tid + i * GM_THREADS;
        if (!a.trans) { am[i] = e / BK; ak[i] = e % BK; }
        else { ak[i] = e / BM; am[i] = e % BM; }
    }

    T ra[NA], rb[NB];
    // this CTA's K range (split K: the partial products meet in GEMM_ATOMIC)
    const int kb = kz * a.kchunk;
    const int kend = min(K, kb + a.kchunk);
    auto load = [&](int k0) {
#pragma unroll
        for (int i = 0; i < NA; i++) {
            const int gm = m0 + am[i], gk = k0 + ak[i];
            T v = T(0);
            if (gm < M && gk < kend) v = a.trans ? A[(long)gk * lda + gm] : A[(long)gm * lda + gk];
            ra[i] = v;
        }
#pragma unroll
        for (int i = 0; i < NB; i++) {
            const int gk = k0 + bk[i];
            rb[i] = (bcol[i] && gk < kend) ? bcol[i][gk] : T(0);
        }
    };
    auto store = [&](int buf) {
#pragma unroll
        for (int i = 0; i < NA; i++) As[buf][ak[i]][am[i]] = ra[i];
#pragma unroll
        for (int i = 0; i < NB; i++) Bs[buf][bk[i]][bj[i]] = rb[i];
    };

    T acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; i++)
#pragma unroll
        for (int j = 0; j < TN; j++) acc[i][j] = T(0);

    const int nk = (kend - kb + BK - 1) / BK;
    load(kb);
    store(0);
    __syncthreads();
    for (int kt = 0; kt < nk; kt++) {
        const int buf = kt & 1;
        if (kt + 1 < nk) load(kb + (kt + 1) * BK);
#pragma unroll
        for (int kk = 0; kk < BK; kk++) {
            T av[TM], bv[TN];
#pragma unroll
            for (int i = 0; i < TM; i += 4) {
                const float4 v = *reinterpret_cast<const float4*>(&As[buf][kk][ty * TM + i]);
                av[i] = v.x; av[i + 1] = v.y; av[i + 2] = v.z; av[i + 3] = v.w;
            }
            const float4 v = *reinterpret_cast<const float4*>(&Bs[buf][kk][tx * TN]);
            bv[0] = v.x; bv[1] = v.y; bv[2] = v.z; bv[3] = v.w;
#pragma unroll
            for (int i = 0; i < TM; i++)
#pragma unroll
                for (int j = 0; j < TN; j++) acc[i][j] += av[i] * bv[j];
        }
        if (kt + 1 < nk) store(buf ^ 1);
        __syncthreads();
    }
    // resolve the output columns before the first store (no load behind a store)
    T* dcols[TN];
#pragma unroll
    for (int j = 0; j < TN; j++) {
        const int c = col0 + tx * TN + j;
        dcols[j] = nullptr;
        if (c < ncols) {
            const int p = c / a.nrhs, r = c % a.nrhs;
            dcols[j] = a.D + (long)a.out_cell[pair0 + p] * ldd + (long)r * M;
        }
    }
#pragma unroll
    for (int j = 0; j < TN; j++) {
        T* dcol = dcols[j];
        if (!dcol) continue;
#pragma unroll
        for (int i = 0; i < TM; i++) {
            const int gm = m0 + ty * TM + i;
            if (gm >= M) continue;
            if (a.mode == GEMM_STORE) dcol[gm] = acc[i][j];
            else if (a.mode == GEMM_ADD) dcol[gm] += acc[i][j];
            else atomic_add_t<T>(&dcol[gm], acc[i][j]);
        }
    }
}

template <int BM>
__global__ void __launch_bounds__(GM_THREADS) grouped_gemm_kernel(const GemmArgs<float> a)
{
    gemm_tile<BM>(a, blockIdx.x, blockIdx.y, blockIdx.z);
}

// Row tile for m rows: the one that pads m the least (128 on a tie).
inline int gemm_bm(int m)
{
    const int p128 = (m + 127) / 128 * 128, p64 = (m + 63) / 64 * 64;
    return p64 < p128 ? 64 : 128;
}

// ------------------------------------------------- FP32 GEMM, few columns
//
// The level sums of one operator and one right-hand side are small products
// (64 to 4,096 columns of 256 rows), paced by latency: with 64-wide tiles a
// launch is 8 to 128 CTAs, each waiting for L2 once per 16 depths.  Tiles of 32 x 32 by
// 64 threads (4 x 4 outputs each, rows tm + 8 i and columns tn + 8 j) spread
// the launch over the chip, and three stages of 32 depths filled by cp.async
// keep two steps in flight (eight CTAs per SM).  Both tiles stay depth-contiguous as they
// lie in memory, rows padded to 36 floats: the 16-byte reads of a warp touch
// every bank once.  A thread multiplies 4 rows x 4 columns x 4
// depths between eight shared loads; every output is one chain over ascending
// depth, over the same split of the depth as the large tiles' (run_rect), so
// both sum alike.  B columns are read in 16-byte pieces (a depth of a multiple
// of four), A too (VA) unless it is transposed.  98,304-point fault, per
// operator: the M2M levels 38 + 18 + 15 + 12 us with the large tiles, 22 + 11 +
// 8 + 7 now; a 960-point sphere's compression (56 columns) 14.5 and 7.1.
constexpr int SG_B = 32, SG_K = 32, SG_PAD = SG_K + 4, SG_STAGES = 3, SG_THREADS = 64;

__device__ __forceinline__ void sg_copy16(float* dst, const float* src, bool in)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)),
                 "l"(src), "r"(in ? 16u : 0u)
                 : "memory");
}
__device__ __forceinline__ void sg_copy4(float* dst, const float* src, bool in)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)),
                 "l"(src), "r"(in ? 4u : 0u)
                 : "memory");
}

template <bool VA>
__global__ void __launch_bounds__(SG_THREADS) small_gemm_kernel(const GemmArgs<float> a)
{
    __shared__ __align__(16) float As[SG_STAGES][SG_B][SG_PAD], Bs[SG_STAGES][SG_B][SG_PAD];
    const int tid = threadIdx.x, tm = tid % 8, tn = tid / 8;
    const int g = a.tile_group[blockIdx.x], col0 = a.tile_col0[blockIdx.x];
    const int m0 = blockIdx.y * SG_B, M = a.m, K = a.k, lda = a.lda;
    const float* __restrict__ A = a.A[g];
    const long pair0 = a.g_pair0[g];
    const int ncols = a.g_npairs[g] * a.nrhs;
    const int kb = blockIdx.z * a.kchunk, kend = min(K, kb + a.kchunk);
    const int steps = (kend - kb + SG_K - 1) / SG_K;

    const float* bcol[4];  // this thread's B columns: tid / 8 + 8 i of the tile
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int c = col0 + tid / 8 + 8 * i;
        bcol[i] = nullptr;
        if (c < ncols) {
            const int p = c / a.nrhs, r = c - p * a.nrhs;
            bcol[i] = a.B + ((long)a.in_cell[pair0 + p] * a.nrhs + r) * K;
        }
    }
    auto load = [&](int st, int k0) {
        if constexpr (VA) {
            const int k = k0 + (tid % 8) * 4;
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const int r = tid / 8 + 8 * i;
                const bool in = m0 + r < M && k < kend;
                sg_copy16(&As[st][r][(tid % 8) * 4], in ? A + (long)(m0 + r) * lda + k : A, in);
            }
        } else {
#pragma unroll
            for (int i = 0; i < 16; i++) {
                // A^T: along the rows of the tile; A: along the depth
                const int r = a.trans ? tid % 32 : tid / 32 + 2 * i, kk = a.trans ? tid / 32 + 2 * i : tid % 32;
                const bool in = m0 + r < M && k0 + kk < kend;
                const float* src = a.trans ? A + (long)(k0 + kk) * lda + m0 + r : A + (long)(m0 + r) * lda + k0 + kk;
                sg_copy4(&As[st][r][kk], in ? src : A, in);
            }
        }
        const int k = k0 + (tid % 8) * 4;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const bool in = bcol[i] && k < kend;
            sg_copy16(&Bs[st][tid / 8 + 8 * i][(tid % 8) * 4], in ? bcol[i] + k : a.B, in);
        }
    };
#pragma unroll
    for (int q = 0; q < SG_STAGES - 1; q++) {
        if (q < steps) load(q, kb + q * SG_K);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = 0.f;
    for (int q = 0; q < steps; q++) {
        asm volatile("cp.async.wait_group %0;" ::"n"(SG_STAGES - 2) : "memory");
        __syncthreads();  // step q has landed, and every thread is done with step q - 1's stage
        const int next = q + SG_STAGES - 1;
        if (next < steps) load(next % SG_STAGES, kb + next * SG_K);
        asm volatile("cp.async.commit_group;" ::: "memory");
        const int st = q % SG_STAGES;
#pragma unroll
        for (int k = 0; k < SG_K; k += 4) {
            float4 x[4], y[4];
#pragma unroll
            for (int i = 0; i < 4; i++) x[i] = *reinterpret_cast<const float4*>(&As[st][tm + 8 * i][k]);
#pragma unroll
            for (int j = 0; j < 4; j++) y[j] = *reinterpret_cast<const float4*>(&Bs[st][tn + 8 * j][k]);
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    acc[i][j] = fmaf(x[i].x, y[j].x, acc[i][j]);
                    acc[i][j] = fmaf(x[i].y, y[j].y, acc[i][j]);
                    acc[i][j] = fmaf(x[i].z, y[j].z, acc[i][j]);
                    acc[i][j] = fmaf(x[i].w, y[j].w, acc[i][j]);
                }
        }
    }
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const int c = col0 + tn + 8 * j;
        if (c >= ncols) continue;
        const int p = c / a.nrhs, r = c - p * a.nrhs;
        float* d = a.D + ((long)a.out_cell[pair0 + p] * a.nrhs + r) * M;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int row = m0 + tm + 8 * i;
            if (row >= M) continue;
            if (a.mode == GEMM_STORE) d[row] = acc[i][j];
            else if (a.mode == GEMM_ADD) d[row] += acc[i][j];
            else atomicAdd(d + row, acc[i][j]);
        }
    }
}

// ----------------------------------------- FP32 products of one to four columns
//
// Between trees of different points almost every (level difference, offset)
// class of the M2L has its own operator and one to four pairs: 1,382 classes
// for 4,615 pairs at 6,144 sources and 4,096 observers.  Such a product reads
// its operator once for two multiply-adds per value: HBM-bound, where a tensor
// tile multiplies 64 columns for two and reads three bf16 planes (6 bytes per
// value against 4).  few_gemm_kernel<P, R>: a warp takes R rows at a time, the
// lanes their depths in P 16-byte pieces (the columns stay in registers), and
// the row sums meet in a transposing butterfly.  few_gemm_t_kernel: a thread
// per four columns of A, eight rows in flight, the rows split over blockIdx.y.
// Both add atomically.  At those sizes (ranks 320 x 288; 1,053 of 1,382 classes,
// 388 MB of operators) the geometry gradient, one product and one transposed
// one, went from 3.80 to 3.45 ms; the tensor-core launches had taken 190 and
// 223 us.
constexpr int FEW_COLS = 4, FEW_THREADS = 128, FEW_ROWS = 64, FEW_SPLIT = 2;
constexpr int FEW_MAX_K = 512;  // P <= 4

// ---------------------------------------------------------------- FP64 GEMM
//
// GB300 issues two FP64 FMAs per SM and clock (1.25 TFLOP/s), so an FP64
// translation is paced by that pipe alone: a 64 x 64 tile with K = 297 keeps
// one SM busy for 0.3 ms, and every padded row or column costs as much as a
// real one.  So the work is cut as finely as a warp allows: one warp owns 8
// rows x 4 TN columns (lane: row lane % 8, columns lane / 8 + 4 j), TN = 1 ..
// 4 being what the tile's columns need, so at most 7 rows and 3 columns per
// group are padding, and four warps of a CTA take neighbouring row blocks of
// the same columns (their B values meet in L1).  Operands are loaded straight
// from global memory (L1 keeps the lines over 16 depths): a warp needs 24
// values per 64-FMA-clock step at TN = 4, far below what L1 and L2 deliver,
// so there is no staging and no barrier.  The next U depths are in registers
// while the current U are multiplied; U = 16 / TN keeps about 1,000 pipe
// clocks of work in flight over an L2 latency.
//
// Every output is one chain over ascending depth (in GEMM_ATOMIC launches of
// too few warps K is split over blockIdx.z).
constexpr int DG_WARPS = 4, DG_ROWS = 8;

template <int TN>
__device__ __forceinline__ void dgemm_warp(const GemmArgs<double>& a, int g, int col0, int ncols, int m0, int kb,
                                           int kend)
{
    constexpr int U = TN == 1 ? 16 : TN == 2 ? 8 : 4;
    const int lane = threadIdx.x % 32, lr = lane % DG_ROWS, lc = lane / DG_ROWS;
    const int M = a.m, K = a.k, nrhs = a.nrhs;
    const long pair0 = a.g_pair0[g];
    const long ldb = (long)nrhs * K, ldd = (long)nrhs * M;
    const int row = m0 + lr;
    // rows and columns past the end read the last valid one and are not stored
    const int rrow = min(row, M - 1);
    const long astep = a.trans ? a.lda : 1;
    const double* __restrict__ ap = a.A[g] + (a.trans ? (long)rrow : (long)rrow * a.lda) + (long)kb * astep;
    const double* bp[TN];
#pragma unroll
    for (int j = 0; j < TN; j++) {
        const int c = min(col0 + lc + 4 * j, ncols - 1);
        const int p = c / nrhs, r = c - p * nrhs;
        bp[j] = a.B + (long)a.in_cell[pair0 + p] * ldb + (long)r * K + kb;
    }
    double acc[TN];
#pragma unroll
    for (int j = 0; j < TN; j++) acc[j] = 0.0;

    const int n = kend - kb, nfull = n / U;
    double av[U], bv[TN][U];
    auto load = [&](int k0) {
#pragma unroll
        for (int u = 0; u < U; u++) {
            av[u] = ap[(long)(k0 + u) * astep];
#pragma unroll
            for (int j = 0; j < TN; j++) bv[j][u] = bp[j][k0 + u];
        }
    };
    if (nfull > 0) load(0);
    for (int q = 0; q < nfull; q++) {
        double ac[U], bc[TN][U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            ac[u] = av[u];
#pragma unroll
            for (int j = 0; j < TN; j++) bc[j][u] = bv[j][u];
        }
        if (q + 1 < nfull) load((q + 1) * U);
#pragma unroll
        for (int u = 0; u < U; u++)
#pragma unroll
            for (int j = 0; j < TN; j++) acc[j] = fma(ac[u], bc[j][u], acc[j]);
    }
    for (int k = nfull * U; k < n; k++) {
        const double x = ap[(long)k * astep];
#pragma unroll
        for (int j = 0; j < TN; j++) acc[j] = fma(x, bp[j][k], acc[j]);
    }
    if (row >= M) return;
#pragma unroll
    for (int j = 0; j < TN; j++) {
        const int c = col0 + lc + 4 * j;
        if (c >= ncols) continue;
        const int p = c / nrhs, r = c - p * nrhs;
        double* d = a.D + (long)a.out_cell[pair0 + p] * ldd + (long)r * M + row;
        if (a.mode == GEMM_STORE) *d = acc[j];
        else if (a.mode == GEMM_ADD) *d += acc[j];
        else atomic_add_t<double>(d, acc[j]);
    }
}

// bn: columns per tile (4, 8 or 16); blockIdx.x the column tile, .y the group
// of DG_WARPS row blocks, .z the K split
__global__ void __launch_bounds__(32 * DG_WARPS) dgemm_warp_kernel(const GemmArgs<double> a, int bn);

// Columns per warp tile for `cols` columns of m rows on `sms` SMs: as wide as
// possible (fewer operand loads per FMA) while every SM gets 16 warps; below
// that a launch is one chain of K dependent FMAs per output, and the narrow
// tile makes the chain the shortest.
inline int dgemm_bn(long cols, int m, int sms)
{
    const long rows = (m + DG_ROWS - 1) / DG_ROWS;
    for (int bn : {16, 8})
        if (rows * ((cols + bn - 1) / bn) >= 16L * sms) return bn;
    return 4;
}

}  // namespace tbem
