// FP64 grouped gather/scatter GEMM on the bf16 tensor cores for the FP64
// compressed form's M2L:  D[:, out(p), r] += A_g B[:, in(p), r].
//
// Error-free splitting (Ozaki, Ogita, Oishi and Rump, "Error-free
// transformations of matrix multiplication by using fast routines of matrix
// multiplication and its applications", Numer. Algorithms 59 (2012); on tensor
// cores: Mukunoki et al., ISC 2020).  Every row of A and every column of B is
// scaled by a power of two to below one and cut into OZ_S = 8 digits of 8 bits
// (integers of magnitude at most 128, exact in bf16):
//   a = 2^ea sum_i A_i 2^(-7 - 8 i),  |rest| <= 2^(ea - 64).
// A digit product is an integer of at most 2^14 and the products of equal
// weight, i + j = d, are summed in one FP32 accumulator over 128 depths: at
// most 8 x 128 of them, so no partial sum exceeds 2^24 and every accumulator
// is exact whatever the order of the tensor core's additions.  Deeper products
// run as several tiles of 128 depths.  The eight diagonals (36 of the 64 digit
// products; those with d >= 8 are below 2^-60 of the scales) are put together
// as two integers below 2^53, so a tile's result is rounded once, where the
// FP64 pipe rounds at every addition.
//
// What that bounds: an output is off by at most K 2^-58 max|row of A| max|column
// of B| (K the depth) and a rounding per tile.  The FP64 pipe's bound is
// relative to sum |a_k b_k|: where a row and a column are graded against each
// other over more than about 2^11 the digits hold less than it does.  The M2L
// bases do not grade that way: at rank tolerances 1e-7 to 1e-13 and densities
// over twelve decades the two paths differ by 1.0e-16 to 4.4e-16 of the
// result's norm (two operators on the FP64 pipe: 0.5e-16 to 3.2e-16) and, entry
// by entry, by at most 2.7e-15 of the larger of the entry and the rms (1.3e-15).
//
// Why: GB300's FP64 pipe does 1.25 TFLOP/s, and the 494,158 128 x 128 products
// of a 61,440-point bumpy sphere (16 GFLOP) keep it busy for 13.3 ms; 36 bf16
// products of each are 0.58 TFLOP, 0.3 ms of the tensor pipe.  That case: M2L
// 13.3 -> 1.6 ms, the apply 20.0 -> 8.4 ms, its deviation from linearity
// 9.5e-16 before and 9.7e-16 after.
//
// Layout as tc_gemm.cu: persistent, warp-specialized (8 epilogue warps, 4
// producer warps, one MMA thread), 128 x 64 output tiles, K in chunks of 32
// through a ring of two stages of 16 digit planes (64-byte rows, 64-byte
// swizzle), the eight accumulators of 64 columns filling tensor memory.  Every
// wait is bounded; a timed-out wait raises a CTA-wide abort flag, the MMAs in
// flight are drained before tensor memory is freed, and the host reports it.
#include <cuda_bf16.h>
#include <stdint.h>

#include "plan.h"
#include "tc_ptx.cuh"

namespace tbem {

namespace {

constexpr int OZ_S = OzPlanes::S, OZ_BM = 128, OZ_BN = 64, OZ_BK = 32;
constexpr int OZ_RB = OZ_BK * 2;
constexpr int OZ_A_TILE = OZ_BM * OZ_RB, OZ_B_TILE = OZ_BN * OZ_RB;
constexpr int OZ_DEPTH = 128;  // depths per tile: what keeps the digit sums exact
constexpr int OZ_STAGES = 2, OZ_STAGE_BYTES = OZ_S * (OZ_A_TILE + OZ_B_TILE);
constexpr int OZ_SMEM = OZ_STAGES * OZ_STAGE_BYTES + 1024;
constexpr uint32_t OZ_TMEM_COLS = OZ_S * OZ_BN;
constexpr uint32_t OZ_IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(OZ_BN >> 3) << 17) |
                              ((uint32_t)(OZ_BM >> 4) << 24);
constexpr int OZ_EPILOGUE = 256, OZ_PRODUCERS = 128, OZ_THREADS = OZ_EPILOGUE + OZ_PRODUCERS + 32;
static_assert(OZ_SMEM <= 227 * 1024 && OZ_TMEM_COLS == 512, "shared and tensor memory");
constexpr int OZ_NAN = INT32_MAX;  // exponent of a row holding an infinity or a NaN

struct OzArgs {
    const __nv_bfloat16* A;   // [digit][op][m_pad][k_pad]
    const int* a_exp;         // [op][m_pad]
    long a_digit, a_op;       // strides
    const __nv_bfloat16* B;   // [digit][cell * rhs][k_pad]
    const int* b_exp;         // [cell * rhs]
    long b_digit;
    int k_pad, m_pad;
    const int4* tiles;        // as in tc_gemm.cu
    const int *in_cell, *out_cell;
    int nrhs;
    double* D;                // [cell][rhs][n]
    int n;
    int* err;
    long long wait_cycles;
};

// The exponent e with |v| < 2^e (0 for a zero) and the digits of v 2^-e.
__device__ __forceinline__ int oz_exponent(double v)
{
    const int be = (__double2hiint(v) >> 20) & 0x7ff;
    return be == 0x7ff ? OZ_NAN : be == 0 ? (v == 0.0 ? INT32_MIN : -1022) : be - 1022;
}

__device__ __forceinline__ void oz_digits(double v, int e, __nv_bfloat16* out, long stride)
{
    double r = e == OZ_NAN ? 0.0 : scalbn(v, 7 - e);
#pragma unroll
    for (int i = 0; i < OZ_S; i++) {
        const double d = rint(r);
        out[i * stride] = __float2bfloat16_rn((float)d);
        r = (r - d) * 256.0;
    }
}

// `blocks` matrices [rows][n] -> digits [OZ_S][blocks][rows_pad][n_pad] (the
// digits digit_stride apart) and exponents [blocks][rows_pad], a warp per row;
// the padding is zero
__global__ void oz_split_kernel(const double* in, long blocks, int rows, int rows_pad, int n, int n_pad,
                                __nv_bfloat16* out, long digit_stride, int* exps)
{
    const int lane = threadIdx.x % 32;
    const long total = blocks * rows_pad;
    for (long w = ((long)blockIdx.x * blockDim.x + threadIdx.x) / 32; w < total;
         w += (long)gridDim.x * blockDim.x / 32) {
        const long b = w / rows_pad;
        const int r = (int)(w % rows_pad);
        const double* src = in + (b * rows + r) * (long)n;
        int e = INT32_MIN;
        if (r < rows)
            for (int k = lane; k < n; k += 32) e = max(e, oz_exponent(src[k]));
        e = __reduce_max_sync(0xffffffffu, e);
        if (e == INT32_MIN) e = 0;  // a zero row
        if (lane == 0) exps[w] = e;
        for (int k = lane; k < n_pad; k += 32)
            oz_digits(r < rows && k < n ? src[k] : 0.0, e, out + w * n_pad + k, digit_stride);
    }
}

__global__ void __launch_bounds__(OZ_THREADS, 1) oz_gemm_kernel(const OzArgs a, int n_ctiles, int m_tiles, int k_tiles)
{
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t full_bar[OZ_STAGES], empty_bar[OZ_STAGES], accf_bar, acce_bar, drain_bar;
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_flag;
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
    // tile t: column tile, row tile and depth tile (the depth tiles of one
    // output back to back)
    const int per_col = m_tiles * k_tiles, total = n_ctiles * per_col;
    auto row_of = [&](int t) { return (t % per_col) / k_tiles * OZ_BM; };
    auto k_of = [&](int t) { return t % k_tiles * OZ_DEPTH; };
    auto chunks_of = [&](int t) { return min(OZ_DEPTH, a.k_pad - k_of(t)) / OZ_BK; };

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                     "r"(OZ_TMEM_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (tid == 0) {
        for (int s = 0; s < OZ_STAGES; s++) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(&full_bar[s])), "r"(OZ_PRODUCERS));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&empty_bar[s])));
        }
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&accf_bar)));
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(&acce_bar)), "r"(OZ_EPILOGUE));
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&drain_bar)));
        abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_slot, smem0 = smem_u32(smem);

    // bounded wait that also gives up as soon as another role aborted
    auto wait = [&](uint64_t* bar, uint32_t parity) -> bool {
        const uint32_t b = smem_u32(bar);
        const long long t0 = clock64();
        while (!mbar_try(b, parity)) {
            if (*reinterpret_cast<volatile int*>(&abort_flag)) return false;
            if (clock64() - t0 > a.wait_cycles) {
                atomicExch(&abort_flag, 1);
                return false;
            }
        }
        return true;
    };

    bool mma_issued = false;
    if (warp >= 8 && warp < 12) {
        // ---------------- producers: 16-byte pieces, four per 64-byte row
        constexpr int PPR = OZ_RB / 16, RSTEP = OZ_PRODUCERS / PPR;
        constexpr int A_PER = OZ_BM / RSTEP, B_PER = OZ_BN / RSTEP;
        const int pt = tid - OZ_EPILOGUE, pj = pt % PPR, prow = pt / PPR;
        int j = 0;
        bool ok = true;
        for (int t = blockIdx.x; t < total && ok; t += gridDim.x) {
            const int4 ti = a.tiles[t / per_col];
            const int m0 = row_of(t), k_begin = k_of(t), nk = chunks_of(t);
            const __nv_bfloat16* ap = a.A + (long)ti.x * a.a_op + (long)(m0 + prow) * a.k_pad + pj * 8;
            long boff[B_PER];
#pragma unroll
            for (int i = 0; i < B_PER; i++) {
                const int c = ti.z + prow + RSTEP * i;
                boff[i] = c < ti.w ? ((long)a.in_cell[ti.y + c / a.nrhs] * a.nrhs + c % a.nrhs) * a.k_pad + pj * 8 : -1;
            }
            for (int kc = 0; kc < nk; kc++, j++) {
                const int s = j % OZ_STAGES;
                if (j >= OZ_STAGES && !wait(&empty_bar[s], ((j / OZ_STAGES) - 1) & 1)) {
                    ok = false;
                    break;
                }
                const uint32_t st = smem0 + s * OZ_STAGE_BYTES;
                const int k0 = k_begin + kc * OZ_BK;
#pragma unroll
                for (int q = 0; q < OZ_S; q++) {
#pragma unroll
                    for (int i = 0; i < A_PER; i++) {
                        const int row = prow + RSTEP * i;
                        const uint32_t dst = st + q * OZ_A_TILE + row * OZ_RB + (sw_piece<OZ_RB>(row, pj) << 4);
                        const __nv_bfloat16* src = ap + q * a.a_digit + (long)RSTEP * i * a.k_pad + k0;
                        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
                    }
#pragma unroll
                    for (int i = 0; i < B_PER; i++) {
                        const int row = prow + RSTEP * i;
                        const uint32_t dst = st + OZ_S * OZ_A_TILE + q * OZ_B_TILE + row * OZ_RB +
                                             (sw_piece<OZ_RB>(row, pj) << 4);
                        const bool v = boff[i] >= 0;
                        // a column past the end is zero-filled (nothing read)
                        const __nv_bfloat16* src = v ? a.B + q * a.b_digit + boff[i] + k0 : a.B;
                        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src),
                                     "r"(v ? 16u : 0u)
                                     : "memory");
                    }
                }
                asm volatile("cp.async.commit_group;" ::: "memory");
                if (j >= 1) {  // the chunk before has landed: hand its stage over
                    asm volatile("cp.async.wait_group 1;" ::: "memory");
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    mbar_arrive(smem_u32(&full_bar[(j - 1) % OZ_STAGES]));
                }
            }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        if (ok && j > 0) {
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            mbar_arrive(smem_u32(&full_bar[(j - 1) % OZ_STAGES]));
        }
    } else if (warp == 12) {
        // ---------------- MMA issue (one thread): digit products by diagonal
        if (lane == 0) {
            int j = 0, tc = 0;
            bool ok = true;
            for (int t = blockIdx.x; t < total && ok; t += gridDim.x, tc++) {
                if (tc >= 1 && !wait(&acce_bar, (tc - 1) & 1)) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const int nk = chunks_of(t);
                for (int kc = 0; kc < nk; kc++, j++) {
                    const int s = j % OZ_STAGES;
                    if (!wait(&full_bar[s], (j / OZ_STAGES) & 1)) {
                        ok = false;
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t st = smem0 + s * OZ_STAGE_BYTES;
#pragma unroll
                    for (int kk = 0; kk < OZ_BK / 16; kk++) {
                        const uint32_t a0 = st + kk * 32, b0 = st + OZ_S * OZ_A_TILE + kk * 32;
#pragma unroll
                        for (int d = 0; d < OZ_S; d++)
#pragma unroll
                            for (int i = 0; i <= d; i++)
                                mma_bf16(tmem + d * OZ_BN, sw_desc<OZ_RB>(a0 + i * OZ_A_TILE),
                                         sw_desc<OZ_RB>(b0 + (d - i) * OZ_B_TILE), OZ_IDESC,
                                         (uint32_t)((kc | kk | i) != 0));
                    }
                    mma_issued = true;
                    mma_commit(smem_u32(&empty_bar[s]));
                }
                if (!ok) break;
                mma_commit(smem_u32(&accf_bar));
            }
        }
    } else {
        // ---------------- epilogue (warps 0-7): warp w reads lane quarter w % 4
        // and the columns of half w / 4, eight at a time
        int tc = 0;
        for (int t = blockIdx.x; t < total; t += gridDim.x, tc++) {
            const int4 ti = a.tiles[t / per_col];
            const int row = row_of(t) + (warp % 4) * 32 + lane;
            const int c = ti.z + (warp / 4) * 32 + lane;  // lane q resolves column q of the half
            long my_off = -1;
            int my_exp = 0;
            if (c < ti.w) {
                const int p = ti.y + c / a.nrhs, r = c % a.nrhs;
                my_off = ((long)a.out_cell[p] * a.nrhs + r) * a.n;
                my_exp = a.b_exp[(long)a.in_cell[p] * a.nrhs + r];
            }
            const int ea = a.a_exp[(long)ti.x * a.m_pad + row];
            // the whole warp goes on or gives up: tcgen05.ld takes all its lanes,
            // converged
            if (!__all_sync(0xffffffffu, wait(&accf_bar, tc & 1))) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
            for (int c8 = 0; c8 < 32; c8 += 8) {
                __syncwarp();
                uint32_t v[OZ_S][8];
                const uint32_t base = tmem + ((uint32_t)((warp % 4) * 32) << 16) + (warp / 4) * 32 + c8;
#pragma unroll
                for (int d = 0; d < OZ_S; d++) tmem_ld8(base + d * OZ_BN, v[d]);
                tmem_wait_ld();
#pragma unroll
                for (int q = 0; q < 8; q++) {
                    const long off = __shfl_sync(0xffffffffu, my_off, c8 + q);
                    const int eb = __shfl_sync(0xffffffffu, my_exp, c8 + q);
                    // the upper and the lower four diagonals as integers below
                    // 2^53, in units of 2^(ea + eb - 38) and 2^-32 of that
                    auto join = [&](int d) {
                        long long x = __float2int_rn(__uint_as_float(v[d][q]));
#pragma unroll
                        for (int i = 1; i < 4; i++) x = x * 256 + __float2int_rn(__uint_as_float(v[d + i][q]));
                        return (double)x;
                    };
                    const double x = fma(join(4), 0x1p-32, join(0));
                    if (off < 0 || row >= a.n) continue;
                    const int e = ea + (eb == OZ_NAN ? 0 : eb) - 38;
                    double y = e > -1000 && e < 900 ? x * __hiloint2double((e + 1023) << 20, 0) : scalbn(x, e);
                    if (eb == OZ_NAN) y = __longlong_as_double(0x7ff8000000000000ll);
                    atomicAdd(a.D + off + row, y);
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            mbar_arrive(smem_u32(&acce_bar));
        }
    }
    __syncthreads();
    // every MMA this CTA issued has completed before tensor memory is released
    if (warp == 12 && lane == 0 && mma_issued) {
        mma_commit(smem_u32(&drain_bar));
        if (!mbar_wait(smem_u32(&drain_bar), 0)) atomicExch(&abort_flag, 1);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(OZ_TMEM_COLS));
    if (tid == 0 && abort_flag) atomicExch(a.err, 1);
}

unsigned split_grid(long rows) { return (unsigned)std::max<long>(1, std::min<long>((rows + 7) / 8, 152L * 32)); }

}  // namespace

void OzPlanes::build(const double* ops, long n_ops, int m_, int k_, cudaStream_t s)
{
    m = m_;
    k = k_;
    m_pad = (m + OZ_BM - 1) / OZ_BM * OZ_BM;
    k_pad = (k + OZ_BK - 1) / OZ_BK * OZ_BK;
    this->n_ops = n_ops;
    a.alloc((size_t)S * n_ops * m_pad * k_pad);
    a_exp.alloc((size_t)n_ops * m_pad);
    oz_split_kernel<<<split_grid(n_ops * m_pad), 256, 0, s>>>(ops, n_ops, m, m_pad, k, k_pad, a.p,
                                                             n_ops * (long)m_pad * k_pad, a_exp.p);
    TBEM_CK(cudaGetLastError());
    err.alloc(1);
    TBEM_CK(cudaMemsetAsync(err.p, 0, sizeof(int), s));
    TBEM_CK(cudaFuncSetAttribute(oz_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, OZ_SMEM));
}

void OzPlanes::split_b(const double* cells, long rows, cudaStream_t s)
{
    b.ensure((size_t)S * rows * k_pad);
    b_exp.ensure(rows);
    b_digit = rows * (long)k_pad;
    oz_split_kernel<<<split_grid(rows), 256, 0, s>>>(cells, 1, (int)rows, (int)rows, k, k_pad, b.p, b_digit, b_exp.p);
    TBEM_CK(cudaGetLastError());
}

void GemmSet::run_oz(const OzPlanes& P, double* D, int nrhs, cudaStream_t s, long* launches)
{
    if (empty()) return;
    auto it = oz_tiles.find(nrhs);
    if (it == oz_tiles.end()) {
        // column tiles: (operator, group's first pair, first column, the group's columns)
        std::vector<int4> t;
        const long nn = (long)P.m * P.k;
        for (size_t g = 0; g < npairs.size(); g++) {
            const long ncols = (long)npairs[g] * nrhs;
            if (ncols > INT32_MAX || pair0[g] > INT32_MAX)
                throw Error(TBEM_ERR_ARG, "tensor-core GEMM group too large");
            for (long c = 0; c < ncols; c += OZ_BN)
                t.push_back(make_int4((int)(A_off[g] / nn), (int)pair0[g], (int)c, (int)ncols));
        }
        if (t.size() > (size_t)INT32_MAX / 8) throw Error(TBEM_ERR_ARG, "too many tensor-core tiles");
        oz_tiles[nrhs].upload(t);
        it = oz_tiles.find(nrhs);
    }
    OzArgs a;
    a.A = P.a.p;
    a.a_exp = P.a_exp.p;
    a.a_op = (long)P.m_pad * P.k_pad;
    a.a_digit = P.n_ops * a.a_op;
    a.B = P.b.p;
    a.b_exp = P.b_exp.p;
    a.b_digit = P.b_digit;
    a.k_pad = P.k_pad;
    a.m_pad = P.m_pad;
    a.tiles = it->second.p;
    a.in_cell = d_in;
    a.out_cell = d_out;
    a.nrhs = nrhs;
    a.D = D;
    a.n = P.m;
    a.err = P.err.p;
    a.wait_cycles = P.wait_cycles > 0 ? P.wait_cycles : TC_WAIT_CYCLES;
    const int n_ctiles = (int)it->second.n, m_tiles = P.m_pad / OZ_BM, k_tiles = (P.k_pad + OZ_DEPTH - 1) / OZ_DEPTH;
    if ((long)n_ctiles * m_tiles * k_tiles > INT32_MAX) throw Error(TBEM_ERR_ARG, "too many tensor-core tiles");
    int dev = 0, sms = 0;
    TBEM_CK(cudaGetDevice(&dev));
    TBEM_CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const unsigned grid = (unsigned)std::min<long>((long)n_ctiles * m_tiles * k_tiles, std::max(sms, 1));
    oz_gemm_kernel<<<grid, OZ_THREADS, OZ_SMEM, s>>>(a, n_ctiles, m_tiles, k_tiles);
    TBEM_CK(cudaGetLastError());
    if (launches) (*launches)++;
}

}  // namespace tbem
