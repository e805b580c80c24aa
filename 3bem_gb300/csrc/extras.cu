// Direct FP64 N-body sum on the GPU and the CSR operator.
#include <algorithm>
#include <cstring>
#include <memory>
#include <string>
#include <type_traits>
#include <vector>

#include "handle.h"
#include "nearfield.h"

namespace {

struct Staged {
    const double* p = nullptr;
    tbem::DBuf<double> own;
};

bool is_device(const void* p)
{
    cudaPointerAttributes a{};
    bool dev = p && cudaPointerGetAttributes(&a, p) == cudaSuccess &&
               (a.type == cudaMemoryTypeDevice || a.type == cudaMemoryTypeManaged);
    cudaGetLastError();
    return dev;
}

// Device view of a caller array (copied in when it is host memory).
void stage(Staged& s, const double* p, size_t n, cudaStream_t st)
{
    if (n == 0) { s.p = nullptr; return; }
    if (is_device(p)) { s.p = p; return; }
    s.own.alloc(n);
    TBEM_CK(cudaMemcpyAsync(s.own.p, p, n * sizeof(double), cudaMemcpyHostToDevice, st));
    s.p = s.own.p;
}

__global__ void widen_kernel(const double* in, double* out, long n)
{
    for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
        out[3 * i] = in[2 * i];
        out[3 * i + 1] = in[2 * i + 1];
        out[3 * i + 2] = 0.0;
    }
}

// Device view of caller points [n][sdim] as [n][3] (2D points get z = 0).
void stage_points(Staged& s, const double* p, long n, int sdim, cudaStream_t st)
{
    if (sdim == 3) {
        stage(s, p, 3 * (size_t)n, st);
        return;
    }
    Staged raw;
    stage(raw, p, 2 * (size_t)n, st);
    s.own.alloc(3 * (size_t)n);
    widen_kernel<<<(unsigned)std::max<long>(1, std::min<long>((n + 255) / 256, 9728)), 256, 0, st>>>(
        raw.p, s.own.p, n);
    TBEM_CK(cudaGetLastError());
    // raw's own buffer (if any) is freed on return: finish the copy first
    TBEM_CK(cudaStreamSynchronize(st));
    s.p = s.own.p;
}

__global__ void weight_kernel(const double* x, const double* w, double* s, long N, long total)
{
    for (long t = (long)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (long)gridDim.x * blockDim.x)
        s[t] = w[t % N] * x[t];
}

__global__ void narrow_kernel(const long* in, int* out, long n)
{
    for (long t = (long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long)gridDim.x * blockDim.x)
        out[t] = (int)in[t];
}

// y = A x (add = 0) or y += A x (add = 1).  L lanes per row (L chosen per
// matrix from its mean row length): a lane takes the row's entries k = b +
// lane, + L, ..., CSR_UNROLL of them per step, and the L partial sums meet in
// shuffles.  HBM-bound: 12 bytes per entry (FP64 value, 32-bit column; 64-bit
// columns only where there are 2^31 of them).
constexpr int CSR_UNROLL = 4, CSR_THREADS = 256, CSR_CTAS_PER_SM = 4, CSR_RHS = 4;

// The step of the row ending at entry e that starts at entry b: this lane's
// values and columns (-1 past the end), all loads independent.
template <int L, typename I>
__device__ __forceinline__ void csr_step(const double* val, const I* col, long b, long e, int lane,
                                         double (&v)[CSR_UNROLL], I (&c)[CSR_UNROLL])
{
    const int n = (int)min(e - b, (long)CSR_UNROLL * L);
    const double* pv = val + b + lane;
    const I* pc = col + b + lane;
#pragma unroll
    for (int u = 0; u < CSR_UNROLL; u++) {
        const bool in = lane + u * L < n;
        v[u] = in ? __ldg(pv + u * L) : 0.0;
        c[u] = in ? __ldg(pc + u * L) : I(-1);
    }
}

// NR right-hand sides (up to CSR_RHS; the entries are read once for all of
// them).  Two things pace it besides HBM.  The FP64 pipe takes
// 16 clocks per warp instruction, so the L-lane sums matter: a row of 50
// entries on 16 lanes is 4 FMA and 4 shuffle additions for two rows, on 4
// lanes 13 and 2 for eight.  And a row is three dependent reads (row start,
// entries, gather of x), so a thread that lived for one row would have its
// entry loads in flight a third of the time: the CTAs that fit the chip walk
// the rows, a warp's 32 / L rows in step, and load the next step -- of these
// rows, or the first of the warp's next ones, whose row starts are read one
// set ahead -- before they gather for the current one.  184,320
// rows of 50 entries (110 MB): 61 us with one row per 16-lane group and 64-bit
// columns, 33 us now; deeper or shallower steps and other occupancies (2 to 8
// entries, 3 to 8 CTAs per SM) measured within 3 % of that.
template <int L, int NR, typename I>
__global__ void __launch_bounds__(CSR_THREADS, NR == 1 ? CSR_CTAS_PER_SM : CSR_CTAS_PER_SM - 1)
csr_kernel(const long* __restrict__ rowptr, const I* __restrict__ col, const double* __restrict__ val,
           const double* __restrict__ x, double* y, long n_rows, long n_cols, int add)
{
    constexpr int U = CSR_UNROLL;
    const int lane = threadIdx.x % L;
    const long stride = (long)gridDim.x * (CSR_THREADS / L);
    long row = (long)blockIdx.x * (CSR_THREADS / L) + threadIdx.x / L;
    const long row0 = row - (threadIdx.x % 32) / L;  // the warp's first row
    double v[U], v2[U];
    I c[U], c2[U];
    // rows past the end have no entries
    auto bounds = [&](long r, long& rb, long& re) {
        rb = r < n_rows ? rowptr[r] : 0;
        re = r < n_rows ? rowptr[r + 1] : 0;
    };
    long b, e, nb, ne;
    bounds(row, b, e);
    bounds(row + stride, nb, ne);
    csr_step<L>(val, col, b, e, lane, v, c);
    for (long set = row0; set < n_rows; set += stride) {
        long nnb, nne;
        bounds(row + 2 * stride, nnb, nne);
        // steps of the longest of the warp's rows
        const long mine = (e - b + U * L - 1) / (U * L);
        const int steps = (int)max(1u, __reduce_max_sync(0xffffffffu, (unsigned)min(mine, (long)INT32_MAX)));
        double acc[NR];
#pragma unroll
        for (int r = 0; r < NR; r++) acc[r] = 0.0;
        for (int st = 1; st <= steps; st++) {
            b += U * L;
            if (st < steps) csr_step<L>(val, col, min(b, e), e, lane, v2, c2);
            else csr_step<L>(val, col, nb, ne, lane, v2, c2);
#pragma unroll
            for (int u = 0; u < U; u++)
                if (c[u] >= 0) {
#pragma unroll
                    for (int r = 0; r < NR; r++) acc[r] += v[u] * x[r * n_cols + c[u]];
                }
#pragma unroll
            for (int u = 0; u < U; u++) {
                v[u] = v2[u];
                c[u] = c2[u];
            }
        }
#pragma unroll
        for (int r = 0; r < NR; r++) {
#pragma unroll
            for (int o = L / 2; o > 0; o >>= 1) acc[r] += __shfl_xor_sync(0xffffffffu, acc[r], o);
            if (lane == 0 && row < n_rows) {
                double* d = y + r * n_rows + row;
                *d = add ? *d + acc[r] : acc[r];
            }
        }
        row += stride;
        b = nb;
        e = ne;
        nb = nnb;
        ne = nne;
    }
}

// FMA-rate microbenchmark: FMA_CHAINS independent chains a = a * b + c per
// thread, FMA_UNROLL steps per iteration.  b < 1 keeps the values bounded;
// the store happens only for a sum no chain reaches, so nothing is written
// while the compiler must still compute every chain.
constexpr int FMA_CHAINS = 8, FMA_UNROLL = 16, FMA_THREADS = 256;

template <typename T>
__global__ void __launch_bounds__(FMA_THREADS) fma_peak_kernel(T* out, int iters, T b, T c)
{
    T a[FMA_CHAINS];
#pragma unroll
    for (int i = 0; i < FMA_CHAINS; i++) a[i] = T(threadIdx.x + i) * T(1e-3);
    for (int it = 0; it < iters; it++) {
#pragma unroll
        for (int k = 0; k < FMA_UNROLL; k++)
#pragma unroll
            for (int i = 0; i < FMA_CHAINS; i++) a[i] = fma(a[i], b, c);
    }
    T s = T(0);
#pragma unroll
    for (int i = 0; i < FMA_CHAINS; i++) s += a[i];
    if (s == T(-1)) out[(long)blockIdx.x * blockDim.x + threadIdx.x] = s;
}

template <typename T>
double fma_peak(int device)
{
    using namespace tbem;
    DeviceGuard guard(device);
    int sms = 0, threads = 0;
    TBEM_CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
    TBEM_CK(cudaDeviceGetAttribute(&threads, cudaDevAttrMaxThreadsPerMultiProcessor, device));
    const int blocks = sms * std::max(threads / FMA_THREADS, 1);
    const double per_iter = 2.0 * FMA_CHAINS * FMA_UNROLL * (double)blocks * FMA_THREADS;
    DBuf<T> out;
    out.alloc((size_t)blocks * FMA_THREADS);
    cudaStream_t s;
    TBEM_CK(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
    cudaEvent_t e0, e1;
    TBEM_CK(cudaEventCreate(&e0));
    TBEM_CK(cudaEventCreate(&e1));
    // size the run to ~10 ms from a short first run
    int iters = 64;
    double best = 0.0;
    for (int run = 0; run < 5; run++) {
        TBEM_CK(cudaEventRecord(e0, s));
        fma_peak_kernel<T><<<blocks, FMA_THREADS, 0, s>>>(out.p, iters, T(0.999), T(1e-3));
        TBEM_CK(cudaGetLastError());
        TBEM_CK(cudaEventRecord(e1, s));
        TBEM_CK(cudaEventSynchronize(e1));
        float ms = 0.f;
        TBEM_CK(cudaEventElapsedTime(&ms, e0, e1));
        const double tf = per_iter * iters / (ms * 1e-3) / 1e12;
        if (run >= 2) best = std::max(best, tf);  // runs 0-1: sizing and warm-up
        if (run == 0) iters = std::max(1, (int)std::min(1e8, iters * 10.0 / std::max((double)ms, 1e-3)));
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cudaStreamDestroy(s);
    return best;
}
}  // namespace

struct TbemCsr {
    long n_rows = 0, n_cols = 0, nnz = 0;
    int lanes = 32;  // lanes per row of the SpMV kernel (csr_lanes, csr_block_lanes)
    tbem::DBuf<long> rowptr;
    tbem::DBuf<int> col;        // n_cols <= 2^31 - 1
    tbem::DBuf<long> col_wide;  // else
    tbem::DBuf<double> val;
};

namespace {
// y (+)= A x on stream s (A non-empty)
// Lanes per row: the fewest that take a mean row in one unrolled step (its
// latency), but no more than give the chip a thousand threads per SM: from
// there on fewer lanes add less on the FP64 pipe.  The rows of a warp walk in
// step with the longest of them, so the matrix's longest row also sets a
// least: 24 steps, or twice the steps of an even share where that is more
// (100,000 rows, one of a thousand with 5,000 entries and 12 else: 178 us with
// 4 lanes, 99 with 16; one row of 200,000 among rows of 20: 4.8 ms with 4, 0.67
// with 32; one of a hundred with 500 entries and 50 else: 62 with 4, 56 with 8).
int csr_lanes(const long* row_ptrs, long n_rows, long nnz, int sms)
{
    const double mean = n_rows > 0 ? (double)nnz / (double)n_rows : 0.0;
    const long threads = 1024L * sms;
    long longest = 0;
    for (long i = 0; i < n_rows; i++) longest = std::max(longest, row_ptrs[i + 1] - row_ptrs[i]);
    const long most = CSR_UNROLL * std::max(24L, nnz / (2 * threads));  // entries per lane
    int lanes = mean <= 4 * CSR_UNROLL ? 4 : mean <= 8 * CSR_UNROLL ? 8 : mean <= 16 * CSR_UNROLL ? 16 : 32;
    while (lanes > 4 && n_rows * (lanes / 2) >= threads) lanes /= 2;
    while (lanes < 32 && longest > most * lanes) lanes *= 2;
    return lanes;
}

// The lanes of a launch of `nr` right-hand sides: long mean rows read best in
// longer pieces where the gathers do not pace (40,000 rows of 500, 1,000 and
// 2,000 entries, 4 / 16 lanes, us: one right-hand side 97 / 79, 163 / 122, 296
// / 207; two 117 / 127, 200 / 212, 364 / 382; four 193 / 218, 351 / 324, 666 /
// 591).
int csr_block_lanes(const TbemCsr* A, int nr)
{
    const double mean = (double)A->nnz / (double)A->n_rows;
    const bool pieces = (nr == 1 && mean > 256) || (nr == CSR_RHS && mean > 768);
    return pieces ? std::max(A->lanes, 16) : A->lanes;
}

void csr_launch(const TbemCsr* A, const double* x, double* y, int nrhs, int add, cudaStream_t s)
{
    const int sms = tbem::sm_count();
    auto block = [&](auto lanes, const auto* col, int r0, int nr) {
        constexpr int LL = decltype(lanes)::value;
        const long need = (A->n_rows * LL + CSR_THREADS - 1) / CSR_THREADS;
        const unsigned blocks = (unsigned)std::min<long>(need, (long)CSR_CTAS_PER_SM * sms);
        const double* xr = x + (long)r0 * A->n_cols;
        double* yr = y + (long)r0 * A->n_rows;
        auto launch = [&](auto kern) {
            kern<<<blocks, CSR_THREADS, 0, s>>>(A->rowptr.p, col, A->val.p, xr, yr, A->n_rows, A->n_cols, add);
        };
        using I = std::remove_const_t<std::remove_pointer_t<decltype(col)>>;
        switch (nr) {
        case 1: launch(csr_kernel<LL, 1, I>); break;
        case 2: launch(csr_kernel<LL, 2, I>); break;
        case 3: launch(csr_kernel<LL, 3, I>); break;
        default: launch(csr_kernel<LL, 4, I>);
        }
    };
    auto go = [&](const auto* col) {
        for (int r0 = 0; r0 < nrhs; r0 += CSR_RHS) {
            const int nr = std::min(nrhs - r0, CSR_RHS), L = csr_block_lanes(A, nr);
            if (L == 4) block(std::integral_constant<int, 4>(), col, r0, nr);
            else if (L == 8) block(std::integral_constant<int, 8>(), col, r0, nr);
            else if (L == 16) block(std::integral_constant<int, 16>(), col, r0, nr);
            else block(std::integral_constant<int, 32>(), col, r0, nr);
        }
    };
    if (A->col.p) go(A->col.p);
    else go(A->col_wide.p);
    TBEM_CK(cudaGetLastError());
}
}  // namespace

extern "C" {

int tbem_direct_apply(int kernel, const double* kernel_params, const double* obs_locs,
                      const double* obs_normals, long n_obs, const double* src_locs,
                      const double* src_normals, const double* src_weights, long n_src,
                      const double* x, double* y, int n_rhs, void* stream)
{
    using namespace tbem;
    try {
        if (!kernel_valid(kernel) || n_obs < 0 || n_src < 0 || n_rhs <= 0 || !y)
            throw Error(TBEM_ERR_ARG, "bad argument");
        if (n_src > (long)INT32_MAX) throw Error(TBEM_ERR_ARG, "too many sources");
        if (n_obs > 0 && n_src > 0 && (!obs_locs || !obs_normals || !src_locs || !src_normals ||
                                       !src_weights || !x))
            throw Error(TBEM_ERR_ARG, "null point or input array");
        const int R = kernel_dim(kernel);
        const int sdim = kernel_space_dim(kernel);
        const double mu = (kernel_params && R > 1) ? kernel_params[0] : 1.0;
        const double nu = (kernel_params && R > 1) ? kernel_params[1] : 0.25;
        const KParams kp = make_kparams(kernel, mu, nu);
        cudaStream_t s = (cudaStream_t)stream;
        const bool y_dev = is_device(y);
        const size_t ny = (size_t)R * n_obs * n_rhs;
        if (n_obs == 0) return TBEM_OK;
        DBuf<double> ybuf;
        double* yd = y;
        if (!y_dev) { ybuf.alloc(ny); yd = ybuf.p; }
        if (n_src == 0) {
            TBEM_CK(cudaMemsetAsync(yd, 0, ny * sizeof(double), s));
        } else {
            Staged ol, on, sl, sn, sw, xs;
            stage_points(ol, obs_locs, n_obs, sdim, s);
            stage_points(on, obs_normals, n_obs, sdim, s);
            stage_points(sl, src_locs, n_src, sdim, s);
            stage_points(sn, src_normals, n_src, sdim, s);
            stage(sw, src_weights, n_src, s);
            stage(xs, x, (size_t)R * n_src * n_rhs, s);
            DBuf<double> str;
            str.alloc((size_t)R * n_src * n_rhs);
            const long tot = (long)R * n_src * n_rhs;
            weight_kernel<<<std::max<long>(1, std::min<long>((tot + 255) / 256, 9728)), 256, 0, s>>>(xs.p, sw.p, str.p, n_src, tot);
            TBEM_CK(cudaGetLastError());
            // tasks: chunks of observation points against all sources
            TaskSet ts;
            const int chunk = 1024;
            double org[3] = {0, 0, 0};
            for (long b = 0; b < n_obs; b += chunk)
                ts.add(b, (int)std::min<long>(chunk, n_obs - b), org, {{0L, (int)n_src}});
            const int tpt = direct_tpt(n_obs, sm_count());
            ts.upload({tpt});
            EvalArgs<double> a{};
            ts.fill(a);
            a.t_xyz = ol.p;
            a.t_nrm = on.p;
            a.s_xyz = sl.p;
            a.s_nrm = sn.p;
            a.s_str = str.p;
            a.s_n = n_src;
            a.y = yd;
            a.y_n = n_obs;
            a.nrhs = n_rhs;
            a.add = 0;
            a.c2 = kp.c2;
            a.scale = kp.scale;
            const TaskSet::Items& it = ts.cuts.at(tpt);
            TaskSet::fill_items(a, it);  // one number of threads per target for all items
            for (a.tpt_log = 0; (1 << a.tpt_log) < tpt;) a.tpt_log++;
            EvalLaunch L{kernel, false, false, false, it.n, EVAL_PER_ITEM};
            for (int r0 = 0; r0 < n_rhs; r0 += (n_rhs - r0 > 1 ? EVAL_NR : 1)) {
                a.rhs0 = r0;
                TBEM_CK(launch_eval<double>(L, a, s));
            }
        }
        if (!y_dev) TBEM_CK(cudaMemcpyAsync(y, yd, ny * sizeof(double), cudaMemcpyDeviceToHost, s));
        TBEM_CK(cudaStreamSynchronize(s));
        return TBEM_OK;
    } catch (...) {
        return tbem::api_status();
    }
}

int tbem_csr_create(long n_rows, long n_cols, const double* values, const long* column_indices,
                    const long* row_ptrs, TbemCsr** out)
{
    using namespace tbem;
    if (!out || n_rows < 0 || n_cols < 0 || !row_ptrs) return TBEM_ERR_ARG;
    *out = nullptr;
    try {
        if (row_ptrs[0] != 0) throw Error(TBEM_ERR_ARG, "row_ptrs[0] must be 0");
        for (long i = 0; i < n_rows; i++)
            if (row_ptrs[i + 1] < row_ptrs[i]) throw Error(TBEM_ERR_ARG, "row_ptrs must not decrease");
        const long nnz = row_ptrs[n_rows];
        if (nnz > 0 && (!values || !column_indices)) throw Error(TBEM_ERR_ARG, "null values");
        // column check on all host cores, in blocks (one flag per block)
        const long block = 1 << 20, n_blocks = (nnz + block - 1) / block;
        std::vector<char> bad(n_blocks, 0);
        nf::parallel_for(
            n_blocks,
            [&](long b) {
                for (long k = b * block; k < std::min(nnz, (b + 1) * block); k++)
                    if (column_indices[k] < 0 || column_indices[k] >= n_cols) bad[b] = 1;
            },
            1);
        if (std::find(bad.begin(), bad.end(), 1) != bad.end())
            throw Error(TBEM_ERR_ARG, "column index out of range");
        auto h = std::make_unique<TbemCsr>();
        h->n_rows = n_rows;
        h->n_cols = n_cols;
        h->nnz = nnz;
        h->lanes = csr_lanes(row_ptrs, n_rows, nnz, sm_count());
        h->rowptr.upload(row_ptrs, (size_t)n_rows + 1);
        if (nnz > 0) {
            // narrowed on the device (on the host its fresh pages took longer
            // than the copy: 9.2 M entries 4.65 ms, 2.3 without)
            DBuf<long> full;
            full.upload(column_indices, (size_t)nnz);
            if (n_cols > (long)INT32_MAX) {
                h->col_wide = std::move(full);
            } else {
                h->col.alloc((size_t)nnz);
                narrow_kernel<<<(unsigned)std::min<long>((nnz + 255) / 256, 9728), 256>>>(full.p, h->col.p, nnz);
                TBEM_CK(cudaGetLastError());
            }
            h->val.upload(values, (size_t)nnz);  // (waits for the narrowing as well)
        }
        *out = h.release();
        return TBEM_OK;
    } catch (...) {
        return tbem::api_status();
    }
}

int tbem_csr_apply(TbemCsr* h, const double* x, double* y, int n_rhs, void* stream)
{
    using namespace tbem;
    if (!h || !y || n_rhs <= 0 || (!x && h->n_cols > 0)) {
        tbem::set_last_error("null argument or n_rhs <= 0");
        return TBEM_ERR_ARG;
    }
    try {
        cudaStream_t s = (cudaStream_t)stream;
        if (h->n_rows == 0) return TBEM_OK;
        const size_t ny = (size_t)h->n_rows * n_rhs;
        const bool y_dev = is_device(y);
        DBuf<double> ybuf;
        double* yd = y;
        if (!y_dev) { ybuf.alloc(ny); yd = ybuf.p; }
        if (h->nnz == 0) {
            TBEM_CK(cudaMemsetAsync(yd, 0, ny * sizeof(double), s));
        } else {
            Staged xs;
            stage(xs, x, (size_t)h->n_cols * n_rhs, s);
            csr_launch(h, xs.p, yd, n_rhs, 0, s);
        }
        if (!y_dev) TBEM_CK(cudaMemcpyAsync(y, yd, ny * sizeof(double), cudaMemcpyDeviceToHost, s));
        TBEM_CK(cudaStreamSynchronize(s));
        return TBEM_OK;
    } catch (...) {
        return tbem::api_status();
    }
}

long tbem_csr_nnz(const TbemCsr* h) { return h ? h->nnz : TBEM_ERR_ARG; }

int tbem_csr_shape(const TbemCsr* h, long* n_rows, long* n_cols)
{
    if (!h) return TBEM_ERR_ARG;
    if (n_rows) *n_rows = h->n_rows;
    if (n_cols) *n_cols = h->n_cols;
    return TBEM_OK;
}

int tbem_csr_download(const TbemCsr* h, double* values, long* column_indices, long* row_ptrs)
{
    using namespace tbem;
    if (!h) return TBEM_ERR_ARG;
    try {
        if (row_ptrs)
            TBEM_CK(cudaMemcpy(row_ptrs, h->rowptr.p, sizeof(long) * (h->n_rows + 1), cudaMemcpyDeviceToHost));
        if (h->nnz > 0 && values)
            TBEM_CK(cudaMemcpy(values, h->val.p, sizeof(double) * h->nnz, cudaMemcpyDeviceToHost));
        if (h->nnz > 0 && column_indices) {
            if (h->col.p) {
                std::vector<int> narrow(h->nnz);
                TBEM_CK(cudaMemcpy(narrow.data(), h->col.p, sizeof(int) * h->nnz, cudaMemcpyDeviceToHost));
                std::copy(narrow.begin(), narrow.end(), column_indices);
            } else {
                TBEM_CK(cudaMemcpy(column_indices, h->col_wide.p, sizeof(long) * h->nnz, cudaMemcpyDeviceToHost));
            }
        }
        return TBEM_OK;
    } catch (...) {
        return tbem::api_status();
    }
}

void tbem_csr_destroy(TbemCsr* h) { delete h; }


// ---- IntegralOperator: y = G (F (I x)) + N x + C x on the device -------------

}  // extern "C"

struct TbemIntegral {
    TbemCsr *near = nullptr, *corr = nullptr, *galerkin = nullptr, *interp = nullptr;
    TbemFmm* far = nullptr;
    long n_rows = 0, n_cols = 0;
    tbem::DBuf<double> xi, xf, yf, yo;  // I x, F (I x), staged output
};

namespace {
void csr_into(const TbemCsr* A, const double* x, double* y, int nrhs, int add, cudaStream_t s)
{
    if (A->n_rows == 0) return;
    if (A->nnz == 0) {
        if (!add) TBEM_CK(cudaMemsetAsync(y, 0, sizeof(double) * A->n_rows * nrhs, s));
        return;
    }
    csr_launch(A, x, y, nrhs, add, s);
}
}  // namespace

extern "C" {

int tbem_integral_create(TbemCsr* nearfield, TbemCsr* correction, TbemCsr* galerkin,
                         TbemFmm* farfield, TbemCsr* interp, TbemIntegral** out)
{
    if (!out) return TBEM_ERR_ARG;
    *out = nullptr;
    if (!nearfield || !correction || !galerkin || !farfield || !interp) {
        tbem::set_last_error("null operator");
        return TBEM_ERR_ARG;
    }
    const long fr = tbem_fmm_n_rows(farfield), fc = tbem_fmm_n_cols(farfield);
    const long n = nearfield->n_rows, m = nearfield->n_cols;
    if (correction->n_rows != n || correction->n_cols != m || galerkin->n_rows != n ||
        galerkin->n_cols != fr || interp->n_rows != fc || interp->n_cols != m) {
        tbem::set_last_error("operator shapes do not chain: G (n x F rows), F, I (F cols x m), N and C (n x m)");
        return TBEM_ERR_ARG;
    }
    TbemIntegral* h = new TbemIntegral();
    h->near = nearfield;
    h->corr = correction;
    h->galerkin = galerkin;
    h->far = farfield;
    h->interp = interp;
    h->n_rows = n;
    h->n_cols = m;
    *out = h;
    return TBEM_OK;
}

int tbem_integral_apply(TbemIntegral* h, const double* x, double* y, int n_rhs, void* stream)
{
    using namespace tbem;
    if (!h || !y || n_rhs <= 0 || (!x && h->n_cols > 0)) {
        set_last_error("null argument or n_rhs <= 0");
        return TBEM_ERR_ARG;
    }
    try {
        // one stream for the whole chain: the caller's, else the farfield's own
        // (the FMM apply would otherwise run on that one, unordered with the
        // sparse steps)
        cudaStream_t s = stream ? (cudaStream_t)stream : h->far->plan.stream;
        if (h->n_rows == 0) return TBEM_OK;
        const size_t ny = (size_t)h->n_rows * n_rhs;
        const bool y_dev = is_device(y);
        double* yd = y;
        if (!y_dev) {
            h->yo.ensure(ny);
            yd = h->yo.p;
        }
        Staged xs;
        stage(xs, x, (size_t)h->n_cols * n_rhs, s);
        const long fr = tbem_fmm_n_rows(h->far), fc = tbem_fmm_n_cols(h->far);
        h->xi.ensure(std::max<size_t>((size_t)fc * n_rhs, 1));
        h->xf.ensure(std::max<size_t>((size_t)fr * n_rhs, 1));
        csr_into(h->interp, xs.p, h->xi.p, n_rhs, 0, s);               // I x
        h->far->plan.apply(h->xi.p, h->xf.p, n_rhs, s, false);        // F (I x)
        csr_into(h->galerkin, h->xf.p, yd, n_rhs, 0, s);               // G F I x
        csr_into(h->near, xs.p, yd, n_rhs, 1, s);                      // + N x
        csr_into(h->corr, xs.p, yd, n_rhs, 1, s);                      // + C x
        if (!y_dev) TBEM_CK(cudaMemcpyAsync(y, yd, ny * sizeof(double), cudaMemcpyDeviceToHost, s));
        TBEM_CK(cudaStreamSynchronize(s));
        return TBEM_OK;
    } catch (...) {
        return api_status();
    }
}

long tbem_integral_n_rows(const TbemIntegral* h) { return h ? h->n_rows : TBEM_ERR_ARG; }
long tbem_integral_n_cols(const TbemIntegral* h) { return h ? h->n_cols : TBEM_ERR_ARG; }
void tbem_integral_destroy(TbemIntegral* h) { delete h; }

int tbem_setup_cache_clear(void)
{
    tbem::clear_setup_cache();
    return TBEM_OK;
}

int tbem_fma_peak(int device, int fp64, double* tflops)
{
    using namespace tbem;
    if (!tflops) {
        set_last_error("null output");
        return TBEM_ERR_ARG;
    }
    try {
        *tflops = fp64 ? fma_peak<double>(device) : fma_peak<float>(device);
        return TBEM_OK;
    } catch (...) {
        return api_status();
    }
}

}  // extern "C"
