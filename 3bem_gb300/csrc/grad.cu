// Kernel-gradient pass: derivatives of  L = r^T A x,  A_ij = w_j K(x_i, y_j; n_i, n_j),
// with respect to every point position, normal and weight, and to x (the
// direct operator's transpose apply), in FP64.
//
// The contraction c = rho^T K(d; no, ns) chi of every kernel is a rational
// function of d, its length and a few dot products, so its derivatives in the
// separation d = y - x (d/dy = d/dd, d/dx = -d/dd) and in the normals are
// written out (grad_pair) in the powers of 1 / |d| that the value needs
// anyway.  The direct passes each own their outputs (no atomics): a
// source-owner pass (gradients of y_j, n_j, w_j and x_j) and an
// observation-owner pass (gradients of x_i and n_i), O(N M) sums.
#include <string>
#include <type_traits>

#include "plan.h"

namespace tbem {
namespace {

// Which derivatives of one pair are wanted besides the value.
enum GradNormal { GN_NONE = 0, GN_SRC = 1, GN_OBS = 2 };

// The normal a kernel's value depends on, as seen from one side: the normals'
// derivatives are taken at the target of the pass only.
__host__ __device__ constexpr bool grad_src_normal(int kid) { return kid == LAP_D || kid == EL_TRAC || kid == EL_HYP; }
__host__ __device__ constexpr bool grad_obs_normal(int kid) { return kid == EL_ADJ || kid == EL_HYP; }

__device__ __forceinline__ double dot3(const double* a, const double* b)
{
    return a[0] * b[0] + a[1] * b[1] + a[2] * b[2];
}

// c = rho^T K(d; m, n) chi without the kernel's leading constant (m the
// observation normal, n the source normal), its gradient gd in d and gn in
// the source (WN = GN_SRC) or observation (GN_OBS) normal, by the formulas of
// kernels.cuh:
//   displacement  c = q (c2 rho.chi + a b q^2),  q = 1 / |d|, a = rho.d, b = chi.d
//   traction / adjoint traction, w their normal, g = w.d, s = -1 / +1:
//     c = s q^3 (c2 rho.chi g + 3 a b g q^2 + s c2 (w.chi a - w.rho b))
//   hypersingular, h = n.d, g = m.d:
//     c = q^3 C0 + 3 q^5 Q - 15 q^7 a b g h
// Zero for the self pair.
template <int KID, int WN>
__device__ __forceinline__ void grad_pair(const double* d, const double* m, const double* n, const double* rho,
                                          const double* chi, double c2, double& c, double* gd, double* gn)
{
    c = 0;
#pragma unroll
    for (int k = 0; k < 3; k++) gd[k] = gn[k] = 0;
    const double r2 = dot3(d, d);
    if (r2 < 1e-12) return;
    if constexpr (KID == IDENT) {
        c = rho[0] * chi[0];
        return;
    }
    const double q = rsqrt(r2), q2 = q * q, q3 = q2 * q;
    if constexpr (KID == LAP_S) {
        c = rho[0] * chi[0] * q;
        const double f = -c * q2;
#pragma unroll
        for (int k = 0; k < 3; k++) gd[k] = f * d[k];
    } else if constexpr (KID == LAP_D) {
        const double f = rho[0] * chi[0] * q3;
        c = f * dot3(n, d);
        const double e = -3.0 * c * q2;
#pragma unroll
        for (int k = 0; k < 3; k++) {
            gd[k] = f * n[k] + e * d[k];
            if (WN == GN_SRC) gn[k] = f * d[k];
        }
    } else if constexpr (KID == EL_DISP) {
        const double a = dot3(rho, d), b = dot3(chi, d), P = c2 * dot3(rho, chi);
        const double t = a * b * q2;
        c = q * (P + t);
        const double e = -q3 * (P + 3.0 * t), fa = q3 * a, fb = q3 * b;
#pragma unroll
        for (int k = 0; k < 3; k++) gd[k] = e * d[k] + fb * rho[k] + fa * chi[k];
    } else if constexpr (KID == EL_TRAC || KID == EL_ADJ) {
        const double sg = KID == EL_TRAC ? -1.0 : 1.0;
        const double* w = KID == EL_TRAC ? n : m;
        const double a = dot3(rho, d), b = dot3(chi, d), g = dot3(w, d);
        const double wc = sg * c2 * dot3(w, chi), wr = sg * c2 * dot3(w, rho);
        const double P = c2 * dot3(rho, chi), t = 3.0 * a * b * q2;
        const double f = sg * q3;
        const double u = P + t;
        const double N = u * g + wc * a - wr * b;
        c = f * N;
        const double g3 = 3.0 * g * q2;
        const double er = f * (g3 * b + wc), ec = f * (g3 * a - wr), ew = f * u;
        const double ed = -f * q2 * (3.0 * N + 2.0 * t * g);
#pragma unroll
        for (int k = 0; k < 3; k++) {
            gd[k] = er * rho[k] + ec * chi[k] + ew * w[k] + ed * d[k];
            if (WN != GN_NONE) gn[k] = f * (u * d[k] + sg * c2 * (a * chi[k] - b * rho[k]));
        }
    } else {
        const double nu = 0.5 * (1.0 - c2), c4 = 4.0 * nu - 1.0;
        const double a = dot3(rho, d), b = dot3(chi, d), g = dot3(m, d), h = dot3(n, d);
        const double rm = dot3(rho, m), rn = dot3(rho, n), xm = dot3(chi, m), xn = dot3(chi, n);
        const double rx = dot3(rho, chi), nm = dot3(n, m);
        const double C0 = c2 * (rx * nm + rn * xm) + c4 * xn * rm;
        const double Q = c2 * (rm * b * h + xn * a * g) + nu * (xm * a * h + rx * g * h + rn * b * g + nm * a * b);
        const double q5 = q3 * q2, q7 = q5 * q2, ab = a * b, gh = g * h;
        c = q3 * C0 + 3.0 * q5 * Q - 15.0 * q7 * ab * gh;
        const double ed = -3.0 * q5 * C0 - 15.0 * q7 * Q + 105.0 * q7 * q2 * ab * gh;
        const double er = 3.0 * q5 * (nu * (xm * h + nm * b) + c2 * xn * g) - 15.0 * q7 * b * gh;
        const double ec = 3.0 * q5 * (nu * (rn * g + nm * a) + c2 * rm * h) - 15.0 * q7 * a * gh;
        const double em = 3.0 * q5 * (nu * (rx * h + rn * b) + c2 * xn * a) - 15.0 * q7 * ab * h;
        const double en = 3.0 * q5 * (nu * (xm * a + rx * g) + c2 * rm * b) - 15.0 * q7 * ab * g;
#pragma unroll
        for (int k = 0; k < 3; k++) {
            gd[k] = ed * d[k] + er * rho[k] + ec * chi[k] + em * m[k] + en * n[k];
            if (WN == GN_SRC)
                gn[k] = q3 * (c2 * (rx * m[k] + xm * rho[k]) + c4 * rm * chi[k]) + en * d[k] +
                        3.0 * q5 * (c2 * a * g * chi[k] + nu * (b * g * rho[k] + ab * m[k]));
            if (WN == GN_OBS)
                gn[k] = q3 * (c2 * (rx * n[k] + rn * chi[k]) + c4 * xn * rho[k]) + em * d[k] +
                        3.0 * q5 * (c2 * b * h * rho[k] + nu * (a * h * chi[k] + ab * n[k]));
        }
    }
}

// Source owner: g_y, g_ns, g_w, g_x (= A^T r) for source j.
template <int KID>
__global__ void grad_src_kernel(KParams p, const double* ox, const double* on, long n_obs,
                                const double* sx, const double* sn, const double* sw, long n_src,
                                const double* x, const double* r, double* g_y, double* g_ns,
                                double* g_w, double* g_x)
{
    const long j = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n_src) return;
    constexpr int R = kernel_dim(KID);
    double xv[3] = {0, 0, 0};
    for (int b = 0; b < R; b++) xv[b] = x[b * n_src + j];
    const double y[3] = {sx[3 * j], sx[3 * j + 1], sx[3 * j + 2]};
    const double nsj[3] = {sn[3 * j], sn[3 * j + 1], sn[3 * j + 2]};
    double gy[3] = {0, 0, 0}, gn[3] = {0, 0, 0}, gw = 0, gx[3] = {0, 0, 0};
    for (long i = 0; i < n_obs; i++) {
        const double d[3] = {y[0] - ox[3 * i], y[1] - ox[3 * i + 1], y[2] - ox[3 * i + 2]};
        const double noi[3] = {on[3 * i], on[3 * i + 1], on[3 * i + 2]};
        double rv[3] = {0, 0, 0};
        for (int a = 0; a < R; a++) rv[a] = r[a * n_obs + i];
        double c, gd[3], g2[3];
        grad_pair<KID, grad_src_normal(KID) ? GN_SRC : GN_NONE>(d, noi, nsj, rv, xv, p.c2, c, gd, g2);
        gw += c;
        for (int k = 0; k < 3; k++) {
            gy[k] += gd[k];
            gn[k] += g2[k];
        }
        accumulate<KID, true, double>(d[0], d[1], d[2], noi[0], noi[1], noi[2], nsj[0], nsj[1], nsj[2], p.c2, rv, gx);
    }
    const double w = sw[j] * p.scale;
    for (int k = 0; k < 3; k++) {
        if (g_y) g_y[3 * j + k] = w * gy[k];
        if (g_ns) g_ns[3 * j + k] = w * gn[k];
    }
    if (g_w) g_w[j] = p.scale * gw;
    if (g_x)
        for (int b = 0; b < R; b++) g_x[b * n_src + j] = w * gx[b];
}

// Observation owner: g_x_obs (= -dL/dd summed) and g_no for observer i.
template <int KID>
__global__ void grad_obs_kernel(KParams p, const double* ox, const double* on, long n_obs,
                                const double* sx, const double* sn, const double* sw, long n_src,
                                const double* x, const double* r, double* g_o, double* g_no)
{
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_obs) return;
    constexpr int R = kernel_dim(KID);
    double rv[3] = {0, 0, 0};
    for (int a = 0; a < R; a++) rv[a] = r[a * n_obs + i];
    const double o[3] = {ox[3 * i], ox[3 * i + 1], ox[3 * i + 2]};
    const double noi[3] = {on[3 * i], on[3 * i + 1], on[3 * i + 2]};
    double go[3] = {0, 0, 0}, gn[3] = {0, 0, 0};
    for (long j = 0; j < n_src; j++) {
        const double d[3] = {sx[3 * j] - o[0], sx[3 * j + 1] - o[1], sx[3 * j + 2] - o[2]};
        const double nsj[3] = {sn[3 * j], sn[3 * j + 1], sn[3 * j + 2]};
        double xv[3] = {0, 0, 0};
        for (int b = 0; b < R; b++) xv[b] = sw[j] * x[b * n_src + j];
        double c, gd[3], g2[3];
        grad_pair<KID, grad_obs_normal(KID) ? GN_OBS : GN_NONE>(d, noi, nsj, rv, xv, p.c2, c, gd, g2);
        for (int k = 0; k < 3; k++) {
            go[k] -= gd[k];
            gn[k] += g2[k];
        }
    }
    for (int k = 0; k < 3; k++) {
        if (g_o) g_o[3 * i + k] = p.scale * go[k];
        if (g_no) g_no[3 * i + k] = p.scale * gn[k];
    }
}

// f(std::integral_constant<int, KID>) for a 3D kernel id
template <typename F>
void with_kernel(int kid, F&& f)
{
    switch (kid) {
    case LAP_S: f(std::integral_constant<int, LAP_S>()); break;
    case LAP_D: f(std::integral_constant<int, LAP_D>()); break;
    case EL_DISP: f(std::integral_constant<int, EL_DISP>()); break;
    case EL_TRAC: f(std::integral_constant<int, EL_TRAC>()); break;
    case EL_ADJ: f(std::integral_constant<int, EL_ADJ>()); break;
    case EL_HYP: f(std::integral_constant<int, EL_HYP>()); break;
    case IDENT: f(std::integral_constant<int, IDENT>()); break;
    default: throw Error(TBEM_ERR_ARG, "gradients take the 3D kernels");
    }
}

// Source-side gradients through the FMM's transposed passes.  For every
// source point j (a target here) and every source z of one transposed pass
// -- an observation point with density r (P2P^T), or a point of a check
// surface with the transposed state as its density (P2M^T, P2L^T) -- the
// contraction c = v(z)^T K(y_j - z; n_z, n_j) x_j, its gradient in y_j and
// (kernels with a source normal) in n_j are summed; the sums of c are
// dL/dw_j.  The pass is paced by the FP64 pipe (two FMAs per SM and clock, 40
// to 110 of them per pair), so what matters is that every SM has pairs: the
// task sets' work items are cut into CTAs of one warp per target, whose lanes
// split its sources and meet in shuffles, or one target for the longest lists.  With one CTA of four threads per target per item and
// forward-mode dual numbers through the kernel tensors, the four passes of
// 6,144 sources and 4,096 observers took 28.4 ms in 107 to 182 CTAs; now 2.3 ms.
struct GradEvalArgs {
    const int* item_task;
    const int* item_start;
    const int* item_tpt;   // log2 of the item's threads per target
    const long* task_tgt;
    const int* task_tgt_count;
    const int* task_src_ptr;
    const long* src_blk;
    const int* src_blk_count;
    const double* t_xyz;   // source points, tree order [n][3]
    const double* t_nrm;
    const double* t_x;     // their densities x, tree order [R][t_n]
    long t_n;
    const double* s_xyz;   // point sources (observation points, tree order)
    const double* s_nrm;
    const double* s_v;     // their densities r [R][s_n]
    long s_n;
    const double* s_center;  // surface sources: cell centres, radii, the unit sphere
    const double* s_rad;
    double s_rref;
    const double* unit;
    int ns;
    const float* q32;      // surface densities [cell][R ns] (one right-hand side)
    const double* q64;
    int kid;
    KParams kp;
    // 0: the targets are the operator's source points (contraction v^T K x_j,
    // derivatives in y_j and n_j); 1: its observation points (r_i^T K v,
    // derivatives in x_i and the observation normal n_i)
    int obs_side;
    double* g;             // [t_n][7]: d/dposition (3), d/dnormal (3), value (1); accumulated
};
constexpr int GRAD_THREADS = 128, GRAD_WARPS = GRAD_THREADS / 32;
static_assert(GRAD_THREADS == EVAL_LONG, "a long item is one target");

template <int KID, bool OBS_SIDE, bool SRC_SURF>
__global__ void __launch_bounds__(GRAD_THREADS) grad_eval_kernel(const GradEvalArgs a)
{
    constexpr int R = kernel_dim(KID);
    constexpr int WN = OBS_SIDE ? (grad_obs_normal(KID) ? GN_OBS : GN_NONE) : (grad_src_normal(KID) ? GN_SRC : GN_NONE);
    constexpr bool NORMALS = normal_dot_kernel(KID);  // the kernel's value depends on a normal
    const int task = a.item_task[blockIdx.x];
    const int tpt = 1 << a.item_tpt[blockIdx.x];  // 32 or GRAD_THREADS
    const int ti = a.item_start[blockIdx.x] + (int)threadIdx.x / tpt;
    const int lane = threadIdx.x % tpt;
    const bool active = ti < a.task_tgt_count[task];
    double acc[7] = {0, 0, 0, 0, 0, 0, 0};
    if (active) {
        const long j = a.task_tgt[task] + ti;
        const double y[3] = {a.t_xyz[3 * j], a.t_xyz[3 * j + 1], a.t_xyz[3 * j + 2]};
        double nj[3] = {0, 0, 0};
        if (NORMALS)
            for (int k = 0; k < 3; k++) nj[k] = a.t_nrm[3 * j + k];
        double xv[3] = {0, 0, 0};
#pragma unroll
        for (int b = 0; b < R; b++) xv[b] = a.t_x[b * a.t_n + j];
        for (int blk = a.task_src_ptr[task]; blk < a.task_src_ptr[task + 1]; blk++) {
            const long sb = a.src_blk[blk];
            const int cnt = a.src_blk_count[blk];
            // a surface's points are c + t u: y - z = (y - c) - t u
            double yc[3] = {0, 0, 0}, t = 0;
            if (SRC_SURF) {
                t = a.s_rad[sb] * a.s_rref;
#pragma unroll
                for (int k = 0; k < 3; k++) yc[k] = y[k] - a.s_center[3 * sb + k];
            }
            for (int li = lane; li < cnt; li += tpt) {
                double dd[3], nz[3] = {0, 0, 0}, rv[3] = {0, 0, 0};
                if (SRC_SURF) {
#pragma unroll
                    for (int k = 0; k < 3; k++) {
                        const double u = a.unit[3 * li + k];
                        dd[k] = fma(-t, u, yc[k]);
                        if (NORMALS) nz[k] = u;
                    }
                    const long base = sb * (long)(R * a.ns) + li;
#pragma unroll
                    for (int d = 0; d < R; d++)
                        rv[d] = a.q32 ? (double)a.q32[base + d * a.ns] : a.q64[base + d * a.ns];
                } else {
                    const long p = sb + li;
#pragma unroll
                    for (int k = 0; k < 3; k++) {
                        dd[k] = y[k] - a.s_xyz[3 * p + k];
                        if (NORMALS) nz[k] = a.s_nrm[3 * p + k];
                    }
#pragma unroll
                    for (int d = 0; d < R; d++) rv[d] = a.s_v[d * a.s_n + p];
                }
                double c, gd[3], gn[3];
                if (!OBS_SIDE) {
                    // forward separation y_j - z, the target the source side
                    grad_pair<KID, WN>(dd, nz, nj, rv, xv, a.kp.c2, c, gd, gn);
                    acc[6] += c;
#pragma unroll
                    for (int k = 0; k < 3; k++) acc[k] += gd[k];
                } else {
                    // forward separation z - x_i: d/dx_i = -d/dd
                    const double df[3] = {-dd[0], -dd[1], -dd[2]};
                    grad_pair<KID, WN>(df, nj, nz, xv, rv, a.kp.c2, c, gd, gn);
#pragma unroll
                    for (int k = 0; k < 3; k++) acc[k] -= gd[k];
                }
                if (WN != GN_NONE) {
#pragma unroll
                    for (int k = 0; k < 3; k++) acc[3 + k] += gn[k];
                }
            }
        }
    }
#pragma unroll
    for (int off = 16; off > 0; off /= 2)
#pragma unroll
        for (int i = 0; i < 7; i++) acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], off);
    if (tpt > 32) {  // one target per CTA: the warps' sums in warp order
        __shared__ double red[GRAD_WARPS][7];
        if (threadIdx.x % 32 == 0)
            for (int i = 0; i < 7; i++) red[threadIdx.x / 32][i] = acc[i];
        __syncthreads();
        if (threadIdx.x == 0)
            for (int w = 1; w < GRAD_WARPS; w++)
                for (int i = 0; i < 7; i++) acc[i] += red[w][i];
    }
    if (!active || lane != 0) return;
    double* g = a.g + 7 * (a.task_tgt[task] + ti);
#pragma unroll
    for (int i = 0; i < 7; i++) g[i] += a.kp.scale * acc[i];
}

// Tree order [n][7] -> the caller's order: g_y = w dL/dy, g_n = w dL/dn,
// g_w = the value sum (any output may be null; w null: no weight).
__global__ void grad_scatter_kernel(const double* g7, const long* perm, const double* w, long n,
                                    double* g_y, double* g_n, double* g_w)
{
    for (long j = (long)blockIdx.x * blockDim.x + threadIdx.x; j < n; j += (long)gridDim.x * blockDim.x) {
        const long o = perm[j];
        const double wj = w ? w[j] : 1.0;
        for (int k = 0; k < 3; k++) {
            if (g_y) g_y[3 * o + k] = wj * g7[7 * j + k];
            if (g_n) g_n[3 * o + k] = wj * g7[7 * j + 3 + k];
        }
        if (g_w) g_w[o] = g7[7 * j + 6];
    }
}

bool dev_ptr(const void* p)
{
    cudaPointerAttributes a{};
    bool d = p && cudaPointerGetAttributes(&a, p) == cudaSuccess &&
             (a.type == cudaMemoryTypeDevice || a.type == cudaMemoryTypeManaged);
    cudaGetLastError();
    return d;
}

struct In {
    DBuf<double> own;
    const double* p = nullptr;
    void stage(const double* h, size_t n, cudaStream_t s)
    {
        if (!n) return;
        if (dev_ptr(h)) { p = h; return; }
        own.alloc(n);
        TBEM_CK(cudaMemcpyAsync(own.p, h, n * sizeof(double), cudaMemcpyHostToDevice, s));
        p = own.p;
    }
};

struct Out {
    DBuf<double> own;
    double* user = nullptr;
    double* p = nullptr;
    size_t n = 0;
    void stage(double* h, size_t count)
    {
        user = h;
        n = count;
        if (!h || !count) return;
        if (dev_ptr(h)) { p = h; return; }
        own.alloc(count);
        p = own.p;
    }
    void finish(cudaStream_t s)
    {
        if (user && p && p != user)
            TBEM_CK(cudaMemcpyAsync(user, p, n * sizeof(double), cudaMemcpyDeviceToHost, s));
    }
};

// One transposed pass of the source gradients over a task set.
void grad_pass(const TaskSet& ts, bool src_surf, GradEvalArgs a, cudaStream_t s, long* launches)
{
    if (ts.empty()) return;
    a.task_tgt = ts.d_tgt;
    a.task_tgt_count = ts.d_tgt_count;
    a.task_src_ptr = ts.d_src_ptr;
    a.src_blk = ts.d_blk;
    a.src_blk_count = ts.d_blk_count;
    const TaskSet::Items& it = ts.cuts.at(TaskSet::SPLIT + 32);
    a.item_task = it.task;
    a.item_start = it.start;
    a.item_tpt = it.tpt_log;
    with_kernel(a.kid, [&](auto K) {
        constexpr int kid = decltype(K)::value;
        if (a.obs_side) {
            if (src_surf) grad_eval_kernel<kid, true, true><<<it.n, GRAD_THREADS, 0, s>>>(a);
            else grad_eval_kernel<kid, true, false><<<it.n, GRAD_THREADS, 0, s>>>(a);
        } else {
            if (src_surf) grad_eval_kernel<kid, false, true><<<it.n, GRAD_THREADS, 0, s>>>(a);
            else grad_eval_kernel<kid, false, false><<<it.n, GRAD_THREADS, 0, s>>>(a);
        }
    });
    TBEM_CK(cudaGetLastError());
    if (launches) (*launches)++;
}

// [R][n] in the caller's order -> tree order, times w (tree order) when given
__global__ void gather_rows_kernel(const double* x, const long* perm, double* out, long n, int R,
                                   const double* w = nullptr)
{
    for (long t = (long)blockIdx.x * blockDim.x + threadIdx.x; t < n * R; t += (long)gridDim.x * blockDim.x) {
        const long i = t % n, d = t / n;
        out[t] = w ? w[i] * x[d * n + perm[i]] : x[d * n + perm[i]];
    }
}

__global__ void widen_kernel(const float* in, double* out, long n)
{
    for (long t = (long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long)gridDim.x * blockDim.x)
        out[t] = (double)in[t];
}

unsigned blocks_for(long n) { return (unsigned)std::max<long>(1, std::min<long>((n + 255) / 256, 152L * 32)); }

}  // namespace

// The transposed apply of r leaves the transposed states of the source
// leaves' up-check surfaces (cu) and of the P2L cells' down-check surfaces
// (cd) in the work buffers; the three passes that reach source points
// (P2P^T, P2M^T, P2L^T) are then run again with the kernel's derivatives.
// The compressed forms only: their transposed states are check potentials
// on fixed surfaces, so every dependence on a source point's position and
// normal sits in these three passes.
void Plan::source_gradients(const double* x, const double* r, double* g_y, double* g_n,
                            double* g_w, cudaStream_t s)
{
    if (opt.host_only) throw Error(TBEM_ERR_STATE, "operator was built with host_only");
    if (sdim != 3) throw Error(TBEM_ERR_ARG, "source gradients take the 3D kernels");
    if (!batch_off.empty())
        throw Error(TBEM_ERR_STATE, "source gradients are not defined for the batched form "
                                    "(its meshes are rescaled by their own bounding boxes)");
    if (!(f.mixed && f.m2l_compressed) || f.m2l_on_the_fly)
        throw Error(TBEM_ERR_STATE, "source gradients need a compressed form (the precision or "
                                    "FP64 compressed form with compressible M2L operators)");
    if (!x || !r) throw Error(TBEM_ERR_ARG, "null input");
    DeviceGuard guard(opt.device);
    if (!s) s = stream;
    const long NS = n_src, NO = n_obs;
    if (NS == 0) return;
    // the work arrays: tree-order gradients [NS][7], x in tree order, r in
    // tree order, the transposed apply's output, the caller-order outputs
    const size_t off_x = 7 * (size_t)NS, off_r = off_x + R * (size_t)NS,
                 off_o = off_r + R * (size_t)std::max<long>(NO, 1), off_u = off_o + R * (size_t)NS,
                 total = off_u + 7 * (size_t)NS;
    grad_buf.ensure(total);
    double* g7 = grad_buf.p;
    double* xt = grad_buf.p + off_x;
    double* rt = grad_buf.p + off_r;
    double* out = grad_buf.p + off_o;
    double* gu = grad_buf.p + off_u;
    apply(r, out, 1, s, true);  // r is at x_dev now, the transposed states in cu / cd
    // x to the device (io_y is free after the apply), then both to tree order
    TBEM_CK(cudaMemcpyAsync(io_y.p, x, sizeof(double) * R * NS, cudaMemcpyDefault, s));
    gather_rows_kernel<<<blocks_for(NS * R), 256, 0, s>>>(io_y.p, dsrc->perm.p, xt, NS, R);
    TBEM_CK(cudaGetLastError());
    if (NO > 0) {
        gather_rows_kernel<<<blocks_for(NO * R), 256, 0, s>>>(x_dev, dobs.perm.p, rt, NO, R);
        TBEM_CK(cudaGetLastError());
    }
    TBEM_CK(cudaMemsetAsync(g7, 0, sizeof(double) * 7 * NS, s));
    GradEvalArgs a{};
    a.t_xyz = dsrc->xyz.p;
    a.t_nrm = dsrc->nrm64.p;
    a.t_x = xt;
    a.t_n = NS;
    a.unit = d_unit.p;
    a.ns = ns;
    a.g = g7;
    // P2P^T: the observation points with the densities r
    a.kid = kid;
    a.kp = make_kparams(kid, mu, nu);
    a.s_xyz = dobs.xyz.p;
    a.s_nrm = dobs.nrm64.p;
    a.s_v = rt;
    a.s_n = NO;
    grad_pass(p2p_t, false, a, s, &launches);
    // P2M^T and P2L^T: check surfaces with the transposed states
    a.kid = f.ks_kid;
    a.kp = make_kparams(f.ks_kid, mu, nu);
    a.q32 = f.f64 ? nullptr : cu32.p;
    a.q64 = f.f64 ? cu64.p : nullptr;
    a.s_center = dsrc->center.p;
    a.s_rad = dsrc->rad.p;
    a.s_rref = f.r_uc;
    grad_pass(p2m_t, true, a, s, &launches);
    if (!L.p2l.empty()) {
        a.q32 = f.f64 ? nullptr : cd32.p;
        a.q64 = f.f64 ? cd64.p : nullptr;
        a.s_center = dobs.center.p;
        a.s_rad = dobs.rad.p;
        a.s_rref = f.r_dc;
        grad_pass(p2l_t, true, a, s, &launches);
    }
    // to the caller's order (device scratch, then wherever the caller's arrays are)
    grad_scatter_kernel<<<blocks_for(NS), 256, 0, s>>>(g7, dsrc->perm.p, dsrc->w.p, NS, gu, gu + 3 * NS,
                                                       gu + 6 * NS);
    TBEM_CK(cudaGetLastError());
    if (g_y) TBEM_CK(cudaMemcpyAsync(g_y, gu, sizeof(double) * 3 * NS, cudaMemcpyDefault, s));
    if (g_n) TBEM_CK(cudaMemcpyAsync(g_n, gu + 3 * NS, sizeof(double) * 3 * NS, cudaMemcpyDefault, s));
    if (g_w) TBEM_CK(cudaMemcpyAsync(g_w, gu + 6 * NS, sizeof(double) * NS, cudaMemcpyDefault, s));
    check_tc_flags(true, s);
}

// The forward apply of x leaves the downward coefficients of every cell
// (cdc) and the M2P sources' equivalent densities in the work buffers.  The
// passes that reach observation points -- P2P (the source points with
// densities w x), M2P (those densities on the sources' up-equivalent
// surfaces) and L2P (the leaves' down-equivalent densities, rebuilt here as
// C2E_down(level) V cdc, the product the leaf operators E V fold in) -- are
// run again with the kernel's derivatives in the observation point and its
// normal.  Compressed forms only, as for the source side.
void Plan::observation_gradients(const double* x, const double* r, double* g_x, double* g_n,
                                 cudaStream_t s)
{
    if (opt.host_only) throw Error(TBEM_ERR_STATE, "operator was built with host_only");
    if (sdim != 3) throw Error(TBEM_ERR_ARG, "observation gradients take the 3D kernels");
    if (!batch_off.empty())
        throw Error(TBEM_ERR_STATE, "observation gradients are not defined for the batched form "
                                    "(its meshes are rescaled by their own bounding boxes)");
    if (!(f.mixed && f.m2l_compressed) || f.m2l_on_the_fly)
        throw Error(TBEM_ERR_STATE, "observation gradients need a compressed form (the precision "
                                    "or FP64 compressed form with compressible M2L operators)");
    if (!x || !r) throw Error(TBEM_ERR_ARG, "null input");
    DeviceGuard guard(opt.device);
    if (!s) s = stream;
    const long NS = n_src, NO = n_obs;
    if (NO == 0) return;
    const Tree& O = otree;
    const long nco = (long)O.cells.size();
    // work arrays: tree-order gradients [NO][7], r and w x in tree order, the
    // forward output, the caller-order outputs, the leaves' down-check
    // potentials and down-equivalent densities (FP64, [cell][n])
    const size_t off_r = 7 * (size_t)NO, off_x = off_r + R * (size_t)NO,
                 off_o = off_x + R * (size_t)std::max<long>(NS, 1), off_u = off_o + R * (size_t)NO,
                 off_c = off_u + 6 * (size_t)NO, off_q = off_c + (size_t)nco * n,
                 total = off_q + (size_t)nco * n;
    grad_buf.ensure(total);
    double* g7 = grad_buf.p;
    double* rt = grad_buf.p + off_r;
    double* xt = grad_buf.p + off_x;
    double* out = grad_buf.p + off_o;
    double* gu = grad_buf.p + off_u;
    double* uck = grad_buf.p + off_c;
    double* qdn = grad_buf.p + off_q;
    apply(x, out, 1, s, false);  // x is at x_dev now, the states in cdc / the M2P buffers
    TBEM_CK(cudaMemcpyAsync(io_y.p, r, sizeof(double) * R * NO, cudaMemcpyDefault, s));
    gather_rows_kernel<<<blocks_for(NO * R), 256, 0, s>>>(io_y.p, dobs.perm.p, rt, NO, R);
    TBEM_CK(cudaGetLastError());
    if (NS > 0) {
        gather_rows_kernel<<<blocks_for(NS * R), 256, 0, s>>>(x_dev, dsrc->perm.p, xt, NS, R, dsrc->w.p);
        TBEM_CK(cudaGetLastError());
    }
    // down-check potentials of the L2P leaves (V cdc), then their
    // down-equivalent densities C2E_down(level) u, level by level in FP64
    TBEM_CK(cudaMemsetAsync(uck, 0, sizeof(double) * nco * n, s));
    if (f.f64) {
        f.decomp_l2p.run_rect<double>(cdc64.p, uck, n, f.r_out, f.r_out, 1, 0, GEMM_STORE, s, &launches);
    } else {
        TBEM_CK(cudaMemsetAsync(cd32.p, 0, sizeof(float) * nco * n, s));
        f.decomp_l2p.run_rect<float>(cdc32.p, cd32.p, n, f.r_out, f.r_out, 1, 0, GEMM_STORE, s, &launches);
        widen_kernel<<<blocks_for(nco * n), 256, 0, s>>>(cd32.p, uck, nco * n);
        TBEM_CK(cudaGetLastError());
    }
    for (int l = 0; l < O.n_levels() && l < (int)f.c2e_l2p.size(); l++)
        f.c2e_l2p[l].run<double>(uck, qdn, n, 1, 0, GEMM_STORE, s, &launches);
    TBEM_CK(cudaMemsetAsync(g7, 0, sizeof(double) * 7 * NO, s));
    GradEvalArgs a{};
    a.obs_side = 1;
    a.t_xyz = dobs.xyz.p;
    a.t_nrm = dobs.nrm64.p;
    a.t_x = rt;
    a.t_n = NO;
    a.unit = d_unit.p;
    a.ns = ns;
    a.g = g7;
    // P2P: the source points with densities w x
    a.kid = kid;
    a.kp = make_kparams(kid, mu, nu);
    a.s_xyz = dsrc->xyz.p;
    a.s_nrm = dsrc->nrm64.p;
    a.s_v = xt;
    a.s_n = NS;
    grad_pass(p2p, false, a, s, &launches);
    // M2P and L2P: equivalent surfaces, the kernel that reaches the targets
    a.kid = f.kt_kid;
    a.kp = make_kparams(f.kt_kid, mu, nu);
    if (!L.m2p.empty()) {
        a.q32 = nullptr;
        a.q64 = f.f64 ? cu64.p : qu64.p;
        a.s_center = dsrc->center.p;
        a.s_rad = dsrc->rad.p;
        a.s_rref = f.r_ue;
        grad_pass(m2p, true, a, s, &launches);
    }
    a.q32 = nullptr;
    a.q64 = qdn;
    a.s_center = dobs.center.p;
    a.s_rad = dobs.rad.p;
    a.s_rref = f.r_de;
    grad_pass(l2p, true, a, s, &launches);
    grad_scatter_kernel<<<blocks_for(NO), 256, 0, s>>>(g7, dobs.perm.p, nullptr, NO, gu, gu + 3 * NO,
                                                       nullptr);
    TBEM_CK(cudaGetLastError());
    if (g_x) TBEM_CK(cudaMemcpyAsync(g_x, gu, sizeof(double) * 3 * NO, cudaMemcpyDefault, s));
    if (g_n) TBEM_CK(cudaMemcpyAsync(g_n, gu + 3 * NO, sizeof(double) * 3 * NO, cudaMemcpyDefault, s));
    check_tc_flags(true, s);
}

}  // namespace tbem

extern "C" int tbem_direct_gradients(int kernel, const double* kernel_params,
                                     const double* obs_locs, const double* obs_normals, long n_obs,
                                     const double* src_locs, const double* src_normals,
                                     const double* src_weights, long n_src, const double* x,
                                     const double* r, double* g_obs_locs, double* g_obs_normals,
                                     double* g_src_locs, double* g_src_normals,
                                     double* g_src_weights, double* g_x, void* stream)
{
    using namespace tbem;
    try {
        if (kernel < 0 || kernel > 6 || n_obs < 0 || n_src < 0) throw Error(TBEM_ERR_ARG, "bad argument");
        const int R = kernel_dim(kernel);
        const double mu = (kernel_params && R == 3) ? kernel_params[0] : 1.0;
        const double nu = (kernel_params && R == 3) ? kernel_params[1] : 0.25;
        const KParams kp = make_kparams(kernel, mu, nu);
        cudaStream_t s = (cudaStream_t)stream;
        In ol, on, sl, sn, sw, xs, rs;
        ol.stage(obs_locs, 3 * n_obs, s);
        on.stage(obs_normals, 3 * n_obs, s);
        sl.stage(src_locs, 3 * n_src, s);
        sn.stage(src_normals, 3 * n_src, s);
        sw.stage(src_weights, n_src, s);
        xs.stage(x, (size_t)R * n_src, s);
        rs.stage(r, (size_t)R * n_obs, s);
        Out go, gno, gs, gns, gw, gx;
        go.stage(g_obs_locs, 3 * n_obs);
        gno.stage(g_obs_normals, 3 * n_obs);
        gs.stage(g_src_locs, 3 * n_src);
        gns.stage(g_src_normals, 3 * n_src);
        gw.stage(g_src_weights, n_src);
        gx.stage(g_x, (size_t)R * n_src);
        if (n_src > 0 && (gs.p || gns.p || gw.p || gx.p)) {
            if (n_obs == 0) {
                for (Out* o : {&gs, &gns, &gw, &gx})
                    if (o->p) TBEM_CK(cudaMemsetAsync(o->p, 0, o->n * sizeof(double), s));
            } else {
                with_kernel(kernel, [&](auto K) {
                    grad_src_kernel<decltype(K)::value><<<(unsigned)((n_src + 127) / 128), 128, 0, s>>>(
                        kp, ol.p, on.p, n_obs, sl.p, sn.p, sw.p, n_src, xs.p, rs.p, gs.p, gns.p, gw.p, gx.p);
                });
                TBEM_CK(cudaGetLastError());
            }
        }
        if (n_obs > 0 && (go.p || gno.p)) {
            if (n_src == 0) {
                for (Out* o : {&go, &gno})
                    if (o->p) TBEM_CK(cudaMemsetAsync(o->p, 0, o->n * sizeof(double), s));
            } else {
                with_kernel(kernel, [&](auto K) {
                    grad_obs_kernel<decltype(K)::value><<<(unsigned)((n_obs + 127) / 128), 128, 0, s>>>(
                        kp, ol.p, on.p, n_obs, sl.p, sn.p, sw.p, n_src, xs.p, rs.p, go.p, gno.p);
                });
                TBEM_CK(cudaGetLastError());
            }
        }
        for (Out* o : {&go, &gno, &gs, &gns, &gw, &gx}) o->finish(s);
        TBEM_CK(cudaStreamSynchronize(s));
        return TBEM_OK;
    } catch (...) {
        return tbem::api_status();
    }
}
