// Host-side launcher of the obs-owner evaluation kernels (eval.cuh).
#pragma once
#include <cuda_runtime.h>
#include "eval.cuh"

namespace tbem {

struct EvalLaunch {
    int kid;
    bool trans;
    bool tgt_surf;
    bool src_surf;
    int n_items;
    int tpt = 4;  // threads per target (point-to-point: EVAL_PER_ITEM in FP64, 2, 4 or 8 in FP32;
                  // 1, 2 or 4 for points to a check surface; 4 otherwise)
    bool wide_shared = false;  // many right-hand sides: the sums in shared memory
};

// One function per kernel id (eval_k<id>.cu) so that the instantiations
// compile in parallel.
cudaError_t launch_eval_k0(const EvalLaunch&, const void* args, bool fp32, cudaStream_t);
cudaError_t launch_eval_k1(const EvalLaunch&, const void* args, bool fp32, cudaStream_t);
cudaError_t launch_eval_k2(const EvalLaunch&, const void* args, bool fp32, cudaStream_t);
cudaError_t launch_eval_k3(const EvalLaunch&, const void* args, bool fp32, cudaStream_t);
cudaError_t launch_eval_k4(const EvalLaunch&, const void* args, bool fp32, cudaStream_t);
cudaError_t launch_eval_k5(const EvalLaunch&, const void* args, bool fp32, cudaStream_t);
cudaError_t launch_eval_k6(const EvalLaunch&, const void* args, bool fp32, cudaStream_t);
// 2D kernels (FP64 only)
cudaError_t launch_eval_k16(const EvalLaunch&, const void* args, bool fp32, cudaStream_t);
cudaError_t launch_eval_k17(const EvalLaunch&, const void* args, bool fp32, cudaStream_t);
cudaError_t launch_eval_k18(const EvalLaunch&, const void* args, bool fp32, cudaStream_t);
cudaError_t launch_eval_k19(const EvalLaunch&, const void* args, bool fp32, cudaStream_t);
cudaError_t launch_eval_k20(const EvalLaunch&, const void* args, bool fp32, cudaStream_t);
cudaError_t launch_eval_k21(const EvalLaunch&, const void* args, bool fp32, cudaStream_t);
cudaError_t launch_eval_k22(const EvalLaunch&, const void* args, bool fp32, cudaStream_t);
cudaError_t launch_eval_k23(const EvalLaunch&, const void* args, bool fp32, cudaStream_t);

// rhs chunk per launch (the kernel keeps NR x R accumulators per thread)
constexpr int EVAL_NR = 4;
// FP32 scalar kernels with point sources, not transposed: 16 right-hand
// sides per launch (the kernel value is shared by all of them)
constexpr int EVAL_NR_WIDE = 16;

// Right-hand sides one launch of the evaluation kernel handles when
// `remaining` are left from the launch's first one.
inline int eval_rhs_block(const EvalLaunch& L, bool fp32, int remaining)
{
    if (remaining <= 1) return 1;
    if (fp32 && kernel_dim(L.kid) == 1 && kernel_space_dim(L.kid) == 3 && !L.trans && !L.src_surf &&
        remaining >= EVAL_NR_WIDE)
        return EVAL_NR_WIDE;
    return EVAL_NR;
}

// Whether an operator's passes of many right-hand sides (both of them) keep
// their sums in shared memory, from the CTAs of its point-to-point pass and
// that pass's threads per target.  What it buys is occupancy, so small batches
// lose: with fewer CTAs than fit anyway the shared accesses only cost, and with
// eight threads per target a thread has 16 pairs per tile to set against them,
// of which the single layer's are a third of the double layer's work.  Batches
// of 3 to 16 spheres, 16 to 64 right-hand sides (registers / shared, us; CTAs
// per SM): double layer 972 / 1125 (2.6), 1277 / 1283 (4.4), 1320 / 1258 (4.8),
// 1826 / 1603 (6.6), 12204 / 10799 (26); single layer with eight threads 662 /
// 749 (2.6), 922 / 942 (6.6), 2042 / 2281 (9.7), with four 1365 / 1412 (7.5),
// 1903 / 1686 (9.7), 3332 / 3603 (10.2), 4824 / 4644 (15), 7661 / 7505 (26).
inline bool wide_shared(int kid, int p2p_items, int p2p_tpt)
{
    if (kid == LAP_D) return p2p_items >= 700;
    return p2p_tpt <= 4 && p2p_items >= 9 * 152;
}

// SMs of the current device (152 where there is none to ask: argument checks
// come before any launch).
inline int sm_count()
{
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) == cudaSuccess &&
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && sms > 0)
        return sms;
    cudaGetLastError();
    return 152;
}

// Threads per target of the direct sum, 8, 16 or 32, one number for all its
// CTAs of EVAL_THREADS / tpt targets.  Every target sees all sources, so the
// pass lasts as long as the SM with most targets, ceil(CTAs / SMs) * targets
// per CTA, times what staging the sources adds per pair: a CTA stages each
// source once for its targets, about 1/512 of the pair work per thread per
// target.  Few points need many threads for an even share, where shares are
// even anyway fewer threads stage less.  Measured (4 / 8 / 16 / 32 threads,
// us): single layer, 4,705 points 886 / 867 / 879 / 897, 4,900 points 1449 /
// 1174 / 1044 / 1005, 12,000 points 4480 / 3831 / 3886 / 4013; traction, 3,457
// points 1545 / 1541 / 1247 / 1279, 6,145 points 4656 / 3601 / 3635 / 3440.  Over
// 46 sizes, kernels and counts of right-hand sides the rule's choice is within
// 4 % of the best.
inline int direct_tpt(long n_obs, int sms)
{
    int best = 8;
    double least = 1e300;
    for (int tpt : {8, 16, 32}) {
        const long targets = EVAL_THREADS / tpt, ctas = (n_obs + targets - 1) / targets;
        const double cost = (double)((ctas + sms - 1) / sms * targets) * (1.0 + tpt / 512.0);
        if (cost < least) {
            least = cost;
            best = tpt;
        }
    }
    return best;
}

template <typename T>
inline cudaError_t launch_eval(const EvalLaunch& L, const EvalArgs<T>& a, cudaStream_t s)
{
    const bool fp32 = sizeof(T) == 4;
    switch (L.kid) {
    case 0: return launch_eval_k0(L, &a, fp32, s);
    case 1: return launch_eval_k1(L, &a, fp32, s);
    case 2: return launch_eval_k2(L, &a, fp32, s);
    case 3: return launch_eval_k3(L, &a, fp32, s);
    case 4: return launch_eval_k4(L, &a, fp32, s);
    case 5: return launch_eval_k5(L, &a, fp32, s);
    case 6: return launch_eval_k6(L, &a, fp32, s);
    case 16: return launch_eval_k16(L, &a, fp32, s);
    case 17: return launch_eval_k17(L, &a, fp32, s);
    case 18: return launch_eval_k18(L, &a, fp32, s);
    case 19: return launch_eval_k19(L, &a, fp32, s);
    case 20: return launch_eval_k20(L, &a, fp32, s);
    case 21: return launch_eval_k21(L, &a, fp32, s);
    case 22: return launch_eval_k22(L, &a, fp32, s);
    case 23: return launch_eval_k23(L, &a, fp32, s);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace tbem
