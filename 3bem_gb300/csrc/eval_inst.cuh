// Instantiates the evaluation kernels of one kernel id (EVAL_KID); with
// EVAL_FP64_ONLY (the 2D kernels, which have the plain FP64 form only) the
// FP32 variants are not built and asking for them is an error.
#include "eval_launch.h"

namespace tbem {

namespace {
template <typename T, bool TR, bool TS, bool SS, int TPT>
void go_tpt(const EvalLaunch& L, int nr, int n_items, const EvalArgs<T>& a, cudaStream_t s)
{
    if (nr == 1) {
        eval_kernel<EVAL_KID, TR, T, 1, TS, SS, TPT><<<n_items, EVAL_THREADS, 0, s>>>(a);
        return;
    }
    if constexpr (sizeof(T) == 4 && kernel_dim(EVAL_KID) == 1 && kernel_space_dim(EVAL_KID) == 3 &&
                  !TR && !SS && TPT != EVAL_PER_ITEM) {
        if (nr == EVAL_NR_WIDE) {
            auto kern = L.wide_shared ? eval_wide_kernel<EVAL_KID, TS, TPT, EVAL_NR_WIDE, true>
                                      : eval_wide_kernel<EVAL_KID, TS, TPT, EVAL_NR_WIDE, false>;
            kern<<<n_items, EVAL_THREADS / 2, 0, s>>>(a);
            return;
        }
    }
    eval_kernel<EVAL_KID, TR, T, EVAL_NR, TS, SS, TPT><<<n_items, EVAL_THREADS, 0, s>>>(a);
}

template <typename T, bool TR, bool TS, bool SS>
cudaError_t go(const EvalLaunch& L, int nr, int tpt, const void* args, cudaStream_t s)
{
    const int n_items = L.n_items;
    const EvalArgs<T>& a = *static_cast<const EvalArgs<T>*>(args);
    if (n_items <= 0) return cudaSuccess;
    // the FP64 point-to-point passes take it per item (their pace is the FP64
    // pipe's: the shifts cost nothing); the FP32 point-to-point pass (2, 4, 8)
    // and the points-to-check-surface pass (1, 2, 4) have autotuned variants;
    // every other pass uses 4
    if constexpr (sizeof(T) == 8 && !TS && !SS) {
        if (tpt == EVAL_PER_ITEM) go_tpt<T, TR, TS, SS, EVAL_PER_ITEM>(L, nr, n_items, a, s);
        else return cudaErrorInvalidValue;
    } else if constexpr (!TR && !TS && !SS) {
        if (tpt == 2) go_tpt<T, TR, TS, SS, 2>(L, nr, n_items, a, s);
        else if (tpt == 8) go_tpt<T, TR, TS, SS, 8>(L, nr, n_items, a, s);
        else go_tpt<T, TR, TS, SS, 4>(L, nr, n_items, a, s);
    } else if constexpr (!TR && TS && !SS) {
        if (tpt == 1) go_tpt<T, TR, TS, SS, 1>(L, nr, n_items, a, s);
        else if (tpt == 2) go_tpt<T, TR, TS, SS, 2>(L, nr, n_items, a, s);
        else go_tpt<T, TR, TS, SS, 4>(L, nr, n_items, a, s);
    } else {
        go_tpt<T, TR, TS, SS, 4>(L, nr, n_items, a, s);
    }
    return cudaGetLastError();
}

template <typename T>
cudaError_t go_t(const EvalLaunch& L, const void* args, cudaStream_t s)
{
    const EvalArgs<T>& a = *static_cast<const EvalArgs<T>*>(args);
    const int nr = eval_rhs_block(L, sizeof(T) == 4, a.nrhs - a.rhs0);
    const int idx = (L.trans ? 4 : 0) + (L.tgt_surf ? 2 : 0) + (L.src_surf ? 1 : 0);
    switch (idx) {
    case 0: return go<T, false, false, false>(L, nr, L.tpt, args, s);
    case 1: return go<T, false, false, true>(L, nr, 4, args, s);
    case 2: return go<T, false, true, false>(L, nr, L.tpt, args, s);
    case 3: return go<T, false, true, true>(L, nr, 4, args, s);
    case 4: return go<T, true, false, false>(L, nr, L.tpt, args, s);
    case 5: return go<T, true, false, true>(L, nr, 4, args, s);
    case 6: return go<T, true, true, false>(L, nr, 4, args, s);
    default: return go<T, true, true, true>(L, nr, 4, args, s);
    }
}
}  // namespace

#define TBEM_CAT2(a, b) a##b
#define TBEM_CAT(a, b) TBEM_CAT2(a, b)
cudaError_t TBEM_CAT(launch_eval_k, EVAL_KID)(const EvalLaunch& L, const void* args, bool fp32,
                                              cudaStream_t s)
{
#ifdef EVAL_FP64_ONLY
    if (fp32) return cudaErrorInvalidValue;
    return go_t<double>(L, args, s);
#else
    return fp32 ? go_t<float>(L, args, s) : go_t<double>(L, args, s);
#endif
}

}  // namespace tbem
