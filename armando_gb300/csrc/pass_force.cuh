// pass_force.cuh -- launch_force (declared in passes.cuh).
#pragma once
#include "passes.cuh"
#include "staged.cuh"

template <int DIM, int BS>
void launch_force_staged(armando_ctx* ctx, const unsigned* skeys, const StepArgs& S) {
    const int n = (int)ctx->n_work;
    const int reach = ctx->tune.reach;
    const int cap = stage_cap(DIM, reach, BS, true);
    const int bytes = stage_smem_bytes(DIM, reach, BS, true);
    cudaFuncSetAttribute(k_force_st<DIM, BS>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    k_force_st<DIM, BS><<<blocks_for(n, BS), BS, bytes, ctx->stream>>>(
        ctx->B, ctx->A, skeys, ctx->start, ctx->grid, ctx->dp, S, ctx->flags, n, cap);
}

template <int DIM>
void launch_force(armando_ctx* ctx, const unsigned* skeys, const StepArgs& S) {
    const int n = (int)ctx->n_work;
    const bool fuse = fused(ctx);
    const FusedSrc F{ctx->A, fuse ? resort_flags(ctx) : nullptr, S.hdt};
    if (staged_passes(ctx)) {
        if (ctx->tune.block == 256) launch_force_staged<DIM, 256>(ctx, skeys, S);
        else launch_force_staged<DIM, 128>(ctx, skeys, S);
        return;
    }
    with_tuning(ctx->tune, any_periodic(ctx->dp), lean_physics(ctx->dp), step_options(ctx->prm),
                use_lists(ctx), [&](auto tpp, auto bs, auto per, auto lean, auto opt, auto lst) {
        constexpr int T = decltype(tpp)::value, BSZ = decltype(bs)::value;
        constexpr bool PER = decltype(per)::value, LEAN = decltype(lean)::value && T == 1;
        constexpr bool OPT = decltype(opt)::value, LST = decltype(lst)::value;
        constexpr bool FUS_OK = LST && LEAN && !OPT;
        const int grid = blocks_for((int64_t)n * T, BSZ);
        if constexpr (FUS_OK) {
            if (fuse) {  // the next state into the other buffer
                k_force<DIM, T, BSZ, PER, LEAN, OPT, LST, true><<<grid, BSZ, 0, ctx->stream>>>(
                    ctx->B, ctx->A_alt, skeys, ctx->start, ctx->grid, ctx->dp, S, ctx->flags, n, F);
                return;
            }
        }
        k_force<DIM, T, BSZ, PER, LEAN, OPT, LST><<<grid, BSZ, 0, ctx->stream>>>(
            ctx->B, ctx->A, skeys, ctx->start, ctx->grid, ctx->dp, S, ctx->flags, n, F);
    });
}
