// passes.cuh -- launches of the density and force passes. Their kernels come in many
// variants (dimension, lanes per particle, CTA size, periodic axes, physics, lists),
// so each pass and dimension is a translation unit of its own (pass_*.cu).
#pragma once
#include <type_traits>

#include "context.cuh"

template <int DIM>
void launch_density(armando_ctx* ctx, const unsigned* skeys, const StepArgs& S);
template <int DIM>
void launch_force(armando_ctx* ctx, const unsigned* skeys, const StepArgs& S);

// Calls f(tpp, block, periodic, lean, opt) with the context's tuning, whether
// any axis is periodic, whether the physics is lean (no physical viscosity, no
// artificial heat, no wall push, no step option) and whether a single_step
// option (continuity or normalised density, XSPH, h evolution) is on, as
// compile-time constants. Lean variants exist for one thread per particle.
template <class F>
void with_tuning(const armando_tuning& t, bool per, bool lean, bool opt, bool lst, F&& f) {
    using std::integral_constant;
    // lists (one lane per particle only) as a compile-time flag, last argument
    auto pick_lst = [&](auto tpp, auto bs, auto pr, auto ln, auto op) {
        if constexpr (decltype(tpp)::value == 1) {
            if (lst) f(tpp, bs, pr, ln, op, std::true_type{});
            else f(tpp, bs, pr, ln, op, std::false_type{});
        } else {
            f(tpp, bs, pr, ln, op, std::false_type{});
        }
    };
    auto pick_lean = [&](auto tpp, auto bs, auto pr) {
        if (opt) pick_lst(tpp, bs, pr, std::false_type{}, std::true_type{});
        else if (decltype(tpp)::value == 1 && lean) pick_lst(tpp, bs, pr, std::true_type{}, std::false_type{});
        else pick_lst(tpp, bs, pr, std::false_type{}, std::false_type{});
    };
    auto pick_per = [&](auto tpp, auto bs) {
        if (per) pick_lean(tpp, bs, std::true_type{});
        else pick_lean(tpp, bs, std::false_type{});
    };
    auto pick_tpp = [&](auto bs) {
        if (t.threads_per_particle == 4) pick_per(integral_constant<int, 4>{}, bs);
        else if (t.threads_per_particle == 2) pick_per(integral_constant<int, 2>{}, bs);
        else pick_per(integral_constant<int, 1>{}, bs);
    };
    if (t.block == 256) pick_tpp(integral_constant<int, 256>{});
    else pick_tpp(integral_constant<int, 128>{});
}
