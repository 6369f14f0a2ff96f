// adjoint.cuh -- reverse mode of one leapfrog step (hand-written adjoint).
//
// The step is the forward of kernels.cuh: predictor, summation density, Tait
// EOS, pressure force + Monaghan artificial viscosity + pressure work, external
// heat, gravity, corrector (CERNsource time_integration.f:131-218 with
// single_step.f, density.f, eos.f90:255-283, internal_force.f pa_sph = 1,
// art_visc.f). Its reverse runs as three gathers over the step's neighbour
// sets (the topology of the step is frozen), with no atomics:
//   k_adj_out      cotangents of the corrector: a_bar, du_bar of every particle
//   k_adj_force    pair adjoints of every (i, j) and (j, i) a particle takes
//                  part in, then the EOS and external-heat adjoints of the
//                  particle: x_bar, vh_bar (predicted velocity), rho_bar
//   k_adj_density  adjoint of the summation density, assembly of the input
//                  cotangents, scatter to the slot order of the step's input
// Non-smooth points follow the value: art_visc acts while v_ij . r_ij < 0,
// u = max(0, .) and the Tait clamp pass no gradient where they bind.
// Artificial heat (art_heat.f:42-97), when on: du_i += sum_j m_j (psi_i + psi_j)
// A_ij (u_i - u_j), A = G r^2 / (rho_bar (r^2 + (eta h_bar)^2)), psi_i =
// g1 h_i c0 + g2 h_i^2 (|divv_i| - divv_i), divv_i = sum_j m_j G_ij (vh_j - vh_i)
// . (x_i - x_j) / rho_i. k_adj_force takes the psi, u_half, rho, x cotangents of
// those pair terms (walls included: their psi enters their neighbours' rates)
// and turns psi_bar into the cotangent of each particle's divergence sum;
// k_adj_density gathers that sum's reverse onto velocities and positions. |divv|
// follows its sign (no gradient at divv = 0 from one side).
// Physical viscosity (internal_force.f:75-171), when on: tau_i = eta/rho_i^2 T_i,
// T_i = sum_j m_j/rho_j H(vh_j - vh_i, G_ij d_ij) (the shear tensor of every
// particle, walls included), a_i += sum_j m_j (tau_i + tau_j) G_ij d_ij, du_i +=
// eta/(2 rho_i) T_i:T_i. k_adj_force takes the tau cotangents of the pair
// forces and turns them, with the heating term's, into cotangents of each
// particle's shear tensor; k_adj_shear gathers the shear sums' reverse onto
// velocities, positions and densities before the density reverse.
// Supported: pa_sph = 1.
#pragma once
#include "kernels.cuh"

namespace ag {

// Cotangents of the carried state (x, v, u, previous a, previous du), in one
// slot order: xb {x_bar, -}, vb {v_bar, u_bar}, ab {a_bar, du_bar}.
struct AdjState {
    float4* xb;
    float4* vb;
    float4* ab;
};

enum AdjParam { ADJ_ALPHA = 0, ADJ_BETA = 1, ADJ_C0 = 2, ADJ_Q0 = 3, ADJ_NPARAM = 4 };

// What the reverse of one iteration reads, saved when the iteration runs
// forward: the cell-order working set, the neighbour structure (sorted keys,
// cell table, grid, the cell slot -> input slot permutation) and the energy
// rate the iteration output. About 116 B per particle in 2D.
struct TapeSlot {
    float4* xh;
    float4* vm;
    float4* vmin;
    float4* rp;
    float* p;
    int* itype;
    unsigned* nmask;  // mask_words<DIM>() words per slot, word-major
    unsigned* keys;
    int* perm;
    float* du;
    int* start;
    DevGrid* grid;
    float* ulo;  // rounding residual of the predicted energy (artificial heat only)
    float4* tau;   // physical viscosity: eta/rho^2 T {xx, yy, xy, zz}
    float4* tau2;  // 3D: {xz, yz, -, -}
};

// The integrated state from one set of arrays to another (checkpoints). One launch;
// a copy an array took eight times 4 us and their gaps at 261 k particles.
static __global__ void k_copy_state(StateA dst, StateA src, int n) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    dst.xh[s] = src.xh[s];
    dst.vm[s] = src.vm[s];
    dst.ap[s] = src.ap[s];
    dst.u[s] = src.u[s];
    dst.rho[s] = src.rho[s];
    dst.p[s] = src.p[s];
    dst.itype[s] = src.itype[s];
    dst.id[s] = src.id[s];
}

template <int DIM>
__global__ void k_tape_save(StateB B, const unsigned* __restrict__ keys,
                            const int* __restrict__ perm, const float4* __restrict__ ap,
                            const int* __restrict__ start, const DevGrid* __restrict__ grid,
                            TapeSlot T, int n) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s == 0) *T.grid = *grid;
    const int nc = grid->ncells;  // the cells in use, not the table's capacity
    for (int c = s; c <= nc; c += gridDim.x * blockDim.x) T.start[c] = start[c];
    if (s >= n) return;
    T.xh[s] = B.xh[s];
    T.vm[s] = B.vm[s];
    T.vmin[s] = B.vmin[s];
    T.rp[s] = B.rp[s];
    T.p[s] = B.p[s];
    T.itype[s] = B.itype[s];
    if (B.mtpp == 1) {  // chunks of 4 words, chunk-major (the lane is the slot)
#pragma unroll
        for (int c = 0; c < mask_words<DIM>() / 4; ++c)
            reinterpret_cast<uint4*>(T.nmask)[(size_t)c * n + s] =
                reinterpret_cast<const uint4*>(B.nmask)[(size_t)c * B.mstride + s];
    }
    T.keys[s] = keys[s];
    T.perm[s] = perm[s];
    T.du[s] = ap[s].w;
    if (T.ulo) T.ulo[s] = B.ulo ? B.ulo[s] : 0.f;
    if (T.tau) T.tau[s] = B.tau[s];
    if (T.tau2) T.tau2[s] = B.tau2[s];
}

// The working set of a taped iteration as the pass kernels see it.
inline StateB tape_view(StateB B, const TapeSlot& T, int n) {
    B.xh = T.xh;
    B.vm = T.vm;
    B.vmin = T.vmin;
    B.rp = T.rp;
    B.p = T.p;
    B.itype = T.itype;
    B.nmask = T.nmask;
    B.mstride = n;
    B.ulo = T.ulo;
    if (T.tau) {
        B.tau = T.tau;
        B.tau2 = T.tau2;
    }
    return B;
}

// Caller-order cotangents -> slot order of the final state (A.id).
template <int DIM>
__global__ void k_adj_load(const int* __restrict__ id, const float* __restrict__ xbar,
                           const float* __restrict__ vbar, const float* __restrict__ ubar,
                           const float* __restrict__ abar, const float* __restrict__ dubar,
                           const float* __restrict__ pbar, AdjState G, float* __restrict__ pbar_s,
                           int n) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    const int i = id[s];
    auto v3 = [&](const float* a) {
        if (!a) return make_float4(0.f, 0.f, 0.f, 0.f);
        return make_float4(a[DIM * i], a[DIM * i + 1], DIM == 3 ? a[DIM * i + 2] : 0.f, 0.f);
    };
    float4 xb = v3(xbar), vb = v3(vbar), ab = v3(abar);
    vb.w = ubar ? ubar[i] : 0.f;
    ab.w = dubar ? dubar[i] : 0.f;
    G.xb[s] = xb;
    G.vb[s] = vb;
    G.ab[s] = ab;
    pbar_s[s] = pbar ? pbar[i] : 0.f;
}

// Slot order (= caller order after the gather of the inputs) -> caller arrays.
template <int DIM>
__global__ void k_adj_store(AdjState G, int n, float* __restrict__ xbar, float* __restrict__ vbar,
                            float* __restrict__ ubar, float* __restrict__ abar,
                            float* __restrict__ dubar) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 xb = G.xb[i], vb = G.vb[i], ab = G.ab[i];
    const float xs[3] = {xb.x, xb.y, xb.z}, vs[3] = {vb.x, vb.y, vb.z}, as[3] = {ab.x, ab.y, ab.z};
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
        if (xbar) xbar[DIM * i + d] = xs[d];
        if (vbar) vbar[DIM * i + d] = vs[d];
        if (abar) abar[DIM * i + d] = as[d];
    }
    if (ubar) ubar[i] = vb.w;
    if (dubar) dubar[i] = ab.w;
}

// Corrector reverse: x' = x + dt v', v' = v + kdt a, u' = max(0, u + kdt du),
// outputs also carry a and du to the next predictor.
static __global__ void k_adj_out(StateB B, const float* __restrict__ du_out, AdjState G, StepArgs S,
                          float4* __restrict__ abar, float4* __restrict__ xpart,
                          float4* __restrict__ vpart, int n) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
    if (B.itype[s] <= 0) {
        abar[s] = z;
        xpart[s] = z;
        vpart[s] = z;
        return;
    }
    const float4 xb = G.xb[s], vb = G.vb[s], ab = G.ab[s];
    const float4 vt = make_float4(fmaf(S.dt, xb.x, vb.x), fmaf(S.dt, xb.y, vb.y),
                                  fmaf(S.dt, xb.z, vb.z), 0.f);
    const float du = du_out[s];
    const bool clamped = fmaf(S.kdt, du, B.vmin[s].w) < 0.f;
    const float ub = clamped ? 0.f : vb.w;
    abar[s] = make_float4(fmaf(S.kdt, vt.x, ab.x), fmaf(S.kdt, vt.y, ab.y), fmaf(S.kdt, vt.z, ab.z),
                          fmaf(S.kdt, ub, ab.w));
    xpart[s] = make_float4(xb.x, xb.y, xb.z, 0.f);
    vpart[s] = make_float4(vt.x, vt.y, vt.z, ub);
}

// Neighbours of a fluid particle in warp-converged rounds (same candidates and
// pair test as the forward passes; 2D reuses the density pass's bit mask).
template <int DIM>
struct NbrStream {
    Cursor cu;
    bool done, from_mask;
    int wi, rbase;
    unsigned wbits;
    uint4 ch;
};

// use_mask: the density pass left this slot's bits (fluid particles); walls
// test their candidates.
template <int DIM>
__device__ __forceinline__ void nbr_init(NbrStream<DIM>& ns, const StateB& B, const DevGrid& g,
                                         int s, bool work, bool use_mask = true) {
    ns.cu = cursor_begin<DIM>(g);
    ns.done = !work;
    ns.from_mask = false;
    ns.wbits = 0u;
    ns.ch = make_uint4(0u, 0u, 0u, 0u);
    // masks of several lanes per particle are not in this layout: test instead
    if (work && use_mask && B.mtpp == 1) {
        ns.ch = mask_load_chunk<mask_words<DIM>()>(B.nmask, B.mstride, s, 0);
        ns.wbits = ns.ch.x;
        ns.from_mask = !(ns.ch.x == ~0u && ns.ch.y == ~0u);
    }
    ns.wi = 0;
    ns.rbase = 0;
}

template <int DIM>
__device__ __forceinline__ int nbr_fill(NbrStream<DIM>& ns, const StateB& B, const DevGrid& g,
                                        const int* __restrict__ start, const CellCoord& cc,
                                        const float4& xi, int s, int (*s_list)[kPassThreads]) {
    const int tid = threadIdx.x;
    int nl = 0;
    if (DIM == 2 && !ns.done && ns.from_mask && ns.wi == 0 && ns.rbase == 0 && ns.cu.ke == 0 &&
        __popc(ns.ch.x) + __popc(ns.ch.y) + __popc(ns.ch.z) + __popc(ns.ch.w) <= kListCap) {
        mask_slots(ns.ch, g, start, cc, [&](const int k, int) { s_list[nl++][tid] = k; });
        ns.done = true;
    }
    while (!ns.done && ns.from_mask) {
        if (nl == kListCap) break;
        while (ns.wbits == 0u && ns.wi < mask_words<DIM>() - 1) {
            ++ns.wi;
            if (ns.wi % 4 == 0)
                ns.ch = mask_load_chunk<mask_words<DIM>()>(B.nmask, B.mstride, s, ns.wi / 4);
            ns.wbits = chunk_word(ns.ch, ns.wi % 4);
        }
        if (ns.wbits == 0u) {
            ns.done = true;
            break;
        }
        const int o = 32 * ns.wi + __ffs(ns.wbits) - 1;
        ns.wbits &= ns.wbits - 1u;
        bool in_rows = true;
        while (o >= ns.rbase + (ns.cu.ke - ns.cu.k)) {
            ns.rbase += ns.cu.ke - ns.cu.k;
            if (!cursor_next<DIM>(g, start, cc, ns.cu)) {
                in_rows = false;
                break;
            }
        }
        if (!in_rows) {
            ns.done = true;
            break;
        }
        s_list[nl++][tid] = ns.cu.k + (o - ns.rbase);
    }
    while (!ns.done && !ns.from_mask) {
        if (ns.cu.k >= ns.cu.ke) {
            if (!cursor_next<DIM>(g, start, cc, ns.cu)) {
                ns.done = true;
                break;
            }
        }
        if (nl == kListCap) break;
        const int k = ns.cu.k++;
        if (k == s) continue;
        float d[3], dr2;
        if (pair_delta<DIM>(xi, __ldg(B.xh + k), g, d, dr2)) s_list[nl++][tid] = k;
    }
    return nl;
}

// Symmetric tensors as stored by the shear pass: a {xx, yy, xy, zz}, b {xz, yz}.
// H(dv, w) is the shear pass's pair term: diagonal (2/3)(2 dv_a w_a - sum of
// the others), off-diagonal dv_a w_b + dv_b w_a. A . H(dv, w) = dv^T M(A) w,
// M(A) symmetric with M_aa = (2/3)(2 A_aa - the other diagonal entries) and
// M_ab = A_ab.
template <int DIM>
__device__ __forceinline__ void sym_apply(const float4& a, const float4& b, const float* x,
                                          float* y) {  // y = S x, S = {a, b}
    y[0] = a.x * x[0] + a.z * x[1];
    y[1] = a.z * x[0] + a.y * x[1];
    y[2] = 0.f;
    if (DIM == 3) {
        y[0] += b.x * x[2];
        y[1] += b.y * x[2];
        y[2] = b.x * x[0] + b.y * x[1] + a.w * x[2];
    }
}

template <int DIM>
__device__ __forceinline__ void shear_m(const float4& a, const float4& b, float4& ma, float4& mb) {
    const float tr = (DIM == 3) ? a.x + a.y + a.w : a.x + a.y;
    // (2/3)(2 A_aa - (tr - A_aa)) = (2/3)(3 A_aa - tr)
    ma = make_float4((2.f / 3.f) * (3.f * a.x - tr), (2.f / 3.f) * (3.f * a.y - tr), a.z,
                     DIM == 3 ? (2.f / 3.f) * (3.f * a.w - tr) : 0.f);
    mb = b;
}

// Forward geometry of two pairs shared by the adjoint gathers: differences, r^2, the
// gradient factor G and G'(r)/r (0 for a coincident pair), h_i + h_j. G < 0 within the
// support; an absent entry is out of reach (kOutOfReach), where both are zero.
template <int DIM>
struct PairGeo2 {
    f2 d[3], dr2, G, dG, hs;
};

template <int DIM>
__device__ __forceinline__ void pair_geo2(const float4& xi, const float4& xa, const float4& xb,
                                          const DevGrid& g, const DevParams& P, PairGeo2<DIM>& o) {
    o.d[0] = make_float2(xi.x - xa.x, xi.x - xb.x);
    o.d[1] = make_float2(xi.y - xa.y, xi.y - xb.y);
    o.d[2] = DIM == 3 ? make_float2(xi.z - xa.z, xi.z - xb.z) : bc2(0.f);
    if (g.periodic[0]) o.d[0] = min_image2(o.d[0], xi.x, xa.x, xb.x, g, 0);
    if (g.periodic[1]) o.d[1] = min_image2(o.d[1], xi.y, xa.y, xb.y, g, 1);
    if (DIM == 3 && g.periodic[2]) o.d[2] = min_image2(o.d[2], xi.z, xa.z, xb.z, g, 2);
    o.dr2 = fma2(o.d[1], o.d[1], fma2(o.d[0], o.d[0], bc2(kTinyDr2)));
    if (DIM == 3) o.dr2 = fma2(o.d[2], o.d[2], o.dr2);
    o.hs = make_float2(xi.w + xa.w, xi.w + xb.w);
    const f2 ih = mul2(bc2(2.0f), rcp2_rn(o.hs, rcp2(o.hs))), ih2 = mul2(ih, ih);
    f2 kg = mul2(bc2(P.kg), mul2(ih2, ih2));
    if (DIM == 3) kg = mul2(kg, ih);
    const f2 rs = rsqrt2(o.dr2);
    const f2 r = sqrt2(o.dr2, rs);
    const f2 t = min2(fma2(r, ih, bc2(-2.0f)), 0.0f);
    const f2 kt = mul2(kg, mul2(t, t));
    o.G = mul2(kt, t);
    o.dG = mul2(mul2(kt, mul2(ih, bc2(3.0f))), rcp2_rn(r, rs));
    if (!(o.dr2.x > 2.0f * kTinyDr2)) o.dG.x = 0.f;
    if (!(o.dr2.y > 2.0f * kTinyDr2)) o.dG.y = 0.f;
}

// EXT: artificial heat or physical viscosity is on; without them their operands are
// compiled out. The pair's two directions share one set of terms, on two neighbours
// at a time, with two estimated reciprocals a pair that every quotient corrects (div2);
// formed apart, with nine divisions each, they took 152 us at 260,904 particles (2D), now
// 62; EXT's operands are what held it to three blocks an SM.
template <int DIM, bool EXT>
__global__ void __launch_bounds__(kPassThreads, EXT ? 3 : 5)
    k_adj_force(StateB B, const unsigned* __restrict__ keys, const int* __restrict__ start,
                const DevGrid* __restrict__ gp, DevParams P, StepArgs S,
                const float4* __restrict__ abar, const float* __restrict__ pbar_loss,
                float* __restrict__ rhobar, float4* __restrict__ xF, float4* __restrict__ vhb,
                float* __restrict__ divsb, float4* __restrict__ tbar, float4* __restrict__ tbar2,
                double* __restrict__ block_part, int n) {
    __shared__ int s_list[kListCap][kPassThreads];
    __shared__ double s_red[ADJ_NPARAM][kPassThreads / 32];
    const int tid = threadIdx.x;
    const int s = blockIdx.x * blockDim.x + tid;
    const bool valid = s < n;
    const DevGrid g = *gp;
    const bool ah = EXT && P.heat_art != 0;
    const bool vs = EXT && P.visc != 0;
    const int it = valid ? B.itype[s] : 0;
    const bool work = valid && g.ok && it > 0;
    // walls take part for artificial heat (their psi enters their neighbours'
    // energy rates) and physical viscosity (their tau, their neighbours' forces)
    const bool act = valid && g.ok && (it > 0 || ah || vs);
    float4 xi = make_float4(0.f, 0.f, 0.f, 1.f), vi = xi, rpi = xi, abi = make_float4(0.f, 0.f, 0.f, 0.f);
    float pi = 0.f, uloi = 0.f;
    if (act) {
        xi = B.xh[s];
        vi = B.vm[s];
        rpi = B.rp[s];
        pi = B.p[s];
        if (work) abi = abar[s];
        if (ah && B.ulo) uloi = B.ulo[s];
    }
    const float mi = mass_of<DIM>(xi, vi);
    CellCoord cc = {{0, 0, 0}};
    if (act) cc = decode_key<DIM>(keys[s], g);
    float4 tai = make_float4(0.f, 0.f, 0.f, 0.f), tbi = tai;  // tau_i
    float4 tba = tai, tbb = tai;                              // tau_bar_i
    if (act && vs) {
        tai = B.tau[s];
        if (DIM == 3) tbi = B.tau2[s];
    }
    const f2 z2 = bc2(0.f);
    f2 xb2[3] = {z2, z2, z2}, vb2[3] = {z2, z2, z2}, Pb2 = z2, rb2 = z2;
    f2 psib2 = z2, uhb2 = z2;  // artificial heat: psi_bar, u_half_bar of this particle
    // Sums of the art_visc parameters' cotangents, float-float (pair terms of both
    // signs cancel): X = sum T_bar phi / rho_bar, Y = sum T_bar phi^2 / rho_bar;
    // alpha_bar = -c0 X, beta_bar = Y, c0_bar gains -alpha X.
    f2 Xh = z2, Xl = z2, Yh = z2, Yl = z2;
    // per-particle terms, float-float (hi in pa, rounding residuals in palo)
    float pa[ADJ_NPARAM] = {0.f, 0.f, 0.f, 0.f}, palo[ADJ_NPARAM] = {0.f, 0.f, 0.f, 0.f};
    auto pacc = [&](int q, float v) {
        const sph::ff t = sph::two_sum(pa[q], v);
        pa[q] = t.hi;
        palo[q] += t.lo;
    };
    NbrStream<DIM> ns;
    nbr_init<DIM>(ns, B, g, s, act, work);
    const int kself = valid ? s : 0;
    while (__any_sync(0xffffffffu, !ns.done)) {
        const int nl = nbr_fill<DIM>(ns, B, g, start, cc, xi, s, s_list);
        const int ml = __reduce_max_sync(0xffffffffu, nl);
        for (int t = 0; t < ml; t += 2) {
            const int ja = t < nl ? s_list[t][tid] : kself, jb = t + 1 < nl ? s_list[t + 1][tid] : kself;
            float4 xa = __ldg(B.xh + ja), xb = __ldg(B.xh + jb);
            if (t >= nl) xa.x = kOutOfReach;
            if (t + 1 >= nl) xb.x = kOutOfReach;
            const float4 va = __ldg(B.vm + ja), vb = __ldg(B.vm + jb);
            const float4 ra = __ldg(B.rp + ja), rb = __ldg(B.rp + jb);
            const float4 ca = __ldg(abar + ja), cb = __ldg(abar + jb);
            const f2 mj = DIM == 2 ? make_float2(xa.z, xb.z) : make_float2(va.w, vb.w);
            PairGeo2<DIM> pg;
            pair_geo2<DIM>(xi, xa, xb, g, P, pg);
            // 2 rho_bar (a particle without density is its own absent entry: not 0)
            const f2 rs = make_float2(pg.G.x < 0.f ? rpi.x + ra.x : 1.f, pg.G.y < 0.f ? rpi.x + rb.x : 1.f);
            const f2 w0 = make_float2(va.x - vi.x, vb.x - vi.x), w1 = make_float2(va.y - vi.y, vb.y - vi.y);
            const f2 w2 = DIM == 3 ? make_float2(va.z - vi.z, vb.z - vi.z) : z2;
            // The rates of s and of j from the pair: with d = x_s - x_j, w = v_j - v_s,
            // T = P_s + P_j + Pi_sj,
            //   a_s -= m_j T G d, du_s -= m_j T G (w.d)/2, a_j += m_s T G d, du_j likewise:
            // their cotangents enter as A = m_j a_bar_s - m_s a_bar_j and
            // b = m_j du_bar_s + m_s du_bar_j, S_bar = -(A.d + b (w.d)/2) on T G.
            f2 A0 = fma2(mj, bc2(abi.x), mul2(bc2(-mi), make_float2(ca.x, cb.x)));
            f2 A1 = fma2(mj, bc2(abi.y), mul2(bc2(-mi), make_float2(ca.y, cb.y)));
            f2 A2 = DIM == 3 ? fma2(mj, bc2(abi.z), mul2(bc2(-mi), make_float2(ca.z, cb.z))) : z2;
            if (work) {
                const f2 hb = mul2(bc2(0.5f), fma2(mj, bc2(abi.w), mul2(bc2(mi), make_float2(ca.w, cb.w))));
                f2 wd = fma2(w1, pg.d[1], mul2(w0, pg.d[0]));
                f2 Ad = fma2(A1, pg.d[1], mul2(A0, pg.d[0]));
                f2 ad = fma2(bc2(abi.y), pg.d[1], mul2(bc2(abi.x), pg.d[0]));
                if (DIM == 3) {
                    wd = fma2(w2, pg.d[2], wd);
                    Ad = fma2(A2, pg.d[2], Ad);
                    ad = fma2(bc2(abi.z), pg.d[2], ad);
                }
                const f2 Sb = neg2(fma2(hb, wd, Ad));
                f2 T = within2(pg.G, make_float2(rpi.y + ra.y, rpi.y + rb.y));
                f2 Tb = mul2(pg.G, Sb), rv = z2, r2b = z2;
                if (P.visc_art) {  // Pi = (beta phi - alpha c0) phi / rho_bar, phi = mh vr / den, vr = -w.d < 0
                    const f2 mh = mul2(pg.hs, bc2(0.5f));
                    const f2 den = fma2(mul2(mh, mh), bc2(P.av_eta2), pg.dr2);
                    const f2 rho = mul2(bc2(0.5f), rs), yd = rcp2(den), yr = rcp2(rho);
                    const f2 phi = div2(mul2(mh, neg2(max2(wd, 0.0f))), den, yd);
                    const f2 pf = div2(phi, rho, yr);
                    const f2 pv = mul2(fma2(bc2(P.av_beta), phi, bc2(-P.av_alpha * P.c0)), pf);
                    T = add2(T, pv);
                    const f2 Tr = div2(Tb, rho, yr);
                    rb2 = fma2(mul2(bc2(-0.5f), Tr), pv, rb2);
                    f2 phib = mul2(Tr, fma2(bc2(2.0f * P.av_beta), phi, bc2(-P.av_alpha * P.c0)));
                    if (!(wd.x > 0.f)) phib.x = 0.f;
                    if (!(wd.y > 0.f)) phib.y = 0.f;
                    const f2 pd = div2(phib, den, yd);
                    rv = mul2(pd, mh);          // vr_bar
                    r2b = mul2(pd, neg2(phi));  // (r^2)_bar
                    // the parameters: the rates of s alone
                    const f2 Ts = mul2(mul2(mj, pg.G), neg2(fma2(bc2(0.5f * abi.w), wd, ad)));
                    const f2 x = mul2(Ts, pf);
                    acc_ff2(Xh, Xl, x);
                    acc_ff2(Yh, Yl, mul2(x, phi));
                }
                const f2 TG = mul2(T, pg.G), c = fma2(mul2(T, Sb), pg.dG, mul2(bc2(2.0f), r2b));
                const f2 e = fma2(TG, hb, rv);  // on w: x_bar -= e w, and v_bar += e d
                const f2 nTG = neg2(TG), ne = neg2(e);
                xb2[0] = fma2(nTG, A0, fma2(ne, w0, fma2(c, pg.d[0], xb2[0])));
                xb2[1] = fma2(nTG, A1, fma2(ne, w1, fma2(c, pg.d[1], xb2[1])));
                vb2[0] = fma2(e, pg.d[0], vb2[0]);
                vb2[1] = fma2(e, pg.d[1], vb2[1]);
                if (DIM == 3) {
                    xb2[2] = fma2(nTG, A2, fma2(ne, w2, fma2(c, pg.d[2], xb2[2])));
                    vb2[2] = fma2(e, pg.d[2], vb2[2]);
                }
                Pb2 = add2(Pb2, Tb);
            }
            if (ah) {
                // du_s and du_j terms m (psi_s + psi_j) A (u_s - u_j), A = G r^2 / (rho_bar
                // (e + r^2)): weights du_bar_s m_j - du_bar_j m_s on the pair (s, j).
                const f2 mh = mul2(pg.hs, bc2(0.5f));
                const f2 den = fma2(mul2(mh, mh), bc2(P.ah_eta2), pg.dr2);
                const f2 rho = mul2(bc2(0.5f), rs);
                const f2 iden = rcp2_rn(den, rcp2(den)), irho = rcp2_rn(rho, rcp2(rho));
                const f2 q = mul2(iden, irho);  // 1 / (rho_bar den)
                const f2 Ah = mul2(mul2(pg.G, pg.dr2), q);
                const f2 dA = fma2(fma2(mul2(bc2(0.5f), pg.dG), pg.dr2, pg.G), q, neg2(mul2(Ah, iden)));
                const f2 ps = within2(pg.G, make_float2(rpi.w + ra.w, rpi.w + rb.w));
                f2 lo = z2;
                if (B.ulo) lo = make_float2(uloi - __ldg(B.ulo + ja), uloi - __ldg(B.ulo + jb));
                const f2 du = add2(make_float2(rpi.z - ra.z, rpi.z - rb.z), lo);
                const f2 cdu = fma2(bc2(abi.w), mj, mul2(bc2(-mi), make_float2(ca.w, cb.w)));
                const f2 Ac = mul2(Ah, cdu);
                psib2 = fma2(Ac, du, psib2);
                uhb2 = fma2(ps, Ac, uhb2);
                rb2 = fma2(mul2(bc2(-0.5f), mul2(ps, Ac)), mul2(du, irho), rb2);
                const f2 cx = mul2(mul2(mul2(bc2(2.0f), dA), mul2(ps, du)), cdu);
#pragma unroll
                for (int k = 0; k < DIM; ++k) xb2[k] = fma2(cx, pg.d[k], xb2[k]);
            }
            if (vs) {
                // a_s += m_j (tau_s + tau_j) w, a_j += m_s (tau_j + tau_s) (-w), w = G d:
                // cotangent A on (tau_s + tau_j) w.
                const float4 ta = __ldg(B.tau + ja), tb = __ldg(B.tau + jb);
                float4 ua = make_float4(0.f, 0.f, 0.f, 0.f), ub = ua;
                if (DIM == 3) {
                    ua = __ldg(B.tau2 + ja);
                    ub = __ldg(B.tau2 + jb);
                }
                const float Av[2][3] = {{A0.x, A1.x, A2.x}, {A0.y, A1.y, A2.y}};
                const float dv[2][3] = {{pg.d[0].x, pg.d[1].x, pg.d[2].x}, {pg.d[0].y, pg.d[1].y, pg.d[2].y}};
                const float Gv[2] = {pg.G.x, pg.G.y}, dGv[2] = {pg.dG.x, pg.dG.y};
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const float4 taj = e ? tb : ta, tbj = e ? ub : ua;
                    const float* bv = Av[e];
                    const float y0 = Gv[e] * dv[e][0], y1 = Gv[e] * dv[e][1], y2 = Gv[e] * dv[e][2];
                    tba.x = fmaf(bv[0], y0, tba.x);
                    tba.y = fmaf(bv[1], y1, tba.y);
                    tba.z += bv[0] * y1 + bv[1] * y0;
                    if (DIM == 3) {
                        tba.w = fmaf(bv[2], y2, tba.w);
                        tbb.x += bv[0] * y2 + bv[2] * y0;
                        tbb.y += bv[1] * y2 + bv[2] * y1;
                    }
                    if (work) {  // d_bar = J u, u = (tau_s + tau_j) b, J = G I + (G'/r) d d^T
                        const float4 sa = make_float4(tai.x + taj.x, tai.y + taj.y, tai.z + taj.z,
                                                      tai.w + taj.w);
                        const float4 sb = make_float4(tbi.x + tbj.x, tbi.y + tbj.y, 0.f, 0.f);
                        float u[3];
                        sym_apply<DIM>(sa, sb, bv, u);
                        float du_ = u[0] * dv[e][0] + u[1] * dv[e][1];
                        if (DIM == 3) du_ += u[2] * dv[e][2];
#pragma unroll
                        for (int k = 0; k < DIM; ++k) xb2[k].x += Gv[e] * u[k] + dGv[e] * du_ * dv[e][k];
                    }
                }
            }
        }
    }
    float xb[3], vb[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        xb[k] = xb2[k].x + xb2[k].y;
        vb[k] = vb2[k].x + vb2[k].y;
    }
    const float Pb = Pb2.x + Pb2.y, psib = psib2.x + psib2.y, uhb = uhb2.x + uhb2.y;
    float rb = rb2.x + rb2.y;
    if (act && vs) {
        // tau = sc T, sc = eta / rho^2; du += tds = eta/(2 rho) T:T (fluid only).
        const float rho = rpi.x;
        const float sc = P.eta / (rho * rho);
        const float isc = P.eta != 0.f ? 1.f / sc : 0.f;
        const float4 Ta = make_float4(tai.x * isc, tai.y * isc, tai.z * isc, tai.w * isc);
        const float4 Tb = make_float4(tbi.x * isc, tbi.y * isc, 0.f, 0.f);
        const float tdsb = work ? abi.w : 0.f;
        const float k = tdsb * P.eta / rho;  // d tds / d T_aa = eta/rho T_aa, off-diagonal 2x
        float4 Ga = make_float4(fmaf(sc, tba.x, k * Ta.x), fmaf(sc, tba.y, k * Ta.y),
                                fmaf(sc, tba.z, 2.f * k * Ta.z), 0.f);
        float4 Gb = make_float4(0.f, 0.f, 0.f, 0.f);
        float q = Ta.x * Ta.x + Ta.y * Ta.y + 2.f * Ta.z * Ta.z;
        float tt = tba.x * tai.x + tba.y * tai.y + tba.z * tai.z;
        if (DIM == 3) {
            Ga.w = fmaf(sc, tba.w, k * Ta.w);
            Gb = make_float4(fmaf(sc, tbb.x, 2.f * k * Tb.x), fmaf(sc, tbb.y, 2.f * k * Tb.y), 0.f,
                             0.f);
            q += Ta.w * Ta.w + 2.f * (Tb.x * Tb.x + Tb.y * Tb.y);
            tt += tba.w * tai.w + tbb.x * tbi.x + tbb.y * tbi.y;
        }
        if (work) rb += -2.f * tt / rho - tdsb * 0.5f * P.eta * q / (rho * rho);
        tbar[s] = Ga;
        if (DIM == 3) tbar2[s] = Gb;
    } else if (valid && vs) {
        tbar[s] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (DIM == 3) tbar2[s] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    float dsb = 0.f;  // cotangent of the divergence sum (artificial heat)
    if (act && ah) {
        // psi = g1 h c0 + g2 h^2 (|divv| - divv), divv = divs / rho: divv from psi
        const float h = xi.w, base = P.ah_g1 * h * P.c0;
        pacc(ADJ_C0, psib * P.ah_g1 * h);
        if (P.ah_g2 != 0.f && rpi.w > base) {  // divv < 0
            const float k2 = 2.f * P.ah_g2 * h * h;
            const float divv = -(rpi.w - base) / k2;
            const float divvb = -k2 * psib;
            dsb = divvb / rpi.x;
            if (work) rb -= divvb * divv / rpi.x;
        }
    }
    if (work) {
        const float rho = rpi.x;
        if (S.heat_on) {  // du += q0 exp(-|x - xc|^2 k) / rho
            const float e0 = xi.x - P.heat_center[0], e1 = xi.y - P.heat_center[1];
            const float e2 = (DIM == 3) ? xi.z - P.heat_center[2] : 0.f;
            const float ex = expf(-(e0 * e0 + e1 * e1 + e2 * e2) * P.heat_k);
            const float dub = abi.w;
            pacc(ADJ_Q0, dub * ex / rho);
            rb -= dub * P.heat_q0 * ex / (rho * rho);
            const float gx = -2.f * P.heat_k * dub * P.heat_q0 * ex / rho;
            xb[0] += gx * e0;
            xb[1] += gx * e1;
            if (DIM == 3) xb[2] += gx * e2;
        }
        // Tait EOS and P = p/rho^2 (the clamp p < pmin sets constants: no gradient).
        const bool clamped = (P.pmin > -FLT_MAX) && pi == 0.f && rho == P.rho0;
        float rtot = 0.f;
        if (!clamped) {
            const float pb = Pb / (rho * rho) + pbar_loss[s];
            const float ratio = rho * P.inv_rho0;
            const float r3 = ratio * ratio * ratio;
            rtot = rb - 2.f * Pb * pi / (rho * rho * rho) + pb * P.c0 * P.c0 * r3 * r3;
            if (P.c0 > 0.f) pacc(ADJ_C0, pb * 2.f * pi / P.c0);
        }
        rhobar[s] = rtot;
        xF[s] = make_float4(xb[0], xb[1], xb[2], 0.f);
        // .w: u_half_bar (the predicted energy of artificial heat)
        vhb[s] = make_float4(vb[0], vb[1], vb[2], ah ? uhb : 0.f);
    } else if (valid) {
        rhobar[s] = 0.f;
        xF[s] = make_float4(0.f, 0.f, 0.f, 0.f);
        vhb[s] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    if (valid && divsb) divsb[s] = dsb;
    // Deterministic per-block partial sums of the parameter cotangents, in
    // double (a fixed shuffle order, then the warps in order).
    const double X = ((double)Xh.x + (double)Xh.y) + ((double)Xl.x + (double)Xl.y);
    const double Y = ((double)Yh.x + (double)Yh.y) + ((double)Yl.x + (double)Yl.y);
#pragma unroll
    for (int q = 0; q < ADJ_NPARAM; ++q) {
        double v = (double)pa[q] + (double)palo[q];
        if (q == ADJ_ALPHA) v -= (double)P.c0 * X;
        if (q == ADJ_BETA) v += Y;
        if (q == ADJ_C0) v -= (double)P.av_alpha * X;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if ((tid & 31) == 0) s_red[q][tid >> 5] = v;
    }
    __syncthreads();
    if (tid < ADJ_NPARAM) {
        double v = 0.0;
        for (int w2 = 0; w2 < kPassThreads / 32; ++w2) v += s_red[tid][w2];
        block_part[blockIdx.x * ADJ_NPARAM + tid] = v;
    }
}

// Shear-tensor reverse (physical viscosity): T_j = sum_k m_k/rho_k H(vh_k - vh_j,
// G_jk d_jk) for every particle j, cotangents tbar. For a fluid particle i the
// pair (i, j) enters T_i (weight m_j/rho_j) and T_j (weight m_i/rho_i, with
// dv and w both reversed: the same H): with Ab = m_j/rho_j tbar_i + m_i/rho_i
// tbar_j, vh_bar_i -= M(Ab) w, x_bar_i += J M(Ab) dv, and rho_i's weight in T_j
// gives rho_bar_i -= m_i/rho_i^2 dv^T M(tbar_j) w. Added to the force reverse's
// cotangents of i (the density's where the Tait clamp did not bind).
template <int DIM>
__global__ void __launch_bounds__(kPassThreads)
    k_adj_shear(StateB B, const unsigned* __restrict__ keys, const int* __restrict__ start,
                const DevGrid* __restrict__ gp, DevParams P, const float4* __restrict__ tbar,
                const float4* __restrict__ tbar2, float* __restrict__ rhobar,
                float4* __restrict__ xF, float4* __restrict__ vhb, int n) {
    __shared__ int s_list[kListCap][kPassThreads];
    const int tid = threadIdx.x;
    const int s = blockIdx.x * blockDim.x + tid;
    const bool valid = s < n;
    const DevGrid g = *gp;
    const bool work = valid && g.ok && B.itype[s] > 0;
    float4 xi = make_float4(0.f, 0.f, 0.f, 1.f), vi = xi;
    float4 tai = make_float4(0.f, 0.f, 0.f, 0.f), tbi = tai;
    float rhoi = 1.f;
    if (work) {
        xi = B.xh[s];
        vi = B.vm[s];
        rhoi = B.rp[s].x;
        tai = tbar[s];
        if (DIM == 3) tbi = tbar2[s];
    }
    const float mi = mass_of<DIM>(xi, vi);
    const float ci = mi / rhoi;
    CellCoord cc = {{0, 0, 0}};
    if (work) cc = decode_key<DIM>(keys[s], g);
    float xb[3] = {0.f, 0.f, 0.f}, vb[3] = {0.f, 0.f, 0.f}, rb = 0.f;
    NbrStream<DIM> ns;
    nbr_init<DIM>(ns, B, g, s, work);
    while (__any_sync(0xffffffffu, !ns.done)) {
        const int nl = nbr_fill<DIM>(ns, B, g, start, cc, xi, s, s_list);
        const int ml = __reduce_max_sync(0xffffffffu, nl);
        for (int t = 0; t < ml; ++t) {
            if (t >= nl) continue;
            const int j = s_list[t][tid];
            const float4 xj = __ldg(B.xh + j);
            const float4 vj = __ldg(B.vm + j);
            const float rhoj = __ldg(&B.rp[j].x);
            const float4 taj = __ldg(tbar + j);
            float4 tbj = make_float4(0.f, 0.f, 0.f, 0.f);
            if (DIM == 3) tbj = __ldg(tbar2 + j);
            const float cj = mass_of<DIM>(xj, vj) / rhoj;
            PairGeo2<DIM> p2;
            pair_geo2<DIM>(xi, xj, xj, g, P, p2);
            struct {
                float d[3], G, dGdr_r;
            } pg = {{p2.d[0].x, p2.d[1].x, p2.d[2].x}, p2.G.x, p2.dG.x};
            const float w[3] = {pg.G * pg.d[0], pg.G * pg.d[1], DIM == 3 ? pg.G * pg.d[2] : 0.f};
            const float dv[3] = {vj.x - vi.x, vj.y - vi.y, DIM == 3 ? vj.z - vi.z : 0.f};
            const float4 Aa = make_float4(cj * tai.x + ci * taj.x, cj * tai.y + ci * taj.y,
                                          cj * tai.z + ci * taj.z, cj * tai.w + ci * taj.w);
            const float4 Ab = make_float4(cj * tbi.x + ci * tbj.x, cj * tbi.y + ci * tbj.y, 0.f, 0.f);
            float4 ma, mb;
            shear_m<DIM>(Aa, Ab, ma, mb);
            float mw[3], mdv[3];
            sym_apply<DIM>(ma, mb, w, mw);
            sym_apply<DIM>(ma, mb, dv, mdv);
            float dmd = mdv[0] * pg.d[0] + mdv[1] * pg.d[1];
            if (DIM == 3) dmd += mdv[2] * pg.d[2];
#pragma unroll
            for (int k = 0; k < DIM; ++k) {
                vb[k] -= mw[k];
                xb[k] += pg.G * mdv[k] + pg.dGdr_r * dmd * pg.d[k];
            }
            float4 mja, mjb;
            shear_m<DIM>(taj, tbj, mja, mjb);
            float mjw[3];
            sym_apply<DIM>(mja, mjb, w, mjw);
            float h = dv[0] * mjw[0] + dv[1] * mjw[1];
            if (DIM == 3) h += dv[2] * mjw[2];
            rb -= mi / (rhoi * rhoi) * h;
        }
    }
    if (!work) return;
    // the Tait clamp (p < pmin) set rho_i = rho0: no gradient reaches the sum
    const bool clamped = (P.pmin > -FLT_MAX) && B.p[s] == 0.f && rhoi == P.rho0;
    if (!clamped) rhobar[s] += rb;
    float4 f = xF[s];
    f.x += xb[0];
    f.y += xb[1];
    f.z += xb[2];
    xF[s] = f;
    float4 v = vhb[s];
    v.x += vb[0];
    v.y += vb[1];
    v.z += vb[2];
    vhb[s] = v;
}

// Density reverse (rho_i = m_i W(0) + sum m_j W_ij), the reverse of the
// divergence sums of artificial heat (divs_i = sum_j m_j G_ij (vh_j - vh_i) .
// d_ij, cotangents divsb), assembly, scatter to the slot order of the step's
// input (perm: cell slot -> input slot).
template <int DIM>
__global__ void __launch_bounds__(kPassThreads)
    k_adj_density(StateB B, const unsigned* __restrict__ keys, const int* __restrict__ start,
                  const DevGrid* __restrict__ gp, DevParams P, StepArgs S,
                  const float* __restrict__ rhobar, const float4* __restrict__ xF,
                  const float4* __restrict__ vhb, const float4* __restrict__ xpart,
                  const float4* __restrict__ vpart, const float* __restrict__ divsb,
                  const int* __restrict__ perm, AdjState Gp, int n) {
    __shared__ int s_list[kListCap][kPassThreads];
    const int tid = threadIdx.x;
    const int s = blockIdx.x * blockDim.x + tid;
    const bool valid = s < n;
    const DevGrid g = *gp;
    const bool work = valid && g.ok && B.itype[s] > 0;
    float4 xi = make_float4(0.f, 0.f, 0.f, 1.f), vi = xi;
    float rbi = 0.f;
    if (work) {
        xi = B.xh[s];
        vi = B.vm[s];
        rbi = rhobar[s];
    }
    const float mi = mass_of<DIM>(xi, vi);
    CellCoord cc = {{0, 0, 0}};
    if (work) cc = decode_key<DIM>(keys[s], g);
    const bool ah = P.heat_art != 0 && divsb != nullptr;
    const float dsi = (work && ah) ? divsb[s] : 0.f;
    const f2 z2 = bc2(0.f);
    f2 xb2[3] = {z2, z2, z2}, vd2[3] = {z2, z2, z2};
    NbrStream<DIM> ns;
    nbr_init<DIM>(ns, B, g, s, work);
    const int kself = valid ? s : 0;
    while (__any_sync(0xffffffffu, !ns.done)) {
        const int nl = nbr_fill<DIM>(ns, B, g, start, cc, xi, s, s_list);
        const int ml = __reduce_max_sync(0xffffffffu, nl);
        for (int t = 0; t < ml; t += 2) {
            const int ja = t < nl ? s_list[t][tid] : kself, jb = t + 1 < nl ? s_list[t + 1][tid] : kself;
            float4 xa = __ldg(B.xh + ja), xb = __ldg(B.xh + jb);
            if (t >= nl) xa.x = kOutOfReach;
            if (t + 1 >= nl) xb.x = kOutOfReach;
            float4 va = make_float4(0.f, 0.f, 0.f, 0.f), vb = va;
            if (DIM == 3 || ah) {
                va = __ldg(B.vm + ja);
                vb = __ldg(B.vm + jb);
            }
            const f2 mj = DIM == 2 ? make_float2(xa.z, xb.z) : make_float2(va.w, vb.w);
            PairGeo2<DIM> pg;
            pair_geo2<DIM>(xi, xa, xb, g, P, pg);
            const f2 wr = fma2(bc2(rbi), mj, mul2(bc2(mi), make_float2(__ldg(rhobar + ja), __ldg(rhobar + jb))));
            const f2 c = mul2(within2(pg.G, wr), pg.G);
#pragma unroll
            for (int k = 0; k < DIM; ++k) xb2[k] = fma2(c, pg.d[k], xb2[k]);
            if (ah) {
                // d/d(vh_s), d/d(x_s) of divs_s (weight dsb_s m_j) and of divs_j
                // (weight dsb_j m_s, d_js = -d, w_js = -w): the same forms.
                const f2 cd = within2(
                    pg.G, fma2(bc2(dsi), mj, mul2(bc2(mi), make_float2(__ldg(divsb + ja), __ldg(divsb + jb)))));
                const f2 w[3] = {make_float2(va.x - vi.x, vb.x - vi.x), make_float2(va.y - vi.y, vb.y - vi.y),
                                 DIM == 3 ? make_float2(va.z - vi.z, vb.z - vi.z) : z2};
                f2 wd = fma2(w[1], pg.d[1], mul2(w[0], pg.d[0]));
                if (DIM == 3) wd = fma2(w[2], pg.d[2], wd);
                const f2 cg = mul2(cd, pg.G), ce = mul2(cd, mul2(pg.dG, wd));
#pragma unroll
                for (int k = 0; k < DIM; ++k) {
                    vd2[k] = fma2(neg2(cg), pg.d[k], vd2[k]);
                    xb2[k] = fma2(cg, w[k], fma2(ce, pg.d[k], xb2[k]));
                }
            }
        }
    }
    float xb[3], vdb[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        xb[k] = xb2[k].x + xb2[k].y;
        vdb[k] = vd2[k].x + vd2[k].y;
    }
    if (!valid) return;
    float4 gx = make_float4(0.f, 0.f, 0.f, 0.f), gv = gx, ga = gx;
    if (work) {
        const float4 xp = xpart[s], f = xF[s], vp = vpart[s];
        float4 vh = vhb[s];
        vh.x += vdb[0];
        vh.y += vdb[1];
        vh.z += vdb[2];
        // u_half = max(0, u + hdt du_prev): no gradient where it clamped to 0
        const float uh = (ah && B.rp[s].z != 0.f) ? vh.w : 0.f;
        gx = make_float4(xp.x + f.x + xb[0], xp.y + f.y + xb[1], xp.z + f.z + xb[2], 0.f);
        // predictor: vh = v + hdt a_prev (v_bar gets vh_bar; a_prev_bar = hdt vh_bar)
        gv = make_float4(vp.x + vh.x, vp.y + vh.y, vp.z + vh.z, vp.w + uh);
        ga = make_float4(S.hdt * vh.x, S.hdt * vh.y, S.hdt * vh.z, S.hdt * uh);
    }
    const int j = perm[s];
    Gp.xb[j] = gx;
    Gp.vb[j] = gv;
    Gp.ab[j] = ga;
}

// Adds the step's parameter cotangents (block partials, fixed order) to acc.
static __global__ void __launch_bounds__(256)
    k_adj_params(const double* __restrict__ block_part, int nblocks, double* __restrict__ acc) {
    __shared__ double s[ADJ_NPARAM][256];
    for (int q = 0; q < ADJ_NPARAM; ++q) {
        double v = 0.0;
        for (int b = threadIdx.x; b < nblocks; b += blockDim.x) v += block_part[b * ADJ_NPARAM + q];
        s[q][threadIdx.x] = v;
    }
    __syncthreads();
    for (int st = blockDim.x / 2; st > 0; st >>= 1) {
        if ((int)threadIdx.x < st)
            for (int q = 0; q < ADJ_NPARAM; ++q) s[q][threadIdx.x] += s[q][threadIdx.x + st];
        __syncthreads();
    }
    if (threadIdx.x < ADJ_NPARAM) acc[threadIdx.x] += s[threadIdx.x][0];
}

}  // namespace ag
