// gpuc.cuh -- the GPU-C step variant (armando_params.scheme 1 and 2).
//
// Third-order TVD Runge-Kutta with continuity density and one neighbour list
// per step, as the GPU-C codes run it (ArmandoThrust/acpu.c:2338-2379):
// X = X0 + alpha (X + dt dX/dt - X0) for alpha = 1, 1/4, 2/3. Pair rates:
//   scheme 1, the host path (acpu.c:346-437): every listed pair contributes
//     continuity m_j (x_ij . v_ij) W'/r, pressure -(p_i + p_j)/(rho_i rho_j),
//     the shock corrections of mass and momentum, and between different
//     itype a push 0.02 (W/W0) c_i c_j / r scaled by m_j/(m_i + m_j);
//   scheme 2, the device kernels (armando.cu:429-513): the same terms, with
//     pressure -(p_i/rho_i^2 + p_j/rho_j^2), for pairs of equal itype only;
//     pairs of different itype push 0.5 W m_j/(rho_j h_j) c_j^2.
// Energy: de/dt = p drho/dt / rho^2 (acpu.c:510-534); gravity and the load
// zones on itype > 0 (acpu.c:1047-1076); fix zones after the update.
// Update and EOS per material |itype| (acpu.c:873-966, armando.cu:987-1074).
// Kernels with h_i. The list of a step holds the j != i with
// sqrtf(|x0_i - x0_j|^2) < 2 h_i at the step's start (updateListHost,
// acpu.c:2201-2240), without the reference's 21-entry cap; each stage tests
// the candidates of the step's cell grid against the start positions (kept
// for the step anyway) and evaluates the physics at the stage's positions.
//
// State in cell order: the step's start (x0, v0, rho0/u0) and two working copies
// that the stages ping-pong between, laid out so that a pair reads two float4s of
// its neighbour in 2D and three in 3D; the last stage's rates go out as dv/dt, de/dt.
#pragma once
#include "kernels.cuh"

namespace ag {

struct DevMaterial {
    int type;  // 0 boundary, 1 ideal gas, 2 polynomial, 3 shock, 4 Tait, 5 ESS
    float prop[10];
};

// Load and fix zones (acpu.c:33-48; armando.cu:43-58): open boxes lo < x < hi,
// x and y only in 2D (armando2D.cu:756-762).
struct DevLoadZone {
    float lo[3], hi[3], g[3], w;
};
struct DevFixZone {
    float lo[3], hi[3], v[3];
    float tau;  // 0: fix zone (velocity set after the update); > 0: pump zone (a rate)
};
struct DevZones {
    int n_load, n_fix;
    DevLoadZone load[10];
    DevFixZone fix[10];
};

template <int DIM>
__device__ __forceinline__ bool in_zone(const float* lo, const float* hi, const float4& x) {
    bool in = x.x > __ldg(lo) && x.x < __ldg(hi) && x.y > __ldg(lo + 1) && x.y < __ldg(hi + 1);
    if (DIM == 3) in = in && x.z > __ldg(lo + 2) && x.z < __ldg(hi + 2);
    return in;
}

struct GpucState {
    float4* x0;    // {x, y, m, h} (2D) / {x, y, z, h} (3D) at the step's start
    float4* v0;    // {v, -} (2D) / {v, m} (3D)
    float2* q0;    // {rho, u} at the step's start
    // Working copies, 2D: w0 {x, y, vx, vy}, w1 {rho, p, m, itype's bits}, w2 {u, c, h, -}
    //                 3D: w0 {x, y, z, m}, w1 {vx, vy, vz, itype's bits}, w2 {rho, p, c, h}
    float4* w0[2];
    float4* w1[2];
    float4* w2[2];
    float* uw[2];   // 3D: u
    int* id;
    float4* xsort;  // lazy sorting: positions at the last sort (nullptr: every step sorts)
    // Neighbour lists of the last sort (StateB's blocks; entries within 2 h_i + skin in
    // cursor order) and, per step, the entries in reach at the step's start: bit t % 32 of
    // pass[(t / 32) * n + i].
    const int* nlist;
    const int* ncount;
    int lstride;
    unsigned* pass;
};

// One particle of a working copy.
struct GpucPart {
    float x[3], v[3], m, h, rho, u, p, c;
    int it;
};
template <int DIM>
__device__ __forceinline__ GpucPart gpuc_load(const GpucState& S, int w, int i) {
    const float4 a = (w ? S.w0[1] : S.w0[0])[i], b = (w ? S.w1[1] : S.w1[0])[i];
    const float4 c = (w ? S.w2[1] : S.w2[0])[i];
    GpucPart q;
    if (DIM == 2)
        q = {{a.x, a.y, 0.f}, {a.z, a.w, 0.f}, b.z, c.z, b.x, c.x, b.y, c.y, __float_as_int(b.w)};
    else
        q = {{a.x, a.y, a.z}, {b.x, b.y, b.z}, a.w, c.w, c.x, (w ? S.uw[1] : S.uw[0])[i], c.y, c.z,
             __float_as_int(b.w)};
    return q;
}
template <int DIM>
__device__ __forceinline__ void gpuc_store(const GpucState& S, int w, int i, const GpucPart& q) {
    float4* a = w ? S.w0[1] : S.w0[0];
    float4* b = w ? S.w1[1] : S.w1[0];
    float4* c = w ? S.w2[1] : S.w2[0];
    if (DIM == 2) {
        a[i] = make_float4(q.x[0], q.x[1], q.v[0], q.v[1]);
        b[i] = make_float4(q.rho, q.p, q.m, __int_as_float(q.it));
        c[i] = make_float4(q.u, q.c, q.h, 0.f);
    } else {
        a[i] = make_float4(q.x[0], q.x[1], q.x[2], q.m);
        b[i] = make_float4(q.v[0], q.v[1], q.v[2], __int_as_float(q.it));
        c[i] = make_float4(q.rho, q.p, q.c, q.h);
        (w ? S.uw[1] : S.uw[0])[i] = q.u;
    }
}

// The EOS of one particle after its update (acpu.c:932-962 with the property
// functions of acpu.c:560-870; ESS of Code/armando.cu:572-598 on absolute
// density). rho is clamped where the type clamps.
__device__ __forceinline__ void gpuc_eos(const DevMaterial& M, float& rho, float u, float& p, float& c) {
    const float* q = M.prop;
    switch (M.type) {
    case 0:  // boundary
        if (rho < 0.9f * q[0]) rho = 0.9f * q[0];
        p = 0.f;
        c = q[1];
        break;
    case 1:  // ideal gas
        p = __fadd_rn(__fmul_rn(__fmul_rn(q[1] - 1.0f, rho), u), q[2]);
        c = sqrtf(__fmul_rn(__fmul_rn(q[1], q[1] - 1.0f), u));
        break;
    case 2: {  // Mie-Gruneisen polynomial
        if (rho < 0.9f * q[0]) rho = 0.9f * q[0];
        const float mu = __fdiv_rn(rho - q[0], q[0]);
        const float mu2 = __fmul_rn(mu, mu);
        if (mu < 0.f)
            p = __fadd_rn(__fadd_rn(__fmul_rn(q[6], mu), __fmul_rn(q[7], mu2)),
                          __fmul_rn(__fmul_rn(q[4], q[0]), u));
        else
            p = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(q[1], mu), __fmul_rn(q[2], mu2)),
                                    __fmul_rn(q[3], __fmul_rn(mu2, mu))),
                          __fmul_rn(__fmul_rn(__fadd_rn(q[4], __fmul_rn(q[5], mu)), q[0]), u));
        c = sqrtf(__fdiv_rn(q[1], rho));
        break;
    }
    case 3: {  // Mie-Gruneisen shock
        if (rho < 0.9f * q[0]) rho = 0.9f * q[0];
        const float mu = __fdiv_rn(rho - q[0], q[0]);
        const float den = __fsub_rn(1.0f, __fmul_rn(q[3] - 1.0f, mu));
        const float ph = __fdiv_rn(__fmul_rn(__fmul_rn(__fmul_rn(q[0], __fmul_rn(q[1], q[1])), mu),
                                             1.0f + mu),
                                   __fmul_rn(den, den));
        const float corr = __fmul_rn(__fdiv_rn(__fmul_rn(0.5f, ph), q[0]), __fdiv_rn(mu, 1.0f + mu));
        p = __fadd_rn(ph, __fmul_rn(__fmul_rn(q[2], q[0]), __fsub_rn(u, corr)));
        c = q[1];
        break;
    }
    case 4: {  // Tait
        if (rho < 0.9f * q[0]) rho = 0.9f * q[0];
        const float r = __fdiv_rn(rho, q[0]);
        const float r2 = __fmul_rn(r, r), r4 = __fmul_rn(r2, r2);
        const float r7 = __fmul_rn(__fmul_rn(r4, r2), r);
        p = __fmul_rn(__fdiv_rn(__fmul_rn(q[0], __fmul_rn(q[1], q[1])), 7.0f), r7 - 1.0f);
        c = q[1];
        break;
    }
    case 5: {  // ESS
        const float mu = __fdiv_rn(rho, q[0]) - 1.0f;
        p = __fadd_rn(__fmul_rn(__fmul_rn(mu, q[0]), __fmul_rn(q[1], q[1])),
                      __fmul_rn(__fmul_rn(u, q[0]), q[2]));
        if (p < q[3]) p = q[3];
        c = q[1];
        break;
    }
    default:
        p = 0.f;
        break;
    }
}

__device__ __forceinline__ int gpuc_material(int itype, int n_mat, unsigned* flags) {
    const int k = itype < 0 ? -itype : itype;
    if (k >= n_mat) {
        atomicOr(flags, (unsigned)FLAG_BAD_MATERIAL);
        return 0;
    }
    return k;
}

// Cell order of the step: start state, first working copy, sound speeds.
// A is in the cell order of the last sort, so a step that does not sort
// (lazy sorting) takes it slot for slot.
template <int DIM>
__global__ void k_gpuc_gather(StateA A, const int* __restrict__ perm, GpucState S,
                              const DevMaterial* __restrict__ mat, int n_mat,
                              unsigned* __restrict__ flags, int n,
                              const int* __restrict__ resort = nullptr) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    const bool sorted = !sort_skipped(resort);
    const int j = sorted ? perm[s] : s;
    const float4 xh = A.xh[j], vm = A.vm[j];
    if (sorted && S.xsort) S.xsort[s] = xh;
    const int it = A.itype[j];
    float rho = A.rho[j];
    const float u = A.u[j], p = A.p[j];
    float pp = 0.f, c = 0.f, r = rho;
    gpuc_eos(mat[gpuc_material(it, n_mat, flags)], r, u, pp, c);  // Sound of the last update
    S.x0[s] = xh;
    S.v0[s] = vm;
    S.q0[s] = make_float2(rho, u);
    gpuc_store<DIM>(S, 0, s, GpucPart{{xh.x, xh.y, DIM == 3 ? xh.z : 0.f}, {vm.x, vm.y, vm.z},
                                      mass_of<DIM>(xh, vm), xh.w, rho, u, p, c, it});
    S.id[s] = A.id[j];
}

// Wendland C2 with h_i as the GPU-C codes evaluate it (acpu.c:146-201):
// W = K/h^dim (1 - q/2)^4 (1 + 2q), dW/dr = K/h^(dim+1) 5/8 q (q - 2)^3.
// The particle's factors: ih = 1/h, alpha = K/h^dim (as K ih^dim).
template <int DIM>
__device__ __forceinline__ void gpuc_kernel_norm(float h, float K, float& ih, float& alpha) {
    ih = __frcp_rn(h);
    alpha = DIM == 2 ? __fmul_rn(K, __fmul_rn(ih, ih)) : __fmul_rn(K, __fmul_rn(__fmul_rn(ih, ih), ih));
}

// The smallest t with sqrt_rn(t) >= lim, so that sqrt_rn(r2) < lim exactly when
// r2 < t (sqrt_rn is monotone): updateListHost's test without a square root
// per candidate. lim^2 rounded lies within one step of t (checked on random
// FP32 lims over [1e-30, 1e19] against IEEE square roots, in the CPU tests);
// the loops allow four. lim <= 0 or NaN: no r2 passes.
__device__ __forceinline__ float sqrt_less_bound(float lim) {
    if (!(lim > 0.f)) return -INFINITY;
    float t = __fmul_rn(lim, lim);
    if (isinf(t)) return t;  // every finite r2 has sqrt_rn(r2) < lim
#pragma unroll 1
    for (int q = 0; q < 4 && __fsqrt_rn(t) < lim; ++q) t = nextafterf(t, INFINITY);
#pragma unroll 1
    for (int q = 0; q < 4; ++q) {
        const float d = nextafterf(t, 0.f);
        if (!(__fsqrt_rn(d) >= lim)) break;
        t = d;
    }
    return t;
}

// Neighbours a lane collects before it evaluates them (a longer list is
// evaluated in pieces of this length): about the lane's share of the 2D / 3D
// neighbours, at least 8, within 48 KB of static shared memory per CTA.
template <int DIM, int TPP, int BS>
__host__ __device__ constexpr int gpuc_list_len() {
    constexpr int want = (DIM == 2 ? 32 : 64) / TPP < 8 ? 8 : (DIM == 2 ? 32 : 64) / TPP;
    return want * BS * 4 > 48 * 1024 ? 48 * 1024 / (4 * BS) : want;
}

// One RK3 stage: rates of every particle from working copy `cur`, update into the
// other (X0 + alpha (X + dt dX/dt - X0)), EOS. VAR 1: host path, 2: device.
// TPP lanes per particle split its candidates (lane `sub` takes slots
// k0 + sub, k0 + sub + TPP, ... of every cell range) and sum their rates with
// an xor butterfly; lane 0 updates. TPP = 1 sums in candidate order.
// LST: between sorts the neighbours come from the lists of the last sort, whose
// entries the step's first stage (stage 0) tests against the start positions;
// its pass bits serve the other two. Without lists, and for particles whose list
// overflowed, each lane lists the candidates that pass the start-position test
// in shared memory (candidate order) and evaluates that list. Both evaluate two
// neighbours at a time (pair2.cuh), each operation rounded as a single pair's in the
// reference's order, divisions and square roots too (div2, sqrt2 in pair2.cuh).
//
// Issue and latency bound the stage (42-57% of cycles): it walked its cells three
// times a step, with the divider's code five times a pair. Measured a stage,
// 85,773 / 361,201 particles: 28.7 / 84.9 us walking the cells, 15.1 / 34.2 on lists
// (8 / 22 us a sort to build them); 96 registers, so that five blocks of 128 fit.
template <int DIM, int VAR, int TPP = 1, int BS = kPassThreads, bool LST = false>
__global__ void __launch_bounds__(BS, LST && BS <= 256 ? 640 / BS : 1)
    k_gpuc_stage(GpucState S, int cur, const unsigned* __restrict__ keys,
                 const int* __restrict__ start, const DevGrid* __restrict__ gp, DevParams P,
                 const DevMaterial* __restrict__ mat, int n_mat, const DevZones* __restrict__ zones,
                 unsigned* __restrict__ flags, float alpha, float dt, int n, int stage, StateA A) {
    static_assert(!LST || TPP == 1, "lists: one lane per particle");
    const int i0 = blockIdx.x * (BS / TPP) + (int)threadIdx.x / TPP;
    const int sub = (TPP == 1) ? 0 : (int)(threadIdx.x & (TPP - 1));
    const bool valid = i0 < n;
    const int i = valid ? i0 : n - 1;  // (a lane past the end repeats the last particle's walk)
    const DevGrid g = *gp;
    const float4* __restrict__ n0 = cur ? S.w0[1] : S.w0[0];
    const float4* __restrict__ n1 = cur ? S.w1[1] : S.w1[0];
    const float4* __restrict__ n2 = cur ? S.w2[1] : S.w2[0];
    const GpucPart q = gpuc_load<DIM>(S, cur, i);
    const float r2_bound = sqrt_less_bound(__fmul_rn(2.0f, q.h));
    float ih, kal;
    gpuc_kernel_norm<DIM>(q.h, P.kw_hi, ih, kal);
    const float aih = __fmul_rn(kal, ih), dead = __fmul_rn(0.01f, q.h);
    // the device variant's own pressure term (armando.cu:483-485)
    const float p_i = (VAR == 2) ? __fdiv_rn(q.p, __fmul_rn(q.rho, q.rho)) : q.p;
    float rd = 0.f, a0 = 0.f, a1 = 0.f, a2 = 0.f;
    // Push between particles of different itype (acpu.c:424-429; armando.cu:507-513).
    auto push = [&](int k, float mk, float rhok, float ck3, float hk3, float dr, float qk) {
        if (!(qk < 2.f)) return 0.f;
        const float4 o = DIM == 2 ? __ldg(n2 + k) : make_float4(0.f, ck3, hk3, 0.f);
        float t = fmaf(-0.5f, qk, 1.0f);
        t = __fmul_rn(t, t);
        t = __fmul_rn(t, t);
        const float w = __fmul_rn(__fmul_rn(t, fmaf(2.0f, qk, 1.0f)), kal);
        if (VAR == 1)
            return __fmul_rn(__fdiv_rn(mk, q.m + mk),
                             __fdiv_rn(__fmul_rn(__fmul_rn(0.02f, __fdiv_rn(w, kal)), __fmul_rn(q.c, o.y)), dr));
        return __fmul_rn(__fdiv_rn(__fdiv_rn(__fmul_rn(__fmul_rn(0.5f, w), mk), rhok), o.z),
                         __fmul_rn(o.y, o.y));
    };
    // Two neighbours; ina, inb: whether they count.
    auto pair2 = [&](int ka, int kb, const float4& xa, const float4& xb, const float4& ya,
                     const float4& yb, const float4& za, const float4& zb, bool ina, bool inb) {
        const f2 d0 = make_float2(q.x[0] - xa.x, q.x[0] - xb.x), d1 = make_float2(q.x[1] - xa.y, q.x[1] - xb.y);
        const f2 d2 = DIM == 3 ? make_float2(q.x[2] - xa.z, q.x[2] - xb.z) : bc2(0.f);
        f2 r2 = fma2(d1, d1, fma2(d0, d0, bc2(kTinyDr2)));
        if (DIM == 3) r2 = fma2(d2, d2, r2);
        const f2 rs = rsqrt2(r2);
        const f2 dr = sqrt2(r2, rs);
        // dr < 0.01 h: dr := 100 h, W = dW/dr = 0 (acpu.c:379)
        f2 mk = DIM == 2 ? make_float2(ya.z, yb.z) : make_float2(xa.w, xb.w);
        // (the others' terms are left out by selects: they may be infinite or NaN)
        ina = ina && !(dr.x < dead);
        inb = inb && !(dr.y < dead);
        mk.x = ina ? mk.x : 0.f;
        mk.y = inb ? mk.y : 0.f;
        const f2 ir = rcp2_rn(dr, rs);
        // dW/dr = K/h^(dim+1) 5/8 q (q - 2)^3 (acpu.c:146-201)
        const f2 qk = div2(dr, bc2(q.h), bc2(ih));
        const f2 qm = min2(sub2(qk, bc2(2.0f)), 0.0f);
        const f2 dw = mul2(mul2(mul2(bc2(0.625f), qk), mul2(mul2(qm, qm), qm)), bc2(aih));
        f2 dvr;
        if (DIM == 2) {
            dvr = mul2(d0, make_float2(q.v[0] - xa.z, q.v[0] - xb.z));
            dvr = fma2(d1, make_float2(q.v[1] - xa.w, q.v[1] - xb.w), dvr);
        } else {
            dvr = mul2(d0, make_float2(q.v[0] - ya.x, q.v[0] - yb.x));
            dvr = fma2(d1, make_float2(q.v[1] - ya.y, q.v[1] - yb.y), dvr);
            dvr = fma2(d2, make_float2(q.v[2] - ya.z, q.v[2] - yb.z), dvr);
        }
        const f2 rk = DIM == 2 ? make_float2(ya.x, yb.x) : make_float2(za.x, zb.x);
        const f2 pk = DIM == 2 ? make_float2(ya.y, yb.y) : make_float2(za.y, zb.y);
        const int ita = __float_as_int(ya.w), itb = __float_as_int(yb.w);
        f2 ms = mk;  // the pairs that take the density, pressure and shock terms
        if (VAR == 2) {
            if (ita != q.it) ms.x = 0.f;
            if (itb != q.it) ms.y = 0.f;
        }
        f2 f;
        if (VAR == 1) {
            f = div2(neg2(make_float2(q.p + pk.x, q.p + pk.y)), mul2(bc2(q.rho), rk));
        } else {
            const f2 pr = div2(pk, mul2(rk, rk));
            f = neg2(make_float2(p_i + pr.x, p_i + pr.y));
        }
        f = mul2(ms, f);
        const f2 cs = div2(bc2(__fmul_rn(2.0f, q.c)), make_float2(q.rho + rk.x, q.rho + rk.y));
        f2 sh = div2(mul2(dvr, bc2(q.h)), fma2(bc2(0.01f * q.h), bc2(q.h), mul2(dr, dr)));
        sh = mul2(mul2(sh, cs), bc2(0.03f));
        f2 mq = ms;
        if (!(dvr.x < 0.f)) mq.x = 0.f;
        if (!(dvr.y < 0.f)) mq.y = 0.f;
        f = fma2(mq, sh, f);
        f2 ps = bc2(0.f);
        if (ita != q.it && ina) ps.x = push(ka, mk.x, rk.x, za.z, za.w, dr.x, qk.x);
        if (itb != q.it && inb) ps.y = push(kb, mk.y, rk.y, zb.z, zb.w, dr.y, qk.y);
        f2 c1 = mul2(ms, dvr), c2 = mul2(dw, ir);
        f2 c3 = mul2(ms, mul2(make_float2(q.rho - rk.x, q.rho - rk.y), cs));
        if (!ina) c1.x = c3.x = f.x = 0.f;
        if (!inb) c1.y = c3.y = f.y = 0.f;
        rd = fmaf(c3.x, dw.x, fmaf(c1.x, c2.x, rd));
        rd = fmaf(c3.y, dw.y, fmaf(c1.y, c2.y, rd));
        const f2 tot = mul2(fma2(f, dw, ps), ir);
        a0 = dot2(tot, d0, a0);
        a1 = dot2(tot, d1, a1);
        if (DIM == 3) a2 = dot2(tot, d2, a2);
    };
    const int lc = (LST && g.ok) ? list_near(__ldg(S.ncount + i)) : -1;
    if (LST) prefetch_list(S.nlist, S.lstride, i, lc);
    const float4 x0i = S.x0[i];
    // updateListHost's test on the step's start positions (unfused)
    auto in_reach = [&](const float4& x0k) {
        const float e0 = __fsub_rn(x0i.x, x0k.x), e1 = __fsub_rn(x0i.y, x0k.y);
        float r2 = __fadd_rn(__fmul_rn(e0, e0), __fmul_rn(e1, e1));
        if (DIM == 3) {
            const float e2 = __fsub_rn(x0i.z, x0k.z);
            r2 = __fadd_rn(r2, __fmul_rn(e2, e2));
        }
        return r2 < r2_bound;
    };
    if (LST) {
        constexpr int NB = DIM == 2 ? 4 : 2;  // entries whose loads issue together
        const int nb = blocks_of(lc);
        const int bm = __reduce_max_sync(0xffffffffu, nb);
        unsigned word = 0u;
        int4 kn = list_block(S.nlist, S.lstride, i, 0, nb, i);
        for (int b = 0; b < bm; ++b) {
            const int t0 = 4 * b;
            if (t0 % 32 == 0) word = (stage != 0 && t0 < lc) ? S.pass[(size_t)(t0 / 32) * n + i] : 0u;
            const int4 q4 = kn;
            if (b + 1 < bm) kn = list_block(S.nlist, S.lstride, i, b + 1, nb, i);
            const int kb[4] = {q4.x, q4.y, q4.z, q4.w};
#pragma unroll
            for (int v = 0; v < 4; v += NB) {
                float4 xb[NB], yb[NB], zb[NB];
#pragma unroll
                for (int u = 0; u < NB; ++u) {
                    xb[u] = __ldg(n0 + kb[v + u]);
                    yb[u] = __ldg(n1 + kb[v + u]);
                    zb[u] = DIM == 3 ? __ldg(n2 + kb[v + u]) : yb[u];
                }
                if (stage == 0) {  // the working positions are the start's
#pragma unroll
                    for (int u = 0; u < NB; ++u)
                        if (t0 + v + u < lc && in_reach(xb[u])) word |= 1u << ((t0 + v + u) % 32);
                }
                const unsigned w = word >> ((t0 + v) % 32);
#pragma unroll
                for (int u = 0; u < NB; u += 2)
                    pair2(kb[v + u], kb[v + u + 1], xb[u], xb[u + 1], yb[u], yb[u + 1], zb[u], zb[u + 1],
                          (w >> u) & 1u, (w >> (u + 1)) & 1u);
            }
            if (stage == 0 && valid && t0 < lc && ((t0 + 4) % 32 == 0 || t0 + 4 >= lc))
                S.pass[(size_t)(t0 / 32) * n + i] = word;
        }
    }
    if (g.ok && (!LST || __any_sync(0xffffffffu, lc < 0))) {
        constexpr int ML = LST ? kListCapLst : gpuc_list_len<DIM, TPP, BS>();
        __shared__ int s_list[ML][BS];
        const int tid = threadIdx.x;
        int nl = 0;
        auto eval = [&](int cnt) {
            for (int e = 0; e < cnt; e += 2) {
                const int ka = s_list[e][tid], kb = e + 1 < cnt ? s_list[e + 1][tid] : i;
                const float4 xa = __ldg(n0 + ka), xb = __ldg(n0 + kb), ya = __ldg(n1 + ka), yb = __ldg(n1 + kb);
                const float4 za = DIM == 3 ? __ldg(n2 + ka) : ya, zb = DIM == 3 ? __ldg(n2 + kb) : yb;
                pair2(ka, kb, xa, xb, ya, yb, za, zb, true, e + 1 < cnt);
            }
        };
        if (!LST || lc < 0) {
            const CellCoord cc = decode_key<DIM>(keys[i], g);
            Cursor cu = cursor_begin<DIM>(g);
            while (cursor_next<DIM>(g, start, cc, cu))
                for (int k = cu.k + sub; k < cu.ke; k += TPP) {
                    if (k == i || !in_reach(__ldg(S.x0 + k))) continue;
                    s_list[nl++][tid] = k;
                    if (nl == ML) {  // a full list: evaluate it and go on collecting
                        eval(ML);
                        nl = 0;
                    }
                }
        }
        eval(nl);
    }
    if (TPP > 1) {  // the particle's lanes reach this point together
        rd = group_sum<TPP>(rd);
        a0 = group_sum<TPP>(a0);
        a1 = group_sum<TPP>(a1);
        if (DIM == 3) a2 = group_sum<TPP>(a2);
        if (sub != 0) return;
    }
    if (!valid) return;
    // the start state, read after the pair loop (not held in registers across it)
    const float4 v0i = S.v0[i];
    const float2 q0 = S.q0[i];
    const int it = q.it;
    const float4 xi = make_float4(q.x[0], q.x[1], q.x[2], 0.f);
    float wz = 0.f;
    if (it > 0) {  // updateLoadsHost: gravity over every fluid particle, then the zones
        float g0 = P.gravity[0], g1 = P.gravity[1], g2 = P.gravity[2];
        const int nl = __ldg(&zones->n_load);
#pragma unroll 1
        for (int z = 0; z < nl; ++z) {
            const DevLoadZone* Z = zones->load + z;
            if (!in_zone<DIM>(Z->lo, Z->hi, xi)) continue;
            g0 = __fadd_rn(g0, __ldg(&Z->g[0]));
            g1 = __fadd_rn(g1, __ldg(&Z->g[1]));
            g2 = __fadd_rn(g2, __ldg(&Z->g[2]));
            wz = __fadd_rn(wz, __ldg(&Z->w));
        }
        const int np = __ldg(&zones->n_fix);
#pragma unroll 1
        for (int z = 0; z < np; ++z) {  // pump zones: (vel - v) / tau (Code/armando.cu:1046-1055)
            const DevFixZone* Z = zones->fix + z;
            const float tau = __ldg(&Z->tau);
            if (!(tau > 0.f) || !in_zone<DIM>(Z->lo, Z->hi, xi)) continue;
            g0 = __fadd_rn(g0, __fdiv_rn(__fsub_rn(__ldg(&Z->v[0]), q.v[0]), tau));
            g1 = __fadd_rn(g1, __fdiv_rn(__fsub_rn(__ldg(&Z->v[1]), q.v[1]), tau));
            if (DIM == 3) g2 = __fadd_rn(g2, __fdiv_rn(__fsub_rn(__ldg(&Z->v[2]), q.v[2]), tau));
        }
        a0 += g0;
        a1 += g1;
        if (DIM == 3) a2 += g2;
    }
    // balanceEnergyHost on top of the loads' w
    const float du = __fadd_rn(wz, __fdiv_rn(__fmul_rn(q.p, rd), __fmul_rn(q.rho, q.rho)));
    GpucPart o = q;
    if (VAR == 2 || it != 0) {  // acpu.c:894 leaves itype 0 alone
        o.x[0] = fmaf(alpha, fmaf(dt, q.v[0], q.x[0]) - x0i.x, x0i.x);
        o.x[1] = fmaf(alpha, fmaf(dt, q.v[1], q.x[1]) - x0i.y, x0i.y);
        if (DIM == 3) o.x[2] = fmaf(alpha, fmaf(dt, q.v[2], q.x[2]) - x0i.z, x0i.z);
        o.v[0] = fmaf(alpha, fmaf(dt, a0, q.v[0]) - v0i.x, v0i.x);
        o.v[1] = fmaf(alpha, fmaf(dt, a1, q.v[1]) - v0i.y, v0i.y);
        if (DIM == 3) o.v[2] = fmaf(alpha, fmaf(dt, a2, q.v[2]) - v0i.z, v0i.z);
        o.rho = fmaf(alpha, fmaf(dt, rd, q.rho) - q0.x, q0.x);
        o.u = fmaf(alpha, fmaf(dt, du, q.u) - q0.y, q0.y);
        const DevMaterial& M = mat[gpuc_material(it, n_mat, flags)];
        auto keep_v = [&]() {
            o.v[0] = v0i.x;
            o.v[1] = v0i.y;
            if (DIM == 3) o.v[2] = v0i.z;
        };
        if (VAR == 1 && it <= 0) keep_v();  // acpu.c:910-914
        const float4 xn = make_float4(o.x[0], o.x[1], o.x[2], 0.f);
        const int nf = __ldg(&zones->n_fix);
#pragma unroll 1
        for (int z = 0; z < nf; ++z) {  // fix zones at the new position
            const DevFixZone* Z = zones->fix + z;
            if (__ldg(&Z->tau) > 0.f || !in_zone<DIM>(Z->lo, Z->hi, xn)) continue;  // pumps: above
            o.v[0] = __ldg(&Z->v[0]);
            o.v[1] = __ldg(&Z->v[1]);
            if (DIM == 3) o.v[2] = __ldg(&Z->v[2]);
        }
        if (M.type == 0) keep_v();  // boundary materials keep their velocity
        o.p = 0.f;
        gpuc_eos(M, o.rho, o.u, o.p, o.c);
        const float chk = o.x[0] + o.x[1] + o.x[2] + o.v[0] + o.v[1] + o.v[2] + o.rho + o.u + o.p;
        if (!isfinite(chk)) atomicOr(flags, (unsigned)FLAG_NONFINITE);
    }
    if (stage < 2) {
        gpuc_store<DIM>(S, cur ^ 1, i, o);
        return;
    }
    // The step's result to A (cell order of this step, like the force pass). As a kernel
    // of its own five steps took 464 us at 86 k particles, now 454, and at 361 k, where
    // the copy itself counts, 1,013 and 1,010.
    // Lazy sorting: a particle farther than half the skin from where it was binned
    // makes the next step sort (the cells of the last sort hold every pair within
    // 2 max(h) of the step's start positions only while none is).
    if (S.xsort) {
        const float4 xb = S.xsort[i];
        const float e0 = o.x[0] - xb.x, e1 = o.x[1] - xb.y, e2 = (DIM == 3) ? o.x[2] - xb.z : 0.f;
        if (g.half_skin2 > 0.f && e0 * e0 + e1 * e1 + e2 * e2 > g.half_skin2 &&
            *(volatile unsigned*)(flags + 2) == 0u)
            atomicExch(flags + 2, 1u);
    }
    A.xh[i] = DIM == 2 ? make_float4(o.x[0], o.x[1], o.m, o.h) : make_float4(o.x[0], o.x[1], o.x[2], o.h);
    A.vm[i] = make_float4(o.v[0], o.v[1], o.v[2], DIM == 3 ? o.m : 0.f);
    A.rho[i] = o.rho;
    A.u[i] = o.u;
    A.p[i] = o.p;
    A.ap[i] = make_float4(a0, a1, a2, du);
    A.itype[i] = o.it;
    A.id[i] = S.id[i];
}

}  // namespace ag

namespace ag {

// ---------------------------------------------------------------------------
// Open boundaries (armando.cu:2640-2856): outlets and the box remove particles,
// keeping the order of the rest (a block scan over tiles of kGhostTile).
// ---------------------------------------------------------------------------
struct DevOutlet {
    float o[3], n[3], R;
};

struct OpenSpec {
    DevOutlet out[10];
    int n_out;
    float lo[3], hi[3];
};

// checkOutDevice (armando.cu:2682-2722) in FP32, operations in order, unfused.
template <int DIM>
__device__ __forceinline__ bool open_leaves(const float4& xh, const OpenSpec& O) {
    const float x[3] = {xh.x, xh.y, DIM == 3 ? xh.z : 0.f};
    for (int q = 0; q < O.n_out; ++q) {
        const DevOutlet& Q = O.out[q];
        float dn = 0.f;
        for (int d = 0; d < DIM; ++d) dn = __fadd_rn(dn, __fmul_rn(__fsub_rn(x[d], Q.o[d]), Q.n[d]));
        float dr = 0.f;
        for (int d = 0; d < DIM; ++d) {
            const float e = __fsub_rn(__fsub_rn(x[d], Q.o[d]), __fmul_rn(dn, Q.n[d]));
            dr = __fadd_rn(dr, __fmul_rn(e, e));
        }
        if (dn < 0.f && __fsqrt_rn(dr) < Q.R) return true;
    }
    for (int d = 0; d < DIM; ++d)
        if (x[d] > O.hi[d] || x[d] < O.lo[d]) return true;
    return false;
}

template <int DIM>
__global__ void __launch_bounds__(kGhostThreads)
    k_open_flags(StateA A, int n, OpenSpec O, int* __restrict__ keep,
                 unsigned* __restrict__ tile_count) {
    __shared__ unsigned s_warp[32];
    __shared__ unsigned s_total;
    unsigned mine = 0;
    for (int it = 0; it < kGhostItems; ++it) {
        const int i = blockIdx.x * kGhostTile + it * kGhostThreads + (int)threadIdx.x;
        if (i >= n) break;
        const int k = open_leaves<DIM>(A.xh[i], O) ? 0 : 1;
        keep[i] = k;
        mine += k;
    }
    block_excl_scan<kGhostThreads>(mine, s_warp, &s_total);
    if (threadIdx.x == 0) tile_count[blockIdx.x] = s_total;
}

// The kept particles of A, in order, into D.
static __global__ void __launch_bounds__(kGhostThreads)
    k_open_compact(StateA A, StateA D, int n, const int* __restrict__ keep,
                   const unsigned* __restrict__ tile_off) {
    __shared__ unsigned s_warp[32];
    __shared__ unsigned s_total;
    unsigned base = tile_off[blockIdx.x];
    for (int it = 0; it < kGhostItems; ++it) {
        const int i = blockIdx.x * kGhostTile + it * kGhostThreads + (int)threadIdx.x;
        const int k = (i < n) ? keep[i] : 0;
        const unsigned rank = block_excl_scan<kGhostThreads>((unsigned)k, s_warp, &s_total);
        if (k) {
            const int o = (int)(base + rank);
            D.xh[o] = A.xh[i];
            D.vm[o] = A.vm[i];
            D.u[o] = A.u[i];
            D.ap[o] = A.ap[i];
            D.rho[o] = A.rho[i];
            D.p[o] = A.p[i];
            D.itype[o] = A.itype[i];
            D.id[o] = A.id[i];
        }
        base += s_total;
    }
}

// Keys of the output order: the particles' serial numbers.
static __global__ void k_open_id_keys(StateA A, int n, unsigned* __restrict__ keys) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s < n) keys[s] = (unsigned)A.id[s];
}

// Output r = the particle of rank r in serial order: every field, staged.
template <int DIM>
__global__ void k_open_out(StateA A, const int* __restrict__ order, int n, float* __restrict__ x,
                           float* __restrict__ v, float* __restrict__ m, float* __restrict__ rho,
                           float* __restrict__ p, float* __restrict__ u, float* __restrict__ h,
                           int* __restrict__ itype, float* __restrict__ dvdt,
                           float* __restrict__ dudt) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n) return;
    const int s = order[r];
    const float4 a = A.xh[s], b = A.vm[s], q = A.ap[s];
    x[DIM * r] = a.x;
    x[DIM * r + 1] = a.y;
    v[DIM * r] = b.x;
    v[DIM * r + 1] = b.y;
    dvdt[DIM * r] = q.x;
    dvdt[DIM * r + 1] = q.y;
    if (DIM == 3) {
        x[3 * r + 2] = a.z;
        v[3 * r + 2] = b.z;
        dvdt[3 * r + 2] = q.z;
    }
    m[r] = (DIM == 2) ? a.z : b.w;
    h[r] = a.w;
    dudt[r] = q.w;
    u[r] = A.u[s];
    rho[r] = A.rho[s];
    p[r] = A.p[s];
    itype[r] = A.itype[s];
}

}  // namespace ag
