// kernels.cuh -- sm_103a kernels of one leapfrog step of Armando's SPH.
//
// Step pipeline (one CUDA graph per step):
//   bbox_grid                         grid of CERNsource/link_list.f:39-67
//   cell_count                        cell id, link_list.f:75-88 / acpu.c:2085-2105, and
//                                     the particles of every cell
//   cell_sums -> cell_scan            first slot of every cell (empty cells included)
//   cell_place -> cell_rank           the particles by (cell, previous slot)
//   reorder                           gather state into cell order + leapfrog predictor
//                                     (time_integration.f:136-154)
//   density                           summation density + Tait EOS + div v
//                                     (density.f:1-62, eos.f90:255-283, art_heat.f:46-67)
//   shear (physical viscosity only)   shear tensor T_ab (internal_force.f:75-171)
//   force                             pressure + viscous force, art_visc, art_heat,
//                                     external heat, gravity, leapfrog corrector
//                                     (internal_force.f:178-435, art_visc.f:55-101,
//                                     art_heat.f:69-97, time_integration.f:186-218)
// Every pass is a gather over the 3^dim neighbour cells of a particle: no
// atomics on particle data, so a step is deterministic. Layout (float4, sorted
// by cell):
//   xh  2D {x, y, m, h}        3D {x, y, z, h}
//   vm  2D {vx, vy, 0, 0}      3D {vx, vy, vz, m}
//   rp  {rho, pf, u, psi}      pf = p/rho^2 (pa_sph 1) or p (pa_sph 0),
//                              psi = art_heat coefficient of the particle
#pragma once
#include <cfloat>
#include <cstdint>

#include <type_traits>

#include "pair2.cuh"
#include "sph_math.cuh"

namespace ag {

constexpr int kSortThreads = 256;
constexpr int kSortItems = 8;
constexpr int kSortTile = kSortThreads * kSortItems;
constexpr int kRadix = 256;
constexpr int kPassThreads = 128;
constexpr int kBBoxBlocks = 608;  // 4 x 152 SMs

enum DevFlag : unsigned {
    FLAG_GRID_OVERFLOW = 1u,
    FLAG_NONFINITE = 2u,
    FLAG_OUT_OF_GRID = 4u,
    FLAG_PERIODIC_SMALL = 8u,
    FLAG_BAD_MATERIAL = 16u,  // an itype outside the material table (GPU-C schemes)
    FLAG_TIMEOUT = 32u,       // a bounded wait on a bulk copy gave up
};

struct DevGrid {
    float o[3], size[3], L[3], half[3];
    int n[3];
    int ncells;    // cells of this grid
    int ok;        // 0 when the grid did not fit; passes then do nothing
    int periodic[3];
    int cell_off;  // first cell of this grid in the shared cell table (batches)
    int reach;       // stencil half-width in cells: cell size (2 max(h) + skin) / reach
    float half_skin2;  // (skin / 2)^2: a particle this far from its binned position forces a sort
    float skin;        // sort skin (length): neighbour lists hold pairs within h_i + h_j + skin
    float hmax;        // largest h
    int huni;          // every particle has the same h (the passes' per-pair h terms are constants)
};

// A unit of work of the persistent passes: slots [s0, s1) of one instance.
struct WorkItem {
    int s0, s1, inst, pad;
};

struct DevParams {
    int dim, pa_sph, visc, visc_art, heat_art, heat_ext;
    int periodic[3];
    float rho0, inv_rho0, B, c0, pmin, eta;
    float av_alpha, av_beta, av_eta2;
    float ah_g1, ah_g2, ah_eta2;
    float gravity[3];
    float heat_q0, heat_k, heat_center[3];
    float period_lo[3], period_hi[3], period_L[3], period_half[3];
    float kw_hi, kw_lo;  // K_dim as float-float
    float kg;            // K_dim * 5/8
    float dt;            // time step of this instance (batches)
    float heat_t_end;    // external heat gate its*dt <= heat_t_end
    int reach;           // neighbour-grid cells per support radius (tuning; 1 = link_list)
    float skin;          // sort skin as a fraction of max h (tuning; 0 = sort every step)
    // Wall treatment: 0 like any pair, 1 push only, 2 push and every sum between
    // different itype; 3 like 0 plus mirror ghosts (particles with id >= n_real).
    int wall_model;
    int n_real;          // real particles; ids from n_real on are mirror ghosts
    // single_step options: density 0 summation, 1 continuity, 2 normalised
    // summation; XSPH; smoothing-length evolution 0, 1, 2.
    int density_form, xsph, sle, pad2_;
};

__host__ __device__ inline bool repulsive_walls(const DevParams& P) {
    return P.wall_model == 1 || P.wall_model == 2;
}

struct StepArgs {
    float kdt;    // corrector step: dt (its > 1) or dt/2 (its == 1)
    float hdt;    // predictor half step: dt/2 (its > 1) or 0 (its == 1)
    float dt;     // drift
    int heat_on;  // external heat gate its*dt <= t_end
    int dform;    // density form (1: the predictor advances rho with the carried drho/dt)
};

struct StateA {  // integrated state (slot order of the last sort)
    float4* xh;
    float4* vm;
    float* u;
    float4* ap;  // previous rates {a, du}
    float* rho;
    float* p;
    int* itype;
    int* id;
    int* inst;  // instance of each slot (batches; nullptr for one system)
    float* drho;  // drho/dt of the last iteration (continuity density; else nullptr)
};

struct StateB {  // working set of one step (cell order)
    float4* xh;
    float4* vm;    // predicted velocity (+ mass in 3D)
    float4* vmin;  // velocity and energy at the start of the step
    float4* rp;
    float* p;
    int* itype;
    int* id;
    float4* tau;   // eta T_ab / rho^2 (or eta T_ab): {xx, yy, xy, zz}
    float4* tau2;  // {xz, yz, -, -}
    float* tds;    // T ds/dt
    float* ulo;    // rounding residual of the predicted energy u (rp.z + ulo exact)
    float* q;      // density at the iteration's start (continuity and normalised density)
    float* rlo;    // rounding residual of the predicted density (continuity)
    float4* vr;    // 2D: {vx, vy, rho, P} after the density pass (one neighbour load in the force pass)
    float4* xsort; // position of each slot when the particles were last sorted
    // Neighbour lists of a lazily sorting context (built on the iterations that
    // sort): the candidates within h_i + h_j + skin, first the near ones (q <
    // list_near_q2() when sorted; in 3D all) in cursor order, then the far ones in
    // reverse cursor order, four to an int4: block b of slot s at int4 index
    // b * lstride + s, the last block filled up with s itself; ncount[s] =
    // near | far << 16, -1 when more than lcap (that slot walks its cells instead).
    int* nlist;
    int* ncount;
    int lcap;      // list entries per slot
    int lstride;   // slots per list row (the context's capacity)
    // Neighbour bits of each fluid slot over its first 32 * mask_words<DIM>()
    // candidates (cursor order); words 0 and 1 all ones: more candidates than
    // bits. With TPP lanes per particle, lane L = s * TPP + sub keeps
    // mask_words / TPP words of its own candidates, in chunks of up to 4 words
    // stored chunk-major (mask_word_index), so one vector load per warp reads
    // a chunk of every lane.
    unsigned* nmask;
    int* inst;     // instance of each slot (batches; nullptr for one system)
    int mstride;   // lanes: n * TPP
    int mtpp;      // the TPP the masks were written with
};

template <int DIM>
__host__ __device__ constexpr int mask_words() {
    return DIM == 2 ? 4 : 16;
}

// Words per chunk of a lane holding W mask words.
template <int W>
__host__ __device__ constexpr int mask_chunk() {
    return W < 4 ? W : 4;
}

// Word w of lane L (nl lanes).
template <int W>
__device__ __forceinline__ size_t mask_word_index(int w, size_t nl, size_t L) {
    constexpr int CW = mask_chunk<W>();
    return ((size_t)(w / CW) * nl + L) * CW + (size_t)(w % CW);
}

// Chunk c of lane L as up to four words.
template <int W>
__device__ __forceinline__ uint4 mask_load_chunk(const unsigned* __restrict__ m, size_t nl,
                                                 size_t L, int c) {
    constexpr int CW = mask_chunk<W>();
    const size_t at = (size_t)c * nl + L;
    if (CW == 4) return __ldg(reinterpret_cast<const uint4*>(m) + at);
    if (CW == 2) {
        const uint2 v = __ldg(reinterpret_cast<const uint2*>(m) + at);
        return make_uint4(v.x, v.y, 0u, 0u);
    }
    return make_uint4(__ldg(m + at), 0u, 0u, 0u);
}

__device__ __forceinline__ unsigned chunk_word(const uint4& ch, int j) {
    return j == 0 ? ch.x : j == 1 ? ch.y : j == 2 ? ch.z : ch.w;
}

template <int DIM>
__device__ __forceinline__ float mass_of(const float4& xh, const float4& vm) {
    return DIM == 2 ? xh.z : vm.w;
}

// Lazy sorting (sort skin). resort[1] != 0 asks for a sort: the force pass
// sets it when a particle has moved more than half the skin from where it was
// binned, the host after loading a state. The first kernel of an iteration
// (resort_begin) turns it into resort[0] (this iteration sorts) and clears it.
// The grid, hash, sort and cell-table kernels return at once on an iteration
// that does not sort (their outputs from the last sort stay valid: cells of
// 2 max(h) + skin hold every pair within 2 max(h) while no particle is farther
// than skin / 2 from its binned position). resort == nullptr: always sort.
__device__ __forceinline__ bool sort_skipped(const int* resort) {
    return resort != nullptr && *(volatile const int*)resort == 0;
}

// Start of a lazily sorting iteration (one thread); counts the sorts.
__device__ __forceinline__ unsigned resort_begin(int* resort, int* sorts) {
    const unsigned sort = resort[1] != 0 ? 1u : 0u;
    resort[0] = (int)sort;
    resort[1] = 0;
    if (sort) ++sorts[0];
    return sort;
}

static __global__ void k_resort_begin(int* __restrict__ resort, int* __restrict__ sorts) {
    if (threadIdx.x == 0 && blockIdx.x == 0) resort_begin(resort, sorts);
}

// Head of a lazily sorting step graph: starts the iteration; the IF node
// after it runs the grid, hash, sort and cell-table kernels only when this
// iteration sorts.
static __global__ void k_resort_cond(cudaGraphConditionalHandle handle, int* __restrict__ resort,
                              int* __restrict__ sorts) {
    if (threadIdx.x == 0 && blockIdx.x == 0)
        cudaGraphSetConditional(handle, resort_begin(resort, sorts));
}

// ---------------------------------------------------------------------------
// Small block-level helpers
// ---------------------------------------------------------------------------
__device__ __forceinline__ unsigned warp_incl_scan(unsigned v) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        unsigned t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += t;
    }
    return v;
}

// Exclusive scan of one value per thread over a block of NT threads.
template <int NT>
__device__ __forceinline__ unsigned block_excl_scan(unsigned v, unsigned* s_warp,
                                                    unsigned* total = nullptr) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned inc = warp_incl_scan(v);
    if (lane == 31) s_warp[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        unsigned w = (lane < NT / 32) ? s_warp[lane] : 0u;
        unsigned wi = warp_incl_scan(w);
        if (lane < NT / 32) s_warp[lane] = wi - w;
        if (lane == NT / 32 - 1 && total) *total = wi;
    }
    __syncthreads();
    unsigned r = s_warp[warp] + inc - v;
    __syncthreads();
    return r;
}

// ---------------------------------------------------------------------------
// Grid: bbox of all particles and the link_list grid in FP32.
// ---------------------------------------------------------------------------
// {min[3], max[3], max h, min h} of a CTA's particles (grid stride), to o[8] by its
// first 8 threads.
__device__ __forceinline__ void bbox_of_block(const float4* __restrict__ xh, int n, int dim,
                                              float (*s)[8], float* o) {
    float v[8] = {FLT_MAX, FLT_MAX, FLT_MAX, -FLT_MAX, -FLT_MAX, -FLT_MAX, 0.f, FLT_MAX};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float4 a = xh[i];
        v[0] = fminf(v[0], a.x);
        v[3] = fmaxf(v[3], a.x);
        v[1] = fminf(v[1], a.y);
        v[4] = fmaxf(v[4], a.y);
        if (dim == 3) {
            v[2] = fminf(v[2], a.z);
            v[5] = fmaxf(v[5], a.z);
        }
        v[6] = fmaxf(v[6], a.w);
        v[7] = fminf(v[7], a.w);
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1)
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const float t = __shfl_xor_sync(0xffffffffu, v[k], off);
            v[k] = (k < 3 || k == 7) ? fminf(v[k], t) : fmaxf(v[k], t);
        }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0)
        for (int k = 0; k < 8; ++k) s[warp][k] = v[k];
    __syncthreads();
    if (threadIdx.x < 8) {
        const int k = threadIdx.x;
        float r = s[0][k];
        for (int w = 1; w < (int)(blockDim.x >> 5); ++w)
            r = (k < 3 || k == 7) ? fminf(r, s[w][k]) : fmaxf(r, s[w][k]);
        o[k] = r;
    }
}

static __global__ void __launch_bounds__(256)
    k_bbox_partial(const float4* __restrict__ xh, int n, int dim, float* __restrict__ part) {
    __shared__ float s[8][8];
    bbox_of_block(xh, n, dim, s, part + blockIdx.x * 8);
}

__device__ __forceinline__ DevGrid grid_from_bbox(const float* mm, const DevParams& P,
                                                  long long capacity, unsigned& fl);

// The grid of `nparts` partial boxes (a CTA of 256 threads).
__device__ __forceinline__ void grid_of_parts(const float* part, int nparts, const DevParams& P,
                                              long long capacity, DevGrid* grid, unsigned* flags,
                                              float (*s)[8]) {
    float v[8] = {FLT_MAX, FLT_MAX, FLT_MAX, -FLT_MAX, -FLT_MAX, -FLT_MAX, 0.f, FLT_MAX};
    for (int b = threadIdx.x; b < nparts; b += blockDim.x) {
        const float4 lo = __ldcg(reinterpret_cast<const float4*>(part) + 2 * b);
        const float4 hi = __ldcg(reinterpret_cast<const float4*>(part) + 2 * b + 1);
        v[0] = fminf(v[0], lo.x);
        v[1] = fminf(v[1], lo.y);
        v[2] = fminf(v[2], lo.z);
        v[3] = fmaxf(v[3], lo.w);
        v[4] = fmaxf(v[4], hi.x);
        v[5] = fmaxf(v[5], hi.y);
        v[6] = fmaxf(v[6], hi.z);
        v[7] = fminf(v[7], hi.w);
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1)
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const float t = __shfl_xor_sync(0xffffffffu, v[k], off);
            v[k] = (k < 3 || k == 7) ? fminf(v[k], t) : fmaxf(v[k], t);
        }
    if ((threadIdx.x & 31) == 0)
        for (int k = 0; k < 8; ++k) s[threadIdx.x >> 5][k] = v[k];
    __syncthreads();
    if (threadIdx.x != 0) return;
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w)
        for (int k = 0; k < 8; ++k)
            v[k] = (k < 3 || k == 7) ? fminf(v[k], s[w][k]) : fmaxf(v[k], s[w][k]);
    unsigned fl = 0;
    *grid = grid_from_bbox(v, P, capacity, fl);
    if (fl) atomicOr(flags, fl);
}

static __global__ void __launch_bounds__(256)
    k_bbox_final(const float* __restrict__ part, int nparts, DevParams P, long long capacity,
                 DevGrid* __restrict__ grid, unsigned* __restrict__ flags) {
    __shared__ float s[8][8];
    grid_of_parts(part, nparts, P, capacity, grid, flags, s);
}

// Both in one launch: the CTA that finishes last reduces the partials. `ticket`
// counts the finished CTAs and wraps to 0 for the next launch.
static __global__ void __launch_bounds__(256)
    k_bbox_grid(const float4* __restrict__ xh, int n, int dim, float* part, DevParams P,
                long long capacity, DevGrid* __restrict__ grid, unsigned* __restrict__ flags,
                unsigned* __restrict__ ticket, const int* __restrict__ resort) {
    if (sort_skipped(resort)) return;
    __shared__ float s[8][8];
    __shared__ bool last;
    bbox_of_block(xh, n, dim, s, part + blockIdx.x * 8);
    if (threadIdx.x < 8) __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        last = atomicInc(ticket, gridDim.x - 1) == gridDim.x - 1;
        __threadfence();
    }
    __syncthreads();
    if (last) grid_of_parts(part, (int)gridDim.x, P, capacity, grid, flags, s);
}

// The link_list grid (CERNsource/link_list.f:39-67) of a bbox mm = {min[3],
// max[3], max h, min h}, in FP32; periodic axes split their box into >= 3 cells.
// With P.reach = f the cells are (2 mh + skin) / f wide, skin = P.skin * mh,
// and the passes search (2f + 1)^dim cells. Unless f = 1 and skin = 0 (which
// keep link_list's cell exactly) the cells are widened by a margin larger
// than the rounding of a cell index ((x - o) / size: a few ulp of the index,
// i.e. n * 2^-23 cells), so no pair the exact test accepts is outside the
// stencil.
__device__ __forceinline__ DevGrid grid_from_bbox(const float* mm, const DevParams& P,
                                                  long long capacity, unsigned& fl) {
    DevGrid g;
    const float mh = mm[6];
    const int f = P.reach > 1 ? P.reach : 1;
    const float skin = P.skin > 0.f ? P.skin * mh : 0.f;
    float cell = __fmul_rn(2.0f, mh);  // scale_k * mh, scale_k = 2
    if (f > 1 || skin > 0.f) {
        float span = 0.f;
        for (int d = 0; d < P.dim; ++d)
            span = fmaxf(span, P.periodic[d] ? P.period_L[d] : mm[3 + d] - mm[d] + 2.f * mh);
        const float cf = (cell + skin) / (float)f;
        const float nmax = span / fmaxf(cf, FLT_MIN);
        cell = cf * (1.0f + 0x1p-12f + fminf(nmax, 1.0e7f) * 0x1p-20f);
    }
    long long ncells = 1;
    for (int d = 0; d < 3; ++d) {
        g.periodic[d] = P.periodic[d];
        g.o[d] = 0.f;
        g.size[d] = 1.f;
        g.L[d] = 0.f;
        g.half[d] = 0.f;
        g.n[d] = 1;
        if (d >= P.dim) continue;
        if (P.periodic[d]) {
            const float L = P.period_L[d];
            float nf = __fdiv_rn(L, cell);
            const float nmin = (float)(2 * f + 1);
            int nn = (nf >= nmin && nf < 1.0e9f) ? (int)nf : 2 * f + 1;
            if (!(nf >= nmin)) fl |= FLAG_PERIODIC_SMALL;
            g.o[d] = P.period_lo[d];
            g.size[d] = __fdiv_rn(L, (float)nn);
            g.L[d] = L;
            g.half[d] = P.period_half[d];
            g.n[d] = nn;
        } else {
            const float lo = __fsub_rn(mm[d], mh);
            const float hi = __fadd_rn(mm[3 + d], mh);
            float nf = __fdiv_rn(__fsub_rn(hi, lo), cell);
            g.o[d] = lo;
            g.size[d] = cell;
            if (nf < 1.0e9f) {
                g.n[d] = (int)nf + 1;
            } else {
                g.n[d] = 1;
                fl |= FLAG_GRID_OVERFLOW;
            }
        }
        // Saturates once above the capacity: three axes of up to 1e9 cells
        // each would overflow the product (a far outlier in 3D).
        if (ncells <= capacity) ncells *= g.n[d];
    }
    g.ok = 1;
    g.cell_off = 0;
    g.reach = f;
    g.half_skin2 = 0.25f * skin * skin;
    g.skin = skin;
    g.hmax = mh;
    g.huni = mm[7] == mh ? 1 : 0;
    if (ncells > capacity || (fl & FLAG_GRID_OVERFLOW) || (fl & FLAG_PERIODIC_SMALL)) {
        fl |= (ncells > capacity) ? FLAG_GRID_OVERFLOW : 0u;
        g.ok = 0;
        ncells = capacity;
    }
    g.ncells = (int)ncells;
    return g;
}

template <int DIM>
__device__ __forceinline__ unsigned cell_key(const float4& a, const DevGrid& g) {
    const float xv[3] = {a.x, a.y, a.z};
    unsigned key = 0;
#pragma unroll
    for (int d = DIM - 1; d >= 0; --d) {
        int c = (int)__fdiv_rn(__fsub_rn(xv[d], g.o[d]), g.size[d]);
        c = c < 0 ? 0 : (c > g.n[d] - 1 ? g.n[d] - 1 : c);
        key = key * (unsigned)g.n[d] + (unsigned)c;
    }
    if (!g.ok) key = 0;
    return key + (unsigned)g.cell_off;
}

// Bbox partials straight from caller-layout arrays x[n*DIM], h[n].
template <int DIM>
__global__ void __launch_bounds__(256) k_bbox_partial_raw(const float* __restrict__ x,
                                                          const float* __restrict__ h, int n,
                                                          float* __restrict__ part) {
    float mn[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, mx[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX}, mh = 0.f,
          lh = FLT_MAX;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
#pragma unroll
        for (int d = 0; d < DIM; ++d) {
            const float v = x[(size_t)DIM * i + d];
            mn[d] = fminf(mn[d], v);
            mx[d] = fmaxf(mx[d], v);
        }
        mh = fmaxf(mh, h[i]);
        lh = fminf(lh, h[i]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            mn[d] = fminf(mn[d], __shfl_xor_sync(0xffffffffu, mn[d], o));
            mx[d] = fmaxf(mx[d], __shfl_xor_sync(0xffffffffu, mx[d], o));
        }
        mh = fmaxf(mh, __shfl_xor_sync(0xffffffffu, mh, o));
        lh = fminf(lh, __shfl_xor_sync(0xffffffffu, lh, o));
    }
    __shared__ float s[8][8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) {
        for (int d = 0; d < 3; ++d) {
            s[warp][d] = mn[d];
            s[warp][3 + d] = mx[d];
        }
        s[warp][6] = mh;
        s[warp][7] = lh;
    }
    __syncthreads();
    if (threadIdx.x < 8) {
        int k = threadIdx.x;
        float v = s[0][k];
        for (int w = 1; w < (int)(blockDim.x >> 5); ++w)
            v = (k < 3 || k == 7) ? fminf(v, s[w][k]) : fmaxf(v, s[w][k]);
        part[blockIdx.x * 8 + k] = v;
    }
}

// Cell keys straight from caller-layout positions x[n*DIM].
template <int DIM>
__global__ void k_keys_raw(const float* __restrict__ x, int n, const DevGrid* __restrict__ gp,
                           int* __restrict__ out) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    DevGrid g = *gp;
    const float4 a = make_float4(x[(size_t)DIM * i], x[(size_t)DIM * i + 1],
                                 DIM == 3 ? x[(size_t)DIM * i + 2] : 0.f, 0.f);
    out[i] = (int)cell_key<DIM>(a, g);
}

// Cell keys only (caller order), for the cell-id entry point.
template <int DIM>
__global__ void k_keys_only(const float4* __restrict__ xh, int n, const DevGrid* __restrict__ gp,
                            int* __restrict__ out) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    DevGrid g = *gp;
    out[i] = (int)cell_key<DIM>(xh[i], g);
}

// ---------------------------------------------------------------------------
// LSD radix sort, reduce-then-scan (no inter-block waiting): the mirror ghosts' wall
// grid and the output order of open runs.
// ---------------------------------------------------------------------------
static __global__ void __launch_bounds__(kSortThreads)
    k_radix_hist(const unsigned* __restrict__ keys, int n, int shift, unsigned* __restrict__ hist,
                 int num_tiles) {
    __shared__ unsigned sh[kRadix];
    sh[threadIdx.x] = 0;
    __syncthreads();
    const int base = blockIdx.x * kSortTile;
#pragma unroll
    for (int k = 0; k < kSortItems; ++k) {
        int i = base + k * kSortThreads + threadIdx.x;
        if (i < n) atomicAdd(&sh[(keys[i] >> shift) & 255u], 1u);
    }
    __syncthreads();
    hist[threadIdx.x * num_tiles + blockIdx.x] = sh[threadIdx.x];
}

// Block d: exclusive scan of the tile counts of digit d; total per digit.
static __global__ void __launch_bounds__(256)
    k_radix_scan(unsigned* __restrict__ hist, int num_tiles, unsigned* __restrict__ dtotal) {
    __shared__ unsigned s_warp[32];
    __shared__ unsigned s_total;
    unsigned* row = hist + (size_t)blockIdx.x * num_tiles;
    const int per = (num_tiles + blockDim.x - 1) / blockDim.x;
    const int b = threadIdx.x * per;
    const int e = min(b + per, num_tiles);
    unsigned sum = 0;
    for (int i = b; i < e; ++i) sum += row[i];
    unsigned off = block_excl_scan<256>(sum, s_warp, &s_total);
    for (int i = b; i < e; ++i) {
        unsigned c = row[i];
        row[i] = off;
        off += c;
    }
    if (threadIdx.x == 0) dtotal[blockIdx.x] = s_total;
}

// Stable scatter of one tile by one 8-bit digit. vals_in == nullptr means
// the values are the slot indices themselves.
static __global__ void __launch_bounds__(kSortThreads)
    k_radix_scatter(const unsigned* __restrict__ keys_in, const int* __restrict__ vals_in,
                    unsigned* __restrict__ keys_out, int* __restrict__ vals_out, int n, int shift,
                    const unsigned* __restrict__ hist, const unsigned* __restrict__ dtotal,
                    int num_tiles) {
    __shared__ unsigned s_warp[32];
    __shared__ unsigned s_base[kRadix];
    __shared__ unsigned s_tstart[kRadix];
    __shared__ unsigned s_wcnt[kSortThreads / 32][kRadix];
    __shared__ unsigned s_keys[kSortTile];
    __shared__ int s_vals[kSortTile];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tile = blockIdx.x;
    const int tile_base = tile * kSortTile;
    const int tile_n = min(kSortTile, n - tile_base);

    unsigned excl = block_excl_scan<kSortThreads>(dtotal[tid], s_warp);
    s_base[tid] = excl + hist[(size_t)tid * num_tiles + tile];
#pragma unroll
    for (int w = 0; w < kSortThreads / 32; ++w) s_wcnt[w][tid] = 0;
    __syncthreads();

    unsigned mykey[kSortItems];
    int myval[kSortItems];
    unsigned myrank[kSortItems];
#pragma unroll
    for (int it = 0; it < kSortItems; ++it) {
        const int idx = warp * (32 * kSortItems) + it * 32 + lane;
        const bool valid = idx < tile_n;
        unsigned key = valid ? keys_in[tile_base + idx] : 0u;
        int val = valid ? (vals_in ? vals_in[tile_base + idx] : tile_base + idx) : 0;
        unsigned d = (key >> shift) & 255u;
        unsigned peers = __match_any_sync(0xffffffffu, valid ? d : 0x100u);
        unsigned lt = peers & ((1u << lane) - 1u);
        unsigned base = valid ? s_wcnt[warp][d] : 0u;
        __syncwarp();
        if (valid && lt == 0u) s_wcnt[warp][d] = base + __popc(peers);
        __syncwarp();
        mykey[it] = key;
        myval[it] = val;
        myrank[it] = base + __popc(lt);
    }
    __syncthreads();
    unsigned run = 0;
#pragma unroll
    for (int w = 0; w < kSortThreads / 32; ++w) {
        unsigned c = s_wcnt[w][tid];
        s_wcnt[w][tid] = run;
        run += c;
    }
    unsigned ts = block_excl_scan<kSortThreads>(run, s_warp);
    s_tstart[tid] = ts;
    __syncthreads();
#pragma unroll
    for (int it = 0; it < kSortItems; ++it) {
        const int idx = warp * (32 * kSortItems) + it * 32 + lane;
        if (idx < tile_n) {
            unsigned d = (mykey[it] >> shift) & 255u;
            unsigned pos = s_tstart[d] + s_wcnt[warp][d] + myrank[it];
            s_keys[pos] = mykey[it];
            s_vals[pos] = myval[it];
        }
    }
    __syncthreads();
    for (int i = tid; i < tile_n; i += kSortThreads) {
        unsigned key = s_keys[i];
        unsigned d = (key >> shift) & 255u;
        unsigned dst = s_base[d] + (unsigned)i - s_tstart[d];
        keys_out[dst] = key;
        vals_out[dst] = s_vals[i];
    }
}

// start[c] = first sorted slot of cell c (the number of keys below c), for c in
// [0, ncells]; empty cells get start[c] == start[c+1]. One thread per slot
// s in [0, n]: slot s is the first slot of every cell in (key[s-1], key[s]]
// (slot n: of every cell after the last key, up to ncells), so each entry is
// written exactly once. Runs longer than a warp (empty regions of the grid;
// neighbouring slots often own one each, e.g. the empty rows between two walls)
// are queued in shared memory and written by the whole block, 256 entries at a
// time. Entries past `cap` (the table's last index) are never written.
constexpr int kCellStartThreads = 256;

static __global__ void __launch_bounds__(kCellStartThreads)
    k_cell_start(const unsigned* __restrict__ keys, int n, const int* __restrict__ ncells_total,
                 int cap, int* __restrict__ start) {
    __shared__ int q_lo[kCellStartThreads], q_hi[kCellStartThreads], q_s[kCellStartThreads];
    __shared__ int q_n;
    if (threadIdx.x == 0) q_n = 0;
    __syncthreads();
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    const bool valid = s <= n;
    int lo = 0, hi = -1;  // cells [lo, hi] start at slot s
    if (valid) {
        const int nc = min(*ncells_total, cap);
        lo = (s == 0) ? 0 : (int)__ldg(keys + s - 1) + 1;
        hi = (s == n) ? nc : (int)__ldg(keys + s);
        hi = min(hi, cap);
    }
    if (hi - lo + 1 <= 32) {
        for (int c = lo; c <= hi; ++c) start[c] = s;
    } else {
        const int k = atomicAdd(&q_n, 1);  // at most one entry per thread
        q_lo[k] = lo;
        q_hi[k] = hi;
        q_s[k] = s;
    }
    __syncthreads();
    const int nq = q_n;
    for (int q = 0; q < nq; ++q) {
        const int bs = q_s[q], bhi = q_hi[q];
        for (int c = q_lo[q] + (int)threadIdx.x; c <= bhi; c += kCellStartThreads) start[c] = bs;
    }
}

// ---------------------------------------------------------------------------
// Counting sort of the particles by (cell, previous slot): five launches, or four
// with one scan tile, against 4 x passes + 1 of the radix sort it replaced (three
// passes for 2^17 to 2^24 cells: 13). Small systems are bound by those launches'
// latency; large ones moved every key and slot three times.
// Measured, grid and sort: 42 k particles 49 -> 17 us, 2.03 M (13.8 M cells, every
// slot moved) 0.20 -> 0.09 ms; the 42 k step call 115 -> 87 us.
//
// The cell of a particle takes its place from a counter (any order); the ranks
// within a cell are then set by the previous slot, so the order does not depend
// on the counters' timing and equals the stable sort's. Ranking reads the cell's
// m members (4 bytes each) for each of them, as many as the neighbour passes test for
// each fluid particle there; in a cell crowded with walls it reads more than they do.
// ---------------------------------------------------------------------------
constexpr int kScanThreads = 256;
constexpr int kScanTile = 32 * kScanThreads;  // cells of one scan CTA

// Cell of every slot, its arrival number there, and the cells' counts (cnt zero
// before; k_cell_scan zeroes it again). No grid (g.ok == 0): nothing is counted.
template <int DIM>
__global__ void __launch_bounds__(256)
    k_cell_count(const float4* __restrict__ xh, int n, const DevGrid* __restrict__ gp,
                 unsigned* __restrict__ keys, int* __restrict__ arrival, int* __restrict__ cnt,
                 const int* __restrict__ resort) {
    if (sort_skipped(resort)) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const DevGrid g = *gp;
    const unsigned key = cell_key<DIM>(xh[i], g);
    keys[i] = key;
    arrival[i] = g.ok ? atomicAdd(cnt + key, 1) : i;
}

// One grid per instance. An instance without a grid keeps its slots (they are
// contiguous, before and after a sort); its particles count for the cell its
// cells would start at, so the other instances' slots follow.
template <int DIM>
__global__ void __launch_bounds__(256)
    k_cell_count_batch(const float4* __restrict__ xh, const int* __restrict__ inst, int n,
                       const DevGrid* __restrict__ grids, unsigned* __restrict__ keys,
                       int* __restrict__ arrival, int* __restrict__ cnt) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const unsigned key = cell_key<DIM>(xh[i], grids[inst[i]]);
    keys[i] = key;
    arrival[i] = atomicAdd(cnt + key, 1);
}

// Particles of each scan tile (skipped when one tile holds every cell).
static __global__ void __launch_bounds__(kScanThreads)
    k_cell_sums(const int* __restrict__ cnt, const int* __restrict__ ncells_total, int cap,
                int* __restrict__ sums, const int* __restrict__ resort) {
    if (sort_skipped(resort)) return;
    const int nc = min(*ncells_total, cap);
    if (blockIdx.x * kScanTile > nc) return;
    __shared__ int sw[kScanThreads / 32];
    const int4* c4 = reinterpret_cast<const int4*>(cnt + (size_t)blockIdx.x * kScanTile);
    int v = 0;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const int4 a = c4[q * kScanThreads + threadIdx.x];
        v += (a.x + a.y) + (a.z + a.w);
    }
    v = __reduce_add_sync(0xffffffffu, v);
    if ((threadIdx.x & 31) == 0) sw[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        int t = 0;
        for (int w = 0; w < kScanThreads / 32; ++w) t += sw[w];
        sums[blockIdx.x] = t;
    }
}

// start[c] = particles in the cells below c, c in [0, ncells]. Each CTA adds up the
// tiles before its own: a few thousand sums for tens of millions of cells, 131,072 for the
// 2^30 a table may hold. A sparse system, 42 k particles over 2.7e8 cells: 0.70 ms a step
// in all (20 ms with the radix sort's cell table). A warp owns 1,024 consecutive cells,
// 128 per step.
static __global__ void __launch_bounds__(kScanThreads)
    k_cell_scan(int* __restrict__ cnt, const int* __restrict__ ncells_total, int cap,
                const int* __restrict__ sums, int* __restrict__ start,
                const int* __restrict__ resort) {
    if (sort_skipped(resort)) return;
    const int nc = min(*ncells_total, cap);
    if (blockIdx.x * kScanTile > nc) return;
    __shared__ int sw[kScanThreads / 32], sb[kScanThreads / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int before = 0;
    for (int b = threadIdx.x; b < (int)blockIdx.x; b += kScanThreads) before += sums[b];
    before = __reduce_add_sync(0xffffffffu, before);
    const size_t c0 = (size_t)blockIdx.x * kScanTile + (size_t)warp * 1024;
    int4* c4 = reinterpret_cast<int4*>(cnt + c0);
    int4 a[8];
    int off[8], run = 0;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        a[q] = c4[q * 32 + lane];
        c4[q * 32 + lane] = make_int4(0, 0, 0, 0);
        const int mine = (a[q].x + a[q].y) + (a[q].z + a[q].w);
        const int inc = (int)warp_incl_scan((unsigned)mine);
        off[q] = run + inc - mine;
        run += __shfl_sync(0xffffffffu, inc, 31);
    }
    if (lane == 0) {
        sw[warp] = run;
        sb[warp] = before;
    }
    __syncthreads();
    int base = 0;
    for (int w = 0; w < kScanThreads / 32; ++w) {
        base += sb[w];
        if (w < warp) base += sw[w];
    }
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const size_t c = c0 + (size_t)(q * 32 + lane) * 4;
        int4 o;
        o.x = base + off[q];
        o.y = o.x + a[q].x;
        o.z = o.y + a[q].y;
        o.w = o.z + a[q].z;
        if (c + 3 <= (size_t)nc) {
            *reinterpret_cast<int4*>(start + c) = o;
        } else {
            if (c <= (size_t)nc) start[c] = o.x;
            if (c + 1 <= (size_t)nc) start[c + 1] = o.y;
            if (c + 2 <= (size_t)nc) start[c + 2] = o.z;
        }
    }
}

// The particles of each cell, in order of arrival, and their cells.
static __global__ void __launch_bounds__(256)
    k_cell_place(const unsigned* __restrict__ keys, const int* __restrict__ arrival,
                 const int* __restrict__ start, const DevGrid* __restrict__ gp, int n,
                 int* __restrict__ placed, unsigned* __restrict__ skeys,
                 const int* __restrict__ resort) {
    if (sort_skipped(resort)) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const unsigned key = keys[i];
    const int at = (gp && !gp->ok) ? i : start[key] + arrival[i];
    placed[at] = i;
    skeys[at] = key;
}

// perm: the particles of each cell by their previous slot. xsort (may be null):
// their positions in that order, for the list build. inst, grids: batches (gp null).
static __global__ void __launch_bounds__(256)
    k_cell_rank(const int* __restrict__ placed, const unsigned* __restrict__ skeys,
                const int* __restrict__ start, const DevGrid* __restrict__ gp, int n,
                int* __restrict__ perm, const float4* __restrict__ xh, float4* __restrict__ xsort,
                const int* __restrict__ inst, const DevGrid* __restrict__ grids,
                const int* __restrict__ resort) {
    if (sort_skipped(resort)) return;
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    const int i = placed[s];
    int at = i;
    if (gp ? gp->ok != 0 : grids[inst[i]].ok != 0) {
        const unsigned key = skeys[s];
        const int b = __ldg(start + key), e = __ldg(start + key + 1);
        at = b;
        for (int q = b; q < e; ++q) at += __ldg(placed + q) < i ? 1 : 0;
    }
    perm[at] = i;
    if (xsort) xsort[at] = xh[i];
}

// ---------------------------------------------------------------------------
// State movement
// ---------------------------------------------------------------------------
// Caller arrays -> A, in two parts: what the grid and sort read (positions,
// h; the 2D mass rides in xh.z) and the rest. The input density and pressure
// of a fluid particle are read only where the step uses them (rho_fl, p_fl):
// summation density and the equation of state replace them otherwise.
template <int DIM>
__device__ __forceinline__ void gather_pos_one(int i, const float* __restrict__ x,
                                               const float* __restrict__ m,
                                               const float* __restrict__ h, StateA& A) {
    if (DIM == 2) A.xh[i] = make_float4(x[2 * i], x[2 * i + 1], m[i], h[i]);
    else A.xh[i] = make_float4(x[3 * i], x[3 * i + 1], x[3 * i + 2], h[i]);
    A.id[i] = i;
}
template <int DIM>
__device__ __forceinline__ void gather_rest_one(int i, const float* __restrict__ v,
                                                const float* __restrict__ m,
                                                const float* __restrict__ rho,
                                                const float* __restrict__ p,
                                                const float* __restrict__ u,
                                                const int* __restrict__ itype,
                                                const float* __restrict__ dvdt,
                                                const float* __restrict__ dudt, StateA& A,
                                                bool rho_fl, bool p_fl) {
    const int it = itype[i];
    if (DIM == 2) {
        A.vm[i] = make_float4(v[2 * i], v[2 * i + 1], 0.f, 0.f);
        A.ap[i] = dvdt ? make_float4(dvdt[2 * i], dvdt[2 * i + 1], 0.f, dudt[i])
                       : make_float4(0.f, 0.f, 0.f, 0.f);
    } else {
        A.vm[i] = make_float4(v[3 * i], v[3 * i + 1], v[3 * i + 2], m[i]);
        A.ap[i] = dvdt ? make_float4(dvdt[3 * i], dvdt[3 * i + 1], dvdt[3 * i + 2], dudt[i])
                       : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    A.u[i] = u[i];
    A.rho[i] = (rho_fl || it <= 0) ? rho[i] : 0.f;
    A.p[i] = (p_fl || it <= 0) ? p[i] : 0.f;
    A.itype[i] = it;
}

template <int DIM>
__global__ void k_gather_in(const float* __restrict__ x, const float* __restrict__ v,
                            const float* __restrict__ m, const float* __restrict__ rho,
                            const float* __restrict__ p, const float* __restrict__ u,
                            const float* __restrict__ h, const int* __restrict__ itype,
                            const float* __restrict__ dvdt, const float* __restrict__ dudt,
                            StateA A, int n, const int* __restrict__ inst0, int rho_fl,
                            int p_fl, unsigned* __restrict__ sort_next) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (i == 0) *sort_next = 1u;  // A is in caller order now (lazy sorting)
    if (inst0) A.inst[i] = inst0[i];
    gather_pos_one<DIM>(i, x, m, h, A);
    gather_rest_one<DIM>(i, v, m, rho, p, u, itype, dvdt, dudt, A, rho_fl, p_fl);
}

// The two parts apart: a host-memory call loads the positions first and the
// rest from a few CTAs on a second stream while the sort runs.
template <int DIM>
__global__ void k_gather_pos(const float* __restrict__ x, const float* __restrict__ m,
                             const float* __restrict__ h, StateA A, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) gather_pos_one<DIM>(i, x, m, h, A);
}
template <int DIM>
__global__ void k_gather_rest(const float* __restrict__ v, const float* __restrict__ m,
                              const float* __restrict__ rho, const float* __restrict__ p,
                              const float* __restrict__ u, const int* __restrict__ itype,
                              const float* __restrict__ dvdt, const float* __restrict__ dudt,
                              StateA A, int n, int rho_fl, int p_fl) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        gather_rest_one<DIM>(i, v, m, rho, p, u, itype, dvdt, dudt, A, rho_fl, p_fl);
}

// Positions and h only (neighbour / cell-id entry points).
template <int DIM>
__global__ void k_load_xh(const float* __restrict__ x, const float* __restrict__ h, StateA A,
                          int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (DIM == 2) A.xh[i] = make_float4(x[2 * i], x[2 * i + 1], 0.f, h[i]);
    else A.xh[i] = make_float4(x[3 * i], x[3 * i + 1], x[3 * i + 2], h[i]);
    A.id[i] = i;
}

// inv[id[s]] = s: the cell-order slot of each caller index.
// dst[id[s]] = src[s]: a slot-order array back to caller order.
static __global__ void k_scatter_by_id(const float* __restrict__ src, const int* __restrict__ id,
                                float* __restrict__ dst, int n) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s < n) dst[id[s]] = src[s];
}

// Smoothing lengths of A in caller order.
static __global__ void k_hsml_out(StateA A, float* __restrict__ h, int n) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s < n) h[A.id[s]] = A.xh[s].w;
}

static __global__ void k_invert_ids(const int* __restrict__ id, int* __restrict__ inv, int n) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s < n) inv[id[s]] = s;
}

// A -> caller arrays walking the caller order: the form for caller arrays in
// host memory that the device maps, where every write crosses the host link, and for
// large systems' arrays in device memory (kGatherOutMin).
// The interleaved x, v, dv/dt of a block's kScatterSeq particles are staged in
// shared memory and written as one contiguous run each (consecutive threads,
// consecutive addresses: whole lines, no alignment needed); the reads of A are
// the scattered side.
constexpr int kScatterSeq = 256;

// The output density and pressure of a summation-density iteration, final
// after the density pass (the force pass copies them): written to the caller's
// arrays from a few CTAs on a second stream while the force pass runs. inv is
// the inverse of B.id.
static __global__ void k_scatter_rp(StateB B, const int* __restrict__ inv, int n, float* __restrict__ rho,
                             float* __restrict__ p) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int s = inv[i];
        rho[i] = B.rp[s].x;
        p[i] = B.p[s];
    }
}

// count floats of shared memory to dst by the block's threads, the first of them t = 0:
// 16 bytes a store where dst allows (a block's run starts at a multiple of 16 bytes
// from its array). Host arrays, 2.03 M particles over the host link: 483 us with 4
// bytes a store, now 422 (154 GB/s).
__device__ __forceinline__ void store_run(float* __restrict__ dst, const float* sm, int count, int t) {
    int k = t;
    if ((reinterpret_cast<uintptr_t>(dst) & 15u) == 0) {
        const int q = count >> 2;
        for (; k < q; k += kScatterSeq) reinterpret_cast<float4*>(dst)[k] = reinterpret_cast<const float4*>(sm)[k];
        k = 4 * q + t;
    }
    for (; k < count; k += kScatterSeq) dst[k] = sm[k];
}

template <int DIM>
__global__ void __launch_bounds__(kScatterSeq)
    k_scatter_out_seq(StateA A, const int* __restrict__ inv, int n, float* __restrict__ x,
                      float* __restrict__ v, float* __restrict__ rho, float* __restrict__ p,
                      float* __restrict__ u, float* __restrict__ dvdt,
                      float* __restrict__ dudt) {
    __shared__ alignas(16) float sx[DIM * kScatterSeq], sv[DIM * kScatterSeq], sa[DIM * kScatterSeq];
    __shared__ alignas(16) float sc[4][kScatterSeq];  // u, dudt, rho, p
    const int t = threadIdx.x;
    const int i0 = blockIdx.x * kScatterSeq;
    const int i = i0 + t;
    if (i < n) {
        const int s = inv[i];
        const float4 a = A.xh[s], b = A.vm[s], r = A.ap[s];
        sx[DIM * t] = a.x;
        sx[DIM * t + 1] = a.y;
        sv[DIM * t] = b.x;
        sv[DIM * t + 1] = b.y;
        sa[DIM * t] = r.x;
        sa[DIM * t + 1] = r.y;
        if (DIM == 3) {
            sx[3 * t + 2] = a.z;
            sv[3 * t + 2] = b.z;
            sa[3 * t + 2] = r.z;
        }
        sc[0][t] = A.u[s];
        sc[1][t] = r.w;
        if (rho) {  // null: already with the caller
            sc[2][t] = A.rho[s];
            sc[3][t] = A.p[s];
        }
    }
    __syncthreads();
    const int m = min(kScatterSeq, n - i0);
    const size_t o = (size_t)DIM * i0;
    store_run(x + o, sx, DIM * m, t);
    store_run(v + o, sv, DIM * m, t);
    store_run(dvdt + o, sa, DIM * m, t);
    // two warps an array
    store_run(u + i0, sc[0], m, t);
    store_run(dudt + i0, sc[1], m, (t + 64) & (kScatterSeq - 1));
    if (rho) {
        store_run(rho + i0, sc[2], m, (t + 128) & (kScatterSeq - 1));
        store_run(p + i0, sc[3], m, (t + 192) & (kScatterSeq - 1));
    }
}

template <int DIM>
__global__ void k_scatter_out(StateA A, int n, float* __restrict__ x, float* __restrict__ v,
                              float* __restrict__ rho, float* __restrict__ p,
                              float* __restrict__ u, float* __restrict__ dvdt,
                              float* __restrict__ dudt) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    const int i = A.id[s];
    const float4 a = A.xh[s], b = A.vm[s], r = A.ap[s];
    x[DIM * i] = a.x;
    x[DIM * i + 1] = a.y;
    v[DIM * i] = b.x;
    v[DIM * i + 1] = b.y;
    dvdt[DIM * i] = r.x;
    dvdt[DIM * i + 1] = r.y;
    if (DIM == 3) {
        x[3 * i + 2] = a.z;
        v[3 * i + 2] = b.z;
        dvdt[3 * i + 2] = r.z;
    }
    dudt[i] = r.w;
    u[i] = A.u[s];
    rho[i] = A.rho[s];
    p[i] = A.p[s];
}

// Cell-ordered working set + leapfrog predictor (time_integration.f:136-154).
template <int DIM>
// An iteration that does not sort keeps the slot order (perm = identity).
// only_sorted: an iteration that does not sort skips the copy (the passes of
// such an iteration read A themselves, FusedSrc).
__global__ void k_reorder_dim(StateA A, const int* __restrict__ perm, StateB B, StepArgs S,
                              int n, const int* __restrict__ resort = nullptr,
                              bool only_sorted = false) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    const bool sorted = !sort_skipped(resort);
    if (only_sorted && !sorted) return;
    const int j = sorted ? perm[s] : s;
    const float4 xh = A.xh[j];
    if (sorted && B.xsort) B.xsort[s] = xh;
    float4 vm = A.vm[j];
    float u = A.u[j];
    const int it = A.itype[j];
    B.vmin[s] = make_float4(vm.x, vm.y, vm.z, u);
    float ulo = 0.f;
    if (it > 0 && S.hdt != 0.f) {
        const float4 ap = A.ap[j];
        vm.x = fmaf(S.hdt, ap.x, vm.x);
        vm.y = fmaf(S.hdt, ap.y, vm.y);
        if (DIM == 3) vm.z = fmaf(S.hdt, ap.z, vm.z);
        // u + dt/2 du kept as hi + lo: art_heat differences u_i - u_j of nearly
        // equal energies would otherwise carry the rounding of u_half.
        const sph::ff uh = sph::two_sum(u, __fmul_rn(S.hdt, ap.w));
        u = uh.hi;
        ulo = uh.lo;
        if (u < 0.f) {
            u = 0.f;
            ulo = 0.f;
        }
    }
    if (B.ulo) B.ulo[s] = ulo;
    // Continuity density: rho + dt/2 drho/dt as hi + lo (time_integration.f:
    // 144-147), the start density kept for the corrector.
    float rho = A.rho[j], rlo = 0.f;
    if (B.q) B.q[s] = rho;
    if (S.dform == 1 && it > 0 && S.hdt != 0.f) {
        const sph::ff rh = sph::two_sum(rho, __fmul_rn(S.hdt, A.drho[j]));
        rho = rh.hi;
        rlo = rh.lo;
    }
    if (B.rlo) B.rlo[s] = rlo;
    B.xh[s] = xh;
    B.vm[s] = vm;
    B.rp[s] = make_float4(rho, 0.f, u, 0.f);
    B.p[s] = A.p[j];
    B.itype[s] = it;
    B.id[s] = A.id[j];
}

// Positions only (neighbour entry point).
static __global__ void k_reorder_xh(StateA A, const int* __restrict__ perm, StateB B, int n) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    const int j = perm[s];
    B.xh[s] = A.xh[j];
    B.id[s] = A.id[j];
}

// ---------------------------------------------------------------------------
// Batched grid, hash and reorder (one cell grid per instance).
// ---------------------------------------------------------------------------
// Bbox partial {min[3], max[3], max h} of every work item.
static __global__ void __launch_bounds__(kPassThreads)
    k_bbox_items(const float4* __restrict__ xh, const WorkItem* __restrict__ items, int dim,
                 float* __restrict__ part) {
    const WorkItem w = items[blockIdx.x];
    const int s = w.s0 + threadIdx.x;
    float v[8] = {FLT_MAX, FLT_MAX, FLT_MAX, -FLT_MAX, -FLT_MAX, -FLT_MAX, 0.f, FLT_MAX};
    if (s < w.s1) {
        const float4 a = xh[s];
        v[0] = v[3] = a.x;
        v[1] = v[4] = a.y;
        if (dim == 3) v[2] = v[5] = a.z;
        v[6] = v[7] = a.w;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const float t = __shfl_xor_sync(0xffffffffu, v[k], o);
            v[k] = (k < 3 || k == 7) ? fminf(v[k], t) : fmaxf(v[k], t);
        }
    __shared__ float sw[kPassThreads / 32][8];
    if ((threadIdx.x & 31) == 0)
        for (int k = 0; k < 8; ++k) sw[threadIdx.x >> 5][k] = v[k];
    __syncthreads();
    if (threadIdx.x < 8) {
        const int k = threadIdx.x;
        float r = sw[0][k];
        for (int w2 = 1; w2 < kPassThreads / 32; ++w2) r = (k < 3 || k == 7) ? fminf(r, sw[w2][k]) : fmaxf(r, sw[w2][k]);
        part[blockIdx.x * 8 + k] = r;
    }
}

// Grid of instance blockIdx.x from the partials of its items.
static __global__ void __launch_bounds__(256)
    k_bbox_final_batch(const float* __restrict__ part, const int* __restrict__ inst_items,
                       const DevParams* __restrict__ params, DevGrid* __restrict__ grids,
                       int* __restrict__ ncells_inst, unsigned* __restrict__ flags) {
    __shared__ float sv[8][256];
    const int k = blockIdx.x;
    float v[8] = {FLT_MAX, FLT_MAX, FLT_MAX, -FLT_MAX, -FLT_MAX, -FLT_MAX, 0.f, FLT_MAX};
    for (int b = inst_items[k] + threadIdx.x; b < inst_items[k + 1]; b += blockDim.x)
        for (int q = 0; q < 8; ++q)
            v[q] = (q < 3 || q == 7) ? fminf(v[q], part[b * 8 + q]) : fmaxf(v[q], part[b * 8 + q]);
    for (int q = 0; q < 8; ++q) sv[q][threadIdx.x] = v[q];
    __syncthreads();
    for (int st = blockDim.x / 2; st > 0; st >>= 1) {
        if ((int)threadIdx.x < st)
            for (int q = 0; q < 8; ++q)
                sv[q][threadIdx.x] = (q < 3 || q == 7) ? fminf(sv[q][threadIdx.x], sv[q][threadIdx.x + st])
                                             : fmaxf(sv[q][threadIdx.x], sv[q][threadIdx.x + st]);
        __syncthreads();
    }
    if (threadIdx.x != 0) return;
    const float mm[8] = {sv[0][0], sv[1][0], sv[2][0], sv[3][0],
                         sv[4][0], sv[5][0], sv[6][0], sv[7][0]};
    unsigned fl = 0;
    DevGrid g = grid_from_bbox(mm, params[k], (long long)1 << 30, fl);
    grids[k] = g;
    ncells_inst[k] = g.ok ? g.ncells : 0;
    if (fl) atomicOr(flags, fl);
}

// Cell offsets of the instances in the shared table (exclusive scan of their
// cell counts); a total above the table's capacity disables every grid.
static __global__ void __launch_bounds__(1024)
    k_cell_offsets(const int* __restrict__ ncells_inst, int n_inst, long long capacity,
                   DevGrid* __restrict__ grids, int* __restrict__ total_cells,
                   unsigned* __restrict__ flags) {
    __shared__ unsigned s_warp[32];
    __shared__ unsigned s_total;
    const int per = (n_inst + blockDim.x - 1) / blockDim.x;
    const int b = threadIdx.x * per, e = min(b + per, n_inst);
    unsigned sum = 0;
    for (int k = b; k < e; ++k) sum += (unsigned)ncells_inst[k];
    unsigned off = block_excl_scan<1024>(sum, s_warp, &s_total);
    const bool over = (long long)s_total > capacity;
    for (int k = b; k < e; ++k) {
        grids[k].cell_off = over ? 0 : (int)off;
        if (over) grids[k].ok = 0;
        off += (unsigned)ncells_inst[k];
    }
    if (threadIdx.x == 0) {
        *total_cells = over ? (int)capacity : (int)s_total;
        if (over) atomicOr(flags, (unsigned)FLAG_GRID_OVERFLOW);
    }
}

// Cell-ordered working set + leapfrog predictor, per-instance time step.
template <int DIM>
__global__ void k_reorder_batch(StateA A, const int* __restrict__ perm, StateB B,
                                const DevParams* __restrict__ params, const int* __restrict__ its,
                                int n) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    const int j = perm[s];
    const int k = A.inst[j];
    const float hdt = (*its == 1) ? 0.f : 0.5f * __ldg(&params[k].dt);
    const float4 xh = A.xh[j];
    float4 vm = A.vm[j];
    float u = A.u[j];
    const int it = A.itype[j];
    B.vmin[s] = make_float4(vm.x, vm.y, vm.z, u);
    float ulo = 0.f;
    if (it > 0 && hdt != 0.f) {
        const float4 ap = A.ap[j];
        vm.x = fmaf(hdt, ap.x, vm.x);
        vm.y = fmaf(hdt, ap.y, vm.y);
        if (DIM == 3) vm.z = fmaf(hdt, ap.z, vm.z);
        const sph::ff uh = sph::two_sum(u, __fmul_rn(hdt, ap.w));
        u = uh.hi;
        ulo = uh.lo;
        if (u < 0.f) {
            u = 0.f;
            ulo = 0.f;
        }
    }
    B.ulo[s] = ulo;
    B.xh[s] = xh;
    B.vm[s] = vm;
    B.rp[s] = make_float4(A.rho[j], 0.f, u, 0.f);
    B.p[s] = A.p[j];
    B.itype[s] = it;
    B.id[s] = A.id[j];
    B.inst[s] = k;
}

static __global__ void k_advance_its(int* its) { *its += 1; }

// ---------------------------------------------------------------------------
// Neighbour-cell iteration
// ---------------------------------------------------------------------------
struct CellCoord {
    int c[3];
};

template <int DIM>
__device__ __forceinline__ CellCoord decode_key(unsigned key, const DevGrid& g) {
    CellCoord cc;
    key -= (unsigned)g.cell_off;
    cc.c[0] = (int)(key % (unsigned)g.n[0]);
    unsigned t = key / (unsigned)g.n[0];
    if (DIM == 2) {
        cc.c[1] = (int)t;
        cc.c[2] = 0;
    } else {
        cc.c[1] = (int)(t % (unsigned)g.n[1]);
        cc.c[2] = (int)(t / (unsigned)g.n[1]);
    }
    return cc;
}

// Difference x_i - x_j (minimum image) and the exact pair test.
template <int DIM>
__device__ __forceinline__ bool pair_delta(const float4& xi, const float4& xj, const DevGrid& g,
                                           float* d, float& dr2) {
    d[0] = __fsub_rn(xi.x, xj.x);
    d[1] = __fsub_rn(xi.y, xj.y);
    d[2] = (DIM == 3) ? __fsub_rn(xi.z, xj.z) : 0.f;
#pragma unroll
    for (int a = 0; a < DIM; ++a)
        if (g.periodic[a]) d[a] = sph::min_image(d[a], g.L[a], g.half[a]);
    dr2 = sph::dist2_exact<DIM>(d);
    return sph::within_support(dr2, xi.w, xj.w);
}

// Exact pair difference x_i - x_j = dh + dl per axis, minimum image applied
// exactly on periodic axes (the wrap decision is the pair test's).
template <int DIM>
__device__ __forceinline__ void exact_delta(const float4& xi, const float4& xj, const DevGrid& g,
                                            float* dh, float* dl) {
    const float a[3] = {xi.x, xi.y, xi.z}, b[3] = {xj.x, xj.y, xj.z};
#pragma unroll
    for (int k = 0; k < DIM; ++k) {
        sph::ff s = sph::two_diff(a[k], b[k]);
        if (g.periodic[k]) {
            if (s.hi > g.half[k]) {
                sph::ff u = sph::two_sum(s.hi, -g.L[k]);
                s.hi = u.hi;
                s.lo = __fadd_rn(s.lo, u.lo);
            } else if (s.hi < -g.half[k]) {
                sph::ff u = sph::two_sum(s.hi, g.L[k]);
                s.hi = u.hi;
                s.lo = __fadd_rn(s.lo, u.lo);
            }
            s = sph::two_sum(s.hi, s.lo);  // a wrapped difference's residual may exceed an ulp
        }
        dh[k] = s.hi;
        dl[k] = s.lo;
    }
}

// Minimum image of two differences x_i - x_a, x_i - x_b along axis k, for the force
// passes: a difference that wraps is the exact one rounded once (exact_delta); one
// that does not is already.
__device__ __forceinline__ f2 min_image2(f2 d, float xi, float xa, float xb, const DevGrid& g, int k) {
    if (fabsf(d.x) > g.half[k]) {
        const sph::ff s = sph::two_diff(xi, xa);
        const sph::ff u = sph::two_sum(s.hi, s.hi > 0.f ? -g.L[k] : g.L[k]);
        d.x = __fadd_rn(u.hi, __fadd_rn(s.lo, u.lo));
    }
    if (fabsf(d.y) > g.half[k]) {
        const sph::ff s = sph::two_diff(xi, xb);
        const sph::ff u = sph::two_sum(s.hi, s.hi > 0.f ? -g.L[k] : g.L[k]);
        d.y = __fadd_rn(u.hi, __fadd_rn(s.lo, u.lo));
    }
    return d;
}

template <int DIM>
__device__ __forceinline__ sph::ff ff_pow_dim(sph::ff ih) {
    sph::ff a = sph::ff_sqr(ih);
    if (DIM == 3) a = sph::ff_mul(a, ih);
    return a;
}

template <int DIM>
__device__ __forceinline__ float pow_grad(float ih) {
    float ih2 = __fmul_rn(ih, ih);
    float ih4 = __fmul_rn(ih2, ih2);
    return DIM == 2 ? ih4 : __fmul_rn(ih4, ih);
}

// ---------------------------------------------------------------------------
// Candidate cursor and per-thread neighbour lists.
//
// A pass walks the candidate slots of its particle row by row (a "row" is the
// contiguous slot range of the 3 x-adjacent cells at one (y, z), or a single
// cell on a periodic x axis), tests them, and appends the neighbours to a list
// in shared memory (slot-major [t][thread], conflict-free). The physics then
// runs over the lists in a warp-converged loop, so lanes do not idle on
// candidates that failed the pair test. Lists hold kListCap entries; a
// particle with more neighbours takes several rounds.
// ---------------------------------------------------------------------------
constexpr int kListCap = 32;      // force pass list
// Neighbour-list entries per particle of a lazily sorting context (pairs
// within h_i + h_j + skin; the lattice counts are ~20 / ~85 at a 10% skin,
// ~28 / ~125 at 40%); a particle with more walks its cells. Each must fit the
// neighbour bits of one lane (mask_words * 32).
constexpr int kListCap2 = 64;
constexpr int kListCap3 = 256;
// Blocks of four per slot: the capacity's and room for the far entries' own while a
// list is built.
__host__ __device__ constexpr int list_blocks(int lcap) { return lcap / 4 + 2; }
constexpr int kRing = 16;    // entries a thread of the build holds back of each kind
constexpr int kListPad = 3;  // positions readable past the last slot
static_assert(kListCap2 <= 32 * mask_words<2>() && kListCap3 <= 32 * mask_words<3>(),
              "a list's neighbour bits fit one lane's mask");
constexpr int kListCapD = 24;     // density pass: near and far lists each
// With neighbour lists only the particles whose list overflowed fill these
// candidate lists: smaller ones leave the SM's shared storage to L1.
constexpr int kListCapLst = 4;
template <bool LST>
__host__ __device__ constexpr int cap_density() {
    return LST ? kListCapLst : kListCapD;
}
template <bool LST>
__host__ __device__ constexpr int cap_force() {
    return LST ? kListCapLst : kListCap;
}
constexpr int kTestBatch = 4;     // candidate loads issued together

// A warp's blocks of neighbour-list entries (block b of its 32 slots is one run of
// 512 bytes) requested into L2 at once, one line per lane, so the walk's loads hit L2
// instead of waiting on DRAM.
__device__ __forceinline__ void prefetch_list(const int* nlist, int lstride, int s, int entries) {
    const int lane = (int)(threadIdx.x & 31u);
    const int blocks = (__reduce_max_sync(0xffffffffu, entries > 0 ? entries : 0) + 3) >> 2;
    const int s0 = __shfl_sync(0xffffffffu, s, 0) & ~31;
    for (int r = lane; r < 4 * blocks; r += 32)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(nlist + ((size_t)(r >> 2) * lstride + s0) * 4 + (r & 3) * 32));
}
// Block b of slot s; `none` in place of a block past the slot's last.
__device__ __forceinline__ int4 list_block(const int* nlist, int lstride, int s, int b, int blocks,
                                           int none) {
    return b < blocks ? __ldg(reinterpret_cast<const int4*>(nlist) + (size_t)b * lstride + s)
                      : make_int4(none, none, none, none);
}
__host__ __device__ constexpr int blocks_of(int entries) { return entries > 0 ? (entries + 3) >> 2 : 0; }

// A slot's list counts from ncount: near entries (-1: no list, walk the
// cells) and far entries.
__device__ __forceinline__ int list_near(int packed) { return packed >= 0 ? (packed & 0xffff) : -1; }
__device__ __forceinline__ int list_far(int packed) { return packed >= 0 ? (packed >> 16) : 0; }
// 2D density pairs with q = r/h < near_q() are evaluated in float-float, the
// others (W below ~1% of W(0) each, ~8 of ~20 pairs) in FP32. In 3D every pair
// is float-float: ~50 of ~80 pairs lie beyond q = 1.6, and the FP32 rounding of
// their sum (a few 1e-7 of ~1% of rho each) would exceed 1e-5 of the pressure
// of a quiescent flow, whose p is ~1e-5 of rho0 c0^2.
template <int DIM>
__host__ __device__ constexpr float near_q() {
    return DIM == 2 ? 1.6f : 2.0f;
}
// The 2D neighbour lists' split (at the sort): float-float below q = 1.5, under
// a lattice's second neighbours (r = 2 dx, q = 1.54 at h = 1.3 dx), which take
// the FP32 path with the farther ones: 2% of the step for a one-step pressure
// error of 1.5e-6 instead of 5.7e-7 at the cell walk's 1.6 (gate 1e-5).
__host__ __device__ constexpr float list_near_q2() { return 1.5f; }

// Candidate rows: for each (dy, dz) in [-f, f]^(DIM-1) the cells cx-f..cx+f of
// that row are consecutive keys, so one contiguous slot range. On a periodic x
// axis the part past either end (at most one side, as n[0] >= 2f + 1) is a
// second piece. Rows come in (dz, dy, piece) order, the same for every pass.
struct Cursor {
    int k, ke;  // current slot range [k, ke)
    int st;     // row state: dy + 8 (bits 0-3), dz + 8 (bits 4-7), piece (bit 8),
                // piece 0 the in-range cells, 1 the wrapped ones
};

// The cells of the row at (dy, dz) of a cell, from its x = 0 cell on; null outside.
template <int DIM>
__device__ __forceinline__ const int* cell_row(const DevGrid& g, const int* __restrict__ start,
                                               const CellCoord& cc, int dy, int dz) {
    int cy = cc.c[1] + dy, cz = DIM == 3 ? cc.c[2] + dz : 0;
    if (cy < 0 || cy >= g.n[1]) {
        if (!g.periodic[1]) return nullptr;
        cy += cy < 0 ? g.n[1] : -g.n[1];
    }
    if (DIM == 3 && (cz < 0 || cz >= g.n[2])) {
        if (!g.periodic[2]) return nullptr;
        cz += cz < 0 ? g.n[2] : -g.n[2];
    }
    return start + g.cell_off + (cz * g.n[1] + cy) * g.n[0];
}

// The candidates that the bits ch of the density pass name, in candidate order
// (2D, one lane a particle): put(slot, row) for each.
template <class Put>
__device__ __forceinline__ void mask_slots(const uint4& ch, const DevGrid& g, const int* __restrict__ start,
                                           const CellCoord& cc, Put put) {
    unsigned long long lo = ch.x | (unsigned long long)ch.y << 32, hi = ch.z | (unsigned long long)ch.w << 32;
    const int f = g.reach, c0 = max(cc.c[0] - f, 0), c1 = min(cc.c[0] + f, g.n[0] - 1) + 1;
    auto range = [&](const int b, const int e, const int r) {
        for (int k = b; k < e; k += 32) {
            const int n = min(e - k, 32);
            unsigned bits = (unsigned)lo & (0xffffffffu >> (32 - n));
            lo = lo >> n | hi << (64 - n);
            hi >>= n;
            for (; bits; bits &= bits - 1u) put(k + __ffs(bits) - 1, r);
        }
    };
    for (int dy = -f; dy <= f; ++dy) {
        const int* const row = cell_row<2>(g, start, cc, dy, 0);
        if (!row) continue;
        range(__ldg(row + c0), __ldg(row + c1), dy + f);
        if (g.periodic[0]) {
            if (cc.c[0] < f) range(__ldg(row + cc.c[0] - f + g.n[0]), __ldg(row + g.n[0]), dy + f);
            else if (cc.c[0] + f >= g.n[0]) range(__ldg(row), __ldg(row + cc.c[0] + f - g.n[0] + 1), dy + f);
        }
    }
}

template <int DIM>
__device__ __forceinline__ Cursor cursor_begin(const DevGrid& g) {
    Cursor c;
    c.k = c.ke = 0;
    const int dy = -g.reach - 1, dz = (DIM == 3) ? -g.reach : 0;
    c.st = (dy + 8) | ((dz + 8) << 4) | (1 << 8);
    return c;
}

// Advances to the next non-empty range; false when the candidates are
// exhausted (and stays false).
template <int DIM>
__device__ __forceinline__ bool cursor_next(const DevGrid& g, const int* __restrict__ start,
                                            const CellCoord& cc, Cursor& cu) {
    const int f = g.reach;
    const bool px = g.periodic[0] != 0;
    int dy = (cu.st & 15) - 8, dz = ((cu.st >> 4) & 15) - 8, pc = cu.st >> 8;
    bool found = false;
    for (;;) {
        if (px && pc == 0) {
            pc = 1;
        } else {
            pc = 0;
            if (++dy > f) {
                if (DIM == 2 || dz >= f) {
                    dy = f + 1;
                    cu.k = cu.ke = 0;
                    break;
                }
                dy = -f;
                ++dz;
            }
        }
        int cy = cc.c[1] + dy;
        if (cy < 0 || cy >= g.n[1]) {
            if (!g.periodic[1]) continue;
            cy += (cy < 0) ? g.n[1] : -g.n[1];
        }
        int cz = 0;
        if (DIM == 3) {
            cz = cc.c[2] + dz;
            if (cz < 0 || cz >= g.n[2]) {
                if (!g.periodic[2]) continue;
                cz += (cz < 0) ? g.n[2] : -g.n[2];
            }
        }
        const int row = g.cell_off + (cz * g.n[1] + cy) * g.n[0];
        const int cx = cc.c[0];
        int c0, c1;
        if (pc == 0) {
            c0 = max(cx - f, 0);
            c1 = min(cx + f, g.n[0] - 1);
        } else if (cx - f < 0) {
            c0 = cx - f + g.n[0];
            c1 = g.n[0] - 1;
        } else if (cx + f >= g.n[0]) {
            c0 = 0;
            c1 = cx + f - g.n[0];
        } else {
            continue;
        }
        const int kb = __ldg(start + row + c0), ke = __ldg(start + row + c1 + 1);
        if (kb < ke) {
            cu.k = kb;
            cu.ke = ke;
            found = true;
            break;
        }
    }
    cu.st = (dy + 8) | ((dz + 8) << 4) | (pc << 8);
    return found;
}

// Calls fn(k) for every candidate slot k of the particle in cell cc (its own
// slot included; callers skip it).
template <int DIM, class F>
__device__ __forceinline__ void for_candidates(const DevGrid& g, const int* __restrict__ start,
                                               const CellCoord& cc, F&& fn) {
    Cursor cu = cursor_begin<DIM>(g);
    while (cursor_next<DIM>(g, start, cc, cu))
        for (int k = cu.k; k < cu.ke; ++k) fn(k);
}

// Periodic wrap of a drifted coordinate (same branch order as the oracle).
__device__ __forceinline__ float wrap_axis(float c, const DevParams& P, int d, bool& outside) {
    if (!(c < P.period_hi[d])) c = __fsub_rn(c, P.period_L[d]);
    else if (c < P.period_lo[d]) c = __fadd_rn(c, P.period_L[d]);
    if (!(c >= P.period_lo[d] && c < P.period_hi[d])) outside = true;
    return c;
}

__device__ __forceinline__ float fast_sqrt_pos(float x) {
    return x > 0.f ? x * rsqrtf(x) : 0.f;
}

// Lanes of one particle: TPP consecutive threads split its candidates, lane
// `sub` taking slots kb + sub, kb + sub + TPP, ... of every candidate range.
template <int TPP>
__device__ __forceinline__ unsigned group_mask() {
    const unsigned lane = threadIdx.x & 31u;
    return (TPP == 1) ? (1u << lane) : (((1u << TPP) - 1u) << (lane & ~(unsigned)(TPP - 1)));
}

// Sum over the lanes of one particle (xor butterfly; every lane gets the same
// value, a + b being commutative).
template <int TPP>
__device__ __forceinline__ float group_sum(float v) {
#pragma unroll
    for (int o = 1; o < TPP; o <<= 1) v += __shfl_xor_sync(group_mask<TPP>(), v, o);
    return v;
}

// The lane's candidates left in the cursor's current range.
template <int TPP>
__device__ __forceinline__ int lane_len(const Cursor& cu) {
    return cu.k < cu.ke ? (cu.ke - cu.k + TPP - 1) / TPP : 0;
}

// Candidates of a CTA staged in shared memory (staged passes, one thread per
// particle, no periodic axis): slot k of stencil row r sits at k + shift[r].
struct StageView {
    const float4* x;    // xh of the staged slots
    const float4* v;    // density 3D: vm (mass); force 2D: vr; force 3D: vm
    const float4* r;    // force 3D: rp
    const int* shift;   // per stencil row, cursor order
};

// The integrated state A of a lazily sorting context with lean physics, read
// by the passes on the iterations that do not sort: they skip the reorder
// copy into B, apply the leapfrog predictor (time_integration.f:136-154) on
// load, and the force pass writes the next state into the other A buffer.
// rs: the context's lazy-sort flags (which iterations sort).
struct FusedSrc {
    StateA A;
    const int* rs;
    float hdt;  // predictor half step of this iteration
};

// Stencil row of the cursor's current range (non-periodic grids: one piece
// per row), r = (dz + f) (2f + 1) + (dy + f).
template <int DIM>
__device__ __forceinline__ int cursor_row(const Cursor& cu, int f) {
    const int dy = (cu.st & 15) - 8, dz = ((cu.st >> 4) & 15) - 8;
    return DIM == 2 ? dy + f : (dz + f) * (2 * f + 1) + (dy + f);
}

// ---------------------------------------------------------------------------
// Pass 1: summation density (float-float near pairs), Tait EOS, div v.
// ---------------------------------------------------------------------------
// LEAN: the parameters have no physical viscosity and no artificial heat, so
// their operands and branches are compiled out.
// STG: the candidates come from the CTA's staged copy SV (LT: the list entry
// type, staged indices), else from global memory through L1.
// LST: a lazily sorting context's neighbour lists (B.nlist) replace the cell
// walk for slots whose list fits; those slots leave no neighbour bits (the
// force pass re-tests their lists).
// FUS: on iterations that do not sort, read the state from F.A (FusedSrc).
template <int DIM, int TPP = 1, int BS = kPassThreads, bool LEAN = false, bool OPT = false,
          bool STG = false, class LT = int, bool LST = false, bool FUS = false>
__device__ __forceinline__ void density_body(const StateB& B, const unsigned* __restrict__ keys,
                                             const int* __restrict__ start, const DevGrid& g,
                                             const DevParams& P, const int s, const bool valid,
                                             LT (*s_near)[BS], LT (*s_far)[BS],
                                             const StageView& SV = StageView{},
                                             const FusedSrc& F = FusedSrc{}) {
    static_assert(!STG || (TPP == 1 && LEAN && !OPT), "staged: one lane per particle, lean physics");
    static_assert(!LST || (TPP == 1 && !STG), "lists: one lane per particle, unstaged");
    static_assert(!FUS || (LST && LEAN && !OPT), "fused predictor: lists, lean physics");
    const int tid = threadIdx.x;
    const int sub = (TPP == 1) ? 0 : (tid & (TPP - 1));
    const bool need_div = !LEAN && P.heat_art != 0;
    const bool from_a = FUS && sort_skipped(F.rs);
    const float4* __restrict__ xsrc = from_a ? F.A.xh : B.xh;
    const float4* __restrict__ vsrc = from_a ? F.A.vm : B.vm;  // 3D masses (.w)
    float4 xi = make_float4(0.f, 0.f, 0.f, 1.f), vi = xi, rp = xi;
    float p = 0.f;
    int it_i = 0;
    bool fluid = false;
    if (valid && from_a) {
        xi = F.A.xh[s];
        it_i = F.A.itype[s];
        fluid = it_i > 0;
        vi = F.A.vm[s];
        p = F.A.p[s];
        rp = make_float4(F.A.rho[s], 0.f, 0.f, 0.f);
        if (fluid && F.hdt != 0.f) {  // predictor (k_reorder_dim's, same operations)
            const float4 ap = F.A.ap[s];
            vi.x = fmaf(F.hdt, ap.x, vi.x);
            vi.y = fmaf(F.hdt, ap.y, vi.y);
            if (DIM == 3) vi.z = fmaf(F.hdt, ap.z, vi.z);
        }
        if (DIM == 3) B.vm[s] = vi;  // the force pass reads neighbours' predicted v here
    } else if (valid) {
        xi = B.xh[s];
        rp = B.rp[s];
        p = B.p[s];
        it_i = B.itype[s];
        fluid = it_i > 0;
        vi = B.vm[s];
    }
    const bool work = valid && g.ok && (fluid || need_div);
    const sph::ff kw = {P.kw_hi, P.kw_lo};
    const sph::ff ih_i = sph::ff_recip(xi.w);
    const sph::ff al_i = sph::ff_mul(kw, ff_pow_dim<DIM>(ih_i));
    const float mi = mass_of<DIM>(xi, vi);
    const float kgih_i = __fmul_rn(P.kg, pow_grad<DIM>(ih_i.hi));
    // Normalised summation (nor_density, density.f:65-158): the denominator
    // m_i W(0)/rho_i + sum_j m_j/rho_j W_ij on the start densities, float-float.
    const bool nor = OPT && P.density_form == 2 && fluid;
    // Density sums of the even (.x) and odd (.y) entries, float-float: of m_j W_ij,
    // or with every h alike (UNI) of m_j W_ij h^dim / K, the factor applied once to
    // the sum. The self term (density.f:39-42) opens the first lane's even one.
    f2 Sh = bc2(0.f), Sl = bc2(0.f);
    f2 Fh = bc2(0.f), Fl = bc2(0.f);  // the far pairs' with their factors (kFarOwn)
    // 2D lists: a far pair's weight is rounded as the written formula has it, dr^2 its
    // unfused sum and K m / h^dim taken to each. Lists serve the large systems, where
    // the last bit of the pressure sets how many positions round the other way: with
    // the unscaled form 26% of the pressures of a 2.03 M dam break had another last bit,
    // now 4%, for 7 us of 126 (the cell walk's 18.1 us at 42 k became 20.9: not there).
    constexpr bool kFarOwn = LST && DIM == 2;
    f2 Wh = bc2(0.f), Wl = bc2(0.f);  // the normalised summation's denominator, alike
    float divs = 0.f;
    bool done = !work;
    // Differences x_i - x_j of near pairs are exact in FP32 unless the coordinates
    // differ by more than a factor of two (near a coordinate's zero) or wrap: a
    // particle farther than that from both skips the residuals. rmax: farther than
    // any entry of a list (h_i + h_j + skin when built, each moved skin/2 since).
    bool plain = true;
    {
        const float rmax = 1.01f * (xi.w + g.hmax + 2.0f * g.skin);
        const float c[3] = {xi.x, xi.y, xi.z};
#pragma unroll
        for (int k = 0; k < DIM; ++k) {
            plain = plain && fabsf(c[k]) >= 2.0f * rmax;
            if (g.periodic[k]) plain = plain && c[k] - g.o[k] > rmax && g.o[k] + g.L[k] - c[k] > rmax;
        }
    }
    // (listed particles, LST, need no bits: the force pass walks their list)
    const int lpk = (LST && work) ? B.ncount[s] : -1;
    const int lc = list_near(lpk);  // near list entries (-1: walk the cells)
    const int lf = list_far(lpk);   // far list entries (2D)
    if (LST) prefetch_list(B.nlist, B.lstride, s, lc + lf);
    // The place of an absent entry: the particle itself, with no mass.
    int kself = valid ? s : 0;
    if (STG) kself = work ? s + SV.shift[DIM == 2 ? g.reach : g.reach * (2 * g.reach + 2)] : 0;
    // The divisors of normalised density; 1 beyond the support, where a particle
    // without density has no part.
    auto rho_in = [&](const int ka, const int kb, const f2 t) {
        return make_float2(t.x > 0.f ? __ldg(B.q + ka) : 1.f, t.y > 0.f ? __ldg(B.q + kb) : 1.f);
    };
    // Two entries. NEAR: float-float weights on the exact pair difference, else
    // (2D) FP32 weights, the pair's r and q rounded once. The kernel is zero beyond
    // its support, so entries in a list's skin margin need no pair test.
    // ka, kb: the entries; ina, inb: whether they count; x, v: their {x, h} and v (3D:
    // the mass; artificial heat).
    // Issue-bound (72-89% of cycles): the packed forms take half the slots, and
    // K/h^dim once per sum, Fast2Sum where the larger term is known and no residuals
    // for `plain` particles save about 30 of 85 operations a near pair. Measured: 3D
    // lists (8.78 M channel) 5.24 -> 3.45 ms, 2D lists (2.03 M dam break) 0.179 ->
    // 0.154 ms, 2D cells (42 k) 21.6 -> 19.8 us (with blocks of entries 3.00 and 0.126
    // ms, with the walk by rows 13.2 us).
    auto pair2 = [&](auto uni, auto ph, auto near, bool ina, bool inb, const int ka, const int kb,
                     const float4& xa, const float4& xb, const float4& va, const float4& vb) {
        constexpr bool UNI = decltype(uni)::value, NEAR = decltype(near)::value;
        constexpr int PH = decltype(ph)::value;
        f2 mj = DIM == 2 ? make_float2(xa.z, xb.z) : make_float2(va.w, vb.w);
        if ((PH & 4) && P.wall_model == 1) {  // push only
            ina = ina && __ldg(B.itype + ka) == it_i;
            inb = inb && __ldg(B.itype + kb) == it_i;
        }
        if (!ina) mj.x = 0.f;
        if (!inb) mj.y = 0.f;
        f2 d0 = make_float2(xi.x - xa.x, xi.x - xb.x), d1 = make_float2(xi.y - xa.y, xi.y - xb.y);
        f2 d2 = DIM == 3 ? make_float2(xi.z - xa.z, xi.z - xb.z) : bc2(0.f);
        f2 ddl = bc2(0.f);  // 2 dh . dl of the residuals dl
        if (!plain) {
            float ha[3], la[3], hb[3], lb[3];
            exact_delta<DIM>(xi, xa, g, ha, la);
            exact_delta<DIM>(xi, xb, g, hb, lb);
            d0 = make_float2(ha[0], hb[0]);
            d1 = make_float2(ha[1], hb[1]);
            ddl = fma2(d1, make_float2(la[1], lb[1]), mul2(d0, make_float2(la[0], lb[0])));
            if (DIM == 3) {
                d2 = make_float2(ha[2], hb[2]);
                ddl = fma2(d2, make_float2(la[2], lb[2]), ddl);
            }
            ddl = add2(ddl, ddl);
        }
        ff2 ih = {bc2(ih_i.hi), bc2(ih_i.lo)}, cm = {mj, bc2(0.f)};  // 1/h; the term's factor
        if (!UNI) {
            ih = recip_ff2(mul2(bc2(0.5f), make_float2(xi.w + xa.w, xi.w + xb.w)));
            ff2 al = sqr_ff2(ih);
            if (DIM == 3) al = mul_ff2(al, ih);
            cm = mul_ff2_f(mul_ff2(ff2{bc2(kw.hi), bc2(kw.lo)}, al), mj);
        }
        f2 t;  // 1 - q/2, 0 beyond the support
        if (NEAR) {
            ff2 dr2 = two_prod2(d0, d0);
            {
                const ff2 p1 = two_prod2(d1, d1), w = two_sum2(dr2.hi, p1.hi);
                dr2.lo = add2(add2(add2(dr2.lo, p1.lo), w.lo), ddl);
                dr2.hi = w.hi;
            }
            if (DIM == 3) {
                const ff2 p2 = two_prod2(d2, d2), w = two_sum2(dr2.hi, p2.hi);
                dr2.lo = add2(add2(dr2.lo, p2.lo), w.lo);
                dr2.hi = w.hi;
            }
            const ff2 q = mul_ff2(sqrt_ff2(dr2), ih);
            ff2 T = fast_affine2(q, -0.5f, 1.0f);
            T.hi = max2(T.hi, 0.0f);
            t = T.hi;
            if (fluid) {
                const ff2 f = mul_ff2(sqr_ff2(sqr_ff2(T)), fast_affine2(T, -4.0f, 5.0f));  // t^4 (1 + 2q)
                const ff2 m = UNI ? mul_ff2_f(f, mj) : mul_ff2(f, cm);
                acc_ff2(Sh, Sl, m);
                if ((PH & 4) && nor)
                    acc_ff2(Wh, Wl, mul_ff2(m, recip_ff2(rho_in(ka, kb, t))));
            }
        } else {
            // With uniform h and m every pair would share the rounding of K m / h^dim
            // and of 1/h: a bias that adds up over the far pairs. So the prefactor
            // and 1/h stay float-float, r is the Newton-corrected square root, and
            // q = r (ih.hi + ih.lo) is rounded once.
            const f2 dr2 = kFarOwn ? add2(prod2(d0, d0), prod2(d1, d1)) : fma2(d1, d1, prod2(d0, d0));
            const f2 rs = rsqrt2(dr2);
            f2 r = mul2(dr2, rs);
            r = fma2(fma2(neg2(r), r, dr2), mul2(rs, bc2(0.5f)), r);
            const f2 q = fma2(r, ih.hi, mul2(r, ih.lo));
            t = max2(fma2(q, bc2(-0.5f), bc2(1.0f)), 0.0f);
            if (fluid) {
                const f2 t2 = mul2(t, t);
                const f2 f = mul2(mul2(t2, t2), fma2(q, bc2(2.0f), bc2(1.0f)));
                const f2 m = UNI ? mul2(mj, f) : fma2(cm.hi, f, mul2(cm.lo, f));
                if ((PH & 4) && nor)
                    acc_ff2(Wh, Wl, div2(m, rho_in(ka, kb, t)));
                if (UNI && kFarOwn) {
                    const ff2 c = mul_ff2_f(ff2{bc2(al_i.hi), bc2(al_i.lo)}, mj);
                    acc_ff2(Fh, Fl, fma2(c.hi, f, mul2(c.lo, f)));
                } else {
                    acc_ff2(Sh, Sl, m);
                }
            }
        }
        if ((PH & 1) && need_div) {  // art_heat.f:46-67: grad W = kg (q - 2)^3 d = -8 kg t^3 d
            f2 kg = bc2(kgih_i);
            if (!UNI) {
                const f2 i2 = mul2(ih.hi, ih.hi);
                kg = mul2(bc2(P.kg), mul2(i2, i2));
                if (DIM == 3) kg = mul2(kg, ih.hi);
            }
            const f2 gm = mul2(mul2(mul2(t, t), mul2(t, bc2(-8.0f))), mul2(kg, mj));
            f2 vd = fma2(make_float2(va.y - vi.y, vb.y - vi.y), d1,
                         mul2(make_float2(va.x - vi.x, vb.x - vi.x), d0));
            if (DIM == 3) vd = fma2(make_float2(va.z - vi.z, vb.z - vi.z), d2, vd);
            if (PH & 4) vd = make_float2(mj.x != 0.f ? vd.x : 0.f, mj.y != 0.f ? vd.y : 0.f);
            divs = dot2(gm, vd, divs);
        }
    };
    constexpr int W = mask_words<DIM>() / TPP;  // mask words of this lane
    const size_t mlane = (size_t)s * TPP + sub;
    bool mask_on = false;
    int ord = 0;  // candidate ordinal (cursor order, self included)
    int wb = 0;   // the accumulator holds the bits of ordinals 32 wb .. 32 wb + 63
    unsigned long long cur = 0ull;
    auto walk = [&](auto uni, auto ph) {
    constexpr bool UNI = decltype(uni)::value;
    constexpr bool VJ = DIM == 3 || (decltype(ph)::value & 1) != 0;  // the neighbour's v is read
    const std::true_type kNear{};
    const std::false_type kFar{};
    {
        const sph::ff self = UNI ? sph::ff{mi, 0.f} : sph::ff_mul_f(al_i, mi);
        if (sub == 0) {
            Sh.x = self.hi;
            Sl.x = self.lo;
            if (nor) {
                const sph::ff w = sph::ff_mul(self, sph::ff_recip(B.q[s]));
                Wh.x = w.hi;
                Wl.x = w.lo;
            }
        }
    }
    // A listed particle evaluates each list entry as it is read, the near ones in
    // float-float, the far ones (2D) like the cell walk's far pairs: no candidate
    // lists in shared memory, no second load. The cell walk below serves the others.
    if (LST) {
        // Entries [first, first + count) of this slot's list, the next block loaded
        // ahead. A block with both near and far entries is read twice, each kind
        // evaluated in its own arithmetic.
        auto entries = [&](auto near, const int first, const int count) {
            const int b0 = first >> 2, last = count > 0 ? blocks_of(first + count) : b0;
            const int cm = __reduce_max_sync(0xffffffffu, last - b0);
            int4 kn = list_block(B.nlist, B.lstride, s, b0, last, kself);
            int t = 4 * b0 - first;
            for (int b = 0; b < cm; ++b, t += 4) {
                const int4 q = kn;
                if (b + 1 < cm) kn = list_block(B.nlist, B.lstride, s, b0 + b + 1, last, kself);
                const int kb[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
                for (int u = 0; u < 4; u += 2) {
                    const float4 xa = __ldg(xsrc + kb[u]), xb = __ldg(xsrc + kb[u + 1]);
                    const float4 va = VJ ? __ldg(vsrc + kb[u]) : xa, vb = VJ ? __ldg(vsrc + kb[u + 1]) : xb;
                    pair2(uni, ph, near, (unsigned)(t + u) < (unsigned)count,
                          (unsigned)(t + u + 1) < (unsigned)count, kb[u], kb[u + 1], xa, xb, va, vb);
                }
            }
        };
        entries(kNear, 0, max(lc, 0));
        if (DIM == 2) entries(kFar, max(lc, 0), lf);
        if (lc >= 0) done = true;
    }
    if (!__any_sync(0xffffffffu, !done)) return;
    CellCoord cc = {{0, 0, 0}};
    if (!done) {
        cc = decode_key<DIM>(keys[s], g);
        mask_on = fluid;
    }
    auto evaluate = [&](const int nn, const int nf) {
        const int mn = __reduce_max_sync(0xffffffffu, nn);
        const int mf = __reduce_max_sync(0xffffffffu, nf);
        auto listed = [&](auto near, LT (*lst)[BS], const int cnt, const int cm) {
            for (int t = 0; t < cm; t += 2) {
                int kb[2];
                float4 xb[2], vb[2];
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const int k = kb[u] = t + u < cnt ? (int)lst[t + u][tid] : kself;
                    xb[u] = STG ? SV.x[k] : __ldg(xsrc + k);
                    vb[u] = !VJ ? xb[u] : STG ? SV.v[k] : __ldg(vsrc + k);
                }
                pair2(uni, ph, near, t < cnt, t + 1 < cnt, kb[0], kb[1], xb[0], xb[1], vb[0], vb[1]);
            }
        };
        listed(kNear, s_near, nn, mn);
        if (DIM == 2) listed(kFar, s_far, nf, mf);
    };
    if constexpr (TPP == 1) {
        // The rows of cells as plain loops of converged lanes; a lane whose lists are full
        // leaves off at (row r_at, slot k_at) and goes on there after the evaluation. With
        // the cursor's step in the loop of the batches, of which some lane took one nearly
        // each time, a batch cost a warp 260 instructions. Measured: 1,920 particles 18.9 ->
        // 11.6 us, 42 k 18.0 -> 13.2, 2.03 M 307 -> 238, 2.76 M in 64 instances 518 -> 394.
        const int f = g.reach, c0 = max(cc.c[0] - f, 0), c1 = min(cc.c[0] + f, g.n[0] - 1) + 1;
        const float near_k = 0.25f * near_q<DIM>() * near_q<DIM>();
        const float hs_u = __fadd_rn(xi.w, xi.w), lim_u = __fmul_rn(hs_u, hs_u), near_u = near_k * hs_u * hs_u;
        int r_at = 0, k_at = 0;
        while (__any_sync(0xffffffffu, !done)) {
            int nn = 0, nf = 0;
            bool open = !done;
            auto range = [&](const int b, const int e, const int r, const int shift) {
                for (int k0 = max(b, k_at); k0 < e; k0 += kTestBatch) {
                    if (nn > cap_density<LST>() - kTestBatch || nf > cap_density<LST>() - kTestBatch) {
                        open = false;
                        r_at = r;
                        k_at = k0;
                        return;
                    }
                    float4 xb[kTestBatch];
#pragma unroll
                    for (int u = 0; u < kTestBatch; ++u)
                        xb[u] = STG ? SV.x[min(k0 + u, e - 1) + shift] : __ldg(xsrc + k0 + u);  // (padded)
                    unsigned pb = 0u;  // pass bits of this batch
#pragma unroll
                    for (int u = 0; u < kTestBatch; u += 2) {
                        f2 d0 = make_float2(__fsub_rn(xi.x, xb[u].x), __fsub_rn(xi.x, xb[u + 1].x));
                        f2 d1 = make_float2(__fsub_rn(xi.y, xb[u].y), __fsub_rn(xi.y, xb[u + 1].y));
                        if (g.periodic[0]) d0 = make_float2(sph::min_image(d0.x, g.L[0], g.half[0]), sph::min_image(d0.y, g.L[0], g.half[0]));
                        if (g.periodic[1]) d1 = make_float2(sph::min_image(d1.x, g.L[1], g.half[1]), sph::min_image(d1.y, g.L[1], g.half[1]));
                        f2 r2 = add2(prod2(d0, d0), prod2(d1, d1));  // dist2_exact's roundings (prod2 rounds an exact tie up)
                        if (DIM == 3) {
                            f2 d2 = make_float2(__fsub_rn(xi.z, xb[u].z), __fsub_rn(xi.z, xb[u + 1].z));
                            if (g.periodic[2]) d2 = make_float2(sph::min_image(d2.x, g.L[2], g.half[2]), sph::min_image(d2.y, g.L[2], g.half[2]));
                            r2 = add2(r2, prod2(d2, d2));
                        }
#pragma unroll
                        for (int q = 0; q < 2; ++q) {
                            const int k = k0 + u + q;
                            const float rr = q ? r2.y : r2.x;
                            const float hs = UNI ? hs_u : __fadd_rn(xi.w, xb[u + q].w);
                            const bool in = rr < (UNI ? lim_u : __fmul_rn(hs, hs)) && k < e && k != s;
                            const bool near = DIM == 3 || rr < (UNI ? near_u : near_k * hs * hs);
                            const LT at = (LT)(k + shift);
                            if (in) pb |= 1u << (u + q);
                            if (in && near) s_near[nn++][tid] = at;
                            if (DIM == 2 && in && !near) s_far[nf++][tid] = at;
                        }
                    }
                    if (ord - 32 * wb >= 32) {  // word wb is complete
                        if (mask_on && wb < W) B.nmask[mask_word_index<W>(wb, B.mstride, mlane)] = (unsigned)cur;
                        cur >>= 32;
                        ++wb;
                    }
                    cur |= (unsigned long long)pb << (ord - 32 * wb);
                    ord += min(kTestBatch, e - k0);
                }
                r_at = r + 1;
                k_at = 0;
            };
            int r = 0;  // rows, and on a periodic x axis their wrapped parts
            for (int dz = DIM == 3 ? -f : 0; dz <= (DIM == 3 ? f : 0); ++dz)
                for (int dy = -f; dy <= f; ++dy, r += 2) {
                    if (!open || r + 1 < r_at) continue;
                    const int* const row = cell_row<DIM>(g, start, cc, dy, dz);
                    if (!row) continue;
                    const int shift = STG ? SV.shift[DIM == 2 ? dy + f : (dz + f) * (2 * f + 1) + (dy + f)] : 0;
                    if (r >= r_at) range(__ldg(row + c0), __ldg(row + c1), r, shift);
                    if (g.periodic[0] && open) {
                        if (cc.c[0] < f)
                            range(__ldg(row + cc.c[0] - f + g.n[0]), __ldg(row + g.n[0]), r + 1, shift);
                        else if (cc.c[0] + f >= g.n[0])
                            range(__ldg(row), __ldg(row + cc.c[0] + f - g.n[0] + 1), r + 1, shift);
                    }
                }
            if (open) done = true;
            evaluate(nn, nf);
        }
    } else {
        Cursor cu = cursor_begin<DIM>(g);
        static_assert(!STG, "staged passes: one lane per particle");
        while (__any_sync(0xffffffffu, !done)) {
            int nn = 0, nf = 0;
            // Test phase: fill the near / far lists, kTestBatch candidate loads in flight.
            while (!done) {
                int kb[kTestBatch];
                int cnt;
                float4 xb[kTestBatch];
                if (cu.k >= cu.ke) {
                    if (!cursor_next<DIM>(g, start, cc, cu)) {
                        done = true;
                        break;
                    }
                    cu.k += sub;
                    continue;
                }
                if (nn > cap_density<LST>() - kTestBatch || nf > cap_density<LST>() - kTestBatch) break;
                const int k0 = cu.k;
                cnt = min(kTestBatch, lane_len<TPP>(cu));
#pragma unroll
                for (int u = 0; u < kTestBatch; ++u) {
                    const int ku = min(k0 + u * TPP, cu.ke - 1);
                    kb[u] = k0 + u * TPP;
                    xb[u] = __ldg(xsrc + ku);
                }
                cu.k += cnt * TPP;
                unsigned pb = 0u;  // pass bits of this batch
#pragma unroll
                for (int u = 0; u < kTestBatch; ++u) {
                    float d[3], dr2;
                    const int k = kb[u];
                    if (u >= cnt || k == s || !pair_delta<DIM>(xi, xb[u], g, d, dr2)) continue;
                    pb |= 1u << u;
                    const float hs = xi.w + xb[u].w;  // near: q < near_q() with h = hs/2
                    if (DIM == 3 || dr2 < (0.25f * near_q<DIM>() * near_q<DIM>()) * hs * hs)
                        s_near[nn++][tid] = (LT)k;
                    else
                        s_far[nf++][tid] = (LT)k;
                }
                if (ord - 32 * wb >= 32) {  // word wb is complete
                    if (mask_on && wb < W) B.nmask[mask_word_index<W>(wb, B.mstride, mlane)] = (unsigned)cur;
                    cur >>= 32;
                    ++wb;
                }
                cur |= (unsigned long long)pb << (ord - 32 * wb);
                ord += cnt;
            }
            evaluate(nn, nf);
        }
    }
    };
    using std::integral_constant;
    const bool uni = TPP == 1 && g.huni && (LEAN || OPT || P.wall_model != 1);
    if constexpr (LEAN) {
        if (uni) walk(std::true_type{}, integral_constant<int, 0>{});
        else walk(std::false_type{}, integral_constant<int, 0>{});
    } else if constexpr (TPP == 1 && !OPT) {
        if (uni && !need_div) walk(std::true_type{}, integral_constant<int, 0>{});
        else if (uni) walk(std::true_type{}, integral_constant<int, 1>{});
        else walk(std::false_type{}, integral_constant<int, 7>{});
    } else {
        if (uni) walk(std::true_type{}, integral_constant<int, 7>{});
        else walk(std::false_type{}, integral_constant<int, 7>{});
    }
    sph::ff S = {Sh.x, Sl.x}, Wn = {Wh.x, Wl.x};
    sph::ff_acc(S, sph::ff{Sh.y, Sl.y});
    if (OPT) sph::ff_acc(Wn, sph::ff{Wh.y, Wl.y});
    if (uni) {
        S = sph::ff_mul(al_i, S);
        if (kFarOwn) {
            sph::ff_acc(S, sph::ff{Fh.x, Fl.x});
            sph::ff_acc(S, sph::ff{Fh.y, Fl.y});
        }
        if (OPT) Wn = sph::ff_mul(al_i, Wn);
    }
    if (TPP > 1) {  // the particle's lanes reach this point together
        const unsigned gm = group_mask<TPP>();
#pragma unroll
        for (int o = 1; o < TPP; o <<= 1) {
            const sph::ff t = {__shfl_xor_sync(gm, S.hi, o), __shfl_xor_sync(gm, S.lo, o)};
            sph::ff_acc(S, t);
            if (OPT) {
                const sph::ff tw = {__shfl_xor_sync(gm, Wn.hi, o), __shfl_xor_sync(gm, Wn.lo, o)};
                sph::ff_acc(Wn, tw);
            }
        }
        divs = group_sum<TPP>(divs);
    }
    if (!valid) return;
    if (mask_on) {
        if (ord > 32 * W) {
            B.nmask[mask_word_index<W>(0, B.mstride, mlane)] = ~0u;
            if (W > 1) B.nmask[mask_word_index<W>(1, B.mstride, mlane)] = ~0u;
        } else {
            for (; wb < W; ++wb) {
                B.nmask[mask_word_index<W>(wb, B.mstride, mlane)] = (unsigned)cur;
                cur >>= 32;
            }
        }
    }
    if (sub != 0) return;
    if (!work) {  // wall without div v (or no grid): fixed rho and p
        rp.y = (P.pa_sph == 1) ? __fdiv_rn(p, __fmul_rn(rp.x, rp.x)) : p;
        B.rp[s] = rp;
        if (DIM == 2) B.vr[s] = make_float4(vi.x, vi.y, rp.x, rp.y);
        return;
    }
    float rho = rp.x;
    if (fluid) {
        float drho;
        if (OPT && P.density_form == 1) {  // continuity: the predicted density
            drho = __fadd_rn(__fsub_rn(rp.x, P.rho0), B.rlo[s]);
        } else if (nor) {  // S / Wn to float-float accuracy
            const float qh = __fdiv_rn(S.hi, Wn.hi);
            const float res = fmaf(-qh, Wn.hi, S.hi) + S.lo - qh * Wn.lo;
            drho = __fadd_rn(__fsub_rn(qh, P.rho0), __fdiv_rn(res, Wn.hi));
        } else {
            drho = __fadd_rn(__fsub_rn(S.hi, P.rho0), S.lo);
        }
        p = sph::tait_poly(__fmul_rn(drho, P.inv_rho0), P.B);
        if (p < P.pmin) {  // eos.f90:277-280
            p = 0.f;
            drho = 0.f;
        }
        rho = __fadd_rn(P.rho0, drho);
        B.p[s] = p;
    }
    rp.x = rho;
    rp.y = (P.pa_sph == 1) ? __fdiv_rn(p, __fmul_rn(rho, rho)) : p;
    if (need_div) {
        // a mirror ghost's psi waits for its owner's density (k_ghost_sync)
        if (P.wall_model == 3 && !fluid) B.tds[s] = divs;
        const float divv = __fdiv_rn(divs, rho);
        rp.w = fmaf(P.ah_g2 * xi.w * xi.w, fabsf(divv) - divv, __fmul_rn(P.ah_g1 * xi.w, P.c0));
    }
    if (LST && fluid && !(fabsf(rp.y) < 1.0e34f && rho > 1.0e-18f)) {  // the force pass walks its cells
        B.ncount[s] = -1;
        B.nmask[mask_word_index<W>(0, B.mstride, mlane)] = ~0u;
        if (W > 1) B.nmask[mask_word_index<W>(1, B.mstride, mlane)] = ~0u;
    }
    B.rp[s] = rp;
    if (DIM == 2) B.vr[s] = make_float4(vi.x, vi.y, rp.x, rp.y);
}

// ---------------------------------------------------------------------------
// Pass 1b: shear tensor (physical viscosity), every particle.
// ---------------------------------------------------------------------------
// The sums M_ab = sum_j m_j/rho_j G (v_j - v_i)_a (x_i - x_j)_b give the tensor
// T_ab = M_ab + M_ba - (2/3) delta_ab tr M once per particle (internal_force.f:
// 75-171 forms it per pair). Listed particles (LST) walk their lists; the others
// collect the cells' candidates that pass the pair test in s_list. A cell walk of
// its own, with divisions and a square root per pair in the branch of the test,
// took 23.8 us at 26,880 particles; the lists' walk 11.
template <int DIM, bool LST = false>
__device__ __forceinline__ void shear_body(const StateB& B, const unsigned* __restrict__ keys,
                                           const int* __restrict__ start, const DevGrid& g,
                                           const DevParams& P, const int s, const bool valid,
                                           int (*s_list)[kPassThreads]) {
    const int tid = threadIdx.x;
    const bool work = valid && g.ok;
    const int kself = valid ? s : 0;
    float4 xi = make_float4(0.f, 0.f, 0.f, 1.f), vi = xi;
    float rhoi = 1.f;
    int it_i = 0;
    if (work) {
        xi = B.xh[s];
        vi = B.vm[s];
        rhoi = B.rp[s].x;
        it_i = B.itype[s];
    }
    float m[DIM][DIM];
#pragma unroll
    for (int a = 0; a < DIM; ++a)
#pragma unroll
        for (int b = 0; b < DIM; ++b) m[a][b] = 0.f;
    // Two entries; an absent one is the particle itself (d = 0, dv = 0). Beyond the
    // support G = 0.
    auto pair2 = [&](const int ka, const int kb) {
        const float4 xa = __ldg(B.xh + ka), xb = __ldg(B.xh + kb);
        const float4 va = __ldg(B.vm + ka), vb = __ldg(B.vm + kb);
        f2 mj = DIM == 2 ? make_float2(xa.z, xb.z) : make_float2(va.w, vb.w);
        bool pa = false, pb = false;  // push only: nothing else of the other is read
        if (P.wall_model == 1) {
            pa = __ldg(B.itype + ka) != it_i;
            pb = __ldg(B.itype + kb) != it_i;
            if (pa) mj.x = 0.f;
            if (pb) mj.y = 0.f;
        }
        f2 d[3], dv[3];
        d[0] = make_float2(xi.x - xa.x, xi.x - xb.x);
        d[1] = make_float2(xi.y - xa.y, xi.y - xb.y);
        dv[0] = make_float2(va.x - vi.x, vb.x - vi.x);
        dv[1] = make_float2(va.y - vi.y, vb.y - vi.y);
        if (g.periodic[0]) d[0] = min_image2(d[0], xi.x, xa.x, xb.x, g, 0);
        if (g.periodic[1]) d[1] = min_image2(d[1], xi.y, xa.y, xb.y, g, 1);
        f2 dr2 = fma2(d[1], d[1], fma2(d[0], d[0], bc2(kTinyDr2)));
        if (DIM == 3) {
            d[2] = make_float2(xi.z - xa.z, xi.z - xb.z);
            dv[2] = make_float2(va.z - vi.z, vb.z - vi.z);
            if (g.periodic[2]) d[2] = min_image2(d[2], xi.z, xa.z, xb.z, g, 2);
            dr2 = fma2(d[2], d[2], dr2);
        }
#pragma unroll
        for (int a = 0; a < DIM; ++a) dv[a] = make_float2(pa ? 0.f : dv[a].x, pb ? 0.f : dv[a].y);
        const f2 hs = make_float2(xi.w + xa.w, xi.w + xb.w);
        const f2 ih = mul2(bc2(2.0f), rcp2_rn(hs, rcp2(hs)));
        const f2 ih2 = mul2(ih, ih);
        f2 kg = mul2(bc2(P.kg), mul2(ih2, ih2));
        if (DIM == 3) kg = mul2(kg, ih);
        const f2 t = min2(fma2(sqrt2(dr2, rsqrt2(dr2)), ih, bc2(-2.0f)), 0.0f);
        const f2 mr = within2(t, div2(mj, make_float2(__ldg(&B.rp[ka].x), __ldg(&B.rp[kb].x))));
        const f2 c = mul2(mul2(mul2(mul2(t, t), t), kg), mr);
#pragma unroll
        for (int a = 0; a < DIM; ++a) {
            const f2 u = mul2(c, dv[a]);
#pragma unroll
            for (int b = 0; b < DIM; ++b) m[a][b] = dot2(u, d[b], m[a][b]);
        }
    };
    bool done = !work;
    if (LST) {
        const int lpk = work ? __ldg(B.ncount + s) : -1;
        const int lc = lpk >= 0 ? list_near(lpk) + list_far(lpk) : -1, nb = blocks_of(lc);
        const int bm = __reduce_max_sync(0xffffffffu, nb);
        int4 kn = list_block(B.nlist, B.lstride, s, 0, nb, kself);
        for (int b = 0; b < bm; ++b) {
            const int4 q = kn;
            if (b + 1 < bm) kn = list_block(B.nlist, B.lstride, s, b + 1, nb, kself);
            pair2(q.x, q.y);
            pair2(q.z, q.w);
        }
        if (lc >= 0) done = true;
    }
    if (__any_sync(0xffffffffu, !done)) {
        CellCoord cc = {{0, 0, 0}};
        if (!done) cc = decode_key<DIM>(keys[s], g);
        const int f = g.reach, c0 = max(cc.c[0] - f, 0), c1 = min(cc.c[0] + f, g.n[0] - 1) + 1;
        int r_at = 0, k_at = 0;  // rows as in the density pass
        while (__any_sync(0xffffffffu, !done)) {
            int nl = 0;
            bool open = !done;
            auto range = [&](const int b, const int e, const int r) {
                for (int k0 = max(b, k_at); k0 < e; k0 += kTestBatch) {
                    if (nl > cap_force<LST>() - kTestBatch) {
                        open = false;
                        r_at = r;
                        k_at = k0;
                        return;
                    }
                    // in flight together: one at a time, 1,920 particles took 20.1 us, and
                    // with the cursor's step per batch 16.5, now 14.0
                    float4 xb[kTestBatch];
#pragma unroll
                    for (int u = 0; u < kTestBatch; ++u) xb[u] = __ldg(B.xh + k0 + u);  // (padded)
#pragma unroll
                    for (int u = 0; u < kTestBatch; ++u) {
                        const int k = k0 + u;
                        float d[3], dr2;
                        if (k < e && k != s && pair_delta<DIM>(xi, xb[u], g, d, dr2)) s_list[nl++][tid] = k;
                    }
                }
                r_at = r + 1;
                k_at = 0;
            };
            int r = 0;
            for (int dz = DIM == 3 ? -f : 0; dz <= (DIM == 3 ? f : 0); ++dz)
                for (int dy = -f; dy <= f; ++dy, r += 2) {
                    if (!open || r + 1 < r_at) continue;
                    const int* const row = cell_row<DIM>(g, start, cc, dy, dz);
                    if (!row) continue;
                    if (r >= r_at) range(__ldg(row + c0), __ldg(row + c1), r);
                    if (g.periodic[0] && open) {
                        if (cc.c[0] < f)
                            range(__ldg(row + cc.c[0] - f + g.n[0]), __ldg(row + g.n[0]), r + 1);
                        else if (cc.c[0] + f >= g.n[0])
                            range(__ldg(row), __ldg(row + cc.c[0] + f - g.n[0] + 1), r + 1);
                    }
                }
            if (open) done = true;
            const int ml = __reduce_max_sync(0xffffffffu, nl);
            for (int t = 0; t < ml; t += 2)
                pair2(t < nl ? s_list[t][tid] : kself, t + 1 < nl ? s_list[t + 1][tid] : kself);
        }
    }
    if (!work) return;
    float tr = m[0][0] + m[1][1];
    if (DIM == 3) tr += m[DIM - 1][DIM - 1];
    const float c3 = (-2.f / 3.f) * tr;
    const float txx = fmaf(2.f, m[0][0], c3), tyy = fmaf(2.f, m[1][1], c3);
    const float tzz = DIM == 3 ? fmaf(2.f, m[DIM - 1][DIM - 1], c3) : 0.f;
    const float txy = m[0][1] + m[1][0];
    const float txz = DIM == 3 ? m[0][DIM - 1] + m[DIM - 1][0] : 0.f;
    const float tyz = DIM == 3 ? m[1][DIM - 1] + m[DIM - 1][1] : 0.f;
    float q = fmaf(2.f * txy, txy, fmaf(tyy, tyy, __fmul_rn(txx, txx)));
    if (DIM == 3) q = fmaf(2.f * txz, txz, fmaf(2.f * tyz, tyz, fmaf(tzz, tzz, q)));
    B.tds[s] = 0.5f * P.eta / rhoi * q;
    if (rhoi == 0.f) {  // no mass near it: only others' list margins read its tau
        B.tau[s] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (DIM == 3) B.tau2[s] = make_float4(0.f, 0.f, 0.f, 0.f);
        return;
    }
    const float sc = (P.pa_sph == 1) ? P.eta / (rhoi * rhoi) : P.eta;
    B.tau[s] = make_float4(sc * txx, sc * tyy, sc * txy, sc * tzz);
    if (DIM == 3) B.tau2[s] = make_float4(sc * txz, sc * tyz, 0.f, 0.f);
}

// ---------------------------------------------------------------------------
// Pass 2: forces, heat, leapfrog corrector. Reads B, writes the next state A.
// ---------------------------------------------------------------------------
// STG: neighbours from the CTA's staged copy SV (see density_body).
// FUS: on iterations that do not sort, the state comes from F.A (FusedSrc);
// A is then the other buffer, which receives the next state.
template <int DIM, int TPP = 1, int BS = kPassThreads, bool LEAN = false, bool OPT = false,
          bool STG = false, class LT = int, bool LST = false, bool FUS = false>
__device__ __forceinline__ void force_body(const StateB& B, const StateA& A,
                                           const unsigned* __restrict__ keys,
                                           const int* __restrict__ start, const DevGrid& g,
                                           const DevParams& P, const StepArgs& S,
                                           unsigned* __restrict__ flags, const int s,
                                           const bool valid, LT (*s_list)[BS],
                                           const StageView& SV = StageView{},
                                           const FusedSrc& F = FusedSrc{}) {
    static_assert(!STG || (TPP == 1 && LEAN && !OPT), "staged: one lane per particle, lean physics");
    static_assert(!LST || (TPP == 1 && !STG), "lists: one lane per particle, unstaged");
    static_assert(!FUS || (LST && LEAN && !OPT), "fused predictor: lists, lean physics");
    const int tid = threadIdx.x;
    const int sub = (TPP == 1) ? 0 : (tid & (TPP - 1));
    const bool from_a = FUS && sort_skipped(F.rs);
    const float4* __restrict__ xsrc = from_a ? F.A.xh : B.xh;
    float4 xi = make_float4(0.f, 0.f, 0.f, 1.f), vi = xi, rpi = xi;
    int it = 0;
    if (valid && from_a) {
        xi = F.A.xh[s];
        it = F.A.itype[s];
        vi = F.A.vm[s];
        rpi = B.rp[s];
        if (it > 0 && F.hdt != 0.f) {  // predictor, as the density pass applied it
            const float4 ap = F.A.ap[s];
            vi.x = fmaf(F.hdt, ap.x, vi.x);
            vi.y = fmaf(F.hdt, ap.y, vi.y);
            if (DIM == 3) vi.z = fmaf(F.hdt, ap.z, vi.z);
        }
    } else if (valid) {
        xi = B.xh[s];
        it = B.itype[s];
        vi = B.vm[s];
        rpi = B.rp[s];
    }
    // The next state goes to the slot of this sort, or with mirror ghosts
    // (wall_model 3) to the particle's own index, the ghosts being dropped.
    const bool ghosts = !LEAN && P.wall_model == 3;
    if (valid && (it <= 0 || !g.ok) && sub == 0) {  // wall: fixed state, zero rates
        const int id = from_a ? F.A.id[s] : B.id[s];
        if (!ghosts || id < P.n_real) {
            const int o = ghosts ? id : s;
            A.xh[o] = xi;
            A.vm[o] = vi;
            A.u[o] = from_a ? F.A.u[s] : B.vmin[s].w;
            A.ap[o] = make_float4(0.f, 0.f, 0.f, 0.f);
            A.rho[o] = rpi.x;
            A.p[o] = from_a ? F.A.p[s] : B.p[s];
            A.itype[o] = it;
            A.id[o] = id;
            if (A.inst) A.inst[o] = B.inst[s];
        }
    }
    const bool work = valid && it > 0 && g.ok;
    const float ihf = DIM == 2 ? __fdividef(1.0f, xi.w) : __frcp_rn(xi.w);
    const float kgih_i = P.kg * pow_grad<DIM>(ihf);
    float4 ti = make_float4(0.f, 0.f, 0.f, 0.f), ti2 = make_float4(0.f, 0.f, 0.f, 0.f);
    const bool visc = !LEAN && P.visc, heat_art = !LEAN && P.heat_art;
    if (work && visc) {
        ti = B.tau[s];
        if (DIM == 3) ti2 = B.tau2[s];
    }
    const float ulo_i = (work && heat_art) ? B.ulo[s] : 0.f;
    // Pair sums in the order of the walk (an entry beyond the support adds a zero,
    // so lists and cell walks in the same order sum alike): acceleration, twice
    // the pressure and art_visc energy rate, art_heat's.
    const f2 zero2 = bc2(0.f);
    float a0 = 0.f, a1 = 0.f, a2 = 0.f, e_sum = 0.f, ah_du = 0.f;
    // single_step options: continuity drho/dt, XSPH velocity, div v for h
    const bool cont = OPT && P.density_form == 1, xsph = OPT && P.xsph, sle2 = OPT && P.sle == 2;
    float drho_s = 0.f, divh = 0.f, x0s = 0.f, x1s = 0.f, x2s = 0.f;
    bool done = !work;
    // A listed particle walks its neighbour list (coalesced rows of entries);
    // the others decode the density pass's bits.
    const int lpk = (LST && work) ? __ldg(B.ncount + s) : -1;
    const int lc = lpk >= 0 ? list_near(lpk) + list_far(lpk) : -1;  // entries (-1: no list)
    if (LST) prefetch_list(B.nlist, B.lstride, s, lc);
    // The place of an absent entry (the odd end of a list, a lane without
    // entries): the particle itself, whose terms vanish with d = 0 and dv = 0 unless
    // one of its own values is infinite (a particle without mass that is alone has no
    // density). The cell walk leaves those out by selects (ina, inb below); a listed
    // particle with such values walks its cells (the density pass says so): putting the
    // entries past the end of every list out of reach instead took 36 us of a 2.03 M dam
    // break's 2,732 (six iterations).
    int kself = valid ? s : 0;
    if (STG) kself = work ? s + SV.shift[DIM == 2 ? g.reach : g.reach * (2 * g.reach + 2)] : 0;
    const float k_alpha = P.visc_art ? P.av_alpha * P.c0 : 0.f;        // times h_i + h_j
    const float k_beta = P.visc_art ? 0.5f * P.av_beta : 0.f;          // times (h_i + h_j)^2
    // Push between particles of different type (ArmandoThrust/armando.cu:507-513
    // for wall_model 1, acpu.c:424-429 for 2) along (x_i - x_j)/r, c = c0; with
    // wall_model 1 the pair's only interaction: true, its mass zeroed.
    auto push = [&](const int k, const float4& xj, float rhoj, float e0, float e1, float e2, float dr2,
                    float tt, float t, float ih, float& mj, float& p0, float& p1, float& p2) {
        if (__ldg(B.itype + k) == it) return false;
        const float r = fast_sqrt_pos(dr2);
        if (dr2 > 2.0f * kTinyDr2 && t < 0.f) {
            const float w = 0.0625f * tt * tt * fmaf(2.0f, t, 5.0f);  // W / W(0)
            const float c2 = P.c0 * P.c0;
            float f;
            if (P.wall_model == 1) {
                const float alpha = P.kw_hi * (DIM == 2 ? ih * ih : ih * ih * ih);
                f = 0.5f * alpha * w * mj / (rhoj * xj.w) * c2;
            } else {
                f = 0.02f * w * c2 / r * mj / (mass_of<DIM>(xi, vi) + mj);
            }
            f /= r;
            p0 = fmaf(f, e0, p0);
            p1 = fmaf(f, e1, p1);
            if (DIM == 3) p2 = fmaf(f, e2, p2);
        }
        if (P.wall_model != 1) return false;
        mj = 0.f;
        return true;
    };
    // Terms of two entries (pressure, viscosity, art_visc, art_heat, options).
    // va, vb: the neighbours' 2D {vx, vy, rho, P} (ra, rb unused) or 3D v and
    // {rho, P, u, psi}. No pair test: the kernel's gradient is zero beyond its
    // support, so the entries in the skin margin add nothing. P of a particle
    // without density (no mass near it) is not finite, and a zero gradient times
    // it no zero: `taking` leaves out what the margin and absent entries have there.
    // ina, inb: whether the entries are real (without lists).
    //
    // Pressure, art_visc and their energy rates share one factor per pair: with
    // s = m_j G (grad W = G d), T = P_i + P_j + Pi_ij and dv = v_j - v_i,
    //   a_i -= s T d,   du_i -= s T (dv.d) / 2
    // (internal_force.f:179-428 and art_visc.f:71-100 summed), G = kg (q - 2)^3.
    // art_visc: Pi_ij = alpha c0 A + beta rho_bar A^2, A = mh (dv.d)+ / (rho_bar
    // (r^2 + (eta mh)^2)): one reciprocal, of rho_bar's and the distance's product,
    // serves both of its divisions, and (dv.d)+ = max(dv.d, 0) its condition.
    // In 2D the pressure's products are rounded in the order of the written formula,
    // m_j ((P_i + P_j) (G d)), and Pi_ij's terms added by themselves: the pressure terms
    // nearly cancel in a column of water at rest, and with the shared factor their
    // rounding moved 2,000 coordinates of a 2.03 M dam break by an ulp in 6 iterations,
    // which then move dv/dt there by up to 8e-4.
    // The pass was bound by issue (62% of cycles) and its neighbours' loads: about 80
    // instructions an entry, 50 now. Measured: 2D lists (2.03 M dam break) 0.213 ->
    // 0.160 ms, 3D lists (8.78 M channel) 6.77 -> 4.41 ms (3.84 with blocks of entries),
    // 2D cells (42 k) 17.6 -> 16.1 us (10.5 with bits decoded by rows).
    // UNI: every particle has the same h (g.huni), whose factors are constants.
    // PH: the physics beyond pressure and art_visc compiled in, bits 1 art_heat,
    // 2 physical viscosity, 4 repulsive walls and the single_step options.
    auto pair2 = [&](auto uni, auto ph, const bool ina, const bool inb, const int ka, const int kb,
                     const float4& xa, const float4& xb, const float4& va, const float4& vb, const float4& ra,
                     const float4& rb) {
        constexpr bool UNI = decltype(uni)::value;
        constexpr int PH = decltype(ph)::value;
        f2 d0 = make_float2(xi.x - xa.x, xi.x - xb.x), d1 = make_float2(xi.y - xa.y, xi.y - xb.y);
        f2 d2 = DIM == 3 ? make_float2(xi.z - xa.z, xi.z - xb.z) : zero2;
        if (g.periodic[0]) d0 = min_image2(d0, xi.x, xa.x, xb.x, g, 0);
        if (g.periodic[1]) d1 = min_image2(d1, xi.y, xa.y, xb.y, g, 1);
        if (DIM == 3 && g.periodic[2]) d2 = min_image2(d2, xi.z, xa.z, xb.z, g, 2);
        const f2 dd0 = fma2(d0, d0, bc2(kTinyDr2));
        const f2 dr2 = DIM == 2 ? add2(dd0, prod2(d1, d1)) : fma2(d2, d2, fma2(d1, d1, dd0));
        f2 mj = DIM == 2 ? make_float2(xa.z, xb.z) : make_float2(va.w, vb.w);
        f2 ih = bc2(ihf), kg = bc2(kgih_i), hs = bc2(2.0f * xi.w);
        if (!UNI) {
            hs = make_float2(xi.w + xa.w, xi.w + xb.w);
            ih = mul2(bc2(2.0f), rcp2(hs));
            const f2 ih2 = mul2(ih, ih);
            kg = mul2(bc2(P.kg), mul2(ih2, ih2));
            if (DIM == 3) kg = mul2(kg, ih);
        }
        const f2 r = mul2(dr2, rsqrt2(dr2));
        // q - 2, 0 beyond the support
        const f2 t = min2(DIM == 2 ? add2(prod2(r, ih), bc2(-2.0f)) : fma2(r, ih, bc2(-2.0f)), 0.0f);
        const f2 tt = mul2(t, t);
        auto taking = [&](f2 v) {
            return LST ? within2(t, v) : make_float2(ina ? v.x : 0.f, inb ? v.y : 0.f);
        };
        const f2 rhoj = DIM == 2 ? make_float2(va.z, vb.z) : make_float2(ra.x, rb.x);
        bool pa = false, pb = false;  // push only: nothing else of the other is read
        if ((PH & 4) && repulsive_walls(P)) {
            pa = push(ka, xa, rhoj.x, d0.x, d1.x, d2.x, dr2.x, tt.x, t.x, ih.x, mj.x, a0, a1, a2);
            pb = push(kb, xb, rhoj.y, d0.y, d1.y, d2.y, dr2.y, tt.y, t.y, ih.y, mj.y, a0, a1, a2);
        }
        auto others = [&](f2 v) { return make_float2(pa ? 0.f : v.x, pb ? 0.f : v.y); };
        const f2 gw = mul2(mul2(mul2(kg, t), t), t);  // G (2D)
        const f2 sm = DIM == 2 ? mul2(mj, gw) : mul2(mul2(tt, t), mul2(mj, kg));
        const f2 vx = others(make_float2(va.x - vi.x, vb.x - vi.x)), vy = others(make_float2(va.y - vi.y, vb.y - vi.y));
        const f2 vz = DIM == 3 ? others(make_float2(va.z - vi.z, vb.z - vi.z)) : zero2;
        f2 vr = fma2(vy, d1, mul2(vx, d0));
        if (DIM == 3) vr = fma2(vz, d2, vr);
        const f2 rs = make_float2(rpi.x + rhoj.x, rpi.x + rhoj.y);
        f2 T = DIM == 2 ? make_float2(rpi.y + va.w, rpi.y + vb.w) : make_float2(rpi.y + ra.y, rpi.y + rb.y);
        f2 sv = sm;  // the viscous terms' factor
        if (P.pa_sph != 1) {
            f2 irr = rcp2(mul2(bc2(rpi.x), rhoj));
            if (PH & 2) irr = taking(irr);
            T = mul2(T, irr);
            sv = mul2(sv, irr);
        }
        T = others(taking(T));
        const f2 hs2 = UNI ? bc2(4.0f * xi.w * xi.w) : mul2(hs, hs);
        const f2 D = UNI ? add2(dr2, bc2(P.av_eta2 * (xi.w * xi.w)))
                         : fma2(hs2, bc2(0.25f * P.av_eta2), dr2);
        const f2 rc = rcp_prod2(D, rs);
        const f2 A = mul2(max2(vr, 0.0f), rc);
        const f2 ka2 = UNI ? bc2(k_alpha * (2.0f * xi.w)) : mul2(bc2(k_alpha), hs);
        f2 V = DIM == 2 ? mul2(A, ka2) : fma2(A, ka2, T);  // Pi_ij (3D: and T)
        if (k_beta != 0.f) V = fma2(mul2(mul2(A, A), rs), mul2(bc2(k_beta), hs2), V);
        const f2 c = neg2(mul2(sm, DIM == 2 ? add2(T, V) : V));
        if (DIM == 2) {  // m_j ((-T) (G d)), then -(m_j Pi_ij) (G d)
            const f2 w0 = mul2(gw, d0), w1 = mul2(gw, d1), fs = neg2(T), mv = neg2(mul2(mj, V));
            const f2 h0 = mul2(fs, w0), h1 = mul2(fs, w1);
            a0 = fmaf(mv.x, w0.x, fmaf(mj.x, h0.x, a0));
            a1 = fmaf(mv.x, w1.x, fmaf(mj.x, h1.x, a1));
            a0 = fmaf(mv.y, w0.y, fmaf(mj.y, h0.y, a0));
            a1 = fmaf(mv.y, w1.y, fmaf(mj.y, h1.y, a1));
        } else {
            a0 = dot2(c, d0, a0);
            a1 = dot2(c, d1, a1);
            a2 = dot2(c, d2, a2);
        }
        e_sum = dot2(c, vr, e_sum);
        if (cont) drho_s = dot2(neg2(sm), vr, drho_s);  // con_density, density.f:203-216
        if (sle2) {                                   // hsml.f:75-90
            const f2 dq = taking(make_float2(__fdiv_rn(sm.x, rhoj.x), __fdiv_rn(sm.y, rhoj.y)));
            divh = dot2(dq, vr, divh);
        }
        if (xsph) {  // av_vel.f:47-58: -eps m_j / rho_ij (v_i - v_j) W_ij, eps = 0.3
            const f2 ih2 = mul2(ih, ih);
            // W = kw ih^dim (q - 2)^4 (2 (q - 2) + 5) / 16; 0.3 / rho_bar = 0.6 / rs
            f2 wv = mul2(mul2(mul2(tt, tt), fma2(bc2(2.0f), t, bc2(5.0f))), mul2(bc2(0.0625f * P.kw_hi), ih2));
            if (DIM == 3) wv = mul2(wv, ih);
            const f2 cx = taking(div2(mul2(mul2(bc2(0.6f), mj), wv), rs));
            x0s = dot2(cx, vx, x0s);
            x1s = dot2(cx, vy, x1s);
            if (DIM == 3) x2s = dot2(cx, vz, x2s);
        }
        if ((PH & 2) && visc) {
            const int ia = pa ? s : ka, ib = pb ? s : kb;  // (sv is 0 there)
            const float4 qa = __ldg(B.tau + ia), qb = __ldg(B.tau + ib);
            const f2 sxx = make_float2(ti.x + qa.x, ti.x + qb.x), syy = make_float2(ti.y + qa.y, ti.y + qb.y);
            const f2 sxy = make_float2(ti.z + qa.z, ti.z + qb.z);
            f2 h0 = fma2(sxy, d1, mul2(sxx, d0)), h1 = fma2(syy, d1, mul2(sxy, d0));
            if (DIM == 3) {
                const float4 ua = __ldg(B.tau2 + ia), ub = __ldg(B.tau2 + ib);
                const f2 szz = make_float2(ti.w + qa.w, ti.w + qb.w);
                const f2 sxz = make_float2(ti2.x + ua.x, ti2.x + ub.x), syz = make_float2(ti2.y + ua.y, ti2.y + ub.y);
                h0 = fma2(sxz, d2, h0);
                h1 = fma2(syz, d2, h1);
                a2 = dot2(sv, fma2(szz, d2, fma2(syz, d1, mul2(sxz, d0))), a2);
            }
            a0 = dot2(sv, h0, a0);
            a1 = dot2(sv, h1, a1);
        }
        if ((PH & 1) && heat_art) {  // art_heat.f:69-97: grad W . d = G r^2
            f2 rh = rc;
            if (P.ah_eta2 != P.av_eta2)
                rh = rcp_prod2(fma2(hs2, bc2(0.25f * P.ah_eta2), dr2), rs);
            float4 qa = ra, qb = rb;
            if (DIM == 2) {  // u and psi are not in the 2D record
                qa = __ldg(B.rp + ka);
                qb = __ldg(B.rp + kb);
            }
            const f2 ps = make_float2(rpi.w + qa.w, rpi.w + qb.w);
            const f2 lo = make_float2(ulo_i - __ldg(B.ulo + ka), ulo_i - __ldg(B.ulo + kb));
            const f2 du2 = others(add2(make_float2(rpi.z - qa.z, rpi.z - qb.z), lo));
            const f2 pr = others(taking(mul2(ps, rh)));
            ah_du = dot2(mul2(mul2(mul2(sm, dr2), pr), bc2(2.0f)), du2, ah_du);
        }
    };
    // The entries, two at a time, with every particle's h alike or not.
    auto walk = [&](auto uni, auto ph) {
    // A listed particle takes each entry's terms as the entry is read, without
    // a candidate list; the mask decoding and cell walk below serve the others.
    if (LST) {
        constexpr int NB = DIM == 2 ? 4 : 2;  // entries whose loads issue together (registers)
        const int nb = blocks_of(lc);
        const int bm = __reduce_max_sync(0xffffffffu, nb);
        // 3D: the next block is loaded ahead (8.78 M: 3.89 -> 3.84 ms; 2D, 2.03 M, would
        // lose: 161 -> 163 us)
        constexpr bool kAhead = DIM == 3;
        int4 kn = kAhead ? list_block(B.nlist, B.lstride, s, 0, nb, kself) : make_int4(0, 0, 0, 0);
        for (int b = 0; b < bm; ++b) {
            const int4 q = kAhead ? kn : list_block(B.nlist, B.lstride, s, b, nb, kself);
            if (kAhead && b + 1 < bm) kn = list_block(B.nlist, B.lstride, s, b + 1, nb, kself);
            const int kb[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
            for (int v = 0; v < 4; v += NB) {
                float4 xb[NB], va[NB], rb[NB];
#pragma unroll
                for (int u = 0; u < NB; ++u) {
                    xb[u] = __ldg(xsrc + kb[v + u]);
                    va[u] = __ldg((DIM == 2 ? B.vr : B.vm) + kb[v + u]);
                    rb[u] = DIM == 3 ? __ldg(B.rp + kb[v + u]) : va[u];
                }
#pragma unroll
                for (int u = 0; u < NB; u += 2)
                    pair2(uni, ph, true, true, kb[v + u], kb[v + u + 1], xb[u], xb[u + 1], va[u], va[u + 1], rb[u], rb[u + 1]);
            }
        }
        if (lc >= 0) done = true;
        if (!__any_sync(0xffffffffu, !done)) return;
        if (!done) {  // what its absent entries left
            a0 = a1 = a2 = e_sum = ah_du = 0.f;
            drho_s = divh = x0s = x1s = x2s = 0.f;
        }
    }
    if (!__any_sync(0xffffffffu, !done)) return;
    constexpr int W = mask_words<DIM>() / TPP;  // mask words of this lane
    constexpr int CW = mask_chunk<W>();
    const size_t mlane = (size_t)s * TPP + sub;
    CellCoord cc = {{0, 0, 0}};
    Cursor cu = cursor_begin<DIM>(g);
    // The density pass left the neighbour bits of the candidates (word-major).
    bool from_mask = false;
    uint4 ch = make_uint4(0u, 0u, 0u, 0u);  // mask chunk being decoded
    unsigned wbits = 0u;                    // bits left of word wi
    if (!done) {
        cc = decode_key<DIM>(keys[s], g);
        ch = mask_load_chunk<W>(B.nmask, B.mstride, mlane, 0);
        wbits = ch.x;
        from_mask = !(ch.x == ~0u && (W == 1 || ch.y == ~0u));
    }
    // 2D: as many bits as fit the list are decoded row by row, a few instructions
    // each; with the cursor's state they took 80 a bit. Measured: 1,920 particles 14.8
    // -> 10.1 us, 42 k 15.6 -> 10.5, 2.03 M 265 -> 172, 2.76 M in 64 instances 402 -> 316.
    [[maybe_unused]] const bool by_rows = DIM == 2 && TPP == 1 && from_mask &&
                         __popc(ch.x) + __popc(ch.y) + __popc(ch.z) + __popc(ch.w) <= cap_force<LST>();
    int wi = 0, rbase = 0;  // index of wbits; ordinal of the cursor row's first slot
    int shift = 0;          // staged index - slot in the cursor's row
    while (__any_sync(0xffffffffu, !done)) {
        int nl = 0;
        if constexpr (DIM == 2 && TPP == 1) {
            if (!done && by_rows) {
                mask_slots(ch, g, start, cc, [&](const int k, const int r) {
                    s_list[nl++][tid] = (LT)(STG ? k + SV.shift[r] : k);
                });
                done = true;
            }
        }
        while (!done && from_mask) {
            if (nl == cap_force<LST>()) break;
            while (wbits == 0u && wi < W - 1) {
                ++wi;
                if (W > CW && wi % CW == 0) ch = mask_load_chunk<W>(B.nmask, B.mstride, mlane, wi / CW);
                wbits = chunk_word(ch, wi % CW);
            }
            if (wbits == 0u) {
                done = true;
                break;
            }
            const int o = 32 * wi + __ffs(wbits) - 1;
            wbits &= wbits - 1u;
            bool in_rows = true;
            while (o >= rbase + lane_len<TPP>(cu)) {  // move to the range holding ordinal o
                rbase += lane_len<TPP>(cu);
                if (!cursor_next<DIM>(g, start, cc, cu)) {
                    in_rows = false;
                    break;
                }
                cu.k += sub;
                if (STG) shift = SV.shift[cursor_row<DIM>(cu, g.reach)];
            }
            if (!in_rows) {  // cannot happen for a mask of this step's candidates
                done = true;
                break;
            }
            s_list[nl++][tid] = (LT)(cu.k + TPP * (o - rbase) + (STG ? shift : 0));
        }
        while (!done && !from_mask) {
            int kb[kTestBatch];
            int cnt;
            float4 xb[kTestBatch];
            if (cu.k >= cu.ke) {
                if (!cursor_next<DIM>(g, start, cc, cu)) {
                    done = true;
                    break;
                }
                if (STG) shift = SV.shift[cursor_row<DIM>(cu, g.reach)];
                if (TPP > 1) {
                    cu.k += sub;
                    continue;
                }
            }
            if (nl > cap_force<LST>() - kTestBatch) break;
            const int k0 = cu.k;
            cnt = min(kTestBatch, lane_len<TPP>(cu));
#pragma unroll
            for (int u = 0; u < kTestBatch; ++u) {
                const int ku = min(k0 + u * TPP, cu.ke - 1);
                kb[u] = k0 + u * TPP;
                xb[u] = STG ? SV.x[ku + shift] : __ldg(xsrc + ku);
            }
            cu.k += cnt * TPP;
#pragma unroll
            for (int u = 0; u < kTestBatch; ++u) {
                float d[3], dr2;
                const int k = kb[u];
                if (u < cnt && k != s && pair_delta<DIM>(xi, xb[u], g, d, dr2))
                    s_list[nl++][tid] = (LT)(STG ? k + shift : k);
            }
        }
        const int ml = __reduce_max_sync(0xffffffffu, nl);
        for (int t = 0; t < ml; t += 2) {
            int kb[2];
            float4 xb[2], va[2], rb[2];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int k = kb[u] = t + u < nl ? (int)s_list[t + u][tid] : kself;
                xb[u] = STG ? SV.x[k] : __ldg(xsrc + k);
                va[u] = STG ? SV.v[k] : __ldg((DIM == 2 ? B.vr : B.vm) + k);
                rb[u] = DIM == 2 ? va[u] : STG ? SV.r[k] : __ldg(B.rp + k);
                if (LST && t + u >= nl) xb[u].x = kOutOfReach;
            }
            pair2(uni, ph, t < nl, t + 1 < nl, kb[0], kb[1], xb[0], xb[1], va[0], va[1], rb[0], rb[1]);
        }
    }
    };
    using std::integral_constant;
    if constexpr (LEAN) {
        if (TPP == 1 && g.huni) walk(std::true_type{}, integral_constant<int, 0>{});
        else walk(std::false_type{}, integral_constant<int, 0>{});
    } else if constexpr (TPP == 1 && !OPT) {
        if (g.huni && !repulsive_walls(P) && !P.visc) walk(std::true_type{}, integral_constant<int, 1>{});
        else if (g.huni && !repulsive_walls(P) && !P.heat_art) walk(std::true_type{}, integral_constant<int, 2>{});
        else walk(std::false_type{}, integral_constant<int, 7>{});
    } else {
        walk(std::false_type{}, integral_constant<int, 7>{});
    }
    if (TPP > 1) {  // the particle's lanes reach this point together
        a0 = group_sum<TPP>(a0);
        a1 = group_sum<TPP>(a1);
        if (DIM == 3) a2 = group_sum<TPP>(a2);
        e_sum = group_sum<TPP>(e_sum);
        ah_du = group_sum<TPP>(ah_du);
        if (cont) drho_s = group_sum<TPP>(drho_s);
        if (sle2) divh = group_sum<TPP>(divh);
        if (xsph) {
            x0s = group_sum<TPP>(x0s);
            x1s = group_sum<TPP>(x1s);
            if (DIM == 3) x2s = group_sum<TPP>(x2s);
        }
    }
    if (!work || sub != 0) return;
    float du = fmaf(0.5f, e_sum, ah_du);  // internal_force.f:433-435
    if (visc) du += B.tds[s];
    if (S.heat_on) {
        float e0 = xi.x - P.heat_center[0], e1 = xi.y - P.heat_center[1];
        float dd = fmaf(e1, e1, __fmul_rn(e0, e0));
        if (DIM == 3) {
            float e2 = xi.z - P.heat_center[2];
            dd = fmaf(e2, e2, dd);
        }
        du += P.heat_q0 * expf(-dd * P.heat_k) / rpi.x;
    }
    a0 += P.gravity[0];
    a1 += P.gravity[1];
    if (DIM == 3) a2 += P.gravity[2];
    // Corrector (time_integration.f:186-218).
    float4 vmin;
    if (from_a) {
        const float4 v0 = F.A.vm[s];
        vmin = make_float4(v0.x, v0.y, v0.z, F.A.u[s]);
    } else {
        vmin = B.vmin[s];
    }
    float4 vn = vi;
    vn.x = fmaf(S.kdt, a0, vmin.x);
    vn.y = fmaf(S.kdt, a1, vmin.y);
    if (DIM == 3) vn.z = fmaf(S.kdt, a2, vmin.z);
    if (xsph && S.hdt != 0.f) {  // time_integration.f:195: v = v_min + dt dv + av
        vn.x += x0s;
        vn.y += x1s;
        if (DIM == 3) vn.z += x2s;
    }
    float un = fmaf(S.kdt, du, vmin.w);
    if (un < 0.f) un = 0.f;
    float4 xn = xi;
    float rho_out = rpi.x;
    if (cont) rho_out = fmaf(S.kdt, drho_s, B.q[s]);  // time_integration.f:191-193, 207-209
    if (OPT && P.sle == 1) {  // hsml.f:45-48, exponent the single-precision 1./dim
        const float mr = __fdiv_rn(mass_of<DIM>(xi, vi), rpi.x);
        xn.w = 2.0f * (DIM == 2 ? sqrtf(mr) : powf(mr, 1.0f / 3.0f));
    } else if (sle2) {  // hsml.f:92-96
        const float hn = fmaf(S.dt, __fmul_rn(xi.w * (1.0f / DIM), divh), xi.w);
        if (!(hn <= 0.f)) xn.w = hn;
    }
    xn.x = fmaf(S.dt, vn.x, xi.x);
    xn.y = fmaf(S.dt, vn.y, xi.y);
    if (DIM == 3) xn.z = fmaf(S.dt, vn.z, xi.z);
    bool outside = false;
    if (P.periodic[0]) xn.x = wrap_axis(xn.x, P, 0, outside);
    if (P.periodic[1]) xn.y = wrap_axis(xn.y, P, 1, outside);
    if (DIM == 3 && P.periodic[2]) xn.z = wrap_axis(xn.z, P, 2, outside);
    if (outside) atomicOr(flags, (unsigned)FLAG_OUT_OF_GRID);
    if (g.half_skin2 > 0.f && B.xsort) {  // moved more than half the skin since the sort: sort next
        const float4 x0 = B.xsort[s];
        const float e0 = xn.x - x0.x, e1 = xn.y - x0.y, e2 = (DIM == 3) ? xn.z - x0.z : 0.f;
        if (e0 * e0 + e1 * e1 + e2 * e2 > g.half_skin2 && *(volatile unsigned*)(flags + 2) == 0u)
            atomicExch(flags + 2, 1u);
    }
    const float chk = xn.x + xn.y + xn.z + vn.x + vn.y + vn.z + un + a0 + a1 + a2 + du;
    if (!isfinite(chk)) atomicOr(flags, (unsigned)FLAG_NONFINITE);
    const int id = from_a ? F.A.id[s] : B.id[s];
    const int o = ghosts ? id : s;
    A.xh[o] = xn;
    A.vm[o] = vn;
    A.u[o] = un;
    A.ap[o] = make_float4(a0, a1, a2, du);
    A.rho[o] = rho_out;
    if (A.drho) A.drho[o] = drho_s;
    A.p[o] = B.p[s];
    A.itype[o] = it;
    A.id[o] = id;
    if (A.inst) A.inst[o] = B.inst[s];
}

// ---------------------------------------------------------------------------
// Pass kernels of one particle system: one CTA per 128 consecutive slots.
// ---------------------------------------------------------------------------
// The grid of a pass; PER = false (no periodic axis) makes the periodic flags
// compile-time zeros, so the minimum-image code and its registers drop out.
template <bool PER>
__device__ __forceinline__ DevGrid load_grid(const DevGrid* __restrict__ gp) {
    DevGrid g = *gp;
    if (!PER) g.periodic[0] = g.periodic[1] = g.periodic[2] = 0;
    return g;
}

// One CTA per BS / TPP consecutive slots.
template <int DIM, int TPP, int BS, bool PER, bool LEAN, bool OPT = false, bool LST = false,
          bool FUS = false>
__global__ void __launch_bounds__(BS, 1024 / BS)
    k_density(StateB B, const unsigned* __restrict__ keys, const int* __restrict__ start,
              const DevGrid* __restrict__ gp, DevParams P, int n, FusedSrc F) {
    __shared__ int s_near[cap_density<LST>()][BS];
    __shared__ int s_far[cap_density<LST>()][BS];
    const int s = blockIdx.x * (BS / TPP) + (int)threadIdx.x / TPP;
    const DevGrid g = load_grid<PER>(gp);
    density_body<DIM, TPP, BS, LEAN, OPT, false, int, LST, FUS>(B, keys, start, g, P, s, s < n,
                                                                s_near, s_far, StageView{}, F);
}

// Neighbour lists of an iteration that sorts (lazy sorting), built in the
// sort's conditional body after the cell table: for each slot s of the new
// order, the candidates k != s (cursor order) within h_s + h_k + skin, the
// bound widened by 2^-14 over the rounding of the FP32 distances; in 2D the
// pairs the density pass evaluates in FP32 (q >= list_near_q2() at the sort) after
// the others (collected from the last block down, then moved up). Positions are those
// in cell order (B.xsort; the reorder of the rest comes later in the iteration). Until
// the next sort every particle stays within half the skin of where it was binned, so
// every pair the exact test accepts (r < h_i + h_j) on those iterations is in the list.
//
// OWN (the GPU-C schemes): the candidates within 2 h_s + skin, all of them near.
//
// The build was bound by issue (76% of cycles, 22 of 32 lanes, 22 k instructions a
// warp in 3D): a general cursor step per row of cells, minimum-image branches and
// the pair's own bound per candidate, a far entry stored twice. The rows are plain
// loops here, a wrapped row shifts the particle once instead of each difference, the
// bound is a constant when every h is alike and four candidates are tested together.
// Single entries, stored as found, touched 15 sectors a warp and entry, the lanes
// being at different rows; four leave as one int4, and the passes read four at a
// time. They wait in shared memory (a store and an index; collected in registers they
// took seven instructions and a branch each), and the particle's own row is walked
// around it instead of asking each candidate. Measured a build: 185 k particles (3D)
// 208 -> 141 us, 8.78 M 6.60 -> 3.77 ms, 2.03 M (2D) 222 -> 214 us, the last now
// waiting for its loads. (Skipping the cells beyond the bound's sphere: 162 -> 173 us.)
template <int DIM, bool PER, bool OWN = false>
__global__ void __launch_bounds__(kPassThreads)
    k_build_list(StateB B, const unsigned* __restrict__ keys, const int* __restrict__ start,
                 const DevGrid* __restrict__ gp, int n, const int* __restrict__ resort = nullptr) {
    if (sort_skipped(resort)) return;
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    const DevGrid g = load_grid<PER>(gp);
    if (!g.ok) {
        B.ncount[s] = 0;
        return;
    }
    constexpr bool SPLIT = DIM == 2 && !OWN;
    constexpr float kNear2 = 0.25f * list_near_q2() * list_near_q2();
    const float4 xi = B.xsort[s];
    const CellCoord cc = decode_key<DIM>(keys[s], g);
    const int f = g.reach;
    const float pad = (1.0f + 0x1p-14f);
    const bool uni = OWN || g.huni;
    auto bound2 = [&](float hk) {
        const float lim = __fmul_rn(__fadd_rn(__fadd_rn(xi.w, hk), g.skin), pad);
        return __fmul_rn(lim, lim);
    };
    const float lim_u = bound2(xi.w), near_u = kNear2 * (2.0f * xi.w) * (2.0f * xi.w);
    // Entries wait in the thread's column of a ring in shared memory; whole blocks of
    // four leave it for global memory.
    __shared__ int s_ring[SPLIT ? 2 : 1][kRing][kPassThreads];
    int(*const ring_n)[kPassThreads] = s_ring[0];
    int(*const ring_f)[kPassThreads] = s_ring[SPLIT ? 1 : 0];
    const int tid = threadIdx.x;
    int cn = 0, cf = 0;  // near and far entries
    int bn = 0, bf = 0;  // those of them stored: near blocks upwards from the first, far
                         // ones downwards from the last
    const int last = list_blocks(B.lcap) - 1;
    int4* const l4 = reinterpret_cast<int4*>(B.nlist) + s;
    auto flush = [&](int(*const ring)[kPassThreads], const int count, int& done, const bool up) {
        for (; count - done >= 4; done += 4) {
            const int t = done & (kRing - 1);
            const int4 q = make_int4(ring[t][tid], ring[t + 1][tid], ring[t + 2][tid], ring[t + 3][tid]);
            const int b = up ? done >> 2 : last - (done >> 2);
            if (cn + cf <= B.lcap) l4[(size_t)b * B.lstride] = q;
        }
    };
    auto add_near = [&](int k) { ring_n[cn++ & (kRing - 1)][tid] = k; };
    auto add_far = [&](int k) { ring_f[cf++ & (kRing - 1)][tid] = k; };
    // Slots [kb, ke) against the particle at (x, y, z) (wrapped rows: shifted).
    auto range = [&](int kb, int ke, float x, float y, float z) {
        for (int k0 = kb; k0 < ke; k0 += 4) {
            const float4* const src = B.xsort + k0;  // (kListPad entries past the last slot)
            float4 xb[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) xb[u] = __ldg(src + u);
            if (cn - bn > kRing - 4) flush(ring_n, cn, bn, true);
            if (SPLIT && cf - bf > kRing - 4) flush(ring_f, cf, bf, false);
#pragma unroll
            for (int u = 0; u < 4; u += 2) {
                const f2 d0 = make_float2(x - xb[u].x, x - xb[u + 1].x);
                const f2 d1 = make_float2(y - xb[u].y, y - xb[u + 1].y);
                f2 r2 = fma2(d1, d1, mul2(d0, d0));
                if (DIM == 3) {
                    const f2 d2 = make_float2(z - xb[u].z, z - xb[u + 1].z);
                    r2 = fma2(d2, d2, r2);
                }
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int k = k0 + u + e;
                    const float rr = e ? r2.y : r2.x, hk = xb[u + e].w;
                    const bool in = rr < (uni ? lim_u : bound2(hk)) && k < ke;
                    const bool near = !SPLIT || rr < (uni ? near_u : kNear2 * (xi.w + hk) * (xi.w + hk));
                    if (in && near) add_near(k);
                    if (SPLIT && in && !near) add_far(k);
                }
            }
        }
    };
    const int c0 = max(cc.c[0] - f, 0), c1 = min(cc.c[0] + f, g.n[0] - 1) + 1;
    for (int dz = DIM == 3 ? -f : 0; dz <= (DIM == 3 ? f : 0); ++dz) {
        int cz = cc.c[2] + dz;
        float z = xi.z;
        if (DIM == 3 && (cz < 0 || cz >= g.n[2])) {
            if (!PER || !g.periodic[2]) continue;
            z += cz < 0 ? g.L[2] : -g.L[2];
            cz += cz < 0 ? g.n[2] : -g.n[2];
        }
        for (int dy = -f; dy <= f; ++dy) {
            int cy = cc.c[1] + dy;
            float y = xi.y;
            if (cy < 0 || cy >= g.n[1]) {
                if (!PER || !g.periodic[1]) continue;
                y += cy < 0 ? g.L[1] : -g.L[1];
                cy += cy < 0 ? g.n[1] : -g.n[1];
            }
            const int* row = start + g.cell_off + (cz * g.n[1] + cy) * g.n[0];
            const int b = __ldg(row + c0), e = __ldg(row + c1);
            const bool own = dy == 0 && dz == 0;  // the particle's row: around itself
            range(b, own ? s : e, xi.x, y, z);
            if (own) range(s + 1, e, xi.x, y, z);
            if (PER && g.periodic[0]) {  // the part of the row past either end
                if (cc.c[0] < f)
                    range(__ldg(row + cc.c[0] - f + g.n[0]), __ldg(row + g.n[0]), xi.x + g.L[0], y, z);
                else if (cc.c[0] + f >= g.n[0])
                    range(__ldg(row), __ldg(row + cc.c[0] + f - g.n[0] + 1), xi.x - g.L[0], y, z);
            }
            flush(ring_n, cn, bn, true);
        }
    }
    if (cn + cf > B.lcap) {
        B.ncount[s] = -1;
        return;
    }
    B.ncount[s] = cn | (cf << 16);
    flush(ring_n, cn, bn, true);
    if (SPLIT) {
        // The far entries behind the near ones, the latest first: those in the ring, then
        // the blocks upwards from the last one stored. A block is read before the near
        // side, at most (cn + cf) / 4 blocks, can reach it.
        int left = cf;
        cf = 0;
        while (left > bf) {
            add_near(ring_f[--left & (kRing - 1)][tid]);
            flush(ring_n, cn, bn, true);
        }
        for (; left > 0; left -= 4) {
            const int4 q = l4[(size_t)(last - (left >> 2) + 1) * B.lstride];
            add_near(q.w);
            add_near(q.z);
            add_near(q.y);
            add_near(q.x);
            flush(ring_n, cn, bn, true);
        }
    }
    while (cn & 3) add_near(s);
    flush(ring_n, cn, bn, true);
}

template <int DIM, bool LST>
__global__ void __launch_bounds__(kPassThreads)
    k_shear(StateB B, const unsigned* __restrict__ keys, const int* __restrict__ start,
            const DevGrid* __restrict__ gp, DevParams P, int n) {
    __shared__ int s_list[cap_force<LST>()][kPassThreads];
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    const DevGrid g = *gp;
    shear_body<DIM, LST>(B, keys, start, g, P, s, s < n, s_list);
}

template <int DIM, int TPP, int BS, bool PER, bool LEAN, bool OPT = false, bool LST = false,
          bool FUS = false>
__global__ void
    // 64 registers for the lean physics; the others spill there: 80 (six CTAs of 128)
    // take the 3D channel from 4.82 to 4.41 ms, XSPH + normalised density 61 to 40 us
    __launch_bounds__(BS, (LEAN ? 1024 : 768) / BS)
    k_force(StateB B, StateA A, const unsigned* __restrict__ keys, const int* __restrict__ start,
            const DevGrid* __restrict__ gp, DevParams P, StepArgs S, unsigned* __restrict__ flags,
            int n, FusedSrc F) {
    __shared__ int s_list[cap_force<LST>()][BS];
    const int s = blockIdx.x * (BS / TPP) + (int)threadIdx.x / TPP;
    const DevGrid g = load_grid<PER>(gp);
    force_body<DIM, TPP, BS, LEAN, OPT, false, int, LST, FUS>(B, A, keys, start, g, P, S, flags, s,
                                                              s < n, s_list, StageView{}, F);
}

// ---------------------------------------------------------------------------
// Batched (multi-instance) pass kernels: persistent CTAs pull work items
// (one instance's slots [s0, s1), at most kPassThreads) from an atomic queue;
// the item's instance parameters, grid and step arguments are staged in shared
// memory for the CTA. Items are independent, so the order in which CTAs take
// them does not change any result.
// ---------------------------------------------------------------------------
struct ItemCtx {
    DevParams P;
    DevGrid g;
    StepArgs S;
    WorkItem w;
};

template <class T>
__device__ __forceinline__ void copy_to_shared(T* dst, const T* __restrict__ src) {
    static_assert(sizeof(T) % 4 == 0, "word copy");
    const int* a = reinterpret_cast<const int*>(src);
    int* b = reinterpret_cast<int*>(dst);
    for (int k = threadIdx.x; k < (int)(sizeof(T) / 4); k += blockDim.x) b[k] = __ldg(a + k);
}

// Takes the next item; false when the queue is empty. Ends with a barrier.
// Step arguments of iteration `its` of an instance (time_integration.f:131-218).
__device__ __forceinline__ StepArgs step_args_dev(const DevParams& P, int its) {
    StepArgs S;
    S.dt = P.dt;
    S.kdt = (its == 1) ? 0.5f * P.dt : P.dt;
    S.hdt = (its == 1) ? 0.f : 0.5f * P.dt;
    S.heat_on = P.heat_ext && ((double)its * (double)P.dt <= (double)P.heat_t_end);
    return S;
}

__device__ __forceinline__ bool next_item(ItemCtx& c, const WorkItem* __restrict__ items,
                                          int n_items, int* __restrict__ queue,
                                          const DevParams* __restrict__ params,
                                          const DevGrid* __restrict__ grids,
                                          const int* __restrict__ its) {
    __shared__ int s_it;
    __syncthreads();  // every thread is done with the previous item
    if (threadIdx.x == 0) s_it = atomicAdd(queue, 1);
    __syncthreads();
    const int it = s_it;
    if (it >= n_items) return false;
    if (threadIdx.x == 0) {
        c.w = items[it];
        if (its) c.S = step_args_dev(params[c.w.inst], *its);
    }
    __syncthreads();
    const int inst = c.w.inst;
    copy_to_shared(&c.P, params + inst);
    copy_to_shared(&c.g, grids + inst);
    __syncthreads();
    return true;
}

// LEAN: no instance uses physical viscosity, artificial heat, a wall model
// or a single_step option (the passes' lean variant).
template <int DIM, bool LEAN = false>
__global__ void __launch_bounds__(kPassThreads, 8)
    k_density_batch(StateB B, const unsigned* __restrict__ keys, const int* __restrict__ start,
                    const DevGrid* __restrict__ grids, const DevParams* __restrict__ params,
                    const WorkItem* __restrict__ items, int n_items, int* __restrict__ queue) {
    __shared__ int s_near[kListCapD][kPassThreads];
    __shared__ int s_far[kListCapD][kPassThreads];
    __shared__ ItemCtx c;
    while (next_item(c, items, n_items, queue, params, grids, nullptr)) {
        const int s = c.w.s0 + threadIdx.x;
        density_body<DIM, 1, kPassThreads, LEAN>(B, keys, start, c.g, c.P, s, s < c.w.s1, s_near,
                                                 s_far);
    }
}

template <int DIM>
__global__ void __launch_bounds__(kPassThreads)
    k_shear_batch(StateB B, const unsigned* __restrict__ keys, const int* __restrict__ start,
                  const DevGrid* __restrict__ grids, const DevParams* __restrict__ params,
                  const WorkItem* __restrict__ items, int n_items, int* __restrict__ queue) {
    __shared__ int s_list[kListCap][kPassThreads];
    __shared__ ItemCtx c;
    while (next_item(c, items, n_items, queue, params, grids, nullptr)) {
        const int s = c.w.s0 + threadIdx.x;
        if (c.P.visc) shear_body<DIM>(B, keys, start, c.g, c.P, s, s < c.w.s1, s_list);
    }
}

template <int DIM, bool LEAN = false>
__global__ void __launch_bounds__(kPassThreads, 8)
    k_force_batch(StateB B, StateA A, const unsigned* __restrict__ keys,
                  const int* __restrict__ start, const DevGrid* __restrict__ grids,
                  const DevParams* __restrict__ params, const int* __restrict__ its,
                  unsigned* __restrict__ flags, const WorkItem* __restrict__ items, int n_items,
                  int* __restrict__ queue) {
    __shared__ int s_list[kListCap][kPassThreads];
    __shared__ ItemCtx c;
    while (next_item(c, items, n_items, queue, params, grids, its)) {
        const int s = c.w.s0 + threadIdx.x;
        force_body<DIM, 1, kPassThreads, LEAN>(B, A, keys, start, c.g, c.P, c.S, flags, s,
                                               s < c.w.s1, s_list);
    }
}

// ---------------------------------------------------------------------------
// Neighbour lists (diagnostic entry point)
// ---------------------------------------------------------------------------
template <int DIM>
__global__ void k_count_nbrs(StateB B, const unsigned* __restrict__ keys,
                             const int* __restrict__ start, const DevGrid* __restrict__ gp,
                             int* __restrict__ cnt_by_id, int n) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    const DevGrid g = *gp;
    const float4 xi = B.xh[s];
    const CellCoord cc = decode_key<DIM>(keys[s], g);
    int c = 0;
    for_candidates<DIM>(g, start, cc, [&](int k) {
        if (k == s) return;
        float d[3], dr2;
        if (pair_delta<DIM>(xi, B.xh[k], g, d, dr2)) ++c;
    });
    cnt_by_id[B.id[s]] = c;
}

template <int DIM>
__global__ void k_fill_nbrs(StateB B, const unsigned* __restrict__ keys,
                            const int* __restrict__ start, const DevGrid* __restrict__ gp,
                            const long long* __restrict__ offs_by_id, int* __restrict__ nbr,
                            int n) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    const DevGrid g = *gp;
    const float4 xi = B.xh[s];
    const CellCoord cc = decode_key<DIM>(keys[s], g);
    long long o = offs_by_id[B.id[s]];
    for_candidates<DIM>(g, start, cc, [&](int k) {
        if (k == s) return;
        float d[3], dr2;
        if (pair_delta<DIM>(xi, B.xh[k], g, d, dr2)) nbr[o++] = B.id[k];
    });
}

}  // namespace ag
