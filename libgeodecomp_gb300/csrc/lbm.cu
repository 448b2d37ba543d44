// Batched ensemble of D3Q19 BGK lid-driven cavities.
//
// All instances live in one pair of allocations (A, B), each instance as
// structure of arrays: population i of cell (x, y, z) of an L^3 instance at
// base + i * P + (z * L + y) * L + x, with the population pitch P = L^3
// rounded up to 32 elements and every base a multiple of 32, so each
// population array starts on a 128-byte (FP32) boundary.  Warps walk the
// cells of a work item in 32-cell groups aligned to that boundary (lanes
// outside the item idle), so a warp's own-cell loads and stores are whole
// sectors.  Every time step is one launch for all instances, so that 32^3 and
// 192^3 cells share the GPU.  By default it has one thread per cell and one CTA
// per 128 cells (lbm_flat_kernel: 132 us for 5.5 M cells of 40^3 to 115^3 in
// FP32, 6.35 TB/s).  With a launch shape set by the caller, CTAs are persistent
// and their warps pull work items - TY rows of one z plane of one instance,
// largest instances first - from an atomic counter until the list is exhausted
// (188 us at the best shape).  Two steps (A -> B, B -> A) are captured once into
// a CUDA graph and replayed.  With temporal
// blocking (lbm_tb2_kernel) one persistent launch advances two steps, and
// two such launches (four steps) are captured and replayed the same way.
//
// Cell update (pull scheme, the reference LBM example's incompressible BGK
// collision, src/examples/latticeboltzmann/main.cpp:93-170): population i
// comes from x - e_i; outside the box it is bounced back from the cell
// itself, with 6 w_i (e_i . u_lid) added for populations coming from the
// lid (the wall beyond y = L-1).  Traffic: 19 reads + 19 writes per cell and
// step (152 B in FP32), the bounce-back reads hit L1.
//
// lgd_lbm_tune times the default, then searches the tile height TY, threads per
// CTA and CTAs per SM of the persistent kernel by pattern search, the method of
// the reference's PatternOptimizer (misc/patternoptimizer.h:13), and the
// two-step kernel.
#include <algorithm>
#include <functional>
#include <limits>
#include <mutex>
#include <queue>
#include <cstring>
#include <vector>

#include "lgd_internal.h"
#include "k_fp64.cuh"
#include "../../include/lgd_ensemble.h"

namespace lgd {

struct LbmInstance {
    long long base;     // element offset of the instance in A and B
    long long pitch;    // elements between populations: L^3 rounded up to 32
    int L;
    unsigned magic;     // ceil(2^32 / L), for row = c / L
    float omega_f;
    float lid_f;
    double omega;
    double lid;
};

struct FlatBlock;

struct Lbm {
    int count;
    int precision;
    long long total_cells;
    long long total_elems;
    void *buf[2];
    int cur;
    LbmInstance *d_inst;
    std::vector<LbmInstance> inst;
    int4 *d_items;      // (instance, z, y0, y1)
    int n_items;
    int *d_counter;     // one per captured step
    int ty, threads, ctas_per_sm;
    int sms;
    cudaStream_t stream;
    cudaGraphExec_t graph;
    bool graph_valid;
    // four steps of the depth-2 path (two two-step launches, 0 -> 1 -> 0)
    // replayed from a graph; rebuilt when the form, residency or columns change
    cudaGraphExec_t graph2;
    bool graph2_valid;
    int graph2_key[2];
    const int4 *graph2_cols;
    bool idx32;         // every instance indexable with 32 bits (19 L^3 < 2^31)
    int variant;        // 0: plain loads and stores; 1: read-only-path loads, evict-first stores
    uint64_t launches;
    // temporal blocking: depth 1 (one step per launch) or 2 (lbm_tb2_kernel),
    // column shape 0 (32 x 8) or 1 (32 x 4), resident CTAs per SM of the
    // depth-2 kernel; its work items are (instance, x0, y0) columns
    int depth;
    int tb_shape;
    int tb_ctas;
    int4 *d_cols;       // (instance, x0 | y0 << 16, z0, z1)
    int n_cols;
    int cols_shape;
    int cols_per_sm;    // resident CTAs they were cut for
    bool flat;          // single steps by lbm_flat_kernel (until a launch shape is set or found faster)
    FlatBlock *d_blocks;
    int n_blocks;
    long long stage_values;
    double *d_stage;    // conversion staging of uploads and downloads (FP32; from the first one on)
};

// D3Q19 directions in the reference's naming order: C, N, E, W, S, T, B,
// NW, SW, NE, SE, TW, BW, TE, BE, TN, BN, TS, BS (N = +y, E = +x, T = +z)
// (compile-time functions, so that unrolled loops fold them: a __constant__
// table is a runtime value, and e * u would cost a conversion and a
// multiplication per component)
__host__ __device__ constexpr int dir_ex(int i)
{
    return (i == 2 || i == 9 || i == 10 || i == 13 || i == 14) ? 1 : (i == 3 || i == 7 || i == 8 || i == 11 || i == 12) ? -1 : 0;
}
__host__ __device__ constexpr int dir_ey(int i)
{
    return (i == 1 || i == 7 || i == 9 || i == 15 || i == 16) ? 1 : (i == 4 || i == 8 || i == 10 || i == 17 || i == 18) ? -1 : 0;
}
__host__ __device__ constexpr int dir_ez(int i)
{
    return (i == 5 || i == 11 || i == 13 || i == 15 || i == 17) ? 1 : (i == 6 || i == 12 || i == 14 || i == 16 || i == 18) ? -1 : 0;
}

template<int I> struct Q;
#define LGD_Q(I, EX, EY, EZ, OPP) \
    template<> struct Q<I> { static const int ex = EX, ey = EY, ez = EZ, opp = OPP; };
LGD_Q(0, 0, 0, 0, 0)
LGD_Q(1, 0, 1, 0, 4)
LGD_Q(2, 1, 0, 0, 3)
LGD_Q(3, -1, 0, 0, 2)
LGD_Q(4, 0, -1, 0, 1)
LGD_Q(5, 0, 0, 1, 6)
LGD_Q(6, 0, 0, -1, 5)
LGD_Q(7, -1, 1, 0, 10)
LGD_Q(8, -1, -1, 0, 9)
LGD_Q(9, 1, 1, 0, 8)
LGD_Q(10, 1, -1, 0, 7)
LGD_Q(11, -1, 0, 1, 14)
LGD_Q(12, -1, 0, -1, 13)
LGD_Q(13, 1, 0, 1, 12)
LGD_Q(14, 1, 0, -1, 11)
LGD_Q(15, 0, 1, 1, 18)
LGD_Q(16, 0, 1, -1, 17)
LGD_Q(17, 0, -1, 1, 16)
LGD_Q(18, 0, -1, -1, 15)
#undef LGD_Q

template<int I>
struct DirCheck {
    static_assert(dir_ex(I) == Q<I>::ex && dir_ey(I) == Q<I>::ey && dir_ez(I) == Q<I>::ez, "direction tables agree");
    static_assert(Q<Q<I>::opp>::opp == I && Q<Q<I>::opp>::ex == -Q<I>::ex, "opposite directions");
    static const bool ok = DirCheck<I - 1>::ok;
};
template<>
struct DirCheck<-1> {
    static const bool ok = true;
};
static_assert(DirCheck<18>::ok, "D3Q19 tables");

template<typename R>
struct LbmArith;

template<>
struct LbmArith<double> {
    static __device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
    static __device__ __forceinline__ double sub(double a, double b) { return __dadd_rn(a, -b); }
    static __device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
};

template<>
struct LbmArith<float> {
    static __device__ __forceinline__ float add(float a, float b) { return a + b; }
    static __device__ __forceinline__ float sub(float a, float b) { return a - b; }
    static __device__ __forceinline__ float mul(float a, float b) { return a * b; }
};

// Memory paths of the update: NC = 0 (default) plain loads and stores;
// NC = 1 reads through the non-coherent (read-only) path, which allocates
// in L1, and writes with evict-first stores.  NC = 1 measured 4% slower on
// the 512-cavity ensemble (28.2 against 29.6 GLUPS) and is kept for
// comparison.
template<int NC>
struct Mem {
    template<typename R>
    static __device__ __forceinline__ R ld(const R *p) { return NC ? __ldg(p) : *p; }
    template<typename R>
    static __device__ __forceinline__ void st(R *p, R v)
    {
        if (NC) {
            __stcs(p, v);
        } else {
            *p = v;
        }
    }
};

// FP32 rounds the same in every kernel: the products whose bits an FMA keeps
// are written out here and below (as the compiler had chosen them for separate
// directions), not left to what else a kernel does with them.
// Population I back from the lid: + 6 w_i (e_i . u_lid), u_lid = (lid, 0, 0).
template<typename R, int I>
__device__ __forceinline__ R from_lid(R v, R lid)
{
    const R w6 = LbmArith<R>::mul((R)6.0, I < 7 ? (R)(1.0 / 18.0) : (R)(1.0 / 36.0));
    if constexpr (sizeof(R) == 4) return fmaf(w6, (R)Q<I>::ex * lid, v);
    else return LbmArith<R>::add(v, LbmArith<R>::mul(w6, (R)Q<I>::ex * lid));
}

// INTERIOR: the cell is at least one cell away from every wall, so every
// source cell exists (no wall tests)
template<typename R, int I, typename IDX, int NC, bool INTERIOR>
__device__ __forceinline__ void pull_one(const R *__restrict__ src, IDX n3, IDX cell, int L, int x, int y,
                                         int z, R lid, R *f)
{
    const int sx = x - Q<I>::ex;
    const int sy = y - Q<I>::ey;
    const int sz = z - Q<I>::ez;
    if (INTERIOR ||
        ((unsigned)sx < (unsigned)L && (unsigned)sy < (unsigned)L && (unsigned)sz < (unsigned)L)) {
        f[I] = Mem<NC>::ld(src + (I * n3 + cell - (Q<I>::ex + (IDX)Q<I>::ey * L + (IDX)Q<I>::ez * L * L)));
    } else {
        const R v = Mem<NC>::ld(src + (Q<I>::opp * n3 + cell));
        // for every wall but the lid the added term is exactly zero
        f[I] = Q<I>::ey == -1 && Q<I>::ex != 0 && y == L - 1 ? from_lid<R, I>(v, lid) : v;
    }
}

template<typename R, int I, typename IDX, int NC, bool INTERIOR>
struct PullAll {
    static __device__ __forceinline__ void run(const R *src, IDX n3, IDX cell, int L, int x, int y, int z, R lid, R *f)
    {
        pull_one<R, I, IDX, NC, INTERIOR>(src, n3, cell, L, x, y, z, lid, f);
        PullAll<R, I + 1, IDX, NC, INTERIOR>::run(src, n3, cell, L, x, y, z, lid, f);
    }
};

template<typename R, typename IDX, int NC, bool INTERIOR>
struct PullAll<R, 19, IDX, NC, INTERIOR> {
    static __device__ __forceinline__ void run(const R *, IDX, IDX, int, int, int, int, R, R *) {}
};

// e . u for one of a pair of opposite directions, components added in the
// oracle's order (x, y, z).  Its zero components drop out: adding 0 * u does
// not change a sum but for the sign of a zero, which d + eu and eu * eu below
// do not see, and for an infinite u, which collide_with looks for.
template<typename R, int I>
__device__ __forceinline__ R dot_dir(R ux, R uy, R uz)
{
    typedef LbmArith<R> A;
    const R x = Q<I>::ex == 1 ? ux : -ux, y = Q<I>::ey == 1 ? uy : -uy, z = Q<I>::ez == 1 ? uz : -uz;
    if (Q<I>::ex == 0 && Q<I>::ey == 0) return z;
    if (Q<I>::ex == 0) return Q<I>::ez == 0 ? y : A::add(y, z);
    if (Q<I>::ey == 0) return Q<I>::ez == 0 ? x : A::add(x, z);
    return A::add(x, y);
}

// keep f + w x.  FP32: the FMA keeps the bits of keep f (the error of 20 steps
// against FP64 is 2 to 3% smaller than with those of w x, rms over cavities of 9^3
// to 33^3)
template<typename R, typename MUL>
__device__ __forceinline__ R relax(R keep, R f, R w, R x, MUL mul)
{
    if constexpr (sizeof(R) == 4) return fmaf(keep, f, __fmul_rn(w, x));
    else return LbmArith<R>::add(mul(keep, f), mul(w, x));
}

// directions I and its opposite: e . u is the exact negative and its square
// the same, so both are taken once (D3Q19: 9 pairs; the collision was a third
// longer with 18 separate directions)
template<typename R, int I, typename PUT, typename MUL>
__device__ __forceinline__ void collide_pair(const R *f, R keep, R w1, R w2, R d, R ux, R uy, R uz, PUT put, MUL mul)
{
    typedef LbmArith<R> A;
    const R wi = (I < 7) ? w1 : w2;
    const R eu = dot_dir<R, I>(ux, uy, uz);
    R there, back;
    if constexpr (sizeof(R) == 4) {
        const R e2 = __fmul_rn(eu, eu);
        there = fmaf(1.5f, e2, d + eu);
        back = fmaf(1.5f, e2, d - eu);
    } else {
        const R sq = mul((R)1.5, mul(eu, eu));
        there = A::add(A::add(d, eu), sq);
        back = A::add(A::sub(d, eu), sq);
    }
    put(I, relax(keep, f[I], wi, there, mul));
    put(Q<I>::opp, relax(keep, f[Q<I>::opp], wi, back, mul));
}

// not a number or infinite, without the FP64 pipe
__device__ __forceinline__ bool non_finite(float v) { return (__float_as_uint(v) & 0x7f800000u) == 0x7f800000u; }
__device__ __forceinline__ bool non_finite(double v) { return ((unsigned)__double2hiint(v) & 0x7ff00000u) == 0x7ff00000u; }

// BGK collision, operation order of the oracle's lgd_d3q19_collide; put(i,
// v) stores post-collision population i, mul multiplies.  CHECK: velocities may
// be infinite; 0 * u then makes every direction's e . u a NaN (without it mul
// has to report them).
template<typename R, bool CHECK, typename PUT, typename MUL>
__device__ __forceinline__ void collide_with(const R *f, R omega, PUT put, MUL mul)
{
    typedef LbmArith<R> A;
    R rho = f[0];
#pragma unroll
    for (int i = 1; i < 19; ++i) rho = A::add(rho, f[i]);
    // E + NE + SE + TE + BE - (W + NW + SW + TW + BW)
    const R ux = A::sub(A::add(A::add(A::add(A::add(f[2], f[9]), f[10]), f[13]), f[14]),
                        A::add(A::add(A::add(A::add(f[3], f[7]), f[8]), f[11]), f[12]));
    // N + NW + NE + TN + BN - (S + SW + SE + TS + BS)
    const R uy = A::sub(A::add(A::add(A::add(A::add(f[1], f[7]), f[9]), f[15]), f[16]),
                        A::add(A::add(A::add(A::add(f[4], f[8]), f[10]), f[17]), f[18]));
    // T + TW + TE + TN + TS - (B + BW + BE + BN + BS)
    const R uz = A::sub(A::add(A::add(A::add(A::add(f[5], f[11]), f[13]), f[15]), f[17]),
                        A::add(A::add(A::add(A::add(f[6], f[12]), f[14]), f[16]), f[18]));
    R d;
    if constexpr (sizeof(R) == 4) {
        const R usq = fmaf(uz, uz, fmaf(ux, ux, __fmul_rn(uy, uy)));
        d = fmaf(rho, (R)(1.0 / 3.0), -0.5f * usq);
    } else {
        const R usq = A::add(A::add(mul(ux, ux), mul(uy, uy)), mul(uz, uz));
        d = A::sub(mul(rho, (R)(1.0 / 3.0)), mul((R)0.5, usq));
    }
    const R keep = A::sub((R)1.0, omega);
    const R w1 = mul(omega, (R)(1.0 / 6.0));
    const R w2 = mul(omega, (R)(1.0 / 12.0));
    put(0, relax(keep, f[0], omega, d, mul));
    if (CHECK && (non_finite(ux) || non_finite(uy) || non_finite(uz))) d = (R)__int_as_float(0x7fffffff);
    collide_pair<R, 1>(f, keep, w1, w2, d, ux, uy, uz, put, mul);
    collide_pair<R, 2>(f, keep, w1, w2, d, ux, uy, uz, put, mul);
    collide_pair<R, 5>(f, keep, w1, w2, d, ux, uy, uz, put, mul);
    collide_pair<R, 7>(f, keep, w1, w2, d, ux, uy, uz, put, mul);
    collide_pair<R, 8>(f, keep, w1, w2, d, ux, uy, uz, put, mul);
    collide_pair<R, 11>(f, keep, w1, w2, d, ux, uy, uz, put, mul);
    collide_pair<R, 12>(f, keep, w1, w2, d, ux, uy, uz, put, mul);
    collide_pair<R, 15>(f, keep, w1, w2, d, ux, uy, uz, put, mul);
    collide_pair<R, 16>(f, keep, w1, w2, d, ux, uy, uz, put, mul);
}

template<typename R, typename PUT>
__device__ __forceinline__ void collide_to(const R *f, R omega, PUT put)
{
    collide_with<R, true>(f, omega, put, [](R a, R b) { return LbmArith<R>::mul(a, b); });
}

template<typename R, typename IDX, int NC>
__device__ __forceinline__ void collide_store(const R *f, R omega, R *__restrict__ dst, IDX n3, IDX cell)
{
    collide_to<R>(f, omega, [&](int i, R v) { Mem<NC>::st(dst + ((IDX)i * n3 + cell), v); });
}

// Cells of rows [y0, y1) of plane z (contiguous in memory), the threads
// first, first + stride, ... of the group taking cells in that order,
// starting at the 32-cell boundary at or before the first cell (stride a
// multiple of 32).  IDX is the index type inside one instance: 32-bit when
// 19 P < 2^31.
template<typename R, typename IDX, int NC>
__device__ __forceinline__ void lbm_item(const LbmInstance& in, const R *__restrict__ A, R *__restrict__ B, int z, int y0,
                                         int y1, unsigned first, unsigned stride)
{
    const int L = in.L;
    // the population pitch (LbmInstance::pitch), recomputed from L: a
    // loaded pitch makes the compiler keep the 38 addresses live (128
    // registers instead of 56)
    const IDX n3 = ((IDX)L * L * L + 31) & ~(IDX)31;
    const R *src = A + in.base;
    R *dst = B + in.base;
    const R omega = (sizeof(R) == 8) ? (R)in.omega : (R)in.omega_f;
    const R lid = (sizeof(R) == 8) ? (R)in.lid : (R)in.lid_f;
    // plane-relative cell indices [cb, ce); the walk starts at the 32-cell
    // boundary at or before cb (a negative start stays in the plane before)
    const int cb = y0 * L;
    const int ce = y1 * L;
    const int lead = (int)((((IDX)z * L * L) + cb) & 31);
    int k0 = cb - lead + (int)first;
    if (k0 < cb) k0 += (int)stride;                     // lanes before the item start one round later
    for (int k = k0; k < ce; k += (int)stride) {
        const unsigned c = (unsigned)k;                 // index inside the plane
        unsigned r = __umulhi(c, in.magic);
        if (r * (unsigned)L > c) --r;
        const int y = (int)r;
        const int x = (int)(c - r * (unsigned)L);
        // the cell index rebuilt from (x, y, z), not the loop counter: the
        // 38 addresses are then recomputed per cell instead of being kept
        // as induction variables (56 registers instead of 128)
        const IDX cell = ((IDX)z * L + y) * L + x;
        R f[19];
        if ((unsigned)(x - 1) < (unsigned)(L - 2) && (unsigned)(y - 1) < (unsigned)(L - 2) &&
            (unsigned)(z - 1) < (unsigned)(L - 2)) {
            PullAll<R, 0, IDX, NC, true>::run(src, n3, cell, L, x, y, z, lid, f);
        } else {
            PullAll<R, 0, IDX, NC, false>::run(src, n3, cell, L, x, y, z, lid, f);
        }
        collide_store<R, IDX, NC>(f, omega, dst, n3, cell);
    }
}

// Every warp pulls its own work items from the counter - no CTA barrier, so
// a warp that finishes a short item starts the next at once - and claims
// the next item before it processes the current one, which hides the
// atomic's round trip.
template<typename R, typename IDX, int NC>
__global__ void lbm_persistent_kernel(const LbmInstance *__restrict__ inst, const int4 *__restrict__ items, int n_items,
                                      int *counter, const R *__restrict__ A, R *__restrict__ B)
{
    const unsigned lane = threadIdx.x & 31u;
    int it = 0;
    if (lane == 0) it = atomicAdd(counter, 1);
    it = __shfl_sync(0xffffffffu, it, 0);
    while (it < n_items) {
        int next = 0;
        if (lane == 0) next = atomicAdd(counter, 1);
        const int4 w = items[it];
        lbm_item<R, IDX, NC>(inst[w.x], A, B, w.y, w.z, w.w, lane, 32u);
        it = __shfl_sync(0xffffffffu, next, 0);
    }
}

// ------------------------------------------- one thread per cell and step
// A CTA takes FLAT consecutive cells of one instance, found in a table (an
// entry holds all it needs: one load), and is gone: the next CTA's 19 loads per
// cell overlap with this one's stores.  Warps that walk work items wait for a
// cell's loads, collide, store, and only then load again; with 38 streams that
// left DRAM at 5.0 of 6.8 TB/s whatever the registers, warps and item shapes.
constexpr int FLAT = 128;
// how a launch shape says it: more CTAs of 128 threads than an SM holds, which a
// persistent shape is clamped to and never reports
constexpr int FLAT_ROWS = 1, FLAT_CTAS = 32;

struct FlatBlock {
    long long base;
    int L;
    unsigned magic;
    double omega, lid;
    int first;          // cell
    int pad[3];
};

// population I of a cell of which some may lie at a wall: one load, its address
// selected, so that a warp's inner and wall cells stay together
template<typename R, int I, typename IDX, int NC>
__device__ __forceinline__ void pull_select(const R *src, IDX n3, IDX cell, int L, int x, int y, int z, R lid, R *f)
{
    if constexpr (I < 19) {
        const bool inside = (unsigned)(x - Q<I>::ex) < (unsigned)L && (unsigned)(y - Q<I>::ey) < (unsigned)L &&
                            (unsigned)(z - Q<I>::ez) < (unsigned)L;
        const IDX at = inside ? I * n3 + cell - (Q<I>::ex + (IDX)Q<I>::ey * L + (IDX)Q<I>::ez * L * L) : Q<I>::opp * n3 + cell;
        R v = Mem<NC>::ld(src + at);
        if (Q<I>::ey == -1 && Q<I>::ex != 0) {              // see pull_one
            const R lid_v = from_lid<R, I>(v, lid);
            v = !inside && y == L - 1 ? lid_v : v;
        }
        f[I] = v;
        pull_select<R, I + 1, IDX, NC>(src, n3, cell, L, x, y, z, lid, f);
    }
}

// one cell with FP64 multiplications (a call: predicated, they would be paid always)
template<typename IDX, int NC>
__device__ __noinline__ void plain_cell(const double *src, double *dst, IDX n3, IDX cell, int L, int x, int y, int z, double lid,
                                        double omega)
{
    double f[19];
    pull_select<double, 0, IDX, NC>(src, n3, cell, L, x, y, z, lid, f);
    collide_store<double, IDX, NC>(f, omega, dst, n3, cell);
}

template<typename R, typename IDX, int NC>
__global__ void __launch_bounds__(FLAT, sizeof(R) == 4 ? 8 : 5)
lbm_flat_kernel(const FlatBlock *__restrict__ blocks, const R *A, R *B)
{
    dependent_start();
    const FlatBlock in = blocks[blockIdx.x];
    const unsigned L = (unsigned)in.L;
    const unsigned c = (unsigned)in.first + threadIdx.x;
    unsigned row = __umulhi(c, in.magic);                   // c below 2^30: at most one too many
    if (row * L > c) --row;
    unsigned plane = __umulhi(row, in.magic);
    if (plane * L > row) --plane;
    const int x = (int)(c - row * L), y = (int)(row - plane * L), z = (int)plane;
    const IDX n3 = ((IDX)L * L * L + 31) & ~(IDX)31;
    const bool live = plane < L;
    const bool inner = (unsigned)(x - 1) < L - 2 && (unsigned)(y - 1) < L - 2 && (unsigned)(z - 1) < L - 2;
    const R *src = A + in.base;
    R f[19];
    if (__all_sync(0xffffffffu, inner)) {
        PullAll<R, 0, IDX, NC, true>::run(src, n3, (IDX)c, (int)L, x, y, z, (R)in.lid, f);
    } else {
        if (!live) return;
        pull_select<R, 0, IDX, NC>(src, n3, (IDX)c, (int)L, x, y, z, (R)in.lid, f);
    }
    R *dst = B + in.base;
    if constexpr (sizeof(R) == 8) {
        // FP64 is bound by the FP64 pipe: the collision's multiplications run on the
        // integer pipes, bit for bit (4 cavities of 32^3 to 96^3: 408 -> 287 us per step)
        bool ok = true;                 // mul_integer(u, u, ok) reports an infinite u
        collide_with<R, false>(
            f, (R)in.omega, [&](int i, R v) { Mem<NC>::st(dst + ((IDX)i * n3 + (IDX)c), v); },
            [&](R a, R b) { return mul_integer(a, b, ok); });
        if (!ok) plain_cell<IDX, NC>(src, dst, n3, (IDX)c, (int)L, x, y, z, (R)in.lid, (R)in.omega);
    } else {
        collide_store<R, IDX, NC>(f, (R)in.omega, dst, n3, (IDX)c);
    }
}

// one instance, one launch: the looped single-grid comparison
template<typename R, typename IDX, int NC>
__global__ void lbm_single_kernel(const LbmInstance *__restrict__ inst, int j, const R *__restrict__ A, R *__restrict__ B)
{
    const LbmInstance in = inst[j];
    const int z = blockIdx.y;
    const int rows_per_block = max(1, (int)(blockDim.x / in.L));
    const int y0 = blockIdx.x * rows_per_block;
    if (y0 >= in.L) return;
    lbm_item<R, IDX, NC>(in, A, B, z, y0, min(in.L, y0 + rows_per_block), threadIdx.x, blockDim.x);
}

// ------------------------------------------------ two steps per launch
// Temporal blocking of depth 2.  A work item is a column of one instance:
// TX x TY cells of the z planes of its chunk.  The CTA marches z; at each plane it
// first computes step 1 for the tile plus a one-cell rim (the cells whose
// populations step 2 pulls), pulling from the input grid and keeping the 19
// post-collision populations in a ring of three planes in shared memory,
// then step 2 for the tile at the plane below, pulling from the ring and
// writing the output grid.  Walls bounce back from the cell itself at
// either level, exactly as the single step does, so the result is the two
// single steps' bit for bit; HBM traffic per two steps is one read of the
// input (plus the rim's, about a third more, partly from L2) and one write.
template<int TX, int TY>
struct Tb2Geo {
    static constexpr int THREADS = TX * TY;
    static constexpr int HX = TX + 2;
    static constexpr int HY = TY + 2;
    static constexpr int HC = HX * HY;          // step-1 cells of one plane
    template<typename R>
    static constexpr size_t smem() { return (size_t)3 * 19 * HC * sizeof(R); }
};

// step-2 population I of tile cell (tx, ty) at plane zz from the ring
template<typename R, int I, int TX, int TY>
__device__ __forceinline__ R tb2_pull(const R *__restrict__ ring, int L, int x, int y, int zz, int tx, int ty, R lid)
{
    typedef Tb2Geo<TX, TY> G;
    const int sx = x - Q<I>::ex;
    const int sy = y - Q<I>::ey;
    const int sz = zz - Q<I>::ez;
    if ((unsigned)sx < (unsigned)L && (unsigned)sy < (unsigned)L && (unsigned)sz < (unsigned)L) {
        return ring[((sz % 3) * 19 + I) * G::HC + (ty + 1 - Q<I>::ey) * G::HX + (tx + 1 - Q<I>::ex)];
    }
    const R v = ring[((zz % 3) * 19 + Q<I>::opp) * G::HC + (ty + 1) * G::HX + (tx + 1)];
    return Q<I>::ey == -1 && Q<I>::ex != 0 && y == L - 1 ? from_lid<R, I>(v, lid) : v;
}

template<typename R, int I, int TX, int TY>
struct Tb2PullAll {
    static __device__ __forceinline__ void run(const R *ring, int L, int x, int y, int zz, int tx, int ty, R lid, R *f)
    {
        f[I] = tb2_pull<R, I, TX, TY>(ring, L, x, y, zz, tx, ty, lid);
        Tb2PullAll<R, I + 1, TX, TY>::run(ring, L, x, y, zz, tx, ty, lid, f);
    }
};

template<typename R, int TX, int TY>
struct Tb2PullAll<R, 19, TX, TY> {
    static __device__ __forceinline__ void run(const R *, int, int, int, int, int, int, R, R *) {}
};

template<typename R, typename IDX, int TX, int TY>
__global__ void __launch_bounds__(TX * TY)
lbm_tb2_kernel(const LbmInstance *__restrict__ inst, const int4 *__restrict__ items, int n_items, int *counter,
               const R *__restrict__ A, R *__restrict__ B)
{
    typedef Tb2Geo<TX, TY> G;
    extern __shared__ __align__(16) unsigned char tb2_smem[];
    R *ring = reinterpret_cast<R *>(tb2_smem);
    __shared__ int s_item;
    const int tid = threadIdx.x;
    for (;;) {
        if (tid == 0) s_item = atomicAdd(counter, 1);
        __syncthreads();
        const int it = s_item;
        if (it >= n_items) break;
        const int4 w = items[it];
        const LbmInstance in = inst[w.x];
        const int L = in.L;
        const int x0 = w.y & 0xffff;
        const int y0 = w.y >> 16;
        const int z0 = w.z;             // step 2 computes planes z0 .. z1 - 1, step 1 one more on either side
        const int z1 = w.w;
        const IDX n3 = ((IDX)L * L * L + 31) & ~(IDX)31;
        const R *src = A + in.base;
        R *dst = B + in.base;
        const R omega = (sizeof(R) == 8) ? (R)in.omega : (R)in.omega_f;
        const R lid = (sizeof(R) == 8) ? (R)in.lid : (R)in.lid_f;
        for (int z = max(z0 - 1, 0); z <= z1; ++z) {
            if (z < L) {
                // step 1 at plane z: the tile and its rim, inside the instance
                R *plane = ring + (z % 3) * 19 * G::HC;
                for (int c = tid; c < G::HC; c += G::THREADS) {
                    const int x = x0 - 1 + c % G::HX;
                    const int y = y0 - 1 + c / G::HX;
                    if ((unsigned)x < (unsigned)L && (unsigned)y < (unsigned)L) {
                        const IDX cell = ((IDX)z * L + y) * L + x;
                        R f[19];
                        if ((unsigned)(x - 1) < (unsigned)(L - 2) && (unsigned)(y - 1) < (unsigned)(L - 2) &&
                            (unsigned)(z - 1) < (unsigned)(L - 2)) {
                            PullAll<R, 0, IDX, 0, true>::run(src, n3, cell, L, x, y, z, lid, f);
                        } else {
                            PullAll<R, 0, IDX, 0, false>::run(src, n3, cell, L, x, y, z, lid, f);
                        }
                        collide_to<R>(f, omega, [&](int i, R v) { plane[i * G::HC + c] = v; });
                    }
                }
            }
            __syncthreads();
            if (z > z0) {
                // step 2 at plane z - 1: the tile, from the ring
                const int zz = z - 1;
                const int tx = tid % TX;
                const int ty = tid / TX;
                const int x = x0 + tx;
                const int y = y0 + ty;
                if (x < L && y < L) {
                    R f[19];
                    Tb2PullAll<R, 0, TX, TY>::run(ring, L, x, y, zz, tx, ty, lid, f);
                    const IDX cell = ((IDX)zz * L + y) * L + x;
                    collide_store<R, IDX, 0>(f, omega, dst, n3, cell);
                }
            }
            __syncthreads();        // the slot of plane z - 2 is written at z + 1
        }
    }
}

template<typename R>
__global__ void lbm_rest_kernel(const LbmInstance *__restrict__ inst, int count, R *A)
{
    const int j = blockIdx.y;
    if (j >= count) return;
    const LbmInstance in = inst[j];
    const long long n3 = (long long)in.L * in.L * in.L;
    const long long P = in.pitch;
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < n3; c += (long long)gridDim.x * blockDim.x) {
        A[in.base + c] = (R)(1.0 / 3.0);
        for (int i = 1; i < 7; ++i) A[in.base + i * P + c] = (R)(1.0 / 18.0);
        for (int i = 7; i < 19; ++i) A[in.base + i * P + c] = (R)(1.0 / 36.0);
    }
}

// FP32 populations of one instance <-> dense doubles, values first .. first + n
template<bool TO_HOST>
__global__ void __launch_bounds__(256)
convert_kernel(float *f, double *dense, unsigned n3, long long pitch, long long first, long long n)
{
    for (long long k = blockIdx.x * 256ll + threadIdx.x; k < n; k += gridDim.x * 256ll) {
        const long long i = (first + k) / n3;
        float *p = f + i * pitch + (first + k - i * n3);
        if (TO_HOST) dense[k] = *p;
        else *p = (float)dense[k];
    }
}

// Host copy of one instance as 19 * L^3 doubles.  FP32 populations convert on
// the device in bounded chunks (on one host core the conversion took 0.5 ns a
// value, ten times the copy), small instances on the host, where that is less than
// the launch (us by host / device: up 8^3 14.6 / 22.9, 12^3 18.9 / 24.3, 16^3 28.9 / 25.9;
// down 8^3 16.2 / 18.4, 12^3 21.1 / 19.7).
constexpr long long CONVERT_CHUNK = 8ll << 20;
constexpr long long HOST_UP_VALUES = 56 << 10, HOST_DOWN_VALUES = 16 << 10;

static void copy_instance(Lbm& e, const LbmInstance& in, size_t n3, double *host, bool up)
{
    if (e.precision == 8) {
        double *d = (double *)e.buf[e.cur] + in.base;
        if (up) {
            LGD_CHECK_CUDA(cudaMemcpy2DAsync(d, (size_t)in.pitch * 8, host, n3 * 8, n3 * 8, 19, cudaMemcpyHostToDevice,
                                             e.stream));
        } else {
            LGD_CHECK_CUDA(cudaMemcpy2DAsync(host, n3 * 8, d, (size_t)in.pitch * 8, n3 * 8, 19, cudaMemcpyDeviceToHost,
                                             e.stream));
        }
        LGD_CHECK_CUDA(cudaStreamSynchronize(e.stream));
        return;
    }
    float *f = (float *)e.buf[e.cur] + in.base;
    const long long total = 19ll * (long long)n3;
    if (total <= (up ? HOST_UP_VALUES : HOST_DOWN_VALUES)) {
        if (up) {
            const std::vector<float> values(host, host + total);
            LGD_CHECK_CUDA(cudaMemcpy2DAsync(f, (size_t)in.pitch * 4, values.data(), n3 * 4, n3 * 4, 19, cudaMemcpyHostToDevice,
                                             e.stream));
            LGD_CHECK_CUDA(cudaStreamSynchronize(e.stream));
        } else {
            std::vector<float> values(total);
            LGD_CHECK_CUDA(cudaMemcpy2DAsync(values.data(), n3 * 4, f, (size_t)in.pitch * 4, n3 * 4, 19, cudaMemcpyDeviceToHost,
                                             e.stream));
            LGD_CHECK_CUDA(cudaStreamSynchronize(e.stream));
            std::copy(values.begin(), values.end(), host);
        }
        return;
    }
    if (e.d_stage == nullptr) {
        // shorter chunks where the populations leave little room
        e.stage_values = CONVERT_CHUNK;
        while (malloc_on_first_use((void **)&e.d_stage, e.stage_values * sizeof(double)) != cudaSuccess) {
            e.stage_values /= 16;
            LGD_REQUIRE(e.stage_values >= 1024, LGD_ERR_CUDA, "no device memory for the conversion buffer");
        }
    }
    for (long long first = 0; first < total; first += e.stage_values) {
        const long long n = std::min(e.stage_values, total - first);
        const unsigned blocks = (unsigned)std::min<long long>(152 * 16, (n + 255) / 256);
        if (up) {
            LGD_CHECK_CUDA(cudaMemcpyAsync(e.d_stage, host + first, n * 8, cudaMemcpyHostToDevice, e.stream));
            convert_kernel<false><<<blocks, 256, 0, e.stream>>>(f, e.d_stage, (unsigned)n3, in.pitch, first, n);
        } else {
            convert_kernel<true><<<blocks, 256, 0, e.stream>>>(f, e.d_stage, (unsigned)n3, in.pitch, first, n);
            LGD_CHECK_CUDA(cudaMemcpyAsync(host + first, e.d_stage, n * 8, cudaMemcpyDeviceToHost, e.stream));
        }
        check_launch("lbm conversion");
        ++e.launches;
    }
    LGD_CHECK_CUDA(cudaStreamSynchronize(e.stream));
}

static Lbm& lbm_of(lgd_lbm *h)
{
    LGD_REQUIRE(h != nullptr, LGD_ERR_INVALID, "null handle");
    return *reinterpret_cast<Lbm *>(h);
}

static void build_items(Lbm& e)
{
    // items of the largest instances first, so the tail of a step is made
    // of small items
    std::vector<int> order(e.count);
    for (int j = 0; j < e.count; ++j) order[j] = j;
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return e.inst[a].L > e.inst[b].L; });
    std::vector<int4> items;
    for (int j : order) {
        const int L = e.inst[j].L;
        for (int z = 0; z < L; ++z) {
            for (int y0 = 0; y0 < L; y0 += e.ty) {
                items.push_back(make_int4(j, z, y0, std::min(L, y0 + e.ty)));
            }
        }
    }
    if (e.d_items) cudaFree(e.d_items);
    e.d_items = nullptr;
    LGD_CHECK_CUDA(cudaMalloc(&e.d_items, sizeof(int4) * items.size()));
    LGD_CHECK_CUDA(cudaMemcpyAsync(e.d_items, items.data(), sizeof(int4) * items.size(), cudaMemcpyHostToDevice, e.stream));
    LGD_CHECK_CUDA(cudaStreamSynchronize(e.stream));
    e.n_items = (int)items.size();
}

// the flat kernel's table, by instance in blockIdx.y: entries first[j] and on
__global__ void __launch_bounds__(256)
flat_blocks_kernel(const LbmInstance *inst, const int *first, int precision, FlatBlock *blocks)
{
    const LbmInstance in = inst[blockIdx.y];
    FlatBlock *out = blocks + first[blockIdx.y];
    const long long n3 = (long long)in.L * in.L * in.L;
    for (long long k = blockIdx.x * 256ll + threadIdx.x; k * FLAT < n3; k += gridDim.x * 256ll) {
        FlatBlock b = {in.base, in.L, in.magic, in.omega, in.lid, (int)(k * FLAT), {}};
        if (precision == 4) {
            b.omega = in.omega_f;
            b.lid = in.lid_f;
        }
        out[k] = b;
    }
}

// (on one host core the table of 64 cavities of 64^3, and its copy, took 1.3 ms; 0.2)
static void build_blocks(Lbm& e)
{
    std::vector<int> first(e.count);
    long long n = 0;
    for (int j = 0; j < e.count; ++j) {
        first[j] = (int)n;
        n += ((long long)e.inst[j].L * e.inst[j].L * e.inst[j].L + FLAT - 1) / FLAT;
        LGD_REQUIRE(n < (1ll << 31), LGD_ERR_RANGE, "ensemble too large");
    }
    int *d_first = nullptr;
    const size_t bytes = sizeof(FlatBlock) * (size_t)n, index = sizeof(int) * (size_t)e.count;
    if (cudaMalloc(&e.d_blocks, bytes) != cudaSuccess || cudaMalloc(&d_first, index) != cudaSuccess) {
        (void)cudaGetLastError();       // populations that leave no room: the persistent kernel
        cudaFree(e.d_blocks);
        e.d_blocks = nullptr;
        return;
    }
    cudaError_t error = cudaMemcpyAsync(d_first, first.data(), index, cudaMemcpyHostToDevice, e.stream);
    if (error == cudaSuccess) {
        flat_blocks_kernel<<<dim3(64, e.count), 256, 0, e.stream>>>(e.d_inst, d_first, e.precision, e.d_blocks);
        error = cudaGetLastError();
    }
    if (error == cudaSuccess) error = cudaStreamSynchronize(e.stream);
    cudaFree(d_first);
    LGD_CHECK_CUDA(error);
    ++e.launches;
    e.n_blocks = (int)n;
}

// the persistent kernel for the ensemble's precision and index width
template<int NC>
static const void *persistent_fn_nc(const Lbm& e)
{
    if (e.precision == 4) {
        return e.idx32 ? (const void *)lbm_persistent_kernel<float, int, NC>
                       : (const void *)lbm_persistent_kernel<float, long long, NC>;
    }
    return e.idx32 ? (const void *)lbm_persistent_kernel<double, int, NC>
                   : (const void *)lbm_persistent_kernel<double, long long, NC>;
}

static const void *persistent_fn(const Lbm& e)
{
    return e.variant == 1 ? persistent_fn_nc<1>(e) : persistent_fn_nc<0>(e);
}

template<int NC>
static void launch_single_nc(Lbm& e, int j, dim3 grid)
{
    const void *a = e.buf[e.cur];
    void *b = e.buf[1 - e.cur];
    if (e.precision == 4) {
        if (e.idx32) {
            lbm_single_kernel<float, int, NC><<<grid, 256, 0, e.stream>>>(e.d_inst, j, (const float *)a, (float *)b);
        } else {
            lbm_single_kernel<float, long long, NC><<<grid, 256, 0, e.stream>>>(e.d_inst, j, (const float *)a, (float *)b);
        }
    } else {
        if (e.idx32) {
            lbm_single_kernel<double, int, NC><<<grid, 256, 0, e.stream>>>(e.d_inst, j, (const double *)a, (double *)b);
        } else {
            lbm_single_kernel<double, long long, NC><<<grid, 256, 0, e.stream>>>(e.d_inst, j, (const double *)a,
                                                                                  (double *)b);
        }
    }
}

template<typename R, typename IDX>
static void launch_flat_as(Lbm& e, int src)
{
    const R *a = (const R *)e.buf[src];
    R *b = (R *)e.buf[1 - src];
    if (e.variant == 1) {       // reads through the read-only path: not while the step before still writes
        lbm_flat_kernel<R, IDX, 1><<<e.n_blocks, FLAT, 0, e.stream>>>(e.d_blocks, a, b);
    } else {
        launch_dependent(lbm_flat_kernel<R, IDX, 0>, dim3(e.n_blocks), FLAT, 0, e.stream, (const FlatBlock *)e.d_blocks, a, b);
    }
}

static void launch_step(Lbm& e, int which_counter, int src)
{
    if (e.flat) {
        if (e.precision == 4) {
            if (e.idx32) launch_flat_as<float, int>(e, src); else launch_flat_as<float, long long>(e, src);
        } else {
            if (e.idx32) launch_flat_as<double, int>(e, src); else launch_flat_as<double, long long>(e, src);
        }
        check_launch("lbm step");
        return;
    }
    LGD_CHECK_CUDA(cudaMemsetAsync(e.d_counter + which_counter, 0, sizeof(int), e.stream));
    const int grid = e.sms * e.ctas_per_sm;
    int *counter = e.d_counter + which_counter;
    const void *a = e.buf[src];
    void *b = e.buf[1 - src];
    void *args[] = {&e.d_inst, &e.d_items, &e.n_items, &counter, &a, &b};
    LGD_CHECK_CUDA(cudaLaunchKernel(persistent_fn(e), dim3(grid), dim3(e.threads), args, 0, e.stream));
}

template<typename R, typename IDX, int TX, int TY>
static const void *tb2_fn()
{
    return (const void *)lbm_tb2_kernel<R, IDX, TX, TY>;
}

template<int TX, int TY>
static const void *tb2_geo(const Lbm& e, int *threads, size_t *smem)
{
    typedef Tb2Geo<TX, TY> G;
    *threads = G::THREADS;
    *smem = e.precision == 4 ? G::template smem<float>() : G::template smem<double>();
    if (e.precision == 4) return e.idx32 ? tb2_fn<float, int, TX, TY>() : tb2_fn<float, long long, TX, TY>();
    return e.idx32 ? tb2_fn<double, int, TX, TY>() : tb2_fn<double, long long, TX, TY>();
}

// the column shapes of the depth-2 kernel: 0 = 32 x 8, 1 = 32 x 4 (64 x 4
// and 16 x 8 columns measured slower on the 512-cavity ensemble: 33.0 and
// 25.1 GLUPS at their best residency, against 35.6 and 38.5)
constexpr int TB2_SHAPES = 2;
static int tb2_tx(int) { return 32; }
static int tb2_ty(int shape) { return shape == 1 ? 4 : 8; }

// the depth-2 kernel of the ensemble's precision, index width and column
// shape, its threads per CTA and shared memory per CTA
static const void *tb2_kernel(const Lbm& e, int shape, int *threads, size_t *smem)
{
    if (shape == 1) return tb2_geo<32, 4>(e, threads, smem);
    return tb2_geo<32, 8>(e, threads, smem);
}

// column work items of a depth-2 tile shape, largest instances first
// the work items of the two-step kernel with z chunks of about chunk planes,
// instances in the given order
static std::vector<int4> columns(const Lbm& e, const std::vector<int>& order, int shape, long long chunk)
{
    const int TX = tb2_tx(shape), TY = tb2_ty(shape);
    std::vector<int4> cols;
    for (int j : order) {
        const int L = e.inst[j].L;
        const int split = (int)std::max(1ll, (L + chunk / 2) / chunk);
        const int zc = (L + split - 1) / split;
        for (int z0 = 0; z0 < L; z0 += zc) {
            for (int y0 = 0; y0 < L; y0 += TY) {
                for (int x0 = 0; x0 < L; x0 += TX) cols.push_back(make_int4(j, x0 | y0 << 16, z0, std::min(L, z0 + zc)));
            }
        }
    }
    return cols;
}

// when the last of resident CTAs that pull these items is done, in planes (an
// item's own and one more at each end that is not a wall's)
static long long makespan(const Lbm& e, const std::vector<int4>& cols, int resident)
{
    std::priority_queue<long long, std::vector<long long>, std::greater<long long> > free_at;
    long long last = 0;
    for (const int4& c : cols) {
        long long start = 0;
        if ((int)free_at.size() == resident) {
            start = free_at.top();
            free_at.pop();
        }
        const long long end = start + (c.w - c.z) + (c.z > 0) + (c.w < e.inst[c.x].L);
        free_at.push(end);
        last = std::max(last, end);
    }
    return last;
}

static void build_cols(Lbm& e, int shape, int per_sm)
{
    const int TX = tb2_tx(shape), TY = tb2_ty(shape);
    std::vector<int> order(e.count);
    for (int j = 0; j < e.count; ++j) order[j] = j;
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return e.inst[a].L > e.inst[b].L; });
    // z chunks: the columns of a small ensemble are too few for the GPU and its
    // largest instances' would run alone at the end; about four items per
    // resident CTA, chunks of at least 16 planes.  Where whole columns are done
    // sooner (100 cavities of 24^3, 300 columns: 83 us per step against 106) they stay whole.
    long long planes = 0;
    for (const LbmInstance& in : e.inst) planes += (long long)((in.L + TX - 1) / TX) * ((in.L + TY - 1) / TY) * in.L;
    std::vector<int4> cols = columns(e, order, shape, std::max(16ll, planes / (16ll * e.sms)));
    std::vector<int4> whole = columns(e, order, shape, 1 << 20);
    if (makespan(e, whole, e.sms * per_sm) <= makespan(e, cols, e.sms * per_sm)) cols.swap(whole);
    if (e.d_cols) cudaFree(e.d_cols);
    e.d_cols = nullptr;
    LGD_CHECK_CUDA(cudaMalloc(&e.d_cols, sizeof(int4) * cols.size()));
    LGD_CHECK_CUDA(cudaMemcpyAsync(e.d_cols, cols.data(), sizeof(int4) * cols.size(), cudaMemcpyHostToDevice, e.stream));
    LGD_CHECK_CUDA(cudaStreamSynchronize(e.stream));
    e.n_cols = (int)cols.size();
    e.cols_shape = shape;
    e.cols_per_sm = per_sm;
}

// resident CTAs per SM of a depth-2 kernel, set up once per device and kernel
static int tb2_resident(const void *fn, int threads, size_t smem)
{
    static std::mutex m;
    static std::vector<std::pair<std::pair<int, const void *>, int> > known;
    int dev = 0;
    LGD_CHECK_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lock(m);
    for (const auto& k : known) {
        if (k.first.first == dev && k.first.second == fn) return k.second;
    }
    LGD_CHECK_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int per_sm = 0;
    LGD_CHECK_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, smem));
    known.push_back(std::make_pair(std::make_pair(dev, fn), per_sm));
    return per_sm;
}

// two steps of every instance in one launch (src -> 1 - src); with
// capturing set the caller is capturing the stream, so nothing here may
// allocate (prepare_tb2 first)
static void prepare_tb2(Lbm& e)
{
    int threads = 0;
    size_t smem = 0;
    const void *fn = tb2_kernel(e, e.tb_shape, &threads, &smem);
    const int fits = tb2_resident(fn, threads, smem);
    LGD_REQUIRE(fits >= 1, LGD_ERR_UNSUPPORTED, "the two-step kernel does not fit on this GPU");
    const int per_sm = std::min(std::max(1, e.tb_ctas), fits);
    if (e.cols_shape != e.tb_shape || e.cols_per_sm != per_sm || e.d_cols == nullptr) build_cols(e, e.tb_shape, per_sm);
}

static void launch_tb2(Lbm& e, int src)
{
    int threads = 0;
    size_t smem = 0;
    const void *fn = tb2_kernel(e, e.tb_shape, &threads, &smem);
    const int per_sm = tb2_resident(fn, threads, smem);
    LGD_CHECK_CUDA(cudaMemsetAsync(e.d_counter + 2, 0, sizeof(int), e.stream));
    const int grid = e.sms * std::min(std::max(1, e.tb_ctas), per_sm);
    int *counter = e.d_counter + 2;
    const void *a = e.buf[src];
    void *b = e.buf[1 - src];
    void *args[] = {&e.d_inst, &e.d_cols, &e.n_cols, &counter, &a, &b};
    LGD_CHECK_CUDA(cudaLaunchKernel(fn, dim3(grid), dim3(threads), args, smem, e.stream));
}

static void rebuild_graph2(Lbm& e)
{
    prepare_tb2(e);
    if (e.graph2_valid && e.graph2_key[0] == e.tb_shape && e.graph2_key[1] == e.tb_ctas && e.graph2_cols == e.d_cols) {
        return;
    }
    if (e.graph2_valid) {
        cudaGraphExecDestroy(e.graph2);
        e.graph2_valid = false;
    }
    cudaGraph_t g;
    LGD_CHECK_CUDA(cudaStreamBeginCapture(e.stream, cudaStreamCaptureModeThreadLocal));
    try {
        launch_tb2(e, 0);
        launch_tb2(e, 1);
    } catch (...) {
        cudaStreamEndCapture(e.stream, &g);
        throw;
    }
    LGD_CHECK_CUDA(cudaStreamEndCapture(e.stream, &g));
    cudaError_t err = cudaGraphInstantiate(&e.graph2, g, 0);
    cudaGraphDestroy(g);
    LGD_CHECK_CUDA(err);
    e.graph2_valid = true;
    e.graph2_key[0] = e.tb_shape;
    e.graph2_key[1] = e.tb_ctas;
    e.graph2_cols = e.d_cols;
}

static void launch_single(Lbm& e, int j, dim3 grid)
{
    if (e.variant == 1) {
        launch_single_nc<1>(e, j, grid);
    } else {
        launch_single_nc<0>(e, j, grid);
    }
    check_launch("lbm single");
}

static void rebuild_graph(Lbm& e)
{
    if (e.graph_valid) {
        cudaGraphExecDestroy(e.graph);
        e.graph_valid = false;
    }
    cudaGraph_t g;
    LGD_CHECK_CUDA(cudaStreamBeginCapture(e.stream, cudaStreamCaptureModeThreadLocal));
    try {
        launch_step(e, 0, 0);
        launch_step(e, 1, 1);
    } catch (...) {
        cudaStreamEndCapture(e.stream, &g);
        throw;
    }
    LGD_CHECK_CUDA(cudaStreamEndCapture(e.stream, &g));
    cudaError_t err = cudaGraphInstantiate(&e.graph, g, 0);
    cudaGraphDestroy(g);
    LGD_CHECK_CUDA(err);
    e.graph_valid = true;
}

static void set_config(Lbm& e, int ty, int threads, int ctas)
{
    LGD_REQUIRE(ty >= 1 && ty <= 1024, LGD_ERR_INVALID, "tile rows out of range");
    LGD_REQUIRE(threads == 64 || threads == 128 || threads == 256 || threads == 512 || threads == 1024, LGD_ERR_INVALID,
                "threads per CTA must be a power of two in [64, 1024]");
    LGD_REQUIRE(ctas >= 1 && ctas <= 32, LGD_ERR_INVALID, "CTAs per SM out of range");
    int max_ctas = 0;
    LGD_CHECK_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&max_ctas, persistent_fn(e), threads, 0));
    LGD_REQUIRE(max_ctas >= 1, LGD_ERR_INVALID, "kernel does not fit with this many threads");
    ctas = std::min(ctas, max_ctas);   // a persistent grid never exceeds what is resident
    const bool items_change = (ty != e.ty) || e.d_items == nullptr;
    e.ty = ty;
    e.threads = threads;
    e.ctas_per_sm = ctas;
    if (items_change) build_items(e);
    rebuild_graph(e);
}

static void report_config(const Lbm& e, int *tile_rows, int *threads, int *ctas_per_sm)
{
    if (tile_rows) *tile_rows = e.flat ? FLAT_ROWS : e.ty;
    if (threads) *threads = e.flat ? FLAT : e.threads;
    if (ctas_per_sm) *ctas_per_sm = e.flat ? FLAT_CTAS : e.ctas_per_sm;
}

static void run_steps(Lbm& e, int steps)
{
    if (e.depth == 2) {
        // pairs of steps in one launch each (four steps per graph replay
        // from buffer 0), a last odd step on its own
        prepare_tb2(e);
        if (e.cur == 1 && steps >= 2) {
            launch_tb2(e, 1);
            ++e.launches;
            e.cur = 0;
            steps -= 2;
        }
        if (steps >= 4) rebuild_graph2(e);
        for (; steps >= 4; steps -= 4) {
            LGD_CHECK_CUDA(cudaGraphLaunch(e.graph2, e.stream));
            e.launches += 2;
        }
        for (; steps >= 2; steps -= 2) {
            launch_tb2(e, e.cur);
            ++e.launches;
            e.cur = 1 - e.cur;
        }
        if (steps == 1) {
            launch_step(e, 0, e.cur);
            ++e.launches;
            e.cur = 1 - e.cur;
        }
        return;
    }
    int s = 0;
    if (e.cur == 1 && steps > 0) {
        launch_step(e, 0, 1);
        ++e.launches;
        e.cur = 0;
        ++s;
    }
    for (; s + 1 < steps; s += 2) {
        LGD_CHECK_CUDA(cudaGraphLaunch(e.graph, e.stream));
        e.launches += 2;
    }
    if (s < steps) {
        launch_step(e, 0, 0);
        ++e.launches;
        e.cur = 1;
    }
}

// the fastest kernel of single steps, then of two steps per launch; returns its
// milliseconds per step
static double tune(Lbm& e, int trial_steps)
{
    struct Events {
        cudaEvent_t t[2] = {};
        ~Events()
        {
            for (cudaEvent_t ev : t) {
                if (ev) cudaEventDestroy(ev);
            }
        }
    } events;
    for (cudaEvent_t& ev : events.t) LGD_CHECK_CUDA(cudaEventCreate(&ev));
    const cudaEvent_t t0 = events.t[0], t1 = events.t[1];
    // the trial runs advance the ensemble: callers reset or upload afterwards
    auto measure = [&](int ty, int th, int ct) -> double {
        int fits = 0;
        LGD_CHECK_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fits, persistent_fn(e), th, 0));
        if (fits < 1) return std::numeric_limits<double>::infinity();   // too many registers for th threads
        set_config(e, ty, th, ct);
        run_steps(e, 2);   // warm
        LGD_CHECK_CUDA(cudaEventRecord(t0, e.stream));
        run_steps(e, trial_steps);
        LGD_CHECK_CUDA(cudaEventRecord(t1, e.stream));
        LGD_CHECK_CUDA(cudaEventSynchronize(t1));
        float ms = 0.f;
        LGD_CHECK_CUDA(cudaEventElapsedTime(&ms, t0, t1));
        return ms / trial_steps;
    };
    // one thread per cell, then a pattern search over (log2 tile rows,
    // log2 threads, CTAs per SM)
    const bool flat = e.d_blocks != nullptr;
    e.flat = flat;
    const double flat_ms = measure(e.ty, e.threads, e.ctas_per_sm);
    e.flat = false;
    const int tys[] = {1, 2, 4, 8, 16, 32};
    const int ths[] = {128, 256, 512};
    const int cts[] = {1, 2, 3, 4, 6, 8};
    int a = 2, b = 1, c = 3;   // start at (4, 256, 4)
    double best = measure(tys[a], ths[b], cts[c]);
    bool moved = true;
    int evals = 1;
    while (moved && evals < 40) {
        moved = false;
        const int da[6] = {-1, 1, 0, 0, 0, 0};
        const int db[6] = {0, 0, -1, 1, 0, 0};
        const int dc[6] = {0, 0, 0, 0, -1, 1};
        int ba = a, bb = b, bc = c;
        for (int k = 0; k < 6; ++k) {
            const int na = a + da[k], nb = b + db[k], nc = c + dc[k];
            if (na < 0 || na >= 6 || nb < 0 || nb >= 3 || nc < 0 || nc >= 6) continue;
            const double t = measure(tys[na], ths[nb], cts[nc]);
            ++evals;
            if (t < best * 0.99) {
                best = t;
                ba = na;
                bb = nb;
                bc = nc;
                moved = true;
            }
        }
        a = ba;
        b = bb;
        c = bc;
    }
    // the first measurement pays for the ensemble's first steps: repeated
    e.flat = flat;
    const double flat_best = std::min(flat_ms, measure(tys[a], ths[b], cts[c]));
    e.flat = flat && flat_best <= best;
    best = std::min(best, flat_best);
    set_config(e, tys[a], ths[b], cts[c]);
    // then temporal blocking: two steps per launch in each tile shape
    // and residency; the fastest per step wins, one step per launch
    // included (the reference's autotuner tunes the pipeline length of
    // its cache-blocking simulator the same way,
    // misc/cacheblockingsimulationfactory.h:26-28)
    e.depth = 1;
    int best_depth = 1, best_shape = 0, best_ctas = 1;
    for (int shape = 0; shape < TB2_SHAPES; ++shape) {
        int threads = 0;
        size_t smem = 0;
        const void *fn = tb2_kernel(e, shape, &threads, &smem);
        const int per_sm = tb2_resident(fn, threads, smem);
        for (int ct = 1; ct <= std::min(per_sm, 8); ++ct) {
            e.depth = 2;
            e.tb_shape = shape;
            e.tb_ctas = ct;
            run_steps(e, 2);   // warm (builds the columns)
            const int n = 2 * ((trial_steps + 1) / 2);
            LGD_CHECK_CUDA(cudaEventRecord(t0, e.stream));
            run_steps(e, n);
            LGD_CHECK_CUDA(cudaEventRecord(t1, e.stream));
            LGD_CHECK_CUDA(cudaEventSynchronize(t1));
            float ms = 0.f;
            LGD_CHECK_CUDA(cudaEventElapsedTime(&ms, t0, t1));
            const double t = ms / n;
            if (t < best * 0.99) {
                best = t;
                best_depth = 2;
                best_shape = shape;
                best_ctas = ct;
            }
        }
    }
    e.depth = best_depth;
    e.tb_shape = best_shape;
    e.tb_ctas = best_ctas;
    LGD_CHECK_CUDA(cudaStreamSynchronize(e.stream));
    return best;
}

static void lbm_free(Lbm& e)
{
    if (e.stream) cudaStreamSynchronize(e.stream);
    if (e.graph_valid) cudaGraphExecDestroy(e.graph);
    if (e.graph2_valid) cudaGraphExecDestroy(e.graph2);
    cudaFree(e.buf[0]);
    cudaFree(e.buf[1]);
    cudaFree(e.d_inst);
    cudaFree(e.d_items);
    cudaFree(e.d_cols);
    cudaFree(e.d_blocks);
    cudaFree(e.d_stage);
    cudaFree(e.d_counter);
    if (e.stream) cudaStreamDestroy(e.stream);
}

}  // namespace lgd

using namespace lgd;

extern "C" {

int lgd_lbm_create(int count, const int32_t *edges, const double *omegas, double lid, int precision, lgd_lbm **out)
{
    return guard([&] {
        LGD_REQUIRE(out != nullptr, LGD_ERR_INVALID, "null output");
        *out = nullptr;
        LGD_REQUIRE(count > 0 && edges && omegas, LGD_ERR_INVALID, "need at least one instance");
        LGD_REQUIRE(precision == 4 || precision == 8, LGD_ERR_INVALID, "precision must be 4 (FP32) or 8 (FP64)");
        Lbm *e = new Lbm();
        e->count = count;
        e->precision = precision;
        e->inst.resize(count);
        long long off = 0;
        e->idx32 = true;
        for (int j = 0; j < count; ++j) {
            LGD_REQUIRE(edges[j] >= 2 && edges[j] <= 1024, LGD_ERR_RANGE, "instance edge must lie in [2, 1024]");
            LGD_REQUIRE(omegas[j] > 0.0 && omegas[j] < 2.0, LGD_ERR_RANGE, "omega must lie in (0, 2)");
            LbmInstance& in = e->inst[j];
            in.base = off;
            in.L = edges[j];
            in.magic = (unsigned)((0x100000000ull + edges[j] - 1) / edges[j]);
            in.omega = omegas[j];
            in.lid = lid;
            in.omega_f = (float)omegas[j];
            in.lid_f = (float)lid;
            const long long n3 = (long long)edges[j] * edges[j] * edges[j];
            in.pitch = (n3 + 31) / 32 * 32;
            off += 19 * in.pitch;
            e->total_cells += n3;
            if (19 * in.pitch >= (1ll << 31)) e->idx32 = false;
            LGD_REQUIRE(n3 * 19 < (1ll << 31) * 16, LGD_ERR_RANGE, "instance too large");
        }
        e->total_elems = off;
        int dev = 0;
        try {
            LGD_CHECK_CUDA(cudaGetDevice(&dev));
            LGD_CHECK_CUDA(cudaDeviceGetAttribute(&e->sms, cudaDevAttrMultiProcessorCount, dev));
            LGD_CHECK_CUDA(cudaStreamCreateWithFlags(&e->stream, cudaStreamNonBlocking));
            for (int b = 0; b < 2; ++b) LGD_CHECK_CUDA(cudaMalloc(&e->buf[b], (size_t)precision * off));
            LGD_CHECK_CUDA(cudaMalloc(&e->d_inst, sizeof(LbmInstance) * count));
            LGD_CHECK_CUDA(cudaMemcpyAsync(e->d_inst, e->inst.data(), sizeof(LbmInstance) * count,
                                           cudaMemcpyHostToDevice, e->stream));
            LGD_CHECK_CUDA(cudaMalloc(&e->d_counter, sizeof(int) * 3));   // two captured steps, the depth-2 launch
            e->depth = 1;
            e->tb_ctas = 1;
            dim3 grid(256, count);
            if (precision == 4) {
                lbm_rest_kernel<float><<<grid, 256, 0, e->stream>>>(e->d_inst, count, (float *)e->buf[0]);
            } else {
                lbm_rest_kernel<double><<<grid, 256, 0, e->stream>>>(e->d_inst, count, (double *)e->buf[0]);
            }
            check_launch("lbm rest state");
            ++e->launches;
            build_blocks(*e);
            e->flat = e->d_blocks != nullptr;
            set_config(*e, 4, 256, 4);
        } catch (...) {
            lbm_free(*e);
            delete e;
            throw;
        }
        *out = reinterpret_cast<lgd_lbm *>(e);
    });
}

int lgd_lbm_destroy(lgd_lbm *h)
{
    return guard([&] {
        if (!h) return;
        Lbm& e = lbm_of(h);
        lbm_free(e);
        delete &e;
    });
}

int lgd_lbm_step(lgd_lbm *h, int steps)
{
    return guard([&] {
        Lbm& e = lbm_of(h);
        LGD_REQUIRE(steps >= 0, LGD_ERR_INVALID, "negative step count");
        run_steps(e, steps);
    });
}

int lgd_lbm_step_looped(lgd_lbm *h, int steps)
{
    return guard([&] {
        Lbm& e = lbm_of(h);
        LGD_REQUIRE(steps >= 0, LGD_ERR_INVALID, "negative step count");
        for (int s = 0; s < steps; ++s) {
            for (int j = 0; j < e.count; ++j) {
                const int L = e.inst[j].L;
                const int rows = std::max(1, 256 / L);
                launch_single(e, j, dim3((L + rows - 1) / rows, L));
                ++e.launches;
            }
            e.cur = 1 - e.cur;
        }
    });
}

int lgd_lbm_set_config(lgd_lbm *h, int tile_rows, int threads, int ctas_per_sm)
{
    return guard([&] {
        Lbm& e = lbm_of(h);
        const bool before = e.flat;
        e.flat = e.d_blocks != nullptr && tile_rows == FLAT_ROWS && threads == FLAT && ctas_per_sm == FLAT_CTAS;
        try {
            if (e.flat) rebuild_graph(e);
            else set_config(e, tile_rows, threads, ctas_per_sm);
        } catch (...) {
            e.flat = before;
            throw;
        }
    });
}

int lgd_lbm_get_config(lgd_lbm *h, int *tile_rows, int *threads, int *ctas_per_sm)
{
    return guard([&] {
        report_config(lbm_of(h), tile_rows, threads, ctas_per_sm);
    });
}

int lgd_lbm_tune(lgd_lbm *h, int trial_steps, int *tile_rows, int *threads, int *ctas_per_sm, double *best_ms)
{
    return guard([&] {
        Lbm& e = lbm_of(h);
        LGD_REQUIRE(trial_steps >= 2, LGD_ERR_INVALID, "trial_steps must be at least 2");
        const bool flat = e.flat;
        const int depth = e.depth;
        double best = 0.0;
        try {
            best = tune(e, trial_steps);
        } catch (...) {
            // the kernels as they were (the persistent kernel's shape is the search's last)
            e.flat = flat;
            e.depth = depth;
            try {
                rebuild_graph(e);
            } catch (...) {
            }
            throw;
        }
        report_config(e, tile_rows, threads, ctas_per_sm);
        if (best_ms) *best_ms = best;
    });
}

int lgd_lbm_set_time_block(lgd_lbm *h, int depth, int shape, int ctas_per_sm)
{
    return guard([&] {
        Lbm& e = lbm_of(h);
        LGD_REQUIRE(depth == 1 || depth == 2, LGD_ERR_INVALID, "the ensemble fuses one or two steps per launch");
        LGD_REQUIRE(shape >= 0 && shape < TB2_SHAPES, LGD_ERR_INVALID,
                    "column shape must be 0 (32 x 8) or 1 (32 x 4)");
        LGD_REQUIRE(ctas_per_sm >= 1 && ctas_per_sm <= 32, LGD_ERR_INVALID, "CTAs per SM out of range");
        if (depth == 2) {
            int threads = 0;
            size_t smem = 0;
            const void *fn = tb2_kernel(e, shape, &threads, &smem);
            LGD_REQUIRE(tb2_resident(fn, threads, smem) >= 1, LGD_ERR_UNSUPPORTED,
                        "the two-step kernel does not fit on this GPU");
        }
        e.depth = depth;
        e.tb_shape = shape;
        e.tb_ctas = ctas_per_sm;
    });
}

int lgd_lbm_get_time_block(lgd_lbm *h, int *depth, int *shape, int *ctas_per_sm)
{
    return guard([&] {
        Lbm& e = lbm_of(h);
        if (depth) *depth = e.depth;
        if (shape) *shape = e.tb_shape;
        if (ctas_per_sm) *ctas_per_sm = e.tb_ctas;
    });
}

int lgd_lbm_reset(lgd_lbm *h)
{
    return guard([&] {
        Lbm& e = lbm_of(h);
        dim3 grid(256, e.count);
        if (e.precision == 4) {
            lbm_rest_kernel<float><<<grid, 256, 0, e.stream>>>(e.d_inst, e.count, (float *)e.buf[0]);
        } else {
            lbm_rest_kernel<double><<<grid, 256, 0, e.stream>>>(e.d_inst, e.count, (double *)e.buf[0]);
        }
        check_launch("lbm rest state");
        ++e.launches;
        e.cur = 0;
        LGD_CHECK_CUDA(cudaStreamSynchronize(e.stream));
    });
}

int lgd_lbm_download(lgd_lbm *h, int instance, double *f, size_t bytes)
{
    return guard([&] {
        Lbm& e = lbm_of(h);
        LGD_REQUIRE(instance >= 0 && instance < e.count, LGD_ERR_RANGE, "instance out of range");
        const LbmInstance& in = e.inst[instance];
        const size_t n = 19ull * in.L * in.L * in.L;
        LGD_REQUIRE(f != nullptr && bytes == n * sizeof(double), LGD_ERR_INVALID, "buffer must hold 19 * L^3 doubles");
        const size_t n3 = n / 19;
        copy_instance(e, in, n3, f, false);
    });
}

int lgd_lbm_upload(lgd_lbm *h, int instance, const double *f, size_t bytes)
{
    return guard([&] {
        Lbm& e = lbm_of(h);
        LGD_REQUIRE(instance >= 0 && instance < e.count, LGD_ERR_RANGE, "instance out of range");
        const LbmInstance& in = e.inst[instance];
        const size_t n = 19ull * in.L * in.L * in.L;
        LGD_REQUIRE(f != nullptr && bytes == n * sizeof(double), LGD_ERR_INVALID, "buffer must hold 19 * L^3 doubles");
        const size_t n3 = n / 19;
        copy_instance(e, in, n3, const_cast<double *>(f), true);
    });
}

int lgd_lbm_info(lgd_lbm *h, long long *total_cells, int *work_items)
{
    return guard([&] {
        Lbm& e = lbm_of(h);
        if (total_cells) *total_cells = e.total_cells;
        if (work_items) *work_items = e.n_items;
    });
}

int lgd_lbm_synchronize(lgd_lbm *h)
{
    return guard([&] { LGD_CHECK_CUDA(cudaStreamSynchronize(lbm_of(h).stream)); });
}

int lgd_lbm_stream(lgd_lbm *h, void **stream)
{
    return guard([&] {
        LGD_REQUIRE(stream != nullptr, LGD_ERR_INVALID, "null output");
        *stream = (void *)lbm_of(h).stream;
    });
}

int lgd_lbm_set_variant(lgd_lbm *h, int variant)
{
    return guard([&] {
        Lbm& e = lbm_of(h);
        LGD_REQUIRE(variant == 0 || variant == 1, LGD_ERR_INVALID, "LBM kernel variant must be 0 or 1");
        e.variant = variant;
        set_config(e, e.ty, e.threads, e.ctas_per_sm);   // re-checks residency, recaptures the graph
    });
}

int lgd_lbm_launch_count(lgd_lbm *h, uint64_t *count)
{
    return guard([&] {
        LGD_REQUIRE(count != nullptr, LGD_ERR_INVALID, "null output");
        *count = lbm_of(h).launches;
    });
}

}  // extern "C"
