// Variable-coefficient diffusion (FP32, torus), two time steps per pass over
// memory: 12 bytes per cell and pass (u and k read, u written) for two steps.
//
// A CTA owns a box of 64 x (ROWS * WY) cells of every z plane of its z chunk
// and marches in z; every lane owns two x-neighbouring cells of ROWS rows at
// both levels.  At iteration i (input plane i has landed) level 1 computes its
// plane i - 1 from the input and level 2 its plane i - 2 from level 1:
//   - the centre and the z neighbours of u and k sit in the thread's registers
//     (four planes of each rotate, the loop is unrolled four times so that the
//     rotation is a renaming),
//   - the x neighbours come from the adjacent lanes by shuffle,
//   - the rows just outside the thread's block come from shared memory: the
//     input rings of u and k, and a two-slot ring of level-1 planes.
// Input planes arrive by cp.async in 16-byte pieces, two planes ahead; every
// thread wraps the addresses of its own pieces once, so the torus costs
// nothing in the loop.  One __syncthreads per plane.  Level 2 stores the inner
// 56 x (BH - 4) cells, the rim is recomputed by the neighbouring CTAs.
//
// The arithmetic is varcoef_pair_f32's, rounding for rounding, so the result is
// two single steps' bit for bit, but scalar: a face between two of a thread's
// own cells is taken once (its other side is the exact negative, which an FMA
// takes for free), and packed operands of shifted neighbours would have to be
// put together by moves (61 instructions per two cells and level; 36 us per step of
// 256^3 in that form).
//
// Measured, us per step against the single-step TMA kernel: 32^3 2.1 / 9.6,
// 128^3 6.0 / 12.7, 200^3 16.4 / 27.9, 256^3 29.4 / 41.7 (570 GLUPS; DRAM at a
// third of its rate).  Bound by issue and the shared-memory pipe: per two
// cells and level 33 FP32 instructions, 4 shuffles (4 clocks of a quarter
// each) and 2.3 shared-memory accesses of 64 bits (8 clocks each), with three
// warps per SM quarter to cover their latency.
#include <algorithm>
#include <type_traits>

#include "lgd_internal.h"
#include "k_cells.cuh"
#include "z_chunks.h"

namespace lgd {
namespace vctb {

constexpr int BW = 64;
constexpr int XP = 4;               // x halo: two cells are needed, pieces are four
constexpr int OX = BW - 2 * XP;
constexpr int D = 2;                // planes in flight ahead
constexpr int SU = D + 2;           // u ring: planes i - 1, i and D ahead
constexpr int SK = 8;               // k ring: level 2 still reads plane i - 2; two groups of four, so that
                                    // slots are constants in the loop unrolled by four

template<int WY, int ROWS>
struct Geo {
    static constexpr int THREADS = 32 * WY;
    static constexpr int BH = WY * ROWS;
    static constexpr int OY = BH - 4;
    static constexpr int PLANE = BW * BH;           // floats
    static constexpr int SMEM = (SU + SK + 2) * PLANE * 4;
    static constexpr int PIECES = PLANE / 4;        // 16-byte pieces of a plane
    static constexpr int PER = (PIECES + THREADS - 1) / THREADS;
};

__device__ __forceinline__ void copy16(float *dst, const float *src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}

template<int WY, int ROWS, int CTAS>
__global__ void __launch_bounds__(32 * WY, CTAS)
varcoef_tb2_kernel(const float *u, const float *k, float *out, long pitch, int nx, int ny, int nz, int zchunk)
{
    typedef Geo<WY, ROWS> G;
    extern __shared__ __align__(16) float smem[];
    float *const us = smem;
    float *const ks = smem + SU * G::PLANE;
    float *const l1 = smem + (SU + SK) * G::PLANE;

    const int tid = threadIdx.x;
    const int lane = tid & 31;
    const int warp = tid >> 5;
    const int x0 = blockIdx.x * OX;
    const int y0 = blockIdx.y * G::OY;
    const int z0 = blockIdx.z * zchunk;
    const int z1 = min(z0 + zchunk, nz);
    const int nq = (z1 - z0) + 4;               // input plane q is z = z0 - 2 + q
    const long plane = pitch * ny;

    // this thread's pieces of a plane: offsets in the grid and in a slot
    int goff[G::PER], soff[G::PER];
#pragma unroll
    for (int j = 0; j < G::PER; ++j) {
        const int piece = tid + j * G::THREADS;
        const int row = piece / (BW / 4);
        const int cx = piece % (BW / 4) * 4;
        int gx = (x0 - XP + cx) % nx;           // nx is a multiple of 4: a piece never straddles the wrap
        int gy = (y0 - 2 + row) % ny;
        if (gx < 0) gx += nx;
        if (gy < 0) gy += ny;
        goff[j] = (int)(gy * pitch) + gx;       // a plane has fewer than 2^31 elements (host rule)
        soff[j] = piece < G::PIECES ? row * BW + cx : -1;
    }
    int zi = (z0 - 2) % nz;                     // grid plane of the next copy
    if (zi < 0) zi += nz;
    const float *pu = u + zi * plane, *pk = k + zi * plane;
    auto issue = [&](float *du, float *dk) {                    // the next plane into its slots
#pragma unroll
        for (int j = 0; j < G::PER; ++j) {
            if (G::PIECES % G::THREADS == 0 || soff[j] >= 0) {
                copy16(du + soff[j], pu + goff[j]);
                copy16(dk + soff[j], pk + goff[j]);
            }
        }
        if (++zi == nz) {
            zi = 0;
            pu = u;
            pk = k;
        } else {
            pu += plane;
            pk += plane;
        }
    };
    auto commit = [] { asm volatile("cp.async.commit_group;" ::: "memory"); };
    dependent_start();
    issue(us, ks);                                              // nq >= 5
    commit();
    issue(us + G::PLANE, ks + G::PLANE);
    commit();

    const int r0 = warp * ROWS;
    const int cx = 2 * lane;
    const int gx = x0 - XP + cx;
    const int rn = max(r0 - 1, 0) * BW + cx;                    // rim rows, clamped to the box (the clamped
    const int rs = min(r0 + ROWS, G::BH - 1) * BW + cx;         // values only reach cells outside the tile)
    unsigned keep = 0;                                          // rows of the thread that are stored
    if (cx >= XP && cx < XP + OX && gx < nx) {                  // nx is even: both cells or none
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
            if (r0 + r >= 2 && r0 + r < 2 + G::OY && y0 - 2 + r0 + r < ny) keep |= 1u << r;
        }
    }
    float *o = out + (long)z0 * plane + (long)(y0 - 2 + r0) * pitch + gx;

    float2 a0[4][ROWS], a1[4][ROWS], kk[4][ROWS];               // input, level 1, coefficient; plane p in [p % 4]

    auto ld = [](const float *p) { return *reinterpret_cast<const float2 *>(p); };

    // one level: plane c (b below, t above) of v and kk, rim rows from pv / pk
    auto level = [&](const float2 (&vb)[ROWS], const float2 (&vc)[ROWS], const float2 (&vt)[ROWS],
                     const float2 (&kb)[ROWS], const float2 (&kc)[ROWS], const float2 (&kt)[ROWS], const float *pv,
                     const float *pk, float2 (&res)[ROWS]) {
        const float2 vn = ld(pv + rn), vs = ld(pv + rs), kn = ld(pk + rn), ksr = ld(pk + rs);
        // the face between this row and the one above: sum of k, difference of u
        float nk0 = kn.x + kc[0].x, nd0 = vn.x - vc[0].x;
        float nk1 = kn.y + kc[0].y, nd1 = vn.y - vc[0].y;
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
            const float u0 = vc[r].x, u1 = vc[r].y, k0 = kc[r].x, k1 = kc[r].y;
            const float uw = __shfl_up_sync(0xffffffffu, u1, 1), kw = __shfl_up_sync(0xffffffffu, k1, 1);
            const float ue = __shfl_down_sync(0xffffffffu, u0, 1), ke = __shfl_down_sync(0xffffffffu, k0, 1);
            const float km = k0 + k1, dm = u1 - u0;
            const float2 us2 = r == ROWS - 1 ? vs : vc[r + 1];
            const float2 ks2 = r == ROWS - 1 ? ksr : kc[r + 1];
            const float sk0 = k0 + ks2.x, sd0 = us2.x - u0;
            const float sk1 = k1 + ks2.y, sd1 = us2.y - u1;
            float f0 = (k0 + kw) * (uw - u0);                               // west, east, north, south, below, above
            float f1 = km * -dm;
            f0 = fmaf(km, dm, f0);
            f1 = fmaf(k1 + ke, ue - u1, f1);
            f0 = fmaf(nk0, nd0, f0);
            f1 = fmaf(nk1, nd1, f1);
            f0 = fmaf(sk0, sd0, f0);
            f1 = fmaf(sk1, sd1, f1);
            f0 = fmaf(k0 + kb[r].x, vb[r].x - u0, f0);
            f1 = fmaf(k1 + kb[r].y, vb[r].y - u1, f1);
            f0 = fmaf(k0 + kt[r].x, vt[r].x - u0, f0);
            f1 = fmaf(k1 + kt[r].y, vt[r].y - u1, f1);
            res[r] = make_float2(fmaf(0.5f, f0, u0), fmaf(0.5f, f1, u1));
            nk0 = sk0;
            nk1 = sk1;
            nd0 = -sd0;
            nd1 = -sd1;
        }
    };

    auto iteration = [&](auto phase, int i) {
        constexpr int P0 = decltype(phase)::value;              // plane i (i % 4)
        constexpr int P1 = (P0 + 3) % 4;                        // plane i - 1
        constexpr int P2 = (P0 + 2) % 4;
        constexpr int P3 = (P0 + 1) % 4;
        // k slots: this group of four planes and the one before / after it
        float *const kg = ks + (i & 4) * G::PLANE;
        float *const kh = ks + (~i & 4) * G::PLANE;
        asm volatile("cp.async.wait_group %0;" ::"n"(D - 1) : "memory");
        __syncthreads();            // plane i is there for all; the slots the next copies take are free
        if (i + D < nq) issue(us + P2 * G::PLANE, (P0 < 2 ? kg : kh) + P2 * G::PLANE);
        commit();
        const int own = r0 * BW + cx;
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
            a0[P0][r] = ld(us + P0 * G::PLANE + own + r * BW);
            kk[P0][r] = ld(kg + P0 * G::PLANE + own + r * BW);
        }
        if (i < 2) return;
        level(a0[P2], a0[P1], a0[P0], kk[P2], kk[P1], kk[P0], us + P1 * G::PLANE,
              (P0 >= 1 ? kg : kh) + P1 * G::PLANE, a1[P1]);
        // only the block's outer rows are read by other warps
        float *d = l1 + (P1 & 1) * G::PLANE + own;
        *reinterpret_cast<float2 *>(d) = a1[P1][0];
        *reinterpret_cast<float2 *>(d + (ROWS - 1) * BW) = a1[P1][ROWS - 1];
        if (i < 4) return;
        float2 res[ROWS];
        level(a1[P3], a1[P2], a1[P1], kk[P3], kk[P2], kk[P1], l1 + (P2 & 1) * G::PLANE,
              (P0 >= 2 ? kg : kh) + P2 * G::PLANE, res);
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
            if ((keep >> r) & 1u) *reinterpret_cast<float2 *>(o + r * pitch) = res[r];
        }
        o += plane;
    };

    for (int i = 0; i < nq; i += 4) {
        iteration(std::integral_constant<int, 0>(), i);
        if (i + 1 < nq) iteration(std::integral_constant<int, 1>(), i + 1);
        if (i + 2 < nq) iteration(std::integral_constant<int, 2>(), i + 2);
        if (i + 3 < nq) iteration(std::integral_constant<int, 3>(), i + 3);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
}

struct Plan {
    int zchunk;
    double us;          // of a pass, with the input planes that only load counted in full
    double pass_us;     // of a pass
};

template<int WY, int ROWS, int CTAS>
static Plan plan(const Grid& g, double us_per_plane)
{
    typedef Geo<WY, ROWS> G;
    static PerDevice<int> setup;
    const int resident = setup.get([] {
        auto *fn = varcoef_tb2_kernel<WY, ROWS, CTAS>;
        LGD_CHECK_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, G::SMEM));
        int dev = 0, count = 0, per_sm = 0;
        LGD_CHECK_CUDA(cudaGetDevice(&dev));
        LGD_CHECK_CUDA(cudaDeviceGetAttribute(&count, cudaDevAttrMultiProcessorCount, dev));
        LGD_CHECK_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, G::THREADS, G::SMEM));
        return count * std::max(1, per_sm);
    });
    const long long xy = (long long)((g.desc.nx + OX - 1) / OX) * ((g.desc.ny + G::OY - 1) / G::OY);
    Plan best;
    double planes;
    best.zchunk = least_planes(xy, g.desc.nz, resident, 5, &planes, 4);
    best.us = planes * us_per_plane;
    const long long waves = (xy * ((g.desc.nz + best.zchunk - 1) / best.zchunk) + resident - 1) / resident;
    best.pass_us = (double)waves * (best.zchunk + 2.5) * us_per_plane;
    return best;
}

template<int WY, int ROWS, int CTAS>
static void launch(Grid& g, int zchunk)
{
    typedef Geo<WY, ROWS> G;
    launch_dependent(varcoef_tb2_kernel<WY, ROWS, CTAS>,
                     dim3((g.desc.nx + OX - 1) / OX, (g.desc.ny + G::OY - 1) / G::OY, (g.desc.nz + zchunk - 1) / zchunk),
                     G::THREADS, G::SMEM, g.stream, (const float *)g.m[0].buf[g.cur], (const float *)g.m[1].buf[0],
                     (float *)g.m[0].buf[1 - g.cur], (long)(g.pitch_bytes[0] / 4), g.desc.nx, g.desc.ny, g.desc.nz,
                     zchunk);
    check_launch("varcoef two steps");
    ++g.launches;
    g.cur = 1 - g.cur;
}

}  // namespace vctb

// FP32 cells on a full torus whose rows are a multiple of 16 bytes
bool varcoef_tb2_applicable(const Grid& g)
{
    return g.desc.cell == LGD_CELL_VARCOEF_F32 && g.desc.dim == 3 && g.desc.periodic == 7 && g.desc.nx % 4 == 0 &&
           g.pitch_bytes[0] == g.pitch_bytes[1] && (long long)g.pitch_bytes[0] / 4 * g.desc.ny < (1ll << 31);
}

// Two boxes: 48 rows, one CTA per SM, or 24 rows, two per SM (finer bands of
// y); the one whose waves of CTAs times planes per CTA (five of them halo) take
// less by the measured time per plane.  Beside two single steps of single_us by the
// TMA kernel's 64 x 16 boxes, which waste less of thin grids, where the caller asked
// for no depth: false (nothing launched) where those take less.  us per step, two
// steps per pass / single: 1 x 2048 x 4096 48 / 37, 256 x 1 x 4096 33 / 22, 3000 x 64 x
// 64 41 / 32, but 256^3 30 / 40; of 250 grids of 1 to 4096 cells along an axis the rule is
// 1% off the better one on average, and at the worst 25% (256 x 16 x 4096 34 / 42).
bool launch_varcoef_tb2(Grid& g, double single_us)
{
    const vctb::Plan tall = vctb::plan<12, 4, 1>(g, 1.17), low = vctb::plan<8, 3, 2>(g, 1.03);
    const vctb::Plan& best = tall.us <= low.us ? tall : low;
    constexpr double LEAST_US = 4.0;            // any dependent launch
    if (single_us > 0.0 && std::max(best.pass_us, LEAST_US) > 2.0 * std::max(single_us, LEAST_US)) return false;
    if (&best == &tall) vctb::launch<12, 4, 1>(g, tall.zchunk);
    else vctb::launch<8, 3, 2>(g, low.zchunk);
    return true;
}

}  // namespace lgd
