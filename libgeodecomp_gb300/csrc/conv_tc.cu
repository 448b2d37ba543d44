// The surrogate's 3^3 convolutions (C = 24) on the fifth-generation tensor
// cores: tcgen05.mma with BF16 operands in shared memory and FP32 accumulators
// in tensor memory.  One kernel, four input forms:
//   MID    24 channels, ghosted BF16 activations (layers 2 and 3, and the
//          input gradients of layers 2 and 3 with mirrored weights);
//   FIRST  the fields u and kappa in FP32 (layer 1; rounded to BF16 here);
//   LAST   24 channels -> 1 (layer 4);
//   DLAST  the loss gradient 2 (du - target) / N, one channel (the input
//          gradient of layer 4);
// and three epilogues: ACT (bias, GELU, ghosted BF16 output; when training also
// GELU' in FP32 for the backward pass, from the same terms), GRAD
// (times the saved GELU', ghosted BF16 output, bias gradient), OUT (FP32 du, or
// u += du).
//
// Why this shape.  An MMA of 128 voxels x N x 16 reads 4 KB of A and 32 N
// bytes of B from shared memory at 128 B per clock; with N = 24 (one tap at a
// time) that read, not the multiplication, sets the time (2160 clocks per 128
// voxels and layer).  So the three taps in z become N: when input plane q
// arrives, the nine taps in (y, x) of all three output planes q - 2, q - 1, q
// it reaches are multiplied at once, into three adjacent accumulators of 24
// columns (N = 80).  An accumulator is complete after three input planes; the
// epilogue reads it and puts the bias back into it, for the plane that takes
// its place (three slots in rotation: the weights are stored twice over, so
// that the rotation is a start address).  K runs over 9 taps x 24 channels =
// 27 groups of 8; a K-step's two groups come from two taps, so that only the
// last tap needs a zero group: 14 K-steps, 728 clocks of operand reads per 128
// voxels (FIRST and DLAST: the three taps in x sit in the 8 channels of a
// group, 2 K-steps).  And an input plane is used up at once: two or three
// slots of input suffice.
//
// A CTA owns TXW x TY = 512 output voxels of every plane of its z chunk: four
// accumulator tiles of 128 voxels (128 x 1, 64 x 2 or 32 x 4 each).  A plane
// of input sits in shared memory as [channel group][row][8 voxels + 2 halo]
// x 16 B: every 8-voxel core matrix brings its own halo, so tap (dy, dx) of
// any tile is a start address and M may span rows.
//   - two warps (LAST: four) issue the MMAs, each for its share of the tiles;
//   - 16 warps: epilogue, four to a tile, by lane quarter;
//   - four warps fill the input slots (cp.async; FIRST and DLAST build their
//     groups from the FP32 fields).
// At 256^3 the layers take 450 (FIRST), 470 (MID) and 310 us (LAST).  MID is
// bound by the MMAs' operand reads (80% of the cycles); FIRST by the
// epilogue, 900 instructions per 32 voxels and about half of the FMA pipe.
// Every wait is bounded and gives up early once another role has failed; a
// CTA that gives up sets the error word, lets its copies and MMAs finish and
// frees its tensor memory.
#include <algorithm>

#include "lgd_internal.h"
#include "tc_common.cuh"
#include "conv_tc.h"
#include "z_chunks.h"

namespace lgd {
namespace sur {
namespace tc {

enum { MID = 0, FIRST = 1, LAST = 2, DLAST = 3 };
enum { ACT = 0, GRAD = 1, OUT = 2 };

constexpr int TILES = 4;                    // accumulator tiles of 128 voxels per CTA
constexpr int EPI_WARPS = 16;
constexpr int LOAD_WARPS = 4;
constexpr int S = 3;                        // input slots

template<int SRC, int TXW>
struct Geo {
    static constexpr bool WIDE = SRC == MID || SRC == LAST;     // 24 channels with halo, else one built group
    // Between two tiles a warp waits and issues nothing for some 200 clocks; the
    // MMAs of another warp fill that in.  LAST, with 36 clocks per MMA, gains up
    // to four (clocks per plane with 1, 2, 4 warps: 3990, 2640, 2350); MID has
    // its tiles finish together with four and the epilogues then wait for each
    // other (4930, 3610, 3830).
    static constexpr int MMA_WARPS = SRC == LAST ? 4 : 2;
    static constexpr int LOAD0 = MMA_WARPS + EPI_WARPS;
    static constexpr int THREADS = 32 * (LOAD0 + LOAD_WARPS);
    static constexpr int TY = 512 / TXW;
    static constexpr int ROWS = TY + 2;
    static constexpr int NG = TXW / 8;
    static constexpr int VOX = WIDE ? 10 : 8;                   // voxels stored per group of 8
    static constexpr int GS = VOX * 16;                         // bytes of a group (SBO)
    static constexpr int ROWP = NG * GS;
    static constexpr int CGS = ROWS * ROWP;                     // channel-group stride
    static constexpr int SLOT = (WIDE ? 3 : 1) * CGS;
    static constexpr int KSTEPS = WIDE ? 14 : 2;
    static constexpr int N = SRC == LAST ? 16 : 80;
    static constexpr int KS_BYTES = SRC == LAST ? 2 * 2 * 128 : 2 * 16 * 128;     // B of one K-step
    static constexpr int W_BYTES = KSTEPS * KS_BYTES * (SRC == LAST ? 3 : 1);
    static constexpr int TCOLS = SRC == LAST ? 16 : 128;        // columns between tiles
    static constexpr int TMEM = SRC == LAST ? 64 : 512;
    static constexpr int SMEM = 128 + W_BYTES + S * SLOT;
};

struct Params {
    Shape s;
    int zchunk;
    const bf16 *in;             // MID, LAST: ghosted
    const float *f0, *f1;       // FIRST: u, kappa; DLAST: du, target
    float scale;                // DLAST: 2 / N
    const bf16 *w;              // packed weights
    const float *bias;          // ACT, OUT
    bf16 *out;                  // ACT, GRAD: ghosted
    float *g;                   // ACT: GELU' of the pre-activations out (or null); GRAD: in; FP32
                                // [batch][nz][ny][6][nx][4], four channels to a float4.  OUT: receives conv +
                                // bias (or null)
    float *db;                  // GRAD: bias gradient, added to
    float *fout;                // OUT
    int add;                    // OUT: add to fout
    int *err;
};

template<int SRC, int EPI, int TXW>
__global__ void __launch_bounds__((Geo<SRC, TXW>::THREADS), 1)
conv_tc_kernel(const Params p)
{
    typedef Geo<SRC, TXW> G;
    extern __shared__ unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t bar_w;
    __shared__ __align__(8) uint64_t bar_full[S];       // input plane in its slot (one arrive per loader warp)
    __shared__ __align__(8) uint64_t bar_empty[S];      // input slot no longer read (MMA commit)
    __shared__ __align__(8) uint64_t bar_mma[TILES];    // a plane's MMAs of the tile done
    __shared__ __align__(8) uint64_t bar_free[TILES];   // its completed accumulator read and started over
    __shared__ uint32_t s_tmem;
    __shared__ int s_fail;
    __shared__ int s_commits[TILES];                    // planes committed, by tile
    __shared__ float s_db[24];
    __shared__ __align__(16) float s_bias[24];
    volatile int *fail = &s_fail;

    unsigned char *smem = smem_raw + ((128 - (saddr(smem_raw) & 127)) & 127);
    unsigned char *wsm = smem;
    unsigned char *ring = smem + G::W_BYTES;

    const Shape s = p.s;
    const int tid = threadIdx.x;
    const int warp = tid >> 5;
    const int lane = tid & 31;
    const int x0 = blockIdx.x * TXW;
    const int y0 = blockIdx.y * G::TY;
    const int zsplit = (s.nz + p.zchunk - 1) / p.zchunk;
    const int b = blockIdx.z / zsplit;
    const int z0 = (blockIdx.z % zsplit) * p.zchunk;
    const int n = min(z0 + p.zchunk, s.nz) - z0;        // output planes j = 0 .. n - 1; input planes q = 0 .. n + 1

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(saddr(&s_tmem)),
                     "r"(G::TMEM)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        s_fail = 0;
        mbar_init(saddr(&bar_w), 1);
        for (int i = 0; i < S; ++i) {
            mbar_init(saddr(&bar_full[i]), LOAD_WARPS);
            mbar_init(saddr(&bar_empty[i]), G::MMA_WARPS);
        }
        for (int i = 0; i < TILES; ++i) {
            mbar_init(saddr(&bar_mma[i]), 1);
            mbar_init(saddr(&bar_free[i]), 4);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (EPI == GRAD && tid < 24) s_db[tid] = 0.f;
    dependent_start();
    if (EPI == ACT && tid < 24) s_bias[tid] = __ldg(p.bias + tid);
    if (tid == 0) {
        mbar_expect_tx(saddr(&bar_w), G::W_BYTES);
        bulk_copy(saddr(wsm), p.w, G::W_BYTES, saddr(&bar_w));
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = s_tmem;

    if (warp < G::MMA_WARPS) {
        constexpr int OWN = TILES / G::MMA_WARPS;          // tiles of this warp
        int commits = 0;
        bool ok = __all_sync(0xffffffffu, mbar_wait(saddr(&bar_w), 0, fail));
        const uint32_t rbase = saddr(ring), wbase = saddr(wsm);
        constexpr uint32_t ID = idesc(128, G::N, false);
        constexpr uint32_t HI_A = desc_hi(G::GS), HI_B = desc_hi(128);
        for (int q = 0; ok && q < n + 2; ++q) {
            ok = __all_sync(0xffffffffu, mbar_wait(saddr(&bar_full[q % S]), (uint32_t)((q / S) & 1), fail));
            if (!ok) break;
            fence_after();
            const uint32_t a0 = desc_lo(rbase + (uint32_t)((q % S) * G::SLOT), 0);
            // the block order of the three accumulators (see pack_kernel)
            const uint32_t rot = (uint32_t)((3 - q % 3) % 3);
            const uint32_t b0 = SRC == LAST ? desc_lo(wbase + rot * (G::KSTEPS * G::KS_BYTES), 2 * 128)
                                            : desc_lo(wbase + rot * 3 * 128, 16 * 128);
            for (int m = warp * OWN; m < warp * OWN + OWN; ++m) {
                ok = __all_sync(0xffffffffu, mbar_wait(saddr(&bar_free[m]), (uint32_t)(q & 1), fail));
                if (!ok) break;
                fence_after();
                if (elect_one()) {
                    const uint32_t d = tmem + (uint32_t)(m * G::TCOLS);
                    const uint32_t am = a0 + (uint32_t)(m * G::GS);         // 16 groups, in 16-byte units
#pragma unroll
                    for (int k = 0; k < G::KSTEPS; ++k) {
                        int first, lead;                // start and leading offset of the step's two groups, bytes
                        if (G::WIDE) {
                            if (k < 12) {               // taps 2 (k / 3) and 2 (k / 3) + 1, channel group k % 3
                                const int ta = 2 * (k / 3), tb = ta + 1;
                                const int oa = (ta / 3) * G::ROWP + (ta % 3) * 16;
                                const int ob = (tb / 3) * G::ROWP + (tb % 3) * 16;
                                first = oa + (k % 3) * G::CGS;
                                lead = ob - oa;
                            } else {                    // tap 8: groups 0, 1 and 1 (zero weights), 2
                                first = 2 * G::ROWP + 2 * 16 + (k - 12) * G::CGS;
                                lead = G::CGS;
                            }
                        } else {                        // rows 0, 1 and 1 (zero weights), 2
                            first = k * G::ROWP;
                            lead = G::ROWP;
                        }
                        mma<true>(d, desc(am + (uint32_t)((first >> 4) + ((lead >> 4) << 16)), HI_A),
                                  desc(b0 + (uint32_t)((k * G::KS_BYTES) >> 4), HI_B), ID);
                    }
                    mma_commit(saddr(&bar_mma[m]));
                    if (m == warp * OWN + OWN - 1) mma_commit(saddr(&bar_empty[q % S]));
                }
                __syncwarp();
                ++commits;
            }
        }
        if (lane == 0) {
            for (int i = 0; i < OWN; ++i) s_commits[warp * OWN + i] = (commits + OWN - 1 - i) / OWN;
            if (!ok) s_fail = 1;
        }
        __syncwarp();
    } else if (warp >= G::LOAD0) {
        const int lt = tid - G::LOAD0 * 32;
        int published = 0;
        bool ok = true;
        auto publish = [&](int upto) {
            fence_async_proxy();
            __syncwarp();
            for (; published < upto; ++published) {
                if (lane == 0) mbar_arrive(saddr(&bar_full[published % S]));
            }
        };
        // What a thread copies lies at the same place of every plane.
        // Wide: its 16-byte voxels of the slot; else its warp's segments of 32
        // voxels, all at the same x (LOAD_WARPS * 32 is a multiple of TXW).
        constexpr int PER_ROW = G::NG * 10;
        constexpr int SEGS = G::ROWS * TXW / 32;
        constexpr int PER = G::WIDE ? (G::ROWS * PER_ROW + LOAD_WARPS * 32 - 1) / (LOAD_WARPS * 32)
                                    : (SEGS + LOAD_WARPS - 1) / LOAD_WARPS;
        const long long plane = G::WIDE ? (long long)(s.ny + 2) * 3 * (s.nx + 2) : (long long)s.ny * s.nx;
        uint32_t src[PER];                                  // in 16-byte units / floats of a plane (a plane of
                                                            // 2^32 would not fit the device's memory)
        uint32_t dst[G::WIDE ? PER : 1];
        int side = 0;                                       // to the neighbour beyond the segment's end
        if (G::WIDE) {
#pragma unroll
            for (int i = 0; i < PER; ++i) {
                const int v = lt + i * LOAD_WARPS * 32;
                const int row = v / PER_ROW;
                const int j = v - row * PER_ROW;            // group j / 10, voxel j % 10 of it
                const int gy = min(y0 + row, s.ny + 1);     // ghosted row (rows past the grid: any)
                src[i] = (uint32_t)gy * 3u * (uint32_t)(s.nx + 2) + (uint32_t)(x0 + (j / 10) * 8 + j % 10);
                dst[i] = (uint32_t)(row * G::ROWP + j * 16);
            }
        } else {
            const int x = x0 + (lt & ~31) % TXW + lane;
            side = lane == 0 ? (x == 0 ? s.nx - 1 : -1) : (x == s.nx - 1 ? 1 - s.nx : 1);
#pragma unroll
            for (int i = 0; i < PER; ++i) {
                const int seg = (lt >> 5) + i * LOAD_WARPS;
                int y = y0 - 1 + min(seg * 32 / TXW, G::ROWS - 1);
                y = y < 0 ? y + s.ny : (y >= s.ny ? (y - s.ny) % s.ny : y);
                src[i] = (uint32_t)y * (uint32_t)s.nx + (uint32_t)x;
            }
        }
        constexpr int PERF = G::WIDE ? 1 : PER;
        float na[PERF], nc[PERF], ma[PERF], mc[PERF];       // FIRST, DLAST: the next plane's fields
        auto load = [&](int q) {
            int z = z0 - 1 + q;
            z = z < 0 ? z + s.nz : (z >= s.nz ? z - s.nz : z);
            const float *f0 = p.f0 + ((long long)b * s.nz + z) * plane;
            const float *f1 = p.f1 + ((long long)b * s.nz + z) * plane;
#pragma unroll
            for (int i = 0; i < PERF; ++i) {
                na[i] = f0[src[i]];
                nc[i] = f1[src[i]];
                ma[i] = mc[i] = 0.f;
                if (lane == 0 || lane == 31) {
                    ma[i] = f0[src[i] + side];
                    mc[i] = f1[src[i] + side];
                }
            }
        };
        if (!G::WIDE) load(0);
        for (int q = 0; q < n + 2; ++q) {
            // publish what has landed before waiting for a slot: the MMAs that
            // free it never wait on this loader
            if (G::WIDE && q >= 2) {
                asm volatile("cp.async.wait_group 1;" ::: "memory");
                publish(q - 1);
            }
            if (q >= S) {
                const bool got = mbar_wait(saddr(&bar_empty[q % S]), (uint32_t)(((q - S) / S) & 1), fail);
                if (!__all_sync(0xffffffffu, got)) {
                    ok = false;
                    break;
                }
            }
            const uint32_t slot = saddr(ring) + (uint32_t)((q % S) * G::SLOT);
            if (G::WIDE) {
                const uint4 *in = reinterpret_cast<const uint4 *>(p.in) + ((long long)b * (s.nz + 2) + z0 + q) * plane;
#pragma unroll
                for (int i = 0; i < PER; ++i) {
                    if ((i + 1) * LOAD_WARPS * 32 <= G::ROWS * PER_ROW || lt + i * LOAD_WARPS * 32 < G::ROWS * PER_ROW) {
#pragma unroll
                        for (int c = 0; c < 3; ++c) copy16(slot + dst[i] + c * G::CGS, in + src[i] + c * (s.nx + 2));
                    }
                }
                asm volatile("cp.async.commit_group;" ::: "memory");
            } else {
                float va[PERF], vc[PERF], ea[PERF], ec[PERF];
                // a warp builds the groups of 32 consecutive voxels: neighbours
                // by shuffle, the two beyond the ends by the end lanes; the
                // loads of all its segments and of the next plane are in flight
                // together
#pragma unroll
                for (int i = 0; i < PERF; ++i) {
                    va[i] = na[i];
                    vc[i] = nc[i];
                    ea[i] = ma[i];
                    ec[i] = mc[i];
                }
                if (q < n + 1) load(q + 1);
#pragma unroll
                for (int i = 0; i < PERF; ++i) {
                    const int seg = (lt >> 5) + i * LOAD_WARPS;
                    uint32_t mid, edge;                 // FIRST: the pair (u, kappa); DLAST: the gradient
                    if (SRC == FIRST) {
                        mid = pack_bf16(va[i], vc[i]);
                        edge = pack_bf16(ea[i], ec[i]);
                    } else {
                        mid = pack_bf16(p.scale * (va[i] - vc[i]), 0.f);
                        edge = pack_bf16(p.scale * (ea[i] - ec[i]), 0.f);
                    }
                    uint32_t w = __shfl_up_sync(0xffffffffu, mid, 1);
                    uint32_t e = __shfl_down_sync(0xffffffffu, mid, 1);
                    if (lane == 0) w = edge;
                    if (lane == 31) e = edge;
                    const uint4 g = SRC == FIRST ? make_uint4(w, mid, e, 0u) : make_uint4(w | (mid << 16), e, 0u, 0u);
                    if (SEGS % LOAD_WARPS == 0 || seg < SEGS) {
                        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(slot + (uint32_t)((seg * 32 + lane) * 16)),
                                     "r"(g.x), "r"(g.y), "r"(g.z), "r"(g.w)
                                     : "memory");
                    }
                }
                publish(q + 1);
            }
        }
        if (G::WIDE) asm volatile("cp.async.wait_all;" ::: "memory");
        if (ok) publish(n + 2);
        else if (lane == 0) s_fail = 1;
    } else {
        const int m = (warp - G::MMA_WARPS) >> 2;                  // tile
        const int qd = warp & 3;                        // lane quarter this warp may read
        const int vt = m * 128 + qd * 32 + lane;        // voxel of the CTA's 512
        const int x = x0 + vt % TXW;
        const int y = y0 + vt / TXW;
        const bool live = y < s.ny;
        const uint32_t acc = tmem + ((uint32_t)(qd * 32) << 16) + (uint32_t)(m * G::TCOLS);
        // this voxel in plane 0 of the ghosted output (16-byte units) and of
        // GELU' (float4), and whether an axis repeats it among the ghosts
        const long long oplane = (long long)(s.ny + 2) * 3 * (s.nx + 2);
        uint4 *const out0 = reinterpret_cast<uint4 *>(p.out) + b * (s.nz + 2) * oplane + (y + 1) * 3 * (s.nx + 2LL) + x + 1;
        const long long gplane = (long long)s.ny * 6 * s.nx;
        float4 *const g0 = reinterpret_cast<float4 *>(p.g) + (long long)b * s.nz * gplane + y * 6LL * s.nx + x;
        const bool edge_x = x == 0 || x == s.nx - 1, edge_y = y == 0 || y == s.ny - 1;
        const int ghost_x = x == 0 ? s.nx : -s.nx;          // where its copy lies (nx >= 32: only one)
        float db[EPI == GRAD ? 24 : 1] = {};
        const float b1 = EPI == OUT ? __ldg(p.bias) : 0.f;
        // accumulator slot (columns) j % 3 starts at the bias (OUT adds it at the end)
        auto restart = [&](int slot) {
            if constexpr (EPI == OUT) {
                tmem_st1(acc + (uint32_t)slot, 0.f);
            } else {
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    float v[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i) v[i] = EPI == ACT ? s_bias[c * 8 + i] : 0.f;
                    tmem_st8(acc + (uint32_t)(slot * 24 + c * 8), v);
                }
            }
            tmem_st_wait();
            fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(saddr(&bar_free[m]));
        };
        restart(0);
        // What the epilogue reads of a plane is loaded while its MMAs run.  In MID,
        // where the MMAs set the pace, GELU' is not: multiplying before the
        // accumulator is handed back costs more (101 -> 107 us at 64^3 x 8; DLAST
        // 117 -> 97), and after it the registers do not suffice.
        constexpr bool AHEAD = SRC == DLAST;
        float *const fout0 = p.fout + ((long long)b * s.nz * s.ny + y) * s.nx + x;
        const long long fplane = (long long)s.ny * s.nx;
        float before = 0.f;
        float4 g[AHEAD ? 6 : 1];
        if (AHEAD && live) {
#pragma unroll
            for (int c = 0; c < 6; ++c) g[AHEAD ? c : 0] = g0[z0 * gplane + c * s.nx];
        }
        for (int q = 0; q < n + 2; ++q) {
            if (EPI == OUT && p.add && q >= 2 && live) before = fout0[(z0 + q - 2) * fplane];
            const bool ok = mbar_wait(saddr(&bar_mma[m]), (uint32_t)(q & 1), fail);
            if (!__all_sync(0xffffffffu, ok)) {
                if (lane == 0) s_fail = 1;
                break;
            }
            fence_after();
            const int slot = (q + 1) % 3;               // output q - 2 is complete, q + 1 takes its place
            const int z = z0 + q - 2;
            if constexpr (EPI == OUT) {
                const float v = tmem_ld1(acc + (uint32_t)slot);
                restart(slot);
                if (q >= 2 && live) {
                    float *o = fout0 + z * fplane;
                    const float d = v + b1;
                    *o = p.add ? before + d : d;
                    if (p.g) p.g[o - p.fout] = d;
                }
            } else {
                uint4 w[3];
                if constexpr (AHEAD) {
                    const bool use = q >= 2 && live;
                    const float zero[8] = {};
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        float v[8];
                        tmem_ld8(acc + (uint32_t)(slot * 24 + c * 8), v);
                        tmem_st8(acc + (uint32_t)(slot * 24 + c * 8), zero);
                        if (use) {
#pragma unroll
                            for (int i = 0; i < 2; ++i) {
                                const float4 t = g[2 * c + i];
                                v[4 * i] *= t.x;
                                v[4 * i + 1] *= t.y;
                                v[4 * i + 2] *= t.z;
                                v[4 * i + 3] *= t.w;
                                if (q + 1 < n + 2) g[2 * c + i] = g0[(z + 1) * gplane + (2 * c + i) * s.nx];
                            }
#pragma unroll
                            for (int i = 0; i < 8; ++i) db[c * 8 + i] += v[i];
                            w[c] = make_uint4(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]), pack_bf16(v[4], v[5]),
                                              pack_bf16(v[6], v[7]));
                        }
                    }
                    tmem_st_wait();
                    fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(saddr(&bar_free[m]));
                    if (!use) continue;
                } else {
                    float v[24];
                    tmem_ld24(acc + (uint32_t)(slot * 24), v);
                    restart(slot);
                    if (q < 2 || !live) continue;
                    if constexpr (EPI == GRAD) {
                        const float4 *gp = g0 + z * gplane;
#pragma unroll
                        for (int c = 0; c < 6; ++c) {
                            const float4 t = gp[c * s.nx];
                            v[4 * c] *= t.x;
                            v[4 * c + 1] *= t.y;
                            v[4 * c + 2] *= t.z;
                            v[4 * c + 3] *= t.w;
                        }
#pragma unroll
                        for (int c = 0; c < 24; ++c) db[c] += v[c];
                    } else if (p.g) {
                        // training: GELU' for the backward pass, beside GELU
                        float4 *gp = g0 + z * gplane;
#pragma unroll
                        for (int c = 0; c < 6; ++c) {
                            float2 h0, h1, d0, d1;
                            gelu_pair<true>(make_float2(v[4 * c], v[4 * c + 1]), h0, d0);
                            gelu_pair<true>(make_float2(v[4 * c + 2], v[4 * c + 3]), h1, d1);
                            gp[c * s.nx] = make_float4(d0.x, d0.y, d1.x, d1.y);
                            v[4 * c] = h0.x;
                            v[4 * c + 1] = h0.y;
                            v[4 * c + 2] = h1.x;
                            v[4 * c + 3] = h1.y;
                        }
                    } else {
#pragma unroll
                        for (int c = 0; c < 12; ++c) {
                            float2 h, d;
                            gelu_pair<false>(make_float2(v[2 * c], v[2 * c + 1]), h, d);
                            v[2 * c] = h.x;
                            v[2 * c + 1] = h.y;
                        }
                    }
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        w[c] = make_uint4(pack_bf16(v[8 * c], v[8 * c + 1]), pack_bf16(v[8 * c + 2], v[8 * c + 3]),
                                          pack_bf16(v[8 * c + 4], v[8 * c + 5]), pack_bf16(v[8 * c + 6], v[8 * c + 7]));
                    }
                }
                // the voxel and its ghost copies
                auto put = [&](uint4 *o) {
                    o[0] = w[0];
                    o[s.nx + 2] = w[1];
                    o[2 * (s.nx + 2)] = w[2];
                };
                auto put_x = [&](uint4 *o) {
                    put(o);
                    if (edge_x) put(o + ghost_x);
                };
                if (!edge_y && z != 0 && z != s.nz - 1) {
                    put_x(out0 + (z + 1) * oplane);
                } else {
                    // in z and y: itself, the far ghost, the near ghost (an axis of extent 1 has both)
#pragma unroll 1
                    for (int i = 0; i < 9; ++i) {
                        const int iz = i / 3, iy = i - 3 * iz;
                        if ((iz == 1 && z != 0) || (iz == 2 && z != s.nz - 1) || (iy == 1 && y != 0) ||
                            (iy == 2 && y != s.ny - 1)) {
                            continue;
                        }
                        put_x(out0 + (iz == 0 ? z + 1 : (iz == 1 ? s.nz + 1 : 0)) * oplane +
                              (iy == 0 ? 0 : (iy == 1 ? s.ny : -s.ny)) * 3LL * (s.nx + 2));
                    }
                }
            }
        }
        if constexpr (EPI == GRAD) {
#pragma unroll
            for (int c = 0; c < 24; ++c) {
                float t = db[c];
                for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
                if (lane == 0) atomicAdd(&s_db[c], t);
            }
        }
    }

    fence_before();
    __syncthreads();            // every role has left its loop; no copy is in flight
    fence_after();
    if (EPI == GRAD && tid < 24) atomicAdd(p.db + tid, s_db[tid]);
    if (s_fail) {
        // report, then wait (bounded) for the MMAs and the weight copy
        if (tid == 0) {
            atomicExch(p.err, 1);
            for (int m = 0; m < TILES; ++m) {
                if (s_commits[m] > 0) mbar_wait(saddr(&bar_mma[m]), (uint32_t)((s_commits[m] - 1) & 1), nullptr);
            }
            mbar_wait(saddr(&bar_w), 0, nullptr);
        }
        fence_before();
        __syncthreads();
        fence_after();
    }
    if (warp == 0) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(G::TMEM) : "memory");
    }
}

// Weights of one convolution as the MMA's B operand, K-major without swizzle:
// [K-step][group 0, 1][N group of 8][8 columns][8 k].  Columns: blocks of 24
// output channels in the z-tap order 0, 2, 1, 0, 2 (and 8 zeros); at input
// plane q the accumulators 0, 1, 2 take taps (q - s) mod 3, which is the
// window of three blocks that starts at block (3 - q % 3) % 3.  LAST has one
// output channel: columns 0, 1, 2 are the accumulators, one copy per rotation.
// W: FP32 [tap][cin][cout]; mirror: the input-gradient convolution (taps
// mirrored, channel roles swapped).
struct PackJobs {               // by blockIdx.y
    struct Job {
        const float *w;
        bf16 *out;
        int src, mirror;
    } job[7];
};

__global__ void pack_kernel(const PackJobs jobs)
{
    const PackJobs::Job& job = jobs.job[blockIdx.y];
    const float *w = job.w;
    bf16 *out = job.out;
    const int src = job.src, mirror = job.mirror;
    const int ksteps = src == MID || src == LAST ? 14 : 2;
    const int ng = src == LAST ? 2 : 16;
    const int copies = src == LAST ? 3 : 1;
    const int total = copies * ksteps * 2 * ng * 64;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
        const int k8 = i & 7;
        const int col = ((i >> 6) % ng) * 8 + ((i >> 3) & 7);
        const int half = (i / (64 * ng)) & 1;
        const int ks = (i / (128 * ng)) % ksteps;
        const int rot = i / (128 * ng * ksteps);
        int dz = -1, co = 0;
        if (src == LAST) {
            if (col < 3) {
                const int order[5] = {0, 2, 1, 0, 2};
                dz = order[rot + col];
            }
        } else if (col < 120) {
            const int order[5] = {0, 2, 1, 0, 2};
            dz = order[col / 24];
            co = col % 24;
        }
        int tap = -1, ci = 0;                       // tap in (y, x), input channel
        if (src == MID || src == LAST) {
            if (ks < 12) {
                tap = 2 * (ks / 3) + half;
                ci = (ks % 3) * 8 + k8;
            } else if (!(ks == 13 && half == 0)) {
                tap = 8;
                ci = (ks - 12 + half) * 8 + k8;
            }
        } else {
            const int dy = ks + half;               // ks 1, half 0 repeats row 1 with zero weights
            if (!(ks == 1 && half == 0)) {
                if (src == FIRST && k8 < 6) {
                    tap = dy * 3 + k8 / 2;
                    ci = k8 & 1;
                } else if (src == DLAST && k8 < 3) {
                    tap = dy * 3 + k8;
                }
            }
        }
        float v = 0.f;
        if (dz >= 0 && tap >= 0) {
            const int t = dz * 9 + tap;
            if (src == MID) v = mirror ? w[((26 - t) * 24 + co) * 24 + ci] : w[(t * 24 + ci) * 24 + co];
            else if (src == LAST) v = w[t * 24 + ci];
            else if (src == FIRST) v = w[(t * 2 + ci) * 24 + co];
            else v = w[(26 - t) * 24 + co];
        }
        out[i] = __float2bfloat16(v);
    }
}

template<int SRC, int EPI, int TXW>
static void run(Params p, cudaStream_t stream)
{
    typedef Geo<SRC, TXW> G;
    static PerDevice<int> setup;
    const int sms = setup.get([] {
        auto *fn = conv_tc_kernel<SRC, EPI, TXW>;
        LGD_CHECK_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, G::SMEM));
        int dev = 0, count = 0;
        LGD_CHECK_CUDA(cudaGetDevice(&dev));
        LGD_CHECK_CUDA(cudaDeviceGetAttribute(&count, cudaDevAttrMultiProcessorCount, dev));
        return count;
    });
    const int bx = p.s.nx / TXW, by = (p.s.ny + G::TY - 1) / G::TY;
    // one CTA per SM; of its planes two are halo, and about two planes' time to start and to drain
    p.zchunk = least_planes((long long)bx * by * p.s.batch, p.s.nz, sms, 4, nullptr);
    const int zsplit = (p.s.nz + p.zchunk - 1) / p.zchunk;
    launch_dependent(conv_tc_kernel<SRC, EPI, TXW>, dim3(bx, by, p.s.batch * zsplit), G::THREADS, G::SMEM, stream, p);
    check_launch("tensor-core convolution");
}

template<int SRC, int EPI>
static void run_any(const Params& p, cudaStream_t stream)
{
    if (p.s.nx % 128 == 0) run<SRC, EPI, 128>(p, stream);
    else if (p.s.nx % 64 == 0) run<SRC, EPI, 64>(p, stream);
    else run<SRC, EPI, 32>(p, stream);
}

}  // namespace tc

using namespace tc;

bool tc_applicable(int nx, int ny, int channels)
{
    return channels == 24 && nx % 32 == 0 && ny >= 1;
}

static const size_t PACKED = 14 * 2 * 16 * 64;      // elements of the largest packed operand

TcWeights tc_alloc_weights(bool training)
{
    TcWeights w = {};
    bf16 *base = nullptr;
    LGD_CHECK_CUDA(cudaMalloc(&base, (training ? 7 : 4) * PACKED * sizeof(bf16)));
    w.base = base;
    for (int l = 0; l < 4; ++l) w.fwd[l] = base + l * PACKED;
    if (training) {
        for (int l = 1; l < 4; ++l) w.grad[l] = base + (3 + l) * PACKED;
    }
    return w;
}

void tc_free_weights(TcWeights& w) { cudaFree(w.base); }

void tc_pack_weights(const float *const layer[4], const TcWeights& w, cudaStream_t stream)
{
    const int src[4] = {FIRST, MID, MID, LAST};
    const int gsrc[4] = {0, MID, MID, DLAST};
    PackJobs jobs;
    int n = 0;
    for (int l = 0; l < 4; ++l) jobs.job[n++] = {layer[l], (bf16 *)w.fwd[l], src[l], 0};
    for (int l = 1; l < 4 && w.grad[1]; ++l) jobs.job[n++] = {layer[l], (bf16 *)w.grad[l], gsrc[l], 1};
    pack_kernel<<<dim3(56, n), 256, 0, stream>>>(jobs);
    check_launch("pack tensor-core weights");
}

size_t tc_ghost_bytes(int nx, int ny, int nz, int batch)
{
    return (size_t)batch * (nz + 2) * (ny + 2) * 3 * (nx + 2) * 16;
}

void tc_layer1(const float *u, const float *k, const void *w, const float *bias, void *out, float *gelu_grad, const int dims[4],
               int *err, cudaStream_t stream)
{
    Params p = {};
    p.s = {dims[0], dims[1], dims[2], dims[3]};
    p.f0 = u;
    p.f1 = k;
    p.w = (const bf16 *)w;
    p.bias = bias;
    p.out = (bf16 *)out;
    p.g = gelu_grad;
    p.err = err;
    run_any<FIRST, ACT>(p, stream);
}

void tc_layer_mid(const void *in, const void *w, const float *bias, void *out, float *gelu_grad, const int dims[4], int *err,
                  cudaStream_t stream)
{
    Params p = {};
    p.s = {dims[0], dims[1], dims[2], dims[3]};
    p.in = (const bf16 *)in;
    p.w = (const bf16 *)w;
    p.bias = bias;
    p.out = (bf16 *)out;
    p.g = gelu_grad;
    p.err = err;
    run_any<MID, ACT>(p, stream);
}

void tc_layer_last(const void *in, const void *w, const float *bias, float *out, bool add, float *copy, const int dims[4],
                   int *err, cudaStream_t stream)
{
    Params p = {};
    p.s = {dims[0], dims[1], dims[2], dims[3]};
    p.in = (const bf16 *)in;
    p.w = (const bf16 *)w;
    p.bias = bias;
    p.fout = out;
    p.g = copy;
    p.add = add ? 1 : 0;
    p.err = err;
    run_any<LAST, OUT>(p, stream);
}

void tc_grad_mid(const void *dz, const void *w, const float *gelu_grad, void *out, float *db, const int dims[4], int *err,
                 cudaStream_t stream)
{
    Params p = {};
    p.s = {dims[0], dims[1], dims[2], dims[3]};
    p.in = (const bf16 *)dz;
    p.w = (const bf16 *)w;
    p.g = const_cast<float *>(gelu_grad);
    p.out = (bf16 *)out;
    p.db = db;
    p.err = err;
    run_any<MID, GRAD>(p, stream);
}

void tc_grad_last(const float *du, const float *target, float scale, const void *w, const float *gelu_grad, void *out, float *db,
                  const int dims[4], int *err, cudaStream_t stream)
{
    Params p = {};
    p.s = {dims[0], dims[1], dims[2], dims[3]};
    p.f0 = du;
    p.f1 = target;
    p.scale = scale;
    p.w = (const bf16 *)w;
    p.g = const_cast<float *>(gelu_grad);
    p.out = (bf16 *)out;
    p.db = db;
    p.err = err;
    run_any<DLAST, GRAD>(p, stream);
}

}  // namespace sur
}  // namespace lgd
