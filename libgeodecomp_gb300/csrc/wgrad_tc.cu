// Weight gradients of the surrogate's 3^3 convolutions (C = 24) on the
// fifth-generation tensor cores: dW[tap][ci][co] = sum over the voxels v of
// h[v + tap][ci] * dz[v][co], a contraction over the voxels.
//
// Operands lie in shared memory with the channels contiguous (16 bytes = 8
// channels of a voxel, voxels 16 bytes apart), which is the tensor core's
// MN-major form with K = voxels: a unit of eight M or N elements per (row,
// channel group), all units a constant stride apart.  Per MMA (K = 16 voxels):
//   CC (layers 2, 3)  M = 16 units = five rows of h and a third (120 of the
//                     128 rows of D used), N = two rows of dz, each three
//                     times, moved by the taps in x (144): the pairs (row of h,
//                     row of dz) with h at most one row away give the taps in
//                     y, so that one MMA serves nine taps.  Three accumulators,
//                     the taps in z.  An MMA reads 4 KB of h and 32 N bytes of
//                     dz at 128 B per clock and multiplies in N / 2 clocks: 72
//                     either way.  One MMA per tap in x (N = 48) took 46 each,
//                     138 for the three;
//   L (layer 4)       the same h against two rows of the loss gradient, its
//                     three x neighbours in one unit: N = 16, three
//                     accumulators;
//   F (layer 1)       M = 16 rows of x0 (u, kappa of the three x neighbours in
//                     one unit) against four rows of dz: N = 96, three
//                     accumulators.
// The accumulators (FP32, tensor memory) stay for all of a CTA's voxels; at
// the end it folds them into one dW and writes that to its own slice of a
// buffer, which reduce_kernel adds up in a fixed order.  The mma.sync kernel
// before took its operands from shared memory two bytes at a time and added
// every tile's dW to the gradient with atomics.
//
// CTAs are persistent over (column of TXW x TY voxels, z chunk) items and
// march each in z: a dz plane meets three h planes (five slots of h, three of
// dz, so that two planes are on their way: with one the copies' latency set the
// pace).  FL and LL build a field's groups from registers loaded a plane ahead.
// At 64^3 x 8: CC 73 us (127 with one MMA per tap in x and one plane ahead), FL
// 37 (87), LL 51 (69).  Three warps issue the MMAs, four clear the accumulators
// first and fold them at the end, eight fill the slots.  Waits are bounded as in
// conv_tc.cu.
#include <algorithm>

#include "lgd_internal.h"
#include "tc_common.cuh"
#include "conv_tc.h"
#include "z_chunks.h"

namespace lgd {
namespace sur {
namespace tc {

enum { CC = 0, FL = 1, LL = 2 };            // layers 2 and 3; first; last

constexpr int WG_LOADERS = 8;
constexpr int WG_MMA = 3;                   // one per tap in z: the MMAs of one fill the waits of the others
constexpr int WG_LOAD0 = WG_MMA + 4;
constexpr int WG_THREADS = 32 * (WG_LOAD0 + WG_LOADERS);
constexpr int SH = 5, SD = 3;               // slots of h (three in use) and dz (one): two planes ahead

template<int MODE, int TXW>
struct WGeo {
    static constexpr int TY = (MODE == CC ? 256 : 512) / TXW;   // CC: three slots of dz, three times each, take 110 KB
    static constexpr int ROWS = TY + 2;
    static constexpr int NG = TXW / 8;
    static constexpr int GS = 128;                              // bytes of an 8-voxel group
    static constexpr int UA = NG * GS;                          // M unit stride
    static constexpr int UPR = MODE == FL ? 1 : 3;              // M units per row
    static constexpr int HSLOT = ROWS * UPR * UA;
    static constexpr int UB = TXW * 16;                         // N unit stride
    static constexpr int NPR = MODE == LL ? 1 : (MODE == FL ? 3 : 9);   // N units per row
    static constexpr int DSLOT = TY * NPR * UB;
    static constexpr int YB = MODE == FL ? 4 : 2;               // dz rows per MMA
    static constexpr int N = YB * NPR * 8;                      // 144, 96, 16
    static constexpr int TMEM = MODE == CC ? 512 : (MODE == FL ? 512 : 64);
    static constexpr int CIN = MODE == FL ? 2 : 24;
    static constexpr int COUT = MODE == LL ? 1 : 24;
    static constexpr int OUT = 27 * CIN * COUT;
    static constexpr int RING = SH * HSLOT + SD * DSLOT;
    // M always spans 16 units: the last MMA of a slot reads past it
    static constexpr int REACH = SH * HSLOT + 16 * UA;
    static constexpr int USED = RING > REACH ? RING : REACH;
    static constexpr int SMEM = 128 + (USED > OUT * 4 ? USED : OUT * 4);
};

struct WParams {
    Shape s;
    int zchunk, items;
    const bf16 *h;              // CC, LL: ghosted activations
    const uint32_t *x0;         // FL: BF16 pairs (u, kappa) [batch][nz][ny][nx]
    const bf16 *dz;             // CC, FL: ghosted
    const float *du, *target;   // LL
    float scale;                // LL: 2 / N
    double *loss;               // LL: the sum of (du - target)^2, added to
    float *db;                  // LL: the bias gradient, added to
    float *part;                // [gridDim.x][OUT]
    int *err;
};

__device__ __forceinline__ void copy16_or_zero(uint32_t dst, const void *src, bool copy)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(copy ? 16 : 0) : "memory");
}

__device__ __forceinline__ void st_shared16(uint32_t dst, uint4 v)
{
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}

template<int MODE, int TXW>
__global__ void __launch_bounds__(WG_THREADS, 1)
wgrad_tc_kernel(const WParams p)
{
    typedef WGeo<MODE, TXW> G;
    extern __shared__ unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t bar_full[SH];      // h plane q and dz plane q - 2 there (one arrive per loader warp)
    __shared__ __align__(8) uint64_t bar_empty[SH];     // h slot no longer read
    __shared__ __align__(8) uint64_t bar_dempty[SD];    // dz slot no longer read
    __shared__ __align__(8) uint64_t bar_clear;         // accumulators cleared
    __shared__ __align__(8) uint64_t bar_done;          // all MMAs done
    __shared__ uint32_t s_tmem;
    __shared__ int s_fail;
    __shared__ int s_bad;       // the fold gave up (set by its own warps only, so that they agree)
    volatile int *fail = &s_fail;

    unsigned char *smem = smem_raw + ((128 - (saddr(smem_raw) & 127)) & 127);
    const uint32_t hring = saddr(smem);
    const uint32_t dring = hring + SH * G::HSLOT;

    const Shape s = p.s;
    const int tid = threadIdx.x;
    const int warp = tid >> 5;
    const int lane = tid & 31;
    const int bx = s.nx / TXW, by = (s.ny + G::TY - 1) / G::TY;
    const int zsplit = (s.nz + p.zchunk - 1) / p.zchunk;

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(saddr(&s_tmem)),
                     "r"(G::TMEM)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        s_fail = 0;
        s_bad = 0;
        for (int i = 0; i < SH; ++i) {
            mbar_init(saddr(&bar_full[i]), WG_LOADERS);
            mbar_init(saddr(&bar_empty[i]), WG_MMA);
        }
        for (int i = 0; i < SD; ++i) mbar_init(saddr(&bar_dempty[i]), WG_MMA);
        mbar_init(saddr(&bar_clear), 4);
        mbar_init(saddr(&bar_done), WG_MMA);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    dependent_start();
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = s_tmem;

    // item -> column and z range; the same walk in every role
    struct Item {
        int x0, y0, b, z0, n;
    };
    auto item_of = [&](int it) {
        Item t;
        const int col = it / zsplit;
        t.x0 = col % bx * TXW;
        t.y0 = col / bx % by * G::TY;
        t.b = col / (bx * by);
        t.z0 = it % zsplit * p.zchunk;
        t.n = min(t.z0 + p.zchunk, s.nz) - t.z0;
        return t;
    };

    if (warp < WG_MMA) {
        const int dz = warp;        // tap in z
        bool ok = __all_sync(0xffffffffu, mbar_wait(saddr(&bar_clear), 0, fail));
        fence_after();
        constexpr uint32_t ID = idesc(128, G::N, true);
        constexpr uint32_t HI_A = desc_hi(G::UA), HI_B = desc_hi(G::UB);
        int plane = 0;              // h planes so far
        int dplane = 0;             // dz planes so far
        for (int it = blockIdx.x; ok && it < p.items; it += gridDim.x) {
            const Item t = item_of(it);
            for (int q = 0; q < t.n + 2; ++q, ++plane) {
                ok = __all_sync(0xffffffffu, mbar_wait(saddr(&bar_full[plane % SH]), (uint32_t)((plane / SH) & 1), fail));
                if (!ok) break;
                if (q < 2) continue;
                fence_after();
                // dz plane q - 2 against h planes q - 2, q - 1, q
                const uint32_t a0 = desc_lo(hring + (uint32_t)(((plane - 2 + dz) % SH) * G::HSLOT), G::GS);
                const uint32_t b0 = desc_lo(dring + (uint32_t)((dplane % SD) * G::DSLOT), 128);
                const uint32_t d = tmem + (uint32_t)(dz * G::N);
                for (int y = 0; y < G::TY; y += G::YB) {
                    if (elect_one()) {
                        const uint32_t ay = a0 + (uint32_t)((y * G::UPR * G::UA) >> 4);
                        const uint32_t bw = b0 + (uint32_t)((y * G::NPR * G::UB) >> 4);
#pragma unroll
                        for (int k = 0; k < TXW / 16; ++k) {
                            mma<true>(d, desc(ay + (uint32_t)((2 * k * G::GS) / 16), HI_A), desc(bw + (uint32_t)(2 * k * 8), HI_B), ID);
                        }
                    }
                    __syncwarp();
                }
                if (elect_one()) {
                    mma_commit(saddr(&bar_dempty[dplane % SD]));
                    mma_commit(saddr(&bar_empty[(plane - 2) % SH]));
                    if (q == t.n + 1) {
                        mma_commit(saddr(&bar_empty[(plane - 1) % SH]));
                        mma_commit(saddr(&bar_empty[plane % SH]));
                    }
                }
                __syncwarp();
                ++dplane;
            }
        }
        if (elect_one()) mma_commit(saddr(&bar_done));
        if (!ok && lane == 0) s_fail = 1;
        __syncwarp();
    } else if (warp >= WG_LOAD0) {
        const int lt = tid - WG_LOAD0 * 32;
        constexpr int LT = WG_LOADERS * 32;
        bool ok = true;
        int plane = 0, dplane = 0;
        int published = 0;
        auto publish = [&](int upto) {
            fence_async_proxy();
            __syncwarp();
            for (; published < upto; ++published) {
                if (lane == 0) mbar_arrive(saddr(&bar_full[published % SH]));
            }
        };
        // FL, LL: the fields of the next plane, loaded while this one's slots are awaited
        constexpr int PERF = MODE == FL ? (G::ROWS * TXW + LT - 1) / LT : G::TY * TXW / LT;
        uint32_t nx0[MODE == FL ? PERF : 1][3];
        float ng[MODE == LL ? PERF : 1][6];
        auto fetch = [&](const Item& t, int q) {
            if (MODE == FL) {
                int z = t.z0 - 1 + q;
                z = z < 0 ? z + s.nz : (z >= s.nz ? z - s.nz : z);
#pragma unroll
                for (int i = 0; i < PERF; ++i) {
                    const int v = lt + i * LT;
                    const int x = t.x0 + v % TXW;
                    int y = t.y0 - 1 + min(v / TXW, G::ROWS - 1);
                    y = y < 0 ? y + s.ny : (y >= s.ny ? (y - s.ny) % s.ny : y);
                    const uint32_t *row = p.x0 + (((long long)t.b * s.nz + z) * s.ny + y) * s.nx;
                    nx0[i][0] = row[x == 0 ? s.nx - 1 : x - 1];
                    nx0[i][1] = row[x];
                    nx0[i][2] = row[x == s.nx - 1 ? 0 : x + 1];
                }
            }
            if (MODE == LL && q >= 2) {
#pragma unroll
                for (int i = 0; i < PERF; ++i) {
                    const int v = lt + i * LT;
                    const int x = t.x0 + v % TXW;
                    const int y = min(t.y0 + v / TXW, s.ny - 1);
                    const long long row = (((long long)t.b * s.nz + t.z0 + q - 2) * s.ny + y) * s.nx;
                    const int xw = x == 0 ? s.nx - 1 : x - 1, xe = x == s.nx - 1 ? 0 : x + 1;
                    ng[i][0] = p.du[row + xe];
                    ng[i][1] = p.target[row + xe];
                    ng[i][2] = p.du[row + x];
                    ng[i][3] = p.target[row + x];
                    ng[i][4] = p.du[row + xw];
                    ng[i][5] = p.target[row + xw];
                }
            }
        };
        double loss = 0.0;
        float db = 0.f;
        if (blockIdx.x < p.items) fetch(item_of(blockIdx.x), 0);
        for (int it = blockIdx.x; ok && it < p.items; it += gridDim.x) {
            const Item t = item_of(it);
            for (int q = 0; q < t.n + 2; ++q, ++plane) {
                bool got = true;
                // hand over what has landed before waiting for a slot: the MMAs
                // that free it need no more than the planes up to this one's
                // second predecessor
                if (plane >= 2) {
                    asm volatile("cp.async.wait_group 1;" ::: "memory");
                    publish(plane - 1);
                }
                if (plane >= SH) {
                    got = mbar_wait(saddr(&bar_empty[plane % SH]), (uint32_t)(((plane - SH) / SH) & 1), fail);
                }
                const bool has_dz = q >= 2;
                if (has_dz && dplane >= SD) {
                    got = got && mbar_wait(saddr(&bar_dempty[dplane % SD]), (uint32_t)(((dplane - SD) / SD) & 1), fail);
                }
                if (!__all_sync(0xffffffffu, got)) {
                    ok = false;
                    break;
                }
                const uint32_t hs = hring + (uint32_t)((plane % SH) * G::HSLOT);
                const uint32_t ds = dring + (uint32_t)((dplane % SD) * G::DSLOT);
                if (MODE == FL) {
#pragma unroll
                    for (int i = 0; i < PERF; ++i) {
                        const int v = lt + i * LT;
                        if ((i + 1) * LT <= G::ROWS * TXW || v < G::ROWS * TXW) {
                            st_shared16(hs + (uint32_t)(v * 16), make_uint4(nx0[i][0], nx0[i][1], nx0[i][2], 0u));
                        }
                    }
                } else {
                    const bf16 *from = p.h + ghost_row(s, t.b, t.z0 + q, 0) * (s.nx + 2) * 8;
                    for (int v = lt; v < G::ROWS * TXW; v += LT) {
                        const int row = v / TXW, x = v % TXW;
                        const int gy = min(t.y0 + row, s.ny + 1);
                        const bf16 *src = from + (gy * 3LL * (s.nx + 2) + t.x0 + x + 1) * 8;
                        const uint32_t d = hs + (uint32_t)(row * 3 * G::UA + x * 16);
#pragma unroll
                        for (int c = 0; c < 3; ++c) copy16(d + c * G::UA, src + c * (s.nx + 2LL) * 8);
                    }
                }
                if (has_dz) {
                    // rows past the grid count nothing
                    const bf16 *from = MODE == LL ? nullptr : p.dz + ghost_row(s, t.b, t.z0 + q - 1, 0) * (s.nx + 2) * 8;
#pragma unroll
                    for (int i = 0; i < G::TY * TXW / LT; ++i) {
                        const int v = lt + i * LT;
                        const int row = v / TXW, x = v % TXW;
                        const bool in = t.y0 + row < s.ny;
                        const uint32_t d = ds + (uint32_t)(row * G::NPR * G::UB + x * 16);
                        if (MODE == LL) {
                            // taps dx = 0, 1, 2 of voxel x of h meet g at x + 1, x, x - 1
                            uint4 g = make_uint4(0u, 0u, 0u, 0u);
                            if (in) {
                                g.x = pack_bf16(p.scale * (ng[i][0] - ng[i][1]), p.scale * (ng[i][2] - ng[i][3]));
                                g.y = pack_bf16(p.scale * (ng[i][4] - ng[i][5]), 0.f);
                                const float e = ng[i][2] - ng[i][3];
                                loss = fma((double)e, (double)e, loss);
                                db += p.scale * e;
                            }
                            st_shared16(d, g);
                        } else {
                            const bf16 *src = from + ((in ? t.y0 + row + 1 : 0) * 3LL * (s.nx + 2) + t.x0 + x + 1) * 8;
#pragma unroll
                            for (int c = 0; c < 3; ++c) {
                                const bf16 *sc = src + c * (s.nx + 2LL) * 8;
                                if (MODE == FL) {
                                    copy16_or_zero(d + c * G::UB, sc, in);
                                } else {
                                    // tap dx of voxel x of h meets dz at x + 1 - dx
#pragma unroll
                                    for (int dx = 0; dx < 3; ++dx) copy16_or_zero(d + (dx * 3 + c) * G::UB, sc + (1 - dx) * 8, in);
                                }
                            }
                        }
                    }
                    ++dplane;
                }
                asm volatile("cp.async.commit_group;" ::: "memory");
                if (q + 1 < t.n + 2) fetch(t, q + 1);
                else if (it + (int)gridDim.x < p.items) fetch(item_of(it + gridDim.x), 0);
            }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        if (ok) publish(plane);
        else if (lane == 0) s_fail = 1;
        if (MODE == LL) {
            for (int o = 16; o > 0; o >>= 1) {
                loss += __shfl_xor_sync(0xffffffffu, loss, o);
                db += __shfl_xor_sync(0xffffffffu, db, o);
            }
            if (lane == 0) {
                atomicAdd(p.loss, loss);
                atomicAdd(p.db, db);
            }
        }
    } else {
        // the four warps between: lane quarter warp % 4
        const int qd = warp & 3;
        const uint32_t acc = tmem + ((uint32_t)(qd * 32) << 16);
        const float zero[8] = {};
        for (int c = 0; c < 3 * G::N; c += 8) tmem_st8(acc + (uint32_t)c, zero);
        tmem_st_wait();
        fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(saddr(&bar_clear));
        const bool done = __all_sync(0xffffffffu, mbar_wait(saddr(&bar_done), 0, fail));
        fence_after();
        if (!done && lane == 0) s_fail = s_bad = 1;
        asm volatile("bar.sync 1, 128;" ::: "memory");
        if (!s_bad) {
            // every copy has been read by an MMA: the ring becomes dW
            float *dw = reinterpret_cast<float *>(smem);
            const int ft = (warp - WG_MMA) * 32 + lane;
            for (int i = ft; i < G::OUT; i += 128) dw[i] = 0.f;
            asm volatile("bar.sync 1, 128;" ::: "memory");
            const int m = qd * 32 + lane;               // row of D: unit m / 8, element m % 8
            const int w = MODE == FL ? m / 8 : m / 24;  // row of h
            const int e = MODE == FL ? m % 8 : m % 24;  // FL: 2 dx + channel; else input channel
            // rounds over the dz row: one contribution per dW element each
            for (int y = 0; y < G::YB; ++y) {
                const int dy = w - y;
                const bool use = dy >= 0 && dy < 3 && (MODE != FL || e < 6);
                for (int dz = 0; dz < 3; ++dz) {
#pragma unroll
                    for (int c = 0; c < G::NPR; ++c) {
                        float v[8];
                        __syncwarp();
                        tmem_ld8(acc + (uint32_t)(dz * G::N + (y * G::NPR + c) * 8), v);
#pragma unroll
                        for (int i = 0; i < 8 && use; ++i) {
                            if (MODE == LL) {
                                if (i < 3) dw[((dz * 3 + dy) * 3 + i) * 24 + e] += v[i];
                            } else if (MODE == FL) {
                                dw[(((dz * 3 + dy) * 3 + e / 2) * 2 + e % 2) * 24 + c * 8 + i] += v[i];
                            } else {        // c = 3 dx + channel group
                                dw[(((dz * 3 + dy) * 3 + c / 3) * 24 + e) * 24 + c % 3 * 8 + i] += v[i];
                            }
                        }
                    }
                }
                asm volatile("bar.sync 1, 128;" ::: "memory");
            }
            float *out = p.part + (long long)blockIdx.x * G::OUT;
            for (int i = ft; i < G::OUT; i += 128) out[i] = dw[i];
        }
    }

    fence_before();
    __syncthreads();
    fence_after();
    if (s_fail) {
        // report, then wait (bounded) for the MMAs in flight
        if (tid == 0) {
            atomicExch(p.err, 1);
            mbar_wait(saddr(&bar_done), 0, nullptr);
        }
        fence_before();
        __syncthreads();
        fence_after();
    }
    if (warp == 0) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(G::TMEM) : "memory");
    }
}

// grads[off + i] = the sum of the CTAs' dW, in the CTAs' order
struct RParams {
    const float *part[4];
    int ctas[4], n[4];
    long long off[4];
};

// a warp's lanes take 32 consecutive elements, the eight warps every eighth CTA
__global__ void __launch_bounds__(256)
reduce_kernel(const RParams p, float *grads)
{
    __shared__ float sum[8][32];
    dependent_start();
    const int l = blockIdx.y;
    const int n = p.n[l], ctas = p.ctas[l];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int i0 = blockIdx.x * 32; i0 < n; i0 += gridDim.x * 32) {      // uniform
        const int i = i0 + lane;
        float a = 0.f;
        if (i < n) {
#pragma unroll 4
            for (int c = warp; c < ctas; c += 8) a += p.part[l][(long long)c * n + i];
        }
        sum[warp][lane] = a;
        __syncthreads();
        if (warp == 0 && i < n) {
            for (int w = 1; w < 8; ++w) a += sum[w][lane];
            grads[p.off[l] + i] = a;
        }
        __syncthreads();
    }
}

static int sm_count()
{
    static PerDevice<int> setup;
    return setup.get([] {
        int dev = 0, count = 0;
        LGD_CHECK_CUDA(cudaGetDevice(&dev));
        LGD_CHECK_CUDA(cudaDeviceGetAttribute(&count, cudaDevAttrMultiProcessorCount, dev));
        return count;
    });
}

template<int MODE, int TXW>
static int run_w(WParams p, cudaStream_t stream)
{
    typedef WGeo<MODE, TXW> G;
    static PerDevice<bool> setup;
    setup.get([] {
        LGD_CHECK_CUDA(cudaFuncSetAttribute(wgrad_tc_kernel<MODE, TXW>, cudaFuncAttributeMaxDynamicSharedMemorySize, G::SMEM));
        return true;
    });
    const int sms = sm_count();
    const long long cols = (long long)(p.s.nx / TXW) * ((p.s.ny + G::TY - 1) / G::TY) * p.s.batch;
    p.zchunk = least_planes(cols, p.s.nz, sms, 2, nullptr);
    p.items = (int)(cols * ((p.s.nz + p.zchunk - 1) / p.zchunk));
    const int ctas = std::min(sms, p.items);
    launch_dependent(wgrad_tc_kernel<MODE, TXW>, dim3(ctas), WG_THREADS, G::SMEM, stream, p);
    check_launch("tensor-core weight gradient");
    return ctas;
}

template<int MODE>
static int run_w_any(const WParams& p, cudaStream_t stream)
{
    if constexpr (MODE != CC) {             // 256 voxels of CC: 64 x 4 has fewer halo rows than 128 x 2
        if (p.s.nx % 128 == 0) return run_w<MODE, 128>(p, stream);
    }
    if (p.s.nx % 64 == 0) return run_w<MODE, 64>(p, stream);
    return run_w<MODE, 32>(p, stream);
}

}  // namespace tc

using namespace tc;

// elements of a layer's dW, and of all layers' partial buffers
static const int DW[4] = {27 * 2 * 24, 27 * 24 * 24, 27 * 24 * 24, 27 * 24};

size_t tc_partial_floats()
{
    return (size_t)sm_count() * (DW[0] + DW[1] + DW[2] + DW[3]);
}

int tc_wgrad(int layer, const void *h, const void *x0, const void *dz, const float *du, const float *target, float scale,
             double *loss, float *db, float *partials, const int dims[4], int *err, cudaStream_t stream)
{
    WParams p = {};
    p.s = {dims[0], dims[1], dims[2], dims[3]};
    p.h = (const bf16 *)h;
    p.x0 = (const uint32_t *)x0;
    p.dz = (const bf16 *)dz;
    p.du = du;
    p.target = target;
    p.scale = scale;
    p.loss = loss;
    p.db = db;
    size_t off = 0;
    for (int l = 0; l < layer; ++l) off += (size_t)sm_count() * DW[l];
    p.part = partials + off;
    p.err = err;
    if (layer == 0) return run_w_any<FL>(p, stream);
    if (layer == 3) return run_w_any<LL>(p, stream);
    return run_w_any<CC>(p, stream);
}

void tc_wgrad_reduce(const float *partials, const int ctas[4], const long long w_off[4], float *grads, cudaStream_t stream)
{
    RParams r;
    size_t off = 0;
    for (int l = 0; l < 4; ++l) {
        r.part[l] = partials + off;
        r.ctas[l] = ctas[l];
        r.n[l] = DW[l];
        r.off[l] = w_off[l];
        off += (size_t)sm_count() * DW[l];
    }
    launch_dependent(reduce_kernel, dim3((DW[1] + 31) / 32, 4), 256u, 0, stream, r, grads);
    check_launch("weight gradient sum");
}

}  // namespace sur
}  // namespace lgd
