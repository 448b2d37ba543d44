// Game of Life on packed rows: the default path of calls of several
// generations, for any board of at least 32 columns, any topology.
//
// A call packs the board's bytes into bits once (8 MB for 8192^2), runs its
// generations on the bits in passes of up to 32, and unpacks once; between
// the passes the board lives in L2.  In a pass a CTA holds a tile in
// registers: lane l of every warp owns 32-cell word l of a row and R
// consecutive rows, the W warps are stacked, so the tile is W * R rows of
// 1024 cells.  Per generation the warps exchange their outermost rows through
// shared memory (one barrier) and every row takes, in place,
//     2 shuffles + 2 funnel shifts     the words of the cells west and east
//     h = west + self + east           two bit planes (XOR3, majority)
//     the sum of three rows' h         T = u0 + 2 k, the 3 x 3 total
//     next = (T == 3) | (self & T == 4)
// that is two shuffles and eleven logic and shift instructions per 32 cells.  Summing across
// the row before summing down needs the neighbours of one bit plane, not of
// two as in gol_bits_kernel (k_gol.cu), and rows are independent of each
// other, where that kernel's chain runs through all its generations in every
// row.  Wrong values enter at the tile's rim and move one cell per
// generation; with T generations per pass the inner W * R - 2 T rows and, for
// T <= 32, lanes 1 .. 30 are right and are stored.
//
// Bound by the ALU pipe (64 lanes per clock and SM): 11 instructions per word
// allow 57 T cell updates per second on 152 SMs.  A pass of 16 generations of
// 8192^2 takes 33 us (33 T updates per second; 44 with three instructions more
// per word, gol_bits_kernel 99); the rest goes to the rim (6% of rows, 5% of
// words), 144 of 152 SMs at work, 5 us of launch, loads and stores per pass,
// and the exchange of rows.  More warps of fewer rows (24 x 23, 32 x 17) and
// shifts moved to the multiplier pipe gained nothing.
#include <algorithm>

#include "lgd_internal.h"
#include "k_cells.cuh"

namespace lgd {
namespace golp {

constexpr int OUT_WORDS = 30;               // words of a tile row that are stored
constexpr int MAX_T = 32;
constexpr int MAX_WARPS = 16;

struct Board {
    int nx, ny;
    int words;                              // (nx + 31) / 32
    int wpitch;                             // words between rows
    int periodic;                           // bit 0: x wraps, bit 1: y wraps
    uint32_t edge;                          // all bits of a word outside a board that does not wrap
};

// bytes (0 or 1) -> bits, one word per thread; bits past nx are zero
__global__ void __launch_bounds__(256)
pack_kernel(const uint8_t *in, long pitch, uint32_t *out, Board b)
{
    dependent_start();
    const long long total = (long long)b.wpitch * b.ny;
    for (long long i = blockIdx.x * 256ll + threadIdx.x; i < total; i += gridDim.x * 256ll) {
        const int y = (int)(i / b.wpitch);
        const int w = (int)(i - (long long)y * b.wpitch);
        uint32_t r = 0;
        if (w < b.words) {
            // rows are pitched to 128 bytes: the 32 bytes exist
            const uint4 *p = reinterpret_cast<const uint4 *>(in + (long)y * pitch + (long)w * 32);
            const uint4 lo = p[0], hi = p[1];
            const uint32_t v[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
            for (int k = 0; k < 8; ++k) r |= (((v[k] & 0x01010101u) * 0x10204080u) >> 28) << (4 * k);
            const int left = b.nx - w * 32;
            if (left < 32) r &= (1u << left) - 1u;
        }
        out[i] = r;
    }
}

__global__ void __launch_bounds__(256)
unpack_kernel(const uint32_t *in, uint8_t *out, long pitch, Board b)
{
    dependent_start();
    const long long total = (long long)b.words * b.ny;
    for (long long i = blockIdx.x * 256ll + threadIdx.x; i < total; i += gridDim.x * 256ll) {
        const int y = (int)(i / b.words);
        const int w = (int)(i - (long long)y * b.words);
        const uint32_t r = in[(long long)y * b.wpitch + w];
        uint32_t v[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) v[k] = (((r >> (4 * k)) & 0xFu) * 0x00204081u) & 0x01010101u;
        uint4 *p = reinterpret_cast<uint4 *>(out + (long)y * pitch + (long)w * 32);
        p[0] = make_uint4(v[0], v[1], v[2], v[3]);
        p[1] = make_uint4(v[4], v[5], v[6], v[7]);
    }
}

__device__ __forceinline__ uint32_t maj(uint32_t a, uint32_t b, uint32_t c) { return (a & b) | (a & c) | (b & c); }

// the sum of a cell and its two neighbours in the row, as two bit planes
__device__ __forceinline__ void row_sum(uint32_t v, uint32_t& h0, uint32_t& h1)
{
    const uint32_t w = __funnelshift_l(__shfl_up_sync(0xffffffffu, v, 1), v, 1);
    const uint32_t e = __funnelshift_r(v, __shfl_down_sync(0xffffffffu, v, 1), 1);
    h0 = w ^ v ^ e;
    h1 = maj(w, v, e);
}

// Next state of the row m from the sums of the rows above, at and below, in
// seven three-input operations: T = u0 + 2 k with k = p + 2 q + cy, and the
// cell lives if T == 3 (u0, k == 1) or, itself alive, T == 4 (~u0, k == 2).  The
// last three use that T == 0 does not occur for a living cell.
__device__ __forceinline__ uint32_t rule(uint32_t m, uint32_t a0, uint32_t a1, uint32_t m0, uint32_t m1, uint32_t c0,
                                         uint32_t c1)
{
    const uint32_t u0 = a0 ^ m0 ^ c0, cy = maj(a0, m0, c0);
    const uint32_t p = a1 ^ m1 ^ c1, q = maj(a1, m1, c1);
    const uint32_t x = (u0 & ~q) | (~u0 & ~m);
    const uint32_t even = (~cy & ~p) | (cy & p & ~q);           // k == 2, k == 0, not k == 1
    return (u0 & x & ~even) | (~u0 & ~x & even);
}

// T generations; the tile's inner rows [T, T + out_rows) are the board's rows
// y0 .. y0 + out_rows - 1.  CUBE: some axis does not wrap, cells beyond it
// hold the edge value in every generation.
template<int R, bool CUBE>
__global__ void __launch_bounds__(32 * MAX_WARPS)
gol_pack_kernel(const uint32_t *in, uint32_t *out, Board b, int T, int out_rows)
{
    __shared__ uint32_t rim[2][MAX_WARPS + 2][2][32];
    dependent_start();
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int warps = blockDim.x >> 5;
    const int y0 = blockIdx.y * out_rows;
    const int cx = (int)blockIdx.x * (OUT_WORDS * 32) - 32 + 32 * lane;     // cell of the word's bit 0

    // where the word's 32 cells sit in a packed row: bits p .. p + 31, and
    // where the row ends before them, the row's first bits (x wraps)
    int p = cx;
    uint32_t colmask = 0xffffffffu;
    bool none = false;                      // no cell of the word on the board
    if (b.periodic & 1) {
        p %= b.nx;
        if (p < 0) p += b.nx;
    } else {
        none = cx < 0 || cx >= b.nx;        // words are aligned to the board
        if (none) {
            p = 0;
            colmask = 0;
        } else if (b.nx - cx < 32) {
            colmask = (1u << (b.nx - cx)) - 1u;
        }
    }
    const int wl = p >> 5;
    const int sh = p & 31;
    const bool has_hi = sh != 0 && wl + 1 < b.words;
    const int fill = b.nx - p;                                  // cells up to the row's end
    const bool wraps = (b.periodic & 1) && fill < 32;

    // rows first .. first + R - 1 of the board (rowin: those that exist); all
    // loads of a kind are in flight together, and only warps with a window that
    // is not one word of the row load more: windows that straddle two words, and
    // the row's last, partial word, which the row's start completes.  That one is
    // aligned and may be the only such window of its warp (lane 31 of a tile that
    // ends there: rows of 1921 .. 1951 cells, and every 960 more)
    uint32_t v[R];
    uint32_t rowin[CUBE ? (R + 31) / 32 : 1] = {};
    int first = y0 - T + warp * R;
    if (b.periodic & 2) {
        first %= b.ny;
        if (first < 0) first += b.ny;
    }
    auto row_of = [&](int r) -> const uint32_t * {
        int y = first + r;
        if (CUBE) {
            if ((b.periodic & 2) && y >= b.ny) y %= b.ny;
            y = min(max(y, 0), b.ny - 1);
        } else if (y >= b.ny) {
            y -= b.ny;
            if (y >= b.ny) y %= b.ny;
        }
        return in + (long long)y * b.wpitch;
    };
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = row_of(r)[wl];
    if (__any_sync(0xffffffffu, sh != 0 || wraps)) {
        const int wh = has_hi ? wl + 1 : wl;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const uint32_t *row = row_of(r);
            const uint32_t hi = row[wh], start = row[0];
            uint32_t x = __funnelshift_r(v[r], has_hi ? hi : 0u, sh);
            if (wraps) x |= start << fill;
            v[r] = x;
        }
    }
    if (CUBE) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const bool inside = (b.periodic & 2) || (unsigned)(first + r) < (unsigned)b.ny;
            v[r] = inside ? (v[r] & colmask) | (b.edge & ~colmask) : b.edge;
            if (inside) rowin[r / 32] |= 1u << (r % 32);
        }
    }

    for (int t = 0; t < T; ++t) {
        uint32_t (*rm)[2][32] = rim[t & 1];
        rm[warp + 1][0][lane] = v[0];
        rm[warp + 1][1][lane] = v[R - 1];
        __syncthreads();            // one per generation: the next one writes the other buffer
        // beyond the tile: any value (rows 0 and warps + 1 are never written)
        const uint32_t above = warp > 0 ? rm[warp][1][lane] : 0u;
        const uint32_t below = warp + 1 < warps ? rm[warp + 2][0][lane] : 0u;
        uint32_t a0, a1, m0, m1;
        row_sum(above, a0, a1);
        row_sum(v[0], m0, m1);
#pragma unroll
        for (int r = 0; r < R; ++r) {
            uint32_t c0, c1;
            row_sum(r + 1 < R ? v[r + 1] : below, c0, c1);
            uint32_t x = rule(v[r], a0, a1, m0, m1, c0, c1);
            if (CUBE) {
                x = (x & colmask) | (b.edge & ~colmask);
                if (!((rowin[r / 32] >> (r % 32)) & 1u)) x = b.edge;
            }
            v[r] = x;
            a0 = m0;
            a1 = m1;
            m0 = c0;
            m1 = c1;
        }
    }

    if (lane < 1 || lane > OUT_WORDS || cx >= b.nx) return;
    const uint32_t keep = b.nx - cx < 32 ? (1u << (b.nx - cx)) - 1u : 0xffffffffu;
    uint32_t *o = out + (cx >> 5);
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int i = warp * R + r;
        const int gy = y0 - T + i;
        if (i >= T && i < T + out_rows && gy < b.ny) o[(long long)gy * b.wpitch] = v[r] & keep;
    }
}

// Tile height and generations per pass, by a model fitted to a sweep of all of
// them on boards from 300^2 to 8192^2 (it finds the sweep's best or one within
// 5%).  A generation takes the busiest SM's rows at 3.75 ns each (its four
// quarters in step: the warps of the fullest count), or one warp's chain of
// rows, 15 ns each, whichever is longer, and 45 ns of exchange; a pass adds
// its launch, loads and stores.
struct Plan {
    int R, W, T, out_rows;
    int per_sm;                             // CTAs on the busiest SM
    double ns;                              // per generation
};

constexpr int SM_SMEM = 224 * 1024;         // shared memory of an SM to divide up, at most
constexpr int CTA_SMEM = 12 * 1024;         // static (the rim) and reserved shared memory of a CTA

constexpr int ROWS[] = {8, 12, 16, 24, 34};     // compiled rows per lane (34: 16 warps hold 512 + 2 * 16 rows)

static Plan plan(int nx, int ny, int sms, int steps)
{
    Plan best = {8, 4, 1, 1, 1, 1e300};
    const long long xt = (nx + OUT_WORDS * 32 - 1) / (OUT_WORDS * 32);
    for (int R : ROWS) {
        for (int W = 4; W <= MAX_WARPS; ++W) {
            for (int T = 4; T <= MAX_T; T += 4) {
                const int room = W * R - 2 * T;
                if (room < 4) break;
                // even bands: no tile is nearly empty
                const long long bands = (ny + room - 1) / room;
                if (bands > 65535) continue;
                const int out_rows = (int)((ny + bands - 1) / bands);
                const long long per_sm = (xt * bands + sms - 1) / sms;
                const double rows = (double)((per_sm * W + 3) / 4 * 4) * R;
                const double gen = std::max(rows * 3.75, R * 15.0) + 45.0;
                const int passes = (steps + T - 1) / T;
                const double ns = (passes * (1600.0 + 100.0 * R) + gen * steps) / steps;
                if (ns < best.ns * 0.999) best = {R, W, T, out_rows, (int)per_sm, ns};
            }
        }
    }
    return best;
}

template<bool CUBE>
static void launch_pass(Grid& g, const Board& b, const Plan& p, int T, const uint32_t *in, uint32_t *out)
{
    const dim3 grid((unsigned)((b.nx + OUT_WORDS * 32 - 1) / (OUT_WORDS * 32)),
                    (unsigned)((b.ny + p.out_rows - 1) / p.out_rows));
    void (*fn)(const uint32_t *, uint32_t *, Board, int, int) = nullptr;
    switch (p.R) {
    case 8: fn = gol_pack_kernel<8, CUBE>; break;
    case 12: fn = gol_pack_kernel<12, CUBE>; break;
    case 16: fn = gol_pack_kernel<16, CUBE>; break;
    case 24: fn = gol_pack_kernel<24, CUBE>; break;
    default: fn = gol_pack_kernel<34, CUBE>; break;
    }
    // Shared memory that only the plan's share of CTAs fits on an SM with: a
    // dependent launch is placed while the pass before still runs, and would
    // pile its CTAs on the SMs that happen to have room (8192^2: 144 CTAs of
    // one per SM, 90 us per pass of 16 piled up, 55 us spread)
    static PerDevice<bool> setup;
    setup.get([] {
        for (const void *f : {(const void *)gol_pack_kernel<8, CUBE>, (const void *)gol_pack_kernel<12, CUBE>,
                              (const void *)gol_pack_kernel<16, CUBE>, (const void *)gol_pack_kernel<24, CUBE>,
                              (const void *)gol_pack_kernel<34, CUBE>}) {
            LGD_CHECK_CUDA(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, SM_SMEM - CTA_SMEM));
        }
        return true;
    });
    const size_t smem = (size_t)std::max(0, std::min(SM_SMEM - CTA_SMEM, SM_SMEM / p.per_sm - CTA_SMEM));
    launch_dependent(fn, grid, 32u * p.W, smem, g.stream, in, out, b, T, p.out_rows);
}

}  // namespace golp

bool gol_packed_applicable(const Grid& g)
{
    const double edge = g.desc.edge[0];
    return g.desc.cell == LGD_CELL_GOL_U8 && g.desc.nz == 1 && g.desc.nx >= 32 && g.desc.nx <= (1 << 30) &&
           g.desc.ny <= (1 << 24) && ((g.desc.periodic & 3) == 3 || edge == 0.0 || edge == 1.0);
}

static golp::Board board_of(const Grid& g)
{
    golp::Board b;
    b.nx = g.desc.nx;
    b.ny = g.desc.ny;
    b.words = (b.nx + 31) / 32;
    b.wpitch = round_up(b.words, 4);
    b.periodic = g.desc.periodic & 3;
    b.edge = (uint8_t)g.desc.edge[0] ? 0xffffffffu : 0u;
    return b;
}

// A quarter of one byte board's memory, kept with the grid; a board that leaves
// no room for it runs on bytes.
bool gol_packed_ready(Grid& g)
{
    const golp::Board b = board_of(g);
    if (g.d_bits == nullptr) (void)malloc_on_first_use((void **)&g.d_bits, 2 * (size_t)b.wpitch * b.ny * sizeof(uint32_t));
    return g.d_bits != nullptr;
}

// steps >= 1 generations of a board whose cells are 0 or 1
void launch_gol_packed(Grid& g, int steps)
{
    using namespace golp;
    static PerDevice<int> setup;
    const int sms = setup.get([] {
        int dev = 0, count = 0;
        LGD_CHECK_CUDA(cudaGetDevice(&dev));
        LGD_CHECK_CUDA(cudaDeviceGetAttribute(&count, cudaDevAttrMultiProcessorCount, dev));
        return count;
    });
    const Board b = board_of(g);
    const size_t elems = (size_t)b.wpitch * b.ny;
    uint32_t *bits[2] = {g.d_bits, g.d_bits + elems};
    const long pitch = (long)g.pitch_bytes[0];
    const unsigned blocks = (unsigned)std::min<long long>(152LL * 32, ((long long)elems + 255) / 256);
    launch_dependent(pack_kernel, dim3(blocks), 256u, 0, g.stream, (const uint8_t *)g.m[0].buf[g.cur], pitch, bits[0],
                     b);
    const Plan p = plan(b.nx, b.ny, sms, steps);
    int src = 0;
    g.launches += 2;
    while (steps > 0) {
        const int T = std::min(steps, p.T);
        if (b.periodic == 3) launch_pass<false>(g, b, p, T, bits[src], bits[1 - src]);
        else launch_pass<true>(g, b, p, T, bits[src], bits[1 - src]);
        src = 1 - src;
        steps -= T;
        ++g.launches;
    }
    launch_dependent(unpack_kernel, dim3(blocks), 256u, 0, g.stream, (const uint32_t *)bits[src],
                     (uint8_t *)g.m[0].buf[1 - g.cur], pitch, b);
    g.cur = 1 - g.cur;
}

}  // namespace lgd
