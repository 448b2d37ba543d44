// Game of Life on uint8 cells (one byte per cell, 0 or 1), Moore radius 1.
//
// The kernels on byte rows: single generations, and the passes that an explicit
// depth selects (gol_bits_kernel, gol_tb_kernel below).  Calls of more than a few
// generations run on packed rows by default (k_golpack.cu).
//
// Single generation (torus, nx a multiple of 16): SWAR on 32-bit words.  A thread
// owns 16 consecutive cells of one row (one 16-byte load per row for the
// rows above, at and below) plus the 4-byte words left and right of them.
// Column sums of the three rows are formed per byte lane (values <= 3),
// shifted by one byte each way with funnel shifts for the horizontal
// neighbours, and the rule is applied with per-byte equality tests.  Every
// cell costs about five integer operations; traffic is 2 B/cell/step.
//
// Generic path (any size, cube or torus): one thread per cell.
#include <algorithm>
#include <mutex>
#include <type_traits>

#include "lgd_internal.h"
#include "k_cells.cuh"

namespace lgd {

// per-byte (x == 0) -> 1, else 0, for bytes below 0x80
__device__ __forceinline__ uint32_t bytes_zero(uint32_t x)
{
    return (~((x + 0x7F7F7F7Fu) | x) & 0x80808080u) >> 7;
}

__device__ __forceinline__ uint32_t gol_word(uint32_t vl_word, uint32_t v, uint32_t vr_word, uint32_t mid)
{
    // vl: byte k holds the column sum of cell k-1; vr: of cell k+1
    uint32_t vl = __funnelshift_l(vl_word, v, 8);
    uint32_t vr = __funnelshift_r(v, vr_word, 8);
    uint32_t tot = vl + v + vr;   // includes the cell itself
    uint32_t eq3 = bytes_zero(tot ^ 0x03030303u);
    uint32_t eq4 = bytes_zero(tot ^ 0x04040404u);
    return eq3 | (mid & eq4);
}

__global__ void __launch_bounds__(256)
gol_swar_torus_kernel(const uint8_t *__restrict__ in, uint8_t *__restrict__ out, int nx, int ny, long pitch)
{
    const int words16 = nx >> 4;
    const long long total = (long long)words16 * ny;
    for (long long gid = blockIdx.x * (long long)blockDim.x + threadIdx.x; gid < total;
         gid += (long long)gridDim.x * blockDim.x) {
        const int xi = (int)(gid % words16);
        const int y = (int)(gid / words16);
        const int x0 = xi << 4;
        const int yu = (y == 0) ? ny - 1 : y - 1;
        const int yd = (y == ny - 1) ? 0 : y + 1;
        const int xl = (x0 == 0) ? nx - 4 : x0 - 4;
        const int xr = (x0 + 16 == nx) ? 0 : x0 + 16;
        const uint8_t *ru = in + yu * pitch;
        const uint8_t *rm = in + y * pitch;
        const uint8_t *rd = in + yd * pitch;
        const uint4 a = *(const uint4 *)(ru + x0);
        const uint4 b = *(const uint4 *)(rm + x0);
        const uint4 c = *(const uint4 *)(rd + x0);
        const uint32_t vl = *(const uint32_t *)(ru + xl) + *(const uint32_t *)(rm + xl) + *(const uint32_t *)(rd + xl);
        const uint32_t vr = *(const uint32_t *)(ru + xr) + *(const uint32_t *)(rm + xr) + *(const uint32_t *)(rd + xr);
        const uint32_t v0 = a.x + b.x + c.x;
        const uint32_t v1 = a.y + b.y + c.y;
        const uint32_t v2 = a.z + b.z + c.z;
        const uint32_t v3 = a.w + b.w + c.w;
        uint4 o;
        o.x = gol_word(vl, v0, v1, b.x);
        o.y = gol_word(v0, v1, v2, b.y);
        o.z = gol_word(v1, v2, v3, b.z);
        o.w = gol_word(v2, v3, vr, b.w);
        *(uint4 *)(out + y * pitch + x0) = o;
    }
}

__global__ void gol_generic_kernel(View<const uint8_t> in, View<uint8_t> out, int periodic, uint8_t edge)
{
    const long long cells = (long long)in.nx * in.ny;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < cells;
         i += (long long)gridDim.x * blockDim.x) {
        const int x = (int)(i % in.nx);
        const int y = (int)(i / in.nx);
        int living = 0;
        for (int dy = -1; dy <= 1; ++dy) {
            for (int dx = -1; dx <= 1; ++dx) {
                living += load_bc(in, x + dx, y + dy, 0, periodic, edge);
            }
        }
        const uint8_t self = in.at(x, y, 0);
        out.at(x, y, 0) = gol_rule(self, living - self);
    }
}

// Temporal blocking on the torus fast path: T generations per pass.
//
// A warp covers 32 consecutive 16-byte chunks of a row (lane l: chunk
// xw * 30 + l - 1, wrapped around the row); lanes 1..30 are its output,
// lanes 0 and 31 its halo (the neighbouring warps' chunks, recomputed).  The
// warp marches down a strip of rows [y0, y1), reading rows y0 - T .. y1 + T
// - 1 (wrapped).  At iteration i, generation t computes row i - t from
// generation t - 1's rows i - t - 1, i - t, i - t + 1, which the lane holds
// in registers (three rows per generation rotate through v[t][i % 3]; the
// loop is unrolled three times so the rotation is a renaming); the column
// sums of the words left and right of the lane's 16 cells come from lanes
// l - 1 and l + 1 by shuffle.  Generation T's rows of the strip are stored.
// A generation's wrong values spread one cell per generation from the
// warp's edges, so with 16 cells of halo per side T <= 16 keeps every
// stored cell exact; the registers limit T to 12 here.  Input rows are
// prefetched two iterations ahead.  HBM / L2 traffic per pass: 2 B per cell
// for T generations.
template<int T>
__global__ void __launch_bounds__(128)
gol_tb_kernel(const uint8_t *__restrict__ in, uint8_t *__restrict__ out, int nx, int ny, long pitch, int strip,
              int xwarps)
{
    const int lane = threadIdx.x & 31;
    const int gw = blockIdx.x * 4 + (threadIdx.x >> 5);
    const int xw = gw % xwarps;
    const int y0 = (gw / xwarps) * strip;
    if (y0 >= ny) return;                                   // warp-uniform
    const int y1 = min(y0 + strip, ny);
    const int nch = nx >> 4;
    const int out_chunk = xw * 30 + lane - 1;
    const int ch = ((out_chunk % nch) + nch) % nch;         // chunk this lane holds
    const bool store = lane >= 1 && lane <= 30 && out_chunk < nch;
    const int nrows = (y1 - y0) + 2 * T;                    // input row j is y0 - T + j
    const uint8_t *col = in + (long)ch * 16;
    auto row_of = [&](int j) { return ((y0 - T + j) % ny + ny) % ny; };

    uint4 v[T][3];
    uint4 pf[3];                                            // input rows prefetched: pf[j % 3] holds row j
    pf[0] = *reinterpret_cast<const uint4 *>(col + (long)row_of(0) * pitch);
    if (nrows > 1) pf[1] = *reinterpret_cast<const uint4 *>(col + (long)row_of(1) * pitch);

    auto iteration = [&](auto phase, int i) {
        constexpr int P = decltype(phase)::value;          // i % 3
        constexpr int PC = (P + 2) % 3;                    // row i - 1 of a generation
        constexpr int PB = (P + 1) % 3;                    // row i - 2
        v[0][P] = pf[P];
        if (i + 2 < nrows) pf[(P + 2) % 3] = *reinterpret_cast<const uint4 *>(col + (long)row_of(i + 2) * pitch);
#pragma unroll
        for (int t = 1; t <= T; ++t) {
            if (i < 2 * t) break;                           // warp-uniform
            const uint4 a = v[t - 1][PB], m = v[t - 1][PC], c = v[t - 1][P];
            const uint32_t s0 = a.x + m.x + c.x;
            const uint32_t s1 = a.y + m.y + c.y;
            const uint32_t s2 = a.z + m.z + c.z;
            const uint32_t s3 = a.w + m.w + c.w;
            const uint32_t sl = __shfl_up_sync(0xffffffffu, s3, 1);
            const uint32_t sr = __shfl_down_sync(0xffffffffu, s0, 1);
            uint4 r;
            r.x = gol_word(sl, s0, s1, m.x);
            r.y = gol_word(s0, s1, s2, m.y);
            r.z = gol_word(s1, s2, s3, m.z);
            r.w = gol_word(s2, s3, sr, m.w);
            if (t < T) {
                v[t][P] = r;
            } else if (store) {
                const int y = y0 - 2 * T + i;               // in [y0, y1)
                *reinterpret_cast<uint4 *>(out + (long)y * pitch + (long)out_chunk * 16) = r;
            }
        }
    };
    for (int i = 0; i < nrows; i += 3) {
        iteration(std::integral_constant<int, 0>(), i);
        if (i + 1 < nrows) iteration(std::integral_constant<int, 1>(), i + 1);
        if (i + 2 < nrows) iteration(std::integral_constant<int, 2>(), i + 2);
    }
}

// Bit-sliced temporal blocking (torus, nx a multiple of 32): a lane holds
// 32 cells of a row as the bits of one 32-bit word (bit k = cell x0 + k),
// a warp 32 words = 1024 cells, lanes 0 and 31 the wrapped halo words.  Per
// generation and row, with a, m, c the rows above, at and below:
//   column sums s = a + m + c as bit planes s0 = a ^ m ^ c, s1 = maj(a, m, c);
//   the neighbour columns' sums by funnel shifts with the words of lanes
//   l - 1 and l + 1 (four shuffles), and the 3 x 3 total, self included,
//   T = sl + s + sr = u0 + 2 k with u0 = sl0 ^ s0 ^ sr0 and
//   k = sl1 + s1 + sr1 + maj(sl0, s0, sr0) (0..4);
//   next = (T == 3) | (m & T == 4) = (u0 & k == 1) | (~u0 & m & k == 2),
// about twenty logic operations per 32 cells.  Rows arrive as bytes and
// are packed with a multiply per 4 cells ((w * 0x10204080) >> 28 gathers
// bytes 0..3 of w, each 0 or 1, into bits 0..3; no partial product reaches
// bit 28 but the wanted ones), and stored back the same way
// ((nibble * 0x00204081) & 0x01010101).  Wrong values spread one cell per
// generation from a warp's halo words, so T <= 32 keeps lanes 1..30 exact.
// The row march, prefetch and strips are those of gol_tb_kernel.
__device__ __forceinline__ uint32_t gol_pack32(const uint4& lo, const uint4& hi)
{
    const uint32_t w[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
    uint32_t r = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) r |= ((w[i] * 0x10204080u) >> 28) << (4 * i);
    return r;
}

__device__ __forceinline__ void gol_unpack32(uint32_t r, uint4& lo, uint4& hi)
{
    uint32_t w[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) w[i] = (((r >> (4 * i)) & 0xFu) * 0x00204081u) & 0x01010101u;
    lo = make_uint4(w[0], w[1], w[2], w[3]);
    hi = make_uint4(w[4], w[5], w[6], w[7]);
}

__device__ __forceinline__ uint32_t gol_bits_row(uint32_t a, uint32_t m, uint32_t c)
{
    const uint32_t s0 = a ^ m ^ c;
    const uint32_t s1 = (a & m) | (a & c) | (m & c);
    const uint32_t s0l = __shfl_up_sync(0xffffffffu, s0, 1);
    const uint32_t s1l = __shfl_up_sync(0xffffffffu, s1, 1);
    const uint32_t s0r = __shfl_down_sync(0xffffffffu, s0, 1);
    const uint32_t s1r = __shfl_down_sync(0xffffffffu, s1, 1);
    const uint32_t x0 = __funnelshift_l(s0l, s0, 1);        // column x - 1
    const uint32_t x1 = __funnelshift_l(s1l, s1, 1);
    const uint32_t z0 = __funnelshift_r(s0, s0r, 1);        // column x + 1
    const uint32_t z1 = __funnelshift_r(s1, s1r, 1);
    const uint32_t u0 = x0 ^ s0 ^ z0;
    const uint32_t c0 = (x0 & s0) | (x0 & z0) | (s0 & z0);
    // k = x1 + s1 + z1 + c0 as two half sums a1 + 2 a2 and b1 + 2 b2
    const uint32_t a1 = x1 ^ s1, a2 = x1 & s1;
    const uint32_t b1 = z1 ^ c0, b2 = z1 & c0;
    const uint32_t k1 = (a1 ^ b1) & ~(a2 | b2);
    const uint32_t k2 = (a2 & ~(b1 | b2)) | (b2 & ~(a1 | a2)) | (a1 & b1);
    return (u0 & k1) | (~u0 & m & k2);
}

template<int T>
__global__ void __launch_bounds__(128)
gol_bits_kernel(const uint8_t *__restrict__ in, uint8_t *__restrict__ out, int nx, int ny, long pitch, int strip,
                int xwarps)
{
    const int lane = threadIdx.x & 31;
    const int gw = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int xw = gw % xwarps;
    const int y0 = (gw / xwarps) * strip;
    if (y0 >= ny) return;                                   // warp-uniform
    const int y1 = min(y0 + strip, ny);
    const int nw = nx >> 5;
    const int out_word = xw * 30 + lane - 1;
    const int wd = ((out_word % nw) + nw) % nw;             // word this lane holds
    const bool store = lane >= 1 && lane <= 30 && out_word < nw;
    const int nrows = (y1 - y0) + 2 * T;                    // input row j is y0 - T + j
    const uint8_t *col = in + (long)wd * 32;
    auto row_of = [&](int j) { return ((y0 - T + j) % ny + ny) % ny; };
    auto load = [&](int j, uint4& lo, uint4& hi) {
        const uint4 *p = reinterpret_cast<const uint4 *>(col + (long)row_of(j) * pitch);
        lo = p[0];
        hi = p[1];
    };
    auto put = [&](int j, uint32_t r) {                     // generation T's row j
        const int y = y0 - T + j;                           // in [y0, y1)
        uint4 lo, hi;
        gol_unpack32(r, lo, hi);
        uint4 *o = reinterpret_cast<uint4 *>(out + (long)y * pitch + (long)out_word * 32);
        o[0] = lo;
        o[1] = hi;
    };

    uint32_t v[T][3];
    uint4 pl[3], ph[3];                                     // raw input rows: [j % 3] holds row j
    load(0, pl[0], ph[0]);
    if (nrows > 1) load(1, pl[1], ph[1]);

    // generation t computes row i - t at iteration i from generation
    // t - 1's rows of iterations i - 2 .. i
    auto iteration = [&](auto phase, int i) {
        constexpr int P = decltype(phase)::value;          // i % 3
        constexpr int PC = (P + 2) % 3;                    // row i - 1 of a generation
        constexpr int PB = (P + 1) % 3;                    // row i - 2
        v[0][P] = gol_pack32(pl[P], ph[P]);
        if (i + 2 < nrows) load(i + 2, pl[(P + 2) % 3], ph[(P + 2) % 3]);
#pragma unroll
        for (int t = 1; t <= T; ++t) {
            if (i < 2 * t) break;                           // warp-uniform
            const uint32_t r = gol_bits_row(v[t - 1][PB], v[t - 1][PC], v[t - 1][P]);
            if (t < T) {
                v[t][P] = r;
            } else if (store) {
                put(i - T, r);
            }
        }
    };
    for (int i = 0; i < nrows; i += 3) {
        iteration(std::integral_constant<int, 0>(), i);
        if (i + 1 < nrows) iteration(std::integral_constant<int, 1>(), i + 1);
        if (i + 2 < nrows) iteration(std::integral_constant<int, 2>(), i + 2);
    }
}

// generations per bit-sliced pass when none are requested
constexpr int GOL_BITS_DEFAULT_DEPTH = 16;

// generations of a call from which the packed board pays for packing and
// unpacking: on boards whose alternative is one launch per generation, and on a
// torus of aligned rows, whose alternative is a bit-sliced pass over bytes.  us per
// call, packed against not: 1001 x 777 x 4 17 / 34; 1024^2 x 6 10 / 21, 8192^2 x 6 44 /
// 49, x 16 60 / 100.  Beyond L2 the passes over bytes, which do their few generations
// in one read and write, win longer: 8192 x 16384 x 6 95 / 75, x 8 104 / 89, x 10 104 /
// 137; 23168^2 x 12 428 / 409, x 14 464 / 586; 32768^2 x 16 1079 / 1011, x 20 1236 / 1449.
// Boards of a few long rows fill little of a tile of 32 rows or more: 1 x 1000000 x 8
// 15.6 / 11.5, x 16 25 / 26, 1 x 4000000 x 32 132 / 120
constexpr int GOL_PACK_MIN = 4;

static int gol_pack_min(const Grid& g, bool aligned_torus)
{
    if (!aligned_torus) return GOL_PACK_MIN;
    const int nx = g.desc.nx, ny = g.desc.ny;
    const long long cells = (long long)nx * ny;
    if (nx % 32 != 0) return 6;
    if (ny < 16 && nx > 1 << 18) return ny < 4 && nx > 1 << 21 ? 96 : 16;
    if (ny < 4) return 8;
    return cells <= 1ll << 26 ? 6 : (cells < 1ll << 28 ? 10 : (cells < 1ll << 30 ? 14 : 20));
}

bool gol_tb_applicable(const Grid& g)
{
    return g.desc.cell == LGD_CELL_GOL_U8 && (g.desc.periodic & 3) == 3 && g.desc.nz == 1 && g.desc.nx % 16 == 0 &&
           g.pitch_bytes[0] % 16 == 0;
}

// one pass of `depth` generations (2, 4, 6, 8, 12 instantiated: other
// depths run as the next smaller one); shape 0 = strips sized for about one
// wave of resident warps (8192^2 at 8 generations: 4041 GLUPS, against 3856
// for strips half as tall, 3013 for twice as tall and 2135 for one
// generation per pass), 1 = twice as tall, 2 = half as tall
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

// resident CTAs per SM of a pass kernel, queried once (the query also
// loads the kernel, which CUDA otherwise does at its first launch)
template<int T>
static int gol_tb_per_sm()
{
    static PerDevice<int> setup;
    return setup.get([] {
        int n = 0;
        LGD_CHECK_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, gol_tb_kernel<T>, 128, 0));
        return std::max(1, n);
    });
}

template<int T>
static void launch_gol_tb_typed(Grid& g, int shape)
{
    const int sms = sm_count();
    const int per_sm = gol_tb_per_sm<T>();
    const int nch = g.desc.nx / 16;
    const int xwarps = (nch + 29) / 30;
    const long long want = 1LL * sms * per_sm * 4;          // one wave of resident warps
    int strip = (int)std::max<long long>(4 * T, ((long long)g.desc.ny * xwarps + want - 1) / want);
    if (shape == 1) strip *= 2;
    if (shape == 2) strip = std::max(2 * T, strip / 2);
    strip = std::min(strip, g.desc.ny);
    const long long warps = (long long)xwarps * ((g.desc.ny + strip - 1) / strip);
    const uint8_t *in = (const uint8_t *)g.m[0].buf[g.cur];
    uint8_t *out = (uint8_t *)g.m[0].buf[1 - g.cur];
    gol_tb_kernel<T><<<(unsigned)((warps + 3) / 4), 128, 0, g.stream>>>(in, out, g.desc.nx, g.desc.ny,
                                                                       (long)g.pitch_bytes[0], strip, xwarps);
}

bool gol_bits_applicable(const Grid& g)
{
    return gol_tb_applicable(g) && g.desc.nx % 32 == 0;
}

constexpr int GOL_BITS_WPB = 4;                             // warps per CTA of the bit-sliced passes

template<int T>
static int gol_bits_per_sm()
{
    static PerDevice<int> setup;
    return setup.get([] {
        int n = 0;
        LGD_CHECK_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, gol_bits_kernel<T>, 32 * GOL_BITS_WPB, 0));
        return std::max(1, n);
    });
}

// one bit-sliced pass of `depth` generations (2, 4, 6, 8, 12, 16, 24, 32
// instantiated; other depths run as the next smaller one); strips as for
// the byte kernel, at least 4 * T rows
template<int T>
static void launch_gol_bits_typed(Grid& g, int shape)
{
    constexpr int WPB = GOL_BITS_WPB;
    const int sms = sm_count();
    const int per_sm = gol_bits_per_sm<T>();
    const int nw = g.desc.nx / 32;
    const int xwarps = (nw + 29) / 30;
    const long long want = 1LL * sms * per_sm * WPB;        // one wave of resident warps
    int strip = (int)std::max<long long>(4 * T, ((long long)g.desc.ny * xwarps + want - 1) / want);
    if (shape == 1) strip *= 2;
    if (shape == 2) strip = std::max(2 * T, strip / 2);
    strip = std::min(strip, g.desc.ny);
    const long long warps = (long long)xwarps * ((g.desc.ny + strip - 1) / strip);
    const uint8_t *in = (const uint8_t *)g.m[0].buf[g.cur];
    uint8_t *out = (uint8_t *)g.m[0].buf[1 - g.cur];
    gol_bits_kernel<T><<<(unsigned)((warps + WPB - 1) / WPB), 32 * WPB, 0, g.stream>>>(in, out, g.desc.nx, g.desc.ny,
                                                                         (long)g.pitch_bytes[0], strip, xwarps);
}

static int gol_bits_pass(Grid& g, int depth, int shape)
{
    int d = 2;
    if (depth >= 32) { launch_gol_bits_typed<32>(g, shape); d = 32; }
    else if (depth >= 24) { launch_gol_bits_typed<24>(g, shape); d = 24; }
    else if (depth >= 16) { launch_gol_bits_typed<16>(g, shape); d = 16; }
    else if (depth >= 12) { launch_gol_bits_typed<12>(g, shape); d = 12; }
    else if (depth >= 8) { launch_gol_bits_typed<8>(g, shape); d = 8; }
    else if (depth >= 6) { launch_gol_bits_typed<6>(g, shape); d = 6; }
    else if (depth >= 4) { launch_gol_bits_typed<4>(g, shape); d = 4; }
    else { launch_gol_bits_typed<2>(g, shape); }
    check_launch("game of life bit-sliced temporal blocking");
    ++g.launches;
    g.cur = 1 - g.cur;
    return d;
}

static int gol_tb_pass(Grid& g, int depth, int shape)
{
    int d = 0;
    if (depth >= 12) { launch_gol_tb_typed<12>(g, shape); d = 12; }
    else if (depth >= 8) { launch_gol_tb_typed<8>(g, shape); d = 8; }
    else if (depth >= 6) { launch_gol_tb_typed<6>(g, shape); d = 6; }
    else if (depth >= 4) { launch_gol_tb_typed<4>(g, shape); d = 4; }
    else { launch_gol_tb_typed<2>(g, shape); d = 2; }
    check_launch("game of life temporal blocking");
    ++g.launches;
    g.cur = 1 - g.cur;
    return d;
}

// Loads every pass kernel once, on a grid's first step: a pass depth first
// used later (after the warm-up steps of a benchmark, say) then costs no
// module load and no occupancy query inside the timed steps
static void prepare_gol_kernels()
{
    static PerDevice<bool> setup;
    setup.get([] {
        (void)sm_count();
        (void)gol_bits_per_sm<2>();
        (void)gol_bits_per_sm<4>();
        (void)gol_bits_per_sm<6>();
        (void)gol_bits_per_sm<8>();
        (void)gol_bits_per_sm<12>();
        (void)gol_bits_per_sm<16>();
        (void)gol_bits_per_sm<24>();
        (void)gol_bits_per_sm<32>();
        (void)gol_tb_per_sm<2>();
        (void)gol_tb_per_sm<4>();
        (void)gol_tb_per_sm<6>();
        (void)gol_tb_per_sm<8>();
        (void)gol_tb_per_sm<12>();
        cudaFuncAttributes attr;
        LGD_CHECK_CUDA(cudaFuncGetAttributes(&attr, gol_swar_torus_kernel));
        LGD_CHECK_CUDA(cudaFuncGetAttributes(&attr, gol_generic_kernel));
        return true;
    });
}

static void gol_single(Grid& g, int steps);

void launch_gol(Grid& g, int steps)
{
    prepare_gol_kernels();
    LGD_REQUIRE(g.desc.nz == 1, LGD_ERR_INVALID, "Game of Life grids are 2D (nz = 1)");
    // no depth asked for: packed passes (k_golpack.cu).  Boards that only the
    // byte-wise kernel served before take their first generation with it: it
    // counts cells by their byte values, so bytes other than 0 and 1 keep
    // their meaning, and leaves 0 and 1 behind
    const bool aligned_torus = gol_tb_applicable(g);
    if (g.variant == 0 && g.time_block == 0 && steps >= gol_pack_min(g, aligned_torus) &&
        gol_packed_applicable(g) && gol_packed_ready(g)) {
        if (!aligned_torus) {
            gol_single(g, 1);
            --steps;
        }
        launch_gol_packed(g, steps);
        return;
    }
    // temporal blocking on the torus: bit-sliced passes (rows of a
    // multiple of 32 cells, up to 32 generations) or byte passes (rows of a
    // multiple of 16 cells, up to 12; variant 1 forces these for
    // comparison), then single generations for a remainder of one
    if (g.variant == 0 && gol_bits_applicable(g)) {
        const int depth = (g.time_block == 0) ? GOL_BITS_DEFAULT_DEPTH : std::min(g.time_block, 32);
        if (depth > 1) {
            while (steps >= 2) steps -= gol_bits_pass(g, std::min(depth, steps), g.tb_shape);
        }
    } else if (g.variant <= 1 && aligned_torus) {
        const int depth = (g.time_block == 0) ? 8 : std::min(g.time_block, 12);
        if (depth > 1) {
            while (steps >= 2) steps -= gol_tb_pass(g, std::min(depth, steps), g.tb_shape);
        }
    }
    gol_single(g, steps);
}

// one generation per launch, on bytes
static void gol_single(Grid& g, int steps)
{
    const bool swar = ((g.desc.periodic & 3) == 3) && (g.desc.nx % 16 == 0) && (g.pitch_bytes[0] % 16 == 0);
    const long pitch = (long)g.pitch_bytes[0];
    for (int s = 0; s < steps; ++s) {
        const uint8_t *in = (const uint8_t *)g.m[0].buf[g.cur];
        uint8_t *out = (uint8_t *)g.m[0].buf[1 - g.cur];
        if (swar) {
            const long long work = (long long)(g.desc.nx / 16) * g.desc.ny;
            long long blocks = (work + 255) / 256;
            if (blocks > 152LL * 64) blocks = 152LL * 64;
            gol_swar_torus_kernel<<<(unsigned)blocks, 256, 0, g.stream>>>(in, out, g.desc.nx, g.desc.ny, pitch);
        } else {
            View<const uint8_t> vi;
            vi.p = in;
            vi.pitch = pitch;
            vi.nx = g.desc.nx;
            vi.ny = g.desc.ny;
            vi.nz = 1;
            View<uint8_t> vo;
            vo.p = out;
            vo.pitch = pitch;
            vo.nx = g.desc.nx;
            vo.ny = g.desc.ny;
            vo.nz = 1;
            const long long cells = (long long)g.desc.nx * g.desc.ny;
            long long blocks = (cells + 255) / 256;
            if (blocks > 152LL * 64) blocks = 152LL * 64;
            gol_generic_kernel<<<(unsigned)blocks, 256, 0, g.stream>>>(vi, vo, g.desc.periodic, (uint8_t)g.desc.edge[0]);
        }
        check_launch("game of life");
        ++g.launches;
        g.cur = 1 - g.cur;
    }
}

}  // namespace lgd
