// Whole-grid kernel of the IEEE FP64 Jacobi-7 cell, for any edge value and any
// axes that wrap.
//
// GB300's FP64 pipe bounds this cell, not memory and not issue: a chain of
// independent additions measured 498 G operations per second on the whole
// GPU.  Everything here serves to keep that pipe busy and to take work off it:
//   - the multiplication by fl(1/7) runs on the integer pipes, bit for bit
//     (mul_seventh), and so do the first three of the six additions (sum4):
//     three FP64 operations per cell instead of seven.  Three is where the
//     FP64 and the integer work take about the same time: at 512^3, in us per
//     step, 1600 with no addition in integers, 1110 with two, 916 with three,
//     1140 with four, 1376 with all six (measured without the one-sided
//     neighbour's rule below and with plain launches).  Where sum4's condition
//     fails in some lane (both signs, zeros, far apart) the warp adds in FP64
//     after all; four +0, an empty part of the field, it does not add.  Smooth
//     fields meet the condition but for the cells beside a zero edge in y; the zero
//     east of the last column is dropped (drop_e);
//   - the rare branches must stay branches: predicated, their FP64 operations
//     would be paid always.  So the z loop stays rolled, and sum4's fallback is
//     a loop;
//   - every thread owns one cell of a plane and marches a few planes; the
//     cells of a plane are numbered through (no idle lanes whatever nx is)
//     and neighbours come straight from global memory (L1 / L2 hits), so
//     there is no barrier and no tile, and a grid is cut into as many small
//     CTAs as it takes to give every SM an even share.
// Measured (us per step, uniform in [0, 1); in brackets the kernel without sum4, then
// the TMA kernel of k_tma.cu): 24 x 20 x 16 1.9 (2.2, 22.6), 64^3 4.0 (5.9, 22.6), 128^3
// 17.2 (25.4, 39.1), 512^3 914 (1598, 1795): 147 GLUPS, 88% of the FP64 pipe's rate at
// three operations per cell.  On a torus, against the register kernel: 64^3 4.3 (45),
// 128^3 19.0 (51), 512^3 1066 (1851).  Other fields, 512^3, cube / torus: of both signs
// 1566 / 1786, a hot spot in an empty field 1058 / 1278 (adding its zeros 1822 / 2040),
// exponents up to 30 apart 1083 / 1252.
// The sum's order is the cell's own: results are bit-identical to every
// other kernel of the cell.
#include <algorithm>

#include "lgd_internal.h"
#include "k_cells.cuh"
#include "k_fp64.cuh"

namespace lgd {
namespace fp64k {

constexpr int THREADS = 128;
constexpr int CTAS = 8;        // per SM: 64 registers

__device__ __forceinline__ bool any_bit(double a, double b, double c, double d)
{
    return ((__double_as_longlong(a) | __double_as_longlong(b)) | (__double_as_longlong(c) | __double_as_longlong(d))) != 0;
}

// WRAP: some axis wraps (a cube of 512^3 takes 886 us without, 1030 with)
template<bool WRAP>
__global__ void __launch_bounds__(THREADS, CTAS)
jacobi7_f64_kernel(const double *in, double *out, long pitch, int nx, int ny, int nz,
                   int zchunk, double edge, int periodic)
{
    dependent_start();
    const unsigned cells = (unsigned)nx * (unsigned)ny;         // below 2^31 (host rule)
    const unsigned c = blockIdx.x * THREADS + threadIdx.x;
    if (c >= cells) return;
    const int y = (int)(c / (unsigned)nx);
    const int x = (int)(c - (unsigned)y * (unsigned)nx);
    const int z0 = blockIdx.y * zchunk;
    const int z1 = min(z0 + zchunk, nz);
    const long plane = pitch * ny;
    // the neighbours in the plane: a fixed distance, around the torus at its
    // ends, or the edge value
    const bool wrap_x = WRAP && (periodic & 1), wrap_y = WRAP && (periodic & 2), wrap_z = WRAP && (periodic & 4);
    const bool has_n = wrap_y || y > 0, has_s = wrap_y || y + 1 < ny;
    const bool has_w = wrap_x || x > 0, has_e = wrap_x || x + 1 < nx;
    const long north = !WRAP || y > 0 ? -pitch : (ny - 1) * pitch, south = !WRAP || y + 1 < ny ? pitch : -(ny - 1) * pitch;
    const int west = !WRAP || x > 0 ? -1 : nx - 1, east = !WRAP || x + 1 < nx ? 1 : 1 - nx;
    const bool drop_e = !has_e && edge == 0.0;      // the sum of the others is not zero where it is taken
    const double *p = in + (long)z0 * plane + (long)y * pitch + x;
    double *o = out + (long)z0 * plane + (long)y * pitch + x;
    double b = z0 > 0 ? *(p - plane) : (wrap_z ? *(p + (nz - 1) * plane) : edge);
    double m = *p;
#pragma unroll 1
    for (int z = z0; z < z1; ++z) {
        const double t = z + 1 < nz ? *(p + plane) : (wrap_z ? *(p - (nz - 1) * plane) : edge);
        const double n = has_n ? *(p + north) : edge;
        const double s = has_s ? *(p + south) : edge;
        const double e = has_e ? *(p + east) : edge;
        const double w = has_w ? *(p + west) : edge;
        double acc;
        if (!sum4(m, n, s, e, drop_e, acc)) {
            acc = m;
            const int adds = any_bit(m, n, s, e) ? 3 : 0;               // +0 four times sum to +0
#pragma unroll 1
            for (int i = 0; i < adds; ++i) acc = __dadd_rn(acc, i == 0 ? n : (i == 1 ? s : e));
        }
        acc = __dadd_rn(acc, w);
        acc = __dadd_rn(acc, t);
        acc = __dadd_rn(acc, b);
        *o = mul_seventh(acc);
        b = m;
        m = t;
        p += plane;
        o += plane;
    }
}

}  // namespace fp64k

// The rule: IEEE Jacobi whose plane fits 32-bit numbering.  The TMA kernel (cube,
// zero edge) and the register kernels keep larger planes.
bool jacobi7_f64_applicable(const Grid& g)
{
    return g.desc.cell == LGD_CELL_JACOBI7_F64 &&
           (long long)g.desc.nx * g.desc.ny < (1ll << 31) - fp64k::THREADS;
}

// Planes per thread: 8 re-read least, but the grid must fall into more CTAs
// than the SMs hold at once (8), or the last wave leaves the pipe idle, so small
// grids march fewer planes until there are 20 CTAs per SM.  us per step with 1,
// 2, 4, 8 planes: 64^3 4.0, 4.8, 7.3, 10.4 (13 CTAs per SM at one plane); 96^3
// 9.3, 8.5, 9.0, 14.0 (23 at two); 128^3 19.7, 17.4, 17.1, 18.0 (27 at four);
// 512^3 1189, 1005, 920, 886.
void launch_jacobi7_f64(Grid& g)
{
    static PerDevice<int> setup;
    const int sms = setup.get([] {
        int dev = 0, count = 0;
        LGD_CHECK_CUDA(cudaGetDevice(&dev));
        LGD_CHECK_CUDA(cudaDeviceGetAttribute(&count, cudaDevAttrMultiProcessorCount, dev));
        return count;
    });
    const long long xy = ((long long)g.desc.nx * g.desc.ny + fp64k::THREADS - 1) / fp64k::THREADS;
    int zchunk = 8;
    while (zchunk > 1 && xy * ((g.desc.nz + zchunk - 1) / zchunk) < 20LL * sms) zchunk /= 2;
    zchunk = std::max(zchunk, (g.desc.nz + 65534) / 65535);
    const dim3 grid((unsigned)xy, (unsigned)((g.desc.nz + zchunk - 1) / zchunk));
    launch_dependent(
        g.desc.periodic & 7 ? fp64k::jacobi7_f64_kernel<true> : fp64k::jacobi7_f64_kernel<false>, grid, fp64k::THREADS, 0, g.stream, (const double *)g.m[0].buf[g.cur], (double *)g.m[0].buf[1 - g.cur], (long)(g.pitch_bytes[0] / 8), g.desc.nx,
        g.desc.ny, g.desc.nz, zchunk, g.desc.edge[0], g.desc.periodic);
    check_launch("jacobi7 f64");
    ++g.launches;
    g.cur = 1 - g.cur;
}

}  // namespace lgd
