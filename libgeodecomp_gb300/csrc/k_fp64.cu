// Whole-grid kernel of the IEEE FP64 Jacobi-7 cell on cube grids.
//
// GB300's FP64 pipe bounds this cell, not memory and not issue: a chain of
// independent additions measured 498 G operations per second on the whole
// GPU.  Everything here serves to keep that pipe busy and to take work off it:
//   - the multiplication by fl(1/7) runs on the integer pipes, bit for bit
//     (mul_seventh): six FP64 operations per cell instead of seven.  The z
//     loop stays rolled: unrolled, the compiler turns mul_seventh's rare
//     branch into predicated code that pays the FP64 multiplication always
//     (512^3: 72 GLUPS with the multiplication, 78 unrolled, 84 rolled);
//   - every thread owns one cell of a plane and marches a few planes; the
//     cells of a plane are numbered through (no idle lanes whatever nx is)
//     and neighbours come straight from global memory (L1 / L2 hits), so
//     there is no barrier and no tile, and a grid is cut into as many small
//     CTAs as it takes to give every SM an even share.
// Measured (us per step, against the TMA kernel of k_tma.cu before): 24 x 20
// x 16 4.2 against 22.6, 64^3 8.2 against 22.6, 128^3 28.7 against 38.9,
// 512^3 1598 against 1795 (84 GLUPS x 6 operations = 503 G/s: the pipe).
// The sum's order is the cell's own: results are bit-identical to every
// other kernel of the cell.
#include <algorithm>

#include "lgd_internal.h"
#include "k_cells.cuh"
#include "k_fp64.cuh"

namespace lgd {
namespace fp64k {

constexpr int THREADS = 128;

__global__ void __launch_bounds__(THREADS, 16)
jacobi7_f64_kernel(const double *in, double *out, long pitch, int nx, int ny, int nz,
                   int zchunk, double edge)
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
    const bool has_n = y > 0, has_s = y + 1 < ny, has_w = x > 0, has_e = x + 1 < nx;
    const double *p = in + (long)z0 * plane + (long)y * pitch + x;
    double *o = out + (long)z0 * plane + (long)y * pitch + x;
    double b = z0 > 0 ? *(p - plane) : edge;
    double m = *p;
#pragma unroll 1
    for (int z = z0; z < z1; ++z) {
        const double t = z + 1 < nz ? *(p + plane) : edge;
        const double n = has_n ? *(p - pitch) : edge;
        const double s = has_s ? *(p + pitch) : edge;
        const double e = has_e ? *(p + 1) : edge;
        const double w = has_w ? *(p - 1) : edge;
        double acc = __dadd_rn(m, n);
        acc = __dadd_rn(acc, s);
        acc = __dadd_rn(acc, e);
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

// The rule: IEEE Jacobi on a cube (any edge value) whose plane fits 32-bit
// numbering.  The TMA kernel keeps larger planes.
bool jacobi7_f64_applicable(const Grid& g)
{
    return g.desc.cell == LGD_CELL_JACOBI7_F64 && g.desc.periodic == 0 &&
           (long long)g.desc.nx * g.desc.ny < (1ll << 31) - fp64k::THREADS;
}

// Planes per thread: 8 re-read least, but the grid must fall into many more
// CTAs than the SMs hold at once (16), or the last wave leaves the pipe idle,
// so small grids march fewer planes (128^3: 28.7 us at 2 and 4, 30.8 at 8
// and 16; 512^3 does not care).
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
    while (zchunk > 1 && xy * ((g.desc.nz + zchunk - 1) / zchunk) < 40LL * sms) zchunk /= 2;
    zchunk = std::max(zchunk, (g.desc.nz + 65534) / 65535);
    const dim3 grid((unsigned)xy, (unsigned)((g.desc.nz + zchunk - 1) / zchunk));
    launch_dependent(
        fp64k::jacobi7_f64_kernel, grid, fp64k::THREADS, 0, g.stream, (const double *)g.m[0].buf[g.cur], (double *)g.m[0].buf[1 - g.cur], (long)(g.pitch_bytes[0] / 8), g.desc.nx,
        g.desc.ny, g.desc.nz, zchunk, g.desc.edge[0]);
    check_launch("jacobi7 f64");
    ++g.launches;
    g.cur = 1 - g.cur;
}

}  // namespace lgd
