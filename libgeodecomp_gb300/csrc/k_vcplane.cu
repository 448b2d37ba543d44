// Variable-coefficient diffusion, one cell of a plane per thread: FP64 grids of
// any shape and boundary, and the FP32 grids that no tiled kernel takes (rows not
// a multiple of 16 bytes, axes that do not wrap).
//
// The cells of a plane are numbered through, so no lane idles whatever nx is, and
// a thread marches a few planes with u and k of the centre and top in registers;
// the neighbours in the plane are L1 hits.  A grid falls into as many small CTAs
// as give every SM an even share.
//
// FP64 is bound by the FP64 pipe, so of the cell's 30 operations it keeps 11, bit
// for bit: the face to the plane below is the exact negative of the face the
// thread took to its top neighbour one plane earlier, and (k + k') / 2 of the other
// five and its product with the difference of u are integer sums and products.
// Where that does not hold for some cell of a warp (coefficients of zero, negative,
// at the ends of the range or more than nine binary exponents from a neighbour's,
// differences of u at the ends of the range), the warp computes this plane and its
// next ones as written, 26 operations a cell: trying each plane again cost such grids
// more than the pair kernel below (256^3 with half of the coefficients zero, of both
// signs or 2^20 apart 1450 us against its 889; now 880, and 679 with insulating blocks).
// The votes that this takes cost a field that never fails 7% (256^3 380 -> 406 us).
//
// us per step (in brackets the pair kernel of k_stencil.cu: two x cells per lane,
// whose blocks at a grid's ragged end loaded cell by cell): FP64 64^3 10.2 (70), 101 x
// 77 x 60 15.6 (246), 128^3 56 (133), 256^3 406 (888): 41.3 GLUPS x 11 operations =
// 454 G/s of the pipe's 498; FP32 101 x 77 x 60 4.3 (162), 253 x 250 x 250 68 (517).
// Without the votes the products in integers gave 256^3 530 -> 380, the sums before
// them 685 -> 530.
#include <algorithm>

#include "lgd_internal.h"
#include "k_cells.cuh"
#include "k_common.cuh"

namespace lgd {
namespace vcp {

constexpr int THREADS = 128;

// whether half_sum takes a and b
__device__ __forceinline__ bool summable(double a, double b)
{
    const unsigned ha = (unsigned)__double2hiint(a), hb = (unsigned)__double2hiint(b);
    const unsigned e0 = min(ha, hb) >> 20;
    const unsigned sa = (ha >> 20) - e0, sb = (hb >> 20) - e0;          // one of them 0
    const bool alone = (hb | (unsigned)__double2loint(b)) == 0u;
    return alone ? (ha >> 20) - 3u < 2030u : (sa | sb) <= 9u && e0 - 3u < 2030u;
}

// fl((a + b) / 2) of positive doubles in integer arithmetic, as sum4 (k_fp64.cuh)
// adds, b possibly +0 (a zero edge coefficient: then the half is a subtraction from
// the exponent).  Not (summable) for other signs, more than nine binary exponents
// apart and the ends of the exponent range.
__device__ __forceinline__ double half_sum(double a, double b)
{
    const unsigned ha = (unsigned)__double2hiint(a), hb = (unsigned)__double2hiint(b);
    const unsigned e0 = min(ha, hb) >> 20;
    const unsigned sa = (ha >> 20) - e0, sb = (hb >> 20) - e0;
    const unsigned ma = (ha & 0xfffffu) | 0x100000u, mb = (hb & 0xfffffu) | 0x100000u;
    const unsigned la = (unsigned)__double2loint(a), lb = (unsigned)__double2loint(b);
    unsigned long long s = (((unsigned long long)__funnelshift_l(la, ma, sa) << 32) | (la << (sa & 31u))) +
                           (((unsigned long long)__funnelshift_l(lb, mb, sb) << 32) | (lb << (sb & 31u)));
    const unsigned k = 11u - (unsigned)__clz((int)(s >> 32));          // bits to drop, 1 .. 10
    const unsigned unit = 1u << (k & 31u);
    s += (unit >> 1) - 1u + (((unsigned)s >> (k & 31u)) & 1u);
    // s >> k holds the leading bit, which adds one to the exponent field; the half takes it off again
    const bool alone = (hb | lb) == 0u;
    const double half = __longlong_as_double((long long)((s >> (k & 31u)) + ((unsigned long long)(e0 + k - 2u) << 52)));
    return alone ? __hiloint2double((int)(ha - 0x00100000u), (int)la) : half;
}

// fl(a b) of a positive normal a in integer arithmetic (mul_integer of k_fp64.cuh
// takes any sign; 399 us at 256^3 with it, 380 with this one); ok becomes false
// where the exponents or the result's leave the middle of the range.  A product of the
// significands has 105 or 106 bits, hi its top 63 or 64; the rest only matters as
// zero or not.
__device__ __forceinline__ double product(double a, double b, bool& ok)
{
    const unsigned ha = (unsigned)__double2hiint(a), hb = (unsigned)__double2hiint(b);
    const unsigned ea = ha >> 20, eb = (hb >> 20) & 0x7ffu;
    const unsigned long long ma = ((unsigned long long)__double_as_longlong(a) << 11) | 0x8000000000000000ull;
    const unsigned long long mb = ((unsigned long long)__double_as_longlong(b) << 11) | 0x8000000000000000ull;
    const unsigned long long hi = __umul64hi(ma, mb), lo = ma * mb;
    const unsigned big = (unsigned)(hi >> 63), drop = 10u + big;
    const unsigned odd = ((unsigned)hi >> drop) & 1u;
    const unsigned long long m = (hi + ((512u << big) - 1u) + (odd | (lo != 0))) >> drop;
    // m holds its leading bit, which adds one to the exponent field
    const unsigned e = ea + eb + big - 1024u;
    const double r = __longlong_as_double((long long)((m + ((unsigned long long)e << 52)) | ((unsigned long long)(hb & 0x80000000u) << 32)));
    const bool zero = ((hb & 0x7fffffffu) | (unsigned)__double2loint(b)) == 0u;
    ok = ok && (zero || (eb - 1u < 2046u && e - 2u < 2040u));
    return zero ? b : r;
}

// the cell as written (a call: predicated, its operations would be paid always),
// given the face to the plane below
struct Written {
    double r, above;        // the cell, the face to the plane above
};
__device__ __noinline__ Written as_written(double uc, double kc, double uw, double kw, double ue, double ke, double un, double kn,
                                           double us, double ks, double below, double ut, double kt)
{
    double flux = VarCoef<double>::face(uc, kc, uw, kw);
    flux = __dadd_rn(flux, VarCoef<double>::face(uc, kc, ue, ke));
    flux = __dadd_rn(flux, VarCoef<double>::face(uc, kc, un, kn));
    flux = __dadd_rn(flux, VarCoef<double>::face(uc, kc, us, ks));
    flux = __dadd_rn(flux, below);
    const double above = VarCoef<double>::face(uc, kc, ut, kt);
    return {__dadd_rn(uc, __dadd_rn(flux, above)), above};
}

__device__ __forceinline__ bool same_bits(double a, double b)
{
    return __double_as_longlong(a) == __double_as_longlong(b);
}

template<typename R>
struct Args {
    const R *u, *k;
    R *out;
    long pitch;
    int nx, ny, nz, zchunk, periodic;
    R edge_u, edge_k;
};

template<typename R>
__global__ void __launch_bounds__(THREADS, sizeof(R) == 8 ? 6 : 8)
varcoef_plane_kernel(const Args<R> a)
{
    dependent_start();
    const int nx = a.nx, ny = a.ny, nz = a.nz;
    const unsigned c = blockIdx.x * THREADS + threadIdx.x;
    const unsigned lanes = __ballot_sync(0xffffffffu, c < (unsigned)nx * (unsigned)ny);     // below 2^31 (host rule)
    if (c >= (unsigned)nx * (unsigned)ny) return;
    const int y = (int)(c / (unsigned)nx);
    const int x = (int)(c - (unsigned)y * (unsigned)nx);
    const int z0 = blockIdx.y * a.zchunk;
    const int z1 = min(z0 + a.zchunk, nz);
    const long plane = a.pitch * ny;
    const bool wrap_z = a.periodic & 4;
    const bool has_w = x > 0 || (a.periodic & 1), has_e = x + 1 < nx || (a.periodic & 1);
    const bool has_n = y > 0 || (a.periodic & 2), has_s = y + 1 < ny || (a.periodic & 2);
    const int west = x > 0 ? -1 : nx - 1, east = x + 1 < nx ? 1 : 1 - nx;
    const long north = y > 0 ? -a.pitch : (ny - 1) * a.pitch, south = y + 1 < ny ? a.pitch : -(ny - 1) * a.pitch;
    const long at = (long)z0 * plane + (long)y * a.pitch + x;
    const R *u = a.u + at, *k = a.k + at;
    R *o = a.out + at;
    R uc = *u, kc = *k, ub, kb;
    {
        const bool has = z0 > 0 || wrap_z;
        const long d = z0 > 0 ? -plane : (nz - 1) * plane;
        ub = has ? u[d] : a.edge_u;
        kb = has ? k[d] : a.edge_k;
    }
    R below = 0;                                            // FP64: the face to the plane below
    if constexpr (sizeof(R) == 8) below = VarCoef<R>::face(uc, kc, ub, kb);
    bool written = false;       // a cell of the warp was computed as written: so are all of its next ones
#pragma unroll 1
    for (int z = z0; z < z1; ++z) {
        const bool has = z + 1 < nz || wrap_z;
        const long d = z + 1 < nz ? plane : -(nz - 1) * plane;
        const R ut = has ? u[d] : a.edge_u, kt = has ? k[d] : a.edge_k;
        const R un = has_n ? u[north] : a.edge_u, kn = has_n ? k[north] : a.edge_k;
        const R us = has_s ? u[south] : a.edge_u, ks = has_s ? k[south] : a.edge_k;
        const R ue = has_e ? u[east] : a.edge_u, ke = has_e ? k[east] : a.edge_k;
        const R uw = has_w ? u[west] : a.edge_u, kw = has_w ? k[west] : a.edge_k;
        R r;
        if constexpr (sizeof(R) == 8) {
            double above = 0.0;
            if (!written) {
                written = __any_sync(lanes, !(summable(kc, kw) && summable(kc, ke) && summable(kc, kn) && summable(kc, ks) &&
                                              summable(kc, kt)));
            }
            if (!written) {
                bool ok = true;
                auto face = [&](double un, double kn) { return product(half_sum(kc, kn), __dadd_rn(un, -uc), ok); };
                double flux = face(uw, kw);
                flux = __dadd_rn(flux, face(ue, ke));
                flux = __dadd_rn(flux, face(un, kn));
                flux = __dadd_rn(flux, face(us, ks));
                flux = __dadd_rn(flux, below);
                above = face(ut, kt);
                r = __dadd_rn(uc, __dadd_rn(flux, above));
                written = __any_sync(lanes, !ok);
            }
            if (written) {
                const Written w = as_written(uc, kc, uw, kw, ue, ke, un, kn, us, ks, below, ut, kt);
                r = w.r;
                above = w.above;
            }
            // the same face from its other side: the difference of u is the exact
            // negative, but for equal values (+0, or NaN, from both sides)
            below = same_bits(ut, uc) ? above : -above;
        } else {
            r = VarCoef<R>::apply(uc, kc, uw, kw, ue, ke, un, kn, us, ks, ub, kb, ut, kt);
        }
        *o = r;
        ub = uc;
        kb = kc;
        uc = ut;
        kc = kt;
        u += plane;
        k += plane;
        o += plane;
    }
}

// Planes per thread: 8 re-read least, fewer until there are 10 CTAs per SM.  us per
// step with 1, 2, 4, 8 planes, FP64 (with 21 operations): 64^3 14.4, 13.5, 21.6, 39.4; 120 x 96 x 100
// 56.7, 52.3, 50.3, 53.2; 256^3 796, 732, 701, 685; FP32 101 x 77 x 60 5.1, 4.3,
// 5.3, 5.6; 130 x 128 x 128 18.2, 12.4, 10.8, 10.7.
template<typename R>
static void launch(Grid& g, int sms)
{
    const long long xy = ((long long)g.desc.nx * g.desc.ny + THREADS - 1) / THREADS;
    int zchunk = 8;
    while (zchunk > 1 && xy * ((g.desc.nz + zchunk - 1) / zchunk) < 10LL * sms) zchunk /= 2;
    zchunk = std::max(zchunk, (g.desc.nz + 65534) / 65535);
    const Args<R> a = {(const R *)g.m[0].buf[g.cur], (const R *)g.m[1].buf[0], (R *)g.m[0].buf[1 - g.cur],
                       (long)(g.pitch_bytes[0] / sizeof(R)), g.desc.nx, g.desc.ny, g.desc.nz, zchunk, g.desc.periodic,
                       (R)g.desc.edge[0], (R)g.desc.edge[1]};
    launch_dependent(varcoef_plane_kernel<R>, dim3((unsigned)xy, (unsigned)((g.desc.nz + zchunk - 1) / zchunk)), THREADS, 0,
                     g.stream, a);
}

}  // namespace vcp

bool varcoef_plane_applicable(const Grid& g)
{
    return (long long)g.desc.nx * g.desc.ny < (1ll << 31) - vcp::THREADS && g.pitch_bytes[0] == g.pitch_bytes[1];
}

void launch_varcoef_plane(Grid& g)
{
    static PerDevice<int> setup;
    const int sms = setup.get([] {
        int dev = 0, count = 0;
        LGD_CHECK_CUDA(cudaGetDevice(&dev));
        LGD_CHECK_CUDA(cudaDeviceGetAttribute(&count, cudaDevAttrMultiProcessorCount, dev));
        return count;
    });
    if (g.desc.cell == LGD_CELL_VARCOEF_F32) vcp::launch<float>(g, sms);
    else vcp::launch<double>(g, sms);
    check_launch("varcoef plane");
    ++g.launches;
    g.cur = 1 - g.cur;
}

}  // namespace lgd
