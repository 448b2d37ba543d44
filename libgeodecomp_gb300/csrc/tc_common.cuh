// Fifth-generation tensor core helpers of the surrogate's kernels: barriers
// with bounded waits, shared-memory and instruction descriptors, MMA issue,
// tensor memory access.
#ifndef LGD_TC_COMMON_CUH
#define LGD_TC_COMMON_CUH

#include <cuda_bf16.h>
#include <stdint.h>

namespace lgd {
namespace sur {
namespace tc {

typedef __nv_bfloat16 bf16;

constexpr long long WAIT_CYCLES = 4000000000LL;     // about two seconds

__device__ __forceinline__ uint32_t saddr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Matrix descriptors (no swizzle): start address, leading and stride offsets in
// 16-byte units, descriptor version 1; see desc_lo and desc_hi.

// kind::f16 instruction descriptor: FP32 accumulator, BF16 operands; mn: both
// operands with M / N contiguous instead of K
__host__ __device__ constexpr uint32_t idesc(int m, int n, bool mn)
{
    return (1u << 4) | (1u << 7) | (1u << 10) | (mn ? (3u << 15) : 0u) | ((uint32_t)(n >> 3) << 17) |
           ((uint32_t)(m >> 4) << 24);
}

// One lane of a converged warp.  The MMA warp runs its loop with all lanes and
// elects one around each batch of MMAs: loop variables and descriptors then
// stay in uniform registers.  Under a branch on the lane number every MMA
// first moves its operands there, and with the epilogue warps competing for
// issue slots an MMA of 52 clocks took 107.
__device__ __forceinline__ bool elect_one()
{
    uint32_t r;
    asm volatile(
        "{\n"
        " .reg .pred p;\n"
        " elect.sync _|p, 0xffffffff;\n"
        " selp.u32 %0, 1, 0, p;\n"
        "}\n"
        : "=r"(r));
    return r != 0;
}

// descriptors as their low words (start address and leading offset, which
// change from MMA to MMA) and constant high words; ACC: add to D
__device__ __forceinline__ uint64_t desc(uint32_t lo, uint32_t hi) { return ((uint64_t)hi << 32) | lo; }

__host__ __device__ constexpr uint32_t desc_hi(uint32_t sbo) { return ((sbo >> 4) & 0x3FFFu) | (1u << 14); }

__device__ __forceinline__ uint32_t desc_lo(uint32_t addr, uint32_t lbo)
{
    return ((addr >> 4) & 0x3FFFu) | (((lbo >> 4) & 0x3FFFu) << 16);
}

template<bool ACC>
__device__ __forceinline__ void mma(uint32_t dtmem, uint64_t a, uint64_t b, uint32_t id)
{
    asm volatile(
        "{\n"
        " .reg .pred p;\n"
        " setp.eq.u32 p, 1, %4;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n"
        "}\n" ::"r"(dtmem),
        "l"(a), "l"(b), "r"(id), "n"(ACC ? 1 : 0)
        : "memory");
}

__device__ __forceinline__ void mma_commit(uint32_t bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// 24 consecutive columns of this thread's tensor-memory lane, eight, and one.
// The loaded values pass through the wait, so that none is used before it: the
// order of volatile statements alone does not hold arithmetic on them back.
__device__ __forceinline__ void tmem_ld24(uint32_t taddr, float (&v)[24])
{
    uint32_t r[24];
#pragma unroll
    for (int c = 0; c < 24; c += 8) {
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                     : "=r"(r[c]), "=r"(r[c + 1]), "=r"(r[c + 2]), "=r"(r[c + 3]), "=r"(r[c + 4]), "=r"(r[c + 5]),
                       "=r"(r[c + 6]), "=r"(r[c + 7])
                     : "r"(taddr + (uint32_t)c)
                     : "memory");
    }
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                   "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]),
                   "+r"(r[16]), "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]), "+r"(r[22]), "+r"(r[23])
                 :
                 : "memory");
#pragma unroll
    for (int i = 0; i < 24; ++i) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float (&v)[8])
{
    uint32_t r[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr)
                 : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7])
                 :
                 : "memory");
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ void tmem_st8(uint32_t taddr, const float (&v)[8])
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr),
                 "r"(__float_as_uint(v[0])), "r"(__float_as_uint(v[1])), "r"(__float_as_uint(v[2])),
                 "r"(__float_as_uint(v[3])), "r"(__float_as_uint(v[4])), "r"(__float_as_uint(v[5])),
                 "r"(__float_as_uint(v[6])), "r"(__float_as_uint(v[7]))
                 : "memory");
}

__device__ __forceinline__ float tmem_ld1(uint32_t taddr)
{
    uint32_t r;
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];" : "=r"(r) : "r"(taddr) : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" : "+r"(r) : : "memory");
    return __uint_as_float(r);
}

__device__ __forceinline__ void tmem_st1(uint32_t taddr, float v)
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x1.b32 [%0], {%1};" ::"r"(taddr), "r"(__float_as_uint(v)) : "memory");
}

__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile(
        "{\n"
        " .reg .pred p;\n"
        " mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n"
        "}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}

// bounded wait that also gives up once another role has failed
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int *fail)
{
    if (mbar_try(bar, parity)) return true;
    const long long t0 = clock64();
    while (!mbar_try(bar, parity)) {
        if ((fail && *fail) || clock64() - t0 > WAIT_CYCLES) return false;
    }
    return true;
}

__device__ __forceinline__ void bulk_copy(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(reinterpret_cast<uint64_t>(src)), "r"(bytes), "r"(bar)
                 : "memory");
}

__device__ __forceinline__ void copy16(uint32_t dst, const void *src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}

__device__ __forceinline__ void fence_async_proxy() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi)
{
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);     // one conversion for the pair
    return *reinterpret_cast<const uint32_t *>(&v);
}

// GELU(z) = z Phi(z) of two values, and GELU'(z) = Phi(z) + z phi(z) where
// asked for, each from packed FMAs, one reciprocal and one exponential:
//   |z| < 1   Phi = 1/2 + z Q(z^2), Q of degree 4 (error of the fit below 1.3e-8)
//   else      Phi(-|z|) = exp(-z^2 / 2) t P(t) with t = 1 / (1 + p |z|): the
//             function exp(z^2 / 2) Phi(-z) / t is smooth in t, and P its
//             polynomial of degree 6 (relative error of the fit below 1.0e-7 up to
//             z = 14; p chosen for the smallest)
// Both are least-squares fits with weights moved towards the largest error until
// that stopped falling.  In FP32, over -16 .. 16, GELU is within 4e-7 (4.5e-7 with
// erff) and GELU' within 1.4e-7; relative to itself Phi's lower tail is within 1.0e-6
// to z = -4 and 9e-6 to z = -13.2, where the exponential's result is flushed to
// zero.  erff and expf took twice the instructions, which set the time of a layer's
// epilogue.
template<bool GRAD>
__device__ __forceinline__ void gelu_pair(float2 z, float2& h, float2& g)
{
    constexpr float P = 0.395f;
    constexpr float C[7] = {0.15760743f, 0.15697990f, 0.13892886f, 0.052616711f,
                            0.11542270f, -0.18699883f, 0.065657586f};
    constexpr float Q[5] = {0.39894220f, -0.066488728f, 0.0099641671f, -0.0011653511f, 0.000092468512f};
    const float2 d = __ffma2_rn(make_float2(fabsf(z.x), fabsf(z.y)), make_float2(P, P), make_float2(1.0f, 1.0f));
    const float2 s = __fmul2_rn(z, z);
    const float2 q = __fmul2_rn(s, make_float2(-0.72134752f, -0.72134752f));        // -z^2 / (2 ln 2)
    float2 t, e;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(t.x) : "f"(d.x));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(t.y) : "f"(d.y));
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e.x) : "f"(q.x));
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e.y) : "f"(q.y));
    float2 p = make_float2(C[6], C[6]), r = make_float2(Q[4], Q[4]);
#pragma unroll
    for (int i = 5; i >= 0; --i) p = __ffma2_rn(p, t, make_float2(C[i], C[i]));
#pragma unroll
    for (int i = 3; i >= 0; --i) r = __ffma2_rn(r, s, make_float2(Q[i], Q[i]));
    r = __ffma2_rn(r, z, make_float2(0.5f, 0.5f));
    const float2 te = __fmul2_rn(t, e);
    // Phi = te P below -1, 1 - te P above 1
    float2 phi = make_float2(z.x >= 0.0f ? fmaf(-p.x, te.x, 1.0f) : p.x * te.x,
                             z.y >= 0.0f ? fmaf(-p.y, te.y, 1.0f) : p.y * te.y);
    phi.x = s.x < 1.0f ? r.x : phi.x;
    phi.y = s.y < 1.0f ? r.y : phi.y;
    h = __fmul2_rn(z, phi);
    if (GRAD) g = __ffma2_rn(__fmul2_rn(e, make_float2(0.39894228f, 0.39894228f)), z, phi);
}

// Ghosted activations of the tensor-core path: BF16
// [batch][nz + 2][ny + 2][3 channel groups][nx + 2][8 channels], the torus'
// wrapped neighbours in a one-voxel layer; element offset of 8 channels
struct Shape {
    int nx, ny, nz, batch;
};

__host__ __device__ __forceinline__ long long ghost_row(const Shape& s, int b, int z, int y)
{
    return (((long long)b * (s.nz + 2) + z) * (s.ny + 2) + y) * 3;      // times (nx + 2) * 8, channel group 0
}

}  // namespace tc
}  // namespace sur
}  // namespace lgd

#endif
