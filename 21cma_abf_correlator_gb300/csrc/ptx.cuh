// ptx.cuh -- thin inline-PTX wrappers used by the kernels (sm_103a).
//
// mbarrier + cp.async.bulk (TMA bulk copies) for the F-engine's input prefetch,
// TMA tile loads for the X-engines, and the clock-bounded waits every spin
// in this library goes through: a wait that runs out records a watchdog code in
// a global flag and returns false instead of spinning for ever.

#ifndef CORR_GB300_PTX_CUH
#define CORR_GB300_PTX_CUH

#include <cstdint>
#include <cuda_runtime.h>

namespace corrgb {

// About two seconds at the GB300's 2.07 GHz maximum SM clock.
constexpr long long kWaitBudgetCycles = 4000000000LL;

__device__ __forceinline__ uint32_t smem_addr(const void *p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ uint64_t gmem_addr(const void *p) {
    uint64_t g;
    asm volatile("cvta.to.global.u64 %0, %1;" : "=l"(g) : "l"(p));
    return g;
}

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count)
                 : "memory");
}

// Make mbarrier initialisation visible to the async proxy.
__device__ __forceinline__ void fence_mbar_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

// Order this thread's prior generic-proxy shared-memory accesses before
// subsequent async-proxy (TMA / tcgen05) accesses.
__device__ __forceinline__ void fence_proxy_async_smem() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)),
                 "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// Wait for phase `parity` of `bar` to complete, for at most kWaitBudgetCycles.
// On timeout writes `code` into *err and returns false. With `abort` given, also
// returns false (recording nothing) as soon as *abort becomes non-zero: another
// role of the CTA already gave up and recorded why.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t *bar, uint32_t parity, int *err,
                                                  int code,
                                                  const volatile int *abort = nullptr) {
    if (mbar_try_wait(bar, parity)) return true;
    const long long t0 = clock64();
    while (true) {
        if (mbar_try_wait(bar, parity)) return true;
        if (abort != nullptr && *abort != 0) return false;
        if (clock64() - t0 > kWaitBudgetCycles) {
            if (err != nullptr) atomicExch(err, code);
            return false;
        }
    }
}

// One-dimensional TMA bulk copy global -> shared, completing on `bar` with
// `bytes` transaction bytes. dst/src 16-byte aligned, bytes a multiple of 16.
__device__ __forceinline__ void bulk_copy_g2s(void *dst, const void *src, uint32_t bytes,
                                              uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
            "r"(smem_addr(dst)),
        "l"(gmem_addr(src)), "r"(bytes), "r"(smem_addr(bar))
        : "memory");
}

// 4-D TMA tile load global -> shared, completing on `bar`; `map` is a CUtensorMap in
// kernel parameter space.
__device__ __forceinline__ void tma_load_4d(void *dst, const void *map, int x, int y, int z,
                                            int w, uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes "
        "[%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(smem_addr(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(w),
        "r"(smem_addr(bar))
        : "memory");
}

// Order tcgen05 operations before / after a thread synchronisation.
__device__ __forceinline__ void tc_fence_after() {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_before() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}

// Tensor memory as per-thread storage: warp w of a CTA reaches lanes
// [32*(w%4), 32*(w%4)+32), a lane per thread, one 32-bit word per column.
// alloc/dealloc by one whole warp; n_cols a power of two >= 32. alloc waits while
// other CTAs on the SM hold too many columns.
__device__ __forceinline__ void tmem_alloc(uint32_t *smem_base, uint32_t n_cols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_addr(smem_base)),
                 "r"(n_cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_dealloc(uint32_t base, uint32_t n_cols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(base), "r"(n_cols)
                 : "memory");
}

// Eight float2 of this thread to / from 16 columns (load: complete only after
// tmem_wait8, which the values must pass through).
__device__ __forceinline__ void tmem_store8(uint32_t taddr, const float2 *v) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
        "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr),
        "f"(v[0].x), "f"(v[0].y), "f"(v[1].x), "f"(v[1].y), "f"(v[2].x), "f"(v[2].y), "f"(v[3].x),
        "f"(v[3].y), "f"(v[4].x), "f"(v[4].y), "f"(v[5].x), "f"(v[5].y), "f"(v[6].x), "f"(v[6].y),
        "f"(v[7].x), "f"(v[7].y)
        : "memory");
}

__device__ __forceinline__ void tmem_store_wait() {
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_load8(uint32_t taddr, float2 *v) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=f"(v[0].x), "=f"(v[0].y), "=f"(v[1].x), "=f"(v[1].y), "=f"(v[2].x), "=f"(v[2].y),
          "=f"(v[3].x), "=f"(v[3].y), "=f"(v[4].x), "=f"(v[4].y), "=f"(v[5].x), "=f"(v[5].y),
          "=f"(v[6].x), "=f"(v[6].y), "=f"(v[7].x), "=f"(v[7].y)
        : "r"(taddr));
}

__device__ __forceinline__ void tmem_wait8(float2 *v) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+f"(v[0].x), "+f"(v[0].y), "+f"(v[1].x), "+f"(v[1].y), "+f"(v[2].x),
                   "+f"(v[2].y), "+f"(v[3].x), "+f"(v[3].y), "+f"(v[4].x), "+f"(v[4].y),
                   "+f"(v[5].x), "+f"(v[5].y), "+f"(v[6].x), "+f"(v[6].y), "+f"(v[7].x),
                   "+f"(v[7].y));
}

// *dst += v, performed at L2, with no value returned to the thread.
__device__ __forceinline__ void red_add_f64(double *dst, double v) {
    asm volatile("red.global.add.f64 [%0], %1;" ::"l"(gmem_addr(dst)), "d"(v) : "memory");
}

// {dst[0], dst[1]} += v in FP32, performed at L2, with no value returned; dst 8-byte
// aligned. FP32 reductions take subnormal values of the row for zeros, so nothing is done
// where v is zero (a station that is missing): they stay as they are. A v that is not
// zero is far above them.
__device__ __forceinline__ void red_add_f32x2(float2 *dst, float2 v) {
    if (v.x != 0.0f || v.y != 0.0f)
        asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(gmem_addr(dst)), "f"(v.x),
                     "f"(v.y)
                     : "memory");
}

// dst[0..3] += {a.x, a.y, b.x, b.y} likewise; dst 16-byte aligned. (One test of all four
// values: a test and a way of its own for each pair made the tensor X-engine's launches of
// few frames up to 5 % longer.)
__device__ __forceinline__ void red_add_f32x4(float2 *dst, float2 a, float2 b) {
    const uint32_t any = __float_as_uint(a.x) | __float_as_uint(a.y) | __float_as_uint(b.x) |
                         __float_as_uint(b.y);
    if ((any << 1) != 0u)   // but for the signs
        asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(gmem_addr(dst)),
                     "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y)
                     : "memory");
}

// (double)x in integer arithmetic. This GPU converts (and computes) doubles at
// 2 lanes per SM and cycle; a normal float only needs its exponent moved.
__device__ __forceinline__ double widen(float x) {
    const uint32_t b = __float_as_uint(x), m = b & 0x7fffffffu;
    const bool normal = m - 0x00800000u < 0x7f000000u;
    if (!normal && m != 0) return static_cast<double>(x);   // subnormal, infinite, NaN
    const uint32_t hi = (b & 0x80000000u) | (normal ? (m >> 3) + 0x38000000u : 0u);
    return __hiloint2double(static_cast<int>(hi), static_cast<int>(normal ? b << 29 : 0u));
}

__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
    return make_float2(fmaf(a.x, b.x, -a.y * b.y), fmaf(a.x, b.y, a.y * b.x));
}

// Complex add and subtract as one packed FP32x2 instruction each (sm_100+):
// the same two IEEE round-to-nearest operations as two scalar ones, in half
// the issue slots.
__device__ __forceinline__ float2 cadd(float2 a, float2 b) {
    float2 d;
    asm("{\n\t.reg .b64 pa, pb, pd;\n\t"
        "mov.b64 pa, {%2, %3};\n\t"
        "mov.b64 pb, {%4, %5};\n\t"
        "add.rn.f32x2 pd, pa, pb;\n\t"
        "mov.b64 {%0, %1}, pd;\n\t}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}

// d = a * b lane by lane as one packed FP32x2 multiply (sm_100+).
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
    float2 d;
    asm("{\n\t.reg .b64 pa, pb, pd;\n\t"
        "mov.b64 pa, {%2, %3};\n\t"
        "mov.b64 pb, {%4, %5};\n\t"
        "mul.rn.f32x2 pd, pa, pb;\n\t"
        "mov.b64 {%0, %1}, pd;\n\t}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}

// d = a * b + c lane by lane as one packed FP32x2 fused multiply-add (sm_100+):
// each lane is the IEEE fma of the scalar instruction, in half the issue slots.
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
    float2 d;
    asm("{\n\t.reg .b64 pa, pb, pc, pd;\n\t"
        "mov.b64 pa, {%2, %3};\n\t"
        "mov.b64 pb, {%4, %5};\n\t"
        "mov.b64 pc, {%6, %7};\n\t"
        "fma.rn.f32x2 pd, pa, pb, pc;\n\t"
        "mov.b64 {%0, %1}, pd;\n\t}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return d;
}

__device__ __forceinline__ float2 csub(float2 a, float2 b) {
    float2 d;
    asm("{\n\t.reg .b64 pa, pb, pd;\n\t"
        "mov.b64 pa, {%2, %3};\n\t"
        "mov.b64 pb, {%4, %5};\n\t"
        "sub.rn.f32x2 pd, pa, pb;\n\t"
        "mov.b64 {%0, %1}, pd;\n\t}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}

} // namespace corrgb

#endif // CORR_GB300_PTX_CUH
