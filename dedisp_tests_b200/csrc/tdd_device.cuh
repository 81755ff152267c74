// Device helpers shared by the time-domain kernels: the output epilogue, the
// integer delay, bounded mbarrier waits and bulk copies, shared loads, and
// the work-item loop of the persistent multi-beam kernels.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "runtime.hpp"
#include "tdd_kernels.hpp"

namespace dedisp {
namespace kern {
namespace {

// ---------------------------------------------------------------------------
// Epilogue: src/tdd/dedisperse/dedisperse_kernel.cuh:45-87
// ---------------------------------------------------------------------------
__device__ __forceinline__ float sum_to_float(uint32_t s) { return __uint2float_rn(s); }
__device__ __forceinline__ float sum_to_float(unsigned long long s) { return __ull2float_rn(s); }

template <typename S>
__device__ __forceinline__ void store_out(void* out, size_t idx, int out_nbits, S sum,
                                          float den, float factor)
{
    const float fs = sum_to_float(sum);
    if (out_nbits == 32) {
        // out_range == 1.f: (fs * 1.f) == fs exactly
        static_cast<float*>(out)[idx] = __fmul_rn(__fdiv_rn(fs, den), factor);
    } else {
        const float out_range = (out_nbits == 8) ? 255.f : 65535.f;
        float v = __fmul_rn(__fdiv_rn(__fmul_rn(fs, out_range), den), factor);
        // min(max(v, 0.), out_range) in double equals the float clip here:
        // both bounds are exact floats and v is never NaN.
        v = fminf(fmaxf(v, 0.f), out_range);
        if (out_nbits == 8) static_cast<uint8_t*>(out)[idx] = (uint8_t)__float2uint_rz(v);
        else static_cast<uint16_t*>(out)[idx] = (uint16_t)__float2uint_rz(v);
    }
}

__device__ __forceinline__ uint32_t delay_rn(float dm, float delay)
{
    // src/tdd/dedisperse/dedisperse_kernel.cuh:163-165
    return __float2uint_rn(__fmul_rn(dm, delay));
}

// mbarrier + bulk asynchronous copy (global -> shared of this CTA only).
__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint64_t* b, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(b)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_inval(uint64_t* b)
{
    asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(smem_addr(b)) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* b, uint32_t bytes)
{
    asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(b)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* b)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(b)) : "memory");
}
// `bytes` (a multiple of 16) from global `src` to shared `dst` (both 16-byte
// aligned); completion counted on mbarrier b.
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* b)
{
    asm volatile("cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_addr(dst)),
                 "l"(src), "r"(bytes), "r"(smem_addr(b))
                 : "memory");
}
// Limit of the bounded mbarrier waits (nanoseconds of global time) and the
// expiry test switch (rt::wait_limit_ns, rt::wait_expiry_test), passed to
// the kernels by value.
struct WaitCfg {
    unsigned long long ns;
    int expiry_test;
};
inline WaitCfg wait_cfg() { return WaitCfg{rt::wait_limit_ns(), rt::wait_expiry_test() ? 1 : 0}; }

// Wait for phase `parity` of b; false after limit_ns of global time (checked
// every 16 polls) or 2^28 polls.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* b, uint32_t parity, unsigned long long limit_ns)
{
    const uint32_t addr = smem_addr(b);
    uint64_t t0 = 0;
    for (uint32_t i = 0; i < (1u << 28); ++i) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(addr), "r"(parity)
            : "memory");
        if (done) return true;
        if ((i & 15u) == 15u) {
            uint64_t t;
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
            if (t0 == 0) t0 = t;
            else if (t - t0 > limit_ns) return false;
        }
    }
    return false;
}
__device__ __forceinline__ uint32_t imad(uint32_t a, uint32_t b, uint32_t c)
{
    uint32_t d;
    asm("mad.lo.u32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}

__device__ __forceinline__ uint4 lds128(uint32_t addr)
{
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];\n"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "r"(addr));
    return v;
}

// Persistent form over many series (beams): block b takes work items b,
// b + gridDim.x, ...; item i belongs to the beam with
// item_start[beam] <= i < item_start[beam + 1] and is tile
// (bx, by) = (local % nbx, local / nbx) of that beam. Each beam's arguments
// are copied to shared memory before its tiles run. TILE runs one tile.
template <typename TILE>
__device__ __forceinline__ void batch_items(const DedisperseArgs* __restrict__ args,
                                            const unsigned long long* __restrict__ item_start,
                                            const int* __restrict__ nbx, int nbeams, TILE&& tile)
{
    __shared__ DedisperseArgs s_a;
    __shared__ int s_beam;
    const unsigned long long total = item_start[nbeams];
    int cur = -1;
    for (unsigned long long item = blockIdx.x; item < total; item += gridDim.x) {
        if (threadIdx.x == 0) {
            int lo = 0, hi = nbeams - 1;  // last beam with item_start <= item
            while (lo < hi) {
                const int mid = (lo + hi + 1) / 2;
                if (item_start[mid] <= item) lo = mid;
                else hi = mid - 1;
            }
            s_beam = lo;
        }
        __syncthreads();
        const int beam = s_beam;
        if (beam != cur) {
            constexpr int NWORDS = (int)(sizeof(DedisperseArgs) / 4);
            static_assert(sizeof(DedisperseArgs) % 4 == 0, "argument block is copied as words");
            const uint32_t* src = reinterpret_cast<const uint32_t*>(args + beam);
            uint32_t* dst = reinterpret_cast<uint32_t*>(&s_a);
            for (int w = threadIdx.x; w < NWORDS; w += blockDim.x) dst[w] = src[w];
            cur = beam;
        }
        __syncthreads();
        const unsigned long long local = item - item_start[beam];
        const int n = nbx[beam];
        tile(s_a, (int)(local % (unsigned long long)n), (size_t)(local / (unsigned long long)n));
        __syncthreads();  // shared memory is reused by the next item
    }
}

}  // namespace
}  // namespace kern
}  // namespace dedisp
