// msod_device.cuh -- device-side building blocks shared by the msod kernels.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "msod.h"

namespace msod {

// Fire-and-forget global reductions (no return value): the element-to-node
// scatter of the residuals (the reference's "!$acc atomic update",
// elem_convec.f90:412-426, elem_diffu.f90:182-192).
__device__ __forceinline__ void red_add(float *addr, float v)
{
    asm volatile("red.global.add.f32 [%0], %1;" ::"l"(addr), "f"(v) : "memory");
}
__device__ __forceinline__ void red_add(double *addr, double v)
{
    asm volatile("red.global.add.f64 [%0], %1;" ::"l"(addr), "d"(v) : "memory");
}

// Programmatic dependent launch: let the next kernel of the stream start; wait
// until the kernel ahead (if this one was launched after it that way) has
// finished and its writes are visible.
__device__ __forceinline__ void grid_dependents_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void grid_dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// The statistics' norm, once the kernel that forms it has finished (it may be
// the kernel ahead that this one overlaps).
__device__ __forceinline__ float entropy_norm(const float *norm)
{
    grid_dependency_wait();
    return *const_cast<const volatile float *>(norm);
}

// Read-only global loads through the non-coherent path.
template <typename T>
__device__ __forceinline__ T ldg(const T *p)
{
    return __ldg(p);
}

// Gathers of node fields and element rows: through L2 only (a block reads a
// sector of them once; what is left of the L1 beside the shared memory holds
// fewer lines than a block has in flight).  Diffusion, porder 7 on 32^3 hexes
// 0.791 against 0.817 ms through L1, porder 6 on 40^3 1.005 / 1.033, porder 4 on
// 64^3 0.951 / 0.961; convection, porder 7 0.781 / 0.795, porder 4 0.941 / 0.936.
template <typename T>
__device__ __forceinline__ T ldg_once(const T *p)
{
    return __ldcg(p);
}

// Order-preserving map of a float onto a signed int (for integer atomics).
__device__ __forceinline__ int f2key(float f)
{
    const int i = __float_as_int(f);
    return i >= 0 ? i : i ^ 0x7FFFFFFF;
}
__device__ __forceinline__ float key2f(int k) { return __int_as_float(k >= 0 ? k : k ^ 0x7FFFFFFF); }

// ---------------------------------------------------------------------------
// 1-D bulk copies (cp.async.bulk, the TMA engine's untiled form) completing on
// a shared-memory mbarrier.  Used to stage the contiguous per-group spans of
// He and gpvol: one elected thread issues the copy, no other thread spends an
// instruction or a register on it, and the data land in shared memory without
// passing through the L1 sector path.
// ---------------------------------------------------------------------------
__device__ __forceinline__ unsigned smem_u32(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(unsigned long long *bar, unsigned count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
// One arrival that also expects `bytes` of asynchronous copies on this phase.
__device__ __forceinline__ void mbar_arrive_expect_tx(unsigned long long *bar, unsigned bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}
// dst (shared) <- src (global), `bytes` bytes; both addresses 16-byte aligned,
// bytes a multiple of 16.
__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, unsigned bytes, unsigned long long *bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}
__device__ __forceinline__ bool mbar_test(unsigned long long *bar, unsigned parity)
{
    unsigned ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// Waits for the phase of the given parity to complete, for at most about
// 2^20 polls (~0.1 s with the back-off; a healthy copy of a group's span
// completes in microseconds).  Returns false if the limit ran out; by then the
// copies have had as long again, so that a late one does not outlive the block
// that gives up on it.
__device__ __forceinline__ bool mbar_wait(unsigned long long *bar, unsigned parity)
{
    constexpr int limit = 1 << 20;
    for (int it = 0; it < 2 * limit; ++it) {
        if (mbar_test(bar, parity)) return it < limit;
        if (it >= 32) __nanosleep(64);
    }
    return false;
}

// L2 prefetch of the 16-byte-aligned interior of [p, p + nbytes) by the bulk
// copy unit (one thread; a hint with nothing to wait for; no byte outside the
// span is touched).  No memory clobber: the prefetch writes nothing, and a
// clobber would keep the compiler from moving loads across it.
__device__ __forceinline__ void prefetch_span_l2(const void *p, size_t nbytes)
{
    const size_t a = reinterpret_cast<size_t>(p);
    const size_t a16 = (a + 15) & ~(size_t)15, e16 = (a + nbytes) & ~(size_t)15;
    if (a16 < e16)
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(a16), "r"((unsigned)(e16 - a16)));
}

// A contiguous global span [src, src + bytes) staged in shared memory at
// dst_base + (src mod 16): the 16-byte-aligned interior by one bulk copy, the
// unaligned head and tail (at most 12 bytes each; spans are 4-byte aligned) by
// threads 0..5 with plain loads.  Returns the bulk bytes the caller's
// mbar_arrive_expect_tx must announce.  Thread `issuer` issues the copy;
// dst_base is 16-byte aligned and holds bytes + 32.
struct SpanPlan {
    const char *src;
    unsigned bytes, head, bulk, tail, shift;
    __device__ __forceinline__ SpanPlan(const void *p, size_t nbytes)
    {
        src = static_cast<const char *>(p);
        const size_t a = reinterpret_cast<size_t>(src);
        shift = (unsigned)(a & 15);
        bytes = (unsigned)nbytes;
        const size_t a16 = (a + 15) & ~(size_t)15, e = a + nbytes, e16 = e & ~(size_t)15;
        if (a16 < e16) {
            head = (unsigned)(a16 - a);
            bulk = (unsigned)(e16 - a16);
            tail = (unsigned)(e - e16);
        } else {
            head = (unsigned)nbytes;
            bulk = 0;
            tail = 0;
        }
    }
    // The bulk part (one thread).
    __device__ __forceinline__ void issue(char *dst_base, unsigned long long *bar) const
    {
        if (bulk) bulk_g2s(dst_base + shift + head, src + head, bulk, bar);
    }
    // Head and tail words: word w < 3 of the head, 3 <= w < 6 of the tail (threads 0..5);
    // all of the span when it is too short for a bulk part.
    __device__ __forceinline__ void plain(char *dst_base, int w) const
    {
        if (bulk == 0) {
            for (unsigned o = 4u * (unsigned)w; o < bytes; o += 24u)
                *reinterpret_cast<float *>(dst_base + shift + o) = __ldg(reinterpret_cast<const float *>(src + o));
            return;
        }
        if (w < 3) {
            const unsigned o = 4u * (unsigned)w;
            if (o < head)
                *reinterpret_cast<float *>(dst_base + shift + o) = __ldg(reinterpret_cast<const float *>(src + o));
        } else if (w < 6) {
            const unsigned o = head + bulk + 4u * (unsigned)(w - 3);
            if (o < bytes)
                *reinterpret_cast<float *>(dst_base + shift + o) = __ldg(reinterpret_cast<const float *>(src + o));
        }
    }
};

// Appends e to list[*count ..] for every lane whose f is set, with one atomic
// per warp; every lane of the warp calls it (the list order is unspecified).
__device__ __forceinline__ void warp_append(bool f, int e, int *list, int *count)
{
    const unsigned m = __ballot_sync(0xffffffffu, f);
    const int lane = threadIdx.x & 31;
    int base = 0;
    if (m && lane == __ffs(m) - 1) base = atomicAdd(count, __popc(m));
    base = __shfl_sync(0xffffffffu, base, m ? __ffs(m) - 1 : 0);
    if (f) list[base + __popc(m & ((1u << lane) - 1u))] = e;
}

// Grid of a persistent kernel: resident blocks per SM x SMs, capped by the work.
template <typename Kernel>
inline int persistent_grid(Kernel kern, int threads, size_t smem, int ngroups)
{
    int dev = 0, sms = 0, per = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kern, threads, smem) != cudaSuccess) return 0;
    if (per < 1) per = 1;
    const long long g = (long long)sms * per;
    return (int)(g < ngroups ? g : ngroups);
}

}  // namespace msod
