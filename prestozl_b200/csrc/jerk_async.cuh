// Bulk (TMA engine) row copies into shared memory and the bounded wait for
// them, and the status bits the kernels report through.
#pragma once

#include <utility>
#include <cuda_runtime.h>

#include <cstdint>

namespace jerk {

__device__ __forceinline__ unsigned smem_u32(const void *p)
{
    return static_cast<unsigned>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void bulk_row_load(void *dst, const void *src, unsigned bytes,
                                              uint64_t *bar)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;"
                 :: "r"(smem_u32(bar)), "r"(bytes) : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 :: "r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}

// Waits for phase `parity` of the mbarrier; gives up after a bounded number
// of polls (each try_wait itself suspends for a bounded time) and returns
// false.
__device__ __forceinline__ bool bar_wait(uint64_t *bar, unsigned parity)
{
    for (int it = 0; it < (1 << 16); it++) {
        unsigned done;
        asm volatile("{\n\t.reg .pred p;\n\t"
                     "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                     "selp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(done) : "r"(smem_u32(bar)), "r"(parity) : "memory");
        if (done)
            return true;
    }
    return false;
}

// Status bits written by the kernels (read back after each pass).
constexpr unsigned kStatusRind = 1u;     // harmsum: a subharmonic r index left its row
constexpr unsigned kStatusCopy = 2u;     // correlation: a copy into shared memory did not complete
constexpr unsigned kStatusSumCopy = 4u;  // harmsum: the same

// SMs of the current device (queried once; every B200 has 148)
inline int sm_count()
{
    static const int n = [] {
        int dev = 0, v = 0;
        return cudaGetDevice(&dev) == cudaSuccess &&
                       cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) ==
                           cudaSuccess && v > 0
                   ? v : 148;
    }();
    return n;
}

// Lets a kernel take all of the shared memory a CTA may have (carveout: and
// asks for the largest shared-memory share of the SM).
template <class K>
inline cudaError_t smem_attrs(K kernel, bool carveout)
{
    cudaFuncAttributes a;
    cudaError_t e = cudaFuncGetAttributes(&a, kernel);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 227 * 1024 - (int)a.sharedSizeBytes);
    if (e == cudaSuccess && carveout)
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                                 (int)cudaSharedmemCarveoutMaxShared);
    return e;
}

// Launches a kernel that may start while the one before it in the stream runs:
// its CTAs take the SMs that the other's last CTAs leave idle, and the launch
// itself costs no gap.  The kernel before calls let_follow, so that this one
// starts once all of the other's CTAs have; without the call, when they have
// ended.  wait_before returns when the kernel before has ended and its writes
// can be read.  A kernel that needs those calls wait_before first thing; one
// that does not calls it last, so that whatever comes after it finds both
// complete.  A kernel that waits first calls let_follow only after: the one
// that follows may count on all that came before.  What the kernel before wrote
// is not read through __ldg or a const __restrict__ parameter: the compiler may
// move such a read to before the wait.
template <class... Par, class... Arg>
inline cudaError_t launch_follow(void (*kernel)(Par...), dim3 grid, unsigned block, size_t smem,
                                 cudaStream_t st, Arg &&...args)
{
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, std::forward<Arg>(args)...);
    const cudaError_t last = cudaGetLastError();  // as after <<<>>>: read and cleared
    return e != cudaSuccess ? e : last;
}

__device__ __forceinline__ void let_follow()
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

__device__ __forceinline__ void wait_before()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// this CTA's rsteps: all of the batch, or a share of them when a small
// group's rows alone would leave SMs idle (ny > 1 chunks)
__device__ __forceinline__ void rstep_chunk(int nb, int ny, int y, int *b0, int *b1)
{
    const int bchunk = (nb + ny - 1) / ny;
    *b0 = min(nb, y * bchunk);
    *b1 = min(nb, *b0 + bchunk);
}

}  // namespace jerk
