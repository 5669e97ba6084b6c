// late_writer.cu -- a kernel that lets its dependents start at once and writes its output late, as an engine's own
// kernel may under programmatic dependent launch.  What a launch after it reads before its dependency wait is the old content.
#include <cuda_runtime.h>
#include <cstdint>
#include <cstddef>

__global__ void __launch_bounds__(256)
k_late_copy(uint32_t* __restrict__ dst, const uint32_t* __restrict__ src, size_t n, unsigned ns) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    unsigned long long t0, t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
    for (int i = 0; i < (1 << 15); ++i) {                    // ends by its count whatever the timer does
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
        if (t - t0 >= ns) break;
        __nanosleep(500);
    }
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) dst[i] = src[i];
}

// bytes: a multiple of 4.  Few and small CTAs, so that the next launch finds room on every SM.
extern "C" int late_copy(void* dst, const void* src, size_t bytes, unsigned us, cudaStream_t stream) {
    k_late_copy<<<32, 256, 0, stream>>>(static_cast<uint32_t*>(dst), static_cast<const uint32_t*>(src), bytes / 4, us * 1000u);
    return (int)cudaGetLastError();
}
