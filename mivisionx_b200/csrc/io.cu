// io.cu -- array transfers between device arrays and page-locked, device-mapped host
// buffers, as kernels a captured CUDA graph can hold.  AGO keeps an array's item count in
// its device buffer header (DATA_GPU_ARRAY_OFFSET, ago_internal.h:171) and reads it back
// with a blocking copy before the items (ago_util_hip.cpp:321-608); here the count word
// and the items cross PCIe inside the graph, so a graph's array inputs and outputs cost no
// host round trip per array.
#include "agocuda_internal.cuh"

uint64_t agocuda_count_launch(unsigned n);

namespace {

constexpr int kIoThreads = 256;
constexpr int kIoBlocks = 16;

// `words` elements by all threads of the grid's x dimension, four loads of a thread in flight: across
// PCIe each is a round trip (eight lists of 1 MB through the four blocks of their group: 684 us with
// one load in flight, 240 us so, 35 GB/s; 310 us by 16 blocks for each list)
template <class T> __device__ __forceinline__ void copy_words(T *d, const T *s, size_t words)
{
    const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x, n = (size_t)gridDim.x * blockDim.x;
    for (size_t i = t; i < words; i += 4 * n) {
        T v[4];
#pragma unroll
        for (int k = 0; k < 4; k++)
            if (i + k * n < words) v[k] = s[i + k * n];
#pragma unroll
        for (int k = 0; k < 4; k++)
            if (i + k * n < words) d[i + k * n] = v[k];
    }
}

__device__ __forceinline__ void copy_bytes(uint8_t *dst, const uint8_t *src, size_t bytes)
{
    if ((((uintptr_t)dst | (uintptr_t)src) & 15) == 0) {
        const size_t whole = bytes & ~(size_t)15;
        copy_words((uint4 *)dst, (const uint4 *)src, bytes / 16);
        copy_words(dst + whole, src + whole, bytes - whole);
    } else if ((((uintptr_t)dst | (uintptr_t)src | bytes) & 3) == 0) {
        copy_words((uint32_t *)dst, (const uint32_t *)src, bytes / 4);
    } else {
        copy_words(dst, src, bytes);
    }
}

__global__ void __launch_bounds__(kIoThreads)
k_array_upload(uint8_t *dev, uint32_t *devCount, const uint8_t *host, const volatile uint32_t *slot,
               uint32_t itemSize, uint32_t capacity)
{
    __shared__ uint32_t n;
    if (threadIdx.x == 0) n = *slot;
    __syncthreads();
    if (n == AGOCUDA_ARRAY_SKIP) return;
    const uint32_t m = min(n, capacity);
    copy_bytes(dev, host, (size_t)m * itemSize);
    if (blockIdx.x == 0 && threadIdx.x == 0) *devCount = m;
}

// Blocks of column y take the transfers kIoGroup * y ...  Their count slots lie in host memory,
// where a read is a PCIe transaction and the transactions queue (about 0.4 us each): one warp
// reads a group's slots at once, and 4 blocks share a group (16 blocks per transfer, each
// reading its slot, took 430 us for 64 arrays that had nothing to copy).
constexpr int kIoGroup = 8, kIoGroupBlocks = 4;
__global__ void __launch_bounds__(kIoThreads) k_array_upload_batch(const agocuda_array_xfer *xfers, uint32_t count)
{
    __shared__ uint32_t slots[kIoGroup];
    const uint32_t first = blockIdx.y * kIoGroup, k = min((uint32_t)kIoGroup, count - first);
    if (threadIdx.x < k) slots[threadIdx.x] = *(const volatile uint32_t *)xfers[first + threadIdx.x].countSlotMapped;
    __syncthreads();
    for (uint32_t i = 0; i < k; i++) {
        if (slots[i] == AGOCUDA_ARRAY_SKIP) continue;
        const agocuda_array_xfer X = xfers[first + i];
        const uint32_t m = min(slots[i], X.capacity);
        copy_bytes((uint8_t *)X.devItems, (const uint8_t *)X.hostItemsMapped, (size_t)m * X.itemSize);
        if (blockIdx.x == 0 && threadIdx.x == 0) *X.devCount = m;
    }
}

// blockIdx.y: the transfer (device -> host; writes are posted)
__global__ void __launch_bounds__(kIoThreads) k_array_download_batch(const agocuda_array_xfer *xfers)
{
    const agocuda_array_xfer X = xfers[blockIdx.y];
    const uint32_t m = min(*X.devCount, X.capacity);
    copy_bytes((uint8_t *)X.hostItemsMapped, (const uint8_t *)X.devItems, (size_t)m * X.itemSize);
    if (blockIdx.x == 0 && threadIdx.x == 0) *(volatile uint32_t *)X.countSlotMapped = m;
}

__global__ void __launch_bounds__(kIoThreads)
k_array_download(uint8_t *host, volatile uint32_t *slot, const uint8_t *dev, const uint32_t *devCount,
                 uint32_t itemSize, uint32_t capacity)
{
    const uint32_t m = min(*devCount, capacity);
    copy_bytes(host, dev, (size_t)m * itemSize);
    if (blockIdx.x == 0 && threadIdx.x == 0) *slot = m;
}

// the device's nanosecond clock, into a mapped host word
__global__ void k_time_stamp(unsigned long long *out)
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    *out = t;
}

}  // namespace

extern "C" int agocuda_time_stamp(void *stream, uint64_t *pMapped)
{
    if (!pMapped) return AGOCUDA_INVALID_PARAMS;
    k_time_stamp<<<1, 1, 0, as_stream(stream)>>>((unsigned long long *)pMapped);
    agocuda_count_launch(1);
    return agocuda_launch_status();
}

extern "C" int agocuda_array_upload(void *stream, void *devItems, uint32_t *devCount, const void *hostItemsMapped,
                                    const uint32_t *countSlotMapped, uint32_t itemSize, uint32_t capacity)
{
    if (!devItems || !devCount || !hostItemsMapped || !countSlotMapped || !itemSize || !capacity)
        return AGOCUDA_INVALID_PARAMS;
    k_array_upload<<<kIoBlocks, kIoThreads, 0, as_stream(stream)>>>((uint8_t *)devItems, devCount,
                                                                    (const uint8_t *)hostItemsMapped, countSlotMapped,
                                                                    itemSize, capacity);
    agocuda_count_launch(1);
    return agocuda_launch_status();
}

extern "C" int agocuda_array_upload_batch(void *stream, const agocuda_array_xfer *xfers, uint32_t count)
{
    if (!xfers || !count || count > 65535) return AGOCUDA_INVALID_PARAMS;
    k_array_upload_batch<<<dim3(kIoGroupBlocks, (count + kIoGroup - 1) / kIoGroup), kIoThreads, 0, as_stream(stream)>>>(xfers, count);
    agocuda_count_launch(1);
    return agocuda_launch_status();
}

extern "C" int agocuda_array_download_batch(void *stream, const agocuda_array_xfer *xfers, uint32_t count)
{
    if (!xfers || !count || count > 65535) return AGOCUDA_INVALID_PARAMS;
    k_array_download_batch<<<dim3(kIoGroupBlocks, count), kIoThreads, 0, as_stream(stream)>>>(xfers);
    agocuda_count_launch(1);
    return agocuda_launch_status();
}

extern "C" int agocuda_array_download(void *stream, void *hostItemsMapped, uint32_t *countSlotMapped,
                                      const void *devItems, const uint32_t *devCount, uint32_t itemSize,
                                      uint32_t capacity)
{
    if (!devItems || !devCount || !hostItemsMapped || !countSlotMapped || !itemSize || !capacity)
        return AGOCUDA_INVALID_PARAMS;
    k_array_download<<<kIoBlocks, kIoThreads, 0, as_stream(stream)>>>((uint8_t *)hostItemsMapped, countSlotMapped,
                                                                      (const uint8_t *)devItems, devCount, itemSize,
                                                                      capacity);
    agocuda_count_launch(1);
    return agocuda_launch_status();
}
