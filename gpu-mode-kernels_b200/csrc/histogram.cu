// 256-bin histogram of bytes for sm_100a: the second task of the reference repository
// (pmpp_v2/histogram_py: `output = bincount(data, minlength=256)` on uint8 input, int64 output,
// reference.py:6-19).
//
// What bounds it: first the shared-memory counters, one update per byte, then HBM.  A block therefore
// counts into a table of 256 rows of 32 words, a word per (value, LANE): lane l only ever touches bank l,
// so an update is one pass over the banks whatever the data is -- random bytes and one value 90 % of
// the time cost the same -- and the word's address comes out of the data with one shift and one
// three-input logic operation.  Warps share the table (32 KB a block), so the updates are atomic, without
// a result.  Measured on 512 MB, random bytes: the launch 85 us = 6.3 TB/s (of 6.55 copied), against 303 us with a
// 256-word table per warp, where 32 random bytes meet in a bank 3.5 deep and the frequent value needed
// ballots; one byte counter per (value, thread) without atomics is two accesses a byte: 256 us.
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "a2a.h"

namespace {

namespace cg = cooperative_groups;

constexpr int kThreads = 512;
constexpr int kBlocksPerSm = 2;
// 16-byte loads per thread and round; the next round's are requested before this one's bytes are counted,
// so 64 KB per SM are on their way at any time: 512 MB 85 us against 91 with three blocks per SM that load,
// then count, and 105 to 127 through shared memory by the copy engine (its reads cost bank passes too).
constexpr int kUnroll = 4;
constexpr int kBins = 256;
constexpr int kCluster = 8;
// One cluster writes the counts itself: no zeroing in front, one launch.  128 KB 4.3 us against 6.3 as
// zero + count; 512 KB 6.3 against 6.2.  A block takes 32 KB at a time, so below 256 KB only some of the
// cluster's blocks count, and at 512 KB 16 blocks of the other launch do.
constexpr size_t kClusterBytes = 256 * 1024;
// Below this a block per SM: 256 sums per block meet at 256 global words, and with few bytes per block
// that is what the call waits for.  Measured against the three blocks per SM that large buffers had then:
// 10 MB 6.3 us / 8.3, 42 MB 12.4 / 12.2, 168 MB 44 / 33.
constexpr size_t kFullBytes = 32 * 1024 * 1024;

// `lane4` = 4 * lane: the byte offset of the lane's word in a row of 32.
__device__ __forceinline__ void count_byte(unsigned* table, unsigned v, unsigned lane4) {
    atomicAdd(reinterpret_cast<unsigned*>(reinterpret_cast<char*>(table) + ((v << 7) | lane4)), 1u);
}

__device__ __forceinline__ void count_vector(unsigned* table, const uint4& q, unsigned lane4) {
    const unsigned w[4] = {q.x, q.y, q.z, q.w};
    char* base = reinterpret_cast<char*>(table);
#pragma unroll
    for (int a = 0; a < 4; ++a) {  // byte b of the word, times 128, in one shift and one and-or
        atomicAdd(reinterpret_cast<unsigned*>(base + (((w[a] << 7) & 0x7f80u) | lane4)), 1u);
        atomicAdd(reinterpret_cast<unsigned*>(base + (((w[a] >> 1) & 0x7f80u) | lane4)), 1u);
        atomicAdd(reinterpret_cast<unsigned*>(base + (((w[a] >> 9) & 0x7f80u) | lane4)), 1u);
        atomicAdd(reinterpret_cast<unsigned*>(base + (((w[a] >> 17) & 0x7f80u) | lane4)), 1u);
    }
}

__device__ __forceinline__ void load_vectors(const uint4* vec, size_t i, size_t nvec, uint4 (&q)[kUnroll]) {
#pragma unroll
    for (int u = 0; u < kUnroll; ++u)
        if (i + u * kThreads < nvec) q[u] = __ldcs(vec + i + u * kThreads);
}

// CLUSTER: the grid is one cluster and stores the counts.  Otherwise the blocks add theirs to `out`, which
// the launch before this one zeroes while the blocks already count.
template <bool CLUSTER>
__global__ void __launch_bounds__(kThreads, kBlocksPerSm) histogram256_kernel(const uint8_t* __restrict__ data, size_t n,
                                                                             unsigned long long* __restrict__ out) {
    __shared__ __align__(16) unsigned table[kBins * 32];
    __shared__ unsigned long long sums[kBins];
    const int tid = threadIdx.x;
    const unsigned lane4 = (tid & 31) * 4;
    // head: bytes before the first 16-byte boundary; body: 16-byte vectors; tail: the rest
    const uintptr_t addr = reinterpret_cast<uintptr_t>(data);
    size_t head = (16 - (addr & 15)) & 15;
    if (head > n) head = n;
    const size_t nvec = (n - head) / 16;
    const uint4* vec = reinterpret_cast<const uint4*>(data + head);
    // a block takes 32 KB at a time
    const size_t step = (size_t)gridDim.x * kThreads * kUnroll;
    size_t i = (size_t)blockIdx.x * kThreads * kUnroll + tid;
    uint4 q[kUnroll], next[kUnroll];
    load_vectors(vec, i, nvec, q);
    for (int v = tid; v < kBins * 8; v += kThreads) reinterpret_cast<uint4*>(table)[v] = make_uint4(0u, 0u, 0u, 0u);
    __syncthreads();
    for (; i < nvec; i += step) {
        load_vectors(vec, i + step, nvec, next);
#pragma unroll
        for (int u = 0; u < kUnroll; ++u) {
            if (i + u * kThreads < nvec) count_vector(table, q[u], lane4);
            q[u] = next[u];
        }
    }
    if (blockIdx.x == 0 && tid < 32) {  // the ragged ends: at most 15 + 15 bytes
        const size_t i = tid < 16 ? (size_t)tid : head + nvec * 16 + (tid - 16);
        if (tid < 16 ? i < head : i < n) count_byte(table, data[i], lane4);
    }
    __syncthreads();
    {
        // two threads per bin, 16 words each; started at the bin's own word so that a warp reads 32 banks
        const int bin = tid >> 1, half = tid & 1;
        unsigned long long sum = 0;
#pragma unroll
        for (int i = 0; i < 16; ++i) sum += table[bin * 32 + half * 16 + ((i + bin) & 15)];
        sum += __shfl_xor_sync(0xffffffffu, sum, 1);
        if (half == 0) sums[bin] = sum;
    }
    if (CLUSTER) {
        const cg::cluster_group cluster = cg::this_cluster();
        cluster.sync();
        constexpr int kShare = kBins / kCluster;  // bins this block adds up over the cluster
        const int bin = cluster.block_rank() * kShare + tid;
        if (tid < kShare) {
            unsigned long long sum = 0;
#pragma unroll
            for (int b = 0; b < kCluster; ++b) sum += *cluster.map_shared_rank(sums + bin, b);
            out[bin] = sum;
        }
        cluster.sync();  // no block leaves while its sums are read
    } else {
        __syncthreads();
        cudaGridDependencySynchronize();  // `out` is zero
        if (tid < kBins && sums[tid]) atomicAdd(out + tid, sums[tid]);
    }
}

// Starts the counting launch at once: by then everything before this launch in the stream has completed, so
// the data is there, and only the adding to `out` waits for the zeros.
__global__ void __launch_bounds__(kBins) zero_counts_kernel(unsigned long long* out) {
    cudaTriggerProgrammaticLaunchCompletion();
    out[threadIdx.x] = 0ull;
}

}  // namespace

extern "C" int a2a_histogram256(const uint8_t* data, size_t n, int64_t* out, void* stream) {
    if (out == nullptr || (n > 0 && data == nullptr)) return A2A_ERR_CONFIG;
    if (reinterpret_cast<uintptr_t>(out) % 8 != 0) return A2A_ERR_CONFIG;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    unsigned long long* counts = reinterpret_cast<unsigned long long*>(out);
    cudaLaunchAttribute attr{};
    cudaLaunchConfig_t launch{};
    launch.blockDim = dim3(kThreads);
    launch.stream = st;
    launch.attrs = &attr;
    launch.numAttrs = 1;
    cudaError_t e;
    if (n <= kClusterBytes) {
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = kCluster;
        attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
        launch.gridDim = dim3(kCluster);
        e = cudaLaunchKernelEx(&launch, histogram256_kernel<true>, data, n, counts);
        return e == cudaSuccess ? A2A_OK : -(int)e;
    }
    int dev = 0, sms = 0;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess) return -(int)e;
    if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return -(int)e;
    cudaLaunchConfig_t zero{};
    zero.gridDim = dim3(1);
    zero.blockDim = dim3(kBins);
    zero.stream = st;
    if ((e = cudaLaunchKernelEx(&zero, zero_counts_kernel, counts)) != cudaSuccess) return -(int)e;
    const size_t want = (n / 16 + kThreads - 1) / kThreads;
    const size_t room = (size_t)sms * (n < kFullBytes ? 1 : kBlocksPerSm);
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    launch.gridDim = dim3((unsigned)(want < room ? want : room));
    e = cudaLaunchKernelEx(&launch, histogram256_kernel<false>, data, n, counts);
    return e == cudaSuccess ? A2A_OK : -(int)e;
}
