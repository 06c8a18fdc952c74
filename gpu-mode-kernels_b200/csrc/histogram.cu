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
// One cluster writes the counts itself: no zeroing in front, one launch, which gets ready while the launch before it ends.
// Calls back to back, 30 KB 2.8 us, captured 2.3 (5.2 without the overlap, and with 32 KB a block one of eight at work), 256 KB 4.0,
// captured 2.6.  Above, the host needs 5.2 us for zero + count where one cluster of 300 KB took 4.0, but the GPU 2.5 to 3.6, which is
// what a captured call takes: the line favours captured calls, and plain ones from 256 to about 500 KB pay a quarter for it.
constexpr size_t kClusterBytes = 256 * 1024;
// Up to here (592 KB with 148 SMs) every block has the one row of 8 KB that its grid of n / 8 KB blocks leaves it: captured, 300 KB
// 2.5 us, 3.3 with 32 KB a block.  From here on 32 KB a block, on a grid of as many blocks as there are rows of 8 KB, one per SM at most:
// up to 4.8 MB some find no data (56 of 75 just above, 84 of 148 at 2 MB) and add nothing.  2 MB 3.0 us, 3.6 with rows a grid apart.
constexpr size_t kSpreadBytesPerSm = 4 * 1024;
// Below this a block per SM: 256 sums per block meet at 256 global words, and with few bytes per block
// that is what the call waits for.  10 MB 4.5 us on the GPU, 20 MB 6.2, 31 MB 7.9; with two blocks from 16 MB on 6.4 and 8.2.
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

// Ordinary loads, past the L1: a launch that overlaps the end of the one before it may not promise that nobody writes the data.
__device__ __forceinline__ void load_vectors(const uint4* vec, size_t i, size_t row, size_t nvec, uint4 (&q)[kUnroll]) {
#pragma unroll
    for (int u = 0; u < kUnroll; ++u)
        if (i + u * row < nvec) q[u] = __ldcg(vec + i + u * row);
}

// The grid is one cluster and stores the counts; or its blocks add theirs to `out`, which the launch before this one zeroes while
// they already count: with one row of data a block (kSpread) or with more (kRounds).
enum Form { kCluster8, kSpread, kRounds };

template <Form FORM>
__global__ void __launch_bounds__(kThreads, kBlocksPerSm) histogram256_kernel(const uint8_t* data, size_t n,
                                                                             unsigned long long* out) {
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
    // A block takes kUnroll rows of 8 KB at a time: one after the other, 32 KB of the memory's pages (512 MB 88 us, 97 with a row from
    // each of four places), or, in the smallest grids, rows a grid apart, so that every block has one.
    constexpr bool cluster = FORM == kCluster8, apart = FORM != kRounds;
    const size_t row = apart ? (size_t)gridDim.x * kThreads : kThreads, step = (size_t)gridDim.x * kThreads * kUnroll;
    size_t i = (size_t)blockIdx.x * kThreads * (apart ? 1 : kUnroll) + tid;
    uint4 q[kUnroll], next[kUnroll];
    if (!cluster) load_vectors(vec, i, row, nvec, q);
    for (int v = tid; v < kBins * 8; v += kThreads) reinterpret_cast<uint4*>(table)[v] = make_uint4(0u, 0u, 0u, 0u);
    if (cluster) {
        cudaGridDependencySynchronize();
        cudaTriggerProgrammaticLaunchCompletion();
        load_vectors(vec, i, row, nvec, q);
    }
    __syncthreads();
    for (; i < nvec; i += step) {
        load_vectors(vec, i + step, row, nvec, next);
#pragma unroll
        for (int u = 0; u < kUnroll; ++u) {
            if (i + u * row < nvec) count_vector(table, q[u], lane4);
            q[u] = next[u];
        }
    }
    if (blockIdx.x == 0 && tid < 32) {  // the ragged ends: at most 15 + 15 bytes
        const size_t i = tid < 16 ? (size_t)tid : head + nvec * 16 + (tid - 16);
        if (tid < 16 ? i < head : i < n) count_byte(table, __ldcg(data + i), lane4);
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
    if (cluster) {
        const cg::cluster_group blocks = cg::this_cluster();
        blocks.sync();
        constexpr int kShare = kBins / kCluster;  // bins this block adds up over the cluster
        const int bin = blocks.block_rank() * kShare + tid;
        if (tid < kShare) {
            unsigned long long sum = 0;
#pragma unroll
            for (int b = 0; b < kCluster; ++b) sum += *blocks.map_shared_rank(sums + bin, b);
            out[bin] = sum;
        }
        blocks.sync();  // no block leaves while its sums are read
    } else {
        __syncthreads();
        cudaGridDependencySynchronize();  // `out` is zero
        cudaTriggerProgrammaticLaunchCompletion();
        if (tid < kBins && sums[tid]) atomicAdd(out + tid, sums[tid]);
    }
}

// Gets ready while the launch before it ends, and starts the counting launch as soon as that has completed: the data is there then, and
// only the adding to `out` waits for the zeros (10 MB 7.0 -> 5.2 us a call then, 512 MB in bursts 87.6 -> 85.9).
__global__ void __launch_bounds__(kBins) zero_counts_kernel(unsigned long long* out) {
    cudaGridDependencySynchronize();
    cudaTriggerProgrammaticLaunchCompletion();
    out[threadIdx.x] = 0ull;
}

}  // namespace

extern "C" int a2a_histogram256(const uint8_t* data, size_t n, int64_t* out, void* stream) {
    if (out == nullptr || (n > 0 && data == nullptr)) return A2A_ERR_CONFIG;
    if (reinterpret_cast<uintptr_t>(out) % 8 != 0) return A2A_ERR_CONFIG;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    unsigned long long* counts = reinterpret_cast<unsigned long long*>(out);
    cudaLaunchAttribute attr[2] = {};
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t launch{};
    launch.blockDim = dim3(kThreads);
    launch.stream = st;
    launch.attrs = attr;
    launch.numAttrs = 1;
    cudaError_t e;
    if (n <= kClusterBytes) {
        attr[1].id = cudaLaunchAttributeClusterDimension;
        attr[1].val.clusterDim.x = kCluster;
        attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
        launch.numAttrs = 2;
        launch.gridDim = dim3(kCluster);
        e = cudaLaunchKernelEx(&launch, histogram256_kernel<kCluster8>, data, n, counts);
        return e == cudaSuccess ? A2A_OK : -(int)e;
    }
    int dev = 0, sms = 0;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess) return -(int)e;
    if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return -(int)e;
    cudaLaunchConfig_t zero{};
    zero.gridDim = dim3(1);
    zero.blockDim = dim3(kBins);
    zero.stream = st;
    zero.attrs = attr;
    zero.numAttrs = 1;
    if ((e = cudaLaunchKernelEx(&zero, zero_counts_kernel, counts)) != cudaSuccess) return -(int)e;
    const size_t want = (n / 16 + kThreads - 1) / kThreads;
    const size_t room = (size_t)sms * (n < kFullBytes ? 1 : kBlocksPerSm);
    launch.gridDim = dim3((unsigned)(want < room ? want : room));
    const auto kernel = n <= (size_t)sms * kSpreadBytesPerSm ? histogram256_kernel<kSpread> : histogram256_kernel<kRounds>;
    e = cudaLaunchKernelEx(&launch, kernel, data, n, counts);
    return e == cudaSuccess ? A2A_OK : -(int)e;
}
