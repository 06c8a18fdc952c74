// World size 1: the whole forward of a pipelined context as ONE ordinary launch whose blocks know
// nothing of each other: calls of few tokens and few rows (solo_two_launches in a2a.cu), traced calls, and rows in host
// memory.  Larger calls, and outputs over the weights or the indices, take the routing and the rows of a2a_near.cuh.
// With a single rank nothing travels, so nothing has to be handed over: a
// block that owns a contiguous range of (token, chunk) items works out the slots of its own tokens
// from the caller's indices alone and then does everything for them -- the slab rows with the
// placeholder expert op applied, the (token, k) words, the slot table and the weighted sum.
#pragma once

#include "a2a_pipe.cuh"

namespace a2a {

constexpr int kSoloWarps = kThreads / 32;
constexpr int kSoloRound = 16;  // tokens whose pairs are resolved together in shared memory

// Indices [k0, k0 + 8) of the token whose indices lie at `row`, -1 past the last; `quads`: they lie in whole 16-byte vectors.
__device__ __forceinline__ void load_indices(const int* row, int k0, int K, bool quads, int (&e8)[8]) {
    if (quads) {
#pragma unroll
        for (int u = 0; u < 8; u += 4) {
            int4 v = make_int4(-1, -1, -1, -1);
            if (k0 + u < K) v = *reinterpret_cast<const int4*>(row + k0 + u);
            e8[u] = v.x;
            e8[u + 1] = v.y;
            e8[u + 2] = v.z;
            e8[u + 3] = v.w;
        }
    } else {
#pragma unroll
        for (int u = 0; u < 8; ++u) e8[u] = k0 + u < K ? ld_input(row + k0 + u) : -1;
    }
}

// Counts of the experts used by tokens [0, t_end) into s_cnt (shared, cleared by the caller).  A
// repeat inside a token counts once, an index out of range not at all.  N tokens' indices are requested together, in 16-byte vectors
// where they lie so: captured, one rank, 256 tokens of 7168, top-8 9.1 us a call, index by index 9.3; 2048 52.3 / 53.7, and with one
// token at a time 52.8.
template <int THREADS, int N = 1>
__device__ __forceinline__ void count_experts_before(const DevParams& p, int t_end, int* s_cnt) {
    const int K = p.K;
    const bool quads = (K & 3) == 0 && (reinterpret_cast<uintptr_t>(p.idx) & 15) == 0;
    for (int t = threadIdx.x; t < t_end; t += N * THREADS) {
        for (int k0 = 0; k0 < K; k0 += 8) {
            int e8[N][8];
#pragma unroll
            for (int n = 0; n < N; ++n)  // tokens whose indices are requested together
                if (n == 0 || t + n * THREADS < t_end) load_indices(p.idx + (size_t)(t + n * THREADS) * K, k0, K, quads, e8[n]);
#pragma unroll
            for (int n = 0; n < N; ++n) {
                if (n > 0 && t + n * THREADS >= t_end) break;
                const int* row = p.idx + (size_t)(t + n * THREADS) * K;
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    const int e = e8[n][u];
                    bool ok = e >= 0 && e < p.E;
#pragma unroll
                    for (int v = 0; v < u; ++v) ok = ok && e8[n][v] != e;
                    for (int kk = 0; ok && kk < k0; ++kk) ok = ld_input(row + kk) != e;
                    if (ok) atomicAdd(s_cnt + e, 1);
                }
            }
        }
    }
}

// U 16-byte vectors per lane of one row of x as the expert's rank holds them after dispatch (FP8:
// through the same quantise / dequantise arithmetic the wire applies).
template <typename T, int PAYLOAD, int U>
__device__ __forceinline__ void load_own_chunk(const DevParams& p, int t, int v0, int nvec, uint4 (&q)[U]) {
    const int lane = threadIdx.x & 31;
    const uint4* src = reinterpret_cast<const uint4*>(p.x) + (size_t)t * nvec;
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int v = v0 + u * 32 + lane;
        if (v < nvec) q[u] = ld_input(src + v);
    }
    if (PAYLOAD == A2A_PAYLOAD_FP8) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int v = v0 + u * 32 + lane;  // nvec % 16 == 0: the 16 lanes of a scale block are all in or all out
            q[u] = fp8_round_trip<T>(q[u], v < nvec);
        }
    }
}

// What bounds it: the stores, K + 1 rows out for every row in; below a few dozen tokens the chain
// launch -> indices -> slots -> stores.  Blocks take contiguous items so that each resolves the pairs
// of the few tokens it touches once; the indices of the tokens before them (64 KB at 2048 x 8, out of
// L2) are counted again by every block, 1 to 3 us that the first row's load hides in part and that no
// exchange between blocks would undercut.  Captured, and the role-split kernel that handed slots, flags and rows from block to
// block (a call): 3.7 / 11.9 us (one token of 2048, top-6), 4.2 / 11.7 (93 tokens of 2880, top-4), 9.1 / 18.7 (256 tokens of
// 7168, top-8: 4.0 TB/s into the L2, what a plain fill of the same 33 MB takes); 2048 tokens of 7168, traced, 60.7, in two launches 52.3.
// The loop that resolves a round's pairs stands in near_dispatch_kernel (a2a_near.cuh) too: as a function it cost this kernel 0.17 us.
template <typename T, int PAYLOAD, int U>
__global__ void __launch_bounds__(kThreads) solo_kernel(const __grid_constant__ DevParams p) {
    __shared__ int s_cnt[A2A_MAX_EXPERTS];                 // tokens before the current round that use expert e
    __shared__ int s_idx[kSoloRound * A2A_MAX_TOPK];       // the round's indices,
    __shared__ float s_w[kSoloRound * A2A_MAX_TOPK];       // weights
    __shared__ int s_row[kSoloRound * A2A_MAX_TOPK];       // and slab rows (-1: dropped pair)
    begin_after_previous();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int K = p.K, nvec = p.H >> 3;
    const int nchunk = (nvec + 32 * U - 1) / (32 * U);
    const long long items = (long long)p.T * nchunk;
    const long long lo = items * blockIdx.x / gridDim.x, hi = items * (blockIdx.x + 1) / gridDim.x;
    const int t0 = (int)(lo / nchunk), t1 = (int)((hi + nchunk - 1) / nchunk);
    const bool last = blockIdx.x == gridDim.x - 1;
    stamp(p, kStampStart);
    stamp_value(p, kStampRole, last ? (kRoleExpert | kRoleRouter) : kRoleExpert);
    uint8_t* self = p.peer[p.rank];
    uint4* rows = reinterpret_cast<uint4*>(self + p.off_rows);
    int* meta = reinterpret_cast<int*>(self + p.off_meta);
    const float scale = (float)(1 + p.rank);

    // the first item's row and the first round's pairs are requested before anything else: they need no routing
    long long it = lo + warp;
    int t = (int)(it / nchunk), c = (int)(it - (long long)t * nchunk);
    uint4 q[U];
    if (it < hi) load_own_chunk<T, PAYLOAD, U>(p, t, c * 32 * U, nvec, q);
    int first_e = 0;
    float first_w = 0.f;
    if (tid < min(kSoloRound, t1 - t0) * K) {
        first_e = ld_input(p.idx + (size_t)t0 * K + tid);
        first_w = ld_input(p.w + (size_t)t0 * K + tid);
    }
    for (int e = tid; e < p.E; e += kThreads) s_cnt[e] = 0;
    __syncthreads();
    count_experts_before<kThreads>(p, t0, s_cnt);

    for (int r0 = t0; r0 < t1; r0 += kSoloRound) {
        const int nt = min(kSoloRound, t1 - r0), pairs = nt * K;
        for (int i = tid; i < pairs; i += kThreads) {
            const bool first = r0 == t0 && i == tid;
            const int e = first ? first_e : ld_input(p.idx + (size_t)r0 * K + i);
            const float w = first ? first_w : ld_input(p.w + (size_t)r0 * K + i);
            s_idx[i] = e;
            s_w[i] = w;
        }
        __syncthreads();
        if (r0 == t0) stamp(p, kStampSourceSeen);
        for (int i = tid; i < pairs; i += kThreads) {
            const int tl = i / K, k = i - tl * K, e = s_idx[i];
            const bool in_range = e >= 0 && e < p.E;
            bool ok = in_range;
            for (int kk = 0; kk < k; ++kk) ok = ok && s_idx[tl * K + kk] != e;
            int j = -1;
            if (ok) {
                j = s_cnt[e];
                for (int u = 0; u < tl; ++u) {
                    bool uses = false;
                    for (int kk = 0; kk < K; ++kk) uses |= s_idx[u * K + kk] == e;
                    j += uses ? 1 : 0;
                }
            }
            s_row[i] = ok ? e * p.T_max + j : -1;
            if ((long long)(r0 + tl) * nchunk >= lo) {  // the block that has the token's first chunk books its pairs
                p.slot[(size_t)r0 * K + i] = j;
                if (ok) meta[(size_t)e * p.T_max + j] = ((r0 + tl) << 8) | k;
                else record_error(p.status, A2A_ERR_ROUTING, p.rank, -1, kPhaseRoute, p.epoch, e);
            }
        }
        __syncthreads();
        for (int i = tid; i < pairs; i += kThreads)
            if (s_row[i] >= 0) atomicAdd(s_cnt + s_idx[i], 1);
        const long long end = min(hi, (long long)(r0 + nt) * nchunk);
        while (it < end) {
            const long long next = it + kSoloWarps;
            int tn = t, cn = c + kSoloWarps;
            while (cn >= nchunk) { cn -= nchunk; ++tn; }
            uint4 qn[U];
            if (next < hi) load_own_chunk<T, PAYLOAD, U>(p, tn, cn * 32 * U, nvec, qn);
            const int v0 = c * 32 * U, pair0 = (t - r0) * K;
            float acc[U][8];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                q[u] = scale8<T>(q[u], scale);  // the placeholder expert op: T(float(row) * (1 + rank))
#pragma unroll
                for (int e = 0; e < 8; ++e) acc[u][e] = 0.f;
            }
            for (int k = 0; k < K; ++k) {
                const int r = s_row[pair0 + k];
                if (r < 0) continue;
                const float w = s_w[pair0 + k];
                uint4* row = rows + (size_t)r * nvec;
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int v = v0 + u * 32 + lane;
                    if (v < nvec) {
                        st_stream(row + v, q[u]);
                        float f[8];
                        unpack8<T>(q[u], f);
                        fma8(f, w, acc[u]);
                    }
                }
            }
            uint4* y = reinterpret_cast<uint4*>(p.y) + (size_t)t * nvec;
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int v = v0 + u * 32 + lane;
                if (v < nvec) st_stream(y + v, pack8<T>(acc[u]));
                q[u] = qn[u];
            }
            it = next;
            t = tn;
            c = cn;
        }
        __syncthreads();
    }
    stamp(p, kStampSourceDone);
    stamp(p, kStampExpertDone);
    if (last) {  // this block's counts now cover every token
        int* counts = reinterpret_cast<int*>(self + p.off_counts);
        for (int e = tid; e < p.E; e += kThreads) counts[e] = p.send_counts[e] = s_cnt[e];
        // phases called on this context after the forward find its flags up
        if (tid == 0) {
            *seen_ptr(p, kFlagDispatch, p.rank) = flag_value(p, 0);
            *seen_ptr(p, kFlagExpert, p.rank) = flag_value(p, 0);
        }
    }
    stamp(p, kStampExpertSeen);
    stamp(p, kStampCombineDone);
}

}  // namespace a2a
