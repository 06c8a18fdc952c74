// The roles of the pipelined schedule for ranks that share ONE GPU: one launch per role serves the whole group
// (a2a_group_step).  Slabs, slots, counts, flags and epochs are those of a group with a GPU each, and so is every
// bit of the results; what differs is what distance costs and a neighbour does not:
//   * a row is not carried to a stage first, and nobody is told of it by a record.  The input rows of all ranks lie in
//     this GPU's memory, and so do all slabs: a warp takes a piece of a token's row, reads it once, and writes
//     every slab row of it, whichever rank's.
//   * with every expert row of a token in its hands that warp also has the token's output: no partial row is written
//     and read again.
//   * the tokens of all ranks are one list that all blocks share: a rank whose experts are popular does not
//     keep its own blocks busy while the others' are through.
//   * every flag of the role before is up when a launch starts (it is awaited all the same, bounded, at gpu
//     scope, unless the launch before it in the same call is that role).
// One rank with many tokens is a group of one, and the phases of a group's call (of one rank: a2a_kernels.cuh) go by the
// same lists of pairs.
// Times in this file and beside the launchers in a2a.cu are us a call, captured (calls one after the other in a graph, without
// the host) unless something else is said.
#pragma once

#include "a2a_solo.cuh"

namespace a2a {

// The ranks a launch serves (`n` of them, all of a group or one) and what role 0 knew or found of every rank.  N: the
// most ranks a group may have; a type of its own for a single rank, whose launches are the cheaper for it (1500 tokens of 2880
// 12.5 with room for eight, 11.9 without; 2048 of 7168 53.4 / 52.3).
template <int N>
struct NearParams {
    DevParams p[N];
    const void* x[N];       // input rows of rank s in this call
    const uint2* pairs[N];  // its (token, k) pairs as near_route_kernel left them
    int T[N];               // and its tokens
    int n;
    int every_rank;  // a PULL combine ends only when every rank's outputs are there, also those no token wants
    int backwards;   // blocks take the items from the end
    int handed_on;   // the launches of one call, one after the other on one stream: no flag is awaited or raised before the last
};
using NearGroup = NearParams<A2A_MAX_WORLD>;

// ---------------------------------------------------------------------------
// Role 0: routing.  A block takes `words` * 32 tokens of a rank: it counts the experts of the tokens before them once
// more for itself (64 KB at 2048 x 8, out of the L2) instead of waiting for another block.  What bounds it: the chain
// launch -> indices -> counts -> slots -> stores.
// ---------------------------------------------------------------------------
__host__ __device__ inline size_t near_route_smem(int words, int E, int K) {
    return ((size_t)(words + 1) * E + (size_t)words * 64 * K) * 4;
}

template <int N, int THREADS>
__global__ void __launch_bounds__(THREADS) near_route_kernel(const __grid_constant__ NearParams<N> g, int words) {
    begin_after_previous();
    const int n = N == 1 ? 1 : g.n;
    const DevParams& p = g.p[blockIdx.x % n];
    const int tid = threadIdx.x, E = p.E, K = p.K, tokens = words * 32, nb = (int)gridDim.x / n;
    const int t0 = (int)blockIdx.x / n * tokens, pairs = max(0, min(tokens, p.T - t0)) * K;
    int* s_cnt = reinterpret_cast<int*>(a2a_pipe_smem);         // [E] tokens before this block's that use expert e
    unsigned* s_bits = reinterpret_cast<unsigned*>(s_cnt + E);  // [words][E] this block's tokens that do
    int* s_idx = s_cnt + (words + 1) * E;                       // [tokens][K]
    float* s_w = reinterpret_cast<float*>(s_idx + tokens * K);  // [tokens][K]
    stamp(p, kStampStart);
    const bool last = p.T > 0 ? pairs > 0 && t0 + tokens >= p.T : t0 == 0;
    if (pairs > 0 || last) {
        for (int i = tid; i < pairs; i += THREADS) {
            s_idx[i] = ld_input(p.idx + (size_t)t0 * K + i);
            s_w[i] = ld_input(p.w + (size_t)t0 * K + i);
        }
        for (int e = tid; e < (words + 1) * E; e += THREADS) s_cnt[e] = 0;
        __syncthreads();
        count_experts_before<THREADS, 4>(p, t0, s_cnt);
        auto first_use = [&](int i) {  // pair i's expert is in range and of no earlier pair of its token
            const int e = s_idx[i];
            bool ok = e >= 0 && e < E;
            for (int j = i / K * K; ok && j < i; ++j) ok = s_idx[j] != e;
            return ok;
        };
        for (int i = tid; i < pairs; i += THREADS)
            if (first_use(i)) atomicOr(s_bits + (i / K >> 5) * E + s_idx[i], 1u << (i / K & 31));
        __syncthreads();
        for (int i = tid; i < pairs; i += THREADS) {
            const size_t at = (size_t)t0 * K + i;
            const int tl = i / K, e = s_idx[i];
            int j = -1;
            unsigned place = kNoPair;
            if (first_use(i)) {
                j = s_cnt[e];
                for (int w = 0; w < tl >> 5; ++w) j += __popc(s_bits[w * E + e]);
                j += __popc(s_bits[(tl >> 5) * E + e] & ((1u << (tl & 31)) - 1u));
                place = pair_place(p, p.rank, e, j);
                reinterpret_cast<int*>(p.peer[place >> 28] + p.off_meta)[place & kPairRow] = ((t0 + tl) << 8) | (i - tl * K);
            } else {
                record_error(p.status, A2A_ERR_ROUTING, p.rank, -1, kPhaseRoute, p.epoch, e);
            }
            p.slot[at] = j;
            p.pairs[at] = make_uint2(place, __float_as_uint(s_w[i]));
        }
        if (last)
            for (int e = tid; e < E; e += THREADS) {
                int c = s_cnt[e];
                for (int w = 0; w < words; ++w) c += __popc(s_bits[w * E + e]);
                const int d = e / p.L;
                reinterpret_cast<int*>(p.peer[d] + p.off_counts)[(size_t)p.rank * kMaxChunks * p.L + (e - d * p.L)] = c;
                p.send_counts[e] = c;
            }
    }
    stamp(p, kStampSent);
    if (g.handed_on) return;
    __syncthreads();
    if (tid < p.ws) arrive_dest(p, tid, (uint32_t)nb);
}

// What has been recorded of the rank whose flags this thread raises.
__device__ __forceinline__ int recorded_of_rank(const NearGroup& g) {
    const int i = threadIdx.x / g.p[0].ws;
    return ld_volatile_i32(&g.p[i < g.n ? i : 0].status->code);
}

// The flags of `kinds` of the ranks served go up, unless a wait of one of them gave up; called by a whole block, which has seen
// what they stand for.
__device__ __forceinline__ void raise_flags(const NearGroup& g, unsigned kinds, int recorded) {
    const int ws = g.p[0].ws, i = threadIdx.x / ws, s = threadIdx.x % ws;
    if (!__syncthreads_and(recorded != A2A_ERR_TIMEOUT) || i >= g.n) return;
    const DevParams& p = g.p[i];
    fence_acq_rel_gpu();
    if (kinds >> kFlagDispatch & 1u)  // rank s has sent to rank i
        st_relaxed_gpu(const_cast<uint32_t*>(await_ptr(p, kFlagDispatch, s)), flag_value(p, 0));
    if (kinds >> kFlagExpert & 1u)  // rank i's outputs are there for the tokens of rank s
        st_relaxed_gpu(s == p.rank ? seen_ptr(p, kFlagExpert, s) : flag_ptr(p.peer[s], p.off_flags, kFlagExpert, p.rank), flag_value(p, 0));
}

// ---------------------------------------------------------------------------
// Role 1.  A warp's item is U 16-byte vectors a lane of a token's row, in blocks that take no second one: a fixed share
// for each resident block leaves the SMs that are farther from the memory the rows go to at work when the others are through.
//   PUSH: y[t] = T(sum over the ranks d holding experts of t, ascending, of float(T(sum over k at d of w[t,k] * float(row k)))),
//         the order and the roundings of a group with a GPU each.
//   PULL: y[t] = T(sum over k of w[t,k] * float(row k)).
// WHOLE, for all ranks together, writes that.  Otherwise a combine follows: where outputs lie over rows that are still to be
// read, where a rank's experts run by themselves, and where the expert rows are the caller's before a PULL combine; PUSH then
// writes the partial rows to the home ranks' buffers.  (The two in one kernel: 2 % slower at the headline workload, 7 % with FP8 rows.)
// What bounds it: the stores, K + 1 for each load; expert rows leave the L2 first, outputs, which the next layer reads, do not.
// Eight ranks of 256 tokens of 7168, top-8 of 256 experts: 54.3, 294 MB at 5.4 TB/s (with partial rows written by one role and
// read by the next 134 a call, not captured); FP8 rows 58.0 (142), the quantiser's arithmetic on top; PULL, 200 tokens 44.0 (91);
// of 2048, top-6 of 64, skewed 17.4 to 17.9 (44).
// Rows stored without evict-first: skewed 18.8 for 17.9, two ranks of 200 tokens 15.2 / 14.4, one rank of 2048 53.0 / 52.3, headline
// no difference.  Inputs loaded with it too: one rank of 2048 51.9, but 1500 of 2880 12.7 / 11.9, two ranks of 200 15.7 / 14.4.
// Slower by more when they were tried: four vectors a lane at two blocks per SM (13 %), two at four (64 registers, spills: 49 %),
// pairs' rows looked up one by one (7 %).
// ---------------------------------------------------------------------------
template <typename T, int PAYLOAD, bool PUSH, bool WHOLE, int U, int N>
__global__ void __launch_bounds__(kThreads, 3) near_rows_kernel(const __grid_constant__ NearParams<N> g) {
    begin_after_previous();
    __shared__ int s_here[A2A_MAX_WORLD];
    const DevParams& p0 = g.p[0];
    const int tid = threadIdx.x, lane = tid & 31, ws = N == 1 ? 1 : p0.ws, K = p0.K, nvec = p0.H >> 3;
    const int nchunk = (nvec + 32 * U - 1) / (32 * U);
    const uint32_t want = flag_value(p0, 0);
    stamp(p0, kStampStart);
    if (!g.handed_on) {  // a rank's flag goes up when all its pairs are written, to whichever rank it is raised
        if (tid < ws) s_here[tid] = wait_flag_gpu(await_ptr(p0, kFlagDispatch, tid), want, p0, kPhaseRecv, tid);
        __syncthreads();
    }
    const long long it = (long long)blockIdx.x * (kThreads / 32) + (tid >> 5);
    long long t = it / nchunk;
    const int v0 = (int)(it - t * nchunk) * 32 * U + lane;
    int s = 0;
    while (s < ws && t >= g.T[s]) t -= g.T[s++];
    if (s < ws && (g.handed_on || s_here[s])) {
        uint4 q[U];
        const uint4* src = reinterpret_cast<const uint4*>(g.x[s]) + (size_t)t * nvec + v0;
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (v0 + u * 32 < nvec) q[u] = ld_input(src + u * 32);
        uint2 pair = make_uint2(kNoPair, 0u);  // lane k: pair k
        if (lane < K) pair = ld_stream(g.pairs[s] + (size_t)t * K + lane);
        // lane k: the rank of pair k, or -1 where it has no row or is not served, and this lane's place in its slab row
        int my_rank = pair.x == kNoPair ? -1 : (int)(pair.x >> 28);
        if (!WHOLE && g.n != ws && my_rank != p0.rank) my_rank = -1;
        unsigned long long my_row = 0;
        if (my_rank >= 0) {
            uint4* rows = reinterpret_cast<uint4*>(p0.peer[N == 1 ? 0 : my_rank] + p0.off_rows);
            my_row = reinterpret_cast<unsigned long long>(rows + (size_t)(pair.x & kPairRow) * nvec);
        }
        if (PAYLOAD == A2A_PAYLOAD_FP8) {  // nvec % 16 == 0: a scale block's lanes are all in or all out
#pragma unroll
            for (int u = 0; u < U; ++u) q[u] = fp8_round_trip<T>(q[u], v0 + u * 32 < nvec);
        }
        float acc[U][8];
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int e = 0; e < 8; ++e) acc[u][e] = 0.f;
        // the slab row of pair k, and its share of a sum
        auto expert_row = [&](int k, const uint4 (&out)[U], float (&sum)[U][8]) {
            uint4* row = reinterpret_cast<uint4*>(__shfl_sync(0xffffffffu, my_row, k)) + v0;
            const float w = __uint_as_float(__shfl_sync(0xffffffffu, pair.y, k));
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (v0 + u * 32 < nvec) __stcs(row + u * 32, out[u]);
                float f[8];
                unpack8<T>(out[u], f);
                fma8(f, w, sum[u]);
            }
        };
        if (PUSH) {
            for (unsigned ranks = __reduce_or_sync(0xffffffffu, my_rank >= 0 ? 1u << my_rank : 0u); ranks != 0u; ranks &= ranks - 1u) {
                const int d = __ffs(ranks) - 1;
                uint4 out[U];
                float part[U][8];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    out[u] = scale8<T>(q[u], (float)(1 + d));
#pragma unroll
                    for (int e = 0; e < 8; ++e) part[u][e] = 0.f;
                }
                for (unsigned left = __ballot_sync(0xffffffffu, my_rank == d); left != 0u; left &= left - 1u)  // k ascending
                    expert_row(__ffs(left) - 1, out, part);
                uint4* home = reinterpret_cast<uint4*>(p0.peer[s] + p0.off_ret) + ((size_t)d * p0.T_max + t) * nvec + v0;
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const uint4 r = pack8<T>(part[u]);
                    if (!WHOLE && v0 + u * 32 < nvec) st_stream(home + u * 32, r);
                    float f[8];
                    unpack8<T>(r, f);
#pragma unroll
                    for (int e = 0; e < 8; ++e) acc[u][e] += f[e];
                }
            }
        } else {
            uint4 out[U];
            if (N == 1) {
#pragma unroll
                for (int u = 0; u < U; ++u) out[u] = scale8<T>(q[u], 1.f);
            }
            for (unsigned left = __ballot_sync(0xffffffffu, my_rank >= 0); left != 0u; left &= left - 1u) {
                const int k = __ffs(left) - 1, d = N == 1 ? 0 : __shfl_sync(0xffffffffu, my_rank, k);
                if (N > 1) {
#pragma unroll
                    for (int u = 0; u < U; ++u) out[u] = scale8<T>(q[u], (float)(1 + d));
                }
                expert_row(k, out, acc);
            }
        }
        if (WHOLE) {
            uint4* y = reinterpret_cast<uint4*>(g.p[s].y) + (size_t)t * nvec + v0;
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (v0 + u * 32 < nvec) st_stream(y + u * 32, pack8<T>(acc[u]));
        }
    }
    if (g.handed_on) {
        // one rank with many tokens: its last launch; phases called on this context after it find its flags up
        if (N == 1 && blockIdx.x == 0 && tid == 0) *seen_ptr(p0, kFlagDispatch, 0) = *seen_ptr(p0, kFlagExpert, 0) = want;
    } else if (grid_arrive_last(p0.ptickets + kPipeTicketSource * A2A_MAX_WORLD, (int)gridDim.x)) {
        // The block that arrives last tells every home rank that the expert outputs and partial rows are there, unless a
        // wait of one of the ranks gave up.  Every block arrives, whatever happened: the ticket is whole for the next call.
        if constexpr (N > 1) raise_flags(g, 1u << kFlagExpert, recorded_of_rank(g));
    }
    stamp(p0, kStampExpertDone);
}

// ---------------------------------------------------------------------------
// Role 2 where role 1 has written the outputs, and RECV of rows that are in their slabs already.  In a call whose launches follow
// one another it raises the flags that nobody has needed until then, also where such a call ends early; otherwise it ends when
// those of the last kind are up.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(A2A_MAX_WORLD * A2A_MAX_WORLD) near_flags_kernel(const __grid_constant__ NearGroup g, int kinds) {
    // looked at while the launch before this one ends: no launch of a call that is handed on waits for anything, or records that it did
    const int recorded = recorded_of_rank(g);
    begin_after_previous();
    const int ws = g.p[0].ws, i = threadIdx.x / ws, s = threadIdx.x % ws;
    const bool expert = kinds >> kFlagExpert & 1;
    stamp(g.p[0], kStampStart);
    if (g.handed_on)
        raise_flags(g, (unsigned)kinds, recorded);
    else if (i < g.n)
        wait_flag_gpu(await_ptr(g.p[i], expert ? kFlagExpert : kFlagDispatch, s), flag_value(g.p[i], 0), g.p[i],
                      expert ? kPhaseCombine : kPhaseRecv, s);
    stamp(g.p[0], kStampCombineDone);
}

// ---------------------------------------------------------------------------
// The phases that a program with its own expert kernels calls, for all ranks of a group on one GPU: the same lists.  A token's
// place in memory follows from its number and its pairs' places are looked up, so that no launch counts, scans or searches before
// its first row.  What bounds them: with tens of MB of rows the latencies (four ranks of 117 tokens of 4096, top-8: SEND 9.7, RECV 3.0,
// EXPERT 8.8, COMBINE 7.1 by themselves, 25.1 handed on from one to the next and 33.5 as four calls, in which tickets, flags and waits
// are in every launch; by counts and bitmaps 33.3 handed on), with hundreds the memory (eight of 200 of 7168, 183 MB: 40, 4, 54, 37 by
// themselves, 130 handed on, 151 as four calls; through the stages 193 handed on).
// ---------------------------------------------------------------------------
// A warp's item in a launch whose blocks take no second one: U vectors a lane, from v0 on, of token t of rank s.
template <int U>
struct NearItem {
    int s, t, v0;
    bool there;
    __device__ __forceinline__ explicit NearItem(const NearGroup& g) {
        const int ws = g.p[0].ws, nvec = g.p[0].H >> 3, nchunk = (nvec + 32 * U - 1) / (32 * U);
        const long long it = (long long)(g.backwards ? gridDim.x - 1 - blockIdx.x : blockIdx.x) * (kThreads / 32) + (threadIdx.x >> 5);
        long long row = it / nchunk;
        v0 = (int)(it - row * nchunk) * 32 * U + (threadIdx.x & 31);
        s = g.n == ws ? 0 : g.p[0].rank;  // the tokens of all ranks, or of the one served
        const int end = g.n == ws ? ws : s + 1;
        while (s < end && row >= g.T[s]) row -= g.T[s++];
        there = s < end;
        t = (int)row;
    }
};

// Lane k: where the slab row of the item's pair k lies (this lane's first vector of it), and at which rank; -1: nowhere.
// LISTED: role 0 or SEND of the group has left the places; else they follow from the slots and the caller's indices.
template <bool LISTED>
__device__ __forceinline__ unsigned long long near_row(const NearGroup& g, int s, int t, int v0, int& rank) {
    const DevParams& p0 = g.p[0];
    const int lane = threadIdx.x & 31;
    unsigned place = kNoPair;
    if (lane < p0.K) {
        const size_t pair = (size_t)t * p0.K + lane;
        if (LISTED) {
            place = ld_stream(g.pairs[s] + pair).x;
        } else {
            const int e = ld_input(g.p[s].idx + pair), j = ld_stream(g.p[s].slot + pair);
            if (j >= 0) place = pair_place(p0, s, e, j);
        }
    }
    rank = place == kNoPair ? -1 : (int)(place >> 28);
    if (rank < 0) return 0;
    uint4* rows = reinterpret_cast<uint4*>(p0.peer[rank] + p0.off_rows);
    return reinterpret_cast<unsigned long long>(rows + (size_t)(place & kPairRow) * (p0.H >> 3));
}

// SEND: routing and sending in one launch.  A block takes a contiguous range of a rank's (token, chunk) items, as solo_kernel does,
// and resolves the pairs of a round by the same loop; it stands in both (a2a_solo.cuh), since as a function it cost solo_kernel
// 0.17 us.  Whatever the payload, a row, read once (and FP8, quantised and dequantised once), goes straight into the slabs: a stage
// is what a link needs.
template <typename T, bool FP8, int U>
__global__ void __launch_bounds__(kThreads, 3) near_dispatch_kernel(const __grid_constant__ NearGroup g) {
    __shared__ int s_cnt[A2A_MAX_EXPERTS];                  // tokens before the current round that use expert e
    __shared__ int s_idx[kSoloRound * A2A_MAX_TOPK];        // the round's indices
    __shared__ unsigned s_place[kSoloRound * A2A_MAX_TOPK]; // and where its pairs' rows go
    begin_after_previous();
    const DevParams& p = g.p[blockIdx.x % g.n];
    const int b = (int)blockIdx.x / g.n, G = (int)gridDim.x / g.n;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int K = p.K, nvec = p.H >> 3, nchunk = (nvec + 32 * U - 1) / (32 * U);
    const long long items = (long long)p.T * nchunk;
    const long long lo = items * b / G, hi = items * (b + 1) / G;
    const int t0 = (int)(lo / nchunk), t1 = (int)((hi + nchunk - 1) / nchunk);
    auto load = [&](int t, int c, uint4 (&q)[U]) {
        const uint4* src = reinterpret_cast<const uint4*>(p.x) + (size_t)t * nvec;
#pragma unroll
        for (int u = 0; u < U; ++u)
            if ((c * U + u) * 32 + lane < nvec) q[u] = ld_input(src + (c * U + u) * 32 + lane);
    };
    // the first item's row and the first round's pairs are requested before anything else: they need no routing
    long long it = lo + warp;
    int t = (int)(it / nchunk), c = (int)(it - (long long)t * nchunk);
    uint4 q[U];
    if (it < hi) load(t, c, q);
    const int first_e = tid < min(kSoloRound, t1 - t0) * K ? ld_input(p.idx + (size_t)t0 * K + tid) : 0;
    for (int e = tid; e < p.E; e += kThreads) s_cnt[e] = 0;
    __syncthreads();
    count_experts_before<kThreads>(p, t0, s_cnt);
    for (int r0 = t0; r0 < t1; r0 += kSoloRound) {
        const int nt = min(kSoloRound, t1 - r0), pairs = nt * K;
        for (int i = tid; i < pairs; i += kThreads) s_idx[i] = r0 == t0 && i == tid ? first_e : ld_input(p.idx + (size_t)r0 * K + i);
        __syncthreads();
        for (int i = tid; i < pairs; i += kThreads) {
            const int tl = i / K, k = i - tl * K, e = s_idx[i];
            bool ok = e >= 0 && e < p.E;
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
            const unsigned place = ok ? pair_place(p, p.rank, e, j) : kNoPair;
            s_place[i] = place;
            if ((long long)(r0 + tl) * nchunk >= lo) {  // the block that has the token's first chunk books its pairs
                p.slot[(size_t)r0 * K + i] = j;
                p.pairs[(size_t)r0 * K + i] = make_uint2(place, 0u);
                if (ok) reinterpret_cast<int*>(p.peer[place >> 28] + p.off_meta)[place & kPairRow] = ((r0 + tl) << 8) | k;
                else record_error(p.status, A2A_ERR_ROUTING, p.rank, -1, kPhaseRoute, p.epoch, e);
            }
        }
        __syncthreads();
        for (int i = tid; i < pairs; i += kThreads)
            if (s_place[i] != kNoPair) atomicAdd(s_cnt + s_idx[i], 1);
        const long long end = min(hi, (long long)(r0 + nt) * nchunk);
        while (it < end) {
            const long long next = it + kSoloWarps;
            int tn = t, cn = c + kSoloWarps;
            while (cn >= nchunk) { cn -= nchunk; ++tn; }
            uint4 qn[U];
            if (next < hi) load(tn, cn, qn);
            const int v0 = c * 32 * U + lane;
            const unsigned place = lane < K ? s_place[(t - r0) * K + lane] : kNoPair;
            unsigned long long my_row = 0;
            if (place != kNoPair) {
                uint4* rows = reinterpret_cast<uint4*>(p.peer[place >> 28] + p.off_rows);
                my_row = reinterpret_cast<unsigned long long>(rows + (size_t)(place & kPairRow) * nvec);
            }
            if (FP8) {  // nvec % 16 == 0: a scale block's lanes are all in or all out
#pragma unroll
                for (int u = 0; u < U; ++u) q[u] = fp8_round_trip<T>(q[u], v0 + u * 32 < nvec);
            }
            for (unsigned left = __ballot_sync(0xffffffffu, place != kNoPair); left != 0u; left &= left - 1u) {
                uint4* row = reinterpret_cast<uint4*>(__shfl_sync(0xffffffffu, my_row, __ffs(left) - 1)) + v0;
#pragma unroll
                for (int u = 0; u < U; ++u)
                    if (v0 + u * 32 < nvec) st_stream(row + u * 32, q[u]);
            }
#pragma unroll
            for (int u = 0; u < U; ++u) q[u] = qn[u];
            it = next;
            t = tn;
            c = cn;
        }
        __syncthreads();
    }
    if (b == G - 1)  // this block's counts now cover every token
        for (int e = tid; e < p.E; e += kThreads) {
            const int d = e / p.L;
            reinterpret_cast<int*>(p.peer[d] + p.off_counts)[(size_t)p.rank * kMaxChunks * p.L + (e - d * p.L)] = s_cnt[e];
            p.send_counts[e] = s_cnt[e];
        }
    if (g.handed_on) return;
    __syncthreads();
    if (tid < p.ws) arrive_dest(p, tid, (uint32_t)G);
}

// EXPERT, and with WAIT RECV_EXPERT: the expert op on the slab rows, in place.
template <typename T, bool WAIT>
__global__ void __launch_bounds__(kThreads) near_expert_kernel(const __grid_constant__ NearGroup g) {
    begin_after_previous();
    __shared__ int s_missing;  // sources whose rows have not come
    const int tid = threadIdx.x, ws = g.p[0].ws, K = g.p[0].K, nvec = g.p[0].H >> 3;
    if (WAIT && g.handed_on) {
        if (blockIdx.x == 0) raise_flags(g, 1u << kFlagDispatch, recorded_of_rank(g));
    } else if (WAIT) {
        if (tid == 0) s_missing = 0;
        __syncthreads();
        if (tid < g.n * ws) {
            const DevParams& p = g.p[tid / ws];
            if (!wait_flag_gpu(await_ptr(p, kFlagDispatch, tid % ws), flag_value(p, 0), p, kPhaseRecv, tid % ws))
                atomicOr(&s_missing, 1 << tid % ws);
        }
        __syncthreads();
    }
    const NearItem<1> at(g);
    if (at.there && (!WAIT || g.handed_on || (s_missing >> at.s & 1) == 0)) {
        int rank;
        const unsigned long long my_row = near_row<true>(g, at.s, at.t, at.v0, rank);
        const unsigned there = __ballot_sync(0xffffffffu, rank >= 0);
        for (int k0 = 0; k0 < K; k0 += 8) {  // eight rows are requested before the first is written
            uint4 q[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                if ((there >> (k0 + i) & 1u) == 0u) continue;  // K <= 32: no bit beyond the last pair's
                const uint4* row = reinterpret_cast<const uint4*>(__shfl_sync(0xffffffffu, my_row, k0 + i)) + at.v0;
                if (at.v0 < nvec) q[i] = ld_stream(row);
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                if ((there >> (k0 + i) & 1u) == 0u) continue;
                uint4* row = reinterpret_cast<uint4*>(__shfl_sync(0xffffffffu, my_row, k0 + i)) + at.v0;
                const float scale = (float)(1 + __shfl_sync(0xffffffffu, rank, k0 + i));
                if (at.v0 < nvec) st_stream(row, scale8<T>(q[i], scale));
            }
        }
    }
    if (!g.handed_on && grid_arrive_last(g.p[0].ptickets + kPipeTicketSource * A2A_MAX_WORLD, (int)gridDim.x))
        raise_flags(g, 1u << kFlagExpert, recorded_of_rank(g));
}

// ---------------------------------------------------------------------------
// Role 2 and the combine of the phases.
//   PUSH: y[t] = T(sum over the ranks d holding experts of t, ascending, of float(partial[d][t])).
//   PULL: y[t] = T(sum over k of w[t,k] * float(row k)), eight rows requested before the first is used.
// ---------------------------------------------------------------------------
template <typename T, bool PUSH, bool LISTED, int U>
__global__ void __launch_bounds__(kThreads) near_combine_kernel(const __grid_constant__ NearGroup g) {
    begin_after_previous();
    const DevParams& p0 = g.p[0];
    const int tid = threadIdx.x, lane = tid & 31, ws = p0.ws, nvec = p0.H >> 3;
    stamp(p0, kStampStart);
    if (!PUSH && g.handed_on) {  // roles that are handed on have written the outputs
        if (blockIdx.x == 0) raise_flags(g, 1u << kFlagExpert, recorded_of_rank(g));
    } else if (PUSH) {
        bool ok = true;
        if (tid < g.n * ws) {
            const DevParams& p = g.p[tid / ws];
            ok = wait_flag_gpu(await_ptr(p, kFlagExpert, tid % ws), flag_value(p, 0), p, kPhaseCombine, tid % ws);
        }
        if (!__syncthreads_and(ok)) return;  // timeout recorded; y is left untouched
    }
    const NearItem<U> at(g);
    bool go = at.there;
    int rank = -1;
    unsigned long long my_row = 0;
    float my_w = 0.f;
    const DevParams& p = g.p[g.n == ws && go ? at.s : 0];
    if (go) {
        // The launch before this one has raised the flags of the ranks whose expert phase ran.  Where one is missing, tokens
        // wait for the ranks that have rows of theirs, and only for those: a rank without rows need not have run.
        bool up = true;  // lane d: rank d's outputs are there
        if (!PUSH && !g.handed_on) {
            if (lane < ws) up = (int32_t)(ld_relaxed_gpu(await_ptr(p, kFlagExpert, lane)) - flag_value(p, 0)) >= 0;
            fence_acq_rel_gpu();
        }
        my_row = near_row<LISTED>(g, at.s, at.t, at.v0, rank);
        if (!PUSH && lane < p0.K) my_w = ld_input(p.w + (size_t)at.t * p0.K + lane);
        const unsigned missing = ~__ballot_sync(0xffffffffu, up);
        if (!PUSH && __any_sync(0xffffffffu, rank >= 0 && (missing >> rank & 1u))) {
            bool ok = true;
            if (rank >= 0 && (missing >> rank & 1u)) {
                bool spent = false;  // one rank's budget is enough: the other ranks' tokens are told at once
                for (int i = 0; i < g.n; ++i) spent = spent || ld_volatile_i32(&g.p[i].status->code) == A2A_ERR_TIMEOUT;
                if (spent) {
                    ok = (int32_t)(ld_relaxed_gpu(await_ptr(p, kFlagExpert, rank)) - flag_value(p, 0)) >= 0;
                    if (!ok) record_timeout(p, kPhaseCombine, rank, flag_value(p, 0));
                    fence_acq_rel_gpu();
                } else {
                    ok = wait_flag_gpu(await_ptr(p, kFlagExpert, rank), flag_value(p, 0), p, kPhaseCombine, rank);
                }
            }
            go = __all_sync(0xffffffffu, ok);  // timeout recorded; the token's output is left untouched
        }
    }
    if (go) {
        float acc[U][8];
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int e = 0; e < 8; ++e) acc[u][e] = 0.f;
        const unsigned mine = PUSH ? __reduce_or_sync(0xffffffffu, rank >= 0 ? 1u << rank : 0u) : __ballot_sync(0xffffffffu, rank >= 0);
        const uint4* ret = reinterpret_cast<const uint4*>(p.peer[p.rank] + p0.off_ret) + (size_t)at.t * nvec + at.v0;
        for (int k0 = 0; k0 < (PUSH ? A2A_MAX_WORLD : p0.K); k0 += 8) {
            uint4 q[8][U];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                if ((mine >> (k0 + i) & 1u) == 0u) continue;  // K <= 32: no bit beyond the last pair's
                const uint4* row = PUSH ? ret + (size_t)i * p0.T_max * nvec
                                        : reinterpret_cast<const uint4*>(__shfl_sync(0xffffffffu, my_row, k0 + i)) + at.v0;
#pragma unroll
                for (int u = 0; u < U; ++u)
                    if (at.v0 + u * 32 < nvec) q[i][u] = __ldcs(row + u * 32);
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                if ((mine >> (k0 + i) & 1u) == 0u) continue;
                const float w = PUSH ? 1.f : __shfl_sync(0xffffffffu, my_w, k0 + i);
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    float f[8];
                    unpack8<T>(q[i][u], f);
                    if (PUSH) {
#pragma unroll
                        for (int e = 0; e < 8; ++e) acc[u][e] += f[e];
                    } else {
                        fma8(f, w, acc[u]);
                    }
                }
            }
        }
        uint4* y = reinterpret_cast<uint4*>(p.y) + (size_t)at.t * nvec + at.v0;
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (at.v0 + u * 32 < nvec) st_stream(y + u * 32, pack8<T>(acc[u]));
    }
    // role 2 is through when every rank is, also those whose outputs no token wants
    if (!PUSH && g.every_rank && !g.handed_on && blockIdx.x == 0 && tid < g.n * ws) {
        const DevParams& p = g.p[tid / ws];
        wait_flag_gpu(await_ptr(p, kFlagExpert, tid % ws), flag_value(p, 0), p, kPhaseCombine, tid % ws);
    }
    stamp(p0, kStampCombineDone);
}

}  // namespace a2a
