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
// One rank with many tokens is a group of one.
#pragma once

#include "a2a_solo.cuh"

namespace a2a {

// The ranks a launch serves (`n` of them, all of a group or one) and what role 0 knew or found of every rank.  N: the
// most ranks a group may have; a type of its own for a single rank, whose launches are the cheaper for it (1500 tokens of 2880
// in two launches 14.4 us with room for eight, 14.0 without).
template <int N>
struct NearParams {
    DevParams p[N];
    const void* x[N];       // input rows of rank s in this call
    const uint2* pairs[N];  // its (token, k) pairs as near_route_kernel left them
    int T[N];               // and its tokens
    int n;
    int every_rank;  // a PULL combine ends only when every rank's outputs are there, also those no token wants
    int output;      // role 1: kOutput...
    int handed_on;   // the launches of one call, one after the other on one stream: no flag is awaited or raised before the last
};
using NearGroup = NearParams<A2A_MAX_WORLD>;
enum NearOutput : int { kOutputNone = 0, kOutputWhole = 1, kOutputPartial = 2 };

// A pair as role 1 reads it: where its slab row lies, as (rank << 28 | row of that rank's slabs), and its weight.
constexpr unsigned kNoPair = 0xffffffffu;
static_assert((long long)A2A_MAX_EXPERTS * 65535 < 1 << 28 && A2A_MAX_WORLD <= 8, "a slab row fits 28 bits, a rank three");

// ---------------------------------------------------------------------------
// Role 0: routing.  A block takes `words` * 32 tokens of a rank: it counts the experts of the tokens before them once
// more for itself (64 KB at 2048 x 8, out of the L2) instead of waiting for another block.  What bounds it: the chain
// launch -> indices -> counts -> slots -> stores.
// ---------------------------------------------------------------------------
constexpr int kRouteThreads = 1024;
__host__ __device__ inline size_t near_route_smem(int words, int E, int K) { return ((size_t)(words + 1) * E + (size_t)words * 64 * K) * 4; }

template <int N>
__global__ void __launch_bounds__(kRouteThreads) near_route_kernel(const __grid_constant__ NearParams<N> g, int words) {
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
        for (int i = tid; i < pairs; i += kRouteThreads) {
            s_idx[i] = ld_input(p.idx + (size_t)t0 * K + i);
            s_w[i] = ld_input(p.w + (size_t)t0 * K + i);
        }
        for (int e = tid; e < (words + 1) * E; e += kRouteThreads) s_cnt[e] = 0;
        __syncthreads();
        count_experts_before<kRouteThreads>(p, t0, s_cnt);
        auto first_use = [&](int i) {  // pair i's expert is in range and of no earlier pair of its token
            const int e = s_idx[i];
            bool ok = e >= 0 && e < E;
            for (int j = i / K * K; ok && j < i; ++j) ok = s_idx[j] != e;
            return ok;
        };
        for (int i = tid; i < pairs; i += kRouteThreads)
            if (first_use(i)) atomicOr(s_bits + (i / K >> 5) * E + s_idx[i], 1u << (i / K & 31));
        __syncthreads();
        for (int i = tid; i < pairs; i += kRouteThreads) {
            const size_t at = (size_t)t0 * K + i;
            const int tl = i / K, e = s_idx[i];
            int j = -1;
            unsigned place = kNoPair;
            if (first_use(i)) {
                j = s_cnt[e];
                for (int w = 0; w < tl >> 5; ++w) j += __popc(s_bits[w * E + e]);
                j += __popc(s_bits[(tl >> 5) * E + e] & ((1u << (tl & 31)) - 1u));
                const int d = e / p.L, row = ((e - d * p.L) * p.ws + p.rank) * p.T_max + j;
                place = (unsigned)d << 28 | (unsigned)row;
                reinterpret_cast<int*>(p.peer[d] + p.off_meta)[row] = ((t0 + tl) << 8) | (i - tl * K);
            } else {
                record_error(p.status, A2A_ERR_ROUTING, p.rank, -1, kPhaseRoute, p.epoch, e);
            }
            p.slot[at] = j;
            p.pairs[at] = make_uint2(place, __float_as_uint(s_w[i]));
        }
        if (last)
            for (int e = tid; e < E; e += kRouteThreads) {
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

// Rank p's expert outputs are there for the tokens of rank s; a fence before.
__device__ __forceinline__ void raise_expert_flag(const DevParams& p, int s) {
    uint32_t* flag = s == p.rank ? seen_ptr(p, kFlagExpert, s) : flag_ptr(p.peer[s], p.off_flags, kFlagExpert, p.rank);
    st_relaxed_gpu(flag, flag_value(p, 0));
}

// ---------------------------------------------------------------------------
// Role 1.  A warp's item is U 16-byte vectors a lane of a token's row, in blocks that take no second one: a fixed share
// for each resident block leaves the SMs that are farther from the memory the rows go to at work when the others are through.
//   PUSH: y[t] = T(sum over the ranks d holding experts of t, ascending, of float(T(sum over k at d of w[t,k] * float(row k)))),
//         the order and the roundings of a group with a GPU each.
//   PULL: y[t] = T(sum over k of w[t,k] * float(row k)).
// kOutputWhole writes that; kOutputPartial the partial rows to the home ranks' buffers, for near_combine_kernel: where
// outputs lie over rows that are still to be read, and where a rank's experts run by themselves; kOutputNone neither.
// What bounds it: the stores, K + 1 for each load; expert rows leave the L2 first, outputs, which the next layer reads, do not.
// Eight ranks of 256 tokens of 7168, top-8 of 256 experts, a call: 56 us, 294 MB at 5.2 TB/s (134 with partial rows written
// by one role, 87, and read by the next, 33; FP8 rows 66, 142; PULL, 200 tokens 44, 91); of 2048, top-6 of 64, skewed 19 (44).
// Slower: rows stored without evict-first (two ranks of 200 tokens 17.2 us against 16.2, skewed 21.6 / 20.4, headline 1 %), four
// vectors a lane at two blocks per SM (13 %), two at four (64 registers, spills: 49 %), pairs' rows looked up one by one (7 %).  One rank
// of 2048 tokens of 7168 54.6, inputs loaded with evict-first too 53.8, but 1500 of 2880 12.9 / 14.1.  FP8: the quantiser's arithmetic on top.
// ---------------------------------------------------------------------------
template <typename T, int PAYLOAD, bool PUSH, int U, int N>
__global__ void __launch_bounds__(kThreads, 3) near_rows_kernel(const __grid_constant__ NearParams<N> g) {
    begin_after_previous();
    __shared__ int s_here[A2A_MAX_WORLD];
    const DevParams& p0 = g.p[0];
    const int tid = threadIdx.x, lane = tid & 31, ws = N == 1 ? 1 : p0.ws, K = p0.K, nvec = p0.H >> 3, nchunk = (nvec + 32 * U - 1) / (32 * U);
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
        if (N > 1 && g.n != ws && my_rank != p0.rank) my_rank = -1;
        unsigned long long my_row = 0;
        if (my_rank >= 0)
            my_row = reinterpret_cast<unsigned long long>(reinterpret_cast<uint4*>(p0.peer[N == 1 ? 0 : my_rank] + p0.off_rows) + (size_t)(pair.x & 0x0fffffffu) * nvec);
        if (PAYLOAD == A2A_PAYLOAD_FP8) {
#pragma unroll
            for (int u = 0; u < U; ++u) q[u] = fp8_round_trip<T>(q[u], v0 + u * 32 < nvec);  // nvec % 16 == 0: a scale block's lanes are all in or all out
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
                for (unsigned left = __ballot_sync(0xffffffffu, my_rank == d); left != 0u; left &= left - 1u) expert_row(__ffs(left) - 1, out, part);  // k ascending
                uint4* home = reinterpret_cast<uint4*>(p0.peer[s] + p0.off_ret) + ((size_t)d * p0.T_max + t) * nvec + v0;
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const uint4 r = pack8<T>(part[u]);
                    if (g.output == kOutputPartial && v0 + u * 32 < nvec) st_stream(home + u * 32, r);
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
        if (g.output == kOutputWhole) {
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
        const DevParams& p = g.p[tid < g.n * ws ? tid / ws : 0];
        const bool whole = __syncthreads_and(ld_volatile_i32(&p.status->code) != A2A_ERR_TIMEOUT);
        fence_acq_rel_gpu();
        if (whole && tid < g.n * ws) raise_expert_flag(p, tid % ws);
    }
    stamp(p0, kStampExpertDone);
}

// ---------------------------------------------------------------------------
// Role 2 where role 1 has written the outputs.  In a call whose launches follow one another it raises the flags of both
// phases, which nobody has needed until then; otherwise it ends when every rank's expert flag is up, as any combine.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(A2A_MAX_WORLD * A2A_MAX_WORLD) near_finish_kernel(const __grid_constant__ NearGroup g) {
    begin_after_previous();
    const int ws = g.p[0].ws, i = threadIdx.x / ws, s = threadIdx.x % ws;
    const DevParams& p = g.p[i < g.n ? i : 0];
    stamp(g.p[0], kStampStart);
    if (!g.handed_on) {
        if (i < g.n) wait_flag_gpu(await_ptr(p, kFlagExpert, s), flag_value(p, 0), p, kPhaseCombine, s);
    } else if (__syncthreads_and(ld_volatile_i32(&p.status->code) != A2A_ERR_TIMEOUT) && i < g.n) {
        fence_acq_rel_gpu();
        st_relaxed_gpu(const_cast<uint32_t*>(await_ptr(p, kFlagDispatch, s)), flag_value(p, 0));
        raise_expert_flag(p, s);
    }
    stamp(g.p[0], kStampCombineDone);
}

// ---------------------------------------------------------------------------
// Role 2.  A warp's item is a piece of a token's output row; the tokens of all ranks are one list, the last rank's
// first: what was written for them was written last and is still in the L2.  What an item reads first, the token's
// experts, is requested one or two items ahead.
//   PUSH: y[t] = T(sum over the ranks d holding experts of t, ascending, of float(partial[d][t])).
//   PULL: y[t] = T(sum over k of w[t,k] * float(row k)), eight rows requested before the first is used.
// Eight ranks of 256 tokens of 7168, top-8 of 256 experts, PUSH: 33 us (154 MB of partial rows read, some from the L2),
// 44 with the ranks side by side and the experts looked up when needed; 200 tokens, PULL: 36, 53.  One vector a lane
// at three or four blocks per SM: 37 and 41 (PULL); PUSH with two: 49 to 56.
// ---------------------------------------------------------------------------
struct NearTokens {
    struct At {  // piece ch of token `row` of the list, one of the tokens of rank position n - 1 - at
        int row, ch, at;
    };
    const int* pre;  // shared memory [n + 1]
    int total, nchunk, step_row, step_ch;
    __device__ __forceinline__ void settle(At& a) const {
        while (a.row < total && a.row >= pre[a.at + 1]) ++a.at;
    }
    __device__ __forceinline__ At first() const {
        const int w = (int)blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5);
        At a = {w / nchunk, w % nchunk, 0};
        settle(a);
        return a;
    }
    __device__ __forceinline__ At after(const At& a) const {
        At b = {a.row + step_row, a.ch + step_ch, a.at};
        if (b.ch >= nchunk) {
            b.ch -= nchunk;
            ++b.row;
        }
        settle(b);
        return b;
    }
};

// The list; with WAIT, once every expert flag of the ranks served is up.  False where one is not.
template <bool WAIT>
__device__ __forceinline__ bool near_tokens(const NearGroup& g, int* s_pre, int nchunk, NearTokens& list) {
    const int tid = threadIdx.x, ws = g.p[0].ws, warps = (int)gridDim.x * (kThreads / 32);
    bool ok = true;
    if (tid < g.n * ws) {
        const DevParams& p = g.p[tid / ws];
        const uint32_t* flag = await_ptr(p, kFlagExpert, tid % ws);
        if (WAIT) {
            ok = wait_flag_gpu(flag, flag_value(p, 0), p, kPhaseCombine, tid % ws);
        } else {
            ok = (int32_t)(ld_relaxed_gpu(flag) - flag_value(p, 0)) >= 0;
            fence_acq_rel_gpu();
        }
    }
    if (tid == 0) {
        int sum = 0;
        for (int i = 0; i <= g.n; ++i) {
            s_pre[i] = sum;
            if (i < g.n) sum += g.p[g.n - 1 - i].T;
        }
    }
    ok = __syncthreads_and(ok);
    list = {s_pre, s_pre[g.n], nchunk, warps / nchunk, warps % nchunk};
    return ok;
}

template <typename T>
__device__ __forceinline__ void near_combine_push(const NearGroup& g, int* s_pre) {
    const int lane = threadIdx.x & 31;
    const DevParams& p0 = g.p[0];
    const int K = p0.K, nvec = p0.H >> 3, T_max = p0.T_max;
    NearTokens list;
    if (!near_tokens<true>(g, s_pre, (nvec + 127) >> 7, list)) return;  // timeout recorded; y is left untouched
    auto bit_of = [&](const NearTokens::At& a) {  // lane k: the rank of pair k
        if (a.row >= list.total || lane >= K) return 0u;
        const int e = ld_input(g.p[g.n - 1 - a.at].idx + (size_t)(a.row - s_pre[a.at]) * K + lane);
        return e >= 0 && e < p0.E ? 1u << (e / p0.L) : 0u;
    };
    NearTokens::At a0 = list.first();
    unsigned bit = bit_of(a0);
    while (a0.row < list.total) {
        const unsigned mask = __reduce_or_sync(0xffffffffu, bit);
        const NearTokens::At a1 = list.after(a0);
        bit = bit_of(a1);
        const DevParams& p = g.p[g.n - 1 - a0.at];
        const int t = a0.row - s_pre[a0.at], v0 = a0.ch * 128 + lane;
        const uint4* ret = reinterpret_cast<const uint4*>(p.peer[p.rank] + p0.off_ret) + (size_t)t * nvec + v0;
        float acc[4][8];
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int e = 0; e < 8; ++e) acc[u][e] = 0.f;
#pragma unroll
        for (int d = 0; d < A2A_MAX_WORLD; d += 4) {  // sixteen loads in flight per lane
            if (((mask >> d) & 0xfu) == 0u) continue;
            uint4 q[4][4];
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if ((mask >> (d + j)) & 1u) {
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                        if (v0 + u * 32 < nvec) q[j][u] = __ldcs(ret + (size_t)(d + j) * T_max * nvec + u * 32);
                }
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if ((mask >> (d + j)) & 1u) {
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        float f[8];
                        unpack8<T>(q[j][u], f);
#pragma unroll
                        for (int e = 0; e < 8; ++e) acc[u][e] += f[e];
                    }
                }
        }
        uint4* y = reinterpret_cast<uint4*>(p.y) + (size_t)t * nvec + v0;
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (v0 + u * 32 < nvec) __stcs(y + u * 32, pack8<T>(acc[u]));
        a0 = a1;
    }
}

template <typename T>
__device__ __forceinline__ void near_combine_pull(const NearGroup& g, int* s_pre) {
    constexpr int U = 2;
    const int lane = threadIdx.x & 31;
    const DevParams& p0 = g.p[0];
    const int ws = p0.ws, K = p0.K, nvec = p0.H >> 3, T_max = p0.T_max;
    NearTokens list;
    // The launch before this one has raised the flags of the ranks whose expert phase ran.  Where one is missing, tokens
    // wait for the ranks that have rows of theirs, and only for those: a rank without rows need not have run.
    const bool all_up = near_tokens<false>(g, s_pre, (nvec + 32 * U - 1) / (32 * U), list);
    struct Pair {  // lane k: expert, slot and weight of pair k
        int e, j;
        float w;
    };
    auto pair_of = [&](const NearTokens::At& a) {
        Pair r = {-1, -1, 0.f};
        if (a.row < list.total && lane < K) {
            const DevParams& p = g.p[g.n - 1 - a.at];
            const size_t i = (size_t)(a.row - s_pre[a.at]) * K + lane;
            r.e = ld_input(p.idx + i);
            r.j = ld_stream(p.slot + i);
            r.w = ld_input(p.w + i);
        }
        return r;
    };
    NearTokens::At a0 = list.first(), a1 = list.after(a0);
    Pair r0 = pair_of(a0), r1 = pair_of(a1);
    auto go_on = [&](const NearTokens::At& a2, const Pair& r2) {
        a0 = a1;
        a1 = a2;
        r0 = r1;
        r1 = r2;
    };
    bool waited = false;
    while (a0.row < list.total) {
        const NearTokens::At a2 = list.after(a1);
        const Pair r2 = pair_of(a2);
        const DevParams& p = g.p[g.n - 1 - a0.at];
        const int t = a0.row - s_pre[a0.at], v0 = a0.ch * 32 * U + lane;
        const bool valid = r0.e >= 0 && r0.e < p0.E && r0.j >= 0;
        const int d = valid ? r0.e / p0.L : 0;
        if (!all_up) {
            const uint32_t* flag = await_ptr(p, kFlagExpert, d);
            const uint32_t want = flag_value(p, 0);
            bool ok = true;
            if (valid && !waited) {
                ok = wait_flag_gpu(flag, want, p, kPhaseCombine, d);
            } else if (valid) {  // one budget is spent: the other ranks' tokens are told at once
                ok = (int32_t)(ld_relaxed_gpu(flag) - want) >= 0;
                if (!ok) record_timeout(p, kPhaseCombine, d, want);
                fence_acq_rel_gpu();
            }
            if (!__all_sync(0xffffffffu, ok)) {  // timeout recorded; the token's output is left untouched
                waited = true;
                go_on(a2, r2);
                continue;
            }
        }
        unsigned long long my_row = 0;
        if (valid)
            my_row = reinterpret_cast<unsigned long long>(reinterpret_cast<const uint4*>(p0.peer[d] + p0.off_rows) +
                                                          (((size_t)(r0.e - d * p0.L) * ws + p.rank) * T_max + r0.j) * nvec);
        const unsigned there = __ballot_sync(0xffffffffu, valid);
        float acc[U][8];
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int e = 0; e < 8; ++e) acc[u][e] = 0.f;
        for (int k0 = 0; k0 < K; k0 += 8) {
            uint4 q[8][U];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                if (((there >> (k0 + i)) & 1u) == 0u) continue;  // K <= 32: no bit beyond the last pair's
                const uint4* row = reinterpret_cast<const uint4*>(__shfl_sync(0xffffffffu, my_row, k0 + i)) + v0;
#pragma unroll
                for (int u = 0; u < U; ++u)
                    if (v0 + u * 32 < nvec) q[i][u] = __ldcs(row + u * 32);
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                if (((there >> (k0 + i)) & 1u) == 0u) continue;
                const float w = __shfl_sync(0xffffffffu, r0.w, k0 + i);
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    float f[8];
                    unpack8<T>(q[i][u], f);
                    fma8(f, w, acc[u]);
                }
            }
        }
        uint4* y = reinterpret_cast<uint4*>(p.y) + (size_t)t * nvec + v0;
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (v0 + u * 32 < nvec) __stcs(y + u * 32, pack8<T>(acc[u]));
        go_on(a2, r2);
    }
    if (!all_up && g.every_rank && blockIdx.x == 0 && threadIdx.x < g.n * ws) {
        const DevParams& p = g.p[threadIdx.x / ws];
        wait_flag_gpu(await_ptr(p, kFlagExpert, threadIdx.x % ws), flag_value(p, 0), p, kPhaseCombine, threadIdx.x % ws);
    }
}

template <typename T, bool PUSH>
__global__ void __launch_bounds__(kThreads, 2) near_combine_kernel(const __grid_constant__ NearGroup g) {
    begin_after_previous();
    __shared__ int s_pre[A2A_MAX_WORLD + 1];
    stamp(g.p[0], kStampStart);
    if (PUSH) near_combine_push<T>(g, s_pre);
    else near_combine_pull<T>(g, s_pre);
    stamp(g.p[0], kStampCombineDone);
}

}  // namespace a2a
