// The roles of the pipelined schedule for ranks that share ONE GPU: one launch per role serves the whole group
// (a2a_group_step).  Routing, records, slabs, partial rows, flags and epochs are those of a group with a GPU each, and
// so is every bit of the results; what differs is what distance costs and a neighbour does not:
//   * a row is not carried to a stage first.  A peer's input rows lie in this GPU's memory, so the expert blocks
//     read them there, as they read their own rank's in every form; with the FP8 payload each row is quantised
//     once, into the source's own stage, and read from there.  16-bit rows therefore have no senders.
//   * the wire rows of all ranks are one list that all blocks share: a rank whose experts are popular does not
//     keep its own blocks busy while the others' are through.
//   * every flag of the role before is up when a launch starts (it is awaited all the same, bounded, at gpu
//     scope), so no warps poll for it or count what is through: the last block of the grid publishes.
#pragma once

#include "a2a_pipe.cuh"

namespace a2a {

// The ranks a launch serves (`n` of them, all of a group or one) and where the rows of every source rank lie.
struct NearParams {
    DevParams p[A2A_MAX_WORLD];
    const void* x[A2A_MAX_WORLD];  // input rows of rank s in this call
    int T[A2A_MAX_WORLD];          // and how many
    int n;
    int every_rank;  // a PULL combine ends only when every rank's outputs are there, also those no token wants
};

// ---------------------------------------------------------------------------
// Role 0.  FP8: quantiser block `b` of `nb` of a rank.  A warp takes 2 KB of a token's row at a time, like the
// expert blocks, and writes its e4m3 bytes and scales into the rank's own stage, wire row t for token t.
// ---------------------------------------------------------------------------
template <typename T>
__device__ __forceinline__ void quantise_role(const DevParams& p, int b, int nb) {
    const int lane = threadIdx.x & 31, nvec = p.H >> 3, npiece = (nvec + 127) >> 7;
    uint8_t* stage = p.peer[p.rank] + p.off_stage + (size_t)p.rank * p.T_max * p.stage_row_bytes;
    for (int it = b * (kThreads / 32) + (threadIdx.x >> 5); it < p.T * npiece; it += nb * (kThreads / 32)) {
        const int t = it / npiece, v0 = (it - t * npiece) * 128;
        const uint4* src = reinterpret_cast<const uint4*>(p.x) + (size_t)t * nvec;
        uint8_t* wire = stage + (size_t)t * p.stage_row_bytes;
        uint4 q[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int v = v0 + u * 32 + lane;
            if (v < nvec) q[u] = ld_input(src + v);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int v = v0 + u * 32 + lane;  // nvec % 16 == 0: the 16 lanes of a scale block are all in or all out
            float sc;
            const uint2 bytes = quantise8<T>(q[u], v < nvec, sc);
            if (v < nvec) {
                st_stream(reinterpret_cast<uint2*>(wire) + v, bytes);
                if ((v & 15) == 0) reinterpret_cast<float*>(wire + p.H)[v >> 4] = sc;
            }
        }
    }
    __syncthreads();
    if (threadIdx.x < p.ws) arrive_dest(p, threadIdx.x, (uint32_t)(nb + p.routers));
}

// Blocks [0, senders) of a rank quantise (FP8 only), the others route: part rb / ws of destination rank + 1 + rb % ws.
template <typename T, int PAYLOAD>
__global__ void __launch_bounds__(kThreads) near_send_kernel(const __grid_constant__ NearParams g) {
    begin_after_previous();
    const DevParams& p = g.p[blockIdx.x % g.n];
    const int b = (int)blockIdx.x / g.n, ns = p.senders;
    stamp(p, kStampStart);
    if (PAYLOAD == A2A_PAYLOAD_FP8 && b < ns) {
        quantise_role<T>(p, b, ns);
    } else {
        const int rb = b - ns, d = (p.rank + 1 + rb % p.ws) % p.ws;
        router_role(p, a2a_pipe_smem, d, rb / p.ws, p.routers, rb == 0, (uint32_t)(ns + p.routers));
    }
    stamp(p, kStampSent);
}

// ---------------------------------------------------------------------------
// Role 1.  The wire rows of all (source, destination) pairs, one after the other, make one list; a warp's item is 2 KB
// of one of them.  The record of an item is requested two items ahead and its row, whose place only the record
// tells, one item ahead.  Sources come one after the other, so that a source's rows, which every rank reads, stay in
// the L2; rows written for the PUSH combine are not read again soon and leave it first.
// What bounds it: the stores.  Eight ranks of 256 tokens of 7168, top-8 of 256 experts: 87 us for 389 MB (4.5 TB/s;
// a plain fill of as much 66), where blocks bound to a rank that read staged rows took 105 (FP8 rows 80, 128);
// of 2048, top-6 of 64, skewed 23 against 57.  Two vectors a lane at three blocks per SM: 82 to 90 and, FP8, 89 to 94.
// ---------------------------------------------------------------------------
template <typename T, int PAYLOAD, bool PUSH>
__global__ void __launch_bounds__(kThreads, 2) near_expert_kernel(const __grid_constant__ NearParams g) {
    begin_after_previous();
    constexpr int U = 4;
    __shared__ int s_pre[A2A_MAX_WORLD * A2A_MAX_WORLD + 1];
    __shared__ int s_whole;
    const int tid = threadIdx.x, lane = tid & 31;
    const DevParams& p0 = g.p[0];
    const int ws = p0.ws, K = p0.K, T_max = p0.T_max, nvec = p0.H >> 3, pairs = g.n * ws;
    const int nchunk = (nvec + 32 * U - 1) / (32 * U);
    const uint32_t want = flag_value(p0, 0);
    stamp(p0, kStampStart);
    // thread i: wire rows of source i / n at the (i % n)-th rank served
    if (tid < A2A_MAX_WORLD * A2A_MAX_WORLD) {
        int rows = 0;
        if (tid < pairs) {
            const DevParams& p = g.p[tid % g.n];
            const int s = tid / g.n;
            if (wait_flag_gpu(await_ptr(p, kFlagDispatch, s), want, p, kPhaseRecv, s)) {
                rows = ld_stream(reinterpret_cast<const int*>(p.peer[p.rank] + p.off_hdr) + s * 8);
                if (rows < 0 || rows > T_max) {
                    record_error(p.status, A2A_ERR_CAPACITY, p.rank, s, kPhaseExpert, p.epoch, rows);
                    rows = 0;
                }
            }
        }
        __syncwarp();
        int inc = rows;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += v;
        }
        s_pre[tid + 1] = inc;
        if (tid == 0) s_pre[0] = 0;
    }
    __syncthreads();
    if (tid >= 32 && tid < 64) s_pre[tid + 1] += s_pre[32];  // the second warp's sums, after the first's
    __syncthreads();
    const int total = s_pre[pairs];

    struct At {  // chunk ch of wire row `row` of the list; the row is one of pair `at`
        int row, ch, at;
    };
    struct Rec {
        int t;
        unsigned ent;  // lane k: record entry of pair k
        float w;       //         and its weight
    };
    const int xw = (int)blockIdx.x * (kThreads / 32) + (tid >> 5), nxw = (int)gridDim.x * (kThreads / 32);
    const int step_row = nxw / nchunk, step_ch = nxw - step_row * nchunk;
    auto settle = [&](At& a) {
        while (a.row < total && a.row >= s_pre[a.at + 1]) ++a.at;
    };
    auto after = [&](const At& a) {
        At b = {a.row + step_row, a.ch + step_ch, a.at};
        if (b.ch >= nchunk) {
            b.ch -= nchunk;
            ++b.row;
        }
        settle(b);
        return b;
    };
    auto record_of = [&](const At& a, Rec& r) {
        if (a.row >= total) return;
        const int s = a.at / g.n, d = a.at - s * g.n;
        const DevParams& p = g.p[d];
        const uint8_t* self = p.peer[p.rank];
        const size_t rec = (size_t)s * T_max + (a.row - s_pre[a.at]);
        r.t = ld_stream(reinterpret_cast<const int*>(self + p0.off_rec_tok) + rec);
        r.ent = lane < K ? (unsigned)ld_stream(reinterpret_cast<const int*>(self + p0.off_rec_ent) + rec * K + lane) : kNoEntry;
        r.w = (PUSH && lane < K) ? ld_stream(reinterpret_cast<const float*>(self + p0.off_rec_w) + rec * K + lane) : 0.f;
    };
    auto row_of = [&](const At& a, const Rec& r, uint4 (&q)[U]) {
        if (a.row >= total) return;
        const int s = a.at / g.n;
        if (r.t < 0 || r.t >= g.T[s]) return;
        const uint8_t* src = PAYLOAD == A2A_PAYLOAD_FP8
            ? p0.peer[s] + p0.off_stage + ((size_t)s * T_max + r.t) * p0.stage_row_bytes
            : reinterpret_cast<const uint8_t*>(g.x[s]) + (size_t)r.t * p0.H * 2;
        load_wire_chunk<T, PAYLOAD, U>(p0, PAYLOAD != A2A_PAYLOAD_FP8, src, a.ch * 32 * U, nvec, q);
    };
    auto process = [&](const At& a, const Rec& r, const uint4 (&q)[U]) {
        const int s = a.at / g.n, d = a.at - s * g.n, v0 = a.ch * 32 * U + lane;
        const DevParams& p = g.p[d];
        if (r.t < 0 || r.t >= g.T[s]) {
            record_error(p.status, A2A_ERR_CAPACITY, p.rank, s, kPhaseRecv, p.epoch, r.t);
            return;
        }
        int my_row = 0;  // lane k: the slab row of pair k here
        bool here = r.ent != kNoEntry;
        if (here) {
            const int l = (int)(r.ent >> 16), j = (int)(r.ent & 0xffffu);
            my_row = (l * ws + s) * T_max + j;
            if (l >= p0.L || j >= T_max) {
                record_error(p.status, A2A_ERR_CAPACITY, p.rank, s, kPhaseExpert, p.epoch, (int)r.ent);
                here = false;
            }
        }
        const unsigned pairs_here = __ballot_sync(0xffffffffu, here);
        uint4* rows = reinterpret_cast<uint4*>(p.peer[p.rank] + p0.off_rows) + v0;
        const float scale = (float)(1 + p.rank);
        uint4 out[U];
        float acc[U][8];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            out[u] = scale8<T>(wire_vector<T, PAYLOAD>(PAYLOAD != A2A_PAYLOAD_FP8, q[u], v0 + u * 32 < nvec), scale);
#pragma unroll
            for (int e = 0; e < 8; ++e) acc[u][e] = 0.f;
        }
        for (unsigned left = pairs_here; left != 0u; left &= left - 1u) {  // k ascending
            const int k = __ffs(left) - 1;
            uint4* row = rows + (size_t)__shfl_sync(0xffffffffu, my_row, k) * nvec;
            const float w = __shfl_sync(0xffffffffu, r.w, k);
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (v0 + u * 32 < nvec) {
                    if (PUSH) __stcs(row + u * 32, out[u]);
                    else st_stream(row + u * 32, out[u]);
                }
                if (PUSH) {
                    float f[8];
                    unpack8<T>(out[u], f);
                    fma8(f, w, acc[u]);
                }
            }
        }
        if (PUSH) {  // the partial row of this token at this rank, straight into the home rank's buffer
            uint4* home = reinterpret_cast<uint4*>(p0.peer[s] + p0.off_ret) + ((size_t)p.rank * T_max + r.t) * nvec + v0;
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (v0 + u * 32 < nvec) st_stream(home + u * 32, pack8<T>(acc[u]));
        }
    };
    At a0 = {xw / nchunk, xw % nchunk, 0};
    settle(a0);
    At a1 = after(a0);
    Rec r0 = {}, r1 = {};
    uint4 q0[U], q1[U];
    record_of(a0, r0);
    record_of(a1, r1);
    row_of(a0, r0, q0);
    while (a0.row < total) {
        const At a2 = after(a1);
        Rec r2 = {};
        record_of(a2, r2);
        row_of(a1, r1, q1);
        process(a0, r0, q0);
        a0 = a1;
        a1 = a2;
        r0 = r1;
        r1 = r2;
#pragma unroll
        for (int u = 0; u < U; ++u) q0[u] = q1[u];
    }
    // The block that arrives last tells every home rank that the expert outputs and partial rows are there, unless a
    // wait of one of the ranks gave up.  Every block arrives, whatever happened: the ticket is whole for the next call.
    if (grid_arrive_last(p0.ptickets + kPipeTicketSource * A2A_MAX_WORLD, (int)gridDim.x)) {
        if (tid == 0) {
            int whole = 1;
            for (int d = 0; d < g.n; ++d) whole &= ld_volatile_i32(&g.p[d].status->code) != A2A_ERR_TIMEOUT;
            fence_acq_rel_gpu();
            s_whole = whole;
        }
        __syncthreads();
        if (s_whole && tid < pairs) {
            const DevParams& p = g.p[tid / ws];
            const int s = tid % ws;
            if (s == p.rank) st_release_gpu(seen_ptr(p, kFlagExpert, s), want);
            else st_relaxed_sys(flag_ptr(p.peer[s], p.off_flags, kFlagExpert, p.rank), want);
        }
    }
    stamp(p0, kStampExpertDone);
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
__device__ __forceinline__ bool near_tokens(const NearParams& g, int* s_pre, int nchunk, NearTokens& list) {
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
__device__ __forceinline__ void near_combine_push(const NearParams& g, int* s_pre) {
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
__device__ __forceinline__ void near_combine_pull(const NearParams& g, int* s_pre) {
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
__global__ void __launch_bounds__(kThreads, 2) near_combine_kernel(const __grid_constant__ NearParams g) {
    begin_after_previous();
    __shared__ int s_pre[A2A_MAX_WORLD + 1];
    stamp(g.p[0], kStampStart);
    if (PUSH) near_combine_push<T>(g, s_pre);
    else near_combine_pull<T>(g, s_pre);
    stamp(g.p[0], kStampCombineDone);
}

}  // namespace a2a
