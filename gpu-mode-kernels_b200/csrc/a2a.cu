// liba2a.so -- host side of the C ABI declared in include/a2a.h: context life cycle,
// symmetric-region layout, CUDA-IPC peer mapping and kernel launches.  No torch
// types, no allocation and no host synchronisation on the data path.
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <new>

#include "a2a.h"
#include "a2a_kernels.cuh"
#include "a2a_near.cuh"
#include "a2a_pipe.cuh"
#include "a2a_solo.cuh"

using namespace a2a;

namespace {

constexpr int kTraceBlocks = 2048;  // blocks the in-kernel trace buffer has room for
constexpr size_t kMaxSmemBytes = 200 * 1024;  // routing bitmap budget per block (227 KB is the sm_100 limit)
constexpr size_t kMaxPipeSmemBytes = 100 * 1024;  // pipelined kernel of several ranks: two blocks per SM must fit (of 113 KB each)

inline size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

struct Layout {
    size_t off_rows, off_meta, off_counts, off_flags, off_stage, total;
    size_t off_rec_tok, off_rec_ent, off_rec_w, off_hdr, off_ret;  // pipelined schedule only
    int stage_row_bytes;
};

// What every rank of a group must agree on, appended to the IPC handle each rank exports.
struct Fingerprint {
    uint32_t magic;
    int32_t world_size, num_experts, experts_per_token, hidden_dim, max_num_tokens, dtype, payload, schedule, combine,
        chunks;
    uint32_t pad;
    uint64_t layout_total;
};
constexpr uint32_t kFingerprintMagic = 0x41324131u;  // "A2A1"
constexpr size_t kHandleBlobBytes = 128;             // CUDA IPC handle (64) + fingerprint, padded
static_assert(sizeof(cudaIpcMemHandle_t) + sizeof(Fingerprint) <= kHandleBlobBytes, "handle blob too small");

Layout make_layout(const a2a_config& c) {
    Layout l{};
    const size_t L = c.num_experts / c.world_size, ws = c.world_size, T = c.max_num_tokens, H = c.hidden_dim;
    size_t off = 0;
    l.off_rows = off;
    off = align_up(off + L * ws * T * H * 2, 256);
    l.off_meta = off;  // everything from here up to the wire rows starts as zero
    off = align_up(off + L * ws * T * sizeof(int32_t), 256);
    l.off_counts = off;
    off = align_up(off + ws * kMaxChunks * L * sizeof(int32_t), 256);
    l.off_flags = off;
    off = align_up(off + (size_t)kNumFlagKinds * A2A_MAX_WORLD * kFlagStride * sizeof(uint32_t), 256);
    l.stage_row_bytes = 0;
    l.off_stage = off;
    if (c.payload != A2A_PAYLOAD_DIRECT) {
        l.stage_row_bytes = (int)(c.payload == A2A_PAYLOAD_FP8 ? align_up(H + 4 * (H / kFp8Block), 16) : H * 2);
        off = align_up(off + ws * T * (size_t)l.stage_row_bytes, 256);
    }
    l.off_rec_tok = l.off_rec_ent = l.off_rec_w = l.off_hdr = l.off_ret = off;
    if (c.schedule == A2A_SCHEDULE_PIPELINED) {
        const size_t K = c.experts_per_token;
        l.off_rec_tok = off;  off = align_up(off + ws * T * 4, 256);
        l.off_rec_ent = off;  off = align_up(off + ws * T * K * 4, 256);
        l.off_rec_w = off;    off = align_up(off + ws * T * K * 4, 256);
        l.off_hdr = off;      off = align_up(off + ws * 8 * 4, 256);
        l.off_ret = off;
        if (c.combine == A2A_COMBINE_PUSH) off = align_up(off + ws * T * H * 2, 256);
    }
    l.total = off;
    return l;
}

}  // namespace

struct a2a_ctx {
    a2a_config cfg;
    Fingerprint print;      // of cfg
    Layout lay;
    DevParams p;            // template of the kernel parameter block (per-call fields patched at launch)
    uint8_t* region;        // our symmetric region (cudaMalloc)
    uint8_t* scratch;       // local scratch (cudaMalloc)
    size_t scratch_bytes;
    void* ipc_mapped[A2A_MAX_WORLD];  // peers opened through CUDA IPC (to close on destroy)
    bool peers_ready;
    bool routed, sent;
    bool recorded;          // roles 1 and 2 can follow: the call was begun by role 0, or by the one launch of several ranks
    bool near;              // ... by role 0 of a group on this GPU: rows stay where they are
    bool whole;             // ... and role 1 of the group has written the outputs too
    bool listed;            // every pair's place is in p.pairs: role 0 or SEND of the group ran
    bool placed;            // ... SEND: and its row in its slab, whatever the payload
    bool backwards;         // the last launch that wrote the expert rows of the group began with the last tokens
    const void* near_x[A2A_MAX_WORLD];  // input rows of every rank in this call
    const uint2* near_pairs[A2A_MAX_WORLD];
    int near_T[A2A_MAX_WORLD];
    uint32_t epoch, barrier_epoch;
    int cur_tokens;
    int64_t launches;
    unsigned direct_opted_in;  // a bit for each receive-side kernel of the direct payload that may have this context's shared memory
    cudaStream_t side;      // private stream for status reads
    int* host_code;         // mapped host word mirroring the device status code
    // device staging for the host-buffer entry point
    void* h_x;
    int32_t* h_idx;
    float* h_w;
    void* h_y;
    int smem_bytes;         // dynamic shared memory of the routing-carrying kernels
    int num_sms;
    int forward_grid;       // co-resident grid of the one-launch kernel
    int pipe_smem;          // dynamic shared memory of the pipelined kernels
    bool fused;             // a2a_forward uses the one-launch kernel
    bool plain_launch;      // A2A_LAUNCH=plain: ordinary instead of cooperative launch of the one-launch kernels
    char errmsg[160];       // detail of the last host-detected error
    long long* trace;       // device trace buffer (always allocated, used only while tracing is on)
    int last_grid;          // grid of the most recent traced launch
};

namespace {

#define CUDA_TRY(expr)                                   \
    do {                                                 \
        cudaError_t e_ = (expr);                         \
        if (e_ != cudaSuccess) return -(int)e_;          \
    } while (0)

struct DeviceGuard {
    int prev = -1;
    bool changed = false;
    explicit DeviceGuard(int dev) {
        if (cudaGetDevice(&prev) == cudaSuccess && prev != dev) {
            changed = (cudaSetDevice(dev) == cudaSuccess);
        }
    }
    ~DeviceGuard() {
        if (changed) cudaSetDevice(prev);
    }
};

// Token chunks a context really uses: whole 32-token words, at most as many as there are words.
int resolved_chunks(const a2a_config& c) {
    const int Wmax = (c.max_num_tokens + 31) / 32;
    const int chunks = c.chunks >= 1 ? c.chunks : 1;
    return chunks < Wmax ? chunks : Wmax;
}

Fingerprint fingerprint_of(const a2a_config& c) {
    Fingerprint f;
    memset(&f, 0, sizeof(f));
    f.magic = kFingerprintMagic;
    f.world_size = c.world_size; f.num_experts = c.num_experts; f.experts_per_token = c.experts_per_token;
    f.hidden_dim = c.hidden_dim; f.max_num_tokens = c.max_num_tokens; f.dtype = c.dtype;
    f.payload = c.payload; f.schedule = c.schedule; f.combine = c.combine; f.chunks = resolved_chunks(c);
    f.layout_total = make_layout(c).total;
    return f;
}

// The gathered blobs against this rank's configuration; fills msg on a mismatch.
int check_blobs(const a2a_config& cfg, const uint8_t* all, size_t nbytes, char* msg, size_t msg_len) {
    if (msg && msg_len) msg[0] = 0;
    if (nbytes != (size_t)cfg.world_size * kHandleBlobBytes) {
        if (msg) snprintf(msg, msg_len, "handle blobs: got %zu bytes, expected %zu (%d ranks x %zu)", nbytes,
                          (size_t)cfg.world_size * kHandleBlobBytes, cfg.world_size, kHandleBlobBytes);
        return A2A_ERR_CONFIG;
    }
    const Fingerprint mine = fingerprint_of(cfg);
    for (int r = 0; r < cfg.world_size; ++r) {
        Fingerprint f;
        memcpy(&f, all + (size_t)r * kHandleBlobBytes + sizeof(cudaIpcMemHandle_t), sizeof(f));
        if (memcmp(&f, &mine, sizeof(f)) != 0) {
            if (msg) snprintf(msg, msg_len, "rank %d was created with a different configuration than rank %d%s", r,
                              cfg.rank, f.magic != kFingerprintMagic ? " (or its handle blob is damaged)" : "");
            return A2A_ERR_CONFIG;
        }
    }
    return A2A_OK;
}

// Sender blocks of the pipelined kernel.  16-bit payload: one thread per block drives the copy
// engine (two 14 KB loads ahead, four stores in flight).  Measured at 8 GPUs, the sending role alone
// takes 52 us + 624 us / blocks (78 / 65 / 63 / 60 us with 24 / 48 / 64 / 96 blocks) and the whole
// call 126.7 / 113.8 / 110.6 / 109.1 us: 96 blocks at 8 ranks, where there is most to send; 48 below,
// where the call is a chain of latencies and the expert blocks are better served.  FP8: 96, chosen
// when a block quantised a row for each of its destinations; not measured again since it does so once.
int pipe_senders(const a2a_config& c) {
    if (c.world_size == 1) return 0;
    if (c.senders > 0) return c.senders;
    return (c.payload == A2A_PAYLOAD_FP8 || c.world_size >= 8) ? 96 : 48;
}

int validate(const a2a_config& c) {
    if (c.world_size < 1 || c.world_size > A2A_MAX_WORLD) return A2A_ERR_CONFIG;
    if (c.rank < 0 || c.rank >= c.world_size) return A2A_ERR_CONFIG;
    if (c.num_experts < 1 || c.num_experts > A2A_MAX_EXPERTS || c.num_experts % c.world_size != 0) return A2A_ERR_CONFIG;
    if (c.experts_per_token < 1 || c.experts_per_token > A2A_MAX_TOPK || c.experts_per_token > c.num_experts)
        return A2A_ERR_CONFIG;
    if (c.hidden_dim < 8 || c.hidden_dim % 8 != 0) return A2A_ERR_CONFIG;
    if (c.max_num_tokens < 1) return A2A_ERR_CONFIG;
    if (c.dtype != A2A_DTYPE_BF16 && c.dtype != A2A_DTYPE_FP16) return A2A_ERR_CONFIG;
    if (c.payload != A2A_PAYLOAD_DIRECT && c.payload != A2A_PAYLOAD_DEDUP && c.payload != A2A_PAYLOAD_FP8)
        return A2A_ERR_CONFIG;
    if (c.max_num_tokens > 65535) return A2A_ERR_CONFIG;  // slots travel in 16 bits
    if (c.payload == A2A_PAYLOAD_FP8 && c.hidden_dim % kFp8Block != 0) return A2A_ERR_CONFIG;
    if (block_smem_ints(c.num_experts, c.max_num_tokens, c.experts_per_token) * sizeof(int) > kMaxSmemBytes) return A2A_ERR_CONFIG;
    if (c.device < 0) return A2A_ERR_CONFIG;
    if (c.schedule != A2A_SCHEDULE_PHASED && c.schedule != A2A_SCHEDULE_PIPELINED) return A2A_ERR_CONFIG;
    if (c.combine != A2A_COMBINE_PULL && c.combine != A2A_COMBINE_PUSH) return A2A_ERR_CONFIG;
    if (c.chunks < 0 || c.chunks > kMaxChunks || c.senders < 0 || c.senders > 128) return A2A_ERR_CONFIG;
    if (c.combine == A2A_COMBINE_PUSH && c.schedule != A2A_SCHEDULE_PIPELINED) return A2A_ERR_CONFIG;
    if (c.schedule == A2A_SCHEDULE_PIPELINED) {
        // the senders move one wire row per (token, destination): the per-pair DIRECT payload has none
        if (c.payload != A2A_PAYLOAD_DEDUP && c.payload != A2A_PAYLOAD_FP8) return A2A_ERR_CONFIG;
        // FP8: a block assembles a whole wire row in one stage of the sender ring
        if (c.payload == A2A_PAYLOAD_FP8 && make_layout(c).stage_row_bytes > kFp8StageBytes) return A2A_ERR_CONFIG;
        if (c.chunks > 1) return A2A_ERR_CONFIG;
        // one rank has no senders and routes inside its one kernel; only its stepped roles need the tables
        const size_t router_room = c.world_size == 1 ? kMaxSmemBytes : kMaxPipeSmemBytes;
        const int senders = pipe_senders(c);
        if (c.world_size > 1 && senders < 2) return A2A_ERR_CONFIG;  // blocks 0 and 1 carry the watchers
        if ((c.world_size > 1 && pipe_sender_smem(c.max_num_tokens, c.world_size, senders) > kMaxPipeSmemBytes) ||
            pipe_router_smem(c.max_num_tokens, c.num_experts / c.world_size) > router_room)
            return A2A_ERR_CONFIG;
    }
    return A2A_OK;
}

inline cudaStream_t as_stream(void* s) { return reinterpret_cast<cudaStream_t>(s); }

// Rows are moved as 16-byte vectors and by the copy engine: both need 16-byte alignment.
inline bool rows_aligned(const void* ptr) { return reinterpret_cast<uintptr_t>(ptr) % 16 == 0; }

inline int grid_for(const a2a_ctx* c, long long items, int per_sm) {
    long long cap = (long long)c->num_sms * per_sm;
    long long g = items < cap ? items : cap;
    return g < 1 ? 1 : (int)g;
}

DevParams call_params(a2a_ctx* c) {
    DevParams p = c->p;
    p.T = c->cur_tokens;
    p.epoch = c->epoch;
    return p;
}

// ---- kernel selection by (element type, payload) ---------------------------
template <template <typename, int> class F, typename... A>
auto select_tp(const a2a_ctx* c, A... a) {
    const bool bf = c->cfg.dtype == A2A_DTYPE_BF16;
    switch (c->cfg.payload) {
        case A2A_PAYLOAD_DEDUP:
            return bf ? F<__nv_bfloat16, A2A_PAYLOAD_DEDUP>::get(a...) : F<__half, A2A_PAYLOAD_DEDUP>::get(a...);
        case A2A_PAYLOAD_FP8:
            return bf ? F<__nv_bfloat16, A2A_PAYLOAD_FP8>::get(a...) : F<__half, A2A_PAYLOAD_FP8>::get(a...);
        default:
            return bf ? F<__nv_bfloat16, A2A_PAYLOAD_DIRECT>::get(a...) : F<__half, A2A_PAYLOAD_DIRECT>::get(a...);
    }
}

using KernelFn = void (*)(DevParams);
// a phase's kernel for one rank and for a group
struct PhaseFn {
    void (*one)(RankParams);
    void (*group)(GroupParams);
};
template <typename T, int P> struct SendSel {
    static PhaseFn get() { return {send_kernel<T, P, RankParams>, send_kernel<T, P, GroupParams>}; }
};
template <typename T, int P> struct ForwardSel { static KernelFn get() { return forward_kernel<T, P>; } };
template <typename T, int P> struct ExpertSel {
    template <bool WAIT, bool FANOUT, bool SCALE, bool PUBLISH>
    static PhaseFn pair() {
        return {expert_kernel<T, P, WAIT, FANOUT, SCALE, PUBLISH, RankParams>,
                expert_kernel<T, P, WAIT, FANOUT, SCALE, PUBLISH, GroupParams>};
    }
    // the receive-side launches of the public phases
    static PhaseFn get(bool wait, bool fanout, bool scale, bool publish) {
        if (wait && fanout && scale && publish) return pair<true, true, true, true>();      // recv + expert fused
        if (wait && fanout && !scale && !publish) return pair<true, true, false, false>();  // dispatch_recv
        if (!wait && !fanout && scale && publish) return pair<false, false, true, true>();  // expert_placeholder
        return pair<false, false, false, true>();                                           // expert_done
    }
};
// pipelined schedule: (element type, payload, push/pull) -> kernel
template <typename T, int P, bool PUSH> struct PipeForward {
    static PhaseFn get() { return {pipe_forward_kernel<T, P, PUSH, RankParams>, pipe_forward_kernel<T, P, PUSH, GroupParams>}; }
};

template <typename T, int P, bool PUSH> struct PipeRole {
    // what is sent does not depend on the combine, nor the combine on how rows travelled
    template <int PP, bool PUSHP, int ROLE>
    static PhaseFn pair() {
        return {pipe_role_kernel<T, PP, PUSHP, ROLE, RankParams>, pipe_role_kernel<T, PP, PUSHP, ROLE, GroupParams>};
    }
    static PhaseFn get(int role) {
        if (role == 0) return {pipe_role_kernel<T, P, true, 0, RankParams>, nullptr};  // a group's role 0 is a near one
        return role == 1 ? pair<P, PUSH, 1>() : pair<A2A_PAYLOAD_DEDUP, PUSH, 2>();
    }
};
template <template <typename, int, bool> class F, typename T, typename... A>
auto select_pipe_t(const a2a_ctx* c, A... a) {
    const bool push = c->cfg.combine == A2A_COMBINE_PUSH;
    if (c->cfg.payload == A2A_PAYLOAD_FP8)
        return push ? F<T, A2A_PAYLOAD_FP8, true>::get(a...) : F<T, A2A_PAYLOAD_FP8, false>::get(a...);
    return push ? F<T, A2A_PAYLOAD_DEDUP, true>::get(a...) : F<T, A2A_PAYLOAD_DEDUP, false>::get(a...);
}
template <template <typename, int, bool> class F, typename... A>
auto select_pipe(const a2a_ctx* c, A... a) {
    return c->cfg.dtype == A2A_DTYPE_BF16 ? select_pipe_t<F, __nv_bfloat16>(c, a...) : select_pipe_t<F, __half>(c, a...);
}

// the one launch of a pipelined context of world size 1
template <int U>
KernelFn solo_fn(const a2a_ctx* c) {
    const bool bf = c->cfg.dtype == A2A_DTYPE_BF16;
    if (c->cfg.payload == A2A_PAYLOAD_FP8)
        return bf ? solo_kernel<__nv_bfloat16, A2A_PAYLOAD_FP8, U> : solo_kernel<__half, A2A_PAYLOAD_FP8, U>;
    return bf ? solo_kernel<__nv_bfloat16, A2A_PAYLOAD_DEDUP, U> : solo_kernel<__half, A2A_PAYLOAD_DEDUP, U>;
}

// role 1 of ranks on one GPU
template <typename T, int P, int N>
const void* rows_fn(bool push, bool whole, bool narrow) {
    if constexpr (N > 1) {
        if (!whole)
            return push ? (const void*)near_rows_kernel<T, P, true, false, 1, N> : (const void*)near_rows_kernel<T, P, false, false, 1, N>;
        if (push)
            return narrow ? (const void*)near_rows_kernel<T, P, true, true, 1, N> : (const void*)near_rows_kernel<T, P, true, true, 2, N>;
    }
    return narrow ? (const void*)near_rows_kernel<T, P, false, true, 1, N> : (const void*)near_rows_kernel<T, P, false, true, 2, N>;
}

// the kernels of the phases and the combine of ranks on one GPU: element type, U vectors a lane
template <typename T, int U>
const void* near_combine_fn(bool push, bool listed) {
    if (push) return (const void*)near_combine_kernel<T, true, true, U>;
    return listed ? (const void*)near_combine_kernel<T, false, true, U> : (const void*)near_combine_kernel<T, false, false, U>;
}
template <typename T, int U>
const void* near_dispatch_fn(bool fp8) {
    return fp8 ? (const void*)near_dispatch_kernel<T, true, U> : (const void*)near_dispatch_kernel<T, false, U>;
}

PhaseFn combine_fn(const a2a_ctx* c) {
    if (c->cfg.dtype == A2A_DTYPE_BF16) return {combine_kernel<__nv_bfloat16, RankParams>, combine_kernel<__nv_bfloat16, GroupParams>};
    return {combine_kernel<__half, RankParams>, combine_kernel<__half, GroupParams>};
}

// A launch that may get ready while the one before it in the stream ends; its kernel begins with begin_after_previous().
cudaError_t launch_after_previous(const void* fn, int grid, int smem, void** args, cudaStream_t st, int threads = kThreads) {
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t launch{};
    launch.gridDim = dim3(grid);
    launch.blockDim = dim3(threads);
    launch.dynamicSmemBytes = smem;
    launch.stream = st;
    launch.attrs = &attr;
    launch.numAttrs = 1;
    return cudaLaunchKernelExC(&launch, fn, args);
}

int launch(a2a_ctx* c, const void* fn, int grid, int smem, cudaStream_t st, bool cooperative = false) {
    static_assert(sizeof(RankParams) == sizeof(DevParams), "a kernel of one rank takes either");
    DevParams p = call_params(c);
    if (p.trace != nullptr && grid > kTraceBlocks) p.trace = nullptr;
    if (p.trace != nullptr) c->last_grid = grid;
    void* args[] = {&p};
    cudaError_t e = !cooperative ? launch_after_previous(fn, grid, smem, args, st)
        : c->plain_launch ? cudaLaunchKernel(fn, dim3(grid), dim3(kThreads), args, smem, st)
                          : cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(kThreads), args, smem, st);
    c->launches++;
    if (e != cudaSuccess) return -(int)e;
    return A2A_OK;
}

// One phase of the `n` contexts in cs[] as one launch of `blocks` blocks for each.  A trace has a slot per block of
// the grid, so contexts that are being traced are launched one by one.
int launch_ranks(a2a_ctx* const* cs, int n, const PhaseFn& fn, int blocks, int smem, cudaStream_t st) {
    bool traced = false;
    for (int r = 0; r < n; ++r) traced |= cs[r]->p.trace != nullptr;
    if (n == 1 || traced) {
        for (int r = 0; r < n; ++r) {
            const int rc = launch(cs[r], (const void*)fn.one, blocks, smem, st);
            if (rc != A2A_OK) return rc;
        }
        return A2A_OK;
    }
    GroupParams g;
    for (int r = 0; r < n; ++r) {
        g.p[r] = call_params(cs[r]);
        g.p[r].local = 1;
        cs[r]->launches++;
    }
    g.n = n;
    void* args[] = {&g};
    const cudaError_t e = launch_after_previous((const void*)fn.group, n * blocks, smem, args, st);
    return e == cudaSuccess ? A2A_OK : -(int)e;
}

// What a launch for a group on one GPU is told, or for one rank of it in a call that the group began together.
void near_params(a2a_ctx* const* cs, int n, NearGroup& g) {
    for (int r = 0; r < n; ++r) {
        g.p[r] = cs[r]->p;
        g.p[r].T = cs[r]->cur_tokens;
        g.p[r].epoch = cs[r]->epoch;
        g.p[r].local = 1;
        if (n > 1) g.p[r].trace = nullptr;  // a trace has a slot per block of one rank's grid
        g.x[r] = cs[r]->p.x;
        g.pairs[r] = cs[r]->p.pairs;
        g.T[r] = cs[r]->cur_tokens;
    }
    if (n == 1) {
        memcpy(g.x, cs[0]->near_x, sizeof(g.x));
        memcpy(g.pairs, cs[0]->near_pairs, sizeof(g.pairs));
        memcpy(g.T, cs[0]->near_T, sizeof(g.T));
    }
    g.n = n;
    g.every_rank = g.backwards = g.handed_on = 0;
}

// The same of the launches of one call, one after the other with nothing in between: `call` (n 0 before the first) keeps it from one to the
// next.  Of a launch by itself (`call` null): in `own`.
NearGroup& near_call(a2a_ctx* const* cs, int n, NearGroup* call, NearGroup& own) {
    if (call == nullptr) {
        near_params(cs, n, own);
        return own;
    }
    if (call->n == 0) near_params(cs, n, *call);
    call->handed_on = 1;
    return *call;
}

template <int N>
int launch_near(a2a_ctx* const* cs, NearParams<N>& g, const void* fn, int blocks, int smem, cudaStream_t st, int threads = kThreads,
                int arg = 0) {
    if (blocks > kTraceBlocks) g.p[0].trace = nullptr;
    if (g.p[0].trace != nullptr) cs[0]->last_grid = blocks;
    for (int r = 0; r < g.n; ++r) cs[r]->launches++;
    void* args[] = {&g, &arg};
    const cudaError_t e = launch_after_previous(fn, blocks, smem, args, st, threads);
    return e == cudaSuccess ? A2A_OK : -(int)e;
}

// Role 0 of ranks on one GPU.  Tokens a block: 32 (64: eight ranks of 256 tokens of 7168 56.5 for 54.3, two of 200 15.8 / 14.4), or
// 64 and 256 where there are so many that counting the tokens before the block's shows (32 at 5000 tokens of 512, one rank: 13.0 for
// 10.9; 2048 of 7168: 52.0 / 52.3).  Threads: one for each token up to 256 (1024: four ranks of two tokens 6.7 for 6.4, eight of
// 16 10.6 / 9.6, of 256 54.8 / 54.3), else 1024 (256 at two ranks of 1000 tokens of 2048: 18.7 for 17.6; four of 2000 of 512 15.5 / 13.4).
template <int N>
int launch_near_route(a2a_ctx* const* cs, NearParams<N>& g, cudaStream_t st) {
    int most = 1;
    for (int r = 0; r < g.n; ++r) most = cs[r]->cur_tokens > most ? cs[r]->cur_tokens : most;
    const bool few = N > 1 && most <= kThreads;
    const int words = most > 8192 ? 8 : most > 1024 ? 2 : 1, nb = (most + 32 * words - 1) / (32 * words);
    const void* fn = (const void*)near_route_kernel<N, 1024>;
    if constexpr (N > 1)
        if (few) fn = (const void*)near_route_kernel<N, kThreads>;
    return launch_near(cs, g, fn, g.n * nb, (int)near_route_smem(words, cs[0]->cfg.num_experts, cs[0]->cfg.experts_per_token), st,
                       few ? kThreads : 1024, words);
}

// Role 1: a warp per 1 KB of a token's row, three blocks per SM, or per 512 bytes where that would be too few rounds of blocks:
// 2.2 where six or more stores follow each load, one where fewer do.  512 bytes / 1 KB (rounds of the latter): top-8 of 7168,
// 256 tokens, eight ranks 55.8 / 54.4 (8.1), two ranks 17.2 / 17.6 (2.0), 200 tokens 14.4 / 15.1 (1.6); top-6 of 2048, 256 tokens,
// eight ranks 17.8 / 17.6 (2.3); top-2 of 6144, 110 tokens, eight 16.3 / 14.0 (2.9), four 10.6 / 9.8 (1.5), 256, two 10.3 / 9.7 (1.7);
// top-4 of 2880, 110, eight 12.8 / 12.2 (1.5).
template <int N>
int launch_near_rows(a2a_ctx* const* cs, NearParams<N>& g, bool push, bool whole, cudaStream_t st) {
    const a2a_ctx* c = cs[0];
    const long long nvec = c->cfg.hidden_dim / 8, wide = (nvec + 63) / 64, narrow = (nvec + 31) / 32, warps = kThreads / 32;
    long long tokens = 0;
    for (int s = 0; s < c->cfg.world_size; ++s) tokens += g.T[s];
    const bool many = whole && 2 * tokens * wide >= (c->cfg.experts_per_token >= 6 ? 13LL : 6LL) * c->num_sms * warps;
    const long long items = tokens * (many ? wide : narrow), blocks = items > 0 ? (items + warps - 1) / warps : 1;
    const bool bf = c->cfg.dtype == A2A_DTYPE_BF16;
    const void* fn;
    if (c->cfg.payload == A2A_PAYLOAD_FP8)
        fn = bf ? rows_fn<__nv_bfloat16, A2A_PAYLOAD_FP8, N>(push, whole, !many) : rows_fn<__half, A2A_PAYLOAD_FP8, N>(push, whole, !many);
    else
        fn = bf ? rows_fn<__nv_bfloat16, A2A_PAYLOAD_DEDUP, N>(push, whole, !many) : rows_fn<__half, A2A_PAYLOAD_DEDUP, N>(push, whole, !many);
    return launch_near(cs, g, fn, (int)blocks, 0, st);
}

// Blocks of a launch in which each warp has one item, `U` vectors a lane of a token's row.
template <int N>
int near_blocks(const a2a_ctx* c, const NearParams<N>& g, int U) {
    const long long chunks = (c->cfg.hidden_dim / 8 + 32 * U - 1) / (32 * U);
    long long items = 0;
    for (int s = 0; s < c->cfg.world_size; ++s)
        if (g.n > 1 || c->cfg.world_size == 1 || s == c->cfg.rank) items += g.T[s] * chunks;
    const long long blocks = (items + kThreads / 32 - 1) / (kThreads / 32);
    return blocks < 1 ? 1 : (int)blocks;
}

constexpr int kBothFlags = 1 << kFlagDispatch | 1 << kFlagExpert;

// Where the expert rows are more than the L2 keeps, a phase begins with those that the one before it wrote last: eight ranks of 200
// tokens of 7168, top-8 of 256 experts, 183 MB, 129.7 a call by phases, 131.9 without; 128 tokens, 117 MB, 79.8 / 80.9.  Below
// 64 MB no difference.
bool beyond_l2(const a2a_ctx* c, const NearGroup& g) {
    long long tokens = 0;
    for (int s = 0; s < c->cfg.world_size; ++s) tokens += g.T[s];
    return tokens * c->cfg.experts_per_token * c->cfg.hidden_dim * 2 >= 64LL << 20;
}

// The combine: 512 bytes of a token's output a warp, 1 KB where fewer than six rows are added up (a call by
// phases, 512 bytes / 1 KB: four ranks of 200 tokens of 6144, top-2, 25.6 / 25.1; two of 256 of 7168, top-8, 37.7 / 38.7).
int launch_near_combine(a2a_ctx* const* cs, NearGroup& g, bool push, bool listed, cudaStream_t st) {
    g.backwards = !cs[0]->backwards && beyond_l2(cs[0], g);
    const bool bf = cs[0]->cfg.dtype == A2A_DTYPE_BF16, wide = cs[0]->cfg.experts_per_token < 6;
    const void* fn = wide ? (bf ? near_combine_fn<__nv_bfloat16, 2>(push, listed) : near_combine_fn<__half, 2>(push, listed))
                          : (bf ? near_combine_fn<__nv_bfloat16, 1>(push, listed) : near_combine_fn<__half, 1>(push, listed));
    return launch_near(cs, g, fn, near_blocks(cs[0], g, wide ? 2 : 1), 0, st);
}

// RECV, of rows that SEND has put into their slabs, EXPERT and RECV_EXPERT: 512 bytes a warp (1 KB: two ranks of 256 tokens of
// 7168, by phases, 2 % slower when it was tried).
int launch_near_expert(a2a_ctx* const* cs, NearGroup& g, bool wait, bool scale, cudaStream_t st) {
    if (!scale)
        return launch_near(cs, g, (const void*)near_flags_kernel, 1, 0, st, A2A_MAX_WORLD * A2A_MAX_WORLD, 1 << kFlagDispatch);
    g.backwards = beyond_l2(cs[0], g);
    for (int r = 0; r < g.n; ++r) cs[r]->backwards = g.backwards;
    const bool bf = cs[0]->cfg.dtype == A2A_DTYPE_BF16;
    const void* fn = wait ? (bf ? (const void*)near_expert_kernel<__nv_bfloat16, true> : (const void*)near_expert_kernel<__half, true>)
                          : (bf ? (const void*)near_expert_kernel<__nv_bfloat16, false> : (const void*)near_expert_kernel<__half, false>);
    return launch_near(cs, g, fn, near_blocks(cs[0], g, 1), 0, st);
}

// SEND: as many blocks as are resident together, three per SM, each of which counts the experts of the tokens before its own; a
// second round of them costs 3 us (by phases, two ranks of 256 tokens of 2048, 15.3 with three per SM, 18.8 with six).  1 KB a warp
// where every warp has that much, else 512 bytes.
int launch_near_dispatch(a2a_ctx* const* cs, NearGroup& g, cudaStream_t st) {
    const a2a_ctx* c = cs[0];
    int most = 0;
    for (int r = 0; r < g.n; ++r) most = cs[r]->cur_tokens > most ? cs[r]->cur_tokens : most;
    const long long nvec = c->cfg.hidden_dim / 8, warps = kThreads / 32, cap = (long long)c->num_sms * 3 / g.n;
    const long long two = most * ((nvec + 63) / 64), one = most * ((nvec + 31) / 32);
    const bool bf = c->cfg.dtype == A2A_DTYPE_BF16, wide = two >= cap * warps;
    long long blocks = ((wide ? two : one) + warps - 1) / warps;
    if (blocks > cap) blocks = cap;
    if (blocks < 1) blocks = 1;
    const bool fp8 = c->cfg.payload == A2A_PAYLOAD_FP8;
    const void* fn = wide ? (bf ? near_dispatch_fn<__nv_bfloat16, 2>(fp8) : near_dispatch_fn<__half, 2>(fp8))
                          : (bf ? near_dispatch_fn<__nv_bfloat16, 1>(fp8) : near_dispatch_fn<__half, 1>(fp8));
    return launch_near(cs, g, fn, g.n * (int)blocks, 0, st);
}

// The forward of one rank.  A warp's item is one or two 16-byte vectors per lane of a token's row: two
// where that still gives every warp of two blocks per SM an item (headline workload, 256 tokens of 7168:
// 9.1 against 9.6 with one; with four 8 % slower when it was tried), one below that, where
// more warps with less to do each finish sooner (93 tokens of 2880: 4.3 against 4.5; one token of 2048 3.8 either way).  Two
// blocks per SM: with a third that does not fit beside them a second, nearly empty wave of
// blocks starts after the first (headline 12.9).
// Rows in host memory: 74 blocks fill the link, and more only get in each other's way (a call from pinned memory, 3.7 MB read and as
// much written, by 37 / 74 / 148 / 296 blocks: 131.6 / 131 / 138.5 / 149 us).
// Many tokens, or rows that outweigh a second launch: the routing of a group of one and then its rows (a2a_near.cuh).  Not captured,
// us a call back to back, the one launch and the two (MB of expert rows): 40 MB: top-8 of 7168, 400 tokens 12.9 / 12.8 (46), 512
// 15.7 / 15.3 (59), 1000 29.7 / 26.6, 2048 61.6 / 52.6; top-8 of 4096, 512 10.9 / 11.3 (34), 640 13.2 / 12.6 (42), 1279 22.2 / 20.7.
// 800 tokens and 16 MB: top-2 of 6144, 640 9.0 / 8.9 (16), 800 10.3 / 10.0 (20); top-6 of 2048, 640 8.9 / 9.0 (16), 800 9.9 / 9.4 (20);
// top-4 of 2880, 640 8.2 / 8.9 (15), 800 9.7 / 9.2 (18).  Below, the host's two launches, 6.5 to 7, are what a call waits for until the
// counting in every block of the one launch does, 1280 tokens and 4 MB: top-2 of 512, 800 6.6 / 6.5 to 7.0 (2), 2048 10.5 / 7.5 (4);
// of 2048, 800 7.3 / 7.0 (7), 2048 12.2 / 10.2 (17).
bool solo_two_launches(const a2a_ctx* c) {
    const long long mb = (long long)c->cur_tokens * c->cfg.experts_per_token * c->cfg.hidden_dim * 2 >> 20;
    return mb >= 40 || (mb >= 16 && c->cur_tokens >= 800) || (mb >= 4 && c->cur_tokens >= 1280);
}

inline bool overlap(const void* a, size_t na, const void* b, size_t nb) {
    const uintptr_t x = reinterpret_cast<uintptr_t>(a), y = reinterpret_cast<uintptr_t>(b);
    return x < y + nb && y < x + na;
}

int launch_solo(a2a_ctx* c, cudaStream_t st, bool host_rows = false) {
    const long long nvec = c->cfg.hidden_dim / 8, warps = kThreads / 32, cap = host_rows ? c->num_sms / 2 : 2LL * c->num_sms;
    const long long two = c->cur_tokens * ((nvec + 63) / 64), one = c->cur_tokens * ((nvec + 31) / 32);
    // An output laid over the weights or the indices: the one launch reads them block by block while other blocks already write,
    // the routing launch reads them all before the first row is written.
    const size_t tk = (size_t)c->cur_tokens * c->cfg.experts_per_token * 4, rows = (size_t)c->cur_tokens * c->cfg.hidden_dim * 2;
    const bool over = !host_rows && tk > 0 && (overlap(c->p.y, rows, c->p.w, tk) || overlap(c->p.y, rows, c->p.idx, tk));
    if (over || (!host_rows && c->p.trace == nullptr && solo_two_launches(c))) {
        NearParams<1> g = {{call_params(c)}, {c->p.x},         {c->p.pairs},    {c->cur_tokens},
                           /*n=*/1,          /*every_rank=*/0, /*backwards=*/0, /*handed_on=*/1};
        const int rc = launch_near_route(&c, g, st);
        return rc != A2A_OK ? rc : launch_near_rows(&c, g, /*push=*/false, /*whole=*/true, st);
    }
    const bool wide = two >= cap * warps;
    long long blocks = ((wide ? two : one) + warps - 1) / warps;
    if (blocks > cap) blocks = cap;
    if (blocks < 1) blocks = 1;
    return launch(c, (const void*)(wide ? solo_fn<2>(c) : solo_fn<1>(c)), (int)blocks, 0, st);
}

// The device address of host memory that kernels can reach -- pinned, all `bytes` of it in one allocation or
// registration -- or nullptr.
void* mapped_address(const void* host, size_t bytes) {
    using Query = CUresult (*)(unsigned, CUpointer_attribute*, void**, CUdeviceptr);
    static const Query query = [] {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult found;
        const cudaError_t e = cudaGetDriverEntryPointByVersion("cuPointerGetAttributes", &fn, 12000, cudaEnableDefault, &found);
        return reinterpret_cast<Query>(e == cudaSuccess && found == cudaDriverEntryPointSuccess ? fn : nullptr);
    }();
    if (query == nullptr) return nullptr;
    unsigned type = 0;
    CUdeviceptr device = 0, start = 0;
    size_t size = 0;
    // attributes of memory the driver does not know come back as zeros
    CUpointer_attribute what[] = {CU_POINTER_ATTRIBUTE_MEMORY_TYPE, CU_POINTER_ATTRIBUTE_DEVICE_POINTER,
                                  CU_POINTER_ATTRIBUTE_RANGE_START_ADDR, CU_POINTER_ATTRIBUTE_RANGE_SIZE};
    void* into[] = {&type, &device, &start, &size};
    const CUdeviceptr at = reinterpret_cast<CUdeviceptr>(host);
    if (query(4, what, into, at) != CUDA_SUCCESS || type != CU_MEMORYTYPE_HOST || device == 0) return nullptr;
    if (at < start || at + bytes > start + size) return nullptr;
    return reinterpret_cast<void*>(device);
}

int check_call(const a2a_ctx* c, const int32_t* idx, int T) {
    if (!c->peers_ready) return A2A_ERR_STATE;
    if (T < 0 || T > c->cfg.max_num_tokens || (T > 0 && idx == nullptr)) return A2A_ERR_CONFIG;
    if (reinterpret_cast<uintptr_t>(idx) % 4 != 0) return A2A_ERR_CONFIG;
    return A2A_OK;
}

int begin_call(a2a_ctx* c, const int32_t* idx, int T) {
    const int rc = check_call(c, idx, T);
    if (rc != A2A_OK) return rc;
    c->epoch++;
    c->cur_tokens = T;
    c->p.idx = idx;
    c->routed = true;
    c->sent = c->recorded = c->near = c->whole = c->listed = c->placed = c->backwards = false;
    return A2A_OK;
}

int do_route(a2a_ctx* c, const int32_t* idx, int T, cudaStream_t st) {
    int r = begin_call(c, idx, T);
    if (r != A2A_OK) return r;
    return launch(c, (const void*)route_kernel, 1, c->smem_bytes, st);
}

// The phases below take the contexts of all ranks that share this launch: one, or a whole group on one GPU.
// Arguments are checked for every rank before anything is launched.

int most_tokens(a2a_ctx* const* cs, int n) {
    int t = 0;
    for (int r = 0; r < n; ++r) t = cs[r]->cur_tokens > t ? cs[r]->cur_tokens : t;
    return t;
}

// Blocks per rank: the grid that serves `items` of one rank, or this rank's share of the chip.
int grid_for_ranks(const a2a_ctx* c, int n, long long items, int per_sm) {
    const int share = c->num_sms * per_sm / n;
    const int g = grid_for(c, items, per_sm);
    return g < share ? g : (share < 1 ? 1 : share);
}

bool any_traced(a2a_ctx* const* cs, int n) {
    for (int r = 0; r < n; ++r)
        if (cs[r]->p.trace != nullptr) return true;
    return false;
}

// All ranks of a group on one GPU in a launch of a2a_near.cuh?
bool near_phases(a2a_ctx* const* cs, int n) { return n > 1 && cs[0]->p.chunks == 1 && !any_traced(cs, n); }

int do_send(a2a_ctx* const* cs, int n, const void* const* x, cudaStream_t st, NearGroup* call = nullptr) {
    for (int r = 0; r < n; ++r) {
        if (!cs[r]->routed || cs[r]->sent) return A2A_ERR_STATE;
        if (cs[r]->cur_tokens > 0 && x[r] == nullptr) return A2A_ERR_CONFIG;
        if (!rows_aligned(x[r])) return A2A_ERR_CONFIG;
    }
    for (int r = 0; r < n; ++r) cs[r]->p.x = x[r];
    const a2a_ctx* c = cs[0];
    if (near_phases(cs, n)) {
        NearGroup own, &g = near_call(cs, n, call, own);
        const int rc = launch_near_dispatch(cs, g, st);
        if (rc == A2A_OK)
            for (int r = 0; r < n; ++r) cs[r]->sent = cs[r]->listed = cs[r]->placed = true;
        return rc;
    }
    // a warp per 2 KB of a pair's row (DIRECT) or 512 bytes of a token's, no more blocks than four per SM, each of which
    // builds the routing tables
    const bool direct = c->cfg.payload == A2A_PAYLOAD_DIRECT;
    const long long T = most_tokens(cs, n), nvec = c->cfg.hidden_dim / 8, warps = kThreads / 32;
    const long long items = direct ? T * c->cfg.experts_per_token * ((nvec + 127) / 128) : T * ((nvec + 31) / 32);
    const int rc = launch_ranks(cs, n, select_tp<SendSel>(c), grid_for_ranks(c, n, (items + warps - 1) / warps, 4), c->smem_bytes, st);
    if (rc == A2A_OK)
        for (int r = 0; r < n; ++r) cs[r]->sent = true;
    return rc;
}

// grid of the receive-side kernels: a multiple of the world size so every source gets the same share
int expert_grid(const a2a_ctx* c, int n, int per_sm) {
    const int ws = c->cfg.world_size;
    int g = c->num_sms * per_sm / n;
    g = (g / ws) * ws;
    return g < ws ? ws : g;
}

int do_expert(a2a_ctx* const* cs, int n, bool wait, bool fanout, bool scale, bool publish, int grid, cudaStream_t st,
              NearGroup* call = nullptr) {
    bool placed = true;
    for (int r = 0; r < n; ++r) {
        if (!cs[r]->sent) return A2A_ERR_STATE;
        placed = placed && cs[r]->placed;
    }
    if (placed && near_phases(cs, n)) {
        NearGroup own, &g = near_call(cs, n, call, own);
        return launch_near_expert(cs, g, wait, scale, st);
    }
    if (!placed || cs[0]->cfg.payload == A2A_PAYLOAD_DIRECT)
        return launch_ranks(cs, n, select_tp<ExpertSel>(cs[0], wait, fanout, scale, publish), grid, cs[0]->smem_bytes, st);
    // Sent together, received rank by rank: there is nothing in the stages.
    const PhaseFn fn = cs[0]->cfg.dtype == A2A_DTYPE_BF16 ? ExpertSel<__nv_bfloat16, A2A_PAYLOAD_DIRECT>::get(wait, fanout, scale, publish)
                                                          : ExpertSel<__half, A2A_PAYLOAD_DIRECT>::get(wait, fanout, scale, publish);
    const unsigned kernel = 1u << ((wait ? 1 : 0) + (scale ? 2 : 0));
    if ((cs[0]->direct_opted_in & kernel) == 0) {  // a2a_create has opted in for the context's own payload
        CUDA_TRY(cudaFuncSetAttribute((const void*)fn.one, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxSmemBytes));
        cs[0]->direct_opted_in |= kernel;
    }
    for (int r = 0; r < n; ++r) {
        const int rc = launch(cs[r], (const void*)fn.one, grid, cs[r]->smem_bytes, st);
        if (rc != A2A_OK) return rc;
    }
    return A2A_OK;
}

int do_combine(a2a_ctx* const* cs, int n, const float* const* w, void* const* y, cudaStream_t st, NearGroup* call = nullptr) {
    for (int r = 0; r < n; ++r) {
        if (!cs[r]->sent) return A2A_ERR_STATE;
        if (cs[r]->cur_tokens > 0 && (w[r] == nullptr || y[r] == nullptr)) return A2A_ERR_CONFIG;
        if (!rows_aligned(y[r]) || reinterpret_cast<uintptr_t>(w[r]) % 4 != 0) return A2A_ERR_CONFIG;
    }
    for (int r = 0; r < n; ++r) {
        cs[r]->p.w = w[r];
        cs[r]->p.y = y[r];
    }
    const a2a_ctx* c = cs[0];
    bool listed = true;
    for (int r = 0; r < n; ++r) listed = listed && cs[r]->listed;
    if (near_phases(cs, n)) {
        NearGroup own, &g = near_call(cs, n, call, own);
        for (int r = 0; r < n; ++r) {
            g.p[r].w = w[r];
            g.p[r].y = y[r];
        }
        return launch_near_combine(cs, g, /*push=*/false, listed, st);
    }
    const int nseg = (c->cfg.hidden_dim / 8 + 63) / 64;  // a warp per (token, 1 KB segment)
    const long long warps = (long long)most_tokens(cs, n) * nseg;
    return launch_ranks(cs, n, combine_fn(c), grid_for_ranks(c, n, (warps + kThreads / 32 - 1) / (kThreads / 32), 8), 0, st);
}

// The tensors of a pipelined call are checked and the call begun on every rank.
int begin_pipe_call(a2a_ctx* const* cs, int n, const a2a_call* calls) {
    for (int r = 0; r < n; ++r) {
        const a2a_call& k = calls[r];
        const int rc = check_call(cs[r], k.topk_idx, k.num_tokens);
        if (rc != A2A_OK) return rc;
        if (k.num_tokens > 0 && (k.x == nullptr || k.topk_weights == nullptr || k.y == nullptr)) return A2A_ERR_CONFIG;
        if (!rows_aligned(k.x) || !rows_aligned(k.y) || reinterpret_cast<uintptr_t>(k.topk_weights) % 4 != 0) return A2A_ERR_CONFIG;
    }
    for (int r = 0; r < n; ++r) {
        const a2a_call& k = calls[r];
        begin_call(cs[r], k.topk_idx, k.num_tokens);
        cs[r]->p.x = k.x;
        cs[r]->p.w = k.topk_weights;
        cs[r]->p.y = k.y;  // with one rank and the PUSH combine the expert blocks already write the output
    }
    return A2A_OK;
}

// A role of the pipelined schedule for one rank, in the form of a rank whose peers are on other GPUs.
int launch_role(a2a_ctx* c, int role, int blocks, int smem, cudaStream_t st) {
    return launch(c, (const void*)select_pipe<PipeRole>(c, role).one, blocks, smem, st);
}

// Role 0.  Contexts that are being traced are launched one by one, in the forms of a GPU per rank: a trace has a slot
// per block of one rank's grid.  `call`: roles 1 and 2 follow on this stream, with nothing in between.
int do_pipe_send(a2a_ctx* const* cs, int n, const a2a_call* calls, cudaStream_t st, NearGroup* call = nullptr) {
    const int begun = begin_pipe_call(cs, n, calls);
    if (begun != A2A_OK) return begun;
    const a2a_ctx* c = cs[0];
    int rc = A2A_OK;
    if (n == 1 || any_traced(cs, n)) {
        for (int r = 0; r < n && rc == A2A_OK; ++r)
            rc = launch_role(cs[r], 0, c->p.senders + c->cfg.world_size * c->p.routers, c->pipe_smem, st);
    } else {
        for (int r = 0; r < n; ++r)
            for (int s = 0; s < n; ++s) {
                cs[r]->near_x[s] = calls[s].x;
                cs[r]->near_pairs[s] = cs[s]->p.pairs;
                cs[r]->near_T[s] = calls[s].num_tokens;
            }
        NearGroup own, &g = near_call(cs, n, call, own);
        rc = launch_near_route(cs, g, st);
        if (rc == A2A_OK)
            for (int r = 0; r < n; ++r) cs[r]->near = cs[r]->listed = true;
    }
    if (rc == A2A_OK)
        for (int r = 0; r < n; ++r) cs[r]->sent = cs[r]->recorded = true;
    return rc;
}

// Does an output of the call lie over input rows?  Role 1 may then not write outputs while other warps still read rows.
bool outputs_over_rows(const a2a_call* calls, int n, size_t row_bytes) {
    for (int r = 0; r < n; ++r)
        for (int s = 0; s < n; ++s)
            if (overlap(calls[r].y, row_bytes * calls[r].num_tokens, calls[s].x, row_bytes * calls[s].num_tokens)) return true;
    return false;
}

// Roles 1 and 2, of a call whose role 0 ran: the one launch of a single rank writes nothing for them, and what role 1 would
// find there belongs to an earlier call.  A call begun for ranks on one GPU goes on in that form, whoever asks for it.
int do_pipe_rest(a2a_ctx* const* cs, int n, int role, cudaStream_t st, NearGroup* call = nullptr) {
    bool near = true, whole = true;
    for (int r = 0; r < n; ++r) {
        if (!cs[r]->sent || !cs[r]->recorded) return A2A_ERR_STATE;
        near = near && cs[r]->near;
        whole = whole && cs[r]->whole;
    }
    const a2a_ctx* c = cs[0];
    const bool push = c->cfg.combine == A2A_COMBINE_PUSH;
    const int blocks = c->num_sms * 2, push_smem = role == 1 && push ? (int)kReturnSmemBytes : 0;
    if (n > 1 && !any_traced(cs, n)) {
        if (!near)
            // Begun rank by rank: one launch, in which each rank has its share of two blocks per SM.  Role 0 of eight ranks one by
            // one and these two, 4 tokens of 2048 146 us a call (294 with a launch for each rank), 128 of 7168 222 (404).
            return launch_ranks(cs, n, select_pipe<PipeRole>(c, role), blocks / n, push_smem, st);
        NearGroup own, &g = near_call(cs, n, call, own);
        if (role == 1) {
            a2a_call calls[A2A_MAX_WORLD];
            for (int r = 0; r < n; ++r) calls[r] = {g.x[r], nullptr, nullptr, cs[r]->p.y, g.T[r]};
            // PULL: between these roles the expert rows are the caller's
            whole = call != nullptr || (push && !outputs_over_rows(calls, n, (size_t)c->cfg.hidden_dim * 2));
            const int rc = launch_near_rows(cs, g, push, whole, st);
            if (rc == A2A_OK)
                for (int r = 0; r < n; ++r) cs[r]->whole = whole;
            return rc;
        }
        // a role 2 is through when every rank is through with this call, whoever's rows its tokens want
        if (whole) return launch_near(cs, g, (const void*)near_flags_kernel, 1, 0, st, A2A_MAX_WORLD * A2A_MAX_WORLD, kBothFlags);
        g.every_rank = 1;
        return launch_near_combine(cs, g, push, /*listed=*/true, st);
    }
    for (int r = 0; r < n; ++r) {
        int rc;
        if (!cs[r]->near) {
            rc = launch_role(cs[r], role, 1 + blocks, push_smem, st);
        } else if (role == 1) {
            NearGroup g;
            near_params(cs + r, 1, g);
            if (!push) cs[r]->whole = false;  // the expert rows are written anew, and the caller's again
            rc = launch_near_rows(cs + r, g, push, /*whole=*/false, st);
        } else if (cs[r]->whole) {
            NearGroup g;
            near_params(cs + r, 1, g);
            rc = launch_near(cs + r, g, (const void*)near_flags_kernel, 1, 0, st, A2A_MAX_WORLD * A2A_MAX_WORLD, kBothFlags);
        } else {
            NearGroup g;
            near_params(cs + r, 1, g);
            g.every_rank = 1;
            rc = launch_near_combine(cs + r, g, push, /*listed=*/true, st);
        }
        if (rc != A2A_OK) return rc;
    }
    return A2A_OK;
}

// The one launch of all ranks of a group on one GPU, two blocks per SM shared out among them.  Unlike in the
// phases above nothing is shortened for ranks that are near: this is the kernel a GPU per rank runs, and here so
// that one GPU can hold it to the oracle.  The cooperative launch keeps every block running, so no block waits
// for one that is not, and each wait is bounded.  It needs room for the watchers, two senders, and twice the routers.
int do_group_forward(a2a_ctx* const* cs, int n, const a2a_call* calls, cudaStream_t st) {
    const a2a_ctx* c = cs[0];
    const int blocks = 2 * c->num_sms / n, watchers = c->cfg.payload == A2A_PAYLOAD_FP8 ? 2 : 0;
    int routers = blocks / (4 * n) < c->p.routers ? blocks / (4 * n) : c->p.routers;
    if (routers < 1) routers = 1;
    const int room = blocks - watchers - 2 * n * routers;
    const int senders = room < c->p.senders ? room : c->p.senders;
    if (n < 2 || senders < 2) return A2A_ERR_CONFIG;
    const size_t a = pipe_sender_smem(c->cfg.max_num_tokens, n, senders), b = pipe_router_smem(c->cfg.max_num_tokens, c->p.L);
    if (a > kMaxPipeSmemBytes) return A2A_ERR_CONFIG;
    const int begun = begin_pipe_call(cs, n, calls);
    if (begun != A2A_OK) return begun;
    GroupParams g;
    for (int r = 0; r < n; ++r) {
        g.p[r] = call_params(cs[r]);
        g.p[r].senders = senders;
        g.p[r].routers = routers;
        g.p[r].trace = nullptr;  // a trace has a slot per block of one rank's grid
        cs[r]->launches++;
    }
    g.n = n;
    void* args[] = {&g};
    const cudaError_t e = cudaLaunchCooperativeKernel((const void*)select_pipe<PipeForward>(c).group, dim3(n * blocks),
                                                      dim3(kThreads), args, align_up(a > b ? a : b, 128), st);
    if (e != cudaSuccess) return -(int)e;
    for (int r = 0; r < n; ++r) cs[r]->sent = cs[r]->recorded = true;
    return A2A_OK;
}

// The contexts of every rank of one group, all on one GPU, attached to one another and at the same call?  A launch
// for all of them takes every rank's memory for this GPU's own, and none of its blocks watches for a rank that is
// behind.
int check_group(a2a_ctx* const* group) {
    if (group == nullptr || group[0] == nullptr) return A2A_ERR_CONFIG;
    for (int r = 0; r < group[0]->cfg.world_size; ++r) {
        const a2a_ctx* c = group[r];
        if (c == nullptr || c->cfg.rank != r || c->cfg.device != group[0]->cfg.device) return A2A_ERR_CONFIG;
        if (memcmp(&c->print, &group[0]->print, sizeof(c->print)) != 0) return A2A_ERR_CONFIG;
        if (!c->peers_ready || c->epoch != group[0]->epoch) return A2A_ERR_STATE;
    }
    for (int r = 0; r < group[0]->cfg.world_size; ++r)
        for (int s = 0; s < group[0]->cfg.world_size; ++s)
            if (group[r]->p.peer[s] != group[s]->region) return A2A_ERR_CONFIG;
    return A2A_OK;
}

// One phase of all ranks of a group that check_group has passed.
int group_phase(a2a_ctx* const* group, int phase, const a2a_call* calls, cudaStream_t st, NearGroup* call = nullptr) {
    const a2a_ctx* c = group[0];
    const int n = c->cfg.world_size;
    const bool pipe_phase = phase == A2A_GROUP_PIPE_SEND || phase == A2A_GROUP_PIPE_EXPERT || phase == A2A_GROUP_PIPE_COMBINE;
    if (pipe_phase && c->cfg.schedule != A2A_SCHEDULE_PIPELINED) return A2A_ERR_STATE;
    const bool takes_tensors = phase == A2A_GROUP_PIPE_SEND || phase == A2A_GROUP_SEND || phase == A2A_GROUP_COMBINE;
    if (takes_tensors && calls == nullptr) return A2A_ERR_CONFIG;
    const void* x[A2A_MAX_WORLD];
    const float* w[A2A_MAX_WORLD];
    void* y[A2A_MAX_WORLD];
    for (int r = 0; takes_tensors && r < n; ++r) {
        x[r] = calls[r].x;
        w[r] = calls[r].topk_weights;
        y[r] = calls[r].y;
    }
    switch (phase) {
        case A2A_GROUP_PIPE_SEND: return do_pipe_send(group, n, calls, st);
        case A2A_GROUP_PIPE_EXPERT: return do_pipe_rest(group, n, 1, st);
        case A2A_GROUP_PIPE_COMBINE: return do_pipe_rest(group, n, 2, st);
        case A2A_GROUP_SEND:
            for (int r = 0; r < n; ++r) {
                const int rc = check_call(group[r], calls[r].topk_idx, calls[r].num_tokens);
                if (rc != A2A_OK) return rc;
                if (calls[r].num_tokens > 0 && x[r] == nullptr) return A2A_ERR_CONFIG;
                if (!rows_aligned(x[r])) return A2A_ERR_CONFIG;
            }
            for (int r = 0; r < n; ++r) begin_call(group[r], calls[r].topk_idx, calls[r].num_tokens);
            return do_send(group, n, x, st, call);
        case A2A_GROUP_RECV:
            return do_expert(group, n, true, true, false, false,
                             c->cfg.payload == A2A_PAYLOAD_DIRECT ? n : expert_grid(c, n, 4), st, call);
        case A2A_GROUP_EXPERT: return do_expert(group, n, false, false, true, true, expert_grid(c, n, 4), st, call);
        case A2A_GROUP_RECV_EXPERT: return do_expert(group, n, true, true, true, true, expert_grid(c, n, 4), st, call);
        case A2A_GROUP_COMBINE: return do_combine(group, n, w, y, st, call);
        default: return A2A_ERR_CONFIG;
    }
}

// The end of several phases of a group in one call, `last` the last that was launched.  Where they were handed on and a later one was
// refused, or not launched, the flags that it would have raised go up now: the caller may go on phase by phase.
int end_steps(a2a_ctx* const* group, NearGroup& call, int last, int rc, cudaStream_t st) {
    if (rc == A2A_OK || call.n == 0) return rc;
    int owed = 0;
    switch (last) {
        case A2A_GROUP_SEND:
        case A2A_GROUP_PIPE_SEND: owed = 1 << kFlagDispatch; break;
        case A2A_GROUP_EXPERT:
        case A2A_GROUP_RECV_EXPERT: owed = 1 << kFlagExpert; break;
        case A2A_GROUP_PIPE_EXPERT: owed = kBothFlags; break;
        default: break;
    }
    if (owed != 0 && launch_near(group, call, (const void*)near_flags_kernel, 1, 0, st, A2A_MAX_WORLD * A2A_MAX_WORLD, owed) != A2A_OK)
        for (int r = 0; r < call.n; ++r) group[r]->sent = false;  // nothing can follow: later phases are refused and wait for nothing
    return rc;
}

}  // namespace

extern "C" {

const char* a2a_strerror(int status) {
    switch (status) {
        case A2A_OK: return "ok";
        case A2A_ERR_CONFIG: return "invalid configuration or argument";
        case A2A_ERR_CAPACITY: return "slab capacity exceeded (an expert got more than max_num_tokens rows from one source)";
        case A2A_ERR_TIMEOUT: return "a device-side wait on a peer ran out of its time budget";
        case A2A_ERR_STATE: return "call order violated";
        case A2A_ERR_ROUTING: return "expert index out of range";
        default: break;
    }
    if (status < 0) return cudaGetErrorString((cudaError_t)(-status));
    return "unknown status";
}

size_t a2a_ipc_handle_bytes(void) { return kHandleBlobBytes; }

const char* a2a_last_error(a2a_ctx* c) { return c ? c->errmsg : "no context"; }

int a2a_fingerprint(const a2a_config* cfg, uint8_t* out) {
    if (cfg == nullptr || out == nullptr) return A2A_ERR_CONFIG;
    int v = validate(*cfg);
    if (v != A2A_OK) return v;
    memset(out, 0, kHandleBlobBytes - sizeof(cudaIpcMemHandle_t));
    const Fingerprint f = fingerprint_of(*cfg);
    memcpy(out, &f, sizeof(f));
    return A2A_OK;
}

int a2a_check_handles(const a2a_config* cfg, const uint8_t* all, size_t nbytes, char* msg, size_t msg_len) {
    if (cfg == nullptr || all == nullptr) return A2A_ERR_CONFIG;
    return check_blobs(*cfg, all, nbytes, msg, msg_len);
}

int a2a_create(a2a_ctx** out, const a2a_config* cfg) {
    if (out == nullptr || cfg == nullptr) return A2A_ERR_CONFIG;
    *out = nullptr;
    int v = validate(*cfg);
    if (v != A2A_OK) return v;
    int ndev = 0;
    CUDA_TRY(cudaGetDeviceCount(&ndev));
    if (cfg->device >= ndev) return A2A_ERR_CONFIG;
    DeviceGuard guard(cfg->device);

    a2a_ctx* c = new (std::nothrow) a2a_ctx();
    if (c == nullptr) return -(int)cudaErrorMemoryAllocation;
    memset(c, 0, sizeof(*c));
    c->cfg = *cfg;
    if (c->cfg.timeout_ms <= 0) c->cfg.timeout_ms = 2000;
    c->print = fingerprint_of(c->cfg);
    c->lay = make_layout(c->cfg);
    const int E = cfg->num_experts, K = cfg->experts_per_token, T = cfg->max_num_tokens, H = cfg->hidden_dim;
    const int L = E / cfg->world_size;

    cudaError_t e = cudaMalloc(&c->region, c->lay.total);
    if (e != cudaSuccess) { delete c; return -(int)e; }
    // every flag word starts at zero = "epoch 0, nothing has happened" (the staged wire rows need no clearing)
    cudaMemset(c->region + c->lay.off_meta, 0, c->lay.off_stage - c->lay.off_meta);

    // local scratch: slot | send_counts | tickets | seen words | status | trace | host-path staging
    size_t off = 0;
    const size_t o_slot = off;      off = align_up(off + (size_t)T * K * 4, 256);
    const size_t o_pairs = off;     off = align_up(off + (size_t)T * K * sizeof(uint2), 256);
    const size_t o_send = off;      off = align_up(off + (size_t)E * 4, 256);
    const size_t o_tick = off;      off = align_up(off + 8 * 4, 256);
    const size_t o_ptick = off;     off = align_up(off + 2 * A2A_MAX_WORLD * 4, 256);
    const size_t o_seen = off;      off = align_up(off + 2 * A2A_MAX_WORLD * kFlagStride * 4, 256);
    const size_t o_stat = off;      off = align_up(off + sizeof(StatusBlock), 256);
    const size_t o_trace = off;     off = align_up(off + (size_t)kTraceBlocks * kNumStamps * 8, 256);
    const size_t o_hx = off;        off = align_up(off + (size_t)T * H * 2, 256);
    const size_t o_hy = off;        off = align_up(off + (size_t)T * H * 2, 256);
    const size_t o_hidx = off;      off = align_up(off + (size_t)T * K * 4, 256);
    const size_t o_hw = off;        off = align_up(off + (size_t)T * K * 4, 256);
    c->scratch_bytes = off;
    e = cudaMalloc(&c->scratch, off);
    if (e != cudaSuccess) { cudaFree(c->region); delete c; return -(int)e; }
    cudaMemset(c->scratch, 0, off);
    e = cudaStreamCreateWithFlags(&c->side, cudaStreamNonBlocking);
    if (e != cudaSuccess) { cudaFree(c->scratch); cudaFree(c->region); delete c; return -(int)e; }
    e = cudaHostAlloc(reinterpret_cast<void**>(&c->host_code), 64, cudaHostAllocMapped);
    if (e != cudaSuccess) { cudaStreamDestroy(c->side); cudaFree(c->scratch); cudaFree(c->region); delete c; return -(int)e; }
    *c->host_code = 0;
    {
        StatusBlock sb;
        memset(&sb, 0, sizeof(sb));
        sb.host_code = c->host_code;  // unified addressing: the host pointer is valid on the device
        cudaMemcpy(c->scratch + o_stat, &sb, sizeof(sb), cudaMemcpyHostToDevice);
    }

    DevParams& p = c->p;
    p.peer[cfg->rank] = c->region;
    p.off_rows = c->lay.off_rows; p.off_meta = c->lay.off_meta; p.off_counts = c->lay.off_counts;
    p.off_flags = c->lay.off_flags; p.off_stage = c->lay.off_stage;
    p.off_rec_tok = c->lay.off_rec_tok; p.off_rec_ent = c->lay.off_rec_ent; p.off_rec_w = c->lay.off_rec_w;
    p.off_hdr = c->lay.off_hdr; p.off_ret = c->lay.off_ret;
    p.stage_row_bytes = c->lay.stage_row_bytes;
    p.senders = pipe_senders(c->cfg);
    {
        // router blocks per destination: about 32 in all, never more than there are 32-token words
        const int words = (T + 31) / 32;
        int r = 32 / cfg->world_size;
        if (r > 8) r = 8;
        if (r > words) r = words;
        p.routers = r < 1 ? 1 : r;
    }
    p.rank = cfg->rank; p.ws = cfg->world_size; p.E = E; p.K = K; p.H = H; p.T_max = T; p.L = L;
    p.timeout_ns = (long long)c->cfg.timeout_ms * 1000000LL;
    {
        // Token chunks the call is pipelined in (whole 32-token words).  Default 1: measured on
        // B200 the per-chunk publication (a ticket round and a system fence each) costs more than
        // the overlap returns -- c4, DEDUP: 32.7 / 37.5 / 59.3 us with 1 / 2 / 4 chunks on one GPU,
        // 70.7 / 68.1 / 89.3 us on two.  cfg.chunks = 2..4 opts in; every rank of a group must agree
        // (the value is part of the fingerprint the ranks exchange).
        const int Wmax = (T + 31) / 32;
        const int chunks = resolved_chunks(*cfg);
        p.wpc = (Wmax + chunks - 1) / chunks;
        p.chunks = (Wmax + p.wpc - 1) / p.wpc;
    }
    p.slot = reinterpret_cast<int*>(c->scratch + o_slot);
    p.pairs = reinterpret_cast<uint2*>(c->scratch + o_pairs);
    p.send_counts = reinterpret_cast<int*>(c->scratch + o_send);
    p.tickets = reinterpret_cast<uint32_t*>(c->scratch + o_tick);
    p.ptickets = reinterpret_cast<uint32_t*>(c->scratch + o_ptick);
    p.seen = reinterpret_cast<uint32_t*>(c->scratch + o_seen);
    p.status = reinterpret_cast<a2a_status_t*>(c->scratch + o_stat);
    c->trace = reinterpret_cast<long long*>(c->scratch + o_trace);
    c->h_x = c->scratch + o_hx; c->h_y = c->scratch + o_hy;
    c->h_idx = reinterpret_cast<int32_t*>(c->scratch + o_hidx);
    c->h_w = reinterpret_cast<float*>(c->scratch + o_hw);

    // Kernel attributes are per function and device, not per context: opt every routing-carrying
    // kernel in for the whole shared-memory budget, then size this context's own launches.
    c->smem_bytes = (int)(block_smem_ints(E, T, K) * sizeof(int));
    auto opt_in = [&e](const void* fn) {
        if (e == cudaSuccess) e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxSmemBytes);
    };
    auto opt_in_both = [&opt_in](const PhaseFn& fn) {
        opt_in((const void*)fn.one);
        opt_in((const void*)fn.group);
    };
    opt_in((const void*)route_kernel);
    opt_in((const void*)select_tp<ForwardSel>(c));
    opt_in_both(select_tp<SendSel>(c));
    opt_in_both(select_tp<ExpertSel>(c, true, true, true, true));
    opt_in_both(select_tp<ExpertSel>(c, true, true, false, false));
    opt_in_both(select_tp<ExpertSel>(c, false, false, true, true));
    opt_in_both(select_tp<ExpertSel>(c, false, false, false, true));
    int coop = 0, occ = 0;
    const bool pipelined = cfg->schedule == A2A_SCHEDULE_PIPELINED;
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&c->num_sms, cudaDevAttrMultiProcessorCount, cfg->device);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, cfg->device);
    if (pipelined) {
        const size_t a = cfg->world_size > 1 ? pipe_sender_smem(T, cfg->world_size, p.senders) : 0, b = pipe_router_smem(T, L);
        c->pipe_smem = (int)align_up(a > b ? a : b, 128);
        opt_in_both(select_pipe<PipeForward>(c));
        opt_in((const void*)select_pipe<PipeRole>(c, 0).one);
        opt_in((const void*)near_route_kernel<1, 1024>);
        opt_in((const void*)near_route_kernel<A2A_MAX_WORLD, 1024>);
        opt_in((const void*)near_route_kernel<A2A_MAX_WORLD, kThreads>);
        if (e == cudaSuccess && cfg->world_size == 1) {
            c->forward_grid = c->num_sms;
            c->fused = true;  // the solo kernel: no block waits for another
        } else if (e == cudaSuccess) {
            e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, (const void*)select_pipe<PipeForward>(c).one, kThreads, c->pipe_smem);
            if (occ > 2) occ = 2;
            c->forward_grid = c->num_sms * occ;
            c->fused = true;
            // the one launch needs every block resident and room for the roles: senders, one router per
            // destination, and at least as many expert blocks again
            const int watchers = cfg->payload == A2A_PAYLOAD_FP8 ? 2 : 0;
            if (e == cudaSuccess && (coop == 0 || c->forward_grid < watchers + p.senders + 2 * cfg->world_size * p.routers)) {
                a2a_destroy(c);
                return A2A_ERR_CONFIG;
            }
        }
    } else if (e == cudaSuccess) {
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, (const void*)select_tp<ForwardSel>(c), kThreads,
                                                          c->smem_bytes);
        if (e == cudaSuccess) {
            if (occ > 8) occ = 8;
            c->forward_grid = c->num_sms * occ;
            c->fused = (coop != 0 && occ >= 1);
        }
    }
    if (e == cudaSuccess) e = cudaDeviceSynchronize();  // memsets done before any peer may write here
    if (e != cudaSuccess) { a2a_destroy(c); return -(int)e; }
    {
        // Opt-in, for measurement: launch the one-launch kernels like any other kernel.  The grid is sized
        // to be co-resident either way, but only the cooperative launch makes the driver GUARANTEE it; with
        // an ordinary launch a grid that did not get all its blocks running at once ends in
        // A2A_ERR_TIMEOUT (every wait is bounded), not in a hang.
        const char* env = getenv("A2A_LAUNCH");
        c->plain_launch = (env != nullptr && strcmp(env, "plain") == 0);
    }
    c->peers_ready = (cfg->world_size == 1);
    *out = c;
    return A2A_OK;
}

int a2a_destroy(a2a_ctx* c) {
    if (c == nullptr) return A2A_OK;
    DeviceGuard guard(c->cfg.device);
    cudaDeviceSynchronize();
    for (int r = 0; r < A2A_MAX_WORLD; ++r)
        if (c->ipc_mapped[r]) cudaIpcCloseMemHandle(c->ipc_mapped[r]);
    if (c->side) cudaStreamDestroy(c->side);
    if (c->host_code) cudaFreeHost(c->host_code);
    if (c->scratch) cudaFree(c->scratch);
    if (c->region) cudaFree(c->region);
    delete c;
    return A2A_OK;
}

int a2a_export_handle(a2a_ctx* c, uint8_t* out) {
    if (c == nullptr || out == nullptr) return A2A_ERR_CONFIG;
    DeviceGuard guard(c->cfg.device);
    cudaIpcMemHandle_t h;
    CUDA_TRY(cudaIpcGetMemHandle(&h, c->region));
    memset(out, 0, kHandleBlobBytes);
    memcpy(out, &h, sizeof(h));
    const Fingerprint f = fingerprint_of(c->cfg);
    memcpy(out + sizeof(h), &f, sizeof(f));
    return A2A_OK;
}

int a2a_open_peers(a2a_ctx* c, const uint8_t* all, size_t nbytes) {
    if (c == nullptr || all == nullptr) return A2A_ERR_CONFIG;
    if (c->peers_ready && c->cfg.world_size > 1) return A2A_ERR_STATE;
    // every rank must have been created with the same problem, payload and schedule: a rank that
    // differs would lay its region out differently and the peers would write into the wrong places
    const int chk = check_blobs(c->cfg, all, nbytes, c->errmsg, sizeof(c->errmsg));
    if (chk != A2A_OK) return chk;
    DeviceGuard guard(c->cfg.device);
    for (int r = 0; r < c->cfg.world_size; ++r) {
        if (r == c->cfg.rank) continue;
        cudaIpcMemHandle_t h;
        memcpy(&h, all + (size_t)r * kHandleBlobBytes, sizeof(h));
        void* ptr = nullptr;
        CUDA_TRY(cudaIpcOpenMemHandle(&ptr, h, cudaIpcMemLazyEnablePeerAccess));
        c->ipc_mapped[r] = ptr;
        c->p.peer[r] = static_cast<uint8_t*>(ptr);
    }
    c->peers_ready = true;
    return A2A_OK;
}

int a2a_attach_local_peers(a2a_ctx* c, a2a_ctx* const* peers) {
    if (c == nullptr || peers == nullptr) return A2A_ERR_CONFIG;
    DeviceGuard guard(c->cfg.device);
    for (int r = 0; r < c->cfg.world_size; ++r) {
        a2a_ctx* q = peers[r];
        if (q == nullptr || q->cfg.rank != r) return A2A_ERR_CONFIG;
        const Fingerprint a = fingerprint_of(c->cfg), b = fingerprint_of(q->cfg);
        if (memcmp(&a, &b, sizeof(a)) != 0) {
            snprintf(c->errmsg, sizeof(c->errmsg), "rank %d was created with a different configuration than rank %d", r,
                     c->cfg.rank);
            return A2A_ERR_CONFIG;
        }
        if (q->cfg.device != c->cfg.device) {
            cudaError_t e = cudaDeviceEnablePeerAccess(q->cfg.device, 0);
            if (e == cudaErrorPeerAccessAlreadyEnabled) cudaGetLastError();
            else if (e != cudaSuccess) return -(int)e;
        }
        c->p.peer[r] = q->region;
    }
    c->peers_ready = true;
    return A2A_OK;
}

int a2a_route(a2a_ctx* c, const int32_t* idx, int T, void* stream) {
    if (c == nullptr) return A2A_ERR_CONFIG;
    DeviceGuard guard(c->cfg.device);
    return do_route(c, idx, T, as_stream(stream));
}

int a2a_dispatch_send(a2a_ctx* c, const void* x, void* stream) {
    if (c == nullptr) return A2A_ERR_CONFIG;
    DeviceGuard guard(c->cfg.device);
    return do_send(&c, 1, &x, as_stream(stream));
}

int a2a_dispatch_recv(a2a_ctx* c, void* stream) {
    if (c == nullptr) return A2A_ERR_CONFIG;
    DeviceGuard guard(c->cfg.device);
    // DIRECT: the rows are already in place; a minimal grid just waits for every source
    const int grid = c->cfg.payload == A2A_PAYLOAD_DIRECT ? c->cfg.world_size : expert_grid(c, 1, 4);
    return do_expert(&c, 1, true, true, false, false, grid, as_stream(stream));
}

int a2a_expert_placeholder(a2a_ctx* c, void* stream) {
    if (c == nullptr) return A2A_ERR_CONFIG;
    DeviceGuard guard(c->cfg.device);
    return do_expert(&c, 1, false, false, true, true, expert_grid(c, 1, 4), as_stream(stream));
}

int a2a_dispatch_recv_expert(a2a_ctx* c, void* stream) {
    if (c == nullptr) return A2A_ERR_CONFIG;
    DeviceGuard guard(c->cfg.device);
    return do_expert(&c, 1, true, true, true, true, expert_grid(c, 1, 4), as_stream(stream));
}

int a2a_expert_done(a2a_ctx* c, void* stream) {
    if (c == nullptr) return A2A_ERR_CONFIG;
    DeviceGuard guard(c->cfg.device);
    return do_expert(&c, 1, false, false, false, true, expert_grid(c, 1, 1), as_stream(stream));
}

int a2a_combine(a2a_ctx* c, const float* w, void* y, void* stream) {
    if (c == nullptr) return A2A_ERR_CONFIG;
    DeviceGuard guard(c->cfg.device);
    return do_combine(&c, 1, &w, &y, as_stream(stream));
}

int a2a_set_fused(a2a_ctx* c, int on) {
    if (c == nullptr) return A2A_ERR_CONFIG;
    if (on && c->forward_grid < 1) return A2A_ERR_STATE;
    c->fused = (on != 0);
    return A2A_OK;
}

int a2a_forward(a2a_ctx* c, const void* x, const int32_t* idx, const float* w, void* y, int T, void* stream) {
    if (c == nullptr) return A2A_ERR_CONFIG;
    DeviceGuard guard(c->cfg.device);
    cudaStream_t st = as_stream(stream);
    int r = begin_call(c, idx, T);
    if (r != A2A_OK) return r;
    if (T > 0 && (x == nullptr || w == nullptr || y == nullptr)) return A2A_ERR_CONFIG;
    if (!rows_aligned(x) || !rows_aligned(y) || reinterpret_cast<uintptr_t>(w) % 4 != 0) return A2A_ERR_CONFIG;
    if (c->cfg.schedule == A2A_SCHEDULE_PIPELINED) {
        c->p.x = x;
        c->p.w = w;
        c->p.y = y;
        r = c->cfg.world_size == 1
            ? launch_solo(c, st)
            : launch(c, (const void*)select_pipe<PipeForward>(c).one, c->forward_grid, c->pipe_smem, st, /*cooperative=*/true);
        if (r == A2A_OK) {
            c->sent = true;
            c->recorded = c->cfg.world_size > 1;
        }
        return r;
    }
    if (c->fused) {
        c->p.x = x;
        c->p.w = w;
        c->p.y = y;
        r = launch(c, (const void*)select_tp<ForwardSel>(c), c->forward_grid, c->smem_bytes, st, /*cooperative=*/true);
        if (r == A2A_OK) c->sent = true;
        return r;
    }
    r = do_send(&c, 1, &x, st);
    if (r != A2A_OK) return r;
    r = do_expert(&c, 1, true, true, true, true, expert_grid(c, 1, 4), st);
    if (r != A2A_OK) return r;
    return do_combine(&c, 1, &w, &y, st);
}

int a2a_forward_host(a2a_ctx* c, const void* x, const int32_t* idx, const float* w, void* y, int T, void* stream) {
    if (c == nullptr) return A2A_ERR_CONFIG;
    if (T < 0 || T > c->cfg.max_num_tokens) return A2A_ERR_CONFIG;
    if (T > 0 && (x == nullptr || idx == nullptr || w == nullptr || y == nullptr)) return A2A_ERR_CONFIG;
    DeviceGuard guard(c->cfg.device);
    cudaStream_t st = as_stream(stream);
    const size_t row = (size_t)c->cfg.hidden_dim * 2, tk = (size_t)T * c->cfg.experts_per_token * 4;
    if (T > 0 && c->cfg.world_size == 1 && c->cfg.schedule == A2A_SCHEDULE_PIPELINED) {
        // One rank reads every row once and writes every output once: where the kernel can reach the caller's
        // memory it does so itself, and the link carries both directions at the same time instead of one copy
        // after the other (256 tokens of 7168: 128 to 131 us a call; 192 with copies around the kernel).  The indices, which
        // every block reads, are copied.
        void *dx, *dw, *dy;
        if (!overlap(y, row * T, x, row * T) && !overlap(y, row * T, w, tk) && !overlap(y, row * T, idx, tk) &&
            (dx = mapped_address(x, row * T)) != nullptr && (dw = mapped_address(w, tk)) != nullptr &&
            (dy = mapped_address(y, row * T)) != nullptr && rows_aligned(dx) && rows_aligned(dy) &&
            reinterpret_cast<uintptr_t>(dw) % 4 == 0) {
            CUDA_TRY(cudaMemcpyAsync(c->h_idx, idx, tk, cudaMemcpyHostToDevice, st));
            const int r = begin_call(c, c->h_idx, T);
            if (r != A2A_OK) return r;
            c->p.x = dx;
            c->p.w = static_cast<const float*>(dw);
            c->p.y = dy;
            const int rc = launch_solo(c, st, /*host_rows=*/true);
            if (rc == A2A_OK) c->sent = true;
            c->p.x = c->p.y = nullptr;  // the caller's host memory, which may be gone by the next launch
            c->p.w = nullptr;
            return rc;
        }
    }
    if (T > 0) {
        CUDA_TRY(cudaMemcpyAsync(c->h_idx, idx, tk, cudaMemcpyHostToDevice, st));
        CUDA_TRY(cudaMemcpyAsync(c->h_x, x, row * T, cudaMemcpyHostToDevice, st));
        CUDA_TRY(cudaMemcpyAsync(c->h_w, w, tk, cudaMemcpyHostToDevice, st));
    }
    int r = a2a_forward(c, c->h_x, c->h_idx, c->h_w, c->h_y, T, stream);
    if (r != A2A_OK) return r;
    if (T > 0) CUDA_TRY(cudaMemcpyAsync(y, c->h_y, row * T, cudaMemcpyDeviceToHost, st));
    return A2A_OK;
}

int a2a_pipe_step(a2a_ctx* c, int role, const void* x, const int32_t* idx, const float* w, void* y, int T, void* stream) {
    if (c == nullptr || role < 0 || role > 2) return A2A_ERR_CONFIG;
    if (c->cfg.schedule != A2A_SCHEDULE_PIPELINED) return A2A_ERR_STATE;
    DeviceGuard guard(c->cfg.device);
    if (role != 0) return do_pipe_rest(&c, 1, role, as_stream(stream));
    const a2a_call call = {x, idx, w, y, T};
    return do_pipe_send(&c, 1, &call, as_stream(stream));
}

int a2a_group_step(a2a_ctx* const* group, int phase, const a2a_call* calls, void* stream) {
    const int rc = check_group(group);
    if (rc != A2A_OK) return rc;
    DeviceGuard guard(group[0]->cfg.device);
    return group_phase(group, phase, calls, as_stream(stream));
}

int a2a_group_steps(a2a_ctx* const* group, const int32_t* phases, int num_phases, const a2a_call* calls, void* stream, int32_t* done) {
    if (done == nullptr || num_phases < 0 || (num_phases > 0 && phases == nullptr)) return A2A_ERR_CONFIG;
    *done = 0;
    int rc = check_group(group);
    if (rc != A2A_OK) return rc;
    const a2a_ctx* c = group[0];
    const int n = c->cfg.world_size;
    DeviceGuard guard(c->cfg.device);
    cudaStream_t st = as_stream(stream);
    NearGroup call;
    call.n = 0;
    // The roles of a whole call: with nothing between them role 1 writes the outputs of a PULL combine too, and no launch
    // waits for flags of the one before it.
    static const int32_t whole[] = {A2A_GROUP_PIPE_SEND, A2A_GROUP_PIPE_EXPERT, A2A_GROUP_PIPE_COMBINE};
    const bool roles = num_phases == 3 && memcmp(phases, whole, sizeof(whole)) == 0;
    if (roles && n > 1 && calls != nullptr && c->cfg.schedule == A2A_SCHEDULE_PIPELINED && !any_traced(group, n) &&
        !outputs_over_rows(calls, n, (size_t)c->cfg.hidden_dim * 2)) {
        rc = do_pipe_send(group, n, calls, st, &call);
        for (; rc == A2A_OK && ++*done < 3;) rc = do_pipe_rest(group, n, *done, st, &call);
        return *done == 0 ? rc : end_steps(group, call, phases[*done - 1], rc, st);
    }
    static const int32_t four[] = {A2A_GROUP_SEND, A2A_GROUP_RECV, A2A_GROUP_EXPERT, A2A_GROUP_COMBINE};
    static const int32_t three[] = {A2A_GROUP_SEND, A2A_GROUP_RECV_EXPERT, A2A_GROUP_COMBINE};
    const bool handed_on = near_phases(group, n) && ((num_phases == 4 && memcmp(phases, four, sizeof(four)) == 0) ||
                                                     (num_phases == 3 && memcmp(phases, three, sizeof(three)) == 0));
    for (; rc == A2A_OK && *done < num_phases; *done += rc == A2A_OK)
        rc = group_phase(group, phases[*done], calls, st, handed_on ? &call : nullptr);
    return *done == 0 ? rc : end_steps(group, call, phases[*done - 1], rc, st);
}

int a2a_group_forward(a2a_ctx* const* group, const a2a_call* calls, void* stream) {
    const int rc = check_group(group);
    if (rc != A2A_OK) return rc;
    if (calls == nullptr) return A2A_ERR_CONFIG;
    if (group[0]->cfg.schedule != A2A_SCHEDULE_PIPELINED) return A2A_ERR_STATE;
    DeviceGuard guard(group[0]->cfg.device);
    return do_group_forward(group, group[0]->cfg.world_size, calls, as_stream(stream));
}

int a2a_barrier(a2a_ctx* c, void* stream) {
    if (c == nullptr) return A2A_ERR_CONFIG;
    if (!c->peers_ready) return A2A_ERR_STATE;
    DeviceGuard guard(c->cfg.device);
    c->barrier_epoch++;
    barrier_kernel<<<1, 32, 0, as_stream(stream)>>>(call_params(c), c->barrier_epoch);
    c->launches++;
    CUDA_TRY(cudaGetLastError());
    return A2A_OK;
}

int a2a_link_probe(a2a_ctx* c, int peer, size_t bytes, void* stream) {
    if (c == nullptr || peer < 0 || peer >= c->cfg.world_size) return A2A_ERR_CONFIG;
    if (!c->peers_ready) return A2A_ERR_STATE;
    const size_t room = c->lay.off_meta - c->lay.off_rows;  // the slab rows: dead between calls
    if (bytes == 0 || bytes > room) return A2A_ERR_CONFIG;
    DeviceGuard guard(c->cfg.device);
    CUDA_TRY(cudaMemcpyAsync(c->p.peer[peer] + c->lay.off_rows, c->region + c->lay.off_rows, bytes,
                             cudaMemcpyDeviceToDevice, as_stream(stream)));
    return A2A_OK;
}

int a2a_export_dispatch(a2a_ctx* c, int32_t* counts, void* rows, int32_t* meta, void* stream) {
    if (c == nullptr || counts == nullptr || rows == nullptr || meta == nullptr) return A2A_ERR_CONFIG;
    if (!c->sent) return A2A_ERR_STATE;
    DeviceGuard guard(c->cfg.device);
    export_dispatch_kernel<<<c->num_sms * 2, kThreads, 0, as_stream(stream)>>>(call_params(c), counts,
                                                                              static_cast<uint4*>(rows), meta);
    c->launches++;
    CUDA_TRY(cudaGetLastError());
    return A2A_OK;
}

int a2a_expert_buffers(a2a_ctx* c, void** rows, int32_t** counts) {
    if (c == nullptr) return A2A_ERR_CONFIG;
    if (rows) *rows = c->region + c->lay.off_rows;
    if (counts) *counts = reinterpret_cast<int32_t*>(c->region + c->lay.off_counts);
    return A2A_OK;
}

int a2a_route_buffers(a2a_ctx* c, int32_t** slots, int32_t** send_counts) {
    if (c == nullptr) return A2A_ERR_CONFIG;
    if (slots) *slots = c->p.slot;
    if (send_counts) *send_counts = c->p.send_counts;
    return A2A_OK;
}

int a2a_copy_route(a2a_ctx* c, int32_t* slots_out, int32_t* send_counts_out, void* stream) {
    if (c == nullptr) return A2A_ERR_CONFIG;
    if (!c->routed) return A2A_ERR_STATE;
    DeviceGuard guard(c->cfg.device);
    const size_t pairs = (size_t)c->cur_tokens * c->cfg.experts_per_token;
    if (slots_out && pairs)
        CUDA_TRY(cudaMemcpyAsync(slots_out, c->p.slot, pairs * 4, cudaMemcpyDeviceToDevice, as_stream(stream)));
    if (send_counts_out)
        CUDA_TRY(cudaMemcpyAsync(send_counts_out, c->p.send_counts, (size_t)c->cfg.num_experts * 4,
                                 cudaMemcpyDeviceToDevice, as_stream(stream)));
    return A2A_OK;
}

int a2a_trace_enable(a2a_ctx* c, int on) {
    if (c == nullptr) return A2A_ERR_CONFIG;
    DeviceGuard guard(c->cfg.device);
    CUDA_TRY(cudaDeviceSynchronize());
    if (on) CUDA_TRY(cudaMemset(c->trace, 0, (size_t)kTraceBlocks * kNumStamps * 8));
    c->p.trace = on ? c->trace : nullptr;
    return A2A_OK;
}

int a2a_trace_read(a2a_ctx* c, int64_t* out, int max_blocks, int* blocks, int* stamps_per_block) {
    if (c == nullptr || out == nullptr || max_blocks < 0) return A2A_ERR_CONFIG;
    DeviceGuard guard(c->cfg.device);
    CUDA_TRY(cudaDeviceSynchronize());
    int n = c->last_grid < max_blocks ? c->last_grid : max_blocks;
    if (n > 0) CUDA_TRY(cudaMemcpy(out, c->trace, (size_t)n * kNumStamps * 8, cudaMemcpyDeviceToHost));
    if (blocks) *blocks = n;
    if (stamps_per_block) *stamps_per_block = kNumStamps;
    return A2A_OK;
}

int a2a_status(a2a_ctx* c, a2a_status_t* out) {
    if (c == nullptr || out == nullptr) return A2A_ERR_CONFIG;
    DeviceGuard guard(c->cfg.device);
    CUDA_TRY(cudaMemcpyAsync(out, c->p.status, sizeof(*out), cudaMemcpyDeviceToHost, c->side));
    CUDA_TRY(cudaStreamSynchronize(c->side));
    return A2A_OK;
}

int a2a_status_peek(a2a_ctx* c) { return c ? *reinterpret_cast<volatile int*>(c->host_code) : A2A_ERR_CONFIG; }

int a2a_status_clear(a2a_ctx* c) {
    if (c == nullptr) return A2A_ERR_CONFIG;
    DeviceGuard guard(c->cfg.device);
    CUDA_TRY(cudaDeviceSynchronize());
    CUDA_TRY(cudaMemset(c->p.status, 0, sizeof(a2a_status_t)));
    *reinterpret_cast<volatile int*>(c->host_code) = 0;
    CUDA_TRY(cudaMemset(c->p.tickets, 0, 8 * sizeof(uint32_t)));
    CUDA_TRY(cudaMemset(c->p.ptickets, 0, 2 * A2A_MAX_WORLD * sizeof(uint32_t)));
    return A2A_OK;
}

int64_t a2a_launch_count(a2a_ctx* c) { return c ? c->launches : 0; }

size_t a2a_symmetric_bytes(a2a_ctx* c) { return c ? c->lay.total : 0; }

}  // extern "C"
