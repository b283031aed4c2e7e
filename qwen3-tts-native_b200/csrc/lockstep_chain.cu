// The lockstep chain: the code predictor's part of a frame of 9 to 64 sessions, sixteen positions of five layers with their
// heads and draws, in ONE launch (or, for draws that it does not make, a position each).
//
// Launched one by one a position is 40 dependent kernels of 3.5 to 5 us each, whatever they compute: the weights of a layer
// (15.7 MB) take 2.4 us and its products less.  Here 128 CTAs, 32 clusters of four, stay on their SMs and what is left is the
// hand-overs.  Every projection is the one that gemm_int8_tc.cu makes, with the same K-slices summed in the same order and the
// same epilogues, every norm, attention and draw that of the launches: a frame made here is bit for bit the frame made
// launch by launch.
//
//   rank q of a cluster has a quarter of K for all rows (half of it in gate/up, where a cluster has two tiles)
//     weights        TMA into a ring, converted to bf16 in tensor memory as far ahead as that reaches: six steps of 128 K, more
//                    than most projections have, so that conversion and HBM are behind the hand-overs
//     activations    polled for where they are handed over and copied to shared memory, which they are laid out for
//     products       tcgen05.mma as in gemm_int8_tc.cu (half a cycle a column, 10 at least).  Narrow tiles (64 channels) whose rank
//                    has two of the K-slices put one into the lower and one into the upper half of the lanes, with the rows of both
//                    side by side as columns: one product of twice the columns in place of two that leave 64 lanes idle, as long,
//                    but half the steps of conversion, arrivals and issue
//     K-slices       meet in the cluster by asynchronous stores counted where they land; each rank finishes a share of the rows
//   tiles: q/k/v 32 of 128 channels, one a cluster; gate/up 48 of 64 + 64, two a cluster; o, down and the input projection
//   16 of 64 channels, whose finishing threads keep the residual stream in registers; head 16 of 128.
//   norms: a CTA per row; attention: a warp per (row, KV head), one page of 16 tokens; draws: a CTA per row.
//
// Hand-overs.  A reader polls the values themselves: a word of two bf16 that is no longer the mark (all ones, which no rounding
// yields) has been written.  Each of a piece's four words is looked at, so nothing rests on 16 bytes arriving at once.  No fence, no
// counter, no flag to unpack: with counters and bulk copies a hand-over took 3,700 cycles, so 1,600 to 2,000; with words of six
// values and a number 5,000, most of it unpacking.  Each kind of value has buffers that take turns.  Whoever has published use u of
// a kind marks its own places of use u - 1 again, and fences.
//   Not too early: everybody who reads use u - 1 has read it, since what leads to use u has been through all of them.  Position 0
//   ends at its last q/k/v and position 1 begins with what no reader of it has made; there it is the attention of a ninth row, whose
//   CTAs, clusters 16 and 17, wait for every tile before they take part in position 1's input.  So not for 8 rows and fewer.
//   Not too late: a reader of the next use of the same buffer knows of the mark.  Nothing is fenced between two polls of a layer:
//   writers vouch with the fence at the end of a layer for what they had marked by their barrier before, readers count what they
//   have seen by such a fence and a barrier behind it.  So a buffer comes round only after so many uses that this lies between,
//   also for the clusters that read but every second normed row and none of the head's: 8 buffers of those, 4 of the others, 3
//   where a whole position lies between two uses (turns_of; tests/test_lockstep_protocol.py walks through it).
// The next launch takes the turns up where this one ends.  The marks are the rows' of one row count: another count starts with all
// places marked (restart_lockstep).  The buffers of the K-slices alternate: a CTA may be one projection ahead of its
// neighbours (attention ties rows and heads together, not the whole cluster), never two.
//
// What bounds it (B200, cycles; 23 rows): a layer takes 29,500, of which products 6,000, K-slices' sums 4,500, attention 4,800, norms
// 2,000, and the rest hand-overs with the wait for the slowest CTA.  The predictor's part of a frame by events, launch by launch and
// here (ms): 9 rows 1.92 / 1.40, 16 2.05 / 1.45, 23 2.16 / 1.65, 32 2.21 / 1.71, 40 2.42 / 1.92, 48 2.46 / 1.98, 64 2.70 / 2.17; whole
// frames at contexts of 64 to 512 tokens (us) 9 sessions 3,158 / 2,639, 23 3,572 / 3,071, 64 4,803 / 4,249.  96 registers at launch,
// 8 to 24 bytes spilled.
//
// The launch is cooperative.  Every wait is bounded by a deadline; one that gives up marks the run, all others give up too,
// the kernel runs through on whatever it holds and the host refuses the result.

#include "q3t_attention_page.cuh"
#include "q3t_kernels.cuh"
#include "q3t_sampler.cuh"
#include "q3t_tcgen05.cuh"

#include <cstring>
#include <type_traits>

namespace q3t {
namespace {

using namespace tc;

constexpr int kRanks = 4;                            // of a cluster
constexpr int kClusters = 32;
constexpr int kCtas = kRanks * kClusters;
constexpr int kIoThreads = 256;                      // warps 0..7: activations, K-slices, epilogues, attention
constexpr int kIoWarps = kIoThreads / kWarp;
constexpr int kDequantWarp = 8, kNormWarp = 12, kRoleWarp = 16;     // four warps each
constexpr int kThreads = 640;
// Registers are handed out to groups of four warps: 96 a thread at launch
constexpr int kIoRegisters = 136, kDequantRegisters = 96, kNormRegisters = 64, kRoleRegisters = 48;
static_assert(2 * kIoRegisters + kDequantRegisters + kNormRegisters + kRoleRegisters <= 5 * 96, "registers of the block");
constexpr unsigned long long kBudgetNs = 2000000000ull;

constexpr int H = 1024, I = 3072, Layers = 5, QWidth = 2048, kQkvWidth = 4096, KvHeads = 8, TalkerH = 2048;
constexpr int kBK = 128;
constexpr int kWStageBytes = 128 * kBK;
constexpr int kAccCols = 128, kAStages = 6, kAStageCols = kBK / 2;
static_assert(kAccCols + kAStages * kAStageCols <= 512, "tensor memory");

// ---- exchange: turns_of() buffers a kind.  What one row's reader wants lies row by row, what all rows' readers want as it lies in
// their shared memory: [64 K][rows of the tile][128 bytes, swizzled]
enum Value { vIn, vMid, vQkv, vLogits, vTokens, vNormed, vAtt, vAct, kValues };
__host__ __device__ constexpr int value_bytes(int v) {
    return kMaxRows * (v == vIn || v == vMid || v == vNormed ? H * 2 : v == vQkv ? kQkvWidth * 2 : v == vLogits ? kPredictorVocab * 2
                       : v == vTokens ? 16 : v == vAtt ? QWidth * 2 : I * 2);
}
__host__ __device__ constexpr int turns_of(int v) { return v == vNormed ? 8 : (v == vLogits || v == vTokens ? 3 : 4); }
__host__ __device__ constexpr int at_value(int v) { return v == 0 ? 0 : at_value(v - 1) + turns_of(v - 1) * value_bytes(v - 1); }
constexpr int kAtState = at_value(kValues);           // [0] launches begun, [1] the launch that was given up, then a turn a kind
constexpr int kExchangeBytes = kAtState + 128;
constexpr uint32_t kNoLaunch = ~0u;                  // [1] as long as none was given up: no launch has that number

__device__ unsigned int g_lockstep_errors = 0;
__device__ unsigned int* g_lockstep_error_sink = nullptr;

enum Kind { kMtp, kQkv, kO, kGateUp, kDown, kHead };
__host__ __device__ constexpr bool is_narrow(int kind) { return kind == kO || kind == kDown || kind == kMtp; }
__host__ __device__ constexpr bool is_normed(int kind) { return kind == kQkv || kind == kGateUp || kind == kHead; }

// What a rank does of a projection.  Channels: rows of the weight tile (lanes of the accumulators); Out: results of the
// tile; Parts: K-slices of the operator that a rank has; Sharers: ranks that share a tile.
enum Shape { kNarrow, kWide, kPair };
template <int SHAPE>
struct Of {
    static constexpr int Channels = SHAPE == kNarrow ? 64 : 128;
    static constexpr int Out = SHAPE == kWide ? 128 : 64;
    static constexpr int Parts = SHAPE == kNarrow ? 2 : 1;
    static constexpr int Sharers = SHAPE == kPair ? 2 : 4;
    static constexpr int AllParts = Sharers * Parts;
    static constexpr int StageStride = Out == 64 ? 72 : 136;         // of a row of results, elements: 16-byte pieces, banks apart
};
__device__ __forceinline__ bool takes_part(int kind, int cluster) {
    if (kind == kQkv) return true;
    if (kind == kGateUp) return cluster < 24;
    if (kind == kHead) return cluster < 16;
    return cluster >= 16;
}
__device__ __forceinline__ int tile_of(int kind, int cluster, int rank) {
    if (kind == kGateUp) return 2 * cluster + (rank >> 1);
    return kind == kQkv || kind == kHead ? cluster : cluster - 16;
}
// steps of 128 K, of both K-slices at once where a rank has two
__device__ __forceinline__ int steps_of(int kind) { return kind == kDown ? 3 : (kind == kGateUp ? 4 : 2); }
__device__ __forceinline__ int first_k(int kind, int rank) {
    return kind == kGateUp ? (rank & 1) * 512 : rank * (kind == kDown ? 768 : (is_narrow(kind) ? 512 : 256));
}

struct LockstepArgs {
    const LockstepModel* model;
    const FrameTable* table;
    const int* pages;                // [rows] page of the predictor's cache
    KvLayout kv;                     // offsets of layer 0
    long long kv_layer_elems;
    const uint32_t* rope_table;
    const bf16* codec_embedding;
    const bf16* const* embeddings;
    bf16* logits;                    // [rows][vocabulary]
    unsigned char* exchange;
    int rows, first, last, draws;    // positions; whether their tokens are drawn here
    float eps;
};

struct Barriers {
    uint64_t full_w[6], empty_w[6], full_a[kAStages], empty_a[kAStages];
    uint64_t x_full, acc_done, sums_full[2];
    uint32_t tmem;
    int abort;
};

constexpr int kUnitBytes = 2048 + 16;                // q, q, k, v of a row and head (later the result), the queries in fp32
template <int MT>
struct Layout {
    static constexpr int WStages = MT == 64 ? 3 : (MT == 48 ? 5 : 6);
    static constexpr int XBytes = 12 * MT * 128;                     // 768 K of all rows
    static constexpr int SumBytes = MT * 512;                        // K-slices' parts of the rows finished here
    static constexpr int AtW = XBytes;
    static constexpr int AtSums = AtW + WStages * kWStageBytes;
    static constexpr int AtStage = AtSums + 2 * SumBytes;            // results of a tile, [row][channel]
    static constexpr int AtUnits = AtStage + 32 * 72 * 2;            // attention of the CTA's units
    static constexpr int AtNormRow = AtUnits + 4 * kUnitBytes;
    static constexpr int AtPartial = AtNormRow + H * 2;
    static constexpr int AtBarriers = AtPartial + 256 * 4;
    static constexpr size_t Bytes = 1024 + AtBarriers + sizeof(Barriers);
    static_assert(XBytes % 1024 == 0 && 16 * 136 <= 32 * 72 && Bytes <= 227 * 1024, "fits");
};

__device__ __noinline__ bool lockstep_gives_up(volatile int* abort_flag, uint32_t* run, uint32_t base, unsigned long long deadline) {
    if (*abort_flag != 0) return true;
    uint32_t marked;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(marked) : "l"(run) : "memory");
    if (marked != base && now_ns() <= deadline) return false;
    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(run), "r"(base) : "memory");
    *abort_flag = 1;
    return true;
}
struct Waiter {
    volatile int* abort_flag;
    uint32_t* run;
    uint32_t base;
    unsigned long long deadline;
    __device__ __forceinline__ bool gives_up() const { return lockstep_gives_up(abort_flag, run, base, deadline); }
    __device__ __forceinline__ void wait(uint64_t* bar, uint32_t parity) const {
        uint32_t polls = 0;
        while (!mbar_try_wait(bar, parity)) {
            if ((++polls & 63u) == 0 && gives_up()) return;
        }
    }
};

// (lanes leave a poll one by one: a warp that has not come together counts at a barrier more than once)
__device__ __forceinline__ void io_barrier() {
    __syncwarp();
    asm volatile("bar.sync 1, %0;" ::"n"(kIoThreads) : "memory");
}
__device__ __forceinline__ void norm_barrier() {
    __syncwarp();
    asm volatile("bar.sync 2, 128;" ::: "memory");
}
template <int N>
__device__ __forceinline__ void more_registers() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N>
__device__ __forceinline__ void fewer_registers() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }

__device__ __forceinline__ void put_piece(void* p, const int4& v) {
    asm volatile(
        "{\n\t.reg .b128 t;\n\t.reg .b64 a, b;\n\t"
        "mov.b64 a, {%1, %2};\n\tmov.b64 b, {%3, %4};\n\tmov.b128 t, {a, b};\n\t"
        "st.relaxed.gpu.global.b128 [%0], t;\n\t}"
        ::"l"(p), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w)
        : "memory");
}
__device__ __forceinline__ int4 get_piece(const void* p) {
    int4 v;
    asm volatile(
        "{\n\t.reg .b128 t;\n\t.reg .b64 a, b;\n\t"
        "ld.relaxed.gpu.global.b128 t, [%4];\n\t"
        "mov.b128 {a, b}, t;\n\tmov.b64 {%0, %1}, a;\n\tmov.b64 {%2, %3}, b;\n\t}"
        : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
        : "l"(p)
        : "memory");
    return v;
}
// Pieces of one thread, `apart` bytes from each other: all are asked for again until none of their words is the mark.
// (The largest of all words, in a tree: a comparison for each of them, and a condition for rows that nobody has, took 1.5 to 2.9 % of
// a frame.  With the tree frames of 40 sessions 3,759 -> 3,561 us, of 64 4,331 -> 4,240, of 12 2,668 -> 2,683.)
template <int N>
__device__ __forceinline__ void poll(const unsigned char* at, int apart, int4 (&v)[N], const Waiter& w) {
    for (uint32_t polls = 0;;) {
        uint32_t most[N];
#pragma unroll
        for (int i = 0; i < N; ++i) v[i] = get_piece(at + i * apart);
#pragma unroll
        for (int i = 0; i < N; ++i) most[i] = max(max((uint32_t)v[i].x, (uint32_t)v[i].y), max((uint32_t)v[i].z, (uint32_t)v[i].w));
#pragma unroll
        for (int half = 1; half < N; half *= 2)
#pragma unroll
            for (int i = 0; i + half < N; i += 2 * half) most[i] = max(most[i], most[i + half]);
        if (most[0] != 0xffffffffu) return;
        if ((++polls & 255u) == 0 && w.gives_up()) return;
    }
}
__device__ __forceinline__ int4 mark() { return make_int4(-1, -1, -1, -1); }
// what was marked again is that for everybody before this thread (or those it meets at a barrier) publishes anything more
__device__ __forceinline__ void marks_stand() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }

// Whose turn the buffers are, as a walk through the projections counts it.
struct Turns {
    uint32_t now[kValues];
    __device__ __forceinline__ void read(const uint32_t* state) {
#pragma unroll
        for (int v = 0; v < kValues; ++v) now[v] = __ldcg(state + 2 + v);
    }
    template <Value V> __device__ __forceinline__ void next() { now[V] = now[V] == turns_of(V) - 1 ? 0 : now[V] + 1; }
    template <Value V> __device__ __forceinline__ int at() const { return at_value(V) + (int)now[V] * value_bytes(V); }
    template <Value V> __device__ __forceinline__ int before() const { return at_value(V) + (int)(now[V] == 0 ? turns_of(V) - 1 : now[V] - 1) * value_bytes(V); }
};

// where 16 bytes (8 channels from k of a row) lie in a slice of MT rows
template <int MT>
__device__ __forceinline__ int piece_at(int row, int k) {
    return (k >> 6) * (MT * 128) + row * 128 + ((((k >> 3) & 7) ^ (row & 7)) << 4);
}

// calls f(kind, layer, position) for every projection of the launch, in order
template <class F>
__device__ __forceinline__ void projections(const LockstepArgs& a, F f) {
#pragma unroll 1
    for (int p = a.first; p <= a.last; ++p) {
        const int stages = p == 0 ? 2 + 4 * (Layers - 1) : 2 + 4 * Layers;     // nobody reads position 0's hidden row
#pragma unroll 1
        for (int i = 0; i < stages; ++i) {
            const int kind = i == 0 ? static_cast<int>(kMtp) : (i == 1 + 4 * Layers ? static_cast<int>(kHead) : 1 + (i - 1) % 4);
            f(kind, (i - 1) / 4, p);
        }
    }
}
static_assert(kMtp == 0 && kQkv == 1 && kO == 2 && kGateUp == 3 && kDown == 4 && kHead == 5, "order of a position");

// fp32 accumulators, A and B bf16, K-major, 128 lanes
__device__ __forceinline__ constexpr uint32_t instruction(int columns) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(columns >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
}

template <int MT>
__global__ void __launch_bounds__(kThreads, 1) lockstep_chain_kernel(const LockstepArgs a) {
    using L = Layout<MT>;
    constexpr int kXAtom = MT * 128;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    unsigned char* xs = smem;
    unsigned char* w8 = smem + L::AtW;
    bf16* stage = reinterpret_cast<bf16*>(smem + L::AtStage);
    Barriers& b = *reinterpret_cast<Barriers*>(smem + L::AtBarriers);
    const int tid = threadIdx.x;
    const int warp = __shfl_sync(0xffffffffu, tid / kWarp, 0);
    const int lane = tid % kWarp;
    const int rank = (int)cluster_rank();
    const int cluster = blockIdx.x / kRanks;
    const int cta = blockIdx.x;
    const int rows = a.rows;
    const LockstepModel& m = *a.model;

    Waiter wt;
    wt.abort_flag = &b.abort;
    uint32_t* const state = reinterpret_cast<uint32_t*>(a.exchange + kAtState);
    wt.run = state + 1;
    wt.base = __ldcg(state);
    wt.deadline = now_ns() + kBudgetNs;
    unsigned char* const ex = a.exchange;

    if (tid == 0) {
        for (int s = 0; s < 6; ++s) {
            mbar_init(&b.full_w[s], 1);
            mbar_init(&b.empty_w[s], 4);
        }
        for (int s = 0; s < kAStages; ++s) {
            mbar_init(&b.full_a[s], 4);
            mbar_init(&b.empty_a[s], 1);
        }
        mbar_init(&b.x_full, kIoWarps);
        mbar_init(&b.acc_done, 1);
        mbar_init(&b.sums_full[0], 1);
        mbar_init(&b.sums_full[1], 1);
        b.abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == kRoleWarp + 2) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&b.tmem)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    cluster_sync();                                                  // barriers of all four are set up
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = b.tmem;

    if (warp >= kRoleWarp) {
        fewer_registers<kRoleRegisters>();
        if (warp == kRoleWarp) {
            if (elect_one()) {
                // ---- weight producer
                int t = 0;
                projections(a, [&](int kind, int layer, int p) {
                    if (!takes_part(kind, cluster)) return;
                    const int map = kind == kMtp ? kLockstepMtpMap : (kind == kHead ? kLockstepHeadMap + p - 1
                                    : 4 * layer + (kind == kQkv ? 0 : (kind == kO ? 1 : (kind == kGateUp ? 2 : 3))));
                    const CUtensorMap* w_map = reinterpret_cast<const CUtensorMap*>(m.maps[map]);
                    const int tile = tile_of(kind, cluster, rank), k0 = first_k(kind, rank), steps = steps_of(kind);
                    const bool narrow = is_narrow(kind);
                    for (int i = 0; i < steps; ++i, ++t) {
                        const int s = t % L::WStages;
                        if (t >= L::WStages) wt.wait(&b.empty_w[s], ((t / L::WStages) - 1) & 1);
                        if (b.abort != 0) return;
                        unsigned char* dst = w8 + s * kWStageBytes;
                        mbar_expect_tx(&b.full_w[s], kWStageBytes);
                        if (kind == kGateUp) {
                            tma_load_2d(dst, w_map, k0 + i * kBK, tile * 64, &b.full_w[s]);
                            tma_load_2d(dst + kWStageBytes / 2, w_map, k0 + i * kBK, I + tile * 64, &b.full_w[s]);
                        } else if (narrow) {                         // a step of either K-slice
                            tma_load_2d(dst, w_map, k0 + i * kBK, tile * 64, &b.full_w[s]);
                            tma_load_2d(dst + kWStageBytes / 2, w_map, k0 + (steps + i) * kBK, tile * 64, &b.full_w[s]);
                        } else {
                            tma_load_2d(dst, w_map, k0 + i * kBK, tile * 128, &b.full_w[s]);
                        }
                    }
                });
            }
        } else if (warp == kRoleWarp + 1) {
            if (elect_one()) {
                // ---- MMA issuer
                int t = 0, turn = 0;
                const uint64_t x_desc = umma_desc(smem_u32(xs));
                projections(a, [&](int kind, int, int) {
                    if (!takes_part(kind, cluster)) return;
                    const int steps = steps_of(kind);
                    // columns: the rows, or those of two K-slices side by side
                    const uint32_t idesc = is_narrow(kind) ? instruction(2 * MT) : instruction(MT);
                    const uint64_t atom = is_narrow(kind) ? 2 * kXAtom / 16 : kXAtom / 16;
                    wt.wait(&b.x_full, turn & 1);
                    ++turn;
                    uint64_t desc = x_desc;
#pragma unroll 1
                    for (int i = 0; i < steps; ++i, ++t) {
                        const int sa = t % kAStages;
                        wt.wait(&b.full_a[sa], (t / kAStages) & 1);
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        const uint32_t a_col = tmem + kAccCols + sa * kAStageCols;
#pragma unroll
                        for (int j = 0; j < kBK / 16; ++j) {
                            umma_f16_ts(tmem, a_col + 8 * j, desc + (uint64_t)(2 * (j % 4)), idesc, (i | j) != 0 ? 1u : 0u);
                            if (j % 4 == 3) desc += atom;
                        }
                        umma_commit(&b.empty_a[sa]);
                    }
                    umma_commit(&b.acc_done);
                });
            }
        }
    } else if (warp >= kNormWarp) {
        // ---- norms: the row of this CTA, if it has one
        fewer_registers<kNormRegisters>();
        const int row = cta / 2;
        if (cta % 2 == 0 && row < rows) {
            const int n = tid - kNormWarp * kWarp;                   // eight channels each
            bf16* values = reinterpret_cast<bf16*>(smem + L::AtNormRow);
            float* partial = reinterpret_cast<float*>(smem + L::AtPartial);
            const int to = piece_at<MT>(row, 8 * n);
            Turns turns;
            turns.read(state);
            projections(a, [&](int kind, int layer, int) {
                if (is_normed(kind)) {
                    const bf16* norm_w = kind == kHead ? m.final_norm : (kind == kQkv ? m.layers[layer].in_norm : m.layers[layer].post_norm);
                    const int4 nw = __ldg(reinterpret_cast<const int4*>(norm_w) + n);
                    int4 mine[1];
                    poll<1>(ex + (kind == kGateUp ? turns.at<vMid>() : turns.at<vIn>()) + row * (H * 2) + n * 16, 0, mine, wt);
                    reinterpret_cast<int4*>(values)[n] = mine[0];
                    norm_barrier();
                    // talker_kernels.cu:27-48: strided sums of 256 threads, then their tree
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        float ss = 0.0f;
#pragma unroll
                        for (int e = 0; e < H / 256; ++e) {
                            const float x = bf2f(values[n + 128 * u + 256 * e]);
                            ss = fmaf(x, x, ss);
                        }
                        partial[n + 128 * u] = ss;
                    }
                    norm_barrier();
                    const float inv = rsqrtf(tree_sum_256(partial, lane) / static_cast<float>(H) + a.eps);
                    auto scaled = [inv](int x, int w) {
                        return static_cast<int>(page::pack_bf16x2(rbf(bf_lo((uint32_t)x) * inv) * bf_lo((uint32_t)w), rbf(bf_hi((uint32_t)x) * inv) * bf_hi((uint32_t)w)));
                    };
                    put_piece(ex + turns.at<vNormed>() + to, make_int4(scaled(mine[0].x, nw.x), scaled(mine[0].y, nw.y), scaled(mine[0].z, nw.z), scaled(mine[0].w, nw.w)));
                    put_piece(ex + turns.before<vNormed>() + to, mark());
                    marks_stand();
                    turns.next<vNormed>();
                }
                // an input and a mid row have been read by now
                if (kind == kQkv || kind == kHead) turns.next<vIn>();
                if (kind == kGateUp) turns.next<vMid>();
            });
        }
    } else if (warp >= kDequantWarp) {
        // ---- dequantisers: a thread a channel
        fewer_registers<kDequantRegisters>();
        const int c = (warp % 4) * 32 + lane;
        const uint32_t lane_base = tmem + ((uint32_t)((warp % 4) * 32) << 16) + kAccCols;
        int t = 0;
        projections(a, [&](int kind, int, int) {
            if (!takes_part(kind, cluster)) return;
            const int steps = steps_of(kind);
#pragma unroll 1
            for (int i = 0; i < steps; ++i, ++t) {
                const int s = t % L::WStages, sa = t % kAStages;
                wt.wait(&b.full_w[s], (t / L::WStages) & 1);
                const unsigned char* rowp = w8 + s * kWStageBytes + c * 128;
                if (t >= kAStages) wt.wait(&b.empty_a[sa], ((t / kAStages) - 1) & 1);
                __syncwarp();
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    uint32_t out[32];
#pragma unroll
                    for (int p = 0; p < 4; ++p) {
                        const int4 v = *reinterpret_cast<const int4*>(rowp + (((4 * h + p) ^ (c & 7)) << 4));
                        dequant4(static_cast<uint32_t>(v.x), out[8 * p + 0], out[8 * p + 1]);
                        dequant4(static_cast<uint32_t>(v.y), out[8 * p + 2], out[8 * p + 3]);
                        dequant4(static_cast<uint32_t>(v.z), out[8 * p + 4], out[8 * p + 5]);
                        dequant4(static_cast<uint32_t>(v.w), out[8 * p + 6], out[8 * p + 7]);
                    }
                    tmem_store_32(lane_base + sa * kAStageCols + 32 * h, out);
                }
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(&b.full_a[sa]);
                    mbar_arrive(&b.empty_w[s]);
                }
            }
        });
    } else {
        // ---- activations in, K-slices together, results out; attention
        more_registers<kIoRegisters>();
        int turn = 0;
        float own[4] = {0.0f, 0.0f, 0.0f, 0.0f};       // the residual stream where this thread finishes it
        Turns turns;
        turns.read(state);
        // where eight channels of a row that a projection publishes lie
        auto place = [&](auto which, int kind, int row, int channel) {
            if (decltype(which)::value == kPair) return piece_at<MT>(row, channel);
            return (row * (decltype(which)::value == kNarrow ? H : (kind == kHead ? kPredictorVocab : kQkvWidth)) + channel) * 2;
        };
        // the input of a position: embeddings of the tokens before, into the slice that this rank multiplies; a warp every
        // eighth row, whose tokens its first lanes look up
        auto bring_embeddings = [&](int p) {
            const bf16* mine = nullptr;
            const int my_row = warp + kIoWarps * lane;
            if (lane < kMaxRows / kIoWarps && my_row < rows) {
                if (p == 0) {
                    mine = a.table->last_hidden[my_row];
                } else {
                    int token;
                    if (a.draws == 0 || p == 1) {
                        token = a.table->frame_tokens[my_row][p - 1];
                    } else {
                        int4 v[1];
                        poll<1>(ex + turns.before<vTokens>() + my_row * 16, 0, v, wt);
                        token = v[0].x;
                    }
                    if (token >= 0 && token < (p == 1 ? kMaxVocab : kPredictorVocab)) {
                        mine = (p == 1 ? a.codec_embedding : a.embeddings[p - 2]) + (size_t)token * TalkerH;
                    }
                }
            }
            __syncwarp();
            const int k0 = first_k(kMtp, rank);
#pragma unroll 4
            for (int i = 0; i < MT / kIoWarps; ++i) {
                const bf16* src = reinterpret_cast<const bf16*>(__shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(mine), i));
                const int row = warp + kIoWarps * i;
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const int k = 8 * (lane + 32 * u), atom = k >> 6;
                    const int4 v = src != nullptr ? __ldcg(reinterpret_cast<const int4*>(src + k0 + k)) : make_int4(0, 0, 0, 0);
                    *reinterpret_cast<int4*>(xs + (atom < 4 ? 2 * atom : 2 * atom - 7) * kXAtom + piece_at<MT>(row, k & 63)) = v;
                }
            }
        };
        // a rank's slice of all rows' activations, PIECES of 16 bytes a thread
        auto bring_in = [&](auto pieces, const unsigned char* src, bool narrow) {
            constexpr int PIECES = decltype(pieces)::value, kBatch = PIECES % 8 == 0 ? 8 : (PIECES % 6 == 0 ? 6 : (PIECES % 4 == 0 ? 4 : 2));
            constexpr int kAtoms = PIECES * 32 / MT;
#pragma unroll 1
            for (int u0 = 0; u0 < PIECES; u0 += kBatch) {
                int4 v[kBatch];
                poll<kBatch>(src + (tid + kIoThreads * u0) * 16, kIoThreads * 16, v, wt);
#pragma unroll
                for (int u = 0; u < kBatch; ++u) {
                    const int i = tid + kIoThreads * (u0 + u), atom = i / (8 * MT);
                    // two K-slices: the rows of the second behind those of the first
                    const int to = narrow ? (atom < kAtoms / 2 ? 2 * atom : 2 * atom - kAtoms + 1) : atom;
                    *reinterpret_cast<int4*>(xs + to * kXAtom + (i - atom * (8 * MT)) * 16) = v[u];
                }
            }
        };
        auto project = [&](auto which, int kind, int layer, int p) {
            using K = Of<decltype(which)::value>;
            constexpr int SHAPE = decltype(which)::value;
            if (!takes_part(kind, cluster)) return;
            const ChainLayer& lc = m.layers[kind == kMtp || kind == kHead ? 0 : layer];
            const int tile = tile_of(kind, cluster, rank);
            constexpr int Share = MT / K::Sharers;                   // rows that a rank finishes
            const int sharer = SHAPE == kPair ? rank & 1 : rank;
            const int row0 = sharer * Share;
            const int my_rows = max(0, min(Share, rows - row0));
            const int groups = (my_rows + 3) / 4;
            const uint32_t parity = turn & 1, use = turn >> 1;
            float* sums = reinterpret_cast<float*>(smem + L::AtSums + parity * L::SumBytes);
            if (tid == 0) mbar_expect_tx(&b.sums_full[parity], (uint32_t)((K::Sharers - 1) * K::Parts * groups * K::Channels * 16));
            // what the epilogue needs, asked for ahead of the waits
            const int c = tid % K::Out;
            const int channel = tile * K::Out + c;
            const float* scales = SHAPE == kPair ? lc.gu_s : SHAPE == kWide ? (kind == kHead ? m.head_scales[p - 1] : lc.qkv_s)
                                  : (kind == kMtp ? m.mtp_scales : kind == kO ? lc.o_s : lc.down_s);
            const float scale = scales[channel];
            const float scale_up = SHAPE == kPair ? scales[I + channel] : 0.0f;
            const float bias = SHAPE == kNarrow && kind == kMtp ? bf2f(m.mtp_bias[channel]) : 0.0f;

            // ---- activations
            if (kind == kMtp) {
                bring_embeddings(p);
            } else {
                const unsigned char* src = ex + (SHAPE != kNarrow ? turns.at<vNormed>() : (kind == kO ? turns.at<vAtt>() : turns.at<vAct>())) + first_k(kind, rank) / 64 * kXAtom;
                if (SHAPE == kWide) bring_in(std::integral_constant<int, MT / 8>(), src, false);
                else if (SHAPE == kPair) bring_in(std::integral_constant<int, MT / 4>(), src, false);
                else if (kind == kO) bring_in(std::integral_constant<int, MT / 4>(), src, true);
                else bring_in(std::integral_constant<int, 3 * MT / 8>(), src, true);
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&b.x_full);

            // ---- accumulators to the ranks that finish their rows
            wt.wait(&b.acc_done, parity);
            __syncwarp();
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            {
                // lanes by quarters, columns by halves; a narrow tile's second K-slice has the upper lanes and columns
                const int quarter = warp & 3, half = warp >> 2;
                constexpr int kCols = MT / 2;
                constexpr int kChunk = kCols % 16 == 0 ? 16 : 8;
                const int col0 = half * kCols;
                const int slice = SHAPE == kNarrow ? quarter >> 1 : 0;
                const int part = sharer * K::Parts + slice;
                const uint32_t from = tmem + ((uint32_t)(quarter * 32) << 16) + slice * MT + col0;
                const int mine = (SHAPE == kNarrow ? quarter & 1 : quarter) * 32 + lane;
                const uint32_t to = smem_u32(sums) + (uint32_t)((part * (Share / 4) * K::Channels + mine) * 16);
#pragma unroll 1
                for (int j0 = 0; j0 < kCols; j0 += kChunk) {
                    if (col0 + j0 >= rows) break;
                    float v[kChunk];
                    tmem_load_row<kChunk>(from + j0, v);
#pragma unroll
                    for (int j = 0; j < kChunk; j += 4) {
                        const int r = col0 + j0 + j;
                        if (r >= rows) break;
                        const int owner = r / Share, within = (r - owner * Share) / 4;
                        const uint32_t at = to + (uint32_t)(within * K::Channels * 16);
                        if (owner == sharer) {
                            asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(at), "f"(v[j]), "f"(v[j + 1]), "f"(v[j + 2]), "f"(v[j + 3]) : "memory");
                        } else {
                            const uint32_t peer = SHAPE == kPair ? (uint32_t)((rank & 2) | owner) : (uint32_t)owner;
                            st_async_v4(peer_smem(at, peer), v[j], v[j + 1], v[j + 2], v[j + 3], peer_smem(smem_u32(&b.sums_full[parity]), peer));
                        }
                    }
                }
            }
            io_barrier();
            wt.wait(&b.sums_full[parity], use & 1);
            // ---- sums in slice order, epilogue
#pragma unroll 1
            for (int i = tid; i < groups * K::Out; i += kIoThreads) {
                const int g = i / K::Out;                            // i % Out == c
                const float4* at = reinterpret_cast<const float4*>(sums) + g * K::Channels + c;
                float acc[4], up[4];
#pragma unroll
                for (int sp = 0; sp < K::AllParts; ++sp) {
                    const float4 v = at[sp * (Share / 4) * K::Channels];
                    const float v4[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                    for (int e = 0; e < 4; ++e) acc[e] = sp == 0 ? v4[e] : acc[e] + v4[e];
                    if (SHAPE == kPair) {
                        const float4 w = at[sp * (Share / 4) * K::Channels + 64];
                        const float w4[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
                        for (int e = 0; e < 4; ++e) up[e] = sp == 0 ? w4[e] : up[e] + w4[e];
                    }
                }
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    float val;
                    if (SHAPE == kPair) {
                        const float gate = acc[e] * scale;
                        val = __fdividef(gate, 1.0f + __expf(-gate)) * (up[e] * scale_up);
                    } else if (SHAPE == kNarrow) {
                        val = kind == kMtp ? rbf(acc[e] * scale) + bias : fmaf(acc[e], scale, own[e]);
                    } else {
                        val = acc[e] * scale;
                    }
                    const bf16 rounded = f2bf(val);
                    if (SHAPE == kNarrow) own[e] = bf2f(rounded);    // one group a thread: at most 16 rows of 64 channels
                    stage[(4 * g + e) * K::StageStride + c] = rounded;
                }
            }
            ++turn;
            io_barrier();
            // ---- results
            {
                constexpr int kPieces = K::Out / 8;
                unsigned char* const to = ex + (SHAPE == kWide ? (kind == kHead ? turns.at<vLogits>() : turns.at<vQkv>())
                                                : SHAPE == kPair ? turns.at<vAct>() : (kind == kO ? turns.at<vMid>() : turns.at<vIn>()));
                for (int i = tid; i < my_rows * kPieces; i += kIoThreads) {
                    const int row = i / kPieces, piece = i % kPieces;
                    const int4 v = *reinterpret_cast<const int4*>(stage + row * K::StageStride + 8 * piece);
                    if (SHAPE == kWide && kind == kHead && a.draws == 0) {
                        *reinterpret_cast<int4*>(a.logits + (size_t)(row0 + row) * kPredictorVocab + tile * 128 + 8 * piece) = v;
                    } else {
                        put_piece(to + place(which, kind, row0 + row, tile * K::Out + 8 * piece), v);
                    }
                }
            }
        };
        // marks what project() published there
        auto mark_again = [&](auto which, int kind, unsigned char* at) {
            using K = Of<decltype(which)::value>;
            if (!takes_part(kind, cluster)) return;
            constexpr int Share = MT / K::Sharers, kPieces = K::Out / 8;
            const int row0 = (K::Sharers == 2 ? rank & 1 : rank) * Share, my_rows = max(0, min(Share, rows - row0));
            for (int i = tid; i < my_rows * kPieces; i += kIoThreads) {
                put_piece(at + place(which, kind, row0 + i / kPieces, tile_of(kind, cluster, rank) * K::Out + 8 * (i % kPieces)), mark());
            }
        };

        // ---- attention of this CTA's (row, KV head) units, a warp each
        const int unit = cta + kCtas * warp;
        const bool has_unit = warp < 4 && unit < rows * KvHeads;
        const int arow = unit / KvHeads, head = unit % KvHeads;
        const int att_at = piece_at<MT>(arow, head * 256 + 8 * lane);
        bf16 *kpage = nullptr, *vpage = nullptr;
        if (has_unit) {
            const int pid = a.pages[arow];
            bf16* slab = a.kv.slabs[pid >> a.kv.slab_shift] + (long long)(pid & ((1 << a.kv.slab_shift) - 1)) * a.kv.page_elems
                         + (size_t)head * (kPageTokens * 128);
            kpage = slab + a.kv.k_offset;
            vpage = slab + a.kv.v_offset;
        }
        auto attention = [&](int layer, int pos) {
            if (has_unit) {
                unsigned char* scratch = smem + L::AtUnits + warp * kUnitBytes;
                bf16* raw = reinterpret_cast<bf16*>(scratch);                       // q, q, k, v as projected; k, v as kept
                float* qf = reinterpret_cast<float*>(scratch + 1024);
                bf16* result = raw;                                                  // the queries as projected have been read by then
                bf16* kdst = kpage + layer * a.kv_layer_elems;
                bf16* vdst = vpage + layer * a.kv_layer_elems;
                const ChainLayer& lc = m.layers[layer];
                bf16 wq[4], wk[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    wq[j] = lc.q_norm[lane + 32 * j];
                    wk[j] = lc.k_norm[lane + 32 * j];
                }
                const uint32_t cs0 = a.rope_table[pos * 64 + lane], cs1 = a.rope_table[pos * 64 + 32 + lane];
                page::Fragments f;
                page::load(f, kdst, vdst, pos, lane);
                // lanes 0..15 the first query head and the key, the others the second and the value
                const unsigned char* src = ex + turns.at<vQkv>() + arow * (kQkvWidth * 2) + (lane & 15) * 16;
                const bool upper = lane >= 16;
                int4 v[2];
                const int q_at = (2 * head + (upper ? 1 : 0)) * 256, kv_at = ((upper ? 24 : 16) + head) * 256;
                poll<2>(src + q_at, kv_at - q_at, v, wt);
                __syncwarp();
                reinterpret_cast<int4*>(raw)[lane] = v[0];
                reinterpret_cast<int4*>(raw)[32 + lane] = v[1];
                __syncwarp();
                float kept[4];
#pragma unroll
                for (int h = 0; h < 3; ++h) {
                    float x[4], y[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) x[j] = bf2f(raw[h * 128 + lane + 32 * j]);
                    page::rotate(x, h < 2 ? wq : wk, cs0, cs1, a.eps, y);
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        if (h < 2) qf[h * 128 + lane + 32 * j] = y[j];
                        else kept[j] = y[j];
                    }
                }
                __syncwarp();
#pragma unroll
                for (int j = 0; j < 4; ++j) raw[256 + lane + 32 * j] = f2bf(kept[j]);
                __syncwarp();
                {
                    const int4 piece = *reinterpret_cast<const int4*>(raw + 256 + lane * 8);
                    *reinterpret_cast<int4*>((upper ? vdst : kdst) + (size_t)pos * 128 + (lane % 16) * 8) = piece;
                }
                if (pos > 0 || layer < Layers - 1) {
                    page::patch(f, raw + 256, raw + 384, pos, lane);
                    float mx, lsum, o[8][4];
                    page::attend(f, qf, pos + 1, rsqrtf(128.0f), lane, mx, lsum, o);
                    const int tig = lane & 3, gid = lane >> 2;
                    const float inv0 = 1.0f / __shfl_sync(0xffffffffu, lsum, (2 * tig) * 4 % kWarp);
                    const float inv1 = 1.0f / __shfl_sync(0xffffffffu, lsum, (2 * tig + 1) * 4 % kWarp);
                    if (tig == 0) {
#pragma unroll
                        for (int g = 0; g < 2; ++g)
#pragma unroll
                            for (int half = 0; half < 2; ++half) {
                                const float inv = g == 0 ? inv0 : inv1;
                                float v8[8];
#pragma unroll
                                for (int x = 0; x < 8; ++x) v8[x] = o[x][2 * half + g] * inv;
                                int4 packed;
                                packed.x = static_cast<int>(page::pack_bf16x2(v8[0], v8[1]));
                                packed.y = static_cast<int>(page::pack_bf16x2(v8[2], v8[3]));
                                packed.z = static_cast<int>(page::pack_bf16x2(v8[4], v8[5]));
                                packed.w = static_cast<int>(page::pack_bf16x2(v8[6], v8[7]));
                                *reinterpret_cast<int4*>(result + g * 128 + 64 * half + 8 * gid) = packed;
                            }
                    }
                    __syncwarp();
                    put_piece(ex + turns.at<vAtt>() + att_at, *reinterpret_cast<const int4*>(result + 8 * lane));
                }
            }
        };

        // ---- a row's draw, one CTA
        const int draw_row = cta / 2;
        const bool has_draw = a.draws != 0 && cta % 2 == 1 && draw_row < rows;
        auto draw = [&](int p) {
            if (!has_draw) return;
            unsigned int* keys = reinterpret_cast<unsigned int*>(xs);
            TopKScratch& scratch = *reinterpret_cast<TopKScratch*>(xs + kPredictorVocab * sizeof(unsigned int));
            static_assert(kPredictorVocab * sizeof(unsigned int) + sizeof(TopKScratch) <= L::XBytes, "the draw lies over the activations");
            const SamplingParams sp = a.table->predictor[draw_row];
            int4 v[1];
            poll<1>(ex + turns.at<vLogits>() + draw_row * (kPredictorVocab * 2) + tid * 16, 0, v, wt);
            const int four[4] = {v[0].x, v[0].y, v[0].z, v[0].w};
            unsigned long long best = 0ull;
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const uint32_t w = (uint32_t)four[e / 2];
                const unsigned int key = order_key(e % 2 == 0 ? bf_lo(w) : bf_hi(w));
                keys[8 * tid + e] = key;
                const unsigned long long k = (static_cast<unsigned long long>(key) << 12) | static_cast<unsigned long long>(4095 - (8 * tid + e));
                best = k > best ? k : best;
            }
            int token;
            if (sp.do_sample == 0) {
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    const unsigned long long other = __shfl_xor_sync(0xffffffffu, best, o);
                    best = other > best ? other : best;
                }
                if (lane == 0) scratch.warp_best[warp] = best;
                io_barrier();
                for (int w = 0; w < kIoWarps; ++w) best = scratch.warp_best[w] > best ? scratch.warp_best[w] : best;
                token = 4095 - static_cast<int>(best & 0xfffull);
            } else {
                io_barrier();
                token = sample_top_k_block<kIoThreads, kPredictorVocab / kIoThreads>(keys, kPredictorVocab, min(sp.top_k, kPredictorVocab), sp.top_p, sp.temperature,
                                                                                   a.table->rng[draw_row], scratch, tid, [] { io_barrier(); });
            }
            if (tid == 0) {
                put_piece(ex + turns.at<vTokens>() + draw_row * 16, make_int4(token, 0, 0, 0));
                put_piece(ex + turns.before<vTokens>() + draw_row * 16, mark());
                a.table->frame_tokens[draw_row][p] = token;
                marks_stand();
            }
            io_barrier();                                            // the next activations lie where the draw did
        };

        using Narrow = std::integral_constant<int, kNarrow>;
        using Wide = std::integral_constant<int, kWide>;
        using Pair = std::integral_constant<int, kPair>;
        projections(a, [&](int kind, int layer, int p) {
            if (is_narrow(kind)) project(Narrow(), kind, layer, p);
            else if (kind == kGateUp) project(Pair(), kind, layer, p);
            else project(Wide(), kind, layer, p);
            const bool ends_early = p == 0 && layer == Layers - 1;
            if (kind == kQkv) attention(layer, p);
            if (is_normed(kind)) turns.next<vNormed>();
            if (kind == kQkv || kind == kHead) turns.next<vIn>();
            // What was published in a layer is followed up at its end, while the next norm is under way.
            if (kind == kMtp) {
                mark_again(Narrow(), kMtp, ex + turns.before<vIn>());
                marks_stand();
            } else if (kind == kDown || (kind == kQkv && ends_early)) {
                mark_again(Wide(), kQkv, ex + turns.before<vQkv>());
                if (kind == kDown) {
                    if (has_unit) put_piece(ex + turns.before<vAtt>() + att_at, mark());
                    mark_again(Narrow(), kO, ex + turns.before<vMid>());
                    mark_again(Pair(), kGateUp, ex + turns.before<vAct>());
                    mark_again(Narrow(), kDown, ex + turns.before<vIn>());
                    turns.next<vAtt>();
                    turns.next<vMid>();
                    turns.next<vAct>();
                }
                marks_stand();
                turns.next<vQkv>();
            } else if (kind == kHead && a.draws != 0) {
                draw(p);
                mark_again(Wide(), kHead, ex + turns.before<vLogits>());
                marks_stand();
                turns.next<vLogits>();
                turns.next<vTokens>();
            }
        });
        if (cta == 0 && tid == 0) {
#pragma unroll
            for (int v = 0; v < kValues; ++v) state[2 + v] = turns.now[v];
        }
    }

    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (b.abort != 0) {
        // give copies that are still in flight time to land before the CTA's memory is released
        if (tid == 0) {
            atomicAdd(&g_lockstep_errors, 1u);
            if (g_lockstep_error_sink != nullptr) atomicAdd_system(g_lockstep_error_sink, 1u);
        }
        const unsigned long long until = now_ns() + 200000ull;
        while (now_ns() < until) __nanosleep(1000);
    }
    // a neighbour may still send here, and every CTA has read the launch's base by now
    cluster_sync();
    if (cta == 0 && tid == 0) *state = wt.base >= kNoLaunch - 1 ? 0 : wt.base + 1;
    if (warp == kRoleWarp + 2) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
    }
}

// Every place marked, all turns at their first buffer, no launch given up.  Places of the tile's rows that nobody has are zeros, there
// from the beginning: whoever polls for a tile takes them as they are.
__global__ void __launch_bounds__(512) restart_kernel(unsigned char* exchange, int rows, int tile) {
    static_assert(kAtState % 16 == 0 && 4 * (2 + kValues) <= 128, "the state behind the values");
    for (int at = 16 * (blockIdx.x * blockDim.x + threadIdx.x); at < kAtState; at += 16 * gridDim.x * blockDim.x) {
        bool nobodys = false;
        for (int v : {vNormed, vAtt, vAct}) {
            if (at >= at_value(v) && at < at_value(v + 1)) nobodys = (at - at_value(v)) % value_bytes(v) % (tile * 128) / 128 >= rows;
        }
        *reinterpret_cast<int4*>(exchange + at) = nobodys ? make_int4(0, 0, 0, 0) : mark();
    }
    uint32_t* state = reinterpret_cast<uint32_t*>(exchange + kAtState);
    if (blockIdx.x == 0 && threadIdx.x < 2 + kValues) state[threadIdx.x] = threadIdx.x == 1 ? kNoLaunch : 0u;
}

// ---------------------------------------------------------------------------------- host side

bool g_lockstep_fits[64] = {};

template <int MT>
void cluster_launch(cudaLaunchConfig_t& cfg, cudaLaunchAttribute (&attr)[2], cudaStream_t stream) {
    cfg = {};
    cfg.gridDim = dim3(kCtas);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = Layout<MT>::Bytes;
    cfg.stream = stream;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = kRanks;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeCooperative;
    attr[1].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
}

template <int MT>
cudaError_t configure_variant(bool& fits) {
    cudaFuncAttributes built;
    cudaError_t e = cudaFuncGetAttributes(&built, lockstep_chain_kernel<MT>);
    if (e == cudaSuccess) {
        e = cudaFuncSetAttribute(lockstep_chain_kernel<MT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Layout<MT>::Bytes);
    }
    if (e != cudaSuccess) return e;
    fits = fits && built.numRegs >= 96;                              // what setmaxnreg hands out has to be there
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr[2];
    cluster_launch<MT>(cfg, attr, nullptr);
    cfg.numAttrs = 1;
    int clusters = 0;
    e = cudaOccupancyMaxActiveClusters(&clusters, lockstep_chain_kernel<MT>, &cfg);
    fits = fits && clusters >= kClusters;
    return e;
}

template <int MT>
cudaError_t launch_variant(const LockstepArgs& a, cudaStream_t stream) {
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr[2];
    cluster_launch<MT>(cfg, attr, stream);
    return cudaLaunchKernelEx(&cfg, lockstep_chain_kernel<MT>, a);
}

}  // namespace

cudaError_t configure_lockstep_kernels() {
    int device = 0, cooperative = 0;
    bool fits = true;
    cudaError_t e = cudaGetDevice(&device);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&cooperative, cudaDevAttrCooperativeLaunch, device);
    if (e == cudaSuccess) e = configure_variant<16>(fits);
    if (e == cudaSuccess) e = configure_variant<32>(fits);
    if (e == cudaSuccess) e = configure_variant<48>(fits);
    if (e == cudaSuccess) e = configure_variant<64>(fits);
    if (e == cudaSuccess && device >= 0 && device < 64) g_lockstep_fits[device] = fits && cooperative != 0;
    return e;
}

// The kernel sums the K-slices that these are.  (8 rows and fewer: see the hand-overs.)
bool lockstep_chain_available(int rows) {
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= 64 || !g_lockstep_fits[device] || rows <= kChainRows || rows > kMaxRows) return false;
    return gemm_tc_slices(4096, H, rows, false) == 4 && gemm_tc_slices(H, QWidth, rows, false) == 8 && gemm_tc_slices(I, H, rows, true) == 2
           && gemm_tc_slices(H, I, rows, false) == 8 && gemm_tc_slices(kPredictorVocab, H, rows, false) == 4
           && gemm_tc_slices(H, TalkerH, rows, false) == 8;
}

bool make_lockstep_map(LockstepModel* model, int index, const int8_t* weights, int in_features, int matrix_rows, bool wide) {
    CUtensorMap map;
    if (!make_map(&map, CU_TENSOR_MAP_DATA_TYPE_UINT8, weights, in_features, matrix_rows, in_features, kBK, wide ? 128 : 64, CU_TENSOR_MAP_SWIZZLE_128B)) {
        return false;
    }
    static_assert(sizeof(map) == sizeof(model->maps[0]), "a tensor map");
    std::memcpy(model->maps[index], &map, sizeof(map));
    return true;
}

size_t lockstep_exchange_bytes() { return kExchangeBytes; }

cudaError_t restart_lockstep(void* exchange, int rows, cudaStream_t stream) {
    restart_kernel<<<148, 512, 0, stream>>>(static_cast<unsigned char*>(exchange), rows, gemm_tc_tile(rows));
    return cudaGetLastError();
}

cudaError_t launch_lockstep_chain(const LockstepLaunch& c, cudaStream_t stream) {
    if (!lockstep_chain_available(c.rows) || c.first < 0 || c.first > c.last || c.last >= kCodebooks) return cudaErrorInvalidValue;
    LockstepArgs a;
    a.model = c.model; a.table = c.table; a.pages = c.pages; a.kv = c.kv; a.kv_layer_elems = c.kv_layer_elems;
    a.rope_table = c.rope_table; a.codec_embedding = c.codec_embedding; a.embeddings = c.embeddings; a.logits = c.logits;
    a.exchange = static_cast<unsigned char*>(c.exchange);
    a.rows = c.rows; a.first = c.first; a.last = c.last; a.draws = c.draws ? 1 : 0; a.eps = kRmsEps;
    switch (gemm_tc_tile(c.rows)) {
        case 16: return launch_variant<16>(a, stream);
        case 32: return launch_variant<32>(a, stream);
        case 48: return launch_variant<48>(a, stream);
        default: return launch_variant<64>(a, stream);
    }
}

unsigned int lockstep_error_count() {
    unsigned int v = 0;
    if (cudaMemcpyFromSymbol(&v, g_lockstep_errors, sizeof(v)) != cudaSuccess) return ~0u;
    return v;
}

cudaError_t set_lockstep_error_sink(unsigned int* device_visible_word) {
    return cudaMemcpyToSymbol(g_lockstep_error_sink, &device_visible_word, sizeof(device_visible_word));
}

}  // namespace q3t
