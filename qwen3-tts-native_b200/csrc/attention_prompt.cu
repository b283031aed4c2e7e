// Attention of a prompt pass: many consecutive positions of one session attend to the session's paged
// cache, each up to itself.
//
// Semantics as in attention.cu (the reference's batch_causal_gqa_attention_fast_kernel,
// native/qwen3-tts-native/native/src/talker_kernels.cu:506-595, after the per-head RMSNorm, RoPE and
// cache append of :50-70, :597-658); the decode kernel there treats every row as a session of its own
// and reads its whole context again, which for a prompt of n positions is n^2 / 2 cache rows a layer.
// Here a CTA takes 64 positions of the two query heads of a KV head, 128 rows of the tensor cores, and walks their
// common context once, 64 tokens at a time, with a running softmax.
//
//   scores    S = Q K^T, tcgen05.mma from shared memory into 64 columns of tensor memory
//   softmax   two threads a row, half of the step's tokens each: S to registers (the next step's products may begin), weights as
//             bf16 hi + lo (16 bits kept) back to tensor memory
//   output    O += P V, hi and lo as the A operand from tensor memory, V as it lies in its pages
//   copies    K and V, by two warps each, two steps ahead of their products (cp.async: the pages lie anywhere), the queries by the softmax's
// A row's reference is its first maximum until a score exceeds it by 2^8: weights above one cost no precision in floating point,
// and an output in tensor memory is rescaled at almost no step instead of almost every one (some row of 32 has a new maximum).
//
// Short passes are one or two steps a CTA, bound by the way of the first operands from the L2: the first pages are looked up ahead
// of the launch's wait, the softmax warps bring the queries, and a CTA takes 32 positions (half of its rows idle) while twice as
// many CTAs fit the SMs.  A prompt of 64 positions (us) 1,441 -> 1,406, 12 1,162 -> 1,151, 128 1,648 -> 1,628 (halves against whole
// blocks: 64 1,431 -> 1,406, 128 1,646 -> 1,628); with mma.sync 1,412, 1,155 and 1,690.
//
// What bounds it else: the chain of a step in its softmax threads, times the steps of the longest context; two CTAs an SM take turns
// at the issue slots.  1,500 positions: 68 us a layer with mma.sync (32 positions a CTA, the weights' two halves as 3 x 64 x 64 x 128
// products a step at the legacy rate), 54 so with K and V in one buffer, 45 with a buffer each, 43 with two threads a row.

#include "q3t_kernels.cuh"
#include "q3t_tcgen05.cuh"

namespace q3t {
namespace {

constexpr int kHd = 128;
constexpr int kBlockPositions = 64;
constexpr int kStepTokens = 64;
constexpr int kRows = 2 * kBlockPositions;              // of the tensor cores: position + 64 * head
constexpr int kFlashThreads = 416;                      // warps 0..7 softmax, 8..11 copies, 12 products
// Registers: 72 a thread at launch (two CTAs an SM); the copying warps hand 16 each to the softmax's, which spill with 72
constexpr int kLaunchRegisters = 72, kSoftmaxRegisters = 80, kCopyRegisters = 56;
static_assert(2 * kSoftmaxRegisters + kCopyRegisters <= 3 * kLaunchRegisters, "registers of the three groups of four warps");
constexpr int kCopyWarp = 8, kProductWarp = 12;
constexpr int kHalf = kStepTokens / 2;                  // tokens of a step, to each of a row's two threads
constexpr int kTileBytes = kStepTokens * kHd * 2;       // 16 KB of K or V: [64 dims][token][128 bytes, swizzled]
constexpr int kQueryBytes = kRows * kHd * 2;
constexpr int kBuffers = 2;
constexpr int kFlashCtas = 2;
constexpr int kSms = 148;
constexpr uint32_t kTmemCols = 256, kScores = 0, kHi = 64, kLo = 96, kOut = 128;
constexpr float kSlack = 8.0f;                          // log2 of the largest weight
constexpr unsigned long long kBudgetNs = 2000000000ull;
constexpr size_t kFlashSmem = 1024 + kQueryBytes + kBuffers * 2 * kTileBytes + 4 * kRows * 4 + 128;

__device__ unsigned int g_prompt_attention_errors = 0;
__device__ unsigned int* g_prompt_attention_error_sink = nullptr;

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ uint32_t pack_pair(float lo, float hi) {
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}
__device__ __forceinline__ void copy16(uint32_t dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}

// 2^x, x <= kSlack (the reference may lie that far below a row's maximum, so that weights reach 256): as exp2f, but what would be
// subnormal is zero
__device__ __forceinline__ float exp2_ftz(float x) {
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

struct PromptArgs {
    bf16* qkv;                 // [rows][qkv_stride]: q | k | v; q is normalised and rotated in place by the append
    const bf16* q_norm_w;
    const bf16* k_norm_w;
    const uint32_t* rope_table;
    bf16* out;                 // [rows][q_heads * 128]
    KvLayout kv;               // the session's page list is row 0 of the table
    int qkv_stride;
    int base;                  // position of row 0
    int rows;
    int q_heads, kv_heads;
    float eps;
};

__device__ __forceinline__ bf16* page_of(const PromptArgs& a, int token, int kvh, bool value) {
    const int pid = a.kv.page_table[token / kPageTokens];
    bf16* slab = a.kv.slabs[pid >> a.kv.slab_shift];
    const long long in_slab = (long long)(pid & ((1 << a.kv.slab_shift) - 1)) * a.kv.page_elems;
    return slab + in_slab + (value ? a.kv.v_offset : a.kv.k_offset) + (size_t)kvh * (kPageTokens * kHd);
}

// One CTA per position, one warp per head in turn: per-head RMSNorm and rotation of q (in place) and
// k (into the cache), v copied into the cache; the arithmetic of the decode kernel's prologue.
__global__ void __launch_bounds__(256) prompt_append_kernel(const PromptArgs a) {
    const int lane = threadIdx.x % kWarp;
    const int warp = threadIdx.x / kWarp;
    const int row = blockIdx.x;
    const int pos = a.base + row;
    float wq[4], wk[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        wq[j] = bf2f(a.q_norm_w[lane + 32 * j]);
        wk[j] = bf2f(a.k_norm_w[lane + 32 * j]);
    }
    uint32_t cs[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) cs[j] = a.rope_table[(size_t)pos * (kHd / 2) + lane + 32 * j];
    // where the position lies in its page, of KV head 0: looked up ahead of the wait, two loads one behind the other
    bf16* const place = page_of(a, pos, 0, false) + (size_t)(pos % kPageTokens) * kHd;
    pdl_wait();
    pdl_trigger();
    // three heads a warp at a time (all of the talker's 16 + 8), requested together: one latency
    constexpr int kJobs = 3;
    const int total = a.q_heads + a.kv_heads;
    for (int first = warp; first < total; first += 8 * kJobs) {
        bf16 raw[kJobs][4], value[kJobs][4];
#pragma unroll
        for (int u = 0; u < kJobs; ++u) {
            const int job = first + 8 * u;
            const bf16* src = a.qkv + (size_t)row * a.qkv_stride + (size_t)job * kHd;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (job < total) raw[u][j] = src[lane + 32 * j];
                if (job >= a.q_heads && job < total) value[u][j] = src[(size_t)a.kv_heads * kHd + lane + 32 * j];
            }
        }
#pragma unroll
        for (int u = 0; u < kJobs; ++u) {
            const int job = first + 8 * u;
            if (job >= total) break;
            const bool is_key = job >= a.q_heads;
            float x[4], sq[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                x[j] = bf2f(raw[u][j]);
                sq[j] = fmaf(x[j], x[j], 0.0f);
            }
            float c = (sq[0] + sq[2]) + (sq[1] + sq[3]);
            c = warp_sum_down(c);
            c = __shfl_sync(0xffffffffu, c, 0);
            const float inv = rsqrtf(c / static_cast<float>(kHd) + a.eps);
            float y[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) y[j] = rbf(rbf(x[j] * inv) * (is_key ? wk[j] : wq[j]));
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                float o1, o2;
                rope_pair_cs(y[j], y[j + 2], bf_lo(cs[j]), bf_hi(cs[j]), o1, o2);
                y[j] = o1;
                y[j + 2] = o2;
            }
            if (is_key) {
                const int kvh = job - a.q_heads;
                bf16* kdst = place + (size_t)kvh * (kPageTokens * kHd);
                bf16* vdst = kdst + (a.kv.v_offset - a.kv.k_offset);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    kdst[lane + 32 * j] = f2bf(y[j]);
                    vdst[lane + 32 * j] = value[u][j];
                }
            } else {
                bf16* dst = a.qkv + (size_t)row * a.qkv_stride + (size_t)job * kHd;
#pragma unroll
                for (int j = 0; j < 4; ++j) dst[lane + 32 * j] = f2bf(y[j]);
            }
        }
    }
}

// 16-byte piece `piece` (0..15) of row `t` of a tile of `rows`: K-major for the products over dims, and for those over tokens
// as it is, with the dims contiguous
__device__ __forceinline__ uint32_t tile_offset(int rows, int t, int piece) {
    return (uint32_t)((piece >> 3) * rows * 128 + t * 128 + (((piece & 7) ^ (t & 7)) << 4));
}
// B operand whose rows are contiguous: 64 of them in 128 bytes (swizzled), the next 64 a tile of tokens further on, eight of K 1024 bytes
__device__ __forceinline__ uint64_t desc_rows_contiguous(uint32_t smem) {
    return (uint64_t)((smem >> 4) & 0x3FFFu) | ((uint64_t)(kStepTokens * 128 / 16) << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ void umma_ss(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void tmem_store_16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
          "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}

template <int BLOCK>                                          // positions of a CTA: kBlockPositions, or half of them
__global__ void __launch_bounds__(kFlashThreads, kFlashCtas) prompt_attention_kernel(const PromptArgs a) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    unsigned char* queries = smem;
    unsigned char* tiles = smem + kQueryBytes;                // buffer: K, V
    float* tops = reinterpret_cast<float*>(tiles + kBuffers * 2 * kTileBytes);             // [step % 2][half][row]
    uint64_t* full_k = reinterpret_cast<uint64_t*>(tops + 4 * kRows);
    uint64_t* full_v = full_k + kBuffers;
    uint64_t* empty_k = full_v + kBuffers;
    uint64_t* empty_v = empty_k + kBuffers;
    uint64_t* s_ready = empty_v + kBuffers;                   // scores in tensor memory
    uint64_t* s_free = s_ready + 1;                           // and in registers
    uint64_t* p_ready = s_free + 1;                           // weights in tensor memory
    uint64_t* o_ready = p_ready + 1;                          // multiplied
    uint64_t* q_ready = o_ready + 1;                          // queries in shared memory
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(q_ready + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int tid = threadIdx.x;
    const int warp = __shfl_sync(0xffffffffu, tid / kWarp, 0);
    const int lane = tid % kWarp;
    // the last positions have the longest context: they go first, all KV heads of a block together
    const int kvh = (int)blockIdx.x % a.kv_heads;
    const int block = ((int)gridDim.x - 1 - (int)blockIdx.x) / a.kv_heads;
    const int row0 = block * BLOCK;
    const int rows_end = BLOCK == kBlockPositions ? a.rows : min(a.rows, row0 + BLOCK);
    const int length = a.base + min(a.rows, row0 + BLOCK);      // tokens the CTA walks
    const int steps = (length + kStepTokens - 1) / kStepTokens;

    tc::Guard guard;
    guard.deadline = tc::now_ns() + kBudgetNs;
    guard.abort_flag = abort_flag;
    if (tid == 0) {
        for (int i = 0; i < kBuffers; ++i) {
            tc::mbar_init(&full_k[i], 2);
            tc::mbar_init(&full_v[i], 2);
            tc::mbar_init(&empty_k[i], 1);
            tc::mbar_init(&empty_v[i], 1);
        }
        tc::mbar_init(s_ready, 1);
        tc::mbar_init(s_free, 8);
        tc::mbar_init(p_ready, 8);
        tc::mbar_init(o_ready, 1);
        tc::mbar_init(q_ready, 8);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kProductWarp) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc::smem_u32(tmem_slot)), "r"(kTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;

    if (warp >= kCopyWarp && warp < kProductWarp) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kCopyRegisters));
        // ---- copies: K by the first two warps, V by the others; thread t takes piece t % 16 of tokens t / 16, + 4, + 8, + 12 of every
        // page.  Pages are looked up a step ahead, two loads one behind the other; the first step's ahead of the launch's wait, since the
        // page table is older than the launch before.
        const bool values = warp >= kCopyWarp + 2;
        const int t = (tid - kCopyWarp * kWarp) % (2 * kWarp), piece = t & 15;
        uint64_t* const landed = values ? full_v : full_k;
        uint64_t* const used = values ? empty_v : empty_k;
        constexpr int kPages = kStepTokens / kPageTokens;
        const bf16* pages[kPages];
        auto look_up = [&](int step) {
#pragma unroll
            for (int page = 0; page < kPages; ++page) {
                const int first = step * kStepTokens + page * kPageTokens;
                pages[page] = first < length ? page_of(a, first, kvh, values) + (t >> 4) * kHd + piece * 8 : nullptr;
            }
        };
        const uint32_t at = tile_offset(kStepTokens, t >> 4, piece);
        look_up(0);
        pdl_wait();
        pdl_trigger();
        for (int step = 0; step < steps; ++step) {
            const int buffer = step % kBuffers;
            if (step >= kBuffers && !__all_sync(0xffffffffu, guard.wait(&used[buffer], ((step / kBuffers) - 1) & 1))) break;
            unsigned char* const tile = tiles + (buffer * 2 + (values ? 1 : 0)) * kTileBytes;
#pragma unroll
            for (int page = 0; page < kPages; ++page) {
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    // (four tokens further on: another swizzle of the 16-byte pieces)
                    unsigned char* const to = tile + (at ^ ((u & 1) * 64)) + (page * kPageTokens + 4 * u) * 128;
                    if (step * kStepTokens + page * kPageTokens + 4 * u + (t >> 4) < length) {
                        copy16(smem_addr(to), pages[page] + 4 * u * kHd);
                    } else {
                        // past the end: the scores are masked, but 0 * (stale bits that decode as NaN) is not zero
                        *reinterpret_cast<int4*>(to) = make_int4(0, 0, 0, 0);
                    }
                }
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
            look_up(step + 1);
            if (step > 0) {
                asm volatile("cp.async.wait_group 1;" ::: "memory");
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) tc::mbar_arrive(&landed[(step - 1) % kBuffers]);
            }
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0 && *abort_flag == 0) tc::mbar_arrive(&landed[(steps - 1) % kBuffers]);
    } else if (warp == kProductWarp) {
        if (tc::elect_one()) {
            // ---- products
            const uint32_t scores_idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kStepTokens >> 3) << 17) | ((uint32_t)(kRows >> 4) << 24);
            // B with its rows (dims) contiguous: bit 16
            const uint32_t out_idesc = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) | ((uint32_t)(kHd >> 3) << 17) | ((uint32_t)(kRows >> 4) << 24);
            auto scores = [&](int step) {
                const uint32_t q = tc::smem_u32(queries), k = tc::smem_u32(tiles + (step % kBuffers) * 2 * kTileBytes);
#pragma unroll
                for (int j = 0; j < kHd / 16; ++j) {
                    umma_ss(tmem + kScores, tc::umma_desc(q + (j / 4) * kRows * 128 + 32 * (j % 4)),
                            tc::umma_desc(k + (j / 4) * kStepTokens * 128 + 32 * (j % 4)), scores_idesc, j != 0 ? 1u : 0u);
                }
                tc::umma_commit(s_ready);
                tc::umma_commit(&empty_k[step % kBuffers]);
            };
            bool ok = guard.wait(q_ready, 0) && guard.wait(&full_k[0], 0);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (ok) scores(0);
            for (int step = 0; step < steps && ok; ++step) {
                if (step + 1 < steps) {
                    ok = guard.wait(&full_k[(step + 1) % kBuffers], ((step + 1) / kBuffers) & 1) && guard.wait(s_free, step & 1);
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    scores(step + 1);
                }
                ok = guard.wait(&full_v[step % kBuffers], (step / kBuffers) & 1) && guard.wait(p_ready, step & 1);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t v = tc::smem_u32(tiles + (step % kBuffers) * 2 * kTileBytes + kTileBytes);
#pragma unroll
                for (int j = 0; j < kStepTokens / 16; ++j) {
                    const uint64_t tokens = desc_rows_contiguous(v + j * 16 * 128);
                    tc::umma_f16_ts(tmem + kOut, tmem + kHi + 8 * j, tokens, out_idesc, (step | j) != 0 ? 1u : 0u);
                    tc::umma_f16_ts(tmem + kOut, tmem + kLo + 8 * j, tokens, out_idesc, 1u);
                }
                tc::umma_commit(&empty_v[step % kBuffers]);
                tc::umma_commit(o_ready);
            }
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kSoftmaxRegisters));
        // ---- softmax: two threads a row, each half of a step's tokens
        pdl_wait();
#pragma unroll
        for (int i = 0; i < kRows * kHd / 8 / 256; ++i) {
            const int q_row = (tid >> 4) + 16 * i, q_piece = tid & 15;
            const bf16* q = a.qkv + (size_t)min(row0 + q_row % kBlockPositions, rows_end - 1) * a.qkv_stride + (size_t)(kvh * 2 + q_row / kBlockPositions) * kHd;
            copy16(smem_addr(queries) + tile_offset(kRows, q_row, q_piece), q + 8 * q_piece);
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(q_ready);
        const int half = warp >> 2, quarter = warp & 3;
        const int row = quarter * kWarp + lane;
        const int position = row % kBlockPositions;
        const int last = a.base + row0 + position;            // the newest token that the row sees
        const uint32_t lanes = tmem + ((uint32_t)(quarter * kWarp) << 16);
        // scores are kept in units of log2(e) / sqrt(128), so that exp is one exp2
        const float scale = rsqrtf(static_cast<float>(kHd)) * 1.4426950408889634f;
        auto meet = [&]() {                                   // the two warps of these rows
            __syncwarp();
            asm volatile("bar.sync %0, 64;" ::"r"(1 + quarter) : "memory");
        };
        float m = -INFINITY, l = 0.0f;                        // of both; of this half
        for (int step = 0; step < steps; ++step) {
            guard.wait(s_ready, step & 1);
            __syncwarp();
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            float sc[kHalf];
            tc::tmem_load_row<kHalf>(lanes + kScores + half * kHalf, sc);
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(s_free);
            const int t0 = step * kStepTokens + half * kHalf;
            if (t0 + kHalf - 1 > a.base + row0 + (quarter & 1) * kWarp) {          // some row of the warp ends in this half
#pragma unroll
                for (int j = 0; j < kHalf; ++j)
                    if (t0 + j > last) sc[j] = -INFINITY;
            }
            float mx[4] = {sc[0], sc[1], sc[2], sc[3]};
#pragma unroll
            for (int j = 4; j < kHalf; ++j) mx[j & 3] = fmaxf(mx[j & 3], sc[j]);
            float top = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * scale;
            float* const at = tops + (step & 1) * 2 * kRows + row;
            at[half * kRows] = top;
            meet();
            top = fmaxf(top, at[(half ^ 1) * kRows]);
            const float moved = step == 0 || top > m + kSlack ? top : m;
            const bool rescale = __any_sync(0xffffffffu, moved != m) && step > 0;
            const float f = moved == m ? 1.0f : (step == 0 ? 0.0f : exp2_ftz(m - moved));
            m = moved;
            // (nothing but -inf so far: weights of zero)
            const float reference = m == -INFINITY ? 0.0f : m;
            // (pairs of ordinary operations: this part is bound by the issue of its instructions)
            const unsigned long long scale2 = pack2(scale, scale), minus2 = pack2(-reference, -reference), negative2 = pack2(-1.0f, -1.0f);
            unsigned long long sums[2] = {pack2(l * f, 0.0f), pack2(0.0f, 0.0f)};
            uint32_t hi[kHalf / 2], lo[kHalf / 2];
#pragma unroll
            for (int j = 0; j < kHalf / 2; ++j) {
                float p0, p1, rest0, rest1;
                unpack2(fma2(pack2(sc[2 * j], sc[2 * j + 1]), scale2, minus2), p0, p1);
                p0 = exp2_ftz(p0);
                p1 = exp2_ftz(p1);
                const unsigned long long weights = pack2(p0, p1);
                sums[j & 1] = add2(sums[j & 1], weights);
                hi[j] = pack_pair(p0, p1);
                unpack2(fma2(pack2(bf_lo(hi[j]), bf_hi(hi[j])), negative2, weights), rest0, rest1);       // exact
                lo[j] = pack_pair(rest0, rest1);
            }
            float s0, s1, s2, s3;
            unpack2(sums[0], s0, s1);
            unpack2(sums[1], s2, s3);
            l = (s0 + s1) + (s2 + s3);
            // what the step before has left in tensor memory is being multiplied up to here
            if (step > 0) guard.wait(o_ready, (step - 1) & 1);
            __syncwarp();
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (rescale) {
#pragma unroll 1
                for (int c = half * (kHd / 2); c < (half + 1) * (kHd / 2); c += 16) {
                    float o[16];
                    uint32_t bits[16];
                    tc::tmem_load_row<16>(lanes + kOut + c, o);
#pragma unroll
                    for (int j = 0; j < 16; ++j) bits[j] = __float_as_uint(o[j] * f);
                    tmem_store_16(lanes + kOut + c, bits);
                }
            }
            tmem_store_16(lanes + kHi + 16 * half, hi);
            tmem_store_16(lanes + kLo + 16 * half, lo);
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(p_ready);
        }
        float* const sum_at = tops + (steps & 1) * 2 * kRows + row;
        sum_at[half * kRows] = l;
        meet();
        const float inv = 1.0f / (tops[(steps & 1) * 2 * kRows + row] + tops[(steps & 1) * 2 * kRows + kRows + row]);
        guard.wait(o_ready, (steps - 1) & 1);
        __syncwarp();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        bf16* dst = a.out + (size_t)(row0 + position) * a.q_heads * kHd + (size_t)(kvh * 2 + row / kBlockPositions) * kHd;
#pragma unroll 1
        for (int c = half * (kHd / 2); c < (half + 1) * (kHd / 2); c += 16) {
            float o[16];
            tc::tmem_load_row<16>(lanes + kOut + c, o);
            if (row0 + position < rows_end && *abort_flag == 0) {
#pragma unroll
                for (int j = 0; j < 16; j += 8) {
                    int4 v;
                    v.x = (int)pack_pair(o[j] * inv, o[j + 1] * inv);
                    v.y = (int)pack_pair(o[j + 2] * inv, o[j + 3] * inv);
                    v.z = (int)pack_pair(o[j + 4] * inv, o[j + 5] * inv);
                    v.w = (int)pack_pair(o[j + 6] * inv, o[j + 7] * inv);
                    *reinterpret_cast<int4*>(dst + c + j) = v;
                }
            }
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    }
    __syncwarp();
    __syncthreads();
    if (*abort_flag != 0 && tid == 0) {
        atomicAdd(&g_prompt_attention_errors, 1u);
        if (g_prompt_attention_error_sink != nullptr) atomicAdd_system(g_prompt_attention_error_sink, 1u);
        const unsigned long long until = tc::now_ns() + 200000ull;       // products that are still under way
        while (tc::now_ns() < until) __nanosleep(1000);
    }
    if (*abort_flag != 0) __syncthreads();
    if (warp == kProductWarp) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
    }
}

}  // namespace

namespace {
template <int BLOCK>
cudaError_t configure_block() {
    cudaFuncAttributes built;
    cudaError_t e = cudaFuncGetAttributes(&built, prompt_attention_kernel<BLOCK>);
    if (e == cudaSuccess && built.numRegs < kLaunchRegisters) e = cudaErrorInvalidConfiguration;     // what setmaxnreg hands out has to be there
    return e != cudaSuccess ? e : cudaFuncSetAttribute(prompt_attention_kernel<BLOCK>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFlashSmem);
}
}  // namespace

cudaError_t configure_prompt_kernels() {
    const cudaError_t e = configure_block<kBlockPositions>();
    return e != cudaSuccess ? e : configure_block<kBlockPositions / 2>();
}

bool prompt_attention_supports(const AttentionArgs& a) {
    return a.head_dim == kHd && a.fused != 0 && a.q_heads == 2 * a.kv_heads && a.kv.page_table != nullptr
           && a.kv.table_stride == 0 && a.rope_table != nullptr && a.out32 == nullptr;
}

// rows are the consecutive positions base .. base + rows - 1 of the session whose pages row 0 lists;
// a.q, a.k_new and a.v_new are the parts of one packed projection, q is overwritten
cudaError_t launch_prompt_attention(const AttentionArgs& a, int base, cudaStream_t stream) {
    if (!prompt_attention_supports(a) || a.rows < 1 || base < 0 || base + a.rows > a.rope_positions
        || a.k_new != a.q + (size_t)a.q_heads * kHd || a.v_new != a.k_new + (size_t)a.kv_heads * kHd
        || a.q_stride != a.kv_new_stride) {
        return cudaErrorInvalidValue;
    }
    PromptArgs p;
    p.qkv = const_cast<bf16*>(a.q); p.q_norm_w = a.q_norm_w; p.k_norm_w = a.k_norm_w; p.rope_table = a.rope_table;
    p.out = a.out; p.kv = a.kv; p.qkv_stride = a.q_stride; p.base = base; p.rows = a.rows;
    p.q_heads = a.q_heads; p.kv_heads = a.kv_heads; p.eps = a.eps;
    const cudaError_t e = launch_pdl(prompt_append_kernel, dim3((unsigned)a.rows), dim3(256), 0, stream, p);
    if (e != cudaSuccess) return e;
    // twice as many CTAs of half as many positions, while each has an SM of its own (two on an SM as well: a prompt of 700 positions
    // the same, of 900 0.9 % longer)
    const bool halves = a.rows > kBlockPositions / 2 && (a.rows + kBlockPositions - 1) / kBlockPositions * a.kv_heads * 2 <= kSms;
    const int block = halves ? kBlockPositions / 2 : kBlockPositions;
    const dim3 grid((unsigned)((a.rows + block - 1) / block * a.kv_heads));
    return launch_pdl(halves ? prompt_attention_kernel<kBlockPositions / 2> : prompt_attention_kernel<kBlockPositions>, grid, dim3(kFlashThreads), kFlashSmem, stream, p);
}

unsigned int prompt_attention_error_count() {
    unsigned int v = 0;
    if (cudaMemcpyFromSymbol(&v, g_prompt_attention_errors, sizeof(v)) != cudaSuccess) return ~0u;
    return v;
}

cudaError_t set_prompt_attention_error_sink(unsigned int* device_visible_word) {
    return cudaMemcpyToSymbol(g_prompt_attention_error_sink, &device_visible_word, sizeof(device_visible_word));
}

}  // namespace q3t
