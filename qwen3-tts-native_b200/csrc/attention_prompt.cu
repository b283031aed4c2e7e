// Attention of a prompt pass: many consecutive positions of one session attend to the session's paged
// cache, each up to itself.
//
// Semantics as in attention.cu (the reference's batch_causal_gqa_attention_fast_kernel,
// native/qwen3-tts-native/native/src/talker_kernels.cu:506-595, after the per-head RMSNorm, RoPE and
// cache append of :50-70, :597-658); the decode kernel there treats every row as a session of its own
// and reads its whole context again, which for a prompt of n positions is n^2 / 2 cache rows a layer.
// Here a CTA takes 32 positions of the two query heads of a KV head (64 rows of MMA) and walks their
// common context once, 64 tokens at a time, with a running softmax.
//
// What bounds it: the chain of a step, 64 tokens' scores, softmax and products, times the steps of the longest
// context.  The probabilities go through the second product as bf16 hi + lo (16 bits kept), so a 64-row, 64-token step is
// 3 x 64 x 64 x 128 MACs: 0.9 us of an SM's mma.sync rate, 31 steps an SM for 1500 positions.  Two groups of four
// warps of 16 rows take half of every step's tokens each and meet at the end; K and V of the next step are in flight
// (cp.async, two buffers of 32 KB); two CTAs fit an SM at 128 registers (the query fragments come from shared memory).
// 1500 positions: 71 us a layer; four warps on whole steps 81, with a page lookup per token, masks on every score
// and heads one after the other 118.

#include "q3t_kernels.cuh"

namespace q3t {
namespace {

constexpr int kHd = 128;
constexpr int kBlockPositions = 32;
constexpr int kStepTokens = 64;
constexpr int kFlashThreads = 256;
constexpr int kTileBytes = kStepTokens * kHd * 2;       // 16 KB of K or V
constexpr int kFlashCtas = 2;
constexpr int kHalfTokens = kStepTokens / 2;            // of a step, to each group of four warps
constexpr size_t kFlashSmem = 5 * kTileBytes;           // two buffers of (K, V), the queries

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void mma_16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
        "{%0, %1, %2, %3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ldmatrix_x4(uint32_t addr, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t addr, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ uint32_t pack_pair(float lo, float hi) {
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}
__device__ __forceinline__ void copy16(uint32_t dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}

// 2^x, x <= 0: as exp2f, but what would be subnormal (below 2^-126 of the largest weight) is zero
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
    pdl_wait();
    pdl_trigger();
    const int t = pos % kPageTokens;
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
                bf16* kdst = page_of(a, pos, kvh, false) + (size_t)t * kHd;
                bf16* vdst = page_of(a, pos, kvh, true) + (size_t)t * kHd;
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

// 16-byte piece `piece` (0..15) of token `t` in a K or V tile: pieces are XORed with the token so that the
// eight rows of an ldmatrix fall into different banks
__device__ __forceinline__ uint32_t tile_offset(int t, int piece) { return (uint32_t)(t * 256 + ((piece ^ (t & 7)) << 4)); }

__global__ void __launch_bounds__(kFlashThreads, kFlashCtas) prompt_attention_kernel(const PromptArgs a) {
    extern __shared__ __align__(128) unsigned char smem[];
    const int tid = threadIdx.x;
    const int lane = tid % kWarp;
    const int group = tid / (kFlashThreads / 2);          // tokens 32 group .. + 31 of every step
    const int warp = tid / kWarp % 4;
    const int gid = lane >> 2;
    const int tig = lane & 3;
    // the last positions have the longest context: they go first, all KV heads of a block together
    const int kvh = (int)blockIdx.x % a.kv_heads;
    const int block = ((int)gridDim.x - 1 - (int)blockIdx.x) / a.kv_heads;
    const int row0 = block * kBlockPositions;
    const int head = kvh * 2 + (warp >> 1);
    const int my_row = row0 + (warp & 1) * 16;            // rows my_row + gid and + 8 of this lane
    const int length = a.base + min(a.rows, row0 + kBlockPositions);      // tokens the CTA walks
    const int steps = (length + kStepTokens - 1) / kStepTokens;

    pdl_wait();
    pdl_trigger();

    auto load_step = [&](int step, int buffer) {
        const uint32_t kdst = smem_addr(smem) + buffer * 2 * kTileBytes;
        // 64 tokens x 16 pieces of K and as many of V: thread t takes piece t % 16 of token t / 16 of every page
        const int piece = tid & 15;
#pragma unroll
        for (int page = 0; page < kStepTokens / kPageTokens; ++page) {
            const int t = page * kPageTokens + (tid >> 4);
            const uint32_t off = tile_offset(t, piece);
            if (step * kStepTokens + t < length) {
                const bf16* k = page_of(a, step * kStepTokens + page * kPageTokens, kvh, false) + (size_t)(tid >> 4) * kHd + piece * 8;
                copy16(kdst + off, k);
                copy16(kdst + kTileBytes + off, k + (a.kv.v_offset - a.kv.k_offset));
            } else {
                // past the end: the scores are masked, but 0 * (stale bits that decode as NaN) is not zero
                *reinterpret_cast<int4*>(smem + buffer * 2 * kTileBytes + off) = make_int4(0, 0, 0, 0);
                *reinterpret_cast<int4*>(smem + buffer * 2 * kTileBytes + kTileBytes + off) = make_int4(0, 0, 0, 0);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // the queries: row 32 head + position, as the K tiles
    {
        const uint32_t to = smem_addr(smem) + 4 * kTileBytes;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int row = (tid >> 4) + 16 * i;
            const bf16* q = a.qkv + (size_t)min(row0 + row % kBlockPositions, a.rows - 1) * a.qkv_stride
                            + (size_t)(kvh * 2 + row / kBlockPositions) * kHd;
            copy16(to + tile_offset(row, tid & 15), q + 8 * (tid & 15));
        }
    }
    load_step(0, 0);

    float o[16][4];
#pragma unroll
    for (int n = 0; n < 16; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) o[n][e] = 0.0f;
    float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.0f, 0.0f};
    // scores are kept in units of log2(e) / sqrt(128), so that exp is one exp2
    const float scale = rsqrtf(static_cast<float>(kHd)) * 1.4426950408889634f;
    const int last_lo = a.base + my_row + gid;            // the newest token each of the lane's two rows sees
    const int last_hi = last_lo + 8;

    for (int step = 0; step < steps; ++step) {
        const int buffer = step & 1;
        if (step + 1 < steps) {
            load_step(step + 1, buffer ^ 1);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();
        const uint32_t kt = smem_addr(smem) + buffer * 2 * kTileBytes + group * kHalfTokens * 256;
        const uint32_t vt = kt + kTileBytes;
        const uint32_t qt = smem_addr(smem) + 4 * kTileBytes;
        const int t0 = step * kStepTokens + group * kHalfTokens;
        // ---- scores of 16 rows x 32 tokens
        float s[4][4];
#pragma unroll
        for (int n = 0; n < 4; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) s[n][e] = 0.0f;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            // matrices: rows 16 warp .. + 7 and + 8 .. + 15, dims 16 k .. + 7, then dims 16 k + 8 .. + 15
            uint32_t qa[4];
            ldmatrix_x4(qt + tile_offset(16 * warp + (lane & 15), 2 * k + (lane >> 4)), qa);
#pragma unroll
            for (int n2 = 0; n2 < 2; ++n2) {
                // matrices: tokens 16 n2 .. + 7 and + 8 .. + 15, dims 16 k .. + 7 and + 8 .. + 15
                const int t = 16 * n2 + (lane & 7) + ((lane >> 4) << 3);
                const int piece = 2 * k + ((lane >> 3) & 1);
                uint32_t b[4];
                ldmatrix_x4(kt + tile_offset(t, piece), b);
                mma_16816(s[2 * n2], qa, b[0], b[1]);
                mma_16816(s[2 * n2 + 1], qa, b[2], b[3]);
            }
        }
        // ---- running softmax
        const bool masked = t0 + kHalfTokens - 1 > a.base + my_row;       // some row of the warp ends in this step
        if (masked) {
#pragma unroll
            for (int n = 0; n < 4; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (t0 + 8 * n + 2 * tig + (e & 1) > (e < 2 ? last_lo : last_hi)) s[n][e] = -INFINITY;
        }
        float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
        for (int n = 0; n < 4; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) mx[e >> 1] = fmaxf(mx[e >> 1], s[n][e]);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            mx[h] = fmaxf(mx[h], __shfl_xor_sync(0xffffffffu, mx[h], 1));
            mx[h] = fmaxf(mx[h], __shfl_xor_sync(0xffffffffu, mx[h], 2));
            mx[h] = fmaxf(m[h], mx[h] * scale);
        }
        if (__any_sync(0xffffffffu, mx[0] != m[0] || mx[1] != m[1])) {       // seldom, once the context is some steps long
            float f[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                // a half whose tokens so far all lie past the row has no maximum yet, and zeros to scale
                f[h] = m[h] == -INFINITY ? 0.0f : exp2_ftz(m[h] - mx[h]);
                m[h] = mx[h];
                l[h] *= f[h];
            }
#pragma unroll
            for (int n = 0; n < 16; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) o[n][e] *= f[e >> 1];
        }
#pragma unroll
        for (int n = 0; n < 4; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float pr = s[n][e] == -INFINITY ? 0.0f : exp2_ftz(fmaf(s[n][e], scale, -m[e >> 1]));
                s[n][e] = pr;
                l[e >> 1] += pr;
            }
        // ---- output: P (16 x 32) V (32 x 128), P as hi + lo
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            uint32_t hi[4], lo[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float p0 = s[2 * k + (q >> 1)][2 * (q & 1)], p1 = s[2 * k + (q >> 1)][2 * (q & 1) + 1];
                hi[q] = pack_pair(p0, p1);
                lo[q] = pack_pair(p0 - __uint_as_float(hi[q] << 16), p1 - __uint_as_float(hi[q] & 0xffff0000u));
            }
#pragma unroll
            for (int n2 = 0; n2 < 8; ++n2) {
                // matrices: tokens 16 k .. + 7 and + 8 .. + 15, dims 16 n2 .. + 7 and + 8 .. + 15
                const int t = 16 * k + (lane & 15);
                const int piece = 2 * n2 + (lane >> 4);
                uint32_t b[4];
                ldmatrix_x4_trans(vt + tile_offset(t, piece), b);
                mma_16816(o[2 * n2], hi, b[0], b[1]);
                mma_16816(o[2 * n2], lo, b[0], b[1]);
                mma_16816(o[2 * n2 + 1], hi, b[2], b[3]);
                mma_16816(o[2 * n2 + 1], lo, b[2], b[3]);
            }
        }
        __syncthreads();        // the buffer is refilled by the step after the next
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        l[h] += __shfl_xor_sync(0xffffffffu, l[h], 1);
        l[h] += __shfl_xor_sync(0xffffffffu, l[h], 2);
    }
    // ---- the two halves of every row meet: the second group's in shared memory (the last barrier of the loop has freed it)
    float* meet = reinterpret_cast<float*>(smem) + (warp * kWarp + lane);
    constexpr int kPlane = 4 * kWarp;                     // one value of every thread of a group
    if (group == 1) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            meet[h * kPlane] = m[h];
            meet[(2 + h) * kPlane] = l[h];
        }
#pragma unroll
        for (int n = 0; n < 16; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) meet[(4 + 4 * n + e) * kPlane] = o[n][e];
    }
    __syncthreads();
    if (group == 1) return;
    float inv[2], f1[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        // token 0 is visible to every row: the first group's maximum is finite
        const float m1 = meet[h * kPlane];
        const float top = fmaxf(m[h], m1);
        const float f0 = exp2_ftz(m[h] - top);
        f1[h] = exp2_ftz(m1 - top);
        inv[h] = 1.0f / (l[h] * f0 + meet[(2 + h) * kPlane] * f1[h]);
        f1[h] *= inv[h];
        inv[h] *= f0;
    }
#pragma unroll
    for (int n = 0; n < 16; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) o[n][e] = fmaf(meet[(4 + 4 * n + e) * kPlane], f1[e >> 1], o[n][e] * inv[e >> 1]);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int row = my_row + gid + 8 * h;
        if (row < a.rows) {
            bf16* dst = a.out + (size_t)row * a.q_heads * kHd + (size_t)head * kHd + 2 * tig;
#pragma unroll
            for (int n = 0; n < 16; ++n) {
                *reinterpret_cast<uint32_t*>(dst + 8 * n) = pack_pair(o[n][2 * h], o[n][2 * h + 1]);
            }
        }
    }
}

}  // namespace

cudaError_t configure_prompt_kernels() {
    return cudaFuncSetAttribute(prompt_attention_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFlashSmem);
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
    const dim3 grid((unsigned)((a.rows + kBlockPositions - 1) / kBlockPositions * a.kv_heads));
    return launch_pdl(prompt_attention_kernel, grid, dim3(kFlashThreads), kFlashSmem, stream, p);
}

}  // namespace q3t
