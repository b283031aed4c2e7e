// Decode attention in the decode chain's order, as a launch of its own.
//
// Where a frame of up to eight sessions is made launch by launch because the GPU is shared with other frames or a
// prompt, it has to be the frame that the chain (decode_chain.cu) would have made, to the bit: which way is taken depends
// on what else runs at the moment.  Everything else of a frame is the same either way; the attention of
// decode_attention_walk_kernel merges a row in 64-token chunks, the chain in slots and classes of pages.  Here a warp is a
// class of a slot of a (row, KV head); a CTA's eight warps are as many slots as the classes in use leave room for, and the
// CTA that draws the last ticket folds the slots.
//
// What bounds it: the latency of a page (K and V are requested ahead of the dependency wait), the merges behind it and the
// ticket.  It runs beside other work, so it takes no more CTAs than it has pages for: with a slot to every CTA, six of
// eight warps idle up to 512 tokens, 16 sessions stepped alone made 758 frames/s instead of 802.

#include "q3t_attention_page.cuh"
#include "q3t_kernels.cuh"

namespace q3t {

namespace {

constexpr int kThreads = page::kClasses * kWarp;
constexpr int kPartFloats = 132;                        // maximum, sum, weighted V of a head, padded to 16 bytes

__global__ void __launch_bounds__(kThreads) attention_blocks_kernel(const AttentionArgs a) {
    __shared__ __align__(16) float queries[2 * 128];
    __shared__ __align__(16) bf16 newest[2][128];       // this step's key and value
    __shared__ __align__(16) float acc[page::kClasses * 256];
    __shared__ float m[page::kClasses * 2], l[page::kClasses * 2];
    __shared__ __align__(16) float own[page::kClasses / page::kBlock * 2 * kPartFloats];      // this CTA's slots, merged
    __shared__ int last;
    const int tid = threadIdx.x, lane = tid % kWarp, warp = tid / kWarp;
    const int kvh = blockIdx.y, row = blockIdx.z;

    // settled inputs, ahead of the wait: position, page list, older cache rows, norm weights, rotations
    int pos = a.positions[row];
    pos = min(max(pos, 0), a.rope_positions - 1);
    const int pages = pos / kPageTokens + 1, slots = page::slots_of(pages);
    // classes in use (slot 0 has the most), and what they leave room for
    int classes = page::kBlock;
    while (classes < page::kClasses && page::class_page(0, classes) < pages) classes += page::kBlock;
    const int per_cta = page::kClasses / classes;
    const int slot0 = blockIdx.x * per_cta;
    if (slot0 >= slots) {
        pdl_wait();
        return;
    }
    const int here = min(per_cta, slots - slot0);       // slots of this CTA
    const int cls = warp % classes;
    const int slot = warp / classes < here ? slot0 + warp / classes : page::kSlots;
    auto page_at = [&](int pg, bool value) {
        const int pid = a.kv.page_table[(size_t)row * a.kv.table_stride + pg];
        return a.kv.slabs[pid >> a.kv.slab_shift] + (long long)(pid & ((1 << a.kv.slab_shift) - 1)) * a.kv.page_elems
               + (value ? a.kv.v_offset : a.kv.k_offset) + (size_t)kvh * (kPageTokens * 128);
    };
    auto older_in = [&](int pg) { return min(kPageTokens, pos - pg * kPageTokens); };
    const int first = slot < slots ? page::class_page(slot, cls) : pages;
    page::Fragments f;
    bf16 *k = nullptr, *v = nullptr;
    if (first < pages) {
        k = page_at(first, false);
        v = page_at(first, true);
        page::load(f, k, v, older_in(first), lane);
    }
    bf16 w[4];
    uint32_t cs[2];
    if (warp < 3) {
        const bf16* norm = warp < 2 ? a.q_norm_w : a.k_norm_w;
#pragma unroll
        for (int j = 0; j < 4; ++j) w[j] = norm[lane + 32 * j];
        cs[0] = a.rope_table[(size_t)pos * 64 + lane];
        cs[1] = a.rope_table[(size_t)pos * 64 + lane + 32];
    }
    pdl_wait();
    pdl_trigger();
    if (warp < 3) {
        const bf16* src = warp < 2 ? a.q + (size_t)row * a.q_stride + (size_t)(2 * kvh + warp) * 128
                                   : a.k_new + (size_t)row * a.kv_new_stride + (size_t)kvh * 128;
        float x[4], o[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) x[j] = bf2f(src[lane + 32 * j]);
        page::rotate(x, w, cs[0], cs[1], a.eps, o);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (warp < 2) queries[warp * 128 + lane + 32 * j] = o[j];
            else newest[0][lane + 32 * j] = f2bf(o[j]);
        }
    } else if (warp == 3) {
        const bf16* src = a.v_new + (size_t)row * a.kv_new_stride + (size_t)kvh * 128;
#pragma unroll
        for (int j = 0; j < 4; ++j) newest[1][lane + 32 * j] = src[lane + 32 * j];
    }
    __syncthreads();
    if (first < pages) {
        const float scale = rsqrtf(128.0f);
        page::Running run;
        page::start(run);
#pragma unroll 1
        for (int pg = first; pg < pages; pg += page::kPageStep) {
            if (pg != first) {
                k = page_at(pg, false);
                v = page_at(pg, true);
                page::load(f, k, v, older_in(pg), lane);
            }
            const int t_new = pos - pg * kPageTokens;
            if (t_new < kPageTokens) {
                page::patch(f, newest[0], newest[1], t_new, lane);
                reinterpret_cast<uint2*>(k + t_new * 128)[lane] = reinterpret_cast<const uint2*>(newest[0])[lane];
                reinterpret_cast<uint2*>(v + t_new * 128)[lane] = reinterpret_cast<const uint2*>(newest[1])[lane];
            }
            float mp, lp, op[8][4];
            page::attend(f, queries, min(kPageTokens, t_new + 1), scale, lane, mp, lp, op);
            page::add(run, pg == first, mp, lp, op);
        }
        const int at = (slot - slot0) * classes + cls;
        page::put_class(run, acc + at * 256, m + at * 2, l + at * 2, lane);
    }
    __syncthreads();
    const int g = tid >> 7, d = tid & 127;
    float* parts = a.scratch + (size_t)(row * a.kv_heads + kvh) * page::kSlots * 2 * kPartFloats;
    const bool alone = here == slots;
    for (int u = 0; u < here; ++u) {
        const int at = u * classes;
        float top, sum, value;
        page::merge_classes(acc + at * 256, m + at * 2, l + at * 2, slot0 + u, pages, g, d, top, sum, value);
        float* mine = alone ? own + (u * 2 + g) * kPartFloats : parts + (size_t)((slot0 + u) * 2 + g) * kPartFloats;
        if (d == 0) {
            mine[0] = top;
            mine[1] = sum;
        }
        mine[2 + d] = value;
    }
    bf16* out = a.out + ((size_t)row * a.q_heads + 2 * kvh + g) * 128 + d;
    if (alone) {
        __syncthreads();
        *out = f2bf(page::fold([&](int u, int n) { return own[(u * 2 + g) * kPartFloats + n]; }, slots, d, lane));
        return;
    }
    __threadfence();
    __syncthreads();
    unsigned int* counter = a.counters + row * a.kv_heads + kvh;
    if (tid == 0) last = atomicAdd(counter, 1u) == (unsigned int)((slots + per_cta - 1) / per_cta - 1) ? 1 : 0;
    __syncthreads();
    if (last == 0) return;
    __threadfence();
    if (tid == 0) *counter = 0u;                        // ready for the next launch
    // read past the L1: its lines may hold a neighbour's parts from before
    *out = f2bf(page::fold([&](int u, int n) { return __ldcg(parts + (size_t)(u * 2 + g) * kPartFloats + n); }, slots, d, lane));
}

}  // namespace

size_t chain_order_scratch_floats(int rows, int kv_heads) { return (size_t)rows * kv_heads * page::kSlots * 2 * kPartFloats; }

cudaError_t launch_chain_order_attention(const AttentionArgs& a, cudaStream_t stream) {
    if (a.rows < 1 || a.rows > kChainRows || a.head_dim != 128 || a.q_heads != 2 * a.kv_heads || a.fused == 0 || a.append_mode != 0
        || a.kv.page_table == nullptr || a.kv.slabs == nullptr || a.kv.table_stride < 1 || a.rope_table == nullptr || a.rope_positions < 1
        || a.q == nullptr || a.k_new == nullptr || a.v_new == nullptr || a.q_norm_w == nullptr || a.k_norm_w == nullptr
        || a.positions == nullptr || a.out == nullptr || a.scratch == nullptr || a.counters == nullptr || a.out32 != nullptr
        || a.q_stride < 1 || a.kv_new_stride < 1) {
        return cudaErrorInvalidValue;
    }
    return launch_pdl(attention_blocks_kernel, dim3(page::kSlots, (unsigned)a.kv_heads, (unsigned)a.rows), dim3(kThreads), 0, stream, a);
}

}  // namespace q3t
