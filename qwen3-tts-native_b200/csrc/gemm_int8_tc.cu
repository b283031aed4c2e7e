// Skinny int8 weight-only GEMM for 9..64 activation rows, and for prompt passes of some hundred, on the 5th-generation
// tensor cores.
//
// y[r][n] = epilogue( scale[n] * sum_k W[n][k] * x[r][k] ) like the SIMT kernels, but the weights
// are the UMMA "A" operand: a CTA owns 128 output channels (one TMEM lane each) and a slice of K,
// the sessions are the UMMA "N" dimension (16, 32, 48 or 64 columns of fp32 accumulators in TMEM; prompt passes 96, 128 or
// 160: a weight is then converted once for 160 rows instead of once for 64, and K can be split where blocks of 64 filled the
// GPU.  150 rows: q/k/v 11.1 -> 9.3 us, o 8.3 -> 7.8, gate/up 18.6 -> 16.3, down 14.4 -> 11.2).
//
//   TMA, 128-byte swizzle           int8 W tile 128 x 128 -> shared ring (6 stages of 16 KB)
//   TMA, 128-byte swizzle           bf16 x tile MT x 128  -> shared ring (4 stages), UMMA K-major
//   2 x 4 warps, steps in turn      a thread owns a channel: 128 int8 of its row -> bf16 in
//                                   registers (exact: PRMT, two masks, packed subtract) ->
//                                   tcgen05.st into the TMEM columns of an A stage.  The dequantised weights never touch
//                                   shared memory, whose bandwidth bounds this kernel.
//   1 thread                        tcgen05.mma.cta_group::1.kind::f16 with A from TMEM and B
//                                   (activations) from shared memory, 128 x MT x 16 per
//                                   instruction; tcgen05.commit frees the stages
//   the same 8 warps                tcgen05.ld the accumulators, then the K-slice exchange below
//                                   and the same epilogues as the SIMT path
// K is split across the CTAs of a thread-block cluster (up to 8) so that every SM streams
// weights; each CTA pushes the rows of its slice into the shared memory of the CTA that owns
// them (asynchronous stores to distributed shared memory, counted on a barrier there), which sums the
// rows it owns over all slices in slice order (deterministic).
//
// The reference has no counterpart: its int8 path stops at 8 rows of SIMT FMAs
// (int8_gemv.cu:329) and its larger row counts go through cuBLAS bf16 GEMMs.
//
// Every wait is bounded by a wall-clock budget; a kernel that runs out records an error, lets
// its copies land, frees its TMEM columns and returns.

#include "q3t_kernels.cuh"
#include "q3t_tcgen05.cuh"

#include <cstdlib>
#include <mutex>
#include <type_traits>
#include <utility>

namespace q3t {
namespace {

using namespace tc;

// Warp roles: 0 weight copies, 1 MMA issue, 2 activation copies, 3 TMEM allocation (one elected
// thread each); 4..7 and 8..11 are the two dequantiser groups.  Warp w may touch TMEM lanes
// 32 * (w % 4) .. + 31 only, so a dequantiser owns the channel (w % 4) * 32 + lane.
constexpr int kGroups = 2;
constexpr int kTcThreads = 128 + 128 * kGroups;
constexpr int kTileN = 128;            // output channels per CTA = TMEM lanes
constexpr int kBK = 128;               // K elements per pipeline step
constexpr int kWStageBytes = kTileN * kBK;          // 16 KB
constexpr int kAStageCols = kBK / 2;   // 64 TMEM columns: two bf16 per 32-bit column
constexpr uint32_t kTmemCols = 512;
// What a tile of MT rows has.  Up to 64 rows the exchange of the K-slices has memory of its own.  Prompt passes take tiles of
// up to 160: their activations leave no room for it, and it lies over the rings, which costs a barrier of the cluster between
// the last product and the first part sent.
template <int MT>
struct Tile {
    static constexpr bool kTall = MT > 64;
    static constexpr int kWStages = MT == 160 ? 4 : 6;       // int8 ring in shared memory
    static constexpr int kStages = 4;                        // activations in shared memory; dequantised A in TMEM: stage i of one pairs with stage i of the other
    static constexpr int kAccCols = kTall ? 256 : 64;        // accumulators first, A stages behind them
    static constexpr int kXAtomBytes = MT * 128;             // MT rows x 64 bf16, one 128-byte-swizzled atom
    static constexpr int kXStageBytes = 2 * kXAtomBytes;     // 128 K elements per step
    static constexpr int kRings = kWStages * kWStageBytes + kStages * kXStageBytes;
    // up to 8 slices x ceil(MT / slices) rows, in fours, x 128 fp32
    static constexpr int kRedBytes = kTall ? 0 : 44 * 1024;
    static constexpr size_t kSmem = 1024 + (size_t)kRings + kRedBytes + (2 * kWStages + 3 * kStages + 2) * sizeof(uint64_t) + 64;
    static_assert(kWStages % kGroups == 0 && kStages % kGroups == 0, "a stage is always consumed by the same group");
    static_assert(kAccCols >= MT && kAccCols + kStages * kAStageCols <= (int)kTmemCols && kSmem <= 227 * 1024, "fits");
    static_assert(!kTall || (MT + 8 * 4) * kTileN * 4 <= kRings, "the exchange lies over the rings");
};
constexpr unsigned long long kBudgetNs = 2000000000ull;   // 2 s for the whole kernel

__device__ unsigned int g_tc_errors = 0;

__device__ unsigned int* g_tc_error_sink = nullptr;   // host-mapped word of the engine, if any

struct TcParams {
    const float* scales;
    bf16* y;
    float* y32;
    const bf16* bias;
    bf16* resid;
    int out_features;         // N (GATEUP: channels, the matrix has 2N rows)
    int rows;                 // valid sessions
    int epilogue;
    int splits;               // K-slices per channel tile = CTAs per cluster
    int chunks;               // K chunks of 64 in the whole contraction
    int tiles;
    int residual_settled;     // GemvArgs::residual_settled
};

template <int EPI>
__device__ __forceinline__ float finish(float acc, float scale, float bias, float base) {
    if (EPI == EPI_ADD) return fmaf(acc, scale, base);
    if (EPI == EPI_BIAS) return rbf(acc * scale) + bias;
    if (EPI == EPI_BIAS_SILU) {
        const float v = rbf(acc * scale) + bias;
        return __fdividef(v, 1.0f + __expf(-v));
    }
    if (EPI == EPI_BIAS_ADD) return base + rbf(rbf(acc * scale) + bias);
    return acc * scale;
}

// Everybody's products are done: what their rings held has been used.
__device__ __forceinline__ void cluster_meet() { cluster_sync(); }

__device__ __forceinline__ void dequant_barrier() {
    asm volatile("bar.sync 1, %0;" ::"n"(128 * kGroups) : "memory");
}

template <int MT, bool GATEUP>
__global__ void __launch_bounds__(kTcThreads, 1)
gemm_tc_kernel(const __grid_constant__ CUtensorMap w_map, const __grid_constant__ CUtensorMap x_map,
               const TcParams p) {
    using T = Tile<MT>;
    constexpr int kWStages = T::kWStages, kStages = T::kStages, kAccCols = T::kAccCols;
    constexpr int kXAtomBytes = T::kXAtomBytes, kXStageBytes = T::kXStageBytes;
    // fp32 accumulate, A and B bf16 (format 1), both K-major
    constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(MT >> 3) << 17)
                                | ((uint32_t)(kTileN >> 4) << 24);
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    unsigned char* w8 = smem;
    unsigned char* xs = w8 + kWStages * kWStageBytes;
    float* red = reinterpret_cast<float*>(T::kTall ? smem : smem + T::kRings);
    uint64_t* full_w = reinterpret_cast<uint64_t*>(smem + T::kRings + T::kRedBytes);
    uint64_t* empty_w = full_w + kWStages;
    uint64_t* full_a = empty_w + kWStages;
    uint64_t* empty_a = full_a + kStages;
    uint64_t* acc_done = empty_a + kStages;
    uint64_t* red_full = acc_done + 1;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(red_full + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int tid = threadIdx.x;
    const int warp = __shfl_sync(0xffffffffu, tid / kWarp, 0);      // warp-uniform by construction
    const int lane = tid % kWarp;
    const int split = (int)cluster_rank();           // cluster = the K-slices of one channel tile
    const int tile = blockIdx.x / p.splits;
    const int row_first = blockIdx.y * MT;           // activation rows of this CTA: a block of MT of them
    const int rows = min(MT, p.rows - row_first);
    const int step_first = p.chunks * split / p.splits;             // slices may differ by one step
    const int nk = p.chunks * (split + 1) / p.splits - step_first;
    const int k_first = step_first * kBK;
    const int N = p.out_features;
    // Rows a CTA owns in the K-slice sum, in groups of four; the exchange buffer is [slice][group][channel][4].
    const int share_groups = ((MT + p.splits - 1) / p.splits + 3) / 4;
    const int row0 = split * share_groups * 4;
    const int my_rows = max(0, min(share_groups * 4, rows - row0));
    const int row_a = GATEUP ? tile * 64 : tile * kTileN;          // first W row of the tile
    const int row_b = N + tile * 64;                               // GATEUP: first row of the "up" half

    // the channel this thread finishes in the K-slice sum, and its scales: asked for now, so that
    // the (cold) loads are long back when the epilogue needs them
    constexpr int kPerRow = GATEUP ? 64 : kTileN;
    const int c = tid % kPerRow;                       // kTcThreads is a multiple of kPerRow
    const int channel = tile * kPerRow + c;
    float scale = 0.0f, scale_up = 0.0f;
    if (channel < N) {
        scale = p.scales[channel];
        if (GATEUP) scale_up = p.scales[N + channel];
    }
    Guard guard;
    guard.deadline = now_ns() + kBudgetNs;
    guard.abort_flag = abort_flag;

    if (tid == 32) prefetch_map(&w_map);
    if (tid == 64) prefetch_map(&x_map);
    if (tid == 0) {
        for (int s = 0; s < kWStages; ++s) {
            mbar_init(&full_w[s], 1);
            mbar_init(&empty_w[s], 4);
        }
        for (int s = 0; s < kStages; ++s) {
            mbar_init(&full_a[s], 4 + 1);     // four dequantiser warps + the activation copy (bytes)
            mbar_init(&empty_a[s], 1);
        }
        mbar_init(acc_done, 1);
        mbar_init(red_full, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        // the other slices' parts of the rows owned here, counted in bytes (none: an arrival that completes at once)
        mbar_expect_tx(red_full, (uint32_t)((p.splits - 1) * ((my_rows + 3) / 4) * kTileN * 16));
    }
    if (warp == 3) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(tmem_slot)), "r"(kTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = *tmem_slot;
    // a peer's barriers have to be set up before anything is sent to it (tall tiles: its rings used up): waited for just
    // before that
    if (!T::kTall) cluster_arrive();
    // The weight copies (warp 0) start at once: weights never depend on the kernel before this
    // one.  Everyone else first waits for that kernel to complete (activations, residual), and
    // only then is the kernel after this one let in: every kernel of the library but the norm
    // signals its dependents after its own wait, so that a kernel may read, ahead of its wait, whatever
    // was written before the last such kernel upstream.
    // The dequantisers (warps 4..) touch only weights and tensor memory until the K-slice sum, so
    // they too run ahead and wait there.
    if (warp >= 1 && warp <= 3) {
        pdl_wait();
        if (warp == 1) pdl_trigger();
    }

    if (warp == 0) {
        if (elect_one()) {
            // ---- weight producer ----------------------------------------------------------
            for (int i = 0; i < nk; ++i) {
                const int s = i % kWStages;
                if (i >= kWStages && !guard.wait(&empty_w[s], ((i / kWStages) - 1) & 1)) break;
                mbar_expect_tx(&full_w[s], kWStageBytes);
                unsigned char* dst = w8 + s * kWStageBytes;
                if (GATEUP) {
                    tma_load_2d(dst, &w_map, k_first + i * kBK, row_a, &full_w[s]);
                    tma_load_2d(dst + kWStageBytes / 2, &w_map, k_first + i * kBK, row_b, &full_w[s]);
                } else {
                    tma_load_2d(dst, &w_map, k_first + i * kBK, row_a, &full_w[s]);
                }
            }
        }
    } else if (warp == 2) {
        if (elect_one()) {
            // ---- activation producer ------------------------------------------------------
            for (int i = 0; i < nk; ++i) {
                const int sx = i % kStages;
                if (i >= kStages && !guard.wait(&empty_a[sx], ((i / kStages) - 1) & 1)) break;
                // the activation tile lands on the same barrier the dequantisers arrive on, so
                // that the MMA issuer has one thing to wait for per step
                mbar_expect_tx(&full_a[sx], kXStageBytes);
                unsigned char* dst = xs + sx * kXStageBytes;
                tma_load_2d(dst, &x_map, k_first + i * kBK, row_first, &full_a[sx]);
                tma_load_2d(dst + kXAtomBytes, &x_map, k_first + i * kBK + 64, row_first, &full_a[sx]);
            }
        }
    } else if (warp == 1) {
        if (elect_one()) {
            // ---- MMA issuer ---------------------------------------------------------------
            for (int i = 0; i < nk; ++i) {
                const int sa = i % kStages;
                if (!guard.wait(&full_a[sa], (i / kStages) & 1)) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t a_col = tmem_base + kAccCols + sa * kAStageCols;
                const uint32_t b_addr = smem_u32(xs + sa * kXStageBytes);
#pragma unroll
                for (int j = 0; j < kBK / 16; ++j) {
                    // 16 K elements = 8 TMEM columns of A, 32 bytes within a row of the B atom
                    umma_f16_ts(tmem_base, a_col + 8 * j,
                                umma_desc(b_addr + (j / 4) * kXAtomBytes + 32 * (j % 4)), kIdesc,
                                (i | j) != 0 ? 1u : 0u);
                }
                umma_commit(&empty_a[sa]);       // frees the TMEM stage and the activation stage
            }
            umma_commit(acc_done);   // fires when every MMA issued above has completed
        }
    } else if (warp >= 4) {
        // ---- dequantisers, then accumulator readers -----------------------------------------
        const int group = (warp - 4) / 4;            // steps group, group + kGroups, ...
        const int t = (warp % 4) * 32 + lane;        // channel within the tile = TMEM lane
        const uint32_t lane_base = tmem_base + ((uint32_t)((warp % 4) * 32) << 16);
        bool ok = true;
        for (int i = group; i < nk && ok; i += kGroups) {
            const int s = i % kWStages;
            const int sa = i % kStages;
            // a wait that gives up does so for the whole warp: the warp-level syncs below must be
            // reached by all 32 lanes or by none
            if (!__all_sync(0xffffffffu, guard.wait(&full_w[s], (i / kWStages) & 1))) { ok = false; break; }
            // this thread's row: 128 bytes, whose 16-byte pieces sit at piece ^ (row & 7)
            const unsigned char* rowp = w8 + s * kWStageBytes + t * 128;
            int4 raw[8];
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                raw[c] = *reinterpret_cast<const int4*>(rowp + ((c ^ (t & 7)) << 4));
            }
            if (i >= kStages
                && !__all_sync(0xffffffffu, guard.wait(&empty_a[sa], ((i / kStages) - 1) & 1))) {
                ok = false;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                uint32_t out[32];
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const int4 v = raw[4 * h + c];
                    dequant4(static_cast<uint32_t>(v.x), out[8 * c + 0], out[8 * c + 1]);
                    dequant4(static_cast<uint32_t>(v.y), out[8 * c + 2], out[8 * c + 3]);
                    dequant4(static_cast<uint32_t>(v.z), out[8 * c + 4], out[8 * c + 5]);
                    dequant4(static_cast<uint32_t>(v.w), out[8 * c + 6], out[8 * c + 7]);
                }
                tmem_store_32(lane_base + kAccCols + sa * kAStageCols + 32 * h, out);
            }
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&full_a[sa]);
                mbar_arrive(&empty_w[s]);
            }
        }
        if (ok) ok = guard.wait(acc_done, 0);
        if (!ok) *abort_flag = 1;
        // all accumulator readers meet here, so that they agree on whether the tile is complete
        dequant_barrier();
        if (__all_sync(0xffffffffu, *abort_flag == 0)) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            // each group takes half of the accumulator columns (= activation rows), some at a time; every row of
            // this K-slice goes to the shared memory of the CTA that owns the row
            constexpr int kCols = MT / kGroups, kChunk = T::kTall ? 16 : kCols;
            float v[kChunk];
            tmem_load_row<kChunk>(lane_base + group * kCols, v);
            if (T::kTall) cluster_meet();
            else cluster_wait();
            const uint32_t mine = smem_u32(red) + (uint32_t)((split * share_groups * kTileN + t) * 16);
            int owner = (group * kCols / 4) / share_groups;      // one division, then counted up
            int within = group * kCols / 4 - owner * share_groups;
#pragma unroll 1
            for (int j0 = 0; j0 < kCols; j0 += kChunk) {
                if (j0 > 0) tmem_load_row<kChunk>(lane_base + group * kCols + j0, v);
#pragma unroll
                for (int j = 0; j < kChunk; j += 4) {
                    if (group * kCols + j0 + j < rows) {
                        const uint32_t at = mine + (uint32_t)(within * kTileN * 16);
                        if (owner == split) {
                            *reinterpret_cast<float4*>(reinterpret_cast<unsigned char*>(red) + (at - smem_u32(red)))
                                = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
                        } else {
                            st_async_v4(peer_smem(at, (uint32_t)owner), v[j], v[j + 1], v[j + 2], v[j + 3],
                                        peer_smem(smem_u32(red_full), (uint32_t)owner));
                        }
                    }
                    if (++within == share_groups) {
                        within = 0;
                        ++owner;
                    }
                }
            }
        } else if (T::kTall) {
            cluster_meet();
        } else {
            cluster_wait();
        }
    }
    if (warp < 4) {
        __syncwarp();
        if (T::kTall) cluster_meet();
        else cluster_wait();
    }

    // ---- the K-slices of a channel tile live in the CTAs of one cluster; each CTA sums the rows it owns over all slices
    // in slice order, a thread four rows of a channel.  The slices' parts arrive as asynchronous stores counted on a barrier
    // here: one way across the cluster, where a cluster barrier behind plain stores was three.
    // The values a residual epilogue adds to, requested before the wait hides their
    // latency (and, when their writer is known to be long done, before the dependency wait).
    constexpr int kStride = kTcThreads / kPerRow;      // row groups at a time
    constexpr int kBasePre = 2;
    float base_pre[kBasePre][4];
    const bool base_wanted = !GATEUP && channel < N && (p.epilogue == EPI_ADD || p.epilogue == EPI_BIAS_ADD);
    const bf16* base_src = p.epilogue == EPI_ADD ? p.y : p.resid;
    auto fetch_bases = [&]() {
#pragma unroll
        for (int u = 0; u < kBasePre; ++u)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int j = 4 * (tid / kPerRow + u * kStride) + e;
                base_pre[u][e] = j < my_rows ? bf2f(base_src[(size_t)(row_first + row0 + j) * N + channel]) : 0.0f;
            }
    };
    if (base_wanted && p.residual_settled != 0) fetch_bases();
    if (warp == 0 || warp >= 4) pdl_wait();
    if (base_wanted && p.residual_settled == 0) fetch_bases();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();                                   // this slice's own part
    if (*abort_flag == 0 && !guard.wait(red_full, 0)) *abort_flag = 1;
    if (*abort_flag == 0 && channel < N) {
        bf16* dst = (!GATEUP && p.epilogue == EPI_BIAS_ADD ? p.resid : p.y) + (size_t)(row_first + row0) * N + channel;
        // one loop per epilogue: what a row costs here is instructions behind the last wait of the launch
        auto finish_rows = [&](auto which) {
            constexpr int EPI = decltype(which)::value;
            const float bias = EPI == EPI_BIAS || EPI == EPI_BIAS_SILU || EPI == EPI_BIAS_ADD ? bf2f(p.bias[channel]) : 0.0f;
            int u = 0;
            for (int g = tid / kPerRow; 4 * g < my_rows; g += kStride, ++u) {
                const float4* at = reinterpret_cast<const float4*>(red) + g * kTileN + c;
                float acc[4], acc_up[4];
#pragma unroll
                for (int sp = 0; sp < 8; ++sp) {
                    if (sp < p.splits) {
                        const float4 part = at[sp * share_groups * kTileN];
                        const float a4[4] = {part.x, part.y, part.z, part.w};
#pragma unroll
                        for (int e = 0; e < 4; ++e) acc[e] = sp == 0 ? a4[e] : acc[e] + a4[e];
                        if (GATEUP) {
                            const float4 part_up = at[sp * share_groups * kTileN + 64];
                            const float u4[4] = {part_up.x, part_up.y, part_up.z, part_up.w};
#pragma unroll
                            for (int e = 0; e < 4; ++e) acc_up[e] = sp == 0 ? u4[e] : acc_up[e] + u4[e];
                        }
                    }
                }
                bf16* row = dst + (size_t)(4 * g) * N;
                float base[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    base[e] = u == 0 ? base_pre[0][e] : base_pre[1][e];
                    if ((EPI == EPI_ADD || EPI == EPI_BIAS_ADD) && u >= kBasePre && 4 * g + e < my_rows) base[e] = bf2f(row[(size_t)e * N]);
                }
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    float val;
                    if (GATEUP) {
                        const float gate = acc[e] * scale;
                        // hardware exp2/reciprocal (good to about 2^-21); this path is compared at bf16 tolerance
                        val = __fdividef(gate, 1.0f + __expf(-gate)) * (acc_up[e] * scale_up);
                    } else {
                        val = finish<EPI>(acc[e], scale, bias, base[e]);
                    }
                    if (4 * g + e < my_rows) {
                        if (p.y32 != nullptr) p.y32[(size_t)(row_first + row0 + 4 * g + e) * N + channel] = val;
                        row[(size_t)e * N] = f2bf(val);
                    }
                }
            }
        };
        if (GATEUP) {
            finish_rows(std::integral_constant<int, EPI_GATE_UP_SILU>());
        } else {
            switch (p.epilogue) {
                case EPI_ADD: finish_rows(std::integral_constant<int, EPI_ADD>()); break;
                case EPI_BIAS: finish_rows(std::integral_constant<int, EPI_BIAS>()); break;
                case EPI_BIAS_SILU: finish_rows(std::integral_constant<int, EPI_BIAS_SILU>()); break;
                case EPI_BIAS_ADD: finish_rows(std::integral_constant<int, EPI_BIAS_ADD>()); break;
                default: finish_rows(std::integral_constant<int, EPI_PLAIN>()); break;
            }
        }
    }
    __syncthreads();
    if (*abort_flag) {
        // give copies that are still in flight time to land before the CTA's memory is released
        if (tid == 0) {
            atomicAdd(&g_tc_errors, 1u);
            if (g_tc_error_sink != nullptr) atomicAdd_system(g_tc_error_sink, 1u);
        }
        const unsigned long long until = now_ns() + 200000ull;
        while (now_ns() < until) __nanosleep(1000);
        __syncthreads();
        // a slice that is merely late may still send here: stay until it has ended, well or not
        cluster_sync();
    }
    if (warp == 3) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols)
                     : "memory");
    }
}

// ---------------------------------------------------------------------------------- host side

// Rows of a tile.  Over 64: prompt passes only.
constexpr int kTileRows[] = {16, 32, 48, 64, 96, 128, 160};
constexpr int kVariants = sizeof(kTileRows) / sizeof(kTileRows[0]);
int variant_of(int mt) {
    for (int i = 0; i < kVariants; ++i)
        if (kTileRows[i] == mt) return i;
    return -1;
}

// Per-device scratch of the tensor-core path: a buffer for normalised activations.  Allocated
// once per device by configure_tc_kernels(); launches on one device that use it must be ordered
// (the engine issues them on one stream).
struct TcScratch {
    bf16* normalized = nullptr;
    int sms = 148;
    // clusters of 1..8 CTAs that the device can hold at once, per kernel variant [index in kTileRows][GATEUP]
    int resident_clusters[kVariants][2][9] = {};
    bool ready = false;
};
constexpr size_t kNormalizedElems = (size_t)kMaxRows * 8192;
TcScratch g_scratch[64];
std::mutex g_scratch_guard;

TcScratch* scratch_for_current_device() {
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= 64) return nullptr;
    return g_scratch[device].ready ? &g_scratch[device] : nullptr;
}

template <int MT, bool GATEUP>
cudaError_t configure_one(int (&resident)[9]) {
    cudaError_t e = cudaFuncSetAttribute(gemm_tc_kernel<MT, GATEUP>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(Tile<MT>::kSmem));
    for (int size = 1; size <= 8 && e == cudaSuccess; ++size) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)(size * 64), 1, 1);
        cfg.blockDim = dim3(kTcThreads, 1, 1);
        cfg.dynamicSmemBytes = Tile<MT>::kSmem;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = (unsigned)size;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        int clusters = 0;
        e = cudaOccupancyMaxActiveClusters(&clusters, gemm_tc_kernel<MT, GATEUP>, &cfg);
        resident[size] = clusters;
    }
    return e;
}

template <int MT, bool GATEUP>
cudaError_t launch_mt(const CUtensorMap& wm, const CUtensorMap& xm, const TcParams& p, cudaStream_t stream) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(p.tiles * p.splits), (unsigned)((p.rows + MT - 1) / MT), 1);
    cfg.blockDim = dim3(kTcThreads, 1, 1);
    cfg.dynamicSmemBytes = Tile<MT>::kSmem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)p.splits;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = pdl_enabled() ? 1 : 0;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    return cudaLaunchKernelEx(&cfg, gemm_tc_kernel<MT, GATEUP>, wm, xm, p);
}

template <int... MTS>
cudaError_t configure_all(TcScratch& s, std::integer_sequence<int, MTS...>) {
    cudaError_t e = cudaSuccess;
    int v = 0;
    ((e = e == cudaSuccess ? configure_one<MTS, false>(s.resident_clusters[v][0]) : e,
      e = e == cudaSuccess ? configure_one<MTS, true>(s.resident_clusters[v][1]) : e, ++v), ...);
    return e;
}
template <bool GATEUP>
cudaError_t launch_tile(int mt, const CUtensorMap& wm, const CUtensorMap& xm, const TcParams& p, cudaStream_t stream) {
    switch (mt) {
        case 16: return launch_mt<16, GATEUP>(wm, xm, p, stream);
        case 32: return launch_mt<32, GATEUP>(wm, xm, p, stream);
        case 48: return launch_mt<48, GATEUP>(wm, xm, p, stream);
        case 96: return launch_mt<96, GATEUP>(wm, xm, p, stream);
        case 128: return launch_mt<128, GATEUP>(wm, xm, p, stream);
        case 160: return launch_mt<160, GATEUP>(wm, xm, p, stream);
        default: return launch_mt<64, GATEUP>(wm, xm, p, stream);
    }
}

int g_tc_min_rows = 9;

}  // namespace

void set_tc_min_rows(int rows) { g_tc_min_rows = rows < 2 ? 2 : rows; }
int tc_min_rows() { return g_tc_min_rows; }

cudaError_t configure_tc_kernels() {
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return e;
    if (device < 0 || device >= 64) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lock(g_scratch_guard);
    TcScratch& s = g_scratch[device];
    if (s.ready) return cudaSuccess;
    e = configure_all(s, std::integer_sequence<int, 16, 32, 48, 64, 96, 128, 160>());
    if (e != cudaSuccess) return e;
    e = cudaMalloc(&s.normalized, kNormalizedElems * sizeof(bf16));
    if (e != cudaSuccess) return e;
    int sms = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) == cudaSuccess && sms > 0) s.sms = sms;
    s.ready = encode_tiled() != nullptr;
    return s.ready ? cudaSuccess : cudaErrorNotSupported;
}

bool gemm_tc_supports(const GemvArgs& a) {
    if (a.rows < g_tc_min_rows || a.rows > kMaxPromptRows) return false;
    if (a.in_features % kBK != 0 || a.in_features > 8192) return false;
    if ((reinterpret_cast<uintptr_t>(a.w) & 15u) != 0 || (reinterpret_cast<uintptr_t>(a.x) & 15u) != 0) return false;
    return scratch_for_current_device() != nullptr;
}

namespace {
// The smallest tile that takes the rows at once, or in as many blocks as tiles of 64 would: activations and exchange
// cost what the tile has, used or not (16 projections of 48 rows: 128.4 us by a tile of 64, 124.0 by one of 48).
int tile_rows(int rows) {
    if (rows <= 48) return (rows + 15) / 16 * 16;
    return rows <= (rows + 63) / 64 * 48 ? 48 : 64;
}
// K-slices per tile = cluster size: as many as still let every cluster be resident at once (a second wave would
// double the time); slices and row shares may be ragged
int choose_splits(const TcScratch& scratch, const GemvArgs& a, int mt) {
    const bool gateup = a.epilogue == EPI_GATE_UP_SILU;
    const int nk = a.in_features / kBK;
    const int clusters = (gateup ? (a.out_features + 63) / 64 : (a.out_features + kTileN - 1) / kTileN) * ((a.rows + mt - 1) / mt);
    const int (&resident)[9] = scratch.resident_clusters[variant_of(mt)][gateup ? 1 : 0];
    static const int split_cap = [] {
        const char* v = std::getenv("QWEN3_TTS_TC_MAX_SPLITS");
        const int n = v != nullptr ? std::atoi(v) : 8;
        return n < 1 ? 1 : (n > 8 ? 8 : n);
    }();
    int splits = 1;
    for (int s = 2; s <= split_cap && s <= nk; ++s) {
        // (as few as have the longest slice this short: each one more is another part to exchange)
        if (clusters <= resident[s] && (nk + s - 1) / s < (nk + splits - 1) / splits) splits = s;
    }
    return splits;
}
}  // namespace

int gemm_tc_tile(int rows) { return tile_rows(rows); }
int gemm_tc_slices(int out_features, int in_features, int rows, bool gate_up) {
    TcScratch* scratch = scratch_for_current_device();
    if (scratch == nullptr || rows < g_tc_min_rows || in_features % kBK != 0) return 0;
    GemvArgs a;
    a.out_features = out_features; a.in_features = in_features; a.rows = rows; a.epilogue = gate_up ? EPI_GATE_UP_SILU : EPI_PLAIN;
    return choose_splits(*scratch, a, tile_rows(rows));
}

float gemm_tc_estimate_us(const GemvArgs& a, int tile) {
    TcScratch* scratch = scratch_for_current_device();
    if (scratch == nullptr || a.in_features % kBK != 0) return 1.0e9f;
    const bool gateup = a.epilogue == EPI_GATE_UP_SILU;
    const int mt = tile > 0 ? tile : tile_rows(a.rows), splits = choose_splits(*scratch, a, mt);
    const int ctas = (gateup ? (a.out_features + 63) / 64 : (a.out_features + kTileN - 1) / kTileN) * ((a.rows + mt - 1) / mt) * splits;
    const int waves = (ctas + scratch->sms - 1) / scratch->sms;
    const int steps = (a.in_features / kBK + splits - 1) / splits;
    if (mt <= 64) return waves * (splits > 1 ? 5.3f + 0.39f * steps : 4.5f + 0.43f * steps);
    // tall tiles: the exchange and the epilogue grow with the rows; a residual is another read of them
    const bool adds = a.epilogue == EPI_ADD || a.epilogue == EPI_BIAS_ADD;
    return waves * ((adds || gateup ? 3.0f : 2.1f) + 0.0385f * mt + 0.42f * steps);
}

cudaError_t launch_int8_gemm_tc(const GemvArgs& a, cudaStream_t stream, int tile) {
    TcScratch* scratch = scratch_for_current_device();
    if (scratch == nullptr || (tile > 0 && variant_of(tile) < 0) || !gemm_tc_supports(a) || a.out_features < 1 || a.w == nullptr
        || a.scales == nullptr || a.x == nullptr) {
        return cudaErrorInvalidValue;
    }
    const bool gateup = a.epilogue == EPI_GATE_UP_SILU;
    if (a.epilogue == EPI_BIAS_ADD ? (a.resid == nullptr) : (a.y == nullptr)) return cudaErrorInvalidValue;
    if ((a.epilogue == EPI_BIAS || a.epilogue == EPI_BIAS_SILU || a.epilogue == EPI_BIAS_ADD)
        && a.bias == nullptr) {
        return cudaErrorInvalidValue;
    }
    const int K = a.in_features;
    const int N = a.out_features;
    const bf16* x = a.x;
    if (a.norm_w != nullptr) {
        // RMSNorm as its own launch here: at 9+ rows one more launch is noise, and every CTA of the
        // GEMM reads the normalised rows
        bf16* normalized = a.norm_out != nullptr ? a.norm_out : scratch->normalized;
        if (a.norm_out == nullptr && (size_t)a.rows * K > kNormalizedElems) return cudaErrorInvalidValue;
        const cudaError_t e = launch_rms_norm_rows(a.x, a.norm_w, normalized, a.rows, K, a.eps, stream);
        if (e != cudaSuccess) return e;
        x = normalized;
    }
    const int mt = tile > 0 ? tile : tile_rows(a.rows);
    TcParams p;
    p.scales = a.scales; p.y = a.y; p.y32 = a.y32; p.bias = a.bias; p.resid = a.resid;
    p.out_features = N; p.rows = a.rows; p.epilogue = a.epilogue;
    p.tiles = gateup ? (N + 63) / 64 : (N + kTileN - 1) / kTileN;
    p.residual_settled = a.residual_settled ? 1 : 0;
    const int nk = K / kBK;
    p.splits = choose_splits(*scratch, a, mt);
    p.chunks = nk;

    alignas(64) CUtensorMap wm, xm;
    const uint64_t w_rows = gateup ? 2ull * N : (uint64_t)N;
    if (!make_map(&wm, CU_TENSOR_MAP_DATA_TYPE_UINT8, a.w, K, w_rows, K, kBK, gateup ? 64 : kTileN,
                  CU_TENSOR_MAP_SWIZZLE_128B)
        || !make_map(&xm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, x, K, a.rows, (uint64_t)K * 2, 64, mt,
                     CU_TENSOR_MAP_SWIZZLE_128B)) {
        return cudaErrorInvalidValue;
    }
    return gateup ? launch_tile<true>(mt, wm, xm, p, stream) : launch_tile<false>(mt, wm, xm, p, stream);
}

unsigned int gemm_tc_error_count() {
    unsigned int v = 0;
    if (cudaMemcpyFromSymbol(&v, g_tc_errors, sizeof(v)) != cudaSuccess) return ~0u;
    return v;
}

cudaError_t set_tc_error_sink(unsigned int* device_visible_word) {
    return cudaMemcpyToSymbol(g_tc_error_sink, &device_visible_word, sizeof(device_visible_word));
}

}  // namespace q3t
