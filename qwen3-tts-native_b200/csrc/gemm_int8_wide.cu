// Int8 weight-only GEMM for the passes of a prompt: 65 to 2048 activation rows on the 5th-generation
// tensor cores.
//
// Same operation and epilogues as gemm_int8_tc.cu, without its split of K: there are enough output
// tiles here to fill the GPU.  A CTA owns NT tiles of 128 output channels (TMEM lanes) by 128
// activation rows (TMEM columns).
//
// What bounds it: the way of a step through conversion, tensor memory and products.  A step of 128 x 128 weights is 512 cycles of
// products and some 500 of integer instructions on every scheduler; it takes 0.32 us with NT = 2 and 0.46 with NT = 1, of one CTA
// alone as of 148.  The issuing thread does not look at barriers (await_step), and weights are converted ahead of the wait for
// their place (1,500 rows of down 48 -> 41 us, gate/up 75.5 -> 69, q/k/v 37 -> 34).  NT = 2 has its activations once for two steps;
// NT = 1 has more CTAs, for passes of few rows.
// The two tiles of a gate/up projection are the gate rows and the up rows of the same 128 channels, so
// that a thread finds both values of a channel in its own TMEM lane; with NT = 1 a tile holds 64 of
// each and the up half crosses over through shared memory.
//
// Warp roles as in gemm_int8_tc.cu: 0 weight copies, 1 MMA issue, 2 activation copies, 3 TMEM; 4..19 in four
// groups dequantise (a thread turns 128 int8 of its channel into bf16 and stores them to tensor memory as the
// A operand), then read the accumulators; 3 is also the look-out for steps whose operands are all there.  Every wait is bounded.

#include "q3t_kernels.cuh"
#include "q3t_tcgen05.cuh"

namespace q3t {
namespace {

using namespace tc;

constexpr int kGroups = 4;
constexpr int kThreads = 128 + 128 * kGroups;
constexpr int kTileN = 128;                   // channels per tile
constexpr int kTileM = 128;                   // activation rows per CTA
constexpr int kBK = 128;                      // K elements per step
constexpr int kSms = 148;
constexpr int kTallRowsMost = 640;            // see launch_int8_gemm_prompt
constexpr int kWStages = 8;
constexpr int kXStages = 3;
constexpr int kAStages = 4;
// A slot's fills must be consumed by one group: copies may land out of order, and a group that waits for a fill two
// phases ahead of the one in flight would read its parity as already complete.
static_assert(kWStages % kGroups == 0 && kAStages % kGroups == 0, "one group per stage");
constexpr int kWStageBytes = kTileN * kBK;            // 16 KB
constexpr int kXAtomBytes = kTileM * 128;             // 128 rows x 64 bf16
constexpr int kXStageBytes = 2 * kXAtomBytes;         // 32 KB
constexpr int kAStageCols = kBK / 2;
constexpr int kAStageBase = 256;                      // accumulators in columns [0, 256)
constexpr uint32_t kTmemCols = 512;
constexpr unsigned long long kBudgetNs = 2000000000ull;
constexpr size_t kSmemBytes = 1024 + (size_t)kWStages * kWStageBytes + (size_t)kXStages * kXStageBytes
    + (2 * kWStages + 2 * kXStages + 2 * kAStages + 1) * sizeof(uint64_t) + 64;

__device__ unsigned int g_wide_errors = 0;
__device__ unsigned int* g_wide_error_sink = nullptr;

struct WideParams {
    const float* scales;
    bf16* y;
    const bf16* bias;
    bf16* resid;
    int out_features;       // N (gate/up: channels, the matrix has 2N rows)
    int rows;
    int row_blocks;
    int steps;              // K / kBK
    int epilogue;
};

__device__ __forceinline__ void readers_barrier() {
    asm volatile("bar.sync 1, %0;" ::"n"(128 * kGroups) : "memory");
}

template <int NT, bool GATEUP>
__global__ void __launch_bounds__(kThreads, 1)
gemm_wide_kernel(const __grid_constant__ CUtensorMap w_map, const __grid_constant__ CUtensorMap x_map,
                 const WideParams p) {
    constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kTileM >> 3) << 17)
                                | ((uint32_t)(kTileN >> 4) << 24);
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    unsigned char* w8 = smem;
    unsigned char* xs = w8 + kWStages * kWStageBytes;
    uint64_t* full_w = reinterpret_cast<uint64_t*>(xs + kXStages * kXStageBytes);
    uint64_t* empty_w = full_w + kWStages;
    uint64_t* full_x = empty_w + kWStages;
    uint64_t* empty_x = full_x + kXStages;
    uint64_t* full_a = empty_x + kXStages;
    uint64_t* empty_a = full_a + kAStages;
    uint64_t* acc_done = empty_a + kAStages;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_done + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    uint32_t* steps_ready = tmem_slot + 2;

    const int tid = threadIdx.x;
    const int warp = __shfl_sync(0xffffffffu, tid / kWarp, 0);
    const int lane = tid % kWarp;
    // row blocks fastest: the CTAs in flight share few weight tiles and all of the activations
    const int tile = blockIdx.x / p.row_blocks;
    const int row_base = (blockIdx.x % p.row_blocks) * kTileM;
    const int N = p.out_features;
    const int nk = p.steps;
    constexpr int kChannels = GATEUP ? (NT == 2 ? 128 : 64) : NT * kTileN;    // output channels of the CTA

    Guard guard;
    guard.deadline = now_ns() + kBudgetNs;
    guard.abort_flag = abort_flag;

    if (tid == 0) {
        for (int s = 0; s < kWStages; ++s) {
            mbar_init(&full_w[s], 1);
            mbar_init(&empty_w[s], 4);
        }
        for (int s = 0; s < kXStages; ++s) {
            mbar_init(&full_x[s], 1);
            mbar_init(&empty_x[s], 1);
        }
        for (int s = 0; s < kAStages; ++s) {
            mbar_init(&full_a[s], 4);
            mbar_init(&empty_a[s], 1);
        }
        mbar_init(acc_done, 1);
        *abort_flag = 0;
        *steps_ready = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
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
    // weights never depend on the launch before; activations, residuals and outputs do
    if (warp >= 1 && warp <= 3) {
        pdl_wait();
        if (warp == 1) pdl_trigger();
    }

    if (warp == 0) {
        if (elect_one()) {
            for (int item = 0; item < nk * NT; ++item) {
                const int s = item % kWStages;
                if (item >= kWStages && !guard.wait(&empty_w[s], ((item / kWStages) - 1) & 1)) break;
                mbar_expect_tx(&full_w[s], kWStageBytes);
                unsigned char* dst = w8 + s * kWStageBytes;
                const int k = (item / NT) * kBK;
                const int u = item % NT;
                if (GATEUP && NT == 1) {
                    tma_load_2d(dst, &w_map, k, tile * 64, &full_w[s]);
                    tma_load_2d(dst + kWStageBytes / 2, &w_map, k, N + tile * 64, &full_w[s]);
                } else if (GATEUP) {
                    tma_load_2d(dst, &w_map, k, u * N + tile * kTileN, &full_w[s]);
                } else {
                    tma_load_2d(dst, &w_map, k, (tile * NT + u) * kTileN, &full_w[s]);
                }
            }
        }
    } else if (warp == 2) {
        if (elect_one()) {
            for (int i = 0; i < nk; ++i) {
                const int s = i % kXStages;
                if (i >= kXStages && !guard.wait(&empty_x[s], ((i / kXStages) - 1) & 1)) break;
                mbar_expect_tx(&full_x[s], kXStageBytes);
                unsigned char* dst = xs + s * kXStageBytes;
                tma_load_2d(dst, &x_map, i * kBK, row_base, &full_x[s]);
                tma_load_2d(dst + kXAtomBytes, &x_map, i * kBK + 64, row_base, &full_x[s]);
            }
        }
    } else if (warp == 1) {
        if (elect_one()) {
            bool ok = true;
            uint32_t seen = 0;
            for (int i = 0; i < nk && ok; ++i) {
                const int sx = i % kXStages;
                const uint32_t b_addr = smem_u32(xs + sx * kXStageBytes);
#pragma unroll
                for (int u = 0; u < NT; ++u) {
                    const int item = i * NT + u;
                    const int sa = item % kAStages;
                    ok = ok && await_step(guard, steps_ready, (uint32_t)item, seen);
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t a_col = tmem_base + kAStageBase + sa * kAStageCols;
#pragma unroll
                    for (int j = 0; j < kBK / 16; ++j) {
                        umma_f16_ts(tmem_base + u * kTileM, a_col + 8 * j,
                                    umma_desc(b_addr + (j / 4) * kXAtomBytes + 32 * (j % 4)), kIdesc,
                                    (i | j) != 0 ? 1u : 0u);
                    }
                    umma_commit(&empty_a[sa]);
                }
                if (ok) umma_commit(&empty_x[sx]);
            }
            umma_commit(acc_done);
        }
    } else if (warp == 3) {
        if (elect_one()) {
            for (int item = 0; item < nk * NT; ++item) {
                const int i = item / NT;
                if (item % NT == 0 && !guard.wait(&full_x[i % kXStages], (i / kXStages) & 1)) break;
                if (!guard.wait(&full_a[item % kAStages], (item / kAStages) & 1)) break;
                publish_steps(steps_ready, (uint32_t)item + 1);
            }
        }
    } else if (warp >= 4) {
        const int group = (warp - 4) / 4;
        const int t = (warp % 4) * 32 + lane;        // channel within the tile = TMEM lane
        const uint32_t lane_base = tmem_base + ((uint32_t)((warp % 4) * 32) << 16);
        bool ok = true;
        for (int item = group; item < nk * NT && ok; item += kGroups) {
            const int s = item % kWStages;
            const int sa = item % kAStages;
            if (!__all_sync(0xffffffffu, guard.wait(&full_w[s], (item / kWStages) & 1))) { ok = false; break; }
            const unsigned char* rowp = w8 + s * kWStageBytes + t * 128;
            // converted ahead of the wait for its place: what the place still holds is being multiplied meanwhile
            uint32_t out[2][32];
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                const int4 v = *reinterpret_cast<const int4*>(rowp + ((c ^ (t & 7)) << 4));
                uint32_t* to = out[c / 4] + 8 * (c & 3);
                dequant4(static_cast<uint32_t>(v.x), to[0], to[1]);
                dequant4(static_cast<uint32_t>(v.y), to[2], to[3]);
                dequant4(static_cast<uint32_t>(v.z), to[4], to[5]);
                dequant4(static_cast<uint32_t>(v.w), to[6], to[7]);
            }
            compute_now(out[0]);
            compute_now(out[1]);
            if (item >= kAStages && !__all_sync(0xffffffffu, guard.wait(&empty_a[sa], ((item / kAStages) - 1) & 1))) {
                ok = false;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            tmem_store_32(lane_base + kAStageBase + sa * kAStageCols, out[0]);
            tmem_store_32(lane_base + kAStageBase + sa * kAStageCols + 32, out[1]);
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&full_a[sa]);
                mbar_arrive(&empty_w[s]);
            }
        }
        // Group g finishes the activation rows [32 g, 32 g + 32) of the CTA; a thread has one channel of each tile.  What a
        // residual epilogue adds to is requested a tile's 32 rows at a time, the first before the last MMAs are waited for.
        constexpr int kShare = kTileM / kGroups;
        const int first_row = row_base + group * kShare;
        const int rows_here = min(kShare, p.rows - first_row);
        const bool up_lane = GATEUP && NT == 1 && t >= 64;
        const bool adds = !GATEUP && (p.epilogue == EPI_ADD || p.epilogue == EPI_BIAS_ADD);
        bf16* out = (p.epilogue == EPI_BIAS_ADD ? p.resid : p.y) + (size_t)first_row * N;
        bf16 base[kShare];
        auto fetch_bases = [&](int channel) {
#pragma unroll
            for (int j = 0; j < kShare; ++j) {
                base[j] = channel < N && j < rows_here ? out[(size_t)j * N + channel] : __ushort_as_bfloat16(0);
            }
        };
        pdl_wait();
        if (adds) fetch_bases(tile * kChannels + t);
        if (ok) ok = guard.wait(acc_done, 0);
        if (!ok) *abort_flag = 1;
        readers_barrier();       // everybody agrees on whether the tile is complete
        if (*abort_flag == 0 && (rows_here > 0 || (GATEUP && NT == 1))) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            float* exchange = reinterpret_cast<float*>(smem) + (size_t)group * kShare * 64;   // the rings are idle now
            if (GATEUP && NT == 1) {
                if (up_lane) {
                    float v[kShare];
                    tmem_load_row<kShare>(lane_base + group * kShare, v);
#pragma unroll
                    for (int j = 0; j < kShare; ++j) exchange[j * 64 + t - 64] = v[j];
                }
                readers_barrier();
            }
            if (!up_lane && rows_here > 0) {
#pragma unroll 1
                for (int u = 0; u < (GATEUP ? 1 : NT); ++u) {
                    const int channel = tile * kChannels + u * kTileN + t;
                    float scale = 0.0f, scale_up = 0.0f, bias = 0.0f;
                    if (channel < N) {
                        scale = p.scales[channel];
                        if (GATEUP) scale_up = p.scales[N + channel];
                        if (!GATEUP && p.bias != nullptr) bias = bf2f(p.bias[channel]);
                    }
                    if (adds && u > 0) fetch_bases(channel);
                    bf16* dst = out + channel;
#pragma unroll
                    for (int c0 = 0; c0 < kShare; c0 += 16) {
                        float v[16], w[16];
                        tmem_load_row<16>(lane_base + u * kTileM + group * kShare + c0, v);
                        if (GATEUP) {
                            if (NT == 2) {
                                tmem_load_row<16>(lane_base + kTileM + group * kShare + c0, w);
                            } else {
#pragma unroll
                                for (int j = 0; j < 16; ++j) w[j] = exchange[(c0 + j) * 64 + t];
                            }
                        }
#pragma unroll
                        for (int j = 0; j < 16; ++j) {
                            float val;
                            if (GATEUP) {
                                const float gate = v[j] * scale;
                                val = __fdividef(gate, 1.0f + __expf(-gate)) * (w[j] * scale_up);
                            } else if (p.epilogue == EPI_ADD) {
                                val = fmaf(v[j], scale, bf2f(base[c0 + j]));
                            } else if (p.epilogue == EPI_PLAIN) {
                                val = v[j] * scale;
                            } else {
                                val = rbf(v[j] * scale) + bias;
                                if (p.epilogue == EPI_BIAS_SILU) val = __fdividef(val, 1.0f + __expf(-val));
                                else if (p.epilogue == EPI_BIAS_ADD) val = bf2f(base[c0 + j]) + rbf(val);
                            }
                            if (channel < N && c0 + j < rows_here) dst[(size_t)(c0 + j) * N] = f2bf(val);
                        }
                    }
                }
            }
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    }
    __syncwarp();
    __syncthreads();
    if (*abort_flag) {
        // copies still in flight get time to land before the CTA's memory is released
        if (tid == 0) {
            atomicAdd(&g_wide_errors, 1u);
            if (g_wide_error_sink != nullptr) atomicAdd_system(g_wide_error_sink, 1u);
        }
        const unsigned long long until = now_ns() + 200000ull;
        while (now_ns() < until) __nanosleep(1000);
        __syncthreads();
    }
    if (warp == 3) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols)
                     : "memory");
    }
}

template <int NT, bool GATEUP>
cudaError_t launch_variant(const CUtensorMap& wm, const CUtensorMap& xm, const WideParams& p, int tiles, cudaStream_t stream) {
    return launch_pdl(gemm_wide_kernel<NT, GATEUP>, dim3((unsigned)(tiles * p.row_blocks)), dim3(kThreads), kSmemBytes, stream,
                      wm, xm, p);
}

}  // namespace

cudaError_t configure_wide_kernels() {
    cudaError_t e = cudaFuncSetAttribute(gemm_wide_kernel<1, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBytes);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(gemm_wide_kernel<1, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBytes);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(gemm_wide_kernel<2, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBytes);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(gemm_wide_kernel<2, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBytes);
    return e;
}

// `channel_tiles`: 1 or 2 (see the top of the file)
cudaError_t launch_int8_gemm_wide(const GemvArgs& a, cudaStream_t stream, int channel_tiles) {
    const bool gateup = a.epilogue == EPI_GATE_UP_SILU;
    if (a.rows < 1 || a.rows > kMaxPromptRows || a.out_features < 1 || a.in_features % kBK != 0 || a.in_features < kBK
        || a.w == nullptr || a.scales == nullptr || a.x == nullptr || a.norm_w != nullptr || a.y32 != nullptr
        || (a.epilogue == EPI_BIAS_ADD ? a.resid == nullptr : a.y == nullptr)) {
        return cudaErrorInvalidValue;
    }
    if ((a.epilogue == EPI_BIAS || a.epilogue == EPI_BIAS_SILU || a.epilogue == EPI_BIAS_ADD) && a.bias == nullptr) {
        return cudaErrorInvalidValue;
    }
    WideParams p;
    p.scales = a.scales; p.y = a.y; p.bias = a.bias; p.resid = a.resid;
    p.out_features = a.out_features; p.rows = a.rows; p.epilogue = a.epilogue;
    p.row_blocks = (a.rows + kTileM - 1) / kTileM;
    p.steps = a.in_features / kBK;
    const int per_single = gateup ? 64 : kTileN;                // output channels of a CTA with one tile
    const int nt = channel_tiles == 2 ? 2 : 1;
    const int tiles = (a.out_features + nt * per_single - 1) / (nt * per_single);
    alignas(64) CUtensorMap wm, xm;
    const uint64_t w_rows = gateup ? 2ull * a.out_features : (uint64_t)a.out_features;
    const uint32_t box_rows = gateup && nt == 1 ? 64 : kTileN;
    if (!make_map(&wm, CU_TENSOR_MAP_DATA_TYPE_UINT8, a.w, a.in_features, w_rows, a.in_features, kBK, box_rows,
                  CU_TENSOR_MAP_SWIZZLE_128B)
        || !make_map(&xm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, a.x, a.in_features, a.rows, (uint64_t)a.in_features * 2, 64, kTileM,
                     CU_TENSOR_MAP_SWIZZLE_128B)) {
        return cudaErrorInvalidValue;
    }
    if (gateup) return nt == 2 ? launch_variant<2, true>(wm, xm, p, tiles, stream) : launch_variant<1, true>(wm, xm, p, tiles, stream);
    return nt == 2 ? launch_variant<2, false>(wm, xm, p, tiles, stream) : launch_variant<1, false>(wm, xm, p, tiles, stream);
}

// Which kernel takes a projection of a prompt pass: the one with the shortest estimate.  A wave of CTAs of this
// file's kernel costs its steps (0.46 us each with one channel tile, 0.63 us with two) and 5 to 9 us of start and epilogue;
// the kernel of gemm_int8_tc.cu, in blocks of up to 64 rows or of 96, 128 or 160 side by side and with K split where that fits
// one wave, and the one of gemm_int8_pair.cu are estimated there.  Above 640 rows tc's never has fewer waves.  Measured there (us, one tile /
// two tiles / pairs): 700 rows q/k/v 20.8 / 17.2 / 15.2, o 13.2 / 17.6 / 13.7, gate/up 53.6 / 34.9 / 34.2, down 28.4 / 38.1 / 25.7;
// 2,048 rows 42.6 / 34.6 / 32.8, 25.6 / 19.4 / 20.6, 142 / 99.9 / 93.8, 56.6 / 41.8 / 38.6.
// Measured from 65 to 640 rows (us, blocks of 64 / best of the tall ones / one tile / two tiles of this file): gate/up 65 rows
// 19.0 / 12.5 / 14.8 / 17.2, 128 21.1 / 14.7 / 15.6 / 18.0, 150 22.3 / 16.3 / 27.3 / 18.6, 300 41.5 / 27.2 / 29.6 / 19.8, 448
// 53.7 / 31.3 / 43.2 / 36.8; q/k/v 128 8.3 / 9.0 / 11.6 / 18.2, 300 20.8 / 11.3 / 12.5 / 18.2, 512 23.2 / 15.0 / 13.1 / 18.6;
// down 128 10.6 / 10.8 / 28.2 / 44.3, 300 25.4 / 14.5 / 28.7 / 45.0, 640 49.7 / 20.2 / 29.9 / 44.9; o 150 8.3 / 7.8 / 12.6 /
// 19.9, 300 12.6 / 10.0 / 12.7 / 19.9.  Gate/up again, out of more weights than the L2 holds (best tall tile / one tile / pairs): 65 rows
// 11.8 / 13.5 / 13.0, 96 12.5 / 13.8 / 13.1, 112 13.5 / 14.3 / 13.2, 128 14.1 / 14.3 / 13.3, 150 15.5 / 24.8 / 15.6.  One tile's
// estimate errs on the same side as theirs, by 0.5 to 1.3 us (without the 2.6 us it took 65 to 128 rows, a prompt of 65 1,575 us for 1,505).
int gemm_prompt_kernel(const GemvArgs& a) {
    const int per_single = a.epilogue == EPI_GATE_UP_SILU ? 64 : kTileN;
    const int row_blocks = (a.rows + kTileM - 1) / kTileM, steps = a.in_features / kBK;
    auto waves = [&](int tiles) {
        return ((a.out_features + tiles * per_single - 1) / (tiles * per_single) * row_blocks + kSms - 1) / kSms;
    };
    const bool adds = a.epilogue == EPI_ADD || a.epilogue == EPI_BIAS_ADD;         // another read of the rows
    const bool crosses = a.epilogue == EPI_GATE_UP_SILU;                           // the up half, through shared memory
    const float one = waves(1) * (4.9f + (adds ? 1.5f : 0.0f) + (crosses ? 2.6f : 0.0f) + 0.456f * steps);
    const float two = waves(2) * (7.2f + (adds ? 2.0f : 0.0f) + 0.63f * steps);
    int kernel = one <= two ? 1 : 2;
    float best = one < two ? one : two;
    const float pairs = gemm_pair_estimate_us(a);
    if (pairs < best) {
        best = pairs;
        kernel = 256;
    }
    for (int t : {0, 96, 128, 160}) {
        if (t > 0 && a.rows > kTallRowsMost) break;
        const float estimate = gemm_tc_estimate_us(a, t);
        if (estimate <= best) {
            best = estimate;
            kernel = t > 0 ? t : 3;
        }
    }
    return kernel;
}

cudaError_t launch_int8_gemm_prompt(const GemvArgs& args, cudaStream_t stream) {
    GemvArgs a = args;
    if (a.norm_w != nullptr) {
        if (a.norm_out == nullptr) return cudaErrorInvalidValue;
        const cudaError_t e = launch_rms_norm_rows(a.x, a.norm_w, a.norm_out, a.rows, a.in_features, a.eps, stream);
        if (e != cudaSuccess) return e;
        a.x = a.norm_out;
        a.norm_w = nullptr;
        a.norm_out = nullptr;
    }
    const int kernel = gemm_prompt_kernel(a);
    if (kernel == 256) return launch_int8_gemm_pair(a, stream);
    return kernel < 3 ? launch_int8_gemm_wide(a, stream, kernel) : launch_int8_gemm_tc(a, stream, kernel == 3 ? 0 : kernel);
}

unsigned int gemm_wide_error_count() {
    unsigned int v = 0;
    if (cudaMemcpyFromSymbol(&v, g_wide_errors, sizeof(v)) != cudaSuccess) return ~0u;
    return v;
}

cudaError_t set_wide_error_sink(unsigned int* device_visible_word) {
    return cudaMemcpyToSymbol(g_wide_error_sink, &device_visible_word, sizeof(device_visible_word));
}

}  // namespace q3t
