// Int8 weight-only GEMM for long prompt passes: pairs of CTAs on the 5th-generation tensor cores.
//
// Same operation and epilogues as gemm_int8_wide.cu.  A cluster of two CTAs multiplies 256 weight rows by up to 256 activation
// rows with tcgen05.mma.cta_group::2: each CTA converts 128 weight rows into its tensor memory (the A operand, and later the
// accumulators of the same lanes) and fetches half of the activation rows (its half of B), which the tensor cores of both read.
//
// What bounds it: the products, 4 cycles for a step of 128 K and a row, at the clock that the power leaves; below 140 rows the conversion of
// the weights, 0.36 us a step of 128 K.  A weight is converted once for up to 256 rows, where gemm_int8_wide.cu converts it for
// 128; its two tiles of 128 x 128 take 0.63 us a step, this kernel's 256 x 256 of two SMs 0.7.
//
// The rows of a pair are a multiple of 16 chosen at the launch, so that whole rounds of pairs are full: 1,500 rows of a projection
// to 2048 channels are 9 blocks of 176 by 8 tiles, 72 of the GPU's 74 pairs at once, instead of 6 by 8 of 256.
// Measured (B200, 1,500 rows, us; gemm_int8_wide.cu / here): q/k/v 33.7 / 27.9, o 19.5 / 17.2, gate/up 68.9 / 67.3, down 41.4 / 30.6.
// What it took: arrivals at the other CTA's barriers without a cluster-wide release, which waited 2,000 cycles and more for the
// arriving thread's other accesses (down 48.7 -> 29.9 with one pair a tile); the look at the next step's barriers ahead of
// this one's products (110 cycles an answer, three a step).
//
// Warp roles: 0 weight copies, 1 product issue (in the first CTA only), 2 activation copies, 3 tensor memory, then in the second CTA the
// relay that tells the first one of activations that have landed; 4..19 in four groups dequantise, then read the accumulators.
// A pair of CTAs stays for all of its tiles: weights and activations of the next one are on their way while the last one's
// accumulators are read.  The two tiles of gate/up lie side by
// side in the lanes (64 channels each a CTA); the values that a channel's other lane finishes cross through
// shared memory.  Every wait is bounded.

#include "q3t_kernels.cuh"
#include "q3t_tcgen05.cuh"

namespace q3t {
namespace {

using namespace tc;

constexpr int kGroups = 4;
constexpr int kThreads = 128 + 128 * kGroups;
constexpr int kTileN = 128;                   // weight rows of a CTA
constexpr int kMostRows = 256;                // activation rows of a pair
constexpr int kBK = 128;
constexpr int kWStages = 4, kAStages = 4;
constexpr int kMostXStages = 8;               // as many as fit the ring: 5 of 256 rows, 7 of 176
static_assert(kWStages % kGroups == 0 && kAStages % kGroups == 0, "one group per stage");
constexpr int kWStageBytes = kTileN * kBK;                    // 16 KB
constexpr int kXRingBytes = 5 * kMostRows / 2 * kBK * 2;      // 160 KB, of which gate/up takes 32 for values that cross lanes
constexpr int kCrossingBytes = kGroups * 16 * kTileN * 4;
constexpr int kAStageCols = kBK / 2;
constexpr int kAStageBase = 256;
constexpr uint32_t kTmemCols = 512;
constexpr unsigned long long kBudgetNs = 2000000000ull;
constexpr int kBarriers = 2 * kWStages + 3 * kMostXStages + 2 * kAStages + 2;
constexpr size_t kSmemBytes = 1024 + (size_t)kWStages * kWStageBytes + kXRingBytes + kBarriers * sizeof(uint64_t) + 64;

__device__ unsigned int g_pair_errors = 0;
__device__ unsigned int* g_pair_error_sink = nullptr;

struct PairParams {
    const float* scales;
    bf16* y;
    const bf16* bias;
    bf16* resid;
    int out_features;       // N (gate/up: channels, the matrix has 2N rows)
    int rows;
    int pair_rows;          // activation rows of a pair, a multiple of 16
    int row_blocks;
    int pairs;              // tiles of a pair in all: each pair of CTAs takes every so manieth
    int steps;              // K / kBK
    int x_stages;
    int epilogue;
};

// a barrier of the first CTA of the pair, wherever this runs
__device__ __forceinline__ void arrive_at_first(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(peer_smem(smem_u32(bar), 0u)) : "memory");
}
__device__ __forceinline__ void umma_pair(uint32_t d, uint32_t a, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(d), "r"(a), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// the same barrier of both CTAs, once the products issued so far are done
__device__ __forceinline__ void commit_both(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(smem_u32(bar)), "h"((uint16_t)3) : "memory");
}
// Whether any of the readers says so; they all get the same answer, and leave together or not at all.
__device__ __forceinline__ bool any_reader(bool says) {
    uint32_t any;
    __syncwarp();
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 q, %1, 0;\n\t"
        "barrier.cta.red.or.pred p, 1, %2, q;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(any)
        : "r"(says ? 1u : 0u), "n"(128 * kGroups)
        : "memory");
    return any != 0;
}
__device__ __forceinline__ void group_barrier(int group) {
    __syncwarp();
    asm volatile("bar.sync %0, 128;" ::"r"(2 + group) : "memory");
}

template <bool GATEUP>
__global__ void __launch_bounds__(kThreads, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap w_map, const __grid_constant__ CUtensorMap x_map, const PairParams p) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    unsigned char* w8 = smem;
    unsigned char* xs = w8 + kWStages * kWStageBytes;
    uint64_t* full_w = reinterpret_cast<uint64_t*>(xs + kXRingBytes);
    uint64_t* empty_w = full_w + kWStages;
    uint64_t* full_x = empty_w + kWStages;        // landed here
    uint64_t* peer_x = full_x + kMostXStages;     // landed in the other CTA (the first one's)
    uint64_t* empty_x = peer_x + kMostXStages;
    uint64_t* full_a = empty_x + kMostXStages;        // converted in both (the first CTA's)
    uint64_t* empty_a = full_a + kAStages;
    uint64_t* acc_done = empty_a + kAStages;
    uint64_t* acc_free = acc_done + 1;            // accumulators read in both (the first CTA's)
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_free + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int tid = threadIdx.x;
    const int warp = __shfl_sync(0xffffffffu, tid / kWarp, 0);
    const int lane = tid % kWarp;
    const int rank = (int)cluster_rank();
    const int first_pair = blockIdx.x / 2, stride = gridDim.x / 2;
    // row blocks fastest: the pairs in flight share few weight tiles and all of the activations
    auto tile_of = [&](int pair) { return pair / p.row_blocks; };
    auto row_base_of = [&](int pair) { return (pair % p.row_blocks) * p.pair_rows; };
    const int half_rows = p.pair_rows / 2;
    const int N = p.out_features;
    const int nk = p.steps;
    const int x_atom = half_rows * 128;           // 64 K of this CTA's rows
    const int x_stages = p.x_stages;

    Guard guard;
    guard.deadline = now_ns() + kBudgetNs;
    guard.abort_flag = abort_flag;

    if (tid == 0) {
        for (int s = 0; s < kWStages; ++s) {
            mbar_init(&full_w[s], 1);
            mbar_init(&empty_w[s], 4);
        }
        for (int s = 0; s < kMostXStages; ++s) {
            mbar_init(&full_x[s], 1);
            mbar_init(&peer_x[s], 1);
            mbar_init(&empty_x[s], 1);
        }
        for (int s = 0; s < kAStages; ++s) {
            mbar_init(&full_a[s], 8);
            mbar_init(&empty_a[s], 1);
        }
        mbar_init(acc_done, 1);
        mbar_init(acc_free, 8 * kGroups);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 3) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(kTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_sync();                               // the other CTA's barriers are set up
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = *tmem_slot;
    // weights never depend on the launch before; activations, residuals and outputs do
    if (warp >= 1 && warp <= 3) {
        pdl_wait();
        if (warp == 1) pdl_trigger();
    }

    if (warp == 0) {
        if (elect_one()) {
            int n = 0;
            for (int pair = first_pair; pair < p.pairs; pair += stride) {
                const int tile = tile_of(pair);
                for (int i = 0; i < nk; ++i, ++n) {
                    const int s = n % kWStages;
                    if (n >= kWStages && !guard.wait(&empty_w[s], ((n / kWStages) - 1) & 1)) break;
                    mbar_expect_tx(&full_w[s], kWStageBytes);
                    unsigned char* dst = w8 + s * kWStageBytes;
                    if (GATEUP) {
                        tma_load_2d(dst, &w_map, i * kBK, tile * 128 + rank * 64, &full_w[s]);
                        tma_load_2d(dst + kWStageBytes / 2, &w_map, i * kBK, N + tile * 128 + rank * 64, &full_w[s]);
                    } else {
                        tma_load_2d(dst, &w_map, i * kBK, (2 * tile + rank) * kTileN, &full_w[s]);
                    }
                }
                if (*abort_flag) break;
            }
        }
    } else if (warp == 2) {
        if (elect_one()) {
            int s = 0, turn = 0;
            for (int pair = first_pair; pair < p.pairs; pair += stride) {
                const int first = row_base_of(pair) + rank * half_rows;
                for (int i = 0; i < nk; ++i) {
                    if (turn > 0 && !guard.wait(&empty_x[s], (turn - 1) & 1)) break;
                    mbar_expect_tx(&full_x[s], 2 * x_atom);
                    unsigned char* dst = xs + s * 2 * x_atom;
                    tma_load_2d(dst, &x_map, i * kBK, first, &full_x[s]);
                    tma_load_2d(dst + x_atom, &x_map, i * kBK + 64, first, &full_x[s]);
                    if (++s == x_stages) {
                        s = 0;
                        ++turn;
                    }
                }
                if (*abort_flag) break;
            }
        }
    } else if (warp == 3) {
        if (rank == 1 && elect_one()) {
            int s = 0, turn = 0;
            const int steps = nk * ((p.pairs - first_pair + stride - 1) / stride);
            for (int n = 0; n < steps; ++n) {
                if (!guard.wait(&full_x[s], turn & 1)) break;
                arrive_at_first(&peer_x[s]);
                if (++s == x_stages) {
                    s = 0;
                    ++turn;
                }
            }
        }
    } else if (warp == 1) {
        if (rank == 0 && elect_one()) {
            // fp32 accumulators, A and B bf16, K-major, 256 lanes of two CTAs
            const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(p.pair_rows >> 3) << 17) | ((uint32_t)(256 >> 4) << 24);
            int sx = 0, turn = 0, n = 0, tiles = 0;
            // A look at a barrier takes 110 cycles and more to answer, complete or not, and there are three a step: the next step's are
            // asked ahead of this one's products.
            auto there = [&](int x, int x_turn, int step) {
                return mbar_test(&full_x[x], x_turn & 1) & mbar_test(&peer_x[x], x_turn & 1) & mbar_test(&full_a[step % kAStages], (step / kAStages) & 1);
            };
            uint32_t ready = 0;
            bool ok = true;
            for (int pair = first_pair; pair < p.pairs && ok; pair += stride, ++tiles) {
                if (tiles > 0 && !guard.wait(acc_free, (tiles - 1) & 1)) break;
                for (int i = 0; i < nk; ++i, ++n) {
                    const int sa = n % kAStages;
                    if (ready == 0) {
                        ok = guard.wait(&full_x[sx], turn & 1) && guard.wait(&peer_x[sx], turn & 1) && guard.wait(&full_a[sa], (n / kAStages) & 1);
                        if (!ok) break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t b_addr = smem_u32(xs + sx * 2 * x_atom);
                    const uint32_t a_col = tmem_base + kAStageBase + sa * kAStageCols;
                    uint64_t* const done = &empty_x[sx];
                    if (++sx == x_stages) {
                        sx = 0;
                        ++turn;
                    }
                    ready = there(sx, turn, n + 1);
#pragma unroll
                    for (int j = 0; j < kBK / 16; ++j) {
                        umma_pair(tmem_base, a_col + 8 * j, umma_desc(b_addr + (j / 4) * x_atom + 32 * (j % 4)), idesc, (i | j) != 0 ? 1u : 0u);
                    }
                    commit_both(&empty_a[sa]);
                    commit_both(done);
                }
                if (ok) commit_both(acc_done);
            }
        }
    } else {
        const int group = (warp - 4) / 4;
        const int t = (warp % 4) * 32 + lane;        // weight row within the CTA's = TMEM lane
        const uint32_t lane_base = tmem_base + ((uint32_t)((warp % 4) * 32) << 16);
        const int upper = t >> 6;
        const bool adds = !GATEUP && (p.epilogue == EPI_ADD || p.epilogue == EPI_BIAS_ADD);
        float* const crossing = reinterpret_cast<float*>(xs + kXRingBytes - kCrossingBytes) + group * 16 * kTileN;      // [16 rows][128 lanes]
        bool ok = true;
        int n = group, tiles = 0;                    // the group's next step, of all tiles'
        const int all_steps = nk * ((p.pairs - first_pair + stride - 1) / stride);
        for (int pair = first_pair; pair < p.pairs; pair += stride, ++tiles) {
            // and the first step of the next tile, so that its products can begin when the accumulators have been read
            const int end = min(all_steps, (tiles + 1) * nk + kGroups);
            for (; n < end && ok; n += kGroups) {
                const int s = n % kWStages, sa = n % kAStages;
                if (!__all_sync(0xffffffffu, guard.wait(&full_w[s], (n / kWStages) & 1))) { ok = false; break; }
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
                __syncwarp();
                if (lane == 0) mbar_arrive(&empty_w[s]);
                if (n >= kAStages && !__all_sync(0xffffffffu, guard.wait(&empty_a[sa], ((n / kAStages) - 1) & 1))) {
                    ok = false;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                tmem_store_32(lane_base + kAStageBase + sa * kAStageCols, out[0]);
                tmem_store_32(lane_base + kAStageBase + sa * kAStageCols + 32, out[1]);
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) arrive_at_first(&full_a[sa]);
            }
            // Group g finishes the activation rows 16 (g + 4 i) .. + 15 of the pair; a thread has one weight row.  What a residual
            // epilogue adds to is requested sixteen rows at a time, the first before the last products are waited for.
            const int tile = tile_of(pair), rows_here = min(p.pair_rows, p.rows - row_base_of(pair));
            const int chunks = (rows_here + 15) / 16;
            const int channel = GATEUP ? tile * 128 + rank * 64 + (t & 63) : (2 * tile + rank) * kTileN + t;
            const bool mine = channel < N;
            bf16* out = (p.epilogue == EPI_BIAS_ADD ? p.resid : p.y) + (size_t)row_base_of(pair) * N + channel;
            bf16 base[16];
            auto fetch_bases = [&](int chunk) {
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    const int r = 16 * chunk + j;
                    base[j] = mine && r < rows_here ? out[(size_t)r * N] : __ushort_as_bfloat16(0);
                }
            };
            float scale = 0.0f, scale_up = 0.0f, bias = 0.0f;
            if (mine) {
                scale = p.scales[channel];
                if (GATEUP) scale_up = p.scales[N + channel];
                if (!GATEUP && p.bias != nullptr) bias = bf2f(p.bias[channel]);
            }
            if (tiles == 0) pdl_wait();
            if (adds && group < chunks) fetch_bases(group);
            if (ok) ok = guard.wait(acc_done, tiles & 1);
            if (!ok) *abort_flag = 1;
            if (any_reader(*abort_flag != 0)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            auto finish = [&](int chunk, const float (&v)[16], const float* other) {
                bf16* dst = out + (size_t)(16 * chunk) * N;
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    float val;
                    if (GATEUP) {
                        const float across = other[j * kTileN];
                        const float gate = (upper ? across : v[j]) * scale;
                        val = __fdividef(gate, 1.0f + __expf(-gate)) * ((upper ? v[j] : across) * scale_up);
                    } else if (p.epilogue == EPI_ADD) {
                        val = fmaf(v[j], scale, bf2f(base[j]));
                    } else if (p.epilogue == EPI_PLAIN) {
                        val = v[j] * scale;
                    } else {
                        val = rbf(v[j] * scale) + bias;
                        if (p.epilogue == EPI_BIAS_SILU) val = __fdividef(val, 1.0f + __expf(-val));
                        else if (p.epilogue == EPI_BIAS_ADD) val = bf2f(base[j]) + rbf(val);
                    }
                    if (mine && 16 * chunk + j < rows_here) dst[(size_t)j * N] = f2bf(val);
                }
            };
            if (GATEUP) {
                // two chunks of a group at a time: the gate's lanes finish the first and the up lanes the second, each with what the
                // other's lane of the same channel holds of it
                for (int chunk = group; chunk < chunks; chunk += 2 * kGroups) {
                    float v[16];
                    if (chunk != group) group_barrier(group);        // the last two have been read
                    tmem_load_row<16>(lane_base + 16 * (chunk + (upper ? 0 : kGroups)), v);
#pragma unroll
                    for (int j = 0; j < 16; ++j) crossing[j * kTileN + t] = v[j];
                    tmem_load_row<16>(lane_base + 16 * (chunk + (upper ? kGroups : 0)), v);
                    group_barrier(group);
                    finish(chunk + (upper ? kGroups : 0), v, crossing + (t ^ 64));
                }
            } else {
                for (int chunk = group; chunk < chunks; chunk += kGroups) {
                    if (adds && chunk != group) fetch_bases(chunk);
                    float v[16];
                    tmem_load_row<16>(lane_base + 16 * chunk, v);
                    finish(chunk, v, nullptr);
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) arrive_at_first(acc_free);
            if (GATEUP) group_barrier(group);
        }
    }
    __syncwarp();
    __syncthreads();
    if (*abort_flag) {
        // copies still in flight get time to land before the CTA's memory is released
        if (tid == 0) {
            atomicAdd(&g_pair_errors, 1u);
            if (g_pair_error_sink != nullptr) atomicAdd_system(g_pair_error_sink, 1u);
        }
        const unsigned long long until = now_ns() + 200000ull;
        while (now_ns() < until) __nanosleep(1000);
        __syncthreads();
    }
    cluster_sync();                               // the other CTA's products read this one's activations, and arrive here
    if (warp == 3) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
    }
}

constexpr int kPairs = 74;                    // of CTAs at once

template <bool GATEUP>
cudaError_t launch_variant(const CUtensorMap& wm, const CUtensorMap& xm, const PairParams& p, cudaStream_t stream) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(2 * (p.pairs < kPairs ? p.pairs : kPairs)));
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = kSmemBytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = pdl_enabled() ? 1 : 0;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    return cudaLaunchKernelEx(&cfg, gemm_pair_kernel<GATEUP>, wm, xm, p);
}

int tiles_of(const GemvArgs& a) {
    const int per_pair = a.epilogue == EPI_GATE_UP_SILU ? 128 : 256;
    return (a.out_features + per_pair - 1) / per_pair;
}
// A step of 128 K takes 0.0026 us a row, but no less than 0.36; a round an epilogue that grows with the rows, the launch 5.6.
// Measured / estimated (us): 1,500 rows o 17.2 / 16.9, down 30.7 / 31.5, q/k/v (two rounds) 27.9 / 28.2, gate/up (four) 68 / 70; 800 rows
// down 25.9 / 25.4.
float estimate(const GemvArgs& a, int blocks, int* pair_rows) {
    const int rows = ((a.rows + blocks - 1) / blocks + 15) / 16 * 16;
    const int rounds = (tiles_of(a) * blocks + kPairs - 1) / kPairs;
    const float step = 0.0026f * rows > 0.36f ? 0.0026f * rows : 0.36f;
    *pair_rows = rows;
    return 5.6f + rounds * (0.8f + 0.018f * rows + a.in_features / kBK * step);
}
int best_blocks(const GemvArgs& a, float* us, int* pair_rows) {
    int best = 0;
    const int fewest = (a.rows + kMostRows - 1) / kMostRows;
    for (int blocks = fewest; blocks <= 3 * fewest + 1 && blocks <= (a.rows + 63) / 64; ++blocks) {
        int rows = 0;
        const float e = estimate(a, blocks, &rows);
        if (best == 0 || e < *us) {
            best = blocks;
            *us = e;
            *pair_rows = rows;
        }
    }
    return best;
}

}  // namespace

cudaError_t configure_pair_kernels() {
    cudaError_t e = cudaFuncSetAttribute(gemm_pair_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBytes);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(gemm_pair_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBytes);
    return e;
}

float gemm_pair_estimate_us(const GemvArgs& a) {
    float us = 1.0e9f;
    int pair_rows = 0;
    best_blocks(a, &us, &pair_rows);
    return us;
}

cudaError_t launch_int8_gemm_pair(const GemvArgs& a, cudaStream_t stream) {
    const bool gateup = a.epilogue == EPI_GATE_UP_SILU;
    if (a.rows < 1 || a.rows > kMaxPromptRows || a.out_features < 1 || a.in_features % kBK != 0 || a.in_features < kBK
        || a.w == nullptr || a.scales == nullptr || a.x == nullptr || a.norm_w != nullptr || a.y32 != nullptr
        || (a.epilogue == EPI_BIAS_ADD ? a.resid == nullptr : a.y == nullptr)) {
        return cudaErrorInvalidValue;
    }
    if ((a.epilogue == EPI_BIAS || a.epilogue == EPI_BIAS_SILU || a.epilogue == EPI_BIAS_ADD) && a.bias == nullptr) {
        return cudaErrorInvalidValue;
    }
    PairParams p;
    float us = 0.0f;
    p.scales = a.scales; p.y = a.y; p.bias = a.bias; p.resid = a.resid;
    p.out_features = a.out_features; p.rows = a.rows; p.epilogue = a.epilogue;
    p.row_blocks = best_blocks(a, &us, &p.pair_rows);
    p.steps = a.in_features / kBK;
    p.pairs = tiles_of(a) * p.row_blocks;
    p.x_stages = (kXRingBytes - (gateup ? kCrossingBytes : 0)) / (p.pair_rows * kBK);
    if (p.x_stages > kMostXStages) p.x_stages = kMostXStages;
    alignas(64) CUtensorMap wm, xm;
    const uint64_t w_rows = gateup ? 2ull * a.out_features : (uint64_t)a.out_features;
    if (!make_map(&wm, CU_TENSOR_MAP_DATA_TYPE_UINT8, a.w, a.in_features, w_rows, a.in_features, kBK, gateup ? 64 : kTileN, CU_TENSOR_MAP_SWIZZLE_128B)
        || !make_map(&xm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, a.x, a.in_features, a.rows, (uint64_t)a.in_features * 2, 64, p.pair_rows / 2,
                     CU_TENSOR_MAP_SWIZZLE_128B)) {
        return cudaErrorInvalidValue;
    }
    return gateup ? launch_variant<true>(wm, xm, p, stream) : launch_variant<false>(wm, xm, p, stream);
}

unsigned int gemm_pair_error_count() {
    unsigned int v = 0;
    if (cudaMemcpyFromSymbol(&v, g_pair_errors, sizeof(v)) != cudaSuccess) return ~0u;
    return v;
}

cudaError_t set_pair_error_sink(unsigned int* device_visible_word) {
    return cudaMemcpyToSymbol(g_pair_error_sink, &device_visible_word, sizeof(device_visible_word));
}

}  // namespace q3t
