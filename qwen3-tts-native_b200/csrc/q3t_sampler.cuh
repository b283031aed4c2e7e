// Device functions of the seeded sampler shared by the stand-alone kernels (sampler.cu) and the decode
// chain (decode_chain.cu): order keys, the xorshift64* draw, and the top-k / top-p draw of one row by
// one block.  The reference's sampler is native/qwen3-tts-native/native/src/sampling_kernels.cu:30-388;
// sampler.cu states what of it is kept to the bit.
#pragma once

#include "q3t_common.cuh"

namespace q3t {

__device__ __forceinline__ unsigned int order_key(float v) {
    unsigned int u = __float_as_uint(v);
    if (u == 0x80000000u) u = 0u;   // -0 ties with +0
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

__device__ __forceinline__ float order_value(unsigned int k) {
    return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

// xorshift64* (sampling_kernels.cu:53-69)
__device__ __forceinline__ float uniform_random(unsigned long long* state) {
    unsigned long long v = *state;
    if (v == 0) v = 0x9e3779b97f4a7c15ULL;
    v ^= v >> 12;
    v ^= v << 25;
    v ^= v >> 27;
    *state = v;
    const unsigned long long r = v * 0x2545f4914f6cdd1dULL;
    constexpr double scale = 1.0 / 9007199254740992.0;
    return static_cast<float>(static_cast<double>(r >> 11) * scale);
}

constexpr int kTopKMost = 128;           // largest top-k drawn by sample_top_k_block
constexpr int kTopKCandidates = 256;     // candidates it ranks by counting
constexpr int kDistanceBins = 768;       // 704 used

struct TopKScratch {
    unsigned long long cand[kTopKCandidates];
    double weights[kTopKMost];
    double prefix[kTopKMost];
    int index[kTopKMost];
    unsigned int hist[kDistanceBins];
    unsigned long long warp_best[32];
    unsigned int warp_total[8];
    unsigned int limit;
    int counter, taken, token;
    float uniform;
};

// One draw from the `selections` largest of keys[0..V) (order keys; ties by lower index), 1 <= selections
// <= kTopKMost, cut at top_p; the same token and random state as the sequential fp64 arithmetic of
// the reference (sampling_kernels.cu:300-388).  Called by all THREADS threads of a block (or of a named
// barrier), which `sync` joins; every thread returns the token.
//
// What bounds it: barriers, serial fp64 chains (17 cycles an addition) and the fetching of its own code, not the logits.  A
// thread keeps its keys in registers.  The k-th key is found by one histogram of the keys' distances from the largest, in
// steps that grow with the distance (exact to 127 bf16 ulps, then 64 to an octave), so that one pass is enough whatever the
// logits' spread, and shared-memory atomics do not pile up on a few digits as they do in a radix select from the top.
// Every step exists once in the code: the decode chain runs it once in five layers, out of a cold instruction cache.
// (A draw of 50 from 2048 in the chain: 9,400 cycles with bins of one ulp, coarser ones as long as they held too few, one
// thread that searched and everything unrolled; 8,300 so.)
__device__ __forceinline__ unsigned int distance_bin(unsigned int distance) {        // distance < 2^16
    const int shift = max(0, 25 - __clz(static_cast<int>(distance)));
    return static_cast<unsigned int>(shift * 64) + (distance >> shift);
}
template <int THREADS, int PER, class Sync>                // a thread's keys: V <= PER * THREADS
__device__ __forceinline__ int sample_top_k_block(const unsigned int* keys, int V, int selections, float top_p,
                                                  float temperature, unsigned long long* rng, TopKScratch& s,
                                                  int tid, Sync sync) {
    constexpr int kWarps = THREADS / kWarp;
    const int lane = tid % kWarp;
    const int warp = tid / kWarp;
    unsigned int mine[PER], best = 0u;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
        const int t = tid + i * THREADS;
        mine[i] = t < V ? keys[t] : 0u;
        best = max(best, mine[i]);
    }
    best = __reduce_max_sync(0xffffffffu, best);
    if (lane == 0) s.warp_best[warp] = best;
    for (int i = tid; i < kDistanceBins; i += THREADS) s.hist[i] = 0u;
    if (tid == 0) s.counter = 0;
    if (tid == THREADS - 1) s.uniform = uniform_random(rng);                 // (the draw's one random number)
    sync();
    best = __reduce_max_sync(0xffffffffu, lane < kWarps ? static_cast<unsigned int>(s.warp_best[lane]) : 0u);
#pragma unroll
    for (int i = 0; i < PER; ++i) {
        if (tid + i * THREADS < V) atomicAdd(&s.hist[distance_bin((best - mine[i]) >> 16)], 1u);
    }
    sync();
    // the bin of the `selections`-th key: 256 threads, three bins each
    static_assert(THREADS >= 256 && kDistanceBins == 3 * 256, "eight warps count");
    unsigned int own[3], incl = 0u;
    if (tid < 256) {
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            own[j] = s.hist[3 * tid + j];
            incl += own[j];
        }
        const unsigned int total = incl;
#pragma unroll
        for (int o = 1; o < kWarp; o <<= 1) {
            const unsigned int n = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += n;
        }
        if (lane == kWarp - 1) s.warp_total[warp] = incl;
        incl -= total;                                                         // keys in bins before this thread's, of its warp
    }
    sync();
    if (tid < 256) {
        const unsigned int before = lane < warp ? static_cast<unsigned int>(s.warp_total[lane & 7]) : 0u;
        unsigned int count = incl + __reduce_add_sync(0xffffffffu, before);
        const unsigned int want = static_cast<unsigned int>(selections);
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            if (count < want && count + own[j] >= want) {
                const unsigned int bin = static_cast<unsigned int>(3 * tid + j);
                const int shift = max(0, static_cast<int>(bin >> 6) - 1);
                s.limit = ((bin - static_cast<unsigned int>(shift * 64) + 1u) << shift) - 1u;      // its largest distance
                s.taken = static_cast<int>(count + own[j]);
            }
            count += own[j];
        }
    }
    sync();
    const unsigned int limit = s.limit;
    const int taken = s.taken;
    unsigned long long* chosen_keys = reinterpret_cast<unsigned long long*>(s.prefix);      // the selections, largest first
    if (taken <= kTopKCandidates) {
        // a place for each thread's candidates: one atomic a warp
        int held = 0;
#pragma unroll
        for (int i = 0; i < PER; ++i) held += tid + i * THREADS < V && ((best - mine[i]) >> 16) <= limit ? 1 : 0;
        int at = held;
#pragma unroll
        for (int o = 1; o < kWarp; o <<= 1) {
            const int n = __shfl_up_sync(0xffffffffu, at, o);
            if (lane >= o) at += n;
        }
        int base = 0;
        if (lane == kWarp - 1 && at > 0) base = atomicAdd(&s.counter, at);
        at += __shfl_sync(0xffffffffu, base, kWarp - 1) - held;
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            const int t = tid + i * THREADS;
            if (t < V && ((best - mine[i]) >> 16) <= limit) {
                s.cand[at++] = (static_cast<unsigned long long>(mine[i]) << 12) | static_cast<unsigned long long>(4095 - t);
            }
        }
        sync();
        // rank by counting (keys are unique), four threads to a candidate
#pragma unroll 1
        for (int first = 0; first < taken; first += THREADS / 4) {
            const int i = first + (tid >> 2), part = tid & 3;
            const unsigned long long k = i < taken ? s.cand[i] : 0ull;
            int rank = 0;
#pragma unroll 4
            for (int j = part; j < taken; j += 4) rank += s.cand[j] > k ? 1 : 0;
            rank += __shfl_xor_sync(0xffffffffu, rank, 1);
            rank += __shfl_xor_sync(0xffffffffu, rank, 2);
            if (part == 0 && i < taken && rank < selections) chosen_keys[rank] = k;
        }
    } else {
        // hundreds of keys tie around the k-th: take the largest one after the other
        unsigned long long below = ~0ull;
#pragma unroll 1
        for (int r = 0; r < selections; ++r) {
            unsigned long long top = 0ull;
#pragma unroll 1
            for (int t = tid; t < V; t += THREADS) {
                const unsigned long long k = (static_cast<unsigned long long>(keys[t]) << 12) | static_cast<unsigned long long>(4095 - t);
                if (k < below && k > top) top = k;
            }
#pragma unroll 1
            for (int o = 16; o > 0; o >>= 1) {
                const unsigned long long other = __shfl_xor_sync(0xffffffffu, top, o);
                top = other > top ? other : top;
            }
            sync();
            if (lane == 0) s.warp_best[warp] = top;
            sync();
#pragma unroll 1
            for (int w = 0; w < kWarps; ++w) top = s.warp_best[w] > top ? s.warp_best[w] : top;
            below = top;
            if (tid == 0) chosen_keys[r] = top;
        }
    }
    sync();
    static_assert(THREADS >= kTopKMost, "a thread per selection");
    const int padded = (selections + 7) / 8 * 8;              // the chains below go in eights
    if (tid < padded) {
        double weight = 0.0;
        if (tid < selections) {
            const unsigned long long k = chosen_keys[tid];
            const float maximum = order_value(best) / temperature;
            s.index[tid] = 4095 - static_cast<int>(k & 0xfffull);
            weight = exp(static_cast<double>(order_value(static_cast<unsigned int>(k >> 12)) / temperature - maximum));
        }
        s.weights[tid] = weight;
    }
    sync();
    if (warp == 0) {
        double* cumulative = reinterpret_cast<double*>(s.cand);           // sums of the weights' shares
        static_assert(kTopKCandidates >= kTopKMost && kTopKMost % 8 == 0, "room for the sums");
#pragma unroll 1
        for (int pass = 0; pass < 2; ++pass) {
            double* sums = pass == 0 ? s.prefix : cumulative;
            if (lane == 0) {
                // one thread, the reference's order of additions; eight loads ahead of the chain
                double running = 0.0, ahead[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) ahead[u] = s.weights[u];
#pragma unroll 1
                for (int i = 0; i < padded; i += 8) {
                    double w8[8];
#pragma unroll
                    for (int u = 0; u < 8; ++u) {
                        w8[u] = ahead[u];
                        ahead[u] = s.weights[min(i + 8, kTopKMost - 8) + u];
                    }
#pragma unroll
                    for (int u = 0; u < 8; ++u) {
                        running += w8[u];
                        sums[i + u] = running;
                    }
                }
            }
            __syncwarp();
            if (pass == 0) {
                const double denominator = s.prefix[selections - 1];
#pragma unroll 1
                for (int i = lane; i < selections; i += kWarp) s.weights[i] = s.weights[i] / denominator;
                __syncwarp();
            }
        }
        // the first of n sums that reaches a bound, n if none does
        auto first_reaching = [&](const double* sums, int n, double bound) {
            int found = n;
#pragma unroll 1
            for (int first = 0; first < n; first += kWarp) {
                const int i = first + lane;
                const unsigned int reached = __ballot_sync(0xffffffffu, i < n && sums[min(i, n - 1)] >= bound);
                if (reached != 0u) {
                    found = first + __ffs(reached) - 1;
                    break;
                }
            }
            return found;
        };
        int keep = selections, first = 0;
#pragma unroll 1
        for (int search = 0; search < 2; ++search) {
            const double bound = search == 0 ? static_cast<double>(top_p) : static_cast<double>(s.uniform) * s.prefix[keep - 1];
            first = first_reaching(search == 0 ? cumulative : s.prefix, keep, bound);
            if (search == 0) keep = min(first + 1, selections);
        }
        if (lane == 0) s.token = s.index[first < keep ? first : keep - 1];
    }
    sync();
    return s.token;
}

}  // namespace q3t
