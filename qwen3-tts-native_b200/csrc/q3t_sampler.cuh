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

struct TopKScratch {
    unsigned long long cand[kTopKCandidates];
    double weights[kTopKMost];
    double prefix[kTopKMost];
    int index[kTopKMost];
    unsigned int hist[256];
    unsigned long long warp_best[32];
    int counter, token;
};

// One draw from the `selections` largest of keys[0..V) (order keys; ties by lower index), 1 <= selections
// <= kTopKMost, cut at top_p; the same token and random state as the sequential fp64 arithmetic of
// the reference (sampling_kernels.cu:300-388).  Called by all THREADS threads of a block (or of a named
// barrier), which `sync` joins; every thread returns the token.
//
// What bounds it: barriers and serial fp64 chains, not the logits.  The k-th key is found by one histogram
// of distances from the largest key in steps of one bf16 ulp: only the few dozen keys within 255 steps of
// the maximum are counted, so shared-memory atomics do not pile up on a few digits as they do in a radix
// select from the top (coarser steps follow when those hold fewer than k keys).
template <int THREADS, class Sync>
__device__ __forceinline__ int sample_top_k_block(const unsigned int* keys, int V, int selections, float top_p,
                                                  float temperature, unsigned long long* rng, TopKScratch& s,
                                                  int tid, Sync sync) {
    constexpr int kWarps = THREADS / kWarp;
    const int lane = tid % kWarp;
    const int warp = tid / kWarp;
    unsigned int best = 0u;
    for (int t = tid; t < V; t += THREADS) best = max(best, keys[t]);
    best = __reduce_max_sync(0xffffffffu, best);
    if (lane == 0) s.warp_best[warp] = best;
    for (int i = tid; i < 256; i += THREADS) s.hist[i] = 0u;
    if (tid == 0) s.counter = 0;
    sync();
#pragma unroll
    for (int w = 0; w < kWarps; ++w) best = max(best, static_cast<unsigned int>(s.warp_best[w]));
    // bin d lies at (d % 8) * 32 + d / 8: lane l then reads bins 8 l .. 8 l + 7 without bank conflicts
    int shift = 16, last = -1, taken = 0;
    for (;; shift += 4) {
        for (int t = tid; t < V; t += THREADS) {
            const unsigned int d = (best - keys[t]) >> shift;
            if (d < 256u) atomicAdd(&s.hist[(d & 7u) * 32u + (d >> 3)], 1u);
        }
        sync();
        // every warp finds the bin of the `selections`-th key for itself
        unsigned int mine[8];
        unsigned int local = 0;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            mine[j] = s.hist[32 * j + lane];
            local += mine[j];
        }
        unsigned int incl = local;
#pragma unroll
        for (int o = 1; o < kWarp; o <<= 1) {
            const unsigned int n = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += n;
        }
        const unsigned int ballot = __ballot_sync(0xffffffffu, static_cast<int>(incl) >= selections);
        if (ballot != 0u) {            // with shift 28 every key is within 16 steps
            const int owner = __ffs(ballot) - 1;
            int c = static_cast<int>(incl - local);
            int chosen = 7;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                if (c < selections) {
                    c += static_cast<int>(mine[j]);
                    chosen = j;
                }
            }
            last = 8 * owner + __shfl_sync(0xffffffffu, chosen, owner);
            taken = __shfl_sync(0xffffffffu, c, owner);
            break;
        }
        sync();
        for (int i = tid; i < 256; i += THREADS) s.hist[i] = 0u;
        sync();
    }
    const float maximum = order_value(best) / temperature;
    auto place = [&](unsigned long long k, int rank) {
        const float v = order_value(static_cast<unsigned int>(k >> 12));
        s.index[rank] = 4095 - static_cast<int>(k & 0xfffull);
        s.weights[rank] = exp(static_cast<double>(v / temperature - maximum));
    };
    if (taken <= kTopKCandidates) {
        for (int t = tid; t < V; t += THREADS) {
            const unsigned int k = keys[t];
            if (((best - k) >> shift) <= static_cast<unsigned int>(last)) {
                const int p = atomicAdd(&s.counter, 1);
                if (p < kTopKCandidates) s.cand[p] = (static_cast<unsigned long long>(k) << 12) | static_cast<unsigned long long>(4095 - t);
            }
        }
        sync();
        // rank by counting (keys are unique); four threads share a candidate when they suffice
        if (4 * taken <= THREADS) {
            const int i = tid >> 2, part = tid & 3;
            const unsigned long long k = i < taken ? s.cand[i] : 0ull;
            int rank = 0;
#pragma unroll 4
            for (int j = part; j < taken; j += 4) rank += s.cand[j] > k ? 1 : 0;
            rank += __shfl_xor_sync(0xffffffffu, rank, 1);
            rank += __shfl_xor_sync(0xffffffffu, rank, 2);
            if (part == 0 && i < taken && rank < selections) place(k, rank);
        } else {
            for (int i = tid; i < taken; i += THREADS) {
                const unsigned long long k = s.cand[i];
                int rank = 0;
#pragma unroll 4
                for (int j = 0; j < taken; ++j) rank += s.cand[j] > k ? 1 : 0;
                if (rank < selections) place(k, rank);
            }
        }
    } else {
        // hundreds of keys tie around the k-th: take the largest one after the other
        unsigned long long below = ~0ull;
        for (int r = 0; r < selections; ++r) {
            unsigned long long top = 0ull;
            for (int t = tid; t < V; t += THREADS) {
                const unsigned long long k = (static_cast<unsigned long long>(keys[t]) << 12) | static_cast<unsigned long long>(4095 - t);
                if (k < below && k > top) top = k;
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const unsigned long long other = __shfl_xor_sync(0xffffffffu, top, o);
                top = other > top ? other : top;
            }
            sync();
            if (lane == 0) s.warp_best[warp] = top;
            sync();
            for (int w = 0; w < kWarps; ++w) top = s.warp_best[w] > top ? s.warp_best[w] : top;
            below = top;
            if (tid == 0) place(top, r);
        }
    }
    sync();
    if (warp == 0) {
    if (lane == 0) {
        // one thread, the reference's order of additions; eight loads at a time ahead of the chain
        double running = 0.0;
        int i = 0;
        for (; i + 8 <= selections; i += 8) {
            double w8[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) w8[u] = s.weights[i + u];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                running += w8[u];
                s.prefix[i + u] = running;
            }
        }
        for (; i < selections; ++i) {
            running += s.weights[i];
            s.prefix[i] = running;
        }
    }
    __syncwarp();
    const double denominator = s.prefix[selections - 1];
    for (int i = lane; i < selections; i += kWarp) s.weights[i] = s.weights[i] / denominator;
    __syncwarp();
    if (lane == 0) {
        double cumulative = 0.0;
        int keep = selections;
        const double limit = static_cast<double>(top_p);
        bool found = false;
        for (int i = 0; !found && i < selections; i += 8) {
            double w8[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) w8[u] = i + u < selections ? s.weights[i + u] : 0.0;
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                if (i + u < selections) cumulative += w8[u];
                if (!found && i + u < selections && cumulative >= limit) {
                    keep = i + u + 1;
                    found = true;
                }
            }
        }
        // one draw; first prefix that reaches the target
        const double target = static_cast<double>(uniform_random(rng)) * s.prefix[keep - 1];
        int first = keep;
        for (int i = 0; i < keep && first == keep; i += 8) {
            double p8[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) p8[u] = i + u < keep ? s.prefix[i + u] : 0.0;
#pragma unroll
            for (int u = 7; u >= 0; --u) {
                if (i + u < keep && p8[u] >= target) first = i + u;
            }
        }
        s.token = s.index[first < keep ? first : keep - 1];
    }
    }
    sync();
    return s.token;
}

}  // namespace q3t
