// One warp, one 16-token KV page, the two query heads of its KV head (head_dim 128): the arithmetic of
// decode_attention_kernel's inner step (attention.cu explains the fragment layouts), for kernels that
// walk pages on their own.  Same operations in the same order, so the same bits.
#pragma once

#include "q3t_common.cuh"

namespace q3t {
namespace page {

__device__ __forceinline__ void mma_bf16_16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                               uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
        "{%0, %1, %2, %3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}

// K: tokens 8 nt + gid, dims 32 jj + 8 tig .. + 7; V: tokens 8 h + 2 tig + p, dims 64 jb + 8 gid .. + 7
struct Fragments {
    int4 k[2][4];
    int4 v[2][2][2];
};

// rows [0, bound) of a page ([16][128] bf16 at k and v); rows past it read as zero
__device__ __forceinline__ void load(Fragments& f, const bf16* k, const bf16* v, int bound, int lane) {
    const int gid = lane >> 2, tig = lane & 3;
    const int4 zero4 = make_int4(0, 0, 0, 0);
#pragma unroll
    for (int nt = 0; nt < 2; ++nt) {
        const int t = 8 * nt + gid;
#pragma unroll
        for (int jj = 0; jj < 4; ++jj) {
            f.k[nt][jj] = t < bound ? __ldcg(reinterpret_cast<const int4*>(k + (size_t)t * 128 + 32 * jj + 8 * tig)) : zero4;
        }
    }
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int pp = 0; pp < 2; ++pp) {
            const int t = 8 * h + 2 * tig + pp;
#pragma unroll
            for (int jb = 0; jb < 2; ++jb) {
                f.v[h][pp][jb] = t < bound ? __ldcg(reinterpret_cast<const int4*>(v + (size_t)t * 128 + 64 * jb + 8 * gid)) : zero4;
            }
        }
}

// replaces row `t_new` (this step's token) by rows held in shared memory
__device__ __forceinline__ void patch(Fragments& f, const bf16* krow, const bf16* vrow, int t_new, int lane) {
    const int gid = lane >> 2, tig = lane & 3;
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
        if (8 * nt + gid == t_new) {
#pragma unroll
            for (int jj = 0; jj < 4; ++jj) f.k[nt][jj] = *reinterpret_cast<const int4*>(krow + 32 * jj + 8 * tig);
        }
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int pp = 0; pp < 2; ++pp)
            if (8 * h + 2 * tig + pp == t_new) {
#pragma unroll
                for (int jb = 0; jb < 2; ++jb) f.v[h][pp][jb] = *reinterpret_cast<const int4*>(vrow + 64 * jb + 8 * gid);
            }
}

// A page's scores (columns 2 tig, + 1 of tokens 8 nt ..) -> its maximum, the sum of its weights over the first `count` tokens,
// and the weights as bf16 hi + lo.
__device__ __forceinline__ void probabilities(const float (&sc)[2][4], int count, float scale, int tig, float& mx, float& lsum,
                                              uint32_t (&ph)[2], uint32_t (&pl)[2]) {
    mx = -INFINITY;
    lsum = 0.0f;
    float pr[2][2];
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const bool valid = 8 * nt + 2 * tig + e < count;
            pr[nt][e] = valid ? sc[nt][e] * scale : -INFINITY;
            mx = fmaxf(mx, pr[nt][e]);
        }
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            pr[nt][e] = pr[nt][e] == -INFINITY ? 0.0f : expf(pr[nt][e] - mx);
            lsum += pr[nt][e];
        }
    lsum += __shfl_xor_sync(0xffffffffu, lsum, 1);
    lsum += __shfl_xor_sync(0xffffffffu, lsum, 2);
#pragma unroll
    for (int nt = 0; nt < 2; ++nt) {
        ph[nt] = pack_bf16x2(pr[nt][0], pr[nt][1]);
        pl[nt] = pack_bf16x2(pr[nt][0] - __uint_as_float(ph[nt] << 16), pr[nt][1] - __uint_as_float(ph[nt] & 0xffff0000u));
    }
}

// Scores, softmax within the page and weighted V over its first `count` tokens.  mx, lsum: of head gid (lanes of
// gid < 2); o[x][0], o[x][2]: head 2 tig, dims 8 gid + x and 64 + 8 gid + x; o[x][1], o[x][3]: head 2 tig + 1.
// q: [2][128] fp32 (bf16-valued) in shared memory, 16-byte aligned.
__device__ __forceinline__ void attend(const Fragments& f, const float* q, int count, float scale, int lane, float& mx,
                                       float& lsum, float (&o)[8][4]) {
    const int gid = lane >> 2, tig = lane & 3;
    float sc[2][4];
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) sc[nt][e] = 0.0f;
    const float* mine = q + (gid & 1) * 128;
    const bool real = gid < 2;
#pragma unroll
    for (int jj = 0; jj < 4; ++jj) {
        const float4 q0 = *reinterpret_cast<const float4*>(mine + 32 * jj + 8 * tig);
        const float4 q1 = *reinterpret_cast<const float4*>(mine + 32 * jj + 8 * tig + 4);
        const uint32_t a00 = real ? pack_bf16x2(q0.x, q0.y) : 0u, a01 = real ? pack_bf16x2(q0.z, q0.w) : 0u;
        const uint32_t a10 = real ? pack_bf16x2(q1.x, q1.y) : 0u, a11 = real ? pack_bf16x2(q1.z, q1.w) : 0u;
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
            mma_bf16_16816(sc[nt], a00, 0u, a01, 0u, (uint32_t)f.k[nt][jj].x, (uint32_t)f.k[nt][jj].y);
            mma_bf16_16816(sc[nt], a10, 0u, a11, 0u, (uint32_t)f.k[nt][jj].z, (uint32_t)f.k[nt][jj].w);
        }
    }
    uint32_t ph[2], pl[2];
    probabilities(sc, count, scale, tig, mx, lsum, ph, pl);
    uint32_t tv[2][2][2][4];
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int pp = 0; pp < 2; ++pp)
#pragma unroll
            for (int jb = 0; jb < 2; ++jb) {
                tv[h][pp][jb][0] = (uint32_t)f.v[h][pp][jb].x;
                tv[h][pp][jb][1] = (uint32_t)f.v[h][pp][jb].y;
                tv[h][pp][jb][2] = (uint32_t)f.v[h][pp][jb].z;
                tv[h][pp][jb][3] = (uint32_t)f.v[h][pp][jb].w;
            }
#pragma unroll
    for (int x = 0; x < 8; ++x) {
#pragma unroll
        for (int e = 0; e < 4; ++e) o[x][e] = 0.0f;
        const uint32_t sel = (x & 1) ? 0x7632u : 0x5410u;
        const uint32_t a0 = __byte_perm(tv[0][0][0][x >> 1], tv[0][1][0][x >> 1], sel);
        const uint32_t a1 = __byte_perm(tv[0][0][1][x >> 1], tv[0][1][1][x >> 1], sel);
        const uint32_t a2 = __byte_perm(tv[1][0][0][x >> 1], tv[1][1][0][x >> 1], sel);
        const uint32_t a3 = __byte_perm(tv[1][0][1][x >> 1], tv[1][1][1][x >> 1], sel);
        mma_bf16_16816(o[x], a0, a1, a2, a3, ph[0], ph[1]);
        mma_bf16_16816(o[x], a0, a1, a2, a3, pl[0], pl[1]);
    }
}

// ---- a row's pages over sixteen slots of eight classes -------------------------------------------------------------
// kBlock consecutive pages go to one slot (a CTA), block after block over the slots, and there to classes, one page to a
// class at first; a class is walked by one warp.  The classes of a slot and then the slots are merged in order.  The
// grouping depends on the row's length only, so whoever computes it, the decode chain or a launch of its own, gets the
// same bits.
constexpr int kSlots = 16;
constexpr int kClasses = 8;
constexpr int kBlock = 2;
constexpr int kPageStep = kClasses * kSlots;             // from a class's page to its next
__device__ __forceinline__ int slots_of(int pages) { return min(kSlots, (pages + kBlock - 1) / kBlock); }
__device__ __forceinline__ int class_page(int slot, int cls) { return kBlock * (slot + kSlots * (cls / kBlock)) + cls % kBlock; }

// One head vector, lane l dims l, l + 32, l + 64, l + 96: RMSNorm, then the rotation cs0 (dims l, l + 64) and cs1.
__device__ __forceinline__ void rotate(const float (&x)[4], const bf16 (&w)[4], uint32_t cs0, uint32_t cs1, float eps, float (&o)[4]) {
    float sq[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) sq[j] = fmaf(x[j], x[j], 0.0f);
    float c = (sq[0] + sq[2]) + (sq[1] + sq[3]);
    c = warp_sum_down(c);
    c = __shfl_sync(0xffffffffu, c, 0);
    const float inv = rsqrtf(c / 128.0f + eps);
    float y[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) y[j] = rbf(rbf(x[j] * inv) * bf2f(w[j]));
    rope_pair_cs(y[0], y[2], bf_lo(cs0), bf_hi(cs0), o[0], o[2]);
    rope_pair_cs(y[1], y[3], bf_lo(cs1), bf_hi(cs1), o[1], o[3]);
}

// What a class has so far: maximum, sum and weighted V, as attend() leaves a page's.
struct Running {
    float m, l, o[8][4];
};
__device__ __forceinline__ void start(Running& r) {
    r.m = -INFINITY;
    r.l = 0.0f;
#pragma unroll
    for (int x = 0; x < 8; ++x)
#pragma unroll
        for (int e = 0; e < 4; ++e) r.o[x][e] = 0.0f;
}
__device__ __forceinline__ void add(Running& r, bool first, float mp, float lp, const float (&op)[8][4]) {
    // the first page replaces nothing: m is -inf, its factor 0 and the page's own 1, exactly
    const float top = fmaxf(r.m, mp);
    const float fo = first ? 0.0f : expf(r.m - top), fn = expf(mp - top);
    r.l = first ? lp : fmaf(r.l, fo, lp * fn);
    r.m = top;
    // columns 2 tig and 2 tig + 1 are heads; only tig = 0 holds real ones
    const float fo0 = __shfl_sync(0xffffffffu, fo, 0), fo1 = __shfl_sync(0xffffffffu, fo, 4);
    const float fn0 = __shfl_sync(0xffffffffu, fn, 0), fn1 = __shfl_sync(0xffffffffu, fn, 4);
#pragma unroll
    for (int x = 0; x < 8; ++x) {
        r.o[x][0] = fmaf(r.o[x][0], fo0, op[x][0] * fn0);
        r.o[x][2] = fmaf(r.o[x][2], fo0, op[x][2] * fn0);
        r.o[x][1] = fmaf(r.o[x][1], fo1, op[x][1] * fn1);
        r.o[x][3] = fmaf(r.o[x][3], fo1, op[x][3] * fn1);
    }
}
// acc: [head][128], m and l: [head], of this class
__device__ __forceinline__ void put_class(const Running& r, float* acc, float* m, float* l, int lane) {
    if ((lane & 3) != 0) return;
    const int gid = lane >> 2;
    if (gid < 2) {
        m[gid] = r.m;
        l[gid] = r.l;
    }
#pragma unroll
    for (int c = 0; c < 2; ++c)
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const int e = 2 * half + c;
            float4* d4 = reinterpret_cast<float4*>(acc + 8 * gid + 128 * c + 64 * half);
            d4[0] = make_float4(r.o[0][e], r.o[1][e], r.o[2][e], r.o[3][e]);
            d4[1] = make_float4(r.o[4][e], r.o[5][e], r.o[6][e], r.o[7][e]);
        }
}
// the classes of a slot in order, for dim d of head g: acc [class][head][128], m and l [class][head]
__device__ __forceinline__ void merge_classes(const float* acc, const float* m, const float* l, int slot, int pages, int g, int d,
                                              float& top, float& sum, float& value) {
    int classes = 1;
    while (classes < kClasses && class_page(slot, classes) < pages) ++classes;
    top = -INFINITY;
    for (int c = 0; c < classes; ++c) top = fmaxf(top, m[c * 2 + g]);
    sum = 0.0f;
    value = 0.0f;
    for (int c = 0; c < classes; ++c) {
        const float fac = expf(m[c * 2 + g] - top);
        sum = fmaf(l[c * 2 + g], fac, sum);
        value = fmaf(acc[c * 256 + g * 128 + d], fac, value);
    }
}
// the slots in order, by a warp: get(k, 0) is slot k's maximum, get(k, 1) its sum, get(k, 2 + dim) its weighted V
template <class Get>
__device__ __forceinline__ float fold(Get get, int slots, int dim, int lane) {
    // lane k holds what the fold needs of slot k: its factor and sum
    const float mine = lane < slots ? get(lane, 0) : -INFINITY;
    const float sum = lane < slots ? get(lane, 1) : 0.0f;
    const float fac = expf(mine - warp_max_xor(mine));
    float total = 0.0f, value = 0.0f;
#pragma unroll 4
    for (int k = 0; k < slots; ++k) {
        const float fk = __shfl_sync(0xffffffffu, fac, k);
        total = fmaf(__shfl_sync(0xffffffffu, sum, k), fk, total);
        value = fmaf(get(k, 2 + dim), fk, value);
    }
    return value * (1.0f / total);
}

}  // namespace page
}  // namespace q3t
