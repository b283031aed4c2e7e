// The decode chain: the code predictor's 16 positions, or the talker's 28 layers, of up to eight sessions in
// ONE launch.
//
// A frame of few sessions is a chain of some 540 dependent projections and attentions whose bytes are few:
// launched one by one, each costs 0.6 us of hand-over, 0.9 us until its activations are fetched and
// converted, and its exchange and epilogue, 3.5-9 us a link whatever it streams.  Here 128 CTAs stay on
// their SMs for the whole chain.  What bounds it now is what a hand-over between them costs: 0.3 us for a word within a
// die and 0.5 across, 0.4 to 1.1 us with the wait for the slowest, and 0.3 to 1.5 us of instructions on either side.  So
// the split of the work is the one that needs fewest:
//
//   8 groups of 16 CTAs; group c owns KV head c (and its two query heads), i.e. slice c of eight of every
//   contraction whose input it produced itself.
//     q/k/v          CTA computes 32 of the group's 512 rows over all of K       -> exchange in the group
//     attention      of the group's own heads, by the group                       (talker: pages spread over it)
//     o projection   partial sums over the group's 256 attention values, 1/16 of the outputs per CTA
//                                                                                  -> exchange over the grid
//     gate/up, SiLU  1/16 of the group's eighth of the channels, all of K         -> exchange in the group
//     down           partial sums over the group's channels                       -> exchange over the grid
//   Dependent hand-overs a layer, instead of five launches: an exchange over the grid is one hop where every CTA adds up
//   all columns itself (the predictor at one row) and two elsewhere (partial sums, then the new hidden rows in the
//   group); talker attention adds one (pages' partials), with several rows two (folded heads).  Predictor 4 at one row
//   and 6 at more, talker 7 and 8.
//
// The eight partial sums of a K-split projection are the eight K-slices that gemv_int8_mma.cu gives its eight
// warps: same fixed-point conversion per slice, exact integer sums, the slices added in the same order.
// A frame made here is bit for bit the frame made launch by launch with attention_blocks.cu for the talker's
// attention, and a row's result does not depend on the rows beside it.
//
// Exchanges carry their own flags: a 16-byte store holds three words of data and the exchange's number, the
// reader polls the data itself (single-copy atomic 128-bit relaxed accesses), so a hand-over is one trip
// through the L2 and needs no fence or counter.  Buffers alternate by exchange; a CTA can be at most one
// exchange of a kind ahead of the slowest reader (it has read what that reader wrote after reading).  The numbers
// are 32 bits and are restarted, buffers cleared, long before they would come round (restart_chain_numbers).
//
// Weights: at load time every CTA's share is laid out as one contiguous stream in the order the chain uses
// it, each 1 KB block holding the MMA fragments of 16 rows x 64 K as the lanes read them.  It flows through a
// ring in shared memory in 8 KB bulk copies, requested by a warp of their own as far ahead as the ring
// reaches, so that HBM (talker) or the L2 (predictor) keeps delivering while the CTAs wait for each other.
//
// Where the CTAs and the buffers are.  The GPU is two dies.  A word written on one die and read on the same one from memory
// that is at home there is read 550 cycles after the store; where one of the three lies on the other die it is 950 to 1,050.
// Homes alternate by pages of 4 KB.  So a group's CTAs are taken from one die and its buffers from pages of that die: each CTA
// claims a place on its SM's die at the start (claim_place).  chain_places.cu measures which SM and which page lies where; where
// it cannot tell, any place will do.
//
// The launch is cooperative (all CTAs resident or none) and the engine orders the chains of a device one
// after the other.  Every wait is bounded by a deadline; a wait that gives up marks the run, all others then
// give up at once, the kernel runs through on whatever it holds and the host refuses the result.

#include "q3t_attention_page.cuh"
#include "q3t_kernels.cuh"
#include "q3t_sampler.cuh"
#include "q3t_tcgen05.cuh"

namespace q3t {
namespace {

using tc::mbar_expect_tx;
using tc::mbar_init;
using tc::mbar_try_wait;
using tc::now_ns;
using tc::smem_u32;

constexpr int kSlices = 8;
constexpr int kRanks = 16;
constexpr int kCtas = kSlices * kRanks;
constexpr int kWorkers = 256;                        // eight warps that compute
constexpr int kThreads = kWorkers + 4 * kWarp;       // and a group of four, one of which requests weights
// Registers are handed out to groups of four warps: 168 a thread at launch, 232 to those that compute and 40 to the others
// (256 * 232 + 128 * 40 = 384 * 168).
constexpr int kWorkerRegisters = 232, kRequestRegisters = 40;
static_assert(kWorkers * kWorkerRegisters + 4 * kWarp * kRequestRegisters <= kThreads * 168, "registers of the block");
constexpr int kSlot = 8192;                          // bytes of a ring slot
constexpr int kSlotUnits = 4;                        // a slot is free once all of its 2 KB units have been read
constexpr int kLimbs = 3;
constexpr int kRowsMost = 8;
constexpr unsigned long long kBudgetNs = 2000000000ull;

template <bool TALKER>
struct Dim;
template <>
struct Dim<true> {
    static constexpr int H = 2048, I = 6144, Layers = 28, HeadRows = 24, HeadTiles = 2;
};
template <>
struct Dim<false> {
    static constexpr int H = 1024, I = 3072, Layers = 5, HeadRows = 16, HeadTiles = 1;
};
template <bool TALKER>
struct Shape : Dim<TALKER> {
    using B = Dim<TALKER>;
    static constexpr int J = B::H / 512;                 // 64-wide K blocks of a warp in a projection over all of K
    static constexpr int Out = B::H / kRanks;            // outputs of a K-split projection per CTA (128 / 64)
    static constexpr int OutTiles = Out / 16;
    static constexpr int Gu = B::I / kCtas;              // gate/up channels per CTA (48 / 24)
    static constexpr int GuTiles = 2 * Gu / 16;
    static constexpr int Slice = B::I / kSlices;         // K of a CTA's share of the down projection (768 / 384)
    static constexpr int QkvBytes = 32 * B::H, OBytes = Out * 256, GuBytes = 2 * Gu * B::H, DownBytes = Out * Slice;
    static constexpr int LayerBytes = QkvBytes + OBytes + GuBytes + DownBytes;
    static constexpr int LayerSlots = LayerBytes / kSlot;
    static constexpr int HeadBytes = B::HeadTiles * 16 * B::H;
    static constexpr int HeadSlots = HeadBytes / kSlot;
    static constexpr int Groups = 3 * OutTiles;          // column groups of a CTA's outputs: 6 + 6 + 4 of a tile (24 / 12)
    static_assert(QkvBytes % kSlot == 0 && OBytes % kSlot == 0 && GuBytes % kSlot == 0 && DownBytes % kSlot == 0
                  && HeadBytes % kSlot == 0, "phases start at slot boundaries");
    static_assert(Gu % 6 == 0, "gate/up channels travel six to a quad");
};

// ---- exchange buffers, in quads of 16 bytes ----------------------------------------------------------------
struct alignas(16) Quad {
    uint32_t x, y, z, flag;
};
constexpr int kPartQuads = 2 * kSlices * kRanks * kRowsMost * 48;
constexpr int kHiddenQuads = 2 * kRanks * kRowsMost * 24;
constexpr int kGroupRow = 8;                         // quads of a CTA's q/k/v rows (6) or gate/up channels (4 or 8) of an activation row
constexpr int kGroupQuads = 2 * kRanks * kRowsMost * kGroupRow;
constexpr int kAttnPartQuads = 2 * kRanks * kRowsMost * 88;
constexpr int kAttnQuads = 2 * kRanks * 22;
constexpr int kLogitQuads = 2 * kCtas * kRowsMost * 3;
constexpr int kTokenQuads = 2 * kRowsMost;
constexpr int kAppendedQuads = 2 * kSlices * kRowsMost;
// what stays in a group: behind the rest, in pages of the group's die; offsets in a group's own space
constexpr int kAtHidden = 0;
constexpr int kAtGroup = kAtHidden + kHiddenQuads;
constexpr int kAtAttnPart = kAtGroup + kGroupQuads;
constexpr int kAtAttn = kAtAttnPart + kAttnPartQuads;
constexpr int kPageQuads = kPlacePage / 16;
static_assert((kAtAttn + kAttnQuads + kPageQuads - 1) / kPageQuads <= kGroupPages, "pages of a group");
constexpr int kAtLogits = kPartQuads;
constexpr int kAtTokens = kAtLogits + kLogitQuads;
constexpr int kAtAppended = kAtTokens + kTokenQuads;
constexpr int kSharedQuads = (kAtAppended + kAppendedQuads + kPageQuads - 1) / kPageQuads * kPageQuads;

__device__ unsigned int g_chain_errors = 0;
__device__ unsigned int* g_chain_error_sink = nullptr;

__device__ __forceinline__ void put_quad(Quad* p, uint32_t x, uint32_t y, uint32_t z, uint32_t flag) {
    asm volatile(
        "{\n\t.reg .b128 t;\n\t.reg .b64 a, b;\n\t"
        "mov.b64 a, {%1, %2};\n\tmov.b64 b, {%3, %4};\n\tmov.b128 t, {a, b};\n\t"
        "st.relaxed.gpu.global.b128 [%0], t;\n\t}"
        ::"l"(p), "r"(x), "r"(y), "r"(z), "r"(flag)
        : "memory");
}
__device__ __forceinline__ Quad get_quad(const Quad* p) {
    Quad v;
    asm volatile(
        "{\n\t.reg .b128 t;\n\t.reg .b64 a, b;\n\t"
        "ld.relaxed.gpu.global.b128 t, [%4];\n\t"
        "mov.b128 {a, b}, t;\n\tmov.b64 {%0, %1}, a;\n\tmov.b64 {%2, %3}, b;\n\t}"
        : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.flag)
        : "l"(p)
        : "memory");
    return v;
}

// A number that stands for plain stores: whoever reads it may read what was stored (by this thread, or by others that
// met it at a barrier) before it was put.
__device__ __forceinline__ void put_behind(Quad* p, uint32_t number) {
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(&p->flag), "r"(number) : "memory");
}
__device__ __forceinline__ uint32_t get_ahead(const Quad* p) {
    uint32_t number;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(number) : "l"(&p->flag) : "memory");
    return number;
}

struct LayerConst {
    const float *qkv_s, *o_s, *gu_s, *down_s;
    const bf16 *in_norm, *post_norm, *q_norm, *k_norm;
};

struct ChainArgs {
    const uint8_t* stream;           // packed layers: [128 CTAs][layers][LayerBytes]
    const uint8_t* heads;            // packed heads: [128 CTAs][heads][HeadBytes]
    const LayerConst* layers;
    const bf16* final_norm;
    const float* const* head_s;      // row scales of each head
    const bf16* hidden;              // [rows][H] input of the first layer (predictor: of position 0)
    bf16* normalized;                // talker: [rows][H] final-normed hidden
    bf16* logits;                    // talker: [rows][vocabulary]
    const bf16* const* projected;    // predictor: input row of every token, per codebook
    FrameTable* table;
    const int* positions;            // talker: [rows]
    KvLayout kv;                     // offsets of layer 0
    long long kv_layer_elems;        // elements from one layer's planes to the next's
    const uint32_t* rope_table;      // [positions][64] bf16 cos | sin
    Quad* exchange;
    uint32_t* epoch;                 // [0] number of the last exchange, [1] the run that was given up
    const ChainPlaces* places;
    uint32_t* claims;                // [0], [1] CTAs of a die that have asked for a place, [2] CTAs that have an answer
    int rows;
    float eps;
};

// ROWS: 1 or 2 exactly that many activation rows; 4 and 8 stand for 3..4 and 5..8
template <bool TALKER, int ROWS>
struct Layout {
    using S = Shape<TALKER>;
    static constexpr int XStride = S::H + 64;                      // bytes between limb rows: next limb half a bank row on
    static constexpr int XBytes = ROWS * kLimbs * XStride;
    static constexpr int RedRows = 2 * S::Gu > 32 ? 2 * S::Gu : 32;
    static constexpr int UBytesA = ROWS * S::H * 2, UBytesB = 8 * ROWS * RedRows * 4;
    static constexpr int UBytesC = TALKER && ROWS == 1 ? 16 * 2 * 132 * 4 : 0;     // gathered attention partials
    static constexpr int UBytes = UBytesA > UBytesB ? (UBytesA > UBytesC ? UBytesA : UBytesC) : (UBytesB > UBytesC ? UBytesB : UBytesC);
    static constexpr int QkvBytes = ROWS * 1024;                   // [rows][512] bf16; also [rows][256] fp32 partial squares
    static constexpr int AttBytes = ROWS * S::Slice * 2;           // [rows][256] bf16, each row as long as one of the next
    static constexpr int ActBytes = ROWS * S::Slice * 2;           // [rows][Slice] bf16
    static constexpr bool OneHop = !TALKER && ROWS == 1;           // every CTA sums all columns itself
    static constexpr int OwnBytes = OneHop ? S::H * 2 : ROWS * S::Out * 2;
    static constexpr int QBytes = ROWS * 1024;                     // [rows][2][128] fp32
    static constexpr int KNewBytes = ROWS * 256;
    static constexpr int StageBytes = 512;
    static constexpr int SampleBytes = TALKER ? 0 : 2048 * 4 + (int)sizeof(TopKScratch);
    static constexpr int AtX = 0;                                  // attention scratch overlays X and U
    static constexpr int AtU = AtX + (XBytes + 127) / 128 * 128;
    static constexpr int AtQkv = AtU + (UBytes + 127) / 128 * 128;
    static constexpr int AtAtt = AtQkv + QkvBytes;
    static constexpr int AtAct = AtAtt + AttBytes;
    static constexpr int AtOwn = AtAct + ActBytes;
    static constexpr int AtQ = AtOwn + OwnBytes;
    static constexpr int AtKNew = AtQ + QBytes;
    static constexpr int AtStage = AtKNew + KNewBytes;
    static constexpr int AtSample = AtStage + StageBytes;
    static constexpr int AtMisc = AtSample + (SampleBytes + 15) / 16 * 16;
    static constexpr int MiscBytes = 1280;
    // One or two rows of the predictor: every CTA of a group keeps the group's cache, one page of 16 tokens a layer, to
    // itself (K as rows, V with the tokens of a dimension side by side): nothing to fetch, nothing to publish.
    static constexpr bool LocalKv = !TALKER && ROWS <= 2;
    static constexpr int KvPage = 2 * kPageTokens * 128 * 2;
    static constexpr int AtPages = AtMisc + MiscBytes;             // of the group's buffers
    static constexpr int AtConst = AtPages + kGroupPages * 4;      // the layers' constants
    static constexpr int AtKv = (AtConst + S::Layers * (int)sizeof(LayerConst) + 127) / 128 * 128;
    static constexpr int AtRing = AtKv + (LocalKv ? ROWS * S::Layers * KvPage : 0);
    static constexpr int Budget = 227 * 1024;
    static constexpr int SlotsFit = (Budget - AtRing) / kSlot;
    static constexpr int Slots = SlotsFit > 24 ? 24 : SlotsFit;
    static constexpr int Bytes = AtRing + Slots * kSlot;
    // talker attention: per (row, class, head) a weighted V of 128, maximum and sum; then 16 ranks' partials of one
    // row's two heads (one row) or of one head
    static constexpr int ClassFloats = ROWS * 8 * 2 * (128 + 2);
    static_assert(!TALKER || ClassFloats * 4 + 4 * ROWS * 2 * 132 <= AtQkv, "attention scratch fits over X and U");
    static_assert(!TALKER || 16 * 2 * 132 * 4 <= AtQkv, "gathered attention partials fit over X and U");
};

struct Misc {
    uint64_t full[24];
    uint64_t empty[24];            // counts the units of the slot that have been read
    unsigned int asked[24];        // copies requested into the slot
    int place;
    uint32_t base, landed;         // landed: slots of the stream, in order
    int abort;
    int position[kRowsMost];
    int token[kRowsMost];
    float unscale[kRowsMost];
    float inverse[kRowsMost];      // of the rows' root mean squares
    unsigned long long rng[kRowsMost];
    unsigned short codes[kRowsMost][kCodebooks];
    SamplingParams sampling[kRowsMost];
};
static_assert(sizeof(Misc) <= 1280, "misc area");

__device__ __forceinline__ void imma(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k32.row.col.s32.s8.u8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
template <int kByte>
__device__ __forceinline__ uint32_t gather_byte(uint32_t w0, uint32_t w1, uint32_t w2, uint32_t w3) {
    const uint32_t lo = __byte_perm(w0, w1, ((4 + kByte) << 4) | kByte);
    const uint32_t hi = __byte_perm(w2, w3, ((4 + kByte) << 4) | kByte);
    return __byte_perm(lo, hi, 0x5410);
}

// 2 Q consecutive bf16 of one row and K-slice per lane -> three byte limbs in shared memory; returns the factor
// that undoes the scaling (the conversion of gemv_int8_mma.cu, see there)
template <int Q>
__device__ __forceinline__ float to_limbs(const uint32_t (&raw)[Q], unsigned char* dst, int stride) {
    __nv_bfloat162 m2 = __habs2(*reinterpret_cast<const __nv_bfloat162*>(&raw[0]));
#pragma unroll
    for (int m = 1; m < Q; ++m) m2 = __hmax2(m2, __habs2(*reinterpret_cast<const __nv_bfloat162*>(&raw[m])));
    const uint32_t mbits = *reinterpret_cast<const uint32_t*>(&m2);
    const uint32_t top = __reduce_max_sync(0xffffffffu, max(mbits & 0xffffu, mbits >> 16));
    const uint32_t eb_raw = (top >> 7) & 0xffu;
    const uint32_t eb = min(max(eb_raw, 21u), 240u);
    const float scale = __uint_as_float((274u - eb) << 23);
    uint32_t fixed[2 * Q];
#pragma unroll
    for (int m = 0; m < Q; ++m) {
        fixed[2 * m] = __float_as_uint(fmaf(bf_lo(raw[m]), scale, 12582912.0f));
        fixed[2 * m + 1] = __float_as_uint(fmaf(bf_hi(raw[m]), scale, 12582912.0f));
    }
#pragma unroll
    for (int m = 0; m < Q / 2; ++m) {
        const uint32_t f0 = fixed[4 * m], f1 = fixed[4 * m + 1], f2 = fixed[4 * m + 2], f3 = fixed[4 * m + 3];
        reinterpret_cast<uint32_t*>(dst)[m] = gather_byte<0>(f0, f1, f2, f3);
        reinterpret_cast<uint32_t*>(dst + stride)[m] = gather_byte<1>(f0, f1, f2, f3);
        reinterpret_cast<uint32_t*>(dst + 2 * stride)[m] = gather_byte<2>(f0, f1, f2, f3);
    }
    return eb_raw == 255u ? __uint_as_float(0x7fc00000u) : __uint_as_float((eb - 20u) << 23);
}

__device__ __forceinline__ void sync_workers() { asm volatile("bar.sync 1, %0;" ::"n"(kWorkers) : "memory"); }

// The rare side of a wait.  True: stop waiting.  (A function of plain values: the chain's state stays in registers.)
__device__ __noinline__ bool chain_gives_up(int* abort_word, uint32_t* run_word, uint32_t base, unsigned long long deadline) {
    if (*reinterpret_cast<volatile int*>(abort_word) != 0) return true;
    if (*reinterpret_cast<volatile uint32_t*>(run_word) == base || now_ns() > deadline) {
        *reinterpret_cast<volatile uint32_t*>(run_word) = base;
        *reinterpret_cast<volatile int*>(abort_word) = 1;
        return true;
    }
    return false;
}

// The code of a layer runs once per layer, so instruction fetch is a cost of its own: what both halves of a layer
// share (norm, exchange of partial sums) exists once, inner loops stay rolled where they are short.
template <bool TALKER, int ROWS>
struct Chain {
    using S = Shape<TALKER>;
    using L = Layout<TALKER, ROWS>;
    static constexpr int NT = (ROWS + 1) / 2;                // 8-column groups of B: two activation rows each

    const ChainArgs& a;
    unsigned char* smem;
    Misc* misc;
    int tid, lane, warp, rows;
    int cta = 0, slice = 0, rank = 0;                   // the CTA's place among the kCtas
    uint32_t seq = 0;              // ring slots consumed by the phases so far
    uint32_t step = 0;             // exchanges so far
    uint32_t base = 0;
    uint32_t flips = 0;            // buffer in use, one bit per kind of exchange
    unsigned long long deadline = 0;

    enum Kind { kPart = 0, kHid = 1, kGroup = 2, kAttnPart = 4, kAttn = 5, kLogits = 6, kTokens = 7, kAppended = 8 };

    __device__ Chain(const ChainArgs& args, unsigned char* s)
        : a(args), smem(s), misc(reinterpret_cast<Misc*>(s + L::AtMisc)), tid(threadIdx.x), lane(threadIdx.x % kWarp),
          warp(__shfl_sync(0xffffffffu, (int)threadIdx.x / kWarp, 0)),
          rows(ROWS <= 2 ? ROWS : args.rows) {}

    // ---- bounded waits -------------------------------------------------------------------------------------
    __device__ __forceinline__ bool given_up() { return *reinterpret_cast<volatile int*>(&misc->abort) != 0; }
    __device__ __forceinline__ bool slow_check() { return chain_gives_up(&misc->abort, a.epoch + 1, base, deadline); }
    template <int N>
    __device__ __forceinline__ void poll(const Quad* const (&p)[N], Quad (&v)[N], uint32_t flag) {
        for (uint32_t polls = 0;;) {
            bool all = true;
#pragma unroll
            for (int i = 0; i < N; ++i) v[i] = get_quad(p[i]);
#pragma unroll
            for (int i = 0; i < N; ++i) all = all && v[i].flag == flag;
            if (all) return;
            if ((++polls & 31u) == 0u && slow_check()) return;
        }
    }
    __device__ __forceinline__ Quad poll_one(const Quad* p, uint32_t flag) {
        const Quad* q[1] = {p};
        Quad v[1];
        poll(q, v, flag);
        return v[0];
    }
    // The predictor's cache rows are appended by one CTA of the group (rank r for row r) with plain stores and read by the
    // others at the next position: the appending warp says so when its position is done, the reading ones look before
    // their first load.  (The talker's rows are read by the next launch.)
    uint32_t appended_flag = 0;
    const Quad* appended_at = nullptr;
    __device__ __forceinline__ void say_appended(bool last) {
        const int b = flip(kAppended);
        appended_flag = next_flag();
        Quad* at = a.exchange + kAtAppended + (b * kSlices + slice) * kRowsMost + min(warp, rows - 1);
        appended_at = at;
        if (!last && warp < rows && rank == warp && lane == 0) put_behind(at, appended_flag);
    }
    __device__ __forceinline__ void await_appended() {
        if (lane == 0) {
            for (uint32_t polls = 0; get_ahead(appended_at) != appended_flag;) {
                if ((++polls & 31u) == 0u && slow_check()) break;
            }
        }
        __syncwarp();
    }
    // Slot `s` and all before it have landed.  (A warp of its own counts them: looking at the count costs those that compute 30
    // cycles, a wait on the slot's own barrier 110, data there or not.)
    __device__ __forceinline__ void wait_slot(uint32_t s) {
        uint32_t landed;
        for (uint32_t polls = 0;;) {
            asm volatile("ld.acquire.cta.shared::cta.u32 %0, [%1];" : "=r"(landed) : "r"(smem_u32(&misc->landed)) : "memory");
            if (landed > s) return;
            if ((++polls & 63u) == 0u && slow_check()) return;
        }
    }
    __device__ __forceinline__ uint32_t next_flag() { return base + ++step; }
    // which of the two buffers of a kind this exchange uses
    __device__ __forceinline__ int flip(Kind k) {
        const int b = (flips >> k) & 1u;
        flips ^= 1u << k;
        return b;
    }

    // ---- ring ----------------------------------------------------------------------------------------------
    static constexpr uint32_t kLayerSlots = S::Layers * S::LayerSlots;
    // Of the predictor's position 0 only the keys and values are needed: its last layer ends with them.  (3 and 8 sessions 2,140
    // -> 2,123 and 3,207 -> 3,176 us; with one or two rows it gains nothing, 1,569 and 1,575.)
    static constexpr bool kEndsEarly = !TALKER && !L::LocalKv;
    static constexpr uint32_t kUnused = kEndsEarly ? S::LayerSlots - S::QkvBytes / kSlot : 0;
    static constexpr uint32_t kAllSlots = TALKER ? kLayerSlots + S::HeadSlots : kCodebooks * kLayerSlots + 15 * S::HeadSlots - kUnused;
    // The requesting warp's one thread: slot after slot of the CTA's stream, each once what lay in its place has been read.
    __device__ __forceinline__ void request_weights() {
        const uint8_t* layers = a.stream + (size_t)cta * S::Layers * S::LayerBytes;
        const uint8_t* heads = a.heads + (size_t)cta * (TALKER ? 1 : 15) * S::HeadBytes;
        // the layers, then a head; the predictor's sixteen positions all read the layers, and position 0 has no head
        const uint8_t* src = layers;
        uint32_t left = kLayerSlots - kUnused, at = 0, fill = 0;
        bool in_layers = true, headless = !TALKER;
#pragma unroll 1
        for (uint32_t s = 0; s < kAllSlots; ++s) {
            uint64_t* bar = &misc->full[at];
            if (fill > 0) {
                for (uint32_t polls = 0; !mbar_try_wait(&misc->empty[at], (fill - 1) & 1u);) {
                    if ((++polls & 15u) == 0u && slow_check()) return;
                }
            }
            *reinterpret_cast<volatile unsigned int*>(&misc->asked[at]) = fill + 1;
            mbar_expect_tx(bar, kSlot);
            asm volatile(
                "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                ::"r"(smem_u32(smem + L::AtRing + at * kSlot)), "l"(src), "r"(kSlot), "r"(smem_u32(bar))
                : "memory");
            src += kSlot;
            if (++at == L::Slots) {
                at = 0;
                ++fill;
            }
            if (--left == 0) {
                if (in_layers && !headless) {
                    src = heads;
                    heads += S::HeadBytes;
                    left = S::HeadSlots;
                    in_layers = false;
                } else {
                    src = layers;
                    left = kLayerSlots;
                    in_layers = true;
                    headless = false;
                }
            }
        }
    }
    // The counting warp's one thread.
    __device__ __forceinline__ void count_landed() {
        uint32_t at = 0, fill = 0;
#pragma unroll 1
        for (uint32_t s = 0; s < kAllSlots; ++s) {
            for (uint32_t polls = 0; !mbar_try_wait(&misc->full[at], fill & 1u);) {
                if ((++polls & 15u) == 0u && slow_check()) return;
            }
            asm volatile("st.release.cta.shared::cta.u32 [%0], %1;" ::"r"(smem_u32(&misc->landed)), "r"(s + 1) : "memory");
            if (++at == L::Slots) {
                at = 0;
                ++fill;
            }
        }
    }
    // Gives back bytes [off, off + len) of the phase that started at slot `first`, lane i the i-th slot touched.
    __device__ __forceinline__ void release(uint32_t first, uint32_t off, uint32_t len) {
        __syncwarp();
        const uint32_t lo = off / kSlot, hi = (off + len - 1) / kSlot;
        if (lo + lane <= hi) {
            const uint32_t from = max(off, (lo + lane) * kSlot), end = min(off + len, (lo + lane + 1) * kSlot);
            give_back(first + lo + lane, (end - from) / (kSlot / kSlotUnits));
        }
    }
    __device__ __forceinline__ void give_back(uint32_t s, uint32_t units) {
        asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(&misc->empty[s % L::Slots])), "r"(units) : "memory");
    }
    // The predictor's ring is deeper than a layer: one warp gives back everything up to slot `end` behind a barrier that all
    // readers have met at, instead of every warp its own on the way from one exchange to the next.
    uint32_t given_back = 0;
    __device__ __forceinline__ void release_all(uint32_t end) {
        if (warp == kWorkers / kWarp - 1 && given_back + lane < end) give_back(given_back + lane, kSlotUnits);
        given_back = end;
    }

    // ---- MMA -----------------------------------------------------------------------------------------------
    // B fragment of 64 K at byte `k` of the limb rows, 8-column group q: activation rows 2q and 2q + 1
    __device__ __forceinline__ void load_b(const unsigned char* at, int q, uint32_t (&b)[4]) {
        const int limb = (lane >> 2) & 3, row = 2 * q + (lane >> 4);
        if (limb < 3 && row < rows) {
            const int4 v = *reinterpret_cast<const int4*>(at + (size_t)(row * kLimbs + limb) * L::XStride);
            b[0] = v.x; b[1] = v.y; b[2] = v.z; b[3] = v.w;
        } else {
            const uint32_t fill = limb == 3 ? 0x01010101u : 0u;
            b[0] = fill; b[1] = fill; b[2] = fill; b[3] = fill;
        }
    }
    // a tile's accumulators of one column group -> fp32 sums of weight rows g and g + 8 for activation row
    // 2 q + t / 2, in lanes of even t
    __device__ __forceinline__ void combine(const int (&d)[4], float unscale, float (&part)[2]) {
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const int first = d[2 * half], second = d[2 * half + 1];
            part[half] = (lane & 1) ? static_cast<float>(first - 64 * second) * 65536.0f
                                    : fmaf(static_cast<float>(second), 256.0f, static_cast<float>(first));
            part[half] += __shfl_xor_sync(0xffffffffu, part[half], 1);
            part[half] *= unscale;
        }
    }
    // Projection over all of K: warp w has K-slice w of every row; its sums go to red[w][row][kRedRow].  `tiles` is not known
    // to the compiler, so that all projections of this kind share one copy of the code.
    //
    // kAhead: one or two rows of the predictor take the weights of a projection and of the K-split one behind it from the ring
    // to registers while the exchange before them is under way.  The wait for the slots and the reads
    // then cost nothing between one exchange and the next (a predictor layer at one row 18.2 -> 16.9 thousand cycles).
    static constexpr int kRedRow = L::RedRows;
    static constexpr bool kAhead = !TALKER && ROWS <= 2;
    static constexpr int kSide = TALKER ? 2 : S::GuTiles;      // tiles side by side (the predictor: all of a phase)
    static constexpr int kSliceBlocks = S::Slice / 64;         // of the down projection; the o projection has 4
    static constexpr int kSliceSide = TALKER ? 2 : kSliceBlocks;
    static constexpr uint32_t kTile = S::J * 1024;              // a tile's blocks lie in one slot
    // The predictor's slots are given back behind a projection over all of K.  What is asked for before the next of these has to
    // fit the ring beside what has not been given back: held ahead, everything to the end of the K-split one behind it.
    static constexpr int kUnreleasedSlots = (S::OBytes + S::GuBytes + (kAhead ? S::DownBytes : 0)) / kSlot;
    static constexpr int kUnreleasedNext = (S::DownBytes + (S::QkvBytes > S::HeadBytes ? S::QkvBytes : S::HeadBytes) + (kAhead ? S::OBytes : 0)) / kSlot;
    static_assert(TALKER || (kUnreleasedSlots <= L::Slots && kUnreleasedNext <= L::Slots), "phases held fit the ring");
    static_assert(S::OutTiles * kSliceBlocks <= 8 * L::Slots, "a K-split phase fits the ring");
    int4 held_full[2 * kSide * S::J], held_slice[2 * kSliceSide];
    __device__ __forceinline__ const int4* ring_at(uint32_t first, uint32_t at) {
        return reinterpret_cast<const int4*>(smem + L::AtRing + (first + at / kSlot) % L::Slots * kSlot + at % kSlot) + lane;
    }
    __device__ __forceinline__ void hold_full(uint32_t first, int tiles, int t0) {
        const uint32_t off = (warp * tiles + t0) * kTile;
        if (!kAhead) wait_slot(first + (off + min(kSide, tiles) * kTile - 1) / kSlot);
#pragma unroll
        for (int i = 0; i < kSide; ++i) {
            if (!TALKER && i >= tiles) break;
            const uint32_t at = off + i * kTile;
            const int4* w = ring_at(first, at);
#pragma unroll
            for (int j = 0; j < 2 * S::J; ++j) held_full[2 * S::J * i + j] = w[kWarp * j];
        }
    }
    __device__ __forceinline__ void hold_slice(uint32_t first, int blocks, int j0) {
        if (!kAhead) wait_slot(first + ((warp % S::OutTiles * blocks + j0 + min(kSliceSide, blocks)) * 1024u - 1u) / kSlot);
        // two blocks at a time: 2 KB units never cross a slot
#pragma unroll
        for (int j = 0; j < kSliceSide; j += 2) {
            if (!TALKER && j >= blocks) break;
            const uint32_t at = (warp % S::OutTiles * blocks + j0 + j) * 1024u;
            const int4* w = ring_at(first, at);
#pragma unroll
            for (int i = 0; i < 4; ++i) held_slice[2 * j + i] = w[kWarp * i];
        }
    }
    // the weights of a layer's half, or of a head (blocks = 0)
    __device__ __forceinline__ void hold_ahead(int tiles, int blocks) {
        if constexpr (kAhead) {
            wait_slot(seq + tiles * S::J + S::OutTiles * blocks * 1024 / kSlot - 1);
            hold_full(seq, tiles, 0);
            if (blocks > 0 && warp < S::OutTiles) hold_slice(seq + tiles * S::J, blocks, 0);
        }
    }
    __device__ __forceinline__ void mma_full(int tiles, float unscale_mine) {
        float* red = reinterpret_cast<float*>(smem + L::AtU) + (size_t)warp * rows * kRedRow;
        const unsigned char* xs = smem + L::AtX + warp * 64 * S::J + 16 * (lane & 3);
        float u[NT];                                            // of the row this lane will hold: 2 q + t / 2
#pragma unroll
        for (int q = 0; q < NT; ++q) u[q] = __shfl_sync(0xffffffffu, unscale_mine, 2 * q + ((lane >> 1) & 1));
#pragma unroll 1
        for (int t0 = 0; t0 < tiles; t0 += kSide) {
            if (!kAhead) hold_full(seq, tiles, t0);
            constexpr int kChains = kSide * NT <= 4 ? 2 : 1;   // accumulators per tile (integers: any order)
            int acc[kChains][kSide][NT][4];
#pragma unroll
            for (int c = 0; c < kChains; ++c)
#pragma unroll
                for (int i = 0; i < kSide; ++i)
#pragma unroll
                    for (int q = 0; q < NT; ++q)
#pragma unroll
                        for (int e = 0; e < 4; ++e) acc[c][i][q][e] = 0;
            // all of B first where the registers allow it (the talker's is twice as long)
            uint32_t b[TALKER ? 1 : S::J][NT][4];
            auto fetch_b = [&](int j) {
#pragma unroll
                for (int q = 0; q < NT; ++q) load_b(xs + 64 * j, q, b[TALKER ? 0 : j][q]);
            };
            auto multiply = [&](int i, int j) {
                const int4 wa = held_full[2 * (S::J * i + j)], wb = held_full[2 * (S::J * i + j) + 1];
#pragma unroll
                for (int q = 0; q < NT; ++q) {
                    const uint32_t (&bq)[4] = b[TALKER ? 0 : j][q];
                    imma(acc[0][i][q], wa.x, wb.x, wa.y, wb.y, bq[0], bq[1]);
                    imma(acc[kChains - 1][i][q], wa.z, wb.z, wa.w, wb.w, bq[2], bq[3]);
                }
            };
            if (TALKER) {
#pragma unroll
                for (int j = 0; j < S::J; ++j) {
                    fetch_b(j);
#pragma unroll
                    for (int i = 0; i < kSide; ++i) multiply(i, j);
                }
            } else {
#pragma unroll
                for (int j = 0; j < S::J; ++j) fetch_b(j);
#pragma unroll
                for (int i = 0; i < kSide; ++i) {
                    if (i >= tiles) break;
#pragma unroll
                    for (int j = 0; j < S::J; ++j) multiply(i, j);
                }
            }
            // the talker's gate/up is as long as its ring: what comes next has to come into its places at once
            if (TALKER && tiles == S::GuTiles) release(seq, (warp * tiles + t0) * kTile, kSide * kTile);
            const int t = lane & 3;
#pragma unroll
            for (int i = 0; i < kSide; ++i) {
                if (!TALKER && i >= tiles) break;
#pragma unroll
                for (int q = 0; q < NT; ++q) {
                    const int row = 2 * q + (t >> 1);
                    if (kChains == 2) {
#pragma unroll
                        for (int e = 0; e < 4; ++e) acc[0][i][q][e] += acc[kChains - 1][i][q][e];
                    }
                    float part[2];
                    combine(acc[0][i][q], u[q], part);
                    if ((t & 1) == 0 && row < rows) {
                        float* out = red + row * kRedRow + (t0 + i) * 16 + (lane >> 2);
                        out[0] = part[0];
                        out[8] = part[1];
                    }
                }
            }
        }
    }
    // behind the barrier that joins the sums (predictor), or once they are on their way
    __device__ __forceinline__ void end_full(int tiles) {
        const uint32_t first = seq;
        seq += tiles * S::J;
        if (!TALKER) release_all(seq);
        else if (tiles != S::GuTiles) release(first, warp * tiles * kTile, tiles * kTile);
    }
    // K-split projection: a warp has 16 of the CTA's outputs over the whole slice and sends its partial sums to everybody: six
    // quads of three columns per row.  The predictor has four such tiles: with several column groups its warps w and w + 4
    // share one, half of the groups each, with one the upper four are done without.
    static constexpr int kShare = S::OutTiles == 4 && NT > 1 ? 2 : 1;
    static constexpr int kSliceWarps = S::OutTiles * kShare;
    __device__ __forceinline__ void mma_slice(int blocks, int b, uint32_t flag) {
        if (warp < kSliceWarps) {
            constexpr int NQ = NT / kShare;
            const int tile = warp % S::OutTiles, q0 = kShare == 1 ? 0 : warp / S::OutTiles * NQ;
            const unsigned char* xs = smem + L::AtX + 16 * (lane & 3);
            int acc[2][NQ][4];
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int q = 0; q < NQ; ++q)
#pragma unroll
                    for (int e = 0; e < 4; ++e) acc[i][q][e] = 0;
#pragma unroll 1
            for (int j0 = 0; j0 < blocks; j0 += kSliceSide) {
                if (!kAhead) hold_slice(seq, blocks, j0);
#pragma unroll
                for (int j = 0; j < kSliceSide; ++j) {
                    if (!TALKER && j >= blocks) break;
                    const int4 wa = held_slice[2 * j], wb = held_slice[2 * j + 1];
#pragma unroll
                    for (int q = 0; q < NQ; ++q) {
                        uint32_t bf[4];
                        load_b(xs + 64 * (j0 + j), q0 + q, bf);
                        imma(acc[j & 1][q], wa.x, wb.x, wa.y, wb.y, bf[0], bf[1]);
                        imma(acc[j & 1][q], wa.z, wb.z, wa.w, wb.w, bf[2], bf[3]);
                    }
                }
            }
#pragma unroll
            for (int q = 0; q < NQ; ++q) {
                const int t = lane & 3;
                const int row = 2 * (q0 + q) + (t >> 1);
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[0][q][e] += acc[1][q][e];
                float part[2];
                combine(acc[0][q], row < rows ? misc->unscale[row] : 1.0f, part);
                // lane -> (row of the pair, quad): column c of the row sits in lane 4 (c % 8) + 2 (row % 2)
                const int pair = lane >> 4, quad = lane & 15;
                uint32_t v[3];
#pragma unroll
                for (int e = 0; e < 3; ++e) {
                    const int c = min(3 * quad + e, 15);
                    const float lo = __shfl_sync(0xffffffffu, part[0], 4 * (c & 7) + 2 * pair);
                    const float hi = __shfl_sync(0xffffffffu, part[1], 4 * (c & 7) + 2 * pair);
                    v[e] = __float_as_uint(c < 8 ? lo : hi);
                }
                if (quad < 6 && 2 * (q0 + q) + pair < rows) {
                    put_quad(part_at(b, slice, rank, 2 * (q0 + q) + pair) + tile * 6 + quad, v[0], v[1], v[2], flag);
                }
            }
            if (TALKER) release(seq, warp * blocks * 1024u, blocks * 1024u);
        }
        seq += (uint32_t)(S::OutTiles * blocks * 1024) / kSlot;         // (predictor: given back with the next phase)
    }

    // ---- norm and conversion ----------------------------------------------------------------------------------
    // RMSNorm of the hidden rows in U into limbs; warp w keeps its K-slice.  Returns the unscale factor of row `lane`.
    __device__ __forceinline__ float norm_to_limbs(const uint32_t (&nw)[S::J], bf16* norm_out) {
        const bf16* hid = reinterpret_cast<const bf16*>(smem + L::AtU);
        float* partial = reinterpret_cast<float*>(smem + L::AtQkv);
        // thread t of the stand-alone kernel sums elements t, t + 256, ...
        if (ROWS <= 2) {
#pragma unroll
            for (int r = 0; r < ROWS; ++r) {
                float ss = 0.0f;
#pragma unroll
                for (int i = 0; i < S::H / kWorkers; ++i) {
                    const float v = bf2f(hid[r * S::H + tid + i * kWorkers]);
                    ss = fmaf(v, v, ss);
                }
                partial[r * kWorkers + tid] = ss;
            }
            sync_workers();
        } else {
            // two such threads' sums to a thread, two rows at a time; then a warp per row instead of every warp every row
            // (8 rows: a norm 4,370 cycles before)
#pragma unroll 2
            for (int r = tid >> 7; r < rows; r += 2) {
                float lo = 0.0f, hi = 0.0f;
#pragma unroll
                for (int i = 0; i < S::H / kWorkers; ++i) {
                    const uint32_t x = reinterpret_cast<const uint32_t*>(hid + r * S::H + i * kWorkers)[tid & 127];
                    lo = fmaf(bf_lo(x), bf_lo(x), lo);
                    hi = fmaf(bf_hi(x), bf_hi(x), hi);
                }
                reinterpret_cast<float2*>(partial + r * kWorkers)[tid & 127] = make_float2(lo, hi);
            }
            sync_workers();
            if (warp < rows) {
                const float total = tree_sum_256(partial + warp * kWorkers, lane);
                if (lane == 0) misc->inverse[warp] = rsqrtf(total / static_cast<float>(S::H) + a.eps);
            }
            sync_workers();
        }
        float unscale_mine = 1.0f;
        const int at = warp * 64 * S::J + 2 * S::J * lane;
        unsigned char* xs = smem + L::AtX;
#pragma unroll(ROWS <= 4 ? ROWS : 4)
        for (int r = 0; r < rows; ++r) {
            const float inv = ROWS <= 2 ? rsqrtf(tree_sum_256(partial + r * kWorkers, lane) / static_cast<float>(S::H) + a.eps)
                                        : misc->inverse[r];
            uint32_t raw[S::J];
            const uint32_t* src = reinterpret_cast<const uint32_t*>(hid + r * S::H + at);
#pragma unroll
            for (int m = 0; m < S::J; ++m) {
                const uint32_t x = src[m];
                const float lo = rbf(bf_lo(x) * inv) * bf_lo(nw[m]);
                const float hi = rbf(bf_hi(x) * inv) * bf_hi(nw[m]);
                raw[m] = page::pack_bf16x2(lo, hi);
            }
            if (TALKER && norm_out != nullptr) {
                uint32_t* dst = reinterpret_cast<uint32_t*>(norm_out + (size_t)r * S::H + at);
#pragma unroll
                for (int m = 0; m < S::J; ++m) dst[m] = raw[m];
            }
            const float u = to_limbs<S::J>(raw, xs + (size_t)r * kLimbs * L::XStride + at, L::XStride);
            if (lane == r) unscale_mine = u;
        }
        __syncwarp();
        return unscale_mine;
    }
    __device__ __forceinline__ void load_norm(const bf16* w, uint32_t (&nw)[S::J]) {
        const uint32_t* src = reinterpret_cast<const uint32_t*>(w + warp * 64 * S::J + 2 * S::J * lane);
#pragma unroll
        for (int m = 0; m < S::J; ++m) nw[m] = src[m];
    }
    // rows of a K-slice held in shared memory ([rows][64 Q], 2 Q elements a lane) -> limbs; warp r has row r
    template <int Q>
    __device__ __forceinline__ void slice_to_limbs(const unsigned char* src, int row_bytes) {
        if (warp < rows) {
            uint32_t raw[Q];
            const uint32_t* s = reinterpret_cast<const uint32_t*>(src + (size_t)warp * row_bytes) + Q * lane;
#pragma unroll
            for (int m = 0; m < Q; ++m) raw[m] = s[m];
            const float u = to_limbs<Q>(raw, smem + L::AtX + (size_t)warp * kLimbs * L::XStride + 2 * Q * lane, L::XStride);
            if (lane == 0) misc->unscale[warp] = u;
        }
        sync_workers();
    }

    // ---- exchanges ---------------------------------------------------------------------------------------------
    __device__ __forceinline__ Quad* part_at(int b, int s, int rk, int r) {
        return a.exchange + (((b * kSlices + s) * kRanks + rk) * kRowsMost + r) * (2 * S::Groups);
    }
    __device__ __forceinline__ Quad* group_quad(int at) {
        return a.exchange + reinterpret_cast<const uint32_t*>(smem + L::AtPages)[at / kPageQuads] + at % kPageQuads;
    }
    __device__ __forceinline__ Quad* group_at(int kind_base, int quads_per_row, int b, int rk, int r, int quad) {
        return group_quad(kind_base + ((b * kRanks + rk) * kRowsMost + r) * quads_per_row + quad);
    }
    // One value per lane (lanes < n, n a multiple of 2) -> quads of six bf16, sent by the first ceil(n / 6) lanes
    __device__ __forceinline__ void put_values(float v, int n, Quad* dst, uint32_t flag) {
        const float next = __shfl_down_sync(0xffffffffu, v, 1);
        const uint32_t pair = page::pack_bf16x2(v, next);
        const uint32_t w0 = __shfl_sync(0xffffffffu, pair, min(6 * lane, 31));
        const uint32_t w1 = __shfl_sync(0xffffffffu, pair, min(6 * lane + 2, 31));
        const uint32_t w2 = __shfl_sync(0xffffffffu, pair, min(6 * lane + 4, 31));
        if (6 * lane < n) put_quad(dst + lane, w0, w1, w2, flag);
    }

    // The partial sums of all groups, added up in slice order, times `scales`, onto the residual: the new hidden rows
    // in U (and this CTA's own columns in Own).
    __device__ __forceinline__ void collect_partials(const float* scales, int b, uint32_t flag) {
        bf16* own = reinterpret_cast<bf16*>(smem + L::AtOwn);
        bf16* hid = reinterpret_cast<bf16*>(smem + L::AtU);
        // group g of a row: columns 16 (g / 3) + 6 (g % 3) .. + 5 (+ 3 for the last of a tile)
        auto column_of = [](int g) { return 16 * (g / 3) + 6 * (g % 3); };
        auto sum_group = [&](int rk, int r, int g, const bf16* base_cols, uint32_t (&packed)[3]) {
            const int col = column_of(g), most = g % 3 == 2 ? 3 : 5;
            float sc[6], bs[6];
#pragma unroll
            for (int e = 0; e < 6; ++e) {
                sc[e] = scales[rk * S::Out + col + min(e, most)];
                bs[e] = bf2f(base_cols[col + min(e, most)]);
            }
            const Quad* p[2 * kSlices];
            Quad v[2 * kSlices];
#pragma unroll
            for (int s = 0; s < kSlices; ++s) {
                p[2 * s] = part_at(b, s, rk, r) + 2 * g;
                p[2 * s + 1] = p[2 * s] + 1;
            }
            poll(p, v, flag);
            float out[6];
#pragma unroll
            for (int e = 0; e < 6; ++e) {
                float sum = 0.0f;
#pragma unroll
                for (int s = 0; s < kSlices; ++s) {
                    const Quad& x = v[2 * s + e / 3];
                    sum += __uint_as_float(e % 3 == 0 ? x.x : (e % 3 == 1 ? x.y : x.z));
                }
                out[e] = fmaf(sum, sc[e], bs[e]);
            }
#pragma unroll
            for (int e = 0; e < 3; ++e) packed[e] = page::pack_bf16x2(out[2 * e], out[2 * e + 1]);
        };
        auto store_group = [&](bf16* row_columns, int g, const uint32_t (&packed)[3]) {
            uint32_t* d = reinterpret_cast<uint32_t*>(row_columns + column_of(g));
            d[0] = packed[0];
            d[1] = packed[1];
            if (g % 3 != 2) d[2] = packed[2];
        };
        if constexpr (L::OneHop) {
            static_assert(TALKER || kRanks * S::Groups <= kWorkers, "one pass");
            const int rk = tid / S::Groups, g = tid % S::Groups;
            if (tid < kRanks * S::Groups) {
                uint32_t packed[3];
                sum_group(rk, 0, g, own + rk * S::Out, packed);
                store_group(own + rk * S::Out, g, packed);
                store_group(hid + rk * S::Out, g, packed);
            }
        } else {
            const int bh = flip(kHid);
            const uint32_t flag_h = next_flag();
#pragma unroll 1
            for (int i = tid; i < rows * S::Groups; i += kWorkers) {
                const int r = i / S::Groups, g = i % S::Groups;
                uint32_t packed[3];
                bf16* mine = own + r * S::Out;
                sum_group(rank, r, g, mine, packed);
                store_group(mine, g, packed);
                put_quad(group_at(kAtHidden, S::Groups, bh, rank, r, g), packed[0], packed[1], packed[2], flag_h);
            }
            // a thread's quads, up to six, requested together
            constexpr int kEach = (ROWS * kRanks * S::Groups + kWorkers - 1) / kWorkers < 6 ? (ROWS * kRanks * S::Groups + kWorkers - 1) / kWorkers : 6;
#pragma unroll 1
            for (int i = tid; i < kRanks * rows * S::Groups; i += kEach * kWorkers) {
                const Quad* p[kEach];
                Quad v[kEach];
                int at[kEach], g[kEach];
#pragma unroll
                for (int k = 0; k < kEach; ++k) {
                    const int n = min(i + k * kWorkers, kRanks * rows * S::Groups - 1);
                    g[k] = n % S::Groups;
                    const int r = n / S::Groups % rows, rk = n / S::Groups / rows;
                    p[k] = group_at(kAtHidden, S::Groups, bh, rk, r, g[k]);
                    at[k] = r * S::H + rk * S::Out;
                }
                poll(p, v, flag_h);
#pragma unroll
                for (int k = 0; k < kEach; ++k) {
                    const uint32_t packed[3] = {v[k].x, v[k].y, v[k].z};
                    store_group(hid + at[k], g[k], packed);
                }
            }
        }
        sync_workers();
    }
    // quads of six bf16 from every CTA of the group ([rank][row][kGroupRow], the first per_row of them) -> rows of `row_words`
    // words in shared memory, rank after rank (`rank_words` words each).  A thread's quads are requested together.
    __device__ __forceinline__ void collect_group(int per_row, int rank_words, int b, uint32_t flag, uint32_t* dst, int row_words) {
        constexpr int kEach = (ROWS * kRanks * kGroupRow + kWorkers - 1) / kWorkers;
        const int g = tid % kGroupRow, rk = tid / kGroupRow % kRanks;
        const Quad* p[kEach];
        Quad v[kEach];
        const int r0 = tid / (kGroupRow * kRanks);
        if (g < per_row && r0 < rows) {
#pragma unroll
            for (int i = 0; i < kEach; ++i) p[i] = group_at(kAtGroup, kGroupRow, b, rk, min(r0 + 2 * i, rows - 1), g);
            poll(p, v, flag);
#pragma unroll
            for (int i = 0; i < kEach; ++i) {
                const int r = r0 + 2 * i;
                if (r < rows) {
                    uint32_t* d = dst + r * row_words + rk * rank_words + 3 * g;
                    d[0] = v[i].x;
                    if (3 * g + 1 < rank_words) d[1] = v[i].y;
                    if (3 * g + 2 < rank_words) d[2] = v[i].z;
                }
            }
        }
        sync_workers();
    }

    // ---- attention ---------------------------------------------------------------------------------------------
    __device__ __forceinline__ bf16* page_at(const KvLayout& kv, int row, int page, bool value) {
        const int pid = kv.page_table[(size_t)row * kv.table_stride + page];
        bf16* slab = kv.slabs[pid >> kv.slab_shift];
        return slab + (long long)(pid & ((1 << kv.slab_shift) - 1)) * kv.page_elems + (value ? kv.v_offset : kv.k_offset)
               + (size_t)slice * (kPageTokens * 128);
    }
    struct HeadNorm {
        bf16 q[4], k[4];
    };
    // cos | sin of the head vectors this warp rotates: fixed for a launch (talker) or a position (predictor)
    static constexpr int kJobs = (3 * ROWS + 7) / 8;
    uint32_t cs[TALKER ? kJobs : 1][2];                      // (the predictor's rows are all at one position)
    __device__ __forceinline__ void load_rotations(int position) {
#pragma unroll
        for (int i = 0; i < (TALKER ? kJobs : 1); ++i) {
            const int job = warp + 8 * i;
            if (TALKER) position = misc->position[job < 3 * rows ? job / 3 : 0];
            const uint32_t* at = a.rope_table + (size_t)position * 64 + lane;
            cs[i][0] = at[0];
            cs[i][1] = at[32];
        }
    }
    // q heads of every row (and the new key where this CTA will need it) from the exchanged projections: per-head
    // RMSNorm and rotation, one warp per head vector, lane l dims l, l + 32, l + 64, l + 96
    template <class Needs>
    __device__ __forceinline__ void rotate_heads(const HeadNorm& hn, Needs needs) {
        const bf16* qkv = reinterpret_cast<const bf16*>(smem + L::AtQkv);
        float* qs = reinterpret_cast<float*>(smem + L::AtQ);
        bf16* knew = reinterpret_cast<bf16*>(smem + L::AtKNew);
#pragma unroll
        for (int i = 0; i < kJobs; ++i) {
            const int job = warp + 8 * i;
            const int r = job / 3, h = job % 3;
            if (job >= 3 * rows || !needs(r, h == 2)) continue;
            const bf16* src = qkv + r * 512 + h * 128;
            float x[4], o[4];
            bf16 w[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                x[j] = bf2f(src[lane + 32 * j]);
                w[j] = h == 2 ? hn.k[j] : hn.q[j];
            }
            page::rotate(x, w, cs[TALKER ? i : 0][0], cs[TALKER ? i : 0][1], a.eps, o);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (h == 2) knew[r * 128 + lane + 32 * j] = f2bf(o[j]);
                else qs[r * 256 + h * 128 + lane + 32 * j] = o[j];
            }
        }
        sync_workers();
    }
    __device__ __forceinline__ void append(bf16* k, bf16* v, const bf16* knew, const bf16* vnew) {
        reinterpret_cast<uint2*>(k)[lane] = reinterpret_cast<const uint2*>(knew)[lane];
        reinterpret_cast<uint2*>(v)[lane] = reinterpret_cast<const uint2*>(vnew)[lane];
    }

    // ---- the predictor's attention over pages in shared memory (LocalKv)
    // 16-byte piece of K of token `t`: pieces of odd tokens change halves, so that a fragment load meets every bank once
    static __device__ __forceinline__ int k_piece(int t, int piece) { return t * 256 + ((piece ^ ((t & 1) << 2)) << 4); }
    // byte of V of token `t` behind its dimension's 32: the words of an MMA lane, tokens 2 tig (+ 1) and 8 more, lie together
    static __device__ __forceinline__ int v_token(int t) { return ((t & 7) >> 1) * 8 + (t >> 3) * 4 + (t & 1) * 2; }
    __device__ __forceinline__ unsigned char* local_page(int row, int index) {
        return smem + L::AtKv + (row * S::Layers + index) * L::KvPage;
    }
    __device__ __forceinline__ void clear_local_values() {
        // places of tokens to come: their probability is zero, and zero times what lies there has to be zero
        for (int i = tid; i < ROWS * S::Layers * (L::KvPage / 2 / 16); i += kWorkers) {
            const int page = i / (L::KvPage / 2 / 16), at = i % (L::KvPage / 2 / 16);
            reinterpret_cast<int4*>(smem + L::AtKv + page * L::KvPage + L::KvPage / 2)[at] = make_int4(0, 0, 0, 0);
        }
    }
    // A row's scores are computed by all of its warps (8 / ROWS), its 128 dimensions, 16 to a tile, are dealt to them.
    // The arithmetic is that of q3t_attention_page.cuh: a value does not depend on the tile that it is computed in.
    __device__ __forceinline__ void local_attention(const HeadNorm& hn, int index, int pos) {
        const bf16* qkv = reinterpret_cast<const bf16*>(smem + L::AtQkv);
        bf16* qs = reinterpret_cast<bf16*>(smem + L::AtQ);                 // [row][head][128]
#pragma unroll
        for (int i = 0; i < (4 * ROWS + 7) / 8; ++i) {
            // four vectors a row: two query heads, key, value
            const int job = warp + 8 * i, r = job >> 2, h = job & 3;
            if (job >= 4 * rows) continue;
            unsigned char* page = local_page(r, index);
            const bf16* src = qkv + r * 512 + h * 128;
            if (h == 3) {
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    *reinterpret_cast<bf16*>(page + L::KvPage / 2 + (lane + 32 * j) * 32 + v_token(pos)) = src[lane + 32 * j];
                continue;
            }
            float x[4], o[4];
            bf16 w[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                x[j] = bf2f(src[lane + 32 * j]);
                w[j] = h == 2 ? hn.k[j] : hn.q[j];
            }
            page::rotate(x, w, cs[0][0], cs[0][1], a.eps, o);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                bf16* at = h == 2 ? reinterpret_cast<bf16*>(page + k_piece(pos, 4 * j + (lane >> 3))) + (lane & 7)
                                  : qs + r * 256 + h * 128 + lane + 32 * j;
                *at = f2bf(o[j]);
            }
        }
        sync_workers();
        constexpr int kWarpsRow = 8 / ROWS;
        const int r = warp / kWarpsRow, gid = lane >> 2, tig = lane & 3;
        const unsigned char* page = local_page(r, index);
        float sc[2][4] = {};
        const bool real = gid < 2;
#pragma unroll
        for (int jj = 0; jj < 4; ++jj) {
            const int4 q = real ? *reinterpret_cast<const int4*>(qs + r * 256 + gid * 128 + 32 * jj + 8 * tig) : make_int4(0, 0, 0, 0);
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) {
                const int4 k = *reinterpret_cast<const int4*>(page + k_piece(8 * nt + gid, 4 * jj + tig));
                page::mma_bf16_16816(sc[nt], (uint32_t)q.x, 0u, (uint32_t)q.y, 0u, (uint32_t)k.x, (uint32_t)k.y);
                page::mma_bf16_16816(sc[nt], (uint32_t)q.z, 0u, (uint32_t)q.w, 0u, (uint32_t)k.z, (uint32_t)k.w);
            }
        }
        float mx, lsum;
        uint32_t ph[2], pl[2];
        page::probabilities(sc, pos + 1, rsqrtf(128.0f), tig, mx, lsum, ph, pl);
        const float inv0 = 1.0f / __shfl_sync(0xffffffffu, lsum, 0);
        const float inv1 = 1.0f / __shfl_sync(0xffffffffu, lsum, 4);
        bf16* att = reinterpret_cast<bf16*>(smem + L::AtAtt) + r * S::Slice;
#pragma unroll
        for (int u = 0; u < ROWS; ++u) {
            const int dim = 16 * (warp % kWarpsRow * ROWS + u) + gid;
            const uint2 lo = *reinterpret_cast<const uint2*>(page + L::KvPage / 2 + dim * 32 + tig * 8);
            const uint2 hi = *reinterpret_cast<const uint2*>(page + L::KvPage / 2 + (dim + 8) * 32 + tig * 8);
            float o[4] = {};
            page::mma_bf16_16816(o, lo.x, hi.x, lo.y, hi.y, ph[0], ph[1]);
            page::mma_bf16_16816(o, lo.x, hi.x, lo.y, hi.y, pl[0], pl[1]);
            if (tig == 0) {
                att[dim] = f2bf(o[0] * inv0);
                att[128 + dim] = f2bf(o[1] * inv1);
                att[dim + 8] = f2bf(o[2] * inv0);
                att[128 + dim + 8] = f2bf(o[3] * inv1);
            }
        }
        sync_workers();
    }

    // More rows: the predictor's caches are one page; warp r of every CTA of the group attends for row r.
    __device__ __forceinline__ void predictor_attention(const HeadNorm& hn, page::Fragments& f, bf16* k, bf16* v, int pos) {
        const bf16* qkv = reinterpret_cast<const bf16*>(smem + L::AtQkv);
        const bf16* knew = reinterpret_cast<const bf16*>(smem + L::AtKNew);
        rotate_heads(hn, [](int, bool) { return true; });
        if (warp < rows) {
            const int r = warp;
            page::patch(f, knew + r * 128, qkv + r * 512 + 384, pos, lane);
            if (rank == r) append(k + pos * 128, v + pos * 128, knew + r * 128, qkv + r * 512 + 384);
            float mx, lsum, o[8][4];
            page::attend(f, reinterpret_cast<const float*>(smem + L::AtQ) + r * 256, pos + 1, rsqrtf(128.0f), lane, mx, lsum, o);
            const float inv0 = 1.0f / __shfl_sync(0xffffffffu, lsum, 0);
            const float inv1 = 1.0f / __shfl_sync(0xffffffffu, lsum, 4);
            if ((lane & 3) == 0) {
                bf16* att = reinterpret_cast<bf16*>(smem + L::AtAtt) + r * S::Slice + 8 * (lane >> 2);
#pragma unroll
                for (int c = 0; c < 2; ++c)
#pragma unroll
                    for (int half = 0; half < 2; ++half) {
                        const float inv = c == 0 ? inv0 : inv1;
                        int4 packed;
                        packed.x = (int)page::pack_bf16x2(o[0][2 * half + c] * inv, o[1][2 * half + c] * inv);
                        packed.y = (int)page::pack_bf16x2(o[2][2 * half + c] * inv, o[3][2 * half + c] * inv);
                        packed.z = (int)page::pack_bf16x2(o[4][2 * half + c] * inv, o[5][2 * half + c] * inv);
                        packed.w = (int)page::pack_bf16x2(o[6][2 * half + c] * inv, o[7][2 * half + c] * inv);
                        *reinterpret_cast<int4*>(att + c * 128 + 64 * half) = packed;
                    }
            }
        }
        sync_workers();
    }

    // Talker: the slots of a row (q3t_attention_page.cuh) are the group's 16 CTAs, counted from one that depends on the
    // row, so that the rows of a batch spread.  (Blocks: the fewer CTAs hold parts of a row, the fewer partial results
    // everybody has to collect; the more pages a CTA has to fetch.)
    static_assert(kRanks == page::kSlots && kWorkers / kWarp == page::kClasses, "a CTA per slot, a warp per class");
    struct Walk {
        int row, page;
        bf16 *k, *v;          // its rows in layer 0
        bool any;
    };
    __device__ __forceinline__ int pages_of(int row) { return misc->position[row] / kPageTokens + 1; }
    __device__ __forceinline__ int slots_of(int row) { return page::slots_of(pages_of(row)); }
    __device__ __forceinline__ int my_slot(int row) { return (rank - 2 * row) & (kRanks - 1); }
    __device__ __forceinline__ int rank_of(int row, int slot) { return (slot + 2 * row) & (kRanks - 1); }
    __device__ __forceinline__ Walk first_page() {
        Walk w{0, 0, nullptr, nullptr, false};
        for (w.row = 0; w.row < rows; ++w.row) {
            w.page = page::class_page(my_slot(w.row), (warp - w.row) & 7);
            if (w.page < pages_of(w.row)) {
                w.k = page_at(a.kv, w.row, w.page, false);
                w.v = page_at(a.kv, w.row, w.page, true);
                w.any = true;
                return w;
            }
        }
        return w;
    }
    __device__ __forceinline__ int older_in(int row, int pg) { return min(kPageTokens, misc->position[row] - pg * kPageTokens); }
    __device__ __forceinline__ void talker_attention(const HeadNorm& hn, long long layer_elems, page::Fragments& f, const Walk& w0) {
        const bf16* qkv = reinterpret_cast<const bf16*>(smem + L::AtQkv);
        const bf16* knew = reinterpret_cast<const bf16*>(smem + L::AtKNew);
        float* acc_s = reinterpret_cast<float*>(smem + L::AtX);                  // [row][class][head][128]
        float* m_s = acc_s + ROWS * 8 * 2 * 128;                                  // [row][class][head]
        float* l_s = m_s + ROWS * 8 * 2;
        float* out_s = l_s + ROWS * 8 * 2;                                        // [row][head][132]: max, sum, weighted V
        bf16* att = reinterpret_cast<bf16*>(smem + L::AtAtt);
        const float scale = rsqrtf(128.0f);
        rotate_heads(hn, [&](int r, bool key) { return key ? (pages_of(r) - 1) / page::kBlock % kRanks == my_slot(r) : my_slot(r) < slots_of(r); });
        if (w0.any) {
            bool loaded = true;
#pragma unroll 1
            for (int row = w0.row; row < rows; ++row) {
                const int np = pages_of(row), cls = (warp - row) & 7;
                page::Running run;
                page::start(run);
                const int first = page::class_page(my_slot(row), cls);
#pragma unroll 1
                for (int pg = first; pg < np; pg += page::kPageStep) {
                    bf16 *kp = w0.k + layer_elems, *vp = w0.v + layer_elems;
                    if (!loaded) {
                        kp = page_at(a.kv, row, pg, false) + layer_elems;
                        vp = page_at(a.kv, row, pg, true) + layer_elems;
                        page::load(f, kp, vp, older_in(row, pg), lane);
                    }
                    loaded = false;
                    const int t_new = misc->position[row] - pg * kPageTokens;
                    if (t_new < kPageTokens) {
                        page::patch(f, knew + row * 128, qkv + row * 512 + 384, t_new, lane);
                        append(kp + t_new * 128, vp + t_new * 128, knew + row * 128, qkv + row * 512 + 384);
                    }
                    float mp, lp, op[8][4];
                    page::attend(f, reinterpret_cast<const float*>(smem + L::AtQ) + row * 256, min(kPageTokens, t_new + 1), scale, lane,
                                 mp, lp, op);
                    page::add(run, pg == first, mp, lp, op);
                }
                if (first < np) page::put_class(run, acc_s + (row * 8 + cls) * 256, m_s + (row * 8 + cls) * 2, l_s + (row * 8 + cls) * 2, lane);
            }
        }
        sync_workers();
        // the classes of this CTA, in order
        const int g = tid >> 7, d = tid & 127;
#pragma unroll 1
        for (int r = 0; r < rows; ++r) {
            const int np = pages_of(r), slot = my_slot(r);
            if (slot >= slots_of(r)) continue;
            float M, Lsum, A;
            page::merge_classes(acc_s + r * 8 * 256, m_s + r * 8 * 2, l_s + r * 8 * 2, slot, np, g, d, M, Lsum, A);
            float* dst = out_s + (r * 2 + g) * 132;
            if (d == 0) {
                dst[0] = M;
                dst[1] = Lsum;
                dst[130] = 0.0f;
                dst[131] = 0.0f;
            }
            dst[2 + d] = A;
        }
        sync_workers();
        const int b = flip(kAttnPart);
        const uint32_t flag = next_flag();
#pragma unroll 1
        for (int i = tid; i < rows * 88; i += kWorkers) {
            const int r = i / 88, q = i % 88;
            if (my_slot(r) >= slots_of(r)) continue;
            const float* src = out_s + (r * 2 + q / 44) * 132 + 3 * (q % 44);
            put_quad(group_at(kAtAttnPart, 88, b, rank, r, q), __float_as_uint(src[0]), __float_as_uint(src[1]), __float_as_uint(src[2]), flag);
        }
        float* gathered = reinterpret_cast<float*>(smem + L::AtX);              // [rank][132] of a head
        auto fold = [&](const float* from, int stride, int ranks, int dim) {
            return page::fold([&](int k, int n) { return from[k * stride + n]; }, ranks, dim, lane);
        };
        sync_workers();        // out_s has been read; the area is written again below
        if constexpr (ROWS == 1) {
            const int ranks = slots_of(0);
#pragma unroll 1
            for (int i = tid; i < ranks * 88; i += 3 * kWorkers) {
                const Quad* p[3];
                Quad v[3];
                float* dst[3];
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    const int n = min(i + k * kWorkers, ranks * 88 - 1);
                    const int rk = n / 88, q = n % 88;
                    p[k] = group_at(kAtAttnPart, 88, b, rank_of(0, rk), 0, q);
                    dst[k] = gathered + (rk * 2 + q / 44) * 132 + 3 * (q % 44);
                }
                poll(p, v, flag);
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    dst[k][0] = __uint_as_float(v[k].x);
                    dst[k][1] = __uint_as_float(v[k].y);
                    dst[k][2] = __uint_as_float(v[k].z);
                }
            }
            sync_workers();
            att[g * 128 + d] = f2bf(fold(gathered + g * 132, 2 * 132, ranks, d));
        } else {
            // CTA j of the group folds head j % 2 of row j / 2, then everybody collects the heads
            const int row = rank >> 1, head = rank & 1;
            const int bo = flip(kAttn);
            const uint32_t flag_o = next_flag();
            bf16* mine = reinterpret_cast<bf16*>(smem + L::AtStage);
            if (row < rows) {
                const int ranks = slots_of(row);
#pragma unroll 1
                for (int i = tid; i < ranks * 44; i += kWorkers) {
                    const int rk = i / 44, q = i % 44;
                    const Quad v = poll_one(group_at(kAtAttnPart, 88, b, rank_of(row, rk), row, head * 44 + q), flag);
                    float* dst = gathered + rk * 132 + 3 * q;
                    dst[0] = __uint_as_float(v.x);
                    dst[1] = __uint_as_float(v.y);
                    dst[2] = __uint_as_float(v.z);
                }
                sync_workers();
                if (warp < 4) mine[tid] = f2bf(fold(gathered, 132, ranks, tid));
                else if (tid < 132) mine[tid] = f2bf(0.0f);
                sync_workers();
                if (tid < 22) {
                    const uint32_t* w = reinterpret_cast<const uint32_t*>(mine) + 3 * tid;
                    put_quad(group_quad(kAtAttn + (bo * kRanks + rank) * 22 + tid), w[0], w[1], w[2], flag_o);
                }
            }
#pragma unroll 1
            for (int i = tid; i < 2 * rows * 22; i += kWorkers) {
                const int rk = i / 22, q = i % 22;
                const Quad v = poll_one(group_quad(kAtAttn + (bo * kRanks + rk) * 22 + q), flag_o);
                uint32_t* dst = reinterpret_cast<uint32_t*>(att + (rk >> 1) * S::Slice + (rk & 1) * 128) + 3 * q;
                dst[0] = v.x;
                if (q < 21) {
                    dst[1] = v.y;
                    dst[2] = v.z;
                }
            }
        }
        sync_workers();
    }

    __device__ __forceinline__ const LayerConst& constants(int index) { return reinterpret_cast<const LayerConst*>(smem + L::AtConst)[index]; }
    // ---- a layer -------------------------------------------------------------------------------------------------
    // In: hidden rows in U, this CTA's residual columns in Own, the layer's input norm weights and q/k/v weights (they are
    // fetched ahead).  Out: the same for what comes next, a projection of `next_tiles` tiles.
    __device__ __forceinline__ void layer(int index, int pos, int next_tiles, uint32_t (&nw)[S::J], const Walk& walk) {
        const LayerConst& lc = constants(index);
        HeadNorm hn;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            hn.q[j] = lc.q_norm[lane + 32 * j];
            hn.k[j] = lc.k_norm[lane + 32 * j];
        }
        // older cache rows: asked into the L2 a layer ahead (a page of one head is 4 KB), fetched behind the q/k/v exchange
        page::Fragments f;
        const long long layer_elems = index * a.kv_layer_elems;
        if (TALKER && walk.any && lane < 2 && index + 1 < S::Layers) {
            const bf16* p = (lane == 0 ? walk.k : walk.v) + layer_elems + a.kv_layer_elems;
            asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(kPageTokens * 128 * 2) : "memory");
        }
#pragma unroll 1
        for (int half = 0; half < 2; ++half) {
            // the units of this half's sums: an activation row's 32 q/k/v rows, or 24 of its channels (gate and up)
            constexpr int kChunks = S::Gu / 24;
            const int n = half == 0 ? 32 : 24, chunk = half == 0 ? 0 : warp % kChunks;
            const int qkv_row = rank < 8 ? 256 * slice + 32 * rank
                                         : (rank < 12 ? 2048 + 128 * slice + 32 * (rank - 8) : 3072 + 128 * slice + 32 * (rank - 12));
            const int channel = slice * S::Slice + rank * S::Gu + 24 * chunk + min(lane, 23);
            const float scale = half == 0 ? lc.qkv_s[qkv_row + lane] : lc.gu_s[channel];
            const float scale_up = half == 0 ? 0.0f : lc.gu_s[S::I + channel];
            const float u = norm_to_limbs(nw, nullptr);
            load_norm(half == 0 ? lc.post_norm : constants(index + 1 < S::Layers ? index + 1 : 0).in_norm, nw);
            sync_workers();           // everybody has read the hidden rows: their place takes the sums
            mma_full(half == 0 ? 2 : S::GuTiles, u);
            sync_workers();
            const int b = flip(kGroup);
            const uint32_t flag_g = next_flag();
            const float* red = reinterpret_cast<const float*>(smem + L::AtU);
#pragma unroll 1
            for (int unit = warp; unit < (half == 0 ? rows : rows * kChunks); unit += 8) {
                const int r = half == 0 ? unit : unit / kChunks;              // (8 is a multiple of kChunks)
                const float* at = red + r * kRedRow + 24 * chunk + min(lane, n - 1);
                float sum = 0.0f;
#pragma unroll
                for (int w = 0; w < 8; ++w) sum += at[w * rows * kRedRow];
                float value = sum * scale;
                if (half != 0) {
                    float sum_up = 0.0f;
#pragma unroll
                    for (int w = 0; w < 8; ++w) sum_up += at[w * rows * kRedRow + S::Gu];
                    const float up = sum_up * scale_up;
                    value = value / (1.0f + expf(-value)) * up;
                }
                put_values(value, n, group_at(kAtGroup, kGroupRow, b, rank, r, 4 * chunk), flag_g);
            }
            end_full(half == 0 ? 2 : S::GuTiles);
            if (half == 0) {
                if constexpr (!L::LocalKv) {
                    if (walk.any) {
                        if (!TALKER && index == 0 && pos > 0) await_appended();
                        page::load(f, walk.k + layer_elems, walk.v + layer_elems, TALKER ? older_in(walk.row, walk.page) : pos, lane);
                    }
                }
            }
            collect_group(half == 0 ? 6 : S::Gu / 6, half == 0 ? 16 : S::Gu / 2, b, flag_g,
                          reinterpret_cast<uint32_t*>(smem + (half == 0 ? L::AtQkv : L::AtAct)), half == 0 ? 256 : S::Slice / 2);
            if (half == 0) {
                if constexpr (TALKER) talker_attention(hn, layer_elems, f, walk);
                else if constexpr (L::LocalKv) local_attention(hn, index, pos);
                else predictor_attention(hn, f, walk.k + layer_elems, walk.v + layer_elems, pos);
                if (kEndsEarly && pos == 0 && index + 1 == S::Layers) {
                    static_assert(!kEndsEarly || !kAhead, "nothing is held for what is left out");
                    load_norm(constants(0).in_norm, nw);
                    return;
                }
            }
            // the o projection is over the group's 256 attention values, the down projection over its channels
            slice_to_limbs<S::Slice / 64>(smem + (half == 0 ? L::AtAtt : L::AtAct), S::Slice * 2);
            const int bp = flip(kPart);               // (here and not ahead of the early end: a buffer is taken for what is sent)
            const uint32_t flag = next_flag();
            mma_slice(half == 0 ? 4 : kSliceBlocks, bp, flag);
            hold_ahead(half == 0 ? S::GuTiles : next_tiles, half == 0 ? kSliceBlocks : (next_tiles == 2 ? 4 : 0));
            collect_partials(half == 0 ? lc.o_s : lc.down_s, bp, flag);
        }
    }

    // input rows of the first layer: `row_of(r)` in global memory -> U and Own
    template <class RowOf>
    __device__ __forceinline__ void load_hidden(RowOf row_of) {
        bf16* hid = reinterpret_cast<bf16*>(smem + L::AtU);
        bf16* own = reinterpret_cast<bf16*>(smem + L::AtOwn);
        constexpr int kVec = S::H / 8;
#pragma unroll 1
        for (int i = tid; i < rows * kVec; i += kWorkers) {
            const int r = i / kVec, v = i % kVec;
            const int4 x = reinterpret_cast<const int4*>(row_of(r))[v];
            reinterpret_cast<int4*>(hid + r * S::H)[v] = x;
            if (L::OneHop) {
                reinterpret_cast<int4*>(own)[v] = x;
            } else if (8 * v / S::Out == rank) {
                reinterpret_cast<int4*>(own + r * S::Out)[v - rank * (S::Out / 8)] = x;
            }
        }
        sync_workers();
    }

    // ---- predictor head and draw ---------------------------------------------------------------------------------
    __device__ __forceinline__ void predictor_head(int p, const float* scales, const uint32_t (&nw)[S::J]) {
        const float scale = scales[cta * 16 + (lane & 15)];
        const float u = norm_to_limbs(nw, nullptr);
        sync_workers();
        mma_full(S::HeadTiles, u);
        sync_workers();
        const int b = flip(kLogits);
        const uint32_t flag = next_flag();
        const float* red = reinterpret_cast<const float*>(smem + L::AtU);
        if (warp < rows) {
            float sum = 0.0f;
#pragma unroll
            for (int w = 0; w < 8; ++w) sum += red[(w * rows + warp) * kRedRow + (lane & 15)];
            put_values(sum * scale, 16, a.exchange + kAtLogits + ((b * kCtas + cta) * kRowsMost + warp) * 3, flag);
        }
        end_full(S::HeadTiles);
        if (p + 1 < kCodebooks) hold_ahead(2, 4);                // the next position's q/k/v
        const int bt = flip(kTokens);
        const uint32_t flag_t = next_flag();
        // one row: every CTA draws for itself (same logits, same state, same token); several: group r draws row r
        const int draws = ROWS == 1 ? 0 : (rank == 0 && slice < rows ? slice : -1);
        if (draws >= 0) {
            unsigned int* keys = reinterpret_cast<unsigned int*>(smem + L::AtSample);
            TopKScratch& scratch = *reinterpret_cast<TopKScratch*>(smem + L::AtSample + 2048 * 4);
            const Quad* at[2];
            Quad v[2];
            int quad[2];
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                quad[k] = min(tid + k * kWorkers, kCtas * 3 - 1);
                at[k] = a.exchange + kAtLogits + ((b * kCtas + quad[k] / 3) * kRowsMost + draws) * 3 + quad[k] % 3;
            }
            static_assert(kCtas * 3 <= 2 * kWorkers, "two quads a thread");
            poll(at, v, flag);
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const uint32_t w[3] = {v[k].x, v[k].y, v[k].z};
                const int first = quad[k] / 3 * 16 + quad[k] % 3 * 6;
#pragma unroll
                for (int e = 0; e < 3; ++e) {
                    if (quad[k] % 3 * 6 + 2 * e < 16) {
                        *reinterpret_cast<uint2*>(keys + first + 2 * e) = make_uint2(order_key(bf_lo(w[e])), order_key(bf_hi(w[e])));
                    }
                }
            }
            sync_workers();
            const SamplingParams sp = misc->sampling[draws];
            int token;
            if (sp.do_sample == 0) {
                unsigned long long best = 0ull;
#pragma unroll 1
                for (int t = tid; t < 2048; t += kWorkers) {
                    const unsigned long long k = ((unsigned long long)keys[t] << 12) | (unsigned long long)(4095 - t);
                    best = k > best ? k : best;
                }
#pragma unroll 1
                for (int o = 16; o > 0; o >>= 1) {
                    const unsigned long long other = __shfl_xor_sync(0xffffffffu, best, o);
                    best = other > best ? other : best;
                }
                if (lane == 0) scratch.warp_best[warp] = best;
                sync_workers();
#pragma unroll 1
                for (int w = 0; w < 8; ++w) best = scratch.warp_best[w] > best ? scratch.warp_best[w] : best;
                token = 4095 - (int)(best & 0xfffull);
            } else {
                token = sample_top_k_block<kWorkers, 2048 / kWorkers>(keys, 2048, min(sp.top_k, 2048), sp.top_p, sp.temperature, &misc->rng[draws],
                                                     scratch, tid, [] { sync_workers(); });
            }
            token = min(max(token, 0), 2047);
            if (ROWS == 1) {
                if (tid == 0) misc->token[0] = token;
            } else if (tid == 0) {
                put_quad(a.exchange + kAtTokens + bt * kRowsMost + draws, (uint32_t)token, 0u, 0u, flag_t);
            }
        }
        if (ROWS > 1 && tid < rows) {
            misc->token[tid] = min(max((int)poll_one(a.exchange + kAtTokens + bt * kRowsMost + tid, flag_t).x, 0), 2047);
        }
        sync_workers();
        if (tid < rows) misc->codes[tid][p] = (unsigned short)misc->token[tid];
    }

    // ---- the whole chain ------------------------------------------------------------------------------------------
    // A place on the die that the SM lies on, or none (-1).  CTAs of the first die take places from the first one up, those of the
    // second from the last one down.  The launch has as many CTAs as give both dies all of their places on a quiet device:
    // 128 where these lie as the places do, more on a part whose dies are filled unevenly (128 lie 60 and 68 on one of 72 and 76
    // SMs, where one session's frame was 1.5 % longer and three sessions' up to 4 %; 140 are enough there).  Where more CTAs
    // lie on a die than it has places, they wait until all have asked and take what the other die's left over, so that all
    // places are taken however the CTAs lie.  Who is done last clears the counts for the next launch.
    __device__ __forceinline__ int claim_place() {
        uint32_t sm;
        asm("mov.u32 %0, %%smid;" : "=r"(sm));
        const int die = a.places->die_of_sm[sm % kPlaceSms];
        const int share = die == 0 ? a.places->on_first : kCtas - a.places->on_first;
        const int n = (int)atomicAdd(a.claims + die, 1u);
        int most = share;
        if (n >= share) {
            // (all CTAs of the launch are resident, so this takes a microsecond; a run that is given up goes on with what it has)
            const unsigned long long until = now_ns() + kBudgetNs;
            int asked[2];
            for (;;) {
                asked[0] = (int)*reinterpret_cast<volatile uint32_t*>(a.claims);
                asked[1] = (int)*reinterpret_cast<volatile uint32_t*>(a.claims + 1);
                if (asked[0] + asked[1] >= (int)gridDim.x) break;
                if (now_ns() > until) {
                    *reinterpret_cast<volatile uint32_t*>(a.epoch + 1) = *reinterpret_cast<volatile uint32_t*>(a.epoch);
                    break;
                }
                __nanosleep(100);
            }
            most = max(share, kCtas - asked[1 - die]);
        }
        __threadfence();
        if (atomicInc(a.claims + 2, gridDim.x - 1) == gridDim.x - 1) {
            __threadfence();
            *reinterpret_cast<volatile uint32_t*>(a.claims) = 0u;
            *reinterpret_cast<volatile uint32_t*>(a.claims + 1) = 0u;
        }
        return n >= most ? -1 : (die == 0 ? n : kCtas - 1 - n);
    }
    __device__ __forceinline__ void run() {
        if (tid == 0) misc->place = claim_place();
        if (tid == 32) {
            for (int s = 0; s < L::Slots; ++s) {
                mbar_init(&misc->full[s], 1);
                mbar_init(&misc->empty[s], kSlotUnits);
                misc->asked[s] = 0u;
            }
            misc->abort = 0;
            misc->landed = 0u;
            misc->base = *reinterpret_cast<volatile uint32_t*>(a.epoch);
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        }
        __syncthreads();
        cta = misc->place;
        if (cta < 0) return;
        slice = cta / kRanks;
        rank = cta % kRanks;
        if (tid >= kWorkers && tid < kWorkers + kGroupPages) {
            reinterpret_cast<uint32_t*>(smem + L::AtPages)[tid - kWorkers] = a.places->pages[slice][tid - kWorkers];
        }
        if (tid < rows) {
            if (TALKER) {
                misc->position[tid] = a.positions[tid];
            } else {
                misc->rng[tid] = *a.table->rng[tid];
                misc->sampling[tid] = a.table->predictor[tid];
                misc->token[tid] = *a.table->sampled[tid];
            }
        }
        __syncthreads();
        base = misc->base;
        deadline = now_ns() + kBudgetNs;
        if (warp >= kWorkers / kWarp) {
            asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRequestRegisters));
            if (warp == kWorkers / kWarp && tc::elect_one()) request_weights();
            if (warp == kWorkers / kWarp + 1 && tc::elect_one()) count_landed();
            __syncwarp();
            __syncthreads();
            return;
        }
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kWorkerRegisters));
        uint32_t nw[S::J];
        load_norm(a.layers[0].in_norm, nw);
        for (int i = tid; i < S::Layers * (int)(sizeof(LayerConst) / 8); i += kWorkers) {
            reinterpret_cast<uint64_t*>(smem + L::AtConst)[i] = reinterpret_cast<const uint64_t*>(a.layers)[i];
        }
        // behind a row's attention values: zeros, so that its conversion is the next slice's (barriers follow)
        for (int i = tid; i < L::AttBytes / 4; i += kWorkers) reinterpret_cast<uint32_t*>(smem + L::AtAtt)[i] = 0u;
        hold_ahead(2, 4);
        if constexpr (TALKER) {
            const Walk walk = first_page();
            load_rotations(0);
            load_hidden([&](int r) { return a.hidden + (size_t)r * S::H; });
#pragma unroll 1
            for (int l = 0; l < S::Layers; ++l) layer(l, 0, l + 1 < S::Layers ? 2 : S::HeadTiles, nw, walk);
            load_norm(a.final_norm, nw);
            const float u = norm_to_limbs(nw, cta == 0 ? a.normalized : nullptr);
            sync_workers();
            mma_full(S::HeadTiles, u);
            sync_workers();
            const float* red = reinterpret_cast<const float*>(smem + L::AtU);
#pragma unroll 1
            for (int i = tid; i < rows * S::HeadRows; i += kWorkers) {
                const int r = i / S::HeadRows, n = i % S::HeadRows;
                float sum = 0.0f;
#pragma unroll
                for (int w = 0; w < 8; ++w) sum += red[(w * rows + r) * kRedRow + n];
                const int channel = cta * S::HeadRows + n;
                a.logits[(size_t)r * (kCtas * S::HeadRows) + channel] = f2bf(sum * a.head_s[0][channel]);
            }
        } else {
            Walk walk{warp, 0, nullptr, nullptr, !L::LocalKv && warp < rows};
            if constexpr (L::LocalKv) clear_local_values();        // (several barriers ahead of the first use)
            if (walk.any) {
                walk.k = page_at(a.kv, warp, 0, false);
                walk.v = page_at(a.kv, warp, 0, true);
            }
            if (tid < rows) misc->codes[tid][0] = (unsigned short)misc->token[tid];
            load_rotations(0);
            uint32_t head_norm[S::J];
            load_norm(a.final_norm, head_norm);
#pragma unroll 1
            for (int p = 0; p < kCodebooks; ++p) {
                const float* head_scales = p > 0 ? a.head_s[p - 1] : nullptr;
                load_hidden([&](int r) {
                    const int most = p == 1 ? kMaxVocab - 1 : kPredictorVocab - 1;
                    return p == 0 ? a.hidden + (size_t)r * S::H : a.projected[p - 1] + (size_t)min(max(misc->token[r], 0), most) * S::H;
                });
#pragma unroll 1
                for (int l = 0; l < S::Layers; ++l) layer(l, p, l + 1 < S::Layers || p == 0 ? 2 : S::HeadTiles, nw, walk);
                load_rotations(min(p + 1, kCodebooks - 1));              // the next position's
                if (p > 0) predictor_head(p, head_scales, head_norm);
                if constexpr (!L::LocalKv) say_appended(p + 1 == kCodebooks);
            }
            if (ROWS == 1 ? cta == 0 && tid == 0 : rank == 0 && slice < rows && tid == 0) {
                const int r = ROWS == 1 ? 0 : slice;
                *a.table->rng[r] = misc->rng[r];
            }
            // the frame's codes, once all are drawn: sixteen stores in the way of the draws cost a microsecond each
            sync_workers();
            if (cta == 0 && tid < rows * kCodebooks) {
                const int r = tid / kCodebooks, p = tid % kCodebooks;
                const unsigned short code = misc->codes[r][p];
                a.table->frame_tokens[r][p] = code;
                a.table->frame_codes[r][p] = code;
                if (a.table->host_codes[r] != nullptr) a.table->host_codes[r][p] = code;
            }
        }
        __syncthreads();        // no further requests
        if (given_up() && tid < L::Slots && misc->asked[tid] > 0) {
            // a copy that nobody waited for must have landed before the CTA leaves
            for (uint32_t polls = 0; polls < (1u << 14) && !mbar_try_wait(&misc->full[tid], (misc->asked[tid] - 1) & 1u); ++polls) {}
        }
        sync_workers();
        if (cta == 0 && tid == 0) {
            if (given_up()) {
                atomicAdd(&g_chain_errors, 1u);
                if (g_chain_error_sink != nullptr) atomicAdd_system(g_chain_error_sink, 1u);
            }
            *reinterpret_cast<volatile uint32_t*>(a.epoch) = base + step;
        }
    }
};

template <bool TALKER, int ROWS>
__global__ void __launch_bounds__(kThreads, 1) decode_chain_kernel(const __grid_constant__ ChainArgs a) {
    extern __shared__ __align__(128) unsigned char smem[];
    Chain<TALKER, ROWS> chain(a, smem);
    chain.run();
}

// ---- weights as streams ------------------------------------------------------------------------------------
// One 1 KB block per warp: lane l holds rows (l / 4) and (l / 4) + 8 of the tile, 16 bytes each at K offset 16 (l % 4).
enum PackPhase { kPackQkv, kPackO, kPackGateUp, kPackDown, kPackHead };

__global__ void pack_stream_kernel(const int8_t* __restrict__ w, uint8_t* __restrict__ dst, long long cta_stride, int phase, int H, int I,
                                   int tiles, int head_rows) {
    const int cta = blockIdx.x;
    const int slice = cta / kRanks, rank = cta % kRanks;
    const int lane = threadIdx.x % kWarp;
    const int warps = blockDim.x / kWarp;
    const bool split = phase == kPackO || phase == kPackDown;
    const int J = split ? (phase == kPackO ? 4 : I / 512) : H / 512;
    const int blocks = split ? tiles * J : 8 * tiles * J;
    for (int blk = blockIdx.y * warps + threadIdx.x / kWarp; blk < blocks; blk += gridDim.y * warps) {
        const int j = blk % J, tile = blk / J % tiles, part = blk / J / tiles;      // part: the K-slice of warp `part`
        int4 v[2];
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const int i = tile * 16 + half * 8 + lane / 4;          // row within the CTA's share
            long long row;
            int K = H, k0 = part * (H / 8);
            bool valid = true;
            if (phase == kPackQkv) {
                row = (rank < 8 ? 256 * slice + 32 * rank
                                : (rank < 12 ? 2048 + 128 * slice + 32 * (rank - 8) : 3072 + 128 * slice + 32 * (rank - 12))) + i;
            } else if (phase == kPackO) {
                row = rank * (H / kRanks) + i;
                K = 2048;
                k0 = 256 * slice;
            } else if (phase == kPackDown) {
                row = rank * (H / kRanks) + i;
                K = I;
                k0 = (I / kSlices) * slice;
            } else if (phase == kPackGateUp) {
                const int gu = I / kCtas;
                row = (long long)(i < gu ? 0 : I) + slice * (I / kSlices) + rank * gu + (i < gu ? i : i - gu);
            } else {
                valid = i < head_rows;
                row = (long long)cta * head_rows + (valid ? i : 0);
            }
            v[half] = valid ? *reinterpret_cast<const int4*>(w + row * K + k0 + 64 * j + 16 * (lane % 4)) : make_int4(0, 0, 0, 0);
        }
        int4* out = reinterpret_cast<int4*>(dst + (size_t)cta * cta_stride + (size_t)blk * 1024);
        out[lane] = v[0];
        out[kWarp + lane] = v[1];
    }
}

// `fits`: false where the kernel was compiled (with other flags than the library's) for fewer registers than its warps hand out
// among themselves; they would wait for the rest of them for good.
template <bool TALKER, int ROWS>
cudaError_t configure_variant(bool& fits) {
    cudaFuncAttributes built;
    const cudaError_t e = cudaFuncGetAttributes(&built, decode_chain_kernel<TALKER, ROWS>);
    if (e != cudaSuccess) return e;
    fits = fits && kThreads * built.numRegs >= kWorkers * kWorkerRegisters + 4 * kWarp * kRequestRegisters;
    return cudaFuncSetAttribute(decode_chain_kernel<TALKER, ROWS>, cudaFuncAttributeMaxDynamicSharedMemorySize, Layout<TALKER, ROWS>::Bytes);
}

template <bool TALKER, int ROWS>
cudaError_t launch_variant(const ChainArgs& a, int grid, cudaStream_t stream) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = Layout<TALKER, ROWS>::Bytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, decode_chain_kernel<TALKER, ROWS>, a);
}

template <bool TALKER>
cudaError_t launch_rows(const ChainArgs& a, int grid, cudaStream_t stream) {
    if (a.rows <= 2) return a.rows == 1 ? launch_variant<TALKER, 1>(a, grid, stream) : launch_variant<TALKER, 2>(a, grid, stream);
    return a.rows <= 4 ? launch_variant<TALKER, 4>(a, grid, stream) : launch_variant<TALKER, 8>(a, grid, stream);
}

bool g_chain_fits[64] = {};

}  // namespace

cudaError_t configure_chain_kernels() {
    int device = 0, sms = 0, cooperative = 0;
    bool fits = true;
    cudaError_t e = cudaGetDevice(&device);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&cooperative, cudaDevAttrCooperativeLaunch, device);
    if (e == cudaSuccess) e = configure_variant<true, 1>(fits);
    if (e == cudaSuccess) e = configure_variant<true, 2>(fits);
    if (e == cudaSuccess) e = configure_variant<true, 4>(fits);
    if (e == cudaSuccess) e = configure_variant<true, 8>(fits);
    if (e == cudaSuccess) e = configure_variant<false, 1>(fits);
    if (e == cudaSuccess) e = configure_variant<false, 2>(fits);
    if (e == cudaSuccess) e = configure_variant<false, 4>(fits);
    if (e == cudaSuccess) e = configure_variant<false, 8>(fits);
    if (e == cudaSuccess && device >= 0 && device < 64) g_chain_fits[device] = fits && cooperative != 0 && sms >= kCtas && sms <= kPlaceSms;
    return e;
}

bool chain_available() {
    int device = 0;
    return cudaGetDevice(&device) == cudaSuccess && device >= 0 && device < 64 && g_chain_fits[device];
}

size_t chain_stream_bytes(bool talker) {
    return (size_t)kCtas * (talker ? (size_t)Shape<true>::Layers * Shape<true>::LayerBytes : (size_t)Shape<false>::Layers * Shape<false>::LayerBytes);
}
size_t chain_head_bytes(bool talker) { return (size_t)kCtas * (talker ? Shape<true>::HeadBytes : 15 * Shape<false>::HeadBytes); }
size_t chain_exchange_bytes() { return (size_t)kSharedQuads * sizeof(Quad) + (size_t)kPoolPages * kPlacePage + kPlacePage; }
size_t chain_pool_at(const void* exchange) {
    const size_t at = reinterpret_cast<uintptr_t>(exchange) + (size_t)kSharedQuads * sizeof(Quad);
    return (at + kPlacePage - 1) / kPlacePage * kPlacePage - reinterpret_cast<uintptr_t>(exchange);
}

cudaError_t launch_pack_layer(bool talker, int layer, const int8_t* qkv, const int8_t* o, const int8_t* gate_up, const int8_t* down,
                              uint8_t* stream_base, cudaStream_t stream) {
    const int H = talker ? 2048 : 1024, I = talker ? 6144 : 3072;
    const int layer_bytes = talker ? Shape<true>::LayerBytes : Shape<false>::LayerBytes;
    const long long cta = (long long)layer_bytes * (talker ? Shape<true>::Layers : Shape<false>::Layers);
    uint8_t* dst = stream_base + (size_t)layer * layer_bytes;
    const int out_tiles = H / kRanks / 16, gu_tiles = 2 * (I / kCtas) / 16;
    const dim3 grid(kCtas, 4);
    pack_stream_kernel<<<grid, 256, 0, stream>>>(qkv, dst, cta, kPackQkv, H, I, 2, 0);
    dst += 32 * H;
    pack_stream_kernel<<<grid, 256, 0, stream>>>(o, dst, cta, kPackO, H, I, out_tiles, 0);
    dst += (H / kRanks) * 256;
    pack_stream_kernel<<<grid, 256, 0, stream>>>(gate_up, dst, cta, kPackGateUp, H, I, gu_tiles, 0);
    dst += 2 * (I / kCtas) * H;
    pack_stream_kernel<<<grid, 256, 0, stream>>>(down, dst, cta, kPackDown, H, I, out_tiles, 0);
    return cudaGetLastError();
}

cudaError_t launch_pack_head(bool talker, int index, const int8_t* head, uint8_t* heads_base, cudaStream_t stream) {
    const int H = talker ? 2048 : 1024;
    const int bytes = talker ? Shape<true>::HeadBytes : Shape<false>::HeadBytes;
    const long long cta = (long long)bytes * (talker ? 1 : 15);
    pack_stream_kernel<<<dim3(kCtas, 4), 256, 0, stream>>>(head, heads_base + (size_t)index * bytes, cta, kPackHead, H, 0,
                                                           talker ? 2 : 1, talker ? 24 : 16);
    return cudaGetLastError();
}

cudaError_t launch_decode_chain(const ChainLaunch& c, cudaStream_t stream) {
    static_assert(sizeof(LayerConst) == sizeof(ChainLayer), "the same eight pointers");
    if (c.rows < 1 || c.rows > kRowsMost || !chain_available()) return cudaErrorInvalidValue;
    ChainArgs a;
    a.stream = c.stream; a.heads = c.heads; a.layers = reinterpret_cast<const LayerConst*>(c.layers); a.final_norm = c.final_norm;
    a.head_s = c.head_scales; a.hidden = c.hidden; a.normalized = c.normalized; a.logits = c.logits; a.projected = c.projected;
    a.table = c.table; a.positions = c.positions; a.kv = c.kv; a.kv_layer_elems = c.kv_layer_elems; a.rope_table = c.rope_table;
    a.exchange = static_cast<Quad*>(c.exchange); a.epoch = c.epoch; a.places = c.places; a.claims = c.claims; a.rows = c.rows; a.eps = kRmsEps;
    return c.talker ? launch_rows<true>(a, c.grid, stream) : launch_rows<false>(a, c.grid, stream);
}

// The last number used becomes 0, the run given up one that no launch reaches before the next restart, and no word of
// the exchange carries a number that will be used.
cudaError_t restart_chain_numbers(void* exchange, uint32_t* epoch, cudaStream_t stream) {
    cudaError_t e = cudaMemsetAsync(exchange, 0, chain_exchange_bytes(), stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(epoch, 0, sizeof(uint32_t), stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(epoch + 1, 0xff, sizeof(uint32_t), stream);
    return e;
}

unsigned int chain_error_count() {
    unsigned int v = 0;
    if (cudaMemcpyFromSymbol(&v, g_chain_errors, sizeof(v)) != cudaSuccess) return ~0u;
    return v;
}

cudaError_t set_chain_error_sink(unsigned int* device_visible_word) {
    return cudaMemcpyToSymbol(g_chain_error_sink, &device_visible_word, sizeof(device_visible_word));
}

}  // namespace q3t
