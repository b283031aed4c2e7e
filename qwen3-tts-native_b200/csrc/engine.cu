// Model / session / frame engine (see engine.hpp).

#include "engine.hpp"

#include <algorithm>
#include <atomic>
#include <chrono>
#include <cmath>
#include <cstddef>
#include <cstdlib>
#include <cstdio>
#include <cstring>
#include <functional>
#include <limits>
#include <numeric>

namespace q3t {

namespace {
constexpr int kTalkerLayers = 28;
constexpr int kPredictorLayers = 5;
constexpr int kResidualCodebooks = 15;
constexpr int kTalkerVocab = 3072;
constexpr int kTextVocab = 151936;
constexpr int kPredictorSequence = 16;
constexpr int kEos = 2150;
constexpr uint32_t kPhaseCreated = 0, kPhaseReady = 1, kPhasePrefilled = 2, kPhaseEnded = 3;

constexpr size_t kChainLeaves = 4ull << 30;      // device memory that has to stay free behind the decode chain's image

size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

int env_int(const char* name, int fallback) {
    const char* v = std::getenv(name);
    return v != nullptr && *v != '\0' ? std::atoi(v) : fallback;
}
}  // namespace

void check_cuda(cudaError_t status, const char* what) {
    if (status != cudaSuccess) {
        throw CudaFailure(std::string(what) + " failed: " + cudaGetErrorString(status));
    }
}

namespace {
std::atomic<int> g_fail_launch{0}, g_fail_allocation{0};
std::atomic<uint64_t> g_next_session_id{1};

// true exactly once, when an armed countdown reaches zero
bool countdown_fires(std::atomic<int>& countdown) {
    int left = countdown.load(std::memory_order_relaxed);
    while (left > 0) {
        if (countdown.compare_exchange_weak(left, left - 1, std::memory_order_relaxed)) return left == 1;
    }
    return false;
}
}  // namespace

void fail_launch_after(int n) { g_fail_launch.store(n > 0 ? n : 0); }
void fail_allocation_after(int n) { g_fail_allocation.store(n > 0 ? n : 0); }

void check_launch(cudaError_t status, const char* what) {
    if (status == cudaSuccess && countdown_fires(g_fail_launch)) status = cudaErrorLaunchOutOfResources;
    check_cuda(status, what);
}

// ------------------------------------------------------------------ what runs on a device at the moment

namespace {

// Chains wait between their CTAs, so two of them must not share the GPU's SMs: the chains of a device run one after the
// other, whatever streams (and models) they come from.  And a chain takes 128 SMs whole: launches of other frames or of a
// prompt beside it get on between two chains only (a frame of 23 sessions beside one session stepped alone took 25 ms
// instead of 6, a prompt of 64 positions 10 ms instead of 3.5).  So a frame that could run as a chain is made launch by
// launch, with the same bits, while the device is at work on something that is no chain.
//
// Frames are known by the workspace that they run on: its last frame's end is the event talker_stop.
struct Traffic {
    enum Kind { kChain, kInPlaceOfChain, kOther };
    struct Entry {
        const Workspace* workspace;
        int rows;
        Kind kind;
        bool enqueued;          // the whole frame is on its stream, talker_stop behind it
    };
    std::mutex mutex;
    std::vector<Entry> entries;
    cudaEvent_t chain_done = nullptr;
    cudaStream_t chain_stream = nullptr;
    std::chrono::steady_clock::time_point crowd_until{}, shared_until{};

    Entry* find(const Workspace* w) {
        for (Entry& e : entries) if (e.workspace == w) return &e;
        return nullptr;
    }
    void drop_finished() {
        for (size_t i = 0; i < entries.size();) {
            if (entries[i].enqueued && cudaEventQuery(entries[i].workspace->talker_stop) == cudaSuccess) {
                entries[i] = entries.back();
                entries.pop_back();
            } else {
                ++i;
            }
        }
        cudaGetLastError();     // "not ready" is no error
    }
    // Whether a frame of n rows that may run as a chain should.  Three and more sessions stepped alone get on faster side by
    // side, launch by launch, than chain after chain (frames/s of 3, 4, 6, 8, 16 of them: 737, 784, 841, 791, 802 against 635);
    // two are as fast either way (643 and 637), so that a second one joins a first that is made launch by launch instead of
    // waiting for it.  Their frames end together and begin one after the other, so that the first of a round sees nobody:
    // a crowd is remembered for a while.  Beside a lockstep frame the chain's is the shorter one (8 sessions and 3 alone
    // 8.0 ms against 9.6).
    bool chain_pays(const Workspace* w, int n) {
        const auto now = std::chrono::steady_clock::now();
        int alone = n == 1 ? 1 : 0;
        bool lockstep = n > 1, launches = false;
        for (const Entry& e : entries) {
            if (e.workspace == w) continue;
            if (e.kind == kOther) {
                shared_until = now + std::chrono::milliseconds(5);       // past the host's part between two prompts
                return false;
            }
            if (e.kind == kInPlaceOfChain && !e.enqueued) return false;
            launches = launches || e.kind == kInPlaceOfChain;
            if (e.rows == 1) ++alone;
            else lockstep = true;
        }
        if (now < shared_until) return false;
        if (lockstep) return true;
        if (alone >= 3) crowd_until = now + std::chrono::milliseconds(20);
        return !launches && now >= crowd_until;
    }
    // Whether nothing else is at work, nor was a moment ago: the lockstep chain takes 128 SMs for the predictor's part of a
    // frame, and what runs beside it gets the rest.  Launch by launch such a frame has the same bits.
    bool alone(const Workspace* w) {
        const auto now = std::chrono::steady_clock::now();
        drop_finished();
        for (const Entry& e : entries) {
            if (e.workspace == w) continue;
            shared_until = now + std::chrono::milliseconds(5);
            return false;
        }
        return now >= shared_until;
    }
    void enter(const Workspace* w, int rows, Kind kind) {
        Entry* e = find(w);
        if (e != nullptr) *e = Entry{w, rows, kind, false};
        else entries.push_back(Entry{w, rows, kind, false});
    }
    void leave(const Workspace* w) {
        for (size_t i = 0; i < entries.size(); ++i) {
            if (entries[i].workspace == w) {
                entries[i] = entries.back();
                entries.pop_back();
                return;
            }
        }
    }
};
Traffic* traffic_of(int device) {
    static Traffic* const all = new Traffic[64];       // outlives every session
    return device >= 0 && device < 64 ? &all[device] : nullptr;
}

// A prompt or a frame in the census, from its construction until it is known to have ended.
class InFlight {
public:
    InFlight(Traffic* traffic, const Workspace& w, int rows, Traffic::Kind kind) : traffic_(traffic), workspace_(&w) {
        if (traffic_ == nullptr) return;
        std::lock_guard<std::mutex> lock(traffic_->mutex);
        traffic_->enter(workspace_, rows, kind);
    }
    // a frame that may run as a chain: kind() tells whether it does
    InFlight(Traffic* traffic, const Workspace& w, int rows, bool never_chain) : traffic_(traffic), workspace_(&w) {
        std::lock_guard<std::mutex> lock(traffic_->mutex);
        traffic_->drop_finished();
        kind_ = !never_chain && traffic_->chain_pays(workspace_, rows) ? Traffic::kChain : Traffic::kInPlaceOfChain;
        traffic_->enter(workspace_, rows, kind_);
    }
    // a frame of more rows than a chain takes: alone() tells whether nothing else was at work when it entered the census
    struct Large {};
    InFlight(Traffic* traffic, const Workspace& w, int rows, Large) : traffic_(traffic), workspace_(&w) {
        std::lock_guard<std::mutex> lock(traffic_->mutex);
        alone_ = traffic_->alone(workspace_);
        traffic_->enter(workspace_, rows, Traffic::kOther);
    }
    InFlight(const InFlight&) = delete;
    InFlight& operator=(const InFlight&) = delete;
    // from here on the workspace's talker_stop tells the end
    void enqueued() {
        if (traffic_ == nullptr) return;
        std::lock_guard<std::mutex> lock(traffic_->mutex);
        if (Traffic::Entry* e = traffic_->find(workspace_)) e->enqueued = true;
        traffic_ = nullptr;
    }
    ~InFlight() {
        if (traffic_ == nullptr) return;
        std::lock_guard<std::mutex> lock(traffic_->mutex);
        traffic_->leave(workspace_);
    }
    Traffic::Kind kind() const { return kind_; }
    bool alone() const { return alone_; }
private:
    Traffic* traffic_;
    const Workspace* workspace_;
    Traffic::Kind kind_ = Traffic::kOther;
    bool alone_ = false;
};

// Held while a frame's chains are enqueued; whatever chain was enqueued by then, the next holder's stream waits for it, and
// for the frames that stand in for one.
class ChainTurn {
public:
    ChainTurn(Traffic* traffic, const Workspace& w) : traffic_(traffic), stream_(w.stream) {
        if (traffic_ == nullptr) return;
        lock_ = std::unique_lock<std::mutex>(traffic_->mutex);
        if (traffic_->chain_done == nullptr) {
            check_cuda(cudaEventCreateWithFlags(&traffic_->chain_done, cudaEventDisableTiming), "cudaEventCreate(chain order)");
        } else if (traffic_->chain_stream != stream_) {
            check_cuda(cudaStreamWaitEvent(stream_, traffic_->chain_done, 0), "cudaStreamWaitEvent(chain order)");
        }
        for (const Traffic::Entry& e : traffic_->entries) {
            if (e.workspace == &w || e.kind != Traffic::kInPlaceOfChain || !e.enqueued) continue;
            check_cuda(cudaStreamWaitEvent(stream_, e.workspace->talker_stop, 0), "cudaStreamWaitEvent(frame)");
        }
    }
    ~ChainTurn() {
        if (traffic_ == nullptr) return;
        cudaEventRecord(traffic_->chain_done, stream_);
        traffic_->chain_stream = stream_;
    }
private:
    Traffic* traffic_;
    cudaStream_t stream_;
    std::unique_lock<std::mutex> lock_;
};

}  // namespace

// ------------------------------------------------------------------ DeviceBuffer

DeviceBuffer::DeviceBuffer(size_t bytes) : bytes_(bytes) {
    if (bytes == 0) return;
    if (countdown_fires(g_fail_allocation)) throw std::bad_alloc();
    const cudaError_t e = cudaMalloc(&ptr_, bytes);
    if (e == cudaErrorMemoryAllocation) {
        cudaGetLastError();
        throw std::bad_alloc();
    }
    check_cuda(e, "cudaMalloc");
}
DeviceBuffer::DeviceBuffer(DeviceBuffer&& o) noexcept : ptr_(o.ptr_), bytes_(o.bytes_), owned_(o.owned_) {
    o.ptr_ = nullptr;
    o.bytes_ = 0;
}
DeviceBuffer& DeviceBuffer::operator=(DeviceBuffer&& o) noexcept {
    if (this != &o) {
        if (ptr_ != nullptr && owned_) cudaFree(ptr_);
        ptr_ = o.ptr_;
        bytes_ = o.bytes_;
        owned_ = o.owned_;
        o.ptr_ = nullptr;
        o.bytes_ = 0;
    }
    return *this;
}
DeviceBuffer::~DeviceBuffer() {
    if (ptr_ != nullptr && owned_) cudaFree(ptr_);
}

namespace {
// Clears (source null) or fills device memory before it returns.  cudaMemset and cudaMemcpy are of no use for that: they may
// return before their work on the default stream is done, which the engine's streams do not wait for.
void set_now(void* destination, const void* source, size_t bytes, cudaStream_t s, const char* what) {
    check_cuda(source == nullptr ? cudaMemsetAsync(destination, 0, bytes, s)
                                 : cudaMemcpyAsync(destination, source, bytes, cudaMemcpyHostToDevice, s), what);
    check_cuda(cudaStreamSynchronize(s), what);
}
}  // namespace

// ------------------------------------------------------------------ KvPool

KvPool::KvPool(int layers, int kv_width, int slab_shift, cudaStream_t stream)
    : stream_(stream), layers_(layers), kv_width_(kv_width), slab_shift_(slab_shift),
      page_elems_((long long)kPageTokens * kv_width),
      plane_elems_(((long long)1 << slab_shift) * kPageTokens * kv_width),
      slab_table_(kMaxSlabs * sizeof(bf16*)) {
    set_now(slab_table_.as<void>(), nullptr, kMaxSlabs * sizeof(bf16*), stream_, "clear slab table");
}

void KvPool::add_slab() {
    if (static_cast<int>(slabs_.size()) >= kMaxSlabs) throw std::bad_alloc();
    const size_t bytes = (size_t)layers_ * 2 * plane_elems_ * sizeof(bf16);
    DeviceBuffer slab(bytes);
    bf16* base = slab.as<bf16>();
    const int index = static_cast<int>(slabs_.size());
    set_now(slab_table_.as<bf16*>() + index, &base, sizeof(base), stream_, "fill slab table");
    slabs_.push_back(std::move(slab));
    const int per = 1 << slab_shift_;
    for (int i = per - 1; i >= 0; --i) free_.push_back(index * per + i);
}

int KvPool::allocate() {
    if (free_.empty()) add_slab();
    const int page = free_.back();
    free_.pop_back();
    return page;
}

void KvPool::release(int page) { free_.push_back(page); }

KvLayout KvPool::layout(int layer, const int* page_table, int table_stride) const {
    KvLayout l;
    l.page_table = page_table;
    l.table_stride = table_stride;
    l.slabs = slab_table_.as<bf16*>();
    l.slab_shift = slab_shift_;
    l.page_elems = page_elems_;
    l.k_offset = (long long)(layer * 2) * plane_elems_;
    l.v_offset = (long long)(layer * 2 + 1) * plane_elems_;
    return l;
}

const bf16* KvPool::page_rows(int page, int layer, bool value) const {
    const int slab = page >> slab_shift_;
    if (page < 0 || slab >= static_cast<int>(slabs_.size()) || layer < 0 || layer >= layers_) {
        throw std::runtime_error("KV page or layer out of range");
    }
    return slabs_[slab].as<bf16>() + (long long)(page & ((1 << slab_shift_) - 1)) * page_elems_
           + (long long)(layer * 2 + (value ? 1 : 0)) * plane_elems_;
}

uint64_t KvPool::page_bytes() const { return (uint64_t)layers_ * 2 * page_elems_ * sizeof(bf16); }

// ------------------------------------------------------------------ Workspace

Workspace::Workspace(int capacity_, int device_, int rows_, bool lockstep)
    : capacity(capacity_), rows(std::max(capacity_, rows_)), device(device_) {
    check_cuda(cudaSetDevice(device), "cudaSetDevice(workspace)");
    const size_t e = sizeof(bf16);
    size_t c = rows;
    const size_t one = capacity;
    // one allocation: a session's workspace is made when the session is, and fourteen of them were half of that
    const std::pair<DeviceBuffer*, size_t> parts[] = {
        {&table, sizeof(FrameTable)}, {&counters, one * 16 * sizeof(unsigned int)},
        {&chain_order_scratch, chain_order_scratch_floats(std::min(capacity, kChainRows), 8) * sizeof(float)},
        {&hidden, c * 2048 * e}, {&qkv, c * 4096 * e}, {&attention, c * 2048 * e}, {&gate, c * 6144 * e},
        {&logits, one * kTalkerVocab * e}, {&x_in, c * 2048 * e}, {&projection, c * 2048 * e}, {&normalized, c * 2048 * e},
        {&prompt_positions, c * sizeof(int)}, {&talker_pages, one * kMaxPagesPerRow * sizeof(int)},
        {&lockstep_exchange, lockstep ? lockstep_exchange_bytes() : 0},
        {&predictor_pages, one * sizeof(int)}, {&predictor_positions, (size_t)kPredictorSequence * kMaxRows * sizeof(int)}};
    size_t total = 0;
    for (const auto& part : parts) total += align_up(part.second, 1024);
    arena = DeviceBuffer(total);
    size_t at = 0;
    for (const auto& part : parts) {
        *part.first = DeviceBuffer(arena, at, part.second);
        at += align_up(part.second, 1024);
    }
    c = capacity;
    try {
        check_cuda(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking), "cudaStreamCreate");
        const size_t host_bytes = align_up(sizeof(FrameTable), 1024);
        check_cuda(cudaHostAlloc(reinterpret_cast<void**>(&host_table), host_bytes + c * (kMaxPagesPerRow + 1) * sizeof(int),
                                 cudaHostAllocDefault), "cudaHostAlloc(frame table, page tables)");
        std::memset(host_table, 0, sizeof(FrameTable));
        host_pages = reinterpret_cast<int*>(reinterpret_cast<char*>(host_table) + host_bytes);
        check_cuda(cudaMemsetAsync(table.as<void>(), 0, align_up(table.bytes(), 1024) + counters.bytes(), stream),
                   "cudaMemset(frame table, counters)");
        std::vector<int> positions((size_t)kPredictorSequence * kMaxRows);
        for (int p = 0; p < kPredictorSequence; ++p)
            for (int r = 0; r < kMaxRows; ++r) positions[(size_t)p * kMaxRows + r] = p;
        check_cuda(cudaMemcpyAsync(predictor_positions.as<void>(), positions.data(),
                                   positions.size() * sizeof(int), cudaMemcpyHostToDevice, stream),
                   "cudaMemcpy(predictor positions)");
        check_cuda(cudaEventCreate(&predictor_start), "cudaEventCreate");
        check_cuda(cudaEventCreate(&predictor_stop), "cudaEventCreate");
        check_cuda(cudaEventCreate(&talker_start), "cudaEventCreate");
        check_cuda(cudaEventCreate(&talker_stop), "cudaEventCreate");
        check_cuda(cudaEventCreateWithFlags(&table_uploaded, cudaEventDisableTiming), "cudaEventCreate");
        for (int i = 0; i < capacity && i < kMaxRows; ++i) {
            check_cuda(cudaEventCreateWithFlags(&join_events[i], cudaEventDisableTiming),
                       "cudaEventCreate(join)");
        }
    } catch (...) {
        release();
        throw;
    }
}

void Workspace::release() noexcept {
    destroy_graphs();
    for (cudaEvent_t& ev : join_events) {
        if (ev != nullptr) cudaEventDestroy(ev);
        ev = nullptr;
    }
    for (cudaEvent_t* ev : {&predictor_start, &predictor_stop, &talker_start, &talker_stop,
                            &table_uploaded}) {
        if (*ev != nullptr) cudaEventDestroy(*ev);
        *ev = nullptr;
    }
    host_pages = nullptr;            // behind the host table
    if (host_table != nullptr) cudaFreeHost(host_table);
    host_table = nullptr;
    if (stream != nullptr) cudaStreamDestroy(stream);
    stream = nullptr;
}

Workspace::~Workspace() {
    cudaSetDevice(device);
    if (stream != nullptr) cudaStreamSynchronize(stream);
    if (Traffic* traffic = traffic_of(device)) {
        std::lock_guard<std::mutex> lock(traffic->mutex);
        traffic->leave(this);
    }
    release();
}

void Workspace::destroy_graphs() noexcept {
    for (auto& kv : graphs) {
        if (kv.second.predictor != nullptr) cudaGraphExecDestroy(kv.second.predictor);
        if (kv.second.talker != nullptr) cudaGraphExecDestroy(kv.second.talker);
    }
    graphs.clear();
}

void Workspace::ensure_scratch(int splits) {
    if (splits <= scratch_splits) return;
    check_cuda(cudaStreamSynchronize(stream), "cudaStreamSynchronize(scratch)");
    destroy_graphs();   // captured launches hold the old scratch pointer
    scratch = DeviceBuffer();
    scratch = DeviceBuffer(attention_scratch_floats(capacity, 16, 128, splits) * sizeof(float));
    scratch_splits = splits;
}

uint64_t Workspace::bytes() const {
    return hidden.bytes() + qkv.bytes() + attention.bytes() + gate.bytes() + logits.bytes()
        + x_in.bytes() + projection.bytes() + normalized.bytes() + table.bytes()
        + talker_pages.bytes() + predictor_pages.bytes() + predictor_positions.bytes()
        + counters.bytes() + scratch.bytes() + chain_order_scratch.bytes() + lockstep_exchange.bytes();
}

// ------------------------------------------------------------------ Model

Model::Model(int device) : device_(device) {
    check_cuda(cudaSetDevice(device_), "cudaSetDevice(model)");
    check_cuda(cudaStreamCreateWithFlags(&upload_stream_, cudaStreamNonBlocking),
               "cudaStreamCreate(upload)");
    talker = {2048, 6144, 16, 8, 128, 2048, 1024, kTalkerLayers};
    // The checkpoint's code predictor has head_dim 128 (q 2048 wide, k/v 1024 wide);
    // QWEN3_TTS_PREDICTOR_HEAD_DIM=64 selects the 64-wide variant for experiments.
    const int phd = env_int("QWEN3_TTS_PREDICTOR_HEAD_DIM", 128) == 64 ? 64 : 128;
    predictor = {1024, 3072, 16, 8, phd, 16 * phd, 8 * phd, kPredictorLayers};
    mask_eos = env_int("QWEN3_TTS_MASK_EOS", 0) != 0;
    use_graphs = env_int("QWEN3_TTS_DISABLE_GRAPHS", 0) == 0;

    const uint64_t H = talker.hidden, PH = predictor.hidden;
    add_keep("talker.model.codec_embedding.weight", {kTalkerVocab, H}, &codec_embedding);
    add_keep("talker.model.text_embedding.weight", {kTextVocab, H}, &text_embedding);
    text_fc1 = add_quant_matrix("talker.text_projection.linear_fc1.weight", H, H);
    add_keep("talker.text_projection.linear_fc1.bias", {H}, &text_fc1_bias);
    text_fc2 = add_quant_matrix("talker.text_projection.linear_fc2.weight", H, H);
    add_keep("talker.text_projection.linear_fc2.bias", {H}, &text_fc2_bias);
    add_keep("talker.model.norm.weight", {H}, &talker_norm);
    codec_head = add_quant_matrix("talker.codec_head.weight", kTalkerVocab, H);
    plan_layers("talker.model.layers.", talker, talker_layers);
    small_to_mtp = add_quant_matrix("talker.code_predictor.small_to_mtp_projection.weight", PH, H);
    add_keep("talker.code_predictor.small_to_mtp_projection.bias", {PH}, &small_to_mtp_bias);
    add_keep("talker.code_predictor.model.norm.weight", {PH}, &predictor_norm);
    plan_layers("talker.code_predictor.model.layers.", predictor, predictor_layers);
    for (int g = 0; g < kResidualCodebooks; ++g) {
        add_keep("talker.code_predictor.model.codec_embedding." + std::to_string(g) + ".weight",
                 {(uint64_t)kPredictorVocab, H}, &predictor_embeddings[g]);
        predictor_heads[g] = add_quant_matrix(
            "talker.code_predictor.lm_head." + std::to_string(g) + ".weight", kPredictorVocab, PH);
    }
}

Model::~Model() {
    cudaSetDevice(device_);
    batch_.reset();
    if (upload_stream_ != nullptr) {
        cudaStreamSynchronize(upload_stream_);
        cudaStreamDestroy(upload_stream_);
    }
}

void Model::add_keep(const std::string& name, std::vector<uint64_t> shape, const bf16** slot) {
    size_t elements = 1;
    for (uint64_t d : shape) elements *= d;
    storage_.emplace_back(elements * sizeof(bf16));
    Spec s;
    s.shape = std::move(shape);
    s.destination = storage_.back().as<void>();
    *slot = storage_.back().as<bf16>();
    specs_.emplace(name, std::move(s));
}

void Model::add_quant_rows(const std::string& name, uint64_t rows, uint64_t cols, int8_t* data,
                           float* scales) {
    Spec s;
    s.shape = {rows, cols};
    s.quantize = true;
    s.destination = data;
    s.scales = scales;
    specs_.emplace(name, std::move(s));
    staging_bytes_ = std::max(staging_bytes_, (size_t)(rows * cols * sizeof(bf16)));
}

Quantized Model::allocate_quantized(uint64_t rows, uint64_t cols) {
    storage_.emplace_back(rows * cols);
    int8_t* data = storage_.back().as<int8_t>();
    storage_.emplace_back(rows * sizeof(float));
    float* scales = storage_.back().as<float>();
    return Quantized{data, scales};
}

Quantized Model::add_quant_matrix(const std::string& name, uint64_t rows, uint64_t cols) {
    const Quantized q = allocate_quantized(rows, cols);
    add_quant_rows(name, rows, cols, const_cast<int8_t*>(q.data), const_cast<float*>(q.scales));
    return q;
}

void Model::plan_layers(const std::string& prefix, const ModelDims& d, std::vector<LayerWeights>& out) {
    const uint64_t H = d.hidden, I = d.intermediate, QW = d.q_width, KW = d.kv_width, HD = d.head_dim;
    out.resize(d.layers);
    for (int l = 0; l < d.layers; ++l) {
        LayerWeights& w = out[l];
        const std::string p = prefix + std::to_string(l);
        add_keep(p + ".input_layernorm.weight", {H}, &w.input_norm);
        w.qkv = allocate_quantized(QW + 2 * KW, H);
        int8_t* qd = const_cast<int8_t*>(w.qkv.data);
        float* qs = const_cast<float*>(w.qkv.scales);
        add_quant_rows(p + ".self_attn.q_proj.weight", QW, H, qd, qs);
        add_quant_rows(p + ".self_attn.k_proj.weight", KW, H, qd + QW * H, qs + QW);
        add_quant_rows(p + ".self_attn.v_proj.weight", KW, H, qd + (QW + KW) * H, qs + QW + KW);
        w.o = add_quant_matrix(p + ".self_attn.o_proj.weight", H, QW);
        add_keep(p + ".self_attn.q_norm.weight", {HD}, &w.q_norm);
        add_keep(p + ".self_attn.k_norm.weight", {HD}, &w.k_norm);
        add_keep(p + ".post_attention_layernorm.weight", {H}, &w.post_norm);
        w.gate_up = allocate_quantized(2 * I, H);
        int8_t* gd = const_cast<int8_t*>(w.gate_up.data);
        float* gs = const_cast<float*>(w.gate_up.scales);
        add_quant_rows(p + ".mlp.gate_proj.weight", I, H, gd, gs);
        add_quant_rows(p + ".mlp.up_proj.weight", I, H, gd + I * H, gs + I);
        w.down = add_quant_matrix(p + ".mlp.down_proj.weight", H, I);
    }
}

void Model::upload_tensor(const char* name, const void* data, uint64_t bytes, int rank,
                          const uint64_t* shape) {
    check_cuda(cudaSetDevice(device_), "cudaSetDevice(upload)");
    if (finalized_) throw std::runtime_error("model weights are already finalized");
    if (name == nullptr || *name == '\0' || data == nullptr || shape == nullptr) {
        throw std::runtime_error("tensor upload received a null argument");
    }
    if (rank <= 0 || rank > 4 || bytes == 0) {
        throw std::runtime_error("tensor upload has an invalid rank or byte size");
    }
    uint64_t elements = 1;
    std::vector<uint64_t> dims;
    for (int i = 0; i < rank; ++i) {
        if (shape[i] == 0 || elements > std::numeric_limits<uint64_t>::max() / shape[i]) {
            throw std::runtime_error("tensor shape is empty or overflows");
        }
        elements *= shape[i];
        dims.push_back(shape[i]);
    }
    if (elements > std::numeric_limits<uint64_t>::max() / sizeof(bf16)
        || elements * sizeof(bf16) != bytes) {
        throw std::runtime_error("tensor byte size does not match BF16 shape");
    }
    const auto found = specs_.find(name);
    if (found == specs_.end()) {
        throw std::runtime_error(std::string("tensor is not part of the talker checkpoint: ") + name);
    }
    Spec& spec = found->second;
    if (spec.seen) throw std::runtime_error(std::string("duplicate tensor upload: ") + name);
    if (spec.shape != dims) throw std::runtime_error(std::string("unexpected shape for tensor ") + name);
    if (spec.quantize) {
        if (staging_.bytes() < staging_bytes_) staging_ = DeviceBuffer(staging_bytes_);
        check_cuda(cudaMemcpyAsync(staging_.as<void>(), data, bytes, cudaMemcpyHostToDevice,
                                   upload_stream_), "cudaMemcpyAsync(weight H2D)");
        check_cuda(launch_quantize_weight_rows(staging_.as<bf16>(),
                                               static_cast<int8_t*>(spec.destination), spec.scales,
                                               static_cast<int>(dims[1]), static_cast<int>(dims[0]),
                                               upload_stream_), "quantize decode weight");
        // the staging buffer is reused by the next upload; the host copy above has already
        // left the caller's buffer when cudaMemcpyAsync returns for pageable memory, but a
        // pinned source is read asynchronously, so wait before handing control back
        check_cuda(cudaStreamSynchronize(upload_stream_), "cudaStreamSynchronize(upload)");
    } else {
        check_cuda(cudaMemcpyAsync(spec.destination, data, bytes, cudaMemcpyHostToDevice,
                                   upload_stream_), "cudaMemcpyAsync(weight H2D)");
        check_cuda(cudaStreamSynchronize(upload_stream_), "cudaStreamSynchronize(upload)");
    }
    spec.seen = true;
    weight_bytes_ += bytes;
    ++tensor_count_;
}

Model::TensorImage Model::tensor_image(const char* name) const {
    if (name == nullptr) throw std::runtime_error("tensor name is null");
    const auto found = specs_.find(name);
    if (found == specs_.end()) {
        throw std::runtime_error(std::string("tensor is not part of the talker checkpoint: ") + name);
    }
    const Spec& spec = found->second;
    uint64_t elements = 1;
    for (uint64_t d : spec.shape) elements *= d;
    TensorImage image;
    image.data = spec.destination;
    image.quantized = spec.quantize;
    image.loaded = spec.seen;
    if (spec.quantize) {
        image.data_bytes = elements;                          // one int8 per weight
        image.scales = spec.scales;
        image.scales_bytes = spec.shape[0] * sizeof(float);   // one scale per output row
    } else {
        image.data_bytes = elements * sizeof(bf16);
    }
    return image;
}

void Model::adopt_tensor(const char* name) {
    check_cuda(cudaSetDevice(device_), "cudaSetDevice(adopt)");
    if (finalized_) throw std::runtime_error("model weights are already finalized");
    if (name == nullptr) throw std::runtime_error("tensor name is null");
    const auto found = specs_.find(name);
    if (found == specs_.end()) {
        throw std::runtime_error(std::string("tensor is not part of the talker checkpoint: ") + name);
    }
    Spec& spec = found->second;
    if (spec.seen) throw std::runtime_error(std::string("duplicate tensor upload: ") + name);
    uint64_t elements = 1;
    for (uint64_t d : spec.shape) elements *= d;
    spec.seen = true;
    weight_bytes_ += elements * sizeof(bf16);     // counted as the checkpoint tensor it stands for
    ++tensor_count_;
}

void Model::finalize(uint64_t* weight_bytes, uint32_t* tensor_count) {
    check_cuda(cudaSetDevice(device_), "cudaSetDevice(finalize)");
    if (finalized_) throw std::runtime_error("model weights are already finalized");
    if (tensor_count_ != 404 || specs_.size() != 404) {
        for (const auto& kv : specs_) {
            if (!kv.second.seen) {
                throw std::runtime_error("checkpoint is missing required tensor " + kv.first);
            }
        }
        throw std::runtime_error("expected exactly 404 VoiceDesign tensors, found "
                                 + std::to_string(tensor_count_));
    }
    check_cuda(cudaStreamSynchronize(upload_stream_), "cudaStreamSynchronize(upload)");
    staging_ = DeviceBuffer();
    embedding_ptrs_ = DeviceBuffer(kResidualCodebooks * sizeof(const bf16*));
    set_now(embedding_ptrs_.as<void>(), predictor_embeddings.data(), kResidualCodebooks * sizeof(const bf16*), upload_stream_,
            "embedding table");
    predictor_embedding_table = embedding_ptrs_.as<const bf16*>();
    talker_rope_ = DeviceBuffer((size_t)kRopePositions * (talker.head_dim / 2) * sizeof(uint32_t));
    check_cuda(launch_build_rope_table(talker_rope_.as<uint32_t>(), kRopePositions, talker.head_dim,
                                       kRopeTheta, upload_stream_), "rope table");
    talker_rope = talker_rope_.as<uint32_t>();
    if (predictor.head_dim == talker.head_dim) {
        predictor_rope = talker_rope;
    } else {
        predictor_rope_ = DeviceBuffer((size_t)kRopePositions * (predictor.head_dim / 2) * sizeof(uint32_t));
        check_cuda(launch_build_rope_table(predictor_rope_.as<uint32_t>(), kRopePositions, predictor.head_dim,
                                           kRopeTheta, upload_stream_), "rope table");
        predictor_rope = predictor_rope_.as<uint32_t>();
    }
    check_cuda(cudaStreamSynchronize(upload_stream_), "cudaStreamSynchronize(rope tables)");
    try {
        build_chain();
    } catch (const std::bad_alloc&) {
        // frames run launch by launch without it
        cudaStreamSynchronize(upload_stream_);
        chain = DecodeChain();
    }
    try {
        build_lockstep();
    } catch (const std::bad_alloc&) {
        lockstep = DeviceBuffer();          // frames of 9 and more sessions likewise
    }
    talker_pool.reset(new KvPool(talker.layers, talker.kv_width, 8, upload_stream_));
    predictor_pool.reset(new KvPool(predictor.layers, predictor.kv_width, 6, upload_stream_));
    finalized_ = true;
    *weight_bytes = weight_bytes_;
    *tensor_count = tensor_count_;
}

void Model::build_chain() {
    if (!chain_available() || predictor.head_dim != 128) return;
    // The chain is a second image of the decode matrices, for speed alone: it is not to take the memory that sessions and
    // prompts need.
    size_t free_bytes = 0, total_bytes = 0;
    check_cuda(cudaMemGetInfo(&free_bytes, &total_bytes), "cudaMemGetInfo");
    const size_t wanted = chain_stream_bytes(false) + chain_stream_bytes(true) + chain_head_bytes(false) + chain_head_bytes(true);
    if (free_bytes < wanted + kChainLeaves) return;
    // The streams are made from the weights as they lie there now: what a caller has enqueued on streams of its own to fill
    // adopted storage has to be done.
    check_cuda(cudaDeviceSynchronize(), "cudaDeviceSynchronize(adopted weights)");
    auto table = [this](DeviceBuffer& b, const void* host, size_t bytes) {
        b = DeviceBuffer(bytes);
        set_now(b.as<void>(), host, bytes, upload_stream_, "chain table");
    };
    for (int t = 0; t < 2; ++t) {
        const bool big = t == 1;
        chain.streams[t] = DeviceBuffer(chain_stream_bytes(big));
        chain.heads[t] = DeviceBuffer(chain_head_bytes(big));
        std::vector<ChainLayer> constants;
        const std::vector<LayerWeights>& layers = big ? talker_layers : predictor_layers;
        for (size_t l = 0; l < layers.size(); ++l) {
            const LayerWeights& lw = layers[l];
            check_cuda(launch_pack_layer(big, static_cast<int>(l), lw.qkv.data, lw.o.data, lw.gate_up.data, lw.down.data,
                                         chain.streams[t].as<uint8_t>(), upload_stream_), "pack layer");
            constants.push_back({lw.qkv.scales, lw.o.scales, lw.gate_up.scales, lw.down.scales, lw.input_norm, lw.post_norm,
                                 lw.q_norm, lw.k_norm});
        }
        table(chain.layers[t], constants.data(), constants.size() * sizeof(ChainLayer));
        std::vector<const float*> scales;
        for (int h = 0; h < (big ? 1 : kResidualCodebooks); ++h) {
            const Quantized& head = big ? codec_head : predictor_heads[h];
            check_cuda(launch_pack_head(big, h, head.data, chain.heads[t].as<uint8_t>(), upload_stream_), "pack head");
            scales.push_back(head.scales);
        }
        table(chain.head_scales[t], scales.data(), scales.size() * sizeof(const float*));
    }
    // input row of predictor position p >= 1 for every token of codebook p - 1: the projection the frame would
    // otherwise make of the token's embedding, by the same kernel (exact sums: same bits whatever rows run together)
    const size_t PH = predictor.hidden;
    std::vector<const bf16*> rows;
    chain.projected_rows = DeviceBuffer(((size_t)kTalkerVocab + 14 * (size_t)kPredictorVocab) * PH * sizeof(bf16));
    bf16* out = chain.projected_rows.as<bf16>();
    for (int c = 0; c < kResidualCodebooks; ++c) {
        const bf16* in = c == 0 ? codec_embedding : predictor_embeddings[c - 1];
        const int tokens = c == 0 ? kTalkerVocab : kPredictorVocab;
        rows.push_back(out);
        for (int first = 0; first < tokens; first += kMaxRows) {
            GemvArgs g;
            g.w = small_to_mtp.data; g.scales = small_to_mtp.scales; g.bias = small_to_mtp_bias;
            g.x = in + (size_t)first * talker.hidden; g.y = out + (size_t)first * PH;
            g.in_features = talker.hidden; g.out_features = static_cast<int>(PH);
            g.rows = std::min(kMaxRows, tokens - first); g.epilogue = EPI_BIAS;
            check_cuda(launch_int8_gemv_mma(g, upload_stream_), "project embeddings");
        }
        out += (size_t)tokens * PH;
    }
    table(chain.projected, rows.data(), rows.size() * sizeof(const bf16*));
    chain.exchange = DeviceBuffer(chain_exchange_bytes());
    chain.epoch = DeviceBuffer(2 * sizeof(uint32_t));
    chain.places = DeviceBuffer(sizeof(ChainPlaces));
    const uint32_t none[3] = {0, 0, 0};
    table(chain.claims, none, sizeof(none));
    place_chain();
    chain.ready = true;
}

void Model::build_lockstep() {
    if (predictor.head_dim != 128) return;
    std::unique_ptr<LockstepModel> host(new LockstepModel());
    const int PH = predictor.hidden, PI = predictor.intermediate, qkv = predictor.q_width + 2 * predictor.kv_width;
    bool ok = true;
    for (int l = 0; l < predictor.layers; ++l) {
        const LayerWeights& lw = predictor_layers[l];
        ok = ok && make_lockstep_map(host.get(), 4 * l, lw.qkv.data, PH, qkv, true)
             && make_lockstep_map(host.get(), 4 * l + 1, lw.o.data, predictor.q_width, PH, false)
             && make_lockstep_map(host.get(), 4 * l + 2, lw.gate_up.data, PH, 2 * PI, false)
             && make_lockstep_map(host.get(), 4 * l + 3, lw.down.data, PI, PH, false);
        host->layers[l] = {lw.qkv.scales, lw.o.scales, lw.gate_up.scales, lw.down.scales, lw.input_norm, lw.post_norm, lw.q_norm, lw.k_norm};
    }
    for (int h = 0; h < kResidualCodebooks; ++h) {
        ok = ok && make_lockstep_map(host.get(), kLockstepHeadMap + h, predictor_heads[h].data, PH, kPredictorVocab, true);
        host->head_scales[h] = predictor_heads[h].scales;
    }
    ok = ok && make_lockstep_map(host.get(), kLockstepMtpMap, small_to_mtp.data, talker.hidden, PH, false);
    host->mtp_scales = small_to_mtp.scales;
    host->mtp_bias = small_to_mtp_bias;
    host->final_norm = predictor_norm;
    if (!ok) return;
    lockstep = DeviceBuffer(sizeof(LockstepModel));
    set_now(lockstep.as<void>(), host.get(), sizeof(LockstepModel), upload_stream_, "lockstep table");
}

void Model::place_chain() {
    ChainPlaces places;
    check_cuda(find_chain_places(chain.exchange.as<void>(), &places, upload_stream_), "chain places");
    set_now(chain.places.as<void>(), &places, sizeof(places), upload_stream_, "chain places");
    chain.grid = places.grid;
    check_cuda(restart_chain_numbers(chain.exchange.as<void>(), chain.epoch.as<uint32_t>(), upload_stream_), "chain numbers");
    check_cuda(cudaStreamSynchronize(upload_stream_), "cudaStreamSynchronize(decode chain)");
    chain.numbers = 0;
}

void Model::set_chain_places(const uint8_t* die_of_sm, const uint32_t* pages, int grid) {
    if (!chain.ready) return;
    check_cuda(cudaDeviceSynchronize(), "cudaDeviceSynchronize(chain places)");
    ++option_epoch;                 // captured graphs launch the grid of before
    if (die_of_sm == nullptr) return place_chain();
    int sms = 0;
    check_cuda(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device_), "cudaDeviceGetAttribute");
    if (grid < 128 || grid > sms) throw std::invalid_argument("a chain of fewer than 128 CTAs, or more than SMs");
    ChainPlaces places;
    places.on_first = 64;
    chain.grid = places.grid = grid;
    std::vector<bool> taken(kPoolPages, false);
    for (int sm = 0; sm < kPlaceSms; ++sm) {
        if (die_of_sm[sm] > 1) throw std::invalid_argument("a die that is neither 0 nor 1");
        places.die_of_sm[sm] = die_of_sm[sm];
    }
    const uint32_t first = static_cast<uint32_t>(chain_pool_at(chain.exchange.as<void>()) / 16);
    for (int i = 0; i < kPlaceGroups * kGroupPages; ++i) {
        if (pages[i] >= (uint32_t)kPoolPages || taken[pages[i]]) throw std::invalid_argument("a page that is not there or taken");
        taken[pages[i]] = true;
        places.pages[i / kGroupPages][i % kGroupPages] = first + pages[i] * (kPlacePage / 16);
    }
    set_now(chain.places.as<void>(), &places, sizeof(places), upload_stream_, "chain places");
}

void Model::set_chain_numbers(uint64_t used, uint32_t given_up) {
    if (!chain.ready) return;
    const uint32_t epoch[2] = {static_cast<uint32_t>(used), given_up};
    check_cuda(cudaDeviceSynchronize(), "cudaDeviceSynchronize(chain numbers)");
    set_now(chain.epoch.as<void>(), epoch, sizeof(epoch), upload_stream_, "chain numbers");
    chain.numbers = used;
}

unsigned int Model::device_errors() const {
    volatile unsigned int* word = device_error_word(device_);
    return word != nullptr ? *word : 0u;
}

void Model::check_device_errors(unsigned int count_at_enqueue) const {
    if (device_errors() != count_at_enqueue) {
        throw CudaFailure("a bounded device-side wait ran out: the results of this call cannot be trusted");
    }
}

Workspace& Model::batch_workspace() {
    std::lock_guard<std::mutex> lock(mutex);
    if (!batch_) batch_.reset(new Workspace(kMaxRows, device_, 0, true));
    return *batch_;
}

Workspace& Model::prefill_workspace() {
    std::lock_guard<std::mutex> lock(mutex);
    if (!prefill_) {
        try {
            prefill_.reset(new Workspace(kMaxRows, device_, kMaxPromptRows));
        } catch (const std::bad_alloc&) {
            prefill_.reset(new Workspace(kMaxRows, device_));       // 3 MB instead of 85: prompts in passes of 64
        }
    }
    return *prefill_;
}

// ------------------------------------------------------------------ frame enqueue

namespace {

// Observation points of a prompt pass for the parity hooks (QWEN3_TTS_PARITY_TRACE,
// QWEN3_TTS_STAGE_DUMP): called with the stage name, the layer and one activation row in device
// memory.  Each call synchronises the stream, so a probed pass is never captured in a graph.
struct Probe {
    int row = 0;       // which row of the pass is observed (the last prompt position)
    std::function<void(const char* stage, int layer, const bf16* values, int width)> emit;
};

// `last_keys_only`: nothing behind the last layer's cache rows is needed (the predictor's position 0, whose hidden row no head reads)
void enqueue_layers(Workspace& w, const ModelDims& d, const std::vector<LayerWeights>& layers,
                    const uint32_t* rope_table, const KvPool& pool, const int* page_table, int table_stride,
                    const int* positions, int n, int splits, cudaStream_t s, int prompt_base = -1,
                    const Probe* probe = nullptr, bool chain_order = false, bool last_keys_only = false) {
    const int qkv_width = d.q_width + 2 * d.kv_width;
    // a prompt pass (prompt_base >= 0): the rows are consecutive positions of one session
    const bool shared_cache = prompt_base >= 0;
    auto project = [&](GemvArgs& g, const char* what) {
        if (g.norm_w != nullptr && n >= tc_min_rows()) g.norm_out = w.normalized.as<bf16>();
        check_launch(n > kMaxRows ? launch_int8_gemm_prompt(g, s) : launch_int8_gemm(g, s), what);
    };
    for (size_t l = 0; l < layers.size(); ++l) {
        const LayerWeights& lw = layers[l];
        const int layer = static_cast<int>(l);
        auto observe = [&](const char* stage, const bf16* base, int stride, int width) {
            if (probe != nullptr) probe->emit(stage, layer, base + (size_t)probe->row * stride, width);
        };
        GemvArgs g;
        g.w = lw.qkv.data; g.scales = lw.qkv.scales;
        g.x = w.hidden.as<bf16>(); g.y = w.qkv.as<bf16>();
        g.norm_w = lw.input_norm;
        if (probe != nullptr) g.norm_out = w.normalized.as<bf16>();
        g.in_features = d.hidden; g.out_features = qkv_width; g.rows = n; g.epilogue = EPI_PLAIN;
        project(g, "qkv projection");
        observe("input_norm", w.normalized.as<bf16>(), d.hidden, d.hidden);
        observe("q_projection", w.qkv.as<bf16>(), qkv_width, d.q_width);
        observe("k_projection", w.qkv.as<bf16>() + d.q_width, qkv_width, d.kv_width);
        observe("v_projection", w.qkv.as<bf16>() + d.q_width + d.kv_width, qkv_width, d.kv_width);

        AttentionArgs a;
        a.q = w.qkv.as<bf16>();
        a.k_new = w.qkv.as<bf16>() + d.q_width;
        a.v_new = w.qkv.as<bf16>() + d.q_width + d.kv_width;
        a.q_stride = qkv_width; a.kv_new_stride = qkv_width;
        a.q_norm_w = lw.q_norm; a.k_norm_w = lw.k_norm;
        a.positions = positions;
        a.out = w.attention.as<bf16>();
        a.kv = pool.layout(static_cast<int>(l), page_table, table_stride);
        a.scratch = w.scratch.as<float>();
        a.counters = w.counters.as<unsigned int>();
        a.rows = n; a.q_heads = d.q_heads; a.kv_heads = d.kv_heads; a.head_dim = d.head_dim;
        a.max_splits = splits; a.fused = 1;
        a.rope_table = rope_table; a.rope_positions = Model::kRopePositions;
        // The kernel directly before attention is the qkv projection; positions, page table and
        // the older cache rows all date from earlier launches (the kernel ignores this outside
        // plain decode steps).
        a.inputs_settled = 1;
        if (shared_cache && n >= tc_min_rows() && attention_mode() != 0 && prompt_attention_supports(a)) {
            // With the projections on the tensor cores nothing promises a row the bits it would have
            // alone, and the positions share their passes over the cache.
            check_launch(launch_prompt_attention(a, prompt_base, s), "prompt attention");
        } else if (shared_cache) {
            // the rows are consecutive positions of one session: every row's K/V goes into the
            // cache first, then every row attends up to its own position
            a.append_mode = 1;
            check_launch(launch_attention(a, s), "prompt KV append");
            a.append_mode = 2;
            check_launch(launch_attention(a, s), "prompt attention");
        } else if (chain_order) {
            a.scratch = w.chain_order_scratch.as<float>();
            check_launch(launch_chain_order_attention(a, s), "decode attention");
        } else {
            check_launch(launch_attention(a, s), "decode attention");
        }
        observe("attention", w.attention.as<bf16>(), d.q_width, d.q_width);
        if (last_keys_only && l + 1 == layers.size()) break;

        GemvArgs o;
        o.w = lw.o.data; o.scales = lw.o.scales;
        o.x = w.attention.as<bf16>(); o.y = w.hidden.as<bf16>();
        o.in_features = d.q_width; o.out_features = d.hidden; o.rows = n; o.epilogue = EPI_ADD;
        o.residual_settled = true;     // hidden was last written before the qkv projection
        project(o, "attention output projection");
        observe("attention_residual", w.hidden.as<bf16>(), d.hidden, d.hidden);

        GemvArgs u;
        u.w = lw.gate_up.data; u.scales = lw.gate_up.scales;
        u.x = w.hidden.as<bf16>(); u.y = w.gate.as<bf16>();
        u.norm_w = lw.post_norm;
        if (probe != nullptr) u.norm_out = w.normalized.as<bf16>();
        u.in_features = d.hidden; u.out_features = d.intermediate; u.rows = n;
        u.epilogue = EPI_GATE_UP_SILU;
        u.leave_room = chain_order;
        project(u, "gate/up projection");
        observe("post_attention_norm", w.normalized.as<bf16>(), d.hidden, d.hidden);
        observe("gated_activation", w.gate.as<bf16>(), d.intermediate, d.intermediate);

        GemvArgs dn;
        dn.w = lw.down.data; dn.scales = lw.down.scales;
        dn.x = w.gate.as<bf16>(); dn.y = w.hidden.as<bf16>();
        dn.in_features = d.intermediate; dn.out_features = d.hidden; dn.rows = n;
        dn.epilogue = EPI_ADD;
        dn.residual_settled = true;    // hidden was last written by the output projection, two launches up
        project(dn, "down projection");
        observe("layer_output", w.hidden.as<bf16>(), d.hidden, d.hidden);
    }
}

void enqueue_chain(Workspace& w, Model& m, bool talker, int n, cudaStream_t s) {
    const Model::DecodeChain& c = m.chain;
    const int t = talker ? 1 : 0;
    const KvPool& pool = talker ? *m.talker_pool : *m.predictor_pool;
    ChainLaunch a;
    a.talker = talker;
    a.stream = c.streams[t].as<uint8_t>(); a.heads = c.heads[t].as<uint8_t>();
    a.layers = c.layers[t].as<ChainLayer>(); a.head_scales = c.head_scales[t].as<const float*>();
    a.final_norm = talker ? m.talker_norm : m.predictor_norm;
    a.hidden = w.hidden.as<bf16>();
    a.table = w.table.as<FrameTable>();
    if (talker) {
        a.normalized = w.normalized.as<bf16>(); a.logits = w.logits.as<bf16>();
        a.positions = w.table.as<FrameTable>()->position;
        a.kv = pool.layout(0, w.talker_pages.as<int>(), Workspace::kMaxPagesPerRow);
        a.rope_table = m.talker_rope;
    } else {
        a.projected = c.projected.as<const bf16*>();
        a.kv = pool.layout(0, w.predictor_pages.as<int>(), 1);
        a.rope_table = m.predictor_rope;
    }
    a.kv_layer_elems = 2 * pool.plane_elems();
    a.exchange = c.exchange.as<void>(); a.epoch = c.epoch.as<uint32_t>();
    a.places = c.places.as<const ChainPlaces>(); a.claims = c.claims.as<uint32_t>(); a.grid = c.grid;
    a.rows = n;
    check_launch(launch_decode_chain(a, s), talker ? "talker chain" : "predictor chain");
}

// The predictor's part of a frame as one chain; only the projection of the hidden state stays a launch of its own.
void enqueue_predictor_chain(Workspace& w, Model& m, int n, cudaStream_t s) {
    const int H = m.talker.hidden;
    check_launch(launch_predictor_input(w.table.as<FrameTable>(), 0, m.codec_embedding, m.predictor_embedding_table,
                                        w.x_in.as<bf16>(), H, n, s), "predictor input");
    GemvArgs g;
    g.w = m.small_to_mtp.data; g.scales = m.small_to_mtp.scales;
    g.x = w.x_in.as<bf16>(); g.y = w.hidden.as<bf16>(); g.bias = m.small_to_mtp_bias;
    g.in_features = H; g.out_features = m.predictor.hidden; g.rows = n; g.epilogue = EPI_BIAS;
    check_launch(launch_int8_gemm(g, s), "predictor input projection");
    enqueue_chain(w, m, false, n, s);
}

// How a frame's predictor is made: launch by launch, a launch of the lockstep chain for each position with the draws between
// them, or one launch for all.
enum class Lockstep { kNone, kPositions, kWhole };
// Whether it may run on the lockstep chain: enough rows, the default kernels (it computes what they compute).
bool lockstep_may_run(const Workspace& w, const Model& m, int n) {
    return n > kChainRows && n >= tc_min_rows() && m.use_chain == 1 && m.use_graphs != 0 && attention_mode() == 1 && m.lockstep.bytes() != 0
           && w.lockstep_exchange.bytes() != 0 && lockstep_chain_available(n);
}

// Whether the chains make these draws of the predictor: greedy ones, and from no more candidates than their sampler ranks.
bool draws_fit_chains(const FrameTable& t, int n) {
    for (int i = 0; i < n; ++i) {
        const SamplingParams& p = t.predictor[i];
        if (p.do_sample != 0 && (p.top_k < 1 || p.top_k > kChainTopK)) return false;
    }
    return true;
}

// 16 predictor positions, 15 sampled codebooks, packed codes (talker.cu:1549-1701)
void enqueue_predictor(Workspace& w, Model& m, int n, Lockstep lockstep, cudaStream_t s) {
    const FrameTable* table = w.table.as<FrameTable>();
    const int H = m.talker.hidden, PH = m.predictor.hidden;
    check_launch(launch_frame_begin(table, n, s), "frame begin");
    LockstepLaunch c;
    if (lockstep != Lockstep::kNone) {
        c.model = m.lockstep.as<LockstepModel>();
        c.table = table; c.pages = w.predictor_pages.as<int>();
        c.kv = m.predictor_pool->layout(0, c.pages, 1);
        c.kv_layer_elems = 2 * m.predictor_pool->plane_elems();
        c.rope_table = m.predictor_rope;
        c.codec_embedding = m.codec_embedding; c.embeddings = m.predictor_embedding_table;
        c.logits = w.logits.as<bf16>(); c.exchange = w.lockstep_exchange.as<void>();
        c.rows = n;
    }
    if (lockstep == Lockstep::kWhole) {
        c.last = kPredictorSequence - 1;
        c.draws = true;
        check_launch(launch_lockstep_chain(c, s), "lockstep chain");
    }
    for (int p = 0; p < kPredictorSequence && lockstep != Lockstep::kWhole; ++p) {
        if (lockstep == Lockstep::kPositions) {
            c.first = c.last = p;
            check_launch(launch_lockstep_chain(c, s), "lockstep chain");
            if (p >= 1) {
                check_launch(launch_sample_table(table, w.logits.as<bf16>(), kPredictorVocab, kPredictorVocab, 0, p, 0, kEos, n, s),
                             "sample predictor logits");
            }
            continue;
        }
        check_launch(launch_predictor_input(table, p, m.codec_embedding, m.predictor_embedding_table,
                                          w.x_in.as<bf16>(), H, n, s), "predictor input");
        GemvArgs g;
        g.w = m.small_to_mtp.data; g.scales = m.small_to_mtp.scales;
        g.x = w.x_in.as<bf16>(); g.y = w.hidden.as<bf16>(); g.bias = m.small_to_mtp_bias;
        g.in_features = H; g.out_features = PH; g.rows = n; g.epilogue = EPI_BIAS;
        check_launch(launch_int8_gemm(g, s), "predictor input projection");
        enqueue_layers(w, m.predictor, m.predictor_layers, m.predictor_rope, *m.predictor_pool,
                       w.predictor_pages.as<int>(), 1,
                       w.predictor_positions.as<int>() + (size_t)p * kMaxRows, n, 1, s, -1, nullptr, false, p == 0);
        if (p >= 1) {
            GemvArgs h;
            h.w = m.predictor_heads[p - 1].data; h.scales = m.predictor_heads[p - 1].scales;
            h.x = w.hidden.as<bf16>(); h.y = w.logits.as<bf16>(); h.norm_w = m.predictor_norm;
            h.in_features = PH; h.out_features = kPredictorVocab; h.rows = n; h.epilogue = EPI_PLAIN;
            // (not the tensor-core path's own buffer: another model may be running on the device)
            if (n >= tc_min_rows()) h.norm_out = w.normalized.as<bf16>();
            check_launch(launch_int8_gemm(h, s), "predictor head");
            check_launch(launch_sample_table(table, w.logits.as<bf16>(), kPredictorVocab,
                                           kPredictorVocab, 0, p, 0, kEos, n, s),
                       "sample predictor logits");
        }
    }
    check_launch(launch_pack_codes(table, n, s), "pack codec frame");
}

void enqueue_text_projection(Workspace& w, Model& m, int n, bool residual, cudaStream_t s) {
    const int H = m.talker.hidden;
    GemvArgs f1;
    f1.w = m.text_fc1.data; f1.scales = m.text_fc1.scales;
    f1.x = w.x_in.as<bf16>(); f1.y = w.projection.as<bf16>(); f1.bias = m.text_fc1_bias;
    f1.in_features = H; f1.out_features = H; f1.rows = n; f1.epilogue = EPI_BIAS_SILU;
    check_launch(n > kMaxRows ? launch_int8_gemm_prompt(f1, s) : launch_int8_gemm(f1, s), "text projection fc1");
    GemvArgs f2;
    f2.w = m.text_fc2.data; f2.scales = m.text_fc2.scales;
    f2.x = w.projection.as<bf16>(); f2.bias = m.text_fc2_bias;
    f2.in_features = H; f2.out_features = H; f2.rows = n;
    if (residual) {
        f2.resid = w.hidden.as<bf16>(); f2.epilogue = EPI_BIAS_ADD;
    } else {
        f2.y = w.hidden.as<bf16>(); f2.epilogue = EPI_BIAS;
    }
    check_launch(n > kMaxRows ? launch_int8_gemm_prompt(f2, s) : launch_int8_gemm(f2, s), "text projection fc2");
}

void enqueue_talker_head(Workspace& w, Model& m, int n, int advance, cudaStream_t s) {
    FrameTable* table = w.table.as<FrameTable>();
    const int H = m.talker.hidden;
    GemvArgs h;
    h.w = m.codec_head.data; h.scales = m.codec_head.scales;
    h.x = w.hidden.as<bf16>(); h.y = w.logits.as<bf16>();
    h.norm_w = m.talker_norm; h.norm_out = w.normalized.as<bf16>();
    h.in_features = H; h.out_features = kTalkerVocab; h.rows = n; h.epilogue = EPI_PLAIN;
    check_launch(launch_int8_gemm(h, s), "codec head");
    check_launch(launch_sample_table(table, w.logits.as<bf16>(), kTalkerVocab, kTalkerVocab, 1, 0,
                                   m.mask_eos, kEos, n, s), "sample talker logits");
    check_launch(launch_frame_end(table, w.normalized.as<bf16>(), H, n, advance, s), "frame end");
}

// next talker input, 28 layers, head, sample (talker.cu:1703-1880)
// `chain_order`: with the bits of enqueue_talker_chain
void enqueue_talker(Workspace& w, Model& m, int n, int splits, cudaStream_t s, bool chain_order = false) {
    FrameTable* table = w.table.as<FrameTable>();
    const int H = m.talker.hidden;
    check_launch(launch_talker_input(table, m.codec_embedding, m.predictor_embedding_table,
                                   m.text_embedding, kTextVocab, w.hidden.as<bf16>(),
                                   w.x_in.as<bf16>(), H, n, s), "talker input");
    enqueue_text_projection(w, m, n, true, s);
    enqueue_layers(w, m.talker, m.talker_layers, m.talker_rope, *m.talker_pool, w.talker_pages.as<int>(),
                   Workspace::kMaxPagesPerRow, table->position, n, splits, s, -1, nullptr, chain_order);
    enqueue_talker_head(w, m, n, 1, s);
}

void enqueue_talker_chain(Workspace& w, Model& m, int n, cudaStream_t s) {
    FrameTable* table = w.table.as<FrameTable>();
    const int H = m.talker.hidden;
    check_launch(launch_talker_input(table, m.codec_embedding, m.predictor_embedding_table,
                                   m.text_embedding, kTextVocab, w.hidden.as<bf16>(),
                                   w.x_in.as<bf16>(), H, n, s), "talker input");
    enqueue_text_projection(w, m, n, true, s);
    enqueue_chain(w, m, true, n, s);
    check_launch(launch_sample_table(table, w.logits.as<bf16>(), kTalkerVocab, kTalkerVocab, 1, 0, m.mask_eos, kEos, n, s),
                 "sample talker logits");
    check_launch(launch_frame_end(table, w.normalized.as<bf16>(), H, n, 1, s), "frame end");
}

// Whether a frame of these rows may run on the decode chain: few rows, the default kernels (it computes what they
// compute), draws small enough for its sampler.
bool frame_may_chain(const Model& m, const FrameTable& t, int n) {
    if (!m.chain.ready || m.use_chain == 0 || m.use_graphs == 0 || n > kChainRows || n >= tc_min_rows() || gemv_mode() != 1 || attention_mode() != 1
        || traffic_of(m.device()) == nullptr) {
        return false;
    }
    return draws_fit_chains(t, n);
}

// one prompt position of row 0 (talker.cu:1058-1064 + one decoder pass)
void enqueue_prompt_step(Workspace& w, Model& m, const int* text_ids, const int* codec_ids,
                         int splits, cudaStream_t s) {
    FrameTable* table = w.table.as<FrameTable>();
    const int H = m.talker.hidden;
    check_launch(launch_prompt_gather(table, text_ids, m.text_embedding, kTextVocab,
                                    w.x_in.as<bf16>(), H, s), "prompt gather");
    enqueue_text_projection(w, m, 1, false, s);
    check_launch(launch_prompt_combine(table, text_ids, codec_ids, m.codec_embedding, kTalkerVocab,
                                     w.hidden.as<bf16>(), H, s), "prompt combine");
    enqueue_layers(w, m.talker, m.talker_layers, m.talker_rope, *m.talker_pool, w.talker_pages.as<int>(),
                   Workspace::kMaxPagesPerRow, table->position, 1, splits, s);
    check_launch(launch_advance_position(table, s), "advance position");
}

// prompt positions base .. base + rows - 1 of row 0's session as the rows of one decoder pass
void enqueue_prompt_chunk(Workspace& w, Model& m, const int* text_ids, const int* codec_ids, int base,
                          int rows, int splits, cudaStream_t s, const Probe* probe = nullptr) {
    const int H = m.talker.hidden;
    check_launch(launch_prompt_rows(text_ids, codec_ids, base, rows, m.text_embedding, kTextVocab,
                                  w.x_in.as<bf16>(), w.prompt_positions.as<int>(), H, s), "prompt rows");
    enqueue_text_projection(w, m, rows, false, s);
    check_launch(launch_prompt_combine_rows(text_ids, codec_ids, base, rows, m.codec_embedding, kTalkerVocab,
                                          w.hidden.as<bf16>(), H, s), "prompt combine");
    if (probe != nullptr) probe->emit("input", -1, w.hidden.as<bf16>() + (size_t)probe->row * H, H);
    // page-table stride 0: every row reads and writes the cache of the session bound to row 0
    enqueue_layers(w, m.talker, m.talker_layers, m.talker_rope, *m.talker_pool, w.talker_pages.as<int>(), 0,
                   w.prompt_positions.as<int>(), rows, splits, s, base, probe);
}

// ---- parity hooks of the prompt path --------------------------------------------------------
// QWEN3_TTS_PARITY_TRACE: one line per observed vector on stderr, in the reference's format
// (talker.cu:2342-2432: "QWEN3_TTS_TRACE {json}" with stage, layer, mean, rms, maximum and the first
// 16 values; the 20 largest logits at the end), for the input row, every layer's output, the final
// norm and the logits of the last prompt position.  QWEN3_TTS_STAGE_DUMP: the layer-0 stages and the
// final logits as raw bf16 files named <stage>.bf16, in the directory the variable names (a value
// without a slash selects the reference's /tmp/native_stages, talker.cu:2503-2538).
struct ParityHooks {
    bool trace = false;
    std::string dump_dir;
    cudaStream_t stream = nullptr;

    static ParityHooks from_environment(cudaStream_t s) {
        ParityHooks h;
        h.stream = s;
        h.trace = std::getenv("QWEN3_TTS_PARITY_TRACE") != nullptr;
        if (const char* d = std::getenv("QWEN3_TTS_STAGE_DUMP")) {
            h.dump_dir = std::strchr(d, '/') != nullptr ? d : "/tmp/native_stages";
        }
        return h;
    }
    bool active() const { return trace || !dump_dir.empty(); }

    std::vector<float> fetch(const bf16* values, int width) const {
        std::vector<bf16> raw(width);
        check_cuda(cudaMemcpyAsync(raw.data(), values, (size_t)width * sizeof(bf16), cudaMemcpyDeviceToHost,
                                   stream), "copy parity vector to host");
        check_cuda(cudaStreamSynchronize(stream), "synchronize parity vector");
        std::vector<float> out(width);
        for (int i = 0; i < width; ++i) out[i] = __bfloat162float(raw[i]);
        return out;
    }
    void dump(const char* stage, const bf16* values, int width) const {
        if (dump_dir.empty()) return;
        std::vector<bf16> raw(width);
        check_cuda(cudaMemcpyAsync(raw.data(), values, (size_t)width * sizeof(bf16), cudaMemcpyDeviceToHost,
                                   stream), "copy stage dump to host");
        check_cuda(cudaStreamSynchronize(stream), "synchronize stage dump");
        const std::string path = dump_dir + "/" + stage + ".bf16";
        std::FILE* f = std::fopen(path.c_str(), "wb");
        if (f == nullptr) throw std::runtime_error("failed to create stage dump " + path);
        const size_t written = std::fwrite(raw.data(), sizeof(bf16), raw.size(), f);
        if (std::fclose(f) != 0 || written != raw.size()) throw std::runtime_error("failed to write stage dump " + path);
    }
    void vector_line(const char* stage, int layer, const bf16* values, int width) const {
        if (!trace) return;
        const std::vector<float> v = fetch(values, width);
        double sum = 0.0, squares = 0.0;
        float largest = 0.0f;
        for (float x : v) {
            sum += x;
            squares += (double)x * x;
            largest = std::max(largest, std::fabs(x));
        }
        std::string line = "QWEN3_TTS_TRACE {\"stage\":\"" + std::string(stage) + "\",\"layer\":" + std::to_string(layer);
        char number[64];
        std::snprintf(number, sizeof(number), ",\"mean\":%.9g", sum / width); line += number;
        std::snprintf(number, sizeof(number), ",\"rms\":%.9g", std::sqrt(squares / width)); line += number;
        std::snprintf(number, sizeof(number), ",\"maximum\":%.9g,\"first\":[", largest); line += number;
        for (int i = 0; i < std::min(width, 16); ++i) {
            std::snprintf(number, sizeof(number), "%s%.9g", i == 0 ? "" : ",", v[i]);
            line += number;
        }
        std::fprintf(stderr, "%s]}\n", line.c_str());
    }
    void logits_line(const bf16* logits, int vocabulary) const {
        if (!trace) return;
        const std::vector<float> v = fetch(logits, vocabulary);
        std::vector<int> order(vocabulary);
        std::iota(order.begin(), order.end(), 0);
        const int top = std::min(20, vocabulary);
        std::partial_sort(order.begin(), order.begin() + top, order.end(),
                          [&v](int a, int b) { return v[a] == v[b] ? a < b : v[a] > v[b]; });
        std::string line = "QWEN3_TTS_TRACE {\"stage\":\"logits\",\"top\":[";
        char item[96];
        for (int r = 0; r < top; ++r) {
            std::snprintf(item, sizeof(item), "%s{\"token\":%d,\"logit\":%.9g}", r == 0 ? "" : ",", order[r], v[order[r]]);
            line += item;
        }
        std::fprintf(stderr, "%s]}\n", line.c_str());
    }
    // the probe a prompt pass is run with
    Probe probe(int row) const {
        Probe p;
        p.row = row;
        const ParityHooks* self = this;
        p.emit = [self](const char* stage, int layer, const bf16* values, int width) {
            const bool input = std::strcmp(stage, "input") == 0;
            const bool output = std::strcmp(stage, "layer_output") == 0;
            if (input) self->vector_line("input", -1, values, width);
            if (output) self->vector_line("layer", layer, values, width);
            if (input || layer == 0) self->dump(stage, values, width);
        };
        return p;
    }
};

int count_kernel_nodes(cudaGraph_t graph) {
    size_t total = 0;
    if (cudaGraphGetNodes(graph, nullptr, &total) != cudaSuccess || total == 0) return 0;
    std::vector<cudaGraphNode_t> nodes(total);
    if (cudaGraphGetNodes(graph, nodes.data(), &total) != cudaSuccess) return 0;
    int kernels = 0;
    for (size_t i = 0; i < total; ++i) {
        cudaGraphNodeType type;
        if (cudaGraphNodeGetType(nodes[i], &type) == cudaSuccess && type == cudaGraphNodeTypeKernel) {
            ++kernels;
        }
    }
    return kernels;
}

template <class Enqueue>
cudaGraphExec_t capture(cudaStream_t s, Enqueue&& enqueue, int* kernel_nodes = nullptr) {
    check_cuda(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal), "cudaStreamBeginCapture");
    cudaGraph_t graph = nullptr;
    try {
        enqueue();
    } catch (...) {
        cudaStreamEndCapture(s, &graph);
        if (graph != nullptr) cudaGraphDestroy(graph);
        throw;
    }
    check_cuda(cudaStreamEndCapture(s, &graph), "cudaStreamEndCapture");
    if (kernel_nodes != nullptr) *kernel_nodes = count_kernel_nodes(graph);
    cudaGraphExec_t exec = nullptr;
    const cudaError_t e = cudaGraphInstantiate(&exec, graph, 0);
    cudaGraphDestroy(graph);
    check_cuda(e, "cudaGraphInstantiate");
    return exec;
}

int split_bucket(int max_length) {
    const int splits = (max_length + kAttnChunk - 1) / kAttnChunk;
    return (splits + 7) / 8 * 8;
}

void validate_sampling_params(const SamplingParams& p) {
    if (p.top_k < 0 || !(p.top_p > 0.0f) || p.top_p > 1.0f || !(p.temperature > 0.0f)
        || !(p.penalty > 0.0f)) {
        throw std::runtime_error("invalid sampling configuration");
    }
}

}  // namespace

// ------------------------------------------------------------------ Session

Session::Session(std::shared_ptr<Model> model, int max_sequence_length, uint64_t seed)
    : model_(std::move(model)), id_(g_next_session_id.fetch_add(1)), device_(model_->device()),
      max_seq_(max_sequence_length) {
    if (max_sequence_length < 16 || max_sequence_length > 8192) {
        throw std::runtime_error("max sequence length must be in [16, 8192]");
    }
    if (!model_->finalized()) {
        throw std::runtime_error("model weights must be finalized before creating a session");
    }
    check_cuda(cudaSetDevice(device_), "cudaSetDevice(session)");
    solo_.reset(new Workspace(1, device_));
    stream_ = solo_->stream;
    try {
        check_cuda(cudaEventCreateWithFlags(&codes_ready_, cudaEventDisableTiming), "cudaEventCreate");
        check_cuda(cudaEventCreateWithFlags(&semantic_ready_, cudaEventDisableTiming), "cudaEventCreate");
        const size_t off_tokens = 0;
        const size_t off_codes = align_up(off_tokens + kCodebooks * sizeof(int), 256);
        const size_t off_sampled = align_up(off_codes + kCodebooks * sizeof(unsigned short), 256);
        const size_t off_rng = align_up(off_sampled + sizeof(int), 256);
        const size_t off_hidden = align_up(off_rng + sizeof(unsigned long long), 256);
        const size_t off_history = align_up(off_hidden + 2048 * sizeof(bf16), 256);
        const size_t total = off_history + (size_t)max_seq_ * sizeof(int);
        state_ = DeviceBuffer(total);
        check_cuda(cudaMemsetAsync(state_.as<void>(), 0, total, stream_), "cudaMemset(session state)");
        char* base = state_.as<char>();
        d_frame_tokens_ = reinterpret_cast<int*>(base + off_tokens);
        d_frame_codes_ = reinterpret_cast<unsigned short*>(base + off_codes);
        d_sampled_ = reinterpret_cast<int*>(base + off_sampled);
        d_rng_ = reinterpret_cast<unsigned long long*>(base + off_rng);
        d_last_hidden_ = reinterpret_cast<bf16*>(base + off_hidden);
        d_history_ = reinterpret_cast<int*>(base + off_history);
        check_cuda(cudaHostAlloc(reinterpret_cast<void**>(&h_token_), 128 + kCodebooks * sizeof(unsigned short),
                                 cudaHostAllocMapped), "cudaHostAlloc(sampled token, frame codes)");
        h_codes_ = reinterpret_cast<unsigned short*>(reinterpret_cast<char*>(h_token_) + 128);
        *h_token_ = -1;
        {
            std::lock_guard<std::mutex> lock(model_->mutex);
            const int pages = (max_seq_ + kPageTokens - 1) / kPageTokens;
            for (int i = 0; i < pages; ++i) talker_pages_.push_back(model_->talker_pool->allocate());
            predictor_page_ = model_->predictor_pool->allocate();
            talker_kv_bytes = (uint64_t)pages * model_->talker_pool->page_bytes();
            predictor_kv_bytes = model_->predictor_pool->page_bytes();
        }
        solo_->ensure_scratch(split_bucket(max_seq_ < 512 ? max_seq_ : 512));
        workspace_bytes = solo_->bytes() + state_.bytes();
        reset(seed);
    } catch (...) {
        release();
        throw;
    }
}

void Session::release() noexcept {
    if (model_) {
        std::lock_guard<std::mutex> lock(model_->mutex);
        for (int page : talker_pages_) model_->talker_pool->release(page);
        talker_pages_.clear();
        if (predictor_page_ >= 0) model_->predictor_pool->release(predictor_page_);
        predictor_page_ = -1;
    }
    h_codes_ = nullptr;              // behind the token
    if (h_token_ != nullptr) cudaFreeHost(h_token_);
    h_token_ = nullptr;
    if (semantic_ready_ != nullptr) cudaEventDestroy(semantic_ready_);
    semantic_ready_ = nullptr;
    if (codes_ready_ != nullptr) cudaEventDestroy(codes_ready_);
    codes_ready_ = nullptr;
}

Session::~Session() {
    cudaSetDevice(device_);
    // A lockstep frame of this session that was begun and never finished may still be running on
    // the shared workspace: its last event is this session's own, so no other thread's stream (which
    // may be capturing a graph at this moment) has to be touched.  Workspaces remember bound sessions
    // by id, and ids are never reused, so nothing has to be erased from them either.
    if (frame_in_flight_ && semantic_ready_ != nullptr) cudaEventSynchronize(semantic_ready_);
    if (stream_ != nullptr) cudaStreamSynchronize(stream_);
    release();
    solo_.reset();
}

void Session::reset(uint64_t seed) {
    own_stream_busy_ = true;
    check_cuda(cudaSetDevice(device_), "cudaSetDevice(reset)");
    if (frame_in_flight_) throw std::runtime_error("cannot reset while a device frame lease is in flight");
    position_ = 0;
    generated_ = 0;
    frames_generated = 0;
    device_sample_count = 0;
    host_sync_count = 0;
    current_token_ = 0;
    phase_ = model_->finalized() ? kPhaseReady : kPhaseCreated;
    const unsigned long long state = seed == 0 ? 0x9e3779b97f4a7c15ULL : seed;
    check_cuda(cudaMemcpyAsync(d_rng_, &state, sizeof(state), cudaMemcpyHostToDevice, stream_),
               "reset device random state");
    check_cuda(cudaStreamSynchronize(stream_), "synchronize reset random state");
}

void Session::fill_row(FrameTable& t, int row, int trailing_text, const SamplingParams& talker,
                       const SamplingParams& predictor, bool host_codes) const {
    t.position[row] = position_;
    t.history_count[row] = generated_;
    t.trailing_text[row] = trailing_text;
    t.frame_tokens[row] = d_frame_tokens_;
    t.frame_codes[row] = d_frame_codes_;
    t.history[row] = d_history_;
    t.rng[row] = d_rng_;
    t.sampled[row] = d_sampled_;
    t.last_hidden[row] = d_last_hidden_;
    t.host_token[row] = h_token_;
    t.host_codes[row] = host_codes ? h_codes_ : nullptr;
    t.talker[row] = talker;
    t.predictor[row] = predictor;
}

// the checks of the reference's begin_frame, in its order (talker.cu:1103-1127)
void Session::validate_begin(int semantic_token, int trailing_text, const SamplingParams& talker,
                             const SamplingParams& predictor) const {
    if (poisoned_) throw std::runtime_error("talker session is poisoned and must be destroyed");
    if (frame_in_flight_) throw std::runtime_error("a device frame lease is already in flight");
    if (phase_ != kPhasePrefilled) {
        throw std::runtime_error("talker must be prefilled before frame generation");
    }
    if (semantic_token == kEos) throw std::runtime_error("EOS must not be expanded into a codec frame");
    if (semantic_token >= kTalkerVocab) {
        throw std::runtime_error("semantic token is outside the talker vocabulary");
    }
    if (semantic_token != current_token_) {
        throw std::runtime_error("semantic token does not match talker session state");
    }
    if (trailing_text < 0 || trailing_text >= kTextVocab) {
        throw std::runtime_error("next-frame text token is outside the text vocabulary");
    }
    if (position_ >= max_seq_) throw std::runtime_error("talker KV cache is full");
    if (generated_ >= max_seq_) {
        throw std::runtime_error("semantic history exceeds configured sequence capacity");
    }
    validate_sampling_params(talker);
    validate_sampling_params(predictor);
}

// Makes the page lists of s[0..n) resident in the workspace's page tables.
void Session::bind_rows(Workspace& w, Session** s, int n) {
    bool same = static_cast<int>(w.bound.size()) == n;
    for (int i = 0; same && i < n; ++i) same = w.bound[i] == s[i]->id_;
    if (same) return;
    check_cuda(cudaStreamSynchronize(w.stream), "cudaStreamSynchronize(rebind)");
    const int stride = Workspace::kMaxPagesPerRow;
    int* talker_rows = w.host_pages;
    int* predictor_rows = w.host_pages + (size_t)w.capacity * stride;
    for (int i = 0; i < n; ++i) {
        const std::vector<int>& pages = s[i]->talker_pages_;
        std::copy(pages.begin(), pages.end(), talker_rows + (size_t)i * stride);
        predictor_rows[i] = s[i]->predictor_page_;
    }
    check_cuda(cudaMemcpyAsync(w.talker_pages.as<void>(), talker_rows,
                               (size_t)n * stride * sizeof(int), cudaMemcpyHostToDevice, w.stream),
               "upload talker page table");
    check_cuda(cudaMemcpyAsync(w.predictor_pages.as<void>(), predictor_rows, (size_t)n * sizeof(int),
                               cudaMemcpyHostToDevice, w.stream), "upload predictor page table");
    w.bound.resize(n);
    for (int i = 0; i < n; ++i) w.bound[i] = s[i]->id_;
}

Workspace::Graphs& Session::frame_graphs(Workspace& w, Model& m, int n, int splits, Way way, int lockstep) {
    const bool chain = way == Way::kChain;
    const auto key = std::make_tuple(n, chain ? 0 : (way == Way::kInItsPlace ? -1 : splits), lockstep);
    auto found = w.graphs.find(key);
    if (found != w.graphs.end()) return found->second;
    Workspace::Graphs g;
    g.predictor = capture(w.stream, [&] {
                              if (chain) enqueue_predictor_chain(w, m, n, w.stream);
                              else enqueue_predictor(w, m, n, static_cast<Lockstep>(lockstep), w.stream);
                          },
                          &g.predictor_kernels);
    try {
        g.talker = capture(w.stream, [&] {
                               if (chain) enqueue_talker_chain(w, m, n, w.stream);
                               else enqueue_talker(w, m, n, splits, w.stream, way == Way::kInItsPlace);
                           },
                           &g.talker_kernels);
    } catch (...) {
        cudaGraphExecDestroy(g.predictor);
        throw;
    }
    return w.graphs.emplace(key, g).first->second;
}

// Enqueues one frame for rows s[0..n) on w.stream.  The host table must be filled.
void Session::launch_frame(Workspace& w, Model& m, Session** s, int n, bool upload_table,
                           bool record_session_events, int ahead) {
    int max_length = 1;
    for (int i = 0; i < n; ++i) max_length = std::max(max_length, w.host_table->position[i] + ahead + 1);
    const int splits = split_bucket(max_length);
    ++w.frame_serial;
    if (w.option_epoch != m.option_epoch) {
        check_cuda(cudaStreamSynchronize(w.stream), "cudaStreamSynchronize(options)");
        w.destroy_graphs();
        w.option_epoch = m.option_epoch;
    }
    Traffic* const traffic = traffic_of(m.device());
    std::unique_ptr<InFlight> in_flight;
    Way way = Way::kLaunches;
    Lockstep lockstep = Lockstep::kNone;
    if (frame_may_chain(m, *w.host_table, n)) {
        in_flight.reset(new InFlight(traffic, w, n, m.use_chain == 2));
        way = in_flight->kind() == Traffic::kChain ? Way::kChain : Way::kInItsPlace;
    } else if (lockstep_may_run(w, m, n) && traffic != nullptr) {
        in_flight.reset(new InFlight(traffic, w, n, InFlight::Large()));
        if (in_flight->alone()) lockstep = draws_fit_chains(*w.host_table, n) ? Lockstep::kWhole : Lockstep::kPositions;
    } else {
        in_flight.reset(new InFlight(traffic, w, n, Traffic::kOther));
    }
    if (way == Way::kLaunches) w.ensure_scratch(splits);
    bind_rows(w, s, n);
    Workspace::Graphs* const g = m.use_graphs ? &frame_graphs(w, m, n, splits, way, static_cast<int>(lockstep)) : nullptr;
    {
        const ChainTurn turn(way == Way::kChain ? traffic : nullptr, w);
        if (upload_table) {
            check_cuda(cudaMemcpyAsync(w.table.as<void>(), w.host_table, sizeof(FrameTable),
                                       cudaMemcpyHostToDevice, w.stream), "upload frame table");
            check_cuda(cudaEventRecord(w.table_uploaded, w.stream), "cudaEventRecord(table)");
        }
        if (way == Way::kChain && (m.chain.numbers += kChainNumbersPerFrame) > kChainNumbers) {
            check_cuda(restart_chain_numbers(m.chain.exchange.as<void>(), m.chain.epoch.as<uint32_t>(), w.stream), "chain numbers");
            m.chain.numbers = kChainNumbersPerFrame;
        }
        if (lockstep != Lockstep::kNone && (w.lockstep_rows != n || w.lockstep_errors != m.device_errors())) {
            w.lockstep_errors = m.device_errors();
            check_cuda(restart_lockstep(w.lockstep_exchange.as<void>(), n, w.stream), "lockstep exchange");
            w.lockstep_rows = n;
        }
        check_cuda(cudaEventRecord(w.predictor_start, w.stream), "cudaEventRecord");
        if (g != nullptr) check_cuda(cudaGraphLaunch(g->predictor, w.stream), "cudaGraphLaunch(predictor)");
        else enqueue_predictor(w, m, n, lockstep, w.stream);
        check_cuda(cudaEventRecord(w.predictor_stop, w.stream), "cudaEventRecord");
        if (record_session_events) {
            for (int i = 0; i < n; ++i) {
                check_cuda(cudaEventRecord(s[i]->codes_ready_, w.stream), "cudaEventRecord(codes)");
            }
        }
        check_cuda(cudaEventRecord(w.talker_start, w.stream), "cudaEventRecord");
        if (g != nullptr) check_cuda(cudaGraphLaunch(g->talker, w.stream), "cudaGraphLaunch(talker)");
        else enqueue_talker(w, m, n, splits, w.stream);
        check_cuda(cudaEventRecord(w.talker_stop, w.stream), "cudaEventRecord");
        if (g != nullptr) m.kernel_launches += static_cast<uint64_t>(g->predictor_kernels + g->talker_kernels);
    }
    in_flight->enqueued();
    if (record_session_events) {
        for (int i = 0; i < n; ++i) {
            check_cuda(cudaEventRecord(s[i]->semantic_ready_, w.stream), "cudaEventRecord(semantic)");
        }
    }
}

uint64_t Session::take_lease(Workspace* w, bool host_codes) {
    const uint64_t lease = next_lease_++;
    if (next_lease_ == 0) next_lease_ = 1;
    frame_in_flight_ = true;
    pending_host_codes_ = host_codes;
    pending_lease_ = lease;
    pending_position_ = static_cast<uint32_t>(position_);
    pending_workspace_ = w;
    pending_frame_serial_ = w != nullptr ? w->frame_serial + 1 : 0;    // the frame about to be launched
    pending_errors_ = model_->device_errors();
    return lease;
}

void Session::drop_lease_poisoned() noexcept {
    poisoned_ = true;
    frame_in_flight_ = false;
    pending_host_codes_ = false;
    pending_lease_ = 0;
    pending_workspace_ = nullptr;
}

FrameView Session::begin_frame(uint16_t semantic_token, int trailing_text, const SamplingParams& talker,
                               const SamplingParams& predictor, bool host_codes) {
    check_cuda(cudaSetDevice(device_), "cudaSetDevice(begin frame)");
    validate_begin(semantic_token, trailing_text, talker, predictor);
    Workspace& w = *solo_;
    own_stream_busy_ = true;
    const uint64_t lease = take_lease(&w, host_codes);
    try {
        check_cuda(cudaEventSynchronize(w.table_uploaded), "cudaEventSynchronize(table)");
        fill_row(*w.host_table, 0, trailing_text, talker, predictor, host_codes);
        Session* self = this;
        launch_frame(w, *model_, &self, 1, true, true);
    } catch (...) {
        cudaStreamSynchronize(stream_);
        drop_lease_poisoned();
        throw;
    }
    device_sample_count += kPredictorSequence;
    ++generated_;
    ++position_;
    FrameView view;
    view.device_codes = d_frame_codes_;
    view.ready_event = codes_ready_;
    view.lease_id = lease;
    view.device = device_;
    return view;
}

void Session::batch_begin(Model* model, Session** s, int n, const int* trailing_text,
                          const SamplingParams* talker, const SamplingParams* predictor,
                          FrameView* views) {
    if (model == nullptr || s == nullptr || n <= 0 || n > kMaxRows) {
        throw std::runtime_error("invalid batch frame arguments");
    }
    check_cuda(cudaSetDevice(model->device()), "cudaSetDevice(batch frame)");
    for (int i = 0; i < n; ++i) {
        if (s[i]->model_.get() != model) {
            throw std::runtime_error("batched session belongs to a different model");
        }
        for (int j = 0; j < i; ++j) {
            if (s[j] == s[i]) throw std::runtime_error("a session appears twice in one batch");
        }
        s[i]->validate_begin(s[i]->current_token_, trailing_text[i], talker[i], predictor[i]);
    }
    std::lock_guard<std::mutex> one_batch(model->batch_mutex);
    Workspace& w = model->batch_workspace();
    const bool host_codes = model->batch_host_codes != 0;
    for (int i = 0; i < n; ++i) s[i]->take_lease(&w, host_codes);
    try {
        check_cuda(cudaEventSynchronize(w.table_uploaded), "cudaEventSynchronize(table)");
        for (int i = 0; i < n; ++i) {
            s[i]->fill_row(*w.host_table, i, trailing_text[i], talker[i], predictor[i], host_codes);
        }
        // order the batch stream after each session's earlier work
        for (int i = 0; i < n; ++i) {
            if (!s[i]->own_stream_busy_) continue;      // nothing of its own since the last lockstep frame
            check_cuda(cudaEventRecord(w.join_events[i], s[i]->stream_), "cudaEventRecord(join)");
            check_cuda(cudaStreamWaitEvent(w.stream, w.join_events[i], 0), "cudaStreamWaitEvent(join)");
            s[i]->own_stream_busy_ = false;
        }
        launch_frame(w, *model, s, n, true, true);
        for (int i = 0; i < n; ++i) {
            s[i]->device_sample_count += kPredictorSequence;
            ++s[i]->generated_;
            ++s[i]->position_;
            check_cuda(cudaStreamWaitEvent(s[i]->stream_, s[i]->semantic_ready_, 0),
                       "cudaStreamWaitEvent(rejoin)");
        }
    } catch (...) {
        cudaStreamSynchronize(w.stream);
        for (int i = 0; i < n; ++i) s[i]->drop_lease_poisoned();
        w.destroy_graphs();
        throw;
    }
    for (int i = 0; i < n; ++i) {
        views[i].device_codes = s[i]->d_frame_codes_;
        views[i].ready_event = s[i]->codes_ready_;
        views[i].lease_id = s[i]->pending_lease_;
        views[i].device = s[i]->device_;
    }
}

FrameResult Session::finish_frame(uint64_t lease_id, cudaEvent_t consumer_done) {
    check_cuda(cudaSetDevice(device_), "cudaSetDevice(finish frame)");
    if (poisoned_) throw std::runtime_error("talker session is poisoned and must be destroyed");
    if (!frame_in_flight_) throw std::runtime_error("no device frame lease is in flight");
    if (lease_id == 0 || lease_id != pending_lease_) {
        throw std::runtime_error("device frame lease ID is stale or invalid");
    }
    if (consumer_done != nullptr) {
        check_cuda(cudaStreamWaitEvent(stream_, consumer_done, 0), "cudaStreamWaitEvent(consumer done)");
        own_stream_busy_ = true;
    }
    check_cuda(cudaEventSynchronize(semantic_ready_), "cudaEventSynchronize(semantic ready)");
    ++host_sync_count;
    const int next = *h_token_;
    try {
        model_->check_device_errors(pending_errors_);
        if (next < 0 || next >= kTalkerVocab) {
            throw std::runtime_error("device sampler returned an invalid token");
        }
    } catch (...) {
        drop_lease_poisoned();
        throw;
    }
    FrameResult r{};
    r.talker_position = pending_position_;
    Workspace* w = pending_workspace_;
    if (w != nullptr && w->timed_frame == pending_frame_serial_ && pending_frame_serial_ != 0) {
        r.predictor_ms = w->timed_predictor_ms;      // a sibling of this lockstep frame already asked
        r.talker_ms = w->timed_talker_ms;
    } else if (w == nullptr || w->frame_serial != pending_frame_serial_
               || cudaEventElapsedTime(&r.predictor_ms, w->predictor_start, w->predictor_stop) != cudaSuccess
               || cudaEventElapsedTime(&r.talker_ms, w->talker_start, w->talker_stop) != cudaSuccess) {
        // a later frame of a shared workspace has re-recorded the timing events
        cudaGetLastError();
        r.predictor_ms = 0.0f;
        r.talker_ms = 0.0f;
    } else {
        w->timed_frame = pending_frame_serial_;
        w->timed_predictor_ms = r.predictor_ms;
        w->timed_talker_ms = r.talker_ms;
    }
    if (pending_host_codes_) std::copy_n(h_codes_, kCodebooks, r.codes);
    r.next_semantic = static_cast<uint16_t>(next);
    r.ended = next == kEos ? 1u : 0u;
    current_token_ = r.next_semantic;
    ++frames_generated;
    phase_ = r.ended ? kPhaseEnded : kPhasePrefilled;
    frame_in_flight_ = false;
    pending_host_codes_ = false;
    pending_lease_ = 0;
    pending_workspace_ = nullptr;
    return r;
}

void Session::prefill(const int32_t* text_ids, const int32_t* codec_ids, int count,
                      const SamplingParams& sampling, uint16_t* first_token, float* gpu_ms) {
    own_stream_busy_ = true;
    check_cuda(cudaSetDevice(device_), "cudaSetDevice(prefill)");
    if (poisoned_) throw std::runtime_error("talker session is poisoned and must be destroyed");
    if (frame_in_flight_) throw std::runtime_error("cannot prefill while a device frame lease is in flight");
    if (text_ids == nullptr || codec_ids == nullptr || count <= 0) {
        throw std::runtime_error("prefill requires non-empty text and codec ID arrays");
    }
    if (count > max_seq_) throw std::runtime_error("prompt exceeds the configured KV-cache capacity");
    for (int i = 0; i < count; ++i) {
        if (text_ids[i] < 0 && codec_ids[i] < 0) {
            throw std::runtime_error("a prompt position must contain text or codec input");
        }
        if (text_ids[i] >= kTextVocab || codec_ids[i] >= kTalkerVocab) {
            throw std::runtime_error("embedding token is outside its vocabulary");
        }
    }
    validate_sampling_params(sampling);
    Model& m = *model_;
    // A prompt runs as chunks of up to prefill_chunk positions per decoder pass (the rows of a
    // skinny GEMM) on the model's prompt workspace, one prompt at a time; with prefill_chunk = 1,
    // or a prompt of one position, it runs position by position on the session's own workspace.
    const ParityHooks hooks = ParityHooks::from_environment(nullptr);
    // Passes above kMaxRows exist on the tensor-core kernels only; the parity modes and hooks keep to it.
    const int most = tc_min_rows() <= kMaxRows && attention_mode() != 0 && !hooks.active() ? kMaxPromptRows : kMaxRows;
    int chunk = std::min(std::max(m.prefill_chunk, 1), most);
    // the parity hooks observe the chunked pass (they synchronise, so nothing of it may be captured)
    const bool chunked = (chunk > 1 && count > 1) || hooks.active();
    std::unique_lock<std::mutex> one_prompt(m.prefill_mutex, std::defer_lock);
    if (chunked) one_prompt.lock();
    Workspace& w = chunked ? m.prefill_workspace() : *solo_;
    if (chunked) chunk = std::min(chunk, w.rows);
    const InFlight in_flight(traffic_of(device_), w, 1, Traffic::kOther);      // until the call returns
    position_ = 0;
    generated_ = 0;
    const unsigned int errors_before = m.device_errors();
    try {
        DeviceBuffer ids(2 * (size_t)count * sizeof(int));
        int* d_text = ids.as<int>();
        int* d_codec = d_text + count;
        check_cuda(cudaMemcpyAsync(d_text, text_ids, (size_t)count * sizeof(int),
                                   cudaMemcpyHostToDevice, w.stream), "upload prompt text ids");
        check_cuda(cudaMemcpyAsync(d_codec, codec_ids, (size_t)count * sizeof(int),
                                   cudaMemcpyHostToDevice, w.stream), "upload prompt codec ids");
        check_cuda(cudaEventSynchronize(w.table_uploaded), "cudaEventSynchronize(table)");
        fill_row(*w.host_table, 0, 0, sampling, sampling, false);
        const int splits = split_bucket(count);
        w.ensure_scratch(splits);
        Session* self = this;
        bind_rows(w, &self, 1);
        check_cuda(cudaMemcpyAsync(w.table.as<void>(), w.host_table, sizeof(FrameTable),
                                   cudaMemcpyHostToDevice, w.stream), "upload frame table");
        check_cuda(cudaEventRecord(w.table_uploaded, w.stream), "cudaEventRecord(table)");
        check_cuda(cudaEventRecord(w.talker_start, w.stream), "cudaEventRecord");
        if (chunked) {
            int last_rows = 0;
            ParityHooks observed = hooks;
            observed.stream = w.stream;
            for (int base = 0; base < count; base += chunk) {
                last_rows = std::min(chunk, count - base);
                if (hooks.active() && base + last_rows == count) {
                    const Probe probe = observed.probe(last_rows - 1);     // the last prompt position
                    enqueue_prompt_chunk(w, m, d_text, d_codec, base, last_rows, splits, w.stream, &probe);
                } else {
                    enqueue_prompt_chunk(w, m, d_text, d_codec, base, last_rows, splits, w.stream);
                }
            }
            if (last_rows > 1) {
                // the head and the sampler read row 0: bring the last position's hidden state there
                const size_t row_bytes = (size_t)m.talker.hidden * sizeof(bf16);
                check_cuda(cudaMemcpyAsync(w.hidden.as<bf16>(),
                                           w.hidden.as<bf16>() + (size_t)(last_rows - 1) * m.talker.hidden,
                                           row_bytes, cudaMemcpyDeviceToDevice, w.stream), "last prompt row");
            }
        } else if (m.use_graphs) {
            // The prompt ids live in a buffer of this call, so the captured step graph is rebuilt
            // per prefill; capture costs far less than the steps it replays.
            cudaGraphExec_t step = capture(w.stream, [&] {
                enqueue_prompt_step(w, m, d_text, d_codec, splits, w.stream);
            });
            try {
                for (int i = 0; i < count; ++i) {
                    check_cuda(cudaGraphLaunch(step, w.stream), "cudaGraphLaunch(prompt step)");
                }
            } catch (...) {
                cudaStreamSynchronize(w.stream);
                cudaGraphExecDestroy(step);
                throw;
            }
            check_cuda(cudaStreamSynchronize(w.stream), "cudaStreamSynchronize(prompt)");
            cudaGraphExecDestroy(step);
        } else {
            for (int i = 0; i < count; ++i) enqueue_prompt_step(w, m, d_text, d_codec, splits, w.stream);
        }
        enqueue_talker_head(w, m, 1, 0, w.stream);
        if (hooks.active()) {
            ParityHooks observed = hooks;
            observed.stream = w.stream;
            observed.vector_line("final_norm", m.talker.layers, w.normalized.as<bf16>(), m.talker.hidden);
            observed.dump("final_logits", w.logits.as<bf16>(), kTalkerVocab);
            observed.logits_line(w.logits.as<bf16>(), kTalkerVocab);
        }
        check_cuda(cudaEventRecord(w.talker_stop, w.stream), "cudaEventRecord");
        check_cuda(cudaStreamSynchronize(w.stream), "synchronize sampled token");
        ++host_sync_count;
        ++device_sample_count;
        check_cuda(cudaEventElapsedTime(gpu_ms, w.talker_start, w.talker_stop), "cudaEventElapsedTime");
        m.check_device_errors(errors_before);
    } catch (...) {
        cudaStreamSynchronize(w.stream);
        poisoned_ = true;
        throw;
    }
    const int first = *h_token_;
    if (first < 0 || first >= kTalkerVocab) throw std::runtime_error("device sampler returned an invalid token");
    position_ = count;
    generated_ = 1;
    current_token_ = static_cast<uint16_t>(first);
    phase_ = first == kEos ? kPhaseEnded : kPhasePrefilled;
    *first_token = current_token_;
}

void Session::run_frames(Model* model, Session** s, int n, int frames, int trailing_text,
                         const SamplingParams& talker, const SamplingParams& predictor,
                         float* frame_ms, float* total_ms) {
    if (model == nullptr || s == nullptr || n <= 0 || n > kMaxRows || frames <= 0) {
        throw std::runtime_error("invalid frame-loop arguments");
    }
    check_cuda(cudaSetDevice(model->device()), "cudaSetDevice(frame loop)");
    for (int i = 0; i < n; ++i) {
        if (s[i]->model_.get() != model) throw std::runtime_error("session belongs to a different model");
        for (int j = 0; j < i; ++j) {
            if (s[j] == s[i]) throw std::runtime_error("a session appears twice in one batch");
        }
        s[i]->validate_begin(s[i]->current_token_, trailing_text, talker, predictor);
        if (s[i]->position_ + frames > s[i]->max_seq_) {
            throw std::runtime_error("frame loop would overflow the talker KV cache");
        }
    }
    std::unique_lock<std::mutex> one_batch(model->batch_mutex, std::defer_lock);
    if (n > 1) one_batch.lock();
    Workspace& w = n == 1 ? *s[0]->solo_ : model->batch_workspace();
    const unsigned int errors_before = model->device_errors();
    std::vector<cudaEvent_t> marks;
    try {
        check_cuda(cudaEventSynchronize(w.table_uploaded), "cudaEventSynchronize(table)");
        int longest = 0;
        for (int i = 0; i < n; ++i) {
            s[i]->fill_row(*w.host_table, i, trailing_text, talker, predictor, false);
            longest = std::max(longest, s[i]->position_ + frames);
            check_cuda(cudaEventRecord(w.join_events[i], s[i]->stream_), "cudaEventRecord(join)");
            check_cuda(cudaStreamWaitEvent(w.stream, w.join_events[i], 0), "cudaStreamWaitEvent(join)");
        }
        w.ensure_scratch(split_bucket(longest));
        marks.resize(frames + 1, nullptr);
        for (cudaEvent_t& ev : marks) check_cuda(cudaEventCreate(&ev), "cudaEventCreate(frame mark)");
        check_cuda(cudaEventRecord(marks[0], w.stream), "cudaEventRecord(frame mark)");
        for (int f = 0; f < frames; ++f) {
            launch_frame(w, *model, s, n, f == 0, false, f);        // the device table advances itself
            check_cuda(cudaEventRecord(marks[f + 1], w.stream), "cudaEventRecord(frame mark)");
        }
        check_cuda(cudaStreamSynchronize(w.stream), "cudaStreamSynchronize(frame loop)");
        model->check_device_errors(errors_before);
        if (frame_ms != nullptr) {
            for (int f = 0; f < frames; ++f) {
                check_cuda(cudaEventElapsedTime(&frame_ms[f], marks[f], marks[f + 1]), "cudaEventElapsedTime");
            }
        }
        if (total_ms != nullptr) {
            check_cuda(cudaEventElapsedTime(total_ms, marks[0], marks[frames]), "cudaEventElapsedTime");
        }
        for (int i = 0; i < n; ++i) {
            Session* c = s[i];
            c->position_ += frames;
            c->generated_ += frames;
            c->frames_generated += frames;
            c->device_sample_count += (uint64_t)frames * kPredictorSequence;
            ++c->host_sync_count;
            const int token = *c->h_token_;
            if (token < 0 || token >= kTalkerVocab) throw std::runtime_error("device sampler returned an invalid token");
            c->current_token_ = static_cast<uint16_t>(token);
            c->phase_ = token == kEos ? kPhaseEnded : kPhasePrefilled;
        }
    } catch (...) {
        cudaStreamSynchronize(w.stream);
        for (cudaEvent_t ev : marks) if (ev != nullptr) cudaEventDestroy(ev);
        for (int i = 0; i < n; ++i) s[i]->poisoned_ = true;
        throw;
    }
    for (cudaEvent_t ev : marks) cudaEventDestroy(ev);
}

void Session::synthetic_prefill(int position, uint64_t seed) {
    own_stream_busy_ = true;
    check_cuda(cudaSetDevice(device_), "cudaSetDevice(synthetic prefill)");
    if (poisoned_) throw std::runtime_error("talker session is poisoned and must be destroyed");
    if (frame_in_flight_) throw std::runtime_error("a device frame lease is in flight");
    if (position < 1 || position >= max_seq_) {
        throw std::runtime_error("synthetic prefill position must be in [1, max_sequence_length)");
    }
    Workspace& w = *solo_;
    Model& m = *model_;
    Session* self = this;
    bind_rows(w, &self, 1);
    const int pages = (position + kPageTokens - 1) / kPageTokens;
    const KvPool& pool = *m.talker_pool;
    check_cuda(launch_fill_kv_pages(pool.slab_table(), pool.slab_shift(), pool.page_elems(),
                                    pool.plane_elems(), w.talker_pages.as<int>(), pages,
                                    pool.layers() * 2, seed * 2 + 1, w.stream), "fill KV pages");
    check_cuda(launch_fill_normal(d_last_hidden_, 2048, seed * 2 + 2, w.stream), "fill last hidden");
    const int token = static_cast<int>(seed % 2048);
    check_cuda(cudaMemcpyAsync(d_sampled_, &token, sizeof(int), cudaMemcpyHostToDevice, w.stream),
               "store semantic token");
    check_cuda(cudaMemcpyAsync(d_history_, &token, sizeof(int), cudaMemcpyHostToDevice, w.stream),
               "store semantic history");
    check_cuda(cudaStreamSynchronize(w.stream), "cudaStreamSynchronize(synthetic prefill)");
    position_ = position;
    generated_ = 1;
    current_token_ = static_cast<uint16_t>(token);
    *h_token_ = token;
    phase_ = kPhasePrefilled;
}

void Session::read_state(uint16_t* last_hidden, int* frame_tokens, unsigned long long* rng) const {
    check_cuda(cudaSetDevice(device_), "cudaSetDevice(read state)");
    check_cuda(cudaStreamSynchronize(stream_), "cudaStreamSynchronize(read state)");
    if (last_hidden != nullptr) {
        check_cuda(cudaMemcpy(last_hidden, d_last_hidden_, 2048 * sizeof(bf16), cudaMemcpyDeviceToHost),
                   "cudaMemcpy(last hidden)");
    }
    if (frame_tokens != nullptr) {
        check_cuda(cudaMemcpy(frame_tokens, d_frame_tokens_, kCodebooks * sizeof(int),
                              cudaMemcpyDeviceToHost), "cudaMemcpy(frame tokens)");
    }
    if (rng != nullptr) {
        check_cuda(cudaMemcpy(rng, d_rng_, sizeof(unsigned long long), cudaMemcpyDeviceToHost),
                   "cudaMemcpy(rng)");
    }
}

void Session::read_kv(int layer, int first, int count, uint16_t* keys, uint16_t* values) const {
    check_cuda(cudaSetDevice(device_), "cudaSetDevice(read kv)");
    if (first < 0 || count < 0 || first + count > position_) {
        throw std::runtime_error("KV positions outside what the session has written");
    }
    check_cuda(cudaStreamSynchronize(stream_), "cudaStreamSynchronize(read kv)");
    const KvPool& pool = *model_->talker_pool;
    const int width = model_->talker.kv_width;
    const int hd = model_->talker.head_dim;
    const int heads = model_->talker.kv_heads;
    // a page holds [kv head][16 tokens][head_dim]: fetch the page whole, hand out token-major rows
    std::vector<uint16_t> page_copy((size_t)kPageTokens * width);
    for (int token = first; token < first + count;) {
        const int in_page = token % kPageTokens;
        const int run = std::min(kPageTokens - in_page, first + count - token);
        const int page = talker_pages_.at(token / kPageTokens);
        for (int plane = 0; plane < 2; ++plane) {
            uint16_t* out = plane == 0 ? keys : values;
            if (out == nullptr) continue;
            check_cuda(cudaMemcpy(page_copy.data(), pool.page_rows(page, layer, plane == 1),
                                  page_copy.size() * sizeof(uint16_t), cudaMemcpyDeviceToHost), "cudaMemcpy(read kv)");
            for (int t = 0; t < run; ++t) {
                for (int h = 0; h < heads; ++h) {
                    std::memcpy(out + (size_t)(token - first + t) * width + (size_t)h * hd,
                                page_copy.data() + ((size_t)h * kPageTokens + in_page + t) * hd, (size_t)hd * sizeof(uint16_t));
                }
            }
        }
        token += run;
    }
}

}  // namespace q3t
