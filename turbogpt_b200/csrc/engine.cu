// Engine: allocation and the kernel sequence of the dense training step.  The reference runs the
// whole step inside one persistent cooperative kernel sized for a 16-wide model
// (cuda/trainer.cuh:103-125); here a step is a stream of large kernels — tcgen05 GEMMs, fused
// attention, 128-bit elementwise passes, one optimizer pass — with all per-step control
// (sampling seed, schedule point, loss-history row) read from device-resident counters.
#include "engine.h"
#include <algorithm>
#include <array>
#include <cmath>
#include <cstring>
#include <dlfcn.h>
#include <iterator>
#include <type_traits>

constexpr int64_t TwoSideLanes = int64_t(1) << 22; // tokens x columns up to which weight gradients have two lanes
constexpr size_t SimtScratchBytes = SplitScratchBytes; // bounds gemm_simt_scratch_bytes for every shape it cuts

const char *const family_names[FamilyCount] = {
    "sample", "embedding", "norm", "gemm_forward", "gemm_input_grad", "gemm_weight_grad", "attention_forward",
    "attention_backward", "activation", "cross_entropy", "norm_backward", "embedding_backward", "optimizer",
    "muon", "gradient_exchange", "misc"};

// ------------------------------------------------------------------------------- NCCL --------
const Nccl &Nccl::get() {
    static Nccl api;
    static bool loaded = false;
    static std::string failure;
    if (!loaded && failure.empty()) {
        void *lib = nullptr;
        if (const char *path = getenv("TURBOGPT_NCCL_LIBRARY"))
            lib = dlopen(path, RTLD_NOW | RTLD_GLOBAL);
        for (const char *name : {"libnccl.so.2", "libnccl.so"})
            if (!lib)
                lib = dlopen(name, RTLD_NOW | RTLD_GLOBAL);
        if (!lib) {
            failure = "NCCL library not found (set TURBOGPT_NCCL_LIBRARY)";
        } else {
            api.GetUniqueId = reinterpret_cast<decltype(api.GetUniqueId)>(dlsym(lib, "ncclGetUniqueId"));
            api.CommInitRank = reinterpret_cast<decltype(api.CommInitRank)>(dlsym(lib, "ncclCommInitRank"));
            api.CommInitRankConfig =
                reinterpret_cast<decltype(api.CommInitRankConfig)>(dlsym(lib, "ncclCommInitRankConfig"));
            api.AllReduce = reinterpret_cast<decltype(api.AllReduce)>(dlsym(lib, "ncclAllReduce"));
            api.AllGather = reinterpret_cast<decltype(api.AllGather)>(dlsym(lib, "ncclAllGather"));
            api.CommDestroy = reinterpret_cast<decltype(api.CommDestroy)>(dlsym(lib, "ncclCommDestroy"));
            api.GetErrorString = reinterpret_cast<decltype(api.GetErrorString)>(dlsym(lib, "ncclGetErrorString"));
            if (!api.GetUniqueId || !api.CommInitRank || !api.AllReduce || !api.AllGather || !api.CommDestroy)
                failure = "NCCL library lacks a required symbol";
            else
                loaded = true;
        }
    }
    if (!loaded)
        throw std::runtime_error(failure);
    return api;
}
void Nccl::check(int result, const char *what) const {
    if (result != 0)
        throw std::runtime_error(std::string(what) + ": " +
                                 (GetErrorString ? GetErrorString(result) : "NCCL error"));
}

constexpr int ReferenceGraphSteps = 8; // steps of the reference architecture (three kernels each) per captured graph
constexpr int ExchangeSms = 4; // CTAs of the gradient all-reduce = SMs the backward GEMMs leave free for it

// ------------------------------------------------------------------------------- setup -------
template <class T> void Engine::allocate(T *&p, size_t n, bool zero) {
    void *raw = nullptr;
    size_t bytes = std::max<size_t>(n * sizeof(T), 16);
    CHECK_CUDA(cudaMalloc(&raw, bytes));
    p = static_cast<T *>(raw);
    allocations.push_back(raw);
    allocated_bytes += bytes;
    if (zero)
        CHECK_CUDA(cudaMemsetAsync(raw, 0, bytes, stream));
}
void Engine::set_device() const { CHECK_CUDA(cudaSetDevice(config.base.device)); }
const void *Engine::weight(int64_t offset) const {
    return act == Dtype::BF16 ? (const void *)(weight_high + offset) : (const void *)(weight_fp32 + offset);
}

Engine::Engine(const TgConfigEx &c) : config(c) {
    try {
        initialize();
    } catch (...) {
        release();
        throw;
    }
}
Engine::~Engine() { release(); }

void Engine::initialize() {
    const TgConfigEx &c = config;
    validate_config(c);
    layout = make_layout(c);
    if (layout.count > (int64_t(1) << 31) - 1)
        throw std::runtime_error("parameter count exceeds signed 32-bit indexing of the engine interface");
    set_device();
    cudaDeviceProp prop{};
    CHECK_CUDA(cudaGetDeviceProperties(&prop, c.base.device));
    if (prop.major != 10)
        throw std::runtime_error("This library is built for sm_100a (B200); device is sm_" +
                                 std::to_string(prop.major) + std::to_string(prop.minor));
    sms = c.base.blocks > 0 ? std::min(c.base.blocks, prop.multiProcessorCount) : prop.multiProcessorCount;
    act = c.precision == TG_PRECISION_FP32 ? Dtype::FP32 : Dtype::BF16;
    tensor_cores = !(c.flags & TG_FLAG_NO_TENSOR_CORES);
    profile = c.flags & TG_FLAG_PROFILE;
    tokens = c.base.batch * c.base.context;
    gemm_sms = sms;
    CHECK_CUDA(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking));
    lanes[0].stream = stream;
    // Profiling times kernels one at a time, and gradient buckets leave in the order the layers finish: both keep one lane.
    concurrent = !profile && c.world == 1 && tensor_cores;
    // Above these sizes one product fills the GPU for several rounds of tiles and a second lane has nothing to fill; the step
    // is then bound by power and the lanes cost what they add.  Measured per step, one lane -> two: 12 layers d 768, 4096
    // tokens 4.85 -> 4.32 ms, 8192 7.27 -> 7.05, 16384 12.44 -> 12.2, 32768 no difference; 16 layers d 1024, 32768 tokens
    // 71.2 -> 71.5 ms.  Muon families: 6 layers d 384 1.74 -> 1.58 ms; 12 layers d 768 and 16 layers d 1024 no difference.
    // With one lane of weight gradients that lane was as long as the chain (4 layers d 256, 2048 tokens: 48 us a layer each, four gradients
    // of 10 us on 4 to 16 SMs one after another), and nothing that shortened the chain showed.  One lane -> two: that step 394 -> 384 us,
    // with attention's backward pass in one launch 401 -> 361; 6 layers d 384, 2331 tokens with Muon 1219 -> 1141 us; 8 layers d 512, 4096 tokens 2206 -> 2189,
    // 12 layers d 768, 4096 tokens 1 %, 8192 tokens level; 8 layers d 640, 8192 tokens and 14 layers d 960, 8192 tokens 0.2 and 0.7 % slower.  Three: slower
    // than two everywhere (361 -> 369 us).
    const int64_t work = int64_t(tokens) * c.width;
    // FP32 products fill the GPU from width 64 on, and a second lane of them is in the chain's way (training steps, one lane -> two, level to 4 %
    // longer; no lane at all 5 to 15 %); the widths of the reference architecture, on CUDA cores, leave it idle over many tokens: 4 layers d 16, 64 tokens
    // 560 -> 567 us, 256 tokens 1127 -> 725, 11520 tokens 1096 -> 973.
    const bool second = work <= TwoSideLanes && (act == Dtype::BF16 || (c.width < 64 && tokens >= 256));
    side_lanes = !concurrent || work > int64_t(1) << 24 ? 0 : second ? 2 : 1;
    muon_lanes = concurrent && c.hidden_optimizer == TG_HIDDEN_MUON && int64_t(c.base.depth) * c.width * c.width <= int64_t(1) << 22;
    for (int l = 1; l < (muon_lanes ? LaneCount : 1 + side_lanes); ++l)
        CHECK_CUDA(cudaStreamCreateWithFlags(&lanes[l].stream, cudaStreamNonBlocking));

    const int64_t P = layout.count;
    const int W = c.width, Hd = c.hidden, T = c.base.context, depth = c.base.depth;
    const size_t e = dtype_size(act), M = size_t(tokens);
    allocate(weight_high, P);
    allocate(weight_low, P);
    if (act == Dtype::FP32)
        allocate(weight_fp32, P);
    allocate(momentum, P);
    allocate(variance, P);
    allocate(gradient, P);
    allocate(adam_mode, P / 8);
    allocate(x, M);
    allocate(y, M);
    uint8_t *records = nullptr; // the counters and, right behind them, the losses: one copy takes both
    allocate(records, sizeof(StepCounters) + size_t(MaxLaunchSteps) * T * sizeof(float));
    counters = reinterpret_cast<StepCounters *>(records);
    loss_history = reinterpret_cast<float *>(counters + 1);
    allocate(token_losses, M);
    allocate(mean_loss, 1);

    const int wide = c.mlp == TG_MLP_SWIGLU ? 2 * Hd : Hd;
    layers.resize(depth);
    auto bytes = [&](void *&p, size_t elements) {
        uint8_t *raw = nullptr;
        allocate(raw, elements * e, false);
        p = raw;
    };
    for (LayerActivations &a : layers) {
        bytes(a.x, M * W);
        bytes(a.normed1, M * W);
        bytes(a.qkv, M * 3 * W);
        bytes(a.attended, M * W);
        bytes(a.middle, M * W);
        bytes(a.normed2, M * W);
        bytes(a.wide, M * wide);
        bytes(a.activated, M * Hd);
        a.selected = nullptr, a.gates = a.derivatives = a.lse = nullptr;
        allocate(a.stats1, M * 2, false);
        allocate(a.stats2, M * 2, false);
        if (c.attention == TG_ATTENTION_ARGMAX) {
            allocate(a.selected, M * c.heads, false);
            allocate(a.gates, M * c.heads, false);
            allocate(a.derivatives, M * c.heads, false);
        } else {
            allocate(a.lse, M * c.heads, false);
        }
    }
    bytes(final_x, M * W);
    bytes(final_normed, M * W);
    allocate(final_stats, M * 2, false);
    bytes(logits, M * Vocabulary);
    // A ring's buffers lie in one allocation (a cudaMalloc of a megabyte or more takes 0.3 ms, whatever its size).  Without a
    // side lane to wait for, the rings are no longer than the chain itself needs.
    auto ring = [&](auto &slots, size_t distinct, size_t bytes_each) {
        uint8_t *raw = nullptr;
        bytes_each = (bytes_each + 255) / 256 * 256;
        allocate(raw, distinct * bytes_each, false);
        for (size_t i = 0; i < std::size(slots); ++i)
            slots[i] = reinterpret_cast<std::remove_reference_t<decltype(slots[i])>>(raw + i % distinct * bytes_each);
    };
    ring(dhidden, side_lanes ? HiddenRing : 2, M * W * e);
    bytes(dbranch, M * W);
    ring(dwide, side_lanes ? LayerRing : 1, M * wide * e);
    ring(dqkv, side_lanes ? LayerRing : 1, M * 3 * W * e);
    bytes(dactivated, M * Hd);
    allocate(attention_scratch,
             std::max<size_t>(size_t(M) * c.heads, flash_attention_backward_scratch_bytes(c.base.batch, T, c.heads) / sizeof(float)),
             false);
    ring(simt_scratch, 1 + side_lanes, SimtScratchBytes); // the lanes of the forward and backward pass
    norm_blocks = norm_backward_blocks(tokens, sms);
    ring(norm_partial, side_lanes ? HiddenRing : 1, size_t(norm_blocks) * 2 * W * sizeof(float));
    if (embedding_backward_sliced(tokens, W))
        allocate(embedding_partial, size_t(EmbeddingSlices) * Vocabulary * W, false);
    sumsq_blocks = sms * 8;
    allocate(sumsq_partial, sumsq_blocks);
    allocate(adam_ticket, 1);

    // Per 8 parameters: 0 = Muon, 1 = AdamW, 2 = AdamW with decay (reference cuda/optim.cuh:5-15:
    // decay on the head only; with AdamW on hidden matrices they decay too; a tied embedding is the head).
    std::vector<uint8_t> mode(P / 8, 1);
    bool any_muon = false;
    for (const TensorInfo &t : layout.tensors) {
        uint8_t m = 1;
        if (t.kind == 3)
            m = 2;
        else if (t.kind == 2) {
            m = c.hidden_optimizer == TG_HIDDEN_MUON ? 0 : 2;
            any_muon |= m == 0;
        }
        int64_t count = int64_t(t.rows) * (t.cols ? t.cols : 1);
        std::fill(mode.begin() + t.offset / 8, mode.begin() + (t.offset + count) / 8, m);
    }
    CHECK_CUDA(cudaMemcpyAsync(adam_mode, mode.data(), mode.size(), cudaMemcpyHostToDevice, stream));
    CHECK_CUDA(cudaStreamSynchronize(stream)); // `mode` is about to go out of scope
    if (any_muon) { // q, k and v orthogonalised as one matrix (reference cuda/optim.cuh:109-117)
        const LayerOffsets &p = layout.layers[0];
        muon.push_back({p.qkv, 3 * W, W});
        muon.push_back({p.attention, W, W});
        muon.push_back({p.gate, Hd, W});
        muon.push_back({p.down, W, Hd});
        if (c.mlp == TG_MLP_SWIGLU)
            muon.push_back({p.up, Hd, W});
        auto side = [](const MuonFamily &f) { return size_t(std::min(f.rows, f.cols)); };
        auto padded = [&](size_t elements) { return (elements * depth + 127) / 128 * 128; };
        // Side by side the families need scratch of their own, one after another the largest family's serves all.
        size_t matrix = 0, square = 0, total = 0;
        for (const MuonFamily &f : muon) {
            matrix = std::max(matrix, padded(size_t(f.rows) * f.cols)), square = std::max(square, padded(side(f) * side(f)));
            total += 2 * (padded(size_t(f.rows) * f.cols) + padded(side(f) * side(f)));
        }
        bf16 *scratch = nullptr;
        float *sumsq = nullptr;
        allocate(scratch, muon_lanes ? total : 2 * (matrix + square), false);
        allocate(sumsq, (muon_lanes ? muon.size() : 1) * depth * MuonBlocks);
        unsigned *progress = nullptr;
        allocate(progress, muon.size() * depth);
        muon_persistent = tensor_cores && c.world == 1;
        for (MuonFamily &f : muon) {
            if (muon_lanes)
                matrix = padded(size_t(f.rows) * f.cols), square = padded(side(f) * side(f));
            f.x[0] = scratch, f.x[1] = f.x[0] + matrix, f.a = f.x[1] + matrix, f.b = f.a + square, f.sumsq = sumsq;
            if (muon_lanes)
                scratch = f.b + square, sumsq += depth * MuonBlocks;
            f.progress = progress, progress += depth;
            muon_persistent &= newton_schulz_supported(f.rows, f.cols, f.x[0]);
        }
    }
    if (tensor_cores && !profile && c.world == 1 && reference_step_supported(c))
        prepare_reference_step();
    if (c.world > 1 && !(c.flags & TG_FLAG_NO_COMMUNICATOR)) {
        const Nccl &nccl = Nccl::get();
        Nccl::UniqueId id;
        memcpy(id.internal, c.nccl_id, sizeof(id.internal));
        // The GEMM kernel is one persistent CTA per SM holding all of its shared memory, so a collective
        // kernel cannot share an SM with it: it either waits for a GEMM to end or takes SMs the next GEMM
        // then waits for, with its tiles statically assigned.  The exchange needs little bandwidth
        // (one layer's gradients per ~1.5 ms of backward), so the communicator is limited to
        // ExchangeSms CTAs and the backward GEMMs leave that many SMs free (Engine::gemm_sms).
        if (nccl.CommInitRankConfig) {
            Nccl::Config limits{};
            limits.size = sizeof(limits), limits.magic = 0xcafebeefu, limits.version = 21700;
            limits.blocking = 1, limits.cga_cluster_size = INT32_MIN, limits.min_ctas = 1, limits.max_ctas = ExchangeSms;
            limits.net_name = nullptr;
            nccl.check(nccl.CommInitRankConfig(&comm, c.world, id, c.rank, &limits), "ncclCommInitRankConfig");
        } else {
            nccl.check(nccl.CommInitRank(&comm, c.world, id, c.rank), "ncclCommInitRank");
        }
        int least, greatest;
        CHECK_CUDA(cudaDeviceGetStreamPriorityRange(&least, &greatest));
        CHECK_CUDA(cudaStreamCreateWithPriority(&exchange_stream, cudaStreamNonBlocking, greatest));
        bucket_events.resize(depth + 2);
        for (cudaEvent_t &ev : bucket_events)
            CHECK_CUDA(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
        CHECK_CUDA(cudaEventCreateWithFlags(&exchange_done, cudaEventDisableTiming));
        if (c.flags & TG_FLAG_BF16_GRADIENT_EXCHANGE)
            allocate(gradient_bf16, P, false);
    }
    allocate(outbox, 1, false);
    mailbox = std::make_unique<Outbox>();
    copies.create(layout, depth, !comm); // under data parallelism the gradients are added up over the ranks after the pass
    CHECK_CUDA(cudaStreamSynchronize(stream));
}

void Engine::prepare_reference_step() {
    const TgConfigEx &c = config;
    reference_step = true;
    reference_plan = reference_step_plan(c, sms);
    allocate(reference_partial, size_t(reference_plan.blocks) * reference_plan.partial_stride, false);
    allocate(reference_norm, reference_plan.gradient_blocks);
    std::vector<float2> rope(c.base.context);
    for (int p = 0; p < c.base.context; ++p)
        rope[p] = make_float2(float(std::cos(double(p))), float(std::sin(double(p))));
    std::vector<SmallMatrix> matrices;
    for (const TensorInfo &t : layout.tensors)
        if (t.kind == 2)
            matrices.push_back({int(t.offset), t.rows, t.cols});
    small_matrix_count = int(matrices.size());
    allocate(reference_rope, rope.size(), false);
    allocate(small_matrices, matrices.size(), false);
    CHECK_CUDA(cudaMemcpyAsync(reference_rope, rope.data(), rope.size() * sizeof(float2), cudaMemcpyHostToDevice, stream));
    CHECK_CUDA(cudaMemcpyAsync(small_matrices, matrices.data(), matrices.size() * sizeof(SmallMatrix), cudaMemcpyHostToDevice, stream));
    CHECK_CUDA(cudaStreamSynchronize(stream)); // the host arrays are about to go out of scope
}

void Engine::release() {
    cudaSetDevice(config.base.device);
    if (stream)
        cudaStreamSynchronize(stream);
    if (exchange_stream)
        cudaStreamSynchronize(exchange_stream);
    if (comm)
        Nccl::get().CommDestroy(comm);
    drop_graphs();
    for (Lane &l : lanes)
        if (l.stream)
            cudaStreamSynchronize(l.stream);
    for (cudaEvent_t ev : fork_events)
        cudaEventDestroy(ev);
    copies.destroy();
    results.reset();
    for (auto &t : timed) {
        cudaEventDestroy(t.start);
        cudaEventDestroy(t.stop);
    }
    for (cudaEvent_t ev : event_pool)
        cudaEventDestroy(ev);
    for (cudaEvent_t ev : bucket_events)
        cudaEventDestroy(ev);
    if (exchange_done)
        cudaEventDestroy(exchange_done);
    for (void *p : allocations)
        cudaFree(p);
    for (Lane &l : lanes) {
        release_gemm_workspace(l.workspace);
        if (l.stream && l.stream != stream)
            cudaStreamDestroy(l.stream);
    }
    if (exchange_stream)
        cudaStreamDestroy(exchange_stream);
    if (stream)
        cudaStreamDestroy(stream);
}

// ------------------------------------------------------------------------------- launches ----
template <class F> void Engine::run(Family f, F &&launch) {
    ++launches;
    if (!profile) {
        launch(lanes[lane].stream);
        return;
    }
    auto take = [&] {
        if (event_pool.empty()) {
            cudaEvent_t ev;
            CHECK_CUDA(cudaEventCreate(&ev));
            return ev;
        }
        cudaEvent_t ev = event_pool.back();
        event_pool.pop_back();
        return ev;
    };
    Timed t{int(f), take(), take()};
    CHECK_CUDA(cudaEventRecord(t.start, stream));
    launch(stream);
    CHECK_CUDA(cudaEventRecord(t.stop, stream));
    timed.push_back(t);
    if (timed.size() >= 8192)
        flush_profile();
}
void Engine::flush_profile() {
    if (timed.empty())
        return;
    CHECK_CUDA(cudaStreamSynchronize(stream));
    for (Timed &t : timed) {
        float ms = 0;
        CHECK_CUDA(cudaEventElapsedTime(&ms, t.start, t.stop));
        family_ms[t.family] += ms;
        family_launches[t.family] += 1;
        event_pool.push_back(t.start);
        event_pool.push_back(t.stop);
    }
    timed.clear();
}
bool Engine::on_tensor_cores(GemmArgs g) const {
    g.in = act;
    return tensor_cores && gemm_tc_supported(g);
}
void Engine::gemm(Family f, GemmArgs g) {
    g.in = act;
    run(f, [&](cudaStream_t s) {
        if (on_tensor_cores(g))
            launches += launch_gemm_tc(g, gemm_sms, counters, s, &lanes[lane].workspace) - 1;
        else if (tensor_cores && gemm_split_supported(g))
            launch_gemm_split(g, sms, counters, s, simt_scratch[lane]);
        else
            launch_gemm_simt(g, s, gemm_simt_scratch_bytes(g) <= SimtScratchBytes ? simt_scratch[lane] : nullptr);
    });
}
// Records an event for a stream outside the captured sequence (every replay records it again).
void Engine::announce(cudaEvent_t event, int on) {
    cudaStreamCaptureStatus capturing;
    CHECK_CUDA(cudaStreamIsCapturing(lanes[on].stream, &capturing));
    CHECK_CUDA(cudaEventRecordWithFlags(event, lanes[on].stream,
                                        capturing == cudaStreamCaptureStatusActive ? cudaEventRecordExternal : cudaEventRecordDefault));
}
cudaEvent_t Engine::mark(int on) {
    if (next_fork_event == fork_events.size()) {
        cudaEvent_t event;
        CHECK_CUDA(cudaEventCreateWithFlags(&event, cudaEventDisableTiming));
        fork_events.push_back(event);
    }
    const cudaEvent_t event = fork_events[next_fork_event++];
    CHECK_CUDA(cudaEventRecord(event, lanes[on].stream));
    return event;
}
void Engine::await(int on, cudaEvent_t event) { CHECK_CUDA(cudaStreamWaitEvent(lanes[on].stream, event, 0)); }
// Waits for the stream, and reports what its kernels recorded.  `out` (may be null) first receives `count` values: the losses of training steps, which lie
// behind the counters, or what the call's last kernel has left in the outbox.  One copy, since each into ordinary memory is a wait: losses of a finished step
// 14.7 us, counters and losses in copies of their own 27, both through pinned memory 15.7 (and 0.65 ms to pin it).
void Engine::finish(float *out, const float *values, size_t count) {
    const bool together = count <= std::size(outbox->values), collected = values != loss_history;
    const size_t behind = out && together ? count : 0;
    if (out && !together)
        CHECK_CUDA(cudaMemcpyAsync(out, values, count * sizeof(float), cudaMemcpyDeviceToHost, stream));
    CHECK_CUDA(cudaMemcpyAsync(mailbox.get(), behind && collected ? static_cast<const void *>(outbox) : counters,
                               sizeof(StepCounters) + behind * sizeof(float), cudaMemcpyDeviceToHost, stream));
    CHECK_CUDA(cudaStreamSynchronize(stream));
    std::copy_n(mailbox->values, behind, out);
    flush_profile();
    if (const int code = mailbox->counters.error)
        throw std::runtime_error("a device-side wait gave up (code " + std::to_string(code) +
                                 "); results of this launch are invalid");
}

// ------------------------------------------------------------------------------- state -------
void Engine::set_weights(const float *w) {
    set_device();
    const int64_t P = layout.count;
    float *staging = act == Dtype::FP32 ? weight_fp32 : gradient; // gradient is free before a step
    CHECK_CUDA(cudaMemcpyAsync(staging, w, P * 4, cudaMemcpyHostToDevice, stream));
    launch_split_weights(staging, weight_high, weight_low, P, stream);
    CHECK_CUDA(cudaMemsetAsync(momentum, 0, P * 4, stream));
    CHECK_CUDA(cudaMemsetAsync(variance, 0, P * 4, stream));
    CHECK_CUDA(cudaMemsetAsync(counters, 0, sizeof(StepCounters), stream));
    step = 0;
    CHECK_CUDA(cudaStreamSynchronize(stream));
}
void Engine::get_weights(float *w) {
    set_device();
    const int64_t P = layout.count;
    launch_join_weights(weight_high, weight_low, gradient, P, stream); // gradient doubles as staging
    CHECK_CUDA(cudaMemcpyAsync(w, gradient, P * 4, cudaMemcpyDeviceToHost, stream));
    CHECK_CUDA(cudaStreamSynchronize(stream));
}
void Engine::set_data(const uint8_t *bytes, int64_t size) {
    drop_graphs();
    set_device();
    if (size <= 8)
        throw std::runtime_error("Dataset needs at least 9 bytes");
    if (size <= config.base.context)
        throw std::runtime_error("Dataset must be longer than the context");
    if (data)
        throw std::runtime_error("Dataset already loaded");
    allocate(data, size_t(size), false);
    data_size = size;
    CHECK_CUDA(cudaMemcpyAsync(data, bytes, size, cudaMemcpyHostToDevice, stream));
    CHECK_CUDA(cudaStreamSynchronize(stream));
}
void Engine::set_onecycle(const TgOneCycle &s) {
    drop_graphs();
    set_device();
    if (schedule || step)
        throw std::runtime_error("Set OneCycle once, before training");
    onecycle_point(s, 0); // validate before allocating
    std::vector<TgStepRates> rates(s.total_steps);
    for (int i = 0; i < s.total_steps; ++i)
        rates[i] = onecycle_point(s, i);
    allocate(schedule, rates.size(), false);
    CHECK_CUDA(cudaMemcpyAsync(schedule, rates.data(), rates.size() * sizeof(TgStepRates), cudaMemcpyHostToDevice,
                               stream));
    CHECK_CUDA(cudaStreamSynchronize(stream));
    schedule_steps = s.total_steps;
}

// ------------------------------------------------------------------------------- forward -----
// `embedded`: the sampling kernel has left the embeddings.
void Engine::forward(bool want_gradient, bool dump_logits, bool embedded) {
    const TgConfigEx &c = config;
    const int B = forward_batch ? forward_batch : c.base.batch, T = c.base.context, M = B * T;
    const int W = c.width, Hd = c.hidden, H = c.heads;
    const int depth = c.base.depth;
    const bool layer_norm = c.norm == TG_NORM_LAYER;
    auto norm = [&](const void *in, int64_t scale, int64_t bias, void *out, float *stats) {
        NormArgs a{c.norm, in, weight_high + scale, layer_norm ? weight_high + bias : nullptr, weight_low + scale,
                   layer_norm ? weight_low + bias : nullptr, out, M, W, stats, true}; // the embedding, at least, lies between them and the optimizer
        run(FNorm, [&](cudaStream_t s) { launch_norm(act, a, s); });
    };
    if (!embedded)
        run(FEmbedding, [&](cudaStream_t s) { launch_embedding(act, weight(layout.embedding), x, layers[0].x, M, W, s); });
    for (int l = 0; l < depth; ++l) {
        LayerActivations &a = layers[l];
        const LayerOffsets &p = layout.layers[l];
        void *next = l + 1 < depth ? layers[l + 1].x : final_x;
        norm(a.x, p.attention_norm, p.attention_norm_bias, a.normed1, a.stats1);
        GemmArgs qkv;
        qkv.a = a.normed1, qkv.a_row = W, qkv.b = weight(p.qkv), qkv.b_row = W, qkv.c = a.qkv, qkv.ldc = 3 * W;
        qkv.m = M, qkv.n = 3 * W, qkv.k = W, qkv.out = act;
        qkv.b_settled = !want_gradient; // the embedding, at least, lies between the weights and what wrote them
        gemm(FGemmForward, qkv);
        if (c.rope == TG_ROPE_PARTIAL)
            run(FMisc, [&](cudaStream_t s) { launch_rope(act, a.qkv, M, T, W, H, false, s); });
        if (c.attention == TG_ATTENTION_ARGMAX) {
            ArgmaxAttentionArgs at{a.qkv, a.attended, a.selected, a.gates, a.derivatives, B, T, W, H};
            run(FAttentionForward, [&](cudaStream_t s) { launch_argmax_attention(act, at, s); });
        } else {
            SoftmaxAttentionArgs at{a.qkv, a.attended, a.lse, B, T, W, H};
            run(FAttentionForward, [&](cudaStream_t s) {
                if (tensor_cores && act == Dtype::BF16 && flash_attention_supported(W, H))
                    launch_flash_attention_forward(a.qkv, a.attended, a.lse, B, T, H, counters, s);
                else if (tensor_cores && act == Dtype::FP32 && attention_split_supported(W, H))
                    launch_attention_split_forward(at, s);
                else
                    launch_softmax_attention(act, at, s);
            });
        }
        GemmArgs proj;
        proj.a = a.attended, proj.a_row = W, proj.b = weight(p.attention), proj.b_row = W, proj.c = a.middle;
        proj.ldc = W, proj.m = M, proj.n = W, proj.k = W, proj.out = act;
        proj.epilogue = Epilogue::Residual, proj.r = a.x, proj.ldr = W;
        proj.b_settled = !want_gradient;
        gemm(FGemmForward, proj);
        norm(a.middle, p.mlp_norm, p.mlp_norm_bias, a.normed2, a.stats2);
        GemmArgs up;
        up.a = a.normed2, up.a_row = W, up.b = weight(p.gate), up.b_row = W, up.c = a.wide, up.m = M, up.k = W;
        up.out = act;
        up.b_settled = !want_gradient;
        if (c.mlp == TG_MLP_SWIGLU) { // gate and up are adjacent: one projection computes both
            up.n = 2 * Hd, up.ldc = 2 * Hd;
            gemm(FGemmForward, up);
            run(FActivation, [&](cudaStream_t s) { launch_swiglu(act, a.wide, a.activated, M, Hd, s); });
        } else {
            up.n = Hd, up.ldc = Hd, up.epilogue = Epilogue::GeluDual, up.c2 = a.activated;
            if (!want_gradient && on_tensor_cores(up)) // the derivative is for the backward pass
                up.epilogue = Epilogue::Gelu, up.c = a.activated, up.c2 = nullptr;
            gemm(FGemmForward, up);
        }
        GemmArgs down;
        down.a = a.activated, down.a_row = Hd, down.b = weight(p.down), down.b_row = Hd, down.c = next;
        down.ldc = W, down.m = M, down.n = W, down.k = Hd, down.out = act;
        down.epilogue = Epilogue::Residual, down.r = a.middle, down.ldr = W;
        down.b_settled = !want_gradient;
        gemm(FGemmForward, down);
    }
    norm(final_x, layout.final_norm, layout.final_norm_bias, final_normed, final_stats);
    GemmArgs head;
    head.a = final_normed, head.a_row = W, head.b = weight(layout.head), head.b_row = W, head.c = logits;
    head.ldc = Vocabulary, head.m = M, head.n = Vocabulary, head.k = W, head.out = act;
    head.b_settled = !want_gradient;
    const float divisor = float(int64_t(B) * c.world * T);
    // Training steps take the loss and its gradient from the head product's FP32 accumulators (the reference
    // fuses them the same way, cuda/model.cuh:31-58); calls that return logits run the two kernels.
    GemmArgs fused = head;
    fused.in = act, fused.epilogue = Epilogue::CrossEntropy, fused.r = y, fused.c2 = token_losses;
    fused.c = want_gradient ? logits : nullptr, fused.alpha = 1.f / divisor;
    if (tensor_cores && !dump_logits && act == Dtype::BF16 && gemm_tc_supported(fused)) {
        gemm(FGemmForward, fused);
        return;
    }
    gemm(FGemmForward, head);
    CrossEntropyArgs ce{logits, y, token_losses, want_gradient ? logits : nullptr,
                        dump_logits ? logits_fp32 : nullptr, divisor, M};
    if (!want_gradient && (forward_batch || size_t(M) <= std::size(outbox->values))) // an evaluation's last kernel
        ce.outbox = outbox, ce.counters = counters, ce.last_logits = forward_batch;
    run(FCrossEntropy, [&](cudaStream_t s) { launch_cross_entropy(act, ce, s); });
}

// ------------------------------------------------------------------------------- backward ----
void Engine::exchange_bucket(int64_t begin, int64_t end, int index) {
    if (!comm || end <= begin)
        return;
    const Nccl &nccl = Nccl::get();
    CHECK_CUDA(cudaEventRecord(bucket_events[index], stream));
    CHECK_CUDA(cudaStreamWaitEvent(exchange_stream, bucket_events[index], 0));
    ++launches;
    if (gradient_bf16) {
        launch_cast(Dtype::FP32, gradient + begin, Dtype::BF16, gradient_bf16 + begin, end - begin, exchange_stream);
        nccl.check(nccl.AllReduce(gradient_bf16 + begin, gradient_bf16 + begin, size_t(end - begin), Nccl::Bfloat16,
                                  Nccl::Sum, comm, exchange_stream),
                   "ncclAllReduce");
        launch_cast(Dtype::BF16, gradient_bf16 + begin, Dtype::FP32, gradient + begin, end - begin, exchange_stream);
    } else {
        nccl.check(nccl.AllReduce(gradient + begin, gradient + begin, size_t(end - begin), Nccl::Float32, Nccl::Sum,
                                  comm, exchange_stream),
                   "ncclAllReduce");
    }
}
void Engine::finish_exchange() {
    if (!comm)
        return;
    CHECK_CUDA(cudaEventRecord(exchange_done, exchange_stream));
    CHECK_CUDA(cudaStreamWaitEvent(stream, exchange_done, 0));
}

// Nothing of the step waits for its row of the losses but the count of steps: beside the backward pass, which joins its lanes.
void Engine::record_losses() {
    next_fork_event = 0;
    if (side_lanes)
        fork(0, 1);
    OnLane on(*this, side_lanes ? 1 : 0);
    run(FMisc, [&](cudaStream_t s) { launch_loss_history(token_losses, loss_history, counters, config.base.batch, config.base.context, s); });
}

void Engine::backward() {
    const TgConfigEx &c = config;
    const int W = c.width, Hd = c.hidden, M = tokens, B = c.base.batch, T = c.base.context, H = c.heads;
    const int depth = c.base.depth;
    const bool layer_norm = c.norm == TG_NORM_LAYER;
    const int wide = c.mlp == TG_MLP_SWIGLU ? 2 * Hd : Hd;
    // Nothing in backward waits for a weight gradient or for the sums of a norm's scale and bias gradients: they run on
    // lanes of their own (1 .. side_lanes) beside the chain of input gradients.
    next_fork_event = 0;
    int asides = 0;
    auto aside = [&] { // launches go to the side lanes in turn, after everything the main lane holds
        const int side = side_lanes ? 1 + asides++ % side_lanes : 0;
        if (side)
            fork(0, side);
        return OnLane(*this, side);
    };
    using SideMarks = std::array<cudaEvent_t, 2>; // after everything the side lanes hold
    auto mark_sides = [&] {
        SideMarks marks{};
        for (int k = 0; k < side_lanes; ++k)
            marks[k] = mark(1 + k);
        return marks;
    };
    auto await_sides = [&](const SideMarks &marks) {
        for (int k = 0; k < side_lanes; ++k)
            await(0, marks[k]);
    };
    // dW[out, in] = dy^T x: both operands are read "MN-major" (tokens are the contraction).
    auto weight_grad = [&](const void *dy, int out, const void *xin, int in, int64_t offset) {
        const OnLane on = aside();
        GemmArgs g;
        g.a = dy, g.a_row = 1, g.a_col = out, g.b = xin, g.b_row = 1, g.b_col = in;
        g.c = gradient + offset, g.ldc = in, g.m = out, g.n = in, g.k = M, g.out = Dtype::FP32;
        gemm(FGemmWeightGrad, g);
    };
    // dx[M, in] = dy[M, out] W[out, in].
    auto input_grad = [&](const void *dy, int out, int64_t w_offset, int in, void *dx) {
        GemmArgs g;
        g.a = dy, g.a_row = out, g.b = weight(w_offset), g.b_row = 1, g.b_col = in;
        g.c = dx, g.ldc = in, g.m = M, g.n = in, g.k = out, g.out = act;
        return g;
    };
    int norms = 0;
    auto norm_back = [&](const void *xin, const void *dy, int64_t scale, int64_t bias, const void *residual,
                         void *dx, const float *stats) {
        NormBackwardArgs a{c.norm, xin, dy, weight_high + scale, weight_low + scale, residual, dx, norm_partial[norms++ % HiddenRing],
                           gradient + scale, layer_norm ? gradient + bias : nullptr, M, W, norm_blocks, stats, true};
        run(FNormBackward, [&](cudaStream_t s) { launch_norm_backward(act, a, s); });
        const OnLane on = aside();
        run(FNormBackward, [&](cudaStream_t s) { launch_norm_backward_reduce(a, s); });
    };
    int hidden = 0; // ring position of the running residual-stream gradient
    auto dh = [&] { return dhidden[hidden % HiddenRing]; };
    auto dh_next = [&] { return dhidden[(hidden + 1) % HiddenRing]; };
    // From the first bucket to the end of backward a collective may be running beside the GEMMs.
    struct Reserve {
        Engine &e;
        explicit Reserve(Engine &engine) : e(engine) {
            if (e.comm && e.sms > 4 * ExchangeSms)
                e.gemm_sms = (e.sms - ExchangeSms) & ~1;
        }
        ~Reserve() { e.gemm_sms = e.sms; }
    } reserve(*this);

    weight_grad(logits, Vocabulary, final_normed, W, layout.head);
    gemm(FGemmInputGrad, input_grad(logits, Vocabulary, layout.head, W, dbranch));
    norm_back(final_x, dbranch, layout.final_norm, layout.final_norm_bias, nullptr, dh(), final_stats);
    if (!c.tied) // final norm + head form the first bucket; a tied head waits for the embedding scatter
        exchange_bucket(layout.final_norm, layout.count, depth);
    else
        exchange_bucket(layout.final_norm, layout.final_norm + (layer_norm ? 2 : 1) * W, depth);

    std::vector<SideMarks> layer_done(depth); // the side lanes' end of each layer
    const SideMarks head_done = mark_sides();
    for (int l = depth - 1; l >= 0; --l) {
        if (l + 2 < depth)
            await_sides(layer_done[l + 2]); // its buffers are about to be written again
        void *dwide = this->dwide[l % LayerRing], *dqkv = this->dqkv[l % LayerRing];
        LayerActivations &a = layers[l];
        const LayerOffsets &p = layout.layers[l];
        weight_grad(dh(), W, a.activated, Hd, p.down);
        GemmArgs dact = input_grad(dh(), W, p.down, Hd, c.mlp == TG_MLP_SWIGLU ? dactivated : dwide);
        if (c.mlp == TG_MLP_SWIGLU) {
            gemm(FGemmInputGrad, dact);
            run(FActivation, [&](cudaStream_t s) { launch_swiglu_backward(act, a.wide, dactivated, dwide, M, Hd, s); });
        } else {
            dact.epilogue = Epilogue::GeluGrad, dact.r = a.wide, dact.ldr = Hd;
            gemm(FGemmInputGrad, dact);
        }
        weight_grad(dwide, wide, a.normed2, W, p.gate);
        gemm(FGemmInputGrad, input_grad(dwide, wide, p.gate, W, dbranch));
        norm_back(a.middle, dbranch, p.mlp_norm, p.mlp_norm_bias, dh(), dh_next(), a.stats2);
        ++hidden;

        weight_grad(dh(), W, a.attended, W, p.attention);
        gemm(FGemmInputGrad, input_grad(dh(), W, p.attention, W, dbranch));
        if (c.attention == TG_ATTENTION_ARGMAX) {
            ArgmaxAttentionBackwardArgs at{a.qkv, dbranch, a.selected, a.gates, a.derivatives, attention_scratch,
                                           dqkv, B, T, W, H};
            run(FAttentionBackward, [&](cudaStream_t s) { launch_argmax_attention_backward(act, at, s); });
        } else {
            SoftmaxAttentionBackwardArgs at{a.qkv, a.attended, dbranch, a.lse, attention_scratch, dqkv, B, T, W, H};
            run(FAttentionBackward, [&](cudaStream_t s) {
                if (tensor_cores && act == Dtype::BF16 && flash_attention_supported(W, H)) {
                    launches += launch_flash_attention_backward(a.qkv, a.attended, dbranch, a.lse, attention_scratch, dqkv, B, T, H,
                                                                counters, s) - 1;
                } else if (tensor_cores && act == Dtype::FP32 && attention_split_supported(W, H)) {
                    launch_attention_split_backward(at, s);
                } else {
                    launch_softmax_attention_backward(act, at, s);
                }
            });
        }
        if (c.rope == TG_ROPE_PARTIAL)
            run(FMisc, [&](cudaStream_t s) { launch_rope(act, dqkv, M, T, W, H, true, s); });
        weight_grad(dqkv, 3 * W, a.normed1, W, p.qkv);
        gemm(FGemmInputGrad, input_grad(dqkv, 3 * W, p.qkv, W, dbranch));
        norm_back(a.x, dbranch, p.attention_norm, p.attention_norm_bias, dh(), dh_next(), a.stats1);
        ++hidden;
        layer_done[l] = mark_sides();
        if (announce_gradients)
            for (const BatchCopies::Piece &piece : copies.pieces)
                if (piece.layer == l) {
                    if (side_lanes == 2)
                        fork(2, 1);
                    announce(piece.ready, side_lanes ? 1 : 0);
                }
        int64_t layer_end = l + 1 < depth ? layout.layers[l + 1].attention_norm : layout.final_norm;
        exchange_bucket(p.attention_norm, layer_end, l);
    }
    await_sides(head_done); // a tied head's gradient is added to
    run(FEmbeddingBackward, [&](cudaStream_t s) {
        launch_embedding_backward(act, dh(), x, gradient + layout.embedding, M, W, c.tied != 0, embedding_partial,
                                  s);
    });
    if (embedding_partial)
        ++launches; // slices kernel + sum kernel
    exchange_bucket(layout.embedding, layout.embedding + int64_t(Vocabulary) * W, depth + 1);
    finish_exchange();
    for (int side = 1; side <= side_lanes; ++side)
        fork(side, 0); // join
}

// ------------------------------------------------------------------------------- optimizer ---
// Momentum and the normalised direction, in x[0].
void Engine::muon_direction(const MuonFamily &family) {
    const TgConfigEx &c = config;
    const int depth = c.base.depth, rows = family.rows, cols = family.cols;
    const int64_t first_offset = family.first, stride = depth > 1 ? layout.layers[1].qkv - layout.layers[0].qkv : 0;
    MuonPrepareArgs prep{gradient + first_offset, momentum + first_offset, family.x[0], family.sumsq, sumsq_partial,
                         sumsq_blocks, schedule, counters, c.base.momentum, c.base.clip, rows, cols, depth, stride, family.progress};
    run(FMuon, [&](cudaStream_t s) { launch_muon_prepare(prep, s); });
    run(FMuon, [&](cudaStream_t s) { launch_muon_normalize(family.x[0], family.sumsq, int64_t(rows) * cols, depth, sms, s); });
}
// The Newton-Schulz iterations as products of their own; returns where every layer's result is.
bf16 *Engine::muon_products(const MuonFamily &family) {
    const TgConfigEx &c = config;
    const int depth = c.base.depth, rows = family.rows, cols = family.cols;
    const int r = std::min(rows, cols), n = std::max(rows, cols); // orthogonalise the wide orientation
    const int64_t per = int64_t(rows) * cols;
    // Under data parallelism the gradients are identical on every rank after the exchange, so the
    // Newton-Schulz iterations (the expensive part: 15 GEMMs per family) are sharded by layer: rank k
    // orthogonalises layers k*depth/world .. (k+1)*depth/world-1 and the BF16 results are
    // all-gathered; momentum and the weight update run for every layer on every rank, so replicas
    // stay bit-identical and any rank can write a checkpoint.
    const bool sharded = comm && depth % c.world == 0 && depth >= c.world;
    const int mine = sharded ? depth / c.world : depth, first = sharded ? c.rank * mine : 0;
    bf16 *cur = family.x[0] + first * per, *nxt = family.x[1] + first * per;
    bf16 *a_buffer = family.a + int64_t(first) * r * r, *b_buffer = family.b + int64_t(first) * r * r;
    const bool small = muon_newton_schulz_small_supported(r, n); // the reference architecture: one launch, in place
    if (small)
        run(FMuon, [&](cudaStream_t s) { launch_muon_newton_schulz_small(cur, r, n, c.base.ns_steps, mine, s); });
    for (int it = 0; !small && it < c.base.ns_steps; ++it) {
        GemmArgs a; // A = X X^T
        a.a = cur, a.a_row = n, a.b = cur, a.b_row = n, a.c = a_buffer, a.ldc = r, a.m = r, a.n = r, a.k = n;
        a.batch = mine, a.a_batch = per, a.b_batch = per, a.c_batch = int64_t(r) * r, a.out = Dtype::BF16;
        GemmArgs b; // B = -4.775 A + 2.0315 A A
        b.a = a_buffer, b.a_row = r, b.b = a_buffer, b.b_row = 1, b.b_col = r, b.c = b_buffer, b.ldc = r;
        b.m = r, b.n = r, b.k = r, b.batch = mine, b.a_batch = b.b_batch = b.c_batch = b.r_batch = int64_t(r) * r;
        b.epilogue = Epilogue::Axpby, b.alpha = 2.0315f, b.beta = -4.775f, b.r = a_buffer, b.ldr = r;
        b.out = Dtype::BF16;
        GemmArgs x2; // X' = 3.4445 X + B X
        x2.a = b_buffer, x2.a_row = r, x2.b = cur, x2.b_row = 1, x2.b_col = n, x2.c = nxt, x2.ldc = n;
        x2.m = r, x2.n = n, x2.k = r, x2.batch = mine, x2.a_batch = int64_t(r) * r;
        x2.b_batch = x2.c_batch = x2.r_batch = per;
        x2.epilogue = Epilogue::Axpby, x2.alpha = 1.f, x2.beta = 3.4445f, x2.r = cur, x2.ldr = n;
        x2.out = Dtype::BF16;
        for (GemmArgs *g : {&a, &b, &x2}) {
            run(FMuon, [&](cudaStream_t s) {
                g->in = Dtype::BF16;
                if (tensor_cores && gemm_tc_supported(*g))
                    launches += launch_gemm_tc(*g, sms, counters, s, &lanes[lane].workspace) - 1;
                else
                    launch_gemm_simt(*g, s);
            });
        }
        std::swap(cur, nxt);
    }
    bf16 *all = cur - first * per; // the buffer holding every layer's result
    if (sharded) {
        const Nccl &nccl = Nccl::get();
        run(FExchange, [&](cudaStream_t s) {
            nccl.check(nccl.AllGather(cur, all, size_t(mine) * per, Nccl::Bfloat16, comm, s), "ncclAllGather");
        });
    }
    return all;
}
// The same in one launch; false: it was refused, and the products are to be launched instead, from now on.
bool Engine::muon_iterations(const MuonFamily *families, int count) {
    NewtonSchulzArgs a;
    for (int i = 0; i < count; ++i)
        a.family[i] = {{families[i].x[0], families[i].x[1]}, families[i].a, families[i].b, families[i].rows, families[i].cols};
    a.count = count, a.batch = config.base.depth, a.steps = config.base.ns_steps, a.progress = families[0].progress, a.counters = counters;
    if (a.steps > 0)
        run(FMuon, [&](cudaStream_t s) { muon_persistent = launch_newton_schulz(a, sms, s); });
    return muon_persistent;
}
void Engine::muon_apply(const MuonFamily &family, bf16 *all) {
    const TgConfigEx &c = config;
    const int depth = c.base.depth, rows = family.rows, cols = family.cols;
    const int64_t first_offset = family.first, stride = depth > 1 ? layout.layers[1].qkv - layout.layers[0].qkv : 0;
    MuonApplyArgs apply{all, weight_high + first_offset, weight_low + first_offset,
                        weight_fp32 ? weight_fp32 + first_offset : nullptr, schedule, counters, c.base.muon_lr,
                        c.base.weight_decay, rows, cols, depth, stride};
    run(FMuon, [&](cudaStream_t s) { launch_muon_apply(apply, sms, s); });
}

void Engine::optimize() {
    const TgConfigEx &c = config;
    run(FOptimizer, [&](cudaStream_t s) { launch_sum_squares(gradient, layout.count, sumsq_partial, sumsq_blocks, s); });
    AdamArgs a{gradient, momentum, variance, weight_high, weight_low, weight_fp32, adam_mode, sumsq_partial,
               sumsq_blocks, schedule, counters, c.base.learning_rate, c.base.beta1, c.base.beta2,
               c.base.weight_decay, c.base.epsilon, c.base.clip, layout.count};
    if (muon.empty()) // the step's last kernel
        a.advance = counters, a.ticket = adam_ticket;
    next_fork_event = 0; // backward has joined its lanes
    const cudaEvent_t norm_ready = muon_lanes && !muon.empty() ? mark(0) : nullptr;
    run(FOptimizer, [&](cudaStream_t s) { launch_adamw(a, sms, s); });
    // The families are independent of one another: each on a lane of its own, but for the iterations in one launch.
    const int chains = muon_lanes ? std::min(int(muon.size()), LaneCount - 1) : 0;
    const bool together = chains && muon_persistent;
    auto join = [&] {
        for (int l = 1; l <= chains; ++l)
            fork(l, 0);
    };
    auto finish_family = [&](const MuonFamily &family, bool iterated) {
        muon_apply(family, iterated ? family.x[c.base.ns_steps % 2] : muon_products(family));
    };
    for (int l = 1; l <= chains; ++l)
        await(l, norm_ready);
    for (size_t f = 0; f < muon.size(); ++f) {
        OnLane on(*this, chains ? 1 + int(f) % chains : 0);
        muon_direction(muon[f]);
        if (!together)
            finish_family(muon[f], muon_persistent && muon_iterations(&muon[f], 1));
    }
    join();
    if (together) {
        const bool iterated = muon_iterations(muon.data(), int(muon.size()));
        for (int l = 1; l <= chains; ++l)
            fork(0, l);
        for (size_t f = 0; f < muon.size(); ++f) {
            OnLane on(*this, 1 + int(f) % chains);
            finish_family(muon[f], iterated);
        }
        join();
    }
    if (!muon.empty())
        run(FMisc, [&](cudaStream_t s) { launch_advance(counters, s); });
}

// ------------------------------------------------------------------------------- modes -------
// One optimizer step of the reference architecture.  `save`: leave the activations where read_activation finds them.
void Engine::reference_train_step(bool sample, bool save) {
    const TgConfig &b = config.base;
    ReferenceActivations saved{};
    if (save) {
        for (int l = 0; l < b.depth; ++l) {
            const LayerActivations &a = layers[l];
            saved.layer[l] = {a.x, a.normed1, a.qkv, a.attended, a.middle, a.normed2, a.activated};
        }
        saved.final_x = final_x, saved.final_normed = final_normed;
    }
    ReferenceStepArgs step{sample ? data : nullptr, data_size, b.seed, x, y, counters, weight_high, weight_low, reference_rope,
                           reference_partial, token_losses, loss_history, gradient, reference_norm, b.batch, b.context, b.depth,
                           save ? &saved : nullptr};
    run(FMisc, [&](cudaStream_t s) { launch_reference_step(step, reference_plan, s); });
    ++launches; // step kernel + reduce kernel
    SmallOptimizerArgs update{{gradient, momentum, variance, weight_high, weight_low, nullptr, adam_mode, reference_norm,
                               reference_plan.gradient_blocks, schedule, counters, b.learning_rate, b.beta1, b.beta2, b.weight_decay,
                               b.epsilon, b.clip, layout.count},
                              b.muon_lr, b.momentum, b.ns_steps, small_matrices, small_matrix_count, counters};
    run(FOptimizer, [&](cudaStream_t s) { launch_small_optimizer(update, s); });
}

// `last`: no other step follows in this call, so the activations it leaves can be read.
void Engine::one_step(RunMode mode, bool last) {
    if (mode == RunMode::Train && reference_step) {
        reference_train_step(true, last);
        return;
    }
    if (mode == RunMode::Train) {
        SampleArgs sampling{data, data_size, config.base.seed, counters, -1, config.base.batch, config.base.context,
                     config.world, config.rank, x, y};
        run(FSample, [&](cudaStream_t s) {
            if (profile) // every family has its own kernels there
                launch_sample(sampling, s);
            else
                launch_sample_embedding(act, sampling, weight(layout.embedding), layers[0].x, config.width, s);
        });
    }
    if (mode != RunMode::OptimizerOnly) {
        forward(mode != RunMode::Evaluate, mode != RunMode::Train && logits_fp32 != nullptr, mode == RunMode::Train && !profile);
        if (mode == RunMode::Gradients)
            announce(copies.forward_done, 0);
        if (mode == RunMode::Evaluate)
            return;
        if (mode == RunMode::Train)
            record_losses();
        announce_gradients = mode == RunMode::Gradients;
        backward();
        announce_gradients = false;
        if (mode == RunMode::Gradients)
            return;
    }
    optimize();
}

void Engine::drop_graphs() {
    for (StepGraph &g : graphs) {
        if (g.exec)
            cudaGraphExecDestroy(g.exec);
        g.exec = nullptr;
    }
}

// Runs a kernel sequence that reads everything that changes between calls from device memory: directly the first time (which
// sizes every workspace), then captured once and replayed.
template <class F> void Engine::replay(GraphKind kind, F &&body) {
    StepGraph &g = graphs[kind];
    if (!use_graphs() || !g.warm) {
        body();
        g.warm = true;
        return;
    }
    uint64_t generation = 0;
    for (const Lane &l : lanes)
        generation += l.workspace.generation;
    if (g.exec && g.generation != generation) { // a split-K workspace moved since the capture
        cudaGraphExecDestroy(g.exec);
        g.exec = nullptr;
    }
    if (!g.exec) {
        g.generation = generation;
        const int64_t before = launches;
        cudaGraph_t graph = nullptr;
        CHECK_CUDA(cudaStreamBeginCapture(stream, cudaStreamCaptureModeThreadLocal));
        try {
            body();
        } catch (...) {
            cudaStreamEndCapture(stream, &graph);
            if (graph)
                cudaGraphDestroy(graph);
            throw;
        }
        CHECK_CUDA(cudaStreamEndCapture(stream, &graph));
        const cudaError_t status = cudaGraphInstantiate(&g.exec, graph, 0);
        cudaGraphDestroy(graph);
        CHECK_CUDA(status);
        g.launches = launches - before;
        launches = before;
    }
    CHECK_CUDA(cudaGraphLaunch(g.exec, stream));
    launches += g.launches;
}

void Engine::train(int steps) {
    set_device();
    if (!data || steps < 1 || steps > MaxLaunchSteps)
        throw std::runtime_error("Load data first; each invocation permits 1.." + std::to_string(MaxLaunchSteps) +
                                 " steps");
    if (config.world > 1 && !comm)
        throw std::runtime_error("This engine was created without a communicator: it cannot train on its own");
    if (step + uint64_t(steps) > uint64_t(INT32_MAX))
        throw std::runtime_error("Training step count exceeds signed 32-bit indexing");
    if (schedule && step + uint64_t(steps) > uint64_t(schedule_steps))
        throw std::runtime_error("Training would exceed the OneCycle schedule");
    CHECK_CUDA(cudaMemsetAsync(&counters->iteration, 0, sizeof(int), stream));
    // The last step of a call leaves its activations for read_activation: the reference architecture's step kernel, whose
    // activations otherwise stay on chip, is launched in another form for it, outside the graph.
    const int outside = reference_step ? 1 : 0, graph_steps = reference_step ? ReferenceGraphSteps : 1;
    for (int i = 0; i < steps;) {
        if (steps - i - outside < graph_steps) {
            one_step(RunMode::Train, i + 1 == steps);
            ++i;
            continue;
        }
        replay(GraphTrain, [&] {
            for (int k = 0; k < graph_steps; ++k)
                one_step(RunMode::Train, false);
        });
        i += graph_steps;
    }
    last_train_steps = steps;
    losses_reduced = false;
    step += steps;
}

void Engine::training_losses(float *out, int count) {
    if (!out && count)
        throw std::runtime_error("Missing training loss output");
    if (count < 0 || count > last_train_steps)
        throw std::runtime_error("Training loss count exceeds the last launch");
    set_device();
    const int T = config.base.context;
    if (comm && !losses_reduced) { // per-position means of the global batch = mean over ranks
        const Nccl &nccl = Nccl::get();
        nccl.check(nccl.AllReduce(loss_history, loss_history, size_t(last_train_steps) * T, Nccl::Float32, Nccl::Sum,
                                  comm, stream),
                   "ncclAllReduce");
        losses_reduced = true;
        std::vector<float> all(size_t(last_train_steps) * T);
        CHECK_CUDA(cudaMemcpyAsync(all.data(), loss_history, all.size() * 4, cudaMemcpyDeviceToHost, stream));
        CHECK_CUDA(cudaStreamSynchronize(stream));
        for (float &v : all)
            v /= config.world;
        CHECK_CUDA(cudaMemcpyAsync(loss_history, all.data(), all.size() * 4, cudaMemcpyHostToDevice, stream));
    }
    finish(out, loss_history, size_t(count) * T);
}

float Engine::train_mean_loss(int steps) {
    train(steps);
    std::vector<float> all(size_t(steps) * config.base.context);
    training_losses(all.data(), steps);
    double sum = 0;
    for (int p = 0; p < config.base.context; ++p)
        sum += all[size_t(steps - 1) * config.base.context + p];
    return float(sum / config.base.context);
}

// Memory that CUDA knows (pinned, managed) is the copy engine's to fill, and has its pages.
static bool ordinary(const ResultCopies::Segment &s) {
    for (const char *end : {static_cast<const char *>(s.to), static_cast<const char *>(s.to) + s.bytes - 1}) {
        cudaPointerAttributes known{};
        CHECK_CUDA(cudaPointerGetAttributes(&known, end));
        if (known.type != cudaMemoryTypeUnregistered)
            return false;
    }
    return true;
}
// Bytes of a call's results where they may go through the ring: arrays in ordinary memory only, a megabyte of them together.  Small results are there as
// soon by the driver's way.
static size_t for_the_ring(const std::vector<ResultCopies::Segment> &arrays) {
    size_t bytes = 0;
    for (const ResultCopies::Segment &s : arrays) {
        if (!ordinary(s))
            return 0;
        bytes += s.bytes;
    }
    return bytes >= size_t(1) << 20 ? bytes : 0;
}

// With gradients, the results leave while the GPU is at work: the logits during the backward pass, the gradients in pieces of two
// megabytes or more as their layers are finished.
void Engine::batch(const uint8_t *bx, const uint8_t *by, float *logits_out, float *gradient_out,
                   float *per_position) {
    set_device();
    const int B = config.base.batch, T = config.base.context;
    std::vector<float> losses(tokens); // here, so that it cannot throw between the first copy into the caller's arrays and the wait for it
    if (!logits_fp32)
        allocate(logits_fp32, size_t(tokens) * Vocabulary, false);
    const size_t logit_bytes = size_t(tokens) * Vocabulary * 4, gradient_bytes = size_t(layout.count) * 4;
    // What leaves, in this order: the logits, the layers as they are finished, last first, then what is left.
    std::vector<ResultCopies::Segment> segments, arrays;
    if (logits_out) {
        segments.push_back({logits_out, logits_fp32, logit_bytes, gradient_out ? copies.stream : stream, gradient_out ? copies.forward_done : nullptr});
        arrays.push_back(segments.back());
    }
    if (gradient_out) {
        int64_t left = layout.count;
        for (const BatchCopies::Piece &piece : copies.pieces) {
            segments.push_back({gradient_out + piece.begin, gradient + piece.begin, size_t(left - piece.begin) * 4, copies.stream, piece.ready});
            left = piece.begin;
        }
        segments.push_back({gradient_out, gradient, size_t(left) * 4, stream, nullptr});
        arrays.push_back({gradient_out, gradient, gradient_bytes, stream, nullptr});
    }
    const size_t large = for_the_ring(arrays);
    CHECK_CUDA(cudaMemcpyAsync(x, bx, tokens, cudaMemcpyHostToDevice, stream));
    CHECK_CUDA(cudaMemcpyAsync(y, by, tokens, cudaMemcpyHostToDevice, stream));
    replay(gradient_out ? GraphGradients : GraphEvaluate,
           [&] {
               one_step(gradient_out ? RunMode::Gradients : RunMode::Evaluate);
               if (gradient_out && size_t(tokens) <= std::size(outbox->values))
                   run(FMisc, [&](cudaStream_t s) { launch_collect(counters, token_losses, tokens, outbox, s); });
           });
    // Of 32 MB and more the C library maps an array afresh each time; smaller ones mostly lie in memory that it has kept.
    auto kept = [](const ResultCopies::Segment &s) { return s.bytes < size_t(32) << 20 || !ordinary(s); };
    arrays.erase(std::remove_if(arrays.begin(), arrays.end(), kept), arrays.end());
    if (large && !results)
        results = ResultCopies::of(config.base.device, result_bytes += large, ResultCopies::threads_for(ResultCopies::processors()));
    if (!large || !results || !results->run(segments.data(), segments.size(), arrays.data(), arrays.size())) {
        for (const ResultCopies::Segment &s : arrays) // while the GPU computes (first calls: 76 MB 19.2 -> 16.1 ms, 340 MB 78 -> 59)
            ResultCopies::map_pages(s.to, s.bytes);
        for (const ResultCopies::Segment &s : segments) {
            if (s.ready)
                CHECK_CUDA(cudaStreamWaitEvent(s.stream, s.ready, 0));
            CHECK_CUDA(cudaMemcpyAsync(s.to, s.from, s.bytes, cudaMemcpyDeviceToHost, s.stream));
        }
        if (gradient_out)
            CHECK_CUDA(cudaStreamSynchronize(copies.stream)); // a pinned array's copy returns before it is done
    }
    finish(losses.data(), token_losses, size_t(tokens));
    if (per_position)
        for (int p = 0; p < T; ++p) { // reference cuda/runtime.cu:279-290
            double sum = 0;
            for (int b = 0; b < B; ++b)
                sum += losses[size_t(b) * T + p];
            per_position[p] = float(sum / B);
        }
}

void Engine::predict(const uint8_t *context, float *logits256) {
    if (!context || !logits256)
        throw std::runtime_error("Missing prediction input or output");
    set_device();
    const int T = config.base.context;
    if (!logits_fp32)
        allocate(logits_fp32, size_t(tokens) * Vocabulary, false);
    // One sequence through the forward pass.  The reference fills the whole batch with copies of the
    // context (cuda/runtime.cu:322-351) and reads row T-1 of the first; sequences are independent, so
    // the single row gives the same logits for 1/batch of the work.
    CHECK_CUDA(cudaMemcpyAsync(x, context, T, cudaMemcpyHostToDevice, stream));
    CHECK_CUDA(cudaMemsetAsync(y, 0, T, stream));
    forward_batch = 1;
    try {
        replay(GraphPredict, [&] { one_step(RunMode::Evaluate); });
    } catch (...) {
        forward_batch = 0;
        throw;
    }
    forward_batch = 0;
    finish(logits256, logits_fp32 + size_t(T - 1) * Vocabulary, Vocabulary);
}

void Engine::optimizer_test(const float *g, int steps) {
    set_device();
    if (steps < 1 || steps > 64)
        throw std::runtime_error("steps must be 1..64");
    if (schedule && step + uint64_t(steps) > uint64_t(schedule_steps))
        throw std::runtime_error("Optimizer test would exceed the OneCycle schedule");
    CHECK_CUDA(cudaMemcpyAsync(gradient, g, layout.count * 4, cudaMemcpyHostToDevice, stream));
    for (int i = 0; i < steps; ++i)
        one_step(RunMode::OptimizerOnly);
    step += steps;
    finish();
}

void Engine::sample(uint64_t at_step, uint8_t *bx, uint8_t *by) {
    set_device();
    if (!data)
        throw std::runtime_error("Load data first");
    SampleArgs sampling{data, data_size, config.base.seed, counters, (long long)at_step, config.base.batch,
                 config.base.context, config.world, config.rank, x, y};
    run(FSample, [&](cudaStream_t s) { launch_sample(sampling, s); });
    CHECK_CUDA(cudaMemcpyAsync(bx, x, tokens, cudaMemcpyDeviceToHost, stream));
    CHECK_CUDA(cudaMemcpyAsync(by, y, tokens, cudaMemcpyDeviceToHost, stream));
    CHECK_CUDA(cudaStreamSynchronize(stream));
}

void Engine::set_optimizer_state(const float *m, const float *v, uint64_t at_step) {
    if (!m || !v)
        throw std::runtime_error("Missing optimizer state input");
    set_device();
    CHECK_CUDA(cudaMemcpyAsync(momentum, m, layout.count * 4, cudaMemcpyHostToDevice, stream));
    CHECK_CUDA(cudaMemcpyAsync(variance, v, layout.count * 4, cudaMemcpyHostToDevice, stream));
    StepCounters host{};
    host.step = at_step;
    CHECK_CUDA(cudaMemcpyAsync(counters, &host, sizeof(host), cudaMemcpyHostToDevice, stream));
    step = at_step;
    CHECK_CUDA(cudaStreamSynchronize(stream));
}
void Engine::get_optimizer_state(float *m, float *v, uint64_t *at_step) {
    if (!m || !v || !at_step)
        throw std::runtime_error("Missing optimizer state output");
    set_device();
    CHECK_CUDA(cudaMemcpyAsync(m, momentum, layout.count * 4, cudaMemcpyDeviceToHost, stream));
    CHECK_CUDA(cudaMemcpyAsync(v, variance, layout.count * 4, cudaMemcpyDeviceToHost, stream));
    CHECK_CUDA(cudaStreamSynchronize(stream));
    *at_step = step;
}

// Diagnostic read-back of an activation the last forward pass saved (they are kept for backward).
int64_t Engine::read_activation(int layer, const char *name, float *out, int64_t capacity) {
    set_device();
    const std::string which = name ? name : "";
    const int W = config.width;
    const void *source = nullptr;
    int64_t columns = W;
    if (layer < 0) {
        if (which == "final_x")
            source = final_x;
        else if (which == "final_normed")
            source = final_normed;
    } else if (layer < int(layers.size())) {
        const LayerActivations &a = layers[layer];
        if (which == "x")
            source = a.x;
        else if (which == "normed1")
            source = a.normed1;
        else if (which == "qkv")
            source = a.qkv, columns = 3 * W;
        else if (which == "attended")
            source = a.attended;
        else if (which == "middle")
            source = a.middle;
        else if (which == "normed2")
            source = a.normed2;
        else if (which == "activated")
            source = a.activated, columns = config.hidden;
    }
    if (!source)
        throw std::runtime_error("Unknown activation '" + which + "' for layer " + std::to_string(layer));
    const int64_t count = int64_t(tokens) * columns;
    if (!out)
        return count;
    if (capacity < count)
        throw std::runtime_error("Activation buffer too small");
    if (act == Dtype::FP32) {
        CHECK_CUDA(cudaMemcpyAsync(out, source, count * 4, cudaMemcpyDeviceToHost, stream));
        CHECK_CUDA(cudaStreamSynchronize(stream));
        return count;
    }
    std::vector<uint16_t> raw(count);
    CHECK_CUDA(cudaMemcpyAsync(raw.data(), source, count * 2, cudaMemcpyDeviceToHost, stream));
    CHECK_CUDA(cudaStreamSynchronize(stream));
    for (int64_t i = 0; i < count; ++i) {
        const uint32_t bits = uint32_t(raw[i]) << 16;
        memcpy(out + i, &bits, 4);
    }
    return count;
}

// One optimizer step on bytes supplied by the caller instead of the resident corpus.
void Engine::train_batch(const uint8_t *bx, const uint8_t *by, float *per_position) {
    set_device();
    if (!bx || !by)
        throw std::runtime_error("Missing batch input");
    if (config.world > 1 && !comm)
        throw std::runtime_error("This engine was created without a communicator: it cannot train on its own");
    if (schedule && step + 1 > uint64_t(schedule_steps))
        throw std::runtime_error("Training would exceed the OneCycle schedule");
    CHECK_CUDA(cudaMemcpyAsync(x, bx, tokens, cudaMemcpyHostToDevice, stream));
    CHECK_CUDA(cudaMemcpyAsync(y, by, tokens, cudaMemcpyHostToDevice, stream));
    CHECK_CUDA(cudaMemsetAsync(&counters->iteration, 0, sizeof(int), stream));
    replay(GraphTrainBatch, [&] {
        if (reference_step) {
            reference_train_step(false, true);
            return;
        }
        forward(true, false);
        record_losses();
        backward();
        optimize();
    });
    step += 1;
    last_train_steps = 1;
    losses_reduced = false;
    if (per_position)
        training_losses(per_position, 1);
}
