// The training engine behind the C ABI: device arena, the kernel sequence of one step
// (forward, loss, backward, gradient exchange, optimizer) and its evaluation modes.
#pragma once
#include "batch_copies.h"
#include "kernels.cuh"
#include "result_copies.h"
#include <memory>
#include <string>
#include <vector>

// Minimal NCCL surface, resolved with dlopen so the library loads without NCCL present.
struct Nccl {
    using Comm = void *;
    struct UniqueId {
        char internal[128];
    };
    int (*GetUniqueId)(UniqueId *) = nullptr;
    int (*CommInitRank)(Comm *, int, UniqueId, int) = nullptr;
    // ncclConfig_t as NCCL 2.17 laid it out; later libraries read `size` and `version` and fill the
    // fields added since with their defaults.
    struct Config {
        size_t size;
        unsigned magic, version;
        int blocking, cga_cluster_size, min_ctas, max_ctas;
        const char *net_name;
    };
    int (*CommInitRankConfig)(Comm *, int, UniqueId, int, Config *) = nullptr; // optional (NCCL >= 2.17)
    int (*AllReduce)(const void *, void *, size_t, int, int, Comm, cudaStream_t) = nullptr;
    int (*AllGather)(const void *, void *, size_t, int, Comm, cudaStream_t) = nullptr;
    int (*CommDestroy)(Comm) = nullptr;
    const char *(*GetErrorString)(int) = nullptr;
    static const Nccl &get(); // throws when NCCL cannot be loaded
    void check(int result, const char *what) const;
    static constexpr int Float32 = 7, Bfloat16 = 9, Sum = 0;
};

enum Family {
    FSample, FEmbedding, FNorm, FGemmForward, FGemmInputGrad, FGemmWeightGrad, FAttentionForward,
    FAttentionBackward, FActivation, FCrossEntropy, FNormBackward, FEmbeddingBackward, FOptimizer, FMuon,
    FExchange, FMisc, FamilyCount
};
extern const char *const family_names[FamilyCount];

struct LayerActivations { // saved by forward for backward (reference cuda/types.cuh:40-44)
    void *x, *normed1, *qkv, *attended, *middle, *normed2, *wide, *activated; // wide: gate|up, or gelu'(pre-activation)
    int *selected;
    float *gates, *derivatives, *lse;
    float *stats1, *stats2; // per row: mean and 1/sigma of the two norms, saved by forward for backward
};

// Kernels that do not depend on one another run side by side on the engine's lanes: lane 0 is the engine's stream, the
// others carry work forked from it (weight gradients beside the input-gradient chain, the families of Muon matrices) and
// are joined before the step ends.  Each lane has its own split-K scratch.
constexpr int LaneCount = 5;
struct Lane {
    cudaStream_t stream = nullptr;
    GemmWorkspace workspace;
};
// A captured kernel sequence; pointers it holds are fixed, so it is dropped when one of them may change.
struct StepGraph {
    cudaGraphExec_t exec = nullptr;
    bool warm = false; // the sequence has run once directly, which sizes every workspace
    int64_t launches = 0;
    uint64_t generation = 0;
};
enum GraphKind { GraphTrain, GraphTrainBatch, GraphEvaluate, GraphGradients, GraphPredict, GraphKinds };

enum class RunMode { Evaluate, Gradients, Train, OptimizerOnly }; // reference cuda/trainer.cuh:6

struct Engine {
    TgConfigEx config{};
    Layout layout{};
    Dtype act = Dtype::BF16;
    int sms = 0, tokens = 0;
    bool tensor_cores = true, profile = false;
    cudaStream_t stream = nullptr, exchange_stream = nullptr;
    std::vector<void *> allocations;
    size_t allocated_bytes = 0;

    // parameters and optimizer state (flat, layout order)
    bf16 *weight_high = nullptr;
    uint16_t *weight_low = nullptr;
    float *weight_fp32 = nullptr, *momentum = nullptr, *variance = nullptr, *gradient = nullptr;
    uint8_t *adam_mode = nullptr;
    bf16 *gradient_bf16 = nullptr; // staging for BF16 gradient exchange
    // data
    uint8_t *data = nullptr, *x = nullptr, *y = nullptr;
    int64_t data_size = 0;
    // activations
    std::vector<LayerActivations> layers;
    void *final_x = nullptr, *final_normed = nullptr, *logits = nullptr;
    float *final_stats = nullptr;
    // Gradients that the weight-gradient lane reads: it may be up to two layers behind, so the buffers rotate.
    static constexpr int HiddenRing = 6, LayerRing = 2;
    void *dhidden[HiddenRing] = {}, *dbranch = nullptr, *dwide[LayerRing] = {}, *dactivated = nullptr, *dqkv[LayerRing] = {};
    float *attention_scratch = nullptr; // dt (arg-max) or delta (softmax)
    float *token_losses = nullptr, *loss_history = nullptr, *norm_partial[HiddenRing] = {}, *sumsq_partial = nullptr,
          *logits_fp32 = nullptr, *mean_loss = nullptr, *embedding_partial = nullptr;
    int norm_blocks = 0, sumsq_blocks = 0;
    StepCounters *counters = nullptr;
    TgStepRates *schedule = nullptr;
    int schedule_steps = 0;
    // Muon scratch
    struct MuonFamily { // q|k|v, attention, gate, down, up: the same matrix of every layer
        int64_t first = 0;
        int rows = 0, cols = 0;
        bf16 *x[2] = {nullptr, nullptr}, *a = nullptr, *b = nullptr;
        float *sumsq = nullptr;
        unsigned *progress = nullptr;
    };
    std::vector<MuonFamily> muon;
    bool muon_persistent = false; // the iterations in one launch for all families, or, where they share scratch, for each
    // the reference architecture's step in three kernels (reference_step.cu, small_optimizer_kernel); unset: operator by operator
    bool reference_step = false;
    ReferenceStepPlan reference_plan;
    float *reference_partial = nullptr, *reference_norm = nullptr;
    float2 *reference_rope = nullptr;
    SmallMatrix *small_matrices = nullptr;
    int small_matrix_count = 0;
    unsigned *adam_ticket = nullptr;
    // host mirrors
    uint64_t step = 0;
    int last_train_steps = 0;
    bool losses_reduced = true;
    // data parallel
    Nccl::Comm comm = nullptr;
    int gemm_sms = 0; // SMs the GEMMs of the current phase may use (fewer while a gradient bucket may be in flight)
    std::vector<cudaEvent_t> bucket_events;
    cudaEvent_t exchange_done = nullptr;
    // profiling
    struct Timed {
        int family;
        cudaEvent_t start, stop;
    };
    std::vector<Timed> timed;
    std::vector<cudaEvent_t> event_pool;
    double family_ms[FamilyCount] = {};
    int64_t family_launches[FamilyCount] = {};
    int64_t launches = 0;
    Lane lanes[LaneCount];
    int lane = 0;            // where run() launches
    bool concurrent = false; // whether work may be forked at all
    int side_lanes = 0;      // lanes of weight gradients beside the chain
    bool muon_lanes = false; // the Muon families beside each other
    std::vector<cudaEvent_t> fork_events; // as many as a backward pass marks: none is recorded again before its last wait
    size_t next_fork_event = 0;
    float *simt_scratch[3] = {nullptr, nullptr, nullptr}; // per lane: partial tiles of CUDA-core GEMMs that are cut along K (6 MB bounds every shape)
    BatchCopies copies; // of tg_batch's results
    std::shared_ptr<ResultCopies> results; // the device's, once it is worth its making
    size_t result_bytes = 0;               // that calls without it have returned
    Outbox *outbox = nullptr;          // what a call brings back with its last wait,
    std::unique_ptr<Outbox> mailbox;   // and where it arrives
    bool announce_gradients = false;
    StepGraph graphs[GraphKinds];
    int forward_batch = 0; // sequences the next forward pass covers (0: the configured batch)
    void drop_graphs();

    explicit Engine(const TgConfigEx &c);
    ~Engine();
    Engine(const Engine &) = delete;

    template <class T> void allocate(T *&p, size_t n, bool zero = true);
    const void *weight(int64_t offset) const;
    void set_device() const;

    void set_weights(const float *w);
    void get_weights(float *w);
    void set_data(const uint8_t *bytes, int64_t size);
    void set_onecycle(const TgOneCycle &s);
    void train(int steps);
    void training_losses(float *out, int count);
    void batch(const uint8_t *bx, const uint8_t *by, float *logits_out, float *gradient_out, float *per_position);
    void predict(const uint8_t *context, float *logits256);
    void optimizer_test(const float *g, int steps);
    void sample(uint64_t at_step, uint8_t *bx, uint8_t *by);
    void set_optimizer_state(const float *m, const float *v, uint64_t at_step);
    void get_optimizer_state(float *m, float *v, uint64_t *at_step);
    float train_mean_loss(int steps);
    void train_batch(const uint8_t *bx, const uint8_t *by, float *per_position);
    void flush_profile();
    int64_t read_activation(int layer, const char *name, float *out, int64_t capacity);

  private:
    struct OnLane { // run() launches on another lane while this lives
        Engine &e;
        OnLane(Engine &engine, int l) : e(engine) { e.lane = l; }
        OnLane(const OnLane &) = delete;
        ~OnLane() { e.lane = 0; }
    };
    void initialize();
    void release();
    template <class F> void run(Family f, F &&launch);
    bool on_tensor_cores(GemmArgs g) const; // whether gemm() takes it there
    void gemm(Family f, GemmArgs g);
    void forward(bool want_gradient, bool dump_logits, bool embedded = false);
    void record_losses();
    void backward();
    void exchange_bucket(int64_t begin, int64_t end, int index);
    void finish_exchange();
    void optimize();
    void muon_direction(const MuonFamily &family);
    bf16 *muon_products(const MuonFamily &family);
    bool muon_iterations(const MuonFamily *families, int count);
    void muon_apply(const MuonFamily &family, bf16 *direction);
    bool use_graphs() const { return !profile && !comm && !(config.flags & TG_FLAG_NO_GRAPH); }
    template <class F> void replay(GraphKind kind, F &&body);
    void announce(cudaEvent_t event, int on);
    cudaEvent_t mark(int on); // an event after everything lane `on` holds
    void await(int on, cudaEvent_t event);
    void fork(int from, int to) {
        if (concurrent)
            await(to, mark(from));
    }
    void prepare_reference_step();
    void reference_train_step(bool sample, bool save);
    void one_step(RunMode mode, bool last = true);
    void finish(float *out = nullptr, const float *values = nullptr, size_t count = 0);
};
