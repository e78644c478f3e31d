// Host side of the network engine: one Engine holds any number of resident
// network instances (a plain run is an engine with one instance, a sweep is
// a batch, serving adds and removes instances at step boundaries) and
// advances them together, one fused kernel launch per step or per several
// steps (Span in asg_engine.cuh), K steps per
// captured CUDA graph ("chunk").
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdint>
#include <memory>
#include <mutex>
#include <string>
#include <vector>

#include "asg_b200.h"
#include "asg_common.hpp"
#include "asg_engine.cuh"

namespace asg {

struct SpikeRec {
    std::int64_t step;
    std::uint32_t source;
};

// Where admission takes device memory: a stream-ordered pool of the engine's
// own.  (The default pool gives its memory back at every synchronisation and
// the next allocation maps it again; cudaMalloc and cudaFree wait for the
// device and, beside running chunks, took from 0.4 to tens of ms each.)  A
// server's pool also holds the arenas and keeps up to 2 GB beside them, within
// the memory budget, between requests (Engine::claim); other engines trim it
// after their last admission and take their arenas, which stay, from cudaMalloc
// (pool = nullptr).
struct Scratch {
    cudaStream_t stream;
    cudaMemPool_t pool;
    bool* no_room = nullptr;  // set when an allocation failed for lack of memory
};

// Device memory from there.  Freeing pool memory does not wait for the device
// (cudaFree would, and stall the chunks in flight): its last user must have
// finished, or be on the same stream.
struct AsyncBuf {
    void* p = nullptr;
    Scratch from{};
    AsyncBuf() = default;
    AsyncBuf(const AsyncBuf&) = delete;
    AsyncBuf& operator=(const AsyncBuf&) = delete;
    cudaError_t alloc(std::size_t bytes, const Scratch& sc) {
        from = sc;
        bytes = std::max<std::size_t>(bytes, 16);
        return sc.pool ? cudaMallocFromPoolAsync(&p, bytes, sc.pool, sc.stream) : cudaMalloc(&p, bytes);
    }
    void* get() const { return p; }
    template <class T>
    T* as() const { return static_cast<T*>(p); }
    void release() {
        if (p && from.pool) cudaFreeAsync(p, from.stream);
        if (p && !from.pool) cudaFree(p);
        p = nullptr;
    }
    ~AsyncBuf() { release(); }
};

// Mapped host buffers (spike logs, record rows) that leaving instances give
// back for the next ones: locking their pages took 4 ms of the 15 ms of
// admitting a 40,000-neuron request.  Keeps at most kKeep bytes, frees them
// with the engine's last instance; used by the admission and the stepping
// thread.
struct HostPool {
    static constexpr std::size_t kKeep = 64u << 20;
    std::mutex mu;
    std::vector<std::pair<std::size_t, void*>> kept;
    std::size_t held = 0;
    // A kept buffer of at least `bytes` and at most twice as many, the smallest,
    // or a new one of just as many (rounding sizes up so that more requests match
    // cost a server's first 270,000-neuron request 4 ms of page locking).
    cudaError_t take(std::size_t bytes, void** p, std::size_t* got);
    void give(void* p, std::size_t bytes);
    ~HostPool();
};

// Device memory of the buffers that launches of several steps need beside the
// arenas, of one or more instances; counted in the engine's total while held.
struct SpanBlock {
    AsyncBuf buf;
    std::uint64_t bytes;
    std::atomic<std::uint64_t>& total;
    SpanBlock(std::uint64_t b, std::atomic<std::uint64_t>& t) : bytes(b), total(t) { total += bytes; }
    ~SpanBlock() { total -= bytes; }
};

// One resident instance.
struct Instance {
    int id = -1;
    InstDev dev{};             // host copy of the device descriptor
    AsyncBuf arena;            // every device array of the instance
    std::size_t arena_bytes = 0;
    // Launches of several steps (see Span): the most steps this instance's
    // delays allow (1: none), the spike lists and SIC factor rows they use,
    // held while the engine runs them, and whether the factors live there now
    // or in the arena.
    int span_max = 1;
    int step_push_blocks = 0;  // PUSH items (a quarter in the wide form of several steps)
    std::shared_ptr<SpanBlock> span;
    double* span_fac = nullptr;
    std::uint32_t* span_fany = nullptr;
    bool fac_in_span = false;
    std::size_t fac_off = 0, fany_off = 0;  // the arena's factor rows and flags
    std::int64_t step = 0;     // next step to run
    std::int64_t end = INT64_MAX;
    bool done() const { return step >= end; }
    // outputs gathered on the host
    std::vector<SpikeRec> spikes;
    std::vector<std::int64_t> astro_rec_steps, neuron_rec_steps;
    std::vector<double> rec_Ca, rec_IP3, rec_V, rec_Isic;
    std::int64_t spike_edges = 0, sic_edges = 0, n_spikes = 0;
    // mapped host buffers for logs and record rows, two per parity
    unsigned long long* log_h[2] = {nullptr, nullptr};
    unsigned long long* log_d[2] = {nullptr, nullptr};
    double* rec_h[2] = {nullptr, nullptr};  // Ca | IP3 | V | Isic rows
    double* rec_d[2] = {nullptr, nullptr};
    std::shared_ptr<HostPool> host_pool;
    std::size_t log_bytes[2] = {0, 0}, rec_bytes[2] = {0, 0};
    std::uint32_t log_cap = 0;
    std::uint32_t rec_rows = 0;
    std::int64_t chunk_first[2] = {0, 0};   // first step of the chunk written to parity p
    std::int64_t chunk_last[2] = {0, 0};
    bool keep_spikes = true;
    int max_chunk = 0;  // longest chunk the output buffers were sized for
    ~Instance();
};

struct EngineConfig {
    int device = 0;
    int chunk_steps = 32;
    int block = 128;
    int use_graphs = 1;  // 1 graphs of launches (of several steps where the delays allow),
                         // -1 plain launches of one step, 2 persistent
    int sic_mode = 0;  // 0 auto, 1 fused, 2 split
    bool pdl = true;   // programmatic dependent launch between steps
    int push_mode = 0; // 0 deferred push when delays allow, 1 always in the spiking block
    std::uint64_t mem_budget = 0;
    int occupancy = 0;  // 0 auto, 1 latency form, 2 high-occupancy form of the step kernel
    bool large_total = false;  // the engine will hold 2^16+ neurons in all (auto SIC form)
    bool astro_fp32 = false;   // precision study: astrocyte update in FP32
    bool keep_memory = false;  // instances come and go (a server): see Scratch
    bool item_loop = true;     // high-occupancy form: one wave, several items per block
};

class Engine {
public:
    explicit Engine(const EngineConfig& cfg);
    ~Engine();
    int init();

    // Adds an instance from a descriptor; it runs steps [first, end).
    // add = prepare + commit.
    int add(const asg_network_desc& d, const asg_record_opts* rec, std::int64_t first,
            std::int64_t end, bool keep_spikes, int* id);
    // Validates the descriptor, builds the instance's tables and uploads its
    // arena on the upload stream.  Uses nothing the chunks in flight use, so
    // it may run on another host thread while run_chunk steps (one prepare
    // at a time).  check_budget: refuse beyond cfg.mem_budget (a caller that
    // accounts for memory itself passes false).
    int prepare(const asg_network_desc& d, const asg_record_opts* rec, std::int64_t first,
                std::int64_t end, bool keep_spikes, bool check_budget,
                std::unique_ptr<Instance>* out);
    // Gives the memory that admissions worked in back to the device (an engine
    // whose instances stay: after the last of them).
    void release_scratch();
    // Joins a prepared instance at this chunk boundary (same thread as run).
    int commit(std::unique_ptr<Instance> inst, int* id);
    int remove(int id);
    Instance* find(int id);
    // Bytes an instance of this descriptor would hold on the device.
    static int footprint(const asg_network_desc& d, int chunk_steps, std::uint64_t* bytes);

    // Runs chunks until every instance advanced by n_steps (or reached its
    // end).  Outputs are gathered into each Instance.  A call runs as equal
    // chunks of at most chunk_steps (1000 steps at chunk 512: two of 500),
    // each one captured graph.
    int run(std::int64_t n_steps);
    // One chunk of up to chunk_steps (serving loop granularity).
    int run_chunk(std::int64_t max_steps);

    // Waits for every chunk in flight and gathers its outputs.
    int flush() { return finish_pending(); }

    int pull_state(int id, asg_state* out);
    int pull_stp(int id, double* x, double* u, double* t);

    EngineConfig cfg;
    std::vector<std::unique_ptr<Instance>> insts;
    double last_ms = 0.0;
    std::int64_t last_kernels = 0;
    double total_ms = 0.0;
    std::int64_t total_kernels = 0;
    std::int64_t chunks = 0;
    double chunk_device_ms = 0.0;  // sum over collected chunks (serving)
    std::int64_t launched_kernels = 0;
    std::atomic<std::uint64_t> resident_bytes{0};  // arenas; also read by a preparing thread
    std::atomic<std::uint64_t> span_bytes{0};      // span buffers of all instances
    // Bytes a server has promised to its requests, admitted or being admitted:
    // span buffers stay out of them, and the pool keeps what it needs for more.
    void claim(std::uint64_t bytes);
    std::atomic<std::uint64_t> claimed_bytes{0};
    // The next chunk decides again whether the span buffers have room.
    void review_spans() { dirty = true; }
    cudaStream_t stream = nullptr;
    int sms = 148;

    // The next chunk first recomputes the SIC values of the arrival steps
    // step .. step+lead-1 (after a restore: the ring may come from another
    // launch mode).
    void mark_side_prime() { side_prime = true; }
    // Brings the factor rows of the instance's arena up to date (its state
    // between chunks is then all in the arena).
    int sync_arena(Instance& I);
    // The arena was overwritten (a restore): takes the factor rows from it.
    int arena_restored(Instance& I);

    int set_block(int block);
    int set_chunk(int chunk);
    int set_mode(int use_graphs);

private:
    int rebuild();          // work table + graph after the instance set changed
    // The launches of a chunk of `steps` steps take several each, or one where a
    // chunk is too short to begin, go on and end (see plan).  A call of a few
    // steps runs the single-step kernels as any engine without several steps does:
    // through the several-step kernels, one step at a time, calls of 1, 5 and 6 steps
    // took 79 -> 89 us (200,000 neurons), 25.4 -> 26.5 and 23.4 -> 25.0 us per step
    // (100,000).
    bool several_steps(int steps) const { return span > 1 && steps >= span + 2; }
    std::vector<Span> plan(int steps) const;  // the launches of a chunk
    cudaError_t issue_steps(int steps);  // step launches + side-stream SIC batches
    int copy_factors(Instance& I, bool to_span);
    int hold_span_buffers();
    int span = 1;  // most steps per launch
    int launch_chunk(int parity, int steps);
    int collect(int parity);
    void order_spikes(const unsigned long long* log, std::size_t n, std::int64_t first,
                      std::int64_t last, std::vector<SpikeRec>& out);
    std::vector<std::size_t> step_end;  // its scratch
    std::vector<std::uint32_t> by_step;
    int finish_pending();

    DevBuf d_insts, d_work;
    InstDev* h_insts[2] = {nullptr, nullptr};  // pinned staging
    unsigned long long* h_stats[2] = {nullptr, nullptr};  // pinned: per inst log_n + counters
    // [n][kStatWords]: log_n, spike_edges, sic_edges, spikes, overflow, then the
    // span spike-list headers; cleared together at the end of each chunk
    static constexpr std::size_t kStatWords = 16 + 3 * kHeaderStride;
    DevBuf d_stats;
    DevBuf d_barrier;      // GridBarrier of the persistent chunk kernel
    unsigned* h_barrier_err[2] = {nullptr, nullptr};  // pinned copy of its error word
    int persistent_grid = 0;
    std::size_t cap_insts = 0;
    // The work of one launch: [0] of one step, [1] of several.
    struct Table {
        std::vector<Work> work;
        std::vector<std::int32_t> push_blocks, push_helpers;  // by instance
        std::size_t at = 0;  // first item in d_work
        bool wide = false;   // the high-occupancy form of the kernel
        int grid = 0;        // its grid: one wave of resident blocks (0: one block per item)
    };
    Table tables[2];
    void fill_table(bool several);
    // Captured chunk graphs by length, most recently used first: the
    // chunk_steps graph and the lengths run() splits its calls into.
    static constexpr std::size_t kMaxGraphs = 4;
    std::vector<std::pair<int, cudaGraphExec_t>> graphs;
    bool graph_mode() const { return cfg.use_graphs == 0 || cfg.use_graphs == 1; }
    cudaGraphExec_t find_graph(int steps);
    int capture_graph(int steps);
    void drop_graphs();
    bool dirty = true;
    // side-stream SIC batches (instances with InstDev::sic_side)
    static constexpr int kSideEvents = 8;
    cudaStream_t side = nullptr;
    cudaStream_t upload = nullptr;  // table uploads of add(), beside the chunks in flight
    cudaMemPool_t pool = nullptr;  // admission scratch (and a server's arenas)
    int prepare_instance(const asg_network_desc& d, const asg_record_opts* rec, std::int64_t first,
                         std::int64_t end, bool keep_spikes, bool check_budget, bool on_device,
                         bool* no_room, std::unique_ptr<Instance>* out);
    std::shared_ptr<HostPool> host_pool = std::make_shared<HostPool>();
    std::vector<Work> side_work;
    DevBuf d_side_work;
    int side_lead = 0, side_lead_max = 0;
    bool side_prime = true;
    cudaError_t prime_side();
    cudaEvent_t ev_side_fork = nullptr, ev_side_join = nullptr;
    cudaEvent_t ev_side_pre[kSideEvents] = {}, ev_side_done[kSideEvents] = {};
    cudaEvent_t ev_start = nullptr, ev_end = nullptr;
    cudaEvent_t ev_chunk[2] = {nullptr, nullptr};
    cudaEvent_t ev_chunk0[2] = {nullptr, nullptr};
    bool pending[2] = {false, false};
    std::size_t launched_insts[2] = {0, 0};
    int next_parity = 0;
    int next_id = 0;
};

}  // namespace asg
