// engine.cu -- the engine handle and the C ABI of the GB300 tick.
//
// An engine holds R worlds ("replicates") on one device: their agents are concatenated in
// 256-slot chunks, their bordered bit and byte planes and claim planes laid end to end, and every
// kernel of kernels.cuh serves all of them in one launch per hour.  The single-engine API
// (epi_engine_*) is the R = 1 case; the ensemble API (epi_ensemble_*) runs many replicates
// of uneven population and grid size in lockstep.  Hour segments between intervention
// points run as one captured CUDA graph, replayed with the first hour read on the device.
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <cstdio>
#include <cstring>
#include <map>
#include <memory>
#include <mutex>
#include <string>
#include <thread>
#include <tuple>
#include <utility>
#include <vector>

#include "../../include/epi_surrogate.h"
#include "host.hpp"
#include "kernels.cuh"
#include "world.cuh"

using namespace epi;
using namespace epi::kern;

// A field of the launch shape that k_commit, which takes its work from lists, has no use for: the
// value reported by default and the largest accepted, as callers know them.
constexpr int kCommitSlots = 4, kMaxCommitSlots = 8;

enum KernelKind { kKDecide = 0, kKCommit, kKSleep, kKLock, kKVaccinate, kKBuildPlane, kKCheck, kKindCount };
static const char* kKernelNames[kKindCount] = {"k_decide", "k_commit", "k_sleep", "k_lock", "k_vaccinate", "k_build_plane", "k_check"};

// A timed kernel launch: its kind and the events recorded around it.
struct TimedLaunch {
    int kind;
    cudaEvent_t begin, end;
    bool pooled;  // the pair returns to the engine's pool once read
};

// One world on the device.
struct Replica {
    epi_params p{};
    epi_geography geo0{}, geo{};
    DevParams hp{};
    uint32_t n = 0;
    InterventionState iv;
    std::vector<epi_counts> rows;
    bool active = true;
    uint32_t par = 0;  // the position and occupancy buffer that holds the current state
    // checkpoint of the host-side state (epi_engine_save_state)
    InterventionState s_iv;
    epi_geography s_geo{};
    uint32_t s_hosp_code = kHosp0;
    bool s_active = true;
    uint32_t s_par = 0;
    std::vector<epi_counts> s_rows;
};

// How one launch runs a world's hours (k_small): not, in one cluster, or on a grid of all SMs.
enum class Together { kNo, kCluster, kGrid };

struct epi_engine {
    std::vector<Replica> reps;
    uint32_t slots = 0;        // agent slots (chunk-padded replicates)
    size_t plane_bytes = 0;    // all bordered byte planes
    size_t occ_words = 0;      // all bit planes (one buffer)
    size_t claim_cells = 0;    // all claim planes
    size_t claim_bytes = 0;    // of d_claim
    int grid_blocks = 0;       // grid of the counting kernels (k_decide, k_sleep)
    int commit_slots = kCommitSlots;  // of the launch shape (k_commit takes its work from lists)
    int resident_blocks = 0;   // SMs x resident k_decide blocks per SM
    uint32_t sms = 0;
    Together together = Together::kNo;  // a world whose hours one launch runs (k_small)
    uint32_t wait_polls = kGridSpinLimit;  // SmallArgs::polls
    uint32_t together_most = 0;  // hours of the longest call that one launch runs: longest_together, 0 once a launch
                                 // shape was asked for, fewer where the autotuner found a grid faster
    // device
    DevParams* d_params = nullptr;
    uint32_t* d_chunk_rep = nullptr;  // null for a single replicate
    uint32_t *d_home = nullptr, *d_work = nullptr, *d_wsa = nullptr;
    // Positions and occupancy bit planes have two buffers each (slots and occ_words long): the
    // hours of day 7..22 write the next state to the other one, and Replica::par names the one
    // holding the replicate's current state; the other bit plane is all zero between hours.
    uint32_t *d_pos = nullptr, *d_occ = nullptr;
    uint2* d_st = nullptr;
    uint8_t* d_cls = nullptr;     // class bytes (plane_bytes)
    uint8_t* d_danger = nullptr;  // infectious-neighbour counts, same layout
    uint32_t* d_claim = nullptr;
    uint32_t* d_displaced = nullptr;  // the hour's lists (HourLists)
    uint2 *d_acts = nullptr, *d_list_n = nullptr;
    uint32_t* d_sums = nullptr;     // SmallArgs::sums
    uint32_t* d_piece_rep = nullptr;  // replicate of every kPieceWords of the bit planes (ensembles)
    uint32_t* d_par = nullptr;        // Replica::par, uploaded for the checks
    uint32_t* d_counts = nullptr;  // [hour of segment][replicate][8]
    SegDev* d_seg = nullptr;       // hour base of the running piece and first hour of the chain
    uint32_t* d_ivn = nullptr;     // per replicate: the guard's new-infections figure
    int* d_err = nullptr;
    unsigned long long* d_scratch = nullptr;
    uint32_t counts_capacity = 0;  // hours
    // host
    uint32_t* h_counts = nullptr;  // pinned mirror of d_counts
    SegDev* h_seg = nullptr;       // pinned staging of d_seg and d_ivn
    int* h_err = nullptr;          // SmallArgs::err_out (in the same allocation, as is h_ivn)
    uint32_t* h_ivn = nullptr;
    int halt_row = -1;             // chain offset of the row the guard marked in the last chain
    cudaStream_t stream = nullptr;
    bool own_stream = false;
    // piece graphs by (first hour mod 24, hours, profiling | stream << 1 | run loop << 2); a
    // profiling graph carries an event-record node before and after each kernel
    struct HourGraph {
        cudaGraphExec_t exec = nullptr;
        std::vector<TimedLaunch> events;
    };
    std::map<std::tuple<uint32_t, uint32_t, uint32_t>, HourGraph> graphs;
    std::string err;
    bool profiling = false;
    uint32_t launches[kKindCount] = {};
    double total_ms[kKindCount] = {};
    std::vector<TimedLaunch> pending;          // launches whose events are not read yet
    std::vector<cudaEvent_t> event_pool;
    std::vector<TimedLaunch>* capture = nullptr;  // set while a profiling graph is captured
    uint64_t kernels_launched = 0;
    int64_t last_claim_hour = -1;  // latest hour whose claims may sit in the claim plane (-1: clean)
    bool stop_rule = false;        // inside the run loop: hours after a replicate's stop do nothing
    uint32_t loop_hour = 0;        // next hour of a paused run loop (0: none in progress)
    uint32_t s_loop_hour = 0;      // ... at the last save_state
    const uint8_t* init_flags = nullptr;  // during creation: Csv population flags of replicate 0
    // citizen-state stream (single world): per-hour codes written by k_state_delta
    FILE* stream_file = nullptr;
    uint32_t* d_prev = nullptr;     // cell of every agent at the previous record
    uint8_t* d_codes = nullptr;     // kStreamChunk x slots
    uint2* d_exc = nullptr;         // kStreamChunk x slots (worst case: everyone jumps)
    uint32_t* d_exc_n = nullptr;    // kStreamChunk
    uint8_t* h_codes = nullptr;     // pinned mirrors
    uint2* h_exc = nullptr;
    uint32_t* h_exc_n = nullptr;
    // device-side checkpoint
    uint32_t *s_pos = nullptr, *s_wsa = nullptr;
    uint2* s_st = nullptr;
    uint32_t* s_occ = nullptr;
    uint8_t *s_cls = nullptr, *s_danger = nullptr;
    bool saved = false;

    uint32_t R() const { return (uint32_t)reps.size(); }
};

struct epi_ensemble {
    epi_engine core;
};

static thread_local std::string g_create_error;

#define CK(call)                                                                             \
    do {                                                                                     \
        cudaError_t e_ = (call);                                                             \
        if (e_ != cudaSuccess) {                                                             \
            h->err = std::string(#call) + ": " + cudaGetErrorString(e_);                     \
            return EPI_ERR_CUDA;                                                             \
        }                                                                                    \
    } while (0)

static Rect to_rect(const epi_area& a) { return Rect{a.x0, a.y0, a.x1, a.y1}; }

#ifndef EPI_DEPENDENT_LAUNCH
#define EPI_DEPENDENT_LAUNCH 1
#endif

// Launch of an hour kernel with programmatic stream serialisation: its blocks may be
// scheduled before the previous kernel of the stream has finished and wait on the device
// (dep_wait) for it, which hides the launch gap between the hour's kernels.  Captured into
// the hour graphs as programmatic edges.
template <typename... KArgs, typename... Args>
static cudaError_t launch_hour_kernel(void (*kern)(KArgs...), uint32_t blocks, cudaStream_t s, Args&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = EPI_DEPENDENT_LAUNCH;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, std::forward<Args>(args)...);
}

// Device parameters of one world: areas, random key, disease thresholds.
static DevParams make_dev_params(const epi_params& p, const epi_geography& geo0, uint32_t n) {
    DevParams d;
    std::memset(&d, 0, sizeof d);
    d.n = n;
    d.G = (int32_t)p.grid_size;
    d.W = d.G + 1;
    d.WP = d.G + 3;
    d.PW = ((uint32_t)d.G + 3u + 31u) / 32u;
    d.hosp_code = kHosp0;
    d.area[kTransport] = to_rect(geo0.transport);
    d.area[kHousing] = to_rect(geo0.housing);
    d.area[kHosp0] = to_rect(geo0.hospital);
    d.area[kHosp1] = to_rect(grown_hospital(geo0));
    d.key0 = (uint32_t)p.seed;
    d.key1 = (uint32_t)(p.seed >> 32);
    uint32_t mk[4];
    philox4x32(0u, kWorldHour, kBlkMoveKey, 0u, d.key0, d.key1, mk);
    d.move_key = mk[0];
    d.reg_start = p.regular_transmission_start_day;
    d.high_start = p.high_transmission_start_day;
    d.last_day = p.last_day;
    d.exposed_duration = p.exposed_duration;
    d.pre_duration = p.pre_symptomatic_duration;
    const double rates[3] = {0.0, p.regular_transmission_rate, p.high_transmission_rate};
    for (int c = 0; c < 3; ++c) {
        d.thr_rate[c] = bernoulli_threshold(rates[c]);
        if (rates[c] >= p.high_transmission_rate) d.hosp_if_class |= 1u << c;  // is_to_be_hospitalized
    }
    d.thr_death = bernoulli_threshold(p.death_rate);
    d.thr_symptoms = bernoulli_threshold(1.0 - p.percentage_asymptomatic_population);
    d.thr_severe = bernoulli_threshold(p.percentage_severe_infected_population);
    d.active = 1;
    return d;
}

// ------------------------------------------------------------------ launch bookkeeping
// Eagerly launched kernels take their event pair from the pool and return it once read;
// kernels captured into a profiling graph get a pair of their own, recorded as external
// event nodes, which the graph keeps and re-records at every replay.
static int record_launch_begin(epi_engine* h, int kind, cudaEvent_t* out_end) {
    if (!h->profiling) return EPI_OK;
    cudaEvent_t a, b;
    if (h->capture) {
        CK(cudaEventCreate(&a));
        CK(cudaEventCreate(&b));
        CK(cudaEventRecordWithFlags(a, h->stream, cudaEventRecordExternal));
        h->capture->push_back({kind, a, b, false});
    } else {
        if (h->event_pool.size() >= 2) {
            a = h->event_pool.back(); h->event_pool.pop_back();
            b = h->event_pool.back(); h->event_pool.pop_back();
        } else {
            CK(cudaEventCreate(&a));
            CK(cudaEventCreate(&b));
        }
        CK(cudaEventRecord(a, h->stream));
        h->pending.push_back({kind, a, b, true});
    }
    *out_end = b;
    return EPI_OK;
}

static int record_launch_end(epi_engine* h, cudaEvent_t end) {
    if (!h->profiling) return EPI_OK;
    if (h->capture) CK(cudaEventRecordWithFlags(end, h->stream, cudaEventRecordExternal));
    else CK(cudaEventRecord(end, h->stream));
    return EPI_OK;
}

// Read the pending launches' durations (the stream has been synchronised).
static int harvest_events(epi_engine* h) {
    for (auto& pe : h->pending) {
        float ms = 0.f;
        CK(cudaEventElapsedTime(&ms, pe.begin, pe.end));
        h->launches[pe.kind]++;
        h->total_ms[pe.kind] += ms;
        if (pe.pooled) {
            h->event_pool.push_back(pe.begin);
            h->event_pool.push_back(pe.end);
        }
    }
    h->pending.clear();
    return EPI_OK;
}

static void destroy_graphs(epi_engine* h) {
    for (auto& g : h->graphs) {
        cudaGraphExecDestroy(g.second.exec);
        for (auto& t : g.second.events) { cudaEventDestroy(t.begin); cudaEventDestroy(t.end); }
    }
    h->graphs.clear();
}

#define LAUNCH(kind, ...)                                                                    \
    do {                                                                                     \
        cudaEvent_t end_ = nullptr;                                                          \
        int rc_ = record_launch_begin(h, kind, &end_);                                       \
        if (rc_) return rc_;                                                                 \
        __VA_ARGS__;                                                                         \
        CK(cudaGetLastError());                                                              \
        rc_ = record_launch_end(h, end_);                                                    \
        if (rc_) return rc_;                                                                 \
    } while (0)

static int push_params(epi_engine* h) {
    std::vector<DevParams> all(h->R());
    for (uint32_t r = 0; r < h->R(); ++r) {
        Replica& rep = h->reps[r];
        const GuardParams g = guard_params(rep.p, rep.iv, rep.geo.hospital);
        rep.hp.guard_flags = g.flags;
        rep.hp.lock_threshold = g.lock_threshold;
        rep.hp.spread_threshold = g.spread_threshold;
        rep.hp.occ_threshold = g.occ_threshold;
        all[r] = rep.hp;
    }
    CK(cudaMemcpyAsync(h->d_params, all.data(), all.size() * sizeof(DevParams), cudaMemcpyHostToDevice, h->stream));
    CK(cudaStreamSynchronize(h->stream));
    return EPI_OK;
}

static int ensure_counts(epi_engine* h, uint32_t hours_needed) {
    if (hours_needed <= h->counts_capacity) return EPI_OK;
    uint32_t cap = std::max<uint32_t>(hours_needed, 48);
    if (h->d_counts) CK(cudaFree(h->d_counts));
    if (h->h_counts) CK(cudaFreeHost(h->h_counts));
    h->d_counts = nullptr;
    h->h_counts = nullptr;
    const size_t words = (size_t)cap * h->R() * 8;
    CK(cudaMalloc(&h->d_counts, words * sizeof(uint32_t)));
    CK(cudaMallocHost(&h->h_counts, words * sizeof(uint32_t)));
    h->counts_capacity = cap;
    destroy_graphs(h);  // they reference the old buffer
    return EPI_OK;
}

// ------------------------------------------------------------------ the hour loop
using DecideKernel = void (*)(const DevParams*, const uint32_t*, uint32_t, const HourBuffers, HourArgs);
using CommitKernel = void (*)(const DevParams*, const uint32_t*, uint32_t, const uint32_t*, const HourBuffers, HourArgs, uint64_t);

// Hours 2..6 of a day change nothing once hour 1 has sent everyone but hospital staff home
// (routine, citizen/mod.rs:244-248, sets current_area = home_location and nothing else), so
// when the previous hour ran in the same chain the hour's kernel is skipped and its counts
// row repeats the previous one.  (A piece that starts at hours 2..6 always starts a chain.)
static bool sleep_hour_skipped(uint32_t first_hour, uint32_t k) {
    const uint32_t hod = (first_hour + k) % 24u;
    return k > 0 && hod >= 2u && hod <= 6u;
}

// The k_decide (single world) or k_decide_ens (ensemble) instance of an hour of the day.
static DecideKernel decide_kernel(uint32_t hod, bool ensemble = false) {
#define EPI_PICK(HC) (ensemble ? (DecideKernel)k_decide_ens<HC> : (DecideKernel)k_decide<HC>)
    switch (hour_class(hod)) {
        case kHcStart: return EPI_PICK(kHcStart);
        case kHcEnd: return EPI_PICK(kHcEnd);
        case kHcTransport: return EPI_PICK(kHcTransport);
        case kHcWork: return EPI_PICK(kHcWork);
        case kHcNoon: return EPI_PICK(kHcNoon);
        case kHcHome: return EPI_PICK(kHcHome);
        default: return EPI_PICK(kHcMove);
    }
#undef EPI_PICK
}
static CommitKernel commit_kernel(bool patch, bool ensemble) {
    return ensemble ? (patch ? (CommitKernel)k_commit<true, true> : (CommitKernel)k_commit<true, false>)
                    : (patch ? (CommitKernel)k_commit<false, true> : (CommitKernel)k_commit<false, false>);
}

// The hours of day 7..22 write positions and occupancy to the other buffers, 16 a day, so the
// buffer that holds the state after hour x is the parity of the number of such hours among
// 1..x (hour_parity): a function of x mod 24.  The other hours patch the current buffers.
static bool rebuild_hour(uint32_t hod) { return hod >= 7u && hod <= 22u; }
static uint32_t* pos_buf(const epi_engine* h, uint32_t par) { return h->d_pos + (size_t)par * h->slots; }
static uint32_t* occ_buf(const epi_engine* h, uint32_t par) { return h->d_occ + (size_t)par * h->occ_words; }

static uint32_t threads_of(uint32_t n, uint32_t blocks) { return ((n + blocks - 1) / blocks + 31u) / 32u * 32u; }

// How one launch can run the world's hours: an agent per thread, a bit plane that the threads
// zero in a few stores each, and a device that schedules clusters of 16 CTAs, or an SM for
// each block.
static Together runs_together(uint32_t n, size_t occ_words, uint32_t sms) {
    if (n <= kSmallAgents && occ_words <= 16u * (size_t)kSmallCluster * threads_of(n, kSmallCluster)) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(kSmallCluster);
        cfg.blockDim = dim3(threads_of(n, kSmallCluster));
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = kSmallCluster;
        at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        int clusters = 0;
        if (cudaFuncSetAttribute(k_small<false>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
            cudaOccupancyMaxActiveClusters(&clusters, k_small<false>, &cfg) == cudaSuccess && clusters > 0)
            return Together::kCluster;
        cudaGetLastError();
    }
    const uint32_t threads = threads_of(n, sms);
    if (threads <= kSmallThreads && occ_words <= 16u * (size_t)sms * threads) {
        int dev = 0, cooperative = 0, per_sm = 0;
        if (cudaGetDevice(&dev) == cudaSuccess &&
            cudaDeviceGetAttribute(&cooperative, cudaDevAttrCooperativeLaunch, dev) == cudaSuccess && cooperative &&
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_small<true>, (int)threads, 0) == cudaSuccess && per_sm > 0)
            return Together::kGrid;
        cudaGetLastError();
    }
    return Together::kNo;
}

constexpr uint32_t kEnsembleBlockChunks = 18;  // (see the default grid)

// The group of an ensemble's launch: 1 to 16 chunks, by the time of the busiest block, whose
// chunks are whole groups and each group a switch of replicate, 0.2 chunks of time; 8 from 32
// chunks a block, where the last group is a small part.  (One GB300,
// groups of 1 / 2 / 4 / 7 / 8 / 14 / 28: 64 replicates of 50,000 agents, 13.8 chunks a block,
// 51.7 / 47.8 / 45.8 / 45.1 / 48.0 / 45.2 / 56 ms; 256 replicates on the resident grid, 142 chunks
// a block, 145 / 134 / 125.5 / 121.7 / 122.0 / 122.9 / 143 ms.  Chosen here / always 8: 4 replicates of 3,000 to
// 10,000 agents 0.61 / 1.48 ms for 100 hours, 32 of 10,000 to 100,000 2.5 / 2.7.)
static ChunkGroup chunk_group(uint32_t n_chunks, uint32_t grid) {
    uint32_t best = 8u;
    double least = 1e300;
    for (uint32_t g = 1; g <= 16u && n_chunks < 32u * (uint64_t)grid; ++g) {
        const uint64_t groups = (n_chunks + (uint64_t)g - 1u) / g, most = (groups + grid - 1u) / grid;
        const double t = (double)most * (g + 0.2);
        if (t < least) {
            least = t;
            best = g;
        }
    }
    return ChunkGroup{best, best > 1u ? (uint32_t)(((1ull << 32) + best - 1u) / best) : 0u};
}

// The arrays of a launch that starts from buffer par.
static HourBuffers hour_buffers(const epi_engine* h, uint32_t par) {
    HourBuffers b;
    b.pos = pos_buf(h, par);
    b.pos_next = pos_buf(h, 1u - par);
    b.st = h->d_st;
    b.home = h->d_home;
    b.work = h->d_work;
    b.wsa = h->d_wsa;
    b.occ = occ_buf(h, par);
    b.occ_next = occ_buf(h, 1u - par);
    b.cls = h->d_cls;
    b.danger = h->d_danger;
    b.claim = h->d_claim;
    b.lists = HourLists{h->d_displaced, h->d_acts, h->d_list_n};
    b.group = chunk_group(h->slots / kChunk, (uint32_t)h->grid_blocks);
    b.err = h->d_err;
    return b;
}

// The citizen states at the end of hour k of a piece (arguments ha), into the stream buffers.
static int record_state(epi_engine* h, uint32_t first_hour, uint32_t k, const HourArgs& ha) {
    const uint32_t n = h->reps[0].n;
    k_state_delta<<<(n + kThreads - 1) / kThreads, kThreads, 0, h->stream>>>(
        h->d_params, ha, n, pos_buf(h, hour_parity((first_hour + k) % 24u)), h->d_st, h->d_prev,
        h->d_codes + (size_t)k * h->slots, h->d_exc + (size_t)k * h->slots, h->d_exc_n + k);
    CK(cudaGetLastError());
    return EPI_OK;
}

// Kernels of one piece: hours first_hour .. first_hour + nh - 1 of a chain; the hour base is
// read on the device, so a captured piece serves every start hour with the same hour of the
// day.  A piece that does not end its chain ends after an hour of day 0.  In the run loop a
// guard follows every hour of day 0.
static int enqueue_piece(epi_engine* h, uint32_t first_hour, uint32_t nh) {
    const uint32_t row_words = h->R() * 8u;
    const uint32_t n_chunks = h->slots / kChunk;
    int last_row = -1;  // the latest hour of the piece whose counts the kernels computed
    HourArgs recorded{};  // of the hour before (the citizen-state stream)
    for (uint32_t k = 0; k < nh; ++k) {
        const uint32_t hod = (first_hour + k) % 24u;
        // rows back to the previous computed hour: within the piece, or the hour before it
        // (a day boundary, computed) unless the piece starts the chain (checked on the device)
        const uint32_t prev_back = !h->stop_rule ? 0u : (last_row >= 0 ? k - (uint32_t)last_row : 1u);
        const HourArgs ha{h->d_seg, h->d_counts, row_words, k, prev_back};
        if (h->stream_file && k > 0) {  // record the previous hour's end state before this hour changes it
            const int rc = record_state(h, first_hour, k - 1, recorded);
            if (rc) return rc;
        }
        recorded = ha;
        if (sleep_hour_skipped(first_hour, k)) continue;
        last_row = (int)k;
        if (hod >= 1u && hod <= 6u) {
            LAUNCH(kKSleep, CK(launch_hour_kernel(k_sleep, h->grid_blocks, h->stream, (const DevParams*)h->d_params,
                                                  (const uint32_t*)h->d_chunk_rep, n_chunks,
                                                  chunk_group(n_chunks, (uint32_t)h->grid_blocks).size, h->d_st, ha)));
        } else {
            const HourBuffers b = hour_buffers(h, hour_parity((hod + 23u) % 24u));
            const bool ens = h->R() > 1;
            LAUNCH(kKDecide, CK(launch_hour_kernel(decide_kernel(hod, ens), h->grid_blocks, h->stream,
                                                   (const DevParams*)h->d_params, (const uint32_t*)h->d_chunk_rep, n_chunks,
                                                   b, ha)));
            LAUNCH(kKCommit, CK(launch_hour_kernel(commit_kernel(!rebuild_hour(hod), ens), h->grid_blocks, h->stream,
                                                   (const DevParams*)h->d_params, (const uint32_t*)h->d_chunk_rep,
                                                   (uint32_t)(h->occ_words / kPieceWords), (const uint32_t*)h->d_piece_rep,
                                                   b, ha, (uint64_t)h->claim_cells)));
        }
        // the run loop's guard after every day boundary but the piece's last hour (the piece
        // end below takes that one)
        if (h->stop_rule && hod == 0u && k + 1 < nh) {
            k_piece_end<<<1, kThreads, 0, h->stream>>>(h->d_params, h->R(), h->d_seg, h->d_counts, row_words, k, 0u, h->d_ivn);
            CK(cudaGetLastError());
        }
    }
    if (h->stream_file) {
        const int rc = record_state(h, first_hour, nh - 1, recorded);
        if (rc) return rc;
    }
    const bool guard_last = h->stop_rule && (first_hour + nh - 1) % 24u == 0u;
    k_piece_end<<<1, kThreads, 0, h->stream>>>(h->d_params, h->R(), h->d_seg, h->d_counts, row_words,
                                               guard_last ? nh - 1 : kNoGuard, nh, h->d_ivn);
    CK(cudaGetLastError());
    return EPI_OK;
}

// Kernel launches of a piece, for the launch counter.
static uint64_t piece_launches(const epi_engine* h, uint32_t first_hour, uint32_t nh) {
    uint64_t n = 1;  // k_piece_end
    for (uint32_t k = 0; k < nh; ++k) {
        const uint32_t hod = (first_hour + k) % 24u;
        if (h->stream_file) n += 1;  // k_state_delta
        if (h->stop_rule && hod == 0u && k + 1 < nh) n += 1;
        if (sleep_hour_skipped(first_hour, k)) continue;
        n += (hod >= 1u && hod <= 6u) ? 1u : 2u;
    }
    return n;
}

// The graph of a piece (captured on first use).
static int piece_graph(epi_engine* h, uint32_t first_hour, uint32_t nh, cudaGraphExec_t* out,
                       std::vector<TimedLaunch>** events) {
    auto key = std::make_tuple(first_hour % 24u, nh,
                               (h->profiling ? 1u : 0u) | (h->stream_file ? 2u : 0u) | (h->stop_rule ? 4u : 0u));
    auto it = h->graphs.find(key);
    if (it == h->graphs.end()) {
        epi_engine::HourGraph hg;
        cudaGraph_t g;
        CK(cudaStreamBeginCapture(h->stream, cudaStreamCaptureModeThreadLocal));
        h->capture = &hg.events;
        int rc = enqueue_piece(h, first_hour, nh);
        h->capture = nullptr;
        cudaError_t ce = cudaStreamEndCapture(h->stream, &g);
        if (rc == EPI_OK && ce == cudaSuccess) {
            ce = cudaGraphInstantiate(&hg.exec, g, 0);
            cudaGraphDestroy(g);
        }
        if (rc != EPI_OK || ce != cudaSuccess) {
            for (auto& t : hg.events) { cudaEventDestroy(t.begin); cudaEventDestroy(t.end); }
            if (rc) return rc;
            h->err = std::string("hour graph: ") + cudaGetErrorString(ce);
            return EPI_ERR_CUDA;
        }
        it = h->graphs.emplace(key, std::move(hg)).first;
    }
    *out = it->second.exec;
    *events = &it->second.events;
    return EPI_OK;
}

static int check_error_flag(epi_engine* h);
static int report_error_flag(epi_engine* h, int e);

// Replicate r's state in the buffers of parity par, and its other bit plane zero, as the hours
// want it (a chain that starts out of step: a restore, hours run out of order).
static int move_to_buffer(epi_engine* h, uint32_t r, uint32_t par) {
    Replica& rep = h->reps[r];
    if (rep.par == par) return EPI_OK;
    const size_t off = rep.hp.agent_off, w0 = rep.hp.occ_off,
                 w1 = r + 1 < h->R() ? (size_t)h->reps[r + 1].hp.occ_off : h->occ_words;
    CK(cudaMemcpyAsync(pos_buf(h, par) + off, pos_buf(h, rep.par) + off, (size_t)rep.n * sizeof(uint32_t),
                       cudaMemcpyDeviceToDevice, h->stream));
    CK(cudaMemcpyAsync(occ_buf(h, par) + w0, occ_buf(h, rep.par) + w0, (w1 - w0) * sizeof(uint32_t),
                       cudaMemcpyDeviceToDevice, h->stream));
    CK(cudaMemsetAsync(occ_buf(h, rep.par) + w0, 0, (w1 - w0) * sizeof(uint32_t), h->stream));
    rep.par = par;
    return EPI_OK;
}

// Longest piece (one captured graph): two days.  Back-to-back pieces cost nothing measurable
// on the device, while every new engine captures its pieces once: two-day pieces made a
// fresh engine's 1M-agent 4,800-hour run 1.5 % faster than eight-day ones, at equal speed once warm.
constexpr uint32_t kPieceHours = 24u * 2u;

// The chain's hours as captured pieces, launched back to back; the counts rows land in h_counts.
static int run_pieces(epi_engine* h, uint32_t first_hour, uint32_t nh) {
    int rc = EPI_OK;
    const size_t row_words = (size_t)h->R() * 8;
    CK(cudaMemsetAsync(h->d_counts, 0, (size_t)nh * row_words * sizeof(uint32_t), h->stream));
    if (h->stream_file) CK(cudaMemsetAsync(h->d_exc_n, 0, (size_t)nh * sizeof(uint32_t), h->stream));
    h->h_seg->hour_base = first_hour;
    h->h_seg->first = first_hour;
    CK(cudaMemcpyAsync(h->d_seg, h->h_seg, sizeof(SegDev), cudaMemcpyHostToDevice, h->stream));
    // pieces: at most kPieceHours, ending after an hour of day 0 unless they end the chain, so
    // that a chain of whole days replays one graph; the stream's chunks stay whole (their
    // code buffers are indexed by the hour)
    for (uint32_t k0 = 0; k0 < nh;) {
        uint32_t len = nh - k0;
        if (!h->stream_file && len > kPieceHours) {
            const uint32_t head = (24u - (first_hour + k0) % 24u) % 24u + 1u;  // through the next hour of day 0
            len = head + (kPieceHours - std::min(head, kPieceHours)) / 24u * 24u;
        }
        cudaGraphExec_t exec;
        std::vector<TimedLaunch>* events;
        rc = piece_graph(h, first_hour + k0, len, &exec, &events);
        if (rc) return rc;
        CK(cudaGraphLaunch(exec, h->stream));
        h->kernels_launched += piece_launches(h, first_hour + k0, len);
        if (h->profiling) {  // the piece's event nodes hold this launch's times until its next launch
            h->pending.insert(h->pending.end(), events->begin(), events->end());
            CK(cudaStreamSynchronize(h->stream));
            rc = harvest_events(h);
            if (rc) return rc;
        }
        k0 += len;
    }
    CK(cudaMemcpyAsync(h->h_counts, h->d_counts, (size_t)nh * row_words * sizeof(uint32_t), cudaMemcpyDeviceToHost,
                       h->stream));
    CK(cudaStreamSynchronize(h->stream));
    return check_error_flag(h);
}

// The longest call that one launch runs.  A cluster's world: any.  A grid has a block on every SM,
// and the grids of engines in other threads run beside it only while all their threads fit
// (64 registers each: 1,024 threads an SM).  Two weeks of hours in one call, ms, one / four
// engines, one GB300: 30,000 agents (224 threads) 1.63 / 2.30, captured launches 1.76 / 2.20;
// 98,000 (672) 2.02 / 7.68, launches 1.91 / 2.89; so any call while four grids fit.  Above that a
// short call is still mostly launch and wait, which the grid has one of: 96 hours in calls of 1 /
// 3 / 6 hours, ms, grid : launches, 77,000 agents, one engine 2.12 : 3.89, 1.11 : 1.65, 0.86 : 1.10,
// four 3.97 : 5.16, 1.90 : 2.29, 1.60 : 1.55, eight 8.56 : 9.07, 3.59 : 3.61, 3.15 : 2.54; 98,000 agents, one
// 2.22 : 3.89, 1.17 : 1.69, 0.92 : 1.15, four 3.75 : 5.17, 2.80 : 2.34, 2.47 : 1.61.  So 3 hours while two grids
// fit and 1 hour beyond: no number of engines up to eight is slower than by launches.
constexpr uint32_t kSharedThreads = 256, kShortHours = 3;
static uint32_t longest_together(const epi_engine* h) {
    if (h->together != Together::kGrid) return h->together == Together::kCluster ? 0xFFFFFFFFu : 0u;
    const uint32_t threads = threads_of(h->reps[0].n, h->sms);
    return threads <= kSharedThreads ? 0xFFFFFFFFu : threads <= 2u * kSharedThreads ? kShortHours : 1u;
}

// The chain's hours of a small world in one launch (k_small), which writes the counts rows to
// pinned memory itself: one launch and one wait per call, where a captured piece takes a copy
// of the hour base, the graph, and two copies back with a wait each.
static int run_together(epi_engine* h, uint32_t first_hour, uint32_t nh) {
    const Replica& rep = h->reps[0];
    SmallArgs a;
    a.pos = pos_buf(h, rep.par);
    for (uint32_t k = 0; k < 2; ++k) {
        a.pos_buf[k] = pos_buf(h, k);
        a.occ_buf[k] = occ_buf(h, k);
    }
    a.st = h->d_st;
    a.home = h->d_home;
    a.work = h->d_work;
    a.wsa = h->d_wsa;
    a.cls = h->d_cls;
    a.danger = h->d_danger;
    a.claim = h->d_claim;
    a.claim_cells = (uint32_t)h->claim_cells;
    a.occ_words = (uint32_t)h->occ_words;
    a.first = first_hour;
    a.hours = nh;
    a.run_loop = h->stop_rule ? 1u : 0u;
    a.ivn = h->d_ivn;
    a.sums = h->d_sums;
    a.rows = h->h_counts;
    a.err = h->d_err;
    a.polls = h->wait_polls;
    a.err_out = h->h_err;
    const bool grid = h->together == Together::kGrid;
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(threads_of(rep.n, grid ? h->sms : kSmallCluster));
    cfg.gridDim = dim3(grid ? (rep.n + cfg.blockDim.x - 1) / cfg.blockDim.x : kSmallCluster);
    cfg.stream = h->stream;
    cudaLaunchAttribute at[1];
    if (grid) {
        at[0].id = cudaLaunchAttributeCooperative;
        at[0].val.cooperative = 1;
        CK(cudaMemsetAsync(h->d_sums, 0, kGridWords * sizeof(uint32_t), h->stream));
    } else {
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = kSmallCluster;
        at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    }
    cfg.attrs = at;
    cfg.numAttrs = 1;
    h->h_err[0] = h->h_err[1] = 0;
    CK(cudaLaunchKernelEx(&cfg, grid ? k_small<true> : k_small<false>, (const DevParams*)h->d_params, a));
    h->kernels_launched += 1;
    CK(cudaStreamSynchronize(h->stream));
    return report_error_flag(h, h->h_err[0] | h->h_err[1]);
}

// Simulate hours first_hour .. first_hour + nh - 1 for every active replicate as one chain:
// pieces of whole days, launched back to back with one host synchronisation at the end
// (after each piece when profiling, whose events are read per launch).  The
// counts of hour k of replicate r land in h_counts[(k * R + r) * 8 ..]; in the run loop,
// h->halt_row is the chain offset of a row the guard marked, or -1.
static int run_hours_chunk(epi_engine* h, uint32_t first_hour, uint32_t nh) {
    h->halt_row = -1;
    if (nh == 0) return EPI_OK;
    if ((uint64_t)first_hour + nh > 0xFFFFFFFFull) { h->err = "hour out of range"; return EPI_ERR_ARG; }
    int rc = ensure_counts(h, nh);
    if (rc) return rc;
    const bool small = nh <= h->together_most && !h->profiling && !h->stream_file;
    // claims left by an earlier hour of another window, or by a later hour, must go first
    if (h->last_claim_hour >= 0 &&
        ((int64_t)first_hour <= h->last_claim_hour || first_hour / kClaimWindow != (uint64_t)h->last_claim_hour / kClaimWindow))
        CK(cudaMemsetAsync(h->d_claim, 0xFF, h->claim_cells * sizeof(uint32_t), h->stream));
    h->last_claim_hour = INT64_MAX;  // until the hours have run
    // the chain reads the state after first_hour - 1 from its parity's buffers
    const uint32_t need = hour_parity((first_hour + 23u) % 24u);
    std::vector<uint8_t> ran(h->R(), 0);  // a world whose run has ended runs no hour kernel
    for (uint32_t r = 0; r < h->R(); ++r) {
        if (!h->reps[r].active) continue;
        ran[r] = 1;
        rc = move_to_buffer(h, r, need);
        if (rc) return rc;
    }
    const size_t row_words = (size_t)h->R() * 8;
    if (small) {
        rc = run_together(h, first_hour, nh);
        if (rc) return rc;
    } else {
        rc = run_pieces(h, first_hour, nh);
        if (rc) return rc;
    }
    for (uint32_t k = 1; k < nh; ++k)
        if (sleep_hour_skipped(first_hour, k))
            std::memcpy(h->h_counts + (size_t)k * row_words, h->h_counts + (size_t)(k - 1) * row_words,
                        row_words * sizeof(uint32_t));
    std::vector<uint8_t> ended(h->R(), 0);  // stop rule met at an earlier hour of this chain
    std::vector<uint32_t> last(h->R(), nh - 1);  // the last row whose hour ran
    for (uint32_t k = 0; k < nh && h->halt_row < 0; ++k) {
        for (uint32_t r = 0; r < h->R(); ++r) {
            if (!h->reps[r].active || ended[r]) continue;
            const uint32_t* c = h->h_counts + ((size_t)k * h->R() + r) * 8;
            if (h->stop_rule && c[1] == 0 && c[2] == 0 && c[3] == 0) {
                ended[r] = 1;
                last[r] = k;
            }
            const uint64_t total = (uint64_t)c[0] + c[1] + c[2] + c[3] + c[4] + c[5];
            if (total != h->reps[r].n) {  // assert_eq!(csv_record.total(), current_population), allocation_map.rs:128
                h->err = "replicate " + std::to_string(r) + ": counts total " + std::to_string(total) + " != population " +
                         std::to_string(h->reps[r].n);
                return EPI_ERR_INVARIANT;
            }
        }
        if (h->stop_rule && h->h_counts[(size_t)k * row_words + 6] != 0u) h->halt_row = (int)k;  // later rows did not run
    }
    for (uint32_t r = 0; r < h->R(); ++r) {  // the buffers of the last hour whose kernels ran
        if (!ran[r]) continue;
        if (h->halt_row >= 0) last[r] = std::min(last[r], (uint32_t)h->halt_row);
        h->reps[r].par = hour_parity((first_hour + last[r]) % 24u);
    }
    // The hour kernels open every claim window of the chain, whether or not a world still runs;
    // k_small none that its world did not get to.
    if (!small) h->last_claim_hour = (int64_t)first_hour + nh - 1;
    else if (ran[0]) h->last_claim_hour = (int64_t)first_hour + last[0];
    return EPI_OK;
}

static int check_error_flag(epi_engine* h) {
    int e = 0;
    CK(cudaMemcpyAsync(&e, h->d_err, sizeof(int), cudaMemcpyDeviceToHost, h->stream));
    CK(cudaStreamSynchronize(h->stream));
    return report_error_flag(h, e);
}

static int report_error_flag(epi_engine* h, int e) {
    if (e & kErrWait) {
        h->err = "a block gave up waiting for the others of its launch; the world is somewhere within an hour";
        return EPI_ERR_TIMEOUT;
    }
    if (e) {
        h->err = "device invariant violated (flag " + std::to_string(e) + "): a rule addressed a cell outside the plane";
        return EPI_ERR_INVARIANT;
    }
    return EPI_OK;
}

// ------------------------------------------------------------------ citizen-state stream
constexpr uint32_t kStreamChunk = 24;  // hours per stream buffer fill

// Append hours first_hour .. first_hour + m - 1 of the stream buffers to the file: per hour
// {hour, agents, exceptions} (u32 each), the agents' code bytes, then the exceptions
// {agent, x | y << 16} in agent order.
static int stream_write(epi_engine* h, uint32_t first_hour, uint32_t m) {
    const uint32_t n = h->reps[0].n;
    CK(cudaMemcpyAsync(h->h_exc_n, h->d_exc_n, m * sizeof(uint32_t), cudaMemcpyDeviceToHost, h->stream));
    for (uint32_t k = 0; k < m; ++k)
        CK(cudaMemcpyAsync(h->h_codes + (size_t)k * h->slots, h->d_codes + (size_t)k * h->slots, n,
                           cudaMemcpyDeviceToHost, h->stream));
    CK(cudaStreamSynchronize(h->stream));
    for (uint32_t k = 0; k < m; ++k) {
        const uint32_t ne = std::min(h->h_exc_n[k], n);
        if (ne) CK(cudaMemcpy(h->h_exc, h->d_exc + (size_t)k * h->slots, ne * sizeof(uint2), cudaMemcpyDeviceToHost));
        std::sort(h->h_exc, h->h_exc + ne, [](const uint2& a, const uint2& b) { return a.x < b.x; });
        const uint32_t head[3] = {first_hour + k, n, ne};
        if (std::fwrite(head, sizeof head, 1, h->stream_file) != 1 ||
            std::fwrite(h->h_codes + (size_t)k * h->slots, 1, n, h->stream_file) != n ||
            (ne && std::fwrite(h->h_exc, sizeof(uint2), ne, h->stream_file) != ne)) {
            h->err = "citizen-state stream: write failed";
            return EPI_ERR_IO;
        }
    }
    return EPI_OK;
}

// Hours first_hour .. first_hour + nh - 1 (see run_hours_chunk); with the stream open they run
// in chunks of at most kStreamChunk hours, each written out before the next.
static int run_hours(epi_engine* h, uint32_t first_hour, uint32_t nh) {
    if (h->stop_rule) {  // the guard's new-infections figures as the host has them (the chunks carry them on)
        CK(cudaStreamSynchronize(h->stream));  // the pinned staging may still feed an earlier copy
        for (uint32_t r = 0; r < h->R(); ++r) h->h_ivn[r] = h->reps[r].iv.new_infections_in_a_day;
        CK(cudaMemcpyAsync(h->d_ivn, h->h_ivn, h->R() * sizeof(uint32_t), cudaMemcpyHostToDevice, h->stream));
    }
    if (!h->stream_file) return run_hours_chunk(h, first_hour, nh);
    int rc = ensure_counts(h, std::max(nh, kStreamChunk));
    if (rc) return rc;
    const size_t row = (size_t)h->R() * 8;
    std::vector<uint32_t> all((size_t)nh * row, 0u);
    int halt = -1;
    for (uint32_t k0 = 0; k0 < nh; k0 += kStreamChunk) {
        const uint32_t m = std::min(kStreamChunk, nh - k0);
        rc = run_hours_chunk(h, first_hour + k0, m);
        if (rc) return rc;
        // in the run loop the record ends with the hour the stop rule fires (the reference
        // publishes no later hour), or with a row the guard marked (the hours after it did
        // not run; the run loop runs them again)
        // (each chunk is a chain of its own, so the host, not the device, ends the run here)
        uint32_t keep = m;
        bool over = false;
        if (h->stop_rule)
            for (uint32_t k = 0; k < m; ++k) {
                const uint32_t* c = h->h_counts + (size_t)k * row;
                if ((c[1] | c[2] | c[3]) == 0u) { keep = k + 1; over = true; break; }
            }
        if (h->halt_row >= 0 && (uint32_t)h->halt_row < keep) {
            keep = (uint32_t)h->halt_row + 1;
            halt = (int)(k0 + (uint32_t)h->halt_row);
            over = true;
        }
        rc = stream_write(h, first_hour + k0, keep);
        if (rc) return rc;
        std::memcpy(all.data() + (size_t)k0 * row, h->h_counts, (size_t)keep * row * sizeof(uint32_t));
        if (over) break;
    }
    std::memcpy(h->h_counts, all.data(), all.size() * sizeof(uint32_t));
    h->halt_row = halt;
    return EPI_OK;
}

static void stream_free(epi_engine* h) {
    if (h->stream_file) std::fclose(h->stream_file);
    h->stream_file = nullptr;
    cudaFree(h->d_prev); cudaFree(h->d_codes); cudaFree(h->d_exc); cudaFree(h->d_exc_n);
    if (h->h_codes) cudaFreeHost(h->h_codes);
    if (h->h_exc) cudaFreeHost(h->h_exc);
    if (h->h_exc_n) cudaFreeHost(h->h_exc_n);
    h->d_prev = nullptr; h->d_codes = nullptr; h->d_exc = nullptr; h->d_exc_n = nullptr;
    h->h_codes = nullptr; h->h_exc = nullptr; h->h_exc_n = nullptr;
}

static epi_counts counts_of(const epi_engine* h, uint32_t k, uint32_t r, uint32_t hour) {
    const uint32_t* c = h->h_counts + ((size_t)k * h->R() + r) * 8;
    epi_counts o;
    o.hour = hour;
    o.susceptible = c[0];
    o.exposed = c[1];
    o.infected = c[2];
    o.hospitalized = c[3];
    o.recovered = c[4];
    o.deceased = c[5];
    return o;
}

// ------------------------------------------------------------------ interventions
static int bulk_done(epi_engine* h) {
    CK(cudaStreamSynchronize(h->stream));
    h->kernels_launched += 1;
    return harvest_events(h);
}

static int blocks_for(uint32_t n) { return (int)std::max<uint32_t>(1u, std::min<uint32_t>((n + kThreads - 1) / kThreads, 4096u)); }

static int lock_city(epi_engine* h, uint32_t r, int on) {
    const Replica& rep = h->reps[r];
    LAUNCH(kKLock, (k_lock<<<blocks_for(rep.n), kThreads, 0, h->stream>>>(h->d_st, rep.hp.agent_off, rep.n, on)));
    return bulk_done(h);
}

static int vaccinate(epi_engine* h, uint32_t r, uint32_t hour, double percent) {
    const Replica& rep = h->reps[r];
    const uint64_t thr = bernoulli_threshold(percent);
    LAUNCH(kKVaccinate, (k_vaccinate<<<blocks_for(rep.n), kThreads, 0, h->stream>>>(h->d_st, rep.hp.agent_off, rep.n,
                                                                                    rep.hp.key0, rep.hp.key1, hour, thr)));
    return bulk_done(h);
}

static void grow_hospital(epi_engine* h, uint32_t r) {
    Replica& rep = h->reps[r];
    const epi_area grown = grown_hospital(rep.geo0);
    rep.geo.hospital = grown;
    rep.hp.hosp_code = rect_eq(to_rect(grown), rep.hp.area[kHosp0]) ? kHosp0 : kHosp1;
}

// process_interventions of one replicate; returns EPI_IV_* bits in *applied.  Parameter
// changes (the hospital, and the device guard's armed triggers after any action) are left
// for the caller to push.
static int process_interventions(epi_engine* h, uint32_t r, const epi_counts& c, uint32_t* applied, bool* params_dirty) {
    Replica& rep = h->reps[r];
    InterventionActions a = decide_interventions(rep.p, rep.iv, c, rep.geo.hospital);
    int rc = EPI_OK;
    if (a.vaccinate && (rc = vaccinate(h, r, c.hour, a.vaccinate_percent))) return rc;
    if (a.lock && (rc = lock_city(h, r, 1))) return rc;
    if (a.unlock && (rc = lock_city(h, r, 0))) return rc;
    if (a.grow_hospital) grow_hospital(h, r);
    if (a.applied) *params_dirty = true;
    if (applied) *applied = a.applied;
    return EPI_OK;
}

// run_single_engine for every replicate in lockstep: segments end at any replicate's
// intervention point or final hour; after each segment every active replicate takes its
// rows, its interventions and its stop rule (epidemiology_simulation.rs:223-269, 564-575).
static int set_all_active(epi_engine* h) {
    for (auto& rep : h->reps) {
        rep.active = true;
        rep.hp.active = 1;
    }
    return push_params(h);
}

static int run_loop_body(epi_engine* h, uint32_t until);

// The run loop through hour `until` (all of it for 0xFFFFFFFF), starting at hour 1 or where a
// paused run stopped.  Replicates drop out of the lockstep loop as their runs end; once the
// run is over all of them are active again, so that direct hour calls keep working on every
// world (a paused run keeps its flags for the continuation).
static int run_loop(epi_engine* h, uint32_t until = 0xFFFFFFFFu) {
    h->stop_rule = true;
    int rc = run_loop_body(h, until);
    h->stop_rule = false;
    if (rc) h->loop_hour = 0;  // a failed run cannot be continued
    if (h->loop_hour != 0 && !rc) return EPI_OK;
    int rc2 = set_all_active(h);
    return rc ? rc : rc2;
}

// Longest chain of the run loop: a chain that the guard halts early has launched its later
// pieces for nothing (their kernels see the mark and return at once), so the cap bounds that
// waste while the host synchronises once per chain instead of once per day.
constexpr uint32_t kChainHours = 24u * 8u;

static int run_loop_body(epi_engine* h, uint32_t until) {
    uint32_t last = 0;  // last simulated hour over all replicates
    if (h->loop_hour == 0) {  // a fresh run
        for (auto& rep : h->reps) {
            rep.rows.clear();
            rep.active = rep.p.hours >= 2;
            rep.hp.active = rep.active ? 1u : 0u;
        }
        h->loop_hour = 1;
    }
    for (const auto& rep : h->reps)
        if (rep.p.hours >= 2) last = std::max(last, rep.p.hours - 1);
    uint32_t hour = h->loop_hour;
    bool dirty = true;
    while (hour <= last && hour <= until) {
        bool any = false;
        for (auto& rep : h->reps) any |= rep.active;
        if (!any) break;
        if (dirty) {
            int rc = push_params(h);
            if (rc) return rc;
            dirty = false;
        }
        // the chain ends at the first hour where the host must act whatever the counts are: a
        // replicate's final hour or fixed intervention; data-dependent triggers halt it on
        // the device at the day boundary where they fire
        uint64_t end = std::min<uint64_t>(std::min(last, until), (uint64_t)hour + kChainHours - 1);
        for (const auto& rep : h->reps) {
            if (!rep.active) continue;
            end = std::min<uint64_t>(end, rep.p.hours - 1);
            end = std::min<uint64_t>(end, next_fixed_event(rep.p, rep.iv, hour));
        }
        const uint32_t nh = (uint32_t)end - hour + 1;
        int rc = run_hours(h, hour, nh);
        if (rc) return rc;
        uint32_t next = (uint32_t)end + 1;
        for (uint32_t k = 0; k < nh; ++k) {
            const uint32_t hr = hour + k;
            bool acted = false;
            for (uint32_t r = 0; r < h->R(); ++r) {
                Replica& rep = h->reps[r];
                if (!rep.active) continue;
                const epi_counts c = counts_of(h, k, r, hr);
                rep.rows.push_back(c);
                if (is_event_hour(rep.p, hr)) {
                    uint32_t applied = 0;
                    rc = process_interventions(h, r, c, &applied, &dirty);
                    if (rc) return rc;
                    acted |= applied != 0u;
                }
                const bool stop = c.exposed == 0 && c.infected == 0 && c.hospitalized == 0;
                if (stop || hr + 1 >= rep.p.hours) {
                    rep.active = false;
                    rep.hp.active = 0;
                    dirty = true;
                }
            }
            const bool halted = h->halt_row == (int)k;
            if (acted && !halted && k + 1 < nh) {
                // an intervention the device guard did not see: the later hours ran without it
                h->err = "run loop: an intervention fired at hour " + std::to_string(hr) +
                         " inside a chain without the device guard's mark";
                return EPI_ERR_INVARIANT;
            }
            if (acted || halted) {
                next = hr + 1;
                break;
            }
        }
        hour = next;
    }
    bool any = false;
    for (const auto& rep : h->reps) any |= rep.active;
    h->loop_hour = (any && hour <= last) ? hour : 0u;
    if (dirty) return push_params(h);
    return EPI_OK;
}

// ------------------------------------------------------------------ create / destroy
static void free_device(epi_engine* h) {
    destroy_graphs(h);
    stream_free(h);
    cudaFree(h->d_params); cudaFree(h->d_chunk_rep); cudaFree(h->d_pos); cudaFree(h->d_home); cudaFree(h->d_work);
    cudaFree(h->d_wsa); cudaFree(h->d_st); cudaFree(h->d_occ); cudaFree(h->d_cls); cudaFree(h->d_danger); cudaFree(h->d_claim);
    cudaFree(h->d_displaced); cudaFree(h->d_acts); cudaFree(h->d_list_n); cudaFree(h->d_piece_rep); cudaFree(h->d_par);
    cudaFree(h->d_sums);
    cudaFree(h->d_counts); cudaFree(h->d_seg); cudaFree(h->d_ivn); cudaFree(h->d_err); cudaFree(h->d_scratch);
    cudaFree(h->s_pos); cudaFree(h->s_wsa); cudaFree(h->s_st); cudaFree(h->s_occ); cudaFree(h->s_cls); cudaFree(h->s_danger);
    if (h->h_counts) cudaFreeHost(h->h_counts);
    if (h->h_seg) cudaFreeHost(h->h_seg);
    for (auto& pe : h->pending)
        if (pe.pooled) { cudaEventDestroy(pe.begin); cudaEventDestroy(pe.end); }
    for (auto e : h->event_pool) cudaEventDestroy(e);
    if (h->own_stream && h->stream) cudaStreamDestroy(h->stream);
}

static size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

static int finish_upload(epi_engine* h);

// World build on the device (world.cuh) for every replicate, from the host plan.
static int build_on_device(epi_engine* h) {
    const uint32_t R = h->R(), n_chunks = h->slots / kChunk;
    std::vector<WorldDev> W(R);
    std::vector<uint4> infections;
    std::vector<WorldPlan> plans(R);
    std::vector<int> status(R, EPI_OK);
    std::vector<std::string> errs(R);
    const unsigned workers = std::max(1u, std::min<unsigned>(R, std::thread::hardware_concurrency()));
    std::vector<std::thread> pool;
    for (unsigned w = 0; w < workers; ++w)
        pool.emplace_back([&, w] {
            for (uint32_t r = w; r < R; r += workers) {
                const bool csv = h->reps[r].p.population_source == 1;
                if (csv && (R != 1 || !h->init_flags)) {
                    status[r] = EPI_ERR_ARG;
                    errs[r] = "a Csv population comes with its rows (epi_engine_create_population, single engines)";
                    continue;
                }
                status[r] = world_plan(h->reps[r].p, plans[r], errs[r], csv ? h->init_flags : nullptr);
            }
        });
    for (auto& t : pool) t.join();
    for (uint32_t r = 0; r < R; ++r) {
        if (status[r]) {
            h->err = (R > 1 ? "replicate " + std::to_string(r) + ": " : std::string()) + errs[r];
            return status[r];
        }
        const WorldPlan& pl = plans[r];
        const Replica& rep = h->reps[r];
        WorldDev& d = W[r];
        d.n = pl.n;
        d.agent_off = rep.hp.agent_off;
        d.first_chunk = rep.hp.agent_off / kChunk;
        d.houses = pl.houses;
        d.houses_x = pl.geo.houses_x;
        d.offices = pl.offices;
        d.offices_x = pl.geo.offices_x;
        d.hx0 = pl.geo.housing.x0; d.hy0 = pl.geo.housing.y0;
        d.ox0 = pl.geo.work.x0; d.oy0 = pl.geo.work.y0;
        d.key0 = pl.key0; d.key1 = pl.key1;
        d.transport_points = (uint32_t)std::min<uint64_t>(pl.transport_points, 0xFFFFFFFFull);
        d.csv = pl.flags ? 1u : 0u;
        d.thr_work = pl.thr_work; d.thr_pt = pl.thr_pt; d.thr_staff = pl.thr_staff; d.thr_ess = pl.thr_ess;
        for (const auto& f : pl.infections) infections.push_back(make_uint4(rep.hp.agent_off + f.agent, f.state, f.day, 0u));
    }
    WorldDev* d_w = nullptr;
    uint4* d_inf = nullptr;
    uint8_t* d_flags = nullptr;
    CK(cudaMalloc(&d_w, R * sizeof(WorldDev)));
    if (h->init_flags) {  // single Csv world: slot = agent
        CK(cudaMalloc(&d_flags, h->slots));
        CK(cudaMemsetAsync(d_flags, 0, h->slots, h->stream));
        CK(cudaMemcpyAsync(d_flags, h->init_flags, h->reps[0].n, cudaMemcpyHostToDevice, h->stream));
    }
    if (!infections.empty()) CK(cudaMalloc(&d_inf, infections.size() * sizeof(uint4)));
    int rc = EPI_OK;
    cudaError_t e = cudaMemcpyAsync(d_w, W.data(), R * sizeof(WorldDev), cudaMemcpyHostToDevice, h->stream);
    if (e == cudaSuccess && d_inf)
        e = cudaMemcpyAsync(d_inf, infections.data(), infections.size() * sizeof(uint4), cudaMemcpyHostToDevice, h->stream);
    if (e == cudaSuccess) {
        // scratch: the hour lists hold the eligibility flags and the per-chunk counts
        uint32_t *d_elig = h->d_displaced, *d_chunk_elig = reinterpret_cast<uint32_t*>(h->d_acts);
        const int blocks = (int)std::min<uint64_t>(n_chunks, (uint64_t)h->resident_blocks * 2);
        k_world_citizens<<<blocks, kThreads, 0, h->stream>>>(d_w, h->d_chunk_rep, n_chunks, h->d_pos, h->d_st, h->d_home,
                                                             h->d_work, h->d_wsa, d_elig, d_chunk_elig, d_flags);
        k_world_scan<<<1, 1024, 0, h->stream>>>(d_chunk_elig, n_chunks);
        k_world_pt<<<blocks, kThreads, 0, h->stream>>>(d_w, h->d_chunk_rep, n_chunks, d_elig, d_chunk_elig, h->d_st);
        if (d_inf)
            k_world_infect<<<(int)std::min<size_t>((infections.size() + kThreads - 1) / kThreads, 1024), kThreads, 0,
                             h->stream>>>(d_inf, (uint32_t)infections.size(), h->d_st);
        e = cudaGetLastError();
        if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
        h->kernels_launched += d_inf ? 4 : 3;
    }
    if (e != cudaSuccess) {
        h->err = std::string("device world build: ") + cudaGetErrorString(e);
        rc = EPI_ERR_CUDA;
    }
    cudaFree(d_w);
    cudaFree(d_inf);
    cudaFree(d_flags);
    return rc;
}

// Lay out and upload R worlds given as per-replicate record arrays (nullptr: build them on
// the device).
static int engine_init(epi_engine* h, const epi_params* params, const epi_agent_record* const* recs, uint32_t R) {
    if (R == 0) { h->err = "no replicates"; return EPI_ERR_ARG; }
    h->reps.resize(R);
    uint64_t slots = 0, plane = 0, claim = 0, occ = 0;
    for (uint32_t r = 0; r < R; ++r) {
        Replica& rep = h->reps[r];
        rep.p = params[r];
        const std::string bad = validate_params(rep.p);
        if (!bad.empty()) { h->err = "replicate " + std::to_string(r) + ": " + bad; return EPI_ERR_CONFIG; }
        rep.n = rep.p.number_of_agents;
        rep.geo0 = define_geography(rep.p.grid_size);
        resize_hospital(rep.geo0, (int32_t)rep.n, 0.002, rep.p.hospital_beds_percentage);
        rep.geo = rep.geo0;
        rep.hp = make_dev_params(rep.p, rep.geo0, rep.n);
        rep.hp.agent_off = (uint32_t)slots;
        rep.hp.plane_off = plane;
        rep.hp.claim_off = claim;
        rep.hp.occ_off = occ;
        const uint64_t side = (uint64_t)rep.p.grid_size + 1;
        slots += align_up(rep.n, kChunk);
        plane += align_up((side + 2) * (side + 2) + 16, 256);
        claim += side * side;
        occ += align_up((side + 2) * rep.hp.PW, kPieceWords);
        if (slots >= 0xFFFFFFFFull - kChunk) { h->err = "too many agents for one engine"; return EPI_ERR_CAPACITY; }
    }
    h->slots = (uint32_t)slots;
    h->plane_bytes = plane;
    h->claim_cells = claim;
    h->occ_words = occ;
    int dev = 0, sms = 0, per_sm = 0;
    CK(cudaGetDevice(&dev));
    CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, (const void*)decide_kernel(9u, R > 1), kThreads, 0));
    per_sm = std::max(per_sm, 1);
    const uint64_t n_chunks = slots / kChunk;
    h->resident_blocks = sms * per_sm;
    h->sms = (uint32_t)sms;
    // A world takes the resident grid (4M agents, 15,625 chunks: 68.8 ms a run; a block per 4 chunks
    // 88, per chunk 111).  A large ensemble takes more blocks, whose uneven chunks then spread
    // over the SMs as they come (256 replicates, 130,000 chunks: resident 122 ms, a block per 24 /
    // 18 / 14 / 10 chunks 113.7 / 112.2 / 114 / 113; resident / per 18, ms: 25,700 chunks 10.6 / 11.1, 38,600
    // 14.8 / 14.8, 52,500 11.55 / 11.33, 78,600 17.3 / 16.6, 120,000 22.2 / 21.1, 183,000 35.3 / 31.4).
    h->grid_blocks = (int)std::min<uint64_t>(
        n_chunks, std::max<uint64_t>(h->resident_blocks, R > 1 ? n_chunks / kEnsembleBlockChunks : 0u));
    CK(cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking));
    h->own_stream = true;
    CK(cudaMalloc(&h->d_params, R * sizeof(DevParams)));
    if (R > 1) {
        std::vector<uint32_t> chunk_rep(n_chunks);
        for (uint32_t r = 0; r < R; ++r) {
            const uint64_t c0 = h->reps[r].hp.agent_off / kChunk, c1 = c0 + align_up(h->reps[r].n, kChunk) / kChunk;
            for (uint64_t c = c0; c < c1; ++c) chunk_rep[c] = r;
        }
        CK(cudaMalloc(&h->d_chunk_rep, n_chunks * sizeof(uint32_t)));
        CK(cudaMemcpyAsync(h->d_chunk_rep, chunk_rep.data(), n_chunks * sizeof(uint32_t), cudaMemcpyHostToDevice, h->stream));
        std::vector<uint32_t> piece_rep(occ / kPieceWords);
        for (uint32_t r = 0; r < R; ++r) {
            const uint64_t q1 = (r + 1 < R ? h->reps[r + 1].hp.occ_off : occ) / kPieceWords;
            for (uint64_t q = h->reps[r].hp.occ_off / kPieceWords; q < q1; ++q) piece_rep[q] = r;
        }
        CK(cudaMalloc(&h->d_piece_rep, piece_rep.size() * sizeof(uint32_t)));
        CK(cudaMemcpyAsync(h->d_piece_rep, piece_rep.data(), piece_rep.size() * sizeof(uint32_t), cudaMemcpyHostToDevice,
                           h->stream));
        CK(cudaStreamSynchronize(h->stream));
    }
    CK(cudaMalloc(&h->d_pos, 2u * slots * sizeof(uint32_t)));
    CK(cudaMalloc(&h->d_home, slots * sizeof(uint32_t)));
    CK(cudaMalloc(&h->d_work, slots * sizeof(uint32_t)));
    CK(cudaMalloc(&h->d_wsa, slots * sizeof(uint32_t)));
    CK(cudaMalloc(&h->d_st, slots * sizeof(uint2)));
    CK(cudaMalloc(&h->d_occ, 2u * h->occ_words * sizeof(uint32_t)));
    CK(cudaMalloc(&h->d_cls, h->plane_bytes));
    CK(cudaMalloc(&h->d_danger, h->plane_bytes));
    CK(cudaMalloc(&h->d_displaced, slots * sizeof(uint32_t)));
    CK(cudaMalloc(&h->d_acts, slots * sizeof(uint2)));
    CK(cudaMalloc(&h->d_list_n, n_chunks * (kThreads / 32) * sizeof(uint2)));  // grids have at most n_chunks blocks
    CK(cudaMalloc(&h->d_par, R * sizeof(uint32_t)));
    // (room for one record, which snapshots lay out here: a grid of 2 has 9 cells)
    h->claim_bytes = std::max(h->claim_cells * sizeof(uint32_t), sizeof(epi_agent_record));
    CK(cudaMalloc(&h->d_claim, h->claim_bytes));
    CK(cudaMalloc(&h->d_seg, sizeof(SegDev)));
    CK(cudaMalloc(&h->d_ivn, R * sizeof(uint32_t)));
    CK(cudaMemset(h->d_ivn, 0, R * sizeof(uint32_t)));
    CK(cudaMalloc(&h->d_err, sizeof(int)));
    CK(cudaMalloc(&h->d_scratch, 6 * sizeof(unsigned long long)));
    CK(cudaMallocHost(&h->h_seg, sizeof(SegDev) + 2 * sizeof(int) + R * sizeof(uint32_t)));  // with h_err and h_ivn
    h->h_err = reinterpret_cast<int*>(h->h_seg + 1);
    h->h_ivn = reinterpret_cast<uint32_t*>(h->h_err + 2);
    if (R == 1) h->together = runs_together(h->reps[0].n, h->occ_words, h->sms);
    if (h->together == Together::kGrid) CK(cudaMalloc(&h->d_sums, kGridWords * sizeof(uint32_t)));
    h->together_most = longest_together(h);
    int rc = ensure_counts(h, 48);
    if (rc) return rc;
    if (!recs) {
        rc = build_on_device(h);
        if (rc) return rc;
        return finish_upload(h);
    }
    // The records go to the device as they are (replicate r's at slot agent_off(r)) and
    // k_pack_records checks and packs them there; the first bad one is reported.
    rc = push_params(h);
    if (rc) return rc;
    struct DeviceBuffer {
        void* p = nullptr;
        ~DeviceBuffer() { if (p) cudaFree(p); }
    } stage;
    CK(cudaMalloc(&stage.p, slots * sizeof(epi_agent_record)));
    epi_agent_record* d_recs = static_cast<epi_agent_record*>(stage.p);
    for (uint32_t r = 0; r < R; ++r)
        CK(cudaMemcpyAsync(d_recs + h->reps[r].hp.agent_off, recs[r], (size_t)h->reps[r].n * sizeof(epi_agent_record),
                           cudaMemcpyHostToDevice, h->stream));
    CK(cudaMemsetAsync(h->d_scratch, 0xFF, sizeof(unsigned long long), h->stream));
    k_pack_records<<<blocks_for(h->slots), kThreads, 0, h->stream>>>(h->d_params, h->d_chunk_rep, h->slots, d_recs,
                                                                     h->d_pos, h->d_st, h->d_home, h->d_work, h->d_wsa,
                                                                     h->d_scratch);
    CK(cudaGetLastError());
    unsigned long long bad = ~0ull;
    CK(cudaMemcpyAsync(&bad, h->d_scratch, sizeof bad, cudaMemcpyDeviceToHost, h->stream));
    CK(cudaStreamSynchronize(h->stream));
    if (bad != ~0ull) {  // the replicate holding the slot, and the record's index within it
        const uint64_t slot = bad >> 1;
        uint32_t r = 0;
        while (r + 1 < R && h->reps[r + 1].hp.agent_off <= slot) ++r;
        h->err = "replicate " + std::to_string(r) + ": agent record " + std::to_string(slot - h->reps[r].hp.agent_off) +
                 ((bad & 1u) ? ": current area is not one of its areas" : " out of range");
        return EPI_ERR_ARG;
    }
    return finish_upload(h);
}

// Everything after the agent arrays are on the device: scratch words, planes, parameters.
static int finish_upload(epi_engine* h) {
    CK(cudaMemsetAsync(h->d_occ, 0, 2u * h->occ_words * sizeof(uint32_t), h->stream));
    CK(cudaMemsetAsync(h->d_cls, 0, h->plane_bytes, h->stream));
    CK(cudaMemsetAsync(h->d_danger, 0, h->plane_bytes, h->stream));
    CK(cudaMemsetAsync(h->d_claim, 0xFF, h->claim_cells * sizeof(uint32_t), h->stream));
    for (auto& rep : h->reps) rep.par = 0;
    CK(cudaMemsetAsync(h->d_err, 0, sizeof(int), h->stream));
    int rc = push_params(h);
    if (rc) return rc;
    LAUNCH(kKBuildPlane, (k_build_plane<<<blocks_for(h->slots), kThreads, 0, h->stream>>>(
                              h->d_params, h->d_chunk_rep, h->slots, h->d_pos, h->d_st, h->d_occ, h->d_cls, h->d_danger,
                              h->d_err)));
    CK(cudaStreamSynchronize(h->stream));
    rc = harvest_events(h);
    if (rc) return rc;
    return check_error_flag(h);
}

// Replicate r's records.  They are laid out on the device in the claim plane (free between
// chains: the next chain resets it), as many at a time as it holds.
static int snapshot_replica(epi_engine* h, uint32_t r, epi_agent_record* out, size_t n) {
    const Replica& rep = h->reps[r];
    if (!out || n != rep.n) return EPI_ERR_ARG;
    const size_t room = h->claim_bytes / sizeof(epi_agent_record);
    h->last_claim_hour = INT64_MAX;
    touch_pages(out, n * sizeof(epi_agent_record));
    for (size_t first = 0; first < n; first += room) {
        const uint32_t count = (uint32_t)std::min(room, n - first);
        k_unpack_records<<<(count + kThreads - 1) / kThreads, kThreads, 0, h->stream>>>(
            h->d_params, r, rep.hp.agent_off, (uint32_t)first, count, pos_buf(h, rep.par), h->d_st, h->d_home, h->d_work,
            h->d_wsa, h->d_claim);
        CK(cudaGetLastError());  // (not counted: the counter is of the simulation's launches)
        CK(cudaMemcpyAsync(out + first, h->d_claim, count * sizeof(epi_agent_record), cudaMemcpyDeviceToHost, h->stream));
    }
    CK(cudaStreamSynchronize(h->stream));
    return EPI_OK;
}

static int check_all(epi_engine* h) {
    std::vector<uint32_t> par(h->R());
    for (uint32_t r = 0; r < h->R(); ++r) par[r] = h->reps[r].par;
    CK(cudaMemcpyAsync(h->d_par, par.data(), par.size() * sizeof(uint32_t), cudaMemcpyHostToDevice, h->stream));
    CK(cudaMemsetAsync(h->d_scratch, 0, 6 * sizeof(unsigned long long), h->stream));
    LAUNCH(kKCheck, (k_check_agents<<<blocks_for(h->slots), kThreads, 0, h->stream>>>(
                         h->d_params, h->d_chunk_rep, h->slots, h->d_pos, h->d_occ, h->occ_words, h->d_par, h->d_st,
                         h->d_cls, h->d_scratch)));
    LAUNCH(kKCheck, (k_check_planes<<<h->grid_blocks, kThreads, 0, h->stream>>>(
                         h->R(), h->d_params, h->d_occ, h->occ_words, h->d_par, h->plane_bytes, h->d_cls,
                         h->d_scratch + 2, h->d_scratch + 3, h->d_scratch + 4)));
    LAUNCH(kKCheck, (k_check_danger<<<dim3(64, std::min<uint32_t>(h->R(), 4096u)), kThreads, 0, h->stream>>>(
                         h->d_params, h->R(), h->d_cls, h->d_danger, h->d_scratch + 5)));
    unsigned long long v[6] = {0, 0, 0, 0, 0, 0};
    CK(cudaMemcpyAsync(v, h->d_scratch, sizeof v, cudaMemcpyDeviceToHost, h->stream));
    CK(cudaStreamSynchronize(h->stream));
    int rc = harvest_events(h);
    if (rc) return rc;
    uint64_t population = 0;
    for (const auto& rep : h->reps) population += rep.n;
    if (v[0] || v[2] != population || v[3] || v[4] != v[1] || v[5]) {
        h->err = "invariants: " + std::to_string(v[0]) + " agents off their cell class, " + std::to_string(v[2]) +
                 " occupied cells for " + std::to_string(population) + " agents, " + std::to_string(v[3]) +
                 " claims left in the spent plane, " + std::to_string(v[4]) + " class bytes for " + std::to_string(v[1]) +
                 " infectious agents, " + std::to_string(v[5]) + " cells with a wrong infectious-neighbour count";
        return EPI_ERR_INVARIANT;
    }
    return EPI_OK;
}

static int save_state(epi_engine* h);
static int restore_state(epi_engine* h);

static int set_launch_shape(epi_engine* h, uint32_t decide_blocks, uint32_t commit_slots) {
    const uint32_t n_chunks = h->slots / kChunk;
    if (decide_blocks == 0 || decide_blocks > n_chunks || commit_slots == 0 || commit_slots > (uint32_t)kMaxCommitSlots) {
        h->err = "launch shape: k_decide blocks in [1, " + std::to_string(n_chunks) + "], k_commit slots in [1, " +
                 std::to_string(kMaxCommitSlots) + "]";
        return EPI_ERR_ARG;
    }
    CK(cudaStreamSynchronize(h->stream));
    h->grid_blocks = (int)decide_blocks;
    h->commit_slots = (int)commit_slots;
    destroy_graphs(h);  // they bake the launch shapes in
    return EPI_OK;
}

// Launch-shape autotuner: times hours 1..hours of the engine's current world under each
// candidate k_decide grid (the present one, three quarters of the resident grid, the resident
// grid, twice it, one chunk per block) and, where it applies, in one launch, restarting every candidate from the same state, and keeps the fastest.
// Results do not depend on the shape; the state, the run's rows and the launch counter are
// restored afterwards (the saved checkpoint is replaced).
static int autotune(epi_engine* h, uint32_t hours, epi_launch_shape* out) {
    if (hours == 0 || hours > 24u * 7u) { h->err = "autotune hours must be in [1, 168]"; return EPI_ERR_ARG; }
    const uint32_t n_chunks = h->slots / kChunk;
    std::vector<uint32_t> grids;
    // three quarters of the resident grid too: fewer warps per SM share the L1 that holds the
    // plane rows their agents read
    const uint64_t cand[5] = {(uint64_t)h->grid_blocks, (uint64_t)h->resident_blocks * 3u / 4u, (uint64_t)h->resident_blocks,
                              2ull * (uint64_t)h->resident_blocks, (uint64_t)n_chunks};
    for (uint64_t g : cand) {
        const uint32_t v = (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>(g, n_chunks));
        if (std::find(grids.begin(), grids.end(), v) == grids.end()) grids.push_back(v);
    }
    const bool prof = h->profiling;
    const uint64_t launched = h->kernels_launched;
    h->profiling = false;
    int rc = save_state(h);
    if (rc) return rc;
    double best = 1e300;
    uint32_t best_g = (uint32_t)h->grid_blocks;
    // one launch for the hours (0) is a candidate where it would run a call of so many
    const uint32_t most = longest_together(h), before = h->together_most;
    bool keep_together = hours > most;
    if (hours <= most) grids.insert(grids.begin(), 0u);
    for (uint32_t g : grids) {
        h->together_most = g ? 0u : most;
        if (g) rc = set_launch_shape(h, g, (uint32_t)h->commit_slots);
        double t_min = 1e300;
        for (int rep = 0; rep < 5 && !rc; ++rep) {  // the first pass captures the graphs
            rc = restore_state(h);
            if (rc) break;
            const auto t0 = std::chrono::steady_clock::now();
            rc = run_hours(h, 1, hours);
            const double t = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
            if (rep > 0) t_min = std::min(t_min, t);
        }
        if (rc) break;
        if (t_min < best) {
            best = t_min;
            keep_together = g == 0u || hours > most;
            if (g) best_g = g;
        }
    }
    h->profiling = prof;
    int rc2 = set_launch_shape(h, best_g, (uint32_t)h->commit_slots);
    // a grid that beat one launch over these hours has shorter calls, mostly launch and wait, left to it
    h->together_most = rc ? before : keep_together ? most : std::min({most, hours - 1u, kShortHours});
    if (!rc2) rc2 = restore_state(h);
    h->kernels_launched = launched;
    if (rc) return rc;
    if (rc2) return rc2;
    if (out) {
        out->decide_blocks = best_g;
        out->commit_slots = (uint32_t)h->commit_slots;
        out->hour_us = best * 1e6 / hours;
    }
    return EPI_OK;
}

// Every replicate in the buffers of one parity (replicates that ended early may differ).
static int same_buffer(epi_engine* h) {
    for (uint32_t r = 1; r < h->R(); ++r) {
        int rc = move_to_buffer(h, r, h->reps[0].par);
        if (rc) return rc;
    }
    return EPI_OK;
}

static int save_state(epi_engine* h) {
    const size_t n = h->slots;
    int rc = EPI_OK;
    if (!h->s_pos) {
        CK(cudaMalloc(&h->s_pos, n * sizeof(uint32_t)));
        CK(cudaMalloc(&h->s_wsa, n * sizeof(uint32_t)));
        CK(cudaMalloc(&h->s_st, n * sizeof(uint2)));
        CK(cudaMalloc(&h->s_occ, h->occ_words * sizeof(uint32_t)));
        CK(cudaMalloc(&h->s_cls, h->plane_bytes));
        CK(cudaMalloc(&h->s_danger, h->plane_bytes));
    }
    rc = same_buffer(h);
    if (rc) return rc;
    const uint32_t par = h->reps[0].par;
    CK(cudaMemcpyAsync(h->s_pos, pos_buf(h, par), n * sizeof(uint32_t), cudaMemcpyDeviceToDevice, h->stream));
    CK(cudaMemcpyAsync(h->s_wsa, h->d_wsa, n * sizeof(uint32_t), cudaMemcpyDeviceToDevice, h->stream));
    CK(cudaMemcpyAsync(h->s_st, h->d_st, n * sizeof(uint2), cudaMemcpyDeviceToDevice, h->stream));
    CK(cudaMemcpyAsync(h->s_occ, occ_buf(h, par), h->occ_words * sizeof(uint32_t), cudaMemcpyDeviceToDevice, h->stream));
    CK(cudaMemcpyAsync(h->s_cls, h->d_cls, h->plane_bytes, cudaMemcpyDeviceToDevice, h->stream));
    CK(cudaMemcpyAsync(h->s_danger, h->d_danger, h->plane_bytes, cudaMemcpyDeviceToDevice, h->stream));
    CK(cudaStreamSynchronize(h->stream));
    for (auto& rep : h->reps) {
        rep.s_iv = rep.iv;
        rep.s_geo = rep.geo;
        rep.s_hosp_code = rep.hp.hosp_code;
        rep.s_active = rep.active;
        rep.s_par = par;
        rep.s_rows = rep.rows;
    }
    h->s_loop_hour = h->loop_hour;
    h->saved = true;
    return EPI_OK;
}

static int restore_state(epi_engine* h) {
    if (!h->saved) { h->err = "no saved state"; return EPI_ERR_ARG; }
    const size_t n = h->slots;
    const uint32_t par = h->reps[0].s_par;
    CK(cudaMemcpyAsync(pos_buf(h, par), h->s_pos, n * sizeof(uint32_t), cudaMemcpyDeviceToDevice, h->stream));
    CK(cudaMemcpyAsync(h->d_wsa, h->s_wsa, n * sizeof(uint32_t), cudaMemcpyDeviceToDevice, h->stream));
    CK(cudaMemcpyAsync(h->d_st, h->s_st, n * sizeof(uint2), cudaMemcpyDeviceToDevice, h->stream));
    CK(cudaMemcpyAsync(occ_buf(h, par), h->s_occ, h->occ_words * sizeof(uint32_t), cudaMemcpyDeviceToDevice, h->stream));
    CK(cudaMemsetAsync(occ_buf(h, 1u - par), 0, h->occ_words * sizeof(uint32_t), h->stream));
    CK(cudaMemcpyAsync(h->d_cls, h->s_cls, h->plane_bytes, cudaMemcpyDeviceToDevice, h->stream));
    CK(cudaMemcpyAsync(h->d_danger, h->s_danger, h->plane_bytes, cudaMemcpyDeviceToDevice, h->stream));
    CK(cudaMemsetAsync(h->d_claim, 0xFF, h->claim_cells * sizeof(uint32_t), h->stream));
    h->last_claim_hour = -1;
    for (auto& rep : h->reps) {
        rep.iv = rep.s_iv;
        rep.geo = rep.s_geo;
        rep.hp.hosp_code = rep.s_hosp_code;
        rep.active = rep.s_active;
        rep.hp.active = rep.s_active ? 1u : 0u;
        rep.par = rep.s_par;
        rep.rows = rep.s_rows;
    }
    h->loop_hour = h->s_loop_hour;
    return push_params(h);
}

static int create_engine(const epi_params* params, const epi_agent_record* const* recs, uint32_t R, epi_engine** out) {
    epi_engine* h = new epi_engine();
    int rc = engine_init(h, params, recs, R);
    if (rc) {
        g_create_error = h->err;
        free_device(h);
        delete h;
        return rc;
    }
    *out = h;
    return EPI_OK;
}

// ------------------------------------------------------------------ C ABI: config, geography, world
extern "C" {

int epi_params_from_json(const char* json_text, epi_params* out, char* err, size_t errlen) {
    if (!json_text || !out) return EPI_ERR_ARG;
    try {
        *out = params_from_json(json_text);
    } catch (const std::exception& e) {
        if (err && errlen) { std::snprintf(err, errlen, "%s", e.what()); }
        return EPI_ERR_CONFIG;
    }
    std::string bad = validate_params(*out);
    if (!bad.empty()) {
        if (err && errlen) std::snprintf(err, errlen, "%s", bad.c_str());
        return EPI_ERR_CONFIG;
    }
    return EPI_OK;
}

int epi_define_geography(uint32_t grid_size, epi_geography* out) {
    if (!out || grid_size < 1 || grid_size > 32766) return EPI_ERR_ARG;
    *out = define_geography(grid_size);
    return EPI_OK;
}

int epi_resize_hospital(epi_geography* geo, int32_t number_of_agents, double staff, double beds) {
    if (!geo) return EPI_ERR_ARG;
    resize_hospital(*geo, number_of_agents, staff, beds);
    return EPI_OK;
}

int epi_geography_increase_hospital_size(epi_geography* geo, uint32_t grid_size) {
    if (!geo || grid_size > 32766) return EPI_ERR_ARG;
    epi_geography g = *geo;
    g.grid_size = grid_size;
    geo->hospital = grown_hospital(g);
    return EPI_OK;
}

int epi_interventions_replay(const epi_params* p, const epi_counts* rows, uint32_t n, uint32_t* applied,
                             uint8_t* guard) {
    if (!p || (n && (!rows || !applied))) return EPI_ERR_ARG;
    const std::string bad = validate_params(*p);
    if (!bad.empty()) { g_create_error = bad; return EPI_ERR_CONFIG; }
    epi_geography geo = define_geography(p->grid_size);
    resize_hospital(geo, (int32_t)p->number_of_agents, 0.002, p->hospital_beds_percentage);
    const epi_geography geo0 = geo;
    InterventionState st;
    uint32_t ivn = 0;  // the device guard's new-infections figure
    for (uint32_t k = 0; k < n; ++k) {
        const epi_counts& c = rows[k];
        if (guard) {  // k_piece_end's verdict on this row, from the thresholds pushed before it
            uint8_t fire = 0;
            if (c.hour % 24u == 0u) {
                const GuardParams g = guard_params(*p, st, geo.hospital);
                const uint32_t fresh = c.infected > ivn ? c.infected - ivn : 0u;
                ivn = fresh;
                fire = ((g.flags & 1u) && c.infected > g.lock_threshold) || ((g.flags & 2u) && fresh >= g.spread_threshold) ||
                       ((g.flags & 4u) && c.hospitalized >= g.occ_threshold);
            }
            guard[k] = fire;
        }
        const InterventionActions a = decide_interventions(*p, st, c, geo.hospital);
        if (a.grow_hospital) geo.hospital = grown_hospital(geo0);
        applied[k] = a.applied;
    }
    return EPI_OK;
}

int epi_outputs_write(const char* dir, const char* engine_id, const epi_params* p, const epi_counts* rows, uint32_t n) {
    if (!dir || !engine_id || !p || (n && !rows)) return EPI_ERR_ARG;
    const std::string bad = validate_params(*p);
    if (!bad.empty()) { g_create_error = bad; return EPI_ERR_CONFIG; }
    epi_geography geo = define_geography(p->grid_size);
    resize_hospital(geo, (int32_t)p->number_of_agents, 0.002, p->hospital_beds_percentage);
    const epi_geography geo0 = geo;
    InterventionState st;
    for (uint32_t k = 0; k < n; ++k)
        if (decide_interventions(*p, st, rows[k], geo.hospital).grow_hospital) geo.hospital = grown_hospital(geo0);
    std::string err;
    const int rc = write_outputs(dir, engine_id, std::vector<epi_counts>(rows, rows + n), st.reports, err);
    if (rc) g_create_error = err;
    return rc;
}

double epi_disease_transmission_rate(const epi_params* p, uint32_t day) {
    switch (rate_class(p->regular_transmission_start_day, p->high_transmission_start_day, p->last_day, day)) {
        case 1: return p->regular_transmission_rate;
        case 2: return p->high_transmission_rate;
        default: return 0.0;
    }
}

int epi_disease_is_to_be_hospitalized(const epi_params* p, uint32_t day) {
    return epi_disease_transmission_rate(p, day) >= p->high_transmission_rate;
}

int epi_population_read_csv(const char* path, uint8_t* flags, uint32_t cap, uint32_t* n) {
    if (!path || !n) return EPI_ERR_ARG;
    std::vector<uint8_t> f;
    std::string err;
    int rc = read_population_csv(path, f, err);
    if (rc) { g_create_error = err; return rc; }
    *n = (uint32_t)f.size();
    if (flags) std::memcpy(flags, f.data(), std::min<size_t>(f.size(), cap));
    return EPI_OK;
}

int epi_world_build_population(const epi_params* p, const uint8_t* flags, uint32_t n, epi_agent_record* out,
                               epi_geography* geo) {
    if (!p || !flags || !out || n != p->number_of_agents) return EPI_ERR_ARG;
    std::vector<epi_agent_record> recs;
    epi_geography g;
    std::string err;
    int rc = build_world(*p, recs, g, err, flags);
    if (rc) { g_create_error = err; return rc; }
    std::memcpy(out, recs.data(), (size_t)n * sizeof(epi_agent_record));
    if (geo) *geo = g;
    return EPI_OK;
}

int epi_engine_create_population(const epi_params* params, const uint8_t* flags, uint32_t n, epi_engine** out) {
    if (!params || !flags || !out || n != params->number_of_agents) return EPI_ERR_ARG;
    *out = nullptr;
    epi_params p = *params;
    p.population_source = 1;
    epi_engine* h = new epi_engine();
    h->init_flags = flags;
    int rc = engine_init(h, &p, nullptr, 1);
    h->init_flags = nullptr;
    if (rc) {
        g_create_error = h->err;
        free_device(h);
        delete h;
        return rc;
    }
    *out = h;
    return EPI_OK;
}

int epi_world_build(const epi_params* p, epi_agent_record* out, size_t n, epi_geography* geo) {
    if (!p || !out || n != p->number_of_agents) return EPI_ERR_ARG;
    if (p->population_source == 1) { g_create_error = "Csv population: use epi_world_build_population"; return EPI_ERR_ARG; }
    std::vector<epi_agent_record> recs;
    epi_geography g;
    std::string err;
    int rc = build_world(*p, recs, g, err);
    if (rc) { g_create_error = err; return rc; }
    std::memcpy(out, recs.data(), n * sizeof(epi_agent_record));
    if (geo) *geo = g;
    return EPI_OK;
}

// ------------------------------------------------------------------ C ABI: single engine
int epi_engine_create_from_records(const epi_params* params, const epi_agent_record* recs, size_t n, epi_engine** out) {
    if (!params || !recs || !out) return EPI_ERR_ARG;
    *out = nullptr;
    if (n != params->number_of_agents || n == 0 || n >= 0xFFFFFFFFull) {
        g_create_error = "record count != number_of_agents";
        return EPI_ERR_ARG;
    }
    const epi_agent_record* one[1] = {recs};
    return create_engine(params, one, 1, out);
}

int epi_engine_create(const epi_params* params, epi_engine** out) {
    if (!params || !out) return EPI_ERR_ARG;
    *out = nullptr;
    return create_engine(params, nullptr, 1, out);
}

int epi_engine_create_json(const char* config_json, uint64_t seed, epi_engine** out) {
    if (!out) return EPI_ERR_ARG;
    *out = nullptr;
    epi_params p;
    char msg[512] = {0};
    int rc = epi_params_from_json(config_json, &p, msg, sizeof msg);
    if (rc) { g_create_error = msg; return rc; }
    p.seed = seed;
    if (p.population_source == 1) {  // Population::Csv: read the rows of its file
        std::vector<uint8_t> flags;
        std::string err;
        rc = read_population_csv(p.population_file, flags, err);
        if (rc) { g_create_error = err; return rc; }
        return epi_engine_create_population(&p, flags.data(), (uint32_t)flags.size(), out);
    }
    return epi_engine_create(&p, out);
}

void epi_engine_destroy(epi_engine* h) {
    if (!h) return;
    free_device(h);
    delete h;
}

const char* epi_engine_last_error(const epi_engine* h) { return h ? h->err.c_str() : g_create_error.c_str(); }

int epi_engine_set_stream(epi_engine* h, void* cuda_stream) {
    if (!h) return EPI_ERR_ARG;
    CK(cudaStreamSynchronize(h->stream));
    if (h->own_stream) CK(cudaStreamDestroy(h->stream));
    if (cuda_stream) {
        h->stream = (cudaStream_t)cuda_stream;
        h->own_stream = false;
    } else {
        CK(cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking));
        h->own_stream = true;
    }
    return EPI_OK;
}

int epi_engine_simulate_hours(epi_engine* h, uint32_t first_hour, uint32_t n, epi_counts* out) {
    if (!h || (!out && n)) return EPI_ERR_ARG;
    int rc = run_hours(h, first_hour, n);
    if (rc) return rc;
    for (uint32_t k = 0; k < n; ++k) out[k] = counts_of(h, k, 0, first_hour + k);
    return EPI_OK;
}

int epi_engine_simulate(epi_engine* h, uint32_t hour, epi_counts* out) {
    if (!h || !out) return EPI_ERR_ARG;
    return epi_engine_simulate_hours(h, hour, 1, out);
}

int epi_engine_lock_city(epi_engine* h) { return h ? lock_city(h, 0, 1) : EPI_ERR_ARG; }
int epi_engine_unlock_city(epi_engine* h) { return h ? lock_city(h, 0, 0) : EPI_ERR_ARG; }

int epi_engine_vaccinate(epi_engine* h, uint32_t hour, double percent) {
    if (!h || !(percent >= 0.0 && percent <= 1.0)) return EPI_ERR_ARG;
    return vaccinate(h, 0, hour, percent);
}

int epi_engine_increase_hospital_size(epi_engine* h) {
    if (!h) return EPI_ERR_ARG;
    grow_hospital(h, 0);
    return push_params(h);
}

int epi_engine_process_interventions(epi_engine* h, const epi_counts* counts, uint32_t* applied) {
    if (!h || !counts) return EPI_ERR_ARG;
    bool dirty = false;
    int rc = process_interventions(h, 0, *counts, applied, &dirty);
    if (rc) return rc;
    return dirty ? push_params(h) : EPI_OK;
}

int epi_engine_run(epi_engine* h, epi_counts* rows, uint32_t max_rows, uint32_t* n_rows) {
    if (!h || !n_rows) return EPI_ERR_ARG;
    *n_rows = 0;
    int rc = run_loop(h);
    if (rc) return rc;
    const std::vector<epi_counts>& got = h->reps[0].rows;
    const uint32_t nr = (uint32_t)got.size();
    if (rows) {
        if (max_rows < nr) { h->err = "rows buffer too small"; return EPI_ERR_ARG; }
        std::memcpy(rows, got.data(), nr * sizeof(epi_counts));
    }
    *n_rows = nr;
    return EPI_OK;
}

int epi_engine_run_until(epi_engine* h, uint32_t last_hour, epi_counts* rows, uint32_t max_rows, uint32_t* n_rows,
                         uint32_t* next_hour) {
    if (!h || !n_rows || !next_hour) return EPI_ERR_ARG;
    *n_rows = 0;
    *next_hour = 0;
    int rc = run_loop(h, last_hour);
    if (rc) return rc;
    const std::vector<epi_counts>& got = h->reps[0].rows;
    const uint32_t nr = (uint32_t)got.size();
    if (rows) {
        if (max_rows < nr) { h->err = "rows buffer too small"; return EPI_ERR_ARG; }
        std::memcpy(rows, got.data(), nr * sizeof(epi_counts));
    }
    *n_rows = nr;
    *next_hour = h->loop_hour;
    return EPI_OK;
}

}  // extern "C"

// ---- checkpoint file
namespace {
constexpr uint32_t kCheckpointMagic = 0x4B435045u;  // "EPCK"
constexpr uint32_t kCheckpointVersion = 1;

uint64_t fnv1a64(const std::vector<uint8_t>& b) {  // FNV-1a (Fowler, Noll, Vo), 64-bit
    uint64_t x = 0xCBF29CE484222325ull;
    for (uint8_t c : b) {
        x ^= c;
        x *= 0x100000001B3ull;
    }
    return x;
}
template <typename T>
void put(std::vector<uint8_t>& b, const T& v) {
    const uint8_t* p = reinterpret_cast<const uint8_t*>(&v);
    b.insert(b.end(), p, p + sizeof(T));
}
void put_bytes(std::vector<uint8_t>& b, const void* p, size_t n) {
    b.insert(b.end(), static_cast<const uint8_t*>(p), static_cast<const uint8_t*>(p) + n);
}
void put_string(std::vector<uint8_t>& b, const std::string& s) {
    put(b, (uint32_t)s.size());
    put_bytes(b, s.data(), s.size());
}
struct Reader {
    const std::vector<uint8_t>& b;
    size_t at = 0;
    bool ok = true;
    bool bytes(void* dst, size_t n) {
        if (!ok || n > b.size() - at) return ok = false;
        std::memcpy(dst, b.data() + at, n);
        at += n;
        return true;
    }
    template <typename T>
    bool get(T& v) { return bytes(&v, sizeof(T)); }
    bool string(std::string& s) {
        uint32_t n = 0;
        if (!get(n) || n > b.size() - at) return ok = false;
        s.assign(reinterpret_cast<const char*>(b.data() + at), n);
        at += n;
        return true;
    }
};
}  // namespace

extern "C" {

int epi_engine_checkpoint_write(epi_engine* h, const char* path) {
    if (!h || !path) return EPI_ERR_ARG;
    if (h->R() != 1) { h->err = "checkpoints are for single engines"; return EPI_ERR_ARG; }
    const Replica& rep = h->reps[0];
    std::vector<epi_agent_record> recs(rep.n);
    int rc = snapshot_replica(h, 0, recs.data(), recs.size());
    if (rc) return rc;
    std::vector<uint8_t> b;
    for (uint32_t v : {kCheckpointMagic, kCheckpointVersion, (uint32_t)sizeof(epi_params), (uint32_t)sizeof(epi_geography),
                       (uint32_t)sizeof(epi_agent_record), (uint32_t)sizeof(epi_counts), rep.n, h->loop_hour,
                       (uint32_t)rep.rows.size(), (uint32_t)rep.iv.reports.size(), rep.active ? 1u : 0u,
                       rep.iv.locked ? 1u : 0u, rep.iv.zero_infection_hour, rep.iv.new_infections_in_a_day,
                       rep.iv.hospital_applied ? 1u : 0u})
        put(b, v);
    put(b, rep.p);
    put(b, rep.geo);
    put_bytes(b, rep.rows.data(), rep.rows.size() * sizeof(epi_counts));
    for (const Report& r : rep.iv.reports) {
        put(b, r.hour);
        put_string(b, r.name);
        put_string(b, r.data);
    }
    put_bytes(b, recs.data(), recs.size() * sizeof(epi_agent_record));
    put(b, fnv1a64(b));
    FILE* f = std::fopen(path, "wb");
    if (!f) { h->err = std::string("checkpoint: cannot write ") + path; return EPI_ERR_IO; }
    const bool ok = std::fwrite(b.data(), 1, b.size(), f) == b.size();
    if (std::fclose(f) != 0 || !ok) { h->err = std::string("checkpoint: write failed: ") + path; return EPI_ERR_IO; }
    return EPI_OK;
}

int epi_engine_create_from_checkpoint(const char* path, epi_engine** out) {
    if (!path || !out) return EPI_ERR_ARG;
    *out = nullptr;
    auto fail = [](const std::string& m) {
        g_create_error = "checkpoint: " + m;
        return EPI_ERR_IO;
    };
    std::vector<uint8_t> b;
    {
        FILE* f = std::fopen(path, "rb");
        if (!f) return fail(std::string("cannot read ") + path);
        uint8_t buf[1 << 16];
        size_t k;
        while ((k = std::fread(buf, 1, sizeof buf, f)) > 0) b.insert(b.end(), buf, buf + k);
        std::fclose(f);
    }
    if (b.size() < 15 * 4 + 8) return fail("truncated file");
    uint64_t sum = 0;
    std::memcpy(&sum, b.data() + b.size() - 8, 8);
    b.resize(b.size() - 8);
    if (fnv1a64(b) != sum) return fail("checksum mismatch (truncated or corrupt file)");
    Reader rd{b};
    uint32_t hdr[15];
    for (uint32_t& v : hdr) rd.get(v);
    if (hdr[0] != kCheckpointMagic) return fail("not a checkpoint file");
    if (hdr[1] != kCheckpointVersion) return fail("unsupported version " + std::to_string(hdr[1]));
    if (hdr[2] != sizeof(epi_params) || hdr[3] != sizeof(epi_geography) || hdr[4] != sizeof(epi_agent_record) ||
        hdr[5] != sizeof(epi_counts))
        return fail("written by a build with other struct layouts");
    const uint32_t n = hdr[6], loop_hour = hdr[7], n_rows = hdr[8], n_reports = hdr[9];
    epi_params p;
    epi_geography geo;
    rd.get(p);
    rd.get(geo);
    if (!rd.ok || p.number_of_agents != n || n == 0) return fail("inconsistent header");
    if ((uint64_t)n_rows * sizeof(epi_counts) > b.size()) return fail("truncated file");
    std::vector<epi_counts> rows(n_rows);
    rd.bytes(rows.data(), rows.size() * sizeof(epi_counts));
    std::vector<Report> reports(std::min<uint32_t>(n_reports, 1u << 20));
    for (Report& r : reports) {
        rd.get(r.hour);
        rd.string(r.name);
        rd.string(r.data);
    }
    if ((uint64_t)n * sizeof(epi_agent_record) > b.size()) return fail("truncated file");
    std::vector<epi_agent_record> recs(n);
    rd.bytes(recs.data(), recs.size() * sizeof(epi_agent_record));
    if (!rd.ok || rd.at != b.size() || reports.size() != n_reports) return fail("truncated or malformed file");
    const std::string bad = validate_params(p);
    if (!bad.empty()) return fail(bad);
    epi_engine* h = nullptr;
    const epi_agent_record* one[1] = {recs.data()};
    int rc = create_engine(&p, one, 1, &h);
    if (rc) return rc;
    Replica& rep = h->reps[0];
    rep.geo = geo;
    rep.hp.hosp_code = rect_eq(to_rect(geo.hospital), rep.hp.area[kHosp0]) ? kHosp0 : kHosp1;
    rep.iv.locked = hdr[11] != 0;
    rep.iv.zero_infection_hour = hdr[12];
    rep.iv.new_infections_in_a_day = hdr[13];
    rep.iv.hospital_applied = hdr[14] != 0;
    rep.iv.reports = std::move(reports);
    rep.rows = std::move(rows);
    rep.active = hdr[10] != 0;
    rep.hp.active = rep.active ? 1u : 0u;
    h->loop_hour = loop_hour;
    rc = push_params(h);
    if (rc) {
        g_create_error = h->err;
        epi_engine_destroy(h);
        return rc;
    }
    *out = h;
    return EPI_OK;
}

int epi_engine_write_outputs(epi_engine* h, const char* dir, const char* engine_id) {
    if (!h || !dir || !engine_id) return EPI_ERR_ARG;
    return write_outputs(dir, engine_id, h->reps[0].rows, h->reps[0].iv.reports, h->err);
}

int epi_engine_population(const epi_engine* h, uint32_t* out) {
    if (!h || !out) return EPI_ERR_ARG;
    *out = h->reps[0].n;
    return EPI_OK;
}

int epi_engine_geography(const epi_engine* h, epi_geography* out) {
    if (!h || !out) return EPI_ERR_ARG;
    *out = h->reps[0].geo;
    return EPI_OK;
}

int epi_engine_snapshot(epi_engine* h, epi_agent_record* out, size_t n) {
    if (!h) return EPI_ERR_ARG;
    return snapshot_replica(h, 0, out, n);
}

int epi_engine_check(epi_engine* h) { return h ? check_all(h) : EPI_ERR_ARG; }
int epi_engine_save_state(epi_engine* h) { return h ? save_state(h) : EPI_ERR_ARG; }
int epi_engine_restore_state(epi_engine* h) { return h ? restore_state(h) : EPI_ERR_ARG; }

int epi_engine_autotune(epi_engine* h, uint32_t hours, epi_launch_shape* chosen) {
    if (!h) return EPI_ERR_ARG;
    if (h->stream_file) { h->err = "autotune: close the citizen-state stream first"; return EPI_ERR_ARG; }
    return autotune(h, hours, chosen);
}

// Citizen-state stream file: "EPCS", version 1, agents, grid (u32 each); the keyframe (per
// agent x, y as u16, then every agent's state letter byte); then hour records (stream_write).
int epi_engine_state_stream_open(epi_engine* h, const char* path) {
    if (!h || !path) return EPI_ERR_ARG;
    if (h->R() != 1) { h->err = "the citizen-state stream is for single engines"; return EPI_ERR_ARG; }
    if (h->stream_file) { h->err = "citizen-state stream already open"; return EPI_ERR_ARG; }
    const uint32_t n = h->reps[0].n;
    std::vector<epi_agent_record> recs(n);
    int rc = snapshot_replica(h, 0, recs.data(), n);
    if (rc) return rc;
    FILE* f = std::fopen(path, "wb");
    if (!f) { h->err = std::string("cannot open ") + path; return EPI_ERR_IO; }
    const uint32_t head[4] = {0x53435045u /* "EPCS" */, 1u, n, h->reps[0].p.grid_size};
    std::vector<uint16_t> xy((size_t)n * 2);
    std::vector<uint8_t> letters(n);
    for (uint32_t i = 0; i < n; ++i) {
        xy[2 * i] = (uint16_t)recs[i].x;
        xy[2 * i + 1] = (uint16_t)recs[i].y;
        const uint32_t v = recs[i].state;
        letters[i] = (uint8_t)(v == EPI_S ? 0 : v == EPI_E ? 1 : v == EPI_R ? 3 : v == EPI_D ? 4 : 2);
    }
    if (std::fwrite(head, sizeof head, 1, f) != 1 || std::fwrite(xy.data(), sizeof(uint16_t), xy.size(), f) != xy.size() ||
        std::fwrite(letters.data(), 1, n, f) != n) {
        std::fclose(f);
        h->err = "citizen-state stream: write failed";
        return EPI_ERR_IO;
    }
    h->stream_file = f;
    const size_t cap = (size_t)kStreamChunk * h->slots;
    CK(cudaMalloc(&h->d_prev, (size_t)h->slots * sizeof(uint32_t)));
    CK(cudaMalloc(&h->d_codes, cap));
    CK(cudaMalloc(&h->d_exc, cap * sizeof(uint2)));
    CK(cudaMalloc(&h->d_exc_n, kStreamChunk * sizeof(uint32_t)));
    CK(cudaMallocHost(&h->h_codes, cap));
    CK(cudaMallocHost(&h->h_exc, (size_t)h->slots * sizeof(uint2)));
    CK(cudaMallocHost(&h->h_exc_n, kStreamChunk * sizeof(uint32_t)));
    CK(cudaMemcpyAsync(h->d_prev, pos_buf(h, h->reps[0].par), (size_t)h->slots * sizeof(uint32_t), cudaMemcpyDeviceToDevice, h->stream));
    CK(cudaStreamSynchronize(h->stream));
    destroy_graphs(h);  // hour graphs now carry the encoding kernel
    return EPI_OK;
}

int epi_engine_state_stream_close(epi_engine* h) {
    if (!h) return EPI_ERR_ARG;
    if (!h->stream_file) return EPI_OK;
    const int bad = std::fflush(h->stream_file);
    stream_free(h);
    destroy_graphs(h);
    if (bad) { h->err = "citizen-state stream: flush failed"; return EPI_ERR_IO; }
    return EPI_OK;
}

int epi_engine_set_launch_shape(epi_engine* h, const epi_launch_shape* shape) {
    if (!h || !shape) return EPI_ERR_ARG;
    const int rc = set_launch_shape(h, shape->decide_blocks, shape->commit_slots);
    if (!rc) h->together_most = 0;  // a shape that was asked for runs the hour kernels
    return rc;
}

int epi_engine_set_wait_limit(epi_engine* h, uint32_t polls) {
    if (!h) return EPI_ERR_ARG;
    h->wait_polls = polls;
    return EPI_OK;
}

int epi_engine_launch_shape(const epi_engine* h, epi_launch_shape* out) {
    if (!h || !out) return EPI_ERR_ARG;
    out->decide_blocks = (uint32_t)h->grid_blocks;
    out->commit_slots = (uint32_t)h->commit_slots;
    out->hour_us = 0.0;
    return EPI_OK;
}

int epi_engine_kernels_launched(const epi_engine* h, uint64_t* out) {
    if (!h || !out) return EPI_ERR_ARG;
    *out = h->kernels_launched;
    return EPI_OK;
}

int epi_engine_set_profiling(epi_engine* h, int on) {
    if (!h) return EPI_ERR_ARG;
    h->profiling = on != 0;
    for (int k = 0; k < kKindCount; ++k) { h->launches[k] = 0; h->total_ms[k] = 0.0; }
    return EPI_OK;
}

int epi_engine_kernel_stats(const epi_engine* h, uint32_t* launches, double* total_ms, int n) {
    if (!h || !launches || !total_ms) return EPI_ERR_ARG;
    for (int k = 0; k < n && k < kKindCount; ++k) { launches[k] = h->launches[k]; total_ms[k] = h->total_ms[k]; }
    return EPI_OK;
}

const char* epi_engine_kernel_name(int k) { return (k >= 0 && k < kKindCount) ? kKernelNames[k] : ""; }
int epi_engine_kernel_kinds(void) { return kKindCount; }

size_t epi_abi_struct_size(const char* name) {
    if (!name) return 0;
    if (!std::strcmp(name, "epi_params")) return sizeof(epi_params);
    if (!std::strcmp(name, "epi_agent_record")) return sizeof(epi_agent_record);
    if (!std::strcmp(name, "epi_counts")) return sizeof(epi_counts);
    if (!std::strcmp(name, "epi_geography")) return sizeof(epi_geography);
    if (!std::strcmp(name, "epi_mlp_config")) return sizeof(epi_mlp_config);
    return 0;
}

// Algorithmic bytes of one hour over all replicates (the roofline numerator): the agent
// words the hour's kernels must read and write plus one pass over each plane they touch throughout.
//   hours 7..22: pos 4 + st 8 + home 4 + work 4 read, pos 4 written; per cell of (G+1)^2 a bit read,
//   a bit written and an infectious-neighbour count of a byte read.
//   hours 0 and 23: the same words read; the few agents that act patch theirs and the planes.
//   hour 1: st.x read 4 + write 4; hours 2-6 of a segment move no data.
int epi_engine_hour_bytes(const epi_engine* h, uint32_t hour, double* bytes) {
    if (!h || !bytes) return EPI_ERR_ARG;
    const uint32_t hod = hour % 24u;
    double b = 0.0;
    for (const auto& rep : h->reps) {
        const double n = (double)rep.n, side = (double)rep.p.grid_size + 1.0;
        if (hod >= 1u && hod <= 6u) b += hod == 1u ? n * 8.0 : 0.0;
        else b += rebuild_hour(hod) ? n * 24.0 + 1.25 * side * side : n * 20.0;
    }
    *bytes = b;
    return EPI_OK;
}

// ------------------------------------------------------------------ C ABI: ensemble
int epi_ensemble_create(const epi_params* params, uint32_t replicates, epi_ensemble** out) {
    if (!params || !out || replicates == 0) return EPI_ERR_ARG;
    *out = nullptr;
    epi_ensemble* e = new epi_ensemble();
    int rc = engine_init(&e->core, params, nullptr, replicates);
    if (rc) {
        g_create_error = e->core.err;
        free_device(&e->core);
        delete e;
        return rc;
    }
    *out = e;
    return EPI_OK;
}

void epi_ensemble_destroy(epi_ensemble* e) {
    if (!e) return;
    free_device(&e->core);
    delete e;
}

const char* epi_ensemble_last_error(const epi_ensemble* e) { return e ? e->core.err.c_str() : g_create_error.c_str(); }

int epi_ensemble_set_stream(epi_ensemble* e, void* cuda_stream) {
    return e ? epi_engine_set_stream(&e->core, cuda_stream) : EPI_ERR_ARG;
}

int epi_ensemble_run(epi_ensemble* e, epi_counts* rows, uint32_t max_rows_per_replicate, uint32_t* n_rows) {
    if (!e || !n_rows) return EPI_ERR_ARG;
    epi_engine* h = &e->core;
    int rc = run_loop(h);
    if (rc) return rc;
    for (uint32_t r = 0; r < h->R(); ++r) {
        const std::vector<epi_counts>& got = h->reps[r].rows;
        n_rows[r] = (uint32_t)got.size();
        if (rows) {
            if (got.size() > max_rows_per_replicate) { h->err = "rows buffer too small"; return EPI_ERR_ARG; }
            std::memcpy(rows + (size_t)r * max_rows_per_replicate, got.data(), got.size() * sizeof(epi_counts));
        }
    }
    return EPI_OK;
}

int epi_ensemble_replicates(const epi_ensemble* e, uint32_t* out) {
    if (!e || !out) return EPI_ERR_ARG;
    *out = e->core.R();
    return EPI_OK;
}

int epi_ensemble_snapshot(epi_ensemble* e, uint32_t replicate, epi_agent_record* out, size_t n) {
    if (!e || replicate >= e->core.R()) return EPI_ERR_ARG;
    return snapshot_replica(&e->core, replicate, out, n);
}

int epi_ensemble_check(epi_ensemble* e) { return e ? check_all(&e->core) : EPI_ERR_ARG; }
int epi_ensemble_save_state(epi_ensemble* e) { return e ? save_state(&e->core) : EPI_ERR_ARG; }
int epi_ensemble_restore_state(epi_ensemble* e) { return e ? restore_state(&e->core) : EPI_ERR_ARG; }
int epi_ensemble_set_profiling(epi_ensemble* e, int on) { return e ? epi_engine_set_profiling(&e->core, on) : EPI_ERR_ARG; }

int epi_ensemble_kernel_stats(const epi_ensemble* e, uint32_t* launches, double* total_ms, int n) {
    return e ? epi_engine_kernel_stats(&e->core, launches, total_ms, n) : EPI_ERR_ARG;
}

int epi_ensemble_autotune(epi_ensemble* e, uint32_t hours, epi_launch_shape* chosen) {
    return e ? autotune(&e->core, hours, chosen) : EPI_ERR_ARG;
}

int epi_ensemble_kernels_launched(const epi_ensemble* e, uint64_t* out) {
    return e ? epi_engine_kernels_launched(&e->core, out) : EPI_ERR_ARG;
}

int epi_ensemble_hour_bytes(const epi_ensemble* e, uint32_t hour, double* bytes) {
    return e ? epi_engine_hour_bytes(&e->core, hour, bytes) : EPI_ERR_ARG;
}

}  // extern "C"

// ------------------------------------------------------------------ no-allocation hour
// epi_tick_hour_noalloc: one simulated hour on device arrays the caller owns, for callers
// that cannot allocate device memory (see include/epi_engine.h).  Its scratch -- the
// parameter block, the hour word, the error word, the per-agent proposal buffer and the
// (G+1)^2 claim plane -- lives in the file-scope array below, which every GPU that loads
// this library holds until the process exits.  All calls share it: calls whose work overlaps
// on the GPU (two streams, two host threads) race on it and must be serialised by the caller.
namespace {

constexpr size_t kNoAllocScratchBytes = size_t(48) << 20;  // 48 MiB
constexpr size_t kNoAllocParamsOff = 0;                     // DevParams
constexpr size_t kNoAllocHourOff = 256;                     // SegDev {hour, hour}
constexpr size_t kNoAllocErrOff = 264;                      // int error flags
constexpr size_t kNoAllocTgtOff = 512;                      // u32 per agent
static_assert(sizeof(DevParams) <= kNoAllocHourOff, "parameter block must fit its slot");

static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];

struct NoAllocDevice {
    unsigned char* base = nullptr;  // device address of g_noalloc_scratch on this device
    int grid_blocks = 0;            // resident grid of k_decide / k_sleep
};
constexpr int kNoAllocMaxDevices = 64;
NoAllocDevice g_noalloc_devices[kNoAllocMaxDevices];
std::mutex g_noalloc_mutex;

size_t align256(size_t v) { return (v + 255) & ~size_t(255); }

using DecideBytesKernel = void (*)(const DevParams*, uint32_t, const uint32_t*, uint2*, const uint32_t*, const uint32_t*,
                                   uint32_t*, const uint8_t*, uint32_t*, uint32_t*, HourArgs, int*);
DecideBytesKernel decide_bytes_kernel(uint32_t hod) {
    switch (hour_class(hod)) {
        case kHcStart: return k_decide_bytes<kHcStart>;
        case kHcEnd: return k_decide_bytes<kHcEnd>;
        case kHcTransport: return k_decide_bytes<kHcTransport>;
        case kHcWork: return k_decide_bytes<kHcWork>;
        case kHcNoon: return k_decide_bytes<kHcNoon>;
        case kHcHome: return k_decide_bytes<kHcHome>;
        default: return k_decide_bytes<kHcMove>;
    }
}

DevParams noalloc_params(const epi_params& p, uint32_t hospital_grown) {
    epi_geography g = define_geography(p.grid_size);
    resize_hospital(g, (int32_t)p.number_of_agents, 0.002, p.hospital_beds_percentage);
    DevParams d = make_dev_params(p, g, p.number_of_agents);
    d.hosp_code = (hospital_grown && !rect_eq(d.area[kHosp1], d.area[kHosp0])) ? kHosp1 : kHosp0;
    return d;
}

int noalloc_fail(int rc, const std::string& msg) {
    g_create_error = msg;
    return rc;
}

#define NOALLOC_CK(call)                                                                     \
    do {                                                                                     \
        cudaError_t e_ = (call);                                                             \
        if (e_ != cudaSuccess) return noalloc_fail(EPI_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
    } while (0)

// Once per device, with that device current: the device address of the scratch array (the
// host-side symbol is only a stand-in) and the launch shape.
int noalloc_setup(int dev, NoAllocDevice** out) {
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    NoAllocDevice& d = g_noalloc_devices[dev];
    if (!d.base) {
        void* ptr = nullptr;
        NOALLOC_CK(cudaGetSymbolAddress(&ptr, g_noalloc_scratch));
        int sms = 0, per_sm = 0;
        NOALLOC_CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        NOALLOC_CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, (const void*)decide_bytes_kernel(9u), kThreads, 0));
        d.grid_blocks = sms * std::max(per_sm, 1);
        d.base = static_cast<unsigned char*>(ptr);
    }
    *out = &d;
    return EPI_OK;
}

}  // namespace

extern "C" int epi_tick_hour_noalloc(const epi_params* params, uint32_t hour, uint32_t hospital_grown, uint32_t* pos,
                                     uint32_t* state, const uint32_t* home, const uint32_t* work, uint32_t* work_start_at,
                                     uint8_t* plane, uint32_t* counts, void* cuda_stream) {
    if (!params || !pos || !state || !home || !work || !work_start_at || !plane || !counts)
        return noalloc_fail(EPI_ERR_ARG, "epi_tick_hour_noalloc: null pointer argument");
    if (reinterpret_cast<uintptr_t>(state) % 8 != 0)
        return noalloc_fail(EPI_ERR_ARG, "epi_tick_hour_noalloc: state must be 8-byte aligned (two words per agent)");
    // the neighbourhood reads take each plane row in aligned 32-bit words; the per-agent
    // arrays and the counts are read and written as 32-bit words
    if (reinterpret_cast<uintptr_t>(plane) % 4 != 0)
        return noalloc_fail(EPI_ERR_ARG, "epi_tick_hour_noalloc: plane must be 4-byte aligned");
    for (const void* w : {(const void*)pos, (const void*)home, (const void*)work, (const void*)work_start_at,
                          (const void*)counts})
        if (reinterpret_cast<uintptr_t>(w) % 4 != 0)
            return noalloc_fail(EPI_ERR_ARG,
                                "epi_tick_hour_noalloc: pos, home, work, work_start_at and counts must be 4-byte aligned");
    const std::string bad = validate_params(*params);
    if (!bad.empty()) return noalloc_fail(EPI_ERR_CONFIG, bad);
    const uint32_t n = params->number_of_agents;
    const size_t side = (size_t)params->grid_size + 1;
    const size_t claim_off = align256(kNoAllocTgtOff + (size_t)n * sizeof(uint32_t));
    const size_t claim_bytes = side * side * sizeof(uint32_t);
    if (claim_off + claim_bytes > kNoAllocScratchBytes)
        return noalloc_fail(EPI_ERR_CAPACITY,
                            "epi_tick_hour_noalloc: " + std::to_string(n) + " agents on a grid of " +
                                std::to_string(params->grid_size) + " need " + std::to_string(claim_off + claim_bytes) +
                                " bytes of scratch; the fixed maximum is " + std::to_string(kNoAllocScratchBytes));
    int dev = 0;
    NOALLOC_CK(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kNoAllocMaxDevices) return noalloc_fail(EPI_ERR_ARG, "epi_tick_hour_noalloc: device index too large");
    NoAllocDevice* d = nullptr;
    int rc = noalloc_setup(dev, &d);
    if (rc) return rc;
    cudaStream_t s = static_cast<cudaStream_t>(cuda_stream);
    const DevParams hp = noalloc_params(*params, hospital_grown);
    DevParams* d_params = reinterpret_cast<DevParams*>(d->base + kNoAllocParamsOff);
    SegDev* d_hour = reinterpret_cast<SegDev*>(d->base + kNoAllocHourOff);
    const SegDev seg{hour, hour};
    const HourArgs ha{d_hour, counts, 8u, 0u, 0u};
    int* d_err = reinterpret_cast<int*>(d->base + kNoAllocErrOff);
    uint32_t* d_tgt = reinterpret_cast<uint32_t*>(d->base + kNoAllocTgtOff);
    uint32_t* d_claim = reinterpret_cast<uint32_t*>(d->base + claim_off);
    // every call starts from clean scratch: the claim plane free, the error word zero
    NOALLOC_CK(cudaMemcpyAsync(d_params, &hp, sizeof hp, cudaMemcpyHostToDevice, s));
    NOALLOC_CK(cudaMemcpyAsync(d_hour, &seg, sizeof seg, cudaMemcpyHostToDevice, s));
    NOALLOC_CK(cudaMemsetAsync(d_err, 0, sizeof(int), s));
    NOALLOC_CK(cudaMemsetAsync(counts, 0, 8 * sizeof(uint32_t), s));
    uint2* st = reinterpret_cast<uint2*>(state);
    const uint32_t n_chunks = (n + kChunk - 1) / kChunk;
    const int blocks = (int)std::min<uint64_t>(n_chunks, (uint64_t)d->grid_blocks);
    const uint32_t hod = hour % 24u;
    if (hod >= 1u && hod <= 6u) {
        k_sleep<<<blocks, kThreads, 0, s>>>(d_params, nullptr, n_chunks, 1u, st, ha);
    } else {
        NOALLOC_CK(cudaMemsetAsync(d_claim, 0xFF, claim_bytes, s));
        decide_bytes_kernel(hod)<<<blocks, kThreads, 0, s>>>(d_params, n_chunks, pos, st, home, work, work_start_at, plane,
                                                             d_claim, d_tgt, ha, d_err);
        k_commit_bytes<<<blocks, kThreads, 0, s>>>(d_params, n, pos, d_tgt, plane, d_claim);
    }
    NOALLOC_CK(cudaGetLastError());
    int err = 0;
    NOALLOC_CK(cudaMemcpyAsync(&err, d_err, sizeof err, cudaMemcpyDeviceToHost, s));
    NOALLOC_CK(cudaStreamSynchronize(s));
    if (err) return noalloc_fail(EPI_ERR_INVARIANT, "epi_tick_hour_noalloc: a rule addressed a cell outside the plane");
    return EPI_OK;
}
