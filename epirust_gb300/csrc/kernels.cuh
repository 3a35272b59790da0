// kernels.cuh -- the sm_103a kernels of the hourly tick, over one or many replicates.
//
// Agent slots of all replicates are concatenated; each replicate starts on a 256-slot chunk
// boundary, so a chunk belongs to one replicate (chunk_rep[c]; absent when there is one).
// The counting kernels walk chunks with a grid-stride loop, stage the chunk's replicate
// parameters in shared memory and flush their per-block histogram whenever the replicate
// changes; the commit kernel takes the lists they leave.  Philox counters and claim values use
// the agent's index within its replicate, so a replicate evolves exactly as a lone engine
// with the same parameters would.
//
// Per simulated hour (CitizenLocationMap::simulate, engine/src/allocation_map.rs:67-129):
//   hours 1..6 of a day   k_sleep   current_area = home (non-staff), counts
//   other hours           k_decide  per-agent rules on the previous-hour planes, proposals,
//                                   an occupancy bit claimed per agent, counts
//                         k_commit  displaced claimants back to their cells, class planes, spent buffers zeroed
#pragma once

#include "tick.cuh"

namespace epi {
namespace kern {

constexpr int kThreads = (int)kChunk;

// Programmatic dependent launch: the hour kernels are launched so that the next kernel's
// launch is set up while the one before it runs.  dep_wait() returns once every earlier
// kernel of the stream has completed and its writes are visible (a no-op for a normal
// launch), so each hour kernel calls it before its first global access.  The kernels signal
// nothing early: blocks of the next kernel resident (and waiting) beside the running one were
// measured 1.7 % slower per hour than letting them start at its completion.
__device__ __forceinline__ void dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Warp-aggregated 6-bin histogram: three ballots carry the bits of each lane's bin (invalid
// lanes vote bin 7), lane b (< 6) counts the lanes whose bits spell b in a register, and the
// warp adds its counts to the block's when they are due.
struct Tally {
    uint32_t n0, n1, n2, n = 0;  // all ones where the lane number's bit is clear
    __device__ __forceinline__ Tally() {
        const uint32_t lane = threadIdx.x & 31u;
        n0 = (lane & 1u) - 1u;
        n1 = ((lane >> 1) & 1u) - 1u;
        n2 = ((lane >> 2) & 1u) - 1u;
    }
    __device__ __forceinline__ void add(bool valid, uint32_t bin) {
        const uint32_t v = valid ? bin : 7u;
        const uint32_t b0 = __ballot_sync(0xFFFFFFFFu, v & 1u), b1 = __ballot_sync(0xFFFFFFFFu, v & 2u),
                       b2 = __ballot_sync(0xFFFFFFFFu, v & 4u);
        n += (uint32_t)__popc((b0 ^ n0) & (b1 ^ n1) & (b2 ^ n2));
    }
    // all valid lanes in bin 0
    __device__ __forceinline__ void add_susceptible(bool valid) {
        n += (uint32_t)__popc(__ballot_sync(0xFFFFFFFFu, valid)) & n0 & n1 & n2;
    }
    __device__ __forceinline__ void flush(uint32_t* sh) {
        if ((threadIdx.x & 31u) < 6u && n) atomicAdd(&sh[threadIdx.x & 31u], n);
        n = 0;
    }
};

// Consecutive chunks a block takes per grid-stride step.  A single world takes 1: the plain
// stride, where the resident blocks sweep one contiguous band of agents, was measured fastest
// (groups of 2, 4, 8 were 2, 8, 15 % slower, a scattered chunk order 6 % slower).  An ensemble
// block that strides one chunk at a time switches replicate at nearly every step (a parameter
// reload and a histogram flush), so it takes groups of `size`; inverse = ceil(2^32 / size).
struct ChunkGroup {
    uint32_t size, inverse;
};

// Block-uniform bookkeeping of the replicate a block is working on.
struct BlockRep {
    uint32_t r = 0xFFFFFFFFu;
};

// Hours run in chains of captured pieces (a piece ends at a day boundary) launched back to
// back; the chain's counts rows are [hour - first][replicate][8], words 0-5 the bins and
// word 6 the halt mark of the run loop's guard.  The hour of a launch is read on the device,
// so one captured piece serves every day.
struct SegDev {
    uint32_t hour_base;  // first hour of the piece now running (advanced by k_piece_end)
    uint32_t first;      // first hour of the chain
};
struct HourArgs {
    SegDev* seg;
    uint32_t* counts;    // the chain's rows
    uint32_t row_words;  // R * 8
    uint32_t offset;     // hour within the piece
    uint32_t prev_back;  // hours back to the previous computed row (0: the stop rule is off)
};
// The hour of a launch and its row in the chain.  The row pointers are recomputed where they
// are used (from kernel parameters) rather than held in registers across the kernel.
struct HourRow {
    uint32_t hour, row;
};
__device__ __forceinline__ HourRow hour_row(const HourArgs& a) {
    const uint32_t hour = a.seg->hour_base + a.offset;
    return HourRow{hour, hour - a.seg->first};
}
__device__ __forceinline__ uint32_t* row_ptr(const HourArgs& a, uint32_t row) {
    return a.counts + (size_t)row * a.row_words;
}
// The previous computed row: nullptr for the first hour of a chain and outside the run loop.
__device__ __forceinline__ const uint32_t* prev_ptr(const HourArgs& a, uint32_t row) {
    return (a.prev_back && row >= a.prev_back) ? a.counts + (size_t)(row - a.prev_back) * a.row_words : nullptr;
}

// The stop rule of run_single_engine (epidemiology_simulation.rs:564-575): a replicate whose
// last computed counts row (prev, [replicate][8]) has no exposed, infected or hospitalized
// agent has ended, and the later hours of the chain leave it untouched; so do they after a
// row the guard marked (an intervention fires there, and the host takes over).
__device__ __forceinline__ bool run_ended(const uint32_t* prev, uint32_t r) {
    if (!prev) return false;
    const uint32_t* c = prev + (size_t)r * 8u;
    return (c[1] | c[2] | c[3]) == 0u || c[6] != 0u;
}

// Switch the block to replicate r: flush the histogram of the previous one into its counts
// row (counts[r * 8 + bin]), stage r's parameters, clear the histogram.  Block-uniform.
__device__ __forceinline__ void switch_rep(BlockRep& br, uint32_t r, const DevParams* __restrict__ Pall, DevParams& sP,
                                           Tally& tally, uint32_t* sh, uint32_t* counts, Box* boxes = nullptr) {
    if (br.r != 0xFFFFFFFFu) tally.flush(sh);
    __syncthreads();
    if (br.r != 0xFFFFFFFFu && threadIdx.x < 6 && sh[threadIdx.x]) atomicAdd(&counts[br.r * 8 + threadIdx.x], sh[threadIdx.x]);
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < sizeof(DevParams) / 4; k += blockDim.x)
        reinterpret_cast<uint32_t*>(&sP)[k] = reinterpret_cast<const uint32_t*>(Pall + r)[k];
    if (threadIdx.x < 8) sh[threadIdx.x] = 0;
    if (boxes) stage_boxes(boxes, Pall[r]);
    __syncthreads();
    br.r = r;
}

__device__ __forceinline__ void flush_rep(const BlockRep& br, Tally& tally, uint32_t* sh, uint32_t* counts) {
    if (br.r != 0xFFFFFFFFu) tally.flush(sh);
    __syncthreads();
    if (br.r != 0xFFFFFFFFu && threadIdx.x < 6 && sh[threadIdx.x]) atomicAdd(&counts[br.r * 8 + threadIdx.x], sh[threadIdx.x]);
}

// First vacant hospital cell of the snapshot in AreaIterator order (area.rs:131-148), found
// by the whole block; kNoAction when the hospital is full.
template <class V>
__device__ uint32_t block_first_vacant(const DevParams& P, const V& pl) {
    __shared__ uint32_t best;
    const Rect h = P.area[P.hosp_code];
    const uint32_t w = (uint32_t)(h.x1 - h.x0 + 1), total = w * (uint32_t)(h.y1 - h.y0 + 1);
    if (threadIdx.x == 0) best = kNoAction;
    __syncthreads();
    for (uint32_t base = 0; base < total; base += blockDim.x) {
        const uint32_t c = base + threadIdx.x;
        bool vac = false;
        if (c < total) vac = pl.vacant(h.x0 + (int32_t)(c % w), h.y0 + (int32_t)(c / w));
        if (vac) atomicMin(&best, c);
        if (__syncthreads_or(vac)) break;
    }
    const uint32_t c = best;
    __syncthreads();
    if (c == kNoAction) return kNoAction;
    return pack_xy(h.x0 + (int32_t)(c % w), h.y0 + (int32_t)(c / w));
}

// Hours 1..6 (SLEEP_START_TIME..=SLEEP_END_TIME, citizen/mod.rs:244-248).  A single world
// takes its chunks kSleepBatch at a time with all their state loads in flight together (the
// kernel is one load and a compare per agent, so one load round per chunk set its time).
constexpr uint32_t kSleepBatch = 4;

__device__ __forceinline__ void sleep_agent(uint2* __restrict__ st, uint32_t slot, bool valid, uint32_t s, Tally& tally) {
    if (valid && st_ws(s) != EPI_WS_HOSPITAL_STAFF && st_area(s) != kHome) st[slot].x = with_area(s, kHome);
    tally.add(valid, count_bin(s));
}

__global__ void __launch_bounds__(kThreads) k_sleep(const DevParams* __restrict__ Pall, const uint32_t* __restrict__ chunk_rep,
                                                    uint32_t n_chunks, uint32_t grp, uint2* __restrict__ st, HourArgs ha) {
    __shared__ uint32_t sh[8];
    __shared__ DevParams sP;
    dep_wait();
    const HourRow hr = hour_row(ha);
    BlockRep br;
    Tally tally;
    bool ended = false;  // run_ended of the block's replicate (its prev row is fixed during the launch)
    if (!chunk_rep) {
        if (blockIdx.x < n_chunks) {
            switch_rep(br, 0u, Pall, sP, tally, sh, row_ptr(ha, hr.row));
            ended = run_ended(prev_ptr(ha, hr.row), 0u);
        }
        if (blockIdx.x < n_chunks && sP.active && !ended) {
            for (uint32_t c0 = blockIdx.x; c0 < n_chunks; c0 += kSleepBatch * gridDim.x) {
                uint32_t sv[kSleepBatch];
#pragma unroll
                for (uint32_t q = 0; q < kSleepBatch; ++q) {
                    const uint32_t c = c0 + q * gridDim.x, slot = c * kChunk + threadIdx.x;
                    sv[q] = (c < n_chunks && slot < sP.n) ? st[slot].x : 0u;  // slot = agent (agent_off 0)
                }
#pragma unroll
                for (uint32_t q = 0; q < kSleepBatch; ++q) {
                    const uint32_t c = c0 + q * gridDim.x, slot = c * kChunk + threadIdx.x;
                    if (c >= n_chunks) break;  // block-uniform
                    sleep_agent(st, slot, slot < sP.n, sv[q], tally);
                }
            }
        }
        flush_rep(br, tally, sh, row_ptr(ha, hr.row));
        return;
    }
    for (uint32_t c = blockIdx.x * grp, k = 0; c < n_chunks;
         c = (++k < grp) ? c + 1u : c + (gridDim.x - 1u) * grp + 1u, k = (k < grp) ? k : 0u) {
        const uint32_t r = chunk_rep ? chunk_rep[c] : 0u;
        if (r != br.r) {
            switch_rep(br, r, Pall, sP, tally, sh, row_ptr(ha, hr.row));
            ended = run_ended(prev_ptr(ha, hr.row), r);
        }
        if (!sP.active || ended) continue;
        const uint32_t slot = c * kChunk + threadIdx.x;
        const bool valid = slot - sP.agent_off < sP.n;
        sleep_agent(st, slot, valid, valid ? st[slot].x : 0u, tally);
    }
    flush_rep(br, tally, sh, row_ptr(ha, hr.row));
}

// ---------------------------------------------------------------- the hour's two kernels
// Claims.  A mover claims its target with an atomicMin of claim_key (lowest index of the hour
// wins) on the cell's claim word, and the value it finds names the claimant it competes with:
// of the two the higher index has lost.  Every claimant but the cell's lowest is named so
// exactly once -- by itself, which then simply stays, or by the one that displaces it, which
// puts it on its warp's list.  The hour's blocks sweep the agents in index order, so most
// losers find a lower index before them and few are ever displaced: k_commit, which sends the
// listed ones back, has a short list (1.3 % of the agents in office hours, 0.04 % at home)
// where a pass over all agents would settle every move.  One GB300, 1M agents on a 2,500 grid:
// k_commit 5 us per waking hour in a launch list, against 9 us for a pass over target words,
// loss marks and byte-plane stores; 4M agents 5.2 us against 26 us.
//
// The occupancy of the next hour is a bit plane that starts the hour all zero: the first
// claimant of a cell sets the target's bit, an agent that stays or lost sets its own cell's.
//
// Positions have two buffers as well.  In the hours of day 7..22 every agent writes its
// proposal to the other one, so the old cell of a claimant that lost is at hand; at hours 0
// and 23 (PATCH), where few agents act, the current buffer and bit plane are patched in place
// and the agents that act leave their old position in the other buffer.
//
// A warp's lists lie over the slots of its own chunks, in the order the warp takes them: entry
// e of a warp is at the slot of lane e % 32 in the warp's (e / 32)-th chunk.
struct HourLists {
    uint32_t* displaced;  // slots of claimants that a lower index has displaced
    uint2* acts;          // {slot, target word}: infectious agents that move or change class (PATCH: every mover too)
    uint2* n;             // per warp: entries of the two lists
};

// The k-th chunk of this block: plain stride for a single world, groups for an ensemble.
template <bool ENS>
__device__ __forceinline__ uint32_t chunk_at(ChunkGroup g, uint32_t k) {
    if (!ENS) return blockIdx.x + k * gridDim.x;
    const uint32_t q = g.size > 1u ? __umulhi(k, g.inverse) : k;  // k / size (k < 2^28)
    return (q * gridDim.x + blockIdx.x) * g.size + (k - q * g.size);
}
template <bool ENS>
__device__ __forceinline__ uint32_t list_slot(ChunkGroup g, uint32_t e) {
    return chunk_at<ENS>(g, e >> 5) * kChunk + (threadIdx.x & ~31u) + (e & 31u);
}
// Append the entries of the lanes with f set to the warp's list (whole warps; n is uniform).
template <bool ENS, class T>
__device__ __forceinline__ void list_append(ChunkGroup g, T* list, uint32_t& n, bool f, const T& v) {
    const uint32_t m = __ballot_sync(0xFFFFFFFFu, f);
    if (f) list[list_slot<ENS>(g, n + (uint32_t)__popc(m & ((1u << (threadIdx.x & 31u)) - 1u)))] = v;
    n += (uint32_t)__popc(m);
}

// What one agent's hour leaves to its warp: the counts bin and the list entries.
struct AgentHour {
    uint32_t bin = 0;
    uint32_t target = 0;
    uint32_t loser = 0;  // slot this agent displaced
    bool displaces = false, act = false;
};

// The rules of one agent for the hour: proposal, claim, infection update, state and position
// words.  next is the replicate's zeroed bit plane, pos_next the other position buffer.
template <int HC, bool PATCH>
__device__ __forceinline__ AgentHour decide_agent(const DevParams& P, const BitView<>& pl, const MoveTables& tables,
                                                  const Box* boxes, uint32_t* __restrict__ next,
                                                  uint32_t* __restrict__ rclaim, uint32_t* __restrict__ wsa,
                                                  uint2* __restrict__ st, uint32_t* pos, uint32_t* pos_next, uint32_t slot,
                                                  uint32_t i, uint32_t s, uint32_t at, uint32_t p, uint32_t hm, uint32_t wk,
                                                  uint32_t hour, uint32_t hosp_first) {
    const uint32_t s0 = s, at0 = at;
    Draws dr{i, hour, P.key0, P.key1, P.move_key};
    uint32_t q;  // the proposal: the agent's cell, a vacant cell or a valid neighbour, so inside the plane
    bool infect = false;
    if (HC == kHcStart) q = routine_start(P, pl, s, hm, p, hosp_first, dr);
    else if (HC == kHcEnd) q = routine_end(P, pl, s, hm, p, dr);
    else q = perform_movements<HC>(P, pl, tables, boxes, s, wsa + slot, hm, wk, p, hour, dr, infect);
    // The claim goes out before the infection update so that its round trip overlaps it.
    AgentHour out;
    const uint32_t key = claim_key(hour, i), wanted = q;
    const uint32_t found = q != p ? atomicMin(&rclaim[(q >> 16) * (uint32_t)P.W + (q & 0xFFFFu)], key) : kNoClaim;
    if (infect) infection_dynamics(P, pl, tables, boxes, s, at, hm, wk, wanted, hour, dr);
    // (an untouched word looks like a key of the window's first hour, but for its index)
    if (found != kNoClaim && (found >> kClaimAgentBits) == (key >> kClaimAgentBits)) {
        const uint32_t j = found & kMaxAgentsPerWorld;
        out.displaces = j > i;
        out.loser = P.agent_off + j;
        if (j < i) q = p;
    }
    const bool moving = q != p;
    if (!PATCH) {
        if (!out.displaces) {
            const uint32_t X = (q & 0xFFFFu) + 1u;
            atomicOr(&next[((q >> 16) + 1u) * P.PW + (X >> 5)], 1u << (X & 31u));
        }
        pos_next[slot] = q;
    }
    out.bin = count_bin(s);
    if (out.bin != 0u) {  // not susceptible: infectious, perhaps, before or after
        if (infected(s0) || infected(s)) {  // the planes follow its class (a healthy agent's is 1 throughout)
            const uint32_t cls0 = cell_class(P, s0), cls = cell_class(P, s);
            out.act = (cls0 >= 2u || cls >= 2u) && (moving || cls != cls0);
            out.target = encode_target(q, cls, cls0);
        }
    }
    if (PATCH && moving && !out.act) {
        out.act = true;
        out.target = encode_target(q, 1u, 1u);
    }
    if (PATCH && out.act) {
        pos_next[slot] = p;
        if (moving) pos[slot] = q;
    }
    if (s != s0 || at != at0) st[slot] = make_uint2(s, at);
    return out;
}

// One hour of per-agent rules (hour of day 0, 7..22 or 23), specialised per hour class HC,
// over one world (ENS false: slot = agent, the parameters staged once) or the chunks of many
// replicates (ENS true: chunk_rep names each chunk's replicate).  The body is shared by two
// kernels that differ in their launch bounds: k_decide for a single world (5 resident blocks,
// 48 registers) and k_decide_ens for ensembles (6 blocks, 40 registers), whose per-chunk
// replicate switches favour occupancy.  Every hour class has the same bound because one grid,
// the resident one, serves them all: left to the compiler the mixed hours took 54 registers,
// ran the 760-block grid in two waves and cost a run a quarter more.  (One GB300, two weeks of
// hours: 1M agents 5.39 ms at 5 blocks, 5.43 at 6, 6.08 at 7; 4M agents 5.83, 5.69, 6.15; the
// 256-replicate ensemble 49.9 at 4 blocks, 48.0 at 5, 47.1 at 6, 60.1 at 8.)
//
// What bounds it: dependent latency with issue behind it.  Walking agents cost about 350 warp
// instructions per 32 and three dependent L2 round trips (words, the rows around the cell, the
// claim); 48 % of the issue slots are busy (1M agents cold, 5 blocks per SM).
constexpr int kWorldMinBlocks = 5;
constexpr int kEnsembleMinBlocks = 6;

// The arrays of an hour's launch (see the claims above).
struct HourBuffers {
    uint32_t* pos;        // positions before the hour
    uint32_t* pos_next;   // the other buffer
    uint2* st;
    const uint32_t *home, *work;
    uint32_t* wsa;
    uint32_t* occ;        // occupancy before the hour
    uint32_t* occ_next;   // the other buffer, all zero
    uint8_t *cls, *danger;
    uint32_t* claim;
    HourLists lists;
    ChunkGroup group;
    int* err;
};

template <int HC, bool ENS>
__device__ __forceinline__ void decide_body(const DevParams* __restrict__ Pall, const uint32_t* __restrict__ chunk_rep,
                                            uint32_t n_chunks, const HourBuffers& B, const HourArgs& ha) {
    constexpr bool PATCH = HC == kHcStart || HC == kHcEnd;
    __shared__ uint32_t sh[8];
    __shared__ DevParams sP;
    __shared__ MoveTables tables;
    __shared__ Box boxes[kNumAreas];
    const DevParams& P = sP;
    if (!PATCH) stage_tables(tables);  // read after switch_rep's barriers
    dep_wait();
    const HourRow hr = hour_row(ha);
    const uint32_t hour = hr.hour;
    BlockRep br;
    Tally tally;
    uint32_t hosp_first = kNoAction, n_displaced = 0u, n_acts = 0u;
    bool hosp_known = false;
    if (!ENS) {
        if (blockIdx.x < n_chunks) switch_rep(br, 0u, Pall, sP, tally, sh, row_ptr(ha, hr.row), boxes);
        if (blockIdx.x < n_chunks && P.active && !run_ended(prev_ptr(ha, hr.row), 0u)) {
            const BitView<> pl{B.occ, B.cls, B.danger, P.G, P.WP, P.PW, B.err};
            const uint32_t n = P.n;
            for (uint32_t c = blockIdx.x; c < n_chunks; c += gridDim.x) {
                const uint32_t slot = c * kChunk + threadIdx.x;  // = agent index (a lone world starts at slot 0)
                const bool valid = slot < n;
                uint32_t s = 0, at = 0, p = 0;
                if (valid) {
                    const uint2 sv = B.st[slot];
                    s = sv.x;
                    at = sv.y;
                    p = B.pos[slot];
                }
                if (HC == kHcStart) {
                    const bool need = valid && wants_hospital(P, infected(s) ? with_day(s, st_day(s) + 1u) : s);
                    if (__syncthreads_or(need) && !hosp_known) {
                        hosp_first = block_first_vacant(P, pl);
                        hosp_known = true;
                    }
                }
                AgentHour a;
                if (valid)
                    a = decide_agent<HC, PATCH>(P, pl, tables, boxes, B.occ_next, B.claim, B.wsa, B.st, B.pos, B.pos_next, slot, slot, s, at, p,
                                                B.home[slot], B.work[slot], hour, hosp_first);
                // most warps of a young epidemic: all susceptible, no one displaced
                if (!__any_sync(0xFFFFFFFFu, a.bin != 0u || a.displaces || a.act)) {
                    tally.add_susceptible(valid);
                } else {
                    tally.add(valid, a.bin);
                    list_append<ENS>(B.group, B.lists.displaced, n_displaced, a.displaces, a.loser);
                    list_append<ENS>(B.group, B.lists.acts, n_acts, a.act, make_uint2(slot, a.target));
                }
            }
        }
    } else {
        bool ended = false;
        // The replicate of the next chunk is read one chunk ahead, and a chunk's agent words are
        // read before its replicate is known (every chunk of an ensemble is whole in the slot
        // arrays), so neither waits on the other.
        uint32_t c = blockIdx.x * B.group.size, left = B.group.size;
        uint32_t r_next = c < n_chunks ? chunk_rep[c] : 0u;
        while (c < n_chunks) {
            const uint32_t r = r_next;
            const uint32_t slot = c * kChunk + threadIdx.x;
            ++c;
            if (--left == 0u) {  // the block's next group
                c += (gridDim.x - 1u) * B.group.size;
                left = B.group.size;
            }
            r_next = c < n_chunks ? chunk_rep[c] : 0u;
            const uint2 sv = B.st[slot];
            const uint32_t pw = B.pos[slot], hw = B.home[slot], ww = B.work[slot];
            if (r != br.r) {
                switch_rep(br, r, Pall, sP, tally, sh, row_ptr(ha, hr.row), boxes);
                hosp_known = false;
                ended = run_ended(prev_ptr(ha, hr.row), r);  // an earlier row: fixed during the launch
            }
            if (!P.active || ended) continue;
            const BitView<> pl{B.occ + P.occ_off, B.cls + P.plane_off, B.danger + P.plane_off, P.G, P.WP, P.PW, B.err};
            const uint32_t i = slot - P.agent_off;  // index within the replicate
            const bool valid = i < P.n;
            const uint32_t s = valid ? sv.x : 0u, at = valid ? sv.y : 0u, p = valid ? pw : 0u;
            if (HC == kHcStart) {
                const bool need = valid && wants_hospital(P, infected(s) ? with_day(s, st_day(s) + 1u) : s);
                if (__syncthreads_or(need) && !hosp_known) {
                    hosp_first = block_first_vacant(P, pl);
                    hosp_known = true;
                }
            }
            AgentHour a;
            if (valid)
                a = decide_agent<HC, PATCH>(P, pl, tables, boxes, B.occ_next + P.occ_off, B.claim + P.claim_off, B.wsa, B.st, B.pos,
                                            B.pos_next, slot, i, s, at, p, hw, ww, hour, hosp_first);
            if (!__any_sync(0xFFFFFFFFu, a.bin != 0u || a.displaces || a.act)) {
                tally.add_susceptible(valid);
            } else {
                tally.add(valid, a.bin);
                list_append<ENS>(B.group, B.lists.displaced, n_displaced, a.displaces, a.loser);
                list_append<ENS>(B.group, B.lists.acts, n_acts, a.act, make_uint2(slot, a.target));
            }
        }
    }
    flush_rep(br, tally, sh, row_ptr(ha, hr.row));
    if ((threadIdx.x & 31u) == 0u) B.lists.n[(blockIdx.x * kThreads + threadIdx.x) >> 5] = make_uint2(n_displaced, n_acts);
}

template <int HC>
__global__ void __launch_bounds__(kThreads, kWorldMinBlocks) k_decide(const DevParams* __restrict__ Pall, const uint32_t* __restrict__ chunk_rep,
                                                     uint32_t n_chunks, const __grid_constant__ HourBuffers B, HourArgs ha) {
    decide_body<HC, false>(Pall, chunk_rep, n_chunks, B, ha);
}
template <int HC>
__global__ void __launch_bounds__(kThreads, kEnsembleMinBlocks)
    k_decide_ens(const DevParams* __restrict__ Pall, const uint32_t* __restrict__ chunk_rep, uint32_t n_chunks,
                 const __grid_constant__ HourBuffers B, HourArgs ha) {
    decide_body<HC, true>(Pall, chunk_rep, n_chunks, B, ha);
}

// A claimant that lost (slot of replicate P): back to its old cell.  dest holds its proposal,
// old its position before the hour; occ is the plane of the hour's end.
template <bool PATCH>
__device__ __forceinline__ void send_back(const DevParams& P, uint32_t slot, const uint2* __restrict__ st,
                                          uint32_t* dest, const uint32_t* old, uint32_t* occ, uint8_t* cls_plane,
                                          uint8_t* danger) {
    const uint32_t o = old[slot], s = st[slot].x, proposal = dest[slot];
    // The position is changed by an atomic too: a plain store beside the atomic below made the
    // launch wait 3.3 us (10,000 agents) to 5.6 us (1M agents, office hours) for its stores to
    // drain at the end, whatever its cache operator.
    atomicXor(&dest[slot], o ^ proposal);
    const uint32_t X = (uint32_t)unpack_x(o) + 1u, w = ((uint32_t)unpack_y(o) + 1u) * P.PW + (X >> 5);
    // PATCH: its entry in acts flips the bit too, so that two flips leave it set in either order
    if (PATCH) atomicXor(&occ[w], 1u << (X & 31u));
    else atomicOr(&occ[w], 1u << (X & 31u));
    const uint32_t cls = cell_class(P, s);
    if (cls >= 2u) {
        class_add(cls_plane, danger, (uint32_t)P.WP, proposal, cls, true);
        class_add(cls_plane, danger, (uint32_t)P.WP, o, cls, false);
    }
}

// Completes the hour (the serial resolve of allocation_map.rs:93-102 in index order) from the
// lists of k_decide, launched with the same grid: a warp takes its own lists.  Everything it
// does to one word adds up or is idempotent, so the order of entries does not matter.  Not
// PATCH: the planes and positions read this hour become the next hour's other buffers, so the
// spent bit plane is zeroed (pieces of kPieceWords words; piece_rep names a piece's replicate
// in an ensemble, where a replicate whose run has ended keeps its plane).
constexpr uint32_t kPieceWords = 512;

template <bool ENS, bool PATCH>
__global__ void __launch_bounds__(kThreads) k_commit(const DevParams* __restrict__ Pall, const uint32_t* __restrict__ chunk_rep,
                                                     uint32_t n_pieces, const uint32_t* __restrict__ piece_rep,
                                                     const __grid_constant__ HourBuffers B, HourArgs ha, uint64_t claim_cells) {
    dep_wait();
    const HourRow hr = hour_row(ha);
    const uint32_t lane = threadIdx.x & 31u;
    const uint2 n = B.lists.n[(blockIdx.x * kThreads + threadIdx.x) >> 5];
    uint32_t* dest = PATCH ? B.pos : B.pos_next;
    const uint32_t* old = PATCH ? B.pos_next : B.pos;
    uint32_t* occ = PATCH ? B.occ : B.occ_next;
    for (uint32_t e = lane; e < n.x; e += 32u) {
        const uint32_t slot = B.lists.displaced[list_slot<ENS>(B.group, e)];
        const DevParams& P = Pall[ENS ? chunk_rep[slot / kChunk] : 0u];
        send_back<PATCH>(P, slot, B.st, dest, old, occ + P.occ_off, B.cls + P.plane_off, B.danger + P.plane_off);
    }
    for (uint32_t e = lane; e < n.y; e += 32u) {
        const uint2 a = B.lists.acts[list_slot<ENS>(B.group, e)];
        const DevParams& P = Pall[ENS ? chunk_rep[a.x / kChunk] : 0u];
        const uint32_t o = old[a.x], t = target_xy(a.y), cls = target_class(a.y), cls0 = target_old_class(a.y);
        uint8_t *cp = B.cls + P.plane_off, *dg = B.danger + P.plane_off;
        if (cls0 >= 2u) class_add(cp, dg, (uint32_t)P.WP, o, cls0, true);
        if (cls >= 2u) class_add(cp, dg, (uint32_t)P.WP, t, cls, false);
        if (PATCH && t != o) {
            const uint32_t Xo = (uint32_t)unpack_x(o) + 1u, X = (uint32_t)unpack_x(t) + 1u;
            const uint32_t w = ((uint32_t)unpack_y(t) + 1u) * P.PW + (X >> 5);
            uint32_t* ro = occ + P.occ_off;
            atomicXor(&ro[((uint32_t)unpack_y(o) + 1u) * P.PW + (Xo >> 5)], 1u << (Xo & 31u));
            atomicOr(&ro[w], 1u << (X & 31u));
        }
    }
    if (!PATCH) {
        const uint32_t* prev = prev_ptr(ha, hr.row);
        const uint32_t per = kPieceWords / 4u;  // 16-byte words
        const uint32_t stride = gridDim.x * (kThreads / per);
        if (ENS || (Pall[0].active && !run_ended(prev, 0u)))
            for (uint32_t q = blockIdx.x * (kThreads / per) + threadIdx.x / per; q < n_pieces; q += stride) {
                if (ENS) {
                    const uint32_t r = piece_rep[q];
                    if (!Pall[r].active || run_ended(prev, r)) continue;
                }
                reinterpret_cast<uint4*>(B.occ)[(size_t)q * per + threadIdx.x % per] = make_uint4(0u, 0u, 0u, 0u);
            }
    }
    // A new claim window (kClaimWindow hours) opens before the next hour that claims (hour of
    // day 0 claims next at 7): every claim word is reset for it.
    const uint32_t next = hr.hour % 24u == 0u ? hr.hour + 7u : hr.hour + 1u;
    if (next / kClaimWindow != hr.hour / kClaimWindow)
        for (size_t i = (size_t)blockIdx.x * kThreads + threadIdx.x; i < claim_cells; i += (size_t)gridDim.x * kThreads)
            B.claim[i] = kNoClaim;
}

// ---------------------------------------------------------------- small worlds
// An hour of a world of a few thousand agents is launches and latency: two launches of at most
// 64 blocks, each a chain of dependent L2 round trips.  k_small runs all hours of a call in one
// launch: an agent per thread, its words in registers from hour to hour, and two barriers per
// hour where the launches were.
//   before the first   proposals, an atomicMin of the agent's claim key on the target's claim
//                      word, infection update, the block's counts added to the world's
//   between them       a mover reads its claim word back: it holds its key (it moves) or a lower
//                      index's (it stays); occupancy bits and class planes are written, the
//                      spent bit plane zeroed
// The stop rule and the run loop's guard are read from the world's counts by every thread, and
// the rows go to the caller (pinned host memory) from the first block.  Two forms:
//   GRID false  one cluster of 16 CTAs, hardware barriers, counts in the first CTA's shared
//               memory: up to 16,384 agents.  Two weeks of hours on one GB300, captured
//               launches / cluster: 2,000 agents 1.53 / 0.84 ms, 10,000 1.62 / 1.16, 16,000
//               1.63 / 1.48.  An hour of the 10,000's spends 1.7 of its 4.6 us in the barriers
//               and the atomics they wait for, 1.6 in proposals.
//   GRID true   a cooperative grid of one CTA per SM, barriers at L2: up to 155,648 agents.
//               96 hours of 30,000 / 98,000 agents, ms: hour by hour 3.8 / 3.8 by captured
//               launches, 1.9 / 2.0 here; six hours a call 1.01 / 1.05 and 0.66 / 0.77; in one
//               call 0.49 / 0.53 and 0.44 / 0.55 (the rule of use: longest_together).  Its counts
//               lie a cache line per bin apart: side by side, 152 blocks' atomics on one sector
//               held every barrier up (98,000 agents, a day's mean hour 7.4 us, 6.0 apart).
constexpr uint32_t kSmallCluster = 16;
constexpr uint32_t kSmallThreads = 1024;
constexpr uint32_t kSmallAgents = kSmallCluster * kSmallThreads;  // most agents of a world run so

struct SmallArgs {
    uint32_t* pos;        // the buffer that holds the positions before the first hour
    uint32_t* pos_buf[2];
    uint32_t* occ_buf[2];
    uint2* st;
    const uint32_t *home, *work;
    uint32_t* wsa;
    uint8_t *cls, *danger;
    uint32_t* claim;      // no keys but earlier hours' of the first hour's window
    uint32_t claim_cells;
    uint32_t occ_words;
    uint32_t first, hours;
    uint32_t run_loop;    // 1: the stop rule and the guard apply
    uint32_t* ivn;        // the guard's new-infections figure
    uint32_t* sums;       // k_small<true>: zero, kGridWords: 3 x 8 sums of an hour's counts and the barrier's
                          // arrivals, a cache line each
    uint32_t* rows;       // hours x 8: bins, word 6 the halt mark; rows that did not run are zero
    uint32_t polls;       // k_small<true>: of a barrier before its block gives up
    int* err;             // device error word
    int* err_out;         // where the caller reads it: [0] what the first block finds there at its end, [1] kErrWait
                          // from a block that gave up (a word of its own, so that neither undoes the other)
};
constexpr int kErrWait = 4;  // the error word: a wait for the other blocks ran out

// The hours of day 7..22 write the other buffer, 16 a day (engine.cu: hour_parity).
__host__ __device__ constexpr uint32_t hour_parity(uint32_t hod) {
    return (hod >= 7u ? (hod < 22u ? hod : 22u) - 6u : 0u) & 1u;
}

__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
// The shared-memory address of p in the cluster's first CTA.
__device__ __forceinline__ uint32_t in_first_cta(const void* p) {
    uint32_t a;
    asm("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(a) : "r"((uint32_t)__cvta_generic_to_shared(p)));
    return a;
}
__device__ __forceinline__ void add_in_cluster(uint32_t addr, uint32_t v) {
    asm volatile("red.relaxed.cluster.shared::cluster.add.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ uint32_t load_in_cluster(uint32_t addr) {
    uint32_t v;
    asm volatile("ld.relaxed.cluster.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
    return v;
}

// The barrier of a grid whose blocks all run (a cooperative launch): false, on every thread of
// the block, when the others did not arrive within `polls` (kGridSpinLimit: some seconds).
constexpr uint32_t kLineWords = 32, kGridWords = 25 * kLineWords;
constexpr uint32_t kGridSpinLimit = 1u << 22;
__device__ __forceinline__ bool grid_sync(uint32_t* arrived, uint32_t& target, uint32_t polls) {
    target += gridDim.x;
    bool ok = true;
    __syncthreads();
    if (threadIdx.x == 0) {
        asm volatile("fence.acq_rel.gpu;\n\tred.release.gpu.global.add.u32 [%0], 1;" ::"l"(arrived) : "memory");
        ok = false;
        for (uint32_t it = 0; it < polls && !ok; ++it) {
            uint32_t v;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(arrived) : "memory");
            ok = (int32_t)(v - target) >= 0;
        }
        asm volatile("fence.acq_rel.gpu;" ::: "memory");
    }
    return !__syncthreads_or(!ok);
}

template <bool GRID>
__global__ void __launch_bounds__(kSmallThreads, 1) k_small(const DevParams* __restrict__ Pall, const __grid_constant__ SmallArgs a) {
    __shared__ uint32_t sh[8];
    __shared__ uint32_t total[3][8];  // the first CTA's are the cluster's
    __shared__ DevParams sP;
    __shared__ MoveTables tables;
    __shared__ Box boxes[kNumAreas];
    const DevParams& P = sP;
    const uint32_t rank = blockIdx.x, tid = threadIdx.x, i = rank * blockDim.x + tid;
    stage_tables(tables);
    stage_boxes(boxes, Pall[0]);
    for (uint32_t k = tid; k < sizeof(DevParams) / 4; k += blockDim.x)
        reinterpret_cast<uint32_t*>(&sP)[k] = reinterpret_cast<const uint32_t*>(Pall)[k];
    if (tid < 8) sh[tid] = total[0][tid] = total[1][tid] = total[2][tid] = 0u;
    if (GRID) __syncthreads();
    else cluster_sync();  // every CTA of the cluster runs, and its counters are clear
    const uint32_t sums = GRID ? 0u : in_first_cta(&total[0][0]);
    uint32_t arrivals = 0u;  // GRID: of all blocks at all barriers so far
    bool ok = true;
    // the counts of the hour, from a block's sums to the world's
    auto add_counts = [&](uint32_t slot) {
        if (tid < 6u) {
            if (!sh[tid]) return;
            if (GRID) atomicAdd(&a.sums[(slot * 8u + tid) * kLineWords], sh[tid]);
            else add_in_cluster(sums + (slot * 8u + tid) * 4u, sh[tid]);
            sh[tid] = 0u;
        }
    };
    auto count_of = [&](uint32_t slot, uint32_t bin) {
        return GRID ? __ldcg(&a.sums[(slot * 8u + bin) * kLineWords]) : load_in_cluster(sums + (slot * 8u + bin) * 4u);
    };
    auto sync = [&] {
        if (GRID) ok = grid_sync(a.sums + 24u * kLineWords, arrivals, a.polls) && ok;
        else cluster_sync();
    };
    const bool valid = i < P.n;
    uint32_t s = 0u, at = 0u, p = 0u, hm = 0u, wk = 0u;
    if (valid) {
        const uint2 sv = a.st[i];
        s = sv.x;
        at = sv.y;
        p = a.pos[i];
        hm = a.home[i];
        wk = a.work[i];
    }
    uint32_t ivn = a.run_loop ? *a.ivn : 0u;
    uint32_t slot = 0u;        // of total: the hour running
    uint32_t last = a.first;   // the last hour that ran
    uint32_t written = 0u;     // rows written by the first CTA
    uint32_t window = a.first / kClaimWindow;  // of the claim plane's keys
    bool over = !P.active;
    for (uint32_t k = 0; k < a.hours && !over && ok; ++k) {
        const uint32_t hour = a.first + k, hod = hour % 24u;
        if (k > 0 && hod >= 2u && hod <= 6u) {  // hour 1 has sent everyone home: nothing changes
            if (rank == 0 && tid < 8) a.rows[(size_t)k * 8u + tid] = 0u;
            written = k + 1u;
            last = hour;
            continue;
        }
        Tally tally;
        const uint32_t s0 = s;
        uint32_t e, inf, hos;
        if (hod >= 1u && hod <= 6u) {
            if (valid && st_ws(s) != EPI_WS_HOSPITAL_STAFF) s = with_area(s, kHome);
            tally.add(valid, count_bin(s));
            tally.flush(sh);
            __syncthreads();
            add_counts(slot);
            sync();
            e = count_of(slot, 1u), inf = count_of(slot, 2u), hos = count_of(slot, 3u);
        } else {
            const bool patch = hod == 0u || hod == 23u;
            if (hour / kClaimWindow != window) {
                for (uint32_t c = i; c < a.claim_cells; c += gridDim.x * blockDim.x) a.claim[c] = kNoClaim;
                window = hour / kClaimWindow;
                sync();
            }
            uint32_t* occ = a.occ_buf[hour_parity((hod + 23u) % 24u)];
            uint32_t* next = a.occ_buf[hour_parity(hod)];
            const BitView<true> pl{occ, a.cls, a.danger, P.G, P.WP, P.PW, a.err};
            uint32_t nc = p;
            Draws dr{i, hour, P.key0, P.key1, P.move_key};
            bool infect = false;
            if (hod == 0u) {
                const bool need = valid && wants_hospital(P, infected(s) ? with_day(s, st_day(s) + 1u) : s);
                const uint32_t hosp_first = __syncthreads_or(need) ? block_first_vacant(P, pl) : kNoAction;
                if (valid) nc = routine_start(P, pl, s, hm, p, hosp_first, dr);
            } else if (valid) {
                switch (hour_class(hod)) {
                    case kHcEnd: nc = routine_end(P, pl, s, hm, p, dr); break;
                    case kHcTransport: nc = perform_movements<kHcTransport>(P, pl, tables, boxes, s, a.wsa + i, hm, wk, p, hour, dr, infect); break;
                    case kHcWork: nc = perform_movements<kHcWork>(P, pl, tables, boxes, s, a.wsa + i, hm, wk, p, hour, dr, infect); break;
                    case kHcNoon: nc = perform_movements<kHcNoon>(P, pl, tables, boxes, s, a.wsa + i, hm, wk, p, hour, dr, infect); break;
                    case kHcHome: nc = perform_movements<kHcHome>(P, pl, tables, boxes, s, a.wsa + i, hm, wk, p, hour, dr, infect); break;
                    default: nc = perform_movements<kHcMove>(P, pl, tables, boxes, s, a.wsa + i, hm, wk, p, hour, dr, infect); break;
                }
            }
            const bool moving = nc != p;
            uint32_t* claim = &a.claim[(nc >> 16) * (uint32_t)P.W + (nc & 0xFFFFu)];
            const uint32_t key = claim_key(hour, i);
            if (moving) atomicMin(claim, key);
            if (infect) infection_dynamics(P, pl, tables, boxes, s, at, hm, wk, nc, hour, dr);
            tally.add(valid, count_bin(s));
            tally.flush(sh);
            __syncthreads();
            add_counts(slot);
            sync();  // every claim is in, and the bit plane of before has been read
            e = count_of(slot, 1u), inf = count_of(slot, 2u), hos = count_of(slot, 3u);
            const bool win = moving && *(volatile const uint32_t*)claim == key;
            const uint32_t q = win ? nc : p;
            const uint32_t Xo = (p & 0xFFFFu) + 1u, X = (q & 0xFFFFu) + 1u;
            uint32_t* word = &next[((q >> 16) + 1u) * P.PW + (X >> 5)];
            if (patch ? win : valid) atomicOr(word, 1u << (X & 31u));
            if (patch && win) atomicAnd(&next[((p >> 16) + 1u) * P.PW + (Xo >> 5)], ~(1u << (Xo & 31u)));
            if (valid && (infected(s0) || infected(s))) {
                const uint32_t cls0 = cell_class(P, s0), cls = cell_class(P, s);
                if (win || cls != cls0) {
                    if (cls0 >= 2u) class_add(a.cls, a.danger, (uint32_t)P.WP, p, cls0, true);
                    if (cls >= 2u) class_add(a.cls, a.danger, (uint32_t)P.WP, q, cls, false);
                }
            }
            p = q;
            if (!patch)
                for (uint32_t w = i; w < a.occ_words / 4u; w += gridDim.x * blockDim.x)
                    reinterpret_cast<uint4*>(occ)[w] = make_uint4(0u, 0u, 0u, 0u);
            sync();
        }
        last = hour;
        // the row, the stop rule and the guard
        bool fire = false;
        if (a.run_loop) {
            if (hod == 0u) {
                const uint32_t fresh = inf > ivn ? inf - ivn : 0u;
                ivn = fresh;
                fire = ((P.guard_flags & kGuardLock) && inf > P.lock_threshold) ||
                       ((P.guard_flags & kGuardSpread) && fresh >= P.spread_threshold) ||
                       ((P.guard_flags & kGuardOccupancy) && hos >= P.occ_threshold);
            }
            over = fire || (e | inf | hos) == 0u;
        }
        if (rank == 0 && tid < 8u) {
            a.rows[(size_t)k * 8u + tid] = tid < 6u ? count_of(slot, tid) : (tid == 6u && fire ? 1u : 0u);
            // (cleared two hours before its next use: its readers have passed a barrier by then)
            if (GRID) a.sums[((slot + 2u) % 3u * 8u + tid) * kLineWords] = 0u;
            else total[(slot + 2u) % 3u][tid] = 0u;
        }
        written = k + 1u;
        slot = (slot + 1u) % 3u;
    }
    if (valid) {
        a.st[i] = make_uint2(s, at);
        (written ? a.pos_buf[hour_parity(last % 24u)] : a.pos)[i] = p;
    }
    if (rank == 0) {
        for (uint32_t w = written * 8u + tid; w < a.hours * 8u; w += blockDim.x) a.rows[w] = 0u;
        if (tid == 0) {
            if (a.run_loop) *a.ivn = ivn;
            *a.err_out = *(volatile int*)a.err;
        }
    }
    if (!GRID) cluster_sync();  // the first CTA's counters outlive their readers
    if (!ok && tid == 0) {
        atomicOr(a.err, kErrWait);  // stays: the world is somewhere within an hour
        *(volatile int*)(a.err_out + 1) = kErrWait;
    }
}

// ---------------------------------------------------------------- the caller-owned planes
// The hour of epi_tick_hour_noalloc, whose caller owns one byte plane and no second buffers:
// claims are an atomicMin per mover on a claim plane that every call resets, and
// the commit reads the winner back and patches the plane in place.
template <int HC>
__global__ void __launch_bounds__(kThreads) k_decide_bytes(const DevParams* __restrict__ Pall, uint32_t n_chunks,
                                                           const uint32_t* __restrict__ pos, uint2* __restrict__ st,
                                                           const uint32_t* __restrict__ home, const uint32_t* __restrict__ work,
                                                           uint32_t* __restrict__ wsa, const uint8_t* __restrict__ plane,
                                                           uint32_t* __restrict__ claim, uint32_t* __restrict__ tgt,
                                                           HourArgs ha, int* err) {
    __shared__ uint32_t sh[8];
    __shared__ DevParams sP;
    __shared__ MoveTables tables;
    __shared__ Box boxes[8];  // (the caller's state words hold any 3-bit code)
    const DevParams& P = sP;
    stage_tables(tables);  // read after switch_rep's barriers
    const HourRow hr = hour_row(ha);
    const uint32_t hour = hr.hour;
    BlockRep br;
    Tally tally;
    uint32_t hosp_first = kNoAction;
    bool hosp_known = false;
    if (blockIdx.x >= n_chunks) return;  // block-uniform
    switch_rep(br, 0u, Pall, sP, tally, sh, row_ptr(ha, hr.row), boxes);
    const ByteView pl{plane, P.G, P.WP, err};
    for (uint32_t c = blockIdx.x; c < n_chunks; c += gridDim.x) {
        const uint32_t i = c * kChunk + threadIdx.x;
        const bool valid = i < P.n;
        uint2 sv = valid ? st[i] : make_uint2(0u, 0u);
        uint32_t s = sv.x, at = sv.y;
        const uint32_t p = valid ? pos[i] : 0u;
        if (HC == kHcStart) {
            const bool need = valid && wants_hospital(P, infected(s) ? with_day(s, st_day(s) + 1u) : s);
            if (__syncthreads_or(need) && !hosp_known) {
                hosp_first = block_first_vacant(P, pl);
                hosp_known = true;
            }
        }
        if (valid) {
            const uint32_t hm = home[i], wk = work[i];
            Draws dr{i, hour, P.key0, P.key1, P.move_key};
            uint32_t q;
            bool infect = false;
            if (HC == kHcStart) q = routine_start(P, pl, s, hm, p, hosp_first, dr);
            else if (HC == kHcEnd) q = routine_end(P, pl, s, hm, p, dr);
            else q = perform_movements<HC>(P, pl, tables, boxes, s, wsa + i, hm, wk, p, hour, dr, infect);
            // house and office words are as the caller has them: no proposal outside the plane from them
            const uint32_t edge = (uint32_t)P.G * 0x00010001u;
            if (q != p && max2(q, edge) != edge) {
                atomicOr(err, 1);
                q = p;
            }
            if (q != p) atomicMin(&claim[(size_t)(q >> 16) * P.W + (q & 0xFFFFu)], i);
            if (infect) infection_dynamics(P, pl, tables, boxes, s, at, hm, wk, q, hour, dr);
            const uint32_t cls0 = cell_class(P, sv.x), cls = cell_class(P, s);
            tgt[i] = q != p || cls != cls0 ? encode_target(q, cls, cls0) : kNoAction;
            if (s != sv.x || at != sv.y) st[i] = make_uint2(s, at);
        }
        tally.add(valid, valid ? count_bin(s) : 0u);
    }
    flush_rep(br, tally, sh, row_ptr(ha, hr.row));
}

// Winners move, losers stay, plane bytes updated (lowest index wins a cell).
__global__ void __launch_bounds__(kThreads) k_commit_bytes(const DevParams* __restrict__ Pall, uint32_t n_agents,
                                                           uint32_t* __restrict__ pos, const uint32_t* __restrict__ tgt,
                                                           uint8_t* __restrict__ plane, const uint32_t* __restrict__ claim) {
    const uint32_t WP = (uint32_t)Pall[0].WP, W = (uint32_t)Pall[0].W;
    for (uint32_t i = blockIdx.x * kThreads + threadIdx.x; i < n_agents; i += gridDim.x * kThreads) {
        const uint32_t t = tgt[i];
        if (t == kNoAction) continue;
        const uint32_t p = pos[i], xy = target_xy(t), cls = target_class(t);
        const size_t old_cell = (size_t)(unpack_y(p) + 1) * WP + (unpack_x(p) + 1);
        if (xy != p && claim[(size_t)unpack_y(xy) * W + unpack_x(xy)] == i) {
            pos[i] = xy;
            plane[old_cell] = 0;
            plane[(size_t)(unpack_y(xy) + 1) * WP + (unpack_x(xy) + 1)] = (uint8_t)cls;
        } else if (cls != target_old_class(t)) {
            plane[old_cell] = (uint8_t)cls;
        }
    }
}

// End of a piece: the run loop's guard at a day boundary (row `guard_offset` of the piece;
// kNoGuard for none), then the piece's hours are added to the chain's hour base.  The guard
// evaluates the data-dependent triggers of process_interventions -- lockdown when infected >
// its threshold, a new hospital when the day's new infections (infected minus the previous
// boundary's figure, floored at 0) reach the spread threshold or hospitalized reaches the
// occupancy threshold -- for every replicate whose row ran, keeping the new-infections figure
// per replicate in ivn; if any fires, the row of every replicate gets the halt mark, and the
// rest of the chain does nothing.  One block.
constexpr uint32_t kNoGuard = 0xFFFFFFFFu;

__global__ void k_piece_end(const DevParams* __restrict__ Pall, uint32_t R, SegDev* seg, uint32_t* counts,
                            uint32_t row_words, uint32_t guard_offset, uint32_t advance, uint32_t* __restrict__ ivn) {
    __shared__ int fire;
    if (threadIdx.x == 0) fire = 0;
    __syncthreads();
    if (guard_offset != kNoGuard) {
        uint32_t* rows = counts + (size_t)(seg->hour_base + guard_offset - seg->first) * row_words;
        for (uint32_t r = threadIdx.x; r < R; r += blockDim.x) {
            const DevParams& P = Pall[r];
            const uint32_t* c = rows + (size_t)r * 8u;
            if (!P.active || (c[0] | c[1] | c[2] | c[3] | c[4] | c[5]) == 0u) continue;  // the hour did not run
            const uint32_t infected = c[2], hospitalized = c[3];
            const uint32_t fresh = infected > ivn[r] ? infected - ivn[r] : 0u;
            ivn[r] = fresh;
            const bool f = ((P.guard_flags & kGuardLock) && infected > P.lock_threshold) ||
                           ((P.guard_flags & kGuardSpread) && fresh >= P.spread_threshold) ||
                           ((P.guard_flags & kGuardOccupancy) && hospitalized >= P.occ_threshold);
            if (f) fire = 1;
        }
        __syncthreads();
        if (fire)
            for (uint32_t r = threadIdx.x; r < R; r += blockDim.x) rows[(size_t)r * 8u + 6u] = 1u;
    }
    __syncthreads();
    if (advance && threadIdx.x == 0) seg->hour_base += advance;
}

// Occupancy bits and class planes of every agent of every replicate (world upload; the planes
// start all zero).
__global__ void k_build_plane(const DevParams* __restrict__ Pall, const uint32_t* __restrict__ chunk_rep, uint32_t n_slots,
                              const uint32_t* __restrict__ pos, const uint2* __restrict__ st, uint32_t* __restrict__ occ,
                              uint8_t* __restrict__ cls_plane, uint8_t* __restrict__ danger, int* err) {
    for (uint32_t slot = blockIdx.x * blockDim.x + threadIdx.x; slot < n_slots; slot += gridDim.x * blockDim.x) {
        const DevParams& P = Pall[chunk_rep ? chunk_rep[slot / kChunk] : 0u];
        if (slot - P.agent_off >= P.n) continue;
        const uint32_t p = pos[slot];
        const int32_t x = unpack_x(p), y = unpack_y(p);
        if (x > P.G || y > P.G) { atomicOr(err, 2); continue; }
        const uint32_t X = (uint32_t)x + 1u;
        atomicOr(&occ[P.occ_off + ((uint32_t)y + 1u) * P.PW + (X >> 5)], 1u << (X & 31u));
        const uint32_t cls = cell_class(P, st[slot].x);
        if (cls >= 2u) class_add(cls_plane + P.plane_off, danger + P.plane_off, (uint32_t)P.WP, p, cls, false);
    }
}

// LockdownIntervention apply / revoke (allocation_map.rs:349-365) on slots [off, off + n).
__global__ void k_lock(uint2* __restrict__ st, uint32_t off, uint32_t n, int on) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        uint32_t s = st[off + i].x;
        uint32_t ns = on ? (st_ws(s) != EPI_WS_ESSENTIAL ? (s | kIso) : s) : (s & ~kIso);
        if (ns != s) st[off + i].x = ns;
    }
}

// vaccinate (allocation_map.rs:381-387): susceptible agents with Philox block 3 word 0 < thr.
__global__ void k_vaccinate(uint2* __restrict__ st, uint32_t off, uint32_t n, uint32_t key0, uint32_t key1,
                            uint32_t hour, uint64_t thr) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        uint32_t s = st[off + i].x;
        if ((s & kStateMask) != EPI_S) continue;
        uint32_t u[4];
        philox4x32(i, hour, kBlkVaccine, 0u, key0, key1, u);
        if ((uint64_t)u[0] < thr) st[off + i].x = s | kVacc;
    }
}

// Invariants: each agent's cell is occupied and holds its class byte (bad[0] counts those that
// do not); bad[1] counts the agents that leave a class byte.  pos and occ are the two buffers
// of each, par[r] the one that holds replicate r's state.
__global__ void k_check_agents(const DevParams* __restrict__ Pall, const uint32_t* __restrict__ chunk_rep,
                               uint32_t n_slots, const uint32_t* __restrict__ pos, const uint32_t* __restrict__ occ,
                               size_t occ_words, const uint32_t* __restrict__ par, const uint2* __restrict__ st,
                               const uint8_t* __restrict__ cls_plane, unsigned long long* bad) {
    for (uint32_t slot = blockIdx.x * blockDim.x + threadIdx.x; slot < n_slots; slot += gridDim.x * blockDim.x) {
        const uint32_t r = chunk_rep ? chunk_rep[slot / kChunk] : 0u;
        const DevParams& P = Pall[r];
        if (slot - P.agent_off >= P.n) continue;
        const uint32_t p = pos[(size_t)par[r] * n_slots + slot];
        const int32_t x = unpack_x(p), y = unpack_y(p);
        const uint32_t cls = cell_class(P, st[slot].x), X = (uint32_t)x + 1u;
        if (cls >= 2u) atomicAdd(bad + 1, 1ull);
        if (x > P.G || y > P.G ||
            !((occ[par[r] * occ_words + P.occ_off + ((uint32_t)y + 1u) * P.PW + (X >> 5)] >> (X & 31u)) & 1u) ||
            cls_plane[P.plane_off + (size_t)(y + 1) * P.WP + (x + 1)] != (cls >= 2u ? class_amount(cls) : 0u))
            atomicAdd(bad, 1ull);
    }
}

// Citizen-state stream: one byte per agent for the hour -- bits 0-3 the step taken since the
// previous hour (0 none, 1 + k for the k-th Moore neighbour in NeighborIterator order, 15 a
// jump recorded as an exception {agent, x | y << 16}), bits 4-6 the state letter
// (CitizenState::state_str, models/events/citizen_state.rs:33-44: s e i r d = 0..4).
// prev holds each agent's cell at the previous record.  Single world (slot = agent).
__device__ __forceinline__ uint32_t state_letter(uint32_t s) {
    const uint32_t v = s & kStateMask;
    return v == EPI_S ? 0u : v == EPI_E ? 1u : v == EPI_R ? 3u : v == EPI_D ? 4u : 2u;
}

// An hour that did not run (ha are its hour's arguments) leaves prev as it is: the buffer its
// parity names does not hold the state.
__global__ void k_state_delta(const DevParams* __restrict__ Pall, HourArgs ha, uint32_t n, const uint32_t* __restrict__ pos,
                              const uint2* __restrict__ st, uint32_t* __restrict__ prev, uint8_t* __restrict__ codes,
                              uint2* __restrict__ exc, uint32_t* __restrict__ exc_count) {
    if (!Pall[0].active || run_ended(prev_ptr(ha, hour_row(ha).row), 0u)) return;
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const bool valid = i < n;
    uint32_t code = 0u, p = 0u;
    bool jump = false;
    if (valid) {
        p = pos[i];
        const uint32_t q = prev[i];
        const int32_t dx = unpack_x(p) - unpack_x(q), dy = unpack_y(p) - unpack_y(q);
        uint32_t step = 0u;
        if (dx != 0 || dy != 0) {
            if (dx >= -1 && dx <= 1 && dy >= -1 && dy <= 1) {
                const int k9 = (dy + 1) * 3 + (dx + 1);     // row-major 3x3 index, centre 4
                step = 1u + (uint32_t)(k9 < 4 ? k9 : k9 - 1);  // NeighborIterator order
            } else {
                step = 15u;
                jump = true;
            }
            prev[i] = p;
        }
        code = step | (state_letter(st[i].x) << 4);
        codes[i] = (uint8_t)code;
    }
    // exceptions: one atomic per warp, lanes in order
    const uint32_t lane = threadIdx.x & 31u, m = __ballot_sync(0xFFFFFFFFu, jump);
    if (m) {
        uint32_t base = 0;
        if (lane == 0) base = atomicAdd(exc_count, (uint32_t)__popc(m));
        base = __shfl_sync(0xFFFFFFFFu, base, 0);
        if (jump) exc[base + (uint32_t)__popc(m & ((1u << lane) - 1u))] = make_uint2(i, p);
    }
}

// Cells of [0, G]^2 whose infectious-neighbour count differs from the 3x3 of the class bytes
// (replicates r = blockIdx.y, blockIdx.y + gridDim.y, ...).
__global__ void k_check_danger(const DevParams* __restrict__ Pall, uint32_t R, const uint8_t* __restrict__ cls_plane,
                               const uint8_t* __restrict__ danger, unsigned long long* bad) {
    unsigned long long b = 0;
    for (uint32_t r = blockIdx.y; r < R; r += gridDim.y) {
        const DevParams& P = Pall[r];
        const uint32_t side = (uint32_t)P.G + 1u, cells = side * side, WP = (uint32_t)P.WP;
        const uint8_t* pl = cls_plane + P.plane_off;
        const uint8_t* dg = danger + P.plane_off;
        for (uint32_t q = blockIdx.x * blockDim.x + threadIdx.x; q < cells; q += gridDim.x * blockDim.x) {
            const size_t c = (size_t)(q / side + 1) * WP + (q % side + 1);
            const uint32_t n = (pl[c - WP - 1] != 0u) + (pl[c - WP] != 0u) + (pl[c - WP + 1] != 0u) + (pl[c - 1] != 0u) +
                               (pl[c + 1] != 0u) + (pl[c + WP - 1] != 0u) + (pl[c + WP] != 0u) + (pl[c + WP + 1] != 0u);
            b += n != dg[c];
        }
    }
    if (b) atomicAdd(bad, b);
}

// Over the whole buffers, borders and slack included: occupied cells of the replicates' current
// bit planes, set bits of their other buffers (which must be none), and class bytes in use.
__global__ void k_check_planes(uint32_t R, const DevParams* __restrict__ Pall, const uint32_t* __restrict__ occ,
                               size_t occ_words, const uint32_t* __restrict__ par, size_t plane_bytes,
                               const uint8_t* __restrict__ cls_plane, unsigned long long* occupied, unsigned long long* stray,
                               unsigned long long* classed) {
    unsigned long long o = 0, x = 0, c = 0;
    const size_t stride = (size_t)gridDim.x * blockDim.x, first = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    for (uint32_t r = 0; r < R; ++r) {
        const size_t w0 = Pall[r].occ_off, w1 = r + 1 < R ? Pall[r + 1].occ_off : occ_words;
        for (size_t k = w0 + first; k < w1; k += stride) {
            o += __popc(occ[par[r] * occ_words + k]);
            x += __popc(occ[(1u - par[r]) * occ_words + k]);
        }
    }
    for (size_t k = first; k < plane_bytes; k += stride) c += cls_plane[k] != 0;
    for (int off = 16; off; off >>= 1) {
        o += __shfl_down_sync(0xFFFFFFFFu, o, off);
        x += __shfl_down_sync(0xFFFFFFFFu, x, off);
        c += __shfl_down_sync(0xFFFFFFFFu, c, off);
    }
    if ((threadIdx.x & 31) == 0) {
        if (o) atomicAdd(occupied, o);
        if (x) atomicAdd(stray, x);
        if (c) atomicAdd(classed, c);
    }
}

}  // namespace kern
}  // namespace epi
