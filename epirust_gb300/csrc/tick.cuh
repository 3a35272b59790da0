// tick.cuh -- the per-agent hourly rules as sm_103a device code.
//
// One thread owns one agent for one hour.  It reads the agent's packed words and the
// previous-hour occupancy (never another agent's record), proposes a target cell, updates its
// own disease state and claims the target (kernels.cuh).
// The rules follow engine/src/citizen/mod.rs:215-454,
// engine/src/state_machine/default_disease_handler.rs:31-103 and
// engine/src/allocation_map.rs:136-163; random draws are fixed words of per-agent-hour
// Philox blocks (movement: Philox2x32, counter = agent | which, hour; disease: Philox4x32,
// counter = agent, hour, block, 0).
//
// Moore neighbourhoods are evaluated as bit masks of the 3x3 block (bit 3 (dy + 1) + dx + 1;
// without the centre that is NeighborIterator order), which a view of the previous hour's
// world delivers:
//   BitView   the engine's: one occupancy bit per cell, a class byte per cell that is non-zero
//             only under an infectious agent, and a per-cell count of infectious neighbours
//             that lets a susceptible agent skip the exposure block when it is zero;
//   ByteView  the caller's byte plane of epi_tick_hour_noalloc (0 vacant, 1 occupied, 2 / 3
//             infectious at the regular / high rate).
// Both carry a one-cell border, so the 3x3 block around any cell of [0, G]^2 is in bounds.
// The area and grid filters of get_neighbors_of / is_point_in_grid become a second mask.
#pragma once

#include "epi_internal.h"

namespace epi {

// The eight neighbour bytes of a 3x3 block in NeighborIterator order, as two words: bytes of
// lo = neighbours 0-3 (row 0 bytes 0-2, row 1 byte 0), bytes of hi = neighbours 4-7 (row 1
// byte 2, row 2 bytes 0-2).  Two byte permutes; byte 3 of a row is never selected.
struct Nb8 {
    uint32_t lo, hi;
};
__device__ __forceinline__ Nb8 neighbour_bytes(uint32_t r0, uint32_t r1, uint32_t r2) {
    return Nb8{__byte_perm(r0, r1, 0x4210u), __byte_perm(r1, r2, 0x6542u)};
}
// Bit 0 of each byte of f (other bits zero) -> 4 bits, byte k to bit k: the product spreads
// byte k's bit to bit 24 + k with no carries (the other partial products land on distinct
// bits below 24 or beyond bit 31).
__device__ __forceinline__ uint32_t pack4(uint32_t f) { return (f * 0x01020408u) >> 24; }
__device__ __forceinline__ uint32_t pack8(uint32_t flo, uint32_t fhi) { return pack4(flo) | (pack4(fhi) << 4); }

// 8 neighbours (NeighborIterator order) <-> the 9 cells of the block (centre bit 4 clear).
constexpr uint32_t kNeighbours9 = 0x1EFu;
__host__ __device__ constexpr uint32_t block9(uint32_t m8) { return (m8 & 0xFu) | ((m8 & 0xF0u) << 1); }
__host__ __device__ constexpr uint32_t neighbours8(uint32_t m9) { return (m9 & 0xFu) | ((m9 >> 1) & 0xF0u); }

// A view's loads: through the read-only path for planes that nothing writes while the kernel
// runs; as plain loads for planes that other SMs change between the hours of one kernel (the
// barriers order them; loads at L2, which no L1 serves, made an hour of 5,000 agents 3 % longer).
template <bool SHARED, class T>
__device__ __forceinline__ T plane_load(const T* p) {
    return SHARED ? *p : __ldg(p);
}

// Bytes of (x-1, y), (x, y), (x+1, y) of a bordered byte plane (cell (x, y) at
// (y + 1) * WP + x + 1) in bits 0-7, 8-15, 16-23 (bits 24-31: the next byte of the row, which
// no caller reads): two aligned 32-bit loads and a funnel shift.
template <bool SHARED = false>
__device__ __forceinline__ uint32_t byte_row3(const uint8_t* plane, int32_t WP, int32_t x, int32_t y) {
    const uintptr_t a = (uintptr_t)(plane + (size_t)(y + 1) * (size_t)WP + (size_t)x);
    const uint32_t* w = (const uint32_t*)(a & ~(uintptr_t)3);
    const uint32_t lo = plane_load<SHARED>(w), hi = plane_load<SHARED>(w + 1);
    return __funnelshift_r(lo, hi, (uint32_t)(a & 3u) * 8u);
}

// Three rows of the 3x3 block around a cell, in a view's own form.
struct Rows3 {
    uint32_t r0, r1, r2;
};
// Infectious and high-rate neighbours of a cell, 8-bit masks in NeighborIterator order.
struct InfMasks {
    uint32_t inf, high;
};

// Cells outside [0, G]^2 are never addressed by construction; if one were, it is reported
// through err and treated as occupied (and not infectious) instead of being dereferenced.
__device__ __forceinline__ bool in_plane(int32_t G, int* err, int32_t x, int32_t y) {
    if ((uint32_t)x <= (uint32_t)G && (uint32_t)y <= (uint32_t)G) return true;
    atomicOr(err, 1);
    return false;
}

// A caller's byte plane: bytes 0..3, occupied <=> bit0|bit1, infectious <=> bit1, high rate
// <=> bit0&bit1.
struct ByteView {
    const uint8_t* __restrict__ cells;
    int32_t G, WP;
    int* err;
    __device__ __forceinline__ bool inside(int32_t x, int32_t y) const { return in_plane(G, err, x, y); }
    __device__ __forceinline__ bool vacant(int32_t x, int32_t y) const {
        return inside(x, y) && __ldg(cells + (size_t)(y + 1) * (size_t)WP + (size_t)(x + 1)) == 0u;
    }
    __device__ __forceinline__ uint32_t row(int32_t x, int32_t y) const { return byte_row3(cells, WP, x, y); }
    __device__ __forceinline__ Rows3 rows(int32_t x, int32_t y) const {
        if (!inside(x, y)) return Rows3{0x010101u, 0x010101u, 0x010101u};
        return Rows3{row(x, y - 1), row(x, y), row(x, y + 1)};
    }
    static __device__ __forceinline__ bool centre_vacant(uint32_t r1) { return ((r1 >> 8) & 0xFFu) == 0u; }
    static __device__ __forceinline__ uint32_t occupied(const Rows3& r) {
        const Nb8 b = neighbour_bytes(r.r0, r.r1, r.r2);
        const uint32_t m = 0x01010101u;
        return block9(pack8((b.lo | (b.lo >> 1)) & m, (b.hi | (b.hi >> 1)) & m));
    }
    // no infectious neighbour for sure (never known without reading the block)
    __device__ __forceinline__ bool safe(int32_t, int32_t) const { return false; }
    __device__ __forceinline__ InfMasks infectious(int32_t x, int32_t y) const {
        const Rows3 r = rows(x, y);
        const Nb8 b = neighbour_bytes(r.r0, r.r1, r.r2);
        const uint32_t m = 0x01010101u;
        return InfMasks{pack8((b.lo >> 1) & m, (b.hi >> 1) & m), pack8(b.lo & (b.lo >> 1) & m, b.hi & (b.hi >> 1) & m)};
    }
};

// The engine's planes.  occ: one bit per cell, cell (x, y) bit (x + 1) & 31 of word
// (y + 1) * PW + ((x + 1) >> 5) -- a 3x3 block is three words (six where it straddles one),
// and the whole plane of a 2,500 grid is 0.8 MB where a byte plane took 6.3 MB, so the blocks
// that sweep the agents find it in L1 far more often.  cls: class bytes, bit 0 of a byte an
// infectious agent at the regular rate, bit 4 one at the high rate.  danger: infectious agents
// among the 8 neighbours.
template <bool SHARED = false>
struct BitView {
    const uint32_t* occ;
    const uint8_t* cls;
    const uint8_t* danger;
    int32_t G, WP;
    uint32_t PW;
    int* err;
    __device__ __forceinline__ bool inside(int32_t x, int32_t y) const { return in_plane(G, err, x, y); }
    __device__ __forceinline__ bool vacant(int32_t x, int32_t y) const {
        if (!inside(x, y)) return false;
        const uint32_t X = (uint32_t)x + 1u;
        return ((plane_load<SHARED>(occ + ((uint32_t)y + 1u) * PW + (X >> 5)) >> (X & 31u)) & 1u) == 0u;
    }
    // bits of (x-1, y), (x, y), (x+1, y) in bits 0-2 (higher bits: later cells)
    __device__ __forceinline__ uint32_t row(int32_t x, int32_t y) const {
        const uint32_t* w = occ + ((uint32_t)y + 1u) * PW + ((uint32_t)x >> 5);
        const uint32_t sh = (uint32_t)x & 31u;
        const uint32_t lo = plane_load<SHARED>(w), hi = sh > 29u ? plane_load<SHARED>(w + 1) : 0u;
        return __funnelshift_r(lo, hi, sh);
    }
    static __device__ __forceinline__ bool centre_vacant(uint32_t r1) { return (r1 & 2u) == 0u; }
    static __device__ __forceinline__ uint32_t occupied(const Rows3& r) {
        return (r.r0 & 7u) | ((r.r1 & 7u) << 3) | ((r.r2 & 7u) << 6);
    }
    // (x, y) is a proposal: inside the plane
    __device__ __forceinline__ bool safe(int32_t x, int32_t y) const {
        return plane_load<SHARED>(danger + (size_t)(y + 1) * (size_t)WP + (size_t)(x + 1)) == 0u;
    }
    __device__ __forceinline__ InfMasks infectious(int32_t x, int32_t y) const {
        if (!inside(x, y)) return InfMasks{0u, 0u};
        const Nb8 b = neighbour_bytes(byte_row3<SHARED>(cls, WP, x, y - 1), byte_row3<SHARED>(cls, WP, x, y), byte_row3<SHARED>(cls, WP, x, y + 1));
        const uint32_t m = 0x01010101u;
        return InfMasks{pack8((b.lo | (b.lo >> 4)) & m, (b.hi | (b.hi >> 4)) & m), pack8((b.lo >> 4) & m, (b.hi >> 4) & m)};
    }
};

// Cells and areas as packed words, x | y << 16: bounds are tested and clamped for both
// coordinates at once (values stay below 2^14, so sums with kHalf = 2^14 per half never carry).
// An area is its low and high corner, both inside it.
struct Box {
    uint32_t lo, hi;
};
constexpr uint32_t kHalf = 0x40004000u;
__device__ __forceinline__ uint32_t max2(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("max.u16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ uint32_t min2(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("min.u16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ bool box_has(const Box& b, uint32_t c) {
    return (max2(b.lo + kHalf - c, kHalf) | max2(c + kHalf - b.hi, kHalf)) == kHalf;
}

// Tables of the kernels' shared memory.
//   valid[i]   cells of a 3x3 block inside bounds, i = columns cut off on the left | rows cut
//              off above << 2 | columns on the right << 4 | rows below << 6 (3 cuts all)
//   step[m][j] Moore step of the j-th set bit of a 9-cell mask m, (dx + 1) | (dy + 1) << 4
// Lanes with different entries cost bank conflicts there instead of cache lines.
struct __align__(16) MoveTables {
    uint16_t valid[256];
    uint8_t step[512][8];
};
constexpr MoveTables make_move_tables() {
    MoveTables t{};
    for (int i = 0; i < 256; ++i) {
        const int cl = i & 3, rl = (i >> 2) & 3, cr = (i >> 4) & 3, rr = (i >> 6) & 3;
        int m = 0;
        for (int k = 0; k < 9; ++k) {
            const int c = k % 3, r = k / 3;
            if (c >= cl && c < 3 - cr && r >= rl && r < 3 - rr) m |= 1 << k;
        }
        t.valid[i] = (uint16_t)m;
    }
    for (int m = 0; m < 512; ++m) {
        int j = 0;
        for (int k = 0; k < 9; ++k)
            if (k != 4 && ((m >> k) & 1)) t.step[m][j++] = (uint8_t)((k % 3) | ((k / 3) << 4));
    }
    return t;
}
__device__ const MoveTables kMoveTables = make_move_tables();
// The block's copy (the caller synchronises before it is read).
__device__ __forceinline__ void stage_tables(MoveTables& sh) {
    const uint4* src = reinterpret_cast<const uint4*>(&kMoveTables);
    for (uint32_t k = threadIdx.x; k < sizeof(MoveTables) / 16; k += blockDim.x)
        reinterpret_cast<uint4*>(&sh)[k] = __ldg(src + k);
}

// Cells of the block around c inside area b and the grid (last = the grid's last cell
// G - 1 | G - 1 << 16; Area::get_neighbors_of filtered by is_point_in_grid): how many columns
// and rows lie beyond the bounds on either side, clamped to 0..3, index the table.
__device__ __forceinline__ uint32_t valid_block(const MoveTables& t, const Box& b, uint32_t last, uint32_t c) {
    const uint32_t beyond = kHalf + 0x00010001u;
    const uint32_t l = min2(max2(b.lo + beyond - c, kHalf), kHalf | 0x00030003u);
    const uint32_t h = min2(max2(c + beyond - min2(b.hi, last), kHalf), kHalf | 0x00030003u);
    const uint32_t i = (l | (h << 4)) & 0x00330033u;  // columns in bits 0-1, 4-5; rows in 16-17, 20-21
    return t.valid[(i | (i >> 14)) & 0xFFu];
}

// Lazily materialised Philox blocks of one agent-hour: m(0), m(1) the random-point words
// and m(2) the choice word (Philox2x32 each), d(), d2() the disease blocks (Philox4x32).
struct Draws {
    uint32_t agent, hour, k0, k1, mk;
    uint32_t have = 0;
    uint32_t pt[2], ch[2], b1[4], b2[4];
    __device__ __forceinline__ uint32_t m(int w) {
        if (w < 2) {
            if (!(have & 1u)) { philox2x32(agent | kMovePoint, hour, mk, pt); have |= 1u; }
            return pt[w];
        }
        if (!(have & 8u)) { philox2x32(agent | kMoveChoice, hour, mk, ch); have |= 8u; }
        return ch[0];
    }
    // One movement block chosen per lane (the point block when go, else the choice block),
    // computed before a work-status branch so that a warp whose lanes take both arms runs
    // the Philox rounds once instead of once per arm; the words are the ones m() returns.
    __device__ __forceinline__ void prime(bool go) {
        uint32_t o[2];
        philox2x32(agent | (go ? kMovePoint : kMoveChoice), hour, mk, o);
        if (go) { pt[0] = o[0]; pt[1] = o[1]; have |= 1u; }
        else { ch[0] = o[0]; ch[1] = o[1]; have |= 8u; }
    }
    __device__ __forceinline__ uint32_t d(int w) {
        if (!(have & 2u)) { philox4x32(agent, hour, kBlkDisease, 0u, k0, k1, b1); have |= 2u; }
        return b1[w];
    }
    __device__ __forceinline__ uint32_t d2(int w) {
        if (!(have & 4u)) { philox4x32(agent, hour, kBlkDisease2, 0u, k0, k1, b2); have |= 4u; }
        return b2[w];
    }
};

struct Cell { int32_t x, y; };

// (house and office corners are packed words already)
__device__ __forceinline__ Box home_box(uint32_t home) { return Box{home, home + 0x00010001u}; }
__device__ __forceinline__ Box office_box(uint32_t work) { return Box{work, work + 0x00090009u}; }
// The area of a code; boxes holds the packed global areas.
__device__ __forceinline__ Box area_box(const Box* boxes, uint32_t code, uint32_t home, uint32_t work) {
    Box b;
    b.lo = code == kWork ? work : home;
    b.hi = b.lo + (code == kWork ? 0x00090009u : 0x00010001u);
    if (code >= kTransport) b = boxes[code];
    return b;
}
// The packed global areas of P into shared memory (the caller synchronises).
__device__ __forceinline__ void stage_boxes(Box* boxes, const DevParams& P) {
    if (threadIdx.x < kNumAreas) {
        const Rect& r = P.area[threadIdx.x];
        boxes[threadIdx.x] = Box{pack_xy(r.x0, r.y0), pack_xy(r.x1, r.y1)};
    }
}
__device__ __forceinline__ uint32_t random_cell(const Box& b, uint32_t ux, uint32_t uy) {
    const uint32_t w = b.hi - b.lo + 0x00010001u;
    return b.lo + (uniform_index(ux, w & 0xFFFFu) | (uniform_index(uy, w >> 16) << 16));
}

// Citizen::can_move, citizen/mod.rs:452-454
__device__ __forceinline__ bool can_move(uint32_t s) {
    uint32_t v = s & kStateMask;
    return !(v == EPI_I_MILD || v == EPI_I_SEVERE || v == EPI_D || (s & (kHosp | kIso)));
}

// Plane byte of an occupied cell: 1 + transmission-rate class of an infectious occupant.
__device__ __forceinline__ uint32_t cell_class(const DevParams& P, uint32_t s) {
    if (!infected(s) || (s & kHosp)) return 1u;
    uint32_t d = (uint32_t)((int32_t)st_day(s) + st_imm(s));  // (day as i32 + immunity) as Day
    return 1u + rate_class(P.reg_start, P.high_start, P.last_day, d);
}

// A lane's move: act false keeps the cell p.  jump is Citizen::goto_area of an agent that works
// (citizen/mod.rs:367-395: a random point of the target area, kept when vacant), otherwise
// Citizen::move_agent_from over the current area (citizen/mod.rs:415-432: uniform choice among
// the vacant neighbours of the cell, or of a random point of the area when outside it); `area`
// is the one or the other's.  Both are one code path: the centre is the lane's cell or its
// random point, the row through it is read in the same pass (a jump tests the centre bit), and
// walkers also read the rows above and below.  JUMPS false: no lane of the hour jumps but
// hospital staff (rarely).
template <bool JUMPS, class V>
__device__ __forceinline__ uint32_t move_lane(const V& pl, const MoveTables& tables, bool act, bool jump, const Box& area,
                                              uint32_t p, Draws& dr) {
    if (JUMPS) dr.prime(jump);
    if (!act) return p;
    uint32_t c = p;
    if (jump || !box_has(area, p)) c = random_cell(area, dr.m(0), dr.m(1));
    const uint32_t edge = (uint32_t)pl.G * 0x00010001u;
    if (max2(c, edge) != edge) {  // reads as occupied (and is reported)
        atomicOr(pl.err, 1);
        return p;
    }
    const int32_t x = (int32_t)(c & 0xFFFFu), y = (int32_t)(c >> 16);
    const uint32_t r1 = pl.row(x, y);
    if (JUMPS && jump) return V::centre_vacant(r1) ? c : p;
    const Rows3 rows{pl.row(x, y - 1), r1, pl.row(x, y + 1)};
    // The choice word is drawn before the rows are used, so that its Philox rounds run while
    // the row loads are in flight (it is needed unless every neighbour is taken).
    const uint32_t u = dr.m(2);
    if (!JUMPS && jump) return V::centre_vacant(r1) ? c : p;
    const uint32_t cand = valid_block(tables, area, edge - 0x00010001u, c) & ~V::occupied(rows) & kNeighbours9;
    if (!cand) return p;
    const uint32_t e = tables.step[cand][uniform_index(u, (uint32_t)__popc(cand))];
    return c + ((e | (e << 12)) & 0x00030003u) - 0x00010001u;  // vacant by construction: move_agent keeps it
}

// DiseaseStateMachine::next with the default DiseaseHandler (ddh:41-86) for the hour's
// proposed cell; at is the Exposed/Pre at_hour word.
// (The agent's current area, needed only when an infectious neighbour exists, is decoded from
// its code and home / work corners here rather than by the caller.)
template <class V>
__device__ __forceinline__ void infection_dynamics(const DevParams& P, const V& pl, const MoveTables& tables,
                                                   const Box* boxes, uint32_t& s, uint32_t& at, uint32_t home,
                                                   uint32_t work, uint32_t p, uint32_t hour, Draws& dr) {
    const Cell cell{(int32_t)(p & 0xFFFFu), (int32_t)(p >> 16)};
    const uint32_t v = s & kStateMask;
    if (v == EPI_S) {
        if (s & (kWq | kVacc)) return;
        // no infectious neighbour: no draw can succeed (the centre is vacant or the agent's own)
        if (pl.safe(cell.x, cell.y)) return;
        const InfMasks masks = pl.infectious(cell.x, cell.y);
        if (!masks.inf) return;
        const Box cur = area_box(boxes, st_area(s), home, work);
        const uint32_t cand = neighbours8(valid_block(tables, cur, (uint32_t)(pl.G - 1) * 0x00010001u, p)) & masks.inf;
        if (!cand) return;
        const uint32_t high = masks.high;
        const uint64_t thr_reg = P.thr_rate[1], thr_high = P.thr_rate[2];
        // neighbours in NeighborIterator order; the first successful Bernoulli exposes
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            if (!((cand >> k) & 1u)) continue;
            const uint32_t u = k < 4 ? dr.d(k) : dr.d2(k - 4);
            if ((uint64_t)u < (((high >> k) & 1u) ? thr_high : thr_reg)) {
                s = with_state(s, EPI_E);
                at = hour;
                return;
            }
        }
    } else if (v == EPI_E) {
        int32_t jitter = (int32_t)uniform_index(dr.d(0), 3u) - 1;
        uint32_t need = (uint32_t)((int32_t)P.exposed_duration + jitter);
        if (hour - at >= need) {
            bool symptoms = (uint64_t)dr.d(1) < P.thr_symptoms;
            s = with_day(s, 0u);
            if (symptoms) { s = with_state(s, EPI_I_PRE); at = hour; }
            else s = with_state(s, EPI_I_ASYM);
        }
    } else if (v == EPI_I_PRE) {
        if (hour - at >= P.pre_duration)
            s = with_state(s, (uint64_t)dr.d(0) < P.thr_severe ? EPI_I_SEVERE : EPI_I_MILD);
    }
}

// Hour-of-day classes of the routine (constants.rs:27-36); the kernels are specialised per
// class so that each launch carries only the branches its hour can take.
enum HourClass : int {
    kHcStart = 0,     // 0: ROUTINE_START_TIME
    kHcEnd = 1,       // 23: ROUTINE_END_TIME
    kHcMove = 2,      // 9-11, 13-15, 18-22: everyone but hospital staff walks (move_agent_from)
    kHcTransport = 3, // 7, 17: ROUTINE_TRAVEL_START/END_TIME
    kHcWork = 4,      // 8: ROUTINE_WORK_TIME
    kHcNoon = 5,      // 12: NON_WORKING_TRAVEL_END_TIME
    kHcHome = 6,      // 16: ROUTINE_WORK_END_TIME
    kHcSleep = 7      // 1-6: SLEEP_START_TIME..=SLEEP_END_TIME
};

__host__ __device__ constexpr int hour_class(uint32_t hod) {
    return hod == 0u ? kHcStart
         : hod == 23u ? kHcEnd
         : (hod >= 1u && hod <= 6u) ? kHcSleep
         : (hod == 7u || hod == 17u) ? kHcTransport
         : hod == 8u ? kHcWork
         : hod == 12u ? kHcNoon
         : hod == 16u ? kHcHome
         : kHcMove;
}

// Citizen::perform_movements, citizen/mod.rs:257-349, for the movement classes (hours 7..22):
// the work-status arms (Normal|Essential, HospitalStaff, NA) at hour class HC.  Each arm is a
// jump, a walk or nothing (a non-worker's goto_area is move_agent_from over its current area),
// so the arms only choose and one move_lane serves them all.  Returns the proposed cell;
// infect is cleared when the hour ends before the infection update of
// DiseaseStateMachine::next, which the caller runs on the proposed cell otherwise.
template <int HC, class V>
__device__ __forceinline__ uint32_t perform_movements(const DevParams& P, const V& pl, const MoveTables& tables,
                                                      const Box* boxes, uint32_t& s, uint32_t* wsa, uint32_t home,
                                                      uint32_t work, uint32_t p, uint32_t hour, Draws& dr, bool& infect) {
    const uint32_t ws = st_ws(s);
    Box area = area_box(boxes, st_area(s), home, work);
    bool act = can_move(s), jump = false;
    infect = true;
    if (ws == EPI_WS_HOSPITAL_STAFF) {  // citizen/mod.rs:292-328; wsa: its work_start_at
        const uint32_t w = *wsa, since = hour >= w ? hour - w : 0u;  // saturating_sub
        if (since == 24u * 14u) {
            s |= kWq;
            act = infect = false;
        } else if (since == 24u * 14u * 2u) {
            jump = true;
            area = home_box(home);
            s = with_area(s, kHome);
            *wsa = hour + 24u * 14u;
            infect = false;
        } else if (HC == kHcWork) {
            const Box hosp = boxes[P.hosp_code];
            jump = (area.lo != hosp.lo || area.hi != hosp.hi) && w <= hour;
            act = act && jump;
            if (jump) {
                area = hosp;
                s = with_area(s, P.hosp_code);
                *wsa = hour;
            }
            s &= ~kWq;
        } else if (HC == kHcHome) {
            s |= kWq;
            act = false;
        } else {
            act = act && !(s & kWq);
        }
    } else {
        const bool worker = ws != EPI_WS_NA;  // Normal or Essential here
        if (HC == kHcTransport) {  // a worker with public transport: goto_area(transport)
            jump = worker && (s & kPt);
            if (jump) {
                area = boxes[kTransport];
                s = with_area(s, kTransport);
            }
        } else if (HC == kHcWork) {  // a worker: goto_area(office); the others: goto_area(housing), a walk
            jump = worker;
            if (jump) area = office_box(work);
            s = with_area(s, worker ? kWork : kHousing);
        } else if (HC == kHcNoon) {  // a worker walks; the others: goto_area(home), a walk
            if (!worker) s = with_area(s, kHome);
        } else if (HC == kHcHome) {  // a worker: goto_area(home)
            jump = worker;
            if (jump) {
                area = home_box(home);
                s = with_area(s, kHome);
            }
        }
        if (jump && !act) {  // goto_area's symptomatic override of a worker going home from the office
            const uint32_t v = s & kStateMask;
            const Box house = home_box(home);
            act = (v == EPI_I_MILD || v == EPI_I_SEVERE) && box_has(office_box(work), p) && area.lo == house.lo &&
                  area.hi == house.hi;
        }
    }
    return move_lane<HC == kHcTransport || HC == kHcWork || HC == kHcHome>(pl, tables, act, jump, area, p, dr);
}

// Hour 0 of the day: increment_infection_day, then Citizen::hospitalize
// (citizen/mod.rs:240-243, 351-365; allocation_map.rs:144-150).  hosp_first is the first
// vacant hospital cell of the snapshot in area-iterator order (packed) or kNoAction.
__device__ __forceinline__ bool wants_hospital(const DevParams& P, uint32_t s) {
    if ((s & kHosp) || (s & kStateMask) != EPI_I_SEVERE) return false;
    uint32_t d = (uint32_t)((int32_t)st_day(s) + st_imm(s));
    return (P.hosp_if_class >> rate_class(P.reg_start, P.high_start, P.last_day, d)) & 1u;
}

template <class V>
__device__ __forceinline__ uint32_t routine_start(const DevParams& P, const V& pl, uint32_t& s, uint32_t home, uint32_t p,
                                                  uint32_t hosp_first, Draws& dr) {
    if (infected(s)) s = with_day(s, st_day(s) + 1u);
    if (!wants_hospital(P, s)) return p;
    if (hosp_first != kNoAction) {
        s |= kHosp;
        return hosp_first;
    }
    const uint32_t q = random_cell(home_box(home), dr.m(0), dr.m(1));
    return pl.vacant(unpack_x(q), unpack_y(q)) ? q : p;
}

// Hour 23: Citizen::deceased with on_routine_end (citizen/mod.rs:397-413, ddh:88-102).
template <class V>
__device__ __forceinline__ uint32_t routine_end(const DevParams& P, const V& pl, uint32_t& s, uint32_t home, uint32_t p,
                                                Draws& dr) {
    const uint32_t v = s & kStateMask, day = st_day(s);
    if (v == EPI_I_ASYM && day == 9u) s = with_state(s, EPI_R);          // ASYMPTOMATIC_LAST_DAY
    else if (v == EPI_I_MILD && day == 12u) s = with_state(s, EPI_R);    // MILD_INFECTED_LAST_DAY
    else if (v == EPI_I_SEVERE && day == P.last_day)
        s = with_state(s, (uint64_t)dr.m(2) < P.thr_death ? EPI_D : EPI_R);
    uint32_t nc = p;
    const uint32_t nv = s & kStateMask;
    if (nv == EPI_R) {
        const uint32_t q = random_cell(home_box(home), dr.m(0), dr.m(1));
        if (pl.vacant(unpack_x(q), unpack_y(q))) nc = q;
    }
    if (nv == EPI_R || nv == EPI_D) s &= ~kHosp;
    return nc;
}

// Counts::update_counts bin (counts.rs:126-140): 0 S, 1 E, 2 I, 3 H, 4 R, 5 D.
__device__ __forceinline__ uint32_t count_bin(uint32_t s) {
    // bins of the eight states, four bits each (2..5 are the infected ones)
    const uint32_t bin = (0x54222210u >> ((s & kStateMask) * 4u)) & 7u;
    return bin == 2u && (s & kHosp) ? 3u : bin;
}

// tgt word: target x | y << 16 (14 bits each, grids up to 16,383) with the new plane class
// in bits 15 (low) and 31 (high) and the class before the hour in bits 14 and 30.
__device__ __forceinline__ uint32_t encode_target(uint32_t xy, uint32_t cls, uint32_t old_cls) {
    return xy | ((cls & 1u) << 15) | ((cls >> 1) << 31) | ((old_cls & 1u) << 14) | ((old_cls >> 1) << 30);
}
__device__ __forceinline__ uint32_t target_xy(uint32_t t) { return t & 0x3FFF3FFFu; }
__device__ __forceinline__ uint32_t target_class(uint32_t t) { return ((t >> 15) & 1u) | ((t >> 30) & 2u); }
__device__ __forceinline__ uint32_t target_old_class(uint32_t t) { return ((t >> 14) & 1u) | ((t >> 29) & 2u); }

// Class planes.  An infectious agent of plane class c (2 regular, 3 high rate) on a cell adds
// one to its field of the cell's class byte and one to the infectious-neighbour count of the
// 8 cells around; taking it away subtracts the same.  The updates of an hour only add up
// (atomically, on the 32-bit words holding the bytes), so their order does not matter and a
// proposal may be entered before its claim is settled and taken back after: at the end of the
// hour class fields are 0 or 1 and counts 0..8.
__device__ __forceinline__ void byte_add(uint8_t* plane, size_t c, uint32_t amount, bool minus) {
    const uintptr_t a = (uintptr_t)(plane + c);
    uint32_t* w = (uint32_t*)(a & ~(uintptr_t)3);
    const uint32_t v = amount << ((a & 3u) * 8u);
    atomicAdd(w, minus ? 0u - v : v);
}
__device__ __forceinline__ uint32_t class_amount(uint32_t cls) { return cls == 2u ? 0x01u : 0x10u; }
// The agent of class cls >= 2 on cell (x, y) enters (minus false) or leaves the class planes.
__device__ __forceinline__ void class_add(uint8_t* cls_plane, uint8_t* danger, uint32_t WP, uint32_t cell_xy, uint32_t cls,
                                          bool minus) {
    const size_t c = (size_t)(unpack_y(cell_xy) + 1) * WP + (size_t)(unpack_x(cell_xy) + 1);
    byte_add(cls_plane, c, class_amount(cls), minus);
    const size_t nb[8] = {c - WP - 1, c - WP, c - WP + 1, c - 1, c + 1, c + WP - 1, c + WP, c + WP + 1};
#pragma unroll
    for (int k = 0; k < 8; ++k) byte_add(danger, nb[k], 1u, minus);
}

}  // namespace epi
