// Register allocation over packed step records (rv_generator_avx.cpp:1018-1420), for
// programs in which every virtual result is its instruction's own word and functions name
// only their own words.  Other programs take the general forms of ptl_ra.cuh.
//
// The allocator is a chain: a function's step needs its previous one, and the lane-0
// functions (f % 8 == 0) meet at every step through row 0 of the register state.  So what
// bounds it is the latency of one step, not bandwidth, and the step is made short:
//   * a step's instruction is one 8-byte record (operands as distances back in words), not
//     four words with range checks;
//   * a function's symbols (its words' registers) live in a ring of bytes in shared
//     memory, indexed by the word: no tags, and older words are rare (99.9% of the operands
//     of the synthetic workloads name one of the last 128 words);
//   * only registers 5..31 (integers) and 37 (floats) are ever allocated to a symbol, so
//     only those row-0 positions ever hold one and only triggers and writes there act on
//     anything: every mask over physical registers is one 32-bit word (register codes);
//   * the independent functions store a step's swap triggers as one such mask; a pass of
//     its own folds them into per-step rows of (least, greatest) triggering group, instead
//     of two global atomics per trigger;
//   * a lane-0 slot reads and marks its own symbols only; what crosses slots within a step
//     are masks of positions (written, triggered, read by their owner) and one maximum per
//     position (the group whose write row 0 keeps).
#pragma once

#include "ptl_ra.cuh"
#include "ptl_scalar.cuh"

#if defined(__GNUC__) || defined(__CUDACC__)
#define PTL_RARE(x) __builtin_expect(!!(x), 0)
#else
#define PTL_RARE(x) (x)
#endif

namespace ptl {

// ---------------------------------------------------------------- step records
// Bits 0-23 and 24-47: distance from the word to its rs1 / rs2 symbol (0: none, or a
// symbol whose state is still the initial one); 48-53: the code of a physical rd; 54: rd
// is the word itself; 55: rs1 or rs2 is the word itself; 56: float operation.
constexpr uint32_t kStepMaxDist = 1u << 24;
constexpr uint32_t kStepDef = 1u << 22, kStepSelf = 1u << 23, kStepFloat = 1u << 24;  // in the high word
PTL_HD uint32_t step_d1(uint64_t r) { return static_cast<uint32_t>(r) & 0xFFFFFFu; }
PTL_HD uint32_t step_d2(uint64_t r) { return static_cast<uint32_t>(r >> 24) & 0xFFFFFFu; }
PTL_HD uint32_t step_phys(uint32_t hi) { return (hi >> 16) & 63u; }

// Register codes: 0 for register 37, 1..31 for those registers, and 32 or more for a
// register whose position never holds a symbol (38 and register 0 apart, a symbol never
// has such a one).
constexpr uint32_t kCodeNone = 32u, kCode38 = 38u;
PTL_HD uint32_t code_of(uint32_t reg) {
    return reg == 37u ? 0u : (reg == 38u ? kCode38 : (reg != 0 && reg < 32u ? reg : kCodeNone));
}
PTL_HD uint32_t reg_of(uint32_t code) {  // of a symbol: 0, 5..31, 37 or 38
    return code == 0 ? 37u : (code < 32u || code == kCode38 ? code : 0u);
}
// The position's bit; 0 for codes from 32 on.
PTL_HD uint32_t code_bit(uint32_t code) {
#if defined(__CUDA_ARCH__)
    uint32_t b;
    asm("shl.b32 %0, 1, %1;" : "=r"(b) : "r"(code));  // shl clamps its count
    return b;
#else
    return code < 32u ? 1u << code : 0u;
#endif
}
PTL_HD uint32_t low_bit(uint32_t m) {  // m != 0
#if defined(__CUDA_ARCH__)
    return static_cast<uint32_t>(__ffs(static_cast<int>(m)) - 1);
#else
    return static_cast<uint32_t>(__builtin_ctz(m));
#endif
}

constexpr uint64_t kStepIdle = static_cast<uint64_t>(kCodeNone) << 48;  // no operands, no result

// Word i's record, and what keeps the program from the record form: bit 0, a virtual
// register outside the word's function (the serial order); bit 1, an operand or result
// that a record cannot say (the general form).
PTL_HD uint32_t st_step_record(const Prog& P, uint32_t i, uint32_t* hint = nullptr) {
    const uint32_t lo = function_of(P, i, hint ? *hint : 0xFFFFFFFFu);
    if (hint) *hint = lo;
    const uint32_t r1 = P.rs1[i], r2 = P.rs2[i], rd = P.rd[i];
    if (!ra_own(P, lo, r1) || !ra_own(P, lo, r2) || !ra_own(P, lo, rd)) return 1u;
    const uint32_t st = P.fn_start0[lo], size = P.fn_size0[lo];
    uint64_t rec = kStepIdle;
    uint32_t out = 0;
    if (s32(size) > 0 && i >= st && i - st < size) {
        rec = 0;
        const uint32_t ins = P.instr[i];
        if (ins == 0x000000EFu) record_error(P.err, ST_UNSUPPORTED, (lo & 7u) ? W_RA1 : W_RA2, i);
        if ((ins & 0x7Fu) == 0x53u) rec |= static_cast<uint64_t>(kStepFloat) << 32;
        if (s32(rd) > 63) {
            if (rd - 64u == i) rec |= static_cast<uint64_t>(kStepDef) << 32;
            else out = 2u;
        } else if (s32(rd) < 0) {
            out = 2u;
        }
        rec |= static_cast<uint64_t>(s32(rd) >= 0 && s32(rd) <= 63 ? code_of(rd) : kCodeNone) << 48;
        const uint32_t op[2] = {r1, r2};
        for (int k = 0; k < 2; ++k) {
            if (!(s32(op[k]) > 63)) continue;
            const uint32_t x = op[k] - 64u;
            if (x == i) rec |= static_cast<uint64_t>(kStepSelf) << 32;
            if (x >= i) continue;  // not defined yet: reads and writes the initial state
            if (i - x >= kStepMaxDist) out = 2u;
            rec |= static_cast<uint64_t>(i - x) << (24 * k);
        }
    }
    P.rec[i] = rec;
    return out;
}

// Function f's range overlaps no other one and stays within the words (else the general
// form); the starts never decrease.
PTL_HD uint32_t st_step_range(const Prog& P, uint32_t f) {
    const uint32_t size = P.fn_size0[f];
    if (s32(size) <= 0) return 0u;
    const uint64_t end = static_cast<uint64_t>(P.fn_start0[f]) + size;
    const uint32_t next = f + 1u < P.F ? P.fn_start0[f + 1u] : P.W;
    return end > next ? 2u : 0u;
}

// ---------------------------------------------------------------- one step
// The allocation of a step whose operands read the registers of codes c1 and c2:
// triggered positions, the live mask after the step (bit 0: register 37; 1..4 always set),
// and the code of rd.
constexpr uint32_t kLiveInit = 0x1Eu;
struct StepOut {
    uint32_t trig, live, rd;
};
PTL_HD StepOut step_allocate(uint32_t hi, uint32_t live, uint32_t c1, uint32_t c2) {
    const uint32_t ops = code_bit(c1) | code_bit(c2);
    const uint32_t cleared = live & ~ops;
    const uint32_t open = ~(cleared | 1u);
    const uint32_t any = (hi & kStepFloat) ? 0u : (open ? low_bit(open) : 5u);
    StepOut o;
    o.rd = (hi & kStepDef) ? any : step_phys(hi);
    const uint32_t rdm = code_bit(o.rd);
    o.trig = (live & ops) | (cleared & rdm);
    o.live = cleared | rdm;
    return o;
}

// ---------------------------------------------------------------- independent functions
// Function f (f % 8 != 0): no swap mark reaches its symbols, so a symbol's register is
// the one its definition took.  Ring entry of word x: ring[(x % K) * stride].  Writes the
// symbols' registers and each step's trigger mask (tmask).  kStepAhead records are in
// flight per thread (a warp's lanes read 32 streams, so a load covers one sector a lane).
// Whole groups of steps run without end checks, and one branch covers both old operands:
// the chain is bound by its instructions (4.1M nodes: the allocation 3.71 to 3.50 ms).
constexpr uint32_t kStepAhead = 8;
PTL_HD void step_free_function(const Prog& P, uint32_t f, uint8_t* ring, uint32_t stride, uint32_t K) {
    const uint32_t start = P.fn_start0[f];
    const int32_t size = s32(P.fn_size0[f]);
    if (size <= 0) return;
    const unsigned long long* rec = P.rec + start;
    uint32_t* tm = P.tmask + start;
    uint32_t* sym = P.symreg + start;
    const uint32_t n = static_cast<uint32_t>(size), mask = K - 1u;
    uint32_t live = kLiveInit;
    unsigned long long next[kStepAhead];
#pragma unroll
    for (uint32_t k = 0; k < kStepAhead; ++k) next[k] = k < n ? rec[k] : 0ull;
    auto step = [&](uint32_t i, unsigned long long now) {
        const uint32_t d1 = step_d1(now), d2 = step_d2(now);
        const uint32_t hi = static_cast<uint32_t>(now >> 32);
        uint32_t c1 = ring[((i - d1) & mask) * stride], c2 = ring[((i - d2) & mask) * stride];
        if (PTL_RARE((d1 | d2) >= K)) {  // K is a power of two: one of them is
            if (d1 >= K) c1 = code_of(sym[i - d1]);
            if (d2 >= K) c2 = code_of(sym[i - d2]);
        }
        c1 = d1 ? c1 : kCodeNone;
        c2 = d2 ? c2 : kCodeNone;
        const StepOut o = step_allocate(hi, live, c1, c2);
        live = o.live;
        // an operand that names the word itself rewrites the definition's register by 0
        const bool def = (hi & (kStepDef | kStepSelf)) == kStepDef;
        ring[(i & mask) * stride] = static_cast<uint8_t>(def ? o.rd : kCodeNone);
        if (def) sym[i] = o.rd ? o.rd : 37u;
        tm[i] = o.trig;
    };
    uint32_t b = 0;
    for (; b + kStepAhead <= n; b += kStepAhead) {
        unsigned long long now[kStepAhead];
#pragma unroll
        for (uint32_t k = 0; k < kStepAhead; ++k) {
            now[k] = next[k];
            next[k] = b + kStepAhead + k < n ? rec[b + kStepAhead + k] : 0ull;
        }
#pragma unroll
        for (uint32_t k = 0; k < kStepAhead; ++k) step(b + k, now[k]);
    }
#pragma unroll
    for (uint32_t k = 0; k < kStepAhead; ++k)
        if (b + k < n) step(b + k, next[k]);
}

// ---------------------------------------------------------------- trigger rows
// Step i, position p (a register code below 32) of the independent functions' triggers: the least triggering group
// + 1 in the low half (0xFFFF: none), the greatest + 1 in the high half (0: none).  tany
// has a bit per position triggered at all.
constexpr uint32_t kRowNone = 0x0000FFFFu;
constexpr uint32_t kRowPos = 32;   // positions per row
constexpr uint32_t kRowTile = 32;  // steps per tile; rows are laid out in whole tiles
PTL_HD uint32_t row_min(uint32_t r) { return r & 0xFFFFu; }
PTL_HD uint32_t row_max(uint32_t r) { return r >> 16; }
PTL_HD uint64_t row_tiles(uint64_t steps) { return (steps + kRowTile - 1u) / kRowTile; }

// Group g's triggers of step i among its independent functions (8g+1 .. 8g+7).
PTL_HD uint32_t group_triggers(const Prog& P, uint32_t g, uint32_t i) {
    uint32_t m = 0;
    for (uint32_t k = 1; k < 8u; ++k) {
        const uint32_t f = 8u * g + k;
        if (f < P.F && s32(i) < s32(P.fn_size0[f])) m |= P.tmask[P.fn_start0[f] + i];
    }
    return m;
}

// ---------------------------------------------------------------- lane-0 lock-step
// Row 0 keeps, per position, the write of the highest group of the last step that wrote
// it.  own: the slot whose symbol is there, read between the step's two barriers and
// written after them; oidx: that symbol's word within its function, read by its owner
// only and written by the new owner one step late, after the next barrier (a displaced
// owner may still read its own until then; LaneSlot::new_p is the write not yet made).
// Three sets of the step's buffers take turns: the one after next is cleared behind a
// step's first barrier, when every slot is done with the step before.  win needs no
// clearing but where the step tags of its values start again.
struct LaneMasks {
    uint32_t wr;      // positions written in the step
    uint32_t trig;  // positions triggered by a lane-0 function
    uint32_t use;   // positions whose symbol its owner reads and no later independent group triggers
    uint32_t need;  // ... and no earlier independent group triggers
};
// What the slots of higher groups held elsewhere (other CTAs of a cluster) add to a step.
struct LaneAbove {
    uint32_t wr, trig;
};
struct LaneStep {
    uint32_t win[kRowPos];          // step tag and highest group + 1 writing the position
    LaneMasks m;
    uint32_t before;            // of need: an earlier lane-0 group triggers the position
    uint32_t later;             // of use: a later lane-0 group does
};
struct LaneShared {
    LaneStep st[3];
    uint32_t own[kRowPos], oidx[kRowPos];
    uint32_t before2;            // the next Jacobi round's
    uint32_t tail;               // positions triggered after the last lane-0 function has ended
    uint32_t s0;                 // the longest lane-0 function
};
constexpr uint32_t kWinTagBits = 17;  // win = tag << 14 | group + 1 (at most 8,192 groups)
PTL_HD uint32_t win_value(uint32_t i, uint32_t g1) { return (((i & ((1u << kWinTagBits) - 1u)) + 1u) << 14) | g1; }
PTL_HD bool win_wraps(uint32_t i) { return i != 0 && (i & ((1u << kWinTagBits) - 1u)) == 0; }
PTL_HD void lane_clear(LaneStep& s) {
    s.m = LaneMasks{0, 0, 0, 0};
    s.before = s.later = 0;
}
// Whether v holds in any lane: the lane-0 phases run with whole warps, and a branch that
// all lanes take together needs no reconvergence.
PTL_HD bool warp_any(bool v) {
#if defined(__CUDA_ARCH__)
    return __any_sync(0xFFFFFFFFu, v);
#else
    return v;
#endif
}
// *p = max(*p, v) in shared memory if on, without a branch around the atomic.
PTL_HD void max_if(bool on, uint32_t* p, uint32_t v) {
#if defined(__CUDA_ARCH__)
    asm volatile("{\n .reg .pred q;\n setp.ne.u32 q, %2, 0;\n @q red.shared.max.u32 [%0], %1;\n}" ::"r"(
                     static_cast<uint32_t>(__cvta_generic_to_shared(p))),
                 "r"(v), "r"(static_cast<uint32_t>(on)));  // read after a barrier only
#else
    if (on && v > *p) *p = v;
#endif
}
PTL_HD void or_u32(uint32_t* p, uint32_t v) {
#if defined(__CUDA_ARCH__)
    atomicOr(p, v);
#else
    *p |= v;
#endif
}

// One lane-0 function.  Symbol bytes: register code (bits 0-5), swapped (6), moved (7: the
// register is no longer the row-0 position its definition wrote).
constexpr uint32_t kSymSwapped = 0x40u, kSymMoved = 0x80u;
struct LaneSlot {
    // held: positions where row 0 has a symbol of this slot; marked: those of them whose
    // symbol is swapped -- the symbol's own swapped state is written when it leaves row 0
    // (most are read before that, which ends the swap).
    uint32_t live, held, marked;
    uint32_t j, size;
    uint32_t* symreg;   // of the function's first word
    uint32_t* symswp;
    const unsigned long long* rec_at;
    uint32_t new_p, new_i;  // oidx[new_p] = new_i is still to be written (kCodeNone: nothing)
    // the step
    uint64_t rec;       // kStepIdle past the function's end
    StepOut o;
    uint32_t e1, e2;    // operand symbols
    uint32_t c1, c2;    // the registers they are read into
    uint32_t m1, m2;    // their row-0 positions, as bits (0: not in row 0)
    bool b1, b2;        // an earlier group triggers it there
    bool l1, l2;        // a later independent group does
};
struct LaneRing {
    uint8_t* at;        // this slot's column
    uint32_t stride, K;
};

PTL_HD void lane_init(const Prog& P, LaneSlot& L, uint32_t j) {
    L.j = j;
    L.live = kLiveInit;
    L.held = L.marked = 0;
    L.new_p = kCodeNone;
    L.new_i = 0;
    L.o.trig = 0;
    const uint32_t f = 8u * j;
    const int32_t size = f < P.F ? s32(P.fn_size0[f]) : 0;
    L.size = size > 0 ? static_cast<uint32_t>(size) : 0u;
    const uint32_t start = f < P.F ? P.fn_start0[f] : 0u;
    L.symreg = P.symreg + start;
    L.symswp = P.symswp + start;
    L.rec_at = P.rec + start;
}

// An operand symbol older than the ring: global memory holds every symbol's state.
PTL_HD uint32_t lane_old_symbol(const LaneSlot& L, uint32_t x) {
    return code_of(L.symreg[x]) | (L.symswp[x] ? kSymSwapped : 0u) | kSymMoved;
}
// The word whose symbol row 0 has at position p (which the slot holds).
PTL_HD uint32_t lane_index(const uint32_t* oidx, const LaneSlot& L, uint32_t p) {
    return p == L.new_p ? L.new_i : oidx[p];
}
// The row-0 bit of a symbol whose register no longer tells its position (0: not there).
PTL_HD uint32_t lane_find(const uint32_t* oidx, const LaneSlot& L, uint32_t idx) {
    for (uint32_t m = L.held; m; m &= m - 1)
        if (lane_index(oidx, L, low_bit(m)) == idx) return m & (~m + 1u);
    return 0;
}

// The allocation with the operands' swap state as known (b1, b2).
PTL_HD void lane_allocate(LaneSlot& L) {
    const uint32_t hi = static_cast<uint32_t>(L.rec >> 32);
    const bool fop = (hi & kStepFloat) != 0;
    L.c1 = ((L.e1 & kSymSwapped) || (L.m1 & L.marked) || L.b1) ? (fop ? 0u : 5u) : (L.e1 & 63u);
    L.c2 = ((L.e2 & kSymSwapped) || (L.m2 & L.marked) || L.b2) ? (fop ? kCode38 : 6u) : (L.e2 & 63u);
    L.o = step_allocate(hi, L.live, L.c1, L.c2);
}
// The step's row-0 writes (rd's symbol or physical register, the cleared rs1 / rs2
// positions) and triggers.  kAlone: a program with one lane-0 function, whose writes
// always win.
template <bool kAlone>
PTL_HD void lane_emit(LaneStep& st, const LaneSlot& L, uint32_t i, LaneMasks& m) {
    if (!kAlone) {
        const uint32_t v = win_value(i, L.j + 1u);
        max_if(L.o.rd < 32u, &st.win[L.o.rd & 31u], v);
        max_if(L.c1 < 32u, &st.win[L.c1 & 31u], v);
        max_if(L.c2 < 32u, &st.win[L.c2 & 31u], v);
    }
    m.wr |= code_bit(L.o.rd) | code_bit(L.c1) | code_bit(L.c2);
    m.trig |= L.o.trig;
}

// Phase A of a slot's step: look up, allocate, publish (m: this thread's share).  Written
// without branches but for the rare cases: a branch costs a lone warp more than the few
// instructions it skips.
template <bool kAlone>
PTL_HD void lane_step_a(const LaneShared& sh, LaneStep& st, const uint32_t* row, LaneSlot& L, const LaneRing& r,
                        uint32_t i, LaneMasks& m) {
    const uint32_t d1 = step_d1(L.rec), d2 = step_d2(L.rec);
    uint32_t e1 = r.at[((i - d1) & (r.K - 1u)) * r.stride], e2 = r.at[((i - d2) & (r.K - 1u)) * r.stride];
    if (PTL_RARE(warp_any((d1 | d2) >= r.K))) {  // K is a power of two: one of them is
        if (d1 >= r.K) e1 = lane_old_symbol(L, i - d1);
        if (d2 >= r.K) e2 = lane_old_symbol(L, i - d2);
    }
    e1 = d1 ? e1 : kCodeNone;
    e2 = d2 ? e2 : kCodeNone;
    const uint32_t p1 = e1 & 31u, p2 = e2 & 31u;
    uint32_t m1 = lane_index(sh.oidx, L, p1) == i - d1 ? code_bit(e1 & 63u) & L.held : 0u;
    uint32_t m2 = lane_index(sh.oidx, L, p2) == i - d2 ? code_bit(e2 & 63u) & L.held : 0u;
    uint32_t row1 = row[p1], row2 = row[p2];
    if (PTL_RARE(warp_any(((e1 | e2) & kSymMoved) && L.held))) {
        if (e1 & kSymMoved) { m1 = lane_find(sh.oidx, L, i - d1); row1 = m1 ? row[low_bit(m1)] : 0u; }
        if (e2 & kSymMoved) { m2 = lane_find(sh.oidx, L, i - d2); row2 = m2 ? row[low_bit(m2)] : 0u; }
    }
    L.e1 = e1;
    L.e2 = e2;
    L.m1 = m1;
    L.m2 = m2;
    L.b1 = L.b2 = L.l1 = L.l2 = false;
    if (!kAlone) {  // else every other function is in the slot's own group
        L.b1 = m1 && row_min(row1) <= L.j;
        L.b2 = m2 && row_min(row2) <= L.j;
        L.l1 = m1 && row_max(row1) > L.j + 1u;
        L.l2 = m2 && row_max(row2) > L.j + 1u;
        m.use |= (L.l1 ? 0u : m1) | (L.l2 ? 0u : m2);
        m.need |= (L.b1 ? 0u : m1) | (L.b2 ? 0u : m2);
    }
    lane_allocate(L);
    lane_emit<kAlone>(st, L, i, m);
}

// Phase T (m: the masks over all slots): this slot's triggers of symbols that their owner
// reads in this step.  Returns whether one changes what phase A assumed (then the Jacobi
// rounds run).
PTL_HD bool lane_step_t(LaneShared& sh, LaneStep& st, const LaneMasks& m, const LaneSlot& L) {
    bool redo = false;
    uint32_t t = L.o.trig & (m.use | m.need) & ~(L.m1 | L.m2);
    while (warp_any(t != 0)) {
        if (t) {
            const uint32_t p = low_bit(t), bit = t & (~t + 1u);
            const uint32_t o = sh.own[p];
            t ^= bit;
            if (L.j > o) or_u32(&st.later, bit);
            if (L.j < o && (m.need & bit)) {
                or_u32(&st.before, bit);
                redo = true;
            }
        }
    }
    return redo;
}
// The new owner's part of row 0 (see LaneShared::oidx).
PTL_HD void lane_commit(LaneShared& sh, LaneSlot& L) {
    if (L.new_p < 32u) sh.oidx[L.new_p] = L.new_i;
    L.new_p = kCodeNone;
}
// A Jacobi round: with the flags so far, the allocation again and the next round's flags.
PTL_HD void lane_round(LaneShared& sh, const LaneStep& st, const LaneMasks& m, const uint32_t* row, LaneSlot& L) {
    if (L.m1 | L.m2) {  // outside need, b1 / b2 come from the independent groups and stay
        if (L.m1 & m.need) L.b1 = (L.m1 & st.before) != 0;
        if (L.m2 & m.need) L.b2 = (L.m2 & st.before) != 0;
        lane_allocate(L);
    }
    for (uint32_t t = L.o.trig & m.need; t; t &= t - 1)
        if (L.j < sh.own[low_bit(t)]) or_u32(&sh.before2, t & (~t + 1u));
}

// An operand's symbol keeps the register it was read into, and is no longer swapped.
PTL_HD void lane_store(const LaneSlot& L, const LaneRing& r, uint32_t i, uint32_t d, uint32_t old, uint32_t code) {
    const uint32_t idx = i - d;
    if (d < r.K)
        r.at[(idx & (r.K - 1u)) * r.stride] =
            static_cast<uint8_t>(code | ((old & kSymMoved) || code != (old & 63u) ? kSymMoved : 0u));
    L.symreg[idx] = reg_of(code);
    if (old & kSymSwapped) L.symswp[idx] = 0;
}

// Phase B, first part: the symbols after the step, but for swaps.  again: after the
// allocation has changed.
PTL_HD void lane_step_b1(LaneSlot& L, const LaneRing& r, uint32_t i, bool again) {
    const uint32_t hi = static_cast<uint32_t>(L.rec >> 32);
    const uint32_t d1 = step_d1(L.rec), d2 = step_d2(L.rec);
    const bool def = (hi & (kStepDef | kStepSelf)) == kStepDef;
    r.at[(i & (r.K - 1u)) * r.stride] =
        static_cast<uint8_t>((def ? L.o.rd : kCodeNone) | ((hi & kStepSelf) ? kSymMoved : 0u));
    if (def) L.symreg[i] = L.o.rd ? L.o.rd : 37u;
    const bool s1 = d1 && d1 != d2 && (L.e1 != L.c1 || again), s2 = d2 && (L.e2 != L.c2 || again);
    if (warp_any(s1 || s2)) {
        if (s1) lane_store(L, r, i, d1, L.e1, L.c1);
        if (s2) lane_store(L, r, i, d2, L.e2, L.c2);
    }
}

// Swapped symbols at the positions of t leave row 0.
PTL_HD void lane_leave(const LaneShared& sh, const LaneSlot& L, const LaneRing& r, uint32_t i, uint32_t t) {
    do {  // seldom more than one
        if (t) {
            const uint32_t idx = sh.oidx[low_bit(t)];
            t &= t - 1;
            L.symswp[idx] = 0xFFFFFFFFu;
            if (i - idx < r.K) r.at[(idx & (r.K - 1u)) * r.stride] |= kSymSwapped;
        }
    } while (PTL_RARE(warp_any(t != 0)));
}

// Phase B, second part: swaps and row 0 after the step (a slot whose function has ended
// takes part while row 0 has symbols of it).  m: the masks over all slots; others:
// positions the independent functions trigger.
template <bool kAlone>
PTL_HD void lane_step_b2(LaneShared& sh, const LaneStep& st, const LaneMasks& m, const LaneAbove& ab, uint32_t others,
                         LaneSlot& L, const LaneRing& r, uint32_t i) {
    const uint32_t hi = static_cast<uint32_t>(L.rec >> 32);
    L.live = L.o.live;
    // a symbol in row 0 that the slot reads ends swapped only when a later group triggers
    // its position in this step; one that it does not read, when any function does
    bool l1 = L.l1, l2 = L.l2;
    if (!kAlone) {
        const uint32_t later = st.later | ab.trig;
        l1 = l1 || (L.m1 & later) != 0;
        l2 = l2 || (L.m2 & later) != 0;
    }
    const uint32_t operands = L.m1 | L.m2;
    L.marked = (L.marked & ~operands) | (l1 ? L.m1 : 0u) | (l2 ? L.m2 : 0u) | (L.held & ~operands & (others | m.trig));
    const uint32_t leave = L.marked & m.wr;
    if (warp_any(leave != 0)) lane_leave(sh, L, r, i, leave);
    L.held &= ~m.wr;
    L.marked &= L.held;
    const uint32_t bit = code_bit(L.o.rd);
    if ((hi & kStepDef) && (kAlone || (st.win[L.o.rd] == win_value(i, L.j + 1u) && !(ab.wr & bit)))) {
        if (!kAlone) sh.own[L.o.rd] = L.j;
        L.new_p = L.o.rd;
        L.new_i = i;
        L.held |= bit;
    }
}

// After the last lane-0 function's last step: the remaining steps only mark the symbols
// that row 0 holds at positions an independent function triggers (tail: those positions).
PTL_HD void lane_tail(const LaneShared& sh, const LaneSlot& L, uint32_t tail) {
    for (uint32_t m = L.held & (L.marked | tail); m; m &= m - 1) L.symswp[sh.oidx[low_bit(m)]] = 0xFFFFFFFFu;
}

// ---------------------------------------------------------------- the scalar generator
// Its functions (ptl_scalar.cuh) have a register state each, so every function is on its
// own like a lone lane-0 slot, with three differences: physical operands clear and swap
// like symbols' registers, a call out of the function frees and swaps the caller-saved
// registers, and the live mask's callee-saved registers are gathered (preserve).
//
// Records: bits 0-19 and 20-39, distances of the operand symbols (0: none); 40-45 rd's
// code, 46-51 and 52-57 physical operands' codes; 58 rd is the word itself, 59 an operand
// is, 60 float result, 61 float operands, 62 a call out of the function, 63 used.
constexpr uint32_t kScalarDist = 1u << 20;
constexpr uint32_t kSDef = 1u << 26, kSSelf = 1u << 27, kSFloatRd = 1u << 28, kSFloatOp = 1u << 29, kSCall = 1u << 30,
                   kSUsed = 1u << 31;  // in the high word
constexpr uint32_t kScalarPreserved = 0x0FFC031Eu;  // kPreservedRegisterMask in register codes

PTL_HD uint32_t st_scalar_record(const Prog& P, uint32_t i, uint32_t* hint = nullptr) {
    const uint32_t lo = function_of(P, i, hint ? *hint : 0xFFFFFFFFu);
    if (hint) *hint = lo;
    const uint32_t op[2] = {P.rs1[i], P.rs2[i]}, rd = P.rd[i];
    if (!ra_own(P, lo, op[0]) || !ra_own(P, lo, op[1]) || !ra_own(P, lo, rd)) return 1u;
    const uint32_t st = P.fn_start0[lo], size = P.fn_size0[lo];
    uint64_t rec = 0;
    uint32_t out = 0;
    if (i >= st && i - st < size && P.used_instrs[i]) {
        const uint32_t ins = P.instr[i], j = P.jt[i];
        uint32_t hi = kSUsed;
        if (ins == 0x000000EFu && (j < st || j - st >= size)) hi |= kSCall;
        if (s_needs_float(ins, 0)) hi |= kSFloatRd;
        if (s_needs_float(ins, 1)) hi |= kSFloatOp;
        rec = 0;
        uint32_t code[3] = {kCodeNone, kCodeNone, kCodeNone};
        if (rd >= 64u) {
            if (rd - 64u == i) hi |= kSDef;
            else out = 2u;
        } else {
            code[0] = code_of(rd);
            if (rd >= 32u && ((kNonscratchRegisters >> rd) & 1ull)) out = 2u;  // not in the 32-bit live mask
        }
        for (int k = 0; k < 2; ++k) {
            if (op[k] < 64u) {
                code[k + 1] = code_of(op[k]);
                continue;
            }
            const uint32_t x = op[k] - 64u;
            if (x == i) hi |= kSSelf;
            if (x >= i) continue;  // not defined yet: reads and writes the initial state
            if (i - x >= kScalarDist) out = 2u;
            rec |= static_cast<uint64_t>((i - x) & (kScalarDist - 1u)) << (20 * k);
        }
        rec |= static_cast<uint64_t>(code[0]) << 40 | static_cast<uint64_t>(code[1]) << 46 |
               static_cast<uint64_t>(code[2]) << 52 | static_cast<uint64_t>(hi) << 32;
    }
    P.rec[i] = rec;
    return out;
}
PTL_HD uint32_t st_scalar_range(const Prog& P, uint32_t f) {
    return s_ra_function_ok(P, f) ? st_step_range(P, f) : 2u;  // the other forms report the error
}

// Function f (past the end: nothing but the other lanes' turns; a whole warp calls this).
// Ring entries as in the lane-0 pass; oidx[p * ostride]: the word whose symbol position p
// holds.
PTL_HD void step_scalar_function(const Prog& P, uint32_t f, uint8_t* ring, uint32_t stride, uint32_t K, uint32_t* oidx,
                                 uint32_t ostride, unsigned long long* preserve) {
    const bool real = f < P.F;
    const uint32_t start = real ? P.fn_start0[f] : 0u, n = real ? P.fn_size0[f] : 0u, mask = K - 1u;
    const unsigned long long* rec = P.rec + start;
    uint32_t* symreg = P.symreg + start;
    uint32_t* symswp = P.symswp + start;
    uint32_t live = kLiveInit, held = 0, marked = 0, kept = 0;
#if defined(__CUDA_ARCH__)
    const uint32_t steps = __reduce_max_sync(0xFFFFFFFFu, n);
#else
    const uint32_t steps = n;
#endif
    constexpr uint32_t kAhead = 4;
    unsigned long long next[kAhead];
#pragma unroll
    for (uint32_t k = 0; k < kAhead; ++k) next[k] = k < n ? rec[k] : 0ull;
    for (uint32_t b = 0; b < steps; b += kAhead) {
        unsigned long long now[kAhead];
#pragma unroll
        for (uint32_t k = 0; k < kAhead; ++k) {
            now[k] = next[k];
            next[k] = b + kAhead + k < n ? rec[b + kAhead + k] : 0ull;
        }
#pragma unroll
        for (uint32_t k = 0; k < kAhead; ++k) {
            const uint32_t i = b + k;
            const uint32_t hi = static_cast<uint32_t>(now[k] >> 32);
            const uint32_t d1 = static_cast<uint32_t>(now[k]) & (kScalarDist - 1u);
            const uint32_t d2 = static_cast<uint32_t>(now[k] >> 20) & (kScalarDist - 1u);
            const bool used = (hi & kSUsed) != 0, call = (hi & kSCall) != 0;
            uint32_t e1 = ring[((i - d1) & mask) * stride], e2 = ring[((i - d2) & mask) * stride];
            // seldom: an operand older than the ring, or one whose register has moved
            const bool old = (d1 | d2) >= K;
            const bool rare = warp_any(old || ((d1 ? e1 : 0u) | (d2 ? e2 : 0u)) & kSymMoved);
            if (PTL_RARE(rare)) {
                if (d1 >= K) e1 = code_of(symreg[i - d1]) | (symswp[i - d1] ? kSymSwapped : 0u) | kSymMoved;
                if (d2 >= K) e2 = code_of(symreg[i - d2]) | (symswp[i - d2] ? kSymSwapped : 0u) | kSymMoved;
            }
            e1 = d1 ? e1 : (hi >> 14) & 63u;
            e2 = d2 ? e2 : (hi >> 20) & 63u;
            e1 = used ? e1 : kCodeNone;
            e2 = used ? e2 : kCodeNone;
            // an operand symbol's position: the one it was defined in, while it is held
            uint32_t m1 = d1 && oidx[(e1 & 31u) * ostride] == i - d1 ? code_bit(e1 & 63u) & held : 0u;
            uint32_t m2 = d2 && oidx[(e2 & 31u) * ostride] == i - d2 ? code_bit(e2 & 63u) & held : 0u;
            if (PTL_RARE(rare)) {
                for (uint32_t m = held; m; m &= m - 1) {
                    const uint32_t x = oidx[low_bit(m) * ostride], bit = m & (~m + 1u);
                    if (d1 && x == i - d1) m1 = bit;
                    if (d2 && x == i - d2) m2 = bit;
                }
            }
            const bool fop = (hi & kSFloatOp) != 0;
            const uint32_t c1 = (e1 & kSymSwapped) || (m1 & marked) ? (fop ? 0u : 5u) : e1 & 63u;
            const uint32_t c2 = (e2 & kSymSwapped) || (m2 & marked) ? (fop ? kCode38 : 6u) : e2 & 63u;
            // step_allocate's fields in their places of a lane-0 record's high word
            const StepOut o = step_allocate(((hi & kSDef) ? kStepDef : 0u) | ((hi & kSFloatRd) ? kStepFloat : 0u) |
                                                (used ? ((hi >> 8) & 63u) << 16 : kCodeNone << 16),
                                            live, c1, c2);
            const bool def = (hi & (kSDef | kSSelf)) == kSDef && !call;
            if (i < n) ring[(i & mask) * stride] = static_cast<uint8_t>((def ? o.rd : kCodeNone) | ((hi & kSSelf) ? kSymMoved : 0u));
            if (def) symreg[i] = o.rd ? o.rd : 37u;
            const bool s1 = d1 && d1 != d2 && e1 != c1 && !call, s2 = d2 && e2 != c2 && !call;
            // swapped: the held symbols of the triggered registers, but those just read; a
            // call triggers the caller-saved ones
            const uint32_t trig = call ? live & ~kScalarPreserved : o.trig;
            live = call ? live & kScalarPreserved : o.live;
            marked = (marked | (held & trig)) & ~(call ? 0u : m1 | m2);
            const uint32_t gone = call ? ~live : code_bit(o.rd) | code_bit(c1) | code_bit(c2);
            uint32_t t = held & marked & gone;  // swapped symbols that leave their positions
            if (warp_any(s1 || s2 || t != 0)) {
                if (s1) {
                    if (d1 < K)
                        ring[((i - d1) & mask) * stride] =
                            static_cast<uint8_t>(c1 | ((e1 & kSymMoved) || c1 != (e1 & 63u) ? kSymMoved : 0u));
                    symreg[i - d1] = reg_of(c1);
                    if (e1 & kSymSwapped) symswp[i - d1] = 0;
                }
                if (s2) {
                    if (d2 < K)
                        ring[((i - d2) & mask) * stride] =
                            static_cast<uint8_t>(c2 | ((e2 & kSymMoved) || c2 != (e2 & 63u) ? kSymMoved : 0u));
                    symreg[i - d2] = reg_of(c2);
                    if (e2 & kSymSwapped) symswp[i - d2] = 0;
                }
                for (; t; t &= t - 1) {
                    const uint32_t idx = oidx[low_bit(t) * ostride];
                    symswp[idx] = 0xFFFFFFFFu;
                    if (i - idx < K) ring[(idx & mask) * stride] |= kSymSwapped;
                }
            }
            held &= ~gone;
            marked &= held;
            if ((hi & kSDef) && !call) {
                oidx[o.rd * ostride] = i;
                held |= code_bit(o.rd);
            }
            kept |= live;
        }
    }
    for (uint32_t m = held & marked; m; m &= m - 1) symswp[oidx[low_bit(m) * ostride]] = 0xFFFFFFFFu;
    if (real) preserve[f] = kept & static_cast<uint32_t>(kNonscratchRegisters);
}

}  // namespace ptl
