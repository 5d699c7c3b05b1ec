// The lane-0 functions of register allocation in chunks of steps that run side by side.
//
// In lock-step (lane_step_a .. lane_step_b2, ptl_steps.cuh) a lane-0 function waits at
// every step for all others: one thread-block or cluster is busy, for 1,000 to 5,700 cycles
// a step.  What a function needs of the others is little, though: per step and position,
// the least and the greatest group that triggers it, the greatest that writes it, and
// whether any does (a row).  So all chunks of all functions run at once, each from a
// guessed start state and guessed rows; then the rows are folded again from what the runs
// wrote and triggered, and the chunks whose rows or start state have changed run again,
// until nothing changes.
//
// The result is the lock-step's: a step's writes and triggers depend on the steps before
// it, and within the step on triggers of lower groups, so by induction over (step, group)
// only one assignment of rows and states agrees with itself.  A wrong guess dies out fast
// because a state forgets: an expression's values are read once, soon, and the live mask
// fills up (registers whose symbol was read swapped are never freed).  For that a state
// only holds what can still matter: a symbol is dropped at its last read, which the
// records tell.  Rounds until nothing changes: 10 for 18 chunks of one function, 30 for
// 148 of 64, 100 for 175 of 1,229 (with dead symbols in the state, three times as many).
// What becomes of a dead symbol in row 0 is found in a last pass, when the rows are final.
//
// A chunk's run is a chain of 32 dependent steps of about 650 cycles (a lone warp; 32
// functions side by side take little longer), so what bounds the allocation is rounds times
// a run, and for wide programs the folds (ptl_chunks.cu).  Chunks of 64 steps took fewer
// rounds but more steps in all (26 x 64 against 32 x 32 for 64 functions), chunks of 16
// more rounds (41), each with its fold and waits.  Before and after, the whole allocation:
// 1.46 to 0.65 ms (two lane-0 functions of 1,449 steps), 4.18 to 1.80 (64 of 2,830), 11.7
// to 3.5 (256 of 8,151), 12.7 to 9.1 (1,229 of 4,072).
#pragma once

#include "ptl_steps.cuh"

namespace ptl {

constexpr uint32_t kChunk = kRowTile;  // steps; a row tile per chunk
constexpr uint32_t kLiveGuess = 0xFFFFFFFEu;

// Symbols live in slots: a symbol takes the lowest free one at its definition and gives it
// back at its last read (step_slot_chunk), so a state is a few slots however far apart
// definition and read are.  Slot 0 always reads as "no symbol".  A program with more than
// kSlots - 1 symbols alive at once runs in lock-step.
//
// A slot holds the symbol's register code (bits 0-5), whether it is swapped (6) and the
// row-0 position of its definition (8-12).  For each position, oidx tells the slot whose
// symbol row 0 has there (the function's held mask tells whether one is).  Both are 16-bit
// halves of words laid out [word][lane], so a warp's lanes never meet in a bank; a slot is
// named by the byte offset of its half.
constexpr uint32_t kSlots = 64u, kChunkLanes = 32u;
PTL_HD uint32_t slot_at(uint32_t k) { return (k >> 1) * (kChunkLanes * 4u) + (k & 1u) * 2u; }
PTL_HD uint32_t slot_of(uint32_t at) { return (at >> 7) * 2u + ((at >> 1) & 1u); }
constexpr uint32_t kOidxAt = kSlots / 2u * kChunkLanes * 4u;
constexpr uint32_t kOidxWords = kRowPos / 2u;
constexpr uint32_t kChunkMemWords = (kSlots + kRowPos) / 2u * kChunkLanes;
// Slot records, 8 bytes a word and 32 of them an item: operands' slots in the halves of
// the low word; the own symbol's slot in bits 0-15 of the high word (0: never read), above
// it the fields of a step record and whether this is the operand symbols' last read.
constexpr uint32_t kStepLast1 = 1u << 25, kStepLast2 = 1u << 26;

// A state in memory, in vectors of 16 bytes: live, held, marked, 0; oidx (0 where nothing
// is held); the function's slots.  A state may be read while its writer, in the same
// round, is at it: the reader then runs again in the next round, and whatever mixture it
// saw names only slots and positions that exist.
struct alignas(16) ChunkVec {
    uint32_t v[4];
};
PTL_HD bool operator!=(const ChunkVec& a, const ChunkVec& b) {
    return ((a.v[0] ^ b.v[0]) | (a.v[1] ^ b.v[1]) | (a.v[2] ^ b.v[2]) | (a.v[3] ^ b.v[3])) != 0;
}
constexpr uint32_t kOidxVecs = kOidxWords / 4u, kStateVecs = 1u + kOidxVecs + kSlots / 8u;
#if defined(__CUDA_ARCH__)
// Other SMs write states, outputs and rows between rounds: past the L1.
__device__ __forceinline__ ChunkVec chunk_load(const ChunkVec* p) {
    const uint4 x = __ldcg(reinterpret_cast<const uint4*>(p));
    return ChunkVec{{x.x, x.y, x.z, x.w}};
}
__device__ __forceinline__ void chunk_store(ChunkVec* p, const ChunkVec& v) {
    __stcg(reinterpret_cast<uint4*>(p), make_uint4(v.v[0], v.v[1], v.v[2], v.v[3]));
}
#else
inline ChunkVec chunk_load(const ChunkVec* p) { return *p; }
inline void chunk_store(ChunkVec* p, const ChunkVec& v) { *p = v; }
#endif

// The rows of a chunk's steps: [kChunk][kRowPos] triggers (as P.trow, lane-0 functions
// included), [kChunk][kRowPos] greatest writing group + 1, [kChunk] positions triggered
// and written at all.
struct ChunkRows {
    const uint32_t* row;
    const uint16_t* win;
    const ChunkPair* pair;
};

PTL_HD uint32_t chunks_of(const Prog& P, uint32_t j) {
    const int32_t size = s32(P.fn_size0[8u * j]);
    return size > 0 ? (static_cast<uint32_t>(size) + kChunk - 1u) / kChunk : 0u;
}

PTL_HD void chunk_max(uint32_t* p, uint32_t v) {
#if defined(__CUDA_ARCH__)
    atomicMax(p, v);
#else
    if (*p < v) *p = v;
#endif
}
// Step i of lane-0 function 8j: the last word that reads each symbol, and for each chunk how
// far the symbols from before it reach (last, reach: zero before).
constexpr uint32_t kChunkReach = 256u;  // chunks a symbol may live through (else the lock-step)
PTL_HD void chunk_last_read(const Prog& P, uint32_t j, uint32_t i) {
    const uint32_t start = P.fn_start0[8u * j];
    const uint64_t r = P.rec[start + i];
    const uint32_t d[2] = {step_d1(r), step_d2(r)};
    for (int k = 0; k < 2; ++k) {
        if (!d[k]) continue;
        chunk_max(&P.ch.last[start + i - d[k]], start + i);
        const uint32_t to = i / kChunk;
        uint32_t c = (i - d[k]) / kChunk + 1u;
        if (to >= c + kChunkReach) {
            *P.ch.lock = 1u;
            continue;
        }
        for (; c <= to; ++c) chunk_max(&P.ch.reach[P.ch.off[j] + c], start + i);
    }
}

// Slot records.  Between two steps where no symbol is alive (statements mostly) the slots
// are a matter of their own, so a thread takes the stretches that begin in chunk c of
// function 8j, from its first such point to the first one behind it (ring: the last words'
// slots).  One thread per function instead took 528 cycles a step, and as long as the
// independent functions and more (9,275 steps: the allocation 4.7 ms, now 3.8).  Sets *lock if the
// slots do not suffice.
PTL_HD void step_slot_chunk(const Prog& P, uint32_t j, uint32_t c, uint8_t* ring, uint32_t stride, uint32_t K) {
    const uint32_t start = P.fn_start0[8u * j], n = P.fn_size0[8u * j], base = c * kChunk, mask = K - 1u;
    const unsigned long long* rec = P.rec + start;
    const uint32_t* last = P.ch.last + start;
    unsigned long long* out = P.ch.rec + static_cast<size_t>(P.ch.off[j]) * kChunk;
    uint32_t i = base;
    if (c) {
        uint32_t alive = P.ch.reach[P.ch.off[j] + c];  // to the last read of any symbol so far
        for (; i < n && i < base + kChunk && alive >= start + i; ++i) alive = alive > last[i] ? alive : last[i];
        if (i >= n || i >= base + kChunk) return;
    }
    uint64_t open = ~1ull;
    uint32_t most = 0;
    bool full = false;
    for (; i < n && (i < base + kChunk || open != ~1ull); ++i) {
        const uint64_t now = rec[i];
        const uint32_t d1 = step_d1(now), d2 = step_d2(now);
        uint32_t s1 = ring[((i - d1) & mask) * stride], s2 = ring[((i - d2) & mask) * stride];
        if (d1 >= K) s1 = slot_of(static_cast<uint32_t>(out[i - d1] >> 32) & 0xFFFFu);
        if (d2 >= K) s2 = slot_of(static_cast<uint32_t>(out[i - d2] >> 32) & 0xFFFFu);
        s1 = d1 ? s1 : 0u;
        s2 = d2 ? s2 : 0u;
        const bool last1 = !d1 || last[i - d1] == start + i, last2 = !d2 || last[i - d2] == start + i;
        if (last1) open |= (1ull << s1) & ~1ull;
        if (last2) open |= (1ull << s2) & ~1ull;
        uint32_t own = 0;
        if (last[i]) {
            const uint32_t low = static_cast<uint32_t>(open), high = static_cast<uint32_t>(open >> 32);
            if (open) own = low ? low_bit(low) : 32u + low_bit(high);
            else full = true;
            open &= ~((1ull << own) & ~1ull);
            most = own > most ? own : most;
        }
        ring[(i & mask) * stride] = static_cast<uint8_t>(own);
        // (rd's code, 6 bits, and the flags are bits 48-56 of both records)
        out[i] = static_cast<uint64_t>(slot_at(s1)) | static_cast<uint64_t>(slot_at(s2)) << 16 |
                 static_cast<uint64_t>(slot_at(own)) << 32 | ((now >> 48 & 0x1FFull) << 48) |
                 static_cast<uint64_t>((last1 ? kStepLast1 : 0u) | (last2 ? kStepLast2 : 0u)) << 32;
        if (full) break;
    }
    chunk_max(&P.ch.slots[j], most + 1u);
    if (full) *P.ch.lock = 1u;
}

// Whether the dead symbol that row 0 holds at position p after step t - 1 ends swapped: it
// does if any function triggers the position before one writes it.  A position may see
// neither for thousands of steps (a search step by step took up to 2 ms), so tiles without
// are skipped.
PTL_HD bool chunk_fate(const Prog& P, uint32_t t, uint32_t p) {
    const uint32_t tiles = static_cast<uint32_t>(row_tiles(P.S));
    for (;;) {
        for (; t % kRowTile; ++t) {
            const ChunkPair x = P.ch.pair[t];
            if ((x.any >> p) & 1u) return true;
            if ((x.wr >> p) & 1u) return false;
        }
        uint32_t c = t / kRowTile;
#pragma unroll 4
        while (c < tiles && !((P.ch.touch[c] >> p) & 1u)) ++c;
        if (c >= tiles) return false;
        t = c * kRowTile;
        const ChunkPair x = P.ch.pair[t];
        if ((x.any >> p) & 1u) return true;
        if ((x.wr >> p) & 1u) return false;
        ++t;
    }
}

// Steps [kChunk * c, + kChunk) of slot j (nothing if not on; a whole warp calls this, c
// the same).  first: there is no state and no output yet.  kFinal: write the symbols'
// registers and swaps instead of the outputs and the next chunk's state.  mem: this lane's
// column of kChunkMemWords.  Returns bit 0: outputs changed, bit 1: the next chunk's start
// state changed.
constexpr uint32_t kChunkOut = 1u, kChunkNext = 2u;
template <bool kFinal>
PTL_HD uint32_t chunk_run(const Prog& P, const ChunkRows& rows, uint32_t* mem, uint32_t j, uint32_t c, bool on, bool first) {
    const uint32_t base = c * kChunk;
    const uint32_t start = on ? P.fn_start0[8u * j] : 0u, size = on ? P.fn_size0[8u * j] : 0u;
    const uint32_t n = on ? (size - base < kChunk ? size - base : kChunk) : 0u;
    const uint32_t vecs = on ? kOidxVecs + (P.ch.slots[j] + 7u) / 8u : 0u;
    const size_t item = on ? P.ch.off[j] + c : 0u;
    const ChunkVec* rec = reinterpret_cast<const ChunkVec*>(P.ch.rec) + item * (kChunk / 2u);
    ChunkVec* out = reinterpret_cast<ChunkVec*>(P.ch.out) + item * (kChunk / 2u);
    uint8_t* const sym = reinterpret_cast<uint8_t*>(mem);
    uint8_t* const oidx = sym + kOidxAt;
    auto half = [](uint8_t* p) -> uint16_t& { return *reinterpret_cast<uint16_t*>(p); };
    uint32_t live = c ? kLiveGuess : kLiveInit, held = 0, marked = 0, result = first ? kChunkOut : 0u;
    // word w of a state's vectors: oidx first, then the slots
    auto word = [&](uint32_t w) -> uint32_t& {
        return mem[(w < kOidxWords ? kOidxAt / 4u + w * kChunkLanes : (w - kOidxWords) * kChunkLanes)];
    };
    ChunkVec next[2] = {};
    if (on) {
        next[0] = rec[0];
        next[1] = rec[1];
    }
    if (c == 0 || first) {
        for (uint32_t w = 0; w < 4u * vecs; ++w) word(w) = w < kOidxWords ? 0u : kCodeNone * 0x00010001u;
    } else if (on) {
        const ChunkVec* st = reinterpret_cast<const ChunkVec*>(P.ch.state) + item * kStateVecs;
        const ChunkVec h = chunk_load(st);
        live = h.v[0];
        held = h.v[1];
        marked = h.v[2];
#pragma unroll 6
        for (uint32_t q = 0; q < vecs; ++q) {
            const ChunkVec x = chunk_load(st + 1u + q);
#pragma unroll
            for (uint32_t k = 0; k < 4u; ++k) word(4u * q + k) = x.v[k];
        }
    }
    half(sym) = kCodeNone;
#pragma unroll 1
    for (uint32_t b = 0; b < kChunk; b += 4u) {
        const ChunkVec now[2] = {next[0], next[1]};
        ChunkVec was[2] = {}, is[2];
        if (on) {
            const uint32_t ahead = b + 4u < kChunk ? b / 2u + 2u : b / 2u;
            next[0] = rec[ahead];
            next[1] = rec[ahead + 1u];
            if (!kFinal && !first) {
                was[0] = chunk_load(out + b / 2u);
                was[1] = chunk_load(out + b / 2u + 1u);
            }
        }
#pragma unroll
        for (uint32_t k = 0; k < 4u; ++k) {
            const uint32_t t = b + k, i = base + t;
            const bool in = t < n;
            const uint32_t lo = in ? now[k / 2u].v[2u * (k & 1u)] : 0u;
            const uint32_t hi = in ? now[k / 2u].v[2u * (k & 1u) + 1u] : (kCodeNone << 16 | kStepLast1 | kStepLast2);
            const uint32_t s1 = lo & 0xFFFFu, s2 = lo >> 16, s0 = hi & 0xFFFFu;
            const uint32_t* row = rows.row + t * kRowPos;
            const ChunkPair pair = rows.pair[t];
            const uint32_t e1 = half(sym + s1), e2 = half(sym + s2);
            const uint32_t p1 = e1 >> 8, p2 = e2 >> 8;
            const uint32_t row1 = row[p1], row2 = row[p2];
            const uint32_t m1 = half(oidx + slot_at(p1)) == s1 ? (1u << p1) & held : 0u;
            const uint32_t m2 = half(oidx + slot_at(p2)) == s2 ? (1u << p2) & held : 0u;
            const bool b1 = m1 && row_min(row1) <= j, b2 = m2 && row_min(row2) <= j;
            const bool l1 = m1 && row_max(row1) > j + 1u, l2 = m2 && row_max(row2) > j + 1u;
            const bool fop = (hi & kStepFloat) != 0;
            const uint32_t c1 = ((e1 & kSymSwapped) || (m1 & marked) || b1) ? (fop ? 0u : 5u) : (e1 & 63u);
            const uint32_t c2 = ((e2 & kSymSwapped) || (m2 & marked) || b2) ? (fop ? kCode38 : 6u) : (e2 & 63u);
            const StepOut o = step_allocate(hi, live, c1, c2);
            const uint32_t own = code_bit(o.rd) | code_bit(c1) | code_bit(c2);
            is[k / 2u].v[2u * (k & 1u)] = own;
            is[k / 2u].v[2u * (k & 1u) + 1u] = o.trig;
            live = o.live;
            // the symbols after the step: a last read empties the slot, which the own one
            // may take
            const bool def = (hi & (kStepDef | kStepSelf)) == kStepDef;
            const bool last1 = (hi & kStepLast1) != 0, last2 = (hi & kStepLast2) != 0;
            half(sym + s1) = static_cast<uint16_t>(last1 ? kCodeNone : c1 | (e1 & 0xFF00u));
            half(sym + s2) = static_cast<uint16_t>(last2 ? kCodeNone : c2 | (e2 & 0xFF00u));
            half(sym + s0) = static_cast<uint16_t>(s0 ? (def ? o.rd : kCodeNone) | (o.rd & 31u) << 8 : kCodeNone);
            // swaps and row 0 after the step; a symbol that was read for the last time is
            // forgotten
            const uint32_t operands = m1 | m2, gone = (last1 ? m1 : 0u) | (last2 ? m2 : 0u), wr = pair.wr | own;
            marked = (marked & ~operands) | (l1 ? m1 : 0u) | (l2 ? m2 : 0u) | (held & ~operands & (pair.any | o.trig));
            const bool wins = (hi & kStepDef) && rows.win[t * kRowPos + (o.rd & 31u)] <= j + 1u;
            if (kFinal && in) {
                const uint64_t r = P.rec[start + i];
                const uint32_t x1 = start + i - step_d1(r), x2 = start + i - step_d2(r);
                if (def && !s0) P.symreg[start + i] = o.rd ? o.rd : 37u;
                if (s1 && s1 != s2 && last1) P.symreg[x1] = reg_of(c1);
                if (s2 && last2) P.symreg[x2] = reg_of(c2);
                // dead symbols: in row 0 and swapped, or to be swapped there
                auto fate = [&](uint32_t m, uint32_t x) {
                    if (m && ((m & marked) || (!(m & wr) && chunk_fate(P, i + 1u, low_bit(m))))) P.symswp[x] = 0xFFFFFFFFu;
                };
                if (last1) fate(m1, x1);
                if (last2) fate(m2, x2);
                if (!s0 && wins && chunk_fate(P, i + 1u, o.rd)) P.symswp[start + i] = 0xFFFFFFFFu;
            }
            held &= ~gone;
            marked &= held;
            uint32_t leave = marked & wr;
            while (PTL_RARE(warp_any(leave != 0))) {
                if (leave) {
                    half(sym + half(oidx + slot_at(low_bit(leave)))) |= kSymSwapped;
                    leave &= leave - 1;
                }
            }
            held &= ~wr;
            marked &= held;
            if (wins && s0) {  // row 0 keeps the write of the highest group
                half(oidx + slot_at(o.rd)) = static_cast<uint16_t>(s0);
                held |= code_bit(o.rd);
            }
        }
        if (!kFinal && on) {
#pragma unroll
            for (uint32_t k = 0; k < 2u; ++k) {
                if (first || is[k] != was[k]) {
                    chunk_store(out + b / 2u + k, is[k]);
                    result |= kChunkOut;
                    if (!first) {
#pragma unroll
                        for (uint32_t w = 0; w < 4u; ++w) {
                            const uint32_t d = is[k].v[w] ^ was[k].v[w];
                            if (d) or_u32(P.ch.delta + 2u * (base + b + 2u * k) + w, d);
                        }
                    }
                }
            }
        }
    }
    if (!on) return 0;
    if (!kFinal && base + kChunk < size) {
        ChunkVec* st = reinterpret_cast<ChunkVec*>(P.ch.state) + (item + 1u) * kStateVecs;
        const ChunkVec h{{live, held, marked, 0}};
        if (first || h != chunk_load(st)) {
            chunk_store(st, h);
            result |= kChunkNext;
        }
#pragma unroll 6
        for (uint32_t q = 0; q < vecs; ++q) {
            ChunkVec x;
#pragma unroll
            for (uint32_t k = 0; k < 4u; ++k) {
                const uint32_t w = 4u * q + k;
                x.v[k] = word(w);
                if (w < kOidxWords)
                    x.v[k] &= (((held >> (2u * w)) & 1u) ? 0xFFFFu : 0u) | (((held >> (2u * w + 1u)) & 1u) ? 0xFFFF0000u : 0u);
            }
            if (first || x != chunk_load(st + 1u + q)) {
                chunk_store(st + 1u + q, x);
                result |= kChunkNext;
            }
        }
    }
    return result;
}

// What a launch whose blocks have lost one another leaves: none of its programs has its
// lane-0 functions allocated, so the error is every program's (one without it would go on,
// with registers that nothing allocated).  Done by thread `thread` of `threads`.
template <class ProgramOf>
PTL_HD void chunks_lost(const ProgramOf& program, uint32_t n, uint32_t thread, uint32_t threads, uint32_t round) {
    for (uint32_t k = thread; k < n; k += threads) record_error(program(k).err, ST_DEVICE_TIMEOUT, W_RA2, round);
}

}  // namespace ptl
