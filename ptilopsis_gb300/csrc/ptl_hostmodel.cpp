// Host model of the GPU pipeline -- test-only build.
//
// Runs the per-thread stage functions of ptl_stages.cuh / ptl_sort.cuh sequentially on
// the CPU, with sequential versions of the cross-thread steps (scans, the depth-order
// rounds, the lock-step lane-0 allocator).  The CPU test suite compares it with the
// oracle so the GPU algorithm is checked before it runs on a GPU.  The library API
// never calls it: without the CUDA library the package refuses to compile anything.
#include <algorithm>
#include <array>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <stdexcept>
#include <vector>

#include "ptl_common.cuh"
#include "ptl_sort.cuh"
#include "ptl_stages.cuh"
#include "ptl_ra.cuh"
#include "ptl_chunks.cuh"
#include "ptl_flatten.cuh"
#include "ptl_scalar.cuh"

using namespace ptl;

namespace {

bool g_last_locked = false;  // the last program's symbols did not fit the slots
bool g_chunks = true;  // lane-0 functions in chunks (else in lock-step)
uint32_t g_chunk_rounds = 0;  // rounds of the chunks at most (0: the kernel's limit)
bool g_last_lock_step = false;  // the last program's lane-0 functions went in lock-step
uint32_t g_ring_k = 16;  // words per function in the record form's symbol ring (small: old words too)
uint32_t g_cache_k = 4;  // entries per function of the lane-0 symbol cache
bool g_force_general = false; // the general form for every program
bool g_force_hashed = false;  // ... which finds row-0 values by hashing even when definitions are unique
bool g_last_hashed = false;   // the last compile did
bool g_last_cross = false;    // the last scalar compile took the serial register allocation
bool g_force_tiles = false;   // scalar register allocation by word tiles for every program
bool g_force_serial = false;  // scalar register allocation in the reference's order for every program

template <typename T>
struct HBuf {
    std::vector<T> v;
    T* p = nullptr;
    size_t n = 0;
    void ensure(size_t count, T fill = T{}) {
        n = count;
        v.assign(count + 16 + 80, fill);
        p = v.data() + 16;
    }
};

inline size_t r8(size_t n) { return (n + 7) & ~size_t(7); }

struct Model {
    CodeTables tab;
    ErrorWord err{};
    uint32_t flags[4] = {0, 0, 0, 0};
    HBuf<uint8_t> in_type, in_rtype, fflag, used, smark, defpos, nt, rt;
    HBuf<int32_t> in_parent, in_depth, in_child, par, ci, dep;
    HBuf<uint32_t> in_data, nd1, nd, sizes, loc0, loc, regs, pos, decl, fn_id, fn_start, fn_size,
        fn_end, fn_start0, fn_size0, fn_end0, fn_ra_start, fn_ra_end, fn_ra_size, instr, rd, rs1, rs2, jt,
        used_instrs, symreg, symswp, stamp, trig_min, trig_max, spill, roffs, ni, nrd, nr1, nr2, njt, fsz,
        joffs, out;
    HBuf<unsigned long long> owner, lifetime;
    HBuf<uint32_t> tmask, tany, trow;
    Prog P{};

    void bind() {
        P.in_type = in_type.p; P.in_rtype = in_rtype.p; P.in_parent = in_parent.p; P.in_depth = in_depth.p;
        P.in_child = in_child.p; P.in_data = in_data.p;
        P.nt = nt.p; P.rt = rt.p; P.nd1 = nd1.p; P.nd = nd.p; P.par = par.p; P.ci = ci.p; P.dep = dep.p;
        P.fflag = fflag.p; P.sizes = sizes.p; P.loc0 = loc0.p; P.loc = loc.p; P.regs = regs.p; P.pos = pos.p;
        P.owner = owner.p; P.rec = owner.p; P.tmask = tmask.p; P.tany = tany.p; P.trow = trow.p; P.decl = decl.p; P.fn_id = fn_id.p; P.fn_start = fn_start.p; P.fn_size = fn_size.p;
        P.fn_end = fn_end.p; P.fn_start0 = fn_start0.p; P.fn_size0 = fn_size0.p; P.instr = instr.p;
        P.rd = rd.p; P.rs1 = rs1.p; P.rs2 = rs2.p; P.jt = jt.p; P.used = used.p; P.smark = smark.p;
        P.used_instrs = used_instrs.p; P.symreg = symreg.p; P.symswp = symswp.p; P.stamp = stamp.p;
        P.defpos = defpos.p;
        P.lifetime = lifetime.p; P.trig_min = trig_min.p; P.trig_max = trig_max.p; P.spill = spill.p;
        P.roffs = roffs.p; P.ni = ni.p; P.nrd = nrd.p; P.nr1 = nr1.p; P.nr2 = nr2.p; P.njt = njt.p;
        P.fsz = fsz.p; P.joffs = joffs.p; P.out = out.p;
        P.tab.t = &tab;
        P.err = &err;
        P.flags = flags;
    }

    template <class F>
    static void exclusive_scan(uint32_t count, F load, uint32_t* out) {
        uint32_t acc = 0;
        for (uint32_t i = 0; i < count; ++i) {
            const uint32_t v = load(i);
            out[i] = acc;
            acc += v;
        }
    }

    bool check() { return err.code == 0; }

    // Depth-order emulation with the same round structure as the kernels.
    void depth_sort(uint32_t n) {
        std::vector<unsigned long long> a(n);
        for (uint32_t i = 0; i < n; ++i) a[i] = (static_cast<unsigned long long>(static_cast<uint32_t>(dep.p[i])) << 32) | i;
        std::vector<uint32_t> apos(n), bpos(n);
        std::vector<SortSeg> cur, next;
        std::vector<std::pair<uint32_t, uint32_t>> leaves, heaps;
        std::vector<std::array<uint32_t, 3>> locals;
        std::vector<std::pair<uint32_t, uint32_t>> equal;
        auto emit = [&](uint32_t first, uint32_t last, uint32_t dl, bool eq) {
            if (eq && last - first <= kSortThreshold) return;  // a stable sort of equal keys
            if (eq && dl >= equal_levels(last - first)) { equal.push_back({first, last}); return; }
            if (last - first <= kSortThreshold) { if (last - first > 1) leaves.push_back({first, last}); return; }
            if (dl > 0 && last - first <= kSortBlock) { locals.push_back({first, last, dl}); return; }
            if (dl == 0) { heaps.push_back({first, last}); return; }
            SortSeg c{}; c.first = first; c.last = last; c.dl = dl;
            next.push_back(c);
        };
        if (n > 1) emit(0, n, 2u * floor_log2(n), false);  // the whole array: rounds, or one block
        cur.swap(next);
        while (!cur.empty()) {
            next.clear();
            for (SortSeg& g : cur) {
                median_to_first(a.data(), g.first, g.last);
                g.pivot = skey(a[g.first]);
                g.kmin = g.kmax = g.pivot;
                for (uint32_t p = g.first + 1; p < g.last; ++p) {
                    g.kmin = std::min(g.kmin, skey(a[p]));
                    g.kmax = std::max(g.kmax, skey(a[p]));
                }
                uint32_t nl = 0, nr_total = 0;
                for (uint32_t p = g.first + 1; p < g.last; ++p) nr_total += is_rstop(skey(a[p]), g.pivot);
                uint32_t rl = 0;
                for (uint32_t p = g.first + 1; p < g.last; ++p) {
                    const int32_t k = skey(a[p]);
                    if (is_lstop(k, g.pivot)) apos[g.first + nl++] = p;
                    if (is_rstop(k, g.pivot)) bpos[g.first + (nr_total - 1 - rl++)] = p;
                }
                g.nL = nl;
                g.nR = nr_total;
                g.K = partition_k(apos.data() + g.first, bpos.data() + g.first, g.nL, g.nR);
                g.cut = partition_cut(apos.data() + g.first, bpos.data() + g.first, g.nL, g.K);
                for (uint32_t k = 0; k < g.K; ++k) sswap(a.data(), apos[g.first + k], bpos[g.first + k]);
                emit(g.first, g.cut, g.dl - 1, g.kmin == g.pivot);
                emit(g.cut, g.last, g.dl - 1, g.kmax == g.pivot);
            }
            cur.swap(next);
        }
        for (auto& h : heaps) heap_sort_range(a.data() + h.first, h.second - h.first);
        for (auto& l : leaves) leaf_sort(a.data(), l.first, l.second);
        for (auto& r : locals) {  // one thread per range on the device, in a strided buffer
            std::vector<unsigned long long> buf(static_cast<size_t>(r[1] - r[0]) * 3);
            const Strided sb{buf.data() + 1, 3};
            for (uint32_t i = 0; i < r[1] - r[0]; ++i) sb[i] = a[r[0] + i];
            local_introsort(sb, 0u, r[1] - r[0], r[2]);
            for (uint32_t i = 0; i < r[1] - r[0]; ++i) a[r[0] + i] = sb[i];
        }
        for (auto& r : equal) {  // one block per range on the device, through apos
            const uint32_t m = r.second - r.first;
            for (uint32_t i = 0; i < m; ++i) apos[r.first + equal_final_index(i, m)] = sidx(a[r.first + i]);
            const unsigned long long key = a[r.first] & 0xFFFFFFFF00000000ull;
            for (uint32_t i = 0; i < m; ++i) a[r.first + i] = key | apos[r.first + i];
        }
        for (uint32_t p = 0; p < n; ++p) pos.p[sidx(a[p])] = p;
    }

    uint32_t hm_cache_k = g_cache_k;

    // The lane-0 pass with the same phase functions as k_ra_lane0_cached.
    void lane0_cached(uint32_t S, uint32_t K, bool hashed) {
        const uint32_t G0 = (P.F + 7) / 8;
        const Prog Psave = P;
        if (hashed) P.defpos = nullptr;
        Ra2Shared sh{};
        std::vector<uint32_t> cur(4 * G0), tag(static_cast<size_t>(G0) * K);
        std::vector<uint32_t> val(static_cast<size_t>(G0) * K);
        const SymCache c{tag.data(), val.data(), K};
        std::vector<Ra2Slot> L(G0);
        for (uint32_t j = 0; j < G0; ++j) {
            L[j].act = false;
            L[j].have_next = false;
            ra2_slot_init(P, c, L[j], j, j);
        }
        for (int p = 0; p < 64; ++p) { sh.R0[p] = 0xFFFFFFFFu; sh.R0own[p] = 0xFFFFFFFFu; }
        if (S > 0) for (uint32_t p = 0; p < 64; ++p) ra2_begin_p(sh, 0, p, P.trig_min[p], P.trig_max[p], hashed);
        uint32_t s0 = 0;  // steps with a lane-0 function still running
        for (uint32_t j = 0; j < G0; ++j) s0 = std::max(s0, ra2_lane0_size(L[j]));
        s0 = std::min(s0, S);
        for (uint32_t i = 0; i < s0; ++i) {
            bool in_row0 = false;
            for (uint32_t j = 0; j < G0; ++j) {
                ra2_load(P, L[j], i, cur.data() + 4 * j);
                in_row0 |= ra2_compute0(P, c, sh, L[j], j, i);
            }
            bool flag = false;
            if (in_row0) for (uint32_t j = 0; j < G0; ++j) flag |= ra2_check(sh, L[j]);
            for (uint32_t j = 0; j < G0; ++j) ra2_apply(P, c, sh, L[j], j, i, cur.data() + 4 * j);
            if (flag) {
                for (uint32_t p = 0; p < 64; ++p) sh.r0grp[p] = 0;
                for (uint32_t round = 0;; ++round) {
                    for (uint32_t j = 0; j < G0; ++j) ra2_round(sh, L[j]);
                    bool changed = false;
                    for (uint32_t p = 0; p < 64; ++p) changed |= ra2_round_p(sh, p);
                    if (!changed) break;
                    if (round > G0 + 2) { record_error(P.err, ST_DEVICE_TIMEOUT, W_RA2, i); break; }
                }
                for (uint32_t j = 0; j < G0; ++j) ra2_apply(P, c, sh, L[j], j, i, cur.data() + 4 * j);
            }
            if (hashed) for (uint32_t p = 0; p < 64; ++p) snap_clear_next(sh, i, p);
            for (uint32_t p = 0; p < 64; ++p) {
                ra2_end_p(P, c, sh, p, cur.data());
            }
            if (i + 1 < S) {
                for (uint32_t p = 0; p < 64; ++p) {
                    ra2_begin_p(sh, i + 1, p, P.trig_min[static_cast<size_t>(i + 1) * 64 + p],
                                P.trig_max[static_cast<size_t>(i + 1) * 64 + p], hashed);
                }
            }
        }
        {  // the steps after the last lane-0 function only mark row 0's symbols
            for (uint32_t p = 0; p < 64; ++p) ra2_tail_p(P, c, sh, p, s0, S);
        }
        P = Psave;
    }

    // The lane-0 functions in chunks (ptl_chunks.cuh), round by round as its kernel runs
    // them (the runs of a round one after the other).  False: the rounds ran out.
    bool chunk_lanes(uint32_t S, uint32_t K) {
        const uint32_t G0 = (P.F + 7) / 8, tiles = static_cast<uint32_t>(row_tiles(S)), rounds = g_chunk_rounds ? g_chunk_rounds : tiles + 64;
        const size_t steps = static_cast<size_t>(tiles) * kRowTile;
        auto size = [&](uint32_t j) { return static_cast<uint32_t>(std::max(s32(P.fn_size0[8 * j]), 0)); };
        std::vector<uint32_t> off(G0 + 1);
        for (uint32_t j = 0; j < G0; ++j) off[j + 1] = off[j] + chunks_of(P, j);
        const size_t items = off[G0];
        std::vector<uint32_t> last(P.W, 0), reach(items + 1, 0), slots(G0, 0), need(items + 1, 0), delta(2 * steps, 0), dirty(tiles, 0), moved(tiles, 0);
        std::vector<unsigned long long> rec(items * kChunk);
        std::vector<ChunkVec> out(items * kChunk / 2), state((items + 1) * kStateVecs);
        std::vector<uint32_t> row(steps * kRowPos), mem(kChunkMemWords);
        std::vector<uint16_t> win(steps * kRowPos);
        std::vector<ChunkPair> pair(steps);
        std::vector<uint32_t> touch(tiles, 0);
        uint32_t lock = 0;
        P.ch = LaneChunks{last.data(), reach.data(), off.data(), slots.data(), rec.data(), need.data(), out.data(), state.data(), row.data(),
                          win.data(), pair.data(), touch.data(), nullptr, delta.data(), dirty.data(), moved.data(), &lock};
        std::vector<uint8_t> ring(K);
        for (uint32_t j = 0; j < G0; ++j)
            for (uint32_t i = 0; i < size(j); ++i) chunk_last_read(P, j, i);
        for (uint32_t j = 0; j < G0; ++j)
            for (uint32_t c = 0; c < chunks_of(P, j); ++c) step_slot_chunk(P, j, c, ring.data(), 1, K);
        g_last_locked = lock != 0;
        if (lock) return false;
        const std::vector<uint16_t> no_win(kChunk * kRowPos, 0);
        for (uint32_t round = 1;; ++round) {
            const bool first = round == 1;
            bool changed = false;
            for (uint32_t c = 0; c < tiles; ++c) {
                const size_t at = static_cast<size_t>(c) * kChunk;
                std::vector<ChunkPair> none(kChunk);
                for (uint32_t t = 0; t < kChunk; ++t) none[t] = ChunkPair{P.tany[at + t], 0};
                const ChunkRows rows = first ? ChunkRows{P.trow + at * kRowPos, no_win.data(), none.data()}
                                             : ChunkRows{&row[at * kRowPos], &win[at * kRowPos], &pair[at]};
                for (uint32_t j = 0; j < G0; ++j) {
                    if (size(j) <= c * kChunk || !(first || moved[c] == round || need[off[j] + c] >= round)) continue;
                    const uint32_t r = chunk_run<false>(P, rows, mem.data(), j, c, true, first);
                    if (r & kChunkNext) { need[off[j] + c + 1] = round + 1; changed = true; }
                    if (r & kChunkOut) dirty[c] = round;
                }
            }
            for (uint32_t c = 0; c < tiles; ++c) {
                if (!first && dirty[c] != round) continue;
                for (uint32_t t = 0; t < kChunk; ++t) {
                    const size_t i = static_cast<size_t>(c) * kChunk + t;
                    ChunkPair x{P.tany[i], 0};
                    std::vector<uint32_t> r(P.trow + i * kRowPos, P.trow + (i + 1) * kRowPos);
                    uint16_t w[kRowPos] = {};
                    for (uint32_t j = 0; j < G0; ++j) {
                        if (size(j) <= c * kChunk) continue;
                        const uint32_t* o = reinterpret_cast<const uint32_t*>(out.data()) + (static_cast<size_t>(off[j] + c) * kChunk + t) * 2;
                        x.wr |= o[0];
                        x.any |= o[1];
                        for (uint32_t m = o[0]; m; m &= m - 1) w[low_bit(m)] = static_cast<uint16_t>(j + 1);
                        for (uint32_t m = o[1]; m; m &= m - 1) {
                            uint32_t& v = r[low_bit(m)];
                            v = std::min(row_min(v), j + 1) | std::max(row_max(v), j + 1) << 16;
                        }
                    }
                    if (first || !std::equal(r.begin(), r.end(), &row[i * kRowPos]) || !std::equal(w, w + kRowPos, &win[i * kRowPos])) {
                        moved[c] = round + 1;
                        changed = true;
                    }
                    std::copy(r.begin(), r.end(), &row[i * kRowPos]);
                    std::copy(w, w + kRowPos, &win[i * kRowPos]);
                    pair[i] = x;
                }
            }
            if (!changed) break;
            if (round >= rounds) return false;
        }
        for (size_t i = 0; i < steps; ++i) touch[i / kChunk] |= pair[i].any | pair[i].wr;
        for (uint32_t c = 0; c < tiles; ++c) {
            const size_t at = static_cast<size_t>(c) * kChunk;
            for (uint32_t j = 0; j < G0; ++j)
                if (size(j) > c * kChunk)
                    chunk_run<true>(P, ChunkRows{&row[at * kRowPos], &win[at * kRowPos], &pair[at]}, mem.data(), j, c, true, false);
        }
        return true;
    }

    // The record form's allocation (ptl_steps.cuh), phase by phase as its kernels run it.
    void step_regalloc(uint32_t S, uint32_t K) {
        std::vector<uint8_t> ring(K);
        for (uint32_t f = 0; f < P.F; ++f)
            if (f & 7u) step_free_function(P, f, ring.data(), 1, K);
        const uint32_t G0 = (P.F + 7) / 8;
        tany.ensure(row_tiles(S) * kRowTile);
        trow.ensure(row_tiles(S) * kRowTile * kRowPos, kRowNone);
        bind();
        for (uint32_t i = 0; i < S; ++i) {
            for (uint32_t g = 0; g < G0; ++g) {
                const uint32_t m = group_triggers(P, g, i);
                P.tany[i] |= m;
                for (uint32_t t = m; t; t &= t - 1) {
                    uint32_t& r = P.trow[static_cast<size_t>(i) * kRowPos + low_bit(t)];
                    r = std::min(row_min(r), g + 1) | (std::max(row_max(r), g + 1) << 16);
                }
            }
        }
        g_last_lock_step = !(g_chunks && chunk_lanes(S, K));
        if (!g_last_lock_step) return;
        LaneShared sh{};
        std::vector<uint8_t> rings(static_cast<size_t>(G0) * K);
        std::vector<LaneSlot> L(G0);
        for (uint32_t j = 0; j < G0; ++j) {
            L[j] = LaneSlot{};
            lane_init(P, L[j], j);
            sh.s0 = std::max(sh.s0, L[j].size);
        }
        const uint32_t s0 = std::min(sh.s0, S);
        for (uint32_t i = 0; i < s0; ++i) {
            LaneStep& st = sh.st[i % 3u];
            const uint32_t* row = P.trow + static_cast<size_t>(i) * kRowPos;
            auto ring_of = [&](uint32_t j) { return LaneRing{rings.data() + j, G0, K}; };
            if (win_wraps(i)) for (LaneStep& x : sh.st) std::memset(x.win, 0, sizeof(x.win));
            for (uint32_t j = 0; j < G0; ++j) {
                L[j].rec = i < L[j].size ? L[j].rec_at[i] : kStepIdle;
                if (G0 == 1) lane_step_a<true>(sh, st, row, L[j], ring_of(j), i, st.m);
                else lane_step_a<false>(sh, st, row, L[j], ring_of(j), i, st.m);
            }
            lane_clear(sh.st[(i + 2u) % 3u]);
            bool redo = false;
            for (uint32_t j = 0; j < G0; ++j) {
                lane_commit(sh, L[j]);
                redo |= lane_step_t(sh, st, st.m, L[j]);
            }
            if (redo) {
                for (uint32_t round = 0;; ++round) {
                    for (uint32_t j = 0; j < G0; ++j) lane_round(sh, st, st.m, row, L[j]);
                    const bool changed = st.before != sh.before2;
                    st.before = sh.before2;
                    sh.before2 = 0;
                    if (!changed) break;
                    if (round > G0 + 2) { record_error(P.err, ST_DEVICE_TIMEOUT, W_RA2, i); break; }
                }
                std::memset(st.win, 0, sizeof(st.win));
                st.m.wr = st.m.trig = st.later = 0;
                for (uint32_t j = 0; j < G0; ++j) lane_emit<false>(st, L[j], i, st.m);
                for (uint32_t j = 0; j < G0; ++j) lane_step_t(sh, st, st.m, L[j]);
            }
            for (uint32_t j = 0; j < G0; ++j) {
                lane_step_b1(L[j], ring_of(j), i, false);
                if (G0 == 1) lane_step_b2<true>(sh, st, st.m, LaneAbove{0, 0}, P.tany[i], L[j], ring_of(j), i);
                else lane_step_b2<false>(sh, st, st.m, LaneAbove{0, 0}, P.tany[i], L[j], ring_of(j), i);
            }
        }
        uint32_t tail = 0;
        for (uint32_t i = s0; i < S; ++i) tail |= P.tany[i];
        for (uint32_t j = 0; j < G0; ++j) {
            lane_commit(sh, L[j]);
            lane_tail(sh, L[j], tail);
        }
    }

    // The scalar generator's register allocation (ptl_scalar.cuh), from the optimized words
    // to the regalloc output (the spill offsets, the count scan, the scatter, the moved
    // function table and the frame words).
    void scalar_regalloc(uint32_t F, uint32_t W, uint32_t wb8) {
        uint32_t flagbits = g_force_tiles ? 2u : 0u;
        for (uint32_t f = 0; f < F; ++f) flagbits |= st_scalar_range(P, f);
        for (uint32_t i = 0; i < W; ++i) flagbits |= st_scalar_record(P, i);
        const uint32_t cross = flagbits & 1u;
        std::vector<unsigned long long> preserve(F, 0);
        if (cross || g_force_serial) {
            std::vector<int32_t> sregs(static_cast<size_t>(F) * 64);
            std::vector<SRaStep> steps(F);
            s_ra_serial(P, sregs.data(), steps.data(), preserve.data());
        } else if (!(flagbits & 2u)) {
            std::vector<uint8_t> ring(g_ring_k);
            std::vector<uint32_t> oidx(32);
            for (uint32_t f = 0; f < F; ++f)
                step_scalar_function(P, f, ring.data(), 1, g_ring_k, oidx.data(), 1, preserve.data());
        } else {
            int32_t sregs[64];
            // the GPU's word tiles (functions by their first word, symbols as bytes)
            constexpr uint32_t T = 4096;
            std::vector<uint8_t> sym;
            for (uint32_t b = 0; b <= W / T; ++b) {
                uint32_t first, last, base;
                s_ra_tile_functions(P, b, T, &first, &last);
                const uint32_t count = s_ra_tile_span(P, first, last, &base);
                sym.assign(count + 1, 0);
                const SymBytes sy{sym.data(), base, count, P.err};
                for (uint32_t f = first; f < last; ++f) s_ra_function(P, sy, f, sregs, preserve.data());
                for (uint32_t k = 0; k < count; ++k) s_ra_tile_writeback(P, sym.data(), base, count, k);
            }
        }
        g_last_cross = cross != 0;
        if (!check()) return;
        for (uint32_t v = 0; v < W; ++v) st_ra_spill(P, v);
        std::vector<uint32_t> extra(wb8 + 16, 0);
        for (uint32_t f = 0; f < F; ++f) st_s_preserve_counts(P, f, preserve.data(), extra.data());
        if (!check()) return;
        exclusive_scan(wb8, [&](uint32_t i) { return st_s_ra_count(P, i, extra.data()); }, roffs.p);
        if (!check()) return;
        const uint32_t W2 = roffs.p[W - 1] + 1;
        const uint32_t w2b8 = static_cast<uint32_t>(r8(W2));
        for (auto* b : {&ni, &nrd, &nr1, &nr2, &njt, &fsz, &joffs}) b->ensure(w2b8 + 16);
        P.W2 = W2; P.w2b8 = w2b8;
        bind();
        for (uint32_t i = 0; i < wb8; ++i) st_s_ra_scatter(P, i);
        for (uint32_t f = 0; f < F; ++f) st_fix_functab(P, f, P.roffs, W);
        for (uint32_t pass = 0; pass < 3; ++pass)
            for (uint32_t f = 0; f < F; ++f) st_s_frame(P, f, pass, preserve.data(), 0, nullptr);
    }

    int run(const uint8_t* type, const uint8_t* rtype, const int32_t* parent, const int32_t* depth,
            const int32_t* child, const uint32_t* data, size_t n_, size_t max_depth, bool scalar) {
        build_code_tables(&tab);
        const uint32_t n = static_cast<uint32_t>(n_);
        const uint32_t nb8 = static_cast<uint32_t>(r8(n));
        in_type.ensure(n); in_rtype.ensure(n); in_parent.ensure(n); in_depth.ensure(n); in_child.ensure(n); in_data.ensure(n);
        std::memcpy(in_type.p, type, n); std::memcpy(in_rtype.p, rtype, n);
        std::memcpy(in_parent.p, parent, 4ull * n); std::memcpy(in_depth.p, depth, 4ull * n);
        std::memcpy(in_child.p, child, 4ull * n); std::memcpy(in_data.p, data, 4ull * n);
        for (auto* b : {&nd1, &nd, &sizes, &loc0, &loc, &pos, &decl}) b->ensure(nb8);
        nt.ensure(nb8);
        rt.ensure(nb8);
        for (auto* b : {&par, &ci, &dep}) b->ensure(nb8);
        fflag.ensure(nb8);
        regs.ensure(3ull * n);
        P = Prog{};
        P.n = n; P.nb8 = nb8; P.max_depth = static_cast<uint32_t>(max_depth);
        P.scalar = scalar ? 1u : 0u;
        bind();
        bool reach = false;
        for (uint32_t i = 0; i < nb8; ++i) reach |= st_ingest(P, i);
        if (!check()) return err.code;
        if (!reach) return ST_INVALID_AST;
        if (scalar) {
            for (uint32_t i = 0; i < nb8; ++i) st_s_pre_lists(P, i);
            for (uint32_t i = 0; i < nb8; ++i) st_s_pre_float(P, i);
        } else {
            for (uint32_t i = 0; i < nb8; ++i) st_pre_lists(P, i);
            for (uint32_t i = 0; i < nb8; ++i) st_pre_float(P, i);
        }
        for (uint32_t i = 0; i < nb8; ++i) st_pre_float_apply(P, i);
        if (!check()) return err.code;
        exclusive_scan(nb8, [&](uint32_t i) { const uint32_t v = st_count(P, i); P.sizes[i] = v; return v; }, loc0.p);
        for (uint32_t i = 0; i < nb8; ++i) st_fix_own(P, i);
        for (uint32_t i = 0; i < nb8; ++i) st_fix_cond(P, i);
        uint32_t F = 0;
        for (uint32_t i = 0; i < nb8; ++i) if (P.nt[i] == RV_FUNC_DECL) P.decl[F++] = i;
        if (!check()) return err.code;
        if (F == 0) return ST_UNSUPPORTED;
        const uint32_t fb8 = static_cast<uint32_t>(r8(F));
        for (auto* b : {&fn_id, &fn_start, &fn_size, &fn_end, &fn_start0, &fn_size0, &fn_end0, &fn_ra_start, &fn_ra_end, &fn_ra_size}) b->ensure(fb8 + 8);
        P.F = F; P.fb8 = fb8;
        bind();
        for (uint32_t f = 0; f < fb8; ++f) st_functab(P, f);
        uint32_t S = 0;
        for (uint32_t f = 0; f < fb8; ++f) {
            st_functab_end(P, f);
            if (f < F) S = std::max(S, P.fn_size[f]);
        }
        for (uint32_t f = 0; f < F; ++f) fn_end0.p[f] = fn_end.p[f];
        const uint32_t W = P.loc[n - 1];
        const uint32_t wb8 = static_cast<uint32_t>(r8(W));
        for (auto* b : {&instr, &rd, &rs1, &rs2, &jt, &used_instrs, &symreg, &symswp, &stamp, &spill, &roffs}) b->ensure(wb8);
        owner.ensure(wb8);
        used.ensure(wb8);
        smark.ensure(wb8);
        P.W = W; P.wb8 = wb8; P.S = S;
        bind();
        depth_sort(n);
        if (scalar) {
            for (uint32_t x = 0; x < n; ++x) st_s_gen_prop(P, x);
            for (uint32_t x = 0; x < n; ++x) st_s_gen_claim(P, x);
            for (uint32_t x = 0; x < n; ++x) st_s_gen_write(P, x);
        } else {
            for (uint32_t x = 0; x < n; ++x) st_gen_prop(P, x);
            for (uint32_t x = 0; x < n; ++x) st_gen_claim(P, x);
            for (uint32_t x = 0; x < n; ++x) st_gen_write(P, x);
        }
        if (!check()) return err.code;
        for (uint32_t i = 0; i < wb8; ++i) st_opt_mark(P, i);
        for (;;) {
            bool changed = false;
            for (uint32_t i = 0; i < wb8; ++i) changed |= st_opt_sweep(P, i);
            if (!changed) break;
        }
        for (uint32_t i = 0; i < wb8; ++i) st_opt_final(P, i);
        if (!check()) return err.code;
        lifetime.ensure(fb8);
        for (uint32_t f = 0; f < F; ++f) lifetime.p[f] = 0x1Full;
        trig_min.ensure(static_cast<size_t>(std::max<uint32_t>(S, 1)) * 64, 0xFFFFFFFFu);
        trig_max.ensure(static_cast<size_t>(std::max<uint32_t>(S, 1)) * 64, 0u);
        defpos.ensure(wb8);
        bind();
        if (scalar) {
            scalar_regalloc(F, W, wb8);
            if (!check()) return err.code;
        } else {
            uint32_t flagbits = g_force_general || g_force_hashed ? 2u : 0u;
            for (uint32_t f = 0; f < F; ++f) flagbits |= st_step_range(P, f);
            for (uint32_t i = 0; i < W; ++i) flagbits |= st_step_record(P, i);
            g_last_hashed = false;
            const uint32_t G0 = (F + 7) / 8;
            if ((flagbits & 1u) || G0 > 8192u) {
                st_ra_serial(P, stamp.p);
            } else if (flagbits & 2u) {
                std::vector<uint32_t> tag(64), val(64);
                const SymCache c1{tag.data(), val.data(), 64};
                Prog Pfree = P;
                Pfree.defpos = nullptr;
                for (uint32_t f = 0; f < F; ++f) if (f & 7u) ra_free_function_cached(Pfree, c1, 0, f);
                g_last_hashed = g_force_hashed;
                for (uint32_t f = 0; f < F; ++f) g_last_hashed |= st_step_range(P, f) != 0;
                for (uint32_t i = 0; i < W; ++i) g_last_hashed |= st_ra_definition(P, i);
                lane0_cached(S, hm_cache_k, g_last_hashed);
            } else {
                tmask.ensure(wb8);
                bind();
                step_regalloc(S, g_ring_k);
            }
            for (uint32_t v = 0; v < W; ++v) st_ra_spill(P, v);
            exclusive_scan(wb8, [&](uint32_t i) { return st_ra_count(P, i); }, roffs.p);
            if (!check()) return err.code;
            const uint32_t W2 = roffs.p[W - 1] + 1;
            const uint32_t w2b8 = static_cast<uint32_t>(r8(W2));
            for (auto* b : {&ni, &nrd, &nr1, &nr2, &njt, &fsz, &joffs}) b->ensure(w2b8 + 16);
            P.W2 = W2; P.w2b8 = w2b8;
            bind();
            for (uint32_t i = 0; i < wb8; ++i) st_ra_scatter(P, i);
            for (uint32_t f = 0; f < F; ++f) st_fix_functab(P, f, P.roffs, W);
            for (uint32_t f = 0; f < F; ++f) st_ra_frame(P, f);
        }
        for (uint32_t f = 0; f < F; ++f) { fn_ra_start.p[f] = fn_start.p[f]; fn_ra_end.p[f] = fn_end.p[f]; fn_ra_size.p[f] = fn_size.p[f]; }
        const uint32_t W2 = P.W2, w2b8 = P.w2b8;
        exclusive_scan(w2b8, [&](uint32_t i) { const uint32_t v = i < W2 ? st_fj_size(P, i) : 0u; P.fsz[i] = v; return v; }, joffs.p);
        const uint32_t W3 = fsz.p[W2 - 1] + joffs.p[W2 - 1];
        out.ensure(r8(W3) + 8);
        P.W3 = W3;
        bind();
        for (uint32_t i = 0; i < W2; ++i) st_fj_emit(P, i);
        for (uint32_t f = 0; f < F; ++f) st_fix_functab(P, f, P.joffs, W2);
        return check() ? 0 : err.code;
    }
};

}  // namespace

extern "C" {

struct ptlhm_buf {
    uint32_t* p;
    size_t n;
};

// Same slot numbers as ptl_generator_snapshot (include/ptl_codegen.h).
// scalar: the scalar generator's semantics.
int ptlhm_compile_mode(const uint8_t* type, const uint8_t* rtype, const int32_t* parent, const int32_t* depth,
                       const int32_t* child, const uint32_t* data, size_t n, size_t max_depth, ptlhm_buf* bufs,
                       int nbufs, uint32_t* err_out, int scalar) {
    Model* m = new Model();
    int rc = 0;
    try {
        rc = m->run(type, rtype, parent, depth, child, data, n, max_depth, scalar != 0);
    } catch (const std::exception&) {
        rc = ST_UNSUPPORTED;
    }
    if (err_out) { err_out[0] = m->err.code; err_out[1] = m->err.where; err_out[2] = m->err.detail; }
    auto put = [&](int k, const uint32_t* src, size_t len) {
        if (k >= nbufs) return;
        bufs[k].n = len;
        bufs[k].p = static_cast<uint32_t*>(std::malloc(std::max<size_t>(1, len) * 4));
        if (len) std::memcpy(bufs[k].p, src, len * 4);
    };
    for (int k = 0; k < nbufs; ++k) { bufs[k].p = nullptr; bufs[k].n = 0; }
    if (rc == 0) {
        const Prog& P = m->P;
        put(0, P.out, P.W3);
        put(1, P.fn_start, P.F); put(2, P.fn_end, P.F); put(3, P.fn_size, P.F); put(4, P.fn_id, P.F);
        {
            std::vector<uint32_t> wide(P.n);
            for (uint32_t i = 0; i < P.n; ++i) wide[i] = P.nt[i];
            put(5, wide.data(), P.n);
            for (uint32_t i = 0; i < P.n; ++i) wide[i] = P.rt[i];
            put(6, wide.data(), P.n);
        }
        put(7, P.nd, P.n);
        put(8, P.sizes, P.n); put(9, P.loc, P.n);
        put(10, P.fn_id, P.F); put(11, P.fn_start0, P.F); put(12, m->fn_end0.p, P.F); put(13, P.fn_size0, P.F);
        put(14, P.instr, P.W); put(15, P.rd, P.W); put(16, P.rs1, P.W); put(17, P.rs2, P.W); put(18, P.jt, P.W);
        put(19, P.used_instrs, P.W);
        put(20, P.ni, P.W2); put(21, P.nrd, P.W2); put(22, P.nr1, P.W2); put(23, P.nr2, P.W2); put(24, P.njt, P.W2);
        put(25, m->fn_ra_start.p, P.F); put(26, m->fn_ra_end.p, P.F); put(27, m->fn_ra_size.p, P.F);
        put(40, P.pos, P.n);
    }
    delete m;
    return rc;
}

int ptlhm_compile(const uint8_t* type, const uint8_t* rtype, const int32_t* parent, const int32_t* depth,
                  const int32_t* child, const uint32_t* data, size_t n, size_t max_depth, ptlhm_buf* bufs,
                  int nbufs, uint32_t* err_out) {
    return ptlhm_compile_mode(type, rtype, parent, depth, child, data, n, max_depth, bufs, nbufs, err_out, 0);
}

int ptlhm_last_cross(void) { return g_last_cross ? 1 : 0; }

// Whether isn_gen's packed table fields decode to the code tables.
int ptlhm_gen_desc_ok(void) {
    static CodeTables t;
    build_code_tables(&t);
    return gen_desc_ok(&t) ? 1 : 0;
}
int ptlhm_last_locked(void) { return g_last_locked ? 1 : 0; }
// The flattening's walks over a valid tree's tour: the longest, its limit, the splitters
// and their limit.
void ptlhm_flatten_walks(const int32_t* parent, const int32_t* child, uint32_t n, uint32_t out[4]) {
    std::vector<uint32_t> deg(n, 0), off(n + 1, 0), kids(n), succ(2 * static_cast<size_t>(n));
    for (uint32_t v = 0; v < n; ++v)
        if (parent[v] >= 0) ++deg[parent[v]];
    for (uint32_t v = 0; v < n; ++v) off[v + 1] = off[v] + deg[v];
    uint32_t root = 0;
    for (uint32_t v = 0; v < n; ++v) {
        if (parent[v] >= 0) kids[off[parent[v]] + child[v]] = v;
        else root = v;
    }
    const uint32_t lg = splitter_lg(n), end = 2 * n;
    for (uint32_t v = 0; v < n; ++v) {
        const uint32_t p = static_cast<uint32_t>(parent[v]), c = static_cast<uint32_t>(child[v]) + 1u;
        succ[2 * v] = deg[v] ? 2 * kids[off[v]] : 2 * v + 1;
        succ[2 * v + 1] = v == root ? end : (c < deg[p] ? 2 * kids[off[p] + c] : 2 * p + 1);
    }
    uint32_t longest = 0, steps = 0, splitters = 1;  // the root's enter
    for (uint32_t x = succ[2 * root]; x != end; x = succ[x]) {
        ++steps;
        if (is_splitter(x, lg)) {
            ++splitters;
            steps = 0;
        }
        longest = std::max(longest, steps);
    }
    out[0] = longest;
    out[1] = walk_most(lg);
    out[2] = splitters;
    out[3] = splitters_most(n);
}
// Of a buffer of n elements: the bytes it needs, those that clearing it writes, and those
// allocated for it.
void ptlhm_buffer_bytes(size_t n, size_t elem, size_t out[3]) {
    out[0] = buffer_bytes(n, elem);
    out[1] = cleared_bytes(out[0]);
    out[2] = allocated_bytes(out[0]);
}
// The error codes of n programs after a lost chunk launch of `threads` threads a block.
void ptlhm_chunks_lost(uint32_t n, uint32_t threads, uint32_t* codes) {
    std::vector<ErrorWord> err(n);
    std::vector<Prog> progs(n);
    for (uint32_t k = 0; k < n; ++k) progs[k].err = &err[k];
    for (uint32_t t = 0; t < threads; ++t) chunks_lost([&](uint32_t k) -> const Prog& { return progs[k]; }, n, t, threads, 3u);
    for (uint32_t k = 0; k < n; ++k) codes[k] = err[k].code;
}
int ptlhm_last_lock_step(void) { return g_last_lock_step ? 1 : 0; }
void ptlhm_set_chunks(int on) { g_chunks = on != 0; }
void ptlhm_set_chunk_rounds(uint32_t rounds) { g_chunk_rounds = rounds; }
void ptlhm_set_scalar_tiles(int on) { g_force_tiles = on != 0; }
void ptlhm_set_scalar_serial(int on) { g_force_serial = on != 0; }

void ptlhm_set_cache_entries(uint32_t k) { g_cache_k = k; }
void ptlhm_set_ring_words(uint32_t k) { g_ring_k = k; }  // a power of two
void ptlhm_set_general(int on) { g_force_general = on != 0; }
void ptlhm_set_hashed(int on) { g_force_hashed = on != 0; }
int ptlhm_last_hashed(void) { return g_last_hashed ? 1 : 0; }

void ptlhm_free(ptlhm_buf* bufs, int nbufs) {
    for (int k = 0; k < nbufs; ++k) { std::free(bufs[k].p); bufs[k].p = nullptr; bufs[k].n = 0; }
}

// The sort emulation alone: perm receives the order of iota(n) sorted by keys.
void ptlhm_depth_sort(const int32_t* keys, size_t n, uint32_t* perm) {
    Model m;
    m.dep.ensure(n);
    m.pos.ensure(n);
    std::memcpy(m.dep.p, keys, 4 * n);
    m.depth_sort(static_cast<uint32_t>(n));
    for (size_t x = 0; x < n; ++x) perm[m.pos.p[x]] = static_cast<uint32_t>(x);
}

}  // extern "C"
