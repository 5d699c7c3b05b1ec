// Kernel of the lane-0 functions in chunks (ptl_chunks.cuh): rounds of runs and row folds
// in one launch, over one program or many.
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "ptl_chunks.cuh"
#include "ptl_kernels.cuh"

namespace ptl {
namespace {

constexpr uint32_t kWarps = 16, kThreads = 32 * kWarps;

// Every block waits for all (the launch is cooperative: they are resident together).
// False after `most` cycles without them.
struct GridBarrier {
    uint32_t* count;
    long long most;
    uint32_t goal = 0;
    __device__ bool wait() {
        __shared__ uint32_t lost;
        __syncthreads();
        if (threadIdx.x == 0) {
            goal += gridDim.x;
            __threadfence();
            atomicAdd(count, 1u);
            const long long since = clock64();
            for (;;) {
                uint32_t seen;
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(count) : "memory");
                lost = static_cast<int32_t>(seen - goal) < 0;
                if (!lost || clock64() - since > most) break;
            }
            __threadfence();
        }
        __syncthreads();
        return !lost;
    }
};

// Shared memory of a warp: a run's rows, slots and oidx, or (a team's first warp) a fold's
// rows.
constexpr uint32_t kRowsAt = 0, kWinsAt = kChunk * kRowPos * 4u, kPairsAt = kWinsAt + kChunk * kRowPos * 2u,
                   kMemAt = kPairsAt + kChunk * 8u, kRunBytes = kMemAt + kChunkMemWords * 4u;
constexpr uint32_t kFoldStride = kRowPos + 1u, kFoldBytes = 3u * kChunk * kFoldStride * 4u + kChunk * 8u;
constexpr uint32_t kListMost = 512u, kListBytes = kListMost * 6u;  // a folding warp's functions (8,192 groups, a block)
constexpr uint32_t kWarpBytes = ((kRunBytes > kFoldBytes ? kRunBytes : kFoldBytes) + 15u) & ~15u;

// The rows of chunk c again from its functions' outputs, at the positions where some
// output has changed (P.ch.delta; in the first round all), by a team of kTeam warps of which
// this is one; lane = step, then lane = position.  A warp has the outputs of 16 functions
// in flight at a time.  Returns whether the rows
// changed (kTeam > 1: this warp's share).
template <uint32_t kTeam>
__device__ bool fold(const Prog& P, uint32_t c, uint32_t* smem, uint32_t warp, bool first) {
    // (up to kBatch << kHigh functions a warp: 8,192 groups for a block)
    constexpr uint32_t kBits = kTeam == 1 ? 3 : 4, kBatch = 1u << kBits, kHigh = kTeam == kWarps ? 5 : 1;
    constexpr uint32_t kSteps = kChunk / kTeam, kPart = kSteps < 8u ? kSteps : 8u;
    const uint32_t lane = threadIdx.x & 31u, G0 = (P.F + 7u) / 8u;
    const size_t at = static_cast<size_t>(c) * kChunk;
    uint32_t* lo = smem;
    uint32_t* hi = lo + kChunk * kFoldStride;
    uint32_t* win = hi + kChunk * kFoldStride;
    uint32_t* any = win + kChunk * kFoldStride;  // what the step's functions trigger and write now
    uint32_t* wrote = any + kChunk;
    auto sync = [&] {
        if constexpr (kTeam == 1) __syncwarp();
        else if constexpr (kTeam == kWarps) __syncthreads();
        else asm volatile("bar.sync %0, %1;" ::"r"(1u + (threadIdx.x >> 5) / kTeam), "r"(32u * kTeam) : "memory");
    };
    // positions to fold again, of the lane's step
    const uint2 delta = first ? make_uint2(~0u, ~0u) : __ldcg(reinterpret_cast<const uint2*>(P.ch.delta) + at + lane);
    const uint32_t dw = delta.x, dt = delta.y;
    uint32_t *mylo = lo + lane * kFoldStride, *myhi = hi + lane * kFoldStride, *mywin = win + lane * kFoldStride;
    if (warp == 0) {
        for (uint32_t m = dt; m; m &= m - 1) {
            mylo[low_bit(m)] = kRowNone;
            myhi[low_bit(m)] = 0;
        }
        for (uint32_t m = dw; m; m &= m - 1) mywin[low_bit(m)] = 0;
        any[lane] = wrote[lane] = 0;
    }
    sync();
    const uint2* out = reinterpret_cast<const uint2*>(P.ch.out);
    const uint32_t* off = P.ch.off;
    // For every position (a bit), the least and the greatest triggering and the greatest
    // writing function of this warp's, as its number among them in bit slices: a function
    // costs an operation per slice, where a loop over its positions diverges (and took up
    // to 450,000 cycles).
    uint32_t lo_s[kBits + kHigh] = {}, hi_s[kBits + kHigh] = {}, win_s[kBits + kHigh] = {}, trigs = 0, wrote_s = 0;
    // This warp's functions that reach the chunk, in order: how many they are, and where the
    // k-th one's outputs are.  Few reach a wide program's last chunks (1,229 functions: the
    // allocation 10.2 to 9.1 ms).
    uint32_t count = (G0 - min(G0, warp) + kTeam - 1u) / kTeam;
    uint32_t* items = nullptr;
    uint16_t* numbers = nullptr;
    if constexpr (kTeam > 1) {
        items = smem + (kWarpBytes + warp * kListBytes) / 4u;
        numbers = reinterpret_cast<uint16_t*>(items + kListMost);
        uint32_t all = count, n = 0;
        for (uint32_t x0 = 0; x0 < all; x0 += 32u) {
            const uint32_t x = x0 + lane, j = min(warp + x * kTeam, G0 - 1u), item = off[j] + c;
            const bool has = x < all && item < off[j + 1u];
            const uint32_t mask = __ballot_sync(0xFFFFFFFFu, has), at = n + __popc(mask & ((1u << lane) - 1u));
            if (has) {
                items[at] = item;
                numbers[at] = static_cast<uint16_t>(x);
            }
            n += __popc(mask);
        }
        count = n;
        __syncwarp();
    }
    for (uint32_t x0 = 0, nb = 0; x0 < count; x0 += kBatch, ++nb) {
        uint2 x[kBatch];
#pragma unroll
        for (uint32_t k = 0; k < kBatch; ++k) {  // no branches, so that all loads are in flight
            bool has = x0 + k < count;
            uint32_t item;
            if constexpr (kTeam > 1) {
                item = items[has ? x0 + k : 0u];
            } else {
                const uint32_t j = min(warp + (x0 + k) * kTeam, G0 - 1u);
                item = off[j] + c;
                has = has && item < off[j + 1u];
            }
            x[k] = __ldcg(out + static_cast<size_t>(has ? item : 0u) * kChunk + lane);
            if (!has) x[k] = make_uint2(0, 0);
        }
        uint32_t lo_b[kBits] = {}, hi_b[kBits] = {}, win_b[kBits] = {}, t = 0, w = 0;  // of the batch
#pragma unroll
        for (uint32_t k = 0; k < kBatch; ++k) {
            const uint32_t up = x[k].y & dt, down = x[kBatch - 1u - k].y & dt, wr = x[k].x & dw;
            t |= up;
            w |= wr;
#pragma unroll
            for (uint32_t i = 0; i < kBits; ++i) {
                hi_b[i] = (k >> i & 1u) ? hi_b[i] | up : hi_b[i] & ~up;
                win_b[i] = (k >> i & 1u) ? win_b[i] | wr : win_b[i] & ~wr;
                lo_b[i] = ((kBatch - 1u - k) >> i & 1u) ? lo_b[i] | down : lo_b[i] & ~down;
            }
        }
        const uint32_t fresh = t & ~trigs;
#pragma unroll
        for (uint32_t i = 0; i < kBits + kHigh; ++i) {
            const uint32_t high = i < kBits ? 0u : 0u - (nb >> (i - kBits) & 1u);
            hi_s[i] = (hi_s[i] & ~t) | (i < kBits ? hi_b[i % kBits] : high & t);
            win_s[i] = (win_s[i] & ~w) | (i < kBits ? win_b[i % kBits] : high & w);
            lo_s[i] |= fresh & (i < kBits ? lo_b[i % kBits] : high);
        }
        trigs |= t;
        wrote_s |= w;
    }
    for (uint32_t all = __reduce_or_sync(0xFFFFFFFFu, trigs | wrote_s); all; all &= all - 1) {
        const uint32_t p = low_bit(all);
        uint32_t l = 0, h = 0, v = 0;
#pragma unroll
        for (uint32_t i = 0; i < kBits + kHigh; ++i) {
            l |= (lo_s[i] >> p & 1u) << i;
            h |= (hi_s[i] >> p & 1u) << i;
            v |= (win_s[i] >> p & 1u) << i;
        }
        if constexpr (kTeam > 1) {
            l = numbers[l];
            h = numbers[h];
            v = numbers[v];
        }
        const uint32_t group = warp + 1u;
        if (trigs >> p & 1u) {
            atomicMin(mylo + p, group + l * kTeam);
            atomicMax(myhi + p, group + h * kTeam);
        }
        if (wrote_s >> p & 1u) atomicMax(mywin + p, group + v * kTeam);
    }
    if (trigs) atomicOr(&any[lane], trigs);
    if (wrote_s) atomicOr(&wrote[lane], wrote_s);
    const bool busy = (dw | dt) != 0;
    const uint32_t steps = __ballot_sync(0xFFFFFFFFu, busy);  // of the chunk, with something to fold
    sync();
    bool changed = first;
    if (warp == 0) {
        uint2* pair = reinterpret_cast<uint2*>(P.ch.pair) + at + lane;
        uint2 x = first ? make_uint2(0, 0) : __ldcg(pair);
        if (busy) {
            x = make_uint2((x.x & ~dt) | any[lane] | (P.tany[at + lane] & dt), (x.y & ~dw) | wrote[lane]);
            __stcg(pair, x);
            if (!first) __stcg(reinterpret_cast<uint2*>(P.ch.delta) + at + lane, make_uint2(0, 0));
        }
        const uint32_t touch = __reduce_or_sync(0xFFFFFFFFu, x.x | x.y);
        if (lane == 0) P.ch.touch[c] = touch;
    }
    for (uint32_t t0 = warp * kSteps; t0 < (warp + 1u) * kSteps; t0 += kPart) {
        if ((steps >> t0 & ((1ull << kPart) - 1u)) == 0) continue;
        uint32_t base[kPart], was[kPart];
        uint16_t wwas[kPart];
        bool t[kPart], w[kPart];
#pragma unroll
        for (uint32_t k = 0; k < kPart; ++k) {
            const size_t x = (at + t0 + k) * kRowPos + lane;
            t[k] = __shfl_sync(0xFFFFFFFFu, dt, t0 + k) >> lane & 1u;
            w[k] = __shfl_sync(0xFFFFFFFFu, dw, t0 + k) >> lane & 1u;
            base[k] = t[k] ? __ldg(P.trow + x) : 0u;
            was[k] = t[k] && !first ? __ldcg(P.ch.row + x) : 0u;
            wwas[k] = w[k] && !first ? __ldcg(P.ch.win + x) : static_cast<uint16_t>(0);
        }
#pragma unroll
        for (uint32_t k = 0; k < kPart; ++k) {
            const size_t x = (at + t0 + k) * kRowPos + lane;
            const uint32_t y = (t0 + k) * kFoldStride + lane;
            const uint32_t row = min(row_min(base[k]), lo[y]) | max(row_max(base[k]), hi[y]) << 16;
            const uint16_t v = static_cast<uint16_t>(win[y]);
            if (t[k] && (first || was[k] != row)) {
                changed = true;
                __stcg(P.ch.row + x, row);
            }
            if (w[k] && (first || wwas[k] != v)) {
                changed = true;
                __stcg(P.ch.win + x, v);
            }
        }
    }
    sync();  // the shared rows are the next fold's
    return __any_sync(0xFFFFFFFFu, changed);
}

// One block of 16 warps per SM: as many as the shared memory of a run or a fold allows.
__global__ void __launch_bounds__(kThreads, 1)
    k_lane_chunks(const __grid_constant__ ChunkBatch b, const __grid_constant__ Prog one) {
    static_assert(kChunkNarrow <= 8u << 1 && kChunkWide <= 4u * 16u << 1 && 8192u <= kWarps * 16u << 5, "folds");
    static_assert(kWarps * kListBytes <= (kWarps - 1u) * kWarpBytes && 4u * kListBytes <= 3u * kWarpBytes, "fold lists");
    extern __shared__ __align__(16) unsigned char smem[];
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    uint32_t* changed = b.sync + 2;  // [round]
    GridBarrier grid{b.sync, b.wait};
    auto prog = [&](uint32_t k) -> const Prog& { return b.progs ? b.progs[b.order[k]] : one; };
    auto first_of = [&](const uint32_t* off, uint32_t k) { return b.progs ? off[k] : 0u; };
    auto owner = [&](const uint32_t* off, uint32_t q) {  // off[lo] <= q < off[lo + 1]
        uint32_t lo = 0, hi = b.n;
        while (hi - lo > 1u) {
            const uint32_t mid = (lo + hi) >> 1;
            if (off[mid] <= q) lo = mid; else hi = mid;
        }
        return lo;
    };
    auto late = [&](uint32_t round) {
        chunks_lost(prog, b.n, threadIdx.x, kThreads, round);
    };
    // Rows of the chunks with new outputs (or of all), of programs with least < groups <=
    // most, by teams of kTeam warps.  A program with one lane-0 function needs none: what
    // it writes and triggers itself, its run knows.
    auto fold_tiles = [&](auto team, uint32_t least, uint32_t most, uint32_t round, bool all, bool last) {
        constexpr uint32_t kTeam = decltype(team)::value;
        const uint32_t member = warp % kTeam, index = warp / kTeam, teams = kWarps / kTeam;
        for (uint32_t q = index * gridDim.x + blockIdx.x; q < b.tiles; q += teams * gridDim.x) {
            const uint32_t k = owner(b.tile_off, q), c = q - first_of(b.tile_off, k);
            const Prog& P = prog(k);
            const uint32_t G0 = (P.F + 7u) / 8u;
            if (G0 <= least || G0 > most || (!all && __ldcg(P.ch.dirty + c) != round)) continue;
            const bool moved = fold<kTeam>(P, c, reinterpret_cast<uint32_t*>(smem + index * kTeam * kWarpBytes), member, all);
            if (moved && !last && lane == 0) {
                P.ch.moved[c] = round + 1u;
                changed[round + 1u] = 1u;
            }
        }
        __syncthreads();  // the shared rows are the next class's
    };
    unsigned char* mine = smem + warp * kWarpBytes;
    uint32_t* row = reinterpret_cast<uint32_t*>(mine + kRowsAt);
    uint16_t* win = reinterpret_cast<uint16_t*>(mine + kWinsAt);
    ChunkPair* pair = reinterpret_cast<ChunkPair*>(mine + kPairsAt);
    uint32_t* mem = reinterpret_cast<uint32_t*>(mine + kMemAt) + lane;
    bool final = false;
    for (uint32_t round = 1;; ++round) {
        const bool first = round == 1;
        for (uint32_t q = warp * gridDim.x + blockIdx.x; q < b.runs; q += kWarps * gridDim.x) {
            const uint32_t k = owner(b.run_off, q);
            const Prog& P = prog(k);
            const uint32_t G0 = (P.F + 7u) / 8u, NW = (G0 + 31u) / 32u, local = q - first_of(b.run_off, k);
            const uint32_t c = local / NW, w = local % NW;
            const bool lone = G0 == 1u, rows_moved = first || final || __ldcg(P.ch.moved + c) == round;
            if (!rows_moved && __ldcg(P.ch.tag + local) < round) continue;
            const uint32_t j = w * 32u + lane;
            bool on = j < G0 && P.ch.off[j] + c < P.ch.off[j + 1u] && *P.ch.lock == 0;
            if (on && !rows_moved) on = __ldcg(P.ch.need + P.ch.off[j] + c) >= round;
            if (!__any_sync(0xFFFFFFFFu, on)) continue;
            const size_t at = static_cast<size_t>(c) * kChunk;
            const uint4* grow = reinterpret_cast<const uint4*>((first || lone ? P.trow : P.ch.row) + at * kRowPos);
            const uint4* gwin = reinterpret_cast<const uint4*>(P.ch.win + at * kRowPos);
#pragma unroll
            for (uint32_t x = 0; x < 8u; ++x) reinterpret_cast<uint4*>(row)[x * 32u + lane] = __ldcg(grow + x * 32u + lane);
#pragma unroll
            for (uint32_t x = 0; x < 4u; ++x)
                reinterpret_cast<uint4*>(win)[x * 32u + lane] = first || lone ? make_uint4(0, 0, 0, 0) : __ldcg(gwin + x * 32u + lane);
            const uint2 pr = first || lone ? make_uint2(P.tany[at + lane], 0) : __ldcg(reinterpret_cast<const uint2*>(P.ch.pair) + at + lane);
            pair[lane] = ChunkPair{pr.x, pr.y};
            __syncwarp();
            const ChunkRows rows{row, win, pair};
            if (final) {
                chunk_run<true>(P, rows, mem, j, c, on, false);
            } else {
                const uint32_t r = chunk_run<false>(P, rows, mem, j, c, on, first);
                if (r & kChunkNext) {
                    P.ch.need[P.ch.off[j] + c + 1u] = round + 1u;
                    P.ch.tag[local + NW] = round + 1u;
                    changed[round + 1u] = 1u;
                }
                if (r & kChunkOut) P.ch.dirty[c] = round;
            }
            __syncwarp();
        }
        if (final) return;
        if (!grid.wait()) return late(round);
        if (b.classes & 2u) fold_tiles(std::integral_constant<uint32_t, 1>{}, 1, kChunkNarrow, round, first, false);
        if (b.classes & 4u) fold_tiles(std::integral_constant<uint32_t, 4>{}, kChunkNarrow, kChunkWide, round, first, false);
        if (b.classes & 8u) fold_tiles(std::integral_constant<uint32_t, kWarps>{}, kChunkWide, 0xFFFFFFFFu, round, first, false);
        if (b.classes != 1u && !grid.wait()) return late(round);
        final = __ldcg(changed + round + 1u) == 0;  // not written any more: all threads read the same
        if (final && (b.classes & 1u)) {  // a lone function's rows, for its dead symbols
            fold_tiles(std::integral_constant<uint32_t, 1>{}, 0, 1, round, true, true);
            if (!grid.wait()) return late(round);
        }
        if (!final && round >= b.rounds) {  // the lock-step does it
            if (blockIdx.x == 0)
                for (uint32_t k = threadIdx.x; k < b.n; k += kThreads) *prog(k).ch.lock = 1u;
            return;
        }
    }
}

}  // namespace

ChunkSizes chunk_sizes(uint32_t F, uint32_t S, uint32_t W, uint32_t items) {
    const uint64_t tiles = row_tiles(S), G0 = (F + 7u) / 8u;
    ChunkSizes z{};
    z.runs = tiles * ((G0 + 31u) / 32u);
    z.tiles = tiles;
    uint64_t at = 0;
    auto take = [&](uint64_t bytes) {
        const uint64_t here = at;
        at = (at + bytes + 255u) & ~255ull;
        return here;
    };
    z.last = take(4ull * W);
    z.reach = take(4ull * (items + 1ull));
    z.slots = take(4ull * G0);
    z.need = take(4ull * (items + 1ull));
    z.tag = take(4ull * (z.runs + (G0 + 31u) / 32u));
    z.delta = take(8ull * tiles * kRowTile);
    z.dirty = take(4ull * tiles);
    z.moved = take(4ull * tiles);
    z.lock = take(4ull);
    z.zeroed = at;
    z.off = take(4ull * (G0 + 1u));
    z.rec = take(static_cast<uint64_t>(items) * kChunk * 8u);
    z.out = take(static_cast<uint64_t>(items) * kChunk * 8u);
    z.state = take((items + 1ull) * kStateVecs * 16u);
    z.row = take(tiles * kRowTile * kRowPos * 4u);
    z.win = take(tiles * kRowTile * kRowPos * 2u);
    z.pair = take(tiles * kRowTile * 8u);
    z.touch = take(4ull * tiles);
    z.total = at;
    return z;
}
void chunk_bind(LaneChunks& ch, const ChunkSizes& z, void* zeroed, void* rest) {
    char* a = static_cast<char*>(zeroed);
    char* b = static_cast<char*>(rest) - z.zeroed;
    ch.last = reinterpret_cast<uint32_t*>(a + z.last);
    ch.reach = reinterpret_cast<uint32_t*>(a + z.reach);
    ch.slots = reinterpret_cast<uint32_t*>(a + z.slots);
    ch.need = reinterpret_cast<uint32_t*>(a + z.need);
    ch.tag = reinterpret_cast<uint32_t*>(a + z.tag);
    ch.delta = reinterpret_cast<uint32_t*>(a + z.delta);
    ch.dirty = reinterpret_cast<uint32_t*>(a + z.dirty);
    ch.moved = reinterpret_cast<uint32_t*>(a + z.moved);
    ch.lock = reinterpret_cast<uint32_t*>(a + z.lock);
    ch.off = reinterpret_cast<uint32_t*>(b + z.off);
    ch.rec = reinterpret_cast<unsigned long long*>(b + z.rec);
    ch.out = b + z.out;
    ch.state = b + z.state;
    ch.row = reinterpret_cast<uint32_t*>(b + z.row);
    ch.win = reinterpret_cast<uint16_t*>(b + z.win);
    ch.pair = reinterpret_cast<ChunkPair*>(b + z.pair);
    ch.touch = reinterpret_cast<uint32_t*>(b + z.touch);
}

bool chunks_fit() {
    int dev = 0, coop = 0, per_sm = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop)
        return false;
    constexpr size_t bytes = kWarps * kWarpBytes;
    if (allow_dynamic_smem(reinterpret_cast<const void*>(&k_lane_chunks), bytes) != cudaSuccess) return false;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_lane_chunks, kThreads, bytes) == cudaSuccess && per_sm >= 1;
}

cudaError_t run_lane_chunks(const ChunkBatch& b, const Prog& one, cudaStream_t s) {
    if (b.n == 0 || b.runs == 0) return cudaSuccess;
    constexpr size_t bytes = kWarps * kWarpBytes;
    const void* fn = reinterpret_cast<const void*>(&k_lane_chunks);
    cudaError_t e = allow_dynamic_smem(fn, bytes);
    if (e != cudaSuccess) return e;
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    // small programs leave most SMs out: four warps fill an SM's schedulers
    const uint32_t most = b.share > 0.0 && b.share < 1.0 ? static_cast<uint32_t>(sms * b.share) : static_cast<uint32_t>(sms);
    const uint32_t grid = std::max(1u, std::min(most, (b.runs + 3u) / 4u));
    note_launch();
    ChunkBatch arg = b;
    Prog p = one;
    void* args[] = {&arg, &p};
    return launch_cooperative(fn, grid, kThreads, args, bytes, s);
}

}  // namespace ptl
