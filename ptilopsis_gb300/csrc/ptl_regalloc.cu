// Kernels of the record form of register allocation (ptl_steps.cuh): the independent
// functions, the trigger rows, and the lane-0 functions in lock-step.  One program's view
// comes as a kernel argument, or many programs' views from device memory.
#include <cuda_runtime.h>

#include <algorithm>

#include "ptl_chunks.cuh"
#include "ptl_kernels.cuh"

namespace ptl {
namespace {

// Where a block's program and its share of it come from: one program, or the programs
// order[0..n) of a batch, program order[k] owning blocks off[k] .. off[k+1].
struct OneProgram {
    Prog P;
    __device__ void take(uint32_t block, uint32_t* local, Prog& dst) const {
        *local = block;
        const uint64_t* src = reinterpret_cast<const uint64_t*>(&P);
        uint64_t* to = reinterpret_cast<uint64_t*>(&dst);
        for (uint32_t k = threadIdx.x; k < sizeof(Prog) / 8; k += blockDim.x) to[k] = src[k];
        __syncthreads();
    }
};
struct ManyPrograms {
    const Prog* progs;
    const uint32_t* off;
    const uint32_t* order;
    uint32_t n;
    __device__ void take(uint32_t block, uint32_t* local, Prog& dst) const {
        uint32_t lo = 0, hi = n;  // off[lo] <= block < off[hi]
        if (off) {
            while (hi - lo > 1) {
                const uint32_t mid = (lo + hi) >> 1;
                if (off[mid] <= block) lo = mid; else hi = mid;
            }
            *local = block - off[lo];
        } else {  // a block per program
            lo = block;
            *local = 0;
        }
        const uint64_t* src = reinterpret_cast<const uint64_t*>(&progs[order[lo]]);
        uint64_t* to = reinterpret_cast<uint64_t*>(&dst);
        for (uint32_t k = threadIdx.x; k < sizeof(Prog) / 8; k += blockDim.x) to[k] = src[k];
        __syncthreads();
    }
};

// ---- independent functions: one thread each, one warp a block.  A step is about 70
// instructions of one dependent chain, so a warp is latency-bound and small blocks spread
// the warps over the SMs; the ring's column stride of 36 bytes spreads a warp's entries
// (different words of 32 functions) over the banks.  A lone program's functions are spread
// over more warps, per_warp each, while the chip has room (scalar_per_warp): a warp's loads
// and stores of a step go to as many lines as it has functions (4.1M nodes: the allocation
// 3.90 to 3.71 ms; 20k: 0.73 to 0.70).  A batch fills its warps.
constexpr uint32_t kFreeRing = 256, kFreeStride = 36;
template <class Src>
__global__ void __launch_bounds__(32) k_step_free(Src src, uint32_t per_warp) {
    __shared__ Prog P;
    __shared__ uint8_t ring[kFreeRing * kFreeStride];
    uint32_t local;
    src.take(blockIdx.x, &local, P);
    const uint32_t G0 = (P.F + 7u) / 8u, free_blocks = (P.F - G0 + per_warp - 1u) / per_warp;
    if (local >= free_blocks) {  // the lane-0 functions' slots: a block per run tile (with chunks only)
        const uint32_t NW = (G0 + 31u) / 32u, tile = local - free_blocks;
        const uint32_t c = tile / NW, j = tile % NW * 32u + threadIdx.x;
        if (j < G0 && s32(P.fn_size0[8u * j]) > s32(c * kChunk))
            step_slot_chunk(P, j, c, ring + threadIdx.x, kFreeStride, kFreeRing);
        return;
    }
    const uint32_t x = local * per_warp + threadIdx.x;
    if (threadIdx.x >= per_warp || x >= P.F - G0) return;
    const uint32_t f = P.ra_order ? P.ra_order[x] : (x / 7u) * 8u + (x % 7u) + 1u;
    step_free_function(P, f, ring + threadIdx.x, kFreeStride, kFreeRing);
}

// ---- the scalar generator's functions: one thread each, one warp a block.  The warp form
// (k_s_ra_warp: every lane runs the same function) took 790 cycles a step and a warp per
// function; this one takes 560 (a function a warp) to 720 (32 side by side) and a lane.
constexpr uint32_t kScalarRing = 256, kScalarStride = 36;
template <class Src>
__global__ void __launch_bounds__(32) k_step_scalar(Src src, unsigned long long* preserve, uint32_t per_warp) {
    __shared__ Prog P;
    __shared__ uint8_t ring[kScalarRing * kScalarStride];
    __shared__ uint32_t oidx[32 * 32];
    uint32_t local;
    src.take(blockIdx.x, &local, P);
    const uint32_t lane = threadIdx.x;
    step_scalar_function(P, lane < per_warp ? local * per_warp + lane : P.F, ring + threadIdx.x, kScalarStride, kScalarRing,
                         oidx + threadIdx.x, 32u, preserve ? preserve : P.s_preserve);
}

// ---- trigger rows: a block per 32 steps; lane = step, so a function's masks load
// coalesced, and the warps share out the groups.  The least group of a position is the
// first to show it on the way up, the greatest the first on the way down.
constexpr uint32_t kRowWarps = 8;
template <class Src>
__global__ void __launch_bounds__(32 * kRowWarps) k_step_rows(Src src) {
    __shared__ Prog P;
    __shared__ uint32_t lo[kRowTile][kRowPos + 1u], hi[kRowTile][kRowPos + 1u];
    __shared__ uint32_t any[kRowTile];
    uint32_t tile;
    src.take(blockIdx.x, &tile, P);
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    for (uint32_t k = threadIdx.x; k < kRowTile * (kRowPos + 1u); k += 32u * kRowWarps) {
        (&lo[0][0])[k] = kRowNone;
        (&hi[0][0])[k] = 0;
    }
    if (threadIdx.x < kRowTile) any[threadIdx.x] = 0;
    __syncthreads();
    const uint32_t i = tile * kRowTile + lane;
    const uint32_t G = (P.F + 7u) / 8u;
    uint32_t seen = 0;
    for (uint32_t g = warp; g < G; g += kRowWarps) {
        uint32_t m = group_triggers(P, g, i) & ~seen;
        seen |= m;
        for (; m; m &= m - 1) atomicMin(&lo[lane][low_bit(m)], g + 1u);
    }
    if (seen) atomicOr(&any[lane], seen);
    uint32_t left = seen;  // positions whose greatest group in this warp's share is open
    if (warp < G) {
        const uint32_t last = warp + (G - 1u - warp) / kRowWarps * kRowWarps;
        for (uint32_t g = last; __any_sync(0xFFFFFFFFu, left != 0); g -= kRowWarps) {
            uint32_t m = group_triggers(P, g, i) & left;
            left &= ~m;
            for (; m; m &= m - 1) atomicMax(&hi[lane][low_bit(m)], g + 1u);
            if (g < kRowWarps) break;
        }
    }
    __syncthreads();
    uint32_t* row = P.trow + static_cast<size_t>(tile) * kRowTile * kRowPos;
    for (uint32_t k = threadIdx.x; k < kRowTile * kRowPos; k += 32u * kRowWarps)
        row[k] = lo[k / kRowPos][k % kRowPos] | (hi[k / kRowPos][k % kRowPos] << 16);
    if (threadIdx.x < kRowTile) P.tany[tile * kRowTile + threadIdx.x] = any[threadIdx.x];
}

// ---- what the lane-0 functions' slots need (ptl_chunks.cuh): their items (a block per
// program), then each symbol's last reader (blocks as above).
template <class Src>
__global__ void __launch_bounds__(32 * kRowWarps) k_chunk_items(Src src) {
    __shared__ Prog P;
    __shared__ uint32_t part[32 * kRowWarps];
    uint32_t local;
    src.take(blockIdx.x, &local, P);
    constexpr uint32_t T = 32u * kRowWarps;
    const uint32_t G0 = (P.F + 7u) / 8u, per = (G0 + T - 1u) / T;
    const uint32_t lo = min(G0, threadIdx.x * per), hi = min(G0, lo + per);
    uint32_t sum = 0;
    for (uint32_t j = lo; j < hi; ++j) sum += chunks_of(P, j);
    part[threadIdx.x] = sum;
    __syncthreads();
    for (uint32_t d = 1; d < T; d <<= 1) {
        const uint32_t y = threadIdx.x >= d ? part[threadIdx.x - d] : 0u;
        __syncthreads();
        part[threadIdx.x] += y;
        __syncthreads();
    }
    uint32_t at = part[threadIdx.x] - sum;
    for (uint32_t j = lo; j < hi; ++j) {
        P.ch.off[j] = at;
        at += chunks_of(P, j);
    }
    if (hi == G0 && lo < hi) P.ch.off[G0] = at;
}
template <class Src>
__global__ void __launch_bounds__(32 * kRowWarps) k_chunk_last(Src src) {
    __shared__ Prog P;
    uint32_t tile;
    src.take(blockIdx.x, &tile, P);
    const uint32_t i = tile * kChunk + (threadIdx.x & 31u), G0 = (P.F + 7u) / 8u;
    for (uint32_t j = threadIdx.x >> 5; j < G0; j += kRowWarps)
        if (s32(P.fn_size0[8u * j]) > s32(i)) chunk_last_read(P, j, i);
}

// ---- lane-0 functions in lock-step: a thread per slot (slot = group), a block per
// program.  At most two barriers a step: after phase A (lookups, allocation, row-0 writes)
// and, when some slot's operand is open to other slots' triggers, after phase T, whose
// barrier also tells whether a trigger changed what phase A assumed.  Trigger rows come in tiles of 32 steps by cp.async, one tile
// ahead, and a slot's records by fours, four steps ahead: one commit group every four
// steps.  (Records in registers need the loop unrolled as often, which no longer fits the
// instruction cache; a group every step costs 130 cycles of it.)
//
// A program with many groups spreads them over the CTAs of a cluster, ascending by rank.
// Each CTA resolves a step among its own slots as above, then writes its masks into every
// CTA's shared memory; one cluster barrier later each CTA has all it needs from the
// others: a write of its own wins unless a higher rank writes the position, a trigger of
// a lower (higher) rank is before (after) any of its own.  A trigger of a lower rank that
// changes what phase A assumed is seen by every CTA in the same masks, so all of them
// agree on another round.
enum LaneMode { kAlone, kOneWarp, kManyWarps, kCluster };
constexpr uint32_t kRowBufs = 2, kClusterMax = 8, kClusterSlots = 256;
__device__ __forceinline__ void copy16_async(void* dst, const void* src) {
    const uint32_t at = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(at), "l"(src));
}
__device__ __forceinline__ void copy8_async(void* dst, const void* src) {
    const uint32_t at = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(at), "l"(src));
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::); }
constexpr uint32_t kRecBufs = 8, kRecGroup = 4;  // records per slot in shared memory, in groups; powers of two
__device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }
// Tile t's trigger rows and positions triggered at all, into buffer t % kRowBufs.
__device__ __forceinline__ void copy_rows_async(const Prog& P, uint32_t* rows, uint32_t* any, uint32_t t,
                                                uint32_t tid, uint32_t T) {
    const uint32_t b = t & (kRowBufs - 1u);
    uint32_t* to = rows + b * kRowTile * kRowPos;
    const uint32_t* from = P.trow + static_cast<size_t>(t) * kRowTile * kRowPos;
    for (uint32_t k = tid; k < kRowTile * kRowPos / 4u; k += T) copy16_async(to + 4u * k, from + 4u * k);
    for (uint32_t k = tid; k < kRowTile / 4u; k += T)
        copy16_async(any + b * kRowTile + 4u * k, P.tany + static_cast<size_t>(t) * kRowTile + 4u * k);
}

// Barriers among the first T threads of the block: one warp, or a named barrier.
template <bool kWarp>
struct LaneBarrier {
    uint32_t T;
    __device__ __forceinline__ void sync() const {
        if constexpr (kWarp) __syncwarp();
        else asm volatile("bar.sync 1, %0;" ::"r"(T) : "memory");
    }
    __device__ __forceinline__ bool any(bool v) const {
        if constexpr (kWarp) {
            __syncwarp();  // orders the lanes' stores; the vote alone does not
            return __any_sync(0xFFFFFFFFu, v);
        } else {
            uint32_t r;
            asm volatile(
                "{\n .reg .pred p, q;\n setp.ne.u32 p, %1, 0;\n bar.red.or.pred q, 1, %2, p;\n selp.u32 %0, 1, 0, q;\n}"
                : "=r"(r)
                : "r"(static_cast<uint32_t>(v)), "r"(T)
                : "memory");
            return r != 0;
        }
    }
};
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// The exchange of a cluster's masks: each CTA stores its own into every CTA's copy, and
// the stores complete transactions of the copy's mbarrier there (st.async).  No fence and
// no cluster barrier: a barrier's release would also wait for the step's global stores
// (2,600 cycles a step, measured; the step itself takes 2,000).
__device__ __forceinline__ uint32_t shared_at(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ uint32_t remote_at(uint32_t at, uint32_t rank) {
    uint32_t to;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(to) : "r"(at), "r"(rank));
    return to;
}
__device__ __forceinline__ void store_async(uint32_t to, const LaneMasks& m, uint32_t bar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.u32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(to),
                 "r"(m.wr), "r"(m.trig), "r"(m.use), "r"(m.need), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void mbar_init(const void* bar) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(shared_at(bar)) : "memory");
}
__device__ __forceinline__ void mbar_expect(const void* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(shared_at(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_test(const void* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(shared_at(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
constexpr long long kExchangeCycles = 1ll << 31;  // about a second
__device__ __forceinline__ void or_if(uint32_t on, uint32_t* p, uint32_t v) {
    asm volatile("{\n .reg .pred q;\n setp.ne.u32 q, %2, 0;\n @q red.shared.or.b32 [%0], %1;\n}" ::"r"(shared_at(p)), "r"(v),
                 "r"(on));  // read after a barrier only
}
__device__ __forceinline__ uint32_t warp_or(uint32_t v) { return __reduce_or_sync(0xFFFFFFFFu, v); }

// The masks over all slots.  One warp keeps them in registers (one slot has them already);
// more warps add theirs to the step's shared ones, complete after the next barrier.
template <int kMode>
__device__ __forceinline__ void lane_share(LaneStep& st, LaneMasks& m) {
    if constexpr (kMode == kAlone) return;
    LaneMasks all{warp_or(m.wr), warp_or(m.trig), 0, 0};
    const bool open = warp_any((m.use | m.need) != 0);
    if (open) {
        all.use = warp_or(m.use);
        all.need = warp_or(m.need);
    }
    if constexpr (kMode >= kManyWarps) {
        const uint32_t first = (threadIdx.x & 31u) == 0;
        or_if(first, &st.m.wr, all.wr);
        or_if(first, &st.m.trig, all.trig);
        if (open) {
            or_if(first, &st.m.use, all.use);
            or_if(first, &st.m.need, all.need);
        }
    } else {
        m = all;
    }
}
template <int kMode>
__device__ __forceinline__ void lane_masks(const LaneStep& st, LaneMasks& m) {
    if constexpr (kMode >= kManyWarps) m = st.m;
}

// The cluster's masks of a step, by buffer and rank.
struct LaneExchange {
    LaneMasks m[2][kClusterMax];  // 16-byte stores
    unsigned long long bar[2];    // mbarriers, one per buffer
};

// Dynamic shared memory of a CTA with T slots.
struct LaneLayout {
    uint32_t K;  // ring words per slot
    __host__ __device__ static size_t up16(size_t n) { return (n + 15u) & ~size_t(15); }  // mbarriers, 16-byte copies
    __host__ __device__ static size_t exchange_at() { return up16(sizeof(LaneShared)); }
    __host__ __device__ static size_t rows_at() { return up16(exchange_at() + sizeof(LaneExchange)); }
    __host__ __device__ static size_t any_at() { return rows_at() + kRowBufs * kRowTile * kRowPos * 4u; }
    __host__ __device__ static size_t rec_at() { return any_at() + kRowBufs * kRowTile * 4u; }
    __host__ __device__ static size_t ring_at(uint32_t T) { return rec_at() + static_cast<size_t>(T) * kRecBufs * 8u; }
    // a column per slot; the stride is not a multiple of 32 banks' 128 bytes
    __host__ __device__ static uint32_t stride(uint32_t T) { return T + 4u; }
    __host__ __device__ size_t bytes(uint32_t T) const { return ring_at(T) + static_cast<size_t>(K) * stride(T); }
};

// The program's slots [j0, j1) on the first T threads of this CTA (rank of C).
template <int kMode>
__device__ void lane_pass(const Prog& P, unsigned char* smem, uint32_t T, uint32_t K, uint32_t j0, uint32_t j1,
                          uint32_t rank, uint32_t C) {
    constexpr bool kOne = kMode == kAlone;
    const uint32_t tid = threadIdx.x, lane = tid & 31u;
    const LaneBarrier<kMode <= kOneWarp> bar{T};
    LaneShared& sh = *reinterpret_cast<LaneShared*>(smem);
    LaneExchange& ex = *reinterpret_cast<LaneExchange*>(smem + LaneLayout::exchange_at());
    uint32_t* rows = reinterpret_cast<uint32_t*>(smem + LaneLayout::rows_at());
    uint32_t* any = reinterpret_cast<uint32_t*>(smem + LaneLayout::any_at());
    unsigned long long* recs = reinterpret_cast<unsigned long long*>(smem + LaneLayout::rec_at()) + tid;  // [kRecBufs][T]
    const uint32_t G0 = (P.F + 7u) / 8u;
    auto clear_win = [&] {
        for (uint32_t p = tid; p < kRowPos; p += T) sh.st[0].win[p] = sh.st[1].win[p] = sh.st[2].win[p] = 0;
    };
    clear_win();
    if (tid == 0) {
        lane_clear(sh.st[0]);
        lane_clear(sh.st[1]);
        lane_clear(sh.st[2]);
        sh.before2 = sh.tail = 0;
        sh.s0 = 0;
        if (kMode == kCluster) {
            mbar_init(&ex.bar[0]);
            mbar_init(&ex.bar[1]);
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
            mbar_expect(&ex.bar[0], C * 16u);
            mbar_expect(&ex.bar[1], C * 16u);
        }
    }
    if (kMode == kCluster) cluster_barrier();  // every CTA's mbarriers are ready before a store to it
    bar.sync();
    LaneSlot L;
    const uint32_t j = j0 + tid;
    lane_init(P, L, j);
    if (j >= j1) L.size = 0;
    const LaneRing ring{smem + LaneLayout::ring_at(T) + tid, LaneLayout::stride(T), K};
    if (kMode == kCluster) {  // the longest lane-0 function of the whole program
        for (uint32_t g = tid; g < G0; g += T) {
            const int32_t size = s32(P.fn_size0[8u * g]);
            if (size > 0) atomicMax(&sh.s0, static_cast<uint32_t>(size));
        }
    } else if (L.size) {
        atomicMax(&sh.s0, L.size);
    }
    auto fetch = [&](uint32_t i) {  // the records of the group from step i on
#pragma unroll
        for (uint32_t k = 0; k < kRecGroup; ++k)
            if (i + k < L.size) copy8_async(recs + ((i + k) & (kRecBufs - 1u)) * T, L.rec_at + i + k);
    };
    copy_rows_async(P, rows, any, 0, tid, T);
    fetch(0);
    copy_commit();
    copy_wait();
    bar.sync();
    const uint32_t s0 = min(sh.s0, P.S);
    uint32_t turn = 0;   // exchanges so far
    uint32_t remote_m = 0, remote_bar = 0;  // where thread k < C puts this CTA's masks in CTA k
    if (kMode == kCluster && tid < C) {
        remote_m = remote_at(shared_at(&ex.m[0][rank]), tid);
        remote_bar = remote_at(shared_at(&ex.bar[0]), tid);
    }
    uint32_t at = 0;     // i % 3
    bool busy = true;
    unsigned long long next = L.size ? recs[0] : kStepIdle;
#pragma unroll 1
    for (uint32_t i = 0; i < s0; ++i) {
        if (PTL_RARE(win_wraps(i))) {
            bar.sync();
            clear_win();
            bar.sync();
        }
        LaneStep& st = sh.st[at];
        const uint32_t slot = i & (kRowBufs * kRowTile - 1u);
        const uint32_t* row = rows + slot * kRowPos;
        const uint32_t others = any[slot];
        LaneMasks m{0, 0, 0, 0};
        if (busy) {
            L.rec = next;
            lane_step_a<kOne>(sh, st, row, L, ring, i, m);
            lane_share<kMode>(st, m);
        }
        bar.sync();
        if ((i & (kRecGroup - 1u)) == kRecGroup - 1u) copy_wait();  // the next group
        if ((i & (kRecGroup - 1u)) == 0) {
            fetch(i + kRecGroup);
            if ((i & (kRowTile - 1u)) == 0 && i + kRowTile < s0) copy_rows_async(P, rows, any, i / kRowTile + 1u, tid, T);
            copy_commit();
            // a warp whose functions have ended and left row 0 only keeps the barriers
            if constexpr (kMode >= kManyWarps) busy = __any_sync(0xFFFFFFFFu, i < L.size || L.held != 0);
        }
        next = i + 1u < L.size ? recs[((i + 1u) & (kRecBufs - 1u)) * T] : kStepIdle;
        lane_masks<kMode>(st, m);
        LaneAbove above{0, 0};
        if constexpr (!kOne) {
            if (tid == 0) lane_clear(sh.st[at == 0 ? 2u : at - 1u]);
            // Jacobi rounds among this CTA's slots: until the positions triggered before
            // their owners stop changing (a DAG in group order), then the step's writes
            // and triggers again.
            uint32_t below = 0;  // triggers of lower ranks
            auto settle = [&] {
                for (uint32_t round = 0;; ++round) {
                    if (tid == 0) sh.before2 = below & m.need;
                    bar.sync();
                    if (busy) lane_round(sh, st, m, row, L);
                    bar.sync();
                    const uint32_t before = st.before, before2 = sh.before2;
                    bar.sync();
                    if (before == before2) break;
                    if (tid == 0) st.before = before2;
                    if (round > G0 + 2u) {
                        if (tid == 0) record_error(P.err, ST_DEVICE_TIMEOUT, W_RA2, i);
                        break;
                    }
                }
                for (uint32_t p = tid; p < kRowPos; p += T) st.win[p] = 0;
                if (tid == 0) st.m.wr = st.m.trig = st.later = 0;
                bar.sync();
                LaneMasks again{0, 0, 0, 0};
                if (busy) {
                    lane_emit<false>(st, L, i, again);
                    again.use = m.use;
                    again.need = m.need;
                    lane_share<kMode>(st, again);
                }
                bar.sync();
                m = again;
                lane_masks<kMode>(st, m);
                if (busy) lane_step_t(sh, st, m, L);
                bar.sync();
            };
            if (busy) lane_commit(sh, L);
            // with nothing open no trigger can act across slots: no phase T, and no barrier
            if (m.use | m.need) {
                const bool redo = busy && lane_step_t(sh, st, m, L);
                if (PTL_RARE(bar.any(redo))) settle();
            }
            if constexpr (kMode == kCluster) {
                uint32_t used = 0;  // of rank `lane`: what its last round took from lower ranks
                for (uint32_t round = 0;; ++round) {
                    // A buffer is written again two exchanges later, when every CTA has
                    // sent its part of the one between, which each does after a barrier
                    // of its own threads behind their reads of this one.
                    LaneMasks* x = ex.m[turn & 1u];
                    const void* xbar = &ex.bar[turn & 1u];
                    if (tid < C) {
                        const uint32_t off = (turn & 1u) * static_cast<uint32_t>(sizeof(ex.m[0]));
                        store_async(remote_m + off, m, remote_bar + (turn & 1u) * 8u);
                    }
                    if (busy) lane_step_b1(L, ring, i, round != 0);  // while the masks travel
                    // The first warp waits for the masks, then the block's barrier lets the
                    // others at them and tells all whether the wait gave up.
                    bool lost = false;
                    if (tid < 32u) {
                        const uint32_t parity = (turn >> 1) & 1u;
                        const long long since = clock64();
                        while (!lost && !mbar_test(xbar, parity)) lost = clock64() - since > kExchangeCycles;
                        if (lane == 0) mbar_expect(xbar, C * 16u);  // its next phase
                    }
                    if (bar.any(lost)) {
                        if (tid == 0) record_error(P.err, ST_DEVICE_TIMEOUT, W_RA2, i);
                        return;  // this CTA sends no more, so the others' waits end too
                    }
                    ++turn;
                    const LaneMasks theirs = lane < C ? x[lane] : LaneMasks{0, 0, 0, 0};
                    above.wr = warp_or(lane > rank ? theirs.wr : 0u);
                    above.trig = warp_or(lane > rank ? theirs.trig : 0u);
                    // every rank's triggers from lower ranks: a prefix over the lanes
                    uint32_t takes = 0;
                    if (warp_any(theirs.need != 0)) {
                        uint32_t lower = theirs.trig;
#pragma unroll
                        for (uint32_t d = 1; d < kClusterMax; d <<= 1) {
                            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, lower, d);
                            if (lane >= d) lower |= y;
                        }
                        lower = __shfl_up_sync(0xFFFFFFFFu, lower, 1);
                        takes = lane > 0 ? lower & theirs.need : 0u;
                    }
                    if (!warp_any(takes != used)) {
                        m.wr = warp_or(theirs.wr);
                        m.trig = warp_or(theirs.trig);
                        break;
                    }
                    if (round > G0 + 2u) {
                        if (tid == 0) record_error(P.err, ST_DEVICE_TIMEOUT, W_RA2, i);
                        break;
                    }
                    used = takes;
                    below = __shfl_sync(0xFFFFFFFFu, takes, static_cast<int>(rank));
                    settle();
                }
            }
        } else {
            lane_commit(sh, L);
        }
        if (busy) {
            if constexpr (kMode != kCluster) lane_step_b1(L, ring, i, false);
            lane_step_b2<kOne>(sh, st, m, above, others, L, ring, i);
        }
        at = at == 2u ? 0u : at + 1u;
    }
    uint32_t tail = 0;
    for (uint32_t i = s0 + tid; i < P.S; i += T) tail |= P.tany[i];
    if (tail) atomicOr(&sh.tail, tail);
    bar.sync();
    tail = sh.tail;
    lane_commit(sh, L);
    lane_tail(sh, L, tail);
}

// Whether the lane-0 functions are still to be done.
__device__ bool lock_step(const Prog& P) { return !P.ch.lock || *P.ch.lock != 0; }

// The block has the threads of the widest listed program; a narrower one's extra warps
// leave at once.
template <class Src, int MAXT>
__global__ void __launch_bounds__(MAXT) k_step_lane0(Src src, uint32_t K) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ Prog P;
    uint32_t local;
    src.take(blockIdx.x, &local, P);
    if (P.S == 0 || !lock_step(P)) return;
    const uint32_t G0 = (P.F + 7u) / 8u;
    const uint32_t T = min(blockDim.x, (G0 + 31u) & ~31u);
    if (threadIdx.x >= T) return;
    if (G0 == 1u) lane_pass<kAlone>(P, smem, T, K, 0, G0, 0, 1);
    else if (T == 32u) lane_pass<kOneWarp>(P, smem, T, K, 0, G0, 0, 1);
    else lane_pass<kManyWarps>(P, smem, T, K, 0, G0, 0, 1);
}
template <int MAXT>
__global__ void __launch_bounds__(MAXT) k_step_lane0_cluster(OneProgram src, uint32_t K, uint32_t per_cta) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ Prog P;
    uint32_t local;
    src.take(0, &local, P);
    if (!lock_step(P)) return;  // every CTA alike
    const uint32_t G0 = (P.F + 7u) / 8u, C = gridDim.x;
    const uint32_t rank = cluster_rank();
    const uint32_t j0 = rank * per_cta, j1 = min(G0, j0 + per_cta);
    lane_pass<kCluster>(P, smem, blockDim.x, K, j0, j1, rank, C);
    cluster_barrier();  // none ends while another may still write to it
}

// Ring words per slot: a power of two of at most `most`, within the budget.
LaneLayout lane_layout(uint32_t T, uint32_t most) {
    constexpr size_t kBudget = 200u * 1024u;
    LaneLayout l{most};
    while (l.K > 4u && l.bytes(T) > kBudget) l.K >>= 1;
    return l;
}

template <class Src>
cudaError_t launch_lane0(const Src& src, uint32_t programs, uint32_t max_g0, uint32_t ring, cudaStream_t s) {
    const uint32_t T = (max_g0 + 31u) & ~31u;
    const LaneLayout l = lane_layout(T, ring);
    auto go = [&](auto kernel) -> cudaError_t {
        const cudaError_t e = allow_dynamic_smem(reinterpret_cast<const void*>(kernel), l.bytes(T));
        if (e != cudaSuccess) return e;
        note_launch();
        kernel<<<programs, T, l.bytes(T), s>>>(src, l.K);
        return cudaGetLastError();
    };
    return T <= 256u ? go(k_step_lane0<Src, 256>) : go(k_step_lane0<Src, 1024>);
}

// The lane-0 pass of one program on a cluster; *placed: whether the device can place it
// (nothing is launched otherwise, nor with dry set).
cudaError_t launch_lane0_cluster(const Prog& P, uint32_t G0, cudaStream_t s, bool dry, bool* placed) {
    *placed = false;
    const uint32_t C = std::min(kClusterMax, (G0 + kClusterSlots - 1u) / kClusterSlots), per_cta = (G0 + C - 1u) / C;
    const uint32_t T = (per_cta + 31u) & ~31u;
    const LaneLayout l = lane_layout(T, 256u);
    auto go = [&](auto kernel) -> cudaError_t {
        const void* fn = reinterpret_cast<const void*>(kernel);
        cudaError_t e = allow_dynamic_smem(fn, l.bytes(T));
        if (e != cudaSuccess) return e;
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(C);
        cfg.blockDim = dim3(T);
        cfg.dynamicSmemBytes = l.bytes(T);
        cfg.stream = s;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = C;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        int clusters = 0;
        if (cudaOccupancyMaxActiveClusters(&clusters, fn, &cfg) != cudaSuccess || clusters < 1) {
            cudaGetLastError();
            return cudaSuccess;
        }
        *placed = true;
        if (dry) return cudaSuccess;
        note_launch();
        return cudaLaunchKernelEx(&cfg, kernel, OneProgram{P}, l.K, per_cta);
    };
    return T <= 256u ? go(k_step_lane0_cluster<256>) : go(k_step_lane0_cluster<1024>);
}

}  // namespace

bool step_cluster_fits(uint32_t G0) {
    bool placed = false;
    return G0 <= kClusterMax * 1024u && launch_lane0_cluster(Prog{}, G0, nullptr, true, &placed) == cudaSuccess && placed;
}

cudaError_t run_step_regalloc(const Prog& P, const ChunkBatch* chunks, cudaStream_t s) {
    const OneProgram src{P};
    const uint32_t G0 = (P.F + 7u) / 8u, free_fns = P.F - G0;
    const uint32_t tiles = static_cast<uint32_t>(row_tiles(P.S));
    if (chunks) {
        note_launch();
        k_chunk_items<<<1, 32u * kRowWarps, 0, s>>>(src);
        note_launch();
        k_chunk_last<<<tiles, 32u * kRowWarps, 0, s>>>(src);
    }
    const uint32_t per = std::max(1u, scalar_per_warp(free_fns));
    const uint32_t blocks = (free_fns + per - 1u) / per + (chunks ? chunks->runs : 0u);
    if (blocks) {
        note_launch();
        k_step_free<<<blocks, 32, 0, s>>>(src, per);
    }
    if (tiles == 0) return cudaGetLastError();
    note_launch();
    k_step_rows<<<tiles, 32u * kRowWarps, 0, s>>>(src);
    if (chunks) {
        const cudaError_t e = run_lane_chunks(*chunks, P, s);
        if (e != cudaSuccess) return e;
    }
    // the lock-step, where that has not done it (lock_step)
    if (G0 > kStepClusterMin) {
        bool placed = false;
        const cudaError_t e = launch_lane0_cluster(P, G0, s, false, &placed);
        if (e != cudaSuccess || placed) return e;
        if (G0 > kStepBlockMax) return cudaErrorInvalidConfiguration;  // not a program of this form (ra_form)
    }
    return launch_lane0(src, 1, G0, 1024u, s);
}

// Functions per warp: a warp's step takes the branches of all its lanes, so as few as keep
// the chip's warps busy (one function: 560 cycles a step; 32 side by side: 720).
uint32_t scalar_per_warp(uint64_t functions) {
    constexpr uint64_t kWarps = 152u * 8u;
    return static_cast<uint32_t>(std::min<uint64_t>(32, (functions + kWarps - 1u) / kWarps));
}

cudaError_t run_step_scalar(const Prog& P, unsigned long long* preserve, cudaStream_t s) {
    note_launch();
    const uint32_t per = scalar_per_warp(P.F);
    k_step_scalar<<<(P.F + per - 1u) / per, 32, 0, s>>>(OneProgram{P}, preserve, per);
    return cudaGetLastError();
}

cudaError_t batch_step_scalar(const StepBatch& b, cudaStream_t s) {
    if (b.n == 0 || b.free_blocks == 0) return cudaSuccess;
    note_launch();
    k_step_scalar<<<b.free_blocks, 32, 0, s>>>(ManyPrograms{b.progs, b.free_off, b.order, b.n}, nullptr, b.per_block);
    return cudaGetLastError();
}

cudaError_t batch_step_regalloc(const StepBatch& b, cudaStream_t s) {
    if (b.n == 0) return cudaSuccess;
    if (b.chunks) {
        note_launch();
        k_chunk_items<<<b.chunks->n, 32u * kRowWarps, 0, s>>>(ManyPrograms{b.progs, nullptr, b.chunks->order, b.chunks->n});
        note_launch();
        k_chunk_last<<<b.chunks->tiles, 32u * kRowWarps, 0, s>>>(
            ManyPrograms{b.progs, b.chunks->tile_off, b.chunks->order, b.chunks->n});
    }
    if (b.free_blocks) {
        note_launch();
        k_step_free<<<b.free_blocks, 32, 0, s>>>(ManyPrograms{b.progs, b.free_off, b.order, b.n}, 32u);
    }
    if (b.row_blocks) {
        note_launch();
        k_step_rows<<<b.row_blocks, 32u * kRowWarps, 0, s>>>(ManyPrograms{b.progs, b.row_off, b.order, b.n});
    }
    if (b.chunks) {
        const cudaError_t e = run_lane_chunks(*b.chunks, Prog{}, s);
        if (e != cudaSuccess) return e;
    }
    return launch_lane0(ManyPrograms{b.progs, nullptr, b.order, b.n}, b.n, b.max_g0, 128u, s);
}

}  // namespace ptl
