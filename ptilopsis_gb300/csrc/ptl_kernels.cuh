// Kernel launch interface of the GB300 code generator (ptl_kernels.cu).
#pragma once

#include <cuda_runtime.h>

#include "ptl_device.h"
#include "ptl_stages.cuh"
#include "ptl_sort.cuh"
#include "ptl_scalar.cuh"

namespace ptl {

// Device scratch that a compile needs besides the Prog arrays; sized by the arena.
struct SortScratch {
    unsigned long long* a;     // (key, index) pairs, n
    uint32_t* apos;            // L-stop positions by rank, n
    uint32_t* bpos;            // R-stop positions by rank from the right, n
    SortSeg* seg[2];           // segment lists of this and the next round
    uint32_t seg_cap;
    uint32_t* tile_seg;        // tile -> segment
    uint32_t* tile_l;          // L-stop count per tile, then its exclusive offset
    uint32_t* tile_r;
    uint32_t* stops;           // per tile: its keys' L-stop bits, then their R-stop bits
                               // (kSortTile / 32 words each), written by the count pass
    uint32_t tile_cap;
    uint32_t* leaf;            // leaf ranges (first, last)
    uint32_t* heap;            // heap-sorted ranges
    uint32_t leaf_cap;
    uint32_t* local;           // ranges of at most kSortBlock keys (first, last, depth budget),
                               // finished one block each (k_sort_block)
    uint32_t* equal;           // equal-key ranges (first, last) found by the rounds
    uint32_t* counters;        // [0] tiles [1] next segments [2] leaves [3] heaps [4] segments of
                               // this round [5] capacity overflow [6] block ranges [7] equal ranges
};

constexpr size_t kScanTileElems = 4096;  // elements per scan tile (ptl_kernels.cu)

struct ScanScratch {
    unsigned long long* status;  // per tile: (flag << 32) | value
    uint32_t* counter;           // dynamic tile ticket
    uint32_t tile_cap;
};

// Kernel launches issued by this library since load (counted at each launch site).
uint64_t launch_count();
void note_launch();
// Raises a kernel's dynamic shared memory limit to at least bytes (never lowers it).
cudaError_t allow_dynamic_smem(const void* kernel, size_t bytes);
// A launch whose blocks wait on one another.  Launches from several streams take turns:
// two that are each resident in part would wait for good.
cudaError_t launch_cooperative(const void* kernel, uint32_t blocks, uint32_t threads, void** args, size_t smem, cudaStream_t s);

// Up to kZeroMost memory ranges zeroed by one launch: a compile clears some 45 buffers,
// and a memset of a small one costs the stream about 2 us whatever its size.  Ranges start
// on 16-byte boundaries; their lengths round up to 16 bytes (allocations are in whole 16-byte
// words).  launch_zero refuses a list that was given more.
constexpr int kZeroMost = 24;
struct ZeroList {
    uint4* p[kZeroMost];
    uint64_t n16[kZeroMost];
    int count = 0;
    void add(void* q, size_t bytes) {
        if (count < kZeroMost) {
            p[count] = static_cast<uint4*>(q);
            n16[count] = cleared_bytes(bytes) / 16u;
        }
        ++count;
    }
};
cudaError_t launch_zero(const ZeroList& z, cudaStream_t s);

// Element-wise stages (grid-stride launches of the per-thread functions).
void launch_ingest(const Prog& P, cudaStream_t s);  // input checks + copy; flags[3]: max_depth reached
void launch_preprocess(const Prog& P, cudaStream_t s);
void launch_count_scan(const Prog& P, const ScanScratch& sc, cudaStream_t s);
void launch_fix(const Prog& P, cudaStream_t s);
void launch_decl_scan(const Prog& P, uint32_t* flags_tmp, const ScanScratch& sc, cudaStream_t s);
void launch_functab(const Prog& P, uint32_t* meta, cudaStream_t s);

void launch_gen(const Prog& P, cudaStream_t s);
// work: optimize_work_bytes(W) of scratch, 16-byte aligned.
size_t optimize_work_bytes(uint32_t W);
cudaError_t run_optimize(const Prog& P, void* work, cudaStream_t s, uint32_t* sweeps_out);
// Register allocation of one program.  ra_form builds the step records (P.rec) and tells
// which form the program takes; the caller then provides that form's arrays:
//   Steps: tmask (one per word), trow and tany (row_tiles(S) tiles of kRowTile steps);
//   General: trig_min / trig_max (set to none), ra_chunks, and defpos (ra_positions_tell);
//   Serial: none.
struct ChunkBatch;
enum class RaForm { Steps, General, Serial };
// items: chunks of the lane-0 functions.
cudaError_t ra_form(const Prog& P, cudaStream_t s, bool general, RaForm* form, uint32_t* items);
// General form: whether definition positions (P.defpos, zeroed) tell where row 0 has a
// symbol: no virtual register of a lane-0 function has two definitions, and no word is in
// two functions.  P.stamp: zeroed.
cudaError_t ra_positions_tell(const Prog& P, cudaStream_t s, bool* tell);
// Where positions pay, measured through the general form, positions and hash, ms: one lane-0
// function (which then has a form of its own) 132 and 364 with 111k nodes, 9 and 300 functions
// 24.8 and 29.3, 15.6 and 18.1, 1,025 on a cluster 10.45 and 10.88; several groups a thread
// of one block 3.95 and 3.80 (1,025 groups), 19.7 and 18.8 (4,125).
bool ra_positions_pay(uint32_t G0);
cudaError_t run_regalloc_steps(const Prog& P, RaForm form, const ChunkBatch* chunks, cudaStream_t s);

// The lane-0 functions in chunks of steps (ptl_chunks.cuh): of one program (progs null),
// or of the programs order[0..n) of a batch, program order[k] having the run tiles
// run_off[k].. (a chunk of 32 functions each) and the row tiles tile_off[k]..  sync:
// chunk_sync_words zeroed words.  A program that does not settle, or whose symbols do not
// fit the slots, has its lock set: the lock-step, launched after, does it.
struct ChunkSizes {  // offsets in bytes into the program's arrays; [0, zeroed) start as zeros
    uint64_t last, reach, slots, need, tag, delta, dirty, moved, lock, zeroed, off, rec, out, state, row, win, pair, touch, total;
    uint64_t runs, tiles;
};
ChunkSizes chunk_sizes(uint32_t F, uint32_t S, uint32_t W, uint32_t items);
void chunk_bind(LaneChunks& ch, const ChunkSizes& z, void* zeroed, void* rest);
constexpr long long kChunkWait = 1ll << 31;  // about a second
struct ChunkBatch {
    const Prog* progs;
    const uint32_t* order;
    const uint32_t* run_off;   // [n + 1]
    const uint32_t* tile_off;  // [n + 1]
    uint32_t n, runs, tiles;
    uint32_t classes;          // chunk_class of the programs, or'ed
    uint32_t rounds;           // at most
    uint32_t* sync;
    double share;              // part of the SMs the launch may take (0: all)
    long long wait = kChunkWait;  // cycles that a block waits for the others
};
// Steps from which on chunks pay.  Their passes and rounds have a cost of their own, about
// 0.12 ms: with 403 steps (one function) the allocation took 0.36 ms in lock-step and 0.45
// in chunks, with 1,449 (two functions) 1.46 and 0.65.  At other widths, lock-step below and
// chunks above the line, ms: 8 lane-0 functions of 605 steps 0.75, of 1,093 0.91; 64 of 614
// 1.03, of 1,176 1.46; 512 of 591 2.76, of 1,210 2.88; 1,024 of 613 3.85, of 1,175 4.54.
constexpr uint32_t kChunkMinSteps = 768;
// Lane-0 functions up to which one warp, and four, fold a chunk's rows (else a block).
constexpr uint32_t kChunkNarrow = 16, kChunkWide = 128;
inline uint32_t chunk_class(uint32_t G0) { return G0 <= 1u ? 1u : (G0 <= kChunkNarrow ? 2u : (G0 <= kChunkWide ? 4u : 8u)); }
// Batches: the lock-step runs programs side by side, so it lasts as long as its longest
// program, where chunks last as long as all their runs.  Measured cycles: a lock-step's
// step 1,000 with one lane-0 function, 1,450 with up to 32, 2,350 with more; a round, of a
// sixth of the chunks and some, 20,000 and for each wave of 2,432 runs (16 warps on 152 SMs)
// 15,000, with more than kChunkNarrow functions (which run again more often, and have folds)
// four times as much.  64 programs of up to 4,575 steps took 3.0 to 4.3 ms in lock-step and
// 2.0 to 2.6 in chunks, 512 of up to 4,058 steps and 64 functions 8.4 and 18.5.
//
// The rule counts all SMs also for a batch held to a share of them.  At half of them that is
// right for the few large programs of a compile server's lane (16 of 100k to 2M nodes 7.1 ms
// in chunks, 13.0 in lock-step) and wrong for many middling ones (128 of 70k nodes 9.7 and
// 7.4); with the waves of the share the first would go the wrong way.
inline uint64_t lock_step_cycles(uint64_t S, uint32_t G0) { return S * (G0 <= 1u ? 1000u : (G0 <= 32u ? 1450u : 2350u)); }
inline uint64_t chunk_work(uint64_t tiles, uint32_t G0) { return tiles * ((G0 + 31u) / 32u) * (G0 <= kChunkNarrow ? 1u : 4u); }
inline bool chunk_pays(uint64_t tiles, uint64_t work, uint64_t before, uint64_t after) {
    return (tiles / 6u + 6u) * (20000u + 15000u * work / 2432u) + after < before;
}
// Rounds before the lock-step takes over: they have been 10 for 18 chunks, 30 for 148 and 100
// for 175.
inline uint32_t chunk_rounds(uint32_t tiles) { return tiles + 64u; }
// Other limits of a generator or a batch (0: the above), so that tests see what comes after.
struct ChunkLimits {
    uint32_t rounds = 0;
    long long wait = 0;
    void apply(ChunkBatch& b) const {
        if (rounds) b.rounds = rounds < b.rounds ? rounds : b.rounds;  // b.sync has words for no more
        if (wait) b.wait = wait;
    }
};
inline uint32_t chunk_sync_words(uint32_t rounds) { return rounds + 4u; }
cudaError_t run_lane_chunks(const ChunkBatch& b, const Prog& one, cudaStream_t s);
bool chunks_fit();  // whether the current device can run its blocks together (else the lock-step)
// The record form of one program, and of the programs order[0..n) of a batch: program
// order[k] has its independent functions (32 a block) in blocks free_off[k].. and its
// trigger rows (kRowTile steps a block) in blocks row_off[k]..
// The lane-0 pass of a program with more than kStepClusterMin groups runs on a
// thread-block cluster where the device can place one; with more than kStepBlockMax it
// has to (else the program takes the general form).
constexpr uint32_t kStepClusterMin = 256, kStepBlockMax = 1024;
bool step_cluster_fits(uint32_t G0);
bool ra_cluster_disabled();
cudaError_t run_step_regalloc(const Prog& P, const ChunkBatch* chunks, cudaStream_t s);
struct StepBatch {
    const Prog* progs;
    const uint32_t* order;
    const uint32_t* free_off;  // [n + 1]
    const uint32_t* row_off;   // [n + 1]
    uint32_t n, free_blocks, row_blocks, max_g0;
    uint32_t per_block;        // batch_step_scalar: functions per block (scalar_per_warp)
    const ChunkBatch* chunks;  // the programs in chunks (each with a block per run tile for its slots behind its independent functions'), or null
};
cudaError_t batch_step_regalloc(const StepBatch& b, cudaStream_t s);
uint32_t scalar_per_warp(uint64_t functions);
// The same for the scalar generator (free_off: blocks of per_block functions), leaving the
// preserve masks (one program: preserve; a batch: each program's s_preserve).
cudaError_t run_step_scalar(const Prog& P, unsigned long long* preserve, cudaStream_t s);
cudaError_t batch_step_scalar(const StepBatch& b, cudaStream_t s);
// Lane-0 passes too wide for one block: programs with more than kRaClusterMin lane-0
// groups (at most 8,192) run theirs on a thread-block cluster when the device can place
// it.  ra_cluster_fits tells whether it can; launch_ra_wide launches the program's
// independent functions (Pfree: no definition positions), then the cluster pass (P0),
// and sets *launched, or launches nothing.
constexpr uint32_t kRaClusterMin = 1024;
bool ra_cluster_fits(uint32_t G0);
cudaError_t launch_ra_wide(const Prog& P0, const Prog& Pfree, uint32_t G0, cudaStream_t s, bool* launched);
void launch_regalloc_count_scan(const Prog& P, const ScanScratch& sc, cudaStream_t s);
void launch_regalloc_emit(const Prog& P, cudaStream_t s);
void launch_fixjumps_scan(const Prog& P, const ScanScratch& sc, cudaStream_t s);
void launch_fixjumps_emit(const Prog& P, cudaStream_t s);

// The scalar generator's stages where they differ (ptl_scalar.cuh).  Register
// allocation: scalar_ra_form builds the step records (functions naming each other's words
// take the serial order, words that a record cannot say the general form, a warp or a
// thread per function), then that form's launch (regs: F x 64, steps: F),
// each leaving the preserve masks; the count scan with the preserve words (extra: wb8
// counts); the scatter, the moved function table and the frame words (claim: W2 keys).
void launch_preprocess_scalar(const Prog& P, cudaStream_t s);
void launch_gen_scalar(const Prog& P, cudaStream_t s);
cudaError_t scalar_ra_form(const Prog& P, cudaStream_t s, RaForm* form);
void launch_scalar_ra_free(const Prog& P, unsigned long long* preserve, cudaStream_t s);
void launch_scalar_ra_serial(const Prog& P, int32_t* regs, SRaStep* steps, unsigned long long* preserve,
                             cudaStream_t s);
void launch_scalar_ra_count_scan(const Prog& P, const unsigned long long* preserve, uint32_t* extra,
                                 const ScanScratch& sc, cudaStream_t s);
void launch_scalar_ra_emit(const Prog& P, const unsigned long long* preserve, unsigned long long* claim,
                           cudaStream_t s);

// Two partition rounds as one CUDA graph.  Every launch of a round takes its arguments
// from the scratch layout (pointers, capacities) and reads its counts on the device, and
// the segment lists alternate, so a pair of rounds ends where it began and replays as one
// graph launch.  Captured on first use and again when the layout changes.
struct SortRoundGraph {
    cudaGraphExec_t exec = nullptr;
    SortScratch ss{};
    ErrorWord* err = nullptr;
    SortRoundGraph() = default;
    SortRoundGraph(const SortRoundGraph&) = delete;
    SortRoundGraph& operator=(const SortRoundGraph&) = delete;
    ~SortRoundGraph() {
        if (exec) cudaGraphExecDestroy(exec);
    }
};

// Depth-order emulation; returns a CUDA error and needs the host for its round loop.
cudaError_t run_depth_sort(const Prog& P, const SortScratch& ss, cudaStream_t s, uint32_t* rounds_out,
                           SortRoundGraph* graph = nullptr);

// Introsort rounds over prepared segments (ss.seg[0], counters), then heaps and leaves.
// With graph, rounds run as replays of a captured pair.
cudaError_t run_sort_rounds(const SortScratch& ss, uint32_t nseg0, uint32_t first_batch, uint32_t max_rounds,
                            ErrorWord* err, cudaStream_t s, uint32_t* rounds_out, SortRoundGraph* graph = nullptr);

// ---- batched programs: per-program Prog views in device memory (progs[B]); off[B+1]
// holds each program's first tile for the stage's element count.
struct BatchLaunch {
    const Prog* progs;
    const uint32_t* off;   // tile table built with `tile` elements per tile
    uint32_t B;
    cudaStream_t s;
    uint32_t tile;
};
enum class BatchStage {
    Ingest, Preprocess, Fix, Functab, Gen, OptMark, OptFinal, InitLifetime, Records, ScalarRecords, ScalarRange, Definitions, Ranges, RaHist, Spill,
    Scatter, RaFunctab, FjEmit, FjFunctab,
    // the scalar generator's (ptl_scalar.cuh): preprocess, isn_gen, preserve counts
    // (per function), scatter (per word), the function table after regalloc (per
    // function), the frame words and preserve stores (3 items per function)
    PreprocessScalar, GenScalar, SPreserveCounts, SScatter, SFunctab, SFrames
};
enum class BatchScan { Count, Decl, RaCount, FjSize, SRaCount };
uint32_t batch_tile();       // default elements per tile of the element-wise stages
// Tile sizes the element-wise kernels and the optimize sweeps accept (powers of two).
bool batch_tile_ok(uint32_t tile);
bool batch_sweep_tile_ok(uint32_t tile);
uint32_t batch_scan_tile();  // elements per scan tile
void batch_stage(BatchStage st, const BatchLaunch& bl, uint32_t total, uint32_t* meta);

// Batched arenas: a program's region in an array family holds kArenaFront zero elements,
// its elements, then zeros up to the next multiple of 32 that is at least kArenaBack past
// them (stages read a little before and past a program's elements).
constexpr uint64_t kArenaFront = 16, kArenaBack = 80;
PTL_HD uint64_t arena_region(uint64_t count) { return (count + kArenaFront + kArenaBack + 31) & ~uint64_t(31); }
// Families whose elements the stages write in full before reading them; only the pads
// need zeroing, which batch_guards does (per program, region(count) - written elements):
//   Nodes: nt rt nd1 nd par ci dep loc0 loc fflag, written [0, nb8), count nb8;
//   Words: used_instrs spill roffs, written from [0, W), count wb8;
//   Words2: joffs, written [0, w2b8), count w2b8 + 16.
enum class ArenaGuard { Nodes, Words, Words2 };
void batch_guards(ArenaGuard g, const BatchLaunch& bl, uint32_t total);
void batch_sort_keys(const BatchLaunch& bl, uint32_t total, unsigned long long* a, const uint64_t* aoff, bool out);
// One optimize sweep over the tiles marked in cur (all when cur is null); marks in next
// the tiles a cleared mark makes live again.  Both hold total + 1 bytes: the last says
// whether any tile is marked (a sweep with none returns at once).  Valid only when the
// OptMark stage found every virtual result to be its instruction's own word (its flag
// 0); otherwise pass cur = null.
void batch_sweep(const BatchLaunch& bl, uint32_t total, uint32_t* changed, const uint8_t* cur, uint8_t* next);

// One input field of every program copied from the caller's host arrays into the device
// input arena by a kernel that reads host memory directly (devices with coherent access
// to pageable memory).  Program p's elements go to dst + din[p] * esize, din[p] a multiple
// of 16; the table bl.off counts tiles of kGatherTile elements per program.
struct HostGather {
    const void* const* src;  // [B] host arrays of this field
    const uint64_t* din;     // [B] first element in dst
    const uint64_t* n;       // [B] elements
    uint8_t* dst;
    uint32_t esize;          // 1 or 4
};
constexpr uint32_t kGatherTile = 32768;
void batch_gather_host(const BatchLaunch& bl, uint32_t total, const HostGather& g);
// A kernel copying bytes (a multiple of 16, both 16-byte aligned) from host memory it
// reads directly into device memory.
cudaError_t read_host(const void* src, void* dst, size_t bytes, cudaStream_t s);
// Copies bytes between memories a kernel can address (device memory, pinned host memory,
// pageable host memory where the device accesses it coherently), both 16-byte aligned,
// with kernel loads and stores: over the host link faster than the copy engine here.
cudaError_t kernel_copy(const void* src, void* dst, size_t bytes, cudaStream_t s);
void batch_scan(BatchScan which, const BatchLaunch& bl, uint32_t tiles, const ScanScratch& sc, uint32_t* meta);
void batch_sizes(bool w3, const Prog* progs, const uint32_t* list, uint32_t count, uint32_t* meta, cudaStream_t s);
// ra_order of each listed program: its independent functions, longest first.
void batch_free_order(const Prog* progs, const uint32_t* list, uint32_t count, cudaStream_t s);
void batch_serial(const Prog* progs, const uint32_t* list, uint32_t count, cudaStream_t s);
// Register allocation steps of n programs in one persistent launch: program order[k]
// owns work items item_off[k] .. item_off[k+1] (its independent functions in tiles of
// batch_ra_threads(max_g0), then its lane-0 pass, which follows their progress through
// the program's ra_chunks record: histogram (BatchStage::RaHist) then zeroed counts).
uint32_t batch_ra_threads(uint32_t max_g0);
// The scalar generator's register allocation of the listed programs' functions, one warp
// per function (a tile: scalar_warp_fns() functions of one program; the tile table over
// F in bl), each warp with `stride` symbol bytes (at least the listed programs' longest
// function, at most scalar_warp_cap()).  The serial and tile forms run per program
// through launch_scalar_ra_serial / launch_scalar_ra_free.
void batch_scalar_ra_warp(const BatchLaunch& bl, uint32_t total, uint32_t stride);
uint32_t scalar_warp_fns();
uint32_t scalar_warp_cap();
// share: the part of the device's resident blocks the persistent launch may take (1 =
// all; less leaves room for other streams' kernels, e.g. a compile server's other lanes).
cudaError_t batch_regalloc(const Prog* progs, const uint32_t* item_off, const uint32_t* order, uint32_t n,
                           uint32_t items, uint32_t max_g0, uint32_t* queue, cudaStream_t s, double share = 1.0);

}  // namespace ptl
