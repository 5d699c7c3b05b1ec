// AST flattening on the GPU (ptl_flatten in include/ptl_codegen.h).
//
// Replaces DepthTree::DepthTree(ASTNode*) (pareas-ast/src/codegen/depthtree.cpp:11-100):
// a depth-first walk of the parser's pointer tree that emits each node after its
// children (children in order), with its depth, its child index (SIZE_MAX, -1 as int32,
// for the root) and its parent rewritten to the emitted index.  A pointer tree does not
// cross to a GPU, so the input here is the same tree as arrays in any node order -- what a
// parser that builds nodes in parallel produces: node v's parent is parent[v] (-1 for the
// root) and its place among the parent's children is child_idx[v].
//
// The walk becomes an Euler tour and a list ranking:
//   1. children per node (the greatest child index + 1; their sum must be n - 1), an
//      exclusive scan, each child in its slot off[parent] + child_idx: a child index out
//      of range or taken twice, or a slot left empty, is an error;
//   2. the tour: events enter(v) = 2v and exit(v) = 2v+1, and an end event 2n.  enter(v)
//      goes to enter(first child) or exit(v); exit(v) to enter(next sibling), exit(parent)
//      or, for the root, the end;
//   3. the ranking by splitters: one event in 16 or 32 (ptl_flatten.cuh) and the root's
//      enter.  A thread per splitter walks the tour to the next splitter and sums two
//      weights -- 1 per exit (post-order: v's index is n minus the exits from exit(v) on)
//      and +1 per enter / -1 per exit (depth); pointer jumping sums them over the splitters
//      to the end; a second walk gives every node its index and depth;
//   4. the six arrays in post-order.
// The root's enter must see all n exits; fewer means nodes the root does not reach (a
// cycle of parents), an INVALID_AST.  No kernel waits on another block.
//
// What bounds it: random 4-byte reads of the tour out of L2, twice, by dependent chains of
// some 16 to 32 events (the longest, about ln(splitters) times that, ends last).  4.3M
// nodes on the device: 0.90 ms; pointer jumping over all events, which read and wrote 32
// bytes per event in each of 24 rounds, with a same-address atomic per node for the depth
// and per child for the counts, took 4.1 ms.  Where some walk is longer than walk_most (the
// nodes' numbers follow the hash), that ranking is done after all.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "../../include/ptl_codegen.h"
#include "ptl_device.h"
#include "ptl_flatten.cuh"

namespace {

using namespace ptl;

constexpr int kThreads = 256;
constexpr uint32_t kEmpty = 0xFFFFFFFFu;
constexpr int kScanThreads = 1024;
constexpr uint32_t kScanTile = 4096;  // elements per scan tile (4 per thread)

struct Rank {
    uint32_t next;  // splitter further on (count: the end)
    uint32_t exits; // exits from here up to there
    int32_t level;  // enters minus exits
    uint32_t pad;
};

// A node's inputs, one sector of a random read.
struct NodeRec {
    int32_t parent, child;
    uint32_t data, types;
};

// An event of the ranking by pointer jumping over all of them.
struct Event {
    uint32_t next;   // event further on (2n: the end)
    uint32_t exits;  // exits from here up to there
    int32_t level;   // enters minus exits
    uint32_t pad;
};

constexpr uint32_t kFar = 2;  // some walk is longer than walk_most: the ranking is still to be done

struct FlatErr {
    uint32_t code;     // 0 ok, 1 invalid, kFar
    uint32_t detail;   // the first node found bad
    uint32_t roots;    // nodes with parent -1
    uint32_t max_depth;
    uint32_t reached;  // exits the root's enter sees
    uint32_t splitters;
    unsigned long long slots;  // sum of the children counts
};

__device__ void flag(FlatErr* e, uint32_t v) {
    if (atomicCAS(&e->code, 0u, 1u) == 0u) e->detail = v;
}

#define FL_FOR(i, count)                                                                  \
    for (uint64_t i##_ = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;    \
         i##_ < (count); i##_ += static_cast<uint64_t>(gridDim.x) * blockDim.x)           \
        if (const uint32_t i = static_cast<uint32_t>(i##_); true)

unsigned grid_of(uint64_t n) {
    return static_cast<unsigned>(std::max<uint64_t>(1, std::min<uint64_t>((n + kThreads - 1) / kThreads, 152u * 16u)));
}

// one thread per splitter: the walks are latency-bound
unsigned walk_grid(uint64_t n) { return static_cast<unsigned>(std::max<uint64_t>(1, (n + kThreads - 1) / kThreads)); }

// children per node (greatest child index + 1); the root; the nodes' records.  deg is
// read before it is raised: with the children of a node in any order few of them raise
// it, and a node with many children (a function or statement list) would serialise one
// atomic per child (430k children of a root: 300 us).
__global__ void k_fl_count(const int32_t* parent, const int32_t* child, const uint32_t* data, const uint8_t* type,
                           const uint8_t* rtype, uint32_t n, uint32_t* deg, NodeRec* rec, FlatErr* e) {
    FL_FOR(v, n) {
        const int32_t p = parent[v], c = child[v];
        rec[v] = NodeRec{p, c, data[v], type[v] | static_cast<uint32_t>(rtype[v]) << 8};
        if (p == -1) {
            atomicAdd(&e->roots, 1u);
        } else if (p < 0 || static_cast<uint32_t>(p) >= n || c < 0 || static_cast<uint32_t>(c) >= n) {
            flag(e, v);
        } else if (deg[p] <= static_cast<uint32_t>(c)) {
            atomicMax(&deg[p], static_cast<uint32_t>(c) + 1u);
        }
    }
}

// exclusive scan of deg into off[0..n] (three passes: tile sums, their scan, the tiles)
__device__ uint32_t block_excl(uint32_t x, uint32_t* total) {
    __shared__ uint32_t warp_sum[kScanThreads / 32];
    const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
    uint32_t incl = x;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, d);
        if (lane >= static_cast<uint32_t>(d)) incl += y;
    }
    if (lane == 31) warp_sum[w] = incl;
    __syncthreads();
    if (w == 0) {
        const uint32_t t = lane < kScanThreads / 32 ? warp_sum[lane] : 0u;
        uint32_t s = t;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, s, d);
            if (lane >= static_cast<uint32_t>(d)) s += y;
        }
        if (lane < kScanThreads / 32) warp_sum[lane] = s - t;
        if (lane == 31) *total = s;
    }
    __syncthreads();
    const uint32_t r = warp_sum[w] + incl - x;
    __syncthreads();
    return r;
}

__global__ void __launch_bounds__(kScanThreads) k_fl_tile_sums(const uint32_t* deg, uint32_t n, uint32_t* tsum,
                                                               FlatErr* e) {
    const uint64_t base = static_cast<uint64_t>(blockIdx.x) * kScanTile;
    unsigned long long s = 0;  // the counts of a malformed input may add up past 32 bits
    for (uint32_t k = threadIdx.x; k < kScanTile; k += kScanThreads)
        if (base + k < n) s += deg[base + k];
    __shared__ unsigned long long wide;
    __shared__ uint32_t total;
    if (threadIdx.x == 0) wide = 0;
    block_excl(static_cast<uint32_t>(s), &total);  // its barriers publish wide
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) s += __shfl_down_sync(0xFFFFFFFFu, s, d);
    if ((threadIdx.x & 31u) == 0 && s) atomicAdd(&wide, s);
    __syncthreads();
    if (threadIdx.x == 0) {
        tsum[blockIdx.x] = total;
        if (wide) atomicAdd(&e->slots, wide);
    }
}

__global__ void __launch_bounds__(kScanThreads) k_fl_scan_sums(uint32_t* tsum, uint32_t tiles, uint32_t n, FlatErr* e) {
    __shared__ uint32_t total;
    if (threadIdx.x == 0 && e->slots != n - 1u) flag(e, 0);  // a gap in some node's child indices
    uint32_t carry = 0;
    for (uint32_t b = 0; b < tiles; b += kScanThreads) {
        const uint32_t k = b + threadIdx.x;
        const uint32_t x = k < tiles ? tsum[k] : 0u;
        const uint32_t ex = block_excl(x, &total);
        if (k < tiles) tsum[k] = carry + ex;
        carry += total;
        __syncthreads();
    }
}

__global__ void __launch_bounds__(kScanThreads) k_fl_tiles(const uint32_t* deg, uint32_t n, const uint32_t* tsum,
                                                           uint32_t* off) {
    const uint64_t base = static_cast<uint64_t>(blockIdx.x) * kScanTile;
    constexpr uint32_t kItems = kScanTile / kScanThreads;
    uint32_t v[kItems], s = 0;
#pragma unroll
    for (uint32_t j = 0; j < kItems; ++j) {  // thread t takes elements t*kItems .. +kItems-1
        const uint64_t i = base + threadIdx.x * kItems + j;
        v[j] = i < n ? deg[i] : 0u;
        s += v[j];
    }
    __shared__ uint32_t total;
    uint32_t run = tsum[blockIdx.x] + block_excl(s, &total);
#pragma unroll
    for (uint32_t j = 0; j < kItems; ++j) {
        const uint64_t i = base + threadIdx.x * kItems + j;
        if (i <= n) off[i] = run;  // off[n]: the total
        run += v[j];
    }
}

__device__ __forceinline__ bool bad(const FlatErr* e) { return *reinterpret_cast<const volatile uint32_t*>(&e->code) != 0; }

// each child into its slot (the counts add up to n - 1, so every slot is in range)
__global__ void k_fl_place(const NodeRec* rec, uint32_t n, const uint32_t* deg, const uint32_t* off, uint32_t* kids,
                           FlatErr* e) {
    if (bad(e)) return;
    FL_FOR(v, n) {
        const int2 r = *reinterpret_cast<const int2*>(&rec[v]);  // parent, child
        if (r.x < 0) continue;  // the root
        const uint32_t c = static_cast<uint32_t>(r.y);
        if (c >= deg[r.x] || atomicCAS(&kids[off[r.x] + c], kEmpty, v) != kEmpty) flag(e, v);
    }
}

// The tour (successors of enter(v) and exit(v)), and the splitters in any order: split[k]
// is splitter k's event, sidx of its node is k.  From here on the input is flagged or every slot holds
// one child, so no two events have the same successor but the end.
__global__ void k_fl_tour(const NodeRec* rec, uint32_t n, const uint32_t* deg, const uint32_t* off,
                          const uint32_t* kids, uint32_t lg, uint2* succ, uint32_t* split, uint32_t cap, uint32_t* sidx,
                          FlatErr* e) {
    if (bad(e)) return;
    const uint32_t end = 2u * n;
    FL_FOR(v, n) {
        const int2 r = *reinterpret_cast<const int2*>(&rec[v]);  // parent, child
        uint32_t s = 2u * v + 1u;  // enter(v) -> exit(v) for a leaf
        if (deg[v] > 0) {
            const uint32_t c = kids[off[v]];
            s = c < n ? 2u * c : end;
        }
        uint32_t x = end;  // exit(root) -> the end
        if (r.x >= 0) {
            const uint32_t c = static_cast<uint32_t>(r.y) + 1u;
            if (c < deg[r.x]) {
                const uint32_t sib = kids[off[r.x] + c];
                x = sib < n ? 2u * sib : end;
            } else {
                x = 2u * static_cast<uint32_t>(r.x) + 1u;
            }
        }
        succ[v] = make_uint2(s, x);
        auto add = [&](uint32_t event) {
            const uint32_t k = atomicAdd(&e->splitters, 1u);
            if (k < cap) {
                split[k] = event;
                sidx[v] = k;
            } else {
                flag(e, v);  // several roots
            }
        };
        // The root's enter, which follows nothing, is always one, and its exit may be too:
        // sidx is the latter's.  (One add for both kinds: the counter's atomics are 0.1 ms
        // of 4.3M nodes' as it is.)
        const bool enter = r.x < 0 || is_splitter(2u * v, lg), exit = is_splitter(2u * v + 1u, lg);
        if (enter || exit) add(enter ? 2u * v : 2u * v + 1u);
        if (r.x < 0 && exit) add(2u * v + 1u);
    }
}

// From each splitter to the next: how far, and to which.
__global__ void k_fl_walk(const uint32_t* succ, const uint32_t* split, const uint32_t* sidx,
                          uint32_t n, uint32_t lg, Rank* rank, FlatErr* e) {
    if (bad(e)) return;
    const uint32_t count = e->splitters, end = 2u * n;
    FL_FOR(k, count) {
        uint32_t x = split[k], exits = 0, steps = 0;
        int32_t level = 0;
        uint32_t next = count;
        for (;;) {
            exits += x & 1u;
            level += (x & 1u) ? -1 : 1;
            x = succ[x];
            if (x == end) break;
            if (is_splitter(x, lg)) {
                next = sidx[x >> 1];
                break;
            }
            if (++steps == walk_most(lg)) {
                e->code = kFar;
                break;
            }
        }
        rank[k] = Rank{next, exits, level, 0u};
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) rank[count] = Rank{count, 0u, 0, 0u};
}

// one round of pointer jumping over the splitters
__global__ void k_fl_jump(const Rank* __restrict__ in, Rank* __restrict__ out, const FlatErr* e) {
    if (bad(e)) return;
    FL_FOR(k, static_cast<uint64_t>(e->splitters) + 1u) {
        const uint4 a = reinterpret_cast<const uint4*>(in)[k];
        const uint4 b = reinterpret_cast<const uint4*>(in)[a.x];
        reinterpret_cast<uint4*>(out)[k] = make_uint4(b.x, a.y + b.y, a.z + b.z, 0u);
    }
}

// The walks again (all within walk_most), with what lies behind each splitter known: every
// node's post-order index (post), and by index its node and depth (at).
__global__ void k_fl_number(const uint32_t* succ, const NodeRec* rec, const uint32_t* split, uint32_t n, uint32_t lg,
                            const Rank* rank, int32_t* post, uint2* at, FlatErr* e) {
    if (bad(e)) return;
    const uint32_t count = e->splitters, end = 2u * n;
    uint32_t deepest = 0;
    FL_FOR(k, count) {
        uint32_t x = split[k];
        uint32_t exits = rank[k].exits;  // from x to the end
        int32_t level = rank[k].level;
        if (!(x & 1u) && rec[x >> 1].parent == -1) e->reached = exits;
        for (;;) {
            if (x & 1u) {
                const uint32_t v = x >> 1, q = n - exits;
                const int32_t depth = -(level + 1);
                if (q < n) {
                    post[v] = static_cast<int32_t>(q);
                    at[q] = make_uint2(v, static_cast<uint32_t>(depth));
                }
                if (depth > 0) deepest = max(deepest, static_cast<uint32_t>(depth));
                --exits;
                ++level;
            } else {
                --level;
            }
            x = succ[x];
            if (x == end || is_splitter(x, lg)) break;
        }
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) deepest = max(deepest, __shfl_down_sync(0xFFFFFFFFu, deepest, d));
    if ((threadIdx.x & 31u) == 0 && deepest) atomicMax(&e->max_depth, deepest);
}

// The ranking without splitters, of a tour with a walk longer than walk_most: pointer
// jumping over all events, as many rounds whatever the nodes' numbers.  A call so numbered,
// n = 117k: 0.45 ms (0.1 of it the walk up to its limit), where the longest walk took 37.
__global__ void k_fl_events(const uint32_t* succ, uint32_t n, Event* ev) {
    const uint64_t end = 2ull * n;
    FL_FOR(x, end) ev[x] = Event{succ[x], x & 1u, (x & 1u) ? -1 : 1, 0u};
    if (blockIdx.x == 0 && threadIdx.x == 0) ev[end] = Event{static_cast<uint32_t>(end), 0u, 0, 0u};
}
__global__ void k_fl_event_jump(const Event* __restrict__ in, Event* __restrict__ out, uint64_t events) {
    FL_FOR(x, events) {
        const uint4 a = reinterpret_cast<const uint4*>(in)[x];
        const uint4 b = reinterpret_cast<const uint4*>(in)[a.x];
        reinterpret_cast<uint4*>(out)[x] = make_uint4(b.x, a.y + b.y, a.z + b.z, 0u);
    }
}
__global__ void k_fl_event_number(const Event* ev, const NodeRec* rec, uint32_t n, int32_t* post, uint2* at, FlatErr* e) {
    uint32_t deepest = 0;
    FL_FOR(v, n) {
        const uint32_t q = n - ev[2ull * v + 1u].exits;
        const int32_t depth = -ev[2ull * v].level;
        if (q < n) {  // else a node the root does not reach
            post[v] = static_cast<int32_t>(q);
            at[q] = make_uint2(v, static_cast<uint32_t>(depth));
        }
        if (depth > 0) deepest = max(deepest, static_cast<uint32_t>(depth));
        if (rec[v].parent == -1) e->reached = ev[2ull * v].exits;
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) deepest = max(deepest, __shfl_down_sync(0xFFFFFFFFu, deepest, d));
    if ((threadIdx.x & 31u) == 0 && deepest) atomicMax(&e->max_depth, deepest);
}

// The outputs in post-order: coalesced but for one read of the node's record and one of
// its parent's index.
__global__ void k_fl_emit(const NodeRec* rec, uint32_t n, const int32_t* post, const uint2* at, uint8_t* o_type,
                          uint8_t* o_rtype, int32_t* o_parent, int32_t* o_depth, int32_t* o_child, uint32_t* o_data,
                          int32_t* order, const FlatErr* e) {
    if (bad(e) || e->roots != 1u || e->reached != n) return;
    FL_FOR(q, n) {
        const uint2 a = at[q];
        const uint4 r = reinterpret_cast<const uint4*>(rec)[a.x];
        const int32_t p = static_cast<int32_t>(r.x);
        o_type[q] = static_cast<uint8_t>(r.w);
        o_rtype[q] = static_cast<uint8_t>(r.w >> 8);
        o_parent[q] = p >= 0 ? post[p] : -1;
        o_depth[q] = static_cast<int32_t>(a.y);
        o_child[q] = p >= 0 ? static_cast<int32_t>(r.y) : -1;
        o_data[q] = r.z;
        if (order) order[q] = post[q];  // q as a node here
    }
}

template <class T>
cudaError_t dev_alloc(T** p, size_t count, cudaStream_t s) {
    return cudaMallocAsync(reinterpret_cast<void**>(p), std::max<size_t>(count, 1) * sizeof(T), s);
}

}  // namespace

extern "C" ptl_status ptl_flatten(const ptl_tree_view* in, ptl_depth_tree_out* out, int device, void* stream) {
    if (!in || !out) return PTL_BAD_ARGUMENT;
    const size_t n64 = in->n;
    if (n64 == 0 || n64 >= (1ull << 31)) return PTL_BAD_ARGUMENT;
    if (!in->type || !in->rtype || !in->parent || !in->child_idx || !in->data || !out->type || !out->rtype ||
        !out->parent || !out->depth || !out->child_idx || !out->data)
        return PTL_BAD_ARGUMENT;
    const uint32_t n = static_cast<uint32_t>(n64);
    const ptl::DeviceScope on_device(device);
    if (!on_device.ok()) return PTL_CUDA_ERROR;
    cudaStream_t s = static_cast<cudaStream_t>(stream);

    // device copies of the inputs (or the caller's device arrays) and of the outputs
    const uint8_t *d_type = in->type, *d_rtype = in->rtype;
    const int32_t *d_parent = in->parent, *d_child = in->child_idx;
    const uint32_t* d_data = in->data;
    uint8_t *o_type = out->type, *o_rtype = out->rtype;
    int32_t *o_parent = out->parent, *o_depth = out->depth, *o_child = out->child_idx, *o_order = out->order;
    uint32_t* o_data = out->data;
    uint8_t* in_bytes = nullptr;   // staged inputs (host views): 18 bytes per node
    uint8_t* out_bytes = nullptr;  // staged outputs (host views): 22 bytes per node
    // the scratch, two allocations in all: with one per array 20,274 nodes took 262 us, where
    // they take 256
    uint8_t *kept = nullptr, *rest = nullptr;
    uint32_t *deg = nullptr, *off = nullptr, *kids = nullptr, *tsum = nullptr;
    int32_t* post = nullptr;
    NodeRec* rec = nullptr;
    uint2 *succ = nullptr, *at = nullptr;
    uint32_t *split = nullptr, *sidx = nullptr;
    Rank *rank0 = nullptr, *rank1 = nullptr;
    Event *ev0 = nullptr, *ev1 = nullptr;
    FlatErr* err = nullptr;
    FlatErr herr{};
    const uint32_t tiles = static_cast<uint32_t>((n64 + 1 + kScanTile - 1) / kScanTile);
    const uint32_t lg = splitter_lg(n), cap = splitters_most(n);
    ptl_status st = PTL_OK;
    cudaError_t ce = cudaSuccess;
#define FL_CU(x)                       \
    do {                               \
        ce = (x);                      \
        if (ce != cudaSuccess) goto done; \
    } while (0)
    if (!in->on_device) {
        FL_CU(dev_alloc(&in_bytes, 18 * n64, s));
        uint8_t* b = in_bytes;
        FL_CU(cudaMemcpyAsync(b, in->parent, 4 * n64, cudaMemcpyHostToDevice, s));
        d_parent = reinterpret_cast<const int32_t*>(b);
        FL_CU(cudaMemcpyAsync(b + 4 * n64, in->child_idx, 4 * n64, cudaMemcpyHostToDevice, s));
        d_child = reinterpret_cast<const int32_t*>(b + 4 * n64);
        FL_CU(cudaMemcpyAsync(b + 8 * n64, in->data, 4 * n64, cudaMemcpyHostToDevice, s));
        d_data = reinterpret_cast<const uint32_t*>(b + 8 * n64);
        FL_CU(cudaMemcpyAsync(b + 12 * n64, in->type, n64, cudaMemcpyHostToDevice, s));
        d_type = b + 12 * n64;
        FL_CU(cudaMemcpyAsync(b + 13 * n64, in->rtype, n64, cudaMemcpyHostToDevice, s));
        d_rtype = b + 13 * n64;
    }
    if (!out->on_device) {
        FL_CU(dev_alloc(&out_bytes, 22 * n64, s));
        uint8_t* b = out_bytes;
        o_parent = reinterpret_cast<int32_t*>(b);
        o_depth = reinterpret_cast<int32_t*>(b + 4 * n64);
        o_child = reinterpret_cast<int32_t*>(b + 8 * n64);
        o_data = reinterpret_cast<uint32_t*>(b + 12 * n64);
        o_order = out->order ? reinterpret_cast<int32_t*>(b + 16 * n64) : nullptr;
        o_type = b + 20 * n64;
        o_rtype = b + 21 * n64;
    }
    {  // what the ranking by pointer jumping needs too, and the rest
        auto take = [](size_t& total, size_t bytes) {
            const size_t here = total;
            total = (total + bytes + 255u) & ~size_t(255);
            return here;
        };
        size_t a = 0, b = 0;
        const size_t at_err = take(a, sizeof(FlatErr)), at_deg = take(a, 4 * n64), zeroed = a;
        const size_t at_rec = take(a, sizeof(NodeRec) * n64), at_succ = take(a, 8 * n64), at_at = take(a, 8 * n64),
                     at_post = take(a, 4 * n64);
        const size_t at_kids = take(b, 4 * n64), at_off = take(b, 4 * (n64 + 1)), at_tsum = take(b, 4ull * tiles),
                     at_sidx = take(b, 4 * n64), at_split = take(b, 4ull * cap),
                     at_rank0 = take(b, sizeof(Rank) * (cap + 1ull)), at_rank1 = take(b, sizeof(Rank) * (cap + 1ull));
        FL_CU(dev_alloc(&kept, a, s));
        FL_CU(dev_alloc(&rest, b, s));
        err = reinterpret_cast<FlatErr*>(kept + at_err);
        deg = reinterpret_cast<uint32_t*>(kept + at_deg);
        rec = reinterpret_cast<NodeRec*>(kept + at_rec);
        succ = reinterpret_cast<uint2*>(kept + at_succ);
        at = reinterpret_cast<uint2*>(kept + at_at);
        post = reinterpret_cast<int32_t*>(kept + at_post);
        kids = reinterpret_cast<uint32_t*>(rest + at_kids);
        off = reinterpret_cast<uint32_t*>(rest + at_off);
        tsum = reinterpret_cast<uint32_t*>(rest + at_tsum);
        sidx = reinterpret_cast<uint32_t*>(rest + at_sidx);
        split = reinterpret_cast<uint32_t*>(rest + at_split);
        rank0 = reinterpret_cast<Rank*>(rest + at_rank0);
        rank1 = reinterpret_cast<Rank*>(rest + at_rank1);
        FL_CU(cudaMemsetAsync(kept, 0, zeroed, s));
        FL_CU(cudaMemsetAsync(kids, 0xFF, 4 * n64, s));
    }

    k_fl_count<<<grid_of(n), kThreads, 0, s>>>(d_parent, d_child, d_data, d_type, d_rtype, n, deg, rec, err);
    k_fl_tile_sums<<<tiles, kScanThreads, 0, s>>>(deg, n, tsum, err);
    k_fl_scan_sums<<<1, kScanThreads, 0, s>>>(tsum, tiles, n, err);
    k_fl_tiles<<<tiles, kScanThreads, 0, s>>>(deg, n, tsum, off);
    k_fl_place<<<grid_of(n), kThreads, 0, s>>>(rec, n, deg, off, kids, err);
    k_fl_tour<<<grid_of(n), kThreads, 0, s>>>(rec, n, deg, off, kids, lg, succ, split, cap, sidx, err);
    k_fl_walk<<<walk_grid(cap), kThreads, 0, s>>>(reinterpret_cast<const uint32_t*>(succ), split, sidx, n, lg, rank0,
                                                  err);
    for (uint32_t r = 0; (1ull << r) < cap + 1ull; ++r) {
        k_fl_jump<<<grid_of(cap), kThreads, 0, s>>>(rank0, rank1, err);
        std::swap(rank0, rank1);
    }
    k_fl_number<<<walk_grid(cap), kThreads, 0, s>>>(reinterpret_cast<const uint32_t*>(succ), rec, split, n, lg, rank0,
                                                    post, at, err);
    k_fl_emit<<<grid_of(n), kThreads, 0, s>>>(rec, n, post, at, o_type, o_rtype, o_parent, o_depth, o_child, o_data,
                                              o_order, err);
    FL_CU(cudaGetLastError());
    FL_CU(cudaMemcpyAsync(&herr, err, sizeof(herr), cudaMemcpyDeviceToHost, s));
    FL_CU(cudaStreamSynchronize(s));
    if (herr.code == kFar) {
        const uint64_t events = 2 * n64 + 1;
        cudaFreeAsync(rest, s);  // done with; the events take 64 bytes a node
        rest = nullptr;
        FL_CU(cudaMemsetAsync(&err->code, 0, sizeof(err->code), s));
        FL_CU(dev_alloc(&ev0, events, s));
        FL_CU(dev_alloc(&ev1, events, s));
        k_fl_events<<<grid_of(events), kThreads, 0, s>>>(reinterpret_cast<const uint32_t*>(succ), n, ev0);
        for (uint32_t r = 0; (1ull << r) < events; ++r) {
            k_fl_event_jump<<<grid_of(events), kThreads, 0, s>>>(ev0, ev1, events);
            std::swap(ev0, ev1);
        }
        k_fl_event_number<<<grid_of(n), kThreads, 0, s>>>(ev0, rec, n, post, at, err);
        k_fl_emit<<<grid_of(n), kThreads, 0, s>>>(rec, n, post, at, o_type, o_rtype, o_parent, o_depth, o_child, o_data,
                                                  o_order, err);
        FL_CU(cudaGetLastError());
        FL_CU(cudaMemcpyAsync(&herr, err, sizeof(herr), cudaMemcpyDeviceToHost, s));
    }
    if (!out->on_device) {
        FL_CU(cudaMemcpyAsync(out->parent, o_parent, 4 * n64, cudaMemcpyDeviceToHost, s));
        FL_CU(cudaMemcpyAsync(out->depth, o_depth, 4 * n64, cudaMemcpyDeviceToHost, s));
        FL_CU(cudaMemcpyAsync(out->child_idx, o_child, 4 * n64, cudaMemcpyDeviceToHost, s));
        FL_CU(cudaMemcpyAsync(out->data, o_data, 4 * n64, cudaMemcpyDeviceToHost, s));
        if (out->order) FL_CU(cudaMemcpyAsync(out->order, o_order, 4 * n64, cudaMemcpyDeviceToHost, s));
        FL_CU(cudaMemcpyAsync(out->type, o_type, n64, cudaMemcpyDeviceToHost, s));
        FL_CU(cudaMemcpyAsync(out->rtype, o_rtype, n64, cudaMemcpyDeviceToHost, s));
    }
    FL_CU(cudaStreamSynchronize(s));
    if (herr.code != 0 || herr.roots != 1 || herr.reached != n) st = PTL_INVALID_AST;
    out->max_depth = herr.max_depth;
done:
#undef FL_CU
    for (void* p : {static_cast<void*>(in_bytes), static_cast<void*>(out_bytes), static_cast<void*>(kept),
                    static_cast<void*>(rest), static_cast<void*>(ev0), static_cast<void*>(ev1)})
        if (p) cudaFreeAsync(p, s);
    if (ce != cudaSuccess) {
        cudaStreamSynchronize(s);
        return ce == cudaErrorMemoryAllocation ? PTL_OOM : PTL_CUDA_ERROR;
    }
    return st;
}
