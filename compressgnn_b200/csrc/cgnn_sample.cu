// Neighbour sampling on the compressed graph (device side of one hop).
//
// ref: neighbor_sample_sim_impl, src/sample/csrc/neighbor_sample.h:27-131, with get_neighbor and
// get_neighbor_list of src/sample/csrc/storage_api.h:7-118 (host code there; bound as
// compressgnn_sample.neighbor_sample_cg_sim).  A node's neighbours are its v2v entries followed by the
// expansion of its v2r rules; `vertex_degree` / `rule_degree` (gen_degree) give the sizes, so the i-th
// neighbour is found by skipping whole rules.  Per hop the reference does, node by node in frontier
// order: degree <= fan-out -> all neighbours in list order (v2v, then the rules breadth first, then every
// listed rule's own vertices); otherwise Floyd's scheme draws `fan-out` distinct neighbour indices
// (for j = degree - k .. degree - 1: a uniform index below j, replaced by j if already drawn).  New nodes
// get local ids in the order they are first seen.
//
// Here a hop is four steps on the device: every frontier node picks its neighbours (one thread per node:
// the picks of a node are sequential by definition and few), then first-seen relabelling without a hash
// map: atomicMin of the pick position into a per-vertex table, a flag for the winning positions, a scan,
// and a scatter.  Random indices come from Philox4x32 counted by (hop, frontier position, draw) under the
// caller's seed instead of the host generator the reference asks, so a hop does not depend on thread
// order and the CPU restatement can draw the same numbers.
//
// The children of a rule are read from ONE rule -> rule CSR (the union of the reference's level blocks,
// each rule's children live in exactly one of them).  storage_api.h looks a rule's children up in the
// level numbered by the descent depth, which finds them only for rules without nested rules; on such
// graphs both orders below are the reference's, on deeper ones they are what its comments describe.
#include <algorithm>
#include <vector>

#include "cgnn_common.cuh"

namespace cgnn {
namespace {

constexpr int THREADS = 128;
constexpr int32_t NO_LOCAL_ID = INT32_MAX;  // value of local_of[] and first[] for a vertex not seen yet
static inline unsigned blocks_for(int64_t count) {
    return (unsigned)std::max<int64_t>(1, std::min<int64_t>(ceil_div(count, THREADS), 148 * 32));
}
#define GRID_STRIDE(i, count) \
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < (count); i += (int64_t)blockDim.x * gridDim.x)

static __device__ int g_sample_status = 0;

// Philox4x32 with 7 rounds (Salmon et al., SC 2011): counter (c0, c1, c2, c3), key (k0, k1).
__device__ __forceinline__ uint32_t philox_first_word(uint32_t c0, uint32_t c1, uint32_t c2, uint32_t c3, uint64_t seed) {
    uint32_t k0 = (uint32_t)seed, k1 = (uint32_t)(seed >> 32);
#pragma unroll
    for (int round = 0; round < 7; ++round) {
        const uint32_t hi0 = __umulhi(0xD2511F53u, c0), lo0 = 0xD2511F53u * c0;
        const uint32_t hi1 = __umulhi(0xCD9E8D57u, c2), lo1 = 0xCD9E8D57u * c2;
        c0 = hi1 ^ c1 ^ k0;
        c1 = lo1;
        c2 = hi0 ^ c3 ^ k1;
        c3 = lo0;
        k0 += 0x9E3779B9u;
        k1 += 0xBB67AE85u;
    }
    return c0;
}

struct GraphView {
    const int64_t *v2v_ptr, *v2v_col, *v2r_ptr, *v2r_col, *r2v_ptr, *r2v_col, *r2r_ptr, *r2r_col;
    const int64_t *v_degree, *r_degree;
    int64_t n, r;
};

// The `index`-th neighbour of `node` (index < vertex_degree[node]); -1 if the degree tables do not match.
__device__ int64_t neighbor_at(const GraphView &g, int64_t node, int64_t index) {
    const int64_t vb = g.v2v_ptr[node], vcount = g.v2v_ptr[node + 1] - vb;
    if (index < vcount) return g.v2v_col[vb + index];
    index -= vcount;
    for (int64_t e = g.v2r_ptr[node]; e < g.v2r_ptr[node + 1]; ++e) {
        int64_t rule = g.v2r_col[e];
        const int64_t size = g.r_degree[rule];
        if (index >= size) {
            index -= size;
            continue;
        }
        for (int depth = 0; depth < 64; ++depth) {  // a rule graph is far shallower; the bound keeps the walk finite
            const int64_t rb = g.r2v_ptr[rule], own = g.r2v_ptr[rule + 1] - rb;
            if (index < own) return g.r2v_col[rb + index];
            index -= own;
            int64_t next = -1;
            for (int64_t c = g.r2r_ptr[rule]; c < g.r2r_ptr[rule + 1]; ++c) {
                const int64_t child = g.r2r_col[c], below = g.r_degree[child];
                if (index < below) {
                    next = child;
                    break;
                }
                index -= below;
            }
            if (next < 0) return -1;
            rule = next;
        }
        return -1;
    }
    return -1;
}

__global__ void count_kernel(const GraphView g, const int64_t *samples, int64_t begin, int64_t frontier, int64_t fanout,
                             int64_t *count) {
    GRID_STRIDE(i, frontier) {
        const int64_t node = samples[begin + i];
        int64_t k = 0;
        if (node >= 0 && node < g.n) {
            const int64_t degree = g.v_degree[node];
            k = degree <= 0 ? 0 : (fanout >= degree ? degree : (fanout > 0 ? fanout : 0));
        } else {
            atomicOr(&g_sample_status, STATUS_BAD_INDEX);
        }
        count[i] = k;
    }
}

// offset = exclusive scan of count.  picked[offset[i] .. +count[i]) receives the neighbours of frontier node i,
// source[...] its local id; `queue` (same layout) is scratch for the breadth-first rule list of a take-all node.
__global__ void pick_kernel(const GraphView g, const int64_t *samples, int64_t begin, int64_t frontier, int64_t fanout,
                            const int64_t *count, const int64_t *offset, uint32_t hop, uint64_t seed, int64_t *picked,
                            int64_t *source, int64_t *queue) {
    GRID_STRIDE(i, frontier) {
        const int64_t k = count[i];
        if (k == 0) continue;
        const int64_t node = samples[begin + i], at = offset[i], degree = g.v_degree[node];
        for (int64_t j = 0; j < k; ++j) source[at + j] = begin + i;
        if (k == degree) {  // everything, in list order
            int64_t out = 0;
            for (int64_t e = g.v2v_ptr[node]; e < g.v2v_ptr[node + 1] && out < k; ++e) picked[at + out++] = g.v2v_col[e];
            int64_t rules = 0;  // breadth-first list of the rules below the node (each holds >= 1 vertex: rules <= k)
            for (int64_t e = g.v2r_ptr[node]; e < g.v2r_ptr[node + 1] && rules < k; ++e) queue[at + rules++] = g.v2r_col[e];
            for (int64_t head = 0; head < rules; ++head) {
                const int64_t rule = queue[at + head];
                for (int64_t c = g.r2r_ptr[rule]; c < g.r2r_ptr[rule + 1] && rules < k; ++c) queue[at + rules++] = g.r2r_col[c];
            }
            for (int64_t head = 0; head < rules; ++head) {
                const int64_t rule = queue[at + head];
                for (int64_t e = g.r2v_ptr[rule]; e < g.r2v_ptr[rule + 1] && out < k; ++e) picked[at + out++] = g.r2v_col[e];
            }
            if (out != k) {
                atomicOr(&g_sample_status, STATUS_BAD_CSR);  // the degree table does not match the graph
                for (; out < k; ++out) picked[at + out] = node;
            }
        } else {  // Floyd: k distinct indices below degree; queue[] keeps the indices drawn so far
            for (int64_t t = 0; t < k; ++t) {
                const int64_t j = degree - k + t;  // >= 1
                const uint32_t word = philox_first_word((uint32_t)(begin + i), (uint32_t)((begin + i) >> 32), (uint32_t)t, hop, seed);
                int64_t index = (int64_t)(((uint64_t)word * (uint64_t)j) >> 32);  // uniform below j
                for (int64_t s = 0; s < t; ++s)
                    if (queue[at + s] == index) {
                        index = j;
                        break;
                    }
                queue[at + t] = index;
                int64_t v = neighbor_at(g, node, index);
                if (v < 0) {
                    atomicOr(&g_sample_status, STATUS_BAD_CSR);
                    v = node;
                }
                picked[at + t] = v;
            }
        }
    }
}

// first[v] = smallest pick position of a vertex that has no local id yet
__global__ void claim_kernel(const int64_t *picked, int64_t total, int64_t n, const int32_t *local_of, int32_t *first) {
    GRID_STRIDE(p, total) {
        const int64_t v = picked[p];
        if (v < 0 || v >= n) {
            atomicOr(&g_sample_status, STATUS_BAD_INDEX);
            continue;
        }
        if (local_of[v] == NO_LOCAL_ID) atomicMin(&first[v], (int32_t)p);
    }
}

__global__ void flag_kernel(const int64_t *picked, int64_t total, int64_t n, const int32_t *local_of, const int32_t *first,
                            int64_t *is_new) {
    GRID_STRIDE(p, total) {
        const int64_t v = picked[p];
        is_new[p] = (v >= 0 && v < n && local_of[v] == NO_LOCAL_ID && first[v] == (int32_t)p) ? 1 : 0;
    }
}

// rank = exclusive scan of is_new.  Local id of a new vertex = end + rank of its first pick.
__global__ void relabel_kernel(const int64_t *picked, int64_t total, int64_t n, const int32_t *local_of, const int32_t *first,
                               const int64_t *is_new, const int64_t *rank, int64_t end, int64_t *target,
                               int64_t *samples) {
    GRID_STRIDE(p, total) {
        const int64_t v = picked[p];
        int64_t local = 0;
        if (v >= 0 && v < n) local = local_of[v] != NO_LOCAL_ID ? local_of[v] : end + rank[first[v]];
        target[p] = local;
        if (is_new[p]) samples[end + rank[p]] = v;
    }
}

__global__ void commit_kernel(const int64_t *picked, int64_t total, const int64_t *is_new, const int64_t *rank, int64_t end,
                              int32_t *local_of, int32_t *first) {
    GRID_STRIDE(p, total) {
        if (is_new[p]) {
            const int64_t v = picked[p];
            local_of[v] = (int32_t)(end + rank[p]);
            first[v] = NO_LOCAL_ID;
        }
    }
}

__global__ void seed_kernel(const int64_t *samples, int64_t count, int64_t n, int32_t *local_of) {
    GRID_STRIDE(i, count) {
        const int64_t v = samples[i];
        if (v >= 0 && v < n) atomicMin(&local_of[v], (int32_t)i);  // a repeated seed keeps its first position
        else atomicOr(&g_sample_status, STATUS_BAD_INDEX);
    }
}

// ---------------------------------------------------------------------------------------
// All hops of a batch without a host round trip (cgnn_sample_hops).
//
// What bounds a batch is latency: 60 k edges are a few microseconds of traffic, but hop by hop the host learns two
// sizes per hop (edges, new vertices) before it can allocate and go on, a pick is one thread's
// chain of dependent index reads, and ~15 small launches stand between them.  Here frontier node i of a hop owns `stride` = min(fan-out, largest degree) pick slots, so the buffers are
// sized by a bound the host knows beforehand and the true sizes stay on the device:
//   * a slot's position counts over the whole batch (seeds first, then hop after hop), and first[v] keeps
//     the smallest position that named vertex v -- earlier hops have smaller positions, so one
//     table serves seeds and all hops and nothing is committed in between;
//   * edges and new vertices are numbered in two small launches: blocks of TILE slots number their own and leave their
//     totals (hops_count_kernel), and the launch that writes the edges adds up the totals before each block, in
//     shared memory, every block for itself (hops_relabel_kernel); the number at first[v] IS the local id of v;
//   * a warp picks for one node: the children of up to 32 rules are listed per step, and the lookups of Floyd's
//     draws run side by side.
//   * a launch is scheduled while the one before it ends (hops_launch).
// A batch of 1024 seeds with fan-outs 25 and 10 on the 325 k-node graph: 119 us; 131 with a library scan over the slots
// in place of the numbering (three launches a hop where two do now, and none of them overlapping), hop by hop 505.  Going
// hop by hop stays for batches whose slots would exceed MAX_POSITIONS.
// ---------------------------------------------------------------------------------------
constexpr int32_t EMPTY_SLOT = -1;  // picked[]: no pick here
constexpr int32_t BAD_VERTEX = -2;  // picked[]: an edge to a vertex outside the graph (reported; local id 0)
constexpr int64_t MAX_POSITIONS = 8 << 20;  // see cgnn_sample_hops_bytes

// The launches of a batch follow one another at once: each opens the next one's scheduling when it starts and touches
// memory only after the one before it is complete (hops_follow).
__device__ __forceinline__ void hops_open() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void hops_follow() {
    hops_open();
    asm volatile("griddepcontrol.wait;" ::: "memory");
}
template <typename... Params, typename... Args>
static cudaError_t hops_launch(void (*kernel)(Params...), unsigned grid, cudaStream_t stream, Args... args) {
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3(grid);
    config.blockDim = dim3(THREADS);
    config.stream = stream;
    cudaLaunchAttribute follows = {};
    follows.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    follows.val.programmaticStreamSerializationAllowed = 1;
    config.attrs = &follows;
    config.numAttrs = 1;
    return cudaLaunchKernelEx(&config, kernel, static_cast<Params>(args)...);
}

// counts[h], h = 0 .. hops + 1: (edges << 32 | samples) before hop h - 1 has run; counts[0] = 0, counts[1] = the seeds
__global__ void hops_begin_kernel(const int64_t *seeds, int64_t batch, int64_t n, int64_t *samples, int32_t *first,
                                  int32_t *ids, uint64_t *counts) {
    hops_open();
    GRID_STRIDE(i, batch) {
        const int64_t v = seeds[i];
        samples[i] = v;
        ids[i] = (int32_t)i;
        if (v >= 0 && v < n) atomicMin(&first[v], (int32_t)i);  // a repeated seed keeps its first position
        else atomicOr(&g_sample_status, STATUS_BAD_INDEX);
        if (i == 0) {
            counts[0] = 0;
            counts[1] = (uint64_t)batch;
        }
    }
}

__device__ __forceinline__ int32_t warp_exclusive(int32_t x, int lane, int32_t *sum) {
    int32_t s = x;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int32_t t = __shfl_up_sync(0xffffffffu, s, d);
        if (lane >= d) s += t;
    }
    *sum = __shfl_sync(0xffffffffu, s, 31);
    return s - x;
}

// Hands the children of the listed rules queue[0 .. rules) under (ptr, col), in list order, to store(position,
// child) with positions from `used` up, below `most`; returns the position reached.  APPEND: the children join
// the list itself while it is walked (`used` is its length).
template <bool APPEND, typename Store>
__device__ __forceinline__ int32_t list_children(const int64_t *ptr, const int64_t *col, const int32_t *queue,
                                                 int32_t rules, int32_t used, int32_t most, int lane, Store store) {
    for (int32_t head = 0; head < (APPEND ? used : rules); ) {
        const int32_t chunk = min(32, (APPEND ? used : rules) - head);
        int64_t b = 0;
        int32_t cnt = 0, sum = 0;
        if (lane < chunk) {
            const int32_t rule = queue[head + lane];
            b = ptr[rule];
            cnt = (int32_t)max(min(ptr[rule + 1] - b, (int64_t)most), (int64_t)0);
        }
        const int32_t at = used + warp_exclusive(cnt, lane, &sum);
        for (int32_t c = 0; c < cnt && at + c < most; ++c) store(at + c, col[b + c]);
        used = min(most, used + sum);
        head += chunk;
        __syncwarp();
        if (!APPEND && used == most) break;
    }
    return used;
}

// One warp per frontier node (grid-stride over the bound `nodes`; nodes past the real frontier leave empty
// slots).  `queue` has the layout of `picked`.
__global__ void __launch_bounds__(THREADS) hops_pick_kernel(const GraphView g, const int64_t *samples, const uint64_t *counts,
                                                            int64_t nodes, int32_t stride, int64_t fanout, uint32_t hop,
                                                            uint64_t seed, int32_t base, int32_t *picked, int32_t *queue,
                                                            int32_t *first) {
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * (THREADS / 32);
    hops_follow();
    const int64_t begin = (uint32_t)counts[0], end = (uint32_t)counts[1];
    for (int64_t i = (int64_t)blockIdx.x * (THREADS / 32) + (threadIdx.x >> 5); i < nodes; i += warps) {
        int32_t *slots = picked + i * stride, *list = queue + i * stride;
        const int32_t base_i = base + (int32_t)(i * stride);
        int64_t node = -1, degree = 0;
        if (begin + i < end) {
            node = samples[begin + i];
            if (node >= 0 && node < g.n) degree = g.v_degree[node];
            else if (lane == 0) atomicOr(&g_sample_status, STATUS_BAD_INDEX);
        }
        const int32_t k = degree <= 0 ? 0 : (int32_t)min(degree, (int64_t)stride);
        auto pick = [&](int32_t t, int64_t v) {
            if (v < 0 || v >= g.n) {
                atomicOr(&g_sample_status, STATUS_BAD_INDEX);
                slots[t] = BAD_VERTEX;
                return;
            }
            slots[t] = (int32_t)v;
            if (first[v] > base_i + t) atomicMin(&first[v], base_i + t);
        };
        if (k > 0 && fanout >= degree) {  // everything, in list order
            const int64_t vb = g.v2v_ptr[node], rb = g.v2r_ptr[node];
            int32_t out = (int32_t)max(min(g.v2v_ptr[node + 1] - vb, (int64_t)k), (int64_t)0);
            int32_t rules = (int32_t)max(min(g.v2r_ptr[node + 1] - rb, (int64_t)k), (int64_t)0);
            for (int32_t t = lane; t < out; t += 32) pick(t, g.v2v_col[vb + t]);
            if (out < k) {
                // breadth-first list of the rules below the node (each holds >= 1 vertex: rules <= k)
                for (int32_t t = lane; t < rules; t += 32) list[t] = (int32_t)g.v2r_col[rb + t];
                __syncwarp();
                rules = list_children<true>(g.r2r_ptr, g.r2r_col, list, 0, rules, k, lane,
                                            [&](int32_t t, int64_t rule) { list[t] = (int32_t)rule; });
                out = list_children<false>(g.r2v_ptr, g.r2v_col, list, rules, out, k, lane, pick);
            }
            if (out < k) {
                if (lane == 0) atomicOr(&g_sample_status, STATUS_BAD_CSR);  // the degree table does not match the graph
                for (int32_t t = out + lane; t < k; t += 32) pick(t, node);
            }
        } else if (k > 0) {  // Floyd: k distinct indices below degree; list[] keeps the indices of earlier chunks
            const int64_t frontier_id = begin + i;
            for (int32_t t0 = 0; t0 < k; t0 += 32) {
                const int32_t t = t0 + lane, j = (int32_t)(degree - k + t);  // j >= 1
                int32_t index = -1 - lane;                                   // idle lanes: equal to nothing
                if (t < k) {
                    const uint32_t word =
                        philox_first_word((uint32_t)frontier_id, (uint32_t)(frontier_id >> 32), (uint32_t)t, hop, seed);
                    index = (int32_t)(((uint64_t)word * (uint64_t)j) >> 32);  // uniform below j
                }
                bool taken = false;
                for (int32_t s = 0; s < t0; ++s) taken |= list[s] == index;
                if (taken) index = j;
                const int32_t drawn = index;
                const int32_t chunk = min(32, k - t0);
                for (int32_t u = 0; u < chunk; ++u) {  // lane u is final when its turn comes
                    const int32_t other = __shfl_sync(0xffffffffu, index, u);
                    if (!taken && lane > u && t < k && other == drawn) {
                        taken = true;
                        index = j;
                    }
                }
                if (t < k) {
                    list[t] = index;
                    int64_t v = neighbor_at(g, node, index);
                    if (v < 0) {
                        atomicOr(&g_sample_status, STATUS_BAD_CSR);
                        v = node;
                    }
                    pick(t, v);
                }
                __syncwarp();
            }
        }
        for (int32_t t = k + lane; t < stride; t += 32) slots[t] = EMPTY_SLOT;
        __syncwarp();
    }
}

// The slots of a hop: an edge in each that is not empty, a new vertex in the first that names it.
struct HopSlots {
    const int32_t *picked, *first;
    int64_t slots;
    int32_t base;  // position of slot 0
    __device__ bool is_new(int64_t p, int32_t v) const { return v >= 0 && first[v] == base + (int32_t)p; }
};

constexpr int TILE_ROUNDS = 16;
constexpr int TILE = THREADS * TILE_ROUNDS;  // slots a block numbers: 2048, so that two counts fit a word
constexpr int MAX_TILES = (int)(MAX_POSITIONS / TILE);
static_assert(MAX_TILES % THREADS == 0 && TILE < 1 << 15, "tiles are shared out evenly; counts are 16 bits each");

// local[p] = edges before slot p in its tile (low half), new vertices before it (high half); totals[] of the tiles alike.
__global__ void __launch_bounds__(THREADS) hops_count_kernel(const HopSlots hop, uint32_t *local, uint32_t *totals) {
    constexpr int WARPS = THREADS / 32, CELLS = TILE_ROUNDS * WARPS;
    static_assert(CELLS == 64, "a warp scans two cells a lane");
    __shared__ uint32_t cells[CELLS];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t tile0 = (int64_t)blockIdx.x * TILE;
    hops_follow();
    int32_t v[TILE_ROUNDS];
#pragma unroll
    for (int r = 0; r < TILE_ROUNDS; ++r) {
        const int64_t p = tile0 + r * THREADS + threadIdx.x;
        v[r] = p < hop.slots ? hop.picked[p] : EMPTY_SLOT;
    }
    uint32_t edges[TILE_ROUNDS], fresh[TILE_ROUNDS];
#pragma unroll
    for (int r = 0; r < TILE_ROUNDS; ++r) {
        const int64_t p = tile0 + r * THREADS + threadIdx.x;
        edges[r] = __ballot_sync(0xffffffffu, v[r] != EMPTY_SLOT);
        fresh[r] = __ballot_sync(0xffffffffu, hop.is_new(p, v[r]));
        if (lane == 0) cells[r * WARPS + warp] = (uint32_t)__popc(edges[r]) | (uint32_t)__popc(fresh[r]) << 16;
    }
    __syncthreads();
    if (warp == 0) {
        const uint32_t low = cells[2 * lane], high = cells[2 * lane + 1];
        int32_t sum;
        const uint32_t before = (uint32_t)warp_exclusive((int32_t)(low + high), lane, &sum);
        cells[2 * lane] = before;
        cells[2 * lane + 1] = before + low;
        if (lane == 0) totals[blockIdx.x] = (uint32_t)sum;
    }
    __syncthreads();
    const uint32_t below = (1u << lane) - 1;
#pragma unroll
    for (int r = 0; r < TILE_ROUNDS; ++r) {
        const int64_t p = tile0 + r * THREADS + threadIdx.x;
        if (p < hop.slots)
            local[p] = cells[r * WARPS + warp] + ((uint32_t)__popc(edges[r] & below) | (uint32_t)__popc(fresh[r] & below) << 16);
    }
}

// Writes the hop's edges, its new vertices and their ids, and the totals after it.
__global__ void __launch_bounds__(THREADS) hops_relabel_kernel(const HopSlots hop, int32_t stride, const uint32_t *local,
                                                               const uint32_t *totals, int32_t tiles, uint64_t *counts,
                                                               int32_t *ids, int32_t *rows, int32_t *cols,
                                                               int64_t *samples) {
    __shared__ uint64_t bases[MAX_TILES];  // (edges << 32 | samples) before each tile
    __shared__ uint64_t warp_sums[THREADS / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    hops_follow();
    auto widened = [](uint32_t c) { return (uint64_t)(c & 0xffffu) << 32 | (c >> 16); };
    const int32_t begin = (int32_t)(uint32_t)counts[0];
    const int per_thread = (tiles + THREADS - 1) / THREADS;
    const int t0 = threadIdx.x * per_thread;
    uint64_t sum = 0;
    for (int t = t0; t < min(t0 + per_thread, tiles); ++t) sum += widened(totals[t]);
    uint64_t upto = sum;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint64_t x = __shfl_up_sync(0xffffffffu, upto, d);
        if (lane >= d) upto += x;
    }
    if (lane == 31) warp_sums[warp] = upto;
    __syncthreads();
    uint64_t before = counts[1] + upto - sum;
    for (int w = 0; w < warp; ++w) before += warp_sums[w];
    for (int t = t0; t < min(t0 + per_thread, tiles); ++t) {
        bases[t] = before;
        before += widened(totals[t]);
    }
    if (blockIdx.x == 0 && t0 < tiles && t0 + per_thread >= tiles) counts[2] = before;  // the thread of the last tile
    __syncthreads();
    GRID_STRIDE(p, hop.slots) {
        const int32_t v = hop.picked[p];
        const uint64_t here = bases[p / TILE] + widened(local[p]);
        ids[hop.base + p] = (int32_t)(uint32_t)here;  // what later hops find at first[v]
        if (v != EMPTY_SLOT) {
            const uint32_t edge = (uint32_t)(here >> 32);
            rows[edge] = begin + (int32_t)((uint32_t)p / (uint32_t)stride);
            int32_t id = 0;
            if (v >= 0) {
                const int32_t q = hop.first[v] - hop.base;
                id = q < 0 ? ids[hop.base + q] : (int32_t)((uint32_t)bases[q / TILE] + (local[q] >> 16));
                if (q == (int32_t)p) samples[(uint32_t)here] = v;
            }
            cols[edge] = id;
        }
    }
}

// The results in their own arrays, and the table back to "nothing seen" for the next batch.
__global__ void hops_finish_kernel(const int64_t *samples, const int32_t *rows, const int32_t *cols, int64_t nodes,
                                   int64_t edges, int64_t n, int32_t *first, int64_t *samples_out, int64_t *rows_out,
                                   int64_t *cols_out) {
    GRID_STRIDE(i, nodes) {
        const int64_t v = samples[i];
        samples_out[i] = v;
        if (v >= 0 && v < n) first[v] = NO_LOCAL_ID;
    }
    GRID_STRIDE(e, edges) {
        rows_out[e] = rows[e];
        cols_out[e] = cols[e];
    }
}

// Slots of every hop and the layout of the workspace.
struct HopsLayout {
    std::vector<int64_t> nodes, stride;  // per hop: bound of the frontier, slots per node
    int64_t slots = 0, room = 0;         // all slots; bound of the samples
    size_t counts = 0, samples = 0, ids = 0, picked = 0, rows = 0, cols = 0, local = 0, totals = 0, total = 0;
    bool fits = false;
};

static HopsLayout hops_layout(const cgnn_sample_graph *g, int64_t batch, int hops, const int64_t *fanouts,
                              int64_t largest_degree) {
    HopsLayout L;
    if (batch > MAX_POSITIONS || g->vertices >= INT32_MAX || g->rules >= INT32_MAX || largest_degree >= INT32_MAX) return L;
    int64_t frontier = batch, most = 0;
    L.room = batch;
    for (int h = 0; h < hops; ++h) {
        const int64_t stride = std::min(fanouts[h], largest_degree);
        if (stride <= 0 || frontier == 0) break;  // nothing from here on
        if (stride > MAX_POSITIONS || frontier * stride + L.slots + batch > MAX_POSITIONS) return L;
        L.nodes.push_back(frontier);
        L.stride.push_back(stride);
        const int64_t slots = frontier * stride;
        most = std::max(most, slots);
        L.slots += slots;
        frontier = std::min(slots, g->vertices);
    }
    L.room = batch + std::min(L.slots, g->vertices);
    size_t used = 0;
    auto span = [&](size_t bytes) {
        const size_t at = used;
        used += align_up(std::max<size_t>(bytes, 16), 256);
        return at;
    };
    L.counts = span(((size_t)hops + 2) * 8);
    L.samples = span((size_t)L.room * 8);
    L.ids = span((size_t)(batch + L.slots) * 4);
    L.picked = span((size_t)L.slots * 4);
    L.rows = span((size_t)L.slots * 4);
    L.cols = span((size_t)L.slots * 4);
    L.local = span((size_t)most * 4);
    L.totals = span((size_t)ceil_div(most, TILE) * 4);
    L.total = used;
    L.fits = true;
    return L;
}

static GraphView view_of(const cgnn_sample_graph *g) {
    GraphView v;
    v.v2v_ptr = g->v2v_ptr, v.v2v_col = g->v2v_col, v.v2r_ptr = g->v2r_ptr, v.v2r_col = g->v2r_col;
    v.r2v_ptr = g->r2v_ptr, v.r2v_col = g->r2v_col, v.r2r_ptr = g->r2r_ptr, v.r2r_col = g->r2r_col;
    v.v_degree = g->vertex_degree, v.r_degree = g->rule_degree, v.n = g->vertices, v.r = g->rules;
    return v;
}

}  // namespace

int sample_status(int *out) {
    int zero = 0;
    CGNN_CUDA(cudaMemcpyFromSymbol(out, g_sample_status, sizeof(int)));
    CGNN_CUDA(cudaMemcpyToSymbol(g_sample_status, &zero, sizeof(int)));
    return CGNN_OK;
}

}  // namespace cgnn

using namespace cgnn;

extern "C" {

int cgnn_sample_seed(const int64_t *samples, int64_t count, int64_t vertices, int32_t *local_of, cgnn_stream_t stream) {
    CGNN_REQUIRE(count >= 0 && (count == 0 || (samples != nullptr && local_of != nullptr)), "sample_seed: null argument");
    if (count == 0) return CGNN_OK;
    seed_kernel<<<blocks_for(count), THREADS, 0, (cudaStream_t)stream>>>(samples, count, vertices, local_of);
    CGNN_LAUNCH_CHECK();
    return CGNN_OK;
}

int cgnn_sample_count(const cgnn_sample_graph *graph, const int64_t *samples, int64_t begin, int64_t frontier,
                      int64_t fanout, int64_t *count, cgnn_stream_t stream) {
    CGNN_REQUIRE(graph != nullptr && frontier >= 0 && (frontier == 0 || (samples != nullptr && count != nullptr)),
                 "sample_count: null argument");
    if (frontier == 0) return CGNN_OK;
    count_kernel<<<blocks_for(frontier), THREADS, 0, (cudaStream_t)stream>>>(view_of(graph), samples, begin, frontier, fanout,
                                                                            count);
    CGNN_LAUNCH_CHECK();
    return CGNN_OK;
}

int cgnn_sample_pick(const cgnn_sample_graph *graph, const int64_t *samples, int64_t begin, int64_t frontier, int64_t fanout,
                     const int64_t *count, const int64_t *offset, uint32_t hop, uint64_t seed, int64_t *picked,
                     int64_t *source, int64_t *scratch, cgnn_stream_t stream) {
    CGNN_REQUIRE(graph != nullptr && frontier >= 0, "sample_pick: null graph");
    if (frontier == 0) return CGNN_OK;
    CGNN_REQUIRE(samples && count && offset && picked && source && scratch, "sample_pick: null argument");
    pick_kernel<<<blocks_for(frontier), THREADS, 0, (cudaStream_t)stream>>>(view_of(graph), samples, begin, frontier, fanout,
                                                                           count, offset, hop, seed, picked, source, scratch);
    CGNN_LAUNCH_CHECK();
    return CGNN_OK;
}

int cgnn_sample_claim(const int64_t *picked, int64_t total, int64_t vertices, const int32_t *local_of, int32_t *first,
                      int64_t *is_new, cgnn_stream_t stream_) {
    cudaStream_t stream = (cudaStream_t)stream_;
    CGNN_REQUIRE(total >= 0 && total < INT32_MAX, "sample_claim: too many picks for one hop");
    if (total == 0) return CGNN_OK;
    CGNN_REQUIRE(picked && local_of && first && is_new, "sample_claim: null argument");
    claim_kernel<<<blocks_for(total), THREADS, 0, stream>>>(picked, total, vertices, local_of, first);
    CGNN_LAUNCH_CHECK();
    flag_kernel<<<blocks_for(total), THREADS, 0, stream>>>(picked, total, vertices, local_of, first, is_new);
    CGNN_LAUNCH_CHECK();
    return CGNN_OK;
}

int cgnn_sample_relabel(const int64_t *picked, int64_t total, int64_t vertices, const int64_t *is_new, const int64_t *rank,
                        int64_t end, int32_t *local_of, int32_t *first, int64_t *target, int64_t *samples,
                        cgnn_stream_t stream_) {
    cudaStream_t stream = (cudaStream_t)stream_;
    if (total == 0) return CGNN_OK;
    CGNN_REQUIRE(picked && is_new && rank && local_of && first && target && samples, "sample_relabel: null argument");
    relabel_kernel<<<blocks_for(total), THREADS, 0, stream>>>(picked, total, vertices, local_of, first, is_new, rank, end,
                                                             target, samples);
    CGNN_LAUNCH_CHECK();
    commit_kernel<<<blocks_for(total), THREADS, 0, stream>>>(picked, total, is_new, rank, end, local_of, first);
    CGNN_LAUNCH_CHECK();
    return CGNN_OK;
}

size_t cgnn_sample_hops_bytes(const cgnn_sample_graph *graph, int64_t batch, int hops, const int64_t *fanouts,
                              int64_t largest_degree) {
    if (graph == nullptr || batch <= 0 || hops < 0 || (hops > 0 && fanouts == nullptr)) return 0;
    const HopsLayout L = hops_layout(graph, batch, hops, fanouts, largest_degree);
    return L.fits ? L.total : 0;
}

int cgnn_sample_hops(const cgnn_sample_graph *graph, const int64_t *seeds, int64_t batch, int hops, const int64_t *fanouts,
                     int64_t largest_degree, uint64_t seed, int32_t *first, void *workspace, size_t workspace_bytes,
                     int64_t sizes[2], cgnn_stream_t stream_) {
    cudaStream_t stream = (cudaStream_t)stream_;
    CGNN_REQUIRE(graph && seeds && first && workspace && sizes && batch > 0 && hops >= 0 && (hops == 0 || fanouts),
                 "sample_hops: null argument");
    const HopsLayout L = hops_layout(graph, batch, hops, fanouts, largest_degree);
    CGNN_REQUIRE(L.fits && workspace_bytes >= L.total, "sample_hops: the workspace does not fit this batch");
    CGNN_REQUIRE((reinterpret_cast<uintptr_t>(workspace) & 255) == 0, "sample_hops: workspace must be 256-byte aligned");
    char *base = reinterpret_cast<char *>(workspace);
    uint64_t *counts = reinterpret_cast<uint64_t *>(base + L.counts);
    int32_t *ids = reinterpret_cast<int32_t *>(base + L.ids);
    uint32_t *local = reinterpret_cast<uint32_t *>(base + L.local), *totals = reinterpret_cast<uint32_t *>(base + L.totals);
    int64_t *samples = reinterpret_cast<int64_t *>(base + L.samples);
    int32_t *picked = reinterpret_cast<int32_t *>(base + L.picked), *rows = reinterpret_cast<int32_t *>(base + L.rows);
    int32_t *cols = reinterpret_cast<int32_t *>(base + L.cols);
    const GraphView view = view_of(graph);
    hops_begin_kernel<<<blocks_for(batch), THREADS, 0, stream>>>(seeds, batch, graph->vertices, samples, first, ids, counts);
    CGNN_LAUNCH_CHECK();
    int64_t done = 0;  // slots of the hops before this one
    const int run = (int)L.nodes.size();
    for (int h = 0; h < run; ++h) {
        const int64_t nodes = L.nodes[h], stride = L.stride[h], slots = nodes * stride;
        const HopSlots hop{picked + done, first, slots, (int32_t)(batch + done)};
        const int32_t tiles = (int32_t)ceil_div(slots, TILE);
        // the rule lists use the slots' own part of `rows`: edges are written below it (edges <= slots so far)
        const unsigned grid = (unsigned)std::min<int64_t>(ceil_div(nodes, THREADS / 32), 148 * 64);
        CGNN_CUDA(hops_launch(hops_pick_kernel, grid, stream, view, samples, counts + h, nodes, (int32_t)stride, fanouts[h],
                              (uint32_t)h, seed, hop.base, picked + done, rows + done, first));
        CGNN_CUDA(hops_launch(hops_count_kernel, (unsigned)tiles, stream, hop, local, totals));
        // every block adds up all totals: no more blocks than run at once
        const unsigned blocks = (unsigned)std::min<int64_t>(ceil_div(slots, THREADS), 148 * 6);
        CGNN_CUDA(hops_launch(hops_relabel_kernel, blocks, stream, hop, (int32_t)stride, local, totals, tiles, counts + h, ids,
                              rows, cols, samples));
        done += slots;
    }
    uint64_t last = 0;
    CGNN_CUDA(cudaMemcpyAsync(&last, counts + run + 1, sizeof(last), cudaMemcpyDeviceToHost, stream));
    CGNN_CUDA(cudaStreamSynchronize(stream));
    sizes[0] = (int64_t)(last & 0xffffffffu);
    sizes[1] = (int64_t)(last >> 32);
    return CGNN_OK;
}

int cgnn_sample_hops_result(const cgnn_sample_graph *graph, int64_t batch, int hops, const int64_t *fanouts,
                            int64_t largest_degree, const int64_t sizes[2], int32_t *first, const void *workspace,
                            int64_t *samples_out, int64_t *rows_out, int64_t *cols_out, cgnn_stream_t stream) {
    CGNN_REQUIRE(graph && first && workspace && sizes && batch > 0, "sample_hops_result: null argument");
    const HopsLayout L = hops_layout(graph, batch, hops, fanouts, largest_degree);
    CGNN_REQUIRE(L.fits && sizes[0] >= 0 && sizes[0] <= L.room && sizes[1] >= 0 && sizes[1] <= L.slots &&
                     samples_out != nullptr && (sizes[1] == 0 || (rows_out != nullptr && cols_out != nullptr)),
                 "sample_hops_result: the sizes do not fit this batch");
    const char *base = reinterpret_cast<const char *>(workspace);
    hops_finish_kernel<<<blocks_for(std::max(sizes[0], sizes[1])), THREADS, 0, (cudaStream_t)stream>>>(
        reinterpret_cast<const int64_t *>(base + L.samples), reinterpret_cast<const int32_t *>(base + L.rows),
        reinterpret_cast<const int32_t *>(base + L.cols), sizes[0], sizes[1], graph->vertices, first, samples_out, rows_out,
        cols_out);
    CGNN_LAUNCH_CHECK();
    return CGNN_OK;
}

}  // extern "C"
