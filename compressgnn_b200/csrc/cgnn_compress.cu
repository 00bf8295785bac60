// Batch pair-substitution grammar compressor on the device.
//
// The reference reaches its CUDA compressor through `compress_csr_batch` of the module
// compressgnn_batch_cuda (src/offline/bindings/batch_cuda.cpp:3-9, chosen by
// loader/compression_backend.py:6-40); the source behind that binding is an external project that is
// not part of the reference tree.  What the reference's tests pin is the contract
// (tests/test_batch_compression.py:15-59): int32 (vlist, elist, n, rules), rule bodies made of smaller
// symbols, exact in-order expansion, and the CUDA result equal to the CPU result array for array.
// This file runs the same rounds as the host compressor of this package (host/cgnn_host.cpp,
// cgnn_host_compress_csr_batch) and produces the same arrays:
//   1. key of every adjacent symbol pair of every vertex row, radix-sorted, run-length counted;
//   2. pairs seen at least `min_frequency` times become candidate rules, ids ascending with the key;
//   3. parse: a candidate is substituted where it outweighs both overlapping neighbours
//      (weight = (count, id)), what is left is taken greedily from the left of each row;
//   4. rows are compacted with a scan, candidates the parse never used are dropped and the ids closed up.
// Everything is integer work on flat arrays: sort, scan and run-length steps are CUB calls, the rest
// are one-thread-per-symbol kernels; the left-to-right step of the parse is one thread per run of open
// positions.  Two small device-to-host reads per round (candidate count; new length and rules kept).
#include <cub/cub.cuh>

#include <algorithm>
#include <memory>

#include "cgnn_common.cuh"

struct cgnn_compressed {
    const int32_t *vlist = nullptr;  // device, rows + 1
    const int32_t *elist = nullptr;  // device, entries
    int64_t n = 0, rules = 0, entries = 0;
    void *owned = nullptr;           // device block the arrays lie in, unless that is the caller's workspace
};

namespace cgnn {
namespace {

constexpr uint64_t NO_PAIR = ~0ull;
constexpr int THREADS = 256;
static inline unsigned blocks_for(int64_t count) {
    return (unsigned)std::max<int64_t>(1, std::min<int64_t>(ceil_div(count, THREADS), 148 * 64));
}
#define GRID_STRIDE(i, count) \
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < (count); i += (int64_t)blockDim.x * gridDim.x)

// Device buffers of one compression, result included, carved out of one block (sized by a dry pass of the same requests):
// the caller's workspace, or an allocation of this call.  What a call without a workspace pays for is
// not the kernels but the driver mapping and unmapping 280 MB.  325 k-node graph, device arrays in and out: 4.0 ms
// without a workspace, 2.6 with one.
struct Arena {
    char *block = nullptr;
    size_t used = 0;
    bool sizing = true;
    template <typename T>
    void carve(T **p, size_t count) {
        const size_t bytes = align_up(std::max<size_t>(count, 1) * sizeof(T), 256);
        *p = sizing ? nullptr : reinterpret_cast<T *>(block + used);
        used += bytes;
    }
};

struct Buffers {
    int32_t *rowptr[2], *sym[2], *row_of[2], *keep, *value, *slot, *run_count, *flag, *cand_count, *uses, *remap, *rule_pairs;
    int32_t *final_vlist;
    uint64_t *key, *key_sorted, *run_key, *cand_key, *weight;
    uint8_t *take, *temp;
    int32_t *scalars;  // 0: bad input, 1: runs, 2: candidates, 3: new total, 4: rules kept
    size_t cand_cap, temp_bytes;
};

// Requests the buffers of a compression of `cap` symbols (rows only shrink); returns the bytes they take.
static size_t carve_buffers(Arena &arena, Buffers &b, int64_t n, int64_t cap, int min_frequency) {
    for (int i = 0; i < 2; ++i) {
        arena.carve(&b.rowptr[i], (size_t)n + 1);
        arena.carve(&b.sym[i], (size_t)cap);
        arena.carve(&b.row_of[i], (size_t)cap);
    }
    b.cand_cap = (size_t)(cap / min_frequency + 1);  // at most one candidate per min_frequency pairs
    for (int32_t **p : {&b.keep, &b.value, &b.slot, &b.run_count, &b.flag}) arena.carve(p, (size_t)cap);
    for (uint64_t **p : {&b.key, &b.key_sorted, &b.run_key, &b.weight}) arena.carve(p, (size_t)cap);
    arena.carve(&b.take, (size_t)cap);
    arena.carve(&b.scalars, 8);
    arena.carve(&b.cand_key, b.cand_cap);
    for (int32_t **p : {&b.cand_count, &b.uses, &b.remap}) arena.carve(p, b.cand_cap);
    // a kept rule is used, and every use takes a symbol away: at most `cap` rules, and symbols + rules <= cap
    arena.carve(&b.rule_pairs, 2 * (size_t)cap);
    arena.carve(&b.final_vlist, (size_t)n + (size_t)cap + 1);
    size_t need = 0;
    b.temp_bytes = 0;
    const int cap32 = (int)std::max<int64_t>(cap, 1);
    uint64_t *k = nullptr;
    int32_t *w = nullptr;
    cub::DeviceRadixSort::SortKeys(nullptr, need, k, k, cap32, 0, 64);
    b.temp_bytes = std::max(b.temp_bytes, need);
    cub::DeviceRunLengthEncode::Encode(nullptr, need, k, k, w, w, cap32);
    b.temp_bytes = std::max(b.temp_bytes, need);
    cub::DeviceScan::ExclusiveSum(nullptr, need, w, w, cap32);
    b.temp_bytes = std::max(b.temp_bytes, need);
    arena.carve(&b.temp, b.temp_bytes);
    return arena.used;
}

__global__ void load_rows_kernel(const int64_t *vlist, const int64_t *elist, int64_t n, int64_t total, int32_t *rowptr,
                                 int32_t *sym, int *bad) {
    GRID_STRIDE(i, n + 1) {
        const int64_t v = vlist[i];
        if (v < 0 || v > total || (i > 0 && v < vlist[i - 1]) || (i == 0 && v != 0)) atomicOr(bad, 1);
        rowptr[i] = (int32_t)v;
    }
    GRID_STRIDE(i, total) {
        const int64_t e = elist[i];
        if (e < 0 || e >= n) atomicOr(bad, 2);
        sym[i] = (int32_t)e;
    }
}

__global__ void row_of_kernel(const int32_t *rowptr, int64_t n, int32_t *row_of) {
    GRID_STRIDE(r, n)
        for (int32_t i = rowptr[r]; i < rowptr[r + 1]; ++i) row_of[i] = (int32_t)r;
}

// key[i] = (sym[i], sym[i+1]) packed into 2 * shift bits when both belong to one row
__global__ void pair_keys_kernel(const int32_t *sym, const int32_t *row_of, int64_t total, int shift, uint64_t *key) {
    GRID_STRIDE(i, total) {
        uint64_t k = NO_PAIR;
        if (i + 1 < total && row_of[i] == row_of[i + 1]) k = ((uint64_t)(uint32_t)sym[i] << shift) | (uint32_t)sym[i + 1];
        key[i] = k;
    }
}

__global__ void flag_candidates_kernel(const uint64_t *run_key, const int32_t *run_count, const int *num_runs,
                                       int min_frequency, int32_t *flag) {
    const int64_t runs = *num_runs;
    GRID_STRIDE(r, runs) flag[r] = (run_key[r] != NO_PAIR && run_count[r] >= min_frequency) ? 1 : 0;
}

__global__ void gather_candidates_kernel(const uint64_t *run_key, const int32_t *run_count, const int32_t *flag,
                                         const int32_t *slot, const int *num_runs, uint64_t *cand_key,
                                         int32_t *cand_count, int32_t *cand_total) {
    const int64_t runs = *num_runs;
    GRID_STRIDE(r, runs) {
        if (flag[r]) {
            cand_key[slot[r]] = run_key[r];
            cand_count[slot[r]] = run_count[r];
        }
        if (r == runs - 1) *cand_total = slot[r] + flag[r];
    }
    if (runs == 0 && blockIdx.x == 0 && threadIdx.x == 0) *cand_total = 0;
}

// weight[i] = (count of the pair at i) << 32 | (its candidate id), or 0 when the pair is no candidate
__global__ void weights_kernel(const uint64_t *key, int64_t total, const uint64_t *cand_key, const int32_t *cand_count,
                               int32_t candidates, int32_t base, uint64_t *weight) {
    GRID_STRIDE(i, total) {
        const uint64_t k = key[i];
        uint64_t w = 0;
        if (k != NO_PAIR) {
            int32_t lo = 0, hi = candidates;
            while (lo < hi) {
                const int32_t mid = (lo + hi) >> 1;
                if (cand_key[mid] < k) lo = mid + 1;
                else hi = mid;
            }
            if (lo < candidates && cand_key[lo] == k) w = ((uint64_t)(uint32_t)cand_count[lo] << 32) | (uint32_t)(base + lo);
        }
        weight[i] = w;
    }
}

// First step of the parse: a candidate that outweighs the pair before it and is not outweighed by the
// pair after it (pairs of its own row only).
__global__ void take_heavier_kernel(const uint64_t *key, const uint64_t *weight, int64_t total, uint8_t *take) {
    GRID_STRIDE(i, total) {
        const uint64_t w = weight[i];
        bool t = false;
        if (w != 0) {
            const bool has_prev = i > 0 && key[i - 1] != NO_PAIR;       // a pair of the same row sits before / after
            const bool has_next = i + 1 < total && key[i] != NO_PAIR && key[i + 1] != NO_PAIR;
            t = (!has_prev || w > weight[i - 1]) && (!has_next || w >= weight[i + 1]);
        }
        take[i] = t ? 1 : 0;
    }
}

// Second step: left to right along each row, a remaining candidate whose neighbours are free.
//
// That rule is a chain, but a short one: a position is OPEN when it is a candidate the first step left, with no
// pair of the first step behind it.  Along a run of open positions the taken ones simply alternate, starting with
// the first unless the pair before the run was taken; everything between two runs is settled already.  So the
// thread of a run's first position walks the run (rows of the web graph: a few symbols); one thread to a row would
// walk whole rows, the longest of 10,000 symbols.  Five rounds on the 325 k-node graph: 90 us, by rows 649.
// take[]: bit 0 the first step, bit 1 this one; a run's bytes are written by its own thread and other threads
// look at bit 0 only.
__global__ void take_greedy_kernel(const uint64_t *key, const uint64_t *weight, int64_t total, uint8_t *take) {
    // (a candidate is a pair of one row, so weight != 0 implies key != NO_PAIR; the key after a row's last pair is NO_PAIR)
    auto open = [&](int64_t i) {
        return weight[i] != 0 && !(take[i] & 1) && (i + 1 == total || key[i + 1] == NO_PAIR || !(take[i + 1] & 1));
    };
    GRID_STRIDE(i, total) {
        if (!open(i)) continue;
        const bool has_prev = i > 0 && key[i - 1] != NO_PAIR;
        if (has_prev && open(i - 1)) continue;  // inside a run
        bool taken = has_prev && (take[i - 1] & 1);
        int64_t at = i;
        do {
            taken = !taken;
            if (taken) take[at] = 2;
            ++at;
        } while (at < total && key[at] != NO_PAIR && open(at));
    }
}

// A symbol is kept unless the pair before it was substituted; a substituted pair leaves its rule id.
__global__ void emit_kernel(const int32_t *sym, const uint64_t *key, const uint64_t *weight, const uint8_t *take,
                            int64_t total, int32_t base, int32_t *keep, int32_t *value, int32_t *uses) {
    GRID_STRIDE(i, total) {
        const bool swallowed = i > 0 && key[i - 1] != NO_PAIR && take[i - 1];
        const bool head = key[i] != NO_PAIR && take[i];
        keep[i] = swallowed ? 0 : 1;
        int32_t v = sym[i];
        if (head) {
            v = (int32_t)(uint32_t)weight[i];
            atomicAdd(&uses[v - base], 1);
        }
        value[i] = v;
    }
}

__global__ void compact_kernel(const int32_t *keep, const int32_t *slot, const int32_t *value, const int32_t *row_of,
                               int64_t total, int32_t *sym_out, int32_t *row_of_out, int32_t *new_total) {
    GRID_STRIDE(i, total) {
        if (keep[i]) {
            sym_out[slot[i]] = value[i];
            row_of_out[slot[i]] = row_of[i];
        }
        if (i == total - 1) *new_total = slot[i] + keep[i];
    }
}

// The first symbol of a row is always kept, so a row starts where its old first symbol went.
__global__ void move_rowptr_kernel(const int32_t *rowptr, const int32_t *slot, const int32_t *new_total, int64_t n,
                                   int64_t total, int32_t *rowptr_out) {
    GRID_STRIDE(r, n + 1) {
        const int32_t old = rowptr[r];
        rowptr_out[r] = old < total ? slot[old] : *new_total;
    }
}

__global__ void used_flags_kernel(const int32_t *uses, int32_t candidates, int32_t *used) {
    GRID_STRIDE(k, candidates) used[k] = uses[k] > 0 ? 1 : 0;
}

__global__ void keep_rules_kernel(const uint64_t *cand_key, const int32_t *used, const int32_t *rank, int32_t candidates,
                                  int shift, int32_t base, int32_t *remap, int32_t *rule_pairs, int32_t *kept) {
    const uint64_t low = (1ull << shift) - 1;
    GRID_STRIDE(k, candidates) {
        if (used[k]) {
            remap[k] = base + rank[k];
            rule_pairs[2 * (int64_t)rank[k]] = (int32_t)(cand_key[k] >> shift);
            rule_pairs[2 * (int64_t)rank[k] + 1] = (int32_t)(cand_key[k] & low);
        } else {
            remap[k] = -1;
        }
        if (k == candidates - 1) *kept = rank[k] + used[k];
    }
}

__global__ void remap_kernel(int32_t *sym, int64_t total, int32_t base, const int32_t *remap) {
    GRID_STRIDE(i, total) {
        const int32_t s = sym[i];
        if (s >= base) sym[i] = remap[s - base];
    }
}

__global__ void final_vlist_kernel(const int32_t *rowptr, int64_t n, int64_t rules, int32_t total, int32_t *vlist) {
    GRID_STRIDE(i, n + rules + 1) vlist[i] = i <= n ? rowptr[i] : total + 2 * (int32_t)(i - n);
}

static int bits_for(int64_t largest) {
    int bits = 1;
    while ((largest >> bits) != 0) ++bits;
    return bits;
}

}  // namespace
}  // namespace cgnn

using namespace cgnn;

extern "C" {

size_t cgnn_compress_workspace_bytes(int64_t n, int64_t entries, int min_frequency) {
    if (n < 0 || entries < 0 || min_frequency < 3 || n + entries >= INT32_MAX) return 0;
    Arena arena;
    Buffers b;
    return carve_buffers(arena, b, n, entries, min_frequency);
}

int cgnn_compress_csr_batch(const int64_t *vlist, const int64_t *elist, int64_t n, int rounds, int min_frequency,
                            cgnn_compressed **out, cgnn_stream_t stream) {
    return cgnn_compress_csr_batch_in(vlist, elist, n, rounds, min_frequency, nullptr, 0, out, stream);
}

int cgnn_compress_csr_batch_in(const int64_t *vlist, const int64_t *elist, int64_t n, int rounds, int min_frequency,
                               void *workspace, size_t workspace_bytes, cgnn_compressed **out, cgnn_stream_t stream_) {
    cudaStream_t stream = (cudaStream_t)stream_;
    CGNN_REQUIRE(out != nullptr, "compress_csr_batch: null result pointer");
    *out = nullptr;
    CGNN_REQUIRE(n >= 0 && (n == 0 || vlist != nullptr), "compress_csr_batch: null row pointers");
    CGNN_REQUIRE(min_frequency >= 3, "Batch compression needs min_pair_frequency >= 3");
    CGNN_REQUIRE(rounds >= 1, "compression_rounds must be positive");
    int64_t total64 = 0;
    if (n > 0) CGNN_CUDA(cudaMemcpyAsync(&total64, vlist + n, sizeof(int64_t), cudaMemcpyDeviceToHost, stream));
    CGNN_CUDA(cudaStreamSynchronize(stream));
    CGNN_REQUIRE(total64 >= 0 && n + total64 < INT32_MAX, "CSR array exceeds int32 capacity");
    CGNN_REQUIRE(total64 == 0 || elist != nullptr, "compress_csr_batch: null edge list");
    const int64_t cap = total64;  // rows only shrink

    Arena arena;
    Buffers buf;
    const size_t bytes = carve_buffers(arena, buf, n, cap, min_frequency);
    std::unique_ptr<cgnn_compressed, decltype(&cgnn_compressed_destroy)> res(new cgnn_compressed(), cgnn_compressed_destroy);
    if (workspace == nullptr) {
        CGNN_CUDA(cudaMalloc(&res->owned, bytes));
        workspace = res->owned;
    } else {
        CGNN_REQUIRE(workspace_bytes >= bytes && (reinterpret_cast<uintptr_t>(workspace) & 255) == 0,
                     "compress_csr_batch: workspace of %zu bytes on a 256-byte boundary needed, %zu given", bytes,
                     workspace_bytes);
    }
    arena.block = static_cast<char *>(workspace);
    arena.used = 0;
    arena.sizing = false;
    carve_buffers(arena, buf, n, cap, min_frequency);
    int32_t **rowptr = buf.rowptr, **sym = buf.sym, **row_of = buf.row_of, *keep = buf.keep, *value = buf.value;
    int32_t *slot = buf.slot, *run_count = buf.run_count, *flag = buf.flag, *cand_count = buf.cand_count, *uses = buf.uses;
    int32_t *remap = buf.remap, *scalars = buf.scalars;
    uint64_t *key = buf.key, *key_sorted = buf.key_sorted, *run_key = buf.run_key, *cand_key = buf.cand_key;
    uint64_t *weight = buf.weight;
    uint8_t *take = buf.take, *temp = buf.temp;
    const size_t cand_cap = buf.cand_cap, temp_bytes = buf.temp_bytes;
    size_t need = 0;
    CGNN_CUDA(cudaMemsetAsync(scalars, 0, 8 * sizeof(int32_t), stream));
    int32_t *used = flag, *rank = slot;  // free again once the rows are compacted

    load_rows_kernel<<<blocks_for(std::max(n + 1, cap)), THREADS, 0, stream>>>(vlist, elist, n, cap, rowptr[0], sym[0],
                                                                              scalars);
    CGNN_LAUNCH_CHECK();
    int32_t host_scalars[8];
    CGNN_CUDA(cudaMemcpyAsync(host_scalars, scalars, sizeof(host_scalars), cudaMemcpyDeviceToHost, stream));
    CGNN_CUDA(cudaStreamSynchronize(stream));
    // nothing indexes with the row pointers before they are known to be sound
    CGNN_REQUIRE(!(host_scalars[0] & 1), "compress_csr_batch: row pointers must ascend from 0 to the edge count");
    CGNN_REQUIRE(!(host_scalars[0] & 2), "CSR value exceeds vertex range");
    row_of_kernel<<<blocks_for(n), THREADS, 0, stream>>>(rowptr[0], n, row_of[0]);
    CGNN_LAUNCH_CHECK();

    int64_t total = cap, rules = 0;
    int cur = 0;
    for (int round = 0; round < rounds && total > 1; ++round) {
        const int32_t base = (int32_t)(n + rules);
        const int shift = bits_for(std::max<int64_t>(base - 1, 1));
        const int total32 = (int)total;
        pair_keys_kernel<<<blocks_for(total), THREADS, 0, stream>>>(sym[cur], row_of[cur], total, shift, key);
        CGNN_LAUNCH_CHECK();
        need = temp_bytes;
        // pair keys use 2 * shift bits and the key of "no pair" is all ones: bit 2 * shift puts it last
        CGNN_CUDA(cub::DeviceRadixSort::SortKeys(temp, need, key, key_sorted, total32, 0, std::min(64, 2 * shift + 1),
                                                 stream));
        need = temp_bytes;
        CGNN_CUDA(cub::DeviceRunLengthEncode::Encode(temp, need, key_sorted, run_key, run_count, scalars + 1, total32,
                                                     stream));
        flag_candidates_kernel<<<blocks_for(total), THREADS, 0, stream>>>(run_key, run_count, scalars + 1, min_frequency,
                                                                          flag);
        CGNN_LAUNCH_CHECK();
        // (slots past the number of runs hold stale flags; the gather below stops at the number of runs)
        need = temp_bytes;
        CGNN_CUDA(cub::DeviceScan::ExclusiveSum(temp, need, flag, slot, total32, stream));
        gather_candidates_kernel<<<blocks_for(total), THREADS, 0, stream>>>(run_key, run_count, flag, slot, scalars + 1,
                                                                            cand_key, cand_count, scalars + 2);
        CGNN_LAUNCH_CHECK();
        CGNN_CUDA(cudaMemcpyAsync(host_scalars, scalars, sizeof(host_scalars), cudaMemcpyDeviceToHost, stream));
        CGNN_CUDA(cudaStreamSynchronize(stream));
        const int32_t candidates = host_scalars[2];
        if (candidates == 0) break;
        CGNN_REQUIRE((int64_t)base + candidates < INT32_MAX, "rule ids exceed int32 capacity");
        CGNN_REQUIRE((size_t)candidates <= cand_cap, "compress_csr_batch: candidate table overflow");

        weights_kernel<<<blocks_for(total), THREADS, 0, stream>>>(key, total, cand_key, cand_count, candidates, base,
                                                                  weight);
        CGNN_LAUNCH_CHECK();
        take_heavier_kernel<<<blocks_for(total), THREADS, 0, stream>>>(key, weight, total, take);
        CGNN_LAUNCH_CHECK();
        take_greedy_kernel<<<blocks_for(total), THREADS, 0, stream>>>(key, weight, total, take);
        CGNN_LAUNCH_CHECK();
        CGNN_CUDA(cudaMemsetAsync(uses, 0, (size_t)candidates * sizeof(int32_t), stream));
        emit_kernel<<<blocks_for(total), THREADS, 0, stream>>>(sym[cur], key, weight, take, total, base, keep, value,
                                                               uses);
        CGNN_LAUNCH_CHECK();
        need = temp_bytes;
        CGNN_CUDA(cub::DeviceScan::ExclusiveSum(temp, need, keep, slot, total32, stream));
        compact_kernel<<<blocks_for(total), THREADS, 0, stream>>>(keep, slot, value, row_of[cur], total, sym[cur ^ 1],
                                                                  row_of[cur ^ 1], scalars + 3);
        CGNN_LAUNCH_CHECK();
        move_rowptr_kernel<<<blocks_for(n + 1), THREADS, 0, stream>>>(rowptr[cur], slot, scalars + 3, n, total,
                                                                      rowptr[cur ^ 1]);
        CGNN_LAUNCH_CHECK();
        cur ^= 1;
        // candidates the parse never used are dropped, the others keep their order
        used_flags_kernel<<<blocks_for(candidates), THREADS, 0, stream>>>(uses, candidates, used);
        CGNN_LAUNCH_CHECK();
        need = temp_bytes;
        CGNN_CUDA(cub::DeviceScan::ExclusiveSum(temp, need, used, rank, candidates, stream));
        keep_rules_kernel<<<blocks_for(candidates), THREADS, 0, stream>>>(cand_key, used, rank, candidates, shift, base,
                                                                          remap, buf.rule_pairs + 2 * rules, scalars + 4);
        CGNN_LAUNCH_CHECK();
        CGNN_CUDA(cudaMemcpyAsync(host_scalars, scalars, sizeof(host_scalars), cudaMemcpyDeviceToHost, stream));
        CGNN_CUDA(cudaStreamSynchronize(stream));
        total = host_scalars[3];
        const int32_t kept = host_scalars[4];
        if (kept != candidates) {
            remap_kernel<<<blocks_for(total), THREADS, 0, stream>>>(sym[cur], total, base, remap);
            CGNN_LAUNCH_CHECK();
        }
        rules += kept;
    }

    CGNN_REQUIRE(total + 2 * rules < INT32_MAX, "compressed arrays exceed int32 capacity");
    res->n = n;
    res->rules = rules;
    res->entries = total + 2 * rules;
    final_vlist_kernel<<<blocks_for(n + rules + 1), THREADS, 0, stream>>>(rowptr[cur], n, rules, (int32_t)total,
                                                                          buf.final_vlist);
    CGNN_LAUNCH_CHECK();
    // rows, then rule bodies: the pair keys are free by now and hold 2 * cap words
    int32_t *elist_out = reinterpret_cast<int32_t *>(key);
    if (total > 0)
        CGNN_CUDA(cudaMemcpyAsync(elist_out, sym[cur], (size_t)total * sizeof(int32_t), cudaMemcpyDeviceToDevice, stream));
    if (rules > 0)
        CGNN_CUDA(cudaMemcpyAsync(elist_out + total, buf.rule_pairs, 2 * (size_t)rules * sizeof(int32_t),
                                  cudaMemcpyDeviceToDevice, stream));
    res->vlist = buf.final_vlist;
    res->elist = elist_out;
    if (res->owned) {  // the work arrays go, the result moves to an allocation of its own size
        const size_t v_bytes = align_up((size_t)(n + rules + 1) * sizeof(int32_t), 256);
        const size_t e_bytes = std::max<size_t>((size_t)res->entries, 1) * sizeof(int32_t);
        void *exact = nullptr;
        CGNN_CUDA(cudaMalloc(&exact, v_bytes + e_bytes));
        std::swap(res->owned, exact);
        std::unique_ptr<void, cudaError_t (*)(void *)> work(exact, cudaFree);
        char *base = static_cast<char *>(res->owned);
        CGNN_CUDA(cudaMemcpyAsync(base, res->vlist, (size_t)(n + rules + 1) * sizeof(int32_t), cudaMemcpyDeviceToDevice,
                                  stream));
        CGNN_CUDA(cudaMemcpyAsync(base + v_bytes, res->elist, (size_t)res->entries * sizeof(int32_t),
                                  cudaMemcpyDeviceToDevice, stream));
        CGNN_CUDA(cudaStreamSynchronize(stream));
        res->vlist = reinterpret_cast<const int32_t *>(base);
        res->elist = reinterpret_cast<const int32_t *>(base + v_bytes);
    }
    *out = res.release();
    return CGNN_OK;
}

int cgnn_compressed_info(const cgnn_compressed *c, int64_t info[3]) {
    CGNN_REQUIRE(c != nullptr && info != nullptr, "compressed_info: null argument");
    info[0] = c->n;
    info[1] = c->rules;
    info[2] = c->entries;
    return CGNN_OK;
}

int cgnn_compressed_copy(const cgnn_compressed *c, int32_t *vlist_out, int32_t *elist_out, cgnn_stream_t stream_) {
    cudaStream_t stream = (cudaStream_t)stream_;
    CGNN_REQUIRE(c != nullptr && vlist_out != nullptr, "compressed_copy: null argument");
    CGNN_REQUIRE(c->entries == 0 || elist_out != nullptr, "compressed_copy: null edge list");
    CGNN_CUDA(cudaMemcpyAsync(vlist_out, c->vlist, (size_t)(c->n + c->rules + 1) * sizeof(int32_t), cudaMemcpyDefault,
                              stream));
    if (c->entries > 0)
        CGNN_CUDA(cudaMemcpyAsync(elist_out, c->elist, (size_t)c->entries * sizeof(int32_t), cudaMemcpyDefault, stream));
    return CGNN_OK;
}

void cgnn_compressed_destroy(cgnn_compressed *c) {
    if (!c) return;
    if (c->owned) cudaFree(c->owned);
    delete c;
}

}  // extern "C"
