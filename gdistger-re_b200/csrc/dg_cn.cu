// Common-neighbour counts per edge on the device: the job of the reference's
// gcn tool (src/tools/gcn.cpp:249-373), whose output becomes the edge data the
// HuGE transition reads (cn = (int)data, walk.hpp:920).
//
// The tool builds the CSR (both directions with --make-undirected), sorts every
// row by neighbour (duplicates kept), and for each input edge (s, d), in input
// order, computes I = the elements of the shorter of N(s), N(d) (N(s) when they
// are equally long) that occur in the other list, with the shorter list's
// multiplicity, ascending (its galloping search, gcn.cpp:152-197).  Then
// cn = |I|, minus one if I[0] is s or d, and, if cn is still above 1, minus one
// for every later element that repeats its predecessor or is s or d
// (gcn.cpp:327-343).  The value is stored on the first CSR entry (s -> d) and its
// mirror, so every later edge over the same unordered pair reports the value
// computed in the orientation of the pair's first occurrence.
//
// Here: one 64-bit sort builds the row-sorted CSR, a stable sort of the pairs'
// unordered keys finds each pair's first occurrence, one warp per first
// occurrence walks the shorter row and looks its elements up in the longer one (a
// bitmap of the longest rows, a binary search in the others), and the counts are
// scattered back to input order.
#include "dg_internal.h"

#include <cub/cub.cuh>

#include <algorithm>
#include <memory>

namespace {

// Keys of two ids in 2 * bits bits: the sorts pass over no others.
__global__ void cn_keys(const uint32_t *src, const uint32_t *dst, uint64_t n, int undirected, int bits, uint64_t *dir) {
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t s = src[i], d = dst[i];
        if (undirected) {
            dir[2 * i] = (s << bits) | d;
            dir[2 * i + 1] = (d << bits) | s;
        } else {
            dir[i] = (s << bits) | d;
        }
    }
}

__global__ void cn_pairs(const uint32_t *src, const uint32_t *dst, uint64_t n, int bits, uint64_t *pair, uint64_t *idx) {
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t s = src[i], d = dst[i];
        pair[i] = s < d ? (s << bits) | d : (d << bits) | s;
        idx[i] = i;
    }
}

__global__ void cn_rows(const uint64_t *dir, uint64_t m, uint32_t v_num, int bits, uint64_t *offsets, uint32_t *nbr) {
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t src = (uint32_t)(dir[i] >> bits);
        const int64_t prev = i == 0 ? -1 : (int64_t)(dir[i - 1] >> bits);
        for (int64_t v = prev + 1; v <= (int64_t)src; v++) offsets[v] = i;
        if (i == m - 1)
            for (uint64_t v = (uint64_t)src + 1; v <= v_num; v++) offsets[v] = m;
        nbr[i] = (uint32_t)(dir[i] & (((uint64_t)1 << bits) - 1));
    }
}

__device__ __forceinline__ bool in_row(const uint32_t *row, uint64_t len, uint32_t x) {
    uint64_t lo = 0, hi = len;
    while (lo < hi) {
        const uint64_t mid = lo + (hi - lo) / 2;
        if (row[mid] < x) lo = mid + 1;
        else hi = mid;
    }
    return lo < len && row[lo] == x;
}

// The longest rows as bitmaps over the vertices: kept to kHubBytes, so that they stay
// in L2, and to rows of at least 2^kHubLog entries, below which a search is as quick.
constexpr uint64_t kHubBytes = 64ull << 20;
constexpr int kHubLog = 7;

struct CnHubs {
    uint32_t *hist;    // [33] rows by length (floor of log2 + 1); then [33]: shortest length that gets a bitmap, [34]: slots given
    int32_t *slot;     // [v_num] bitmap of the vertex's row, -1: none (NULL: no row has one)
    uint32_t *bits;    // [slots][words]
    uint32_t slots, words;
};

__global__ void cn_lengths(const uint64_t *offsets, uint32_t v_num, CnHubs h) {
    __shared__ uint32_t count[33];
    if (threadIdx.x < 33) count[threadIdx.x] = 0;
    __syncthreads();
    for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < v_num; v += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t n = offsets[v + 1] - offsets[v];
        const int log = n ? min(32, 64 - __clzll((long long)n)) : 0;
        if (log > kHubLog) atomicAdd(&count[log], 1u);
    }
    __syncthreads();
    if (threadIdx.x < 33 && count[threadIdx.x]) atomicAdd(&h.hist[threadIdx.x], count[threadIdx.x]);
}

// The smallest power of two that at most `slots` rows reach.
__global__ void cn_pick(CnHubs h) {
    uint32_t rows = 0;
    int log = 33;
    while (log > kHubLog + 1 && rows + h.hist[log - 1] <= h.slots) rows += h.hist[--log];
    h.hist[33] = log > 32 ? ~0u : 1u << (log - 1);
}

__global__ void cn_slots(const uint64_t *offsets, uint32_t v_num, CnHubs h) {
    const uint32_t least = h.hist[33];
    for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < v_num; v += (uint64_t)gridDim.x * blockDim.x)
        h.slot[v] = offsets[v + 1] - offsets[v] >= least ? (int32_t)atomicAdd(&h.hist[34], 1u) : -1;
}

__global__ void cn_bits(const uint64_t *dir, uint64_t m, int bits, CnHubs h) {
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m; i += (uint64_t)gridDim.x * blockDim.x) {
        const int32_t s = h.slot[dir[i] >> bits];
        if (s < 0) continue;
        const uint32_t x = (uint32_t)(dir[i] & (((uint64_t)1 << bits) - 1));
        atomicOr(&h.bits[(uint64_t)s * h.words + (x >> 5)], 1u << (x & 31));
    }
}

// Sum over the warp of counts below 2^48.
__device__ __forceinline__ unsigned long long cn_sum(unsigned long long v) {
    const uint32_t a = __reduce_add_sync(0xffffffffu, (uint32_t)(v & 0xFFFFFFu));
    const uint32_t b = __reduce_add_sync(0xffffffffu, (uint32_t)(v >> 24));
    return (unsigned long long)a + ((unsigned long long)b << 24);
}

// One warp per sorted pair position that starts a group (the pair's first
// occurrence): the count in that occurrence's orientation.  What bounds it is the
// probes of the longer rows: the YouTube-shaped graph's 3.25M pairs have 227M
// elements in their shorter rows, and a binary search each is 2.7G probes of L1 and
// L2 (5.7 ms).  Two fifths to four fifths of the elements are looked up in the few
// hundred longest rows, where a bitmap takes one probe (a pass, host to host: 16 -> 11 ms).
__global__ void cn_count(const uint64_t *pair_sorted, const uint64_t *idx_sorted, uint64_t n, const uint32_t *src,
                         const uint32_t *dst, const uint64_t *offsets, const uint32_t *nbr, CnHubs h, int32_t *cn_sorted) {
    const int lane = threadIdx.x & 31;
    const uint64_t warps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t i = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < n; i += warps) {
        if (i > 0 && pair_sorted[i] == pair_sorted[i - 1]) continue;
        const uint64_t e = idx_sorted[i];
        const uint32_t s = src[e], d = dst[e];
        const uint32_t *r1 = nbr + offsets[s], *r2 = nbr + offsets[d];
        const uint64_t n1 = offsets[s + 1] - offsets[s], n2 = offsets[d + 1] - offsets[d];
        const bool first_long = n1 > n2;                 // gcn.cpp:166-172
        const uint32_t *sh = first_long ? r2 : r1, *lg = first_long ? r1 : r2;
        const uint64_t ns = first_long ? n2 : n1, nl = first_long ? n1 : n2;
        const int32_t slot = h.slot ? h.slot[first_long ? s : d] : -1;
        const uint32_t *bits = h.bits + (slot < 0 ? 0 : (uint64_t)slot * h.words);
        unsigned long long count = 0, dups = 0, sd = 0;
        uint64_t first = ~0ull;
        if (ns > 0 && nl > 0) {
            for (uint64_t j = lane; j < ns; j += 32) {
                const uint32_t x = sh[j];
                if (slot >= 0 ? !((bits[x >> 5] >> (x & 31)) & 1u) : !in_row(lg, nl, x)) continue;
                count++;
                first = min(first, j);
                if (j > 0 && sh[j - 1] == x) dups++;
                else if (x == s || x == d) sd++;
            }
        }
        count = cn_sum(count);
        if (count == 0) {
            if (lane == 0) cn_sorted[i] = 0;
            continue;
        }
        dups = cn_sum(dups);
        sd = cn_sum(sd);
        for (int o = 16; o; o >>= 1) first = min(first, (uint64_t)__shfl_xor_sync(0xffffffffu, (unsigned long long)first, o));
        if (lane == 0) {
            long long c = (long long)count;
            const uint32_t i0 = sh[first];
            const bool i0_sd = i0 == s || i0 == d;
            if (i0_sd) c--;
            // The first element is never a repeat; an s/d first element was taken off above.
            if (c > 1) c -= (long long)dups + (long long)sd - (i0_sd ? 1 : 0);
            cn_sorted[i] = (int32_t)(uint32_t)c;
        }
    }
}

// Every sorted position takes its group head's count and writes it to input order.
__global__ void cn_scatter(const uint64_t *pair_sorted, const uint64_t *idx_sorted, uint64_t n,
                           const int32_t *cn_sorted, int32_t *cn) {
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        uint64_t h = i;
        while (h > 0 && pair_sorted[h - 1] == pair_sorted[i]) h--;
        cn[idx_sorted[i]] = cn_sorted[h];
    }
}

// Bits that hold every id below v_num.
int bits_of(uint32_t v_num) {
    int b = 1;
    while (b < 32 && ((uint64_t)1 << b) < v_num) b++;
    return b;
}

}  // namespace

extern "C" int dg_common_neighbours(const uint32_t *src, const uint32_t *dst, uint64_t n_edges, uint32_t v_num,
                                    int undirected, int device, int32_t *cn) {
    DG_CHECK(n_edges == 0 || (src && dst && cn), DG_ERR_ARG, "dg_common_neighbours: NULL argument");
    DG_CHECK(v_num > 0, DG_ERR_ARG, "dg_common_neighbours: v_num must be positive");
    uint32_t top = 0;   // the largest id: a loop the compiler vectorises
    for (uint64_t i = 0; i < n_edges; i++) top = std::max(top, std::max(src[i], dst[i]));
    if (top >= v_num)
        for (uint64_t i = 0; i < n_edges; i++)
            DG_CHECK(src[i] < v_num && dst[i] < v_num, DG_ERR_ARG, "edge %llu (%u, %u) has a vertex id >= v_num = %u",
                     (unsigned long long)i, src[i], dst[i], v_num);
    if (n_edges == 0) return DG_OK;
    int n_dev = 0;
    DG_CUDA(cudaGetDeviceCount(&n_dev));
    DG_CHECK(device >= 0 && device < n_dev, DG_ERR_ARG, "device %d out of range (%d)", device, n_dev);
    dg::DeviceGuard guard(device);
    cudaStream_t s = nullptr;
    DG_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
    struct StreamGuard {
        cudaStream_t s;
        ~StreamGuard() { cudaStreamSynchronize(s); cudaStreamDestroy(s); }
    } sg{s};
    const uint64_t n = n_edges, m = undirected ? 2 * n : n;
    const unsigned grid = (unsigned)dg::sm_count(device) * 8;
    // One allocation for everything (each costs hundreds of microseconds), cut into
    // 256-byte aligned parts.  The rows' keys are done with when the pairs' are made, and
    // the pairs' sort before the counts: each takes the place of the one before, so the
    // call needs no more memory (64 bytes an edge, 60 of a directed graph, and 8 a vertex,
    // beside the bitmaps) than one with an array each, freed in turn.  Where the bitmaps'
    // room is refused, the call does without them.
    const int key_bits = bits_of(v_num);
    size_t cub_rows = 0, cub_pairs = 0;
    DG_CUDA(cub::DeviceRadixSort::SortKeys(nullptr, cub_rows, (uint64_t *)nullptr, (uint64_t *)nullptr, m, 0, 2 * key_bits, s));
    DG_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, cub_pairs, (uint64_t *)nullptr, (uint64_t *)nullptr,
                                            (uint64_t *)nullptr, (uint64_t *)nullptr, n, 0, 2 * key_bits, s));
    size_t need = 0;
    auto part = [&](size_t bytes) {
        const size_t at = need;
        need += (bytes + 255) / 256 * 256;
        return at;
    };
    const size_t o_src = part(n * 4), o_dst = part(n * 4), o_nbr = part(m * 4), o_off = part(((size_t)v_num + 1) * 8);
    const size_t o_shared = need;
    const size_t o_dir = part(m * 8), o_dir2 = part(m * 8), o_cub_rows = part(cub_rows);
    const size_t rows_end = need;
    need = o_shared;
    const size_t o_pair = part(n * 8), o_pair2 = part(n * 8), o_idx = part(n * 8), o_idx2 = part(n * 8), o_cub_pairs = need;
    part(cub_pairs);
    const size_t pairs_end = need;
    need = o_cub_pairs;
    const size_t o_sorted = part(n * 4), o_cn = part(n * 4);
    need = std::max(need, std::max(rows_end, pairs_end));
    const size_t plain_need = need;
    CnHubs hubs{};
    hubs.words = (v_num + 31) / 32;
    // No more rows than this can have 2^kHubLog entries.
    hubs.slots = (uint32_t)std::min<uint64_t>(kHubBytes / ((uint64_t)hubs.words * 4), m >> kHubLog);
    const size_t hub_bytes = (size_t)hubs.slots * hubs.words * 4;
    const size_t o_hist = part(35 * 4), o_slot = part((size_t)v_num * 4), o_bits = part(hub_bytes);
    dg::DevArray<uint8_t> block;
    if (hubs.slots) {
        const cudaError_t e = block.alloc(need);
        if (e == cudaErrorMemoryAllocation) {
            cudaGetLastError();
            hubs.slots = 0;
        } else {
            DG_CUDA(e);
        }
    }
    if (!hubs.slots) DG_CUDA(block.alloc(plain_need));
    auto u32 = [&](size_t at) { return reinterpret_cast<uint32_t *>(block.p + at); };
    auto u64 = [&](size_t at) { return reinterpret_cast<uint64_t *>(block.p + at); };
    uint32_t *const d_src = u32(o_src), *const d_dst = u32(o_dst), *const nbr = u32(o_nbr);
    uint64_t *const offsets = u64(o_off), *const dir = u64(o_dir), *const dir2 = u64(o_dir2), *const pair = u64(o_pair),
             *const pair2 = u64(o_pair2), *const idx = u64(o_idx), *const idx2 = u64(o_idx2);
    int32_t *const cn_sorted = reinterpret_cast<int32_t *>(block.p + o_sorted), *const d_cn = reinterpret_cast<int32_t *>(block.p + o_cn);
    DG_CUDA(cudaMemcpyAsync(d_src, src, n * 4, cudaMemcpyHostToDevice, s));
    DG_CUDA(cudaMemcpyAsync(d_dst, dst, n * 4, cudaMemcpyHostToDevice, s));
    cn_keys<<<grid, 256, 0, s>>>(d_src, d_dst, n, undirected, key_bits, dir);
    dg::note_launch();
    DG_CUDA(cudaGetLastError());
    // Row-sorted CSR (gcn.cpp:130-137 sorts every row by neighbour).
    DG_CUDA(cub::DeviceRadixSort::SortKeys(block.p + o_cub_rows, cub_rows, dir, dir2, m, 0, 2 * key_bits, s));
    cn_rows<<<grid, 256, 0, s>>>(dir2, m, v_num, key_bits, offsets, nbr);
    dg::note_launch();
    DG_CUDA(cudaGetLastError());
    if (hubs.slots) {
        hubs.hist = u32(o_hist);
        hubs.slot = reinterpret_cast<int32_t *>(block.p + o_slot);
        hubs.bits = u32(o_bits);
        DG_CUDA(cudaMemsetAsync(hubs.hist, 0, 35 * 4, s));
        DG_CUDA(cudaMemsetAsync(hubs.bits, 0, hub_bytes, s));
        cn_lengths<<<grid, 256, 0, s>>>(offsets, v_num, hubs);
        cn_pick<<<1, 1, 0, s>>>(hubs);
        cn_slots<<<grid, 256, 0, s>>>(offsets, v_num, hubs);
        cn_bits<<<grid, 256, 0, s>>>(dir2, m, key_bits, hubs);
        dg::note_launches(4);
        DG_CUDA(cudaGetLastError());
    }
    // Pairs grouped by unordered key, input order kept inside a group (stable sort).
    cn_pairs<<<grid, 256, 0, s>>>(d_src, d_dst, n, key_bits, pair, idx);
    dg::note_launch();
    DG_CUDA(cub::DeviceRadixSort::SortPairs(block.p + o_cub_pairs, cub_pairs, pair, pair2, idx, idx2, n, 0, 2 * key_bits, s));
    cn_count<<<grid, 256, 0, s>>>(pair2, idx2, n, d_src, d_dst, offsets, nbr, hubs, cn_sorted);
    dg::note_launch();
    cn_scatter<<<grid, 256, 0, s>>>(pair2, idx2, n, cn_sorted, d_cn);
    dg::note_launch();
    DG_CUDA(cudaGetLastError());
    DG_CUDA(cudaMemcpyAsync(cn, d_cn, n * 4, cudaMemcpyDeviceToHost, s));
    DG_CUDA(cudaStreamSynchronize(s));
    return DG_OK;
}
