// Hogwild CBOW on FP32 rows (cbow_kernel, word2vec.cu:401-509), two centres at a
// time: the form of DG_SGNS_CBOW that trains walks of at most 32 tokens with rows
// of 128 columns (sizes 65 to 128) and up to five negatives, or, with hierarchical
// softmax, up to 256 columns and eight negatives (sgns_cbow_kernel, dg_sgns_w2v.cu,
// trains the others and the one-warp deterministic runs).
//
// What bounds the rule is the L2's reduction rate.  A centre with cw contexts and
// n negatives reads cw + 1 + n rows and adds to as many; on rows that L2 holds, a
// B200 reads 18.1 TB/s of 512-byte rows but reduces into them at 5.9 TB/s (a
// vector atomic and a bulk reduction alike).  9 contexts and 6 targets are 1.30 ns
// of reductions and 0.42 ns of reads a centre; the kernel that trains one centre at
// a time takes 1.75.  The windows of two neighbouring centres are nearly the same
// rows, so here a warp reads the rows of both at once and each row receives the sum
// of both centres' e in one atomic: 6.2 row reads and reductions a centre for the
// contexts, not 9.
//
// Measured on a B200, size 128, window 10, negative 5: two YouTube-shaped rounds with
// their read-back in 101 ms instead of 115, three of the 10,000-vertex graph at size
// 100 (whose padding columns are no longer moved) in 1.76 ms instead of 2.29.  What
// bounds it now: the L2 reductions (12.2 rows a centre, 1.06 ns a token), DRAM (5 KB a
// token, 0.76 ns), and the latency of a turn's four groups of targets.
//
// A Hogwild run's rows depend on how many updates are under way unseen and on how
// many walks are trained at once.  So 16 warps of an SM train two centres each,
// where sgns_cbow_kernel's 32 train one, and each holds two walks that it trains in
// turn: 32 walks, 32 centres under way; and the targets are read as that kernel reads
// them, after the mean, three at a time, each group written before the next is read.
// All of them read before the contexts were 9 % faster (92 ms), but an output row then
// misses twice as much, and whole jobs from learning rate 0.025 ended 0.0043 lower in
// link-prediction AUC (32 jobs on the 10,000-vertex graph; all at once after the mean:
// 0.0012; as here: 0.0002 +- 0.0002).
// Measured against sgns_cbow_kernel's rows, over the distance of two equal runs of that
// kernel (graphs of 10,000 to 1.1M vertices, windows 1 to 10, a job's last learning rate):
//   columns   negatives   input rows   output rows
//   65..128   0..5        1.1 .. 2.2   1.0 .. 1.7
//   65..128   7, 8        2.1 .. 3.0   1.6 .. 2.0
//   32, 64    1..8        1.2 .. 3.0   1.1 .. 1.8
//   200, 256  3..8        1.9 .. 3.1   1.2 .. 2.8    (no hierarchical softmax)
//   64..256   3..8, HS    0.9 .. 1.8   0.9 .. 1.3
// Hence the rule: with more negatives than five, and at 64 columns on small graphs, single
// values end further off than that kernel's own runs show; at 256 columns its registers
// leave it eight warps, so eight warps of two centres have twice as many under way.  With
// hierarchical softmax the updates of the rows near the root outweigh all that, and both
// kernels' runs differ alike.
// Other schedules were further off: 14 or 12 warps of 16 (up to 4.9 and 6.0), four
// centres at a time (8.06 ms for 300,000 walks, two: 9.3).
#include "dg_pair_grid.h"
#include "dg_sgns.h"
#include "dg_sgns_dev.cuh"

#include <algorithm>

namespace dgs {

constexpr int kCbowWarps = 8;             // warps of a block
constexpr uint32_t kCbowMaxTokens = 32;   // a lane per token
constexpr int kCbowPairNeg = 5;           // the largest negative count of this kernel
constexpr int kCbowPairHsNeg = 8;         // the same with hierarchical softmax
constexpr int kCbowPairSize = 128;        // the row without it

constexpr int cbow_pair_group(int vec) { return vec <= 2 ? 4 : vec == 4 ? 3 : 2; }   // target rows read together, as sgns_cbow_kernel
constexpr int cbow_pair_walks(int vec) { return vec <= 4 ? 2 : 1; }    // walks that a warp trains in turn
constexpr int cbow_pair_blocks(int vec) { return vec <= 4 ? 2 : 1; }   // blocks per SM

// Hierarchical softmax: the table's kHotNodes last rows, spread.
constexpr uint32_t kHotNodes = 64;
constexpr uint32_t kHotPiece = 256;   // floats from one piece of a row to the next: the L2's slices change
constexpr uint32_t kHotFloats = kHotNodes * 8 * kHotPiece;

// Floats from the buffer's start to lane l's columns of hot row r: four lanes to a piece.
template <int VEC>
__device__ __forceinline__ uint32_t hot_offset(uint32_t r, uint32_t l) {
    static_assert(4 * VEC <= (int)kHotPiece, "a piece holds four lanes' columns");
    return (r * 8 + (l >> 2)) * kHotPiece + (l & 3) * VEC;
}

// Output rows [from, from + gridDim.x) into the buffer (in) or back, a warp per row.
template <int VEC>
__global__ void cbow_hot_rows(float *syn1, float *hot, int32_t from, bool in) {
    float *row = syn1 + (size_t)(from + blockIdx.x) * (32 * VEC) + threadIdx.x * VEC;
    float *at = hot + hot_offset<VEC>(blockIdx.x, threadIdx.x);
    RowVec<VEC> r;
    load_row<VEC>(in ? row : at, r);
    store_row<VEC>(in ? at : row, r);
}

// A walk under way: its length, its next centre, and for token / centre `lane` the
// word, the positions that hold the same word, the window as a mask of positions
// and the targets' flags (bit j: target j trains, 0 being the centre's word; bit
// 31: a target repeats).
struct CbowWalk {
    uint32_t n = 0, p = 0;
    int32_t word = 0;
    uint32_t same = 0, win = 0, flags = 0;
    int32_t *sen = nullptr, *negs = nullptr;   // shared: the words, the negatives of every centre
};

// Lane l owns columns [l * VEC, l * VEC + VEC) of every row and, beside that, token
// l of the walk (CbowWalk).  A warp holds `walks` walks and trains two centres of
// each in turn.
//
// The second centre's context rows were read before the first centre's e: they
// are short of it by e times the number of (position of one window, position of
// the other) pairs that hold one word, which is added to their sum.  So this
// warp's own updates are all seen.  Target rows are read after their centre's
// mean, and so after the reductions of the centre before.
//
// Room for NS negatives; FIXED: NS of them (word2vec's default), else a.negative.
//
// HS: hierarchical softmax over the centre's Huffman path before its targets
// (word2vec.cu:436-455; hs_path, dg_sgns_dev.cuh).  Every path runs through the
// nodes near the root, and what bounds it is that the L2 serves one row's read and
// reduction per 8.3 ns as long as both rows of a kilobyte are one slice's work: the
// root and its two neighbours cost 1.1M tokens 9 ms of 10.3.  So for the launch the
// kHotNodes most visited nodes' rows (the last inner nodes made, so the highest ids)
// move to a buffer whose rows lie in eight pieces a kilobyte apart (hot_offset),
// each another slice's.  A path's nodes are read two at a time: a round of the
// 50,000-vertex graph, size 128, window 5, with its read-back 11.3 -> 7.4 ms (one at a
// time 7.4, four 7.2).  Read together, a node misses the updates that reach it while the
// others are summed, and every centre trains the root: link-prediction AUC of whole jobs
// on the 10,000-vertex graph (16 each) from learning rate 0.01 is 0.548 with hs_path, whose
// nodes wait for one another, 0.524 with four, 0.557 with two, 0.595 with one (from
// 0.025 0.486, 0.479, 0.483, 0.487): two is what differs least.  (On the YouTube-shaped
// graph from 0.01: 0.570 with hs_path, 0.606 here; without hierarchical softmax 0.828 in
// both kernels.)
template <int VEC, bool HS, bool FIXED>
__global__ void __launch_bounds__(kCbowWarps * 32, cbow_pair_blocks(VEC))
    sgns_cbow_pair_kernel(SgnsArgs a, WalkSet ws, uint32_t walks, float *hot, int32_t hot_from) {
    constexpr int NS = HS ? kCbowPairHsNeg : kCbowPairNeg;
    constexpr int D = 32 * VEC, G = cbow_pair_group(VEC), M = pow2_at_least(G), GROUP = 32 / M;
    constexpr int BATCH = VEC <= 4 ? 8 : 4;   // context rows in flight together
    constexpr uint32_t kAll = 0xffffffffu;
    __shared__ __align__(16) int32_t sen_all[kCbowWarps][2][kCbowMaxTokens];
    __shared__ int32_t negs_all[kCbowWarps][2][kCbowMaxTokens * NS];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int neg = FIXED ? NS : a.negative;
    const uint32_t w = (uint32_t)a.window;
    // Lanes whose columns are all padding (a size such as 100 or 200, stored with
    // the next power of two) read lane 0's columns, hold x = 0, give 0 to every sum
    // (0 times an infinity would be no number) and write nothing.
    const bool own = lane * VEC < (uint32_t)a.used;
    float *const syn0 = a.syn0 + (own ? lane * VEC : 0), *const syn1 = a.syn1 + (own ? lane * VEC : 0);
    // This lane's columns of output row `id`.
    auto out_row = [&](int32_t id) {
        if (HS && id >= hot_from) return hot + hot_offset<VEC>((uint32_t)(id - hot_from), own ? lane : 0);
        return syn1 + (size_t)id * D;
    };
    unsigned long long n_words = 0, n_trained = 0, n_pairs = 0;
    CbowWalk A, B;
    A.sen = sen_all[warp][0];
    A.negs = negs_all[warp][0];
    B.sen = sen_all[warp][1];
    B.negs = negs_all[warp][1];
    bool more = true;

    // The next walk of at least two tokens into A; A.n = 0 when there is none left.
    auto fetch = [&]() {
        A.n = A.p = 0;
        while (more) {
            uint32_t walk = 0;
            if (lane == 0) walk = atomicAdd(a.queue, 1u);
            walk = __shfl_sync(kAll, walk, 0);
            more = walk < ws.n_walks;
            if (!more) return;
            const uint32_t wid = ws.ids ? ws.ids[walk] : walk + ws.id_base;
            uint32_t words;
            __syncwarp();
            const uint32_t n = warp_sentence<kCbowMaxTokens>(ws, walk, a, A.sen, words);
            n_words += words;
            n_trained += n;
            if (n < 2) continue;
            A.n = n;
            A.word = lane < n ? A.sen[lane] : -1 - (int32_t)lane;
            A.same = __match_any_sync(kAll, A.word);
            A.win = 0;
            if (lane < n) {   // positions within the shrunk span, the centre excluded
                const uint32_t span = w - philox(lane, wid, a.pass, kWinTag, a.seed_lo, a.seed_hi).x % w;
                const uint32_t lo = lane > span ? lane - span : 0u, hi = min(n - 1, lane + span);
                A.win = ((kAll >> (31 - (hi - lo))) << lo) & ~(1u << lane);
                n_pairs += __popc(A.win);
            }
            for (uint32_t q = lane; q < n * (uint32_t)neg; q += 32) {
                const uint32_t p = q / (uint32_t)neg, j = q % (uint32_t)neg;
                A.negs[p * NS + j] = tagged_negative(a, p, wid, kCbowTag, (int)j);
            }
            __syncwarp();
            A.flags = 1;
            if (lane < n)
                for (int j = 0; j < neg; j++) {
                    const int32_t t = A.negs[lane * NS + j];
                    if (t == A.word) continue;
                    A.flags |= 2u << j;
                    for (int i = 0; i < j; i++)
                        if (A.negs[lane * NS + i] == t) A.flags |= 0x80000000u;
                }
            return;
        }
    };
    // The target rows of centre p of walk W on their way to L2, a lane per row.
    auto prefetch_targets = [&](const CbowWalk &W, uint32_t p) {
        if (p >= W.n || (int)lane > neg) return;
        const int32_t t = lane == 0 ? W.sen[p] : W.negs[p * NS + lane - 1];
        prefetch_l2(a.syn1 + (size_t)t * D, D * 4);
    };
    // Centre p's targets against x, the mean of its context rows: e receives the
    // gradient of x, the target rows their updates (word2vec.cu:453-497).  G rows are
    // read together, after the mean, and their updates sent before the next are read.
    auto train_targets = [&](uint32_t p, const RowVec<VEC> &x, RowVec<VEC> &e) {
        const uint32_t fl = __shfl_sync(kAll, A.flags, p);
#pragma unroll
        for (int g0 = 0; g0 <= NS; g0 += G) {
            if (g0 > neg) break;
            int32_t t[G];   // -1: no target, or one that does not train
            RowVec<VEC> row[G];
#pragma unroll
            for (int k = 0; k < G; k++) {
                const int j = g0 + k;
                t[k] = j == 0 ? A.sen[p] : j <= NS && ((fl >> j) & 1u) ? A.negs[p * NS + j - 1] : -1;
                if (t[k] >= 0) load_row<VEC>(out_row(t[k]), row[k]);
                else zero_row(row[k]);
            }
            if (!(fl & 0x80000000u)) {   // the group's sums and gradients at once
                float f[M];
#pragma unroll
                for (int k = 0; k < M; k++) f[k] = k < G && own ? row_dot(x, row[k < G ? k : 0]) : 0.f;
                const float mine = warp_sums_split<M>(f, lane);
                const float gm = sg_grad(mine, g0 == 0 && lane < GROUP, a.exp_table, a.alpha);
#pragma unroll
                for (int k = 0; k < G; k++) {
                    const float g = __shfl_sync(kAll, gm, k * GROUP);
                    if (t[k] < 0) continue;
                    row_fma(e, g, row[k]);
                    if (own) add_row<VEC>(out_row(t[k]), row_mul(g, x));
                }
            } else {   // a target repeats: one after the other, each seeing the updates before it
#pragma unroll
                for (int k = 0; k < G; k++) {
                    if (t[k] < 0) continue;
                    if (!own) zero_row(row[k]);
                    const float g = sg_grad(warp_dot<VEC>(x, row[k]), g0 + k == 0, a.exp_table, a.alpha);
                    row_fma(e, g, row[k]);
                    const RowVec<VEC> upd = row_mul(g, x);
                    row_add(row[k], upd);
                    if (own) add_row<VEC>(out_row(t[k]), upd);
#pragma unroll
                    for (int q = k + 1; q < G; q++)
                        if (t[q] == t[k]) row[q] = row[k];
                }
            }
        }
    };
    // x / cw, correctly rounded from the rounded reciprocal (Markstein 1990):
    // q = x r, then q + (x - q cw) r; infinities stay as they are.  Padding lanes become 0.
    auto mean = [&](RowVec<VEC> &x, uint32_t window) {
        const float cw = (float)__popc(window), r = __frcp_rn(cw);
#pragma unroll
        for (int i = 0; i < VEC; i++) {
            const float q = x.v[i] * r;
            x.v[i] = !own ? 0.f : fabsf(q) < INFINITY ? fmaf(fmaf(-q, cw, x.v[i]), r, q) : q;
        }
    };

    // Centre p's path against x: the nodes are distinct, so two are read, summed and
    // updated together.
    auto train_path = [&](uint32_t p, const RowVec<VEC> &x, RowVec<VEC> &e) {
        constexpr int H = 2;
        const int32_t word = A.sen[p], k1 = a.hs_off[word + 1];
        for (int32_t k = a.hs_off[word]; k < k1; k += H) {
            int32_t point = -1;
            float label = 0.f;
            if ((int)lane < H && k + (int32_t)lane < k1) {
                point = a.hs_point[k + lane];
                label = (float)(1 - a.hs_code[k + lane]);
            }
            int32_t node[H];
            RowVec<VEC> row[H];
            float f[H];
#pragma unroll
            for (int j = 0; j < H; j++) {
                node[j] = __shfl_sync(kAll, point, j);
                if (node[j] >= 0) load_row<VEC>(out_row(node[j]), row[j]);
                else zero_row(row[j]);
            }
#pragma unroll
            for (int j = 0; j < H; j++) f[j] = own ? row_dot(x, row[j]) : 0.f;
            const float mine = warp_sums_split<H>(f, lane);
            const float lab = __shfl_sync(kAll, label, lane / (32 / H));
            const bool skip = mine <= -kMaxExp || mine >= kMaxExp;
            float gm = 0.f;
            if (!skip)
                gm = (lab - __ldg(a.exp_table + (int)((mine + kMaxExp) * (kExpTableSize / kMaxExp / 2)))) * a.alpha;
            const uint32_t skipped = __ballot_sync(kAll, skip);
#pragma unroll
            for (int j = 0; j < H; j++) {
                const float g = __shfl_sync(kAll, gm, j * (32 / H));
                if (node[j] < 0 || ((skipped >> (j * (32 / H))) & 1u)) continue;
                row_fma(e, g, row[j]);
                if (own) add_row<VEC>(out_row(node[j]), row_mul(g, x));
            }
        }
    };

    for (;;) {
        if (A.p >= A.n) {
            fetch();
            if (A.n == 0 && B.p >= B.n) break;
        }
        if (A.n) {
            const uint32_t p = A.p;
            const uint32_t wp = __shfl_sync(kAll, A.win, p);
            const uint32_t wq = p + 1 < A.n ? __shfl_sync(kAll, A.win, (p + 1) & 31) : 0u;
            const uint32_t all = wp | wq, b0 = ((uint32_t)__ffs(all) - 1) & ~3u;
            if (walks == 1) prefetch_targets(A, p);
            prefetch_targets(A, p + 1);
            prefetch_targets(B, B.p);
            // Context rows of both centres, summed in window order (word2vec.cu:419-428).
            RowVec<VEC> x, y, e;
            zero_row(x);
            zero_row(y);
            for (uint32_t b = b0; b < 32 && (all >> b); b += BATCH) {
                RowVec<VEC> r[BATCH];
#pragma unroll
                for (int h = 0; h < BATCH; h += 4) {
                    if (b + h >= 32) break;
                    const int4 c = *reinterpret_cast<const int4 *>(A.sen + b + h);
                    const int32_t id[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
                    for (int k = 0; k < 4; k++)
                        if ((all >> (b + h + k)) & 1u) load_row<VEC>(syn0 + (size_t)id[k] * D, r[h + k]);
                }
#pragma unroll
                for (int k = 0; k < BATCH; k++) {
                    if (b + k >= 32) break;
                    if ((wp >> (b + k)) & 1u) row_add(x, r[k]);
                    if ((wq >> (b + k)) & 1u) row_add(y, r[k]);
                }
            }
            mean(x, wp);
            zero_row(e);
            if (HS) train_path(p, x, e);
            train_targets(p, x, e);
            if (wq) {
                const int pairs = __reduce_add_sync(kAll, ((wq >> lane) & 1u) ? __popc(A.same & wp) : 0);
                if (pairs) row_fma(y, (float)pairs, e);   // 0 of an infinite e would be no number
                mean(y, wq);
                zero_row(x);   // from here the second centre's e
                if (HS) train_path(p + 1, y, x);
                train_targets(p + 1, y, x);
            }
            // e to every context row (word2vec.cu:498-505), both centres' at once.
            for (uint32_t b = b0; b < 32 && (all >> b); b += 4) {
                const int4 c = *reinterpret_cast<const int4 *>(A.sen + b);
                const int32_t id[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    if (!((all >> (b + k)) & 1u)) continue;
                    RowVec<VEC> s;
                    zero_row(s);
                    if ((wp >> (b + k)) & 1u) s = e;
                    if ((wq >> (b + k)) & 1u) row_add(s, x);
                    if (own) add_row<VEC>(syn0 + (size_t)id[k] * D, s);
                }
            }
            A.p = p + 2;
        }
        if (walks > 1) {
            const CbowWalk t = A;
            A = B;
            B = t;
        }
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) n_pairs += __shfl_xor_sync(kAll, n_pairs, o);
    if (lane == 0) {
        atomicAdd(&a.stats[0], n_words);
        atomicAdd(&a.stats[1], n_trained);
        atomicAdd(&a.stats[2], n_pairs);
    }
}

bool cbow_pair_applies(const dg_sgns *s, const SgnsArgs &a, const WalkSet &ws) {
    return s->p.mode == DG_SGNS_CBOW && !s->p.deterministic && ws.max_len > 0 && ws.max_len <= kCbowMaxTokens &&
           (a.hs ? s->p.size <= 256 : s->p.size == kCbowPairSize) && a.negative <= (a.hs ? kCbowPairHsNeg : kCbowPairNeg) &&
           a.vocab_size > 1;
}

template <int V, bool HS, bool FIXED>
static int cbow_pair_launch(dg_sgns *s, const SgnsArgs &a, const WalkSet &ws) {
    auto kern = sgns_cbow_pair_kernel<V, HS, FIXED>;
    int per_sm = 0;
    DG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 32 * kCbowWarps, 0));
    const PairGrid g = pair_grid(s->p.workers, {std::min(std::max(per_sm, 1), cbow_pair_blocks(V)) * dg::sm_count(s->device),
                                                kCbowWarps, (uint32_t)cbow_pair_walks(V)});
    // The last rows of the table: inner nodes are rows 0 .. vocabulary - 2, the root the last of them.
    const uint32_t n_hot = HS ? std::min(kHotNodes, s->vocab_size) : 0;
    const int32_t hot_from = HS ? (int32_t)(s->vocab_size - n_hot) : 0;
    if (HS) {
        if (s->hs_hot.n == 0) DG_CUDA(s->hs_hot.alloc(kHotFloats));
        cbow_hot_rows<V><<<n_hot, 32, 0, s->stream>>>(s->syn1.p, s->hs_hot.p, hot_from, true);
        dg::note_launch();
    }
    kern<<<g.blocks, 32 * g.warps, 0, s->stream>>>(a, ws, g.walks, s->hs_hot.p, hot_from);
    dg::note_launch();
    if (HS) {
        cbow_hot_rows<V><<<n_hot, 32, 0, s->stream>>>(s->syn1.p, s->hs_hot.p, hot_from, false);
        dg::note_launch();
    }
    DG_CUDA(cudaGetLastError());
    return DG_OK;
}

template <int V>
static int cbow_pair_size(dg_sgns *s, const SgnsArgs &a, const WalkSet &ws) {
    if (a.hs) return cbow_pair_launch<V, true, false>(s, a, ws);
    if constexpr (32 * V == kCbowPairSize)
        return a.negative == kCbowPairNeg ? cbow_pair_launch<V, false, true>(s, a, ws)
                                          : cbow_pair_launch<V, false, false>(s, a, ws);
    return dg::fail(DG_ERR_STATE, "rows of %d columns are not trained two centres at a time", 32 * V);
}

int launch_cbow_pair(dg_sgns *s, const SgnsArgs &a, const WalkSet &ws) {
    switch (s->p.size / 32) {
    case 1: return cbow_pair_size<1>(s, a, ws);
    case 2: return cbow_pair_size<2>(s, a, ws);
    case 4: return cbow_pair_size<4>(s, a, ws);
    default: return cbow_pair_size<8>(s, a, ws);
    }
}

}  // namespace dgs
