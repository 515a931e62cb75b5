// Hogwild shared-negative skip-gram on FP32 rows (__sgNegReuse, word2vec.cu:231-303),
// two pairs at a time: the form of DG_SGNS_SG_SHARED that trains walks of at most
// 64 tokens with rows of 256 columns (sizes 129 to 256) and four or five negatives
// (sgns_negshare_kernel, dg_sgns_w2v.cu, trains the others and the deterministic
// runs).
//
// What bounds the rule is the L2's reduction rate (5.9 TB/s of 512-byte rows on a
// B200, against 18.1 TB/s of reads; the two times add up): a walk's negatives stay
// in L2, and each pair read and updated n + 1 rows there.  A walk's pairs share
// the negatives, so here a warp reads them once for two pairs of a centre, lets
// the second pair see the first one's update in registers, and sends the sum of
// both: n + 2 rows for two pairs instead of 2 n + 2.  Padding columns (size 200 in
// rows of 256) are not moved.
//
// A Hogwild run's rows depend on how many pairs are under way unseen and on how
// many walks are trained at once, so half as many warps as sgns_negshare_kernel's
// hold two walks each and train two pairs of either in turn.
//
// A round of the 50,000-vertex graph at size 200, window 5, negative 5, with its
// read-back: 21.2 -> 11.9 ms.  What bounds it now: the L2's reductions, 4.8 TB/s of them,
// for a lane's eight columns are two 16-byte atomics and each sector is reduced twice.
//
// Why 256 columns and four or five negatives.  Each negative row is read once for two
// pairs, so it misses the updates of more pairs of other walks.  Over the distance of two
// equal runs of the one-pair kernel from each other (graphs of 10,000 to 200,000
// vertices), rows of 256 columns with four or five negatives end 1.0 to 1.6 times as far
// from that kernel's after one pass and 1.4 to 2.7 times after two (its own runs: 1.3 to
// 2.5).  With three they are up to 2.0 and 2.7 times as far, with seven and eight up to
// 1.9.  At 64 and 128 columns, where that kernel has 32 warps an SM and not 16, it is up to
// 3.0 (64 columns, seven negatives), and single values of the output rows end up to 11
// times further off than its own runs show, on graphs of 10,000 to 16,000 vertices above
// all.  Below three there is little to share: one negative takes 3.9 ms against 3.3
// (40,000 vertices, size 64), two 10.6 against 10.7 (120,000, size 128).
#include "dg_pair_grid.h"
#include "dg_sgns.h"
#include "dg_sgns_dev.cuh"

namespace dgs {

constexpr int kShareWarps = 8;             // warps of a block
constexpr uint32_t kShareTokens = 64;      // the longest walk of this kernel
constexpr int kShareLeastNeg = 4;          // the negative counts of this kernel
constexpr int kShareMostNeg = 5;
constexpr int kShareSize = 256;            // the row of this kernel, kShareVec columns to a lane
constexpr int kShareVec = kShareSize / 32;

// A walk under way: its length, centre and the centre's next pair, its words and
// negatives (shared), whether a negative occurs twice, and this lane's columns of
// the centre's output row, as it was read and as it is between turns (shared).
struct ShareWalk {
    uint32_t n = 0, p = 0, k = 0;
    int32_t *sen = nullptr, *negs = nullptr;
    float *pos0 = nullptr, *pos = nullptr;
    bool repeat = false;
};

__device__ __forceinline__ void share_put(float *p, const RowVec<kShareVec> &r) {
#pragma unroll
    for (int i = 0; i < kShareVec; i += 4)
        *reinterpret_cast<float4 *>(p + i) = make_float4(r.v[i], r.v[i + 1], r.v[i + 2], r.v[i + 3]);
}
__device__ __forceinline__ void share_get(const float *p, RowVec<kShareVec> &r) {
#pragma unroll
    for (int i = 0; i < kShareVec; i += 4) {
        const float4 q = *reinterpret_cast<const float4 *>(p + i);
        r.v[i] = q.x; r.v[i + 1] = q.y; r.v[i + 2] = q.z; r.v[i + 3] = q.w;
    }
}

// Lane l owns columns [l * VEC, l * VEC + VEC) of every row.  FIXED: NS negatives
// (word2vec's default), else up to NS, read from a.negative.  One block to an SM.
template <bool FIXED>
__global__ void __launch_bounds__(kShareWarps * 32, 1)
    sgns_negshare_pair_kernel(SgnsArgs a, WalkSet ws, uint32_t walks) {
    constexpr int VEC = kShareVec, NS = kShareMostNeg, D = kShareSize, M = pow2_at_least(NS + 1), GROUP = 32 / M;
    constexpr uint32_t kAll = 0xffffffffu;
    __shared__ int32_t sen_all[kShareWarps][2][kShareTokens];
    __shared__ int32_t negs_all[kShareWarps][2][NS];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int neg = FIXED ? NS : a.negative;
    const uint32_t w = (uint32_t)a.window;
    // Lanes whose columns are all padding read and write nothing: every row, sum and
    // update that they hold is 0.
    const bool own = lane * VEC < (uint32_t)a.used;
    float *const syn0 = a.syn0 + lane * VEC, *const syn1 = a.syn1 + lane * VEC;
    unsigned long long n_words = 0, n_trained = 0, n_pairs = 0;
    ShareWalk A, B;
    extern __shared__ __align__(16) float share_smem[];   // per walk the centre's row, twice
    float *const rows = share_smem + (size_t)warp * 4 * D + lane * VEC;
    A.sen = sen_all[warp][0];
    A.negs = negs_all[warp][0];
    A.pos0 = rows;
    A.pos = rows + D;
    B.sen = sen_all[warp][1];
    B.negs = negs_all[warp][1];
    B.pos0 = rows + 2 * D;
    B.pos = rows + 3 * D;
    bool more = true;

    auto fetch = [&]() {   // the next walk of at least two tokens into A; A.n = 0 when there is none left
        A.n = A.p = A.k = 0;
        while (more) {
            uint32_t walk = 0;
            if (lane == 0) walk = atomicAdd(a.queue, 1u);
            walk = __shfl_sync(kAll, walk, 0);
            more = walk < ws.n_walks;
            if (!more) return;
            const uint32_t wid = ws.ids ? ws.ids[walk] : walk + ws.id_base;
            uint32_t words;
            __syncwarp();
            const uint32_t n = warp_sentence<kShareTokens>(ws, walk, a, A.sen, words);
            n_words += words;
            n_trained += n;
            if (n < 2) continue;
            A.n = n;
            int32_t t = -1 - (int32_t)lane;
            if ((int)lane < neg) A.negs[lane] = t = tagged_negative(a, 0, wid, kShareTag, (int)lane);
            const uint32_t same = __match_any_sync(kAll, t);
            A.repeat = __any_sync(kAll, (same & (same - 1)) != 0u);
            __syncwarp();
            return;
        }
    };
    auto load = [&](const float *table, int32_t word, RowVec<VEC> &r) {
        zero_row(r);
        if (own) load_row<VEC>(table + (size_t)word * D, r);
    };

    for (;;) {
        if (A.p >= A.n) {
            fetch();
            if (A.n == 0 && B.p >= B.n) break;
        }
        if (A.n) {
            const uint32_t p = A.p, n = A.n;
            const int32_t word = A.sen[p];
            RowVec<VEC> pos;
            if (A.k == 0) {
                load(syn1, word, pos);
                share_put(A.pos0, pos);
            } else {
                share_get(A.pos, pos);
            }
            int32_t t[NS];
            uint32_t live = 0;   // bit j: negative j trains (it is not the centre's word)
#pragma unroll
            for (int j = 0; j < NS; j++) {
                t[j] = j < neg ? A.negs[j] : word;
                if (j < neg && t[j] != word) live |= 1u << j;
            }
            const uint32_t lo = p > w ? p - w : 0u, hi = min(n, p + w + 1);   // positions; p itself is no context
            const uint32_t m = hi - lo - 1;
            auto at = [&](uint32_t k) { return A.sen[lo + k + (lo + k >= p ? 1u : 0u)]; };
            // The gradients of the pair (l, centre): lane group j holds negative j's, group neg's the
            // positive's; all sums are of the rows as they are.
            auto gradients = [&](const RowVec<VEC> &l, const RowVec<VEC> (&row)[NS]) {
                float f[M];
#pragma unroll
                for (int j = 0; j < M; j++) f[j] = j < NS ? row_dot(l, row[j < NS ? j : 0]) : j == NS ? row_dot(l, pos) : 0.f;
                const float mine = warp_sums_split<M>(f, lane);
                const uint32_t jm = lane / GROUP;
                float g = 0.f;
                if (jm == (uint32_t)NS || ((live >> jm) & 1u)) g = sg_grad(mine, jm == (uint32_t)NS, a.exp_table, a.alpha);
                return g;
            };
            const uint32_t k = A.k;   // this turn's pairs: k and, where there is one, k + 1
            n_pairs += min(2u, m - k);
            if (!A.repeat) {
                {
                    const bool two = k + 1 < m;
                    const int32_t w1 = at(k), w2 = two ? at(k + 1) : w1;
                    RowVec<VEC> l1, l2, e, row[NS];
                    load(syn0, w1, l1);
                    load(syn0, w2, l2);
#pragma unroll
                    for (int j = 0; j < NS; j++)
                        if (j < neg) load(syn1, t[j], row[j]);
                        else zero_row(row[j]);
                    const float ga = gradients(l1, row);
                    zero_row(e);
#pragma unroll
                    for (int j = 0; j < NS; j++) {
                        const float g = __shfl_sync(kAll, ga, j * GROUP);
                        if (!((live >> j) & 1u)) continue;
                        row_fma(e, g, row[j]);
                        if (two) row_fma(row[j], g, l1);
                    }
                    {
                        const float g = __shfl_sync(kAll, ga, NS * GROUP);
                        row_fma(e, g, pos);
                        row_fma(pos, g, l1);
                    }
                    if (own) add_row<VEC>(syn0 + (size_t)w1 * D, e);
                    float gb = 0.f;
                    if (two) {
                        if (w2 == w1) row_add(l2, e);   // one word twice: the second pair sees the first one's update
                        gb = gradients(l2, row);
                        zero_row(e);
#pragma unroll
                        for (int j = 0; j < NS; j++) {
                            const float g = __shfl_sync(kAll, gb, j * GROUP);
                            if ((live >> j) & 1u) row_fma(e, g, row[j]);
                        }
                        const float g = __shfl_sync(kAll, gb, NS * GROUP);
                        row_fma(e, g, pos);
                        row_fma(pos, g, l2);
                        if (own) add_row<VEC>(syn0 + (size_t)w2 * D, e);
                    }
#pragma unroll
                    for (int j = 0; j < NS; j++) {
                        const float g1 = __shfl_sync(kAll, ga, j * GROUP), g2 = __shfl_sync(kAll, gb, j * GROUP);
                        if (!((live >> j) & 1u)) continue;
                        RowVec<VEC> upd = row_mul(g1, l1);
                        if (two) row_fma(upd, g2, l2);
                        if (own) add_row<VEC>(syn1 + (size_t)t[j] * D, upd);
                    }
                }
            } else {   // a negative occurs twice: one target after the other
                for (uint32_t c = k; c < min(k + 2, m); c++) {
                    const int32_t w1 = at(c);
                    RowVec<VEC> l1, e;
                    load(syn0, w1, l1);
                    zero_row(e);
                    for (int j = 0; j < neg; j++) {
                        const int32_t tj = A.negs[j];
                        if (tj == word) continue;
                        RowVec<VEC> row;
                        load(syn1, tj, row);
                        const float g = sg_grad(warp_dot<VEC>(l1, row), 0, a.exp_table, a.alpha);
                        row_fma(e, g, row);
                        if (own) add_row<VEC>(syn1 + (size_t)tj * D, row_mul(g, l1));
                    }
                    const float g = sg_grad(warp_dot<VEC>(l1, pos), 1, a.exp_table, a.alpha);
                    row_fma(e, g, pos);
                    row_fma(pos, g, l1);
                    if (own) add_row<VEC>(syn0 + (size_t)w1 * D, e);
                }
            }
            A.k = k + 2;
            if (A.k < m) {
                share_put(A.pos, pos);
            } else {   // the centre is done
                RowVec<VEC> was;
                share_get(A.pos0, was);
#pragma unroll
                for (int i = 0; i < VEC; i++) pos.v[i] -= was.v[i];
                if (own) add_row<VEC>(syn1 + (size_t)word * D, pos);
                A.p = p + 1;
                A.k = 0;
            }
        }
        if (walks > 1) {
            const ShareWalk x = A;
            A = B;
            B = x;
        }
    }
    if (lane == 0) {
        atomicAdd(&a.stats[0], n_words);
        atomicAdd(&a.stats[1], n_trained);
        atomicAdd(&a.stats[2], n_pairs);
    }
}

bool negshare_pair_applies(const dg_sgns *s, const SgnsArgs &a, const WalkSet &ws) {
    return !s->p.deterministic && ws.max_len > 0 && ws.max_len <= kShareTokens && s->p.size == kShareSize &&
           a.negative >= kShareLeastNeg && a.negative <= kShareMostNeg && a.vocab_size > 1;
}

template <bool FIXED>
static int negshare_pair_launch(dg_sgns *s, const SgnsArgs &a, const WalkSet &ws) {
    auto kern = sgns_negshare_pair_kernel<FIXED>;
    const size_t smem = (size_t)kShareWarps * 4 * kShareSize * sizeof(float);
    DG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const PairGrid g = pair_grid(s->p.workers, {dg::sm_count(s->device), kShareWarps, 2});
    kern<<<g.blocks, 32 * g.warps, smem / kShareWarps * g.warps, s->stream>>>(a, ws, g.walks);
    dg::note_launch();
    DG_CUDA(cudaGetLastError());
    return DG_OK;
}

int launch_negshare_pair(dg_sgns *s, const SgnsArgs &a, const WalkSet &ws) {
    return a.negative == kShareMostNeg ? negshare_pair_launch<true>(s, a, ws) : negshare_pair_launch<false>(s, a, ws);
}

}  // namespace dgs
