// Bucket reduction of the MSM: per window V = sum_k (k + 1) B_k over its
// buckets, weighted by 2^(c w), by binary folding.
//
// With index k = 2i + e the weighted sum folds as
//   sum_k k B_k = 2 sum_i i (B_2i + B_2i+1) + sum_i B_2i+1,
// so after one addition per pair the odd-index points form a plain sum T_0
// and the pair sums R the same problem of half the size.  Over log2(M) levels
//   V = R + sum_j 2^j T_j,   T_j = sum of the B_k whose index has bit j set,
// R the sum of all buckets.  Every T_j folds by halves together with the
// levels after it, so a level of M / 2^(l + 1) pairs is (l + 1) M / 2^(l + 1)
// independent additions: two additions per bucket in all, as a running sum
// has, but log2(M) deep.  In place: element i 2^(l+1) + r (r = 0 for R, 2^j for
// T_j) takes element 2^l further on; the R element passed over becomes T_l.
//
// Additions take four lanes and four product latencies (xyzz_add_quad_pt), or in
// rounds of few additions eight lanes and three (xyzz_add_oct_pt).
//
// What bounds it: with few buckets the latency of its products (about 1 us
// each on one warp), with many the multiply pipe.  Measured against running
// sums per thread with a suffix scan and two trees over each block's threads
// (24 levels deep whatever the number of buckets): 524 K buckets (BLS12-381
// 2^22) 2.04 -> 1.17 ms, 262 K (1000003 points in G1) 1.38 -> 0.88 ms, one window
// of 4096 (KZG commit) 0.36 -> 0.185 ms, 96 uneven commits 9.4 -> 5.9 ms in all.
#pragma once
#include "curve.cuh"
#include "msm_desc.cuh"
#include "runtime.cuh"

namespace kb200 {

// Words of a point slot in shared memory: 4N words and four of padding, so
// that slots keep 16-byte alignment and consecutive ones start four banks
// further on modulo 16.
template <class F>
constexpr int RED_PS = 4 * F::N + 4;

// Shared-memory points of a reduction block: the sub-chunk's buckets (in
// stage 2 the block results of a window), the sub-chunk totals, the T_j sums
// over sub-chunks, and the final points.
constexpr int RED_SUB_MAX = 1 << RED_LOGQ_MAX;
constexpr int RED_LOOP_MAX = 1 << RED_LOGL_MAX;
constexpr int RED_TREE = RED_SUB_MAX + RED_LOOP_MAX + RED_PTS;
constexpr int RED_FINAL = 32;
// Additions of a round that get eight lanes each: one warp per scheduler.
constexpr uint32_t RED_OCTS = RED_THREADS / 16;

// One quad copies a point of 4N words, a coordinate per lane.
template <class F>
KB_DEV void quad_copy(uint32_t* dst, const uint32_t* src) {
    const int ql = threadIdx.x & 3;
    ld_st_words16<F::N>(dst + ql * F::N, src + ql * F::N);
}
template <class F>
KB_DEV void quad_set_inf(uint32_t* dst) {
    uint4* d = reinterpret_cast<uint4*>(dst + (threadIdx.x & 3) * F::N);
#pragma unroll
    for (int k = 0; k < F::N / 4; ++k) d[k] = make_uint4(0, 0, 0, 0);
}

// A bucket whose sum lies in several chunk records: the sub-chunk slot it is
// summed in, the records after the first, and the index of the next one.
struct RedPieces {
    uint32_t slot, extra, next;
};

// dst = the first piece of B_g (see k_accumulate for where each piece lives); one
// quad.  Buckets with more pieces go to the list, and only when the whole
// sub-chunk is loaded do quads add those: with the additions here, a warp whose
// eight buckets have one further piece among them ran an addition for all
// eight (about 0.3 records past the first per bucket cost one addition: 524 K buckets
// 1.50 -> 1.32 ms, 24 windows of 2048 in 100003 points 1.07 -> 0.94 ms).
template <class F>
KB_DEV void quad_load_bucket(uint32_t* dst, const RedArgs& a, uint32_t g, uint32_t slot, RedPieces* list,
                             uint32_t* listed) {
    constexpr int PW = 4 * F::N;
    const uint32_t o = a.offsets[g], c = a.offsets[g + 1] - o;
    if (c == 0) {
        quad_set_inf<F>(dst);
        return;
    }
    const uint32_t t0 = o / a.K, t1 = (o + c - 1) / a.K;
    const uint32_t* first;
    if (t0 == t1) {
        const uint32_t e0 = t0 * a.K, e1 = min(e0 + a.K, a.offsets[a.B]);
        first = (o == e0) ? a.rec_first + (size_t)t0 * PW
                : (o + c == e1) ? a.rec_last + (size_t)t0 * PW
                                : a.buckets + (size_t)g * PW;
    } else {
        first = ((o == t0 * a.K) ? a.rec_first : a.rec_last) + (size_t)t0 * PW;
        // a big bucket's records t0+1..t1 were folded into rec_first[t0+1]
        if ((threadIdx.x & 3) == 0)
            list[atomicAdd(listed, 1u)] = RedPieces{slot, t1 - t0 > (uint32_t)a.K2 ? 1u : t1 - t0, t0 + 1};
    }
    quad_copy<F>(dst, first);
}

// Two points of shared memory to add, the sum in dst.
struct RedPair {
    uint32_t *dst, *src;
};

// Task t of folding level l over elements x: the (l + 1) 2^(n - l - 1) pairs
// of one weighted fold of 2^n elements (see the head of this file).
template <class F>
KB_DEV RedPair fold_task(uint32_t* x, int l, uint32_t t) {
    const uint32_t i = t / (uint32_t)(l + 1), r = t - i * (uint32_t)(l + 1);
    const uint32_t lo = (i << (l + 1)) + (r ? 1u << (r - 1) : 0u);
    return {x + (size_t)lo * RED_PS<F>, x + (size_t)(lo + (1u << l)) * RED_PS<F>};
}

// A block's round of n independent additions, task(t) the pair of the t-th: eight
// lanes each up to octs additions, else four.
template <class F, class Task>
KB_DEV void add_round(uint32_t n, uint32_t octs, const Task& task) {
    if (n <= octs) {
        const uint32_t oct = threadIdx.x >> 3;
        if (oct < n) {
            const RedPair p = task(oct);
            xyzz_add_oct_pt<F>(p.dst, p.src);
        }
    } else {
        for (uint32_t t = threadIdx.x >> 2; t < n; t += RED_QUADS) {
            const RedPair p = task(t);
            xyzz_add_quad_pt<F>(p.dst, p.src);
        }
    }
    __syncthreads();
}

// The results of nb <= 2^ln consecutive blocks (every stride-th slot from out0 on,
// T_j of lb index bits each) folded over the block index: afterwards x[0] is
// their total, x[2^i] the T of block index bit i, and y[j 2^lg] (y behind the
// 2^ln slots of x; returns 2^lg slots per T_j, as many as fit) the sum of their
// T_j.  The blocks' results are read after the fence that ordered their
// stores before their completion count.
template <class F>
__device__ __noinline__ int reduce_blocks(uint32_t* x, const uint32_t* out0, uint32_t nb, uint32_t stride,
                                          int lb, int ln) {
    constexpr int PW = 4 * F::N, PS = RED_PS<F>;
    const uint32_t quad = threadIdx.x >> 2;
    const uint32_t NB = 1u << ln;
    const size_t step = (size_t)stride * RED_PTS * PW;
    int lg = 0;
    while (lg < ln && (((size_t)lb << (lg + 1)) + NB) <= (size_t)RED_TREE) ++lg;
    uint32_t* y = x + (size_t)NB * PS;
    const uint32_t cols = (uint32_t)lb << lg;
    for (uint32_t t = quad; t < NB + cols; t += RED_QUADS) {
        if (t < cols) {
            const uint32_t j = t >> lg, s = t & ((1u << lg) - 1);
            uint32_t* dst = y + (size_t)t * PS;
            if (s >= nb) {
                quad_set_inf<F>(dst);
                continue;
            }
            quad_copy<F>(dst, out0 + s * step + (1 + j) * PW);
            __syncwarp(0xFu << (threadIdx.x & 28));
            for (uint32_t b = s + (1u << lg); b < nb; b += 1u << lg)
                xyzz_add_quad_pt<F>(dst, out0 + b * step + (1 + j) * PW);
        } else {
            const uint32_t b = t - cols;
            uint32_t* dst = x + (size_t)b * PS;
            if (b < nb)
                quad_copy<F>(dst, out0 + b * step);
            else
                quad_set_inf<F>(dst);
        }
    }
    __syncthreads();
    for (int l = 0; l < ln; ++l) {
        const uint32_t nr = (uint32_t)(l + 1) << (ln - l - 1);
        const uint32_t half = l < lg ? 1u << (lg - l - 1) : 0u;
        const uint32_t nt = (uint32_t)lb * half;
        add_round<F>(nr + nt, RED_OCTS, [&](uint32_t t) -> RedPair {
            if (t < nr) return fold_task<F>(x, l, t);
            const uint32_t j = (t - nr) / half, s = (t - nr) - j * half;
            uint32_t* p = y + (((size_t)j << lg) + s) * PS;
            return {p, p + (size_t)half * PS};
        });
    }
    return lg;
}

// One group's blocks, by the block that finished it last: their results become
// one block's with three more T_j, in the group's first slot.
template <class F>
__device__ __noinline__ void reduce_group(uint32_t* out0, uint32_t nb, int lb, uint32_t* x) {
    constexpr int PW = 4 * F::N, PS = RED_PS<F>;
    constexpr int LN = RED_LOG_GROUP;
    const int lg = reduce_blocks<F>(x, out0, nb, 1, lb, LN);
    const uint32_t* y = x + ((size_t)PS << LN);
    const uint32_t quad = threadIdx.x >> 2;
    if (quad == 0)
        quad_copy<F>(out0, x);
    else if (quad <= (uint32_t)lb)
        quad_copy<F>(out0 + (size_t)quad * PW, y + (((size_t)quad - 1) << lg) * PS);
    else if (quad <= (uint32_t)(lb + LN))
        quad_copy<F>(out0 + (size_t)quad * PW, x + ((size_t)1 << (quad - 1 - lb)) * PS);
}

// Stage 2 of window w, by the block that finished it last: its blocks' (or its
// groups') results folded over their index, then 2^(shift + j) on every T_j and
// 2^shift on the total (all doubling chains at once, four to a warp), and the
// sum of those points.
template <class C>
__device__ __noinline__ void reduce_window(const RedArgs& a, uint32_t w, bool grouped, uint32_t* sm) {
    using F = typename C::F;
    constexpr int PW = 4 * F::N, PS = RED_PS<F>;
    const WinDesc wd = a.wins[w];
    const uint32_t quad = threadIdx.x >> 2;
    uint32_t* x = sm;
    uint32_t* z = sm + (size_t)RED_TREE * PS;
    const int gl = grouped ? RED_LOG_GROUP : 0;
    const int lb = (int)(wd.log_q + wd.log_l) + gl;  // T_j of one block or group
    const uint32_t nb = (wd.nb + (1u << gl) - 1) >> gl;
    int ln = 0;
    while ((1u << ln) < nb) ++ln;
    const int lg = reduce_blocks<F>(x, a.blk_out + (size_t)wd.blk_base * RED_PTS * PW, nb, 1u << gl, lb, ln);
    const uint32_t* y = x + ((size_t)PS << ln);
    // final points: 0 the total (weight 2^shift), 1 + j the T_j (2^(shift + j))
    const uint32_t np = (uint32_t)(1 + lb + ln);
    if (quad < RED_FINAL) {
        uint32_t* dst = z + (size_t)quad * PS;
        if (quad == 0)
            quad_copy<F>(dst, x);
        else if (quad <= (uint32_t)lb)
            quad_copy<F>(dst, y + (((size_t)quad - 1) << lg) * PS);
        else if (quad < np)
            quad_copy<F>(dst, x + ((size_t)1 << (quad - 1 - lb)) * PS);
        else
            quad_set_inf<F>(dst);
    }
    __syncthreads();
    {
        const uint32_t idx = threadIdx.x >> 3;  // eight lanes per chain
        uint32_t* p = z + (size_t)idx * PS;
        const uint32_t k = (idx < np && !point_is_inf<F>(p)) ? wd.shift + (idx ? idx - 1 : 0u) : 0u;
        xyzz_dbl_chain_oct<F>(p, k, x + (size_t)idx * 8 * F::N);
    }
    __syncthreads();
    for (uint32_t d = np > 16 ? 16 : 8; d >= 1; d >>= 1)
        add_round<F>(d, RED_OCTS, [&](uint32_t t) -> RedPair {
            return {z + (size_t)t * PS, z + (size_t)(t + d) * PS};
        });
    if (quad == 0) quad_copy<F>(a.win_out + (size_t)w * PW, z);
}

// One block per blk = 2^(log_q + log_l) consecutive buckets of a window,
// as 2^log_l sub-chunks of 2^log_q.  Writes the block's total and its T_j;
// the block that completes its window's count runs the window's stage 2 at
// once, so the windows' doubling chains (the longest first: blocks run top
// window first) overlap the remaining blocks instead of following them.  No
// block waits for another.  win_done holds one zeroed counter per window,
// grp_done one per block.
//
// From RED_GROUPED blocks a window on, stage 2 is a tree as well: the last block
// of eight folds their results first, on as many SMs as there are groups.  One
// SM alone summed 64 blocks' T_j in about 11 rounds of quad additions, 128 blocks'
// in 27; groups and window now take 8 and 10.  Reductions: 16 windows of 32768
// buckets 1.38 -> 1.22 ms, 8 (1000003 points in G1) 1.00 -> 0.90, 2^21 skewed
// BN254 points 0.45 -> 0.35, one window of 4096 0.244 -> 0.229.  From 16 blocks
// on it measured the same.
template <class C>
__global__ void __launch_bounds__(RED_THREADS, 2) k_reduce(RedArgs a) {
    using F = typename C::F;
    constexpr int PW = 4 * F::N, PS = RED_PS<F>;
    extern __shared__ __align__(16) uint32_t smr[];
    __shared__ uint32_t s_last, s_listed;
    __shared__ RedPieces s_list[RED_SUB_MAX];
    uint32_t* x = smr;                                  // the sub-chunk's buckets
    uint32_t* rs = x + (size_t)RED_SUB_MAX * PS;        // sub-chunk totals
    uint32_t* at = rs + (size_t)RED_LOOP_MAX * PS;      // T_j over the sub-chunks so far
    const uint32_t bi = gridDim.x - 1u - blockIdx.x;    // top window first
    const BlkDesc bd = a.blks[bi];
    const WinDesc wd = a.wins[bd.win];
    const uint32_t quad = threadIdx.x >> 2;
    const int lq = (int)wd.log_q, ll = (int)wd.log_l;
    // eight lanes an addition cost half as much again of the multiply pipe: only
    // where all blocks run at once (100003 points, 768 blocks: 2505 us with quads
    // in the blocks, 2560 with eight lanes)
    const uint32_t octs = a.one_wave ? RED_OCTS : 0u;
    for (uint32_t it = 0; it < (1u << ll); ++it) {
        const uint32_t first = bd.b * wd.blk + (it << lq);
        if (threadIdx.x == 0) s_listed = 0;
        __syncthreads();
        for (uint32_t s = quad; s < (1u << lq); s += RED_QUADS) {
            if (first + s < wd.Mw)
                quad_load_bucket<F>(x + (size_t)s * PS, a, wd.bucket_base + first + s, s, s_list, &s_listed);
            else
                quad_set_inf<F>(x + (size_t)s * PS);
        }
        __syncthreads();
        for (uint32_t t = quad; t < s_listed; t += RED_QUADS) {
            const RedPieces p = s_list[t];
            for (uint32_t k = 0; k < p.extra; ++k)
                xyzz_add_quad_pt<F>(x + (size_t)p.slot * PS, a.rec_first + (size_t)(p.next + k) * PW);
        }
        __syncthreads();
        for (int l = 0; l < lq; ++l) {
            add_round<F>((uint32_t)(l + 1) << (lq - l - 1), octs, [&](uint32_t t) { return fold_task<F>(x, l, t); });
        }
        if (ll > 0) {
            if (quad < (uint32_t)lq) {
                if (it == 0)
                    quad_copy<F>(at + (size_t)quad * PS, x + ((size_t)1 << quad) * PS);
                else
                    xyzz_add_quad_pt<F>(at + (size_t)quad * PS, x + ((size_t)1 << quad) * PS);
            } else if (quad == (uint32_t)lq) {
                quad_copy<F>(rs + (size_t)it * PS, x);
            }
            __syncthreads();
        }
    }
    for (int l = 0; l < ll; ++l) {
        add_round<F>((uint32_t)(l + 1) << (ll - l - 1), octs, [&](uint32_t t) { return fold_task<F>(rs, l, t); });
    }
    const uint32_t* tot = ll > 0 ? rs : x;
    uint32_t* out = a.blk_out + (size_t)bi * RED_PTS * PW;
    if (quad == 0)
        quad_copy<F>(out, tot);
    else if (quad <= (uint32_t)lq)
        quad_copy<F>(out + (size_t)quad * PW,
                     ll > 0 ? at + (size_t)(quad - 1) * PS : x + ((size_t)1 << (quad - 1)) * PS);
    else if (quad <= (uint32_t)(lq + ll))
        quad_copy<F>(out + (size_t)quad * PW, rs + ((size_t)1 << (quad - 1 - lq)) * PS);
    // counts are taken after the results they announce
    auto last_of = [&](uint32_t* count, uint32_t n) {
        __threadfence();
        __syncthreads();
        if (threadIdx.x == 0) {
            s_last = atomicAdd(count, 1u) + 1u == n;
            __threadfence();
        }
        __syncthreads();
        return s_last != 0;
    };
    const bool grouped = wd.nb >= RED_GROUPED && lq + ll + RED_LOG_GROUP < RED_PTS;
    uint32_t n = wd.nb;
    if (grouped) {
        constexpr uint32_t G = 1u << RED_LOG_GROUP;
        const uint32_t in_group = bd.b % G, size = min(G, n - (bd.b - in_group));
        if (!last_of(a.grp_done + (bi - in_group), size)) return;
        reduce_group<F>(out - (size_t)in_group * RED_PTS * PW, size, lq + ll, smr);
        n = (n + G - 1) / G;
    }
    if (last_of(a.win_done + bd.win, n)) reduce_window<C>(a, bd.win, grouped, smr);
}

// Fold level l >= 2: the level's (big bucket, group) items are flattened by
// the prefix of group counts; one block per item.  Group q of bucket g sums
// FK consecutive items of its previous level (records rec_first[t0+1 ..] at
// level 2), a quad per FOLD_QUADS-th record and a tree over the quads; the
// level that reaches one group writes the bucket's total to rec_first[t0 + 1].
// Bound by latency: two to seven quad additions deep for up to FK = 64 records,
// against three serial additions a level of four before (a KZG commit's
// fold 0.155 -> 0.052 ms, 2^21 skewed BN254 points 0.22 -> 0.08 ms).
constexpr int FOLD_THREADS = 128, FOLD_QUADS = FOLD_THREADS / 4;

template <class C>
__global__ void __launch_bounds__(FOLD_THREADS) k_fold(FoldArgs a, int level,
                                                       const uint32_t* __restrict__ in,
                                                       uint32_t* __restrict__ out) {
    using F = typename C::F;
    constexpr int PW = 4 * F::N, PS = RED_PS<F>;
    __shared__ __align__(16) uint32_t s[FOLD_QUADS * PS];
    const uint32_t base = a.prefix[0];  // the level's slice of the all-levels scan
    const uint32_t total = a.prefix[a.big_cap] - base;
    const uint32_t quad = threadIdx.x >> 2;
    for (uint32_t i = blockIdx.x; i < total; i += gridDim.x) {
        uint32_t lo_k = 0, hi_k = a.big_cap;  // largest k with prefix[k] - base <= i
        while (hi_k - lo_k > 1) {
            const uint32_t mid = (lo_k + hi_k) >> 1;
            if (a.prefix[mid] - base <= i)
                lo_k = mid;
            else
                hi_k = mid;
        }
        const uint32_t g = a.big_list[1 + lo_k];
        const uint32_t q = i - (a.prefix[lo_k] - base);
        const uint32_t o = a.offsets[g], c = a.offsets[g + 1] - o;
        uint32_t t0, n_prev, n_cur;
        fold_sizes(o, c, a.K, a.FK, level, t0, n_prev, n_cur);
        const uint32_t lo = q * (uint32_t)a.FK, hi = min(lo + (uint32_t)a.FK, n_prev);
        const uint32_t* src = in + (size_t)(t0 + 1) * PW;
        uint32_t* mine = s + (size_t)quad * PS;
        if (lo + quad < hi) {
            quad_copy<F>(mine, src + (size_t)(lo + quad) * PW);
            __syncwarp(0xFu << (threadIdx.x & 28));
            for (uint32_t j = lo + quad + FOLD_QUADS; j < hi; j += FOLD_QUADS)
                xyzz_add_quad_pt<F>(mine, src + (size_t)j * PW);
        } else {
            quad_set_inf<F>(mine);
        }
        __syncthreads();
        for (uint32_t d = FOLD_QUADS / 2; d >= 1; d >>= 1) {
            if (quad < d && lo + quad + d < hi) xyzz_add_quad_pt<F>(mine, mine + (size_t)d * PS);
            __syncthreads();
        }
        if (quad == 0) quad_copy<F>((n_cur == 1 ? a.rec_first : out) + (size_t)(t0 + 1 + q) * PW, s);
        __syncthreads();
    }
}

}  // namespace kb200
