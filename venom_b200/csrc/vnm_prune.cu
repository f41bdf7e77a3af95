// Magnitude pruner to the V:2:m pattern (CUDA).
//
// Follows group_n_m2 of the reference (end2end/grouped_nmv_tensor.py:81-343, driver :746-779): for every
// V x m block all C(m,4) column quadruples are scored in lexicographic order; the score of a quadruple is
// the fp32 sum, accumulated row by row (largest first, then second largest), of the two largest |w| among
// its four columns; the first quadruple with the strictly largest score wins (a block whose best score is
// not > 0 keeps nothing and gets columns {0,0,0,0}).  Inside every row of the winner the two largest
// entries are kept.
//
// The result is bit-identical to the reference except in one corner: when the second and third largest |w| of a row of the
// winning quadruple are exactly equal, the reference's choice depends on scratch state left by all earlier blocks; here such
// a tie keeps the entries a freshly initialised partial sort would keep.  Scores, and therefore the chosen columns, never
// depend on ties.
#include "vnm_internal.h"

namespace vnm {

namespace {

enum : int { W_F32 = 0, W_F16 = 1 };   // type of the weights

__device__ __forceinline__ long long binom4(int n)  // C(n,4), n >= 0
{
    return n < 4 ? 0 : (long long)n * (n - 1) * (n - 2) * (n - 3) / 24;
}
__device__ __forceinline__ int binom3(int n) { return n < 3 ? 0 : n * (n - 1) * (n - 2) / 6; }
__device__ __forceinline__ int binom2(int n) { return n < 2 ? 0 : n * (n - 1) / 2; }

// idx-th 4-subset of {0..m-1} in lexicographic order.
__device__ __forceinline__ void unrank4(int idx, int m, int c[4])
{
    int a = 0;
    for (;; ++a) {
        const int cnt = binom3(m - 1 - a);  // quadruples starting with a
        if (idx < cnt) break;
        idx -= cnt;
    }
    int b = a + 1;
    for (;; ++b) {
        const int cnt = binom2(m - 1 - b);
        if (idx < cnt) break;
        idx -= cnt;
    }
    int cc = b + 1;
    for (;; ++cc) {
        const int cnt = m - 1 - cc;
        if (idx < cnt) break;
        idx -= cnt;
    }
    c[0] = a; c[1] = b; c[2] = cc; c[3] = cc + 1 + idx;
}

// std::partial_sort(idx, idx+2, idx+4, v[A] > v[B]) on a fresh idx = {0,1,2,3} (libstdc++ heap select).
__device__ __forceinline__ void top2_of4(const float v[4], int &i0, int &i1)
{
    int idx[4] = {0, 1, 2, 3};
    if (!(v[idx[1]] > v[idx[0]])) { int t = idx[0]; idx[0] = idx[1]; idx[1] = t; }
#pragma unroll
    for (int i = 2; i < 4; i++) {
        if (v[idx[i]] > v[idx[0]]) {
            const int value = idx[i];
            idx[i] = idx[0];
            idx[0] = idx[1];
            if (v[idx[0]] > v[value]) { idx[1] = idx[0]; idx[0] = value; }
            else idx[1] = value;
        }
    }
    i0 = idx[1];  // after sort_heap: largest first
    i1 = idx[0];
}

// The reference's score of one quadruple: an fp32 sum in row order, the larger magnitude of a row first.
__device__ __forceinline__ float exact_score(const float *tile, int pitch, int V, const int c[4])
{
    float total = 0.0f;
    for (int r = 0; r < V; r++) {
        const float *row = tile + r * pitch;
        const float v0 = fabsf(row[c[0]]), v1 = fabsf(row[c[1]]), v2 = fabsf(row[c[2]]), v3 = fabsf(row[c[3]]);
        const float hi01 = fmaxf(v0, v1), lo01 = fminf(v0, v1), hi23 = fmaxf(v2, v3), lo23 = fminf(v2, v3);
        total += fmaxf(hi01, hi23);
        total += fmaxf(fminf(hi01, hi23), fmaxf(lo01, lo23));
    }
    return total;
}

// ------------------------------------------------------------------------------------------------
// Pruner by candidates (m <= PRUNE_MAX_M), optionally fused with the compressor.
//
// Scoring every quadruple exactly costs about 13 instructions a row; nearly all quadruples lose by far.  So scores
// are first taken from magnitudes quantised to integers, where they are sums that need no order and two rows fit a word:
//   * q = floor(|w| * Q / max), Q = min(4095, 65535 / (V / 2)): a 16-bit half of a word can add up V / 2 of them;
//   * for a < b < c < d with t1 >= t2 the two largest of (a, b, c), the two largest of the quadruple add up to
//     t1 + max(t2, d), so a quadruple costs one max and one add a word (two rows) behind the triple's part.
// Quantisation is monotone and floors, and the fp32 sums of the reference stray by at most 2V ulps of their value, so a
// quadruple whose integer score is more than W = 2V + V/8 + 2 below the best cannot win.  The others, one or two of 1820 as a
// rule, are scored exactly and in the reference's order; the best exact score, of equal ones the first in lexicographic order,
// wins.  Blocks whose candidates overflow the list (many equal weights), or whose magnitudes are not finite, all zero or tiny,
// take the exhaustive exact search.
//
// A CTA takes V rows x G groups (G * m = 64 columns or more, whole metadata tiles).  A task is (b, c) x two values of a x four
// of d: eight quadruples from four loads (b, c, a pair, d quad) of the group's [row pair][column] words in shared memory,
// whose bandwidth bounds the kernel together with integer issue.
// ------------------------------------------------------------------------------------------------
constexpr int PRUNE_MAX_M = 64;
constexpr int CAND_MAX = 64;      // candidates a group may collect
constexpr int PRUNE_THREADS = 256;

struct PruneGroup {
    uint32_t max_bits;    // largest magnitude of the block, as bits
    uint32_t best;        // best integer score so far
    int count;            // candidates pushed
    int cols[4];          // the winner; cols[0] < 0: nothing is kept
    uint32_t score[CAND_MAX], key[CAND_MAX];
};

struct PruneParams {
    const void *w;
    int64_t ldw, ldm, Ksp;
    uint32_t one;                           // 1, which the compiler must not know (see the scoring loop)
    int M, K, V, m, mp, G, groups, pitch;   // mp: columns of a group in the quantised tile (m rounded up to 4); pitch: floats of a tile row
    int32_t *mask;                          // pruner: the mask; null when fused
    uint32_t *colloc;
    uint32_t *values, *meta;                // fused: the compressed arrays
    unsigned long long *violations;
};

__device__ __forceinline__ uint32_t max2(uint32_t a, uint32_t b)
{
    uint32_t d;
    asm("max.u16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}
__device__ __forceinline__ uint32_t min2(uint32_t a, uint32_t b)
{
    uint32_t d;
    asm("min.u16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}
// Division of e by d through the reciprocal ceil(2^32 / d): exact while e * d < 2^32 (d > 1; d = 1 has no such reciprocal).
struct Divisor {
    uint32_t d, inv;
    __device__ __forceinline__ explicit Divisor(int x) : d((uint32_t)x), inv(x > 1 ? 0xFFFFFFFFu / (uint32_t)x + 1u : 0u) {}
    __device__ __forceinline__ int div(int e) const { return d > 1 ? (int)__umulhi((uint32_t)e, inv) : e; }
};
__device__ __forceinline__ uint32_t halves_sum(uint32_t x) { return (x & 0xFFFFu) + (x >> 16); }

// M_: m where it is known at compile time (8, 16, 32), else 0
template <int WT, bool FUSED, int M_>
__global__ void __launch_bounds__(PRUNE_THREADS) prune_candidates_kernel(const PruneParams p)
{
    extern __shared__ __align__(16) uint8_t psm[];
    const int V = p.V, m = M_ ? M_ : p.m, mp = M_ ? M_ : p.mp, G = p.G;
    uint32_t *q = reinterpret_cast<uint32_t *>(psm);                        // [G][V / 2][mp] pairs of rows
    float *tile = reinterpret_cast<float *>(q + (size_t)G * (V / 2) * mp);  // [V][pitch] weights
    PruneGroup *grp = reinterpret_cast<PruneGroup *>(tile + (size_t)V * p.pitch);
    const int spans = (int)((p.Ksp / 2 + G - 1) / G);                       // the format's padding groups included
    const int bi = blockIdx.x / spans, g0 = (blockIdx.x - bi * spans) * G;
    const int ng = p.groups <= g0 ? 0 : p.groups - g0 < G ? p.groups - g0 : G;
    const int span = ng * m;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

    if (tid < G) { grp[tid].max_bits = 0; grp[tid].best = 0; grp[tid].count = 0; grp[tid].cols[0] = -1; }
    __syncthreads();
    // ---- the block's weights, and the largest magnitude of every group
    {
        const int64_t base = (int64_t)bi * V * p.ldw + (int64_t)g0 * m;
        constexpr int PER = WT == W_F16 ? 8 : 4;      // weights of a 16-byte load
        const bool vec = span % PER == 0 && p.ldw % PER == 0 && base % PER == 0 && ((uintptr_t)p.w & 15) == 0;
        if (vec) {
            const int per_row = span / PER;
            const Divisor by(per_row > 0 ? per_row : 1);
            for (int e = tid; e < V * per_row; e += PRUNE_THREADS) {
                const int r = by.div(e), c = (e - r * per_row) * PER;
                float x[PER];
                if (WT == W_F16) {
                    const uint4 v = __ldg(reinterpret_cast<const uint4 *>((const __half *)p.w + base + (int64_t)r * p.ldw + c));
                    const uint32_t w4[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&w4[i]));
                        x[(2 * i) % PER] = f.x; x[(2 * i + 1) % PER] = f.y;
                    }
                } else {
                    const float4 v = __ldg(reinterpret_cast<const float4 *>((const float *)p.w + base + (int64_t)r * p.ldw + c));
                    x[0] = v.x; x[1] = v.y; x[2] = v.z; x[3] = v.w;
                }
#pragma unroll
                for (int i = 0; i < PER; i += 4) *reinterpret_cast<float4 *>(tile + r * p.pitch + c + i) = make_float4(x[i], x[i + 1], x[i + 2], x[i + 3]);
            }
        } else {
            const Divisor by(span > 0 ? span : 1);
            for (int e = tid; e < V * span; e += PRUNE_THREADS) {
                const int r = by.div(e), c = e - r * span;
                const int64_t at = base + (int64_t)r * p.ldw + c;
                tile[r * p.pitch + c] = WT == W_F16 ? __half2float(((const __half *)p.w)[at]) : ((const float *)p.w)[at];
            }
        }
        __syncthreads();
        for (int g = warp; g < ng; g += PRUNE_THREADS / 32) {   // a warp per group: lanes along the columns, then down the rows
            uint32_t mx = 0;
            const Divisor by(m);
            for (int e = lane; e < V * m; e += 32) {
                const int r = by.div(e), c = e - r * m;
                mx = max(mx, __float_as_uint(fabsf(tile[r * p.pitch + g * m + c])));
            }
            mx = __reduce_max_sync(0xffffffffu, mx);
            if (lane == 0) grp[g].max_bits = mx;
        }
    }
    __syncthreads();
    const int Q = min(4095, 65535 / (V / 2));
    const uint32_t window = (uint32_t)(2 * V + V / 8 + 2);
    auto quantised = [&](int g) {   // integer scores are safe for this block
        const float mx = __uint_as_float(grp[g].max_bits);
        return grp[g].max_bits < 0x7F800000u && mx > 1e-30f;
    };
    // ---- quantised pairs of rows
    if (m > 4) {
        const Divisor by_mp(mp);
        for (int g = 0; g < ng; g++) {
            const bool fine = quantised(g);
            const float scale = fine ? (float)Q / __uint_as_float(grp[g].max_bits) : 0.0f;
            for (int e = tid; e < (V / 2) * mp; e += PRUNE_THREADS) {
                const int rp = by_mp.div(e), c = e - rp * mp;
                uint32_t word = 0;
                if (c < m && fine) {
                    const float *t = tile + 2 * rp * p.pitch + g * m + c;
                    const int lo = min(Q, (int)(fabsf(t[0]) * scale)), hi = min(Q, (int)(fabsf(t[p.pitch]) * scale));
                    word = (uint32_t)lo | ((uint32_t)hi << 16);
                }
                q[g * (V / 2) * mp + e] = word;
            }
        }
        __syncthreads();
    }
    // ---- integer scores: a warp takes 32 tasks of one group at a time
    int tasks = 0;                 // (c, b, pair of a, four of d): floor(c^2 / 4) pairs (b, a pair) for every c
    if (m > 4)
        for (int c = 2; c <= m - 2; c++) tasks += (mp / 4 - (c + 1) / 4) * (c * c / 4);
    const int wtasks = (tasks + 31) / 32;
    if (m == 4 && tid < ng && quantised(tid)) {          // one quadruple: it wins
#pragma unroll
        for (int i = 0; i < 4; i++) grp[tid].cols[i] = i;
    }
    for (int wt = warp; wt < ng * wtasks; wt += PRUNE_THREADS / 32) {
        const int g = wt / wtasks;
        if (!quantised(g)) continue;
        const int idx = (wt - g * wtasks) * 32 + lane;
        const bool on = idx < tasks;
        int c = 2, left = on ? idx : 0;
        for (;; c++) {
            const int n = (mp / 4 - (c + 1) / 4) * (c * c / 4);
            if (left < n) break;
            left -= n;
        }
        const int pairs = c * c / 4;
        const int d0 = ((c + 1) / 4 + left / pairs) * 4;
        const int r = left % pairs;
        int b = (int)sqrtf(4.0f * (float)r);            // floor(b^2 / 4) <= r < floor((b + 1)^2 / 4)
        while (b * b / 4 > r) --b;
        while ((b + 1) * (b + 1) / 4 <= r) ++b;
        const int a = 2 * (r - b * b / 4);
        const uint32_t *col = q + (size_t)g * (V / 2) * mp;
        uint32_t s1[2] = {0, 0}, s2[2][4] = {{0, 0, 0, 0}, {0, 0, 0, 0}};
#pragma unroll 4
        for (int rp = 0; rp < V / 2; rp++, col += mp) {
            const uint32_t xb = col[b], xc = col[c];
            const uint2 xa = *reinterpret_cast<const uint2 *>(col + a);
            const uint4 xd = *reinterpret_cast<const uint4 *>(col + d0);
            const uint32_t hi = max2(xb, xc), lo = min2(xb, xc);
#pragma unroll
            for (int i = 0; i < 2; i++) {
                const uint32_t x = i ? xa.y : xa.x;
                const uint32_t t2 = max2(lo, min2(hi, x));
                // sums as x * 1 + sum: multiply-adds run beside the comparisons, plain additions share their pipe, which is the
                // one that bounds this loop
                s1[i] = max2(hi, x) * p.one + s1[i];
                s2[i][0] = max2(t2, xd.x) * p.one + s2[i][0];
                s2[i][1] = max2(t2, xd.y) * p.one + s2[i][1];
                s2[i][2] = max2(t2, xd.z) * p.one + s2[i][2];
                s2[i][3] = max2(t2, xd.w) * p.one + s2[i][3];
            }
        }
        uint32_t score[8], mine = 0;
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const bool ok = on && a + (i >> 2) < b && d0 + (i & 3) > c && d0 + (i & 3) < m;
            score[i] = ok ? halves_sum(s1[i >> 2]) + halves_sum(s2[i >> 2][i & 3]) + 1u : 0u;   // 0: no quadruple
            mine = max(mine, score[i]);
        }
        const uint32_t wbest = __reduce_max_sync(0xffffffffu, mine);
        uint32_t best = 0;
        if (lane == 0) best = max(wbest, atomicMax(&grp[g].best, wbest));
        best = __shfl_sync(0xffffffffu, best, 0);
        if (mine && mine + window >= best) {
#pragma unroll
            for (int i = 0; i < 8; i++)
                if (score[i] && score[i] + window >= best) {
                    const int at = atomicAdd(&grp[g].count, 1);
                    if (at < CAND_MAX) {
                        grp[g].score[at] = score[i];
                        grp[g].key[at] = (uint32_t)(a + (i >> 2)) << 24 | (uint32_t)b << 16 | (uint32_t)c << 8 | (uint32_t)(d0 + (i & 3));
                    }
                }
        }
    }
    __syncthreads();
    // ---- exact scores of the candidates: one warp per group
    for (int g = warp; g < ng; g += PRUNE_THREADS / 32) {
        if (m == 4 || !quantised(g) || grp[g].count > CAND_MAX) continue;
        const uint32_t best = grp[g].best;
        float top = -1.0f;
        uint32_t key = 0xFFFFFFFFu;
        int close = 0;
        for (int i = lane; i < grp[g].count; i += 32) close += grp[g].score[i] + window >= best;
        close = __reduce_add_sync(0xffffffffu, close);
        for (int i = lane; i < grp[g].count; i += 32) {
            if (grp[g].score[i] + window < best) continue;
            const uint32_t k = grp[g].key[i];
            const int c[4] = {(int)(k >> 24), (int)(k >> 16 & 255), (int)(k >> 8 & 255), (int)(k & 255)};
            const float t = close == 1 ? 1.0f : exact_score(tile + g * m, p.pitch, V, c);
            if (t > top || (t == top && k < key)) { top = t; key = k; }
        }
        for (int o = 16; o > 0; o >>= 1) {
            const float ot = __shfl_xor_sync(0xffffffffu, top, o);
            const uint32_t ok = __shfl_xor_sync(0xffffffffu, key, o);
            if (ot > top || (ot == top && ok < key)) { top = ot; key = ok; }
        }
        if (lane < 4) grp[g].cols[lane] = (int)(key >> (24 - 8 * lane) & 255);
    }
    // ---- exhaustive exact search where integers do not do
    for (int g = 0; g < ng; g++) {
        if (quantised(g) && grp[g].count <= CAND_MAX) continue;      // the same for every thread
        if (grp[g].max_bits == 0) continue;                          // all zero: nothing is kept
        __shared__ float s_best[PRUNE_THREADS];
        __shared__ int s_idx[PRUNE_THREADS];
        float top = 0.0f;
        int at = -1;
        const int ncombo = (int)binom4(m);
        for (int ci = tid; ci < ncombo; ci += PRUNE_THREADS) {
            int c[4];
            unrank4(ci, m, c);
            const float t = exact_score(tile + g * m, p.pitch, V, c);
            if (t > top) { top = t; at = ci; }                       // strict: the first of equal scores stays
        }
        s_best[tid] = top;
        s_idx[tid] = at;
        __syncthreads();
        for (int s = PRUNE_THREADS / 2; s > 0; s >>= 1) {
            if (tid < s) {
                const float ob = s_best[tid + s], mb = s_best[tid];
                const int oi = s_idx[tid + s], mi = s_idx[tid];
                // larger score wins; equal scores: the lower quadruple index (the one the sequential scan meets first)
                if (oi >= 0 && (mi < 0 || ob > mb || (ob == mb && oi < mi))) { s_best[tid] = ob; s_idx[tid] = oi; }
            }
            __syncthreads();
        }
        if (tid == 0 && s_idx[0] >= 0) unrank4(s_idx[0], m, grp[g].cols);
        __syncthreads();
    }
    __syncthreads();

    const int64_t gpad = p.Ksp / 2;
    const int gout = gpad - g0 < G ? (int)(gpad - g0) : G;           // groups to write, padding included
    for (int e = tid; e < gout * 4; e += PRUNE_THREADS) {
        const int g = e >> 2;
        p.colloc[(int64_t)bi * gpad * 4 + (int64_t)g0 * 4 + e] = g < ng && grp[g].cols[0] >= 0 ? (uint32_t)grp[g].cols[e & 3] : 0u;
    }
    if (FUSED) {
        // four rows of a group are one 16-byte piece of the value order; the nibbles of a tile's four groups meet by shuffles
        unsigned int bad = 0;
        const int64_t tiles = p.Ksp / 8;
        const Divisor by_gout(gout);
        for (int e0 = 0; e0 < (V / 4) * gout; e0 += PRUNE_THREADS) {   // gout is a multiple of four: no lane of a tile is left out
            const int e = e0 + tid;
            const bool on = e < (V / 4) * gout;
            const int rq = on ? by_gout.div(e) : 0, g = on ? e - rq * gout : 0;
            uint32_t out[4] = {0, 0, 0, 0}, nib[4] = {0, 0, 0, 0};
            if (on && g < ng) {
                const int c0 = grp[g].cols[0];
                if (c0 < 0) {
                    bad += 4;
                } else {
                    const int cols[4] = {c0, grp[g].cols[1], grp[g].cols[2], grp[g].cols[3]};
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        const float *row = tile + (4 * rq + i) * p.pitch + g * m;
                        const float x[4] = {row[cols[0]], row[cols[1]], row[cols[2]], row[cols[3]]};
                        const float v[4] = {fabsf(x[0]), fabsf(x[1]), fabsf(x[2]), fabsf(x[3])};
                        int i0, i1;
                        top2_of4(v, i0, i1);
                        const int lo = min(i0, i1), hi = max(i0, i1);
                        out[i] = (uint32_t)__half_as_ushort(__float2half_rn(lo == 0 ? x[0] : lo == 1 ? x[1] : x[2])) |
                                 (uint32_t)__half_as_ushort(__float2half_rn(hi == 1 ? x[1] : hi == 2 ? x[2] : x[3])) << 16;
                        nib[i] = (uint32_t)(lo | hi << 2) << (((g0 + g) & 3) * 4);
                    }
                }
            }
            uint32_t m01 = nib[0] | nib[1] << 16, m23 = nib[2] | nib[3] << 16;
#pragma unroll
            for (int o = 1; o < 4; o <<= 1) {
                m01 |= __shfl_xor_sync(0xffffffffu, m01, o);
                m23 |= __shfl_xor_sync(0xffffffffu, m23, o);
            }
            if (on) {
                const int64_t r = (int64_t)bi * V + 4 * rq, gg = g0 + g;
                *reinterpret_cast<uint4 *>(p.values + ((r / 16) * 16 * p.Ksp + (gg / 4) * 128 + ((r % 16) / 4) * 32 + (gg % 4) * 8) / 2) = make_uint4(out[0], out[1], out[2], out[3]);
                if ((gg & 3) == 0) *reinterpret_cast<uint2 *>(p.meta + (r / 32) * 16 * tiles + (gg / 4) * 16 + (r % 32) / 2) = make_uint2(m01, m23);
            }
        }
        if (p.violations) {
            bad = __reduce_add_sync(0xffffffffu, bad);
            if (lane == 0 && bad) atomicAdd(p.violations, (unsigned long long)bad);
        }
    } else {
        const Divisor by_ng(ng > 0 ? ng : 1), by_span(span > 0 ? span : 1), by_m(m);
        for (int e = tid; e < V * ng; e += PRUNE_THREADS) {          // kept columns of a row, packed over the quantised tile
            const int r = by_ng.div(e), g = e - r * ng;
            uint32_t kept = 0xFFFFu;
            if (grp[g].cols[0] >= 0) {
                const float *row = tile + r * p.pitch + g * m;
                const float v[4] = {fabsf(row[grp[g].cols[0]]), fabsf(row[grp[g].cols[1]]), fabsf(row[grp[g].cols[2]]), fabsf(row[grp[g].cols[3]])};
                int i0, i1;
                top2_of4(v, i0, i1);
                kept = (uint32_t)grp[g].cols[i0] | (uint32_t)grp[g].cols[i1] << 8;
            }
            q[e] = kept;
        }
        __syncthreads();
        int32_t *mrow = p.mask + (int64_t)bi * V * p.ldm + (int64_t)g0 * m;
        for (int e = tid; e < V * span; e += PRUNE_THREADS) {
            const int r = by_span.div(e), c = e - r * span, g = by_m.div(c), cc = c - g * m;
            const uint32_t kept = q[r * ng + g];
            mrow[(int64_t)r * p.ldm + c] = cc == (int)(kept & 255) || cc == (int)(kept >> 8);
        }
    }
}

size_t prune_smem_bytes(int V, int m, int G)
{
    const int mp = (m + 3) / 4 * 4;
    const size_t pitch = ((size_t)G * m + 3) / 4 * 4 + 4;
    return (size_t)G * (V / 2) * mp * 4 + (size_t)V * pitch * 4 + (size_t)G * sizeof(PruneGroup);
}
int prune_groups_per_cta(int m) { return m >= 16 ? 4 : m >= 8 ? 8 : 16; }
bool prune_by_candidates(int V, int m) { return m <= PRUNE_MAX_M && prune_smem_bytes(V, m, prune_groups_per_cta(m)) <= 200 * 1024; }

template <int WT, bool FUSED>
cudaError_t launch_candidates(PruneParams p, cudaStream_t stream)
{
    p.one = 1;
    p.mp = (p.m + 3) / 4 * 4;
    p.G = prune_groups_per_cta(p.m);
    p.groups = p.K / p.m;
    p.pitch = (p.G * p.m + 3) / 4 * 4 + 4;
    p.Ksp = ksp_of(p.K, p.m);
    const size_t smem = prune_smem_bytes(p.V, p.m, p.G);
    const unsigned blocks = (unsigned)((p.M / p.V) * ((p.Ksp / 2 + p.G - 1) / p.G));
    auto launch = [&](auto kernel) -> cudaError_t {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
        if (e != cudaSuccess) return e;
        kernel<<<blocks, PRUNE_THREADS, smem, stream>>>(p);
        return cudaGetLastError();
    };
    switch (p.m) {
    case 8: return launch(prune_candidates_kernel<WT, FUSED, 8>);
    case 16: return launch(prune_candidates_kernel<WT, FUSED, 16>);
    case 32: return launch(prune_candidates_kernel<WT, FUSED, 32>);
    default: return launch(prune_candidates_kernel<WT, FUSED, 0>);
    }
}

__global__ void __launch_bounds__(256) prune_kernel(const float *__restrict__ w, int64_t ldw, int M, int K, int V, int m, int64_t Ksp,
                                                    int32_t *__restrict__ mask, int64_t ldm, uint32_t *__restrict__ colloc)
{
    extern __shared__ float tile[];  // V x m magnitudes
    __shared__ float s_best[256];
    __shared__ int s_idx[256];
    __shared__ int s_cols[4];
    const int groups = K / m;
    const int bi = blockIdx.x / groups, g = blockIdx.x % groups;
    const float *src = w + (int64_t)bi * V * ldw + (int64_t)g * m;
    for (int e = threadIdx.x; e < V * m; e += blockDim.x) tile[e] = fabsf(src[(int64_t)(e / m) * ldw + (e % m)]);
    __syncthreads();

    const int ncombo = (int)binom4(m);
    float best = 0.0f;
    int best_idx = -1;
    for (int ci = threadIdx.x; ci < ncombo; ci += blockDim.x) {
        int c[4];
        unrank4(ci, m, c);
        float total = 0.0f;
        for (int r = 0; r < V; r++) {
            const float *row = tile + r * m;
            const float v0 = row[c[0]], v1 = row[c[1]], v2 = row[c[2]], v3 = row[c[3]];
            // largest and second largest of four (values only: ties do not change the sum)
            const float hi01 = fmaxf(v0, v1), lo01 = fminf(v0, v1), hi23 = fmaxf(v2, v3), lo23 = fminf(v2, v3);
            const float top1 = fmaxf(hi01, hi23);
            const float top2 = fmaxf(fminf(hi01, hi23), fmaxf(lo01, lo23));
            total += top1;
            total += top2;
        }
        if (total > best) { best = total; best_idx = ci; }  // strict: the first of equal scores stays
    }
    s_best[threadIdx.x] = best;
    s_idx[threadIdx.x] = best_idx;
    __syncthreads();
    for (int s = blockDim.x / 2; s > 0; s >>= 1) {
        if (threadIdx.x < s) {
            const float ob = s_best[threadIdx.x + s];
            const int oi = s_idx[threadIdx.x + s];
            const float mb = s_best[threadIdx.x];
            const int mi = s_idx[threadIdx.x];
            // larger score wins; equal scores: the lower quadruple index (the one the sequential scan meets first)
            if (oi >= 0 && (mi < 0 || ob > mb || (ob == mb && oi < mi))) { s_best[threadIdx.x] = ob; s_idx[threadIdx.x] = oi; }
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        int c[4] = {0, 0, 0, 0};
        if (s_idx[0] >= 0) unrank4(s_idx[0], m, c);
        for (int j = 0; j < 4; j++) {
            s_cols[j] = c[j];
            colloc[(int64_t)bi * (Ksp / 2) * 4 + (int64_t)g * 4 + j] = (uint32_t)c[j];
        }
    }
    __syncthreads();
    const bool any = s_idx[0] >= 0;
    for (int r = threadIdx.x; r < V; r += blockDim.x) {
        int32_t *mrow = mask + ((int64_t)bi * V + r) * ldm + (int64_t)g * m;
        for (int j = 0; j < m; j++) mrow[j] = 0;
        if (any) {
            const float *row = tile + r * m;
            const float v[4] = {row[s_cols[0]], row[s_cols[1]], row[s_cols[2]], row[s_cols[3]]};
            int i0, i1;
            top2_of4(v, i0, i1);
            mrow[s_cols[i0]] = 1;
            mrow[s_cols[i1]] = 1;
        }
    }
}

__global__ void zero_padded_colloc(uint32_t *colloc, int nblocks, int groups, int64_t gpad)
{
    const int64_t total = (int64_t)nblocks * (gpad - groups) * 4;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t per = (gpad - groups) * 4;
        const int64_t b = i / per, o = i % per;
        colloc[b * gpad * 4 + groups * 4 + o] = 0;
    }
}

}  // namespace

cudaError_t launch_prune(const float *w, int64_t ldw, int M, int K, int V, int m, int32_t *mask, int64_t ldm, uint32_t *colloc,
                         cudaStream_t stream)
{
    if (prune_by_candidates(V, m)) {
        PruneParams p = {};
        p.w = w; p.ldw = ldw; p.ldm = ldm; p.M = M; p.K = K; p.V = V; p.m = m; p.mask = mask; p.colloc = colloc;
        return launch_candidates<W_F32, false>(p, stream);
    }
    const int64_t Ksp = ksp_of(K, m);
    const int groups = K / m;
    const int nblocks = M / V;
    if (Ksp / 2 > groups) {
        zero_padded_colloc<<<64, 256, 0, stream>>>(colloc, nblocks, groups, Ksp / 2);
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    const size_t smem = (size_t)V * m * sizeof(float);
    prune_kernel<<<(unsigned)(nblocks * groups), 256, smem, stream>>>(w, ldw, M, K, V, m, Ksp, mask, ldm, colloc);
    return cudaGetLastError();
}

bool sparsify_supported(int K, int V, int m) { return K % m == 0 && prune_by_candidates(V, m); }

cudaError_t launch_sparsify(const void *w, bool half, int64_t ldw, int M, int K, int V, int m, void *values, uint32_t *meta, uint32_t *colloc,
                            unsigned long long *violations, cudaStream_t stream)
{
    PruneParams p = {};
    p.w = w; p.ldw = ldw; p.M = M; p.K = K; p.V = V; p.m = m; p.colloc = colloc;
    p.values = (uint32_t *)values; p.meta = meta; p.violations = violations;
    return half ? launch_candidates<W_F16, true>(p, stream) : launch_candidates<W_F32, true>(p, stream);
}

}  // namespace vnm
