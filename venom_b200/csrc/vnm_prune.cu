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

#include <type_traits>

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

template <int WT> struct WeightOf { using T = float; };
template <> struct WeightOf<W_F16> { using T = __half; };
__device__ __forceinline__ float weight(float x) { return x; }
__device__ __forceinline__ float weight(__half x) { return __half2float(x); }

// The two largest magnitudes of a row's four columns, the larger first.
template <typename T>
__device__ __forceinline__ float2 largest_two(const T *row, const int c[4])
{
    const float v0 = fabsf(weight(row[c[0]])), v1 = fabsf(weight(row[c[1]])), v2 = fabsf(weight(row[c[2]])), v3 = fabsf(weight(row[c[3]]));
    const float hi01 = fmaxf(v0, v1), lo01 = fminf(v0, v1), hi23 = fmaxf(v2, v3), lo23 = fminf(v2, v3);
    return make_float2(fmaxf(hi01, hi23), fmaxf(fminf(hi01, hi23), fmaxf(lo01, lo23)));
}
// The reference's score of one quadruple: an fp32 sum in row order, the larger magnitude of a row first.
template <typename T>
__device__ __forceinline__ float exact_score(const T *tile, int pitch, int V, const int c[4])
{
    float total = 0.0f;
    for (int r = 0; r < V; r++) {
        const float2 x = largest_two(tile + r * pitch, c);
        total += x.x;
        total += x.y;
    }
    return total;
}

// ------------------------------------------------------------------------------------------------
// Pruner by candidates (m <= PRUNE_MAX_M), optionally fused with the compressor.
//
// Scoring every quadruple exactly costs about 13 instructions a row; nearly all quadruples lose by far.  So scores
// are first taken from magnitudes quantised to integers, where they are sums that need no order and two rows fit a word:
//   * q = |w| * Q / max rounded, Q = min(4095, 65535 / (V / 2)): a 16-bit half of a word can add up V / 2 of them;
//   * with t1 >= t2 the two largest of (a, b, c), the two largest of the quadruple add up to t1 + max(t2, d), so a quadruple
//     costs one max and one add a word (two rows) behind the triple's part.
// Quantisation is monotone and off by at most half a unit a term, and the fp32 sums of the reference stray by at most 2V ulps of their
// value, so a quadruple whose integer score is more than W = 2V + V/8 + 2 below the best cannot win.  The others, one or two of 1820 as a
// rule, are scored exactly and in the reference's order; the best exact score, of equal ones the first in lexicographic order,
// wins.  Blocks whose candidates overflow the list (many equal weights), or whose magnitudes are not finite, all zero or tiny,
// take the exhaustive exact search.
//
// A CTA takes V rows x G groups (G * m = 64 columns or more, whole metadata tiles).  Its lanes take tasks and add up all rows of them
// from the group's [row pair][column] words in shared memory.
//   * m <= 32: a task is a pair (b, c) with the four columns of a block A and the four of a block D: sixteen quadruples from ten words, four
//     behind every triple (a, b, c).  The list (PruneTasks) has every quadruple once and wastes a quarter of the sixteens at m = 16.
//     Bound: the pipe of the comparisons, 26 a task and word at 2 clocks a warp (75 % active), and the issue slots (82 % used).  The sums
//     are multiply-adds, which run beside it; the largest of a triple is never formed: it is h + a - min(h, a), and the sum of a is the
//     column's.  12288 x 12288, fp16, us, before (the loop for larger m, two values of a x four aligned d, 40 % of them wasted, and a lane
//     for all rows of a candidate) and now: m = 16 V = 128 2598, 1513, V = 32 3740, 1970; m = 8 V = 128 1013, 618; 4096 x 4096, m = 32
//     V = 128 2031, 1320.
//     Not kept: bounds from the sums of minima of triples, which leave 20 % of the quadruples at V = 128 and 2 % at V = 32 to score,
//     with rows added up by mma.sync: as many instructions for the table and the bounds as they save (2030 and 3397 us at m = 16); and
//     loops of their own for the tasks that do not use all sixteen: 1405 us at V = 128, but 2379 at V = 32 (part-filled warps).
//   * larger m: a task is (b, c) x two values of a x four of d, eight quadruples from eight words.
// ------------------------------------------------------------------------------------------------
constexpr int PRUNE_MAX_M = 64;
constexpr int CAND_MAX = 64;      // candidates a group may collect
constexpr int PRUNE_MAX_G = 16;   // groups of a CTA
constexpr int PRUNE_MAX_COLUMNS = 128;   // their columns, m rounded up to 4, for m <= 32

// The tasks of a group of up to eight blocks of four columns, ordered by the highest block, so that fewer blocks take a prefix.  With X, Y, Z, W
// different blocks: (b, c) from Y x Z, A = X, D = W;  a pair of X, A = Y, D = Z;  a pair of X, A = D = Y (a < d);  (0, 1) or (2, 3) of
// X, A = X (the other two), D = Y;  (0, 1) of X, A = D = X (2 and 3).
constexpr int TASK_MAX_BLOCKS = 8;
struct PruneTasks {
    uint32_t task[2416];                 // b | c << 5 | A << 10 | D << 13 | quadruples that count << 16 (bit 4 * i + j: column i of A, j of D)
    int end[TASK_MAX_BLOCKS + 1];        // tasks of so many blocks
};
constexpr PruneTasks make_prune_tasks()
{
    PruneTasks t = {};
    int n = 0;
    auto add = [&](int b, int c, int A, int D, uint32_t mask) { t.task[n++] = (uint32_t)(b | c << 5 | A << 10 | D << 13) | mask << 16; };
    auto pairs = [&](int X, int A, int D, uint32_t mask) {
        for (int b = 4 * X; b < 4 * X + 4; b++)
            for (int c = b + 1; c < 4 * X + 4; c++) add(b, c, A, D, mask);
    };
    for (int top = 0; top < TASK_MAX_BLOCKS; top++) {
        for (int X = 0; X < top; X++)
            for (int Y = X + 1; Y < top; Y++)
                for (int Z = Y + 1; Z < top; Z++)
                    for (int i = 0; i < 16; i++) add(4 * Y + i / 4, 4 * Z + i % 4, X, top, 0xFFFF);
        for (int X = 0; X < top; X++) {
            for (int Y = 0; Y < top; Y++) {
                if (Y != X) pairs(X, Y, top, 0xFFFF);
                if (Y > X) pairs(top, X, Y, 0xFFFF);
            }
            pairs(X, top, top, 0x08CE);
            add(4 * X, 4 * X + 1, X, top, 0xFF00);
            add(4 * X + 2, 4 * X + 3, X, top, 0x00FF);
            add(4 * top, 4 * top + 1, top, X, 0xFF00);
            add(4 * top + 2, 4 * top + 3, top, X, 0x00FF);
        }
        add(4 * top, 4 * top + 1, top, top, 1u << 11);
        t.end[top + 1] = n;
    }
    return t;
}
__device__ const PruneTasks g_tasks = make_prune_tasks();

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
    int M, K, V, m, mp, G, groups, pitch;   // mp: columns of a group in the quantised tile (m rounded up to 4); pitch: weights of a tile row
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

// M_: m where it is known at compile time (8, 16, 32), 0 for any m up to 32, LARGER_M beyond, whose loop needs fewer registers
constexpr int LARGER_M = -1;
template <int WT, bool FUSED, int M_, int THREADS>
__global__ void __launch_bounds__(THREADS, M_ == LARGER_M ? 1 : 768 / THREADS) prune_candidates_kernel(const PruneParams p)
{
    using W = typename WeightOf<WT>::T;
    extern __shared__ __align__(16) uint8_t psm[];
    const int V = p.V, m = M_ > 0 ? M_ : p.m, mp = M_ > 0 ? M_ : p.mp, G = p.G;
    uint32_t *q = reinterpret_cast<uint32_t *>(psm);                        // [G][V / 2][mp] pairs of rows
    W *tile = reinterpret_cast<W *>(q + (size_t)G * (V / 2) * mp);          // [V][pitch] weights
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
        constexpr int PER = 16 / (int)sizeof(W);      // weights of a 16-byte load
        const bool vec = span % PER == 0 && p.ldw % PER == 0 && base % PER == 0 && ((uintptr_t)p.w & 15) == 0;
        if (vec) {
            const int per_row = span / PER;
            const Divisor by(per_row > 0 ? per_row : 1);
#pragma unroll 4
            for (int e = tid; e < V * per_row; e += THREADS) {
                const int r = by.div(e), c = (e - r * per_row) * PER;
                *reinterpret_cast<uint4 *>(tile + r * p.pitch + c) = __ldg(reinterpret_cast<const uint4 *>((const W *)p.w + base + (int64_t)r * p.ldw + c));
            }
        } else {
            const Divisor by(span > 0 ? span : 1);
            for (int e = tid; e < V * span; e += THREADS) {
                const int r = by.div(e), c = e - r * span;
                tile[r * p.pitch + c] = ((const W *)p.w)[base + (int64_t)r * p.ldw + c];
            }
        }
        __syncthreads();
        const Divisor by_m(m);
        if (WT == W_F16 && m % 2 == 0) {
            // a warp per sixteen columns, two of one group a lane, every fourth row; magnitudes of fp16 compare as integers
            for (int c0 = warp * 16; c0 < span; c0 += THREADS / 2) {
                const int at = c0 + 2 * (lane & 7);
                if (at >= span) continue;
                const W *t = tile + at;
                uint32_t mx = 0;
#pragma unroll 8
                for (int r = lane >> 3; r < V; r += 4) mx = max2(mx, *reinterpret_cast<const uint32_t *>(t + r * p.pitch) & 0x7FFF7FFFu);
                atomicMax(&grp[by_m.div(at)].max_bits, __float_as_uint(__half2float(__ushort_as_half((unsigned short)max(mx & 0xFFFFu, mx >> 16)))));
            }
        } else {
            for (int c0 = warp * 8; c0 < span; c0 += THREADS / 4) {   // a warp per eight columns
                const int at = c0 + (lane & 7);
                if (at >= span) continue;
                const W *t = tile + at;
                uint32_t mx = 0;
#pragma unroll 8
                for (int r = lane >> 3; r < V; r += 4) mx = max(mx, __float_as_uint(fabsf(weight(t[r * p.pitch]))));
                atomicMax(&grp[by_m.div(at)].max_bits, mx);
            }
        }
    }
    __syncthreads();
    const int Q = min(4095, 65535 / (V / 2));
    const uint32_t window = (uint32_t)(2 * V + V / 8 + 2);
    __shared__ float s_scale[PRUNE_MAX_G];   // from magnitudes to integers; 0: integer scores are not safe for this block
    if (tid < ng) {
        const float mx = __uint_as_float(grp[tid].max_bits);
        const bool fine = grp[tid].max_bits < 0x7F800000u && mx > 1e-30f;
        s_scale[tid] = fine ? (float)Q / mx : 0.0f;
        if (m == 4 && fine) {          // one quadruple: it wins
#pragma unroll
            for (int i = 0; i < 4; i++) grp[tid].cols[i] = i;
        }
    }
    __syncthreads();
    auto quantised = [&](int g) { return s_scale[g] > 0.0f; };
    // ---- quantised pairs of rows, two columns a thread: rounded to integers in the lowest bits of the sum with 2^23
    if (m > 4) {
        const Divisor by_two(mp / 2), by_half(V / 2);
        for (int e = tid; e < ng * (V / 2) * (mp / 2); e += THREADS) {
            const int at = by_two.div(e), c = 2 * (e - at * (mp / 2)), g = by_half.div(at), rp = at - g * (V / 2);
            const float scale = s_scale[g];
            const W *t = tile + 2 * rp * p.pitch + g * m + c;
            float2 x0 = make_float2(0.0f, 0.0f), x1 = x0;
            if (m % 2 == 0) {
                if (c < m) {
                    if constexpr (WT == W_F16) {
                        x0 = __half22float2(*reinterpret_cast<const __half2 *>(t));
                        x1 = __half22float2(*reinterpret_cast<const __half2 *>(t + p.pitch));
                    } else {
                        x0 = *reinterpret_cast<const float2 *>(t);
                        x1 = *reinterpret_cast<const float2 *>(t + p.pitch);
                    }
                }
            } else {
                if (c < m) { x0.x = weight(t[0]); x1.x = weight(t[p.pitch]); }
                if (c + 1 < m) { x0.y = weight(t[1]); x1.y = weight(t[p.pitch + 1]); }
            }
            auto word = [&](float lo, float hi) {
                return min2(__byte_perm(__float_as_uint(fmaf(fabsf(lo), scale, 8388608.0f)), __float_as_uint(fmaf(fabsf(hi), scale, 8388608.0f)), 0x5410), (uint32_t)Q * 0x10001u);
            };
            *reinterpret_cast<uint2 *>(q + 2 * e) = make_uint2(word(x0.x, x1.x), word(x0.y, x1.y));
        }
        __syncthreads();
    }
    if (M_ != LARGER_M && m > 4) {
        // ---- sums of the columns
        __shared__ uint4 s_sum4[PRUNE_MAX_COLUMNS / 4];      // read four at a time: the type aligns them
        uint32_t *const s_sum = reinterpret_cast<uint32_t *>(s_sum4);
        static_assert(PRUNE_MAX_COLUMNS % 4 == 0 && alignof(decltype(s_sum4)) == sizeof(uint4), "whole vectors, aligned whatever else is in shared memory");
        const Divisor by_mp(mp);
        for (int e = tid; e < ng * mp; e += THREADS) {
            const int g = by_mp.div(e);
            const uint32_t *col = q + (size_t)g * (V / 2) * mp + e - g * mp;
            uint32_t sum = 0;
#pragma unroll 8
            for (int rp = 0; rp < V / 2; rp++) sum = __dp2a_lo(col[rp * mp], 0x0101u, sum);
            s_sum[e] = sum;
        }
        __syncthreads();
        // ---- integer scores: a lane takes a task
        const int tasks = g_tasks.end[mp / 4];
        const Divisor by_tasks(tasks);
        for (int i0 = warp * 32; i0 < ng * tasks; i0 += THREADS) {
            const int idx = i0 + lane;
            const int g = idx < ng * tasks ? by_tasks.div(idx) : 0;
            const uint32_t task = __ldg(g_tasks.task + (idx < ng * tasks ? idx - g * tasks : 0));
            const int b = task & 31, c = task >> 5 & 31, A = (task >> 10 & 7) * 4, D = (task >> 13 & 7) * 4;
            const uint32_t *col = q + (size_t)g * (V / 2) * mp;
            uint32_t sh = 0, s1[4] = {}, s2[4][4] = {};
#pragma unroll 4
            for (int rp = 0; rp < V / 2; rp++, col += mp) {
                const uint32_t xb = col[b], xc = col[c];
                const uint4 xa = *reinterpret_cast<const uint4 *>(col + A), xd = *reinterpret_cast<const uint4 *>(col + D);
                const uint32_t hi = max2(xb, xc), lo = min2(xb, xc);
                sh = hi * p.one + sh;
                const uint32_t as[4] = {xa.x, xa.y, xa.z, xa.w}, ds[4] = {xd.x, xd.y, xd.z, xd.w};
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    // the largest of (a, b, c) is hi + a - min(hi, a).  Sums as x * 1 + sum: multiply-adds run beside the comparisons
                    const uint32_t mid = min2(hi, as[i]), t2 = max2(lo, mid);
                    s1[i] = mid * p.one + s1[i];
#pragma unroll
                    for (int j = 0; j < 4; j++) s2[i][j] = max2(t2, ds[j]) * p.one + s2[i][j];
                }
            }
            const uint4 sa = s_sum4[(g * mp + A) / 4];
            const uint32_t sas[4] = {sa.x, sa.y, sa.z, sa.w};
            uint32_t mine = 0, valid = idx < ng * tasks && quantised(g) ? task >> 16 : 0u;
            if (m % 4 != 0) {                                // the last block's columns are not all there
                if (max(b, c) >= m) valid = 0;
                if (A + 4 > m) valid &= (1u << 4 * (m - A)) - 1u;
                if (D + 4 > m) valid &= ((1u << (m - D)) - 1u) * 0x1111u;
            }
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const uint32_t first = __dp2a_lo(sh, 0x0101u, sas[i] + 1u) - __dp2a_lo(s1[i], 0x0101u, 0u);   // and 1; 0: no quadruple
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    s2[i][j] = valid >> (4 * i + j) & 1 ? __dp2a_lo(s2[i][j], 0x0101u, first) : 0u;
                    mine = max(mine, s2[i][j]);
                }
            }
            if (mine > *reinterpret_cast<volatile uint32_t *>(&grp[g].best)) atomicMax(&grp[g].best, mine);
            __syncwarp();
            const uint32_t best = *reinterpret_cast<volatile uint32_t *>(&grp[g].best);
            if (mine && mine + window >= best) {
#pragma unroll
                for (int i = 0; i < 16; i++)
                    if (s2[i / 4][i % 4] && s2[i / 4][i % 4] + window >= best) {
                        const int at = atomicAdd(&grp[g].count, 1);
                        if (at < CAND_MAX) {
                            uint32_t k[4] = {(uint32_t)b, (uint32_t)c, (uint32_t)(A + i / 4), (uint32_t)(D + i % 4)};
                            auto order = [&](int x, int y) { const uint32_t l = min(k[x], k[y]), h = max(k[x], k[y]); k[x] = l; k[y] = h; };
                            order(0, 1); order(2, 3); order(0, 2); order(1, 3); order(1, 2);
                            grp[g].score[at] = s2[i / 4][i % 4];
                            grp[g].key[at] = k[0] << 24 | k[1] << 16 | k[2] << 8 | k[3];
                        }
                    }
            }
        }
    }
    // ---- larger m: a warp takes 32 tasks of one group at a time
    int tasks = 0;                 // (c, b, pair of a, four of d): floor(c^2 / 4) pairs (b, a pair) for every c
    if (M_ == LARGER_M)
        for (int c = 2; c <= m - 2; c++) tasks += (mp / 4 - (c + 1) / 4) * (c * c / 4);
    const int wtasks = (tasks + 31) / 32;
    for (int wt = warp; wt < ng * wtasks; wt += THREADS / 32) {
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
    // ---- exact scores of the candidates: one warp per group.  The rows' terms side by side into the group's part of q, which nobody reads any
    // more, then a lane per candidate adds them up in order.
    for (int g = warp; g < ng; g += THREADS / 32) {
        if (m == 4 || !quantised(g) || grp[g].count > CAND_MAX) continue;
        const uint32_t best = grp[g].best;
        const int count = grp[g].count;
        int close = 0;                                       // those within the window of the final best, moved to the front
        for (int i0 = 0; i0 < count; i0 += 32) {
            const int i = i0 + lane;
            const uint32_t key = i < count ? grp[g].key[i] : 0u;
            const bool on = i < count && grp[g].score[i] + window >= best;
            const uint32_t all = __ballot_sync(0xffffffffu, on);
            if (on) grp[g].key[close + __popc(all & ((1u << lane) - 1u))] = key;
            close += __popc(all);
            __syncwarp();
        }
        float top = -1.0f;
        uint32_t key = 0xFFFFFFFFu;
        if (close == 1) {
            key = grp[g].key[0];
        } else {
            float *terms = reinterpret_cast<float *>(q + (size_t)g * (V / 2) * mp);
            const int held = min(32, mp / 4);                // candidates whose 2V terms fit
            for (int i0 = 0; i0 < close; i0 += held) {
                const int n = min(held, close - i0);
                for (int i = 0; i < n; i++) {
                    const uint32_t k = grp[g].key[i0 + i];
                    const int c[4] = {(int)(k >> 24), (int)(k >> 16 & 255), (int)(k >> 8 & 255), (int)(k & 255)};
                    for (int r = lane; r < V; r += 32) *reinterpret_cast<float2 *>(terms + i * 2 * V + 2 * r) = largest_two(tile + r * p.pitch + g * m, c);
                }
                __syncwarp();
                if (lane < n) {
                    const float4 *x = reinterpret_cast<const float4 *>(terms + lane * 2 * V);
                    float total = 0.0f;
#pragma unroll 8
                    for (int r = 0; r < V / 2; r++) {
                        const float4 v = x[r];
                        total += v.x;
                        total += v.y;
                        total += v.z;
                        total += v.w;
                    }
                    const uint32_t k = grp[g].key[i0 + lane];
                    if (total > top || (total == top && k < key)) { top = total; key = k; }
                }
                __syncwarp();
            }
            for (int o = 16; o > 0; o >>= 1) {
                const float ot = __shfl_xor_sync(0xffffffffu, top, o);
                const uint32_t ok = __shfl_xor_sync(0xffffffffu, key, o);
                if (ot > top || (ot == top && ok < key)) { top = ot; key = ok; }
            }
        }
        if (lane < 4) grp[g].cols[lane] = (int)(key >> (24 - 8 * lane) & 255);
    }
    // ---- exhaustive exact search where integers do not do
    const bool some = tid < ng && !(quantised(tid) && grp[tid].count <= CAND_MAX) && grp[tid].max_bits != 0;
    for (int g = __syncthreads_or(some) ? 0 : ng; g < ng; g++) {
        if (quantised(g) && grp[g].count <= CAND_MAX) continue;      // the same for every thread
        if (grp[g].max_bits == 0) continue;                          // all zero: nothing is kept
        __shared__ float s_best[THREADS];
        __shared__ int s_idx[THREADS];
        float top = 0.0f;
        int at = -1;
        const int ncombo = (int)binom4(m);
        for (int ci = tid; ci < ncombo; ci += THREADS) {
            int c[4];
            unrank4(ci, m, c);
            const float t = exact_score(tile + g * m, p.pitch, V, c);
            if (t > top) { top = t; at = ci; }                       // strict: the first of equal scores stays
        }
        s_best[tid] = top;
        s_idx[tid] = at;
        __syncthreads();
        for (int s = THREADS / 2; s > 0; s >>= 1) {
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
    for (int e = tid; e < gout * 4; e += THREADS) {
        const int g = e >> 2;
        p.colloc[(int64_t)bi * gpad * 4 + (int64_t)g0 * 4 + e] = g < ng && grp[g].cols[0] >= 0 ? (uint32_t)grp[g].cols[e & 3] : 0u;
    }
    if (FUSED) {
        // four rows of a group are one 16-byte piece of the value order; the nibbles of a tile's four groups meet by shuffles
        unsigned int bad = 0;
        const int64_t tiles = p.Ksp / 8;
        const Divisor by_gout(gout);
        for (int e0 = 0; e0 < (V / 4) * gout; e0 += THREADS) {   // gout is a multiple of four: no lane of a tile is left out
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
                        const W *row = tile + (4 * rq + i) * p.pitch + g * m;
                        const float x[4] = {weight(row[cols[0]]), weight(row[cols[1]]), weight(row[cols[2]]), weight(row[cols[3]])};
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
        for (int e = tid; e < V * ng; e += THREADS) {          // kept columns of a row, packed over the quantised tile
            const int r = by_ng.div(e), g = e - r * ng;
            uint32_t kept = 0xFFFFu;
            if (grp[g].cols[0] >= 0) {
                const W *row = tile + r * p.pitch + g * m;
                const float v[4] = {fabsf(weight(row[grp[g].cols[0]])), fabsf(weight(row[grp[g].cols[1]])), fabsf(weight(row[grp[g].cols[2]])), fabsf(weight(row[grp[g].cols[3]]))};
                int i0, i1;
                top2_of4(v, i0, i1);
                kept = (uint32_t)grp[g].cols[i0] | (uint32_t)grp[g].cols[i1] << 8;
            }
            q[e] = kept;
        }
        __syncthreads();
        int32_t *mrow = p.mask + (int64_t)bi * V * p.ldm + (int64_t)g0 * m;
        for (int e = tid; e < V * span; e += THREADS) {
            const int r = by_span.div(e), c = e - r * span, g = by_m.div(c), cc = c - g * m;
            const uint32_t kept = q[r * ng + g];
            mrow[(int64_t)r * p.ldm + c] = cc == (int)(kept & 255) || cc == (int)(kept >> 8);
        }
    }
}

int prune_pitch(int m, int G, int elem) { return (G * m * elem + 15) / 16 * 16 / elem + 16 / elem; }
size_t prune_smem_bytes(int V, int m, int G, int elem)
{
    const int mp = (m + 3) / 4 * 4;
    return (size_t)G * (V / 2) * mp * 4 + (size_t)V * prune_pitch(m, G, elem) * elem + (size_t)G * sizeof(PruneGroup);
}
int prune_groups_per_cta(int m) { return m >= 16 ? 4 : m >= 8 ? 8 : PRUNE_MAX_G; }
bool prune_by_candidates(int V, int m) { return m <= PRUNE_MAX_M && prune_smem_bytes(V, m, prune_groups_per_cta(m), 4) <= 200 * 1024; }

template <int WT, bool FUSED>
cudaError_t launch_candidates(PruneParams p, cudaStream_t stream)
{
    p.one = 1;
    p.mp = (p.m + 3) / 4 * 4;
    p.G = prune_groups_per_cta(p.m);
    p.groups = p.K / p.m;
    const int elem = WT == W_F16 ? 2 : 4;
    p.pitch = prune_pitch(p.m, p.G, elem);
    p.Ksp = ksp_of(p.K, p.m);
    const size_t smem = prune_smem_bytes(p.V, p.m, p.G, elem);
    const unsigned blocks = (unsigned)((p.M / p.V) * ((p.Ksp / 2 + p.G - 1) / p.G));
    // 128 threads: five or six CTAs of an SM are in different phases and their tasks fill the warps better (12288 x 12288, m = 16, V = 32: 2044 us, with
    // 256 threads 2411, before the last change of the loop).  With fewer than four CTAs for each of a B200's 148 SMs 256 (1024 x 1024, m = 32, V = 128: 235, with
    // 128 threads 296); where exactly the line lies was not measured.
    const bool few = blocks < 4 * 148;
    auto launch = [&](auto kernel, int threads) -> cudaError_t {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
        if (e != cudaSuccess) return e;
        kernel<<<blocks, threads, smem, stream>>>(p);
        return cudaGetLastError();
    };
    auto either = [&](auto m_) -> cudaError_t {
        constexpr int M_ = decltype(m_)::value;
        return few ? launch(prune_candidates_kernel<WT, FUSED, M_, 256>, 256) : launch(prune_candidates_kernel<WT, FUSED, M_, 128>, 128);
    };
    switch (p.m) {
    case 8: return either(std::integral_constant<int, 8>());
    case 16: return either(std::integral_constant<int, 16>());
    case 32: return either(std::integral_constant<int, 32>());
    default:
        // larger m: an instance with the registers that its loop needs, and 256 threads: 4096 x 4096, fp32, V = 64, m = 64 22.2 ms (29.2 with 128 threads and
        // the registers of the other loop), fp16, V = 64, m = 40 4.91 (5.52), V = 32, m = 64 29.2 (31.1)
        if (p.m > 4 * TASK_MAX_BLOCKS) return launch(prune_candidates_kernel<WT, FUSED, LARGER_M, 256>, 256);
        return either(std::integral_constant<int, 0>());
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
