// Format kernels: dense -> V:N:M compressor + metadata packer, decompressor, and the re-pack of the
// reference-format arrays into the kernel-private layout.  All are HBM-bound byte/bit shuffles.
#include "vnm_internal.h"

namespace vnm {

// ------------------------------------------------------------------------------------------------
// Compressor, general form (any m, alignment and K, with or without a mask).  A thread owns one group of the 16 rows of a value
// strip; neighbouring lanes own neighbouring groups.  Of every row it loads the four candidate entries only (two bytes each; the
// lanes of a warp cover a contiguous piece of the row, so a sector is fetched once and only if a candidate lies in it), four rows
// at a time, and keeps the first two in ascending order.  The kept pairs of four consecutive rows are one 16-byte piece of the
// reference's value order [sub-block][group][row][slot]; the four lanes of a tile OR their metadata nibbles with shuffles and write
// the strip's 32 bytes of the tile's metadata.  Bound by the sectors fetched (HBM); staging whole rows in shared memory
// instead (the kernel before this one) took 113 us at 12288 x 12280, m = 20, 93 at m = 32, and 398 with a mask at m = 16.
// Follows Format_sr_nm<T>::to_sparse_sr_nm (format_sr_nm.cpp:441-536): candidates with an original
// column >= K contribute a (position 0, value 0) slot for j < 2 only (:486-500).
// ------------------------------------------------------------------------------------------------
constexpr int GATHER_THREADS = 128;
template <bool kHasMask>
__global__ void __launch_bounds__(GATHER_THREADS) compress_gather_kernel(const __half *__restrict__ dense, int64_t ldd, const int32_t *__restrict__ mask,
                                                                         const uint32_t *__restrict__ colloc, int K, int V, int m, int64_t Ksp, uint32_t spans,
                                                                         uint32_t items, int wide, uint32_t *__restrict__ values, uint32_t *__restrict__ meta,
                                                                         unsigned long long *violations)
{
    const int lane = threadIdx.x & 31, gi = lane & 3;
    const int64_t tiles = Ksp / 8;
    unsigned int bad = 0;
    for (uint32_t item = blockIdx.x; item < items; item += gridDim.x) {
        const uint32_t strip = item / spans;
        const int64_t G = (int64_t)(item - strip * spans) * GATHER_THREADS + threadIdx.x;
        const bool on = G < Ksp / 2;              // whole tiles: the four lanes of one agree
        const int64_t T = on ? G >> 2 : 0;
        const int64_t r0 = (int64_t)strip * 16;
        uint32_t cand[4] = {0, 0, 0, 0};
        if (on) {
            const uint4 c4 = __ldg(reinterpret_cast<const uint4 *>(colloc + (r0 / V) * (Ksp / 2) * 4) + G);
            cand[0] = c4.x; cand[1] = c4.y; cand[2] = c4.z; cand[3] = c4.w;
        }
        const int64_t col0 = G * m;
        // a column offset outside its group: nothing of the group is read, its slots are zero and every row counts as a violation
        const bool corrupt = cand[0] >= (uint32_t)m || cand[1] >= (uint32_t)m || cand[2] >= (uint32_t)m || cand[3] >= (uint32_t)m;
        bool inside[4];
#pragma unroll
        for (int j = 0; j < 4; j++) inside[j] = on && !corrupt && col0 + (int64_t)cand[j] < K;
        uint32_t words[8];
        const __half *row = dense + r0 * ldd + col0;
        const int32_t *mrow = kHasMask ? mask + r0 * ldd + col0 : nullptr;
        uint32_t *vdst = values + (r0 * Ksp + T * 128) / 2 + gi * 4;
#pragma unroll
        for (int sb = 0; sb < 4; sb++) {
            unsigned short x[4][4];
            int32_t keep[4][4];
#pragma unroll
            for (int r = 0; r < 4; r++)
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const int64_t at = (int64_t)(sb * 4 + r) * ldd + cand[j];
                    x[r][j] = inside[j] ? __ldg(reinterpret_cast<const unsigned short *>(row) + at) : (unsigned short)0;
                    if (kHasMask) keep[r][j] = inside[j] ? __ldg(mrow + at) : 0;
                }
            uint32_t out[4];
#pragma unroll
            for (int r = 0; r < 4; r++) {
                uint32_t two = 0, nib = 0;
                int pos = 0;
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    if (inside[j]) {
                        if (kHasMask ? keep[r][j] != 0 : (x[r][j] & 0x7FFFu) != 0) {  // value != +-0
                            if (pos < 2) {
                                two |= (uint32_t)x[r][j] << (16 * pos);
                                nib |= (uint32_t)j << (2 * pos);
                            }
                            pos++;
                        }
                    } else if (j < 2) {
                        pos++;   // slot (position 0, value 0): nothing to OR in
                    }
                }
                bad += on && (corrupt || pos != 2);
                out[r] = two;
                // word of rows (2i, 2i + 1) of the strip: 16 bits a row, four a group
                if (r & 1) words[sb * 2 + (r >> 1)] |= nib << (16 + 4 * gi);
                else words[sb * 2 + (r >> 1)] = nib << (4 * gi);
            }
            if (on) {
                if (wide) {
                    *reinterpret_cast<uint4 *>(vdst + sb * 16) = make_uint4(out[0], out[1], out[2], out[3]);
                } else {
#pragma unroll
                    for (int r = 0; r < 4; r++) vdst[sb * 16 + r] = out[r];
                }
            }
        }
#pragma unroll
        for (int w = 0; w < 8; w++) {
            words[w] |= __shfl_xor_sync(0xffffffffu, words[w], 1);
            words[w] |= __shfl_xor_sync(0xffffffffu, words[w], 2);
        }
        if (on) {
            uint32_t *mdst = meta + (int64_t)(strip >> 1) * 16 * tiles + T * 16 + (strip & 1u) * 8 + gi * 2;
            const uint32_t lo = gi == 0 ? words[0] : gi == 1 ? words[2] : gi == 2 ? words[4] : words[6];
            const uint32_t hi = gi == 0 ? words[1] : gi == 1 ? words[3] : gi == 2 ? words[5] : words[7];
            if (wide) {
                *reinterpret_cast<uint2 *>(mdst) = make_uint2(lo, hi);
            } else {
                mdst[0] = lo;
                mdst[1] = hi;
            }
        }
    }
    if (violations != nullptr) {
        bad = __reduce_add_sync(0xffffffffu, bad);
        if (lane == 0 && bad) atomicAdd(violations, (unsigned long long)bad);
    }
}

// ------------------------------------------------------------------------------------------------
// Compressor, register form, for the common shapes: no mask, m in {4, 8, 16}, K % (4 * m) == 0 (whole tiles, no
// padded group), V a multiple of 16 and 16-byte aligned rows.  The lanes of a warp lie ALONG a row: a thread owns 16
// bytes of the row or one group, whichever is larger (two groups for m = 4, one for m = 8 and 16), so a load instruction
// of a warp reads 512 contiguous bytes (1 KiB for m = 16).  The thread walks the 16 rows of a value strip four at a
// time: for its group the kept pairs of four consecutive rows are exactly one 16-byte piece of the reference's value
// order [sub-block][group][row][slot], so it is stored straight from registers, without any exchange between lanes; the
// candidates' select predicates depend on the column-loc entry only and are shared by the 16 rows.  The lanes of a tile
// (4, or 2 for m = 4) OR their metadata nibbles together with shuffles and write the strip's 32 bytes of the tile's
// metadata as one sector.  A CTA (8 warps) covers 16 rows x 4 KiB (8 KiB for m = 16); the grid is one resident wave
// and walks the items in row-major order, so neighbouring CTAs read neighbouring pieces of the same rows.
// ------------------------------------------------------------------------------------------------
// m = 8 fits 64 registers without spilling (four CTAs per SM: measured 11 % faster than three); m = 4 and 16 do not
template <int M_>
__global__ void __launch_bounds__(256, M_ == 8 ? 4 : 1) compress_direct_kernel(const __half *__restrict__ dense, int64_t ldd, const uint32_t *__restrict__ colloc,
                                                              int V, int tiles, uint32_t spans, uint32_t items, uint32_t *__restrict__ values,
                                                              uint32_t *__restrict__ meta, unsigned long long *violations)
{
    constexpr int NW = M_ / 2;             // 32-bit words per group
    constexpr int GPT = M_ == 4 ? 2 : 1;   // groups per thread
    constexpr int TW = GPT * NW;           // words per thread and row (4, 4, 8)
    constexpr int LPR = TW / 4;            // 16-byte loads per thread and row
    constexpr int TL = 4 / GPT;            // lanes per tile
    constexpr int TPW = 32 / TL;           // tiles per warp
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int tli = lane % TL, g0 = tli * GPT;   // this thread's first group inside its tile
    const int64_t Ksp = (int64_t)tiles * 8;
    unsigned int bad = 0;
    // where the thread's 16 rows start for an item (lanes past the last tile repeat it: they take part in the shuffles)
    auto row0_of = [&](uint32_t item) {
        const uint32_t strip = item / spans;
        const int t = (int)(item - strip * spans) * (8 * TPW) + warp * TPW + lane / TL;
        const int T = t < tiles ? t : tiles - 1;
        return dense + (int64_t)strip * 16 * ldd + ((int64_t)T * 4 + g0) * M_;
    };
    auto load4 = [&](const __half *row0, int sb, uint32_t (&w)[4][TW]) {   // rows 4*sb .. 4*sb+3
#pragma unroll
        for (int r = 0; r < 4; r++) {
            const uint4 *src = reinterpret_cast<const uint4 *>(row0 + (int64_t)(sb * 4 + r) * ldd);
#pragma unroll
            for (int i = 0; i < LPR; i++) {
                const uint4 v = __ldg(src + i);
                w[r][4 * i] = v.x; w[r][4 * i + 1] = v.y; w[r][4 * i + 2] = v.z; w[r][4 * i + 3] = v.w;
            }
        }
    };
    // The loads run one step (four rows) ahead of the arithmetic, across item boundaries: two register buffers
    uint32_t wa[4][TW], wb[4][TW];
    const __half *row0 = blockIdx.x < items ? row0_of(blockIdx.x) : dense;
    if (blockIdx.x < items) load4(row0, 0, wa);
    for (uint32_t item = blockIdx.x; item < items; item += gridDim.x) {
        const uint32_t strip = item / spans;
        const int t = (int)(item - strip * spans) * (8 * TPW) + warp * TPW + lane / TL;
        const bool valid = t < tiles;          // whole tiles: the lanes of a tile are valid together
        const int T = valid ? t : tiles - 1;
        const int64_t G = (int64_t)T * 4 + g0; // first group of this thread in its row
        const __half *next_row0 = item + gridDim.x < items ? row0_of(item + gridDim.x) : row0;
        // candidates of the thread's groups: the same for the 16 rows (V % 16 == 0)
        uint32_t cand[GPT][4];
        uint32_t okmask[GPT];   // 0 for a group whose column-loc entry is corrupt (an offset outside the group): every row counts a violation
        {
            const uint4 *c4p = reinterpret_cast<const uint4 *>(colloc + ((int64_t)(strip * 16u / (uint32_t)V) * (Ksp / 2) + G) * 4);
#pragma unroll
            for (int j = 0; j < GPT; j++) {
                const uint4 c4 = __ldg(c4p + j);
                const bool corrupt = max(max(c4.x, c4.y), max(c4.z, c4.w)) >= (uint32_t)M_;
                okmask[j] = corrupt ? 0u : 0xFFFFFFFFu;
                cand[j][0] = c4.x & okmask[j]; cand[j][1] = c4.y & okmask[j]; cand[j][2] = c4.z & okmask[j]; cand[j][3] = c4.w & okmask[j];
            }
        }
        uint4 *vdst = reinterpret_cast<uint4 *>(values) + ((int64_t)strip * 16 * Ksp + (int64_t)T * 128) / 8 + g0;
        uint32_t keep[4] = {0, 0, 0, 0};   // metadata words this lane stores at the end: 2 (TL = 4) or 4 (TL = 2)
        auto work = [&](int sb, const uint32_t (&w)[4][TW]) {
            uint32_t hw[4] = {0, 0, 0, 0};   // per row: the metadata nibbles of this thread's groups, at their place in the tile's 16 bits
#pragma unroll
            for (int j = 0; j < GPT; j++) {
                uint32_t out[4];
#pragma unroll
                for (int r = 0; r < 4; r++) {
                    const uint32_t *wg = &w[r][j * NW];
                    uint32_t h[4];
                    bool nz[4];
#pragma unroll
                    for (int c = 0; c < 4; c++) {
                        const uint32_t cc = cand[j][c];
                        // half cc of the group's NW words: a binary select tree down to a pair of words, then one byte permute
                        uint32_t lo, hi;
                        if (NW == 2) {
                            lo = wg[0]; hi = wg[1];
                        } else if (NW == 4) {
                            const bool up = (cc & 4u) != 0;
                            lo = up ? wg[2] : wg[0];
                            hi = up ? wg[3] : wg[1];
                        } else {
                            const bool up8 = (cc & 8u) != 0, up4 = (cc & 4u) != 0;
                            const uint32_t a0 = up8 ? wg[4] : wg[0], a1 = up8 ? wg[5] : wg[1];
                            const uint32_t a2 = up8 ? wg[6] : wg[2], a3 = up8 ? wg[7] : wg[3];
                            lo = up4 ? a2 : a0;
                            hi = up4 ? a3 : a1;
                        }
                        const uint32_t h2 = (cc & 3u) * 2u;
                        h[c] = __byte_perm(lo, hi, ((h2 + 1u) << 4) | h2);   // the half in the low 16 bits (the upper 16 are not used)
                        nz[c] = (h[c] & 0x7FFFu) != 0;                                // kept entries are the non-zero values
                    }
                    // exactly two candidates are non-zero in a valid matrix: the first from the front and the first from the back
                    const uint32_t v0 = nz[0] ? h[0] : (nz[1] ? h[1] : h[2]), i0 = nz[0] ? 0u : (nz[1] ? 1u : 2u);
                    const uint32_t v1 = nz[3] ? h[3] : (nz[2] ? h[2] : h[1]), i1 = nz[3] ? 3u : (nz[2] ? 2u : 1u);
                    const int cnt = (int)nz[0] + (int)nz[1] + (int)nz[2] + (int)nz[3];
                    const bool good = cnt == 2 && okmask[j] != 0;
                    bad += (valid && !good);
                    // fewer than two kept entries leave zeros in the open slots, more than two keep the first two (as the scalar form does)
                    uint32_t o, nib;
                    if (cnt == 2) {
                        o = __byte_perm(v0, v1, 0x5410u);   // low halves of both
                        nib = i0 | (i1 << 2);
                    } else {
                        o = 0; nib = 0;
                        int pos = 0;
#pragma unroll
                        for (int c = 0; c < 4; c++)
                            if (nz[c]) {
                                if (pos < 2) { o |= (h[c] & 0xFFFFu) << (16 * pos); nib |= (uint32_t)c << (pos * 2); }
                                pos++;
                            }
                    }
                    out[r] = o & okmask[j];
                    hw[r] |= (nib & okmask[j]) << ((g0 + j) * 4);
                }
                // rows 4*sb .. 4*sb+3 of group g0 + j: one 16-byte piece of [sub-block][group][row][slot]
                if (valid) vdst[sb * 4 + j] = make_uint4(out[0], out[1], out[2], out[3]);
            }
            // the tile's 16 metadata bits per row, two rows per word: OR over the lanes of the tile
            uint32_t m01 = hw[0] | (hw[1] << 16), m23 = hw[2] | (hw[3] << 16);
#pragma unroll
            for (int o = 1; o < TL; o <<= 1) {
                m01 |= __shfl_xor_sync(0xffffffffu, m01, o);
                m23 |= __shfl_xor_sync(0xffffffffu, m23, o);
            }
            if (TL == 4) {
                if (tli == sb) { keep[0] = m01; keep[1] = m23; }
            } else {
                if (tli == (sb >> 1)) { keep[(sb & 1) * 2] = m01; keep[(sb & 1) * 2 + 1] = m23; }
            }
        };
        load4(row0, 1, wb);
        work(0, wa);
        load4(row0, 2, wa);
        work(1, wb);
        load4(row0, 3, wb);
        work(2, wa);
        load4(next_row0, 0, wa);   // the next item's first rows (the last item loads its own again: in bounds, unused)
        work(3, wb);
        row0 = next_row0;
        // the strip's half of the tile's 16 metadata words (rows 16*(strip & 1) ..): 32 bytes, one sector per tile
        uint32_t *mdst = meta + (int64_t)(strip >> 1) * 16 * tiles + (int64_t)T * 16 + (strip & 1u) * 8;
        if (valid) {
            if (TL == 4) *reinterpret_cast<uint2 *>(mdst + tli * 2) = make_uint2(keep[0], keep[1]);
            else *reinterpret_cast<uint4 *>(mdst + tli * 4) = make_uint4(keep[0], keep[1], keep[2], keep[3]);
        }
    }
    if (violations != nullptr) {
        for (int o = 16; o > 0; o >>= 1) bad += __shfl_xor_sync(0xffffffffu, bad, o);
        if (lane == 0 && bad) atomicAdd(violations, (unsigned long long)bad);
    }
}

// one resident wave of the register-form compressor on the current device (cached per kernel and device)
template <int M_>
static int compress_direct_wave()
{
    static int cached[64] = {0};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) dev = 0;
    if (cached[dev] == 0) {
        int per_sm = 0, sms = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, compress_direct_kernel<M_>, 256, 0);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        cached[dev] = (per_sm > 0 && sms > 0) ? per_sm * sms : 148 * 4;
    }
    return cached[dev];
}

cudaError_t launch_compress(const void *dense, int64_t ldd, const int32_t *mask, const uint32_t *colloc, int M, int K, int V, int m,
                            void *values, uint32_t *meta, unsigned long long *violations, cudaStream_t stream)
{
    const int64_t Ksp = ksp_of(K, m);
    const int threads = 256;
    // register form: no mask, whole tiles, 16-byte aligned rows and outputs
    if (!mask && (m == 4 || m == 8 || m == 16) && K % (4 * m) == 0 && Ksp == (int64_t)K / m * 2 && M % 16 == 0 && V % 16 == 0 && ldd % 8 == 0 &&
        ((uintptr_t)dense & 15) == 0 && ((uintptr_t)values & 15) == 0 && ((uintptr_t)colloc & 15) == 0 && ((uintptr_t)meta & 15) == 0) {
        const int tiles = (int)(Ksp / 8);
        const int tiles_per_item = m == 4 ? 8 * 16 : 8 * 8;   // 8 warps x tiles per warp
        const int64_t spans = (tiles + tiles_per_item - 1) / tiles_per_item, items = (int64_t)(M / 16) * spans;
        if (items < ((int64_t)1 << 31)) {
            const int wave = m == 4 ? compress_direct_wave<4>() : m == 8 ? compress_direct_wave<8>() : compress_direct_wave<16>();
            const unsigned blocks = items < wave ? (unsigned)items : (unsigned)wave;
            if (m == 4)
                compress_direct_kernel<4><<<blocks, threads, 0, stream>>>((const __half *)dense, ldd, colloc, V, tiles, (uint32_t)spans, (uint32_t)items, (uint32_t *)values, meta, violations);
            else if (m == 8)
                compress_direct_kernel<8><<<blocks, threads, 0, stream>>>((const __half *)dense, ldd, colloc, V, tiles, (uint32_t)spans, (uint32_t)items, (uint32_t *)values, meta, violations);
            else
                compress_direct_kernel<16><<<blocks, threads, 0, stream>>>((const __half *)dense, ldd, colloc, V, tiles, (uint32_t)spans, (uint32_t)items, (uint32_t *)values, meta, violations);
            return cudaGetLastError();
        }
    }
    const int64_t spans = (Ksp / 2 + GATHER_THREADS - 1) / GATHER_THREADS, items = (int64_t)(M / 16) * spans;
    if (items >= ((int64_t)1 << 32)) return cudaErrorInvalidValue;
    const unsigned blocks = (unsigned)(items < (1 << 20) ? items : (1 << 20));
    const int wide = ((uintptr_t)values & 15) == 0 && ((uintptr_t)meta & 7) == 0;
    if (mask)
        compress_gather_kernel<true><<<blocks, GATHER_THREADS, 0, stream>>>((const __half *)dense, ldd, mask, colloc, K, V, m, Ksp, (uint32_t)spans, (uint32_t)items, wide,
                                                                            (uint32_t *)values, meta, violations);
    else
        compress_gather_kernel<false><<<blocks, GATHER_THREADS, 0, stream>>>((const __half *)dense, ldd, mask, colloc, K, V, m, Ksp, (uint32_t)spans, (uint32_t)items, wide,
                                                                             (uint32_t *)values, meta, violations);
    return cudaGetLastError();
}

// ------------------------------------------------------------------------------------------------
// Decompressor, general form (Format_sr_nm<T>::to_dense, format_sr_nm.cpp:327-417).  The output is zero-filled by
// the caller side of the launch; one thread scatters the two values of one (row, group), slot 0
// first, so a padded slot overwrites exactly as the reference's loop order does.
// ------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) decompress_kernel(const __half *__restrict__ values, const uint32_t *__restrict__ meta,
                                                         const uint32_t *__restrict__ colloc, int M, int K, int V, int m, int64_t Ksp,
                                                         __half *__restrict__ dense, int64_t ldd)
{
    const int64_t G = Ksp / 2;
    const int64_t total = (int64_t)M * G;
    for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += (int64_t)gridDim.x * blockDim.x) {
        const int64_t r = idx / G;
        const int64_t g = idx - r * G;
        const uint32_t w = meta[meta_index(r, g, Ksp)];
        const uint32_t *c4 = colloc + (r / V) * G * 4 + g * 4;
#pragma unroll
        for (int s = 0; s < 2; s++) {
            const uint32_t sel = (w >> meta_shift(r, g, s)) & 3u;
            const int64_t col = g * m + (int64_t)c4[sel];
            if (col < K) dense[r * ldd + col] = values[values_index(r, g, s, Ksp)];
        }
    }
}

// ------------------------------------------------------------------------------------------------
// Tiled decompressor (m not a multiple of four, or rows aligned to two bytes only):  A CTA takes 32 rows x
// TS tiles: the values (TS * 256 contiguous bytes per 16 rows) and metadata (TS * 64 bytes) come in with 16-byte
// loads, lane = row / warp = tile scatters the two values of every (row, group) into a zeroed shared-memory image
// of the 32 dense row segments (slot 0 first, like the general kernel), and the image leaves with 8-byte stores.
// Every output element is written exactly once, so no memset pass is needed.
// ------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) decompress_tiled_kernel(const uint32_t *__restrict__ values, const uint32_t *__restrict__ meta,
                                                               const uint32_t *__restrict__ colloc, int M, int K, int V, int m, int64_t Ksp, int TS,
                                                               __half *__restrict__ dense, int64_t ldd)
{
    extern __shared__ __align__(16) uint8_t csm[];
    const int span = TS * 4 * m;
    const int pitch = span + 4;  // halves; rows 8-byte aligned, pitch / 2 = 2 mod 32
    uint32_t *val_s = reinterpret_cast<uint32_t *>(csm);                 // [2][TS][64]
    uint32_t *meta_s = val_s + 2 * TS * 64;                              // [TS][16]
    unsigned short *out_s = reinterpret_cast<unsigned short *>(meta_s + TS * 16);  // [32][pitch]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t tiles = Ksp / 8;
    const int spans = (int)((tiles + TS - 1) / TS);
    const int64_t chunks = (int64_t)(M / 32) * spans;
    for (int64_t ch = blockIdx.x; ch < chunks; ch += gridDim.x) {
        const int64_t rc = ch / spans;
        const int sp = (int)(ch - rc * spans);
        const int64_t R0 = rc * 32;
        const int64_t t0 = (int64_t)sp * TS;
        const int tcount = (int)(tiles - t0 < TS ? tiles - t0 : TS);
        const int64_t c0 = t0 * 4 * m;
        const int valid = (int)(c0 >= K ? 0 : (K - c0 < span ? K - c0 : span));
        // ---- compressed arrays -> shared memory, dense image zeroed
        const int vq = tcount * 16;
        for (int i = threadIdx.x; i < 2 * vq; i += 256) {
            const int rg = i >= vq ? 1 : 0;
            const int k = i - rg * vq;
            reinterpret_cast<uint4 *>(val_s + rg * TS * 64)[k] = __ldg(reinterpret_cast<const uint4 *>(values + ((R0 / 16 + rg) * 16 * Ksp + t0 * 128) / 2) + k);
        }
        for (int i = threadIdx.x; i < tcount * 4; i += 256)
            reinterpret_cast<uint4 *>(meta_s)[i] = __ldg(reinterpret_cast<const uint4 *>(meta + (R0 / 32) * 16 * tiles + t0 * 16) + i);
        for (int i = threadIdx.x; i < 32 * pitch / 4; i += 256) reinterpret_cast<uint2 *>(out_s)[i] = make_uint2(0u, 0u);
        __syncthreads();
        // ---- lane = row, warp = tile
        const uint32_t *crow = colloc + (R0 / V) * (Ksp / 2) * 4;
        unsigned short *my_out = out_s + lane * pitch;
        for (int tl = warp; tl < tcount; tl += 8) {
            const uint32_t hw = (meta_s[tl * 16 + (lane >> 1)] >> ((lane & 1) * 16)) & 0xFFFFu;
            const uint32_t *vsrc = val_s + ((lane >> 4) * TS + tl) * 64 + ((lane & 15) >> 2) * 16 + (lane & 3);
            const uint4 *c4p = reinterpret_cast<const uint4 *>(crow + (t0 + tl) * 16);
#pragma unroll
            for (int gi = 0; gi < 4; gi++) {
                const uint4 c4 = __ldg(c4p + gi);
                const int cand[4] = {(int)c4.x, (int)c4.y, (int)c4.z, (int)c4.w};
                const int lg = (tl * 4 + gi) * m;
                const uint32_t two = vsrc[gi * 4];
#pragma unroll
                for (int sl = 0; sl < 2; sl++) {
                    const int sel = (int)((hw >> (gi * 4 + sl * 2)) & 3u);
                    const int lc = lg + (sel == 0 ? cand[0] : sel == 1 ? cand[1] : sel == 2 ? cand[2] : cand[3]);
                    if (lc < valid) my_out[lc] = (unsigned short)(two >> (16 * sl));
                }
            }
        }
        __syncthreads();
        // ---- dense image -> global memory
        const int nq = valid / 4;  // whole 8-byte pieces per row
        for (int r = warp; r < 32; r += 8) {
            __half *drow = dense + (R0 + r) * ldd + c0;
            const unsigned short *srow = out_s + r * pitch;
            for (int q = lane; q < nq; q += 32) reinterpret_cast<uint2 *>(drow)[q] = reinterpret_cast<const uint2 *>(srow)[q];
            for (int c = nq * 4 + lane; c < valid; c += 32) drow[c] = __ushort_as_half(srow[c]);
        }
        __syncthreads();
    }
}

// ------------------------------------------------------------------------------------------------
// Decompressor, piece form, for m a multiple of 8 (PW = 8) or of 4 (PW = 4) and rows aligned to PW halves: lanes lie along the
// OUTPUT row.  A thread owns PW consecutive columns, all of one group, of the 16 rows of a strip; the m / PW threads of a group
// load the same values and metadata (one sector for all of them) and each keeps the slots that fall into its columns.
// Every store instruction of a warp writes 512 contiguous bytes (256 for PW = 4).  Bound by HBM writes: 12288 x 12288, m = 16
// takes 60 us (floor 54); through the tiled kernel (shared-memory scatter, two barriers a chunk) it took 78.  A thread per group instead of
// a piece (m = 8: the same; m = 4: two groups) in one resident wave took 76 us at m = 8 and 96 at m = 4, against 68 and 84.
// ------------------------------------------------------------------------------------------------
template <int PW>
__global__ void __launch_bounds__(256) decompress_piece_kernel(const uint32_t *__restrict__ values, const uint32_t *__restrict__ meta,
                                                               const uint32_t *__restrict__ colloc, int K, int V, int m, int64_t Ksp, uint32_t spans,
                                                               uint32_t items, __half *__restrict__ dense, int64_t ldd)
{
    constexpr int NW = PW / 2;
    const int64_t tiles = Ksp / 8;
    for (uint32_t item = blockIdx.x; item < items; item += gridDim.x) {
        const uint32_t strip = item / spans;
        const int col = (int)((item - strip * spans) * 256u + threadIdx.x) * PW;
        if (col >= K) continue;
        const int G = col / m, o = col - G * m;
        const int T = G >> 2, g0 = G & 3;
        const uint4 c4 = __ldg(reinterpret_cast<const uint4 *>(colloc + ((int64_t)(strip * 16u / (uint32_t)V) * (Ksp / 2) + G) * 4));
        const uint32_t cand = (c4.x & 0xFFu) | ((c4.y & 0xFFu) << 8) | ((c4.z & 0xFFu) << 16) | ((c4.w & 0xFFu) << 24);
        const uint4 *vsrc = reinterpret_cast<const uint4 *>(values) + ((int64_t)strip * 16 * Ksp + (int64_t)T * 128) / 8 + g0;
        const uint4 *msrc = reinterpret_cast<const uint4 *>(meta + (int64_t)(strip >> 1) * 16 * tiles + (int64_t)T * 16 + (strip & 1u) * 8);
        uint4 vals[4];
#pragma unroll
        for (int sb = 0; sb < 4; sb++) vals[sb] = __ldg(vsrc + sb * 4);
        const uint4 ma = __ldg(msrc), mb = __ldg(msrc + 1);
        const uint32_t mw[8] = {ma.x, ma.y, ma.z, ma.w, mb.x, mb.y, mb.z, mb.w};   // word 2*sb + (r >> 1): rows r, r+1 of sub-block sb
        __half *dst = dense + (int64_t)strip * 16 * ldd + col;
#pragma unroll
        for (int sb = 0; sb < 4; sb++) {
#pragma unroll
            for (int r = 0; r < 4; r++) {
                const uint32_t nib = mw[sb * 2 + (r >> 1)] >> ((r & 1) * 16 + g0 * 4);
                const uint32_t two = r == 0 ? vals[sb].x : r == 1 ? vals[sb].y : r == 2 ? vals[sb].z : vals[sb].w;
                // columns of the two slots inside the piece (no word of it matches a slot that lies outside)
                const int p0 = (int)__byte_perm(cand, 0u, 0x4440u | (nib & 3u)) - o, p1 = (int)__byte_perm(cand, 0u, 0x4440u | ((nib >> 2) & 3u)) - o;
                const int w0 = p0 >> 1, w1 = p1 >> 1;
                const uint32_t x0 = (p0 & 1) ? two << 16 : two & 0xFFFFu;
                const uint32_t x1 = (p1 & 1) ? two & 0xFFFF0000u : two >> 16, keep = (p1 & 1) ? 0xFFFFu : 0xFFFF0000u;
                uint32_t w[NW];
#pragma unroll
                for (int k = 0; k < NW; k++) {
                    w[k] = w0 == k ? x0 : 0u;
                    if (w1 == k) w[k] = (w[k] & keep) | x1;   // slot 1 after slot 0: a padded slot overwrites, as in the general kernel
                }
                if constexpr (PW == 8) *reinterpret_cast<uint4 *>(dst) = make_uint4(w[0], w[1], w[2], w[3]);
                else *reinterpret_cast<uint2 *>(dst) = make_uint2(w[0], w[1]);
                dst += ldd;
            }
        }
    }
}

cudaError_t launch_decompress(const void *values, const uint32_t *meta, const uint32_t *colloc, int M, int K, int V, int m,
                              void *dense, int64_t ldd, cudaStream_t stream)
{
    const int64_t Ksp = ksp_of(K, m);
    const bool arrays_aligned = M % 16 == 0 && V % 16 == 0 && ((uintptr_t)values & 15) == 0 && ((uintptr_t)colloc & 15) == 0 && ((uintptr_t)meta & 15) == 0;
    // piece form: a piece never straddles groups or the end of a row
    const int pw = m % 8 == 0 && K % 8 == 0 && ldd % 8 == 0 && ((uintptr_t)dense & 15) == 0 ? 8 : m % 4 == 0 && K % 4 == 0 && ldd % 4 == 0 && ((uintptr_t)dense & 7) == 0 ? 4 : 0;
    if (arrays_aligned && pw && m <= 256) {
        const int64_t spans = (K / pw + 255) / 256, items = (int64_t)(M / 16) * spans;
        if (items < ((int64_t)1 << 31)) {
            const unsigned blocks = (unsigned)(items < (1 << 20) ? items : (1 << 20));
            if (pw == 8)
                decompress_piece_kernel<8><<<blocks, 256, 0, stream>>>((const uint32_t *)values, meta, colloc, K, V, m, Ksp, (uint32_t)spans, (uint32_t)items, (__half *)dense, ldd);
            else
                decompress_piece_kernel<4><<<blocks, 256, 0, stream>>>((const uint32_t *)values, meta, colloc, K, V, m, Ksp, (uint32_t)spans, (uint32_t)items, (__half *)dense, ldd);
            return cudaGetLastError();
        }
    }
    const bool aligned = ldd % 4 == 0 && ((uintptr_t)dense & 7) == 0 && ((uintptr_t)values & 15) == 0 && ((uintptr_t)meta & 15) == 0 &&
                         m <= 128 && M % 32 == 0 && V % 32 == 0;
    if (aligned) {
        const int TS = m >= 128 ? 1 : (m <= 8 ? 16 : 128 / m);
        const int span = TS * 4 * m;
        const size_t smem = (size_t)(2 * TS * 64 + TS * 16) * 4 + (size_t)32 * (span + 4) * 2;
        const int64_t chunks = (int64_t)(M / 32) * ((Ksp / 8 + TS - 1) / TS);
        int64_t blocks = chunks < (int64_t)148 * 5 ? chunks : (int64_t)148 * 5;
        if (blocks < 1) blocks = 1;
        cudaError_t e = cudaFuncSetAttribute(decompress_tiled_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 96 * 1024);
        if (e != cudaSuccess) return e;
        decompress_tiled_kernel<<<(unsigned)blocks, 256, smem, stream>>>((const uint32_t *)values, meta, colloc, M, K, V, m, Ksp, TS,
                                                                         (__half *)dense, ldd);
        return cudaGetLastError();
    }
    cudaError_t e = cudaMemset2DAsync(dense, (size_t)ldd * 2, 0, (size_t)K * 2, (size_t)M, stream);
    if (e != cudaSuccess) return e;
    const int64_t total = (int64_t)M * (Ksp / 2);
    int64_t blocks = (total + 255) / 256;
    const int64_t cap = (int64_t)148 * 64;
    if (blocks > cap) blocks = cap;
    decompress_kernel<<<(unsigned)blocks, 256, 0, stream>>>((const __half *)values, meta, colloc, M, K, V, m, Ksp, (__half *)dense, ldd);
    return cudaGetLastError();
}

// ------------------------------------------------------------------------------------------------
// Re-pack into the kernel-private layout (see vnm_common.cuh).  One thread writes one 16-byte chunk:
// chunks [0, 1024) of a block are the swizzled value image, chunks [1024, 1152) the metadata image.
// ------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) prepare_am_kernel(const __half *__restrict__ values, const uint32_t *__restrict__ meta, int M,
                                                         int64_t Ksp, int mtiles, int ktiles, uint4 *__restrict__ am)
{
    const int chunks_per_block = AM_BLOCK_BYTES / 16;  // 1152
    const int64_t total = (int64_t)mtiles * ktiles * chunks_per_block;
    for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += (int64_t)gridDim.x * blockDim.x) {
        const int64_t blk = idx / chunks_per_block;
        const int ch = (int)(idx - blk * chunks_per_block);
        const int mt = (int)(blk / ktiles);
        const int kt = (int)(blk - (int64_t)mt * ktiles);
        uint4 o = make_uint4(0, 0, 0, 0);
        if (ch < A_IMG_BYTES / 16) {
            const int i = ch >> 3;                  // MMA row inside the tile
            const int cphys = ch & 7;               // stored chunk
            const int c = cphys ^ (i & 7);          // logical chunk = 8 compressed columns = one reference tile
            const int64_t r = (int64_t)mt * TILE_M + mma_row_to_actual(i);
            const int64_t t = (int64_t)kt * 8 + c;  // reference tile index (four groups)
            if (r < M && t < Ksp / 8) {
                const __half *src = values + (r / 16) * 16 * Ksp + t * 128 + ((r % 16) / 4) * 32 + (r % 4) * 2;
                uint32_t w[4];
#pragma unroll
                for (int gi = 0; gi < 4; gi++) w[gi] = *reinterpret_cast<const uint32_t *>(src + gi * 8);
                o = make_uint4(w[0], w[1], w[2], w[3]);
            }
        } else {
            const int lane = ch - A_IMG_BYTES / 16;  // tensor-memory lane 0..127
            const int m0 = lane & 7, k1 = (lane >> 3) & 1, m2 = lane >> 4;
            const int64_t r = (int64_t)mt * TILE_M + m2 * 16 + m0 * 2;  // even row of the pair
            uint32_t w[4];
#pragma unroll
            for (int kb = 0; kb < 4; kb++) {
                const int64_t t = (int64_t)kt * 8 + kb * 2 + k1;
                // padding: positions (0,1) in every group, a valid 2:4 pattern for zero values
                w[kb] = (r < M && t < Ksp / 8) ? meta[(r / 32) * 16 * (Ksp / 8) + t * 16 + (r % 32) / 2] : 0x44444444u;
            }
            o = make_uint4(w[0], w[1], w[2], w[3]);
        }
        am[idx] = o;
    }
}

// Absolute B rows per (V-block, group); groups are padded to whole k-tiles and V-blocks to whole row tiles.
__global__ void __launch_bounds__(256) prepare_rows_kernel(const uint32_t *__restrict__ colloc, int M, int K, int V, int m, int64_t Ksp,
                                                           int vblocks_padded, int ktiles, int4 *__restrict__ rows)
{
    const int64_t gpad = (int64_t)ktiles * KT_GROUPS;
    const int64_t total = (int64_t)vblocks_padded * gpad;
    for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += (int64_t)gridDim.x * blockDim.x) {
        const int64_t vb = idx / gpad;
        const int64_t g = idx - vb * gpad;
        int4 o = make_int4(K, K, K, K);
        if (vb < M / V && g < Ksp / 2) {
            const uint4 c4 = *reinterpret_cast<const uint4 *>(colloc + vb * (Ksp / 2) * 4 + g * 4);
            const int64_t base = g * m;
            const int64_t a = base + c4.x, b = base + c4.y, c = base + c4.z, d = base + c4.w;
            o.x = a < K ? (int)a : K;
            o.y = b < K ? (int)b : K;
            o.z = c < K ? (int)c : K;
            o.w = d < K ? (int)d : K;
        }
        rows[idx] = o;
    }
}

// ------------------------------------------------------------------------------------------------
// "Dense-B" re-pack: the V:2:m pattern re-expressed as plain 2:4 over ALL K columns.
// A row keeps two entries per group of m columns, so any aligned chunk of four original columns
// (m % 4 == 0: chunks never straddle groups) holds at most two of them -- a valid 2:4 pattern once the
// missing slots are filled with explicit zeros.  The product can then read B as ordinary 64-row tiles
// that every vector block shares (no per-block gather, no lane masks), at the price of m/4 times the MMA
// work.  Same block format as prepare_am_kernel, but a k-tile now covers 128 ORIGINAL columns.
// One thread handles one (row pair, 16 original columns): two 16-byte value chunks and one metadata word.  The column-loc, the values and
// the metadata of a group are loaded once for both rows and all of its chunks in the slab (loading them per row, chunk and slot took
// 436 us at 12288 x 12288, 128:2:8, against 165 now).
// ------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) prepare_dense_b_kernel(const __half *__restrict__ values, const uint32_t *__restrict__ meta,
                                                              const uint32_t *__restrict__ colloc, int M, int K, int V, int m, int64_t Ksp,
                                                              int mtiles, int ktiles, uint8_t *__restrict__ am)
{
    const int64_t total = (int64_t)mtiles * ktiles * 64 * 8;
    for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += (int64_t)gridDim.x * blockDim.x) {
        const int q = (int)(idx & 7);          // 16-column slab of the 128-column k-tile
        const int pr = (int)((idx >> 3) & 63);  // row pair inside the 128-row tile
        const uint32_t blk = (uint32_t)(idx >> 9);
        const int mt = (int)(blk / (uint32_t)ktiles);
        const int kt = (int)(blk - (uint32_t)mt * (uint32_t)ktiles);
        uint8_t *block = am + (size_t)blk * AM_BLOCK_BYTES;
        uint32_t word = 0;
        const int i0 = actual_to_mma_row(2 * pr);  // MMA row of the even row; the odd row sits 8 rows further
        const int64_t r0 = (int64_t)mt * TILE_M + 2 * pr;
        unsigned short v8[2][8] = {{0, 0, 0, 0, 0, 0, 0, 0}, {0, 0, 0, 0, 0, 0, 0, 0}};
        int cb = kt * 128 + q * 16;                // first original column of the chunk
        int g = cb / m, o0 = cb - g * m;
        uint4 c4 = make_uint4(0, 0, 0, 0);
        uint2 two = make_uint2(0, 0);              // slots 0 and 1 of the even row, of the odd row
        uint32_t w = 0;
        bool fresh = true;                         // the group's words are still to be loaded
#pragma unroll
        for (int c = 0; c < 4; c++) {
            const bool in = r0 < M && cb < K;
            if (in && fresh) {
                c4 = __ldg(reinterpret_cast<const uint4 *>(colloc + (r0 / V) * (Ksp / 2) * 4) + g);
                const uint32_t *v = reinterpret_cast<const uint32_t *>(values + values_index(r0, g, 0, Ksp));   // 4-byte aligned at least
                two = make_uint2(__ldg(v), __ldg(v + 1));
                w = __ldg(meta + meta_index(r0, g, Ksp));
            }
#pragma unroll
            for (int h = 0; h < 2; h++) {
                int npos = 0;
                uint32_t pos[2] = {0, 1};
                unsigned short val[2] = {0, 0};
                if (in) {
                    const uint32_t nib = w >> meta_shift(r0 + h, g, 0), v2 = h ? two.y : two.x;
#pragma unroll
                    for (int sl = 0; sl < 2; sl++) {
                        const uint32_t sel = (nib >> (2 * sl)) & 3u;
                        const int off = (int)(sel == 0 ? c4.x : sel == 1 ? c4.y : sel == 2 ? c4.z : c4.w) - o0;
                        if (off >= 0 && off < 4 && cb + off < K) {
                            const unsigned short x = (unsigned short)(v2 >> (16 * sl));
                            if (npos == 0) { pos[0] = (uint32_t)off; val[0] = x; }
                            else { pos[1] = (uint32_t)off; val[1] = x; }
                            npos++;
                        }
                    }
                }
                if (npos == 1) {  // partner slot with an explicit zero, positions kept ascending
                    if (pos[0] == 3) { pos[1] = 3; pos[0] = 2; val[1] = val[0]; val[0] = 0; }
                    else { pos[1] = pos[0] + 1; val[1] = 0; }
                } else if (npos == 2 && pos[0] == pos[1]) {  // duplicate offsets only arise from padded slots (zero values)
                    if (pos[0] == 3) pos[0] = 2; else pos[1] = pos[0] + 1;
                }
                v8[h][2 * c] = val[0];
                v8[h][2 * c + 1] = val[1];
                word |= (pos[0] | (pos[1] << 2)) << (4 * c + 16 * h);
            }
            cb += 4;
            o0 += 4;
            fresh = o0 == m;
            if (fresh) { o0 = 0; g++; }
        }
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int i = i0 + 8 * h;
            uint4 o;
            o.x = (uint32_t)v8[h][0] | ((uint32_t)v8[h][1] << 16);
            o.y = (uint32_t)v8[h][2] | ((uint32_t)v8[h][3] << 16);
            o.z = (uint32_t)v8[h][4] | ((uint32_t)v8[h][5] << 16);
            o.w = (uint32_t)v8[h][6] | ((uint32_t)v8[h][7] << 16);
            *reinterpret_cast<uint4 *>(block + i * 128 + ((q ^ (i & 7)) << 4)) = o;
        }
        const int lane = (i0 & 7) + 8 * (q & 1) + 16 * (i0 >> 4);
        *reinterpret_cast<uint32_t *>(block + A_IMG_BYTES + (lane * 4 + (q >> 1)) * 4) = word;
    }
}

// ------------------------------------------------------------------------------------------------
// Transpose of an activation, [N, K] -> [K, N] (fp16), for the gather form, which needs rows of B.  A block takes 64 n x 64 k:
// a thread reads 16 bytes (8 k) of two neighbouring n, interleaves them into eight words (n, n + 1) and puts them into shared
// memory as [k][n pair] (pitch 33 words); then eight threads write the 128 bytes of one k.  Bound by HBM / L2: both
// sides move 128 contiguous bytes a row.  The n blocks are the grid's second dimension and, beyond its 65535 (4194240 rows), the third.
// ------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) transpose_kernel(const __half *__restrict__ src, int64_t ld, int N, int K, __half *__restrict__ dst)
{
    __shared__ uint32_t tile[64 * 33];
    const unsigned first = (blockIdx.y + blockIdx.z * gridDim.y) * 64u;
    const int k0 = blockIdx.x * 64, n0 = (int)first;
    grid_dependency_wait();
    grid_launch_dependents();   // the product's set-up may begin
    if (first >= (unsigned)N) return;   // the whole block
    {
        const int c = threadIdx.x & 7, np = threadIdx.x >> 3;   // 8 k at k0 + 8 c of rows n0 + 2 np, + 1 (N is even: both exist or neither)
        const int k = k0 + 8 * c, n = n0 + 2 * np;
        if (n < N && k < K) {
            const __half *r0 = src + (int64_t)n * ld + k, *r1 = r0 + ld;
            uint32_t a[4] = {0, 0, 0, 0}, b[4] = {0, 0, 0, 0};
            if (k + 8 <= K) {
                const uint4 x = __ldg(reinterpret_cast<const uint4 *>(r0)), y = __ldg(reinterpret_cast<const uint4 *>(r1));
                a[0] = x.x; a[1] = x.y; a[2] = x.z; a[3] = x.w;
                b[0] = y.x; b[1] = y.y; b[2] = y.z; b[3] = y.w;
            } else {   // K ends inside the piece
                for (int i = 0; i < K - k; i++) {
                    a[i >> 1] |= (uint32_t)__half_as_ushort(r0[i]) << (16 * (i & 1));
                    b[i >> 1] |= (uint32_t)__half_as_ushort(r1[i]) << (16 * (i & 1));
                }
            }
#pragma unroll
            for (int i = 0; i < 4; i++) {
                tile[(8 * c + 2 * i) * 33 + np] = __byte_perm(a[i], b[i], 0x5410);
                tile[(8 * c + 2 * i + 1) * 33 + np] = __byte_perm(a[i], b[i], 0x7632);
            }
        }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 2; i++) {
        const int k = (threadIdx.x >> 3) + 32 * i, q = threadIdx.x & 7;
        const int n = n0 + 8 * q;
        if (k0 + k < K && n < N) {   // N is a multiple of 8
            const uint32_t *w = tile + k * 33 + 4 * q;
            *reinterpret_cast<uint4 *>(dst + (int64_t)(k0 + k) * N + n) = make_uint4(w[0], w[1], w[2], w[3]);
        }
    }
}

cudaError_t launch_transpose(const void *src, int64_t ld_src, int N, int K, void *dst, cudaStream_t stream)
{
    const unsigned kblocks = ((unsigned)K + 63u) / 64u, nblocks = ((unsigned)N + 63u) / 64u, rows = nblocks < 65535u ? nblocks : 65535u;
    cudaLaunchConfig_t lc = {};
    cudaLaunchAttribute attr = early_launch();
    lc.gridDim = dim3(kblocks, rows, (nblocks + rows - 1) / rows);
    lc.blockDim = dim3(256, 1, 1);
    lc.stream = stream;
    lc.attrs = &attr;
    lc.numAttrs = 1;
    return cudaLaunchKernelEx(&lc, transpose_kernel, (const __half *)src, ld_src, N, K, (__half *)dst);
}

cudaError_t launch_prepare_dense_b(const void *values, const uint32_t *meta, const uint32_t *colloc, int M, int K, int V, int m,
                                   void *am, int mtiles, int ktiles, cudaStream_t stream)
{
    const int64_t Ksp = ksp_of(K, m);
    const int64_t cap = (int64_t)148 * 64;
    const int64_t total = (int64_t)mtiles * ktiles * 512;
    int64_t blocks = (total + 255) / 256;
    if (blocks > cap) blocks = cap;
    prepare_dense_b_kernel<<<(unsigned)blocks, 256, 0, stream>>>((const __half *)values, meta, colloc, M, K, V, m, Ksp, mtiles, ktiles,
                                                               (uint8_t *)am);
    return cudaGetLastError();
}

cudaError_t launch_prepare(const void *values, const uint32_t *meta, const uint32_t *colloc, int M, int K, int V, int m,
                           void *am, void *rows, int mtiles, int ktiles, int vblocks_padded, cudaStream_t stream)
{
    const int64_t Ksp = ksp_of(K, m);
    {
        const int64_t total = (int64_t)mtiles * ktiles * (AM_BLOCK_BYTES / 16);
        int64_t blocks = (total + 255) / 256;
        const int64_t cap = (int64_t)148 * 64;
        if (blocks > cap) blocks = cap;
        prepare_am_kernel<<<(unsigned)blocks, 256, 0, stream>>>((const __half *)values, meta, M, Ksp, mtiles, ktiles, (uint4 *)am);
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    {
        const int64_t total = (int64_t)vblocks_padded * ktiles * KT_GROUPS;
        int64_t blocks = (total + 255) / 256;
        const int64_t cap = (int64_t)148 * 64;
        if (blocks > cap) blocks = cap;
        prepare_rows_kernel<<<(unsigned)blocks, 256, 0, stream>>>(colloc, M, K, V, m, Ksp, vblocks_padded, ktiles, (int4 *)rows);
        return cudaGetLastError();
    }
}

}  // namespace vnm
