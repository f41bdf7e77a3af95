// Internal interface between the C ABI (vnm_capi.cu) and the kernel translation units.
#pragma once

#include "vnm_common.cuh"
#include <cuda.h>

namespace vnm {

// Device-side status word values (sticky, OR-ed): which bounded wait gave up.
enum : int {
    DEV_OK = 0,
    DEV_TIMEOUT_PRODUCER = 1,  // producer waited for a free stage
    DEV_TIMEOUT_MMA = 2,       // MMA issuer waited for a filled stage
    DEV_TIMEOUT_EPILOGUE = 4,  // epilogue waited for the accumulator
    DEV_TIMEOUT_DRAIN = 8      // drain of in-flight copies after an abort gave up
};

struct SpmmParams {
    const uint8_t *am;    // [mtiles][ktiles][AM_BLOCK_BYTES] value + metadata images
    const int4 *rows;     // [vblocks_padded][ktiles*32] absolute B rows
    const __half *bias;   // [M] or null
    __half *out;
    int64_t ldo;
    int M, N, K;
    int V;
    int mtiles, ktiles, ntiles;
    int layout;           // 0 = [M,N], 1 = [N,M] + bias
    int *status;          // device status word
    int gather_mode;      // GATHER_* below
    int total_tiles;      // mtiles * ntiles
    const __half *B;      // gather kernel, GATHER_CPASYNC: the dense operand [K, N] itself (row pieces are copied by address)
    int64_t ldb;
    int hybrid_rows;      // gather kernel, GATHER_CPASYNC: of 64 rows of a block, those fetched by TMA gather4 beside the copies (0, 16, 32, 48)
    int group_m;          // band of the tile order (tile_coords): > 0 row groups per band, < 0 column tiles per band
    uint64_t hint_a, hint_b;  // pair kernel: L2 eviction-priority policies of the A and B loads (L2_EVICT_*)
    int b_nk;             // dense-B kernel only: the dense operand is given as [N, K] row-major (K contiguous)
    int b_wide_ok;        // dense-B kernel only: the 4-D tensor map exists (column tiles with 256 columns inside N use one box per stage)
    int l2_ahead;         // pair kernel: k-tiles by which L2 prefetches run ahead of the loads into shared memory (0 = none)
    int out32;            // gather kernel, layout MN: 32-bit stores (ablation)
    int tma_out;          // gather kernel, layout NM: the result leaves through shared memory and TMA stores (tmap_out / OutMaps valid), else from registers
    int n_out;            // destinations of every output tile stored through TMA (1 = `out` only; more: the OutMaps argument, e.g. peers' buffers)
};

// Destinations 2 .. MAX_OUTS of a product whose every output tile is stored to several buffers of one geometry
// (a rank's own result buffer and the same rows of its peers' buffers): tensor maps like the first output map.
constexpr int MAX_OUTS = 8;
struct alignas(64) OutMaps {
    CUtensorMap m[MAX_OUTS - 1];
};

// How the producer warps bring the selected rows of B into shared memory.
enum : int {
    GATHER_TMA4 = 0,    // TMA tile::gather4, four rows (one group) per instruction (default for m > 4)
    GATHER_CONTIG = 1,  // plain TMA tiles of 64 consecutive rows: exact when m == 4 (every row is
                        // selected), otherwise an ablation that drops the column-loc indirection
    GATHER_NONE = 2,    // ablation only: B is not loaded at all (results are meaningless)
    GATHER_CPASYNC = 3  // per-thread 16-byte asynchronous copies of the selected rows, optionally split with TMA gather4 (ablation: measured slower)
};

struct SpmmConfig {
    int bn;      // tile N
    int nb;      // V-blocks per 128-row tile
    int part;    // columns per epilogue part (width of a TMA store box)
    int stages;  // gather kernel: number of B-producer warps; dense-B kernels: SMs per tile
    int smem_bytes;
    int threads;
    int grid;    // persistent CTAs
};

// Host-side helpers shared by the translation units that implement C-ABI entry points (defined in vnm_capi.cu).
int set_last_error(int code, const char *msg);       // message of vnm_last_error_string() for this thread; returns code
int check_format(int M, int K, int V, int n, int m);  // VNM_OK or an error code with the message set
typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                                  const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
CUresult encode_out_map(EncodeTiledFn enc, CUtensorMap *map, void *out, int M, int N, int64_t ldo, int layout, int part);  // result buffer, for TMA stores
EncodeTiledFn get_encode_fn();                        // cuTensorMapEncodeTiled from the driver, or null (thread-safe)

cudaError_t launch_compress(const void *dense, int64_t ldd, const int32_t *mask, const uint32_t *colloc, int M, int K, int V, int m,
                            void *values, uint32_t *meta, unsigned long long *violations, cudaStream_t stream);
cudaError_t launch_decompress(const void *values, const uint32_t *meta, const uint32_t *colloc, int M, int K, int V, int m,
                              void *dense, int64_t ldd, cudaStream_t stream);
cudaError_t launch_prepare(const void *values, const uint32_t *meta, const uint32_t *colloc, int M, int K, int V, int m, void *am,
                           void *rows, int mtiles, int ktiles, int vblocks_padded, cudaStream_t stream);

cudaError_t launch_prepare_dense_b(const void *values, const uint32_t *meta, const uint32_t *colloc, int M, int K, int V, int m,
                                   void *am, void *rows, int mtiles, int ktiles, cudaStream_t stream);

cudaError_t launch_prune(const float *w, int64_t ldw, int M, int K, int V, int m, int32_t *mask, int64_t ldm, uint32_t *colloc,
                         cudaStream_t stream);

// Chooses the tile configuration for (V, N).  Returns false for an unsupported V.
bool spmm_select_config(int V, int N, int M, int max_ctas, SpmmConfig *cfg);  // max_ctas: 0 = one per SM
// Opt-in to large dynamic shared memory for every kernel instance on the CURRENT device (call once per device).
cudaError_t spmm_init_kernels();
cudaError_t launch_spmm(const SpmmConfig &cfg, const CUtensorMap &tmap_rows, const CUtensorMap &tmap_tile, const CUtensorMap &tmap_out,
                        const OutMaps &more_out, const SpmmParams &p,
                        cudaStream_t stream);

// Dense-B form: 256 x 128 tiles, two accumulators sharing every B stage (vnm_spmm_dense_b.cu).
cudaError_t spmm_dense_b_init();
cudaError_t launch_wait_expiry_selftest(int *status, cudaStream_t stream);
void spmm_dense_b_config(int M, int N, int max_ctas, SpmmConfig *cfg);  // max_ctas: 0 = one per SM
cudaError_t launch_spmm_dense_b(const SpmmConfig &cfg, const CUtensorMap &tmap_tile, const CUtensorMap &tmap_tile2, const CUtensorMap &tmap_out, const OutMaps &more_out,
                                const SpmmParams &p, cudaStream_t stream);

// Dense-B form on pairs of SMs (clusters of two CTAs, tcgen05 cta_group::2): 512 x 240 pair tiles (vnm_spmm_dense_b2.cu).
cudaError_t spmm_dense_b_pair_init();
bool spmm_dense_b_pair_config(int M, int N, int K, int max_ctas, int force_rows, SpmmConfig *cfg);  // false: use the single-CTA kernel; force_rows: 0 auto, 1 / 2 row tiles per CTA
cudaError_t launch_spmm_dense_b_pair(const SpmmConfig &cfg, const CUtensorMap &tmap_tile, const CUtensorMap &tmap_tile2, const CUtensorMap &tmap_out, const OutMaps &more_out,
                                     const SpmmParams &p, cudaStream_t stream);

#if defined(__CUDACC__)
// ---- bounded waits of the persistent kernels ----
constexpr long long WAIT_LIMIT_CYCLES = 4000000000LL;  // ~2 s at B200 clocks

// Single-thread bounded wait (no warp convergence needed) that probes without suspending the thread: the fastest
// hand-off, for the few threads that a critical hand-off waits for.
__device__ __forceinline__ bool wait_one(uint64_t *bar, uint32_t parity, volatile int *abort_flag, int *status, int code)
{
    if (mbar_test_wait(bar, parity)) return true;
    const long long t0 = clock64();
    for (uint32_t it = 0;; ++it) {
        if (mbar_test_wait(bar, parity)) return true;
        if ((it & 1023u) == 1023u) {
            if (*abort_flag) return false;
            if (clock64() - t0 > WAIT_LIMIT_CYCLES) {
                *abort_flag = 1;
                atomicOr(status, code);
                return false;
            }
        }
    }
}

// The same wait with the suspending probe, for roles of many warps: spinning warps would take issue slots and
// shared-memory cycles from the others.
__device__ __forceinline__ bool wait_quiet(uint64_t *bar, uint32_t parity, volatile int *abort_flag, int *status, int code)
{
    if (mbar_try_wait(bar, parity)) return true;
    const long long t0 = clock64();
    for (uint32_t it = 0;; ++it) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((it & 63u) == 63u) {
            if (*abort_flag) return false;
            if (clock64() - t0 > WAIT_LIMIT_CYCLES) {
                *abort_flag = 1;
                atomicOr(status, code);
                return false;
            }
        }
    }
}

// Whole-warp wait: lane 0 polls.
__device__ __forceinline__ bool wait_warp(uint64_t *bar, uint32_t parity, volatile int *abort_flag, int *status, int code)
{
    int ok = 1;
    if ((threadIdx.x & 31) == 0) ok = wait_quiet(bar, parity, abort_flag, status, code) ? 1 : 0;
    return __shfl_sync(0xffffffffu, ok, 0) != 0;
}

// Bounded wait used only while draining after an abort: until the copies of one ring slot have landed.
__device__ __forceinline__ void drain_slot(uint64_t *bar, uint32_t parity, int *status)
{
    const long long t0 = clock64();
    while (clock64() - t0 < WAIT_LIMIT_CYCLES / 4) {
        if (mbar_try_wait(bar, parity)) return;
    }
    atomicOr(status, DEV_TIMEOUT_DRAIN);
}

// ---- epilogue of one warp straight from tensor memory to global memory (32 accumulator lanes x BN columns) ----
// Nothing of it passes through shared memory, whose port the mainloop needs: the operand reads of the MMAs and the TMA
// writes of the rings together keep it busy all the time.  `trow` is the address of the accumulator at this warp's lane
// quadrant q, `row0` the actual row of accumulator lane 0 of the tile.  `release` runs (converged) once the last column has
// been read.  Columns >= N and rows >= M are not stored.

// [M,N]: a lane owns a row and stores 16 columns, one 32-byte sector, at a time (two 16-byte pieces where the rows are
// not 32-byte aligned or N ends inside; 4-byte words for the `out32` ablation, the reference's OUT_32B build,
// common/epilogue.h:34-61).
template <int BN, typename Release>
__device__ __forceinline__ void store_tile_mn(uint32_t trow, int q, int64_t row0, int n0, const SpmmParams &p, Release release)
{
    constexpr int SPAN = BN % 48 == 0 ? 48 : BN < 32 ? BN : 32;
    static_assert(BN % SPAN == 0 && SPAN % 16 == 0, "column spans");
    const int lane = threadIdx.x & 31;
    const int64_t row = row0 + mma_row_to_actual(q * 32 + lane);
    __half *orow = p.out + row * p.ldo + n0;
    const bool row_ok = row < p.M;
    const bool wide = (p.ldo & 15) == 0 && ((uintptr_t)p.out & 31) == 0;
#pragma unroll 1
    for (int c0 = 0; c0 < BN; c0 += SPAN) {
        uint32_t v[SPAN / 16][16];
#pragma unroll
        for (int i = 0; i < SPAN / 16; i++) tc_ld_32x32b_x16(trow + (uint32_t)(c0 + 16 * i), v[i]);
        tc_wait_ld();
        if (c0 == BN - SPAN) release();
#pragma unroll
        for (int i = 0; i < SPAN / 16; i++) {
            uint32_t pk[8];
#pragma unroll
            for (int k = 0; k < 8; k++) pk[k] = pack_half2(v[i][2 * k], v[i][2 * k + 1]);
            const int c = c0 + 16 * i, left = p.N - n0 - c;
            if (!row_ok || left <= 0) continue;
            if (p.out32) {
#pragma unroll
                for (int k = 0; k < 8; k++)
                    if (2 * k < left) *reinterpret_cast<uint32_t *>(orow + c + 2 * k) = pk[k];
            } else if (wide && left >= 16) {
                st_global_v8(orow + c, pk);
            } else {
                *reinterpret_cast<uint4 *>(orow + c) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
                if (left >= 16) *reinterpret_cast<uint4 *>(orow + c + 8) = make_uint4(pk[4], pk[5], pk[6], pk[7]);
            }
        }
    }
}

// [N,M] (+ bias): accumulator lanes w and w + 8 of a 16-lane group are the actual rows 2w and 2w + 1, and the fragment
// order hands both to one thread: a 32-bit word of two neighbouring m.  Eight threads store one 32-byte sector of an n row, a
// store instruction four of them.
template <int BN, typename Release>
__device__ __forceinline__ void store_tile_nm(uint32_t trow, int q, int64_t row0, int n0, const SpmmParams &p, Release release)
{
    const int lane = threadIdx.x & 31;
    const int64_t m0 = row0 + q * 32 + (lane >> 2) * 2;      // rows m0, m0 + 1 of the first 16-row group; + 16 for the second
    const bool ok[2] = {m0 < p.M, m0 + 16 < p.M};            // M is a multiple of 32
    const bool words = (p.ldo & 1) == 0 && ((uintptr_t)p.out & 3) == 0;
    __half2 bias[2];
#pragma unroll
    for (int g = 0; g < 2; g++) bias[g] = (p.bias && ok[g]) ? __halves2half2(p.bias[m0 + 16 * g], p.bias[m0 + 16 * g + 1]) : __half2half2(__ushort_as_half((unsigned short)0));
    const bool has_bias = p.bias != nullptr;
    const int ncol = n0 + (lane & 3) * 2;
#pragma unroll 1
    for (int c0 = 0; c0 < BN; c0 += 16) {
        uint32_t v[2][8];
        tc_ld_16x256b_x2(trow + (uint32_t)c0, v[0]);
        tc_ld_16x256b_x2(trow + (16u << 16) + (uint32_t)c0, v[1]);
        tc_wait_ld();
        if (c0 == BN - 16) release();
#pragma unroll
        for (int j = 0; j < 2; j++)
#pragma unroll
            for (int e = 0; e < 2; e++) {
                const int n = ncol + c0 + 8 * j + e;
                if (n >= p.N) continue;
                __half *dst = p.out + (int64_t)n * p.ldo + m0;
#pragma unroll
                for (int g = 0; g < 2; g++) {
                    __half2 h = __floats2half2_rn(__uint_as_float(v[g][4 * j + e]), __uint_as_float(v[g][4 * j + 2 + e]));
                    if (has_bias) h = __hadd2(h, bias[g]);
                    if (!ok[g]) continue;
                    if (words) {
                        *reinterpret_cast<__half2 *>(dst + 16 * g) = h;
                    } else {
                        dst[16 * g] = __low2half(h);
                        dst[16 * g + 1] = __high2half(h);
                    }
                }
            }
    }
}
#endif  // __CUDACC__

}  // namespace vnm
