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

// 160 bytes: four more cost the small kernel's launches 0.5 us each (5.5 -> 6.0 us a call at 1024 x 1024, 8 columns).
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
    int total_tiles;      // mtiles * ntiles; gather kernel: tiles and halves of tiles
    const __half *B;      // gather kernel, GATHER_CPASYNC: the dense operand [K, N] itself (row pieces are copied by address)
    int64_t ldb;
    int16_t producer_warps;   // gather kernel: how much of the warps that load B is at work, in 16ths: 16 except for an ablation
    int16_t hybrid_rows;  // gather kernel, GATHER_CPASYNC: of 64 rows of a block, those fetched by TMA gather4 beside the copies (0, 16, 32, 48)
    int group_m;          // band of the tile order (tile_coords): > 0 row groups per band, < 0 column tiles per band
    uint64_t hint_a, hint_b;  // pair kernel: L2 eviction-priority policies of the A and B loads (L2_EVICT_*)
    int b_nk;             // dense-B form only: the dense operand is given as [N, K] row-major (K contiguous)
    int b_wide_ok;        // pair kernel: the 4-D tensor map exists (halves with 128 columns inside N use one box per stage)
    int l2_ahead;         // pair kernel: k-tiles by which L2 prefetches run ahead of the loads into shared memory (0 = none)
    int out32;            // gather kernel, layout MN: 32-bit stores (ablation)
    int tma_out;          // gather kernel, layout NM: the result leaves through shared memory and TMA stores (tmap_out / OutMaps valid), else from registers
    int early;            // small kernel: the kernel ahead only transposes B; all else may be read before it has finished
    int split_k;          // small kernel: CTAs of a cluster that share one tile's k-tiles
    int n_out;            // destinations of every output tile stored through TMA (1 = `out` only; more: the OutMaps argument, e.g. peers' buffers)
};
static_assert(sizeof(SpmmParams) <= 160, "see above");

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
    int stages;  // gather kernel: number of B-producer warps; the others: SMs per tile
    int smem_bytes;
    int threads;
    int grid;    // CTAs (persistent ones, except in the small kernel)
    int split;   // small kernel: CTAs that share a tile's k-tiles
    int resident;  // small kernel: CTAs per SM
    int deep;      // small kernel: the instance whose ring takes an SM's whole shared memory
    int tiles;     // gather kernel: tiles of the launch, halves counted
    int cut_from;  // gather kernel: first of the tiles that are cut in two (`tiles`: none)
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
                                   void *am, int mtiles, int ktiles, cudaStream_t stream);

cudaError_t launch_transpose(const void *src, int64_t ld_src, int N, int K, void *dst, cudaStream_t stream);  // [N, K] -> [K, N], fp16

cudaError_t launch_prune(const float *w, int64_t ldw, int M, int K, int V, int m, int32_t *mask, int64_t ldm, uint32_t *colloc,
                         cudaStream_t stream);

// Pruner and compressor in one pass over the weights (fp16 or fp32).
bool sparsify_supported(int K, int V, int m);
cudaError_t launch_sparsify(const void *w, bool half, int64_t ldw, int M, int K, int V, int m, void *values, uint32_t *meta, uint32_t *colloc,
                            unsigned long long *violations, cudaStream_t stream);

// Tile configuration of the gather kernel.
constexpr int GATHER_PRODUCER_WARPS = 16;   // all of them, in the units of vnm_set_producer_warps
float spmm_select_config(int V, int N, int M, int ktiles, int max_ctas, int gather_mode, SpmmConfig *cfg);  // max_ctas: 0 = one per SM; returns an estimate in microseconds, < 0 for an unsupported V
// Opt-in to large dynamic shared memory for every kernel instance on the CURRENT device (call once per device).
cudaError_t spmm_init_kernels();
cudaError_t launch_spmm(const SpmmConfig &cfg, const CUtensorMap &tmap_rows, const CUtensorMap &tmap_tile, const CUtensorMap &tmap_out,
                        const OutMaps &more_out, const SpmmParams &p,
                        cudaStream_t stream);

// Few columns or few tiles, both operand forms: 128 x (16 .. 128) tiles, several CTAs per SM, k-tiles split over a cluster
// for N <= SMALL_SPLIT_N (vnm_spmm_small.cu).  nb: vector blocks per row tile (1 for the dense-B form).
constexpr int SMALL_SPLIT_N = 64;
cudaError_t spmm_small_init();
cudaError_t launch_wait_expiry_selftest(int *status, cudaStream_t stream);
float spmm_small_config(int mtiles, int ktiles, int N, int nb, bool gather, bool every_row, bool b_nk, SpmmConfig *cfg);   // returns its estimate in microseconds
CUresult spmm_small_encode(EncodeTiledFn enc, CUtensorMap *map, const void *B, int64_t ldb, int K, int N, int b_nk, int gather_mode, int bn);
cudaError_t launch_spmm_small(const SpmmConfig &cfg, const CUtensorMap &tmap_b, const SpmmParams &p, cudaStream_t stream);

// Dense-B form on pairs of SMs (clusters of two CTAs, tcgen05 cta_group::2): pair tiles of 512 or 256 rows (vnm_spmm_dense_b2.cu).
cudaError_t spmm_dense_b_pair_init();
float spmm_dense_b_pair_config(int M, int N, int K, int b_nk, int max_ctas, int force_rows, bool multi, SpmmConfig *cfg);  // < 0: not for this problem, else an estimate in microseconds; force_rows: 0 auto, 1 / 2 row tiles per CTA
cudaError_t launch_spmm_dense_b_pair(const SpmmConfig &cfg, const CUtensorMap &tmap_tile, const CUtensorMap &tmap_tile2, const CUtensorMap &tmap_out, const OutMaps &more_out,
                                     const SpmmParams &p, cudaStream_t stream);

// Every product (and the transpose ahead of one) is launched with this attribute: it may be scheduled once all blocks of the kernel
// ahead of it in the stream have called grid_launch_dependents() or left, sets up its barriers beside that kernel's last blocks,
// and waits for its end in grid_dependency_wait() before it touches memory that others use.  Tensor memory is allocated after that
// wait and dependents are let in only after the allocation: a block that waits for another kernel holds none of what that kernel's
// blocks may still be waiting for.
inline cudaLaunchAttribute early_launch()
{
    cudaLaunchAttribute a = {};
    a.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    a.val.programmaticStreamSerializationAllowed = 1;
    return a;
}

#if defined(__CUDACC__)
// Programmatic dependent launch: waits until the kernels this launch depends on have finished; lets dependents start.
__device__ __forceinline__ void grid_dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

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

// Fill j of a ring goes to slot j % slots in phase j / slots.  The last of `fills` fills that slot `slot` got, or -1.
__host__ __device__ constexpr int last_fill(int slot, int slots, int fills) { return fills > slot ? fills - 1 - (fills - 1 - slot) % slots : -1; }
// Whatever the number of slots and fills: a fill of this slot, none of a later round beside it (whose phase has the parity that the wait for an
// older one waits for, so that it never ends), and no slot forgotten.
constexpr bool last_fill_holds()
{
    for (int slots = 2; slots <= 9; slots++)
        for (int fills = 0; fills <= 3 * slots; fills++)
            for (int slot = 0; slot < slots; slot++) {
                const int j = last_fill(slot, slots, fills);
                if (j < 0 ? fills > slot : j % slots != slot || j >= fills || j + slots < fills) return false;
            }
    return true;
}
static_assert(last_fill_holds(), "the fills that a drain waits for");

// After an abort, one warp, when no other issues loads any more: waits until the last fill of every slot has landed.  Older ones have: their slot was free
// again before it was refilled, whichever warp did that.
__device__ __forceinline__ void drain_ring(uint64_t *full, int slots, int fills, int *status)
{
    const int lane = threadIdx.x & 31, j = lane < slots ? last_fill(lane, slots, fills) : -1;
    if (j >= 0) drain_slot(&full[lane], (uint32_t)(j / slots) & 1u, status);
    __syncwarp();
}

// ---- epilogue of one warp straight from tensor memory to global memory (32 accumulator lanes x BN columns) ----
// Nothing of it passes through shared memory, whose port the mainloop needs: the operand reads of the MMAs and the TMA
// writes of the rings together keep it busy all the time.  What the stores must not do is flood L2 with small pieces, behind
// which the loads of the next tile queue: sectors of 32 bytes from 32 different rows cost the next tile about 3500 of its
// 11000 clocks (4096 x 1024 x 16384, [M,N]).  So lanes exchange words of [M,N] results until an instruction writes 128
// contiguous bytes of a row.  Accumulators are read in fragment order: thread t holds columns 2 (t % 4), + 1 of every eight for lanes t / 4 and
// t / 4 + 8 of a 16-lane group, which are the actual rows 2 (t / 4) and 2 (t / 4) + 1.  Work goes in chunks of 64 columns,
// 32 packed words a thread.  Columns >= N and rows >= M are not stored.

__device__ __forceinline__ void quad_swap(uint32_t &a, uint32_t &b, bool up, int mask)   // exchanges b of the lower lane with a of the upper one
{
    const uint32_t got = __shfl_xor_sync(0xffffffffu, up ? a : b, mask);
    if (up) a = got; else b = got;
}

// [M,N]: a quad of threads holds 64 columns of a row as words (8 j + 2 i, + 1); two 4 x 4 transposes give each thread 16
// consecutive columns, so that a store instruction (32 bytes a thread) writes 128 contiguous bytes of eight rows.  16-byte pieces
// where the rows are not 32-byte aligned or N ends inside; 4-byte words for the `out32` ablation, the reference's
// OUT_32B build, common/epilogue.h:34-61.
struct TileStoreMN {
    __half *dst;         // row 2 (t / 4) of the warp's first 16-row group, this thread's 16 columns of the first chunk
    int64_t ldo;
    int left;            // columns from there to N
    bool ok[2], wide, words;   // ok: rows of the two 16-row groups exist (M is a multiple of 32)
    uint32_t taddr;
    // `trow`: the accumulator at this warp's lane quadrant q; row0: the actual row of the tile's first lane
    __device__ __forceinline__ TileStoreMN(uint32_t trow, int q, int64_t row0, int n0, const SpmmParams &p)
    {
        const int lane = threadIdx.x & 31;
        const int64_t row = row0 + q * 32 + (lane >> 2) * 2;
        const int n = n0 + (lane & 3) * 16;
        dst = p.out + row * p.ldo + n;
        ldo = p.ldo;
        left = p.N - n;
        ok[0] = row < p.M; ok[1] = row + 16 < p.M;
        wide = (p.ldo & 15) == 0 && ((uintptr_t)p.out & 31) == 0;
        words = p.out32 != 0;
        taddr = trow;
    }
    // one group: words pk[0..7] of row 2w, pk[8..15] of row 2w + 1; word j: columns 8 j + 2 (t % 4), + 1 of the chunk
    __device__ __forceinline__ static void pack(const uint32_t (&v)[32], uint32_t *pk)
    {
#pragma unroll
        for (int j = 0; j < 8; j++) {
            pk[j] = pack_half2(v[4 * j], v[4 * j + 1]);
            pk[8 + j] = pack_half2(v[4 * j + 2], v[4 * j + 3]);
        }
    }
    __device__ __forceinline__ void store(int c, int g, int cols, uint32_t *pk) const
    {
        const int lane = threadIdx.x & 31;
        const bool odd = (lane & 1) != 0, upper = (lane & 2) != 0;
#pragma unroll
        for (int r = 0; r < 2; r++) {
            uint32_t *w = pk + 8 * r;
            // words of groups 0, 2, 4, 6 and of 1, 3, 5, 7: thread i ends with groups 2 i and 2 i + 1
#pragma unroll
            for (int h = 0; h < 2; h++) {
                quad_swap(w[0 + h], w[2 + h], odd, 1);
                quad_swap(w[4 + h], w[6 + h], odd, 1);
                quad_swap(w[0 + h], w[4 + h], upper, 2);
                quad_swap(w[2 + h], w[6 + h], upper, 2);
            }
            const uint32_t o[8] = {w[0], w[2], w[4], w[6], w[1], w[3], w[5], w[7]};
            const int rest = left - c;
            if (!ok[g] || rest <= 0 || (lane & 3) * 16 >= cols) continue;
            __half *d = dst + (int64_t)(16 * g + r) * ldo + c;
            if (words) {
#pragma unroll
                for (int k = 0; k < 8; k++)
                    if (2 * k < rest) *reinterpret_cast<uint32_t *>(d + 2 * k) = o[k];
            } else if (wide && rest >= 16) {
                st_global_v8(d, o);
            } else {
                *reinterpret_cast<uint4 *>(d) = make_uint4(o[0], o[1], o[2], o[3]);
                if (rest >= 16) *reinterpret_cast<uint4 *>(d + 8) = make_uint4(o[4], o[5], o[6], o[7]);
            }
        }
    }
};

// [N,M] (+ bias): a word is two neighbouring m (rows 2w, 2w + 1), so that eight threads fill a 32-byte sector of an n row and a
// store instruction writes four of them.  (Exchanging words for 64 contiguous bytes of two n rows took 2.4 times as long.)
struct TileStoreNM {
    __half *dst;         // first n this thread stores, its two m of the first 16-row group
    int64_t ldo;
    int left;
    bool ok[2], words;   // ok: rows of the two 16-row groups exist (M is a multiple of 32)
    __half2 bias[2];     // -0 without a bias: x + -0 is x, bit for bit
    uint32_t taddr;
    __device__ __forceinline__ TileStoreNM(uint32_t trow, int q, int64_t row0, int n0, const SpmmParams &p)
    {
        const int lane = threadIdx.x & 31;
        const int64_t m0 = row0 + q * 32 + (lane >> 2) * 2;
        const int n = n0 + (lane & 3) * 2;
        dst = p.out + (int64_t)n * p.ldo + m0;
        ldo = p.ldo;
        left = p.N - n;
        words = (p.ldo & 1) == 0 && ((uintptr_t)p.out & 3) == 0;
#pragma unroll
        for (int g = 0; g < 2; g++) {
            ok[g] = m0 + 16 * g < p.M;
            bias[g] = (p.bias && ok[g]) ? __halves2half2(p.bias[m0 + 16 * g], p.bias[m0 + 16 * g + 1]) : __half2half2(__ushort_as_half((unsigned short)0x8000));
        }
        taddr = trow;
    }
    // one group: word 2 j + e of pk: column 8 j + 2 (t % 4) + e of the chunk
    __device__ __forceinline__ static void pack(const uint32_t (&v)[32], uint32_t *pk)
    {
#pragma unroll
        for (int j = 0; j < 8; j++) {
            pk[2 * j] = pack_half2(v[4 * j], v[4 * j + 2]);
            pk[2 * j + 1] = pack_half2(v[4 * j + 1], v[4 * j + 3]);
        }
    }
    __device__ __forceinline__ void store(int c, int cols, const uint32_t *pk) const   // both groups
    {
        __half *d = dst + (int64_t)c * ldo;
        if (words && ok[0] && ok[1] && c + 64 <= left) {
            // whole chunk (columns past `cols` belong to nobody): two adds, a half2 add and a store a word.  With the checks below
            // around every word the stores of a tile took 11500 clocks, longer than the MMAs of a tile of eight k-tiles.
#pragma unroll
            for (int j = 0; j < 8; j++) {
                if (8 * j >= cols) break;
#pragma unroll
                for (int e = 0; e < 2; e++) {
#pragma unroll
                    for (int g = 0; g < 2; g++) {
                        uint32_t w = pk[16 * g + 2 * j + e];
                        *reinterpret_cast<__half2 *>(d + e * ldo + 16 * g) = __hadd2(*reinterpret_cast<__half2 *>(&w), bias[g]);
                    }
                }
                d += 8 * ldo;
            }
            return;
        }
#pragma unroll
        for (int j = 0; j < 8; j++) {
            if (8 * j >= cols) break;
#pragma unroll
            for (int e = 0; e < 2; e++) {
                if (c + 8 * j + e >= left) continue;
#pragma unroll
                for (int g = 0; g < 2; g++) {
                    if (!ok[g]) continue;
                    uint32_t w = pk[16 * g + 2 * j + e];
                    const __half2 h = __hadd2(*reinterpret_cast<__half2 *>(&w), bias[g]);
                    __half *dd = d + (8 * j + e) * ldo + 16 * g;
                    if (words) {
                        *reinterpret_cast<__half2 *>(dd) = h;
                    } else {
                        dd[0] = __low2half(h);
                        dd[1] = __high2half(h);
                    }
                }
            }
        }
    }
};
__device__ __forceinline__ void store_chunk(const TileStoreMN &st, int c, int cols, uint32_t *pk) { st.store(c, 0, cols, pk); st.store(c, 1, cols, pk + 16); }
__device__ __forceinline__ void store_chunk(const TileStoreNM &st, int c, int cols, uint32_t *pk) { st.store(c, cols, pk); }

// BN columns in chunks of 64 (a last chunk of fewer reads on into columns that it does not store).  `release` runs
// (converged) once the last column has been read.  HOLD: all columns are read into registers first, for kernels whose next
// tile waits for this accumulator.
template <int BN, bool HOLD, typename Store, typename Release>
__device__ __forceinline__ void store_tile(const Store &st, Release release)
{
    constexpr int CHUNKS = (BN + 63) / 64;
    if (HOLD) {
        uint32_t pk[CHUNKS][32];
#pragma unroll
        for (int k = 0; k < CHUNKS; k++) {
            uint32_t v0[32], v1[32];   // both groups in flight before the wait: the next tile's MMAs wait for this
            tc_ld_16x256b(st.taddr + (uint32_t)(64 * k), v0);
            tc_ld_16x256b(st.taddr + (16u << 16) + (uint32_t)(64 * k), v1);
            tc_wait_ld();
            Store::pack(v0, pk[k]);
            Store::pack(v1, pk[k] + 16);
        }
        release();
#pragma unroll
        for (int k = 0; k < CHUNKS; k++) store_chunk(st, 64 * k, BN - 64 * k, pk[k]);
    } else {
#pragma unroll 1
        for (int k = 0; k < CHUNKS; k++) {
            uint32_t pk[32];
#pragma unroll
            for (int g = 0; g < 2; g++) {
                uint32_t v[32];
                tc_ld_16x256b(st.taddr + ((uint32_t)(16 * g) << 16) + (uint32_t)(64 * k), v);
                tc_wait_ld();
                Store::pack(v, pk + 16 * g);
            }
            if (k == CHUNKS - 1) release();
            store_chunk(st, 64 * k, BN - 64 * k, pk);
        }
    }
}
#endif  // __CUDACC__

}  // namespace vnm
